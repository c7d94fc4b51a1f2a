"""A warp that leaves the packet walk hands each lane the packet's stack: what stands there must not keep a lane from a
closer hit, down to hits that differ by the smallest float. Against the oracle, bit for bit."""
import numpy as np
import pytest

from cudart_b200 import scenes

pytestmark = pytest.mark.gpu

TINY = np.float32(1.401298464324817e-45)  # the smallest float above 0


def _layers():
    """8 triangles at x = -10, then, around the origin, 24 in the plane z = 0 and 32 in the plane z = TINY. The root record
    of the cluster tree has the slots [0..3], [4..7], [8..31], [32..63]."""
    tri = np.array([[-1, -1, 0], [1, -1, 0], [-1, 1, 0]], np.float32)
    v = np.zeros((64, 3, 4), np.float32)
    v[:, :, :3] = tri
    v[:8, :, 0] -= 10
    v[32:, :, 2] = TINY
    f = np.zeros((64, 4), np.uint32)
    f[:, :3] = np.arange(192).reshape(64, 3)
    return scenes.Mesh(v.reshape(192, 4), f)


@pytest.mark.parametrize("threshold", [4, 5, 8, 16, 28, 29, 32])
def test_hits_a_smallest_float_apart(oracle, threshold):
    """28 lanes go to the first 8 triangles; the last four meet the triangles of [8..31] at t = TINY first, with [32..63],
    which they hit at t = 0, on the packet's stack."""
    import torch
    from cudart_b200 import core
    mesh = _layers()
    hit = [-16, -16, -16, 0, 16, 16, 16, 0]
    tree = core.build_lbvh(torch.from_numpy(mesh.vertices).cuda(), torch.from_numpy(mesh.faces.view(np.int32)).cuda(), hitbox=hit,
                           clusters=True)
    o, d = np.zeros((64, 4), np.float32), np.zeros((64, 4), np.float32)
    d[:, 2] = -1
    o[:, 0], o[:, 1] = np.linspace(-0.9, -0.1, 64), -0.5
    o[:, 2] = TINY
    o[:28, 0] -= 10
    o[:28, 2] = 0.25
    o[32:60, 0] -= 10
    ref = oracle.lbvh_build(mesh.vertices, mesh.faces, np.array(hit, np.float32))
    e = oracle.trace(ref["nodes"], ref["tris"], ref["indices"], o, d, None, mode=0)
    assert (e["id"][28:32] == 32).all() and (e["t"][28:32] == 0).all()
    for persistent in (1, 16):
        out = core.trace(tree, torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda(),
                         schedule=dict(clusters=True, persistent=True, blocks_per_sm=persistent, packet=True, lane_threshold=threshold))
        assert int(out["err"].item()) == 0
        assert np.array_equal(out["id"].cpu().numpy(), e["id"])
        assert np.array_equal(out["t"].cpu().numpy().view(np.uint32), e["t"].view(np.uint32))
        assert np.array_equal(out["uv"].cpu().numpy().view(np.uint32), e["uv"].view(np.uint32))
