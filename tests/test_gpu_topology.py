"""The Morton levels held in shared memory (8192 nodes in a single build, 2560 in a batched one) and beyond it, with split
lists longer than the part kept beside them: nodes and counters against the CPU oracle, batched meshes against their own
builds. Exact."""
import numpy as np
import pytest

from cudart_b200 import scenes

pytestmark = pytest.mark.gpu


def _u32(a):
    return np.ascontiguousarray(a).view(np.uint32)


def _mesh(kind, n):
    if kind == "terrain":
        return scenes.terrain(int((n / 2) ** 0.5) + 1, 5)
    m = scenes.soup(n, seed=n)
    if kind == "clumps":  # most faces in a few cells: long runs of one code, levels without entries
        m.vertices[:, :3] = np.round(m.vertices[:, :3] * 4) / 4 + m.vertices[:, :3] * np.float32(1e-4)
    return m


@pytest.mark.parametrize("kind,n,depth", [("soup", 30000, 12), ("soup", 65000, 14), ("soup", 90000, 20), ("clumps", 90000, 32),
                                          ("terrain", 70000, 16), ("soup", 17, 12)])
def test_single(oracle, kind, n, depth):
    import torch
    from cudart_b200 import core
    m = _mesh(kind, n)
    t = core.build_lbvh(torch.from_numpy(m.vertices).cuda(), torch.from_numpy(m.faces.view(np.int32)).cuda(), tree_depth=depth)
    ref = oracle.lbvh_build(m.vertices, m.faces, oracle.hitbox(m.vertices), tree_depth=depth)
    info = t.info_host()
    assert info["error"] == 0
    for k in ("node_count", "leaf_count", "real_depth", "split_count", "overrun_visits", "nondet_reads", "past_end_reads"):
        assert info[k] == ref["info"][k], k
    nc = info["node_count"]
    assert np.array_equal(_u32(t.nodes.cpu().numpy()[:nc]), _u32(ref["nodes"]))
    assert np.array_equal(_u32(t.faces.cpu().numpy()), _u32(ref["faces"]))


@pytest.mark.parametrize("depth", [12, 20])
def test_batched(depth):
    import torch
    from cudart_b200 import core
    meshes = [_mesh(k, n) for k, n in (("soup", 40), ("soup", 25000), ("clumps", 60000), ("terrain", 3000), ("soup", 9000), ("soup", 1))]
    verts, faces, fo, vo = scenes.concat_batch(meshes)
    t = core.batch_build(torch.from_numpy(verts).cuda(), torch.from_numpy(faces.view(np.int32)).cuda(), fo, vo, tree_depth=depth)
    for i, m in enumerate(meshes):
        one = core.build_lbvh(torch.from_numpy(m.vertices).cuda(), torch.from_numpy(m.faces.view(np.int32)).cuda(), tree_depth=depth)
        nc = one.info_host()["node_count"]
        assert torch.equal(t.info[i], one.info)
        assert torch.equal(t.mesh_nodes(i, nc), one.nodes[:nc])
