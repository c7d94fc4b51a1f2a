"""A tree of 46 levels whose boxes all hold the rays' origins, so that every level leaves something on a walk's stack: each
walk of the node records against the two-child per-lane walk, without a stack error."""
import numpy as np
import pytest

from cudart_b200 import scenes

pytestmark = pytest.mark.gpu

HIT = [0, 0, 0, 0, 2047, 2047, 1023, 0]  # codes are the coordinates
CELL = 16 << 13                          # triangles of the last cell: 14 median levels above leaves of 8


def _mesh():
    """The codes 2^k and 2^k + 2^(k-1) (8 triangles each) and CELL triangles of code 0. The deeper a triangle, the farther
    back its box begins, so that a walk goes down to the last cell before it looks at anything else."""
    codes = np.concatenate([np.zeros(CELL, np.int64), np.ones(16, np.int64),
                            np.concatenate([np.repeat([1 << k, (1 << k) + (1 << (k - 1))], 8) for k in range(1, 32)])])
    c = np.zeros((len(codes), 3), np.float32)
    for k in range(11):
        c[:, 1] += ((codes >> (3 * k)) & 1) << k
        c[:, 0] += ((codes >> (3 * k + 1)) & 1) << k
        if k < 10:
            c[:, 2] += ((codes >> (3 * k + 2)) & 1) << k
    e = np.where(codes == 0, 16384, 8192).astype(np.float32)[:, None, None]
    corners = np.array([[-1, -1, -1], [1, 1, 1], [1, -1, -1]], np.float32)
    v = np.zeros((len(codes), 3, 4), np.float32)
    v[:, :, :3] = (c[:, None, :] + 0.5) + e * corners
    f = np.zeros((len(codes), 4), np.uint32)
    f[:, :3] = np.arange(3 * len(codes)).reshape(-1, 3)
    return scenes.Mesh(v.reshape(-1, 4), f)


def test_every_level_is_stacked():
    import torch
    from cudart_b200 import core
    mesh = _mesh()
    tree = core.build_lbvh(torch.from_numpy(mesh.vertices).cuda(), torch.from_numpy(mesh.faces.view(np.int32)).cuda(), hitbox=HIT,
                           tree_depth=32, max_leaf=16)
    info = tree.info_host()
    assert info["error"] == 0 and info["real_depth"] >= 46
    rng = np.random.default_rng(3)
    o, d = np.zeros((96, 4), np.float32), np.zeros((96, 4), np.float32)
    o[:, :3] = (1000, 1000, 500) + rng.uniform(-100, 100, (96, 3))
    d[:, :3] = rng.normal(size=(96, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    o, d = torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda()
    e = core.trace(tree, o, d, schedule=dict(while_while=True))
    assert int(e["err"].item()) == 0 and bool((e["id"] >= 0).any())
    for sch in (None, dict(wide=True), dict(wide=True, while_while=True), dict(coop=True, wide=True),
                dict(coop=True, wide=True, persistent=True), dict(wide=True, while_while=True, persistent=True, treelet=3)):
        h = core.trace(tree, o, d, schedule=sch)
        assert int(h["err"].item()) == 0, sch
        assert torch.equal(h["id"], e["id"]) and torch.equal(h["t"], e["t"]) and torch.equal(h["uv"], e["uv"]), sch
