"""A trace that asks for no schedule (the warp-cooperative walk of the 4-wide records) against the oracle, bit for
bit: leaves at the sizes where groups and leaves split, ray counts around a warp and a CTA, image tiles with ragged
edges, tmax cut-offs, original face ids, and rays that start on a triangle's plane, whose t is a zero of either sign
(every schedule, since the merge of the lanes' hits orders t by its bits)."""
import numpy as np
import pytest

from cudart_b200 import scenes

pytestmark = pytest.mark.gpu


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _check(oracle, mesh, o, d, tmax=None, id_mode=0, schedules=(None,), clusters=False):
    import torch
    from cudart_b200 import core
    tree = core.build_lbvh(_dev(mesh.vertices), _dev(mesh.faces.view(np.int32)), clusters=clusters)
    ref = oracle.lbvh_build(mesh.vertices, mesh.faces, oracle.hitbox(mesh.vertices))
    e = oracle.trace(ref["nodes"], ref["tris"], ref["indices"], o, d, tmax, mode=0, id_mode=id_mode)
    for sch in schedules:
        out = core.trace(tree, _dev(o), _dev(d), tmax=None if tmax is None else _dev(tmax), id_mode=id_mode, schedule=sch)
        torch.cuda.synchronize()
        assert int(out["err"].item()) == 0
        assert np.array_equal(out["id"].cpu().numpy(), e["id"]), sch
        assert np.array_equal(out["t"].cpu().numpy().view(np.uint32), e["t"].view(np.uint32)), sch
        assert np.array_equal(out["uv"].cpu().numpy().view(np.uint32), e["uv"].view(np.uint32)), sch
    return e


@pytest.mark.parametrize("n", [1, 7, 8, 9, 223, 224, 225, 257, 4097, 70001])
def test_default_walk_mesh_sizes(oracle, n):
    mesh = scenes.soup(n, seed=900 + n)
    o, d = scenes.sphere_rays(mesh, 47, seed=n)
    tmax = np.full(o.shape[0], 3.402823466e38, np.float32)
    tmax[::5], tmax[::17], tmax[::19] = 0.4, 0.0, -1.0
    _check(oracle, mesh, o, d)
    _check(oracle, mesh, o, d, tmax, id_mode=1)


@pytest.mark.parametrize("rays", [1, 31, 32, 33, 127, 128, 129])
def test_default_walk_ray_counts(oracle, rays):
    mesh = scenes.terrain(40, seed=3)
    o, d = scenes.sphere_rays(mesh, 12, seed=rays)
    _check(oracle, mesh, o[:rays], d[:rays], schedules=(None, dict(image_width=rays), dict(image_width=1)))


def test_rays_starting_on_triangles(oracle):
    """A flat grid of triangles in z = 0 and copies of it: origins in the plane, directions to either side, so that
    hits at t = +0 and t = -0 (and ties between copies) decide."""
    g = scenes.terrain(17, seed=1, amplitude=0.0)
    v = g.vertices.copy()
    v[:, [1, 2]] = v[:, [2, 1]]
    f = np.concatenate([g.faces, g.faces[::-1], g.faces[:, [1, 0, 2, 3]]])
    mesh = scenes.Mesh(v, f)
    rng = np.random.default_rng(5)
    o = np.zeros((640, 4), np.float32)
    d = np.zeros((640, 4), np.float32)
    o[:, :2] = rng.uniform(-0.9, 0.9, (640, 2))
    d[:, :3] = rng.normal(size=(640, 3))
    o[::3, 2] = -0.0
    schedules = [None, dict(while_while=True), dict(wide=True), dict(coop=True), dict(coop=True, wide=True, persistent=True),
                 dict(clusters=True), dict(clusters=True, persistent=True, coop=True), dict(clusters=True, persistent=True, packet=True),
                 dict(clusters=True, persistent=True, packet=True, lane_threshold=16),
                 dict(clusters=True, persistent=True, refill=True, lane_threshold=8)]
    e = _check(oracle, mesh, o, d, schedules=schedules, clusters=True)
    zero = e["t"][e["id"] >= 0] == 0.0
    assert zero.any() and np.signbit(e["t"][e["id"] >= 0][zero]).any()
