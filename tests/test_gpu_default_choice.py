"""What a trace without a schedule chooses, at the edges of its rules and on rays that agree: hits against the oracle and
counts against the walk that the header names, bit for bit."""
import numpy as np
import pytest

from cudart_b200 import scenes

pytestmark = pytest.mark.gpu


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _same(out, e, what):
    assert int(out["err"].item()) == 0
    for k in ("id", "t", "uv"):
        assert np.array_equal(out[k].cpu().numpy().view(np.uint32), e[k].view(np.uint32)), (what, k)


def _setup(oracle, mesh, depth=12):
    from cudart_b200 import core
    tree = core.build_lbvh(_dev(mesh.vertices), _dev(mesh.faces.view(np.int32)), tree_depth=depth)
    return tree, oracle.lbvh_build(mesh.vertices, mesh.faces, oracle.hitbox(mesh.vertices), tree_depth=depth)


def _camera(width, height, center=(0.5, 0.5, -0.4)):
    from cudart_b200 import core
    o, d = core.primary_rays(core.make_camera(center, (0.5, 0.5, 0.5), fov=scenes.FOV_60, ratio=width / height), width, height)
    return o, d, o.cpu().numpy(), d.cpu().numpy()


@pytest.mark.parametrize("width,height", [(48, 39), (48, 40), (8, 999), (8, 1000), (7999, 1), (8001, 1)])
def test_many_rays_a_triangle(oracle, width, height):
    """20 triangles: per lane from 96 rays each in tiles (1920) and from 400 in rows (8000), without a tmax."""
    from cudart_b200 import core
    tree, ref = _setup(oracle, scenes.soup(20, seed=8))
    o, d, oh, dh = _camera(width, height)
    tmax = np.full(width * height, 0.7, np.float32)
    for tm in (None, tmax):
        e = oracle.trace(ref["nodes"], ref["tris"], ref["indices"], oh, dh, tm, mode=0)
        for sch in (None, dict(image_width=width), dict(per_lane=True), dict(per_lane=True, image_width=width)):
            _same(core.trace(tree, o, d, tmax=None if tm is None else _dev(tm), schedule=sch), e, (sch, tm is None))


@pytest.mark.parametrize("depth", [1, 3, 6, 12])
@pytest.mark.parametrize("coop", [None, dict(coop=True), dict(coop=True, wide=True, persistent=True)])
def test_rays_that_agree(oracle, depth, coop):
    """Warps whose rays want the same groups of large leaves, some of them, or none: a camera close by and far off, rays
    that are all alike, and alike but for one."""
    from cudart_b200 import core
    mesh = scenes.soup(6000, seed=3)
    tree, ref = _setup(oracle, mesh, depth)
    for center in ((0.5, 0.5, -0.4), (0.5, 0.5, 0.45), (0.5, 0.5, -20.0)):
        o, d, oh, dh = _camera(72, 44, center)
        e = oracle.trace(ref["nodes"], ref["tris"], ref["indices"], oh, dh, None, mode=0)
        for sch in (coop, dict(coop or {}, image_width=72)):
            _same(core.trace(tree, o, d, schedule=sch), e, (center, sch))
    oh, dh = (np.repeat(a[:8], 40, 0) for a in scenes.sphere_rays(mesh, 8, seed=2))
    oh[7::64], dh[7::64] = (a[20:25] for a in scenes.sphere_rays(mesh, 8, seed=4))
    e = oracle.trace(ref["nodes"], ref["tris"], ref["indices"], oh, dh, None, mode=0)
    _same(core.trace(tree, _dev(oh), _dev(dh), schedule=coop), e, "alike")


def test_counts_of_the_default_are_the_per_lane_walks():
    from cudart_b200 import core
    mesh = scenes.soup(6000, seed=3)
    tree = core.build_lbvh(_dev(mesh.vertices), _dev(mesh.faces.view(np.int32)))
    o, d = (_dev(a) for a in scenes.sphere_rays(mesh, 32, seed=2))
    a, b = core.trace(tree, o, d, counters=True), core.trace(tree, o, d, counters=True, schedule=dict(per_lane=True))
    for k in ("id", "t", "visits", "tests"):
        assert (a[k] == b[k]).all(), k
