"""What the packet walk counts for a ray: the boxes and triangles that the ray wants itself, whatever its warp visits."""
import numpy as np
import pytest

from cudart_b200 import scenes

pytestmark = pytest.mark.gpu


def _run(tree, o, d, tmax=None, **schedule):
    import torch
    from cudart_b200 import core
    h = core.trace(tree, torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda(), tmax=None if tmax is None else torch.from_numpy(tmax).cuda(),
                   counters=True, schedule=dict(clusters=True, persistent=True, blocks_per_sm=8, **schedule))
    return {k: h[k].cpu().numpy() for k in ("id", "visits", "tests")}


def test_counts_are_the_rays_own():
    import torch
    from cudart_b200 import core
    mesh = scenes.soup(20000, seed=4)
    tree = core.build_lbvh(torch.from_numpy(mesh.vertices).cuda(), torch.from_numpy(mesh.faces.view(np.int32)).cuda(), clusters=True)
    o, d = scenes.sphere_rays(mesh, 64, seed=6)
    away = np.arange(len(o)) % 5 == 0
    d[away] = o[away] - 0.5  # from the sphere around the mesh outwards
    d[away, 3] = 0
    p = _run(tree, o, d, packet=True)
    lane = _run(tree, o, d)
    assert np.array_equal(p["id"], lane["id"])
    hit = p["id"] >= 0  # a miss prunes nothing, so that its counts do not depend on the order of the walk
    assert not hit[away].any()
    for k in ("visits", "tests"):
        assert np.array_equal(p[k][~hit], lane[k][~hit])
    assert hit.any() and (p["tests"][hit] >= 1).all()
    # one live ray per warp: the ray's own walk
    tmax = np.full(len(o), -1.0, np.float32)
    tmax[::32] = 3.402823466e38
    one = _run(tree, o, d, tmax, packet=True)
    own = _run(tree, o, d, tmax)
    for k in ("visits", "tests"):
        assert (one[k][tmax < 0] == 0).all()
        assert abs(int(one[k].sum()) - int(own[k].sum())) <= 0.02 * int(own[k].sum())  # the packet orders near-equal distances its own way
