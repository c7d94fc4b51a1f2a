"""The warp-cooperative walks with few rays, where a group's eight triangles are split among lanes: against the per-lane
walk, for one ray to a warp and one more, over leaves of one to 223 triangles. Exact."""
import numpy as np
import pytest

from cudart_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R", [1, 2, 4, 5, 8, 9, 16, 17, 32, 33])
@pytest.mark.parametrize("mesh", ["one leaf", "odd leaves", "large leaves"])
def test_few_rays(mesh, R):
    import torch
    from cudart_b200 import core
    m = {"one leaf": scenes.soup(13, seed=4), "odd leaves": scenes.soup(3001, seed=5), "large leaves": scenes.soup(6000, seed=6)}[mesh]
    v, f = torch.from_numpy(m.vertices).cuda(), torch.from_numpy(m.faces.view(np.int32)).cuda()
    t = core.build_lbvh(v, f, tree_depth=5 if mesh == "large leaves" else 12, clusters=True)
    o, d = scenes.sphere_rays(m, 40, seed=R)
    for k in range(4):
        oo, dd = (torch.from_numpy(np.ascontiguousarray(x[k * 331:k * 331 + R])).cuda() for x in (o, d))
        want = core.trace(t, oo, dd, schedule=dict(while_while=True))
        for sch in (None, dict(coop=True), dict(coop=True, wide=True), dict(coop=True, persistent=True, clusters=True)):
            h = core.trace(t, oo, dd, schedule=sch)
            assert int(h["err"].cpu()[0]) == 0
            assert torch.equal(h["id"], want["id"]) and torch.equal(h["t"], want["t"]) and torch.equal(h["uv"], want["uv"]), sch
