"""A SAH build into the buffers of an LBVH build with a cluster tree: the blob holds no cluster tree any more."""
import numpy as np
import pytest

from cudart_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("depth", [0, 6])
def test_old_cluster_tree_is_gone(depth):
    import torch
    from cudart_b200 import _abi, core
    a, b = scenes.soup(3000, seed=1), scenes.soup(3000, seed=2)
    f = torch.from_numpy(a.faces.view(np.int32)).cuda()
    o, d = (torch.from_numpy(x).cuda() for x in scenes.sphere_rays(a, 24, seed=3))
    nodes = core.sah_sizes(3000, depth)[1]
    t = core.build_lbvh(torch.from_numpy(a.vertices).cuda(), f, clusters=True)
    t.nodes = torch.zeros((nodes, 8), dtype=torch.int32, device="cuda")
    t = core.build_lbvh(torch.from_numpy(a.vertices).cuda(), f, clusters=True, out=t)
    assert int(core.trace(t, o, d, schedule=dict(clusters=True))["err"].item()) == 0
    t = core.build_sah(torch.from_numpy(b.vertices).cuda(), f, lbvh_depth=depth, out=t)
    assert not t.clusters
    plain = core.trace(t, o, d)
    assert int(plain["err"].item()) == 0 and bool((plain["id"] >= 0).any())
    for sch in (dict(clusters=True), dict(clusters=True, persistent=True, packet=True), dict(clusters=True, persistent=True, refill=True)):
        h = core.trace(t, o, d, schedule=sch)
        assert int(h["err"].item()) & _abi.DEVERR_ACCEL_MISSING, sch
        assert bool((h["id"] == -1).all()), sch
