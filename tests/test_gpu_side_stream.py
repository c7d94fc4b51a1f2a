"""Builds and the rasteriser fork part of their work onto a stream that belongs to the host thread. While a call of the same
thread is being captured, calls on other streams have to leave that capture alone."""
import numpy as np
import pytest

from cudart_b200 import scenes

pytestmark = pytest.mark.gpu


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _cat(meshes):
    v, f, fo, vo = scenes.concat_batch(meshes)
    return _dev(v), _dev(f.view(np.int32)), fo, vo


def test_calls_beside_a_capture():
    import torch
    from cudart_b200 import core
    a, b = scenes.soup(5000, seed=1), scenes.soup(7000, seed=2)
    av, af, bv, bf = _dev(a.vertices), _dev(a.faces.view(np.int32)), _dev(b.vertices), _dev(b.faces.view(np.int32))
    cam = core.make_camera((0.55, 0.6, -0.4), (0.5, 0.5, 0.5), fov=scenes.FOV_60, ratio=1.5)
    matrix = core.raster_matrix(cam, (0.5, 0.5, 0.5))
    batch = _cat([scenes.soup(300, seed=3), scenes.soup(900, seed=4)])

    def others(tree, many, image):
        core.build_lbvh(bv, bf, out=tree, clusters=True)
        core.batch_build(*batch, out=many, clusters=True)
        image["id"].zero_(), image["uv"].zero_(), image["depth"].fill_(core.HUGE)
        core.rasterize(bv, bf, matrix, 96, 64, out=image)

    # what the calls give by themselves; every buffer and the scratch exist before the capture
    want = core.build_lbvh(av, af, clusters=True)
    tree, many, image = core.build_lbvh(bv, bf, clusters=True), core.batch_build(*batch, clusters=True), core.rasterize(bv, bf, matrix, 96, 64)
    expect = [x.clone() for x in (tree.nodes[:tree.node_count], tree.accel, many.tris, image["id"], image["depth"])]
    mine = core.build_lbvh(av, af, clusters=True)
    torch.cuda.synchronize()
    s, t = torch.cuda.Stream(), torch.cuda.Stream()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s, capture_error_mode="relaxed"):
        core.build_lbvh(av, af, out=mine, clusters=True)
        with torch.cuda.stream(t):
            others(tree, many, image)
        core.build_lbvh(av, af, out=mine, clusters=True)  # the capture still has its side branch
    t.synchronize()
    mine.nodes.zero_()
    g.replay()
    torch.cuda.synchronize()
    n = want.node_count
    assert torch.equal(mine.nodes[:n], want.nodes[:n]) and torch.equal(mine.tris, want.tris)
    got = (tree.nodes[:tree.node_count], many.tris, image["id"], image["depth"])
    for x, y in zip(got, (expect[0], expect[2], expect[3], expect[4])):
        assert torch.equal(x, y)
    with torch.cuda.stream(t):
        others(tree, many, image)
    torch.cuda.synchronize()
    assert torch.equal(tree.nodes[:tree.node_count], expect[0]) and torch.equal(image["id"], expect[3])
