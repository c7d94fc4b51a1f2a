"""Frames without a single (zone, face) pair, or with one: the surfaces against the oracle, bit for bit, over surfaces that
hold something already."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["off the screen", "too fine", "one pixel"])
@pytest.mark.parametrize("n", [1, 129, 5000])
def test_no_pairs(oracle, kind, n):
    import torch
    from cudart_b200 import core
    w, h = 70, 50
    rng = np.random.default_rng(n)
    v = np.zeros((3 * n, 4), np.float32)
    v[:, :2] = rng.uniform(-1, 1, (3 * n, 2)) * 1e-5  # determinants of about 1e-10
    v[:, 2] = 0.5
    if kind == "off the screen":
        v[:, :2] = rng.uniform(2, 3, (3 * n, 2))
    f = np.zeros((n, 4), np.uint32)
    f[:, :3] = np.arange(3 * n).reshape(n, 3)
    if kind == "one pixel":
        v[:3, :3] = [[-0.01, -0.01, 0.1], [0.03, -0.01, 0.1], [-0.01, 0.03, 0.1]]
    m = np.eye(4, dtype=np.float32).ravel()
    fid, uv, dep = rng.integers(0, 9, w * h).astype(np.uint32), rng.random((w * h, 2)).astype(np.float32), rng.uniform(0.3, 0.7, w * h).astype(np.float32)
    e = oracle.rasterize(v, f, m, w, h, fid, uv, dep)
    assert (kind == "one pixel") == bool((e[2] != dep).any())
    out = dict(id=torch.from_numpy(fid.view(np.int32)).cuda(), uv=torch.from_numpy(uv).cuda(), depth=torch.from_numpy(dep).cuda(),
               err=torch.zeros(1, dtype=torch.int32, device="cuda"))
    for cap in (0, 1):
        got = core.rasterize(torch.from_numpy(v).cuda(), torch.from_numpy(f.view(np.int32)).cuda(), m, w, h, pair_capacity=cap, out=out)
        for x, y in zip((got["id"], got["uv"], got["depth"]), e):
            assert np.array_equal(x.cpu().numpy().view(np.uint32), y.view(np.uint32))
