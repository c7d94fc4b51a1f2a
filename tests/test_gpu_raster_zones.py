"""The rasteriser's zone lists leave out zones that a face's test cannot pass; the surfaces must not change. Triangles
given straight in device coordinates -- slivers with determinants down to the threshold, triangles smaller than a
pixel, larger than the screen (shared by a warp) and with edges through pixel centres -- at screen sizes from one
pixel to ragged zones, in one chunk and in several, against the oracle bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _faces(kind, n, w, h, rng):
    c = rng.uniform(-1.2, 1.2, (n, 1, 2))
    if kind == "slivers":
        d = rng.normal(size=(n, 1, 2))
        p = c + d * rng.uniform(-0.4, 0.4, (n, 3, 1)) + rng.normal(size=(n, 3, 2)) * 10.0 ** rng.uniform(-7, -2, (n, 1, 1))
    elif kind == "tiny":
        p = c + rng.normal(size=(n, 3, 2)) * (1.0 / max(w, h))
    elif kind == "huge":
        p = rng.normal(size=(n, 3, 2)) * 10.0 ** rng.uniform(0, 2.5, (n, 1, 1))
    else:  # corners on pixel positions
        p = np.stack([rng.integers(-2, w + 2, (n, 3)) * 2.0 / w - 1.0, 1.0 - rng.integers(-2, h + 2, (n, 3)) * 2.0 / h], 2)
    v = np.zeros((3 * n, 4), np.float32)
    v[:, :2] = p.reshape(-1, 2)
    v[:, 2] = rng.uniform(0.1, 2.0, 3 * n)
    f = np.zeros((n, 4), np.uint32)
    f[:, :3] = np.arange(3 * n).reshape(n, 3)
    return v, f


@pytest.mark.parametrize("w,h", [(1, 1), (8, 4), (9, 5), (200, 123), (640, 360)])
@pytest.mark.parametrize("kind", ["slivers", "tiny", "huge", "corners"])
def test_zone_lists_change_nothing(oracle, kind, w, h):
    import torch
    from cudart_b200 import core
    rng = np.random.default_rng(w * 7 + len(kind))
    v, f = _faces(kind, 300 if kind == "huge" else 1500, w, h, rng)
    m = np.eye(4, dtype=np.float32).ravel()  # the vertices are device coordinates already
    fo, uo, do = oracle.rasterize(v, f, m, w, h)
    for cap in (0, 1):  # one chunk; chunks of a block of faces
        got = core.rasterize(torch.from_numpy(v).cuda(), torch.from_numpy(f.view(np.int32)).cuda(), m, w, h, pair_capacity=cap)
        torch.cuda.synchronize()
        assert int(got["err"].item()) == 0
        assert np.array_equal(got["depth"].cpu().numpy().view(np.uint32), do.view(np.uint32))
        assert np.array_equal(got["uv"].cpu().numpy().view(np.uint32), uo.view(np.uint32))
        hit = do != oracle.HUGE
        assert np.array_equal(got["id"].cpu().numpy()[hit].view(np.uint32), fo[hit].astype(np.uint32))


@pytest.mark.parametrize("depths", ["equal", "ulps apart", "steep", "wide", "negative", "infinite"])
def test_faces_behind_a_zone_change_nothing(oracle, depths):
    """Many faces over few zones, where the walk leaves out faces behind a zone's farthest depth: ties and near ties by
    index, planes steep enough for their rounding to matter, depths of every magnitude and sign."""
    import torch
    from cudart_b200 import core
    w, h, n = 40, 22, 3000
    rng = np.random.default_rng(len(depths))
    v, f = _faces("corners", n, w, h, rng)
    z = {"equal": lambda: np.full(3 * n, 0.5), "ulps apart": lambda: np.repeat(0.5 + rng.integers(-3, 4, n) * 2.0 ** -24, 3),
         "steep": lambda: np.where(rng.random(3 * n) < 0.3, 1e4, 1.0) * rng.uniform(0.999, 1.001, 3 * n),
         "wide": lambda: 10.0 ** rng.uniform(-30, 30, 3 * n), "negative": lambda: rng.uniform(-1, 0.2, 3 * n),
         "infinite": lambda: np.where(rng.random(3 * n) < 0.01, np.inf, rng.uniform(0.1, 2.0, 3 * n))}[depths]()
    v[:, 2] = z
    m = np.eye(4, dtype=np.float32).ravel()
    with np.errstate(all="ignore"):
        fo, uo, do = oracle.rasterize(v, f, m, w, h)
    for cap in (0, 1):
        got = core.rasterize(torch.from_numpy(v).cuda(), torch.from_numpy(f.view(np.int32)).cuda(), m, w, h, pair_capacity=cap)
        assert np.array_equal(got["id"].cpu().numpy().ravel(), fo.ravel())
        assert np.array_equal(got["depth"].cpu().numpy().ravel().view(np.uint32), do.ravel().view(np.uint32))
        assert np.array_equal(got["uv"].cpu().numpy().ravel().view(np.uint32), uo.ravel().view(np.uint32))
