"""Sorts of few chunks, whose CTAs count the keys themselves, around the sizes where that begins and ends: against torch's
stable sort. Exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4097, 6143, 6145, 16383, 16384, 16385, 24575, 24576, 24577, 32769])
@pytest.mark.parametrize("values", ["random", "equal", "few", "descending"])
def test_against_torch(n, values):
    import torch
    from cudart_b200 import core
    rng = np.random.default_rng(n)
    keys = {"random": rng.integers(0, 1 << 32, n, dtype=np.uint64), "equal": np.full(n, 0xFFFFFFFF, np.uint64),
            "few": rng.integers(0, 3, n, dtype=np.uint64) << 13, "descending": np.arange(n, 0, -1, dtype=np.uint64) * 977}[values]
    keys = (keys & 0xFFFFFFFF).astype(np.uint32)
    for bits in (8, 24, 32):
        k = keys if bits == 32 else keys & np.uint32((1 << bits) - 1)
        order = np.argsort(k, kind="stable")
        given = rng.integers(0, 1 << 31, n).astype(np.int32)
        for vals in (None, given):
            a, w = torch.from_numpy(k.view(np.int32).copy()).cuda(), torch.from_numpy(given.copy()).cuda()
            core.sort_pairs(a, w, bits, init_values=vals is None)
            assert np.array_equal(a.cpu().numpy().view(np.uint32), k[order])
            assert np.array_equal(w.cpu().numpy(), order.astype(np.int32) if vals is None else given[order])
        a = torch.from_numpy(k.view(np.int32).copy()).cuda()
        core.sort_keys(a, bits)
        assert np.array_equal(a.cpu().numpy().view(np.uint32), k[order])


@pytest.mark.parametrize("n", [4097, 16384, 16385, 24576, 24577])
def test_builds(oracle, n):
    import torch
    from cudart_b200 import core, scenes
    m = scenes.soup(n, seed=n)
    t = core.build_lbvh(torch.from_numpy(m.vertices).cuda(), torch.from_numpy(m.faces.view(np.int32)).cuda())
    ref = oracle.lbvh_build(m.vertices, m.faces, oracle.hitbox(m.vertices))
    assert np.array_equal(t.codes.cpu().numpy().view(np.uint32), ref["codes"])
    assert np.array_equal(t.indices.cpu().numpy().view(np.uint32), ref["indices"])
    assert np.array_equal(t.nodes_host().numpy().view(np.uint32), np.ascontiguousarray(ref["nodes"]).view(np.uint32))
