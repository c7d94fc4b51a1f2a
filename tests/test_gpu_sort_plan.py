"""The chunked radix sort at the sizes where its plan changes (tile sizes, one tile or several per chunk, whole groups of
chunks) and on key distributions that crowd the digit counters, against a stable host sort; and the segmented sort of a
batched build, whose meshes' sizes straddle tiles, chunks and groups, against each mesh's own build. Exact."""
import numpy as np
import pytest

from cudart_b200 import scenes

pytestmark = pytest.mark.gpu


def _keys(kind, n, rng):
    if kind == "random":
        return rng.integers(0, 1 << 32, n, dtype=np.uint32)
    if kind == "constant":
        return np.full(n, 0xABCD1234, np.uint32)
    if kind == "few":
        return rng.choice(np.array([0, 7, 0x80000000, 0xFFFFFFFF], np.uint32), n)
    return np.sort(rng.integers(0, 1 << 32, n, dtype=np.uint32))[::-1].copy()  # descending


@pytest.mark.parametrize("n,kind", [(4097, "random"), (6143, "few"), (6145, "descending"), (32769, "constant"), (606208, "random"),
                                    (606209, "few"), (1818624, "descending"), (1818625, "random"), (2424833, "random"), (4849665, "few")])
def test_sort_sizes(n, kind):
    import torch
    from cudart_b200 import core
    rng = np.random.default_rng(n)
    k = _keys(kind, n, rng)
    v = rng.integers(0, 1 << 32, n, dtype=np.uint32)
    for bits, mode in ((32, "given"), (8, "positions"), (24, "none")):
        masked = k if bits == 32 else k & np.uint32((1 << bits) - 1)
        order = np.argsort(masked, kind="stable")
        kd, vd = torch.from_numpy(k.view(np.int32).copy()).cuda(), torch.from_numpy(v.view(np.int32).copy()).cuda()
        if mode == "none":
            core.sort_keys(kd, bits)
        else:
            core.sort_pairs(kd, vd, bits, init_values=mode == "positions")
        assert np.array_equal(kd.cpu().numpy().view(np.uint32), k[order])
        if mode != "none":
            want = order.astype(np.uint32) if mode == "positions" else v[order]
            assert np.array_equal(vd.cpu().numpy().view(np.uint32), want)


@pytest.mark.parametrize("sizes", [[1, 2, 1], [3] * 300 + [70001, 5], [2047, 2048, 2049, 1, 4096, 33000], [700001, 1, 8193, 16384, 90000]])
def test_batched_segments(sizes):
    import torch
    from cudart_b200 import core
    meshes = [scenes.soup(n, seed=i) for i, n in enumerate(sizes)]
    verts, faces, fo, vo = scenes.concat_batch(meshes)
    t = core.batch_build(torch.from_numpy(verts).cuda(), torch.from_numpy(faces.view(np.int32)).cuda(), fo, vo)
    for m in sorted(set([0, 1, len(sizes) // 2, len(sizes) - 2, len(sizes) - 1])):
        one = core.build_lbvh(torch.from_numpy(meshes[m].vertices).cuda(), torch.from_numpy(meshes[m].faces.view(np.int32)).cuda())
        a, b = fo[m], fo[m + 1]
        assert torch.equal(t.codes[a:b], one.codes) and torch.equal(t.indices[a:b], one.indices) and torch.equal(t.faces[a:b], one.faces)
        info = one.info_host()
        assert torch.equal(t.info[m], one.info)
        assert torch.equal(t.mesh_nodes(m, info["node_count"]), one.nodes[:info["node_count"]])
