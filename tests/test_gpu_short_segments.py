"""Builds of few faces, and batches of many small meshes, whose sorts run whole in one CTA, beside longer meshes whose sorts
do not: codes, order, nodes and counters against the CPU oracle. Exact."""
import numpy as np
import pytest

from cudart_b200 import scenes

pytestmark = pytest.mark.gpu


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _mesh(n, seed):
    m = scenes.soup(n, seed=seed)
    if seed % 3 == 0:  # runs of equal codes
        m.vertices[:, :3] = np.round(m.vertices[:, :3] * 3) / 3
    return m


def _ref(oracle, m):
    return oracle.lbvh_build(m.vertices, m.faces, oracle.hitbox(m.vertices))


def _check(ref, codes, indices, nodes, info):
    assert np.array_equal(codes.cpu().numpy().view(np.uint32), ref["codes"])
    assert np.array_equal(indices.cpu().numpy().view(np.uint32), ref["indices"])
    got = info.cpu().tolist()
    assert got == [ref["info"][k] for k in ("node_count", "leaf_count", "real_depth", "split_count", "overrun_visits", "nondet_reads",
                                            "past_end_reads", "error")]
    assert np.array_equal(nodes[:got[0]].cpu().numpy().view(np.uint32), np.ascontiguousarray(ref["nodes"]).view(np.uint32))


@pytest.mark.parametrize("n", [1, 2, 3, 31, 32, 33, 511, 512, 513, 1025, 4095, 4096, 4097])
def test_few_faces(oracle, n):
    from cudart_b200 import core
    for seed in (n, 3 * n):
        m = _mesh(n, seed)
        t = core.build_lbvh(_dev(m.vertices), _dev(m.faces.view(np.int32)))
        _check(_ref(oracle, m), t.codes, t.indices, t.nodes, t.info)


BATCHES = {
    "one window": [1, 2, 300, 17, 5, 1000],
    "4096 faces": [4000, 1, 2, 3, 90],
    "4097 faces": [4000, 1, 2, 3, 91],
    "short and long about the limit": [2047, 2048, 2049, 1, 2050, 2047, 7, 1, 1, 2048] * 3 + [10] * 200,
    "a long one in the middle": [3] * 900 + [20000] + [3] * 900,
    "more segments than a digit holds": [1] * 2500 + [2, 3] * 400 + [2049, 1, 5000, 1],
    "a long one at each end": [9000] + [11] * 700 + [9000],
    "as many as windows": [2048] * 8,
    "one more than windows": [2048] * 7 + [1000, 1048],
}


@pytest.mark.parametrize("name", BATCHES)
def test_batches(oracle, name):
    from cudart_b200 import core
    sizes = BATCHES[name]
    kinds = [_mesh(n, 5 * n + i % 2) for i, n in enumerate(sizes)]
    verts, faces, fo, vo = scenes.concat_batch(kinds)
    t = core.batch_build(_dev(verts), _dev(faces.view(np.int32)), fo, vo)
    refs = {}
    for i, n in enumerate(sizes):
        key = (n, i % 2)
        if key not in refs:
            refs[key] = _ref(oracle, kinds[i])
        s = slice(fo[i], fo[i + 1])
        if i < 40 or i > len(sizes) - 40 or n > 100 or i % 13 == 0:
            _check(refs[key], t.codes[s], t.indices[s], t.mesh_nodes(i, refs[key]["info"]["node_count"]), t.info[i])
