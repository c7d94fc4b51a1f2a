"""The cluster tree at the edges of its chunks (512 positions; one, few and hundreds of them), with ordinary, constant (all codes equal) and skewed Morton codes: closest hits against the node tree's. Exact."""
import numpy as np
import pytest

from cudart_b200 import scenes

pytestmark = pytest.mark.gpu


def _mesh(kind, n):
    m = scenes.soup(n, seed=n)
    if kind == "equal":  # every face the same triangle: one Morton code, ties by position
        m.vertices[:, :3] = np.tile(m.vertices[:3, :3], (m.vertices.shape[0] // 3, 1))
    elif kind == "skewed":  # most faces in one cell
        k = m.vertices.shape[0] // 3 * 2 // 3 * 3
        m.vertices[:k, :3] *= np.float32(1e-3)
    return m


@pytest.mark.parametrize("kind", ["soup", "equal", "skewed"])
@pytest.mark.parametrize("n", [511, 513, 1025, 126 * 512 - 1, 127 * 512, 128 * 512 + 1, 300 * 512 + 77])
def test_chunk_edges(n, kind):
    import torch
    from cudart_b200 import core
    m = _mesh(kind, n)
    t = core.build_lbvh(torch.from_numpy(m.vertices).cuda(), torch.from_numpy(m.faces.view(np.int32)).cuda(), clusters=True)
    o, d = scenes.sphere_rays(m, 24, seed=3)
    o, d = torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda()
    a, b = core.trace(t, o, d), core.trace(t, o, d, schedule=dict(clusters=True))
    assert int(a["err"].cpu()[0]) == 0 and int(b["err"].cpu()[0]) == 0
    assert torch.equal(a["id"], b["id"]) and torch.equal(a["t"], b["t"]) and torch.equal(a["uv"], b["uv"])


@pytest.mark.parametrize("sizes", [[126 * 512, 5, 40000, 128 * 512 + 1], [1] * 127 + [1300, 70000, 1, 513]])
def test_batched_chunks(sizes):
    import torch
    from cudart_b200 import core
    meshes = [_mesh("skewed" if i % 2 else "soup", n) for i, n in enumerate(sizes)]
    verts, faces, fo, vo = scenes.concat_batch(meshes)
    t = core.batch_build(torch.from_numpy(verts).cuda(), torch.from_numpy(faces.view(np.int32)).cuda(), fo, vo, clusters=True)
    rays = [scenes.sphere_rays(m, 12, seed=i) for i, m in enumerate(meshes)]
    ro = torch.from_numpy(np.concatenate([[0], np.cumsum([len(r[0]) for r in rays])]).astype(np.int32)).cuda()
    o, d = (torch.from_numpy(np.concatenate([r[k] for r in rays])).cuda() for k in (0, 1))
    a, b = core.batch_trace(t, o, d, ro), core.batch_trace(t, o, d, ro, schedule=dict(clusters=True))
    assert int(a["err"].cpu()[0]) == 0 and int(b["err"].cpu()[0]) == 0
    assert torch.equal(a["id"], b["id"]) and torch.equal(a["t"], b["t"]) and torch.equal(a["uv"], b["uv"])
