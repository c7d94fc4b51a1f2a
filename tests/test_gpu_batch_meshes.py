"""A batched build with more meshes than warps have lanes and sizes from one face up: every mesh's nodes, triangles and
hits against its own build, with and without cluster trees. Exact."""
import numpy as np
import pytest

from cudart_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("clusters", [False, True])
@pytest.mark.parametrize("sizes", [[1] * 65, [1, 2, 3, 1] * 150 + [4099] + [1] * 33 + [257, 2], [256, 255, 257, 511, 513, 1, 1, 31, 33]])
def test_uneven_meshes(sizes, clusters):
    import torch
    from cudart_b200 import core
    meshes = [scenes.soup(n, seed=i) for i, n in enumerate(sizes)]
    verts, faces, fo, vo = scenes.concat_batch(meshes)
    t = core.batch_build(torch.from_numpy(verts).cuda(), torch.from_numpy(faces.view(np.int32)).cuda(), fo, vo, clusters=clusters)
    rays = [scenes.sphere_rays(m, 4, seed=i) for i, m in enumerate(meshes)]
    ro = np.concatenate([[0], np.cumsum([len(o) for o, _ in rays])]).astype(np.int32)
    O, D = (torch.from_numpy(np.concatenate([r[k] for r in rays])).cuda() for k in (0, 1))
    hits = core.batch_trace(t, O, D, torch.from_numpy(ro).cuda(), schedule=dict(clusters=True) if clusters else None)
    assert int(hits["err"].cpu()[0]) == 0
    for m in range(0, len(sizes), max(1, len(sizes) // 40)):
        one = core.build_lbvh(torch.from_numpy(meshes[m].vertices).cuda(), torch.from_numpy(meshes[m].faces.view(np.int32)).cuda(),
                              clusters=clusters)
        nc = one.info_host()["node_count"]
        assert torch.equal(t.info[m], one.info)
        assert torch.equal(t.mesh_nodes(m, nc), one.nodes[:nc])
        assert torch.equal(t.boxes[fo[m]:fo[m + 1]], one.boxes) and torch.equal(t.tris[fo[m]:fo[m + 1]], one.tris)
        s = slice(int(ro[m]), int(ro[m + 1]))
        h = core.trace(one, O[s], D[s], schedule=dict(clusters=True) if clusters else None)
        assert torch.equal(h["id"], hits["id"][s]) and torch.equal(h["t"], hits["t"][s])


@pytest.mark.parametrize("count", [511, 513])
def test_hit_box_shares(count):
    """The batched hit box in eight shares per mesh and in four (many meshes), down to fewer vertices than shares: the
    codes of every mesh against its own build."""
    import torch
    from cudart_b200 import core
    meshes = [scenes.soup(1 + (i * 37) % 29, seed=i) for i in range(count - 1)] + [scenes.soup(9001, seed=7)]
    verts, faces, fo, vo = scenes.concat_batch(meshes)
    t = core.batch_build(torch.from_numpy(verts).cuda(), torch.from_numpy(faces.view(np.int32)).cuda(), fo, vo)
    for m in list(range(0, count - 1, 17)) + [count - 1]:
        one = core.build_lbvh(torch.from_numpy(meshes[m].vertices).cuda(), torch.from_numpy(meshes[m].faces.view(np.int32)).cuda())
        assert torch.equal(t.codes[fo[m]:fo[m + 1]], one.codes) and torch.equal(t.indices[fo[m]:fo[m + 1]], one.indices)
