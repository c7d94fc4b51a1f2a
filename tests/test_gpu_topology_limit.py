"""Batched meshes whose Morton nodes just fit the 2560 that a mesh's CTA holds in shared memory, or just do not, many of
them side by side and again and again: all threads of a CTA have to agree on which of the two it is, at the same level.
Nodes, counters and faces against the CPU oracle. Exact."""
import numpy as np
import pytest

from cudart_b200 import scenes

PER_CELL = 15  # faces of a cell: below the 16 that a node needs to be split, two cells above it


def cells_mesh(cells, seed):
    """PER_CELL small triangles in each of `cells` cells: the 1024 of ten Morton levels, as many of them cut once more as it
    takes (2 * cells - 1 nodes; 1024 to 2048 cells)."""
    rng = np.random.default_rng(seed)
    code = np.concatenate([np.arange(1024) * 2, rng.choice(1024, cells - 1024, replace=False) * 2 + 1]).astype(np.int64) << 21
    q = np.zeros((cells, 3), np.float32)
    for k in range(11):
        q[:, 1] += ((code >> (3 * k)) & 1) << k
        q[:, 0] += ((code >> (3 * k + 1)) & 1) << k
        if k < 10:
            q[:, 2] += ((code >> (3 * k + 2)) & 1) << k
    c = np.repeat(q, PER_CELL, 0)[:, None, :] + 0.5
    tri = c + rng.uniform(-0.2, 0.2, (cells * PER_CELL, 3, 3))
    v = np.zeros((3 * cells * PER_CELL + 2, 4), np.float32)
    v[:-2, :3] = tri.reshape(-1, 3)
    v[-1, :3] = 2047, 2047, 1023  # with the zero before it the hit box: codes are the coordinates
    f = np.zeros((cells * PER_CELL, 4), np.uint32)
    f[:, :3] = np.arange(3 * cells * PER_CELL).reshape(-1, 3)
    return scenes.Mesh(v, f)


def _oracle(oracle, m):
    return oracle.lbvh_build(m.vertices, m.faces, oracle.hitbox(m.vertices))


@pytest.mark.parametrize("cells", [1279, 1280, 1281])
def test_cells_mesh_has_the_nodes_it_says(oracle, cells):
    info = _oracle(oracle, cells_mesh(cells, cells))["info"]
    assert info["node_count"] == 2 * cells - 1


@pytest.mark.gpu
def test_nodes_around_the_limit(oracle):
    import torch
    from cudart_b200 import core
    kinds = {cells: cells_mesh(cells, cells) for cells in (1280, 1281, 1282, 2000, 2048, 1279)}
    order = [list(kinds)[i % len(kinds)] for i in range(60)]
    verts, faces, fo, vo = scenes.concat_batch([kinds[c] for c in order])
    v, f = torch.from_numpy(verts).cuda(), torch.from_numpy(faces.view(np.int32)).cuda()
    ref = {c: _oracle(oracle, m) for c, m in kinds.items()}
    nodes = {c: torch.from_numpy(np.ascontiguousarray(r["nodes"]).view(np.int32)).cuda() for c, r in ref.items()}
    for _ in range(20):
        t = core.batch_build(v, f, fo, vo)
        info = t.info.cpu().numpy()
        for i, c in enumerate(order):
            got = dict(zip(("node_count", "leaf_count", "real_depth", "split_count", "overrun_visits", "nondet_reads", "past_end_reads",
                            "error"), info[i].tolist()))
            assert got["error"] == 0
            assert all(got[k] == ref[c]["info"][k] for k in got if k != "error"), (c, got)
            assert torch.equal(t.mesh_nodes(i, 2 * c - 1), nodes[c].view(-1, 8))
