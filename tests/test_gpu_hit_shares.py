"""The batched hit box in one to eight shares a mesh, around the vertex and mesh counts where their number changes: the
codes and order of every mesh against its own build. Exact."""
import numpy as np
import pytest

from cudart_b200 import scenes

pytestmark = pytest.mark.gpu


def _mesh(verts, seed):
    """A small soup with its vertices scattered among unused ones that reach farther out."""
    rng = np.random.default_rng(seed)
    n = max(1, min(40, verts // 3))
    v = np.zeros((verts, 4), np.float32)
    v[:, :3] = rng.uniform(-1, 1, (verts, 3)) * rng.uniform(0.5, 3, 3)
    f = np.zeros((n, 4), np.uint32)
    f[:, :3] = rng.integers(0, verts, (n, 3))
    return scenes.Mesh(v, f)


@pytest.mark.parametrize("meshes,verts", [(1, 1), (1, 2047), (1, 2048), (2, 4095), (2, 4096), (2, 8191), (2, 8192), (3, 20000), (74, 2048), (75, 2048),
                                          (75, 16383), (75, 16384), (75, 32768), (75, 65536), (600, 5)])
def test_shares(meshes, verts):
    import torch
    from cudart_b200 import core
    kinds = [_mesh(verts, s) for s in range(min(meshes, 7))]
    all_ = [kinds[i % len(kinds)] for i in range(meshes)]
    v, f, fo, vo = scenes.concat_batch(all_)
    t = core.batch_build(torch.from_numpy(v).cuda(), torch.from_numpy(f.view(np.int32)).cuda(), fo, vo)
    own = [core.build_lbvh(torch.from_numpy(k.vertices).cuda(), torch.from_numpy(k.faces.view(np.int32)).cuda()) for k in kinds]
    for i in range(meshes):
        o = own[i % len(kinds)]
        assert torch.equal(t.codes[fo[i]:fo[i + 1]], o.codes) and torch.equal(t.indices[fo[i]:fo[i + 1]], o.indices)
