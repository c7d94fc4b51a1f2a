"""SAH builds at the sizes where a node passes from a warp to a CTA and from a CTA to tiles of several, with last steps and
tiles of one face, and a Hybrid build whose subtrees span all three, against the oracle bit for bit."""
import numpy as np
import pytest

from cudart_b200 import scenes
from tests.test_gpu_sah import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [224, 225, 511, 512, 513, 769, 8191, 8192, 8193, 10241, 40961])
def test_sah_sizes(oracle, n):
    _check(oracle, scenes.soup(n, 60 + n))


def test_hybrid_of_a_big_and_a_small_cluster(oracle):
    big, small = scenes.soup(30000, 7), scenes.soup(300, 8, lo=(4.0, 4.0, 4.0), hi=(4.2, 4.2, 4.2))
    _check(oracle, scenes.concat(big, small), 1)


@pytest.mark.parametrize("n,ratio", [(300, 0.8), (500, 0.9), (3000, 0.99)])
def test_lopsided_trees(oracle, n, ratio):
    """Faces whose sizes and places fall off geometrically: splits peel off a few, so the levels of small nodes run on."""
    m = scenes.soup(n, 70)
    m.vertices[:, :3] *= (ratio ** np.repeat(np.arange(n), 3)).astype(np.float32)[:, None]
    _check(oracle, m)
    _check(oracle, m, 3)
