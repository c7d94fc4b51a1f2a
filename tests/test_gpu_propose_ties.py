"""The fused proposal's top-1 sweep (16 logits compared at a time, the column looked up per tile) where columns tie or are
extreme: the logits are the biases (zero weights), so the winner is the first column holding the largest bias. Exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bias(kind, n):
    b = np.linspace(-1, 1, n, dtype=np.float32)[np.random.default_rng(n).permutation(n)]
    if kind == "all equal":
        b[:] = 0.25
    elif kind == "inside a group":
        b[[35, 36, 47]] = 2.0
    elif kind == "across groups":
        b[[47, 48, n - 1]] = 2.0
    elif kind == "across tiles":
        b[[n // 2 - 1, n // 2]] = 2.0
    elif kind == "last":
        b[n - 1] = 2.0
    elif kind == "ascending":
        b.sort()
    elif kind == "lowest":
        b[:] = np.finfo(np.float32).min
    elif kind == "infinite":
        b[:] = -np.inf
        b[[200, 213]] = np.inf
    elif kind == "one finite":
        b[:] = -np.inf
        b[77] = -3.0
    return b


@pytest.mark.parametrize("classes", [256, 4096])
@pytest.mark.parametrize("kind", ["all equal", "inside a group", "across groups", "across tiles", "last", "ascending", "lowest",
                                  "infinite", "one finite"])
def test_ties(classes, kind):
    import torch
    from cudart_b200 import proposal as P
    net = P.ProposalNet(classes=classes, seed=1)
    net.W16[3].zero_()
    bias = _bias(kind, classes)
    net.b[3].copy_(torch.from_numpy(bias))
    R = 128 * 3 + 5
    g = torch.Generator(device="cuda").manual_seed(2)
    o, d = torch.rand((R, 4), device="cuda", generator=g), torch.rand((R, 4), device="cuda", generator=g) + 0.1
    box = (0.0, 0.0, 0.0, 1.0, 1.0, 1.0)
    a = net.propose(o, d, box, fused=True)
    b = net.propose(o, d, box, fused=False)
    assert int(net.err.item()) == 0
    if kind == "infinite":  # the layered path always takes the margin, which is NaN here, and makes no proposal
        assert (b == -1).all()
    else:
        assert torch.equal(a, b)
    assert (a == int(np.argmax(bias))).all()
