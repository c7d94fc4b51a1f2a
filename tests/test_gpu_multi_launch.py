"""Several products, column sums or optimizer tensors in one launch against the same ones launched singly, bit for bit:
tile counts that differ between the problems, odd columns (which take their own launch), grouped inputs, biases."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("groups", [1, 3])
def test_gemm_and_colsum_multi(groups):
    import torch
    from cudart_b200 import proposal
    g = torch.Generator(device="cuda").manual_seed(groups)

    def rnd(r, c):
        return torch.randn((groups * r, c), generator=g, device="cuda").to(torch.bfloat16)

    shapes = [(128, 16, 64), (384, 208, 128), (128, 128, 1024), (256, 512, 192)]
    ab = [(rnd(m, k), rnd(n, k)) for m, n, k in shapes]
    one = [torch.zeros((groups * m, n), device="cuda") for m, n, _ in shapes]
    many = [torch.zeros_like(x) for x in one]
    for (a, b), c in zip(ab, one):
        proposal.gemm(a, b, out_f32=c, groups=groups)
    proposal.gemm_multi([dict(a=a, b=b, out_f32=c, groups=groups) for (a, b), c in zip(ab, many)])
    for (m, n, k), x, y, (a, b) in zip(shapes, one, many, ab):
        assert torch.equal(x, y)
        want = torch.bmm(a.double().view(groups, m, k), b.double().view(groups, n, k).transpose(1, 2)).view(groups * m, n)
        assert (y.double() - want).abs().max() <= k * 2.0 ** -22 * want.abs().max()  # FP32 sums of exact products
    xs = [rnd(r, c) for r, c in ((1, 2), (255, 64), (256, 66), (257, 33), (2050, 130))]
    one = [torch.zeros(groups * x.shape[1], device="cuda") for x in xs]
    many = [torch.zeros_like(x) for x in one]
    for x, o in zip(xs, one):
        proposal.colsum_grouped(x, groups, o)
    proposal.colsum_multi(list(zip(xs, many)), groups=groups)
    for x, a, b in zip(xs, one, many):
        r = x.shape[0] // groups
        assert torch.equal(a, b)
        want = x.double().view(groups, r, -1).sum(1).view(-1)
        assert (b.double() - want).abs().max() <= r * 2.0 ** -23 * x.double().abs().max()


def test_adam_multi_equals_single_steps():
    import ctypes as C
    import torch
    from cudart_b200 import _abi, core, proposal
    nets = [proposal.ProposalNet(classes=256, seed=5) for _ in range(2)]
    g = torch.Generator(device="cuda").manual_seed(1)
    for _ in range(2):
        for k, gr in enumerate(nets[0].grads):
            gr.copy_(torch.randn(gr.shape, generator=g, device="cuda"))
            nets[1].grads[k].copy_(gr)
        nets[0].adam()
        n = nets[1]
        n.step_count += 1
        for i, (p, gr, m, v) in enumerate(zip(n.params, n.grads, n.m, n.v)):  # one call per tensor
            d = _abi.AdamDesc()
            d.param, d.grad, d.m, d.v = p.data_ptr(), gr.data_ptr(), m.data_ptr(), v.data_ptr()
            d.rows, d.cols = p.shape if p.dim() == 2 else (1, p.shape[0])
            if p.dim() == 2:
                a, t = n.W16[i // 2], n.W16t[i // 2]
                d.out_bf16, d.ld_bf16, d.out_bf16_t, d.ld_bf16_t = a.data_ptr(), a.stride(0), t.data_ptr(), t.stride(0)
            d.lr, d.beta1, d.beta2, d.eps, d.step = 1e-3, 0.9, 0.999, 1e-8, n.step_count
            _abi.check("rt_adam_step", _abi.lib().rt_adam_step(C.byref(d), core._stream()))
    for a, b in zip(nets[0].params + nets[0].m + nets[0].v + nets[0].W16 + nets[0].W16t,
                    nets[1].params + nets[1].m + nets[1].v + nets[1].W16 + nets[1].W16t):
        assert torch.equal(a, b)


@pytest.mark.parametrize("rows", [1, 7, 8, 9, 255, 256, 257, 511, 512, 513, 770, 8192, 10001])
@pytest.mark.parametrize("cols,groups", [(32, 1), (34, 3), (4096, 1), (130, 400)])
def test_colsum_order(rows, cols, groups):
    """Wide and narrow column sums (many and few blocks) add in the order of the one-column kernel, which an odd leading
    dimension takes: the same bits."""
    import torch
    from cudart_b200 import proposal
    if rows * groups > 500000:
        rows = 500000 // groups
    g = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn((groups * rows, cols), device="cuda", generator=g).to(torch.bfloat16)
    odd = torch.zeros((groups * rows, cols + 1), device="cuda", dtype=torch.bfloat16)
    odd[:, :cols] = x
    a, b = torch.empty(groups * cols, device="cuda"), torch.empty(groups * cols, device="cuda")
    proposal.colsum_multi([(x, a)], groups=groups)
    proposal.colsum_multi([(odd[:, :cols], b)], groups=groups)
    assert torch.equal(a.view(torch.int32), b.view(torch.int32))


@pytest.mark.parametrize("rows,classes,groups", [(128, 256, 1), (128, 4096, 1), (384, 1024, 2), (2432, 512, 1), (9472, 512, 1), (9600, 512, 1)])
def test_xent_shares(rows, classes, groups):
    """The gradient's tiles shared out among the CTAs of a row block (few rows: up to 16 shares) against the same rows
    padded to a batch that leaves one share: the same bits, and the loss once."""
    import torch
    from cudart_b200 import proposal
    g = torch.Generator(device="cuda").manual_seed(rows)
    pad = 128 * 160  # more row blocks than SMs: one share
    a = torch.randn((groups, pad, 128), device="cuda", generator=g).to(torch.bfloat16)
    b = torch.randn((groups * classes, 128), device="cuda", generator=g).to(torch.bfloat16)
    bias = torch.randn(groups * classes, device="cuda", generator=g)
    lab = torch.randint(0, classes, (groups, pad), dtype=torch.int32, device="cuda", generator=g)
    got = {}
    for m in (rows, pad):
        x, y = a[:, :m].reshape(groups * m, 128).contiguous(), lab[:, :m].reshape(-1).contiguous()
        out = torch.empty((groups * m, classes), device="cuda", dtype=torch.bfloat16)
        out_t = torch.empty((groups * classes, m), device="cuda", dtype=torch.bfloat16)
        loss, err = torch.zeros(1, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
        proposal.gemm_xent(x, b, bias, y, 1.0 / rows, out, out_t, loss=loss, err=err, groups=groups)
        assert int(err.item()) == 0
        got[m] = out.view(groups, m, classes)[:, :rows], out_t.view(groups, classes, m)[:, :, :rows], loss
    assert torch.equal(got[rows][0].view(torch.int16), got[pad][0].view(torch.int16))
    assert torch.equal(got[rows][1].view(torch.int16), got[pad][1].view(torch.int16))
    logits = (a[:, :rows].double() @ b.view(groups, classes, 128).transpose(1, 2).double()) + bias.view(groups, 1, classes)
    want = torch.nn.functional.cross_entropy(logits.reshape(-1, classes), lab[:, :rows].reshape(-1).long(), reduction="sum") / rows
    # a row's loss holds a handful of float32 roundings and __expf errors of up to 2^-21: 1e-5 of the sum is wide of both
    assert abs(float(got[rows][2]) - float(want)) <= 1e-5 * float(want) + 1e-6
