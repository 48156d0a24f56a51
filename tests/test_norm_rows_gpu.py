"""Norms at the edges of what a warp, a lane and a CTA take, against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rms", [False, True])
@pytest.mark.parametrize("rows,cols,dtype", [
    (1, 8, torch.bfloat16), (3, 256, torch.float16), (5, 264, torch.bfloat16), (4097, 512, torch.bfloat16), (601, 520, torch.float16), (7, 768, torch.bfloat16),
    (1187, 776, torch.bfloat16), (9, 1024, torch.float16), (595, 1032, torch.bfloat16), (300, 2048, torch.bfloat16), (297, 2056, torch.float16),
    (2, 4096, torch.bfloat16), (149, 4104, torch.bfloat16), (151, 8192, torch.float16), (1, 8184, torch.bfloat16)])
def test_norm(rows, cols, dtype, rms):
    from megatronapp_b200 import ops

    g = torch.Generator("cuda").manual_seed(rows + cols)
    rnd = lambda *n: torch.randn(*n, generator=g, device="cuda")  # noqa: E731
    ins = [(3 + rnd(rows, cols)).to(dtype), (1 + 0.1 * rnd(cols)).to(dtype)] + ([] if rms else [(0.1 * rnd(cols)).to(dtype)])
    dy = rnd(rows, cols).to(dtype)
    for zero_centered in (False, True):
        own, wide = ([t.detach().to(d or dtype).requires_grad_() for t in ins] for d in (None, torch.float64))
        y = ops.layer_norm(own[0], own[1], None if rms else own[2], 1e-5, rms=rms, zero_centered=zero_centered)
        x, w = wide[0], wide[1] + 1 if zero_centered else wide[1]
        mu = 0 if rms else x.mean(-1, keepdim=True)
        want = (x - mu) * torch.rsqrt((x - mu).pow(2).mean(-1, keepdim=True) + 1e-5) * w
        want = want if rms else want + wide[2]
        got = [y, *torch.autograd.grad(y, own, dy)]
        again = torch.autograd.grad(ops.layer_norm(own[0], own[1], None if rms else own[2], 1e-5, rms=rms, zero_centered=zero_centered), own, dy)
        for i, (a, b) in enumerate(zip(got, [want, *torch.autograd.grad(want, wide, dy.double())])):
            # half a unit of the result's type: 2^-8 of a value of 8 bits, 2^-11 of one of 11; fp32 sums over the rows, whose terms have either sign, and a
            # difference from the mean of 3 before them
            tol = (2.0 ** -8 if dtype is torch.bfloat16 else 2.0 ** -11) + 2.0 ** -22 * (rows ** 0.5 if i > 1 else 1)
            if cols == 8 and i == 1:
                tol *= 8                                           # of few columns the gradient is what two projections leave over
            assert a.dtype == dtype and torch.isfinite(a).all()
            assert float((a.detach().double() - b.detach()).norm()) <= tol * float(b.norm()), (i, zero_centered)
        assert all(torch.equal(a, b) for a, b in zip(got[1:], again))
