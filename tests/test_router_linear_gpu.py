"""Router logits and gradients against 64 bits: odd numbers of tokens, columns and experts, weights of either type."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,wide", [(torch.bfloat16, False), (torch.bfloat16, True), (torch.float16, False)])
@pytest.mark.parametrize("n,h,e", [(1, 8, 1), (5, 264, 9), (33, 2048, 8), (4100, 1032, 32), (8200, 520, 16)])
def test_against_64_bits(n, h, e, dtype, wide):
    from megatronapp_b200.ops import moe

    g = torch.Generator("cuda").manual_seed(n + h + e)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    x = rnd(n, h).to(dtype).requires_grad_()
    w = rnd(e, h).to(torch.float32 if wide else dtype).requires_grad_()
    dl = rnd(n, e)
    out = moe.router_linear(x, w)
    assert out.dtype == torch.float32 and "_RouterLinear" in str(out.grad_fn.next_functions[0][0])
    dx, dw = torch.autograd.grad(out, (x, w), dl)
    x64, w64, d64 = x.detach().double(), w.detach().double(), dl.double()
    step = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11, torch.float32: 0.0}
    for got, a, b in ((out, x64, w64.t()), (dx, d64, w64), (dw, d64.t(), x64)):
        want, size, k = a @ b, a.abs() @ b.abs(), a.shape[1]
        # k products added in fp32 in any order, then one rounding to the result's type (fp16: also its smallest spacing)
        bound = k * 2.0 ** -24 * size + step[got.dtype] * want.abs() + 2.0 ** -24 * (got.dtype == torch.float16)
        assert got.dtype == (torch.float32 if got is out else dtype if got is dx else w.dtype)
        assert bool(((got.detach().double() - want).abs() <= bound).all())
    # a view that is not contiguous, one gradient only, a second derivative
    view = torch.cat([x.detach(), x.detach()], 1)[:, :h].requires_grad_()
    assert torch.equal(torch.autograd.grad(moe.router_linear(view, w.detach()), view, dl)[0], dx)
    assert torch.equal(torch.autograd.grad(moe.router_linear(x.detach(), w), w, dl)[0], dw)
    again, = torch.autograd.grad(moe.router_linear(x, w), x, dl, create_graph=True)
    plain, = torch.autograd.grad(torch.nn.functional.linear(x.float(), w.float()), x, dl, create_graph=True)
    second, want = (torch.autograd.grad(t.float().square().sum(), w)[0] for t in (again, plain))
    assert torch.allclose(second.float(), want.float(), rtol=2.0 ** -7, atol=2.0 ** -7 * float(want.abs().max()))


@pytest.mark.parametrize("shape,h,e", [((1,), 264, 4), ((2048, 2), 2048, 8), ((33, 3), 520, 32), ((4100,), 1024, 16)])
def test_logits_choose_the_experts_of_the_plain_product(shape, h, e):
    """Two experts of a token can lie closer than fp32 sums in another order leave them, so the logits are the plain product's bits."""
    from megatronapp_b200.ops import moe

    g = torch.Generator("cuda").manual_seed(h)
    x = torch.randn(*shape, h, generator=g, device="cuda").bfloat16().requires_grad_()
    w = (0.02 * torch.randn(e, h, generator=g, device="cuda")).bfloat16().requires_grad_()
    for a in (x, x.detach().transpose(0, -2).contiguous().transpose(0, -2).requires_grad_()):
        for grad in (True, False):
            with torch.set_grad_enabled(grad):
                assert torch.equal(moe.router_linear(a, w), torch.nn.functional.linear(a.float(), w.float()))
