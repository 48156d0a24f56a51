"""Column sums behind norms and biases: one launch, the parameter's type, the same result every time."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols", [(1, 8), (31, 72), (511, 64), (512, 136), (4096, 768), (5000, 4096), (700, 20000)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_bias_grad(rows, cols, dtype):
    from megatronapp_b200 import ops

    dy = torch.randn(rows, cols, device="cuda").to(dtype)
    want = dy.double().sum(0)
    got, same, narrow = ops.bias_grad(dy), ops.bias_grad(dy), ops.bias_grad(dy, dtype)
    assert got.dtype == torch.float32 and narrow.dtype == dtype and torch.equal(got, same)
    # fp32 sums of `rows` terms of about one: their rounding is below 2^-24 of the terms' total size
    assert float((got.double() - want).abs().max()) <= 2.0 ** -24 * rows * 4
    assert torch.equal(narrow, got.to(dtype))


@pytest.mark.parametrize("rows,cols,rms", [(1, 8, False), (5, 264, True), (295, 768, False), (297, 1024, True), (1000, 8192, False)])
def test_norm_parameter_gradients(rows, cols, rms):
    from megatronapp_b200 import ops

    x, dy = torch.randn(2, rows, cols, device="cuda").bfloat16()
    g, b = (1 + 0.1 * torch.randn(cols, device="cuda")).bfloat16(), None if rms else torch.zeros(cols, device="cuda").bfloat16()
    ins = [t.requires_grad_() for t in (x.clone(), g, b) if t is not None]
    got = torch.autograd.grad(ops.layer_norm(ins[0], ins[1], None if rms else ins[2], 1e-5, rms=rms), ins, dy)
    xd = x.double()
    mu = 0 if rms else xd.mean(-1, keepdim=True)
    xh = (xd - mu) * torch.rsqrt((xd - mu).pow(2).mean(-1, keepdim=True) + 1e-5)
    want = [(dy.double() * xh).sum(0), dy.double().sum(0)]
    for a, w in zip(got[1:], want):
        assert a.dtype == torch.bfloat16
        # one rounding to bf16 (7 stored bits: at most 2^-8 of the value), beside fp32 sums
        assert float((a.double() - w).abs().max()) <= 2.0 ** -8 * float(w.abs().max()) + 1e-5 * rows ** 0.5 * 8


@pytest.mark.parametrize("rows,cols,launches", [
    (513, 20000, 2), (4096, 64, 1), (4097, 64, 2), (4128, 72, 2), (70001, 256, 2), (200000, 8, 2), (1024, 12288, 1), (2049, 12288, 2), (5000, 16392, 2)])
def test_long_bias_grad(rows, cols, launches):
    """Shares of more than 512 rows are cut finer than a cluster has CTAs, so that few columns do not leave the device idle; remainders of rows
    and columns around that line."""
    from megatronapp_b200 import ops

    dy = torch.randn(rows, cols, device="cuda", dtype=torch.bfloat16)
    want = dy.double().sum(0)
    for dtype in (torch.float32, torch.bfloat16):
        before = ops.launch_count()
        got = ops.bias_grad(dy, dtype)
        assert ops.launch_count() == before + launches and got.dtype == dtype and torch.equal(got, ops.bias_grad(dy, dtype))
        # fp32 as above, then one rounding to 16 bits
        bound = 2.0 ** -24 * rows * 4 + (2.0 ** -8 * want.abs() if dtype is torch.bfloat16 else 0.0)
        assert bool(((got.double() - want).abs() <= bound).all())
