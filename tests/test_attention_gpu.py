"""Flash attention kernels at the edges of their tiles, against the same operation in 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _no_wait_ran_out():
    from megatronapp_b200 import ops

    yield
    assert ops.ext().attn_status() == 0


def _oracle(q, k, v, scale, causal, do):
    rep = q.shape[1] // k.shape[1]
    q, k, v = (t.detach().double().requires_grad_() for t in (q, k, v))
    s = q @ k.repeat_interleave(rep, 1).transpose(-1, -2) * scale
    if causal:
        s = s.masked_fill(torch.ones(s.shape[-2:], dtype=torch.bool, device=s.device).triu(1), float("-inf"))
    o = torch.softmax(s, -1) @ v.repeat_interleave(rep, 1)
    return [o.detach(), *torch.autograd.grad(o, (q, k, v), do.double())] if do is not None else [o.detach()]


def _close(got, want, dtype):
    # 16-bit weights and results: each element carries one rounding of the weight and one of the result (half a unit each),
    # gradients three of them in turn; the 2-norm of independent roundings stays below the bound of a single one
    unit = 2.0 ** -8 if dtype is torch.bfloat16 else 2.0 ** -11
    for a, b in zip(got, want):
        a = a.detach().double()
        assert torch.isfinite(a).all()
        assert float((a - b).norm()) <= 2 * unit * max(float(b.norm()), 1e-3)


@pytest.mark.parametrize("b,hq,hkv,sq,sk,d,causal,dtype", [
    (1, 1, 1, 64, 64, 64, True, torch.bfloat16),            # half a row block, one iteration: a warpgroup without work
    (2, 4, 2, 192, 192, 128, True, torch.bfloat16),         # odd number of column blocks, groups, batch
    (3, 2, 2, 320, 320, 64, True, torch.float16),
    (1, 8, 1, 448, 448, 128, True, torch.float16),          # one key head: blocks of eight heads in one loop
    (2, 2, 1, 128, 576, 128, False, torch.bfloat16),        # lengths that differ
    (1, 4, 4, 576, 64, 64, False, torch.bfloat16),
    (1, 2, 1, 1088, 1088, 128, True, torch.bfloat16)])
def test_backward_row_blocks(b, hq, hkv, sq, sk, d, causal, dtype):
    from megatronapp_b200 import ops

    g = torch.Generator("cuda").manual_seed(5)
    rnd = lambda s, h: torch.randn(s, b, h, d, generator=g, device="cuda", dtype=torch.float32).to(dtype)  # noqa: E731
    q, k, v, do = rnd(sq, hq), rnd(sk, hkv), rnd(sk, hkv), rnd(sq, hq)
    q, k, v = (t.permute(1, 2, 0, 3).requires_grad_() for t in (q, k, v))
    do = do.permute(1, 2, 0, 3)
    before = ops.launch_count()
    o = ops.attention(q, k, v, d ** -0.5, causal)
    grads = torch.autograd.grad(o, (q, k, v), do)
    assert ops.launch_count() > before
    _close([o, *grads], _oracle(q, k, v, d ** -0.5, causal, do), dtype)


@pytest.mark.parametrize("b,hq,hkv,sq,sk,d,causal,dtype", [
    (1, 1, 1, 1, 1, 64, True, torch.bfloat16),
    (2, 2, 1, 127, 127, 128, True, torch.float16),          # one tile, its last row and column missing
    (1, 3, 3, 129, 129, 64, True, torch.bfloat16),          # one row in the second tile
    (1, 2, 2, 257, 257, 128, True, torch.bfloat16),         # a second block with one row
    (1, 4, 1, 200, 65, 128, False, torch.bfloat16),         # the second half of every key block almost empty
    (2, 2, 2, 1, 700, 64, False, torch.float16),
    (1, 2, 1, 1100, 1100, 64, True, torch.float16)])
def test_forward_tiles(b, hq, hkv, sq, sk, d, causal, dtype):
    from megatronapp_b200 import ops

    g = torch.Generator("cuda").manual_seed(7)
    # a few large keys make the running maximum jump, so that accumulators are rescaled in the middle of a row
    q, k, v = (torch.randn(s, b, h, d, generator=g, device="cuda") for s, h in ((sq, hq), (sk, hkv), (sk, hkv)))
    k[::97] *= 6
    q, k, v = (t.to(dtype).permute(1, 2, 0, 3) for t in (q, k, v))
    _close([ops.attention(q, k, v, d ** -0.5, causal)], _oracle(q, k, v, d ** -0.5, causal, None), dtype)


@pytest.mark.parametrize("sq,sk,d,causal", [(300, 300, 128, True), (64, 64, 64, True), (256, 640, 64, False)])
def test_a_wait_that_runs_out_shows(sq, sk, d, causal):
    """Waits that give up at once: the kernel ends by itself, its rows are NaN and the status says so; the next call is sound again."""
    from megatronapp_b200 import ops

    ext = ops.ext()
    assert ext.attn_status() == 0
    g = torch.Generator("cuda").manual_seed(3)
    q, k, v = (torch.randn(s, 2, 4, d, generator=g, device="cuda").bfloat16().permute(1, 2, 0, 3) for s in (sq, sk, sk))
    scale = d ** -0.5
    o, lse, _ = ext.attn_fwd_limited(q, k, v, scale, causal, False, 0)
    assert ext.attn_status() == 1 and ext.attn_status(True) == 1 and ext.attn_status() == 0
    assert torch.isnan(o).all() and torch.isnan(lse).all()
    o, lse, _ = ext.attn_fwd(q, k, v, scale, causal, False)
    _close([o], _oracle(q, k, v, scale, causal, None), torch.bfloat16)
    if sq % 64 == 0:
        do = torch.randn(sq, 2, 4, d, generator=g, device="cuda").bfloat16().permute(1, 2, 0, 3)
        for t in ext.attn_bwd_limited(do, q, k, v, o, lse, scale, causal, None, None, None, 0):
            assert torch.isnan(t).all()
        assert ext.attn_status(True) == 1
        got = ext.attn_bwd(do, q, k, v, o, lse, scale, causal, None, None, None)
        _close(got, _oracle(q, k, v, scale, causal, do)[1:], torch.bfloat16)
    assert ext.attn_status() == 0
