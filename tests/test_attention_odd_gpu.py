"""Training attention at short lengths that are no whole blocks of 64 rows, against the same operation in 64 bits."""
import pytest
import torch

from test_attention_gpu import _close, _oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b,hq,hkv,s,d,dtype", [
    (1, 1, 1, 1, 64, torch.bfloat16), (2, 2, 1, 63, 128, torch.float16), (1, 2, 2, 65, 64, torch.bfloat16), (3, 2, 1, 127, 128, torch.bfloat16),
    (1, 4, 2, 129, 64, torch.float16), (2, 3, 1, 191, 128, torch.bfloat16), (8, 16, 4, 459, 64, torch.bfloat16), (1, 2, 2, 511, 128, torch.float16)])
@pytest.mark.parametrize("packed", [False, True])
def test_lengths_that_are_no_whole_blocks(b, hq, hkv, s, d, dtype, packed):
    from megatronapp_b200 import ops

    if packed and hq != hkv:
        pytest.skip("packed projections have as many heads of each")
    assert ops.native_attention_available()
    g = torch.Generator("cuda").manual_seed(6)
    rnd = lambda *n: torch.randn(*n, generator=g, device="cuda", dtype=torch.float32).to(dtype)  # noqa: E731
    before, launches = ops.fallback_counts["attention_sdpa"], ops.launch_count()
    do = rnd(b, hq, s, d)
    if packed:
        mixed = rnd(s, b, hq, 3 * d).requires_grad_()
        q, k, v = (t.permute(1, 2, 0, 3) for t in mixed.split(d, -1))
        o = ops.attention_packed_qkv(mixed)
        grads = [t.permute(1, 2, 0, 3) for t in torch.autograd.grad(o, mixed, do)[0].split(d, -1)]
    else:
        q, k, v = (t.permute(1, 2, 0, 3).requires_grad_() for t in (rnd(s, b, hq, d), rnd(s, b, hkv, d), rnd(s, b, hkv, d)))
        o = ops.attention(q, k, v, d ** -0.5)
        grads = torch.autograd.grad(o, (q, k, v), do)
    assert ops.launch_count() - launches == 3                          # the forward, the statistics and the gradients
    assert ops.fallback_counts["attention_sdpa"] == before
    _close([o, *grads], _oracle(q, k, v, d ** -0.5, True, do), dtype)


def test_scores_far_below_zero():
    """The rows behind the last one read zeros, whose weights against sums of such scores would be infinite."""
    from megatronapp_b200 import ops

    g = torch.Generator("cuda").manual_seed(8)
    q, k, v, do = (torch.randn(2, 4, 100, 64, generator=g, device="cuda").bfloat16() for _ in range(4))
    q[..., 0], k[..., 0] = 40, -40                                     # -200 each: e^200 is no fp32 number
    q, k, v = (t.requires_grad_() for t in (q, k, v))
    o = ops.attention(q, k, v, 0.125)
    dq, dk, dv = torch.autograd.grad(o, (q, k, v), do)
    want = _oracle(q, k, v, 0.125, True, do)
    assert torch.isfinite(dq).all()                                    # (its first column is a sum that cancels)
    _close([o, dq[..., 1:], dk, dv], [want[0], want[1][..., 1:], want[2], want[3]], torch.bfloat16)


def test_who_watches_the_operators_keeps_the_library():
    from megatronapp_b200 import ops

    q, k, v = (torch.randn(1, 2, 100, 64, device="cuda").bfloat16().requires_grad_() for _ in range(3))
    before = ops.fallback_counts["attention_sdpa"]
    with torch.autograd.forward_ad.dual_level():
        ops.attention(q, k, v, 0.125)
        assert ops.attention_packed_qkv(torch.randn(100, 1, 2, 192, device="cuda").bfloat16()) is None
    assert ops.fallback_counts["attention_sdpa"] == before + 1


def test_second_derivatives_are_refused():
    from megatronapp_b200 import ops

    q, k, v = (torch.randn(1, 2, 100, 64, device="cuda").bfloat16().requires_grad_() for _ in range(3))
    mixed = torch.randn(100, 1, 2, 192, device="cuda").bfloat16().requires_grad_()
    for o, leaf in ((ops.attention(q, k, v, 0.125), q), (ops.attention_packed_qkv(mixed), mixed)):
        plain, = torch.autograd.grad(o.float().sum(), leaf, retain_graph=True)
        again, = torch.autograd.grad(o.float().sum(), leaf, create_graph=True)
        assert torch.equal(plain, again)
        with pytest.raises(RuntimeError, match="not implemented"):
            torch.autograd.grad(again.float().square().sum() + leaf.float().sum(), leaf)
