"""The embedding table's gradient against 64-bit sums: tile edges, runs of one id over many tiles, strided gradients."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture
def kernels_for_all_lengths(monkeypatch):
    from megatronapp_b200 import ops

    monkeypatch.setattr(ops, "_EMBED_FROM", 1)


def _ids(kind, n, vocab, g):
    if kind == "same":
        return torch.full((n,), vocab - 1)
    if kind == "few":
        return torch.randint(0, 3, (n,), generator=g)
    return torch.randint(0, vocab, (n,), generator=g)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("kind", ["spread", "few", "same"])
@pytest.mark.parametrize("n,h,vocab", [(1, 8, 1), (15, 768, 40), (16, 1032, 7), (17, 64, 5), (96, 256, 50304), (4100, 768, 1024), (16384, 264, 512)])
def test_against_64_bits(n, h, vocab, kind, dtype, kernels_for_all_lengths):
    from megatronapp_b200 import ops

    vocab = max(vocab, 3) if kind == "few" else vocab
    g = torch.Generator().manual_seed(n + h)
    ids = _ids(kind, n, vocab, g).cuda()
    w = torch.randn(vocab, h, generator=g).to(dtype).cuda().requires_grad_()
    dy = torch.randn(n, h, generator=g).to(dtype).cuda()
    out = ops.embedding(ids, w)
    assert out.grad_fn.name().startswith("_EmbeddingFn") and torch.equal(out, w[ids])
    out.backward(dy)
    want = torch.zeros(vocab, h, dtype=torch.float64, device="cuda").index_add_(0, ids, dy.double())
    size = torch.zeros(vocab, h, dtype=torch.float64, device="cuda").index_add_(0, ids, dy.double().abs())
    # fp32 sums of n terms in any order, then one rounding to 16 bits (fp16: also the spacing of its smallest numbers)
    bound = n * 2.0 ** -24 * size + (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11) * want.abs() + 2.0 ** -24
    assert bool(((w.grad.double() - want).abs() <= bound).all())
    again = torch.autograd.grad(ops.embedding(ids, w), w, dy)[0]
    assert torch.equal(again, w.grad)


def test_layouts_and_other_ways_of_differentiating(kernels_for_all_lengths):
    from megatronapp_b200 import ops

    g = torch.Generator().manual_seed(3)
    w = torch.randn(100, 72, generator=g).bfloat16().cuda().requires_grad_()
    ids = torch.randint(0, 100, (3, 50), generator=g).cuda()
    dy = torch.randn(50, 3, 72, generator=g).bfloat16().cuda()
    want = torch.zeros(100, 72, dtype=torch.float64, device="cuda").index_add_(0, ids.reshape(-1), dy.transpose(0, 1).reshape(-1, 72).double())
    size = torch.zeros(100, 72, dtype=torch.float64, device="cuda").index_add_(0, ids.reshape(-1), dy.transpose(0, 1).reshape(-1, 72).double().abs())
    bound = 150 * 2.0 ** -24 * size + 2.0 ** -8 * want.abs()

    def check(got):
        assert bool(((got.double() - want).abs() <= bound).all())

    odd = torch.empty(3 * 50 * 73 + 1, dtype=torch.bfloat16, device="cuda")[1:].view(3, 50, 73)[..., :72]    # rows on odd addresses
    odd.copy_(dy.transpose(0, 1))
    for i in (ids, ids.int(), ids.t().contiguous().t()):
        for d in (dy.transpose(0, 1), dy.transpose(0, 1).contiguous(), odd):
            check(torch.autograd.grad(ops.embedding(i, w), w, d)[0])
    # differentiated again, and under a transform: PyTorch's own form, bit for bit (its sums of few tokens round to 16 bits at each step)
    v = dy.transpose(0, 1).clone().requires_grad_()
    (own,) = torch.autograd.grad(torch.nn.functional.embedding(ids, w), w, v)
    (dw,) = torch.autograd.grad(ops.embedding(ids, w), w, v, create_graph=True)
    assert torch.equal(dw, own)
    assert torch.equal(torch.autograd.grad(dw, v, torch.ones_like(dw))[0], torch.ones_like(v))
    assert torch.equal(torch.func.vjp(lambda t: ops.embedding(ids, t), w.detach())[1](v.detach())[0], own)


@pytest.mark.parametrize("n,own", [(1, False), (64, False), (2048, False), (2049, True), (16384, True), (16385, False)])
def test_lengths_that_come_this_way(n, own):
    """Few tokens need no sort, and PyTorch's one launch beats three and a Python node."""
    from megatronapp_b200 import ops

    w = torch.zeros(64, 8, dtype=torch.bfloat16, device="cuda", requires_grad=True)
    out = ops.embedding(torch.zeros(n, dtype=torch.long, device="cuda"), w)
    assert out.grad_fn.name().startswith("_EmbeddingFn" if own else "EmbeddingBackward")
