"""Autograd nodes of the native module against the ``torch.autograd.Function`` classes that tracing, functorch and forward mode still get."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _calls():
    from megatronapp_b200 import ops

    g = torch.Generator("cuda").manual_seed(3)

    def t(*shape, grad=True):
        return torch.randn(*shape, generator=g, device="cuda").bfloat16().requires_grad_(grad)

    x, gamma, beta = t(40, 2, 256), t(256), t(256)
    q, k, v, mixed = t(2, 8, 128, 64), t(2, 2, 128, 64), t(2, 2, 128, 64), t(128, 2, 4, 192)
    return {
        "norm": (lambda *a: ops.layer_norm(*a), lambda *a: ops._NormFn.apply(*a, 1e-5, False, False), [x, gamma, beta]),
        "norm_strided": (lambda x, w: ops.layer_norm(x.transpose(0, 1), w, rms=True), lambda x, w: ops._NormFn.apply(x.transpose(0, 1), w, None, 1e-5, True, False),
                         [x, gamma]),
        "norm_frozen": (lambda x, w: ops.layer_norm(x, w, rms=True), lambda x, w: ops._NormFn.apply(x, w, None, 1e-5, True, False), [x, gamma.detach()]),
        "attention": (lambda *a: ops.attention(*a), lambda *a: ops._AttnFn.apply(*a, 0.125, True), [q, k, v]),
        "packed": (lambda m: ops.attention_packed_qkv(m), lambda m: ops._PackedQKVAttnFn.apply(m, 0.125, True), [mixed]),
        "bias_add": (lambda *a: ops.bias_dropout_add(*a, 0.0, True), lambda *a: ops._BdaFn.apply(*a, 0.0, 0, 0), [x, beta, t(40, 2, 256)]),
        "bias_only": (lambda x, b: ops.bias_dropout_add(x, b, None, 0.0, True), lambda x, b: ops._BdaFn.apply(x, b, None, 0.0, 0, 0), [x, beta]),
    }


NAMES = ["norm", "norm_strided", "norm_frozen", "attention", "packed", "bias_add", "bias_only"]


@pytest.mark.parametrize("name", NAMES)
def test_same_values_gradients_and_saved_tensors(name):
    own, fn, ins = _calls()[name]
    saved, outs = [], []
    for f in (own, fn):
        seen = []
        with torch.autograd.graph.saved_tensors_hooks(lambda t: (seen.append(t.shape), t.clone())[1], lambda t: t):
            y = f(*ins)
        dy = torch.randn(y.shape, generator=torch.Generator("cuda").manual_seed(5), device="cuda").to(y.dtype)
        want = [i for i in ins if i.requires_grad]
        outs.append([y, *torch.autograd.grad(y, want, dy, retain_graph=True)])
        outs[-1] += torch.autograd.grad(y, want, dy.transpose(0, 1).contiguous().transpose(0, 1))     # a strided gradient
        saved.append([s for s in seen if 0 not in s])
        with pytest.raises(RuntimeError, match="second time"):
            torch.autograd.grad(y, want, dy)
    assert saved[0] == saved[1]
    for a, b in zip(*outs):
        assert a.dtype == b.dtype and a.stride() == b.stride() and torch.equal(a, b)
    assert "Fn" not in own(*ins).grad_fn.name()
    with torch.no_grad():
        assert own(*ins).grad_fn is None


@pytest.mark.parametrize("name", NAMES)
def test_watched_calls_go_by_the_function_classes(name):
    own, fn, ins = _calls()[name]
    with torch.autograd.forward_ad.dual_level():
        assert own(*ins).grad_fn.name().endswith("FnBackward")
    for f in (own, fn):
        with pytest.raises(RuntimeError):
            torch.func.vmap(f)(*(i.detach().unsqueeze(0) for i in ins))


def test_products_that_the_kernels_do_not_take():
    from megatronapp_b200 import ops

    def t(*shape):
        return torch.randn(*shape, device="cuda").bfloat16()

    flat = t(64 * 128 + 1)
    for a, b, out in [(t(64, 100)[:, :50], t(32, 50), None), (t(128, 64).t(), t(32, 128), None), (flat[1:].view(64, 128), t(32, 128), None),
                      (t(64, 128), t(36, 128), None), (t(64, 128), t(32, 128), t(32, 64).t())]:
        before = ops.fallback_counts["gemm"]
        got = ops.gemm(a, b, out=out)
        assert ops.fallback_counts["gemm"] == before + 1 and (out is None or got is out)
        assert torch.allclose(got.float(), (a.double() @ b.double().t()).float(), rtol=2 ** -7, atol=2 ** -7 * a.shape[1] ** 0.5)
    a, b, out = t(64, 128), t(32, 128), t(64, 32)
    before = ops.fallback_counts["gemm"]
    assert ops.gemm(a, b, out=out) is out and ops.fallback_counts["gemm"] == before
