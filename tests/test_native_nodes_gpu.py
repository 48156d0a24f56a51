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


def _linears():
    """name -> (x, weight, bias, act)"""
    from megatronapp_b200.parallel import state as ps

    if not ps.model_parallel_is_initialized():
        ps.initialize_model_parallel(1, 1)
    g = torch.Generator("cuda").manual_seed(4)

    def t(*shape, grad=True):
        return (torch.randn(*shape, generator=g, device="cuda") * 0.1).bfloat16().requires_grad_(grad)

    return {
        "bias": (t(40, 2, 256), t(136, 256), t(136), 0), "plain": (t(300, 64), t(64, 64), None, 0), "one_row": (t(1, 128), t(8, 128), t(8), 0),
        "gelu": (t(40, 2, 256), t(128, 256), t(128), 1), "frozen_weight": (t(40, 256), t(72, 256, grad=False), t(72), 0),
        "frozen_input": (t(40, 256, grad=False), t(72, 256), None, 0), "frozen_bias": (t(40, 256), t(72, 256), t(72, grad=False), 0)}


@pytest.mark.parametrize("fuse", [None, "add", "store", "unowned", "bf16"])
@pytest.mark.parametrize("name", ["bias", "plain", "one_row", "gelu", "frozen_weight", "frozen_input", "frozen_bias"])
def test_linear_node(name, fuse):
    """Outputs, gradients, buffers, marks and calls of the hook: the node and the class."""
    from megatronapp_b200 import ops
    from megatronapp_b200.parallel import tp_layers

    x, w, b, act = _linears()[name]
    results = []
    for native in (True, False):
        calls = []
        if fuse:
            dtype = torch.bfloat16 if fuse == "bf16" else torch.float32
            w.main_grad = torch.full(w.shape, 2.0, dtype=dtype, device="cuda")
            w.grad_added_to_main_grad, w.b200_wgrad_store_first = fuse == "add", fuse != "unowned"
            w.grad_ready_hook = lambda: calls.append(bool(w.grad_added_to_main_grad))
        seen = []
        with torch.autograd.graph.saved_tensors_hooks(lambda t: (seen.append(t.shape), t)[1], lambda t: t):
            y = ops.ext().linear(x, w, b, act, bool(fuse) and w.requires_grad) if native else \
                tp_layers._ColumnParallelFn.apply(x, w, b, False, bool(fuse) and w.requires_grad, False, act)
        dy = torch.randn(y.shape, generator=torch.Generator("cuda").manual_seed(5), device="cuda").to(y.dtype)
        want = [i for i in (x, w, b) if i is not None and i.requires_grad]
        got = [y]
        got += torch.autograd.grad(y, want, dy, retain_graph=True, allow_unused=True)
        got += torch.autograd.grad(y, want, dy.unsqueeze(-1).expand(*dy.shape, 2).contiguous()[..., 0], allow_unused=True)      # a strided gradient
        with pytest.raises(RuntimeError, match="second time"):
            torch.autograd.grad(y, want, dy, allow_unused=True)
        results.append((got, seen, calls, w.main_grad.clone() if fuse else None, getattr(w, "grad_added_to_main_grad", None)))
    (a, *ra), (c, *rc) = results
    assert len(a) == len(c) and all((p is None and q is None) or (p.dtype == q.dtype and p.stride() == q.stride() and torch.equal(p, q)) for p, q in zip(a, c))
    assert ra[:2] == rc[:2] and ra[3] == rc[3] and (ra[2] is None or torch.equal(ra[2], rc[2]))
    with torch.no_grad():
        assert ops.ext().linear(x, w, b, act, False).grad_fn is None


def test_linear_node_leaves_the_rest_to_the_class():
    from megatronapp_b200 import ops

    t = lambda *s, **k: torch.zeros(*s, device="cuda", dtype=torch.bfloat16, **k)  # noqa: E731
    linear = ops.ext().linear
    assert linear(t(4, 12), t(8, 12), None, 0, False) is None and linear(t(4, 16), t(12, 16), None, 0, False) is None      # rows of no 16 bytes
    assert linear(t(16, 4).t(), t(8, 16), None, 0, False) is None and linear(t(4, 16), t(16, 8).t(), None, 0, False) is None
    assert linear(t(0, 16), t(8, 16), None, 0, False) is None and linear(t(4, 16).half(), t(8, 16), None, 0, False) is None
    assert linear(t(65)[1:].view(4, 16), t(8, 16), None, 0, False) is None and linear(t(4, 16), t(8, 16), t(8).float(), 0, False) is None


def test_what_a_hook_raises():
    from megatronapp_b200 import ops

    class Odd(Exception):
        pass

    def hook():
        raise Odd("hook")

    x, w, b, _ = _linears()["bias"]
    w.main_grad, w.b200_wgrad_store_first, w.grad_ready_hook = torch.zeros(w.shape, device="cuda"), True, hook
    with pytest.raises(Odd, match="hook"):
        ops.ext().linear(x, w, b, 0, True).sum().backward()


def test_layers_take_the_node():
    from megatronapp_b200.config.transformer_config import TransformerConfig
    from megatronapp_b200.parallel import state as ps
    from megatronapp_b200.parallel.tp_layers import ColumnParallelLinear, RowParallelLinear

    if not ps.model_parallel_is_initialized():
        ps.initialize_model_parallel(1, 1)
    cfg = TransformerConfig(num_layers=1, hidden_size=64, num_attention_heads=1, params_dtype=torch.bfloat16, bf16=True)
    init = torch.nn.init.normal_
    x = torch.randn(5, 2, 64, device="cuda").bfloat16().requires_grad_()
    for layer in (ColumnParallelLinear(64, 128, config=cfg, init_method=init, bias=True, gather_output=False, skip_bias_add=False),
                  RowParallelLinear(64, 128, config=cfg, init_method=init, bias=True, input_is_parallel=True, skip_bias_add=True)):
        layer = layer.cuda()
        assert "Fn" not in layer(x)[0].grad_fn.name()
        with torch.autograd.forward_ad.dual_level():
            assert layer(x)[0].grad_fn.name().endswith("FnBackward")
