"""Expert weight gradients: the first micro-batch of a step stores, the next ones add, experts without tokens leave zeros."""
import pytest
import torch


def _layout(counts, topk_total, device):
    from megatronapp_b200.ops.moe import build_layout

    E = len(counts)
    rm = torch.zeros(sum(counts), E, dtype=torch.bool)
    t = 0
    for e, c in enumerate(counts):
        rm[t:t + c, e] = True
        t += c
    return build_layout(rm.to(device), None, 0, E, 1)


@pytest.mark.parametrize("device", ["cpu", pytest.param("cuda", marks=pytest.mark.gpu)])
@pytest.mark.parametrize("counts", [[5, 0, 300, 1], [0, 0, 7], [256, 257, 0, 0, 3]])
def test_store_then_add(device, counts):
    from megatronapp_b200.ops.moe import grouped_wgrad

    E, out_f, in_f = len(counts), 256, 136
    lay = _layout(counts, 1, device)
    g = torch.Generator().manual_seed(1)
    rows = lambda w: (torch.randn(lay.cap, w, generator=g).to(device) * (lay.row_slot >= 0).unsqueeze(1)).bfloat16()  # noqa: E731
    dy, x = rows(out_f), rows(in_f)
    w = torch.nn.Parameter(torch.zeros(E * out_f, in_f, dtype=torch.bfloat16, device=device))
    w.main_grad = torch.full((E * out_f, in_f), 7.0, device=device)               # what the step before left
    w.b200_wgrad_store_first, w.grad_added_to_main_grad = True, False
    offs = lay.offsets.tolist()
    want = torch.zeros(E * out_f, in_f, dtype=torch.float64)
    for e in range(E):
        a, b = dy[offs[e]:offs[e + 1]].cpu().double(), x[offs[e]:offs[e + 1]].cpu().double()
        want[e * out_f:(e + 1) * out_f] = a.t() @ b
    for times in (1, 2):
        assert grouped_wgrad(dy, x, w, lay, out_f, True) is None
        # fp32 sums of exact products of at most 300 terms
        assert float((w.main_grad.cpu().double() - times * want).abs().max()) <= 1e-4 * times * max(1.0, float(want.abs().max()))
    del w.main_grad
    dw = grouped_wgrad(dy, x, w, lay, out_f, False)
    assert float((dw.cpu().double() - want).abs().max()) <= 2.0 ** -8 * float(want.abs().max())


def test_gradient_outside_the_grouped_path_replaces_what_was_left():
    """A stored-first weight whose gradient arrives through autograd: its buffer is not zeroed, so the first contribution replaces it."""
    from megatronapp_b200.config.transformer_config import TransformerConfig
    from megatronapp_b200.parallel import state as ps
    from megatronapp_b200.parallel.ddp import DistributedDataParallel, DistributedDataParallelConfig

    ps.initialize_model_parallel(1, 1)
    lin = torch.nn.Linear(4, 3, bias=False)
    lin.weight.b200_wgrad_store_first = True
    cfg = TransformerConfig(num_layers=1, hidden_size=4, num_attention_heads=1, use_cpu_initialization=True)
    ddp = DistributedDataParallel(cfg, DistributedDataParallelConfig(grad_reduce_in_fp32=True), lin)
    for _ in range(2):
        ddp.zero_grad_buffer()
        for _ in range(2):
            ddp(torch.ones(2, 4)).sum().backward()
        assert torch.equal(lin.weight.main_grad, torch.full((3, 4), 4.0))
