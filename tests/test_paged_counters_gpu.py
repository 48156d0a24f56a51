"""Counters of cut decode contexts in calls that write no keys themselves, beside portions of prompts: zeroed in front of every launch."""
import pytest
import torch

from test_paged_attention_gpu import _oracle, _step

REQS = [(300, 100), (2000, 1), (0, 1), (1500, 1)]


def _unwritten(d=64):
    cx, q, k, v = _step(REQS, 8, 2, d, 16, torch.bfloat16)
    off = torch.empty(*k.shape[:2], d + 4, dtype=k.dtype, device="cuda")     # rows off 16-byte boundaries: written by PyTorch
    off[..., :d] = k
    return cx, q, off[..., :d], v


@pytest.mark.gpu
def test_values():
    cx, q, k, v = _unwritten()
    want, kc, vc = _oracle(cx, REQS, q, k, v, 0.125, 16)
    for _ in range(5):
        rest = [torch.full((n,), -1, dtype=torch.int32, device="cuda") for n in (1 << 14, 1 << 18, 1 << 20)]      # what a workspace may have held
        del rest
        got = cx.attend(1, q, k, v, 0.125)
        assert torch.equal(cx.kv[1][0], kc) and torch.equal(cx.kv[1][1], vc)
        assert float((got.double() - want).abs().max()) <= 2.0 ** -8 * max(1.0, float(want.abs().max()))


@pytest.mark.gpu
def test_order_of_the_launches():
    """The call as a graph of three launches: the memset is the one that waits for none."""
    from cuda.bindings import runtime as rt

    cx, q, k, v = _unwritten()
    cx.attend(1, q, k, v, 0.125)
    from megatronapp_b200 import ops

    decode, cuts = cx._paged_plans[(4, 2, 64)]
    kc, vc = cx.kv[1]
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        ops.ext().paged_attention(q, kc, vc, cx._block_table, cx._tok_req, cx._tok_len, 16, 0.125, decode, None, None, None, cx.packed.cu, *cuts)
    raw = rt.cudaGraph_t(init_value=graph.raw_cuda_graph())
    _, _, count = rt.cudaGraphGetNodes(raw)
    err, roots, n = rt.cudaGraphGetRootNodes(raw, 4)
    assert err == rt.cudaError_t.cudaSuccess and count == 3 and n == 1
    err, kind = rt.cudaGraphNodeGetType(roots[0])
    assert err == rt.cudaError_t.cudaSuccess and kind == rt.cudaGraphNodeType.cudaGraphNodeTypeMemset
