"""Decode parts that the CTA which comes last puts together: requests beyond those in registers, rows that leave threads over, a call that writes nothing."""
import pytest
import torch

from test_paged_attention_gpu import _oracle, _step


@pytest.mark.gpu
@pytest.mark.parametrize("reqs,hq,hkv,d", [
    ([(700, 1), (20, 1)] * 150, 32, 4, 64),                # 300 requests, three searches
    ([(9000, 1)], 1, 1, 128),                              # one row, more parts than a warp has lanes
    ([(6000, 3)], 2, 2, 64),                               # three rows
    ([(4000, 2), (4000, 1)], 8, 1, 64),                    # 16 rows
    ([(448, 1)], 8, 8, 128), ([(447, 1)], 8, 8, 128),      # the shortest context that is cut, and the longest that is not
    ([(0, 1), (300, 100), (2000, 1)], 8, 2, 128)])         # beside a chunk
def test_parts(reqs, hq, hkv, d):
    from megatronapp_b200 import ops

    cx, q, k, v = _step(reqs, hq, hkv, d, 16, torch.bfloat16)
    want, kc, vc = _oracle(cx, reqs, q, k, v, d ** -0.5, 16)
    tol = 2.0 ** -8 * max(1.0, float(want.abs().max()))    # the result's rounding
    _, (tiles, _, longest, mean, *_) = cx._kernel_plan(hq // hkv, hkv, d)
    assert (ops.ext().paged_decode_cut(len(reqs), hkv, hq // hkv, d, longest, mean, tiles > 0) > 0) == ((447, 1) not in reqs)
    for _ in range(3):                                     # workspaces that earlier calls have used
        got = cx.attend(1, q, k, v, d ** -0.5)
        assert float((got.double() - want).abs().max()) <= tol
    got = ops.ext().paged_attention(q, kc, vc, cx._block_table, cx._tok_req, cx._tok_len, 16, d ** -0.5, 1)
    assert float((got.double() - want).abs().max()) <= tol


@pytest.mark.gpu
@pytest.mark.parametrize("requests,ng,group,d,longest,mean,beside,ctas", [
    (1, 8, 1, 128, 448, 448, False, 0), (1, 8, 1, 128, 449, 449, False, 32),                     # few (request, head) pairs: eight stages
    (8, 4, 4, 128, 512, 300, False, 0), (8, 4, 4, 128, 513, 300, False, 144),                    # more than 16: nine
    (47, 8, 4, 128, 529, 299, False, 0), (47, 8, 4, 128, 640, 299, False, 444),                  # six stages more than a CTA's share
    (24, 4, 4, 128, 513, 300, True, 432), (25, 4, 4, 128, 896, 400, True, 0), (25, 4, 4, 128, 897, 400, True, 444),       # beside chunks
    (30, 12, 1, 64, 1024, 600, True, 0), (30, 12, 1, 64, 1025, 600, False, 444), (64, 8, 4, 64, 512, 300, False, 0), (64, 8, 4, 64, 513, 300, False, 444)])
def test_which_contexts_are_cut(requests, ng, group, d, longest, mean, beside, ctas):
    """Either side of the lengths and counts at which cut contexts were measured faster than whole ones."""
    from megatronapp_b200 import ops

    assert ops.ext().paged_decode_cut(requests, ng, group, d, longest, mean, beside) == ctas


@pytest.mark.gpu
@pytest.mark.parametrize("d,group,n", [(128, 4, 3), (64, 1, 3), (128, 1, 90), (64, 2, 200)])      # few CTAs, and more than run at once
def test_what_follows_waits_for_portions_too(d, group, n):
    """Decoding requests that are done long before the portion beside them: the next launch of the stream sees the portion's rows."""
    reqs = [(6000, 500)] + [(5, 1)] * n
    cx, q, k, v = _step(reqs, 8 * group, 8, d, 16, torch.bfloat16)
    want = cx.attend(1, q, k, v, d ** -0.5)
    torch.cuda.synchronize()
    for _ in range(5):
        out = cx.attend(1, q, k, v, d ** -0.5)
        copy = out.clone()
        out.zero_()
        torch.cuda.synchronize()
        assert torch.equal(copy, want) and not out.any()
