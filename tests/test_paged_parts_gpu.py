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
    ([(257, 1)], 8, 8, 128),                               # the shortest context that is cut
    ([(0, 1), (300, 100), (2000, 1)], 8, 2, 128)])         # beside a chunk
def test_parts(reqs, hq, hkv, d):
    from megatronapp_b200 import ops

    cx, q, k, v = _step(reqs, hq, hkv, d, 16, torch.bfloat16)
    want, kc, vc = _oracle(cx, reqs, q, k, v, d ** -0.5, 16)
    tol = 2.0 ** -8 * max(1.0, float(want.abs().max()))    # the result's rounding
    for _ in range(3):                                     # workspaces that earlier calls have used
        got = cx.attend(1, q, k, v, d ** -0.5)
        assert float((got.double() - want).abs().max()) <= tol
    got = ops.ext().paged_attention(q, kc, vc, cx._block_table, cx._tok_req, cx._tok_len, 16, d ** -0.5, 1)
    assert float((got.double() - want).abs().max()) <= tol
