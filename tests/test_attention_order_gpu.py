"""Products with V add their keys in a fixed order."""
import pytest
import torch


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,large,small", [(torch.bfloat16, 2.0 ** 30, 1.0), (torch.float16, 2.0 ** 15, 2.0 ** -10)])
@pytest.mark.parametrize("d", [64, 128])
def test_first_halves_of_a_block_go_first(d, dtype, large, small):
    """Equal weights, and values of one block of 128 keys that cancel in front of a small one: fp32 sums keep that only where the large ones, of the first
    32 keys of both halves, have met before it comes."""
    from megatronapp_b200 import ops

    q, k, v = (torch.zeros(1, 2, 128, d, dtype=dtype, device="cuda") for _ in range(3))
    v[:, :, 0], v[:, :, 40], v[:, :, 70] = large, small, -large
    o, lse, _ = ops.ext().attn_fwd(q, k, v, 1.0, False, False)
    assert torch.equal(o.double(), torch.full_like(o, 1.0).double() * (small / 128))
