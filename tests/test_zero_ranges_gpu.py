"""Zeroing of several ranges of a gradient buffer in one launch: odd starts and ends, lengths around a block."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("ranges", [[(0, 1)], [(1, 2), (3, 10), (15, 64)], [(7, 7 + 32768), (40000, 40000 + 16384)], [(16383, 16385), (32767, 200001)],
                                    [(i * 3000 + i, i * 3000 + 1500) for i in range(60)]])
def test_only_the_ranges(ranges, dtype):
    from megatronapp_b200 import ops

    data = torch.ones(200003, dtype=dtype, device="cuda")
    want = data.clone()
    for a, b in ranges:
        want[a:b] = 0
    table, blocks = ops.ext().zero_ranges_plan(data.element_size(), ranges)
    ops.ext().zero_ranges(data, table.cuda(), blocks)
    assert torch.equal(data, want)
    with pytest.raises(RuntimeError):
        ops.ext().zero_ranges_plan(data.element_size(), [(5, 5)])
