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


@pytest.mark.parametrize("change", [lambda g: g, lambda g: g.bfloat16(), lambda g: torch.cat([g, g])[1:g.numel() + 1], lambda g: g[:1000].clone(),
                                    lambda g: torch.stack([g, g], 1)[:, 0]])
def test_a_buffer_that_was_put_in_place_of_the_first(change):
    """A gradient buffer of another type, size, alignment or stride: its ranges become zeros, and nothing else does."""
    from megatronapp_b200.parallel.ddp import DistributedDataParallelConfig, ParamAndGradBuffer

    params = [torch.nn.Parameter(torch.zeros(n, device="cuda")) for n in (640, 1000, 64)]
    params[1].b200_wgrad_store_first = True
    buf = ParamAndGradBuffer(DistributedDataParallelConfig(), torch.float32, torch.float32, params, None, 1, None, 1.0, "cuda")
    s, e, _ = buf.param_index[params[1]]
    buf.grad_data = change(torch.full_like(buf.grad_data, 3.0))
    want = buf.grad_data.clone()
    want[:s], want[e:] = 0, 0
    around = buf.grad_data._base if buf.grad_data._base is not None else buf.grad_data
    rest = int((around == 3).sum()) - int((buf.grad_data == 3).sum())
    buf.zero()
    assert torch.equal(buf.grad_data, want) and int((around == 3).sum()) - int((buf.grad_data == 3).sum()) == rest


@pytest.mark.parametrize("dtype", [torch.float8_e4m3fn, torch.bfloat16, torch.float64])
def test_buffers_of_any_type(dtype):
    """One-byte gradients, whose ranges may start off the kernel's two bytes, are filled range by range."""
    from megatronapp_b200.parallel.ddp import DistributedDataParallelConfig, ParamAndGradBuffer

    params = [torch.nn.Parameter(torch.zeros(n, device="cuda")) for n in (640, 1001, 64)]
    params[1].b200_wgrad_store_first = True
    buf = ParamAndGradBuffer(DistributedDataParallelConfig(), torch.float32, dtype, params, None, 1, None, 1.0, "cuda")
    s, e, _ = buf.param_index[params[1]]
    buf.grad_data.view(torch.uint8).fill_(1)
    buf.zero()
    size = buf.grad_data.element_size()
    got = buf.grad_data.view(torch.uint8)
    assert bool((got[s * size:e * size] == 1).all()) and not got[:s * size].any() and not got[e * size:].any()
