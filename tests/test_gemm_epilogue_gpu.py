"""Epilogue of the tcgen05 GEMMs, both kernels: slabs of 32 rows and 64 columns at the edges of the matrix, bias at any address, every form of store."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# one-SM kernel (below 256 rows or 128 columns), wide tiles of the pair kernel with the last slabs outside, one row or column inside them
@pytest.mark.parametrize("M,N,K", [(1, 64, 64), (33, 200, 136), (255, 1032, 72), (300, 72, 264), (257, 19008, 64), (4097, 776, 136), (2336, 2320, 64)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_store_bias_gelu(M, N, K, dtype):
    from megatronapp_b200 import ops

    g = torch.Generator().manual_seed(M + N + K)
    A, B = (torch.randn(r, K, generator=g).to(dtype).cuda() for r in (M, N))
    bias = torch.randn(N + 1, generator=g).to(dtype).cuda()[1:]                     # two bytes past a 4-byte boundary
    want, size = A.double() @ B.double().t(), A.double().abs() @ B.double().abs().t()
    fp32 = K * 2.0 ** -23 * size                      # K exact products added, each sum off by at most one unit of its last place
    ulp = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)
    frame = torch.full((M + 1, N), 7.0, dtype=dtype, device="cuda")                 # a row behind the result stays as it is
    ops.gemm(A, B, out=frame[:M])
    assert bool(((frame[:M].double() - want).abs() <= fp32 + ulp * want.abs() + 2.0 ** -24).all()) and bool((frame[M] == 7.0).all())
    z = want + bias.double()
    out = ops.gemm(A, B, bias=bias)
    assert bool(((out.double() - z).abs() <= fp32 + ulp * z.abs() + 2.0 ** -24).all())
    pre = torch.empty_like(out)
    act = ops.gemm(A, B, bias=bias, act=1, out_pre=pre)
    assert torch.equal(pre, out)
    # tanh-GELU: a slope of at most 1.13, the hardware's tanh (relative error 2^-10.9), its own value rounded to 16 bits
    gelu = torch.nn.functional.gelu(z, approximate="tanh")
    assert bool(((act.double() - gelu).abs() <= 1.2 * fp32 + ulp * gelu.abs() + 2.0 ** -11 * z.abs() + 2.0 ** -20).all())
    if N % 4 == 0:
        d = torch.randn(M, N, generator=g).cuda()
        acc = d.clone()
        ops.gemm(A, B, out=acc, epilogue=1)
        assert bool(((acc.double() - d.double() - want).abs() <= fp32 + 2.0 ** -23 * (want.abs() + d.double().abs())).all())
        ops.gemm(A, B, out=d, epilogue=2)
        assert bool(((d.double() - want).abs() <= fp32).all())
