"""The two-SM GEMM's tiles of 128 columns (problems whose tiles all run at once): edges of rows, columns and k-blocks, every layout and epilogue."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
@pytest.mark.parametrize("M,N,K", [(256, 128, 64), (264, 136, 8), (512, 1000, 520), (776, 2304, 1088), (296, 9472, 72), (1280, 1920, 136)])
def test_against_64_bits(M, N, K, a_mn, b_mn):
    from megatronapp_b200 import ops

    g = torch.Generator().manual_seed(M + N + K)
    A = torch.randn((K, M) if a_mn else (M, K), generator=g).bfloat16().cuda()
    B = torch.randn((K, N) if b_mn else (N, K), generator=g).bfloat16().cuda()
    a64, b64 = (A.t() if a_mn else A).double(), (B if b_mn else B.t()).double()
    want, size = a64 @ b64, a64.abs() @ b64.abs()
    fp32 = K * 2.0 ** -23 * size                      # K exact products added, each sum off by at most one unit of its last place
    out = ops.gemm(A, B, a_mn=a_mn, b_mn=b_mn)
    assert bool(((out.double() - want).abs() <= fp32 + 2.0 ** -8 * want.abs()).all())
    if a_mn == b_mn:
        d = torch.randn(M, N, generator=g).cuda()
        acc = d.clone()
        ops.gemm(A, B, out=acc, a_mn=a_mn, b_mn=b_mn, epilogue=1)
        assert bool(((acc.double() - d.double() - want).abs() <= fp32 + 2.0 ** -23 * (want.abs() + d.double().abs())).all())
        ops.gemm(A, B, out=d, a_mn=a_mn, b_mn=b_mn, epilogue=2)
        assert bool(((d.double() - want).abs() <= fp32).all())
    if not a_mn and not b_mn:
        bias, pre = torch.randn(N, generator=g).bfloat16().cuda(), torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
        act = ops.gemm(A, B, bias=bias, act=1, out_pre=pre)
        z = want + bias.double()
        assert bool(((pre.double() - z).abs() <= fp32 + 2.0 ** -8 * z.abs()).all())
        # tanh-GELU: a slope of at most 1.13, the hardware's tanh (relative error 2^-10.9), its own value rounded to 16 bits
        gelu = torch.nn.functional.gelu(z, approximate="tanh")
        assert bool(((act.double() - gelu).abs() <= 1.2 * fp32 + 2.0 ** -8 * gelu.abs() + 2.0 ** -11 * z.abs() + 2.0 ** -20).all())
