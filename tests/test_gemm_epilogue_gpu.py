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


def test_launches_that_overlap():
    """A product's kernel starts while the one before it still runs: chains of them, results that the next reads or overwrites, in order and in a graph."""
    from megatronapp_b200 import ops

    g = torch.Generator().manual_seed(1)
    x = torch.randn(2048, 512, generator=g).bfloat16().cuda()
    w = [(torch.randn(512, 512, generator=g) * 512 ** -0.5).bfloat16().cuda() for _ in range(4)]
    acc, bufs = torch.zeros(512, 512, device="cuda"), [torch.empty_like(x) for _ in range(2)]

    def chain(pause):
        acc.zero_()
        a = x
        for i in range(24):
            out = bufs[i & 1]                                # read by the product before this one's predecessor
            ops.gemm(a, w[i & 3], out=out)
            pause()
            if i % 5 == 4:
                out.mul_(1.0)                                # a kernel of another kind between them
            ops.gemm(out, a, out=acc, a_mn=True, b_mn=True, epilogue=1)
            pause()
            a = out
        return a.clone(), acc.clone()

    want = chain(torch.cuda.synchronize)
    for _ in range(5):
        for got, ref in zip(chain(lambda: None), want):
            assert torch.equal(got, ref)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        outs = chain(lambda: None)
    for _ in range(3):
        for o in outs:
            o.zero_()
        graph.replay()
        for got, ref in zip(outs, want):
            assert torch.equal(got, ref)


def test_bias_scales_and_groups_that_the_launch_before_writes():
    """What a product's epilogue reads beside its operands may be the result of the launch that it overlaps: other values each time, in the same buffers."""
    from megatronapp_b200 import ops

    g = torch.Generator().manual_seed(2)
    cap, G, N, K = 1024, 3, 512, 256
    a = [(torch.randn(256, K, generator=g) * (i + 1)).bfloat16().cuda() for i in range(4)]
    b = torch.randn(max(N, cap), K, generator=g).bfloat16().cuda()
    x, w = torch.randn(cap, K, generator=g).bfloat16().cuda(), torch.randn(G * N, K, generator=g).bfloat16().cuda()
    offsets = torch.tensor([0, 256, 256, 1024], dtype=torch.int32, device="cuda")
    y16, y32 = torch.empty(256, N, dtype=torch.bfloat16, device="cuda"), torch.empty(256, cap, device="cuda")

    def chain(pause):
        outs = []
        for i in range(24):
            z, zg = torch.empty(cap, N, dtype=torch.bfloat16, device="cuda"), torch.empty(cap, N, dtype=torch.bfloat16, device="cuda")
            ops.gemm(a[i & 3], b[:N], out=y16)
            pause()
            ops.gemm(x, w[:N], out=z, bias=y16[i & 7])
            pause()
            ops.gemm(a[i & 3], b[:cap], out=y32, epilogue=2)
            pause()
            ops.ext().gemm_grouped(x, w, zg, offsets, 1, False, y16[:G], 0, None, y32[i & 7], G, N)
            pause()
            outs += [z, zg]
        return outs

    want = chain(torch.cuda.synchronize)
    assert not torch.equal(want[0], want[2]) and not torch.equal(want[1], want[3])
    z = x.double() @ w[:N].double().t() + (a[0].double() @ b[:N].double().t()).bfloat16()[0].double()
    assert float((want[0].double() - z).abs().max()) <= 2.0 ** -7 * float(z.abs().max())
    for _ in range(5):
        assert all(torch.equal(p, q) for p, q in zip(chain(lambda: None), want))
