"""Paged attention of the continuous-batching engine at the edges of its tiles, stages and key ranges, against 64 bits."""
import pytest
import torch


def _step(reqs, hq, hkv, d, block, dtype, seed=0):
    """A context holding ``reqs = [(tokens in the cache, new tokens)]`` and the new queries, keys and values (as strided views)."""
    from megatronapp_b200.inference.dynamic import DynamicInferenceContext

    g = torch.Generator("cuda").manual_seed(seed)
    cx = DynamicInferenceContext(max(a + n for a, n in reqs) + 1, sum(-(-(a + n) // block) for a, n in reqs) + 1, block, 1 << 16, len(reqs))
    for i in range(len(reqs)):
        cx.add_request(str(i))
    old = [(str(i), a) for i, (a, _) in enumerate(reqs) if a]
    if old:
        cx.begin_step(old[::-1], "cuda")
        cx.end_step()
    cx.begin_step([(str(i), n) for i, (_, n) in enumerate(reqs)], "cuda")
    for t in cx.kv_pages(1, (hkv, d), (hkv, d), dtype):
        t.normal_(generator=g)
    T = sum(n for _, n in reqs)
    q = torch.randn(T, hq, d, generator=g, device="cuda").to(dtype)
    kv = torch.randn(T, hkv, 2, d, generator=g, device="cuda").to(dtype)
    return cx, q, kv[:, :, 0], kv[:, :, 1]


def _oracle(cx, reqs, q, k, v, scale, block):
    kc, vc = (t.clone() for t in cx.kv[1])
    kc[cx.write_slots], vc[cx.write_slots] = k, v
    rep, t0, out = q.shape[1] // k.shape[1], 0, []
    for i, (a, n) in enumerate(reqs):
        slots = (torch.tensor(cx.seqs[str(i)].blocks).unsqueeze(1) * block + torch.arange(block)).view(-1)[:a + n].cuda()
        kk, vv = (t[slots].double().repeat_interleave(rep, 1) for t in (kc, vc))
        for j in range(n):
            L = a + j + 1                                     # no masked key enters the sum
            w = torch.softmax(torch.einsum("hd,lhd->hl", q[t0 + j].double(), kk[:L]) * scale, -1)
            out.append(torch.einsum("hl,lhd->hd", w, vv[:L]))
        t0 += n
    return torch.stack(out), kc, vc


@pytest.mark.gpu
@pytest.mark.parametrize("reqs,hq,hkv,d,block,dtype", [
    ([(0, 1)], 4, 4, 64, 16, torch.bfloat16),                                    # one key
    ([(63, 1), (64, 1), (127, 1), (500, 1)], 8, 1, 128, 16, torch.bfloat16),     # around a stage
    ([(5000, 1)], 8, 2, 128, 16, torch.float16),                                 # one item over many CTAs
    ([(16383, 1), (3, 1)], 4, 4, 64, 32, torch.bfloat16),                        # cuts inside one item and around the other
    ([(3000, 1)] * 7 + [(1, 1)] * 50 + [(5000, 1)], 4, 1, 64, 16, torch.bfloat16),
    ([(9000, 30)], 8, 2, 128, 16, torch.bfloat16),                               # few tiles, long context: key ranges in a cluster
    ([(1100, 40), (0, 20)], 4, 1, 64, 16, torch.float16),                        # a tile whose later ranges are empty
    ([(10, 4), (0, 5), (100, 16), (7, 17)], 4, 1, 128, 16, torch.bfloat16),      # 16 rows and just more
    ([(0, 64), (130, 1), (1000, 65)], 16, 2, 64, 16, torch.float16),             # whole row tiles and one token more
    ([(40, 9), (900, 200), (0, 1), (77, 300)], 12, 12, 128, 24, torch.bfloat16),  # a block size that is no power of two
    ([(0, 3)] * 40 + [(20, 70)] + [(5, 1)] * 30, 8, 8, 64, 16, torch.bfloat16)])  # more requests than a warp searches at once
def test_tiles(reqs, hq, hkv, d, block, dtype):
    cx, q, k, v = _step(reqs, hq, hkv, d, block, dtype)
    want, kc, vc = _oracle(cx, reqs, q, k, v, d ** -0.5, block)
    got = cx.attend(1, q, k, v, d ** -0.5)
    assert cx.kernel_calls == 1
    assert torch.equal(cx.kv[1][0], kc) and torch.equal(cx.kv[1][1], vc)
    # fp32 sums of exact products: what is left is the result's own rounding, half a unit in the last place
    unit = 2.0 ** -8 if dtype is torch.bfloat16 else 2.0 ** -11
    assert float((got.double() - want).abs().max()) <= unit * max(1.0, float(want.abs().max()))
    assert float((got.double() - want).norm()) <= 0.5 * unit * float(want.norm())


@pytest.mark.gpu
def test_values_of_later_tokens_stay_out():
    """An infinite value of a chunk's token reaches the tokens that see it and no others."""
    reqs = [(70, 100)]
    cx, q, k, v = _step(reqs, 4, 2, 64, 16, torch.bfloat16)
    v[60, 0, 5], v[60, 1, 3] = float("inf"), float("nan")
    want, _, _ = _oracle(cx, reqs, q, k, v, 0.125, 16)
    got = cx.attend(1, q, k, v, 0.125).double()
    assert torch.equal(torch.isfinite(got), torch.isfinite(want))
    ok = torch.isfinite(want)
    assert ok[:60].all() and not ok[60:, :2, 5].any() and not ok[60:, 2:, 3].any()
    assert float((got[ok] - want[ok]).abs().max()) <= 2.0 ** -7


def test_key_ranges():
    from megatronapp_b200.inference.dynamic import key_ranges

    assert key_ranges(8, 100) == 1                                 # too short to cut
    assert key_ranges(8, 1 << 20) == 16 and key_ranges(149, 1 << 20) == 1
    for tiles in (1, 7, 64, 500):
        for n in (1, 255, 512, 1000, 4096, 100000):
            r = key_ranges(tiles, n)
            assert r in (1, 2, 4, 8, 16) and (r == 1 or n >= 256 * r)


def _four_keys(dtype, scores, values, d=64):
    """One decoding request that sees four keys; ``scores [heads][4]`` lie along the first axis (the query is one there), ``values [4, heads]``
    in every column."""
    heads = len(scores)
    cx, q, k, v = _step([(3, 1)], heads, heads, d, 16, dtype)
    q.zero_()
    q[:, :, 0] = 1
    kk, vv = torch.zeros(4, heads, d, device="cuda", dtype=dtype), torch.zeros(4, heads, d, device="cuda", dtype=dtype)
    kk[:, :, 0] = torch.tensor(scores, device="cuda").t().to(dtype)
    vv[:] = values.to(dtype).unsqueeze(-1)
    kc, vc = cx.kv[1]
    slots = torch.tensor(cx.seqs["0"].blocks[0] * 16) + torch.arange(4)
    kc[slots.cuda()], vc[slots.cuda()] = kk, vv
    return cx, q, kk[3:], vv[3:], kk[..., 0].double()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_weights_enter_with_all_their_bits(dtype):
    """Values that cancel but for 2^-24 of their sum: the weights' own rounding is all that is left."""
    g = torch.Generator().manual_seed(1)
    scores = (torch.rand(32, 4, generator=g, dtype=torch.float64) * 0.5).to(dtype)
    scores[:, 0] = 0.625                                     # the largest: its weight is one
    w = torch.exp2((scores.double() - 0.625) * 1.4426950408889634).cuda()
    val = torch.zeros(4, 32, dtype=torch.float64, device="cuda")
    val[1] = 1
    for i in (0, 2, 3):                                      # each takes the rest away as far as its 16 bits go
        val[i] = (-(w.t() * val).sum(0) / w[:, i]).to(dtype)
    cx, q, k, v, _ = _four_keys(dtype, scores.tolist(), val)
    want = (w.t() * val).sum(0) / w.sum(1)
    got = cx.attend(1, q, k, v, 1.0)[0].double()
    # exp2f is within 2 ulp (2^-23) and so are fp32 sums of four terms of at most one
    assert float((got - want.unsqueeze(-1)).abs().max()) <= 2.0 ** -21


@pytest.mark.gpu
def test_small_weights_of_fp16():
    """Weights below fp16's normal range, of keys whose values are large, beside one large weight whose value is zero."""
    scores = [[0.0, -12.0 - 0.0625 * h, -13.0, -14.5] for h in range(16)]
    val = torch.tensor([[0.0] * 16, [60000.0] * 16, [30000.0] * 16, [-50000.0] * 16], device="cuda")
    cx, q, k, v, s = _four_keys(torch.float16, scores, val)
    w = torch.exp(s)
    want = (w * val.half().double()).sum(0) / w.sum(0)
    got = cx.attend(1, q, k, v, 1.0)[0].double()
    assert float(((got - want.unsqueeze(-1)) / want.unsqueeze(-1)).abs().max()) <= 2.0 ** -11 + 2.0 ** -18


@pytest.mark.gpu
@pytest.mark.parametrize("reqs", [[(500, 1)], [(5000, 1), (3, 1)], [(300, 70)], [(2000, 40)]])
@pytest.mark.parametrize("dtype,scale", [(torch.float16, -1.0), (torch.bfloat16, -0.5), (torch.float16, 0.0), (torch.bfloat16, 0.0)])
def test_scales_that_are_not_positive(reqs, dtype, scale):
    cx, q, k, v = _step(reqs, 4, 2, 64, 16, dtype)
    want, _, _ = _oracle(cx, reqs, q, k, v, scale, 16)
    got = cx.attend(1, q, k, v, scale).double()
    unit = 2.0 ** -8 if dtype is torch.bfloat16 else 2.0 ** -11
    # scores of up to 50: their own fp32 rounding moves a weight by 2^-18
    assert float((got - want).abs().max()) <= unit * max(1.0, float(want.abs().max()))


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,size", [(torch.float16, 30000.0), (torch.bfloat16, 1e6)])
def test_scores_beyond_the_exponent(dtype, size):
    """Scores so large that one unit of their rounding is more than any weight can hold: the largest key has all the weight."""
    scores = [[0.25, -0.5, 0.5, 0.125], [0.0, 0.0, -1.0, -1.0], [-0.5, -0.25, -0.25, -1.0]]
    val = torch.arange(12, device="cuda").view(4, 3) + 1.0
    cx, q, k, v, s = _four_keys(dtype, [[x * size for x in r] for r in scores], val)
    q *= size
    got = cx.attend(1, q, k, v, 64.0)[0, :, 0].double().cpu()
    assert torch.equal(got, torch.tensor([7.0, (2 + 5) / 2, (6 + 9) / 2], dtype=torch.float64))


@pytest.mark.gpu
@pytest.mark.parametrize("n,longest,chunk,hq,hkv,d,block,dtype", [
    (130, 128, 0, 4, 4, 64, 16, torch.bfloat16),              # group 1, some 500 pairs, short contexts
    (250, 250, 0, 4, 4, 128, 24, torch.float16),              # 1000 pairs; a block size that is no power of two
    (300, 600, 70, 8, 4, 64, 16, torch.bfloat16),             # group 2 beside a chunk of several tiles
    (225, 128, 9, 8, 4, 128, 16, torch.float16),              # ... beside a chunk of one tile, one of more tokens than a decoding request
    (230, 32, 0, 16, 4, 128, 32, torch.bfloat16)])            # group 4
def test_many_requests_with_few_rows(n, longest, chunk, hq, hkv, d, block, dtype):
    """One CTA per (request, KV head) instead of tiles, against 64 bits; contexts of one key and of the longest length among them."""
    from megatronapp_b200 import ops

    g = torch.Generator().manual_seed(n)
    reqs = [(0, 1), (longest - 1, 1)] + [(int(a), 1) for a in torch.randint(0, longest, (n - 2,), generator=g)]
    if chunk:
        reqs.insert(n // 2, (33, chunk))
    assert ops.ext().paged_decode_by_rows(len(reqs), hkv, hq // hkv, d, longest, longest // 2, True)
    cx, q, k, v = _step(reqs, hq, hkv, d, block, dtype)
    want, kc, vc = _oracle(cx, reqs, q, k, v, d ** -0.5, block)
    for _ in range(2):
        got = cx.attend(1, q, k, v, d ** -0.5)
        assert torch.equal(cx.kv[1][0], kc) and torch.equal(cx.kv[1][1], vc)
        unit = 2.0 ** -8 if dtype is torch.bfloat16 else 2.0 ** -11
        assert float((got.double() - want).abs().max()) <= unit * max(1.0, float(want.abs().max()))
        assert float((got.double() - want).norm()) <= 0.5 * unit * float(want.norm())


@pytest.mark.gpu
@pytest.mark.parametrize("requests,ng,group,d,longest,mean,single,rows", [
    (64, 8, 1, 128, 100, 100, True, True), (512, 32, 1, 64, 600, 600, True, True), (512, 32, 1, 64, 2048, 2048, True, True),
    (512, 32, 1, 64, 2049, 2049, True, False), (256, 12, 2, 64, 600, 600, True, True), (256, 12, 2, 128, 600, 600, True, False),
    (512, 8, 4, 128, 16, 16, True, True), (512, 8, 4, 128, 63, 63, True, False), (512, 8, 8, 128, 16, 16, True, False),
    (64, 8, 1, 128, 600, 600, True, False), (32, 12, 1, 64, 100, 100, True, False), (512, 32, 1, 64, 100, 100, False, False),
    (96, 12, 1, 128, 1000, 1000, True, True), (96, 12, 1, 128, 1000, 532, True, False), (96, 12, 1, 64, 1000, 532, True, True)])
def test_which_decode_kernel(requests, ng, group, d, longest, mean, single, rows):
    """Lengths and counts at which a CTA per (request, KV head) was measured faster than tiles, and some at which it was not."""
    from megatronapp_b200 import ops

    assert ops.ext().paged_decode_by_rows(requests, ng, group, d, longest, mean, single) == rows


def test_a_plan_looks_at_the_contexts_that_it_cuts():
    """Key ranges follow the portions' own contexts, and the decode kernels hear of the others' only."""
    from megatronapp_b200.inference.dynamic import DynamicInferenceContext

    def plan(reqs, group, ng):
        cx = DynamicInferenceContext(1 << 16, sum(-(-(a + n) // 16) for a, n in reqs) + 1, 16, 1 << 16, len(reqs))
        for i in range(len(reqs)):
            cx.add_request(str(i))
        old = [(str(i), a) for i, (a, _) in enumerate(reqs) if a]
        if old:
            cx.begin_step(old, "cpu")
            cx.end_step()
        cx.begin_step([(str(i), n) for i, (_, n) in enumerate(reqs)], "cpu")
        return cx._paged_plan(group, ng)

    # (requests of up to 16 rows, tiles, key ranges of those, longest and average context of the former, one token each)
    assert plan([(0, 16), (4095, 1)], 4, 8) == (1, 1, 1, 4096, 4096, True)          # a fresh portion is not cut for its neighbour's context
    assert plan([(8000, 64), (99, 1), (199, 1)], 1, 8) == (2, 1, 16, 200, 150, True)
    assert plan([(10, 3), (20, 1)], 4, 8) == (2, 0, 1, 21, 17, False)
    assert plan([(0, 100)], 4, 8) == (0, 7, 1, 0, 0, True)
