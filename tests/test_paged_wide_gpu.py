"""Chunks in tiles of 128 rows: page sizes around a stage of 64 keys, rows around a tile, key ranges, and cache rows that no token may see."""
import pytest
import torch

from test_paged_attention_gpu import _oracle, _step


def _by_wide_tiles(cx, hq, hkv, d, block):
    """The step's portions go by tiles of 128 rows, whatever the rule says of them; whether they do is looked at."""
    from megatronapp_b200 import ops
    from megatronapp_b200.inference.dynamic import key_ranges

    group = hq // hkv
    portions = [p for p in cx._plan if p[2] * group > 16]
    tiles, longest = sum(-(-p[2] * group // 128) for p in portions), max(p[2] + p[3] for p in portions)
    decode, cuts = cx._kernel_plan(group, hkv, d)
    cx._paged_plans[group, hkv, d] = decode, (*cuts[:-2], tiles, key_ranges(2 * tiles * hkv, longest))
    assert ops.ext().paged_chunk_rows(*cx.kv[1], block, tiles) == 128


@pytest.mark.gpu
@pytest.mark.parametrize("reqs,hq,hkv,d,block,dtype", [
    ([(0, 127), (64, 128), (165, 129)], 2, 2, 64, 8, torch.bfloat16),            # a row less and more than a tile, the smallest pages
    ([(63, 200), (0, 70)], 4, 4, 128, 64, torch.float16),                        # a page is a stage
    ([(300, 90), (1, 80)], 8, 2, 128, 128, torch.bfloat16),                      # a page is two
    ([(191, 33), (192, 64), (1000, 1)], 8, 1, 64, 32, torch.float16),            # 16 tokens a tile, stages that end with the context
    ([(5000, 150)], 4, 1, 128, 16, torch.bfloat16),                              # key ranges in a cluster
    ([(1500, 300), (2, 300)], 2, 1, 64, 16, torch.bfloat16)])                    # a tile whose later ranges are empty
def test_wide_tiles(reqs, hq, hkv, d, block, dtype):
    from megatronapp_b200 import ops

    cx, q, k, v = _step(reqs, hq, hkv, d, block, dtype)
    kc, vc = cx.kv[1]
    seen = torch.zeros(kc.shape[0], dtype=torch.bool, device="cuda")
    for i, (a, n) in enumerate(reqs):
        seen[(torch.tensor(cx.seqs[str(i)].blocks).unsqueeze(1) * block + torch.arange(block)).view(-1)[:a + n].cuda()] = True
    kc[~seen], vc[~seen] = float("nan"), float("inf")              # pages of nobody, and what lies behind the last token
    want, _, _ = _oracle(cx, reqs, q, k, v, d ** -0.5, block)
    _by_wide_tiles(cx, hq, hkv, d, block)
    got = cx.attend(1, q, k, v, d ** -0.5)
    unit = 2.0 ** -8 if dtype is torch.bfloat16 else 2.0 ** -11    # the result's own rounding, as in the tests of the other tiles
    assert float((got.double() - want).abs().max()) <= unit * max(1.0, float(want.abs().max()))
    assert float((got.double() - want).norm()) <= 0.5 * unit * float(want.norm())
    assert ops.ext().paged_status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_values_of_later_tokens_stay_out_of_wide_tiles(dtype):
    """Values that are not finite, in both halves of a stage and in its first and last key."""
    reqs = [(60, 260)]
    cx, q, k, v = _step(reqs, 8, 2, 128, 16, dtype)
    v[4, 0, 5], v[67, 0, 127], v[68, 1, 64], v[140, 1, 63] = float("inf"), float("-inf"), float("nan"), float("inf")
    want, _, _ = _oracle(cx, reqs, q, k, v, 0.1, 16)
    _by_wide_tiles(cx, 8, 2, 128, 16)
    got = cx.attend(1, q, k, v, 0.1).double()
    assert torch.equal(torch.isfinite(got), torch.isfinite(want))
    ok = torch.isfinite(want)
    assert ok[:4].all() and not ok[4:, :4, 5].any() and ok[:68, 4:].all()
    assert float((got[ok] - want[ok]).abs().max()) <= 2.0 ** -7


@pytest.mark.gpu
@pytest.mark.parametrize("d", [64, 128])
def test_all_clusters_find_room(d):
    """No more key ranges than let the clusters of all (tile, head) pairs run at once, and no fewer."""
    from megatronapp_b200 import ops

    plan = ops.ext().paged_wide_ranges
    for pairs in (1, 2, 5, 8, 9, 12, 18, 37, 74, 500):
        for asked in (1, 3, 16):
            ranges, resident = plan(pairs, asked, 1, d, True)
            assert ranges in (1, 2, 4, 8, 16) and ranges <= asked and (ranges == 1 or resident >= pairs)
            assert 2 * ranges > asked or plan(1, 2 * ranges, 1, d, True)[1] < pairs
    reqs = [(9000, 32)]                                            # nine clusters of 16 have no room on 148 SMs
    cx, q, k, v = _step(reqs, 9, 9, d, 16, torch.bfloat16)
    want, _, _ = _oracle(cx, reqs, q, k, v, d ** -0.5, 16)
    _by_wide_tiles(cx, 9, 9, d, 16)
    got = cx.attend(1, q, k, v, d ** -0.5)
    assert float((got.double() - want).abs().max()) <= 2.0 ** -8 * max(1.0, float(want.abs().max()))


@pytest.mark.gpu
@pytest.mark.parametrize("reqs,hq,hkv,d,ranges", [
    ([(300, 100), (50, 1), (0, 70)], 4, 2, 64, 1),
    ([(5000, 150)], 4, 1, 128, 8),                                 # a cluster
    ([(1100, 40), (1, 1), (0, 30)], 2, 1, 64, 2)])                 # ... one of whose CTAs has no keys of the second portion
def test_a_wait_that_runs_out_shows(reqs, hq, hkv, d, ranges):
    """Waits that give up at once: the kernel ends by itself, the portions' rows are NaN and the status says so; the next call is sound again."""
    from megatronapp_b200 import ops

    ext, scale = ops.ext(), d ** -0.5
    cx, q, k, v = _step(reqs, hq, hkv, d, 16, torch.bfloat16)
    want, kc, vc = _oracle(cx, reqs, q, k, v, scale, 16)
    tiles = sum(-(-n * (hq // hkv) // 128) for _, n in reqs if n > 1)

    def call(**limit):
        return ext.paged_attention(q, kc, vc, cx._block_table, cx._tok_req, cx._tok_len, 16, scale, sum(n == 1 for _, n in reqs), None, None, None,
                                   cx.packed.cu, 1, 1, 0, 0, False, tiles, ranges, **limit)

    portion = torch.tensor([n > 1 for _, n in reqs for _ in range(n)], device="cuda")
    assert ext.paged_status() == 0
    got = call(wait_limit=0)
    assert ext.paged_status() == 1 and ext.paged_status(True) == 1 and ext.paged_status() == 0
    assert torch.isnan(got[portion]).all() and torch.isfinite(got[~portion]).all()
    got = call()
    assert float((got.double() - want).abs().max()) <= 2.0 ** -8 * max(1.0, float(want.abs().max()))
    assert ext.paged_status() == 0


@pytest.mark.gpu
def test_which_pages_go_by_which_tiles():
    """Whole pages to a stage of 64 keys, or whole stages to a page, of a multiple of eight slots: 128 rows where the plan has such tiles, 64 rows elsewhere."""
    from megatronapp_b200 import ops

    for d in (64, 128):
        cache = torch.empty(768, 2, d, dtype=torch.bfloat16, device="cuda")
        assert [ops.ext().paged_chunk_rows(cache, cache, b, 1) for b in (8, 16, 32, 64, 128, 192, 4, 12, 24, 48, 96)] == [128] * 6 + [64] * 5
        assert ops.ext().paged_chunk_rows(cache, cache, 16, 0) == 64


@pytest.mark.gpu
@pytest.mark.parametrize("scale", [0.1, -0.5, 0.0])
@pytest.mark.parametrize("reqs,hq,hkv,d,ranges,dtype", [
    ([(9000, 30)], 8, 2, 128, 16, torch.bfloat16),
    ([(5000, 30), (3, 1)], 4, 4, 64, 16, torch.float16),
    ([(1100, 40), (0, 20)], 4, 1, 64, 4, torch.float16)])           # a tile whose later ranges are empty
def test_key_ranges_of_64_row_tiles(reqs, hq, hkv, d, ranges, dtype, scale):
    """Pages that only the 64-row tiles take: their clusters' merge."""
    from megatronapp_b200 import ops

    cx, q, k, v = _step(reqs, hq, hkv, d, 24, dtype)
    want, _, _ = _oracle(cx, reqs, q, k, v, scale, 24)
    assert cx._kernel_plan(hq // hkv, hkv, d)[1][1] == ranges and ops.ext().paged_chunk_rows(*cx.kv[1], 24, 1) == 64
    got = cx.attend(1, q, k, v, scale)
    unit = 2.0 ** -8 if dtype is torch.bfloat16 else 2.0 ** -11
    # scores of up to 50: their own fp32 rounding moves a weight by 2^-18
    assert float((got.double() - want).abs().max()) <= unit * max(1.0, float(want.abs().max()))
