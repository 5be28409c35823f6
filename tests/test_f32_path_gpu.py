"""The 32-bit path's product and attention: every kernel a batch may go to gives a row the same bits."""
from __future__ import annotations

import pytest
import torch

import plain_kernels as P
from test_kernels_gpu import DEV, K, _cache_case, _Ctx, randn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k", [(130, 257), (130, 260), (33, 16), (16, 5), (513, 129), (3072, 128)])
def test_product_rows_have_the_same_bits_in_every_kernel(n, k):
    """1 to 16 rows take the kernel of decode steps, more take tiles of 32 or 64 rows (128: see below); edges of all of them.
    The error of a sum of k products, each addition rounded: below k/2 units of 2^-24 of the terms' magnitudes."""
    x, w = randn(700, k, dtype=torch.float32, seed=1), randn(n, k, dtype=torch.float32, seed=2)
    bias = randn(n, dtype=torch.float32, seed=3)
    full = K().linear(x, w, bias)
    bound = (x.double().abs() @ w.double().abs().T + bias.double().abs()) * ((k + 2) * 2.0 ** -24)
    assert ((full.double() - (x.double() @ w.double().T + bias.double())).abs() <= bound).all()
    for rows in (1, 7, 8, 9, 16, 17, 32, 33, 64, 65, 128, 129, 300):
        assert torch.equal(K().linear(x[:rows].contiguous(), w, bias), full[:rows]), rows
    wide = torch.zeros(20, k + 3, dtype=torch.float32, device=DEV)          # rows that start off 16-byte boundaries
    wide[:, 3:] = x[:20]
    assert torch.equal(K().linear(wide[:, 3:], w, bias), full[:20])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("heads,kv_heads,dim,page,window,keep", [
    (6, 2, 128, 16, None, 0), (4, 2, 16, 16, None, 0), (3, 1, 72, 8, None, 0), (4, 4, 256, 32, None, 0), (4, 1, 130, 4, None, 0),
    (6, 2, 64, 16, 100, 0), (6, 2, 128, 16, 300, 0), (4, 1, 64, 16, 70, 65), (24, 2, 32, 16, 33, 5)])
def test_attention_rows_have_the_same_bits_in_every_kernel(dtype, heads, kv_heads, dim, page, window, keep):
    """A prompt in tiles of 64 rows against its last tokens alone, whose segments are read by different blocks; lengths
    around segments (256) and chunks (64)."""
    for total in (1, 63, 257, 513, 700):
        case = _cache_case(dtype, heads, kv_heads, dim, page, [(0, total)], seed=total)

        def run(first, count, reserved):
            part = dict(case, positions=case["positions"][first:first + count], lens=[(first, count)],
                        req_index=case["req_index"][first:first + count],
                        query_start=torch.tensor([0, count], dtype=torch.int32, device=DEV),
                        context_lens=torch.tensor([first], dtype=torch.int32, device=DEV))
            ctx = _Ctx(part)
            ctx.max_seq_len_bound = first + count + reserved
            return K().paged_attention(case["qkv"][first:first + count], case["k_cache"], case["v_cache"], case["table"], ctx,
                                       heads, kv_heads, dim, dim ** -0.5, window, keep_first=keep, force_general=True)
        whole = run(0, total, 0)
        for count in (1, 2, 8, 40):
            if count <= total:
                assert torch.equal(run(total - count, count, 600), whole[total - count:]), (total, count)
        want = P.paged_attention_plain(case["qkv"], case["k_cache"], case["v_cache"], case["table"], case["positions"],
                                       case["req_index"], heads, kv_heads, dim, dim ** -0.5, window, keep)
        torch.testing.assert_close(whole, want, **(dict(rtol=2e-5, atol=2e-5) if dtype == torch.float32
                                                   else dict(rtol=2e-2, atol=2e-2)))
    assert K().read_status() == 0


def _attention(dtype, heads, kv_heads, dim, page, lens, window=None, keep=0, seed=1):
    """A batch for the general attention kernels, and the call on caches of the caller's."""
    case = _cache_case(dtype, heads, kv_heads, dim, page, lens, seed=seed)

    def attend(k_cache, v_cache, qkv=case["qkv"]):
        return K().paged_attention(qkv, k_cache, v_cache, case["table"], _Ctx(case), heads, kv_heads, dim, dim ** -0.5, window,
                                   keep_first=keep, force_general=True)
    return case, attend


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("window,keep", [(None, 0), (40, 0), (70, 9)])
def test_values_a_row_does_not_see_do_not_count(dtype, value, window, keep):
    """Keys and values of one position hold no number: rows in front of it, and rows whose window lies behind it, keep their
    bits, rows that see it do not hide it.  A prompt (tiles of 64 rows), its last 2 tokens (a block a segment), and
    what the pages hold behind the last position."""
    heads, kv_heads, dim, page, total = 6, 2, 40, 16, 333
    for first, count in ((0, total), (total - 2, 2)):
        case, attend = _attention(dtype, heads, kv_heads, dim, page, [(first, count)], window, keep)
        want = attend(case["k_cache"], case["v_cache"])
        position = torch.arange(first, first + count, device=DEV)
        for at in (0, 7, 100, 255, 256, 300, total - 2, total - 1, total + 1):
            planes = [case["k_cache"].clone(), case["v_cache"].clone()]
            for plane in planes[1:] if value == float("inf") else planes:
                plane[int(case["table"][0, at // page]), :, at % page] = value
            got = attend(*planes)
            sees = position >= at
            if window is not None:
                sees &= (position - window < at) | (at < keep)
            assert torch.equal(got[~sees], want[~sees]), at
            assert (~torch.isfinite(got[sees].float())).all(), at
    assert K().read_status() == 0


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("dim", [40, 128])
def test_a_chunk_without_weight_does_not_count_however_the_rows_are_cut(dtype, dim):
    """Every score of 64 positions is -infinity and their values are infinite: rows of a prompt's tiles, decoded tokens with one
    block and with one a chunk have the bits that they have where those values are zero."""
    heads, kv_heads, page, total = 6, 2, 16, 300
    case, attend = _attention(dtype, heads, kv_heads, dim, page, [(0, total)])
    qkv, planes = case["qkv"].clone(), [case["k_cache"].clone(), case["v_cache"].clone()]
    qkv[:, : heads * dim : dim] = qkv[:, : heads * dim : dim].abs() + 0.5
    for at in range(64, 128):
        planes[0][int(case["table"][0, at // page]), :, at % page, 0] = float("-inf")
        planes[1][int(case["table"][0, at // page]), :, at % page] = 0.0
    want = attend(*planes, qkv)
    for at in range(64, 128):
        planes[1][int(case["table"][0, at // page]), :, at % page] = float("inf")
    assert want.isfinite().all() and torch.equal(attend(*planes, qkv), want)
    for at in (63, 64, 100, 127, 128, 255, 299):
        one = dict(case, positions=case["positions"][at:at + 1], lens=[(at, 1)], req_index=case["req_index"][:1],
                   query_start=torch.tensor([0, 1], dtype=torch.int32, device=DEV),
                   context_lens=torch.tensor([at], dtype=torch.int32, device=DEV))
        ctx = _Ctx(one)
        for bound in (at + 1, 2000):
            ctx.max_seq_len_bound = bound
            got = K().paged_attention(qkv[at:at + 1], *planes, case["table"], ctx, heads, kv_heads, dim, dim ** -0.5, None,
                                      force_general=True)
            assert torch.equal(got, want[at:at + 1]), (at, bound)
    assert K().read_status() == 0


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_a_query_that_is_no_number_is_not_hidden(dtype):
    """All of a row's scores are NaN, in one segment or several: so is its result, as that of plain attention."""
    for lens in ([(0, 70)], [(0, 300)], [(700, 1)], [(100, 1)]):
        case, attend = _attention(dtype, 4, 2, 64, 16, lens)
        qkv = case["qkv"].clone()
        qkv[-1, 64:128] = float("nan")                # the last token's second head
        got, want = attend(case["k_cache"], case["v_cache"], qkv), attend(case["k_cache"], case["v_cache"])
        assert got[-1, 64:128].isnan().all()
        got[-1, 64:128] = want[-1, 64:128]
        assert torch.equal(got, want)


def test_scratch_of_few_rows_is_bounded():
    """One long context beside many short ones: the scratch is bounded, whatever the longest asks for, and requests that are
    taken in several lots have the bits they have alone."""
    heads, kv_heads, dim, page = 16, 8, 64, 16
    lens = [(60000, 1)] + [(50 + 7 * i, 1) for i in range(99)]
    case, attend = _attention(torch.float32, heads, kv_heads, dim, page, lens)
    attend(case["k_cache"], case["v_cache"])
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    got = attend(case["k_cache"], case["v_cache"])
    assert torch.cuda.max_memory_allocated() - before <= (64 << 20) + 2 * got.nbytes
    for row in (0, 1, 37, 99):
        part = dict(case, positions=case["positions"][row:row + 1], lens=[lens[row]], req_index=case["req_index"][:1],
                    query_start=case["query_start"][:2], context_lens=case["context_lens"][row:row + 1])
        alone = K().paged_attention(case["qkv"][row:row + 1], case["k_cache"], case["v_cache"], case["table"][row:row + 1],
                                    _Ctx(part), heads, kv_heads, dim, dim ** -0.5, None)
        assert torch.equal(alone, got[row:row + 1])
    assert K().read_status() == 0


@pytest.mark.parametrize("heads,kv_heads,dim,window,keep", [(6, 2, 128, None, 0), (32, 1, 64, None, 0), (4, 2, 16, 50, 7), (8, 8, 256, None, 0)])
def test_short_portions_have_the_bits_of_tiles(heads, kv_heads, dim, window, keep):
    """Portions around 8 rows, 32 tokens and the end of the first segment, alone and beside one another, with a bound on the
    positions that is exact and one that is not: the bits of a whole prompt in tiles."""
    case, attend = _attention(torch.float32, heads, kv_heads, dim, 16, [(0, 300)], window, keep)
    whole = attend(case["k_cache"], case["v_cache"])
    parts = [(0, 1), (0, 3), (0, 9), (0, 32), (0, 33), (224, 32), (225, 32), (223, 33), (249, 7), (250, 7), (299, 1)]
    for batch in [[part] for part in parts] + [parts, parts[:4] + parts[5:6]]:
        rows = torch.cat([torch.arange(first, first + count, device=DEV) for first, count in batch])
        ctx = _Ctx(dict(case, positions=rows.to(torch.int32), lens=batch, req_index=None,
                        query_start=torch.tensor([0] + [n for _, n in batch], device=DEV).cumsum(0).to(torch.int32),
                        context_lens=torch.tensor([c for c, _ in batch], dtype=torch.int32, device=DEV)))
        for bound in (max(c + n for c, n in batch), 2000):
            ctx.max_seq_len_bound = bound
            got = K().paged_attention(case["qkv"][rows].contiguous(), case["k_cache"], case["v_cache"],
                                      case["table"].repeat(len(batch), 1), ctx, heads, kv_heads, dim, dim ** -0.5, window,
                                      keep_first=keep, force_general=True)
            assert torch.equal(got, whole[rows]), (batch, bound)
    assert K().read_status() == 0


@pytest.mark.parametrize("m,n,k,tile", [(600, 28673, 36, 128), (620, 28676, 33, 128), (700, 3072, 131, 64), (513, 3100, 260, 64),
                                        (300, 515, 67, 32)])
def test_product_rows_have_the_same_bits_in_every_tile(m, n, k, tile):
    """Sizes that the rule sends to tiles of 128, 64 and 32 rows (rounds of 148 SMs; see kvb_gemm_f32), each with ragged
    rows and columns, read in pieces of four and one by one: against the kernel of decode steps."""
    rounds = lambda tm, tn: -(-(-(-m // tm) * -(-n // tn)) // K().api.sm_count(torch.device(DEV)))  # noqa: E731
    cost = {128: 266.0 if rounds(128, 128) < 2 else 210.0 * rounds(128, 128), 64: 58.0 * max(2.2, rounds(64, 64)),
            32: 38.0 * max(2.7, rounds(32, 64))}
    assert min(cost, key=cost.get) == tile
    x, w = randn(m, k, dtype=torch.float32, seed=1), randn(n, k, dtype=torch.float32, seed=2)
    bias = randn(n, dtype=torch.float32, seed=3)
    full = K().linear(x, w, bias)
    for first in (0, 63, 127, 240, m - 16):
        assert torch.equal(K().linear(x[first:first + 16].contiguous(), w, bias), full[first:first + 16]), first


@pytest.mark.parametrize("n,k", [(128, 2048), (130, 2052), (515, 2108), (9601, 2048), (3072, 3072), (16390, 2064)])
def test_product_in_pieces_has_the_same_bits_for_every_number_of_rows(n, k):
    """Weights from K 2,048 on: tiles of 16 to 128 rows, ragged columns, k and last chunks, one stretch of K and several; rows
    off 16-byte boundaries.  A float is three bf16 exactly and three of nine products are left out (2^-24 of a term in all);
    a chunk's accumulator may lose one unit of 2^-23 at each of 24 additions of up to its 64 terms, 2^-18.4 of them; and
    k / 64 + 16 sums are rounded to nearest."""
    x, w = randn(300, k, dtype=torch.float32, seed=1), randn(n, k, dtype=torch.float32, seed=2)
    bias = randn(n, dtype=torch.float32, seed=3)
    full = K().linear(x, w, bias)
    terms = x.double().abs() @ w.double().abs().T + bias.double().abs()
    error = (full.double() - (x.double() @ w.double().T + bias.double())).abs()
    assert (error <= terms * (24 * 2.0 ** -23 + (k / 64 + 20) * 2.0 ** -24)).all()
    by_fma = K().api
    out = torch.empty_like(full)
    by_fma._call("kvb_gemm_f32", out.data_ptr(), x.data_ptr(), w.data_ptr(), bias.data_ptr(), 300, n, k, k, n, by_fma._stream())
    assert error.norm() <= (out.double() - (x.double() @ w.double().T + bias.double())).norm()
    for rows in (1, 16, 17, 32, 33, 64, 65, 128, 129, 200):
        assert torch.equal(K().linear(x[:rows].contiguous(), w, bias), full[:rows]), rows
    wide = torch.zeros(20, k + 3, dtype=torch.float32, device=DEV)
    wide[:, 3:] = x[:20]
    assert torch.equal(K().linear(wide[:, 3:], w, bias), full[:20])
    assert K().read_status() == 0


@pytest.mark.parametrize("rows,n,k", [(4300, 2048, 2048), (2101, 6144, 3072)])
def test_product_in_pieces_takes_many_rows_in_lots(rows, n, k):
    """More rows than the scratch for sums of stretches holds: the pieces, the sums and the rows' map are the next lot's while the
    lot in front is being added up.  Rows on both sides of every lot's end, of x whose rows lie apart, into rows that lie apart."""
    x, w = randn(rows, 2, k, dtype=torch.float32, seed=1), randn(2, n, k, dtype=torch.float32, seed=2)
    K().api.ensure_built()
    launches = lambda m: K().api._lib.kvb_gemm_f32_split_launches(m, n, k)  # noqa: E731
    lot = next(m for m in range(128, rows, 128) if launches(m + 1) > launches(m))
    assert launches(rows) == -(-rows // lot) * launches(1) and launches(1) == 3
    got = K().heads_linear(x, w)
    for h in range(2):
        for first in [0, rows - 16] + [end - 9 for end in range(lot, rows, lot)]:
            assert torch.equal(K().linear(x[first:first + 16, h].contiguous(), w[h]), got[first:first + 16, h]), (h, first)
        assert ((got[:, h].double() - x[:, h].double() @ w[h].double().T).norm() <= 2.0 ** -21 * got[:, h].double().norm())
    assert K().read_status() == 0


def test_product_in_pieces_of_numbers_that_are_not_finite_or_too_large_for_bf16():
    """Infinities, NaN, numbers above the largest bf16 and sums that leave the range: as the product by FMA has them."""
    x, w = randn(40, 2048, dtype=torch.float32, seed=1), randn(256, 2048, dtype=torch.float32, seed=2)
    x[3, 5] = float("inf")
    x[4, 7] = float("nan")
    x[5, 64], x[5, 65] = float("inf"), float("-inf")
    x[6, 0] = 3.4e38
    w[9, 0] = 0.0
    w[:, 5][17] = 0.0
    w[20, 100] = float("-inf")
    w[21, 2047] = float("nan")
    x[30] *= 2.0 ** 126
    w[30] *= 2.0 ** 126
    x[31] *= 2.0 ** -100
    got, api = K().linear(x, w), K().api
    want = torch.empty_like(got)
    api._call("kvb_gemm_f32", want.data_ptr(), x.data_ptr(), w.data_ptr(), None, 40, 256, 2048, 2048, 256, api._stream())
    assert torch.equal(got.isnan(), want.isnan())
    assert torch.equal(got.isinf(), want.isinf()) and torch.equal(got[got.isinf()], want[want.isinf()])
    both = want.isfinite()
    terms = (x.double().nan_to_num(0, 0, 0).abs() @ w.double().nan_to_num(0, 0, 0).abs().T)[both]
    assert ((got - want)[both].double().abs() <= terms * 2049 * 2.0 ** -24).all()


@pytest.mark.parametrize("m,n,k", [(150, 300, 2052), (33, 515, 2048), (5, 16390, 2064), (130, 19000, 2048)])
def test_product_in_pieces_whose_rows_or_columns_are_not_finite(m, n, k):
    """Infinities through a whole column of weights, a row of weights, a row of x and NaN behind them, one stretch of K and
    several, rows of x on 16-byte boundaries and off them: every output is what the product by FMA has for it, or finite in both."""
    api, room = K().api, torch.zeros(m, k + 1, dtype=torch.float32, device=DEV)
    for where in ("column", "row", "x", "all"):
        x, w = randn(m, k, dtype=torch.float32, seed=1), randn(n, k, dtype=torch.float32, seed=2)
        if where in ("column", "all"):
            w[:, 5] = float("inf")
        if where in ("row", "all"):
            w[n - 1, k - 1] = float("-inf")
        if where in ("x", "all"):
            x[m - 1, 70], x[1, k - 2], x[2] = float("inf"), float("nan"), 3e38
        room[:, 1:] = x
        want = torch.empty(m, n, dtype=torch.float32, device=DEV)
        api._call("kvb_gemm_f32", want.data_ptr(), x.data_ptr(), w.data_ptr(), None, m, n, k, k, n, api._stream())
        assert not want.isfinite().all()
        for rows in (x, room[:, 1:]):
            got = K().linear(rows, w)
            assert torch.equal(got.isnan(), want.isnan()), where
            assert torch.equal(got.isinf(), want.isinf()) and torch.equal(got[got.isinf()], want[want.isinf()]), where
    assert K().read_status() == 0


@pytest.mark.parametrize("most", [45, 4])
def test_product_in_pieces_that_is_not_finite_does_not_stall(most):
    """An infinite column of weights makes every output infinite, an infinite number of x a row: below 45 and 4 times the product
    by FMA (22 and 1.8 as measured; 94 and 6.4 with one output behind the other)."""
    api, (m, n, k) = K().api, (256, 5120, 3072)
    x, w = randn(m, k, dtype=torch.float32, seed=1), randn(n, k, dtype=torch.float32, seed=2)
    where = w[:, 5] if most == 45 else x[0, 5:6]
    where.fill_(float("inf"))
    out, times = torch.empty(m, n, dtype=torch.float32, device=DEV), []
    for call in (lambda: api._call("kvb_gemm_f32", out.data_ptr(), x.data_ptr(), w.data_ptr(), None, m, n, k, k, n, api._stream()),
                 lambda: K().linear(x, w)):
        taken = []
        for _ in range(4):
            begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            begin.record()
            call()
            end.record()
            torch.cuda.synchronize()
            taken.append(begin.elapsed_time(end))
        times.append(min(taken))
    assert times[1] < most * times[0], times


@pytest.mark.parametrize("down,up", [(60, 0), (100, 0), (110, 20), (114, 40), (118, 60), (123, 60)])
@pytest.mark.parametrize("n,k", [(130, 2052), (3072, 2048)])
def test_product_in_pieces_of_small_numbers_keeps_their_bits(n, k, down, up):
    """Numbers between 2^-3 and 2^3, times an exact power of two that leaves them floats of 24 bits: the result of the unscaled
    ones times that power, whichever side is small.  Down to 2^-117 bit for bit; below, pieces that are no normal numbers stand
    lower in the pipe than the others, which may turn a rounding: as far from 64 bits as the unscaled ones, but for a quarter
    (without the third piece it would be ten times as far)."""
    apart = lambda t: t + torch.copysign(torch.full_like(t, 0.125), t)  # noqa: E731
    x, w = (apart(randn(20, k, dtype=torch.float32, seed=1).clamp(-7, 7)), apart(randn(n, k, dtype=torch.float32, seed=2).clamp(-7, 7)))
    assert torch.equal(x * 2.0 ** -down * 2.0 ** down, x)
    plain, exact, back = K().linear(x, w).double(), x.double() @ w.double().T, 2.0 ** (down - up)
    assert ((plain.float() / back).abs() > 2.0 ** -120).float().mean() > 0.99
    for got in (K().linear(x * 2.0 ** -down, w * 2.0 ** up), K().linear(x * 2.0 ** up, w * 2.0 ** -down)):
        if down <= 114:
            assert torch.equal(got, (plain / back).float())
        assert (got.double() * back - exact).norm() <= 1.25 * (plain - exact).norm()
    assert K().read_status() == 0


def test_product_in_pieces_of_numbers_below_the_smallest_normal_float():
    """Whole multiples of 2^-149 are three bf16 exactly too; in the pipe a number below 2^-126 stands as high as 2^-126: the bound
    of ordinary numbers for these, half of 2^-149 of a number a term."""
    k = 2048
    x = torch.randint(-(1 << 23), 1 << 23, (20, k), generator=torch.Generator().manual_seed(1)).to(DEV)
    x[10:] >>= 12
    x, w = (x.double() * 2.0 ** -149).float(), randn(200, k, dtype=torch.float32, seed=2) * 2.0 ** 100
    error = (K().linear(x, w).double() - x.double() @ w.double().T).abs()
    assert (error <= 2.0 ** -126 * w.double().abs().sum(1) * (24 * 2.0 ** -23 + (k / 64 + 20) * 2.0 ** -24)).all()


@pytest.mark.parametrize("terms", [1, 2, 3, 5, 16])
@pytest.mark.parametrize("numbers", ["random", "worst"])
def test_product_in_pieces_of_few_terms(terms, numbers):
    """Sums of few terms that are not zero, also of numbers whose pieces left out are the largest (2^-24 of a term in all, all of
    one sign): each term may cost the accumulator one unit of 2^-23 and, but for the first, the sum proper 2^-24; the sums of
    smaller pieces may lose 0.3 of 2^-24 at most."""
    x, w = torch.zeros(32, 2048, device=DEV), randn(256, 2048, dtype=torch.float32, seed=2)
    values = randn(32, terms, dtype=torch.float32, seed=3)
    if numbers == "worst":
        worst = 1 + 2.0 ** -8 - 2.0 ** -16 + 2.0 ** -17 - 2.0 ** -23
        values, w = torch.full_like(values, worst), torch.full_like(w, worst)
    for r in range(32):
        x[r, torch.randperm(2048, generator=torch.Generator().manual_seed(r))[:terms].to(DEV)] = values[r]
    error = (K().linear(x, w).double() - x.double() @ w.double().T).abs()
    assert (error <= (x.double().abs() @ w.double().abs().T) * (3 * terms + 0.3) * 2.0 ** -24).all()


def test_heads_product_in_pieces():
    x, w = randn(20, 3, 2048, dtype=torch.float32, seed=1), randn(3, 130, 2048, dtype=torch.float32, seed=2)
    got = K().heads_linear(x, w)
    for h in range(3):
        assert torch.equal(got[:, h], K().linear(x[:, h].contiguous(), w[h]))
