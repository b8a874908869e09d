"""Edges of the prompt kernels: rows and columns that cut a box or leave a tile an odd number of them, and attention items in the
forms the persistent kernels walk (one key tile of either parity, many short requests beside a portion, more items than one
list holds)."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def fast():
    from hipinfer_b200.kernels import fast as f
    return f


def rnd(*shape, seed=0, scale=1.0):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn(*shape, generator=g) * scale).to(torch.bfloat16).to(DEV)


def i32(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


# rows around a warp's 32 and a tile's 128; K of one, an odd number and many blocks of 64; more column tiles than CTAs with one box in the last
@pytest.mark.parametrize("M,N,K", [(65, 64, 64), (159, 320, 192), (287, 544, 520), (300, 4128, 64), (1531, 288, 320)])
@pytest.mark.parametrize("tile_n", [128, 256, 512])
def test_rows_that_cut_a_box(M, N, K, tile_n):
    f = fast()
    a, w = rnd(M, K, seed=1), rnd(N, K, seed=2, scale=0.1)
    ref = a.double() @ w.double().T
    tol = 2e-5 * max(1.0, float(ref.abs().max())) * math.sqrt(K)       # 32-bit sums of K products
    for epi in (f.EPI_F32, f.EPI_BF16):
        out = torch.full((M + 1, N), 7.0, dtype=torch.float32 if epi == f.EPI_F32 else torch.bfloat16, device=DEV)
        f.gemm_tc(a, w, out[:M], epi, tile_n)
        torch.cuda.synchronize()
        f.check_status()
        rounding = 0.0 if epi == f.EPI_F32 else 2.0 ** -8              # and one rounding to bfloat16
        assert bool(((out[:M].double() - ref).abs() <= tol + rounding * ref.abs()).all())
        assert bool((out[M] == 7.0).all()), "wrote past the last row"
    act = torch.full((M + 1, N // 2), 7.0, dtype=torch.bfloat16, device=DEV)
    f.gemm_tc(a, w, act[:M], f.EPI_SWIGLU_BF16, tile_n)
    torch.cuda.synchronize()
    f.check_status()
    gu = ref.view(M, N // 32, 2, 16)
    want = (torch.nn.functional.silu(gu[:, :, 0]) * gu[:, :, 1]).reshape(M, N // 2)
    scale = (1.0 + gu.abs()).amax(2).reshape(M, N // 2)                # an error of the sums times the other factor, and the rounding
    assert bool(((act[:M].double() - want).abs() <= 3 * tol * scale + 2.0 ** -8 * want.abs()).all())
    assert bool((act[M] == 7.0).all()), "wrote past the last row"


def test_last_column_of_one_box_over_many_tiles():
    """Two tiles in a row of the same CTA pair whose last column has a single box each: each box leaves before the next fills its place."""
    f = fast()
    M, N, K = 256 * 150, 288, 64
    a, w = rnd(M, K, seed=3), rnd(N, K, seed=4, scale=0.1)
    out = torch.empty(M, N, dtype=torch.float32, device=DEV)
    f.gemm_tc(a, w, out, f.EPI_F32, 512)
    torch.cuda.synchronize()
    f.check_status()
    ref = a.float() @ w.float().T
    assert float((out - ref).abs().max()) < 1e-4 * max(1.0, float(ref.abs().max()))


def attention_case(Hq, Hkv, D, ps, ctx, rows, window, seed):
    """Paged caches with shuffled pages, and the plain result in 64 bits of every request."""
    lens = [c + n for c, n in zip(ctx, rows)]
    pages = [-(-n // ps) for n in lens]
    order = torch.randperm(sum(pages), generator=torch.Generator().manual_seed(seed)).tolist()
    bt = torch.zeros(len(rows), max(pages), dtype=torch.int32)
    at = 0
    for r, n in enumerate(pages):
        bt[r, :n] = torch.tensor(order[at:at + n], dtype=torch.int32)
        at += n
    kc, vc = rnd(at, Hkv, ps, D, seed=seed + 1), rnd(at, Hkv, ps, D, seed=seed + 2)
    T = sum(rows)
    q = rnd(T, Hq * D, seed=seed + 3)
    want = torch.full((T, Hq, D), 7.0, dtype=torch.float64, device=DEV)
    s = 0
    for r, n in enumerate(rows):
        if n >= 16:
            idx = bt[r, :pages[r]].long().to(DEV)
            k, v = (c[idx].transpose(1, 2).reshape(-1, Hkv, D)[:lens[r]].double().repeat_interleave(Hq // Hkv, 1) for c in (kc, vc))
            sc = torch.einsum("thd,shd->hts", q[s:s + n].view(n, Hq, D).double(), k) / math.sqrt(D)
            i, j = torch.arange(ctx[r], lens[r], device=DEV)[:, None], torch.arange(lens[r], device=DEV)[None]
            seen = (j <= i) & (j > i - window if window else j >= 0)
            want[s:s + n] = torch.einsum("hts,shd->thd", torch.softmax(sc.masked_fill(~seen, -math.inf), -1), v)
        s += n
    return q, kc, vc, bt.to(DEV), T, want


# windows that leave one key tile, of an even and of an odd number; short requests (left alone) between portions; portions of one row more
# than a tile; a long context
@pytest.mark.parametrize("D,Hq,Hkv", [(64, 4, 2), (128, 3, 1)])
@pytest.mark.parametrize("ctx,rows,window", [
    ([130, 260, 0], [20, 16, 17], 3),
    ([300] * 40 + [0] + [77] * 20, [1] * 40 + [700] + [1] * 20, 0),
    ([0, 127, 128, 129, 1000], [129, 128, 16, 257, 40], 0),
    ([900, 0, 5], [300, 33, 1], 200),
])
@pytest.mark.parametrize("ps", [8, 16, 128])
def test_attention_items(D, Hq, Hkv, ctx, rows, window, ps):
    q, kc, vc, bt, T, want = attention_case(Hq, Hkv, D, ps, ctx, rows, window, 11)
    out = torch.full((T, Hq * D), 7.0, dtype=torch.bfloat16, device=DEV)
    starts = [sum(rows[:i]) for i in range(len(rows))]
    fast().flash_prefill_tc(q, kc, vc, bt, i32(starts), i32(rows), i32(ctx), out, max(rows), Hq, Hkv, D, ps, window, 1 / math.sqrt(D), 16)
    torch.cuda.synchronize()
    fast().check_status()
    # P and the result are rounded to bfloat16: 2^-9 of values of about 3, and of the result
    torch.testing.assert_close(out.double().view(T, Hq, D), want, rtol=2e-2, atol=2e-2)


def items_behind_one_another(D, tiles):
    """(heads, contexts) of requests of one query tile, 100 rows: for each (key tiles, first key tile) so many items that every CTA walks one
    of them. The list goes by falling work and keeps the order of equals, so a CTA meets them in the order of `tiles`."""
    heads = 16
    ctas = torch.cuda.get_device_properties(0).multi_processor_count * (2 if D == 64 else 1)
    return heads, [128 * (first + n - 1) + 20 for n, first in tiles for _ in range(-(-ctas // heads))]


# key tiles of the items that a CTA walks one behind the other, and the first of them: an item of an odd number hands its chains' stages over
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("tiles,window", [
    ([(5, 0), (3, 0), (3, 0), (2, 0), (1, 0)], 0),
    ([(4, 0), (3, 0), (1, 0)], 0),
    ([(3, 1), (3, 2), (3, 1), (3, 0), (1, 0)], 200),
])
def test_items_of_several_key_tiles_behind_one_another(D, tiles, window):
    """Against 64 bits, and a request's bits are the same as by itself, every time."""
    f = fast()
    Hq, ctx = items_behind_one_another(D, tiles)
    rows, Hkv, ps = [100] * len(ctx), 4, 16
    q, kc, vc, bt, T, want = attention_case(Hq, Hkv, D, ps, ctx, rows, window, 41)
    starts = [sum(rows[:i]) for i in range(len(rows))]
    meta = (i32(starts), i32(rows), i32(ctx))
    call = lambda q, bt, meta, out: f.flash_prefill_tc(q, kc, vc, bt, *meta, out, max(rows), Hq, Hkv, D, ps, window, 1 / math.sqrt(D), 16)
    alone = torch.empty(T, Hq * D, dtype=torch.bfloat16, device=DEV)
    for r, (s, n, c) in enumerate(zip(starts, rows, ctx)):
        call(q[s:s + n], bt[r:r + 1], (i32([0]), i32([n]), i32([c])), alone[s:s + n])
    torch.testing.assert_close(alone.double().view(T, Hq, D), want, rtol=2e-2, atol=2e-2)      # as above
    for _ in range(10):
        out = torch.zeros(T, Hq * D, dtype=torch.bfloat16, device=DEV)
        call(q, bt, meta, out)
        torch.cuda.synchronize()
        f.check_status()
        assert torch.equal(out, alone)


# items whose last tile has pages that are not loaded (and, with a window, whose first one has), behind items of requests with infinities and NaN
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("ps", [8, 16, 64])
@pytest.mark.parametrize("tiles,window", [
    ([(3, 0), (3, 0), (2, 0), (1, 0)], 0),
    ([(3, 1), (3, 2), (3, 1), (1, 0)], 200),
])
def test_items_leave_nothing_to_other_requests(D, ps, tiles, window):
    """Keys and values that are not finite in every second request's cache: the other requests' rows keep every bit."""
    f = fast()
    Hq, ctx = items_behind_one_another(D, tiles)
    n, Hkv = 25, 4                                        # rows to position 44 of the last tile
    q, kc, vc, bt, T, _ = attention_case(Hq, Hkv, D, ps, ctx, [n] * len(ctx), window, 51)
    meta = (i32([n * r for r in range(len(ctx))]), i32([n] * len(ctx)), i32(ctx))
    outs = []
    for bad in (False, True):
        if bad:
            for r in range(0, len(ctx), 2):
                pages = bt[r, :-(-(ctx[r] + n) // ps)].long()
                kc[pages], vc[pages] = (math.nan, math.inf) if r % 4 else (-math.inf, math.nan)
        out = torch.zeros(T, Hq * D, dtype=torch.bfloat16, device=DEV)
        f.flash_prefill_tc(q, kc, vc, bt, *meta, out, n, Hq, Hkv, D, ps, window, 1 / math.sqrt(D), 16)
        torch.cuda.synchronize()
        f.check_status()
        outs.append(out.view(len(ctx), n, -1))
    assert bool(torch.isfinite(outs[0].float()).all()) and bool(torch.isnan(outs[1][::2].float()).all())
    assert torch.equal(outs[0][1::2], outs[1][1::2])


@pytest.mark.parametrize("D", [64, 128])
def test_a_row_whose_scores_are_all_minus_infinity(D):
    """With a sink the denominator is the sink's alone: the row is 0, as far as its values are finite."""
    f = fast()
    Hq, Hkv, ps, n = 2, 1, 16, 200
    q, kc, vc, bt, T, _ = attention_case(Hq, Hkv, D, ps, [0], [n], 0, 71)
    q.view(n, Hq, D)[:, :, 0], q.view(n, Hq, D)[0, :, 0] = 0, 1e30         # the first row, which sees the first key alone, scores it -1e60
    kc[bt[0, 0].long(), :, 0, 0] = -1e30
    sink = torch.tensor([0.5, -3.0], device=DEV)
    out = torch.full((T, Hq * D), 7.0, dtype=torch.bfloat16, device=DEV)
    f.flash_prefill_tc(q, kc, vc, bt, i32([0]), i32([n]), i32([0]), out, n, Hq, Hkv, D, ps, 0, 1 / math.sqrt(D), 16, sink=sink)
    torch.cuda.synchronize()
    f.check_status()
    assert bool((out[0] == 0).all()) and bool(torch.isfinite(out.float()).all())


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("requests,rows,long", [(700, 16, 0), (40, 16, 16000)])      # more requests, and more query tiles, than one list holds
def test_attention_of_more_items_than_a_list(D, requests, rows, long):
    q_len = [rows] * requests + ([long] if long else [])
    ctx = [3] * requests + ([0] if long else [])
    Hq = Hkv = 1
    f = fast()
    q, kc, vc, bt, T, want = attention_case(Hq, Hkv, D, 16, ctx, q_len if not long else q_len[:-1] + [16], 0, 21)
    if long:        # the long portion's rows read their own short prefix: a window of one key
        q_len[-1] = long
        T = sum(q_len)
        q = torch.cat([q[:-16], rnd(long, D, seed=31)])
        pages = -(-long // 16)
        kc = torch.cat([kc, rnd(pages, 1, 16, D, seed=32)])
        vc = torch.cat([vc, rnd(pages, 1, 16, D, seed=33)])
        wide = torch.zeros(len(q_len), pages, dtype=torch.int32, device=DEV)
        wide[:, :bt.shape[1]] = bt
        wide[-1] = torch.arange(kc.shape[0] - pages, kc.shape[0], device=DEV)
        bt = wide
        for window in (1,):
            out = torch.zeros(T, D, dtype=torch.bfloat16, device=DEV)
            f.flash_prefill_tc(q, kc, vc, bt, i32([sum(q_len[:i]) for i in range(len(q_len))]), i32(q_len), i32(ctx), out, long, 1, 1, D, 16,
                               window, 1 / math.sqrt(D), 16)
            torch.cuda.synchronize()
            f.check_status()
            own = vc[bt[-1].long()].transpose(1, 2).reshape(-1, D)[:long]
            assert torch.equal(out[-long:], own)              # a row that sees its own key alone is that key's value
        return
    out = torch.zeros(T, D, dtype=torch.bfloat16, device=DEV)
    f.flash_prefill_tc(q, kc, vc, bt, i32([sum(q_len[:i]) for i in range(len(q_len))]), i32(q_len), i32(ctx), out, max(q_len), 1, 1, D, 16, 0,
                       1 / math.sqrt(D), 16)
    torch.cuda.synchronize()
    f.check_status()
    torch.testing.assert_close(out.double().view(T, 1, D), want, rtol=2e-2, atol=2e-2)


# rows around tiles of 16 and 160; N and K off the tiles of 128 and 64, with slices (few tiles, K of 1,024 and more) and without
@pytest.mark.parametrize("M", [9, 16, 17, 160, 161, 330])
@pytest.mark.parametrize("N,K", [(260, 260), (128, 4100), (20004, 320), (2048, 1024)])
def test_products_of_split_32_bit_operands(M, N, K):
    """Against 64 bits, stored and added. The bound: an MMA's sum is off by at most a unit in its last place, 2^-23 of the terms' magnitudes,
    24 of them a block of 64 k; the blocks' and the slices' sums are rounded to nearest."""
    from hipinfer_b200.kernels import ops

    g = torch.Generator().manual_seed(M + N)
    a = (torch.randn(M, K, generator=g) * torch.exp(3 * torch.randn(M, 1, generator=g))).to(DEV)
    w = (torch.randn(N, K, generator=g) * 0.1).to(DEV)
    ref = a.double() @ w.double().T
    bound = (32 + K / 64) * 2.0 ** -23 * (a.double().abs() @ w.double().abs().T)
    out = torch.full((M + 1, N), 7.0, device=DEV)
    assert fast().linear32(a, w, out[:M], False)
    torch.cuda.synchronize()
    fast().check_status()
    assert bool(((out[:M].double() - ref).abs() <= bound).all()) and bool((out[M] == 7.0).all())
    plain = torch.empty(M, N, device=DEV)
    ops.gemm_plain(a, w, plain)
    assert float((out[:M] - ref).norm()) <= float((plain - ref).norm())          # no less exact than the FFMA chains
    acc = torch.randn(M, N, generator=g).to(DEV)
    want = acc + out[:M]
    assert fast().linear32(a, w, acc, True)
    assert torch.equal(acc, want)


@pytest.mark.parametrize("N,K", [(2048, 8192), (3072, 2048), (260, 1028), (4096, 4096), (20004, 1024)])
def test_split_products_give_a_row_the_same_bits_whatever_the_rows(N, K):
    """From nine rows on: tiles of other widths, more tiles than SMs, flagged rows and weights among them."""
    f = fast()
    g = torch.Generator().manual_seed(N)
    a, w = torch.randn(700, K, generator=g).to(DEV), (torch.randn(N, K, generator=g) * 0.1).to(DEV)
    a[5, 600], a[8] = 3.4e38, a[8] * 1e-35
    w[30, 100], w[200] = math.inf, w[200] * 1e-35
    whole = torch.empty(700, N, device=DEV)
    assert f.linear32(a, w, whole, False)
    for M in (9, 16, 40, 160, 161, 301, 400):
        for start in (0, 700 - M):
            out = torch.empty(M, N, device=DEV)
            assert f.linear32(a[start:start + M], w, out, False)
            assert torch.equal(out.view(torch.int32), whole[start:start + M].view(torch.int32)), (M, start)
    f.check_status()


@pytest.mark.parametrize("M,N,K", [(70, 260, 1028), (200, 20000, 512), (33, 1024, 4096)])
def test_split_operands_that_are_no_sum_of_three(M, N, K):
    """Infinities, NaN, numbers that round to an infinite bfloat16, and rows below the range of their remainders: where FFMA gives an infinity
    or NaN so does this, and the rest is as exact."""
    from hipinfer_b200.kernels import ops

    a, w = torch.randn(M, K, generator=torch.Generator().manual_seed(1)).to(DEV), torch.randn(N, K, generator=torch.Generator().manual_seed(2)).to(DEV) * 0.1
    a[3, 5], a[7, 9], a[20, 100] = math.inf, math.nan, 3.4e38
    w[11, 3], w[130, 200] = -math.inf, 3.39e38
    a[9] *= 1e-30
    a[12] *= 1e-36
    w[77] *= 1e-33
    a[11], w[40] = 0, 0
    plain, out = torch.empty(M, N, device=DEV), torch.empty(M, N, device=DEV)
    ops.gemm_plain(a, w, plain)
    assert fast().linear32(a, w, out, False)
    torch.cuda.synchronize()
    fast().check_status()
    assert torch.equal(torch.isinf(plain), torch.isinf(out)) and torch.equal(torch.isnan(plain), torch.isnan(out))
    fine = torch.isfinite(plain)
    size = a.double().abs() @ w.double().abs().T
    # both within their bounds of the sum, and of a few units of the smallest number
    assert bool(((plain.double() - out.double()).abs() <= (K + 96) * 2.0 ** -23 * size + 2.0 ** -140)[fine].all())


def test_split_products_that_stay_plain():
    """Forms the kernel does not take: few rows, K or rows off four, a view that starts off 16 bytes, other types."""
    f = fast()
    t = lambda *s: torch.zeros(*s, device=DEV)
    assert not f.linear32(t(8, 512), t(512, 512), t(8, 512), False)
    assert not f.linear32(t(16, 510), t(512, 510), t(16, 512), False)
    assert not f.linear32(t(16, 512), t(511, 512), t(16, 511), False)
    assert not f.linear32(t(16, 516)[:, 1:513], t(512, 512), t(16, 512), False)
    assert not f.linear32(t(16, 512), t(512, 512).bfloat16(), t(16, 512), False)
    assert not f.linear32(t(16, 512), t(64, 512), t(16, 64), False)


# widths at and off the steps of the kernel's forms; rows at the lines where it changes from 512 threads a row to 256
@pytest.mark.parametrize("H", [8, 1000, 1024, 2048, 2052, 3072, 4096])
@pytest.mark.parametrize("slices", [1, 3, 4])
def test_norm_of_slices_has_the_same_bits_in_every_form(H, slices):
    """A row's sum and norm do not depend on how many rows there are, nor on whether slices of zeros follow (more than four take another form)."""
    f = fast()
    rows = 300
    g = torch.Generator().manual_seed(H + slices)
    x0, part = torch.randn(rows, H, generator=g).to(DEV), torch.randn(slices, rows, H, generator=g).to(DEV)
    w = rnd(H, seed=61)

    def norm(m, count):
        sl = f.Slices()
        sl.ws = torch.cat([part[:, :m], torch.zeros(count - slices, m, H, device=DEV)]).contiguous()
        sl.ksplit, sl.row_stride, sl.slice_stride, sl.M, sl.N, sl.K, sl.gen = count, H, m * H, m, H, 0, None
        x, y = x0[:m].clone(), torch.empty(m, H, dtype=torch.bfloat16, device=DEV)
        f.add_rmsnorm_slices(x, sl, w, 1e-5, y)
        torch.cuda.synchronize()
        return x, y

    x, y = norm(rows, 6)
    total = x0.double() + part.double().sum(0)
    want = total * torch.rsqrt(total.square().mean(1, keepdim=True) + 1e-5) * w.double()
    torch.testing.assert_close(y.double(), want, rtol=2.0 ** -8, atol=1e-5)       # one rounding to bfloat16 of 32-bit sums
    for m in (1, 9, 148, 149, 296, 297, 300):
        a, b = norm(m, slices)
        assert torch.equal(a, x[:m]) and torch.equal(b, y[:m]), m


def test_launches_of_large_attention_steps():
    """One request, some long ones, and a portion beside hundreds of single rows are one launch; sizes beyond a list are a few."""
    launches = fast()._fn("hb_flash_prefill_tc_launches")
    for D in (64, 128):
        assert launches(32768, 1, 32768, 32, D, 16) == 1
        assert launches(131072, 3, 131072, 32, D, 16) == 1
        assert launches(32768 + 300, 301, 32768, 32, D, 16) == 1
        assert launches(1 << 20, 1, 1 << 20, 32, D, 16) <= 5
        assert launches(1 << 20, 8, 1 << 20, 32, D, 16) <= 40


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("requests,tokens,heads", [(850, 16, 128), (4300, 16, 1), (3, 32000, 128)])
def test_attention_of_more_pairs_than_a_launch_takes(D, requests, tokens, heads):
    """Cut by requests, and by query tiles. Each row sees its own key alone (a window of one), so it is that key's value."""
    f = fast()
    T, ps = requests * tokens, 16
    assert f._fn("hb_flash_prefill_tc_launches")(T, requests, tokens, heads, D, 16) > 1
    q, kc, vc = torch.ones(T, heads * D, dtype=torch.bfloat16, device=DEV), rnd(T // ps, 1, ps, D, seed=82), rnd(T // ps, 1, ps, D, seed=83)
    bt = torch.arange(T // ps, dtype=torch.int32, device=DEV).view(requests, -1)
    out = torch.zeros(T, heads * D, dtype=torch.bfloat16, device=DEV)
    f.flash_prefill_tc(q, kc, vc, bt, i32(list(range(0, T, tokens))), i32([tokens] * requests), i32([0] * requests), out, tokens, heads, 1, D, ps, 1,
                       1 / math.sqrt(D), 16)
    torch.cuda.synchronize()
    f.check_status()
    assert bool((out.view(T, heads, D) == vc.transpose(1, 2).reshape(T, 1, D)).all())


@pytest.mark.parametrize("ctx,rows,window,extras", [
    ([0, 0, 700, 5], [700, 16, 300, 1300], 0, False),        # items of one to eleven key tiles
    ([900, 130], [300, 40], 200, False),
    ([0, 1000], [600, 128], 0, True),
])
def test_both_head_sizes_sum_in_the_same_order(ctx, rows, window, extras):
    """A head of 64 padded with zeros to 128: the scores, the values and with them every bit are those of the kernel for 64, whose tiles
    go through one chain. The scores grow along the keys, so that the maximum is raised again and again."""
    from types import SimpleNamespace

    f = fast()
    Hq, Hkv, ps = 4, 2, 16
    q, kc, vc, bt, T, _ = attention_case(Hq, Hkv, 64, ps, ctx, rows, window, 91)
    for r, n in enumerate(c + m for c, m in zip(ctx, rows)):
        pages = bt[r, :-(-n // ps)].long()
        kc[pages] *= torch.linspace(0.5, 12, len(pages), device=DEV, dtype=torch.bfloat16).view(-1, 1, 1, 1)
    pad = lambda t: torch.cat([t, torch.zeros_like(t)], -1)
    meta = (i32([sum(rows[:i]) for i in range(len(rows))]), i32(rows), i32(ctx))
    kw = {}
    if extras:
        kw = dict(distance=SimpleNamespace(r1=torch.linspace(0, 1, Hq, device=DEV), r2=torch.linspace(0.1, 1, Hq, device=DEV)), sink=torch.linspace(-1, 1, Hq, device=DEV))
    outs = []
    for D, args in ((64, (q, kc, vc)), (128, (pad(q.view(T, Hq, 64)).view(T, -1), pad(kc), pad(vc)))):
        out = torch.zeros(T, Hq * D, dtype=torch.bfloat16, device=DEV)
        f.flash_prefill_tc(*(t.contiguous() for t in args), bt, *meta, out, max(rows), Hq, Hkv, D, ps, window, 0.125, 16, **kw)
        torch.cuda.synchronize()
        f.check_status()
        outs.append(out.view(T, Hq, D))
    assert torch.equal(outs[0], outs[1][:, :, :64]) and bool((outs[1][:, :, 64:] == 0).all())


@pytest.mark.parametrize("tile_n", [128, 192, 256])
def test_single_cta_tiles_with_an_odd_number_of_boxes(tile_n):
    """More tiles than SMs for the kernel without pairs, the last column's of a single box: a box leaves before the next tile fills its place."""
    f = fast()
    M, N, K = 128 * 160, 288, 64
    a, w = rnd(M, K, seed=5), rnd(N, K, seed=6, scale=0.1)
    ref = a.double() @ w.double().T
    tol = 2e-5 * max(1.0, float(ref.abs().max())) * math.sqrt(K)       # 32-bit sums of K products
    for epi in (f.EPI_F32, f.EPI_BF16):
        if epi == f.EPI_BF16 and tile_n == 192:      # 32-bit results only
            continue
        out = torch.full((M, N), 7.0, dtype=torch.float32 if epi == f.EPI_F32 else torch.bfloat16, device=DEV)
        f.gemm_tc(a, w, out, epi, tile_n)
        torch.cuda.synchronize()
        f.check_status()
        rounding = 0.0 if epi == f.EPI_F32 else 2.0 ** -8              # and one rounding to bfloat16
        assert bool(((out.double() - ref).abs() <= tol + rounding * ref.abs()).all())
