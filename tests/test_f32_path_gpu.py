"""The kernels of 32-bit prompt steps: the product in bfloat16 parts (tc_f32.cu) at the edges of its tiles, its blocks and its
pieces of K, nearer to 64 bits than the FFMA product; infinities and NaN; the attention by tiles of 64 queries and keys."""
import math

import pytest
import torch

import kernel_harness as KH

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def K():
    from spissa_b200.csrc import lib
    yield lib
    lib.check_status(DEV)


def operands(M, N, Kd):
    torch.manual_seed(M + 3 * N + Kd)
    return torch.randn(M, Kd, device=DEV), torch.randn(N, Kd, device=DEV) * 0.02


@pytest.mark.parametrize("M", [1, 17, 32, 33, 64, 65, 128, 129, 300])
@pytest.mark.parametrize("N,Kd", [(1, 8), (130, 128), (127, 136), (128, 2048), (260, 1096)])
def test_product_against_64_bits(K, M, N, Kd):
    a, w = operands(M, N, Kd)
    ref = a.double() @ w.double().t()
    size = a.double().abs() @ w.double().abs().t()
    out, ffma = torch.full((M, N), float("nan"), device=DEV), torch.empty(M, N, device=DEV)
    assert K.tc_f32_supported(a, w, out)
    K.tc_f32(a, w, out)
    K.gemm_generic(a, w, ffma)
    # the three products of parts left out are below 2^-21 of |a||w|; a block of 64 terms takes 24 additions that truncate
    # (2^-23 each of what has been added up so far), and K / 64 sums that round
    bound = (2.0 ** -21 + 24 * 2.0 ** -23 + (Kd / 64 + 1) * 2.0 ** -24) * size
    assert bool(((out.double() - ref).abs() <= bound).all())
    if Kd >= 128 and M * N > 1000:
        assert float((out.double() - ref).norm()) <= float((ffma.double() - ref).norm())
    c0 = torch.randn(M, N, device=DEV)
    acc = c0.clone()
    K.tc_f32(a, w, acc, accumulate=True)
    assert torch.equal(acc, c0 + out)                                   # one addition of the same sums


def test_rows_apart_and_operands_it_does_not_take(K):
    a, w = operands(40, 70, 136)
    wide_a, wide_w, wide_c = (torch.full((t.shape[0], t.shape[1] + 8), 9.0, device=DEV) for t in (a, w, torch.empty(40, 70)))
    wide_a[:, :136], wide_w[:, :136] = a, w
    K.tc_f32(wide_a[:, :136], wide_w[:, :136], wide_c[:, 3:73])         # C off a 16-byte boundary
    out = torch.empty(40, 70, device=DEV)
    K.tc_f32(a, w, out)
    assert torch.equal(wide_c[:, 3:73], out) and bool((wide_c[:, :3] == 9.0).all()) and bool((wide_c[:, 73:] == 9.0).all())
    assert not K.tc_f32_supported(a[:, :132], w[:, :132], out)          # K and the rows' distance in eights
    assert not K.tc_f32_supported(a[:, 4:132], w[:, 4:132], out)        # operands off a 32-byte boundary
    assert not K.tc_f32_supported(a.bfloat16(), w, out)
    with pytest.raises(K.KernelError):
        K.tc_f32(a[:, :132], w[:, :132], out)


@pytest.mark.parametrize("M,N,Kd", [(20, 130, 256), (200, 300, 2048)])
def test_infinities_nan_and_extremes(K, M, N, Kd):
    """What a plain float32 sum of products gives: a value that is not finite changes the results it enters and no others."""
    a, w = operands(M, N, Kd)
    a[3, 5], a[7, Kd - 1], a[11, 0] = float("inf"), float("-inf"), float("nan")
    w[9, 17], w[N - 1, 2] = float("inf"), float("nan")
    a[13, 8], w[20, 8] = 3.0e38, 3.0e38                                 # a product beyond the range of float32
    out = torch.empty(M, N, device=DEV)
    K.tc_f32(a, w, out)
    ref = (a.double() @ w.double().t()).float()
    assert torch.equal(torch.isnan(out), torch.isnan(ref))
    assert torch.equal(out[torch.isinf(ref)], ref[torch.isinf(ref)])
    fine = torch.isfinite(ref)
    assert float((out[fine] - ref[fine]).abs().max() / ref[fine].abs().max()) <= 1e-5
    tiny = torch.full((M, Kd), 1e-30, device=DEV)
    K.tc_f32(tiny, w.nan_to_num(0, 0, 0).clamp(-1, 1), out)
    ref = tiny.double() @ w.nan_to_num(0, 0, 0).clamp(-1, 1).double().t()
    assert float((out.double() - ref).norm() / ref.norm()) <= 1e-6


@pytest.mark.parametrize("M", [1, 2, 3, 4, 5, 8, 9, 16])
@pytest.mark.parametrize("N,Kd", [(5, 4), (90, 508), (64, 512), (33, 516), (17, 1024), (40, 1540)])
def test_few_rows_slices_of_k(K, M, N, Kd):
    a, w = operands(M, N, Kd)
    out = torch.empty(M, N, device=DEV)
    K.gemm_generic(a, w, out)
    size = a.double().abs() @ w.double().abs().t()
    # a lane adds Kd / 32 terms in order, then five rounds of sums
    assert bool(((out.double() - a.double() @ w.double().t()).abs() <= (Kd / 32 + 8) * 2.0 ** -24 * size).all())


@pytest.mark.parametrize("M", [1, 4, 5, 16])
@pytest.mark.parametrize("N,Kd", [(9, 1024), (24, 2048), (17, 2564), (9, 3076), (24, 4096), (17, 4612), (3, 5000), (2048, 8192)])
def test_few_rows_columns_shared_by_ctas(K, M, N, Kd):
    a, w = operands(M, N, Kd)
    c0 = torch.randn(M, N, device=DEV)
    out, acc = torch.empty(M, N, device=DEV), c0.clone()
    K.gemm_generic(a, w, out)
    K.gemm_generic(a, w, acc, accumulate=True)
    size = a.double().abs() @ w.double().abs().t()
    # a lane adds Kd / 32 terms or fewer in order, five rounds of sums, at most three sums of pieces
    assert bool(((out.double() - a.double() @ w.double().t()).abs() <= (Kd / 32 + 11) * 2.0 ** -24 * size).all())
    assert torch.equal(acc, out + c0)


def test_short_sums_are_not_shared(K):
    """Where a cluster costs more than it saves (the figures stand at the rule) one CTA takes all of K."""
    pieces = K.load("generic").sp_gemm_f32_pieces
    for N, one, more in ((32, 3072, 4096), (512, 3072, 4096), (1024, 2048, 3072), (2048, 2048, 3072)):
        assert pieces(1, N, one - 1) == pieces(2, N, more - 1) == pieces(4, N, more - 1) == pieces(5, N, 14336) == 1
        assert pieces(1, N, one) > 1 and pieces(2, N, more) > 1 and pieces(4, N, more) > 1
    assert pieces(1, 100000, 8192) == 1


@pytest.mark.parametrize("nh,nkv,hd,vd", [(4, 2, 64, 64), (3, 1, 32, 32), (2, 2, 20, 20), (8, 2, 128, 128), (8, 1, 96, 36), (10, 2, 4, 128)])
@pytest.mark.parametrize("window", [None, 1, 100])
@pytest.mark.parametrize("extra", [False, True])
def test_attention_of_a_decode_step(K, nh, nkv, hd, vd, window, extra):
    before = [0, 1, 63, 64, 511, 512, 700, 2100]
    torch.manual_seed(hd + vd + (window or 0))
    meta = KH.paged_meta([1] * len(before), before, DEV, seed=hd)
    qs = [torch.randn(nh, hd) for _ in before]
    ks = [torch.randn(t, nkv, hd) for t in meta.total_len]
    vs = [torch.randn(t, nkv, vd) for t in meta.total_len]
    k_pool, _ = KH.fill_cache(meta, ks, ks, nkv, hd, torch.float32, DEV)
    v_pool, _ = KH.fill_cache(meta, vs, vs, nkv, vd, torch.float32, DEV)
    q = torch.stack(qs).reshape(-1, nh * hd).to(DEV)
    out = torch.full((len(before), nh * vd), float("nan"), device=DEV)
    sink = torch.randn(nh, device=DEV) if extra else None
    bias = torch.randn(nh, 50, device=DEV) if extra else None
    if extra:
        bias[0, 7:] = float("-inf")                                     # whole batches of keys that a head does not see
    scale = 1.0 / math.sqrt(hd)
    K.attention_generic(q, k_pool, v_pool, out, meta, nh, nkv, hd, window, scale, vd=vd, sink=sink, dist_bias=bias)
    rows = []
    for qb, kb, vb in zip(qs, ks, vs):
        L = kb.shape[0]
        dist = L - 1 - torch.arange(L)
        for h in range(nh):
            s = kb[:, h // (nh // nkv)].double() @ qb[h].double() * scale
            if bias is not None:
                s = s + bias[h].double().cpu()[dist.clamp(0, 49)]
            s = s.masked_fill(dist >= (window or L), float("-inf"))
            if sink is not None:
                s = torch.cat([s, sink[h:h + 1].double().cpu()])
            rows.append(torch.softmax(s, dim=-1)[:L] @ vb[:, h // (nh // nkv)].double())
    ref = torch.cat(rows).view(len(before), nh * vd)
    # as for the tiles below: the error of scores of size sqrt(hd) goes into the weights as a factor
    assert float((out.double().cpu() - ref).abs().max()) <= 3e-6 * float(ref.abs().max())


def test_many_short_sequences_take_no_clusters(K):
    """The lines of the rule (its figures stand there), and both ways' results on the same step."""
    pays = K.load("generic").sp_attention_decode_f32_pays
    for rep, hd, least, few in ((1, 64, 64, 128), (4, 64, 64, 128), (1, 32, 64, 128), (4, 32, 64, 64), (4, 128, 64, 256),
                                (8, 64, 16, 32), (8, 128, 16, 64)):
        for keys, most in ((1, least), (64, least), (65, few), (256, few)):
            assert pays(most, rep, 1, hd, hd, keys) and not pays(most + 1, rep, 1, hd, hd, keys)
        assert pays(256, rep, 1, hd, hd, 257) and bool(pays(257, rep, 1, hd, hd, 512)) == (hd > 32) and pays(9999, rep, 1, hd, hd, 513)
    nh, nkv, hd, B = 4, 2, 64, 70
    torch.manual_seed(3)
    meta = KH.paged_meta([1] * B, [3 * i for i in range(B)], DEV, seed=3)
    kv = [[torch.randn(t, nkv, hd) for t in meta.total_len] for _ in range(2)]
    k_pool, v_pool = KH.fill_cache(meta, *kv, nkv, hd, torch.float32, DEV)
    q = torch.randn(B, nh * hd, device=DEV)
    outs = [torch.full((B, nh * hd), float("nan"), device=DEV) for _ in range(2)]
    for out, longest in zip(outs, (210, 300)):
        K.attention_generic(q, k_pool, v_pool, out, meta, nh, nkv, hd, None, 0.125, longest=longest)
    # two orders of the same sums, each as near to them as the test above allows
    assert float((outs[0] - outs[1]).abs().max()) <= 6e-6 * float(outs[1].abs().max())


def test_a_value_that_is_not_finite_stays_with_its_group(K):
    """A decode step's NaN key and infinite value reach the heads and the sequence that see them, and no others."""
    nh, nkv, hd, before = 4, 2, 64, [600, 600]
    torch.manual_seed(5)
    meta = KH.paged_meta([1, 1], before, DEV, seed=3)
    ks = [torch.randn(t, nkv, hd) for t in meta.total_len]
    vs = [torch.randn(t, nkv, hd) for t in meta.total_len]
    ks[0][17, 0, 3], vs[0][599, 1, 5] = float("nan"), float("inf")
    k_pool, v_pool = KH.fill_cache(meta, ks, vs, nkv, hd, torch.float32, DEV)
    out = torch.zeros(2, nh * hd, device=DEV)
    K.attention_generic(torch.randn(2, nh * hd, device=DEV), k_pool, v_pool, out, meta, nh, nkv, hd, None, 0.125)
    out = out.view(2, nh, hd).cpu()
    assert bool(out[0, :2].isnan().all()) and bool(out[1].isfinite().all())
    assert bool((out[0, 2:, 5] == float("inf")).all()) and bool(out[0, 2:, [i for i in range(hd) if i != 5]].isfinite().all())


@pytest.mark.parametrize("nh,nkv,hd,vd", [(4, 2, 64, 64), (3, 1, 32, 32), (2, 2, 20, 20), (4, 1, 128, 128), (2, 1, 96, 36), (2, 2, 4, 128)])
@pytest.mark.parametrize("window", [None, 1, 63, 100])
@pytest.mark.parametrize("extra", [False, True])
def test_attention_tiles(K, nh, nkv, hd, vd, window, extra):
    new_counts, before = [64, 1, 65, 130, 7], [0, 199, 64, 31, 300]
    torch.manual_seed(hd + vd + (window or 0))
    meta = KH.paged_meta(new_counts, before, DEV, seed=hd)
    qs = [torch.randn(t, nh, hd) for t in meta.total_len]
    ks = [torch.randn(t, nkv, hd) for t in meta.total_len]
    vs = [torch.randn(t, nkv, vd) for t in meta.total_len]
    k_pool, _ = KH.fill_cache(meta, ks, ks, nkv, hd, torch.float32, DEV)
    v_pool, _ = KH.fill_cache(meta, vs, vs, nkv, vd, torch.float32, DEV)
    q = torch.cat([qb[-n:] for qb, n in zip(qs, new_counts)], 0).reshape(-1, nh * hd).to(DEV)
    out = torch.full((q.shape[0], nh * vd), float("nan"), device=DEV)
    sink = torch.randn(nh, device=DEV) if extra else None
    bias = torch.randn(nh, 50, device=DEV) if extra else None
    scale = 1.0 / math.sqrt(hd)
    assert K.attention_tile_f32_supported(q, k_pool, v_pool, len(new_counts), nh, nkv, hd, vd)
    K.attention_tile_f32(q, k_pool, v_pool, out, meta, meta.seq_start, len(new_counts), max(new_counts), nh, nkv, hd, window, scale,
                         vd=vd, sink=sink, dist_bias=bias)
    rows = []
    for qb, kb, vb, n in zip(qs, ks, vs, new_counts):
        L = qb.shape[0]
        dist = torch.arange(L)[:, None] - torch.arange(L)[None, :]
        see = (dist >= 0) & (dist < (window or L))
        heads = []
        for h in range(nh):
            s = qb[:, h].double() @ kb[:, h // (nh // nkv)].double().t() * scale
            if bias is not None:
                s = s + bias[h].double().cpu()[dist.clamp(0, 49)]
            s = s.masked_fill(~see, float("-inf"))
            if sink is not None:
                s = torch.cat([s, sink[h].double().cpu().expand(L, 1)], dim=1)
            p = torch.softmax(s, dim=-1)[:, :L]
            heads.append(p @ vb[:, h // (nh // nkv)].double())
        rows.append(torch.cat(heads, dim=-1)[-n:])
    ref = torch.cat(rows)
    # scores of size sqrt(hd) in float32 sums of hd terms: their error goes into the weights as a factor
    assert float((out.double().cpu() - ref).abs().max()) <= 3e-6 * float(ref.abs().max())


def visible(L, window):
    dist = torch.arange(L)[:, None] - torch.arange(L)[None, :]
    return (dist >= 0) & (dist < (window or L))


@pytest.mark.parametrize("nh,nkv,hd,vd", [(4, 2, 64, 64), (2, 1, 96, 36), (2, 2, 4, 128)])
@pytest.mark.parametrize("window", [None, 1, 20, 100])
@pytest.mark.parametrize("bad", [float("inf"), float("-inf"), float("nan")])
def test_values_that_are_not_finite_reach_who_sees_them(K, nh, nkv, hd, vd, window, bad):
    """A token's value row with an infinity or NaN in it: the tokens that may not see it (earlier ones, and later ones whose
    window has left it behind) keep their results, the others get what a sum over the visible keys gives."""
    new_counts, before = [150, 70], [0, 130]
    torch.manual_seed(hd + (window or 0))
    meta = KH.paged_meta(new_counts, before, DEV, seed=hd)
    qs, ks, vs = ([torch.randn(t, n, d) for t in meta.total_len] for n, d in ((nh, hd), (nkv, hd), (nkv, vd)))
    for b, at in ((0, 40), (0, 127), (1, 100), (1, 150)):               # in front of, within and at the end of tiles of 64
        vs[b][at, 0, vd // 2] = bad
    k_pool, _ = KH.fill_cache(meta, ks, ks, nkv, hd, torch.float32, DEV)
    v_pool, _ = KH.fill_cache(meta, vs, vs, nkv, vd, torch.float32, DEV)
    q = torch.cat([qb[-n:] for qb, n in zip(qs, new_counts)], 0).reshape(-1, nh * hd).to(DEV)
    out = torch.full((q.shape[0], nh * vd), 7.0, device=DEV)
    K.attention_tile_f32(q, k_pool, v_pool, out, meta, meta.seq_start, len(new_counts), max(new_counts), nh, nkv, hd, window,
                         1.0 / math.sqrt(hd), vd=vd)
    rows = []
    for qb, kb, vb, n in zip(qs, ks, vs, new_counts):
        see, heads = visible(qb.shape[0], window), []
        for h in range(nh):
            g = h // (nh // nkv)
            s = (qb[:, h].double() @ kb[:, g].double().t() / math.sqrt(hd)).masked_fill(~see, float("-inf"))
            terms = torch.softmax(s, dim=-1)[:, :, None] * vb[None, :, g].double()
            heads.append(terms.masked_fill(~see[:, :, None], 0.0).sum(1))
        rows.append(torch.cat(heads, dim=-1)[-n:])
    ref, got = torch.cat(rows), out.double().cpu()
    assert torch.equal(torch.isnan(got), torch.isnan(ref))
    assert torch.equal(got[torch.isinf(ref)], ref[torch.isinf(ref)])
    fine = torch.isfinite(ref)
    assert bool((~fine).any()) and float((got[fine] - ref[fine]).abs().max()) <= 3e-6 * float(ref[fine].abs().max())


@pytest.mark.parametrize("window", [None, 33, 64, 100])
def test_distances_that_a_bias_rules_out(K, window):
    """A bias of -inf from a distance on: a tile whose visible keys are all ruled out for a query leaves its sums alone."""
    nh, nkv, hd, L, near = 2, 1, 32, 200, 30
    torch.manual_seed(window or 0)
    meta = KH.paged_meta([L], [0], DEV, seed=3)
    q, k, v = torch.randn(L, nh, hd), torch.randn(L, nkv, hd), torch.randn(L, nkv, hd)
    k_pool, v_pool = KH.fill_cache(meta, [k], [v], nkv, hd, torch.float32, DEV)
    bias = torch.randn(nh, 41)
    bias[:, near:] = float("-inf")
    out = torch.empty(L, nh * hd, device=DEV)
    K.attention_tile_f32(q.reshape(L, -1).to(DEV), k_pool, v_pool, out, meta, meta.seq_start, 1, L, nh, nkv, hd, window, 0.2,
                         dist_bias=bias.to(DEV))
    dist = (torch.arange(L)[:, None] - torch.arange(L)[None, :]).clamp(0, 40)
    heads = []
    for h in range(nh):
        s = (q[:, h].double() @ k[:, 0].double().t() * 0.2 + bias[h].double()[dist]).masked_fill(~visible(L, window), float("-inf"))
        heads.append(torch.softmax(s, dim=-1) @ v[:, 0].double())
    ref = torch.cat(heads, dim=-1)
    assert float((out.double().cpu() - ref).abs().max()) <= 3e-6 * float(ref.abs().max())


@pytest.mark.parametrize("M", [24, 500])
@pytest.mark.parametrize("Kd", [128, 192, 512, 2048])
@pytest.mark.parametrize("kind", ["uniform", "exponential", "all bits"])
def test_product_of_one_sign_is_as_near_as_ffma(K, M, Kd, kind):
    """What the parts leave out and what the accumulator cuts off goes toward zero: operands of one sign add it all up."""
    torch.manual_seed(Kd + M)
    if kind == "uniform":
        a, w = torch.rand(M, Kd, device=DEV), torch.rand(520, Kd, device=DEV)
    elif kind == "exponential":
        a, w = torch.empty(M, Kd, device=DEV).exponential_(), torch.empty(520, Kd, device=DEV).exponential_()
    else:                                                               # every part as large as it can be: 2^-21 is left out
        a, w = (torch.full((n, Kd), 1 + 2.0 ** -7 - 2.0 ** -23, device=DEV) for n in (M, 520))
    out, ffma = (torch.empty(M, 520, device=DEV) for _ in range(2))
    K.tc_f32(a, w, out)
    K.gemm_generic(a, w, ffma)
    ref = a.double() @ w.double().t()
    err = (out.double() - ref).abs()
    assert bool((err <= (2.0 ** -21 + 24 * 2.0 ** -23 + (Kd / 64 + 1) * 2.0 ** -24) * ref).all())
    if kind != "all bits":
        assert float(err.norm()) <= float((ffma.double() - ref).norm())


@pytest.mark.parametrize("size", [1e-33, 1e-36, 1e-38])
def test_values_whose_parts_run_out_of_exponents(K, size):
    a, w = operands(40, 130, 256)
    a *= size
    out = torch.empty(40, 130, device=DEV)
    K.tc_f32(a, w, out)
    ref, terms = a.double() @ w.double().t(), a.double().abs() @ w.double().abs().t()
    bound = (2.0 ** -21 + 24 * 2.0 ** -23 + 5 * 2.0 ** -24) * terms + 2.0 ** -133 * w.double().abs().sum(1) + 2.0 ** -145
    assert bool(((out.double() - ref).abs() <= bound).all())
