"""The product with W's rows as the instruction's M and up to 256 tokens as its N (tc_mid.cu), at the sizes where its tiles
end: tokens that are no multiple of 16, several token tiles, pieces of K that are not equally long, rows of W that do not
fill a tile; and every epilogue in the divisions that the sizes choose."""
import pytest
import torch

import kernel_harness as KH
from plain import llama_plain as P

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def K():
    from spissa_b200.csrc import lib
    yield lib
    lib.check_status(DEV)


def within(got, a, w, extra=None, rel=0.0):
    """Against the exact sum of the bfloat16 products. A float32 sum of K terms in any order is off by less than
    K · 2^-23 · Σ|a||w| (2^-24 for each addition that rounds to nearest, twice that where it truncates); ``rel``: the
    storage's rounding of the result."""
    ref, size = a.double() @ w.double().t(), a.double().abs() @ w.double().abs().t()
    if extra is not None:
        ref, size = ref + extra.double(), size + extra.double().abs()
    bound = a.shape[1] * 2.0 ** -23 * size + rel * ref.abs() + 1e-30
    assert bool(((got.double() - ref).abs() <= bound).all())


def operands(M, N, Kd, seed=0):
    torch.manual_seed(M * 7 + N + Kd + seed)
    return torch.randn(M, Kd, device=DEV).bfloat16(), (torch.randn(N, Kd, device=DEV) * 0.1).bfloat16()


@pytest.mark.parametrize("M", [1, 16, 17, 33, 160, 161, 256, 257, 301, 1023])
@pytest.mark.parametrize("N,Kd", [(8, 8), (136, 72), (128, 2048), (3072, 2048), (72, 1096)])
def test_store_and_accumulate(K, M, N, Kd):
    a, w = operands(M, N, Kd)
    tiles, nt, pieces, stages = K.tc_mid_plan(K.TC_STORE, M, N, Kd)
    assert nt % 16 == 0 and nt <= 256 and (tiles - 1) * nt < M <= tiles * nt and stages >= 1
    blocks = -(-Kd // 64)
    assert (pieces - 1) * -(-blocks // pieces) < blocks                 # no CTA of a cluster without a block of K
    out = torch.full((M, N), float("nan"), device=DEV)
    assert K.tc_mid_supported(a, w, out)
    K.tc_mid(a, w, out)
    within(out, a, w)
    short = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=DEV)
    K.tc_mid(a, w, short)
    within(short, a, w, rel=2.0 ** -8)
    c0 = torch.randn(M, N, device=DEV)
    acc, again = c0.clone(), c0.clone()
    K.tc_mid(a, w, acc, K.TC_ACCUMULATE)
    within(acc, a, w, extra=c0)
    K.tc_mid(a, w, again, K.TC_ACCUMULATE)
    assert torch.equal(acc, again)                                      # a fixed order of sums


def test_rows_further_apart_than_they_are_long(K):
    a, w = operands(70, 264, 136)
    wide_a, wide_w, wide_c = (torch.full((t.shape[0], t.shape[1] + 24), 9.0, dtype=t.dtype, device=DEV)
                              for t in (a, w, torch.empty(70, 264)))
    wide_a[:, :136], wide_w[:, :136] = a, w
    K.tc_mid(wide_a[:, :136], wide_w[:, :136], wide_c[:, :264])
    within(wide_c[:, :264], a, w)
    assert bool((wide_c[:, 264:] == 9.0).all())


def test_operands_it_does_not_take(K):
    a, w = operands(64, 256, 128)
    out = torch.empty(64, 256, device=DEV)
    assert K.tc_mid_supported(a, w, out)
    assert not K.tc_mid_supported(a, w, torch.empty(64, 258, device=DEV)[:, 1:257])          # C off a 16-byte boundary
    assert not K.tc_mid_supported(a[:, 1:125], w[:, 1:125], out)
    assert not K.tc_mid_supported(a, w[:252], out[:, :252])                                  # rows of W in eights
    assert not K.tc_mid_supported(a, w, torch.empty(64, 128, device=DEV), K.TC_SILU_MUL, 64)
    with pytest.raises(K.KernelError):
        K.tc_mid(a, w, torch.empty(64, 128, device=DEV), K.TC_SILU_MUL, 64)
    with pytest.raises(K.KernelError):
        K.tc_mid(a, w, torch.empty(64, 256, dtype=torch.bfloat16, device=DEV), K.TC_ACCUMULATE)
    K.check_status(DEV)


@pytest.mark.parametrize("M,I,H", [(20, 128, 264), (64, 8192, 2048), (100, 8192, 2048), (301, 1024, 512), (700, 2048, 2048), (257, 128, 4096)])
@pytest.mark.parametrize("act", ["silu", "gelu", "clamped"])
def test_gated_rows(K, M, I, H, act):
    """With rows scaled by 1/rms (silu) and without (the other activations); one piece of K and several."""
    x, w = operands(M, 2 * I, H)
    v = w.reshape(I // 128, 2, 128, H)
    g, u = (x.double() @ v[:, i].reshape(I, H).double().t() for i in (0, 1))
    out = torch.full((M, I), float("nan"), dtype=torch.bfloat16, device=DEV)
    if act == "silu":
        ssq = torch.rand(M, 5, device=DEV) * H
        K.tc_mid_fused(x, w, out, K.TC_SILU_MUL, 128, row_ssq=ssq, norm_width=H, eps=1e-6)
        rs = 1.0 / torch.sqrt(ssq.double().sum(1, keepdim=True) / H + 1e-6)
        ref = P.silu(g * rs) * (u * rs)
    elif act == "gelu":
        K.tc_mid(x, w, out, K.TC_SILU_MUL, 128, act=K.ACT_GELU, mult=0.5)
        ref = torch.nn.functional.gelu(g, approximate="tanh") * u * 0.5
    else:
        K.tc_mid(x, w, out, K.TC_SILU_MUL, 128, act=K.ACT_CLAMPED, limit=2.0, slope=1.702)
        gc, uc = g.clamp(max=2.0), u.clamp(-2.0, 2.0)
        ref = gc * torch.sigmoid(1.702 * gc) * (uc + 1.0)
    # bfloat16 rounds by 2^-9; the float32 sums of H terms and the activation are far below that
    assert float((out.double() - ref).abs().max()) <= 2.0 ** -8 * float(ref.abs().max())
    assert float((out.double() - ref).norm() / ref.norm()) <= 2.0 ** -8


@pytest.mark.parametrize("M,N,Kd", [(17, 520, 264), (100, 2048, 8192), (301, 2048, 2048), (1000, 256, 2048)])
def test_accumulate_prepares_the_next_norm(K, M, N, Kd):
    a, w = operands(M, N, Kd)
    c0 = torch.randn(M, N, device=DEV)
    next_w = (1 + 0.2 * torch.randn(N, device=DEV)).bfloat16()
    c = c0.clone()
    xw = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=DEV)
    ssq = torch.full((M, K.tc_stream_n_tiles(N)), float("nan"), device=DEV)
    K.tc_mid_fused(a, w, c, K.TC_ACCUMULATE, xw=xw, next_w=next_w, ssq_out=ssq)
    within(c, a, w, extra=c0)
    assert torch.equal(xw, (c * next_w.float()).bfloat16())             # of the very sums it stored
    want = (c.double() ** 2).sum(1)
    assert float(((ssq.double().sum(1) - want) / want).abs().max()) <= 128 * 2.0 ** -24


@pytest.mark.parametrize("hd,nh,nkv", [(64, 6, 2), (64, 5, 1), (64, 32, 8), (128, 4, 2), (128, 3, 1)])
@pytest.mark.parametrize("new_counts,before", [([9, 7, 1], [0, 100, 61]), ([130, 7, 70], [0, 100, 61]), ([400, 1, 330], [0, 64, 5])])
def test_qkv_rotates_and_writes_the_cache(K, hd, nh, nkv, new_counts, before):
    torch.manual_seed(hd + nh)
    H, T, N = 1032, sum(new_counts), (nh + 2 * nkv) * hd
    meta = KH.paged_meta(new_counts, before, DEV, seed=hd)
    x, w = operands(T, N, H)
    ssq = torch.rand(T, 3, device=DEV) * H
    inv_freq = P.rope_inv_freq(10000.0, hd).to(DEV)
    cs, tok_page = torch.empty(T, hd // 2, 2, device=DEV), torch.empty(T, dtype=torch.int32, device=DEV)
    K.rope_table(meta, inv_freq, hd // 2, cs, tok_page)
    pools = [torch.full((meta.n_pages, nkv, 64, hd), 7.0, dtype=torch.bfloat16, device=DEV) for _ in range(2)]
    q = torch.full((T, nh * hd), float("nan"), dtype=torch.bfloat16, device=DEV)
    K.tc_mid_fused(x, w, None, K.TC_QKV_ROPE, row_ssq=ssq, norm_width=H, eps=1e-5,
                   rope=dict(cs=cs, tok_page=tok_page, positions=meta.positions, q_out=q, k_pool=pools[0], v_pool=pools[1],
                             nh=nh, nkv=nkv, hd=hd, page_size=64))
    rows = (x.double() @ w.double().t()) / torch.sqrt(ssq.double().sum(1, keepdim=True) / H + 1e-5)
    rows = rows.reshape(T, nh + 2 * nkv, hd)
    c, s = cs[..., 0].double()[:, None], cs[..., 1].double()[:, None]
    lo, hi = rows[..., :hd // 2], rows[..., hd // 2:]
    turned = torch.cat([lo * c - hi * s, hi * c + lo * s], dim=-1)
    want = [turned[:, :nh], turned[:, nh:nh + nkv], rows[:, nh + nkv:]]
    page, at = tok_page.long(), meta.positions.long() % 64
    for got, ref in zip([q.view(T, nh, hd)] + [p[page, :, at] for p in pools], want):
        assert float((got.double() - ref).abs().max()) <= 2.0 ** -8 * float(ref.abs().max())
    for p in pools:                                                     # nothing else was written
        p[page, :, at] = 7.0
        assert bool((p == 7.0).all())


@pytest.mark.parametrize("counts", [[0, 1, 128, 129, 256, 257, 513, 600], [0, 0, 0, 1500, 0, 0, 0, 0], [96] * 8])
@pytest.mark.parametrize("unit", ["clamped", "silu", "relu2"])
def test_runs_of_an_expert_of_any_length(K, counts, unit):
    """Grouped products: runs that end at, before and behind the 128 rows of the table and the 256 tokens of a tile."""
    E, W, F, top = 8, 256, 384, 1
    T = sum(counts)
    torch.manual_seed(T)
    ids = torch.cat([torch.full((n,), e, dtype=torch.int32) for e, n in enumerate(counts)])[torch.randperm(T)].to(DEV).view(T, top)
    x = torch.randn(T, W, device=DEV).bfloat16()
    up = (torch.randn(E, F, W, device=DEV) * 0.1).bfloat16()
    gate = (torch.randn(E, F, W, device=DEV) * 0.1).bfloat16()
    down = (torch.randn(E, W, F, device=DEV) * 0.1).bfloat16()
    weights = torch.rand(T, top, device=DEV)
    y = torch.randn(T, W, device=DEV)
    before = y.clone()
    both = torch.stack([gate.view(E, F // 128, 128, W), up.view(E, F // 128, 128, W)], dim=2).reshape(E, 2 * F, W).contiguous()
    if unit == "relu2":
        K.moe_experts(x, ids, weights, up, down, y, top, 0.0, 0.0, 0, act=K.ACT_RELU2)
    else:
        K.moe_experts(x, ids, weights, both, down, y, top, 7.0 if unit == "clamped" else 0.0, 1.702 if unit == "clamped" else 0.0, 128)
    ref = before.double()
    for e in range(E):
        at = (ids.view(-1) == e).nonzero().view(-1)
        u, g = x[at].double() @ up[e].double().t(), x[at].double() @ gate[e].double().t()
        if unit == "relu2":
            h = u.clamp(min=0.0) ** 2
        elif unit == "silu":
            h = P.silu(g) * u
        else:
            g, u = g.clamp(max=7.0), u.clamp(-7.0, 7.0)
            h = g * torch.sigmoid(1.702 * g) * (u + 1.0)
        ref[at] += weights[at].double() * (h @ down[e].double().t())
    # the hidden rows are rounded to bfloat16 (2^-9 each, independent), everything else is float32
    assert float((y.double() - ref).abs().max()) <= 2.0 ** -8 * float((ref - before.double()).abs().max()) + 2.0 ** -20 * float(ref.abs().max())
    rows = (y.double() - before.double()) - (ref - before.double())
    assert float(rows.norm() / (ref - before.double()).norm()) <= 2.0 ** -8


@pytest.mark.parametrize("act", ["silu", "gelu", "clamped"])
def test_gated_rows_keep_the_bits_of_32_bit_arithmetic(K, act):
    """Gates that are one bfloat16 each, exactly: of ordinary size, tiny, beyond the exponential's range, infinite and NaN. A
    float32 result is as near to 64 bits as float32 arithmetic is, and a bfloat16 one is that result rounded."""
    M, I, H = 1000, 128, 64
    g = torch.Generator().manual_seed(1)
    x = (torch.randn(M, H, generator=g) * torch.logspace(-6, 1.7, H)).bfloat16()
    x[5, :10] = torch.tensor([-87.0, -87.5, -88.0, -88.5, -90.0, 90.0, 3e38, -100.0, 1e-38, -1e-38]).bfloat16()
    x[6, 0], x[7, 1], x[8, 2] = float("inf"), float("-inf"), float("nan")
    x[:, H - 1] = 1.0
    w = torch.zeros(2, 128, H)
    w[0, torch.arange(128), torch.arange(128) % (H - 1)] = 1.0          # a gate row is one column of x
    w[1, :, H - 1] = 1.0
    w = w.reshape(256, H).bfloat16()
    keep = torch.isfinite(x).all(1)                                     # (0 times an infinity is NaN in the other columns)
    kw = dict(silu={}, gelu=dict(act=K.ACT_GELU), clamped=dict(act=K.ACT_CLAMPED, limit=7.0, slope=1.702))[act]
    assert K.tc_mid_plan(K.TC_SILU_MUL, M, 2 * I, H)[2] == 1
    full, short = (torch.full((M, I), 7.0, dtype=dt, device=DEV) for dt in (torch.float32, torch.bfloat16))
    for out in (full, short):
        K.tc_mid(x.to(DEV), w.to(DEV), out, K.TC_SILU_MUL, 128, **kw)
    assert torch.equal(full.bfloat16().view(torch.int16)[keep.to(DEV)], short.view(torch.int16)[keep.to(DEV)])
    assert torch.equal(torch.isnan(full), torch.isnan(short)) and bool(torch.isnan(full[~keep.to(DEV)]).any())
    gate = x[keep][:, torch.arange(128) % (H - 1)].double()
    if act == "clamped":
        gate = gate.clamp(max=7.0)
        ref = gate * torch.sigmoid(1.702 * gate) * 2.0
    else:
        ref = torch.nn.functional.gelu(gate, approximate="tanh") if act == "gelu" else P.silu(gate)
    got = full[keep.to(DEV)].double().cpu()
    # the exponential is off by one unit (2^-23), the sum and the quotient by half of one each, the slope's product turns into
    # |slope · gate| halves; from where the exponential overflows (88) the quotient is 0, and below 2^-126 units are absolute
    bound = (4.0 + (1.702 * gate.abs().clamp(max=90.0) if act == "clamped" else 0.0)) * 2.0 ** -23 * ref.abs() + 2.0 ** -118
    if act != "gelu":
        assert bool(((got - ref).abs() <= bound).all())


@pytest.mark.parametrize("counts", [[0, 1, 128, 129, 256, 257, 513, 600], [0, 3000, 0, 5], [16, 17, 15], [9, 0, 0, 0, 31], [5] + 11998 * [0] + [7],
                                    [3] + 11999 * [0] + [200]])
def test_parts_of_an_experts_rows(K, counts):
    """The table that the grouped products read: an expert's rows in equal parts of a multiple of 16, at most 256 each, and
    nothing that a product has to look for among its neighbours."""
    import ctypes as C
    E, W, T = len(counts), 64, sum(counts)
    g = torch.Generator().manual_seed(T)
    ids = torch.cat([torch.full((n,), e, dtype=torch.int32) for e, n in enumerate(counts)])[torch.randperm(T, generator=g)].to(DEV)
    if E == 5:
        ids = torch.cat([ids[:1], ids])[1:]                             # not on a 16-byte boundary
    x = torch.randn(T, W, device=DEV).bfloat16()
    most = -(-T // 128) + E
    ints = lambda n: torch.full((n,), -7, dtype=torch.int32, device=DEV)       # noqa: E731
    per, order, pos, tiles, up, down = ints(E), ints(most * 128), ints(T), ints(most * 3), ints(most), ints(most)
    xs = torch.empty(most * 128, W, dtype=torch.bfloat16, device=DEV)
    run = int(K.load("tc_mid").sp_tc_mid_run())
    ptr = lambda t: C.c_void_p(t.data_ptr())                            # noqa: E731
    assert K.load("hybrid").sp_moe_plan_tiles(ptr(x), ptr(ids), T, 1, W, E, 3, 5, ptr(per), ptr(order), ptr(pos), ptr(tiles), ptr(up),
                                              ptr(down), most, run, ptr(xs), C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    want, first = [], 0
    for e, n in enumerate(counts):
        cut = -(-n // run)
        part = -(-(-(-n // cut)) // 16) * 16 if n else 1
        entries = [(e, first + i, min(part, n - i)) for i in range(0, n, part)]
        assert len(entries) <= -(-n // 128) and all(0 < c <= run for _, _, c in entries)
        want += entries
        first += -(-n // 128) * 128
    got = tiles.view(-1, 3).tolist()
    assert [tuple(t) for t in got if t[0] >= 0] == want and len(got) == most
    for e, at, c in want:
        assert torch.equal(ids[order[at:at + c].long()], torch.full((c,), e, dtype=torch.int32, device=DEV))
        assert torch.equal(xs[at:at + c], x[order[at:at + c].long()]) and bool((order[at:at + c].diff() > 0).all())
    assert per.tolist() == counts


def test_more_experts_than_a_block_counts(K):
    E, W, F, T, top = 12001, 16, 8, 5, 2
    g = torch.Generator().manual_seed(1)
    x, up, down = (torch.randn(*s, generator=g) for s in ((T, W), (E, F, W), (E, W, F)))
    ids = torch.tensor([[0, 12000], [12000, 7], [11999, 3], [7, 0], [5000, 12000]], dtype=torch.int32)
    weights = torch.rand(T, top, generator=g)
    y = torch.zeros(T, W, device=DEV)
    K.moe_experts(x.to(DEV), ids.to(DEV), weights.to(DEV), up.to(DEV), down.to(DEV), y, top, 0.0, 0.0, act=K.ACT_RELU2)
    h = torch.relu(torch.einsum("tkfw,tw->tkf", up[ids.long()].double(), x.double())) ** 2
    ref = torch.einsum("tk,tkwf,tkf->tw", weights.double(), down[ids.long()].double(), h)
    # sums of 16 and 8 terms, a square: some twenty roundings of 2^-24 on sums of absolute values a few times the result
    assert float((y.double().cpu() - ref).abs().max()) <= 1e-5 * float(ref.abs().max())


def test_experts_of_many_tokens_take_the_tiles_of_128(K, monkeypatch):
    E, W, F, T = 2, 128, 256, 700
    torch.manual_seed(5)
    ids = (torch.rand(T, 1, device=DEV) < 0.9).int()
    x, y = torch.randn(T, W, device=DEV).bfloat16(), torch.zeros(T, W, device=DEV)
    both, down = (torch.randn(E, 2 * F, W, device=DEV) * 0.1).bfloat16(), (torch.randn(E, W, F, device=DEV) * 0.1).bfloat16()
    weights = torch.rand(T, 1, device=DEV)
    rows = []
    for most in (K.MID_EXPERT_TOKENS, 1):
        monkeypatch.setattr(K, "MID_EXPERT_TOKENS", most)
        y.zero_()
        K.moe_experts(x, ids, weights, both, down, y, 1, 7.0, 1.702, 128)
        rows.append(y.clone())
    # the hidden rows are bfloat16 of the same 32-bit sums in another order
    assert float((rows[0] - rows[1]).norm() / rows[0].norm()) <= 2.0 ** -8
    with pytest.raises(K.KernelError):
        K._check("hybrid", K.load("hybrid").sp_moe_plan_tiles(None, None, 8, 1, 64, 1, 1, 1, None, None, None, None, None, None, 4, 100, None, None))


@pytest.mark.parametrize("act", ["ACT_SILU", "ACT_GELU", "ACT_CLAMPED"])
@pytest.mark.parametrize("M", [129, 255, 256, 257, 400, 513, 1025, 1152, 1300])
def test_gated_products_by_pairs_of_ctas(K, M, act):
    """The tiles of 256 rows that gated products take from 129 tokens on: rows behind the last token, gates of all sizes."""
    act = getattr(K, act)
    limit, slope = (7.0, 1.7) if act == K.ACT_CLAMPED else (0.0, 0.0)
    a, w = operands(M, 768, 200)
    a[0], a[M - 1] = 0.0, a[M - 1] * 60.0                               # gates of zero, and some beyond the branch-free range
    out = torch.full((M + 3, 384), 9.0, device=DEV)
    K.tc_gemm(a, w, out[:M], K.TC_SILU_MUL, 256, act=act, limit=limit, slope=slope)
    y = (a.double() @ w.double().t()).view(M, 3, 2, 128)
    g, u = y[:, :, 0].reshape(M, 384), y[:, :, 1].reshape(M, 384)
    if act == K.ACT_CLAMPED:
        g, u = g.clamp(max=limit), u.clamp(-limit, limit) + 1.0
    ref = torch.nn.functional.gelu(g, approximate="tanh") * u if act == K.ACT_GELU else g * torch.sigmoid((slope or 1.0) * g) * u
    # the sums' error (200 terms of at most 0.1 · 60 · 4 in 2^-23 each) through an activation of slope 1.1 and the other factor
    bound = 1.2 * 200 * 2.0 ** -23 * (a.double().abs() @ w.double().abs().t()).amax(1, keepdim=True) * (1.0 + g.abs() + u.abs())
    assert bool(((out[:M].double() - ref).abs() <= bound).all())
    assert bool((out[M:] == 9.0).all())


def test_the_choice_between_the_two_kernels(K):
    for N, Kd in ((3072, 2048), (16384, 2048), (28672, 4096), (4096, 14336), (40, 64)):
        for M in (1, 128, 129, 300, 1023, 1024, 1500, 2048, 2049, 6000):
            for mode in (K.TC_STORE, K.TC_SILU_MUL):
                width = K.tc_mid_or_pairs(mode, M, N, Kd, 128)
                assert width in (0, 128, 256) and not (width and M <= 128) and (width or M <= 2048)
                assert mode == K.TC_SILU_MUL or not width or M >= 1024
                assert mode != K.TC_SILU_MUL or width in (0, 256)
    if torch.cuda.get_device_properties(DEV).multi_processor_count != 148:
        return                                                          # what follows was measured on 148
    assert K.tc_mid_or_pairs(K.TC_ACCUMULATE, 1280, 2048, 8192) == 0 and K.tc_mid_or_pairs(K.TC_ACCUMULATE, 2048, 2048, 8192) == 256
    assert K.tc_mid_or_pairs(K.TC_SILU_MUL, 301, 16384, 2048) == 0 and K.tc_mid_or_pairs(K.TC_SILU_MUL, 512, 16384, 2048) == 256
    assert [K.tc_mid_or_pairs(K.TC_STORE, M, 512, 512) for M in (1024, 1280, 1800, 2048)] == [0, 0, 128, 128]
    # gated rows of the 3B and 8B layers: the kernel that the figures beside the rule show as the faster one
    assert [K.tc_mid_or_pairs(K.TC_SILU_MUL, M, 16384, 3072) for M in (200, 256, 257, 800)] == [256, 256, 0, 256]
    assert [K.tc_mid_or_pairs(K.TC_SILU_MUL, M, 28672, 4096) for M in (200, 257, 512, 768, 880, 1100, 1281)] == [0, 0] + 5 * [256]


@pytest.mark.parametrize("M", [1024, 1279, 1537, 2048])
@pytest.mark.parametrize("N,Kd", [(2048, 512), (520, 1096)])
def test_linear_of_more_tokens(K, M, N, Kd):
    from spissa_b200.parts.linear import Linear
    a, w = operands(M, N, Kd)
    c0 = torch.randn(M, N, device=DEV)
    acc = c0.clone()
    Linear(w)(a, out=acc, accumulate=True)
    within(acc, a, w, extra=c0)


@pytest.mark.parametrize("act", ["ACT_SILU", "ACT_GELU", "ACT_CLAMPED"])
@pytest.mark.parametrize("kernel,width", [("tc_mid", 128), ("tc_gemm", 256), ("tc_gemm", 128)])
def test_a_tokens_gated_values_do_not_depend_on_its_neighbours(K, act, kernel, width):
    """Gates beyond the branch-free range in every sixteenth token leave the others' bits as they are."""
    kw = dict(act=getattr(K, act))
    if act == "ACT_CLAMPED":
        kw.update(limit=100.0, slope=1.702)
    a, w = operands(2048, 16384, 64)
    b = a.clone()
    b[::16] *= 1000.0
    plain, beside = torch.empty(2048, 8192, device=DEV), torch.empty(2048, 8192, device=DEV)
    getattr(K, kernel)(a, w, plain, K.TC_SILU_MUL, width, **kw)
    getattr(K, kernel)(b, w, beside, K.TC_SILU_MUL, width, **kw)
    rest = torch.arange(2048, device=DEV) % 16 != 0
    assert torch.equal(plain[rest], beside[rest])


@pytest.mark.parametrize("kernel,width", [("tc_mid", 128), ("tc_gemm", 256), ("tc_gemm", 128)])
@pytest.mark.parametrize("slope,gate", [(0.2526956572140501, 0.020345522090792656), (0.5680828327219911, 0.007325529120862484),
                                        (0.7441885108658084, 0.0013069163542240858), (0.7441885108658084, 0.10660775750875473),
                                        (0.974886949234209, 0.012287044897675514), (2.8710412953340563, 0.0016809902153909206),
                                        (4.926993966922774, 0.005847701337188482), (None, 0.050509825348854065)])
def test_units_whose_quotient_lies_near_the_middle_of_two_floats(K, kernel, width, slope, gate):
    """Gates whose quotient by an unrefined reciprocal is a last bit off (a clamped unit's slope, or gelu): the same value alone and
    beside a large gate."""
    parts, left = [], torch.tensor(gate)
    for _ in range(3):                                                  # the gate as an exact sum of three bfloat16 numbers
        parts.append(left.bfloat16())
        left = left - parts[-1].float()
    assert float(left) == 0.0
    half = width if kernel == "tc_mid" else width // 2
    w = torch.zeros(512, 64, dtype=torch.bfloat16, device=DEV)
    w.view(-1, 2, half, 64)[:, 0, :, :3] = 1.0                          # gate rows
    if slope is None:
        w.view(-1, 2, half, 64)[:, 1, :, 3] = 1.0                       # up is 1; the clamped unit adds one to zero
    a = torch.zeros(130, 64, dtype=torch.bfloat16, device=DEV)
    a[:, :3] = torch.stack(parts).to(DEV)
    a[:, 3] = 1.0
    b = a.clone()
    b[1::2, 0] = 512.0
    outs = [torch.empty(130, 256, device=DEV) for _ in range(2)]
    for x, out in zip((a, b), outs):
        kw = dict(act=K.ACT_GELU) if slope is None else dict(act=K.ACT_CLAMPED, limit=1000.0, slope=slope)
        getattr(K, kernel)(x, w, out, K.TC_SILU_MUL, width, **kw)
    assert torch.equal(outs[0][::2], outs[1][::2])
    exponent = -slope * gate if slope is not None else -1.5957691216057308 * (gate + 0.044715 * gate ** 3)
    want = gate / (1.0 + float(torch.exp(torch.tensor(exponent, dtype=torch.float64))))
    # half a unit, and an expf that is two units of 2^-24 off below 1
    assert float((outs[0][::2].double() - want).abs().max()) <= 4 * 2.0 ** -24 * want


@pytest.mark.parametrize("M", [129, 200, 256, 257, 449, 512, 800, 1023])
def test_gated_products_by_pairs_with_row_statistics(K, M):
    """What a prompt's step asks of the pairs' tiles: the normed residual's 1/rms folded into the epilogue."""
    H, N = 264, 768
    torch.manual_seed(M)
    x, weight = torch.randn(M, H, device=DEV) * 2.0, (1.0 + 0.1 * torch.randn(H, device=DEV)).bfloat16()
    x[M // 2] *= 1e-3                                                   # a small row: its 1/rms is large
    w = (torch.randn(N, H, device=DEV) * 0.1).bfloat16()
    xw, ssq = torch.empty(M, H, dtype=torch.bfloat16, device=DEV), torch.empty(M, 1, device=DEV)
    K.norm_prepare(x, weight, xw, ssq)
    out = torch.full((M + 2, N // 2), 9.0, device=DEV)
    K.tc_gemm_fused(xw, w, out[:M], K.TC_SILU_MUL, 256, row_ssq=ssq, norm_width=H, eps=1e-5)
    rstd = 1.0 / torch.sqrt((x.double() ** 2).sum(1, keepdim=True) / H + 1e-5)
    y = (xw.double() @ w.double().t() * rstd).view(M, 3, 2, 128)
    g, u = y[:, :, 0].reshape(M, 384), y[:, :, 1].reshape(M, 384)
    size = (xw.double().abs() @ w.double().abs().t() * rstd).amax(1, keepdim=True)
    # the sums' error (H terms of 2^-23 each) and 1/rms's (H / 32 + 8 roundings of 2^-24) through an activation of slope 1.1
    bound = 1.2 * (H + 16) * 2.0 ** -23 * size * (1.0 + g.abs() + u.abs())
    assert bool(((out[:M].double() - g * torch.sigmoid(g) * u).abs() <= bound).all())
    assert bool((out[M:] == 9.0).all())


@pytest.mark.parametrize("M", [17, 64, 200, 301])
@pytest.mark.parametrize("Kd", [8, 64, 136, 512, 1096, 4096])
def test_weights_asked_for_ahead(K, M, Kd):
    """The ring's first tiles of W fetched before the predecessor has ended, for fewer, as many and more blocks of K than the ring
    holds: the same bits, behind a kernel that writes the other operand."""
    H = Kd
    torch.manual_seed(Kd + M)
    x, weight = torch.randn(M, H, device=DEV), (1.0 + 0.1 * torch.randn(H, device=DEV)).bfloat16()
    w_store, w_gate = ((torch.randn(n, H, device=DEV) * 0.1).bfloat16() for n in (2056, 1024))
    stages = {K.tc_mid_plan(mode, M, w.shape[0], Kd)[2:] for mode, w in ((K.TC_STORE, w_store), (K.TC_SILU_MUL, w_gate))}
    assert all(pieces >= 1 and n >= 1 for pieces, n in stages)
    got = {}
    for settled in (False, True):
        rows = []
        for _ in range(4):
            xw, ssq = torch.zeros(M, H, dtype=torch.bfloat16, device=DEV), torch.empty(M, 1, device=DEV)
            store = torch.full((M, 2056), float("nan"), dtype=torch.bfloat16, device=DEV)
            acc, act = torch.zeros(M, 2056, device=DEV), torch.full((M, 512), float("nan"), dtype=torch.bfloat16, device=DEV)
            K.norm_prepare(x, weight, xw, ssq)
            kw = dict(row_ssq=ssq, norm_width=H, eps=1e-5, w_settled=settled)
            K.tc_mid_fused(xw, w_gate, act, K.TC_SILU_MUL, 128, **kw)
            K.tc_mid_fused(xw, w_store, store, K.TC_STORE, **kw)
            K.tc_mid_fused(xw, w_store, acc, K.TC_ACCUMULATE, w_settled=settled)
            rows.append((act, store, acc))
        got[settled] = rows
    for again in got[False][1:] + got[True]:
        assert all(torch.equal(a, b) for a, b in zip(got[False][0], again))
    within(got[True][0][2], xw, w_store)


@pytest.mark.parametrize("block", [64, 128])
@pytest.mark.parametrize("poison", [float("nan"), 3e4])
def test_experts_do_not_read_what_the_memory_held(K, block, poison):
    """The rows of holes among the gathered ones are not written: whatever stands there, the tokens' results have the same bits."""
    E, W, F, top, T = 8, 256, 384, 2, 700
    torch.manual_seed(block)
    x = torch.randn(T, W, device=DEV).bfloat16()
    gate, up = ((torch.randn(E, F // block, block, W, device=DEV) * 0.1).bfloat16() for _ in range(2))
    both = torch.stack([gate, up], dim=2).reshape(E, 2 * F, W).contiguous()
    down = (torch.randn(E, W, F, device=DEV) * 0.1).bfloat16()
    ids, weights = torch.randint(0, E, (T, top), dtype=torch.int32, device=DEV), torch.rand(T, top, device=DEV)
    ys = []
    for fill in (0.0, poison):
        torch.cuda.empty_cache()
        held = [torch.full((n, W), fill, dtype=dt, device=DEV) for n in (1500, 2500, 4000) for dt in (torch.bfloat16, torch.float32)]
        torch.cuda.synchronize()
        del held
        y = torch.zeros(T, W, device=DEV)
        K.moe_experts(x, ids, weights, both, down, y, top, 7.0, 1.702, block)
        ys.append(y)
    assert bool(ys[0].isfinite().all()) and torch.equal(*ys)
