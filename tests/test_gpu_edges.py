"""Edges of the kernels' tiles and of the rules that choose between kernels, against plain 64-bit references."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def K():
    from dllama_b200.ops import kernels
    return kernels


def L():
    from dllama_b200.ops import layers
    return layers


def lib():
    from dllama_b200.ops import lib
    return lib


@pytest.mark.parametrize("heads,kv,hs,n_splits", [(4, 1, 128, 1), (3, 1, 128, 4), (4, 2, 64, 1), (8, 2, 64, 3), (2, 2, 128, 2)])
def test_decode_attention_half_pages(heads, kv, hs, n_splits):
    """Contexts around the borders of half pages, of the warps' turns and of the split rule (24 pages); an infinite key that a head's
    score sends to -inf takes no weight and leaves the rest finite, as in f32.  Bound: f32 sums of some hundred terms and an
    exponential of relative error 2^-22 on scores below 8 in units of log2: 2e-6 of the largest value is several times that."""
    positions = [0, 14, 15, 16, 31, 32, 63, 64, 127, 767, 768, 901]
    M, pages = len(positions), 30
    g = torch.Generator().manual_seed(heads * 1000 + hs)
    q = torch.randn(M, heads * hs, generator=g)
    kc, vc = (torch.randn(M * pages, kv, 32, hs, generator=g).half() for _ in range(2))
    bt = torch.randperm(M * pages, generator=g).int().view(M, pages)
    kc[bt[11, 3], :, 5] = 0                        # one key of the last row: -inf along its first dimension
    kc[bt[11, 3], :, 5, 0] = -float("inf")
    q[11].view(heads, hs)[:, 0] = 1.5
    y = torch.zeros(M, heads * hs, device="cuda")
    scratch = torch.zeros(K().attention_scratch_bytes(M, heads, hs, n_splits), dtype=torch.uint8, device="cuda")
    for _ in range(2):                              # twice: the split counters reset themselves
        K().attention(q.cuda(), M, heads, kv, hs, kc.cuda(), vc.cuda(), torch.tensor(positions, dtype=torch.int32, device="cuda"),
                      torch.arange(M, dtype=torch.int32, device="cuda"), bt.cuda(), pages, n_splits, scratch, None, None, M, y)
    want = torch.empty(M, heads, hs, dtype=torch.float64)
    for m, p in enumerate(positions):
        k, v = (c[bt[m].long()].transpose(1, 2).reshape(-1, kv, hs)[:p + 1].double().repeat_interleave(heads // kv, dim=1) for c in (kc, vc))
        s = torch.einsum("hd,thd->ht", q[m].double().view(heads, hs), k) * hs ** -0.5
        want[m] = torch.einsum("ht,thd->hd", s.softmax(dim=1), v)
    got = y.cpu().double().view(M, heads, hs)
    assert torch.isfinite(got).all()
    assert (got - want).abs().max() <= 2e-6 * want.abs().max()


@pytest.mark.parametrize("M,N,K_", [(1, 8, 128), (7, 200, 128), (32, 1000, 384), (33, 6000, 256), (64, 40, 1024), (100, 2056, 512), (127, 7000, 128),
                                    (128, 40008, 128), (128, 5888, 640)])
def test_dense_rows_shares(M, N, K_):
    """Few-row products: shares that end inside a 128-column tile, one and two accumulators, odd and even ring depths, one k tile, more
    columns than one wave of CTAs holds, clusters that split K.  bf16 products are exact in f32; a tensor-core chain of K / 16 steps
    truncates, each step by at most 2^-22 of the largest partial sum: 1e-5 relative covers K = 1024 several times over."""
    g = torch.Generator(device="cuda").manual_seed(N + M)
    w = (torch.randn(N, K_, generator=g, device="cuda") * K_ ** -0.5).bfloat16()
    x, ncap = torch.randn(M, K_, generator=g, device="cuda"), (M + 7) // 8 * 8
    bias, aux = torch.randn(N, generator=g, device="cuda"), torch.randn(M, N, generator=g, device="cuda")
    xh = torch.zeros(L().xh_bytes(K_, ncap), dtype=torch.uint8, device="cuda")
    L().xh_from_rows(x, M, K_, ncap, xh)
    wh, z = L().make_wh(w), x.bfloat16().double() @ w.double().t()

    def close(y, want):
        assert (y.double() - want).norm() <= 1e-5 * want.norm() + 1e-12

    y = torch.full((M + 2, N + 3), 7.0, device="cuda")
    L().dense_tc(wh, N, K_, xh, ncap, y, M, bias=bias)
    close(y[:M, :N], z + bias.double())
    assert (y[M:] == 7).all() and (y[:, N:] == 7).all()          # nothing past the rows and columns asked for
    L().dense_tc(wh, N, K_, xh, ncap, y, M, epi=L().DENSE_SIGMOID_MUL, aux=aux)
    close(y[:M, :N], aux.double() * z.sigmoid())
    half = torch.zeros(M, N // 2, device="cuda")
    L().dense_tc(wh, N, K_, xh, ncap, half, M, epi=L().DENSE_GLU_GELU)
    close(half, torch.nn.functional.gelu(z[:, 0::2], approximate="tanh") * z[:, 1::2])
    if N % 256 == 0:
        img, direct = (torch.zeros(L().xh_bytes(N // 2, ncap), dtype=torch.uint8, device="cuda") for _ in range(2))
        L().dense_tc(wh, N, K_, xh, ncap, half, M, epi=L().DENSE_GLU_GELU, image=(img, ncap))
        L().xh_from_rows(half, M, N // 2, ncap, direct)
        live = lambda t: t.view(-1, ncap // 8, 16, 8, 16).permute(1, 3, 0, 2, 4).reshape(ncap, -1)[:M]
        assert torch.equal(live(img), live(direct))


@pytest.mark.parametrize("M", [1, 2, 3, 8])
def test_gemv_extreme_nibbles(M):
    """The largest products of a block (nibbles 0 and 15, activations of +-127) through the integer-to-float step, and every sign mixed:
    integers below 2^20 times one scale are exact in f32, a row of 4 such blocks to its last additions (4 * 2^-24)."""
    d, n = 256, 512
    g = torch.Generator().manual_seed(M)
    nib = torch.randint(0, 16, (d, n // 32, 32), generator=g, dtype=torch.uint8)
    nib[0::4], nib[1::4] = 15, 0
    nib[2::4, :, ::2], nib[2::4, :, 1::2] = 15, 0
    scale = torch.full((d, n // 32, 1), 0.5).half()
    raw = torch.cat([scale.view(torch.uint8), nib[:, :, :16] | (nib[:, :, 16:] << 4)], dim=2)
    x = torch.where(torch.rand(M, n, generator=g) < 0.5, -1.0, 1.0)
    x[0], x[M - 1, ::2] = 1.0, -1.0
    k = K()
    xq = k.alloc_xq(n, M, "cuda")
    k.quant_q80(x.cuda(), M, n, M, xq_out=xq)
    y = torch.zeros(M, d, device="cuda")
    k.gemv_q40(k.make_q40t(raw.reshape(-1).cuda(), d, n), d, n, xq, M, k.epi_store([y.data_ptr()], d))
    w = (nib.double() - 8).reshape(d, n) * 0.5
    xd = x.double().sign() * 127 * float(torch.tensor(1 / 127).half())
    want = xd @ w.t()
    assert (y.cpu().double() - want).abs().max() <= 2.0 ** -21 * want.abs().max()


@pytest.mark.parametrize("d,n,k_split,rows", [(19200, 256, 1, [4, 17, 33, 100, 128]), (19072, 384, 1, [5, 64]), (384, 1024, 2, [4, 33, 128]), (256, 1024, 4, [6, 100]),
                                              (256, 1152, 8, [5, 16, 65])])
def test_q40_tc_pairs_and_shares(d, n, k_split, rows):
    """Row tiles side by side (more even row tiles than SMs; an odd number stays alone) and K shares whose ranks finish part of the rows
    each (also ranks left without a row).  Bound: the operands are taken as the kernel rounds them, f32 accumulation of n <= 1152 terms: 1e-5."""
    k = K()
    g = torch.Generator(device="cuda").manual_seed(d + n)
    nib = torch.randint(0, 16, (d, n // 32, 32), generator=g, device="cuda", dtype=torch.uint8)
    scale = (0.01 + 0.01 * torch.rand(d, n // 32, 1, generator=g, device="cuda")).half()
    raw = torch.cat([scale.view(torch.uint8), nib[:, :, :16] | (nib[:, :, 16:] << 4)], dim=2)
    w = ((nib.half() - 8) * scale).double().reshape(d, n)
    q40t = k.make_q40t(raw.reshape(-1), d, n)
    for M in rows:
        x = torch.randn(M, n, generator=g, device="cuda")
        ncap = 16 if M <= 16 else 32 if M <= 32 else 64 if M <= 64 else 128
        xh = k.alloc_xh(n, ncap, "cuda")
        k.quant_q80(x, M, n, ncap, xh_out=xh)
        blocks = x.view(M, n // 32, 32)
        s = blocks.abs().amax(dim=2, keepdim=True) / 127
        xq = ((blocks * (1 / s)).round() * s.half().float()).half().double().view(M, n)
        y = torch.full((M + 1, d), 3.0, device="cuda")
        k.gemm_q40_tc(q40t, d, n, xh, ncap, M, k.epi_store([y.data_ptr()], d), k_split)
        want = xq @ w.t()
        assert (y[:M].double() - want).norm() <= 1e-5 * want.norm()
        assert (y[M] == 3).all()


@pytest.mark.parametrize("dim,vdim,form", [(48, 66, "lower"), (128, 128, "keys"), (64, 64, "ahead"), (20, 130, "delta"), (128, 64, "delta")])
def test_gated_scan_two_columns(dim, vdim, form):
    """Token by token with two columns per thread (160 CTAs and more): widths that end inside a CTA's 64 columns, head sizes that end inside
    a group of 16 rows, several rows per sequence, fresh and continued sequences.  f32 chains of at most 128 terms: 1e-5."""
    lib, H, S, per = L(), 4, 40, 3
    g = torch.Generator(device="cuda").manual_seed(dim * 1000 + vdim)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    M = S * per
    q, v, f, fb = rnd(M, H * dim), rnd(M, H * vdim), rnd(M, H * dim), rnd(H * dim)
    key, state = rnd(M, H * dim) * dim ** -0.5, rnd(S, H, dim, vdim)
    i32 = lambda t: torch.tensor(t, dtype=torch.int32, device="cuda")
    start = [0 if s % 3 == 0 else 7 for s in range(S)]
    slots = list(range(S))[::-1]
    keep = dict(pos=i32([start[m // per] + m % per for m in range(M)]), row_seq=i32([m // per for m in range(M)]), seq_start=i32([s * per for s in range(S + 1)]),
                seq_rows=i32(list(range(M))), seq_slot=i32(slots), seq_pos0=i32(start))
    lower, beta, bonus = torch.rand(H * dim, generator=g, device="cuda"), rnd(M, H), rnd(H * dim)
    kw = dict(f=f, f_bias=fb)
    if form == "lower":
        kw.update(lower=lower, gate=lib.GATE_LOWER)
    else:
        kw.update(k=key, gate=lib.GATE_ROOT_SIGMOID, tau=4.0)
        kw.update({"ahead": dict(bonus=bonus), "delta": dict(beta=beta)}.get(form, {}))
    y, st = torch.zeros(M, H * vdim, device="cuda"), state.clone()
    lib.gated_scan(lib.mamba_batch(**keep), S, q, v, y, st, H, dim, vdim, **kw)
    z = (f + fb).double().view(S, per, H, dim)
    gate = lower.double().view(H, dim) + (1 - lower.double().view(H, dim)) * z.sigmoid() if form == "lower" else z.sigmoid() ** 0.25
    kk = (1 - gate) if form == "lower" else key.double().view(S, per, H, dim)
    qq, vv = q.double().view(S, per, H, dim), v.double().view(S, per, H, vdim)
    cur = state.double()[slots] * torch.tensor([p != 0 for p in start], device="cuda").view(S, 1, 1, 1)
    for t in range(per):
        if form == "ahead":
            out = torch.einsum("shd,shdv->shv", qq[:, t], cur) + (qq[:, t] * bonus.double().view(H, dim) * kk[:, t]).sum(-1, keepdim=True) * vv[:, t]
        cur = gate[:, t, :, :, None] * cur
        u = vv[:, t]
        if form == "delta":
            u = beta.double().view(S, per, H, 1)[:, t].sigmoid() * (u - torch.einsum("shd,shdv->shv", kk[:, t], cur))
        cur = cur + kk[:, t, :, :, None] * u[:, :, None, :]
        if form != "ahead":
            out = torch.einsum("shd,shdv->shv", qq[:, t], cur)
        got = y.view(S, per, H, vdim)[:, t].double()
        assert (got - out).norm() <= 1e-5 * out.norm()
    assert (st.double()[slots] - cur).norm() <= 1e-5 * cur.norm()


@pytest.mark.parametrize("M,dim", [(1, 32), (3, 2080), (1183, 256), (1185, 4096), (1200, 4128), (1187, 96)])
def test_norm_q80_rows_per_cta(M, dim):
    """Norm and Q80 cast with a CTA per row and per 8 rows: rows and blocks that leave lanes without work, rows longer than the registers
    hold.  The cast agrees with the norm's own output to one step of the block (a sum in another order may move a value across a half)."""
    from test_gpu_kernels import _decode_xh
    k = K()
    g = torch.Generator(device="cuda").manual_seed(M + dim)
    x, part, w = (torch.randn(*s, generator=g, device="cuda") for s in ((M, dim), (M, dim), (dim,)))
    ncap, kp = (M + 7) // 8 * 8, (dim + 127) // 128 * 128
    xq, xh = k.alloc_xq(kp, ncap, "cuda"), k.alloc_xh(kp, ncap, "cuda")
    x_out, y = torch.zeros(M, dim, device="cuda"), torch.zeros(M, dim, device="cuda")
    k.reduce_norm_quant(x, x_out, part.data_ptr(), 1, M * dim, None, None, 0, 0, w, 1e-5, dim, M, ncap, xq, xh, y_out=y)
    s = x.double() + part.double()
    want = w.double() * s / (s.square().mean(dim=1, keepdim=True) + 1e-5).sqrt()
    assert (x_out.double() - s).abs().max() <= 1e-6 * s.abs().max()
    assert (y.double() - want).norm() <= 1e-6 * want.norm()
    step = want.view(M, dim // 32, 32).abs().amax(dim=2, keepdim=True) / 127
    raw = xq.view(kp // 128, ncap, 160)[:, :M]
    q = raw[:, :, :128].view(torch.int8).double().view(kp // 128, M, 4, 32)
    d = raw[:, :, 128:144].contiguous().view(torch.float32).double().view(kp // 128, M, 4, 1)
    for got in ((q * d).permute(1, 0, 2, 3).reshape(M, kp // 32, 32)[:, :dim // 32], torch.from_numpy(_decode_xh(xh, kp, ncap, M)).cuda().double().view(M, kp // 32, 32)[:, :dim // 32]):
        assert ((got - want.view(M, dim // 32, 32)).abs() <= 1.01 * step + 1e-9).all()
    sums = raw[:, :, 144:160].contiguous().view(torch.int32).view(kp // 128, M, 4)
    live = sums.permute(1, 0, 2).reshape(M, kp // 32)[:, :dim // 32]
    assert (live == 8 * q.sum(dim=3).long().permute(1, 0, 2).reshape(M, kp // 32)[:, :dim // 32]).all()


@pytest.mark.parametrize("window,chunk,softcap,extra", [(0, 0, 0.0, False), (50, 0, 0.0, True), (130, 0, 30.0, True), (0, 64, 0.0, False), (1, 0, 0.0, False)])
def test_window_prompt_tiles(window, chunk, softcap, extra):
    """Tiles of many rows (tcgen05, two neighbours on 128 lanes where the second continues the first) beside decoding tiles, in one call: pairs
    that fit and that do not, a last tile of few rows, windows that start inside a page, pages ahead of a window full of NaN and never
    touched.  Bound: queries and weights are rounded to bf16 (2^-9 each), so about 2e-3 of a row; 8e-3."""
    heads, kv, dim, pages = 8, 2, 128, 12
    g = torch.Generator().manual_seed(window + chunk)
    runs = [(100, 37), (211, 1), (0, 20), (300, 16), (64, 16), (0, 3), (31, 64)]             # (first position, rows) per sequence
    M, S = sum(n for _, n in runs), len(runs)
    cache = torch.randn(S * pages, kv, 32, 2 * dim, generator=g).bfloat16()
    bt = torch.randperm(S * pages, generator=g).int().view(S, pages)
    pos, slot, tiles = [], [], []
    for s, (p0, n) in enumerate(runs):
        rows = list(range(len(pos), len(pos) + n))
        pos += list(range(p0, p0 + n))
        slot += [s] * n
        tiles += [rows[i:i + 16] for i in range(0, n, 16)]
        lo = max(0, p0 - window + 1) if window else p0 // chunk * chunk if chunk else 0
        cache[bt[s, :lo // 32].long()] = float("nan")
        cache[bt[s, (p0 + n + 31) // 32:].long()] = float("nan")
    q, sink, slope, gate = torch.randn(M, heads * dim, generator=g), torch.randn(heads, generator=g), torch.rand(heads, generator=g) * 0.1, torch.randn(M, heads, generator=g)
    opt = dict(sink=sink.cuda(), slope=slope.cuda(), gate=gate.cuda()) if extra else {}
    out = torch.zeros(M, heads * dim, device="cuda")
    L().window_attention_tiles(q.cuda(), out, heads, kv, dim, 0, 0.2, softcap, window, torch.tensor(pos, dtype=torch.int32, device="cuda"),
                               torch.tensor(slot, dtype=torch.int32, device="cuda"), bt.cuda(), cache.cuda(), tiles, vdim=dim, chunk=chunk, **opt)
    got = out.cpu().double().view(M, heads, dim)
    for m in range(M):
        p = pos[m]
        lo = max(p - window + 1 if window else 0, p // chunk * chunk if chunk else 0, 0)
        line = cache[bt[slot[m]].long()].transpose(1, 2).reshape(-1, kv, 2 * dim)[lo:p + 1].double().repeat_interleave(heads // kv, dim=1)
        s = torch.einsum("hd,thd->ht", q[m].bfloat16().double().view(heads, dim), line[..., :dim]) * 0.2
        if softcap:
            s = softcap * (s / softcap).tanh()
        if extra:
            s = torch.cat([s - slope.double()[:, None] * (p - torch.arange(lo, p + 1))[None], sink.double()[:, None]], dim=1)
        want = torch.einsum("ht,thd->hd", s.softmax(dim=1)[:, :p + 1 - lo], line[..., dim:])
        if extra:
            want = want * gate[m].double().sigmoid()[:, None]
        assert (got[m] - want).norm() <= 8e-3 * want.norm(), (m, p)


@pytest.mark.parametrize("M,N,K_,dtype,round_x", [(1, 24, 8, "bf16", True), (2, 40, 136, "bf16", True), (8, 1000, 264, "bf16", True), (9, 5008, 128, "bf16", True),
                                                  (16, 10000, 392, "bf16", True), (17, 48, 1160, "bf16", True), (32, 2064, 256, "bf16", True), (1, 9, 8200, "f32", False),
                                                  (4, 64, 2056, "f32", False), (8, 24, 1032, "bf16", False), (31, 33, 72, "f32", False)])
def test_dense_few_rows(M, N, K_, dtype, round_x):
    """Few-row products straight from the weight rows: one row, the MMA form's row and column tiles and their remainders, K that ends inside
    a staged step and inside a batch of loads, both weight types, paired columns and an output gate.  f32 sums of K terms: 3e-6."""
    g = torch.Generator(device="cuda").manual_seed(M * 1000 + N)
    w = (torch.randn(N, K_, generator=g, device="cuda") * K_ ** -0.5).to(torch.bfloat16 if dtype == "bf16" else torch.float32)
    x, aux, bias = torch.randn(M, K_ + 4, generator=g, device="cuda")[:, :K_], torch.randn(M, N, generator=g, device="cuda"), torch.randn(N, generator=g, device="cuda")
    z = (x.bfloat16() if round_x else x).double() @ w.double().t()
    close = lambda y, want: (y.double() - want).norm() <= 3e-6 * want.norm() + 1e-12
    y = torch.full((M + 1, N + 2), 5.0, device="cuda")
    L().dense(w, x, y, M, round_x, bias=bias)
    assert close(y[:M, :N], z + bias.double()) and (y[M] == 5).all() and (y[:, N:] == 5).all()
    L().dense(w, x, y, M, round_x, epi=L().DENSE_SIGMOID_MUL, aux=aux)
    assert close(y[:M, :N], aux.double() * z.sigmoid())
    if N % 2 == 0:
        half = torch.zeros(M, N // 2, device="cuda")
        L().dense(w, x, half, M, round_x, epi=L().DENSE_GLU_GELU)
        assert close(half, torch.nn.functional.gelu(z[:, 0::2], approximate="tanh") * z[:, 1::2])


def _one_row_tiles(contexts, heads, kv, seed, extra=0):
    """Decoding rows of sequences of these lengths on 128 / 128 bf16 lines: call(out) runs the attention, n_splits == 1.  extra: rows of q behind them."""
    M, dim = len(contexts), 128
    g = torch.Generator(device="cuda").manual_seed(seed)
    need = [(t + 31) // 32 for t in contexts]
    bt = torch.zeros(M, max(need), dtype=torch.int32)
    perm = torch.randperm(sum(need), generator=torch.Generator().manual_seed(seed)).int()
    for m in range(M):
        bt[m, :need[m]] = perm[sum(need[:m]):sum(need[:m + 1])]
    cache = torch.randn(sum(need), kv, 32, 2 * dim, generator=g, device="cuda").bfloat16()
    q = torch.randn(M + extra, heads * dim, generator=g, device="cuda")
    rq = L().window_tc_rows(heads, kv)
    assert L().window_tc_route(heads, kv, dim, dim, M + extra, M, rq) == (3 if extra else 1)
    tiles = torch.full((M, rq), -1, dtype=torch.int32)
    tiles[:, 0] = torch.arange(M, dtype=torch.int32)
    pos, slot = torch.tensor([t - 1 for t in contexts], dtype=torch.int32, device="cuda"), torch.arange(M, dtype=torch.int32, device="cuda")
    bt, tiles = bt.cuda(), tiles.cuda()
    return lambda out: L().window_attention_tc(q, out, heads, kv, dim, 0, dim ** -0.5, 0.0, 0, pos, slot, bt, cache, tiles, M, rq, vdim=dim)


@pytest.mark.parametrize("M,heads,kv,graph", [(80, 16, 4, False), (40, 32, 8, True)])
def test_window_decode_is_whole_before_what_follows(M, heads, kv, graph, extra=0):
    """Many decoding rows without page shares, one context much longer than the others, and behind them a programmatically launched product
    that reads the output (a gate on it, then its image): the same bits as with a synchronisation in between."""
    width, N = heads * 128, 256
    attend = _one_row_tiles([4000] + [1] * (M - 1), heads, kv, M, extra)
    g = torch.Generator(device="cuda").manual_seed(1)
    w, w2 = (L().make_wh((torch.randn(n, k, generator=g, device="cuda") * k ** -0.5).bfloat16()) for n, k in ((width, N), (N, width)))
    x, ncap = torch.randn(M, N, generator=g, device="cuda"), (M + 7) // 8 * 8
    xh, oh = (torch.zeros(L().xh_bytes(k, ncap), dtype=torch.uint8, device="cuda") for k in (N, width))
    L().xh_from_rows(x, M, N, ncap, xh)
    out, gated, y = (torch.zeros(M, k, device="cuda") for k in (width, width, N))

    def step(between=lambda: None):
        attend(out)
        between()
        L().dense_tc(w, width, N, xh, ncap, gated, M, epi=L().DENSE_SIGMOID_MUL, aux=out)
        L().xh_from_rows(out, M, width, ncap, oh)
        L().dense_tc(w2, N, width, oh, ncap, y, M)

    step(torch.cuda.synchronize)
    want = [t.clone() for t in (out, gated, y)]
    run = step
    if graph:
        cg, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.graph(cg, stream=side):
            step()
        run = cg.replay
    for _ in range(20):
        for t in (out, gated, y):
            t.zero_()
        run()
        torch.cuda.synchronize()
        for t, ref in zip((out, gated, y), want):
            assert torch.equal(t, ref)


@pytest.mark.parametrize("M,heads,kv,graph", [(80, 16, 4, False), (40, 32, 8, True)])
def test_window_decode_beside_another_grid_is_whole_before_what_follows(M, heads, kv, graph):
    """The same with rows enough said for a prompt among them, so that the grid of the tall tiles is launched between, too."""
    test_window_decode_is_whole_before_what_follows(M, heads, kv, graph, extra=1000)


def test_window_routes_of_an_engine(tmp_path, monkeypatch):
    """An engine says its batch's rows, not its own capacity: a portion of 700 rows of 1024 is tcgen05's alone, decoding mma.sync's, both together both."""
    from dllama_b200.models import registry
    from dllama_b200.models.layered import write_random_model
    layer = {"type": "attention", "mixer": {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 0.1, "mask": {"size": 512}},
             "mlp": {"kind": "dense", "ff": 64}}
    write_random_model(str(tmp_path), {"architecture": "Venadra", "width": 64, "vocab": 64, "norm": {"eps": 1e-5}, "embedding": {"scale": 1.0},
                                       "canon": {"taps": 3}, "layers": [layer]}, seed=2)
    eng = registry.engine_for_dir(str(tmp_path), max_rows=1024, n_slots=4, max_seq_len=1024, dtype="bfloat16")
    routes, call = [], L().window_attention_tc

    def spy(q, out, heads, kv, dim, rd, *a, **opts):
        n_tiles, rq, n_splits = a[-4:-1]
        routes.append(L().window_tc_route(heads, kv, dim, opts["vdim"], opts.get("rows", q.shape[0]), n_tiles, rq, n_splits))
        call(q, out, heads, kv, dim, rd, *a, **opts)
    monkeypatch.setattr(L(), "window_attention_tc", spy)
    tokens = torch.randint(0, 64, (700,), generator=torch.Generator().manual_seed(0)).tolist()
    slots = [eng.alloc_slot() for _ in range(3)]
    eng.forward(tokens, range(700), [slots[0]] * 700)
    eng.forward(tokens[:2], [700, 0], slots[:2])
    eng.forward(tokens[:200] + [5], list(range(200)) + [701], [slots[2]] * 200 + [slots[0]])
    assert routes == [2, 1, 3]
    eng.close()


def _prompt(rows, heads, kv, scale=None, keys=None, seed=5, **opt):
    """A prompt of `rows` positions in one sequence on 128 / 128 bf16 lines, no page shares: call() runs it and returns the output rows."""
    dim, pages = 128, (rows + 31) // 32
    g = torch.Generator(device="cuda").manual_seed(seed)
    cache = torch.randn(128, kv, 32, 2 * dim, generator=g, device="cuda").bfloat16()
    q = torch.randn(4096, heads * dim, generator=g, device="cuda")[:rows]
    if opt.get("bf16_queries"):
        q = q.bfloat16().float()
    if keys is not None:
        keys(cache)
    bt = torch.arange(pages, dtype=torch.int32, device="cuda").view(1, pages)
    rq = L().window_tc_rows(heads, kv)
    n = (rows + rq - 1) // rq
    tiles = torch.full((n * rq,), -1, dtype=torch.int32)
    tiles[:rows] = torch.arange(rows, dtype=torch.int32)
    tiles, pos, slot = tiles.cuda(), torch.arange(rows, dtype=torch.int32, device="cuda"), torch.zeros(rows, dtype=torch.int32, device="cuda")

    def call():
        out = torch.zeros(rows, heads * dim, device="cuda")
        L().window_attention_tc(q, out, heads, kv, dim, 0, dim ** -0.5 if scale is None else scale, opt.get("softcap", 0.0), opt.get("window", 0), pos, slot, bt, cache,
                                tiles, n, rq, vdim=dim)
        return out
    call.q, call.cache = q, cache
    return call


@pytest.mark.parametrize("rows", [20, 1201, 1202, 1203, 1204])
def test_window_prompt_tiles_have_one_owner(rows):
    """The last tile of a prompt has 1 to 4 positions behind a full even tile: fifty runs give the same bits, and its rows are those of the same
    prompt with more positions behind them (which the first rows do not see)."""
    call = _prompt(rows, 16, 4)
    want = _prompt((rows + 31) // 32 * 32, 16, 4)()[:rows]
    for _ in range(50):
        assert torch.equal(call(), want)


def _window_want(call, heads, kv, scale, softcap, window, rows):
    """Output of these rows of a _prompt in 64 bits, from queries as they are."""
    line = call.cache.double().transpose(1, 2).reshape(-1, kv, 256)
    k, v = (line[..., o:o + 128].repeat_interleave(heads // kv, dim=1) for o in (0, 128))
    at = torch.arange(k.shape[0], device="cuda")
    out = []
    for m in rows:
        seen = (at <= m) & ((m - at < window) if window else torch.ones_like(at, dtype=torch.bool))
        s = torch.einsum("hd,thd->ht", call.q[m].double().view(heads, 128), k[seen]) * scale
        if softcap:
            s = softcap * (s / softcap).tanh()
        out.append(torch.einsum("ht,thd->hd", s.softmax(dim=1), v[seen]).reshape(-1))
    return torch.stack(out)


@pytest.mark.parametrize("window,softcap,rows", [(0, 0.0, 1333), (256, 0.0, 2000), (1000, 50.0, 2000)])
def test_window_prompt_probabilities(window, softcap, rows):
    """Queries that bf16 holds, so that the probabilities are all that is rounded: two bf16 numbers each, 2^-17, and a tensor-core chain of at most
    16 steps of 16 tokens that truncates by 2^-24 of the running sum each: 5e-5 covers both several times, one bf16 number (1e-3) misses it."""
    call = _prompt(rows, 16, 4, softcap=softcap, window=window, bf16_queries=True)
    got, some = call().double(), [0, 1, 127, 128, 129, 700, rows - 20, rows - 1]
    want = _window_want(call, 16, 4, 128 ** -0.5, softcap, window, some)
    assert (got[some] - want).norm() <= 5e-5 * want.norm()


@pytest.mark.parametrize("scale", [-0.2, 0.0])
def test_window_prompt_factor_without_order(scale):
    """A score factor that is negative (the smallest product takes the weight) or zero (all positions alike)."""
    rows = 700
    call = _prompt(rows, 16, 4, scale=scale, window=300)
    got, some = call().double(), [0, 1, 299, 300, 511, rows - 1]
    want = _window_want(call, 16, 4, scale, 0.0, 300, some)
    assert (got[some] - want).norm() <= 8e-3 * want.norm()


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_window_prompt_non_finite_keys(value):
    """A key that is not finite, at each place of a group of four: the rows that see it have no finite result (as on the mma.sync kernel), the
    others are as without it."""
    rows, window = 700, 150
    clean = _prompt(rows, 16, 4, window=window)()
    for at in (40, 41, 42, 43, 330):
        def spoil(cache):
            cache[at // 32, :, at % 32, :128] = value
        out = _prompt(rows, 16, 4, window=window, keys=spoil)()
        seen = torch.zeros(rows, dtype=torch.bool, device="cuda")
        seen[at:at + window] = True
        assert torch.equal(out[~seen], clean[~seen])
        bad = ~torch.isfinite(out[seen].view(-1, 128)).all(dim=1)
        assert bad.all() if value != value else bad.view(-1, 16).any(dim=1).float().mean() > 0.9


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("window,at", [(0, 104), (0, 680), (0, 1130), (256, 650), (150, 330), (1000, 40)])
def test_window_prompt_non_finite_values(value, window, at):
    """A value that is not finite reaches the tile of 32 positions that holds it and those that see it, or whose first page does: the tile beside one of them in
    a CTA is as without it."""
    rows = 1201
    clean = _prompt(rows, 16, 4, window=window)()

    def spoil(cache):
        cache[at // 32, :, at % 32, 128:] = value
    out = _prompt(rows, 16, 4, window=window, keys=spoil)()
    first = torch.arange(rows, device="cuda") // 32 * 32                       # of a row's tile
    reached = (first + 31 >= at) & (((first - window + 1).clamp(min=0) // 32 * 32 <= at) if window else torch.ones_like(first, dtype=torch.bool))
    assert torch.equal(out[~reached], clean[~reached])
    seen = torch.arange(rows, device="cuda")
    seen = (seen >= at) & ((seen - at < window) if window else True)
    assert not torch.isfinite(out[seen]).any()


@pytest.mark.parametrize("M,N,K_,batch,dtype", [(1, 40, 2048, 1, "bf16"), (1, 30000, 256, 1, "bf16"), (2, 24, 512, 3, "bf16"), (2, 9000, 128, 2, "f32"), (3, 20000, 264, 1, "bf16"),
                                                (4, 1000, 256, 24, "bf16"), (4, 64, 4096, 1, "f32"), (8, 3000, 72, 8, "f32"), (32, 64, 64, 1, "f32"), (16, 2000, 64, 16, "f32"),
                                                (25, 100, 520, 1, "f32")])
def test_dense_rows_by_shape(M, N, K_, batch, dtype):
    """Few rows on every side of the rules that choose between staged and direct rows, mma, rounds and tiles, plain and in pairs, one product and a
    batch of them.  f32 sums of K terms: 3e-6."""
    g = torch.Generator(device="cuda").manual_seed(M * 1000 + N)
    w = (torch.randn(batch, N, K_, generator=g, device="cuda") * K_ ** -0.5).to(torch.bfloat16 if dtype == "bf16" else torch.float32)
    x = torch.randn(M, batch * K_, generator=g, device="cuda")
    z = torch.einsum("mbk,bnk->mbn", (x.bfloat16() if dtype == "bf16" else x).double().view(M, batch, K_), w.double())
    for pair in (False, True):
        width = N // 2 if pair else N
        want = torch.nn.functional.gelu(z[..., 0::2], approximate="tanh") * z[..., 1::2] if pair else z
        y = torch.zeros(M, batch * width, device="cuda")
        a = lib().DlDenseArgs()
        a.W, a.wtype, a.ldw, a.w_bs = w.data_ptr(), 1 if dtype == "bf16" else 0, K_, N * K_
        a.X, a.ldx, a.x_bs, a.Y, a.ldy, a.y_bs = x.data_ptr(), batch * K_, K_, y.data_ptr(), batch * width, width
        a.M, a.N, a.K, a.batch, a.round_x, a.epi = M, N, K_, batch, 1 if dtype == "bf16" else 0, L().DENSE_GLU_GELU if pair else 0
        L().check_layers(L().layers_lib().dl_dense(a, torch.cuda.current_stream().cuda_stream), "dl_dense")
        got = y.double().view(M, batch, width)
        assert (got - want).norm() <= 3e-6 * want.norm()


@pytest.mark.parametrize("M,N,K_", [(3, 2048, 512), (8, 100, 2048), (16, 4096, 520), (31, 200, 8200)])
def test_dense_mma_rounds_once(M, N, K_):
    """Products of numbers of one sign, which nothing cancels: off by no more than one rounding to f32 (half a unit in the last place, 2^-24;
    truncated sums chained to each other were off by 8e-8 to 9e-8).  An infinite sum stays infinite."""
    g = torch.Generator(device="cuda").manual_seed(M * 1000 + N)
    w, x = torch.randn(N, K_, generator=g, device="cuda").abs().bfloat16(), torch.randn(M, K_, generator=g, device="cuda").abs()
    want, y = x.bfloat16().double() @ w.double().t(), torch.zeros(M, N, device="cuda")
    L().dense(w, x, y, M, True)
    assert (y - want).norm() <= 2.0 ** -24 * want.norm()
    over, w[0], x[1, 5] = torch.zeros(M, N, device="cuda"), 0.5, float("inf")
    L().dense(w, x, over, M, True)
    assert over[1, 0] == float("inf") and not torch.isfinite(over[1]).any() and torch.equal(over[2, 1:], y[2, 1:])


def _decode_one(q, k, v, kv_heads):
    """One row of decode attention over these keys and values [tokens][kv][hs] and its result in 64 bits."""
    heads, hs, T = q.shape[0], q.shape[1], k.shape[0]
    pages = (T + 31) // 32
    kc, vc = (torch.zeros(pages * 32, kv_heads, hs, dtype=torch.float16) for _ in range(2))
    kc[:T], vc[:T] = k.half(), v.half()
    paged = [c.view(pages, 32, kv_heads, hs).transpose(1, 2).contiguous().cuda() for c in (kc, vc)]
    y = torch.zeros(1, heads * hs, device="cuda")
    scratch = torch.zeros(K().attention_scratch_bytes(1, heads, hs, 2), dtype=torch.uint8, device="cuda")
    K().attention(q.reshape(1, -1).cuda(), 1, heads, kv_heads, hs, *paged, torch.tensor([T - 1], dtype=torch.int32, device="cuda"),
                  torch.zeros(1, dtype=torch.int32, device="cuda"), torch.arange(pages, dtype=torch.int32, device="cuda").view(1, -1), pages, 2, scratch,
                  None, None, 1, y)
    kk, vv = (c[:T].double().repeat_interleave(heads // kv_heads, dim=1) for c in (kc, vc))
    p = (torch.einsum("hd,thd->ht", q.double(), kk) * hs ** -0.5).softmax(dim=1)
    return y.cpu().double().view(heads, hs), torch.einsum("ht,thd->hd", p, vv)


@pytest.mark.parametrize("hs", [64, 128])
@pytest.mark.parametrize("q_size,k_size", [(1.0, 1.0), (1e-3, 1e3), (1e-4, 1e4), (1e-5, 1e4), (2000.0, 1e-3)])
def test_decode_attention_small_queries(hs, q_size, k_size):
    """Queries far from 1 against keys that make up for it: f32 products keep 24 bits of each.  Bound: a score's terms add up to at most 20 here, so
    its f32 sum is within a few 2^-24 of that, 2e-6, as the softmax and its sums are."""
    g = torch.Generator().manual_seed(hs)
    q, k, v = torch.randn(4, hs, generator=g) * q_size, torch.randn(300, 1, hs, generator=g) * k_size, torch.randn(300, 1, hs, generator=g)
    got, want = _decode_one(q, k, v, 1)
    assert (got - want).norm() <= 2e-6 * want.norm()


@pytest.mark.parametrize("hs", [64, 128])
@pytest.mark.parametrize("tokens", [16, 40, 300])
def test_decode_attention_as_exact_as_f32(hs, tokens):
    """128 rows over as many tokens each: no further from 64 bits than the f32 arithmetic that a cache of f32 takes on the same numbers."""
    M, heads, kv, pages = 128, 32, 8, (tokens + 31) // 32
    g = torch.Generator(device="cuda").manual_seed(hs + tokens)
    q = torch.randn(M, heads * hs, generator=g, device="cuda")
    k, v = (torch.randn(M * pages, kv, 32, hs, generator=g, device="cuda").half() for _ in range(2))
    bt, slot = torch.arange(M * pages, dtype=torch.int32, device="cuda").view(M, pages), torch.arange(M, dtype=torch.int32, device="cuda")
    scratch = torch.zeros(K().attention_scratch_bytes(M, heads, hs, 1), dtype=torch.uint8, device="cuda")
    kk, vv = (c.double().view(M, pages, kv, 32, hs).transpose(2, 3).reshape(M, -1, kv, hs)[:, :tokens].repeat_interleave(heads // kv, dim=2) for c in (k, v))
    want = torch.einsum("mht,mthd->mhd", (torch.einsum("mhd,mthd->mht", q.double().view(M, heads, hs), kk) * hs ** -0.5).softmax(dim=2), vv).reshape(M, -1)
    off = []
    for cast in (torch.half, torch.float):
        y = torch.zeros(M, heads * hs, device="cuda")
        K().attention(q, M, heads, kv, hs, k.to(cast), v.to(cast), torch.full((M,), tokens - 1, dtype=torch.int32, device="cuda"), slot, bt, pages, 1, scratch,
                      None, None, M, y)
        off.append(float((y - want).norm() / want.norm()))
    assert off[0] <= off[1], off


@pytest.mark.parametrize("hs", [64, 128])
@pytest.mark.parametrize("below", [13, 20, 30])
def test_decode_attention_small_weights(hs, below):
    """One token takes the weight and has no value; the others are 2^-below of it and make up the output.  f32 weights keep 24 bits each; a score
    near -below in units of log2 is rounded to 2^-24 of itself, 2e-6 for 30, which is the largest share: 6e-6."""
    g = torch.Generator().manual_seed(below)
    q, k, v = torch.zeros(4, hs), torch.zeros(200, 1, hs), torch.randn(200, 1, hs, generator=g) * 1000
    q[:, 0] = hs ** 0.5 * 0.6931471805599453
    k[:, 0, 0] = -(below + torch.rand(200, generator=g))
    k[7], v[7] = 0, 0
    got, want = _decode_one(q, k, v, 1)
    assert (got - want).norm() <= 6e-6 * want.norm()


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_window_decode_non_finite_values_far_below(value):
    """A value that is not finite, under a weight that a share's merge rounds to zero, on shares with and without pages: the column that it stands in is not
    finite (0 times it), and no other column changes."""
    heads, kv, dim, tokens, n_splits = 8, 2, 128, 300, 16
    g = torch.Generator(device="cuda").manual_seed(5)
    pages = (tokens + 31) // 32
    cache = torch.randn(pages, kv, 32, 2 * dim, generator=g, device="cuda").bfloat16()
    q = torch.ones(1, heads * dim, device="cuda")
    cache[0, :, :, :dim] = -2.0                    # the first page: scores of -256, the others' some 10
    rq = L().window_tc_rows(heads, kv)
    tiles = torch.full((1, rq), -1, dtype=torch.int32, device="cuda")
    tiles[0, 0] = 0
    pos, slot, bt = (torch.tensor(v, dtype=torch.int32, device="cuda") for v in ([tokens - 1], [0], [list(range(pages))]))
    partial, outs = torch.full((kv * n_splits * 64 * (dim + 2),), float("nan"), device="cuda"), []
    for bad in (False, True):
        if bad:
            cache[0, 1, 7, dim + 3] = value
        outs.append(torch.zeros(1, heads * dim, device="cuda"))
        L().window_attention_tc(q, outs[-1], heads, kv, dim, 0, 1.0, 0.0, 0, pos, slot, bt, cache, tiles, 1, rq, n_splits, partial, vdim=dim)
    clean, out = (o.view(kv, heads // kv, dim) for o in outs)
    assert torch.isfinite(clean).all() and not torch.isfinite(out[1, :, 3]).any()
    out[1, :, 3] = clean[1, :, 3]
    assert torch.equal(out, clean)


@pytest.mark.parametrize("heads,kv,segs", [(40, 40, [(0, 0, 257), (257, 50, 200)]), (32, 8, [(0, 7, 385), (385, 0, 129)]), (33, 11, [(0, 1, 640)])])
def test_prompt_attention_two_tiles(heads, kv, segs):
    """More tiles than SMs: two heads of a key/value head side by side, or (heads alone, or three of them) two row tiles of one head, the second one
    missing or a step longer; several items per CTA."""
    from test_gpu_kernels import test_attention_prefill_matches_reference as check
    check(heads, kv, 128, segs, True)


@pytest.mark.parametrize("runs,n_splits,rows,ld", [([(1500, 40)], 8, True, 0), ([(1500, 40)], 8, False, 2), ([(900, 64), (40, 3), (1200, 1), (0, 17)], 6, True, 0),
                                                   ([(700, 1), (5, 1), (1999, 1)], 7, True, 0), ([(0, 16)], 4, True, 0), ([(640, 130), (3, 20)], 16, True, 0)])
def test_window_shares(runs, n_splits, rows, ld):
    """Page shares of tall tiles and of decoding ones, alone and in one call, with and without the number of rows said, output rows of 8 bytes: against
    the per-row kernel (queries and weights rounded to bf16 here: 8e-3)."""
    heads, kv, dim, pages = 8, 2, 128, 64
    g = torch.Generator().manual_seed(n_splits)
    M = sum(n for _, n in runs)
    cache = torch.randn(len(runs) * pages, kv, 32, 2 * dim, generator=g).bfloat16().cuda()
    bt = torch.randperm(len(runs) * pages, generator=g).int().view(len(runs), pages).cuda()
    pos, slot, tiles = [], [], []
    for s, (p0, n) in enumerate(runs):
        at = list(range(len(pos), len(pos) + n))
        pos += list(range(p0, p0 + n))
        slot += [s] * n
        tiles += [at[i:i + 16] for i in range(0, n, 16)]
    tr = torch.tensor([t + [-1] * (16 - len(t)) for t in tiles], dtype=torch.int32, device="cuda")
    q = torch.randn(M if rows else M + 1000, heads * dim, generator=g).bfloat16().float().cuda()
    pos, slot = (torch.tensor(v, dtype=torch.int32, device="cuda") for v in (pos, slot))
    wide = torch.zeros(M, heads * dim + ld, device="cuda")
    got = wide[:, :heads * dim]
    want = torch.zeros(M, heads * dim, device="cuda")
    partial = torch.full((L().window_tc_partial_floats(len(tiles), kv, n_splits, dim),), float("nan"), device="cuda")
    L().window_attention_tc(q, got, heads, kv, dim, 0, 0.1, 0.0, 0, pos, slot, bt, cache, tr, len(tiles), 16, n_splits, partial, vdim=dim)
    L().window_attention(q, want, M, heads, kv, dim, 0, 0.1, 0.0, 0, pos, slot, bt, cache, vdim=dim)
    assert ((got - want).norm(dim=1) <= 8e-3 * want.norm(dim=1)).all()


def _window_batch(runs, heads, kv, window=0, softcap=0.0, chunk=0):
    """Portions (first position, rows) of one sequence each on 128 / 128 bf16 lines, full list tiles, queries that bf16 holds: the tensor-core kernels' output
    rows (a call of them) and the per-row kernel's."""
    dim, rq = 128, L().window_tc_rows(heads, kv)
    pages = max((p0 + n + 31) // 32 for p0, n in runs)
    g = torch.Generator().manual_seed(len(runs) * 1000 + runs[0][1])
    M = sum(n for _, n in runs)
    cache = torch.randn(len(runs) * pages, kv, 32, 2 * dim, generator=g).bfloat16().cuda()
    bt = torch.randperm(len(runs) * pages, generator=g).int().view(len(runs), pages).cuda()
    pos, slot, tiles = [], [], []
    for s, (p0, n) in enumerate(runs):
        at = list(range(len(pos), len(pos) + n))
        pos += list(range(p0, p0 + n))
        slot += [s] * n
        tiles += [at[i:i + rq] for i in range(0, n, rq)]
    tr = torch.tensor([t + [-1] * (rq - len(t)) for t in tiles], dtype=torch.int32, device="cuda")
    q = torch.randn(M, heads * dim, generator=g).bfloat16().float().cuda()
    pos, slot = (torch.tensor(v, dtype=torch.int32, device="cuda") for v in (pos, slot))
    want = torch.zeros(M, heads * dim, device="cuda")
    L().window_attention(q, want, M, heads, kv, dim, 0, 0.1, softcap, window, pos, slot, bt, cache, vdim=dim, chunk=chunk)

    def call():
        out = torch.full((M, heads * dim), float("nan"), device="cuda")
        L().window_attention_tc(q, out, heads, kv, dim, 0, 0.1, softcap, window, pos, slot, bt, cache, tr, len(tiles), rq, vdim=dim, chunk=chunk)
        return out
    return call, want


@pytest.mark.parametrize("runs,heads,kv,opt", [([(0, 272), (0, 400)], 32, 8, {}),                       # one tile of a prompt and three of the next in a CTA
                                               ([(96, 688), (0, 17)], 32, 8, {}),                      # three and one, the second tile a step longer
                                               ([(100, 1100)], 32, 8, dict(window=1000)), ([(300, 1100)], 32, 8, dict(window=1024)),
                                               ([(100, 1100)], 32, 8, dict(window=1024, softcap=50.0)), ([(300, 1100)], 32, 8, dict(window=1000, softcap=50.0)),
                                               ([(300, 1200)], 16, 4, dict(window=256, softcap=50.0)),
                                               ([(100, 1100)], 32, 8, dict(chunk=1024)),               # the border between the tiles' first positions
                                               ([(300, 500), (0, 200), (1000, 1), (50, 1), (31, 1), (700, 3)], 32, 8, dict(window=512)),
                                               ([(7 * k, 40 + 9 * k) for k in range(12)], 64, 8, {}), ([(k, 20 + k) for k in range(40)], 32, 8, dict(window=30))])
def test_window_tiles_of_several_portions(runs, heads, kv, opt):
    """Groups of four list tiles (more of them than SMs): several runs in a CTA, runs of one tile ahead of two and the reverse, tiles that start and end at
    different steps; twenty calls give the same bits.  Probabilities in two bf16 numbers (2^-17), a chain of at most 32 steps that truncates by 2^-24 of the
    running sum each, fast exponentials (2^-22): 2e-4 of a row covers them several times."""
    assert (sum((n - 1) // (64 * kv // heads) + 1 for _, n in runs) + 1) // 2 * kv > 148
    call, want = _window_batch(runs, heads, kv, **opt)
    got = call()
    assert ((got - want).norm(dim=1) <= 2e-4 * want.norm(dim=1)).all()
    for _ in range(20):
        assert torch.equal(call(), got)


def _give_up(library):
    """A limit that is over before the kernel starts: its waits for copies end at once, none is left forever."""
    library.dl_debug_set_attention_limit.argtypes = [C.c_ulonglong]
    library.dl_debug_set_attention_limit(0)
    return lambda: library.dl_debug_set_attention_limit(4_000_000_000)


def test_a_wait_that_gives_up_reaches_the_caller(tmp_path):
    """Prompt attention of both kinds: the status word changes once for a launch whose waits gave up and never for others; an engine raises where it
    reads its tokens, and at the next batch where it does not, once, and goes on."""
    from dllama_b200.formats import mfile
    from dllama_b200.models.llama import LlamaEngine
    from dllama_b200.ops import lib as B
    call = _prompt(300, 16, 4)
    status, want = B.WaitStatus(B.layers_lib()), call()
    restore = _give_up(B.layers_lib())
    try:
        out = call()
        torch.cuda.synchronize()
    finally:
        restore()
    assert out.isnan().any()
    with pytest.raises(B.NativeLibraryError, match="gave up"):
        status.check()
    assert torch.equal(call(), want)
    status.check()

    path = str(tmp_path / "m.m")
    mfile.write_random_model(path, dict(mfile.MODEL_SHAPES["tiny"], dim=1024, hidden_dim=2048), exact=True, seed=3)
    e = LlamaEngine(path, max_rows=256, n_slots=2, max_seq_len=512, use_graphs=False)
    slot, n = e.alloc_slot(), 200
    batch = (np.random.default_rng(0).integers(1, 1000, n).tolist(), list(range(n)), [slot] * n)
    token = e.decode_step_greedy(*batch, logits_from=n - 1)
    for step in (e.decode_step_greedy, e.forward):
        restore = _give_up(B.cuda_lib())
        try:
            with pytest.raises(B.NativeLibraryError, match="gave up"):
                step(*batch, logits_from=n - 1)
                torch.cuda.synchronize()             # forward alone: the next batch raises
                step(*batch, logits_from=n - 1)
        finally:
            restore()
        torch.cuda.synchronize()
        assert e.decode_step_greedy(*batch, logits_from=n - 1) == token
    e.close()
