"""Epilogues by whole warps (plain, SiLU and rotary), Q40 expansion, tile widths and the norm's wide form of the Q40 products, and the walk over the states of a gated scan, at
the sizes where they can go wrong: remainders of tiles and chunks, addresses that are not 16-byte aligned, scales at the ends of fp16."""
import numpy as np
import pytest
import torch

from dllama_b200.ops import quant

pytestmark = pytest.mark.gpu


def K():
    from dllama_b200.ops import kernels
    return kernels


def L():
    from dllama_b200.ops import layers
    return layers


def _q40(d, n, seed):
    rng = np.random.default_rng(seed)
    raw = quant.quantize_q40((rng.standard_normal((d, n)) * 0.05).astype(np.float32))
    return torch.from_numpy(raw.reshape(-1)).cuda(), quant.dequantize_q40(raw).reshape(d, n)


def _activations(n, M, ncap, seed):
    x = np.random.default_rng(seed).standard_normal((M, n)).astype(np.float32)
    xh = K().alloc_xh(n, ncap, "cuda")
    K().quant_q80(torch.from_numpy(x).cuda(), M, n, ncap, None, xh)
    return quant.q80_roundtrip(x).astype(np.float64), xh


@pytest.mark.parametrize("d,n,M,S", [(300, 512, 5, 1), (132, 512, 16, 2), (512, 1024, 33, 4), (256, 512, 70, 2), (388, 512, 128, 4), (38912, 128, 20, 1),
                                     (38912, 128, 128, 1), (9600, 256, 150, 1), (9600, 256, 430, 1), (130, 512, 9, 1), (768, 4096, 20, 8), (1280, 2048, 40, 8), (384, 1024, 3, 8)])
@pytest.mark.parametrize("roundtrip", [False, True])
def test_store_epilogue_aligned_or_not(d, n, M, S, roundtrip):
    """The same values, bit for bit, whether rows start on 16 bytes (four values per thread) or not (one); tiles alone, in pairs, in shares of K and of
    every width.  Against f64: operands rounded to fp16, sums of n terms."""
    k = K()
    ncap = (M + 255) // 256 * 256 if M > 128 else 16 if M <= 16 else 32 if M <= 32 else 64 if M <= 64 else 128
    w, wdq = _q40(d, n, d + M)
    w = k.make_q40t(w, d, n)
    x, xh = _activations(n, M, ncap, M)
    res = torch.randn(M, d + 3, device="cuda")
    out = []
    for shift, ld in ((0, (d + 3) // 4 * 4), (1, d + 3)):
        buf = torch.full((M * ld + 8,), float("nan"), device="cuda")
        r = torch.zeros(M * ld + 8, device="cuda")
        r[shift:shift + M * ld].view(M, ld)[:, :d] = res[:, :d]
        k.gemm_q40_tc(w, d, n, xh, ncap, M, k.epi_store([buf.data_ptr() + 4 * shift], ld, 0, roundtrip, residual=r.data_ptr() + 4 * shift, residual_ld=ld), S)
        y = buf[shift:shift + M * ld].view(M, ld)
        assert torch.isnan(y[:, d:]).all() and not torch.isnan(y[:, :d]).any()
        out.append(y[:, :d].clone())
    assert torch.equal(out[0], out[1])
    want = x @ wdq.T.astype(np.float64)
    scale = np.abs(want).max()
    tol = 2e-3 * scale + (scale / 127 if roundtrip else 0)      # a cast of blocks is good to half a step of the block's largest value
    assert np.abs(out[0].double().cpu().numpy() - res[:, :d].double().cpu().numpy() - want).max() <= tol


@pytest.mark.parametrize("d,n,M,force_cg", [(512, 256, 300, 0), (384, 256, 129, 0), (300, 256, 257, 0), (4096, 256, 768, 0), (132, 128, 40, 1)])
def test_prompt_product_aligned_or_not(d, n, M, force_cg):
    """As above for the product on expanded weights, whose tiles have 128 to 256 rows."""
    k = K()
    ncap = (M + 7) // 8 * 8
    w, wdq = _q40(d, n, d + M)
    wh = k.q40t_to_wh(k.make_q40t(w, d, n), d, n)
    x, xh = _activations(n, M, ncap, M)
    out = []
    for shift, ld in ((0, (d + 3) // 4 * 4), (1, d + 1)):
        buf = torch.full((M * ld + 8,), float("nan"), device="cuda")
        k.gemm_wh_tc(wh, d, n, xh, ncap, M, k.epi_store([buf.data_ptr() + 4 * shift], ld, 0, False), force_cg)
        out.append(buf[shift:shift + M * ld].view(M, ld)[:, :d].clone())
    assert torch.equal(out[0], out[1])
    want = x @ wdq.T.astype(np.float64)
    np.testing.assert_allclose(out[0].cpu().numpy(), want, rtol=0, atol=2e-3 * np.abs(want).max())


@pytest.mark.parametrize("d,n,M", [(4096, 4096, 768), (4096, 4096, 2001), (9728, 4096, 1100), (512, 8192, 300), (2048, 4096, 150), (1280, 5120, 40)])
def test_prompt_product_pairs_and_single_ctas(d, n, M):
    """Pairs of CTAs, whose ring of three stages wraps many times in a tile and across tiles with one CTA ahead of the other, give the bits that single CTAs
    give (both add the same products in the same order), call for call."""
    k = K()
    ncap = (M + 7) // 8 * 8 + 8
    w, _ = _q40(d, n, d + M)
    wh = k.q40t_to_wh(k.make_q40t(w, d, n), d, n)
    _, xh = _activations(n, M, ncap, M)
    out = []
    for force_cg in [1] + [0] * 10:
        y = torch.zeros(M, d, device="cuda")
        k.gemm_wh_tc(wh, d, n, xh, ncap, M, k.epi_store([y.data_ptr()], d, 0, False), force_cg)
        out.append(y)
    assert out[0].abs().max() > 0 and all(torch.equal(y, out[0]) for y in out[1:])


@pytest.mark.parametrize("force_cg", [0, 1])
def test_prompt_product_of_an_images_last_part(force_cg):
    """Activations that are the last part of a larger image, which ends behind their last row (a tile has more): the same bits as from an image of their own."""
    k = K()
    d, n, M, parts = 512, 512, 136, 5
    w, _ = _q40(d, n, 3)
    wh = k.q40t_to_wh(k.make_q40t(w, d, n), d, n)
    _, xh = _activations(n, M, M, 5)
    image = torch.zeros(n // 128, parts, M // 8 * 2048, dtype=torch.uint8, device="cuda")
    image[:, -1] = xh.view(n // 128, -1)
    part = image.view(-1)[(parts - 1) * (M // 8) * 2048:]
    out = []
    for x, ncap in ((xh, M), (part, parts * M)):
        y = torch.zeros(M, d, device="cuda")
        k.gemm_wh_tc(wh, d, n, x, ncap, M, k.epi_store([y.data_ptr()], d, 0, False), force_cg)
        out.append(y)
    assert out[0].abs().max() > 0 and torch.equal(*out)


def _product(kernel, w, d, n, xh, ncap, M, S, epi):
    k = K()
    if kernel == "q40":
        k.gemm_q40_tc(w, d, n, xh, ncap, M, epi, S)
    else:
        k.gemm_wh_tc(k.q40t_to_wh(w, d, n), d, n, xh, ncap, M, epi)


# rows that end inside a group of 8, ranks whose rows start inside one, ranks with a row or none, several tiles, chunks of 64 rows
CASES = [("q40", M, S) for M in (1, 3, 13, 33, 70) for S in (1, 2, 4)] + [("q40", 9, 8), ("q40", 150, 1), ("q40", 256, 2), ("wh", 1, 1), ("wh", 129, 1), ("wh", 300, 1)]


@pytest.mark.parametrize("kernel,M,S", CASES)
@pytest.mark.parametrize("hid,gelu", [(384, False), (160, True)])
def test_silu_epilogue_by_warps_or_by_values(kernel, M, S, hid, gelu):
    """The image of act(gate) * up is the same bit for bit whether whole warps write it or (with a second image asked for) one value per thread does, and the
    rows behind the last stay as they were.  Against f64: half a step of the cast and fp16 operands."""
    k = K()
    d, n = 2 * hid, 1024
    ncap = 16 if M <= 16 else 32 if M <= 32 else 64 if M <= 64 else (M + 255) // 256 * 256
    w, wdq = _q40(d, n, d)
    w = k.make_q40t(w, d, n)
    x, xh = _activations(n, M, ncap, M)
    wide, out = (hid + 127) // 128 * 128, []
    for xq in (None, k.alloc_xq(wide, ncap, "cuda")):
        image = torch.full((k.xh_bytes(wide, ncap),), 0x3A, dtype=torch.uint8, device="cuda")
        _product(kernel, w, d, n, xh, ncap, M, S, k.epi_silu_mul(xq, image, ncap, gelu))
        out.append(image)
    assert torch.equal(*out)
    rows = out[0].view(wide // 128, ncap // 8, 16, 8, 16).permute(1, 3, 0, 2, 4).reshape(ncap, -1)       # a row's 16-byte pieces
    assert (rows[M:] == 0x3A).all()
    y = x @ wdq.T.astype(np.float64)
    g, u = y[:, 0::2], y[:, 1::2]
    want = (0.5 * g * (1 + np.tanh(0.797884560802865 * (g + 0.044715 * g ** 3))) if gelu else g / (1 + np.exp(-g))) * u
    # K-slot order inside a block of 32 (xh_slot): value 16 hi + 4 w + r at piece w, place 4 hi + (0, 2, 1, 3)[r]
    got = rows[:M].contiguous().view(torch.float16).view(M, -1, 4, 8).double().cpu().numpy()             # [row][block][piece][place]
    e = np.arange(32)
    got = got[:, :, (e & 15) >> 2, (e >> 4) * 4 + np.array([0, 2, 1, 3])[e & 3]].reshape(M, -1)[:, :hid]
    scale = np.abs(want).max()
    assert np.abs(got - want).max() <= scale / 127 * 0.51 + 5e-3 * scale


@pytest.mark.parametrize("kernel,M,S", CASES)
@pytest.mark.parametrize("heads,kv_heads,hs,dtype", [(3, 1, 64, torch.float16), (5, 3, 64, torch.float32), (3, 2, 128, torch.float16), (1, 1, 128, torch.float32)])
def test_rope_epilogue_by_warps_or_by_values(kernel, M, S, heads, kv_heads, hs, dtype):
    """Rotated queries and keys, and values, of heads whose regions begin and end inside a tile, into caches of both types: the same bit for bit whether rows start
    on 16 bytes (two pairs per thread) or not (one value).  Against f64: fp16 operands and, in the caches, results; angles in f32."""
    k = K()
    q_dim, kv_dim, n, pages = heads * hs, kv_heads * hs, 1024, 12
    d = q_dim + 2 * kv_dim
    ncap = 16 if M <= 16 else 32 if M <= 32 else 64 if M <= 64 else (M + 255) // 256 * 256
    w, wdq = _q40(d, n, d)
    w = k.make_q40t(w, d, n)
    x, xh = _activations(n, M, ncap, M)
    freqs = 10000.0 ** (-torch.arange(hs // 2, dtype=torch.float64) / (hs // 2))
    freqs = freqs.float().cuda()
    rng = np.random.default_rng(M)
    slots = rng.integers(0, 2, M)                                    # two sequences, their rows mixed
    pos = np.array([5 + 7 * s + int((slots[:i] == s).sum()) for i, s in enumerate(slots)])
    table = rng.permutation(2 * pages).reshape(2, pages).astype(np.int32)
    i32 = lambda t: torch.tensor(np.asarray(t), dtype=torch.int32, device="cuda")
    out = []
    for shift in (0, 1):
        q = torch.full((M * q_dim + 8,), 7.0, device="cuda")
        kc, vc = (torch.full((2 * pages, kv_heads, 32, hs), 7.0, dtype=dtype, device="cuda") for _ in range(2))
        keep = (i32(pos), i32(slots), i32(table))
        _product(kernel, w, d, n, xh, ncap, M, S, k.epi_qkv_rope(q[shift:], q_dim, kv_dim, hs, freqs, *keep, pages, kv_heads, kc, vc))
        torch.cuda.synchronize()
        assert (q[shift + M * q_dim:] == 7).all()
        out.append((q[shift:shift + M * q_dim].view(M, q_dim), kc, vc))
    assert all(torch.equal(a, b) for a, b in zip(*out))
    y = x @ wdq.T.astype(np.float64)
    ang = pos[:, None].astype(np.float64) * freqs.double().cpu().numpy()
    rot = lambda t: np.stack([t[..., 0::2] * np.cos(ang)[:, None] - t[..., 1::2] * np.sin(ang)[:, None],
                              t[..., 0::2] * np.sin(ang)[:, None] + t[..., 1::2] * np.cos(ang)[:, None]], axis=-1).reshape(t.shape)
    parts = [rot(y[:, :q_dim].reshape(M, -1, hs)), rot(y[:, q_dim:q_dim + kv_dim].reshape(M, -1, hs)), y[:, q_dim + kv_dim:].reshape(M, -1, hs)]
    q, kc, vc = (t.double().cpu().numpy() for t in out[0])
    tol = 3e-3 * np.abs(y).max()
    assert np.abs(q.reshape(M, -1, hs) - parts[0]).max() <= tol
    at = table[slots, pos // 32], slice(None), pos % 32
    assert np.abs(kc[at] - parts[1]).max() <= tol and np.abs(vc[at] - parts[2]).max() <= tol
    kc[at] = vc[at] = 7
    assert (kc == 7).all() and (vc == 7).all()


@pytest.mark.parametrize("scales", [(6e-8, 1e-6, 3e-5, 1e-4), (9e-4, 0.0039, 0.03, 0.0624), (0.0624, 0.0625, 0.07, 1.0), (-0.0624, -0.0625, -3.0, 1e-4), (0.0, 2.0, -1e-5, 500.0)])
def test_q40_expansion_rounds_once(scales):
    """Every nibble under scales from fp16's subnormals up, on both sides of the largest that one fma takes: (nibble - 8) d rounded once, in the expanded
    image and in the fused product, which agree."""
    k = K()
    d, n, M = 128, 256, 16
    rng = np.random.default_rng(1)
    nib = rng.integers(0, 16, (d, n // 32, 32))
    nib[:, 0, :16], nib[:, 0, 16:] = np.arange(16), np.arange(16)[::-1]
    sc = np.asarray(scales, dtype=np.float16)[rng.integers(0, len(scales), (d, n // 32))]
    raw = np.concatenate([sc[..., None].view(np.uint8), (nib[..., :16] | nib[..., 16:] << 4).astype(np.uint8)], axis=2)
    w = k.make_q40t(torch.from_numpy(raw.reshape(-1)).cuda(), d, n)
    want = ((nib - 8) * sc[..., None].astype(np.float64)).astype(np.float16).astype(np.float64).reshape(d, n)
    # unit activations pick the expanded values out one by one: column c of 16 rows at a time
    got = np.zeros_like(want)
    wh = k.q40t_to_wh(w, d, n)
    for c0 in range(0, n, M):
        x = np.zeros((M, n), dtype=np.float32)
        x[np.arange(M), c0 + np.arange(M)] = 127.0
        xh = k.alloc_xh(n, M, "cuda")
        k.quant_q80(torch.from_numpy(x).cuda(), M, n, M, None, xh)
        for run in (lambda e: k.gemm_q40_tc(w, d, n, xh, M, M, e, 1), lambda e: k.gemm_wh_tc(wh, d, n, xh, M, M, e, 1)):
            y = torch.zeros(M, d, device="cuda")
            run(k.epi_store([y.data_ptr()], d))
            assert np.array_equal(y.double().cpu().numpy().T, want[:, c0:c0 + M] * 127.0)


@pytest.mark.parametrize("M,dim", [(1184, 4096), (1185, 4128), (1191, 8192), (1200, 544)])
def test_norm_of_many_rows(M, dim):
    """Eight rows per CTA (from 1184) against a row per CTA: the merged sums bit for bit, the norm but for the order of its sum of squares, the cast
    but for one step of a block's values (the 127th part of its largest, no more than the largest of all); dims beyond what a thread keeps in registers, rows
    that end inside a CTA."""
    k = K()
    torch.manual_seed(M)
    ncap = (M + 127) // 128 * 128
    x, parts, w = torch.randn(M, dim, device="cuda"), torch.randn(2, M, dim, device="cuda"), torch.rand(dim, device="cuda") + 0.5
    img = []
    for step in (M, 592):
        xh, xo, yo = k.alloc_xh((dim + 127) // 128 * 128, ncap, "cuda"), torch.zeros(M, dim, device="cuda"), torch.zeros(M, dim, device="cuda")
        for m0 in range(0, M, step):
            m1 = min(M, m0 + step)
            k.reduce_norm_quant(x[m0:m1], xo[m0:m1], parts[:, m0:m1].contiguous().data_ptr(), 2, (m1 - m0) * dim, None, None, 0, 0, w, 1e-5, dim, m1 - m0, ncap, None,
                                xh[m0 // 8 * 2048:], yo[m0:m1])
        img.append((xh.view(torch.float16).float(), xo, yo))
    (h0, x0, y0), (h1, x1, y1) = img
    assert torch.equal(x0, x1) and torch.equal(x0, (x + parts[0]) + parts[1])
    assert ((y0 - y1).abs() <= 1e-6 * y0.abs()).all()
    assert (h0 - h1).abs().max() <= y0.abs().max() / 127 * 1.001 and (h0 != h1).float().mean() < 1e-3 and h0.abs().max() > 1


@pytest.mark.parametrize("vdim,rows", [(36, [64 * 8 + 1, 200]), (37, [64 * 9, 130]), (128, [64 * 17 + 5, 129])])
def test_chunked_scan_walks_every_chunk(vdim, rows):
    """States in pieces of four (vdim % 4 == 0) and one by one, chunks that do not fill the last eight, a fresh and a continued sequence: as token by token.
    f32 sums in two orders: 1e-5."""
    lib, H, dim, S = L(), 2, 32, len(rows)
    g = torch.Generator(device="cuda").manual_seed(vdim)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    M = sum(rows)
    starts = np.cumsum([0] + rows).tolist()
    i32 = lambda t: torch.tensor(t, dtype=torch.int32, device="cuda")
    pos0 = [0, 900]
    keep = dict(pos=i32([pos0[s] + t for s in range(S) for t in range(rows[s])]), row_seq=i32([s for s in range(S) for _ in range(rows[s])]), seq_start=i32(starts),
                seq_rows=i32(list(range(M))), seq_slot=i32([1, 0]), seq_pos0=i32(pos0))
    q, v, f, key = rnd(M, H * dim), rnd(M, H * vdim), rnd(M, H * dim) + 2, rnd(M, H * dim) * dim ** -0.5
    state = rnd(S, H, dim, vdim)
    kw = dict(f=f, f_bias=torch.zeros(H * dim, device="cuda"), k=key, gate=lib.GATE_ROOT_SIGMOID, tau=4.0, q_scale=0.3)
    got = []
    for chunked in (False, True):
        y, st = torch.zeros(M, H * vdim, device="cuda"), state.clone()
        more = {}
        if chunked:
            more = dict(max_chunks=(max(rows) + lib.GATED_CHUNK - 1) // lib.GATED_CHUNK, chunk_slots=M // lib.GATED_CHUNK + S,
                        scratch=torch.full((lib.gated_chunk_floats(M, S, H, dim, vdim),), float("nan"), device="cuda"))
        lib.gated_scan(lib.mamba_batch(**keep), S, q, v, y, st, H, dim, vdim, **kw, **more)
        got.append((y.double(), st.double()))
    for a, b in zip(*got):
        assert (a - b).norm() <= 1e-5 * a.norm()


@pytest.mark.parametrize("rows,splits", [(1, 1), (5, 2), (9, 1), (18, 1), (19, 1), (37, 1), (38, 1)])
def test_decode_attention_by_ring_depth(rows, splits):
    """Heads of 128 with two, three and four stages per warp (CTAs for up to half, one or two of the SMs' worth, more): contexts of 1 to 700 tokens, which end
    inside a half page and leave warps without one.  Against 64 bits: f32 sums on an fp16 cache, 1e-5."""
    k, G, H, hs = K(), 8, 32, 128
    g = torch.Generator(device="cuda").manual_seed(rows)
    pos = [int(p) for p in np.random.default_rng(rows).integers(0, 700, rows)]
    pos[0] = 0 if rows > 1 else 333
    pages = [(p + 32) // 32 for p in pos]
    bt = torch.zeros(rows, max(pages), dtype=torch.int32, device="cuda")
    perm, at = torch.randperm(sum(pages), generator=g, device="cuda", dtype=torch.int32), 0
    for i, n in enumerate(pages):
        bt[i, :n] = perm[at:at + n]
        at += n
    kc, vc = (torch.randn(at, G, 32, hs, generator=g, device="cuda").half() for _ in range(2))
    q, y = torch.randn(rows, H * hs, generator=g, device="cuda"), torch.zeros(rows, H * hs, device="cuda")
    scratch = torch.zeros(k.attention_scratch_bytes(rows, H, hs, splits), dtype=torch.uint8, device="cuda")
    i32 = lambda t: torch.tensor(t, dtype=torch.int32, device="cuda")
    k.attention(q, rows, H, G, hs, kc, vc, i32(pos), i32(list(range(rows))), bt, bt.shape[1], splits, scratch, None, None, rows, y_out=y)
    for i, p in enumerate(pos):
        kk, vv = (c[bt[i, :pages[i]].long()].double().transpose(1, 2).reshape(-1, G, hs)[:p + 1] for c in (kc, vc))
        s = torch.einsum("ghd,tgd->ght", q[i].double().view(G, H // G, hs), kk) * hs ** -0.5
        want = torch.einsum("ght,tgd->ghd", s.softmax(dim=-1), vv).reshape(-1)
        assert (y[i].double() - want).norm() <= 1e-5 * want.norm()


@pytest.mark.parametrize("M,N,K_,epi", [(1, 12290, 1032, "store"), (1, 6147, 2048, "store"), (1, 6146, 2048, "pair"), (1, 12000, 1096, "pair"), (1, 3076, 4096, "pair"), (1, 4099, 3080, "store"),
                                        (1, 2501, 5040, "store"), (1, 1000, 14336, "store"), (1, 769, 16384, "store"), (1, 2100, 6152, "gate"), (2, 6147, 2048, "store"),
                                        (2, 6146, 2048, "pair"), (2, 3073, 4096, "store"), (2, 5001, 2600, "gate")])
def test_rows_through_the_ring(M, N, K_, epi):
    """One and two rows of enough weights for the ring of bulk copies: rows, pairs and slices that end inside a stage or a warp's share, columns that the SMs do not divide, an
    output with a stride, epilogues that read.  Against 64 bits: bf16 operands, f32 sums of up to 16384 terms, 1e-6 of the result's norm."""
    lib = L()
    g = torch.Generator(device="cuda").manual_seed(N)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    w, x = (rnd(N, K_) * K_ ** -0.5).bfloat16(), rnd(M, K_)
    cols = N // 2 if epi == "pair" else N
    buf, aux = torch.full((M, cols + 5), 3.0, device="cuda"), rnd(M, N)
    y = buf[:, :cols]
    lib.dense(w, x, y, M, True, **dict(store={}, pair=dict(epi=lib.DENSE_GLU_GELU), gate=dict(epi=lib.DENSE_SIGMOID_MUL, aux=aux))[epi])
    want = x.bfloat16().double() @ w.double().t()
    if epi == "pair":
        want = torch.nn.functional.gelu(want[:, 0::2], approximate="tanh") * want[:, 1::2]
    if epi == "gate":
        want = aux.double() * want.sigmoid()
    assert (y.double() - want).norm() <= 1e-6 * want.norm() and (buf[:, cols:] == 3).all()


@pytest.mark.parametrize("M,N,K_,epi", [(1, 6146, 2048, "store"), (2, 6146, 2048, "pair"), (1, 1000, 14336, "store"), (1, 3076, 4096, "pair")])
def test_a_ring_that_gives_up_reaches_the_caller(M, N, K_, epi):
    """A limit that is over at once: all but the first two stages' copies are withheld, so the waits run out.  The status word changes once for that launch, whose
    outputs behind those stages are NaN, and not for the next one, which is right."""
    import ctypes
    from dllama_b200.ops import lib as B
    lib, library = L(), B.layers_lib()
    g = torch.Generator(device="cuda").manual_seed(N)
    w, x = (torch.randn(N, K_, generator=g, device="cuda") * K_ ** -0.5).bfloat16(), torch.randn(M, K_, generator=g, device="cuda")
    y = [torch.zeros(M, N // 2 if epi == "pair" else N, device="cuda") for _ in range(3)]
    run = lambda out: lib.dense(w, x, out, M, True, **(dict(epi=lib.DENSE_GLU_GELU) if epi == "pair" else {}))
    run(y[0])
    status = B.WaitStatus(library)
    library.dl_debug_set_wait_limit.argtypes = [ctypes.c_ulonglong]
    library.dl_debug_set_wait_limit(0)
    try:
        run(y[1])
        torch.cuda.synchronize()
    finally:
        library.dl_debug_set_wait_limit(4_000_000_000)
    assert y[1].isnan().float().mean() > 0.5 and (y[1].isnan() | (y[1] == y[0])).all()
    with pytest.raises(B.NativeLibraryError, match="gave up"):
        status.check()
    run(y[2])
    torch.cuda.synchronize()
    status.check()
    assert torch.equal(y[0], y[2]) and not y[0].isnan().any()


@pytest.mark.parametrize("M", [3, 8, 9, 16, 17, 32])
@pytest.mark.parametrize("N,K_", [(40, 8), (2047, 1032), (2370, 136), (4700, 264), (4790, 1096), (9500, 200)])
def test_few_rows_by_columns_per_cta(M, N, K_):
    """3 to 32 rows by every width of a CTA, with rows, columns and inputs left over, warps without a step of inputs and rings longer than a warp's steps.  Against 64 bits: bf16 operands,
    f32 sums, 1e-6 of the result's norm."""
    lib = L()
    g = torch.Generator(device="cuda").manual_seed(N + M)
    w, x = (torch.randn(N, K_, generator=g, device="cuda") * K_ ** -0.5).bfloat16(), torch.randn(M, K_, generator=g, device="cuda")
    buf = torch.full((M, N + 3), 3.0, device="cuda")
    lib.dense(w, x, buf[:, :N], M, True)
    want = x.bfloat16().double() @ w.double().t()
    assert (buf[:, :N].double() - want).norm() <= 1e-6 * want.norm() and (buf[:, N:] == 3).all()


def _given_up(call):
    """call() under a limit that is over at once, for which copies behind the first ringful are withheld; the status word changes once."""
    import ctypes
    from dllama_b200.ops import lib as B
    library = B.cuda_lib()
    status = B.WaitStatus(library)
    library.dl_debug_set_wait_limit.argtypes = [ctypes.c_ulonglong]
    library.dl_debug_set_wait_limit(0)
    try:
        call()
        torch.cuda.synchronize()
    finally:
        library.dl_debug_set_wait_limit(4_000_000_000)
    with pytest.raises(B.NativeLibraryError, match="gave up"):
        status.check()
    return status


# one tile, shares of K, two row tiles per CTA with more items than stages, wide tiles; rows one by one: alone, in shares, in row parts, behind a norm
@pytest.mark.parametrize("kernel,d,n,M,S", [("tc", 300, 4096, 20, 1), ("tc", 300, 8192, 20, 4), ("tc", 38912, 1024, 40, 1), ("tc", 9600, 2048, 200, 1), ("row", 300, 4096, 2, 1),
                                            ("row", 512, 8192, 8, 4), ("row", 128, 2048, 1, 1), ("norm", 512, 8192, 3, 4), ("norm", 9600, 2048, 1, 1)])
def test_a_product_that_gives_up_reaches_the_caller(kernel, d, n, M, S):
    """Waits that run out: the kernel ends, its outputs are NaN (of the tensor cores' most: a stage may be multiplied as it was), the status word changes once for
    that launch and not for the next one, which is right."""
    k = K()
    ncap = (M + 255) // 256 * 256
    w, _ = _q40(d, n, 1)
    w = k.make_q40t(w, d, n)
    _, xh = _activations(n, M, ncap, 2)
    x, norm = torch.randn(M, n, device="cuda"), torch.ones(n, device="cuda")
    xq = k.alloc_xq(n, M, "cuda")
    k.quant_q80(x, M, n, M, xq, None)
    y = [torch.zeros(M, d, device="cuda") for _ in range(3)]

    def run(out):
        epi = k.epi_store([out.data_ptr()], d)
        if kernel == "tc":
            k.gemm_q40_tc(w, d, n, xh, ncap, M, epi, S)
        elif kernel == "row":
            k.gemv_q40(w, d, n, xq, M, epi, 4 if d == 128 else 1, S)
        else:
            k.gemv_q40(w, d, n, None, M, epi, 1, S, norm=k.norm_prolog(x, None, None, 0, 0, None, None, 0, 0, norm, 1e-5))
    run(y[0])
    status = _given_up(lambda: run(y[1]))
    assert y[1].isnan().float().mean() > 0.5 if kernel == "tc" else y[1].isnan().all()
    run(y[2])
    torch.cuda.synchronize()
    status.check()
    assert torch.equal(y[0], y[2]) and not y[0].isnan().any() and y[0].abs().max() > 0


@pytest.mark.parametrize("splits", [1, 3])
def test_decode_attention_that_gives_up_reaches_the_caller(splits):
    """The same for decode attention on an f32 cache, whose pages come through a ring."""
    k, G, H, hs, p = K(), 2, 8, 64, 32 * 40 - 1
    pages = (p + 32) // 32
    bt = torch.arange(pages, dtype=torch.int32, device="cuda").view(1, -1)
    kc, vc = (torch.randn(pages, G, 32, hs, device="cuda") for _ in range(2))
    q = torch.randn(1, H * hs, device="cuda")
    y = [torch.zeros(1, H * hs, device="cuda") for _ in range(3)]
    scratch = torch.zeros(k.attention_scratch_bytes(1, H, hs, splits), dtype=torch.uint8, device="cuda")
    i32 = lambda t: torch.tensor(t, dtype=torch.int32, device="cuda")
    keep = i32([p]), i32([0])
    run = lambda out: k.attention(q, 1, H, G, hs, kc, vc, *keep, bt, pages, splits, scratch, None, None, 1, y_out=out)
    run(y[0])
    status = _given_up(lambda: run(y[1]))
    assert y[1].isnan().all()
    run(y[2])
    torch.cuda.synchronize()
    status.check()
    assert torch.equal(y[0], y[2]) and not y[0].isnan().any()
