"""Performance cases of the framework: what its users have it do, each through its public entry points.

Kinds (a case is a dict of plain values; "kind" says which):

* ``llama_step``  -- a whole forward of the Q40 Llama engine over decoding rows (one per user) whose sequences have a history:
                     what `dllama chat` (one row) and `dllama-api` (one row per user) run for every token.
* ``q40_ffn``     -- the Q40 feed-forward block of a Llama layer on the kernels its row count takes in the engine: RMSNorm + Q80,
                     W1|W3 with SiLU * mul, W2 with the Q80 cast; few rows: the dp4a kernel, prompt chunks: the fused
                     dequantising one, long prompts: the one on pre-expanded weights.
* ``kv_attention``-- paged grouped-query attention of the Llama path: decoding rows of many users, or one prompt chunk.
* ``dense_ffn``   -- the GELU-gated feed-forward block of a layer-list model (bf16 or f32 weights): norm, gate|up, down.
* ``gated_scan``  -- gated linear attention of a layer-list model: a prompt chunk-parallel, or a token of every user.
* ``window_attn`` -- paged attention of a layer-list model (bf16 cache, values of their own, optional window, soft cap and sink).

Widths, feed-forward sizes, heads, depth and vocabulary are those of the repository's benchmark (bench.py, "w2048" and "w4096", 4
layers, 32768 tokens) and its head sizes of 128 and 64.
"""
import math
import os
import tempfile

import numpy as np
import torch

from dllama_b200.ops import kernels as K
from dllama_b200.ops import layers as L
from dllama_b200.ops.lib import DENSE_GLU_GELU, GATE_LOWER, GATE_ROOT_SIGMOID

WIDTHS = {2048: dict(ff=8192, heads=16), 4096: dict(ff=14336, heads=32)}
KV_HEADS = 8
VOCAB = 32768
N_LAYERS = 4
EPS = 1e-5
PAGE = 32
SMS = 148                     # the page shares that the engine would ask for on a B200


def listed():
    return [
        # one user chatting: the smallest call of the engine, one row through every layer and the logits
        {"name": "llama_decode_1", "kind": "llama_step", "width": 4096, "rows": 1, "context": 192},
        # 32 users being served at once, contexts of different lengths
        {"name": "llama_decode_32", "kind": "llama_step", "width": 4096, "rows": 32, "context": 500},
        # a 128-token prompt (the time to the first token) through a layer's feed-forward
        {"name": "q40_ffn_128", "kind": "q40_ffn", "width": 4096, "rows": 128},
        # a long prompt run as one batch
        {"name": "q40_ffn_2048", "kind": "q40_ffn", "width": 4096, "rows": 2048},
        # 32 users deep in a conversation: the history dominates a step
        {"name": "kv_decode_32", "kind": "kv_attention", "mode": "decode", "heads": 32, "head_size": 128, "rows": 32, "context": 3000},
        # a long prompt as one chunk, an odd number of tokens behind 77 others
        {"name": "kv_prompt_4001", "kind": "kv_attention", "mode": "prompt", "heads": 32, "head_size": 128, "rows": 4001, "context": 77},
        # layer-list models: one user, 32 users
        {"name": "dense_ffn_1", "kind": "dense_ffn", "width": 2048, "rows": 1, "dtype": "bf16"},
        {"name": "dense_ffn_32", "kind": "dense_ffn", "width": 4096, "rows": 32, "dtype": "bf16"},
        # a prompt of 2000 tokens / a token of each of 32 users through a linear-attention mixer
        {"name": "gated_prompt_2000", "kind": "gated_scan", "rows": 2000, "seqs": 1, "heads": 16, "dim": 128, "vdim": 128, "own_keys": True},
        {"name": "gated_decode_32", "kind": "gated_scan", "rows": 32, "seqs": 32, "heads": 16, "dim": 128, "vdim": 128, "own_keys": False},
        # the same for an attention mixer: a prompt under a window of 1024, decoding over all earlier positions
        {"name": "window_prompt_2000", "kind": "window_attn", "mode": "prompt", "rows": 2000, "context": 0, "heads": 16, "kv_heads": 4, "window": 1024, "softcap": 0.0, "sink": False},
        {"name": "window_decode_32", "kind": "window_attn", "mode": "decode", "rows": 32, "context": 2000, "heads": 16, "kv_heads": 4, "window": 0, "softcap": 50.0, "sink": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["llama_step", "q40_ffn", "kv_attention", "dense_ffn", "gated_scan", "window_attn"])
    c = {"kind": kind}
    if kind == "llama_step":
        c.update(width=rng.choice([2048, 4096]), rows=_log(rng, 1, 32), context=_log(rng, 16, 500))
    elif kind == "q40_ffn":
        c.update(width=rng.choice([2048, 4096]), rows=_log(rng, 1, 2048))
    elif kind == "kv_attention":
        c.update(mode=rng.choice(["decode", "prompt"]), heads=rng.choice([16, 32]), head_size=rng.choice([64, 128, 128]))
        if c["mode"] == "decode":
            c.update(rows=_log(rng, 1, 32), context=_log(rng, 32, 3000))
        else:
            c.update(rows=_log(rng, 16, 4000), context=rng.choice([0, _log(rng, 1, 77)]))
    elif kind == "dense_ffn":
        c.update(width=rng.choice([2048, 4096]), dtype=rng.choice(["bf16", "bf16", "f32"]))
        c.update(rows=_log(rng, 1, 2048 if c["dtype"] == "bf16" else 32))
    elif kind == "gated_scan":
        d, dv = rng.choice([(128, 128), (64, 64), (128, 256)])
        c.update(heads=rng.choice([8, 16]), dim=d, vdim=dv, own_keys=rng.random() < 0.5)
        if rng.random() < 0.5:
            c.update(rows=_log(rng, 128, 2000), seqs=1)
        else:
            c.update(seqs=_log(rng, 1, 32))
            c.update(rows=c["seqs"])
    else:
        h = rng.choice([16, 32])
        c.update(mode=rng.choice(["decode", "prompt"]), heads=h, kv_heads=rng.choice([4, 8]), window=rng.choice([0, 256, 1024]),
                 softcap=rng.choice([0.0, 50.0]), sink=rng.random() < 0.5)
        if c["mode"] == "decode":
            c.update(rows=_log(rng, 1, 32), context=_log(rng, 32, 2000))
        else:
            c.update(rows=_log(rng, 32, 2000), context=rng.choice([0, _log(rng, 1, 300)]))
    return c


# ---------------------------------------------------------------------------------------------------------------
# inputs (made from the seed alone)
# ---------------------------------------------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda")


def _ints(g, lo, hi, n):
    return torch.randint(lo, hi, (n,), generator=g, device="cuda", dtype=torch.int32)


def _q40(g, d, n, std=0.02):
    """Q40 file bytes [d][n / 32][18] of a normal matrix: fp16 scale, 16 bytes of nibbles (low: elements 0-15, high: 16-31)."""
    nib = (_randn(g, d, n // 32, 32).mul_(3.5).round_() + 8).clamp_(0, 15).to(torch.uint8)
    scale = (std / 3.5 * (0.8 + 0.4 * torch.rand(d, n // 32, 1, generator=g, device="cuda"))).half()
    return torch.cat([scale.view(torch.uint8), nib[:, :, :16] | (nib[:, :, 16:] << 4)], dim=2)


def _q40_f64(raw):
    """The matrix that _q40's bytes stand for, in 64 bits."""
    s = raw[:, :, :2].contiguous().view(torch.float16).double()
    v = torch.cat([raw[:, :, 2:] & 15, raw[:, :, 2:] >> 4], dim=2)
    return ((v.double() - 8) * s).reshape(raw.shape[0], -1)


def _lengths(case, seed):
    """History length of every row: between half and all of the case's context."""
    r = np.random.default_rng(seed)
    return [int(t) for t in r.integers(max(1, case["context"] // 2), case["context"] + 1, case["rows"])]


def _llama_inputs(case, seed):
    g = _gen(seed)
    W, ff, kv = case["width"], WIDTHS[case["width"]]["ff"], KV_HEADS * 128
    w = {"embedding": _randn(g, VOCAB, W), "layers": []}
    for _ in range(N_LAYERS):
        w["layers"].append({"wq": _q40(g, W, W), "wk": _q40(g, kv, W), "wv": _q40(g, kv, W), "wo": _q40(g, W, W), "w1": _q40(g, ff, W),
                            "w2": _q40(g, W, ff), "w3": _q40(g, ff, W), "rms_att": 1 + 0.1 * _randn(g, W), "rms_ffn": 1 + 0.1 * _randn(g, W)})
    w["rms_final"], w["wcls"] = 1 + 0.1 * _randn(g, W), _q40(g, VOCAB, W)
    lens = _lengths(case, seed)
    hist = [[torch.cat([_randn(g, t, KV_HEADS, 128).half().unsqueeze(0) for _ in range(2)]) for t in lens] for _ in range(N_LAYERS)]
    return w, lens, hist, _ints(g, 1, VOCAB, case["rows"])


def _pages_of(table, t):
    return torch.as_tensor(np.asarray(table[:(t + PAGE - 1) // PAGE]), dtype=torch.long, device="cuda")


def _prepare_llama(case, seed):
    from dllama_b200.formats import mfile
    from dllama_b200.models.llama import LlamaEngine
    from dllama_b200.ops import quant
    w, lens, hist, tokens = _llama_inputs(case, seed)
    W = case["width"]
    shape = dict(dim=W, hidden_dim=WIDTHS[W]["ff"], n_layers=N_LAYERS, n_heads=WIDTHS[W]["heads"], n_kv_heads=KV_HEADS, vocab_size=VOCAB,
                 max_seq_len=8192, rope_theta=10000, rope=None)
    fd, path = tempfile.mkstemp(suffix=".m", dir="/dev/shm" if os.path.isdir("/dev/shm") else None)
    with os.fdopen(fd, "wb") as f:
        mfile.write_header(f, mfile.header_params(shape, quant.Q40))
        w["embedding"].cpu().numpy().tofile(f)
        for layer in w["layers"]:
            for t in layer.values():                       # the file's order
                t.contiguous().cpu().numpy().tofile(f)
        w["rms_final"].cpu().numpy().tofile(f)
        w["wcls"].cpu().numpy().tofile(f)
    del w
    eng = LlamaEngine(path, max_rows=max(case["rows"], 16), n_slots=case["rows"], max_seq_len=max(512, case["context"] + 64))
    os.unlink(path)
    slots = [eng.alloc_slot() for _ in lens]
    for i, (s, t) in enumerate(zip(slots, lens)):
        eng.ensure_capacity(s, t + 1)
        pages = _pages_of(eng.pages.table[s], t)
        for l in range(N_LAYERS):
            for cache, x in zip((eng.k_cache[l], eng.v_cache[l]), hist[l][i]):
                pad = torch.zeros(len(pages) * PAGE, KV_HEADS, 128, dtype=torch.float16, device="cuda")
                pad[:t] = x
                cache[pages] = pad.view(len(pages), PAGE, KV_HEADS, 128).transpose(1, 2)
    return {"eng": eng, "tokens": tokens.tolist(), "pos": lens, "slots": slots}


def _ffn_inputs(case, seed):
    g = _gen(seed)
    W, ff = case["width"], WIDTHS[case["width"]]["ff"]
    return _q40(g, ff, W), _q40(g, ff, W), _q40(g, W, ff), 1 + 0.1 * _randn(g, W), _randn(g, case["rows"], W)


def _prepare_q40_ffn(case, seed):
    w1, w3, w2, norm, x = _ffn_inputs(case, seed)
    W, ff, M = case["width"], WIDTHS[case["width"]]["ff"], case["rows"]
    w13 = torch.zeros(K.q40t_bytes(2 * ff, W), dtype=torch.uint8, device="cuda")
    K.q40_repack(w1.reshape(-1), ff, W, w13, 2 * ff, 0, 2)      # rows interleaved: gate_i, up_i
    K.q40_repack(w3.reshape(-1), ff, W, w13, 2 * ff, 1, 2)
    s = {"M": M, "W": W, "ff": ff, "norm": norm, "x": x, "w13": w13, "w2": K.make_q40t(w2.reshape(-1), W, ff), "y": torch.zeros(M, W, device="cuda")}
    if M <= 3:
        s["xq"] = K.alloc_xq(ff, 8, "cuda")
    else:
        s["ncap"] = ncap = 16 if M <= 16 else 32 if M <= 32 else 64 if M <= 64 else (M + 127) // 128 * 128
        s["xh"], s["xh_hid"] = K.alloc_xh(W, ncap, "cuda"), K.alloc_xh(ff, ncap, "cuda")
        if M >= 768:
            s["wh13"], s["wh2"] = K.q40t_to_wh(s["w13"], 2 * ff, W), K.q40t_to_wh(s["w2"], W, ff)
    return s


def _run_q40_ffn(s):
    M, W, ff, x = s["M"], s["W"], s["ff"], s["x"].data_ptr()
    out = K.epi_store([s["y"].data_ptr()], W, 0, True, residual=x, residual_ld=W)
    if M <= 3:
        norm = K.norm_prolog(s["x"], None, None, 0, 0, None, None, 0, 0, s["norm"], EPS)
        R, S, T = K.choose_splits(2 * ff, W, 2, SMS, M)
        K.gemv_q40(s["w13"], 2 * ff, W, None, M, K.epi_silu_mul(s["xq"], None, M), R, S, norm=norm, pdl=True, tiles_per_cta=T)
        R, S, T = K.choose_splits(W, ff, 0, SMS, M)
        K.gemv_q40(s["w2"], W, ff, s["xq"], M, out, R, S, pdl=True, tiles_per_cta=T)
        return s["y"]
    ncap = s["ncap"]
    K.reduce_norm_quant(s["x"], None, None, 0, 0, None, None, 0, 0, s["norm"], EPS, W, M, ncap, None, s["xh"], pdl=True)
    silu = K.epi_silu_mul(None, s["xh_hid"], ncap)
    if M >= 768:
        K.gemm_wh_tc(s["wh13"], 2 * ff, W, s["xh"], ncap, M, silu, pdl=True)
        K.gemm_wh_tc(s["wh2"], W, ff, s["xh_hid"], ncap, M, out, pdl=True)
    else:
        K.gemm_q40_tc(s["w13"], 2 * ff, W, s["xh"], ncap, M, silu, K.choose_tc_split(2 * ff, W, M, SMS), pdl=True)
        K.gemm_q40_tc(s["w2"], W, ff, s["xh_hid"], ncap, M, out, K.choose_tc_split(W, ff, M, SMS), pdl=True)
    return s["y"]


def _page_table(g, lens):
    """Block table [rows][pages] of sequences of these lengths, pages in a random order, and the number of pages."""
    need = [(t + PAGE - 1) // PAGE for t in lens]
    perm = torch.randperm(sum(need), generator=g, device="cuda", dtype=torch.int32)
    bt = torch.zeros(len(lens), max(need), dtype=torch.int32, device="cuda")
    at = 0
    for i, n in enumerate(need):
        bt[i, :n] = perm[at:at + n]
        at += n
    return bt, at


def _attn_rows(case, seed):
    """Position and sequence of every row, tokens of every sequence."""
    if case["mode"] == "decode":
        pos = _lengths(case, seed)
        return pos, list(range(len(pos))), [p + 1 for p in pos]
    p0, M = case["context"], case["rows"]
    return list(range(p0, p0 + M)), [0] * M, [p0 + M]


def _kv_inputs(case, seed):
    g = _gen(seed)
    pos, slot, lens = _attn_rows(case, seed)
    bt, n = _page_table(g, lens)
    hs = case["head_size"]
    k, v = (_randn(g, n, KV_HEADS, PAGE, hs).half() for _ in range(2))
    return pos, slot, lens, bt, k, v, _randn(g, case["rows"], case["heads"] * hs)


def _i32(v):
    return torch.tensor(v, dtype=torch.int32, device="cuda")


def _prepare_kv(case, seed):
    pos, slot, lens, bt, k, v, q = _kv_inputs(case, seed)
    M, H, hs = case["rows"], case["heads"], case["head_size"]
    s = {"case": dict(case), "pos": _i32(pos), "slot": _i32(slot), "bt": bt, "k": k, "v": v, "q": q, "y": torch.zeros(M, H * hs, device="cuda")}
    if case["mode"] == "decode":
        s["splits"] = int(min(max(1, SMS // (M * KV_HEADS)), max(1, bt.shape[1] // 8), 32))
        s["scratch"] = torch.zeros(K.attention_scratch_bytes(M, H, hs, s["splits"]), dtype=torch.uint8, device="cuda")
    else:
        s["meta"] = _i32([1, 0, M])
    return s


def _run_kv(s):
    c = s["case"]
    a = (s["q"], c["rows"], c["heads"], KV_HEADS, c["head_size"], s["k"], s["v"], s["pos"], s["slot"], s["bt"], s["bt"].shape[1])
    if c["mode"] == "decode":
        K.attention(*a, s["splits"], s["scratch"], None, None, c["rows"], y_out=s["y"])
    else:
        K.attention_prefill(*a, s["meta"], None, None, c["rows"], y_out=s["y"], tc=c["head_size"] == 128 and c["rows"] >= 128)
    return s["y"]


def _dense_inputs(case, seed):
    g = _gen(seed)
    W, ff = case["width"], WIDTHS[case["width"]]["ff"]
    t = torch.bfloat16 if case["dtype"] == "bf16" else torch.float32
    gate_up = (_randn(g, 2 * ff, W) * W ** -0.5).to(t)          # rows interleaved: gate_0, up_0, gate_1, ...
    return gate_up, (_randn(g, W, ff) * ff ** -0.5).to(t), 1 + 0.1 * _randn(g, W), _randn(g, case["rows"], W)


def _prepare_dense(case, seed):
    gate_up, down, norm, x = _dense_inputs(case, seed)
    W, ff, M = case["width"], WIDTHS[case["width"]]["ff"], case["rows"]
    s = {"M": M, "W": W, "ff": ff, "norm": norm, "x": x, "round": case["dtype"] == "bf16", "y": torch.zeros(M, W, device="cuda")}
    s["up"] = torch.zeros(M, ff, device="cuda")
    if case["dtype"] == "bf16" and M >= 32:
        s["ncap"] = ncap = (M + 7) // 8 * 8
        s["wu"], s["wd"] = L.make_wh(gate_up), L.make_wh(down)
        s["xh"], s["xh_up"] = (torch.zeros(L.xh_bytes(n, ncap), dtype=torch.uint8, device="cuda") for n in (W, ff))
    else:
        s["wu"], s["wd"], s["h"] = gate_up, down, torch.zeros(M, W, device="cuda")
    return s


def _run_dense(s):
    M, W, ff, y = s["M"], s["W"], s["ff"], s["y"]
    if "ncap" in s:
        L.residual_step(M, W, EPS, x_in=s["x"], outs=[(s["norm"], (s["xh"], s["ncap"]))])
        L.dense_tc(s["wu"], 2 * ff, W, s["xh"], s["ncap"], s["up"], M, epi=DENSE_GLU_GELU, image=(s["xh_up"], s["ncap"]))
        L.dense_tc(s["wd"], W, ff, s["xh_up"], s["ncap"], y, M)
    else:
        L.residual_step(M, W, EPS, x_in=s["x"], outs=[(s["norm"], s["h"])])
        L.dense(s["wu"], s["h"], s["up"], M, s["round"], epi=DENSE_GLU_GELU)
        L.dense(s["wd"], s["up"], y, M, s["round"])
    return y


def _gated_inputs(case, seed):
    g = _gen(seed)
    M, H, d, dv = case["rows"], case["heads"], case["dim"], case["vdim"]
    t = {"q": _randn(g, M, H * d), "v": _randn(g, M, H * dv), "f": _randn(g, M, H * d), "f_bias": 1 + 0.5 * _randn(g, H * d),
         "state": 0.5 * _randn(g, case["seqs"], H, d, dv)}
    if case["own_keys"]:
        t["k"] = _randn(g, M, H * d) * d ** -0.5
    else:
        t["lower"] = torch.rand(H * d, generator=g, device="cuda") * 0.9
    return t


def _prepare_gated(case, seed):
    t = _gated_inputs(case, seed)
    M, S, H, d, dv = case["rows"], case["seqs"], case["heads"], case["dim"], case["vdim"]
    per = M // S
    fresh = S == 1 and M > 1                                     # a prompt starts its sequence, decoding goes on with one
    p0 = 0 if fresh else 1000
    i32 = {"pos": _i32([p0 + i % per for i in range(M)]), "row_seq": _i32([i // per for i in range(M)]), "seq_start": _i32([i * per for i in range(S + 1)]),
           "seq_rows": _i32(list(range(M))), "seq_slot": _i32(list(range(S))), "seq_pos0": _i32([p0] * S)}
    kw = dict(f=t["f"], f_bias=t["f_bias"])
    if case["own_keys"]:
        kw.update(k=t["k"], gate=GATE_ROOT_SIGMOID, tau=16.0, q_scale=d ** -0.5)
    else:
        kw.update(lower=t["lower"], gate=GATE_LOWER, q_silu=True)
    if per >= 128:
        kw.update(max_chunks=(per + L.GATED_CHUNK - 1) // L.GATED_CHUNK, chunk_slots=M // L.GATED_CHUNK + S,
                  scratch=torch.zeros(L.gated_chunk_floats(M, S, H, d, dv), device="cuda"))
    return {"batch": L.mamba_batch(**i32), "keep": i32, "S": S, "t": t, "kw": kw, "dims": (H, d, dv), "y": torch.zeros(M, H * dv, device="cuda")}


def _run_gated(s):
    t = s["t"]
    L.gated_scan(s["batch"], s["S"], t["q"], t["v"], s["y"], t["state"], *s["dims"], **s["kw"])
    return s["y"], t["state"]


def _window_inputs(case, seed):
    g = _gen(seed)
    pos, slot, lens = _attn_rows(case, seed)
    bt, n = _page_table(g, lens)
    cache = _randn(g, n, case["kv_heads"], PAGE, 256).bfloat16()          # a line: key of 128, value of 128
    return pos, slot, lens, bt, cache, _randn(g, case["rows"], case["heads"] * 128), _randn(g, case["heads"])


def _prepare_window(case, seed):
    pos, slot, lens, bt, cache, q, sink = _window_inputs(case, seed)
    M, H, G = case["rows"], case["heads"], case["kv_heads"]
    rq = L.window_tc_rows(H, G)
    tiles = [[m] for m in range(M)] if case["mode"] == "decode" else [list(range(i, min(i + rq, M))) for i in range(0, M, rq)]
    rows = np.full((len(tiles), rq), -1, dtype=np.int32)
    for i, t in enumerate(tiles):
        rows[i, :len(t)] = t
    pages = case["window"] // PAGE + 1 if case["window"] else bt.shape[1]
    splits = max(1, min(pages, 32, 8 * SMS // (len(tiles) * G))) if len(tiles) * G <= 2 * SMS else 1
    partial = torch.zeros(L.window_tc_partial_floats(len(tiles), G, splits, 128), device="cuda") if splits > 1 else None
    return {"case": dict(case), "pos": _i32(pos), "slot": _i32(slot), "bt": bt, "cache": cache, "q": q, "sink": sink if case["sink"] else None,
            "tiles": torch.from_numpy(rows).cuda(), "n": len(tiles), "rq": rq, "splits": splits, "partial": partial, "y": torch.zeros(M, H * 128, device="cuda")}


def _run_window(s):
    c = s["case"]
    L.window_attention_tc(s["q"], s["y"], c["heads"], c["kv_heads"], 128, 0, 128 ** -0.5, c["softcap"], c["window"], s["pos"], s["slot"], s["bt"],
                          s["cache"], s["tiles"], s["n"], s["rq"], s["splits"], s["partial"], vdim=128, sink=s["sink"])
    return s["y"]


_PREPARE = {"llama_step": _prepare_llama, "q40_ffn": _prepare_q40_ffn, "kv_attention": _prepare_kv, "dense_ffn": _prepare_dense,
            "gated_scan": _prepare_gated, "window_attn": _prepare_window}
_RUN = {"q40_ffn": _run_q40_ffn, "kv_attention": _run_kv, "dense_ffn": _run_dense, "gated_scan": _run_gated, "window_attn": _run_window,
        "llama_step": lambda s: s["eng"].forward(s["tokens"], s["pos"], s["slots"])}


def prepare(case, seed):
    return {"kind": case["kind"], "s": _PREPARE[case["kind"]](case, seed)}


def run(state):
    return _RUN[state["kind"]](state["s"])


# ---------------------------------------------------------------------------------------------------------------
# the work that a case cannot do without, its tolerance, and its results in 64 bits
# ---------------------------------------------------------------------------------------------------------------
def _seen(pos, window):
    return sum(min(p + 1, window) if window else p + 1 for p in pos)


def work(case):
    kind, M = case["kind"], case["rows"]
    if kind == "llama_step":
        W, ff = case["width"], WIDTHS[case["width"]]["ff"]
        n = N_LAYERS * (2 * W * W + 2 * W * KV_HEADS * 128 + 3 * W * ff) + VOCAB * W
        hist = M * case["context"] * 3 // 4 * N_LAYERS
        return {"bytes": n * 9 // 16 + hist * KV_HEADS * 128 * 4 + M * (W + VOCAB) * 4, "flops": 2 * M * n + 4 * hist * W}
    if kind in ("q40_ffn", "dense_ffn"):
        W, ff = case["width"], WIDTHS[case["width"]]["ff"]
        n = 3 * W * ff
        per = (2 if M >= 768 else 9 / 16) if kind == "q40_ffn" else 2 if case["dtype"] == "bf16" else 4
        return {"bytes": int(n * per) + 8 * M * W, "flops": 2 * M * n}
    if kind == "gated_scan":
        H, d, dv, S = case["heads"], case["dim"], case["vdim"], case["seqs"]
        rows = M * H * (d * (3 if case["own_keys"] else 2) + 2 * dv) * 4
        return {"bytes": rows + S * H * d * dv * (4 if S == 1 and M > 1 else 8), "flops": 6 * M * H * d * dv}
    pos, _, lens = _attn_rows(case, 0)
    if kind == "kv_attention":
        H, hs, G, window, size = case["heads"], case["head_size"], KV_HEADS, 0, 2
    else:
        H, hs, G, window, size = case["heads"], 128, case["kv_heads"], case["window"], 2
    kept = sum(min(t, window) if window and case["mode"] == "decode" else t for t in lens)
    return {"bytes": kept * G * 2 * hs * size + 8 * M * H * hs, "flops": 4 * _seen(pos, window) * H * hs}


def tolerance(case):
    """About four times the distance to exact() that was measured on a B200."""
    kind = case["kind"]
    if kind == "llama_step":                 # a Q80 cast turns a difference e into about sqrt(e * step): after a few of them any two orders
        return {"rel": 1e-1}                 # of summation are one step of the 8-bit values (2 %) apart; measured 0.019 to 0.026
    if kind == "q40_ffn":                    # two casts (and fp16 operands from four rows); measured 0.0058
        return {"rel": 2.4e-2}
    if kind == "kv_attention":               # decoding: f32 on an fp16 cache (4e-7); prompts: fp16 probabilities (3e-4)
        return {"rel": 1e-5 if case["mode"] == "decode" else 1.2e-3}
    if kind == "dense_ffn":                  # bf16 operands, rounded between the products (2e-4); f32 (5e-7)
        return {"rel": 1e-3 if case["dtype"] == "bf16" else 1e-5}
    if kind == "gated_scan":                 # f32 throughout (4e-7)
        return {"rel": 1e-5}
    return {"rel": 8e-3}                     # bf16 queries and probabilities (2e-3)


def _q80(x):
    """Values after the cast to Q80 (blocks of 32: int8 and an fp16 scale) and back."""
    b = x.reshape(-1, 32)
    d = b.abs().amax(dim=1, keepdim=True) / 127
    q = torch.where(d > 0, b / d, torch.zeros_like(b)).round()
    return (q * d.half().double()).reshape(x.shape)


def _rms(x, w):
    return w.double() * x / (x.square().mean(dim=-1, keepdim=True) + EPS).sqrt()


def _rotate(x, pos):
    """Rotary on adjacent pairs of heads of 128; x [rows][heads * 128]."""
    f = 1.0 / 10000.0 ** (torch.arange(0, 128, 2, device="cuda", dtype=torch.float64) / 128)
    a = torch.tensor(pos, device="cuda", dtype=torch.float64)[:, None, None] * f
    p = x.reshape(x.shape[0], -1, 64, 2)
    return torch.stack([p[..., 0] * a.cos() - p[..., 1] * a.sin(), p[..., 0] * a.sin() + p[..., 1] * a.cos()], dim=-1).reshape(x.shape)


def _exact_llama(case, seed):
    w, lens, hist, tokens = _llama_inputs(case, seed)
    W, H = case["width"], WIDTHS[case["width"]]["heads"]
    x = w["embedding"][tokens.long()].double()
    for l, lw in enumerate(w["layers"]):
        h = _q80(_rms(x, lw["rms_att"]))
        q, k = (_rotate(h @ _q40_f64(lw[n]).t(), lens) for n in ("wq", "wk"))
        v = h @ _q40_f64(lw["wv"]).t()
        o = torch.empty_like(q)
        for i in range(case["rows"]):
            kk, vv = (torch.cat([hist[l][i][j].double(), t[i].half().double().view(1, KV_HEADS, 128)]) for j, t in enumerate((k, v)))
            s = torch.einsum("ghd,tgd->ght", q[i].view(KV_HEADS, H // KV_HEADS, 128), kk) * 128 ** -0.5
            o[i] = torch.einsum("ght,tgd->ghd", s.softmax(dim=-1), vv).reshape(-1)
        x = x + _q80(_q80(o) @ _q40_f64(lw["wo"]).t())
        h = _q80(_rms(x, lw["rms_ffn"]))
        a = torch.nn.functional.silu(h @ _q40_f64(lw["w1"]).t()) * (h @ _q40_f64(lw["w3"]).t())
        x = x + _q80(_q80(a) @ _q40_f64(lw["w2"]).t())
    return _q80(_rms(x, w["rms_final"])) @ _q40_f64(w["wcls"]).t()


def _exact_q40_ffn(case, seed):
    w1, w3, w2, norm, x = _ffn_inputs(case, seed)
    x = x.double()
    h = _q80(_rms(x, norm))
    a = torch.nn.functional.silu(h @ _q40_f64(w1).t()) * (h @ _q40_f64(w3).t())
    return x + _q80(_q80(a) @ _q40_f64(w2).t())


def _exact_attention(q, pos, lens, bt, keys, values, H, G, hs, mode, window=0, softcap=0.0, sink=None):
    """keys / values: functions of the page list giving [tokens][G][hs] in 64 bits."""
    q, pos_t = q.double().view(-1, G, H // G, hs), torch.tensor(pos, device="cuda")
    out = torch.empty_like(q)
    for i, t in enumerate(lens):
        pages = bt[i, :(t + PAGE - 1) // PAGE].long()
        k, v = keys(pages)[:t], values(pages)[:t]
        rows = slice(i, i + 1) if mode == "decode" else slice(0, len(pos))
        at = torch.arange(t, device="cuda")
        hidden = at[None] > pos_t[rows, None]
        if window:
            hidden |= at[None] <= pos_t[rows, None] - window
        for h in range(H):
            g, j = divmod(h, H // G)
            s = q[rows, g, j] @ k[:, g].t() * hs ** -0.5
            if softcap:
                s = softcap * (s / softcap).tanh()
            s = s.masked_fill(hidden, -math.inf)
            if sink is not None:
                s = torch.cat([s, sink[h].double().expand(s.shape[0], 1)], dim=1)
            out[rows, g, j] = s.softmax(dim=1)[:, :t] @ v[:, g]
    return out.reshape(len(pos), H * hs)


def _exact_kv(case, seed):
    pos, slot, lens, bt, k, v, q = _kv_inputs(case, seed)
    flat = [lambda p, c=c: c[p].double().transpose(1, 2).reshape(-1, KV_HEADS, case["head_size"]) for c in (k, v)]
    return _exact_attention(q, pos, lens, bt, *flat, case["heads"], KV_HEADS, case["head_size"], case["mode"])


def _exact_window(case, seed):
    pos, slot, lens, bt, cache, q, sink = _window_inputs(case, seed)
    flat = [lambda p, o=o: cache[p][..., o:o + 128].double().transpose(1, 2).reshape(-1, case["kv_heads"], 128) for o in (0, 128)]
    return _exact_attention(q, pos, lens, bt, *flat, case["heads"], case["kv_heads"], 128, case["mode"], case["window"], case["softcap"],
                            sink if case["sink"] else None)


def _exact_dense(case, seed):
    gate_up, down, norm, x = _dense_inputs(case, seed)
    rnd = (lambda t: t.bfloat16().double()) if case["dtype"] == "bf16" else (lambda t: t)
    p = rnd(_rms(x.double(), norm)) @ gate_up.double().t()
    a = torch.nn.functional.gelu(p[:, 0::2], approximate="tanh") * p[:, 1::2]
    return rnd(a) @ down.double().t()


def _exact_gated(case, seed):
    t = {n: v.double() for n, v in _gated_inputs(case, seed).items()}
    M, S, H, d, dv = case["rows"], case["seqs"], case["heads"], case["dim"], case["vdim"]
    per = M // S
    if S == 1 and M > 1:
        t["state"].zero_()
    z = (t["f"] + t["f_bias"]).view(S, per, H, d)
    if case["own_keys"]:
        f, k, q = z.sigmoid() ** (1 / 16), t["k"].view(S, per, H, d), t["q"].view(S, per, H, d) * d ** -0.5
    else:
        lo = t["lower"].view(H, d)
        f, q = lo + (1 - lo) * z.sigmoid(), torch.nn.functional.silu(t["q"]).view(S, per, H, d)
        k = (1 - lo) * (-z).sigmoid()
    v, state, y = t["v"].view(S, per, H, dv), t["state"], torch.empty(S, per, H, dv, device="cuda", dtype=torch.float64)
    for i in range(per):
        state = f[:, i, :, :, None] * state + k[:, i, :, :, None] * v[:, i, :, None, :]
        y[:, i] = torch.einsum("shd,shdv->shv", q[:, i], state)
    return y.reshape(M, H * dv), state


_EXACT = {"llama_step": _exact_llama, "q40_ffn": _exact_q40_ffn, "kv_attention": _exact_kv, "dense_ffn": _exact_dense,
          "gated_scan": _exact_gated, "window_attn": _exact_window}


def exact(case, seed):
    return _EXACT[case["kind"]](case, seed)
