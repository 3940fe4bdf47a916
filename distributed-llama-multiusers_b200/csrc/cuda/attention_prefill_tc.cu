// Causal attention for long prompt chunks on the 5th-gen tensor cores (head size 128): the same job as
// attention_prefill.cu (segments of consecutive positions of one sequence, listed in `meta`), with both products
// as tcgen05.mma and the score / probability / output tiles in TENSOR MEMORY instead of registers.
//
// A CTA works on TWO query tiles of 128 rows that meet the same keys and values (two heads of a key/value head, or two row tiles of one head)
// and walks the KV history 128 tokens (four pages) at a time; one tile's softmax runs beside the other's MMAs:
//   S = Q K^T     SS-mode MMA, M = 128 rows, N = 128 tokens, K = 128: Q staged once (fp16, K-major, 128-byte swizzle);
//                 K pages arrive by TMA tensor copies (cp.async.bulk.tensor.2d over this GPU's KV cache, box 64 x 32,
//                 hardware 128-byte swizzle); S (f32) lands in ONE buffer of TMEM that the tiles take in turn, free again as soon as
//                 the softmax threads have it in registers, so that the next scores wait for them there
//   softmax       a thread per query row (= TMEM lane), 128 scores in registers; exp2 -> fp16 probabilities written back to TMEM
//                 (a quarter of the exp2 on the FMA pipe); running maximum with LAZY rescaling: the reference maximum only
//                 moves when a row's maximum grew by more than 2^8, so in the steady state the output accumulator is
//                 never touched by the softmax threads
//   O += P V      TS-mode MMA: A = P straight from TMEM, B = V pages in shared memory as an MN-major operand (V is
//                 [token][head dim] in the cache, i.e. N-contiguous: no transpose anywhere), accumulating in TMEM
// CTAs are persistent: each walks its items (pt_item), long ones first and rounds back and forth, and loads the next item's queries ahead of this one's
// outputs.  What bounds it: the MMAs.  With one tile per CTA scores, softmax and P V of a step followed each other (1950 clk a step for 1024 of MMAs) and
// every CTA paid 13 us for its start and end: 4001 rows of 32 heads 229 us on inputs in turn, 170 here (215 and 147 on the same inputs again and again: two
// steps in 1.75 us; the rest is starts, ends and diagonals).
//
// Warp roles (384 threads): warps 0-3 and 4-7 softmax of tile 0 and 1, warp 8 issues all MMAs (one issuer, or the tiles run in step; in convergent code, see
// pt_mma_ss), warp 9 K producer and warp 10 V producer (one lane each issues 8 tensor copies of 4 KB per step).
//
// The second instance (LINES) serves layer-list models: bf16 cache lines [key 128 | value 128], tiles of up to rq consecutive positions
// of one sequence whose query heads of one key/value head stack on the MMA's rows (row = position * rep + head), so runs of two or four
// neighbouring list tiles of 64 stacked rows fill one or two of its tiles; window or chunk masks (only the steps that a run sees are walked, in
// shares where SMs are idle), soft cap, distance bias, sink, gate; f32 output.  Probabilities are two bf16 numbers each, the second the first one's
// remainder, and P V two MMAs: rounded to
// one (2^-9) they are the larger share of the error, and how large depends on how often a row's maximum, whose probability is exact, moves
// (2000 tokens under a window of 1024, against 64 bits: 1.93e-3 with one number, 1.47e-3 with two).  They take 128 columns, so the tiles take one such
// buffer in turn, too.  2000 rows of 16 heads on 4 under a window of 1024: one run of 128 rows per CTA, in two waves, 55.5 us; 41 here; 512 rows in
// page shares on mma.sync 62 us, 17 to 19 here.  The tiles' values are shared, but each multiplies only the groups of 16 tokens that it sees (the last of them may
// hold some of the other's, where a portion starts inside a group).
//
// Reference semantics: multiheadAtt_F32 (src/nn/nn-cpu-ops.cpp:749-784), softmax in f32, output cast as OP_CAST
// (src/llm.cpp:296-301).  KV cache: fp16 pages [page][kv_head][32][128].
#include <atomic>
#include "epilogue.cuh"
#include "f32_pairs.cuh"
#include "smem_limit.cuh"
#include "tensor_map.cuh"
#include "waits.cuh"
#include "window_tiles.cuh"

#define PT_HS 128
#define PT_ROWS 128
#define PT_KV 128                      // tokens per step
#define PT_THREADS 384
#define PT_MAX_SEG 8
#define PT_TILE_BYTES 32768            // 128 x 128 fp16
#define PT_STAGES 2                    // K tiles and V tiles in flight
#define PT_OUT_LD 20
#define PT_SHARE_STEPS 4

struct PtArgs {
    const float* q;            // [M][n_heads*128]
    const __half* k_cache;     // [pages][n_kv][32][128]
    const __half* v_cache;
    const int* pos;
    const int* slot;
    const int* block_table;
    const int* meta;           // meta[0] = n_seg, then [begin, end) pairs
    int M, n_heads, n_kv_heads, max_pages;
    uint8_t* xq_out;
    uint8_t* xh_out;
    int out_mcap;
    float* y_out;
    unsigned long long* tr;
    WaitLimit limit;
};

struct PtLineArgs {
    DlWindowAttnArgs w;
    const int* tile_rows;      // [n_tiles][rq], -1 where a tile has fewer rows
    int n_tiles, rq, rep;
    int group;                 // list tiles of a CTA: 2 or 4
    int n_splits;
    int least;                 // runs of no more stacked rows belong to the other kernel (0: there is none)
    float* partial;            // [n_tiles][kv_heads][n_splits][64][130] where n_splits > 1: sums, reference maximum, sum of weights
    WaitLimit limit;
};
template <bool LINES> struct PtKernelArgs { typedef PtArgs T; };
template <> struct PtKernelArgs<true> { typedef PtLineArgs T; };

DL_DEVINL void tmem_ld_32x32b_x32(uint32_t taddr, uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, "
        "%20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
          "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]),
          "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]),
          "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr)
        : "memory");
}
DL_DEVINL void tmem_st_32x32b_x32(uint32_t taddr, const uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, "
        "%20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]),
        "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]),
        "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]),
        "r"(v[31])
        : "memory");
}
// instruction descriptor, kind::f16: A fp16 / bf16 K-major (or TMEM), B alike with selectable major-ness, D f32
DL_DEVINL uint32_t pt_idesc(int M, int N, int b_mn_major, bool bf16) {
    uint32_t d = 0;
    d |= 1u << 4;                                  // D = f32
    if (bf16) d |= (1u << 7) | (1u << 10);         // A and B = bf16
    d |= (uint32_t)(b_mn_major & 1) << 16;         // b_major: 0 = K, 1 = MN
    d |= (uint32_t)(N >> 3) << 17;
    d |= (uint32_t)(M >> 4) << 24;
    return d;
}
DL_DEVINL float pt_ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
template <bool LINES> DL_DEVINL uint32_t pt_pack2(float lo, float hi) {
    if (LINES) {
        __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
        return *reinterpret_cast<uint32_t*>(&h);
    }
    __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&h);
}

// exp2 on the FMA pipe (Cody-Waite split + degree-3 polynomial, relative error 8e-5 -- the result is rounded to fp16,
// 5e-4, right after; LINES, whose other kernels form it in full: degree 5, 2e-7): the softmax is bound by the 16 MUFU results
// per clock and SM (128 x 128 exp2 per step = 1024 clk, as long as the MMAs of the step), so every fourth element takes this
// path instead
template <bool LINES> DL_DEVINL pair_f pt_ex2_poly(pair_f x) {
    float lo, hi;                                  // LINES: a NaN stays one, as in the mma.sync kernel
    pair_get(x, lo, hi);
    if (LINES) {
        asm("max.NaN.f32 %0, %0, %1;" : "+f"(lo) : "f"(-126.0f));
        asm("max.NaN.f32 %0, %0, %1;" : "+f"(hi) : "f"(-126.0f));
    } else {
        lo = fmaxf(lo, -126.0f);
        hi = fmaxf(hi, -126.0f);
    }
    auto both = [](float c) { return pair_of(c, c); };
    const pair_f xc = pair_of(lo, hi), t = add2(xc, both(12582912.0f));                 // 1.5 * 2^23: round(x) lands in the low mantissa bits
    const pair_f f = fma2(add2(t, both(-12582912.0f)), both(-1.0f), xc);                // [-0.5, 0.5]
    float tl, th, pl, ph;
    pair_get(t, tl, th);
    if (LINES) {
        const pair_f p = fma2(fma2(fma2(fma2(fma2(both(1.32764725e-3f), f, both(9.67554096e-3f)), f, both(0.0555071309f)), f, both(0.240221202f)), f, both(0.693146944f)), f, both(1.00000012f));
        return mul2(p, pair_of(__int_as_float((__float_as_int(tl) << 23) + 0x3f800000), __int_as_float((__float_as_int(th) << 23) + 0x3f800000)));
    }
    pair_get(fma2(fma2(fma2(both(0.0550886838f), f, both(0.242604051f)), f, both(0.693276242f)), f, both(0.99992894f)), pl, ph);
    return pair_of(__int_as_float(__float_as_int(pl) + (__float_as_int(tl) << 23)), __int_as_float(__float_as_int(ph) + (__float_as_int(th) << 23)));
}

// 32 scores (masked ones are -inf) -> exp2(s * sc - ref) as 16 packed fp16 pairs; their sum is added to `sum`.  LINES: as bf16 and, in `lo`, the
// bf16 remainder of each, 17 bits together
template <bool LINES> DL_DEVINL void pt_probs(const uint32_t (&v)[32], float sc, float ref, uint32_t (&pk)[16], uint32_t (&lo)[LINES ? 16 : 1], pair_f& sum) {
    const pair_f sc2 = pair_of(sc, sc), ref2 = pair_of(-ref, -ref);
#pragma unroll
    for (int e = 0; e < 32; e += 2) {
        pair_f p = fma2(pair_of(__uint_as_float(v[e]), __uint_as_float(v[e + 1])), sc2, ref2);
        float pa, pb;
        if ((e & 6) == 6) {
            p = pt_ex2_poly<LINES>(p);
            pair_get(p, pa, pb);
        } else {
            pair_get(p, pa, pb);
            pa = pt_ex2(pa);
            pb = pt_ex2(pb);
            p = pair_of(pa, pb);
        }
        sum = add2(sum, p);
        pk[e >> 1] = pt_pack2<LINES>(pa, pb);
        if constexpr (LINES) lo[e >> 1] = pt_pack2<LINES>(pa - __uint_as_float(pk[e >> 1] << 16), pb - __uint_as_float(pk[e >> 1] & 0xffff0000u));
    }
}

// One thread's 32 consecutive outputs of row m (a Q80 block) into the slabs of the next matmul: the block's maximum is in the thread's own
// registers.  (A warp per block, lane = element, took a five-step shuffle reduction for each of a warp's 64 blocks, one behind the other:
// 25 k clk of a CTA that multiplies for 31 k; 4096 rows of 32 heads took 331 us, 210 now; into f32
// rows, which take the same path without the cast, 4001 rows 266 -> 229.)
DL_DEVINL void pt_q80_block(const float (&v)[32], int m, int kblock, int mcap, uint8_t* xq, uint8_t* xh) {
    float amax = 0.f;
#pragma unroll
    for (int e = 0; e < 32; e++) amax = fmaxf(amax, fabsf(v[e]));
    const float d = amax / 127.0f;
    const float id = (d != 0.0f) ? (1.0f / d) : 0.0f;
    const float df = __half2float(__float2half_rn(d));
    const int kt = kblock >> 2, kb = kblock & 3;
    int q[32];
#pragma unroll
    for (int e = 0; e < 32; e++) q[e] = __float2int_rn(v[e] * id);
    if (xq != nullptr) {
        uint8_t* row = xq + ((size_t)kt * mcap + m) * XQ_ROW_BYTES;
        int sumq = 0;
#pragma unroll
        for (int e = 0; e < 32; e += 4) {
            sumq += q[e] + q[e + 1] + q[e + 2] + q[e + 3];
            *reinterpret_cast<uint32_t*>(row + kb * 32 + e) =
                (uint32_t)(q[e] & 0xff) | ((uint32_t)(q[e + 1] & 0xff) << 8) | ((uint32_t)(q[e + 2] & 0xff) << 16) | ((uint32_t)(q[e + 3] & 0xff) << 24);
        }
        reinterpret_cast<float*>(row + 128)[kb] = df;
        reinterpret_cast<int*>(row + 144)[kb] = 8 * sumq;
    }
    if (xh != nullptr) {
        const float dfh = fminf(df, 515.0f);       // fp16 operand: saturate (|x| > 65405) instead of producing inf
        uint8_t* base = xh + ((size_t)kt * (size_t)(mcap >> 3) + (size_t)(m >> 3)) * XH_ROWGROUP_BYTES + (size_t)(kb * 4) * 128 + (size_t)(m & 7) * 16;
#pragma unroll
        for (int w = 0; w < 4; w++) {              // chunk w: elements 4w, 4w+2, 4w+1, 4w+3, then the same + 16 (see xh_slot)
            uint4 u;
            u.x = pt_pack2<false>((float)q[4 * w] * dfh, (float)q[4 * w + 2] * dfh);
            u.y = pt_pack2<false>((float)q[4 * w + 1] * dfh, (float)q[4 * w + 3] * dfh);
            u.z = pt_pack2<false>((float)q[4 * w + 16] * dfh, (float)q[4 * w + 18] * dfh);
            u.w = pt_pack2<false>((float)q[4 * w + 17] * dfh, (float)q[4 * w + 19] * dfh);
            *reinterpret_cast<uint4*>(base + w * 128) = u;
        }
    }
}

// The eight MMAs of a group (K = 128) by one thread of the converged warp, elected by a predicate: with one MMA at a time inside an `if (elect)`
// 4001 rows of 32 heads took 150 us, 138 so (on the same inputs again and again, with the queries loaded by warps of their own).
// D += A B^T, both operands 128-byte-swizzled half tiles 16 KB apart (32 B of a row per MMA)
DL_DEVINL void pt_mma_ss(uint32_t d, uint32_t a_lo, uint32_t b_lo, uint32_t desc_hi, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q, r;\n\t.reg .b32 x, y;\n\t.reg .b64 a, b;\n\t"
        "elect.sync _|p, 0xffffffff;\n\tsetp.ne.b32 q, %5, 0;\n\tsetp.eq.b32 r, 0, 0;\n\t"
        "add.u32 x, %1, 0; add.u32 y, %2, 0; mov.b64 a, {x, %3}; mov.b64 b, {y, %3}; @p tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %4, q;\n\t"
        "add.u32 x, %1, 2; add.u32 y, %2, 2; mov.b64 a, {x, %3}; mov.b64 b, {y, %3}; @p tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %4, r;\n\t"
        "add.u32 x, %1, 4; add.u32 y, %2, 4; mov.b64 a, {x, %3}; mov.b64 b, {y, %3}; @p tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %4, r;\n\t"
        "add.u32 x, %1, 6; add.u32 y, %2, 6; mov.b64 a, {x, %3}; mov.b64 b, {y, %3}; @p tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %4, r;\n\t"
        "add.u32 x, %1, 1024; add.u32 y, %2, 1024; mov.b64 a, {x, %3}; mov.b64 b, {y, %3}; @p tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %4, r;\n\t"
        "add.u32 x, %1, 1026; add.u32 y, %2, 1026; mov.b64 a, {x, %3}; mov.b64 b, {y, %3}; @p tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %4, r;\n\t"
        "add.u32 x, %1, 1028; add.u32 y, %2, 1028; mov.b64 a, {x, %3}; mov.b64 b, {y, %3}; @p tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %4, r;\n\t"
        "add.u32 x, %1, 1030; add.u32 y, %2, 1030; mov.b64 a, {x, %3}; mov.b64 b, {y, %3}; @p tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %4, r;\n\t}"
        ::"r"(d), "r"(a_lo), "r"(b_lo), "r"(desc_hi), "r"(idesc), "r"(accumulate)
        : "memory");
}
// D += A B, A in tensor memory (8 columns per MMA), B MN-major (two 8-token groups of 1024 B per MMA)
DL_DEVINL void pt_mma_ts(uint32_t d, uint32_t a, uint32_t b_lo, uint32_t desc_hi, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q, r;\n\t.reg .b32 x, y;\n\t.reg .b64 a, b;\n\t"
        "elect.sync _|p, 0xffffffff;\n\tsetp.ne.b32 q, %5, 0;\n\tsetp.eq.b32 r, 0, 0;\n\t"
        "add.u32 x, %1, 0; add.u32 y, %2, 0; mov.b64 b, {y, %3}; @p tcgen05.mma.cta_group::1.kind::f16 [%0], [x], b, %4, q;\n\t"
        "add.u32 x, %1, 8; add.u32 y, %2, 128; mov.b64 b, {y, %3}; @p tcgen05.mma.cta_group::1.kind::f16 [%0], [x], b, %4, r;\n\t"
        "add.u32 x, %1, 16; add.u32 y, %2, 256; mov.b64 b, {y, %3}; @p tcgen05.mma.cta_group::1.kind::f16 [%0], [x], b, %4, r;\n\t"
        "add.u32 x, %1, 24; add.u32 y, %2, 384; mov.b64 b, {y, %3}; @p tcgen05.mma.cta_group::1.kind::f16 [%0], [x], b, %4, r;\n\t"
        "add.u32 x, %1, 32; add.u32 y, %2, 512; mov.b64 b, {y, %3}; @p tcgen05.mma.cta_group::1.kind::f16 [%0], [x], b, %4, r;\n\t"
        "add.u32 x, %1, 40; add.u32 y, %2, 640; mov.b64 b, {y, %3}; @p tcgen05.mma.cta_group::1.kind::f16 [%0], [x], b, %4, r;\n\t"
        "add.u32 x, %1, 48; add.u32 y, %2, 768; mov.b64 b, {y, %3}; @p tcgen05.mma.cta_group::1.kind::f16 [%0], [x], b, %4, r;\n\t"
        "add.u32 x, %1, 56; add.u32 y, %2, 896; mov.b64 b, {y, %3}; @p tcgen05.mma.cta_group::1.kind::f16 [%0], [x], b, %4, r;\n\t}"
        ::"r"(d), "r"(a), "r"(b_lo), "r"(desc_hi), "r"(idesc), "r"(accumulate)
        : "memory");
}
// ... of those groups of 16 tokens that have a bit in `groups`; `add`: the ones that add to what is there.  Predicates, no branch: with a branch to MMAs one by one
// 2000 rows of 16 heads took 43.6 us under a window of 1024 and 59.8 without one, 41.6 and 56.0 so
DL_DEVINL void pt_mma_ts_of(uint32_t d, uint32_t a, uint32_t b_lo, uint32_t desc_hi, uint32_t idesc, uint32_t add, uint32_t groups) {
    asm volatile(
        "{\n\t.reg .pred p, q, r;\n\t.reg .b32 x, y, z;\n\t.reg .b64 b;\n\t"
        "elect.sync _|p, 0xffffffff;\n\t"
        "and.b32 z, %5, 1; setp.ne.b32 q, z, 0; and.b32 z, %6, 1; setp.ne.and.b32 r, z, 0, p; add.u32 x, %1, 0; add.u32 y, %2, 0; mov.b64 b, {y, %3}; @r tcgen05.mma.cta_group::1.kind::f16 [%0], [x], b, %4, q;\n\t"
        "and.b32 z, %5, 2; setp.ne.b32 q, z, 0; and.b32 z, %6, 2; setp.ne.and.b32 r, z, 0, p; add.u32 x, %1, 8; add.u32 y, %2, 128; mov.b64 b, {y, %3}; @r tcgen05.mma.cta_group::1.kind::f16 [%0], [x], b, %4, q;\n\t"
        "and.b32 z, %5, 4; setp.ne.b32 q, z, 0; and.b32 z, %6, 4; setp.ne.and.b32 r, z, 0, p; add.u32 x, %1, 16; add.u32 y, %2, 256; mov.b64 b, {y, %3}; @r tcgen05.mma.cta_group::1.kind::f16 [%0], [x], b, %4, q;\n\t"
        "and.b32 z, %5, 8; setp.ne.b32 q, z, 0; and.b32 z, %6, 8; setp.ne.and.b32 r, z, 0, p; add.u32 x, %1, 24; add.u32 y, %2, 384; mov.b64 b, {y, %3}; @r tcgen05.mma.cta_group::1.kind::f16 [%0], [x], b, %4, q;\n\t"
        "and.b32 z, %5, 16; setp.ne.b32 q, z, 0; and.b32 z, %6, 16; setp.ne.and.b32 r, z, 0, p; add.u32 x, %1, 32; add.u32 y, %2, 512; mov.b64 b, {y, %3}; @r tcgen05.mma.cta_group::1.kind::f16 [%0], [x], b, %4, q;\n\t"
        "and.b32 z, %5, 32; setp.ne.b32 q, z, 0; and.b32 z, %6, 32; setp.ne.and.b32 r, z, 0, p; add.u32 x, %1, 40; add.u32 y, %2, 640; mov.b64 b, {y, %3}; @r tcgen05.mma.cta_group::1.kind::f16 [%0], [x], b, %4, q;\n\t"
        "and.b32 z, %5, 64; setp.ne.b32 q, z, 0; and.b32 z, %6, 64; setp.ne.and.b32 r, z, 0, p; add.u32 x, %1, 48; add.u32 y, %2, 768; mov.b64 b, {y, %3}; @r tcgen05.mma.cta_group::1.kind::f16 [%0], [x], b, %4, q;\n\t"
        "and.b32 z, %5, 128; setp.ne.b32 q, z, 0; and.b32 z, %6, 128; setp.ne.and.b32 r, z, 0, p; add.u32 x, %1, 56; add.u32 y, %2, 896; mov.b64 b, {y, %3}; @r tcgen05.mma.cta_group::1.kind::f16 [%0], [x], b, %4, q;\n\t}"
        ::"r"(d), "r"(a), "r"(b_lo), "r"(desc_hi), "r"(idesc), "r"(add), "r"(groups)
        : "memory");
}
DL_DEVINL void pt_commit(uint64_t* bar) {
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\t@p tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(smem_u32(bar)) : "memory");
}

// What a CTA works on: two query tiles of up to 128 (stacked) rows that meet the same keys and values, and the steps that they see.
struct PtItem {
    int kvh, p0, slot, seq_end;            // key/value head; position of the first row of the segment (or run); tokens of the sequence that exist
    int first_page, j0, J;                 // pages ahead of first_page are not touched; steps of 128 tokens, the first one at token j0 * 128
    int ja[2], jb[2];                      // steps [ja, jb) of these are tile t's (none: the tile is not there)
    int row0[2], rows, head[2];            // first row of tile t, rows of the segment (or run), the tile's head
    int seen_from[2], seen_to[2];          // LINES: tokens that rows of tile t see, from the start of the first one's page
    int shares;                            // LINES: into how many shares (grid.z) the steps of the run go
    int begin;                             // batch row of the segment's first row; LINES: entry of tile_rows where the run starts
};

// A wait that gives up (the CTA has had its time, WAIT_DEADLINE_NS): the flag ends the other waits, too, every output of the CTA becomes a NaN, and
// the host learns of it by dl_attention_status()
struct PtWaits {
    volatile int* gave_up;
    unsigned long long t0, ns;
    DL_DEVINL void operator()(uint64_t* bar, uint32_t parity) const {
        unsigned n = 0;
        while (!mbar_try_wait(bar, parity)) {
            if ((++n & 0x3FFu) == 0) {
                if (*gave_up) return;
                if (globaltimer_ns() - t0 > ns) { *gave_up = 1; return; }
            }
        }
    }
};

// Llama path: the items of a batch are (128-row tile of a segment, query head), late tiles (long histories) first: two heads of one key/value head
// side by side, or two tiles of one head where the heads come alone; single tiles while there are SMs for all of them.  Item `idx` of the
// order that all roles of all CTAs walk; false behind the last one.
DL_DEVINL bool pt_item(const PtArgs& a, const int (*seg)[4], int n_seg, int idx, PtItem& it) {
    const int rep = a.n_heads / a.n_kv_heads;
    int tiles = 0;
    for (int i = 0; i < n_seg; i++) tiles += (seg[i][1] + PT_ROWS - 1) / PT_ROWS;
    const bool single = tiles * a.n_heads <= (int)gridDim.x, by_heads = !single && rep % 2 == 0, by_rows = !single && !by_heads;
    const int cols = by_heads ? a.n_heads / 2 : a.n_heads;
    for (int i = 0; i < n_seg; i++) {
        const int nt = (seg[i][1] + PT_ROWS - 1) / PT_ROWS, groups = by_rows ? (nt + 1) / 2 : nt;
        if (idx >= groups * cols) { idx -= groups * cols; continue; }
        const int group = groups - 1 - idx / cols, col = idx % cols;
        it.begin = seg[i][0]; it.rows = seg[i][1]; it.p0 = seg[i][2]; it.slot = seg[i][3];
        it.seq_end = it.p0 + it.rows;
        it.first_page = it.j0 = it.J = 0;
#pragma unroll
        for (int t = 0; t < 2; t++) {
            it.row0[t] = (by_rows ? 2 * group + t : group) * PT_ROWS;
            it.head[t] = by_heads ? 2 * col + t : col;
            const bool there = it.row0[t] < it.rows && (t == 0 || !single);
            it.ja[t] = 0;
            it.jb[t] = there ? (it.p0 + min(it.row0[t] + PT_ROWS, it.rows) - 1) / PT_KV + 1 : 0;
            it.J = max(it.J, it.jb[t]);
        }
        it.kvh = it.head[0] / rep;
        return true;
    }
    return false;
}

// Layer-list models: the runs of consecutive positions among the CTA's list tiles, [first tile, positions, first position, slot] each.  (By a whole warp)
DL_DEVINL int pt_runs(const PtLineArgs& a, int (*runs)[4]) {
    const DlWindowAttnArgs& w = a.w;
    const int t0 = ((int)gridDim.x - 1 - (int)blockIdx.x) * a.group, lane = threadIdx.x & 31;          // late tiles (long histories) first
    int cnt[4] = {0, 0, 0, 0}, m = -1;                           // rows of each tile; the first row of tile `lane`
#pragma unroll
    for (int u = 0; u < 4; u++) {
        for (int r0 = 0; r0 < a.rq && u < a.group && t0 + u < a.n_tiles; r0 += 32) {
            const int row = r0 + lane < a.rq ? a.tile_rows[(size_t)(t0 + u) * a.rq + r0 + lane] : -1;
            cnt[u] += __popc(__ballot_sync(0xffffffffu, row >= 0));
            const int first = __shfl_sync(0xffffffffu, row, 0);
            if (r0 == 0 && lane == u) m = first;
        }
    }
    const int pos = m >= 0 ? w.pos[m] : 0, slot = m >= 0 ? w.slot[m] : 0;
    int n = 0, run = 0, start = 0;
#pragma unroll
    for (int u = 0; u < 4; u++) {
        const int pu = __shfl_sync(0xffffffffu, pos, u), su = __shfl_sync(0xffffffffu, slot, u);
        if (run == 0) start = u;
        run += cnt[u];
        // does the next tile go on with this sequence (window_tiles_join)?
        const bool more = u < 3 && cnt[u] == a.rq && cnt[u < 3 ? u + 1 : 3] > 0 && __shfl_sync(0xffffffffu, pos, u < 3 ? u + 1 : 3) == pu + a.rq && __shfl_sync(0xffffffffu, slot, u < 3 ? u + 1 : 3) == su;
        const int p_start = __shfl_sync(0xffffffffu, pos, start);
        if (more) continue;
        if (run * a.rep > a.least) {
            if (lane == 0) { runs[n][0] = t0 + start; runs[n][1] = run; runs[n][2] = p_start; runs[n][3] = su; }
            n++;
        }
        run = 0;
    }
    return n;
}
// the item of a run: its steps go into no more shares than leave each PT_SHARE_STEPS, so that a short run needs no merge
DL_DEVINL void pt_run_item(const PtLineArgs& a, const int (&run)[4], PtItem& it) {
    const DlWindowAttnArgs& w = a.w;
    it.begin = run[0] * a.rq;
    it.rows = run[1] * a.rep;
    it.p0 = run[2];
    it.slot = run[3];
    it.seq_end = it.p0 + run[1];                                 // what lies behind was not written yet, or is of no use here
    it.kvh = blockIdx.y;
    int lo[2], j[2];
#pragma unroll
    for (int u = 0; u < 2; u++) {
        it.row0[u] = u * PT_ROWS;
        it.head[u] = 0;
        const int p = it.p0 + u * PT_ROWS / a.rep, last = it.p0 + min((u + 1) * PT_ROWS / a.rep, run[1]) - 1;
        lo[u] = w.window > 0 ? max(0, p - w.window + 1) : 0;
        if (w.chunk > 0) lo[u] = max(lo[u], p / w.chunk * w.chunk);
        j[u] = it.row0[u] < it.rows ? last / PT_KV + 1 : 0;
        it.seen_from[u] = lo[u] & ~31;
        it.seen_to[u] = last + 1;
    }
    it.first_page = lo[0] / 32;                                  // (tile 1 starts no earlier)
    it.j0 = lo[0] / PT_KV;
    it.J = max(j[0], j[1]) - it.j0;
    it.shares = max(1, min((int)gridDim.z, it.J / PT_SHARE_STEPS));
    const int per = (it.J + it.shares - 1) / it.shares, z0 = min(it.J, (int)blockIdx.z * per), z1 = min(it.J, z0 + per);
#pragma unroll
    for (int u = 0; u < 2; u++) {
        it.ja[u] = max(lo[u] / PT_KV - it.j0 - z0, 0);
        it.jb[u] = max(min(j[u] - it.j0 - z0, z1 - z0), it.ja[u]);
    }
    it.j0 += z0;
    it.J = z1 - z0;
    it.first_page = max(it.first_page, it.j0 * (PT_KV / 32));
}

// Queries of 32 rows into the tile's K-major, swizzled image: lane i holds the address of row r0 + i; all in flight, a row a load
template <bool LINES, typename Ready>
DL_DEVINL void pt_load_rows(const float* mine, uint8_t* tile, int r0, Ready ready) {
    const int lane = threadIdx.x & 31;
    uint8_t* qd = tile + r0 * 128 + (lane >> 4) * 16384 + (lane & 1) * 8;
    float4 x[32];
#pragma unroll
    for (int u = 0; u < 32; u++) x[u] = reinterpret_cast<const float4*>(__shfl_sync(0xffffffffu, (unsigned long long)(uintptr_t)mine, u))[lane];
    ready();
#pragma unroll
    for (int u = 0; u < 32; u++)                 // 16-byte piece c of a half row -> swizzled slot c ^ (row & 7)
        *reinterpret_cast<uint2*>(qd + u * 128 + ((((lane >> 1) & 7) ^ (u & 7)) << 4)) = make_uint2(pt_pack2<LINES>(x[u].x, x[u].y), pt_pack2<LINES>(x[u].z, x[u].w));
    fence_proxy_async_smem();
}

template <bool LINES>
__global__ void __launch_bounds__(PT_THREADS, 1) attention_prefill_tc_kernel(const __grid_constant__ typename PtKernelArgs<LINES>::T a,
                                                                             const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap vmap) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ int seg[PT_MAX_SEG][4], n_seg_s, gave_up_s;
    if constexpr (!LINES) trace_begin(a.tr);
    uint8_t* q_s = smem;                                        // [2] query tiles
    uint8_t* k_s = q_s + 2 * PT_TILE_BYTES;                     // [2] K tiles (tokens x head dim, K-major)
    uint8_t* v_s = k_s + PT_STAGES * PT_TILE_BYTES;             // [2] V tiles (tokens x head dim, MN-major for P V)
    float* out_s = reinterpret_cast<float*>(v_s + PT_STAGES * PT_TILE_BYTES);      // [8 warps][32][PT_OUT_LD] f32: rows on their way out
    uint64_t* bars = reinterpret_cast<uint64_t*>(out_s + 8 * 32 * PT_OUT_LD);
    uint64_t* k_full = bars;             // [2] transaction bytes of the step's K copies
    uint64_t* k_empty = bars + 2;        // [2] the scores that read the stage are complete (both tiles')
    uint64_t* v_full = bars + 4;         // [2] transaction bytes of the step's V copies
    uint64_t* v_empty = bars + 6;        // [2] P V of the step has retired (both tiles')
    uint64_t* q_full = bars + 8;         // [2] the tile's queries are there
    uint64_t* q_empty = bars + 10;       // [2] the tile's last scores are complete
    uint64_t* s_full = bars + 12;        // [2] scores complete
    uint64_t* p_full = bars + 14;        // [2] probabilities written
    uint64_t* o_full = bars + 16;        // [2] P V complete (LINES: of the tile's last step of an item)
    uint64_t* s_empty = bars + 18;       // the scores have been read into registers (one buffer for both tiles)
    uint64_t* p_turn = bars + 19;        // [2] LINES: the place for probabilities is the tile's, for one step of it
    uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(bars + 21);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    pdl_launch_dependents();
    if (tid == 0) {
        gave_up_s = a.limit.ns == 0;
        for (int s = 0; s < 2; s++) {
            mbar_init(&k_full[s], 1);
            mbar_init(&k_empty[s], 1);
            mbar_init(&v_full[s], 1);
            mbar_init(&v_empty[s], 1);
            mbar_init(&q_full[s], 128);
            mbar_init(&q_empty[s], 1);
            mbar_init(&s_full[s], 1);
            mbar_init(&p_full[s], 128);
            mbar_init(&o_full[s], 1);
            mbar_init(&p_turn[s], 1);
        }
        mbar_init(s_empty, 128);
        mbar_fence_init();
    }
    if constexpr (!LINES) {
        pdl_wait();                                              // q, this chunk's KV rows and meta come from earlier kernels
        if (warp == 1) {
            const int ns = min(a.meta[0], PT_MAX_SEG);
            if (lane == 0) n_seg_s = ns;
            if (lane < ns) {
                const int b = a.meta[1 + 2 * lane], e = a.meta[2 + 2 * lane];
                seg[lane][0] = b;
                seg[lane][1] = e - b;
                seg[lane][2] = e > b ? a.pos[b] : 0;
                seg[lane][3] = e > b ? a.slot[b] : 0;
            }
        }
    } else {
        // (launched behind a kernel that writes the rows of other tiles and reads the same inputs: nothing to wait for here.  What
        // follows this grid must follow that one too, so this grid may not end ahead of it: a CTA with work waits when it is done, and the
        // first CTA waits even without -- one is enough, a grid ends with its last CTA, and all of the idle ones would keep an SM each
        // from those with work)
        if (warp == 1) {
            const int n = pt_runs(a, seg);
            if (lane == 0) n_seg_s = n;
        }
        __syncthreads();
        if (n_seg_s == 0) {
            if (blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0) pdl_wait();
            return;
        }
    }
    if (warp == 0) tmem_alloc(tmem_holder, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const PtWaits wait = {&gave_up_s, globaltimer_ns(), a.limit.ns};
    const int n_seg = n_seg_s;
    // the items of this CTA, in the same order for every role; rounds run back and forth over the CTAs, so that a long item goes with a short one
    auto item_at = [&](int round, PtItem& it) {
        if constexpr (LINES) {
            if (round < n_seg) pt_run_item(a, seg[round], it);
            return round < n_seg;
        } else {
            const int G = gridDim.x, b = blockIdx.x;
            return pt_item(a, seg, n_seg, round * G + ((round & 1) ? G - 1 - b : b), it);
        }
    };
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_holder, 0);
    // TMEM columns: one buffer of scores at 0, which the tiles take in turn; probabilities at 128, of 64 columns for each tile (LINES: of 128, which
    // the tiles take in turn, too); outputs at 256 + 128 t
    const auto t_p = [&](int t) { return tmem_base + 128 + (LINES ? 0 : t * 64); };
    auto row_of = [&](const PtItem& it, int t, int row) -> const float* {      // the queries of a tile's row (rows that are not there: of the last one)
        const int r = min((t ? it.row0[1] : it.row0[0]) + row, it.rows - 1);
        if constexpr (LINES) return a.w.q + (size_t)a.tile_rows[it.begin + r / a.rep] * a.w.ldq + (it.kvh * a.rep + r % a.rep) * PT_HS;
        else return a.q + (size_t)(it.begin + r) * a.n_heads * PT_HS + (t ? it.head[1] : it.head[0]) * PT_HS;
    };

    // 128-byte-swizzled operands: rows of 128 B (64 halfs), 8-row groups 1024 B apart; the head dimension is split in
    // two such half tiles 16 KB apart.  K-major (Q, K): LBO unused (1), SBO 1024.  MN-major (V as B of P V): LBO =
    // distance between the two 64-wide halves of N (16 KB), SBO = distance between 8-token groups (1024 B).
    if (warp < 8) {
        // ---------------- softmax: warps 0-3 tile 0, warps 4-7 tile 1; a thread per query row (= TMEM lane) ----------------
        asm volatile("setmaxnreg.inc.sync.aligned.u32 208;");
        const int t = warp >> 2, quarter = warp & 3, row = quarter * 32 + lane;
        const uint32_t lane_base = (uint32_t)(quarter * 32) << 16, T_S = tmem_base + lane_base, T_P = t_p(t) + lane_base, T_O = tmem_base + lane_base + 256 + t * 128;
        float* stage = out_s + (size_t)warp * 32 * PT_OUT_LD;
        uint32_t ns = 0, nq = 0;                                 // steps of this tile so far, items whose queries are loaded
        PtItem it, next;
        // the queries of the tile's next item: all rows in flight at once, ahead of this item's outputs
        auto load_queries = [&](const PtItem& of) {
            if (!(t ? of.jb[1] > of.ja[1] : of.jb[0] > of.ja[0])) return;
            pt_load_rows<LINES>(row_of(of, t, row), q_s + t * PT_TILE_BYTES, quarter * 32, [&] {
                if (nq > 0) wait(&q_empty[t], (nq - 1) & 1);      // the tile's last scores have read the queries before
            });
            nq++;
            mbar_arrive(&q_full[t]);
        };
        bool more = item_at(0, it);
        if (more) load_queries(it);
        for (int round = 0; more; round++, it = next) {
            const int ja = t ? it.ja[1] : it.ja[0], jb = t ? it.jb[1] : it.jb[0], row0 = t ? it.row0[1] : it.row0[0], head = t ? it.head[1] : it.head[0];
            const int r_abs = row0 + row, r_live = min(r_abs, it.rows - 1);
            int pos_r, lb = 0, m_row = 0, h_row = 0;             // last and first visible position of this row; LINES: its batch row and head
            float sc, c1 = 0.f, cap_k = 0.f, slope = 0.f;
            bool shaped = false;                                 // scores leave the accumulator through a cap, a bias or a factor that is not positive
            if constexpr (LINES) {
                const DlWindowAttnArgs& w = a.w;
                m_row = a.tile_rows[it.begin + r_live / a.rep];
                h_row = it.kvh * a.rep + r_live % a.rep;
                pos_r = it.p0 + r_live / a.rep;
                if (w.window > 0) lb = max(0, pos_r - w.window + 1);
                if (w.chunk > 0) lb = max(lb, pos_r / w.chunk * w.chunk);
                shaped = w.softcap > 0.f || w.slope != nullptr || !(w.scale > 0.f);      // (a factor that keeps no order meets the scores ahead of mask and maximum)
                sc = 1.4426950408889634f * w.scale;
                c1 = w.softcap > 0.f ? sc * 2.f / w.softcap : sc;
                cap_k = w.softcap * 1.4426950408889634f;
                if (w.slope != nullptr) slope = w.slope[h_row] * 1.4426950408889634f;
                if (shaped) sc = 1.f;
            } else {
                pos_r = it.p0 + r_abs;
                sc = 1.4426950408889634f * rsqrtf((float)PT_HS);     // scores in the log2 domain
            }
            float m_used = -INFINITY, l = 0.0f;
            for (int j = ja; j < jb; j++, ns++) {
                uint32_t v[4][32];
                wait(&s_full[t], ns & 1);
                tc_fence_after();
#pragma unroll
                for (int c = 0; c < 4; c++) tmem_ld_32x32b_x32(T_S + c * 32, v[c]);
                tmem_ld_wait();
                tc_fence_before();
                mbar_arrive(s_empty);                            // the next scores may take the place
                const int tok0 = (it.j0 + j) * PT_KV;
                const int lim = pos_r - tok0, low = LINES ? lb - tok0 : 0;      // columns low <= e <= lim are visible to this row
                if constexpr (LINES) {
                    if (shaped) {
#pragma unroll
                        for (int e = 0; e < PT_KV; e++) {
                            float x = __uint_as_float(v[e >> 5][e & 31]) * c1;
                            if (cap_k > 0.f) {                   // cap tanh(s / cap) in base 2, as the mma.sync kernel forms it
                                float r;
                                asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(pt_ex2(x) + 1.f));
                                x = fmaf(-2.f * cap_k, r, cap_k);
                            }
                            v[e >> 5][e & 31] = __float_as_uint(fmaf(-slope, (float)(lim - e), x));
                        }
                    }
                }
                if (lim < PT_KV - 1 || (LINES && low > 0)) {
#pragma unroll
                    for (int c = 0; c < 4; c++) {                // a bit per column
                        const int hi = lim - c * 32, lo = low - c * 32;
                        uint32_t cols = hi < 0 ? 0u : hi >= 31 ? 0xffffffffu : (2u << hi) - 1;
                        if (LINES) cols &= lo <= 0 ? 0xffffffffu : lo > 31 ? 0u : 0xffffffffu << lo;
#pragma unroll
                        for (int e = 0; e < 32; e++)
                            if (!(cols & (1u << e))) v[c][e] = 0xff800000u;        // -inf
                    }
                }
                float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
                for (int e = 0; e < 32; e += 2)
#pragma unroll
                    for (int c = 0; c < 4; c++) mx4[c] = fmaxf(mx4[c], fmaxf(__uint_as_float(v[c][e]), __uint_as_float(v[c][e + 1])));
                const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * sc;
                const bool need = mx > m_used + 8.0f;            // the reference may lag the maximum by 2^8
                const bool moved = __any_sync(0xffffffffu, need);
                float alpha = 1.f;
                if (moved) {
                    const float m_new = need ? mx : m_used;
                    if (need) alpha = pt_ex2(m_used - m_new);
                    l *= alpha;
                    m_used = m_new;
                }
                const float ref = (m_used == -INFINITY) ? 0.0f : m_used;
                pair_f sum = 0;
                uint32_t pk[4][16], lo[4][LINES ? 16 : 1];
                // LINES: formed ahead of the waits, in the scores' registers, as the place is free only when the other tile's have been multiplied
                if constexpr (LINES) {
#pragma unroll
                    for (int c = 0; c < 4; c++) pt_probs<LINES>(v[c], sc, ref, pk[c], lo[c], sum);
                }
                // this tile's P V before is complete; LINES: and the other's, whose probabilities lie in this place.  Neither barrier can be more than the one
                // phase ahead that a parity tells, as its next phase waits for the probabilities of this step (the phases of the other tile's o_full pass
                // while this tile has no steps)
                if constexpr (LINES) wait(&p_turn[t], ns & 1);
                else if (j > ja) wait(&o_full[t], (ns - 1) & 1);
                tc_fence_after();
                if (moved && j > ja) {      // the accumulated output moves to the new reference (rare after the first steps)
                    uint32_t w[32];
#pragma unroll 1
                    for (int ch = 0; ch < 4; ch++) {
                        tmem_ld_32x32b_x32(T_O + ch * 32, w);
                        tmem_ld_wait();
#pragma unroll
                        for (int e = 0; e < 32; e++) w[e] = __float_as_uint(__uint_as_float(w[e]) * alpha);
                        tmem_st_32x32b_x32(T_O + ch * 32, w);
                    }
                }
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    if constexpr (!LINES) pt_probs<LINES>(v[c], sc, ref, pk[c], lo[c], sum);
                    tmem_st_32x32b_x16(T_P + c * 16, pk[c]);
                    if constexpr (LINES) tmem_st_32x32b_x16(T_P + 64 + c * 16, lo[c]);
                }
                l += pair_sum(sum);
                tmem_st_wait();
                tc_fence_before();
                mbar_arrive(&p_full[t]);
            }
            more = item_at(round + 1, next);
            if (more) load_queries(next);
            // ---- finish: O / l -> f32 rows, partial sums, or the Q80 cast into the slabs of the wo matmul ----
            float inv;
            if constexpr (LINES) {
                if (it.shares == 1 && a.w.sink) l += pt_ex2(a.w.sink[h_row] * 1.4426950408889634f - m_used);
                inv = it.shares > 1 ? 1.f : (a.w.gate ? 1.f / (1.f + expf(-a.w.gate[(size_t)m_row * a.w.ld_gate + h_row])) : 1.f) / l;
            } else {
                inv = l > 0.0f ? 1.0f / l : 0.0f;
            }
            float* out = nullptr;                                // this thread's row; null: none
            bool vec = true;                                     // 16-byte rows
            if constexpr (LINES) {
                if (row0 >= it.rows || (it.shares == 1 && blockIdx.z > 0)) continue;
                out = a.w.out + (size_t)m_row * a.w.ldo + h_row * PT_HS;
                vec = ((uintptr_t)a.w.out & 15) == 0 && (a.w.ldo & 3) == 0;
                if (a.n_splits > 1) {                            // a stacked row's slot among the list tile's partial sums
                    constexpr int step = PT_ROWS / 2 * (PT_HS + 2);
                    const int u = it.begin / a.rq + r_live / (PT_ROWS / 2);
                    float* part = a.partial + (((size_t)u * a.w.kv_heads + it.kvh) * a.n_splits + blockIdx.z) * step + r_live % (PT_ROWS / 2) * (PT_HS + 2);
                    if (r_abs < it.rows) {                       // (-2: no merge, -1: nothing in this share)
                        part[PT_HS] = m_used * 0.6931471805599453f;
                        part[PT_HS + 1] = it.shares == 1 ? -2.f : jb > ja ? l : -1.f;
                        for (int z = gridDim.z; blockIdx.z == 0 && it.shares > 1 && z < a.n_splits; z++) {
                            part[(size_t)z * step + PT_HS] = -INFINITY;
                            part[(size_t)z * step + PT_HS + 1] = -1.f;
                        }
                    }
                    if (it.shares > 1) { out = part; vec = false; }
                }
                if (jb == ja) continue;
            } else {
                if (jb == ja) continue;
                if (a.y_out != nullptr) out = a.y_out + (size_t)(it.begin + r_live) * a.n_heads * PT_HS + head * PT_HS;
                vec = ((uintptr_t)a.y_out & 15) == 0;
            }
            if constexpr (LINES) {                               // (the barrier's phase in the topmost bit)
                wait(&o_full[t], ns >> 31);
                ns ^= 1u << 31;
            } else {
                wait(&o_full[t], (ns - 1) & 1);
            }
            tc_fence_after();
            if (gave_up_s) inv = __int_as_float(0x7fffffff);
            const int live = it.rows - (row0 + quarter * 32);      // rows of this warp that are there
#pragma unroll 1
            for (int ch = 0; ch < 4; ch++) {
                uint32_t o[32];
                float f[32];
                tmem_ld_32x32b_x32(T_O + ch * 32, o);
                tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < 32; e++) f[e] = __uint_as_float(o[e]) * inv;
                if constexpr (!LINES) {
                    if (r_abs < it.rows && (a.xq_out != nullptr || a.xh_out != nullptr))
                        pt_q80_block(f, it.begin + r_abs, head * (PT_HS / 32) + ch, a.out_mcap, a.xq_out, a.xh_out);
                    if (out == nullptr) continue;
                }
#pragma unroll
                for (int h = 0; h < 2; h++) {                    // 16 columns of the warp's rows, then as many lanes along a row
                    __syncwarp();
#pragma unroll
                    for (int e = 0; e < 16; e += 4) *reinterpret_cast<float4*>(stage + lane * PT_OUT_LD + e) = make_float4(f[h * 16 + e], f[h * 16 + e + 1], f[h * 16 + e + 2], f[h * 16 + e + 3]);
                    __syncwarp();
#pragma unroll
                    for (int rr = 0; rr < 32; rr += 8) {
                        const int r = rr + (lane >> 2);
                        float* dst = reinterpret_cast<float*>(__shfl_sync(0xffffffffu, (unsigned long long)(uintptr_t)out, r)) + ch * 32 + h * 16 + (lane & 3) * 4;
                        const float4 x = *reinterpret_cast<const float4*>(stage + r * PT_OUT_LD + (lane & 3) * 4);
                        if (r >= live) continue;
                        if (vec) *reinterpret_cast<float4*>(dst) = x;
                        else { dst[0] = x.x; dst[1] = x.y; dst[2] = x.z; dst[3] = x.w; }
                    }
                }
            }
            tc_fence_before();                                   // the next item's P V may write the output (behind p_full)
        }
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 88;");
        const uint32_t desc_hi = (1024u >> 4) | (1u << 14) | (2u << 29);
        if (warp == 8) {
            // ---------------- MMAs, all by one thread: what it issues runs in that order ----------------
            const uint32_t idesc_s = pt_idesc(PT_ROWS, PT_KV, 0, LINES), idesc_pv = pt_idesc(PT_ROWS, PT_HS, 1, LINES);
            const uint32_t q_lo = ((smem_u32(q_s) & 0x3FFFFu) >> 4) | (1u << 16), k_lo = ((smem_u32(k_s) & 0x3FFFFu) >> 4) | (1u << 16);
            const uint32_t v_lo = ((smem_u32(v_s) & 0x3FFFFu) >> 4) | ((16384u >> 4) << 16);
            uint32_t g = 0, n_s = 0, ns[2] = {0, 0}, nq[2] = {0, 0};      // steps, scores, steps of a tile, items of a tile so far
            PtItem it;
            for (int round = 0; item_at(round, it); round++) {
                auto on = [&](int t, int j) { return j >= it.ja[t] && j < it.jb[t]; };
                auto scores = [&](int t, int j) {                // S = Q K^T of a step
                    const int st = (g + j) & 1;
                    if (!on(t, j)) return;
                    wait(&k_full[st], ((g + j) >> 1) & 1);
                    if (j == it.ja[t]) wait(&q_full[t], nq[t]++ & 1);
                    if (n_s > 0) wait(s_empty, (n_s - 1) & 1);
                    n_s++;
                    tc_fence_after();
                    __syncwarp();
                    pt_mma_ss(tmem_base, q_lo + t * (PT_TILE_BYTES >> 4), k_lo + st * (PT_TILE_BYTES >> 4), desc_hi, idesc_s, 0);
                    pt_commit(&s_full[t]);
                    if (t == 1 || !on(1, j)) pt_commit(&k_empty[st]);
                    if (j + 1 == it.jb[t]) pt_commit(&q_empty[t]);
                };
                auto outputs = [&](int t, int j) {               // O += P V of a step
                    const int st = (g + j) & 1;
                    if (on(t, j)) {
                        // whose P V comes next (between an item's first step and its last one of the tiles has one)
                        const int next = t == 0 && on(1, j) ? 1 : on(0, j + 1) ? 0 : on(1, j + 1) ? 1 : -1;
                        // LINES: the groups of 16 tokens that the tile sees, no others: the other tile's values may not be finite, and zero times those is a NaN
                        const int tok = (it.j0 + j) * PT_KV, k0 = LINES ? max(0, (it.seen_from[t] - tok) >> 4) : 0, k1 = LINES ? min(8, (it.seen_to[t] - tok + 15) >> 4) : 8;
                        const uint32_t groups = (0xFFu << k0) & (0xFFu >> (8 - k1)), add = j > it.ja[t] ? 0xFFu : 0xFFu & ~(1u << k0);
                        wait(&p_full[t], ns[t]++ & 1);
                        tc_fence_after();
                        __syncwarp();
                        const uint32_t b_lo = v_lo + st * (PT_TILE_BYTES >> 4), T_O = tmem_base + 256 + t * 128;
                        if constexpr (LINES) {
                            pt_mma_ts_of(T_O, t_p(t), b_lo, desc_hi, idesc_pv, add, groups);
                            pt_mma_ts_of(T_O, t_p(t) + 64, b_lo, desc_hi, idesc_pv, 0xFFu, groups);
                        } else {
                            pt_mma_ts(T_O, t_p(t), b_lo, desc_hi, idesc_pv, j > it.ja[t] ? 1u : 0u);
                        }
                        if (LINES && next >= 0) pt_commit(&p_turn[next]);
                        if (!LINES || j + 1 == it.jb[t]) pt_commit(&o_full[t]);
                    }
                    if (t == 1) pt_commit(&v_empty[st]);
                };
                // LINES: a tile may store probabilities when all that was issued ahead of its turn is complete
                if (LINES && it.J > 0) {
                    uint64_t* first = &p_turn[on(0, 0) ? 0 : 1];
                    if (n_s > 0) pt_commit(first);
                    else if (lane == 0) mbar_arrive(first);
                }
                scores(0, 0);
                scores(1, 0);
                scores(0, 1);
                for (int j = 0; j < it.J; j++) {
                    const int st = (g + j) & 1;
                    wait(&v_full[st], ((g + j) >> 1) & 1);
                    // tokens that were not copied, or never written: their scores are masked, but a zero probability times a non-finite V would
                    // poison the product -> zero them
                    const int tok0 = (it.j0 + j) * PT_KV;
                    if ((LINES && it.first_page * 32 > tok0) || tok0 + PT_KV > it.seq_end) {
                        uint8_t* vz = v_s + st * PT_TILE_BYTES;
                        const int z0 = LINES ? max(0, it.first_page * 32 - tok0) : 0, z1 = min(PT_KV, it.seq_end - tok0);
                        for (int idx = lane; idx < PT_KV * 16; idx += 32) {      // 16 pieces of 16 B per token row (two halves)
                            const int r = idx >> 4, c = idx & 15;
                            if (r < z0 || r >= z1) *reinterpret_cast<uint4*>(vz + (c >> 3) * 16384 + r * 128 + (c & 7) * 16) = make_uint4(0, 0, 0, 0);
                        }
                        fence_proxy_async_smem();
                        __syncwarp();
                    }
                    // the scores after next wait in the buffer when the softmax threads come for them
                    outputs(0, j);
                    scores(1, j + 1);
                    outputs(1, j);
                    scores(0, j + 2);
                }
                g += it.J;
            }
        } else if (warp == 9 || warp == 10) {
            // ---------------- K producer (warp 9) / V producer (warp 10), one lane each ----------------
            if (lane == 0) {
                const bool is_k = warp == 9;
                const uint64_t map = is_k ? reinterpret_cast<uint64_t>(&kmap) : reinterpret_cast<uint64_t>(&vmap);
                uint64_t* full = is_k ? k_full : v_full;
                uint64_t* empty = is_k ? k_empty : v_empty;
                uint8_t* ring = is_k ? k_s : v_s;
                int n_kv, max_pages;
                const int* table;
                if constexpr (LINES) { n_kv = a.w.kv_heads; max_pages = a.w.max_pages; table = a.w.block_table; }
                else { n_kv = a.n_kv_heads; max_pages = a.max_pages; table = a.block_table; }
                uint32_t g = 0;
                PtItem it;
                for (int round = 0; item_at(round, it); round++) {
                    const int* bt = table + (size_t)it.slot * max_pages;
                    const int total_pages = (it.seq_end + 31) / 32;
                    auto page_of = [&](int p) { return p >= it.first_page && p < total_pages ? bt[p] : 0; };
                    // the page ids of a step are fetched one step ahead, so the table reads (dependent global loads) overlap the
                    // wait for a free stage instead of delaying the copies
                    int pg[4], pg_next[4];
#pragma unroll
                    for (int p4 = 0; p4 < 4; p4++) pg_next[p4] = page_of(4 * it.j0 + p4);
                    for (int j = 0; j < it.J; j++, g++) {
                        const int st = g & 1;
#pragma unroll
                        for (int p4 = 0; p4 < 4; p4++) {
                            pg[p4] = pg_next[p4];
                            pg_next[p4] = page_of(4 * (it.j0 + j + 1) + p4);
                        }
                        if (g >= PT_STAGES) wait(&empty[st], ((g >> 1) & 1) ^ 1);
                        if (gave_up_s) break;                    // no more copies into a CTA that ends
                        const int n_pg = min(4, total_pages - 4 * (it.j0 + j));                          // pages of this step that exist
                        const int p_lo = LINES ? max(0, it.first_page - 4 * (it.j0 + j)) : 0;            // ... and are looked at (at most the first step starts later)
                        mbar_arrive_expect_tx(&full[st], (uint32_t)max(0, n_pg - p_lo) * 2u * 4096u);
                        const uint32_t dst = smem_u32(ring + st * PT_TILE_BYTES), bar = smem_u32(&full[st]);
#pragma unroll
                        for (int p4 = 0; p4 < 4; p4++) {
                            if (p4 >= n_pg) break;
                            if (LINES && p4 < p_lo) continue;
                            const int y = (pg[p4] * n_kv + it.kvh) * 32;      // first row of the page in the [rows][128] view
#pragma unroll
                            for (int h = 0; h < 2; h++)
                                asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
                                                 dst + h * 16384 + p4 * 4096),
                                             "l"(map), "r"((LINES && !is_k ? PT_HS : 0) + h * 64), "r"(y), "r"(bar)
                                             : "memory");
                        }
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (gave_up_s) {
        if (tid == 0) wait_report(a.limit);
        wait_settle();
    }
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
    if constexpr (LINES) pdl_wait();                             // what follows this grid follows the one ahead of it too
    else trace_end(a.tr);
}

extern void dl_set_error(const char* fmt, ...);
extern int dl_device_sm_count();

static std::atomic<unsigned long long> g_pt_limit{WAIT_DEADLINE_NS};
extern "C" void dl_debug_set_attention_limit(unsigned long long ns) { g_pt_limit = ns; }
static int pt_limit(WaitLimit* l) {
    if (dl_wait_limit("attention_prefill_tc", l) != 0) return -1;
    l->ns = g_pt_limit;
    return 0;
}

#define PT_SMEM ((2 + 2 * PT_STAGES) * PT_TILE_BYTES + 8 * 32 * PT_OUT_LD * 4 + 22 * 8)

// [rows][width] fp16 or bf16 view of a KV cache on THIS GPU (rows = pages x kv heads x 32), box = 64 columns x 32 rows (one page of
// one head, half of the head dimension), 128-byte swizzle: the image tcgen05.mma reads as a swizzled K- or MN-major tile
static int pt_make_map(CUtensorMap* m, const void* base, long long rows, int width, bool bf16) {
    const cuuint64_t dims[2] = {(cuuint64_t)width, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)width * 2};
    const cuuint32_t box[2] = {64, 32};
    return dl_tensor_map("attention_prefill_tc", m, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, base, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
}

extern "C" int dl_attention_prefill_tc(const float* q, int M, int n_heads, int n_kv_heads, int head_size, const void* k_cache,
                                       const void* v_cache, const int* pos, const int* slot, const int* block_table,
                                       int max_pages, int page_size, const int* meta, uint8_t* xq_out, uint8_t* xh_out,
                                       int out_mcap, float* y_out, int n_cache_pages, int pdl, void* stream) {
    if (page_size != 32 || head_size != PT_HS) { dl_set_error("dl_attention_prefill_tc: page size 32 and head size 128 only"); return -1; }
    if (n_heads % n_kv_heads != 0) { dl_set_error("dl_attention_prefill_tc: bad head grouping"); return -1; }
    if (n_cache_pages < 1) { dl_set_error("dl_attention_prefill_tc: n_cache_pages < 1"); return -1; }
    PtArgs a;
    a.q = q; a.k_cache = (const __half*)k_cache; a.v_cache = (const __half*)v_cache; a.pos = pos; a.slot = slot;
    a.block_table = block_table; a.meta = meta; a.M = M; a.n_heads = n_heads; a.n_kv_heads = n_kv_heads;
    a.max_pages = max_pages; a.xq_out = xq_out; a.xh_out = xh_out; a.out_mcap = out_mcap; a.y_out = y_out;
    if (pt_limit(&a.limit) != 0) return -1;
    a.tr = dl_trace_next(TR_ATT);
    alignas(64) CUtensorMap kmap, vmap;
    const long long rows = (long long)n_cache_pages * n_kv_heads * 32;
    if (pt_make_map(&kmap, k_cache, rows, PT_HS, false) != 0 || pt_make_map(&vmap, v_cache, rows, PT_HS, false) != 0) return -1;
    const size_t smem = PT_SMEM;
    static SmemLimit given;
    if (const int rc = dl_smem_limit("attention_prefill_tc", attention_prefill_tc_kernel<false>, smem, given)) return rc;
    cudaLaunchConfig_t cfg = {};
    const long long most = ((long long)(M + PT_ROWS - 1) / PT_ROWS + PT_MAX_SEG - 1) * n_heads;        // upper bound of the tiles of all segments
    cfg.gridDim = dim3((unsigned)(most < dl_device_sm_count() ? most : dl_device_sm_count()));
    cfg.blockDim = dim3(PT_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = (cudaStream_t)stream;
    cudaLaunchAttribute attr[1];
    if (pdl) {
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
    }
    cudaError_t e = cudaLaunchKernelEx(&cfg, attention_prefill_tc_kernel<false>, a, kmap, vmap);
    if (e != cudaSuccess) { dl_set_error("attention_prefill_tc launch: %s", cudaGetErrorString(e)); return -(int)e; }
    return 0;
}

// 0 if the kernel's LINES instance takes these sizes: bf16 lines of a key and a value of 128, full tiles of 64 stacked rows
int dl_window_prefill_tc_supported(const DlWindowAttnArgs& a, int rq) {
    const int rep = a.kv_heads > 0 ? a.heads / a.kv_heads : 0;
    return a.dim == PT_HS && a.vdim == PT_HS && a.page_size == 32 && rep > 0 && rq * rep == PT_ROWS / 2 &&
                   ((uintptr_t)a.cache & 15) == 0 ? 0 : -1;
}

// The most shares that a run's steps go into: none where the SMs are taken, or where no run can be long enough.
int dl_window_prefill_tc_shares(const DlWindowAttnArgs& w, int n_tiles, int group, int n_splits) {
    const int ctas = (n_tiles + group - 1) / group * w.kv_heads, spare = dl_device_sm_count() / ctas;
    const long long seen = w.window > 0 && w.window < w.max_pages * 32ll ? w.window + 2 * PT_ROWS : w.max_pages * 32ll;
    const long long most = (seen / PT_KV + 2) / PT_SHARE_STEPS, z = spare < most ? spare : most;
    return z < 1 ? 1 : z < n_splits ? (int)z : n_splits;
}

// The tiles of more than 16 stacked rows, launched behind the kernel that takes the others (programmatic launch: they run side by side), or
// (alone) all of them.
int dl_window_prefill_tc(const DlWindowAttnArgs& w, const int* tile_rows, int n_tiles, int rq, int group, int n_splits, float* partial, bool alone, cudaStream_t stream) {
    PtLineArgs a;
    a.w = w; a.tile_rows = tile_rows; a.n_tiles = n_tiles; a.rq = rq; a.rep = w.heads / w.kv_heads;
    a.group = group; a.n_splits = n_splits; a.partial = partial;
    a.least = alone ? 0 : 16;
    if (pt_limit(&a.limit) != 0) return -1;
    const int groups = (n_tiles + group - 1) / group, z = dl_window_prefill_tc_shares(w, n_tiles, group, n_splits);
    alignas(64) CUtensorMap map;
    // the cache's page count is not known here; every copy reads a page that the block table names
    if (pt_make_map(&map, w.cache, 1ll << 31, 2 * PT_HS, true) != 0) return -1;
    const size_t smem = PT_SMEM;
    static SmemLimit given;
    if (const int rc = dl_smem_limit("window_prefill_tc", attention_prefill_tc_kernel<true>, smem, given)) return rc;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)groups, (unsigned)w.kv_heads, (unsigned)z);
    cfg.blockDim = dim3(PT_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = alone ? 0 : 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, attention_prefill_tc_kernel<true>, a, map, map);
    if (e != cudaSuccess) { dl_set_error("window_prefill_tc launch: %s", cudaGetErrorString(e)); return -(int)e; }
    return 0;
}
