// Paged GQA attention for decode rows and prefill-chunk rows (flash-decode, split-KV).
//
// Replaces OP_MULTIHEAD_ATT (multiheadAtt_F32, src/nn/nn-cpu-ops.cpp:749-784), which materialises
// a [seqLen] score row per head over ONE shared contiguous KV cache.  Here:
//  * every batch row m has its own position pos[m] and its own KV pages (block_table[slot[m]]),
//    so concurrent users never touch each other's cache (fixes reference defects D2/D3);
//  * grid = (split, kv_head, row): each CTA streams a page range of ONE kv head through a
//    4-stage bulk-async-copy ring (a page of one head is contiguous: page_size*head_size
//    elements) and serves all G = n_heads/n_kv_heads query heads of the group from it;
//  * online softmax; scores of 8 tokens x 4 heads are reduced across the warp with a 31-shuffle
//    transpose-reduce, leaving exactly one (token, head) score per lane -> one exp per lane;
//  * split results go to a scratch buffer; the last CTA to finish a (row, kv head) merges them
//    (self-resetting counter), so the whole op is one launch;
//  * the output is cast to Q80 and written directly in the XQ / XH slab layout the wo matmul
//    consumes (OP_CAST y->yq_slice, src/llm.cpp:296-301).
#include <math.h>
#define WAIT_UNIT 4u
#include "epilogue.cuh"
#include "smem_limit.cuh"
#include "waits.cuh"

#define ATT_PAGE 32            // tokens per KV page (fixed)
#define ATT_STAGES 4
#define ATT_MIN_SPLIT_PAGES 24    // contexts up to 768 tokens: one CTA per (row, kv head), no split
#define ATT_WARPS 4
#define ATT_THREADS (ATT_WARPS * 32 + 32)
#define ATT_COUNTER_BYTES 65536   // completion counters live at scratch offset 0; caller zeroes scratch once

struct AttArgs {
    const float* q;            // [M][n_heads*HS]
    const void* k_cache;       // [pages][n_kv][ATT_PAGE][HS]
    const void* v_cache;
    const int* pos;
    const int* slot;
    const int* block_table;
    const int* row_skip;       // NULL, or row_skip[m] != 0: row m is served by the prefill kernel
    int M, n_heads, n_kv_heads, max_pages, n_splits;
    unsigned* counters;        // scratch: [M][n_kv_heads] at offset 0 (fixed 64 KB region, stays zero)
    float* part_o;             //          [M][n_heads][n_splits][HS]
    float* part_ml;            //          [M][n_heads][n_splits][2]
    uint8_t* xq_out;
    uint8_t* xh_out;
    int out_mcap;
    float* y_out;              // [M][n_heads*HS] or NULL
    unsigned long long* tr;
};

// 32 values per lane -> lane i ends with the warp-wide sum of value i (31 shuffles)
DL_DEVINL float warp_transpose_reduce32(float (&v)[32], int lane) {
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
        const bool upper = (lane & o) != 0;
#pragma unroll
        for (int k = 0; k < o; k++) {
            const float send = upper ? v[k] : v[k + o];
            const float keep = upper ? v[k + o] : v[k];
            v[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    return v[0];
}

template <typename T> DL_DEVINL float kv_to_float(T v);
template <> DL_DEVINL float kv_to_float<float>(float v) { return v; }
template <> DL_DEVINL float kv_to_float<__half>(__half v) { return __half2float(v); }

template <int HS, int NCH, typename KV>
__global__ void __launch_bounds__(ATT_THREADS, 1) attention_kernel(const __grid_constant__ AttArgs a, const __grid_constant__ WaitLimit limit) {
    constexpr int DPL = HS / 32;                       // head dims per lane
    constexpr int PAGE_BYTES = ATT_PAGE * HS * (int)sizeof(KV);
    constexpr int GMAX = NCH * 4;
    extern __shared__ __align__(128) uint8_t smem[];
    trace_begin(a.tr);
    uint8_t* ring = smem;                                                   // [STAGES][2][PAGE_BYTES]
    float* q_s = reinterpret_cast<float*>(ring + ATT_STAGES * 2 * PAGE_BYTES);    // [GMAX][HS] pre-scaled
    float* w_acc = q_s + GMAX * HS;                                         // [WARPS][GMAX][HS]
    float* w_ml = w_acc + ATT_WARPS * GMAX * HS;                            // [WARPS][GMAX][2]
    float* c_ml = w_ml + ATT_WARPS * GMAX * 2;                              // [GMAX][2] CTA-level (M, L)
    uint64_t* full = reinterpret_cast<uint64_t*>(c_ml + GMAX * 2);
    uint64_t* empty = full + ATT_STAGES;
    int* s_last = reinterpret_cast<int*>(empty + ATT_STAGES);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int sp = blockIdx.x, kvh = blockIdx.y, m = blockIdx.z;
    const int G = a.n_heads / a.n_kv_heads;

    if (tid == 0) {
        for (int s = 0; s < ATT_STAGES; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], ATT_WARPS);
        }
        mbar_fence_init();
    }
    __syncthreads();
    pdl_launch_dependents();
    pdl_wait();     // q, pos, block tables and the KV cache all come from earlier kernels
    if (a.row_skip != nullptr && a.row_skip[m] != 0) { trace_end(a.tr); return; }      // uniform for the CTA

    const int T = a.pos[m] + 1;                                // attend to positions 0..pos
    const int n_pages = (T + ATT_PAGE - 1) / ATT_PAGE;
    // The grid carries a.n_splits CTAs per (row, kv head) -- sized for the longest context the engine allows --
    // but the split + merge round trip (scratch, counter, last-CTA merge) costs about as much as streaming 12
    // pages, so a row only uses as many splits as its OWN context justifies; the other CTAs leave at once.
    // (measured, 8B decode: ~170-token context 574 tok/s with 4 splits, 603 with 1; 4096-token context 434 tok/s
    // with 18 splits of 7 pages, 454 with 16 of 8)
    const int n_eff = (n_pages <= ATT_MIN_SPLIT_PAGES) ? 1 : min(a.n_splits, (n_pages + 7) / 8);
    if (sp >= n_eff) { trace_end(a.tr); return; }
    const int pps = (n_pages + n_eff - 1) / n_eff;             // pages per split
    const int pg0 = sp * pps;
    const int pg1 = min(n_pages, pg0 + pps);
    const int np = max(0, pg1 - pg0);
    const int* bt = a.block_table + (size_t)a.slot[m] * a.max_pages;

    bool alive = true;                                         // no wait was given up
    if (warp == ATT_WARPS) {
        // producer warp: the 32 lanes fetch 32 block-table entries at once (one load latency instead of one per
        // page in front of every copy), lane 0 issues the bulk copies
        for (int i0 = 0; i0 < np; i0 += 32) {
            const int my_page = (i0 + lane < np) ? bt[pg0 + i0 + lane] : 0;
            const int cnt = min(32, np - i0);
            for (int j = 0; j < cnt; j++) {
                const int page = __shfl_sync(0xffffffffu, my_page, j);
                if (lane == 0) {
                    const int i = i0 + j;
                    const int s = i % ATT_STAGES;
                    if (i >= ATT_STAGES) alive = alive && wait_phase(&empty[s], ((i / ATT_STAGES) & 1) ^ 1, limit, true) && limit.ns != 0;      // (no time: tests)
                    const size_t poff = ((size_t)page * a.n_kv_heads + kvh) * (size_t)PAGE_BYTES;
                    if (alive) {
                        mbar_arrive_expect_tx(&full[s], 2 * PAGE_BYTES);
                        bulk_g2s(ring + (s * 2 + 0) * PAGE_BYTES, reinterpret_cast<const uint8_t*>(a.k_cache) + poff, PAGE_BYTES, &full[s]);
                        bulk_g2s(ring + (s * 2 + 1) * PAGE_BYTES, reinterpret_cast<const uint8_t*>(a.v_cache) + poff, PAGE_BYTES, &full[s]);
                    }
                }
                __syncwarp();
            }
        }
    } else {
        // stage q (pre-scaled by 1/sqrt(HS)); heads >= G are zero
        const float scale = rsqrtf((float)HS);
        for (int i = tid; i < GMAX * HS; i += ATT_WARPS * 32) {
            const int h = i / HS, d = i % HS;
            q_s[i] = (h < G) ? a.q[(size_t)m * a.n_heads * HS + (size_t)(kvh * G + h) * HS + d] * scale : 0.0f;
        }
        asm volatile("bar.sync 1, %0;" ::"n"(ATT_WARPS * 32));

        // running state: lane i owns (m, l) of head (i & 3) of each chunk (replicated over 8 lanes)
        float run_m[NCH], run_l[NCH], acc[NCH][4][DPL];
#pragma unroll
        for (int c = 0; c < NCH; c++) {
            run_m[c] = -INFINITY;
            run_l[c] = 0.0f;
#pragma unroll
            for (int h = 0; h < 4; h++)
#pragma unroll
                for (int d = 0; d < DPL; d++) acc[c][h][d] = 0.0f;
        }
        const int hsel = lane & 3, jsel = lane >> 2;

        for (int i = 0; i < np; i++) {
            const int s = i % ATT_STAGES;
            alive = alive && wait_phase(&full[s], (i / ATT_STAGES) & 1, limit, true);
            const KV* Kp = reinterpret_cast<const KV*>(ring + (s * 2 + 0) * PAGE_BYTES);
            const KV* Vp = reinterpret_cast<const KV*>(ring + (s * 2 + 1) * PAGE_BYTES);
            const int ntok = min(ATT_PAGE, T - (pg0 + i) * ATT_PAGE);   // valid tokens in this page
#pragma unroll
            for (int c = 0; c < NCH; c++) {
                float qv[4][DPL];
#pragma unroll
                for (int h = 0; h < 4; h++)
#pragma unroll
                    for (int d = 0; d < DPL; d++) qv[h][d] = q_s[(c * 4 + h) * HS + lane * DPL + d];
                float sc[32];
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const int t = warp * 8 + j;
                    float kf[DPL];
#pragma unroll
                    for (int d = 0; d < DPL; d++) kf[d] = kv_to_float<KV>(Kp[t * HS + lane * DPL + d]);
#pragma unroll
                    for (int h = 0; h < 4; h++) {
                        float x = 0.0f;
#pragma unroll
                        for (int d = 0; d < DPL; d++) x += qv[h][d] * kf[d];
                        sc[j * 4 + h] = x;
                    }
                }
                float sv = warp_transpose_reduce32(sc, lane);      // score of (token jsel, head hsel)
                const bool valid = (warp * 8 + jsel < ntok) && (c * 4 + hsel < G);
                sv = valid ? sv : -INFINITY;
                float mx = sv;
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
                const float m_new = fmaxf(run_m[c], mx);
                const float m_use = (m_new == -INFINITY) ? 0.0f : m_new;
                const float corr = __expf(run_m[c] - m_use);       // run_m = -inf -> 0
                const float p = valid ? __expf(sv - m_use) : 0.0f;
                float ps = p;
                ps += __shfl_xor_sync(0xffffffffu, ps, 4);
                ps += __shfl_xor_sync(0xffffffffu, ps, 8);
                ps += __shfl_xor_sync(0xffffffffu, ps, 16);
                run_l[c] = run_l[c] * corr + ps;
                run_m[c] = m_new;
#pragma unroll
                for (int h = 0; h < 4; h++) {
                    const float ch = __shfl_sync(0xffffffffu, corr, h);
#pragma unroll
                    for (int d = 0; d < DPL; d++) acc[c][h][d] *= ch;
                }
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const int t = warp * 8 + j;
                    float vf[DPL];
#pragma unroll
                    for (int d = 0; d < DPL; d++) vf[d] = (t < ntok) ? kv_to_float<KV>(Vp[t * HS + lane * DPL + d]) : 0.0f;
#pragma unroll
                    for (int h = 0; h < 4; h++) {
                        const float ph = __shfl_sync(0xffffffffu, p, j * 4 + h);
#pragma unroll
                        for (int d = 0; d < DPL; d++) acc[c][h][d] += ph * vf[d];
                    }
                }
            }
            __syncwarp();
            if (lane == 0 && alive) mbar_arrive(&empty[s]);
        }
        // per-warp partials -> smem
#pragma unroll
        for (int c = 0; c < NCH; c++) {
            if (!alive) {
                run_m[c] = 0.0f;
                run_l[c] = 1.0f;
#pragma unroll
                for (int h = 0; h < 4; h++)
#pragma unroll
                    for (int d = 0; d < DPL; d++) acc[c][h][d] = __int_as_float(0x7fffffff);
            }
#pragma unroll
            for (int h = 0; h < 4; h++)
#pragma unroll
                for (int d = 0; d < DPL; d++) w_acc[(warp * GMAX + c * 4 + h) * HS + lane * DPL + d] = acc[c][h][d];
            if (lane < 4) {
                w_ml[(warp * GMAX + c * 4 + lane) * 2 + 0] = run_m[c];
                w_ml[(warp * GMAX + c * 4 + lane) * 2 + 1] = run_l[c];
            }
        }
    }
    if (!alive) wait_settle();
    __syncthreads();

    // CTA-level merge of the 4 warps: thread d < HS owns head dim d
    const bool single = (n_eff == 1);
    if (tid < HS) {
        for (int h = 0; h < G; h++) {
            float Mx = -INFINITY;
            for (int w = 0; w < ATT_WARPS; w++) Mx = fmaxf(Mx, w_ml[(w * GMAX + h) * 2]);
            const float Mu = (Mx == -INFINITY) ? 0.0f : Mx;
            float L = 0.0f, O = 0.0f;
            for (int w = 0; w < ATT_WARPS; w++) {
                const float e = __expf(w_ml[(w * GMAX + h) * 2] - Mu);
                L += w_ml[(w * GMAX + h) * 2 + 1] * e;
                O += w_acc[(w * GMAX + h) * HS + tid] * e;
            }
            const int head = kvh * G + h;
            if (single) {
                const float y = (L > 0.0f) ? O / L : 0.0f;
                if (a.y_out != nullptr) a.y_out[(size_t)m * a.n_heads * HS + (size_t)head * HS + tid] = y;
                if (a.xq_out != nullptr || a.xh_out != nullptr)
                    q80_block_store(y, lane, m, (head * HS + tid) >> 5, a.out_mcap, a.xq_out, a.xh_out);
            } else {
                const size_t pidx = ((size_t)m * a.n_heads + head) * a.n_splits + sp;
                a.part_o[pidx * HS + tid] = O;
                if (tid == 0) {
                    a.part_ml[pidx * 2 + 0] = Mx;
                    a.part_ml[pidx * 2 + 1] = L;
                }
            }
        }
    }
    if (single) { trace_end(a.tr); return; }

    // last CTA of this (row, kv head) merges the splits
    __threadfence();
    __syncthreads();
    if (tid == 0) {
        const unsigned prev = atomicAdd(&a.counters[m * a.n_kv_heads + kvh], 1u);
        *s_last = (prev == (unsigned)n_eff - 1u) ? 1 : 0;
        if (*s_last) a.counters[m * a.n_kv_heads + kvh] = 0u;
    }
    __syncthreads();
    if (!*s_last) { trace_end(a.tr); return; }
    __threadfence();
    // merge: warp w takes heads w, w+4, ...; lane s holds split s's (max, sum) so the rescale factors come out of
    // two warp reductions, then every lane sums its head dims over the splits (independent loads, one latency)
    if (warp < ATT_WARPS) {
        for (int h = warp; h < G; h += ATT_WARPS) {
            const int head = kvh * G + h;
            const size_t base = ((size_t)m * a.n_heads + head) * a.n_splits;
            float ms = -INFINITY, ls = 0.0f;
            if (lane < n_eff) {
                ms = __ldcg(&a.part_ml[(base + lane) * 2]);
                ls = __ldcg(&a.part_ml[(base + lane) * 2 + 1]);
            }
            const float Mx = warp_max(ms);
            const float Mu = (Mx == -INFINITY) ? 0.0f : Mx;
            const float e = (lane < n_eff) ? __expf(ms - Mu) : 0.0f;
            const float L = warp_sum(ls * e);
            float O[DPL];
#pragma unroll
            for (int d = 0; d < DPL; d++) O[d] = 0.0f;
            for (int s2 = 0; s2 < n_eff; s2++) {
                const float es = __shfl_sync(0xffffffffu, e, s2);
#pragma unroll
                for (int d = 0; d < DPL; d++) O[d] += __ldcg(&a.part_o[(base + s2) * HS + lane * DPL + d]) * es;
            }
            const float inv = (L > 0.0f) ? 1.0f / L : 0.0f;
#pragma unroll
            for (int d = 0; d < DPL; d++) w_acc[h * HS + lane * DPL + d] = O[d] * inv;
        }
        asm volatile("bar.sync 1, %0;" ::"n"(ATT_WARPS * 32));
        if (tid < HS) {
            for (int h = 0; h < G; h++) {
                const int head = kvh * G + h;
                const float y = w_acc[h * HS + tid];
                if (a.y_out != nullptr) a.y_out[(size_t)m * a.n_heads * HS + (size_t)head * HS + tid] = y;
                if (a.xq_out != nullptr || a.xh_out != nullptr)
                    q80_block_store(y, lane, m, (head * HS + tid) >> 5, a.out_mcap, a.xq_out, a.xh_out);
            }
        }
    }
    trace_end(a.tr);
}

// ------------------------------------------------------------------------------------------------
// fp16 caches, head sizes 64 / 128, up to four query heads per key/value head: the same job on mma.sync.
//
// What bounds it: the cache's bytes.  The FMA kernel above spends ~480 instructions per 8 tokens and warp (a 31-shuffle
// reduction of the scores, four f32 conversions and shuffled weights per token) and keeps 7 warps per SM busy: 91 us at 32 rows
// of 1500 to 3000 tokens (8 kv heads of 128), 3.3 TB/s.  Here a warp takes 16 tokens at a time through 32 MMAs: 53 us,
// 5.6 TB/s, and the distance to a 64-bit result went from 4.4e-7 to 1.9e-7.
//
// Nothing is rounded to 16 bits: keys and values ARE fp16, and an f32 query (or softmax weight) is taken as three fp16 numbers,
// q = q1 + 2^-7 q2 + 2^-14 q3, of 8 bits each.  The second and third hold the remainders at a scale of their own, so that they do not fall into
// fp16's subnormals ahead of the first: the sum is exact from 2^-15 of the scaled value on and off by 2^-39 at most below, 2^-45 of a score per
// unit of key and 2^-54 of the largest weight.  One 16-row MMA tile holds the parts of all four heads -- row h: q1 of head h,
// row 4 + h: q2, row 12 + h: q3 -- so the three products cost no extra instruction, and summing three accumulator rows, the small ones first,
// gives the f32 product.  An MMA truncates what it adds.  So parts have 8 bits and not the 11 that fp16 holds: a product with an fp16 number
// then has 19, and a sum of 16 of them loses little or nothing; and chains are short: a quarter of K for a score (two MMAs at most), the
// quarters added in pairs in f32, and 16 tokens for an output.  32 heads of 128 on 8, against 64 bits, the FMA kernel / parts of 11 bits /
// this one: up to 40 tokens 1.26e-7 / 1.30e-7 / 1.19e-7, up to 400 2.06e-7 / 1.66e-7 / 1.54e-7, up to 3000 3.34e-7 / 1.95e-7 / 1.84e-7; 32 rows of 1500 to
// 3000 tokens 54.1 us with parts of 11 bits, 53.2 now.
//
// A warp walks its own 16-token half pages (w, w + 4, ...) through a private ring of cp.async stages, chunks of 16 bytes
// XOR-swizzled by the token so ldmatrix is free of conflicts: no barrier between warps until the final merge.  Tokens past the
// context are zero-filled.  Where an infinity or NaN shows up in a warp's sums (an fp16 cache overflowed: inf - inf between
// splits is not what an f32 product gives) the warp takes its tokens again in plain f32.
// ------------------------------------------------------------------------------------------------
#define AM_TOK 16
#define AM_Q_UP 64.0f                     // 2^6 on the queries: fp16 holds them up to 8000 (beyond, an infinity: the plain f32 form)
#define AM_P_UP 32768.0f                  // 2^15 on the weights, as high as fp16 goes (a factor: added to the exponent ahead of exp2 it rounds the difference)
#define AM_PART 0x1p-7f                   // from one part to the next

DL_DEVINL void am_cp16(uint32_t dst, const void* src, bool live) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(live ? 16 : 0) : "memory");
}
DL_DEVINL void am_ldm(uint32_t (&r)[4], uint32_t a) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
DL_DEVINL void am_ldm_trans(uint32_t (&r)[4], uint32_t a) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
DL_DEVINL void am_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
DL_DEVINL float am_exp2(float x) { float r; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
DL_DEVINL uint32_t am_pack(__half a, __half b) { __half2 h = __halves2half2(a, b); return *reinterpret_cast<uint32_t*>(&h); }
// the fp16 parts of v0 and v1 that this lane's rows hold: row g (first part for g < 4, second for g >= 4) and row g + 8 (none / third)
DL_DEVINL float am_top8(float v) { return __uint_as_float(__float_as_uint(v) & 0xFFFF0000u); }      // 8 significant bits
DL_DEVINL void am_split(float v0, float v1, bool lower, uint32_t& top, uint32_t& bot) {
    const uint32_t h1 = am_pack(__float2half_rn(am_top8(v0)), __float2half_rn(am_top8(v1)));
    const float2 f1 = __half22float2(*reinterpret_cast<const __half2*>(&h1));
    const float r0 = (v0 - f1.x) * (1.f / AM_PART), r1 = (v1 - f1.y) * (1.f / AM_PART);
    const uint32_t h2 = am_pack(__float2half_rn(am_top8(r0)), __float2half_rn(am_top8(r1)));
    const float2 f2 = __half22float2(*reinterpret_cast<const __half2*>(&h2));
    const uint32_t h3 = am_pack(__float2half_rn((r0 - f2.x) * (1.f / AM_PART)), __float2half_rn((r1 - f2.y) * (1.f / AM_PART)));
    top = lower ? h1 : h2;
    bot = lower ? 0u : h3;
}

template <int HS, int ST>             // ST: ring stages (16 tokens) per warp
__global__ void __launch_bounds__(ATT_WARPS * 32, 3) attention_mma_kernel(const __grid_constant__ AttArgs a) {
    constexpr int ROWB = HS * 2, CH = ROWB / 16;               // bytes / 16-byte chunks of a token's line
    constexpr int HALF = AM_TOK * ROWB;                        // K (or V) of a half page
    constexpr int KS = HS / 16, NT = HS / 8;
    extern __shared__ __align__(128) uint8_t smem[];
    trace_begin(a.tr);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int sp = blockIdx.x, kvh = blockIdx.y, m = blockIdx.z;
    const int G = a.n_heads / a.n_kv_heads;
    pdl_launch_dependents();
    pdl_wait();     // q, pos, block tables and the KV cache all come from earlier kernels
    if (a.row_skip != nullptr && a.row_skip[m] != 0) { trace_end(a.tr); return; }      // uniform for the CTA
    const int T = a.pos[m] + 1;
    const int n_pages = (T + ATT_PAGE - 1) / ATT_PAGE;
    const int n_eff = (n_pages <= ATT_MIN_SPLIT_PAGES) ? 1 : min(a.n_splits, (n_pages + 7) / 8);      // as in attention_kernel
    if (sp >= n_eff) { trace_end(a.tr); return; }
    const int pps = (n_pages + n_eff - 1) / n_eff;
    const int pg0 = sp * pps, pg1 = min(n_pages, pg0 + pps);
    const int t_end = min(T, pg1 * ATT_PAGE);
    const int n_hp = max(0, (t_end - pg0 * ATT_PAGE + AM_TOK - 1) / AM_TOK);       // half pages of this CTA; warp w takes w, w + 4, ...
    const int* bt = a.block_table + (size_t)a.slot[m] * a.max_pages;
    const int n_my = (n_hp - warp + ATT_WARPS - 1) / ATT_WARPS;

    float* w_acc = reinterpret_cast<float*>(smem);             // [WARPS][4][HS], after the ring is done with
    float* w_ml = w_acc + ATT_WARPS * 4 * HS;                  // [WARPS][4][2]
    int* s_last = reinterpret_cast<int*>(w_ml + ATT_WARPS * 4 * 2);
    const uint32_t ring = smem_u32(smem) + warp * (ST * 2 * HALF);
    const int g = lane >> 2, qd = lane & 3, head = g & 3;
    const bool lower = g < 4;

    float2 qr[KS][2];
    {
        const float* q = a.q + (size_t)m * a.n_heads * HS + (size_t)(kvh * G + (head < G ? head : 0)) * HS + qd * 2;
#pragma unroll
        for (int k = 0; k < KS; ++k)
#pragma unroll
            for (int u = 0; u < 2; ++u) qr[k][u] = *reinterpret_cast<const float2*>(q + k * 16 + u * 8);
    }
    // this warp's half page i: page pg0 + (w + 4 i) / 2; the lanes hold the next 32 page numbers
    auto page_at = [&](int i) { const int p = pg0 + ((warp + ATT_WARPS * i) >> 1); return i < n_my ? bt[p] : 0; };
    int my_page = page_at(lane);
    const uint8_t* kc = reinterpret_cast<const uint8_t*>(a.k_cache);
    const uint8_t* vc = reinterpret_cast<const uint8_t*>(a.v_cache);
    auto load = [&](int i, int st, int page) {
        const int hp = warp + ATT_WARPS * i;
        const int left = t_end - pg0 * ATT_PAGE - hp * AM_TOK;           // live tokens from this half page on
        const size_t off = (((size_t)page * a.n_kv_heads + kvh) * ATT_PAGE + (hp & 1) * AM_TOK) * (size_t)ROWB;
        const uint32_t dst = ring + st * (2 * HALF);
#pragma unroll
        for (int j = 0; j < AM_TOK * CH / 32; ++j) {
            const int idx = j * 32 + lane, t = idx / CH, c = idx % CH;
            const uint32_t d = dst + t * ROWB + ((c ^ (t & 7)) << 4);
            am_cp16(d, kc + off + (size_t)idx * 16, t < left);
            am_cp16(d + HALF, vc + off + (size_t)idx * 16, t < left);
        }
    };

#pragma unroll
    for (int i = 0; i < ST - 1; ++i) {
        const int page = __shfl_sync(0xffffffffu, my_page, i);
        if (i < n_my) load(i, i, page);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    // queries: three fp16 parts per head in the A fragments, pre-scaled by log2(e) / sqrt(HS) and 2^6
    uint32_t qf[KS][4];
    const float scale = rsqrtf((float)HS) * 1.44269504088896341f * AM_Q_UP;
#pragma unroll
    for (int k = 0; k < KS; ++k)
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            am_split(head < G ? qr[k][u].x * scale : 0.f, head < G ? qr[k][u].y * scale : 0.f, lower, qf[k][2 * u], qf[k][2 * u + 1]);
        }
    float o[NT][4];
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[n][e] = 0.f;
    float run_m = -INFINITY, run_l = 0.f;                      // of head g % 4; run_l: this lane's own tokens
    const float s_up = (lower ? 1.f : AM_PART) / AM_Q_UP;      // row g's part of a score

    int st = 0;
    for (int i = 0; i < n_my; ++i) {
        {
            const int nx = i + ST - 1;
            if ((nx & 31) == 0) my_page = page_at(nx + lane);
            const int page = __shfl_sync(0xffffffffu, my_page, nx & 31);
            if (nx < n_my) load(nx, st == 0 ? ST - 1 : st - 1, page);
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
        asm volatile("cp.async.wait_group %0;" ::"n"(ST - 1) : "memory");
        __syncwarp();
        const uint32_t kb = ring + st * (2 * HALF), vb = kb + HALF;
        // scores of 16 tokens: n-tile j = tokens 8 j ..; quarters of K, added in pairs
        float c[2][4];
        {
            const int t = (lane & 7) + ((lane >> 4) << 3), c1 = (lane >> 3) & 1;
            const uint32_t base = kb + t * ROWB;
            float x[2][2][4];
#pragma unroll
            for (int k = 0; k < KS; ++k) {
                const int u = k / (KS / 4);                    // quarter
                if (k % (KS / 4) == 0) {
#pragma unroll
                    for (int j = 0; j < 2; ++j)
#pragma unroll
                        for (int e = 0; e < 4; ++e) x[u & 1][j][e] = 0.f;
                }
                uint32_t b[4];
                am_ldm(b, base + (((2 * k + c1) ^ (t & 7)) << 4));
                am_mma(x[u & 1][0], qf[k][0], qf[k][1], qf[k][2], qf[k][3], b[0], b[1]);
                am_mma(x[u & 1][1], qf[k][0], qf[k][1], qf[k][2], qf[k][3], b[2], b[3]);
                if (k == KS / 2 - 1 || k == KS - 1) {
#pragma unroll
                    for (int j = 0; j < 2; ++j)
#pragma unroll
                        for (int e = 0; e < 4; ++e) c[j][e] = k < KS / 2 ? x[0][j][e] + x[1][j][e] : c[j][e] + (x[0][j][e] + x[1][j][e]);
                }
            }
        }
        const int left = t_end - pg0 * ATT_PAGE - (warp + ATT_WARPS * i) * AM_TOK;
        float s[4];
        float mx = -INFINITY;
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                float v = fmaf(c[j][e + 2], AM_PART * AM_PART / AM_Q_UP, c[j][e] * s_up);     // rows g and g + 8
                v += __shfl_xor_sync(0xffffffffu, v, 16);                                     // row g +- 4
                v = (j * 8 + qd * 2 + e < left) ? v : -INFINITY;
                s[j * 2 + e] = v;
                mx = fmaxf(mx, v);
            }
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
        const float m_new = fmaxf(run_m, mx), m_use = m_new == -INFINITY ? 0.f : m_new;
        const float corr = am_exp2(run_m - m_use);
        run_m = m_new;
        uint32_t pa[4];
        float ps = 0.f;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const float p0 = am_exp2(s[2 * j] - m_use) * AM_P_UP, p1 = am_exp2(s[2 * j + 1] - m_use) * AM_P_UP;
            ps += p0 + p1;
            am_split(p0, p1, lower, pa[2 * j], pa[2 * j + 1]);
        }
        run_l = fmaf(run_l, corr, ps);
        {
            const int t = (lane & 7) + (((lane >> 3) & 1) << 3), c1 = lane >> 4;
            const uint32_t base = vb + t * ROWB;
#pragma unroll
            for (int n = 0; n < NT; n += 2) {
                uint32_t b[4];
                am_ldm_trans(b, base + (((n + c1) ^ (t & 7)) << 4));
                float x[4] = {0.f, 0.f, 0.f, 0.f}, y[4] = {0.f, 0.f, 0.f, 0.f};
                am_mma(x, pa[0], pa[1], pa[2], pa[3], b[0], b[1]);
                am_mma(y, pa[0], pa[1], pa[2], pa[3], b[2], b[3]);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    o[n][e] = fmaf(o[n][e], corr, x[e]);
                    o[n + 1][e] = fmaf(o[n + 1][e], corr, y[e]);
                }
            }
        }
        __syncwarp();
        st = st == ST - 1 ? 0 : st + 1;
    }
    run_l += __shfl_xor_sync(0xffffffffu, run_l, 1);
    run_l += __shfl_xor_sync(0xffffffffu, run_l, 2);
    // 2^-7 row 4 + h + 2^-14 row 12 + h, then row h: lanes of g < 4 hold head g
    bool bad = !(fabsf(run_l) < INFINITY);
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            float v = fmaf(o[n][e + 2], AM_PART * AM_PART, lower ? o[n][e] : o[n][e] * AM_PART);
            v += __shfl_xor_sync(0xffffffffu, v, 16);
            o[n][e] = v;
            bad |= !(fabsf(v) < INFINITY);
        }
    bad = __any_sync(0xffffffffu, bad);
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();                                           // the ring is done with
    if (!bad) {
        if (lower) {
            float* w = w_acc + (warp * 4 + g) * HS + qd * 2;
#pragma unroll
            for (int n = 0; n < NT; ++n) *reinterpret_cast<float2*>(w + n * 8) = make_float2(o[n][0], o[n][1]);
            if (qd == 0) { w_ml[(warp * 4 + g) * 2] = run_m; w_ml[(warp * 4 + g) * 2 + 1] = run_l; }
        }
    } else {
        // infinities or NaN among this warp's tokens: plain f32, one head at a time, lanes along the head's dimensions
        constexpr int DPL = HS / 32;
        const float scale = rsqrtf((float)HS) * 1.44269504088896341f;
        for (int h = 0; h < G; ++h) {
            float q[DPL], acc[DPL], M = -INFINITY, Ls = 0.f;
#pragma unroll
            for (int d = 0; d < DPL; ++d) { q[d] = a.q[((size_t)m * a.n_heads + kvh * G + h) * HS + lane * DPL + d] * scale; acc[d] = 0.f; }
            for (int i = 0; i < n_my; ++i) {
                const int hp = warp + ATT_WARPS * i, page = bt[pg0 + (hp >> 1)];
                const int n_tok = min(AM_TOK, t_end - pg0 * ATT_PAGE - hp * AM_TOK);
                for (int t = 0; t < n_tok; ++t) {
                    const size_t at = (((size_t)page * a.n_kv_heads + kvh) * ATT_PAGE + (hp & 1) * AM_TOK + t) * HS + lane * DPL;
                    float v = 0.f;
#pragma unroll
                    for (int d = 0; d < DPL; ++d) v = fmaf(q[d], __half2float(reinterpret_cast<const __half*>(a.k_cache)[at + d]), v);
                    v = warp_sum(v);
                    const float mn = fmaxf(M, v), mu = mn == -INFINITY ? 0.f : mn;
                    const float cr = am_exp2(M - mu), p = am_exp2(v - mu) * AM_P_UP;
                    M = mn;
                    Ls = fmaf(Ls, cr, p);
#pragma unroll
                    for (int d = 0; d < DPL; ++d) acc[d] = fmaf(acc[d], cr, p * __half2float(reinterpret_cast<const __half*>(a.v_cache)[at + d]));
                }
            }
#pragma unroll
            for (int d = 0; d < DPL; ++d) w_acc[(warp * 4 + h) * HS + lane * DPL + d] = acc[d];
            if (lane == 0) { w_ml[(warp * 4 + h) * 2] = M; w_ml[(warp * 4 + h) * 2 + 1] = Ls; }
        }
    }
    __syncthreads();

    // the four warps' shares: thread d < HS owns head dim d (maxima are in units of log2)
    const bool single = (n_eff == 1);
    if (tid < HS) {
        for (int h = 0; h < G; h++) {
            float Mx = -INFINITY;
#pragma unroll
            for (int w = 0; w < ATT_WARPS; w++) Mx = fmaxf(Mx, w_ml[(w * 4 + h) * 2]);
            const float Mu = (Mx == -INFINITY) ? 0.0f : Mx;
            float Ls = 0.0f, O = 0.0f;
#pragma unroll
            for (int w = 0; w < ATT_WARPS; w++) {
                const float e = am_exp2(w_ml[(w * 4 + h) * 2] - Mu);
                Ls += w_ml[(w * 4 + h) * 2 + 1] * e;
                O += w_acc[(w * 4 + h) * HS + tid] * e;
            }
            const int hd = kvh * G + h;
            if (single) {
                const float y = (Ls > 0.0f) ? O / Ls : 0.0f;
                if (a.y_out != nullptr) a.y_out[(size_t)m * a.n_heads * HS + (size_t)hd * HS + tid] = y;
                if (a.xq_out != nullptr || a.xh_out != nullptr) q80_block_store(y, lane, m, (hd * HS + tid) >> 5, a.out_mcap, a.xq_out, a.xh_out);
            } else {
                const size_t pidx = ((size_t)m * a.n_heads + hd) * a.n_splits + sp;
                a.part_o[pidx * HS + tid] = O;
                if (tid == 0) { a.part_ml[pidx * 2] = Mx; a.part_ml[pidx * 2 + 1] = Ls; }
            }
        }
    }
    if (single) { trace_end(a.tr); return; }
    __threadfence();
    __syncthreads();
    if (tid == 0) {
        const unsigned prev = atomicAdd(&a.counters[m * a.n_kv_heads + kvh], 1u);
        *s_last = (prev == (unsigned)n_eff - 1u) ? 1 : 0;
        if (*s_last) a.counters[m * a.n_kv_heads + kvh] = 0u;
    }
    __syncthreads();
    if (!*s_last) { trace_end(a.tr); return; }
    __threadfence();
    // warp h merges head h: lane s holds split s's (max, sum), every lane sums its dims over the splits
    if (warp < G) {
        constexpr int DPL = HS / 32;
        const int hd = kvh * G + warp;
        const size_t base = ((size_t)m * a.n_heads + hd) * a.n_splits;
        float ms = -INFINITY, ls = 0.0f;
        if (lane < n_eff) { ms = __ldcg(&a.part_ml[(base + lane) * 2]); ls = __ldcg(&a.part_ml[(base + lane) * 2 + 1]); }
        const float Mx = warp_max(ms);
        const float Mu = (Mx == -INFINITY) ? 0.0f : Mx;
        const float e = (lane < n_eff) ? am_exp2(ms - Mu) : 0.0f;
        const float Ls = warp_sum(ls * e);
        float O[DPL];
#pragma unroll
        for (int d = 0; d < DPL; d++) O[d] = 0.0f;
#pragma unroll 4
        for (int s2 = 0; s2 < n_eff; s2++) {
            const float es = __shfl_sync(0xffffffffu, e, s2);
#pragma unroll
            for (int d = 0; d < DPL; d++) O[d] += __ldcg(&a.part_o[(base + s2) * HS + d * 32 + lane]) * es;
        }
        const float inv = (Ls > 0.0f) ? 1.0f / Ls : 0.0f;
#pragma unroll
        for (int d = 0; d < DPL; d++) {          // 32 dims at a time: one Q80 block
            const float y = O[d] * inv;
            if (a.y_out != nullptr) a.y_out[(size_t)m * a.n_heads * HS + (size_t)hd * HS + d * 32 + lane] = y;
            if (a.xq_out != nullptr || a.xh_out != nullptr) q80_block_store(y, lane, m, (hd * HS) / 32 + d, a.out_mcap, a.xq_out, a.xh_out);
        }
    }
    trace_end(a.tr);
}

extern void dl_set_error(const char* fmt, ...);

static size_t att_smem_bytes(int HS, int NCH, int esize) {
    const int GMAX = NCH * 4;
    return (size_t)ATT_STAGES * 2 * ATT_PAGE * HS * esize + (size_t)GMAX * HS * 4 + (size_t)ATT_WARPS * GMAX * HS * 4 +
           (size_t)ATT_WARPS * GMAX * 2 * 4 + (size_t)GMAX * 2 * 4 + 2 * ATT_STAGES * 8 + 16;
}

template <int HS, int NCH, typename KV>
static int launch_att(const AttArgs& a, int pdl, cudaStream_t stream) {
    WaitLimit limit;
    if (dl_wait_limit("dl_attention", &limit) != 0) return -1;
    const size_t smem = att_smem_bytes(HS, NCH, (int)sizeof(KV));
    static SmemLimit given;
    if (const int rc = dl_smem_limit("attention", attention_kernel<HS, NCH, KV>, smem, given)) return rc;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(a.n_splits, a.n_kv_heads, a.M);
    cfg.blockDim = dim3(ATT_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    if (pdl) {
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
    }
    cudaError_t e = cudaLaunchKernelEx(&cfg, attention_kernel<HS, NCH, KV>, a, limit);
    if (e != cudaSuccess) { dl_set_error("attention launch: %s", cudaGetErrorString(e)); return -(int)e; }
    return 0;
}

template <int HS, int ST>
static int launch_att_mma_st(const AttArgs& a, int pdl, cudaStream_t stream) {
    constexpr int smem = ATT_WARPS * ST * AM_TOK * HS * 4;
    static_assert(ATT_WARPS * 4 * (HS + 2) * 4 + 4 <= smem, "the merge fits the ring");
    static SmemLimit given;
    if (const int rc = dl_smem_limit("attention", attention_mma_kernel<HS, ST>, smem, given)) return rc;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(a.n_splits, a.n_kv_heads, a.M);
    cfg.blockDim = dim3(ATT_WARPS * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    if (pdl) {
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
    }
    cudaError_t e = cudaLaunchKernelEx(&cfg, attention_mma_kernel<HS, ST>, a);
    if (e != cudaSuccess) { dl_set_error("attention launch: %s", cudaGetErrorString(e)); return -(int)e; }
    return 0;
}

// Stages by how many CTAs an SM gets, for heads of 128: 64 KB of rings where three share it, 96 for two and 128 for one, so that as much is on its way (us with
// two stages and so: 16 rows of 1500 to 3000 tokens 38.9 and 35.4, 8 rows 25.1 and 23.9, 32 rows, two CTAs, 55.2 and 55.0; a step of width 4096 and 4 layers
// behind 200 to 400 tokens, 8 rows 320.6 and 313.0, 32 rows 356 and 352).  With CTAs for half the SMs or fewer a warp has two or three stages in all, and the
// larger ring only keeps the next kernel's CTAs out (one row 211.4 and 212.9); heads of 64 gain nothing.
template <int HS>
static int launch_att_mma(const AttArgs& a, int pdl, cudaStream_t stream) {
    if constexpr (HS == 128) {
        const long long ctas = (long long)a.n_splits * a.n_kv_heads * a.M;
        const int n_sms = dl_device_sm_count();
        if (ctas > n_sms / 2 && ctas <= n_sms) return launch_att_mma_st<HS, 4>(a, pdl, stream);
        if (ctas > n_sms && ctas <= 2ll * n_sms) return launch_att_mma_st<HS, 3>(a, pdl, stream);
    }
    return launch_att_mma_st<HS, 256 / HS>(a, pdl, stream);
}

template <int HS, typename KV>
static int launch_att_nch(const AttArgs& a, int G, int pdl, cudaStream_t stream) {
    if (G <= 4) return launch_att<HS, 1, KV>(a, pdl, stream);
    if (G <= 8) return launch_att<HS, 2, KV>(a, pdl, stream);
    return launch_att<HS, 4, KV>(a, pdl, stream);
}

extern "C" long long dl_attention_scratch_bytes(int M, int n_heads, int head_size, int max_splits) {
    long long o = (long long)M * n_heads * max_splits * head_size * 4;
    long long ml = (long long)M * n_heads * max_splits * 2 * 4;
    return ATT_COUNTER_BYTES + ((o + 255) / 256 + (ml + 255) / 256) * 256;
}

extern "C" int dl_attention(const float* q, int M, int n_heads, int n_kv_heads, int head_size, const void* k_cache,
                            const void* v_cache, int kv_f32, const int* pos, const int* slot, const int* block_table,
                            int max_pages, int page_size, int n_splits, void* scratch, uint8_t* xq_out,
                            uint8_t* xh_out, int out_mcap, float* y_out, const int* row_skip, int pdl, void* stream) {
    if (page_size != ATT_PAGE) { dl_set_error("dl_attention: page_size must be %d", ATT_PAGE); return -1; }
    if (n_heads % n_kv_heads != 0 || n_heads / n_kv_heads > 16) { dl_set_error("dl_attention: unsupported head grouping %d/%d", n_heads, n_kv_heads); return -1; }
    if (n_splits < 1) n_splits = 1;
    if (n_splits > 1 && scratch == nullptr) { dl_set_error("dl_attention: n_splits>1 needs scratch"); return -1; }
    AttArgs a;
    a.q = q; a.k_cache = k_cache; a.v_cache = v_cache; a.pos = pos; a.slot = slot; a.block_table = block_table;
    a.row_skip = row_skip;
    a.M = M; a.n_heads = n_heads; a.n_kv_heads = n_kv_heads; a.max_pages = max_pages; a.n_splits = n_splits;
    // the completion counters are only touched by rows that are split
    if (n_splits > 1 && (long long)M * n_kv_heads * 4 > ATT_COUNTER_BYTES) { dl_set_error("dl_attention: M*n_kv_heads too large"); return -1; }
    long long o = ((long long)M * n_heads * n_splits * head_size * 4 + 255) / 256 * 256;
    a.counters = reinterpret_cast<unsigned*>(scratch);
    a.part_o = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(scratch) + ATT_COUNTER_BYTES);
    a.part_ml = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(scratch) + ATT_COUNTER_BYTES + o);
    a.xq_out = xq_out; a.xh_out = xh_out; a.out_mcap = out_mcap; a.y_out = y_out;
    a.tr = dl_trace_next(TR_ATT);
    const int G = n_heads / n_kv_heads;
    cudaStream_t st = (cudaStream_t)stream;
    if (kv_f32) {
        if (head_size == 128) return launch_att_nch<128, float>(a, G, pdl, st);
        if (head_size == 64) return launch_att_nch<64, float>(a, G, pdl, st);
        if (head_size == 32) return launch_att_nch<32, float>(a, G, pdl, st);
    } else {
        // up to four query heads per key/value head fill one MMA tile with their three parts; the queries are read as pairs and the
        // cache in 16-byte pieces (PyTorch's allocations are aligned to 512 bytes, a caller's offset may not be)
        const bool mma = G <= 4 && ((uintptr_t)q & 7) == 0 && (((uintptr_t)k_cache | (uintptr_t)v_cache) & 15) == 0;
        if (head_size == 128) return mma ? launch_att_mma<128>(a, pdl, st) : launch_att_nch<128, __half>(a, G, pdl, st);
        if (head_size == 64) return mma ? launch_att_mma<64>(a, pdl, st) : launch_att_nch<64, __half>(a, G, pdl, st);
        if (head_size == 32) return launch_att_nch<32, __half>(a, G, pdl, st);
    }
    dl_set_error("dl_attention: unsupported head_size %d", head_size);
    return -1;
}
