// Pieces shared by the recurrences with data-dependent gates (gated_scan.cu, delta_scan.cu): how a row's query, key and decay are
// formed, how a sequence is cut into chunks, and the scores inside a chunk under decays per channel.
#pragma once
#include "f32_pairs.cuh"
#include "layer_common.cuh"
#include "../../../include/dllama_b200.h"

#define GC DL_GATED_CHUNK
#define GC_THREADS 256
#define GC_AS 68                  // row stride of the score matrix

enum { GATED_HEAD = 0, GATED_CHANNEL = 1, GATED_AHEAD = 2, GATED_DELTA = 3 };

__device__ __forceinline__ int gated_k_head(const DlGatedArgs& a, int h) { return a.k_heads > 0 ? h / (a.n_heads / a.k_heads) : h; }

__device__ __forceinline__ float gated_q(const DlGatedArgs& a, size_t row, int i) {
    const float v = a.q[row * a.ldq + i];
    if (!a.q_silu) return v * a.q_scale;
    float s, c;
    sigmoid_pair_f(v, s, c);
    return v * s;
}
// what a channel's gate reads besides the row: bias, lower bound, the head's rate
struct GatedChannel { float bias, lower, rate; };
__device__ __forceinline__ GatedChannel gated_channel(const DlGatedArgs& a, int h, int d) {
    GatedChannel c;
    c.bias = a.f_bias ? a.f_bias[h * a.dim + d] : 0.f;
    c.lower = a.gate == DL_GATE_LOWER ? a.lower[h * a.dim + d] : 0.f;
    c.rate = a.gate == DL_GATE_SOFTPLUS ? a.rate[h] : 0.f;
    return c;
}
template <int G> struct GateIs { static constexpr int value = G; };
// decay f from the raw gate z; with DL_GATE_LOWER also the key k
template <int GATE>
__device__ __forceinline__ void gated_form(const DlGatedArgs& a, const GatedChannel& c, float z, float& f, float& k) {
    z += c.bias;
    if (GATE == DL_GATE_LOWER) {
        float s, t;
        sigmoid_pair_f(z, s, t);
        f = fmaf(1.f - c.lower, s, c.lower);
        k = (1.f - c.lower) * t;
    } else {
        f = GATE == DL_GATE_ROOT_SIGMOID ? expf(-softplus_f(-z) * a.inv_tau) : GATE == DL_GATE_EXP_EXP ? expf(-expf(z)) : expf(-c.rate * softplus_f(z));
    }
}
// the same of N rows: the choice is made once, so that the rows' gates are computed side by side
template <int N>
__device__ __forceinline__ void gated_forms(const DlGatedArgs& a, const GatedChannel& c, const float (&z)[N], float (&f)[N], float (&k)[N]) {
    auto form = [&](auto gate) {
#pragma unroll
        for (int r = 0; r < N; ++r) gated_form<decltype(gate)::value>(a, c, z[r], f[r], k[r]);
    };
    if (a.gate == DL_GATE_LOWER) form(GateIs<DL_GATE_LOWER>());
    else if (a.gate == DL_GATE_ROOT_SIGMOID) form(GateIs<DL_GATE_ROOT_SIGMOID>());
    else if (a.gate == DL_GATE_EXP_EXP) form(GateIs<DL_GATE_EXP_EXP>());
    else form(GateIs<DL_GATE_SOFTPLUS>());
}
// decay and key of channel d of head h (its keys are those of head hk)
__device__ __forceinline__ void gated_fk(const DlGatedArgs& a, size_t row, int h, int hk, int d, float& f, float& k) {
    k = a.gate == DL_GATE_LOWER ? 0.f : a.k[row * a.ldk + hk * a.dim + d];
    float z1[1] = {a.f[row * a.ldf + h * a.dim + d]}, f1[1], k1[1] = {k};
    gated_forms(a, gated_channel(a, h, d), z1, f1, k1);
    f = f1[0]; k = k1[0];
}

static inline int gated_args_ok(const DlGatedArgs& a, const char* who) {
    const bool ch = a.f != nullptr;
    if (a.n_heads < 1 || a.dim < 1 || a.vdim < 1 || a.dim > 512) { dl_set_error("%s: bad shape (heads %d, dim %d, vdim %d)", who, a.n_heads, a.dim, a.vdim); return -1; }
    if (ch && a.gate == DL_GATE_LOWER ? (!a.f_bias || !a.lower) : !a.k) { dl_set_error("%s: the gates are incomplete", who); return -1; }
    if (!ch && (!a.log_keep || !a.put || !a.den || !a.n_state)) { dl_set_error("%s: the gates are incomplete", who); return -1; }
    if (ch && ((a.gate == DL_GATE_ROOT_SIGMOID && !(a.inv_tau > 0.f)) || (a.gate == DL_GATE_SOFTPLUS && !a.rate))) { dl_set_error("%s: the gates are incomplete", who); return -1; }
    if ((a.bonus && a.beta) || (!ch && (a.bonus || a.beta || a.k_heads))) { dl_set_error("%s: these forms do not go together", who); return -1; }
    if (a.k_heads < 0 || (a.k_heads > 0 && a.n_heads % a.k_heads)) { dl_set_error("%s: %d heads on %d key heads", who, a.n_heads, a.k_heads); return -1; }
    return 0;
}

struct GatedScratch { float* S; float* dec; float* ns; };

__device__ __forceinline__ bool gated_chunk_of(const DlMambaBatch& b, int n, int c, int& row0, int& len, int& ci) {
    const int s0 = b.seq_start[n], total = b.seq_start[n + 1] - s0;
    if (c * GC >= total) return false;
    row0 = s0 + c * GC;
    len = min(GC, total - c * GC);
    ci = s0 / GC + n + c;
    return true;
}

// the r-th of the eight rows that a warp stages
template <bool PAIRS>
__device__ __forceinline__ int gated_row_of(int warp, int r) { return PAIRS ? 2 * (warp + (r >> 1) * (GC_THREADS / 32)) + (r & 1) : warp + r * (GC_THREADS / 32); }

// V columns c0 .. c0 + VW - 1 (VW: 64 or 128) of the chunk's values into [GC][VW] (zeros beyond the chunk or the head's width); a warp's
// eight rows are in flight together.  PAIRS: rows 2 p and 2 p + 1 of a column side by side, [GC / 2][VW][2], so that two rows are one
// operand of fma2
template <int VW, bool PAIRS = false>
__device__ __forceinline__ void gated_stage_v(const DlGatedArgs& a, const int* rows, int len, int h, int c0, float* vt) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int NRW = GC * 32 / GC_THREADS;
#pragma unroll
    for (int u = 0; u < VW / 32; ++u) {
        const int cc = lane + 32 * u;
        float v[NRW];
#pragma unroll
        for (int r = 0; r < NRW; ++r) {
            const int j = gated_row_of<PAIRS>(warp, r);
            v[r] = (j < len && c0 + cc < a.vdim) ? a.v[(size_t)rows[j] * a.ldv + (size_t)h * a.vdim + c0 + cc] : 0.f;
        }
#pragma unroll
        for (int r = 0; r < NRW; ++r) {
            if (!PAIRS) vt[gated_row_of<false>(warp, r) * VW + cc] = v[r];
            else if (r & 1) *reinterpret_cast<float2*>(vt + (gated_row_of<true>(warp, r - 1) * VW + 2 * cc)) = make_float2(v[r - 1], v[r]);
        }
    }
}

// keys, decays and (Q) queries of a chunk's rows into [GC][ld] each, columns [0, DP4); rows and columns that are not there: k = q = 0,
// f = 1.  COPY: the keys also into Q.  PAIRS: as in gated_stage_v (keys and decays).  A warp's eight rows are in flight together.
template <bool WITH_Q, bool COPY, bool PAIRS = false>
__device__ __forceinline__ void gated_stage_rows(const DlGatedArgs& a, const int* rows, int len, int h, int hk, int DP4, int ld, float* Q, float* K, float* F) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, D = a.dim;
    constexpr int NRW = GC * 32 / GC_THREADS;
    for (int d = lane; d < DP4; d += 32) {
        float q[NRW], k[NRW], z[NRW];
        GatedChannel c = {0.f, 0.f, 0.f};
        if (d < D) c = gated_channel(a, h, d);
#pragma unroll
        for (int r = 0; r < NRW; ++r) {
            const int j = gated_row_of<PAIRS>(warp, r);
            const bool ok = j < len && d < D;
            const size_t row = rows[j];
            z[r] = ok ? a.f[row * a.ldf + h * D + d] : 0.f;
            k[r] = ok && a.gate != DL_GATE_LOWER ? a.k[row * a.ldk + hk * D + d] : 0.f;
            if (WITH_Q) q[r] = ok ? a.q[row * a.ldq + hk * D + d] : 0.f;
        }
        float f[NRW];
        gated_forms(a, c, z, f, k);
#pragma unroll
        for (int r = 0; r < NRW; ++r) {
            const int j = gated_row_of<PAIRS>(warp, r);
            const bool ok = j < len && d < D;
            const float kr = ok ? k[r] : 0.f;
            const float fr = ok ? f[r] : 1.f;
            if (PAIRS) {
                k[r] = kr;
                f[r] = fr;
                if (r & 1) {
                    *reinterpret_cast<float2*>(K + (j - 1) * ld + 2 * d) = make_float2(k[r - 1], kr);
                    *reinterpret_cast<float2*>(F + (j - 1) * ld + 2 * d) = make_float2(f[r - 1], fr);
                }
                continue;
            }
            K[j * ld + d] = kr;
            F[j * ld + d] = fr;
            if (COPY) Q[j * ld + d] = kr;
            if (WITH_Q) {
                float v = q[r] * a.q_scale;
                if (a.q_silu) {
                    float s, t;
                    sigmoid_pair_f(q[r], s, t);
                    v = q[r] * s;
                }
                Q[j * ld + d] = v;
            }
        }
    }
}

__device__ __forceinline__ float dot4(float4 x, float4 y, float acc) { return fmaf(x.x, y.x, fmaf(x.y, y.y, fmaf(x.z, y.z, fmaf(x.w, y.w, acc)))); }

// columns PAR, PAR + 2, .. of a sub-block of 16 rows against its rows: for column j the running product k_j f_(j+1) .. f_i, two channels
// per lane, two columns at a time (a pair of q and f serves both).  The shares for all rows i of a column are reduced together (16
// values over 32 lanes); diag[c] is then row lane / 2 of column 2 c + PAR.
template <bool AHEAD, int PAR>
__device__ __forceinline__ void decayed_diagonal(const float* Qb, const float* Kb, const float* Fb, int D, int D4, int DP, const float* bonus, float (&diag)[8]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int g = 0; g < 4; ++g) {
        pair_f acc[2][16];
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[0][i] = acc[1][i] = 0;
        for (int d = lane * 2; d < D4; d += 64) {
            pair_f p[2] = {ld_pair(Kb + (4 * g + PAR) * DP + d), ld_pair(Kb + (4 * g + PAR + 2) * DP + d)}, bn = 0;
            if (AHEAD) bn = pair_of(d < D ? bonus[d] : 0.f, d + 1 < D ? bonus[d + 1] : 0.f);
#pragma unroll
            for (int i = 4 * g + PAR; i < 16; ++i) {
                const pair_f q = ld_pair(Qb + i * DP + d), f = i > 4 * g + PAR ? ld_pair(Fb + i * DP + d) : 0;
#pragma unroll
                for (int w = 0; w < 2; ++w) {
                    const int j = 4 * g + PAR + 2 * w;
                    if (i < j) continue;
                    if (!AHEAD && i > j) p[w] = mul2(p[w], f);
                    acc[w][i] = fma2(q, AHEAD && i == j ? mul2(bn, p[w]) : p[w], acc[w][i]);
                    if (AHEAD && i > j) p[w] = mul2(p[w], f);
                }
            }
        }
#pragma unroll
        for (int w = 0; w < 2; ++w) {
            float s[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) s[i] = i >= 4 * g + PAR + 2 * w ? pair_sum(acc[w][i]) : 0.f;
#pragma unroll
            for (int o = 16, m = 8; o >= 2; o >>= 1, m >>= 1) {
                const bool hi = lane & o;
#pragma unroll
                for (int t = 0; t < m; ++t) {
                    const float keep = hi ? s[t + m] : s[t], send = hi ? s[t] : s[t + m];
                    s[t] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                }
            }
            diag[2 * g + w] = s[0] + __shfl_xor_sync(0xffffffffu, s[0], 1);
        }
    }
}

// Scores of a chunk's rows against its own rows, put(i, j, sum_d Q_i[d] D_ij[d] K_j[d]) for every i >= j (some i < j inside a
// sub-block are put too), D_ij[d] = product of F_t[d] over j < t <= i (AHEAD: j < t < i, and bonus[d] for i = j).  Q, K, F: [GC][DP] in
// shared memory, complete; put may write over F (every F is read before the first put).  Leaves Q_i scaled by the decay from the
// chunk's start (AHEAD: to the row before i), K_j by the decay to the end of its sub-block of 16 rows, T [4][DP] the sub-blocks'
// whole decays.  No barrier after the last writes.
template <bool AHEAD, typename Put>
__device__ __forceinline__ void decayed_scores(float* Q, float* K, const float* F, float* T, int D, int D4, int DP, const float* bonus, Put put) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tb = threadIdx.x >> 4, cb = threadIdx.x & 15;
    const int blk = warp >> 1;                // two warps per sub-block take its columns in turn
    const float* Qb = Q + (size_t)blk * 16 * DP;
    const float* Kb = K + (size_t)blk * 16 * DP;
    const float* Fb = F + (size_t)blk * 16 * DP;
    float diag[8];
    if (warp & 1) decayed_diagonal<AHEAD, 1>(Qb, Kb, Fb, D, D4, DP, bonus, diag);
    else decayed_diagonal<AHEAD, 0>(Qb, Kb, Fb, D, D4, DP, bonus, diag);
    __syncthreads();
    // rows scaled by the decay from their block's start (Q) / to their block's end (K); T: a block's whole decay
    for (int t = threadIdx.x; t < 2 * D4; t += GC_THREADS) {
        const int bk = t / (D4 / 2), d = (t - bk * (D4 / 2)) * 2;
        float* q = Q + bk * 16 * DP + d;
        float* k = K + bk * 16 * DP + d;
        const float* f = F + bk * 16 * DP + d;
        const pair_f one = pair_of(1.f, 1.f);
        pair_f p = one;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            if (AHEAD) st_pair(q + i * DP, mul2(ld_pair(q + i * DP), p));
            p = mul2(p, ld_pair(f + i * DP));
            if (!AHEAD) st_pair(q + i * DP, mul2(ld_pair(q + i * DP), p));
        }
        st_pair(T + bk * DP + d, p);
        p = one;
#pragma unroll
        for (int i = 15; i >= 0; --i) {
            st_pair(k + i * DP, mul2(ld_pair(k + i * DP), p));
            p = mul2(p, ld_pair(f + i * DP));
        }
    }
    __syncthreads();
    // between sub-blocks: thread (i, j) = (tb, cb) of the six block pairs
    pair_f a10 = 0, a20 = 0, a21 = 0, a30 = 0, a31 = 0, a32 = 0;
#pragma unroll 2
    for (int d = 0; d < D4; d += 4) {
        const ulonglong2 q1 = *reinterpret_cast<const ulonglong2*>(Q + (16 + tb) * DP + d), q2 = *reinterpret_cast<const ulonglong2*>(Q + (32 + tb) * DP + d);
        const ulonglong2 q3 = *reinterpret_cast<const ulonglong2*>(Q + (48 + tb) * DP + d);
        const ulonglong2 k0 = *reinterpret_cast<const ulonglong2*>(K + cb * DP + d), k1 = *reinterpret_cast<const ulonglong2*>(K + (16 + cb) * DP + d);
        const ulonglong2 k2 = *reinterpret_cast<const ulonglong2*>(K + (32 + cb) * DP + d);
        const ulonglong2 t1 = *reinterpret_cast<const ulonglong2*>(T + DP + d), t2 = *reinterpret_cast<const ulonglong2*>(T + 2 * DP + d);
        const pair_f k0x = mul2(k0.x, t1.x), k0y = mul2(k0.y, t1.y), k1x = mul2(k1.x, t2.x), k1y = mul2(k1.y, t2.y);
        a10 = fma2(q1.y, k0.y, fma2(q1.x, k0.x, a10));
        a21 = fma2(q2.y, k1.y, fma2(q2.x, k1.x, a21));
        a32 = fma2(q3.y, k2.y, fma2(q3.x, k2.x, a32));
        a20 = fma2(q2.y, k0y, fma2(q2.x, k0x, a20));
        a31 = fma2(q3.y, k1y, fma2(q3.x, k1x, a31));
        a30 = fma2(q3.y, mul2(k0y, t2.y), fma2(q3.x, mul2(k0x, t2.x), a30));
    }
    __syncthreads();                          // F is done with: the scores may take its place
    put(16 + tb, cb, pair_sum(a10));
    put(32 + tb, cb, pair_sum(a20));
    put(32 + tb, 16 + cb, pair_sum(a21));
    put(48 + tb, cb, pair_sum(a30));
    put(48 + tb, 16 + cb, pair_sum(a31));
    put(48 + tb, 32 + cb, pair_sum(a32));
#pragma unroll
    for (int jj = 0; jj < 8; ++jj) {
        const int j = jj * 2 + (warp & 1), i = lane >> 1;
        if ((lane & 1) == 0) put(blk * 16 + i, blk * 16 + j, diag[jj]);
    }
    // Q: the decay from the chunk's start
    for (int t = threadIdx.x; t < 3 * (D4 / 2); t += GC_THREADS) {
        const int bk = t / (D4 / 2) + 1, d = (t - (bk - 1) * (D4 / 2)) * 2;
        pair_f p = ld_pair(T + d);
        for (int u = 1; u < bk; ++u) p = mul2(p, ld_pair(T + u * DP + d));
        float* q = Q + bk * 16 * DP + d;
#pragma unroll
        for (int i = 0; i < 16; ++i) st_pair(q + i * DP, mul2(ld_pair(q + i * DP), p));
    }
}

int gated_chunk_out_channel(const DlMambaBatch& b, int n_seq, int max_chunks, const DlGatedArgs& a, const GatedScratch& sc, cudaStream_t st);
