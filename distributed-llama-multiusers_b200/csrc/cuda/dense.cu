// Dense (unquantised) weights: embedding gather and  Y[M][N] = epi(X[M][K] . W[N][K]^T)  for bf16 or f32 weights,
// f32 activations, f32 accumulation.  Up to 8 rows a warp per output column streams its weight row (activations staged for
// the CTA, or direct: dense_rows_staged), up to 32 in rounds of 8 or, in bf16 mode from 3 rows on, on mma.sync; more rows, or few columns and inputs
// (dense_in_rounds), take a shared-memory tiled kernel.  All take a batch dimension
// (grid.z) with element strides, which is how per-head products (a head's slice of a weight against a head's slice
// of the activations) run as one launch.  In bf16 mode (`round_x`) the activation operand is rounded to bf16 on
// load, so products are exact in f32 and only the accumulation differs between the kernels; one and two rows of enough weights stream them
// through a ring in shared memory (dense_ring).
//
// Epilogues (what other models of this library fuse into their matmul kernels too): plain store, relu(.)^2,
// aux * sigmoid(.) (an output gate), cap * tanh(. / cap) (logit soft-capping), . * sigmoid(.) (SiLU), aux * (.) (the second
// half of a gated unit), xIELU (a quadratic for z > 0, an exponential for z <= 0, two constants), a constant factor, and a sum
// into Y behind one sigmoid gate per row.  A bias per output column, where given, is added first.
#define WAIT_UNIT 1u
#include "layer_common.cuh"
#include "smem_limit.cuh"
#include "waits.cuh"
#include "../../../include/dllama_b200.h"

__device__ __forceinline__ float dense_epi(float acc, int epi, float aux, float param, float param2) {
    switch (epi) {
        case DL_DENSE_RELU2: { const float r = fmaxf(acc, 0.f); return r * r; }
        case DL_DENSE_SIGMOID_MUL: return aux * sigmoid_f(acc);
        case DL_DENSE_SOFTCAP: return param * tanhf(acc / param);
        case DL_DENSE_SILU: return silu_f(acc);
        case DL_DENSE_MUL: return aux * acc;
        case DL_DENSE_SCALE: return param * acc;
        case DL_DENSE_XIELU: return acc > 0.f ? fmaf(param * acc, acc, 0.5f * acc) : fmaf(param2, expm1f(acc) - acc, 0.5f * acc);
        default: return acc;
    }
}

// element (m, n) of batch b leaves through the epilogue; the row-gated sum reads what Y holds first
__device__ __forceinline__ void dense_store(const DlDenseArgs& a, int b, int m, int n, float acc) {
    float* y = a.Y + (size_t)b * a.y_bs + (size_t)m * a.ldy + n;
    if (a.bias) acc += a.bias[(size_t)b * a.N + n];
    if (a.epi == DL_DENSE_ROWGATE_ADD) {
        *y = fmaf(sigmoid_f(a.aux[(size_t)b * a.aux_bs + (size_t)m * a.ld_aux]), acc, *y);
        return;
    }
    const float aux = a.aux ? a.aux[(size_t)b * a.aux_bs + (size_t)m * a.ld_aux + n] : 0.f;
    *y = dense_epi(acc, a.epi, aux, a.param, a.param2);
}

// paired output columns (weight rows gate_0, up_0, gate_1, up_1, ...): value j of row m from its two products
__device__ __forceinline__ void dense_store_pair(const DlDenseArgs& a, int b, int m, int j, float gate, float up) {
    a.Y[(size_t)b * a.y_bs + (size_t)m * a.ldy + j] = gelu_tanh_f(gate) * up;
}

// ------------------------------------------------------------------------------------------------
// embedding gather: x[m][c] = scale * table[tokens[m]] for each of `copies` copies of the row (row layout [copies][dim])
// ------------------------------------------------------------------------------------------------
template <typename WT>
__global__ void embed_rows_kernel(const WT* __restrict__ table, const int* __restrict__ tokens, float* __restrict__ x, int dim,
                                  float scale, int copies) {
    const int m = blockIdx.x;
    const WT* src = table + (size_t)tokens[m] * dim;
    for (int i = threadIdx.x; i < dim; i += blockDim.x) {
        const float v = ld_f(src + i) * scale;
        for (int c = 0; c < copies; ++c) x[((size_t)m * copies + c) * dim + i] = v;
    }
}

extern "C" int dl_embed_rows(const void* table, int wtype, const int* tokens, float* x, int M, int dim, float scale, int copies,
                             void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    if (copies < 1) { dl_set_error("dl_embed_rows: copies < 1"); return -1; }
    if (wtype == DL_T_BF16) embed_rows_kernel<<<M, 128, 0, st>>>((const __nv_bfloat16*)table, tokens, x, dim, scale, copies);
    else embed_rows_kernel<<<M, 128, 0, st>>>((const float*)table, tokens, x, dim, scale, copies);
    LAYER_CHECK_LAUNCH("dl_embed_rows");
    return 0;
}

// ------------------------------------------------------------------------------------------------
// rows <= 8: one warp per output column, lanes stride K, MT accumulators per lane
// ------------------------------------------------------------------------------------------------
#define GV_WARPS 8

template <typename WT, int MT, bool RX>
__global__ void __launch_bounds__(GV_WARPS * 32) dense_gemv_kernel(DlDenseArgs a) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n = blockIdx.x * GV_WARPS + warp;
    const int b = blockIdx.z;
    if (n >= a.N) return;
    const WT* w = (const WT*)a.W + (size_t)b * a.w_bs + (size_t)n * a.ldw;
    const float* x = a.X + (size_t)b * a.x_bs;
    float acc[MT];
#pragma unroll
    for (int m = 0; m < MT; ++m) acc[m] = 0.f;
    for (int k = lane; k < a.K; k += 32) {
        const float wv = ld_f(w + k);
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            if (m < a.M) {
                float xv = x[(size_t)m * a.ldx + k];
                if (RX) xv = round_bf16(xv);
                acc[m] = fmaf(xv, wv, acc[m]);
            }
        }
    }
#pragma unroll
    for (int m = 0; m < MT; ++m) acc[m] = warp_sum(acc[m]);
    if (lane == 0) {
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            if (m < a.M) dense_store(a, b, m, n, acc[m]);
        }
    }
}

// Staged variant: K % 8 == 0, rows 16-byte aligned (checked on the host).  One warp per output column (PAIR: per gated unit, its gate
// row and its up row), 8 weights per lane and load, a batch of U loads in flight while the last one is multiplied.
// What bounds it: the weights' bytes, which takes many loads in flight and few instructions per weight -- so the CTA's eight warps share
// the activations in shared memory, rounded once (each warp loaded, and rounded, all of them for itself: 8192 inputs x 2048 columns
// took 15.2 us, 2.2 TB/s; 10.2 us now, 3.3 TB/s) -- and the latency of a chain of small kernels: programmatic launch, with the start of
// every weight row on its way into L2 before the previous kernel is waited for.  A lane's products are added in the old order.
template <typename WT> struct WVec;
template <> struct WVec<float> {
    float4 u, v;
    __device__ __forceinline__ void load(const float* p) { u = *reinterpret_cast<const float4*>(p); v = *reinterpret_cast<const float4*>(p + 4); }
    __device__ __forceinline__ void get(float* o) const { o[0] = u.x; o[1] = u.y; o[2] = u.z; o[3] = u.w; o[4] = v.x; o[5] = v.y; o[6] = v.z; o[7] = v.w; }
};
template <> struct WVec<__nv_bfloat16> {
    uint4 u;
    __device__ __forceinline__ void load(const __nv_bfloat16* p) { u = *reinterpret_cast<const uint4*>(p); }
    __device__ __forceinline__ void get(float* o) const {
        const uint32_t r[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            o[2 * i] = __uint_as_float(r[i] << 16);
            o[2 * i + 1] = __uint_as_float(r[i] & 0xffff0000u);
        }
    }
};

// Short weight rows, or very many of them: each warp loads the activations for itself, in a quarter of the staged kernel's registers, so that
// the SMs hold four times the warps and a row's few loads need no barrier ahead of them (dense_rows_staged: where the line lies).  The same
// products in the same order.
template <typename WT, int MT, bool RX, bool PAIR>
__global__ void __launch_bounds__(GV_WARPS * 32) dense_gemv_direct_kernel(DlDenseArgs a) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n = blockIdx.x * GV_WARPS + warp;
    const int b = blockIdx.z;
    if (PAIR ? 2 * n + 1 >= a.N : n >= a.N) return;
    const WT* w0 = (const WT*)a.W + (size_t)b * a.w_bs + (size_t)(PAIR ? 2 * n : n) * a.ldw;
    const WT* w1 = w0 + a.ldw;
    const float* x = a.X + (size_t)b * a.x_bs;
    float g[MT], h[MT];
#pragma unroll
    for (int m = 0; m < MT; ++m) g[m] = h[m] = 0.f;
    for (int k = lane * 8; k < a.K; k += 256) {
        WVec<WT> v0, v1;
        float wg[8], wu[8];
        v0.load(w0 + k);
        if (PAIR) v1.load(w1 + k);
        v0.get(wg);
        if (PAIR) v1.get(wu);
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            if (m < a.M) {
                WVec<float> xm;
                float xv[8];
                xm.load(x + (size_t)m * a.ldx + k);
                xm.get(xv);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float v = RX ? round_bf16(xv[i]) : xv[i];
                    g[m] = fmaf(v, wg[i], g[m]);
                    if (PAIR) h[m] = fmaf(v, wu[i], h[m]);
                }
            }
        }
    }
#pragma unroll
    for (int m = 0; m < MT; ++m) {
        g[m] = warp_sum(g[m]);
        if (PAIR) h[m] = warp_sum(h[m]);
    }
    if (lane == 0) {
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            if (m < a.M) {
                if (PAIR) dense_store_pair(a, b, m, n, g[m], h[m]);
                else dense_store(a, b, m, n, g[m]);
            }
        }
    }
}

template <typename WT, int MT, bool RX, bool PAIR>
__global__ void __launch_bounds__(GV_WARPS * 32) dense_gemv_vec_kernel(DlDenseArgs a) {
    constexpr int XC = 8192 / MT;                                            // inputs staged at a time, per row
    constexpr int U = (sizeof(WT) == 2 ? (MT == 8 ? 4 : 8) : 4) / (PAIR ? 2 : 1);
    static_assert(XC % (256 * U) == 0, "batches end with the staged inputs");
    __shared__ __align__(16) float xs[MT * XC];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n = blockIdx.x * GV_WARPS + warp;
    const int b = blockIdx.z;
    const bool on = PAIR ? 2 * n + 1 < a.N : n < a.N;
    const WT* w0 = (const WT*)a.W + (size_t)b * a.w_bs + (size_t)(PAIR ? 2 * n : n) * a.ldw;
    const WT* w1 = w0 + a.ldw;
    const float* x = a.X + (size_t)b * a.x_bs;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (on && lane < (PAIR ? 2 : 1)) {
        const uint32_t bytes = min((uint32_t)(a.K * sizeof(WT)), 4096u);     // a multiple of 16: K % 8 == 0
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(lane ? w1 : w0), "r"(bytes) : "memory");
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    float g[MT], h[MT];
#pragma unroll
    for (int m = 0; m < MT; ++m) g[m] = h[m] = 0.f;
    WVec<WT> cur[PAIR ? 2 : 1][U], nxt[PAIR ? 2 : 1][U];
    auto fetch = [&](WVec<WT> (&v)[PAIR ? 2 : 1][U], int k0) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int k = k0 + u * 256 + lane * 8;
            if (on && k < a.K) {
                v[0][u].load(w0 + k);
                if (PAIR) v[PAIR ? 1 : 0][u].load(w1 + k);
            }
        }
    };
    fetch(cur, 0);
    for (int c0 = 0; c0 < a.K; c0 += XC) {
        const int kc = min(XC, a.K - c0);
        if (c0) __syncthreads();
#pragma unroll
        for (int m = 0; m < MT; ++m)
            if (m < a.M)
                for (int i = threadIdx.x * 4; i < kc; i += GV_WARPS * 128) {
                    float4 v = *reinterpret_cast<const float4*>(x + (size_t)m * a.ldx + c0 + i);
                    if (RX) { v.x = round_bf16(v.x); v.y = round_bf16(v.y); v.z = round_bf16(v.z); v.w = round_bf16(v.w); }
                    // a block of 256 inputs as the first and the second four of every lane's eight: 16-byte reads without bank conflicts
                    *reinterpret_cast<float4*>(xs + m * XC + (i & ~255) + (i & 4) * 32 + ((i & 255) >> 3) * 4) = v;
                }
        __syncthreads();
        for (int k0 = 0; k0 < kc; k0 += 256 * U) {
            fetch(nxt, c0 + k0 + 256 * U);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int k = k0 + u * 256 + lane * 8;
                if (k < kc) {
                    float wg[8], wu[8];
                    cur[0][u].get(wg);
                    if (PAIR) cur[PAIR ? 1 : 0][u].get(wu);
#pragma unroll
                    for (int m = 0; m < MT; ++m) {
                        if (m < a.M) {
                            const float4 p = *reinterpret_cast<const float4*>(xs + m * XC + k0 + u * 256 + lane * 4), q = *reinterpret_cast<const float4*>(xs + m * XC + k0 + u * 256 + 128 + lane * 4);
                            const float xv[8] = {p.x, p.y, p.z, p.w, q.x, q.y, q.z, q.w};
#pragma unroll
                            for (int i = 0; i < 8; ++i) {
                                g[m] = fmaf(xv[i], wg[i], g[m]);
                                if (PAIR) h[m] = fmaf(xv[i], wu[i], h[m]);
                            }
                        }
                    }
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                cur[0][u] = nxt[0][u];
                if (PAIR) cur[PAIR ? 1 : 0][u] = nxt[PAIR ? 1 : 0][u];
            }
        }
    }
    if (!on) return;
#pragma unroll
    for (int m = 0; m < MT; ++m) {
        g[m] = warp_sum(g[m]);
        if (PAIR) h[m] = warp_sum(h[m]);
    }
    if (lane == 0) {
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            if (m < a.M) {
                if (PAIR) dense_store_pair(a, b, m, n, g[m], h[m]);
                else dense_store(a, b, m, n, g[m]);
            }
        }
    }
}

// ------------------------------------------------------------------------------------------------
// 3 to 32 rows (two of many inputs), bf16 weights, activations rounded to bf16 (K % 8 == 0, aligned rows): mma.sync with the weights as the 16-row operand, so
// the products of 8 activation rows cost one instruction per 16 x 16 weights.
//
// What bounds it: the weights' bytes.  On CUDA cores every row adds 8 FMAs per 16 bytes of weights and lane, and from 9 rows the tiles
// below (16 K steps of scalar loads) left the weights behind entirely: gate|up + down of 4096 x 14336 took 441 us at 8 rows and
// 3150 us at 16; 79 and 117 us here.  (Two rows: launch_dense.)
//
// A lane's 16 bytes of weights are 8 consecutive inputs of row g, and the four pairs fill k slots of two MMAs; the activations' 16 bytes of the same
// inputs fill the same slots, so no shuffle.  A lane copies its weights into places of its own in shared memory (cp.async), one to three halves of a
// step ahead of the half that it multiplies, so nobody waits for anybody; held in registers, half a step ahead, they took 128 of them, one CTA an SM and
// 4 TB/s.  Activations of the next step wait in registers, as many rows as leave the CTAs their places.  Registers and now, us, cold weights: 28672 x 4096 in pairs,
// 3 rows 68 and 47, 8 rows 74 and 50, 16 rows 84 and 76, 24 rows 123 and 114; 4096 x 14336, 3 rows 34.5 and 24.3, 16 rows 56 and 38, 24 rows 84 and 69; 2048 x 8192, 8 rows
// 20.3 and 14.1, 16 rows 28 and 15.5, 32 rows 44 and 25; 2048 x 2048, 8 rows 6.0 and 4.8; 16384 x 2048 in pairs, 16 rows 22.8 and 22.8.  A CTA owns 16 C columns; its eight warps split K, each staging its own activations (bf16, 128 inputs at a time), and meet in
// shared memory at the end, summed in warp order.
//
// An MMA truncates its sum, so none is chained to another: four are added in pairs, rounded, and the last sum keeps its rounding errors
// (two-sum).  8 rows against 64 bits, 2^-24 = 6.0e-8 (one column per warp in f32 FMAs / chains of four / now): normal operands, 256 inputs
// 5.6e-8 / 7.4e-8 / 6.1e-8, 512 inputs 6.3e-8 / 8.3e-8 / 5.8e-8, 2048 7.9e-8 / 9.4e-8 / 6.4e-8, 14336 1.6e-7 / 1.2e-7 / 1.1e-7; operands of one
// sign, 512 inputs 3.3e-8 / 8.2e-8 / 3.3e-8, 2048 3.2e-8 / 8.5e-8 / 2.9e-8.  No slower: norm, gate|up and down of 4096 x 14336 at 8, 16 and 31 rows
// 118.1, 153.3 and 244.7 us with the chains, 117.9, 145.2 and 237.8 without (weights in registers both).
// ------------------------------------------------------------------------------------------------
#define DM_STEP 128                    // inputs staged at a time by a warp
#define DM_LD (DM_STEP + 8)            // row stride of the staged activations (bf16): 16-byte reads of 8 rows without conflicts

__device__ __forceinline__ void dense_two_sum(float& s, float& err, float x) {      // s + x, its rounding error (Knuth) added to err
    const float t = s + x, b = t - s;
    err += (s - (t - b)) + (x - b);
    s = t;
}
__device__ __forceinline__ void dense_mma_bf16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// two: two CTAs an SM (128 registers a thread).  Halves of a step in the ring, and rows of activations on their way a step ahead: as many as fit, but not all of an SM's
// shared memory, from which loads in flight take their places too (28672 x 4096 in pairs, 16 rows: rings of 3 halves 84 to 94 us, of 2 76; 4096 x 4096, 16
// rows: 16 rows ahead 17.2 us, on one CTA an SM, 8 13.3 on two)
static __host__ __device__ constexpr int dense_mma_depth(int NT, int C, bool two) { return NT == 1 ? (C == 1 ? 4 : 3) : C == 1 && !two ? (NT == 4 ? 3 : 4) : NT == 2 && C == 1 ? 4 : 2; }
static __host__ __device__ constexpr int dense_mma_ahead(int NT, int C, bool two) { return NT == 1 ? 8 : C == 1 && !two ? 16 : two && (NT == 4 || C == 2) ? 4 : 8; }
static __host__ __device__ constexpr int dense_mma_xs(int NT, int C) { return NT * 8 * 8 * (DM_LD * 2 > 16 * C * 4 ? DM_LD * 2 : 16 * C * 4); }      // activations, then partial sums

template <int NT, int C, bool TWO>     // 8 NT rows, 16 C columns per CTA
__global__ void __launch_bounds__(256, TWO ? 2 : 1) dense_mma_kernel(DlDenseArgs a) {
    extern __shared__ __align__(16) uint8_t dm_smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int b = blockIdx.z, n0 = blockIdx.x * 16 * C;
    const __nv_bfloat16* W = (const __nv_bfloat16*)a.W + (size_t)b * a.w_bs;
    const float* X = a.X + (size_t)b * a.x_bs;
    __nv_bfloat16* xs = reinterpret_cast<__nv_bfloat16*>(dm_smem) + (size_t)warp * NT * 8 * DM_LD;
    // this warp's inputs: whole steps of DM_STEP, contiguous
    const int steps = (a.K + DM_STEP - 1) / DM_STEP;
    const int s0 = steps * warp / 8, s1 = steps * (warp + 1) / 8;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (s1 > s0 && lane < 16) {          // the start of this warp's weights is on its way into L2 while the previous kernel ends
        const uint32_t bytes = min((uint32_t)(min(a.K, s1 * DM_STEP) - s0 * DM_STEP) * 2u, 2048u);
#pragma unroll
        for (int c = 0; c < C; ++c)
            if (n0 + c * 16 + lane < a.N)
                asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(W + (size_t)(n0 + c * 16 + lane) * a.ldw + s0 * DM_STEP), "r"(bytes) : "memory");
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    float acc[C][NT][4];
#pragma unroll
    for (int c = 0; c < C; ++c)
#pragma unroll
        for (int n = 0; n < NT; ++n) acc[c][n][0] = acc[c][n][1] = acc[c][n][2] = acc[c][n][3] = 0.f;
    // a lane's weights of half a step, [two 32-input pieces][C][rows g and g + 8]: it copies them into places of its own, D - 1 halves ahead
    constexpr int D = dense_mma_depth(NT, C, TWO), SLOTS = 4 * C;
    uint4* ring = reinterpret_cast<uint4*>(dm_smem + dense_mma_xs(NT, C)) + (size_t)warp * D * SLOTS * 32 + lane;
    const int halves = 2 * (s1 - s0);
    auto fetch = [&](int h) {
        if (h < halves) {
#pragma unroll
            for (int p = 0; p < 2; ++p)
#pragma unroll
                for (int c = 0; c < C; ++c)
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const int k = s0 * DM_STEP + h * 64 + p * 32 + t * 8, n = n0 + c * 16 + u * 8 + g;
                        const bool in = k < a.K && n < a.N;
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(ring + ((h % D) * SLOTS + (p * C + c) * 2 + u) * 32)), "l"(in ? W + (size_t)n * a.ldw + k : W), "r"(in ? 16 : 0) : "memory");
                    }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int h = 0; h < D - 1; ++h) fetch(h);
    // a row's 128 inputs of a step by the whole warp; up to 16 rows are on their way a step ahead
    constexpr int AHEAD = dense_mma_ahead(NT, C, TWO);
    float4 xv[AHEAD];
    auto row_step = [&](int m, int s) {
        const int k = s * DM_STEP + lane * 4;
        return m < a.M && k < a.K ? *reinterpret_cast<const float4*>(X + (size_t)m * a.ldx + k) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    auto row_put = [&](int m, float4 v) {
        __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
        *reinterpret_cast<uint2*>(xs + m * DM_LD + lane * 4) = make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
    };
    if (s1 > s0) {
#pragma unroll
        for (int m = 0; m < AHEAD; ++m) xv[m] = row_step(m, s0);
    }
    for (int s = s0; s < s1; ++s) {
        __syncwarp();
#pragma unroll 4
        for (int m = AHEAD; m < NT * 8; ++m) row_put(m, row_step(m, s));
#pragma unroll
        for (int m = 0; m < AHEAD; ++m) row_put(m, xv[m]);
        if (s + 1 < s1) {
#pragma unroll
            for (int m = 0; m < AHEAD; ++m) xv[m] = row_step(m, s + 1);
        }
        __syncwarp();
#pragma unroll
        for (int h = 0; h < 2; ++h) {                // halves of 64 inputs: four MMAs, added in pairs
            const int at = (s - s0) * 2 + h;
            asm volatile("cp.async.wait_group %0;" ::"n"(D - 2) : "memory");
            uint4 x[2][NT], cur[2][C][2];
#pragma unroll
            for (int p = 0; p < 2; ++p)
#pragma unroll
                for (int n = 0; n < NT; ++n) x[p][n] = *reinterpret_cast<const uint4*>(xs + (n * 8 + g) * DM_LD + h * 64 + p * 32 + t * 8);
#pragma unroll
            for (int i = 0; i < SLOTS; ++i) cur[i / (2 * C)][i / 2 % C][i & 1] = ring[((at % D) * SLOTS + i) * 32];
            fetch(at + D - 1);
#pragma unroll
            for (int c = 0; c < C; ++c)
#pragma unroll
                for (int n = 0; n < NT; ++n) {
                    float d[4][4];
#pragma unroll
                    for (int p = 0; p < 2; ++p) {
#pragma unroll
                        for (int e = 0; e < 4; ++e) d[2 * p][e] = d[2 * p + 1][e] = 0.f;
                        dense_mma_bf16(d[2 * p], cur[p][c][0].x, cur[p][c][1].x, cur[p][c][0].y, cur[p][c][1].y, x[p][n].x, x[p][n].y);
                        dense_mma_bf16(d[2 * p + 1], cur[p][c][0].z, cur[p][c][1].z, cur[p][c][0].w, cur[p][c][1].w, x[p][n].z, x[p][n].w);
                    }
#pragma unroll
                    for (int e = 0; e < 4; ++e) acc[c][n][e] += (d[0][e] + d[1][e]) + (d[2][e] + d[3][e]);
                }
        }
    }
    // [warp][row m][16 C columns], in the activations' place
    __syncthreads();
    float* red = reinterpret_cast<float*>(dm_smem);
    constexpr int COLS = 16 * C, PER = NT * 8 * COLS;
#pragma unroll
    for (int c = 0; c < C; ++c)
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) red[warp * PER + (n * 8 + t * 2 + (e & 1)) * COLS + c * 16 + (e >> 1) * 8 + g] = acc[c][n][e];
    __syncthreads();
    const bool pair = a.epi == DL_DENSE_GLU_GELU;
    for (int i = threadIdx.x * 2; i < a.M * COLS; i += 512) {          // two neighbouring columns of a row
        const int m = i / COLS, n = n0 + (i - m * COLS);
        float2 v = make_float2(0.f, 0.f), e = v;
#pragma unroll
        for (int w = 0; w < 8; ++w) {
            const float2 p = *reinterpret_cast<const float2*>(red + w * PER + i);
            dense_two_sum(v.x, e.x, p.x);
            dense_two_sum(v.y, e.y, p.y);
        }
        if (fabsf(e.x) < INFINITY) v.x += e.x;      // (of an infinite sum it is NaN)
        if (fabsf(e.y) < INFINITY) v.y += e.y;
        if (pair) {
            if (n + 1 < a.N) dense_store_pair(a, b, m, n >> 1, v.x, v.y);
        } else {
            if (n < a.N) dense_store(a, b, m, n, v.x);
            if (n + 1 < a.N) dense_store(a, b, m, n + 1, v.y);
        }
    }
}

template <int NT, int C, bool TWO>
static void launch_dense_mma_t(const DlDenseArgs& a, cudaStream_t st) {
    constexpr int smem = dense_mma_xs(NT, C) + 8 * dense_mma_depth(NT, C, TWO) * 4 * C * 512;
    static_assert(smem <= 227 * 1024, "shared memory");
    static SmemLimit given;
    if (dl_smem_limit("dl_dense", dense_mma_kernel<NT, C, TWO>, smem, given) != 0) return;      // (the caller looks at CUDA's last error)
    launch_after(dense_mma_kernel<NT, C, TWO>, dim3((a.N + 16 * C - 1) / (16 * C), 1, a.batch), 256, st, a, smem);
}
// Columns per CTA (they share the staged activations): 16 until every SM has two CTAs, then 32, and 64 for 9 to 16 rows, whose CTAs of 64 have an SM of their own (us, 32 and
// 64 columns: 28672 x 4096 in pairs, 8 rows 49.7 and 55.2, 16 rows 77.1 and 75.7, 16384 x 2048 in pairs, 8 rows 16.9 and 18.5, 16 rows 23.3 and 22.8).
template <int NT>
static void launch_dense_mma(const DlDenseArgs& a, cudaStream_t st, int n_sms) {
    const long long groups = (long long)(a.N + 15) / 16 * a.batch;
    if (NT == 2 && groups >= 4ll * n_sms) launch_dense_mma_t<2, NT == 2 ? 4 : 1, false>(a, st);
    else if (groups >= 2ll * n_sms) launch_dense_mma_t<NT, 2, NT <= 2>(a, st);
    else if (groups > n_sms) launch_dense_mma_t<NT, 1, true>(a, st);
    else launch_dense_mma_t<NT, 1, false>(a, st);
}

// ------------------------------------------------------------------------------------------------
// One row (or two of up to 2048 inputs) against bf16 weights whose rows lie behind one another, activations rounded to bf16: a CTA per SM streams an equal run of weight rows through a
// ring of bulk copies.  A warp keeps its inputs in registers for the whole run: all of up to 2048 (stages of four weight rows, a warp takes one, or both of a gated
// unit, and stores it), or a slice of 2048 of one row (stages of two rows up to 4096 inputs, else of one; the slices meet in shared memory when the run is
// over).  Groups of warps take stages in turn; no warp waits for another before the end.  A lane's products of a slice are added in the order of the kernels above.
//
// What bounds it: the weights' bytes.  The kernels above hold them in registers, two CTAs an SM, and start again every 8 columns.  Cold weights, us, they and
// this: one row, 16384 x 2048 in pairs 15.1 and 12.7, 8192 x 2048 11.2 and 8.6, 32768 x 2048 27.9 and 23.6, 28672 x 4096 in pairs 40.5 and 37.0 (6.3 TB/s), 4096 x
// 4096 9.6 and 8.0, 2048 x 8192 8.5 and 8.0, 4096 x 14336 24.7 and 20.7; two rows, 16384 x 2048 in pairs 18.5 and 13.7, 8192 x 2048 in pairs 11.3 and 9.0.
//
// The price: up to 208 KB of every SM's shared memory.  A kernel behind this one that needs more than 20 KB starts its prologue on an SM when the ring has left it, and
// kernels of other streams wait for one too (norm, gate|up and down of 2048 x 8192 take 24.7 us with that).
// ------------------------------------------------------------------------------------------------
#define DR_K 2048                      // inputs of a warp
#define DR_STAGES 24                   // at most
#define DR_RING (192 * 1024)
#define DR_PART (16 * 1024)
// rows per stage, warps per row (slices of DR_K inputs), warps per stage, groups of them, stages of the ring, stages that are copied at most
struct DenseRing { DlDenseArgs a; int rows, slices, group, groups, stages, most; WaitLimit limit; };

// false: given up (once one wait of the CTA has been, all its later ones).  In line and with the CTA's state in shared memory: a call costs this kernel registers
// (2048 x 8192 7.7 us so, 9.8 by the waits of waits.cuh)
struct DenseRingState { unsigned long long t0; int gave_up; };
__device__ __forceinline__ bool dense_ring_gave_up(const DenseRingState& w) { return *(const volatile int*)&w.gave_up != 0; }
__device__ __forceinline__ bool dense_ring_wait(uint64_t* bar, uint32_t parity, DenseRingState& w, const WaitLimit& l) {
    const uint32_t at = (uint32_t)__cvta_generic_to_shared(bar);
    for (unsigned n = 1; !wait_try(at, parity); ++n) {
        if ((n & 0x3Fu) != 0) continue;
        if (dense_ring_gave_up(w)) return false;
        if ((n & 0x3FFu) != 0) continue;
        unsigned long long now;
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(now));
        const unsigned long long t0 = atomicCAS(&w.t0, 0ull, now);
        if (l.ns != 0 && (t0 == 0 || (long long)(now - t0) <= (long long)l.ns)) continue;
        if (atomicExch(&w.gave_up, 1) == 0) {
            *(volatile unsigned*)l.status = (WAIT_UNIT << 24) + ((atomicAdd(&g_times_given_up, 1u) + 1u) & 0xFFFFFFu);
            __threadfence_system();
        }
        return false;
    }
    return true;
}
// consumers (two rows of activations: their inputs leave registers for eight); one more warp copies
static __host__ __device__ constexpr int dense_ring_warps(int MT, bool pair, bool sliced) { return MT == 2 ? 8 : pair && !sliced ? 12 : 16; }
template <int MT, bool PAIR, bool SLICED>
__global__ void __launch_bounds__((dense_ring_warps(MT, PAIR, SLICED) + 1) * 32, 1) dense_ring_kernel(DenseRing g) {
    constexpr int WARPS = dense_ring_warps(MT, PAIR, SLICED), RW = PAIR && !SLICED ? 2 : 1;      // RW: rows of a stage per warp
    const DlDenseArgs& a = g.a;
    extern __shared__ __align__(128) uint8_t ring[];
    __shared__ uint64_t full[DR_STAGES], empty[DR_STAGES];
    __shared__ DenseRingState ws;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t row_bytes = a.K * 2, stage_bytes = row_bytes * g.rows;
    // this CTA's stages
    const int all = (a.N + g.rows - 1) / g.rows, t0 = (int)((long long)all * blockIdx.x / gridDim.x), nt = (int)((long long)all * (blockIdx.x + 1) / gridDim.x) - t0;
    const __nv_bfloat16* w = (const __nv_bfloat16*)a.W + (size_t)t0 * g.rows * a.K;
    auto rows_of = [&](int t) { return min(g.rows, a.N - (t0 + t) * g.rows); };
    if (threadIdx.x == 0) {
        ws.t0 = 0;
        ws.gave_up = 0;
        for (int s = 0; s < g.stages; ++s) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"((uint32_t)__cvta_generic_to_shared(&full[s])) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"((uint32_t)__cvta_generic_to_shared(&empty[s])), "r"(g.group) : "memory");
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (warp == WARPS && lane < 2 && lane < nt)      // the first weights are on their way into L2 while the previous kernel ends
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(w + (size_t)lane * g.rows * a.K), "r"(row_bytes * rows_of(lane)) : "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (warp == WARPS) {
        if (lane == 0)
            for (int t = 0; t < min(nt, g.most); ++t) {
                const int s = t % g.stages;
                if (t >= g.stages && !dense_ring_wait(&empty[s], ((t / g.stages) & 1) ^ 1, ws, g.limit)) break;
                const uint32_t bar = (uint32_t)__cvta_generic_to_shared(&full[s]), bytes = row_bytes * rows_of(t);
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"((uint32_t)__cvta_generic_to_shared(ring + (size_t)s * stage_bytes)), "l"(w + (size_t)t * g.rows * a.K), "r"(bytes), "r"(bar) : "memory");
            }
        if (dense_ring_gave_up(ws)) __nanosleep(1000000);      // copies in flight land
        return;
    }
    const int grp = warp / g.group, wi = warp - grp * g.group, slice = SLICED ? wi % g.slices : 0, row = SLICED ? wi / g.slices : wi * RW, k0 = slice * DR_K + lane * 8;
    float* part = reinterpret_cast<float*>(ring + (size_t)g.stages * stage_bytes);      // SLICED: [this CTA's rows][slices][MT]
    float x[MT][DR_K / 32];
#pragma unroll
    for (int i = 0; i < DR_K / 256; ++i) {
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            WVec<float> v = {};
            if (k0 + i * 256 < a.K) v.load(a.X + (size_t)m * a.ldx + k0 + i * 256);
            float f[8];
            v.get(f);
#pragma unroll
            for (int j = 0; j < 8; ++j) x[m][i * 8 + j] = round_bf16(f[j]);
        }
    }
    for (int t = grp; grp < g.groups && t < nt; t += g.groups) {
        const int s = t % g.stages, n = (t0 + t) * g.rows + row;
        const bool ok = dense_ring_wait(&full[s], (t / g.stages) & 1, ws, g.limit) && !dense_ring_gave_up(ws);      // (a stage behind one given up shows the parity of the use before)
        float acc[MT][RW];
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int r = 0; r < RW; ++r) acc[m][r] = ok ? 0.f : __int_as_float(0x7fc00000);
        if (ok && n + RW <= a.N) {               // (pairs: N is even)
            const uint8_t* base = ring + (size_t)s * stage_bytes + (size_t)row * row_bytes + k0 * 2;
#pragma unroll
            for (int i = 0; i < DR_K / 256; ++i)
                if (k0 + i * 256 < a.K) {
#pragma unroll
                    for (int r = 0; r < RW; ++r) {
                        WVec<__nv_bfloat16> v;
                        v.u = *reinterpret_cast<const uint4*>(base + r * row_bytes + i * 512);
                        float f[8];
                        v.get(f);
#pragma unroll
                        for (int m = 0; m < MT; ++m)
#pragma unroll
                            for (int j = 0; j < 8; ++j) acc[m][r] = fmaf(x[m][i * 8 + j], f[j], acc[m][r]);
                    }
                }
        }
        __syncwarp();
        if (lane == 0 && ok) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"((uint32_t)__cvta_generic_to_shared(&empty[s])) : "memory");
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int r = 0; r < RW; ++r) acc[m][r] = warp_sum(acc[m][r]);
        if (lane == 0 && n + RW <= a.N) {
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                if (SLICED) part[((t * g.rows + row) * g.slices + slice) * MT + m] = acc[m][0];
                else if (PAIR) dense_store_pair(a, 0, m, n >> 1, acc[m][0], acc[m][RW - 1]);
                else dense_store(a, 0, m, n, acc[m][0]);
            }
        }
    }
    if (dense_ring_gave_up(ws)) __nanosleep(1000000);      // copies in flight land
    if (!SLICED) return;
    asm volatile("bar.sync 1, %0;" ::"n"(WARPS * 32) : "memory");
    const int n0 = t0 * g.rows, rows = min(nt * g.rows, a.N - n0);
    auto sum = [&](int r, int m) {
        float v = part[r * g.slices * MT + m];
        for (int k = 1; k < g.slices; ++k) v += part[(r * g.slices + k) * MT + m];
        return v;
    };
    const int outs = PAIR ? rows / 2 : rows;
    for (int i = threadIdx.x; i < outs * MT; i += WARPS * 32) {
        const int m = i / outs, r = i - m * outs;
        if (PAIR) dense_store_pair(a, 0, m, (n0 >> 1) + r, sum(2 * r, m), sum(2 * r + 1, m));
        else dense_store(a, 0, m, n0 + r, sum(r, m));
    }
}
// From 1025 inputs and 12 Mi weights on (us, the kernels above and this: 65536 x 1024 30.4 and 32.8, 2048 x 2048 3.4 and 4.8, 2048 x 4096 5.2 and 5.9, 6144 x 2048 7.3 and
// 7.4, 3072 x 4096 8.9 and 6.9); two rows, whose inputs leave registers for eight warps, where a warp holds
// them all (in slices 28672 x 4096 in pairs 52.6, by one MMA for both 46.2).
static bool dense_ring(const DlDenseArgs& a, int n_sms, DenseRing& g) {
    if (a.M > 2 || a.batch != 1 || a.ldw != a.K || a.K <= DR_K / 2 || a.K > 8 * DR_K || (long long)a.N * a.K < 12ll << 20) return false;
    if (a.M == 2 && a.K > DR_K) return false;
    const bool pair = a.epi == DL_DENSE_GLU_GELU;
    g.a = a;
    g.slices = (a.K + DR_K - 1) / DR_K;
    g.rows = g.slices == 1 ? 4 : g.slices == 2 ? 2 : 1;
    if (pair && g.rows == 1) return false;
    g.group = g.slices == 1 && pair ? 2 : g.rows * g.slices;
    g.groups = dense_ring_warps(a.M, pair, g.slices > 1) / g.group;
    const int fit = (int)(DR_RING / ((long long)a.K * 2 * g.rows)), n_stages = (a.N + g.rows - 1) / g.rows;
    g.stages = (fit < DR_STAGES ? fit : DR_STAGES) / g.groups * g.groups;          // a stage belongs to one group: a wait cannot see a phase before the last
    return g.stages >= g.groups && (g.slices == 1 || ((long long)n_stages / n_sms + 1) * g.rows * g.slices * a.M * 4 <= DR_PART);
}
template <int MT, bool PAIR, bool SLICED>
static void launch_dense_ring_t(const DenseRing& g, cudaStream_t st, int n_sms) {
    static SmemLimit given;
    if (dl_smem_limit("dl_dense", dense_ring_kernel<MT, PAIR, SLICED>, DR_RING + DR_PART, given) != 0) return;
    launch_after(dense_ring_kernel<MT, PAIR, SLICED>, dim3(n_sms), (dense_ring_warps(MT, PAIR, SLICED) + 1) * 32, st, g, (size_t)g.stages * g.rows * g.a.K * 2 + (SLICED ? DR_PART : 0));
}
template <int MT>
static void launch_dense_ring(const DenseRing& g, cudaStream_t st, int n_sms) {
    constexpr bool SLICED = MT == 1;                 // (two rows of more inputs are no work of this kernel)
    if (g.a.epi == DL_DENSE_GLU_GELU) {
        if (g.slices == 1) launch_dense_ring_t<MT, true, false>(g, st, n_sms);
        else launch_dense_ring_t<MT, true, SLICED>(g, st, n_sms);
    } else {
        if (g.slices == 1) launch_dense_ring_t<MT, false, false>(g, st, n_sms);
        else launch_dense_ring_t<MT, false, SLICED>(g, st, n_sms);
    }
}

// paired columns (GLU): one warp per value, its gate row and its up row side by side
template <typename WT, int MT, bool RX>
__global__ void __launch_bounds__(GV_WARPS * 32) dense_gemv_pair_kernel(DlDenseArgs a) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int j = blockIdx.x * GV_WARPS + warp;
    const int b = blockIdx.z;
    if (2 * j + 1 >= a.N) return;
    const WT* w0 = (const WT*)a.W + (size_t)b * a.w_bs + (size_t)(2 * j) * a.ldw;
    const WT* w1 = w0 + a.ldw;
    const float* x = a.X + (size_t)b * a.x_bs;
    float g[MT], u[MT];
#pragma unroll
    for (int m = 0; m < MT; ++m) g[m] = u[m] = 0.f;
    for (int k = lane; k < a.K; k += 32) {
        const float wg = ld_f(w0 + k), wu = ld_f(w1 + k);
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            if (m < a.M) {
                float v = x[(size_t)m * a.ldx + k];
                if (RX) v = round_bf16(v);
                g[m] = fmaf(v, wg, g[m]);
                u[m] = fmaf(v, wu, u[m]);
            }
        }
    }
#pragma unroll
    for (int m = 0; m < MT; ++m) { g[m] = warp_sum(g[m]); u[m] = warp_sum(u[m]); }
    if (lane == 0) {
#pragma unroll
        for (int m = 0; m < MT; ++m)
            if (m < a.M) dense_store_pair(a, b, m, j, g[m], u[m]);
    }
}

// ------------------------------------------------------------------------------------------------
// more rows: 64 x 64 output tile per CTA, 16-wide K steps through shared memory, 4 x 4 outputs per thread
// ------------------------------------------------------------------------------------------------
#define GT_BM 64
#define GT_BN 64
#define GT_BK 16

template <typename WT, bool RX>
__global__ void __launch_bounds__(256) dense_tile_kernel(DlDenseArgs a) {
    __shared__ float Xs[GT_BK][GT_BM + 1];
    __shared__ float Ws[GT_BK][GT_BN + 1];
    const int b = blockIdx.z;
    const WT* W = (const WT*)a.W + (size_t)b * a.w_bs;
    const float* X = a.X + (size_t)b * a.x_bs;
    const int m0 = blockIdx.y * GT_BM, n0 = blockIdx.x * GT_BN;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
    for (int k0 = 0; k0 < a.K; k0 += GT_BK) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int idx = threadIdx.x + i * 256;
            const int r = idx >> 4, k = idx & 15;
            float xv = 0.f, wv = 0.f;
            if (k0 + k < a.K) {
                if (m0 + r < a.M) xv = X[(size_t)(m0 + r) * a.ldx + k0 + k];
                if (n0 + r < a.N) wv = ld_f(W + (size_t)(n0 + r) * a.ldw + k0 + k);
            }
            Xs[k][r] = RX ? round_bf16(xv) : xv;
            Ws[k][r] = wv;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < GT_BK; ++k) {
            float xr[4], wr[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) { xr[i] = Xs[k][ty * 4 + i]; wr[i] = Ws[k][tx * 4 + i]; }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(xr[i], wr[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int m = m0 + ty * 4 + i;
        if (m >= a.M) continue;
        if (a.epi == DL_DENSE_GLU_GELU) {          // this thread's columns are two (gate, up) pairs
#pragma unroll
            for (int j = 0; j < 4; j += 2) {
                const int n = n0 + tx * 4 + j;
                if (n + 1 < a.N) dense_store_pair(a, b, m, n >> 1, acc[i][j], acc[i][j + 1]);
            }
            continue;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tx * 4 + j;
            if (n >= a.N) continue;
            dense_store(a, b, m, n, acc[i][j]);
        }
    }
}

// Bytes of weights per warp from which the staged kernel is the faster one.  Its CTAs take half an SM's registers: one wave of them streams
// more than the direct kernel from short rows on; every further wave waits for its activations again, where the direct kernel's many warps
// hide each other's start (us, direct and staged, cold weights: one row of bf16, 2048 x 2048 5.8 and 3.4, 8192 x 4096 17.9 and 16.3, 8192 x 512 5.2 and 7.1,
// 32768 x 2048 27.6 and 34.5, 65536 x 4096 93 and 98; two rows 8192 x 4096 22.4 and 23.4, 32768 x 8192 161 and 145; f32, one row 512 x 512 2.1 and
// 2.1, four rows 2048 x 256 3.3 and 3.9, 2048 x 2048 9.2 and 7.7, 32768 x 4096 162 and 170; pairs of 8192 x 2048 in bf16 15.8 and 15.0,
// of 32768 x 2048 43 and 45).  Waves are of 2 CTAs an SM: one, up to eight, more.
static bool dense_rows_staged(const DlDenseArgs& a, int wsize, int mt, bool pair, long long ctas, int n_sms) {
    static const int kb[4][3] = {{1, 8, 32}, {4, 16, 16}, {8, 32, 32}, {2, 16, 16}}, kb_pair[4][3] = {{1, 8, 32}, {4, 8, 16}, {4, 16, 16}, {1, 8, 8}};
    const int r = mt == 1 ? 0 : mt == 2 ? 1 : mt == 4 ? 2 : 3, w = ctas <= 2ll * n_sms ? 0 : ctas <= 16ll * n_sms ? 1 : 2;
    const int least = mt == 2 && w == 0 && wsize == 2 ? 1 : (pair ? kb_pair : kb)[r][w];
    return (long long)a.K * wsize * (pair ? 2 : 1) >= least * 1024ll;
}

template <typename WT, int MT, bool RX>
static void launch_dense_rows(const DlDenseArgs& a, cudaStream_t st, bool vec) {
    const bool pair = a.epi == DL_DENSE_GLU_GELU;
    const dim3 grid(((pair ? a.N / 2 : a.N) + GV_WARPS - 1) / GV_WARPS, 1, a.batch);
    if (!vec) {
        if (pair) dense_gemv_pair_kernel<WT, MT, RX><<<grid, GV_WARPS * 32, 0, st>>>(a);
        else dense_gemv_kernel<WT, MT, RX><<<grid, GV_WARPS * 32, 0, st>>>(a);
        return;
    }
    if constexpr (MT <= 2 || sizeof(WT) != 2 || !RX) {       // (more rows of these run on dense_mma_kernel, or 3 and 4 direct)
        if (dense_rows_staged(a, sizeof(WT), MT, pair, (long long)grid.x * a.batch, dl_device_sm_count())) {
            if (pair) launch_after(dense_gemv_vec_kernel<WT, MT, RX, true>, grid, GV_WARPS * 32, st, a);
            else launch_after(dense_gemv_vec_kernel<WT, MT, RX, false>, grid, GV_WARPS * 32, st, a);
            return;
        }
    }
    if constexpr (MT <= 4 || sizeof(WT) != 2 || !RX) {
        if (pair) dense_gemv_direct_kernel<WT, MT, RX, true><<<grid, GV_WARPS * 32, 0, st>>>(a);
        else dense_gemv_direct_kernel<WT, MT, RX, false><<<grid, GV_WARPS * 32, 0, st>>>(a);
    }
}

// 9 to 32 rows in rounds of 8, each of which streams the weights at their own pace, or in the tiles above (a scalar load per weight, most of 64
// rows empty, but one launch)?  In f32, us by tile and by rounds: gate|up + down of 4096 x 14336 at 16 rows 3460 and 630, 2048 x 64 at 32 rows
// 10.9 and 21.9, 8192 x 128 22 and 64, 16 x 2048 x 512 at 16 rows 133 and 160, at 9 133 and 104.  Both go by what these sweeps (64 to 8192 inputs, 64 to 131072
// columns) fit, in ns: a round by its CTAs and their inputs, or by the length of one; the tiles by their steps of K, side by side on the SMs or in turn.
static bool dense_in_rounds(const DlDenseArgs& a, int n_sms) {
    const bool pair = a.epi == DL_DENSE_GLU_GELU;
    const long long rounds = (a.M + 7) / 8, ctas = ((pair ? a.N / 2 : a.N) + GV_WARPS - 1) / GV_WARPS * (long long)a.batch;
    const long long tiles = (a.N + GT_BN - 1) / GT_BN * (long long)a.batch, deep = tiles > n_sms ? tiles * 60 / n_sms : 60;
    const long long by_ctas = ctas * (6 + (pair ? 34ll : 17ll) * a.K / 1000);
    return rounds * (by_ctas > 4500 ? by_ctas : 4500) <= 5000 + a.K * (35 + deep);
}

template <typename WT, bool RX>
static void launch_dense(const DlDenseArgs& a, cudaStream_t st) {
    const bool vec = a.K % 8 == 0 && a.ldw % 8 == 0 && a.w_bs % 8 == 0 && a.ldx % 4 == 0 && a.x_bs % 4 == 0 &&
                     ((uintptr_t)a.W & 15) == 0 && ((uintptr_t)a.X & 15) == 0;
    const int n_sms = dl_device_sm_count();
    if constexpr (sizeof(WT) == 2 && RX) {
        // With few steps of K most warps of an mma CTA idle, and of few products its sum is the less exact one (from 64 bits, f32 FMAs and mma: 264 inputs 5.5e-8 and
        // 5.7e-8, 320 5.8e-8 and 5.6e-8): of very many columns, 3 and 4 rows of few inputs go direct (us, direct and mma: 16 x 8192 x 256, 3 rows 51.3 and
        // 52.2, 4 rows 60.7 and 52.3; 16 x 2048 x 512, 3 rows 22.1 and 15.9).
        const bool direct = a.M <= 4 && a.K <= (a.M == 3 ? 312 : 256) && (long long)a.N * a.batch >= 128ll * n_sms;
        // Two rows whose inputs a warp cannot hold, of weights enough for two CTAs an SM (us, one by one and here: 4096 x 4096 17.6 and 8.8, 4096 x
        // 14336 37.3 and 23.9, 2400 x 8192 20.1 and 13.7, 32768 x 4096 60.5 and 54.2, 28672 x 4096 in pairs 47.1 and 46.2; 2048 x 8192 12.0 and 13.3).
        const bool two = a.M == 2 && a.K > DR_K && a.N > 16 * n_sms && (long long)a.N * a.K * a.batch >= 12ll << 20;
        if (vec && (two || (a.M >= 3 && a.M <= 32 && !direct))) {
            if (a.M <= 8) launch_dense_mma<1>(a, st, n_sms);
            else if (a.M <= 16) launch_dense_mma<2>(a, st, n_sms);
            else launch_dense_mma<4>(a, st, n_sms);
            return;
        }
    }
    if constexpr (sizeof(WT) == 2 && RX) {
        DenseRing g;
        if (vec && dense_ring(a, n_sms, g) && dl_wait_limit("dl_dense", &g.limit) == 0) {
            g.most = g.limit.ns == 0 ? 2 : 1 << 30;                                        // (no time: tests)
            if (a.M == 1) launch_dense_ring<1>(g, st, n_sms);
            else launch_dense_ring<2>(g, st, n_sms);
            return;
        }
    }
    if (a.M <= 8) {
        if (a.M <= 1) launch_dense_rows<WT, 1, RX>(a, st, vec);
        else if (a.M <= 2) launch_dense_rows<WT, 2, RX>(a, st, vec);
        else if (a.M <= 4) launch_dense_rows<WT, 4, RX>(a, st, vec);
        else launch_dense_rows<WT, 8, RX>(a, st, vec);
    } else if (vec && a.M <= 32 && dense_in_rounds(a, n_sms)) {
        for (int m0 = 0; m0 < a.M; m0 += 8) {
            DlDenseArgs r = a;
            r.M = a.M - m0 < 8 ? a.M - m0 : 8;
            r.X += (size_t)m0 * a.ldx;
            r.Y += (size_t)m0 * a.ldy;
            if (a.aux) r.aux += (size_t)m0 * a.ld_aux;
            launch_dense<WT, RX>(r, st);
        }
    } else {
        dim3 grid((a.N + GT_BN - 1) / GT_BN, (a.M + GT_BM - 1) / GT_BM, a.batch);
        dense_tile_kernel<WT, RX><<<grid, 256, 0, st>>>(a);
    }
}

extern "C" int dl_dense(const DlDenseArgs* args, void* stream) {
    const DlDenseArgs& a = *args;
    if (a.M < 1 || a.N < 1 || a.K < 1 || a.batch < 1) { dl_set_error("dl_dense: empty problem"); return -1; }
    if ((a.epi == DL_DENSE_SIGMOID_MUL || a.epi == DL_DENSE_MUL || a.epi == DL_DENSE_ROWGATE_ADD) && a.aux == nullptr) { dl_set_error("dl_dense: the gate epilogue needs aux"); return -1; }
    if (a.epi == DL_DENSE_GLU_CLAMP || a.epi == DL_DENSE_GLU_SILU) { dl_set_error("dl_dense: the paired-column epilogue belongs to the tensor-core GEMM"); return -1; }
    if (a.bias && a.epi == DL_DENSE_GLU_GELU) { dl_set_error("dl_dense: paired columns take no bias"); return -1; }
    if (a.epi == DL_DENSE_GLU_GELU && (a.N & 1)) { dl_set_error("dl_dense: paired columns need an even number of weight rows"); return -1; }
    cudaStream_t st = (cudaStream_t)stream;
    if (a.wtype == DL_T_BF16) {
        if (a.round_x) launch_dense<__nv_bfloat16, true>(a, st);
        else launch_dense<__nv_bfloat16, false>(a, st);
    } else if (a.wtype == DL_T_F32) {
        if (a.round_x) launch_dense<float, true>(a, st);
        else launch_dense<float, false>(a, st);
    } else {
        dl_set_error("dl_dense: unknown weight type %d", a.wtype);
        return -1;
    }
    LAYER_CHECK_LAUNCH("dl_dense");
    return 0;
}

// ------------------------------------------------------------------------------------------------
// operand images of the tcgen05 GEMM (gemm_wh_tc.cu) for bf16 weights: element (row, k) of a 128 x 128 tile lives at
//   (row >> 3) * 2048 + (k >> 3) * 128 + (row & 7) * 16 + (k & 7) * 2      (8 x 16 B core matrices, K-major)
// weights: tiles [row_tile][k_tile][32 KB]; activations: [k_tile][ncap / 8][2048 B].  One thread per 8 K values.
// ------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) wh_from_dense_kernel(const __nv_bfloat16* __restrict__ w, int N, int K, long long ldw,
                                                            uint8_t* __restrict__ wh, int KT) {
    const int tile = blockIdx.x, rt = tile / KT, kt = tile % KT;
    uint8_t* out = wh + (size_t)tile * 32768;
    for (int i = threadIdx.x; i < 128 * 16; i += blockDim.x) {
        const int r = i >> 4, c = i & 15;
        const int row = rt * 128 + r, k0 = kt * 128 + c * 8;
        __align__(16) __nv_bfloat16 v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = (row < N && k0 + j < K) ? w[(size_t)row * ldw + k0 + j] : __float2bfloat16_rn(0.f);
        *reinterpret_cast<uint4*>(out + (size_t)(r >> 3) * 2048 + c * 128 + (r & 7) * 16) = *reinterpret_cast<const uint4*>(v);
    }
}

__global__ void __launch_bounds__(256) xh_from_rows_kernel(const float* __restrict__ x, long long ldx, int M, int K, int ncap,
                                                           uint8_t* __restrict__ xh) {
    const int g = blockIdx.x, kt = blockIdx.y;           // row group of 8, k tile
    uint8_t* out = xh + ((size_t)kt * (ncap >> 3) + g) * 2048;
    for (int i = threadIdx.x; i < 8 * 16; i += blockDim.x) {
        const int r = i & 7, c = i >> 3;
        const int m = g * 8 + r, k0 = kt * 128 + c * 8;
        __align__(16) __nv_bfloat16 v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = __float2bfloat16_rn((m < M && k0 + j < K) ? x[(size_t)m * ldx + k0 + j] : 0.f);
        *reinterpret_cast<uint4*>(out + c * 128 + r * 16) = *reinterpret_cast<const uint4*>(v);
    }
}

// the same image with a row gather: image row i < n_rows holds source row rows[i] (negative: a row of zeros) -- the rows of
// a routed feed-forward sorted by expert
__global__ void __launch_bounds__(256) xh_gather_rows_kernel(const float* __restrict__ x, long long ldx, int n_rows, int K, int ncap,
                                                             uint8_t* __restrict__ xh, const int* __restrict__ rows) {
    const int g = blockIdx.x, kt = blockIdx.y;
    uint8_t* out = xh + ((size_t)kt * (ncap >> 3) + g) * 2048;
    for (int i = threadIdx.x; i < 8 * 16; i += blockDim.x) {
        const int r = i & 7, c = i >> 3;
        const int k0 = kt * 128 + c * 8;
        const int at = g * 8 + r;
        const int m = at < n_rows ? rows[at] : -1;
        __align__(16) __nv_bfloat16 v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = __float2bfloat16_rn((m >= 0 && k0 + j < K) ? x[(size_t)m * ldx + k0 + j] : 0.f);
        *reinterpret_cast<uint4*>(out + c * 128 + r * 16) = *reinterpret_cast<const uint4*>(v);
    }
}

extern "C" int dl_wh_from_dense(const void* w, int N, int K, long long ldw, uint8_t* wh, void* stream) {
    if (N < 1 || K < 1) { dl_set_error("dl_wh_from_dense: empty matrix"); return -1; }
    const int KT = (K + 127) / 128, RT = (N + 127) / 128;
    wh_from_dense_kernel<<<RT * KT, 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)w, N, K, ldw, wh, KT);
    LAYER_CHECK_LAUNCH("dl_wh_from_dense");
    return 0;
}

extern "C" int dl_xh_from_rows(const float* x, long long ldx, int M, int K, int ncap, uint8_t* xh, void* stream) {
    if (M < 1 || K < 1 || ncap % 8 != 0 || ncap < M) { dl_set_error("dl_xh_from_rows: bad M=%d / ncap=%d", M, ncap); return -1; }
    dim3 grid((M + 7) / 8, (K + 127) / 128);
    xh_from_rows_kernel<<<grid, 128, 0, (cudaStream_t)stream>>>(x, ldx, M, K, ncap, xh);
    LAYER_CHECK_LAUNCH("dl_xh_from_rows");
    return 0;
}

// image row i < n_rows holds source row rows[i] of x (device map; negative: zeros)
extern "C" int dl_xh_gather_rows(const float* x, long long ldx, const int* rows, int n_rows, int K, int ncap, uint8_t* xh, void* stream) {
    if (n_rows < 1 || K < 1 || ncap % 8 != 0 || ncap < n_rows || rows == nullptr) { dl_set_error("dl_xh_gather_rows: bad n_rows=%d / ncap=%d", n_rows, ncap); return -1; }
    dim3 grid((n_rows + 7) / 8, (K + 127) / 128);
    xh_gather_rows_kernel<<<grid, 128, 0, (cudaStream_t)stream>>>(x, ldx, n_rows, K, ncap, xh, rows);
    LAYER_CHECK_LAUNCH("dl_xh_gather_rows");
    return 0;
}
