// Epilogues shared by the dp4a GEMV and the tcgen05 GEMM.  Both kernels end with an f32 tile
// out_s[m * out_ld + r] (r = local output row, m = activation row) in shared memory; the
// epilogue turns it into what the *next* kernel consumes, so no stand-alone elementwise kernels
// (rope / shift / silu / mul / cast / merge-add) exist on the hot path.
#pragma once
#include "common.cuh"
#include <cuda_bf16.h>
#include "../../../include/dllama_b200.h"

// ---- Q80 block writers -------------------------------------------------------------------------
// One warp holds one 32-element block (lane = element).  Writes the XQ slab entry and/or the XH
// fp16 entry for activation row m, global K-block index kblock.
DL_DEVINL void q80_block_store(float val, int lane, int m, int kblock, int mcap, uint8_t* xq, uint8_t* xh) {
    float amax = warp_max(fabsf(val));
    float d = amax / 127.0f;
    float id = (d != 0.0f) ? (1.0f / d) : 0.0f;
    int q = __float2int_rn(val * id);
    __half d16 = __float2half_rn(d);
    float df = __half2float(d16);
    int kt = kblock >> 2, kb = kblock & 3;
    if (xq != nullptr) {
        int sumq = warp_sum_i(q);
        uint8_t* row = xq + ((size_t)kt * mcap + m) * XQ_ROW_BYTES;
        reinterpret_cast<int8_t*>(row)[kb * 32 + lane] = (int8_t)q;
        if (lane == 0) {
            reinterpret_cast<float*>(row + 128)[kb] = df;
            reinterpret_cast<int*>(row + 144)[kb] = 8 * sumq;
        }
    }
    if (xh != nullptr) {
        int w, s;
        xh_slot(lane, w, s);
        size_t off = (size_t)kt * (size_t)(mcap >> 3) * XH_ROWGROUP_BYTES + (size_t)(m >> 3) * XH_ROWGROUP_BYTES +
                     (size_t)(kb * 4 + w) * 128 + (size_t)(m & 7) * 16 + (size_t)s * 2;
        // fp16 operand of the tcgen05 path: a block whose scale exceeds 515 (|x| > 65405) saturates instead of becoming inf
        *reinterpret_cast<__half*>(xh + off) = __float2half_rn((float)q * fminf(df, 515.0f));
    }
}

// quantize->dequantize one 32-element block held by a warp
DL_DEVINL float q80_roundtrip_warp(float val) {
    float amax = warp_max(fabsf(val));
    float d = amax / 127.0f;
    float id = (d != 0.0f) ? (1.0f / d) : 0.0f;
    int q = __float2int_rn(val * id);
    return (float)q * __half2float(__float2half_rn(d));
}

DL_DEVINL float act_silu(float x) { return x / (1.0f + expf(-x)); }
DL_DEVINL float act_gelu(float x) {
    return 0.5f * x * (1.0f + tanhf(0.797884560802865f * (x + 0.044715f * x * x * x)));
}

// ---- the epilogue --------------------------------------------------------------------------------
// epilogue_rows: called by (at least) the first `rows` threads (tid = local output row; rows is a
// multiple of 32 so every warp is either fully in or fully out).  out_s[m*out_ld + r] holds
// activation rows m0..m0+M-1 (M <= 32); grow0 = global row of local row 0, d_real = real (unpadded)
// rows.  A caller with several thread groups per tile passes (m_first, m_step) so group k handles
// rows k, k+step, ...; everything a row needs from global memory (position, KV page) is fetched
// once per warp by lane m and broadcast with shuffles, so the per-row loop has no dependent loads.
// DL_EPI_DENSE has no shuffles and no lane per row, so with that kind alone `rows` may be any multiple
// of 8 and M any number (gemm_wh_rows_kernel: up to 256 and 128).
DL_DEVINL void epilogue_rows(const DlEpilogue& e, const float* out_s, int out_ld, int rows, int grow0, int d_real,
                             int M, int m0, int tid, int m_first = 0, int m_step = 1) {
    const int lane = tid & 31;
    if (e.kind == DL_EPI_STORE) {
        if (tid < rows) {
            const int grow = grow0 + tid;
            const bool live = grow < d_real;
            const bool rt = e.q80_roundtrip != 0;
            const int nd = e.n_dst;
            const size_t ld = (size_t)e.ld;
            const size_t res_ld = (size_t)e.residual_ld;
            const float* res = (e.residual != nullptr && live) ? e.residual + (size_t)m0 * res_ld + grow : nullptr;
            const size_t off0 = (size_t)e.dst_off + (size_t)m0 * ld + grow;
            if (nd == 1) {
                float* d0 = e.dst[0] + off0;
#pragma unroll 4
                for (int m = m_first; m < M; m += m_step) {
                    float v = out_s[m * out_ld + tid];
                    if (rt) v = q80_roundtrip_warp(v);
                    if (live) {
                        if (res != nullptr) v += res[m * res_ld];
                        d0[m * ld] = v;
                    }
                }
            } else if (e.ll == 1) {
                // tensor-parallel push, LL words: value and epoch travel in one 8-byte store per peer; the consumer
                // polls the words themselves, so there is nothing to fence and no flag to release afterwards
                const uint32_t epoch = ld_volatile_u32(e.step_counter) * e.flag_mul + e.flag_add;
                for (int m = m_first; m < M; m += m_step) {
                    float v = out_s[m * out_ld + tid];
                    if (rt) v = q80_roundtrip_warp(v);
                    if (live) {
                        const size_t off = off0 + m * ld;
#pragma unroll 1
                        for (int p = 0; p < nd; p++) ll_store(e.dst[p], off, v, epoch);
                    }
                }
            } else if (e.ll == 2) {
                // tensor-parallel push in the reference's own wire format: Q80 blocks (int8 values + one fp16 scale per
                // 32, src/nn/nn-quants.hpp:64-72) instead of the f32 of their round trip -- 1.06 instead of 4 bytes per
                // value on NVLink, which is what bounds prompt-sized exchanges.  Row R = element offset / ld of the f32
                // layout; a wire row is ld int8 followed by ld/32 fp16 scales.  A warp = one 32-value block.
                const size_t rowb = (size_t)ld + (ld >> 4);
                const size_t row0 = ((size_t)e.dst_off + (size_t)m0 * ld) / ld;
                for (int m = m_first; m < M; m += m_step) {
                    const float v = out_s[m * out_ld + tid];
                    const float amax = warp_max(fabsf(v));
                    const float d = amax / 127.0f;
                    const float id = (d != 0.0f) ? (1.0f / d) : 0.0f;
                    const int q = __float2int_rn(v * id);
                    if (live) {
                        const size_t rb = (row0 + m) * rowb;
#pragma unroll 1
                        for (int p = 0; p < nd; p++) {
                            uint8_t* wrow = reinterpret_cast<uint8_t*>(e.dst[p]) + rb;
                            reinterpret_cast<int8_t*>(wrow)[grow] = (int8_t)q;
                            if (lane == 0) *reinterpret_cast<__half*>(wrow + ld + ((grow >> 5) << 1)) = __float2half_rn(d);
                        }
                    }
                }
            } else {
                for (int m = m_first; m < M; m += m_step) {
                    float v = out_s[m * out_ld + tid];
                    if (rt) v = q80_roundtrip_warp(v);
                    if (live) {
                        if (res != nullptr) v += res[m * res_ld];
                        const size_t off = off0 + m * ld;
#pragma unroll 1
                        for (int p = 0; p < nd; p++) e.dst[p][off] = v;
                    }
                }
            }
        }
    } else if (e.kind == DL_EPI_QKV_ROPE) {
        if (tid < rows) {
            const int grow = grow0 + tid;
            const int hs = e.head_size;
            const int region = (grow < e.q_dim) ? 0 : ((grow < e.q_dim + e.kv_dim) ? 1 : 2);   // warp-uniform
            const int rrow = (region == 0) ? grow : ((region == 1) ? grow - e.q_dim : grow - e.q_dim - e.kv_dim);
            const int hd = rrow % hs;
            const int kvh = rrow / hs;
            const bool live = grow < d_real;
            const float freq = (region < 2 && live) ? e.rope_freqs[hd >> 1] : 0.0f;
            // lane m fetches row m's position and (for k/v rows) its KV page; shuffled to the warp below
            int my_pos = 0, my_page = 0;
            if (lane < M) {
                my_pos = e.pos[m0 + lane];
                if (region != 0) my_page = e.block_table[(size_t)e.slot[m0 + lane] * e.max_pages + my_pos / e.page_size];
            }
            const int page_size = e.page_size, n_kv = e.n_kv_heads, q_dim = e.q_dim;
            float* q_out = e.q_out + (size_t)m0 * q_dim + rrow;
            void* base = (region == 1) ? e.k_cache : e.v_cache;
            const bool kv_f32 = e.kv_f32 != 0;
#pragma unroll 2
            for (int m = m_first; m < M; m += m_step) {
                float v = out_s[m * out_ld + tid];
                const int p = __shfl_sync(0xffffffffu, my_pos, m);
                const int page = __shfl_sync(0xffffffffu, my_page, m);
                if (region < 2) {
                    float other = __shfl_xor_sync(0xffffffffu, v, 1);
                    float sn, cs;
                    sincosf((float)p * freq, &sn, &cs);
                    // even lane holds x0, odd lane holds x1
                    v = (lane & 1) ? (other * sn + v * cs) : (v * cs - other * sn);
                }
                if (!live) {
                    // padded row: nothing to store
                } else if (region == 0) {
                    q_out[(size_t)m * q_dim] = v;
                } else {
                    const size_t off = (((size_t)page * n_kv + kvh) * page_size + (p % page_size)) * hs + hd;
                    if (kv_f32) reinterpret_cast<float*>(base)[off] = v;
                    else reinterpret_cast<__half*>(base)[off] = __float2half_rn(v);
                }
            }
        }
    } else if (e.kind == DL_EPI_DENSE) {
        // dense-weight models: an element-wise op on the f32 result, then a plain store (one destination)
        if (e.dense_op == DL_DENSE_GLU_CLAMP || e.dense_op == DL_DENSE_GLU_SILU || e.dense_op == DL_DENSE_GLU_GELU) {
            // output rows interleaved (gate_j, up_j): thread j < rows/2 owns value j of the tile and stores column
            // grow0 / 2 + j:  a = min(gate, limit), b = clamp(up, +-limit), hidden = a * sigma(1.702 a) * (1 + b)
            const int col = (grow0 >> 1) + tid;
            if (tid < (rows >> 1) && 2 * col + 1 < d_real) {
                const size_t ld = (size_t)e.ld;
                float* d0 = e.dst[0] + (size_t)e.dst_off + (size_t)m0 * ld + col;
                const float lim = e.dense_param;
                uint8_t* xh = e.dense_xh;                              // the next product's bf16 activation image instead of f32 rows
                const bool silu = e.dense_op == DL_DENSE_GLU_SILU;      // silu(gate) * up, no clamps
                const bool gelu = e.dense_op == DL_DENSE_GLU_GELU;      // gelu_tanh(gate) * up
#pragma unroll 4
                for (int m = m_first; m < M; m += m_step) {
                    const float2 gu = *reinterpret_cast<const float2*>(out_s + m * out_ld + 2 * tid);
                    float g = gu.x, u = gu.y;
                    if (silu) { d0[m * ld] = g / (1.0f + expf(-g)) * u; continue; }
                    if (gelu) {
                        const float v = act_gelu(g) * u;
                        if (xh != nullptr)      // element (row, col) of the slabs [K tile of 128][8 rows][8 columns]
                            *reinterpret_cast<__nv_bfloat16*>(xh + ((size_t)(col >> 7) * (e.dense_ncap >> 3) + ((m0 + m) >> 3)) * 2048 +
                                                              ((col & 127) >> 3) * 128 + ((m0 + m) & 7) * 16 + (col & 7) * 2) = __float2bfloat16_rn(v);
                        else d0[m * ld] = v;
                        continue;
                    }
                    if (lim > 0.0f) { g = fminf(g, lim); u = fminf(fmaxf(u, -lim), lim); }
                    d0[m * ld] = g / (1.0f + expf(-1.702f * g)) * (u + 1.0f);
                }
            }
        } else if (tid < rows) {
            const int grow = grow0 + tid;
            if (grow < d_real) {
                const size_t ld = (size_t)e.ld, ald = (size_t)e.dense_aux_ld;
                float* d0 = e.dst[0] + (size_t)e.dst_off + (size_t)m0 * ld + grow;
                const int op = e.dense_op;
                // one gate per row (ROWGATE_ADD) sits at aux[m * ald]; the other ops read aux[m * ald + column]
                const float* aux = e.dense_aux != nullptr ? e.dense_aux + (size_t)m0 * ald + (op == DL_DENSE_ROWGATE_ADD ? 0 : grow) : nullptr;
                const float prm = e.dense_param, prm2 = e.dense_param2;
                const float bias = e.dense_bias != nullptr ? e.dense_bias[grow] : 0.0f;
#pragma unroll 4
                for (int m = m_first; m < M; m += m_step) {
                    float v = out_s[m * out_ld + tid] + bias;
                    if (op == DL_DENSE_RELU2) { v = fmaxf(v, 0.0f); v *= v; }
                    else if (op == DL_DENSE_SIGMOID_MUL) v = aux[m * ald] / (1.0f + expf(-v));
                    else if (op == DL_DENSE_SOFTCAP) v = prm * tanhf(v / prm);
                    else if (op == DL_DENSE_SILU) v = v / (1.0f + expf(-v));
                    else if (op == DL_DENSE_MUL) v = aux[m * ald] * v;
                    else if (op == DL_DENSE_SCALE) v = prm * v;
                    else if (op == DL_DENSE_XIELU) v = v > 0.0f ? fmaf(prm * v, v, 0.5f * v) : fmaf(prm2, expm1f(v) - v, 0.5f * v);
                    else if (op == DL_DENSE_ROWGATE_ADD) v = fmaf(1.0f / (1.0f + expf(-aux[m * ald])), v, d0[m * ld]);
                    d0[m * ld] = v;
                }
            }
        }
    } else {   // DL_EPI_SILU_MUL: rows interleaved (gate_i, up_i); rows/2 hidden values per tile.
        // thread j < rows/2 owns hidden value j: reads local rows 2j, 2j+1; a warp = one Q80 block.
        const int nh = rows >> 1;
        const int hrow0 = grow0 >> 1;
        // d_real % 64 == 0 is required, so validity is uniform per 32-value block (= per warp)
        if (tid < nh && 2 * (hrow0 + (tid & ~31)) < d_real) {
            const bool gelu = e.act_gelu != 0;
            const int mcap = e.out_mcap;
            uint8_t* xq = e.xq_out;
            uint8_t* xh = e.xh_out;
#pragma unroll 2
            for (int m = m_first; m < M; m += m_step) {
                const float2 gu = *reinterpret_cast<const float2*>(out_s + m * out_ld + 2 * tid);
                float h = (gelu ? act_gelu(gu.x) : act_silu(gu.x)) * gu.y;
                q80_block_store(h, lane, m0 + m, (hrow0 + tid) >> 5, mcap, xq, xh);
            }
        }
    }
}

// The same by whole warps that share a tile, four and more consecutive output rows per thread: `warp` of `nw` takes activation rows
// (SiLU: blocks of 8 rows) in turn, ld(m, r) gives the products r .. r + 3 of activation row m (r a multiple of 4).  Nothing is exchanged
// between warps, so the caller needs no barrier but the one that makes ld's source complete.  after() is called once by every thread, behind its last ld.
// U: activation rows in flight per thread.
//
// What bounds it: instructions and the latency of each row's chain.  One value per thread and activation row at a time, half the threads idle
// on paired rows, five shuffles per block and 2-byte image stores (epilogue_rows), the epilogue of a 256 x 256 tile of gate|up took longer than its
// MMAs (4096 x 14336, 2048 rows: 447 us; without any epilogue work 360); here a block of 32 hidden values is four threads, whose image chunk
// is one 16-byte store, eight rows of them one line.
template <int U, class Ld, class After>
DL_DEVINL void epilogue_vec(const DlEpilogue& e, const Ld& ld, int grow0, int d_real, int M, int m0, int warp, int nw, const After& after) {
    const int lane = threadIdx.x & 31;
    if (e.kind == DL_EPI_SILU_MUL) {
        const int w = lane & 3, ml = lane >> 2, n_task = ((M + 7) >> 3) * 2;
        const bool gelu = e.act_gelu != 0;
        const int mcap = e.out_mcap;
        if (warp >= n_task) after();
        for (int t = warp; t < n_task; t += nw) {
            const int blk = t & 1, m = (t >> 1) * 8 + ml, mr = min(m, M - 1);
            // chunk w of the block's image: hidden values 4 w .. 4 w + 3 and 4 w + 16 .. 4 w + 19 (xh_slot)
            float4 x[4];
#pragma unroll
            for (int i = 0; i < 4; i++) x[i] = ld(mr, blk * 64 + (i >> 1) * 32 + 8 * w + (i & 1) * 4);
            if (t + nw >= n_task) after();
            float h[8], amax = 0.0f;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                h[2 * i] = (gelu ? act_gelu(x[i].x) : act_silu(x[i].x)) * x[i].y;
                h[2 * i + 1] = (gelu ? act_gelu(x[i].z) : act_silu(x[i].z)) * x[i].w;
                amax = fmaxf(amax, fmaxf(fabsf(h[2 * i]), fabsf(h[2 * i + 1])));
            }
            amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
            amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
            const float d = amax / 127.0f, id = (d != 0.0f) ? (1.0f / d) : 0.0f;
            const float df = fminf(__half2float(__float2half_rn(d)), 515.0f);      // saturation: q80_block_store
            __align__(16) __half o[8];
#pragma unroll
            for (int i = 0; i < 8; i++) o[(i & 4) + ((i & 3) == 1 ? 2 : (i & 3) == 2 ? 1 : (i & 3))] = __float2half_rn((float)__float2int_rn(h[i] * id) * df);
            if (m < M && grow0 + blk * 64 < d_real) {
                const int kblock = (grow0 >> 6) + blk;
                *reinterpret_cast<uint4*>(e.xh_out + ((size_t)(kblock >> 2) * (size_t)(mcap >> 3) + (size_t)((m0 + m) >> 3)) * XH_ROWGROUP_BYTES +
                                          ((kblock & 3) * 4 + w) * 128 + ((m0 + m) & 7) * 16) = *reinterpret_cast<const uint4*>(o);
            }
        }
        return;
    }
    const int r = lane * 4, grow = grow0 + r;
    const bool live = grow < d_real;                  // d_real is a multiple of 4
    if (warp >= M) after();
    if (e.kind == DL_EPI_STORE) {
        const bool rt = e.q80_roundtrip != 0;
        const float* res = e.residual;
        float* d0 = e.dst[0] + e.dst_off;
        for (int mb = warp; mb < M; mb += U * nw) {
            float4 v[U], x[U];
#pragma unroll
            for (int i = 0; i < U; i++)
                if (res != nullptr && live && mb + i * nw < M) x[i] = *reinterpret_cast<const float4*>(res + (size_t)(m0 + mb + i * nw) * e.residual_ld + grow);
#pragma unroll
            for (int i = 0; i < U; i++) v[i] = ld(min(mb + i * nw, M - 1), r);
            if (mb + U * nw >= M) after();
#pragma unroll
            for (int i = 0; i < U; i++) {
                if (rt) {                             // eight threads hold a block
                    float amax = fmaxf(fmaxf(fabsf(v[i].x), fabsf(v[i].y)), fmaxf(fabsf(v[i].z), fabsf(v[i].w)));
                    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
                    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
                    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 4));
                    const float d = amax / 127.0f, id = (d != 0.0f) ? (1.0f / d) : 0.0f, df = __half2float(__float2half_rn(d));
                    v[i].x = (float)__float2int_rn(v[i].x * id) * df; v[i].y = (float)__float2int_rn(v[i].y * id) * df;
                    v[i].z = (float)__float2int_rn(v[i].z * id) * df; v[i].w = (float)__float2int_rn(v[i].w * id) * df;
                }
                if (live && mb + i * nw < M) {
                    if (res != nullptr) { v[i].x += x[i].x; v[i].y += x[i].y; v[i].z += x[i].z; v[i].w += x[i].w; }
                    *reinterpret_cast<float4*>(d0 + (size_t)(m0 + mb + i * nw) * e.ld + grow) = v[i];
                }
            }
        }
    } else {                                          // DL_EPI_QKV_ROPE: two rotated pairs per thread
        const int region = (grow < e.q_dim) ? 0 : ((grow < e.q_dim + e.kv_dim) ? 1 : 2);
        const int rrow = (region == 0) ? grow : ((region == 1) ? grow - e.q_dim : grow - e.q_dim - e.kv_dim);
        const int hd = rrow % e.head_size, kvh = rrow / e.head_size;
        float2 freq = make_float2(0.0f, 0.0f);
        if (region < 2 && live) freq = make_float2(e.rope_freqs[hd >> 1], e.rope_freqs[(hd >> 1) + 1]);
        // lane i: position and page of this warp's i-th row
        int my_pos = 0, my_page = 0;
        if (warp + lane * nw < M) {
            my_pos = e.pos[m0 + warp + lane * nw];
            if (grow0 + 128 > e.q_dim) my_page = e.block_table[(size_t)e.slot[m0 + warp + lane * nw] * e.max_pages + my_pos / e.page_size];
        }
        void* base = (region == 1) ? e.k_cache : e.v_cache;
        for (int m = warp, i = 0; m < M; m += nw, i++) {
            float4 v = ld(m, r);
            if (m + nw >= M) after();
            const int p = __shfl_sync(0xffffffffu, my_pos, i), page = __shfl_sync(0xffffffffu, my_page, i);
            if (region < 2) {
                float sn, cs;
                sincosf((float)p * freq.x, &sn, &cs);
                v = make_float4(v.x * cs - v.y * sn, v.x * sn + v.y * cs, v.z, v.w);
                sincosf((float)p * freq.y, &sn, &cs);
                v = make_float4(v.x, v.y, v.z * cs - v.w * sn, v.z * sn + v.w * cs);
            }
            if (!live) continue;
            if (region == 0) {
                *reinterpret_cast<float4*>(e.q_out + (size_t)(m0 + m) * e.q_dim + rrow) = v;
            } else {
                const size_t off = (((size_t)page * e.n_kv_heads + kvh) * e.page_size + (p % e.page_size)) * e.head_size + hd;
                if (e.kv_f32) {
                    *reinterpret_cast<float4*>(reinterpret_cast<float*>(base) + off) = v;
                } else {
                    __half2 lo = __floats2half2_rn(v.x, v.y), hi = __floats2half2_rn(v.z, v.w);
                    *reinterpret_cast<uint2*>(reinterpret_cast<__half*>(base) + off) = make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
                }
            }
        }
    }
}
// a tile in shared memory, [m][ld]
struct EpiTile {
    const float* s;
    int ld;
    DL_DEVINL float4 operator()(int m, int r) const { return *reinterpret_cast<const float4*>(s + (size_t)m * ld + r); }
};
#define EPI_TILE_LD 132               // row stride of such a tile: 16-byte reads of two rows and four blocks of 8 (SiLU) without bank conflicts

// Does epilogue_vec take this epilogue?  One destination (what goes to peers keeps one word per thread: neighbouring words leave together),
// whole groups of four rows, 16-byte addresses; an fp16 image alone.
static inline bool epilogue_vec_ok(const DlEpilogue& e, int d) {
    const auto al = [](const void* p, long long ld) { return ((uintptr_t)p & 15) == 0 && ld % 4 == 0; };
    if (e.kind == DL_EPI_SILU_MUL) return e.xh_out != nullptr && e.xq_out == nullptr && ((uintptr_t)e.xh_out & 15) == 0 && d % 64 == 0;
    if (d % 4 != 0) return false;
    if (e.kind == DL_EPI_STORE) return e.n_dst == 1 && e.ll == 0 && al(e.dst[0], e.ld) && e.dst_off % 4 == 0 && (e.residual == nullptr || al(e.residual, e.residual_ld));
    return e.kind == DL_EPI_QKV_ROPE && al(e.q_out, e.q_dim) && al(e.k_cache, e.kv_dim) && al(e.v_cache, e.head_size);
}

// epilogue_complete: called by ALL threads of every CTA that ran epilogue_rows (uses __syncthreads).
// DL_EPI_STORE with flags: every CTA fences its (peer) stores, the last one releases the flags.
DL_DEVINL void epilogue_complete(const DlEpilogue& e, int tid, int n_epi_ctas, int* smem_flag) {
    if (e.kind != DL_EPI_STORE || e.flag[0] == nullptr) return;
    // Ordering chain (PTX memory model, cumulativity): every thread's peer stores -> bar.sync ->
    // thread 0: fence.sys + counter atomic -> (observed by the last CTA's thread 0) atomic + fence.sys
    // -> bar.sync -> st.release.sys of the flags.  One thread fences per CTA instead of all of them.
    __syncthreads();
    if (tid == 0) {
        __threadfence_system();
        unsigned prev = atomicAdd(e.cta_counter, 1u);
        const int last = (prev == (unsigned)n_epi_ctas - 1u) ? 1 : 0;
        if (last) {
            __threadfence_system();
            *e.cta_counter = 0u;
        }
        *smem_flag = last;
    }
    __syncthreads();
    if (*smem_flag && tid < e.n_dst) {
        uint32_t epoch = ld_volatile_u32(e.step_counter) * e.flag_mul + e.flag_add;
        st_release_sys(e.flag[tid], epoch);
    }
}
