// Weight preparation, activation producers (reduce + RMSNorm + Q80), embedding, argmax,
// error plumbing.
#include <stdarg.h>
#include <stdio.h>
#include <atomic>
#include <cstring>
#include <mutex>
#include "epilogue.cuh"
#include "waits.cuh"

static thread_local char g_err[512] = "";
void dl_set_error(const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
}
extern "C" const char* dl_last_error(void) { return g_err; }

// ---- limits of waits -----------------------------------------------------------------
// Words in host memory that kernels whose waits gave up write, one per device: the host reads them where it reads results, without a copy of their own.
static std::atomic<unsigned long long> g_wait_limit{WAIT_DEADLINE_NS};
static unsigned* wait_status_word(int dev = -1) {
    constexpr int devices = 64;
    static std::mutex lock;
    static std::atomic<unsigned*> words{nullptr};
    if ((dev < 0 && cudaGetDevice(&dev) != cudaSuccess) || dev >= devices) return nullptr;
    unsigned* w = words.load(std::memory_order_acquire);
    if (w != nullptr) return w + dev;
    std::lock_guard<std::mutex> guard(lock);
    if ((w = words.load()) == nullptr) {
        void* p = nullptr;
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;       // the first launch may be a captured one
        cudaThreadExchangeStreamCaptureMode(&mode);
        const cudaError_t e = cudaHostAlloc(&p, devices * sizeof(unsigned), cudaHostAllocPortable | cudaHostAllocMapped);
        cudaThreadExchangeStreamCaptureMode(&mode);
        if (e != cudaSuccess) { cudaGetLastError(); return nullptr; }
        words.store(w = (unsigned*)memset(p, 0, devices * sizeof(unsigned)), std::memory_order_release);
    }
    return w + dev;
}
extern "C" const unsigned* dl_attention_status() { return wait_status_word(); }
extern "C" void dl_debug_set_wait_limit(unsigned long long ns) { g_wait_limit = ns; }
int dl_wait_limit(const char* who, WaitLimit* l, int dev) {
    *l = {g_wait_limit, wait_status_word(dev)};
    if (l->status == nullptr) { dl_set_error("%s: no host memory for its status", who); return -1; }
    return 0;
}

// ---- optional launch timeline -----------------------------------------------------------------
static unsigned long long* g_trace_base = nullptr;
static int g_trace_cap = 0, g_trace_n = 0;
static int g_trace_kind[8192];
unsigned long long* dl_trace_next(int kind) {
    if (g_trace_base == nullptr || g_trace_n >= g_trace_cap || g_trace_n >= 8192) return nullptr;
    g_trace_kind[g_trace_n] = kind;
    return g_trace_base + 2 * (size_t)(g_trace_n++);
}
// buf: device array of 2*cap uint64, pre-filled by the caller with {UINT64_MAX, 0} pairs; NULL disables
extern "C" void dl_trace_set(unsigned long long* buf, int cap) { g_trace_base = buf; g_trace_cap = cap; g_trace_n = 0; }
extern "C" int dl_trace_count(void) { return g_trace_n; }
extern "C" int dl_trace_kind(int i) { return (i >= 0 && i < g_trace_n) ? g_trace_kind[i] : -1; }

#define CHECK_LAUNCH(name)                                                              \
    do {                                                                                \
        cudaError_t e__ = cudaGetLastError();                                           \
        if (e__ != cudaSuccess) {                                                       \
            dl_set_error("%s: %s", name, cudaGetErrorString(e__));                      \
            return -(int)e__;                                                           \
        }                                                                               \
    } while (0)

int dl_sm_count(int dev) {
    static std::atomic<int> counts[64];
    int n = 0;
    if (dev < 64 && (n = counts[dev].load(std::memory_order_relaxed)) > 0) return n;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return -1;
    if (dev < 64) counts[dev].store(n, std::memory_order_relaxed);
    return n;
}
extern "C" int dl_device_sm_count(void) {
    int dev = 0;
    return cudaGetDevice(&dev) == cudaSuccess ? dl_sm_count(dev) : -1;
}

// ------------------------------------------------------------------------------------------------
// Q40 file rows -> Q40T tiles
// ------------------------------------------------------------------------------------------------
extern "C" long long dl_q40t_bytes(int d, int n) {
    long long d_pad = ((long long)d + Q40T_TILE_ROWS - 1) / Q40T_TILE_ROWS * Q40T_TILE_ROWS;
    return d_pad / Q40T_TILE_ROWS * (long long)(n / Q40T_TILE_K) * Q40T_TILE_BYTES;
}

__global__ void q40_repack_kernel(const uint8_t* __restrict__ raw, int rows, int nb, uint8_t* __restrict__ out, int KT,
                                  int dst_row0, int dst_row_step) {
    // one thread per (source row, block); 18-byte source blocks are only 2-byte aligned
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)rows * nb) return;
    const int r = (int)(idx / nb), b = (int)(idx % nb);
    const uint16_t* src = reinterpret_cast<const uint16_t*>(raw + ((size_t)r * nb + b) * 18);
    uint16_t v[9];
#pragma unroll
    for (int i = 0; i < 9; i++) v[i] = src[i];
    const int drow = dst_row0 + r * dst_row_step;
    const int rt = drow >> 7, rr = drow & 127;
    const int kt = b >> 2, kb = b & 3;
    uint8_t* tile = out + ((size_t)rt * KT + kt) * Q40T_TILE_BYTES;
    uint4 q;
    q.x = (uint32_t)v[1] | ((uint32_t)v[2] << 16);
    q.y = (uint32_t)v[3] | ((uint32_t)v[4] << 16);
    q.z = (uint32_t)v[5] | ((uint32_t)v[6] << 16);
    q.w = (uint32_t)v[7] | ((uint32_t)v[8] << 16);
    *reinterpret_cast<uint4*>(tile + rr * 64 + (((kb + (rr >> 1)) & 3) << 4)) = q;
    *reinterpret_cast<uint16_t*>(tile + Q40T_SCALE_OFF + rr * 8 + kb * 2) = v[0];
}

extern "C" int dl_q40_repack(const uint8_t* raw, int rows, int n, uint8_t* q40t, int d_pad, int dst_row0,
                             int dst_row_step, void* stream) {
    if (n % Q40T_TILE_K != 0) { dl_set_error("dl_q40_repack: n=%d not a multiple of 128", n); return -1; }
    if (dst_row0 + (rows - 1) * dst_row_step >= d_pad) { dl_set_error("dl_q40_repack: rows exceed destination"); return -1; }
    const int nb = n / 32;
    const long long total = (long long)rows * nb;
    const int threads = 256;
    const unsigned blocks = (unsigned)((total + threads - 1) / threads);
    q40_repack_kernel<<<blocks, threads, 0, (cudaStream_t)stream>>>(raw, rows, nb, q40t, n / Q40T_TILE_K, dst_row0,
                                                                    dst_row_step);
    CHECK_LAUNCH("dl_q40_repack");
    return 0;
}

__global__ void q40t_dequant_kernel(const uint8_t* __restrict__ w, int d, int n, float* __restrict__ out) {
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;   // one thread per (row, block)
    const int nb = n / 32;
    if (idx >= (long long)d * nb) return;
    const int r = (int)(idx / nb), b = (int)(idx % nb);
    const int rt = r >> 7, rr = r & 127, kt = b >> 2, kb = b & 3;
    const uint8_t* tile = w + ((size_t)rt * (n / Q40T_TILE_K) + kt) * Q40T_TILE_BYTES;
    const uint8_t* q = tile + rr * 64 + (((kb + (rr >> 1)) & 3) << 4);
    const float dw = __half2float(*reinterpret_cast<const __half*>(tile + Q40T_SCALE_OFF + rr * 8 + kb * 2));
    float* o = out + (size_t)r * n + (size_t)b * 32;
    for (int j = 0; j < 16; j++) {
        o[j] = (float)((int)(q[j] & 0xF) - 8) * dw;
        o[j + 16] = (float)((int)(q[j] >> 4) - 8) * dw;
    }
}

extern "C" int dl_q40t_dequant(const uint8_t* q40t, int d, int n, float* out, void* stream) {
    const long long total = (long long)d * (n / 32);
    q40t_dequant_kernel<<<(unsigned)((total + 255) / 256), 256, 0, (cudaStream_t)stream>>>(q40t, d, n, out);
    CHECK_LAUNCH("dl_q40t_dequant");
    return 0;
}

// ------------------------------------------------------------------------------------------------
// embedding gather (+ per-forward step counter used as the epoch base of all peer flags)
// ------------------------------------------------------------------------------------------------
__global__ void embedding_kernel(const float* __restrict__ table, const int* __restrict__ tokens, float* __restrict__ x,
                                 int dim, uint32_t* step_counter, unsigned long long* tr) {
    trace_begin(tr);
    pdl_launch_dependents();
    pdl_wait();
    const int m = blockIdx.x;
    const float4* src = reinterpret_cast<const float4*>(table + (size_t)tokens[m] * dim);
    float4* dst = reinterpret_cast<float4*>(x + (size_t)m * dim);
    for (int i = threadIdx.x; i < dim / 4; i += blockDim.x) dst[i] = src[i];
    if (step_counter != nullptr && m == 0 && threadIdx.x == 0) *step_counter = *step_counter + 1u;
    trace_end(tr);
}

extern "C" int dl_embedding(const float* table, const int* tokens, float* x, int M, int dim, uint32_t* step_counter,
                            void* stream) {
    embedding_kernel<<<M, 256, 0, (cudaStream_t)stream>>>(table, tokens, x, dim, step_counter, dl_trace_next(TR_EMBED));
    CHECK_LAUNCH("dl_embedding");
    return 0;
}

// ------------------------------------------------------------------------------------------------
// reduce (merge-add of the peers' partial sums) + residual + RMSNorm + Q80 cast
// one CTA per activation row, or per 8 of them; dim <= 16384
// ------------------------------------------------------------------------------------------------
#define RNQ_THREADS 512
#define RNQ_MAX_PER_THREAD 32     // dim <= 512*32 = 16384
// From here on 8 rows per CTA, which takes a whole SM: 148 CTAs, one for every SM.  Below, fewer cannot pull as much (512 rows of 4096, the
// kernel alone: 6.7 us with a row per CTA, 10.2 with 8).  Above it goes by waves of 1184 rows: whole lines of the image win in full ones and a
// barely begun one loses (norm and feed-forward, us with a row per CTA and with 8: width 2048, 1184 rows 271 and 267, 1300 310 and 314, 1536
// 314 and 314, 2048 352 and 347; width 4096 567 and 561..566, 644 and 653, 657 and 661, 802..805 and 797..801; the kernel alone, 4096 wide,
// 1300 rows 18.5 and 26.6, 2048 25.4 and 26.7, 2368 28.8 and 26.8).
#define RNQ_WIDE_ROWS 1184

struct RnqArgs {
    const float* x_in;
    float* x_out;
    const float* partials;      // [n_src][mcap_p][dim] with src_stride elements between sources
    int n_src;
    long long src_stride;
    const uint32_t* flags;
    const uint32_t* step_counter;
    uint32_t flag_mul, flag_add;
    int ll;                     // partials are LL words {f32 bits, epoch}: poll the data, no flags
    const float* norm_w;
    float eps;
    int dim, M, mcap;
    uint8_t* xq_out;
    uint8_t* xh_out;
    float* y_out;
    unsigned long long* tr;
};

// Four lanes hold a 32-block: lane c its elements 4c .. 4c + 3 and 16 + 4c .. 16 + 4c + 3, which are one 16-byte chunk of the XH image.  A
// warp is 8 such blocks: of 8 rows side by side (ROWS = 8, many rows: a chunk of the 8 rows is one whole 128-byte line of the image), or
// 8 neighbouring blocks of one row (ROWS = 1: a CTA per row).  The merged row stays in registers between the two passes.
// What bounds it: bytes (x, partial sums, image) for many rows, latency for few.  With one thread per block, 128 bytes apart, 2048 rows of
// 4096 took 55.4 us alone, 512 rows 18.3; 25.4 (26.7 with 8 rows per CTA) and 9.3 with this.  32 rows are as fast either way (9 us).
// With 8 rows per CTA each block's loads waited behind the last one's: 2048 rows of 4096 26.4 us, 8192 53.6; 17.1 and 41.1 with all blocks of a
// thread in flight and the norm's weights one block ahead.  (One row per CTA: the same there costs registers, spills, and 1 us a launch.)
template <int ROWS>
__global__ void __launch_bounds__(RNQ_THREADS) reduce_norm_quant_kernel(const __grid_constant__ RnqArgs a) {
    trace_begin(a.tr);
    constexpr int NW = RNQ_THREADS / 32, KEEP = ROWS == 8 ? 8 : 4;
    __shared__ float s_part[NW][8];
    pdl_launch_dependents();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, c = lane & 3;
    const int r = ROWS == 8 ? lane >> 2 : 0, m = blockIdx.x * ROWS + r;
    const int nb = a.dim >> 5;
    const bool live = m < a.M;
    auto block_of = [&](int u) { return ROWS == 8 ? warp + u * NW : (warp + u * NW) * 8 + (lane >> 2); };
    pdl_wait();
    if (a.flags != nullptr && a.n_src > 0) {
        if (tid < a.n_src) {
            const uint32_t epoch = ld_volatile_u32(a.step_counter) * a.flag_mul + a.flag_add;
            wait_flag_ge(a.flags + tid, epoch);
        }
        __syncthreads();
    }
    const int ll = (a.ll == 1) ? 1 : 0;
    const bool wire = a.ll == 2;      // partials are Q80 wire rows: dim int8 + dim/32 fp16 scales (see epilogue.cuh)
    const size_t rowb = (size_t)a.dim + (a.dim >> 4);
    const size_t src_rows = (size_t)a.src_stride / a.dim;
    const uint32_t ll_epoch = ll ? ld_volatile_u32(a.step_counter) * a.flag_mul + a.flag_add : 0u;
    const size_t row = (size_t)m * a.dim;
    auto add_partial = [&](int s, int b, int h, float4& v) {
        const int e = b * 32 + h * 16 + c * 4;
        float4 p;
        if (wire) {
            const uint8_t* wr = reinterpret_cast<const uint8_t*>(a.partials) + ((size_t)s * src_rows + m) * rowb;
            const int q4 = *reinterpret_cast<const int*>(wr + e);
            const float d = __half2float(*reinterpret_cast<const __half*>(wr + a.dim + (b << 1)));
            p = make_float4((float)(int8_t)(q4 & 0xff) * d, (float)(int8_t)((q4 >> 8) & 0xff) * d,
                            (float)(int8_t)((q4 >> 16) & 0xff) * d, (float)(q4 >> 24) * d);
        } else {
            p = part_load4(a.partials, (size_t)s * a.src_stride + row + e, ll, ll_epoch);
        }
        v.x += p.x; v.y += p.y; v.z += p.z; v.w += p.w;
    };
    auto load = [&](int b, int h) { return *reinterpret_cast<const float4*>(a.x_in + row + b * 32 + h * 16 + c * 4); };
    auto merged = [&](int b, float4 (&v)[2]) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
            v[h] = load(b, h);
            for (int s = 0; s < a.n_src; s++) add_partial(s, b, h, v[h]);
        }
    };
    // pass 1: merged residual -> x_out, sum of squares
    float4 keep[KEEP][2];
    float ss = 0.0f;
    auto first = [&](int b, const float4 (&v)[2]) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
            if (a.x_out != nullptr) *reinterpret_cast<float4*>(a.x_out + row + b * 32 + h * 16 + c * 4) = v[h];
            ss += v[h].x * v[h].x + v[h].y * v[h].y + v[h].z * v[h].z + v[h].w * v[h].w;
        }
    };
    if (ROWS == 8) {                  // a thread's blocks are in flight together (one row per CTA: a thread has one block of up to 4096 columns)
#pragma unroll
        for (int u = 0; u < KEEP; u++) {
#pragma unroll
            for (int h = 0; h < 2; h++) keep[u][h] = live && block_of(u) < nb ? load(block_of(u), h) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        for (int s = 0; s < a.n_src; s++)
#pragma unroll
            for (int u = 0; u < KEEP; u++)
#pragma unroll
                for (int h = 0; h < 2; h++)
                    if (live && block_of(u) < nb) add_partial(s, block_of(u), h, keep[u][h]);
#pragma unroll
        for (int u = 0; u < KEEP; u++)
            if (live && block_of(u) < nb) first(block_of(u), keep[u]);
    } else {
#pragma unroll
        for (int u = 0; u < KEEP; u++)
            if (live && block_of(u) < nb) {
                merged(block_of(u), keep[u]);
                first(block_of(u), keep[u]);
            }
    }
    for (int u = KEEP; live && block_of(u) < nb; u++) {
        float4 v[2];
        merged(block_of(u), v);
        first(block_of(u), v);
    }
    float inv = 1.0f;
    float4 wn[2];
    if (a.norm_w != nullptr) {
        if (ROWS == 8 && live && block_of(0) < nb)
#pragma unroll
            for (int h = 0; h < 2; h++) wn[h] = *reinterpret_cast<const float4*>(a.norm_w + block_of(0) * 32 + h * 16 + c * 4);
        ss += __shfl_xor_sync(0xffffffffu, ss, 1);
        ss += __shfl_xor_sync(0xffffffffu, ss, 2);
        if (c == 0) s_part[warp][lane >> 2] = ss;
        __syncthreads();
        float t = 0.0f;
        if (ROWS == 8) {              // lane (r, c) sums the warps c, c + 4, ... of row r
#pragma unroll
            for (int w = 0; w < NW; w += 4) t += s_part[w + c][r];
            t += __shfl_xor_sync(0xffffffffu, t, 1);
            t += __shfl_xor_sync(0xffffffffu, t, 2);
        } else {
#pragma unroll
            for (int w = 0; w < NW * 8; w += 32) t += (&s_part[0][0])[w + lane];
            t = warp_sum(t);
        }
        inv = 1.0f / sqrtf(t / (float)a.dim + a.eps);
    }
    // pass 2: norm, Q80
    auto weight = [&](int b, int h) { return *reinterpret_cast<const float4*>(a.norm_w + b * 32 + h * 16 + c * 4); };
    auto second = [&](int b, bool on, float4 (&v)[2], auto w_of) {
        float amax = 0.0f;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            if (a.norm_w != nullptr && on) {
                const float4 w4 = w_of(h);
                v[h].x = w4.x * (inv * v[h].x); v[h].y = w4.y * (inv * v[h].y);
                v[h].z = w4.z * (inv * v[h].z); v[h].w = w4.w * (inv * v[h].w);
            }
            amax = fmaxf(amax, fmaxf(fmaxf(fabsf(v[h].x), fabsf(v[h].y)), fmaxf(fabsf(v[h].z), fabsf(v[h].w))));
            if (a.y_out != nullptr && on) *reinterpret_cast<float4*>(a.y_out + row + b * 32 + h * 16 + c * 4) = v[h];
        }
        if (a.xq_out == nullptr && a.xh_out == nullptr) return;
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
        const float d = amax / 127.0f;
        const float id = (d != 0.0f) ? (1.0f / d) : 0.0f;
        const float df = __half2float(__float2half_rn(d));
        int q[2][4];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            q[h][0] = __float2int_rn(v[h].x * id); q[h][1] = __float2int_rn(v[h].y * id);
            q[h][2] = __float2int_rn(v[h].z * id); q[h][3] = __float2int_rn(v[h].w * id);
        }
        const int kt = b >> 2, kb = b & 3;
        if (a.xq_out != nullptr) {
            int sumq = q[0][0] + q[0][1] + q[0][2] + q[0][3] + q[1][0] + q[1][1] + q[1][2] + q[1][3];
            sumq += __shfl_xor_sync(0xffffffffu, sumq, 1);
            sumq += __shfl_xor_sync(0xffffffffu, sumq, 2);
            if (on) {
                uint8_t* rowp = a.xq_out + ((size_t)kt * a.mcap + m) * XQ_ROW_BYTES;
#pragma unroll
                for (int h = 0; h < 2; h++)
                    *reinterpret_cast<uint32_t*>(rowp + kb * 32 + h * 16 + c * 4) = (uint32_t)(q[h][0] & 0xff) | ((uint32_t)(q[h][1] & 0xff) << 8) |
                                                                                    ((uint32_t)(q[h][2] & 0xff) << 16) | ((uint32_t)(q[h][3] & 0xff) << 24);
                if (c == 0) {
                    reinterpret_cast<float*>(rowp + 128)[kb] = df;
                    reinterpret_cast<int*>(rowp + 144)[kb] = 8 * sumq;
                }
            }
        }
        if (a.xh_out != nullptr && on) {
            // chunk c holds elements [4c, 4c+2, 4c+1, 4c+3, 4c+16, 4c+18, 4c+17, 4c+19] (see xh_slot)
            const float dfh = fminf(df, 515.0f);       // fp16 operand: saturate (|x| > 65405) instead of producing inf
            uint32_t w[4];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                __half2 h0 = __floats2half2_rn((float)q[h][0] * dfh, (float)q[h][2] * dfh), h1 = __floats2half2_rn((float)q[h][1] * dfh, (float)q[h][3] * dfh);
                w[2 * h] = *reinterpret_cast<uint32_t*>(&h0);
                w[2 * h + 1] = *reinterpret_cast<uint32_t*>(&h1);
            }
            *reinterpret_cast<uint4*>(a.xh_out + ((size_t)kt * (size_t)(a.mcap >> 3) + (size_t)(m >> 3)) * XH_ROWGROUP_BYTES + (size_t)(kb * 4 + c) * 128 +
                                      (size_t)(m & 7) * 16) = make_uint4(w[0], w[1], w[2], w[3]);
        }
    };
#pragma unroll
    for (int u = 0; u < KEEP; u++) {
        const bool on = live && block_of(u) < nb;
        if (!on) keep[u][0] = keep[u][1] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (ROWS == 8) {
            const float4 w[2] = {wn[0], wn[1]};
            if (a.norm_w != nullptr && u + 1 < KEEP && live && block_of(u + 1) < nb) {      // on their way while this block is cast
                wn[0] = weight(block_of(u + 1), 0);
                wn[1] = weight(block_of(u + 1), 1);
            }
            if (__any_sync(0xffffffffu, on)) second(block_of(u), on, keep[u], [&](int h) { return w[h]; });
        } else if (__any_sync(0xffffffffu, on)) {
            second(block_of(u), on, keep[u], [&](int h) { return weight(block_of(u), h); });
        }
    }
    for (int u = KEEP; ROWS == 8 ? block_of(u) < nb : (warp + u * NW) * 8 < nb; u++) {
        const bool on = live && block_of(u) < nb;
        float4 v[2] = {make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)};
        if (on) merged(block_of(u), v);
        second(block_of(u), on, v, [&](int h) { return weight(block_of(u), h); });
    }
    trace_end(a.tr);
}

extern "C" int dl_reduce_norm_quant(const float* x_in, float* x_out, const float* partials, int n_src, int src_stride,
                                    const uint32_t* flags, const uint32_t* step_counter, uint32_t flag_mul,
                                    uint32_t flag_add, int ll, const float* norm_w, float eps, int dim, int M, int mcap,
                                    uint8_t* xq_out, uint8_t* xh_out, float* y_out, int pdl, void* stream) {
    if (dim % 32 != 0 || dim > RNQ_THREADS * RNQ_MAX_PER_THREAD) { dl_set_error("dl_reduce_norm_quant: bad dim %d", dim); return -1; }
    if (n_src > DL_MAX_PEERS) { dl_set_error("dl_reduce_norm_quant: n_src > 8"); return -1; }
    RnqArgs a;
    a.x_in = x_in; a.x_out = x_out; a.partials = partials; a.n_src = n_src; a.src_stride = src_stride;
    a.flags = flags; a.step_counter = step_counter; a.flag_mul = flag_mul; a.flag_add = flag_add; a.ll = ll;
    a.norm_w = norm_w; a.eps = eps; a.dim = dim; a.M = M; a.mcap = mcap;
    a.xq_out = xq_out; a.xh_out = xh_out; a.y_out = y_out;
    a.tr = dl_trace_next(TR_RNQ);
    cudaLaunchConfig_t cfg = {};
    const bool wide = M >= RNQ_WIDE_ROWS;
    cfg.gridDim = dim3(wide ? (M + 7) / 8 : M);
    cfg.blockDim = dim3(RNQ_THREADS);
    cfg.stream = (cudaStream_t)stream;
    cudaLaunchAttribute attr[1];
    if (pdl) {
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
    }
    cudaError_t e = wide ? cudaLaunchKernelEx(&cfg, reduce_norm_quant_kernel<8>, a) : cudaLaunchKernelEx(&cfg, reduce_norm_quant_kernel<1>, a);
    if (e != cudaSuccess) { dl_set_error("dl_reduce_norm_quant: %s", cudaGetErrorString(e)); return -(int)e; }
    return 0;
}

extern "C" int dl_quant_q80(const float* x, int M, int K, int mcap, uint8_t* xq_out, uint8_t* xh_out, void* stream) {
    // the same kernel with no residual/partials/norm: y = x
    return dl_reduce_norm_quant(x, nullptr, nullptr, 0, 0, nullptr, nullptr, 0, 0, 0, nullptr, 0.0f, K, M, mcap, xq_out,
                                xh_out, nullptr, 0, stream);
}

// ------------------------------------------------------------------------------------------------
// greedy sampling on device (+ optional wait for the peers' logits slices, + device-resident
// decode loop support: feed the token back, advance the position, record a history)
// ------------------------------------------------------------------------------------------------
struct ArgmaxArgs {
    const float* logits;
    int vocab, ld;
    int* tokens_out;
    const uint32_t* flags;
    int n_flags;
    const uint32_t* step_counter;
    uint32_t flag_mul, flag_add;
    int* pos_inc;
    int* history;
    int history_cap;
    uint8_t* scratch;
    unsigned long long* tr;
};

#define ARGMAX_CHUNKS 32
#define ARGMAX_THREADS 256

DL_DEVINL void argmax_combine(float& best, int& bi, float ov, int oi) {
    if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
}

// grid (ARGMAX_CHUNKS, M): every CTA reduces one vocabulary chunk; the last CTA of a row (self-
// resetting counter in scratch) reduces the chunk winners and publishes the token.
__global__ void __launch_bounds__(ARGMAX_THREADS) argmax_kernel(const __grid_constant__ ArgmaxArgs a) {
    __shared__ float s_v[ARGMAX_THREADS / 32];
    __shared__ int s_i[ARGMAX_THREADS / 32];
    __shared__ int s_last;
    trace_begin(a.tr);
    pdl_launch_dependents();
    pdl_wait();
    if (a.flags != nullptr) {
        if ((int)threadIdx.x < a.n_flags) {
            const uint32_t epoch = ld_volatile_u32(a.step_counter) * a.flag_mul + a.flag_add;
            wait_flag_ge(a.flags + threadIdx.x, epoch);
        }
        __syncthreads();
    }
    const int m = blockIdx.y, ch = blockIdx.x, M = gridDim.y;
    unsigned* counters = reinterpret_cast<unsigned*>(a.scratch);                       // [M]
    float* part_v = reinterpret_cast<float*>(a.scratch + 1024);                        // [M][CHUNKS]
    int* part_i = reinterpret_cast<int*>(a.scratch + 1024 + (size_t)M * ARGMAX_CHUNKS * 4);
    const int per = ((a.vocab + ARGMAX_CHUNKS - 1) / ARGMAX_CHUNKS + 3) & ~3;
    const int i0 = ch * per, i1 = min(a.vocab, i0 + per);
    const float* row = a.logits + (size_t)m * a.ld;
    float best = -INFINITY;
    int bi = 0x7fffffff;
    for (int i = i0 + threadIdx.x; i < i1; i += ARGMAX_THREADS) argmax_combine(best, bi, row[i], i);
    for (int o = 16; o > 0; o >>= 1)
        argmax_combine(best, bi, __shfl_xor_sync(0xffffffffu, best, o), __shfl_xor_sync(0xffffffffu, bi, o));
    if ((threadIdx.x & 31) == 0) { s_v[threadIdx.x >> 5] = best; s_i[threadIdx.x >> 5] = bi; }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < ARGMAX_THREADS / 32; w++) argmax_combine(best, bi, s_v[w], s_i[w]);
        part_v[m * ARGMAX_CHUNKS + ch] = best;
        part_i[m * ARGMAX_CHUNKS + ch] = bi;
        __threadfence();
        const unsigned prev = atomicAdd(&counters[m], 1u);
        s_last = (prev == ARGMAX_CHUNKS - 1) ? 1 : 0;
        if (s_last) counters[m] = 0u;
    }
    __syncthreads();
    if (!s_last) { trace_end(a.tr); return; }
    if (threadIdx.x < 32) {
        __threadfence();
        best = __ldcg(&part_v[m * ARGMAX_CHUNKS + threadIdx.x]);
        bi = __ldcg(&part_i[m * ARGMAX_CHUNKS + threadIdx.x]);
        for (int o = 16; o > 0; o >>= 1)
            argmax_combine(best, bi, __shfl_xor_sync(0xffffffffu, best, o), __shfl_xor_sync(0xffffffffu, bi, o));
        if (threadIdx.x == 0) {
            if (bi == 0x7fffffff) bi = 0;      // all-NaN row: stay in range
            a.tokens_out[m] = bi;
            if (a.pos_inc != nullptr) a.pos_inc[m] += 1;
            if (a.history != nullptr) {
                const uint32_t c = ld_volatile_u32(a.step_counter);
                a.history[(size_t)((c - 1u) % (uint32_t)a.history_cap) * M + m] = bi;
            }
        }
    }
    trace_end(a.tr);
}

extern "C" long long dl_argmax_scratch_bytes(int M) { return 1024 + (long long)M * ARGMAX_CHUNKS * 8; }

extern "C" int dl_argmax(const float* logits, int M, int vocab, int ld, int* tokens_out, const uint32_t* flags,
                         int n_flags, const uint32_t* step_counter, uint32_t flag_mul, uint32_t flag_add, int* pos_inc,
                         int* history, int history_cap, void* scratch, int pdl, void* stream) {
    static_assert(ARGMAX_CHUNKS == 32, "final reduce assumes one warp of chunk winners");
    ArgmaxArgs a;
    a.logits = logits; a.vocab = vocab; a.ld = ld; a.tokens_out = tokens_out;
    a.flags = flags; a.n_flags = n_flags; a.step_counter = step_counter; a.flag_mul = flag_mul; a.flag_add = flag_add;
    a.pos_inc = pos_inc; a.history = history; a.history_cap = history_cap;
    a.scratch = reinterpret_cast<uint8_t*>(scratch);
    a.tr = dl_trace_next(TR_ARGMAX);
    if (history != nullptr && step_counter == nullptr) { dl_set_error("dl_argmax: history needs step_counter"); return -1; }
    if (scratch == nullptr) { dl_set_error("dl_argmax: needs zero-initialised scratch (dl_argmax_scratch_bytes(min(M, 256)))"); return -1; }
    if (M > 256 && history != nullptr) { dl_set_error("dl_argmax: the device-loop history supports M <= 256"); return -1; }
    // the scratch holds 256 rows of counters and chunk winners: larger batches go through it 256 rows at a time
    // (launches on one stream run in order, and the counters return to zero)
    for (int m0 = 0; m0 < M; m0 += 256) {
        const int mb = (M - m0 < 256) ? M - m0 : 256;
        a.logits = logits + (size_t)m0 * ld;
        a.tokens_out = tokens_out + m0;
        a.pos_inc = pos_inc != nullptr ? pos_inc + m0 : nullptr;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(ARGMAX_CHUNKS, mb);
        cfg.blockDim = dim3(ARGMAX_THREADS);
        cfg.stream = (cudaStream_t)stream;
        cudaLaunchAttribute attr[1];
        if (pdl && m0 == 0) {
            attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            attr[0].val.programmaticStreamSerializationAllowed = 1;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
        }
        cudaError_t e = cudaLaunchKernelEx(&cfg, argmax_kernel, a);
        if (e != cudaSuccess) { dl_set_error("dl_argmax: %s", cudaGetErrorString(e)); return -(int)e; }
    }
    return 0;
}

// ------------------------------------------------------------------------------------------------
// dl_argmax_noalloc: greedy pick for callers that must not allocate device memory.
//
// Who this is for: code that runs where cudaMalloc is off limits -- a plugin inside a host
// application that owns the whole memory budget, a latency-critical serving loop that forbids
// allocator calls after start-up, or a caller that only holds raw pointers and no allocator at
// all.  dl_argmax() needs a caller-provided scratch buffer (chunk winners + completion counters);
// this variant keeps that scratch in a fixed array inside the library instead, so the caller
// passes nothing but its logits and its output.
//
// Limits and rules:
//  * at most DL_ARGMAX_NOALLOC_MAX_ROWS (64) rows per call; larger M is refused with an error.
//    The array (17 KB) is part of the loaded module: every GPU that loads this library holds it
//    until the process exits.
//  * the first call on each device resolves the array's device address (cudaGetSymbolAddress, with
//    that device current).  Make that first call before starting any stream capture.
//  * all calls on a device share the one array: two calls whose kernels may overlap on the GPU
//    (different streams, no ordering between them) race on it.  Serialise them.
//  * the array keeps whatever the previous call left; the counters the kernel relies on being zero
//    are cleared on the caller's stream at the start of every call (cudaMemsetAsync, no allocation).
//  * no cudaMalloc / cudaFree / allocating library routine is called, here or in the kernel.
// ------------------------------------------------------------------------------------------------
#define DL_ARGMAX_NOALLOC_MAX_ROWS 64
#define DL_ARGMAX_NOALLOC_BYTES (1024 + DL_ARGMAX_NOALLOC_MAX_ROWS * ARGMAX_CHUNKS * 8)
static __device__ __align__(256) unsigned char g_argmax_noalloc_scratch[DL_ARGMAX_NOALLOC_BYTES];

extern "C" int dl_argmax_noalloc(const float* logits, int M, int vocab, int ld, int* tokens_out, void* stream) {
    // In host code `g_argmax_noalloc_scratch` is only a handle for the runtime, not a device address:
    // the real address is looked up once per device and cached here.
    static unsigned char* dev_addr[64] = {nullptr};
    if (M < 1 || M > DL_ARGMAX_NOALLOC_MAX_ROWS) {
        dl_set_error("dl_argmax_noalloc: M=%d is outside 1..%d (the built-in scratch is sized for %d rows; use "
                     "dl_argmax with your own scratch for more)", M, DL_ARGMAX_NOALLOC_MAX_ROWS, DL_ARGMAX_NOALLOC_MAX_ROWS);
        return -1;
    }
    if (logits == nullptr || tokens_out == nullptr || vocab < 1 || ld < vocab) {
        dl_set_error("dl_argmax_noalloc: bad arguments (logits/tokens_out NULL, vocab < 1 or ld < vocab)");
        return -1;
    }
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || dev < 0 || dev >= 64) {
        dl_set_error("dl_argmax_noalloc: cudaGetDevice: %s", e != cudaSuccess ? cudaGetErrorString(e) : "device index out of range");
        return e != cudaSuccess ? -(int)e : -1;
    }
    if (dev_addr[dev] == nullptr) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_argmax_noalloc_scratch);
        if (e != cudaSuccess || p == nullptr) {
            dl_set_error("dl_argmax_noalloc: cudaGetSymbolAddress: %s", cudaGetErrorString(e));
            return e != cudaSuccess ? -(int)e : -1;
        }
        dev_addr[dev] = reinterpret_cast<unsigned char*>(p);
    }
    unsigned char* scratch = dev_addr[dev];
    // completion counters (first 1 KB) must be zero when the kernel starts
    e = cudaMemsetAsync(scratch, 0, 1024, (cudaStream_t)stream);
    if (e != cudaSuccess) { dl_set_error("dl_argmax_noalloc: cudaMemsetAsync: %s", cudaGetErrorString(e)); return -(int)e; }
    ArgmaxArgs a;
    a.logits = logits; a.vocab = vocab; a.ld = ld; a.tokens_out = tokens_out;
    a.flags = nullptr; a.n_flags = 0; a.step_counter = nullptr; a.flag_mul = 0; a.flag_add = 0;
    a.pos_inc = nullptr; a.history = nullptr; a.history_cap = 0;
    a.scratch = scratch;
    a.tr = nullptr;
    argmax_kernel<<<dim3(ARGMAX_CHUNKS, M), ARGMAX_THREADS, 0, (cudaStream_t)stream>>>(a);
    e = cudaGetLastError();
    if (e != cudaSuccess) { dl_set_error("dl_argmax_noalloc: launch: %s", cudaGetErrorString(e)); return -(int)e; }
    return 0;
}

// wait until flags[i] >= epoch for i < n (orders later stream work after the peers' pushes)
__global__ void wait_flags_kernel(const uint32_t* flags, int n, const uint32_t* step_counter, uint32_t mul, uint32_t add) {
    pdl_launch_dependents();
    pdl_wait();
    if ((int)threadIdx.x < n) {
        const uint32_t epoch = ld_volatile_u32(step_counter) * mul + add;
        wait_flag_ge(flags + threadIdx.x, epoch);
    }
}

extern "C" int dl_wait_flags(const uint32_t* flags, int n, const uint32_t* step_counter, uint32_t flag_mul,
                             uint32_t flag_add, void* stream) {
    wait_flags_kernel<<<1, 32, 0, (cudaStream_t)stream>>>(flags, n, step_counter, flag_mul, flag_add);
    CHECK_LAUNCH("dl_wait_flags");
    return 0;
}
