// Causal attention for long prompt chunks on the 5th-gen tensor cores (head size 128): the same job as
// attention_prefill.cu (segments of consecutive positions of one sequence, listed in `meta`), with both products
// as tcgen05.mma and the score / probability / output tiles in TENSOR MEMORY instead of registers.
//
// A CTA owns 128 query rows x one query head and walks the KV history 128 tokens (four pages) at a time:
//   S = Q K^T     SS-mode MMA, M = 128 rows, N = 128 tokens, K = 128: Q staged once (fp16, K-major, 128-byte swizzle);
//                 K pages arrive by TMA tensor copies (cp.async.bulk.tensor.2d over this GPU's KV cache, box 64 x 32,
//                 hardware 128-byte swizzle); S (f32) lands in TMEM, double-buffered
//   softmax       two threads per query row (= TMEM lane), 64 score columns each, read into registers with tcgen05.ld
//                 in one pass (the score buffer is handed back at once); the row maximum is exchanged through shared
//                 memory; exp2 -> fp16 probabilities written back to TMEM with tcgen05.st (every fourth exp2 on the
//                 FMA pipe: the step is MUFU-bound); running maximum with LAZY rescaling: the reference maximum only
//                 moves when a row's maximum grew by more than 2^8, so in the steady state the output accumulator is
//                 never touched by the softmax threads
//   O += P V      TS-mode MMA: A = P straight from TMEM, B = V pages in shared memory as an MN-major operand (V is
//                 [token][head dim] in the cache, i.e. N-contiguous: no transpose anywhere), accumulating in TMEM
// S(j+1) and S(j+2) are issued while the softmax threads are busy with step j, so the tensor core works ahead of them.  Output: O / l -> shared memory -> Q80 cast into the XQ / XH slabs of the wo matmul.
//
// Warp roles (384 threads): warp 0 issues the S MMAs (+ TMEM owner), warp 6 the P V MMAs (an issuing thread spends ~700 clk
// per group of 8 MMAs, so one thread for both would cap a step at ~1500 clk), warps 1-4 and 8-11 softmax (two threads per
// row = TMEM lane, 64 columns each; the row maximum is exchanged through shared memory), warp 5
// K producer and warp 7 V producer (one lane each issues 8 tensor copies of 4 KB per step: 4 pages x 2 halves of the head
// dimension; K and V have their own 3-stage rings, so a K stage is free again as soon as its scores are complete).
// (The first version copied K/V with cp.async in 16-byte pieces into un-swizzled core matrices: 4096 LDGSTS per step
// cost 3500 clk of issue time, three times the MMAs -- scripts/trace_attention_tc.py.)
// TMEM columns: S0 [0,128) S1 [128,256) P0 [256,320) P1 [320,384) O [384,512).
//
// The second instance (LINES) serves layer-list models: bf16 cache lines [key 128 | value 128], tiles of up to rq consecutive positions
// of one sequence whose query heads of one key/value head stack on the MMA's rows (row = position * rep + head), so two neighbouring
// tiles of 64 stacked rows fill the 128 lanes; window or chunk masks (only the steps that a tile sees are walked), soft cap, distance
// bias, sink, gate; f32 output.  Probabilities are two bf16 numbers each, the second the first one's remainder, and P V two MMAs: rounded to
// one (2^-9) they are the larger share of the error, and how large depends on how often a row's maximum, whose probability is exact, moves
// -- every 32 tokens in the mma.sync kernel, every 128 here (2000 tokens under a window of 1024, against 64 bits: 1.929e-3 with one number,
// 1.926e-3 there, 1.50e-3 with two; 1300 tokens: 2.19e-3, 2.17e-3, 1.64e-3; the time is the same).  The remainders lie in the score buffer that they
// came from, so S of step j + 2 waits for P V of step j.  mma.sync with its 64-row tiles took 142 us for 2000 rows of 16 heads on 4 under a window of 1024
// (88 TFLOP/s); 55 us here.
//
// Reference semantics: multiheadAtt_F32 (src/nn/nn-cpu-ops.cpp:749-784), softmax in f32, output cast as OP_CAST
// (src/llm.cpp:296-301).  KV cache: fp16 pages [page][kv_head][32][128].
#include <cuda.h>
#include "epilogue.cuh"
#include "window_tiles.cuh"

#define PT_HS 128
#define PT_ROWS 128
#define PT_KV 128                      // tokens per step
#define PT_THREADS 384
#define PT_MAX_SEG 8
#define PT_TILE_BYTES 32768            // 128 x 128 fp16
#define PT_STAGES 3                    // KV tiles in flight (K + V: 64 KB each)
#define PT_OUT_LD 129
#define PT_DEADLINE_NS 4000000000ull

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
    long long* stamps;         // debug: clock64 stamps of CTA (0, 0), [tile][8]
    int dbg;                   // timing experiments (results invalid): 1 = no softmax arithmetic, 2 = no KV copies, 4 = no MMAs
    unsigned long long* tr;
};

struct PtLineArgs {
    DlWindowAttnArgs w;
    const int* tile_rows;      // [n_tiles][rq], -1 where a tile has fewer rows
    int n_tiles, rq, rep;
};
template <bool LINES> struct PtKernelArgs { typedef PtArgs T; };
template <> struct PtKernelArgs<true> { typedef PtLineArgs T; };

DL_DEVINL void pt_wait(uint64_t* bar, uint32_t parity, unsigned long long t0) {
    unsigned n = 0;
    while (!mbar_try_wait(bar, parity)) {
        if ((++n & 0x3FFu) == 0 && globaltimer_ns() - t0 > PT_DEADLINE_NS) __trap();
    }
}
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
#define PT_STAMP(slot, j) do { if constexpr (!LINES) { if (a.stamps && blockIdx.x == 0 && blockIdx.y == 0 && (j) < 64) a.stamps[(j) * 8 + (slot)] = clock64(); } } while (0)
#define PT_DBG(bit) (pt_dbg(a) & (bit))
DL_DEVINL int pt_dbg(const PtArgs& a) { return a.dbg; }
DL_DEVINL int pt_dbg(const PtLineArgs&) { return 0; }

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
template <bool LINES> DL_DEVINL float pt_ex2_poly(float x) {
    float xc;                                      // LINES: a NaN stays one, as in the mma.sync kernel
    if (LINES) asm("max.NaN.f32 %0, %1, %2;" : "=f"(xc) : "f"(x), "f"(-126.0f));
    else xc = fmaxf(x, -126.0f);
    const float t = xc + 12582912.0f;              // 1.5 * 2^23: round(x) lands in the low mantissa bits
    const float f = xc - (t - 12582912.0f);        // [-0.5, 0.5]
    const float p = LINES ? fmaf(fmaf(fmaf(fmaf(fmaf(1.32764725e-3f, f, 9.67554096e-3f), f, 0.0555071309f), f, 0.240221202f), f, 0.693146944f), f, 1.00000012f)
                          : fmaf(fmaf(fmaf(0.0550886838f, f, 0.242604051f), f, 0.693276242f), f, 0.99992894f);
    if (LINES) return p * __int_as_float((__float_as_int(t) << 23) + 0x3f800000);
    return __int_as_float(__float_as_int(p) + (__float_as_int(t) << 23));
}

// 32 scores (masked ones are -inf) -> exp2(s * sc - ref) as 16 packed fp16 pairs into TMEM; returns their sum.  LINES: as bf16 and, at
// taddr_lo, the bf16 remainder of each, 17 bits together
template <bool LINES> DL_DEVINL float pt_probs(const uint32_t (&v)[32], float sc, float ref, uint32_t taddr, uint32_t taddr_lo) {
    uint32_t pk[16], lo[LINES ? 16 : 1];
    float sum = 0.0f;
#pragma unroll
    for (int e = 0; e < 32; e += 2) {
        const float pa = pt_ex2(fmaf(__uint_as_float(v[e]), sc, -ref));
        const float xb = fmaf(__uint_as_float(v[e + 1]), sc, -ref);
        const float pb = (e & 2) ? pt_ex2_poly<LINES>(xb) : pt_ex2(xb);
        sum += pa + pb;
        pk[e >> 1] = pt_pack2<LINES>(pa, pb);
        if constexpr (LINES) lo[e >> 1] = pt_pack2<LINES>(pa - __uint_as_float(pk[e >> 1] << 16), pb - __uint_as_float(pk[e >> 1] & 0xffff0000u));
    }
    tmem_st_32x32b_x16(taddr, pk);
    if constexpr (LINES) tmem_st_32x32b_x16(taddr_lo, lo);
    return sum;
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

template <bool LINES>
__global__ void __launch_bounds__(PT_THREADS, 1) attention_prefill_tc_kernel(const __grid_constant__ typename PtKernelArgs<LINES>::T a,
                                                                             const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap vmap) {
    extern __shared__ __align__(1024) uint8_t smem[];
    if constexpr (!LINES) trace_begin(a.tr);
    const unsigned long long t0 = globaltimer_ns();
    uint8_t* q_s = smem;                                        // Q tile, K-major core matrices
    uint8_t* k_s = smem + PT_TILE_BYTES;                        // [3] K tiles (tokens x head dim, K-major)
    uint8_t* v_s = k_s + PT_STAGES * PT_TILE_BYTES;             // [3] V tiles (tokens x head dim, MN-major for P V)
    float* out_s = reinterpret_cast<float*>(k_s);               // [128][129] f32, reuses the KV stages after the loop
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + (1 + 2 * PT_STAGES) * PT_TILE_BYTES);
    uint64_t* k_full = bars;             // [3] transaction bytes of the step's K copies
    uint64_t* k_empty = bars + 3;        // [3] the scores that read the stage are complete
    uint64_t* v_full = bars + 6;         // [3] transaction bytes of the step's V copies
    uint64_t* v_empty = bars + 9;        // [3] P V of the step has retired
    uint64_t* q_full = bars + 12;
    uint64_t* s_full = bars + 13;        // [2] scores complete
    uint64_t* p_full = bars + 15;        // [2] probabilities written (and the score buffer read)
    uint64_t* o_full = bars + 17;        // [2] P V of tile j complete (barrier j & 1)
    uint64_t* s_empty = bars + 19;       // [2] the score buffer has been read into registers
    uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(bars + 21);
    float* mx_s = reinterpret_cast<float*>(bars + 24);          // [2 step parities][2 halves][128 rows] row maxima (and row sums at the end)

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    int kvh, n_rows, r_first, p0, last_pos, seq_end, first_page, j0, j1, max_pages, n_kv, begin = 0, head = 0;
    const int *bt, *rows_of = nullptr;
    pdl_launch_dependents();
    if constexpr (!LINES) {
        head = blockIdx.y;
        kvh = head / (a.n_heads / a.n_kv_heads);
        pdl_wait();                                              // q, this chunk's KV rows and meta come from earlier kernels
        // which (segment, 128-row tile) is this CTA?  Large tiles (late rows: long histories) are handed out first.
        int tile = blockIdx.x, end = 0;
        {
            const int n_seg = min(a.meta[0], PT_MAX_SEG);
            int i = 0;
            for (; i < n_seg; i++) {
                begin = a.meta[1 + 2 * i];
                end = a.meta[2 + 2 * i];
                const int nt = (end - begin + PT_ROWS - 1) / PT_ROWS;
                if (tile < nt) { tile = nt - 1 - tile; break; }
                tile -= nt;
            }
            if (i == n_seg) { trace_end(a.tr); return; }
        }
        n_rows = end - begin;
        r_first = tile * PT_ROWS;
        p0 = a.pos[begin];
        bt = a.block_table + (size_t)a.slot[begin] * a.max_pages;
        last_pos = p0 + r_first + min(PT_ROWS, n_rows - r_first) - 1;
        seq_end = p0 + n_rows;                                   // tokens of this sequence that exist
        first_page = j0 = 0;
        j1 = last_pos / PT_KV + 1;
        n_kv = a.n_kv_heads;
    } else {
        // (launched behind a kernel that writes the rows of other tiles and reads the same inputs: nothing to wait for here.  What
        // follows this grid must follow that one too, so this grid may not end ahead of it: a CTA with work waits when it is done, and the
        // first CTA waits even without -- one is enough, a grid ends with its last CTA, and all of the idle ones would keep an SM each
        // from those with work)
        const DlWindowAttnArgs& w = a.w;
        const bool first_cta = blockIdx.x == 0 && blockIdx.y == 0;
        kvh = blockIdx.y;
        const int t = (int)gridDim.x - 1 - (int)blockIdx.x;      // late tiles (long histories) first
        const int e = t & ~1;                                    // an even tile takes its neighbour along where that continues its sequence
        const int ne = window_tile_count(a.tile_rows, a.n_tiles, a.rq, e), no = window_tile_count(a.tile_rows, a.n_tiles, a.rq, e + 1);
        const bool both = window_tiles_join(w, a.tile_rows, a.rq, e, ne, no);
        const int run = (t & 1) ? (both ? 0 : no) : both ? ne + no : ne;
        if (run * a.rep <= 16) {                                 // taken along by its neighbour, or a decoding tile, which belongs to the other kernel
            if (first_cta) pdl_wait();
            return;
        }
        rows_of = a.tile_rows + (size_t)t * a.rq;
        const int m0 = rows_of[0], p_first = w.pos[m0];
        n_rows = run * a.rep;
        r_first = 0;
        p0 = p_first;
        last_pos = p_first + run - 1;
        seq_end = last_pos + 1;                                  // what lies behind was not written yet, or is of no use here
        bt = w.block_table + (size_t)w.slot[m0] * w.max_pages;
        int lo = w.window > 0 ? max(0, p_first - w.window + 1) : 0;
        if (w.chunk > 0) lo = max(lo, p_first / w.chunk * w.chunk);
        first_page = lo / 32;                                    // pages ahead of it are not touched
        j0 = lo / PT_KV;
        j1 = last_pos / PT_KV + 1;
        n_kv = w.kv_heads;
    }
    const int n_tiles = j1 - j0;                                 // steps of 128 tokens, the first one at token j0 * 128

    if (tid == 0) {
        for (int s = 0; s < PT_STAGES; s++) {
            mbar_init(&k_full[s], 1);
            mbar_init(&k_empty[s], 1);
            mbar_init(&v_full[s], 1);
            mbar_init(&v_empty[s], 1);
        }
        for (int s = 0; s < 2; s++) {
            mbar_init(&s_full[s], 1);
            mbar_init(&s_empty[s], 256);
            mbar_init(&p_full[s], 256);
            mbar_init(&o_full[s], 1);
        }
        mbar_init(q_full, 256);
        mbar_fence_init();
    }
    if (warp == 0) tmem_alloc(tmem_holder, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_holder;
    const uint32_t T_S = tmem_base, T_P = tmem_base + 256, T_O = tmem_base + 384;

    // 128-byte-swizzled operands: rows of 128 B (64 halfs), 8-row groups 1024 B apart; the head dimension is split in
    // two such half tiles 16 KB apart.  K-major (Q, K): LBO unused (1), SBO 1024.  MN-major (V as B of P V): LBO =
    // distance between the two 64-wide halves of N (16 KB), SBO = distance between 8-token groups (1024 B).
    const uint32_t desc_hi = (1024u >> 4) | (1u << 14) | (2u << 29);
    if (warp == 0) {
        // ------------------------------------ S = Q K^T issuer ------------------------------------
        const uint32_t idesc_s = pt_idesc(PT_ROWS, PT_KV, 0, LINES);
        auto lo_k = [](const void* p) { return ((smem_u32(p) & 0x3FFFFu) >> 4) | (1u << 16); };
        pt_wait(q_full, 0, t0);
        for (int j = 0; j < n_tiles; j++) {
            pt_wait(&k_full[j % PT_STAGES], (j / PT_STAGES) & 1, t0);
            if (lane == 0) PT_STAMP(0, j);
            // softmax(j-2) has this score buffer in registers; LINES: P V(j-2) has read the remainders that lay in it
            if (j >= 2) pt_wait(LINES ? &o_full[j & 1] : &s_empty[j & 1], ((j - 2) >> 1) & 1, t0);
            tc_fence_after();
            if (elect_one()) {
                const uint32_t a_lo = lo_k(q_s), b_lo = lo_k(k_s + (j % PT_STAGES) * PT_TILE_BYTES);
#pragma unroll
                for (int k = 0; k < 8; k++) {      // K = 16 per MMA: 32 B inside the swizzled row, the second half tile after four
                    const uint32_t off = (uint32_t)((k >> 2) * (16384 >> 4) + (k & 3) * 2);
                    uint64_t da, db;
                    asm("mov.b64 %0, {%1, %2};" : "=l"(da) : "r"(a_lo + off), "r"(desc_hi));
                    asm("mov.b64 %0, {%1, %2};" : "=l"(db) : "r"(b_lo + off), "r"(desc_hi));
                    if (!PT_DBG(4)) umma_f16_ss(T_S + (j & 1) * 128, da, db, idesc_s, k > 0 ? 1u : 0u);
                }
                umma_commit(&s_full[j & 1]);
                umma_commit(&k_empty[j % PT_STAGES]);
            }
            __syncwarp();
            if (lane == 0) PT_STAMP(1, j);
        }
    } else if (warp == 6) {
        // ------------------------------------ O += P V issuer ------------------------------------
        const uint32_t idesc_pv = pt_idesc(PT_ROWS, PT_HS, 1, LINES);
        for (int i = 0; i < n_tiles; i++) {
            uint8_t* vz = v_s + (i % PT_STAGES) * PT_TILE_BYTES;
            if (LINES && i == 0 && first_page * 32 > j0 * PT_KV) {      // tokens of pages that this tile does not touch
                pt_wait(&v_full[0], 0, t0);
                for (int idx = lane; idx < (first_page * 32 - j0 * PT_KV) * 16; idx += 32)
                    *reinterpret_cast<uint4*>(vz + ((idx >> 3) & 1) * 16384 + (idx >> 4) * 128 + (idx & 7) * 16) = make_uint4(0, 0, 0, 0);
                fence_proxy_async_smem();
                __syncwarp();
            }
            if ((j0 + i + 1) * PT_KV > seq_end) {
                // the step that contains the end of the sequence: rows past it were never written (or not copied at all);
                // their scores are masked, but a zero probability times a non-finite V would poison the product -> zero them
                pt_wait(&v_full[i % PT_STAGES], (i / PT_STAGES) & 1, t0);
                const int r0 = max(0, seq_end - (j0 + i) * PT_KV);
                for (int idx = r0 * 16 + lane; idx < PT_KV * 16; idx += 32) {      // 16 pieces of 16 B per token row (two halves)
                    const int r = idx >> 4, c = idx & 15;
                    *reinterpret_cast<uint4*>(vz + (c >> 3) * 16384 + r * 128 + (c & 7) * 16) = make_uint4(0, 0, 0, 0);
                }
                fence_proxy_async_smem();
                __syncwarp();
            }
            pt_wait(&v_full[i % PT_STAGES], (i / PT_STAGES) & 1, t0);
            pt_wait(&p_full[i & 1], (i >> 1) & 1, t0);
            if (lane == 0) PT_STAMP(2, i);
            tc_fence_after();
            if (elect_one()) {
                const uint32_t b_lo = ((smem_u32(vz) & 0x3FFFFu) >> 4) | ((16384u >> 4) << 16);
#pragma unroll
                for (int k = 0; k < 8; k++) {      // 16 tokens per MMA: 8 TMEM columns of P, two 8-token groups (2048 B) of V
                    uint64_t db;
                    asm("mov.b64 %0, {%1, %2};" : "=l"(db) : "r"(b_lo + k * 128), "r"(desc_hi));
                    if (!PT_DBG(4)) umma_f16_ts(T_O, T_P + (i & 1) * 64 + k * 8, db, idesc_pv, (i > 0 || k > 0) ? 1u : 0u);
                    if constexpr (LINES) umma_f16_ts(T_O, T_S + (i & 1) * 128 + k * 8, db, idesc_pv, 1u);
                }
                umma_commit(&o_full[i & 1]);
                umma_commit(&v_empty[i % PT_STAGES]);
            }
            __syncwarp();
        }
    } else if (warp <= 4 || warp >= 8) {
        // ---------------- softmax: two threads per query row (= TMEM lane), 64 score columns each ----------------
        // warps 1-4 take columns [0, 64) of their lane quarter, warps 8-11 columns [64, 128): the MUFU work of a step
        // (128 x 128 exp2) is fixed, but with two warps per scheduler the loads, maxima, packs and stores overlap it
        const int quarter = warp & 3, row = quarter * 32 + lane, hf = warp >= 8 ? 1 : 0;
        const int r_abs = r_first + row;
        const int r_live = min(r_abs, n_rows - 1);
        int m_row = 0, h_row = 0;                                // LINES: this row's batch row and head
        {
            const float* qg;
            if constexpr (LINES) {
                m_row = rows_of[r_live / a.rep];
                h_row = kvh * a.rep + r_live % a.rep;
                qg = a.w.q + (size_t)m_row * a.w.ldq + h_row * PT_HS + hf * 64;
            } else {
                qg = a.q + (size_t)(begin + r_live) * a.n_heads * PT_HS + head * PT_HS + hf * 64;
            }
            uint8_t* qd = q_s + hf * 16384 + row * 128;
#pragma unroll 4
            for (int c = 0; c < 8; c++) {       // 16-byte piece c of this half of the row -> swizzled slot c ^ (row & 7)
                const float4 x = reinterpret_cast<const float4*>(qg)[2 * c], y = reinterpret_cast<const float4*>(qg)[2 * c + 1];
                uint4 u;
                u.x = pt_pack2<LINES>(x.x, x.y); u.y = pt_pack2<LINES>(x.z, x.w);
                u.z = pt_pack2<LINES>(y.x, y.y); u.w = pt_pack2<LINES>(y.z, y.w);
                *reinterpret_cast<uint4*>(qd + ((c ^ (row & 7)) << 4)) = u;
            }
            fence_proxy_async_smem();
            mbar_arrive(q_full);
        }
        int pos_r, lb = 0;                                       // last and first visible position of this row
        float sc, c1 = 0.f, cap_k = 0.f, slope = 0.f;
        bool shaped = false;                                     // scores leave the accumulator through a cap, a bias or a factor that is not positive
        if constexpr (LINES) {
            const DlWindowAttnArgs& w = a.w;
            pos_r = p0 + r_live / a.rep;
            if (w.window > 0) lb = max(0, pos_r - w.window + 1);
            if (w.chunk > 0) lb = max(lb, pos_r / w.chunk * w.chunk);
            shaped = w.softcap > 0.f || w.slope != nullptr || !(w.scale > 0.f);      // (a factor that keeps no order meets the scores ahead of mask and maximum)
            sc = 1.4426950408889634f * w.scale;
            c1 = w.softcap > 0.f ? sc * 2.f / w.softcap : sc;
            cap_k = w.softcap * 1.4426950408889634f;
            if (w.slope != nullptr) slope = w.slope[h_row] * 1.4426950408889634f;
            if (shaped) sc = 1.f;
        } else {
            pos_r = p0 + r_abs;
            sc = 1.4426950408889634f * rsqrtf((float)PT_HS);     // scores in the log2 domain
        }
        const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
        float m_used = -INFINITY, l = 0.0f;
        uint32_t v0[32], v1[32];
        for (int j = 0; j < n_tiles; j++) {
            pt_wait(&s_full[j & 1], (j >> 1) & 1, t0);
            if (tid == 32) PT_STAMP(3, j);
            tc_fence_after();
            const uint32_t t_s = T_S + lane_base + (j & 1) * 128 + hf * 64;
            const int tok0 = (j0 + j) * PT_KV + hf * 64;
            if PT_DBG(1) { tc_fence_before(); mbar_arrive(&s_empty[j & 1]); mbar_arrive(&p_full[j & 1]); continue; }
            tmem_ld_32x32b_x32(t_s, v0);
            tmem_ld_32x32b_x32(t_s + 32, v1);
            tmem_ld_wait();
            tc_fence_before();
            mbar_arrive(&s_empty[j & 1]);                    // the scores of step j+2 may overwrite the buffer now
            const int lim = pos_r - tok0;                    // columns e <= lim of this half are visible to this row
            const int low = LINES ? lb - tok0 : 0;           // and e >= low
            if constexpr (LINES) {
                if (shaped) {
#pragma unroll
                    for (int e = 0; e < 64; e++) {
                        float x = __uint_as_float(e < 32 ? v0[e & 31] : v1[e & 31]) * c1;
                        if (cap_k > 0.f) {                   // cap tanh(s / cap) in base 2, as the mma.sync kernel forms it
                            float r;
                            asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(pt_ex2(x) + 1.f));
                            x = fmaf(-2.f * cap_k, r, cap_k);
                        }
                        x = fmaf(-slope, (float)(lim - e), x);
                        if (e < 32) v0[e & 31] = __float_as_uint(x); else v1[e & 31] = __float_as_uint(x);
                    }
                }
            }
            float ma = -INFINITY, mb = -INFINITY;
            if (lim >= 63 && (!LINES || low <= 0)) {
#pragma unroll
                for (int e = 0; e < 32; e += 2) {
                    ma = fmaxf(ma, fmaxf(__uint_as_float(v0[e]), __uint_as_float(v1[e])));
                    mb = fmaxf(mb, fmaxf(__uint_as_float(v0[e + 1]), __uint_as_float(v1[e + 1])));
                }
            } else {
#pragma unroll
                for (int e = 0; e < 32; e++) {
                    if (e > lim || (LINES && e < low)) v0[e] = 0xff800000u;        // -inf
                    if (e + 32 > lim || (LINES && e + 32 < low)) v1[e] = 0xff800000u;
                    ma = fmaxf(ma, fmaxf(__uint_as_float(v0[e]), __uint_as_float(v1[e])));
                }
            }
            // row maximum over both halves: exchange through shared memory (slot of step parity: the next write to it
            // comes two steps later, after everybody has passed the barrier of the step in between)
            float mx = fmaxf(ma, mb);
            mx_s[((j & 1) * 2 + hf) * PT_ROWS + row] = mx;
            asm volatile("bar.sync 2, 256;" ::: "memory");
            mx = fmaxf(mx, mx_s[((j & 1) * 2 + (hf ^ 1)) * PT_ROWS + row]);
            if constexpr (LINES) tc_fence_after();           // both halves have read their scores: the remainders take their place
            if (tid == 32) PT_STAMP(4, j);
            mx *= sc;
            const bool need = mx > m_used + 8.0f;            // the reference may lag the maximum by 2^8
            if (__any_sync(0xffffffffu, need)) {
                const float m_new = need ? mx : m_used;
                const float alpha = need ? pt_ex2(m_used - m_new) : 1.0f;
                if (j > 0) {      // the accumulated output moves to the new reference (rare after the first tiles)
                    pt_wait(&o_full[(j - 1) & 1], ((j - 1) >> 1) & 1, t0);
                    tc_fence_after();
                    uint32_t w[32];
#pragma unroll 1
                    for (int ch = 0; ch < 2; ch++) {
                        tmem_ld_32x32b_x32(T_O + lane_base + hf * 64 + ch * 32, w);
                        tmem_ld_wait();
#pragma unroll
                        for (int e = 0; e < 32; e++) w[e] = __float_as_uint(__uint_as_float(w[e]) * alpha);
                        tmem_st_32x32b_x32(T_O + lane_base + hf * 64 + ch * 32, w);
                    }
                    tmem_st_wait();
                }
                l *= alpha;
                m_used = m_new;
            }
            const float ref = (m_used == -INFINITY) ? 0.0f : m_used;
            const uint32_t t_p = T_P + lane_base + (j & 1) * 64 + hf * 32;
            if (j >= 2) {      // P V(j-2) has consumed this probability buffer (long done; the wait keeps it a guarantee)
                pt_wait(&o_full[j & 1], ((j - 2) >> 1) & 1, t0);
                tc_fence_after();
            }
            const uint32_t t_lo = T_S + lane_base + (j & 1) * 128 + hf * 32;
            l += pt_probs<LINES>(v0, sc, ref, t_p, t_lo);
            l += pt_probs<LINES>(v1, sc, ref, t_p + 16, t_lo + 16);
            tmem_st_wait();
            tc_fence_before();
            mbar_arrive(&p_full[j & 1]);
            if (tid == 32) PT_STAMP(5, j);
        }
        // ---- finish: O / l -> shared memory -> Q80 cast into the slabs of the wo matmul ----
        pt_wait(&o_full[(n_tiles - 1) & 1], ((n_tiles - 1) >> 1) & 1, t0);
        tc_fence_after();
        // the two halves of the row sum, through the exchange slots the LAST step did not use (their previous readers
        // have all passed that step's barrier)
        const int fs = (n_tiles & 1) * 2;
        mx_s[(fs + hf) * PT_ROWS + row] = l;
        asm volatile("bar.sync 2, 256;" ::: "memory");
        l += mx_s[(fs + (hf ^ 1)) * PT_ROWS + row];
        float inv;
        if constexpr (LINES) {
            if (a.w.sink) l += pt_ex2(a.w.sink[h_row] * 1.4426950408889634f - m_used);
            inv = (a.w.gate ? 1.f / (1.f + expf(-a.w.gate[(size_t)m_row * a.w.ld_gate + h_row])) : 1.f) / l;
        } else {
            inv = l > 0.0f ? 1.0f / l : 0.0f;
        }
        bool rows_out = true;                                    // f32 rows wanted: through shared memory, lanes along a row
        if constexpr (!LINES) rows_out = a.y_out != nullptr;
#pragma unroll 1
        for (int ch = 0; ch < 2; ch++) {
            tmem_ld_32x32b_x32(T_O + lane_base + hf * 64 + ch * 32, v0);
            tmem_ld_wait();
            float v[32];
#pragma unroll
            for (int e = 0; e < 32; e++) v[e] = __uint_as_float(v0[e]) * inv;
            if constexpr (!LINES) {
                if (r_abs < n_rows && (a.xq_out != nullptr || a.xh_out != nullptr))
                    pt_q80_block(v, begin + r_abs, (head * PT_HS) / 32 + hf * 2 + ch, a.out_mcap, a.xq_out, a.xh_out);
            }
            if (rows_out) {
#pragma unroll
                for (int e = 0; e < 32; e++) out_s[row * PT_OUT_LD + hf * 64 + ch * 32 + e] = v[e];
            }
        }
        if (rows_out) {
            __syncwarp();                                        // a warp only re-reads the 32 rows x 64 columns it wrote
#pragma unroll 4
            for (int rr = 0; rr < 32; rr++) {
                const int rc = r_first + quarter * 32 + rr;
                if (rc >= n_rows) break;
                float* dst;
                if constexpr (LINES) dst = a.w.out + (size_t)__shfl_sync(0xffffffffu, m_row, rr) * a.w.ldo + __shfl_sync(0xffffffffu, h_row, rr) * PT_HS;
                else dst = a.y_out + (size_t)(begin + rc) * a.n_heads * PT_HS + head * PT_HS;
                const float* src = out_s + (quarter * 32 + rr) * PT_OUT_LD + hf * 64 + lane;
                dst[hf * 64 + lane] = src[0];
                dst[hf * 64 + 32 + lane] = src[32];
            }
        }
    } else if (warp == 5 || warp == 7) {
        // ------------------------------------ K producer (warp 5) / V producer (warp 7), one lane each ------------------------------------
        if (lane == 0) {
            const bool is_k = warp == 5;
            const uint64_t map = is_k ? reinterpret_cast<uint64_t>(&kmap) : reinterpret_cast<uint64_t>(&vmap);
            uint64_t* full = is_k ? k_full : v_full;
            uint64_t* empty = is_k ? k_empty : v_empty;
            uint8_t* ring = is_k ? k_s : v_s;
            const int total_pages = (seq_end + 31) / 32;
            auto page_of = [&](int p) { return p >= first_page && p < total_pages ? bt[p] : 0; };
            // the page ids of a step are fetched one step ahead, so the table reads (dependent global loads) overlap the
            // wait for a free stage instead of delaying the copies
            int pg[4], pg_next[4];
#pragma unroll
            for (int p4 = 0; p4 < 4; p4++) pg_next[p4] = page_of(4 * j0 + p4);
            for (int j = 0; j < n_tiles; j++) {
                const int st = j % PT_STAGES;
#pragma unroll
                for (int p4 = 0; p4 < 4; p4++) {
                    pg[p4] = pg_next[p4];
                    pg_next[p4] = page_of(4 * (j0 + j + 1) + p4);
                }
                if (j >= PT_STAGES) pt_wait(&empty[st], ((j / PT_STAGES) & 1) ^ 1, t0);
                if (is_k) PT_STAMP(6, j);
                const int n_pg = PT_DBG(2) ? 0 : min(4, (seq_end - (j0 + j) * PT_KV + 31) / 32);      // pages of this step that exist
                const int p_lo = LINES ? max(0, first_page - 4 * (j0 + j)) : 0;                 // ... and are looked at (at most the first step starts later)
                mbar_arrive_expect_tx(&full[st], (uint32_t)max(0, n_pg - p_lo) * 2u * 4096u);
                const uint32_t dst = smem_u32(ring + st * PT_TILE_BYTES), bar = smem_u32(&full[st]);
#pragma unroll
                for (int p4 = 0; p4 < 4; p4++) {
                    if (p4 >= n_pg) break;
                    if (LINES && p4 < p_lo) continue;
                    const int y = (pg[p4] * n_kv + kvh) * 32;      // first row of the page in the [rows][128] view
#pragma unroll
                    for (int h = 0; h < 2; h++)
                        asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
                                         dst + h * 16384 + p4 * 4096),
                                     "l"(map), "r"((LINES && !is_k ? PT_HS : 0) + h * 64), "r"(y), "r"(bar)
                                     : "memory");
                }
                if (is_k) PT_STAMP(7, j);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
    if constexpr (LINES) pdl_wait();                             // what follows this grid follows the one ahead of it too
    else trace_end(a.tr);
}

extern void dl_set_error(const char* fmt, ...);
static int g_pt_dbg = 0;
static long long* g_pt_stamps = nullptr;
extern "C" void dl_debug_set_pt_mode(int m) { g_pt_dbg = m; }
extern "C" void dl_debug_set_pt_trace(long long* p) { g_pt_stamps = p; }

typedef CUresult (*PtEncodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// [rows][width] fp16 or bf16 view of a KV cache on THIS GPU (rows = pages x kv heads x 32), box = 64 columns x 32 rows (one page of
// one head, half of the head dimension), 128-byte swizzle: the image tcgen05.mma reads as a swizzled K- or MN-major tile
static int pt_make_map(CUtensorMap* m, const void* base, long long rows, int width, bool bf16) {
    static PtEncodeTiled enc = nullptr;
    if (enc == nullptr) {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult qr;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qr) != cudaSuccess || fn == nullptr) {
            dl_set_error("attention_prefill_tc: cuTensorMapEncodeTiled not available");
            return -1;
        }
        enc = (PtEncodeTiled)fn;
    }
    const cuuint64_t dims[2] = {(cuuint64_t)width, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)width * 2};
    const cuuint32_t box[2] = {64, 32}, es[2] = {1, 1};
    const CUresult r = enc(m, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(base), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) { dl_set_error("attention_prefill_tc: cuTensorMapEncodeTiled failed (%d)", (int)r); return -1; }
    return 0;
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
    a.dbg = g_pt_dbg;
    a.stamps = g_pt_stamps;
    a.tr = dl_trace_next(TR_ATT);
    alignas(64) CUtensorMap kmap, vmap;
    const long long rows = (long long)n_cache_pages * n_kv_heads * 32;
    if (pt_make_map(&kmap, k_cache, rows, PT_HS, false) != 0 || pt_make_map(&vmap, v_cache, rows, PT_HS, false) != 0) return -1;
    const size_t smem = (1 + 2 * PT_STAGES) * PT_TILE_BYTES + 24 * 8 + 4 * PT_ROWS * 4;
    static bool set = false;
    if (!set) {
        cudaError_t e = cudaFuncSetAttribute(attention_prefill_tc_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) { dl_set_error("attention_prefill_tc smem attr: %s", cudaGetErrorString(e)); return -(int)e; }
        set = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((M + PT_ROWS - 1) / PT_ROWS + PT_MAX_SEG), (unsigned)n_heads);      // upper bound of the tiles of all segments
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

// The tiles of more than 16 stacked rows; launched behind the kernel that takes the others (programmatic launch: they run side by side).
int dl_window_prefill_tc(const DlWindowAttnArgs& w, const int* tile_rows, int n_tiles, int rq, cudaStream_t stream) {
    PtLineArgs a;
    a.w = w; a.tile_rows = tile_rows; a.n_tiles = n_tiles; a.rq = rq; a.rep = w.heads / w.kv_heads;
    alignas(64) CUtensorMap map;
    // the cache's page count is not known here; every copy reads a page that the block table names
    if (pt_make_map(&map, w.cache, 1ll << 31, 2 * PT_HS, true) != 0) return -1;
    const size_t smem = (1 + 2 * PT_STAGES) * PT_TILE_BYTES + 24 * 8 + 4 * PT_ROWS * 4;
    static bool set = false;
    if (!set) {
        cudaError_t e = cudaFuncSetAttribute(attention_prefill_tc_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) { dl_set_error("window_prefill_tc smem attr: %s", cudaGetErrorString(e)); return -(int)e; }
        set = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)n_tiles, (unsigned)w.kv_heads);
    cfg.blockDim = dim3(PT_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, attention_prefill_tc_kernel<true>, a, map, map);
    if (e != cudaSuccess) { dl_set_error("window_prefill_tc launch: %s", cudaGetErrorString(e)); return -(int)e; }
    return 0;
}
