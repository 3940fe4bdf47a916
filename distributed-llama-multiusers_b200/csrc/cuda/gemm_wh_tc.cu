// Prompt-sized Q40 x Q80 matmul (M >= a few hundred activation rows) on tcgen05, two phases:
//
//   1. q40t_to_wh_kernel expands a Q40T weight image ONCE into "WH": fp16 tiles of 128 rows x 128 K in the UMMA
//      K-major no-swizzle core-matrix image (the same 8 rows x 16 B core matrices and the same K order inside a
//      32-block as the XH activation slabs).  fp16((nibble - 8) * d), one rounding: bit-identical to what the
//      on-the-fly dequantisers of gemm_q40_tc.cu feed the tensor core.  The engine keeps the WH copy resident when
//      it fits (8B: 15 GB of the 180 GB) or rebuilds it per matrix into a scratch buffer.
//   2. gemm_wh_tc_kernel is then a plain fp16 SS-mode GEMM: both operands arrive by bulk or tensor copies of
//      contiguous, pre-tiled pieces of up to 16 KB; nothing is unpacked inside the loop, so the unpack -- the limiter of the
//      fused kernel (ALU pipe 50 %, tensor pipe 14 % at 32 rows of w13), which every M tile
//      repeated -- is paid once per weight instead of once per 256 activation rows.
//
// gemm_wh_tc_kernel<2> pairs two CTAs (cluster of 2 = one TPC) on a 256 weight rows x up to 256 activation rows tile with
// `tcgen05.mma.cta_group::2`: each CTA stages its own 128 weight rows and HALF of the activation rows (64 KB per
// 128-wide k step and CTA instead of 96 KB).  gemm_wh_tc_kernel<1> is the single-CTA variant (odd row-tile counts).
// What bounds it: the MMAs under the power limit (28672 x 4096 at 2048 rows 324 us, 312 without its epilogues; on a faster card 301 without them, 166 without MMAs,
// whose copies then run at 85 B/clk and SM, and cuBLAS 348).
//
// Grouped mode: the same kernel runs one product per group of rows against that group's own weights (the experts of a
// routed feed-forward: rows sorted by expert, segment bounds in device memory), so all experts are ONE launch and the
// host never learns how many rows an expert got.
//
// Persistent CTAs walk the tile list (activation tiles fastest, so the CTAs that run at the same time share one
// weight panel in L2); each CTA owns 128 TMEM lanes x 2 accumulators of 256 columns, so the epilogue of tile i
// (TMEM -> registers -> smem chunk -> the shared fused epilogues of epilogue.cuh) overlaps the MMAs of tile i+1.
//
// Warp roles (576 threads): warp 0 producer (a converged warp, 4-6 of its lanes a copy each per stage), warp 1 MMA issuer (in the first CTA of a pair) + TMEM
// owner, warps 2-17 epilogue.
// Reference semantics: matmul_Q80_Q40_F32 (src/nn/nn-cpu-ops.cpp:352-377), llamafile sgemm (src/nn/llamafile/sgemm.cpp:593-783).
#include "epilogue.cuh"
#include "smem_limit.cuh"
#include "tensor_map.cuh"

#define WH_TILE_BYTES 32768
#define WT_NT 256                      // most activation rows per tile (wh_tile_rows: how many)
#define WT_THREADS 576
#define WT_EPI_CHUNK 32                // activation rows per epilogue pass, one row per warp quarter
#define WT_VEC_CHUNK 64                // the same by whole warps (epilogue_vec): four rows per warp

struct WhArgs {
    const uint8_t* wh;                 // [row_tiles][KT][32 KB]
    const uint8_t* xh;                 // [KT][ncap/8][2048]
    int d_real, row_tiles, KT, ncap, M, m_tiles, n_tiles;
    int nt;                            // activation rows per tile: a multiple of 32 (what an MMA of two CTAs takes), at most WT_NT
    int n_epi_ctas;
    int piece;                         // bytes per bulk copy (4096 / 8192 / 16384)
    int dbg;                           // timing experiments (results invalid): 1 = no epilogue work, 2 = no MMAs, 4 = no activation copies
    int bf16;                          // both operand images hold bf16 instead of fp16 (dense-weight models)
    int vec;                           // epilogue_vec takes the epilogue
    // grouped mode (routed experts): n_groups weight images wh_group_bytes apart; group g multiplies the activation rows
    // [grp[2g], grp[2g] + grp[2g+1]) (device memory; first rows are multiples of 8) and writes those output rows.  The
    // tile list covers m_tiles activation tiles per group; tiles beyond a group's rows are skipped by every role alike.
    const int* grp;
    int n_groups;
    long long wh_group_bytes;
    unsigned long long* tr;
    DlEpilogue epi;
};

template <int CG> DL_DEVINL void wt_tmem_alloc(uint32_t* holder) {
    if (CG == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(holder)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    } else {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(holder)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
}
template <int CG> DL_DEVINL void wt_tmem_dealloc(uint32_t taddr) {
    if (CG == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(512) : "memory");
    else asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(512) : "memory");
}
template <int CG> DL_DEVINL void wt_mma(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t acc) {
    if (CG == 1) {
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                     "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(acc) : "memory");
    } else {
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                     "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(acc) : "memory");
    }
}
// all MMAs issued so far by this thread have completed -> arrive on the barrier (in both CTAs of a pair)
template <int CG> DL_DEVINL void wt_commit(uint64_t* bar) {
    if (CG == 1) {
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
    } else {
        asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
                     "h"((uint16_t)3)
                     : "memory");
    }
}
DL_DEVINL void wt_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// box (256 doublewords, a row group; rows; one slab) at {0, c1, c2} into this CTA, counted by a barrier of either CTA of the pair
DL_DEVINL void wt_copy_pair(uint32_t dst, const CUtensorMap* map, int c1, int c2, uint32_t cluster_bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst),
                 "l"(map), "r"(0), "r"(c1), "r"(c2), "r"(cluster_bar)
                 : "memory");
}

// Bounded waits: a protocol bug must end in a trap (an error the host sees), never in a hung GPU.
#define WT_DEADLINE_NS 4000000000ull
DL_DEVINL void wt_wait(uint64_t* bar, uint32_t parity, unsigned long long t0) {
    unsigned n = 0;
    while (!mbar_try_wait(bar, parity)) {
        if ((++n & 0x3FFu) == 0 && globaltimer_ns() - t0 > WT_DEADLINE_NS) __trap();
    }
}
DL_DEVINL void wt_wait_cluster(uint64_t* bar, uint32_t parity, unsigned long long t0) {
    unsigned n = 0;
    uint32_t ok;
    while (true) {
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(smem_u32(bar)), "r"(parity)
            : "memory");
        if (ok) break;
        if ((++n & 0x3FFu) == 0 && globaltimer_ns() - t0 > WT_DEADLINE_NS) __trap();
    }
}

// tile t -> group, weight row pair, activation tile; false: the tile lies beyond its group's rows
struct WtTile { int g, rp, mt, row0, rows; };
DL_DEVINL bool wt_tile(const WhArgs& a, int t, WtTile& w) {
    const int per_group = a.n_tiles / a.n_groups;
    w.g = t / per_group;
    const int tt = t - w.g * per_group;
    w.rp = tt / a.m_tiles;
    w.mt = tt - w.rp * a.m_tiles;
    if (a.grp) {
        w.row0 = a.grp[2 * w.g];
        w.rows = a.grp[2 * w.g + 1];
    } else {
        w.row0 = 0;
        w.rows = a.M;
    }
    return w.mt * a.nt < w.rows;
}

template <int CG>
__global__ void __launch_bounds__(WT_THREADS, 1) gemm_wh_tc_kernel(const __grid_constant__ WhArgs a, const __grid_constant__ CUtensorMap wmap,
                                                                   const __grid_constant__ CUtensorMap xmap) {
    extern __shared__ __align__(1024) uint8_t smem[];
    constexpr int NS = (CG == 1) ? 2 : 3;                 // stages of one 128-wide k step
    constexpr int STAGE = WH_TILE_BYTES + WT_NT / CG * 256;   // 96 KB / 64 KB
    const int B_ROWS = a.nt / CG;                         // activation rows staged by this CTA
    trace_begin(a.tr);
    const unsigned long long t0 = globaltimer_ns();
    float* out_s = reinterpret_cast<float*>(smem + NS * STAGE);          // [32][128], or [WT_VEC_CHUNK][EPI_TILE_LD]
    uint64_t* bars = reinterpret_cast<uint64_t*>(out_s + WT_VEC_CHUNK * EPI_TILE_LD);
    uint64_t* full = bars;               // [NS]  the copies of a stage have landed (a pair's, of both CTAs: in the first one alone)
    uint64_t* empty = bars + 8;          // [NS]  the MMAs reading the stage have retired (both CTAs)
    uint64_t* acc_full = bars + 12;      // [2]   accumulator complete
    uint64_t* acc_empty = bars + 14;     // [2]   accumulator drained by the epilogue(s)
    uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(bars + 16);
    int* sflag = reinterpret_cast<int*>(tmem_holder + 1);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    uint32_t crank = 0;
    if (CG == 2) asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(crank));
    const int cid = blockIdx.x / CG, ncl = gridDim.x / CG;
    const int KT = a.KT;

    if (tid == 0) {
        for (int s = 0; s < NS; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int u = 0; u < 2; u++) {
            mbar_init(&acc_full[u], 1);
            mbar_init(&acc_empty[u], CG);
        }
        mbar_fence_init();
    }
    if (warp == 1) wt_tmem_alloc<CG>(tmem_holder);
    tc_fence_before();
    __syncthreads();
    if (CG == 2) wt_cluster_sync();      // the partner's barriers exist before anything arrives on them
    tc_fence_after();
    const uint32_t tmem_base = *tmem_holder;
    pdl_launch_dependents();

    if (warp == 0) {
        // ------------------------------------ producer ------------------------------------
        // the whole warp walks the stages together (28672 x 4096 at 2048 rows 359 us, 367 with lanes that wait and issue one by one)
        if (CG == 2) {
            // A stage is two tensor copies of 16 KB of weights and two of half of this CTA's activation rows each, both CTAs' counted by the FIRST one's
            // barrier, so that its MMAs wait for what they read in either CTA by one barrier.  The alternative, bulk copies counted in their own CTA and an
            // arrive by the second one on a barrier of the first, costs a memory barrier of ~1.4 us a stage at cluster scope (28672 x 4096 at 2048 rows 353
            // us, 4096 x 14336 205), and with less the memory model orders nothing between the CTAs.  So: 324 and 182, on a card where the same
            // without epilogues takes 312 (301 above).
            const int bg = a.nt >> 5, i = lane >> 1, half = lane & 1;      // row groups of an activation copy; lane: i = 0 weights, 1 activations
            const CUtensorMap* map = i == 0 ? &wmap : &xmap;
            const uint32_t leader_full = mapa_shared(smem_u32(full), 0);
            const uint32_t dst = i == 0 ? half * 16384 : WH_TILE_BYTES + half * bg * XH_ROWGROUP_BYTES;
            pdl_wait();
            uint32_t it = 0;
            for (int t = cid; t < a.n_tiles; t += ncl) {
                WtTile w;
                if (!wt_tile(a, t, w)) continue;
                const int row0 = w.row0 + w.mt * a.nt;
                auto live = [&](int c, int h) { return !(a.dbg & 4) && row0 + c * B_ROWS + h * bg * 8 < w.row0 + w.rows; };      // the copy has rows of the product
                const uint32_t total = 2 * WH_TILE_BYTES + (live(0, 0) + live(0, 1) + live(1, 0) + live(1, 1)) * bg * XH_ROWGROUP_BYTES;
                const bool on = i == 0 || (i == 1 && live(crank, half));
                const int c1 = i == 0 ? half * 8 : ((row0 + (int)crank * B_ROWS) >> 3) + half * bg;
                const int c2 = i == 0 ? w.g * (int)(a.wh_group_bytes / WH_TILE_BYTES) + (w.rp * CG + (int)crank) * KT : 0;
                for (int kt = 0; kt < KT; kt++, it++) {
                    const uint32_t s = it % NS;
                    if (it >= NS) wt_wait(&empty[s], ((it / NS) & 1) ^ 1, t0);
                    __syncwarp();
                    if (crank == 0 && lane == 0) mbar_arrive_expect_tx(&full[s], total);
                    if (on) wt_copy_pair(smem_u32(smem + s * STAGE) + dst, map, c1, c2 + kt, leader_full + s * 8);
                    __syncwarp();
                }
            }
        } else {
            // the stage is fetched as `piece`-byte bulk copies, one per lane: first the weight tile, then row groups of the
            // activation slab (many requests in flight: one bulk copy streams at only ~16 B/clk)
            const int piece = a.piece, npiece = STAGE / piece, na = WH_TILE_BYTES / piece, prow = piece / 256;
            pdl_wait();
            const size_t x_kt_stride = (size_t)(a.ncap >> 3) * XH_ROWGROUP_BYTES;
            uint32_t it = 0;
            for (int t = cid; t < a.n_tiles; t += ncl) {
                WtTile w;
                if (!wt_tile(a, t, w)) continue;
                const int rp = w.rp, mt = w.mt;
                const int rt = rp * CG + (int)crank;
                const int mrow0 = w.row0 + mt * a.nt + (int)crank * B_ROWS;
                const int row_cap = w.row0 + ((w.rows + 7) & ~7);      // slabs hold 8 rows; the image may be a part of a larger one and end there
                const int b_rows = max(0, min(B_ROWS, row_cap - mrow0));
                const uint8_t* src = nullptr;
                size_t stride = 0;
                uint32_t bytes = 0;
                if (lane < na) {
                    src = a.wh + (size_t)w.g * (size_t)a.wh_group_bytes + (size_t)rt * KT * WH_TILE_BYTES + lane * piece;
                    stride = WH_TILE_BYTES;
                    bytes = piece;
                } else if (lane < npiece) {
                    const int r0 = (lane - na) * prow;
                    src = a.xh + (size_t)((mrow0 + r0) >> 3) * XH_ROWGROUP_BYTES;
                    stride = x_kt_stride;
                    bytes = (a.dbg & 4) ? 0u : (uint32_t)max(0, min(prow, b_rows - r0)) * 256u;
                }
                const uint32_t total = WH_TILE_BYTES + ((a.dbg & 4) ? 0u : (uint32_t)b_rows * 256u);
                for (int kt = 0; kt < KT; kt++, it++) {
                    const uint32_t s = it % NS;
                    if (it >= NS) wt_wait(&empty[s], ((it / NS) & 1) ^ 1, t0);
                    __syncwarp();
                    if (lane == 0) mbar_arrive_expect_tx(&full[s], total);
                    if (bytes) bulk_g2s(smem + s * STAGE + lane * piece, src + (size_t)kt * stride, bytes, &full[s]);
                    __syncwarp();
                }
            }
        }
    } else if (warp == 1) {
        if (CG == 1 || crank == 0) {
            // ------------------------------------ MMA issuer ------------------------------------
            const uint32_t idesc = umma_idesc_f16_f32(128 * CG, a.nt) | (a.bf16 ? ((1u << 7) | (1u << 10)) : 0u);   // a_format = b_format = BF16
            const uint32_t desc_hi = (2048u >> 4) | (1u << 14);      // SBO 2048 B (8-row groups), descriptor version 1
            uint32_t it = 0, tcount = 0;
            for (int t = cid; t < a.n_tiles; t += ncl) {
                WtTile w;
                if (!wt_tile(a, t, w)) continue;
                const uint32_t u = tcount & 1;
                if (tcount >= 2) {      // the epilogue(s) of the tile that last used this accumulator are done with it
                    if (CG == 2) wt_wait_cluster(&acc_empty[u], ((tcount >> 1) & 1) ^ 1, t0);
                    else wt_wait(&acc_empty[u], ((tcount >> 1) & 1) ^ 1, t0);
                }
                tc_fence_after();
                for (int kt = 0; kt < KT; kt++, it++) {
                    const uint32_t s = it % NS, ph = (it / NS) & 1;
                    if (CG == 2) wt_wait_cluster(&full[s], ph, t0);
                    else wt_wait(&full[s], ph, t0);
                    tc_fence_after();
                    if (elect_one()) {
                        const uint32_t sa = smem_u32(smem + s * STAGE);
                        const uint32_t a_lo = ((sa & 0x3FFFFu) >> 4) | ((128u >> 4) << 16);      // LBO 128 B
                        const uint32_t b_lo = (((sa + WH_TILE_BYTES) & 0x3FFFFu) >> 4) | ((128u >> 4) << 16);
#pragma unroll
                        for (int j = 0; j < 8; j++) {      // 8 x K=16: two core matrices (256 B) further along K each
                            if (a.dbg & 2) break;
                            uint64_t da, db;
                            asm("mov.b64 %0, {%1, %2};" : "=l"(da) : "r"(a_lo + j * 16), "r"(desc_hi));
                            asm("mov.b64 %0, {%1, %2};" : "=l"(db) : "r"(b_lo + j * 16), "r"(desc_hi));
                            wt_mma<CG>(tmem_base + u * WT_NT, da, db, idesc, (kt > 0 || j > 0) ? 1u : 0u);
                        }
                        wt_commit<CG>(&empty[s]);
                        if (kt == KT - 1) wt_commit<CG>(&acc_full[u]);
                    }
                    __syncwarp();
                }
                tcount++;
            }
        }
    } else {
        // ------------------------------------ epilogue ------------------------------------
        // warp = (TMEM lane quarter eq, group eg): group eg drains columns [8 eg, 8 eg + 8) of each 32-column chunk
        // into the smem tile and then handles activation rows eg, eg + 4, ... of the chunk
        const int eq = warp & 3, eg = (warp - 2) >> 2;
        const int etid = eq * 32 + lane;
        uint32_t tcount = 0;
        const uint32_t leader_ae = (CG == 2) ? mapa_shared(smem_u32(acc_empty), 0) : 0u;
        bool first = true;
        for (int t = cid; t < a.n_tiles; t += ncl) {
            WtTile w;
            if (!wt_tile(a, t, w)) continue;
            const int rt = w.rp * CG + (int)crank;
            const int m0 = w.mt * a.nt;
            const int Mt = min(a.nt, w.rows - m0);
            const uint32_t u = tcount & 1;
            wt_wait(&acc_full[u], (tcount >> 1) & 1, t0);
            tc_fence_after();
            if (first) { pdl_wait(); first = false; }
            const uint32_t tq = tmem_base + ((uint32_t)(eq * 32) << 16) + u * WT_NT;
            auto drained = [&] {      // every warp has read its last columns: the accumulator is free
                if (tid != 64) return;
                if (CG == 2 && crank != 0) mbar_arrive_remote(leader_ae + u * 8);
                else mbar_arrive(&acc_empty[u]);
            };
            if (a.vec) {
                const int n_chunks = (Mt + WT_VEC_CHUNK - 1) / WT_VEC_CHUNK;
                for (int ch = 0; ch < n_chunks; ch++) {
                    uint32_t v[2][8];
#pragma unroll
                    for (int h = 0; h < 2; h++) tmem_ld_32x32b_x8(tq + (uint32_t)(ch * WT_VEC_CHUNK + eg * 16 + h * 8), v[h]);
                    tmem_ld_wait();
#pragma unroll
                    for (int h = 0; h < 2; h++)
#pragma unroll
                        for (int j = 0; j < 8; j++) out_s[(eg * 16 + h * 8 + j) * EPI_TILE_LD + etid] = __uint_as_float(v[h][j]);
                    tc_fence_before();
                    asm volatile("bar.sync 1, 512;" ::: "memory");
                    if (ch == n_chunks - 1) drained();
                    if (!(a.dbg & 1))
                        epilogue_vec<2>(a.epi, EpiTile{out_s, EPI_TILE_LD}, rt * 128, a.d_real, min(WT_VEC_CHUNK, Mt - ch * WT_VEC_CHUNK),
                                        w.row0 + m0 + ch * WT_VEC_CHUNK, warp - 2, 16, [] {});
                    asm volatile("bar.sync 1, 512;" ::: "memory");
                }
                tcount++;
                continue;
            }
            const int n_chunks = (Mt + WT_EPI_CHUNK - 1) / WT_EPI_CHUNK;
            for (int ch = 0; ch < n_chunks; ch++) {
                const int mc = min(WT_EPI_CHUNK, Mt - ch * WT_EPI_CHUNK);
                uint32_t v[8];
                tmem_ld_32x32b_x8(tq + (uint32_t)(ch * WT_EPI_CHUNK) + eg * 8, v);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 8; j++) out_s[(eg * 8 + j) * 128 + etid] = __uint_as_float(v[j]);
                tc_fence_before();
                asm volatile("bar.sync 1, 512;" ::: "memory");
                if (ch == n_chunks - 1) drained();
                if (!(a.dbg & 1)) epilogue_rows(a.epi, out_s, 128, 128, rt * 128, a.d_real, mc, w.row0 + m0 + ch * WT_EPI_CHUNK, etid, eg, 4);
                asm volatile("bar.sync 1, 512;" ::: "memory");
            }
            tcount++;
        }
    }
    tc_fence_before();
    __syncthreads();
    if (CG == 2) wt_cluster_sync();      // nobody leaves while the partner may still arrive on its barriers
    if (warp == 1) {
        tc_fence_after();
        wt_tmem_dealloc<CG>(tmem_base);
    }
    epilogue_complete(a.epi, tid, a.n_epi_ctas, sflag);
    trace_end(a.tr);
}

// ------------------------------------------------------------------------------------------------
// Q40T -> WH: one CTA per 128 x 128 tile, thread = (row, 32-block).  Same arithmetic as the dequantisers of
// gemm_q40_tc.cu (q40_expand).
// ------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(512) q40t_to_wh_kernel(const uint8_t* __restrict__ q40t, uint8_t* __restrict__ wh) {
    const uint8_t* raw = q40t + (size_t)blockIdx.x * Q40T_TILE_BYTES;
    uint8_t* out = wh + (size_t)blockIdx.x * WH_TILE_BYTES;
    const int r = threadIdx.x & 127, kb = threadIdx.x >> 7;
    const uint4 nb = *reinterpret_cast<const uint4*>(raw + r * 64 + (((kb + (r >> 1)) & 3) << 4));
    const __half d = *reinterpret_cast<const __half*>(raw + Q40T_SCALE_OFF + r * 8 + kb * 2);
    const __half2 d2 = __half2half2(d);
    const uint32_t words[4] = {nb.x, nb.y, nb.z, nb.w};
    uint32_t v[16];
    if (q40_big(*reinterpret_cast<const uint32_t*>(&d2))) q40_expand<true>(words, d2, v);
    else q40_expand<false>(words, d2, v);
    uint8_t* dst = out + (size_t)(r >> 3) * XH_ROWGROUP_BYTES + (size_t)(kb * 4) * 128 + (size_t)(r & 7) * 16;
#pragma unroll
    for (int w = 0; w < 4; w++) *reinterpret_cast<uint4*>(dst + w * 128) = make_uint4(v[4 * w], v[4 * w + 1], v[4 * w + 2], v[4 * w + 3]);
}

extern void dl_set_error(const char* fmt, ...);
extern "C" int dl_device_sm_count();

// ------------------------------------------------------------------------------------------------
// Few activation rows (batched decoding of dense-weight models): y[m][r] for M <= WS_MAX_NT rows, epilogues of DL_EPI_DENSE.
//
// What bounds it: the weights' bytes.  The 256 x 256 pair tiles above give a 4096-wide output 16 of the 74 pairs, and 28672
// columns 112 tiles in two waves: norm, gate|up and down of 4096 x 14336 in bf16 at 32 rows took 184 us, 1.9 TB/s
// (74 here, the launches chained: 42.4 and 25.3 us for the products alone, 5.5 and 4.6 TB/s).  Here the OUTPUT
// COLUMNS are dealt to all SMs in groups of 8 (one core-matrix row group of the weight image, 2 KB per k tile), so every SM
// streams the same number of bytes to within 8 rows; a CTA walks the whole K (or its share of a cluster's) once through a
// ring of bulk copies, MMA M = 128 with the rows past its share reading whatever lies behind (those accumulator lanes are
// never looked at), and drains once.
//
// K split: each cluster of S CTAs reads all activations, (SMs / S) M K against N K of weights, and walks K / S; the shares meet in
// distributed shared memory, each CTA summing and finishing its part of the activation rows in rank order (ws_split: when).
// ------------------------------------------------------------------------------------------------
#define WS_MAX_NT 128
#define WS_THREADS 352
#define WS_MAX_ROWS 256                // output columns per CTA: two accumulators of 128 lanes
#define WS_PIECE 16                    // row groups (2 KB each) per bulk copy: as few copies as the image's tiles allow (32 rows, 4096 x 14336 32.2 us in fours, 26.2 in eights, 25.8 so)
#define WS_HINT 2                      // stages that are asked for while the previous kernel ends: more only delay its own (78.4 us for all nine, 73.8 for two)
#define WS_SMEM (208 * 1024)           // ring + what the last stage's MMA reads behind it

struct WsArgs {
    const uint8_t* wh;
    const uint8_t* xh;
    int d_real, R8, KT, ncap, M, NT, S, NS, nacc, stage, tmem_cols, bf16;
    DlEpilogue epi;
};

__global__ void __launch_bounds__(WS_THREADS, 1) gemm_wh_rows_kernel(const __grid_constant__ WsArgs a) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint64_t full[16], empty[16], acc_full;
    __shared__ uint32_t tmem_holder;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int S = a.S, KT = a.KT, NT = a.NT;
    const int crank = S > 1 ? (int)cg::this_cluster().block_rank() : 0;
    const int c = blockIdx.x / S, n = gridDim.x / S;
    const int g0 = (int)((long long)a.R8 * c / n), g1 = (int)((long long)a.R8 * (c + 1) / n), ng = g1 - g0;      // this CTA's row groups
    const int kt0 = KT * crank / S, nk = KT * (crank + 1) / S - kt0;
    const int nb = (a.M + 7) >> 3;                               // live row groups of the activations
    const int a_bytes = ng * 2048, b_off = a.stage - NT * 256;   // stage: weights, then activations

    const int nacc = min(a.nacc, nk), acc_step = a.tmem_cols >> 1, tile_step = acc_step >> 1;      // accumulators = issuing warps; columns from one to the next
    if (tid == 0) {
        for (int s = 0; s < a.NS; s++) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        mbar_init(&acc_full, nacc);
        mbar_fence_init();
    }
    if (warp == 1) tmem_alloc(&tmem_holder, a.tmem_cols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_holder, 0);
    pdl_launch_dependents();
    // the waits' deadline runs from the end of the kernel ahead: this one may start long before it
    if (warp != 0) pdl_wait();
    unsigned long long t0 = globaltimer_ns();

    if (warp == 0) {
        // lane = one bulk copy per stage: pieces of the weights' row groups (cut at the image's 128-row tiles), then of the activations
        const uint8_t* src = nullptr;
        size_t step = 0;
        uint32_t bytes = 0, dst = 0;
        int l = 0;
        for (int g = g0; g < g1; l++) {
            const int len = min(min(WS_PIECE, g1 - g), 16 - (g & 15));
            if (l == lane) {
                src = a.wh + ((size_t)(g >> 4) * KT + kt0) * WH_TILE_BYTES + (size_t)(g & 15) * 2048;
                step = WH_TILE_BYTES;
                bytes = len * 2048;
                dst = (g - g0) * 2048;
            }
            g += len;
        }
        const bool is_w = bytes != 0;
        for (int g = 0; g < nb; g += WS_PIECE, l++) {
            if (l == lane) {
                src = a.xh + ((size_t)kt0 * (a.ncap >> 3) + g) * 2048;
                step = (size_t)(a.ncap >> 3) * 2048;
                bytes = min(WS_PIECE, nb - g) * 2048;
                dst = b_off + g * 2048;
            }
        }
        // the weights' first stages are on their way into L2 while the previous kernel ends (a hint: a kernel that still writes them is waited for)
        for (int i = 0; is_w && i < min(nk, min(a.NS, WS_HINT)); i++)
            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src + (size_t)i * step), "r"(bytes) : "memory");
        pdl_wait();
        t0 = globaltimer_ns();
        for (int i = 0; i < nk; i++) {
            const int s = i % a.NS;
            if (i >= a.NS) wt_wait(&empty[s], ((i / a.NS) & 1) ^ 1, t0);
            if (lane == 0) mbar_arrive_expect_tx(&full[s], a_bytes + nb * 2048);
            if (bytes) bulk_g2s(smem + (size_t)s * a.stage + dst, src + (size_t)i * step, bytes, &full[s]);
        }
    } else if (warp <= nacc) {
        // up to two warps issue in turn, each into accumulators of its own (the drain adds them): a k tile costs its issuing thread ~570 clk of
        // waits and issue (with one MMA at a time; norm, gate|up and down of 4096 x 14336 at 32 rows 79.9 us then, 78.0 in groups of eight), more than the bytes of a narrow share take to arrive
        const int mw = warp - 1;
        const uint32_t idesc = umma_idesc_f16_f32(128, NT) | (a.bf16 ? ((1u << 7) | (1u << 10)) : 0u);
        const uint32_t desc_hi = (2048u >> 4) | (1u << 14);      // SBO 2048 B, descriptor version 1
        const int tiles = ng > 16 ? 2 : 1;
        const uint32_t lo0 = ((smem_u32(smem) & 0x3FFFFu) >> 4) | ((128u >> 4) << 16);      // LBO 128 B
        for (int i = mw; i < nk; i += nacc) {
            const int s = i % a.NS;
            wt_wait(&full[s], (i / a.NS) & 1, t0);
            tc_fence_after();
            __syncwarp();
            const uint32_t a_lo = lo0 + (uint32_t)((s * a.stage) >> 4), b_lo = a_lo + (uint32_t)(b_off >> 4);
            for (int t = 0; t < tiles; t++)
                umma_f16_ss_x8(tmem + mw * acc_step + t * tile_step, a_lo + t * (WH_TILE_BYTES >> 4), b_lo, desc_hi, idesc, i > mw ? 1u : 0u);
            umma_commit_elected(&empty[s]);
            if (i + nacc >= nk) umma_commit_elected(&acc_full);
        }
    }
    // accumulators -> shared memory [m][rows] in the ring's place (every copy has landed and every MMA is done)
    wt_wait(&acc_full, 0, t0);
    tc_fence_after();
    float* out_s = reinterpret_cast<float*>(smem);
    const int rows = ng * 8;
    if (warp >= 3) {
        const int q = warp & 3, half = (warp - 3) >> 2;           // TMEM lane quarter; the other four warps take every other 8 columns
        for (int t = 0; t * 128 < rows; t++) {
            const int r = t * 128 + q * 32 + lane;
            if (t * 128 + q * 32 >= rows) break;
            for (int m = half * 8; m < a.M; m += 16) {
                const uint32_t at = tmem + ((uint32_t)(q * 32) << 16) + t * tile_step + m;
                uint32_t v[8], w[8];
                tmem_ld_32x32b_x8(at, v);
                if (nacc > 1) tmem_ld_32x32b_x8(at + acc_step, w);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 8; j++)
                    if (r < rows && m + j < a.M) out_s[(m + j) * rows + r] = __uint_as_float(v[j]) + (nacc > 1 ? __uint_as_float(w[j]) : 0.f);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem, a.tmem_cols); }
    int m0 = 0, m1 = a.M;
    if (S > 1) {
        cg::cluster_group cluster = cg::this_cluster();
        cluster.sync();
        m0 = a.M * crank / S;
        m1 = a.M * (crank + 1) / S;
        for (int i = m0 * rows + tid; i < m1 * rows; i += WS_THREADS) {
            float v = 0.f;
            for (int k = 0; k < S; k++) v += cluster.map_shared_rank(out_s, k)[i];
            out_s[i] = v;                                          // nobody else reads these rows
        }
        cluster.sync();                                            // no peer still reads this CTA's memory when it leaves
    }
    const bool pair = a.epi.dense_op == DL_DENSE_GLU_CLAMP || a.epi.dense_op == DL_DENSE_GLU_SILU || a.epi.dense_op == DL_DENSE_GLU_GELU;
    const int na = pair ? rows >> 1 : rows, step = na ? max(1, WS_THREADS / na) : 1;      // threads along the columns, several rows at a time
    for (int t = tid; t < na * step; t += WS_THREADS)
        epilogue_rows(a.epi, out_s + m0 * rows, rows, rows, g0 * 8, a.d_real, m1 - m0, m0, t % na, t / na, step);
}

// CTAs per cluster that share K: shares of fewer than 5 row groups (40 columns) leave an SM more activations than weights to read and
// too many k tiles to walk; a pair halves both (32 rows, us with 1 / 2 / 4: 4096 x 14336 41 / 25 / 38, 2048 x 8192 24 / 16 / 22, 128 x 2048
// 11 / 10 / 10; but 6144 x 2048 at 100 rows 21 / 21 / 41, 16384 x 2048 19 / 25 / 41, 28672 x 4096 47 / 60 / 82)
static int ws_split(int R8, int KT, int n_sms) { return R8 < 5 * n_sms && KT >= 2 ? 2 : 1; }

static int gemm_wh_rows_launch(const uint8_t* wh, int d, int n, const uint8_t* xh, int ncap, int M, const DlEpilogue* epi, int bf16,
                               cudaStream_t stream, int n_sms) {
    WsArgs a;
    a.wh = wh; a.xh = xh; a.d_real = d; a.R8 = (d + 7) / 8; a.KT = n / 128; a.ncap = ncap; a.M = M;
    a.NT = (M + 15) / 16 * 16;
    a.bf16 = bf16; a.epi = *epi;
    a.S = ws_split(a.R8, a.KT, n_sms);
    const int slots = n_sms / a.S;
    int clusters = a.R8 < slots ? a.R8 : slots;
    clusters *= (a.R8 + clusters * (WS_MAX_ROWS / 8) - 1) / (clusters * (WS_MAX_ROWS / 8));      // more columns than one wave holds
    const int ng = (a.R8 + clusters - 1) / clusters;
    a.stage = ng * 2048 + a.NT * 256;
    // an MMA reads 128 (256) rows of weights from the start of its stage whatever the CTA's share is
    const int over = (ng > 16 ? 2 : 1) * WH_TILE_BYTES > a.stage ? (ng > 16 ? 2 : 1) * WH_TILE_BYTES - a.stage : 0;
    a.NS = (WS_SMEM - over) / a.stage;
    if (a.NS > 16) a.NS = 16;
    // A stage must belong to ONE issuer: with an odd count its uses would alternate between the two, and an issuer that runs ahead
    // would take the parity of the use before last for its own.  Two issuers are worth a stage (32 rows, 4096 x 14336: 32.0 us with nine
    // stages and one issuer, 27.6 with eight and two) until only three are left, of wide shares whose bytes cover one issuer.
    if (a.NS > 3) a.NS &= ~1;
    a.nacc = a.NS % 2 == 0 ? 2 : 1;
    a.tmem_cols = 32;
    while (a.tmem_cols < 4 * a.NT) a.tmem_cols *= 2;            // two issuers x two tiles
    static SmemLimit given;
    if (const int rc = dl_smem_limit("gemm wh rows", gemm_wh_rows_kernel, WS_SMEM, given)) return rc;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(clusters * a.S));
    cfg.blockDim = dim3(WS_THREADS);
    cfg.dynamicSmemBytes = WS_SMEM;
    cfg.stream = stream;
    cudaLaunchAttribute attrs[2];
    int na = 0;
    if (a.S > 1) {
        attrs[na].id = cudaLaunchAttributeClusterDimension;
        attrs[na].val.clusterDim.x = a.S;
        attrs[na].val.clusterDim.y = 1;
        attrs[na].val.clusterDim.z = 1;
        na++;
    }
    attrs[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;      // it waits by itself before it reads what others wrote
    attrs[na].val.programmaticStreamSerializationAllowed = 1;
    na++;
    cfg.attrs = attrs;
    cfg.numAttrs = na;
    cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_wh_rows_kernel, a);
    if (e != cudaSuccess) { dl_set_error("gemm wh rows launch: %s", cudaGetErrorString(e)); return -(int)e; }
    return 0;
}

static int g_wh_dbg = 0, g_wh_piece = 16384;      // bytes per bulk copy: 16 KB pieces (4 / 8 KB measured: no gain)
extern "C" void dl_debug_set_wh_piece(int b) { if (b == 4096 || b == 8192 || b == 16384) g_wh_piece = b; }
extern "C" void dl_debug_set_wh_mode(int m) { g_wh_dbg = m; }

extern "C" long long dl_wh_bytes(int d, int n) { return (long long)((d + 127) / 128) * (n / 128) * WH_TILE_BYTES; }

extern "C" int dl_q40t_to_wh(const uint8_t* q40t, int d, int n, uint8_t* wh, void* stream) {
    if (n % 128 != 0 || d < 1) { dl_set_error("dl_q40t_to_wh: n=%d must be a multiple of 128", n); return -1; }
    const int tiles = ((d + 127) / 128) * (n / 128);
    q40t_to_wh_kernel<<<tiles, 512, 0, (cudaStream_t)stream>>>(q40t, wh);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) { dl_set_error("dl_q40t_to_wh: %s", cudaGetErrorString(e)); return -(int)e; }
    return 0;
}

// Rows per tile: the width for which the tiles of the busiest CTA (pair) take least time.  Half of a 256-row tile's time stays whatever its rows are (the
// weights' copies and each stage's hand-off: 768 rows of 4096 x 14336 in one round of tiles of 256 or 192 are 8 % apart), so rows that are not there
// are saved, and rounds are not added for narrower ones.
static int wh_tile_rows(int row_units, int M, int slots) {
    int best = WT_NT;
    long long least = -1;
    for (int nt = WT_NT; nt >= 128; nt -= 32) {
        const long long rounds = ((long long)row_units * ((M + nt - 1) / nt) + slots - 1) / slots, cost = rounds * (nt + 256);
        if (least < 0 || cost < least) { least = cost; best = nt; }
    }
    return best;
}

// the operands of a pair's copies as [slab][row group][2 KB]: of the activations, no row group behind the last that has a row
static int wh_pair_maps(const WhArgs& a, CUtensorMap* wmap, CUtensorMap* xmap) {
    const cuuint64_t tiles = (a.n_groups - 1) * (a.wh_group_bytes / WH_TILE_BYTES) + (cuuint64_t)a.row_tiles * a.KT, x_groups = (a.grp ? a.ncap : a.M + 7) / 8;
    const cuuint64_t wd[3] = {256, 16, tiles}, ws[2] = {XH_ROWGROUP_BYTES, WH_TILE_BYTES}, xd[3] = {256, x_groups, (cuuint64_t)a.KT};
    const cuuint64_t xs[2] = {XH_ROWGROUP_BYTES, (cuuint64_t)a.ncap / 8 * XH_ROWGROUP_BYTES};
    const cuuint32_t wb[3] = {256, 8, 1}, xb[3] = {256, (cuuint32_t)a.nt / 32, 1};
    if (dl_tensor_map("dl_gemm_wh_tc", wmap, CU_TENSOR_MAP_DATA_TYPE_INT64, 3, a.wh, wd, ws, wb, CU_TENSOR_MAP_SWIZZLE_NONE) != 0) return -1;
    return dl_tensor_map("dl_gemm_wh_tc", xmap, CU_TENSOR_MAP_DATA_TYPE_INT64, 3, a.xh, xd, xs, xb, CU_TENSOR_MAP_SWIZZLE_NONE);
}

// force_cg: bit 0: 0 = pairs when the row-tile count is even, 1 = single CTAs (for tests and comparisons);
// bit 1: the images hold bf16 (written by dl_wh_from_dense / dl_xh_from_rows) instead of fp16
static int gemm_wh_launch(const uint8_t* wh, int d, int n, const uint8_t* xh, int ncap, int M, const DlEpilogue* epi,
                          int force_cg, int pdl, const int* grp, int n_groups, long long wh_group_bytes, void* stream) {
    if (n % 128 != 0) { dl_set_error("dl_gemm_wh_tc: n=%d not a multiple of 128", n); return -1; }
    if (M < 1 || ncap % 8 != 0 || ncap < M) { dl_set_error("dl_gemm_wh_tc: bad M=%d / ncap=%d", M, ncap); return -1; }
    if (epi->kind == DL_EPI_SILU_MUL && d % 64 != 0) { dl_set_error("dl_gemm_wh_tc: silu epilogue needs d%%64==0"); return -1; }
    // few rows: all SMs stream equal shares of the weights (force_cg bit 0 keeps the tiles below, for comparisons)
    if (epi->kind == DL_EPI_DENSE && grp == nullptr && M <= WS_MAX_NT && !(force_cg & 1))
        return gemm_wh_rows_launch(wh, d, n, xh, ncap, M, epi, (force_cg & 2) ? 1 : 0, (cudaStream_t)stream, dl_device_sm_count());
    WhArgs a;
    a.wh = wh; a.xh = xh; a.d_real = d;
    a.row_tiles = (d + 127) / 128;
    a.KT = n / 128; a.ncap = ncap; a.M = M;
    const int cg = ((force_cg & 1) || (a.row_tiles & 1) || wh_group_bytes % WH_TILE_BYTES != 0) ? 1 : 2, n_sms = dl_device_sm_count();
    a.nt = grp == nullptr ? wh_tile_rows(a.row_tiles / cg, M, n_sms / cg) : WT_NT;      // (groups: their rows are not known here)
    a.m_tiles = (M + a.nt - 1) / a.nt;
    a.bf16 = (force_cg & 2) ? 1 : 0;
    a.grp = grp; a.n_groups = n_groups; a.wh_group_bytes = wh_group_bytes;
    a.n_tiles = n_groups * (a.row_tiles / cg) * a.m_tiles;
    int grid = (n_sms / cg) * cg;
    if (grid > a.n_tiles * cg) grid = a.n_tiles * cg;
    a.n_epi_ctas = grid;
    a.epi = *epi;
    a.vec = epilogue_vec_ok(*epi, d);
    a.dbg = g_wh_dbg;
    a.piece = g_wh_piece;
    a.tr = dl_trace_next(TR_TC);
    const size_t smem = 196608 + WT_VEC_CHUNK * EPI_TILE_LD * 4 + 16 * 8 + 16;
    static SmemLimit given[2];
    if (const int rc = cg == 2 ? dl_smem_limit("gemm wh", gemm_wh_tc_kernel<2>, smem, given[1]) : dl_smem_limit("gemm wh", gemm_wh_tc_kernel<1>, smem, given[0])) return rc;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(WT_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = (cudaStream_t)stream;
    cudaLaunchAttribute attrs[2];
    int na = 0;
    if (cg == 2) {
        attrs[na].id = cudaLaunchAttributeClusterDimension;
        attrs[na].val.clusterDim.x = 2;
        attrs[na].val.clusterDim.y = 1;
        attrs[na].val.clusterDim.z = 1;
        na++;
    }
    if (pdl) {
        attrs[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attrs[na].val.programmaticStreamSerializationAllowed = 1;
        na++;
    }
    cfg.attrs = attrs;
    cfg.numAttrs = na;
    alignas(64) CUtensorMap wmap = {}, xmap = {};
    if (cg == 2 && wh_pair_maps(a, &wmap, &xmap) != 0) return -1;
    cudaError_t e = (cg == 2) ? cudaLaunchKernelEx(&cfg, gemm_wh_tc_kernel<2>, a, wmap, xmap) : cudaLaunchKernelEx(&cfg, gemm_wh_tc_kernel<1>, a, wmap, xmap);
    if (e != cudaSuccess) { dl_set_error("gemm wh launch: %s", cudaGetErrorString(e)); return -(int)e; }
    return 0;
}

extern "C" int dl_gemm_wh_tc(const uint8_t* wh, int d, int n, const uint8_t* xh, int ncap, int M, const DlEpilogue* epi,
                             int force_cg, int pdl, void* stream) {
    return gemm_wh_launch(wh, d, n, xh, ncap, M, epi, force_cg, pdl, nullptr, 1, 0, stream);
}

// One product per group: group g < n_groups multiplies activation rows [grp[2g], grp[2g] + grp[2g+1]) of xh (grp in DEVICE
// memory, first rows multiples of 8, every group at most max_group_rows rows) with the weight image at
// wh + g * wh_group_bytes, and writes those rows of the output.
extern "C" int dl_gemm_wh_tc_grouped(const uint8_t* wh, long long wh_group_bytes, int n_groups, const int* grp, int d, int n,
                                     const uint8_t* xh, int ncap, int max_group_rows, const DlEpilogue* epi, int force_cg,
                                     void* stream) {
    if (n_groups < 1 || grp == nullptr || max_group_rows < 1) { dl_set_error("dl_gemm_wh_tc_grouped: bad groups"); return -1; }
    if (max_group_rows > ncap) max_group_rows = ncap;
    return gemm_wh_launch(wh, d, n, xh, ncap, max_group_rows, epi, force_cg, 0, grp, n_groups, wh_group_bytes, stream);
}
