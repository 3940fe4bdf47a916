// Q40 x Q80 -> f32 matmul on the 5th-gen tensor cores (tcgen05 / TMEM), M = 9 .. thousands of
// activation rows: batched multi-user decode and prompt prefill.
//
// The reference's exact arithmetic rescales every 32-element block by d_w*d_x (nn-cpu-ops.cpp:
// 352-377), which a TMEM accumulator cannot do between MMAs.  So the scales are folded into the
// operands: W tiles are dequantised Q40 -> fp16 ((nibble-8)*d, one rounding) on the fly, activations
// arrive as fp16(q*d) in the XH layout, and `tcgen05.mma.kind::f16` accumulates in f32 in TMEM.
// "swap-AB": the 128 weight rows are the MMA M dimension (TMEM lanes), activation rows are the N
// dimension (16..256 per CTA), so small user batches still fill the tensor core's M.
//
// The dequantised weights never touch shared memory: the dequant warps read the raw 4.5-bit tile,
// expand it in registers and write it with tcgen05.st straight into TENSOR MEMORY, and the MMA takes
// its A operand from there (`tcgen05.mma [d], [a_tmem], b_desc`).  The first version staged fp16 A
// tiles in smem: 32 KB written + 32 KB read per 9 KB of weights saturated the 128 B/clk crossbar
// (1450 clk per k-tile, all of it in the MMA queue).
//
// Warp roles (608 threads):
//   warp 0       producer: bulk async copies of raw 9 KB Q40T tiles (lanes 0-3) and XH slabs (lanes 4-7)
//   warps 1,18   MMA issuers (one elected lane each; tcgen05.mma / tcgen05.commit), k-tiles round-robin,
//                one accumulator each; warp 1 also allocates TMEM
//   warps 2-17   dequantisers, 4 groups x 4 warps: group = k-tile % 4 = A stage, warp % 4 = TMEM lane
//                quarter, thread = weight row: LDS.128 x4 -> packed fp16x2 registers -> tcgen05.st.32x32b.x16
//   warps 2-17   (again) epilogue: tcgen05.ld TMEM -> registers -> smem tile -> fused epilogue (rows split 4 ways)
// TMEM columns: nacc f32 accumulators of NT columns from column 0, nstg 64-column A stages at the top
// (nacc*NT + 64*nstg <= 512: 2 accumulators + 6 stages up to NT = 64, 2 + 4 for 128, 1 + 4 above).
// What bounds narrow tiles: the dequantisers' stores into tensor memory and their instructions (a k-tile 474 clk; 322, HBM's pace for 112 CTAs, without the
// stores, 395 without the arithmetic).
// Pipelines: raw ring (producer -> dequant), B ring (producer -> MMA), A stages (dequant -> MMA,
// released by tcgen05.commit), accumulator barrier (MMA -> epilogue).  K can be split over a
// thread-block cluster (DSMEM reduction) when there are too few row tiles to fill the chip.
#define WAIT_UNIT 2u
#include "epilogue.cuh"
#include "smem_limit.cuh"
#include "waits.cuh"

#define TC_DEQ_WARPS 16
#define TC_THREADS (64 + TC_DEQ_WARPS * 32 + 32)      // producer, MMA warp 0, dequantisers, MMA warp 1
#define TC_EPI_CHUNK 32           // activation rows per epilogue pass
#define TC_TMEM_COLS 512
#define TC_A_STAGE_COLS 64        // 128 K x fp16 = 64 32-bit columns per lane
// dequantiser groups (k-tile i -> group i % 4).  Four: a stage of either ring must come back to the group that had it, or to one that has waited behind it
// (a parity wait cannot see a phase before the last), so the count divides the raw stages; six groups (48 more registers spilled a thread) are slower, 369 us for 359.
#define TC_GROUPS 4

struct TcArgs {
    const uint8_t* w;
    const uint8_t* xh;
    int d_real, d_pad, KT, ncap, M, NT, S;
    int NSA, NSB, nsb_log;
    int nstg;              // A stages in TMEM (64 columns each), at columns [512 - 64*nstg, 512)
    int pair;              // 1: this CTA multiplies row tiles 2c and 2c + 1 side by side (item i = row tile i & 1, k-tile i >> 1; one accumulator each)
    int nacc;              // MMA-issuing warps = independent TMEM accumulators (1 or 2; nacc*NT <= 256), summed by the epilogue
    int LA, LB;            // issuing lanes per ring; each divides its stage count so a stage has ONE owner lane
    int n_epi_ctas;
    int vec;               // epilogue_vec takes the epilogue
    unsigned long long* tr;
    int dbg_mode;          // debug timing experiments (results invalid): 1 = one MMA per k-tile, 2 = no dequant/STTM; 16 = no weights behind the first ringful (a limit of no time: tests)
    long long* dbg;        // debug: per-tile clock64 stamps of CTA 0 (dl_debug_set_tc_trace), [tile][8]
    DlEpilogue epi;
    WaitLimit limit;
};

#define TC_DBG(slot, i) do { if (a.dbg && blockIdx.x == 0 && blockIdx.y == 0 && (i) < 64) a.dbg[(i) * 8 + (slot)] = clock64(); } while (0)

// The waits of the dequantisers, the issuers and the epilogue have no limit of their own (with one in each a step of 32 rows of width 4096 and 4 layers
// took 353 to 359 us for 350): the producer, which has nothing else to do by then, ends them.  It gives up where it can issue nothing, or has
// issued all and sees no end, for longer than the limit; then, its copies having landed, it fills the weights' ring with scales that are NaN and says of every
// stage that it is full and free until the accumulators are through (a stage may be multiplied as it was, so most of what is stored then is NaN, not all).
static __device__ __noinline__ void tc_end_waits(uint8_t* ringA, int bytes, uint64_t* fullA, uint64_t* fullB, uint64_t* fullH, uint64_t* emptyH, uint64_t* accum_full) {
    wait_settle();
    for (int i = 0; i < bytes / 4; i++) reinterpret_cast<volatile uint32_t*>(ringA)[i] = 0xFFFFFFFFu;
    for (int n = 0; n < (1 << 20) && !mbar_test_wait(accum_full, 0); n++) {
        for (int s = 0; s < 16; s++) {
            mbar_arrive(&fullA[s]);
            if (s >= 8) continue;
            mbar_arrive(&fullB[s]);
            mbar_arrive(&emptyH[s]);
            for (int j = 0; j < 4; j++) mbar_arrive(&fullH[s]);
        }
        __nanosleep(500);
    }
}

__global__ void __launch_bounds__(TC_THREADS, 1) gemm_q40_tc_kernel(const __grid_constant__ TcArgs a) {
    extern __shared__ __align__(1024) uint8_t smem[];
    trace_begin(a.tr);
    if (threadIdx.x == 0) TC_DBG(0, 63);
    const int NT = a.NT;
    const int b_bytes = NT * 256;
    uint8_t* ringB = smem;                                          // [NSB][NT*256]
    uint8_t* ringA = ringB + a.NSB * b_bytes;                       // [NSA][9216]
    float* out_s = reinterpret_cast<float*>(ringA + a.NSA * Q40T_TILE_BYTES);   // [32][128]
    uint64_t* bars = reinterpret_cast<uint64_t*>(out_s + TC_EPI_CHUNK * 128);
    uint64_t* fullA = bars;                     // [16]
    uint64_t* emptyA = fullA + 16;              // [16]
    uint64_t* fullB = emptyA + 16;              // [8] each from here
    uint64_t* emptyB = fullB + 8;
    uint64_t* fullH = emptyB + 8;
    uint64_t* emptyH = fullH + 8;
    uint64_t* accum_full = emptyH + 8;
    uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(accum_full + 1);
    int* sflag = reinterpret_cast<int*>(tmem_holder + 1);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int S = a.S;
    const int crank = (S > 1) ? (int)cg::this_cluster().block_rank() : 0;
    const int P = a.pair ? 2 : 1;
    const int rt = (int)(blockIdx.x / S) * P;      // first row tile
    const int m0 = blockIdx.y * NT;
    const int Mt = min(NT, a.M - m0);
    const int kt0 = (a.KT * crank) / S, kt1 = (a.KT * (crank + 1)) / S;
    const int nk = kt1 - kt0;
    const int n_it = nk * P;               // items: weight tiles of this CTA
    const int nacc = a.pair ? 2 : (a.nacc <= nk) ? a.nacc : (nk >= 2 ? 2 : 1);      // accumulators in use = MMA-issuing warps (power of two)

    if (tid == 0) {
        for (int s = 0; s < 16; s++) {
            mbar_init(&fullA[s], 1);
            mbar_init(&emptyA[s], 4);
        }
        for (int s = 0; s < 8; s++) {
            mbar_init(&fullB[s], 1);
            mbar_init(&emptyB[s], P);
            mbar_init(&fullH[s], 4);
            mbar_init(&emptyH[s], 1);
        }
        mbar_init(accum_full, nacc);
        mbar_fence_init();
    }
    if (warp == 1) tmem_alloc(tmem_holder, TC_TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_holder;
    if (threadIdx.x == 0) TC_DBG(1, 63);
    pdl_launch_dependents();

    if (warp == 0) {
        // ------------------------------------ producer ------------------------------------
        // lanes 0..LA-1 stream the raw weight tiles, lanes 4..4+LB-1 the activation slabs: one issuing thread
        // caps a CTA at ~34 GB/s (measured on the GEMV).  A stage has exactly one owner lane (LA | NSA,
        // LB | NSB): a stage shared by two lanes could be lapped by two phases, which a parity wait cannot see.
        // Every lane polls ITS next stage with a non-blocking test_wait inside one converged loop, so a lane
        // whose stage is still busy never holds back a lane whose stage is free (blocking waits serialise the
        // divergent lanes of a warp and let one role starve the other).
        const bool role_a = lane < a.LA, role_b = lane >= 4 && lane < 4 + a.LB;
        const uint8_t* wt = a.w + ((size_t)rt * a.KT + kt0) * Q40T_TILE_BYTES;
        const uint8_t* xb = a.xh + (size_t)kt0 * (a.ncap >> 3) * XH_ROWGROUP_BYTES + (size_t)(m0 >> 3) * XH_ROWGROUP_BYTES;
        const size_t x_kt_stride = (size_t)(a.ncap >> 3) * XH_ROWGROUP_BYTES;
        const uint64_t pol = l2_policy_evict_first();
        const int n_role = role_a ? n_it : nk;
        int i = role_a ? lane : (role_b ? lane - 4 : nk);
        const int step = role_a ? a.LA : a.LB;
        auto tile_of = [&](int it) { return wt + (P == 2 ? (size_t)(it & 1) * a.KT + (it >> 1) : (size_t)it) * Q40T_TILE_BYTES; };
        if (role_a) {
            // weights do not depend on the previous kernel: fill the whole ring before the PDL wait
            for (; i < n_it && i < a.NSA; i += step) {
                if (!(a.dbg_mode & 4)) TC_DBG(0, i);
                mbar_arrive_expect_tx(&fullA[i], Q40T_TILE_BYTES);
                bulk_g2s_hint(ringA + i * Q40T_TILE_BYTES, tile_of(i), Q40T_TILE_BYTES, &fullA[i], pol);
            }
        }
        __syncwarp();
        pdl_wait();
        unsigned idle = 0;
        while (__any_sync(0xffffffffu, i < n_role)) {
            bool issued = false;
            if (i < n_role) {
                if (role_a) {
                    const int sa = i % a.NSA;
                    if (mbar_test_wait(&emptyA[sa], ((i / a.NSA) & 1) ^ 1) && !(a.dbg_mode & 16)) {      // i >= NSA here
                        if (!(a.dbg_mode & 4)) TC_DBG(0, i);
                        mbar_arrive_expect_tx(&fullA[sa], Q40T_TILE_BYTES);
                        bulk_g2s_hint(ringA + sa * Q40T_TILE_BYTES, tile_of(i), Q40T_TILE_BYTES, &fullA[sa], pol);
                        i += step;
                        issued = true;
                    }
                } else {
                    const int sb = i % a.NSB;
                    if (i < a.NSB || mbar_test_wait(&emptyB[sb], ((i / a.NSB) & 1) ^ 1)) {
                        mbar_arrive_expect_tx(&fullB[sb], b_bytes);
                        bulk_g2s(ringB + sb * b_bytes, xb + (size_t)i * x_kt_stride, b_bytes, &fullB[sb]);
                        i += step;
                        issued = true;
                    }
                }
            }
            if (!__any_sync(0xffffffffu, issued)) {
                __nanosleep(40);      // leave the issue slots to the dequantisers
                if ((++idle & 0xFFFu) == 0 && (unsigned long long)idle * 40 >= a.limit.ns) break;      // about 40 ns and more each time
            }
        }
        const bool stuck = __any_sync(0xffffffffu, i < n_role);
        if (lane == 0) {
            if (stuck) wait_report(a.limit);
            // ranks of a cluster meet right behind their accumulators: there the last stage that is filled is looked at instead
            const int last = (n_it - 1) % a.nstg, turn = ((n_it - 1) / a.nstg) & 1;
            if (stuck || !wait_phase(S > 1 ? &fullH[last] : accum_full, S > 1 ? turn : 0, a.limit, true)) tc_end_waits(ringA, a.NSA * Q40T_TILE_BYTES, fullA, fullB, fullH, emptyH, accum_full);
        }
        __syncwarp();
    } else if (warp == 1 || warp >= 2 + TC_DEQ_WARPS) {
        // ------------------------------------ MMA issuers ------------------------------------
        // One k-tile costs its issuing thread ~900 clk of mostly fixed latency (two barrier waits, fence,
        // eight MMAs issued at ~45 clk each, two commits), far more than the MMAs
        // themselves.  Up to two issuing warps take k-tiles round-robin, each into its OWN accumulator
        // (summed by the epilogue), so the result stays bit-deterministic.  Warp-uniform control flow: every
        // lane walks the barriers, one elected lane issues.
        const int mw = (warp == 1) ? 0 : warp - (2 + TC_DEQ_WARPS) + 1;
        const uint32_t idesc = umma_idesc_f16_f32(128, NT);
        // K-major no-swizzle descriptor of B: LBO 128 B (K core matrices), SBO 2048 B (8-row groups); only the
        // 14-bit start-address field changes between MMAs
        const uint32_t desc_hi = (2048u >> 4) | (1u << 14);
        const uint32_t desc_lo0 = ((smem_u32(ringB) & 0x3FFFFu) >> 4) | ((128u >> 4) << 16);
        const uint32_t acc = tmem_base + (uint32_t)(mw * NT);
        const bool det = (a.dbg_mode & 4) != 0;      // detail stamps of warp 1 only (slots 0..7)
        const bool stamp = (lane == 0 && mw == 0 && !(a.dbg_mode & 8));
        const int nsb_mask = a.NSB - 1, nsb_log = a.nsb_log;
        const int nstg = a.nstg;
        const uint32_t a_col0 = TC_TMEM_COLS - nstg * TC_A_STAGE_COLS;
        if (mw < nacc) {
            int sh = mw, ph = 0;      // A stage of k-tile i = i % nstg, phase parity = (i / nstg) & 1
            for (int i = mw; i < n_it; i += nacc) {
                const int k = a.pair ? i >> 1 : i;
                const int sb = k & nsb_mask, pb = (k >> nsb_log) & 1;
                if (det && stamp) TC_DBG(0, i);
                mbar_wait(&fullH[sh], ph);
                if (stamp) TC_DBG(det ? 1 : 5, i);
                mbar_wait(&fullB[sb], pb);
                if (stamp) TC_DBG(det ? 2 : 6, i);
                tc_fence_after();
                if (det && stamp) TC_DBG(3, i);
                if (elect_one()) {
                    const uint32_t a_tmem = tmem_base + a_col0 + sh * TC_A_STAGE_COLS;
                    const uint32_t lo = desc_lo0 + (uint32_t)((sb * b_bytes) >> 4);
#pragma unroll
                    for (int j = 0; j < 8; j++) {      // 8 x K=16 per 128-wide k-tile: 8 TMEM columns of A, 2 core matrices (256 B) of B
                        if ((a.dbg_mode & 1) && j > 0) break;
                        uint64_t db;
                        asm("mov.b64 %0, {%1, %2};" : "=l"(db) : "r"(lo + j * 16), "r"(desc_hi));
                        umma_f16_ts(acc, a_tmem + j * 8, db, idesc, (i != mw || j > 0) ? 1u : 0u);
                    }
                    if (det && mw == 0) TC_DBG(4, i);
                    umma_commit(&emptyH[sh]);          // implicit tcgen05.fence::before_thread_sync
                    umma_commit(&emptyB[sb]);
                    if (i + nacc >= n_it) umma_commit(accum_full);      // this warp's last k-tile
                    if (det && mw == 0) TC_DBG(6, i);
                }
                __syncwarp();
                if (stamp) TC_DBG(7, i);
                sh += nacc;
                if (sh >= nstg) { sh -= nstg; ph ^= 1; }
            }
        }
    } else if (warp < 2 + TC_DEQ_WARPS) {
        // ------------------------------------ dequantisers ------------------------------------
        // Four groups of four warps; group g owns k-tiles g, g+4, ... and A stage g, so the groups' latency
        // chains (raw wait -> LDS -> unpack -> STTM -> wait::st -> arrive) overlap instead of all 16 warps
        // marching through every tile in lock-step.  Inside a group warp = TMEM lane quarter (warp % 4),
        // thread = weight row r, which it expands for the whole 128-wide k-tile (4 blocks of 32).
        const int q = warp & 3, g = (warp - 2) >> 2;
        const int r = q * 32 + lane;
        // consecutive rows rotate their four 16-byte k-block slots, so the 8 lanes of an LDS.128 phase hit
        // 8 distinct bank groups (same layout the GEMV reads row-per-lane)
        const uint32_t row_off = r * 64, rot = (uint32_t)(r >> 1);
        const uint32_t sc_off = Q40T_SCALE_OFF + r * 8;
        const int nstg = a.nstg;
        const uint32_t a_taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (TC_TMEM_COLS - nstg * TC_A_STAGE_COLS);
        const bool stamp = (tid == 64 && !(a.dbg_mode & 12));
        const bool qstamp = (lane == 0 && (a.dbg_mode & 8));      // mode 8: slots 1..4 = arrival time of lane quarter 0..3
        const int nsa = a.NSA;
        int sh = g, ph = 0;      // A stage of k-tile i = i % nstg (g < 4 <= nstg), phase parity = (i / nstg) & 1
        int sa = g, pa = 0;      // raw ring stage i % NSA and its phase parity
        for (int i = g; i < n_it; i += TC_GROUPS) {
            mbar_wait(&fullA[sa], pa);
            if (stamp) TC_DBG(1, i);
            const uint8_t* raw = ringA + sa * Q40T_TILE_BYTES;
            uint4 nb[4];
#pragma unroll
            for (int kb = 0; kb < 4; kb++) nb[kb] = *reinterpret_cast<const uint4*>(raw + row_off + (((kb + rot) & 3) << 4));
            const uint2 sc = *reinterpret_cast<const uint2*>(raw + sc_off);      // 4 fp16 scales of this row
            // the tile now lives in registers: hand the raw stage back BEFORE the unpack (the ring has to cover
            // DRAM latency + queueing; holding a stage through the ~1300 clk unpack halved its effective depth).
            // The loads above were issued by this warp before the arrive and shared-memory operations of a warp
            // complete in order; the refill is >500 ns away (barrier -> producer poll -> HBM fetch).
            __syncwarp();
            if (lane == 0) mbar_arrive(&emptyA[sa]);
            if (i >= nstg) mbar_wait(&emptyH[sh], ph ^ 1);      // the MMAs that read this A stage have retired
            if (stamp) TC_DBG(2, i);
            tc_fence_after();
            const bool big = __any_sync(0xffffffffu, q40_big(sc.x) || q40_big(sc.y));
            auto expand = [&](auto is_big) {
#pragma unroll
                for (int kb = 0; kb < 4; kb++) {
                    const uint32_t sdup = __byte_perm((kb < 2) ? sc.x : sc.y, 0, (kb & 1) ? 0x3232 : 0x1010);
                    const __half2 d2 = *reinterpret_cast<const __half2*>(&sdup);
                    uint32_t v[16];
                    const uint32_t words[4] = {nb[kb].x, nb[kb].y, nb[kb].z, nb[kb].w};
                    q40_expand<decltype(is_big)::value>(words, d2, v);
                    if (!(a.dbg_mode & 2)) tmem_st_32x32b_x16(a_taddr + sh * TC_A_STAGE_COLS + kb * 16, v);
                }
            };
            if (big) expand(BoolIs<true>());
            else expand(BoolIs<false>());
            tmem_st_wait();
            if (stamp) TC_DBG(3, i);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&fullH[sh]);
            if (stamp) TC_DBG(4, i);
            if (qstamp) TC_DBG(1 + q, i);
            sh += TC_GROUPS;
            if (sh >= nstg) { sh -= nstg; ph ^= 1; }
            sa += TC_GROUPS;
            if (sa >= nsa) { sa -= nsa; pa ^= 1; }
        }
    }

    // ---------------------------------------- epilogue ----------------------------------------
    // all 16 dequant warps: warp = (TMEM lane quarter eq, group eg); group eg drains columns [8eg, 8eg+8) of
    // each 32-column chunk into the smem tile, then handles activation rows eg, eg+4, ... of the chunk
    const bool is_epi = (warp >= 2 && warp < 2 + TC_DEQ_WARPS);
    const int eq = warp & 3, eg = (warp - 2) >> 2;
    const int etid = eq * 32 + lane;      // output row of this thread
    if (is_epi) {
        mbar_wait(accum_full, 0);
        tc_fence_after();
        if (tid == 64) TC_DBG(2, 63);
    }
    const int n_chunks = (Mt + TC_EPI_CHUNK - 1) / TC_EPI_CHUNK;
    // columns [8 eg, 8 eg + 8) of chunk ch of row tile rt + h -> dst[column][ld] (with one row tile: the sum over the accumulators)
    auto drain = [&](int h, int ch, float* dst, int ld) {
        const uint32_t taddr = tmem_base + ((uint32_t)(eq * 32) << 16) + (uint32_t)(h * NT + ch * TC_EPI_CHUNK);
        const int ncol = min(TC_EPI_CHUNK, NT - ch * TC_EPI_CHUNK);
        const int c0 = eg * 8;
        if (c0 < ncol) {
            uint32_t v[8];
            tmem_ld_32x32b_x8(taddr + c0, v);
            tmem_ld_wait();
            float f[8];
#pragma unroll
            for (int j = 0; j < 8; j++) f[j] = __uint_as_float(v[j]);
            for (int ac = 1; ac < nacc && !a.pair; ac++) {
                tmem_ld_32x32b_x8(taddr + c0 + ac * NT, v);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 8; j++) f[j] += __uint_as_float(v[j]);
            }
#pragma unroll
            for (int j = 0; j < 8; j++) dst[(c0 + j) * ld + etid] = f[j];
        }
    };
    if (S > 1) {
        // split-K (of a single row tile: pairs are for more row tiles than SMs): every rank publishes its partial tile in the rings' place, then
        // sums and finishes ITS share of the activation rows over DSMEM, in rank order.  (One rank finishing all rows chunk by chunk took two
        // cluster barriers and S - 1 remote reads of 16 KB per 32 rows.)
        float* all_s = reinterpret_cast<float*>(smem);               // [NT][EPI_TILE_LD]
        cg::cluster_group cluster = cg::this_cluster();
        if (is_epi)
            for (int ch = 0; ch < n_chunks; ch++) drain(0, ch, all_s + (size_t)ch * TC_EPI_CHUNK * EPI_TILE_LD, EPI_TILE_LD);
        tc_fence_before();
        cluster.sync();
        // a rank tells its peers that it has read their shares as soon as it has, ahead of its own epilogue: the barrier at the end then
        // costs nothing (with the epilogue's loads and stores ahead of it a 4-row step of width 2048 took 236 us, now 230)
        auto read_all = [] { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); };
        const int ms = Mt * crank / S, me = Mt * (crank + 1) / S;
        if (!is_epi || ms >= me) read_all();
        if (is_epi) {
            pdl_wait();
            // values r .. r + 3 of activation row m: S <= 8, the ranks' shares in flight together, summed in rank order
            auto sum_of = [&](int m, int r) {
                float4 x[8];
#pragma unroll
                for (int c = 0; c < 8; c++)
                    if (c < S) x[c] = *reinterpret_cast<const float4*>(cluster.map_shared_rank(all_s, c) + (size_t)m * EPI_TILE_LD + r);
                float4 v = x[0];
#pragma unroll
                for (int c = 1; c < 8; c++)
                    if (c < S) { v.x += x[c].x; v.y += x[c].y; v.z += x[c].z; v.w += x[c].w; }
                return v;
            };
            if (a.vec) {
                if (ms < me) epilogue_vec<1>(a.epi, [&](int m, int r) { return sum_of(ms + m, r); }, rt * 128, a.d_real, me - ms, m0 + ms, warp - 2, TC_DEQ_WARPS, read_all);
            } else {
                for (int mb = ms; mb < me; mb += TC_EPI_CHUNK) {
                    const int mc = min(TC_EPI_CHUNK, me - mb);
                    for (int idx = tid - 64; idx < mc * 32; idx += TC_DEQ_WARPS * 32)
                        reinterpret_cast<float4*>(out_s)[idx] = sum_of(mb + (idx >> 5), (idx & 31) * 4);
                    asm volatile("bar.sync 1, 512;" ::: "memory");
                    if (mb + TC_EPI_CHUNK >= me) read_all();
                    epilogue_rows(a.epi, out_s, 128, 128, rt * 128, a.d_real, mc, m0 + mb, etid, eg, TC_GROUPS);
                    asm volatile("bar.sync 1, 512;" ::: "memory");      // out_s is rewritten by the next round
                }
            }
        }
        asm volatile("barrier.cluster.wait.acquire;" ::: "memory");     // nobody leaves while a peer may still read its share
    } else if (is_epi && a.vec) {
        // every MMA is done, so the rings are free: the whole of both tiles is drained there at once
        float* all_s = reinterpret_cast<float*>(smem);               // [P][NT][EPI_TILE_LD]
        for (int h = 0; h < P; h++)
            for (int ch = 0; ch < n_chunks; ch++) drain(h, ch, all_s + (size_t)(h * NT + ch * TC_EPI_CHUNK) * EPI_TILE_LD, EPI_TILE_LD);
        if (tid == 64) TC_DBG(4, 63);
        asm volatile("bar.sync 1, 512;" ::: "memory");
        pdl_wait();
        if (tid == 64) TC_DBG(5, 63);
        for (int h = 0; h < P; h++)
            epilogue_vec<2>(a.epi, EpiTile{all_s + (size_t)h * NT * EPI_TILE_LD, EPI_TILE_LD}, (rt + h) * 128, a.d_real, Mt, m0, warp - 2, TC_DEQ_WARPS, [] {});
        if (tid == 64) TC_DBG(6, 63);
    } else if (is_epi) {
        for (int h = 0; h < P; h++)
            for (int ch = 0; ch < n_chunks; ch++) {
                const int mc = min(TC_EPI_CHUNK, Mt - ch * TC_EPI_CHUNK);
                drain(h, ch, out_s, 128);
                asm volatile("bar.sync 1, 512;" ::: "memory");
                pdl_wait();
                epilogue_rows(a.epi, out_s, 128, 128, (rt + h) * 128, a.d_real, mc, m0 + ch * TC_EPI_CHUNK, etid, eg, TC_GROUPS);
                asm volatile("bar.sync 1, 512;" ::: "memory");
            }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, TC_TMEM_COLS);
    }
    epilogue_complete(a.epi, tid, a.n_epi_ctas, sflag);
    if (threadIdx.x == 0) TC_DBG(3, 63);
    trace_end(a.tr);
}

extern void dl_set_error(const char* fmt, ...);
extern "C" int dl_device_sm_count();
int dl_sm_count(int dev);

static long long* g_tc_dbg = nullptr;
static int g_tc_dbg_mode = 0;
extern "C" void dl_debug_set_tc_mode(int m) { g_tc_dbg_mode = m; }
extern "C" void dl_debug_set_tc_trace(long long* p) { g_tc_dbg = p; }

// Activation rows per tile.  Narrow batches: the next power of two from 16 on.  From 129 rows on: tiles of 128 rows, or of up to 256, as many as those need and
// of equal width (what a tile is short of is multiplied too), which unpack the weights half as often but go through one accumulator and one issuing warp.
// Whichever takes fewer waves of the SMs times clocks of one: a k-tile 520 clk at 128 rows, 950 or its MMAs' 4 per row above, start and epilogue 13000 +
// 30 a row (norm and feed-forward, us in 128s / wide, 4096 x 14336 at 300 rows 156 / 176, 400 rows - / 188 (two tiles of 256: 200), 520 rows - / 255
// (three: 275); 2048 x 8192 at 300 rows 65 / 62); wide ones only where they leave enough CTAs to fill the chip.
static int tc_tile(int d, int n, int M, int ncap, int ks, int n_sms) {
    const int row_tiles = (d + 127) / 128, KT = n / Q40T_TILE_K;
    int nt = (M <= 16) ? 16 : (M <= 32) ? 32 : (M <= 64) ? 64 : 128;
    if (M > 128) {
        const long long m_tiles = (M + 255) / 256, wide = ((M + m_tiles - 1) / m_tiles + 31) / 32 * 32;
        auto clocks = [&](long long tiles, long long item, long long width) {
            return (row_tiles * tiles * ks + n_sms - 1) / n_sms * (KT / ks * item + 13000 + 30 * width);
        };
        if (ncap >= m_tiles * wide && row_tiles * m_tiles * ks >= n_sms / 2 &&
            clocks(m_tiles, wide * 4 > 950 ? wide * 4 : 950, wide) < clocks((M + 127) / 128, 520, 128)) nt = (int)wide;
    }
    // narrow matrices (qkv / wo: 32-48 row tiles) are better off with narrower tiles that launch more
    // CTAs, even though every CTA then unpacks the weight tile again (the unpack overlaps the MMAs)
    while (nt > 32 && nt <= 128 && row_tiles * ((M + nt - 1) / nt) * ks < n_sms / 2) nt >>= 1;
    return nt;
}

// Ranks that share K: the count for which a launch takes least time, as fitted to 330 products of 512 to 8192 columns, 256 to 14336 inputs and 4 to 512 rows, each
// behind the norm that makes its activations (whole models of width 2048, 4096 and 8192 and a rank's part of them in 2, 4 and 8; cold weights; one behind
// the other alone they flatter few CTAs, whose successors start on the idle SMs): us a k-tile by the tile's rows, a start that grows with the CTAs, and
// the ranks' exchange, which grows with both.  Clusters have to find room at once: 36 of four ranks do not, nor 16 of eight.  Us with 1 / 2 / 4 / 8 ranks, the
// norm included: 4096 x 4096 at 8 rows 15.0 / 11.3 / 9.2, 64 rows 16.1 / 13.7 / 12.4; 4096 x 2048 at 8 rows 9.8 / 8.5 / 7.5, 64 rows 10.7 / 10.6 / 10.4;
// 1536 x 4096 at 8 rows 15.0 / 10.9 / 8.6 / 7.7; 1024 x 2048 at 8 rows 9.7 / 8.3 / 7.3 / 6.8; 4096 x 1024 at 8 rows 7.4 / 7.3 / 6.9; 2048 x 2048 at 8 rows 9.9 / 8.2 /
// 7.3 / 11.9; 2048 x 512 at 8 rows 6.5 / 6.8 / 7.0; 4096 x 1792 at 64 rows 10.1 / 10.2 / 10.3.
extern "C" int dl_gemm_q40_tc_split(int d, int n, int M, int n_sms) {
    const int row_tiles = (d + 127) / 128, KT = n / Q40T_TILE_K;
    int best = 1;
    double least = 0;
    for (int S = 1; S <= 8 && S <= KT; S *= 2) {
        const int nt = tc_tile(d, n, M, 1 << 30, S, n_sms), m_tiles = (M + nt - 1) / nt, ctas = row_tiles * m_tiles * S;
        if ((S == 4 && ctas > 128) || (S == 8 && ctas > 96) || (S > 1 && ctas > n_sms)) continue;
        auto ramp = [&](int from, int over) { return ctas <= from ? 0.0 : ctas >= from + over ? 1.0 : (double)(ctas - from) / over; };
        const double item = (nt <= 32 ? 0.41 : nt == 64 ? 0.42 : nt == 128 ? 0.465 : 0.00085 * (4 * nt > 950 ? 4 * nt : 950)) * (S == 1 ? 1.03 : 1.0);
        const double rows = (nt <= 32 ? 0.0 : nt == 64 ? 0.95 : 3.8 + 0.025 * (nt - 128)) * M / ((double)m_tiles * nt);
        const double start = S == 1 ? 1.8 + 1.45 * ramp(47, 90) : S == 2 ? 3.3 + (M <= 32 ? 0.0 : 1.45 * ramp(68, 50)) : S == 4 ? 3.1 + 1.8 * ramp(100, 50) : 2.75 + 0.8 * ramp(55, 32);
        const double us = (KT + S - 1) / S * item + rows + start;
        if (S == 1 || us < least) { best = S; least = us; }
    }
    return best;
}

// the tile that dl_gemm_q40_tc takes on this device, or that one of 148 SMs takes where there is none
extern "C" int dl_gemm_q40_tc_tile(int d, int n, int M, int ncap, int k_split) {
    const int n_sms = dl_device_sm_count();
    return tc_tile(d, n, M, ncap, k_split, n_sms > 0 ? n_sms : 148);
}

extern "C" int dl_gemm_q40_tc(const uint8_t* w_q40t, int d, int n, const uint8_t* xh, int ncap, int M, int k_split,
                              const DlEpilogue* epi, int pdl, void* stream) {
    if (n % Q40T_TILE_K != 0) { dl_set_error("dl_gemm_q40_tc: n=%d not a multiple of 128", n); return -1; }
    if (M < 1) { dl_set_error("dl_gemm_q40_tc: M < 1"); return -1; }
    if (epi->kind == DL_EPI_SILU_MUL && d % 64 != 0) { dl_set_error("dl_gemm_q40_tc: silu epilogue needs d%%64==0"); return -1; }
    TcArgs a;
    a.w = w_q40t; a.xh = xh;
    a.d_real = d;
    a.d_pad = (d + 127) / 128 * 128;
    a.KT = n / Q40T_TILE_K;
    a.ncap = ncap; a.M = M;
    int dev = 0;
    if (const cudaError_t e = cudaGetDevice(&dev)) { dl_set_error("dl_gemm_q40_tc: %s", cudaGetErrorString(e)); return -(int)e; }
    const int row_tiles = (d + 127) / 128, n_sms = dl_sm_count(dev);
    a.NT = tc_tile(d, n, M, ncap, (k_split == 2 || k_split == 4 || k_split == 8) ? k_split : 1, n_sms);
    if (ncap < (M + a.NT - 1) / a.NT * a.NT) { dl_set_error("dl_gemm_q40_tc: ncap=%d too small for M=%d (tile %d)", ncap, M, a.NT); return -1; }
    if (k_split != 1 && k_split != 2 && k_split != 4 && k_split != 8) { dl_set_error("dl_gemm_q40_tc: k_split must be 1,2,4,8"); return -1; }
    if (k_split > a.KT) k_split = 1;
    a.S = k_split;
    // stage counts by tile width: raw 9 KB, B NT*256 B, out 16 KB  (<= ~216 KB)
    if (a.NT <= 64) { a.NSA = 12; a.NSB = 4; }
    else if (a.NT == 128) { a.NSA = 8; a.NSB = 4; }
    else { a.NSA = 8; a.NSB = 2; }
    if (a.NSA < TC_GROUPS || a.NSA > 16) { dl_set_error("dl_gemm_q40_tc: bad NSA=%d", a.NSA); return -1; }
    // nacc must divide nstg: then successive phases of an A stage are consumed by the SAME issuing warp (and
    // written after a retire that is ordered behind the previous one), so a parity wait can never be lapped
    a.nacc = (a.NT <= 128) ? 2 : 1;                        // (also the two row tiles of a pair)
    a.nstg = (a.NT <= 64) ? 6 : 4;
    if (a.nacc * a.NT + a.nstg * TC_A_STAGE_COLS > TC_TMEM_COLS || a.nstg < TC_GROUPS || a.nstg > 8 || a.nstg % a.nacc != 0 || a.nacc < 1 || a.nacc > 2 || a.NSA % TC_GROUPS != 0) {
        dl_set_error("dl_gemm_q40_tc: bad TMEM plan nacc=%d nstg=%d NT=%d", a.nacc, a.nstg, a.NT);
        return -1;
    }
    a.nsb_log = (a.NSB == 8) ? 3 : (a.NSB == 4) ? 2 : 1;
    a.LA = (a.NSA % 4 == 0) ? 4 : (a.NSA % 3 == 0) ? 3 : (a.NSA % 2 == 0) ? 2 : 1;
    a.LB = (a.NSB % 4 == 0) ? 4 : (a.NSB % 3 == 0) ? 3 : (a.NSB % 2 == 0) ? 2 : 1;
    // more row tiles than SMs and one activation tile: two row tiles per CTA share the activations (at 128 rows those are 32 KB per k-tile
    // beside 9 KB of weights) and the second wave's start and end disappear
    a.pair = M <= a.NT && a.NT <= 128 && a.S == 1 && row_tiles % 2 == 0 && row_tiles > n_sms;
    const int cta_rows = row_tiles / (a.pair ? 2 : 1);
    a.n_epi_ctas = cta_rows * a.S * ((M + a.NT - 1) / a.NT);
    a.epi = *epi;
    a.vec = epilogue_vec_ok(*epi, d);
    a.tr = dl_trace_next(TR_TC);
    a.dbg = g_tc_dbg;
    if (dl_wait_limit("dl_gemm_q40_tc", &a.limit, dev) != 0) return -1;
    a.dbg_mode = g_tc_dbg_mode | (a.limit.ns == 0 ? 16 : 0);
    const size_t smem = (size_t)a.NSB * a.NT * 256 + (size_t)a.NSA * Q40T_TILE_BYTES +
                        (size_t)TC_EPI_CHUNK * 128 * 4 + (2 * 16 + 4 * 8) * 8 + 8 + 16;
    static SmemLimit given;
    if (const int rc = dl_smem_limit("gemm tc", gemm_q40_tc_kernel, smem, given, dev)) return rc;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(cta_rows * a.S), (unsigned)((M + a.NT - 1) / a.NT));
    cfg.blockDim = dim3(TC_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = (cudaStream_t)stream;
    cudaLaunchAttribute attrs[2];
    int na = 0;
    if (a.S > 1) {
        attrs[na].id = cudaLaunchAttributeClusterDimension;
        attrs[na].val.clusterDim.x = a.S;
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
    cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_q40_tc_kernel, a);
    if (e != cudaSuccess) { dl_set_error("gemm tc launch: %s", cudaGetErrorString(e)); return -(int)e; }
    return 0;
}
