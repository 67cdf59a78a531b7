// Two-SM form of the GEMM engine (included by qlmb_gemm.cu).
//
// A cluster of two CTAs on neighbouring SMs computes a 256 x 256 tile with
// tcgen05.mma.cta_group::2: each CTA stages its own 128 rows of A and its own
// 128 columns of B (expanding only that half of the weights), the leader CTA
// issues one M=256 instruction per 16-deep step that reads both halves, and each
// CTA's TMEM holds its 128 rows x 256 columns of the result.  Per SM and step the
// tensor core therefore reads half as much shared memory and the dequant warps
// expand half as many weights as in the one-SM form.
//
// Hand-shakes across the pair (all waits bounded, as everywhere in this file):
//   full[s]        leader   one barrier per stage collects everything the MMA needs: the
//                           byte counts of both CTAs' bulk tensor loads (the peer's loads
//                           name the leader's barrier, cta_group::2 form) and one arrival
//                           per dequant warp of either CTA (the peer's arrive remotely)
//   empty[s]       both     released by one tcgen05.commit that arrives in both CTAs
//   tmem_full[a]   both     committed the same way after a tile's last step
//   tmem_empty[a]  leader   8 local + 8 remote epilogue warps
//   full_c[j]      local    byte count of a stage's packed codes.  They are requested once empty[s] has completed, so
//                           a dequant warp that sees them knows that stage s of B is free too, and the multiplies that
//                           complete empty[s] came after the codes of stage s had been read: no further hand-shake.
//                           The warps of one group take every second stage, so j counts stages modulo an even number: a
//                           barrier then serves one group only, which waits for each of its phases.  (With one barrier
//                           per stage of an odd ring a group met every second phase, and a parity cannot tell a phase
//                           from the last but one: where the codes of the phase between were late, a warp expanded
//                           what the stage held before.)  A group's next phase of barrier j cannot complete before the
//                           group has seen this one: its copy waits for multiplies that need the group's stage.
// No bulk copy in this file has more than one destination CTA.
#pragma once

namespace qlmb {

constexpr int P_BN = 256;                 // accumulator columns of the pair tile
constexpr int P_A_STAGE = BM * BK * 2;    // per CTA: 128 rows
constexpr int P_B_STAGE = 128 * BK * 2;   // per CTA: 128 columns of B
constexpr int P_C_STAGE = 128 * BK / 2;   // per CTA: codes of those columns
// barriers for the codes of ns stages that dqg groups of warps take in turn: a multiple of both
constexpr int pair_code_bars(int ns, int dqg) { return ns % dqg ? ns * dqg : ns; }

__device__ __forceinline__ uint32_t cluster_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ void cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// address of the same shared-memory location in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t map_to_cta(uint32_t local, uint32_t rank)
{
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
    return r;
}
// (default semantics: a cluster-scope release here costs a full memory fence per call, which
// throttled the relay to one stage per microsecond)
__device__ __forceinline__ void mbar_arrive_remote(uint32_t cluster_addr)
{ asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory"); }
__device__ __forceinline__ uint32_t mbar_try_cluster(uint32_t bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok;
}
__device__ __forceinline__ bool mbar_wait_cluster(uint32_t bar, uint32_t parity, volatile int *abort_flag, int *errword, int site)
{
    for (uint32_t i = 0; i < WAIT_LIMIT; i++) {
        if (mbar_try_cluster(bar, parity)) return true;
        if ((i & 255u) == 255u && *abort_flag) return false;
    }
    if (!*abort_flag) {
        *abort_flag = 1;
        if (errword && atomicCAS(errword, 0, 201) == 0) { errword[1] = site; errword[2] = (int)blockIdx.x; errword[3] = (int)parity; }
    }
    return false;
}
// bulk tensor load into this CTA's shared memory whose byte count is reported to a barrier
// of either CTA of the pair (cluster address)
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap *map, uint32_t cluster_bar, int x, int y)
{
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                 ::"r"(dst), "l"(map), "r"(cluster_bar), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void tmem_alloc2(uint32_t smem_dst, uint32_t ncols)
{ asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(ncols) : "memory"); }
__device__ __forceinline__ void tmem_relinquish2()
{ asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_dealloc2(uint32_t taddr, uint32_t ncols)
{ asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory"); }
// completion of all MMAs issued so far -> one arrival on the barrier at this cluster address
__device__ __forceinline__ void tc_commit2(uint32_t cluster_bar)
{ asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(cluster_bar) : "memory"); }
// one commit that arrives on the barrier at this shared-memory offset in both CTAs of the pair
__device__ __forceinline__ void tc_commit2_both(uint32_t local_bar)
{
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(local_bar), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ void tc_mma2_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8, %9, %10, %11, %12}, p;\n\t}"
                 ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate),
                   "r"(0), "r"(0), "r"(0), "r"(0), "r"(0), "r"(0), "r"(0), "r"(0) : "memory");
}

// Pair tile: 256 rows starting at m0 (CTA r owns rows m0 + 128 r ...), 256 output columns
// starting at n_t * 256 (CTA r expands columns + 128 r); with the SwiGLU epilogue the pair
// tile is 128 gate + 128 up columns of the same 128 activation columns.
template <int SCHED, bool MATS = false>
__device__ __forceinline__ TileInfo decode_pair_tile(const GemmParams &p, int tile, int ntr)
{
    TileInfo t;
    t.mat = 0;
    if (SCHED == SCHED_DENSE) {
        t.m0 = (tile % p.tiles_m) * 256; t.n_t = tile / p.tiles_m; t.e = 0; t.ksteps = p.ksteps; t.row0 = 0;
        if (MATS && t.n_t >= p.mat_tile[0]) {            // the matrices' column tiles follow one another
            t.mat = t.n_t >= p.mat_tile[1] ? 2 : 1;
            t.n_t -= p.mat_tile[t.mat - 1];
        }
        t.halves = (t.m0 + BM < p.M) ? 2 : 1;
    } else if (SCHED == SCHED_ROWS) {
        // column tiles fastest: the pairs that run side by side share a row tile of A (which can be
        // far larger than L2 in total: 113 MB for dX) and differ in the weight slice (40 MB in total)
        int rt = tile / p.tiles_n;
        int info = p.tile_info[rt];
        t.m0 = (info & 0xFFFFF) * BM; t.e = (info >> 20) & 0x1FF; t.halves = ((info >> 30) & 1) + 1;
        t.n_t = tile % p.tiles_n; t.ksteps = p.ksteps; t.row0 = 0;
    } else {
        int per = p.tiles_m * p.tiles_n;
        t.e = tile / per;
        int r = tile % per;
        t.m0 = (r % p.tiles_m) * 256; t.n_t = r / p.tiles_m;
        // without a table: equal slices of ksteps stages (SCHED_SLICES: the same ones for each B matrix)
        if (SCHED == SCHED_SLICES) t.mat = t.e / p.slices;
        t.row0 = SCHED == SCHED_SLICES ? (t.e - t.mat * p.slices) * p.ksteps * BK : p.off ? p.off[t.e] : t.e * p.ksteps * BK;
        t.ksteps = SCHED != SCHED_SLICES && p.off ? (p.off[t.e + 1] - p.off[t.e]) / BK : p.ksteps;
        t.halves = (t.m0 + BM < p.M) ? 2 : 1;
    }
    return t;
}

template <int BMODE, int EPI, int SCHED, int DQG>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__((BMODE == B_DEQ_MN || BMODE == B_DEQ_K) ? 576 : 320, 1)
k_gemm_pair(const __grid_constant__ GemmParams p)
{
    constexpr bool DEQ = (BMODE == B_DEQ_MN || BMODE == B_DEQ_K);
    constexpr bool DUAL = (EPI == EPI_SWIGLU);           // CTA 0 expands W1 (gate), CTA 1 expands W3 (up)
    constexpr bool GROUPED = SCHED == SCHED_GROUPK || SCHED == SCHED_SLICES;
    constexpr bool MATS = (EPI == EPI_MATS);             // several matrices side by side, or segments of different lengths
    constexpr int NS = EPI == EPI_SWIGLU_BWD ? 4 : 5, NCB = pair_code_bars(NS, DQG);
    // Without weights to expand there is room for a second staging block per epilogue warp (a sixth operand stage brought
    // nothing): 16 KiB of fp32 per warp and tile no longer wait block by block for the store before
    constexpr bool TWO = !DEQ;
    constexpr int GW = DQ_WARPS / DQG;                   // dequant warps per stage group
    constexpr uint32_t IDESC = make_idesc(256, P_BN, BMODE == AB_TMA_MN ? 1 : 0, (BMODE == B_DEQ_MN || BMODE == AB_TMA_MN) ? 1 : 0);
    constexpr uint32_t TMEM_COLS = 2 * P_BN;
    constexpr uint32_t TX_BYTES = 2u * (P_A_STAGE + (DEQ ? 0 : P_B_STAGE));   // both CTAs' loads of a stage

    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t *sA = smem;
    uint8_t *sB = sA + NS * P_A_STAGE;
    uint8_t *sC = sB + NS * P_B_STAGE;
    uint8_t *sE = sC + (DEQ ? NS * P_C_STAGE : 0);
    static_assert((P_C_STAGE % 1024) == 0, "the epilogue staging blocks are bulk-tensor boxes with a 128-byte swizzle: 1 KiB alignment");
    uint64_t *bars = reinterpret_cast<uint64_t *>(sE + EPI_WARPS * epi_stage_bytes(EPI, TWO));
    uint64_t *full = bars, *empty = full + NS;
    uint64_t *full_c = empty + NS;
    uint64_t *tmem_full = full_c + NCB, *tmem_empty = tmem_full + 2, *spare = tmem_empty + 2;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(spare + 1);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();
    const bool leader = rank == 0;

    if (warp == 1 && elect_one()) {                       // the copies' descriptors, ahead of their first use
        for (int i = 0; i < (DUAL ? 1 : p.nseg); i++) prefetch_map(&p.a_map[i]);
        for (int i = 0; i < (DUAL ? 2 : MATS && p.nseg == 1 ? 1 : p.nseg); i++) prefetch_map(&p.w_map[i]);
    }
    if (threadIdx.x == 0) {
        for (int i = 0; i < NS; i++) { mbar_init(smem_u32(&full[i]), 1 + (DEQ ? 2 * GW : 0)); mbar_init(smem_u32(&empty[i]), 1); }
        for (int i = 0; i < NCB; i++) mbar_init(smem_u32(&full_c[i]), 1);
        for (int i = 0; i < 2; i++) { mbar_init(smem_u32(&tmem_full[i]), 1); mbar_init(smem_u32(&tmem_empty[i]), 2 * EPI_WARPS); }
        mbar_init(smem_u32(spare), 1);
        for (int i = 0; i < 2 * EPI_WARPS; i++) mbar_init(smem_u32(bars + 48 + i), 1);   // epilogue input rings
        *abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == 1) { tmem_alloc2(smem_u32(tmem_slot), TMEM_COLS); tmem_relinquish2(); }
    tc_fence_before();
    __syncthreads();
    cluster_sync();
    tc_fence_after();
    pdl_wait();                                          // barriers and TMEM above are this kernel's own; its operands come below
    pdl_trigger();
    const uint32_t tmem_base = *tmem_slot;

    const int npairs = gridDim.x >> 1, pair = blockIdx.x >> 1;
    const int ntr = (SCHED == SCHED_ROWS) ? *p.ntiles_dev : 0;
    const int total = (SCHED == SCHED_DENSE) ? p.tiles_m * p.tiles_n
                    : (SCHED == SCHED_ROWS) ? ntr * p.tiles_n : p.E * p.tiles_m * p.tiles_n;
    const int my_m = (int)rank * BM;                     // this CTA's row offset inside the pair tile
    const int my_n = (int)rank * 128;                    // and its column offset

    if (warp == 0) {
        // =============================== TMA producer (both CTAs) ===============================
        // One thread runs the whole loop.  A stage must be requested within its 512 cycles of multiplies; with the election,
        // the warp's reconvergence and the group scales (4-byte copies by all lanes) inside the loop it took 870.
        if (elect_one()) {
            Ring rs = {0, 0};
            int cb = 0;                                  // barrier of the stage's codes
            bool ok = true;
            const uint32_t full0 = map_to_cta(smem_u32(full), 0), my_full = smem_u32(full), empty0 = smem_u32(empty);
            const uint32_t full_c0 = smem_u32(full_c), sA0 = smem_u32(sA), sB0 = smem_u32(sB), sC0 = smem_u32(sC);
            for (int tile = pair; ok && tile < total; tile += npairs) {
                const TileInfo t = decode_pair_tile<SCHED, MATS>(p, tile, ntr);
                const int xa = t.m0 + my_m, xb = t.n_t * P_BN + my_n;
                for (int seg = 0; ok && seg < p.nseg; seg++) {
                    const CUtensorMap *am = &p.a_map[seg], *wm = &p.w_map[DUAL ? (int)rank : MATS || SCHED == SCHED_SLICES ? seg + t.mat : seg];
                    const int nks = MATS ? p.seg_steps[seg] : t.ksteps;
                    const int wrow = t.e * p.w_rows + (BMODE == B_DEQ_MN ? 0 : xb), wcol = DUAL ? t.n_t * 64 : xb / 2;
                    for (int ks = 0; ks < nks; ks++) {
                        ok = mbar_wait(empty0 + rs.idx * 8u, rs.phase ^ 1u, abort_flag, p.errword, 11);
                        if (!ok) break;
                        if (leader) mbar_expect_tx(my_full + rs.idx * 8u, TX_BYTES);
                        const uint32_t bar = full0 + rs.idx * 8u, dstA = sA0 + rs.idx * P_A_STAGE, dstB = sB0 + rs.idx * P_B_STAGE;
                        if (BMODE == AB_TMA_MN) {
                            const int row = t.row0 + ks * BK;
                            tma_load_2d_pair(dstA, am, bar, xa, row);
                            tma_load_2d_pair(dstA + 8192, am, bar, xa + 64, row);
                            tma_load_2d_pair(dstB, wm, bar, xb, row);
                            tma_load_2d_pair(dstB + 8192, wm, bar, xb + 64, row);
                        } else {
                            tma_load_2d_pair(dstA, am, bar, ks * BK, xa);
                            if (BMODE == B_TMA_K) tma_load_2d_pair(dstB, wm, bar, ks * BK, xb);
                        }
                        if (DEQ) {
                            const uint32_t cbar = full_c0 + cb * 8u, dstC = sC0 + rs.idx * P_C_STAGE;
                            mbar_expect_tx(cbar, P_C_STAGE);
                            if (BMODE == B_DEQ_MN) tma_load_2d(dstC, wm, cbar, wcol, wrow + ks * BK);
                            else tma_load_2d(dstC, wm, cbar, ks * (BK / 2), wrow);
                            if (++cb == NCB) cb = 0;
                        }
                        rs.next(NS);
                    }
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        if (leader) {
            // =============================== MMA issuer (leader CTA) ===============================
            Ring rs = {0, 0};
            bool ok = true;
            int it = 0;
            for (int tile = pair; ok && tile < total; tile += npairs, it++) {
                TileInfo t = decode_pair_tile<SCHED, MATS>(p, tile, ntr);
                const int acc = it & 1;
                ok = mbar_wait_cluster(smem_u32(&tmem_empty[acc]), (((uint32_t)it >> 1) & 1u) ^ 1u, abort_flag, p.errword, 13);
                if (!ok) break;
                tc_fence_after();
                const uint32_t tmem_d = tmem_base + (uint32_t)acc * P_BN;
                uint32_t accumulate = 0;
                for (int seg = 0; ok && seg < p.nseg; seg++) {
                    const int nks = MATS ? p.seg_steps[seg] : t.ksteps;
                    for (int ks = 0; ks < nks; ks++) {
                        ok = mbar_wait_cluster(smem_u32(&full[rs.idx]), rs.phase, abort_flag, p.errword, 14);
                        if (!ok) break;
                        tc_fence_after();
                        if (elect_one()) {
                            const uint32_t a0 = smem_u32(sA + rs.idx * P_A_STAGE);
                            const uint32_t b0 = smem_u32(sB + rs.idx * P_B_STAGE);
#pragma unroll
                            for (int k16 = 0; k16 < BK / 16; k16++) {
                                uint64_t ad = (BMODE == AB_TMA_MN) ? make_desc(a0 + k16 * 2048, 8192, 1024) : make_desc(a0 + k16 * 32, 16, 1024);
                                uint64_t bd = (BMODE == B_DEQ_MN || BMODE == AB_TMA_MN) ? make_desc(b0 + k16 * 2048, 8192, 1024)
                                                                                        : make_desc(b0 + k16 * 32, 16, 1024);
                                tc_mma2_bf16(tmem_d, ad, bd, IDESC, accumulate);
                                accumulate = 1;
                            }
                            tc_commit2_both(smem_u32(&empty[rs.idx]));
                        }
                        __syncwarp();
                        accumulate = 1;
                        rs.next(NS);
                    }
                }
                if (ok) {
                    if (elect_one()) tc_commit2_both(smem_u32(&tmem_full[acc]));
                    __syncwarp();
                }
            }
            if (*abort_flag) {
                if (elect_one()) tc_commit2(smem_u32(spare));
                __syncwarp();
                for (uint32_t i = 0; i < WAIT_LIMIT && !mbar_try(smem_u32(spare), 0); i++) {}
            }
        }
    } else if (warp < 2 + EPI_WARPS) {
        // =============================== epilogue (both CTAs) ===============================
        // warp (q, h): q = TMEM lane quarter (= warp id mod 4), h = which 128 of the 256 columns
        const int q = warp & 3, h = (warp - 2) >> 2;
        uint8_t *stage = sE + (warp - 2) * epi_stage_bytes(EPI, TWO);
        EpiCtx ec = {bars + 48 + 2 * (warp - 2), 0u};
        bool ok = true;
        int it = 0;
        for (int tile = pair; ok && tile < total; tile += npairs, it++) {
            TileInfo t = decode_pair_tile<SCHED, MATS>(p, tile, ntr);
            const int acc = it & 1;
            const long long row0 = (long long)t.m0 + my_m + q * 32;
            int valid = 32;
            if (SCHED == SCHED_ROWS) valid = ((int)rank < t.halves) ? 32 : 0;
            else { long long left = (long long)p.M - row0; valid = left < 0 ? 0 : (left < 32 ? (int)left : 32); }
            const long long rbase = GROUPED ? ((long long)t.e * p.M + row0) : row0;
            const long long col0 = (EPI == EPI_SWIGLU) ? (long long)t.n_t * 128 + h * 64 : (long long)t.n_t * P_BN + h * 128;
            ec.mat = t.mat;
            if (EPI != EPI_SWIGLU && col0 >= (MATS ? p.mat_N[t.mat] : p.N)) valid = 0;     // the half of a last tile that lies past the columns
            if (valid > 0) epilogue_prefetch<EPI>(p, stage, ec, lane, rbase, col0, valid);
            ok = mbar_wait_idle(smem_u32(&tmem_full[acc]), ((uint32_t)it >> 1) & 1u, abort_flag, p.errword, 19);
            if (!ok) break;
            tc_fence_after();
            if (valid > 0) {
                const bool have_acc = !GROUPED || t.ksteps > 0;
                const uint32_t tbase = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)acc * P_BN;
                if (EPI == EPI_SWIGLU)
                    epilogue_rows<EPI, TWO, BMODE == B_DEQ_MN>(p, stage, ec, lane, tbase + (uint32_t)h * 64, rbase, col0, valid, have_acc, 128);
                else
                    epilogue_rows<EPI, TWO, BMODE == B_DEQ_MN>(p, stage, ec, lane, tbase + (uint32_t)h * 128, rbase, col0, valid, have_acc, 0);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                const uint32_t te = smem_u32(&tmem_empty[acc]);
                if (leader) mbar_arrive(te); else mbar_arrive_remote(map_to_cta(te, 0));
            }
        }
        if (elect_one()) bulk_wait_all();                  // outstanding bulk stores of this warp
    } else if (DEQ) {
        // =============================== dequant warps (both CTAs) ===============================
        // The warps form DQG groups; group g expands the stages whose running index is g modulo
        // DQG, so one stage's chain (code read, expand, store, proxy fence, arrive) may take DQG
        // MMA stage times before it limits the tensor pipe.
        const int dw = warp - (2 + EPI_WARPS);
        constexpr int ITERS = (P_C_STAGE / 4) / (GW * 32);           // code words per lane and stage
        const int g = dw / GW, gw = dw % GW;
        // word i of a lane sits ROWS_I rows below word i-1; the swizzle term repeats every PER words
        constexpr int ROWS_I = (BMODE == B_DEQ_MN) ? 2 * GW : 4 * GW;
        constexpr int PER = ROWS_I >= 8 ? 1 : 8 / ROWS_I;
        const int r0 = (BMODE == B_DEQ_MN) ? gw * 2 + (lane >> 4) : gw * 4 + (lane >> 3);   // row of word 0
        const int c0 = (BMODE == B_DEQ_MN) ? (lane & 15) : (lane & 7);
        uint32_t dst0[PER];
#pragma unroll
        for (int i = 0; i < PER; i++) {
            const int r = r0 + i * ROWS_I;
            if (BMODE == B_DEQ_MN) dst0[i] = (uint32_t)((c0 / 8) * 8192 + (r >> 3) * 1024 + (r & 7) * 128 + (((c0 & 7) ^ (r & 7)) << 4));
            else dst0[i] = (uint32_t)((r >> 3) * 1024 + (r & 7) * 128 + ((c0 ^ (r & 7)) << 4));
        }
        constexpr uint32_t DST_STEP = (uint32_t)(PER * ROWS_I / 8) * 1024u;      // bytes per PER words
        Ring rb = {0, 0}, rc = {0, 0};                               // stage of B, barrier of its codes
        bool ok = true;
        const uint32_t full0 = map_to_cta(smem_u32(&full[0]), 0);    // the leader's stage barriers
        const uint32_t full_c0 = smem_u32(full_c);
        // A warp's words of a stage lie in 16 (codes [K][N]) or 32 (codes [N][K]) rows, each with one scale: lane m requests
        // that of row `srow` one stage ahead, and word i takes it from lane i * SPL + sub (one load and one conversion per
        // lane and stage; eight of each per lane took 500 cycles of the 1900 that a group spent on its stage).
        constexpr int SPL = BMODE == B_DEQ_MN ? 2 : 4;
        static_assert(ITERS * SPL <= 32, "one scale per lane");
        const int sub = BMODE == B_DEQ_MN ? lane >> 4 : lane >> 3;
        const int m = BMODE == B_DEQ_MN ? lane & 15 : lane, srow = gw * SPL + m % SPL + m / SPL * ROWS_I;
        int kc = 0;                                                  // running stage index of this CTA
        for (int tile = pair; ok && tile < total; tile += npairs) {
            TileInfo t = decode_pair_tile<SCHED, MATS>(p, tile, ntr);
            for (int seg = 0; ok && seg < p.nseg; seg++) {
                const int nks = MATS ? p.seg_steps[seg] : t.ksteps;
                const int gpr = MATS ? p.seg_gpr[seg + t.mat] : p.w_cols / 128, cols = MATS ? p.mat_N[t.mat] : p.N;
                int ks = (g - kc % DQG + DQG) % DQG;                 // first stage of this group in the segment
                for (int i = 0; i < ks && i < nks; i++) { rb.next(NS); rc.next(NCB); }
                // one stage on is BK rows (codes [K][N]) or half a group (codes [N][K]) on; a half that lies past the
                // columns expands zeros or the next matrix's codes with the scales of the half before it, for nobody
                const int xs = t.n_t * P_BN + my_n < cols ? t.n_t * P_BN + my_n : t.n_t * P_BN;
                const float *sp = p.scales[DUAL ? (int)rank : MATS ? seg + t.mat : seg]
                    + (BMODE == B_DEQ_MN ? (t.e * p.w_rows + srow) * gpr + (DUAL ? t.n_t : xs / 128)
                                         : (t.e * p.w_rows + xs + srow) * gpr);
                const int sstep = BMODE == B_DEQ_MN ? BK * gpr : 0;
                auto scale_at = [&](int k) { return sp[(BMODE == B_DEQ_MN ? k * sstep : (k * BK) / 128)]; };
                float cur = ks < nks ? scale_at(ks) : 0.0f;
                for (; ks < nks; ks += DQG) {
                    const float nxt = ks + DQG < nks ? scale_at(ks + DQG) : 0.0f;
                    const __nv_bfloat162 s2 = __float2bfloat162_rn(cur);
                    ok = mbar_wait(full_c0 + rc.idx * 8u, rc.phase, abort_flag, p.errword, 20);
                    if (!ok) break;
                    const uint32_t *cw = reinterpret_cast<const uint32_t *>(sC + rb.idx * P_C_STAGE) + gw * 32 + lane;
                    uint32_t w[ITERS];
#pragma unroll
                    for (int i = 0; i < ITERS; i++) w[i] = cw[i * GW * 32];
                    uint8_t *bdst = sB + rb.idx * P_B_STAGE;
#pragma unroll
                    for (int i = 0; i < ITERS; i++) {
                        const __nv_bfloat162 sw = __shfl_sync(0xffffffffu, s2, i * SPL + sub);
                        *reinterpret_cast<uint4 *>(bdst + dst0[i % PER] + (uint32_t)(i / PER) * DST_STEP) = (BMODE == B_DEQ_MN) ? dequant8_perm(w[i], sw) : dequant8(w[i], sw);
                    }
                    fence_proxy_async();
                    __syncwarp();
                    if (elect_one()) mbar_arrive_remote(full0 + (uint32_t)rb.idx * 8u);
                    const int adv = ks + DQG <= nks ? DQG : nks - ks;
                    rb.idx += adv;
                    if (rb.idx >= NS) rb.idx -= NS;
                    rc.idx += adv;
                    if (rc.idx >= NCB) { rc.idx -= NCB; rc.phase ^= 1u; }
                    cur = nxt;
                }
                kc += nks;
            }
        }
    }

    // =============================== teardown ===============================
    tc_fence_before();
    __syncthreads();
    cluster_sync();                                      // the peer's shared memory stays alive until the leader's MMAs are done
    if (warp == 1) { tc_fence_after(); tmem_dealloc2(tmem_base, TMEM_COLS); }
}

}  // namespace qlmb
