// Causal (optionally windowed) flash attention for sm_100a, head dimension 64, bf16 operands.
//
// Forward, one CTA per (sequence, head, tile of 128 queries), two CTAs per SM:
//
//   warp 0      TMA producer   Q tile once; K and V tiles of 128 keys through a three-stage ring
//   warp 1      MMA issuer     S = Q K^T (128 x 128 x 64) and O += P V (128 x 64 x 128) with tcgen05.mma; P is an
//                              operand in TMEM, O stays there (S: 128 columns, O: 64, P: 64)
//   warps 2-5   softmax        a thread per query row: the S row into 128 registers, running max / sum in the exp2
//                              domain, P as bf16 back into TMEM, O rescaled there when a row of the warp has a new maximum
//
// The scores of the next step are issued as soon as the softmax warps hold this step's in registers, so they are there when
// those come back for them, and PV runs beside the next step's maximum.
// What bounds it (8 x 1024 x 12 heads, clock trace): a step of a CTA takes 3.5 thousand cycles, 600 for the maximum, 300 for
// O, 1750 for the 128 exponentials of a thread with their conversions, the rest hand-shakes; special-function unit 33 % busy,
// issue slots 28 %: two softmax warps per scheduler do not cover their own latencies.  41 us; with two threads per row (an
// exchange of the row's maximum per step), P through shared memory and O folded in registers it took 54.  A quarter of the
// exponentials as polynomials on the multiply-add pipe: 42.3 instead of 41.2.
// Every mbarrier wait is bounded (qlmb_tc.cuh): a wait that runs out raises the CTA's abort flag, records its site in the
// device error word and all roles leave.
#include <cuda.h>
#include <cuda_bf16.h>
#include <math.h>
#include "qlmb_common.cuh"
#include "qlmb_gemm.cuh"
#include "qlmb_tc.cuh"

namespace qlmb {

constexpr int AT_BM = 128;                    // queries per CTA
constexpr int AT_BN = 128;                    // keys per step
constexpr int AT_HD = 64;
constexpr int AT_TILE = AT_BM * AT_HD * 2;    // bytes of a Q, K or V tile
constexpr int AT_FWD_NS = 3;                  // stages of the K / V ring
constexpr int AT_FWD_SMEM = AT_TILE + 2 * AT_FWD_NS * AT_TILE + 256;   // + barriers
constexpr int AT_FWD_THREADS = 192;

struct AttnFwdParams {
    alignas(64) CUtensorMap q_map, k_map, v_map;
    bf16 *O;
    float *lse;
    int B, T, H, KV, win, nqt;
    float scale_log2;                         // log2(e) / sqrt(hd)
    int *errword;
};

// Bounded wait of the attention kernels: a tile step takes microseconds, so a wait that has polled
// for about a second is broken; it raises the CTA's abort flag and records its site.  CTAs that
// start after an error was recorded leave at once (at_error_seen), so a broken pipeline ends the
// launch quickly instead of timing out CTA by CTA.
constexpr uint32_t AT_WAIT_LIMIT = 1u << 21;               // polls of the drain loops on the abort path
constexpr unsigned long long AT_WAIT_NS = 1000000000ull;    // one second of wall clock per wait
__device__ __forceinline__ unsigned long long at_now()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ uint32_t at_test(uint32_t bar, uint32_t parity)     // non-blocking probe
{
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok;
}
__device__ __forceinline__ bool at_wait(uint32_t bar, uint32_t parity, volatile int *abort_flag, int *errword, int site)
{
    if (mbar_try(bar, parity)) return true;
    unsigned long long t0 = 0;                 // read on the slow path only
    for (uint32_t i = 0;; i++) {
        if (at_test(bar, parity)) return true;
        if ((i & 1023u) == 1023u) {
            if (*abort_flag) return false;
            const unsigned long long now = at_now();
            if (!t0) t0 = now;
            else if (now - t0 > AT_WAIT_NS) break;
        }
    }
    if (!*abort_flag) {
        *abort_flag = 1;
        if (errword && atomicCAS(errword, 0, 200) == 0) { errword[1] = site; errword[2] = (int)blockIdx.x; errword[3] = (int)parity; }
    }
    return false;
}
__device__ __forceinline__ bool at_error_seen(const int *errword) { return errword && *reinterpret_cast<const volatile int *>(errword) != 0; }

// 2^x on the special-function unit (ex2.approx: 2 ulp, flushes denormal results to zero, -inf -> 0)
__device__ __forceinline__ float ex2(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
template <int M> struct AtMode { static constexpr int value = M; };     // which masks a tile needs

// 64 fp32 TMEM columns of this thread's lane, times mul, the rotation of pairs (j, j + 32) undone (cp, sp = the row's 32 cosines
// and sines) -> bf16 in global memory.  part 0: columns 0 .. 31 of the row, 1: columns 32 .. 63, 2: all of it.
__device__ __forceinline__ void attn_store_rot(bf16 *dst, uint32_t taddr, bool live, float mul, const float *cp, const float *sp, int part)
{
#pragma unroll
    for (int ch = 0; ch < 2; ch++) {
        uint32_t a[16], b[16];
        tmem_ld16(taddr + 16 * ch, a);
        tmem_ld16(taddr + 32 + 16 * ch, b);
        tmem_ld_wait();
        if (!live) continue;
#pragma unroll
        for (int u = 0; u < 2; u++) {
            uint32_t lo[4], hi[4];
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const int j = 8 * u + 4 * k;
                const float4 c = *reinterpret_cast<const float4 *>(cp + 16 * ch + j), s = *reinterpret_cast<const float4 *>(sp + 16 * ch + j);
                const float cc[4] = {c.x, c.y, c.z, c.w}, ss[4] = {s.x, s.y, s.z, s.w};
                float l4[4], h4[4];
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const float x = __uint_as_float(a[j + e]) * mul, y = __uint_as_float(b[j + e]) * mul;
                    l4[e] = x * cc[e] + y * ss[e];
                    h4[e] = y * cc[e] - x * ss[e];
                }
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    const __nv_bfloat162 l2 = __floats2bfloat162_rn(l4[2 * e], l4[2 * e + 1]), h2 = __floats2bfloat162_rn(h4[2 * e], h4[2 * e + 1]);
                    lo[2 * k + e] = *reinterpret_cast<const uint32_t *>(&l2); hi[2 * k + e] = *reinterpret_cast<const uint32_t *>(&h2);
                }
            }
            if (part != 1) *reinterpret_cast<uint4 *>(dst + 16 * ch + 8 * u) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
            if (part != 0) *reinterpret_cast<uint4 *>(dst + 32 + 16 * ch + 8 * u) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        }
    }
}
// two floats in one 64-bit register: sm_100's two-wide multiply-add and add
__device__ __forceinline__ uint64_t f2_packu(uint32_t a, uint32_t b) { uint64_t r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(a), "r"(b)); return r; }
__device__ __forceinline__ uint64_t f2_pack(float a, float b) { return f2_packu(__float_as_uint(a), __float_as_uint(b)); }
__device__ __forceinline__ void f2_unpack(uint64_t v, float &a, float &b)
{
    uint32_t x, y;
    asm("mov.b64 {%0, %1}, %2;" : "=r"(x), "=r"(y) : "l"(v));
    a = __uint_as_float(x); b = __uint_as_float(y);
}
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) { uint64_t r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r; }
__device__ __forceinline__ uint64_t f2_add(uint64_t a, uint64_t b) { uint64_t r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }

// 32 fp32 TMEM columns of this thread's lane, times mul -> 64 bytes of bf16 in global memory
// (tcgen05.ld is warp-collective: every lane runs it, only live lanes store)
__device__ __forceinline__ void attn_store_row32(bf16 *dst, uint32_t taddr, bool live, float mul)
{
    uint32_t v[32];
    tmem_ld32(taddr, v);
    tmem_ld_wait();
#pragma unroll
    for (int u = 0; u < 4; u++) {
        uint32_t w[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            __nv_bfloat162 h2 = __floats2bfloat162_rn(__uint_as_float(v[u * 8 + 2 * k]) * mul, __uint_as_float(v[u * 8 + 2 * k + 1]) * mul);
            w[k] = *reinterpret_cast<uint32_t *>(&h2);
        }
        if (live) *reinterpret_cast<uint4 *>(dst + u * 8) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}
__device__ __forceinline__ void attn_store_row64(bf16 *dst, uint32_t taddr, bool live, float mul)
{
    attn_store_row32(dst, taddr, live, mul);
    attn_store_row32(dst + 32, taddr + 32, live, mul);
}

__global__ void __launch_bounds__(AT_FWD_THREADS, 2) k_attn_fwd(const __grid_constant__ AttnFwdParams p)
{
    extern __shared__ __align__(1024) uint8_t at_smem[];
    constexpr int NS = AT_FWD_NS;
    uint8_t *sQ = at_smem, *sK = sQ + AT_TILE, *sV = sK + NS * AT_TILE;
    uint64_t *bars = reinterpret_cast<uint64_t *>(sV + NS * AT_TILE);
    uint64_t *q_full = bars, *s_full = bars + 1, *p_full = bars + 2, *o_full = bars + 3, *spare = bars + 4, *s_free = bars + 5,
             *kv_full = bars + 6, *kv_empty = kv_full + NS;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(kv_empty + NS);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (smem_u32(at_smem) & 1023u) {          // the swizzled tiles need a 1 KiB-aligned base
        if (threadIdx.x == 0 && p.errword && atomicCAS(p.errword, 0, 201) == 0) { p.errword[1] = 100; p.errword[2] = (int)blockIdx.x; }
        pdl_wait();
        return;
    }
    if (__syncthreads_or(threadIdx.x == 0 && at_error_seen(p.errword))) { pdl_wait(); return; }   // uniform over the CTA
    if (threadIdx.x == 0) {
        mbar_init(smem_u32(q_full), 1);
        for (int i = 0; i < NS; i++) { mbar_init(smem_u32(&kv_full[i]), 1); mbar_init(smem_u32(&kv_empty[i]), 1); }
        mbar_init(smem_u32(s_full), 1);
        mbar_init(smem_u32(s_free), 4);
        mbar_init(smem_u32(p_full), 4);
        mbar_init(smem_u32(o_full), 1);
        mbar_init(smem_u32(spare), 1);
        *abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == 1) { tmem_alloc(smem_u32(tmem_slot), 256); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_wait();                               // barriers and TMEM above are this kernel's own; its inputs come below
    pdl_trigger();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t tS = tmem_base, tO = tmem_base + 128, tP = tmem_base + 192;

    // heaviest query tiles first
    const int BH = p.B * p.H;
    const int qt = p.nqt - 1 - (int)blockIdx.x / BH, bh = (int)blockIdx.x % BH;
    const int b = bh / p.H, h = bh % p.H, kvh = h / (p.H / p.KV);
    const int q0 = qt * AT_BM;
    int kt_lo = 0;
    if (p.win > 0) { int lo = q0 - p.win + 1; kt_lo = lo > 0 ? lo / AT_BN : 0; }
    const int kt_hi = (q0 + AT_BM - 1 < p.T ? q0 + AT_BM - 1 : p.T - 1) / AT_BN;     // inclusive
    const int nt = kt_hi - kt_lo + 1;

    if (warp == 0) {
        // =============================== TMA producer ===============================
        bool ok = true;
        int issued = 0;
        if (elect_one()) {
            mbar_expect_tx(smem_u32(q_full), AT_TILE);
            tma_load_2d(smem_u32(sQ), &p.q_map, smem_u32(q_full), h * AT_HD, b * p.T + q0);
        }
        for (int t = 0; ok && t < nt; t++) {
            const int st = t % NS;
            ok = at_wait(smem_u32(&kv_empty[st]), ((uint32_t)(t / NS) & 1u) ^ 1u, abort_flag, p.errword, 101);
            if (!ok) break;
            if (elect_one()) {
                const uint32_t bar = smem_u32(&kv_full[st]);
                const int row = b * p.T + (kt_lo + t) * AT_BN;
                mbar_expect_tx(bar, 2 * AT_TILE);
                tma_load_2d(smem_u32(sK + st * AT_TILE), &p.k_map, bar, kvh * AT_HD, row);
                tma_load_2d(smem_u32(sV + st * AT_TILE), &p.v_map, bar, kvh * AT_HD, row);
            }
            __syncwarp();
            issued = t + 1;
        }
        if (*abort_flag) {
            // aborting: the copies this warp started must land before the CTA gives its shared memory back
            for (uint32_t i = 0; i < AT_WAIT_LIMIT && !mbar_try(smem_u32(q_full), 0); i++) {}
            for (int t = issued > NS ? issued - NS : 0; t < issued; t++)
                for (uint32_t i = 0; i < AT_WAIT_LIMIT && !mbar_try(smem_u32(&kv_full[t % NS]), (uint32_t)(t / NS) & 1u); i++) {}
        }
    } else if (warp == 1) {
        // =============================== MMA issuer ===============================
        constexpr uint32_t IDESC_S = make_idesc(AT_BM, AT_BN, 0, 0);
        constexpr uint32_t IDESC_PV = make_idesc(AT_BM, AT_HD, 0, 1);
        auto issue_s = [&](int st) {
            const uint32_t a0 = smem_u32(sQ), b0 = smem_u32(sK + st * AT_TILE);
#pragma unroll
            for (int k16 = 0; k16 < AT_HD / 16; k16++)
                tc_mma_bf16(tS, make_desc(a0 + k16 * 32, 16, 1024), make_desc(b0 + k16 * 32, 16, 1024), IDESC_S, k16 > 0);
            tc_commit(smem_u32(s_full));
        };
        bool ok = at_wait(smem_u32(q_full), 0, abort_flag, p.errword, 110);
        if (ok) ok = at_wait(smem_u32(&kv_full[0]), 0, abort_flag, p.errword, 111);
        if (ok) {
            tc_fence_after();
            if (elect_one()) issue_s(0);
            __syncwarp();
        }
        for (int t = 0; ok && t < nt; t++) {
            const int st = t % NS;
            // the next scores as soon as the softmax warps hold this step's in registers
            if (t + 1 < nt) {
                const int sn = (t + 1) % NS;
                ok = at_wait(smem_u32(&kv_full[sn]), (uint32_t)((t + 1) / NS) & 1u, abort_flag, p.errword, 113);
                if (ok) ok = at_wait(smem_u32(s_free), (uint32_t)t & 1u, abort_flag, p.errword, 114);
                if (!ok) break;
                tc_fence_after();
                if (elect_one()) issue_s(sn);
                __syncwarp();
            }
            ok = at_wait(smem_u32(p_full), (uint32_t)t & 1u, abort_flag, p.errword, 112);
            if (!ok) break;
            tc_fence_after();
            if (elect_one()) {
                const uint32_t b0 = smem_u32(sV + st * AT_TILE);
#pragma unroll
                for (int kk = 0; kk < AT_BN / 16; kk++)
                    tc_mma_bf16_ta(tO, tP + kk * 8, make_desc(b0 + kk * 2048, 8192, 1024), IDESC_PV, (t > 0 || kk > 0) ? 1u : 0u);
                tc_commit(smem_u32(o_full));
                tc_commit(smem_u32(&kv_empty[st]));
            }
            __syncwarp();
        }
        if (*abort_flag) {                    // let issued MMAs retire (bounded) before TMEM is released
            if (elect_one()) tc_commit(smem_u32(spare));
            __syncwarp();
            for (uint32_t i = 0; i < AT_WAIT_LIMIT && !mbar_try(smem_u32(spare), 0); i++) {}
        }
    } else {
        // =============================== softmax + output ===============================
        const int q = warp & 3, r = q * 32 + lane, i = q0 + r;
        const uint32_t lane_base = (uint32_t)(q * 32) << 16;
        const int iw = q0 + q * 32;                                     // the warp's first query
        const uint64_t scale2 = f2_pack(p.scale_log2, p.scale_log2);
        float m = -1e30f, l = 0.0f;
        bool ok = true;
        for (int t = 0; ok && t < nt; t++) {
            const int k0 = (kt_lo + t) * AT_BN;
            ok = at_wait(smem_u32(s_full), (uint32_t)t & 1u, abort_flag, p.errword, 120);
            if (!ok) break;
            tc_fence_after();
            uint32_t v[2][64];
#pragma unroll
            for (int c = 0; c < 4; c++) tmem_ld32(tS + lane_base + c * 32, &v[c >> 1][(c & 1) * 32]);
            tmem_ld_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(s_free));
            // Halves of 64 keys: all of them visible to the warp's 32 queries, some, or none.  A key that a query does not
            // see becomes -inf and gets the weight 0.
            auto none = [&](int c) { return k0 + c * 64 > iw + 31 || (p.win > 0 && k0 + c * 64 + 63 <= iw - p.win); };
            float mx = -1e30f;
#pragma unroll
            for (int c = 0; c < 2; c++) {
                const int kc = k0 + c * 64;
                if (none(c)) continue;
                if (kc + 63 > iw || (p.win > 0 && kc <= iw + 31 - p.win)) {
                    const int hi = i - kc, lo = p.win > 0 ? hi - p.win : -1;
#pragma unroll
                    for (int j = 0; j < 64; j++) v[c][j] = j <= hi && j > lo ? v[c][j] : 0xff800000u;
                }
                float mm[8];                            // eight chains: a step of one takes its instruction's latency
#pragma unroll
                for (int j = 0; j < 8; j++) mm[j] = __uint_as_float(v[c][j]);
#pragma unroll
                for (int j = 8; j < 56; j += 16)
#pragma unroll
                    for (int e = 0; e < 8; e++) mm[e] = fmaxf(fmaxf(mm[e], __uint_as_float(v[c][j + e])), __uint_as_float(v[c][j + 8 + e]));
#pragma unroll
                for (int e = 0; e < 8; e++) mm[e] = fmaxf(mm[e], __uint_as_float(v[c][56 + e]));
                mm[0] = fmaxf(fmaxf(mm[0], mm[1]), mm[2]); mm[3] = fmaxf(fmaxf(mm[3], mm[4]), mm[5]);
                mm[0] = fmaxf(fmaxf(mm[0], mm[3]), fmaxf(mm[6], mm[7]));
                mx = fmaxf(mx, mm[0] * p.scale_log2);
            }
            // the previous step's PV has read P and written O
            if (t > 0) {
                ok = at_wait(smem_u32(o_full), (uint32_t)(t - 1) & 1u, abort_flag, p.errword, 121);
                if (!ok) break;
                tc_fence_after();
            }
            // m is the running maximum.  Where no row of the warp has a new one O stays in TMEM as it is.  (Moving m only for
            // a growth of 2^8 saved 1.6 us of 42 at 8 x 1024 x 12 heads, but the largest weight is then no longer exactly 1
            // and the error against float64 grew from 2.03e-3 to 2.07e-3.)
            if (__any_sync(0xffffffffu, mx > m)) {
                const float mn = fmaxf(m, mx), corr = ex2(m - mn);
                m = mn;
                l *= corr;
                if (t > 0) {
#pragma unroll
                    for (int c = 0; c < 4; c++) {
                        uint32_t o[16];
                        tmem_ld16(tO + lane_base + c * 16, o);
                        tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 16; j++) o[j] = __float_as_uint(__uint_as_float(o[j]) * corr);
                        tmem_st16(tO + lane_base + c * 16, o);
                    }
                }
            }
            // P = exp2(s - m) as bf16 into the TMEM columns that PV reads as its A operand, partial row sums
            const uint64_t negm2 = f2_pack(-m, -m);
            uint64_t rs[2] = {f2_pack(0.0f, 0.0f), f2_pack(0.0f, 0.0f)};
#pragma unroll
            for (int c = 0; c < 2; c++) {
                uint32_t pk[32];
                if (none(c)) {
#pragma unroll
                    for (int j = 0; j < 32; j++) pk[j] = 0u;
                } else {
#pragma unroll
                    for (int j = 0; j < 32; j++) {
                        float x0, x1;
                        f2_unpack(f2_fma(f2_packu(v[c][2 * j], v[c][2 * j + 1]), scale2, negm2), x0, x1);
                        const float p0 = ex2(x0), p1 = ex2(x1);
                        rs[j & 1] = f2_add(rs[j & 1], f2_pack(p0, p1));
                        const __nv_bfloat162 h2 = __floats2bfloat162_rn(p0, p1);
                        pk[j] = *reinterpret_cast<const uint32_t *>(&h2);
                    }
                }
                tmem_st32(tP + lane_base + c * 32, pk);
            }
            float r0, r1;
            f2_unpack(f2_add(rs[0], rs[1]), r0, r1);
            l += r0 + r1;
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(p_full));
        }
        if (ok) ok = at_wait(smem_u32(o_full), (uint32_t)(nt - 1) & 1u, abort_flag, p.errword, 122);
        if (ok) {
            tc_fence_after();
            const float inv = 1.0f / l;
            attn_store_row64(p.O + ((size_t)b * p.T + i) * ((size_t)p.H * AT_HD) + (size_t)h * AT_HD, tO + lane_base, i < p.T, inv);
            if (i < p.T) p.lse[((size_t)b * p.H + h) * p.T + i] = (m + log2f(l)) * 0.6931471805599453f;
        }
        tc_fence_before();
    }
    __syncthreads();
    if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, 256); }
}


// ------------------------------------------------------------------ backward
// Two kernels, so that every output element has one writer and a fixed summation order:
//   k_attn_bwd_dkv  one CTA per (sequence, K/V head, tile of 128 keys), walks the heads of the
//                   group and the query tiles that see these keys; dK and dV accumulate in TMEM
//                   (few such CTAs: a cluster of them, one per head).
//   k_attn_bwd_dq   one CTA per (sequence, head, tile of 128 queries), walks the key tiles;
//                   dQ accumulates in TMEM.
// Both recompute the scores from Q, K and the saved log-sum-exp:  P = exp(S/sqrt(hd) - lse),
// dS = P * (dP - D) / sqrt(hd) with dP = dA V^T and D = rowsum(dA * O).  dq runs first: its threads make D of their own row, beside
// the first tiles' copies, and leave it for dkv (a launch of its own for D read dA and O once more: 6.5 us at 8 x 1024 x 12).
//
// The walked tiles are 64 wide, so that two CTAs fit an SM (98 and 97 KiB of shared memory, 256 TMEM columns each): the
// element-wise phase of one runs beside the MMAs of the other.
// dq: the scores of the next step are issued as soon as the element-wise warps hold this step's in registers, dS is an operand
// in TMEM.  dkv: P^T and dS^T are operands in TMEM too; its 256 columns leave them no room of their own, so they overwrite the
// scores they were made of, and the next scores follow the accumulating products.
// What bounds them (clock trace of 8 x 1024 x 12 heads): a step of a CTA takes 3.1 (dkv) and 1.6 (dq) thousand cycles, 1.3 and
// 0.9 of them element-wise work, in dkv 1.7 the products and their hand-shakes, which the other CTA fills in part.  128-wide
// tiles with one CTA per SM took 98 + 83 us; 64-wide tiles 85 + 67 us; with the MMAs issued behind elect.sync and masks only
// on the edge tiles 67 + 49; these 62 + 38.  (dkv with the scores ahead and P^T, dS^T through shared memory: 62 as well, its
// shared memory then busy 84 % of the time.)
//
//   warp 0      TMA producer   resident tiles once, the walked tiles through a four-stage ring (dkv:
//                              log-sum-exp and D of a tile's queries beside them)
//   warp 1      MMA issuer     scores and dP (two 128 x 64 x 64 MMAs into TMEM), then the accumulating
//                              products (dkv: two, dq: one) with P / dS in TMEM as the A operand
//   warps 2-9   element-wise   thread = one TMEM lane (a key for dkv, a query for dq) x 32 of the
//                              64 columns: P and dS as pairs of bf16 back into TMEM.  The factor
//                              1/sqrt(hd) of dS (a power of two) is applied to the finished sums.
constexpr int AT_BI = 64;                       // queries (dkv) or keys (dq) per step
constexpr int AT_ITILE = AT_BI * AT_HD * 2;     // bytes of a walked tile
constexpr int AT_BWD_THREADS = 320;             // TMA warp, MMA warp, 8 element-wise warps
constexpr int AT_DKV_NS = 4;                    // stages of the walked tiles in dkv
constexpr int AT_DKV_SMEM = 2 * AT_TILE + 2 * AT_DKV_NS * AT_ITILE + 2 * AT_DKV_NS * AT_BI * 4 + 256;
constexpr int AT_DQ_NS = 4;                     // stages of the walked tiles in dq
constexpr int AT_DQ_SMEM = 2 * AT_TILE + 2 * AT_DQ_NS * AT_ITILE + 2 * AT_BM * 4 + 256;    // + the halves of D, barriers

struct AttnBwdParams {
    alignas(64) CUtensorMap q_map, k_map, v_map, da_map;      // boxes of 128 rows (resident tiles)
    alignas(64) CUtensorMap q_imap, k_imap, v_imap, da_imap;  // boxes of 64 rows (walked tiles)
    const float *lse;
    float *drow;                                              // written by dq, read by dkv
    const bf16 *O, *dA;
    bf16 *dQ, *dK, *dV;                                       // dQ NULL: dq makes drow only
    const float *cosb, *sinb;                                 // not NULL: dQ and dK leave rotated back
    int B, T, H, KV, win, nqt;
    float scale, scale_log2;
    int *errword;
};

// What a cluster of CTAs needs to add its members' sums
__device__ __forceinline__ void at_cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t at_map(uint32_t local, uint32_t rank)
{
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(local), "r"(rank));
    return a;
}
__device__ __forceinline__ float4 at_ld4(uint32_t a)
{
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void at_st4(bf16 *dst, const float4 v)
{
    const __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
    *reinterpret_cast<uint2 *>(dst) = make_uint2(*reinterpret_cast<const uint32_t *>(&a), *reinterpret_cast<const uint32_t *>(&b));
}

// SPLIT: the query heads of a key/value head on a cluster of CTAs, one each, which add their sums at the end
template <bool SPLIT>
__global__ void __launch_bounds__(AT_BWD_THREADS, 2) k_attn_bwd_dkv(const __grid_constant__ AttnBwdParams p)
{
    extern __shared__ __align__(1024) uint8_t at_smem[];
    constexpr int NS = AT_DKV_NS;
    uint8_t *sK = at_smem, *sV = sK + AT_TILE, *sQ = sV + AT_TILE, *sA = sQ + NS * AT_ITILE;
    float *sL = reinterpret_cast<float *>(sA + NS * AT_ITILE), *sD = sL + NS * AT_BI;
    uint64_t *bars = reinterpret_cast<uint64_t *>(sD + NS * AT_BI);
    uint64_t *kv_full = bars, *s_full = bars + 1, *pds_full = bars + 2, *acc_done = bars + 3, *spare = bars + 4,
             *qd_full = bars + 5, *qd_empty = qd_full + NS;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(qd_empty + NS);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (smem_u32(at_smem) & 1023u) {
        if (threadIdx.x == 0 && p.errword && atomicCAS(p.errword, 0, 201) == 0) { p.errword[1] = 200; p.errword[2] = (int)blockIdx.x; }
        return;
    }
    // SPLIT: the CTAs of a cluster read one another's shared memory at the end, so none leaves early
    if (!SPLIT && __syncthreads_or(threadIdx.x == 0 && at_error_seen(p.errword))) { pdl_wait(); return; }   // uniform over the CTA
    if (threadIdx.x == 0) {
        mbar_init(smem_u32(kv_full), 1);
        for (int i = 0; i < NS; i++) { mbar_init(smem_u32(&qd_full[i]), 2); mbar_init(smem_u32(&qd_empty[i]), 1); }
        mbar_init(smem_u32(s_full), 1);
        mbar_init(smem_u32(pds_full), 8);
        mbar_init(smem_u32(acc_done), 1);
        mbar_init(smem_u32(spare), 1);
        *abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == 1) { tmem_alloc(smem_u32(tmem_slot), 256); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_wait();                               // barriers and TMEM above are this kernel's own; its inputs come below
    pdl_trigger();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t tS = tmem_base, tP = tmem_base + 64, tdV = tmem_base + 128, tdK = tmem_base + 192;

    // key tiles that see the most queries first
    const int BK_ = p.B * p.KV, grp = p.H / p.KV;
    const int rank = SPLIT ? (int)blockIdx.x % grp : 0, unit = SPLIT ? (int)blockIdx.x / grp : (int)blockIdx.x;
    const int kt = unit / BK_, bk = unit % BK_;
    const int b = bk / p.KV, kvh = bk % p.KV;
    const int k0 = kt * AT_BN;
    const int qt_lo = k0 / AT_BI;
    int qt_hi = (p.T - 1) / AT_BI;
    if (p.win > 0) { int hi = (k0 + AT_BN - 1 + p.win - 1) / AT_BI; if (hi < qt_hi) qt_hi = hi; }
    const int nq = qt_hi - qt_lo + 1, nit = SPLIT ? nq : nq * grp;     // iteration it: head kvh*grp + it / nq (SPLIT: + rank), query tile qt_lo + it % nq

    if (warp == 0) {
        // =============================== producer ===============================
        bool ok = true;
        int issued = 0;
        if (elect_one()) {
            mbar_expect_tx(smem_u32(kv_full), 2 * AT_TILE);
            tma_load_2d(smem_u32(sK), &p.k_map, smem_u32(kv_full), kvh * AT_HD, b * p.T + k0);
            tma_load_2d(smem_u32(sV), &p.v_map, smem_u32(kv_full), kvh * AT_HD, b * p.T + k0);
        }
        for (int it = 0; ok && it < nit; it++) {
            const int st = it % NS, h = kvh * grp + (SPLIT ? rank : it / nq), q0 = (qt_lo + it % nq) * AT_BI;
            ok = at_wait(smem_u32(&qd_empty[st]), ((uint32_t)(it / NS) & 1u) ^ 1u, abort_flag, p.errword, 201);
            if (!ok) break;
            const uint32_t bar = smem_u32(&qd_full[st]);
            if (elect_one()) {
                mbar_expect_tx(bar, 2 * AT_ITILE);
                tma_load_2d(smem_u32(sQ + st * AT_ITILE), &p.q_imap, bar, h * AT_HD, b * p.T + q0);
                tma_load_2d(smem_u32(sA + st * AT_ITILE), &p.da_imap, bar, h * AT_HD, b * p.T + q0);
            }
            // log-sum-exp (log2 domain) and D of the 64 queries; queries past the sequence get +huge, so P = 0
            const size_t rowb = ((size_t)b * p.H + h) * p.T;
#pragma unroll
            for (int k = 0; k < AT_BI / 32; k++) {
                const int c = lane + 32 * k, qi = q0 + c;
                sL[st * AT_BI + c] = qi < p.T ? p.lse[rowb + qi] * 1.4426950408889634f : 1e30f;
                sD[st * AT_BI + c] = qi < p.T ? p.drow[rowb + qi] : 0.0f;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(bar);
            issued = it + 1;
        }
        if (*abort_flag) {
            for (uint32_t i = 0; i < AT_WAIT_LIMIT && !mbar_try(smem_u32(kv_full), 0); i++) {}
            for (int it = issued > NS ? issued - NS : 0; it < issued; it++)
                for (uint32_t i = 0; i < AT_WAIT_LIMIT && !mbar_try(smem_u32(&qd_full[it % NS]), (uint32_t)(it / NS) & 1u); i++) {}
        }
    } else if (warp == 1) {
        // =============================== MMA issuer ===============================
        constexpr uint32_t IDESC_S = make_idesc(AT_BN, AT_BI, 0, 0);
        constexpr uint32_t IDESC_ACC = make_idesc(AT_BN, AT_HD, 0, 1);
        auto issue_scores = [&](int st) {      // S^T = K Q^T, dP^T = V dA^T
            const uint32_t k_ = smem_u32(sK), v_ = smem_u32(sV), q_ = smem_u32(sQ + st * AT_ITILE), a_ = smem_u32(sA + st * AT_ITILE);
#pragma unroll
            for (int k16 = 0; k16 < AT_HD / 16; k16++)
                tc_mma_bf16(tS, make_desc(k_ + k16 * 32, 16, 1024), make_desc(q_ + k16 * 32, 16, 1024), IDESC_S, k16 > 0);
#pragma unroll
            for (int k16 = 0; k16 < AT_HD / 16; k16++)
                tc_mma_bf16(tP, make_desc(v_ + k16 * 32, 16, 1024), make_desc(a_ + k16 * 32, 16, 1024), IDESC_S, k16 > 0);
            tc_commit(smem_u32(s_full));
        };
        bool ok = at_wait(smem_u32(kv_full), 0, abort_flag, p.errword, 210);
        if (ok) ok = at_wait(smem_u32(&qd_full[0]), 0, abort_flag, p.errword, 211);
        if (ok) {
            tc_fence_after();
            if (elect_one()) issue_scores(0);
            __syncwarp();
        }
        for (int it = 0; ok && it < nit; it++) {
            const int st = it % NS;
            ok = at_wait(smem_u32(pds_full), (uint32_t)it & 1u, abort_flag, p.errword, 212);
            if (!ok) break;
            tc_fence_after();
            if (elect_one()) {
                const uint32_t q_ = smem_u32(sQ + st * AT_ITILE), a_ = smem_u32(sA + st * AT_ITILE);
#pragma unroll
                for (int kk = 0; kk < AT_BI / 16; kk++)       // dV += P^T dA
                    tc_mma_bf16_ta(tdV, tS + (kk >> 1) * 32 + (kk & 1) * 8, make_desc(a_ + kk * 2048, 8192, 1024), IDESC_ACC, (it > 0 || kk > 0) ? 1u : 0u);
#pragma unroll
                for (int kk = 0; kk < AT_BI / 16; kk++)       // dK += dS^T Q
                    tc_mma_bf16_ta(tdK, tP + (kk >> 1) * 32 + (kk & 1) * 8, make_desc(q_ + kk * 2048, 8192, 1024), IDESC_ACC, (it > 0 || kk > 0) ? 1u : 0u);
                tc_commit(smem_u32(acc_done));
                tc_commit(smem_u32(&qd_empty[st]));
            }
            __syncwarp();
            // the next scores overwrite the columns that these products read: the multiplies of a CTA run in the order of
            // their issue, and acc_done makes sure of it
            if (it + 1 < nit) {
                const int sn = (it + 1) % NS;
                ok = at_wait(smem_u32(&qd_full[sn]), (uint32_t)((it + 1) / NS) & 1u, abort_flag, p.errword, 213);
                if (ok) ok = at_wait(smem_u32(acc_done), (uint32_t)it & 1u, abort_flag, p.errword, 214);
                if (!ok) break;
                tc_fence_after();
                if (elect_one()) issue_scores(sn);
                __syncwarp();
            }
        }
        if (*abort_flag) {
            if (elect_one()) tc_commit(smem_u32(spare));
            __syncwarp();
            for (uint32_t i = 0; i < AT_WAIT_LIMIT && !mbar_try(smem_u32(spare), 0); i++) {}
        }
    } else {
        // =============================== element-wise ===============================
        // warp = (TMEM lane quarter qr, 32-column chunk c of the 64)
        const int qr = warp & 3, c = (warp - 2) >> 2, r = qr * 32 + lane, key = k0 + r;
        const uint32_t lane_base = (uint32_t)(qr * 32) << 16;
        bool ok = true;
        for (int it = 0; ok && it < nit; it++) {
            const int st = it % NS, q0 = (qt_lo + it % nq) * AT_BI;
            const bool masked = (q0 < k0 + AT_BN - 1) || p.win > 0;
            ok = at_wait(smem_u32(&qd_full[st]), (uint32_t)(it / NS) & 1u, abort_flag, p.errword, 220);      // lse / D in shared memory
            if (ok) ok = at_wait(smem_u32(s_full), (uint32_t)it & 1u, abort_flag, p.errword, 221);
            if (!ok) break;
            tc_fence_after();
            const float *L2 = sL + st * AT_BI + c * 32, *Dq = sD + st * AT_BI + c * 32;
            uint32_t sv[32], dv[32];                 // both TMEM loads of the step in flight: one round trip
            tmem_ld32(tS + lane_base + c * 32, sv);
            tmem_ld32(tP + lane_base + c * 32, dv);
            tmem_ld_wait();
            {
                uint32_t pp[16], ds[16];
                // MODE 0: every query sees the key; 1: causal edge, queries from j = lo on; 2: window, j below hi as well
                auto compute = [&](auto mode, int lo, int hi) {
                    constexpr int MODE = decltype(mode)::value;
#pragma unroll
                    for (int j = 0; j < 32; j += 4) {
                        const float4 l4 = *reinterpret_cast<const float4 *>(L2 + j), d4 = *reinterpret_cast<const float4 *>(Dq + j);
                        const float ll[4] = {l4.x, l4.y, l4.z, l4.w}, dd[4] = {d4.x, d4.y, d4.z, d4.w};
                        float pv[4], dsv[4];
#pragma unroll
                        for (int e = 0; e < 4; e++) {
                            float pe = ex2(__uint_as_float(sv[j + e]) * p.scale_log2 - ll[e]);
                            if (MODE == 1) pe = j + e >= lo ? pe : 0.0f;
                            if (MODE == 2) pe = j + e >= lo && j + e < hi ? pe : 0.0f;
                            pv[e] = pe;
                            dsv[e] = pe * (__uint_as_float(dv[j + e]) - dd[e]);
                        }
#pragma unroll
                        for (int e = 0; e < 4; e += 2) {
                            __nv_bfloat162 h2 = __floats2bfloat162_rn(pv[e], pv[e + 1]);
                            pp[(j + e) >> 1] = *reinterpret_cast<uint32_t *>(&h2);
                            h2 = __floats2bfloat162_rn(dsv[e], dsv[e + 1]);
                            ds[(j + e) >> 1] = *reinterpret_cast<uint32_t *>(&h2);
                        }
                    }
                };
                const int lo = key - q0 - c * 32;         // query q0 + 32 c + j sees the key from j = lo on
                if (!masked) compute(AtMode<0>(), 0, 0);
                else if (p.win <= 0) compute(AtMode<1>(), lo, 0);
                else compute(AtMode<2>(), lo, lo + p.win);
                // P^T and dS^T over the thread's own score columns: 16 words of 64 columns' bf16 pairs each
                tmem_st16(tS + lane_base + c * 32, pp);
                tmem_st16(tP + lane_base + c * 32, ds);
                tmem_st_wait();
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(pds_full));
        }
        if (ok) ok = at_wait(smem_u32(acc_done), (uint32_t)(nit - 1) & 1u, abort_flag, p.errword, 223);
        if (ok) {
            tc_fence_after();
            if (SPLIT) {                             // this head's sums as fp32 over the tiles, dV | dK, row r: unit u at u ^ (r & 7)
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    uint32_t v[32];
                    tmem_ld32((c ? tdK : tdV) + lane_base + k * 32, v);
                    tmem_ld_wait();
#pragma unroll
                    for (int u = 0; u < 8; u++)
                        *reinterpret_cast<uint4 *>(at_smem + r * 512 + (((c * 16 + k * 8 + u) ^ (r & 7)) << 4)) = make_uint4(v[4 * u], v[4 * u + 1], v[4 * u + 2], v[4 * u + 3]);
                }
            } else {
                // chunk 0: the dV row; chunk 1: the dK row
                bf16 *dst = (c ? p.dK : p.dV) + ((size_t)b * p.T + key) * ((size_t)p.KV * AT_HD) + (size_t)kvh * AT_HD;
                if (c && p.cosb) {
                    const size_t pos = (size_t)(key < p.T ? key : 0) * 32;
                    attn_store_rot(dst, tdK + lane_base, key < p.T, p.scale, p.cosb + pos, p.sinb + pos, 2);
                } else {
                    attn_store_row64(dst, (c ? tdK : tdV) + lane_base, key < p.T, c ? p.scale : 1.0f);
                }
            }
        }
        tc_fence_before();
    }
    __syncthreads();
    if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, 256); }
    if (SPLIT) {
        // every CTA adds 128 / grp of the rows over the group's heads, in the heads' order.  A row is 24 items: four columns of dV,
        // or four of dK with the four that the rotation pairs them with.
        at_cluster_sync();
        const int rows = AT_BN / grp;
        const uint32_t base = smem_u32(at_smem);
        for (int x = threadIdx.x; x < rows * 24; x += AT_BWD_THREADS) {
            const int r = rank * rows + x / 24, u = x % 24, key = k0 + r;
            const bool isk = u >= 16;
            float4 s0 = make_float4(0.f, 0.f, 0.f, 0.f), s1 = s0;
            for (int g = 0; g < grp; g++) {
                const uint32_t peer = at_map(base, (uint32_t)g) + r * 512;
                const float4 v = at_ld4(peer + ((u ^ (r & 7)) << 4));
                s0.x += v.x; s0.y += v.y; s0.z += v.z; s0.w += v.w;
                if (isk) {
                    const float4 w = at_ld4(peer + (((u + 8) ^ (r & 7)) << 4));
                    s1.x += w.x; s1.y += w.y; s1.z += w.z; s1.w += w.w;
                }
            }
            if (key >= p.T) continue;
            const size_t at = ((size_t)b * p.T + key) * ((size_t)p.KV * AT_HD) + (size_t)kvh * AT_HD;
            if (!isk) { at_st4(p.dV + at + 4 * u, s0); continue; }
            const int j = 4 * (u - 16);
            s0.x *= p.scale; s0.y *= p.scale; s0.z *= p.scale; s0.w *= p.scale;
            s1.x *= p.scale; s1.y *= p.scale; s1.z *= p.scale; s1.w *= p.scale;
            if (p.cosb) {
                const float4 cs = *reinterpret_cast<const float4 *>(p.cosb + (size_t)key * 32 + j), sn = *reinterpret_cast<const float4 *>(p.sinb + (size_t)key * 32 + j);
                const float4 lo = make_float4(s0.x * cs.x + s1.x * sn.x, s0.y * cs.y + s1.y * sn.y, s0.z * cs.z + s1.z * sn.z, s0.w * cs.w + s1.w * sn.w);
                s1 = make_float4(s1.x * cs.x - s0.x * sn.x, s1.y * cs.y - s0.y * sn.y, s1.z * cs.z - s0.z * sn.z, s1.w * cs.w - s0.w * sn.w);
                s0 = lo;
            }
            at_st4(p.dK + at + j, s0);
            at_st4(p.dK + at + 32 + j, s1);
        }
        at_cluster_sync();                                    // the others' shared memory stays until everyone has read it
    }
}

__global__ void __launch_bounds__(AT_BWD_THREADS, 2) k_attn_bwd_dq(const __grid_constant__ AttnBwdParams p)
{
    extern __shared__ __align__(1024) uint8_t at_smem[];
    constexpr int NS = AT_DQ_NS;
    uint8_t *sQ = at_smem, *sA = sQ + AT_TILE, *sK = sA + AT_TILE, *sV = sK + NS * AT_ITILE;
    uint64_t *bars = reinterpret_cast<uint64_t *>(sV + NS * AT_ITILE + 2 * AT_BM * 4);
    float *sD = reinterpret_cast<float *>(sV + NS * AT_ITILE);
    uint64_t *qa_full = bars, *s_full = bars + 1, *ds_full = bars + 2, *acc_done = bars + 3, *spare = bars + 4, *s_free = bars + 5,
             *kv_full = bars + 6, *kv_empty = kv_full + NS;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(kv_empty + NS);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (smem_u32(at_smem) & 1023u) {
        if (threadIdx.x == 0 && p.errword && atomicCAS(p.errword, 0, 201) == 0) { p.errword[1] = 300; p.errword[2] = (int)blockIdx.x; }
        return;
    }
    if (__syncthreads_or(threadIdx.x == 0 && at_error_seen(p.errword))) { pdl_wait(); return; }   // uniform over the CTA
    if (threadIdx.x == 0) {
        mbar_init(smem_u32(qa_full), 1);
        for (int i = 0; i < NS; i++) { mbar_init(smem_u32(&kv_full[i]), 1); mbar_init(smem_u32(&kv_empty[i]), 1); }
        mbar_init(smem_u32(s_full), 1);
        mbar_init(smem_u32(s_free), 8);
        mbar_init(smem_u32(ds_full), 8);
        mbar_init(smem_u32(acc_done), 1);
        mbar_init(smem_u32(spare), 1);
        *abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == 1) { tmem_alloc(smem_u32(tmem_slot), 256); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_wait();                               // barriers and TMEM above are this kernel's own; its inputs come below
    pdl_trigger();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t tS = tmem_base, tP = tmem_base + 64, tdQ = tmem_base + 128, tdS = tmem_base + 192;

    const int BH = p.B * p.H;
    const int qt = p.nqt - 1 - (int)blockIdx.x / BH, bh = (int)blockIdx.x % BH;
    const int b = bh / p.H, h = bh % p.H, kvh = h / (p.H / p.KV);
    const int q0 = qt * AT_BM;
    int kt_lo = 0;
    if (p.win > 0) { int lo = q0 - p.win + 1; kt_lo = lo > 0 ? lo / AT_BI : 0; }
    const int kt_hi = (q0 + AT_BM - 1 < p.T ? q0 + AT_BM - 1 : p.T - 1) / AT_BI;
    const int nt = kt_hi - kt_lo + 1;

    if (warp == 0) {
        bool ok = true;
        int issued = 0;
        if (elect_one()) {
            mbar_expect_tx(smem_u32(qa_full), 2 * AT_TILE);
            tma_load_2d(smem_u32(sQ), &p.q_map, smem_u32(qa_full), h * AT_HD, b * p.T + q0);
            tma_load_2d(smem_u32(sA), &p.da_map, smem_u32(qa_full), h * AT_HD, b * p.T + q0);
        }
        for (int t = 0; ok && t < nt; t++) {
            const int st = t % NS;
            ok = at_wait(smem_u32(&kv_empty[st]), ((uint32_t)(t / NS) & 1u) ^ 1u, abort_flag, p.errword, 301);
            if (!ok) break;
            if (elect_one()) {
                const uint32_t bar = smem_u32(&kv_full[st]);
                const int row = b * p.T + (kt_lo + t) * AT_BI;
                mbar_expect_tx(bar, 2 * AT_ITILE);
                tma_load_2d(smem_u32(sK + st * AT_ITILE), &p.k_imap, bar, kvh * AT_HD, row);
                tma_load_2d(smem_u32(sV + st * AT_ITILE), &p.v_imap, bar, kvh * AT_HD, row);
            }
            __syncwarp();
            issued = t + 1;
        }
        if (*abort_flag) {
            for (uint32_t i = 0; i < AT_WAIT_LIMIT && !mbar_try(smem_u32(qa_full), 0); i++) {}
            for (int t = issued > NS ? issued - NS : 0; t < issued; t++)
                for (uint32_t i = 0; i < AT_WAIT_LIMIT && !mbar_try(smem_u32(&kv_full[t % NS]), (uint32_t)(t / NS) & 1u); i++) {}
        }
    } else if (warp == 1) {
        constexpr uint32_t IDESC_S = make_idesc(AT_BM, AT_BI, 0, 0);
        constexpr uint32_t IDESC_ACC = make_idesc(AT_BM, AT_HD, 0, 1);
        auto issue_scores = [&](int st) {      // S = Q K^T, dP = dA V^T
            const uint32_t q_ = smem_u32(sQ), a_ = smem_u32(sA), k_ = smem_u32(sK + st * AT_ITILE), v_ = smem_u32(sV + st * AT_ITILE);
#pragma unroll
            for (int k16 = 0; k16 < AT_HD / 16; k16++)
                tc_mma_bf16(tS, make_desc(q_ + k16 * 32, 16, 1024), make_desc(k_ + k16 * 32, 16, 1024), IDESC_S, k16 > 0);
#pragma unroll
            for (int k16 = 0; k16 < AT_HD / 16; k16++)
                tc_mma_bf16(tP, make_desc(a_ + k16 * 32, 16, 1024), make_desc(v_ + k16 * 32, 16, 1024), IDESC_S, k16 > 0);
            tc_commit(smem_u32(s_full));
        };
        bool ok = at_wait(smem_u32(qa_full), 0, abort_flag, p.errword, 310);
        if (ok) ok = at_wait(smem_u32(&kv_full[0]), 0, abort_flag, p.errword, 311);
        if (ok) {
            tc_fence_after();
            if (elect_one()) issue_scores(0);
            __syncwarp();
        }
        for (int t = 0; ok && t < nt; t++) {
            const int st = t % NS;
            if (t + 1 < nt) {                                 // the next scores as soon as the element-wise warps hold this step's
                const int sn = (t + 1) % NS;
                ok = at_wait(smem_u32(&kv_full[sn]), (uint32_t)((t + 1) / NS) & 1u, abort_flag, p.errword, 313);
                if (ok) ok = at_wait(smem_u32(s_free), (uint32_t)t & 1u, abort_flag, p.errword, 314);
                if (!ok) break;
                tc_fence_after();
                if (elect_one()) issue_scores(sn);
                __syncwarp();
            }
            ok = at_wait(smem_u32(ds_full), (uint32_t)t & 1u, abort_flag, p.errword, 312);
            if (!ok) break;
            tc_fence_after();
            if (elect_one()) {
                const uint32_t k_ = smem_u32(sK + st * AT_ITILE);
#pragma unroll
                for (int kk = 0; kk < AT_BI / 16; kk++)       // dQ += dS K
                    tc_mma_bf16_ta(tdQ, tdS + kk * 8, make_desc(k_ + kk * 2048, 8192, 1024), IDESC_ACC, (t > 0 || kk > 0) ? 1u : 0u);
                tc_commit(smem_u32(acc_done));
                tc_commit(smem_u32(&kv_empty[st]));
            }
            __syncwarp();
        }
        if (*abort_flag) {
            if (elect_one()) tc_commit(smem_u32(spare));
            __syncwarp();
            for (uint32_t i = 0; i < AT_WAIT_LIMIT && !mbar_try(smem_u32(spare), 0); i++) {}
        }
    } else {
        const int qr = warp & 3, c = (warp - 2) >> 2, r = qr * 32 + lane, i = q0 + r;
        const uint32_t lane_base = (uint32_t)(qr * 32) << 16;
        const size_t rowb = ((size_t)b * p.H + h) * p.T;
        const float L2 = i < p.T ? p.lse[rowb + i] * 1.4426950408889634f : 1e30f;
        float Dq = 0.0f;
        {                                            // this thread's half of D, then both halves in order
            if (i < p.T) {
                const size_t at = ((size_t)b * p.T + i) * ((size_t)p.H * AT_HD) + (size_t)h * AT_HD + c * 32;
                uint4 x[4], y[4];
#pragma unroll
                for (int u = 0; u < 4; u++) { x[u] = reinterpret_cast<const uint4 *>(p.dA + at)[u]; y[u] = reinterpret_cast<const uint4 *>(p.O + at)[u]; }
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const uint32_t xw[4] = {x[u].x, x[u].y, x[u].z, x[u].w}, yw[4] = {y[u].x, y[u].y, y[u].z, y[u].w};
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        Dq += __uint_as_float(xw[k] << 16) * __uint_as_float(yw[k] << 16);
                        Dq += __uint_as_float(xw[k] & 0xffff0000u) * __uint_as_float(yw[k] & 0xffff0000u);
                    }
                }
            }
            sD[c * AT_BM + r] = Dq;
            asm volatile("bar.sync 1, 256;" ::: "memory");
            Dq = sD[r] + sD[AT_BM + r];
            if (c == 0 && i < p.T) p.drow[rowb + i] = Dq;
        }
        bool ok = true;
        for (int t = 0; ok && t < nt; t++) {
            const int k0 = (kt_lo + t) * AT_BI;
            const bool masked = (k0 + AT_BI - 1 > q0) || p.win > 0 || (k0 + AT_BI > p.T);
            ok = at_wait(smem_u32(s_full), (uint32_t)t & 1u, abort_flag, p.errword, 321);
            if (!ok) break;
            tc_fence_after();
            uint32_t sv[32], dv[32];                 // both TMEM loads of the step in flight: one round trip
            tmem_ld32(tS + lane_base + c * 32, sv);
            tmem_ld32(tP + lane_base + c * 32, dv);
            tmem_ld_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(s_free));       // the next scores may overwrite these
            {
                uint32_t ds[16];
                auto compute = [&](auto mode, int lo, int hi) {       // keys lo < j <= hi of the thread's 32 (see k_attn_bwd_dkv)
                    constexpr int MODE = decltype(mode)::value;
#pragma unroll
                    for (int j = 0; j < 32; j += 2) {
                        float dsv[2];
#pragma unroll
                        for (int e = 0; e < 2; e++) {
                            float pe = ex2(__uint_as_float(sv[j + e]) * p.scale_log2 - L2);
                            if (MODE == 1) pe = j + e <= hi ? pe : 0.0f;
                            if (MODE == 2) pe = j + e <= hi && j + e > lo ? pe : 0.0f;
                            dsv[e] = pe * (__uint_as_float(dv[j + e]) - Dq);
                        }
                        __nv_bfloat162 h2 = __floats2bfloat162_rn(dsv[0], dsv[1]);
                        ds[j >> 1] = *reinterpret_cast<uint32_t *>(&h2);
                    }
                };
                const int base = k0 + c * 32, hi = (i < p.T ? i : p.T - 1) - base;
                if (!masked) compute(AtMode<0>(), 0, 0);
                else if (p.win <= 0) compute(AtMode<1>(), 0, hi);
                else compute(AtMode<2>(), i - p.win - base, hi);
                if (t > 0) ok = at_wait(smem_u32(acc_done), (uint32_t)(t - 1) & 1u, abort_flag, p.errword, 322);   // dS columns free again
                if (ok) { tc_fence_after(); tmem_st16(tdS + lane_base + c * 16, ds); tmem_st_wait(); }
            }
            if (!ok) break;
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(ds_full));
        }
        if (ok) ok = at_wait(smem_u32(acc_done), (uint32_t)(nt - 1) & 1u, abort_flag, p.errword, 323);
        if (ok && p.dQ) {
            tc_fence_after();
            // each of the row's two threads stores half of it
            bf16 *dst = p.dQ + ((size_t)b * p.T + i) * ((size_t)p.H * AT_HD) + (size_t)h * AT_HD;
            if (p.cosb) {
                const size_t pos = (size_t)(i < p.T ? i : 0) * 32;
                attn_store_rot(dst, tdQ + lane_base, i < p.T, p.scale, p.cosb + pos, p.sinb + pos, c);
            } else {
                attn_store_row32(dst + c * 32, tdQ + lane_base + c * 32, i < p.T, p.scale);
            }
        }
        tc_fence_before();
    }
    __syncthreads();
    if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, 256); }
}

}  // namespace qlmb

using namespace qlmb;

extern "C" int qlmb_attn_fwd(void *O, float *lse, const void *Q, const void *K, const void *V, int B, int T, int H,
                             int KV, int hd, int win, void *stream)
{
    QLMB_REQUIRE(O && lse && Q && K && V, "qlmb_attn_fwd: NULL argument");
    QLMB_REQUIRE(hd == AT_HD, "qlmb_attn_fwd: head dimension %d (only 64 is built)", hd);
    QLMB_REQUIRE(B > 0 && T > 0 && H > 0 && KV > 0 && H % KV == 0, "qlmb_attn_fwd: bad shape B %d T %d H %d KV %d", B, T, H, KV);
    AttnFwdParams p;
    memset(&p, 0, sizeof p);
    const unsigned long long rows = (unsigned long long)B * T;
    int rc = make_map(&p.q_map, Q, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (unsigned long long)H * hd, rows, (unsigned long long)H * hd * 2, AT_HD, AT_BM, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
    rc = make_map(&p.k_map, K, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (unsigned long long)KV * hd, rows, (unsigned long long)KV * hd * 2, AT_HD, AT_BN, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
    rc = make_map(&p.v_map, V, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (unsigned long long)KV * hd, rows, (unsigned long long)KV * hd * 2, AT_HD, AT_BN, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
    p.O = (bf16 *)O; p.lse = lse;
    p.B = B; p.T = T; p.H = H; p.KV = KV; p.win = win;
    p.nqt = (T + AT_BM - 1) / AT_BM;
    p.scale_log2 = 1.4426950408889634f / sqrtf((float)hd);
    p.errword = device_error_word();
    // the attribute belongs to a device's copy of the kernel: set it once per device of this process
    static bool configured_dev[64];
    int dev_ = 0;
    QLMB_CUDA(cudaGetDevice(&dev_));
    QLMB_REQUIRE(dev_ >= 0 && dev_ < 64, "device index %d", dev_);
    if (!configured_dev[dev_]) {
        QLMB_CUDA(cudaFuncSetAttribute(k_attn_fwd, cudaFuncAttributeMaxDynamicSharedMemorySize, AT_FWD_SMEM));
        configured_dev[dev_] = true;
    }
    QLMB_CUDA(pdl_launch_small(k_attn_fwd, dim3((unsigned)(p.nqt * B * H)), dim3(AT_FWD_THREADS), AT_FWD_SMEM, as_stream(stream), p));
    QLMB_LAUNCH_CHECK("k_attn_fwd");
    return QLMB_OK;
}

static int attn_bwd_impl(void *dQ, void *dK, void *dV, float *drow, const void *Q, const void *K, const void *V,
                         const void *O, const void *dA, const float *lse, const float *cosb, const float *sinb, int B, int T,
                         int H, int KV, int hd, int win, void *stream)
{
    QLMB_REQUIRE(dQ && dK && dV && drow && Q && K && V && O && dA && lse, "qlmb_attn_bwd: NULL argument");
    QLMB_REQUIRE(hd == AT_HD, "qlmb_attn_bwd: head dimension %d (only 64 is built)", hd);
    QLMB_REQUIRE(B > 0 && T > 0 && H > 0 && KV > 0 && H % KV == 0, "qlmb_attn_bwd: bad shape B %d T %d H %d KV %d", B, T, H, KV);
    AttnBwdParams p;
    memset(&p, 0, sizeof p);
    const unsigned long long rows = (unsigned long long)B * T, qw = (unsigned long long)H * hd, kw = (unsigned long long)KV * hd;
    struct { CUtensorMap *m; const void *base; unsigned long long width; unsigned box; } maps[8] = {
        {&p.q_map, Q, qw, AT_BM}, {&p.da_map, dA, qw, AT_BM}, {&p.k_map, K, kw, AT_BN}, {&p.v_map, V, kw, AT_BN},
        {&p.q_imap, Q, qw, AT_BI}, {&p.da_imap, dA, qw, AT_BI}, {&p.k_imap, K, kw, AT_BI}, {&p.v_imap, V, kw, AT_BI}};
    for (auto &m : maps) {
        const int rc = make_map(m.m, m.base, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, m.width, rows, m.width * 2, AT_HD, m.box, CU_TENSOR_MAP_SWIZZLE_128B);
        if (rc) return rc;
    }
    p.lse = lse; p.drow = drow; p.O = (const bf16 *)O; p.dA = (const bf16 *)dA;
    p.dQ = (bf16 *)dQ; p.dK = (bf16 *)dK; p.dV = (bf16 *)dV;
    p.cosb = cosb; p.sinb = sinb;
    p.B = B; p.T = T; p.H = H; p.KV = KV; p.win = win;
    p.nqt = (T + AT_BM - 1) / AT_BM;
    p.scale = 1.0f / sqrtf((float)hd);
    p.scale_log2 = 1.4426950408889634f * p.scale;
    p.errword = device_error_word();
    // the attribute belongs to a device's copy of the kernel: set it once per device of this process
    static bool configured_dev[64];
    int dev_ = 0;
    QLMB_CUDA(cudaGetDevice(&dev_));
    QLMB_REQUIRE(dev_ >= 0 && dev_ < 64, "device index %d", dev_);
    if (!configured_dev[dev_]) {
        QLMB_CUDA(cudaFuncSetAttribute(k_attn_bwd_dkv<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, AT_DKV_SMEM));
        QLMB_CUDA(cudaFuncSetAttribute(k_attn_bwd_dkv<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, AT_DKV_SMEM));
        QLMB_CUDA(cudaFuncSetAttribute(k_attn_bwd_dq, cudaFuncAttributeMaxDynamicSharedMemorySize, AT_DQ_SMEM));
        configured_dev[dev_] = true;
    }
    cudaStream_t st = as_stream(stream);
    // dQ in the place of Q or dA, which dkv reads as well: only drow comes first then, dQ behind dkv
    const bool in_place = dQ == Q || dQ == dA;
    auto launch_dq = [&](void *dst) {
        p.dQ = (bf16 *)dst;
        return pdl_launch_small(k_attn_bwd_dq, dim3((unsigned)(p.nqt * B * H)), dim3(AT_BWD_THREADS), AT_DQ_SMEM, st, p);
    };
    QLMB_CUDA(launch_dq(in_place ? nullptr : dQ));
    const int grp = H / KV, units = p.nqt * B * KV;
    if ((grp == 2 || grp == 4 || grp == 8) && units <= 2 * sm_count()) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)(units * grp)); cfg.blockDim = dim3(AT_BWD_THREADS); cfg.dynamicSmemBytes = AT_DKV_SMEM; cfg.stream = st;
        cudaLaunchAttribute at[2];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned)grp; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
        at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = at; cfg.numAttrs = units * grp <= 2 * sm_count() && pdl_enabled() ? 2 : 1;
        QLMB_CUDA(cudaLaunchKernelEx(&cfg, k_attn_bwd_dkv<true>, p));
    } else {
        QLMB_CUDA(pdl_launch_small(k_attn_bwd_dkv<false>, dim3((unsigned)units), dim3(AT_BWD_THREADS), AT_DKV_SMEM, st, p));
    }
    if (in_place) QLMB_CUDA(launch_dq(dQ));
    QLMB_LAUNCH_CHECK("k_attn_bwd");
    return QLMB_OK;
}

extern "C" int qlmb_attn_bwd(void *dQ, void *dK, void *dV, float *drow, const void *Q, const void *K, const void *V,
                             const void *O, const void *dA, const float *lse, int B, int T, int H, int KV, int hd,
                             int win, void *stream)
{
    return attn_bwd_impl(dQ, dK, dV, drow, Q, K, V, O, dA, lse, nullptr, nullptr, B, T, H, KV, hd, win, stream);
}
extern "C" int qlmb_attn_bwd_rope(void *dQ, void *dK, void *dV, float *drow, const void *Q, const void *K, const void *V,
                                  const void *O, const void *dA, const float *lse, const float *cosb, const float *sinb,
                                  int B, int T, int H, int KV, int hd, int win, void *stream)
{
    QLMB_REQUIRE(cosb && sinb && ((((uintptr_t)cosb | (uintptr_t)sinb) & 15) == 0), "qlmb_attn_bwd_rope: tables must be given and 16-byte aligned");
    return attn_bwd_impl(dQ, dK, dV, drow, Q, K, V, O, dA, lse, cosb, sinb, B, T, H, KV, hd, win, stream);
}
