// One decode step's layers in ONE persistent launch (dec_step, cudalm.cu:7168-7212), up to 64 routed slots: embedding, then
// per layer the q, k, v projections with the norm in front, cached attention, output projection + residual + norm,
// router, the routed experts and their combination, and the final norm.  With so few rows a layer is 5 MB of weights,
// which the memory system delivers in under a microsecond; what a step costs is latency: the chain of launches that
// this replaces spent 4-6 us in each of nine launches per layer.
//
// One CTA of 512 threads per SM (cooperative launch); what the seven phases of a layer hand to one another is waited for
// word by word (see DS_NONE below), a hop of 0.8 us, where a grid barrier between two phases and the loads behind it took
// 1.3.  Between two hops the longest chain of dependent instructions sets the time (about five cycles each), so every
// phase is written for a short one:
//   - a weight phase is a set of tasks of 256 output columns x 128 contraction rows: a warp takes eight rows, a lane one
//     code word (eight columns) of each, so a load instruction covers a whole 128-byte line, the sums of a column stay
//     in one lane, and the 16 warps' sums meet once in shared memory;
//   - codes and scales of a phase whose choice of weights is known are in registers before its input is waited for;
//   - slice sums go to the consumer as they are and are added there (its loads are independent of one another), in a
//     fixed order, so a step is reproducible bit for bit;
//   - the cached keys and values of an attention phase and the router's matrix reach shared memory before their phase.
// Products are fp32: x * scale times the exact digit, as in the kernels of the separate entry points.
// Measured (12 layers, D 768, 32 experts top-2 of d_ff 1536, 128-256 cached positions, whole step with the head, a CUDA
// graph replay): one slot 276 us with grid barriers, 199 now, eight slots 477 and 415 (the chain of launches: 615 and
// 801).  Where the form ends stands at ds_fits: with many slots the experts' weights are a stream and no longer a latency.
//
// Built with --fmad=false (router arithmetic); fused multiply-adds are written out.
#include <cuda_bf16.h>
#include <string.h>
#include "qlmb_common.cuh"
#include "qlmb_internal.h"
#include "qlmb_topk.cuh"

namespace qlmb {

struct DsLayer {                                          // the device table's row: pointers only (qlmb_dec_step_args)
    const uint8_t *c[7];                                  // codes of wq, wk, wv, wo, w1, w3, w2
    const float *s[7];                                    // their group scales
    const float *an1, *an2, *wr;
    bf16 *Kc, *Vc;
    float *rt, *rprobs;
    int *assign;
    float *gate;
};
constexpr int DS_LAYER_WORDS = sizeof(DsLayer) / 8;
// alignment of the row's w-th pointer: 16 bytes where it is read in 16-byte pieces (the experts' codes, gains, router, caches)
__device__ __forceinline__ unsigned ds_align_mask(int w) { return (w >= 4 && w < 7) || (w >= 14 && w < 19) ? 15u : 3u; }

struct DsArgs {
    const DsLayer *layers;
    int L, B, D, KD, H, KV, F, E, K, Tm;
    int tq, td, tf;                                       // column tiles of q|k|v, of D and of F
    uint32_t mq, md, mf, mr, mfs;                         // ceil(2^32 / n) of those and of the row slices of D and F
    const float *emb; const int *tok, *pos; const float *cosb, *sinb, *nf;
    bf16 *fn;
    // workspace: the header and three exchange slots
    unsigned *bar;
    uint8_t *slots;
    size_t slot_bytes, att, fnorm, asg, pq, po, pg, pd;   // offsets of a slot's parts; xn is at 0
    int *errword;
};

constexpr int DS_THREADS = 512, DS_WARPS = 16;
constexpr int DS_ROWS = 128;                              // contraction rows of a task: eight per warp
constexpr int DS_COLS = 256;
constexpr int DS_MAX_B = 32, DS_MAX_R = 64;
constexpr int DS_MAX_SL = 8;                              // row slices of D (D <= 1024)
constexpr int DS_RED = DS_WARPS * 4 * DS_COLS * 4;        // up to four rows' sums of the 16 warps
constexpr int DS_WR = 1024 * 32 * 4;                      // the router's matrix, or keys and values of an attention phase
constexpr int DS_XS = 2 * DS_ROWS * 4;
constexpr int DS_FN = 16384;                              // the rows that the experts take: this and what the ring leaves of DS_WR
constexpr int DS_SLOT = DS_ROWS * 136, DS_DEPTH = 7;      // a task's codes and scales; tasks on their way (in the place of DS_WR)
static_assert(DS_DEPTH * DS_SLOT <= DS_WR && DS_DEPTH * DS_SLOT % 16 == 0, "ring");
constexpr int DS_FN_ELEMS = (DS_WR - DS_DEPTH * DS_SLOT + DS_FN) / 2;
constexpr int DS_SMEM = DS_RED + DS_WR + DS_XS + DS_FN;

__device__ __forceinline__ uint32_t ds_smem(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void ds_cp16(uint32_t dst, const void *src)
{ asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory"); }
__device__ __forceinline__ void ds_cp4(uint32_t dst, const void *src)
{ asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory"); }
__device__ __forceinline__ void ds_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void ds_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ float ds_bf(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }
__device__ __forceinline__ float ds_lo(uint32_t x) { return __uint_as_float(x << 16); }
__device__ __forceinline__ float ds_hi(uint32_t x) { return __uint_as_float(x & 0xffff0000u); }
__device__ __forceinline__ uint32_t ds_pack(float a, float b)
{
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t *>(&v);
}
__device__ __forceinline__ float4 ds_bf4(float4 v) { return make_float4(ds_bf(v.x), ds_bf(v.y), ds_bf(v.z), ds_bf(v.w)); }
__device__ __forceinline__ void ds_add4(float4 &a, const float4 b) { a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w; }
__device__ __forceinline__ void ds_fma4(float4 &a, float g, const float4 b)
{ a.x = __fmaf_rn(g, b.x, a.x); a.y = __fmaf_rn(g, b.y, a.y); a.z = __fmaf_rn(g, b.z, a.z); a.w = __fmaf_rn(g, b.w, a.w); }

struct Shared {
    DsLayer layer[2];
    int pos[DS_MAX_B];
    int npair, pexp[DS_MAX_R];                            // distinct experts of slots 0 .. 31 and of 32 .. 63 (expert | half << 8),
    unsigned pmask[DS_MAX_R];                             // and their slots
    int srow[DS_MAX_R];                                   // the row of a slot
    int ab, ah, akv, afirst;                                      // the CTA's attention item: slot, head, key/value head
    float red[DS_WARPS];
    alignas(16) float am[DS_WARPS], al[DS_WARPS];                     // attention: the warps' maxima and sums
    float q[64];
    alignas(16) bf16 kv[128];
    alignas(16) float part[DS_WARPS * 64];
    float logit[DS_WARPS * 32];
    float gate[DS_WARPS];                                 // a row owner's gates
    alignas(16) float x[1024];                                        // a row owner's residual stream (bf16 values), thread q columns 4q .. 4q + 3
};

// ---- exchange between the CTAs.  What a phase hands to the next one goes through 32-bit words that hold DS_NONE until
// they are written: a reader loads the words it needs, all in flight at once, and loads them again while one of them is
// DS_NONE.  A hop is a store and a load; with a grid barrier between the phases it was a store, a fence, an arrival, a
// poll and a load.  DS_NONE is a NaN that no arithmetic makes (results are the canonical NaN), and ds_word keeps it out.
// Layer l writes slot l of three, and its start clears the slot of layer l + 1, which layer l - 2 used (and the q, k, v
// projections of layer l - 1, for xn).  A grid barrier per layer, arrived at behind the output projection and waited for
// at the next layer's start, tells that the slot of two layers ago is read and the next one clear, long before the wait.
// The launch leaves the slots as a further layer would find them; the header keeps which is next, and the shape that they
// are laid out for: another one (or the zeros of a new workspace) clears all three first.
constexpr uint32_t DS_NONE = 0xffffffffu;
__device__ __forceinline__ uint32_t ds_word(uint32_t v) { return v == DS_NONE ? 0x7fff7fffu : v; }
__device__ __forceinline__ void ds_put(void *p, uint32_t v) { asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory"); }
__device__ __forceinline__ void ds_put(float *p, float v) { ds_put((void *)p, ds_word(__float_as_uint(v))); }
__device__ __forceinline__ void ds_putrow(bf16 *p, float4 v)
{
    asm volatile("st.relaxed.gpu.global.v2.u32 [%0], {%1, %2};" ::"l"(p), "r"(ds_word(ds_pack(v.x, v.y))), "r"(ds_word(ds_pack(v.z, v.w))) : "memory");
}
__device__ __forceinline__ uint32_t ds_get(const void *p) { uint32_t v; asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory"); return v; }
__device__ __forceinline__ uint4 ds_get4(const void *p)
{
    uint4 v;
    asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t ds_max4(uint4 v) { return max(max(v.x, v.y), max(v.z, v.w)); }
__device__ __forceinline__ float4 ds_float4(uint4 v) { return make_float4(__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), __uint_as_float(v.w)); }
// Waits are bounded by some seconds of polls (an L2 latency each); when one runs out, the abort word ends every other.
__device__ __noinline__ bool ds_give_up(unsigned *bar, int *errword, unsigned polls)
{
    if (*(volatile unsigned *)(bar + 2)) return true;
    if (polls < (1u << 23)) return false;
    if (atomicExch(bar + 2, 1u) == 0u && errword && atomicCAS(errword, 0, 200) == 0) { errword[1] = 400; errword[2] = (int)blockIdx.x; errword[3] = (int)threadIdx.x; }
    return true;
}
// load() = the largest of the words asked for
template <typename Load> __device__ __forceinline__ void ds_poll(const DsArgs &a, Load load)
{
    unsigned i = 0;
    while (load() == DS_NONE)
        if ((++i & 1023u) == 0u && ds_give_up(a.bar, a.errword, i)) return;
}
// the grid barrier: one counter per launch, reset by the last CTA to leave the kernel
__device__ __forceinline__ void gb_arrive(const DsArgs &a) { asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(a.bar) : "memory"); }
__device__ __forceinline__ void gb_wait(const DsArgs &a, unsigned target)
{
    for (unsigned i = 1;; i++) {
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(a.bar) : "memory");
        if (v >= target || ((i & 1023u) == 0u && ds_give_up(a.bar, a.errword, i))) return;
    }
}
__device__ __forceinline__ void ds_clear(uint8_t *at, size_t bytes)
{
    for (size_t i = (blockIdx.x * DS_THREADS + threadIdx.x) * 16; i < bytes; i += gridDim.x * DS_THREADS * 16)
        *reinterpret_cast<uint4 *>(at + i) = make_uint4(DS_NONE, DS_NONE, DS_NONE, DS_NONE);
}

// ---- weight phases
__device__ __forceinline__ int ds_div(int x, int n, uint32_t m) { return n == 1 ? x : (int)__umulhi((uint32_t)x, m); }   // m = ceil(2^32 / n)
struct Words { uint32_t w[8]; float s[8]; };              // eight rows of a lane's eight columns, and their group scales
__device__ __forceinline__ void ds_words(Words &r, const uint8_t *codes, const float *scales, int N, int col, int k0)
{
    const uint8_t *cp = codes + (size_t)k0 * (N >> 1) + (col >> 1);
    const float *sp = scales + (size_t)k0 * (N >> 7) + (col >> 7);
#pragma unroll
    for (int i = 0; i < 8; i++) {
        r.w[i] = __ldcs(reinterpret_cast<const uint32_t *>(cp));
        r.s[i] = __ldg(sp);
        cp += N >> 1; sp += N >> 7;
    }
}
// eight nibbles of a code word as exact floats (two's complement, element 0 in the low nibble): a byte in 0..15 under
// the exponent of 2^23 is 8388608 + byte, and (nibble ^ 8) - 8 is the value.  Digits are made and multiplied two at a time:
// with many experts chosen the tasks are bound by the instructions they issue (eight slots, with one barrier a pass instead
// of two: 504 -> 476 us a step).
struct Sums { uint64_t v[4]; };                           // a lane's eight columns of a row: pairs of neighbouring columns
__device__ __forceinline__ uint64_t ds_pair(uint32_t x) { uint64_t r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(x << 16), "r"(x & 0xffff0000u)); return r; }
__device__ __forceinline__ uint64_t ds_two(float lo, float hi) { uint64_t r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi)); return r; }
__device__ __forceinline__ uint64_t ds_two(uint32_t lo, uint32_t hi) { uint64_t r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi)); return r; }
__device__ __forceinline__ float2 ds_apart(uint64_t v) { float2 r; asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v)); return r; }
__device__ __forceinline__ uint64_t ds_fma2(uint64_t a, uint64_t b, uint64_t c) { uint64_t r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r; }
__device__ __forceinline__ uint64_t ds_mul2(uint64_t a, uint64_t b) { uint64_t r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ uint64_t ds_add2(uint64_t a, uint64_t b) { uint64_t r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
template <int C>
__device__ __forceinline__ void ds_mul(const Words &r, const float (&x)[C][8], Sums (&acc)[C])
{
    const uint64_t off = ds_two(-8388616.0f, -8388616.0f);
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const uint32_t w = r.w[i] ^ 0x88888888u, ev = w & 0x0F0F0F0Fu, od = (w >> 4) & 0x0F0F0F0Fu;
        uint64_t d[4];
#pragma unroll
        for (int j = 0; j < 4; j++) d[j] = ds_add2(ds_two(__byte_perm(ev, 0x4B000000u, 0x7440 + j), __byte_perm(od, 0x4B000000u, 0x7440 + j)), off);
#pragma unroll
        for (int c = 0; c < C; c++) {
            const float xs = x[c][i] * r.s[i];
            const uint64_t xv = ds_two(xs, xs);
#pragma unroll
            for (int j = 0; j < 4; j++) acc[c].v[j] = i == 0 ? ds_mul2(xv, d[j]) : ds_fma2(xv, d[j], acc[c].v[j]);
        }
    }
}
__device__ __forceinline__ void ds_x8(float (&x)[8], uint4 u)
{
    x[0] = ds_lo(u.x); x[1] = ds_hi(u.x); x[2] = ds_lo(u.y); x[3] = ds_hi(u.y);
    x[4] = ds_lo(u.z); x[5] = ds_hi(u.z); x[6] = ds_lo(u.w); x[7] = ds_hi(u.w);
}
// the 16 warps' sums of C rows -> out[row(c) * N + col0 + column], warp order.  The caller syncs before `red` is used again.
template <int C, typename RowPtr>
__device__ __forceinline__ void ds_reduce(float *red, const Sums (&acc)[C], int n, int col0, int N, RowPtr row)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int c = 0; c < C; c++) {
        float4 *p = reinterpret_cast<float4 *>(red + (warp * C + c) * DS_COLS + lane * 8);
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const float2 u = ds_apart(acc[c].v[2 * h]), v = ds_apart(acc[c].v[2 * h + 1]);
            p[h] = make_float4(u.x, u.y, v.x, v.y);
        }
    }
    __syncthreads();
    const int col = threadIdx.x & 255;
    if (col0 + col < N) {
#pragma unroll 1
        for (int c = threadIdx.x >> 8; c < n; c += 2) {
            float v = 0.0f;
#pragma unroll
            for (int w = 0; w < DS_WARPS; w++) v += red[(w * C + c) * DS_COLS + col];
            ds_put(row(c) + col0 + col, v);
        }
    }
}

// q, k, v projections (KIND 0) and output projection (KIND 1): a task takes C of the B rows
template <int C>
__device__ __forceinline__ void ds_dense(const DsArgs &a, const DsLayer &ly, float *red, bool wo, const uint8_t *in, uint8_t *slot)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tiles = !wo ? a.tq : a.td, NT = !wo ? a.D + 2 * a.KD : a.D, sl = a.D / DS_ROWS, n = tiles * sl * ((a.B + C - 1) / C);
    const bf16 *X = reinterpret_cast<const bf16 *>(in);
    float *out = reinterpret_cast<float *>(slot + (!wo ? a.pq : a.po));
    bool first = true;
#pragma unroll 1
    for (int task = blockIdx.x; task < n; task += gridDim.x) {
        const int ts = ds_div(task, tiles, !wo ? a.mq : a.md), col0 = (task - ts * tiles) * DS_COLS, ch = ds_div(ts, sl, a.mr);
        const int slice = ts - ch * sl, k0 = slice * DS_ROWS + warp * 8, b0 = ch * C;
        int col = col0 + lane * 8;
        if (col >= NT) col = NT - 8;                      // lanes past the last column repeat it and are not read
        int m = wo ? 3 : 0, N = a.D;
        if (!wo) {
            if (col >= a.D) { col -= a.D; m = 1; N = a.KD; if (col >= a.KD) { col -= a.KD; m = 2; } }
        }
        Words w;
        ds_words(w, ly.c[m], ly.s[m], N, col, k0);
        if (first) first = false; else __syncthreads();
        uint4 xr[C];
        ds_poll(a, [&] {
            uint32_t m = 0;
#pragma unroll
            for (int c = 0; c < C; c++) xr[c] = b0 + c < a.B ? ds_get4(X + (size_t)(b0 + c) * a.D + k0) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
            for (int c = 0; c < C; c++) m = max(m, ds_max4(xr[c]));
            return m;
        });
        float x[C][8];
        Sums acc[C];
#pragma unroll
        for (int c = 0; c < C; c++) ds_x8(x[c], xr[c]);
        ds_mul<C>(w, x, acc);
        ds_reduce<C>(red, acc, a.B - b0 < C ? a.B - b0 : C, col0, NT, [&](int c) { return out + ((size_t)slice * a.B + b0 + c) * NT; });
    }
}

// The experts' tasks.  An expert has one or two slots as a rule: a pass multiplies up to two, and the weights, the first
// pass's activations and, in the down projection, the gate and up sums they are made of are requested a task ahead.
struct ExTask { int pair, mat, slice, tile, base, s0, s1, n; unsigned rest; };     // s0, s1: the pass's slots (n of them), rest: those that follow, of base on
__device__ __forceinline__ void ds_pass(ExTask &t, unsigned mask)
{
    t.s0 = t.base + __ffs(mask) - 1;
    mask &= mask - 1;
    t.n = mask ? 2 : 1;
    t.s1 = mask ? t.base + __ffs(mask) - 1 : t.s0;
    t.rest = mask & (mask - 1);
}
__device__ __forceinline__ ExTask ds_ex_task(const DsArgs &a, const Shared &sh, bool down, bool many, int item)
{
    ExTask t;
    if (down) {
        const int fs = a.F / DS_ROWS, q = ds_div(item, a.td, a.md);
        t.tile = item - q * a.td; t.mat = 0;
        t.pair = ds_div(q, fs, a.mfs);
        t.slice = q - t.pair * fs;
    } else {
        const int sl = a.D / DS_ROWS, q = ds_div(item, a.tf, a.mf), pm = ds_div(q, sl, a.mr);
        t.tile = item - q * a.tf;
        t.slice = q - pm * sl;
        t.mat = pm & 1; t.pair = pm >> 1;
    }
    t.base = many ? sh.pexp[t.pair] >> 8 << 5 : 0;
    ds_pass(t, sh.pmask[t.pair]);
    return t;
}
// The codes and scales of a task go through a ring in shared memory, DS_DEPTH tasks ahead: with one task (17 KB per SM)
// ahead a round of tasks took a memory latency.  Every warp copies and reads its own eight rows only.
__device__ __forceinline__ void ds_ex_request(const DsArgs &a, const Shared &sh, bool down, const DsLayer &ly, uint8_t *ring, int slot, const ExTask &t)
{
    const int N = down ? a.D : a.F, m = down ? 6 : 4 + t.mat, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const size_t mat = (size_t)(sh.pexp[t.pair] & 255) * a.D * a.F;
    const int k0 = t.slice * DS_ROWS + warp * 8, r = lane >> 3, c = lane & 7;
    const uint32_t d = ds_smem(ring + slot * DS_SLOT);
    const bool in = t.tile * DS_COLS + c * 32 < N;        // N is a multiple of 128: the last tile may be half as wide
    const uint8_t *p = ly.c[m] + mat / 2 + (size_t)(k0 + r) * (N >> 1) + (in ? t.tile * 128 + c * 16 : 0);
    if (in) {
        ds_cp16(d + warp * 1024 + lane * 16, p);
        ds_cp16(d + warp * 1024 + 512 + lane * 16, p + (size_t)4 * (N >> 1));
    }
    const int g = 2 * t.tile + (lane & 1);
    if (lane < 16 && g < (N >> 7)) ds_cp4(d + 16384 + warp * 64 + lane * 4, ly.s[m] + mat / 128 + (size_t)(k0 + (lane >> 1)) * (N >> 7) + g);
}
__device__ __forceinline__ void ds_ring_words(Words &w, const uint8_t *ring, int slot)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint8_t *p = ring + slot * DS_SLOT + warp * 1024 + lane * 4, *q = ring + slot * DS_SLOT + 16384 + warp * 64 + (lane >> 4) * 4;
#pragma unroll
    for (int i = 0; i < 8; i++) { w.w[i] = *reinterpret_cast<const uint32_t *>(p + i * 128); w.s[i] = *reinterpret_cast<const float *>(q + i * 8); }
}
// down: gate and up sums of one row of the slice (threads 0 .. 127: first slot, 128 .. 255: second)
struct DnActs { uint32_t g[DS_MAX_SL], u[DS_MAX_SL]; };
__device__ __forceinline__ void ds_dn_acts(const DsArgs &a, DnActs &x, const ExTask &t, const uint8_t *slot)
{
    const int R = a.K * a.B, ns = a.D / DS_ROWS;
    if ((int)threadIdx.x >= t.n * DS_ROWS) return;
    const float *p = reinterpret_cast<const float *>(slot + a.pg) + (size_t)((int)threadIdx.x < DS_ROWS ? t.s0 : t.s1) * a.F + t.slice * DS_ROWS + (threadIdx.x & (DS_ROWS - 1));
#pragma unroll
    for (int s = 0; s < DS_MAX_SL; s++) {
        x.g[s] = s < ns ? ds_get(p) : 0u;
        x.u[s] = s < ns ? ds_get(p + (size_t)R * a.F) : 0u;
        p += (size_t)2 * R * a.F;
    }
}
__device__ __forceinline__ float ds_swiglu(const DnActs &x)
{
    float g = 0.0f, u = 0.0f;
#pragma unroll
    for (int s = 0; s < DS_MAX_SL; s++) { g += __uint_as_float(x.g[s]); u += __uint_as_float(x.u[s]); }
    g = ds_bf(g); u = ds_bf(u);
    return ds_bf(g * __fdividef(1.0f, 1.0f + __expf(-g)) * u);
}
template <int C>
__device__ __forceinline__ void ds_ex_pass(const DsArgs &a, const Shared &sh, bool down, float *red, const float *xs, const bf16 *fn, const Words &w, const ExTask &t, uint8_t *slot)
{
    const int warp = threadIdx.x >> 5, R = a.K * a.B, N = down ? a.D : a.F;
    float x[C][8];
    Sums acc[C];
    if (down) {
#pragma unroll
        for (int c = 0; c < C; c++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const float4 v = *reinterpret_cast<const float4 *>(xs + c * DS_ROWS + warp * 8 + 4 * h);
                x[c][4 * h] = v.x; x[c][4 * h + 1] = v.y; x[c][4 * h + 2] = v.z; x[c][4 * h + 3] = v.w;
            }
    } else {
        const bf16 *p = fn + t.slice * DS_ROWS + warp * 8;
        ds_x8(x[0], *reinterpret_cast<const uint4 *>(p + sh.srow[t.s0] * a.D));
        if (C > 1) ds_x8(x[C - 1], *reinterpret_cast<const uint4 *>(p + sh.srow[t.s1] * a.D));
    }
    ds_mul<C>(w, x, acc);
    float *out = reinterpret_cast<float *>(slot + (down ? a.pd : a.pg)) + (down ? (size_t)t.slice * R * a.D : (size_t)(t.slice * 2 + t.mat) * R * a.F);
    ds_reduce<C>(red, acc, t.n, t.tile * DS_COLS, N, [&](int c) { return out + (size_t)(c == 0 ? t.s0 : t.s1) * N; });
}
// The down projection's choice of weights is known: its sums are waited for with the first tasks' weights on their way.
__device__ __forceinline__ void ds_experts_phase(const DsArgs &a, Shared &sh, bool down, const DsLayer &ly, float *red, float *xs, const bf16 *fn, uint8_t *ring, bool multi, bool many, uint8_t *slot8)
{
    const int n = down ? sh.npair * (a.F / DS_ROWS) * a.td : sh.npair * 2 * (a.D / DS_ROWS) * a.tf;
    int ask = blockIdx.x, item = blockIdx.x, slot = 0;
#pragma unroll 1
    for (int k = 0; k < DS_DEPTH; k++) {
        if (ask < n) ds_ex_request(a, sh, down, ly, ring, k, ds_ex_task(a, sh, down, many, ask));
        ds_commit();
        ask += gridDim.x;
    }
    if (item >= n) return;
    ExTask t = ds_ex_task(a, sh, down, many, item);
    DnActs da;
    if (down) ds_dn_acts(a, da, t, slot8);
    Words w;
    bool fresh = true;
    // two places for the warps' sums in turn: a warp is past the barrier inside a pass only when every warp has added up
    // the pass before, so one barrier a pass (two in the down projection, for xs) keeps both and xs safe
    constexpr int HALF = DS_RED / 8;
    int place = 0;
#pragma unroll 1
    for (;;) {
        if (down) {                                       // the slice's activations of this pass
            if ((int)threadIdx.x < t.n * DS_ROWS) {
                unsigned i = 0;
                for (;;) {
                    uint32_t m = 0;
#pragma unroll
                    for (int s = 0; s < DS_MAX_SL; s++) m = max(m, max(da.g[s], da.u[s]));
                    if (m != DS_NONE || ((++i & 1023u) == 0u && ds_give_up(a.bar, a.errword, i))) break;
                    ds_dn_acts(a, da, t, slot8);
                }
                xs[threadIdx.x] = ds_swiglu(da);
            }
            __syncthreads();
        }
        if (fresh) {
            ds_wait<DS_DEPTH - 1>();
            __syncwarp();
            ds_ring_words(w, ring, slot);
            __syncwarp();
            if (ask < n) ds_ex_request(a, sh, down, ly, ring, slot, ds_ex_task(a, sh, down, many, ask));
            ds_commit();
            ask += gridDim.x;
            if (++slot == DS_DEPTH) slot = 0;
        }
        const ExTask cur = t;
        fresh = !(multi && t.rest);                       // else: more slots of the same expert, same weights
        if (!fresh) ds_pass(t, t.rest);
        else {
            item += gridDim.x;
            if (item < n) t = ds_ex_task(a, sh, down, many, item);
        }
        if (down && item < n) ds_dn_acts(a, da, t, slot8);
        if (multi && cur.n == 2) ds_ex_pass<2>(a, sh, down, red + place, xs, fn, w, cur, slot8);
        else ds_ex_pass<1>(a, sh, down, red + place, xs, fn, w, cur, slot8);
        if (item >= n) break;
        place ^= HALF;
    }
    ds_wait<0>();
}

// ---- attention of one (slot, head) by a CTA: the head's q, k, v rows from the projection's slice sums, rotation, cache
// append; then every warp takes 16 of each 256 keys on its own with a running maximum, and the warps' results are merged
// at the end.  Keys and values reach shared memory by asynchronous copies, four whole 128-byte rows per instruction (a
// lane per key, eight 16-byte loads in 32 different lines each, held the load path for 6.5 thousand cycles per 256 keys):
// the first 256 at the layer's start, the next ones while these are multiplied.  Lane (r = lane / 8, c = lane % 8)
// multiplies dimensions 8c .. 8c + 7 of the keys 4i + r.
constexpr int DS_KV = 16 * 256;                           // bytes of a warp's keys and values of one pass
__device__ __forceinline__ void ds_kv_request(const DsArgs &a, const Shared &sh, const DsLayer &ly, uint8_t *kvs, int blk)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, b = sh.ab, kvh = sh.akv;
    const int t = sh.pos[b], s0 = blk * 256 + warp * 16, left = t < 0 || t >= a.Tm ? 0 : t - s0, r = lane >> 3;
    if (left > 0) {
        const size_t base = ((size_t)b * a.Tm + s0) * a.KD + kvh * 64 + (lane & 7) * 8;
        const uint32_t d = ds_smem(kvs + (blk & 1) * DS_WARPS * DS_KV + warp * DS_KV) + lane * 16;
#pragma unroll
        for (int i = 0; i < 4; i++) {                     // rows past the end repeat the first one and get no weight
            const int k = (4 * i + r < left ? 4 * i + r : 0) * a.KD;
            ds_cp16(d + i * 512, ly.Kc + base + k);
            ds_cp16(d + i * 512 + 2048, ly.Vc + base + k);
        }
    }
    ds_commit();
}
__device__ __forceinline__ void ds_item(const DsArgs &a, Shared &sh, int item)      // by one thread
{
    const int rep = a.H / a.KV, b = item / a.H, h = item - b * a.H;
    sh.ab = b; sh.ah = h; sh.akv = h / rep; sh.afirst = h % rep == 0;
}
__device__ __forceinline__ void ds_attention_item(const DsArgs &a, Shared &sh, const DsLayer &ly, uint8_t *kvs, uint8_t *slot)
{
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, b = sh.ab, h = sh.ah, kvh = sh.akv;
    const int t = sh.pos[b], r = lane >> 3, c8 = (lane & 7) * 8, mm = tid >> 6, i64 = tid & 63;
    const bool bad = t < 0 || t >= a.Tm;                  // a slot past its cache: nothing of it is read or written
    float cs = 0.0f, sn = 0.0f;
    if (tid < 128 && !bad) { cs = __ldg(a.cosb + (size_t)t * 32 + (i64 & 31)); sn = __ldg(a.sinb + (size_t)t * 32 + (i64 & 31)); }
    bf16 *out = reinterpret_cast<bf16 *>(slot + a.att) + (size_t)b * a.D + h * 64 + tid;
    if (bad) {
        ds_wait<0>();
        if (tid == 0 && h == 0) report_bad_index(a.errword, 302, b, t);
        if (tid < 64 && !(tid & 1)) ds_put((void *)out, 0u);
        return;
    }
    float x = 0.0f;
    if (tid < 192) {                                      // one of the 64 columns of q, k or v
        const int NQ = a.D + 2 * a.KD, ns = a.D / DS_ROWS;
        const float *pp = reinterpret_cast<const float *>(slot + a.pq) + (size_t)b * NQ + (mm == 0 ? h * 64 : a.D + (mm - 1) * a.KD + kvh * 64) + i64;
        uint32_t pv[DS_MAX_SL];
        ds_poll(a, [&] {
            uint32_t m = 0;
#pragma unroll
            for (int k = 0; k < DS_MAX_SL; k++) pv[k] = k < ns ? ds_get(pp + (size_t)k * a.B * NQ) : 0u;
#pragma unroll
            for (int k = 0; k < DS_MAX_SL; k++) m = max(m, pv[k]);
            return m;
        });
#pragma unroll
        for (int k = 0; k < DS_MAX_SL; k++) x += __uint_as_float(pv[k]);
        x = ds_bf(x);
        sh.part[tid] = x;
    }
    __syncthreads();
    if (tid < 192) {
        if (mm < 2) {                                     // pairs (i, i + 32) of q and k
            const float y = sh.part[tid ^ 32];
            x = i64 < 32 ? x * cs - y * sn : x * cs + y * sn;
        }
        const bf16 xb = __float2bfloat16_rn(x);
        if (mm == 0) sh.q[i64] = __bfloat162float(xb);
        else {
            sh.kv[tid - 64] = xb;
            if (sh.afirst) (mm == 1 ? ly.Kc : ly.Vc)[((size_t)b * a.Tm + t) * a.KD + kvh * 64 + i64] = xb;
        }
    }
    __syncthreads();
    float m = -1e30f, l = 0.0f;
    uint64_t o[4], q[4];                                  // pairs of neighbouring dimensions
#pragma unroll
    for (int d = 0; d < 4; d++) { o[d] = 0ull; q[d] = ds_two(sh.q[c8 + 2 * d], sh.q[c8 + 2 * d + 1]); }
#pragma unroll 1
    for (int blk = 0; blk * 256 <= t; blk++) {
        const int left = t - blk * 256 - warp * 16;       // this warp's keys 0 .. left of the pass, the last one new
        uint8_t *mine = kvs + (blk & 1) * DS_WARPS * DS_KV + warp * DS_KV;
        if ((blk + 1) * 256 <= t) { ds_kv_request(a, sh, ly, kvs, blk + 1); ds_wait<1>(); }
        else ds_wait<0>();
        if (left < 0) continue;
        __syncwarp();                                     // a lane has waited for its own copies only, and row `left` is one's target
        if (left < 16 && r < 2)                           // the new key and value are not read back from the cache
            *reinterpret_cast<uint4 *>(mine + r * 2048 + left * 128 + c8 * 2) = *reinterpret_cast<const uint4 *>(sh.kv + r * 64 + c8);
        __syncwarp();
        float d[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const uint4 k = *reinterpret_cast<const uint4 *>(mine + i * 512 + lane * 16);
            const float2 s = ds_apart(ds_fma2(q[3], ds_pair(k.w), ds_fma2(q[2], ds_pair(k.z), ds_fma2(q[1], ds_pair(k.y), ds_mul2(q[0], ds_pair(k.x))))));
            d[i] = s.x + s.y;
        }
#pragma unroll
        for (int y = 1; y < 8; y <<= 1)
#pragma unroll
            for (int i = 0; i < 4; i++) d[i] += __shfl_xor_sync(0xffffffffu, d[i], y);
        float mx = -1e30f;
#pragma unroll
        for (int i = 0; i < 4; i++) { d[i] = 4 * i + r <= left ? d[i] * 0.125f : -1e30f; mx = fmaxf(mx, d[i]); }
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
        const float mn = fmaxf(m, mx), corr = __expf(m - mn);
        m = mn;
        l *= corr;
#pragma unroll
        for (int e = 0; e < 4; e++) o[e] = ds_mul2(o[e], ds_two(corr, corr));
#pragma unroll
        for (int i = 0; i < 4; i++) {
            if (4 * i + r <= left) {                      // (rows that were never copied must not meet a zero weight)
                const float w = __expf(d[i] - mn);
                const uint4 v = *reinterpret_cast<const uint4 *>(mine + 2048 + i * 512 + lane * 16);
                const uint64_t ww = ds_two(w, w);
                l += w;
                o[0] = ds_fma2(ww, ds_pair(v.x), o[0]); o[1] = ds_fma2(ww, ds_pair(v.y), o[1]);
                o[2] = ds_fma2(ww, ds_pair(v.z), o[2]); o[3] = ds_fma2(ww, ds_pair(v.w), o[3]);
            }
        }
        __syncwarp();                                     // before the keys after the next overwrite these
    }
    // l and o hold the lane's keys only: add the four key rows of the warp, then merge the warps
#pragma unroll
    for (int y = 8; y < 32; y <<= 1) {
        l += __shfl_xor_sync(0xffffffffu, l, y);
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const float2 u = ds_apart(o[e]);
            o[e] = ds_add2(o[e], ds_two(__shfl_xor_sync(0xffffffffu, u.x, y), __shfl_xor_sync(0xffffffffu, u.y, y)));
        }
    }
    __syncthreads();                                      // part held the projections' sums
    if (r == 0) {
        *reinterpret_cast<ulonglong2 *>(sh.part + warp * 64 + c8) = make_ulonglong2(o[0], o[1]);
        *reinterpret_cast<ulonglong2 *>(sh.part + warp * 64 + c8 + 4) = make_ulonglong2(o[2], o[3]);
    }
    if (lane == 0) { sh.am[warp] = m; sh.al[warp] = l; }
    __syncthreads();
    if (tid < 64) {
        float M = sh.am[0], y = 0.0f, sum = 0.0f;
#pragma unroll
        for (int w = 1; w < DS_WARPS; w++) M = fmaxf(M, sh.am[w]);
#pragma unroll 8
        for (int w = 0; w < DS_WARPS; w++) { const float f = __expf(sh.am[w] - M); sum += f * sh.al[w]; y += f * sh.part[w * 64 + tid]; }
        y = __fdividef(y, sum);
        const float z = __shfl_down_sync(0xffffffffu, y, 1);
        if (!(tid & 1)) ds_put((void *)out, ds_word(ds_pack(y, z)));
    }
}

// ---- rows: thread q < D / 4 owns columns 4q .. 4q + 3
//
// this thread's columns of a gain, asked for before what the norm waits for
__device__ __forceinline__ float4 ds_gain(const DsArgs &a, const float *gamma)
{
    const int n = 4 * threadIdx.x;
    return n < a.D ? __ldg(reinterpret_cast<const float4 *>(gamma + n)) : make_float4(0.f, 0.f, 0.f, 0.f);
}
// bf16 values in fp32 -> the normed bf16 row (and, for the router, the same values as fp32 in xrow).  Every thread of the
// CTA takes part.
__device__ __forceinline__ void ds_norm_store(const DsArgs &a, Shared &sh, const float4 x, const float4 gm, bf16 *dst, float *xrow)
{
    const int n = 4 * threadIdx.x;
    float ss = n < a.D ? x.x * x.x + x.y * x.y + x.z * x.z + x.w * x.w : 0.0f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if ((threadIdx.x & 31) == 0) sh.red[threadIdx.x >> 5] = ss;
    __syncthreads();
    float tot = 0.0f;
#pragma unroll
    for (int w = 0; w < 8; w++) tot += sh.red[w];         // D / 4 <= 256 threads: the warps beyond add nothing
    const float rinv = 1.0f / sqrtf(tot / (float)a.D + 1e-5f);
    if (n < a.D) {
        const float4 o = ds_bf4(make_float4(x.x * rinv * gm.x, x.y * rinv * gm.y, x.z * rinv * gm.z, x.w * rinv * gm.w));
        ds_putrow(dst + n, o);
        if (xrow) *reinterpret_cast<float4 *>(xrow + n) = o;
    }
}

// the CTA's items: one as a rule, whose first keys and values were asked for at the layer's start
__device__ __forceinline__ void ds_attention(const DsArgs &a, Shared &sh, const DsLayer &ly, uint8_t *kvs, uint8_t *slot)
{
    const int n = a.B * a.H;
#pragma unroll 1
    for (int item = blockIdx.x; item < n; item += gridDim.x) {
        if (item != (int)blockIdx.x) {
            __syncthreads();
            if (threadIdx.x == 0) ds_item(a, sh, item);
            __syncthreads();
            ds_kv_request(a, sh, ly, kvs, 0);
        }
        ds_attention_item(a, sh, ly, kvs, slot);
    }
    if ((int)(blockIdx.x + gridDim.x) < n) {              // back to the first one, for the next layer
        __syncthreads();
        if (threadIdx.x == 0) ds_item(a, sh, blockIdx.x);
    }
}

// The rows' owners are the last CTAs, which have no attention item with few slots: what they need besides sums (the
// router's matrix) waits in shared memory since the layer's start then, since the attention's end else.
__device__ __forceinline__ int ds_row(const DsArgs &a) { const int b = (int)gridDim.x - 1 - (int)blockIdx.x; return b < a.B ? b : -1; }
__device__ __forceinline__ void ds_wr_request(const DsArgs &a, const DsLayer &ly, float *wr)
{
#pragma unroll 1
    for (int i = threadIdx.x * 4; i < a.D * a.E; i += DS_THREADS * 4) ds_cp16(ds_smem(wr + i), ly.wr + i);
    ds_commit();
}
// residual, norm, router of a row
__device__ __forceinline__ void ds_router(const DsArgs &a, Shared &sh, const DsLayer &ly, float *wr, float *xrow, uint8_t *slot)
{
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, b = ds_row(a);
    if (b < 0) return;
    const float4 gm = ds_gain(a, ly.an2);
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
    const int n = 4 * tid, ns = a.D / DS_ROWS;
    if (n < a.D) {
        uint4 p[DS_MAX_SL];
        float4 y = x;
        const float *pp = reinterpret_cast<const float *>(slot + a.po) + (size_t)b * a.D + n;
        ds_poll(a, [&] {
            uint32_t m = 0;
#pragma unroll
            for (int k = 0; k < DS_MAX_SL; k++) p[k] = k < ns ? ds_get4(pp + (size_t)k * a.B * a.D) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
            for (int k = 0; k < DS_MAX_SL; k++) m = max(m, ds_max4(p[k]));
            return m;
        });
#pragma unroll
        for (int k = 0; k < DS_MAX_SL; k++) ds_add4(y, ds_float4(p[k]));
        x = *reinterpret_cast<const float4 *>(sh.x + n);
        ds_add4(x, ds_bf4(y));
        x = ds_bf4(x);
        *reinterpret_cast<float4 *>(sh.x + n) = x;
    }
    ds_norm_store(a, sh, x, gm, reinterpret_cast<bf16 *>(slot + a.fnorm) + (size_t)b * a.D, xrow);
    ds_wait<0>();
    __syncthreads();
    const int per = a.D / DS_WARPS, j0 = warp * per;      // a multiple of eight
    float acc = 0.0f;
    if (lane < a.E) {
        const float *wp = wr + j0 * a.E + lane;
#pragma unroll 2
        for (int j = j0; j < j0 + per; j += 8) {
            const float4 x0 = *reinterpret_cast<const float4 *>(xrow + j), x1 = *reinterpret_cast<const float4 *>(xrow + j + 4);
            float w[8];
#pragma unroll
            for (int u = 0; u < 8; u++) { w[u] = *wp; wp += a.E; }
            acc = __fmaf_rn(x0.x, w[0], acc); acc = __fmaf_rn(x0.y, w[1], acc); acc = __fmaf_rn(x0.z, w[2], acc); acc = __fmaf_rn(x0.w, w[3], acc);
            acc = __fmaf_rn(x1.x, w[4], acc); acc = __fmaf_rn(x1.y, w[5], acc); acc = __fmaf_rn(x1.z, w[6], acc); acc = __fmaf_rn(x1.w, w[7], acc);
        }
    }
    sh.logit[warp * 32 + lane] = acc;
    __syncthreads();
    if (warp == 0) {
        float lg = 0.0f;
        if (lane < a.E) {
#pragma unroll
            for (int w = 0; w < DS_WARPS; w++) lg += sh.logit[w * 32 + lane];
            ly.rt[(size_t)b * a.E + lane] = lg;
        }
        int *asg = reinterpret_cast<int *>(slot + a.asg);
        router_topk_row(lg, b, lane, ly.rprobs, ly.assign, ly.gate, a.B, a.E, a.K, nullptr, 0, 
                        [&](int k, int pick, float g) { ds_put((void *)(asg + k * a.B + b), (uint32_t)pick); sh.gate[k] = g; });
    }
}

// the step's distinct experts and the slots k * B + b of each (in order of first use, 32 slots at a time), and the rows that
// they take
__device__ __forceinline__ void ds_experts(const DsArgs &a, Shared &sh, bf16 *fn, const uint8_t *slot, bool many)
{
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x, R = a.K * a.B;
        int first = 0;
#pragma unroll 1
        for (int h = 0; h < (many && R > 32 ? 2 : 1); h++) {
            int e = -1;
            if (h * 32 + lane < R) {
                const int *p = reinterpret_cast<const int *>(slot + a.asg) + h * 32 + lane;
                ds_poll(a, [&] { e = (int)ds_get(p); return (uint32_t)e; });
                if ((unsigned)e >= (unsigned)a.E) e = 0;
            }
            __syncwarp();
            const unsigned m = __match_any_sync(0xffffffffu, e), lt = (1u << lane) - 1u;
            const unsigned lead = __ballot_sync(0xffffffffu, e >= 0 && (m & lt) == 0u);
            if ((lead >> lane) & 1u) { const int i = first + __popc(lead & lt); sh.pexp[i] = e | h << 8; sh.pmask[i] = m; }
            first += __popc(lead);
        }
        if (lane == 0) sh.npair = first;
    }
    for (int i = DS_THREADS - 1 - (int)threadIdx.x; i < a.B * a.D / 8; i += DS_THREADS) {          // (warp 0, which is late, last)
        uint4 v;
        ds_poll(a, [&] { v = ds_get4(slot + a.fnorm + (size_t)i * 16); return ds_max4(v); });
        *reinterpret_cast<uint4 *>(fn + (size_t)i * 8) = v;
    }
    __syncthreads();
}

// gate-weighted combination, residual, the next norm of a row
__device__ __forceinline__ void ds_combine(const DsArgs &a, Shared &sh, float *ys, int l, uint8_t *slot)
{
    const int b = ds_row(a);
    if (b < 0) return;
    const int c = 4 * threadIdx.x;
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
    if (c < a.D) x = *reinterpret_cast<const float4 *>(sh.x + c);
    const float4 gm = ds_gain(a, l + 1 < a.L ? sh.layer[(l + 1) & 1].an1 : a.nf);
    const int half = threadIdx.x >> 8, n = 4 * (threadIdx.x & 255), R = a.K * a.B, ns = a.F / DS_ROWS;
    if (n < a.D) {
#pragma unroll 1
        for (int k = half; k < a.K; k += 2) {
            const float *p = reinterpret_cast<const float *>(slot + a.pd) + (size_t)(k * a.B + b) * a.D + n;
            float4 y = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
            for (int s0 = 0; s0 < ns; s0 += 12) {         // twelve slices in flight: d_ff 1536 in one go
                uint4 v[12];
                ds_poll(a, [&] {
                    uint32_t m = 0;
#pragma unroll
                    for (int s = 0; s < 12; s++) v[s] = s0 + s < ns ? ds_get4(p + (size_t)(s0 + s) * R * a.D) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
                    for (int s = 0; s < 12; s++) m = max(m, ds_max4(v[s]));
                    return m;
                });
#pragma unroll
                for (int s = 0; s < 12; s++) ds_add4(y, ds_float4(v[s]));
            }
            *reinterpret_cast<float4 *>(ys + k * a.D + n) = ds_bf4(y);
        }
    }
    __syncthreads();
    if (c < a.D) {
#pragma unroll 1
        for (int k = 0; k < a.K; k++) ds_fma4(x, sh.gate[k], *reinterpret_cast<const float4 *>(ys + k * a.D + c));
        x = ds_bf4(x);
        *reinterpret_cast<float4 *>(sh.x + c) = x;
    }
    ds_norm_store(a, sh, x, gm, (l + 1 < a.L ? reinterpret_cast<bf16 *>(slot) : a.fn) + (size_t)b * a.D, nullptr);
}

// C rows per task of the dense phases; MULTI: an expert can have more than one slot; MANY: a CTA more than one attention
// item, or an item and a row, and more than 32 routed slots (its loops cost the others 1 %)
template <int C, bool MULTI, bool MANY>
__global__ void __launch_bounds__(DS_THREADS, 1) k_dec_step(const __grid_constant__ DsArgs a)
{
    extern __shared__ __align__(128) uint8_t dsm[];
    __shared__ Shared sh;
    float *red = reinterpret_cast<float *>(dsm), *wr = reinterpret_cast<float *>(dsm + DS_RED), *xs = reinterpret_cast<float *>(dsm + DS_RED + DS_WR + DS_FN);
    bf16 *fn = reinterpret_cast<bf16 *>(dsm + DS_RED + DS_DEPTH * DS_SLOT);
    const bool attends = (int)blockIdx.x < a.B * a.H, owns = ds_row(a) >= 0;
    auto load_layer = [&](int l) {
        if (threadIdx.x < DS_LAYER_WORDS)
            reinterpret_cast<unsigned long long *>(&sh.layer[l & 1])[threadIdx.x] = __ldg(reinterpret_cast<const unsigned long long *>(a.layers + l) + threadIdx.x);
    };
    load_layer(0);
    if (threadIdx.x == 0) ds_item(a, sh, blockIdx.x);
    if (threadIdx.x < DS_MAX_R) sh.srow[threadIdx.x] = (int)threadIdx.x % a.B;
    if (threadIdx.x < DS_MAX_B) sh.pos[threadIdx.x] = (int)threadIdx.x < a.B ? __ldg(a.pos + threadIdx.x) : 0;
    // Every CTA looks the whole table over (2 KB from L2, beside the loads above): a pointer that is missing or not aligned
    // for its loads is reported, and the whole grid leaves before its first barrier.
    int bad = 0;
    for (int i = threadIdx.x; i < a.L * DS_LAYER_WORDS; i += DS_THREADS) {
        const unsigned long long p = __ldg(reinterpret_cast<const unsigned long long *>(a.layers) + i);
        if (!p || (p & ds_align_mask(i % DS_LAYER_WORDS))) bad = 1 + i;
    }
    if (bad && blockIdx.x == 0) report_bad_index(a.errword, 304, (bad - 1) / DS_LAYER_WORDS, (bad - 1) % DS_LAYER_WORDS);
    if (__syncthreads_or(bad)) return;
    const unsigned shape0 = 1u + (unsigned)(a.B | a.D / 128 << 6 | a.KD / 64 << 10 | a.K << 15), shape1 = (unsigned)a.F;   // never 0; the last CTA writes them
    const unsigned next = __ldcg(a.bar + 3);
    unsigned gate = 0;                                    // arrivals that the next wait for the grid needs
    if (__ldcg(a.bar + 4) != shape0 || __ldcg(a.bar + 5) != shape1) {
        ds_clear(a.slots, 3 * a.slot_bytes);
        gate += gridDim.x;
        __syncthreads();
        if (threadIdx.x == 0) { gb_arrive(a); gb_wait(a, gate); }
        __syncthreads();
    }
    // slots of the layer before, this one and the one after
    uint8_t *prev = a.slots + (next == 0 ? 2u : next - 1u) * a.slot_bytes, *cur = a.slots + next * a.slot_bytes, *after = a.slots + (next == 2 ? 0u : next + 1u) * a.slot_bytes;
    if (owns) {                                           // embedding row and the first norm
        const int b = ds_row(a), n = 4 * threadIdx.x;
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (n < a.D) {
            x = ds_bf4(__ldg(reinterpret_cast<const float4 *>(a.emb + (size_t)__ldg(a.tok + b) * a.D + n)));
            *reinterpret_cast<float4 *>(sh.x + n) = x;
        }
        ds_norm_store(a, sh, x, ds_gain(a, sh.layer[0].an1), reinterpret_cast<bf16 *>(prev) + (size_t)b * a.D, nullptr);
    }
#pragma unroll 1
    for (int l = 0; l < a.L; l++) {
        const DsLayer &ly = sh.layer[l & 1];
        __syncthreads();
        if (l + 1 < a.L) load_layer(l + 1);               // every thread is past the layer before: the other half is free
        if (attends) ds_kv_request(a, sh, ly, dsm + DS_RED, 0);
        else if (owns) ds_wr_request(a, ly, wr);
        if (l > 0) {                                      // (every path to a store or a poll of this layer's slot has a barrier of the CTA on it)
            gate += gridDim.x;
            if (threadIdx.x == DS_THREADS - 1) gb_wait(a, gate);
        }
        // The two dense phases and the two of the experts are one body of code each with several slots: with a body of
        // their own, 122 KB of instructions went through the instruction cache every layer (eight slots 433 us, 418 so).
        // With one slot, where less code is run, the body of their own is the faster one (204 and 199 us).
        constexpr int TWICE = MULTI ? 1 : 2;
#pragma unroll TWICE
        for (int wo = 0; wo < 2; wo++) {
            ds_dense<C>(a, ly, red, wo, wo ? cur + a.att : prev, cur);
            __syncthreads();
            if (wo) break;
            ds_clear(after, a.slot_bytes);
            if (MANY) ds_attention(a, sh, ly, dsm + DS_RED, cur);
            else if (attends) ds_attention_item(a, sh, ly, dsm + DS_RED, cur);
            __syncthreads();
            if (MANY && attends && owns) ds_wr_request(a, ly, wr);
        }
        if (l + 1 < a.L && threadIdx.x == DS_THREADS - 1) gb_arrive(a);
        ds_router(a, sh, ly, wr, red, cur);
        __syncthreads();
        ds_experts(a, sh, fn, cur, MANY);
#pragma unroll TWICE
        for (int down = 0; down < 2; down++) {
            ds_experts_phase(a, sh, down, ly, red, xs, fn, dsm + DS_RED, MULTI, MANY, cur);
            __syncthreads();
        }
        ds_combine(a, sh, red, l, cur);
        uint8_t *p = prev;
        prev = cur; cur = after; after = p;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(a.bar + 1, 1u) == gridDim.x - 1) {
            a.bar[3] = (next + (unsigned)a.L) % 3u;
            a.bar[4] = *(volatile unsigned *)(a.bar + 2) ? 0u : shape0;      // after an abort the slots hold anything
            a.bar[5] = shape1;
            a.bar[0] = 0u; a.bar[1] = 0u; a.bar[2] = 0u;
            __threadfence();
        }
    }
}

struct DsLayout { size_t att, fnorm, asg, pq, po, pg, pd, slot, bytes; };
static DsLayout ds_layout(int B, int D, int KD, int F, int K)
{
    DsLayout w;
    size_t cur = 0;
    auto take = [&](size_t n) { const size_t at = cur; cur += (n + 255) & ~(size_t)255; return at; };
    const size_t b = B, d = D, r = (size_t)K * B, sd = D / DS_ROWS, sf = F / DS_ROWS;
    take(b * d * 2);                                      // xn
    w.att = take(b * d * 2); w.fnorm = take(b * d * 2); w.asg = take(r * 4);
    w.pq = take(sd * b * (d + 2 * (size_t)KD) * 4);       // slice sums: [D/128][B][NQ], [D/128][B][D], [D/128][2 R][F], [F/128][R][D]
    w.po = take(sd * b * d * 4);
    w.pg = take(sd * 2 * r * F * 4);
    w.pd = take(sf * r * d * 4);
    w.slot = cur;
    w.bytes = 256 + 3 * cur;
    return w;
}
// Above eight slots (six layers, us a step, this form and the chain): nine slots of D 768, 32 experts of 1536, two choices
// 243 and 361, sixteen 340 and 394 (380 and 485 with 900 cached positions); sixteen of D 256, eight experts of 512 140 and
// 238; 32 slots of D 256 with one choice of 32 or eight experts 180 and 293, 178 and 286.  With experts of many slots the
// chain takes sixteen of an expert's rows to the tensor cores at a time, a pass here two: up to four slots per expert, and
// up to 50 M products a matrix of all slots (four layers, twelve slots of D 1024, eight experts top-2: d_ff 2048, 50 M, 253
// and 278; d_ff 4096, 100 M, 367 and 301).  Above 32 routed slots up to 38 M: 24 slots of D 512, 16 experts top-2 of 1536
// (38 M) 325 and 333, 32 of D 256, 16 experts of 512 165 and 289; 20 of D 640, 32 experts of 1536 (39 M) 394 and 384.
// Up to eight slots there is no such limit; one would lie at about 80 M products with more than sixteen routed slots, which the
// chain takes in groups, and none below (three layers, eight slots of D 1024, eight experts, this form and the chain: two choices,
// d_ff 4096 234 and 363, 8192 361 and 497; four choices, 2048 218 and 240, 3072 277 and 248, 4096 326 and 259, 8192 551 and 315).
// Long caches speak for this form at any number of slots, although a CTA walks one slot and head on its own: 4000 positions, three
// layers, nine slots of D 768 210 and 516, sixteen 326 and 576, 32 of D 384 259 and 519.
static bool ds_fits(int B, int Tm, int D, int H, int KV, int F, int E, int K)
{
    return B >= 1 && B <= DS_MAX_B && Tm >= 1 && Tm <= 4096 && D == H * 64 && D % 128 == 0 && D <= 1024 && KV >= 1 && H % KV == 0 &&
           (KV * 64) % 128 == 0 && F >= 128 && F % 128 == 0 && E >= 1 && E <= 32 && K >= 1 && K <= E && K * B <= (B <= 8 ? 32 : DS_MAX_R) && K <= DS_WARPS && K * D * 4 <= DS_RED &&
           B * D <= DS_FN_ELEMS && (B <= 8 ? B * (H + 1) <= sm_count() : B <= sm_count() && K * B <= 4 * E && (size_t)K * B * D * F <= (size_t)(K * B <= 32 ? 48 : 36) << 20);
}

}  // namespace qlmb

using namespace qlmb;

extern "C" size_t qlmb_dec_step_bytes(int B, int Tm, int D, int H, int KV, int F, int E, int K)
{
    return ds_fits(B, Tm, D, H, KV, F, E, K) ? ds_layout(B, D, KV * 64, F, K).bytes : 0;
}

extern "C" int qlmb_dec_step(const qlmb_dec_step_args *p, void *stream)
{
    QLMB_REQUIRE(p && p->layers && p->emb && p->tok && p->pos && p->cosb && p->sinb && p->nf && p->fn && p->ws, "qlmb_dec_step: NULL argument");
    QLMB_REQUIRE(p->L > 0, "qlmb_dec_step: L=%d", p->L);
    QLMB_REQUIRE((((uintptr_t)p->emb | (uintptr_t)p->nf | (uintptr_t)p->fn) & 15) == 0 && ((uintptr_t)p->layers & 7) == 0 &&
                 (((uintptr_t)p->tok | (uintptr_t)p->pos | (uintptr_t)p->cosb | (uintptr_t)p->sinb) & 3) == 0,
                 "qlmb_dec_step: emb, nf and fn must be 16-byte aligned, layers 8, tok, pos, cosb and sinb 4");
    QLMB_REQUIRE(((uintptr_t)p->ws & 255) == 0, "qlmb_dec_step: the workspace must be 256-byte aligned");
    if (!ds_fits(p->B, p->Tm, p->D, p->H, p->KV, p->F, p->E, p->K)) {
        set_error("qlmb_dec_step: shape B %d Tm %d D %d H %d KV %d F %d E %d K %d is not supported", p->B, p->Tm, p->D, p->H, p->KV, p->F, p->E, p->K);
        return QLMB_E_UNSUPPORTED;
    }
    const DsLayout w = ds_layout(p->B, p->D, p->KV * 64, p->F, p->K);
    uint8_t *ws = (uint8_t *)p->ws;
    DsArgs a = {};
    a.layers = (const DsLayer *)p->layers;
    a.L = p->L; a.B = p->B; a.D = p->D; a.KD = p->KV * 64; a.H = p->H; a.KV = p->KV; a.F = p->F; a.E = p->E; a.K = p->K; a.Tm = p->Tm;
    auto recip = [](int n) { return (uint32_t)((0x100000000ull + n - 1) / n); };       // exact quotients for the task numbers that occur
    a.tq = (a.D + 2 * a.KD + DS_COLS - 1) / DS_COLS; a.td = (a.D + DS_COLS - 1) / DS_COLS; a.tf = (a.F + DS_COLS - 1) / DS_COLS;
    a.mq = recip(a.tq); a.md = recip(a.td); a.mf = recip(a.tf); a.mr = recip(a.D / DS_ROWS); a.mfs = recip(a.F / DS_ROWS);
    a.emb = p->emb; a.tok = p->tok; a.pos = p->pos; a.cosb = p->cosb; a.sinb = p->sinb; a.nf = p->nf; a.fn = (bf16 *)p->fn;
    a.bar = (unsigned *)ws;
    a.slots = ws + 256; a.slot_bytes = w.slot;
    a.att = w.att; a.fnorm = w.fnorm; a.asg = w.asg; a.pq = w.pq; a.po = w.po; a.pg = w.pg; a.pd = w.pd;
    a.errword = device_error_word();
    // rows per task of the dense phases: the fewest with which the q, k, v tasks are one round of the device
    int c = 1;
    while (c < 4 && a.tq * (a.D / DS_ROWS) * ((p->B + c - 1) / c) > sm_count()) c *= 2;
    const void *kerns[7] = {(const void *)k_dec_step<1, false, false>, (const void *)k_dec_step<1, true, false>, (const void *)k_dec_step<2, true, false>,
                            (const void *)k_dec_step<4, true, false>, (const void *)k_dec_step<1, true, true>, (const void *)k_dec_step<2, true, true>,
                            (const void *)k_dec_step<4, true, true>};
    const int v = p->B == 1 ? 0 : (c == 1 ? 1 : c == 2 ? 2 : 3) + (p->B > 8 ? 3 : 0);
    const void *kern = kerns[v];
    int dev = 0;
    QLMB_CUDA(cudaGetDevice(&dev));
    QLMB_REQUIRE(dev >= 0 && dev < 64, "device index %d", dev);
    static bool attr_done[64][7];
    if (!attr_done[dev][v]) {
        QLMB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, DS_SMEM));
        attr_done[dev][v] = true;
    }
    void *args[] = {&a};
    QLMB_CUDA(cudaLaunchCooperativeKernel(kern, dim3((unsigned)sm_count()), dim3(DS_THREADS), args, (size_t)DS_SMEM, as_stream(stream)));
    QLMB_LAUNCH_CHECK("k_dec_step");
    return QLMB_OK;
}
