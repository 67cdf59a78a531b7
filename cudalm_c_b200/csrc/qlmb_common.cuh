// Shared declarations for libqlm_b200: status handling, span lookup, nibble
// access and the rounding hash.  Device code here is integer-only, so it is
// safe to include from translation units built with or without --fmad=false.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <stdarg.h>
#include "../../include/qlm_b200.h"

namespace qlmb {

// ---- host-side status ------------------------------------------------------
void set_error(const char *fmt, ...);
int cuda_fail(cudaError_t e, const char *what);          // records + returns QLMB_E_CUDA
int *device_error_word(void);                            // per-device int, lazily allocated
#define QLMB_CUDA(call)                                                        \
    do {                                                                       \
        cudaError_t e__ = (call);                                              \
        if (e__ != cudaSuccess) return qlmb::cuda_fail(e__, #call);            \
    } while (0)
#define QLMB_REQUIRE(cond, ...)                                                \
    do {                                                                       \
        if (!(cond)) { qlmb::set_error(__VA_ARGS__); return QLMB_E_ARG; }      \
    } while (0)
#define QLMB_LAUNCH_CHECK(what)                                                \
    do {                                                                       \
        cudaError_t e__ = cudaGetLastError();                                  \
        if (e__ != cudaSuccess) return qlmb::cuda_fail(e__, what);             \
    } while (0)

static inline cudaStream_t as_stream(void *s) { return (cudaStream_t)s; }
int sm_count(void);                                      // SMs of the current device
// second stream of the device for overlappable work (qlmb_runtime.cu); returns `st` itself when unavailable
cudaStream_t side_fork(cudaStream_t st, int which = 0);   // two side streams per device: which = 0 or 1
void side_wait_main(cudaStream_t side, cudaStream_t st);
void side_join(cudaStream_t side, cudaStream_t st);
// Times the enclosed launches with CUDA events when qlmb_prof_enable(1) was called.
struct ProfScope {
    int slot; cudaStream_t stream;
    ProfScope(const char *name, cudaStream_t st);
    ~ProfScope();
};

// ---- programmatic dependent launch ----------------------------------------
// A kernel launched with pdl_launch may start while the kernel before it in the stream is still running: its blocks
// are scheduled as soon as every block of that kernel has called pdl_trigger() (or exited), and run up to their
// pdl_wait(), which returns once that kernel has completed and its writes are visible.  Rules kept by every such kernel:
// every block executes pdl_wait() exactly once, before its first write, before any early return, and before it loads
// anything that a kernel may write: activations, but the weights too (codes, scales, gains, the router matrix, the
// embedding), for the kernel in front may be an optimizer's.  That a writer does not trigger is not enough: its successor
// then starts when its blocks are done, but sees its stores only behind the wait.  Only where `weights_quiet` answers
// QUIET, no writer of weights being able to run or to be unseen, are they loaded ahead of it.  (Prefetches into L2 ahead of
// the wait, which would be allowed, cost more than they gain: a streaming GEMV of 4096 x 16384 14.3 -> 15 us.)
// The caller decides per launch (`early`): with one to four rows per step the early blocks of the decode chain cost the
// running kernel more than they gain (decode step 0.53 -> 0.56 ms at one slot, 0.85 -> 0.81 ms at eight, CUDA events).
// The tensor-core kernels set up their barriers and TMEM, the others do nothing ahead of the wait: what they save is the
// gap between two launches of a stream.
// QLMB_PDL=0 turns the attribute off everywhere (the instructions are then no-ops).
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// What a kernel reads behind its wait it reads with ordinary loads: __ldg and the like promise that nothing writes the data
// while the kernel runs, which does not hold for a kernel that starts before its predecessor's end, and the compiler may
// move them over the wait.  What it reads ahead of the wait passes by L1, which nothing has emptied since the writer.
__device__ __forceinline__ float ld_cg(const float *p)   // stays where it is written
{ float v; asm volatile("ld.global.cg.f32 %0, [%1];" : "=f"(v) : "l"(__cvta_generic_to_global(p)) : "memory"); return v; }
// Between qlmb_quiet_begin(st) and qlmb_quiet_end() the calling thread launches nothing on `st` that writes weights or
// float parameters.  The first launch that asks inside such a scope gets QUIET_FIRST and waits before it triggers, so
// every writer queued before the scope has ended, and its stores are visible, before a later launch of the scope, which
// gets QUIET, can start.  Outside a scope the answer is 0.
enum { QUIET_FIRST = 1, QUIET = 2 };
int weights_quiet(cudaStream_t st);
bool pdl_enabled(void);                                  // qlmb_runtime.cu
template <typename... KArgs, typename... Args>
static inline cudaError_t pdl_launch(bool early, void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at; cfg.numAttrs = (early && pdl_enabled()) ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, KArgs(args)...);
}
// Early blocks gain the gap between two launches (about 1.5 us) but hold their SM while they wait.  Where other streams
// have work for that SM (an expert layer's backward: 678 -> 700 us with every launch early) or a kernel has several waves
// of blocks beside a small successor (attention of 8 x 1024 x 12 heads 257 -> 267 us) they cost more than they gain: the
// former launches are never early, the latter only with up to two blocks per SM.  Nor does a launch of few long blocks start
// early: beside the last blocks of its predecessor they are placed where there is room, several to an SM, and stay there
// (router logits of 4737 tokens in tiles, behind a kernel that lets them start: 24 -> 63 us).
template <typename... KArgs, typename... Args>
static inline cudaError_t pdl_launch_small(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args... args)
{
    return pdl_launch((size_t)grid.x * grid.y * grid.z <= (size_t)2 * sm_count(), kern, grid, block, smem, st, args...);
}

// ---- device helpers --------------------------------------------------------
// splitmix64 finaliser, low 32 bits (reference qlm.cuh:78-82).
__host__ __device__ __forceinline__ uint32_t hash_u32(uint64_t x)
{
    x += 0x9E3779B97F4A7C15ULL;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ULL;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBULL;
    return (uint32_t)(x ^ (x >> 31));
}
#define QLMB_HASH_I 0x2545F4914F6CDD1DULL   // element-index multiplier (qlm.cuh:85)
#define QLMB_HASH_T 0x9E3779B97F4A7C15ULL   // step multiplier

__host__ __device__ __forceinline__ int clampi(int v, int lo, int hi)
{
    return v < lo ? lo : (v > hi ? hi : v);
}

// A kernel that finds an argument it must not act on (a cache position outside the cache) records code 201 with the
// site, the slot and the value in the device error word and skips the access; qlmb_check_device reports it.
__device__ __forceinline__ void report_bad_index(int *errword, int site, int slot, int value)
{
    if (errword && atomicCAS(errword, 0, 201) == 0) { errword[1] = site; errword[2] = slot; errword[3] = value; }
}

// digit i of a digit array (qlm.cuh:96-101)
__device__ __forceinline__ int digit_at(const int8_t *d, uint64_t i, int packed)
{
    if (!packed) return d[i];
    unsigned b = (uint8_t)d[i >> 1];
    int v = (i & 1) ? (int)(b >> 4) : (int)(b & 15u);
    return v > 7 ? v - 16 : v;
}

// span that owns group gi (qlm.cuh:113-117): returns index, fills start/len
__device__ __forceinline__ int locate_group(const qlmb_span *sp, int nspan, int gi, int group,
                                            uint64_t &j0, int &n)
{
    // spans are appended in ascending group order (qlm_add_span, qlm.cuh:448-455): bisect for the last
    // span that starts at or before gi; a table that is not ascending falls back to the linear scan
    int lo = 0, hi = nspan - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if ((int)sp[mid].gi0 <= gi) lo = mid; else hi = mid - 1;
    }
    int si = lo;
    if (!(gi >= sp[si].gi0 && gi < sp[si].gi0 + sp[si].ngrp)) {
        si = 0;
        for (int i = 0; i < nspan; i++)
            if (gi >= sp[i].gi0 && gi < sp[i].gi0 + sp[i].ngrp) { si = i; break; }
    }
    j0 = (uint64_t)(gi - sp[si].gi0) * (uint64_t)group;
    uint64_t left = sp[si].n - j0;
    n = (int)(left < (uint64_t)group ? left : (uint64_t)group);
    return si;
}

}  // namespace qlmb
