// Router selection of one token by one warp, shared by the routing kernels and the decode step.  Include only from
// translation units built with --fmad=false: probabilities and choices match the reference's CPU build bit for bit.
#pragma once
#include <stdint.h>

namespace qlmb {

// exp as the reference CPU build computes it (cpu_kern.h:28-34): clamp,
// two-part ln2 reduction, degree-6 polynomial, exponent by bit shift.
__device__ __forceinline__ float exp_poly(float x)
{
    x = x < -87.0f ? -87.0f : (x > 88.0f ? 88.0f : x);
    float k = rintf(x * 1.44269504089f);
    float r = x - k * 0.693145751953125f;
    r -= k * 1.428606765330187e-06f;
    float p = 1.0f / 720;
    p = 1.0f / 120 + r * p;
    p = 1.0f / 24 + r * p;
    p = 1.0f / 6 + r * p;
    p = 0.5f + r * p;
    p = 1.0f + r * p;
    p = 1.0f + r * p;
    return p * __uint_as_float((uint32_t)((int)k + 127) << 23);
}

// One warp per token, lane = expert (E <= 32), with the arithmetic of the reference's CPU kernel (cpu_kern.h:413-425): the
// maximum is order-free, the softmax sum is taken in expert order (every lane adds the 32 shuffled terms one after the
// other) and the K selection rounds are warp maxima of an order-preserving integer, with the lowest index winning ties.
//
// unsigned integers in the order of the floats (never 0 for a number above -1e30); -0 counts as +0
__device__ __forceinline__ unsigned order_key(float f)
{
    const unsigned u = __float_as_uint(f + 0.0f);
    return (u & 0x80000000u) ? ~u : u | 0x80000000u;
}
// the softmax and the K selection rounds of token n by one warp; lg = the logit of expert `lane` (0 beyond E).  Lane 0
// hands every round's choice and its gate to tell() besides.
struct TellNobody { __device__ void operator()(int, int, float) const {} };
template <typename Tell = TellNobody>
__device__ __forceinline__ void router_topk_row(float lg, int n, int lane, float *rprobs, int *assign, float *gate, int N,
                                                int E, int K, const float *bias, int bs, Tell tell = Tell())
{
    const bool live = lane < E;
    float top = (live && lg > -1e30f) ? lg : -1e30f;
    const unsigned tk = __reduce_max_sync(0xffffffffu, order_key(top));
    top = __uint_as_float((tk & 0x80000000u) ? tk ^ 0x80000000u : ~tk);
    float p = live ? exp_poly(lg - top) : 0.0f;
    float sum = 0.0f;
#pragma unroll
    for (int e = 0; e < 32; e++) sum += __shfl_sync(0xffffffffu, p, e);             // lanes past E add an exact zero
    float inv = 1.0f / sum;
    float pr = p * inv;
    if (live) rprobs[(size_t)n * E + lane] = pr;
    bool taken = false;
#pragma unroll 1
    for (int k = 0; k < K; k++) {
        const float sc = pr + (bias && live ? bias[k * bs + lane] : 0.0f);
        const unsigned key = live && !taken && (sc > -1e30f) ? order_key(sc) : 0u;
        const unsigned best = __reduce_max_sync(0xffffffffu, key);
        const int pick = best ? __ffs(__ballot_sync(0xffffffffu, key == best)) - 1 : k;    // lowest index on ties; NaN scores: stay in range
        float g = __shfl_sync(0xffffffffu, pr, pick);
        if (lane == 0) { assign[(size_t)k * N + n] = pick; gate[(size_t)k * N + n] = g; tell(k, pick, g); }
        taken = taken || (lane == pick);
    }
}

}  // namespace qlmb
