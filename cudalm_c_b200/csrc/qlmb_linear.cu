// Quantised linear entry points (the reference's g_ab / g_abt / g_abt_b / g_atb
// call sites, cudalm.cu:3133-3202) on top of the tcgen05 GEMM engine.
#include <mutex>
#include "qlmb_common.cuh"
#include "qlmb_gemm.cuh"

namespace qlmb {

// per-device scratch for the bf16 copies of fp32 operands, grown on demand
static void *g_ws[64];
static size_t g_ws_cap[64];
int workspace(size_t bytes, void **out)
{
    int dev = 0;
    QLMB_CUDA(cudaGetDevice(&dev));
    QLMB_REQUIRE(dev >= 0 && dev < 64, "workspace: device index %d", dev);
    if (g_ws_cap[dev] < bytes) {
        if (g_ws[dev]) { QLMB_CUDA(cudaDeviceSynchronize()); QLMB_CUDA(cudaFree(g_ws[dev])); }
        g_ws[dev] = nullptr; g_ws_cap[dev] = 0;
        size_t cap = (bytes + ((size_t)1 << 20) - 1) & ~(((size_t)1 << 20) - 1);
        QLMB_CUDA(cudaMalloc(&g_ws[dev], cap));
        g_ws_cap[dev] = cap;
    }
    *out = g_ws[dev];
    return QLMB_OK;
}

// Scratch of one call, in stream order: calls on several streams and threads get memory of their own, under capture it
// belongs to the graph, and nothing that a captured call uses is ever replaced by a larger piece (the shared piece above
// is).  A pool per device keeps up to SCRATCH_KEPT between calls and gives the rest back at the next synchronisation.
constexpr size_t SCRATCH_KEPT = (size_t)128 << 20;
struct StreamScratch {
    void *p = nullptr;
    cudaStream_t st;
    explicit StreamScratch(cudaStream_t s) : st(s) {}
    bool get(size_t bytes)
    {
        static std::mutex mu;
        static cudaMemPool_t pools[64];
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
        {
            std::lock_guard<std::mutex> lock(mu);
            if (!pools[dev]) {
                cudaMemPoolProps props = {};
                props.allocType = cudaMemAllocationTypePinned;
                props.location.type = cudaMemLocationTypeDevice; props.location.id = dev;
                uint64_t keep = SCRATCH_KEPT;
                if (cudaMemPoolCreate(&pools[dev], &props) != cudaSuccess) { pools[dev] = nullptr; cudaGetLastError(); return false; }
                cudaMemPoolSetAttribute(pools[dev], cudaMemPoolAttrReleaseThreshold, &keep);
            }
        }
        if (cudaMallocFromPoolAsync(&p, bytes, pools[dev], st) != cudaSuccess) { p = nullptr; cudaGetLastError(); return false; }
        return true;
    }
    ~StreamScratch() { if (p) cudaFreeAsync(p, st); }
};

// bf16 view of an activation matrix: the matrix itself, or a converted copy in `slot`
static int as_bf16(const void *x, int dtype, size_t n, bf16 *slot, const bf16 **out, cudaStream_t st)
{
    if (dtype == QLMB_BF16) { *out = (const bf16 *)x; return QLMB_OK; }
    int rc = convert_f32_to_bf16(slot, (const float *)x, n, st);
    *out = slot;
    return rc;
}

static int check_linear(const char *who, int layout, int M, int K, int N, int dtype)
{
    QLMB_REQUIRE(layout == QLMB_KN || layout == QLMB_NK, "%s: layout %d", who, layout);
    QLMB_REQUIRE(dtype == QLMB_F32 || dtype == QLMB_BF16, "%s: dtype %d", who, dtype);
    QLMB_REQUIRE(M >= 0 && K > 0 && N > 0, "%s: M=%d K=%d N=%d", who, M, K, N);
    if ((K % 128) || (N % 128)) {
        set_error("%s: K=%d and N=%d must be multiples of the 128-element scale group", who, K, N);
        return QLMB_E_UNSUPPORTED;
    }
    return QLMB_OK;
}

// dW = beta * dW + part[0] + part[1] + ... in ascending slice order; n is a multiple of 4; a row of the grid per matrix
struct SumMats { float *dW[3]; };
template <bool MATS>
__global__ void __launch_bounds__(256) k_sum_slices(const SumMats m, const float *part, int S, size_t n, float beta)
{
    pdl_wait();
    pdl_trigger();
    const size_t i = ((size_t)blockIdx.x * 256 + threadIdx.x) * 4;
    if (i >= n) return;
    float *dW = m.dW[MATS ? blockIdx.y : 0];
    if (MATS) part += (size_t)blockIdx.y * S * n;
    float4 a = *reinterpret_cast<const float4 *>(part + i);
    for (int s = 1; s < S; s++) {
        const float4 b = *reinterpret_cast<const float4 *>(part + (size_t)s * n + i);
        a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
    }
    if (beta != 0.0f) {
        const float4 o = *reinterpret_cast<const float4 *>(dW + i);
        a.x += beta * o.x; a.y += beta * o.y; a.z += beta * o.z; a.w += beta * o.w;
    }
    *reinterpret_cast<float4 *>(dW + i) = a;
}

}  // namespace qlmb

using namespace qlmb;

extern "C" int qlmb_linear_fwd(void *Y, const void *X, const int8_t *codes, const float *scales, int layout,
                               int M, int K, int N, const void *R, int dtype, void *stream)
{
    int rc = check_linear("qlmb_linear_fwd", layout, M, K, N, dtype);
    if (rc) return rc;
    if (M == 0) return QLMB_OK;
    QLMB_REQUIRE(Y && X && codes && scales, "qlmb_linear_fwd: NULL argument");
    cudaStream_t st = as_stream(stream);
    void *ws = nullptr;
    if (dtype == QLMB_F32) { rc = workspace((size_t)M * K * 2, &ws); if (rc) return rc; }
    const bf16 *xb;
    rc = as_bf16(X, dtype, (size_t)M * K, (bf16 *)ws, &xb, st);
    if (rc) return rc;
    GemmLaunch g = {};
    g.bmode = layout == QLMB_KN ? B_DEQ_MN : B_DEQ_K;
    g.epi = EPI_STORE; g.sched = SCHED_DENSE;
    g.a[0] = xb; g.a_rows = M; g.a_cols = K;
    g.w[0] = codes; g.scales[0] = scales;
    g.w_rows = layout == QLMB_KN ? K : N; g.w_cols = layout == QLMB_KN ? N : K;
    g.nseg = 1; g.ksteps = K / 64; g.M = M; g.N = N; g.E = 1;
    g.out = Y; g.out_dtype = dtype; g.ldo = N; g.resid = R; g.beta = 0.0f;
    return gemm_launch(g, st);
}

extern "C" int qlmb_linear_dgrad(void *dX, const void *dY, const int8_t *codes, const float *scales, int layout,
                                 int M, int K, int N, float beta, int dtype, void *stream)
{
    QLMB_REQUIRE(beta == 0.0f || beta == 1.0f, "qlmb_linear_dgrad: beta %g", beta);
    int rc = check_linear("qlmb_linear_dgrad", layout, M, K, N, dtype);
    if (rc) return rc;
    if (M == 0) return QLMB_OK;
    QLMB_REQUIRE(dX && dY && codes && scales, "qlmb_linear_dgrad: NULL argument");
    cudaStream_t st = as_stream(stream);
    void *ws = nullptr;
    if (dtype == QLMB_F32) { rc = workspace((size_t)M * N * 2, &ws); if (rc) return rc; }
    const bf16 *gb;
    rc = as_bf16(dY, dtype, (size_t)M * N, (bf16 *)ws, &gb, st);
    if (rc) return rc;
    GemmLaunch g = {};
    // the contraction now runs over N: codes W[K][N] are K-major for it, W[N][K] MN-major
    g.bmode = layout == QLMB_KN ? B_DEQ_K : B_DEQ_MN;
    g.epi = EPI_STORE; g.sched = SCHED_DENSE;
    g.a[0] = gb; g.a_rows = M; g.a_cols = N;
    g.w[0] = codes; g.scales[0] = scales;
    g.w_rows = layout == QLMB_KN ? K : N; g.w_cols = layout == QLMB_KN ? N : K;
    g.nseg = 1; g.ksteps = N / 64; g.M = M; g.N = K; g.E = 1;
    g.out = dX; g.out_dtype = dtype; g.ldo = K; g.resid = nullptr; g.beta = beta;
    return gemm_launch(g, st);
}

// Row slices of one matrix's weight gradient [Md][Nd] over M rows
static int wgrad_slices(int Md, int Nd, int M)
{
    const int stages = (M + 63) / 64, tiles = ((Md + 255) / 256) * ((Nd + 255) / 256), pairs = sm_count() / 2;
    int S = 1;
    while (S < 16 && tiles * S * 2 <= pairs && stages / (2 * S) >= 8) S *= 2;
    return S;
}
static bool wgrad_even(int Md, int Nd, int M)             // ... cut into slices that are all as long
{
    const int S = wgrad_slices(Md, Nd, M);
    return S > 1 && M % (256 * S) == 0;
}

// The weight gradients of nmat matrices of one size on the same X: dW[i][K,N] = X^T dY[i] (KN) or dW[i][N,K] = dY[i]^T X (NK).
// A small weight matrix gives few output tiles (768 x 768: 9 tiles of 256 x 256 for 74 SM pairs) over a
// long contraction (the M rows).  Then the rows are cut into S slices that run as the "experts" of the
// grouped weight-gradient schedule, each into its own partial, and the partials are added in ascending
// slice order: every element still has one writer and a fixed order.
// A slice keeps at least eight stages of 64 rows; the rows past M that the last ones name are zeros to the copies.
// (Only row counts that divided evenly were cut before: 8191 rows of 384 x 640, forward and both gradients, 119 -> 39 us.)
static int wgrad_mats(float *const *dW, const void *const *dY, int nmat, int S, const void *X, int layout, int M, int K, int N,
                      float beta, int dtype, cudaStream_t st)
{
    const int Md = layout == QLMB_KN ? K : N, Nd = layout == QLMB_KN ? N : K, stages = (M + 63) / 64;
    const size_t conv = dtype == QLMB_F32 ? ((((size_t)M * K * 2 + 255) & ~(size_t)255) + (((size_t)M * N * 2 + 255) & ~(size_t)255)) : 0;
    // Rows that divide evenly keep their slices' partial sums in the shared piece, behind the converted operands: a step
    // that is captured after a first eager one finds it large enough, and an allocation and a free node for each of its
    // calls would cost 0.6 % of a training step.  Other row counts, which need no scratch uncut, take their own.
    // Evenly: into the slices of one matrix alone, also where several are made together in another number of slices.  Calls
    // whose single gradients have scratch of their own, or need none, may run on several streams at once and be replayed
    // from a graph after larger ones.
    const size_t part_bytes = S > 1 ? (size_t)nmat * S * Md * Nd * sizeof(float) : 0;
    const bool shared = S > 1 && wgrad_even(Md, Nd, M);
    StreamScratch own(st);
    if (S > 1 && !shared && !own.get(part_bytes)) S = 1;
    int rc = QLMB_OK;
    if (S == 1 && nmat > 1) {                            // no scratch: one by one
        for (int i = 0; i < nmat && !rc; i++) rc = wgrad_mats(dW + i, dY + i, 1, 1, X, layout, M, K, N, beta, dtype, st);
        return rc;
    }
    void *ws = nullptr;
    if (conv || shared) { rc = workspace(conv + (shared ? part_bytes : 0), &ws); if (rc) return rc; }
    float *part = shared ? (float *)((uint8_t *)ws + conv) : (float *)own.p;
    const bf16 *xb, *gb;
    bf16 *slot2 = conv ? (bf16 *)((uint8_t *)ws + (((size_t)M * K * 2 + 255) & ~(size_t)255)) : nullptr;
    rc = as_bf16(X, dtype, (size_t)M * K, (bf16 *)ws, &xb, st);
    if (rc) return rc;
    rc = as_bf16(dY[0], dtype, (size_t)M * N, slot2, &gb, st);
    if (rc) return rc;
    GemmLaunch g = {};
    g.bmode = AB_TMA_MN; g.epi = EPI_ACCUM; g.sched = SCHED_DENSE;
    g.a[0] = layout == QLMB_KN ? xb : gb; g.a_rows = M; g.a_cols = Md;
    g.w[0] = layout == QLMB_KN ? gb : xb; g.w_cols = Nd; g.w_rows = 0;
    if (S > 1) {
        for (int i = 1; i < nmat; i++) g.w[i] = dY[i];
        g.sched = nmat > 1 ? SCHED_SLICES : SCHED_GROUPK; g.nmat = nmat;
        g.nseg = 1; g.ksteps = (stages + S - 1) / S; g.M = Md; g.N = Nd; g.E = nmat * S;
        g.out = part; g.out_dtype = QLMB_F32; g.ldo = Nd; g.beta = 0.0f; g.name = "gemm_wgrad_slices";
        rc = gemm_launch(g, st);
        if (rc) return rc;
        const size_t n = (size_t)Md * Nd;
        SumMats m = {};
        for (int i = 0; i < nmat; i++) m.dW[i] = dW[i];
        QLMB_CUDA(pdl_launch(true, nmat > 1 ? k_sum_slices<true> : k_sum_slices<false>, dim3((unsigned)((n / 4 + 255) / 256), (unsigned)nmat), dim3(256), 0, st, m, (const float *)part, S, n, beta));
        QLMB_LAUNCH_CHECK("k_sum_slices");
        return QLMB_OK;
    }
    g.nseg = 1; g.ksteps = (M + 63) / 64; g.M = Md; g.N = Nd; g.E = 1;
    g.out = dW[0]; g.out_dtype = QLMB_F32; g.ldo = Nd; g.beta = beta;
    return gemm_launch(g, st);
}

extern "C" int qlmb_linear_wgrad(float *dW, const void *dY, const void *X, int layout, int M, int K, int N,
                                 float beta, int dtype, void *stream)
{
    QLMB_REQUIRE(dW && (M == 0 || (dY && X)), "qlmb_linear_wgrad: NULL argument");
    QLMB_REQUIRE(beta == 0.0f || beta == 1.0f, "qlmb_linear_wgrad: beta %g", beta);
    int rc = check_linear("qlmb_linear_wgrad", layout, M, K, N, dtype);
    if (rc) return rc;
    cudaStream_t st = as_stream(stream);
    if (M == 0) {
        if (beta == 0.0f) QLMB_CUDA(cudaMemsetAsync(dW, 0, (size_t)K * N * sizeof(float), st));
        return QLMB_OK;
    }
    QLMB_REQUIRE(((uintptr_t)dW & 15) == 0, "qlmb_linear_wgrad: dW must be 16-byte aligned");
    return wgrad_mats(&dW, &dY, 1, layout == QLMB_KN ? wgrad_slices(K, N, M) : wgrad_slices(N, K, M), X, layout, M, K, N, beta, dtype, st);
}

// ---- the three input projections of an attention block (gpu_forward's wq, wk, wv with k_rope, cudalm.cu:5651-5660, and their part
// of gpu_backward).  Each of the three alone is one and a third rounds of tiles for 74 SM pairs at 8192 x 768 x 768.
static int check_qkv(const char *who, const qlmb_qkv *p)
{
    QLMB_REQUIRE(p && p->cosb && p->sinb && p->T > 0, "%s: NULL argument", who);
    for (int i = 0; i < 3; i++) QLMB_REQUIRE(p->codes[i] && p->scales[i], "%s: NULL weights", who);
    int rc = check_linear(who, QLMB_KN, p->M, p->D, p->D, QLMB_BF16);
    return rc ? rc : check_linear(who, QLMB_KN, p->M, p->D, p->KD, QLMB_BF16);
}

extern "C" int qlmb_qkv_fwd(const qlmb_qkv *p, void *Yq, void *Yk, void *Yv, const void *X, void *stream)
{
    int rc = check_qkv("qlmb_qkv_fwd", p);
    if (rc || p->M == 0) return rc;
    QLMB_REQUIRE(Yq && Yk && Yv && X, "qlmb_qkv_fwd: NULL argument");
    QLMB_REQUIRE((((uintptr_t)Yq | (uintptr_t)Yk | (uintptr_t)Yv) & 15) == 0, "qlmb_qkv_fwd: the outputs must be 16-byte aligned");
    cudaStream_t st = as_stream(stream);
    void *const Y[3] = {Yq, Yk, Yv};
    const int N[3] = {p->D, p->KD, p->KD};
    // one launch over the column tiles of all three, q and k rotated on the way out
    if (gemm_pair_takes(p->D) && gemm_pair_takes(p->KD) && (((uintptr_t)p->cosb | (uintptr_t)p->sinb) & 15) == 0) {
        GemmLaunch g = {};
        g.bmode = B_DEQ_MN; g.epi = EPI_MATS; g.sched = SCHED_DENSE;
        g.a[0] = X; g.a_rows = p->M; g.a_cols = p->D;
        for (int i = 0; i < 3; i++) { g.w[i] = p->codes[i]; g.scales[i] = p->scales[i]; g.N_mat[i] = N[i]; g.outs[i] = Y[i]; }
        g.w_rows = p->D; g.w_cols = p->D; g.nmat = 3;
        g.nseg = 1; g.ksteps = p->D / 64; g.M = p->M; g.N = p->D; g.E = 1;
        g.out_dtype = QLMB_BF16; g.ldo = p->D;
        g.cosb = p->cosb; g.sinb = p->sinb; g.rope_T = p->T; g.rope_mats = 2; g.name = "gemm_qkv";
        return gemm_launch(g, st);
    }
    for (int i = 0; i < 3; i++) {
        if ((rc = qlmb_linear_fwd(Y[i], X, p->codes[i], p->scales[i], QLMB_KN, p->M, p->D, N[i], nullptr, QLMB_BF16, stream))) return rc;
        if (i < 2 && (rc = qlmb_rope(Y[i], QLMB_BF16, p->cosb, p->sinb, p->M, N[i] / 64, 64, p->T, 0, stream))) return rc;
    }
    return QLMB_OK;
}

extern "C" int qlmb_qkv_bwd(const qlmb_qkv *p, void *dX, float *dWq, float *dWk, float *dWv, const void *dq, const void *dk,
                            const void *dv, const void *X, float beta, void *stream)
{
    int rc = check_qkv("qlmb_qkv_bwd", p);
    if (rc) return rc;
    QLMB_REQUIRE(dWq && dWk && dWv && (p->M == 0 || (dX && dq && dk && dv && X)), "qlmb_qkv_bwd: NULL argument");
    QLMB_REQUIRE(beta == 0.0f || beta == 1.0f, "qlmb_qkv_bwd: beta %g", beta);
    QLMB_REQUIRE(p->M == 0 || (((uintptr_t)dX | (uintptr_t)dWq | (uintptr_t)dWk | (uintptr_t)dWv) & 15) == 0, "qlmb_qkv_bwd: the outputs must be 16-byte aligned");
    cudaStream_t st = as_stream(stream);
    const int M = p->M, D = p->D, N[3] = {D, p->KD, p->KD};
    const void *const dY[3] = {dq, dk, dv};
    float *const dW[3] = {dWq, dWk, dWv};
    if (M > 0 && gemm_pair_takes(D)) {      // one contraction over the columns of dq, dk and dv
        GemmLaunch g = {};
        g.bmode = B_DEQ_K; g.epi = EPI_MATS; g.sched = SCHED_DENSE;
        g.a_rows = M; g.a_cols = D; g.w_rows = D; g.w_cols = D; g.nmat = 1; g.N_mat[0] = D; g.outs[0] = dX;
        for (int i = 0; i < 3; i++) { g.a[i] = dY[i]; g.w[i] = p->codes[i]; g.scales[i] = p->scales[i]; g.seg_cols[i] = N[i]; }
        g.nseg = 3; g.ksteps = D / 64; g.M = M; g.N = D; g.E = 1;
        g.out = dX; g.out_dtype = QLMB_BF16; g.ldo = D; g.name = "gemm_qkv_dgrad";
        if ((rc = gemm_launch(g, st))) return rc;
    } else if (M > 0) {
        for (int i = 0; i < 3; i++)
            if ((rc = qlmb_linear_dgrad(dX, dY[i], p->codes[i], p->scales[i], QLMB_KN, M, D, N[i], i ? 1.0f : 0.0f, QLMB_BF16, stream))) return rc;
    }
    // The three weight gradients as one launch where they are of one size: of the slice counts the one with the fewest rounds of
    // tiles times stages, six stages for a tile's start and end, and the slices' partial sums at a stage's time per 2 MB.  Scratch
    // of the call's own only as large as its pool keeps it: beyond, every step maps and unmaps it (dX and dW of 8192 x 4096 with a
    // synchronisation every fourth call: 2118 us, three gradients one by one 1447).
    if (M > 0 && p->KD == D && gemm_pair_takes(D)) {
        const int stages = (M + 63) / 64, t1 = (D + 255) / 256, tiles = 3 * t1 * t1, pairs = sm_count() / 2;
        const double mb2 = 3.0 * D * D * 8.0 / 2e6;
        const bool shared = wgrad_even(D, D, M);
        int S = 0;
        double best = 0.0;
        for (int s = 2; s <= 8 && stages / s >= 8 && (shared || (size_t)3 * s * D * D * sizeof(float) <= SCRATCH_KEPT); s++) {
            const double c = (double)((tiles * s + pairs - 1) / pairs) * ((stages + s - 1) / s + 6) + s * mb2;
            if (!S || c < best) { S = s; best = c; }
        }
        if (S) return wgrad_mats(dW, dY, 3, S, X, QLMB_KN, M, D, D, beta, QLMB_BF16, st);
    }
    for (int i = 0; i < 3; i++)
        if ((rc = qlmb_linear_wgrad(dW[i], dY[i], X, QLMB_KN, M, D, N[i], beta, QLMB_BF16, stream))) return rc;
    return QLMB_OK;
}

// Engine check (not part of the reference's operator surface): C[M,N] (fp32) =
// A[M,K] * B[N,K]^T with both bf16 operands delivered by TMA, i.e. the same
// pipeline as the quantised kernels minus the dequant warps.
extern "C" int qlmb_selftest_gemm_bf16(float *C, const void *A, const void *B, int M, int K, int N, void *stream)
{
    QLMB_REQUIRE(C && A && B && M > 0 && K > 0 && N > 0 && K % 64 == 0 && N % 128 == 0, "qlmb_selftest_gemm_bf16: bad shape");
    GemmLaunch g = {};
    g.bmode = B_TMA_K; g.epi = EPI_STORE; g.sched = SCHED_DENSE;
    g.a[0] = A; g.a_rows = M; g.a_cols = K;
    g.w[0] = B; g.w_rows = N; g.w_cols = K;
    g.nseg = 1; g.ksteps = K / 64; g.M = M; g.N = N; g.E = 1;
    g.out = C; g.out_dtype = QLMB_F32; g.ldo = N;
    return gemm_launch(g, as_stream(stream));
}

// ---- unquantised operands (lm_head over the tied embedding, cudalm.cu:5832-5858) ----
// C[M,N] = A[M,K] B[N,K]^T (+ beta * C): both operands bf16, delivered by TMA; C is fp32 or bf16.
extern "C" int qlmb_gemm_nt(void *C, int c_dtype, const void *A, const void *B, int M, int K, int N, float beta, void *stream)
{
    QLMB_REQUIRE(C && A && B, "qlmb_gemm_nt: NULL argument");
    QLMB_REQUIRE(c_dtype == QLMB_F32 || c_dtype == QLMB_BF16, "qlmb_gemm_nt: dtype %d", c_dtype);
    QLMB_REQUIRE(beta == 0.0f || beta == 1.0f, "qlmb_gemm_nt: beta %g", beta);
    QLMB_REQUIRE(M >= 0 && K > 0 && N > 0 && K % 64 == 0 && N % 128 == 0, "qlmb_gemm_nt: M=%d K=%d N=%d (K %% 64, N %% 128)", M, K, N);
    if (M == 0) return QLMB_OK;
    GemmLaunch g = {};
    g.bmode = B_TMA_K; g.epi = EPI_STORE; g.sched = SCHED_DENSE;
    g.a[0] = A; g.a_rows = M; g.a_cols = K;
    g.w[0] = B; g.w_rows = N; g.w_cols = K;
    g.nseg = 1; g.ksteps = K / 64; g.M = M; g.N = N; g.E = 1;
    g.out = C; g.out_dtype = c_dtype; g.ldo = N; g.beta = beta;
    return gemm_launch(g, as_stream(stream));
}

namespace qlmb {
// dst[c][r] = bf16(src[r][c]) through a padded 32 x 32 shared-memory tile
__global__ void __launch_bounds__(256) k_cast_transpose(bf16 *dst, const float *src, int R, int Cc)
{
    pdl_wait();
    pdl_trigger();
    __shared__ float t[32][33];
    const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32, tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    for (int i = ty; i < 32; i += 8) t[i][tx] = (r0 + i < R && c0 + tx < Cc) ? src[(size_t)(r0 + i) * Cc + c0 + tx] : 0.0f;
    __syncthreads();
    for (int i = ty; i < 32; i += 8)
        if (c0 + i < Cc && r0 + tx < R) dst[(size_t)(c0 + i) * R + r0 + tx] = __float2bfloat16_rn(t[tx][i]);
}
}  // namespace qlmb

// bf16 copies of an fp32 matrix src[R][C]: plain (dst, may be NULL) and transposed (dst_t [C][R], may be NULL).
// The tied embedding is a float span; the head GEMMs read these copies (the reference casts it once per
// step as well, cudalm.cu:5822-5829).
extern "C" int qlmb_cast_bf16(void *dst, void *dst_t, const float *src, int R, int Cc, void *stream)
{
    QLMB_REQUIRE(src && (dst || dst_t) && R > 0 && Cc > 0, "qlmb_cast_bf16: bad argument");
    cudaStream_t st = as_stream(stream);
    if (dst) { int rc = convert_f32_to_bf16((bf16 *)dst, src, (size_t)R * Cc, st); if (rc) return rc; }
    if (dst_t) {
        QLMB_CUDA(pdl_launch(true, k_cast_transpose, dim3((Cc + 31) / 32, (R + 31) / 32), dim3(256), 0, st, (bf16 *)dst_t, src, R, Cc));
        QLMB_LAUNCH_CHECK("k_cast_transpose");
    }
    return QLMB_OK;
}
