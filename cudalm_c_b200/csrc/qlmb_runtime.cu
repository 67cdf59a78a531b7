// Status plumbing of libqlm_b200: thread-local error text, the per-device error
// word that kernels with bounded waits report into, and device queries.
#include "qlmb_common.cuh"
#include "qlmb_tc.cuh"
#include <string.h>
#include <stdlib.h>

namespace qlmb {

static thread_local char g_err[512] = "";

void set_error(const char *fmt, ...)
{
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof g_err, fmt, ap);
    va_end(ap);
}

int cuda_fail(cudaError_t e, const char *what)
{
    set_error("CUDA error %d (%s) at %s", (int)e, cudaGetErrorString(e), what);
    return QLMB_E_CUDA;
}

static int *g_errword[64];
static int g_sms[64];

bool pdl_enabled(void)
{
    static int on = -1;
    if (on < 0) { const char *e = getenv("QLMB_PDL"); on = (e && atoi(e) == 0) ? 0 : 1; }
    return on != 0;
}

int *device_error_word(void)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
    if (!g_errword[dev]) {
        int *p = nullptr;
        if (cudaMalloc(&p, 16 * sizeof(int)) != cudaSuccess) return nullptr;
        if (cudaMemset(p, 0, 16 * sizeof(int)) != cudaSuccess) return nullptr;
        g_errword[dev] = p;
    }
    return g_errword[dev];
}

int sm_count(void)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
    if (!g_sms[dev]) {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
        g_sms[dev] = n;
    }
    return g_sms[dev];
}


// ---- scopes in which nothing writes weights (pdl_launch) ----
static thread_local struct { int depth; bool waited; cudaStream_t st; } t_quiet;
int weights_quiet(cudaStream_t st)
{
    if (t_quiet.depth == 0 || t_quiet.st != st) return 0;
    const bool known = t_quiet.waited;
    t_quiet.waited = true;
    return known ? QUIET : QUIET_FIRST;
}
}  // namespace qlmb
extern "C" int qlmb_quiet_begin(void *stream)
{
    QLMB_REQUIRE(qlmb::t_quiet.depth == 0, "qlmb_quiet_begin: this thread is inside such a scope already");
    qlmb::t_quiet.depth = 1; qlmb::t_quiet.waited = false; qlmb::t_quiet.st = qlmb::as_stream(stream);
    return QLMB_OK;
}
extern "C" int qlmb_quiet_end(void)
{
    qlmb::t_quiet.depth = 0;
    return QLMB_OK;
}
namespace qlmb {

// ---- two library-owned streams per device for work that may overlap the caller's stream ----
// side_fork() makes the side stream wait for everything queued on `st` so far, side_join()
// makes `st` wait for everything queued on the side stream; side_wait_main() is a second
// fork point in between.  QLMB_SIDE_STREAM=0 runs everything on the caller's stream.
static cudaStream_t g_side[64][2];
static cudaEvent_t g_side_ev[64][2][3];
static int g_side_on = -1;

cudaStream_t side_fork(cudaStream_t st, int which)
{
    if (g_side_on < 0) { const char *e = getenv("QLMB_SIDE_STREAM"); g_side_on = (e && atoi(e) == 0) ? 0 : 1; }
    int dev = 0;
    if (!g_side_on || which < 0 || which > 1 || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return st;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) return st;
    if (!g_side[dev][which]) {
        if (cudaStreamCreateWithFlags(&g_side[dev][which], cudaStreamNonBlocking) != cudaSuccess) { g_side[dev][which] = nullptr; return st; }
        for (int i = 0; i < 3; i++)
            if (cudaEventCreateWithFlags(&g_side_ev[dev][which][i], cudaEventDisableTiming) != cudaSuccess) return st;
    }
    if (cudaEventRecord(g_side_ev[dev][which][0], st) != cudaSuccess) return st;
    if (cudaStreamWaitEvent(g_side[dev][which], g_side_ev[dev][which][0], 0) != cudaSuccess) return st;
    return g_side[dev][which];
}
static int side_index(cudaStream_t side)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -1;
    for (int w = 0; w < 2; w++) if (g_side[dev][w] && g_side[dev][w] == side) return dev * 2 + w;
    return -1;
}
void side_wait_main(cudaStream_t side, cudaStream_t st)
{
    const int ix = side == st ? -1 : side_index(side);
    if (ix < 0) return;
    cudaEventRecord(g_side_ev[ix / 2][ix % 2][1], st);
    cudaStreamWaitEvent(side, g_side_ev[ix / 2][ix % 2][1], 0);
}
}  // namespace qlmb
extern "C" int qlmb_side_stream_enable(int on)
{
    qlmb::g_side_on = on ? 1 : 0;
    return QLMB_OK;
}
namespace qlmb {
void side_join(cudaStream_t side, cudaStream_t st)
{
    const int ix = side == st ? -1 : side_index(side);
    if (ix < 0) return;
    cudaEventRecord(g_side_ev[ix / 2][ix % 2][2], side);
    cudaStreamWaitEvent(st, g_side_ev[ix / 2][ix % 2][2], 0);
}

// ---- optional per-kernel timing (CUDA events on the launching stream) ----
static bool g_prof_on = false;
static int g_prof_n = 0;
static const int PROF_MAX = 512;
static const char *g_prof_name[PROF_MAX];
static cudaEvent_t g_prof_ev[PROF_MAX][2];
static bool g_prof_have[PROF_MAX];

ProfScope::ProfScope(const char *name, cudaStream_t st) : slot(-1), stream(st)
{
    if (!g_prof_on || g_prof_n >= PROF_MAX) return;
    slot = g_prof_n++;
    if (!g_prof_have[slot]) {
        if (cudaEventCreate(&g_prof_ev[slot][0]) != cudaSuccess || cudaEventCreate(&g_prof_ev[slot][1]) != cudaSuccess) { slot = -1; g_prof_n--; return; }
        g_prof_have[slot] = true;
    }
    g_prof_name[slot] = name;
    cudaEventRecord(g_prof_ev[slot][0], st);
}
ProfScope::~ProfScope()
{
    if (slot >= 0) cudaEventRecord(g_prof_ev[slot][1], stream);
}

}  // namespace qlmb

extern "C" int qlmb_prof_enable(int on)
{
    qlmb::g_prof_on = on != 0;
    qlmb::g_prof_n = 0;
    return QLMB_OK;
}
// Synchronises the device and returns the recorded scopes since the last call:
// names (64 bytes each) and milliseconds; the return value is the count.
extern "C" int qlmb_prof_read(char *names, float *ms, int max)
{
    if (cudaDeviceSynchronize() != cudaSuccess) return -1;
    int n = qlmb::g_prof_n < max ? qlmb::g_prof_n : max;
    for (int i = 0; i < n; i++) {
        float t = 0.0f;
        cudaEventElapsedTime(&t, qlmb::g_prof_ev[i][0], qlmb::g_prof_ev[i][1]);
        ms[i] = t;
        snprintf(names + 64 * i, 64, "%s", qlmb::g_prof_name[i]);
    }
    qlmb::g_prof_n = 0;
    return n;
}

extern "C" const char *qlmb_last_error(void) { return qlmb::g_err; }
extern "C" int qlmb_version(void) { return 1; }

extern "C" int qlmb_check_device(void *stream)
{
    int *w = qlmb::device_error_word();
    if (!w) return qlmb::cuda_fail(cudaGetLastError(), "device_error_word");
    int h[4] = {0, 0, 0, 0};
    QLMB_CUDA(cudaMemcpyAsync(h, w, sizeof h, cudaMemcpyDeviceToHost, qlmb::as_stream(stream)));
    QLMB_CUDA(cudaStreamSynchronize(qlmb::as_stream(stream)));
    if (h[0] != 0) {
        qlmb::set_error("device reported error code %d (site %d, block %d, detail %d)", h[0], h[1], h[2], h[3]);
        QLMB_CUDA(cudaMemsetAsync(w, 0, sizeof h, qlmb::as_stream(stream)));
        return QLMB_E_DEVICE;
    }
    return QLMB_OK;
}

// ---- the error path of the bounded waits, exercised without a fault ----
// One warp initialises an mbarrier that nothing ever arrives at and polls it `polls` times, exactly as the
// waits of the tcgen05 kernels do (mbarrier.try_wait, then give up, record the site in the device error word
// and return).  The kernel ends normally; the context stays usable.
namespace qlmb {
__global__ void k_selftest_wait(int *errword, uint32_t polls)
{
    __shared__ __align__(8) uint64_t bar;
    const uint32_t b = smem_u32(&bar);
    if (threadIdx.x == 0) { mbar_init(b, 1); fence_barrier_init(); }
    __syncthreads();
    if (threadIdx.x != 0) return;
    for (uint32_t i = 0; i < polls; i++)
        if (mbar_try(b, 0)) return;                      // cannot happen: no arrival is ever made
    if (errword && atomicCAS(errword, 0, 200) == 0) { errword[1] = 9999; errword[2] = (int)blockIdx.x; errword[3] = (int)polls; }
}
}  // namespace qlmb
// ---- read-only pass over a code matrix: what a kernel that does nothing but load the same bytes achieves
namespace qlmb {
__global__ void __launch_bounds__(256) k_stream_read(const uint8_t *W, size_t row_bytes, int rows, unsigned *sink)
{
    // block (x, y): 256 bytes of every row of K slice y; warp w takes rows w, w + 8, ..., 16 rows in flight per lane
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint8_t *p = W + (size_t)(blockIdx.y * rows + warp) * row_bytes + (size_t)blockIdx.x * 256 + lane * 8;
    unsigned acc = 0;
    for (int r = warp; r < rows; r += 8 * 16) {
        uint2 v[16];
#pragma unroll
        for (int u = 0; u < 16; u++) v[u] = (r + 8 * u < rows) ? __ldcs(reinterpret_cast<const uint2 *>(p + (size_t)(8 * u) * row_bytes)) : make_uint2(0u, 0u);
#pragma unroll
        for (int u = 0; u < 16; u++) acc += v[u].x + v[u].y;
        p += (size_t)128 * row_bytes;
    }
    if (acc == 0x9E3779B9u) *sink = acc;                 // keeps the loads alive; practically never true
}
}  // namespace qlmb
extern "C" int qlmb_selftest_stream_read(const void *W, unsigned long long row_bytes, int rows, int kslices, void *stream)
{
    QLMB_REQUIRE(W && row_bytes >= 256 && row_bytes % 256 == 0 && rows > 0 && kslices > 0 && rows % kslices == 0,
                 "qlmb_selftest_stream_read: row_bytes %llu rows %d kslices %d", row_bytes, rows, kslices);
    static unsigned *sink[64];
    int dv = 0;
    QLMB_CUDA(cudaGetDevice(&dv));
    QLMB_REQUIRE(dv >= 0 && dv < 64, "qlmb_selftest_stream_read: device %d", dv);
    if (!sink[dv]) QLMB_CUDA(cudaMalloc(&sink[dv], sizeof(unsigned)));
    qlmb::k_stream_read<<<dim3((unsigned)(row_bytes / 256), (unsigned)kslices), 256, 0, qlmb::as_stream(stream)>>>(
        (const uint8_t *)W, (size_t)row_bytes, rows / kslices, sink[dv]);
    QLMB_LAUNCH_CHECK("k_stream_read");
    return QLMB_OK;
}

extern "C" int qlmb_selftest_wait_expires(int polls, void *stream)
{
    QLMB_REQUIRE(polls > 0 && polls <= (1 << 16), "qlmb_selftest_wait_expires: polls %d", polls);
    int *w = qlmb::device_error_word();
    if (!w) return qlmb::cuda_fail(cudaGetLastError(), "device_error_word");
    qlmb::k_selftest_wait<<<1, 32, 0, qlmb::as_stream(stream)>>>(w, (uint32_t)polls);
    QLMB_LAUNCH_CHECK("k_selftest_wait");
    return QLMB_OK;
}

// ---- device memory that other processes of the node can map (CUDA IPC) ----
extern "C" int qlmb_peer_alloc(size_t bytes, void **ptr)
{
    QLMB_REQUIRE(ptr && bytes > 0, "qlmb_peer_alloc: bad argument");
    QLMB_CUDA(cudaMalloc(ptr, bytes));
    return QLMB_OK;
}
extern "C" int qlmb_peer_free(void *ptr)
{
    if (ptr) QLMB_CUDA(cudaFree(ptr));
    return QLMB_OK;
}
extern "C" int qlmb_peer_export(const void *ptr, unsigned char handle[64])
{
    QLMB_REQUIRE(ptr && handle, "qlmb_peer_export: NULL argument");
    static_assert(sizeof(cudaIpcMemHandle_t) == 64, "IPC handle size");
    cudaIpcMemHandle_t h;
    QLMB_CUDA(cudaIpcGetMemHandle(&h, const_cast<void *>(ptr)));
    memcpy(handle, &h, 64);
    return QLMB_OK;
}
extern "C" int qlmb_peer_open(const unsigned char handle[64], void **ptr)
{
    QLMB_REQUIRE(ptr && handle, "qlmb_peer_open: NULL argument");
    cudaIpcMemHandle_t h;
    memcpy(&h, handle, 64);
    QLMB_CUDA(cudaIpcOpenMemHandle(ptr, h, cudaIpcMemLazyEnablePeerAccess));
    return QLMB_OK;
}
extern "C" int qlmb_peer_close(void *ptr)
{
    if (ptr) QLMB_CUDA(cudaIpcCloseMemHandle(ptr));
    return QLMB_OK;
}
