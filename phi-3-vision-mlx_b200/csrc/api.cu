// Error plumbing + version for the C ABI.
#include "common.cuh"
#include "../../include/phi3_b200.h"
#include <cstdarg>
#include <cstdio>
#include <mutex>
#include "tc_common.cuh"

static thread_local char g_err[512] = "";

void p3_set_error(const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
}
extern "C" const char* p3_last_error(void) { return g_err; }
extern "C" int p3_version(void) { return 1; }

// ---- status word of bounded waits. One for the process: every device sees it, and any later call on any thread reports it once.
static int* g_status = nullptr;
int* p3_status_word() {
    static std::once_flag once;
    std::call_once(once, [] {
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;       // the first launch may be a captured one: an allocation is not part of a graph
        cudaThreadExchangeStreamCaptureMode(&mode);
        void* p = nullptr;
        if (cudaHostAlloc(&p, sizeof(int), cudaHostAllocPortable | cudaHostAllocMapped) == cudaSuccess) {
            *static_cast<int*>(p) = 0;
            __atomic_store_n(&g_status, static_cast<int*>(p), __ATOMIC_RELEASE);
        } else cudaGetLastError();
        cudaThreadExchangeStreamCaptureMode(&mode);
    });
    return g_status;
}
bool p3_take_status() {
    int* w = __atomic_load_n(&g_status, __ATOMIC_ACQUIRE);
    return w && __atomic_load_n(w, __ATOMIC_RELAXED) && __atomic_exchange_n(w, 0, __ATOMIC_ACQ_REL);
}

// One warp waits, for a few milliseconds, at a barrier that nothing arrives at, and gives up as the kernels above do: numbers 0 .. 15 behind a wait whose
// tries rest for long, 16 .. 31 behind one whose tries rest as the hardware sees fit
template <bool HINT> __device__ void wait_runs_out(uint32_t bar, volatile int* fail, float* out16, int* status) {
    if (threadIdx.x == 0) *fail = 0;
    __syncwarp();
    mbar_wait_lim<HINT>(bar, 0, fail, 1000000);
    __syncwarp();
    if (*fail) {
        if (threadIdx.x < 16) out16[threadIdx.x] = __int_as_float(0x7fc00000);
        if (threadIdx.x == 0) set_status(status);
    }
    __syncwarp();
}
__global__ void wait_runs_out_kernel(float* out, int* status) {
    __shared__ __align__(8) uint64_t bar_s;
    __shared__ int fail_s;
    const uint32_t bar = smem_u32(&bar_s);
    if (threadIdx.x == 0) mbar_init(bar, 1);
    __syncwarp();
    wait_runs_out<true>(bar, &fail_s, out, status);
    wait_runs_out<false>(bar, &fail_s, out + 16, status);
}
extern "C" int p3_wait_selftest(float* out32, cudaStream_t st) {
    P3_CHECK_ARG(out32, "wait_selftest: null argument");
    wait_runs_out_kernel<<<1, 32, 0, st>>>(out32, p3_status_word());
    P3_CHECK_LAUNCH("wait_selftest");
    return 0;
}

// ---- in-kernel timeline (off unless a buffer is set): every traced launch takes the next slot of
// P3_TRACE_CTAS x 8 u64 and its CTAs' thread 0 store {globaltimer at start, after the dependency wait, first operands ready,
// main loop done, exit, smid, kind}. Diagnostic only; costs one null test per launch when off.
static unsigned long long* g_trace = nullptr;
static int g_trace_slots = 0, g_trace_next = 0;
extern "C" int p3_trace_set(void* buf, int n_slots) { g_trace = (unsigned long long*)buf; g_trace_slots = n_slots; g_trace_next = 0; return 0; }
extern "C" int p3_trace_count(void) { return g_trace_next; }
unsigned long long* p3_trace_slot() {
    if (!g_trace || g_trace_next >= g_trace_slots) return nullptr;
    return g_trace + (size_t)(g_trace_next++) * P3_TRACE_CTAS * 8;
}
