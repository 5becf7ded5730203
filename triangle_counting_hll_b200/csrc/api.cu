// api.cu -- library-wide C-ABI plumbing: error reporting, launch accounting,
// device properties.
#include <stdarg.h>

#include <atomic>

#include "common.cuh"

namespace tchll {

static thread_local char g_err[1024] = "";
static std::atomic<uint64_t> g_launches{0};

void set_error(const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
}

int cuda_status(cudaError_t e, const char* what) {
    set_error("%s: %s (%s)", what, cudaGetErrorString(e), cudaGetErrorName(e));
    return TCHLL_ECUDA;
}

void count_launch(int n) { g_launches.fetch_add((uint64_t)n, std::memory_order_relaxed); }

int sm_count() {
    static int cached[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0) return 148;
    if (dev < 64 && cached[dev]) return cached[dev];
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    if (dev < 64) cached[dev] = n;
    return n;
}

}  // namespace tchll

TCHLL_EXPORT const char* tchll_last_error(void) { return tchll::g_err; }

TCHLL_EXPORT int tchll_version(void) { return 10000; }

TCHLL_EXPORT uint64_t tchll_launch_count(void) { return tchll::g_launches.load(std::memory_order_relaxed); }

// Small device-to-host reads.  A copy into pageable memory goes through the
// driver's staging and costs several times a copy into pinned memory, so each
// host thread keeps one pinned page (made on its first read, freed when the
// thread ends); the wait for the stream is the read's own.
namespace tchll {
namespace {
constexpr size_t kStageBytes = 4096;
struct PinnedStage {
    void* p = nullptr;
    void* get() {
        if (p == nullptr && cudaMallocHost(&p, kStageBytes) != cudaSuccess) {
            cudaGetLastError();  // no pinned memory: the caller copies directly
            p = nullptr;
        }
        return p;
    }
    ~PinnedStage() {
        if (p) cudaFreeHost(p);
    }
};
thread_local PinnedStage g_stage;
}  // namespace

int fetch_small(void* dst, const void* src, size_t n, cudaStream_t st) {
    void* stage = n <= kStageBytes ? g_stage.get() : nullptr;
    TCHLL_CUDA(cudaMemcpyAsync(stage ? stage : dst, src, n, cudaMemcpyDeviceToHost, st));
    TCHLL_CUDA(cudaStreamSynchronize(st));
    if (stage) memcpy(dst, stage, n);
    return TCHLL_OK;
}
}  // namespace tchll

TCHLL_EXPORT int tchll_fetch(void* dst, const void* src, int64_t n, void* stream) {
    TCHLL_ARG(n >= 0 && (n == 0 || (dst && src)), "bad arguments");
    if (n == 0) return TCHLL_OK;
    return tchll::fetch_small(dst, src, (size_t)n, (cudaStream_t)stream);
}

TCHLL_EXPORT int tchll_device_sync(void) {
    TCHLL_CUDA(cudaDeviceSynchronize());
    return TCHLL_OK;
}
