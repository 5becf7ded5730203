// api.cu -- library-wide C-ABI plumbing: error reporting, launch accounting,
// device properties.
#include <stdarg.h>

#include <atomic>
#include <mutex>

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

namespace tchll {
typedef int (*CtxGetCurrentFn)(void** ctx);
typedef int (*CtxGetIdFn)(void* ctx, unsigned long long* id);

bool current_ctx_id(unsigned long long* id) {
    static CtxGetCurrentFn get_cur = nullptr;
    static CtxGetIdFn get_id = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &f, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_cur = (CtxGetCurrentFn)f;
        f = nullptr;
        if (cudaGetDriverEntryPoint("cuCtxGetId", &f, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_id = (CtxGetIdFn)f;
    });
    if (get_cur == nullptr || get_id == nullptr) return false;
    void* ctx = nullptr;
    if (get_cur(&ctx) != 0 || ctx == nullptr) return false;
    return get_id(ctx, id) == 0;
}

// Small device-to-host reads.  A copy into pageable memory goes through the
// driver's staging and costs several times a copy into pinned memory, so a
// read takes a pinned page, and gives it back for later reads; the wait for
// the stream is the read's own.  A page belongs to the context that it was
// made in and is gone with it (cudaDeviceReset), so it is only ever used, or
// freed, while that context is current; at most kStagePages are kept.
namespace {
constexpr size_t kStageBytes = 4096;
constexpr int kStagePages = 64;
struct StagePage {
    unsigned long long ctx_id;
    void* p;
};
std::mutex g_stage_mu;
StagePage g_stage[kStagePages];
int g_stage_n = 0;

// A page of the current context, or p = null: the caller copies directly.
StagePage take_stage() {
    StagePage s{0, nullptr};
    if (!current_ctx_id(&s.ctx_id)) return s;
    {
        std::lock_guard<std::mutex> lock(g_stage_mu);
        for (int i = 0; i < g_stage_n; ++i)
            if (g_stage[i].ctx_id == s.ctx_id) {
                s.p = g_stage[i].p;
                g_stage[i] = g_stage[--g_stage_n];
                return s;
            }
    }
    if (cudaMallocHost(&s.p, kStageBytes) != cudaSuccess) {
        cudaGetLastError();  // no pinned memory
        s.p = nullptr;
    }
    return s;
}

void give_stage(StagePage s) {
    if (s.p == nullptr) return;
    {
        std::lock_guard<std::mutex> lock(g_stage_mu);
        if (g_stage_n < kStagePages) {
            g_stage[g_stage_n++] = s;
            return;
        }
    }
    cudaFreeHost(s.p);
}
}  // namespace

int fetch_small(void* dst, const void* src, size_t n, cudaStream_t st) {
    StagePage s{0, nullptr};
    if (n <= kStageBytes) s = take_stage();
    cudaError_t e = cudaMemcpyAsync(s.p ? s.p : dst, src, n, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e == cudaSuccess && s.p) memcpy(dst, s.p, n);
    if (e != cudaSuccess) return cuda_status(e, "fetch");  // the page may still be written to: it is not used again
    give_stage(s);
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
