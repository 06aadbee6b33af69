// Thread-local error message, version, launch counter and the optional
// per-kernel event timer of the C-ABI library.
#include <stdarg.h>

#include <atomic>
#include <vector>

#include "common.cuh"

namespace pcx {
static thread_local char g_error[512] = "";

void set_error(const char *fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_error, sizeof(g_error), fmt, ap);
    va_end(ap);
}

std::atomic<long long> g_launches{0};

namespace {
struct Words {   // page-locked, one set per thread: copies into it neither stage nor block the stream
    int64_t *words = nullptr;
    int64_t pageable[HANDOVER_WORDS];
    int64_t tickets = 0;
    ~Words() {
        if (words && words != pageable) cudaFreeHost(words);
    }
};
Words &this_threads_words() {
    static thread_local Words h;
    if (!h.words) {
        if (cudaHostAlloc((void **)&h.words, HANDOVER_WORDS * sizeof(int64_t), cudaHostAllocPortable) != cudaSuccess) {
            (void)cudaGetLastError();
            h.words = h.pageable;
        }
        h.words[HandOver::TICKET] = 0;
    }
    return h;
}
}  // namespace

int64_t *handover_words() { return this_threads_words().words; }

HandOver new_hand_over() {
    Words &w = this_threads_words();
    HandOver h;
    if (w.words != w.pageable) h.words = w.words;
    h.ticket = ++w.tickets;
    return h;
}

int wait_for_hand_over(const HandOver &h, cudaStream_t stream) {
    const volatile int64_t *ticket = h.words + HandOver::TICKET;
    for (bool ended = false;;) {
        for (int n = 0; n < 1000; ++n) {
            if (*ticket == h.ticket) {
                std::atomic_thread_fence(std::memory_order_acquire);
                return PCX_OK;
            }
            __builtin_ia32_pause();
        }
        if (ended) PCX_FAIL(PCX_E_LAUNCH, "a kernel ended without its hand-over");
        const cudaError_t e = cudaStreamQuery(stream);   // (so that a failed launch ends the wait)
        if (e == cudaErrorNotReady) (void)cudaGetLastError();
        else if (e != cudaSuccess) PCX_FAIL(PCX_E_LAUNCH, "waiting for a kernel failed: %s", cudaGetErrorString(e));
        else ended = true;
    }
}

int allow_shared_memory(const void *kernel, std::atomic<uint64_t> *done, bool prefer) {
    int dev = 0, most = 0;
    PCX_CUDA(cudaGetDevice(&dev));
    const uint64_t bit = 1ull << (dev & 63);
    if (done->load(std::memory_order_acquire) & bit) return PCX_OK;
    cudaFuncAttributes own;
    PCX_CUDA(cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    PCX_CUDA(cudaFuncGetAttributes(&own, kernel));
    PCX_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most - (int)own.sharedSizeBytes));
    if (prefer) PCX_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
    done->fetch_or(bit, std::memory_order_release);
    return PCX_OK;
}

struct ProfRecord {
    const char *name;
    cudaEvent_t start, stop;
};
static bool g_prof_on = false;
static std::vector<ProfRecord> g_prof;
static size_t g_prof_used = 0;
static constexpr size_t kProfCapacity = 1 << 14;

// Brackets the dominant kernel of an entry point with CUDA events recorded on
// the launch stream.  No effect unless pcx_profile_enable(1) was called.
void prof_begin(const char *name, cudaStream_t stream) {
    if (!g_prof_on || g_prof_used >= kProfCapacity) return;
    if (g_prof_used == g_prof.size()) {
        ProfRecord r{name, nullptr, nullptr};
        if (cudaEventCreate(&r.start) != cudaSuccess || cudaEventCreate(&r.stop) != cudaSuccess) return;
        g_prof.push_back(r);
    }
    g_prof[g_prof_used].name = name;
    cudaEventRecord(g_prof[g_prof_used].start, stream);
}

void prof_end(cudaStream_t stream) {
    if (!g_prof_on || g_prof_used >= g_prof.size()) return;
    cudaEventRecord(g_prof[g_prof_used].stop, stream);
    ++g_prof_used;
}
}  // namespace pcx

extern "C" {
int pcx_version(void) { return 10100; }
const char *pcx_last_error_string(void) { return pcx::g_error; }

long long pcx_launch_count(int reset) {
    long long v = pcx::g_launches.load();
    if (reset) pcx::g_launches.store(0);
    return v;
}

int pcx_profile_enable(int on) {
    pcx::g_prof_on = on != 0;
    pcx::g_prof_used = 0;
    return PCX_OK;
}

int pcx_profile_count(void) { return (int)pcx::g_prof_used; }

int pcx_profile_get(int index, const char **name, float *milliseconds) {
    if (index < 0 || (size_t)index >= pcx::g_prof_used || !name || !milliseconds)
        PCX_FAIL(PCX_E_ARG, "pcx_profile_get: bad index %d", index);
    auto &r = pcx::g_prof[index];
    PCX_CUDA(cudaEventSynchronize(r.stop));
    PCX_CUDA(cudaEventElapsedTime(milliseconds, r.start, r.stop));
    *name = r.name;
    return PCX_OK;
}
}
