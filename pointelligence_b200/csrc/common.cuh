// Shared helpers of the C-ABI library: status reporting, launch checks,
// workspace carving, element-type conversion.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include <atomic>
#include <utility>

#include "../../include/pointelligence_b200.h"

namespace pcx {

void set_error(const char *fmt, ...);
extern std::atomic<long long> g_launches;               // kernels launched by this library
// Where a host hand-over (a copy or stores of a kernel, and a wait, in one call) puts its words.
constexpr int HANDOVER_WORDS = 16;
int64_t *handover_words();

// A hand-over by stores: a kernel puts its words and then the ticket where the host reads them, and the host waits for the
// ticket, not for the kernel's end.  Against two copies and a wait for the stream: some 20 us less
// a search; with the host free while the pairs are written, a rulebook of 150 000 points 211 -> 128 us, binning included.
struct HandOver {
    int64_t *words = nullptr;   // page-locked; null where there is none: the host copies after the kernel's end
    int64_t ticket = 0;
    static constexpr int TICKET = HANDOVER_WORDS - 1;
    __device__ __forceinline__ void put(int n, int64_t v) const { *(volatile int64_t *)(words + n) = v; }
    __device__ __forceinline__ void done() const {
        __threadfence_system();
        *(volatile int64_t *)(words + TICKET) = ticket;
    }
};
HandOver new_hand_over();                                        // of this thread: one at a time
int wait_for_hand_over(const HandOver &h, cudaStream_t stream);
void prof_begin(const char *name, cudaStream_t stream); // event timer around a dominant kernel
void prof_end(cudaStream_t stream);

#define PCX_FAIL(code, ...)            \
    do {                               \
        ::pcx::set_error(__VA_ARGS__); \
        return (code);                 \
    } while (0)

#define PCX_CUDA(expr)                                                          \
    do {                                                                        \
        cudaError_t _e = (expr);                                                \
        if (_e != cudaSuccess)                                                  \
            PCX_FAIL(PCX_E_LAUNCH, "%s failed: %s (%s:%d)", #expr,              \
                     cudaGetErrorString(_e), __FILE__, __LINE__);               \
    } while (0)

#define PCX_LAUNCH_CHECK()            \
    do {                              \
        ::pcx::g_launches.fetch_add(1); \
        PCX_CUDA(cudaGetLastError()); \
    } while (0)

// A kernel launched by launch_after() is set up on the chip while the one before it in the stream is still finishing; it
// starts with start_after_previous(), which returns when that one has ended and its writes can be read, and allows the
// next one the same.  Every thread calls it before it reads or writes global memory, so that an end implies the ends of all
// before.  A kernel with tensor memory takes it, and passes a barrier, before that call: the next one may take its own early, on
// the same multiprocessor, and would be waited for by one that still has to.  With the barriers of its pipeline it is then ready
// when the kernel before it ends: a training call of 942 points and 512 channels 166 -> 159 us.
// A gap between kernels shrinks by 1 to 1.5 us: a training call of 942 points and 512 channels (11 launches) 230 -> 214 us,
// 150 000 points and 64 channels (11) 224 -> 212, an fp32 one (8) 204 -> 194, a norm with its gradient (7) 229 -> 215.
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void let_next_be_set_up() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void start_after_previous() {
    wait_for_previous();
    let_next_be_set_up();
}
// Allows a kernel all the shared memory that a block of the device can have, once per device (a bit each in `done`).  Asked for as
// much as a launch needs, a thread could take back what another had just asked for and was about to launch with.
// `prefer`: multiprocessors are to be set up for as much shared memory as they have, too.
int allow_shared_memory(const void *kernel, std::atomic<uint64_t> *done, bool prefer = false);

template <typename... Params, typename... Args>
void launch_after(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args &&...args) {
    cudaLaunchAttribute early = {};
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t config = {};
    config.gridDim = grid, config.blockDim = block, config.dynamicSmemBytes = smem, config.stream = stream;
    config.attrs = &early, config.numAttrs = 1;
    (void)cudaLaunchKernelEx(&config, kernel, std::forward<Args>(args)...);   // PCX_LAUNCH_CHECK asks for the error
}

// What a kernel is launched for only if an earlier one found a reason: a word from each of that one's blocks, zero where it
// found none.  No words: always.  Asked by a whole block, in variants of their own (AGAIN) of kernels that are mostly launched
// without: asked at run time, a pass over 150 000 points and 64 channels (clear, scatter, round) took 82 us instead of 81.
struct OnlyIf {
    const uint32_t *words = nullptr;
    int n = 0;
    __device__ __forceinline__ bool holds() const {
        bool any = false;
        for (int t = threadIdx.x; t < n; t += blockDim.x) any |= words[t] != 0;
        return __syncthreads_or(any);
    }
};

static inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

// Bump allocator over a caller-owned workspace; every block 256-byte aligned.
struct Carver {
    char *base;
    size_t off;
    explicit Carver(void *p) : base(static_cast<char *>(p)), off(0) {}
    template <typename T>
    T *take(size_t count) {
        T *p = reinterpret_cast<T *>(base + off);
        off += align_up(count * sizeof(T), 256);
        return p;
    }
};

// Product of non-negative sizes; false when a factor is negative or the product exceeds `limit`
// (checked factor by factor, so it cannot wrap on the way).
static inline bool product_within(uint64_t limit, uint64_t *out, int64_t a, int64_t b = 1, int64_t c = 1, int64_t d = 1) {
    const int64_t f[4] = {a, b, c, d};
    uint64_t p = 1;
    for (int i = 0; i < 4; ++i) {
        if (f[i] < 0) return false;
        if (__builtin_mul_overflow(p, (uint64_t)f[i], &p) || p > limit) return false;
    }
    *out = p;
    return true;
}

static inline size_t elem_size(int dtype) { return dtype == PCX_F32 ? 4 : 2; }

template <typename T>
__device__ __forceinline__ float to_f32(T v);
template <>
__device__ __forceinline__ float to_f32<float>(float v) { return v; }
template <>
__device__ __forceinline__ float to_f32<__half>(__half v) { return __half2float(v); }
template <>
__device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

template <typename T>
__device__ __forceinline__ T from_f32(float v);
template <>
__device__ __forceinline__ float from_f32<float>(float v) { return v; }
template <>
__device__ __forceinline__ __half from_f32<__half>(float v) { return __float2half_rn(v); }
template <>
__device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

static inline int num_sms() {
    static int cached = 0;
    if (!cached) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&cached, cudaDevAttrMultiProcessorCount, dev);
        if (cached <= 0) cached = 148;
    }
    return cached;
}

}  // namespace pcx
