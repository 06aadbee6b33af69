// CUDA-core engines for triplets in any order (one warp per triplet), the chunk table of rulebooks with many taps
// and the rounding of the fp32 accumulator into the output element type.  Tap-sorted triplets go to sparse_fma.cu.
#include "sparse_kernels.cuh"

namespace pcx {

// cum[k] = number of L-triplet chunks in the taps before k (one block, any K)
__global__ void chunk_table_kernel(const int64_t *__restrict__ seg, int K, int L, int32_t *cum) {
    __shared__ int32_t warp_sums[32];
    __shared__ int32_t carry;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
    if (tid == 0) carry = 0;
    __syncthreads();
    for (int base = 0; base < K; base += blockDim.x) {
        int k = base + tid;
        int32_t v = k < K ? (int32_t)((seg[k + 1] - seg[k] + L - 1) / L) : 0;
        int32_t inc = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int32_t n = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += n;
        }
        if (lane == 31) warp_sums[warp] = inc;
        __syncthreads();
        int32_t before = carry;
        for (int w = 0; w < warp; ++w) before += warp_sums[w];
        if (k < K) cum[k] = before + inc - v;
        __syncthreads();
        if (tid == 0) {
            int32_t t = carry;
            for (int w = 0; w < nwarps; ++w) t += warp_sums[w];
            carry = t;
        }
        __syncthreads();
    }
    if (tid == 0) cum[K] = carry;
}

namespace {

// one warp per triplet, taps in any order
template <typename T, bool TRANSPOSE>
__global__ void mvmr_unsorted_kernel(const T *__restrict__ W, const T *__restrict__ feat,
                                     const int32_t *__restrict__ gather, const int32_t *__restrict__ scatter,
                                     const int32_t *__restrict__ tap_idx, float *__restrict__ acc,
                                     int64_t Tn, int K, int G, int C, int M, int reverse) {
    int64_t t = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (t >= Tn) return;
    const int lane = threadIdx.x & 31;
    const int inw = TRANSPOSE ? M : C, outw = TRANSPOSE ? C : M;
    const int64_t k = reverse ? K - 1 - tap_idx[t] : tap_idx[t], src = gather[t], dst = scatter[t];
    for (int g = 0; g < G; ++g) {
        const T *Wk = W + (k * G + g) * C * M;
        const T *x = feat + (src * G + g) * inw;
        float *o = acc + (dst * G + g) * outw;
        for (int n = lane; n < outw; n += 32) {
            float s = 0.f;
            for (int c = 0; c < inw; ++c) {
                int64_t off = TRANSPOSE ? (int64_t)n * M + c : (int64_t)c * M + n;
                s = __fmaf_rn(to_f32(x[c]), to_f32(Wk[off]), s);
            }
            atomicAdd(o + n, s);
        }
    }
}

template <typename T>
__global__ void vvor_unsorted_kernel(const T *__restrict__ A, const int32_t *__restrict__ a_idx,
                                     const T *__restrict__ B, const int32_t *__restrict__ b_idx,
                                     const int32_t *__restrict__ o_idx, float *__restrict__ acc,
                                     int64_t Tn, int G, int Ma, int Cb) {
    int64_t t = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (t >= Tn) return;
    const int lane = threadIdx.x & 31;
    const int64_t ia = a_idx[t], ib = b_idx[t], io = o_idx[t];
    for (int g = 0; g < G; ++g) {
        const T *a = A + (ia * G + g) * Ma;
        const T *b = B + (ib * G + g) * Cb;
        float *o = acc + (io * G + g) * Ma * Cb;
        for (int m = 0; m < Ma; ++m) {
            float am = to_f32(a[m]);
            for (int c = lane; c < Cb; c += 32) atomicAdd(o + (int64_t)m * Cb + c, am * to_f32(b[c]));
        }
    }
}

template <typename T, bool AGAIN>
__global__ void round_kernel(const float *__restrict__ acc, T *__restrict__ out, int64_t n, OnlyIf only_if) {
    start_after_previous();
    if (AGAIN && !only_if.holds()) return;
    // Eight numbers a thread and store, two stores in flight (blocks for all of it, or fewer that mostly have nothing to do).  Bound
    // by memory: 150 000 x 64 takes 7.6 us after its convolution, and took 10.9 with four numbers a thread and a store for each.
    const int64_t threads = (int64_t)gridDim.x * blockDim.x, x0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if ((uintptr_t)out % 16 == 0) {
        static_assert(sizeof(T) == 2, "eight numbers to 16 bytes");
        auto eight = [&](int64_t at, const float4 &lo, const float4 &hi) {
            uint4 o;
            T *e = reinterpret_cast<T *>(&o);
            e[0] = from_f32<T>(lo.x), e[1] = from_f32<T>(lo.y), e[2] = from_f32<T>(lo.z), e[3] = from_f32<T>(lo.w);
            e[4] = from_f32<T>(hi.x), e[5] = from_f32<T>(hi.y), e[6] = from_f32<T>(hi.z), e[7] = from_f32<T>(hi.w);
            reinterpret_cast<uint4 *>(out)[at] = o;
        };
        const float4 *src = reinterpret_cast<const float4 *>(acc);
        const int64_t eights = n / 8;
        int64_t t = x0;
        for (; t + threads < eights; t += 2 * threads) {
            const float4 a = src[2 * t], b = src[2 * t + 1], c = src[2 * (t + threads)], d = src[2 * (t + threads) + 1];
            eight(t, a, b), eight(t + threads, c, d);
        }
        for (; t < eights; t += threads) eight(t, src[2 * t], src[2 * t + 1]);
        for (int64_t i = eights * 8 + x0; i < n; i += threads) out[i] = from_f32<T>(acc[i]);
    } else {
        for (int64_t i = x0; i < n; i += threads) out[i] = from_f32<T>(acc[i]);
    }
}

template <typename T>
int mvmr_generic_t(const MvmrArgs &a, cudaStream_t stream) {
    const T *W = (const T *)a.weight, *feat = (const T *)a.feat;
    if (a.seg_offs) {
        return mvmr_sorted_fma(a, stream);
    } else {
        unsigned blocks = (unsigned)((a.T + 7) / 8);
        if (a.transpose)
            mvmr_unsorted_kernel<T, true><<<blocks, 256, 0, stream>>>(W, feat, a.gather, a.scatter, a.tap_idx, a.acc, a.T, a.K, a.G, a.C, a.M, a.reverse);
        else
            mvmr_unsorted_kernel<T, false><<<blocks, 256, 0, stream>>>(W, feat, a.gather, a.scatter, a.tap_idx, a.acc, a.T, a.K, a.G, a.C, a.M, a.reverse);
    }
    PCX_LAUNCH_CHECK();
    return PCX_OK;
}

template <typename T>
int vvor_generic_t(const VvorArgs &a, cudaStream_t stream) {
    const T *A = (const T *)a.a, *B = (const T *)a.b;
    if (a.seg_offs) {
        return vvor_sorted_fma(a, stream);
    } else {
        unsigned blocks = (unsigned)((a.T + 7) / 8);
        vvor_unsorted_kernel<T><<<blocks, 256, 0, stream>>>(A, a.a_idx, B, a.b_idx, a.o_idx, a.acc, a.T, a.G, a.Ma, a.Cb);
    }
    PCX_LAUNCH_CHECK();
    return PCX_OK;
}

}  // namespace

int mvmr_generic(const MvmrArgs &a, cudaStream_t stream) {
    switch (a.dtype) {
        case PCX_F32: return mvmr_generic_t<float>(a, stream);
        case PCX_F16: return mvmr_generic_t<__half>(a, stream);
        case PCX_BF16: return mvmr_generic_t<__nv_bfloat16>(a, stream);
    }
    PCX_FAIL(PCX_E_DTYPE, "unsupported dtype %d", a.dtype);
}

int vvor_generic(const VvorArgs &a, cudaStream_t stream) {
    switch (a.dtype) {
        case PCX_F32: return vvor_generic_t<float>(a, stream);
        case PCX_F16: return vvor_generic_t<__half>(a, stream);
        case PCX_BF16: return vvor_generic_t<__nv_bfloat16>(a, stream);
    }
    PCX_FAIL(PCX_E_DTYPE, "unsupported dtype %d", a.dtype);
}

int round_accumulator(const float *acc, void *out, int64_t n, int dtype, cudaStream_t stream, OnlyIf only_if) {
    if (n == 0) return PCX_OK;
    unsigned blocks = (unsigned)((n / 16 + 255) / 256 + 1);
    const bool again = only_if.words != nullptr;
    if (again) blocks = std::min(blocks, (unsigned)num_sms() * 4);
    if (dtype == PCX_F16) launch_after((again ? round_kernel<__half, true> : round_kernel<__half, false>), blocks, 256, 0, stream, acc, (__half *)out, n, only_if);
    else if (dtype == PCX_BF16) launch_after((again ? round_kernel<__nv_bfloat16, true> : round_kernel<__nv_bfloat16, false>), blocks, 256, 0, stream, acc, (__nv_bfloat16 *)out, n, only_if);
    else PCX_FAIL(PCX_E_DTYPE, "round_accumulator: dtype %d", dtype);
    PCX_LAUNCH_CHECK();
    return PCX_OK;
}

}  // namespace pcx
