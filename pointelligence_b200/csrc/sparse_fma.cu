// CUDA-core engines for tap-sorted triplets: fp32 operands, and whatever the tensor engines do not take.  IEEE
// fp32 multiply-add in the order of the contraction, one fp32 accumulator in global memory.
//
// Both kernels walk contiguous ranges of chunks of tap-sorted triplets; a chunk's rows are gathered into shared
// memory by 16-byte cp.async (several CTAs per SM cover each other's latency, as in the tensor engines) and every
// thread keeps a register tile large enough that shared memory delivers operands faster than the FMA pipe takes
// them: 8 x 4 sums per thread for MVMR (12 vector loads per 128 multiply-adds), 8 x 8 for VVOR (4 per 64).  The
// 4 x 4 tiles with scalar loads and scalar atomics that these replace ran at a tenth of the FMA rate.
#include <algorithm>
#include <type_traits>

#include "sparse_kernels.cuh"
#include "tcgen05.cuh"

namespace pcx {
namespace {

using namespace tc;

constexpr int TABLE_TAPS = 1024;   // taps whose chunk table a CTA builds in shared memory; more: a global table

__device__ __forceinline__ float4 lds_f4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
    return v;
}
__device__ __forceinline__ void red_add_v4(float *addr, float4 v) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(addr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
__device__ __forceinline__ void sts_f32(uint32_t addr, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory"); }

// `rows` rows of `width` elements (columns [c0, c0 + N) of rows `idx`, `pitch` apart) into an fp32 tile of row pitch
// TP floats; columns and rows without a source become zeros.  VEC: 16-byte copies (fp32, everything aligned).
template <typename T, int N, int TP, int ROWS, bool VEC>
__device__ __forceinline__ void gather_f32(uint32_t tile, const T *__restrict__ src, const int32_t *idx, int rows, int c0, int width,
                                           int64_t pitch, int tid, int nthreads) {
    if (VEC) {
        constexpr int PR = N / 4;
        for (int e = tid; e < ROWS * PR; e += nthreads) {
            const int r = e / PR, c = (e - r * PR) * 4;
            const bool ok = r < rows && c0 + c < width;
            cp_async16_zfill(tile + (uint32_t)(r * TP + c) * 4, ok ? (const void *)(src + idx[r] * pitch + c0 + c) : (const void *)src, ok ? 16u : 0u);
        }
    } else {
        for (int e = tid; e < ROWS * N; e += nthreads) {
            const int r = e / N, c = e - r * N;
            sts_f32(tile + (uint32_t)(r * TP + c) * 4, r < rows && c0 + c < width ? to_f32(src[idx[r] * pitch + c0 + c]) : 0.f);
        }
    }
}

// --------------------------------------------------------------------- MVMR ----
constexpr int MC = 128;      // triplets per chunk
constexpr int MK = 32;       // contraction slice
constexpr int MXP = MK + 4;  // row pitch of the gathered tile: neighbouring rows four banks apart
constexpr int WPAD = 4;      // the same for the rows of the weight slices, which a transposed weight fills column by column

struct MvmrFmaParams {
    const int32_t *gather, *scatter;
    const int64_t *seg;
    const int32_t *table;   // chunk table in global memory, or null
    float *acc;
    int K, G, C, M, inw, outw, reverse, vec_in, vec_out;
    int keep;               // the whole weight tile stays in shared memory while the tap lasts
};

// CTAs per SM: the grids are sized for what is resident at once
constexpr int mvmr_ctas(int nt) { return nt == 32 ? 5 : 2; }
constexpr int VVOR_CTAS = 4;

template <typename T, bool TRANSPOSE, int NT>
__global__ void __launch_bounds__(NT * 4, mvmr_ctas(NT)) mvmr_fma_kernel(const T *__restrict__ W, const T *__restrict__ feat, MvmrFmaParams p) {
    start_after_previous();
    constexpr int THREADS = NT * 4, WP = NT + WPAD;
    extern __shared__ __align__(16) uint8_t raw[];
    __shared__ int32_t s_cum[TABLE_TAPS + 1], s_warp_sums[THREADS / 32], s_gather[MC], s_scatter[MC];
    const uint32_t xs = smem_u32(raw), ws = xs + MC * MXP * 4;   // gathered tile | weight slices [slice][MK][WP]
    const int tid = threadIdx.x, tx = tid % (NT / 4), ty = tid / (NT / 4);   // columns 4 tx .., rows ty + 16 r
    const int32_t *cum = p.table;
    if (!cum) {
        build_chunk_table<MC>(p.seg, p.K, s_cum, s_warp_sums);
        cum = s_cum;
    }
    const int g = blockIdx.z, n0 = blockIdx.y * NT;
    feat += (int64_t)g * p.inw;
    float *acc = p.acc + (int64_t)g * p.outw + n0;
    const int64_t in_pitch = (int64_t)p.G * p.inw, out_pitch = (int64_t)p.G * p.outw;
    const int total = cum[p.K], per = (total + gridDim.x - 1) / gridDim.x, lo = blockIdx.x * per, hi = min(total, lo + per);
    const int slices = (p.inw + MK - 1) / MK;
    if (lo >= hi) return;
    ChunkCursorT<MC> cur;
    cur.seek(cum, p.seg, p.K, lo);
    int loaded = -1, pre_g = 0, pre_s = 0;
    auto fetch = [&](int chunk) {   // indices of a chunk into registers
        if (tid < MC && tid < cur.rows(chunk)) pre_g = p.gather[cur.first(chunk) + tid], pre_s = p.scatter[cur.first(chunk) + tid];
    };
    auto load_weight = [&](int tap, int slice, uint32_t dst) {
        const T *w = W + ((int64_t)(p.reverse ? p.K - 1 - tap : tap) * p.G + g) * p.C * p.M;
        for (int e = tid; e < MK * NT; e += THREADS) {
            int kk, n;   // consecutive threads along the rows of W
            if (TRANSPOSE) n = e / MK, kk = e % MK; else kk = e / NT, n = e % NT;
            const int k = slice * MK + kk;
            const bool ok = k < p.inw && n0 + n < p.outw;
            sts_f32(dst + (uint32_t)(kk * WP + n) * 4, ok ? to_f32(w[TRANSPOSE ? (int64_t)(n0 + n) * p.M + k : (int64_t)k * p.M + n0 + n]) : 0.f);
        }
    };
    fetch(lo);
    for (int chunk = lo; chunk < hi; ++chunk) {
        const int rows = cur.rows(chunk), tap = cur.tap;
        __syncthreads();   // the last chunk's tiles and indices have been read
        if (tid < MC) s_gather[tid] = pre_g, s_scatter[tid] = pre_s;
        __syncthreads();
        if (chunk + 1 < hi) {
            cur.advance(cum, p.seg, p.K, chunk + 1);
            fetch(chunk + 1);
        }
        float4 s[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) s[r] = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int slice = 0; slice < slices; ++slice) {
            if (slice) __syncthreads();
            const uint32_t w_at = ws + (p.keep ? (uint32_t)slice * (MK * WP * 4) : 0u);
            if (p.vec_in) gather_f32<T, MK, MXP, MC, sizeof(T) == 4>(xs, feat, s_gather, rows, slice * MK, p.inw, in_pitch, tid, THREADS);
            else gather_f32<T, MK, MXP, MC, false>(xs, feat, s_gather, rows, slice * MK, p.inw, in_pitch, tid, THREADS);
            if (!p.keep || loaded != tap) load_weight(tap, slice, w_at);
            cp_async_commit();
            cp_async_wait<0>();
            __syncthreads();
            const int depth = min(MK, p.inw - slice * MK);   // (zeros beyond; whole fours are multiplied)
            const uint32_t x_at = xs + (uint32_t)ty * MXP * 4, wt = w_at + (uint32_t)tx * 16;
            // Short chunks (a few triplets a tap) multiply the sixteens of rows they have: 300 rows of 512 channels over
            // 125 taps of 12 triplets, 356 -> 209 us.
            auto multiply = [&](auto row_steps) {
                constexpr int R = decltype(row_steps)::value;
#pragma unroll 1
                for (int k = 0; k < depth; k += 4) {
                    float4 w[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) w[q] = lds_f4(wt + (uint32_t)((k + q) * WP) * 4);
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const float4 x = lds_f4(x_at + (uint32_t)(16 * r * MXP + k) * 4);
                        s[r].x = __fmaf_rn(x.x, w[0].x, s[r].x), s[r].y = __fmaf_rn(x.x, w[0].y, s[r].y);
                        s[r].z = __fmaf_rn(x.x, w[0].z, s[r].z), s[r].w = __fmaf_rn(x.x, w[0].w, s[r].w);
                        s[r].x = __fmaf_rn(x.y, w[1].x, s[r].x), s[r].y = __fmaf_rn(x.y, w[1].y, s[r].y);
                        s[r].z = __fmaf_rn(x.y, w[1].z, s[r].z), s[r].w = __fmaf_rn(x.y, w[1].w, s[r].w);
                        s[r].x = __fmaf_rn(x.z, w[2].x, s[r].x), s[r].y = __fmaf_rn(x.z, w[2].y, s[r].y);
                        s[r].z = __fmaf_rn(x.z, w[2].z, s[r].z), s[r].w = __fmaf_rn(x.z, w[2].w, s[r].w);
                        s[r].x = __fmaf_rn(x.w, w[3].x, s[r].x), s[r].y = __fmaf_rn(x.w, w[3].y, s[r].y);
                        s[r].z = __fmaf_rn(x.w, w[3].z, s[r].z), s[r].w = __fmaf_rn(x.w, w[3].w, s[r].w);
                    }
                }
            };
            if (rows > 64) multiply(std::integral_constant<int, 8>());
            else if (rows > 32) multiply(std::integral_constant<int, 4>());
            else if (rows > 16) multiply(std::integral_constant<int, 2>());
            else multiply(std::integral_constant<int, 1>());
        }
        loaded = tap;
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const int row = ty + 16 * r, c = 4 * tx;
            if (row >= rows || n0 + c >= p.outw) continue;
            float *dst = acc + s_scatter[row] * out_pitch + c;
            if (p.vec_out) {
                red_add_v4(dst, s[r]);
            } else {
                const float v[4] = {s[r].x, s[r].y, s[r].z, s[r].w};
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (n0 + c + e < p.outw) atomicAdd(dst + e, v[e]);
            }
        }
    }
}

// --------------------------------------------------------------------- VVOR ----
constexpr int VC = 64;   // triplets per chunk

struct VvorFmaParams {
    const int32_t *a_idx, *b_idx;
    const int64_t *seg;
    const int32_t *table;
    float *acc;
    int n_o, G, Ma, Cb, vec_a, vec_b, vec_out;
};

// Tile of TE x TE sums, 8 x 8 per thread; TE = 32 needs 16 threads, so eight groups of threads share the triplets of a
// chunk (two groups for TE = 64) and each adds its own sums when the tap ends.
template <typename T, int TE>
__global__ void __launch_bounds__(128, VVOR_CTAS) vvor_fma_kernel(const T *__restrict__ A, const T *__restrict__ B, VvorFmaParams p) {
    start_after_previous();
    constexpr int TP = TE + 4, PER = (TE / 8) * (TE / 8), TEAMS = 128 / PER;
    extern __shared__ __align__(16) uint8_t raw[];
    __shared__ int32_t s_cum[TABLE_TAPS + 1], s_warp_sums[4], s_a[VC], s_b[VC];
    const uint32_t at = smem_u32(raw), bt = at + VC * TP * 4;
    const int tid = threadIdx.x, team = tid / PER, tx = tid % (TE / 8), ty = tid % PER / (TE / 8);
    const int32_t *cum = p.table;
    if (!cum) {
        build_chunk_table<VC>(p.seg, p.n_o, s_cum, s_warp_sums);
        cum = s_cum;
    }
    const int ct = (p.Cb + TE - 1) / TE, c0 = (int)blockIdx.y % ct * TE, m0 = (int)blockIdx.y / ct * TE, g = blockIdx.z;
    const int64_t a_pitch = (int64_t)p.G * p.Ma, b_pitch = (int64_t)p.G * p.Cb;
    A += (int64_t)g * p.Ma, B += (int64_t)g * p.Cb;
    const int total = cum[p.n_o], per = (total + gridDim.x - 1) / gridDim.x, lo = blockIdx.x * per, hi = min(total, lo + per);
    if (lo >= hi) return;
    ChunkCursorT<VC> cur;
    cur.seek(cum, p.seg, p.n_o, lo);
    int pre_a = 0, pre_b = 0;
    auto fetch = [&](int chunk) {
        if (tid < VC && tid < cur.rows(chunk)) pre_a = p.a_idx[cur.first(chunk) + tid], pre_b = p.b_idx[cur.first(chunk) + tid];
    };
    fetch(lo);
    // columns of a thread: 4 t .. and TE/2 + 4 t .. (neighbouring threads read neighbouring vectors)
    float s[8][8];
    auto clear = [&]() {
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) s[i][j] = 0.f;
    };
    clear();
    for (int chunk = lo; chunk < hi; ++chunk) {
        const int rows = cur.rows(chunk), o = cur.tap;
        const bool last = chunk + 1 == hi || cur.last_of_tap(chunk);
        __syncthreads();
        if (tid < VC) s_a[tid] = pre_a, s_b[tid] = pre_b;
        __syncthreads();
        if (p.vec_a) gather_f32<T, TE, TP, VC, sizeof(T) == 4>(at, A, s_a, rows, m0, p.Ma, a_pitch, tid, 128);
        else gather_f32<T, TE, TP, VC, false>(at, A, s_a, rows, m0, p.Ma, a_pitch, tid, 128);
        if (p.vec_b) gather_f32<T, TE, TP, VC, sizeof(T) == 4>(bt, B, s_b, rows, c0, p.Cb, b_pitch, tid, 128);
        else gather_f32<T, TE, TP, VC, false>(bt, B, s_b, rows, c0, p.Cb, b_pitch, tid, 128);
        cp_async_commit();
        if (chunk + 1 < hi) {
            cur.advance(cum, p.seg, p.n_o, chunk + 1);
            fetch(chunk + 1);
        }
        cp_async_wait<0>();
        __syncthreads();
#pragma unroll 1
        for (int t = team; t < rows; t += TEAMS) {
            const uint32_t ra = at + (uint32_t)(t * TP + 4 * ty) * 4, rb = bt + (uint32_t)(t * TP + 4 * tx) * 4;
            const float4 a0 = lds_f4(ra), a1 = lds_f4(ra + TE * 2), b0 = lds_f4(rb), b1 = lds_f4(rb + TE * 2);
            const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w}, bv[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) s[i][j] = __fmaf_rn(av[i], bv[j], s[i][j]);
        }
        if (!last) continue;
        float *dst = p.acc + ((int64_t)o * p.G + g) * p.Ma * p.Cb;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int m = m0 + (i < 4 ? 4 * ty + i : TE / 2 + 4 * ty + i - 4);
            if (m >= p.Ma) continue;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int c = c0 + h * (TE / 2) + 4 * tx;
                float *d = dst + (int64_t)m * p.Cb + c;
                if (p.vec_out) {
                    if (c < p.Cb) red_add_v4(d, make_float4(s[i][4 * h], s[i][4 * h + 1], s[i][4 * h + 2], s[i][4 * h + 3]));
                } else {
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (c + e < p.Cb) atomicAdd(d + e, s[i][4 * h + e]);
                }
            }
        }
        clear();
    }
}

// --------------------------------------------------------------------- host ----
int granted_smem(const void *kernel, size_t smem) {   // above 48 KB, its static 5 KB included, a kernel has to ask
    if (smem <= 42 * 1024) return PCX_OK;
    PCX_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 128 * 1024));
    return PCX_OK;
}
bool aligned16(const void *p) { return ((uintptr_t)p & 15) == 0; }

template <typename T, bool TRANSPOSE, int NT>
int launch_mvmr(const MvmrArgs &a, MvmrFmaParams p, cudaStream_t stream) {
    const int slices = (p.inw + MK - 1) / MK;
    p.keep = slices * MK * NT * 4 <= 64 * 1024;
    const size_t smem = (size_t)MC * MXP * 4 + (size_t)(p.keep ? slices : 1) * MK * (NT + WPAD) * 4;
    if (int rc = granted_smem((const void *)mvmr_fma_kernel<T, TRANSPOSE, NT>, smem)) return rc;
    const int64_t tiles = (int64_t)((p.outw + NT - 1) / NT) * p.G;
    const int occ = (int)std::max<size_t>(1, std::min<size_t>(mvmr_ctas(NT), (size_t)220 * 1024 / (smem + 6 * 1024)));
    const int64_t upper = a.T / MC + a.K + 1;
    const dim3 grid((unsigned)std::min<int64_t>(upper, std::max<int64_t>(1, (int64_t)occ * num_sms() / tiles)), (unsigned)(tiles / p.G), (unsigned)p.G);
    prof_begin(TRANSPOSE ? "mvmr_fma_kernel(dgrad)" : "mvmr_fma_kernel(fwd)", stream);
    launch_after(mvmr_fma_kernel<T, TRANSPOSE, NT>, grid, NT * 4, smem, stream, (const T *)a.weight, (const T *)a.feat, p);
    prof_end(stream);
    PCX_LAUNCH_CHECK();
    return PCX_OK;
}

template <typename T, int TE>
int launch_vvor(const VvorArgs &a, const VvorFmaParams &p, cudaStream_t stream) {
    const size_t smem = (size_t)2 * VC * (TE + 4) * 4;
    if (int rc = granted_smem((const void *)vvor_fma_kernel<T, TE>, smem)) return rc;
    const int64_t tiles = (int64_t)((p.Ma + TE - 1) / TE) * ((p.Cb + TE - 1) / TE) * p.G;
    int64_t upper = a.T / VC + a.n_o + 1;
    // Every team of every CTA adds its sums to those of a tap.  With few taps and a full tile these additions meet in the
    // same cells of the L2: 256 CTAs a tap, where there is one tap of 32 x 32 channels: 20 000 triplets 61 -> 29 us,
    // 100 000 78 -> 47, 400 000 90 -> 84.  Smaller tiles add less and lose more to fewer CTAs (3 x 32, 400 000: 72 -> 98).
    if (TE == 32 && a.Ma * a.Cb > 512) upper = std::min(upper, a.n_o * 256);
    const dim3 grid((unsigned)std::min<int64_t>(upper, std::max<int64_t>(1, (int64_t)VVOR_CTAS * num_sms() / tiles)), (unsigned)(tiles / p.G), (unsigned)p.G);
    prof_begin("vvor_fma_kernel", stream);
    launch_after(vvor_fma_kernel<T, TE>, grid, 128, smem, stream, (const T *)a.a, (const T *)a.b, p);
    prof_end(stream);
    PCX_LAUNCH_CHECK();
    return PCX_OK;
}

template <typename T>
int mvmr_t(const MvmrArgs &a, cudaStream_t stream) {
    MvmrFmaParams p = {};
    p.gather = a.gather, p.scatter = a.scatter, p.seg = a.seg_offs, p.acc = a.acc;
    p.K = a.K, p.G = a.G, p.C = a.C, p.M = a.M, p.reverse = a.reverse;
    p.inw = a.transpose ? a.M : a.C, p.outw = a.transpose ? a.C : a.M;
    p.vec_in = sizeof(T) == 4 && p.inw % 4 == 0 && aligned16(a.feat);
    p.vec_out = p.outw % 4 == 0 && aligned16(a.acc);
    if (a.K > TABLE_TAPS) {
        chunk_table_kernel<<<1, 128, 0, stream>>>(a.seg_offs, a.K, MC, a.chunk_table);
        PCX_LAUNCH_CHECK();
        p.table = a.chunk_table;
    }
    if (a.transpose) return p.outw <= 32 ? launch_mvmr<T, true, 32>(a, p, stream) : launch_mvmr<T, true, 64>(a, p, stream);
    return p.outw <= 32 ? launch_mvmr<T, false, 32>(a, p, stream) : launch_mvmr<T, false, 64>(a, p, stream);
}

template <typename T>
int vvor_t(const VvorArgs &a, cudaStream_t stream) {
    VvorFmaParams p = {};
    p.a_idx = a.a_idx, p.b_idx = a.b_idx, p.seg = a.seg_offs, p.acc = a.acc;
    p.n_o = (int)a.n_o, p.G = a.G, p.Ma = a.Ma, p.Cb = a.Cb;
    p.vec_a = sizeof(T) == 4 && a.Ma % 4 == 0 && aligned16(a.a), p.vec_b = sizeof(T) == 4 && a.Cb % 4 == 0 && aligned16(a.b);
    p.vec_out = a.Cb % 4 == 0 && aligned16(a.acc);
    if (a.n_o > TABLE_TAPS) {
        chunk_table_kernel<<<1, 128, 0, stream>>>(a.seg_offs, (int)a.n_o, VC, a.chunk_table);
        PCX_LAUNCH_CHECK();
        p.table = a.chunk_table;
    }
    return a.Ma <= 32 && a.Cb <= 32 ? launch_vvor<T, 32>(a, p, stream) : launch_vvor<T, 64>(a, p, stream);
}

}  // namespace

int mvmr_sorted_fma(const MvmrArgs &a, cudaStream_t stream) {
    switch (a.dtype) {
        case PCX_F32: return mvmr_t<float>(a, stream);
        case PCX_F16: return mvmr_t<__half>(a, stream);
        case PCX_BF16: return mvmr_t<__nv_bfloat16>(a, stream);
    }
    PCX_FAIL(PCX_E_DTYPE, "unsupported dtype %d", a.dtype);
}

int vvor_sorted_fma(const VvorArgs &a, cudaStream_t stream) {
    switch (a.dtype) {
        case PCX_F32: return vvor_t<float>(a, stream);
        case PCX_F16: return vvor_t<__half>(a, stream);
        case PCX_BF16: return vvor_t<__nv_bfloat16>(a, stream);
    }
    PCX_FAIL(PCX_E_DTYPE, "unsupported dtype %d", a.dtype);
}

}  // namespace pcx
