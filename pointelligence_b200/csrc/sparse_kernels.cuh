// Argument blocks shared by the sparse-engine translation units.
#pragma once
#include "common.cuh"

namespace pcx {

struct MvmrArgs {
    const void *weight;      // (K,G,C,M)
    const void *feat;        // (n_feat, G*inw)
    const int32_t *gather;   // (T) rows of feat
    const int32_t *scatter;  // (T) rows of out
    const int64_t *seg_offs; // (K+1) or null
    const int32_t *tap_idx;  // (T) when seg_offs is null
    float *acc;              // (n_out, G*outw) fp32, zeroed by the caller
    void *out_rows;          // tensor engine, fan-in 1: the output itself, written row by row (acc unused)
    int32_t *chunk_table;    // (K+1) scratch of the CUDA-core engine
    int64_t T, n_feat, n_out;
    const void *bias;        // (G*outw) of dtype or null; only the fan-in 1 stores read it, elsewhere acc starts as it
    int K, G, C, M, transpose, dtype;
    int reverse;             // tap k uses weight K-1-k
    OnlyIf only_if;          // (tensor engine)
};

struct VvorArgs {
    const void *a;           // (n_a, G*Ma)
    const int32_t *a_idx;
    const void *b;           // (n_b, G*Cb)
    const int32_t *b_idx;
    const int64_t *seg_offs; // (n_o+1) or null
    const int32_t *o_idx;    // (T) when seg_offs is null
    float *acc;              // (n_o, G, Ma, Cb) fp32, zeroed by the caller
    void *out;               // tensor engine: the output itself, where every tap is completed by one block (acc unused); else null
    int32_t *chunk_table;    // (n_o+1) scratch
    int64_t T, n_a, n_b, n_o, fullest;   // triplets of the fullest o; negative: not known
    int G, Ma, Cb, dtype;
};

// Position of a CTA in the chunk sequence; the bounds of the current tap are
// kept in registers and reloaded only when the chunk index leaves the tap.
// The cumulative chunk table lives in shared memory (built by every CTA from
// the segment offsets), so no separate kernel and no global table are needed.
template <int CHR>
struct ChunkCursorT {
    int tap;
    int cum_lo, cum_hi;
    int64_t seg_lo, seg_hi;
    __device__ __forceinline__ void load(const int32_t *cum, const int64_t *__restrict__ seg) {
        cum_lo = cum[tap], cum_hi = cum[tap + 1];
        seg_lo = seg[tap], seg_hi = seg[tap + 1];
    }
    __device__ __forceinline__ void seek(const int32_t *cum, const int64_t *__restrict__ seg, int K, int chunk) {
        int lo = 0, hi = K;
        while (hi - lo > 1) {
            int mid = (lo + hi) >> 1;
            if (cum[mid] <= chunk) lo = mid; else hi = mid;
        }
        tap = lo;
        load(cum, seg);
    }
    __device__ __forceinline__ void advance(const int32_t *cum, const int64_t *__restrict__ seg, int K, int chunk) {
        if (chunk < cum_hi) return;
        while (tap + 1 < K && cum[tap + 1] <= chunk) ++tap;
        load(cum, seg);
    }
    __device__ __forceinline__ int64_t first(int chunk) const { return seg_lo + (int64_t)(chunk - cum_lo) * CHR; }
    __device__ __forceinline__ int rows(int chunk) const {
        int64_t left = seg_hi - first(chunk);
        return (int)(left < CHR ? left : CHR);
    }
    __device__ __forceinline__ bool last_of_tap(int chunk) const { return chunk + 1 >= cum_hi; }
};

// cum[k] = chunks of CHR triplets in the taps before k; all threads of the CTA call this.
template <int CHR>
__device__ __forceinline__ void build_chunk_table(const int64_t *__restrict__ seg, int K, int32_t *cum,
                                                  int32_t *warp_sums) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
    int32_t carry = 0;
    for (int base = 0; base < K; base += blockDim.x) {
        int k = base + tid;
        int32_t v = k < K ? (int32_t)((seg[k + 1] - seg[k] + CHR - 1) / CHR) : 0;
        int32_t inc = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int32_t n = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += n;
        }
        if (lane == 31) warp_sums[warp] = inc;
        __syncthreads();
        int32_t before = carry, all = carry;
        for (int w = 0; w < nwarps; ++w) {
            if (w < warp) before += warp_sums[w];
            all += warp_sums[w];
        }
        if (k < K) cum[k] = before + inc - v;
        carry = all;
        __syncthreads();
    }
    if (tid == 0) cum[K] = carry;
    __syncthreads();
}

__global__ void chunk_table_kernel(const int64_t *__restrict__ seg, int K, int L, int32_t *cum);

int mvmr_sorted_fma(const MvmrArgs &a, cudaStream_t stream);   // CUDA cores, tap-sorted triplets (sparse_fma.cu)
int vvor_sorted_fma(const VvorArgs &a, cudaStream_t stream);
int mvmr_generic(const MvmrArgs &a, cudaStream_t stream);
int vvor_generic(const VvorArgs &a, cudaStream_t stream);
int clear_accumulator(float *acc, const void *bias, int64_t rows, int width, int dtype, cudaStream_t stream, OnlyIf only_if = {});
int round_accumulator(const float *acc, void *out, int64_t n, int dtype, cudaStream_t stream, OnlyIf only_if = {});
constexpr int MAX_ODD = 1024;
int mvmr_planned(const void *d_weight, const void *d_feat, void *d_plan, size_t plan_bytes, const void *d_bias, void *d_out, int64_t T,
                 int64_t n_feat, int64_t n_out, int K, int groups, int C, int M, int flags, int dtype, int group_blocks,
                 int64_t multi_buckets, uint32_t *odd, int *n_odd, void *d_ws, size_t ws_bytes, void *stream);   // (mvmr_os.cu)

// Rows wider than 256 channels go through the tensor engines in equal parts of at most 256.
inline int parts_of(int width) { return (width + 255) / 256; }
inline bool splits_evenly(int width) { return width >= 16 && width % (16 * parts_of(width)) == 0; }

bool mvmr_tensor_supported(const MvmrArgs &a);
bool vvor_tensor_supported(const VvorArgs &a);
int64_t vvor_store_limit(int64_t n_o, int G, int Ma, int Cb);
bool vvor_stores(const VvorArgs &a);   // whether the tensor engine should store rows itself
int mvmr_tensor(const MvmrArgs &a, cudaStream_t stream);
int vvor_tensor(const VvorArgs &a, cudaStream_t stream);

}  // namespace pcx
