// Column-wise helpers of the convolution layers: the bias gradient (column sums of the output
// gradient) and the accumulator of a biased layer (every row starts as the bias).
#include <algorithm>

#include "common.cuh"

namespace pcx {
namespace {

constexpr int CS_THREADS = 256;
constexpr int CS_BLOCKS_PER_SM = 4;
constexpr int CS_UNROLL = 4;   // rows a thread has in flight

template <typename T, int V>
struct Piece;   // V elements moved as one load
template <>
struct Piece<float, 4> { typedef float4 type; };
template <>
struct Piece<__half, 8> { typedef uint4 type; };
template <>
struct Piece<__nv_bfloat16, 8> { typedef uint4 type; };
template <typename T>
struct Piece<T, 1> { typedef T type; };

// Partial column sums of a contiguous range of rows per block, fp32.  A thread owns one piece of V
// columns and walks down the rows; the rows of a block are folded in shared memory in a fixed order, so
// the result does not depend on scheduling.  Bound by DRAM: 150 000 x 64 bf16 (19 MB) is read in about
// 5 us on B200 where the generic reduction this replaces took 53 us, and 200 000 x 256 in 19 against 113.
template <typename T, int V>
__global__ void __launch_bounds__(CS_THREADS) column_partial_kernel(const T *__restrict__ x, int64_t N, int C, int64_t rows_per_block,
                                                                    float *__restrict__ partial) {
    start_after_previous();
    __shared__ float fold[CS_THREADS * V];
    const int pieces = C / V, per_pass = min(pieces, CS_THREADS), lanes = CS_THREADS / per_pass;
    const int piece0 = threadIdx.x % per_pass, lane = threadIdx.x / per_pass;
    const int64_t r0 = blockIdx.x * rows_per_block, r1 = min(N, r0 + rows_per_block);
    typedef typename Piece<T, V>::type P;
    for (int p0 = 0; p0 < pieces; p0 += per_pass) {
        const int piece = p0 + piece0;
        float s[V];
#pragma unroll
        for (int v = 0; v < V; ++v) s[v] = 0.f;
        if (piece < pieces && lane < lanes) {
            const T *col = x + (int64_t)piece * V;
            int64_t r = r0 + lane;
            for (; r + (int64_t)(CS_UNROLL - 1) * lanes < r1; r += (int64_t)CS_UNROLL * lanes) {
                P q[CS_UNROLL];
#pragma unroll
                for (int u = 0; u < CS_UNROLL; ++u) q[u] = *reinterpret_cast<const P *>(col + (r + (int64_t)u * lanes) * C);
#pragma unroll
                for (int u = 0; u < CS_UNROLL; ++u) {
                    const T *e = reinterpret_cast<const T *>(&q[u]);
#pragma unroll
                    for (int v = 0; v < V; ++v) s[v] += to_f32(e[v]);
                }
            }
            for (; r < r1; r += lanes) {
                const P q = *reinterpret_cast<const P *>(col + r * C);
                const T *e = reinterpret_cast<const T *>(&q);
#pragma unroll
                for (int v = 0; v < V; ++v) s[v] += to_f32(e[v]);
            }
        }
#pragma unroll
        for (int v = 0; v < V; ++v) fold[threadIdx.x * V + v] = s[v];
        __syncthreads();
        for (int c = threadIdx.x; c < per_pass * V; c += CS_THREADS) {
            if (p0 * V + c < C) {
                float t = 0.f;
                for (int l = 0; l < lanes; ++l) t += fold[(l * per_pass) * V + c];
                partial[(int64_t)blockIdx.x * C + p0 * V + c] = t;
            }
        }
        __syncthreads();
    }
}

// One warp per column: the partial sums of all blocks, rounded once.
template <typename T>
__global__ void column_final_kernel(const float *__restrict__ partial, int blocks, int C, T *__restrict__ out) {
    start_after_previous();
    const int c = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (c >= C) return;
    float s = 0.f;
    for (int b = lane; b < blocks; b += 32) s += partial[(int64_t)b * C + c];
#pragma unroll
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) out[c] = from_f32<T>(s);
}

int column_blocks(int64_t N, int C) {
    // enough rows per block that its fold is small against its reading
    const int64_t by_rows = (N * C + 32767) / 32768;
    return (int)std::max<int64_t>(1, std::min<int64_t>(by_rows, (int64_t)CS_BLOCKS_PER_SM * num_sms()));
}

template <typename T, int V>
int launch_column_sums(const void *x, void *out, int64_t N, int C, float *partial, cudaStream_t stream) {
    const int blocks = column_blocks(N, C);
    const int64_t rows = (N + blocks - 1) / blocks;
    if (C % V == 0 && (uintptr_t)x % 16 == 0)
        launch_after(column_partial_kernel<T, V>, blocks, CS_THREADS, 0, stream, (const T *)x, N, C, rows, partial);
    else
        launch_after(column_partial_kernel<T, 1>, blocks, CS_THREADS, 0, stream, (const T *)x, N, C, rows, partial);
    PCX_LAUNCH_CHECK();
    launch_after(column_final_kernel<T>, (C + 7) / 8, 256, 0, stream, partial, blocks, C, (T *)out);
    PCX_LAUNCH_CHECK();
    return PCX_OK;
}

// acc[r][c] = bias[c], or zero; W divides the row width, so a thread's W columns lie in one row.  Bound by the stores: with a
// 64-bit remainder for every one of them, 150 000 x 64 took 8.1 us instead of some 5 (a memset of that size: 4.6, and no kernel
// can be set up behind it).
template <typename T, int W, bool AGAIN>
__global__ void fill_rows_kernel(float *__restrict__ acc, const T *__restrict__ bias, int64_t n, int width, OnlyIf only_if) {
    start_after_previous();
    if (AGAIN && !only_if.holds()) return;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x * W;
    int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * W;
    int c = bias ? (int)(i % width) : 0;
    const int turn = bias ? (int)(stride % width) : 0;   // columns a thread moves on by: none where its stride is whole rows
    float v[W];
    auto value = [&]() {
#pragma unroll
        for (int e = 0; e < W; ++e) v[e] = bias && i < n ? to_f32(bias[c + e]) : 0.f;
    };
    value();
#pragma unroll 4
    for (; i < n; i += stride) {
        if constexpr (W == 4) *reinterpret_cast<float4 *>(acc + i) = make_float4(v[0], v[1], v[2], v[3]);
        else acc[i] = v[0];
        if (turn) {
            c += turn;
            if (c >= width) c -= width;
            value();
        }
    }
}

template <typename T>
int launch_fill(float *acc, const void *bias, int64_t rows, int width, OnlyIf only_if, cudaStream_t stream) {
    const int64_t n = rows * width;
    const int w = (bias ? width : n) % 4 == 0 && (uintptr_t)acc % 16 == 0 ? 4 : 1;
    const unsigned grid = (unsigned)std::min<int64_t>((n / w + 255) / 256, (int64_t)num_sms() * (only_if.words ? 4 : 16));
    const bool again = only_if.words != nullptr;
    if (w == 4) launch_after((again ? fill_rows_kernel<T, 4, true> : fill_rows_kernel<T, 4, false>), grid, 256, 0, stream, acc, (const T *)bias, n, width, only_if);
    else launch_after((again ? fill_rows_kernel<T, 1, true> : fill_rows_kernel<T, 1, false>), grid, 256, 0, stream, acc, (const T *)bias, n, width, only_if);
    PCX_LAUNCH_CHECK();
    return PCX_OK;
}

// dst[o][r][c] = src[o][r][c] where it exists, else zero, for 16-bit elements: rows and columns of a matrix
// are added (padding to the tensor core's channel counts) or dropped.  V output columns per thread.
template <int V>
__global__ void reshape16_kernel(const uint16_t *__restrict__ src, uint16_t *__restrict__ dst, int64_t pieces, int r_in, int c_in, int r_out,
                                 int c_out) {
    start_after_previous();
    const int64_t x = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (x >= pieces) return;
    const int per_row = c_out / V;
    const int64_t row = x / per_row, o = row / r_out;
    const int c = (int)(x - row * per_row) * V, r = (int)(row - o * r_out);
    uint16_t v[V];
#pragma unroll
    for (int e = 0; e < V; ++e) v[e] = r < r_in && c + e < c_in ? __ldg(src + (o * r_in + r) * c_in + c + e) : (uint16_t)0;
    if (V == 8) *reinterpret_cast<uint4 *>(dst + row * c_out + c) = *reinterpret_cast<const uint4 *>(v);
    else dst[row * c_out + c] = v[0];
}

}  // namespace

// Every row of the accumulator starts as `bias` (zeros when null): the bias of a layer costs the store
// that clearing the accumulator costs anyway, not a pass over its output.
int clear_accumulator(float *acc, const void *bias, int64_t rows, int width, int dtype, cudaStream_t stream, OnlyIf only_if) {
    switch (dtype) {
        case PCX_F32: return launch_fill<float>(acc, bias, rows, width, only_if, stream);
        case PCX_F16: return launch_fill<__half>(acc, bias, rows, width, only_if, stream);
        case PCX_BF16: return launch_fill<__nv_bfloat16>(acc, bias, rows, width, only_if, stream);
    }
    PCX_FAIL(PCX_E_DTYPE, "unsupported dtype %d", dtype);
}

}  // namespace pcx

using namespace pcx;

extern "C" {

int pcx_reshape16(const void *d_src, void *d_dst, int64_t outer, int rows_in, int cols_in, int rows_out, int cols_out, void *stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    if (outer < 0 || rows_in <= 0 || cols_in <= 0 || rows_out <= 0 || cols_out <= 0) PCX_FAIL(PCX_E_ARG, "pcx_reshape16: bad sizes");
    if (outer == 0) return PCX_OK;
    if (!d_src || !d_dst) PCX_FAIL(PCX_E_ARG, "pcx_reshape16: null pointer");
    const bool wide = cols_out % 8 == 0 && (uintptr_t)d_dst % 16 == 0;
    const int64_t pieces = outer * rows_out * (cols_out / (wide ? 8 : 1));
    if ((pieces + 255) / 256 > INT32_MAX) PCX_FAIL(PCX_E_UNSUPPORTED, "pcx_reshape16: too large");
    const unsigned grid = (unsigned)((pieces + 255) / 256);
    if (wide) launch_after(reshape16_kernel<8>, grid, 256, 0, stream, (const uint16_t *)d_src, (uint16_t *)d_dst, pieces, rows_in, cols_in, rows_out, cols_out);
    else launch_after(reshape16_kernel<1>, grid, 256, 0, stream, (const uint16_t *)d_src, (uint16_t *)d_dst, pieces, rows_in, cols_in, rows_out, cols_out);
    PCX_LAUNCH_CHECK();
    return PCX_OK;
}

size_t pcx_column_sums_workspace_bytes(int64_t N, int C) {
    if (N < 0 || C <= 0) return 0;
    return align_up((size_t)column_blocks(N, C) * C * sizeof(float), 256);
}

int pcx_column_sums(const void *d_x, void *d_out, int64_t N, int C, int dtype, void *d_ws, size_t ws_bytes, void *stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    if (N < 0 || C <= 0) PCX_FAIL(PCX_E_ARG, "pcx_column_sums: bad sizes (N=%lld C=%d)", (long long)N, C);
    if ((N > 0 && !d_x) || !d_out || !d_ws) PCX_FAIL(PCX_E_ARG, "pcx_column_sums: null pointer");
    if (ws_bytes < pcx_column_sums_workspace_bytes(N, C)) PCX_FAIL(PCX_E_CAPACITY, "pcx_column_sums: workspace too small");
    switch (dtype) {
        case PCX_F32: return launch_column_sums<float, 4>(d_x, d_out, N, C, (float *)d_ws, stream);
        case PCX_F16: return launch_column_sums<__half, 8>(d_x, d_out, N, C, (float *)d_ws, stream);
        case PCX_BF16: return launch_column_sums<__nv_bfloat16, 8>(d_x, d_out, N, C, (float *)d_ws, stream);
    }
    PCX_FAIL(PCX_E_DTYPE, "pcx_column_sums: unsupported dtype %d", dtype);
}

}  // extern "C"
