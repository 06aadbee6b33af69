// Fused layer normalisation over a ragged batch, with the residual add and the
// ReLU of a residual block folded into the same pass:
//
//   y = relu?( (x - mean_s) * rstd_s * weight + bias  (+ residual) )
//
// mean_s and rstd_s are the statistics of ALL elements (rows x channels) of
// sample s, computed in two passes exactly as the reference composes them
// (layers/norm.py:118-130: mean first, then the variance of the centred values,
// rstd = 1 / sqrt(var + eps)); the reference spends about a dozen elementwise
// and reduction launches on it, this file two reads of x from HBM forward (the
// statistics pass centres on block means while a block's rows are still cached
// and merges the blocks exactly) and two passes backward.  HBM-bound: bytes are
// what counts, the arithmetic is fp32.
//
// Backward, with g' = g masked by the ReLU, gh = g' * weight, xh = (x - mean) * rstd,
// n = rows_s * C:
//   dx = rstd * (gh - sum_s(gh) / n - xh * sum_s(gh * xh) / n)
//   dweight[c] = sum over rows of g' * xh,  dbias[c] = sum over rows of g',
//   dresidual = g'.
#include <cooperative_groups.h>
#include <cub/cub.cuh>

#include "rowwise.cuh"
#include "sparse_kernels.cuh"

namespace pcx {
namespace {

constexpr int LN_ROWS = 512;      // rows per block
constexpr int LN_THREADS = 256;

__device__ __forceinline__ float block_sum(float v, float *scratch) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __syncthreads();
    if (lane == 0) scratch[warp] = v;
    __syncthreads();
    float t = 0.f;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += scratch[w];
    return t;
}

__global__ void ln_tail_kernel(int64_t *offsets, int64_t S, int64_t total) {
    if (threadIdx.x == 0 && blockIdx.x == 0) offsets[S] = total;
}

// Row offsets of a batch of a few samples, and zeros for what the backward pass accumulates into (up to three
// arrays), in one small launch.
__global__ void ln_small_offsets_kernel(const int64_t *__restrict__ lengths, int64_t *offsets, int64_t S, int64_t total, float *z0,
                                        int64_t n0, float *z1, float *z2, int64_t n12) {
    start_after_previous();
    for (int64_t t = threadIdx.x; t < n0; t += blockDim.x) z0[t] = 0.f;
    for (int64_t t = threadIdx.x; t < n12; t += blockDim.x) z1[t] = 0.f, z2[t] = 0.f;
    if (threadIdx.x >= 32) return;
    const int lane = threadIdx.x;
    int64_t carry = 0;
    for (int64_t base = 0; base < S; base += 32) {
        const int64_t v = base + lane < S ? lengths[base + lane] : 0;
        int64_t incl = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int64_t up = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += up;
        }
        if (base + lane < S) offsets[base + lane] = carry + incl - v;
        carry += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) offsets[S] = total;
}

// The kernels below share one shape: a block owns `rows` consecutive rows, a thread
// keeps one vector column (VN channels, one 16-byte access when VN > 1) and walks the
// rows of its row lane.  `uniform` blocks lie inside one sample.  The layer norm's kernels work
// a block off in pieces that lie inside one sample each, unless it holds more than MAX_PIECES
// samples (then every row looks its sample up); their blocks are sized for one wave of what is
// resident (layer_rows): with blocks of 512 rows the sums pass spent a quarter of its time folding
// blocks, and clouds of some thousand points kept a fraction of the chip busy.
constexpr int MAX_PIECES = 8;
struct BlockRows {
    int64_t row0, row1, s_first, s_last;
    bool uniform;
    __device__ __forceinline__ BlockRows(const int64_t *__restrict__ offsets, int64_t N, int64_t S, int rows = LN_ROWS) {
        row0 = (int64_t)blockIdx.x * rows;
        row1 = min(N, row0 + rows);
        s_first = segment_of_row(offsets, S, row0);
        s_last = segment_of_row(offsets, S, row1 - 1);
        uniform = s_first == s_last;
    }
    __device__ __forceinline__ bool in_pieces() const { return s_last - s_first < MAX_PIECES; }
};

// Statistics of the layer norm with ONE read of x from HBM.  A thread folds four rows of its column at a time:
// their mean, their squares centred on it, and the exact merge of (count, mean, M2) into what it has; the
// threads of a block merge the same way, and leave one record per (block, sample) piece, which
// ln_combine_kernel merges again (M2 = sum M2_p + n_p (mean_p - mean)^2): the accuracy of the two-pass
// formula, with no barrier while rows are read (sums and squares of a block in turn, each with a block-wide
// reduction, read 1.1 M x 64 bf16 in 52 us).  The piece of sample s in block b is record b + s (pieces are
// ordered, and going to the next piece advances b or s by one), so a sample's pieces are consecutive records.
struct Moments { float n, mean, m2, pad; };

__device__ __forceinline__ void merge(Moments &a, float n, float mean, float m2) {
    if (n == 0.f) return;
    const float total = a.n + n, d = mean - a.mean, share = n / total;
    a.mean += d * share;
    a.m2 += m2 + d * d * a.n * share;
    a.n = total;
}

constexpr int MOM_R = 4;

// Moments of rows [lo, hi) of a block; valid in thread 0.
template <typename T, int VN>
__device__ __forceinline__ Moments moments_of(const T *__restrict__ x, const RowLayout &L, int64_t lo, int64_t hi, int C, Moments *scratch) {
    Moments m{0.f, 0.f, 0.f, 0.f};
    for (int cp = 0; cp * L.vcb < L.vc_total; ++cp) {
        const int vcol = cp * L.vcb + L.vc;
        if (vcol >= L.vc_total || L.lane >= L.lanes) continue;
        const T *col = x + (int64_t)vcol * VN;
        int64_t r = lo + L.lane;
        for (; r + (MOM_R - 1) * L.lanes < hi; r += (int64_t)MOM_R * L.lanes) {
            float v[MOM_R][VN], sum = 0.f, sq = 0.f;
#pragma unroll
            for (int k = 0; k < MOM_R; ++k) load_vec<T, VN>(col + (r + (int64_t)k * L.lanes) * C, v[k]);
#pragma unroll
            for (int k = 0; k < MOM_R; ++k)
#pragma unroll
                for (int i = 0; i < VN; ++i) sum += v[k][i];
            const float mu = sum * (1.f / (MOM_R * VN));
#pragma unroll
            for (int k = 0; k < MOM_R; ++k)
#pragma unroll
                for (int i = 0; i < VN; ++i) sq += (v[k][i] - mu) * (v[k][i] - mu);
            merge(m, (float)(MOM_R * VN), mu, sq);
        }
        for (; r < hi; r += L.lanes) {
            float v[VN], sum = 0.f, sq = 0.f;
            load_vec<T, VN>(col + r * C, v);
#pragma unroll
            for (int i = 0; i < VN; ++i) sum += v[i];
            const float mu = sum * (1.f / VN);
#pragma unroll
            for (int i = 0; i < VN; ++i) sq += (v[i] - mu) * (v[i] - mu);
            merge(m, (float)VN, mu, sq);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float n = __shfl_xor_sync(0xffffffffu, m.n, o), mean = __shfl_xor_sync(0xffffffffu, m.mean, o),
                    m2 = __shfl_xor_sync(0xffffffffu, m.m2, o);
        merge(m, n, mean, m2);
    }
    __syncthreads();
    if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0)
        for (int w = 1; w < LN_THREADS / 32; ++w) merge(m, scratch[w].n, scratch[w].mean, scratch[w].m2);
    return m;
}

template <typename T, int VN>
__global__ void __launch_bounds__(LN_THREADS, 4) ln_moments_kernel(const T *__restrict__ x, const int64_t *__restrict__ offsets, Moments *rec,
                                                                   int64_t N, int64_t S, int C, int rows) {
    start_after_previous();
    __shared__ Moments scratch[LN_THREADS / 32];
    const BlockRows B(offsets, N, S, rows);
    const RowLayout L(C, VN);
    for (int64_t s = B.s_first; s <= B.s_last; ++s) {
        const int64_t lo = max(B.row0, offsets[s]), hi = min(B.row1, offsets[s + 1]);
        if (hi <= lo) continue;   // an empty sample inside the block (same decision in every thread)
        const Moments m = moments_of<T, VN>(x, L, lo, hi, C, scratch);
        if (threadIdx.x == 0) rec[blockIdx.x + s] = m;
    }
}

constexpr int COMBINE_THREADS = 256;

__device__ __forceinline__ double block_sum_f64(double v, double *scratch) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = v;
    __syncthreads();
    double t = 0.0;
    for (int w = 0; w < COMBINE_THREADS / 32; ++w) t += scratch[w];
    return t;
}

// one block per sample: the sample's pieces are spread over the threads, the sums are folded in fp64
__global__ void __launch_bounds__(COMBINE_THREADS) ln_combine_kernel(const Moments *__restrict__ rec,
                                                                     const int64_t *__restrict__ offsets, float *mean,
                                                                     float *rstd, int64_t S, float eps, int mom_rows) {
    start_after_previous();
    __shared__ double scratch[COMBINE_THREADS / 32];
    const int64_t s = blockIdx.x;
    const int64_t lo = offsets[s], hi = offsets[s + 1];
    if (hi <= lo) {   // the same decision in every thread
        if (threadIdx.x == 0) mean[s] = 0.f, rstd[s] = 1.f / sqrtf(eps);
        return;
    }
    const int64_t b0 = lo / mom_rows, b1 = (hi - 1) / mom_rows;
    double n = 0.0, sum = 0.0;
    for (int64_t b = b0 + threadIdx.x; b <= b1; b += COMBINE_THREADS) {
        const Moments m = rec[b + s];
        n += m.n, sum += (double)m.n * m.mean;
    }
    n = block_sum_f64(n, scratch);
    sum = block_sum_f64(sum, scratch);
    const double mu = sum / n;
    double m2 = 0.0;
    for (int64_t b = b0 + threadIdx.x; b <= b1; b += COMBINE_THREADS) {
        const Moments m = rec[b + s];
        const double d = (double)m.mean - mu;
        m2 += (double)m.m2 + (double)m.n * d * d;
    }
    m2 = block_sum_f64(m2, scratch);
    if (threadIdx.x == 0) mean[s] = (float)mu, rstd[s] = 1.f / sqrtf((float)(m2 / n) + eps);
}

template <typename T, int VN>
__global__ void __launch_bounds__(LN_THREADS, 5) ln_apply_kernel(const T *__restrict__ x, const int64_t *__restrict__ offsets,
                                const float *__restrict__ mean, const float *__restrict__ rstd,
                                const float *__restrict__ weight, const float *__restrict__ bias,
                                const T *__restrict__ residual, T *y, int64_t N, int64_t S, int C, int relu, int rows) {
    start_after_previous();
    const BlockRows B(offsets, N, S, rows);
    const RowLayout L(C, VN);
    for (int cp = 0; cp * L.vcb < L.vc_total; ++cp) {
        const int vcol = cp * L.vcb + L.vc;
        if (vcol >= L.vc_total || L.lane >= L.lanes) continue;
        float w[VN], b[VN];
#pragma unroll
        for (int i = 0; i < VN; ++i) {
            w[i] = weight ? weight[vcol * VN + i] : 1.f;
            b[i] = weight ? bias[vcol * VN + i] : 0.f;
        }
        auto row = [&](int64_t r, float mu, float rs) {
            const int64_t at = r * C + (int64_t)vcol * VN;
            float v[VN], res[VN];
            load_vec<T, VN>(x + at, v);
            if (residual) load_vec<T, VN>(residual + at, res);
#pragma unroll
            for (int i = 0; i < VN; ++i) {
                float o = (v[i] - mu) * rs * w[i] + b[i];
                if (residual) o += res[i];
                v[i] = relu ? fmaxf(o, 0.f) : o;
            }
            store_vec<T, VN>(y + at, v);
        };
        if (B.in_pieces()) {
            for (int64_t s = B.s_first; s <= B.s_last; ++s) {
                const int64_t hi = min(B.row1, offsets[s + 1]);
                const float mu = mean[s], rs = rstd[s];
#pragma unroll 4
                for (int64_t r = max(B.row0, offsets[s]) + L.lane; r < hi; r += L.lanes) row(r, mu, rs);
            }
        } else {
            for (int64_t r = B.row0 + L.lane; r < B.row1; r += L.lanes) {
                const int64_t s = segment_of_row(offsets, S, r);
                row(r, mean[s], rstd[s]);
            }
        }
    }
}

// Per-sample sums of gh and gh * xh, per-channel sums of g' * xh and g', and
// (optionally) the masked gradient for the residual branch.  Per-sample partial sums
// stay in registers while a thread's rows belong to one sample; the per-channel sums of
// the row lanes are folded in shared memory, one atomic per channel and block.
template <typename T, int VN>
__global__ void __launch_bounds__(LN_THREADS, 4) ln_bwd_sums_kernel(const T *__restrict__ g, const T *__restrict__ x, const T *__restrict__ y,
                                   const int64_t *__restrict__ offsets, const float *__restrict__ mean,
                                   const float *__restrict__ rstd, const float *__restrict__ weight, float *s1,
                                   float *s2, float *dweight, float *dbias, T *dresidual, int64_t N, int64_t S,
                                   int C, int relu, int rows) {
    start_after_previous();
    __shared__ float scratch[LN_THREADS / 32];
    __shared__ float col_w[LN_THREADS * VN], col_b[LN_THREADS * VN];
    const BlockRows B(offsets, N, S, rows);
    const RowLayout L(C, VN);
    float a = 0.f, b = 0.f;     // running sums of gh and gh * xh for sample `cur`
    int64_t cur = B.s_first;
    for (int cp = 0; cp * L.vcb < L.vc_total; ++cp) {
        const int vcol = cp * L.vcb + L.vc;
        const bool active = vcol < L.vc_total && L.lane < L.lanes;
        float w[VN], dw[VN], db[VN];
#pragma unroll
        for (int i = 0; i < VN; ++i) {
            w[i] = (weight && active) ? weight[vcol * VN + i] : 1.f;
            dw[i] = db[i] = 0.f;
        }
        auto row = [&](int64_t r, float mu, float rs) {
            const int64_t at = r * C + (int64_t)vcol * VN;
            float gv[VN], xv[VN], yv[VN];
            load_vec<T, VN>(g + at, gv);
            load_vec<T, VN>(x + at, xv);
            if (relu) load_vec<T, VN>(y + at, yv);
#pragma unroll
            for (int i = 0; i < VN; ++i) {
                if (relu && !(yv[i] > 0.f)) gv[i] = 0.f;
                const float xh = (xv[i] - mu) * rs;
                a += gv[i] * w[i];
                b += gv[i] * w[i] * xh;
                dw[i] += gv[i] * xh;
                db[i] += gv[i];
            }
            if (dresidual) store_vec<T, VN>(dresidual + at, gv);
        };
        if (B.in_pieces()) {
            for (int64_t s = B.s_first; s <= B.s_last; ++s) {
                const int64_t hi = active ? min(B.row1, offsets[s + 1]) : 0;
                const float mu = mean[s], rs = rstd[s];
#pragma unroll 2
                for (int64_t r = max(B.row0, offsets[s]) + L.lane; r < hi; r += L.lanes) row(r, mu, rs);
                a = block_sum(a, scratch);
                b = block_sum(b, scratch);
                if (threadIdx.x == 0) {
                    atomicAdd(s1 + s, a);
                    atomicAdd(s2 + s, b);
                }
                a = b = 0.f;
            }
        } else if (active) {
            for (int64_t r = B.row0 + L.lane; r < B.row1; r += L.lanes) {
                const int64_t s = segment_of_row(offsets, S, r);
                if (s != cur) {
                    atomicAdd(s1 + cur, a);
                    atomicAdd(s2 + cur, b);
                    a = b = 0.f;
                    cur = s;
                }
                row(r, mean[s], rstd[s]);
            }
        }
        if (dweight) {
            // col_*[lane][column of the pass]: fold the row lanes, then one atomic per channel
#pragma unroll
            for (int i = 0; i < VN; ++i) {
                col_w[(L.lane * L.vcb + L.vc) * VN + i] = dw[i];
                col_b[(L.lane * L.vcb + L.vc) * VN + i] = db[i];
            }
            __syncthreads();
            const int cols = L.vcb * VN;
            for (int t = threadIdx.x; t < cols; t += LN_THREADS) {
                const int c = cp * cols + t;
                if (c < C) {
                    float tw = 0.f, tb = 0.f;
                    for (int q = 0; q < L.lanes; ++q) tw += col_w[q * cols + t], tb += col_b[q * cols + t];
                    atomicAdd(dweight + c, tw);
                    atomicAdd(dbias + c, tb);
                }
            }
            __syncthreads();
        }
    }
    if (!B.in_pieces()) {
        atomicAdd(s1 + cur, a);
        atomicAdd(s2 + cur, b);
    }
}

template <typename T, int VN>
__global__ void __launch_bounds__(LN_THREADS, 4) ln_bwd_apply_kernel(const T *__restrict__ g, const T *__restrict__ x, const T *__restrict__ y,
                                    const int64_t *__restrict__ offsets, const float *__restrict__ mean,
                                    const float *__restrict__ rstd, const float *__restrict__ weight,
                                    const float *__restrict__ s1, const float *__restrict__ s2, T *dx, int64_t N,
                                    int64_t S, int C, int relu, int rows) {
    start_after_previous();
    const BlockRows B(offsets, N, S, rows);
    const RowLayout L(C, VN);
    for (int cp = 0; cp * L.vcb < L.vc_total; ++cp) {
        const int vcol = cp * L.vcb + L.vc;
        if (vcol >= L.vc_total || L.lane >= L.lanes) continue;
        float w[VN];
#pragma unroll
        for (int i = 0; i < VN; ++i) w[i] = weight ? weight[vcol * VN + i] : 1.f;
        auto row = [&](int64_t r, float mu, float rs, float m1, float m2) {
            const int64_t at = r * C + (int64_t)vcol * VN;
            float gv[VN], xv[VN], yv[VN];
            load_vec<T, VN>(g + at, gv);   // with relu == 0 this may be the gradient the sums pass already masked
            load_vec<T, VN>(x + at, xv);
            if (relu) load_vec<T, VN>(y + at, yv);
#pragma unroll
            for (int i = 0; i < VN; ++i) {
                if (relu && !(yv[i] > 0.f)) gv[i] = 0.f;
                const float xh = (xv[i] - mu) * rs;
                gv[i] = rs * (gv[i] * w[i] - m1 - xh * m2);
            }
            store_vec<T, VN>(dx + at, gv);
        };
        if (B.in_pieces()) {
            for (int64_t s = B.s_first; s <= B.s_last; ++s) {
                const int64_t hi = min(B.row1, offsets[s + 1]);
                const float mu = mean[s], rs = rstd[s], inv_n = 1.f / ((float)(offsets[s + 1] - offsets[s]) * (float)C);
                const float m1 = s1[s] * inv_n, m2 = s2[s] * inv_n;
#pragma unroll 2
                for (int64_t r = max(B.row0, offsets[s]) + L.lane; r < hi; r += L.lanes) row(r, mu, rs, m1, m2);
            }
        } else {
            for (int64_t r = B.row0 + L.lane; r < B.row1; r += L.lanes) {
                const int64_t s = segment_of_row(offsets, S, r);
                const float inv_n = 1.f / ((float)(offsets[s + 1] - offsets[s]) * (float)C);
                row(r, mean[s], rstd[s], s1[s] * inv_n, s2[s] * inv_n);
            }
        }
    }
}

// ---------------------------------------------------------------- small batches ----
// Rows of up to 8 MB in up to 32 samples go through one kernel forward and one backward whose blocks are all resident (a
// cooperative launch): sums of a block's rows, a barrier of the grid, the same rows again.  Such norms are bound by launches, of
// which the kernels above take four and three: 2000 rows of 64 channels forward 25 -> 13 us, 5000 of 256 24 -> 13, 40 000 of 96
// 23 -> 15; the 40 norms of a network on 40 000 points 0.34 ms less.  Beyond that the blocks of one launch see too few rows
// in flight (300 000 x 64 29 and 44); larger batches sample by sample, so that the second look at a row is out of the L2,
// lost as well (1.1 M x 64 in eight samples 84 and 120 forward, 130 and 184 backward): a sample a barrier is too little work for
// the latency of its loads and folds.
namespace cg = cooperative_groups;
constexpr int FEW = 32, FEW_CTAS = 4;   // samples; blocks of an SM
constexpr int FEW_BLOCKS = 1024;        // of a launch, at most (what the records have room for)
constexpr int64_t FEW_BYTES = 8 << 20;  // of a tensor

struct FewSamples {
    int64_t offset[FEW + 1];
    // every thread of the block calls
    __device__ __forceinline__ void load(const int64_t *__restrict__ lengths, int S, int64_t N) {
        if (threadIdx.x < 32) {
            const int lane = threadIdx.x;
            int64_t v = lane < S ? lengths[lane] : 0, upto = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int64_t up = __shfl_up_sync(0xffffffffu, upto, o);
                if (lane >= o) upto += up;
            }
            if (lane < S) offset[lane] = upto - v;
            __syncwarp();
            if (lane == 0) offset[S] = N;
        }
        __syncthreads();
    }
};

template <typename T, int VN>
__global__ void __launch_bounds__(LN_THREADS, FEW_CTAS) ln_few_kernel(const T *__restrict__ x, const int64_t *__restrict__ lengths, const float *__restrict__ weight,
                                                                      const float *__restrict__ bias, const T *__restrict__ residual, T *y, float *mean,
                                                                      float *rstd, Moments *rec, int64_t N, int S, int C, float eps, int relu) {
    __shared__ FewSamples samples;
    __shared__ Moments scratch[LN_THREADS / 32];
    __shared__ double scratch64[LN_THREADS / 32];
    const cg::grid_group grid = cg::this_grid();
    samples.load(lengths, S, N);
    const RowLayout L(C, VN);
    const int blocks = (int)gridDim.x;
    const int64_t lo = N * blockIdx.x / blocks, hi = N * (blockIdx.x + 1) / blocks;   // this block's rows
    for (int s = 0; s < S; ++s) {   // rec[sample][block]
        const int64_t a = max(lo, samples.offset[s]), b = min(hi, samples.offset[s + 1]);
        Moments m{0.f, 0.f, 0.f, 0.f};
        if (a < b) m = moments_of<T, VN>(x, L, a, b, C, scratch);
        if (threadIdx.x == 0) rec[(int64_t)s * blocks + blockIdx.x] = m;
    }
    grid.sync();
    for (int s = 0; s < S; ++s) {
        const int64_t a = max(lo, samples.offset[s]), b = min(hi, samples.offset[s + 1]);
        if (samples.offset[s] == samples.offset[s + 1] && blockIdx.x == 0 && threadIdx.x == 0) mean[s] = 0.f, rstd[s] = 1.f / sqrtf(eps);
        if (a >= b) continue;
        // every block folds the records of the samples it has rows of, in fp64 and in the same order
        double n = 0.0, sum = 0.0, m2 = 0.0;
        for (int q = threadIdx.x; q < blocks; q += LN_THREADS) {
            const float4 m = __ldcg(reinterpret_cast<const float4 *>(rec + (int64_t)s * blocks + q));
            n += m.x, sum += (double)m.x * m.y;
        }
        n = block_sum_f64(n, scratch64);
        sum = block_sum_f64(sum, scratch64);
        const double mu64 = sum / n;
        for (int q = threadIdx.x; q < blocks; q += LN_THREADS) {
            const float4 m = __ldcg(reinterpret_cast<const float4 *>(rec + (int64_t)s * blocks + q));
            const double d = (double)m.y - mu64;
            m2 += (double)m.z + (double)m.x * d * d;
        }
        m2 = block_sum_f64(m2, scratch64);
        const float mu = (float)mu64, rs = 1.f / sqrtf((float)(m2 / n) + eps);
        if (a == samples.offset[s] && threadIdx.x == 0) mean[s] = mu, rstd[s] = rs;
        for (int cp = 0; cp * L.vcb < L.vc_total; ++cp) {
            const int vcol = cp * L.vcb + L.vc;
            if (vcol >= L.vc_total || L.lane >= L.lanes) continue;
            float w[VN], c[VN];
#pragma unroll
            for (int i = 0; i < VN; ++i) {
                w[i] = weight ? weight[vcol * VN + i] : 1.f;
                c[i] = weight ? bias[vcol * VN + i] : 0.f;
            }
#pragma unroll 4
            for (int64_t r = a + L.lane; r < b; r += L.lanes) {
                const int64_t at = r * C + (int64_t)vcol * VN;
                float v[VN], res[VN];
                load_vec<T, VN>(x + at, v);
                if (residual) load_vec<T, VN>(residual + at, res);
#pragma unroll
                for (int i = 0; i < VN; ++i) {
                    float o = (v[i] - mu) * rs * w[i] + c[i];
                    if (residual) o += res[i];
                    v[i] = relu ? fmaxf(o, 0.f) : o;
                }
                store_vec<T, VN>(y + at, v);
            }
        }
    }
}

// One pass of vector columns (C / VN <= LN_THREADS): the sums per channel stay in registers over all samples.
template <typename T, int VN>
__global__ void __launch_bounds__(LN_THREADS, FEW_CTAS - 1) ln_few_bwd_kernel(const T *__restrict__ g, const T *__restrict__ x, const T *__restrict__ y,
                                                                          const int64_t *__restrict__ lengths, const float *__restrict__ mean,
                                                                          const float *__restrict__ rstd, const float *__restrict__ weight, float2 *rec,
                                                                          float *dweight, float *dbias, T *dresidual, T *dx, int64_t N, int S, int C,
                                                                          int relu) {
    __shared__ FewSamples samples;
    __shared__ float scratch[LN_THREADS / 32];
    __shared__ double scratch64[LN_THREADS / 32];
    __shared__ float col_w[LN_THREADS * VN], col_b[LN_THREADS * VN];
    const cg::grid_group grid = cg::this_grid();
    samples.load(lengths, S, N);
    const RowLayout L(C, VN);
    const int blocks = (int)gridDim.x;
    const int64_t lo = N * blockIdx.x / blocks, hi = N * (blockIdx.x + 1) / blocks;   // this block's rows
    const bool active = L.lane < L.lanes;
    const bool masked = relu && dresidual;   // the sums wrote the masked gradient: it is read instead of masking again
    float w[VN], dw[VN], db[VN];
#pragma unroll
    for (int i = 0; i < VN; ++i) {
        w[i] = weight && active ? weight[L.vc * VN + i] : 1.f;
        dw[i] = db[i] = 0.f;
    }
    if (dweight && blockIdx.x == 0)   // (the other blocks add to them behind the barrier)
        for (int c = threadIdx.x; c < C; c += LN_THREADS) dweight[c] = 0.f, dbias[c] = 0.f;
    for (int s = 0; s < S; ++s) {
        const int64_t a = max(lo, samples.offset[s]), b = min(hi, samples.offset[s + 1]);
        float sa = 0.f, sb = 0.f;
        if (a < b) {
            const float mu = mean[s], rs = rstd[s];
#pragma unroll 2
            for (int64_t r = active ? a + L.lane : b; r < b; r += L.lanes) {
                const int64_t at = r * C + (int64_t)L.vc * VN;
                float gv[VN], xv[VN], yv[VN];
                load_vec<T, VN>(g + at, gv);
                load_vec<T, VN>(x + at, xv);
                if (relu) load_vec<T, VN>(y + at, yv);
#pragma unroll
                for (int i = 0; i < VN; ++i) {
                    if (relu && !(yv[i] > 0.f)) gv[i] = 0.f;
                    const float xh = (xv[i] - mu) * rs;
                    sa += gv[i] * w[i];
                    sb += gv[i] * w[i] * xh;
                    dw[i] += gv[i] * xh;
                    db[i] += gv[i];
                }
                if (dresidual) store_vec<T, VN>(dresidual + at, gv);
            }
            sa = block_sum(sa, scratch);
            sb = block_sum(sb, scratch);
        }
        if (threadIdx.x == 0) rec[(int64_t)s * blocks + blockIdx.x] = make_float2(sa, sb);
    }
    grid.sync();
    const T *from = masked ? dresidual : g;
    for (int s = 0; s < S; ++s) {
        const int64_t a = max(lo, samples.offset[s]), b = min(hi, samples.offset[s + 1]);
        if (a >= b) continue;
        double s1 = 0.0, s2 = 0.0;
        for (int q = threadIdx.x; q < blocks; q += LN_THREADS) {
            const float2 v = __ldcg(rec + (int64_t)s * blocks + q);
            s1 += v.x, s2 += v.y;
        }
        s1 = block_sum_f64(s1, scratch64);
        s2 = block_sum_f64(s2, scratch64);
        const float mu = mean[s], rs = rstd[s], inv_n = 1.f / ((float)(samples.offset[s + 1] - samples.offset[s]) * (float)C);
        const float m1 = (float)s1 * inv_n, m2 = (float)s2 * inv_n;
#pragma unroll 2
        for (int64_t r = active ? a + L.lane : b; r < b; r += L.lanes) {
            const int64_t at = r * C + (int64_t)L.vc * VN;
            float gv[VN], xv[VN], yv[VN];
            load_vec<T, VN>(from + at, gv);
            load_vec<T, VN>(x + at, xv);
            if (relu && !masked) load_vec<T, VN>(y + at, yv);
#pragma unroll
            for (int i = 0; i < VN; ++i) {
                if (relu && !masked && !(yv[i] > 0.f)) gv[i] = 0.f;
                const float xh = (xv[i] - mu) * rs;
                gv[i] = rs * (gv[i] * w[i] - m1 - xh * m2);
            }
            store_vec<T, VN>(dx + at, gv);
        }
    }
    if (dweight) {
#pragma unroll
        for (int i = 0; i < VN; ++i)
            if (active) col_w[(L.lane * L.vcb + L.vc) * VN + i] = dw[i], col_b[(L.lane * L.vcb + L.vc) * VN + i] = db[i];
        __syncthreads();
        const int cols = L.vcb * VN;
        for (int c = threadIdx.x; c < cols && c < C; c += LN_THREADS) {
            float tw = 0.f, tb = 0.f;
            for (int q = 0; q < L.lanes; ++q) tw += col_w[q * cols + c], tb += col_b[q * cols + c];
            atomicAdd(dweight + c, tw);
            atomicAdd(dbias + c, tb);
        }
    }
}

// ---------------------------------------------------------------- grouped statistics ----
// Group and instance normalisation: the statistics of sample s are kept per channel group g
// (G groups of W = C / G consecutive channels; instance norm is W = 1) in arrays indexed
// s * G + g.  Same block shape as above; a thread's VN channels may fall into different groups,
// so every channel keeps its own running sum.  Blocks inside one sample fold their sums per
// group in shared memory (G floats) and issue one atomic per group; blocks that straddle a
// sample boundary use per-thread atomics.
struct GroupStats {
    float mu[8], rs[8];
    int64_t at = -1;
    template <int VN>
    __device__ __forceinline__ void load(const float *__restrict__ mean, const float *__restrict__ rstd, int64_t s,
                                         int G, const int *g) {
        if (s == at) return;
        at = s;
#pragma unroll
        for (int i = 0; i < VN; ++i) {
            mu[i] = mean ? mean[s * G + g[i]] : 0.f;
            rs[i] = rstd ? rstd[s * G + g[i]] : 1.f;
        }
    }
};

template <int VN>
__device__ __forceinline__ void flush_groups(float *dst, const int *g, float *v) {
#pragma unroll
    for (int i = 0; i < VN; ++i) {
        if (v[i] != 0.f) atomicAdd(dst + g[i], v[i]);
        v[i] = 0.f;
    }
}

// sums[s * G + g] += sum of x (mean == null) or of (x - mean)^2
template <typename T, int VN>
__global__ void gn_sum_kernel(const T *__restrict__ x, const int64_t *__restrict__ offsets,
                              const float *__restrict__ mean, float *sums, int64_t N, int64_t S, int C, int G) {
    extern __shared__ float s_grp[];
    const BlockRows B(offsets, N, S);
    const RowLayout L(C, VN);
    const int W = C / G;
    if (B.uniform) {
        for (int t = threadIdx.x; t < G; t += blockDim.x) s_grp[t] = 0.f;
        __syncthreads();
    }
    for (int cp = 0; cp * L.vcb < L.vc_total; ++cp) {
        const int vcol = cp * L.vcb + L.vc;
        if (vcol >= L.vc_total || L.lane >= L.lanes) continue;
        int g[VN];
        float acc[VN];
#pragma unroll
        for (int i = 0; i < VN; ++i) g[i] = (vcol * VN + i) / W, acc[i] = 0.f;
        GroupStats st;
        int64_t cur = B.s_first;
#pragma unroll 2
        for (int64_t r = B.row0 + L.lane; r < B.row1; r += L.lanes) {
            const int64_t s = B.uniform ? B.s_first : segment_of_row(offsets, S, r);
            if (s != cur) {
                flush_groups<VN>(sums + cur * G, g, acc);
                cur = s;
            }
            st.load<VN>(mean, nullptr, s, G, g);
            float v[VN];
            load_vec<T, VN>(x + r * C + (int64_t)vcol * VN, v);
#pragma unroll
            for (int i = 0; i < VN; ++i) {
                const float d = v[i] - st.mu[i];
                acc[i] += mean ? d * d : d;
            }
        }
        flush_groups<VN>(B.uniform ? s_grp : sums + cur * G, g, acc);
    }
    if (B.uniform) {
        __syncthreads();
        for (int t = threadIdx.x; t < G; t += blockDim.x)
            if (s_grp[t] != 0.f) atomicAdd(sums + B.s_first * G + t, s_grp[t]);
    }
}

__global__ void gn_stats_kernel(const float *__restrict__ sums, const int64_t *__restrict__ offsets, float *mean,
                                float *rstd, int64_t S, int G, int W, float eps, int second) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= S * G) return;
    const int64_t s = t / G, len = offsets[s + 1] - offsets[s];
    const float n = (float)(len > 0 ? len : 1) * (float)W;
    if (!second) mean[t] = sums[t] / n;
    else rstd[t] = 1.f / sqrtf(sums[t] / n + eps);
}

template <typename T, int VN>
__global__ void gn_apply_kernel(const T *__restrict__ x, const int64_t *__restrict__ offsets,
                                const float *__restrict__ mean, const float *__restrict__ rstd,
                                const float *__restrict__ weight, const float *__restrict__ bias, T *y, int64_t N,
                                int64_t S, int C, int G) {
    const BlockRows B(offsets, N, S);
    const RowLayout L(C, VN);
    const int W = C / G;
    for (int cp = 0; cp * L.vcb < L.vc_total; ++cp) {
        const int vcol = cp * L.vcb + L.vc;
        if (vcol >= L.vc_total || L.lane >= L.lanes) continue;
        int g[VN];
        float w[VN], b[VN];
#pragma unroll
        for (int i = 0; i < VN; ++i) {
            g[i] = (vcol * VN + i) / W;
            w[i] = weight ? weight[vcol * VN + i] : 1.f;
            b[i] = weight ? bias[vcol * VN + i] : 0.f;
        }
        GroupStats st;
#pragma unroll 2
        for (int64_t r = B.row0 + L.lane; r < B.row1; r += L.lanes) {
            const int64_t s = B.uniform ? B.s_first : segment_of_row(offsets, S, r);
            st.load<VN>(mean, rstd, s, G, g);
            const int64_t at = r * C + (int64_t)vcol * VN;
            float v[VN];
            load_vec<T, VN>(x + at, v);
#pragma unroll
            for (int i = 0; i < VN; ++i) v[i] = (v[i] - st.mu[i]) * st.rs[i] * w[i] + b[i];
            store_vec<T, VN>(y + at, v);
        }
    }
}

// Backward of the grouped norms, with gh = g * weight, xh = (x - mean) * rstd, n = rows_s * W:
//   dx = rstd * (gh - sum_{s,g}(gh) / n - xh * sum_{s,g}(gh * xh) / n),
//   dweight[c] = sum over rows of g * xh, dbias[c] = sum over rows of g.
template <typename T, int VN>
__global__ void gn_bwd_sums_kernel(const T *__restrict__ g_out, const T *__restrict__ x,
                                   const int64_t *__restrict__ offsets, const float *__restrict__ mean,
                                   const float *__restrict__ rstd, const float *__restrict__ weight, float *s1,
                                   float *s2, float *dweight, float *dbias, int64_t N, int64_t S, int C, int G) {
    extern __shared__ float s_grp[];   // 2 G: sums of gh, sums of gh * xh
    __shared__ float col_w[LN_THREADS * VN], col_b[LN_THREADS * VN];
    const BlockRows B(offsets, N, S);
    const RowLayout L(C, VN);
    const int W = C / G;
    if (B.uniform) {
        for (int t = threadIdx.x; t < 2 * G; t += blockDim.x) s_grp[t] = 0.f;
        __syncthreads();
    }
    for (int cp = 0; cp * L.vcb < L.vc_total; ++cp) {
        const int vcol = cp * L.vcb + L.vc;
        const bool active = vcol < L.vc_total && L.lane < L.lanes;
        int g[VN];
        float w[VN], a[VN], b[VN], dw[VN], db[VN];
#pragma unroll
        for (int i = 0; i < VN; ++i) {
            g[i] = active ? (vcol * VN + i) / W : 0;
            w[i] = (weight && active) ? weight[vcol * VN + i] : 1.f;
            a[i] = b[i] = dw[i] = db[i] = 0.f;
        }
        GroupStats st;
        int64_t cur = B.s_first;
#pragma unroll 2
        for (int64_t r = B.row0 + L.lane; active && r < B.row1; r += L.lanes) {
            const int64_t s = B.uniform ? B.s_first : segment_of_row(offsets, S, r);
            if (s != cur) {
                flush_groups<VN>(s1 + cur * G, g, a);
                flush_groups<VN>(s2 + cur * G, g, b);
                cur = s;
            }
            st.load<VN>(mean, rstd, s, G, g);
            const int64_t at = r * C + (int64_t)vcol * VN;
            float gv[VN], xv[VN];
            load_vec<T, VN>(g_out + at, gv);
            load_vec<T, VN>(x + at, xv);
#pragma unroll
            for (int i = 0; i < VN; ++i) {
                const float xh = (xv[i] - st.mu[i]) * st.rs[i];
                a[i] += gv[i] * w[i];
                b[i] += gv[i] * w[i] * xh;
                dw[i] += gv[i] * xh;
                db[i] += gv[i];
            }
        }
        flush_groups<VN>(B.uniform ? s_grp : s1 + cur * G, g, a);
        flush_groups<VN>(B.uniform ? s_grp + G : s2 + cur * G, g, b);
        if (dweight) {   // fold the row lanes in shared memory, then one atomic per channel and block
#pragma unroll
            for (int i = 0; i < VN; ++i) {
                col_w[(L.lane * L.vcb + L.vc) * VN + i] = dw[i];
                col_b[(L.lane * L.vcb + L.vc) * VN + i] = db[i];
            }
            __syncthreads();
            const int cols = L.vcb * VN;
            for (int t = threadIdx.x; t < cols; t += LN_THREADS) {
                const int c = cp * cols + t;
                if (c < C) {
                    float tw = 0.f, tb = 0.f;
                    for (int q = 0; q < L.lanes; ++q) tw += col_w[q * cols + t], tb += col_b[q * cols + t];
                    atomicAdd(dweight + c, tw);
                    atomicAdd(dbias + c, tb);
                }
            }
            __syncthreads();
        }
    }
    if (B.uniform) {
        __syncthreads();
        for (int t = threadIdx.x; t < G; t += blockDim.x) {
            if (s_grp[t] != 0.f) atomicAdd(s1 + B.s_first * G + t, s_grp[t]);
            if (s_grp[G + t] != 0.f) atomicAdd(s2 + B.s_first * G + t, s_grp[G + t]);
        }
    }
}

template <typename T, int VN>
__global__ void gn_bwd_apply_kernel(const T *__restrict__ g_out, const T *__restrict__ x,
                                    const int64_t *__restrict__ offsets, const float *__restrict__ mean,
                                    const float *__restrict__ rstd, const float *__restrict__ weight,
                                    const float *__restrict__ s1, const float *__restrict__ s2, T *dx, int64_t N,
                                    int64_t S, int C, int G) {
    const BlockRows B(offsets, N, S);
    const RowLayout L(C, VN);
    const int W = C / G;
    for (int cp = 0; cp * L.vcb < L.vc_total; ++cp) {
        const int vcol = cp * L.vcb + L.vc;
        if (vcol >= L.vc_total || L.lane >= L.lanes) continue;
        int g[VN];
        float w[VN], m1[VN], m2[VN];
#pragma unroll
        for (int i = 0; i < VN; ++i) g[i] = (vcol * VN + i) / W, w[i] = weight ? weight[vcol * VN + i] : 1.f;
        GroupStats st;
        int64_t have = -1;
#pragma unroll 2
        for (int64_t r = B.row0 + L.lane; r < B.row1; r += L.lanes) {
            const int64_t s = B.uniform ? B.s_first : segment_of_row(offsets, S, r);
            st.load<VN>(mean, rstd, s, G, g);
            if (s != have) {
                have = s;
                const float inv_n = 1.f / ((float)(offsets[s + 1] - offsets[s]) * (float)W);
#pragma unroll
                for (int i = 0; i < VN; ++i) m1[i] = s1[s * G + g[i]] * inv_n, m2[i] = s2[s * G + g[i]] * inv_n;
            }
            const int64_t at = r * C + (int64_t)vcol * VN;
            float gv[VN], xv[VN];
            load_vec<T, VN>(g_out + at, gv);
            load_vec<T, VN>(x + at, xv);
#pragma unroll
            for (int i = 0; i < VN; ++i) {
                const float xh = (xv[i] - st.mu[i]) * st.rs[i];
                gv[i] = st.rs[i] * (gv[i] * w[i] - m1[i] - xh * m2[i]);
            }
            store_vec<T, VN>(dx + at, gv);
        }
    }
}

struct LnWs {
    int64_t *offsets;
    Moments *rec;  // per (block, sample) piece of the forward statistics (layer norm only)
    float *sums;   // 2 * S
    void *cub_tmp;
    size_t cub_bytes;
};

size_t carve_ln(void *ws, int64_t S, LnWs *out, int64_t pieces = 0) {
    Carver c(ws);
    LnWs w;
    w.offsets = c.take<int64_t>((size_t)S + 1);
    w.rec = c.take<Moments>((size_t)pieces);
    w.sums = c.take<float>((size_t)2 * S + 1);
    size_t bytes = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, bytes, (const int64_t *)nullptr, (int64_t *)nullptr, (int)std::max<int64_t>(S, 1));
    w.cub_bytes = bytes;
    w.cub_tmp = c.take<char>(bytes);
    if (out) *out = w;
    return c.off;
}

// Rows per block: one wave of `ctas` blocks per SM, whole row lanes, at least two rows per thread.
int layer_rows(int64_t N, int C, int dtype, bool vec, int ctas) {
    const int cols = C / (vec ? 16 / (int)elem_size(dtype) : 1), lanes = LN_THREADS / std::min(cols, LN_THREADS);
    const int64_t wave = (int64_t)ctas * num_sms(), rows = (N + wave - 1) / wave;
    return (int)std::min<int64_t>(((std::max<int64_t>(rows, 2 * lanes) + lanes - 1) / lanes) * lanes, (int64_t)1 << 30);
}

// `z1`, `z2` (n12 floats each, or null) and, with `zero_sums`, the workspace's sums are cleared on the way.
int ln_offsets(const int64_t *d_lengths, int64_t S, int64_t N, const LnWs &w, cudaStream_t stream, bool zero_sums = false, float *z1 = nullptr,
               float *z2 = nullptr, int64_t n12 = 0) {
    if (S <= 4096) {
        launch_after(ln_small_offsets_kernel, 1, 256, 0, stream, d_lengths, w.offsets, S, N, w.sums, zero_sums ? 2 * S : 0, z1, z2, z1 ? n12 : 0);
        PCX_LAUNCH_CHECK();
        return PCX_OK;
    }
    if (zero_sums) PCX_CUDA(cudaMemsetAsync(w.sums, 0, (size_t)2 * S * sizeof(float), stream));
    if (z1) {
        PCX_CUDA(cudaMemsetAsync(z1, 0, (size_t)n12 * sizeof(float), stream));
        PCX_CUDA(cudaMemsetAsync(z2, 0, (size_t)n12 * sizeof(float), stream));
    }
    size_t bytes = w.cub_bytes;
    PCX_CUDA(cub::DeviceScan::ExclusiveSum(w.cub_tmp, bytes, d_lengths, w.offsets, (int)S, stream));
    ln_tail_kernel<<<1, 32, 0, stream>>>(w.offsets, S, N);
    PCX_LAUNCH_CHECK();
    return PCX_OK;
}

// (block, sample) pieces of N rows in S samples: record b + s, b < blocks, s < S
// an upper bound for every block height the statistics pass may choose (at least two rows per block)
int64_t ln_pieces(int64_t N, int64_t S) { return std::max<int64_t>((N + 1) / 2 + S, S <= FEW ? S * FEW_BLOCKS : 0); }

bool ln_sizes_ok(int64_t N, int64_t S, int C, int dtype) {
    return N >= 0 && S > 0 && S <= INT32_MAX && C > 0 && (dtype == PCX_F32 || dtype == PCX_F16 || dtype == PCX_BF16);
}

// Blocks of a cooperative launch over N rows: at most what is resident at once, at least two rows a lane.
template <typename Kernel>
int few_blocks(Kernel kernel, int64_t N, int C, int dtype, bool vec, int *cached) {
    if (*cached == 0) {
        int n = 0;
        *cached = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, LN_THREADS, 0) == cudaSuccess && n > 0 ? n : -1;
        (void)cudaGetLastError();
    }
    if (*cached < 0) return 0;
    const int cols = C / (vec ? 16 / (int)elem_size(dtype) : 1), lanes = LN_THREADS / std::min(cols, LN_THREADS);
    return (int)std::max<int64_t>(1, std::min<int64_t>((int64_t)std::min(*cached, FEW_CTAS) * num_sms(), N / (2 * lanes)));
}

constexpr int NOT_TOGETHER = 1;   // the stream has a part of the chip (a green context): its blocks are not resident at once

template <typename... Params, typename... Args>
int launch_together(void (*kernel)(Params...), int blocks, cudaStream_t stream, Args &&...args) {
    cudaLaunchAttribute together = {};
    together.id = cudaLaunchAttributeCooperative;
    together.val.cooperative = 1;
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3((unsigned)blocks), config.blockDim = dim3(LN_THREADS), config.stream = stream;
    config.attrs = &together, config.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&config, kernel, std::forward<Args>(args)...);
    if (e == cudaErrorCooperativeLaunchTooLarge) {
        (void)cudaGetLastError();
        return NOT_TOGETHER;
    }
    PCX_CUDA(e);
    PCX_LAUNCH_CHECK();
    return PCX_OK;
}

// CALL sees T (element type) and VN (channels per access: 16 bytes' worth when `vec`, else 1)
#define PCX_LN_DISPATCH(dtype, vec, CALL)                                                        \
    do {                                                                                         \
        if ((dtype) == PCX_F32) { using T = float; if (vec) { constexpr int VN = 4; CALL; } else { constexpr int VN = 1; CALL; } }           \
        else if ((dtype) == PCX_F16) { using T = __half; if (vec) { constexpr int VN = 8; CALL; } else { constexpr int VN = 1; CALL; } }      \
        else { using T = __nv_bfloat16; if (vec) { constexpr int VN = 8; CALL; } else { constexpr int VN = 1; CALL; } }                       \
    } while (0)

}  // namespace
}  // namespace pcx

using namespace pcx;

extern "C" {

size_t pcx_ragged_layer_norm_workspace_bytes(int64_t N, int64_t S) {
    return (S <= 0 || N < 0) ? 0 : carve_ln(nullptr, S, nullptr, ln_pieces(N, S));
}

int pcx_ragged_layer_norm(const void *d_x, const int64_t *d_lengths, const float *d_weight, const float *d_bias,
                          const void *d_residual, void *d_y, float *d_mean, float *d_rstd, int64_t N, int64_t S, int C,
                          double eps, int relu, int dtype, void *d_ws, size_t ws_bytes, void *stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    if (!ln_sizes_ok(N, S, C, dtype)) PCX_FAIL(PCX_E_ARG, "pcx_ragged_layer_norm: bad sizes or dtype");
    if (!d_lengths || !d_mean || !d_rstd || !d_ws || (N > 0 && (!d_x || !d_y)) || ((d_weight == nullptr) != (d_bias == nullptr)))
        PCX_FAIL(PCX_E_ARG, "pcx_ragged_layer_norm: null pointer (weight and bias come together)");
    if ((uintptr_t)d_ws % 256) PCX_FAIL(PCX_E_ALIGN, "pcx_ragged_layer_norm: workspace must be 256-byte aligned");
    LnWs w;
    size_t need = carve_ln(d_ws, S, &w, ln_pieces(N, S));
    if (ws_bytes < need) PCX_FAIL(PCX_E_CAPACITY, "pcx_ragged_layer_norm: workspace %zu < %zu bytes", ws_bytes, need);
    prof_begin("layer_norm(fwd)", stream);   // all of its kernels
    if (S <= FEW && N > 0 && N * C * (int64_t)elem_size(dtype) <= FEW_BYTES) {
        const bool wide = vec_ok(C, dtype, {d_x, d_y, d_residual});
        int blocks = 0, rc = NOT_TOGETHER;
        PCX_LN_DISPATCH(dtype, wide, {
            static int resident = 0;
            blocks = std::min(FEW_BLOCKS, few_blocks(ln_few_kernel<T, VN>, N, C, dtype, wide, &resident));
            if (blocks > 0)
                rc = launch_together(ln_few_kernel<T, VN>, blocks, stream, (const T *)d_x, d_lengths, d_weight, d_bias, (const T *)d_residual, (T *)d_y, d_mean,
                                     d_rstd, w.rec, N, (int)S, C, (float)eps, relu);
        });
        if (rc != NOT_TOGETHER) {
            prof_end(stream);
            return rc;
        }
    }
    if (int rc = ln_offsets(d_lengths, S, N, w, stream)) return rc;
    const bool vec = vec_ok(C, dtype, {d_x, d_y, d_residual});
    const int mom_rows = layer_rows(N, C, dtype, vec, 4), rows = layer_rows(N, C, dtype, vec, 5);
    if (N > 0) {
        const unsigned mgrid = (unsigned)((N + mom_rows - 1) / mom_rows);
        PCX_LN_DISPATCH(dtype, vec, (launch_after(ln_moments_kernel<T, VN>, mgrid, LN_THREADS, 0, stream, (const T *)d_x, w.offsets, w.rec, N, S, C, mom_rows)));
        PCX_LAUNCH_CHECK();
    }
    launch_after(ln_combine_kernel, (unsigned)S, COMBINE_THREADS, 0, stream, w.rec, w.offsets, d_mean, d_rstd, S, (float)eps, mom_rows);
    PCX_LAUNCH_CHECK();
    if (N > 0) {
        PCX_LN_DISPATCH(dtype, vec, (launch_after(ln_apply_kernel<T, VN>, (unsigned)((N + rows - 1) / rows), LN_THREADS, 0, stream, 
                                   (const T *)d_x, w.offsets, d_mean, d_rstd, d_weight, d_bias, (const T *)d_residual,
                                   (T *)d_y, N, S, C, relu, rows)));
        PCX_LAUNCH_CHECK();
    }
    prof_end(stream);
    return PCX_OK;
}

int pcx_ragged_layer_norm_backward(const void *d_grad_y, const void *d_x, const void *d_y, const int64_t *d_lengths,
                                   const float *d_weight, const float *d_mean, const float *d_rstd, void *d_grad_x,
                                   float *d_grad_weight, float *d_grad_bias, void *d_grad_residual, int64_t N,
                                   int64_t S, int C, int relu, int dtype, void *d_ws, size_t ws_bytes, void *stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    if (!ln_sizes_ok(N, S, C, dtype)) PCX_FAIL(PCX_E_ARG, "pcx_ragged_layer_norm_backward: bad sizes or dtype");
    if (!d_lengths || !d_mean || !d_rstd || !d_ws || (N > 0 && (!d_grad_y || !d_x || !d_grad_x)) || (relu && N > 0 && !d_y) ||
        ((d_grad_weight == nullptr) != (d_grad_bias == nullptr)))
        PCX_FAIL(PCX_E_ARG, "pcx_ragged_layer_norm_backward: null pointer");
    if ((uintptr_t)d_ws % 256) PCX_FAIL(PCX_E_ALIGN, "pcx_ragged_layer_norm_backward: workspace must be 256-byte aligned");
    LnWs w;
    size_t need = carve_ln(d_ws, S, &w, ln_pieces(N, S));
    if (ws_bytes < need) PCX_FAIL(PCX_E_CAPACITY, "pcx_ragged_layer_norm_backward: workspace %zu < %zu bytes", ws_bytes, need);
    prof_begin("layer_norm(bwd)", stream);
    const bool one_pass = C / (vec_ok(C, dtype, {d_grad_y, d_x, d_y, d_grad_x, d_grad_residual}) ? 16 / (int)elem_size(dtype) : 1) <= LN_THREADS;
    if (S <= FEW && N > 0 && one_pass && N * C * (int64_t)elem_size(dtype) <= FEW_BYTES) {
        const bool wide = vec_ok(C, dtype, {d_grad_y, d_x, d_y, d_grad_x, d_grad_residual});
        int blocks = 0, rc = NOT_TOGETHER;
        PCX_LN_DISPATCH(dtype, wide, {
            static int resident = 0;
            blocks = std::min(FEW_BLOCKS, few_blocks(ln_few_bwd_kernel<T, VN>, N, C, dtype, wide, &resident));
            if (blocks > 0)
                rc = launch_together(ln_few_bwd_kernel<T, VN>, blocks, stream, (const T *)d_grad_y, (const T *)d_x, (const T *)d_y, d_lengths, d_mean, d_rstd,
                                     d_weight, (float2 *)w.rec, d_grad_weight, d_grad_bias, (T *)d_grad_residual, (T *)d_grad_x, N, (int)S, C, relu);
        });
        if (rc != NOT_TOGETHER) {
            prof_end(stream);
            return rc;
        }
    }
    if (int rc = ln_offsets(d_lengths, S, N, w, stream, true, d_grad_weight, d_grad_bias, C)) return rc;
    if (N == 0) return PCX_OK;
    const bool vec = vec_ok(C, dtype, {d_grad_y, d_x, d_y, d_grad_x, d_grad_residual});
    const int rows = layer_rows(N, C, dtype, vec, 4);
    const unsigned grid = (unsigned)((N + rows - 1) / rows);
    PCX_LN_DISPATCH(dtype, vec, (launch_after(ln_bwd_sums_kernel<T, VN>, grid, LN_THREADS, 0, stream, 
                               (const T *)d_grad_y, (const T *)d_x, (const T *)d_y, w.offsets, d_mean, d_rstd, d_weight,
                               w.sums, w.sums + S, d_grad_weight, d_grad_bias, (T *)d_grad_residual, N, S, C, relu, rows)));
    PCX_LAUNCH_CHECK();
    // the sums pass wrote the ReLU-masked gradient as the residual's gradient: the second pass reads
    // that instead of masking again, which spares it the read of y
    const bool masked = relu && d_grad_residual;
    PCX_LN_DISPATCH(dtype, vec, (launch_after(ln_bwd_apply_kernel<T, VN>, grid, LN_THREADS, 0, stream, 
                               (const T *)(masked ? d_grad_residual : d_grad_y), (const T *)d_x, (const T *)d_y, w.offsets,
                               d_mean, d_rstd, d_weight, w.sums, w.sums + S, (T *)d_grad_x, N, S, C, masked ? 0 : relu, rows)));
    prof_end(stream);
    PCX_LAUNCH_CHECK();
    return PCX_OK;
}

size_t pcx_ragged_group_norm_workspace_bytes(int64_t S, int G) {
    return (S <= 0 || G <= 0 || S * (int64_t)G > INT32_MAX) ? 0 : carve_ln(nullptr, S * G, nullptr);
}

int pcx_ragged_group_norm(const void *d_x, const int64_t *d_lengths, const float *d_weight, const float *d_bias,
                          void *d_y, float *d_mean, float *d_rstd, int64_t N, int64_t S, int C, int G, double eps,
                          int dtype, void *d_ws, size_t ws_bytes, void *stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    if (!ln_sizes_ok(N, S, C, dtype) || G <= 0 || C % G || S * (int64_t)G > INT32_MAX || G > 8192)
        PCX_FAIL(PCX_E_ARG, "pcx_ragged_group_norm: bad sizes or dtype (C must be a multiple of G <= 8192)");
    if (!d_lengths || !d_mean || !d_rstd || !d_ws || (N > 0 && (!d_x || !d_y)) || ((d_weight == nullptr) != (d_bias == nullptr)))
        PCX_FAIL(PCX_E_ARG, "pcx_ragged_group_norm: null pointer (weight and bias come together)");
    if ((uintptr_t)d_ws % 256) PCX_FAIL(PCX_E_ALIGN, "pcx_ragged_group_norm: workspace must be 256-byte aligned");
    const int64_t SG = S * G;
    LnWs w;
    size_t need = carve_ln(d_ws, SG, &w);
    if (ws_bytes < need) PCX_FAIL(PCX_E_CAPACITY, "pcx_ragged_group_norm: workspace %zu < %zu bytes", ws_bytes, need);
    if (int rc = ln_offsets(d_lengths, S, N, w, stream)) return rc;
    PCX_CUDA(cudaMemsetAsync(w.sums, 0, (size_t)2 * SG * sizeof(float), stream));
    const unsigned grid = (unsigned)((N + LN_ROWS - 1) / LN_ROWS), sgrid = (unsigned)((SG + 127) / 128);
    const bool vec = vec_ok(C, dtype, {d_x, d_y});
    const size_t smem = (size_t)G * sizeof(float);
    const int W = C / G;
    for (int second = 0; second < 2; ++second) {
        if (N > 0) {
            PCX_LN_DISPATCH(dtype, vec, (gn_sum_kernel<T, VN><<<grid, LN_THREADS, smem, stream>>>(
                                       (const T *)d_x, w.offsets, second ? d_mean : nullptr, w.sums + second * SG, N, S, C, G)));
            PCX_LAUNCH_CHECK();
        }
        gn_stats_kernel<<<sgrid, 128, 0, stream>>>(w.sums + second * SG, w.offsets, d_mean, d_rstd, S, G, W, (float)eps, second);
        PCX_LAUNCH_CHECK();
    }
    if (N > 0) {
        prof_begin("gn_apply_kernel", stream);
        PCX_LN_DISPATCH(dtype, vec, (gn_apply_kernel<T, VN><<<grid, LN_THREADS, 0, stream>>>(
                                   (const T *)d_x, w.offsets, d_mean, d_rstd, d_weight, d_bias, (T *)d_y, N, S, C, G)));
        prof_end(stream);
        PCX_LAUNCH_CHECK();
    }
    return PCX_OK;
}

int pcx_ragged_group_norm_backward(const void *d_grad_y, const void *d_x, const int64_t *d_lengths,
                                   const float *d_weight, const float *d_mean, const float *d_rstd, void *d_grad_x,
                                   float *d_grad_weight, float *d_grad_bias, int64_t N, int64_t S, int C, int G,
                                   int dtype, void *d_ws, size_t ws_bytes, void *stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    if (!ln_sizes_ok(N, S, C, dtype) || G <= 0 || C % G || S * (int64_t)G > INT32_MAX || G > 4096)
        PCX_FAIL(PCX_E_ARG, "pcx_ragged_group_norm_backward: bad sizes or dtype (C must be a multiple of G <= 4096)");
    if (!d_lengths || !d_mean || !d_rstd || !d_ws || (N > 0 && (!d_grad_y || !d_x || !d_grad_x)) ||
        ((d_grad_weight == nullptr) != (d_grad_bias == nullptr)))
        PCX_FAIL(PCX_E_ARG, "pcx_ragged_group_norm_backward: null pointer");
    if ((uintptr_t)d_ws % 256) PCX_FAIL(PCX_E_ALIGN, "pcx_ragged_group_norm_backward: workspace must be 256-byte aligned");
    const int64_t SG = S * G;
    LnWs w;
    size_t need = carve_ln(d_ws, SG, &w);
    if (ws_bytes < need) PCX_FAIL(PCX_E_CAPACITY, "pcx_ragged_group_norm_backward: workspace %zu < %zu bytes", ws_bytes, need);
    if (int rc = ln_offsets(d_lengths, S, N, w, stream)) return rc;
    PCX_CUDA(cudaMemsetAsync(w.sums, 0, (size_t)2 * SG * sizeof(float), stream));
    if (d_grad_weight) {
        PCX_CUDA(cudaMemsetAsync(d_grad_weight, 0, (size_t)C * sizeof(float), stream));
        PCX_CUDA(cudaMemsetAsync(d_grad_bias, 0, (size_t)C * sizeof(float), stream));
    }
    if (N == 0) return PCX_OK;
    const unsigned grid = (unsigned)((N + LN_ROWS - 1) / LN_ROWS);
    const bool vec = vec_ok(C, dtype, {d_grad_y, d_x, d_grad_x});
    PCX_LN_DISPATCH(dtype, vec, (gn_bwd_sums_kernel<T, VN><<<grid, LN_THREADS, (size_t)2 * G * sizeof(float), stream>>>(
                               (const T *)d_grad_y, (const T *)d_x, w.offsets, d_mean, d_rstd, d_weight, w.sums, w.sums + SG,
                               d_grad_weight, d_grad_bias, N, S, C, G)));
    PCX_LAUNCH_CHECK();
    PCX_LN_DISPATCH(dtype, vec, (gn_bwd_apply_kernel<T, VN><<<grid, LN_THREADS, 0, stream>>>(
                               (const T *)d_grad_y, (const T *)d_x, w.offsets, d_mean, d_rstd, d_weight, w.sums, w.sums + SG,
                               (T *)d_grad_x, N, S, C, G)));
    PCX_LAUNCH_CHECK();
    return PCX_OK;
}

}  // extern "C"
