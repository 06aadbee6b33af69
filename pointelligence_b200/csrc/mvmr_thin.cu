// MVMR of layers with few input channels (a network's stem: 3 or 6 channels, 27 or 125 taps), on sm_100a.
//
// Such a layer hardly multiplies; on the scatter kernel it is bound by adding a row of fp32 sums per triplet in the L2.
// Here the sums of 128 consecutive output rows stay in tensor memory: the operand of a block is the matrix (128 rows) x
// (taps x 8 channels), a row's features of all its taps side by side, built 64 columns at a time in shared memory, and
// multiplied with the weights as one long contraction.  No plan, no accumulator to clear, to add
// to or to round, and operands as they are: up to eight triplets of a (row, tap) are multiplied one by one.
//
//   preparation   two kernels: the table of a block, [tap][row], holds a feature row, where a (row, tap) has one triplet, or
//                 the first of its several triplets and their number (rows ascend inside a tap, so that they are neighbours);
//                 the weights as the tiles that the tensor core reads; feature rows of eight channels
//   clumps        the features of more than eight triplets are added up in fp32, and the sum is handed on as three 16-bit rows that
//                 hold all its bits, so that a step is taken for at most eight triplets, not for each of the fullest (row, tap)
//                 of 128 rows and eight taps: 100 000 points, of which 200 / 400 / 1000 lie within a centimetre, rows in random order,
//                 27 taps, 6 -> 64 channels 269 / 567 / 1474 -> 56 / 59 / 69 us (scatter kernel 61 / 74 / 144).  Sums beyond the
//                 type's range (and infinities, NaN) stay triplets
//   copies        eight warps, eight taps a step: every (row, tap) a 16-byte copy, or zeros, straight into the
//                 128-byte-swizzled tile.  Where a (row, tap) has several triplets the columns take a step for the
//                 first of each, one for the second of those that have one, and so on
//   MMA thread    four tcgen05.mma (M = 128, N = up to 64 output channels, K = 16) a step; the weights come as bulk copies
//   epilogue      tensor memory + bias, rounded once, rows written side by side
//
// 80 000 points, 125 taps, 3.3 M triplets, 6 -> 32 channels: 170 us on the scatter kernel with its padded copies, clear and rounding,
// 142 here (preparation 8 and 18, this kernel 116).  A step takes some 2000 clocks of a CTA, three of which share an SM: bound
// by the load/store unit and by the fill warps' own instructions.  16-byte copies of 32 rows are taken a lane a clock, whether or
// not a lane has a source, so that zeros are stores.  Slower: tables of a block built by warps beside the copies (in three
// forms, 107 -> 190 us of the kernel at 3 M triplets), second triplets multiplied by the warp that finds them and added in shared
// memory (390), feature rows fetched a slot early (10 %).  16 channels a tap lost to the other kernels everywhere.
//
// Weights that are not finite (a zero in the operand would make no number of them): the same kernel works triplet by
// triplet, slowly, and as the scatter kernel has it.
//
// Every wait is bounded (one second) and abortable, as in the other tensor kernels.
#include "sparse_kernels.cuh"
#include "tcgen05.cuh"

namespace pcx {
int device_status_address(unsigned int **d_status);

namespace {

using namespace tc;

constexpr unsigned STATUS_BIT = 16u;
constexpr int ROWS = 128, A_BYTES = ROWS * 128;       // a step's operand: 128 rows of 64 columns
constexpr int CW = 8, TPS = 64 / CW;                  // channels of a tap, taps of a step
constexpr int MAX_TAPS = 512, MAX_N = 64, MAX_WIDTH = 1024;
constexpr int SLOTS = 3;                              // operand tiles on their way or in use
constexpr int WARPS = 8, MMA_WARP = WARPS, THREADS = (WARPS + 1) * 32, CTAS = 3;   // CTAs of an SM
constexpr int PREP_THREADS = 256, PREP_CTAS = 8;      // of an SM
// an entry of the table: a feature row; none; or 1 << 31 | a code << 27 | the first of several triplets, or the number of a sum.
// The code is the number of triplets - 2, or:
constexpr int32_t NONE = -1;
constexpr int FIRST_BITS = 27, LISTED = 8;            // triplets that are multiplied one by one, at most
constexpr int MORE = 14, SUMMED = 15;                 // more than that, to be counted; the sum of more than that
constexpr int64_t MAX_T = ((int64_t)1 << FIRST_BITS) - 1;
constexpr int PARTS = 3;                              // rows of a sum: 3 x 8 bits of bf16, 3 x 11 of fp16
constexpr size_t SUM_BYTES = PARTS * CW * 2;

struct ThinParams {
    const uint16_t *feat;                 // rows of CW elements: the points, then PARTS for every sum
    const int32_t *gather, *scatter;
    const int64_t *seg;
    const int32_t *table;                 // [block][tap][row]
    const int2 *most;                     // [block][slot]: steps of the fullest (row, tap), at least 1; whether codes are beyond LISTED
    const uint16_t *image;                // [part][slot][N][64]: the weights' tiles, swizzled
    const uint32_t *odd;                  // whether weights are not finite, a word for each block of the preparation
    const uint16_t *bias;
    uint16_t *out;
    unsigned int *status;
    int64_t n_out;
    int K, nq, N, width, nblocks, n_odd, fmt;   // nq: slots (of 64 columns) of a block; N: output channels of a part; width: all
    uint32_t ncols, col_stride, slot_bytes;
    uint32_t first_sum;                   // row of the first sum
};

struct PrepParams {
    const uint16_t *weight, *feat_in;
    uint16_t *feat;
    const int32_t *scatter, *gather;
    const int64_t *seg;
    int32_t *table;
    int2 *most;
    uint16_t *image;
    uint32_t *odd, *n_sums;
    int64_t T, n_feat, image_pieces, table_pieces, most_pieces;
    uint32_t max_sums;
    int K, inw, width, nq, N, transpose, reverse, fmt;
};

__device__ __forceinline__ float widen_one(uint32_t v, int fmt) {   // the low 16 bits
    return fmt ? __uint_as_float(v << 16) : __half2float(__ushort_as_half((uint16_t)v));
}
__device__ __forceinline__ uint32_t pack2(float a, float b, int fmt) {
    if (fmt) {
        __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
        return *reinterpret_cast<uint32_t *>(&v);
    }
    __half2 v = __floats2half2_rn(a, b);
    return *reinterpret_cast<uint32_t *>(&v);
}

// The weights' tiles, the features' rows, and an empty table.
__global__ void __launch_bounds__(PREP_THREADS) thin_prepare_kernel(PrepParams p) {
    start_after_previous();
    const int64_t x0 = blockIdx.x * (int64_t)PREP_THREADS + threadIdx.x, threads = (int64_t)gridDim.x * PREP_THREADS;
    for (int64_t x = x0; x < p.table_pieces; x += threads) reinterpret_cast<int4 *>(p.table)[x] = make_int4(NONE, NONE, NONE, NONE);
    for (int64_t x = x0; x < p.most_pieces; x += threads) p.most[x] = make_int2(1, 0);
    bool odd = false;
    for (int64_t x = x0; x < p.image_pieces; x += threads) {
        // [part][slot][n][piece]
        const int piece = (int)(x & 7), n = (int)(x >> 3) % p.N, slot = (int)((x >> 3) / p.N) % p.nq, part = (int)((x >> 3) / p.N / p.nq);
        const int k = slot * TPS + piece, o = part * p.N + n;
        uint32_t v[4] = {0u, 0u, 0u, 0u};
        if (k < p.K && o < p.width) {
            const int tap = p.reverse ? p.K - 1 - k : k;
            const uint16_t *src = p.weight + (int64_t)tap * p.inw * p.width + (p.transpose ? (int64_t)o * p.inw : o);
            const int step = p.transpose ? 1 : p.width;
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                if (e >= p.inw) continue;
                const uint32_t u = __ldg(src + (int64_t)e * step), most = p.fmt ? 0x7f80u : 0x7c00u;
                odd |= (u & most) == most;
                v[e >> 1] |= u << (16 * (e & 1));
            }
        }
        // (N is a multiple of 16, so that rows of a tile keep their place modulo 8)
        reinterpret_cast<uint4 *>(p.image)[(x >> 3) * 8 + (piece ^ (n & 7))] = make_uint4(v[0], v[1], v[2], v[3]);
    }
    if (x0 == 0) *p.n_sums = 0u;
    for (int64_t x = x0; x < p.n_feat; x += threads) {
        uint32_t v[4] = {0u, 0u, 0u, 0u};
#pragma unroll
        for (int e = 0; e < 8; ++e)
            if (e < p.inw) v[e >> 1] |= (uint32_t)__ldg(p.feat_in + x * p.inw + e) << (16 * (e & 1));
        reinterpret_cast<uint4 *>(p.feat)[x] = make_uint4(v[0], v[1], v[2], v[3]);
    }
    const int any = __syncthreads_or(odd);
    if (threadIdx.x == 0) p.odd[blockIdx.x] = (uint32_t)any;
}

// The triplets from `first` on that have this row (of the tap that ends at `end`), by a whole warp: what enters the table for
// them, and the steps that takes.  An iteration takes 64, three loads one after the other: a clump of 400 points among 100 000 takes 8 us,
// one of 1000 17.
__device__ __forceinline__ int2 sum_up(const PrepParams &p, int64_t first, int64_t end, int32_t row, uint32_t id) {
    const int lane = threadIdx.x & 31;
    float sum[CW];
#pragma unroll
    for (int c = 0; c < CW; ++c) sum[c] = 0.f;
    int n = 0;
    for (int64_t t0 = first;; t0 += 64) {
        bool mine[2];
        uint4 v[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int64_t t = t0 + 32 * u + lane;
            mine[u] = t < end && __ldg(p.scatter + t) == row;
            v[u] = mine[u] ? *reinterpret_cast<const uint4 *>(p.feat + (int64_t)__ldg(p.gather + t) * CW) : make_uint4(0u, 0u, 0u, 0u);
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const uint32_t word[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
#pragma unroll
            for (int c = 0; c < CW; ++c)
                if (mine[u]) sum[c] += widen_one(word[c >> 1] >> (16 * (c & 1)) & 0xffffu, p.fmt);
        }
        n += __popc(__ballot_sync(0xffffffffu, mine[0])) + __popc(__ballot_sync(0xffffffffu, mine[1]));
        if (!__all_sync(0xffffffffu, mine[1])) break;   // (they are neighbours)
    }
    uint32_t word[4] = {0u, 0u, 0u, 0u};   // lane q: part q
    bool in_range = true;
#pragma unroll
    for (int c = 0; c < CW; ++c) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum[c] += __shfl_xor_sync(0xffffffffu, sum[c], o);
        float rest = sum[c];
#pragma unroll
        for (int q = 0; q < PARTS; ++q) {   // (each difference is exact, the last part leaves none)
            const uint32_t part = pack2(rest, 0.f, p.fmt) & 0xffffu, most = p.fmt ? 0x7f80u : 0x7c00u;
            rest -= widen_one(part, p.fmt);
            if (q == 0) in_range = in_range && (part & most) != most;
            if (q == lane) word[c >> 1] |= part << (16 * (c & 1));
        }
    }
    if (!in_range || id >= p.max_sums) return make_int2((int32_t)(1u << 31 | (uint32_t)MORE << FIRST_BITS | (uint32_t)first), n);
    if (lane < PARTS) *reinterpret_cast<uint4 *>(p.feat + (p.n_feat + (int64_t)id * PARTS + lane) * CW) = make_uint4(word[0], word[1], word[2], word[3]);
    return make_int2((int32_t)(1u << 31 | (uint32_t)SUMMED << FIRST_BITS | id), PARTS);
}

// The first triplet of every (row, tap) enters the table, or the sum of its triplets.
__global__ void __launch_bounds__(PREP_THREADS, 8) thin_table_kernel(const __grid_constant__ PrepParams p) {
    wait_for_previous();
    constexpr int EACH = 4;   // triplets of a thread
    constexpr int CLUMPS = (32 * EACH + LISTED) / (LISTED + 1);   // runs of more than LISTED that begin among the triplets of a warp
    __shared__ int64_t s_seg[MAX_TAPS + 1];
    __shared__ int4 s_clump[PREP_THREADS / 32][CLUMPS];   // first triplet, tap, row
    __shared__ int s_clumps[PREP_THREADS / 32];
    __shared__ uint32_t s_sum[PREP_THREADS / 32];   // number of a warp's first sum
    // What the block has said about a slot already (slot << 32 | steps << 1 | beyond), said again only where it is more: of a dense cloud,
    // whose triplets meet few slots, a word each went to the same few lines of the L2 (7.4 M triplets of 10 000 points: 1.3 ms).
    constexpr int SEEN = 64;
    __shared__ uint64_t s_seen[SEEN];
    if (threadIdx.x < SEEN) s_seen[threadIdx.x] = ~0ull;
    for (int k = threadIdx.x; k <= p.K; k += PREP_THREADS) s_seg[k] = p.seg[k];
    if (threadIdx.x < PREP_THREADS / 32) s_clumps[threadIdx.x] = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t t0 = (blockIdx.x * (int64_t)(PREP_THREADS / 32) + warp) * (32 * EACH) + lane;
    int k = 0, hi = p.K;   // last tap that begins at t0 or before
    while (hi - k > 1) {
        const int mid = (k + hi) >> 1;
        if (s_seg[mid] <= t0) k = mid; else hi = mid;
    }
    auto enter = [&](int32_t row, int tap, int32_t entry, int steps, bool beyond) {
        const int64_t block = row >> 7;
        p.table[(block * p.K + tap) * ROWS + (row & (ROWS - 1))] = entry;
        if (steps <= 1) return;
        const uint32_t slot = (uint32_t)(block * p.nq) + (uint32_t)(tap / TPS), said = (uint32_t)steps << 1 | (uint32_t)beyond;
        volatile uint64_t *seen = s_seen + slot % SEEN;
        const uint64_t last = *seen;
        const uint32_t known = (uint32_t)(last >> 32) == slot ? (uint32_t)last : 0u;
        if (known >= said && (known & 1u) >= (said & 1u)) return;
        int2 *most = p.most + slot;
        if (*(volatile int32_t *)&most->x < steps) atomicMax(&most->x, steps);
        if (beyond) most->y = 1;
        *seen = (uint64_t)slot << 32 | max(known | (said & 1u), said | (known & 1u));
    };
    int32_t row[EACH], prev[EACH], point[EACH];
#pragma unroll
    for (int u = 0; u < EACH; ++u) {
        const int64_t t = t0 + 32 * u;
        row[u] = t < p.T ? __ldg(p.scatter + t) : 0;
        prev[u] = t < p.T && t > 0 ? __ldg(p.scatter + t - 1) : -1;
        point[u] = t < p.T ? __ldg(p.gather + t) : 0;
    }
#pragma unroll
    for (int u = 0; u < EACH; ++u) {
        const int64_t t = t0 + 32 * u;
        while (k + 1 < p.K && s_seg[k + 1] <= t) ++k;
        if (t >= p.T || t < s_seg[k] || t >= s_seg[k + 1] || (t > s_seg[k] && prev[u] == row[u])) continue;
        int many = 1;
        while (many <= LISTED && t + many < s_seg[k + 1] && __ldg(p.scatter + t + many) == row[u]) ++many;
        if (many > LISTED) s_clump[warp][atomicAdd(&s_clumps[warp], 1)] = make_int4((int32_t)t, k, row[u], 0);
        else enter(row[u], k, many == 1 ? point[u] : (int32_t)(1u << 31 | (uint32_t)(many - 2) << FIRST_BITS | (uint32_t)t), many, false);
    }
    // a number for every sum, an addition a block
    if (__syncthreads_or(lane == 0 && s_clumps[warp] > 0)) {
        if (warp == 0) {
            int before = 0, all = 0;
#pragma unroll
            for (int w = 0; w < PREP_THREADS / 32; ++w) {
                if (w < lane) before += s_clumps[w];
                all += s_clumps[w];
            }
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(p.n_sums, (uint32_t)all);
            base = __shfl_sync(0xffffffffu, base, 0);
            if (lane < PREP_THREADS / 32) s_sum[lane] = base + (uint32_t)before;
        }
        __syncthreads();
        for (int x = 0, n = s_clumps[warp]; x < n; ++x) {
            const int4 c = s_clump[warp][x];
            const int2 entry = sum_up(p, c.x, s_seg[c.y + 1], c.z, s_sum[warp] + (uint32_t)x);
            if (lane == 0) enter(c.z, c.y, entry.x, entry.y, true);
        }
    }
    let_next_be_set_up();   // only now: see mvmr_thin_kernel
}

// A row of a part: sums (+ bias), rounded.
__device__ __forceinline__ void store16(const ThinParams &p, int64_t row, int col, float *v) {
    const int left = p.width - col;
    if (p.bias) {
#pragma unroll
        for (int e = 0; e < 16; ++e)
            if (e < left) v[e] += widen_one(__ldg(p.bias + col + e), p.fmt);
    }
    uint16_t *dst = p.out + row * p.width + col;
    if ((p.width & 7) == 0) {
#pragma unroll
        for (int e = 0; e < 2; ++e)
            if (8 * e < left)
                reinterpret_cast<uint4 *>(dst)[e] = make_uint4(pack2(v[8 * e], v[8 * e + 1], p.fmt), pack2(v[8 * e + 2], v[8 * e + 3], p.fmt),
                                                               pack2(v[8 * e + 4], v[8 * e + 5], p.fmt), pack2(v[8 * e + 6], v[8 * e + 7], p.fmt));
    } else {
#pragma unroll
        for (int e = 0; e < 16; ++e)
            if (e < left) dst[e] = (uint16_t)pack2(v[e], 0.f, p.fmt);
    }
}

// Triplet by triplet: a warp a tap, a lane an output channel.
__device__ __noinline__ void one_by_one(const ThinParams &p, float *sums, int part) {
    const int pitch = p.N + 1, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int b = blockIdx.x; b < p.nblocks; b += gridDim.x) {
        for (int x = threadIdx.x; x < ROWS * pitch; x += THREADS) sums[x] = 0.f;
        __syncthreads();
        for (int k = warp; k < p.K; k += THREADS / 32) {
            int64_t bound[2];   // the block's triplets of the tap
            for (int e = 0; e < 2; ++e) {
                int64_t lo = p.seg[k], hi = p.seg[k + 1];
                while (lo < hi) {
                    const int64_t mid = (lo + hi) >> 1;
                    if (p.scatter[mid] < (int64_t)(b + e) * ROWS) lo = mid + 1; else hi = mid;
                }
                bound[e] = lo;
            }
            const uint16_t *tile = p.image + ((int64_t)(part * p.nq + k / TPS) * p.N) * 64;
            for (int64_t t = bound[0]; t < bound[1]; ++t) {
                const int64_t row = (int64_t)p.scatter[t] - (int64_t)b * ROWS;
                if (row < 0 || row >= ROWS) continue;
                const uint16_t *x = p.feat + (int64_t)p.gather[t] * CW;
                for (int n = lane; n < p.N; n += 32) {
                    float s = 0.f;
                    for (int c = 0; c < CW; ++c)
                        s = fmaf(widen_one(__ldg(x + c), p.fmt), widen_one(__ldg(tile + n * 64 + ((k % TPS ^ (n & 7)) << 3) + c), p.fmt), s);
                    atomicAdd(sums + row * pitch + n, s);
                }
            }
        }
        __syncthreads();
        for (int x = threadIdx.x; x < ROWS * (p.N / 16); x += THREADS) {
            const int r = x % ROWS, c = x / ROWS * 16;
            if ((int64_t)b * ROWS + r >= p.n_out || part * p.N + c >= p.width) continue;
            float v[16];
            for (int e = 0; e < 16; ++e) v[e] = sums[r * pitch + c + e];
            store16(p, (int64_t)b * ROWS + r, part * p.N + c, v);
        }
        __syncthreads();
    }
}

// The slots of a CTA's blocks, one after the other.
struct At {
    int n = 0, q = 0;   // block of the CTA, slot
    __device__ __forceinline__ void next(int nq) {
        if (++q == nq) q = 0, ++n;
    }
};

// Row `j` of `base` (rows of 16 bytes), or, for NONE, zeros: by a store, four clocks for 32 lanes, where a copy
// takes a clock a lane with or without a source.
__device__ __forceinline__ void copy_or_zeros(uint32_t dst, const uint16_t *base, int32_t j) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 s;\n\tsetp.ne.s32 p, %2, -1;\n\tmad.wide.u32 s, %2, %3, %1;\n\t"
        "@p cp.async.cg.shared.global [%0], [s], 16;\n\t@!p st.shared.v4.b32 [%0], {%4, %4, %4, %4};\n\t}"
        ::"r"(dst), "l"(base), "r"(j), "r"(CW * 2), "r"(0u) : "memory");
}
// a[at] where `there`, else `other`
__device__ __forceinline__ int32_t load_if(bool there, const int32_t *a, int32_t at, int32_t other) {
    int32_t v = other;
    asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 s;\n\tsetp.ne.u32 p, %1, 0;\n\tmad.wide.s32 s, %3, 4, %2;\n\t@p ld.global.nc.b32 %0, [s];\n\t}"
                 : "+r"(v) : "r"((uint32_t)there), "l"(a), "r"(at));
    return v;
}

// The copies of a slot where some row has the sum of a clump, or more than LISTED triplets, of one of the eight taps: in a function
// of its own, so that the registers and the schedule of the ordinary slots stay as they are.  What the ring, the verdict and the last
// weights are afterwards.
__device__ __noinline__ int4 clump_slot(const ThinParams &p, uint64_t *s_full, uint64_t *s_empty, volatile int *abort_flag, const At now, const int row, const int x0,
                                        const int part, const uint32_t slot0, const int4 e4, const int steps, Ring ring, uint32_t last_load) {
    constexpr int CELLS = TPS / 2;
    const int32_t e[CELLS] = {e4.x, e4.y, e4.z, e4.w};
    const int64_t block = (int64_t)blockIdx.x + (int64_t)now.n * gridDim.x;
    int32_t j[CELLS], left[CELLS], t[CELLS];
    uint32_t sums = 0;   // of this lane's cells; t of a sum is its first row
    // (what a load may replace is known before: nothing waits for one here)
#pragma unroll
    for (int x = 0; x < CELLS; ++x) {
        const bool several = e[x] < NONE;
        t[x] = (e[x] & (int32_t)MAX_T) + 1;
        left[x] = several ? (int)((uint32_t)e[x] >> FIRST_BITS & 15u) + 1 : 0;
        const bool sum = left[x] == SUMMED + 1;
        if (sum) sums |= 1u << x, t[x] = (int32_t)(p.first_sum + (uint32_t)(t[x] - 1) * PARTS), left[x] = 0;
        if (left[x] == MORE + 1) {
            const int64_t end = p.seg[now.q * TPS + x0 + x + 1], i = block * ROWS + row;
            left[x] = LISTED;
            while ((int64_t)t[x] + left[x] < end && p.scatter[t[x] + left[x]] == i) ++left[x];
        }
        j[x] = load_if(several && !sum, p.gather - 1, t[x], sum ? t[x] : e[x]);
    }
    bool ok = true;
    for (int m = 0; m < steps; ++m) {
        int32_t j_next[CELLS];
#pragma unroll
        for (int x = 0; x < CELLS; ++x) j_next[x] = load_if(left[x] > m, p.gather, t[x] + m, (sums >> x & 1u) && m + 1 < PARTS ? t[x] + m + 1 : NONE);
        const uint32_t empty = smem_u32(&s_empty[ring.slot]), parity = (ring.turn ^ 1u) & 1u;
        ok = __all_sync(0xffffffffu, mbar_try_wait(empty, parity)) ||
             __all_sync(0xffffffffu, mbar_wait_abortable(empty, parity, STATUS_BIT, p.status, abort_flag));
        if (!ok) break;
        const uint32_t tile = slot0 + ring.slot * p.slot_bytes, full = smem_u32(&s_full[ring.slot]);
        if (threadIdx.x == 0) {
            mbar_arrive_expect_tx(full, (uint32_t)p.N * 128u);
            bulk_load(tile + A_BYTES, p.image + ((int64_t)(part * p.nq + now.q) * p.N) * 64, (uint32_t)p.N * 128u, full);
            last_load = ring.slot | (ring.turn & 1u) << 8 | 1u << 16;
        }
#pragma unroll
        for (int x = 0; x < CELLS; ++x) {
            copy_or_zeros(tile + (uint32_t)row * 128 + (uint32_t)(((x0 + x) ^ (row & 7)) << 4), p.feat, j[x]);
            j[x] = j_next[x];
        }
        cp_async_mbar_arrive(full);
        __syncwarp();
        if ((threadIdx.x & 31) == 0) mbar_arrive(full);
        ring.next(SLOTS);
    }
    return make_int4((int)ring.slot, (int)ring.turn, ok, (int)last_load);
}

// The grid is one wave, three CTAs on every multiprocessor, of which some have a block more to do than others; where the CTAs lie
// decides how many of those share a multiprocessor.  Set up while the blocks of the table kernel still held theirs, they lay
// differently from call to call: 200 000 points, 125 taps 267 to 287 us; the table kernel allows it at its end now: 243.
__global__ void __launch_bounds__(THREADS, CTAS) mvmr_thin_kernel(const __grid_constant__ ThinParams p) {
    constexpr int CELLS = TPS / 2;   // taps of a lane
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t s_full[SLOTS], s_empty[SLOTS], s_acc_full[2], s_acc_empty[2];   // a step's operands are there / have been used; a block's sums
    __shared__ uint32_t s_tmem;
    __shared__ int s_abort;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, part = blockIdx.y;
    const uint32_t slot0 = (smem_u32(smem_raw) + 1023u) & ~1023u;
    volatile int *abort_flag = &s_abort;
    auto wait_one = [&](const uint64_t &bar, uint32_t parity) {
        return mbar_wait_abortable(smem_u32(&bar), parity & 1u, STATUS_BIT, p.status, abort_flag);
    };
    auto wait = [&](const uint64_t &bar, uint32_t parity) {   // the verdict is the same in the whole warp
        if (__all_sync(0xffffffffu, mbar_try_wait(smem_u32(&bar), parity & 1u))) return true;
        return __all_sync(0xffffffffu, wait_one(bar, parity)) != 0;
    };
    if (tid == 0) {
        // every lane's copies, every warp's zeros, the weights
        for (int s = 0; s < SLOTS; ++s) mbar_init(smem_u32(&s_full[s]), WARPS * 33 + 1), mbar_init(smem_u32(&s_empty[s]), 1);
        for (int s = 0; s < 2; ++s) mbar_init(smem_u32(&s_acc_full[s]), 1), mbar_init(smem_u32(&s_acc_empty[s]), 4);
        fence_mbar_init();
        s_abort = 0;
    }
    if (warp == MMA_WARP) tmem_alloc(smem_u32(&s_tmem), p.ncols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    start_after_previous();   // (tensor memory is held by now: see there)
    {
        uint32_t odd = 0;
        for (int x = tid; x < p.n_odd; x += THREADS) odd |= p.odd[x];
        if (__syncthreads_or(odd)) {
            one_by_one(p, reinterpret_cast<float *>(smem_raw), part);
            if (warp == MMA_WARP) tmem_dealloc(tmem, p.ncols);
            return;
        }
    }
    const int blocks = (p.nblocks - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;   // of this CTA
    auto block_of = [&](int n) { return (int64_t)blockIdx.x + (int64_t)n * gridDim.x; };
    auto most_of = [&](const At &at) { return at.n < blocks ? __ldg(p.most + block_of(at.n) * p.nq + at.q) : make_int2(0, 0); };
    Ring ring;

    if (warp < WARPS) {
        // ---------------------------------------------------------------- copies ----
        const int row = warp * 16 + (lane & 15), x0 = (lane >> 4) * CELLS;   // a lane has half of the taps of a row
        uint32_t at[CELLS];   // its cells' first pieces in a tile (which begins at a multiple of 1024)
#pragma unroll
        for (int x = 0; x < CELLS; ++x) at[x] = (uint32_t)row * 128 + (uint32_t)(((x0 + x) ^ (row & 7)) << 4);
        uint32_t last_load = 0;   // slot and turn of the last weights this thread sent for
        auto cells_of = [&](const At &at, int32_t (&e)[CELLS]) {
#pragma unroll
            for (int x = 0; x < CELLS; ++x) {
                const int k = at.q * TPS + x0 + x;
                e[x] = at.n < blocks && k < p.K ? __ldg(p.table + (block_of(at.n) * p.K + k) * ROWS + row) : NONE;
            }
        };
        At now, next;
        next.next(p.nq);
        int32_t e[CELLS], e_next[CELLS];
        cells_of(now, e);
        int2 most = most_of(now);
        bool ok = true;
        for (; now.n < blocks && ok; now = next, next.next(p.nq)) {
            cells_of(next, e_next);
            const int2 most_next = most_of(next);
            if (most.y) {
                const int4 r = clump_slot(p, s_full, s_empty, abort_flag, now, row, x0, part, slot0, make_int4(e[0], e[1], e[2], e[3]), most.x, ring, last_load);
                ring.slot = (uint32_t)r.x, ring.turn = (uint32_t)r.y, ok = r.z != 0, last_load = (uint32_t)r.w;
            } else {
                // this step's feature rows; of several triplets the second, and how many more
                int32_t j[CELLS], left[CELLS], t[CELLS];
#pragma unroll
                for (int x = 0; x < CELLS; ++x) {
                    const bool several = e[x] < NONE;
                    t[x] = (e[x] & (int32_t)MAX_T) + 1;
                    left[x] = several ? (int)((uint32_t)e[x] >> FIRST_BITS & 15u) + 1 : 0;
                    j[x] = load_if(several, p.gather - 1, t[x], e[x]);
                }
                for (int m = 0; m < most.x; ++m) {
                    int32_t j_next[CELLS];
#pragma unroll
                    for (int x = 0; x < CELLS; ++x) j_next[x] = load_if(left[x] > m, p.gather, t[x] + m, NONE);
                    ok = wait(s_empty[ring.slot], ring.turn ^ 1u);
                    if (!ok) break;
                    const uint32_t tile = slot0 + ring.slot * p.slot_bytes, full = smem_u32(&s_full[ring.slot]);
                    if (tid == 0) {
                        mbar_arrive_expect_tx(full, (uint32_t)p.N * 128u);
                        bulk_load(tile + A_BYTES, p.image + ((int64_t)(part * p.nq + now.q) * p.N) * 64, (uint32_t)p.N * 128u, full);
                        last_load = ring.slot | (ring.turn & 1u) << 8 | 1u << 16;
                    }
#pragma unroll
                    for (int x = 0; x < CELLS; ++x) {
                        copy_or_zeros(tile + at[x], p.feat, j[x]);
                        j[x] = j_next[x];
                    }
                    cp_async_mbar_arrive(full);   // fires once this lane's copies have landed
                    __syncwarp();
                    if (lane == 0) mbar_arrive(full);   // the warp's zeros
                    ring.next(SLOTS);
                }
            }
            most = most_next;
#pragma unroll
            for (int x = 0; x < CELLS; ++x) e[x] = e_next[x];
            if (ok && warp < 4 && now.q + 1 == p.nq) {
                // -------------------------------------------------------- epilogue ----
                const int a = now.n & 1;
                ok = wait(s_acc_full[a], (uint32_t)now.n >> 1);
                if (!ok) break;
                tc_fence_after();
                const int64_t i = block_of(now.n) * ROWS + tid;
                for (int c0 = 0; c0 < p.N; c0 += 16) {
                    float v[16];
                    tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)a * p.col_stride + (uint32_t)c0, v);
                    if (i < p.n_out && part * p.N + c0 < p.width) store16(p, i, part * p.N + c0, v);
                    __syncwarp();
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&s_acc_empty[a]));
            }
        }
        cp_async_wait<0>();
        // after a wait that ran out: weights that are still on their way land before the block ends
        if (*abort_flag && last_load) (void)mbar_wait(smem_u32(&s_full[last_load & 0xffu]), last_load >> 8 & 1u, STATUS_BIT, p.status, 1000000ull);
    } else if (elect_one()) {
        // ------------------------------------------------------------------- MMA ----
        const uint32_t idesc = instr_desc(p.fmt, ROWS, p.N, 0, 0);
        const uint64_t ad0 = smem_desc(slot0, 16, 1024), bd0 = smem_desc(slot0 + A_BYTES, 16, 1024);
        bool ok = true;
        At now, next;
        next.next(p.nq);
        int steps = most_of(now).x;
        for (; now.n < blocks && ok; now = next, next.next(p.nq)) {
            const int steps_next = most_of(next).x;
            if (now.q == 0 && !wait_one(s_acc_empty[now.n & 1], ((uint32_t)now.n >> 1) ^ 1u)) break;
            const uint32_t d = tmem + (uint32_t)(now.n & 1) * p.col_stride;
            for (int m = 0; m < steps; ++m) {
                ok = wait_one(s_full[ring.slot], ring.turn);
                if (!ok) break;
                fence_async_smem();   // the copies came through the generic proxy, the tensor core reads through the async proxy
                tc_fence_after();
                const uint64_t at = (uint64_t)(ring.slot * (p.slot_bytes >> 4));
#pragma unroll
                for (int k = 0; k < 4; ++k) tc_mma(d, ad0 + at + 2 * k, bd0 + at + 2 * k, idesc, now.q > 0 || m > 0 || k > 0 ? 1u : 0u);
                tc_commit(smem_u32(&s_empty[ring.slot]));
                ring.next(SLOTS);
            }
            if (ok && now.q + 1 == p.nq) tc_commit(smem_u32(&s_acc_full[now.n & 1]));
            steps = steps_next;
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (warp == MMA_WARP) tmem_dealloc(tmem, p.ncols);
}

struct ThinWs {
    uint32_t *odd, *n_sums;
    int32_t *table;
    int2 *most;
    uint16_t *image, *feat;
};

struct Shape {
    int inw, width, nq, parts, N;
    int64_t nblocks;
};

bool shape_of(int64_t n_out, int K, int C, int M, int transpose, Shape *s) {
    s->inw = transpose ? M : C, s->width = transpose ? C : M;
    if (n_out <= 0 || K <= 0 || K > MAX_TAPS || s->inw <= 0 || s->inw > CW || s->width <= 0 || s->width > MAX_WIDTH) return false;
    s->nq = (K + TPS - 1) / TPS;
    s->parts = (s->width + MAX_N - 1) / MAX_N;
    s->N = ((s->width + s->parts - 1) / s->parts + 15) / 16 * 16;
    s->nblocks = (n_out + ROWS - 1) / ROWS;
    return n_out <= INT32_MAX && s->nblocks * s->nq < INT32_MAX;
}

int prep_blocks() { return num_sms() * PREP_CTAS; }

size_t carve_thin(void *base, int64_t n_feat, int K, const Shape &s, int64_t sums, ThinWs *out) {
    Carver c(base);
    ThinWs w;
    w.odd = c.take<uint32_t>(prep_blocks() + 1), w.n_sums = w.odd + prep_blocks();
    w.table = c.take<int32_t>((size_t)s.nblocks * K * ROWS);
    w.most = c.take<int2>((size_t)s.nblocks * s.nq);
    w.image = c.take<uint16_t>((size_t)s.parts * s.nq * s.N * 64);
    w.feat = c.take<uint16_t>((size_t)(n_feat + PARTS * sums) * CW);
    if (out) *out = w;
    return c.off;
}

int launch_thin(const PrepParams &prep, ThinParams p, const Shape &s, cudaStream_t stream) {
    const int64_t work = std::max(std::max(prep.table_pieces / 8, prep.most_pieces), std::max(prep.image_pieces, prep.n_feat));
    p.n_odd = (int)std::min<int64_t>((work + PREP_THREADS - 1) / PREP_THREADS, prep_blocks());
    launch_after(thin_prepare_kernel, (unsigned)p.n_odd, PREP_THREADS, 0, stream, prep);
    PCX_LAUNCH_CHECK();
    launch_after(thin_table_kernel, (unsigned)((prep.T + 4 * PREP_THREADS - 1) / (4 * PREP_THREADS)), PREP_THREADS, 0, stream, prep);
    PCX_LAUNCH_CHECK();
    const size_t smem = std::max((size_t)1024 + SLOTS * p.slot_bytes, (size_t)ROWS * (p.N + 1) * 4);
    static std::atomic<uint64_t> allowed;
    if (int rc = allow_shared_memory((const void *)mvmr_thin_kernel, &allowed)) return rc;
    const dim3 grid((unsigned)std::min<int64_t>(s.nblocks, std::max(1, CTAS * num_sms() / s.parts)), (unsigned)s.parts);
    prof_begin("mvmr_thin_kernel", stream);
    launch_after(mvmr_thin_kernel, grid, THREADS, smem, stream, p);
    prof_end(stream);
    PCX_LAUNCH_CHECK();
    return PCX_OK;
}

}  // namespace
}  // namespace pcx

using namespace pcx;

extern "C" {

size_t pcx_mvmr_thin_workspace_bytes(int64_t n_feat, int64_t n_out, int K, int C, int M, int transpose) {
    Shape s;
    if (n_feat < 0 || n_feat > INT32_MAX || !shape_of(n_out, K, C, M, transpose, &s)) return 0;
    return carve_thin(nullptr, n_feat, K, s, n_out, nullptr);
}

int pcx_mvmr_thin(const void *d_weight, const void *d_feat, const int32_t *d_gather, const int32_t *d_scatter, const int64_t *d_seg_offs,
                  const void *d_bias, void *d_out, int64_t T, int64_t n_feat, int64_t n_out, int K, int C, int M, int flags, int dtype,
                  void *d_ws, size_t ws_bytes, void *stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    const int transpose = flags & PCX_MVMR_TRANSPOSE ? 1 : 0;
    if (dtype != PCX_F16 && dtype != PCX_BF16) PCX_FAIL(PCX_E_DTYPE, "pcx_mvmr_thin: fp16 or bf16 only (dtype %d)", dtype);
    Shape s;
    if (T <= 0 || T >= MAX_T || n_feat <= 0 || n_feat > INT32_MAX || !shape_of(n_out, K, C, M, transpose, &s))
        PCX_FAIL(PCX_E_UNSUPPORTED, "pcx_mvmr_thin: sizes out of range (T=%lld n_feat=%lld n_out=%lld K=%d C=%d M=%d)", (long long)T,
                 (long long)n_feat, (long long)n_out, K, C, M);
    if (!d_weight || !d_feat || !d_gather || !d_scatter || !d_seg_offs || !d_out || !d_ws) PCX_FAIL(PCX_E_ARG, "pcx_mvmr_thin: null pointer");
    if ((uintptr_t)d_ws % 256 || (uintptr_t)d_out % 16) PCX_FAIL(PCX_E_ALIGN, "pcx_mvmr_thin: workspace must be 256-byte, output 16-byte aligned");
    ThinWs w;
    const size_t need = carve_thin(nullptr, n_feat, K, s, 0, nullptr);
    if (ws_bytes < need) PCX_FAIL(PCX_E_CAPACITY, "pcx_mvmr_thin: workspace %zu < %zu bytes", ws_bytes, need);
    // as many sums as there can be, as there is room for, and as the rows' numbers reach
    const int64_t max_sums = std::min(std::min(T / (LISTED + 1), (int64_t)((ws_bytes - need) / SUM_BYTES)), ((int64_t)UINT32_MAX - 1 - n_feat) / PARTS);
    carve_thin(d_ws, n_feat, K, s, max_sums, &w);
    PrepParams prep = {};
    prep.weight = (const uint16_t *)d_weight, prep.feat_in = (const uint16_t *)d_feat, prep.feat = w.feat;
    prep.n_sums = w.n_sums, prep.max_sums = (uint32_t)max_sums;
    prep.scatter = d_scatter, prep.gather = d_gather, prep.seg = d_seg_offs, prep.table = w.table, prep.most = w.most, prep.image = w.image, prep.odd = w.odd;
    prep.T = T, prep.n_feat = n_feat, prep.image_pieces = (int64_t)s.parts * s.nq * s.N * 8;
    prep.table_pieces = s.nblocks * K * (ROWS / 4), prep.most_pieces = s.nblocks * s.nq;
    prep.K = K, prep.inw = s.inw, prep.width = s.width, prep.nq = s.nq, prep.N = s.N;
    prep.transpose = transpose, prep.reverse = flags & PCX_MVMR_REVERSE_TAPS ? 1 : 0, prep.fmt = dtype == PCX_BF16 ? 1 : 0;
    ThinParams p = {};
    p.feat = w.feat, p.first_sum = (uint32_t)n_feat;
    p.gather = d_gather, p.scatter = d_scatter, p.seg = d_seg_offs, p.table = w.table, p.most = w.most, p.image = w.image, p.odd = w.odd;
    p.bias = (const uint16_t *)d_bias, p.out = (uint16_t *)d_out;
    if (int rc = device_status_address(&p.status)) return rc;
    p.n_out = n_out, p.K = K, p.nq = s.nq, p.N = s.N, p.width = s.width, p.nblocks = (int)s.nblocks, p.fmt = prep.fmt;
    p.col_stride = s.N <= 32 ? 32u : 64u, p.ncols = 2 * p.col_stride;
    p.slot_bytes = A_BYTES + (uint32_t)align_up((size_t)s.N * 128, 1024);
    return launch_thin(prep, p, s, stream);
}

}  // extern "C"
