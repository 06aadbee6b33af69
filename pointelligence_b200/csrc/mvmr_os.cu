// Output-stationary MVMR on sm_100a: the fp32 sums of a block of 128 output rows stay in
// tensor memory (TMEM) across ALL taps and every output row is rounded and written exactly
// once -- no fp32 accumulator in global memory, no zero-fill, no rounding pass, no atomics,
// and a result that does not depend on the order in which CTAs run.
//
// The schedule needs the rulebook regrouped by output row.  That is done once per rulebook
// and direction by pcx_mvmr_plan_build into a caller-owned "plan":
//
//   rows     output rows are ordered by their tap signature (the set of taps that touch the
//            row) and, for a cubic kernel of at most 32 taps, first by the kernel planes that
//            set spans, so that the 128 rows of a block use few distinct taps and the
//            (block, tap) tiles below are well filled; perm[block * 128 + slot] = row
//   tiles    per (block, tap) a table of 128 source rows, one per slot: a feature row, "none",
//            or a row of the per-call scratch that holds the SUM of the feature rows of a
//            (row, tap) bucket with several triplets (the bucket pre-sum of the reference's fused
//            gather-sum schedule, sparse_engines/fused_point_conv.py:344-423); tile_offs is the
//            dense (nblocks * K + 1) table of triplet counts that tells which tiles exist
//   entries  per triplet (slot | position in its bucket << 8, feature row), ordered by
//            (block, tap, slot): the members of a bucket are consecutive
//   buckets  (first entry, length) of every bucket with more than one triplet
//   groups   two consecutive blocks share the weight slices they stream; most expensive first
//   masks    the taps that touch a block: what the walk goes through, so no task lists are built
//
// Per call: a small kernel sums the rows of the multi-triplet buckets into the scratch (fp32 sum,
// one rounding), then one persistent CTA per SM works off its steps (unit, 64-channel slice,
// tap; of rows of 16 or 32 channels four or two taps fill a step):
//
//   walk thread      decides the steps and fetches the source rows of their two tiles into shared memory
//                    eight steps early.  The tables come from DRAM: looked up one step ahead, every step
//                    waited out most of that latency and a tile took 1500 - 1800 clocks
//   copy teams       up to four teams fill the A tiles, a step each in turn: 16-byte cp.async copies of the
//                    tiles' source rows straight into the 128-byte-swizzled slot (rows without a source
//                    are zero-filled by the same instruction).  A copy loop alone
//                    moves a 16 KB tile of random rows in 230 - 290 clocks (a TMA row gather, measured: 2260)
//   weight warp      the 64-channel slice of W[tap] for both blocks, by TMA into the same slot
//   MMA threads      one per block: one wait per step, up to four tcgen05.mma (M = 128, N = out_width)
//                    and one commit
//   epilogue warps   read TMEM (tcgen05.ld), add the bias, round once and write each output row; up to 128
//                    channels the accumulators are double-buffered, so the next group is built meanwhile
//
// What bounds a step (two tiles) is neither memory (the same time with every row in L2) nor the tensor core but
// the instruction chains of the roles, some 1000 clocks each: hence single threads without votes, more teams of
// fewer warps, and several taps a step where rows are narrow.  Forward, 300k points with 22 triplets a row:
// 32 -> 32 channels 64 us (84 with one tap a step), 64 -> 64 93 us, 128 -> 128 185 us; 80k points, kernel 5,
// 16 -> 32: 89 us (209).
//
// Units are groups; where those do not fill the chip (small clouds, deep levels) their taps are split
// over several CTAs, which leave fp32 sums that a last kernel adds in a fixed order.
//
// Every wait is bounded (one second) and abortable: a role that gives up raises a flag in the
// status word and in shared memory, the other roles leave their waits, and the CTA frees its
// TMEM and returns.
#include <cub/cub.cuh>
#include <cuda.h>

#include "sparse_kernels.cuh"
#include "tcgen05.cuh"

namespace pcx {
int device_status_address(unsigned int **d_status);

namespace {

using namespace tc;

constexpr int ROWS = 128;             // output rows per block (the M of the MMA)
constexpr int SLOT_BYTES = ROWS * 128;  // one A tile: 128 rows of a 64-channel slice
constexpr int GROUP_BLOCKS = 2;         // blocks of a group
constexpr int MAX_TAPS = 512;           // taps of a plan
constexpr unsigned STATUS_BIT = 4u;   // bit of the device status word this kernel raises
constexpr unsigned PLAN_MAGIC = 0x70637832u;

// control words at the head of a plan
enum { CTRL_MAGIC = 2, CTRL_GROUP = 3, CTRL_NMULTI = PCX_PLAN_MULTI_WORD, CTRL_UNSORTED = CTRL_NMULTI + 1, CTRL_WORDS = 64 };

struct PlanView {
    uint32_t *ctrl;        // CTRL_WORDS
    int32_t *perm;         // nblocks * ROWS, -1 = padding
    int32_t *tile_offs;    // nblocks * K + 1
    uint2 *entries;        // T
    int32_t *group_order;  // ngroups
    int32_t *tile_rows;    // nblocks * K * ROWS: source row of (tile, slot): >= 0 feature row, -1 none, <= -2 scratch row -2 - x
    uint2 *buckets;        // T / 2 + 1: (first entry, length) of the buckets with several triplets
    uint32_t *tap_masks;   // nblocks * ceil(K / 32): the taps that touch a block
    int64_t nblocks, ngroups;
};

size_t carve_plan(void *base, int64_t T, int64_t n_out, int K, int G, PlanView *out) {
    Carver c(base);
    PlanView v;
    v.nblocks = (n_out + ROWS - 1) / ROWS;
    v.ngroups = (v.nblocks + G - 1) / G;
    v.ctrl = c.take<uint32_t>(CTRL_WORDS);
    v.perm = c.take<int32_t>((size_t)v.nblocks * ROWS);
    v.tile_offs = c.take<int32_t>((size_t)v.nblocks * K + 1);
    v.entries = c.take<uint2>((size_t)std::max<int64_t>(T, 1));
    v.group_order = c.take<int32_t>((size_t)std::max<int64_t>(v.ngroups, 1));
    v.tile_rows = c.take<int32_t>((size_t)v.nblocks * K * ROWS);
    v.buckets = c.take<uint2>((size_t)(T / 2 + 1));
    v.tap_masks = c.take<uint32_t>((size_t)v.nblocks * ((K + 31) / 32));
    if (out) *out = v;
    return c.off;
}

int bits_of(int64_t n) {
    int bits = 1;
    while (((int64_t)1 << bits) < n) ++bits;
    return bits;
}

struct BuildWs {
    uint32_t *sig;                       // n_out
    uint64_t *order, *order_sorted;      // n_out
    int32_t *row, *row_sorted, *rank;    // n_out
    uint32_t *key, *key_sorted;          // T
    int32_t *val, *val_sorted;           // T
    int32_t *tile_cnt;                   // nblocks * K + 1
    uint32_t *cost, *cost_sorted;        // ngroups
    int32_t *gid;                        // ngroups
    void *cub_tmp;
    size_t cub_bytes;
};

size_t carve_build(void *base, int64_t T, int64_t n_out, int K, int G, BuildWs *out) {
    Carver c(base);
    BuildWs w;
    const int64_t nblocks = (n_out + ROWS - 1) / ROWS, ngroups = (nblocks + G - 1) / G;
    const size_t n = (size_t)std::max<int64_t>(n_out, 1), t = (size_t)std::max<int64_t>(T, 1);
    const size_t g = (size_t)std::max<int64_t>(ngroups, 1);
    w.sig = c.take<uint32_t>(n);
    w.order = c.take<uint64_t>(n), w.order_sorted = c.take<uint64_t>(n);
    w.row = c.take<int32_t>(n), w.row_sorted = c.take<int32_t>(n), w.rank = c.take<int32_t>(n);
    w.key = c.take<uint32_t>(t), w.key_sorted = c.take<uint32_t>(t);
    w.val = c.take<int32_t>(t), w.val_sorted = c.take<int32_t>(t);
    w.tile_cnt = c.take<int32_t>((size_t)nblocks * K + 1);
    w.cost = c.take<uint32_t>(g), w.cost_sorted = c.take<uint32_t>(g);
    w.gid = c.take<int32_t>(g);
    size_t b1 = 0, b2 = 0, b3 = 0, b4 = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, b1, (const uint64_t *)nullptr, (uint64_t *)nullptr, (const int32_t *)nullptr,
                                    (int32_t *)nullptr, (int)n, 0, 64);
    cub::DeviceRadixSort::SortPairs(nullptr, b2, (const uint32_t *)nullptr, (uint32_t *)nullptr, (const int32_t *)nullptr,
                                    (int32_t *)nullptr, (int)t, 0, 32);
    cub::DeviceScan::ExclusiveSum(nullptr, b3, (const int32_t *)nullptr, (int32_t *)nullptr, (int)((size_t)nblocks * K + 1));
    cub::DeviceRadixSort::SortPairsDescending(nullptr, b4, (const uint32_t *)nullptr, (uint32_t *)nullptr,
                                              (const int32_t *)nullptr, (int32_t *)nullptr, (int)g, 0, 32);
    w.cub_bytes = std::max(std::max(b1, b2), std::max(b3, b4));
    w.cub_tmp = c.take<char>(w.cub_bytes);
    if (out) *out = w;
    return c.off;
}

__device__ __forceinline__ uint32_t pack2(float a, float b, int fmt) {
    if (fmt) {
        __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
        return *reinterpret_cast<uint32_t *>(&v);
    }
    __half2 v = __floats2half2_rn(a, b);
    return *reinterpret_cast<uint32_t *>(&v);
}

// Tap of triplet t: last k with seg[k] <= t; `seg` is the CTA's copy of the segment offsets.
__device__ __forceinline__ int tap_of(const int64_t *seg, int K, int64_t t) {
    int lo = 0, hi = K;
    while (hi - lo > 1) {
        int mid = (lo + hi) >> 1;
        if (seg[mid] <= t) lo = mid; else hi = mid;
    }
    return lo;
}
__device__ __forceinline__ void copy_seg(const int64_t *__restrict__ seg, int K, int64_t *s_seg) {
    for (int k = threadIdx.x; k <= K; k += blockDim.x) s_seg[k] = seg[k];
    __syncthreads();
}

__global__ void plan_init_kernel(int64_t n_out, uint32_t *sig, int32_t *row, int32_t *tile_cnt, int64_t n_tiles,
                                 uint32_t *ctrl, int G, int4 *tile_rows) {
    start_after_previous();
    const int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, threads = (int64_t)gridDim.x * blockDim.x;
    for (int64_t t = x; t < n_tiles * (ROWS / 4); t += threads) tile_rows[t] = make_int4(-1, -1, -1, -1);   // no source anywhere
    if (x < n_out) sig[x] = 0u, row[x] = (int32_t)x;
    if (x <= n_tiles) tile_cnt[x] = 0;
    if (x < CTRL_WORDS) ctrl[x] = x == CTRL_MAGIC ? PLAN_MAGIC : x == CTRL_GROUP ? (uint32_t)G : 0u;
}

// Tap signature of every output row.  With more than 32 taps the taps are folded onto 32
// bits (tap mod 32): rows that share a signature then share a superset of taps.  Notes rulebooks
// whose rows do not ascend inside a tap.
__global__ void plan_sig_kernel(const int32_t *__restrict__ scatter, const int64_t *__restrict__ seg, int64_t T, int K,
                                uint32_t *sig, uint32_t *ctrl) {
    start_after_previous();
    __shared__ int64_t s_seg[MAX_TAPS + 1];
    copy_seg(seg, K, s_seg);
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= T) return;
    const int k = tap_of(s_seg, K, t);
    const int32_t r = scatter[t];
    if (t > s_seg[k]) {
        const int32_t before = scatter[t - 1];
        if (before == r) return;   // the first triplet of the bucket says it
        if (before > r) ctrl[CTRL_UNSORTED] = 1u;
    }
    atomicOr(&sig[r], 1u << (k & 31));
}

// Sort key of the rows: the signature and, above it for a cubic kernel (K = ks^3 <= 32 taps, tap =
// (kx * ks + ky) * ks + kz), which kx / ky / kz planes of the kernel a row uses at all, kz most
// significant.  Points of a scene lie on surfaces; rows of one surface orientation share these planes
// even where their exact tap sets differ, and sorted by (planes, signature) the blocks of 128 rows need
// a quarter fewer (block, tap) tiles on thin rulebooks than sorted by signature alone.
__global__ void plan_order_kernel(const uint32_t *__restrict__ sig, int64_t n_out, int K, int ks, uint64_t *order) {
    start_after_previous();
    const int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= n_out) return;
    const uint32_t m = sig[x];
    uint32_t px = 0, py = 0, pz = 0;
    if (ks)
        for (int tap = 0; tap < K; ++tap)
            if ((m >> tap) & 1u) px |= 1u << (tap / (ks * ks)), py |= 1u << ((tap / ks) % ks), pz |= 1u << (tap % ks);
    order[x] = (uint64_t)m | (uint64_t)(px | (py << ks) | (pz << (2 * ks))) << (K < 32 ? K : 32);
}

__global__ void plan_rank_kernel(const int32_t *__restrict__ row_sorted, int64_t n_out, int64_t n_pad, int32_t *rank,
                                 int32_t *perm) {
    start_after_previous();
    const int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= n_pad) return;
    if (x < n_out) {
        const int32_t r = row_sorted[x];
        rank[r] = (int32_t)x;
        perm[x] = r;
    } else {
        perm[x] = -1;
    }
}

// ---- rulebooks whose rows ascend inside a tap (what the geometry stage emits): a (row, tap) bucket is a run of
// consecutive triplets, so everything is placed by counting and no triplet is sorted.  Of any other rulebook these two kernels
// touch nothing: placed in vain and cleared again, the strided rulebooks of a training step on 1.04 M points, taken backwards, cost 1.1 ms.

// tile_rows[tile * 128 + slot] = first triplet of the bucket; triplets per tile
__global__ void plan_heads_kernel(const int32_t *__restrict__ scatter, const int64_t *__restrict__ seg, const int32_t *__restrict__ rank,
                                  int64_t T, int K, const uint32_t *__restrict__ ctrl, int32_t *tile_rows, int32_t *tile_cnt) {
    start_after_previous();
    if (ctrl[CTRL_UNSORTED]) return;
    __shared__ int64_t s_seg[MAX_TAPS + 1];
    copy_seg(seg, K, s_seg);
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= T) return;
    const int k = tap_of(s_seg, K, t);
    const int32_t row = scatter[t];
    if (t > s_seg[k] && scatter[t - 1] == row) return;
    int len = 1;
    while (t + len < s_seg[k + 1] && scatter[t + len] == row) ++len;
    const uint32_t r = (uint32_t)rank[row], tile = (r >> 7) * (uint32_t)K + (uint32_t)k;
    tile_rows[((int64_t)tile << 7) | (r & 127u)] = (int32_t)t;
    atomicAdd(&tile_cnt[tile], len);
}

// One warp per (block, tap) tile: entries in slot order, the tile's source rows, its multi-triplet buckets, numbered as the tiles come.
// (Numbered by bins of output rows where the rows of a cloud lie together in memory, bucket_sum_kernel alone gains, 1 M x 96 215 -> 173
// us, but mvmr_os_kernel finds the sums of a tile further apart, and buckets of many triplets follow each other.  A pass then took 0 to 13 %
// more at 32 and 64 channels of a million rows, 2 to 35 % more at 64 of 100 000 to 600 000, sweeps and clumped clouds the most, and 0 to 10 %
// less at 96 and 128 of a million; a training step of 1.04 M points 0.4 % less.  The plan does not know the channels.)
__global__ void plan_tiles_kernel(const int32_t *__restrict__ scatter, const int32_t *__restrict__ gather, const int64_t *__restrict__ seg,
                                  int K, int64_t n_tiles, const int32_t *__restrict__ tile_offs, uint2 *entries, int32_t *tile_rows,
                                  uint2 *buckets, uint32_t *ctrl) {
    start_after_previous();
    const int64_t tile = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (tile >= n_tiles) return;
    const int32_t first = tile_offs[tile];
    if (tile_offs[tile + 1] == first) return;   // no triplets, or none placed here: its rows say "none" already
    const int64_t end = seg[tile % K + 1];
    int4 *slots = reinterpret_cast<int4 *>(tile_rows + (tile << 7)) + lane;
    const int4 h = *slots;
    const int32_t head[4] = {h.x, h.y, h.z, h.w};
    int len[4], sum = 0, multi = 0;
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        len[s] = 0;
        if (head[s] >= 0) {
            const int32_t row = scatter[head[s]];
            len[s] = 1;
            while (head[s] + len[s] < end && scatter[head[s] + len[s]] == row) ++len[s];
        }
        sum += len[s], multi += len[s] > 1;
    }
    int at = sum, nth = multi;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int a = __shfl_up_sync(0xffffffffu, at, o), b = __shfl_up_sync(0xffffffffu, nth, o);
        if (lane >= o) at += a, nth += b;
    }
    const int total = __shfl_sync(0xffffffffu, nth, 31);
    uint32_t base = 0;
    if (lane == 0 && total) base = atomicAdd(&ctrl[CTRL_NMULTI], (uint32_t)total);
    base = __shfl_sync(0xffffffffu, base, 0) + (uint32_t)(nth - multi);
    uint32_t entry = (uint32_t)(first + at - sum);
    int32_t source[4];
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        source[s] = -1;
        for (int m = 0; m < len[s]; ++m) {
            const int32_t j = gather[head[s] + m];
            entries[entry + m] = make_uint2((uint32_t)(lane * 4 + s) | ((uint32_t)min(m, 0xffffff) << 8), (uint32_t)j);
            if (len[s] == 1) source[s] = j;
        }
        if (len[s] > 1) {
            buckets[base] = make_uint2(entry, (uint32_t)len[s]);
            source[s] = -2 - (int32_t)base++;
        }
        entry += (uint32_t)len[s];
    }
    *slots = make_int4(source[0], source[1], source[2], source[3]);
}

// ---- any other tap-sorted rulebook: the triplets are sorted by (block, tap, slot)
__global__ void plan_keys_kernel(const int32_t *__restrict__ scatter, const int32_t *__restrict__ gather,
                                 const int64_t *__restrict__ seg, const int32_t *__restrict__ rank, int64_t T, int K,
                                 uint32_t *key, int32_t *val, int32_t *tile_cnt) {
    start_after_previous();
    __shared__ int64_t s_seg[MAX_TAPS + 1];
    copy_seg(seg, K, s_seg);
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= T) return;
    const int k = tap_of(s_seg, K, t);
    const uint32_t r = (uint32_t)rank[scatter[t]];
    const uint32_t tile = (r >> 7) * (uint32_t)K + (uint32_t)k;
    key[t] = (tile << 7) | (r & 127u);
    val[t] = gather[t];
    atomicAdd(&tile_cnt[tile], 1);
}

// entries[t] = (slot | position within the (row, tap) bucket << 8, feature row); the first entry
// of a bucket also fills the bucket's slot of its tile's row table: the feature row itself, or,
// when more triplets follow, the scratch row the bucket's sum will be written to
__global__ void plan_entries_kernel(const uint32_t *__restrict__ key_sorted, const int32_t *__restrict__ val_sorted,
                                    int64_t T, uint2 *entries, int32_t *tile_rows, uint2 *buckets, uint32_t *ctrl) {
    start_after_previous();
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= T) return;
    const uint32_t k = key_sorted[t];
    uint32_t pos = 0;
    while (pos < 0xffffffu && t - (int64_t)pos - 1 >= 0 && key_sorted[t - pos - 1] == k) ++pos;
    entries[t] = make_uint2((k & 127u) | (pos << 8), (uint32_t)val_sorted[t]);
    if (pos != 0) return;
    uint32_t len = 1;
    while (t + len < T && key_sorted[t + len] == k) ++len;
    if (len == 1) {
        tile_rows[k] = val_sorted[t];   // key = tile * 128 + slot
    } else {
        const uint32_t b = atomicAdd(&ctrl[CTRL_NMULTI], 1u);
        buckets[b] = make_uint2((uint32_t)t, len);
        tile_rows[k] = -2 - (int32_t)b;
    }
}

// scratch[b] = sum of the feature rows of bucket b (fp32 sum in entry order, one rounding); a thread per 16-byte piece.
// Widening and adding is one instruction a value (add.f32 takes a 16-bit operand); a sum starts from its first member.
template <int FMT>
__device__ __forceinline__ void widen(uint4 p, float *s) {
    const uint32_t w[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const float2 f = FMT ? __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&w[q])) : __half22float2(*reinterpret_cast<const __half2 *>(&w[q]));
        s[2 * q] = f.x, s[2 * q + 1] = f.y;
    }
}
template <int FMT>
__device__ __forceinline__ void add(uint4 p, float *s) {
    const uint32_t w[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        float &a = s[2 * q], &b = s[2 * q + 1];
        if (FMT) asm("{.reg .b16 l, h;\n\tmov.b32 {l, h}, %2;\n\tadd.rn.f32.bf16 %0, l, %0;\n\tadd.rn.f32.bf16 %1, h, %1;}" : "+f"(a), "+f"(b) : "r"(w[q]));
        else asm("{.reg .b16 l, h;\n\tmov.b32 {l, h}, %2;\n\tadd.rn.f32.f16 %0, l, %0;\n\tadd.rn.f32.f16 %1, h, %1;}" : "+f"(a), "+f"(b) : "r"(w[q]));
    }
}

// whether one of a word's two numbers is infinite or no number
template <int FMT>
__device__ __forceinline__ bool not_finite(uint32_t w) {
    constexpr uint32_t EXP = FMT ? 0x7f80u : 0x7c00u;   // all ones
    return (w & EXP) == EXP || (w & EXP << 16) == EXP << 16;
}

// a + 0 w, two numbers each: stays what it is while the numbers of w are finite, then no number
template <int FMT>
__device__ __forceinline__ uint32_t times_zero(uint32_t w, uint32_t a) {
    uint32_t r;
    if (FMT) asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(w), "r"(0u), "r"(a));
    else asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(w), "r"(0u), "r"(a));
    return r;
}

constexpr int BUCKET_SUM_THREADS = 256, BUCKET_SUM_WARPS = BUCKET_SUM_THREADS / 32, BUCKET_SUM_CTAS = 4;

// LANES: threads of a bucket.  A warp fetches the descriptors and the first four rows of up to 32 consecutive buckets at
// once, a lane each, then sums them 32 / LANES at a time.
//
// Bound by the latency of the gathers.  With a bucket per LANES threads of a grid that covers them all, each waited for
// its descriptor, its rows' indices and its rows in turn and took 144 instructions (72 now).  The warps of the whole chip
// walk through the buckets together (round after round, not a range each): what they gather at one time lies in few blocks
// of the plan, 250 against 297 us.  Rounds are of equal size: a last one of few buckets left 13 % of the chip idle.
// 200k points, 22 triplets a row: 32 channels 50 -> 44 us, 64 88 -> 70, 96 141 -> 106, 128 160 -> 113, 192 245 -> 197,
// 256 305 -> 250, 512 647 -> 517.  Slower: 5 and 6 CTAs an SM (spills), the next bucket's rows fetched early at 3 CTAs
// (368), several pieces a thread (550 - 1090).
//
// SPLIT: what rounding a sum to `hi` left over goes behind it.  With `odd` given, sums that are not finite, and weights that
// are not (16-byte pieces of them, looked at in passing), are reported in odd[block] and the caller does all of it again;
// without, zero goes behind such sums (infinity less infinity is no number).
template <int FMT, int LANES, bool SPLIT>
__global__ void __launch_bounds__(BUCKET_SUM_THREADS, BUCKET_SUM_CTAS) bucket_sum_kernel(const uint16_t *__restrict__ feat,
                                                                                         const uint2 *__restrict__ entries,
                                                                                         const uint2 *__restrict__ buckets,
                                                                                         const uint32_t *__restrict__ ctrl, int inw,
                                                                                         int most, uint16_t *__restrict__ scratch,
                                                                                         const uint4 *__restrict__ weight,
                                                                                         int64_t weight_pieces, uint32_t *odd) {
    start_after_previous();
    bool seen = false;   // something that is not finite
    uint32_t rest = 0;   // two zeros until what a rounding left over is not finite
    if (SPLIT && odd) {
        const int64_t threads = (int64_t)gridDim.x * gridDim.y * BUCKET_SUM_THREADS;
        const int64_t first = ((int64_t)blockIdx.y * gridDim.x + blockIdx.x) * BUCKET_SUM_THREADS + threadIdx.x;
        for (int64_t t = first; t < weight_pieces; t += threads) {
            const uint4 v = __ldg(weight + t);
            seen |= not_finite<FMT>(v.x) || not_finite<FMT>(v.y) || not_finite<FMT>(v.z) || not_finite<FMT>(v.w);
        }
    }
    constexpr int AT_ONCE = 32 / LANES;
    const int lane = threadIdx.x & 31, sub = lane / LANES, nmulti = min((int)ctrl[CTRL_NMULTI], most);   // never beyond the scratch
    const unsigned piece = blockIdx.y * LANES + lane % LANES, pitch = (unsigned)inw * 2u;
    const bool piece_ok = piece * 16 < pitch;   // a lane without a piece takes part in the shuffles
    const char *col = reinterpret_cast<const char *>(feat) + (piece_ok ? piece * 16 : 0);
    char *dst = reinterpret_cast<char *>(scratch) + piece * 16;
    const int warps = (int)gridDim.x * BUCKET_SUM_WARPS, rounds = max((nmulti + 32 * warps - 1) / (32 * warps), 1);
    const int batch = ((nmulti + warps * rounds - 1) / (warps * rounds) + AT_ONCE - 1) / AT_ONCE * AT_ONCE;   // at most 32
    for (int b0 = ((int)blockIdx.x * BUCKET_SUM_WARPS + (int)(threadIdx.x >> 5)) * batch; b0 < nmulti; b0 += warps * batch) {
        const int n = min(batch, nmulti - b0);
        const uint2 bk = lane < n ? __ldg(buckets + b0 + lane) : make_uint2(0u, 0u);
        uint32_t row[4];
#pragma unroll
        for (int m = 0; m < 4; ++m) row[m] = m < (int)bk.y ? __ldg(&entries[bk.x + m].y) : 0u;
#pragma unroll 1
        for (int i = 0; i < n; i += AT_ONCE) {
            const int src = i + sub;   // (below 32: n is at most the batch, a multiple of AT_ONCE)
            auto piece_of = [&](uint32_t r) { return __ldg(reinterpret_cast<const uint4 *>(col + (uint64_t)r * pitch)); };
            auto member = [&](int m) { return piece_of(__shfl_sync(0xffffffffu, row[m], src)); };   // an absent one reads row 0
            const uint32_t len = __shfl_sync(0xffffffffu, bk.y, src);   // 0 behind the end
            const bool three = __any_sync(0xffffffffu, len > 2), four = __any_sync(0xffffffffu, len > 3);
            const uint4 v0 = member(0), v1 = member(1);
            uint4 v2, v3;
            if (three) v2 = member(2);
            if (four) v3 = member(3);
            float s[8];
            widen<FMT>(v0, s);
            add<FMT>(v1, s);
            if (len > 2) add<FMT>(v2, s);
            if (len > 3) add<FMT>(v3, s);
            if (four) {
                const uint32_t first = __shfl_sync(0xffffffffu, bk.x, src);
                for (uint32_t m = 4; m < len; ++m) add<FMT>(piece_of(__ldg(&entries[first + m].y)), s);
            }
            uint4 o;
            o.x = pack2(s[0], s[1], FMT), o.y = pack2(s[2], s[3], FMT);
            o.z = pack2(s[4], s[5], FMT), o.w = pack2(s[6], s[7], FMT);
            // past the L2's share of the feature rows: the sums are read once, by the next kernel
            const bool store = piece_ok && len;
            uint4 *at = reinterpret_cast<uint4 *>(dst + (uint64_t)(uint32_t)(b0 + src) * (SPLIT ? 2 * pitch : pitch));
            if (store) __stcs(at, o);
            if (SPLIT) {   // ... and behind it what the rounding left over
                float hi[8];
                widen<FMT>(o, hi);
#pragma unroll
                for (int e = 0; e < 8; ++e) s[e] -= hi[e];   // no number or infinite where hi is not finite
                if (!odd) {
#pragma unroll
                    for (int e = 0; e < 8; ++e) s[e] = fabsf(s[e]) < INFINITY ? s[e] : 0.f;
                }
                o.x = pack2(s[0], s[1], FMT), o.y = pack2(s[2], s[3], FMT);
                o.z = pack2(s[4], s[5], FMT), o.w = pack2(s[6], s[7], FMT);
                if (store) {
                    __stcs(reinterpret_cast<uint4 *>(reinterpret_cast<char *>(at) + pitch), o);
                    rest = times_zero<FMT>(o.x, times_zero<FMT>(o.y, times_zero<FMT>(o.z, times_zero<FMT>(o.w, rest))));
                }
            }
        }
    }
    if (SPLIT && odd) {
        const int any = __syncthreads_or(seen || (rest & 0x7fff7fffu));
        if (threadIdx.x == 0) odd[blockIdx.y * gridDim.x + blockIdx.x] = (uint32_t)any;
    }
}

template <int FMT, bool SPLIT>
int launch_bucket_sum(int64_t multi, int inw, const uint16_t *feat, const uint2 *entries, const uint2 *buckets,
                       const uint32_t *ctrl, uint16_t *scratch, const uint4 *weight, int64_t weight_pieces, uint32_t *odd, cudaStream_t stream) {
    // Up to 128 channels the next power of two of lanes, beyond that slices (blockIdx.y) of 32, 16 or 8 lanes, whichever
    // idles least, the widest of equals (200k points, 22 triplets a row): 256 channels 258 us in slices of 32 (266 of 16, 300 of 8),
    // 512 561 (577, 707), 208 247 (274, 292), 192 214 of 8 (222 of 32, 241 of 16), 384 417 of 16 (472 of 32, 511 of 8).
    // Below: 48 channels 63 us in 8 lanes (80 in slices of 2).
    const int ppr = inw >> 3;
    int lanes = 2;
    while (lanes < ppr && lanes < 16) lanes <<= 1;
    if (ppr > 16) {
        lanes = 32;
        for (const int l : {16, 8})
            if ((ppr + l - 1) / l * l < (ppr + lanes - 1) / lanes * lanes) lanes = l;
    }
    const int slices = (ppr + lanes - 1) / lanes, at_once = BUCKET_SUM_THREADS / lanes;
    const int64_t work = std::max((multi + at_once - 1) / at_once, odd ? (weight_pieces + BUCKET_SUM_THREADS - 1) / BUCKET_SUM_THREADS : 0);
    const dim3 grid((unsigned)std::max<int64_t>(1, std::min<int64_t>(work, std::min(num_sms() * BUCKET_SUM_CTAS, MAX_ODD) / slices)), (unsigned)slices);
#define PCX_BS(L) launch_after(bucket_sum_kernel<FMT, L, SPLIT>, grid, BUCKET_SUM_THREADS, 0, stream, feat, entries, buckets, ctrl, inw, (int)multi, scratch, weight, weight_pieces, odd)
    switch (lanes) {
        case 2: PCX_BS(2); break;
        case 4: PCX_BS(4); break;
        case 8: PCX_BS(8); break;
        case 16: PCX_BS(16); break;
        default: PCX_BS(32); break;
    }
#undef PCX_BS
    return (int)(grid.x * grid.y);
}

// cost of a group = its non-empty tiles (each is one A tile to copy and multiply); the tap sets of its blocks
__global__ void plan_cost_kernel(const int32_t *__restrict__ tile_offs, int64_t nblocks, int K, int G, int64_t ngroups,
                                 uint32_t *cost, int32_t *gid, uint32_t *tap_masks) {
    start_after_previous();
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= ngroups) return;
    const int words = (K + 31) / 32;
    uint32_t c = 0;
    for (int64_t b = g * G; b < min((g + 1) * (int64_t)G, nblocks); ++b)
        for (int w = 0; w < words; ++w) {
            uint32_t m = 0;
            for (int k = 32 * w; k < min(K, 32 * w + 32); ++k)
                if (tile_offs[b * K + k + 1] > tile_offs[b * K + k]) m |= 1u << (k & 31);
            tap_masks[b * words + w] = m;
            c += (uint32_t)__popc(m);
        }
    cost[g] = c;
    gid[g] = (int32_t)g;
}

// ------------------------------------------------------------------ kernel ----
constexpr int EPI_WARPS = 4, TEAMS = 4, TEAM_WARPS = 4, COPY_WARPS = TEAMS * TEAM_WARPS;
constexpr int COPY_WARP0 = EPI_WARPS, WALK_WARP = COPY_WARP0 + COPY_WARPS, WEIGHT_WARP = WALK_WARP + 1, MMA_WARP0 = WEIGHT_WARP + 1;
constexpr int THREADS = (MMA_WARP0 + GROUP_BLOCKS) * 32;
constexpr int MAX_SLOTS = 8;
// Output channels whose bias is kept in shared memory (wider rows read it from global memory: behind the copies in the
// SM's memory pipeline every 16 columns waited for it, and 200k points of 256 channels took 383 us instead of 338).
constexpr int BIAS_WIDTH = 1024;
constexpr int AHEAD = 8;                              // steps the walk runs ahead
constexpr uint32_t ENTRY_BYTES = 2 * ROWS * 4;        // source rows of a tap's two tiles
// a step's word: per tap of the step, which of the two tiles have it | contraction steps of 16 << 8 | low parts of split
// sums << 11 | tiles that have
// any << 13 | first of its unit << 15 | end << 16
constexpr uint32_t STEP_LOW = 1u << 11, STEP_FIRST = 1u << 15, STEP_END = 1u << 16;
// The MMA threads read the words from a ring of their own, each marked with the turn of the ring it belongs to.
// The walk is at most AHEAD steps ahead of the copies and these at most MAX_SLOTS ahead of the MMAs, so with
// WORDS entries no word is overwritten before it has been read.
constexpr int WORDS = 32;
static_assert(WORDS >= AHEAD + MAX_SLOTS + TEAMS, "the word ring must hold every step between the walk and the MMAs");
constexpr uint32_t TURN_SHIFT = 17;   // turn (from 1 on) in the upper 15 bits

struct OsParams {
    const uint16_t *feat, *bias;            // rows of in_pitch elements; bias: added before the rounding; null: none
    const uint16_t *scratch;                // sums of the multi-triplet buckets
    uint16_t *out;
    float *partial;                         // nsplit > 1: [split][nblocks][row of out_pitch / 4][ROWS] float4
    const int32_t *perm, *group_order, *tile_rows;
    const uint32_t *tap_masks;
    unsigned int *status;
    int K, C, M, transpose, reverse, fmt;   // reverse: tap k uses weight K-1-k
    int inw, outw, nkb, ngroups, nblocks, nsplit, mask_words;   // inw, outw: of a part; nkb: slices of the contraction
    int nparts, out_parts, in_pitch, out_pitch;   // parts of an output row: groups of the weight, each in out_parts
    int nslots, nacc, teams;
    const uint16_t *weight;                 // read without the tensor map: transposed weights of a step of several taps
    uint32_t slot_bytes, w_box_rows, w_rows, w_tx_bytes, ncols, col_stride;   // w_rows: of the weight slice of all taps of a step
    uint64_t wait_limit_ns;
};

__device__ __forceinline__ float bias_at(const uint16_t *b, int c, int fmt) {
    const uint16_t v = __ldg(b + c);
    return fmt ? __bfloat162float(__ushort_as_bfloat16(v)) : __half2float(__ushort_as_half(v));
}

// Position `n` of a CTA in the list of units (groups, most expensive first, times their parts): rows of
// the list run to and fro over the CTAs, so that the sums of their costs stay close without a shared
// work counter.  -1 behind the end.
__device__ __forceinline__ int unit_at(int n, int units) {
    const int pos = n * (int)gridDim.x + ((n & 1) ? (int)gridDim.x - 1 - (int)blockIdx.x : (int)blockIdx.x);
    return pos < units ? pos : -1;
}

// The steps of a CTA: unit (group, split, part of the output row) after unit, in a unit the 64-channel slices of the contraction, per slice the
// taps that touch one of the group's two blocks.
struct Walk {
    const OsParams &p;
    int n = -1, split = 0, part = 0, block0 = 0, q = 0, word = 0, tap = 0;
    int slices;                     // of the contraction; those of the low parts follow those of the high ones
    int tap_lo = 0, tap_hi = 0;     // taps of this part of the group
    uint32_t m0 = 0, m1 = 0, left = 0;
    uint32_t has = 0;               // of the current step: bit b = block b of the group has the tap
    bool opened = false;            // no step of the unit yet
    bool first = false;             // the current step is the first of its unit
    __device__ __forceinline__ Walk(const OsParams &params, bool split_sums) : p(params), slices(split_sums ? 2 * params.nkb : params.nkb) { q = slices; }

    __device__ __forceinline__ static uint32_t below(int w, int tap) {   // bits of mask word w that belong to taps < tap
        const int n = min(max(tap - 32 * w, 0), 32);
        return n >= 32 ? 0xffffffffu : (1u << n) - 1u;
    }
    __device__ __forceinline__ void load(int w) {
        const uint32_t r = below(w, tap_hi) & ~below(w, tap_lo);
        m0 = __ldg(p.tap_masks + (int64_t)block0 * p.mask_words + w) & r;
        m1 = block0 + 1 < p.nblocks ? __ldg(p.tap_masks + (int64_t)(block0 + 1) * p.mask_words + w) & r : 0u;
        left = m0 | m1;
    }
    __device__ __forceinline__ bool open(int at) {   // the unit at position `at`; false behind the end
        int unit = unit_at(at, p.ngroups * p.nsplit * p.nparts);
        if (unit < 0) return false;
        part = unit % p.nparts, unit /= p.nparts;
        split = unit % p.nsplit, unit /= p.nsplit;
        block0 = __ldg(p.group_order + unit) * GROUP_BLOCKS;
        tap_lo = p.K * split / p.nsplit, tap_hi = p.K * (split + 1) / p.nsplit;
        return true;
    }
    __device__ __forceinline__ void take() {
        const int b = __ffs(left) - 1;
        left &= left - 1;
        tap = word * 32 + b;
        has = ((m0 >> b) & 1u) | (((m1 >> b) & 1u) << 1);
    }
    __device__ __forceinline__ bool next_here() {   // another tap of the unit (of one slice)
        while (!left) {
            if (word + 1 >= p.mask_words) return false;
            load(++word);
        }
        take();
        return true;
    }
    __device__ __forceinline__ bool next() {
        for (;;) {
            if (left) {
                take();
                first = opened, opened = false;
                return true;
            }
            if (q < slices && ++word < p.mask_words) {
                load(word);
            } else if (++q < slices) {
                word = 0;
                if (p.mask_words > 1) load(0);
                else left = m0 | m1;
            } else {
                if (!open(++n)) return false;
                q = 0, word = 0, opened = true;
                load(0);
            }
        }
    }
};

// PACK: taps of a step.  SPLIT: the scratch holds every bucket's sum as two 16-bit rows, the rounded sum and what the
// rounding left over, and the contraction goes over both: sums of twice as many bits (bf16: 2^-16 of the sum is lost where
// one row loses 2^-8), for a second pass over the taps.
template <int PACK, bool SPLIT>
__global__ void __launch_bounds__(THREADS, 1) mvmr_os_kernel(const __grid_constant__ CUtensorMap tmap, const __grid_constant__ OsParams p) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t s_full[MAX_SLOTS], s_empty[MAX_SLOTS], s_acc_full[2], s_acc_empty[2], s_step_full[AHEAD], s_step_empty[AHEAD];
    __shared__ uint32_t s_word[WORDS];
    __shared__ uint4 s_step[AHEAD];   // the step's word, its first feature column, the column of its weights
    constexpr int PIECE_SHIFT = PACK == 4 ? 1 : PACK == 2 ? 2 : 3;   // log2 of the 16-byte pieces a tap has of the 128-byte row of a tile
    __shared__ int s_wrow[AHEAD * PACK];   // and, of each of its taps, the first row
    __shared__ uint32_t s_tmem;
    __shared__ int s_abort;
    __shared__ float s_bias[BIAS_WIDTH];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // a slot: the A tiles of the group's two blocks, then the weight slice both use; behind the slots the
    // source rows of the next steps
    const uint32_t slot0 = (smem_u32(smem_raw) + 1023u) & ~1023u, rows0 = slot0 + (uint32_t)p.nslots * p.slot_bytes;
    const uint32_t entry_bytes = (uint32_t)PACK * ENTRY_BYTES;
    const bool w_plain = PACK > 1 && p.transpose;
    volatile int *abort_flag = &s_abort;
    auto wait = [&](const uint64_t &bar, uint32_t parity) {   // the verdict is the same in the whole warp
        if (__all_sync(0xffffffffu, mbar_try_wait(smem_u32(&bar), parity & 1u))) return true;
        return __all_sync(0xffffffffu, mbar_wait_abortable(smem_u32(&bar), parity & 1u, STATUS_BIT, p.status, abort_flag, p.wait_limit_ns)) != 0;
    };

    auto wait_one = [&](const uint64_t &bar, uint32_t parity) {   // for roles of a single thread
        return mbar_wait_abortable(smem_u32(&bar), parity & 1u, STATUS_BIT, p.status, abort_flag, p.wait_limit_ns);
    };

    if (tid == 0) {
        for (int s = 0; s < p.nslots; ++s)   // a team's copies and the weight slice; both MMA warps
            mbar_init(smem_u32(&s_full[s]), TEAM_WARPS * 32 + (w_plain ? 32 : 1)), mbar_init(smem_u32(&s_empty[s]), GROUP_BLOCKS);
        for (int s = 0; s < 2; ++s) mbar_init(smem_u32(&s_acc_full[s]), GROUP_BLOCKS), mbar_init(smem_u32(&s_acc_empty[s]), EPI_WARPS);
        for (int s = 0; s < WORDS; ++s) s_word[s] = 0u;
        for (int s = 0; s < AHEAD; ++s)   // the walk; a team and the weight warp
            mbar_init(smem_u32(&s_step_full[s]), 1), mbar_init(smem_u32(&s_step_empty[s]), TEAM_WARPS + 1);
        fence_mbar_init();
        s_abort = 0;
        tma_prefetch_desc(&tmap);
    }
    if (warp == 0) tmem_alloc(smem_u32(&s_tmem), p.ncols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    start_after_previous();   // (tensor memory is held by now: see there)
    const bool bias_here = p.bias && p.nsplit == 1 && p.out_pitch <= BIAS_WIDTH;
    if (bias_here) {
        for (int c = tid; c < p.out_pitch; c += THREADS) s_bias[c] = bias_at(p.bias, c, p.fmt);
        __syncthreads();
    }

    if (warp < EPI_WARPS) {
        // -------------------------------------------------------------- epilogue ----
        Walk w(p, false);
        Ring acc;
        for (int n = 0; w.open(n); ++n) {
            uint32_t any0 = 0, any1 = 0;
            for (int x = 0; x < p.mask_words; ++x) w.load(x), any0 |= w.m0, any1 |= w.m1;
            if (any0 | any1) {
                if (!wait(s_acc_full[acc.slot], acc.turn)) break;
                tc_fence_after();
            }
            const int col0 = w.part * p.outw;
            for (int b = 0; b < GROUP_BLOCKS && w.block0 + b < p.nblocks; ++b) {
                const int64_t slot = (int64_t)(w.block0 + b) * ROWS + warp * 32 + lane;
                const int32_t row = __ldg(p.perm + slot);
                const bool has = (b ? any1 : any0) != 0u;
                const uint32_t d = tmem + ((uint32_t)(warp * 32) << 16) + (acc.slot * 2 + (uint32_t)b) * p.col_stride;
                for (int c0 = 0; c0 < p.outw; c0 += 16) {
                    float v[16];
                    if (has) {
                        tmem_ld16(d + (uint32_t)c0, v);
                    } else {
#pragma unroll
                        for (int e = 0; e < 16; ++e) v[e] = 0.f;
                    }
                    if (row >= 0) {
                        if (p.nsplit > 1) {
                            // [split][block][four columns][row]: the lanes of a warp write next to each other
                            float4 *dst = reinterpret_cast<float4 *>(p.partial + ((int64_t)w.split * p.nblocks + w.block0 + b) * ROWS * p.out_pitch) +
                                          ((col0 + c0) >> 2) * ROWS + warp * 32 + lane;
#pragma unroll
                            for (int e = 0; e < 4; ++e) dst[e * ROWS] = make_float4(v[4 * e], v[4 * e + 1], v[4 * e + 2], v[4 * e + 3]);
                        } else {
                            if (bias_here) {
#pragma unroll
                                for (int e = 0; e < 16; ++e) v[e] += s_bias[col0 + c0 + e];
                            } else if (p.bias) {
#pragma unroll
                                for (int e = 0; e < 16; ++e) v[e] += bias_at(p.bias, col0 + c0 + e, p.fmt);
                            }
                            uint4 *dst = reinterpret_cast<uint4 *>(p.out + (int64_t)row * p.out_pitch + col0 + c0);
#pragma unroll
                            for (int e = 0; e < 2; ++e)
                                dst[e] = make_uint4(pack2(v[8 * e], v[8 * e + 1], p.fmt), pack2(v[8 * e + 2], v[8 * e + 3], p.fmt),
                                                    pack2(v[8 * e + 4], v[8 * e + 5], p.fmt), pack2(v[8 * e + 6], v[8 * e + 7], p.fmt));
                        }
                    }
                    __syncwarp();
                }
            }
            if (any0 | any1) {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&s_acc_empty[acc.slot]));
                acc.next(p.nacc);
            }
        }
    } else if (warp < WALK_WARP) {
        // ------------------------------------------------------------------ copies ----
        // Four teams take the steps in turn: while one team's copies go through the load/store unit (230 clocks
        // for a 16 KB tile) the others wait for their slots and fetch their rows.  A warp owns 32 rows of either
        // tile, eight lanes a row, a group of eight lanes eight consecutive rows.
        const int team = (warp - COPY_WARP0) / TEAM_WARPS, piece = lane & 7;
        const int row0 = ((warp - COPY_WARP0) % TEAM_WARPS) * 32 + (lane >> 3) * 8;
        const int tap_slot = piece >> PIECE_SHIFT, sub = piece & ((1 << PIECE_SHIFT) - 1);
        uint32_t dst_off[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) dst_off[k] = (uint32_t)(row0 + k) * 128 + (uint32_t)((piece ^ k) << 4);
        const uint32_t pitch = (uint32_t)p.in_pitch * 2u;
        Ring ring, step;
        for (int n = 0; n < team; ++n) ring.next(p.nslots), step.next(AHEAD);
        while (team < p.teams) {
            if (!wait(s_step_full[step.slot], step.turn)) break;
            const uint32_t word = *(volatile uint32_t *)&s_step[step.slot].x;
            if (word & STEP_END) break;
            const uint32_t at = rows0 + step.slot * entry_bytes + (uint32_t)tap_slot * ENTRY_BYTES + (uint32_t)row0 * 4;
            const uint4 rows[4] = {lds_v4(at), lds_v4(at + 16), lds_v4(at + ROWS * 4), lds_v4(at + ROWS * 4 + 16)};
            const uint32_t column = *(volatile uint32_t *)&s_step[step.slot].y + (uint32_t)sub * 8;
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&s_step_empty[step.slot]));
            const char *col = reinterpret_cast<const char *>(p.feat + column);
            const bool low = SPLIT && (word & STEP_LOW);
            const uint32_t sum_pitch = SPLIT ? 2 * pitch : pitch;
            const char *sums = reinterpret_cast<const char *>(p.scratch + column) + (low ? pitch : 0u) - sum_pitch;
            const bool piece_ok = piece < 2 * (int)((word >> 8) & 7u);
            // the tensor core has finished with what was in the slot
            if (!wait(s_empty[ring.slot], ring.turn ^ 1u)) break;
            const uint32_t dst = slot0 + ring.slot * p.slot_bytes;
            if (piece_ok) {
#pragma unroll
                for (int t = 0; t < 2; ++t) {
                    if (!((word >> (13 + t)) & 1u)) continue;
                    const uint32_t none = PACK == 1 || ((word >> (2 * tap_slot + t)) & 1u) ? 0u : 0xffffffffu;   // the tile has other taps of the step
                    const int32_t rr[8] = {(int32_t)(rows[2 * t].x | none), (int32_t)(rows[2 * t].y | none),
                                           (int32_t)(rows[2 * t].z | none), (int32_t)(rows[2 * t].w | none),
                                           (int32_t)(rows[2 * t + 1].x | none), (int32_t)(rows[2 * t + 1].y | none),
                                           (int32_t)(rows[2 * t + 1].z | none), (int32_t)(rows[2 * t + 1].w | none)};
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        // a feature row x >= 0, the row of bucket sums -2 - x, or nothing (-1: zeros, and a source that is not read)
                        const char *src = (rr[k] < -1 ? sums : col) + (uint64_t)(uint32_t)(rr[k] ^ (rr[k] >> 31)) * (SPLIT && rr[k] < -1 ? sum_pitch : pitch);
                        cp_async16_or_zero(dst + (uint32_t)t * SLOT_BYTES + dst_off[k], src, rr[k] == -1 || (SPLIT && low && rr[k] >= 0));
                    }
                }
            }
            cp_async_mbar_arrive(smem_u32(&s_full[ring.slot]));   // fires once this thread's copies have landed
            ring.skip(p.teams, p.nslots);
            step.skip(p.teams, AHEAD);
        }
        cp_async_wait<0>();
    } else if (warp == WALK_WARP) {
        // -------------------------------------------------------------------- walk ----
        // Decides the steps and brings the source rows of their tiles into shared memory, AHEAD steps early:
        // the tables come from DRAM, once.  One thread and a bulk copy a tile: as a warp with votes, a copy a lane
        // and the divisions of the part in every step it took 1300 clocks a step and held up everything behind it.
        if (elect_one()) {
            Walk w(p, SPLIT);
            Ring step, word;
            bool more = true;
            int column = 0, wx = 0, wy = 0;   // of the unit: first feature column, corner of its weights in the (taps * groups * C, M) matrix
            const int groups = p.nparts / p.out_parts, tap_rows = groups * p.C;
            for (int ends = 0; ends < p.teams;) {   // an end mark for each team
                if (!wait_one(s_step_empty[step.slot], step.turn ^ 1u)) break;
                if (more) more = w.next();
                const uint32_t full = smem_u32(&s_step_full[step.slot]);
                uint4 s = make_uint4(STEP_END, 0u, 0u, 0u);
                uint32_t tx = 0;
                if (more) {
                    if (w.first) {
                        const int g = w.part / p.out_parts, o = (w.part - g * p.out_parts) * p.outw;
                        column = g * p.inw, wx = p.transpose ? 0 : o, wy = g * p.C + (p.transpose ? o : 0);
                    }
                    const int k0 = (SPLIT && w.q >= p.nkb ? w.q - p.nkb : w.q) * 64;
                    uint32_t entry = rows0 + step.slot * entry_bytes, any = 0;
                    s.x = (w.first ? STEP_FIRST : 0u) | (SPLIT && w.q >= p.nkb ? STEP_LOW : 0u);
                    int n = 0;
                    do {
                        const int32_t *src = p.tile_rows + ((int64_t)w.block0 * p.K + w.tap) * ROWS;
                        const int tap = p.reverse ? p.K - 1 - w.tap : w.tap;
                        if (w.has & 1u) bulk_load(entry, src, ROWS * 4, full);
                        if (w.has & 2u) bulk_load(entry + ROWS * 4, src + (int64_t)p.K * ROWS, ROWS * 4, full);
                        s_wrow[step.slot * PACK + n] = tap * tap_rows + wy + (p.transpose ? 0 : k0);
                        s.x |= w.has << (2 * n), any |= w.has, tx += (w.has & 1u) + (w.has >> 1), entry += ENTRY_BYTES;
                    } while (++n < PACK && w.next_here());
                    s.x |= any << 13 | (uint32_t)(PACK > 1 ? n * p.inw : min(64, p.inw - k0)) >> 4 << 8;
                    s.y = (uint32_t)(column + k0);
                    s.z = (uint32_t)(wx + (p.transpose ? k0 : 0));
                    s.w = (uint32_t)n;
                }
                s_step[step.slot] = s;
                *(volatile uint32_t *)&s_word[word.slot] = s.x | ((word.turn + 1u) & 0x7fffu) << TURN_SHIFT;
                if (more) {
                    mbar_arrive_expect_tx(full, tx * (ROWS * 4));
                } else {
                    mbar_arrive(full);
                    ++ends;
                }
                step.next(AHEAD);
                word.next(WORDS);
            }
        }
        __syncwarp();
    } else if (warp == WEIGHT_WARP) {
        // ---------------------------------------------------------------- weights ----
        Ring ring, step;
        for (;;) {
            if (!wait(s_step_full[step.slot], step.turn)) break;
            const uint32_t word = *(volatile uint32_t *)&s_step[step.slot].x;
            if (word & STEP_END) break;
            const int x = *(volatile int *)&s_step[step.slot].z, taps = PACK > 1 ? *(volatile int *)&s_step[step.slot].w : 1;
            int y[PACK];
#pragma unroll
            for (int n = 0; n < PACK; ++n) y[n] = *(volatile int *)&s_wrow[step.slot * PACK + n];
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&s_step_empty[step.slot]));
            if (!wait(s_empty[ring.slot], ring.turn ^ 1u)) break;
            const uint32_t dst = slot0 + ring.slot * p.slot_bytes + 2 * SLOT_BYTES, full = smem_u32(&s_full[ring.slot]);
            if (w_plain) {   // a row (output channel) holds the contraction of all taps of the step: narrower than a box of the map can place
                const int ppt = 1 << PIECE_SHIFT;
#pragma unroll
                for (int n = 0; n < PACK; ++n) {
                    if (n >= taps) continue;
                    for (int c = lane; c < p.outw * ppt; c += 32) {
                        const int row = c >> PIECE_SHIFT, piece = c & (ppt - 1);
                        cp_async16(dst + (uint32_t)row * 128 + (uint32_t)(((n * ppt + piece) ^ (row & 7)) << 4),
                                   p.weight + (int64_t)(y[n] + row) * p.M + piece * 8);
                    }
                }
                cp_async_mbar_arrive(full);
            } else if (lane == 0) {
                mbar_arrive_expect_tx(full, p.w_tx_bytes * (uint32_t)taps);
                if (p.transpose) {   // contraction over m: an m-block of the output channels' rows
                    tma_load_2d(dst, &tmap, x, y[0], full);
                } else {             // contraction over c: the rows of a 64-channel slice or of several taps, one box per 64 output channels
#pragma unroll
                    for (int n = 0; n < PACK; ++n)
                        for (int mb = 0; n < taps && mb * 64 < p.outw; ++mb)
                            tma_load_2d(dst + ((uint32_t)mb * p.w_rows + (uint32_t)n * p.w_box_rows) * 128, &tmap, x + mb * 64, y[n], full);
                }
            }
            ring.next(p.nslots);
            step.next(AHEAD);
        }
        cp_async_wait<0>();
    } else {
        // -------------------------------------------------------------------- MMA ----
        // One warp per block of the group: the issue of a step (waits, descriptors, four tcgen05.mma, commit) is a
        // serial chain of several hundred clocks, and with one warp for both tiles it bounded the kernel.
        const int t = warp - MMA_WARP0;
        const uint32_t idesc = instr_desc(p.fmt, ROWS, p.outw, 0, p.transpose ? 0 : 1);
        // descriptors of slot 0 / contraction step 0; the address field counts 16-byte units, so another
        // slot or step is an addition to the low word
        const uint32_t w0 = slot0 + 2 * SLOT_BYTES;
        const uint64_t a_desc0 = smem_desc(slot0 + (uint32_t)t * SLOT_BYTES, 16, 1024);
        const uint64_t b_desc0 = p.transpose ? smem_desc(w0, 16, 1024) : smem_desc(w0, p.w_rows * 128, 1024);
        const uint32_t b_step = p.transpose ? 2u : 128u;   // 32 bytes along a K-major row / 16 contraction rows of 128 bytes
        if (elect_one()) {   // one thread from here on: no warp-wide votes or barriers in the chain
            Ring ring, acc, step;
            uint32_t started = 0;
            bool open = false, ok = true;
            auto peek = [&]() { return *(volatile uint32_t *)&s_word[step.slot]; };
            uint32_t word = peek();
            for (;;) {
                // the step's word has been written for this turn of the ring (bounded as every wait)
                for (uint64_t t0 = 0; ok && (word >> TURN_SHIFT) != ((step.turn + 1u) & 0x7fffu); word = peek()) {
                    const uint64_t t = global_timer_ns();
                    if (t0 == 0) t0 = t;
                    if (s_abort || t - t0 > p.wait_limit_ns) {
                        if (!s_abort) atomicOr(p.status, STATUS_BIT), *abort_flag = 1;
                        ok = false;
                    }
                }
                if (!ok || (word & STEP_END)) break;
                const uint32_t now = word;
                step.next(WORDS);
                word = peek();   // the next step's, most likely there already
                if (now & STEP_FIRST) {
                    if (open) tc_commit(smem_u32(&s_acc_full[acc.slot])), acc.next(p.nacc);
                    ok = wait_one(s_acc_empty[acc.slot], acc.turn ^ 1u);
                    if (!ok) break;
                    open = true, started = 0;
                }
                ok = wait_one(s_full[ring.slot], ring.turn);
                if (!ok) break;
                if ((now >> (13 + t)) & 1u) {
                    fence_async_smem();   // the copies came through the generic proxy, the tensor core reads through the async proxy
                    tc_fence_after();
                    const uint64_t at = (uint64_t)(ring.slot * (p.slot_bytes >> 4));
                    const int ksteps = (int)((now >> 8) & 7u);
                    const uint64_t ad = a_desc0 + at, bd = b_desc0 + at;
                    const uint32_t d = tmem + (acc.slot * 2 + (uint32_t)t) * p.col_stride;
                    tc_mma(d, ad, bd, idesc, started);
                    if (ksteps == 4) {
                        tc_mma(d, ad + 2, bd + b_step, idesc, 1u);
                        tc_mma(d, ad + 4, bd + 2 * b_step, idesc, 1u);
                        tc_mma(d, ad + 6, bd + 3 * b_step, idesc, 1u);
                    } else {
                        for (int k = 1; k < ksteps; ++k) tc_mma(d, ad + (uint64_t)(2 * k), bd + (uint64_t)(b_step * k), idesc, 1u);
                    }
                    tc_commit(smem_u32(&s_empty[ring.slot]));
                    started = 1u;
                } else {
                    mbar_arrive(smem_u32(&s_empty[ring.slot]));
                }
                ring.next(p.nslots);
            }
            if (ok && open) tc_commit(smem_u32(&s_acc_full[acc.slot]));
        }
        __syncwarp();
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, p.ncols);
}

// out[perm[slot]] = the parts of a split group added in order, plus the bias, rounded once.  Small outputs, so bound
// by latency: four columns a thread, the loads of REDUCE_BATCH parts in flight together.
constexpr int REDUCE_BATCH = 9;
__global__ void __launch_bounds__(128) os_reduce_kernel(const float *__restrict__ partial, const int32_t *__restrict__ perm,
                                                        const uint16_t *__restrict__ bias, int64_t slots, int outw, int nsplit, int fmt,
                                                        uint16_t *out) {
    start_after_previous();
    // a block of threads: the rows of a block of the plan, four columns
    const int64_t block = blockIdx.x;
    const int c = (int)blockIdx.y * 4, lane = threadIdx.x;
    const int32_t row = perm[block * ROWS + lane];
    if (row < 0) return;
    float v[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) v[e] = bias ? bias_at(bias, c + e, fmt) : 0.f;
    const float4 *src = reinterpret_cast<const float4 *>(partial + block * ROWS * outw) + (c >> 2) * ROWS + lane;
    const int64_t part = slots * (outw >> 2);
    for (int s0 = 0; s0 < nsplit; s0 += REDUCE_BATCH) {
        float4 a[REDUCE_BATCH];
#pragma unroll
        for (int s = 0; s < REDUCE_BATCH; ++s) a[s] = s0 + s < nsplit ? __ldcs(src + (s0 + s) * part) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int s = 0; s < REDUCE_BATCH; ++s) v[0] += a[s].x, v[1] += a[s].y, v[2] += a[s].z, v[3] += a[s].w;
    }
    *reinterpret_cast<uint2 *>(out + (int64_t)row * outw + c) = make_uint2(pack2(v[0], v[1], fmt), pack2(v[2], v[3], fmt));
}

// A single thread waits on an mbarrier that nothing arrives at: the bounded wait runs out,
// raises `flag` in the status word and the kernel returns.
__global__ void wait_runs_out_kernel(unsigned int *status, unsigned flag, uint64_t limit_ns) {
    __shared__ uint64_t s_bar;
    __shared__ int s_abort;
    if (threadIdx.x == 0) {
        mbar_init(smem_u32(&s_bar), 1);
        fence_mbar_init();
        s_abort = 0;
        mbar_wait_abortable(smem_u32(&s_bar), 0u, flag, status, &s_abort, limit_ns);
    }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// cuTensorMapEncodeTiled through the runtime's driver entry point table (the library does not
// link against libcuda); null when the driver does not offer it.
EncodeTiledFn encode_tiled() {
    static EncodeTiledFn fn = nullptr;
    static bool tried = false;
    if (!tried) {
        tried = true;
        void *ptr = nullptr;
        cudaDriverEntryPointQueryResult res;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &res) == cudaSuccess &&
            res == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)ptr;
        else
            (void)cudaGetLastError();
    }
    return fn;
}

unsigned int *status_word() {
    static unsigned int *ptr[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
    if (!ptr[dev & 63] && device_status_address(&ptr[dev & 63]) != PCX_OK) return nullptr;
    return ptr[dev & 63];
}

uint64_t wait_limit() {
    static uint64_t v = 0;
    if (!v) {
        const char *e = getenv("PCX_WAIT_LIMIT_NS");
        v = e ? strtoull(e, nullptr, 10) : 0;
        if (!v) v = WAIT_LIMIT_NS;
    }
    return v;
}

// What a group is split into when the groups alone do not fill the chip: parts of its taps, whose fp32 sums go through memory
// to os_reduce_kernel, and of its columns, whose rows are copied once per part.  The pair with the smallest time, by what the
// kernels measured on B200 (in us): 0.6 a step, 0.015 a column of the epilogue, both for every unit a CTA works off in turn;
// 0.27 for a MB of sums, written and read; 0.2 for reading the rows once more.  27 taps and 22 triplets a row, against the
// taps alone at a tenth of a group for every part (ten calls in a graph: alone, a call of 942 points is bound by its host):
//   points  channels   taps x columns   us             points  channels   taps x columns   us
//      942    256       27 -> 14 x 2    22.6 -> 20.1     3000     64        12 -> 9         16.8 -> 14.5
//     2000    256       14 -> 9 x 2     26.8 -> 23.5      500    512        27 -> 14 x 2    25.3 -> 24.4
//     4000 points and more, and 942 of 512 channels: as before
// `slices` of 64 channels the contraction has, `pack` taps a step; `width` columns of a part.
struct Split { int taps, columns; };
Split split_of(int64_t ngroups, int K, int nparts, int width, int slices, int pack, int64_t row_floats) {
    const int64_t sms = num_sms(), units = ngroups * nparts;
    Split best = {1, 1};
    if (units >= 2 * sms) return best;
    const float mb_us = 0.27e-6f * 4.f * (float)(ngroups * GROUP_BLOCKS * ROWS * row_floats);
    float best_us = 1e30f;
    // the fewest parts for every number of taps a part may have: few candidates, as every call asks
    for (int s = 1, taps = K; s <= 64; s = (K + taps - 2) / (taps - 1), taps = (K + s - 1) / s) {
        const float steps = 0.6f * (float)((taps + pack - 1) / pack * slices);
        for (int q = 1; q <= 4 && width % (16 * q) == 0 && (q == 1 || width / q >= 64) && nparts * q <= 64; q *= 2) {
            const float us = (float)((units * q * s + sms - 1) / sms) * (steps + 0.015f * (float)(width / q)) + (s > 1 ? mb_us * (float)s : 0.f) + 0.2f * (float)(q - 1);
            if (us < best_us * 0.999f) best_us = us, best = {s, q};
        }
        if (taps == 1) break;
    }
    return best;
}
int taps_of_a_step(int inw) { return inw == 16 ? 4 : inw == 32 ? 2 : 1; }

// fp32 sums of a rulebook whose taps are split
size_t partial_bytes(int64_t n_out, int outw, int splits) {
    return splits > 1 ? (size_t)splits * ((n_out + ROWS - 1) / ROWS) * ROWS * outw * sizeof(float) : 0;
}

bool plan_sizes_ok(int64_t T, int64_t n_out, int K, int G) {
    if (T < 0 || T > INT32_MAX || n_out <= 0 || n_out > INT32_MAX || K <= 0 || K > MAX_TAPS) return false;
    if (G != GROUP_BLOCKS) return false;
    const int64_t nblocks = (n_out + ROWS - 1) / ROWS;
    return nblocks * K * ROWS <= ((int64_t)1 << 32) && nblocks * K < INT32_MAX;
}

// groups, most tiles first, and the tap sets of their blocks
int order_groups(const PlanView &pv, const BuildWs &w, int K, int G, cudaStream_t stream) {
    launch_after(plan_cost_kernel, (unsigned)((pv.ngroups + 255) / 256), 256, 0, stream, pv.tile_offs, pv.nblocks, K, G, pv.ngroups, w.cost, w.gid,
                                                                               pv.tap_masks);
    PCX_LAUNCH_CHECK();
    size_t bytes = w.cub_bytes;
    PCX_CUDA(cub::DeviceRadixSort::SortPairsDescending(w.cub_tmp, bytes, w.cost, w.cost_sorted, w.gid, pv.group_order, (int)pv.ngroups, 0,
                                                       bits_of((int64_t)G * K + 2), stream));
    return PCX_OK;
}

}  // namespace
}  // namespace pcx

using namespace pcx;

extern "C" {

int pcx_mvmr_plan_group_blocks(int out_width) {
    if (out_width <= 0 || out_width > 256) return 0;   // wider rows are worked off in parts of at most 256
    // Two: both accumulators of the widest rows (256 channels) fill the tensor memory, and every weight
    // slice that is streamed serves 256 output rows.
    return GROUP_BLOCKS;
}

size_t pcx_mvmr_plan_bytes(int64_t T, int64_t n_out, int K, int group_blocks) {
    if (!plan_sizes_ok(T, n_out, K, group_blocks)) return 0;
    return carve_plan(nullptr, T, n_out, K, group_blocks, nullptr);
}

size_t pcx_mvmr_plan_workspace_bytes(int64_t T, int64_t n_out, int K, int group_blocks) {
    if (!plan_sizes_ok(T, n_out, K, group_blocks)) return 0;
    return carve_build(nullptr, T, n_out, K, group_blocks, nullptr);
}

int pcx_mvmr_plan_build(const int32_t *d_scatter, const int32_t *d_gather, const int64_t *d_seg_offs, int64_t T, int K,
                        int64_t n_out, int group_blocks, void *d_plan, size_t plan_bytes, void *d_ws, size_t ws_bytes,
                        void *stream) {
    int64_t multi = 0;
    return pcx_mvmr_plan_build_counted(d_scatter, d_gather, d_seg_offs, T, K, n_out, group_blocks, d_plan, plan_bytes, d_ws, ws_bytes,
                                       &multi, stream);
}

int pcx_mvmr_plan_build_counted(const int32_t *d_scatter, const int32_t *d_gather, const int64_t *d_seg_offs, int64_t T, int K,
                                int64_t n_out, int group_blocks, void *d_plan, size_t plan_bytes, void *d_ws, size_t ws_bytes,
                                int64_t *h_multi, void *stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    const int G = group_blocks;
    if (!plan_sizes_ok(T, n_out, K, G))
        PCX_FAIL(PCX_E_UNSUPPORTED, "pcx_mvmr_plan_build: sizes out of range (T=%lld n_out=%lld K=%d group=%d)", (long long)T,
                 (long long)n_out, K, G);
    if (!d_plan || !d_ws || (T > 0 && (!d_scatter || !d_gather || !d_seg_offs)))
        PCX_FAIL(PCX_E_ARG, "pcx_mvmr_plan_build: null pointer");
    if ((uintptr_t)d_plan % 256 || (uintptr_t)d_ws % 256)
        PCX_FAIL(PCX_E_ALIGN, "pcx_mvmr_plan_build: plan and workspace must be 256-byte aligned");
    PlanView pv;
    BuildWs w;
    const size_t need_plan = carve_plan(d_plan, T, n_out, K, G, &pv), need_ws = carve_build(d_ws, T, n_out, K, G, &w);
    if (plan_bytes < need_plan) PCX_FAIL(PCX_E_CAPACITY, "pcx_mvmr_plan_build: plan buffer %zu < %zu bytes", plan_bytes, need_plan);
    if (ws_bytes < need_ws) PCX_FAIL(PCX_E_CAPACITY, "pcx_mvmr_plan_build: workspace %zu < %zu bytes", ws_bytes, need_ws);
    const int TPB = 256;
    const int64_t n_tiles = pv.nblocks * K, n_pad = pv.nblocks * ROWS;
    auto blocks = [&](int64_t n) { return (unsigned)((n + TPB - 1) / TPB); };
    const int64_t init_n = std::max(std::max<int64_t>(n_out, n_tiles + 1),
                                    std::max<int64_t>(CTRL_WORDS, std::min<int64_t>(n_tiles * (ROWS / 4), (int64_t)num_sms() * 2048)));
    launch_after(plan_init_kernel, blocks(init_n), TPB, 0, stream, n_out, w.sig, w.row, w.tile_cnt, n_tiles, pv.ctrl, G,
                 reinterpret_cast<int4 *>(pv.tile_rows));
    PCX_LAUNCH_CHECK();
    size_t bytes = w.cub_bytes;
    if (T > 0) {
        launch_after(plan_sig_kernel, blocks(T), TPB, 0, stream, d_scatter, d_seg_offs, T, K, w.sig, pv.ctrl);
        PCX_LAUNCH_CHECK();
    }
    // rows by (planes, signature), stable: rows of equal keys keep their order
    int ks = 1;
    while (ks * ks * ks < K) ++ks;
    if (ks * ks * ks != K || K > 32 || K == 1) ks = 0;
    launch_after(plan_order_kernel, blocks(n_out), TPB, 0, stream, w.sig, n_out, K, ks, w.order);
    PCX_LAUNCH_CHECK();
    PCX_CUDA(cub::DeviceRadixSort::SortPairs(w.cub_tmp, bytes, w.order, w.order_sorted, w.row, w.row_sorted, (int)n_out, 0,
                                             std::min(K, 32) + 3 * ks, stream));
    launch_after(plan_rank_kernel, blocks(n_pad), TPB, 0, stream, w.row_sorted, n_out, n_pad, w.rank, pv.perm);
    PCX_LAUNCH_CHECK();
    if (T > 0) {
        launch_after(plan_heads_kernel, blocks(T), TPB, 0, stream, d_scatter, d_seg_offs, w.rank, T, K, pv.ctrl, pv.tile_rows, w.tile_cnt);
        PCX_LAUNCH_CHECK();
    }
    bytes = w.cub_bytes;
    PCX_CUDA(cub::DeviceScan::ExclusiveSum(w.cub_tmp, bytes, w.tile_cnt, pv.tile_offs, (int)(n_tiles + 1), stream));
    if (T > 0) {
        launch_after(plan_tiles_kernel, blocks(n_tiles * 32), TPB, 0, stream, d_scatter, d_gather, d_seg_offs, K, n_tiles, pv.tile_offs, pv.entries,
                                                                   pv.tile_rows, pv.buckets, pv.ctrl);
        PCX_LAUNCH_CHECK();
    }
    if (int rc = order_groups(pv, w, K, G, stream)) return rc;
    if (!h_multi) return PCX_OK;   // rows ascend inside every tap: the caller says so
    uint32_t *h = reinterpret_cast<uint32_t *>(handover_words());
    PCX_CUDA(cudaMemcpyAsync(h, pv.ctrl, 8 * sizeof(uint32_t), cudaMemcpyDeviceToHost, stream));
    PCX_CUDA(cudaStreamSynchronize(stream));
    *h_multi = h[CTRL_NMULTI];
    if (!h[CTRL_UNSORTED]) return PCX_OK;

    // rows out of order inside a tap: nothing has been placed yet, the triplets are sorted
    launch_after(plan_keys_kernel, blocks(T), TPB, 0, stream, d_scatter, d_gather, d_seg_offs, w.rank, T, K, w.key, w.val, w.tile_cnt);
    PCX_LAUNCH_CHECK();
    bytes = w.cub_bytes;
    PCX_CUDA(cub::DeviceRadixSort::SortPairs(w.cub_tmp, bytes, w.key, w.key_sorted, w.val, w.val_sorted, (int)T, 0,
                                             std::min(32, bits_of(n_tiles * ROWS)), stream));
    bytes = w.cub_bytes;
    PCX_CUDA(cub::DeviceScan::ExclusiveSum(w.cub_tmp, bytes, w.tile_cnt, pv.tile_offs, (int)(n_tiles + 1), stream));
    launch_after(plan_entries_kernel, blocks(T), TPB, 0, stream, w.key_sorted, w.val_sorted, T, pv.entries, pv.tile_rows, pv.buckets, pv.ctrl);
    PCX_LAUNCH_CHECK();
    if (int rc = order_groups(pv, w, K, G, stream)) return rc;
    return pcx_mvmr_plan_multi_buckets(d_plan, h_multi, stream);
}

size_t pcx_mvmr_planned_workspace_bytes(int64_t multi_buckets, int in_width) {
    if (multi_buckets < 0 || in_width <= 0) return 0;
    return align_up((size_t)std::max<int64_t>(multi_buckets, 1) * in_width * 2, 256);
}

size_t pcx_mvmr_planned_scratch_bytes(int64_t multi_buckets, int in_width, int64_t n_out, int out_width, int K, int G) {
    if (multi_buckets < 0 || in_width <= 0 || n_out <= 0 || out_width <= 0 || K <= 0 || G <= 0) return 0;
    const int64_t ngroups = (n_out + GROUP_BLOCKS * ROWS - 1) / (GROUP_BLOCKS * ROWS);
    return pcx_mvmr_planned_workspace_bytes(multi_buckets, G * in_width) +
           partial_bytes(n_out, G * out_width, split_of(ngroups, K, G * parts_of(out_width), out_width / parts_of(out_width), (in_width + 63) / 64,
                                                        taps_of_a_step(in_width), G * out_width).taps);
}

int pcx_mvmr_plan_multi_buckets(const void *d_plan, int64_t *h_count, void *stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    if (!d_plan || !h_count) PCX_FAIL(PCX_E_ARG, "pcx_mvmr_plan_multi_buckets: null pointer");
    uint32_t n = 0;
    PCX_CUDA(cudaMemcpyAsync(&n, (const uint32_t *)d_plan + CTRL_NMULTI, sizeof(n), cudaMemcpyDeviceToHost, stream));
    PCX_CUDA(cudaStreamSynchronize(stream));
    *h_count = n;
    return PCX_OK;
}

int pcx_mvmr_planned(const void *d_weight, const void *d_feat, void *d_plan, size_t plan_bytes, void *d_out, int64_t T,
                     int64_t n_feat, int64_t n_out, int K, int C, int M, int transpose, int dtype, int group_blocks,
                     int64_t multi_buckets, void *d_ws, size_t ws_bytes, void *stream) {
    return pcx_mvmr_planned_bias(d_weight, d_feat, d_plan, plan_bytes, nullptr, d_out, T, n_feat, n_out, K, 1, C, M,
                                 transpose ? PCX_MVMR_TRANSPOSE : 0, dtype, group_blocks, multi_buckets, d_ws, ws_bytes, stream);
}

int pcx_mvmr_planned_bias(const void *d_weight, const void *d_feat, void *d_plan, size_t plan_bytes, const void *d_bias, void *d_out,
                          int64_t T, int64_t n_feat, int64_t n_out, int K, int groups, int C, int M, int flags, int dtype,
                          int group_blocks, int64_t multi_buckets, void *d_ws, size_t ws_bytes, void *stream) {
    return mvmr_planned(d_weight, d_feat, d_plan, plan_bytes, d_bias, d_out, T, n_feat, n_out, K, groups, C, M, flags, dtype, group_blocks,
                        multi_buckets, nullptr, nullptr, d_ws, ws_bytes, stream);
}

int pcx_debug_wait_runs_out(unsigned long long limit_ns, void *stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    if (limit_ns == 0 || limit_ns > 100000000ull) PCX_FAIL(PCX_E_ARG, "pcx_debug_wait_runs_out: limit must be within (0, 100 ms]");
    unsigned int *status = status_word();
    if (!status) PCX_FAIL(PCX_E_LAUNCH, "pcx_debug_wait_runs_out: no device status word");
    wait_runs_out_kernel<<<1, 32, 0, stream>>>(status, 8u, (uint64_t)limit_ns);
    PCX_LAUNCH_CHECK();
    return PCX_OK;
}

}  // extern "C"

// The call itself.  odd: null, or room for MAX_ODD words, of which the first *n_odd say afterwards (zero or not) whether a
// split sum or a weight was not finite.
int pcx::mvmr_planned(const void *d_weight, const void *d_feat, void *d_plan, size_t plan_bytes, const void *d_bias, void *d_out, int64_t T,
                      int64_t n_feat, int64_t n_out, int K, int groups, int C, int M, int flags, int dtype, int group_blocks,
                      int64_t multi_buckets, uint32_t *odd, int *n_odd, void *d_ws, size_t ws_bytes, void *stream_) {
    const int transpose = flags & PCX_MVMR_TRANSPOSE;
    const bool split_sums = (flags & PCX_MVMR_SPLIT_SUMS) != 0;
    cudaStream_t stream = (cudaStream_t)stream_;
    const int G = group_blocks;
    if (dtype != PCX_F16 && dtype != PCX_BF16) PCX_FAIL(PCX_E_DTYPE, "pcx_mvmr_planned: fp16 or bf16 only (dtype %d)", dtype);
    if (C <= 0 || M <= 0 || n_feat < 0 || groups <= 0) PCX_FAIL(PCX_E_ARG, "pcx_mvmr_planned: bad sizes");
    if (!plan_sizes_ok(T, n_out, K, G))
        PCX_FAIL(PCX_E_UNSUPPORTED, "pcx_mvmr_planned: sizes out of range (T=%lld n_out=%lld K=%d group=%d)", (long long)T,
                 (long long)n_out, K, G);
    const int inw = transpose ? M : C, outw = transpose ? C : M;
    // output rows wider than the tensor memory's two accumulators (256 channels), and those of a grouped weight, are
    // worked off in parts of the same width
    int out_parts = parts_of(outw), nparts = groups * out_parts;
    if (inw % 16 || outw % (16 * out_parts) || inw > 1024 || groups * inw > 2048 || nparts > 64)
        PCX_FAIL(PCX_E_UNSUPPORTED, "pcx_mvmr_planned: channel counts must be multiples of 16 and the parts of an output row equal (groups=%d C=%d M=%d)", groups, C, M);
    if (!d_weight || !d_plan || !d_out || (T > 0 && !d_feat)) PCX_FAIL(PCX_E_ARG, "pcx_mvmr_planned: null pointer");
    if ((uintptr_t)d_weight % 16 || (uintptr_t)d_feat % 16 || (uintptr_t)d_out % 16 || (uintptr_t)d_plan % 256 || (uintptr_t)d_ws % 256)
        PCX_FAIL(PCX_E_ALIGN, "pcx_mvmr_planned: weight, features and output must be 16-byte aligned, plan and workspace 256-byte aligned");
    if (multi_buckets < 0 || multi_buckets > T / 2) PCX_FAIL(PCX_E_ARG, "pcx_mvmr_planned: multi_buckets out of range");
    const size_t sums_bytes = pcx_mvmr_planned_workspace_bytes(multi_buckets, groups * inw * (split_sums ? 2 : 1));
    if (multi_buckets > 0 && (!d_ws || ws_bytes < sums_bytes))
        PCX_FAIL(PCX_E_CAPACITY, "pcx_mvmr_planned: workspace %zu < %zu bytes", ws_bytes, sums_bytes);
    PlanView pv;
    const size_t need_plan = carve_plan(d_plan, T, n_out, K, G, &pv);
    if (plan_bytes < need_plan) PCX_FAIL(PCX_E_CAPACITY, "pcx_mvmr_planned: plan buffer %zu < %zu bytes", plan_bytes, need_plan);

    // the fp32 sums of split taps lie behind the bucket sums; a caller that made no room for them gets one part
    Split split = split_of(pv.ngroups, K, nparts, outw / out_parts, (inw * (split_sums ? 2 : 1) + 63) / 64, taps_of_a_step(inw * (split_sums ? 2 : 1)),
                           (int64_t)groups * outw);
    if (split.taps > 1 && (!d_ws || ws_bytes < sums_bytes + partial_bytes(n_out, groups * outw, split.taps))) split = {1, 1};
    out_parts *= split.columns, nparts *= split.columns;

    OsParams p = {};
    p.nsplit = split.taps, p.partial = p.nsplit > 1 ? (float *)((char *)d_ws + sums_bytes) : nullptr;
    p.feat = (const uint16_t *)d_feat, p.out = (uint16_t *)d_out, p.bias = (const uint16_t *)d_bias;
    p.perm = pv.perm, p.group_order = pv.group_order, p.tile_rows = pv.tile_rows, p.tap_masks = pv.tap_masks;
    p.scratch = (const uint16_t *)d_ws;
    p.status = status_word();
    if (!p.status) PCX_FAIL(PCX_E_LAUNCH, "pcx_mvmr_planned: no device status word");
    p.K = K, p.C = C, p.M = M, p.transpose = transpose ? 1 : 0, p.fmt = dtype == PCX_BF16 ? 1 : 0;
    p.reverse = (flags & PCX_MVMR_REVERSE_TAPS) ? 1 : 0;
    p.nparts = nparts, p.out_parts = out_parts, p.in_pitch = groups * inw, p.out_pitch = groups * outw;
    p.inw = inw, p.outw = outw / out_parts, p.nkb = (inw + 63) / 64, p.mask_words = (K + 31) / 32;
    p.ngroups = (int)pv.ngroups, p.nblocks = (int)pv.nblocks;
    p.col_stride = (uint32_t)((p.outw + 31) / 32 * 32);
    p.nacc = 4 * p.col_stride <= 512 ? 2 : 1;   // up to 128 channels the next group starts while the last one is written
    p.ncols = 32;
    while (p.ncols < 2u * (uint32_t)p.nacc * p.col_stride) p.ncols <<= 1;
    // A step costs its chain of waits, copies and MMA issue, some 1000 clocks, whatever the width: rows of 16 or 32
    // channels fill the 64 of a step with four or two taps.
    const int pack = taps_of_a_step(inw);
    p.weight = (const uint16_t *)d_weight;
    p.w_box_rows = (uint32_t)(transpose ? p.outw : std::min(64, C));
    p.w_rows = transpose ? p.w_box_rows : p.w_box_rows * (uint32_t)pack;
    const uint32_t boxes = transpose ? 1u : (uint32_t)((p.outw + 63) / 64);
    p.w_tx_bytes = boxes * p.w_box_rows * 128u;
    p.slot_bytes = 2 * SLOT_BYTES + (uint32_t)align_up((size_t)boxes * p.w_rows * 128u, 1024);
    p.wait_limit_ns = wait_limit();
    if (!encode_tiled()) PCX_FAIL(PCX_E_LAUNCH, "pcx_mvmr_planned: the driver offers no cuTensorMapEncodeTiled");

    // widths that are not multiples of 64: the last box of a row ends in zero fill
    CUtensorMap tmap;
    memset(&tmap, 0, sizeof(tmap));
    const cuuint64_t gdim[2] = {(cuuint64_t)M, (cuuint64_t)K * (cuuint64_t)groups * (cuuint64_t)C};
    const cuuint64_t gstride[1] = {(cuuint64_t)M * 2};
    const cuuint32_t box[2] = {64u, p.w_box_rows};
    const cuuint32_t estride[2] = {1u, 1u};
    const CUresult r = encode_tiled()(&tmap, dtype == PCX_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2,
                                      const_cast<void *>(d_weight), gdim, gstride, box, estride, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                      CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) PCX_FAIL(PCX_E_LAUNCH, "pcx_mvmr_planned: cuTensorMapEncodeTiled failed (%d)", (int)r);

    // as many slots as fit: three of 64 KB at 256 output channels, five of 40 KB at 64
    p.nslots = (int)std::min<size_t>(MAX_SLOTS, ((size_t)232448 - 1024 - 1536 - BIAS_WIDTH * sizeof(float) - AHEAD * pack * ENTRY_BYTES) / p.slot_bytes);
    // A team at step n has waited for the release of step n - teams - nslots, and its next wait names step n - nslots
    // by the parity of its turn alone: with more teams than slots that could still be a turn further back.
    p.teams = std::min(TEAMS, p.nslots);
    if (p.nslots < 2) PCX_FAIL(PCX_E_UNSUPPORTED, "pcx_mvmr_planned: shared memory does not fit (C=%d M=%d)", C, M);
    const size_t smem = 1024 + (size_t)p.nslots * p.slot_bytes + AHEAD * pack * ENTRY_BYTES;
    auto kernel = split_sums ? (pack == 4 ? mvmr_os_kernel<4, true> : pack == 2 ? mvmr_os_kernel<2, true> : mvmr_os_kernel<1, true>)
                             : (pack == 4 ? mvmr_os_kernel<4, false> : pack == 2 ? mvmr_os_kernel<2, false> : mvmr_os_kernel<1, false>);
    static std::atomic<uint64_t> allowed[6];
    if (int rc = allow_shared_memory((const void *)kernel, &allowed[(pack >> 1) + (split_sums ? 3 : 0)])) return rc;
    const unsigned grid = (unsigned)std::max<int64_t>(1, std::min<int64_t>(pv.ngroups * p.nsplit * nparts, num_sms()));
    if (multi_buckets > 0 || odd) {   // (with no sums it looks at the weights alone)
        prof_begin("bucket_sum_kernel", stream);
        auto sum = split_sums ? (p.fmt ? launch_bucket_sum<1, true> : launch_bucket_sum<0, true>) : (p.fmt ? launch_bucket_sum<1, false> : launch_bucket_sum<0, false>);
        const int blocks = sum(multi_buckets, p.in_pitch, p.feat, pv.entries, pv.buckets, pv.ctrl, (uint16_t *)d_ws, (const uint4 *)d_weight,
                               (int64_t)K * groups * C * M / 8, odd, stream);
        if (odd) *n_odd = blocks;
        prof_end(stream);
        PCX_LAUNCH_CHECK();
    }
    prof_begin(transpose ? "mvmr_os_kernel(dgrad)" : "mvmr_os_kernel(fwd)", stream);
    launch_after(kernel, grid, THREADS, smem, stream, tmap, p);
    prof_end(stream);
    PCX_LAUNCH_CHECK();
    if (p.nsplit > 1) {
        const int64_t slots = pv.nblocks * ROWS;
        launch_after(os_reduce_kernel, dim3((unsigned)pv.nblocks, (unsigned)(p.out_pitch / 4)), ROWS, 0, stream, p.partial, p.perm, p.bias, slots, p.out_pitch,
                                                                                                     p.nsplit, p.fmt, p.out);
        PCX_LAUNCH_CHECK();
    }
    return PCX_OK;
}
