// Tap-segmented fixed-radius search in one enqueue and one host hand-over (sm_100a).
//
// Same result as pcx_radius_count + pcx_radius_fill with kernel_size > 0 -- the accepted
// (query i, point j) pairs grouped by kernel tap, inside a tap ordered by query, then by candidate
// cell, then by point index (internals/neighbors.py:469-838 followed by the stable sort by tap of
// layers/triplets.py:431-520) -- but built for latency instead of generality:
//
//   * points are binned by a HASH of their cell (side 2R), not by an injective key, so no extent
//     pass and no key-range hand-over precede the binning, and the bucket of a cell is found
//     with one load from a direct table.  Two cells may share a bucket: the foreign points are
//     ordinary candidates that fail the radius predicate (or the sample check), and the points of
//     the right cell keep their relative order (ascending index), so the output does not change.
//   * nothing needs the buckets themselves in any order, so the points are not sorted by key: they are
//     counted per bucket (an atomic addition a point), the buckets are given room as their first points come,
//     and a point goes as many places behind its bucket's start as the bucket has points of lower index.
//     The low three bits of the hash are the parities of the cell coordinates, so the eight cells
//     a query looks at always land in eight different buckets.
//   * a warp serves four queries: a lane looks up the run of one of their 32 cells (cells the ball does not reach are
//     left out) and lists it in shared memory in fours of candidates.  The list of the warp is worked off 32
//     candidates at a time, whatever query and cell they are of, so that no lane waits for a longer run or a query
//     with more candidates, four loads per lane in flight.  Accepted candidates are queued and their taps computed
//     32 at a time.  The first 64 accepted points of a query (128 for more than 27 taps) are kept with their taps, so
//     that the fill pass only places them; a warp with a longer list walks its runs again.  A block of 256 threads
//     serves 32 consecutive queries.
//   * the count pass leaves a per-block tap histogram; its prefix over blocks plus the tap
//     segment offsets give every block its write position in every tap, so the fill pass sorts the
//     pairs of a block by tap (a stable counting sort in shared memory, by counts per tap and query)
//     and writes them where they belong, neighbours next to each other: no sort of the edges, no per-query offsets.
//   * the fill pass writes into caller buffers of a given capacity; when the total exceeds it,
//     nothing is written and the call reports PCX_E_CAPACITY with the total, so that the caller
//     can retry with the exact size from the state kept in the workspace.
#include <cub/block/block_scan.cuh>

#include <algorithm>
#include <cfloat>
#include <cmath>

#include "geometry.cuh"

namespace pcx {
int device_status_address(unsigned int **d_status);   // status word of the bounded waits (sparse_tc.cu)
using namespace geo;
namespace {

constexpr int QPB = 32;           // queries per block
constexpr int THREADS = QPB * 8;  // one lane per (query, candidate cell)
constexpr int MAX_K3 = 128;       // taps this path handles (kernel_size 3 and 5)
constexpr int FOURS = 64;         // fours of candidates that a warp lists at a time
constexpr int SCAN_THREADS = 1024, SCAN_ITEMS = 4;
constexpr int DISTANCE = ~(PCX_RADIUS_WIDE_POINT_IDS | PCX_RADIUS_WIDE_QUERY_IDS | PCX_RADIUS_FULLEST_TAP);
constexpr int BIN_THREADS = 256;
constexpr int CROWDED = 1024;     // points of a bucket that are put in order by counting the lower ones
constexpr int MERGED = 32;        // ... by merging, where a bucket holds up to the MERGED-th part of all

struct TapsWs {
    uint32_t *keys;         // bucket of a point
    int32_t *arrival;       // ... and how many of the bucket's points were counted before it; points of crowded buckets in order
    int32_t *order;         // the points, bucket by bucket, as they arrived
    int32_t *crowded;       // buckets with more than CROWDED points
    float4 *sorted_pts;     // xyz + original index (bit pattern), bucket by bucket, ascending inside a bucket
    int2 *table;            // bucket -> (start, points); 0 points = empty
    int32_t *sorted_sample; // sample ids in bucket order
    int32_t *kept_point;    // Q x kept: the accepted points of a query, in output order
    uint8_t *kept_tap;      // ... and their taps
    uint32_t *counts;       // Q: accepted pairs
    uint32_t *block_hist;   // [tap][block] accepted pairs; exclusive prefix over blocks after the scan
    unsigned long long *tap_total;  // k3
    int64_t *seg;           // k3 + 1
    int64_t *ctrl;          // [0] total pairs, [1] a tap's count does not fit 31 bits, [2] taps scanned,
                            // [3] queries without a neighbour, [4] points given room, [5] crowded buckets,
                            // [6] pairs of the fullest tap
    int64_t buckets, nblocks;
};

// Accepted points of a query that the count pass keeps, at 5 bytes each: 320 bytes a query for kernels of up to 27 taps,
// 640 for larger ones (0.6 gigabytes of workspace at a million queries).  Rooms of 2 cm voxels have 6 to 25 and 16 to
// 75 neighbours there; the runs of a warp with a longer list are walked again.
int kept_per_query(int k3) { return k3 <= 27 ? 64 : 128; }

// Two to four buckets a point: a cell of side 2R holds several points, so that most buckets stay empty and few cells share one.
int bucket_bits(int64_t P) {
    int b = 1;
    while (((int64_t)1 << b) < P) ++b;
    b += 1;
    return b < 8 ? 8 : (b > 28 ? 28 : b);
}

size_t carve_taps(void *ws, int64_t P, int64_t Q, int k3, TapsWs *out) {
    Carver c(ws);
    TapsWs w;
    w.buckets = (int64_t)1 << bucket_bits(P);
    w.nblocks = (Q + QPB - 1) / QPB;
    w.ctrl = c.take<int64_t>(8);
    w.tap_total = c.take<unsigned long long>(k3);
    w.seg = c.take<int64_t>(k3 + 1);
    w.keys = c.take<uint32_t>(P);
    w.arrival = c.take<int32_t>(P);
    w.order = c.take<int32_t>(P);
    w.crowded = c.take<int32_t>(P / CROWDED + 1);
    w.sorted_pts = c.take<float4>(P);
    w.table = c.take<int2>(w.buckets);
    w.sorted_sample = c.take<int32_t>(P);
    w.kept_point = c.take<int32_t>(Q * kept_per_query(k3));
    w.kept_tap = c.take<uint8_t>(Q * kept_per_query(k3));
    w.counts = c.take<uint32_t>(Q);
    w.block_hist = c.take<uint32_t>(w.nblocks * k3);
    if (out) *out = w;
    return c.off;
}

__device__ __forceinline__ uint32_t cell_bucket(int b, int cx, int cy, int cz, uint32_t mask) {
    uint32_t h = (uint32_t)(cx >> 1) * 73856093u ^ (uint32_t)(cy >> 1) * 19349663u ^ (uint32_t)(cz >> 1) * 83492791u ^
                 (uint32_t)b * 0x9E3779B1u;
    h ^= h >> 16, h *= 0x85ebca6bu, h ^= h >> 13, h *= 0xc2b2ae35u, h ^= h >> 16;
    return ((h << 3) | ((uint32_t)(cx & 1) << 2) | ((uint32_t)(cy & 1) << 1) | (uint32_t)(cz & 1)) & mask;
}

// Binning, five kernels: every bucket empty; bucket of every point and its turn there; room for the buckets; the points
// bucket by bucket; ascending inside them.  The turn depends on which atomic addition came first, the result does not.
//
// Bound by launches and latency up to some 200 000 points, then by the random accesses.  Before, the keys went through a
// library's radix sort (two or three passes of 23 to 150 blocks, nine launches): 150 000 points 77 -> 23 us, a million 100 -> 52.
__global__ void taps_clear_kernel(int4 *table, int64_t pairs, int64_t *ctrl) {
    start_after_previous();
    const int64_t t0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, threads = (int64_t)gridDim.x * blockDim.x;
    for (int64_t t = t0; t < pairs; t += threads) table[t] = make_int4(0, 0, 0, 0);
    if (t0 < 8) ctrl[t0] = 0;
}

__global__ void __launch_bounds__(BIN_THREADS) taps_key_kernel(const float *__restrict__ pts, const int32_t *__restrict__ sample, int wide, int64_t P,
                                                               float inv, uint32_t mask, uint32_t *keys, int32_t *arrival, int2 *table) {
    start_after_previous();
    const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (p >= P) return;
    const uint32_t key = cell_bucket(sample ? sample[p << wide] : 0, cell_of(pts[3 * p], inv), cell_of(pts[3 * p + 1], inv),
                                     cell_of(pts[3 * p + 2], inv), mask);
    keys[p] = key;
    arrival[p] = atomicAdd(&table[key].y, 1);
}

// The first to arrive takes room for its bucket: buckets lie in the order of their points' blocks, an addition a block.
__global__ void __launch_bounds__(BIN_THREADS) taps_room_kernel(const uint32_t *__restrict__ keys, const int32_t *__restrict__ arrival, int64_t P,
                                                                int2 *table, int32_t *crowded, int64_t *ctrl) {
    start_after_previous();
    using Scan = cub::BlockScan<int32_t, BIN_THREADS>;
    __shared__ typename Scan::TempStorage tmp;
    __shared__ int32_t s_first;
    const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const bool takes = p < P && arrival[p] == 0;
    const uint32_t key = takes ? keys[p] : 0u;
    const int32_t points = takes ? table[key].y : 0;
    int32_t at, all;
    Scan(tmp).ExclusiveSum(points, at, all);
    if (threadIdx.x == 0) s_first = all ? (int32_t)atomicAdd((unsigned long long *)&ctrl[4], (unsigned long long)all) : 0;
    __syncthreads();
    if (takes) table[key].x = s_first + at;
    if (points > CROWDED) crowded[atomicAdd((unsigned long long *)&ctrl[5], 1ULL)] = (int32_t)key;
}

__global__ void __launch_bounds__(BIN_THREADS) taps_order_kernel(const uint32_t *__restrict__ keys, const int32_t *__restrict__ arrival, int64_t P,
                                                                 const int2 *__restrict__ table, int32_t *order) {
    start_after_previous();
    const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (p < P) order[table[keys[p]].x + arrival[p]] = (int32_t)p;
}

// `n` different numbers in ascending order, by a block: tiles of BIN_THREADS, then pairs of sorted runs, every number by a search in
// the other run of its pair.  From `from` to `to`, with `other` as scratch (n each).
__device__ __forceinline__ void merge_sort(const int32_t *from, int32_t *to, int32_t *other, int n) {
    static_assert(BIN_THREADS == 256, "tiles of four numbers for 64 loads");
    __shared__ int4 s_tile[BIN_THREADS / 4];
    int passes = 0;
    while ((BIN_THREADS << passes) < n) ++passes;
    int32_t *src = passes & 1 ? other : to, *dst = passes & 1 ? to : other;
    for (int first = 0; first < n; first += BIN_THREADS) {
        const int at = first + (int)threadIdx.x;
        const int32_t mine = at < n ? from[at] : INT_MAX;
        reinterpret_cast<int32_t *>(s_tile)[threadIdx.x] = mine;
        __syncthreads();
        int lower = 0;
#pragma unroll 8
        for (int q = 0; q < BIN_THREADS / 4; ++q) {
            const int4 v = s_tile[q];
            lower += (v.x < mine) + (v.y < mine) + (v.z < mine) + (v.w < mine);
        }
        if (at < n) src[first + lower] = mine;
        __syncthreads();
    }
    for (int width = BIN_THREADS; width < n; width *= 2) {
        for (int first = 0; first < n; first += 4 * BIN_THREADS) {
            int32_t mine[4];
            int other_run[4], len[4], lower[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int at = first + u * BIN_THREADS + (int)threadIdx.x;
                mine[u] = at < n ? src[at] : INT_MAX;
                other_run[u] = (at / width ^ 1) * width;
                len[u] = at < n ? max(0, min(width, n - other_run[u])) : 0;
                lower[u] = 0;
            }
            for (int step = width; step > 0; step >>= 1)   // four searches at a time
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (lower[u] + step <= len[u] && src[other_run[u] + lower[u] + step - 1] < mine[u]) lower[u] += step;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int at = first + u * BIN_THREADS + (int)threadIdx.x;
                if (at < n) dst[at / (2 * width) * (2 * width) + at % width + lower[u]] = mine[u];
            }
        }
        __syncthreads();
        int32_t *t = src;
        src = dst, dst = t;
    }
}

__global__ void __launch_bounds__(BIN_THREADS) taps_place_kernel(const float *__restrict__ pts, const int32_t *__restrict__ sample, int wide,
                                                                 const uint32_t *__restrict__ keys, const int32_t *__restrict__ order, int64_t P,
                                                                 const int2 *__restrict__ table, const int32_t *__restrict__ crowded,
                                                                 const int64_t *__restrict__ ctrl, int32_t *arrival, float4 *sorted_pts,
                                                                 int32_t *sorted_sample) {
    start_after_previous();
    auto put = [&](int32_t p, int32_t at) {
        sorted_pts[at] = make_float4(pts[3 * (int64_t)p], pts[3 * (int64_t)p + 1], pts[3 * (int64_t)p + 2], __int_as_float(p));
        if (sample) sorted_sample[at] = sample[(int64_t)p << wide];
    };
    const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (s < P) {
        const int32_t p = order[s];
        const int2 run = table[keys[p]];
        if (run.y <= CROWDED) {
            int32_t lower = 0;
#pragma unroll 4
            for (int t = 0; t < run.y; ++t) lower += order[run.x + t] < p;
            put(p, run.x + lower);
        }
    }
    // Crowded buckets, a block each, at most P / CROWDED of them.  Their points are merged; where a bucket has so many that that takes a
    // block longer, all points are gone through in order (at most MERGED such).  The bucket's part of `arrival`, of no use by
    // now, takes the result, its records the scratch.  This kernel, four million points in cells of 1100: 0.29 ms, and 16.4 where every
    // crowded bucket went through all points; a million in cells of 20 000: 0.72 and 1.06.
    const int64_t n = ctrl[5];
    for (int64_t x = blockIdx.x; x < n; x += gridDim.x) {
        using Scan = cub::BlockScan<int32_t, BIN_THREADS>;
        __shared__ typename Scan::TempStorage tmp;
        const uint32_t key = (uint32_t)crowded[x];
        const int2 run = table[key];
        if ((int64_t)run.y * MERGED <= P) {
            merge_sort(order + run.x, arrival + run.x, reinterpret_cast<int32_t *>(sorted_pts + run.x), run.y);
            for (int q = threadIdx.x; q < run.y; q += BIN_THREADS) put(arrival[run.x + q], run.x + q);
            __syncthreads();
            continue;
        }
        int32_t at = run.x;
        for (int64_t first = 0; first < P; first += 4 * BIN_THREADS) {
            const int64_t p = first + 4 * (int64_t)threadIdx.x;
            int32_t mine[4], before, all;
#pragma unroll
            for (int u = 0; u < 4; ++u) mine[u] = p + u < P && keys[p + u] == key;
            Scan(tmp).ExclusiveSum(mine[0] + mine[1] + mine[2] + mine[3], before, all);
            before += at, at += all;
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (mine[u]) put((int32_t)(p + u), before++);
            __syncthreads();
        }
    }
}

struct TapArgs {
    const float *queries;
    const int32_t *query_sample;   // words of the queries' ids, 1 << query_wide apart (the points' are in sorted_sample)
    int query_wide;
    const float4 *sorted_pts;
    const int2 *table;
    const int32_t *sorted_sample;   // null: no sample ids
    int32_t *kept_point;
    uint8_t *kept_tap;
    int kept;
    uint32_t *counts, *block_hist;
    int64_t *num_neighbors;
    const int64_t *seg, *ctrl;
    int64_t *ctrl_rw;
    int32_t *out_i, *out_j, *out_k;
    HandOver host;                  // fill pass: ctrl[0 .. 3] and the device status word
    const unsigned int *status;
    int64_t Q, nblocks, capacity;
    uint32_t mask;
    float r32, inv, g32, inv_g, s_max, cell, reach;   // cell: side of a cell; reach: square of the radius, with a margin
    int distance_type, variant, K, k3, use_s_max;
};

// The radius predicate without the square root where that is exact: sqrt is monotonic and correctly
// rounded, so sqrt(s) <= R holds exactly for the sums s up to the largest float whose root is <= R
// (s_max, found on the host).  The approximate-root variant and the Chebyshev distance keep the
// shared expression.
// FUSED: the usual case (Euclidean distance, sums of squares by fused multiply-adds) as a compile-time constant.
template <bool FUSED>
__device__ __forceinline__ bool accept_fast(const TapArgs &a, float qx, float qy, float qz, float4 p) {
    if (FUSED || a.use_s_max) {
        const float dx = __fsub_rn(qx, p.x), dy = __fsub_rn(qy, p.y), dz = __fsub_rn(qz, p.z);
        const float s = !FUSED && a.variant == 0 ? __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz))
                                       : __fmaf_rn(dz, dz, __fmaf_rn(dx, dx, __fmul_rn(dy, dy)));
        return s <= a.s_max;
    }
    float d;
    return radius_accept(qx, qy, qz, p, a.r32, a.distance_type, a.variant, &d);
}

// Candidate run of cell c (0 .. 7) of a query: (start, length).
__device__ __forceinline__ int2 run_of(const TapArgs &a, float qx, float qy, float qz, int b, int c) {
    const int cx = corner_of(qx, a.r32, a.inv) + ((c >> 2) & 1);
    const int cy = corner_of(qy, a.r32, a.inv) + ((c >> 1) & 1);
    const int cz = corner_of(qz, a.r32, a.inv) + (c & 1);
    // A cell farther from the query than the radius holds no neighbour.  A point of cell k lies at 2 R k or behind it up to
    // the rounding of its cell, some 3e-7 of the coordinate; the predicate's own rounding is some 1e-6 of R^2.  A cell number
    // at the end of the integers says no more than that the point lies there or beyond: such a cell is always looked at.
    if (a.distance_type == 0) {
        float far = 0.f;
        auto gap = [&](float v, int k) {
            far = fmaxf(far, fabsf((float)k));
            const float lo = (float)k * a.cell, slack = 1e-6f * (fabsf(v) + 2.f * a.cell);
            return fmaxf(fmaxf(lo - v, v - (lo + a.cell)) - slack, 0.f);
        };
        const float gx = gap(qx, cx), gy = gap(qy, cy), gz = gap(qz, cz);
        if (gx * gx + gy * gy + gz * gz > a.reach && far < 0x1p30f) return make_int2(0, 0);
    }
    return a.table[cell_bucket(b, cx, cy, cz, a.mask)];
}

struct Four {
    int first;        // sorted position of its first candidate
    uint32_t about;   // candidates (0 - 4) | query in the warp << 3
};

// The four queries of a warp; lane l looks after cell l & 7 of query l >> 3.
struct Queries {
    float4 *at;   // in shared memory: coordinates, sample id (bit pattern)
    int2 run;     // candidate run of this lane's cell: (start, length)
    __device__ __forceinline__ Queries(const TapArgs &a, int64_t q, int lane, float4 *room) : at(room), run(make_int2(0, 0)) {
        if (q < a.Q) {
            const float x = a.queries[3 * q], y = a.queries[3 * q + 1], z = a.queries[3 * q + 2];
            const int b = a.query_sample ? a.query_sample[q << a.query_wide] : 0;
            run = run_of(a, x, y, z, b, lane & 7);
            if ((lane & 7) == 0) at[lane >> 3] = make_float4(x, y, z, __int_as_float(b));
        }
        __syncwarp();
    }
};

// Walks the candidates of a warp: hit(which of this lane's four are accepted, the first one's sorted position, its query)
// once per 32 fours, lanes in the order of queries, cells and sorted positions.  `list`: room for FOURS entries.
template <bool FUSED, typename Hit>
__device__ __forceinline__ void walk(const TapArgs &a, const Queries &w, Four *list, int lane, Hit hit) {
    const int fours = (w.run.y + 3) >> 2;
    int upto = fours;   // fours of the cells up to this lane's
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += v;
    }
    const int total = __shfl_sync(0xffffffffu, upto, 31), before = upto - fours;
    for (int lo = 0; lo < total; lo += FOURS) {
        const int here = min(total - lo, FOURS);
        for (int k = max(lo - before, 0); k < fours && before + k < lo + FOURS; ++k)
            list[before + k - lo] = Four{w.run.x + 4 * k, (uint32_t)min(w.run.y - 4 * k, 4) | (uint32_t)(lane >> 3) << 3};
        __syncwarp();
#pragma unroll 1
        for (int t = 0; t < here; t += 32) {   // a four a lane
            const Four e = t + lane < here ? list[t + lane] : Four{0, 0u};
            const int query = (int)(e.about >> 3), size = (int)(e.about & 7u);
            const float4 q = w.at[query];
            float4 pt[4];
            bool ok[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) pt[u] = u < size ? a.sorted_pts[e.first + u] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int u = 0; u < 4; ++u) ok[u] = u < size && accept_fast<FUSED>(a, q.x, q.y, q.z, pt[u]);
            if (a.sorted_sample) {   // a foreign cell may share the bucket: its sample differs, or the distance does
                int smp[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) smp[u] = ok[u] ? a.sorted_sample[e.first + u] : 0;
#pragma unroll
                for (int u = 0; u < 4; ++u) ok[u] = ok[u] && smp[u] == __float_as_int(q.w);
            }
            hit(ok, e.first, query);
        }
        __syncwarp();
    }
}

// Accepted candidates of a warp, looked at 32 at a time in the order they came: use(there, sorted position, query, place
// among the accepted of its query).  The whole warp calls `use`.
struct Accepted {
    static constexpr int ROOM = 256;   // a power of two that 31 left over and four of each lane fit
    int2 *queue;                       // ROOM entries in shared memory: sorted position, query
    int head = 0, size = 0;
    int n[4] = {0, 0, 0, 0};
    __device__ __forceinline__ explicit Accepted(int2 *room) : queue(room) {}
    template <typename Use>
    __device__ __forceinline__ void take(int lane, int count, Use use) {
        __syncwarp();
        const bool there = lane < count;
        const int2 e = queue[(head + lane) & (ROOM - 1)];
        int place = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint32_t of = __ballot_sync(0xffffffffu, there && e.y == q);
            if (e.y == q) place = n[q] + __popc(of & ((1u << lane) - 1u));
            n[q] += __popc(of);
        }
        use(there, there ? e.x : 0, there ? e.y : 0, place);
        head += count, size -= count;
        __syncwarp();
    }
    template <typename Use>
    __device__ __forceinline__ void add(int lane, const bool (&ok)[4], int pos, int query, Use use) {
        const uint32_t below = (1u << lane) - 1u;
        int at = head + size;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const uint32_t all = __ballot_sync(0xffffffffu, ok[u]);
            at += __popc(all & below), size += __popc(all);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (ok[u]) queue[at++ & (ROOM - 1)] = make_int2(pos + u, query);
        while (size >= 32) take(lane, 32, use);
    }
    template <typename Use>
    __device__ __forceinline__ void finish(int lane, Use use) {
        if (size) take(lane, size, use);
    }
};

// Bound by issuing instructions (150 000 points with six neighbours: 745 a warp of four queries, issue slots 76 % busy).  One list of candidates a warp and
// a four a lane: 1 M points in eight rooms, 512 000 queries at a stride of two, 230 -> 170 us; 150 000 points 50 -> 35;
// four LiDAR sweeps 68 -> 53.  Eight lanes a query with a list of their own, and pieces of eight candidates: 207, 48, 74.
template <bool FUSED>
__global__ void __launch_bounds__(THREADS) taps_count_kernel(TapArgs a) {
    start_after_previous();
    __shared__ uint32_t s_hist[MAX_K3];
    __shared__ __align__(16) Four s_list[THREADS / 32][FOURS];
    __shared__ float4 s_query[THREADS / 32][4];
    __shared__ int2 s_queue[THREADS / 32][Accepted::ROOM];
    if (threadIdx.x < MAX_K3) s_hist[threadIdx.x] = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t q0 = (int64_t)blockIdx.x * QPB + warp * 4, q = q0 + (lane >> 3);
    const Queries queries(a, q, lane, s_query[warp]);
    Accepted accepted(s_queue[warp]);
    auto count = [&](bool there, int pos, int query, int place) {
        if (!there) return;
        const float4 p = a.sorted_pts[pos], c = queries.at[query];
        const int tap = tap_of_fast(c.x, c.y, c.z, p, a.g32, a.inv_g, a.K);
        atomicAdd(&s_hist[tap], 1u);
        if (place < a.kept) {
            const int64_t at = (q0 + query) * a.kept + place;
            a.kept_point[at] = __float_as_int(p.w), a.kept_tap[at] = (uint8_t)tap;
        }
    };
    walk<FUSED>(a, queries, s_list[warp], lane, [&](const bool (&ok)[4], int first, int query) { accepted.add(lane, ok, first, query, count); });
    accepted.finish(lane, count);
    if (q < a.Q && (lane & 7) == 0) {
        const int n = lane == 0 ? accepted.n[0] : lane == 8 ? accepted.n[1] : lane == 16 ? accepted.n[2] : accepted.n[3];
        a.counts[q] = n;
        a.num_neighbors[q] = n;
        if (n == 0) atomicAdd((unsigned long long *)&a.ctrl_rw[3], 1ULL);
    }
    __syncthreads();
    if ((int)threadIdx.x < a.k3) a.block_hist[(int64_t)threadIdx.x * a.nblocks + blockIdx.x] = s_hist[threadIdx.x];
}

// One block per tap: exclusive prefix of the tap's counts over the query blocks (in place) and
// the tap's total; the block that finishes last turns the totals into the tap segment offsets.
__global__ void __launch_bounds__(SCAN_THREADS) taps_colscan_kernel(uint32_t *block_hist, int64_t nblocks, int k3,
                                                                     unsigned long long *tap_total, int64_t *seg,
                                                                     int64_t *seg_out, int64_t *ctrl) {
    start_after_previous();
    using Scan = cub::BlockScan<uint32_t, SCAN_THREADS>;
    __shared__ typename Scan::TempStorage tmp;
    __shared__ int s_last;
    uint32_t *col = block_hist + (int64_t)blockIdx.x * nblocks;
    unsigned long long carry = 0;
    for (int64_t base = 0; base < nblocks; base += SCAN_THREADS * SCAN_ITEMS) {
        uint32_t v[SCAN_ITEMS], aggregate;
        const int64_t first = base + (int64_t)threadIdx.x * SCAN_ITEMS;
#pragma unroll
        for (int t = 0; t < SCAN_ITEMS; ++t) v[t] = first + t < nblocks ? col[first + t] : 0u;
        Scan(tmp).ExclusiveSum(v, v, aggregate);
#pragma unroll
        for (int t = 0; t < SCAN_ITEMS; ++t)
            if (first + t < nblocks) col[first + t] = (uint32_t)(carry + v[t]);
        carry += aggregate;
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        tap_total[blockIdx.x] = carry;
        if (carry > 0x7fffffffULL) ctrl[1] = 1;
        __threadfence();
        s_last = atomicAdd((unsigned long long *)&ctrl[2], 1ULL) == (unsigned long long)(k3 - 1);
    }
    __syncthreads();
    if (s_last && threadIdx.x < 32) {   // k3 <= 128: four taps per lane, prefix over the warp
        __threadfence();
        const int t0 = threadIdx.x * 4;
        unsigned long long v[4], sum = 0;
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = t0 + u < k3 ? __ldcg(tap_total + t0 + u) : 0ULL, sum += v[u];
        unsigned long long incl = sum, fullest = max(max(v[0], v[1]), max(v[2], v[3]));
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long up = __shfl_up_sync(0xffffffffu, incl, o);
            if ((int)threadIdx.x >= o) incl += up;
            fullest = max(fullest, __shfl_xor_sync(0xffffffffu, fullest, o));
        }
        unsigned long long run = incl - sum;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (t0 + u <= k3) seg[t0 + u] = (int64_t)run, seg_out[t0 + u] = (int64_t)run;
            run += v[u];
        }
        if (threadIdx.x == 31) ctrl[0] = (int64_t)incl, ctrl[6] = (int64_t)fullest, seg[k3] = (int64_t)incl, seg_out[k3] = (int64_t)incl;
    }
}

// Kept pairs are counted by shared-memory additions in any order and put in order within their few neighbours of the same
// query and tap when they are written; matching lanes by tap took 141 us instead of 111 below.
// Before pairs were sorted in shared memory and written side by side: 512 000 queries with 13 neighbours 175 -> 112 us,
// 150 000 points 37 -> 26, LiDAR 67 -> 38 (with 64 instead of 48 kept pairs; 65 with 48: one query in ninety has more,
// and its warp keeps the block waiting), 125 taps, 100 000 queries with 41 152 -> 110.
// Queries with more pairs than are kept: 40 000 with 145 of them 766 us, with 374 4.2 ms (125 taps: 637, 3.3 ms); 1389 and
// 8.5 ms (901, 5.4 ms) when every warp walked its runs again in every round of the block.
template <bool FUSED, int REC_MAX>   // pairs staged per round
__global__ void __launch_bounds__(THREADS, REC_MAX > 1024 ? 4 : 5) taps_fill_kernel(TapArgs a) {
    start_after_previous();
    constexpr int WARPS = THREADS / 32;
    struct Walk {
        Four list[WARPS][FOURS];
        float4 query[WARPS][4];
        int2 queue[WARPS][Accepted::ROOM];
    };
    // pairs of a round as they come (point, tap | query << 8 | place among the query's pairs << 16), then by tap.
    // Warps that walk their runs again do so before the pairs are sorted.
    constexpr uint32_t UNORDERED = 1u << 31;
    __shared__ uint2 s_rec[REC_MAX];
    __shared__ uint16_t s_nth[REC_MAX];                     // where a pair goes among those of its query and tap
    __shared__ union {
        uint2 sorted[REC_MAX];
        Walk walk;
    } s_u;
    extern __shared__ __align__(16) uint16_t s_cnt[];       // [tap][query]: pairs, then those of the queries before (32-bit words, too)
    __shared__ uint32_t s_base[MAX_K3];                     // next write position of each tap for this block
    __shared__ uint32_t s_start[MAX_K3], s_total[MAX_K3];   // first place of each tap among the sorted, its pairs in this round
    if (blockIdx.x == 0 && threadIdx.x == 0 && a.host.words) {   // all there is to hand over is known before this pass
        const int64_t words[4] = {a.ctrl[0], a.ctrl[1], a.ctrl[2], a.ctrl[3]}, fullest = a.ctrl[6];   // (loads before stores: one latency)
        const unsigned int status = *(const volatile unsigned int *)a.status;
        for (int n = 0; n < 4; ++n) a.host.put(n, words[n]);
        a.host.put(4, status), a.host.put(5, fullest);
        a.host.done();
    }
    const bool fits = a.ctrl[0] <= a.capacity && !a.ctrl[1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int c = threadIdx.x & 7, ql = threadIdx.x >> 3;
    const int64_t q0 = (int64_t)blockIdx.x * QPB, q = q0 + ql;
    if ((int)threadIdx.x < a.k3)
        s_base[threadIdx.x] = (uint32_t)a.seg[threadIdx.x] + a.block_hist[(int64_t)threadIdx.x * a.nblocks + blockIdx.x];
    // pairs of the block's queries and where each query's begin: every warp for itself, a query a lane
    const uint32_t n_lane = q0 + lane < a.Q ? a.counts[q0 + lane] : 0u;
    if (!fits) return;   // (the counts were on their way meanwhile)
    uint32_t upto = n_lane;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += v;
    }
    const uint32_t block_total = __shfl_sync(0xffffffffu, upto, 31);
    const uint32_t nq = __shfl_sync(0xffffffffu, n_lane, ql), q_off = __shfl_sync(0xffffffffu, upto, ql) - nq;
    const bool kept = __all_sync(0xffffffffu, nq <= (uint32_t)a.kept);   // all accepted points of the warp's queries were kept
    const uint32_t warp_first = __shfl_sync(0xffffffffu, q_off, 0), warp_end = __shfl_sync(0xffffffffu, q_off + nq, 31);
    for (uint32_t lo = 0; lo < block_total; lo += REC_MAX) {
        const uint32_t cnt = min((uint32_t)REC_MAX, block_total - lo);
        for (int t = threadIdx.x; t < a.k3 * QPB / 2; t += THREADS) reinterpret_cast<uint32_t *>(s_cnt)[t] = 0u;
        __syncthreads();
        // A pair of query x of the block: its place among that query's pairs of the same tap, and into s_rec.  The whole warp
        // calls; pairs of a query come in order, the lanes' queries do not fall.
        auto place = [&](bool there, uint32_t pos, int x, int point, int tap) {
            there = there && pos - lo < (uint32_t)REC_MAX;
            const uint32_t same = __match_any_sync(0xffffffffu, there ? tap | x << 8 : 0x10000 + lane);
            uint16_t *count = s_cnt + tap * QPB + x;
            const uint32_t before = there ? *count : 0u, lower = same & ((1u << lane) - 1u);
            __syncwarp();
            if (there) {
                const uint32_t nth = before + __popc(lower);
                s_rec[pos - lo] = make_uint2((uint32_t)point, (uint32_t)tap | (uint32_t)x << 8 | nth << 16), s_nth[pos - lo] = (uint16_t)nth;
                if (!lower) *count = (uint16_t)(before + __popc(same));
            }
            __syncwarp();
        };
        if (kept) {
            // Counted in any order: what is stored is a pair's place in its query's list, and the few pairs of a query and
            // tap are put in order when they are written.
            const uint32_t most = __reduce_max_sync(0xffffffffu, nq);
            for (uint32_t e0 = c; e0 < most; e0 += 32) {
                uint32_t tap[4], point[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int64_t at = q * a.kept + e0 + 8 * u;
                    if (e0 + 8 * u < nq) tap[u] = a.kept_tap[at], point[u] = (uint32_t)a.kept_point[at];
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const uint32_t e = e0 + 8 * u, pos = q_off + e - lo;
                    if (e >= nq || pos >= (uint32_t)REC_MAX) continue;
                    const uint32_t shift = (ql & 1) * 16;   // (two queries of one warp share a word)
                    const uint32_t nth = atomicAdd(reinterpret_cast<uint32_t *>(s_cnt) + (tap[u] * QPB + ql) / 2, 1u << shift) >> shift & 0xffffu;
                    s_rec[pos] = make_uint2(point[u], tap[u] | (uint32_t)ql << 8 | e << 16 | UNORDERED);
                    s_nth[pos] = (uint16_t)nth;
                }
            }
        } else if (warp_first < lo + REC_MAX && warp_end > lo) {   // only in the rounds that hold pairs of the warp's queries
            const Queries queries(a, q, lane, s_u.walk.query[warp]);
            Accepted accepted(s_u.walk.queue[warp]);
            auto put = [&](bool there, int pos, int query, int nth) {
                const float4 p = a.sorted_pts[pos], at = queries.at[query];
                const int tap = there ? tap_of_fast(at.x, at.y, at.z, p, a.g32, a.inv_g, a.K) : 0;
                place(there, __shfl_sync(0xffffffffu, q_off, query * 8) + (uint32_t)nth, warp * 4 + query, __float_as_int(p.w), tap);
            };
            walk<FUSED>(a, queries, s_u.walk.list[warp], lane, [&](const bool (&ok)[4], int first, int query) { accepted.add(lane, ok, first, query, put); });
            accepted.finish(lane, put);
        }
        __syncthreads();
        // a warp per tap: the pairs of the queries before each query
        for (int tap = warp; tap < a.k3; tap += WARPS) {
            const uint32_t v = s_cnt[tap * QPB + lane];
            uint32_t incl = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t up = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += up;
            }
            s_cnt[tap * QPB + lane] = (uint16_t)(incl - v);
            if (lane == 31) s_total[tap] = incl;
        }
        __syncthreads();
        if (warp == 0) {   // k3 <= 128: four taps per lane
            uint32_t v[4], sum = 0;
#pragma unroll
            for (int u = 0; u < 4; ++u) v[u] = lane * 4 + u < a.k3 ? s_total[lane * 4 + u] : 0u, sum += v[u];
            uint32_t incl = sum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t up = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += up;
            }
            uint32_t first = incl - sum;
#pragma unroll
            for (int u = 0; u < 4; ++u) s_start[lane * 4 + u] = first, first += v[u];
        }
        __syncthreads();
        for (uint32_t x = threadIdx.x; x < cnt; x += THREADS) {
            const uint2 rec = s_rec[x];
            const uint32_t tap = rec.y & 0xffu;
            s_u.sorted[s_start[tap] + s_cnt[tap * QPB + ((rec.y >> 8) & 0xffu)] + s_nth[x]] = rec;
        }
        __syncthreads();
        for (uint32_t x = threadIdx.x; x < cnt; x += THREADS) {
            const uint2 rec = s_u.sorted[x];
            const uint32_t tap = rec.y & 0xffu, of = (rec.y >> 8) & 0xffu, first = s_cnt[tap * QPB + of];
            uint32_t place = x - s_start[tap];
            if (rec.y & UNORDERED) {
                place = first;
                const uint32_t end = of + 1 < QPB ? s_cnt[tap * QPB + of + 1] : s_total[tap];
                if (end - first > 1)
                    for (uint32_t y = first; y < end; ++y) place += s_u.sorted[s_start[tap] + y].y < rec.y;   // (they differ in the list place alone)
            }
            const uint32_t pos = s_base[tap] + place;
            a.out_i[pos] = (int32_t)(q0 + (int)((rec.y >> 8) & 0xffu));
            a.out_j[pos] = (int32_t)rec.x;
            if (a.out_k) a.out_k[pos] = (int32_t)tap;
        }
        if (lo + REC_MAX >= block_total) break;
        __syncthreads();
        if ((int)threadIdx.x < a.k3) s_base[threadIdx.x] += s_total[threadIdx.x];
    }
}

int check_common(int64_t P, int64_t Q, double radius, int distance_type, int kernel_size, double grid,
                 const char *who) {
    if (P <= 0 || Q <= 0) PCX_FAIL(PCX_E_ARG, "%s: P and Q must be positive (got %lld, %lld)", who, (long long)P, (long long)Q);
    if (P > INT32_MAX || Q > INT32_MAX) PCX_FAIL(PCX_E_UNSUPPORTED, "%s: more than 2^31-1 rows", who);
    if (!(radius > 0)) PCX_FAIL(PCX_E_ARG, "radius must be positive; got %g", radius);
    distance_type &= DISTANCE;
    if (distance_type != 0 && distance_type != 1) PCX_FAIL(PCX_E_ARG, "distance_type must be 0 (ball) or 1 (chebyshev)");
    if (kernel_size <= 0 || kernel_size % 2 == 0) PCX_FAIL(PCX_E_ARG, "kernel_size must be a positive odd integer; got %d", kernel_size);
    if (kernel_size * kernel_size * kernel_size > MAX_K3)
        PCX_FAIL(PCX_E_UNSUPPORTED, "%s: kernel_size %d has more than %d taps; use pcx_radius_count / pcx_radius_fill", who, kernel_size, MAX_K3);
    if (!(grid > 0)) PCX_FAIL(PCX_E_ARG, "kernel_grid_size must be positive; got %g", grid);
    return PCX_OK;
}

TapArgs make_args(const TapsWs &w, const float *queries, const int32_t *point_sample, const int32_t *query_sample,
                  int64_t Q, double radius, int distance_type, int kernel_size, double grid) {
    TapArgs a = {};
    a.queries = queries, a.query_sample = query_sample, a.query_wide = distance_type & PCX_RADIUS_WIDE_QUERY_IDS ? 1 : 0;
    distance_type &= DISTANCE;
    a.sorted_pts = w.sorted_pts, a.table = w.table, a.kept_point = w.kept_point, a.kept_tap = w.kept_tap;
    a.sorted_sample = point_sample ? w.sorted_sample : nullptr, a.kept = kept_per_query(kernel_size * kernel_size * kernel_size);
    a.counts = w.counts, a.block_hist = w.block_hist, a.seg = w.seg, a.ctrl = w.ctrl, a.ctrl_rw = w.ctrl;
    a.Q = Q, a.nblocks = w.nblocks, a.mask = (uint32_t)(w.buckets - 1);
    a.r32 = (float)radius, a.inv = (float)(1.0 / (2.0 * radius)), a.g32 = (float)grid;
    a.inv_g = 1.0f / a.g32;
    a.cell = (float)(2.0 * radius), a.reach = a.r32 * a.r32 * 1.0001f;
    a.distance_type = distance_type, a.variant = radius_variant(), a.K = kernel_size;
    a.k3 = kernel_size * kernel_size * kernel_size;
    a.use_s_max = distance_type == 0 && a.variant != 2;
    if (a.use_s_max) {   // largest float whose correctly rounded root is <= r32; r32 * r32 is within a few ulp of it
        float s = a.r32 * a.r32;
        if (!(s <= FLT_MAX)) s = FLT_MAX;
        for (int it = 0; it < 64 && s > 0.f && sqrtf(s) > a.r32; ++it) s = nextafterf(s, 0.f);
        for (int it = 0; it < 64 && s < FLT_MAX && sqrtf(nextafterf(s, FLT_MAX)) <= a.r32; ++it) s = nextafterf(s, FLT_MAX);
        a.use_s_max = sqrtf(s) <= a.r32 && (s == FLT_MAX || sqrtf(nextafterf(s, FLT_MAX)) > a.r32);
        a.s_max = s;
    }
    return a;
}

bool fused(const TapArgs &a) { return a.use_s_max && a.variant == 1; }

// ctrl[0 .. 3] and the device status word, in one wait
// Words 0 to 3 and 6 of ctrl and the device status word, as the fill pass stores them.
int read_ctrl(const TapsWs &w, int64_t *h, cudaStream_t stream) {
    unsigned int *d_status = nullptr;
    if (int rc = device_status_address(&d_status)) return rc;
    h[4] = 0;
    PCX_CUDA(cudaMemcpyAsync(h + 6, w.ctrl, 7 * sizeof(int64_t), cudaMemcpyDeviceToHost, stream));
    PCX_CUDA(cudaMemcpyAsync(h + 4, d_status, sizeof(unsigned int), cudaMemcpyDeviceToHost, stream));
    PCX_CUDA(cudaStreamSynchronize(stream));
    std::copy(h + 6, h + 10, h);
    h[5] = h[12];
    return PCX_OK;
}

}  // namespace
}  // namespace pcx

using namespace pcx;

extern "C" {

int pcx_radius_taps_supported(int kernel_size) {
    return kernel_size > 0 && kernel_size % 2 == 1 && kernel_size * kernel_size * kernel_size <= MAX_K3;
}

size_t pcx_radius_taps_workspace_bytes(int64_t P, int64_t Q, int kernel_size) {
    if (P < 0 || Q < 0 || !pcx_radius_taps_supported(kernel_size)) return 0;
    return carve_taps(nullptr, P, Q, kernel_size * kernel_size * kernel_size, nullptr);
}

int pcx_radius_taps_count(const float *d_points, const float *d_queries, const int32_t *d_point_sample,
                          const int32_t *d_query_sample, int64_t P, int64_t Q, double radius, int distance_type,
                          int kernel_size, double kernel_grid_size, int64_t *d_num_neighbors, int64_t *d_seg_offs,
                          void *d_ws, size_t ws_bytes, void *stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    if (int rc = check_common(P, Q, radius, distance_type, kernel_size, kernel_grid_size, "pcx_radius_taps_count")) return rc;
    if (!d_points || !d_queries || !d_num_neighbors || !d_seg_offs || !d_ws) PCX_FAIL(PCX_E_ARG, "pcx_radius_taps_count: null pointer");
    if ((d_point_sample == nullptr) != (d_query_sample == nullptr)) PCX_FAIL(PCX_E_ARG, "pcx_radius_taps_count: sample ids must be given for both sets or neither");
    const int k3 = kernel_size * kernel_size * kernel_size;
    TapsWs w;
    const size_t need = carve_taps(d_ws, P, Q, k3, &w);
    if (ws_bytes < need) PCX_FAIL(PCX_E_CAPACITY, "pcx_radius_taps_count: workspace %zu < %zu bytes", ws_bytes, need);
    if ((uintptr_t)d_ws % 256) PCX_FAIL(PCX_E_ALIGN, "pcx_radius_taps_count: workspace must be 256-byte aligned");
    const int wide = distance_type & PCX_RADIUS_WIDE_POINT_IDS ? 1 : 0;
    const float inv = (float)(1.0 / (2.0 * radius));
    const uint32_t mask = (uint32_t)(w.buckets - 1);
    const unsigned pblocks = (unsigned)((P + BIN_THREADS - 1) / BIN_THREADS);
    const int64_t pairs = w.buckets / 2;
    launch_after(taps_clear_kernel, (unsigned)std::min<int64_t>((pairs + BIN_THREADS - 1) / BIN_THREADS, 8 * num_sms()), BIN_THREADS, 0, stream,
                 reinterpret_cast<int4 *>(w.table), pairs, w.ctrl);
    PCX_LAUNCH_CHECK();
    launch_after(taps_key_kernel, pblocks, BIN_THREADS, 0, stream, d_points, d_point_sample, wide, P, inv, mask, w.keys, w.arrival, w.table);
    PCX_LAUNCH_CHECK();
    launch_after(taps_room_kernel, pblocks, BIN_THREADS, 0, stream, w.keys, w.arrival, P, w.table, w.crowded, w.ctrl);
    PCX_LAUNCH_CHECK();
    launch_after(taps_order_kernel, pblocks, BIN_THREADS, 0, stream, w.keys, w.arrival, P, w.table, w.order);
    PCX_LAUNCH_CHECK();
    launch_after(taps_place_kernel, pblocks, BIN_THREADS, 0, stream, d_points, d_point_sample, wide, w.keys, w.order, P, w.table, w.crowded, w.ctrl,
                 w.arrival, w.sorted_pts, w.sorted_sample);
    PCX_LAUNCH_CHECK();
    TapArgs a = make_args(w, d_queries, d_point_sample, d_query_sample, Q, radius, distance_type, kernel_size, kernel_grid_size);
    a.num_neighbors = d_num_neighbors;
    prof_begin("taps_count_kernel", stream);
    launch_after((fused(a) ? taps_count_kernel<true> : taps_count_kernel<false>), (unsigned)w.nblocks, THREADS, 0, stream, a);
    prof_end(stream);
    PCX_LAUNCH_CHECK();
    launch_after(taps_colscan_kernel, k3, SCAN_THREADS, 0, stream, w.block_hist, w.nblocks, k3, w.tap_total, w.seg, d_seg_offs, w.ctrl);
    PCX_LAUNCH_CHECK();
    return PCX_OK;
}

int pcx_radius_taps_total(int64_t P, int64_t Q, int kernel_size, int64_t *h_total, void *d_ws, size_t ws_bytes,
                          void *stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    if (!h_total || !d_ws || P <= 0 || Q <= 0 || !pcx_radius_taps_supported(kernel_size)) PCX_FAIL(PCX_E_ARG, "pcx_radius_taps_total: bad arguments");
    TapsWs w;
    if (ws_bytes < carve_taps(d_ws, P, Q, kernel_size * kernel_size * kernel_size, &w)) PCX_FAIL(PCX_E_CAPACITY, "pcx_radius_taps_total: workspace too small");
    int64_t *h = handover_words();
    if (int rc = read_ctrl(w, h, stream)) return rc;
    h_total[0] = h[0], h_total[1] = h[3], h_total[2] = h[4];
    if (h[1] || h[0] > INT32_MAX) PCX_FAIL(PCX_E_UNSUPPORTED, "prepared kernel-segment output currently requires fewer than 2^31 edges; got %lld", (long long)h[0]);
    return PCX_OK;
}

int pcx_radius_taps_fill(const float *d_queries, const int32_t *d_point_sample, const int32_t *d_query_sample,
                         int64_t P, int64_t Q, double radius, int distance_type, int kernel_size,
                         double kernel_grid_size, int64_t capacity, int32_t *d_out_i, int32_t *d_out_j,
                         int32_t *d_out_k, int64_t *h_total, void *d_ws, size_t ws_bytes, void *stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    if (int rc = check_common(P, Q, radius, distance_type, kernel_size, kernel_grid_size, "pcx_radius_taps_fill")) return rc;
    if (!d_queries || !h_total || !d_ws || capacity < 0) PCX_FAIL(PCX_E_ARG, "pcx_radius_taps_fill: bad arguments");
    if (capacity > 0 && (!d_out_i || !d_out_j)) PCX_FAIL(PCX_E_ARG, "pcx_radius_taps_fill: d_out_i and d_out_j are required");
    if ((d_point_sample == nullptr) != (d_query_sample == nullptr)) PCX_FAIL(PCX_E_ARG, "pcx_radius_taps_fill: sample ids must be given for both sets or neither");
    const int k3 = kernel_size * kernel_size * kernel_size;
    TapsWs w;
    const size_t need = carve_taps(d_ws, P, Q, k3, &w);
    if (ws_bytes < need) PCX_FAIL(PCX_E_CAPACITY, "pcx_radius_taps_fill: workspace %zu < %zu bytes", ws_bytes, need);
    TapArgs a = make_args(w, d_queries, d_point_sample, d_query_sample, Q, radius, distance_type, kernel_size, kernel_grid_size);
    a.out_i = d_out_i, a.out_j = d_out_j, a.out_k = d_out_k, a.capacity = capacity;
    int64_t *h = handover_words();
    if (capacity > 0) {
        unsigned int *status = nullptr;
        if (int rc = device_status_address(&status)) return rc;
        a.host = new_hand_over(), a.status = status;
        prof_begin("taps_fill_kernel", stream);
        const auto kernel = k3 <= 27 ? (fused(a) ? taps_fill_kernel<true, 1024> : taps_fill_kernel<false, 1024>)
                                     : (fused(a) ? taps_fill_kernel<true, 1536> : taps_fill_kernel<false, 1536>);
        launch_after(kernel, (unsigned)w.nblocks, THREADS, (size_t)k3 * QPB * sizeof(uint16_t), stream, a);
        prof_end(stream);
        PCX_LAUNCH_CHECK();
    }
    if (int rc = a.host.words ? wait_for_hand_over(a.host, stream) : read_ctrl(w, h, stream)) return rc;
    h_total[0] = h[0], h_total[1] = h[3], h_total[2] = h[4];
    if (distance_type & PCX_RADIUS_FULLEST_TAP) h_total[3] = h[5];
    if (h[1] || h[0] > INT32_MAX) PCX_FAIL(PCX_E_UNSUPPORTED, "prepared kernel-segment output currently requires fewer than 2^31 edges; got %lld", (long long)h[0]);
    if (h[0] > capacity) PCX_FAIL(PCX_E_CAPACITY, "pcx_radius_taps_fill: %lld pairs do not fit the capacity of %lld; nothing was written", (long long)h[0], (long long)capacity);
    return PCX_OK;
}

}  // extern "C"
