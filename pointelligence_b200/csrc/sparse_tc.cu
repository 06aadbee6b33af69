// Tensor-core engine for MVMR that scatters its rows, on sm_100a (tcgen05 + TMEM).
//
// The kernel is persistent: every CTA owns a contiguous range of chunks of
// 128 tap-sorted triplets.  A chunk is gathered row by row with 16-byte
// cp.async copies straight into the 128-byte-swizzled shared-memory layout the
// tensor core reads, so no separate staging pass exists:
//
//   smem tile  = [64-channel block][row][128 bytes], 16-byte pieces XOR-swizzled
//                with (row & 7)  (the SWIZZLE_128B canonical layout)
//
//   MVMR   D[128 triplets x N] = A[128 x Kc] * B[Kc x N]
//          A = gathered feature rows   (K-major: a row is contiguous along Kc)
//          B = W[tap] exactly as stored, (C, M) row-major: read MN-major in the
//              forward (its rows are the contraction index) and K-major in the
//              input gradient (its rows are the output channels)
//          one A tile per CTA; latency is hidden by the other CTAs resident on the
//          SM (5-6 at C = 64), so shared memory per CTA is kept as small as possible
//          epilogue, rows of 64 floats: TMEM -> registers -> a parking area in shared
//          memory (16 rows per warp at a time, aliased with the A tile) -> one bulk
//          reduction (cp.reduce.async.bulk add.f32) per output row;
//          other widths: TMEM -> registers -> red.global.add.v2.f32
//
// Measured on B200, the kernel is bound by latency, not by a pipe: at C = 64 the
// L2 runs at about a third of its throughput and DRAM at a tenth, and every step that
// put more CTAs on an SM (3 -> 5 -> 6) shortened the kernel (78 -> 64 -> 62 us).
//
// One thread issues tcgen05.mma; completion is signalled with tcgen05.commit on
// an mbarrier.  Every wait is bounded (one second): after the limit the kernel raises a flag
// in the status word, frees its TMEM and returns.
#include "sparse_kernels.cuh"
#include "tcgen05.cuh"

namespace pcx {

__device__ unsigned int g_device_status = 0;

namespace {

constexpr int CH = 128;            // triplets per chunk
constexpr int BLK_BYTES = CH * 128; // one 64-channel block of a 128-row tile

using namespace tc;

using ChunkCursor = ChunkCursorT<CH>;

constexpr int MAX_PARTS = 64;        // (group, part, part) combinations of one launch
constexpr int MAX_TAPS_SMEM = 1024;  // taps whose chunk table fits the shared-memory copy

// Gather `rows` rows of `width` 2-byte channels into a swizzled tile; the row indices (rows lie
// `pitch` elements apart) were staged in shared memory beforehand so that the copy loop issues
// cp.async back to back.
__device__ __forceinline__ void gather_tile(uint32_t tile, const uint16_t *__restrict__ src,
                                            const int32_t *s_idx, int rows, int width, int64_t pitch, int tid, int nthreads) {
    const int cpr = width >> 3;  // 16-byte pieces per row
    const uint32_t pitch_bytes = (uint32_t)pitch * 2u;
    if ((cpr & (cpr - 1)) == 0) {
        // power-of-two row length: a thread keeps its 16-byte column and walks down the rows
        const int sh = __ffs(cpr) - 1;
        const int ch = tid & (cpr - 1), rpp = nthreads >> sh;
        const uint32_t dcol = tile + (uint32_t)(ch >> 3) * BLK_BYTES;
        const char *scol = reinterpret_cast<const char *>(src + ch * 8);
#pragma unroll 4
        for (int r = tid >> sh; r < rows; r += rpp)
            cp_async16(dcol + (uint32_t)r * 128 + (uint32_t)(((ch ^ r) & 7) << 4), scol + (uint64_t)(uint32_t)s_idx[r] * pitch_bytes);
        return;
    }
    // (keeping a thread on one column with a single division up front was tried for these row
    // lengths and for the loop above: 96 channels unchanged, 128 and 256 channels 13 % slower)
    for (int e = tid; e < rows * cpr; e += nthreads) {
        const int r = e / cpr, ch = e - r * cpr;
        const uint32_t dst = tile + (uint32_t)(ch >> 3) * BLK_BYTES + (uint32_t)r * 128 + (uint32_t)(((ch & 7) ^ (r & 7)) << 4);
        cp_async16(dst, reinterpret_cast<const char *>(src + ch * 8) + (uint64_t)(uint32_t)s_idx[r] * pitch_bytes);
    }
}

// Scatter through the copy engine: every accumulator row is parked in shared
// memory and handed to one bulk reduction (fp32 add into global memory), so the
// scatter neither occupies the load/store pipeline nor needs one instruction
// per 32-byte piece.
__device__ __forceinline__ void bulk_reduce_add_f32(float *gdst, uint32_t ssrc, uint32_t bytes) {
    asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f32 [%0], [%1], %2;"
                 ::"l"(gdst), "r"(ssrc), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }


__device__ __forceinline__ uint32_t pack_pair(float a, float b, int fmt) {
    if (fmt) {
        __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
        return *reinterpret_cast<uint32_t *>(&h);
    }
    __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<uint32_t *>(&h);
}

__device__ __forceinline__ float unpack_one(uint16_t v, int fmt) {
    return fmt ? __bfloat162float(__ushort_as_bfloat16(v)) : __half2float(__ushort_as_half(v));
}

// Wide and grouped layers run as parts of at most 256 x 256 channels, every part of a width of the same size, a
// multiple of 16.  blockIdx.y counts (group, part of the output row, link of the contraction): a block takes
// p.chain parts of a contraction one after another, each into tensor memory columns of its own, and reduces their
// sum.  (As blocks of their own they meet in the accumulator, with as many reductions more: fp16, 31 852 triplets of
// 512 x 512 channels 75 us, chained 65; 408 976 triplets 726 and 676; 2048 to 128 channels 895 and 817.)  One column
// range for all of them would need no additions (676 would be 657), but the tensor cores drop bits at each step of a
// chain: rows of 2048 channels of one sign came out with ten times the error against fp64, 1.2e-5.

struct MvmrTcParams {
    const uint16_t *weight;  // (K, C, M) as stored
    const uint16_t *feat;
    const int32_t *gather, *scatter;
    const int64_t *seg;
    float *acc;
    uint16_t *out;           // MODE 2: the output rows themselves (every row occurs in exactly one triplet)
    const uint16_t *bias;    // MODE 2: added before the rounding (null: none); the other modes start from it
    int reverse;             // tap k uses weight K-1-k
    OnlyIf only_if;
    int64_t in_pitch, out_pitch, w_pitch, w_tap;   // rows of features / output / one tap's weight, elements of one tap's weight
    int out_parts, in_parts, chain;                // C, M below: the part's; contraction parts a block takes
    int K, C, M, transpose, fmt, nbuf, slab;  // slab: columns parked per bulk reduction (32 or 64)
    int prow_log2;                            // a warp parks 2^prow_log2 rows at a time (8, 16 or 32)
    uint32_t park_bytes;                      // size of the parking area (the chunk table follows it)
    int alias;                                // parking area shares the feature tile's memory
    uint32_t ncols, acc_cols;                 // tensor memory columns of a block, of one part
};

// One A tile by default: the next gather is issued as soon as the multiply has finished (or,
// when the parking area aliases the tile, once the reductions have read it) and the other
// CTAs resident on the SM cover its latency; the indices of chunk c+2 are already on their
// way into registers.  nbuf == 2 keeps a ring of two A tiles instead.
// MODE 0: sums leave through two-float reductions from registers; 1: one bulk reduction per row
// (rows of 64 floats); 2: plain 16-byte stores of the rounded row, for rulebooks in which every output
// row occurs in exactly one triplet (fan-in 1: nothing to accumulate, clear or round afterwards).
// NT: 128 threads, or 256 where shared memory leaves room for few CTAs (mode 0): with four warps an SM a 256 x 256 part
// waited for its own copies and reductions (31 852 triplets of 512 x 512 fp16 channels 69 us, with eight warps 65;
// 256 x 256 channels, 408 976 triplets 212 and 201).
template <int MODE, int NT, bool CHAINED, bool AGAIN>
__global__ void __launch_bounds__(NT, NT == 256 ? 1 : 0) mvmr_tc_kernel(MvmrTcParams p) {
    constexpr bool BULK = MODE == 1;
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t s_bar;
    __shared__ uint32_t s_tmem;
    __shared__ __align__(16) int32_t s_scatter[2][CH];
    __shared__ int32_t s_gather[2][CH];
    __shared__ int32_t s_warp_sums[NT / 32];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int inw = p.transpose ? p.M : p.C, outw = p.transpose ? p.C : p.M;
    int parts;   // of the contraction, in this block
    {
        const int links = p.in_parts / p.chain, ip = (int)blockIdx.y % links * p.chain,
                  op = (int)blockIdx.y / links % p.out_parts, g = (int)blockIdx.y / (links * p.out_parts);
        parts = CHAINED ? p.chain : 1;
        const int64_t out0 = ((int64_t)g * p.out_parts + op) * outw;
        p.feat += ((int64_t)g * p.in_parts + ip) * inw;
        p.acc += out0;
        if (MODE == 2) p.out += out0, p.bias = p.bias ? p.bias + out0 : p.bias;
        const int64_t rows = (int64_t)(p.transpose ? p.out_parts : p.in_parts) * p.C;
        p.weight += ((int64_t)g * rows + (p.transpose ? op : ip) * p.C) * p.w_pitch + (p.transpose ? ip : op) * p.M;
    }
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const int kb = (inw + 63) >> 6;
    const uint32_t a_bytes = (uint32_t)kb * BLK_BYTES;
    // layout: weight tile | feature tile(s) | parking area | chunk table; when the parking area
    // aliases the feature tile (p.alias) it starts where the feature tile starts
    const uint32_t b_tile = base;
    const uint32_t a_tile0 = b_tile + (uint32_t)((p.M + 63) >> 6) * (uint32_t)p.C * 128;
    const bool two = p.nbuf == 2;
    // the weight tile is W[tap] as stored: C rows of M channels, 64-channel blocks
    const uint32_t w_blk = (uint32_t)p.C * 128;
    const uint32_t bar = smem_u32(&s_bar);
    // per-warp parking area of the scatter: 32 rows of slab floats, rows padded by 16 bytes
    const uint32_t park_pitch = (uint32_t)p.slab * 4 + 16;
    const int prow = 1 << p.prow_log2;
    const uint32_t a_all = (uint32_t)p.nbuf * a_bytes;
    const uint32_t park0 = p.alias ? a_tile0 : a_tile0 + a_all;
    const uint32_t park = park0 + (uint32_t)(warp * prow) * park_pitch;
    const uint32_t table_off = p.alias ? max(a_all, p.park_bytes) : a_all + p.park_bytes;
    int32_t *s_cum = reinterpret_cast<int32_t *>(smem_raw + (a_tile0 - smem_u32(smem_raw)) + table_off);

    if (tid == 0) {
        mbar_init(bar, 1);
        fence_mbar_init();
    }
    if (warp == 0) tmem_alloc(smem_u32(&s_tmem), p.ncols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    start_after_previous();   // (tensor memory is held by now: see there)
    if (AGAIN && !p.only_if.holds()) {
        if (warp == 0) tmem_dealloc(tmem, p.ncols);
        return;
    }
    build_chunk_table<CH>(p.seg, p.K, s_cum, s_warp_sums);

    const int total = s_cum[p.K];
    const int per = (total + gridDim.x - 1) / gridDim.x;
    const int lo = blockIdx.x * per, hi = min(total, lo + per);
    // forward: B = W[tap] read MN-major (its rows are the contraction index c);
    // input gradient: B = W[tap] read K-major (its rows are the output index c)
    const uint32_t idesc = instr_desc(p.fmt, 128, outw, 0, p.transpose ? 0 : 1);
    const int ksteps = inw >> 4;
    uint32_t phase = 0;
    int loaded_tap = -1;
    bool alive = true;

    auto load_weight = [&](int tap, int part) {
        const uint16_t *w = p.weight + (p.reverse ? p.K - 1 - tap : tap) * p.w_tap +
                            (p.transpose ? (int64_t)part * p.M : part * p.C * p.w_pitch);
        const int cpr = p.M >> 3;
        const int dc = NT / cpr, dch = NT - dc * cpr;   // from one piece of a thread to its next
        int c = tid / cpr, ch = tid - c * cpr;
        for (int e = tid; e < p.C * cpr; e += NT) {
            uint32_t dst = b_tile + (uint32_t)(ch >> 3) * w_blk + (uint32_t)c * 128 + (uint32_t)(((ch & 7) ^ (c & 7)) << 4);
            cp_async16(dst, w + c * p.w_pitch + ch * 8);
            c += dc, ch += dch;
            if (ch >= cpr) ch -= cpr, ++c;
        }
    };

    ChunkCursor c0, c1, c2;  // chunk, chunk + 1, chunk + 2
    int pre_g = 0, pre_s = 0;
    if (lo < hi) {
        c0.seek(s_cum, p.seg, p.K, lo);
        c1 = c0;
        c2 = c0;
        const int rows = c0.rows(lo);
        if (tid < rows) {
            s_gather[0][tid] = p.gather[c0.first(lo) + tid];
            s_scatter[0][tid] = p.scatter[c0.first(lo) + tid];
        }
        load_weight(c0.tap, 0);
        loaded_tap = c0.tap;
        __syncthreads();
        gather_tile(a_tile0, p.feat, s_gather[0], rows, inw, p.in_pitch, tid, NT);
        cp_async_commit();
        if (lo + 1 < hi) {
            c1.advance(s_cum, p.seg, p.K, lo + 1);
            c2 = c1;
            if (tid < c1.rows(lo + 1)) {
                pre_g = p.gather[c1.first(lo + 1) + tid];
                pre_s = p.scatter[c1.first(lo + 1) + tid];
            }
        }
    }

    for (int chunk = lo; chunk < hi && alive; ++chunk) {
        const int b = (chunk - lo) & 1;
        const int rows = c0.rows(chunk);
        const bool have_next = chunk + 1 < hi;
        const int rows_next = have_next ? c1.rows(chunk + 1) : 0;
        if (have_next && tid < rows_next) {
            s_gather[b ^ 1][tid] = pre_g;
            s_scatter[b ^ 1][tid] = pre_s;
        }
        __syncthreads();
        if (have_next && two)
            gather_tile(a_tile0 + (uint32_t)(b ^ 1) * a_bytes, p.feat, s_gather[b ^ 1], rows_next, inw, p.in_pitch, tid, NT);
        cp_async_commit();
        if (chunk + 2 < hi) {
            c2.advance(s_cum, p.seg, p.K, chunk + 2);
            if (tid < c2.rows(chunk + 2)) {
                pre_g = p.gather[c2.first(chunk + 2) + tid];
                pre_s = p.scatter[c2.first(chunk + 2) + tid];
            }
        }
        for (int part = 0;; ++part) {
            if (two) cp_async_wait<1>();  // everything but the gather just issued has landed
            else cp_async_wait<0>();
            fence_async_smem();
            __syncthreads();

            if (tid == 0) {
                tc_fence_after();
                const uint32_t a_tile = a_tile0 + (two ? (uint32_t)b * a_bytes : 0u);
                for (int s = 0; s < ksteps; ++s) {
                    uint64_t ad = smem_desc(a_tile + (uint32_t)(s >> 2) * BLK_BYTES + (uint32_t)(s & 3) * 32, 16, 1024);
                    uint64_t bd = p.transpose
                                      ? smem_desc(b_tile + (uint32_t)(s >> 2) * w_blk + (uint32_t)(s & 3) * 32, 16, 1024)
                                      : smem_desc(b_tile + (uint32_t)s * 2048, w_blk, 1024);
                    tc_mma(tmem + (uint32_t)part * p.acc_cols, ad, bd, idesc, s > 0 ? 1u : 0u);
                }
                tc_commit(bar);
            }
            alive = __syncthreads_and(mbar_wait(bar, phase, 1u, &g_device_status));
            phase ^= 1u;
            tc_fence_after();
            if (part + 1 >= parts || !alive) break;
            load_weight(c0.tap, part + 1);   // the next part, over both tiles
            gather_tile(a_tile0, p.feat + (int64_t)(part + 1) * inw, s_gather[b], rows, inw, p.in_pitch, tid, NT);
            cp_async_commit();
        }
        // the weight tile is free now: fetch the next tap's if the next chunk needs it
        if (have_next && (c1.tap != loaded_tap || parts > 1)) {
            load_weight(c1.tap, 0);
            loaded_tap = c1.tap;
            cp_async_commit();
        }
        if (have_next && !two && !p.alias) {  // single A tile: it is free as well
            gather_tile(a_tile0, p.feat, s_gather[b ^ 1], rows_next, inw, p.in_pitch, tid, NT);
            cp_async_commit();
        }
        if (BULK && alive && warp * 32 < rows) {
            const int row = warp * 32 + lane;
            const bool row_ok = row < rows;
            float *dst_row = p.acc + (row_ok ? s_scatter[b][row] : 0) * p.out_pitch;
            // a warp parks `prow` rows at a time (32, or 16 when shared memory is better spent
            // on one more resident CTA): lanes of the current batch store, the others only
            // take part in the warp-wide TMEM load
            const uint32_t my_park = park + (uint32_t)(lane & (prow - 1)) * park_pitch;
            for (int batch = 0; batch * prow < 32; ++batch) {
                const bool mine = (lane >> p.prow_log2) == batch;
                if (warp * 32 + batch * prow >= rows) break;
                for (int col0 = 0; col0 < outw; col0 += p.slab) {
                    bulk_wait_read();  // the previous reductions have read this warp's parking area
                    __syncwarp();
                    for (int c32 = 0; c32 < p.slab; c32 += 32) {
                        float v[32];
                        tmem_ld32(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(col0 + c32), v);
                        if (mine) {
#pragma unroll
                            for (int q = 0; q < 8; ++q)
                                asm volatile("st.shared.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(my_park + (uint32_t)(c32 + 4 * q) * 4),
                                             "f"(v[4 * q]), "f"(v[4 * q + 1]), "f"(v[4 * q + 2]), "f"(v[4 * q + 3]) : "memory");
                        }
                    }
                    fence_async_smem();
                    const int cols = min(p.slab, outw - col0);
                    if (row_ok && mine) bulk_reduce_add_f32(dst_row + col0, my_park, (uint32_t)cols * 4);
                    bulk_commit();
                }
            }
        } else if (MODE == 2 && alive && warp * 32 < rows) {
            // one thread per accumulator row: 32 columns at a time, rounded and stored
            const int row = warp * 32 + lane;
            const bool row_ok = row < rows;
            uint16_t *dst_row = p.out + (row_ok ? s_scatter[b][row] : 0) * p.out_pitch;
            for (int col0 = 0; col0 < outw; col0 += 32) {
                float v[32];
                tmem_ld32(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)col0, v);
                if (row_ok) {
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        if (col0 + 8 * q < outw) {
                            if (p.bias) {
#pragma unroll
                                for (int e = 0; e < 8; ++e) v[8 * q + e] += unpack_one(p.bias[col0 + 8 * q + e], p.fmt);
                            }
                            uint4 o;
                            o.x = pack_pair(v[8 * q], v[8 * q + 1], p.fmt), o.y = pack_pair(v[8 * q + 2], v[8 * q + 3], p.fmt);
                            o.z = pack_pair(v[8 * q + 4], v[8 * q + 5], p.fmt), o.w = pack_pair(v[8 * q + 6], v[8 * q + 7], p.fmt);
                            *reinterpret_cast<uint4 *>(dst_row + col0 + 8 * q) = o;
                        }
                    }
                }
            }
        } else if (MODE == 0 && alive && (warp & 3) * 32 < rows) {
            // wide rows: scatter from registers (two-float vector reductions); with several
            // 64-column blocks per row the single parking area would serialise the bulk reductions
            const int32_t *sc = s_scatter[b];
            const int quarter = warp & 3;   // the lanes of tensor memory a warp can read
#pragma unroll 1
            for (int half = 0; half < 2; ++half) {
                if (quarter * 32 + half * 16 >= rows) break;
                const int ra = quarter * 32 + half * 16 + (lane >> 2), rb = ra + 8;
                const int64_t da = ra < rows ? sc[ra] : -1, db = rb < rows ? sc[rb] : -1;
                for (int col0 = (warp >> 2) * 64; col0 < outw; col0 += 64 * (NT / 128)) {
                    float v[32];
                    const uint32_t from = tmem + ((uint32_t)(quarter * 32 + half * 16) << 16) + (uint32_t)col0;
                    tmem_ld_16x64(from, v);
                    for (int part = 1; CHAINED && part < parts; ++part) {
                        float u[32];
                        tmem_ld_16x64(from + (uint32_t)part * p.acc_cols, u);
#pragma unroll
                        for (int e = 0; e < 32; ++e) v[e] += u[e];
                    }
                    scatter_block(p.acc, da, db, outw, p.out_pitch, col0, lane, v);
                }
            }
        }
        if (p.alias) {
            // the parking area lies in the feature tile: gather the next chunk only after the
            // reductions have read it (other resident CTAs cover the latency)
            bulk_wait_read();
            __syncthreads();
            if (have_next) {
                gather_tile(a_tile0, p.feat, s_gather[b ^ 1], rows_next, inw, p.in_pitch, tid, NT);
                cp_async_commit();
            }
        }
        c0 = c1;
        c1 = c2;
        tc_fence_before();
        __syncthreads();
    }
    cp_async_wait<0>();
    bulk_wait_read();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, p.ncols);
}

uint32_t pow2_cols(int n) {
    uint32_t c = 32;
    while ((int)c < n) c <<= 1;
    return c;
}

// CTAs per SM: bounded by shared memory (227 KiB usable, 1 KiB reserved per
// CTA), by TMEM (512 columns) and by registers / warp slots.
int ctas_per_sm(size_t smem, uint32_t ncols, int regs_per_thread, int threads = 128) {
    int by_smem = (int)((size_t)232448 / (smem + 1024));
    int by_tmem = (int)(512 / ncols);
    int by_regs = 65536 / (((regs_per_thread * 32 + 255) / 256 * 256) * (threads / 32));
    int occ = std::min(by_smem, std::min(by_tmem, by_regs));
    if (occ > 8) occ = 8;
    return occ < 1 ? 1 : occ;
}

// Registers per thread of a kernel (asked once per kernel; the persistent grids
// must not exceed what is resident at once, or the surplus CTAs run as a second wave).
template <typename Kernel>
int kernel_registers(Kernel kernel, std::atomic<int> *cached) {
    int n = cached->load(std::memory_order_relaxed);
    if (n == 0) {
        cudaFuncAttributes attr;
        n = cudaFuncGetAttributes(&attr, kernel) == cudaSuccess ? attr.numRegs : 128;
        cached->store(n, std::memory_order_relaxed);
    }
    return n;
}

// Dynamic shared memory padded so that at most 512 / ncols CTAs share an SM
// (their TMEM allocations then always fit).
size_t pad_for_tmem(size_t smem, uint32_t ncols) {
    size_t max_ctas = 512 / ncols;
    size_t floor_bytes = (size_t)232448 / (max_ctas + 1) + 1024;
    return smem > floor_bytes ? smem : floor_bytes;
}

bool aligned16(const void *p) { return ((uintptr_t)p & 15) == 0; }

}  // namespace

bool mvmr_tensor_supported(const MvmrArgs &a) {
    if (a.dtype != PCX_F16 && a.dtype != PCX_BF16) return false;
    if (!a.seg_offs || a.T <= 0 || a.K > MAX_TAPS_SMEM) return false;
    if (!splits_evenly(a.C) || !splits_evenly(a.M) || (int64_t)a.G * parts_of(a.C) * parts_of(a.M) > MAX_PARTS) return false;
    if (a.out_rows && parts_of(a.transpose ? a.M : a.C) > 1) return false;   // rows can be stored only where one pass completes them
    if (!aligned16(a.weight) || !aligned16(a.feat)) return false;
    if (a.T / CH + a.K >= INT32_MAX) return false;
    return true;
}

int mvmr_tensor(const MvmrArgs &a, cudaStream_t stream) {
    const int c_parts = parts_of(a.C), m_parts = parts_of(a.M), C = a.C / c_parts, M = a.M / m_parts;   // the part's
    const int inw = a.transpose ? M : C, outw = a.transpose ? C : M;
    MvmrTcParams p;
    p.in_parts = a.transpose ? m_parts : c_parts, p.out_parts = a.transpose ? c_parts : m_parts;
    p.in_pitch = (int64_t)a.G * p.in_parts * inw, p.out_pitch = (int64_t)a.G * p.out_parts * outw;
    p.w_pitch = a.M, p.w_tap = (int64_t)a.G * a.C * a.M;
    const int64_t upper = a.T / CH + a.K + 1;   // tiles of triplets, at most
    p.weight = (const uint16_t *)a.weight, p.feat = (const uint16_t *)a.feat;
    p.gather = a.gather, p.scatter = a.scatter, p.seg = a.seg_offs, p.acc = a.acc;
    p.out = (uint16_t *)a.out_rows, p.bias = (const uint16_t *)a.bias, p.reverse = a.reverse, p.only_if = a.only_if;
    p.K = a.K, p.C = C, p.M = M, p.transpose = a.transpose, p.fmt = a.dtype == PCX_BF16 ? 1 : 0;
    p.ncols = p.acc_cols = pow2_cols((outw + 63) / 64 * 64);  // the epilogue reads blocks of up to 64 columns
    // Measured on B200: rows of exactly 64 floats leave fastest through one bulk reduction
    // each (64 vs 84 us on the 150k-point scene); narrower and wider rows from registers
    // (C = 32: 50 vs 59 us, C = 128: 160 vs 180 us, C = 256: 390 vs 671 us).  Folding rows
    // with equal destinations in shared memory first was tried and cost more than it saved.
    bool bulk = outw == 64;
    if (const char *e = getenv("PCX_MVMR_SCATTER")) bulk = atoi(e) != 0;
    const bool store = a.out_rows != nullptr;
    if (store) bulk = false;
    const int kb = (inw + 63) / 64, wb = (M + 63) / 64;
    const size_t static_smem = 2176;  // index rings, barrier
    const size_t table = align_up((size_t)(a.K + 1) * 4, 16);
    p.slab = outw >= 64 ? 64 : 32;  // columns parked per bulk reduction
    // Rows a warp parks at a time.  Fewer rows leave shared memory for more resident CTAs,
    // which hide the gather latency (measured on the 150k-point scene, C = 64: 32 rows /
    // 3 CTAs per SM 78 us, 16 rows / 5 CTAs 64 us, 8 rows / 6 CTAs 66 us).
    p.prow_log2 = 4;
    if (const char *e = getenv("PCX_MVMR_PARK_ROWS")) p.prow_log2 = atoi(e) == 32 ? 5 : atoi(e) == 8 ? 3 : 4;
    p.park_bytes = bulk ? (uint32_t)(4 << p.prow_log2) * (p.slab * 4 + 16) : 0;
    // The parking area shares the feature tile's memory: the next gather then waits for the
    // reductions to drain, but one more CTA fits per SM (measured: 62 vs 65 us).
    p.alias = bulk ? 1 : 0;
    if (const char *e = getenv("PCX_MVMR_ALIAS")) p.alias = bulk && atoi(e) != 0;
    const size_t rest = 1024 + (size_t)wb * C * 128 + (p.alias ? 0 : p.park_bytes) + table;
    // One A tile: it is free again as soon as the multiply has finished, so the
    // next gather still overlaps the scatter, and more CTAs fit on an SM.
    p.nbuf = 1;
    if (const char *e = getenv("PCX_MVMR_NBUF"))
        if (atoi(e) == 2 && rest + 2 * (size_t)kb * BLK_BYTES + static_smem <= 232448 - 1024) p.nbuf = 2;
    if (p.alias) p.nbuf = 1;
    size_t smem = rest + std::max((size_t)p.nbuf * kb * BLK_BYTES, p.alias ? (size_t)p.park_bytes : (size_t)0);
    // 256 threads, and parts of a contraction in one block, where one CTA fills an SM's shared memory: as many parts as
    // tensor memory holds, in links of the same length.  Every link gets the same share of the chip, so a shorter one would
    // leave its share idle (300 000 triplets, us, in links as equal as parts allow / of one part / as long as possible:
    // 768 to 512 channels, three parts, two fit: 779 / 779 / 908; 1280 to 128, five, four fit: 409 / 409 / 562; 1536 to 128,
    // six: 450 / 487 / 567; 2048 to 128, eight: 580 / 634 / 580).  A link saves an eighth of its parts' time;
    // where the tiles of so few blocks make more turns of the chip than that, the parts stay blocks of their own (174 tiles:
    // 1024 to 128 channels 38 us, in one link 46, 2048 to 128 60.5 and 62.6; 276 tiles: 1024 to 128 54 and 46, 512 to 512 87 and
    // 71; 808: 768 to 128 99 and 93).  Plain reductions into an accumulator much larger than
    // the L2 cache keep 128 threads: they are bound by its misses (256 x 256 into 184 MB 584 us and with 256 threads
    // 620; into 123 MB 398 and 388, 61 MB 208 and 202).
    const bool one_cta = !store && !bulk && outw > 64 && 2 * (smem + static_smem + 1024) > 232448;
    p.chain = one_cta && p.nbuf == 1 ? std::min(p.in_parts, (int)(512 / p.acc_cols)) : 1;
    while (p.in_parts % p.chain) --p.chain;
    int parts = a.G * p.out_parts * (p.in_parts / p.chain);
    auto turns = [&](int n) { return (upper + std::max(1, num_sms() / n) - 1) / std::max(1, num_sms() / n); };
    if (7 * p.chain * turns(parts) > 8 * turns(parts * p.chain)) parts *= p.chain, p.chain = 1;
    p.ncols = pow2_cols(p.acc_cols * p.chain);
    const bool more = one_cta && (p.chain > 1 || a.n_out * p.out_pitch * 4 <= (int64_t)160 << 20);
    smem = pad_for_tmem(smem, p.ncols);
    if (smem + static_smem > 232448 - 1024) PCX_FAIL(PCX_E_UNSUPPORTED, "mvmr tensor kernel does not fit (smem %zu)", smem);
    // (rows are never stored in a call that may do one again)
    const int mode = (store ? 2 : bulk ? 1 : p.chain > 1 ? 4 : more ? 3 : 0) + (a.only_if.words ? 5 : 0), threads = more ? 256 : 128;
    static std::atomic<uint64_t> allowed[10];   // per kernel
    static std::atomic<int> regs_mvmr[10];
    decltype(&mvmr_tc_kernel<0, 128, false, false>) const kernels[10] = {
        mvmr_tc_kernel<0, 128, false, false>, mvmr_tc_kernel<1, 128, false, false>, mvmr_tc_kernel<2, 128, false, false>,
        mvmr_tc_kernel<0, 256, false, false>, mvmr_tc_kernel<0, 256, true, false>,  mvmr_tc_kernel<0, 128, false, true>,
        mvmr_tc_kernel<1, 128, false, true>,  nullptr,                              mvmr_tc_kernel<0, 256, false, true>,
        mvmr_tc_kernel<0, 256, true, true>};
    const auto kernel = kernels[mode];
    if (!kernel) PCX_FAIL(PCX_E_ARG, "mvmr tensor kernel: no such variant");
    if (int rc = allow_shared_memory((const void *)kernel, &allowed[mode], true)) return rc;
    const int regs = kernel_registers(kernel, &regs_mvmr[mode]);
    const int occ = ctas_per_sm(smem + static_smem, p.ncols, regs, threads);
    const dim3 grid((unsigned)std::min<int64_t>(upper, std::max<int64_t>(1, (int64_t)occ * num_sms() / parts)), (unsigned)parts);
    if (!a.only_if.words)
        prof_begin(store ? (a.transpose ? "mvmr_tc_kernel(dgrad, store)" : "mvmr_tc_kernel(fwd, store)")
                         : (a.transpose ? "mvmr_tc_kernel(dgrad)" : "mvmr_tc_kernel(fwd)"), stream);
    launch_after(kernel, grid, threads, smem, stream, p);
    if (!a.only_if.words) prof_end(stream);
    PCX_LAUNCH_CHECK();
    return PCX_OK;
}

// Device address of the status word, for kernels of other translation units.
int device_status_address(unsigned int **d_status) {
    PCX_CUDA(cudaGetSymbolAddress((void **)d_status, g_device_status));
    return PCX_OK;
}

int read_device_status(unsigned int *h_status, bool clear, cudaStream_t stream) {
    PCX_CUDA(cudaStreamSynchronize(stream));
    PCX_CUDA(cudaMemcpyFromSymbol(h_status, g_device_status, sizeof(unsigned int)));
    if (clear && *h_status) {
        unsigned int zero = 0;
        PCX_CUDA(cudaMemcpyToSymbol(g_device_status, &zero, sizeof(unsigned int)));
    }
    return PCX_OK;
}

}  // namespace pcx
