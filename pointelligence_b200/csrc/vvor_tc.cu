// VVOR on sm_100a (tcgen05 + TMEM): the gradient of the weights.
//
//   D[Ma x Cb] += X[t x Ma]^T * G[t x Cb], t = triplets of a chunk; both operands MN-major (a gathered row
//   is contiguous along M / N, the triplet index is the contraction), accumulated in TMEM over all chunks of
//   a tap and added to the fp32 sums in global memory once per (CTA, tap).
//
// A persistent CTA per SM owns a contiguous range of chunks of tap-sorted triplets.  Its warps play roles, so
// that index fetch, row copies, multiplies and the writing of a finished tap run at the same time:
//
//   index warp     the index rows of a chunk, up to eight chunks early
//   copy teams     up to four; a team gathers the rows of a chunk with 16-byte cp.async copies straight into the
//                  128-byte-swizzled tiles ([64-channel block][row][128 bytes]) of a slot
//   MMA thread     up to CHR / 16 steps of tcgen05.mma per 128 rows of D
//   flush warps    read a finished tap from TMEM and add it to global memory; up to 256 columns of
//                  accumulators are double-buffered, so the next tap starts meanwhile
//
// Bound by what the L2 gives to gathers of whole rows, below 64 channels by the chain of a chunk (waits, copies,
// MMA issue).  300k points, 6.6 M triplets: 64 x 64 148 us, 128 x 128 294, 256 x 256 718 (11.3, 11.4 and 9.4 TB/s of
// gathered rows); 150k points, 0.98 M: 34, 54, 120 us.  With the same warps doing every step of a chunk, and a block
// barrier a chunk: 186, 385, 1042 and 42, 76, 178 us.  16 x 16 is 10 % slower than with those (6 of 8 lanes of a copy
// have nothing to do): 200 000 points, 3.6 M triplets 82 against 73 us.
//
// Few triplets a tap (the deep levels of a network): a CTA takes whole taps, rounds what tensor memory holds and stores it
// (STORE), so that there are no fp32 sums to clear, to add to and to round: the figures stand at vvor_stores().
//
// Every wait is bounded (one second) and abortable: a role that gives up raises a flag in the status word and
// in shared memory, the other roles leave their waits, and the CTA frees its TMEM and returns.
#include "sparse_kernels.cuh"
#include "tcgen05.cuh"

namespace pcx {
int device_status_address(unsigned int **d_status);

namespace {

using namespace tc;

constexpr unsigned STATUS_BIT = 2u;
constexpr int MAX_PARTS = 64;        // (group, part, part) combinations of one launch
constexpr int MAX_TAPS_SMEM = 1024;  // taps whose chunk table fits the shared-memory copy
constexpr int FLUSH_WARPS = 4, TEAMS = 4, TEAM_WARPS = 4;
constexpr int COPY_WARP0 = FLUSH_WARPS, INDEX_WARP = COPY_WARP0 + TEAMS * TEAM_WARPS, MMA_WARP = INDEX_WARP + 1;
constexpr int THREADS = (MMA_WARP + 1) * 32;
constexpr int MAX_SLOTS = 6, AHEAD = 8;   // chunks whose rows / whose indices are in shared memory

struct VvorTcParams {
    const uint16_t *a, *b;  // (n_a, Ma), (n_b, Cb)
    const int32_t *a_idx, *b_idx;
    const int64_t *seg;
    float *acc;             // (n_o, G, rows of Cb)
    uint16_t *out;          // STORE: the same, rounded
    unsigned int *status;
    int64_t a_pitch, b_pitch, acc_pitch, acc_tap;   // rows of a / b / one tap's sums, elements of one tap's sums
    int a_parts, b_parts;                           // blockIdx.y: (group, part of a, part of b)
    int n_o, Ma, Cb, fmt, nslots, nacc, teams;      // Ma, Cb: the part's
    uint32_t ncols, acc_cols;
};

// The rows of a chunk of one operand that this lane copies: CHR / 16 consecutive rows from `row0` on, a 16-byte
// piece of each 64-channel block of a row.  Rows from `rows` up to a multiple of 16 are zeros.
template <int CHR>
__device__ __forceinline__ void copy_operand(uint32_t tile, const uint16_t *src, uint32_t pitch_bytes, uint32_t idx, int row0,
                                             int rows, int piece, int pieces) {
    if (piece >= pieces) return;
    const char *col = reinterpret_cast<const char *>(src + piece * 8);
    const int blocks = (pieces - piece + 7) >> 3, end = (rows + 15) & ~15;
#pragma unroll
    for (int q = 0; q < CHR / 64; ++q) {
        const int r = row0 + 4 * q;
        if (r >= end) return;
        const uint4 i4 = lds_v4(idx + (uint32_t)r * 4);
        const uint32_t at[4] = {i4.x, i4.y, i4.z, i4.w};
        const char *s[4];
        uint32_t dst[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            s[k] = col + (uint64_t)(r + k < rows ? at[k] : 0u) * pitch_bytes;
            dst[k] = tile + (uint32_t)(r + k) * 128 + (uint32_t)((piece ^ ((r + k) & 7)) << 4);
        }
        for (int c = 0;;) {
#pragma unroll
            for (int k = 0; k < 4; ++k) cp_async16_or_zero(dst[k], s[k], r + k >= rows);
            if (++c == blocks) break;
#pragma unroll
            for (int k = 0; k < 4; ++k) dst[k] += CHR * 128, s[k] += 128;
        }
    }
}

// 32 rounded columns of a row (those below `left`) from tensor memory, or zeros; the row may begin at any even address
__device__ __forceinline__ void store_columns(uint16_t *dst, const float *v, int left, int fmt, bool wide) {
    uint32_t o[16];
#pragma unroll
    for (int e = 0; e < 16; ++e) {
        if (fmt) {
            const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * e], v[2 * e + 1]);
            o[e] = *reinterpret_cast<const uint32_t *>(&h);
        } else {
            const __half2 h = __floats2half2_rn(v[2 * e], v[2 * e + 1]);
            o[e] = *reinterpret_cast<const uint32_t *>(&h);
        }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {   // (widths are multiples of 16)
        if (8 * e >= left) continue;
        if (wide) reinterpret_cast<uint4 *>(dst)[e] = make_uint4(o[4 * e], o[4 * e + 1], o[4 * e + 2], o[4 * e + 3]);
        else
#pragma unroll
            for (int q = 0; q < 8; ++q) dst[8 * e + q] = (uint16_t)(o[4 * e + q / 2] >> (16 * (q & 1)));
    }
}

template <int CHR, bool STORE>   // triplets of a chunk: the contraction of one slot
__global__ void __launch_bounds__(THREADS, 1) vvor_tc_kernel(VvorTcParams p) {
    constexpr uint32_t BLK = CHR * 128;   // one 64-channel block of a tile
    using Cursor = ChunkCursorT<CHR>;
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t s_full[MAX_SLOTS], s_empty[MAX_SLOTS], s_acc_full[2], s_acc_empty[2], s_idx_full[AHEAD], s_idx_empty[AHEAD];
    __shared__ uint32_t s_tmem;
    __shared__ int s_abort;
    __shared__ int32_t s_warp_sums[THREADS / 32];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    {
        const int bp = (int)blockIdx.y % p.b_parts, ap = (int)blockIdx.y / p.b_parts % p.a_parts,
                  g = (int)blockIdx.y / (p.b_parts * p.a_parts);
        p.a += ((int64_t)g * p.a_parts + ap) * p.Ma;
        p.b += ((int64_t)g * p.b_parts + bp) * p.Cb;
        const int64_t first = ((int64_t)g * p.a_parts + ap) * p.Ma * p.acc_pitch + bp * p.Cb;
        if (STORE) p.out += first;
        else p.acc += first;
    }
    const int row_tiles = (p.Ma + 127) >> 7;
    const int ablk = (p.Ma + 63) >> 6, bblk = (p.Cb + 63) >> 6;   // an odd ablk borrows the next block as padding
    const uint32_t slot_bytes = (uint32_t)(ablk + bblk) * BLK;
    // behind the slots: the index rings of both operands, then the chunk table
    const uint32_t idx0 = base + (uint32_t)p.nslots * slot_bytes;
    int32_t *s_cum = reinterpret_cast<int32_t *>(smem_raw + (idx0 - smem_u32(smem_raw)) + 2 * AHEAD * CHR * 4);
    volatile int *abort_flag = &s_abort;
    auto wait_one = [&](const uint64_t &bar, uint32_t parity) {
        return mbar_wait_abortable(smem_u32(&bar), parity & 1u, STATUS_BIT, p.status, abort_flag);
    };
    auto wait = [&](const uint64_t &bar, uint32_t parity) {   // the verdict is the same in the whole warp
        if (__all_sync(0xffffffffu, mbar_try_wait(smem_u32(&bar), parity & 1u))) return true;
        return __all_sync(0xffffffffu, wait_one(bar, parity)) != 0;
    };

    if (tid == 0) {
        for (int s = 0; s < p.nslots; ++s) mbar_init(smem_u32(&s_full[s]), TEAM_WARPS * 32), mbar_init(smem_u32(&s_empty[s]), 1);
        for (int s = 0; s < 2; ++s) mbar_init(smem_u32(&s_acc_full[s]), 1), mbar_init(smem_u32(&s_acc_empty[s]), FLUSH_WARPS);
        for (int s = 0; s < AHEAD; ++s) mbar_init(smem_u32(&s_idx_full[s]), 32), mbar_init(smem_u32(&s_idx_empty[s]), TEAM_WARPS);
        fence_mbar_init();
        s_abort = 0;
    }
    if (warp == 0) tmem_alloc(smem_u32(&s_tmem), p.ncols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    start_after_previous();   // (tensor memory is held by now: see there)
    build_chunk_table<CHR>(p.seg, p.n_o, s_cum, s_warp_sums);

    const int total = s_cum[p.n_o];
    const int per = (total + gridDim.x - 1) / gridDim.x;
    const int tap0 = STORE ? (int)((int64_t)p.n_o * blockIdx.x / gridDim.x) : 0, tap1 = STORE ? (int)((int64_t)p.n_o * (blockIdx.x + 1) / gridDim.x) : p.n_o;
    const int lo = STORE ? s_cum[tap0] : blockIdx.x * per, hi = STORE ? s_cum[tap1] : min(total, lo + per);
    Cursor cur;
    if (lo < hi) cur.seek(s_cum, p.seg, p.n_o, lo);

    if (STORE && warp < FLUSH_WARPS) {
        // ----------------------------------------------------------------- store ----
        Ring acc;
        const bool wide = ((uintptr_t)p.out & 15) == 0 && p.acc_pitch % 8 == 0;
        for (int tap = tap0; tap < tap1; ++tap) {
            const bool none = s_cum[tap + 1] == s_cum[tap];
            if (!none) {
                if (!wait(s_acc_full[acc.slot], acc.turn)) break;
                tc_fence_after();
            }
            for (int rt = 0; rt < row_tiles; ++rt) {
                const int m = rt * 128 + warp * 32 + lane;
                if (rt * 128 + warp * 32 >= p.Ma) break;
                uint16_t *dst = p.out + tap * p.acc_tap + m * p.acc_pitch;
                for (int c0 = 0; c0 < p.Cb; c0 += 32) {
                    float v[32];
                    if (none) {
#pragma unroll
                        for (int e = 0; e < 32; ++e) v[e] = 0.f;
                    } else {
                        tmem_ld32(tmem + ((uint32_t)(warp * 32) << 16) + acc.slot * p.acc_cols + (uint32_t)(rt * p.Cb + c0), v);
                    }
                    if (m < p.Ma) store_columns(dst + c0, v, p.Cb - c0, p.fmt, wide);
                    __syncwarp();
                }
            }
            if (none) continue;
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&s_acc_empty[acc.slot]));
            acc.next(p.nacc);
        }
    } else if (lo >= hi) {
    } else if (!STORE && warp < FLUSH_WARPS) {
        // ----------------------------------------------------------------- flush ----
        // a warp reads the 32 TMEM lanes of its quarter
        Ring acc;
        for (int tap = cur.tap; tap < p.n_o && s_cum[tap] < hi; ++tap) {
            if (s_cum[tap + 1] == s_cum[tap]) continue;
            if (!wait(s_acc_full[acc.slot], acc.turn)) break;
            tc_fence_after();
            float *dst = p.acc + tap * p.acc_tap;
            for (int rt = 0; rt < row_tiles; ++rt) {
#pragma unroll 1
                for (int half = 0; half < 2; ++half) {
                    const int m0 = rt * 128 + warp * 32 + half * 16;
                    if (m0 >= p.Ma) break;
                    const int ma = m0 + (lane >> 2), mb = ma + 8;
                    const int64_t da = ma < p.Ma ? ma : -1, db = mb < p.Ma ? mb : -1;
                    for (int c0 = 0; c0 < p.Cb; c0 += 64) {
                        float v[32];
                        tmem_ld_16x64(tmem + ((uint32_t)(warp * 32 + half * 16) << 16) + acc.slot * p.acc_cols + (uint32_t)(rt * p.Cb + c0), v);
                        scatter_block(dst, da, db, p.Cb, p.acc_pitch, c0, lane, v);
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&s_acc_empty[acc.slot]));
            acc.next(p.nacc);
        }
    } else if (warp < INDEX_WARP) {
        // ---------------------------------------------------------------- copies ----
        const int team = (warp - COPY_WARP0) / TEAM_WARPS, piece = lane & 7;
        const int row0 = ((warp - COPY_WARP0) % TEAM_WARPS) * (CHR / 4) + (lane >> 3) * (CHR / 16);
        Ring ring, idx;
        ring.skip(team, p.nslots), idx.skip(team, AHEAD);
        if (team < p.teams) {
            for (int chunk = lo + team; chunk < hi; chunk += p.teams) {
                cur.advance(s_cum, p.seg, p.n_o, chunk);
                const int rows = cur.rows(chunk);
                if (!wait(s_idx_full[idx.slot], idx.turn) || !wait(s_empty[ring.slot], ring.turn ^ 1u)) break;
                const uint32_t tile = base + ring.slot * slot_bytes, ia = idx0 + idx.slot * (CHR * 4);
                copy_operand<CHR>(tile, p.a, (uint32_t)p.a_pitch * 2u, ia, row0, rows, piece, p.Ma >> 3);
                copy_operand<CHR>(tile + (uint32_t)ablk * BLK, p.b, (uint32_t)p.b_pitch * 2u, ia + AHEAD * CHR * 4, row0, rows, piece, p.Cb >> 3);
                cp_async_mbar_arrive(smem_u32(&s_full[ring.slot]));   // fires once this thread's copies have landed
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&s_idx_empty[idx.slot]));
                ring.skip(p.teams, p.nslots);
                idx.skip(p.teams, AHEAD);
            }
        }
        cp_async_wait<0>();
    } else if (warp == INDEX_WARP) {
        // --------------------------------------------------------------- indices ----
        Ring idx;
        for (int chunk = lo; chunk < hi; ++chunk) {
            cur.advance(s_cum, p.seg, p.n_o, chunk);
            const int rows = cur.rows(chunk);
            const int64_t first = cur.first(chunk);
            if (!wait(s_idx_empty[idx.slot], idx.turn ^ 1u)) break;
            const uint32_t ia = idx0 + idx.slot * (CHR * 4);
#pragma unroll 4
            for (int r = lane; r < rows; r += 32) {
                cp_async4(ia + (uint32_t)r * 4, p.a_idx + first + r);
                cp_async4(ia + (uint32_t)(AHEAD * CHR + r) * 4, p.b_idx + first + r);
            }
            cp_async_mbar_arrive(smem_u32(&s_idx_full[idx.slot]));
            idx.next(AHEAD);
        }
        cp_async_wait<0>();
    } else {
        // ------------------------------------------------------------------- MMA ----
        if (elect_one()) {
            const uint32_t idesc = instr_desc(p.fmt, 128, p.Cb, 1, 1);
            const uint64_t ad0 = smem_desc(base, BLK, 1024), bd0 = smem_desc(base + (uint32_t)ablk * BLK, BLK, 1024);
            Ring ring, acc;
            bool fresh = true;   // the next multiply starts a tap
            for (int chunk = lo; chunk < hi; ++chunk) {
                cur.advance(s_cum, p.seg, p.n_o, chunk);
                const int ksteps = (cur.rows(chunk) + 15) >> 4;
                if (fresh && !wait_one(s_acc_empty[acc.slot], acc.turn ^ 1u)) break;
                if (!wait_one(s_full[ring.slot], ring.turn)) break;
                fence_async_smem();   // the copies came through the generic proxy, the tensor core reads through the async proxy
                tc_fence_after();
                const uint64_t at = (uint64_t)(ring.slot * (slot_bytes >> 4));   // (descriptor addresses count 16 bytes)
                for (int rt = 0; rt < row_tiles; ++rt) {
                    const uint32_t d = tmem + acc.slot * p.acc_cols + (uint32_t)(rt * p.Cb);
                    const uint64_t ad = ad0 + at + (uint64_t)(rt * 2) * (BLK >> 4), bd = bd0 + at;
                    for (int s = 0; s < ksteps; ++s) tc_mma(d, ad + (uint64_t)(s * 128), bd + (uint64_t)(s * 128), idesc, fresh && s == 0 ? 0u : 1u);
                }
                tc_commit(smem_u32(&s_empty[ring.slot]));
                ring.next(p.nslots);
                fresh = chunk + 1 == hi || cur.last_of_tap(chunk);
                if (fresh) tc_commit(smem_u32(&s_acc_full[acc.slot])), acc.next(p.nacc);
            }
        }
        __syncwarp();
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, p.ncols);
}

template <int CHR, bool STORE>
int launch_vvor(VvorTcParams &p, int parts, int64_t T, size_t block_rows, cudaStream_t stream) {
    const size_t slot = block_rows * CHR * 128;
    const size_t rest = 1024 + 2 * AHEAD * CHR * 4 + align_up((size_t)(p.n_o + 1) * 4, 16);   // alignment, index rings, chunk table
    p.nslots = (int)std::min<size_t>(MAX_SLOTS, ((size_t)232448 - 1024 - rest) / slot);
    if (p.nslots < 2) PCX_FAIL(PCX_E_UNSUPPORTED, "vvor tensor kernel does not fit (Ma=%d Cb=%d)", p.Ma, p.Cb);
    p.teams = std::min(TEAMS, p.nslots);   // a wait names its turn by parity: no team may be a whole ring ahead of another
    const size_t smem = rest + p.nslots * slot;
    static std::atomic<uint64_t> allowed;
    if (int rc = allow_shared_memory((const void *)vvor_tc_kernel<CHR, STORE>, &allowed)) return rc;
    const dim3 grid((unsigned)std::min<int64_t>(STORE ? p.n_o : T / CHR + p.n_o + 1, std::max(1, num_sms() / parts)), (unsigned)parts);
    prof_begin("vvor_tc_kernel", stream);
    launch_after(vvor_tc_kernel<CHR, STORE>, grid, THREADS, smem, stream, p);
    prof_end(stream);
    PCX_LAUNCH_CHECK();
    return PCX_OK;
}

}  // namespace

bool vvor_tensor_supported(const VvorArgs &a) {
    if (a.dtype != PCX_F16 && a.dtype != PCX_BF16) return false;
    if (!a.seg_offs || a.T <= 0 || a.n_o > MAX_TAPS_SMEM) return false;
    if (!splits_evenly(a.Ma) || !splits_evenly(a.Cb) || (int64_t)a.G * parts_of(a.Ma) * parts_of(a.Cb) > MAX_PARTS) return false;
    if ((uintptr_t)a.a % 16 || (uintptr_t)a.b % 16) return false;
    return a.T / 64 + a.n_o < INT32_MAX;
}

namespace {

// Parts of both operands for CTAs that take whole taps: as few as 256 columns ask for, then halves while that gives the
// chip more CTAs and a part keeps 64 columns.
void store_parts(const VvorArgs &a, int *a_parts, int *b_parts) {
    *a_parts = parts_of(a.Ma), *b_parts = parts_of(a.Cb);
    auto halves = [](int width, int parts) { return width % (32 * parts) == 0 && width / parts >= 128; };
    while (2 * a.n_o * a.G * *a_parts * *b_parts <= num_sms() && 2 * a.G * *a_parts * *b_parts <= MAX_PARTS) {
        const bool b_wider = a.Cb / *b_parts > a.Ma / *a_parts;
        if (b_wider && halves(a.Cb, *b_parts)) *b_parts *= 2;
        else if (halves(a.Ma, *a_parts)) *a_parts *= 2;
        else if (halves(a.Cb, *b_parts)) *b_parts *= 2;
        else break;
    }
}

}  // namespace

// Up to how many triplets of the fullest tap CTAs take whole taps.  The fullest tap decides how long that takes, 10 ns a triplet of
// 256 x 256 channels and 7 of 64 x 64 or 128 x 128; the fp32 sums cost a microsecond a megabyte.  27 taps, fullest tap 950 / 3056 / 5150,
// sums and stored, us: 512 x 512 (28 MB) 44 / 54 / 57 and 29 / 51 / 74, 256 x 256 (7 MB) 28 / 30 / 40 and 18 / 33 / 47,
// 128 x 128 (2 MB) 18 / 20 / 22 and 16 / 31 / 43, 64 x 64 15 / 15 / 17 and 16 / 31 / 43; 125 taps, 5050: 512 x 512 (131 MB) 143 and 96.
int64_t vvor_store_limit(int64_t n_o, int G, int Ma, int Cb) {
    const int64_t sums = n_o * G * Ma * Cb * 4;
    return sums >= (1 << 20) ? 300 + sums / 10000 : 0;
}

// Searches hand the pairs of their fullest tap to the host.  Of other rulebooks nothing but the sizes is known here.  A room on itself
// has a triplet of every point, or 1.1, in its centre tap; strided ones 1.1 to 2.1 for a row of the fewer (2.7 with 125 taps), sweeps
// 1.2 to 1.7; where every tap is dense the fullest has 1.1 to 1.9 times the average.  All in one tap, 512 x 512 channels: 18 000
// triplets 200 us stored and 90 summed, 72 000 736 and 129.
bool vvor_stores(const VvorArgs &a) {
    const int64_t rows = std::min(a.n_a, a.n_b), guess = std::min(a.T, std::max(2 * a.T / a.n_o, a.n_a == a.n_b ? rows : 2 * rows));
    return (a.fullest >= 0 ? a.fullest : guess) <= vvor_store_limit(a.n_o, a.G, a.Ma, a.Cb);
}

int vvor_tensor(const VvorArgs &a, cudaStream_t stream) {
    VvorTcParams p = {};
    p.a = (const uint16_t *)a.a, p.b = (const uint16_t *)a.b, p.a_idx = a.a_idx, p.b_idx = a.b_idx;
    p.seg = a.seg_offs, p.acc = a.acc, p.out = (uint16_t *)a.out;
    const bool store = a.out != nullptr;
    p.a_parts = parts_of(a.Ma), p.b_parts = parts_of(a.Cb);
    if (store) store_parts(a, &p.a_parts, &p.b_parts);
    const int parts = a.G * p.a_parts * p.b_parts;
    p.Ma = a.Ma / p.a_parts, p.Cb = a.Cb / p.b_parts;   // the part's widths
    p.a_pitch = (int64_t)a.G * a.Ma, p.b_pitch = (int64_t)a.G * a.Cb, p.acc_pitch = a.Cb, p.acc_tap = (int64_t)a.G * a.Ma * a.Cb;
    p.n_o = (int)a.n_o, p.fmt = a.dtype == PCX_BF16 ? 1 : 0;
    if (int rc = device_status_address(&p.status)) return rc;
    p.acc_cols = (uint32_t)(((p.Ma + 127) / 128 - 1) * p.Cb + (p.Cb + 63) / 64 * 64);   // read in blocks of 64 (stored: 32) columns
    p.nacc = 2 * p.acc_cols <= 512 ? 2 : 1;
    p.ncols = 32;
    while (p.ncols < (uint32_t)p.nacc * p.acc_cols) p.ncols <<= 1;
    // Slots of up to 64 KB: the chain of a chunk (waits, copies, MMA issue, some 1000 clocks whatever its size) stays
    // below the time its copies take, and three slots fit (64 x 64, 6.6 M triplets: chunks of 64 / 128 / 256 triplets
    // 299 / 197 / 148 us).  Few triplets: shorter chunks, so that every SM has some.
    const size_t blocks = (size_t)((p.Ma + 63) / 64 + (p.Cb + 63) / 64);
    const int64_t ctas = std::max(1, num_sms() / parts);
    int chr = blocks <= 2 ? 256 : blocks <= 4 ? 128 : 64;
    while (chr > 64 && a.T < 4 * ctas * chr) chr /= 2;
    if (store) {
        if (chr == 256) return launch_vvor<256, true>(p, parts, a.T, blocks, stream);
        if (chr == 128) return launch_vvor<128, true>(p, parts, a.T, blocks, stream);
        return launch_vvor<64, true>(p, parts, a.T, blocks, stream);
    }
    if (chr == 256) return launch_vvor<256, false>(p, parts, a.T, blocks, stream);
    if (chr == 128) return launch_vvor<128, false>(p, parts, a.T, blocks, stream);
    return launch_vvor<64, false>(p, parts, a.T, blocks, stream);
}

}  // namespace pcx
