// scan.cu -- scan / scan_inclusive / scanr / scanr_inclusive with (+).
//
// Replaces the serial LoopFold of lowerScanFamily (Lowering.hs:3563-3612; the
// C backend never parallelises a fold, Parallelize.hs:517).
//
// int64: two launches over contiguous ranges, one per warp: the ranges' sums,
// then the scans.  int64 adds wrap and commute, so the result is bit-identical
// to the serial C fold.  Measured against the single-pass look-back this took
// the place of (start -> now): 2^22 elements 30.3 -> 22.6 us, 2e7 94 -> 84 us,
// 2^27 540 -> 512 us; 24 bytes of traffic per element bound it.  float64 takes
// the same form up to 2^17 elements (12.3 -> 10.2 us); above, its third pass of
// FP64 additions costs more than the look-back (1e6: 28.7 against 16.9 us).
//
// float64 above that: single pass, a decoupled look-back (Merrill & Garland,
// "Single-pass Parallel Prefix Scan with Decoupled Look-back", 2016),
// deterministic in two levels.  Tiles of 4096 elements take their id from an
// atomic counter in launch order, so every predecessor a tile waits on has
// already started.  A tile's status is one 16-byte {flag, value} word
// (TileWord), written and read whole, so a look-back window costs one memory
// round trip.  Every spin is bounded (error bit, no hang).  Within a block of 32
// tiles a tile's prefix over its block-mates comes from a fixed warp scan of
// their aggregates; across blocks the block totals are folded left to right
// through the same kind of look-back (lookback_fold).  Every value is defined
// by the data alone, not by timing: results are run-to-run identical.  Within
// a tile the order is fixed too (per-thread serial sums, a fixed shuffle
// tree).  A parallel prefix cannot reproduce the serial fold's roundings; the
// tolerance is |gpu - c| <= 1e-12 * prefix sum of |x| (stated in the tests).
// FP64 bounds it: 2.3 additions per element (15 + 5 + 2 + 16 per thread of 16),
// 586 us of the 735 us at 2^27 (812 with 8 per thread, 2.6 additions, the two
// levels of the look-back one after the other and no prefetch).  The chains of 16
// do not show in the errors, whose size the few additions to the whole prefix
// set: largest one of 2^24 positive elements 4.5 units of 2^-53 of the last value
// with 8 per thread, 4.4 now.
//
// Tiles pass through shared memory padded with one slot per 16 elements, so
// the blocked (16 consecutive elements per thread, 8 per lane in the two-launch
// form) and striped accesses are free of bank conflicts.
//
// Reverse scans read and write index n-1-k for logical position k, exactly the
// ix the reference's lowering computes.
#include "hyd_common.cuh"

namespace hyd {

constexpr int kScanT = 256;
constexpr int kScanWarps = kScanT / 32;
constexpr int kScanIPT = 16;
constexpr int kScanTile = kScanT * kScanIPT;  // 4096
constexpr int kScanCtasPerSm = 4;  // resident CTAs per SM (64 registers per thread)
// Tiles sit in shared memory with one 8-byte pad after every 16 elements: a
// thread's blocked run of 16 (an odd stride between lanes) and the striped
// accesses then both meet no bank conflict.  Unpadded, the blocked accesses
// were 16-way conflicted and the tile copy alone ran at half the copy rate.
constexpr int kScanTileP = kScanTile + kScanTile / 16;
__device__ __forceinline__ int scan_pad(int i) { return i + (i >> 4); }

// Inclusive scan of one value per lane, fixed order.
template <class T>
__device__ __forceinline__ T warp_inclusive_scan(T v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const T y = __shfl_up_sync(0xffffffffu, v, d);
        if (lane >= d) v = y + v;
    }
    return v;
}
// Warp 0: the exclusive prefixes of the warps' totals (lane w gets warp w's,
// computed without a subtraction) and the block's total.
template <class T>
__device__ __forceinline__ T scan_warp_totals(const T* totals, T& total) {
    const int lane = threadIdx.x & 31;
    T w = lane < kScanWarps ? totals[lane] : T(0);
#pragma unroll
    for (int d = 1; d < kScanWarps; d <<= 1) {
        const T y = __shfl_up_sync(0xffffffffu, w, d);
        if (lane >= d) w = y + w;
    }
    total = __shfl_sync(0xffffffffu, w, kScanWarps - 1);
    const T x = __shfl_up_sync(0xffffffffu, w, 1);
    return lane == 0 ? T(0) : x;
}

// Tile load/store in blocked arrangement through shared memory: global
// accesses are coalesced, each thread then owns kScanIPT consecutive logical
// elements.  Logical position k maps to physical index (reverse ? n-1-k : k).
template <class T>
__device__ __forceinline__ void tile_load(const T* in, int64_t n, int64_t base, bool reverse, T* sh,
                                          T (&items)[kScanIPT]) {
    T v[kScanIPT];
#pragma unroll
    for (int j = 0; j < kScanIPT; ++j) {  // all loads in flight before the first store
        const int64_t k = base + threadIdx.x + j * kScanT;
        v[j] = k < n ? in[reverse ? (n - 1 - k) : k] : T(0);
    }
#pragma unroll
    for (int j = 0; j < kScanIPT; ++j) sh[scan_pad(threadIdx.x + j * kScanT)] = v[j];
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kScanIPT; ++j) items[j] = sh[scan_pad(threadIdx.x * kScanIPT + j)];
    __syncthreads();
}

// Brings the tile `ahead` tiles further on into L2: a tile's look-back waits for
// the slowest load among the tiles in flight before it, and L2 hits vary less
// (755 -> 744 us at 2^27, one wave of tiles ahead).
template <class T>
__device__ __forceinline__ void tile_prefetch(const T* in, int64_t n, int64_t base, int64_t ahead, bool reverse) {
    const int64_t k = base + ahead * kScanTile;
    if (k >= n) return;
    const int64_t cnt = n - k < kScanTile ? n - k : kScanTile;
    l2_prefetch(in + (reverse ? n - k - cnt : k), cnt * (int64_t)sizeof(T));
}

template <class T>
__device__ __forceinline__ void tile_store(T* out, int64_t n, int64_t base, bool reverse, T* sh,
                                           const T (&items)[kScanIPT]) {
#pragma unroll
    for (int j = 0; j < kScanIPT; ++j) sh[scan_pad(threadIdx.x * kScanIPT + j)] = items[j];
    __syncthreads();
    for (int i = threadIdx.x; i < kScanTile; i += kScanT) {
        const int64_t k = base + i;
        if (k < n) out[reverse ? (n - 1 - k) : k] = sh[scan_pad(i)];
    }
}

// ---- two launches: sums, then scans ---------------------------------------------
// Every warp takes one contiguous range of the elements, in steps of 256.  The
// first launch sums the ranges (no output); in the second a warp adds up the
// sums of the ranges before its own and scans its range step by step, carrying
// the prefix along.  24 bytes per element instead of the look-back's 16, but
// no tile waits for another: with a look-back a tile spent 40% of its time on
// the slowest of the 600 tiles in flight before it.
constexpr int kRangeT = 256;
constexpr int kRangeWarps = kRangeT / 32;
constexpr int kRangePer = 8;                   // elements per lane and step
constexpr int kRangeStep = 32 * kRangePer;
constexpr int kRangeCtasPerSm = 4;
constexpr int64_t kScanRangesF64 = 1 << 17;
constexpr int kRangeSlots = kRangeStep + kRangeStep / 16;
// per-warp staging, one 8-byte pad after every 16: blocked and striped accesses
// are both free of bank conflicts

// Elements k0 + lane + 32 j (logical positions; past `end` zero).
template <class T>
__device__ __forceinline__ void range_load(const T* __restrict__ in, int64_t n, int64_t k0, int64_t end, bool reverse,
                                           T (&v)[kRangePer]) {
    const int lane = threadIdx.x & 31;
    const T* const p = reverse ? in + (n - 1 - k0) - lane : in + k0 + lane;
    if (k0 + kRangeStep <= end) {
        if (reverse) {
#pragma unroll
            for (int j = 0; j < kRangePer; ++j) v[j] = __ldg(p - 32 * j);
        } else {
#pragma unroll
            for (int j = 0; j < kRangePer; ++j) v[j] = __ldg(p + 32 * j);
        }
    } else {
#pragma unroll
        for (int j = 0; j < kRangePer; ++j)
            v[j] = k0 + lane + 32 * j < end ? __ldg(reverse ? p - 32 * j : p + 32 * j) : T(0);
    }
}

template <class T>
__global__ void __launch_bounds__(kRangeT, kRangeCtasPerSm)
    scan_sums_kernel(const T* __restrict__ in, int64_t n, bool reverse, int64_t range, T* __restrict__ sums) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int64_t w = (int64_t)blockIdx.x * kRangeWarps + (threadIdx.x >> 5);
    const int64_t lo = w * range, end = lo + range < n ? lo + range : n;
    T acc[kRangePer];
#pragma unroll
    for (int j = 0; j < kRangePer; ++j) acc[j] = T(0);
    // from the range's end to its start: what was read last is still in L2 when
    // the second launch reads it first
    int64_t k = end > lo ? lo + (end - lo - 1) / kRangeStep * kRangeStep : lo - kRangeStep;
    for (; k > lo; k -= 2 * kRangeStep) {
        T a[kRangePer], b[kRangePer];
        range_load(in, n, k, end, reverse, a);
        range_load(in, n, k - kRangeStep, end, reverse, b);
#pragma unroll
        for (int j = 0; j < kRangePer; ++j) acc[j] += a[j];
#pragma unroll
        for (int j = 0; j < kRangePer; ++j) acc[j] += b[j];
    }
    if (k == lo) {
        T a[kRangePer];
        range_load(in, n, k, end, reverse, a);
#pragma unroll
        for (int j = 0; j < kRangePer; ++j) acc[j] += a[j];
    }
    T s = ((acc[0] + acc[1]) + (acc[2] + acc[3])) + ((acc[4] + acc[5]) + (acc[6] + acc[7]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) sums[w] = s;
}

template <class T>
__global__ void __launch_bounds__(kRangeT, kRangeCtasPerSm)
    scan_ranges_kernel(const T* __restrict__ in, T* __restrict__ out, int64_t n, T init, bool reverse, bool inclusive,
                       int64_t range, const T* __restrict__ sums) {
    __shared__ T sh[kRangeWarps][kRangeSlots];
    __shared__ T sh_part[kRangeWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    T* const st = sh[warp];
    const int64_t w = (int64_t)blockIdx.x * kRangeWarps + warp;
    const int64_t lo = w * range, end = lo + range < n ? lo + range : n;
    T v[kRangePer];
    if (lo < end) range_load(in, n, lo, end, reverse, v);  // does not depend on the sums
    asm volatile("griddepcontrol.wait;" ::: "memory");
    // the sums of all ranges before this block's (fixed order), then before this warp's
    T part = T(0);
    for (int64_t u = threadIdx.x; u < (int64_t)blockIdx.x * kRangeWarps; u += kRangeT) part += __ldcg(sums + u);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
    if (lane == 0) sh_part[warp] = part;
    __syncthreads();
    // the prefix is `carry` plus, for the first step, `near`: every addition to the
    // whole prefix rounds at its size, so the small sums are added to each other first
    static_assert(kRangeWarps == 8, "the sum below");
    T carry = init + (((sh_part[0] + sh_part[1]) + (sh_part[2] + sh_part[3])) +
                      ((sh_part[4] + sh_part[5]) + (sh_part[6] + sh_part[7])));
    T near = T(0);
    for (int u = 0; u < warp; ++u) near += __ldcg(sums + (int64_t)blockIdx.x * kRangeWarps + u);
    for (int64_t k = lo; k < end; k += kRangeStep) {
        // to blocked: lane l then holds elements k + 8l .. k + 8l + 7
#pragma unroll
        for (int j = 0; j < kRangePer; ++j) st[scan_pad(lane + 32 * j)] = v[j];
        __syncwarp();
        T x[kRangePer];
#pragma unroll
        for (int j = 0; j < kRangePer; ++j) x[j] = st[scan_pad(kRangePer * lane + j)];
        __syncwarp();
        if (k + kRangeStep < end) range_load(in, n, k + kRangeStep, end, reverse, v);  // the next step's
#pragma unroll
        for (int j = 1; j < kRangePer; ++j) x[j] = x[j - 1] + x[j];
        const T incl = warp_inclusive_scan(x[kRangePer - 1]);
        const T left = __shfl_up_sync(0xffffffffu, incl, 1);
        const T p = carry + (lane == 0 ? near : near + left);
        carry = carry + (near + __shfl_sync(0xffffffffu, incl, 31));
        near = T(0);
        if (inclusive) {
#pragma unroll
            for (int j = 0; j < kRangePer; ++j) x[j] = p + x[j];
        } else {
#pragma unroll
            for (int j = kRangePer - 1; j > 0; --j) x[j] = p + x[j - 1];
            x[0] = p;
        }
#pragma unroll
        for (int j = 0; j < kRangePer; ++j) st[scan_pad(kRangePer * lane + j)] = x[j];
        __syncwarp();
#pragma unroll
        for (int j = 0; j < kRangePer; ++j) {
            const int64_t q = k + lane + 32 * j;
            if (q < end) out[reverse ? n - 1 - q : q] = st[scan_pad(lane + 32 * j)];
        }
        __syncwarp();
    }
}

// Blocks, and the launches (`scratch`: one 8-byte word per warp).
static int64_t range_blocks(const Device* d, int64_t n) {
    const int64_t want = (n + kRangeStep * kRangeWarps - 1) / (kRangeStep * kRangeWarps);
    const int64_t cap = (int64_t)d->sm_count * kRangeCtasPerSm;
    return want < cap ? want : cap;
}
template <class T>
static int scan_ranges_launch(const T* in, T* out, int64_t n, T init, bool reverse, bool inclusive, void* scratch,
                              cudaStream_t stream, const char* what) {
    Device* d = nullptr;
    HYD_TRY(device(&d));
    const int64_t blocks = range_blocks(d, n), warps = blocks * kRangeWarps;
    const int64_t steps = (n + kRangeStep - 1) / kRangeStep;
    const int64_t range = (steps + warps - 1) / warps * kRangeStep;
    T* const sums = static_cast<T*>(scratch);
    scan_sums_kernel<T><<<(unsigned)blocks, kRangeT, 0, stream>>>(in, n, reverse, range, sums);
    HYD_TRY(launch_check(what));
    // programmatic dependent launch: the scans' blocks load their first steps
    // while the sums finish
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3(kRangeT);
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    HYD_CUDA_TRY(cudaLaunchKernelEx(&cfg, scan_ranges_kernel<T>, in, out, n, init, reverse, inclusive, range,
                                    (const T*)sums));
    return launch_check(what);
}

// ---- deterministic decoupled look-back (left fold) -----------------------------------
// One TileWord per tile (flag 0 none, 1 aggregate, 2 inclusive prefix; T's
// bits as the value).
template <class T>
struct FoldStatus {
    TileWord* word;
    unsigned* tile_counter;
};
constexpr int kFoldBuf = 1024;                // aggregates one look-back may collect before it restarts
constexpr unsigned kFoldRestarts = 1u << 12;  // restarts before a look-back gives up

// Warp-wide (all 32 lanes of one warp).  The exclusive prefix of `tile`, as
// the left fold inclusive[s] + aggregate[s+1] + ... + aggregate[tile-1] where s
// is the nearest predecessor that has published an inclusive value (`before`
// stands for the inclusive value of tile -1).  Every inclusive value is made
// the same way, so the result is the left fold of all earlier aggregates,
// whatever the timing.
// Aggregates are collected in sbuf (kFoldBuf); when the nearest inclusive
// predecessor is further back than that, the look-back starts again from
// tile - 1 (nearer prefixes will have appeared by then).  Returns false on
// every lane when a wait ran out.
template <class T>
__device__ bool lookback_fold(const FoldStatus<T>& st, int64_t tile, T before, T* sbuf, T& prefix) {
    const int lane = threadIdx.x & 31;
    unsigned restarts = 0;
    int64_t p = tile - 1;
    int cnt = 0;
    T base = before;
    for (;;) {
        unsigned long long bits;
        const unsigned f = lookback_wait_words(st.word, p, lane, bits);
        if (f == 0u) return false;
        const int64_t q = p - lane;
        const unsigned incl = __ballot_sync(0xffffffffu, f == 2u);
        const int stop = incl ? __ffs(incl) - 1 : 32;
        if (lane < stop) sbuf[cnt + lane] = from_bits<T>(bits);  // aggregates, nearest first
        if (stop < 32) {
            const T b = q >= 0 ? from_bits<T>(bits) : before;
            base = __shfl_sync(0xffffffffu, b, stop);
            cnt += stop;
            break;
        }
        cnt += 32;
        p -= 32;
        if (cnt + 32 > kFoldBuf) {
            if (++restarts > kFoldRestarts) return false;
            cnt = 0;
            p = tile - 1;
            __nanosleep(256);
        }
    }
    __syncwarp();
    T acc = base;
    if (lane == 0)
        for (int i = cnt - 1; i >= 0; --i) acc = acc + sbuf[i];
    prefix = __shfl_sync(0xffffffffu, acc, 0);
    return true;
}

// float64 (and any T) scan, deterministic in two levels.  Tiles form blocks
// of 32 (block k = tiles 32k .. 32k+31):
//  * within a block, tile i's prefix over its block-mates is the value at lane
//    i-1 of a warp inclusive scan (fixed shuffle tree) of the block's tile
//    aggregates, and the block total T(k) is its lane-31 value;
//  * across blocks, B(k) = the left fold of T(0), ..., T(k) onto init, found
//    through lookback_fold over per-block status words (the last tile of a
//    block publishes T(k), then B(k));
//  * the tile's exclusive prefix is B(k-1) + (its within-block prefix).
// Every value is defined by the data alone, not by timing, so results are
// run-to-run identical.  A single-level left fold over tile aggregates puts
// one dependent FP64 add per tile on the scan's critical path (about 76
// cycles each on this part: 1.3 ms at 2^27); here the dependent chain is one
// add per block of 32 tiles.
template <class T>
__global__ void __launch_bounds__(kScanT, kScanCtasPerSm) scan_fold_kernel(const T* __restrict__ in, T* __restrict__ out, int64_t n,
                                                            T init, bool reverse, bool inclusive, FoldStatus<T> st,
                                                            FoldStatus<T> bst, int ahead, unsigned* err) {
    __shared__ T sh_tile[kScanTileP];
    __shared__ T sh_total[kScanWarps];  // the warps' totals, then their offsets in the tile
    __shared__ T sh_fold[kFoldBuf];
    __shared__ unsigned sh_tile_id;
    __shared__ T sh_before;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        sh_tile_id = atomicAdd(st.tile_counter, 1u);
        tile_prefetch(in, n, (int64_t)sh_tile_id * kScanTile, ahead, reverse);
    }
    __syncthreads();
    const unsigned tile = sh_tile_id;
    const int64_t base = (int64_t)tile * kScanTile;
    const int64_t blk = tile >> 5;
    const int pos = (int)(tile & 31u);
    T items[kScanIPT];
    tile_load(in, n, base, reverse, sh_tile, items);
    // the thread's running sums, in place: items[j] = x_0 + ... + x_j
#pragma unroll
    for (int j = 1; j < kScanIPT; ++j) items[j] = items[j - 1] + items[j];
    const T incl = warp_inclusive_scan(items[kScanIPT - 1]);
    if (lane == 31) sh_total[warp] = incl;
    __syncthreads();
    T off = T(0), total = T(0), within = T(0);  // (within: of the block's tiles before this one)
    if (warp == 0) {
        T agg;
        off = scan_warp_totals(sh_total, agg);
        if (lane == 0) tile_word_store(&st.word[tile], 1ull, to_bits(agg));
        // the aggregates of the block's tiles before this one (earlier tickets)
        unsigned long long f = 1ull, bits = 0ull;
        if (lane < pos) tile_word_load(&st.word[(blk << 5) + lane], f, bits);
        unsigned spins = 0;
        bool ok = true;
        while (__any_sync(0xffffffffu, f == 0ull)) {
            if (++spins > kSpinLimit) {
                ok = false;
                break;
            }
            if (f == 0ull) tile_word_load(&st.word[(blk << 5) + lane], f, bits);
        }
        if (!ok && lane == 0) raise_error(err, ERRBIT_TIMEOUT);
        const T sc = warp_inclusive_scan(lane < pos ? from_bits<T>(bits) : (lane == pos ? agg : T(0)));
        within = __shfl_sync(0xffffffffu, sc, pos > 0 ? pos - 1 : 0);
        total = __shfl_sync(0xffffffffu, sc, 31);
        if (lane == 0 && pos == 31) tile_word_store(&bst.word[blk], 1ull, to_bits(total));
    } else if (warp == 1) {
        T before = init;  // B(blk - 1)
        if (!lookback_fold(bst, blk, init, sh_fold, before) && lane == 0) raise_error(err, ERRBIT_TIMEOUT);
        if (lane == 0) sh_before = before;
    }
    __syncthreads();
    if (warp == 0) {
        const T before = sh_before;
        if (pos == 31 && lane == 0) tile_word_store(&bst.word[blk], 2ull, to_bits(before + total));
        // the two small sums first: an addition to the whole prefix rounds at its size
        if (lane < kScanWarps) sh_total[lane] = before + (pos == 0 ? off : within + off);
    }
    __syncthreads();
    // outputs: the thread's prefix plus its running sums (one addition each)
    const T left = __shfl_up_sync(0xffffffffu, incl, 1);
    const T p = lane == 0 ? sh_total[warp] : sh_total[warp] + left;
    if (inclusive) {
#pragma unroll
        for (int j = 0; j < kScanIPT; ++j) items[j] = p + items[j];
    } else {
#pragma unroll
        for (int j = kScanIPT - 1; j > 0; --j) items[j] = p + items[j - 1];
        items[0] = p;
    }
    tile_store(out, n, base, reverse, sh_tile, items);
}

}  // namespace hyd

using namespace hyd;

namespace hyd {
// Scratch bytes of an int64 scan, at most.
size_t scan_i64_scratch_bytes(int64_t n) {
    const int64_t steps = (n + kRangeStep - 1) / kRangeStep + kRangeWarps;
    const int64_t most = 1 << 16;  // more warps than any grid here has
    return sizeof(long long) * (size_t)(steps < most ? steps : most);
}

// int64 scan with caller-provided scratch (scan_i64_scratch_bytes(n)).
int scan_i64_launch_with(const long long* in, long long* out, int64_t n, long long init, bool reverse,
                         bool inclusive, void* scratch, cudaStream_t stream) {
    if (n == 0) return HYD_CUDA_OK;
    return scan_ranges_launch<long long>(in, out, n, init, reverse, inclusive, scratch, stream, "scan_i64");
}

// Same, with scratch from the stream's workspace.
int scan_i64_launch(const long long* in, long long* out, int64_t n, long long init, bool reverse,
                    bool inclusive, cudaStream_t stream) {
    if (n == 0) return HYD_CUDA_OK;
    void* scratch = nullptr;
    HYD_TRY(workspace(stream, scan_i64_scratch_bytes(n), nullptr, &scratch));
    return scan_i64_launch_with(in, out, n, init, reverse, inclusive, scratch, stream);
}
}  // namespace hyd

extern "C" int hyd_cuda_scan_i64(const int64_t* in, int64_t* out, int64_t n, int64_t init, int reverse,
                                 int inclusive, void* stream) {
    HYD_CHECK_ARG(n >= 0, "scan_i64: negative length");
    HYD_CHECK_ARG(n == 0 || (in != nullptr && out != nullptr), "scan_i64: null buffer");
    HYD_CHECK_ARG(n <= (int64_t)kScanTile * 0x7fffffffLL, "scan_i64: too long");
    return scan_i64_launch(reinterpret_cast<const long long*>(in), reinterpret_cast<long long*>(out), n, init,
                           reverse != 0, inclusive != 0, as_stream(stream));
}

// Status scratch of the left-fold look-back for `ntiles` tiles of (at most)
// 8-byte values: [0, 256) the tile counter, then `ntiles` tile words and, when `bst` is given, one word per block
// of 32 tiles; all of it zeroed on the stream (one memset).
template <class T>
static int fold_status(cudaStream_t s, int64_t ntiles, FoldStatus<T>* st, FoldStatus<T>* bst = nullptr) {
    static_assert(sizeof(T) <= 8, "a tile word holds a value of at most 8 bytes");
    const int64_t nblocks = bst ? (ntiles + 31) / 32 : 0;
    const size_t bytes = 256 + sizeof(TileWord) * (size_t)(ntiles + nblocks);
    void* scratch = nullptr;
    HYD_TRY(workspace(s, bytes, nullptr, &scratch));
    unsigned char* b = static_cast<unsigned char*>(scratch);  // 256-byte aligned
    st->tile_counter = reinterpret_cast<unsigned*>(b);
    st->word = reinterpret_cast<TileWord*>(b + 256);
    if (bst) {
        *bst = *st;
        bst->word = st->word + ntiles;
    }
    HYD_CUDA_TRY(cudaMemsetAsync(b, 0, bytes, s));
    return HYD_CUDA_OK;
}

extern "C" int hyd_cuda_scan_f64(const double* in, double* out, int64_t n, double init, int reverse,
                                 int inclusive, void* stream) {
    HYD_CHECK_ARG(n >= 0, "scan_f64: negative length");
    HYD_CHECK_ARG(n == 0 || (in != nullptr && out != nullptr), "scan_f64: null buffer");
    if (n == 0) return HYD_CUDA_OK;
    cudaStream_t s = as_stream(stream);
    const int64_t ntiles = (n + kScanTile - 1) / kScanTile;
    HYD_CHECK_ARG(ntiles <= 0x7fffffffLL, "scan_f64: too long");
    Device* d = nullptr;
    HYD_TRY(device(&d));
    if (n <= kScanRangesF64) {
        void* scratch = nullptr;
        HYD_TRY(workspace(s, scan_i64_scratch_bytes(n), nullptr, &scratch));
        return scan_ranges_launch<double>(in, out, n, init, reverse != 0, inclusive != 0, scratch, s, "scan_f64");
    }
    FoldStatus<double> st, bst;
    HYD_TRY(fold_status(s, ntiles, &st, &bst));
    scan_fold_kernel<double><<<(unsigned)ntiles, kScanT, 0, s>>>(in, out, n, init, reverse != 0, inclusive != 0, st,
                                                                 bst, d->sm_count * kScanCtasPerSm, d->d_err);
    return launch_check("scan_f64");
}
