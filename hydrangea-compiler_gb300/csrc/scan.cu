// scan.cu -- scan / scan_inclusive / scanr / scanr_inclusive with (+).
//
// Replaces the serial LoopFold of lowerScanFamily (Lowering.hs:3563-3612; the
// C backend never parallelises a fold, Parallelize.hs:517).
//
// int64: single-pass decoupled look-back (Merrill & Garland, "Single-pass
// Parallel Prefix Scan with Decoupled Look-back", 2016).  Tiles of 4096
// elements take their id from an atomic counter in launch order, so every
// predecessor a tile waits on has already started; a tile publishes its
// aggregate, a warp looks back 32 predecessors at a time, then publishes its
// inclusive prefix.  A tile's status is one 16-byte {flag, value} word
// (TileWord), written and read whole, so a look-back window costs one memory
// round trip.  Every spin is bounded (error bit, no hang).  int64 adds wrap
// and commute, so the result is bit-identical to the serial C fold.  One
// read and one write per element: 16 B/element of HBM traffic.
//
// float64: single pass, deterministic in two levels.  Within a block of 32
// tiles a tile's prefix over its block-mates comes from a fixed warp scan of
// their aggregates; across blocks the block totals are folded left to right
// through the same kind of look-back (lookback_fold).  Every value is defined
// by the data alone, not by timing: results are run-to-run identical.  Within
// a tile the order is fixed too (per-thread serial sums, a fixed shuffle
// tree).  A parallel prefix cannot reproduce the serial fold's roundings; the
// tolerance is |gpu - c| <= 1e-12 * prefix sum of |x| (stated in the tests).
//
// Tiles pass through shared memory padded with one slot per 16 elements, so
// the blocked (8 consecutive elements per thread) and striped accesses are
// free of bank conflicts.
//
// Reverse scans read and write index n-1-k for logical position k, exactly the
// ix the reference's lowering computes.
#include "hyd_common.cuh"

namespace hyd {

constexpr int kScanT = 512;
constexpr int kScanIPT = 8;
constexpr int kScanTile = kScanT * kScanIPT;  // 4096 (32 KiB of static shared memory for int64)
constexpr int kScanCtasPerSm = 4;  // resident CTAs per SM (32 registers per thread)
// Tiles sit in shared memory with one 8-byte pad after every 16 elements: a
// thread's blocked run of 8 (stride 64 B between lanes) and the striped
// accesses then both meet no bank conflict.  Unpadded, the blocked accesses
// were 16-way conflicted and the tile copy alone ran at half the copy rate.
constexpr int kScanTileP = kScanTile + kScanTile / 16;
__device__ __forceinline__ int scan_pad(int i) { return i + (i >> 4); }

// --- block-wide exclusive scan of one value per thread (int64, wrapping) ------
template <class T>
__device__ __forceinline__ T block_exclusive_scan(T v, T* sh /*[32]*/, T& total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    T incl = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        T y = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += y;
    }
    if (lane == 31) sh[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        T w = lane < nw ? sh[lane] : T(0);
        T wi = w;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            T y = __shfl_up_sync(0xffffffffu, wi, d);
            if (lane >= d) wi += y;
        }
        sh[lane] = wi - w;  // exclusive warp offsets
        if (lane == 31) sh[32] = wi;
    }
    __syncthreads();
    total = sh[32];
    T r = sh[warp] + incl - v;
    __syncthreads();
    return r;
}

// The same for float64, without the subtraction the integer form uses for the
// exclusive value (one FP64 operation fewer per thread; the FP64 pipe bounds
// the float64 scan): the exclusive value of a lane is its left neighbour's
// inclusive one.  Fixed order, so run-to-run identical.
template <class T>
__device__ __forceinline__ T block_exclusive_scan_shift(T v, T* sh /*[33]*/, T& total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    T incl = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const T y = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl = y + incl;
    }
    if (lane == 31) sh[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        const T w = lane < nw ? sh[lane] : T(0);
        T wi = w;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const T y = __shfl_up_sync(0xffffffffu, wi, d);
            if (lane >= d) wi = y + wi;
        }
        const T wx = __shfl_up_sync(0xffffffffu, wi, 1);
        sh[lane] = lane == 0 ? T(0) : wx;  // exclusive warp offsets
        if (lane == 31) sh[32] = wi;
    }
    __syncthreads();
    total = sh[32];
    const T lx = __shfl_up_sync(0xffffffffu, incl, 1);
    const T r = lane == 0 ? sh[warp] : sh[warp] + lx;
    __syncthreads();
    return r;
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

// ---- int64 decoupled look-back ----------------------------------------------------
// One TileWord per tile (flag 0 none, 1 aggregate, 2 inclusive prefix).
struct ScanStatus {
    TileWord* word;
    unsigned* tile_counter;
};

__global__ void __launch_bounds__(kScanT, kScanCtasPerSm) scan_i64_lookback_kernel(const long long* __restrict__ in,
                                                                    long long* __restrict__ out, int64_t n,
                                                                    long long init, bool reverse,
                                                                    bool inclusive, ScanStatus st,
                                                                    unsigned* err) {
    __shared__ long long sh_tile[kScanTileP];
    __shared__ long long sh_scan[33];
    __shared__ unsigned sh_tile_id;
    __shared__ long long sh_prefix;
    if (threadIdx.x == 0) sh_tile_id = atomicAdd(st.tile_counter, 1u);
    __syncthreads();
    const unsigned tile = sh_tile_id;
    const int64_t base = (int64_t)tile * kScanTile;

    long long items[kScanIPT];
    tile_load(in, n, base, reverse, sh_tile, items);
    long long tsum = 0;
#pragma unroll
    for (int j = 0; j < kScanIPT; ++j) tsum += items[j];
    long long agg;
    const long long texcl = block_exclusive_scan(tsum, sh_scan, agg);

    // publish and look back (warp 0)
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        if (tile == 0) {
            if (lane == 0) {
                tile_word_store(&st.word[0], 2ull, to_bits(init + agg));
                sh_prefix = init;
            }
        } else {
            if (lane == 0) tile_word_store(&st.word[tile], 1ull, to_bits(agg));
            long long running = 0;
            int64_t p = (int64_t)tile - 1;  // window covers p, p-1, ..., p-31
            for (;;) {
                const int64_t q = p - lane;
                // wait until every tile of the window has published something
                unsigned long long bits;
                const unsigned f = lookback_wait_words(st.word, p, lane, bits);
                if (f == 0u) {
                    if (lane == 0) raise_error(err, ERRBIT_TIMEOUT);
                    break;
                }
                const unsigned incl_mask = __ballot_sync(0xffffffffu, f == 2u);
                // nearest predecessor with an inclusive prefix (lowest lane):
                // the aggregates of the lanes before it, then its prefix (before
                // tile 0: the fold's initial value)
                const int stop = incl_mask ? (__ffs(incl_mask) - 1) : 32;
                long long v = 0;
                if (lane <= stop) v = q >= 0 ? from_bits<long long>(bits) : init;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                running += v;
                if (stop < 32) break;
                p -= 32;
            }
            if (lane == 0) {
                tile_word_store(&st.word[tile], 2ull, to_bits(running + agg));
                sh_prefix = running;
            }
        }
    }
    __syncthreads();
    long long acc = sh_prefix + texcl;
#pragma unroll
    for (int j = 0; j < kScanIPT; ++j) {
        const long long x = items[j];
        if (inclusive) {
            acc += x;
            items[j] = acc;
        } else {
            items[j] = acc;
            acc += x;
        }
    }
    tile_store(out, n, base, reverse, sh_tile, items);
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
                                                            FoldStatus<T> bst, unsigned* err) {
    __shared__ T sh_tile[kScanTileP];
    __shared__ T sh_scan[33];
    __shared__ T sh_fold[kFoldBuf];
    __shared__ unsigned sh_tile_id;
    __shared__ T sh_prefix;
    if (threadIdx.x == 0) sh_tile_id = atomicAdd(st.tile_counter, 1u);
    __syncthreads();
    const unsigned tile = sh_tile_id;
    const int64_t base = (int64_t)tile * kScanTile;
    T items[kScanIPT];
    tile_load(in, n, base, reverse, sh_tile, items);
    // the thread's running sums, in place: items[j] = x_0 + ... + x_j
#pragma unroll
    for (int j = 1; j < kScanIPT; ++j) items[j] = items[j - 1] + items[j];
    T agg;
    const T texcl = block_exclusive_scan_shift(items[kScanIPT - 1], sh_scan, agg);
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        const int64_t blk = tile >> 5;
        const int pos = (int)(tile & 31u);
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
        T sc = lane < pos ? from_bits<T>(bits) : (lane == pos ? agg : T(0));
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const T y = __shfl_up_sync(0xffffffffu, sc, d);
            if (lane >= d) sc = y + sc;
        }
        const T within = __shfl_sync(0xffffffffu, sc, pos > 0 ? pos - 1 : 0);
        const T total = __shfl_sync(0xffffffffu, sc, 31);
        if (pos == 31 && lane == 0) tile_word_store(&bst.word[blk], 1ull, to_bits(total));
        T before = init;  // B(blk - 1)
        if (!lookback_fold(bst, blk, init, sh_fold, before) && lane == 0) raise_error(err, ERRBIT_TIMEOUT);
        if (pos == 31 && lane == 0) tile_word_store(&bst.word[blk], 2ull, to_bits(before + total));
        if (lane == 0) sh_prefix = pos == 0 ? before : before + within;
    }
    __syncthreads();
    // outputs: the thread's prefix plus its running sums (one addition each)
    const T p = sh_prefix + texcl;
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
// Scratch bytes the decoupled look-back needs for n elements.
size_t scan_i64_scratch_bytes(int64_t n) {
    const int64_t ntiles = (n + kScanTile - 1) / kScanTile;
    return sizeof(TileWord) * (size_t)ntiles + 256;  // + room to align the words to 16 bytes
}

// int64 scan with caller-provided status scratch (scan_i64_scratch_bytes(n))
// and a 4-byte tile counter; both are reset here on the stream.
int scan_i64_launch_with(const long long* in, long long* out, int64_t n, long long init, bool reverse,
                         bool inclusive, void* status_scratch, unsigned* tile_counter, cudaStream_t stream) {
    if (n == 0) return HYD_CUDA_OK;
    Device* d = nullptr;
    HYD_TRY(device(&d));
    const int64_t ntiles = (n + kScanTile - 1) / kScanTile;
    ScanStatus st;
    st.word = reinterpret_cast<TileWord*>((reinterpret_cast<uintptr_t>(status_scratch) + 15) & ~(uintptr_t)15);
    st.tile_counter = tile_counter;
    HYD_CUDA_TRY(cudaMemsetAsync(st.word, 0, sizeof(TileWord) * (size_t)ntiles, stream));
    HYD_CUDA_TRY(cudaMemsetAsync(st.tile_counter, 0, 4, stream));
    scan_i64_lookback_kernel<<<(unsigned)ntiles, kScanT, 0, stream>>>(in, out, n, init, reverse, inclusive, st,
                                                                       d->d_err);
    return launch_check("scan_i64");
}

// Same, with scratch from the stream's workspace.
int scan_i64_launch(const long long* in, long long* out, int64_t n, long long init, bool reverse,
                    bool inclusive, cudaStream_t stream) {
    if (n == 0) return HYD_CUDA_OK;
    unsigned* counters = nullptr;
    void* scratch = nullptr;
    HYD_TRY(workspace(stream, scan_i64_scratch_bytes(n), &counters, &scratch));
    return scan_i64_launch_with(in, out, n, init, reverse, inclusive, scratch, counters + 8, stream);
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
    FoldStatus<double> st, bst;
    HYD_TRY(fold_status(s, ntiles, &st, &bst));
    scan_fold_kernel<double><<<(unsigned)ntiles, kScanT, 0, s>>>(in, out, n, init, reverse != 0, inclusive != 0, st,
                                                                 bst, d->d_err);
    return launch_check("scan_f64");
}
