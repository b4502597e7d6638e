// segsum.cu -- sums over the segments of a contiguous array: segmented_reduce
// (+) and the CSR SpMV with the default row split.
//
// Replaces the LoopSegRedOuter loop of segmented_reduce (Lowering.hs:874-944,
// `schedule(dynamic)` per CodegenC.hs:1055-1057) and the generate-of-
// reduce_generate of bench/spmv/spmv.hyd:30-40.  Both are the same problem: an
// array of values cut by ascending offsets (the segment offsets; row_ptr), one
// sum per piece.  For the SpMV a value is the product vals[k] * x[col[k]].
//
// Every warp takes one contiguous range of values and boundaries (the ends of
// segments), equal shares of the two together whatever the segments' lengths
// and however many of them are empty, and walks it in chunks of 256 values:
//  * a run of chunks with no boundary in it is added
//    into eight accumulators per lane, one operation per value;
//  * a chunk with boundaries is summed by a segmented scan: each lane folds
//    its 8 consecutive values, restarting at each head, one warp scan carries
//    the sums across lanes, and the sum before each boundary is written out;
//  * the sum of the piece that was open when the range began, and of the one
//    open when it ends, go to per-warp partials.
// A second kernel adds the partials of the pieces that cross warps (a warp per
// piece, a fixed order).  There is no look-back, no atomic and no flag to wait
// for; every order is fixed by the data, so results are identical over runs.
//
// What bounds it: FP64.  GB300 adds 5.3e11 doubles/s, 254 us for 2^27, against
// 158 us for reading them.  Measured (start -> now): 2^27 float64 values in
// segments of 2^U(0,16), 695 -> 312 us (3.4 TB/s); segments of 2^U(0,5), 783 ->
// 569 us; of one value each, 1136 -> 932 us.  Before, tiles of 4096 values took
// 1.6 FP64 operations per value and waited for a look-back.  SpMV, 2^20 rows of
// Zipf length, 12.9e6 entries: 198 -> 100 us; 8 lanes per row spent about seven
// FP64 lane slots per entry.  Three blocks per SM (80 registers) beat four (64
// and spills): 1014 against 1327 us on one-value segments when that was tried.
//
// Errors, root mean square in units of 2^-53 of a sum's magnitudes, against
// tiles with a look-back (segments) and 8 lanes per row: segments of 300 positive
// values 0.88 and 0.80, of 10^6 4.4 and 0.77; rows of 12 positive products 0.67
// and 0.73, of Zipf length 0.59 and 0.60, of Zipf length with signs 0.42 and 0.39.
//
// Offsets that are not an ascending partition of [0, n_vals] are detected on
// the way (every adjacent pair is looked at by exactly one warp); the second
// kernel then computes every segment on its own, with the reference's
// semantics (an invalid segment yields init and is reported; a row takes
// whatever its two row pointers span).
#include <climits>

#include "hyd_common.cuh"

namespace hyd {

constexpr int kSegT = 256;
constexpr int kSegWarps = kSegT / 32;
constexpr int kSegPer = 8;                  // consecutive values per lane
constexpr int kSegC = 32 * kSegPer;         // values per chunk
constexpr int kSegAlign = 32;               // a range's first chunk begins at a multiple of this
constexpr int kSegCounterWord = 240;  // of the segmented reduce among the stream's counters
// where a chunk's sum i sits: free of bank conflicts for a lane's 8 consecutive values
__device__ __forceinline__ int seg_slot(int i) { return i ^ ((i >> 4) & 7); }

__device__ __forceinline__ void cp_async_16(void* smem_dst, const void* gsrc, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(smem_dst)),
                 "l"(gsrc), "r"(bytes)
                 : "memory");
}
// 16-byte units of a staged chunk: unit u sits at seg_unit(u), so that the
// lanes' reads of their own consecutive units meet few bank conflicts
__device__ __forceinline__ int seg_unit(int u) { return u ^ ((u >> 3) & 3); }

constexpr int64_t kSegNoBoundary = -1;  // none in the range
constexpr int64_t kSegNoPiece = -2;     // some, but no piece was open at the range's start

// One entry per warp of the first kernel.
template <class T>
struct SegPartials {
    T* head;          // the piece open at the range's start, up to its first boundary
    T* tail;          // after the last boundary (the whole range when it has none)
    int64_t* closes;  // the boundary that ends that first piece; kSegNoBoundary, kSegNoPiece
    unsigned* bad;   // invalid offsets were met
    unsigned* done;  // finished blocks of the second kernel
    unsigned* by_lanes;  // SpMV: not 0: the second kernel takes the rows by lanes, the first does nothing
};

// ---- what a position of the array contributes ---------------------------------
// Plain values; mac() adds one to a running sum.
template <class T>
struct SegPlain {
    static constexpr bool kRows = false;
    static constexpr int kCtasPerSm = 3, kUnroll = 2;  // resident blocks; chunks in flight per warp
    static constexpr int kStageBytes = 0;
    static constexpr int kPos = kSegC + 32;  // boundaries of a chunk kept in shared memory; more are read again
    const T* vals;
    int64_t n;
    bool vec;  // 32-byte aligned base
    int64_t share;  // a warp's, of values and boundaries
    struct Item {
        T x[kSegPer];
    };
    __device__ __forceinline__ int64_t first() const { return 0; }
    __device__ __forceinline__ int64_t end() const { return n; }
    void set_share(int64_t nb, int64_t nwarps) {
        share = (n + nb + nwarps - 1) / nwarps;
        if (share < kSegC) share = kSegC;
    }
    __device__ __forceinline__ bool check(const Item&) const { return true; }
    // positions base + i .. base + i + 7, those with i + j outside [lo, hi) zero
    __device__ __forceinline__ void load(Item& it, int64_t base, int i, int lo, int hi) const {
        const T* const vals = this->vals + base;
        if (vec && i >= lo && i + kSegPer <= hi) {
            const u64x4 a = ldg_stream_u64x4(vals + i), b = ldg_stream_u64x4(vals + i + 4);
            it.x[0] = from_bits<T>(a.x); it.x[1] = from_bits<T>(a.y);
            it.x[2] = from_bits<T>(a.z); it.x[3] = from_bits<T>(a.w);
            it.x[4] = from_bits<T>(b.x); it.x[5] = from_bits<T>(b.y);
            it.x[6] = from_bits<T>(b.z); it.x[7] = from_bits<T>(b.w);
        } else {
#pragma unroll
            for (int j = 0; j < kSegPer; ++j) it.x[j] = i + j >= lo && i + j < hi ? vals[i + j] : T(0);
        }
    }
    __device__ __forceinline__ T mac(const Item& it, int j, T acc) const { return acc + it.x[j]; }
};

// Products vals[k] * x[col[k]]; a column outside [0, ncols) contributes
// nothing and is reported.
template <class C>
struct SegProduct {
    // chunks are staged in shared memory by cp.async, two ahead: the entries'
    // latency is off the chain entries -> x -> sums
    static constexpr bool kRows = true;  // rows of even length may go by lanes ...
    static constexpr float kLanesMean = sizeof(C) == 8 ? 16.0f : 20.0f;  // ... from this many entries on average
    static constexpr int kCtasPerSm = 3, kUnroll = 1;
    static constexpr int kStageBytes = kSegC * (8 + (int)sizeof(C));  // values, then columns
    // none: three blocks of two staged chunks per warp just fit the 196 KB
    // setting of shared memory, which leaves 60 KB of L1 for x (at the 228 KB
    // setting, 28 KB of L1, the 2^20-row case took 142 us instead of 108)
    static constexpr int kPos = 0;
    const C* cols;
    const double* vals;
    const double* x;
    const long long* row_ptr;
    int64_t nrows, ncols;
    bool vec;
    struct Item {
        double v[kSegPer], x[kSegPer];
        bool ok;
    };
    __device__ __forceinline__ int64_t first() const { return row_ptr[0]; }
    __device__ __forceinline__ int64_t end() const { return row_ptr[nrows]; }
    static constexpr int64_t share = 0;  // the device knows
    void set_share(int64_t, int64_t) {}
    __device__ __forceinline__ bool check(const Item& it) const { return it.ok; }
    __device__ __forceinline__ void load(Item& it, int64_t base, int i, int lo, int hi) const {
        const C* const cols = this->cols + base;
        const double* const vals = this->vals + base;
        unsigned long long c[kSegPer];
        if (vec && i >= lo && i + kSegPer <= hi) {
            if (sizeof(C) == 8) {
                const u64x4 a = ldg_stream_u64x4(cols + i), b = ldg_stream_u64x4(cols + i + 4);
                c[0] = a.x; c[1] = a.y; c[2] = a.z; c[3] = a.w;
                c[4] = b.x; c[5] = b.y; c[6] = b.z; c[7] = b.w;
            } else {
                const u64x4 a = ldg_stream_u64x4(cols + i);
                const unsigned long long w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    c[2 * j] = (unsigned long long)(long long)(int)(unsigned)w[j];
                    c[2 * j + 1] = (unsigned long long)(long long)(int)(unsigned)(w[j] >> 32);
                }
            }
            const f64x4 p = ldg_stream_f64x4(vals + i), q = ldg_stream_f64x4(vals + i + 4);
            it.v[0] = p.x; it.v[1] = p.y; it.v[2] = p.z; it.v[3] = p.w;
            it.v[4] = q.x; it.v[5] = q.y; it.v[6] = q.z; it.v[7] = q.w;
        } else {
#pragma unroll
            for (int j = 0; j < kSegPer; ++j) {
                const bool in = i + j >= lo && i + j < hi;
                c[j] = in ? (unsigned long long)(long long)cols[i + j] : 0ull;
                it.v[j] = in ? vals[i + j] : 0.0;
            }
        }
        it.ok = true;
#pragma unroll
        for (int j = 0; j < kSegPer; ++j) {
            const bool in = i + j >= lo && i + j < hi;
            const bool ok = c[j] < (unsigned long long)ncols;
            it.x[j] = in && ok ? __ldg(x + c[j]) : 0.0;
            if (!ok) it.v[j] = 0.0;
            it.ok &= ok || !in;
        }
    }
    __device__ __forceinline__ void stage(unsigned char* buf, int64_t base, int p, int lo, int hi) const {
        const int lane = threadIdx.x & 31;
        if (vec) {
            // a unit that begins before `lo` is fetched whole (lo is inside the array)
            const double* const gv = vals + base + p;
            const C* const gc = cols + base + p;
            constexpr int kPerV = 2, kPerC = 16 / (int)sizeof(C);
#pragma unroll
            for (int k = 0; k < kSegC / kPerV / 32; ++k) {
                const int u = lane + 32 * k, left = hi - (p + kPerV * u);
                if (left > 0 && p + kPerV * (u + 1) > lo)
                    cp_async_16(buf + 16 * seg_unit(u), gv + kPerV * u, left >= kPerV ? 16 : left * 8);
            }
#pragma unroll
            for (int k = 0; k < kSegC / kPerC / 32; ++k) {
                const int u = lane + 32 * k, left = hi - (p + kPerC * u);
                if (left > 0 && p + kPerC * (u + 1) > lo)
                    cp_async_16(buf + kSegC * 8 + 16 * seg_unit(u), gc + kPerC * u,
                                left >= kPerC ? 16 : left * (int)sizeof(C));
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    __device__ __forceinline__ void load_staged(Item& it, const unsigned char* buf, int64_t base, int i, int lo,
                                                int hi) const {
        if (!vec) {
            load(it, base, i, lo, hi);
            return;
        }
        const int lane = threadIdx.x & 31;
        unsigned long long c[kSegPer];
        constexpr int kPerC = 16 / (int)sizeof(C);
#pragma unroll
        for (int q = 0; q < kSegPer / kPerC; ++q) {
            const C* const s = reinterpret_cast<const C*>(buf + kSegC * 8 + 16 * seg_unit(kSegPer / kPerC * lane + q));
            C w[kPerC];
            *reinterpret_cast<uint4*>(w) = *reinterpret_cast<const uint4*>(s);
#pragma unroll
            for (int k = 0; k < kPerC; ++k) c[kPerC * q + k] = (unsigned long long)(long long)w[k];
        }
        it.ok = true;
#pragma unroll
        for (int j = 0; j < kSegPer; ++j) {
            const bool in = i + j >= lo && i + j < hi;
            const bool ok = c[j] < (unsigned long long)ncols;
            it.x[j] = in && ok ? __ldg(x + c[j]) : 0.0;
            it.ok &= ok || !in;
            c[j] = in && ok;
        }
#pragma unroll
        for (int q = 0; q < kSegPer / 2; ++q) {
            const double2 v = *reinterpret_cast<const double2*>(buf + 16 * seg_unit(kSegPer / 2 * lane + q));
            it.v[2 * q] = c[2 * q] ? v.x : 0.0;
            it.v[2 * q + 1] = c[2 * q + 1] ? v.y : 0.0;
        }
    }
    __device__ __forceinline__ double mac(const Item& it, int j, double acc) const {
        return fma(it.v[j], it.x[j], acc);
    }
};

// The split of the values [first, end) and of the nb boundaries over the warps,
// in equal shares of the two together: the boundaries are merged into the
// values (boundary b comes before value offsets[b], as item offsets[b] - first +
// b of the merged sequence), and warp w takes the items from w * per on.  With
// shares of the values alone a run of empty segments, whose boundaries all
// stand at one place, fell to one warp: 2^20 rows of Zipf length, half of them
// empty in a run, took 10.0 ms and now 92 us (8 lanes per row: 138); 10^6 empty
// segments between two of 500 values 16.5 ms and now 27 us.
struct SegSplit {
    int64_t lo_valid, hi_valid, per;
    bool ok;
    // share: `per` where the host knows it, else 0
    __device__ __forceinline__ SegSplit(int64_t first, int64_t end, int64_t nb, int64_t nwarps, int64_t share) {
        ok = first >= 0 && end >= first;
        lo_valid = ok ? first : 0;
        hi_valid = ok ? end : 0;
        per = share ? share : (hi_valid - lo_valid + nb + nwarps - 1) / nwarps;
        if (per > (1 << 29)) ok = false;  // positions inside a range are kept in 32 bits
    }
};
// Values before position p and boundaries before number b.
struct SegCut {
    int64_t p, b;
};

// The merged sequence's keys: strictly ascending where the offsets ascend.
__device__ __forceinline__ int64_t seg_key(const int64_t* a, int64_t i) {
    return (int64_t)((unsigned long long)a[i] + (unsigned long long)i);
}
// Narrows [0, m] to at most 33 numbers each, [lo, hi], that hold the first i with
// seg_key(a, i) >= key (m when there is none), for two keys at once.  Warp-wide:
// 32 probes per key and round narrow the range 33-fold.  The result depends on
// the key alone.
__device__ __forceinline__ void warp_narrow2(const int64_t* __restrict__ a, int64_t m, const int64_t (&key)[2],
                                             int64_t (&lo)[2], int64_t (&hi)[2]) {
    const int lane = threadIdx.x & 31;
    lo[0] = lo[1] = 0;
    hi[0] = hi[1] = m;
    while (hi[0] - lo[0] > 32 || hi[1] - lo[1] > 32) {
        int64_t v[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int64_t p = lo[q] + (hi[q] - lo[q]) * (lane + 1) / 33;
            v[q] = p < hi[q] ? seg_key(a, p) : 0;
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int64_t span = hi[q] - lo[q];
            if (span > 32) {  // warp-uniform
                const int k = __popc(__ballot_sync(0xffffffffu, v[q] < key[q]));
                const int64_t nlo = k ? lo[q] + span * k / 33 + 1 : lo[q];
                const int64_t nhi = k < 32 ? lo[q] + span * (k + 1) / 33 : hi[q];
                lo[q] = nlo;
                hi[q] = nhi;
            }
        }
    }
}

// Where warp w's range begins, and where it ends (the next one's begin).
// Warp-wide.  A cut is moved to the nearest whole chunk when no more than about
// 32 boundaries and half a share lie between, with the boundaries at that very
// place before it: ranges then begin and end with whole chunks as long as
// boundaries are not dense (one chunk more for every warp cost 10^6 values 3 us
// of 18).  A cut depends on its number alone, so both neighbours find the same
// one; the cuts of valid offsets ascend.
__device__ __forceinline__ void seg_cuts(const SegSplit& sp, const int64_t* __restrict__ a, int64_t nb, int64_t w,
                                         int64_t nwarps, SegCut& from, SegCut& to) {
    const int lane = threadIdx.x & 31;
    const bool second = lane >= 16;  // the lower lanes work out `from`, the upper ones `to`
    const int64_t d[2] = {sp.lo_valid + w * sp.per, sp.lo_valid + (w + 1) * sp.per};
    int64_t lo[2], hi[2];
    warp_narrow2(a, nb, d, lo, hi);
    // the boundaries that may be the cut's, and 32 on either side of them
    constexpr int kNear = 32, kLoads = 2 * kNear / 32 + 1;
    int64_t x[2][kLoads];
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int k = 0; k < kLoads; ++k) {
            const int64_t i = lo[q] - kNear + 32 * k + lane;
            x[q][k] = i < 0 ? LLONG_MIN : (i < nb ? a[i] : LLONG_MAX);
        }
    int past[2], near[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int64_t i = lo[q] + lane;
        const bool below = i < hi[q] && (int64_t)((unsigned long long)x[q][kNear / 32] + (unsigned long long)i) < d[q];
        past[q] = __popc(__ballot_sync(0xffffffffu, below));
    }
    const int64_t item = second ? d[1] : d[0];
    SegCut c;
    c.b = second ? lo[1] + past[1] : lo[0] + past[0];
    c.p = item - c.b;
    c.p = c.p < sp.lo_valid ? sp.lo_valid : (c.p > sp.hi_valid ? sp.hi_valid : c.p);
    int64_t edge = (c.p + kSegC / 2) / kSegC * kSegC;
    edge = edge < sp.lo_valid ? sp.lo_valid : (edge > sp.hi_valid ? sp.hi_valid : edge);
#pragma unroll
    for (int q = 0; q < 2; ++q) {  // of those boundaries the ones up to the chunk's edge
        const int64_t e = __shfl_sync(0xffffffffu, edge, 16 * q);
        int n = 0;
#pragma unroll
        for (int k = 0; k < kLoads; ++k) n += x[q][k] <= e;
        near[q] = __reduce_add_sync(0xffffffffu, n);
    }
    const int n = second ? near[1] : near[0], by = n - kNear - (second ? past[1] : past[0]);
    const int64_t moved = (edge < c.p ? c.p - edge : edge - c.p) + (by < 0 ? -by : by);
    if (n > 0 && n < 32 * kLoads && 2 * moved <= sp.per) c = SegCut{edge, c.b + by};
    const int64_t number = second ? w + 1 : w;
    if (number == 0) c = SegCut{sp.lo_valid, 0};
    else if (number >= nwarps || item >= sp.hi_valid + nb) c = SegCut{sp.hi_valid, nb};
    from = SegCut{__shfl_sync(0xffffffffu, c.p, 0), __shfl_sync(0xffffffffu, c.b, 0)};
    to = SegCut{__shfl_sync(0xffffffffu, c.p, 16), __shfl_sync(0xffffffffu, c.b, 16)};
}

// ---- rows of even length --------------------------------------------------------
// Where the rows of an SpMV are about equally long, 8 lanes per row waste little
// and need no search, no scan and no staging.  Only the device knows the lengths:
// every block looks at the same 256 groups of four neighbouring rows (what a warp
// takes, with 8 lanes each) and so comes to the same answer.
//
// By lanes go rows of 16 entries and more on average (20 with int32 columns, which
// the entry split reads at less cost), unless they are uneven: the groups' longest
// rows well above the average, or the average well above that of the sampled rows
// (what the sample did not see must then be long).  2^20 rows, int64 / int32
// columns, by 8 lanes and by entries, us: 8 entries each 74 and 71 / 82 and 66; 12
// 108 and 92 / 107 and 86; 16 95 and 112 / 103 and 105; 20 115 and 134 / 121 and 125;
// 32 157 and 194 / 160 and 181; 100 491 and 539 / 463 and 506; 16 to 48 178 and 194 /
// 179 and 181; Zipf lengths 191 and 97 / 182 and 90.  (Looking takes 2 us.)
// Returns 0, or, for the rows by lanes, how many entries make one of them long.
// Called by all threads of a block of 256; sh: sixteen words.
template <class Src>
__device__ __forceinline__ unsigned seg_rows_by_lanes(const int64_t* __restrict__ row_ptr, int64_t nrows, unsigned* sh) {
    const int64_t r = (int64_t)threadIdx.x * (nrows >> 2) / kSegT * 4;
    const float mean = (float)(row_ptr[nrows] - row_ptr[0]) / (float)nrows;
    int64_t p = row_ptr[r];
    unsigned longest = 0, len = 0;
#pragma unroll
    for (int k = 1; k <= 4; ++k) {
        const int64_t e = r + k <= nrows ? row_ptr[r + k] : p, l = e - p;
        const unsigned n = l < 0 ? 0u : (l > (1 << 20) ? 1u << 20 : (unsigned)l);
        longest = n > longest ? n : longest;
        len += n;
        p = e;
    }
    longest = __reduce_add_sync(0xffffffffu, (longest + 7) >> 3);
    len = __reduce_add_sync(0xffffffffu, len);
    if ((threadIdx.x & 31) == 0) {
        sh[threadIdx.x >> 5] = longest;
        sh[kSegWarps + (threadIdx.x >> 5)] = len;
    }
    __syncthreads();
    unsigned eights = 0, sampled = 0;  // of 256 groups, of 1024 rows
#pragma unroll
    for (int w = 0; w < kSegWarps; ++w) {
        eights += sh[w];
        sampled += sh[kSegWarps + w];
    }
    __syncthreads();
    const bool even = mean >= Src::kLanesMean && (float)eights * (1.0f / kSegT) <= mean * (1.25f / 8.0f) + 1.25f &&
                      mean <= (float)sampled * (1.25f / (4 * kSegT));
    return even ? (mean < 128.0f ? 1024u : (unsigned)(8.0f * mean)) : 0u;  // (mean below 1.25 * 2^20)
}

// The rows by 8 lanes each, the sums of spmv_csr_kernel<8>, bit for bit, but for
// rows of more than 1024 entries and eight times the average: the first eight
// that a warp meets wait for the whole block.  The sample sees one row in a
// thousand, and 8 lanes take 0.42 us per 8 entries of a long one: 2^20 rows of 32
// and one of 10^6 entries 55.6 ms, now 2.3.
constexpr int kSegLongKept = 8;
template <class Src>
__device__ __forceinline__ void seg_rows(const Src& src, double* __restrict__ y, unsigned limit, unsigned* err) {
    __shared__ int64_t sh_row[kSegWarps][kSegLongKept];
    __shared__ int sh_kept[kSegWarps];
    __shared__ double sh_sum[kSegWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = threadIdx.x & 7, group = lane >> 3;
    const int64_t warps = (int64_t)gridDim.x * kSegWarps;
    bool bad = false;
    int kept = 0;
    for (int64_t rb = ((int64_t)blockIdx.x * kSegWarps + warp) * 4; rb < src.nrows; rb += warps * 4) {
        const int64_t r = rb + group;
        const long long s = r < src.nrows ? src.row_ptr[r] : 0, e = r < src.nrows ? src.row_ptr[r + 1] : 0;
        const unsigned far = __ballot_sync(0xffffffffu, e - s > (long long)limit && sub == 0);  // the groups with a long row
        const int at = kept + __popc(far & ((1u << (8 * group)) - 1u));
        const bool later = e - s > (long long)limit && at < kSegLongKept;
        kept += __popc(far);
        double acc = 0.0;
        for (long long k = s + sub; k < e && !later; k += 8) {
            const long long c = (long long)__ldg(src.cols + k);
            if ((unsigned long long)c < (unsigned long long)src.ncols) acc = fma(__ldg(src.vals + k), __ldg(src.x + c), acc);
            else bad = true;
        }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o, 8);
        if (sub == 0 && r < src.nrows) {
            if (later) sh_row[warp][at] = r;
            else y[r] = acc;
        }
    }
    if (lane == 0) sh_kept[warp] = kept < kSegLongKept ? kept : kSegLongKept;
    __syncthreads();
    for (int w = 0; w < kSegWarps; ++w)
        for (int i = 0; i < sh_kept[w]; ++i) {
            const int64_t r = sh_row[w][i];
            const long long e = src.row_ptr[r + 1];
            double acc = 0.0;
#pragma unroll 4
            for (long long k = src.row_ptr[r] + threadIdx.x; k < e; k += kSegT) {
                const long long c = (long long)__ldg(src.cols + k);
                const bool ok = (unsigned long long)c < (unsigned long long)src.ncols;
                const double v = __ldg(src.vals + k), x = ok ? __ldg(src.x + c) : 0.0;
                if (ok) acc = fma(v, x, acc);
                bad |= !ok;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
            if (lane == 0) sh_sum[warp] = acc;
            __syncthreads();
            if (threadIdx.x == 0) {
                acc = 0.0;
#pragma unroll
                for (int u = 0; u < kSegWarps; ++u) acc += sh_sum[u];
                y[r] = acc;
            }
            __syncthreads();
        }
    if (bad) raise_error(err, ERRBIT_BOUNDS);
}

// Boundary b is offsets[b], 0 <= b <= nseg; it ends segment b - 1.  A warp takes
// the values and the boundaries between its two cuts.  Positions and boundary
// numbers below are relative to lo, the chunk that its first value is in, and to
// its first boundary b0.
template <class T, class Src>
__global__ void __launch_bounds__(kSegT, Src::kCtasPerSm)
    segsum_kernel(const Src src, const int64_t* __restrict__ offsets, const int64_t nseg, const T init,
                  T* __restrict__ out, const SegPartials<T> part, unsigned* err) {
    // per warp: the chunk's sums, or two staged chunks (a chunk's sums then take the place of its values)
    extern __shared__ __align__(16) unsigned char seg_smem[];
    constexpr bool kStaged = Src::kStageBytes > 0;
    __shared__ unsigned sh_bits[kSegWarps][kSegC / 32];
    __shared__ int sh_pos[kSegWarps][Src::kPos > 0 ? Src::kPos : 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned char* const mine = seg_smem + warp * (kStaged ? 2 * Src::kStageBytes : kSegC * (int)sizeof(T));
    unsigned* const bits = sh_bits[warp];
    int* const pos = sh_pos[warp];
    const int w = blockIdx.x * kSegWarps + warp;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if constexpr (Src::kRows) {
        const unsigned limit = seg_rows_by_lanes<Src>(offsets, nseg, &sh_bits[0][0]);
        if (blockIdx.x == 0 && threadIdx.x == 0) *part.by_lanes = limit;
        if (limit) return;  // the second kernel, of more and smaller warps, takes them
    }
    const int64_t nwarps = (int64_t)gridDim.x * kSegWarps;
    const SegSplit sp(src.first(), src.end(), nseg + 1, nwarps, src.share);
    SegCut from, to;
    seg_cuts(sp, offsets, nseg + 1, w, nwarps, from, to);
    const int64_t b0 = from.b;
    if (sp.ok && from.p == to.p && b0 == to.b) {  // nothing left for this warp
        if (lane == 0) {
            part.tail[w] = T(0);
            part.closes[w] = kSegNoBoundary;
        }
        return;
    }
    const int64_t lo = from.p / kSegAlign * kSegAlign;
    bool bad = !sp.ok || to.b < b0 || to.p < from.p || to.p - lo > (1 << 30);
    bool bad_item = false;
    const int nb = bad ? 0 : (int)(to.b - b0);
    const int64_t* const off = offsets + b0;  // [nb]
    T* const outb = out + b0 - 1;             // segment b0 - 1 + r ends at boundary r
    // a boundary's position: clamped below to "before the range"
    auto rel = [&](int64_t x) {
        const int64_t r = x - lo;
        return r < 0 ? -1 : (r > INT_MAX ? INT_MAX : (int)r);
    };
    const int vlo = (int)(from.p - lo), vhi = bad ? 0 : (int)(to.p - lo);  // valid positions: [vlo, vhi)
    const int stop_p = vhi;  // chunks start below this (the first one always runs)
    int bc = 0;                                      // first boundary not yet passed
    int prev = b0 > 0 ? rel(offsets[b0 - 1]) : -2;   // the one before it
    bool closes = false;   // this lane ended the piece that was open at lo
    T carry = T(0);        // sum of the open piece, up to the last boundary chunk's end
    T acc[kSegPer];        // ... and since then, per lane
    bool have_acc = false;
#pragma unroll
    for (int j = 0; j < kSegPer; ++j) acc[j] = T(0);
    // a window of the next 32 boundaries
    int win = lane < nb ? rel(off[lane]) : INT_MAX;

    int p = 0;
    if constexpr (kStaged) {
        src.stage(mine, lo, 0, vlo, vhi);
        src.stage(mine + Src::kStageBytes, lo, kSegC, vlo, vhi);
    }
    while (!bad) {
        typename Src::Item it;
        unsigned char* buf = mine;
        if constexpr (kStaged) {
            buf += (p / kSegC & 1) * Src::kStageBytes;
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncwarp();
            src.load_staged(it, buf, lo, p + kSegPer * lane, vlo, vhi);
            __syncwarp();
        } else {
            src.load(it, lo, p + kSegPer * lane, vlo, vhi);
        }
        T* const sums = reinterpret_cast<T*>(buf);
        const int next = __shfl_sync(0xffffffffu, win, 0);
        bad_item |= !src.check(it);
        if (next > p + kSegC) {
#pragma unroll
            for (int j = 0; j < kSegPer; ++j) acc[j] = src.mac(it, j, acc[j]);
            have_acc = true;
            if constexpr (kStaged) src.stage(buf, lo, p + 2 * kSegC, vlo, vhi);
            p += kSegC;
            // whole chunks before the next boundary, kUnroll at a time
            const int stop = next - 1 < stop_p ? next - 1 : stop_p;
            for (; !kStaged && p + Src::kUnroll * kSegC <= stop; p += Src::kUnroll * kSegC) {
                typename Src::Item iu[Src::kUnroll];
#pragma unroll
                for (int u = 0; u < Src::kUnroll; ++u)
                    src.load(iu[u], lo, p + u * kSegC + kSegPer * lane, vlo, vhi);
#pragma unroll
                for (int u = 0; u < Src::kUnroll; ++u) {
                    bad_item |= !src.check(iu[u]);
#pragma unroll
                    for (int j = 0; j < kSegPer; ++j) acc[j] = src.mac(iu[u], j, acc[j]);
                }
            }
            if (p >= stop_p) break;
            continue;
        }
        // a chunk with boundaries: mark the heads
        if (lane < kSegC / 32) bits[lane] = 0u;
        __syncwarp();
        bool at_end = false;
        int total = 0, pw = prev;  // boundaries of this chunk so far; the last one
        const int wn = bc + 32 + lane < nb ? rel(off[bc + 32 + lane]) : INT_MAX;
        // one window of 32: false when it is the chunk's last
        auto mark = [&](int xw) {
            const bool in = bc + total + lane < nb && xw <= p + kSegC;
            const unsigned m = __ballot_sync(0xffffffffu, in);
            const int up = __shfl_up_sync(0xffffffffu, xw, 1);
            const int before = lane ? up : pw;
            const int cnt = __popc(m);
            if (in) {
                // ascending, inside the values, and not one that an earlier chunk should have met
                bad |= xw < before || xw > vhi || xw < vlo || !(xw > p || p == 0);
                if (xw > p && xw < p + kSegC) atomicOr(&bits[(xw - p) >> 5], 1u << ((xw - p) & 31));
                at_end |= xw == p + kSegC;
                if (total + lane < Src::kPos) pos[total + lane] = xw;
            }
            bad |= cnt < 32 && (m >> cnt) != 0u;  // not a prefix of the window
            if (cnt) pw = __shfl_sync(0xffffffffu, xw, cnt - 1);
            total += cnt;
            return cnt == 32;
        };
        if (mark(win) && mark(wn)) {
            // many short segments: four windows' loads at once
            bool more = true;
            while (more) {
                int x4[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int b = bc + total + 32 * u + lane;
                    x4[u] = b < nb ? rel(off[b]) : INT_MAX;
                }
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (more) more = mark(x4[u]);
            }
        }
        bad = __any_sync(0xffffffffu, bad);
        if (bad) break;
        at_end = __any_sync(0xffffffffu, at_end);
        if (have_acc) {
            T a = ((acc[0] + acc[1]) + (acc[2] + acc[3])) + ((acc[4] + acc[5]) + (acc[6] + acc[7]));
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
            carry += a;
#pragma unroll
            for (int j = 0; j < kSegPer; ++j) acc[j] = T(0);
            have_acc = false;
        }
        __syncwarp();
        // segmented scan; only segment ends (and the chunk's last value) are
        // read back, so the carry from the lanes before is added once, at the
        // last position before the lane's first head
        const unsigned hb = (bits[lane >> 2] >> ((lane & 3) * 8)) & 0xffu;
        T r[kSegPer];
        r[0] = src.mac(it, 0, T(0));
#pragma unroll
        for (int j = 1; j < kSegPer; ++j) r[j] = src.mac(it, j, (hb >> j) & 1u ? T(0) : r[j - 1]);
        bool h = hb != 0u;
        T v = r[kSegPer - 1];
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const bool hu = __shfl_up_sync(0xffffffffu, h, d);
            const T vu = __shfl_up_sync(0xffffffffu, v, d);
            if (lane >= d) {
                if (!h) v = vu + v;
                h = h || hu;
            }
        }
        const bool hl = __shfl_up_sync(0xffffffffu, h, 1);
        const T vl = __shfl_up_sync(0xffffffffu, v, 1);
        const T ve = lane == 0 ? carry : (hl ? vl : carry + vl);
        const int fix = (hb ? __ffs(hb) - 1 : kSegPer) - 1;  // -1: nothing before the first head
        T sel = T(0);
#pragma unroll
        for (int j = 0; j < kSegPer; ++j)
            if (j == fix) sel = r[j];
        const T fixed = ve + sel;
#pragma unroll
        for (int j = 0; j < kSegPer; ++j) sums[seg_slot(kSegPer * lane + j)] = j == fix ? fixed : r[j];
        const T tail = fix == kSegPer - 1 ? fixed : r[kSegPer - 1];
        carry = at_end ? T(0) : __shfl_sync(0xffffffffu, tail, 31);
        __syncwarp();
        // the sums that end here
        // boundary 0 ends no segment; the piece that was open at lo goes to the partials
        auto finish = [&](int k, int x, int before) {
            const T s = x > p ? sums[seg_slot(x - 1 - p)] : T(0);
            const bool open = before < vlo;
            if (open && (b0 > 0 || bc + k > 0)) {
                part.head[w] = s;
                part.closes[w] = b0;
                closes = true;
            }
            if (!open) outb[bc + k] = before == x ? init : init + s;
        };
        if (Src::kPos == 0 && total <= 32) {
            const int up = __shfl_up_sync(0xffffffffu, win, 1);
            if (lane < total) finish(lane, win, lane ? up : prev);
        } else {
#pragma unroll 2
            for (int k = lane; k < total; k += 32) {
                const int x = k < Src::kPos ? pos[k] : rel(off[bc + k]);
                const int before = k == 0 ? prev : (k <= Src::kPos ? pos[k - 1] : rel(off[bc + k - 1]));
                finish(k, x, before);
            }
        }
        prev = pw;
        bc += total;
        if (total <= 32) {  // the window moves on by `total`: from the lanes above, then from the next 32
            const int from = lane + total;
            const int from_win = __shfl_sync(0xffffffffu, win, from & 31);
            const int from_next = __shfl_sync(0xffffffffu, wn, from & 31);
            win = from < 32 ? from_win : from_next;
        } else {
            win = bc + lane < nb ? rel(off[bc + lane]) : INT_MAX;
        }
        __syncwarp();
        if constexpr (kStaged) src.stage(buf, lo, p + 2 * kSegC, vlo, vhi);
        p += kSegC;
        if (p >= stop_p) break;
    }
    if constexpr (kStaged) asm volatile("cp.async.wait_all;" ::: "memory");
    bad |= bc != nb;
    T a = ((acc[0] + acc[1]) + (acc[2] + acc[3])) + ((acc[4] + acc[5]) + (acc[6] + acc[7]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    const bool any = __any_sync(0xffffffffu, closes);
    if (lane == 0) {
        if (!any) part.closes[w] = nb > 0 ? kSegNoPiece : kSegNoBoundary;
        part.tail[w] = carry + a;
        if (bad) atomicOr(part.bad, 1u);
    }
    if (bad_item) raise_error(err, ERRBIT_BOUNDS);
}

// One segment on its own, by a whole warp; false when it is invalid.
template <class T>
__device__ __forceinline__ bool seg_one(const SegPlain<T>& src, int64_t start, int64_t stop, T init, T* o) {
    const int lane = threadIdx.x & 31;
    const bool ok = start >= 0 && stop <= src.n && stop >= start;
    T acc = T(0);
    if (ok)
        for (int64_t k = start + lane; k < stop; k += 32) acc += src.vals[k];
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, d);
    if (lane == 0) *o = init + acc;
    return ok;
}
template <class C>
__device__ __forceinline__ bool seg_one(const SegProduct<C>& src, int64_t start, int64_t stop, double init,
                                        double* o) {
    const int lane = threadIdx.x & 31;
    bool ok = true;
    double acc = 0.0;
    for (int64_t k = start + lane; k < stop; k += 32) {
        const unsigned long long c = (unsigned long long)(long long)src.cols[k];
        if (c < (unsigned long long)src.ncols) acc = fma(src.vals[k], src.x[c], acc);
        else ok = false;
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, d);
    if (lane == 0) *o = init + acc;
    return ok;
}

// Adds up the pieces that cross warps of the first kernel: warp w of this
// one ends the piece that warp w of that one closed.  With invalid offsets it
// computes every segment instead.
template <class T, class Src>
__global__ void __launch_bounds__(kSegT, Src::kRows ? 8 : 1) segsum_finish_kernel(const Src src, const int64_t* __restrict__ offsets,
                                                              const int64_t nseg, const T init,
                                                              T* __restrict__ out, const SegPartials<T> part,
                                                              const int64_t nwarps, unsigned* err) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t w = (int64_t)blockIdx.x * kSegWarps + warp;
    // launched while the first kernel runs: wait for its results
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if constexpr (Src::kRows) {
        if (const unsigned limit = __ldcg(part.by_lanes)) {
            seg_rows(src, out, limit, err);
            return;
        }
    }
    // the blocks beyond the first kernel's were for the rows by lanes only
    const unsigned nblocks = (unsigned)((nwarps + kSegWarps - 1) / kSegWarps);
    if (blockIdx.x >= nblocks) return;
    const bool invalid = *(volatile const unsigned*)part.bad != 0u;
    if (invalid) {
        bool bad = false;
        for (int64_t s = w; s < nseg; s += (int64_t)nblocks * kSegWarps)
            bad |= !seg_one(src, offsets[s], offsets[s + 1], init, out + s);
        if (bad) raise_error(err, ERRBIT_BOUNDS);
    } else if (w < nwarps) {
        const int64_t b = part.closes[w];
        if (b >= 0) {
            // the warp that took the boundary which opened the piece: the one whose
            // share of the merged sequence it is in, or, where the cut there was
            // moved, one beside it; between it and this warp none has a boundary
            const SegSplit sp(src.first(), src.end(), nseg + 1, nwarps, src.share);
            const unsigned long long item = seg_key(offsets, b - 1) - sp.lo_valid;
            int64_t u = (item >> 32) == 0 ? (unsigned)item / (unsigned)sp.per : (int64_t)(item / sp.per);
            u += lane - 1;
            T s = u >= 0 && u < w ? part.tail[u] : T(0);
            const bool has = lane < 3 && u >= 0 && u < w && part.closes[u] != kSegNoBoundary;
            if (lane < 31 - __clz((int)__ballot_sync(0xffffffffu, has))) s = T(0);  // before the piece
            for (u += 32; u < w; u += 32) s += part.tail[u];
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
            if (lane == 0) out[b - 1] = init + (s + part.head[w]);
        }
    }
    // the last block leaves the two words at zero for the next call
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(part.done, 1u) == nblocks - 1) {
            *part.bad = 0u;
            *part.done = 0u;
        }
    }
}

// Blocks of the first kernel.  `values`: their number, or an estimate of it when
// only the device knows.
template <class Src>
static int64_t segsum_blocks(const Device* d, int64_t nseg, int64_t values) {
    // a warp per 256 values and boundaries while there is a block per SM at most;
    // then per 256 values, or 512 of both (3e5 values in 1.4e5 segments: 14.4 us,
    // 16.4 with a warp per 256 of both; 4e4 in 1.9e4: 13.9 and 12.3)
    const int64_t each = (int64_t)kSegC * kSegWarps, both = values + nseg + 1;
    const int64_t some = values > both / 2 ? values : both / 2, cap = (int64_t)d->sm_count * Src::kCtasPerSm;
    int64_t blocks = (both + each - 1) / each;
    if (blocks > d->sm_count) {
        blocks = (some + each - 1) / each;
        if (blocks < d->sm_count) blocks = d->sm_count;
    }
    return blocks > cap ? cap : blocks;
}
// `counters`: three words, zero the first time; scratch: segsum_bytes(blocks).
static size_t segsum_bytes(int64_t blocks) { return (size_t)blocks * kSegWarps * 24; }

template <class T, class Src>
static int segsum_launch(Src src, const int64_t* offsets, int64_t nseg, T init, T* out, const Device* d,
                         int64_t blocks, unsigned* counters, void* scratch, cudaStream_t s, const char* what) {
    const int64_t nwarps = blocks * kSegWarps;
    src.set_share(nseg + 1, nwarps);
    SegPartials<T> part;
    part.head = static_cast<T*>(scratch);
    part.tail = part.head + nwarps;
    part.closes = reinterpret_cast<int64_t*>(part.tail + nwarps);
    part.bad = counters;
    part.done = counters + 1;
    part.by_lanes = counters + 2;
    auto k = segsum_kernel<T, Src>;
    constexpr size_t kSmem = kSegWarps * (size_t)(Src::kStageBytes ? 2 * Src::kStageBytes : kSegC * (int)sizeof(T));
    HYD_TRY(configure_kernel((const void*)k, d, false));
    k<<<(unsigned)blocks, kSegT, kSmem, s>>>(src, offsets, nseg, init, out, part, d->d_err);
    HYD_TRY(launch_check(what));
    // programmatic dependent launch: the second kernel's blocks are in place
    // when the first one ends; not where it may have all the rows to do, which
    // takes an L1 that the first kernel's shared memory has not cut down (100
    // entries per row, 2^20 rows: 913 us so, 494 without)
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(Src::kRows ? d->sm_count * 16 : blocks));
    cfg.blockDim = dim3(kSegT);
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = Src::kRows ? 0 : 1;
    HYD_CUDA_TRY(cudaLaunchKernelEx(&cfg, segsum_finish_kernel<T, Src>, src, offsets, nseg, init, out, part, nwarps,
                                    d->d_err));
    return launch_check(what);
}

// The SpMV with the default row split (sparse.cu checks the arguments).
// HYD_CUDA_ERR_UNSUPPORTED, with nothing launched, where 8 lanes per row have to
// do: that form is one launch without scratch, so that calls may overlap in any
// way.  This one's scratch lies between its two launches.  Threads that share a
// stream take turns with both, and no other call uses the scratch; but a graph
// may be replayed on any stream, and a handle of the per-thread default stream
// stands for many.
template <class C>
int spmv_segsum(int64_t nrows, int64_t ncols, const long long* row_ptr, const C* cols, const double* vals,
                const double* x, double* y, cudaStream_t s) {
    const bool vec = ((reinterpret_cast<uintptr_t>(cols) | reinterpret_cast<uintptr_t>(vals)) & 31) == 0;
    const SegProduct<C> src{cols, vals, x, row_ptr, nrows, ncols, vec};
    cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
    if (s == cudaStreamPerThread || cudaStreamIsCapturing(s, &capturing) != cudaSuccess) {
        cudaGetLastError();
        return HYD_CUDA_ERR_UNSUPPORTED;
    }
    if (capturing != cudaStreamCaptureStatusNone) return HYD_CUDA_ERR_UNSUPPORTED;
    Device* d = nullptr;
    HYD_TRY(device(&d));
    const int64_t blocks = segsum_blocks<SegProduct<C>>(d, nrows, INT64_MAX / 2);
    constexpr size_t kCounters = 256;
    std::lock_guard<std::mutex> lock(d->spmv_mu);
    Workspace& w = d->spmv_ws[s];
    if (!w.base) {
        const size_t bytes = kCounters + segsum_bytes((int64_t)d->sm_count * SegProduct<C>::kCtasPerSm);
        // (relaxed: a capture that another thread has under way is not disturbed)
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        cudaThreadExchangeStreamCaptureMode(&mode);
        void* p = nullptr;
        const cudaError_t e = cudaMalloc(&p, bytes);
        cudaThreadExchangeStreamCaptureMode(&mode);
        if (e != cudaSuccess) {
            cudaGetLastError();
            return HYD_CUDA_ERR_UNSUPPORTED;
        }
        w.base = static_cast<unsigned char*>(p);
        w.bytes = bytes;
        HYD_CUDA_TRY(cudaMemsetAsync(p, 0, kCounters, s));
    }
    return segsum_launch<double>(src, reinterpret_cast<const int64_t*>(row_ptr), nrows, 0.0, y, d, blocks,
                                 reinterpret_cast<unsigned*>(w.base), w.base + kCounters, s, "spmv_csr");
}
template int spmv_segsum<long long>(int64_t, int64_t, const long long*, const long long*, const double*,
                                    const double*, double*, cudaStream_t);
template int spmv_segsum<int>(int64_t, int64_t, const long long*, const int*, const double*, const double*, double*,
                              cudaStream_t);

template <class T>
static int segreduce_launch(const int64_t* offsets, int64_t n_offsets, const T* vals, int64_t n_vals, T init,
                            T* out, void* stream, const char* what) {
    HYD_CHECK_ARG(n_offsets >= 1, "%s: need at least one offset", what);
    HYD_CHECK_ARG(offsets != nullptr, "%s: null offsets", what);
    HYD_CHECK_ARG(n_vals >= 0 && (n_vals == 0 || vals != nullptr), "%s: bad values", what);
    const int64_t nseg = n_offsets - 1;
    HYD_CHECK_ARG(nseg == 0 || out != nullptr, "%s: null output", what);
    if (nseg == 0) return HYD_CUDA_OK;
    HYD_CHECK_ARG(n_vals <= (int64_t)4096 * 0x7fffffffLL, "%s: too many values", what);
    const SegPlain<T> src{vals, n_vals, (reinterpret_cast<uintptr_t>(vals) & 31) == 0, 0};
    Device* d = nullptr;
    HYD_TRY(device(&d));
    const int64_t blocks = segsum_blocks<SegPlain<T>>(d, nseg, n_vals);
    unsigned* counters = nullptr;
    void* scratch = nullptr;
    HYD_TRY(workspace(as_stream(stream), segsum_bytes(blocks), &counters, &scratch));
    return segsum_launch<T>(src, offsets, nseg, init, out, d, blocks, counters + kSegCounterWord, scratch,
                            as_stream(stream), what);
}

}  // namespace hyd

using namespace hyd;

extern "C" int hyd_cuda_segmented_reduce_i64(const int64_t* offsets, int64_t n_offsets, const int64_t* vals,
                                             int64_t n_vals, int64_t init, int64_t* out, void* stream) {
    return segreduce_launch<long long>(offsets, n_offsets, reinterpret_cast<const long long*>(vals), n_vals,
                                       (long long)init, reinterpret_cast<long long*>(out), stream,
                                       "segmented_reduce_i64");
}

extern "C" int hyd_cuda_segmented_reduce_f64(const int64_t* offsets, int64_t n_offsets, const double* vals,
                                             int64_t n_vals, double init, double* out, void* stream) {
    return segreduce_launch<double>(offsets, n_offsets, vals, n_vals, init, out, stream, "segmented_reduce_f64");
}
