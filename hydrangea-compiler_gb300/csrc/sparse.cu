// sparse.cu -- coo_sum_duplicates, csr_from_sorted_coo, CSR SpMV, and the
// batched COO -> CSR -> SpMV pipeline over many instances of uneven size.
//
// Reference: coo_sum_duplicates (Lowering.hs:966-1080) merges adjacent equal
// (row, col) entries in one serial pass; csr_from_sorted_coo
// (Lowering.hs:1081-1160) counts entries per row, copies cols/vals through and
// turns the counts into row_ptr with a serial running sum; SpMV is the
// generate-of-reduce_generate of bench/spmv/spmv.hyd:30-40 (outer loop over
// rows in `omp parallel for`, sequential sum per row).
//
// GPU forms:
//  * coo_sum_duplicates: one pass over tiles with a look-back that carries the
//    number of runs and the open run's sum (int64, bit-exact); entries past the
//    canonical count are zeroed like the reference's calloc'd outputs.
//  * csr_from_sorted_coo: row counts (one atomic per run of equal rows in a
//    warp) and the copies of cols/vals in one pass, then an exclusive scan.
//  * SpMV: a group of G lanes per row, lane-strided fma partial sums and a
//    fixed xor tree, so results are deterministic; within 1e-12 of
//    sum |v*x| of the C backend's sequential sum.  Large matrices with the
//    default split take segsum.cu.
//  * batched pipeline: instances are described by a device table; persistent
//    CTAs drain a device-side queue of (instance, tile) work items through an
//    atomic cursor, so one launch covers 512 instances of 10^3..10^6 entries
//    with no per-instance launch.  Stages: (1) count entries per global row,
//    (2) one exclusive scan over all instances' rows gives every row's first
//    slot (instance ranges are contiguous, so this is also each instance's
//    row_ptr shifted by its entry base), (3) scatter every entry into its row
//    (atomic slot within the row), (4) per row: sort by column and compute that
//    row's SpMV (one fma chain in column order) in the same warp.  Columns are unique within a row in this
//    workload, so sorting fixes the in-row order and the CSR is bit-exact
//    however the atomics interleaved.
#include <cstdlib>
#include <cstring>
#include <vector>

#include "batch.cuh"
#include "hyd_common.cuh"

namespace hyd {

int scan_i64_launch(const long long* in, long long* out, int64_t n, long long init, bool reverse,
                    bool inclusive, cudaStream_t stream);
size_t scan_i64_scratch_bytes(int64_t n);
int scan_i64_launch_with(const long long* in, long long* out, int64_t n, long long init, bool reverse,
                         bool inclusive, void* scratch, cudaStream_t stream);

// ---------------------------------------------------------------- coo dedup
// One pass over the entries: a tile of 2048 finds its heads (entries that
// differ from the one before), sums each run of equal entries and looks back
// over the earlier tiles' words for the number of heads before it and the sum
// of the run that was open at its start.  A run is written once, by the tile
// it ends in, through shared memory so that the stores are whole sectors.
// HBM bounds it: 24 bytes read per entry and 24 written, 119 us at 2^24
// entries.  Measured there (runs of 4): 160 us, and 47 us for the zeros; head
// flags, a scan of them, three fills and a merge with atomics took 300 us.
constexpr int kCooT = 256;
constexpr int kCooPer = 8;
constexpr int kCooTile = kCooT * kCooPer;

// 8 consecutive entries, those past the end zero.
__device__ __forceinline__ void coo_load8(const long long* __restrict__ a, int64_t i, int64_t n, bool vec,
                                          long long (&v)[kCooPer]) {
    if (vec && i + kCooPer <= n) {
        const u64x4 x = ldg_stream_u64x4(a + i), y = ldg_stream_u64x4(a + i + 4);
        v[0] = (long long)x.x; v[1] = (long long)x.y; v[2] = (long long)x.z; v[3] = (long long)x.w;
        v[4] = (long long)y.x; v[5] = (long long)y.y; v[6] = (long long)y.z; v[7] = (long long)y.w;
    } else {
#pragma unroll
        for (int j = 0; j < kCooPer; ++j) v[j] = i + j < n ? a[i + j] : 0;
    }
}

// Tile word: {state | heads << 2, sum since the last head}; state 1 the tile's
// own, 2 of all entries up to the tile's end (TileWord, one 16-byte access), 3
// none: the tile's look-back gave up.  Such a tile has no place to write to: it
// writes nothing, nor do those that wait for it, and when the last one is among
// them the count is 0 (the caller learns of it from the error word).
__global__ void __launch_bounds__(kCooT, 3)
    coo_sum_kernel(const long long* __restrict__ rows, const long long* __restrict__ cols,
                   const long long* __restrict__ vals, int64_t nnz, bool vec, long long* __restrict__ out_rows,
                   long long* __restrict__ out_cols, long long* __restrict__ out_vals, long long* __restrict__ out_nnz,
                   TileWord* words, unsigned* ticket, unsigned limit, unsigned* err) {
    __shared__ long long sh_out[kCooTile];
    __shared__ long long sh_sum[kCooT / 32];   // per warp: the sum since its last head
    __shared__ int sh_heads[kCooT / 32];
    __shared__ long long sh_carry, sh_before;  // of the tile: the open run's sum, the heads before
    __shared__ unsigned sh_tile;
    __shared__ int sh_head0, sh_end;
    __shared__ bool sh_known;  // the look-back came to its end
    typedef unsigned long long U;  // sums wrap
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) sh_tile = atomicAdd(ticket, 1u);
    __syncthreads();
    const int64_t tile = sh_tile;
    const int64_t base = tile * kCooTile, i0 = base + kCooPer * threadIdx.x;
    long long r[kCooPer], c[kCooPer], v[kCooPer];
    coo_load8(rows, i0, nnz, vec, r);
    coo_load8(cols, i0, nnz, vec, c);
    coo_load8(vals, i0, nnz, vec, v);
    // heads of entries i0 .. i0 + 8 (bit 8: the next thread's first entry, so
    // bit j + 1 says that entry j ends its run; past the end counts as a head)
    long long pr = __shfl_up_sync(0xffffffffu, r[kCooPer - 1], 1), pc = __shfl_up_sync(0xffffffffu, c[kCooPer - 1], 1);
    if (lane == 0 && i0 > 0 && i0 < nnz) {
        pr = rows[i0 - 1];
        pc = cols[i0 - 1];
    }
    unsigned hb = 0;
    if (i0 < nnz && (i0 == 0 || r[0] != pr || c[0] != pc)) hb |= 1u;
#pragma unroll
    for (int j = 1; j < kCooPer; ++j)
        if (i0 + j < nnz && (r[j] != r[j - 1] || c[j] != c[j - 1])) hb |= 1u << j;
    const unsigned first_next = __shfl_down_sync(0xffffffffu, hb, 1) & 1u;
    unsigned ends = hb >> 1;  // bit j: entry j ends its run
    {
        const int64_t nx = i0 + kCooPer;
        unsigned e = first_next;
        if (lane == 31 && nx < nnz) e = rows[nx] != r[kCooPer - 1] || cols[nx] != c[kCooPer - 1];
        if (nx >= nnz) e = 1u;
        ends |= e << (kCooPer - 1);
        if (i0 < nnz && nnz - i0 < kCooPer) ends |= 1u << (nnz - 1 - i0);
        const int64_t left = nnz - i0;
        ends &= left >= kCooPer ? 0xffu : (left > 0 ? (1u << left) - 1u : 0u);
    }
    // this thread: heads, and the sum since its last head
    const int nh = __popc(hb);
    U s = 0;
#pragma unroll
    for (int j = 0; j < kCooPer; ++j) s = ((hb >> j) & 1u ? 0ull : s) + (U)v[j];
    int hs = nh;
    U ss = s;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int hu = __shfl_up_sync(0xffffffffu, hs, d);
        const U su = __shfl_up_sync(0xffffffffu, ss, d);
        if (lane >= d) {
            if (hs == 0) ss += su;
            hs += hu;
        }
    }
    int hx = __shfl_up_sync(0xffffffffu, hs, 1);  // exclusive, within the warp
    U sx = __shfl_up_sync(0xffffffffu, ss, 1);
    if (lane == 0) {
        hx = 0;
        sx = 0;
    }
    if (lane == 31) {
        sh_heads[warp] = hs;
        sh_sum[warp] = (long long)ss;
    }
    if (threadIdx.x == 0) sh_head0 = (int)(hb & 1u);
    const int64_t last = (nnz - base < kCooTile ? nnz - base : kCooTile) - 1;  // the tile's last entry
    if (threadIdx.x == last / kCooPer) sh_end = (int)((ends >> (last % kCooPer)) & 1u);
    __syncthreads();
    int heads = 0;  // of the tile
    int hw = 0;     // of the warps before this one
    U sw = 0;       // sum of the run open at this warp's start, within the tile
    U tsum = 0;     // of the tile: the sum since its last head
#pragma unroll
    for (int w = 0; w < kCooT / 32; ++w) {
        if (w == warp) {
            hw = heads;
            sw = tsum;
        }
        tsum = (sh_heads[w] ? 0ull : tsum) + (U)sh_sum[w];
        heads += sh_heads[w];
    }
    if (warp == 0) {
        U before = 0, carry = 0;
        bool known = true;
        if (tile > 0) {
            if (lane == 0) tile_word_store(&words[tile], 1ull | (U)heads << 2, tsum);
            bool open = true;  // the carry is not complete
            int64_t p = tile - 1;
            for (;;) {
                const int64_t q = p - lane;
                U f = 2ull, b = 0ull;  // before the first tile: no heads, no sum
                if (q >= 0) tile_word_load(&words[q], f, b);
                unsigned spins = 0;
                while (known && __any_sync(0xffffffffu, (f & 3ull) == 0ull)) {
                    known = ++spins <= limit;
                    if ((f & 3ull) == 0ull) tile_word_load(&words[q], f, b);
                }
                known = known && !__any_sync(0xffffffffu, (f & 3ull) == 3ull);
                if (!known) {
                    if (lane == 0) raise_error(err, ERRBIT_TIMEOUT);
                    break;
                }
                const unsigned incl = __ballot_sync(0xffffffffu, (f & 3ull) == 2ull);
                const int stop = incl ? __ffs(incl) - 1 : 31;
                const unsigned with_head = __ballot_sync(0xffffffffu, (f >> 2) != 0ull);
                // the run's sum reaches back to the nearest tile with a head
                const int reach = with_head ? min(stop, __ffs(with_head) - 1) : stop;
                U h = lane <= stop ? f >> 2 : 0ull;
                U x = open && lane <= reach ? b : 0ull;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    h += __shfl_xor_sync(0xffffffffu, h, o);
                    x += __shfl_xor_sync(0xffffffffu, x, o);
                }
                before += h;
                carry += x;
                if (with_head) open = false;
                if (incl) break;
                p -= 32;
            }
        }
        if (lane == 0) {
            if (known) tile_word_store(&words[tile], 2ull | (before + (U)heads) << 2, heads ? tsum : carry + tsum);
            else tile_word_store(&words[tile], 3ull, 0ull);
            sh_before = (long long)before;
            sh_carry = (long long)carry;
            sh_known = known;
            if (base + kCooTile >= nnz) *out_nnz = known ? (long long)before + heads : 0;
        }
    }
    __syncthreads();
    if (!sh_known) return;
    const int head0 = sh_head0;
    const int nruns = heads - head0 + sh_end;                            // runs that end here
    const int64_t at = sh_before - (head0 ? 0 : 1);                      // the first of them
    // the run open at this thread's start: from the lanes, the warps, the tiles before
    U run = sx;
    if (hx == 0) {
        run += sw;
        if (hw == 0) run += (U)sh_carry;
    }
    int slot = hw + hx - head0;  // of the run of the entry before this thread's first
    int my[kCooPer];
#pragma unroll
    for (int j = 0; j < kCooPer; ++j) {
        if ((hb >> j) & 1u) {
            ++slot;
            run = 0ull;
        }
        run += (U)v[j];
        my[j] = slot;
        if ((ends >> j) & 1u) sh_out[slot] = (long long)run;
    }
    __syncthreads();
    for (int k = threadIdx.x; k < nruns; k += kCooT) out_vals[at + k] = sh_out[k];
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kCooPer; ++j)
        if ((ends >> j) & 1u) sh_out[my[j]] = r[j];
    __syncthreads();
    for (int k = threadIdx.x; k < nruns; k += kCooT) out_rows[at + k] = sh_out[k];
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kCooPer; ++j)
        if ((ends >> j) & 1u) sh_out[my[j]] = c[j];
    __syncthreads();
    for (int k = threadIdx.x; k < nruns; k += kCooT) out_cols[at + k] = sh_out[k];
}

// Zeros past the canonical count, as in the reference's calloc'd result.
__global__ void __launch_bounds__(256) coo_zero_tail_kernel(long long* __restrict__ rows, long long* __restrict__ cols,
                                                            long long* __restrict__ vals, int64_t nnz,
                                                            const long long* __restrict__ count) {
    const int64_t k = *count;
    for (int64_t i = k + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nnz; i += (int64_t)gridDim.x * blockDim.x) {
        rows[i] = 0;
        cols[i] = 0;
        vals[i] = 0;
    }
}

// ---------------------------------------------------------------- csr build
// Row counts and the copies in one pass.  Sorted entries come in runs of equal
// rows: a warp adds each run of its 32 entries with one atomic.
__global__ void __launch_bounds__(256) csr_count_copy_kernel(const long long* __restrict__ rows,
                                                             const long long* __restrict__ cols,
                                                             const long long* __restrict__ vals, int64_t nnz,
                                                             int64_t nrows, unsigned long long* __restrict__ counts,
                                                             long long* __restrict__ col_idx,
                                                             long long* __restrict__ out_vals, unsigned* err) {
    const int lane = threadIdx.x & 31;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    bool bad = false;
    // warp-uniform trips: every lane takes part in the shuffles
    for (int64_t b = (int64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31); b < nnz; b += 2 * stride) {
        long long r[2], c[2], v[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int64_t i = b + u * stride + lane;
            const bool in = i < nnz;
            r[u] = in ? __ldg(rows + i) : -1;
            c[u] = in ? __ldg(cols + i) : 0;
            v[u] = in ? __ldg(vals + i) : 0;
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int64_t i = b + u * stride + lane;
            const bool in = i < nnz;
            if (in && nrows > 0) {  // with no rows every entry is out of range: nothing is copied
                col_idx[i] = c[u];
                out_vals[i] = v[u];
            }
            const bool ok = (unsigned long long)r[u] < (unsigned long long)nrows;
            bad |= in && !ok;
            const long long up = __shfl_up_sync(0xffffffffu, r[u], 1);
            const bool head = lane == 0 || up != r[u];
            const unsigned hm = __ballot_sync(0xffffffffu, head);
            if (head && ok) {
                const unsigned later = lane == 31 ? 0u : hm & (0xfffffffeu << lane);
                const int len = (later ? __ffs(later) - 1 : 32) - lane;
                atomicAdd(&counts[r[u]], (unsigned long long)len);
            }
        }
    }
    if (bad) raise_error(err, ERRBIT_BOUNDS);
}

// ---------------------------------------------------------------- SpMV
template <int G, class C>
__global__ void __launch_bounds__(256) spmv_csr_kernel(int64_t nrows, const long long* __restrict__ row_ptr,
                                                       const C* __restrict__ col_idx,
                                                       const double* __restrict__ vals,
                                                       const double* __restrict__ x, int64_t ncols,
                                                       double* __restrict__ y, unsigned* err) {
    const int sub = threadIdx.x & (G - 1);
    constexpr int kRowsPerWarp = 32 / G;
    const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int group = (threadIdx.x & 31) / G;
    bool bad = false;
    // warp-uniform loop: every lane of a warp runs the same iterations, so the
    // full-mask shuffles below always see all 32 lanes
    for (int64_t rb = warp * kRowsPerWarp; rb < nrows; rb += warps * kRowsPerWarp) {
        const int64_t r = rb + group;
        double acc = 0.0;
        if (r < nrows) {
            const long long s = row_ptr[r], e = row_ptr[r + 1];
            for (long long k = s + sub; k < e; k += G) {
                const long long c = (long long)col_idx[k];
                if ((unsigned long long)c < (unsigned long long)ncols) acc = fma(vals[k], x[c], acc);
                else bad = true;
            }
        }
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o, G);
        if (sub == 0 && r < nrows) y[r] = acc;
    }
    if (bad) raise_error(err, ERRBIT_BOUNDS);
}

// segsum.cu: the entries split evenly over the warps, whatever the rows'
// lengths, or, where the rows are even, 8 lanes per row after all: it looks.  It
// launches twice and searches the row pointers, so it takes large matrices only.
// Rows of Zipf length (12 entries on average, int64 columns), so and by 8 lanes
// each: 2^20 rows 97 and 204 us, 3 * 2^18 79 and 149, 2^19 61 and 104, 2^18 43 and
// 54; rows of 8 entries 71 and 74, 60 and 58, 47 and 39, 37 and 22.  From 3 * 2^18
// rows on no kind of row loses more than 5%; below, even rows lose more.
template <class C>
int spmv_segsum(int64_t nrows, int64_t ncols, const long long* row_ptr, const C* cols, const double* vals,
                const double* x, double* y, cudaStream_t s);
constexpr int64_t kSpmvSegMinRows = 3 << 18;

template <class C>
static int spmv_dispatch(int g, int64_t nrows, const long long* row_ptr, const C* col_idx, const double* vals,
                         const double* x, int64_t ncols, double* y, const Device* d, cudaStream_t stream) {
    if (g == 0) {
        if (nrows >= kSpmvSegMinRows) {
            const int st = spmv_segsum<C>(nrows, ncols, row_ptr, col_idx, vals, x, y, stream);
            if (st != HYD_CUDA_ERR_UNSUPPORTED) return st;
        }
        g = 8;
    }
    int64_t blocks = (nrows * g + 255) / 256;
    const int64_t cap = (int64_t)d->sm_count * 16;
    if (blocks > cap) blocks = cap;
    if (blocks < 1) blocks = 1;
    switch (g) {
        case 1: spmv_csr_kernel<1, C><<<(unsigned)blocks, 256, 0, stream>>>(nrows, row_ptr, col_idx, vals, x, ncols, y, d->d_err); break;
        case 2: spmv_csr_kernel<2, C><<<(unsigned)blocks, 256, 0, stream>>>(nrows, row_ptr, col_idx, vals, x, ncols, y, d->d_err); break;
        case 4: spmv_csr_kernel<4, C><<<(unsigned)blocks, 256, 0, stream>>>(nrows, row_ptr, col_idx, vals, x, ncols, y, d->d_err); break;
        case 8: spmv_csr_kernel<8, C><<<(unsigned)blocks, 256, 0, stream>>>(nrows, row_ptr, col_idx, vals, x, ncols, y, d->d_err); break;
        case 16: spmv_csr_kernel<16, C><<<(unsigned)blocks, 256, 0, stream>>>(nrows, row_ptr, col_idx, vals, x, ncols, y, d->d_err); break;
        default: spmv_csr_kernel<32, C><<<(unsigned)blocks, 256, 0, stream>>>(nrows, row_ptr, col_idx, vals, x, ncols, y, d->d_err); break;
    }
    return launch_check("spmv_csr");
}

// ---------------------------------------------------------------- batched pipeline
struct WorkItem {
    int inst;
    int tile;  // tile index inside the instance
};

constexpr int kBatchThreads = 256;
constexpr int kEntryTile = 8192;  // entries per work item (count and scatter stages)
constexpr int kRowTile = 256;     // rows per work item (sort + SpMV stage): one warp per row

__device__ __forceinline__ bool next_item(unsigned* cursor, unsigned nitems, unsigned& item) {
    __shared__ unsigned sh_item;
    if (threadIdx.x == 0) sh_item = atomicAdd(cursor, 1u);
    __syncthreads();
    item = sh_item;
    __syncthreads();
    return item < nitems;
}

// Stage 1: row counts (and validation of every entry).
__global__ void __launch_bounds__(kBatchThreads) batch_count_kernel(const BatchInst* __restrict__ inst,
                                                                    const WorkItem* __restrict__ items, unsigned nitems,
                                                                    unsigned* cursor, unsigned* __restrict__ counts,
                                                                    unsigned* err) {
    unsigned it;
    bool bad = false;
    while (next_item(cursor, nitems, it)) {
        const WorkItem w = items[it];
        const BatchInst I = inst[w.inst];
        const long long t0 = (long long)w.tile * kEntryTile;
        const long long t1 = t0 + kEntryTile < I.nnz ? t0 + kEntryTile : I.nnz;
        for (long long k = t0 + threadIdx.x; k < t1; k += kBatchThreads) {
            const int r = I.rows[k], c = I.cols[k];
            if (r >= 0 && r < I.nrows && c >= 0 && c < I.ncols) atomicAdd(&counts[I.row_base + r], 1u);
            else bad = true;
        }
    }
    if (bad) raise_error(err, ERRBIT_BOUNDS);
}

// Counts (u32) -> int64 for the scan.
__global__ void widen_kernel(const unsigned* __restrict__ c, long long* __restrict__ out, int64_t n) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = c[i];
}

// Stage 3: scatter entries to their row's slots (slot order within a row is
// arbitrary here; stage 4 sorts each row).  counts[] counts down to 0.
__global__ void __launch_bounds__(kBatchThreads) batch_scatter_kernel(const BatchInst* __restrict__ inst,
                                                                      const WorkItem* __restrict__ items,
                                                                      unsigned nitems, unsigned* cursor,
                                                                      const long long* __restrict__ row_start,
                                                                      unsigned* __restrict__ counts,
                                                                      unsigned* __restrict__ coo_idx) {
    unsigned it;
    while (next_item(cursor, nitems, it)) {
        const WorkItem w = items[it];
        const BatchInst I = inst[w.inst];
        const long long t0 = (long long)w.tile * kEntryTile;
        const long long t1 = t0 + kEntryTile < I.nnz ? t0 + kEntryTile : I.nnz;
        for (long long k = t0 + threadIdx.x; k < t1; k += kBatchThreads) {
            const int r = I.rows[k], c = I.cols[k];
            if (r < 0 || r >= I.nrows || c < 0 || c >= I.ncols) continue;  // reported by stage 1
            const long long g = I.row_base + r;
            const unsigned left = atomicSub(&counts[g], 1u);  // slots of row g still free
            const long long slot = row_start[g] - I.scan_base + (long long)left - 1;
            I.csr_cols[slot] = c;
            I.csr_vals[slot] = I.vals[k];
            coo_idx[I.scan_base + slot] = (unsigned)k;  // orders equal columns in stage 4
        }
    }
}

// Warp-wide bitonic sort of up to 32*kPer (key, val) pairs held kPer per lane
// in "lane-major" order (element j*32 + lane in slot j).  Padding uses the
// largest key.
template <int kPer, class K>
__device__ __forceinline__ void warp_bitonic_sort(K (&key)[kPer], double (&val)[kPer]) {
    const int lane = threadIdx.x & 31;
    constexpr int N = 32 * kPer;
#pragma unroll
    for (int size = 2; size <= N; size <<= 1) {
#pragma unroll
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            if (stride >= 32) {
                // partner in another slot of the same lane
                const int sj = stride / 32;
#pragma unroll
                for (int j = 0; j < kPer; ++j) {
                    if ((j & sj) == 0) {
                        const int idx = j * 32 + lane;
                        const bool up = (idx & size) == 0;
                        const int jj = j + sj;
                        const bool swap = up ? (key[j] > key[jj]) : (key[j] < key[jj]);
                        if (swap) {
                            const K tk = key[j]; key[j] = key[jj]; key[jj] = tk;
                            double tv = val[j]; val[j] = val[jj]; val[jj] = tv;
                        }
                    }
                }
            } else {
#pragma unroll
                for (int j = 0; j < kPer; ++j) {
                    const int idx = j * 32 + lane;
                    const K ok = __shfl_xor_sync(0xffffffffu, key[j], stride);
                    const double ov = __shfl_xor_sync(0xffffffffu, val[j], stride);
                    const bool up = (idx & size) == 0;
                    const bool lower = (lane & stride) == 0;
                    // the lower index keeps the smaller key when ascending
                    const bool take = lower ? (up ? ok < key[j] : ok > key[j]) : (up ? ok > key[j] : ok < key[j]);
                    if (take) {
                        key[j] = ok;
                        val[j] = ov;
                    }
                }
            }
        }
    }
}

// Sort key: column, then COO position -- the runtime's stable order for equal
// (row, col) entries.
// Columns are bounded by ncols before x is read: with invalid entries in the
// batch (reported by stage 1) a row can include a slot that no entry wrote,
// and whatever it holds must not index x.
template <int kPer>
__device__ __forceinline__ void sort_row_and_spmv(int* __restrict__ cc, double* __restrict__ cv,
                                                  const unsigned* __restrict__ coo_idx, int len,
                                                  const double* __restrict__ x, long long ncols, double* yrow) {
    const int lane = threadIdx.x & 31;
    long long key[kPer];
    double val[kPer];
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
        const int i = j * 32 + lane;
        key[j] = i < len ? (((long long)cc[i] << 32) | coo_idx[i]) : 0x7fffffffffffffffLL;
        val[j] = i < len ? cv[i] : 0.0;
    }
    warp_bitonic_sort<kPer>(key, val);
    double xv[kPer];
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
        const int i = j * 32 + lane;
        xv[j] = 0.0;
        if (i < len) {
            const int c = (int)(key[j] >> 32);
            cc[i] = c;
            cv[i] = val[j];
            if ((unsigned)c < (unsigned long long)ncols) xv[j] = x[c];
        }
    }
    // y: one fma chain over the row in column order (position i sits on lane
    // i % 32, register i / 32), the order of the bucketed form
    double acc = 0.0;
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
        for (int l = 0; l < 32 && j * 32 + l < len; ++l)
            acc = fma(__shfl_sync(0xffffffffu, val[j], l), __shfl_sync(0xffffffffu, xv[j], l), acc);
    }
    if (lane == 0) *yrow = acc;
}

// Stage 4: per row (one warp): sort by column, write back, y[row] = sum v*x[c].
// Also writes the instance's row_ptr (relative to its entry base).
__global__ void __launch_bounds__(kBatchThreads) batch_sort_spmv_kernel(
    const BatchInst* __restrict__ inst, const WorkItem* __restrict__ items, unsigned nitems, unsigned* cursor,
    const long long* __restrict__ row_start, const unsigned* __restrict__ coo_idx, unsigned* err) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int W = kBatchThreads / 32;
    unsigned it;
    bool bad = false;
    while (next_item(cursor, nitems, it)) {
        const WorkItem w = items[it];
        const BatchInst I = inst[w.inst];
        const long long r0 = (long long)w.tile * kRowTile;
        const long long r1 = r0 + kRowTile < I.nrows ? r0 + kRowTile : I.nrows;
        for (long long r = r0 + warp; r < r1; r += W) {
            const long long g = I.row_base + r;
            long long s = row_start[g] - I.scan_base;
            long long e = (r + 1 < I.nrows) ? row_start[g + 1] - I.scan_base : I.nnz;
            // with invalid entries (reported by stage 1) the counts and the
            // instance's extent disagree: keep the span inside the instance
            s = s < 0 ? 0 : (s > I.nnz ? I.nnz : s);
            e = e < s ? s : (e > I.nnz ? I.nnz : e);
            const int len = (int)(e - s);
            if (lane == 0) {
                I.row_ptr[r] = s;
                if (r == I.nrows - 1) I.row_ptr[I.nrows] = I.nnz;
            }
            int* cc = I.csr_cols + s;
            double* cv = I.csr_vals + s;
            const unsigned* ci = coo_idx + I.scan_base + s;
            if (len <= 32) sort_row_and_spmv<1>(cc, cv, ci, len, I.x, I.ncols, I.y + r);
            else if (len <= 64) sort_row_and_spmv<2>(cc, cv, ci, len, I.x, I.ncols, I.y + r);
            else if (len <= 128) sort_row_and_spmv<4>(cc, cv, ci, len, I.x, I.ncols, I.y + r);
            else if (len <= 256) sort_row_and_spmv<8>(cc, cv, ci, len, I.x, I.ncols, I.y + r);
            else bad = true;  // rows above 256 entries are outside this kernel's contract
        }
    }
    if (bad) raise_error(err, ERRBIT_BOUNDS);
}

// Runs the four stages for a batch described by host-side `inst` (row_base and
// scan_base filled here).  Scratch comes from the named device buffer `key`.
// With `staging` (pinned host memory of `staging_bytes`, kept alive by the
// caller until the stream reaches this point) the tables are copied
// asynchronously and the call returns without synchronizing; otherwise it
// synchronizes the stream before returning.
// Row-atomic form (see the file comment); the fallback of the bucketed form.
int batch_pipeline_rows(std::vector<BatchInst>& inst, const char* key, cudaStream_t s, void* staging,
                        size_t staging_bytes) {
    Device* d = nullptr;
    HYD_TRY(device(&d));
    std::vector<WorkItem> count_items, row_items;
    long long rows_total = 0, entries = 0;
    for (size_t i = 0; i < inst.size(); ++i) {
        BatchInst& I = inst[i];
        I.row_base = rows_total;
        I.scan_base = entries;
        for (long long t = 0; t * kEntryTile < I.nnz; ++t) count_items.push_back(WorkItem{(int)i, (int)t});
        for (long long t = 0; t * kRowTile < I.nrows; ++t) row_items.push_back(WorkItem{(int)i, (int)t});
        rows_total += I.nrows;
        entries += I.nnz;
    }
    if (rows_total >= (1LL << 32)) return set_error(HYD_CUDA_ERR_UNSUPPORTED, "batch: too many rows");
    for (const BatchInst& I : inst)  // COO positions are kept as 32-bit indices
        if (I.nnz > (1LL << 32)) return set_error(HYD_CUDA_ERR_UNSUPPORTED, "batch: instance above 2^32 entries");
    const size_t inst_bytes = (inst.size() * sizeof(BatchInst) + 255) & ~(size_t)255;
    const size_t ci_bytes = ((count_items.size() * sizeof(WorkItem)) + 255) & ~(size_t)255;
    const size_t ri_bytes = ((row_items.size() * sizeof(WorkItem)) + 255) & ~(size_t)255;
    const size_t cnt_bytes = ((size_t)rows_total * 4 + 255) & ~(size_t)255;
    const size_t wide_bytes = ((size_t)rows_total * 8 + 255) & ~(size_t)255;
    void* buf = nullptr;
    const size_t idx_bytes = ((size_t)entries * 4 + 255) & ~(size_t)255;
    HYD_TRY(device_buffer(d, key, inst_bytes + ci_bytes + ri_bytes + cnt_bytes + 2 * wide_bytes + 256 + idx_bytes,
                          &buf));
    unsigned char* b = static_cast<unsigned char*>(buf);
    BatchInst* d_inst = reinterpret_cast<BatchInst*>(b);
    WorkItem* d_ci = reinterpret_cast<WorkItem*>(b + inst_bytes);
    WorkItem* d_ri = reinterpret_cast<WorkItem*>(b + inst_bytes + ci_bytes);
    unsigned* counts = reinterpret_cast<unsigned*>(b + inst_bytes + ci_bytes + ri_bytes);
    long long* wide = reinterpret_cast<long long*>(b + inst_bytes + ci_bytes + ri_bytes + cnt_bytes);
    long long* row_start = wide + (wide_bytes / 8);
    unsigned* cursors = reinterpret_cast<unsigned*>(b + inst_bytes + ci_bytes + ri_bytes + cnt_bytes + 2 * wide_bytes);
    unsigned* coo_idx = reinterpret_cast<unsigned*>(b + inst_bytes + ci_bytes + ri_bytes + cnt_bytes + 2 * wide_bytes + 256);
    const size_t table_bytes = inst_bytes + ci_bytes + ri_bytes;
    const unsigned char* src_inst = reinterpret_cast<const unsigned char*>(inst.data());
    const unsigned char* src_ci = reinterpret_cast<const unsigned char*>(count_items.data());
    const unsigned char* src_ri = reinterpret_cast<const unsigned char*>(row_items.data());
    const bool async_tables = staging != nullptr && staging_bytes >= table_bytes;
    if (async_tables) {
        unsigned char* h = static_cast<unsigned char*>(staging);
        memcpy(h, src_inst, inst.size() * sizeof(BatchInst));
        if (!count_items.empty()) memcpy(h + inst_bytes, src_ci, count_items.size() * sizeof(WorkItem));
        memcpy(h + inst_bytes + ci_bytes, src_ri, row_items.size() * sizeof(WorkItem));
        HYD_CUDA_TRY(cudaMemcpyAsync(b, h, table_bytes, cudaMemcpyHostToDevice, s));
    } else {
        HYD_CUDA_TRY(cudaMemcpyAsync(d_inst, src_inst, inst.size() * sizeof(BatchInst), cudaMemcpyHostToDevice, s));
        if (!count_items.empty())
            HYD_CUDA_TRY(cudaMemcpyAsync(d_ci, src_ci, count_items.size() * sizeof(WorkItem), cudaMemcpyHostToDevice, s));
        HYD_CUDA_TRY(cudaMemcpyAsync(d_ri, src_ri, row_items.size() * sizeof(WorkItem), cudaMemcpyHostToDevice, s));
    }
    HYD_CUDA_TRY(cudaMemsetAsync(counts, 0, (size_t)rows_total * 4, s));
    HYD_CUDA_TRY(cudaMemsetAsync(cursors, 0, 16, s));
    const unsigned grid = (unsigned)(d->sm_count * 8);
    if (!count_items.empty()) {
        batch_count_kernel<<<grid, kBatchThreads, 0, s>>>(d_inst, d_ci, (unsigned)count_items.size(), cursors + 0,
                                                          counts, d->d_err);
        HYD_TRY(launch_check("batch_count"));
    }
    widen_kernel<<<grid, 256, 0, s>>>(counts, wide, rows_total);
    HYD_TRY(launch_check("batch_widen"));
    HYD_TRY(scan_i64_launch(wide, row_start, rows_total, 0, false, false, s));
    if (!count_items.empty()) {
        batch_scatter_kernel<<<grid, kBatchThreads, 0, s>>>(d_inst, d_ci, (unsigned)count_items.size(), cursors + 1,
                                                            row_start, counts, coo_idx);
        HYD_TRY(launch_check("batch_scatter"));
    }
    batch_sort_spmv_kernel<<<grid, kBatchThreads, 0, s>>>(d_inst, d_ri, (unsigned)row_items.size(), cursors + 2,
                                                          row_start, coo_idx, d->d_err);
    HYD_TRY(launch_check("batch_sort_spmv"));
    // pageable tables die with the caller's vectors: the copies must have run
    if (!async_tables) HYD_CUDA_TRY(cudaStreamSynchronize(s));
    return HYD_CUDA_OK;
}

int batch_pipeline_bucketed(std::vector<BatchInst>& bi, const char* key, cudaStream_t s, void* staging,
                            size_t staging_bytes);
size_t batch_pipeline_bucketed_table_bytes(const std::vector<BatchInst>& bi);

// The batched pipeline: the bucketed form (sparse_bucket.cu) when the batch is
// within its limits, otherwise the row-atomic form.
int batch_pipeline(std::vector<BatchInst>& inst, const char* key, cudaStream_t s, void* staging,
                   size_t staging_bytes) {
    const char* force = getenv("HYD_CUDA_BATCH_PIPELINE");  // "rows" forces the row-atomic form
    if (!(force && strcmp(force, "rows") == 0)) {
        const int st = batch_pipeline_bucketed(inst, key, s, staging, staging_bytes);
        if (st != HYD_CUDA_ERR_UNSUPPORTED) return st;
    }
    return batch_pipeline_rows(inst, key, s, staging, staging_bytes);
}

static size_t batch_pipeline_rows_table_bytes(const std::vector<BatchInst>& inst);

// Bytes of pinned staging batch_pipeline needs for `inst`.
size_t batch_pipeline_table_bytes(const std::vector<BatchInst>& inst) {
    const size_t a = batch_pipeline_bucketed_table_bytes(inst), b = batch_pipeline_rows_table_bytes(inst);
    return a > b ? a : b;
}

static size_t batch_pipeline_rows_table_bytes(const std::vector<BatchInst>& inst) {
    size_t ci = 0, ri = 0;
    for (const BatchInst& I : inst) {
        ci += (size_t)((I.nnz + kEntryTile - 1) / kEntryTile);
        ri += (size_t)((I.nrows + kRowTile - 1) / kRowTile);
    }
    return ((inst.size() * sizeof(BatchInst) + 255) & ~(size_t)255) + ((ci * sizeof(WorkItem) + 255) & ~(size_t)255) +
           ((ri * sizeof(WorkItem) + 255) & ~(size_t)255);
}

}  // namespace hyd

using namespace hyd;

// ------------------------------------------------------------------ C ABI
// `left_out`: tiles at the start that no block takes (0 but for the self-test).
static int coo_sum_launch(const int64_t* rows, const int64_t* cols, const int64_t* vals, int64_t nnz,
                          int64_t* out_rows, int64_t* out_cols, int64_t* out_vals, int64_t* out_nnz, int left_out,
                          unsigned limit, cudaStream_t s) {
    Device* d = nullptr;
    HYD_TRY(device(&d));
    const int64_t ntiles = (nnz + kCooTile - 1) / kCooTile;
    HYD_CHECK_ARG(ntiles <= 0x7fffffffLL, "coo_sum_duplicates: too long");
    const size_t bytes = 256 + sizeof(TileWord) * (size_t)ntiles;  // the ticket, then the tile words
    void* scratch = nullptr;
    HYD_TRY(workspace(s, bytes, nullptr, &scratch));
    HYD_CUDA_TRY(cudaMemsetAsync(scratch, 0, bytes, s));
    if (left_out) HYD_CUDA_TRY(cudaMemsetAsync(scratch, left_out, 1, s));  // the first ticket's lowest byte
    const bool vec = ((reinterpret_cast<uintptr_t>(rows) | reinterpret_cast<uintptr_t>(cols) |
                       reinterpret_cast<uintptr_t>(vals)) & 31) == 0;
    coo_sum_kernel<<<(unsigned)(ntiles - left_out), kCooT, 0, s>>>(
        (const long long*)rows, (const long long*)cols, (const long long*)vals, nnz, vec, (long long*)out_rows,
        (long long*)out_cols, (long long*)out_vals, (long long*)out_nnz,
        reinterpret_cast<TileWord*>(static_cast<unsigned char*>(scratch) + 256), static_cast<unsigned*>(scratch),
        limit, d->d_err);
    HYD_TRY(launch_check("coo_sum_duplicates"));
    int64_t blocks = (nnz + 255) / 256;
    if (blocks > d->sm_count * 8) blocks = d->sm_count * 8;
    coo_zero_tail_kernel<<<(unsigned)blocks, 256, 0, s>>>((long long*)out_rows, (long long*)out_cols,
                                                          (long long*)out_vals, nnz, (const long long*)out_nnz);
    return launch_check("coo_sum_duplicates");
}

extern "C" int hyd_cuda_coo_sum_duplicates_i64(const int64_t* rows, const int64_t* cols, const int64_t* vals,
                                               int64_t nnz, int64_t* out_rows, int64_t* out_cols, int64_t* out_vals,
                                               int64_t* out_nnz, void* stream) {
    HYD_CHECK_ARG(nnz >= 0, "coo_sum_duplicates: negative nnz");
    HYD_CHECK_ARG(out_nnz != nullptr, "coo_sum_duplicates: null out_nnz");
    HYD_CHECK_ARG(nnz == 0 || (rows && cols && vals && out_rows && out_cols && out_vals),
                  "coo_sum_duplicates: null buffer");
    cudaStream_t s = as_stream(stream);
    if (nnz == 0) {
        HYD_CUDA_TRY(cudaMemsetAsync(out_nnz, 0, 8, s));
        return HYD_CUDA_OK;
    }
    return coo_sum_launch(rows, cols, vals, nnz, out_rows, out_cols, out_vals, out_nnz, 0, kSpinLimit, s);
}

extern "C" int hyd_cuda_selftest_coo_timeout(const int64_t* rows, const int64_t* cols, const int64_t* vals,
                                             int64_t nnz, int64_t* out_rows, int64_t* out_cols, int64_t* out_vals,
                                             int64_t* out_nnz, uint32_t poll_limit, void* stream) {
    HYD_CHECK_ARG(nnz > kCooTile, "selftest_coo_timeout: needs more than %d entries", kCooTile);
    HYD_CHECK_ARG(rows && cols && vals && out_rows && out_cols && out_vals && out_nnz,
                  "selftest_coo_timeout: null buffer");
    HYD_CHECK_ARG(poll_limit >= 1 && poll_limit <= (1u << 20), "selftest_coo_timeout: poll limit outside 1..2^20");
    return coo_sum_launch(rows, cols, vals, nnz, out_rows, out_cols, out_vals, out_nnz, 1, poll_limit,
                          as_stream(stream));
}

extern "C" int hyd_cuda_csr_from_sorted_coo_i64(int64_t nrows, int64_t nnz, const int64_t* rows, const int64_t* cols,
                                                const int64_t* vals, int64_t* row_ptr, int64_t* col_idx,
                                                int64_t* out_vals, void* stream) {
    HYD_CHECK_ARG(nrows >= 0 && nnz >= 0, "csr_from_sorted_coo: negative size");
    HYD_CHECK_ARG(row_ptr != nullptr, "csr_from_sorted_coo: null row_ptr");
    HYD_CHECK_ARG(nnz == 0 || (rows && cols && vals && col_idx && out_vals), "csr_from_sorted_coo: null buffer");
    cudaStream_t s = as_stream(stream);
    Device* d = nullptr;
    HYD_TRY(device(&d));
    // nrows + 1 counts (the last stays zero), so that their exclusive scan is
    // the whole row_ptr, the total included
    const int64_t m = nrows + 1;
    auto al = [](size_t b) { return (b + 255) & ~(size_t)255; };
    const size_t count_bytes = al((size_t)m * 8);
    void* scratch = nullptr;
    HYD_TRY(workspace(s, count_bytes + al(scan_i64_scratch_bytes(m)), nullptr, &scratch));
    unsigned long long* counts = static_cast<unsigned long long*>(scratch);
    HYD_CUDA_TRY(cudaMemsetAsync(counts, 0, count_bytes, s));
    if (nnz > 0) {
        int64_t blocks = (nnz + 255) / 256;
        if (blocks > d->sm_count * 8) blocks = d->sm_count * 8;
        csr_count_copy_kernel<<<(unsigned)blocks, 256, 0, s>>>((const long long*)rows, (const long long*)cols,
                                                               (const long long*)vals, nnz, nrows, counts,
                                                               (long long*)col_idx, (long long*)out_vals, d->d_err);
        HYD_TRY(launch_check("csr_count"));
    }
    return scan_i64_launch_with((const long long*)counts, (long long*)row_ptr, m, 0, false, false,
                                static_cast<unsigned char*>(scratch) + count_bytes, s);
}

extern "C" int hyd_cuda_spmv_csr_f64(int64_t nrows, int64_t ncols, const int64_t* row_ptr, const int64_t* col_idx,
                                     const double* vals, const double* x, double* y, int lanes_per_row, void* stream) {
    HYD_CHECK_ARG(nrows >= 0 && ncols >= 0, "spmv_csr: negative size");
    HYD_CHECK_ARG(nrows == 0 || (row_ptr && y), "spmv_csr: null buffer");
    HYD_CHECK_ARG(lanes_per_row == 0 || lanes_per_row == 1 || lanes_per_row == 2 || lanes_per_row == 4 ||
                      lanes_per_row == 8 || lanes_per_row == 16 || lanes_per_row == 32,
                  "spmv_csr: lanes_per_row must be 0 (auto) or a power of two up to 32");
    if (nrows == 0) return HYD_CUDA_OK;
    Device* d = nullptr;
    HYD_TRY(device(&d));
    return spmv_dispatch<long long>(lanes_per_row, nrows, (const long long*)row_ptr, (const long long*)col_idx, vals, x, ncols, y, d,
                                    as_stream(stream));
}

extern "C" int hyd_cuda_spmv_csr_i32_f64(int64_t nrows, int64_t ncols, const int64_t* row_ptr, const int32_t* col_idx,
                                         const double* vals, const double* x, double* y, int lanes_per_row,
                                         void* stream) {
    HYD_CHECK_ARG(nrows >= 0 && ncols >= 0, "spmv_csr_i32: negative size");
    HYD_CHECK_ARG(nrows == 0 || (row_ptr && y), "spmv_csr_i32: null buffer");
    HYD_CHECK_ARG(lanes_per_row >= 0 && lanes_per_row <= 32 && (lanes_per_row & (lanes_per_row - 1)) == 0,
                  "spmv_csr_i32: lanes_per_row must be 0 (auto) or a power of two up to 32");
    if (nrows == 0) return HYD_CUDA_OK;
    Device* d = nullptr;
    HYD_TRY(device(&d));
    return spmv_dispatch<int>(lanes_per_row, nrows, (const long long*)row_ptr, (const int*)col_idx, vals, x, ncols, y, d,
                              as_stream(stream));
}

// Batched COO -> CSR -> SpMV.  `desc` is a HOST array of ninst x 3 int64
// (nrows, ncols, nnz); instances are concatenated in the device arrays in that
// order: rows/cols/vals/csr_cols/csr_vals by entries, x by ncols, y by nrows,
// row_ptr by nrows + 1.  row_ptr of each instance starts at 0.
extern "C" int hyd_cuda_batched_coo_csr_spmv_f64(int64_t ninst, const int64_t* desc, const int32_t* rows,
                                                 const int32_t* cols, const double* vals, const double* x,
                                                 int64_t* row_ptr, int32_t* csr_cols, double* csr_vals, double* y,
                                                 void* stream) {
    HYD_CHECK_ARG(ninst >= 0 && ninst < (1LL << 24), "batched_coo_csr_spmv: bad instance count");
    HYD_CHECK_ARG(ninst == 0 || desc != nullptr, "batched_coo_csr_spmv: null descriptor table");
    if (ninst == 0) return HYD_CUDA_OK;
    std::vector<BatchInst> inst((size_t)ninst);
    long long entries = 0, rows_total = 0, xs = 0;
    for (int64_t i = 0; i < ninst; ++i) {
        const long long nr = desc[3 * i], nc = desc[3 * i + 1], nz = desc[3 * i + 2];
        HYD_CHECK_ARG(nr >= 1 && nc >= 1 && nz >= 0 && nr < (1LL << 31) && nc < (1LL << 31),
                      "batched_coo_csr_spmv: instance %lld has a bad shape", (long long)i);
        BatchInst& I = inst[i];
        I.nrows = nr;
        I.ncols = nc;
        I.nnz = nz;
        I.rows = rows + entries;
        I.cols = cols + entries;
        I.vals = vals + entries;
        I.x = x + xs;
        I.row_ptr = (long long*)row_ptr + rows_total + i;
        I.csr_cols = csr_cols + entries;
        I.csr_vals = csr_vals + entries;
        I.y = y + rows_total;
        entries += nz;
        rows_total += nr;
        xs += nc;
    }
    HYD_CHECK_ARG(entries == 0 || (rows && cols && vals && csr_cols && csr_vals), "batched_coo_csr_spmv: null entries");
    HYD_CHECK_ARG(x && y && row_ptr, "batched_coo_csr_spmv: null x / y / row_ptr");
    return batch_pipeline(inst, "batch_tables", as_stream(stream), nullptr, 0);
}
