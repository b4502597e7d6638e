// sparse_bucket.cu -- the batched COO -> CSR -> SpMV pipeline, bucketed form.
//
// Same contract as batch_pipeline in sparse.cu (per instance: CSR of the
// entries sorted by (row, col), y = A x), organised so that no stage walks
// rows one dependent memory chain at a time:
//  1. count   per CTA, a contiguous range of (instance, 6144-entry tile)
//             items: a shared-memory histogram of 64-row buckets (row >> 6),
//             flushed with one global red per non-empty bucket when the
//             instance changes;
//  2. scan    exclusive scan of the ~4e5 bucket counts gives every bucket's
//             first slot (instances are contiguous, so bucket starts are also
//             each instance's entry offsets);
//  3. split   per tile again: each entry gets its rank inside (tile, bucket)
//             from a shared-memory atomic, each (tile, bucket) reserves its run
//             with one global atomic, and the tile, put into bucket order in
//             shared memory, is written to the buckets' regions as 16-byte
//             records: a 32-bit key (row_in_bucket << 24 | col), the COO
//             position and the value;
//  4. bucket  one block per bucket (at most 2048 entries, ncols <= 2^18): a
//             counting pass into as many bins as entries, in (row, col) order,
//             and comparisons inside the bins; the CSR columns/values written
//             in sorted order and the row pointers from the row counts.
//             Buckets with clustered columns are sorted by a warp each, with a
//             stable LSD radix sort of the packed keys; larger buckets by a
//             block-wide bitonic network;
//  5. spmv    one warp per chunk of 32 to 256 rows of an instance: the rows are ordered
//             by length in shared memory and each lane sums one row's fma
//             chain in column order, 32 rows of similar length at a time.
// The work lists of the stages (one item per (instance, tile), per (instance,
// bucket) and per (instance, chunk of rows)) are written on the device; only
// the instance table crosses from the host.
// Requires ncols < 2^24 (24-bit column field) and at most 256 entries per row.
#include <climits>
#include <cstring>
#include <vector>

#include "batch.cuh"
#include "hyd_common.cuh"

namespace hyd {

int scan_i64_launch(const long long* in, long long* out, int64_t n, long long init, bool reverse,
                    bool inclusive, cudaStream_t stream);

constexpr int kBkThreads = 512;
constexpr int kBkShift = 6;                  // 64 rows per bucket
constexpr int kBkRows = 1 << kBkShift;
constexpr int kBkCap = kBkRows * 256;        // entries per bucket at most (256 per row)
constexpr int kSplitThreads = 512;
constexpr int kSplitPerSm = 2;
constexpr int kSplitPer = 12;                // entries per thread of the split
constexpr int kTileEntries = kSplitThreads * kSplitPer;  // entries per count/split work item
static_assert(kTileEntries % kBkThreads == 0, "whole rounds of the count");
constexpr int kMaxSmemBuckets = 4096;        // per instance (2^18 rows)

struct BkInst {
    long long nrows, ncols, nnz;
    long long bucket_base;  // first bucket in the batch-wide bucket space
    long long nbuckets;
    long long tile_base;    // first entry tile in the batch-wide tile list
    long long chunk_base;   // first SpMV chunk in the batch-wide chunk list
    long long scan_base;    // entries of all earlier instances
    const int* rows;
    const int* cols;
    const double* vals;
    const double* x;
    long long* row_ptr;
    int* csr_cols;
    double* csr_vals;
    double* y;
};

struct BkItem {
    int inst;
    int tile;  // entry tile (stages 1, 3) or bucket index (stage 4)
};

__device__ __forceinline__ bool bk_next(unsigned* cursor, unsigned nitems, unsigned& item) {
    __shared__ unsigned sh_item;
    if (threadIdx.x == 0) sh_item = atomicAdd(cursor, 1u);
    __syncthreads();
    item = sh_item;
    __syncthreads();
    return item < nitems;
}

// Stage 1.  Each CTA counts a contiguous range of the tile list (the tiles of
// an instance are consecutive there), keeping its shared-memory bucket counts
// across the tiles of one instance and flushing them with one global red per
// non-empty bucket when the instance changes.  A flush per tile issued about
// one red per two entries for the largest instances, and the L2 atomics bound
// the kernel.  The counts are zero whenever they are not in use (the flush
// zeroes what it reads).
constexpr int kCountPerSm = 4;
__global__ void __launch_bounds__(kBkThreads, kCountPerSm) bk_count_kernel(const BkInst* __restrict__ inst,
                                                              const BkItem* __restrict__ items, unsigned nitems,
                                                              unsigned* __restrict__ bcount, unsigned* err) {
    __shared__ unsigned hist[kMaxSmemBuckets];
    for (int b = threadIdx.x; b < kMaxSmemBuckets; b += kBkThreads) hist[b] = 0u;
    const unsigned per = (nitems + gridDim.x - 1) / gridDim.x;
    const unsigned i0 = blockIdx.x * per;
    const unsigned i1 = i0 + per < nitems ? i0 + per : nitems;
    int cur = -1;
    long long cur_base = 0;
    int cur_nb = 0;
    bool bad = false;
    auto flush = [&]() {
        if (cur >= 0 && cur_nb <= kMaxSmemBuckets)
            for (int b = threadIdx.x; b < cur_nb; b += kBkThreads) {
                const unsigned c = hist[b];
                if (c) {
                    atomicAdd(&bcount[cur_base + b], c);
                    hist[b] = 0u;
                }
            }
    };
    __syncthreads();
    for (unsigned it = i0; it < i1; ++it) {
        const BkItem w = items[it];
        const BkInst I = inst[w.inst];
        if (w.inst != cur) {
            __syncthreads();  // the counting of the previous tile is complete
            flush();
            cur = w.inst;
            cur_base = I.bucket_base;
            cur_nb = (int)I.nbuckets;
            __syncthreads();  // the flush has read and zeroed every count
        }
        const bool smem = cur_nb <= kMaxSmemBuckets;
        const long long t0 = (long long)w.tile * kTileEntries;
        const int tn = (int)(t0 + kTileEntries < I.nnz ? kTileEntries : I.nnz - t0);
        const int* __restrict__ rows = I.rows + t0;
        const unsigned nrows = (unsigned)I.nrows;  // below 2^31: a negative row is above it too
        // all of this thread's rows first (read-only loads, all in flight at
        // once), then the counting: a load next to an atomic would otherwise
        // wait for it, one memory round trip per entry
        unsigned rr[kTileEntries / kBkThreads];
        auto count = [&](bool full) {  // columns are checked by the split, which reads them anyway
#pragma unroll
            for (int j = 0; j < kTileEntries / kBkThreads; ++j) {
                const int q = threadIdx.x + j * kBkThreads;
                if (full || q < tn) rr[j] = (unsigned)__ldg(rows + q);
            }
#pragma unroll
            for (int j = 0; j < kTileEntries / kBkThreads; ++j) {
                if (!full && threadIdx.x + j * kBkThreads >= tn) break;
                if (rr[j] >= nrows) bad = true;
                else if (smem) atomicAdd(&hist[rr[j] >> kBkShift], 1u);
                else atomicAdd(&bcount[cur_base + (rr[j] >> kBkShift)], 1u);
            }
        };
        if (tn == kTileEntries) count(true);
        else count(false);
    }
    __syncthreads();
    flush();
    if (bad) raise_error(err, ERRBIT_BOUNDS);
}

constexpr int kSpRows = 256;    // rows per SpMV chunk, at most
constexpr int kSpMinRows = 32;  // and at least

// The work lists of the count/split stages (one item per (instance, entry
// tile)), of the bucket stage (one per (instance, bucket)) and of the SpMV
// (one per (instance, chunk of rows)), written on the device: block i writes
// instance i's items at its tile_base / bucket_base / chunk_base.
__global__ void bk_items_kernel(const BkInst* __restrict__ inst, int64_t ninst, BkItem* __restrict__ tiles,
                                BkItem* __restrict__ buckets, BkItem* __restrict__ chunks, int chunk_rows) {
    for (int64_t i = blockIdx.x; i < ninst; i += gridDim.x) {
        const BkInst I = inst[i];
        const long long nt = (I.nnz + kTileEntries - 1) / kTileEntries;
        const long long nc = (I.nrows + chunk_rows - 1) / chunk_rows;
        for (long long t = threadIdx.x; t < nt; t += blockDim.x) tiles[I.tile_base + t] = BkItem{(int)i, (int)t};
        for (long long b = threadIdx.x; b < I.nbuckets; b += blockDim.x)
            buckets[I.bucket_base + b] = BkItem{(int)i, (int)b};
        for (long long c = threadIdx.x; c < nc; c += blockDim.x) chunks[I.chunk_base + c] = BkItem{(int)i, (int)c};
    }
}

__global__ void bk_widen_kernel(const unsigned* __restrict__ c, long long* __restrict__ out, int64_t n) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = c[i];
}

// Stage 3.  The tile is put into bucket order in shared memory before it is
// written, so that a bucket's run leaves as consecutive records from
// neighbouring lanes.
//  * the values are copied into shared memory with cp.async as soon as the
//    tile starts, and wait there in COO order;
//  * an entry's place in bucket order (the exclusive scan of the tile's bucket
//    counts, plus its rank) receives its key and, in one word, its bucket and
//    its position in the tile;
//  * the global reservations are in flight while that happens;
//  * the words are then read back in order: record p of the tile goes to
//    hist[bucket] + p, with hist[bucket] the run's first slot less its first
//    place;
//  * thread 0 asks for the next tile's entries to be brought into L2 meanwhile.
// Written from COO order, a lane's record went to a bucket of its own: 32 write
// requests of one sector per warp instruction, and those bounded the kernel.
// 2.9e8 entries in 512 instances of 2^10 to 2^18 rows: 3.88 ms so (8192-entry
// tiles), 2.77 ms in bucket order, 2.49 ms with the prefetch, 2.27 ms since the
// scan and the reservations stop at the instance's last bucket instead of 4096
// (reading and writing 32 bytes per entry takes 1.37 ms at the copy rate).  Two blocks of
// 512 threads with 6144 entries each fill an SM's shared memory; one block of
// 1024 threads with 12288, whose runs are twice as long, has no second block to
// fill its barriers and took 1% more of the whole pipeline.
constexpr int kSplitPosBits = 14;
static_assert(kTileEntries <= 1 << kSplitPosBits, "position in a tile");
static_assert(kMaxSmemBuckets <= 1 << (32 - kSplitPosBits), "bucket beside the position");
constexpr int kSplitBins = kMaxSmemBuckets / kSplitThreads;  // buckets per thread in the scan
constexpr size_t kSplitSmem = (size_t)kTileEntries * 16 + (kMaxSmemBuckets + 4) * 4;

__device__ __forceinline__ void cp_async_8(void* smem_dst, const void* gsrc) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(smem_dst)),
                 "l"(gsrc)
                 : "memory");
}

__global__ void __launch_bounds__(kSplitThreads, kSplitPerSm) bk_split_kernel(
    const BkInst* __restrict__ inst, const BkItem* __restrict__ items, unsigned nitems, unsigned* cursor,
    const long long* __restrict__ bstart, unsigned* __restrict__ bfill, uint4* __restrict__ rec_out, unsigned* err) {
    extern __shared__ __align__(16) double split_vals[];          // [kTileEntries], COO order
    uint2* sent = (uint2*)(split_vals + kTileEntries);  // [kTileEntries], bucket order: key; bucket << 14 | position
    unsigned* hist = (unsigned*)(sent + kTileEntries);  // [kMaxSmemBuckets + 1]
    __shared__ unsigned warp_sum[kSplitThreads / 32];
    __shared__ unsigned sh_it[2];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    bool bad = false;
    unsigned next = 0u;  // thread 0's: the tile after the current one
    if (threadIdx.x == 0) {
        sh_it[0] = blockIdx.x;
        next = gridDim.x + atomicAdd(cursor, 1u);
    }
    __syncthreads();
    for (unsigned turn = 0;; turn ^= 1u) {
        const unsigned it = sh_it[turn];
        if (it >= nitems) break;
        const BkItem w = items[it];
        const BkInst I = inst[w.inst];
        const bool smem = I.nbuckets <= kMaxSmemBuckets;
        const int nb = smem ? (int)I.nbuckets : 0;
        // threads of the counts' scan, whose counts reach one bucket past the last
        const int threads_used = nb < kMaxSmemBuckets ? nb / kSplitBins + 1 : kSplitThreads;
        const long long t0 = (long long)w.tile * kTileEntries;
        const int tn = (int)(t0 + kTileEntries < I.nnz ? kTileEntries : I.nnz - t0);
        // the rows and columns of all this thread's entries first (read-only
        // loads, all in flight at once), then the values' copies
        int bucket[kSplitPer];
        unsigned key[kSplitPer], rank[kSplitPer];
#pragma unroll
        for (int j = 0; j < kSplitPer; ++j) {
            const int q = threadIdx.x + j * kSplitThreads;
            bucket[j] = q < tn ? __ldg(I.rows + t0 + q) : -1;
            key[j] = q < tn ? (unsigned)__ldg(I.cols + t0 + q) : 0u;
        }
#pragma unroll
        for (int j = 0; j < kSplitPer; ++j) {
            const int q = threadIdx.x + j * kSplitThreads;
            if (q < tn) cp_async_8(split_vals + q, I.vals + t0 + q);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        if (threadIdx.x == 0) {
            // the next tile's entries on their way to L2 while this one is sorted
            sh_it[turn ^ 1u] = next;
            if (next < nitems) {
                const BkItem nw = items[next];
                const BkInst N = inst[nw.inst];
                const long long n0 = (long long)nw.tile * kTileEntries;
                const long long nn = n0 + kTileEntries < N.nnz ? kTileEntries : N.nnz - n0;
                l2_prefetch(N.rows + n0, nn * 4);
                l2_prefetch(N.cols + n0, nn * 4);
                l2_prefetch(N.vals + n0, nn * 8);
                next = gridDim.x + atomicAdd(cursor, 1u);
            }
        }
        if (smem)
            for (int b = threadIdx.x; b < threads_used * (kSplitBins / 4); b += kSplitThreads)
                ((uint4*)hist)[b] = make_uint4(0u, 0u, 0u, 0u);
        __syncthreads();
#pragma unroll
        for (int j = 0; j < kSplitPer; ++j) {
            const int q = threadIdx.x + j * kSplitThreads;
            const int r = bucket[j], c = (int)key[j];
            bucket[j] = -1;
            if (q < tn) {
                if (c < 0 || c >= I.ncols) bad = true;                 // (rows were checked by the count)
                if (r >= 0 && r < I.nrows && c >= 0 && c < I.ncols) {
                    bucket[j] = r >> kBkShift;
                    key[j] = ((unsigned)(r & (kBkRows - 1)) << 24) | (unsigned)c;
                    if (smem) rank[j] = atomicAdd(&hist[bucket[j]], 1u);
                }
            }
        }
        __syncthreads();
        if (!smem) {
            // more buckets than the shared counts hold: one global atomic per
            // entry, written where it lands
            asm volatile("cp.async.wait_all;" ::: "memory");  // this thread's own copies
#pragma unroll
            for (int j = 0; j < kSplitPer; ++j) {
                if (bucket[j] < 0) continue;
                const int q = threadIdx.x + j * kSplitThreads;
                const double v = split_vals[q];
                const long long pos =
                    bstart[I.bucket_base + bucket[j]] + atomicAdd(&bfill[I.bucket_base + bucket[j]], 1u);
                rec_out[pos] = make_uint4(key[j], (unsigned)(t0 + q), (unsigned)__double2loint(v),
                                          (unsigned)__double2hiint(v));
            }
            __syncthreads();
            continue;
        }
        // exclusive scan of the counts in place; hist[nb] = all
        {
            unsigned c[kSplitBins], sum = 0u;
#pragma unroll
            for (int i = 0; i < kSplitBins; i += 4) {
                uint4 v = make_uint4(0u, 0u, 0u, 0u);
                if ((int)threadIdx.x < threads_used) v = ((const uint4*)hist)[(threadIdx.x * kSplitBins + i) >> 2];
                c[i] = v.x, c[i + 1] = v.y, c[i + 2] = v.z, c[i + 3] = v.w;
                sum += v.x + v.y + v.z + v.w;
            }
            unsigned incl = sum;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const unsigned o = __shfl_up_sync(0xffffffffu, incl, d);
                if (lane >= d) incl += o;
            }
            if (lane == 31) warp_sum[wid] = incl;
            __syncthreads();
            unsigned before = lane < kSplitThreads / 32 && lane < wid ? warp_sum[lane] : 0u;
            before = __reduce_add_sync(0xffffffffu, before);
            unsigned run = before + incl - sum;
#pragma unroll
            for (int i = 0; i < kSplitBins; i += 4) {
                uint4 v;
                v.x = run, run += c[i];
                v.y = run, run += c[i + 1];
                v.z = run, run += c[i + 2];
                v.w = run, run += c[i + 3];
                if ((int)threadIdx.x < threads_used) ((uint4*)hist)[(threadIdx.x * kSplitBins + i) >> 2] = v;
            }
            if (threadIdx.x == kSplitThreads - 1) hist[kMaxSmemBuckets] = run;
        }
        __syncthreads();
        const int total = (int)hist[nb];
        // reserve this tile's run in every non-empty bucket; the atomics of
        // one thread are independent, and their results are first needed after
        // the placing below
        unsigned first[kSplitBins];
#pragma unroll
        for (int i = 0; i < kSplitBins; ++i) {
            const int b = threadIdx.x + i * kSplitThreads;
            const unsigned c = b < nb ? hist[b + 1] - hist[b] : 0u;
            first[i] = c ? (unsigned)bstart[I.bucket_base + b] + atomicAdd(&bfill[I.bucket_base + b], c) : 0u;
        }
#pragma unroll
        for (int j = 0; j < kSplitPer; ++j) {
            if (bucket[j] < 0) continue;
            const int p = (int)(hist[bucket[j]] + rank[j]);
            sent[p] = make_uint2(key[j], ((unsigned)bucket[j] << kSplitPosBits) |
                                             (unsigned)(threadIdx.x + j * kSplitThreads));
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();  // every place is read and every value has landed
#pragma unroll
        for (int i = 0; i < kSplitBins; ++i) {
            const int b = threadIdx.x + i * kSplitThreads;
            if (b < nb) hist[b] = first[i] - hist[b];  // batch-wide slots (< 2^32, checked on the host), modulo 2^32
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < kSplitPer; ++j) {
            const int p = threadIdx.x + j * kSplitThreads;
            if (p >= total) break;
            const uint2 e = sent[p];
            const unsigned q = e.y & ((1u << kSplitPosBits) - 1u);
            const double v = split_vals[q];
            // one 16-byte record: the key, the entry's COO position (orders
            // equal (row, col) keys) and the value
            rec_out[hist[e.y >> kSplitPosBits] + (unsigned)p] =
                make_uint4(e.x, (unsigned)t0 + q, (unsigned)__double2loint(v), (unsigned)__double2hiint(v));
        }
        __syncthreads();
    }
    if (bad) raise_error(err, ERRBIT_BOUNDS);
}

// ---- stage 4 ------------------------------------------------------------------
// With invalid entries in a batch (reported by the count and split stages) a
// bucket's count can include an entry whose record the split did not write
// (a valid row with an invalid column): every column is bounded by ncols
// before x is read, so such a slot cannot index outside x.
//
// Equal (row, col) keys must keep their COO order (the runtime's stable
// sort_indices).  The split's order inside a bucket is arbitrary, so after the
// sort every run of equal keys is put in COO-position order (insertion sort
// by the thread that owns the run's first slot; duplicates are rare).
__device__ __forceinline__ double bk_rec_val(const uint4& r) { return __hiloint2double((int)r.w, (int)r.z); }

template <class IdxT>
__device__ __forceinline__ void bk_order_equal_keys(const unsigned* key, IdxT* pos, int E,
                                                    const uint4* __restrict__ rec) {
    for (int p = threadIdx.x; p + 1 < E; p += blockDim.x) {
        if (key[p + 1] != key[p] || (p > 0 && key[p - 1] == key[p])) continue;
        int q = p + 2;
        while (q < E && key[q] == key[p]) ++q;
        for (int i = p + 1; i < q; ++i) {
            const IdxT v = pos[i];
            const unsigned kv = rec[v].y;  // COO position
            int j = i - 1;
            while (j >= p && rec[pos[j]].y > kv) {
                pos[j + 1] = pos[j];
                --j;
            }
            pos[j + 1] = v;
        }
    }
}

// The radix form, for buckets with clustered columns.  One warp per bucket: a
// warp sorts its own bucket with no block barrier, so fifteen independent
// buckets are in flight per SM.  (A CTA per ~800-entry bucket pays its fixed
// work -- zeroing and scanning a counter set per warp, five block barriers per
// radix pass -- once per bucket.)
//  * key24 = row_in_bucket << cbits | col, kept to its 6 + cbits <= 24 bits,
//    sorted by stable LSD passes of 8 bits (at most three);
//  * the digit counts of every pass are taken in one sweep when the keys are
//    loaded (the multiset of digits does not change between passes), as
//    16-bit counts packed two to a word (digits d and d + 128);
//  * pass 0 reads key24 with the implicit index = position and writes
//    (key24 >> 8) << 11 | index; later passes move that word, whose bits
//    8k + 3 ... hold digit k, so one 32-bit word per entry carries both the
//    remaining key and the entry index;
//  * each pass ranks 32 positions per round among the lanes holding the same
//    digit (bk_rank_pass), so equal digits keep their order;
//  * after the sort every slot's record is gathered once for its full key,
//    CSR column and value, 32 consecutive slots per step, which also gives
//    the row starts and any equal neighbouring keys; runs of equal keys are
//    then put in COO order.
// Row starts come from the masked keys, which are sorted on every bit they
// have whatever the records hold, so every row range stays inside [0, E].
// It has room for 1536 entries per warp (fifteen warps per SM).
constexpr int kBkRadixCap = 1536;    // entries a bucket of the radix form may have
constexpr int kBkWarpIdxBits = 11;   // entry index bits: buckets of at most 2048 entries
constexpr unsigned kBkWarpIdxMask = (1u << kBkWarpIdxBits) - 1u;
constexpr int kBkWarpMaxCbits = 24 - kBkShift;
constexpr int kBkWarpPerSm = 3;  // resident CTAs of the radix form per SM
constexpr int kBkWarps = 5;
// per warp (32-bit words): two key buffers, packed digit counts of three
// passes, the running digit bases (later the row starts)
template <int kCap>
__host__ __device__ constexpr int bk_warp_words() { return 2 * kCap + 3 * 128 + 256; }
template <int kCap>
constexpr size_t bk_warp_smem() { return (size_t)kBkWarps * bk_warp_words<kCap>() * 4; }

// The sort key of a record: row_in_bucket << cbits | col, kept to its 6 + cbits
// bits (which change nothing for a valid entry, and keep every key's row
// below kBkRows whatever an unwritten slot holds).
__device__ __forceinline__ unsigned bk_key24(unsigned k, int cbits) {
    return (((k >> 24) << cbits) | (k & 0xFFFFFFu)) & ((1u << (kBkShift + cbits)) - 1u);
}

// One stable scatter pass of the warp sort: positions 0 .. E-1 of src, 32 per
// round, go to dst at base[digit] + (their rank among the round's lanes with
// the same digit); base[] holds the running digit offsets.  Lanes holding
// the same digit are found with one ballot per digit bit (the ALU pipe); a
// match instruction per round (the ADU pipe) kept that pipe 66% busy and was
// slower.  (Skipping the digit bits a pass cannot hold made no difference.)
__device__ __forceinline__ void bk_rank_pass(const unsigned* src, unsigned* dst, int E, int shift, bool first,
                                             unsigned* base, int lane, unsigned lt) {
    for (int p0 = 0; p0 < E; p0 += 32) {
        const int p = p0 + lane;
        const bool ok = p < E;
        const unsigned v = ok ? src[p] : 0u;
        const unsigned d = (v >> shift) & 0xFFu;
        unsigned peers = __ballot_sync(0xffffffffu, ok);
#pragma unroll
        for (int b = 0; b < 8; ++b) {
            const unsigned bb = __ballot_sync(0xffffffffu, (d >> b) & 1u);
            peers &= ((d >> b) & 1u) ? bb : ~bb;
        }
        unsigned at = 0;
        if (ok) at = base[d];
        __syncwarp();
        if (ok) {
            const unsigned before = peers & lt;
            dst[at + __popc(before)] = first ? (((v >> 8) << kBkWarpIdxBits) | (unsigned)p) : v;
            if (before == 0u) base[d] = at + __popc(peers);
        }
        __syncwarp();
    }
}

// The bucket sort of the 512-instance batch (2.9e8 entries): 5.22 + 0.21 ms with
// the radix form for every bucket and the block-wide kernel, 1.56 + 0.65 + 0.04
// ms now.  Buckets whose columns are not clustered take no rank chain: one
// counting pass puts every entry into a bin, the bins being in (row, column)
// order, and the few entries that share a bin are ordered by comparing them.
//  * row r owns as many bins as it has entries, its columns spread evenly over
//    them: bin = start + (col - first) * L / width, in float, which is monotone
//    in col.  First the width is the whole row (scattered columns: a bin holds
//    one entry on average); when a bin gets more entries than a rank can count, the
//    row's own smallest and largest column (bands);
//  * an atomic gives each entry its (arbitrary) rank in its bin; a scan of the
//    bin counts gives the bins' starts;
//  * an entry's final place is its bin's start plus the number of entries in
//    the bin that sort before it (equal keys: by COO position).
// The bucket's records come to shared memory in one bulk copy, and four warps
// share the bucket.  The L1 pipe bounds the kernel (about 41 wavefronts per 32
// entries); a thread's at most eight keys, and the packed words made of them,
// stay in registers from the first read to the last placing (kept in shared
// memory, the keys a record apart, they took 14 wavefronts more: 1.77 + 0.70
// ms); with a warp per bucket shared memory left 14 warps per SM and the
// phases' latencies bound it, and reading the values from global memory in
// sorted order, a line per lane, was a third of the pipe's work.  A bucket
// whose bins overflow both ways goes to `clustered` (the radix form below), a
// bucket above kCap, or of an instance with more than 2^18 columns, to
// `overflow`.  The kernel runs twice: over all buckets with room for 1024
// entries (nine per SM), and over the larger ones with room for 2048.
template <int kCap>
constexpr int bk_place_threads() { return kCap <= 1024 ? 128 : 256; }
template <int kCap>
constexpr int bk_place_per_sm() { return kCap <= 1024 ? 9 : 4; }
// A packed word holds an 18-bit column, a bin or entry number and, in the bits
// that are left, a rank in a bin: bins of at most 16 entries, or 8.
template <int kCap>
constexpr int bk_place_idx_bits() { return kCap <= 1024 ? 10 : 11; }
constexpr int kBkColBits = 24 - kBkShift;
// 32-bit words: the records | entries by bin | bin counts, later starts (16
// bits) | row starts and lengths | row minima | row maxima, later scales
template <int kCap>
__host__ __device__ constexpr int bk_place_words() { return 4 * kCap + kCap + 4 + kCap / 2 + 3 * kBkRows; }
template <int kCap>
constexpr size_t bk_place_smem() { return (size_t)bk_place_words<kCap>() * 4; }

// kList: the items are a list that another kernel filled (its length in device
// memory); otherwise every bucket of the batch, in order.
template <int kCap, bool kList>
__global__ void __launch_bounds__(bk_place_threads<kCap>(), bk_place_per_sm<kCap>()) bk_bucket_place_kernel(
    const BkInst* __restrict__ inst, const BkItem* __restrict__ items, unsigned nitems_host,
    const unsigned* nitems_dev, unsigned* cursor,
    const long long* __restrict__ bstart, const unsigned* __restrict__ bcount, const uint4* __restrict__ rec_in,
    BkItem* __restrict__ overflow, unsigned* overflow_count, BkItem* __restrict__ clustered,
    unsigned* clustered_count, unsigned* err) {
    extern __shared__ __align__(128) unsigned bkw_smem[];
    __shared__ __align__(8) unsigned long long sh_bar;
    __shared__ unsigned sh_next, sh_part[bk_place_threads<kCap>() / 32];
    __shared__ BkItem sh_item;    // the next bucket, ...
    __shared__ int sh_entries;    // ... its entries
    __shared__ long long sh_slot;  // and its first slot: read ahead by thread 0
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int T = bk_place_threads<kCap>(), kIdx = bk_place_idx_bits<kCap>(), kPer = kCap / T;
    constexpr int kRankAt = kIdx + kBkColBits, kRankBits = 32 - kRankAt;
    constexpr unsigned kBinMax = 1u << kRankBits, kIdxMask = (1u << kIdx) - 1u;
    constexpr unsigned kColMask = (1u << kBkColBits) - 1u, kRankMask = (kBinMax - 1u) << kRankAt;
    static_assert(kCap <= (1 << kIdx), "entry and bin numbers must fit their field");
    uint4* const rec = reinterpret_cast<uint4*>(bkw_smem);
    unsigned* const ord = reinterpret_cast<unsigned*>(rec + kCap);  // rank | column | entry number, by bin (kRankAt, kIdx)
    unsigned* const cntw = ord + kCap + 4;                          // two 16-bit counts per word
    const unsigned short* const start = reinterpret_cast<const unsigned short*>(cntw);
    unsigned* const rowinfo = cntw + kCap / 2;  // start | length << 16
    unsigned* const rowmin = rowinfo + kBkRows;
    unsigned* const rowmax = rowmin + kBkRows;
    const unsigned bar = (unsigned)__cvta_generic_to_shared(&sh_bar);
    const unsigned nitems = kList ? *(volatile const unsigned*)nitems_dev : nitems_host;
    if (tid == 0) {
        mbar_init(bar, 1);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    // thread 0: draws a bucket and reads what the block needs to start on it
    auto draw = [&]() {
        const unsigned nx = atomicAdd(cursor, 1u);
        sh_next = nx;
        if (nx >= nitems) return;
        const BkItem nw = items[nx];
        const long long gb = kList ? inst[nw.inst].bucket_base + nw.tile : (long long)nx;  // its number in the batch
        const int nE = (int)bcount[gb];
        const long long ns = bstart[gb];
        sh_item = nw;
        sh_entries = nE;
        sh_slot = ns;
        if (nE <= kCap) l2_prefetch(rec_in + ns, (int64_t)nE * 16);
    };
    if (tid == 0) draw();
    unsigned parity = 0;
    int last_inst = -1, skip = 0;
    for (;;) {
        __syncthreads();
        const unsigned it = sh_next;
        if (it >= nitems) break;
        const BkItem w = sh_item;
        const int E = sh_entries;
        const long long s0 = sh_slot;
        const BkInst& I = inst[w.inst];
        const long long ncols = I.ncols;
        // bits of the largest column: the smallest c with 2^c >= ncols
        const int cbits = ncols > 1 ? 64 - __clzll((unsigned long long)(ncols - 1)) : 0;
        const bool fits = E <= kCap && cbits <= kBkWarpMaxCbits;
        // after a clustered bucket the next 31 that this block draws of its
        // instance go the same way untried
        if (w.inst != last_inst) skip = 0;
        last_inst = w.inst;
        const bool tried = skip == 0 || E > kBkRadixCap;
        if (!tried) --skip;
        const bool copied = E > 0 && fits && tried;
        if (copied && tid == 0) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the last bucket's accesses are over
            mbar_expect_tx(bar, (unsigned)E * 16u);
            bulk_load_1d((unsigned)__cvta_generic_to_shared(rec), rec_in + s0, (unsigned)E * 16u, bar);
        }
        const unsigned cmask = (1u << (cbits & 31)) - 1u;
        if (tid < kBkRows) rowinfo[tid] = 0u;
        for (int i = tid; i < (E + 1) / 2 && i < kCap / 2; i += T) cntw[i] = 0u;
        bool ok = true;
        if (copied) {
            ok = mbar_wait_bounded(bar, parity);
            parity ^= 1u;
        }
        if (__syncthreads_or(!ok)) {
            if (tid == 0) {
                raise_error(err, ERRBIT_TIMEOUT);
                mbar_wait_bounded(bar, parity ^ 1u);  // let the copy land before the memory is released
            }
            return;
        }
        if (tid == 0) draw();  // (everyone has read the current one)
        bool big = !tried;
        unsigned kk[kPer];  // this thread's keys, later their packed words
        auto load_keys = [&]() {
#pragma unroll
            for (int j = 0; j < kPer; ++j) kk[j] = tid + j * T < E ? bk_key24(rec[tid + j * T].x, cbits) : 0u;
        };
        if (fits && tried) {
            load_keys();
#pragma unroll
            for (int j = 0; j < kPer; ++j)
                if (tid + j * T < E) atomicAdd(&rowinfo[kk[j] >> cbits], 1u);
            __syncthreads();
            if (warp == 0) {  // lane l owns rows 2l, 2l + 1
                const unsigned n0 = rowinfo[2 * lane], n1 = rowinfo[2 * lane + 1];
                unsigned incl = n0 + n1;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const unsigned y = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += y;
                }
                const unsigned st = incl - n0 - n1;
                rowinfo[2 * lane] = st | n0 << 16;
                rowinfo[2 * lane + 1] = (st + n0) | n1 << 16;
            }
            __syncthreads();
            const float whole = 1.0f / (float)(cmask + 1u);  // a power of two: exact
            for (int tier = 0; tier < 2; ++tier) {
                if (tier == 1) {  // the rows' own widths
                    load_keys();
                    if (tid < kBkRows) {
                        rowmin[tid] = 0xFFFFFFFFu;
                        rowmax[tid] = 0u;
                    }
                    for (int i = tid; i < (E + 1) / 2; i += T) cntw[i] = 0u;
                    __syncthreads();
#pragma unroll
                    for (int j = 0; j < kPer; ++j) {
                        if (tid + j * T >= E) break;
                        const unsigned r = kk[j] >> cbits, c = kk[j] & cmask;
                        atomicMin(&rowmin[r], c);
                        atomicMax(&rowmax[r], c);
                    }
                    __syncthreads();
                    if (tid < kBkRows) {
                        const unsigned L = rowinfo[tid] >> 16;
                        const float f = L ? (float)L / (float)(rowmax[tid] - rowmin[tid] + 1u) : 0.0f;
                        rowmax[tid] = __float_as_uint(f);
                    }
                    __syncthreads();
                }
                big = false;
#pragma unroll
                for (int j = 0; j < kPer; ++j) {
                    if (tid + j * T >= E) break;
                    const unsigned r = kk[j] >> cbits, c = kk[j] & cmask;
                    const unsigned ri = rowinfo[r], L = ri >> 16;
                    const float f = tier == 0 ? (float)c * ((float)L * whole)
                                              : (float)(c - rowmin[r]) * __uint_as_float(rowmax[r]);
                    const unsigned o = (unsigned)f;
                    const unsigned bb = (ri & 0xFFFFu) + (o < L ? o : L - 1u);
                    const unsigned sh = (bb & 1u) << 4;
                    const unsigned rank = (atomicAdd(&cntw[bb >> 1], 1u << sh) >> sh) & 0xFFFFu;
                    big |= rank >= kBinMax;
                    kk[j] = rank << kRankAt | bb << kBkColBits | c;  // (a second try reads the keys again)
                }
                big = __syncthreads_or(big);
                if (!big) break;
            }
            if (big) skip = 31;
        }
        if (!fits || big) {  // block-uniform
            if (tid == 0) {
                if (!fits || E > kBkRadixCap) overflow[atomicAdd(overflow_count, 1u)] = w;
                else clustered[atomicAdd(clustered_count, 1u)] = w;
            }
            continue;
        }
        // counts -> starts; a thread owns an odd number of words (no bank conflicts)
        const int words = (E + 1) >> 1, W = ((words + T - 1) / T) | 1;
        const int w0 = tid * W < words ? tid * W : words, w1 = w0 + W < words ? w0 + W : words;
        unsigned sum = 0;
        for (int q = w0; q < w1; ++q) sum += cntw[q];  // both halves at once: at most kCap in all
        sum = (sum & 0xFFFFu) + (sum >> 16);
        unsigned incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) sh_part[warp] = incl;
        __syncthreads();
        unsigned run = incl - sum;
#pragma unroll
        for (int u = 0; u < T / 32; ++u) run += u < warp ? sh_part[u] : 0u;
        for (int q = w0; q < w1; ++q) {
            const unsigned c = cntw[q], lo = run + (c & 0xFFFFu);
            cntw[q] = run | lo << 16;
            run = lo + (c >> 16);
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            const int p = tid + j * T;
            if (p >= E) break;
            const unsigned v = kk[j], rank = v & kRankMask;
            ord[start[(v >> kBkColBits) & kIdxMask] + (rank >> kRankAt)] = rank | (v & kColMask) << kIdx | (unsigned)p;
        }
        if (tid == 0) ord[E] = 0u;  // the end of the last bin
        __syncthreads();
        const long long e0 = s0 - I.scan_base;
        int* const csr_cols = I.csr_cols + e0;
        double* const csr_vals = I.csr_vals + e0;
#pragma unroll 2
        for (int q = tid; q < E; q += T) {
            const unsigned me = ord[q];
            const uint2 v = *reinterpret_cast<const uint2*>(&rec[me & kIdxMask].z);
            // the bin is the slots from the one of rank 0 to before the next of rank 0
            int k = q - (int)(me >> kRankAt), at = k;
            unsigned other = ord[k];
            do {
                if ((other ^ me) << kRankBits >> (kRankBits + kIdx)) at += other << kRankBits < me << kRankBits;
                else if (k != q)  // equal (row, col): COO order
                    at += rec[other & kIdxMask].y < rec[me & kIdxMask].y;
                other = ord[++k];
            } while (other >> kRankAt);
            csr_cols[at] = (int)((me >> kIdx) & kColMask);
            csr_vals[at] = __hiloint2double((int)v.y, (int)v.x);
        }
        const long long r0 = (long long)w.tile << kBkShift;
        const int nr = (int)((I.nrows - r0) < kBkRows ? (I.nrows - r0) : kBkRows);
        for (int r = tid; r <= nr; r += T) {
            if (r < nr) I.row_ptr[r0 + r] = e0 + (rowinfo[r] & 0xFFFFu);
            else if (r0 + nr == I.nrows) I.row_ptr[I.nrows] = I.nnz;
        }
    }
}

template <int kCap>
__global__ void __launch_bounds__(kBkWarps * 32, kBkWarpPerSm) bk_bucket_radix_kernel(
    const BkInst* __restrict__ inst, const BkItem* __restrict__ items, const unsigned* nitems_dev, unsigned* cursor,
    const long long* __restrict__ bstart, const unsigned* __restrict__ bcount, const uint4* __restrict__ rec_in) {
    extern __shared__ __align__(16) unsigned bkw_smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    static_assert(kCap <= (1 << kBkWarpIdxBits), "entry indices must fit their field");
    unsigned* const a = bkw_smem + (size_t)warp * bk_warp_words<kCap>();
    unsigned* const b = a + kCap;
    unsigned* const hist = b + kCap;  // [3][128]
    const unsigned nitems = *(volatile const unsigned*)nitems_dev;  // a list another kernel filled
    unsigned* const base = hist + 3 * 128;  // [256]; row starts [65] after the sort
    unsigned lt;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));
    for (;;) {
        unsigned it = 0;
        if (lane == 0) it = atomicAdd(cursor, 1u);
        it = __shfl_sync(0xffffffffu, it, 0);
        if (it >= nitems) break;
        const BkItem w = items[it];
        const BkInst I = inst[w.inst];
        const long long gb = I.bucket_base + w.tile;
        const int E = (int)bcount[gb];
        // bits of the largest column: the smallest c with 2^c >= ncols
        const int cbits = I.ncols > 1 ? 64 - __clzll((unsigned long long)(I.ncols - 1)) : 0;
        const long long s0 = bstart[gb];
        const long long e0 = s0 - I.scan_base;
        const long long r0 = (long long)w.tile << kBkShift;
        const int nr = (int)((I.nrows - r0) < kBkRows ? (I.nrows - r0) : kBkRows);
        const int passes = (kBkShift + cbits + 7) >> 3;  // 1..3
        // keys and the digit counts of every pass
        // every lane's key words are in flight at once (4-byte cp.async of
        // each record's key field), so the bucket waits for one memory latency
        for (int p = lane; p < E; p += 32)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(a + p)),
                         "l"(&rec_in[s0 + p].x)
                         : "memory");
        asm volatile("cp.async.commit_group;" ::: "memory");
        for (int i = lane; i < 3 * 128; i += 32) hist[i] = 0u;
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncwarp();
        for (int p = lane; p < E; p += 32) {
            const unsigned key = bk_key24(a[p], cbits);
            a[p] = key;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                if (k < passes) {
                    const unsigned d = (key >> (8 * k)) & 0xFFu;
                    atomicAdd(&hist[k * 128 + (d & 127u)], (d & 128u) ? 0x10000u : 1u);
                }
            }
        }
        __syncwarp();
        unsigned* src = a;
        unsigned* dst = b;
        for (int k = 0; k < passes; ++k) {
            // exclusive scan of the 256 digit counts; lane l owns digits 8l .. 8l+7
            unsigned c[8], sum = 0;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int d = 8 * lane + j;
                c[j] = (hist[k * 128 + (d & 127)] >> ((d & 128) ? 16 : 0)) & 0xFFFFu;
                sum += c[j];
            }
            unsigned incl = sum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            unsigned run = incl - sum;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                base[8 * lane + j] = run;
                run += c[j];
            }
            __syncwarp();
            const int shift = k == 0 ? 0 : 8 * k + 3;
            bk_rank_pass(src, dst, E, shift, k == 0, base, lane, lt);
            unsigned* t = src;
            src = dst;
            dst = t;
        }
        // src: entry indices in (row, col) order; dst: free for the keys
        unsigned* const ord = src;
        unsigned* const key = dst;
        const unsigned cmask = (1u << cbits) - 1u;
        // One pass over the sorted positions, 32 consecutive ones per warp step:
        // gather each record for its key, CSR column and value, and find the
        // row starts and any equal neighbouring keys from the neighbour's key
        // (a shuffle; the step before hands over its last key).
        unsigned* const rowb = base;  // [kBkRows + 1]
        constexpr int kG = 8;         // records in flight per lane
        unsigned prev_key = 0u;
        int prev_row = -1;  // row of the position before the current step (-1: none)
        bool dup = false;
        for (int c0 = 0; c0 < E; c0 += 32 * kG) {
            uint4 r[kG];
#pragma unroll
            for (int u = 0; u < kG; ++u) {
                const int p = c0 + 32 * u + lane;
                if (p < E) r[u] = rec_in[s0 + (ord[p] & kBkWarpIdxMask)];
            }
#pragma unroll
            for (int u = 0; u < kG; ++u) {
                const int p = c0 + 32 * u + lane;
                const bool in = p < E;
                unsigned k24 = 0u;
                if (in) {
                    k24 = bk_key24(r[u].x, cbits);
                    key[p] = k24;
                    I.csr_cols[e0 + p] = (int)(k24 & cmask);
                    I.csr_vals[e0 + p] = bk_rec_val(r[u]);
                }
                const int row = in ? (int)(k24 >> cbits) : kBkRows;
                const unsigned kup = __shfl_up_sync(0xffffffffu, k24, 1);
                const int rup = __shfl_up_sync(0xffffffffu, row, 1);
                const unsigned kprev = lane == 0 ? prev_key : kup;
                const int rprev = lane == 0 ? prev_row : rup;
                if (in) {
                    for (int rr = rprev + 1; rr <= row && rr < kBkRows; ++rr) rowb[rr] = (unsigned)p;
                    dup |= p > 0 && kprev == k24;
                }
                prev_key = __shfl_sync(0xffffffffu, k24, 31);
                prev_row = __shfl_sync(0xffffffffu, row, 31);
            }
        }
        __syncwarp();
        {  // rows after the last entry's row (every row when the bucket is empty) start at E
            const int last_row = E > 0 ? (int)(key[E - 1] >> cbits) : -1;
            for (int rr = last_row + 1 + lane; rr <= kBkRows; rr += 32) rowb[rr] = (unsigned)E;
        }
        // equal (row, col) keys in COO-position order (duplicates are rare)
        if (__any_sync(0xffffffffu, dup)) {
            for (int p = lane; p + 1 < E; p += 32) {
                if (key[p + 1] != key[p] || (p > 0 && key[p - 1] == key[p])) continue;
                int q = p + 2;
                while (q < E && key[q] == key[p]) ++q;
                for (int i = p + 1; i < q; ++i) {
                    const unsigned v = ord[i];
                    const unsigned kv = rec_in[s0 + (v & kBkWarpIdxMask)].y;  // COO position
                    int j = i - 1;
                    while (j >= p && rec_in[s0 + (ord[j] & kBkWarpIdxMask)].y > kv) {
                        ord[j + 1] = ord[j];
                        --j;
                    }
                    ord[j + 1] = v;
                }
                for (int i = p; i < q; ++i)
                    I.csr_vals[e0 + i] = bk_rec_val(rec_in[s0 + (ord[i] & kBkWarpIdxMask)]);
            }
        }
        __syncwarp();
        for (int r = lane; r <= nr; r += 32) {
            if (r < nr) I.row_ptr[r0 + r] = e0 + rowb[r];
            else if (r0 + nr == I.nrows) I.row_ptr[I.nrows] = I.nnz;
        }
        __syncwarp();
    }
}

// Large buckets (up to 64 rows x 256): one CTA sorts the bucket's keys with a
// block-wide bitonic network in shared memory.  Reads its item count from
// device memory (filled by the placing kernels).
constexpr size_t kBkSmem = (size_t)kBkCap * 6 + 1024;

__global__ void __launch_bounds__(kBkThreads) bk_bucket_kernel(const BkInst* __restrict__ inst,
                                                               const BkItem* __restrict__ items,
                                                               const unsigned* nitems_dev, unsigned* cursor,
                                                               const long long* __restrict__ bstart,
                                                               const unsigned* __restrict__ bcount,
                                                               const uint4* __restrict__ rec_in, unsigned* err) {
    extern __shared__ __align__(16) unsigned char bk_smem[];
    unsigned* key = reinterpret_cast<unsigned*>(bk_smem);
    unsigned short* idx = reinterpret_cast<unsigned short*>(bk_smem + (size_t)kBkCap * 4);
    __shared__ int rstart[kBkRows + 1];
    const unsigned nitems = *nitems_dev;
    unsigned it;
    bool bad = false;
    while (bk_next(cursor, nitems, it)) {
        const BkItem w = items[it];
        const BkInst I = inst[w.inst];
        const long long gb = I.bucket_base + w.tile;
        const int E = (int)bcount[gb];
        const long long s0 = bstart[gb];        // batch-wide slot of the bucket's first entry
        const long long e0 = s0 - I.scan_base;  // instance-relative
        const long long r0 = (long long)w.tile << kBkShift;
        const int nr = (int)((I.nrows - r0) < kBkRows ? (I.nrows - r0) : kBkRows);
        if (E > kBkCap) {  // a row above 256 entries: outside the contract
            bad = true;
            continue;
        }
        int P = 1;
        while (P < E) P <<= 1;
        for (int i = threadIdx.x; i < P; i += kBkThreads) {
            key[i] = i < E ? rec_in[s0 + i].x : 0xFFFFFFFFu;
            idx[i] = (unsigned short)i;
        }
        __syncthreads();
        for (int size = 2; size <= P; size <<= 1) {
            for (int stride = size >> 1; stride > 0; stride >>= 1) {
                for (int i = threadIdx.x; i < P / 2; i += kBkThreads) {
                    const int lo = 2 * i - (i & (stride - 1));
                    const int hi = lo + stride;
                    const bool up = (lo & size) == 0;
                    const unsigned a = key[lo], b = key[hi];
                    if ((a > b) == up) {
                        key[lo] = b;
                        key[hi] = a;
                        const unsigned short t = idx[lo];
                        idx[lo] = idx[hi];
                        idx[hi] = t;
                    }
                }
                __syncthreads();
            }
        }
        for (int p = threadIdx.x; p <= E; p += kBkThreads) {
            const int rp = p == 0 ? -1 : (int)(key[p - 1] >> 24);
            const int rc = p == E ? nr : (int)(key[p] >> 24);
            for (int r = rp + 1; r <= rc && r <= nr; ++r) rstart[r] = p;
        }
        bk_order_equal_keys(key, idx, E, rec_in + s0);  // the bitonic network is not stable
        __syncthreads();
        for (int p = threadIdx.x; p < E; p += kBkThreads) {
            I.csr_cols[e0 + p] = (int)(key[p] & 0xFFFFFFu);
            I.csr_vals[e0 + p] = bk_rec_val(rec_in[s0 + idx[p]]);
        }
        for (int r = threadIdx.x; r <= nr; r += kBkThreads) {
            if (r < nr) I.row_ptr[r0 + r] = e0 + rstart[r];
            else if (r0 + nr == I.nrows) I.row_ptr[I.nrows] = I.nnz;
        }
        __syncthreads();
    }
    if (bad) raise_error(err, ERRBIT_BOUNDS);
}

// ---- stage 5 ------------------------------------------------------------------
// y[r] = the row's entries summed in column order as one fma chain (the
// reference's sequential row loop, with fused multiply-adds), computed from
// the finished CSR.  Each FP64 warp instruction holds the FP64 pipe for the
// whole warp whatever its active lanes, so one lane per row only pays when
// the 32 rows of a warp instruction have similar lengths: a warp takes a
// chunk of one instance's rows, counting-sorts them by length (256 bins,
// lengths above 255 share the last) in shared memory, and gives each lane one
// row of every group of 32 consecutive rows in that order.  A lane reads its
// row 4 entries at a time, ahead of the (in-order) chain.  Requests to L2 and
// their latency bound it, most of them x (2.9e8 entries: 2.06 ms with the values
// by 16-byte loads through L1 and x past it, 1.89 ms so; one loop per alignment
// of the values, as a choice inside the loop cost 0.07 ms).
// Chunks have 256 rows, halved down to 32 while the batch has fewer chunks than
// the chip has resident warps.  Whole pipeline: one instance of 2^13.5 to
// 2^16.3 rows 197 -> 153 us, 24 of 2^10 to 2^14 rows 283 -> 232, 4 of 2^16 to
// 2^18 rows 374 -> 351.  (Halving until there are four chunks per warp takes 64
// instances of 2^12 to 2^16 rows from 676 to 723 us.)  Chunks above 256 rows
// fill more lanes of the FP64 pipe, but their rows' entries no longer wait in
// L1 and L2 for the neighbouring rows: 2.2 ms with 512 rows instead of 2.06 for
// 2.9e8 entries, 3.0 ms with 1024.
// Rows above 256 entries are outside the contract and reported.
constexpr int kSpWarps = 8;
constexpr int kSpPerSm = 4;
struct BkSpSmem {
    unsigned cnt[256];
    unsigned start[kSpRows];
    unsigned short len[kSpRows];
    unsigned char order[kSpRows];
};

__global__ void __launch_bounds__(kSpWarps * 32, kSpPerSm)
    bk_spmv_kernel(const BkInst* __restrict__ inst, const BkItem* __restrict__ chunks, unsigned nchunks,
                   int chunk_rows, unsigned* cursor, unsigned* err) {
    __shared__ BkSpSmem sm_all[kSpWarps];
    const int lane = threadIdx.x & 31;
    BkSpSmem& sm = sm_all[threadIdx.x >> 5];
    bool bad = false;
    for (;;) {
        unsigned it = 0;
        if (lane == 0) it = atomicAdd(cursor, 1u);
        it = __shfl_sync(0xffffffffu, it, 0);
        if (it >= nchunks) break;
        const BkItem w = chunks[it];
        const BkInst I = inst[w.inst];
        const long long r0 = (long long)w.tile * chunk_rows;
        const int nr = (int)((I.nrows - r0) < chunk_rows ? (I.nrows - r0) : chunk_rows);
#pragma unroll
        for (int j = 0; j < 8; ++j) sm.cnt[lane + 32 * j] = 0u;
        __syncwarp();
        // row extents, kept inside [0, nnz] whatever the row pointers hold
        for (int i = lane; i < nr; i += 32) {
            long long a = I.row_ptr[r0 + i], e = I.row_ptr[r0 + i + 1];
            a = a < 0 ? 0 : (a > I.nnz ? I.nnz : a);
            e = e < a ? a : (e > I.nnz ? I.nnz : e);
            const long long L = e - a;
            bad |= L > 256;
            const unsigned l = L > 0xFFFF ? 0xFFFFu : (unsigned)L;
            sm.start[i] = (unsigned)a;
            sm.len[i] = (unsigned short)l;
            atomicAdd(&sm.cnt[l > 255u ? 255u : l], 1u);
        }
        __syncwarp();
        {  // exclusive scan of the 256 bin counts; lane l owns bins 8l .. 8l+7
            unsigned c[8], sum = 0;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                c[j] = sm.cnt[8 * lane + j];
                sum += c[j];
            }
            unsigned incl = sum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            unsigned run = incl - sum;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                sm.cnt[8 * lane + j] = run;
                run += c[j];
            }
        }
        __syncwarp();
        for (int i = lane; i < nr; i += 32) {
            const unsigned l = sm.len[i];
            sm.order[atomicAdd(&sm.cnt[l > 255u ? 255u : l], 1u)] = (unsigned char)i;
        }
        __syncwarp();
        const int* __restrict__ cols = I.csr_cols;
        const double* __restrict__ vals = I.csr_vals;
        const double* __restrict__ x = I.x;
        const unsigned long long ncols = (unsigned long long)I.ncols;
        for (int g = lane; g < nr; g += 32) {
            const int i = sm.order[g];
            const long long a = sm.start[i];
            const int L = sm.len[i];
            const int* __restrict__ rc = cols + a;
            const double* __restrict__ rv = vals + a;
            double acc = 0.0;
            // x is gathered through L1: the values pass it by, a whole sector per
            // load, and leave it to the columns' sectors, of two loads each, and x
            auto xat = [&](unsigned c) { return c < ncols ? __ldg(x + c) : 0.0; };
            // entries one at a time until the columns are 16-byte aligned, then
            // 4 per step: the columns by one 16-byte load, the values by one of
            // 32 bytes or two of 16 where their alignment (fixed per row) lets
            // it; the fma chain keeps the row's order throughout
            int k = 0;
            while (k < L && (reinterpret_cast<uintptr_t>(rc + k) & 15)) {
                acc = fma(rv[k], xat((unsigned)rc[k]), acc);
                ++k;
            }
            auto four = [&](double v0, double v1, double v2, double v3, const int4& c4) {
                const double x0 = xat((unsigned)c4.x), x1 = xat((unsigned)c4.y);
                const double x2 = xat((unsigned)c4.z), x3 = xat((unsigned)c4.w);
                acc = fma(v0, x0, acc);
                acc = fma(v1, x1, acc);
                acc = fma(v2, x2, acc);
                acc = fma(v3, x3, acc);
            };
            const unsigned va = (unsigned)reinterpret_cast<uintptr_t>(rv + k) & 31u;
            if (va == 0) {
                for (; k + 4 <= L; k += 4) {
                    const int4 c4 = *reinterpret_cast<const int4*>(rc + k);
                    const f64x4 p = ldg_stream_f64x4(rv + k);
                    four(p.x, p.y, p.z, p.w, c4);
                }
            } else if (va == 16) {
                for (; k + 4 <= L; k += 4) {
                    const int4 c4 = *reinterpret_cast<const int4*>(rc + k);
                    const double2 p = *reinterpret_cast<const double2*>(rv + k);
                    const double2 q = *reinterpret_cast<const double2*>(rv + k + 2);
                    four(p.x, p.y, q.x, q.y, c4);
                }
            } else {
                for (; k + 4 <= L; k += 4)
                    four(rv[k], rv[k + 1], rv[k + 2], rv[k + 3], *reinterpret_cast<const int4*>(rc + k));
            }
            for (; k < L; ++k) acc = fma(rv[k], xat((unsigned)rc[k]), acc);
            I.y[r0 + i] = acc;
        }
        __syncwarp();
    }
    if (bad) raise_error(err, ERRBIT_BOUNDS);
}

// Bucketed pipeline; returns HYD_CUDA_ERR_UNSUPPORTED (nothing launched) when a
// batch falls outside its limits so the caller can take the row-atomic path.
int batch_pipeline_bucketed(std::vector<BatchInst>& bi, const char* key, cudaStream_t s, void* staging,
                            size_t staging_bytes) {
    Device* d = nullptr;
    HYD_TRY(device(&d));
    std::vector<BkInst> inst(bi.size());
    long long nb_total = 0, entries = 0, nt_total = 0, nc_total = 0, rows_total = 0;
    for (const BatchInst& B : bi) rows_total += B.nrows;
    int chunk_rows = kSpRows;
    while (chunk_rows > kSpMinRows && rows_total < (long long)chunk_rows * kSpWarps * kSpPerSm * d->sm_count) chunk_rows /= 2;
    for (size_t i = 0; i < bi.size(); ++i) {
        const BatchInst& B = bi[i];
        if (B.ncols >= (1LL << 24) || B.nrows >= (1LL << 31)) return HYD_CUDA_ERR_UNSUPPORTED;
        BkInst& I = inst[i];
        I.nrows = B.nrows;
        I.ncols = B.ncols;
        I.nnz = B.nnz;
        I.nbuckets = (B.nrows + kBkRows - 1) / kBkRows;
        I.bucket_base = nb_total;
        I.scan_base = entries;
        I.rows = B.rows;
        I.cols = B.cols;
        I.vals = B.vals;
        I.x = B.x;
        I.row_ptr = B.row_ptr;
        I.csr_cols = B.csr_cols;
        I.csr_vals = B.csr_vals;
        I.y = B.y;
        I.tile_base = nt_total;
        I.chunk_base = nc_total;
        nt_total += (B.nnz + kTileEntries - 1) / kTileEntries;
        nc_total += (B.nrows + chunk_rows - 1) / chunk_rows;
        nb_total += I.nbuckets;
        entries += B.nnz;
    }
    if (nb_total >= (1LL << 31) || nt_total >= (1LL << 31) || nc_total >= (1LL << 31) || entries >= (1LL << 32))
        return HYD_CUDA_ERR_UNSUPPORTED;
    auto al = [](size_t b) { return (b + 255) & ~(size_t)255; };
    const size_t inst_b = al(inst.size() * sizeof(BkInst)), tiles_b = al((size_t)nt_total * sizeof(BkItem)),
                 bk_b = al((size_t)nb_total * sizeof(BkItem)), ch_b = al((size_t)nc_total * sizeof(BkItem));
    const size_t cnt_b = al((size_t)nb_total * 4), wide_b = al((size_t)nb_total * 8);
    const size_t vals_b = al((size_t)entries * 8);
    void* buf = nullptr;
    HYD_TRY(device_buffer(d, key, inst_b + tiles_b + 4 * bk_b + ch_b + 2 * cnt_b + 2 * wide_b + vals_b + vals_b + 256,
                          &buf));
    unsigned char* b = static_cast<unsigned char*>(buf);
    size_t off = 0;
    auto take = [&](size_t bytes) {
        unsigned char* p = b + off;
        off += bytes;
        return p;
    };
    BkInst* d_inst = reinterpret_cast<BkInst*>(take(inst_b));
    BkItem* d_tiles = reinterpret_cast<BkItem*>(take(tiles_b));
    BkItem* d_bk = reinterpret_cast<BkItem*>(take(bk_b));
    unsigned* bcount = reinterpret_cast<unsigned*>(take(cnt_b));
    unsigned* bfill = reinterpret_cast<unsigned*>(take(cnt_b));
    long long* wide = reinterpret_cast<long long*>(take(wide_b));
    long long* bstart = reinterpret_cast<long long*>(take(wide_b));
    uint4* recs = reinterpret_cast<uint4*>(take(2 * vals_b));  // (key, COO position, value) per entry
    BkItem* overflow = reinterpret_cast<BkItem*>(take(bk_b));  // buckets for the block-wide kernel
    BkItem* large = reinterpret_cast<BkItem*>(take(bk_b));      // buckets above 1024 entries
    BkItem* clustered = reinterpret_cast<BkItem*>(take(bk_b));  // buckets for the radix form
    BkItem* d_chunks = reinterpret_cast<BkItem*>(take(ch_b));
    unsigned* cursors = reinterpret_cast<unsigned*>(take(256));
    // only the instance table crosses from the host; the work lists are
    // written by bk_items_kernel
    const bool async_tables = staging != nullptr && staging_bytes >= inst_b;
    if (async_tables) {
        memcpy(staging, inst.data(), inst.size() * sizeof(BkInst));
        HYD_CUDA_TRY(cudaMemcpyAsync(d_inst, staging, inst.size() * sizeof(BkInst), cudaMemcpyHostToDevice, s));
    } else {
        HYD_CUDA_TRY(cudaMemcpyAsync(d_inst, inst.data(), inst.size() * sizeof(BkInst), cudaMemcpyHostToDevice, s));
    }
    {
        const int64_t ni = (int64_t)inst.size();
        const unsigned g = (unsigned)(ni < 4096 ? ni : 4096);
        bk_items_kernel<<<g, 256, 0, s>>>(d_inst, ni, d_tiles, d_bk, d_chunks, chunk_rows);
        HYD_TRY(launch_check("bk_items"));
    }
    const size_t n_tiles = (size_t)nt_total, n_buckets = (size_t)nb_total;
    HYD_CUDA_TRY(cudaMemsetAsync(bcount, 0, 2 * cnt_b, s));  // bcount and bfill
    HYD_CUDA_TRY(cudaMemsetAsync(cursors, 0, 64, s));
    const unsigned grid = (unsigned)(d->sm_count * 2);
    if (n_tiles) {
        bk_count_kernel<<<(unsigned)(d->sm_count * kCountPerSm), kBkThreads, 0, s>>>(d_inst, d_tiles,
                                                                                   (unsigned)n_tiles, bcount,
                                                                                   d->d_err);
        HYD_TRY(launch_check("bk_count"));
    }
    bk_widen_kernel<<<grid, 256, 0, s>>>(bcount, wide, nb_total);
    HYD_TRY(launch_check("bk_widen"));
    HYD_TRY(scan_i64_launch(wide, bstart, nb_total, 0, false, false, s));
    if (n_tiles) {
        HYD_TRY(configure_kernel((const void*)bk_split_kernel, d, false));
        bk_split_kernel<<<(unsigned)(d->sm_count * kSplitPerSm), kSplitThreads, kSplitSmem, s>>>(
            d_inst, d_tiles, (unsigned)n_tiles, cursors + 1, bstart, bfill, recs, d->d_err);
        HYD_TRY(launch_check("bk_split"));
    }
    // cursors: 2 the buckets of at most 1024 entries, 9 the larger ones (8: how
    // many), 7 the radix form (6: how many), 3 the block-wide kernel (4: how many)
    {
        auto k0 = bk_bucket_place_kernel<1024, false>;
        HYD_TRY(configure_kernel((const void*)k0, d, false));
        k0<<<(unsigned)(d->sm_count * bk_place_per_sm<1024>()), bk_place_threads<1024>(), bk_place_smem<1024>(), s>>>(
            d_inst, d_bk, (unsigned)n_buckets, nullptr, cursors + 2, bstart, bcount, recs, large, cursors + 8,
            clustered, cursors + 6, d->d_err);
        HYD_TRY(launch_check("bk_bucket_place"));
        auto k1 = bk_bucket_place_kernel<2048, true>;
        HYD_TRY(configure_kernel((const void*)k1, d, false));
        k1<<<(unsigned)(d->sm_count * bk_place_per_sm<2048>()), bk_place_threads<2048>(), bk_place_smem<2048>(), s>>>(
            d_inst, large, 0u, cursors + 8, cursors + 9, bstart, bcount, recs, overflow, cursors + 4, clustered,
            cursors + 6, d->d_err);
        HYD_TRY(launch_check("bk_bucket_place"));
        auto k2 = bk_bucket_radix_kernel<kBkRadixCap>;
        HYD_TRY(configure_kernel((const void*)k2, d, false));
        k2<<<(unsigned)(d->sm_count * kBkWarpPerSm), kBkWarps * 32, bk_warp_smem<kBkRadixCap>(), s>>>(
            d_inst, clustered, cursors + 6, cursors + 7, bstart, bcount, recs);
        HYD_TRY(launch_check("bk_bucket_radix"));
    }
    HYD_TRY(configure_kernel((const void*)bk_bucket_kernel, d, false));
    bk_bucket_kernel<<<grid, kBkThreads, kBkSmem, s>>>(d_inst, overflow, cursors + 4, cursors + 3, bstart, bcount,
                                                       recs, d->d_err);
    HYD_TRY(launch_check("bk_bucket_large"));
    if (nc_total) {
        bk_spmv_kernel<<<(unsigned)(d->sm_count * kSpPerSm), kSpWarps * 32, 0, s>>>(
            d_inst, d_chunks, (unsigned)nc_total, chunk_rows, cursors + 5, d->d_err);
        HYD_TRY(launch_check("bk_spmv"));
    }
    if (!async_tables) HYD_CUDA_TRY(cudaStreamSynchronize(s));
    return HYD_CUDA_OK;
}

size_t batch_pipeline_bucketed_table_bytes(const std::vector<BatchInst>& bi) {
    return (bi.size() * sizeof(BkInst) + 255) & ~(size_t)255;
}

}  // namespace hyd
