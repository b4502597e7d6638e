// sort.cu -- sort_indices (stable LSD radix, 8-bit digits) and gather.
//
// Replaces the runtime's serial hyd_radix_sort_entries / hyd_sort_indices
// (runtime/hydrangea_runtime.h:386-456), reached from `sort_indices`
// (Lowering.hs:961-965).  The result must be the same permutation, so the
// digit function and pass count are the runtime's: digit p of a key is
// (key >> 8p) & 0xFF on the signed key, and the number of passes is the
// number of bytes of max(0, max key) (at least one).  Any stable LSD sort with
// those digits yields exactly that permutation.
//
// One sweep of the keys counts every pass's digits; then each pass is one
// launch that reads and writes every element once (a decoupled look-back per
// digit; Adinets and Merrill, "Onesweep", 2022):
//  * a tile ranks its elements by digit: each warp takes 32 at a time and ranks
//    them among the lanes holding the same digit, which set their bits in a word
//    of the (warp, digit) in shared memory (running counts beside it), in
//    element order;
//  * per digit, one thread publishes the tile's count and looks back over the
//    earlier tiles' words for the digit's first output position;
//  * the tile is put in digit order in shared memory and written out in runs.
// An element travels as the digits still to come and its index: 8 bytes when
// both fit 32 bits (so after the first pass for keys of up to 40 bits), else
// 16.  The first pass reads the int64 keys, the last writes the permutation.
//
// What bounds it: the shared-memory pipe (rank, reorder and write-out take about
// 45 wavefronts per 32 elements) and the chain ticket - load - rank - look-back
// of a tile; the bytes, 16 per element and pass, are a third of the time.
// Measured at 2^24 keys of 36 bits (5 passes): 542 us, 53 of it the counts,
// against 1615 us with three launches per pass (tile histogram, scan, scatter
// straight from registers) and 8-byte keys and indices.
#include <climits>
#include <cstddef>
#include <type_traits>

#include "hyd_common.cuh"

namespace hyd {

// 384 threads, two CTAs per SM (80 registers): 107 us for a middle pass; 512 x 2
// (64 registers, spills) 133, 256 x 4 122, 384 x 3 125.
constexpr int kSortT = 384;
constexpr int kSortCtasPerSm = 2;
constexpr int kSortWarps = kSortT / 32;
constexpr int kSortBins = 256;
constexpr int kSortMaxPasses = 8;
typedef unsigned long long u64;

// What a pass reads and writes.
struct SortKeys {};                  // in: the caller's keys, index = position
struct SortRec8 { unsigned key, idx; };  // one 8-byte record
struct SortRec16 { u64 key, idx; };  // two arrays
struct SortPerm {};                  // out: the permutation

template <class Out, bool kWide>
struct SortTile {  // elements per thread, and what is staged per element in shared memory
    static constexpr int kPer = 16;
    typedef unsigned Staged;
};
template <>
struct SortTile<SortPerm, true> {
    static constexpr int kPer = 8;
    typedef u64 Staged;
};
template <bool kWide>
struct SortTile<SortRec8, kWide> {
    static constexpr int kPer = 16;
    typedef SortRec8 Staged;
};
template <bool kWide>
struct SortTile<SortRec16, kWide> {
    static constexpr int kPer = 8;
    typedef SortRec16 Staged;
};

// A (tile, digit) word of the look-back: the two top bits are the state (0
// nothing, 1 the tile's count, 2 the count of all tiles up to it), the rest
// the count.  64 bits for 2^30 elements and more (kWide).
template <bool kWide>
struct SortWord {
    typedef unsigned T;
};
template <>
struct SortWord<true> {
    typedef u64 T;
};

// Digit counts of all eight possible passes in one read of the keys, and the
// largest key.  Digit 0 is not counted (its count is what is left of n), so
// the passes above the largest key cost next to nothing; a digit that a whole
// warp shares (four warp-wide reductions of the keys' words tell for all eight)
// costs one add.  The shared atomics bound it: 53 us for 2^24 keys of 36 bits,
// 63 with a ballot, a shuffle and 64-bit shifts per digit.  The last block turns
// the counts into each digit's first position (first[pass][digit]).
__global__ void __launch_bounds__(1024) sort_count_kernel(const long long* __restrict__ keys, int64_t n,
                                                          u64* __restrict__ max_key, u64* __restrict__ counts,
                                                          u64* __restrict__ first, unsigned* __restrict__ done) {
    __shared__ unsigned h[kSortMaxPasses * kSortBins];
    __shared__ bool last;
    const int lane = threadIdx.x & 31;
    for (int i = threadIdx.x; i < kSortMaxPasses * kSortBins; i += blockDim.x) h[i] = 0u;
    __syncthreads();
    long long m = 0;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    // warp-uniform trips: every lane sees every ballot
    for (int64_t i0 = (int64_t)blockIdx.x * blockDim.x; i0 < n; i0 += 4 * stride) {
        long long k[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int64_t i = i0 + u * stride + threadIdx.x;
            k[u] = i < n ? __ldg(keys + i) : 0;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) m = k[u] > m ? k[u] : m;
        unsigned w[2][4], any[2], diff[2];  // the keys' words; bits set in one of the warp's keys, bits not alike in all
#pragma unroll
        for (int g = 0; g < 2; ++g) {
#pragma unroll
            for (int u = 0; u < 4; ++u) w[g][u] = (unsigned)((u64)k[u] >> (32 * g));
            any[g] = __reduce_or_sync(0xffffffffu, w[g][0] | w[g][1] | w[g][2] | w[g][3]);
            diff[g] = any[g] ^ __reduce_and_sync(0xffffffffu, w[g][0] & w[g][1] & w[g][2] & w[g][3]);
        }
#pragma unroll
        for (int p = 0; p < kSortMaxPasses; ++p) {
            const int g = p >> 2;
            unsigned* const hp = h + p * kSortBins;
            if ((diff[g] & (0xFFu << (8 * (p & 3)))) == 0u) {
                const unsigned d0 = (any[g] >> (8 * (p & 3))) & 0xFFu;
                if (lane == 0 && d0) atomicAdd(&hp[d0], 128u);
            } else {
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const unsigned d = __byte_perm(w[g][u], 0u, 0x4440u + (p & 3));
                    if (d) atomicAdd(&hp[d], 1u);
                }
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const long long y = __shfl_xor_sync(0xffffffffu, m, o);
        m = y > m ? y : m;
    }
    if (lane == 0 && m > 0) atomicMax(max_key, (u64)m);
    __syncthreads();
    for (int i = threadIdx.x; i < kSortMaxPasses * kSortBins; i += blockDim.x)
        if (h[i]) atomicAdd(&counts[i], (u64)h[i]);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    const int p = threadIdx.x >> 5;
    if (p >= kSortMaxPasses) return;
    u64 c[8], sum = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        c[j] = __ldcg(counts + p * kSortBins + 8 * lane + j);
        sum += c[j];
    }
    u64 all = sum;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) all += __shfl_xor_sync(0xffffffffu, all, o);
    if (lane == 0) {  // digit 0: the rest
        c[0] = (u64)n - all;
        sum += c[0];
    }
    u64 incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const u64 y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    u64 run = incl - sum;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        first[p * kSortBins + 8 * lane + j] = run;
        run += c[j];
    }
}

// One pass: the lowest 8 bits of the key are its digit; the element goes to its
// place in `out` with those bits dropped.  (in_key, out_key: of SortRec16.)
template <class In, class Out, bool kWide>
__global__ void __launch_bounds__(kSortT, kSortCtasPerSm)
    sort_pass_kernel(const void* __restrict__ in_, const u64* __restrict__ in_key, void* __restrict__ out_,
                     u64* __restrict__ out_key, int64_t n, const u64* __restrict__ first, typename SortWord<kWide>::T* words, unsigned* ticket,
                     unsigned* err) {
    typedef SortTile<Out, kWide> Tile;
    typedef typename Tile::Staged Staged;
    typedef typename SortWord<kWide>::T Word;
    constexpr bool kFromKeys = std::is_same<In, SortKeys>::value;
    constexpr bool kToPerm = std::is_same<Out, SortPerm>::value;
    // a record of at most 32 key bits is staged with its digit; otherwise the
    // digits sit in an array of their own
    constexpr bool kDigitInKey = std::is_same<In, SortRec8>::value && std::is_same<Out, SortRec8>::value;
    constexpr int kPer = Tile::kPer, kTile = kSortT * kPer;
    constexpr int kBits = 8 * (int)sizeof(Word) - 2;  // of the count
    constexpr Word kMask = ((Word)1 << kBits) - 1;
    extern __shared__ __align__(16) unsigned char sort_smem[];
    Staged* const staged = reinterpret_cast<Staged*>(sort_smem);                          // [kTile]
    unsigned char* const sdig = sort_smem + sizeof(Staged) * kTile;                       // [kTile]
    // per warp and digit: the running count, and the lanes that hold the digit now
    unsigned (*const wcount)[kSortBins] = reinterpret_cast<unsigned (*)[kSortBins]>(sdig + kTile);  // [2 * warps]
    __shared__ long long place[kSortBins];  // digit's output position minus its place in the tile
    __shared__ unsigned start[kSortBins];   // digit's place in the tile
    __shared__ unsigned wsum[kSortBins / 32];
    __shared__ unsigned sh_tile;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) sh_tile = atomicAdd(ticket, 1u);
    for (int i = lane; i < kSortBins; i += 32) wcount[warp][i] = wcount[kSortWarps + warp][i] = 0u;
    __syncthreads();
    const int64_t tile = sh_tile;
    const int64_t base = tile * kTile;
    const int cnt = (int)(n - base < kTile ? n - base : kTile);
    const int w0 = warp * 32 * kPer;  // this warp's first element of the tile
    unsigned lt;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));

    typedef typename std::conditional<std::is_same<Out, SortRec16>::value, u64, unsigned>::type KeyT;
    typedef typename std::conditional<kWide || std::is_same<Out, SortRec16>::value, u64, unsigned>::type IdxT;
    KeyT key[kPer];       // the digits still to come
    IdxT idx[kFromKeys ? 1 : kPer];  // (of a caller's key: its position)
    unsigned at[kPer];    // digit, then digit << 16 | rank among the warp's elements of that digit
#pragma unroll
    for (int r = 0; r < kPer; ++r) {
        const int e = w0 + r * 32 + lane;
        at[r] = 0x100u;  // past the end
        key[r] = 0;
        if constexpr (!kFromKeys) idx[r] = 0;
        if (e < cnt) {
            if constexpr (kFromKeys) {
                const u64 k = (u64)__ldg(static_cast<const long long*>(in_) + base + e);
                at[r] = (unsigned)k & 0xFFu;
                key[r] = (KeyT)(k >> 8);
            } else if constexpr (std::is_same<In, SortRec8>::value) {
                const uint2 k = __ldcs(static_cast<const uint2*>(in_) + base + e);
                at[r] = k.x & 0xFFu;
                key[r] = (KeyT)(kDigitInKey ? k.x : k.x >> 8);
                idx[r] = (IdxT)k.y;
            } else {
                const u64 k = __ldcs(in_key + base + e);
                at[r] = (unsigned)k & 0xFFu;
                key[r] = (KeyT)(k >> 8);
                idx[r] = (IdxT)__ldcs(static_cast<const u64*>(in_) + base + e);
            }
        }
    }
#pragma unroll
    for (int r = 0; r < kPer; ++r) {
        const unsigned d = at[r];
        const bool ok = d < 0x100u;
        // the lanes holding the same digit set their bits in the digit's word
        // (a ballot per digit bit instead: passes of 110-122 us, against 85-109)
        unsigned* const wc = &wcount[warp][d & 0xFFu];
        unsigned* const wp = wc + kSortWarps * kSortBins;
        if (ok) atomicOr(wp, 1u << lane);
        __syncwarp();
        const unsigned peers = *wp, prior = *wc, before = peers & lt;
        __syncwarp();
        if (ok && before == 0u) {
            *wc = prior + __popc(peers);
            *wp = 0u;
        }
        __syncwarp();
        at[r] = (d << 16) | (prior + __popc(before));
    }
    __syncthreads();
    // per digit: the warps' counts become offsets, the tile's count is
    // published, and a look-back gives the digit's place in the output
    const int d = threadIdx.x;
    unsigned total = 0;
    if (d < kSortBins) {
#pragma unroll
        for (int w = 0; w < kSortWarps; ++w) {
            const unsigned c = wcount[w][d];
            wcount[w][d] = total;
            total += c;
        }
        Word* const mine = words + tile * kSortBins + d;
        *(volatile Word*)mine = ((Word)(tile == 0 ? 2 : 1) << kBits) | total;
        unsigned incl = total;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) wsum[warp] = incl;
        start[d] = incl - total;
    }
    __syncthreads();
    if (d < kSortBins) {
        unsigned add = 0;
        for (int w = 0; w < warp; ++w) add += wsum[w];
        const unsigned s = start[d] + add;
        start[d] = s;
#pragma unroll
        for (int w = 0; w < kSortWarps; ++w) wcount[w][d] += s;
    }
    __syncthreads();
    // into digit order
#pragma unroll
    for (int r = 0; r < kPer; ++r) {
        const unsigned dd = at[r] >> 16;
        if (dd < 0x100u) {
            const unsigned q = wcount[warp][dd] + (at[r] & 0xFFFFu);
            IdxT ix;
            if constexpr (kFromKeys) ix = (IdxT)(base + w0 + r * 32 + lane);
            else ix = idx[r];
            if constexpr (kToPerm) staged[q] = (Staged)ix;
            else staged[q] = Staged{key[r], ix};
            if (!kDigitInKey) sdig[q] = (unsigned char)dd;
        }
    }
    if (d < kSortBins) {
        u64 prefix = 0;
        // four earlier tiles' words at a time, nearest first
        constexpr int kBack = 4;
        int64_t q = tile - 1;
        unsigned spins = 0;
        while (q >= 0) {
            Word v[kBack];
#pragma unroll
            for (int u = 0; u < kBack; ++u)
                v[u] = q - u >= 0 ? *(volatile const Word*)(words + (q - u) * kSortBins + d) : (Word)0;
            bool done = false;
            int used = 0;
#pragma unroll
            for (int u = 0; u < kBack; ++u) {
                if (!done && used == u && (v[u] >> kBits) != 0) {
                    prefix += v[u] & kMask;
                    done = (v[u] >> kBits) == 2;
                    ++used;
                }
            }
            if (done) break;
            q -= used;
            if (used == 0) {
                if (++spins > kSpinLimit) {
                    raise_error(err, ERRBIT_TIMEOUT);
                    break;
                }
            } else {
                spins = 0;
            }
        }
        if (tile > 0) *(volatile Word*)(words + tile * kSortBins + d) = ((Word)2 << kBits) | (Word)(prefix + total);
        place[d] = (long long)(__ldg(first + d) + prefix) - (long long)start[d];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < cnt; i += kSortT) {
        unsigned dd;
        if constexpr (kDigitInKey) dd = staged[i].key & 0xFFu;
        else dd = sdig[i];
        const long long pos = place[dd] + i;
        if constexpr (kToPerm) {
            static_cast<long long*>(out_)[pos] = (long long)staged[i];
        } else if constexpr (std::is_same<Out, SortRec8>::value) {
            SortRec8 rec = staged[i];
            if (kDigitInKey) rec.key >>= 8;
            *reinterpret_cast<uint2*>(static_cast<SortRec8*>(out_) + pos) = make_uint2(rec.key, rec.idx);
        } else {
            out_key[pos] = staged[i].key;
            static_cast<u64*>(out_)[pos] = staged[i].idx;
        }
    }
}

template <class Out, bool kWide>
constexpr size_t sort_pass_smem() {
    typedef SortTile<Out, kWide> Tile;
    return (sizeof(typename Tile::Staged) + 1) * (size_t)(kSortT * Tile::kPer) +
           2 * sizeof(unsigned) * kSortWarps * kSortBins;
}

template <class In, class Out, bool kWide>
static int sort_pass(const void* in, const u64* in_key, void* out, u64* out_key, int64_t n, const u64* first,
                     void* words, unsigned* ticket, Device* d, cudaStream_t s) {
    constexpr int kTile = kSortT * SortTile<Out, kWide>::kPer;
    auto k = sort_pass_kernel<In, Out, kWide>;
    HYD_TRY(configure_kernel((const void*)k, d, false));
    k<<<(unsigned)((n + kTile - 1) / kTile), kSortT, sort_pass_smem<Out, kWide>(), s>>>(
        in, in_key, out, out_key, n, first, static_cast<typename SortWord<kWide>::T*>(words), ticket, d->d_err);
    return launch_check("sort_indices pass");
}

// out[i] = src[perm[i]].  Random reads of src bound it, so every thread has
// eight of them in flight (kVec: perm read and out written as two 32-byte
// groups; the remainder, and unaligned arrays, one at a time).  2^24 int64 of
// a random permutation: 222 -> 197 us.
constexpr int kGatherT = 256;
template <class T, bool kVec>
__global__ void __launch_bounds__(kGatherT) gather_kernel(const long long* __restrict__ perm, int64_t n,
                                                          const T* __restrict__ src, int64_t src_n,
                                                          T* __restrict__ out, unsigned* err) {
    bool bad = false;
    const int64_t t = (int64_t)blockIdx.x * kGatherT + threadIdx.x, nt = (int64_t)gridDim.x * kGatherT;
    int64_t done = 0;
    if (kVec) {
        const int64_t nq = n >> 2;
        for (int64_t q = t; q < nq; q += 2 * nt) {
            const bool two = q + nt < nq;
            const u64x4 a = ldg_stream_u64x4(perm + 4 * q);
            const u64x4 b = two ? ldg_stream_u64x4(perm + 4 * (q + nt)) : a;
            const u64 p[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
            T v[8];
            bool ok = true;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const bool in = p[k] < (u64)src_n;
                ok &= in;
                v[k] = in ? __ldcg(src + p[k]) : T(0);
            }
            bad |= !ok;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (h == 1 && !two) break;
                T* const o = out + 4 * (q + h * nt);
                if (ok) {
                    if (sizeof(T) == 8) {
                        asm volatile("st.global.v4.u64 [%0], {%1,%2,%3,%4};" ::"l"(o), "l"(to_bits(v[4 * h])),
                                     "l"(to_bits(v[4 * h + 1])), "l"(to_bits(v[4 * h + 2])),
                                     "l"(to_bits(v[4 * h + 3]))
                                     : "memory");
                    } else {
                        *reinterpret_cast<int4*>(o) = make_int4((int)v[4 * h], (int)v[4 * h + 1], (int)v[4 * h + 2],
                                                                (int)v[4 * h + 3]);
                    }
                } else {
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        if (p[4 * h + k] < (u64)src_n) o[k] = v[4 * h + k];
                }
            }
        }
        done = nq * 4;
    }
    for (int64_t i = done + t; i < n; i += nt) {
        const long long p = perm[i];
        if ((u64)p < (u64)src_n) out[i] = __ldcg(src + p);
        else bad = true;
    }
    if (bad) raise_error(err, ERRBIT_BOUNDS);
}

// Digit counts, first positions, pass tickets: the fixed part of the scratch.
struct SortTables {
    u64 max_key;
    unsigned done, pad;
    unsigned ticket[kSortMaxPasses];
    u64 counts[kSortMaxPasses * kSortBins];
    u64 first[kSortMaxPasses * kSortBins];
};

// The sort; passes == 0: as many as the largest key needs (one 8-byte read-back).
static int sort_indices_launch(const long long* keys, int64_t n, int passes, long long* perm, cudaStream_t s) {
    Device* d = nullptr;
    HYD_TRY(device(&d));
    auto al = [](size_t b) { return (b + 255) & ~(size_t)255; };
    const bool wide = n >= (1LL << 30);
    constexpr int kTile = kSortT * 8;  // the smaller tile
    const int64_t ntiles = (n + kTile - 1) / kTile;
    HYD_CHECK_ARG(ntiles <= INT_MAX, "sort_indices: too long");
    const size_t word_bytes = al((size_t)ntiles * kSortBins * (wide ? 8 : 4));  // of one pass, at most
    const size_t arr_bytes = al((size_t)n * 8);
    // the records ping-pong between one array here and `perm` itself; the
    // 64-bit keys, while more than 32 bits of key remain, between two more
    auto scratch_bytes = [&](int np) {
        const int arrays = np <= 1 ? 0 : !wide && np <= 5 ? 1 : np == 2 || (!wide && np == 6) ? 2 : 3;
        return al(sizeof(SortTables)) + (wide ? 1 : np) * word_bytes + arrays * arr_bytes;
    };
    void* scratch = nullptr;
    HYD_TRY(workspace(s, passes ? scratch_bytes(passes) : al(sizeof(SortTables)), nullptr, &scratch));
    SortTables* t = static_cast<SortTables*>(scratch);
    HYD_CUDA_TRY(cudaMemsetAsync(t, 0, offsetof(SortTables, first), s));
    int64_t blocks = (n + 4095) / 4096;
    if (blocks > d->sm_count * 2) blocks = d->sm_count * 2;
    sort_count_kernel<<<(unsigned)blocks, 1024, 0, s>>>(keys, n, &t->max_key, t->counts, t->first, &t->done);
    HYD_TRY(launch_check("sort_indices counts"));
    if (passes == 0) {
        u64 mk = 0;
        HYD_CUDA_TRY(cudaMemcpyAsync(&mk, &t->max_key, 8, cudaMemcpyDeviceToHost, s));
        HYD_CUDA_TRY(cudaStreamSynchronize(s));
        for (u64 m = mk; m; m >>= 8) ++passes;
        if (passes == 0) passes = 1;
        bool grew = false;
        HYD_TRY(workspace(s, scratch_bytes(passes), nullptr, &scratch, &grew));
        if (grew) {  // the tables went with the old block: count once more
            t = static_cast<SortTables*>(scratch);
            HYD_CUDA_TRY(cudaMemsetAsync(t, 0, offsetof(SortTables, first), s));
            sort_count_kernel<<<(unsigned)blocks, 1024, 0, s>>>(keys, n, &t->max_key, t->counts, t->first, &t->done);
            HYD_TRY(launch_check("sort_indices counts"));
        }
    }
    unsigned char* b = reinterpret_cast<unsigned char*>(t) + al(sizeof(SortTables));
    unsigned char* const words = b;
    b += (wide ? 1 : passes) * word_bytes;
    void* const rec = b;
    u64* const kbuf[2] = {reinterpret_cast<u64*>(b + arr_bytes), reinterpret_cast<u64*>(b + 2 * arr_bytes)};
    if (!wide) HYD_CUDA_TRY(cudaMemsetAsync(words, 0, passes * word_bytes, s));
    enum { kKeys, k8, k16 };
    int have = kKeys;
    const void* in = keys;
    for (int p = 0; p < passes; ++p) {
        const u64* first = t->first + p * kSortBins;
        void* w = words + (wide ? 0 : p) * word_bytes;
        if (wide) HYD_CUDA_TRY(cudaMemsetAsync(w, 0, word_bytes, s));
        unsigned* ticket = &t->ticket[p];
        const int left = 8 * (passes - 1 - p);  // key bits after this pass
        void* out = (passes - 1 - p) & 1 ? rec : static_cast<void*>(perm);
        const u64* ik = kbuf[(p & 1) ^ 1];
        u64* ok = kbuf[p & 1];
        const int next = wide || left > 32 ? k16 : k8;
        auto run = [&](auto pass) { return pass(in, ik, out, ok, n, first, w, ticket, d, s); };
        int st;
        if (wide) {
            if (left == 0) st = have == kKeys ? run(sort_pass<SortKeys, SortPerm, true>)
                                              : run(sort_pass<SortRec16, SortPerm, true>);
            else st = have == kKeys ? run(sort_pass<SortKeys, SortRec16, true>)
                                    : run(sort_pass<SortRec16, SortRec16, true>);
        } else if (left == 0) {
            st = have == kKeys ? run(sort_pass<SortKeys, SortPerm, false>) : run(sort_pass<SortRec8, SortPerm, false>);
        } else if (next == k8) {
            st = have == kKeys ? run(sort_pass<SortKeys, SortRec8, false>)
                 : have == k8  ? run(sort_pass<SortRec8, SortRec8, false>)
                               : run(sort_pass<SortRec16, SortRec8, false>);
        } else {
            st = have == kKeys ? run(sort_pass<SortKeys, SortRec16, false>)
                               : run(sort_pass<SortRec16, SortRec16, false>);
        }
        HYD_TRY(st);
        have = next;
        in = out;
    }
    return HYD_CUDA_OK;
}

}  // namespace hyd

using namespace hyd;

extern "C" int hyd_cuda_sort_indices_i64(const int64_t* keys, int64_t n, int64_t* perm, void* stream) {
    HYD_CHECK_ARG(n >= 0, "sort_indices: negative length");
    HYD_CHECK_ARG(n == 0 || (keys != nullptr && perm != nullptr), "sort_indices: null buffer");
    HYD_CHECK_ARG(n < (1LL << 40), "sort_indices: too long");
    if (n == 0) return HYD_CUDA_OK;
    return sort_indices_launch(reinterpret_cast<const long long*>(keys), n, 0, reinterpret_cast<long long*>(perm),
                               as_stream(stream));
}

extern "C" int hyd_cuda_sort_indices_bits_i64(const int64_t* keys, int64_t n, int key_bits, int64_t* perm,
                                              void* stream) {
    HYD_CHECK_ARG(n >= 0, "sort_indices_bits: negative length");
    HYD_CHECK_ARG(key_bits >= 0 && key_bits <= 64, "sort_indices_bits: key_bits in [0, 64]");
    HYD_CHECK_ARG(n == 0 || (keys != nullptr && perm != nullptr), "sort_indices_bits: null buffer");
    if (n == 0) return HYD_CUDA_OK;
    int passes = (key_bits + 7) / 8;
    if (passes == 0) passes = 1;
    return sort_indices_launch(reinterpret_cast<const long long*>(keys), n, passes,
                               reinterpret_cast<long long*>(perm), as_stream(stream));
}

template <class T>
static int gather_launch(const int64_t* perm, int64_t n, const T* src, int64_t src_n, T* out, void* stream) {
    HYD_CHECK_ARG(n >= 0 && src_n >= 0, "gather: negative length");
    HYD_CHECK_ARG(n == 0 || (perm && src && out), "gather: null buffer");
    if (n == 0) return HYD_CUDA_OK;
    Device* d = nullptr;
    HYD_TRY(device(&d));
    const bool vec = (reinterpret_cast<uintptr_t>(perm) & 31) == 0 &&
                     (reinterpret_cast<uintptr_t>(out) & (4 * sizeof(T) - 1)) == 0;
    // small arrays: one element per thread, so that every SM has work
    const bool wide = vec && n >= (int64_t)d->sm_count * kGatherT * 8;
    const int per = wide ? 8 : 1;
    int64_t blocks = (n + kGatherT * per - 1) / (kGatherT * per);
    if (blocks > d->sm_count * 8) blocks = d->sm_count * 8;
    auto k = wide ? gather_kernel<T, true> : gather_kernel<T, false>;
    k<<<(unsigned)blocks, kGatherT, 0, as_stream(stream)>>>(reinterpret_cast<const long long*>(perm), n, src, src_n,
                                                            out, d->d_err);
    return launch_check("gather");
}

extern "C" int hyd_cuda_gather_i64(const int64_t* perm, int64_t n, const int64_t* src, int64_t src_n, int64_t* out,
                                   void* stream) {
    return gather_launch<long long>(perm, n, reinterpret_cast<const long long*>(src), src_n,
                                    reinterpret_cast<long long*>(out), stream);
}

extern "C" int hyd_cuda_gather_f64(const int64_t* perm, int64_t n, const double* src, int64_t src_n, double* out,
                                   void* stream) {
    return gather_launch<double>(perm, n, src, src_n, out, stream);
}

extern "C" int hyd_cuda_gather_i32(const int64_t* perm, int64_t n, const int32_t* src, int64_t src_n, int32_t* out,
                                   void* stream) {
    return gather_launch<int>(perm, n, reinterpret_cast<const int*>(src), src_n, reinterpret_cast<int*>(out), stream);
}
