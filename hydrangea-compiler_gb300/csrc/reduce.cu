// reduce.cu -- deterministic fp64 reductions: the fused
// `reduce (+) 0.0 (zipwith (*) xs ys)` (dot) and `reduce (+) 0.0 xs` (sum).
//
// Replaces the parallel reduction template of the reference C backend
// (CodegenC.hs:1328-1353; emitted `omp parallel for simd reduction(+:acc)`,
// README.md:25-33) for the 1-D reduce_generate of Lowering.hs:771-804.
//
// Design (HBM-bound streaming reduction, one launch; dot of 2^24 elements 48.9 ->
// 46.4 us, of 10^6 14.0 -> 12.3 us since the combining steps take a quarter of
// the FP64 instructions):
//  * a fixed grid of 2 blocks x 512 threads per SM; thread t owns the 32-byte
//    vectors t, t+S, t+2S, ... (S = total threads) in two chains of
//    multiply-adds, with four 256-bit loads in flight per thread (eight
//    accumulators round no better: 3e5 elements in [-1, 1) 0.0048 units of 2^-53
//    of sum |xy| with them, 0.0041 so, root mean square);
//  * per-thread order, the halving through shared memory, the last warp's tree
//    and the final combine are all fixed, so a given (n, device) always produces the
//    same bits (the C backend's result instead depends on the thread count);
//  * the block partials go to per-stream scratch; the last block to finish
//    (completion counter) sums them in index order and resets the counter,
//    so no second launch and no memset are needed per call.
// Products are accumulated with fma (one rounding per element instead of the
// C backend's two); the tolerance against the C backend is relative 1e-12.
#include "hyd_common.cuh"

namespace hyd {

constexpr int kRedThreads = 512;
constexpr int kRedBlocksPerSM = 2;

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Fixed-order block reduction; result valid in thread 0.  The sums are halved
// through shared memory down to one warp: 20 FP64 instructions per block of 512
// threads, where a shuffle tree in every warp takes 85, each holding the SM's
// FP64 pipe for 19 cycles.
template <int T>
__device__ __forceinline__ double block_sum(double v, double* sh /*[T]*/) {
    const int t = threadIdx.x;
    sh[t] = v;
#pragma unroll
    for (int half = T / 2; half >= 32; half >>= 1) {
        __syncthreads();
        if (t < half) {
            v += sh[t + half];
            sh[t] = v;
        }
    }
    return t < 32 ? warp_sum(v) : 0.0;
}

// Last-block combine of the per-block partials, in index order.
__device__ __forceinline__ void finish_partials(double bsum, double* partials, unsigned* counter,
                                                double* out, double* sh) {
    __shared__ bool is_last;
    if (threadIdx.x == 0) {
        partials[blockIdx.x] = bsum;
        __threadfence();
        unsigned ticket = atomicAdd(counter, 1u);
        is_last = (ticket == gridDim.x - 1);
    }
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    double v = 0.0;
    for (unsigned i = threadIdx.x; i < gridDim.x; i += blockDim.x)
        v += *((volatile double*)&partials[i]);
    double total = block_sum<kRedThreads>(v, sh);
    if (threadIdx.x == 0) {
        *out = total;
        *counter = 0u;  // leave the counter ready for the next launch
    }
}

template <bool kDot, bool kVec>
__global__ void __launch_bounds__(kRedThreads, kRedBlocksPerSM)
    reduce_f64_kernel(const double* __restrict__ xs, const double* __restrict__ ys, int64_t n,
                      double* partials, unsigned* counter, double* out) {
    __shared__ double sh[kRedThreads];
    const int64_t S = (int64_t)gridDim.x * blockDim.x;
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    double a = 0.0, b = 0.0;  // 32 warps per SM hide the chains' latency
    if (kVec) {
        const int64_t nv = n >> 2;  // 32-byte vectors
        // the up to three elements after them: on their way from the start
        const bool tail = 4 * nv + t < n;
        const double tx = tail ? xs[4 * nv + t] : 0.0, ty = kDot && tail ? ys[4 * nv + t] : 0.0;
        int64_t v = t;
        for (; v + S < nv; v += 2 * S) {
            const f64x4 x0 = ldg_stream_f64x4(xs + 4 * v);
            const f64x4 x1 = ldg_stream_f64x4(xs + 4 * (v + S));
            if (kDot) {
                const f64x4 y0 = ldg_stream_f64x4(ys + 4 * v);
                const f64x4 y1 = ldg_stream_f64x4(ys + 4 * (v + S));
                a = fma(x0.x, y0.x, a); b = fma(x1.x, y1.x, b);
                a = fma(x0.y, y0.y, a); b = fma(x1.y, y1.y, b);
                a = fma(x0.z, y0.z, a); b = fma(x1.z, y1.z, b);
                a = fma(x0.w, y0.w, a); b = fma(x1.w, y1.w, b);
            } else {
                a += x0.x; b += x1.x;
                a += x0.y; b += x1.y;
                a += x0.z; b += x1.z;
                a += x0.w; b += x1.w;
            }
        }
        if (v < nv) {
            const f64x4 x0 = ldg_stream_f64x4(xs + 4 * v);
            if (kDot) {
                const f64x4 y0 = ldg_stream_f64x4(ys + 4 * v);
                a = fma(x0.x, y0.x, a);
                a = fma(x0.y, y0.y, a);
                a = fma(x0.z, y0.z, a);
                a = fma(x0.w, y0.w, a);
            } else {
                a += x0.x;
                a += x0.y;
                a += x0.z;
                a += x0.w;
            }
        }
        if (tail) a = kDot ? fma(tx, ty, a) : a + tx;
    } else {  // pointers that are not 32-byte aligned
        for (int64_t i = t; i < n; i += S) a = kDot ? fma(xs[i], ys[i], a) : a + xs[i];
    }
    const double v = a + b;
    double bsum = block_sum<kRedThreads>(v, sh);
    __syncthreads();
    finish_partials(bsum, partials, counter, out, sh);
}

// Short arrays, by one block: no partials through memory and no completion
// counter.  What counts here is the FP64 pipe of the one SM (a warp instruction
// holds it for 19 cycles), so there are few warps, with all their loads in flight,
// and each thread adds 16 elements in one chain before it adds the chain to the
// ones before: with one chain for all, 16000 elements in [-1, 1) came out with an
// error of 0.029 units of 2^-53 of sum |xy| (root mean square), so with 0.019, as
// in the form for long arrays (0.019).  Per call: 4099 elements 8.2 -> 4.1 us (four
// accumulators all along: 5.8), 8192 9.4 -> 6.1, 16384 9.7 -> 8.2 (512 or 1024
// threads with eight accumulators each and a tree in every warp: 8.2 at 4099).
constexpr int kRedOneThreads = 256;
constexpr int64_t kRedOneBlock = 16384;
template <bool kDot, bool kVec>
__global__ void __launch_bounds__(kRedOneThreads) reduce_one_kernel(const double* __restrict__ xs,
                                                                    const double* __restrict__ ys, int n,
                                                                    double* out) {
    __shared__ double sh[kRedOneThreads];
    constexpr int T = kRedOneThreads, kIn = 4;
    const int t = threadIdx.x;
    double acc = 0.0;
    if (kVec) {
        const int nv = n >> 2;
        const bool tail = 4 * nv + t < n;
        const double tx = tail ? xs[4 * nv + t] : 0.0, ty = kDot && tail ? ys[4 * nv + t] : 0.0;
        auto chain = [&](int v) {
            f64x4 x[kIn], y[kIn];
#pragma unroll
            for (int u = 0; u < kIn; ++u)
                if (v + u * T < nv) {
                    x[u] = ldg_stream_f64x4(xs + 4 * (v + u * T));
                    if (kDot) y[u] = ldg_stream_f64x4(ys + 4 * (v + u * T));
                }
            double c = 0.0;
#pragma unroll
            for (int u = 0; u < kIn; ++u)
                if (v + u * T < nv) {
                    c = kDot ? fma(x[u].x, y[u].x, c) : c + x[u].x;
                    c = kDot ? fma(x[u].y, y[u].y, c) : c + x[u].y;
                    c = kDot ? fma(x[u].z, y[u].z, c) : c + x[u].z;
                    c = kDot ? fma(x[u].w, y[u].w, c) : c + x[u].w;
                }
            return c;
        };
        if (t < nv) acc = chain(t);
        for (int v = t + kIn * T; v < nv; v += kIn * T) acc += chain(v);
        if (tail) acc = kDot ? fma(tx, ty, acc) : acc + tx;
    } else {
        for (int i0 = t; i0 < n; i0 += 4 * kIn * T) {
            double c = 0.0;
#pragma unroll
            for (int u = 0; u < 4 * kIn; ++u) {
                const int i = i0 + u * T;
                if (i < n) c = kDot ? fma(__ldg(xs + i), __ldg(ys + i), c) : c + __ldg(xs + i);
            }
            acc += c;
        }
    }
    acc = block_sum<T>(acc, sh);
    if (t == 0) *out = acc;
}

// Blocks for n elements on `sms` SMs: two vectors per thread until every SM has
// two blocks.
static int64_t reduce_blocks(int64_t n, int sms) {
    const int64_t want = ((n + 3) / 4 + 2LL * kRedThreads - 1) / (2LL * kRedThreads);
    const int64_t most = (int64_t)sms * kRedBlocksPerSM;
    return want < most ? want : most;
}
static void reduce_one(bool dot, bool vec, const double* xs, const double* ys, int64_t n, double* out,
                       cudaStream_t s) {
    auto k = dot ? (vec ? reduce_one_kernel<true, true> : reduce_one_kernel<true, false>)
                 : (vec ? reduce_one_kernel<false, true> : reduce_one_kernel<false, false>);
    k<<<1, kRedOneThreads, 0, s>>>(xs, ys, (int)n, out);
}

static int reduce_launch(bool dot, const double* xs, const double* ys, int64_t n, double* out,
                         cudaStream_t stream) {
    const bool vec = ((reinterpret_cast<uintptr_t>(xs) | (dot ? reinterpret_cast<uintptr_t>(ys) : 0)) & 31) == 0;
    Device* d = nullptr;
    HYD_TRY(device(&d));
    if (n <= kRedOneBlock) {
        reduce_one(dot, vec, xs, dot ? ys : xs, n, out, stream);
        return launch_check(dot ? "dot_f64" : "sum_f64");
    }
    const int64_t blocks = reduce_blocks(n, d->sm_count);
    unsigned* counters = nullptr;
    void* scratch = nullptr;
    HYD_TRY(workspace(stream, sizeof(double) * (size_t)blocks, &counters, &scratch));
    double* partials = static_cast<double*>(scratch);
    unsigned* counter = counters + (dot ? 0 : 1);
    dim3 grid((unsigned)blocks), block(kRedThreads);
    if (dot) {
        if (vec) reduce_f64_kernel<true, true><<<grid, block, 0, stream>>>(xs, ys, n, partials, counter, out);
        else reduce_f64_kernel<true, false><<<grid, block, 0, stream>>>(xs, ys, n, partials, counter, out);
    } else {
        if (vec) reduce_f64_kernel<false, true><<<grid, block, 0, stream>>>(xs, xs, n, partials, counter, out);
        else reduce_f64_kernel<false, false><<<grid, block, 0, stream>>>(xs, xs, n, partials, counter, out);
    }
    return launch_check(dot ? "dot_f64" : "sum_f64");
}

}  // namespace hyd

using namespace hyd;

extern "C" int hyd_cuda_dot_f64(const double* xs, const double* ys, int64_t n, double* out,
                                void* stream) {
    HYD_CHECK_ARG(n >= 0, "dot_f64: negative length %lld", (long long)n);
    HYD_CHECK_ARG(out != nullptr, "dot_f64: null output");
    HYD_CHECK_ARG(n == 0 || (xs != nullptr && ys != nullptr), "dot_f64: null input");
    return reduce_launch(true, xs, ys, n, out, as_stream(stream));
}

extern "C" int hyd_cuda_sum_f64(const double* xs, int64_t n, double* out, void* stream) {
    HYD_CHECK_ARG(n >= 0, "sum_f64: negative length %lld", (long long)n);
    HYD_CHECK_ARG(out != nullptr, "sum_f64: null output");
    HYD_CHECK_ARG(n == 0 || xs != nullptr, "sum_f64: null input");
    return reduce_launch(false, xs, nullptr, n, out, as_stream(stream));
}

// ---------------------------------------------------------------------------
// Allocation-free dot product.
//
// Some callers cannot allocate device memory at the point where they need a
// reduction: a latency-critical serving or real-time loop where cudaMalloc
// (and the cudaFree that pairs with it) may synchronize the device and stall
// work on other streams; a process whose device memory was reserved up front
// by another allocator or capped by a memory policy, where a fresh cudaMalloc
// can fail at an arbitrary moment; an embedding host that requires a fixed
// footprint after start-up.  hyd_cuda_dot_f64 takes its scratch (per-CTA
// partials and a completion counter) from a per-stream workspace that the
// runtime allocates on first use, so it is not usable there.
//
// hyd_cuda_dot_f64_noalloc runs the same kernel with its scratch in the
// file-scope array below instead.  The array is fixed at load time, so every
// GPU that loads this library holds these bytes until the process exits.  Its
// size bounds the launch: kNoAllocMaxBlocks CTAs (two per SM on any GPU with
// up to 1024 SMs); a launch that would need more is rejected.
namespace hyd {

constexpr int kNoAllocMaxBlocks = 2048;
constexpr size_t kNoAllocCounterBytes = 256;
constexpr size_t kNoAllocScratchBytes = kNoAllocCounterBytes + sizeof(double) * kNoAllocMaxBlocks;

static __device__ __align__(256) unsigned char g_dot_noalloc_scratch[kNoAllocScratchBytes];

// Device address of g_dot_noalloc_scratch, looked up once per device with that
// device current.  In host code the symbol itself is only a host-side stand-in,
// never a device address, so kernels must be given this pointer.
static std::mutex g_noalloc_mu;
static unsigned char* g_noalloc_ptr[64] = {nullptr};
static int g_noalloc_sms[64] = {0};

static int noalloc_setup(int dev, unsigned char** scratch, int* sms) {
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if (g_noalloc_ptr[dev] == nullptr) {
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_dot_noalloc_scratch);
        if (e != cudaSuccess)
            return set_error(HYD_CUDA_ERR_CUDA, "dot_f64_noalloc: cudaGetSymbolAddress failed: %s",
                             cudaGetErrorString(e));
        int n = 0;
        e = cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess)
            return set_error(HYD_CUDA_ERR_CUDA, "dot_f64_noalloc: SM count query failed: %s",
                             cudaGetErrorString(e));
        g_noalloc_sms[dev] = n;
        g_noalloc_ptr[dev] = static_cast<unsigned char*>(p);
    }
    *scratch = g_noalloc_ptr[dev];
    *sms = g_noalloc_sms[dev];
    return HYD_CUDA_OK;
}

}  // namespace hyd

extern "C" int hyd_cuda_dot_f64_noalloc(const double* xs, const double* ys, int64_t n, double* out,
                                        void* stream) {
    HYD_CHECK_ARG(n >= 0, "dot_f64_noalloc: negative length %lld", (long long)n);
    HYD_CHECK_ARG(out != nullptr, "dot_f64_noalloc: null output");
    HYD_CHECK_ARG(n == 0 || (xs != nullptr && ys != nullptr), "dot_f64_noalloc: null input");
    int dev = 0;
    HYD_CUDA_TRY(cudaGetDevice(&dev));
    HYD_CHECK_ARG(dev >= 0 && dev < 64, "dot_f64_noalloc: device ordinal %d beyond 63", dev);
    unsigned char* scratch = nullptr;
    int sms = 0;
    HYD_TRY(noalloc_setup(dev, &scratch, &sms));
    // Same kernels and grid rule as hyd_cuda_dot_f64, so both give the same bits.
    const bool vec = ((reinterpret_cast<uintptr_t>(xs) | reinterpret_cast<uintptr_t>(ys)) & 31) == 0;
    if (n <= kRedOneBlock) {
        reduce_one(true, vec, xs, ys, n, out, as_stream(stream));
        return launch_check("dot_f64_noalloc");
    }
    const int64_t blocks = reduce_blocks(n, sms);
    if (blocks > kNoAllocMaxBlocks)
        return set_error(HYD_CUDA_ERR_UNSUPPORTED,
                         "dot_f64_noalloc: needs %lld CTAs of scratch but the static scratch holds %d",
                         (long long)blocks, kNoAllocMaxBlocks);
    unsigned* counter = reinterpret_cast<unsigned*>(scratch);
    double* partials = reinterpret_cast<double*>(scratch + kNoAllocCounterBytes);
    cudaStream_t st = as_stream(stream);
    // The array keeps whatever the previous call left; the counter must start at 0.
    HYD_CUDA_TRY(cudaMemsetAsync(counter, 0, sizeof(unsigned), st));
    if (vec)
        reduce_f64_kernel<true, true><<<(unsigned)blocks, kRedThreads, 0, st>>>(xs, ys, n, partials, counter, out);
    else
        reduce_f64_kernel<true, false><<<(unsigned)blocks, kRedThreads, 0, st>>>(xs, ys, n, partials, counter, out);
    return launch_check("dot_f64_noalloc");
}
