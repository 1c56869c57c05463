// Device helpers shared by the audio kernels.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <utility>

namespace rppb {

void count_launch(int kernels);
void check_cuda(cudaError_t err, const char* what);

// ---------------------------------------------------------------- checked build
// Every global load and store of the kernels names its address through RPPB_RD / RPPB_WR.  In the
// library these expand to the address itself.  Built with -DRPPB_CHECKED (librppb_checked.so,
// `python -m rpp_b200.build --checked`), each access is first compared with the device regions the
// current call may touch (check.cu): the caller's tensors as their descriptors describe them, the
// per-sample tensors, the workspace and the handle's tables.  An access outside them is recorded
// (site, address, size; the first one of the call) and redirected to a dummy buffer, so it neither
// reads nor writes out of bounds, and the call returns a status code for it.
constexpr unsigned check_file_hash(const char* path)
{
    const char* base = path;
    for (const char* q = path; *q; ++q)
        if (*q == '/') base = q + 1;
    unsigned h = 2166136261u;   // FNV-1a of the file's base name
    for (; *base; ++base) h = (h ^ static_cast<unsigned char>(*base)) * 16777619u;
    return h & 0xffffu;
}
template <unsigned kV>
struct CheckConst
{
    static constexpr unsigned value = kV;
};
#define RPPB_SITE ((::rppb::CheckConst<::rppb::check_file_hash(__FILE__)>::value << 16) | (__LINE__ & 0xffff))
#ifdef RPPB_CHECKED
__device__ void* check_addr(const void* p, unsigned bytes, bool write, unsigned site);
template <class T>
__device__ __forceinline__ T* check_ptr(T* p, bool write, unsigned site)
{
    return static_cast<T*>(check_addr(p, unsigned(sizeof(T)), write, site));
}
// a range of `bytes` (bulk copies, prefetches): true when it lies inside one region
__device__ bool check_range(const void* p, unsigned long long bytes, bool write, unsigned site);
#define RPPB_RD(p) ::rppb::check_ptr((p), false, RPPB_SITE)
#define RPPB_WR(p) ::rppb::check_ptr((p), true, RPPB_SITE)
#define RPPB_RANGE_OK(p, bytes) ::rppb::check_range((p), (bytes), false, RPPB_SITE)
#else
#define RPPB_RD(p) (p)
#define RPPB_WR(p) (p)
#define RPPB_RANGE_OK(p, bytes) true
#endif

// A function kept out of line so that its registers do not come on top of its caller's.  Inlined in the checked
// build: relocatable code gives a function of its own more registers than a capped kernel may call.
#ifdef RPPB_CHECKED
#define RPPB_OUT_OF_LINE __forceinline__
#else
#define RPPB_OUT_OF_LINE __noinline__
#endif

// ---------------------------------------------------------------- ragged batches
// A batch of uneven samples is addressed as one flat list of work units (chunks, frame tiles,
// reset blocks ...).  prefix[b] is the number of units of samples 0..b-1 (prefix[n] = total),
// computed on the device from the per-sample tensors, so no call reads lengths on the host.

// Largest b in [0, n) with prefix[b] <= w (w < prefix[n]); empty samples are skipped.
// `prefix` may point to global or shared memory (see cache_prefix).
__device__ __forceinline__ int ragged_find(const long long* prefix, int n, long long w)
{
    int lo = 0, hi = n - 1;
    while (lo < hi)
    {
        int mid = (lo + hi + 1) >> 1;
        if (*RPPB_RD(prefix + mid) <= w) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Shared-memory copy of prefix[0..n] when it fits (batches up to kPrefixCache - 1 samples), so the
// per-unit binary search costs shared-memory rather than global-memory latency.  All threads of
// the CTA must call it; it ends with __syncthreads.
constexpr int kPrefixCache = 512;
template <int CAP = kPrefixCache>
__device__ __forceinline__ const long long* cache_prefix(const long long* prefix, int n, long long* s_cache)
{
    if (n + 1 > CAP)
    {
        __syncthreads();
        return prefix;
    }
    for (int i = threadIdx.x; i <= n; i += blockDim.x) s_cache[i] = *RPPB_RD(prefix + i);
    __syncthreads();
    return s_cache;
}

// Exclusive scan of one value per thread of a CTA of whole warps: warp scans of the values and of the warps' totals
// (each warp its own copy), one barrier.  s_total is shared; before it is used again all threads must have returned.
__device__ __forceinline__ long long block_exclusive_scan(long long value, long long (&s_total)[32])
{
    const int t = threadIdx.x, lane = t & 31;
    auto scan = [&](long long v) {
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
            const long long u = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += u;
        }
        return v;
    };
    const long long incl = scan(value);
    if (lane == 31) s_total[t >> 5] = incl;
    __syncthreads();
    const long long before = scan(lane < (t >> 5) ? s_total[lane] : 0);
    return __shfl_sync(0xffffffffu, before, 31) + incl - value;
}

// One CTA of up to 1024 threads, a clip each (or several): prefix[0..n] = exclusive scan of count(b), and
// zero[0..zeroWords) = 0 (the work counters of the kernel that follows).  It lets a kernel launched after it with
// programmatic stream serialization (launch_dependent) start at once; that kernel runs its
// independent setup, then grid_dependency_wait() before it reads what this kernel writes.
// Latency is all it costs: warp scans and one barrier instead of a 1024-wide scan of ten steps in shared memory, and
// no more threads than clips, took 1.8 us of 12.6 off a spectrogram call of 8 clips.
template <class Count>
__global__ void __launch_bounds__(1024) ragged_prefix_kernel(Count count, int n, long long* __restrict__ prefix,
                                                             unsigned* __restrict__ zero, int zeroWords)
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int t = threadIdx.x, threads = blockDim.x;
    const int per = (n + threads - 1) / threads;
    const int b0 = min(n, t * per), b1 = min(n, b0 + per);
    const long long first = b0 < b1 ? count(b0) : 0;
    for (int i = t; i < zeroWords; i += threads) *RPPB_WR(zero + i) = 0u;
    long long sum = first;
    for (int b = b0 + 1; b < b1; ++b) sum += count(b);
    __shared__ long long s_total[32];
    long long run = block_exclusive_scan(sum, s_total);
    for (int b = b0; b < b1; ++b)
    {
        *RPPB_WR(prefix + b) = run;
        run += b == b0 ? first : count(b);
    }
    if (t == threads - 1) *RPPB_WR(prefix + n) = run;
}

inline int ragged_prefix_threads(int n) { return std::min(1024, std::max(1, (n + 31) / 32) * 32); }

template <class Count>
inline void launch_ragged_prefix(Count count, int n, long long* prefix, cudaStream_t s, unsigned* zero = nullptr,
                                 int zeroWords = 0)
{
    ragged_prefix_kernel<Count><<<1, ragged_prefix_threads(n), 0, s>>>(count, n, prefix, zero, zeroWords);
    count_launch(1);
}

// In a kernel launched by launch_dependent: waits until the kernel before it in the stream has
// completed and its writes are visible (a no-op for a kernel launched the ordinary way).
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// The pointer to something that the kernel waited for has written, to be taken after grid_dependency_wait():
// through a const __restrict__ parameter the compiler may load before the wait (it takes the memory for
// constant), through the returned pointer it cannot.  The address passes as a global one, so that accesses
// through the result stay global, not generic.
template <class T>
__device__ __forceinline__ T* dependency_result(T* p)
{
    size_t g = __cvta_generic_to_global(p);
    asm volatile("" : "+l"(g)::"memory");
    return static_cast<T*>(const_cast<void*>(static_cast<const void*>(__cvta_global_to_generic(g))));
}

// Launches `kernel` with programmatic stream serialization: it may start while the kernel before
// it (which must allow it, as ragged_prefix_kernel does) is still running, so its setup overlaps
// that kernel and the launch gap; it must call grid_dependency_wait() before touching that
// kernel's results.  Kernels earlier in the stream have completed by then.
template <class... KArgs, class... Args>
inline void launch_dependent(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                             const char* what, Args&&... args)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    check_cuda(cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...), what);
}

// ---------------------------------------------------------------- float helpers
// Monotone map of float to uint32 so that atomicMax on the key is a float max (NaN excluded).
// Asks L2 to fetch the bytes of [begin, end) (rounded inward to 16-byte boundaries; nothing when
// that leaves no whole 16-byte block).  A hint: no completion to wait for.
__device__ __forceinline__ void l2_prefetch(const float* begin, const float* end)
{
    const uintptr_t b = (reinterpret_cast<uintptr_t>(begin) + 15) & ~uintptr_t(15);
    const uintptr_t e = reinterpret_cast<uintptr_t>(end) & ~uintptr_t(15);
    if (e <= b) return;
    const uintptr_t n = e - b;
    const uint32_t bytes = n < (uintptr_t(1) << 20) ? uint32_t(n) : (1u << 20);
    if (!RPPB_RANGE_OK(reinterpret_cast<const void*>(b), bytes)) return;
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(b), "r"(bytes) : "memory");
}

// Asynchronous copies of 16 or 4 aligned bytes from global to shared memory (cp.async; the issuing thread waits for
// its own with copy_async_wait).  The caller passes its source through RPPB_RD.
__device__ __forceinline__ void copy_async16(float* to, const float4* from)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(uint32_t(__cvta_generic_to_shared(to))),
                 "l"(from)
                 : "memory");
}
__device__ __forceinline__ void copy_async4(float* to, const float* from)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(uint32_t(__cvta_generic_to_shared(to))),
                 "l"(from)
                 : "memory");
}
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__device__ __forceinline__ unsigned float_key(float f)
{
    unsigned u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float key_float(unsigned k)
{
    unsigned u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
    return __uint_as_float(u);
}

// multiplier * log2(max(minRatio, x * inv)) with the hardware base-2 logarithm.  kNormal: minRatio is a normal
// number, so the argument is one too and the logarithm needs no scaling of subnormal arguments (same bits,
// four instructions less).
template <bool kNormal>
__device__ __forceinline__ float decibel(float x, float inv, float minRatio, float multiplier)
{
    float t = __fmul_rn(x, inv);
    t = minRatio < t ? t : minRatio;
    float l;
    if constexpr (kNormal) asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(l) : "f"(t));
    else l = __log2f(t);
    return __fmul_rn(multiplier, l);
}
constexpr float kMinNormal = 1.17549435e-38f;

__device__ __forceinline__ float warp_max(float v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Reflect an out-of-range index into [minLoc, maxLoc) the way the reference does
// (src/modules/tensor/cpu/kernel/spectrogram.cpp:55-69): mirror without repeating the edge,
// repeatedly for short signals; a signal shorter than 2 maps everything to its last sample.
// The reference's repeated mirroring is periodic with period 2 * (len - 1), so it is evaluated
// in closed form; the result is always inside [minLoc, maxLoc).
__device__ __forceinline__ int reflect_index(int loc, int minLoc, int maxLoc)
{
    const int len = maxLoc - minLoc;
    if (len < 2) return maxLoc - 1;
    const int period = 2 * (len - 1);
    int r = (loc - minLoc) % period;
    if (r < 0) r += period;
    return minLoc + (r < len ? r : period - r);
}

// Resampled length ceil(length * outRate / inRate) in the reference's float arithmetic
// (resample.cpp:57); equal rates keep the length.
__host__ __device__ __forceinline__ int resampled_length(int L, float inRate, float outRate)
{
#ifdef __CUDA_ARCH__
    return inRate == outRate ? L : int(ceilf(__fdiv_rn(__fmul_rn(float(L), outRate), inRate)));
#else
    return inRate == outRate ? L : int(ceilf(float(L) * outRate / inRate));
#endif
}

// Frames of a sample (spectrogram.cpp:47-52), never negative.
__host__ __device__ __forceinline__ int num_windows(int length, int windowLength, int windowStep, bool center)
{
    if (!center) length -= windowLength;
    int f = length / windowStep + 1;
    return f < 0 ? 0 : f;
}

}  // namespace rppb
