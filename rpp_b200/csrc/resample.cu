// resample: band-limited interpolation with the caller's windowed-sinc lookup table.
//
// Reference: src/modules/tensor/cpu/kernel/resample.cpp:46-141 and RpptResamplingWindow
// (api/rppdefs.h:751-790).  Output length ceil(length * outRate / inRate) (float arithmetic);
// equal rates copy.  Outputs go in blocks of 256: a block's origin in the input is FP64
// (outBlock * inRate/outRate), split into an integer sample and a float phase, and the phase
// advances by the float ratio once per output — a sequential float sum the GPU replays in the
// same order.  Output j sums input samples [ceil(phase) - lobes, ceil(phase) + lobes) clipped to
// the signal, each weighted by linear interpolation in the table at x * scale + center.  For
// mono input the reference sums 4 lanes (SSE; truncating table index) and folds them as
// (l0 + l2) + (l1 + l3) before a scalar tail (flooring, clamped index); multi-channel input is
// summed per channel in order.  Every product and sum is explicitly rounded, so outputs are
// bit-identical to the host path.
//
// One CTA of 8 + 1 warps takes its 256-output blocks in groups of eight.  The ninth warp decodes the
// next group into shared memory: where each block lives, its output count and its phase sum, the
// eight sums side by side, one per lane.  Meanwhile the eight compute warps work through the current
// group, each taking one 32-output slice of every block of the group.  A block's first slice, the one
// with the smallest phases, falls to a different warp for each block.  When down-mixing, each warp
// stages its slice's input span (down-mixed once per input sample) in shared memory.  The lookup table
// sits in shared memory as (value, next - value) pairs when they fit, so a tap reads one 8-byte entry.
// Where a slice's phases allow it, the taps take the exact walk (resample_exact_range): each tap reads
// the entry 32 positions past the previous one and uses the same weight.  That is 4 float operations
// and 2 loads per tap, in place of ~10 operations.  Compute-bound.
#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "downmix.cuh"
#include "ops.hpp"

namespace rppb {
namespace {

constexpr int kBlock = 256;        // outputs per block (the reference's block size)
constexpr int kCopyChunk = 4096;   // floats per unit of an equal-rate copy

constexpr int kThreads = kBlock + 32;   // 8 warps compute outputs, the ninth decodes the next group of blocks

// Shared memory (floats): the table -- as padded (value, next - value) pairs when kPairs, else
// plain -- then, when down-mixing, the staged input span.
__host__ __device__ __forceinline__ size_t resample_pair_entries(int lutSize, int padLeft, int padRight)
{
    return size_t(padLeft) + size_t(lutSize - 1) + size_t(padRight);
}
__host__ __device__ __forceinline__ size_t resample_smem_floats(const ResampleWindowDev& w, bool pairs, bool span)
{
    return (pairs ? 2 * resample_pair_entries(w.lutSize, w.padLeft, w.padRight)
                  : ((size_t(w.lutSize) + 3) & ~size_t(3))) +
           (span ? size_t(kBlock / 32) * 256 : 0);   // down-mixing: each compute warp's slice span
}
constexpr size_t kPairTableLimit = 200 * 1024;   // bytes of shared memory for the pair layout

// Pair-table padding: a tap's x lies in (-(lobes + 1), lobes + 1), so its index, trunc or floor of
// x * scale + center, lies within [center - (lobes + 1)|scale| - 2, center + (lobes + 1)|scale| + 2].
// Whether every table position a tap can produce lies in [0, 2^22): the bound the magic-number index of
// Win<kPairs, true> needs (with the pair table, whose padding covers the indices; the clamp of the plain
// table is not applied on that path).  A tap's offset x = l - phase lies in [-lobes, lobes + 1): the
// first tap is ceil(phase) - lobes (or later, at the signal's start), and float rounding keeps x >= -lobes
// because -lobes is representable; x * scale + center is then bounded by its values at the two ends.
inline bool resample_magic_ok(const ResampleWindowDev& w, bool pairs)
{
    const double a = -double(w.lobes) * double(w.scale), b = (double(w.lobes) + 1.0) * double(w.scale);
    const double lo = double(w.center) + std::min(a, b), hi = double(w.center) + std::max(a, b);
    return pairs && lo >= 0.0 && hi < 4194304.0;
}

// A power-of-two table scale (x * scale exact for every finite tap position).
inline bool resample_scale_pow2(const ResampleWindowDev& w)
{
    int e = 0;
    return w.scale > 0.f && std::isfinite(w.scale) && std::frexp(double(w.scale), &e) == 0.5;
}

// The exact walk.  With table scale 32 and an integer center, take an output whose phase p has binary
// exponent E (p in [2^E, 2^(E+1))).  A tap at input sample l has offset l - p, a multiple of 2^(E-23)
// (l is an integer, E <= 23) with |l - p| <= lobes.  When lobes < 2^(E+1) that offset is a float, so the
// reference's float subtraction and its lane increments by 1 and 4 are exact.  The tap's table position
// 32 (l - p) + center is a multiple of 2^(E-18) (E <= 18) below center + 32 lobes; when that is below
// 2^(E+6) the position is a float too, so the fused multiply-add is exact.  The positions of consecutive
// taps then differ by exactly 32: their table indices are 32 apart and their interpolation weights equal.
// The range is empty unless the kernel takes the round-down-add index (kMagic) and the FMA position
// (kFma), whose values these are.
inline void resample_exact_range(ResampleWindowDev& w, bool magic, bool fma)
{
    w.exactMinE = 1 << 30;
    w.exactMaxE = -(1 << 30);
    if (!magic || !fma || w.scale != 32.f || w.center != std::floor(w.center) || w.lobes < 1) return;
    for (int e = -126; e <= 18; ++e)
        if (double(w.lobes) < std::ldexp(1.0, e + 1) &&
            double(w.center) + 32.0 * double(w.lobes) < std::ldexp(1.0, e + 6))
        {
            w.exactMinE = e;
            w.exactMaxE = 18;
            return;
        }
}

inline void resample_pads(ResampleWindowDev& w)
{
    const double reach = (double(w.lobes) + 1.0) * std::fabs(double(w.scale));
    const double lo = std::floor(double(w.center) - reach) - 2.0, hi = std::ceil(double(w.center) + reach) + 2.0;
    const double padL = lo < 0.0 ? -lo : 0.0, padR = hi > double(w.lutSize - 2) ? hi - double(w.lutSize - 2) : 0.0;
    const bool ok = padL < 65536.0 && padR < 65536.0;
    w.padLeft = ok ? int(padL) : -1;
    w.padRight = ok ? int(padR) : -1;
}

__device__ __forceinline__ int out_length(int L, float inRate, float outRate)
{
    return int(ceilf(__fdiv_rn(__fmul_rn(float(L), outRate), inRate)));
}

struct ResampleCount
{
    const float* inRate;
    const float* outRate;
    const int* dims;
    bool mix;
    const RppbClip* clips;   // table mode when set (mono, outRate = outRateAll)
    float outRateAll;
    __device__ long long operator()(int b) const
    {
        int L, C, Cs;
        float ir, orr;
        if (clips)
        {
            const RppbClip* c = RPPB_RD(clips + b);
            L = c->length, C = 1, Cs = 1, ir = c->inRate, orr = outRateAll;
        }
        else
        {
            L = *RPPB_RD(dims + 2 * b), Cs = *RPPB_RD(dims + (2 * b + 1)), C = mix ? 1 : Cs, ir = *RPPB_RD(inRate + b),
            orr = *RPPB_RD(outRate + b);
        }
        if (L <= 0 || Cs <= 0) return 0;
        if (ir == orr) return ((long long)L * C + kCopyChunk - 1) / kCopyChunk;
        const int outEnd = out_length(L, ir, orr);
        return outEnd <= 0 ? 0 : (outEnd + kBlock - 1) / kBlock;
    }
};

// kMagic: the table index comes from adding 1.5 * 2^23 with rounding toward minus infinity, which leaves
// floor(locRaw) in the low mantissa bits and float(floor(locRaw)) one subtraction away, instead of two
// float <-> int conversions per tap (low-throughput instructions).  Used when the host has shown that
// every locRaw a tap can produce lies in [0, 2^22): then trunc == floor, and both are exact this way.
// The pair entry is then addressed as bias + 8 * bits(m): the shared address of entry 0 less 8 * bits of
// 1.5 * 2^23 (mod 2^32), one shift-add per tap.
// kFma: the table scale is a power of two, so x * scale is exact and x * scale + center rounds once
// either way: one fused multiply-add gives the reference's value.
template <bool kPairs, bool kMagic = false, bool kFma = false>
struct Win
{
    const float* lut;     // shared memory: the table (plain layout)
    const float2* pairs;  // shared memory: (value, next - value) at index 0 of the padded pair layout
    int lutSize;
    float scale, center;
    uint32_t bias;        // kMagic with kPairs: shared address of pairs[0] - 8 * bits(1.5 * 2^23)

    __device__ __forceinline__ float interp(int idx, float weight) const
    {
        if constexpr (kPairs)
        {
            // pairs[i] for i in [-padLeft, lutSize - 2 + padRight] holds the entry the clamped index
            // [0, lutSize - 2] selects: no clamp for the indices a tap can produce
            const float2 e = pairs[idx];
            return __fadd_rn(e.x, __fmul_rn(weight, e.y));
        }
        else
        {
            idx = min(max(idx, 0), lutSize - 2);
            const float cur = lut[idx], nxt = lut[idx + 1];
            return __fadd_rn(cur, __fmul_rn(weight, __fsub_rn(nxt, cur)));
        }
    }
    __device__ __forceinline__ float magic_floor(float locRaw) const
    {
        constexpr float kM = 12582912.0f;   // 1.5 * 2^23
        const float m = __fadd_rd(locRaw, kM);
        const float w = __fsub_rn(locRaw, __fsub_rn(m, kM));
        if constexpr (kPairs)
        {
            const uint32_t a = bias + (uint32_t(__float_as_int(m)) << 3);
            float ex, ey;
            asm("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(ex), "=f"(ey) : "r"(a));
            return __fadd_rn(ex, __fmul_rn(w, ey));
        }
        return interp(__float_as_int(m) - __float_as_int(kM), w);
    }
    // rppdefs.h:771-782: truncating index (the SSE lanes)
    __device__ __forceinline__ float lane(float x) const
    {
        const float locRaw = kFma ? __fmaf_rn(x, scale, center) : __fadd_rn(__fmul_rn(x, scale), center);
        if constexpr (kMagic) return magic_floor(locRaw);
        const int idx = int(locRaw);
        return interp(idx, __fsub_rn(locRaw, float(idx)));
    }
    // rppdefs.h:760-769: floor, clamped index (the scalar tail and the multi-channel path)
    __device__ __forceinline__ float scalar(float x) const
    {
        const float locRaw = kFma ? __fmaf_rn(x, scale, center) : __fadd_rn(__fmul_rn(x, scale), center);
        if constexpr (kMagic) return magic_floor(locRaw);
        const int idx = int(floorf(locRaw));
        return interp(idx, __fsub_rn(locRaw, float(idx)));
    }
};

// The exact walk (resample_exact_range): the pair entry at byte offset kOff from shared address a.
template <int kOff>
__device__ __forceinline__ float2 pair_at(uint32_t a)
{
    float2 v;
    asm("ld.shared.v2.f32 {%0, %1}, [%2+%3];" : "=f"(v.x), "=f"(v.y) : "r"(a), "n"(kOff));
    return v;
}

// One output of a mono signal with the reference's operations: 4 lanes, folded as (l0 + l2) + (l1 + l3),
// then a scalar tail.
template <class W, class At>
__device__ __forceinline__ float mono_taps(const W& win, At at, int loc0, int loc1, float inPos)
{
    int l = loc0;
    const float locBegin = __fsub_rn(float(l), inPos);
    float lane4[4] = {__fadd_rn(locBegin, 0.f), __fadd_rn(locBegin, 1.f), __fadd_rn(locBegin, 2.f),
                      __fadd_rn(locBegin, 3.f)};
    float acc4[4] = {0.f, 0.f, 0.f, 0.f};
    for (; l + 3 < loc1; l += 4)
    {
#pragma unroll
        for (int q = 0; q < 4; ++q)
        {
            acc4[q] = __fadd_rn(acc4[q], __fmul_rn(at(l + q), win.lane(lane4[q])));
            lane4[q] = __fadd_rn(lane4[q], 4.f);
        }
    }
    float accum = __fadd_rn(__fadd_rn(acc4[0], acc4[2]), __fadd_rn(acc4[1], acc4[3]));
    float xx = __fsub_rn(float(l), inPos);
    for (; l < loc1; ++l, xx = __fadd_rn(xx, 1.f)) accum = __fadd_rn(accum, __fmul_rn(at(l), win.scalar(xx)));
    return accum;
}

// The same by the exact walk (resample_exact_range): the first tap's pair entry and weight by the same operations,
// then each tap 32 entries (256 bytes) further on at that weight; the same products and sums in the same order.
template <class W, class At>
__device__ __forceinline__ float mono_taps_exact(const W& win, At at, int loc0, int loc1, float inPos)
{
    constexpr float kM = 12582912.0f;   // 1.5 * 2^23
    const float locRaw = __fmaf_rn(__fsub_rn(float(loc0), inPos), win.scale, win.center);
    const float m = __fadd_rd(locRaw, kM);
    const float w = __fsub_rn(locRaw, __fsub_rn(m, kM));
    uint32_t a = win.bias + (uint32_t(__float_as_int(m)) << 3);
    auto tap = [&](int l, float2 e) { return __fmul_rn(at(l), __fadd_rn(e.x, __fmul_rn(w, e.y))); };
    int l = loc0;
    float acc4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 2
    for (; l + 3 < loc1; l += 4, a += 4 * 256)
    {
        acc4[0] = __fadd_rn(acc4[0], tap(l, pair_at<0>(a)));
        acc4[1] = __fadd_rn(acc4[1], tap(l + 1, pair_at<256>(a)));
        acc4[2] = __fadd_rn(acc4[2], tap(l + 2, pair_at<512>(a)));
        acc4[3] = __fadd_rn(acc4[3], tap(l + 3, pair_at<768>(a)));
    }
    float accum = __fadd_rn(__fadd_rn(acc4[0], acc4[2]), __fadd_rn(acc4[1], acc4[3]));
    for (; l < loc1; ++l, a += 256) accum = __fadd_rn(accum, tap(l, pair_at<0>(a)));
    return accum;
}

// One output of an interleaved multi-channel signal: per channel, in order.
template <class W>
__device__ __forceinline__ void channel_taps(const W& win, const float* in, float* out, int C, int loc0, int loc1,
                                             float inPos)
{
    constexpr int kMaxC = 16;
    float acc[kMaxC];
#pragma unroll
    for (int c = 0; c < kMaxC; ++c) acc[c] = 0.f;
    float xx = __fsub_rn(float(loc0), inPos);
    for (int l = loc0; l < loc1; ++l, xx = __fadd_rn(xx, 1.f))
    {
        const float wv = win.scalar(xx);
#pragma unroll
        for (int c = 0; c < kMaxC; ++c)
            if (c < C) acc[c] = __fadd_rn(acc[c], __fmul_rn(__ldg(RPPB_RD(in + (long long)l * C + c)), wv));
    }
#pragma unroll
    for (int c = 0; c < kMaxC; ++c)
        if (c < C) *RPPB_WR(out + c) = acc[c];
}

// The reference's phase sum of a block.
__device__ __forceinline__ void block_phases(float p, float fscale, float* to)
{
    float4* out = reinterpret_cast<float4*>(to);
#pragma unroll 8
    for (int k = 0; k < kBlock / 4; ++k)
    {
        float4 q;
        q.x = p;
        q.y = p = __fadd_rn(p, fscale);
        q.z = p = __fadd_rn(p, fscale);
        q.w = p = __fadd_rn(p, fscale);
        p = __fadd_rn(p, fscale);
        out[k] = q;
    }
}

// A unit of the flat work list, decoded by the phase warp for the compute warps.
constexpr int kUnitSkip = 0, kUnitCopy = 1, kUnitResample = 2;
struct UnitInfo
{
    const float* x;        // the sample's input
    float* y;              // the sample's output
    int L, Csrc, C;        // input length, input channels, channels of the resampled signal
    int unit;              // the unit's index within its sample
    uint32_t dstStride;
    int mode;              // kUnitSkip, kUnitCopy or kUnitResample
    int outEnd;            // resampling: outputs of the sample that the destination takes
    int inBlockRounded;    // resampling: the input sample the unit's phases count from
    float wc;              // down-mixing: the weight of every channel
};

// A CTA takes its units (blockIdx.x + i * gridDim.x, i = 0, 1, ...) in groups of kGroup.  Lane j of the
// phase warp decodes unit j of the next group (the eight phase sums run side by side) while the compute
// warps work through the current group in kGroup steps: at step s, warp w takes outputs [32 s, 32 s + 32)
// of unit (w + s) mod kGroup.  A unit's first outputs have the smallest phases and are the ones the exact
// walk may not cover, so every warp takes one such slice per group and the group barrier waits for no
// single slow warp.
constexpr int kWarps = kBlock / 32;   // compute warps
constexpr int kGroup = kWarps;
constexpr int kSliceSpan = 256;       // down-mixing: input samples of one slice staged by its warp
static_assert(kGroup == kWarps && kBlock == kWarps * 32, "one 32-output slice per compute warp and step");

// kMix: the input is interleaved multi-channel and is down-mixed to mono on the fly (MonoMix), so
// the launch equals rppt_down_mixing_gpu followed by a mono rppt_resample_gpu.
template <bool kMix, bool kTable, bool kPairs, bool kMagic = false, bool kFma = false>
__global__ void __launch_bounds__(kThreads, 4)
    resample_kernel(const float* __restrict__ src, uint32_t srcStride, float* __restrict__ dst, uint32_t dstStride,
                    const float* __restrict__ inRateT, const float* __restrict__ outRateT,
                    const int* __restrict__ dims, ResampleWindowDev wd, bool normalize,
                    const long long* __restrict__ prefix, int n, const RppbClip* __restrict__ clips,
                    float outRateAll)
{
    extern __shared__ float s_lut[];   // the table, then (down-mixing) each compute warp's staged slice span
    __shared__ long long s_prefix[kPrefixCache];
    grid_dependency_wait();   // the prefix, when launched after the held-weights kernel
    prefix = cache_prefix(dependency_result(prefix), n, s_prefix);   // ends with __syncthreads
    const long long total = prefix[n];
    if (total == 0) return;
    const int pairCount = kPairs ? int(resample_pair_entries(wd.lutSize, wd.padLeft, wd.padRight)) : 0;
    float* s_spans = s_lut + (kPairs ? 2 * pairCount : ((wd.lutSize + 3) & ~3));
    __shared__ __align__(16) float s_phase[2][kGroup][kBlock];
    __shared__ UnitInfo s_unit[2][kGroup];
    if (kPairs)
        for (int i = threadIdx.x; i < pairCount; i += kThreads)
        {
            const int e = min(max(i - wd.padLeft, 0), wd.lutSize - 2);   // the clamped entry
            const float v0 = *RPPB_RD(wd.lut + e), v1 = *RPPB_RD(wd.lut + (e + 1));
            reinterpret_cast<float2*>(s_lut)[i] = make_float2(v0, __fsub_rn(v1, v0));
        }
    else
        for (int i = threadIdx.x; i < wd.lutSize; i += kThreads) s_lut[i] = *RPPB_RD(wd.lut + i);
    const Win<kPairs, kMagic, kFma> win{s_lut, reinterpret_cast<const float2*>(s_lut) + (kPairs ? wd.padLeft : 0),
                                        wd.lutSize, wd.scale, wd.center,
                                        uint32_t(__cvta_generic_to_shared(reinterpret_cast<const float2*>(s_lut) +
                                                                          (kPairs ? wd.padLeft : 0))) -
                                            0x5A000000u};   // 8 * 0x4B400000 mod 2^32
    const int lobes = wd.lobes;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    // the CTA's unit j of group g
    auto unit_of = [&](long long g, int j) {
        return (long long)blockIdx.x + (g * kGroup + j) * (long long)gridDim.x;
    };
    // decodes unit w into s_unit[slot][j]: where it lives, what it does and, for a resampling unit, the
    // reference's phase sum into s_phase[slot][j] (replayed in its float order)
    auto decode = [&](long long w, int slot, int j) {
        UnitInfo u;
        u.mode = kUnitSkip;
        if (w < total)
        {
            const int b = ragged_find(prefix, n, w);
            u.unit = int(w - prefix[b]);
            const RppbClip* clip = kTable ? RPPB_RD(clips + b) : nullptr;
            u.L = kTable ? clip->length : *RPPB_RD(dims + 2 * b);
            u.Csrc = kTable ? 1 : *RPPB_RD(dims + (2 * b + 1));
            u.C = kMix ? 1 : u.Csrc;
            const float inRate = kTable ? clip->inRate : *RPPB_RD(inRateT + b);
            const float outRate = kTable ? outRateAll : *RPPB_RD(outRateT + b);
            u.x = kTable ? clip->src : src + size_t(b) * srcStride;
            u.y = kTable ? clip->work : dst + size_t(b) * dstStride;
            u.dstStride = kTable ? 0x7fffffffu : dstStride;   // a clip's work buffer holds the whole resampled clip
            u.wc = kMix ? MonoMix::weight(max(u.Csrc, 1), normalize) : 1.f;
            u.mode = inRate == outRate ? kUnitCopy : (kMix && u.Csrc > 64) ? kUnitSkip : kUnitResample;
            u.outEnd = 0;
            u.inBlockRounded = 0;
            if (u.mode == kUnitResample)
            {
                u.outEnd = min(out_length(u.L, inRate, outRate), int(u.dstStride / uint32_t(u.C)));
                const double scale = __ddiv_rn(double(inRate), double(outRate));
                const float fscale = __double2float_rn(scale);
                const double inBlockRaw = __dmul_rn(double(u.unit * kBlock), scale);
                u.inBlockRounded = int(inBlockRaw);
                block_phases(__double2float_rn(__dsub_rn(inBlockRaw, double(int(inBlockRaw)))), fscale, s_phase[slot][j]);
                // ask L2 for the unit's input span (a group ahead of its use): the taps of its outputs
                // read samples [ceil(first phase) - lobes, ceil(last phase) + lobes) from inBlockRounded on
                const int cnt = min(kBlock, u.outEnd - u.unit * kBlock);
                if (cnt > 0)
                {
                    const float* ph = s_phase[slot][j];
                    const long long lo = max((long long)u.inBlockRounded + int(ceilf(ph[0])) - lobes, 0ll);
                    const long long hi =
                        min((long long)u.inBlockRounded + int(ceilf(ph[cnt - 1])) + lobes, (long long)u.L);
                    if (hi > lo) l2_prefetch(u.x + lo * u.Csrc, u.x + hi * u.Csrc);
                }
            }
        }
        s_unit[slot][j] = u;
    };

    if (warp == kWarps && lane < kGroup) decode(unit_of(0, lane), 0, lane);
    __syncthreads();
    int cur = 0;
    for (long long g = 0; unit_of(g, 0) < total; ++g, cur ^= 1)
    {
        if (warp == kWarps)
        {
            // the phase warp: the next group while the others compute this one
            if (lane < kGroup) decode(unit_of(g + 1, lane), cur ^ 1, lane);
        }
        else
        {
            float* s_span = s_spans + warp * kSliceSpan;
            for (int step = 0; step < kGroup; ++step)
            {
                const int j = (warp + step) % kGroup;
                const UnitInfo u = s_unit[cur][j];
                const float* x = u.x;
                float* y = u.y;
                const int L = u.L, C = u.C;
                const MonoMix mix{x, kMix ? u.Csrc : 1, u.wc};
                if (u.mode == kUnitCopy)
                {
                    constexpr int kPart = kCopyChunk / kGroup;
                    const long long count =
                        kMix ? min((long long)L, (long long)u.dstStride)
                             : (kTable ? (long long)L : min((long long)L * C, (long long)min(srcStride, u.dstStride)));
                    const long long i0 = (long long)u.unit * kCopyChunk + step * kPart;
                    for (long long i = i0 + lane; i < min(count, i0 + kPart); i += 32)
                        *RPPB_WR(y + i) = kMix ? mix(i) : *RPPB_RD(x + i);
                }
                else if (u.mode == kUnitResample)
                {
                    const float* ph = s_phase[cur][j];
                    const int outBlock = u.unit * kBlock;
                    const int cnt = min(kBlock, u.outEnd - outBlock);   // outputs of the unit
                    const int k0 = step * 32;                           // the slice's first output
                    if (k0 < cnt)
                    {
                        const int inBlockRounded = u.inBlockRounded;
                        const float* in = x + (long long)inBlockRounded * C;
                        // down-mixing: the slice's input span [lo, hi), down-mixed once per sample, staged by
                        // this warp (every tap of the slice lies inside it because the phases increase)
                        int lo = 0;
                        bool staged = false;
                        if (kMix)
                        {
                            lo = max(int(ceilf(ph[k0])) - lobes, -inBlockRounded);
                            const int hi = min(int(ceilf(ph[min(k0 + 31, cnt - 1)])) + lobes, L - inBlockRounded);
                            staged = hi - lo <= kSliceSpan;
                            if (staged)
                                for (int i = lane; i < hi - lo; i += 32)
                                    s_span[i] = mix((long long)inBlockRounded + lo + i);
                            __syncwarp();
                        }
                        const int k = k0 + lane;
                        const int outPos = outBlock + k;
                        const float inPos = ph[k];
                        // the exact walk (resample_exact_range) where every output of the slice allows it,
                        // so a warp runs one of the two tap loops
                        bool exact = false;
                        if constexpr (kPairs && kMagic && kFma)
                        {
                            const int e = int((__float_as_uint(inPos) >> 23) & 0xffu) - 127;
                            exact = __all_sync(0xffffffffu, k >= cnt || (e >= wd.exactMinE && e <= wd.exactMaxE));
                        }
                        if (k < cnt)
                        {
                            const int xc = int(ceilf(inPos));
                            int loc0 = xc - lobes, loc1 = xc + lobes;
                            if (loc0 + inBlockRounded < 0) loc0 = -inBlockRounded;
                            if (loc1 + inBlockRounded > L) loc1 = L - inBlockRounded;
                            if (kMix || C == 1)
                            {
                                auto taps = [&](auto at) { return mono_taps(win, at, loc0, loc1, inPos); };
                                auto taps_exact = [&](auto at) { return mono_taps_exact(win, at, loc0, loc1, inPos); };
                                auto run = [&](auto at) {
                                    if constexpr (kPairs && kMagic && kFma)
                                        if (exact) return taps_exact(at);
                                    return taps(at);
                                };
                                float r;
                                if (kMix && staged) r = run([&](int l) { return s_span[l - lo]; });
                                else if (kMix) r = run([&](int l) { return mix((long long)inBlockRounded + l); });
                                else r = run([&](int l) { return __ldg(RPPB_RD(in + l)); });
                                *RPPB_WR(y + outPos) = r;
                            }
                            else
                                channel_taps(win, in, y + (long long)outPos * C, C, loc0, loc1, inPos);
                        }
                        if (kMix) __syncwarp();   // the warp's span is restaged by its next slice
                    }
                }
                // kUnitSkip: no unit, or more than 64 channels to down-mix (rejected by the caller)
            }
        }
        __syncthreads();   // slot cur is rewritten by the next group's decode; slot cur ^ 1 is ready
    }
}

// ---------------------------------------------------------------- held weights (16 lobes)
// The weights of an output's 32 taps depend on its phase alone, and a block's phases follow from its first
// one, so blocks whose first phase has the same bits share all 256 x 32 weights.  For integer rates the first
// phase repeats every P = outRate / gcd(256 inRate, outRate) blocks (5 for 44.1 or 22.05 kHz to 16 kHz, 1 for
// 48 kHz); the FP64 block origin can move it by a rounding, so the bits are compared block by block.  A CTA
// takes an item of up to kItemBlocks blocks P apart, computes the weights once with the reference's
// operations, holds them in registers and runs every block of the item through them: one sample load and
// two float operations per tap instead of two loads and four (or, outside the exact walk, ten) operations.
//
// Four lanes share an output: lane q sums the taps q, q + 4, ..., the reference's SSE lane q, and two
// exchanges fold the sums as (l0 + l2) + (l1 + l3).  A warp's 32 sample loads then cover the span of 8
// neighbouring outputs, 8 ratio + 4 consecutive floats: no bank conflicts up to a ratio of 3.5, where lanes on
// neighbouring outputs (stride ratio) take 2 to 3 shared-memory wavefronts per load.  A thread holds 4
// outputs' quarters, 32 weights (2 outputs and twice the threads: the per-block work of a thread, staging and
// addresses, is then as large as its sums).  The next block's span is loaded into registers while the current
// one is summed.  Blocks whose taps reach past the signal's ends, or whose first phase differs, take the
// reference's operations output by output.
constexpr int kHeldLobes = 16;
constexpr int kItemBlocks = 16;      // blocks of an item
constexpr int kHeldCtas = 2;         // per SM
constexpr int kHeldSpan = 1024;      // staged samples of a block: ratios up to 3.8
constexpr int kHeldPeriod = 64;      // longest period between blocks that share weights
constexpr int kHeldShare = 4;        // blocks of a sample that share weights, at least
constexpr int kHeldMono = 16, kHeldMixed = 32;   // and its blocks: the first and the last are summed output by output
constexpr int kHeldWarps = 8;        // compute warps: 8 outputs per pass and warp, four passes per block
constexpr int kHeldCompute = kHeldWarps * 32, kHeldThreads = kHeldCompute + 32;
constexpr int kHeldOuts = kBlock / (kHeldWarps * 8);   // outputs per thread
constexpr int kSpanLoads = kHeldSpan / kHeldCompute;
static_assert(kHeldOuts == 4, "the fold of the lane sums assumes four outputs per thread");

__device__ __forceinline__ int phase_period(float inRate, float outRate)
{
    const bool whole = inRate >= 1.f && outRate >= 1.f && inRate <= 1048576.f && outRate <= 1048576.f &&
                       inRate == floorf(inRate) && outRate == floorf(outRate);
    if (!whole) return 0;
    const int o = int(outRate);
    int a = int(inRate) * kBlock, b = o;   // at most 2^28
    while (b)
    {
        const int t = a % b;
        a = b;
        b = t;
    }
    const int p = o / a;
    return p <= kHeldPeriod ? p : 0;
}

// Whether the held-weights kernel takes a sample: its rates repeat a phase (48 to 44.1 kHz or 16 to 44.1 kHz, with
// items of one block, took 1230 and 1209 us there and 429 and 380 us in resample_kernel on 64 clips of 8 s), the span of
// a block fits the staging (96 to 16 kHz, every block output by output: stereo 1193 against 319 us), and it has enough
// blocks (4096 stereo clips of 16 blocks 498 against 413 us, 2048 of 32 blocks 368 against 409; mono 247 against 282
// and 218 against 273).
__device__ __forceinline__ bool held_sample(int outEnd, int period, float inRate, float outRate, bool mix)
{
    if (period == 0 || float(kBlock) * inRate > float(kHeldSpan - 2 * kHeldLobes - 4) * outRate) return false;
    return (outEnd + kBlock - 1) / kBlock >= max(kHeldShare * period, mix ? kHeldMixed : kHeldMono);
}

// How its blocks are dealt to items: item i takes blocks i % period + period * (first + j).
struct ItemPlan
{
    int blocks, period, per, groups;
    __device__ __forceinline__ ItemPlan(int outEnd, int phasePeriod)
    {
        blocks = (outEnd + kBlock - 1) / kBlock;
        period = phasePeriod;
        const int each = (blocks + period - 1) / period;
        groups = (each + kItemBlocks - 1) / kItemBlocks;
        per = (each + groups - 1) / groups;
    }
    __device__ __forceinline__ long long items() const { return (long long)period * groups; }
};

// Deals the samples to the two kernels: held[0..n] and general[0..n] are the prefixes of their work units.  The
// held-weights kernel takes what held_sample admits when the batch has minBlocks such blocks, else nothing.
__global__ void __launch_bounds__(1024) resample_split_kernel(const float* __restrict__ inRateT,
                                                              const float* __restrict__ outRateT,
                                                              const int* __restrict__ dims, bool mix, int n,
                                                              int minBlocks, long long* __restrict__ held,
                                                              long long* __restrict__ general,
                                                              unsigned long long* __restrict__ nextItem)
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    struct Units
    {
        long long all;     // of the general kernel
        int items, blocks; // of the held-weights kernel (0: not for it)
        bool copy;         // equal rates: either kernel
    };
    auto units = [&](int b) {
        Units u{0, 0, 0, false};
        const int L = *RPPB_RD(dims + 2 * b), Cs = *RPPB_RD(dims + (2 * b + 1)), C = mix ? 1 : Cs;
        const float ir = *RPPB_RD(inRateT + b), orr = *RPPB_RD(outRateT + b);
        if (L <= 0 || Cs <= 0) return u;
        u.copy = ir == orr;
        if (u.copy)
        {
            u.all = ((long long)L * C + kCopyChunk - 1) / kCopyChunk;
            return u;
        }
        const int outEnd = out_length(L, ir, orr);
        if (outEnd <= 0) return u;
        u.all = (outEnd + kBlock - 1) / kBlock;
        const int period = phase_period(ir, orr);
        if (C != 1 || Cs > 64 || !held_sample(outEnd, period, ir, orr, mix)) return u;
        u.blocks = int(u.all);
        u.items = int(ItemPlan(outEnd, period).items());
        return u;
    };
    __shared__ long long s_total[2][32];
    __shared__ int s_blocks;
    const int t = threadIdx.x, threads = blockDim.x;
    const int per = (n + threads - 1) / threads;
    const int b0 = min(n, t * per), b1 = min(n, b0 + per);
    if (t == 0)
    {
        s_blocks = 0;
        *RPPB_WR(nextItem) = 0ull;
    }
    __syncthreads();
    Units first{0, 0, 0, false};
    int blocks = 0;                           // only whether the sum reaches minBlocks counts
    long long all = 0, items = 0, rest = 0;   // the general kernel's units alone; both kernels' units when both run
    for (int b = b0; b < b1; ++b)
    {
        const Units u = units(b);
        if (b == b0) first = u;
        blocks = min(blocks + min(u.blocks, minBlocks), minBlocks);
        all += u.all;
        items += u.copy ? u.all : (long long)u.items;
        rest += u.copy || u.items > 0 ? 0 : u.all;
    }
    blocks = __reduce_add_sync(0xffffffffu, blocks);
    if ((t & 31) == 0 && blocks > 0) atomicAdd(&s_blocks, blocks);
    __syncthreads();
    const bool use = s_blocks >= minBlocks;
    long long h = use ? items : 0, g = use ? rest : all;
    h = block_exclusive_scan(h, s_total[0]);
    g = block_exclusive_scan(g, s_total[1]);
    for (int b = b0; b < b1; ++b)
    {
        const Units u = b == b0 ? first : units(b);
        *RPPB_WR(held + b) = h;
        *RPPB_WR(general + b) = g;
        const bool mine = use && (u.copy || u.items > 0);
        h += !mine ? 0 : u.copy ? u.all : (long long)u.items;
        g += mine ? 0 : u.all;
    }
    if (t == threads - 1)
    {
        *RPPB_WR(held + n) = h;
        *RPPB_WR(general + n) = g;
    }
}

constexpr int kBlockHeld = 0, kBlockEdge = 1, kBlockOther = 2;
struct HeldItem
{
    const float* x;
    float* y;
    int L, Csrc, unit;         // unit: copies only
    int mode;                  // kUnitSkip, kUnitCopy or kUnitResample; -1: no item left
    int count, held;           // blocks; the first `held` of them share the item's weights
    int lo, span;              // the blocks' samples are [origin + lo, origin + lo + span)
    float wc;
    float fscale;
    int block[kItemBlocks];    // output block
    int origin[kItemBlocks];   // the input sample its phases count from
    int outs[kItemBlocks];     // its outputs
    int kind[kItemBlocks];
    float first[kItemBlocks];  // its first phase
};

// The item's blocks that do not share its weights, an output per thread with the reference's operations.  Not
// inlined: its registers would come on top of the held weights.
template <bool kMix>
__device__ RPPB_OUT_OF_LINE void other_blocks(const Win<true, true, true>& win, const HeldItem& it, const MonoMix& mix,
                                          const float* ph, float* s_other, int exactMinE, int exactMaxE)
{
    for (int e = it.held; e < it.count; ++e)
    {
        const float* phase = ph;
        if (it.kind[e] == kBlockOther)
        {
            asm volatile("bar.sync 1, 256;" ::: "memory");
            if (threadIdx.x == 0) block_phases(it.first[e], it.fscale, s_other);
            asm volatile("bar.sync 1, 256;" ::: "memory");
            phase = s_other;
        }
        const int k = threadIdx.x;
        if (k >= it.outs[e]) continue;
        const float p = phase[k];
        const int origin = it.origin[e], L = it.L;
        const int xc = int(ceilf(p));
        int loc0 = xc - kHeldLobes, loc1 = xc + kHeldLobes;
        if (loc0 + origin < 0) loc0 = -origin;
        if (loc1 + origin > L) loc1 = L - origin;
        const long long outPos = (long long)it.block[e] * kBlock + k;
        auto at = [&](int l) {
            return kMix ? mix((long long)origin + l) : __ldg(RPPB_RD(it.x + ((long long)origin + l)));
        };
        const int ex = int((__float_as_uint(p) >> 23) & 0xffu) - 127;
        *RPPB_WR(it.y + outPos) = ex >= exactMinE && ex <= exactMaxE ? mono_taps_exact(win, at, loc0, loc1, p)
                                                                     : mono_taps(win, at, loc0, loc1, p);
    }
}

template <bool kMix>
__global__ void __launch_bounds__(kHeldThreads, 2)
    resample_held_kernel(const float* __restrict__ src, uint32_t srcStride, float* __restrict__ dst, uint32_t dstStride,
                         const float* __restrict__ inRateT, const float* __restrict__ outRateT,
                         const int* __restrict__ dims, ResampleWindowDev wd, bool normalize,
                         const long long* __restrict__ prefix, unsigned long long* __restrict__ nextItem, int n)
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    extern __shared__ float s_lut[];   // the padded (value, next - value) table, then two staged spans
    const int pairCount = int(resample_pair_entries(wd.lutSize, wd.padLeft, wd.padRight));
    float* s_span = s_lut + 2 * pairCount;
    __shared__ __align__(16) float s_phase[2][kBlock];
    __shared__ __align__(16) float s_other[kBlock];   // phases of a block of kind kBlockOther
    __shared__ HeldItem s_item[2];
    for (int i = threadIdx.x; i < pairCount; i += kHeldThreads)
    {
        const int e = min(max(i - wd.padLeft, 0), wd.lutSize - 2);
        const float v0 = *RPPB_RD(wd.lut + e), v1 = *RPPB_RD(wd.lut + (e + 1));
        reinterpret_cast<float2*>(s_lut)[i] = make_float2(v0, __fsub_rn(v1, v0));
    }
    const float2* pairs = reinterpret_cast<const float2*>(s_lut) + wd.padLeft;
    const Win<true, true, true> win{s_lut, pairs, wd.lutSize, wd.scale, wd.center,
                                    uint32_t(__cvta_generic_to_shared(pairs)) - 0x5A000000u};
    __shared__ long long s_prefix[kPrefixCache];
    grid_dependency_wait();   // the prefix and the zeroed counter
    nextItem = dependency_result(nextItem);
    prefix = cache_prefix(dependency_result(prefix), n, s_prefix);
    const long long total = prefix[n];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    // the phase warp claims the next item and decodes it into slot
    auto decode = [&](int slot) {
        HeldItem& it = s_item[slot];
        long long w = 0;
        if (lane == 0) w = (long long)atomicAdd(RPPB_WR(nextItem), 1ull);
        w = __shfl_sync(0xffffffffu, w, 0);
        if (w >= total)
        {
            if (lane == 0) it.mode = -1;
            return;
        }
        const int b = ragged_find(prefix, n, w);
        const int local = int(w - prefix[b]);
        const int L = *RPPB_RD(dims + 2 * b), Csrc = *RPPB_RD(dims + (2 * b + 1));
        const float inRate = *RPPB_RD(inRateT + b), outRate = *RPPB_RD(outRateT + b);
        const float* x = src + size_t(b) * srcStride;
        const int mode = inRate == outRate ? kUnitCopy : kUnitResample;
        if (lane == 0)
        {
            it.x = x;
            it.y = dst + size_t(b) * dstStride;
            it.L = L;
            it.Csrc = Csrc;
            it.unit = local;
            it.mode = mode;
            it.wc = kMix ? MonoMix::weight(max(Csrc, 1), normalize) : 1.f;
        }
        if (mode != kUnitResample) return;
        const int outFull = out_length(L, inRate, outRate);
        const int outEnd = min(outFull, int(dstStride));
        const ItemPlan plan(outFull, phase_period(inRate, outRate));
        const double scale = __ddiv_rn(double(inRate), double(outRate));
        const float fscale = __double2float_rn(scale);
        const int residue = local % plan.period, j0 = local / plan.period * plan.per;
        // lane j: the item's block j
        const int u = residue + plan.period * (j0 + lane);
        const bool mine = lane < plan.per && u < plan.blocks && u * kBlock < outEnd;
        const double raw = __dmul_rn(double(u * kBlock), scale);
        const int origin = int(raw);
        const float first = __double2float_rn(__dsub_rn(raw, double(origin)));
        const unsigned all = __ballot_sync(0xffffffffu, mine);
        const int count = __popc(all);
        const float held = __shfl_sync(0xffffffffu, first, 0);
        if (lane == 0) block_phases(held, fscale, s_phase[slot]);
        __syncwarp();
        const float* ph = s_phase[slot];
        const int lo = int(ceilf(ph[0])) - kHeldLobes, span = int(ceilf(ph[kBlock - 1])) + kHeldLobes - lo;
        if (mine)
        {
            const int outs = min(kBlock, outEnd - u * kBlock);
            const long long from = (long long)origin + lo;
            const long long to = (long long)origin + int(ceilf(ph[outs - 1])) + kHeldLobes;
            const int kind = __float_as_uint(first) != __float_as_uint(held)              ? kBlockOther
                             : from < 0 || to > L || span > kHeldSpan                      ? kBlockEdge
                                                                                           : kBlockHeld;
            // the blocks that share the weights first
            const unsigned share = __ballot_sync(all, kind == kBlockHeld);
            const unsigned before = (1u << lane) - 1u;
            const int at = kind == kBlockHeld ? __popc(share & before) : __popc(share) + __popc(all & ~share & before);
            it.block[at] = u;
            it.origin[at] = origin;
            it.outs[at] = outs;
            it.first[at] = first;
            it.kind[at] = kind;
            if (lane == 0) it.held = __popc(share);
            // ask L2 for the block's samples an item ahead of their use
            const long long f = max(from, 0ll), t = min(to, (long long)L);
            if (t > f) l2_prefetch(x + f * Csrc, x + t * Csrc);
        }
        if (lane == 0)
        {
            it.count = count;
            if (count == 0) it.held = 0;
            it.lo = lo;
            it.span = span;
            it.fscale = fscale;
        }
    };

    if (threadIdx.x == 0) s_item[0].mode = kUnitSkip;   // the first pass only decodes
    __syncthreads();
    for (int cur = 0;; cur ^= 1)
    {
        const HeldItem& it = s_item[cur];
        const int mode = it.mode;
        if (mode < 0) break;
        if (warp == kHeldWarps) decode(cur ^ 1);
        else if (mode == kUnitCopy)
        {
            const MonoMix mix{it.x, kMix ? it.Csrc : 1, it.wc};
            const long long L = it.L;
            const long long count = kMix ? min(L, (long long)dstStride) : min(L * it.Csrc, (long long)min(srcStride, dstStride));
            const long long i0 = (long long)it.unit * kCopyChunk, end = min(count, i0 + kCopyChunk);
            const float* x = it.x;
            float* y = it.y;
            for (long long i = i0 + threadIdx.x; i < end; i += 4 * kHeldCompute)
            {
                float v[4];
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (i + k * kHeldCompute < end) v[k] = kMix ? mix(i + k * kHeldCompute) : *RPPB_RD(x + (i + k * kHeldCompute));
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (i + k * kHeldCompute < end) *RPPB_WR(y + (i + k * kHeldCompute)) = v[k];
            }
        }
        else if (mode == kUnitResample)
        {
            const int q = lane & 3, o8 = lane >> 2, tid = threadIdx.x;
            const float* ph = s_phase[cur];
            const MonoMix mix{it.x, kMix ? it.Csrc : 1, it.wc};
            const int held = it.held;
            if (held > 0)
            {
                const int lo = it.lo, span = it.span;
                // a block's samples: loaded into registers, then stored (down-mixed) into a span buffer
                const int channels = kMix ? it.Csrc : 1;
                const bool two = channels == 2 && (reinterpret_cast<uintptr_t>(it.x) & 7) == 0;
                const float wc = it.wc;
                const float* base = it.x + (long long)(lo + tid) * (two ? 2 : 1);
                float2 v[kSpanLoads];
                auto load = [&](int j) {
                    const int origin = it.origin[j];
                    const int most = min(span, it.L - origin - lo) - tid;   // samples past the signal are not summed
                    if (two)
                    {
                        const float2* at = reinterpret_cast<const float2*>(base) + origin;
#pragma unroll
                        for (int k = 0; k < kSpanLoads; ++k)
                            if (k * kHeldCompute < most) v[k] = __ldg(RPPB_RD(at + k * kHeldCompute));
                    }
                    else if (channels == 1)
                    {
                        const float* at = base + origin;
#pragma unroll
                        for (int k = 0; k < kSpanLoads; ++k)
                            if (k * kHeldCompute < most) v[k].x = __ldg(RPPB_RD(at + k * kHeldCompute));
                    }
                    else
                    {
#pragma unroll
                        for (int k = 0; k < kSpanLoads; ++k)
                            if (k * kHeldCompute < most) v[k].x = mix((long long)origin + lo + tid + k * kHeldCompute);
                    }
                };
                auto store = [&](int slot) {
                    float* to = s_span + slot * kHeldSpan + tid;
                    if (two)
                    {
                        // MonoMix's sum for two channels
#pragma unroll
                        for (int k = 0; k < kSpanLoads; ++k)
                            if (tid + k * kHeldCompute < span)
                                to[k * kHeldCompute] = __fadd_rn(__fadd_rn(0.f, __fmul_rn(v[k].x, wc)), __fmul_rn(v[k].y, wc));
                    }
                    else
                    {
#pragma unroll
                        for (int k = 0; k < kSpanLoads; ++k)
                            if (tid + k * kHeldCompute < span) to[k * kHeldCompute] = v[k].x;
                    }
                };
                load(0);
                // weights of taps q, q + 4, ... of outputs m * 64 + warp * 8 + o8
                float w[kHeldOuts][8];
                int off[kHeldOuts];
#pragma unroll
                for (int m = 0; m < kHeldOuts; ++m)
                {
                    const float p = ph[m * 64 + warp * 8 + o8];
                    const int l = int(ceilf(p)) - kHeldLobes;
                    off[m] = l - lo + q;
                    const float begin = __fsub_rn(float(l), p);
                    const int e = int((__float_as_uint(p) >> 23) & 0xffu) - 127;
                    if (__all_sync(0xffffffffu, e >= wd.exactMinE && e <= wd.exactMaxE))
                    {
                        // the exact walk: one entry and weight, then 32 entries per tap
                        constexpr float kM = 12582912.0f;   // 1.5 * 2^23
                        const float raw = __fmaf_rn(begin, win.scale, win.center);
                        const float r = __fadd_rd(raw, kM);
                        const float f = __fsub_rn(raw, __fsub_rn(r, kM));
                        const uint32_t a = win.bias + (uint32_t(__float_as_int(r)) << 3) + 256u * q;
                        auto at = [&](float2 e) { return __fadd_rn(e.x, __fmul_rn(f, e.y)); };
                        w[m][0] = at(pair_at<0>(a));
                        w[m][1] = at(pair_at<1024>(a));
                        w[m][2] = at(pair_at<2048>(a));
                        w[m][3] = at(pair_at<3072>(a));
                        w[m][4] = at(pair_at<4096>(a));
                        w[m][5] = at(pair_at<5120>(a));
                        w[m][6] = at(pair_at<6144>(a));
                        w[m][7] = at(pair_at<7168>(a));
                    }
                    else
                    {
                        float t = __fadd_rn(begin, float(q));
#pragma unroll
                        for (int k = 0; k < 8; ++k, t = __fadd_rn(t, 4.f)) w[m][k] = win.lane(t);
                    }
                }
                const bool up = q & 2, odd = q & 1;
                const int mine = q * 64 + warp * 8 + o8;   // the output this lane ends with
                float* y = it.y + mine;
                store(0);
                asm volatile("bar.sync 1, 256;" ::: "memory");
                for (int j = 0; j < held; ++j)
                {
                    if (j + 1 < held) load(j + 1);
                    const float* sp = s_span + (j & 1) * kHeldSpan;
                    float acc[kHeldOuts];
#pragma unroll
                    for (int m = 0; m < kHeldOuts; ++m)
                    {
                        const float* s = sp + off[m];
                        acc[m] = 0.f;
#pragma unroll
                        for (int k = 0; k < 8; ++k) acc[m] = __fadd_rn(acc[m], __fmul_rn(s[4 * k], w[m][k]));
                    }
                    // fold (l0 + l2) + (l1 + l3): after the exchanges lane q has output q * 64 + warp * 8 + o8
                    const float g0 = __shfl_xor_sync(0xffffffffu, up ? acc[0] : acc[2], 2);
                    const float g1 = __shfl_xor_sync(0xffffffffu, up ? acc[1] : acc[3], 2);
                    const float h0 = __fadd_rn(up ? acc[2] : acc[0], g0), h1 = __fadd_rn(up ? acc[3] : acc[1], g1);
                    const float r = __fadd_rn(odd ? h1 : h0, __shfl_xor_sync(0xffffffffu, odd ? h0 : h1, 1));
                    if (mine < it.outs[j]) *RPPB_WR(y + (long long)it.block[j] * kBlock) = r;
                    if (j + 1 < held) store((j + 1) & 1);
                    asm volatile("bar.sync 1, 256;" ::: "memory");
                }
            }
            if (held < it.count) other_blocks<kMix>(win, it, mix, ph, s_other, wd.exactMinE, wd.exactMaxE);
        }
        __syncthreads();   // slot cur is free, slot cur ^ 1 is ready
    }
}

}  // namespace

namespace {

// The held-weights kernel serves windows of 16 lobes with a power-of-two table scale (what kaiser_sinc and the
// reference's own window give at 16 lobes) and the samples of held_sample; the rest take resample_kernel.
bool resample_held_ok(const ResampleWindowDev& w, bool magic, bool fma)
{
    return magic && fma && w.lobes == kHeldLobes &&
           resample_smem_floats(w, true, true) * sizeof(float) <= kPairTableLimit;
}

template <bool kMix>
void launch_held(Handle& h, const float* src, uint32_t srcStride, float* dst, uint32_t dstStride, int n,
                 const float* inRate, const float* outRate, const int* dims, const ResampleWindowDev& w,
                 bool normalize, int minBlocks, long long* held, long long* general, unsigned long long* next)
{
    const size_t smem = resample_smem_floats(w, true, true) * sizeof(float);   // the table and two spans
    static_assert(kWarps * 256 == 2 * kHeldSpan, "resample_smem_floats counts the spans");
    const int grid = persistent_grid(h, reinterpret_cast<const void*>(resample_held_kernel<kMix>), kHeldThreads, smem);
    resample_split_kernel<<<1, ragged_prefix_threads(n), 0, h.stream()>>>(inRate, outRate, dims, kMix, n, minBlocks, held,
                                                                          general, next);
    count_launch();
    check_cuda(cudaGetLastError(), "resample_split_kernel");
    launch_dependent(resample_held_kernel<kMix>, dim3(grid), dim3(kHeldThreads), smem, h.stream(),
                     "resample_held_kernel", src, srcStride, dst, dstStride, inRate, outRate, dims, w, normalize,
                     static_cast<const long long*>(held), next, n);
    count_launch();
}

}  // namespace

size_t resample_scratch_bytes(int n)
{
    Carver cv(nullptr);
    cv.take<long long>(n + 1);
    cv.take<long long>(n + 1);
    cv.take<unsigned long long>(1);
    return cv.used();
}

void launch_resample(Handle& h, void* scratch, const float* src, uint32_t srcStride, float* dst, uint32_t dstStride,
                     int n, const float* inRate, const float* outRate, const int* dims, const ResampleWindowDev& win,
                     int channels, bool downmix, bool normalize)
{
    if (n <= 0) return;
    Carver cv(scratch);
    long long* prefix = cv.take<long long>(n + 1);
    long long* heldPrefix = cv.take<long long>(n + 1);
    unsigned long long* next = cv.take<unsigned long long>(1);
    ResampleWindowDev w = win;
    resample_pads(w);
    const bool pairs = w.padLeft >= 0 && resample_smem_floats(w, true, downmix) * sizeof(float) <= kPairTableLimit;
    const size_t smem = resample_smem_floats(w, pairs, downmix) * sizeof(float);
    const bool magic = resample_magic_ok(w, pairs);
    const bool fma = resample_scale_pow2(w);
    resample_exact_range(w, magic, fma);
    // The held-weights kernel pays from one full item per CTA on, 4736 blocks at 2 CTAs per SM, 1.3 minutes at 16 kHz, and
    // from one and a half when it down-mixes (against resample_kernel, clips of mixed rates: mono 4236 blocks 34 and 35
    // us, 4926 35 and 39, 6895 41 and 50, 9064 44 and 62; stereo 4926 50 and 44 us, 6416 56 and 56, 7135 54 and 58, 9311
    // 67 and 76).  resample_split_kernel counts them; it and the second kernel cost 2 to 4 us, so batches that are below
    // four items per CTA when padded skip both.
    const long long padded = (long long)n * ((dstStride + kBlock - 1) / kBlock);
    const int items = kItemBlocks * kHeldCtas * h.num_sms();
    const int minBlocks = downmix ? items + items / 2 : items;
    const bool split = padded >= 4ll * items && (downmix || channels <= 1) && resample_held_ok(w, magic, fma);
    if (split)
    {
        auto held = downmix ? launch_held<true> : launch_held<false>;
        held(h, src, srcStride, dst, dstStride, n, inRate, outRate, dims, w, normalize, minBlocks, heldPrefix, prefix, next);
    }
    else
        launch_ragged_prefix(ResampleCount{inRate, outRate, dims, downmix, nullptr, 0.f}, n, prefix, h.stream());
    auto go = [&](auto kernel) {
        const int grid = persistent_grid(h, reinterpret_cast<const void*>(kernel), kThreads, smem);
        const long long* units = prefix;
        const RppbClip* clips = nullptr;
        if (split)   // starts while the held-weights kernel ends
            launch_dependent(kernel, dim3(grid), dim3(kThreads), smem, h.stream(), "resample_kernel", src, srcStride, dst,
                             dstStride, inRate, outRate, dims, w, normalize, units, n, clips, 0.f);
        else
            kernel<<<grid, kThreads, smem, h.stream()>>>(src, srcStride, dst, dstStride, inRate, outRate, dims, w,
                                                         normalize, units, n, clips, 0.f);
    };
    if (downmix && magic && fma) go(resample_kernel<true, false, true, true, true>);
    else if (downmix && magic) go(resample_kernel<true, false, true, true>);
    else if (downmix && pairs) go(resample_kernel<true, false, true>);
    else if (downmix) go(resample_kernel<true, false, false>);
    else if (magic && fma) go(resample_kernel<false, false, true, true, true>);
    else if (magic) go(resample_kernel<false, false, true, true>);
    else if (pairs) go(resample_kernel<false, false, true>);
    else go(resample_kernel<false, false, false>);
    count_launch();
    check_cuda(cudaGetLastError(), "resample_kernel");
}

void launch_resample_clips(Handle& h, void* scratch, const RppbClip* clips, int n, float outRate,
                           const ResampleWindowDev& win)
{
    if (n <= 0) return;
    long long* prefix = static_cast<long long*>(scratch);
    ResampleWindowDev w = win;
    resample_pads(w);
    const bool pairs = w.padLeft >= 0 && resample_smem_floats(w, true, false) * sizeof(float) <= kPairTableLimit;
    const size_t smem = resample_smem_floats(w, pairs, false) * sizeof(float);
    const bool magic = resample_magic_ok(w, pairs);
    const bool fma = resample_scale_pow2(w);
    resample_exact_range(w, magic, fma);
    launch_ragged_prefix(ResampleCount{nullptr, nullptr, nullptr, false, clips, outRate}, n, prefix, h.stream());
    auto go = [&](auto kernel) {
        const int grid = persistent_grid(h, reinterpret_cast<const void*>(kernel), kThreads, smem);
        kernel<<<grid, kThreads, smem, h.stream()>>>(nullptr, 0, nullptr, 0, nullptr, nullptr, nullptr, w, false,
                                                     prefix, n, clips, outRate);
    };
    if (magic && fma) go(resample_kernel<false, true, true, true, true>);
    else if (magic) go(resample_kernel<false, true, true, true>);
    else if (pairs) go(resample_kernel<false, true, true>);
    else go(resample_kernel<false, true, false>);
    count_launch();
    check_cuda(cudaGetLastError(), "resample_kernel(clips)");
}

}  // namespace rppb
