// non_silent_region_detection.
//
// Reference: src/modules/tensor/cpu/kernel/non_silent_region_detection.cpp:105-184.  The
// moving mean square (MMS) is a float running sum of squares, restarted every resetInterval
// samples (-1: once per sample) from a fresh sum over the preceding window; the sample's cutoff
// is (referencePower, or the maximum MMS when that is 0) * 10^(cutOffDB/10); the region runs
// from the first to the last MMS at or above the cutoff, its begin moved back by
// windowLength - 1 (clamped at 0); no such MMS gives (0, 0).
//
// The running sum is a dependent float chain of resetInterval + windowLength steps per reset block, and
// its rounding decides the integers wherever an MMS is close to the cutoff.  It need not be replayed
// where it is not close: the true window energies, in FP64, and a bound on the chain's rounding give an
// interval for every MMS and for the cutoff, and the region's ends follow from the intervals unless the
// first (last) candidate's interval meets the cutoff's.  Only then is that candidate's reset block
// replayed, in exactly the reference's order (add the new square, store sum * (1/windowLength), subtract
// the square leaving the window; explicit round-to-nearest intrinsics, no FMA), and, if its exact values
// lie inside the cutoff's interval too, the blocks that may hold the maximum.  Begin and length are
// therefore the host path's on every input.
//   1. energy_kernel: FP64 energies of 64-sample chunks, one streaming pass over the signal (HBM-bound: 31 us
//      for 256 clips of 1 to 16 s, 4.6 TB/s);
//   2. region_kernel: one CTA per sample: scan of the energies, cutoff interval, both ends, replays (15 to
//      20 us without a replay, 73 us with one).
// A clip that ends in silence after sound within one reset block needs a replay as a rule: its running
// sum decays to rounding residue, which no bound can place against the cutoff.  The bare chain is
// latency-bound (8 cycles per sample, 38 us for a block of 8192 with a window of 2048).
// Replaying every block, which this replaces, took 172 us and the search through its stored values 118 us
// on the same batch (288 us per call; now 104 us).
#include <cfloat>
#include <climits>

#include "common.cuh"
#include "ops.hpp"

namespace rppb {
namespace {

constexpr int kThreads = 256;
constexpr int kSub = 64;                       // samples per energy chunk
constexpr int kUnit = kThreads / 32 * 1024;    // samples per CTA step of the energy pass
constexpr int kChains = 8;                     // reset blocks replayed side by side, one per lane of warp 0
constexpr int kTile = 256;                     // samples of each block per replay step
constexpr int kPitch = kTile + 4;              // the 8 chain lanes' 16-byte reads fall in distinct banks
constexpr size_t kReplayBytes = size_t(2) * 3 * kChains * kPitch * sizeof(float);
constexpr int kRun = 1024, kRuns = 512;        // largest_window: samples per run, runs whose maxima are kept
constexpr int kScan = 16;                      // chunks per thread and step of the scan of the energies
constexpr int kHeld = kScan * kThreads;        // prefix energies kept in shared memory until the first replay
static_assert(kReplayBytes >= (kHeld + 1) * sizeof(double), "the replay buffers hold the prefix energies first");
constexpr double kUlp = 1.0 / 16777216.0;      // 2^-24: relative rounding error of a float operation

__device__ __forceinline__ float sq(float v) { return __fmul_rn(v, v); }

// energies[b * pitch + c] = sum of the float-rounded squares of samples [64 c, 64 c + 64) of sample b.
// A warp takes 1024 samples: 8 four-sample loads per lane in flight, then a reduction over each half
// warp that halves the number of values a lane carries at every step (8 FP64 shuffles for 16 chunks).
__global__ void __launch_bounds__(kThreads) energy_kernel(const float* __restrict__ src, uint32_t stride,
                                                          const int* __restrict__ len, double* __restrict__ energies,
                                                          long long pitch, int n, int unitsPerSample)
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
    const long long units = (long long)n * unitsPerSample;
    for (long long w = blockIdx.x; w < units; w += gridDim.x)
    {
        const int b = int(w / unitsPerSample);
        const long long i0 = (w - (long long)b * unitsPerSample) * kUnit + wi * 1024;
        const long long L = min(*RPPB_RD(len + b), int(stride));
        if (i0 >= L) continue;
        const float* x = src + size_t(b) * stride + i0;
        const int left = int(min(L - i0, 1024ll));   // samples of this warp's 1024 that exist
        const bool vec = (reinterpret_cast<uintptr_t>(x) & 15) == 0;
        float4 v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j)
        {
            const int i = 128 * j + 4 * lane;
            v[j] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (vec && i + 4 <= left) v[j] = __ldg(RPPB_RD(reinterpret_cast<const float4*>(x + i)));
            else
            {
                if (i < left) v[j].x = __ldg(RPPB_RD(x + i));
                if (i + 1 < left) v[j].y = __ldg(RPPB_RD(x + (i + 1)));
                if (i + 2 < left) v[j].z = __ldg(RPPB_RD(x + (i + 2)));
                if (i + 3 < left) v[j].w = __ldg(RPPB_RD(x + (i + 3)));
            }
        }
        double s[8];
#pragma unroll
        for (int j = 0; j < 8; ++j)
            s[j] = (double(sq(v[j].x)) + double(sq(v[j].y))) + (double(sq(v[j].z)) + double(sq(v[j].w)));
        // load j of the lanes of half h covers chunk 2 j + h
#pragma unroll
        for (int m = 8, k = 4; m >= 2; m >>= 1, k >>= 1)
        {
            const bool up = lane & m;
#pragma unroll
            for (int q = 0; q < k; ++q)
            {
                const double send = up ? s[q] : s[q + k], keep = up ? s[q + k] : s[q];
                s[q] = keep + __shfl_xor_sync(0xffffffffu, send, m);
            }
        }
        s[0] += __shfl_xor_sync(0xffffffffu, s[0], 1);
        const int c = 2 * ((lane >> 1) & 7) + (lane >> 4);   // bits 3, 2, 1 of the lane chose j
        if (!(lane & 1) && c * kSub < left) *RPPB_WR(energies + (b * pitch + i0 / kSub + c)) = s[0];
    }
}

// What the CTA of region_kernel shares.
struct RegionShared
{
    double warp[kThreads / 32], warp2[kThreads / 32];
    double sums[3 * kSub];               // running sums of squares within the chunks a window enters and leaves
    float run[kRuns];                    // largest window energy of each run
    int hit, sure;
    int list[kChains];                   // blocks to replay
    // per replayed block: first and last index at or above the cutoff interval's low end (with the MMS
    // there in the low word; last: index + 1) and its high end
    unsigned long long firstLow[kChains], lastLow[kChains];
    int firstHigh[kChains], lastHigh[kChains];
    unsigned peak[kChains];              // float_key of the largest MMS
    __device__ __forceinline__ int low_index(int j, bool last) const
    {
        return last ? int(lastLow[j] >> 32) - 1 : int(firstLow[j] >> 32) & INT_MAX;
    }
};

// One sample and its parameters.
struct Clip
{
    const float* x;
    int L, W, R;          // samples, window, reset block
    float meanFactor;
    const double* P;      // P[c] = energy of chunks 0 .. c - 1: the copy in shared memory or `all`
    const double* all;
    int chunks;
    double slack;         // absolute error of a difference of two entries of P
    double top;           // upper bound of every window energy
    __device__ __forceinline__ int pre(int st) const { return max(st - W + 1, 0); }
    __device__ __forceinline__ double prefix(int c) const { return *RPPB_RD(P + c); }
    // every window ending in chunk c lies inside these chunks
    __device__ __forceinline__ double upper(int c) const
    {
        const int o = c * kSub - W + 1;
        return prefix(c + 1) - prefix(o > 0 ? o / kSub : 0);
    }
    // the window ending with chunk c holds these chunks (and nothing else when W is a multiple of kSub)
    __device__ __forceinline__ double attained(int c) const
    {
        const int o = (c + 1) * kSub - W;
        return prefix(c + 1) - prefix(o > 0 ? (o + kSub - 1) / kSub : 0);
    }
    // Rounding of the running sum after `ops` additions and subtractions: each errs by at most 2^-24 of
    // its result, which is at most a window energy, and at most the energy seen since the fresh sum began
    // (1/16 for the growth of the error itself: ops * 2^-24 <= 1/16).
    __device__ __forceinline__ double rounding(double ops, double seen) const
    {
        return ops * (kUlp * 1.0625) * fmin(seen, top) + slack;
    }
    // upper bound of the running sums of chunk c
    __device__ __forceinline__ double chunk_high(int c) const
    {
        const int st = c * kSub / R * R;
        return upper(c) + rounding(W + 2.0 * ((c + 1) * kSub - st), prefix(c + 1) - prefix(pre(st) / kSub));
    }
};

// Replays the `m` reset blocks of sh.list exactly and fills sh's results for the cutoff interval
// [low, high].  Lane j of warp 0 runs block j's chain from squares that the other seven warps stage in
// shared memory one tile ahead; they also compare the MMS values one tile behind.  A square of zero
// stands for "nothing enters / leaves": sum + 0 and sum - 0 == sum exactly.
__device__ void replay(Clip& clip, RegionShared& sh, float* buf, int m, double low, double high)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    auto row = [&](int slot, int what, int j) { return buf + ((slot * 3 + what) * kChains + j) * kPitch; };
    auto start = [&](int j) { return sh.list[j] * clip.R; };
    auto end = [&](int st) { return int(min((long long)clip.L, (long long)st + clip.R)); };
    clip.P = clip.all;   // the buffers below take the place of the copy in shared memory
    if (threadIdx.x < kChains)
    {
        sh.firstLow[threadIdx.x] = ~0ull;
        sh.lastLow[threadIdx.x] = 0ull;
        sh.firstHigh[threadIdx.x] = INT_MAX;
        sh.lastHigh[threadIdx.x] = -1;
        sh.peak[threadIdx.x] = float_key(-FLT_MAX);
    }
    if (threadIdx.x < m)   // the block's samples, ahead of the staging
    {
        const int st = start(threadIdx.x);
        l2_prefetch(clip.x + clip.pre(st), clip.x + end(st));
    }
    __syncthreads();
    int preMax = 0, blkMax = 0;
    for (int j = 0; j < m; ++j)
    {
        const int st = start(j);
        preMax = max(preMax, st - clip.pre(st));
        blkMax = max(blkMax, end(st) - st);
    }
    const int preTiles = (preMax + kTile - 1) / kTile, tiles = preTiles + (blkMax + kTile - 1) / kTile;
    float sum = 0.0f;
    for (int it = 0; it < tiles + 2; ++it)
    {
        if (warp == 0)
        {
            const int t = it - 1, slot = t & 1;
            if (t >= 0 && t < tiles && lane < m)
            {
                const float* in = row(slot, 0, lane);
                if (t < preTiles)
                {
#pragma unroll 8
                    for (int k = 0; k < kTile; k += 4)
                    {
                        const float4 a = *reinterpret_cast<const float4*>(in + k);
                        sum = __fadd_rn(sum, a.x);
                        sum = __fadd_rn(sum, a.y);
                        sum = __fadd_rn(sum, a.z);
                        sum = __fadd_rn(sum, a.w);
                    }
                }
                else
                {
                    const float* out = row(slot, 1, lane);
                    float* val = row(slot, 2, lane);
#pragma unroll 8
                    for (int k = 0; k < kTile; k += 4)
                    {
                        const float4 a = *reinterpret_cast<const float4*>(in + k);
                        const float4 o = *reinterpret_cast<const float4*>(out + k);
                        float4 v;
                        sum = __fadd_rn(sum, a.x);
                        v.x = __fmul_rn(sum, clip.meanFactor);
                        sum = __fsub_rn(sum, o.x);
                        sum = __fadd_rn(sum, a.y);
                        v.y = __fmul_rn(sum, clip.meanFactor);
                        sum = __fsub_rn(sum, o.y);
                        sum = __fadd_rn(sum, a.z);
                        v.z = __fmul_rn(sum, clip.meanFactor);
                        sum = __fsub_rn(sum, o.z);
                        sum = __fadd_rn(sum, a.w);
                        v.w = __fmul_rn(sum, clip.meanFactor);
                        sum = __fsub_rn(sum, o.w);
                        *reinterpret_cast<float4*>(val + k) = v;
                    }
                }
            }
        }
        else
        {
            const int first = threadIdx.x - 32, step = kThreads - 32, count = m * kTile;
            if (it < tiles)
            {
                const int slot = it & 1;
#pragma unroll 2
                for (int e = first; e < count; e += step)
                {
                    const int j = e / kTile, t = e % kTile, st = start(j);
                    if (it < preTiles)
                    {
                        const int i = clip.pre(st) + it * kTile + t;
                        row(slot, 0, j)[t] = i < st ? sq(__ldg(RPPB_RD(clip.x + i))) : 0.0f;
                    }
                    else
                    {
                        const long long i = (long long)st + (it - preTiles) * kTile + t;
                        const long long o = i - clip.W + 1;
                        const bool live = i < end(st);
                        row(slot, 0, j)[t] = live ? sq(__ldg(RPPB_RD(clip.x + i))) : 0.0f;
                        row(slot, 1, j)[t] = live && o >= 0 ? sq(__ldg(RPPB_RD(clip.x + o))) : 0.0f;
                    }
                }
            }
            const int done = it - 2;
            if (done >= preTiles)
            {
                // a warp's 32 consecutive values belong to one block (kTile and the step are multiples of 32)
                for (int e = first; e < count; e += step)
                {
                    const int j = e / kTile, t = e % kTile;
                    const long long i = (long long)start(j) + (done - preTiles) * kTile + t;
                    const bool live = i < end(start(j));
                    const float v = live ? row(done & 1, 2, j)[t] : -FLT_MAX;
                    const unsigned atLow = __ballot_sync(0xffffffffu, live && double(v) >= low);
                    const unsigned atHigh = __ballot_sync(0xffffffffu, live && double(v) >= high);
                    const float mx = warp_max(fmaxf(-FLT_MAX, v));
                    const unsigned long long bits = __float_as_uint(v);
                    const unsigned long long at = (unsigned long long)(i);
                    if (lane == __ffs(atLow) - 1) atomicMin(&sh.firstLow[j], at << 32 | bits);
                    if (lane == 31 - __clz(atLow)) atomicMax(&sh.lastLow[j], (at + 1) << 32 | bits);
                    if (lane == 0)
                    {
                        atomicMax(&sh.peak[j], float_key(mx));
                        if (atHigh)
                        {
                            atomicMin(&sh.firstHigh[j], int(i) + __ffs(atHigh) - 1);
                            atomicMax(&sh.lastHigh[j], int(i) + 31 - __clz(atHigh));
                        }
                    }
                }
            }
        }
        __syncthreads();
    }
}

constexpr int kNone = -1;        // no MMS reaches the cutoff
constexpr int kUnsettled = -2;   // an exact MMS lies inside the cutoff's interval
constexpr int kGiveUp = -3;      // too many candidates: replay everything

// An exact MMS inside the cutoff's interval: the first (last) one at or above its low end.
struct Open
{
    int index;
    float value;
};

// The first (kLast: last) index whose MMS is at or above the cutoff, known to lie in [low, high].
template <bool kLast>
__device__ int find_end(Clip& clip, RegionShared& sh, float* buf, double low, double high, Open& open)
{
    constexpr int kMiss = kLast ? -1 : INT_MAX;
    constexpr double kRel = 4.0 * kUlp;   // the product with meanFactor
    const int tid = threadIdx.x, lane = tid & 31;
    const double mf = clip.meanFactor;
    int edge = kLast ? clip.L - 1 : 0;    // every index before (after) it is below the cutoff
    int replays = 0;
    for (int looks = 0; looks < 64; ++looks)
    {
        // the next chunk that may reach the cutoff
        int c = kMiss;
        for (int c0 = edge / kSub; kLast ? c0 >= 0 : c0 < clip.chunks; c0 += kLast ? -kThreads : kThreads)
        {
            const int k = kLast ? c0 - tid : c0 + tid;
            const bool may = k >= 0 && k < clip.chunks && clip.chunk_high(k) * mf * (1.0 + kRel) >= low;
            __syncthreads();   // the previous step's sh.hit has been read
            if (tid == 0) sh.hit = kMiss;
            __syncthreads();
            if (may)
            {
                if (kLast) atomicMax(&sh.hit, k);
                else atomicMin(&sh.hit, k);
            }
            __syncthreads();
            c = sh.hit;
            if (c != kMiss) break;
        }
        if (c == kMiss) return kNone;
        // its samples' window energies: the prefix energies plus single squares at both ends.  sums holds
        // the running sums of the squares of chunk c and of the two chunks its windows leave, 32 at a time
        const int base = c * kSub, o0 = base - clip.W + 1;
        const int lead = o0 >= 0 ? o0 / kSub : -((kSub - 1 - o0) / kSub);   // floor
        __syncthreads();
        if (tid < 3 * kSub)
        {
            const long long i = tid < kSub ? base + tid : (long long)lead * kSub + (tid - kSub);
            double q = i >= 0 && i < clip.L ? double(sq(__ldg(RPPB_RD(clip.x + i)))) : 0.0;
#pragma unroll
            for (int t = 1; t < 32; t <<= 1)
            {
                const double u = __shfl_up_sync(0xffffffffu, q, t);
                if (lane >= t) q += u;
            }
            sh.sums[tid] = q;
        }
        if (tid == 0)
        {
            sh.hit = kMiss;
            sh.sure = 0;
        }
        __syncthreads();
        // sum of the first k squares of the chunk whose sums start at s (0 <= k <= kSub)
        auto head = [&](int s, int k) {
            return k == 0 ? 0.0 : sh.sums[s + k - 1] + (k > 32 ? sh.sums[s + 31] : 0.0);
        };
        bool sure = false;
        const int i = base + tid;
        const bool asked = tid < kSub && i < clip.L && (kLast ? i <= edge : i >= edge);
        if (asked)
        {
            const double upTo = clip.prefix(c) + head(0, tid + 1);
            const int o = i - clip.W + 1;   // samples before o have left
            const double gone = o > 0 ? clip.prefix(o / kSub) + head(kSub + (o / kSub - lead) * kSub, o % kSub) : 0.0;
            const int st = i / clip.R * clip.R, pre = clip.pre(st);
            const double e = clip.rounding((st - pre) + 2.0 * (i - st) + 1.0, upTo - clip.prefix(pre / kSub) + clip.slack);
            const double sum = upTo - gone;
            sure = (sum - e) * mf * (1.0 - kRel) >= high;
            if ((sum + e) * mf * (1.0 + kRel) >= low)
            {
                if (kLast) atomicMax(&sh.hit, i);
                else atomicMin(&sh.hit, i);
            }
        }
        __syncthreads();
        const int at = sh.hit;
        if (asked && i == at && sure) sh.sure = 1;
        __syncthreads();
        if (at == kMiss)
        {
            edge = kLast ? base - 1 : base + kSub;
            if (edge < 0 || edge >= clip.L) return kNone;
            continue;
        }
        if (sh.sure) return at;
        // undecided: the exact values of that sample's block
        if (++replays > 2) return kGiveUp;
        const int k = at / clip.R;
        if (tid == 0) sh.list[0] = k;
        __syncthreads();
        replay(clip, sh, buf, 1, low, high);
        const bool any = sh.lastLow[0] != 0ull;
        const int lo = sh.low_index(0, kLast), hi = kLast ? sh.lastHigh[0] : sh.firstHigh[0];
        open.index = lo;
        open.value = __uint_as_float(unsigned(kLast ? sh.lastLow[0] : sh.firstLow[0]));
        __syncthreads();
        if (any) return lo == hi ? lo : kUnsettled;
        const long long next = kLast ? (long long)k * clip.R - 1 : (long long)(k + 1) * clip.R;
        if (next < 0 || next >= clip.L) return kNone;
        edge = int(next);
    }
    return kGiveUp;
}

// The largest window energy to within 1e-5 of clip.top, for clips whose replayed values fall inside the
// cutoff's interval: the chunks bound it to 3 % (64 samples of 2048).  Each warp takes 128 samples at a
// time, wherever the chunks allow a window of at least `least`: the window energy before them plus the
// running sum of the squares entering less those leaving (in float; the steps are independent).
// sh.run[r] = the largest of run r (kRuns runs at most).
__device__ double largest_window(const Clip& clip, RegionShared& sh, double least)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    auto square = [&](long long i) { return i >= 0 && i < clip.L ? sq(__ldg(RPPB_RD(clip.x + i))) : 0.0f; };
    for (int r = threadIdx.x; r < kRuns; r += kThreads) sh.run[r] = 0.0f;
    __syncthreads();
    float best = 0.0f;
    for (int c = 2 * warp; c < clip.chunks; c += 2 * (kThreads / 32))
    {
        if (clip.upper(c) < least && (c + 1 >= clip.chunks || clip.upper(c + 1) < least)) continue;
        const int s = c * kSub, o = s - clip.W;
        float before = 0.0f;
        if (o > 0)
        {
            const int c0 = o / kSub * kSub;
            float part = c0 + lane < o ? square(c0 + lane) : 0.0f;
            if (c0 + 32 + lane < o) part += square(c0 + 32 + lane);
#pragma unroll
            for (int t = 16; t > 0; t >>= 1) part += __shfl_xor_sync(0xffffffffu, part, t);
            before = float(clip.prefix(c) - clip.prefix(o / kSub) - double(part));
        }
        else
            before = float(clip.prefix(c));
        const long long i = s + 4 * lane;
        float d[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) d[q] = square(i + q) - square(i + q - clip.W);
        const float mine = (d[0] + d[1]) + (d[2] + d[3]);
        float at = mine;
#pragma unroll
        for (int t = 1; t < 32; t <<= 1)
        {
            const float u = __shfl_up_sync(0xffffffffu, at, t);
            if (lane >= t) at += u;
        }
        float w = before + (at - mine), peak = 0.0f;
#pragma unroll
        for (int q = 0; q < 4; ++q)
        {
            w += d[q];
            if (i + q < clip.L) peak = fmaxf(peak, w);
        }
        peak = warp_max(peak);
        if (lane == 0 && s / kRun < kRuns)
            atomicMax(reinterpret_cast<int*>(&sh.run[s / kRun]), __float_as_int(peak));   // not negative
        best = fmaxf(best, peak);
    }
    if (lane == 0) sh.warp[warp] = best;
    __syncthreads();
    double all = 0.0;
    for (int w = 0; w < kThreads / 32; ++w) all = fmax(all, sh.warp[w]);
    __syncthreads();
    return all;
}

// The largest MMS, by replaying the blocks that `may(k)` (uniform over the CTA) admits.
template <class May>
__device__ float exact_peak(Clip& clip, RegionShared& sh, float* buf, int blocks, May may)
{
    float peak = -FLT_MAX;
    int m = 0;
    for (int k = 0; k <= blocks; ++k)
    {
        if (k < blocks && may(k))
        {
            if (threadIdx.x == 0) sh.list[m] = k;
            ++m;
        }
        if (m == kChains || (k == blocks && m > 0))
        {
            __syncthreads();
            replay(clip, sh, buf, m, double(INFINITY), double(INFINITY));
            for (int j = 0; j < m; ++j) peak = fmaxf(peak, key_float(sh.peak[j]));
            __syncthreads();
            m = 0;
        }
    }
    return peak;
}

// Both ends by replaying blocks from either side until one reaches the exact cutoff.
__device__ void replay_ends(Clip& clip, RegionShared& sh, float* buf, int blocks, double cut, int& first, int& last)
{
    first = last = -1;
    for (int dir = 0; dir < 2; ++dir)
        for (int g = 0; g < blocks; g += kChains)
        {
            const int m = min(kChains, blocks - g);
            if (threadIdx.x < m) sh.list[threadIdx.x] = dir ? blocks - 1 - g - int(threadIdx.x) : g + int(threadIdx.x);
            __syncthreads();
            replay(clip, sh, buf, m, cut, cut);
            int at = -1;
            for (int j = 0; j < m && at < 0; ++j)
                if (sh.lastLow[j] != 0ull) at = sh.low_index(j, dir != 0);
            __syncthreads();
            if (at < 0) continue;
            (dir ? last : first) = at;
            break;
        }
}

__global__ void __launch_bounds__(kThreads) region_kernel(const float* __restrict__ src, uint32_t stride,
                                                          const int* __restrict__ len, int windowLength, int reset,
                                                          float referencePower, float cutOff, double* __restrict__ energies,
                                                          long long pitch, int* __restrict__ outBegin,
                                                          int* __restrict__ outLength)
{
    // kReplayBytes: the prefix energies, then squares entering, squares leaving and MMS in two slots
    extern __shared__ __align__(16) float buf[];
    __shared__ RegionShared sh;
    const int b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int L = min(*RPPB_RD(len + b), int(stride));
    grid_dependency_wait();   // the chunk energies
    if (L <= 0)
    {
        if (tid == 0)
        {
            *RPPB_WR(outBegin + b) = 0;
            *RPPB_WR(outLength + b) = 0;
        }
        return;
    }
    double* P = dependency_result(energies) + b * pitch;
    double* held = reinterpret_cast<double*>(buf);
    Clip clip{src + size_t(b) * stride, L, windowLength, reset == -1 ? L : reset,
              __fdiv_rn(1.0f, float(windowLength)), P, P, (L + kSub - 1) / kSub, 0.0, 0.0};
    const int blocks = int(((long long)L + clip.R - 1) / clip.R);

    // energies -> prefix energies, in place: a warp takes kScan rows of 32 chunks, which it scans side by side
    double total = 0.0;
    for (int c0 = 0; c0 < clip.chunks; c0 += kHeld)
    {
        const int w0 = c0 + warp * kScan * 32 + lane;
        double e[kScan], incl[kScan];
#pragma unroll
        for (int k = 0; k < kScan; ++k) incl[k] = e[k] = w0 + 32 * k < clip.chunks ? *RPPB_RD(P + (w0 + 32 * k)) : 0.0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
#pragma unroll
            for (int k = 0; k < kScan; ++k)
            {
                const double t = __shfl_up_sync(0xffffffffu, incl[k], o);
                if (lane >= o) incl[k] += t;
            }
        double rows = 0.0;
#pragma unroll
        for (int k = 0; k < kScan; ++k)
        {
            const double t = __shfl_sync(0xffffffffu, incl[k], 31);
            incl[k] += rows - e[k];   // before chunk k, within the warp's rows
            rows += t;
        }
        if (lane == 0) sh.warp[warp] = rows;
        __syncthreads();
        double before = total;
#pragma unroll
        for (int w = 0; w < kThreads / 32; ++w)
        {
            if (w < warp) before += sh.warp[w];
            total += sh.warp[w];
        }
#pragma unroll
        for (int k = 0; k < kScan; ++k)
            if (w0 + 32 * k < clip.chunks)
            {
                *RPPB_WR(P + (w0 + 32 * k)) = before + incl[k];
                if (c0 == 0) held[w0 + 32 * k] = before + incl[k];
            }
        __syncthreads();
    }
    if (tid == 0)
    {
        *RPPB_WR(P + clip.chunks) = total;
        if (clip.chunks <= kHeld) held[clip.chunks] = total;
    }
    if (clip.chunks <= kHeld) clip.P = held;
    __syncthreads();

    int first = -1, last = -1;
    const bool peakRef = referencePower == 0.0f;
    const double ops = double(windowLength) + 2.0 * double(min(clip.R, L));
    // Intervals help where the chunks resolve the window, the chain's rounding bound is small and every
    // number is a normal one; elsewhere (and when they do not settle the ends) every block is replayed.
    bool full = !(total <= 1e37) || windowLength < 4 * kSub || clip.R < kSub || ops * kUlp > 1.0 / 16;
    if (total == 0.0)
    {
        // every square is zero and so is every MMS
        if (0.0f >= __fmul_rn(peakRef ? 0.0f : referencePower, cutOff))
        {
            first = 0;
            last = L - 1;
        }
        full = false;
    }
    else if (!full)
    {
        double hi = 0.0, lo = 0.0;
        for (int c = tid; c < clip.chunks; c += kThreads)
        {
            hi = fmax(hi, clip.upper(c));
            lo = fmax(lo, clip.attained(c));
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
        {
            hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
            lo = fmax(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        }
        if (lane == 0)
        {
            sh.warp[warp] = hi;
            sh.warp2[warp] = lo;
        }
        __syncthreads();
#pragma unroll
        for (int w = 0; w < kThreads / 32; ++w)
        {
            hi = fmax(hi, sh.warp[w]);
            lo = fmax(lo, sh.warp2[w]);
        }
        __syncthreads();
        clip.slack = total * (1e-13 + 1e-17 * clip.chunks);
        clip.top = hi + clip.slack;
        const double err = clip.rounding(ops, clip.top), mf = clip.meanFactor;
        double peakLow = lo - err, low, high;   // peakLow: of the running sums
        auto cutoff_interval = [&](double peakHigh) {
            low = high = double(__fmul_rn(referencePower, cutOff));
            if (!peakRef) return;
            low = peakLow * mf * double(cutOff) * (1.0 - 1e-6);
            high = peakHigh * mf * double(cutOff) * (1.0 + 1e-6);
        };
        cutoff_interval(clip.top + err);
        if (!(low > 1e-30) || !(high < 1e37)) full = true;
        else
        {
            // 0: the interval the chunks give, 1: a tighter one, 2: the exact cutoff
            for (int stage = 0;; ++stage)
            {
                Open open{};
                if (first < 0) first = find_end<false>(clip, sh, buf, low, high, open);
                last = first < 0 ? first : find_end<true>(clip, sh, buf, low, high, open);
                if (last != kUnsettled || !peakRef || stage == 2) break;
                if (stage == 0)
                {
                    const double tol = 1e-5 * clip.top;
                    const double peak = largest_window(clip, sh, lo - clip.slack - 2.0 * (err + tol));
                    peakLow = peak - tol - err;
                    cutoff_interval(peak + tol + err);
                }
                else
                {
                    // from the blocks whose energies allow the maximum
                    const float peak = exact_peak(clip, sh, buf, blocks, [&](int k) {
                        const int st = k * clip.R, en = int(min((long long)L, (long long)st + clip.R));
                        bool any = false;
                        for (int r = st / kRun + tid; r <= (en - 1) / kRun; r += kThreads)
                            any = any || r >= kRuns || sh.run[r] + 1e-5 * clip.top + err >= peakLow;
                        return __syncthreads_or(any) != 0;
                    });
                    low = high = double(__fmul_rn(peak, cutOff));
                }
                if (double(open.value) < high) continue;
                // the open value is the end: everything before (after) it is below the interval's old low end
                if (first >= 0)
                {
                    last = open.index;
                    break;
                }
                first = open.index;
            }
            full = first < kNone || last < kNone;
        }
    }
    if (full)
    {
        float base = referencePower;
        if (peakRef) base = exact_peak(clip, sh, buf, blocks, [](int) { return true; });
        replay_ends(clip, sh, buf, blocks, double(__fmul_rn(base, cutOff)), first, last);
    }
    if (tid == 0)
    {
        int detectBegin = 0, detectLength = 0;
        if (first >= 0)
        {
            detectBegin = first;
            detectLength = last - first + 1;
            if (detectBegin != 0 && detectLength != 0)
            {
                const int newBegin = max(detectBegin - (windowLength - 1), 0);
                detectLength += detectBegin - newBegin;
                detectBegin = newBegin;
            }
        }
        *RPPB_WR(outBegin + b) = detectBegin;
        *RPPB_WR(outLength + b) = detectLength;
    }
}

// prefix energies per sample: one more entry than chunks
long long energy_pitch(uint32_t srcStride) { return (long long)(srcStride / kSub) + 2; }

}  // namespace

size_t nsr_scratch_bytes(int n, uint32_t srcStride)
{
    Carver cv(nullptr);
    cv.take<double>(size_t(n) * energy_pitch(srcStride));
    return cv.used();
}

void launch_nsr(Handle& h, void* scratch, const NsrArgs& a)
{
    if (a.n <= 0) return;
    Carver cv(scratch);
    const long long pitch = energy_pitch(a.srcStride);
    double* energies = cv.take<double>(size_t(a.n) * pitch);
    const int ups = int(a.srcStride / kUnit) + 1;
    const long long units = (long long)a.n * ups;
    const int grid = int(std::min<long long>(
        units, persistent_grid(h, reinterpret_cast<const void*>(energy_kernel), kThreads, 0)));
    energy_kernel<<<grid, kThreads, 0, h.stream()>>>(a.src, a.srcStride, a.len, energies, pitch, a.n, ups);
    count_launch();
    check_cuda(cudaGetLastError(), "energy_kernel");
    persistent_grid(h, reinterpret_cast<const void*>(region_kernel), kThreads, kReplayBytes);   // shared-memory opt-in
    launch_dependent(region_kernel, dim3(a.n), dim3(kThreads), kReplayBytes, h.stream(), "region_kernel", a.src,
                     a.srcStride, a.len, a.windowLength, a.resetInterval, a.referencePower, a.cutOff, energies, pitch,
                     a.begin, a.length);
    count_launch();
}

}  // namespace rppb
