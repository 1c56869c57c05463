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
// lie inside the cutoff's interval too, the blocks that may hold the maximum.  Clips that this does not settle have
// every block replayed, and many short ones have from the start (nsr_stored.cu).  Begin and length are
// therefore the host path's on every input.
//   1. energy_kernel: FP64 energies of 64-sample chunks, one streaming pass over the signal (HBM-bound: 30 us
//      for 256 clips of 1 to 16 s, 4.6 TB/s);
//   2. region_kernel: one CTA per sample: scan of the energies, cutoff interval, both ends, replays (15 to
//      20 us without a replay, about 45 us more for each one);
//   3. exact_kernel: the reset blocks of the samples that are left, over the whole GPU (2 us with none).
// A clip that ends in silence after sound within one reset block needs a replay as a rule: its running
// sum decays to rounding residue, which no bound can place against the cutoff.  The bare chain is
// latency-bound (8 cycles per sample, 38 us for a block of 8192 with a window of 2048).
// Replaying every block of every clip and searching the stored values, as an earlier version did, took 271 to 303 us per
// call on this batch; now 52 us where no clip needs a replay, 92 to 147 us, over eight signals, where most do.
// Where every block is replayed (the rule in launch_nsr and region_kernel's `full`) the call costs, against that
// version: the same batch with a window of 200 193 for 376 us, 512 clips of 10 s with a window of 16 267 for 497 us, 10
// minutes in one clip with a window of 200 116 for 167 us and without resets 101 for 113 ms; the blocks replayed by
// each clip's own CTA took 1322, 2047 and 30703 us and 174 ms.
#include <cfloat>
#include <climits>

#include "common.cuh"
#include "ops.hpp"

namespace rppb {
namespace {

constexpr int kThreads = 256;
constexpr int kSub = 64;                       // samples per energy chunk
constexpr int kUnit = kThreads / 32 * 1024;    // samples per CTA step of the energy pass
// A replay: reset blocks side by side (a lane of warp 0 each), samples of each block per step, and the pitch of a row
// of them, at which the lanes' 16-byte reads, up to 8 samples past the row, fall in distinct banks.
template <int CHAINS, int TILE>
struct ReplayShape
{
    static constexpr int kChains = CHAINS, kTile = TILE, kPitch = TILE + 12;
    static constexpr int kStagers = kThreads / 32 - 1;                    // warps that stage
    static constexpr int kRows = (CHAINS + kStagers - 1) / kStagers;     // blocks per staging warp
    static constexpr size_t kBytes = size_t(2) * 3 * CHAINS * kPitch * sizeof(float);
};
using OneShape = ReplayShape<kThreads / 32 - 1, 256>;    // region_kernel: one block, seldom a few
using ManyShape = ReplayShape<28, 128>;                  // exact_kernel: two CTAs per SM
constexpr int kRun = 1024, kRuns = 512;        // largest_window: samples per run, runs whose maxima are kept
constexpr int kSearch = 1024;                  // chunks that largest_window searches at most (50 us; giving up costs 100)
constexpr double kLongChain = 49152.0;         // operations of a reset block's chain from which region_kernel replays none
constexpr int kTallyShift = 36;                // ExactList::tally: clips above, reset blocks (2^36: 256 GB of floats) below
constexpr int kMaxClips = 1 << 27;             // per launch
constexpr int kScan = 16;                      // chunks per thread and step of the scan of the energies
constexpr int kHeld = kScan * kThreads;        // prefix energies kept in shared memory until the first replay
static_assert(OneShape::kBytes >= (kHeld + 1) * sizeof(double), "the replay buffers hold the prefix energies first");
constexpr double kUlp = 1.0 / 16777216.0;      // 2^-24: relative rounding error of a float operation

__device__ __forceinline__ float sq(float v) { return __fmul_rn(v, v); }

// energies[b * pitch + c] = sum of the float-rounded squares of samples [64 c, 64 c + 64) of sample b.
// A warp takes 1024 samples: 8 four-sample loads per lane in flight, then a reduction over each half
// warp that halves the number of values a lane carries at every step (8 FP64 shuffles for 16 chunks).
__global__ void __launch_bounds__(kThreads) energy_kernel(const float* __restrict__ src, uint32_t stride,
                                                          const int* __restrict__ len, double* __restrict__ energies,
                                                          long long pitch, int n, int unitsPerSample,
                                                          unsigned long long* __restrict__ tally)
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (blockIdx.x == 0 && threadIdx.x < 2) *RPPB_WR(tally + threadIdx.x) = 0ull;
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

// The reset blocks that a CTA replays side by side, and what the replay finds.
template <int kChains>
struct ReplayShared
{
    const float* x[kChains];             // the block's sample
    int pre[kChains], start[kChains], end[kChains];   // the fresh sum begins at pre, the block is [start, end)
    float low[kChains], high[kChains];   // an MMS at or above them is at or above the cutoff interval's ends
    // first and last index at or above the interval's low end, with the MMS there, and its high end (-1: none)
    int firstLow[kChains], lastLow[kChains], firstHigh[kChains], lastHigh[kChains];
    float firstValue[kChains], lastValue[kChains];
    float peak[kChains];                 // the largest MMS, -infinity when every MMS is NaN
    __device__ __forceinline__ void set(int j, const float* sample, int L, int W, int st, int R)
    {
        x[j] = sample;
        pre[j] = max(st - W + 1, 0);
        start[j] = st;
        end[j] = int(min((long long)L, (long long)st + R));
    }
};

// What the CTA of region_kernel shares.
struct RegionShared : ReplayShared<OneShape::kChains>
{
    double warp[kThreads / 32], warp2[kThreads / 32];
    double sums[3 * kSub];               // running sums of squares within the chunks a window enters and leaves
    float run[kRuns];                    // largest window energy of each run
    int hit, sure;
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
    bool longChain;       // a replay costs more here than in exact_kernel
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

// Replays the first `m` reset blocks of sh exactly and fills sh's results.  Lane j of warp 0 runs block j's chain
// from squares that the other warps, kRows blocks each, stage in shared memory one tile ahead; they also take the MMS
// values one tile behind: the maximum, and (kEnds) the ends against the cutoff's interval.  A square of zero stands
// for "nothing enters / leaves": sum + 0 and sum - 0 == sum exactly.
template <class Shape, bool kEnds, int kChains>
__device__ void replay(ReplayShared<kChains>& sh, float* buf, int m, int W, float meanFactor)
{
    constexpr int kTile = Shape::kTile, kRows = Shape::kRows, kLoads = kTile / 32, kAhead = 1024;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    auto row = [&](int slot, int what, int j) { return buf + ((slot * 3 + what) * Shape::kChains + j) * Shape::kPitch; };
    if (threadIdx.x < m)
    {
        const int j = threadIdx.x;   // the block's samples travel to L2 kAhead ahead of the staging
        l2_prefetch(sh.x[j] + sh.pre[j], sh.x[j] + min((long long)sh.end[j], (long long)sh.pre[j] + kAhead));
    }
    __syncthreads();
    int preMax = 0, blkMax = 0;
    for (int j = 0; j < m; ++j)
    {
        preMax = max(preMax, sh.start[j] - sh.pre[j]);
        blkMax = max(blkMax, sh.end[j] - sh.start[j]);
    }
    const int preTiles = (preMax + kTile - 1) / kTile, tiles = preTiles + (blkMax + kTile - 1) / kTile;
    if (warp == 0)
    {
        float sum = 0.0f;
        for (int it = 0; it < tiles + 2; ++it)
        {
            const int t = it - 1, slot = t & 1;
            if (t >= 0 && t < tiles && lane < m)
            {
                // two quads ahead of the chain
                const float4* in = reinterpret_cast<const float4*>(row(slot, 0, lane));
                float4 a0 = in[0], a1 = in[1];
                if (t < preTiles)
                {
#pragma unroll 8
                    for (int k = 0; k < kTile / 4; ++k)
                    {
                        const float4 a = a0;
                        a0 = a1;
                        a1 = in[k + 2];
                        sum = __fadd_rn(sum, a.x);
                        sum = __fadd_rn(sum, a.y);
                        sum = __fadd_rn(sum, a.z);
                        sum = __fadd_rn(sum, a.w);
                    }
                }
                else
                {
                    const float4* out = reinterpret_cast<const float4*>(row(slot, 1, lane));
                    float4* val = reinterpret_cast<float4*>(row(slot, 2, lane));
                    float4 o0 = out[0], o1 = out[1];
#pragma unroll 8
                    for (int k = 0; k < kTile / 4; ++k)
                    {
                        const float4 a = a0, o = o0;
                        a0 = a1;
                        o0 = o1;
                        a1 = in[k + 2];
                        o1 = out[k + 2];
                        float4 v;
                        sum = __fadd_rn(sum, a.x);
                        v.x = __fmul_rn(sum, meanFactor);
                        sum = __fsub_rn(sum, o.x);
                        sum = __fadd_rn(sum, a.y);
                        v.y = __fmul_rn(sum, meanFactor);
                        sum = __fsub_rn(sum, o.y);
                        sum = __fadd_rn(sum, a.z);
                        v.z = __fmul_rn(sum, meanFactor);
                        sum = __fsub_rn(sum, o.z);
                        sum = __fadd_rn(sum, a.w);
                        v.w = __fmul_rn(sum, meanFactor);
                        sum = __fsub_rn(sum, o.w);
                        val[k] = v;
                    }
                }
            }
            __syncthreads();
        }
        __syncthreads();
        return;
    }
    float a[kRows][kLoads], o[kRows][kLoads];   // samples entering and leaving, on their way
    auto load = [&](int it) {
        const bool fresh = it < preTiles;
#pragma unroll
        for (int r = 0; r < kRows; ++r)
        {
            const int j = warp - 1 + r * Shape::kStagers;
            if (j >= m) break;
            const int st = sh.start[j], from = fresh ? sh.pre[j] + it * kTile : st + (it - preTiles) * kTile;
            // of the tile's samples the block has those below `left`, and those from `kept` on leave the window
            const int left = (fresh ? st : sh.end[j]) - from;
            const long long kept = (long long)W - 1 - from;
            const float* x = sh.x[j] + from;
            if (it % (kAhead / kTile) == 0 && lane == 0)
            {
                const long long ahead = (long long)from + kAhead;
                l2_prefetch(sh.x[j] + ahead, sh.x[j] + min(ahead + kAhead, (long long)sh.end[j]));
            }
            if (left >= kTile && (fresh || kept <= 0))   // a whole tile: no comparison per sample
            {
#pragma unroll
                for (int k = 0; k < kLoads; ++k) a[r][k] = __ldg(RPPB_RD(x + lane + 32 * k));
                if (fresh) continue;
                const float* gone = x + lane - W + 1;
#pragma unroll
                for (int k = 0; k < kLoads; ++k) o[r][k] = __ldg(RPPB_RD(gone + 32 * k));
                continue;
            }
#pragma unroll
            for (int k = 0; k < kLoads; ++k)
            {
                const int i = lane + 32 * k;
                a[r][k] = i < left ? __ldg(RPPB_RD(x + i)) : 0.0f;
                o[r][k] = !fresh && i < left && i >= kept ? __ldg(RPPB_RD(x + (i - W + 1))) : 0.0f;
            }
        }
    };
    // what each lane has seen of its values, in ascending order
    float peak[kRows], firstValue[kRows], lastValue[kRows];
    int firstLow[kRows], lastLow[kRows], firstHigh[kRows], lastHigh[kRows];
#pragma unroll
    for (int r = 0; r < kRows; ++r)
    {
        peak[r] = -INFINITY;
        firstLow[r] = firstHigh[r] = INT_MAX;
        lastLow[r] = lastHigh[r] = -1;
        firstValue[r] = lastValue[r] = 0.f;
    }
    load(0);
    for (int it = 0; it < tiles + 2; ++it)
    {
        if (it < tiles)
        {
#pragma unroll
            for (int r = 0; r < kRows; ++r)
            {
                const int j = warp - 1 + r * Shape::kStagers;
                if (j >= m) break;
                float* in = row(it & 1, 0, j) + lane;
#pragma unroll
                for (int k = 0; k < kLoads; ++k) in[32 * k] = sq(a[r][k]);
                if (it < preTiles) continue;
                float* out = row(it & 1, 1, j) + lane;
#pragma unroll
                for (int k = 0; k < kLoads; ++k) out[32 * k] = sq(o[r][k]);
            }
            if (it + 1 < tiles) load(it + 1);
        }
        const int done = it - 2;
        if (done >= preTiles)
        {
#pragma unroll
            for (int r = 0; r < kRows; ++r)
            {
                const int j = warp - 1 + r * Shape::kStagers;
                if (j >= m) break;
                const float* val = row(done & 1, 2, j) + lane;
                const int v0 = sh.start[j] + (done - preTiles) * kTile, left = sh.end[j] - v0;
                if (!kEnds && left >= kTile)
                {
#pragma unroll
                    for (int k = 0; k < kLoads; ++k) peak[r] = fmaxf(peak[r], val[32 * k]);
                    continue;
                }
                const float low = sh.low[j], high = sh.high[j];
#pragma unroll
                for (int k = 0; k < kLoads; ++k)
                {
                    const int i = lane + 32 * k;
                    const float v = i < left ? val[32 * k] : NAN;   // a NaN takes part in nothing
                    peak[r] = fmaxf(peak[r], v);
                    if (kEnds && v >= low)
                    {
                        lastLow[r] = v0 + i;
                        lastValue[r] = v;
                        if (firstLow[r] == INT_MAX)
                        {
                            firstLow[r] = v0 + i;
                            firstValue[r] = v;
                        }
                    }
                    if (kEnds && v >= high)
                    {
                        lastHigh[r] = v0 + i;
                        firstHigh[r] = min(firstHigh[r], v0 + i);
                    }
                }
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int r = 0; r < kRows; ++r)
    {
        const int j = warp - 1 + r * Shape::kStagers;
        if (j >= m) break;
        const float top = warp_max(peak[r]);
        if (lane == 0) sh.peak[j] = top;
        if constexpr (kEnds)
        {
            const int f = __reduce_min_sync(0xffffffffu, firstLow[r]), l = __reduce_max_sync(0xffffffffu, lastLow[r]);
            const int fh = __reduce_min_sync(0xffffffffu, firstHigh[r]), lh = __reduce_max_sync(0xffffffffu, lastHigh[r]);
            if (f == firstLow[r]) sh.firstValue[j] = firstValue[r];   // one lane, unless there is none
            if (l == lastLow[r]) sh.lastValue[j] = lastValue[r];
            if (lane == 0)
            {
                sh.firstLow[j] = f == INT_MAX ? -1 : f;
                sh.lastLow[j] = l;
                sh.firstHigh[j] = fh == INT_MAX ? -1 : fh;
                sh.lastHigh[j] = lh;
            }
        }
    }
    __syncthreads();
}

constexpr int kNone = -1;        // no MMS reaches the cutoff
constexpr int kUnsettled = -2;   // an exact MMS lies inside the cutoff's interval
constexpr int kGiveUp = -3;      // too many candidates: exact_kernel replays every block

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
        if (clip.longChain || ++replays > 2) return kGiveUp;
        const int k = at / clip.R;
        if (tid == 0)
        {
            sh.set(0, clip.x, clip.L, clip.W, k * clip.R, clip.R);
            sh.low[0] = __double2float_ru(low);
            sh.high[0] = __double2float_ru(high);
        }
        clip.P = clip.all;   // the replay's buffers take the place of the copy in shared memory
        __syncthreads();
        replay<OneShape, true>(sh, buf, 1, clip.W, clip.meanFactor);
        const int lo = kLast ? sh.lastLow[0] : sh.firstLow[0], hi = kLast ? sh.lastHigh[0] : sh.firstHigh[0];
        open.index = lo;
        open.value = kLast ? sh.lastValue[0] : sh.firstValue[0];
        __syncthreads();
        if (lo >= 0) return lo == hi ? lo : kUnsettled;
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
// sh.run[r] = the largest of run r (kRuns runs at most).  Negative: too many chunks to search (a clip of steady level).
__device__ double largest_window(const Clip& clip, RegionShared& sh, double least)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    auto square = [&](long long i) { return i >= 0 && i < clip.L ? sq(__ldg(RPPB_RD(clip.x + i))) : 0.0f; };
    for (int r = threadIdx.x; r < kRuns; r += kThreads) sh.run[r] = 0.0f;
    if (threadIdx.x == 0) sh.hit = 0;
    __syncthreads();
    int chunks = 0;
    for (int c = threadIdx.x; c < clip.chunks; c += kThreads) chunks += clip.upper(c) >= least;
    chunks = __reduce_add_sync(0xffffffffu, chunks);
    if (lane == 0 && chunks > 0) atomicAdd(&sh.hit, chunks);
    __syncthreads();
    const bool many = sh.hit > kSearch;
    __syncthreads();
    if (many) return -1.0;
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

// What the clips whose ends region_kernel does not settle leave for exact_kernel.
struct ExactList
{
    unsigned long long* tally;   // entries << kTallyShift | their reset blocks, then the blocks claimed; zeroed by energy_kernel
    int* clip;                   // entry -> clip
    long long* first;            // entry -> its first block in blockMax
    int* done;                   // entry -> blocks replayed
    float* blockMax;             // largest MMS of each block, NaN when all are
};

__device__ __forceinline__ void write_region(int first, int last, int W, int b, int* outBegin, int* outLength)
{
    int detectBegin = 0, detectLength = 0;
    if (first >= 0)
    {
        detectBegin = first;
        detectLength = last - first + 1;
        if (detectBegin != 0 && detectLength != 0)
        {
            const int newBegin = max(detectBegin - (W - 1), 0);
            detectLength += detectBegin - newBegin;
            detectBegin = newBegin;
        }
    }
    *RPPB_WR(outBegin + b) = detectBegin;
    *RPPB_WR(outLength + b) = detectLength;
}

__global__ void __launch_bounds__(kThreads) region_kernel(const float* __restrict__ src, uint32_t stride,
                                                          const int* __restrict__ len, int windowLength, int reset,
                                                          float referencePower, float cutOff, double* __restrict__ energies,
                                                          long long pitch, bool intervals, bool local, ExactList exact,
                                                          int* __restrict__ outBegin, int* __restrict__ outLength)
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    // OneShape::kBytes: the prefix energies, then squares entering, squares leaving and MMS in two slots
    extern __shared__ __align__(16) float buf[];
    __shared__ RegionShared sh;
    const int b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int L = min(*RPPB_RD(len + b), int(stride));
    grid_dependency_wait();   // the chunk energies, the zeroed tally
    if (L <= 0)
    {
        if (tid == 0) write_region(-1, -1, windowLength, b, outBegin, outLength);
        return;
    }
    // leaves the clip to exact_kernel (never with `local`: then its blocks fit a replay here, and that kernel is not
    // launched)
    auto pass_on = [&](int blocks) {
        const unsigned long long t =
            atomicAdd(RPPB_WR(dependency_result(exact.tally)), 1ull << kTallyShift | (unsigned long long)blocks);
        const int e = int(t >> kTallyShift);
        *RPPB_WR(exact.clip + e) = b;
        *RPPB_WR(exact.first + e) = (long long)(t & ((1ull << kTallyShift) - 1));
        *RPPB_WR(exact.done + e) = 0;
    };
    double* P = dependency_result(energies) + b * pitch;
    double* held = reinterpret_cast<double*>(buf);
    Clip clip{src + size_t(b) * stride, L, windowLength, reset == -1 ? L : reset,
              __fdiv_rn(1.0f, float(windowLength)), P, P, (L + kSub - 1) / kSub, 0.0, 0.0, false};
    const int blocks = int(((long long)L + clip.R - 1) / clip.R);
    if (!intervals)
    {
        if (tid == 0) pass_on(blocks);
        return;
    }

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
    clip.longChain = ops > kLongChain;
    // Intervals help where the chain's rounding bound is small and every number is a normal one; elsewhere (and
    // when they do not settle the ends) every block is replayed.
    bool full = !(total <= 1e37) || clip.R < kSub || ops * kUlp > 1.0 / 16;
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
            for (int stage = 0;;)
            {
                Open open{};
                if (first < 0) first = find_end<false>(clip, sh, buf, low, high, open);
                last = first < 0 ? first : find_end<true>(clip, sh, buf, low, high, open);
                if (last != kUnsettled || !peakRef || stage == 2) break;
                bool found = true;
                do   // until the open value is outside the interval
                {
                    if (stage == 0)
                    {
                        const double tol = 1e-5 * clip.top;
                        const double peak = largest_window(clip, sh, lo - clip.slack - 2.0 * (err + tol));
                        found = peak >= 0.0;
                        if (!found) break;
                        peakLow = peak - tol - err;
                        cutoff_interval(peak + tol + err);
                    }
                    else
                    {
                        // from the blocks whose energies allow the maximum, unless they are too many
                        if (tid == 0) sh.hit = 0;
                        __syncthreads();
                        for (int k = tid; k < blocks; k += kThreads)
                        {
                            const int st = k * clip.R, en = int(min((long long)L, (long long)st + clip.R));
                            bool any = false;
                            for (int r = st / kRun; !any && r <= (en - 1) / kRun; ++r)
                                any = r >= kRuns || sh.run[r] + 1e-5 * clip.top + err >= peakLow;
                            if (!any) continue;
                            const int at = atomicAdd(&sh.hit, 1);
                            if (at < OneShape::kChains) sh.set(at, clip.x, L, clip.W, st, clip.R);
                        }
                        __syncthreads();
                        const int m = sh.hit;
                        found = m <= OneShape::kChains;
                        if (!found) break;
                        clip.P = clip.all;
                        replay<OneShape, false>(sh, buf, m, clip.W, clip.meanFactor);
                        float peak = -FLT_MAX;
                        for (int j = 0; j < m; ++j)
                            peak = fmaxf(peak, sh.peak[j]);
                        __syncthreads();
                        low = high = double(__fmul_rn(peak, cutOff));
                    }
                    ++stage;
                } while (stage < 2 && double(open.value) >= low && double(open.value) < high);
                if (!found)
                {
                    first = kGiveUp;
                    break;
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
    if (full && local)
    {
        clip.P = clip.all;
        auto all = [&](float cut) {
            __syncthreads();
            if (tid < blocks)
            {
                sh.set(tid, clip.x, L, clip.W, tid * clip.R, clip.R);
                sh.low[tid] = sh.high[tid] = cut;
            }
            __syncthreads();
            replay<OneShape, true>(sh, buf, blocks, clip.W, clip.meanFactor);
        };
        float base = referencePower;
        if (peakRef)
        {
            all(INFINITY);
            base = -FLT_MAX;
            for (int j = 0; j < blocks; ++j) base = fmaxf(base, sh.peak[j]);
        }
        all(__fmul_rn(base, cutOff));
        first = last = -1;
        for (int j = 0; j < blocks; ++j)
        {
            if (sh.lastLow[j] < 0) continue;
            if (first < 0) first = sh.firstLow[j];
            last = sh.lastLow[j];
        }
        full = false;
    }
    if (tid != 0) return;
    if (full) pass_on(blocks);
    else write_region(first, last, windowLength, b, outBegin, outLength);
}

// The clips of the list: their reset blocks, dealt to the CTAs of the whole grid a few at a time, are replayed for
// their maxima; the CTA that replays a clip's last block then has the cutoff, and replays the first and the last block
// that reach it for the ends.  No CTA waits for another.  Bound by the chains' latency (10 cycles per sample) until
// 8288 blocks are in flight, then by the issue of the staging.  28 blocks of 128 samples per CTA: 14 of 256 took 1746
// instead of 1470 us on 512000 blocks of 32 samples, as much elsewhere; 28 of 64 took 359 instead of 267 us on 8200
// blocks of 8192.
__global__ void __launch_bounds__(kThreads, 2) exact_kernel(const float* __restrict__ src, uint32_t stride,
                                                            const int* __restrict__ len, int windowLength, int reset,
                                                            float referencePower, float cutOff, ExactList list,
                                                            int* __restrict__ outBegin, int* __restrict__ outLength)
{
    constexpr int kChains = ManyShape::kChains;
    static_assert(kChains <= 32, "a lane each");
    static_assert(OneShape::kBytes <= ManyShape::kBytes && OneShape::kChains <= kChains, "the ends' replay");
    extern __shared__ __align__(16) float buf[];   // ManyShape::kBytes
    __shared__ ReplayShared<kChains> sh;
    __shared__ int s_entry[kChains], s_last[kChains];   // per replayed block: its entry; the entry again when it was its last
    __shared__ int s_clip[kChains], s_first, s_final;
    __shared__ float s_max[kThreads / 32];
    __shared__ long long s_next;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float meanFactor = __fdiv_rn(1.0f, float(windowLength));
    grid_dependency_wait();
    const unsigned long long tally = *RPPB_RD(dependency_result(list.tally));
    const long long total = (long long)(tally & ((1ull << kTallyShift) - 1));
    if (total == 0) return;
    const int entries = int(tally >> kTallyShift);
    const int* clips = dependency_result(list.clip);
    const long long* firsts = dependency_result(list.first);
    const int per = int(min((long long)kChains, (total + gridDim.x - 1) / gridDim.x));   // blocks per CTA step
    auto samples = [&](int b) { return min(*RPPB_RD(len + b), int(stride)); };
    auto block_len = [&](int L) { return reset == -1 ? L : reset; };
    auto block_count = [&](int L) { return int(((long long)L + block_len(L) - 1) / block_len(L)); };
    for (;;)
    {
        // claimed, not dealt: a CTA that has finished a clip would stay behind, and so finish the next ones too
        if (tid == 0) s_next = (long long)atomicAdd(RPPB_WR(dependency_result(list.tally) + 1), (unsigned long long)per);
        __syncthreads();
        const long long w = s_next;
        if (w >= total) break;
        const int m = int(min((long long)per, total - w));
        if (tid < m)
        {
            const int e = ragged_find(firsts, entries, w + tid), b = *RPPB_RD(clips + e);
            const int L = samples(b), R = block_len(L);
            s_entry[tid] = e;
            sh.set(tid, src + size_t(b) * stride, L, windowLength, int(w + tid - *RPPB_RD(firsts + e)) * R, R);
        }
        __syncthreads();
        replay<ManyShape, false>(sh, buf, m, windowLength, meanFactor);
        if (tid < m)
        {
            const int e = s_entry[tid];
            *RPPB_WR(list.blockMax + (w + tid)) = sh.peak[tid] == -INFINITY ? NAN : sh.peak[tid];
            __threadfence();   // the maximum before the count
            const int before = atomicAdd(RPPB_WR(list.done + e), 1);
            s_last[tid] = before + 1 == block_count(samples(*RPPB_RD(clips + e))) ? e : -1;
        }
        __syncthreads();
        // the clips whose last block this was, as many at a time as their end blocks fit side by side
        int ends = 0;    // end blocks gathered
        auto finish = [&] {
            __syncthreads();
            replay<OneShape, true>(sh, buf, ends, windowLength, meanFactor);
            // a clip's blocks are neighbours, its first one carries the clip
            if (tid < ends && s_clip[tid] >= 0)
            {
                const int other = tid + 1 < ends && s_clip[tid + 1] < 0 ? tid + 1 : tid;
                write_region(sh.firstLow[tid], sh.lastLow[other], windowLength, s_clip[tid], outBegin, outLength);
            }
            __syncthreads();
            ends = 0;
        };
        for (int j = 0; j < m; ++j)
        {
            const int e = s_last[j];
            if (e < 0) continue;
            const int b = *RPPB_RD(clips + e), L = samples(b), R = block_len(L), blocks = block_count(L);
            const float* maxima = list.blockMax + *RPPB_RD(firsts + e);
            __threadfence();
            float base = referencePower;
            if (referencePower == 0.0f)
            {
                float peak = -FLT_MAX;
                for (int k = tid; k < blocks; k += kThreads) peak = fmaxf(peak, __ldcg(RPPB_RD(maxima + k)));
                peak = warp_max(peak);
                if (lane == 0) s_max[warp] = peak;
                __syncthreads();
                base = s_max[0];
                for (int i = 1; i < kThreads / 32; ++i) base = fmaxf(base, s_max[i]);
            }
            const float cut = __fmul_rn(base, cutOff);
            if (tid == 0)
            {
                s_first = INT_MAX;
                s_final = -1;
            }
            __syncthreads();
            for (int k = tid; k < blocks; k += kThreads)
                if (__ldcg(RPPB_RD(maxima + k)) >= cut)
                {
                    atomicMin(&s_first, k);
                    atomicMax(&s_final, k);
                }
            __syncthreads();
            const int first = s_first, final = s_final;
            __syncthreads();   // s_first, s_final and s_max are free
            if (final < 0)
            {
                if (tid == 0) write_region(-1, -1, windowLength, b, outBegin, outLength);
                continue;
            }
            const int need = first == final ? 1 : 2;
            if (ends + need > OneShape::kChains) finish();
            if (tid < need)
            {
                const int at = ends + tid;
                s_clip[at] = tid == 0 ? b : -1;
                sh.set(at, src + size_t(b) * stride, L, windowLength, (tid == 0 ? first : final) * R, R);
                sh.low[at] = sh.high[at] = cut;
            }
            ends += need;
        }
        if (ends > 0) finish();
    }
}

// prefix energies per sample: one more entry than chunks
long long energy_pitch(uint32_t srcStride) { return (long long)(srcStride / kSub) + 2; }

// reset blocks of the batch, at most
size_t block_count(int n, uint32_t srcStride, int resetInterval)
{
    return resetInterval == -1 ? size_t(n) : size_t(n) * ((size_t(srcStride) + resetInterval - 1) / resetInterval);
}

// Many short samples: nsr_stored.cu's kernels.  On signals that end in silence, where intervals need a replay (window 512
// up to 8000 samples a row, 2048 above; 35 % silence at the end), those against these took, us: 1024 samples of 1600 44 and
// 65, of 8000 149 and 233, of 16000 210 and 200, of 32000 288 and 359, of 64000 439 and 347; 8192 of 8000 280 and 1238;
// 512 of 8000 146 and 144, of 32000 253 and 187.  (Without silence intervals are faster from 4000 samples on, 8192 of
// 16000 282 instead of 515 us.)
bool stored(int n, uint32_t srcStride, int windowLength, int resetInterval)
{
    constexpr int kSamples = 1024;
    constexpr long long kSteps = 49152;   // of a sample's chains: 32768 samples with a window of 2048
    const long long blocks = resetInterval == -1 ? 1 : ((long long)srcStride + resetInterval - 1) / resetInterval;
    return n >= kSamples && (long long)srcStride + blocks * windowLength <= kSteps;
}

}  // namespace

size_t nsr_scratch_bytes(int n, uint32_t srcStride, int windowLength, int resetInterval)
{
    if (stored(n, srcStride, windowLength, resetInterval)) return nsr_stored_scratch_bytes(n, srcStride, resetInterval);
    Carver cv(nullptr);
    cv.take<unsigned long long>(2);
    cv.take<double>(size_t(n) * energy_pitch(srcStride));
    cv.take<int>(n);
    cv.take<long long>(n);
    cv.take<int>(n);
    cv.take<float>(block_count(n, srcStride, resetInterval));
    return cv.used();
}

void launch_nsr(Handle& h, void* scratch, const NsrArgs& a)
{
    if (a.n <= 0) return;
    if (stored(a.n, a.srcStride, a.windowLength, a.resetInterval)) return launch_nsr_stored(h, scratch, a);
    Carver cv(scratch);
    const long long pitch = energy_pitch(a.srcStride);
    ExactList list;
    list.tally = cv.take<unsigned long long>(2);
    double* energies = cv.take<double>(size_t(a.n) * pitch);
    list.clip = cv.take<int>(a.n);
    list.first = cv.take<long long>(a.n);
    list.done = cv.take<int>(a.n);
    list.blockMax = cv.take<float>(block_count(a.n, a.srcStride, a.resetInterval));
    // the intervals' chunks have to resolve the window and the reset blocks; else exact_kernel takes every clip
    const bool intervals = a.windowLength >= 4 * kSub && (a.resetInterval == -1 || a.resetInterval >= kSub);
    // samples of few reset blocks are finished by region_kernel whatever their intervals say, and a launch is saved (one
    // clip of 1 s 16.0 -> 12.4 us)
    const bool local = intervals && block_count(1, a.srcStride, a.resetInterval) <= OneShape::kChains;
    const int ups = int(a.srcStride / kUnit) + 1;
    for (int b0 = 0; b0 < a.n; b0 += kMaxClips)
    {
        const int n = std::min(a.n - b0, kMaxClips);
        const float* src = a.src + size_t(b0) * a.srcStride;
        const long long units = intervals ? (long long)n * ups : 1;
        const int grid = int(std::min<long long>(
            units, persistent_grid(h, reinterpret_cast<const void*>(energy_kernel), kThreads, 0)));
        energy_kernel<<<grid, kThreads, 0, h.stream()>>>(src, a.srcStride, a.len + b0, energies, pitch,
                                                         intervals ? n : 0, ups, list.tally);
        count_launch();
        check_cuda(cudaGetLastError(), "energy_kernel");
        persistent_grid(h, reinterpret_cast<const void*>(region_kernel), kThreads, OneShape::kBytes);   // shared-memory opt-in
        launch_dependent(region_kernel, dim3(n), dim3(kThreads), OneShape::kBytes, h.stream(), "region_kernel", src,
                         a.srcStride, a.len + b0, a.windowLength, a.resetInterval, a.referencePower, a.cutOff, energies,
                         pitch, intervals, local, list, a.begin + b0, a.length + b0);
        count_launch();
        if (local) continue;
        const int exactGrid = persistent_grid(h, reinterpret_cast<const void*>(exact_kernel), kThreads, ManyShape::kBytes);
        launch_dependent(exact_kernel, dim3(exactGrid), dim3(kThreads), ManyShape::kBytes, h.stream(), "exact_kernel", src,
                         a.srcStride, a.len + b0, a.windowLength, a.resetInterval, a.referencePower, a.cutOff, list,
                         a.begin + b0, a.length + b0);
        count_launch();
    }
}

}  // namespace rppb
