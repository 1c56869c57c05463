// One tile of STFT frames -> power (or magnitude) spectrum in shared memory, for nfft 128 and 512, whose packed
// transform is R x R points (the other sizes use stft.cuh's stft_tile).
//
// Same framing and real-FFT packing as stft_tile: M = nfft/2 complex points of a frame, R lanes per frame, R-point
// register DFTs, one shared-memory exchange, R-point register DFTs, real unpack.  What differs:
//   - the bins k and M - k that the unpack pairs lie in lanes j and R - j of the frame's lanes, so they meet by warp
//     shuffles and the transform is not stored again;
//   - the power of frames f and f + 1, which one warp transforms, replaces their exchange slots, so a 16-frame
//     tile needs 35 KB instead of 53 KB and four CTAs of 256 threads fit an SM (at 64 registers), not three;
//   - the window is halved (exact), which takes the place of the unpack's factors of 1/2;
//   - the next tile's samples are copied into the span buffer while this tile is transformed.
// On 256 clips of 1 to 16 s (nfft 512) the spectrogram kernel takes 176 us instead of 221 (ncu) and the fused front
// end, which keeps 80 registers and three CTAs (64 registers spill: 302 us), 251 us instead of 262.  The transform is
// not what bounds the spectrogram: without it the kernel takes 167 us, without its stores 52.
// Two frames per lane group in the halves of paired instructions (fewer instructions, 128 registers, 16 warps per
// SM) took 202 and 281 us.
#pragma once

#include "stft.cuh"

namespace rppb {

template <int NFFT>
struct PairShape
{
    static constexpr int THREADS = 256;
    static constexpr int M = NFFT / 2, R = Plan<NFFT>::R1, BINS = M + 1;
    static constexpr int TF = THREADS / R, PAIRS = TF / 2;
    static_assert(!PairPlan<NFFT>::use || (R * R == M && Plan<NFFT>::R2 == R && TF == Plan<NFFT>::TF), "plan");
    // A frame's slot: R rows of R + 1 float2 (no bank conflicts either way); with R = 8 the two frames that an
    // access covers lie half the banks apart.  A pair's two slots are followed by 16 bytes, so that equal bins of
    // the pairs' powers lie 4 banks apart.
    static constexpr int LD = R + 1;
    static constexpr int FRAME = R * LD;   // float2 (R = 8: 72, half the banks past a multiple of all)
    static constexpr int PAIR_FLOATS = 4 * FRAME + 4;
    static constexpr size_t slot_bytes = size_t(PAIRS) * PAIR_FLOATS * 4;
    static_assert(2 * BINS <= 4 * FRAME, "the power of two frames fits their slots");
};

// ---------------------------------------------------------------- the tile's input span
// A tile goes through four steps, so that the next tile's samples travel while this one is transformed:
//   span_issue     starts the copies of a tile's raw samples into the span buffer (asynchronous, no registers);
//   span_arrive    waits for them (a barrier);
//   pair_gather    windows (and, kPreemph, first pre-emphasizes) the frames into registers; after the next barrier
//                  the span buffer is free;
//   pair_transform transforms them and leaves the power in the exchange slots.
// Tiles at a clip's ends, which need reflection or zeros, are staged (and pre-emphasized) by span_arrive instead.
// Pre-emphasis in the gather costs 2.5 times the operations of one pass over the span (hop 160 of 400), and neither
// that pass's shared-memory round trip nor its two barriers.

// Starts the copies of the span of frames f0 .. f0+TF-1 (those < F) and zeroes its tail.  False (and nothing
// started) for a tile that reaches past the signal, or, kPreemph, before its second sample.  The sample before the
// span goes into the last float of the pad (kPreemph).  The span buffer must be free.
template <int NFFT, bool kPreemph>
__device__ __forceinline__ bool span_issue(const float* __restrict__ x, int L, int f0, int F, int W, int hop,
                                           int centerOffset, float* __restrict__ s_span)
{
    using P = PairShape<NFFT>;
    using S = StftShape<NFFT, P::THREADS, P::TF>;
    const int start = f0 * hop - centerOffset, len = (min(P::TF, F - f0) - 1) * hop + W;
    if (start < (kPreemph ? 1 : 0) || start + len > L) return false;
    const float* from = x + start;
    float* to = s_span + S::span_pad(W);
    if ((reinterpret_cast<uintptr_t>(from) & 15) == 0)
    {
        for (int i = 4 * threadIdx.x; i + 4 <= len; i += 4 * P::THREADS)
            copy_async16(to + i, RPPB_RD(reinterpret_cast<const float4*>(from + i)));
        const int i = (len & ~3) + threadIdx.x;
        if (i < len) copy_async4(to + i, RPPB_RD(from + i));
    }
    else
        for (int i = threadIdx.x; i < len; i += P::THREADS) copy_async4(to + i, RPPB_RD(from + i));
    if (kPreemph && threadIdx.x == 0) copy_async4(to - 1, RPPB_RD(from - 1));
    asm volatile("cp.async.commit_group;" ::: "memory");
    for (int i = threadIdx.x; i < S::span_tail(W); i += P::THREADS) to[len + i] = 0.f;
    return true;
}

// stft_stage_span for the tiles at a clip's ends, out of line: its registers would come on top of the kernels'.
template <int NFFT, class Src>
__device__ RPPB_OUT_OF_LINE void span_stage_edge(Src src, int f0, int F, int W, int hop, int centerOffset, float* s_span)
{
    using P = PairShape<NFFT>;
    using S = StftShape<NFFT, P::THREADS, P::TF>;
    if (threadIdx.x == 0) s_span[S::span_pad(W) - 1] = 0.f;   // an earlier tile's sample
    stft_stage_span<NFFT, P::THREADS, P::TF>(src, f0, F, W, hop, centerOffset, s_span);
}

// Makes the tile's span readable by all threads; `issued`: what span_issue returned for it (raw samples), else the
// samples that src gives.
template <int NFFT, class Src>
__device__ __forceinline__ void span_arrive(bool issued, const Src& src, int f0, int F, int W, int hop, int centerOffset,
                                            float* __restrict__ s_span)
{
    if (!issued)
    {
        span_stage_edge<NFFT>(src, f0, F, W, hop, centerOffset, s_span);
        return;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
}

// ---------------------------------------------------------------- the transform

namespace fft {

// x0 = e + W_R^K o, x1 = e - W_R^K o
template <int R, int K>
__device__ __forceinline__ void butterfly(float2& x0, float2& x1, float2 e, float2 o)
{
    constexpr float h = Tw<1, 8>::c;
    if constexpr (K == 0)
    {
        x0 = add2(e, o);
        x1 = sub2(e, o);
    }
    else if constexpr (4 * K == R)   // * (-i)
    {
        x0 = make_float2(e.x + o.y, e.y - o.x);
        x1 = make_float2(e.x - o.y, e.y + o.x);
    }
    else if constexpr (8 * K == R)   // * (1 - i)/sqrt2
    {
        const float p = o.x + o.y, m = o.y - o.x;
        x0 = make_float2(fmaf(h, p, e.x), fmaf(h, m, e.y));
        x1 = make_float2(fmaf(-h, p, e.x), fmaf(-h, m, e.y));
    }
    else if constexpr (8 * K == 3 * R)   // * (-1 - i)/sqrt2
    {
        const float p = o.x + o.y, m = o.y - o.x;
        x0 = make_float2(fmaf(h, m, e.x), fmaf(-h, p, e.y));
        x1 = make_float2(fmaf(-h, m, e.x), fmaf(h, p, e.y));
    }
    else
    {
        const float2 t = cmul_conj(o, Tw<K, R>::c, Tw<K, R>::s);
        x0 = add2(e, t);
        x1 = sub2(e, t);
    }
}

template <int R, int K = 0>
__device__ __forceinline__ void butterflies(float2 (&x)[R], const float2 (&e)[R / 2], const float2 (&o)[R / 2])
{
    if constexpr (K < R / 2)
    {
        butterfly<R, K>(x[K], x[K + R / 2], e[K], o[K]);
        butterflies<R, K + 1>(x, e, o);
    }
}

// In-place forward DFT of R points held in registers, natural order in and out (Dft<R> with the products by
// 1/sqrt2 fused into the butterflies' additions).
template <int R>
__device__ __forceinline__ void dft(float2 (&x)[R])
{
    if constexpr (R > 1)
    {
        float2 e[R / 2], o[R / 2];
#pragma unroll
        for (int i = 0; i < R / 2; ++i)
        {
            e[i] = x[2 * i];
            o[i] = x[2 * i + 1];
        }
        dft<R / 2>(e);
        dft<R / 2>(o);
        butterflies<R>(x, e, o);
    }
}

}  // namespace fft

// Fills the per-CTA constant tables as stft_tables does, with the window halved.
template <int NFFT>
__device__ __forceinline__ void stft_pair_tables(const float2* __restrict__ twiddle, const float* __restrict__ window,
                                                 int W, float2* s_tw, float2* s_tw1, float* s_win, float* s_span)
{
    using P = PairShape<NFFT>;
    stft_tables<NFFT, P::THREADS>(twiddle, window, W, s_tw, s_tw1, s_win, s_span);
    for (int i = threadIdx.x; i < NFFT; i += P::THREADS) s_win[i] *= 0.5f;
    __syncthreads();
}

// The windowed points of this thread's frame (frame threadIdx.x / R of the tile).  kPreemph: of the pre-emphasized
// signal y[i] = x[i] - c x[i - 1], rounded as the pre_emphasis_filter kernel does.
template <int NFFT, bool kPreemph = false>
__device__ __forceinline__ void pair_gather(float2 (&z)[PairShape<NFFT>::R], int W, int hop, const float* __restrict__ s_win,
                                            const float* __restrict__ s_span, float c = 0.f)
{
    using P = PairShape<NFFT>;
    using S = StftShape<NFFT, P::THREADS, P::TF>;
    constexpr int R = P::R;
    const int j = threadIdx.x % R, fl = threadIdx.x / R;
    const int off = S::window_offset(W);
    const float* fs = s_span + S::span_pad(W) + fl * hop - off + 2 * j;   // buffer sample n of the frame at n - 2 j
    const float* win = s_win + 2 * j;
    // scalar products: the assembler may contract paired ones with the transform's first additions, in one kernel
    // and not in another, and the kernels must give the same bits
    auto point = [&](int m, float2 v) {
        const float2 w = *reinterpret_cast<const float2*>(win + 2 * R * m);
        if constexpr (kPreemph)
        {
            const float p = fs[2 * R * m - 1];
            v.y = __fsub_rn(v.y, __fmul_rn(c, v.x));
            v.x = __fsub_rn(v.x, __fmul_rn(c, p));
        }
        return make_float2(__fmul_rn(w.x, v.x), __fmul_rn(w.y, v.y));
    };
    if (((off | hop) & 1) == 0)   // (window, sample) pairs are 8-byte aligned
    {
#pragma unroll
        for (int m = 0; m < R; ++m) z[m] = point(m, *reinterpret_cast<const float2*>(fs + 2 * R * m));
    }
    else
    {
#pragma unroll
        for (int m = 0; m < R; ++m) z[m] = point(m, make_float2(fs[2 * R * m], fs[2 * R * m + 1]));
    }
}

// Transforms the frames: the power of bin k of tile frame fl is s_slots[(fl / 2) * PAIR_FLOATS + 2 * k + fl % 2];
// frames past the tile's valid ones hold undefined values.  The caller synchronizes before it reads the power.
template <int NFFT>
__device__ __forceinline__ void pair_transform(float2 (&z)[PairShape<NFFT>::R], int power, const float2* __restrict__ s_tw,
                                               const float2* __restrict__ s_tw1, float* __restrict__ s_slots)
{
    using P = PairShape<NFFT>;
    constexpr int R = P::R, M = P::M;
    const int j = threadIdx.x % R, fl = threadIdx.x / R;
    float* pair = s_slots + (fl >> 1) * P::PAIR_FLOATS;
    float2* slot = reinterpret_cast<float2*>(pair) + (fl & 1) * P::FRAME;

    fft::dft<R>(z);
    slot[j] = z[0];   // W_M^(j*0) = 1
#pragma unroll
    for (int k1 = 1; k1 < R; ++k1)
    {
        const float2 t = s_tw1[k1 * R + j];
        slot[k1 * P::LD + j] = fft::cmul_conj(z[k1], t.x, t.y);
    }
    __syncwarp();
    float2 y[R];   // row k1 = j
#pragma unroll
    for (int i = 0; i < R; ++i) y[i] = slot[j * P::LD + i];
    __syncwarp();   // the power overwrites the pair's slots
    fft::dft<R>(y);   // y[k2] = Z[j + R * k2]

    // Bins k = j + R i and M - k for i < R/2: Z[M - k] is lane (R - j) mod R's element R - 1 - i (lane 0's own
    // element (R - i) mod R).  X[k] = E + W^k O and X[M-k] = conj(E - W^k O) with E = Z[k] + conj Z[M-k] and
    // O = (Z[k] - conj Z[M-k]) / i, the factors 1/2 being in the window.
    float* out = pair + (fl & 1);
    auto bins = [&](float2 a, float2 b, float2 t, float& p0, float& p1) {
        const float2 sum = fft::add2(a, b), dif = fft::sub2(a, b);   // (er, orr), (-oi, ei)
        const float pr = fmaf(sum.y, t.x, -dif.x * t.y);
        const float pi = fmaf(-dif.x, t.x, -sum.y * t.y);
        const float xr = sum.x + pr, xi = dif.y + pi, yr = sum.x - pr, yi = dif.y - pi;
        p0 = fmaf(xr, xr, xi * xi);
        p1 = fmaf(yr, yr, yi * yi);
    };
    const int partner = (R - j) & (R - 1);
#pragma unroll
    for (int i = 0; i < R / 2; ++i)
    {
        const float2 mine = y[R - 1 - i], zero = y[(R - i) & (R - 1)];
        float2 b;
        b.x = __shfl_sync(0xffffffffu, j == 0 ? zero.x : mine.x, partner, R);
        b.y = __shfl_sync(0xffffffffu, j == 0 ? zero.y : mine.y, partner, R);
        float p0, p1;
        bins(y[i], b, s_tw[j + R * i], p0, p1);
        out[2 * (j + R * i)] = p0;
        out[2 * (M - j - R * i)] = p1;
    }
    if (j == 0)
    {
        float p0, p1;
        bins(y[R / 2], y[R / 2], s_tw[M / 2], p0, p1);
        out[M] = p0;
    }
    if (power == 1)   // magnitudes, in a pass of their own: the square roots would double the loop above
    {
        __syncwarp();
        for (int k = j; k <= M; k += R) out[2 * k] = sqrtf(out[2 * k]);
    }
}

}  // namespace rppb
