// The streaming peak finder of the recorded trajectories: sample by sample, and
// by blocks of samples.  Host and device code (the block form is compared with
// the sample form on the CPU).
#pragma once

#include <cuda_runtime.h>
#include <limits.h>
#include <string.h>

namespace cbf {
namespace {

// ---------------------------------------------------------------------------
// Streaming restatement of peakFinder (cudaLibrary.cu:220-266) over the samples
// d[0..N) in arrival order.  Candidate i is judged when d[i+1] arrives:
//   NORMAL : d[i] > d[i-1] (`rising`) && d[i] >= d[i+1] -> peak at i if d[i] > d[i+1],
//            otherwise a plateau begins (inner loop of :229-246);
//   PLATEAU: compare the plateau value with the next sample: larger -> peak at
//            the plateau end j; smaller -> no peak; equal -> continue;
//   SKIP   : after a peak or a rising plateau the reference sets i = j+1 and its
//            ++i moves on to j+2, so the next arrival is not a candidate.
// The first detected peak is dropped and intervals are (t[k+1]-t[k]) * 0.01
// (:250-262).  NaN is absorbing for these systems, so the inner loop's
// run-to-the-end case never yields a peak, as here.
constexpr double kPeakIntervalUnit = 0.01;  // peakFinder's default h (cudaLibrary.cuh:204)

__host__ __device__ __forceinline__ int highest_bit(unsigned v)
{
#ifdef __CUDA_ARCH__
    return 31 - __clz(v);
#else
    return 31 - __builtin_clz(v);
#endif
}

// The rises of a block of K samples, collected as they come: bit K-1-i is set where
// sample i + 1 of the block is above sample i, sample 0 being the one before the
// block.  The sign of the difference p - v says so -- a subtraction of different
// numbers is never 0, and 0 has no sign bit -- with one exception: (-0) - (+0) is -0.
// A difference whose high word is the sign alone is that, or a negative number below
// 2^-1042, so the smallest high word tells whether the signs can be trusted; where
// they cannot, the block's samples are compared.  The minimum takes two samples an
// instruction; it costs the 1024^2 DBSCAN map 1 of 147 ms (without it 146, with wrong
// peaks from trajectories that start on -0).
template <int K>
struct RiseMask {
    unsigned signs;
    int least;

    __host__ __device__ __forceinline__ void init()
    {
        signs = 0;
        least = INT_MAX;
    }
    // Sample v after sample p: the difference's high word, to be given to seen().
    __host__ __device__ __forceinline__ int add(double p, double v)
    {
        const double d = p - v;
#ifdef __CUDA_ARCH__
        const int hi = __double2hiint(d);
        signs = __funnelshift_l((unsigned)hi, signs, 1);
#else
        long long b;
        memcpy(&b, &d, sizeof(b));
        const int hi = (int)(b >> 32);
        signs = signs << 1 | (unsigned)hi >> 31;
#endif
        return hi;
    }
    __host__ __device__ __forceinline__ void seen(int hi1, int hi2)
    {
#ifdef __CUDA_ARCH__
        least = __vimin3_s32(least, hi1, hi2);
#else
        least = hi1 < least ? hi1 : least;
        least = hi2 < least ? hi2 : least;
#endif
    }
    // The mask of the first m samples after ring[0], all of them added and seen.
    __host__ __device__ __forceinline__ unsigned mask(int m, const double* ring) const
    {
        if (least != INT_MIN) return signs << (K - m);
        unsigned up = 0;
#pragma unroll 1
        for (int i = 0; i < m; ++i) up = up << 1 | (ring[32 * i + 32] > ring[32 * i] ? 1u : 0u);
        return up << (K - m);
    }
};

struct NoPeakHook {
    __host__ __device__ __forceinline__ void operator()(double, int) const {}
    __host__ __device__ __forceinline__ void finish(double) {}
};

// Flags of peakFinderCUDAForCalculationOfPeriodicityByOstrovsky
// (cudaLibrary.cu:288-352) kept while the peaks stream by, over every peak:
// non-increasing consecutive peaks (flag 0), peaks from the second on above /
// not above the threshold (flags 1, 2), and the last recorded sample (flag 4).
struct OstrovskyFlags {
    double prev, last, thr;
    bool nonInc, one, zero;
    __host__ __device__ __forceinline__ void init(double threshold)
    {
        thr = threshold;
        prev = last = 0.0;
        nonInc = true;
        one = zero = false;
    }
    __host__ __device__ __forceinline__ void operator()(double val, int k)
    {
        if (k >= 1) {
            if (val - prev > 0) nonInc = false;
            if (val > thr) one = true;
            else zero = true;
        }
        prev = val;
    }
    __host__ __device__ __forceinline__ void finish(double sample) { last = sample; }
};

struct PeakStream {
    double prev1, pval;  // last sample; value of the running plateau
    int mode;            // 0 NORMAL, 1 PLATEAU, 2 SKIP
    int rising;          // prev1 was above its predecessor
    int detected;
    int lastT;

    __host__ __device__ __forceinline__ void init()
    {
        prev1 = pval = 0.0;
        mode = rising = 0;
        detected = 0;
        lastT = 0;
    }

    // hook(value, k) sees every emitted peak k = 0, 1, ... (also past cap).
    template <bool WITH_INTERVALS, class Hook>
    __host__ __device__ __forceinline__ void emit(double val, int t, double* pk, double* iv, int cap, Hook& hook)
    {
        if (detected >= 1) {
            const int k = detected - 1;
            hook(val, k);
            if (k < cap) {
                pk[k] = val;
                if (WITH_INTERVALS) iv[k] = (double)(t - lastT) * kPeakIntervalUnit;
            }
        }
        lastT = t;
        ++detected;
    }

    template <bool WITH_INTERVALS>
    __host__ __device__ __forceinline__ void push(double v, int t, double* pk, double* iv, int cap)
    {
        NoPeakHook h;
        push<WITH_INTERVALS>(v, t, pk, iv, cap, h);
    }

    template <bool WITH_INTERVALS, class Hook>
    __host__ __device__ __forceinline__ void push(double v, int t, double* pk, double* iv, int cap, Hook& hook)
    {
        if (mode == 2) {
            mode = 0;
        } else if (mode == 1) {
            if (pval < v) {
                mode = 2;
            } else if (pval > v) {
                emit<WITH_INTERVALS>(pval, t - 1, pk, iv, cap, hook);
                mode = 2;
            }
        } else if (rising && prev1 >= v) {
            if (prev1 > v) {
                emit<WITH_INTERVALS>(prev1, t - 1, pk, iv, cap, hook);
                mode = 2;
            } else {
                mode = 1;
                pval = prev1;
            }
        }
        rising = t > 0 && v > prev1;
        prev1 = v;
    }

    // m <= K samples at once: the samples of times t+1 .. t+m (prev1 is time t's),
    // all of them numbers, in ring[32 * 1] .. ring[32 * m] with time t's in ring[0];
    // `up`: the block's rises (RiseMask).  Equal to m calls of push().  A candidate
    // arrival is one that does not rise after one that did.  The SKIP after a peak is
    // implied -- a sample right after a descent cannot be such an arrival -- so only
    // plateaus need the state.
    template <int K, bool WITH_INTERVALS, class Hook>
    __host__ __device__ __forceinline__ void push_block(unsigned up, int t, int m, double last, const double* ring,
                                                        double* pk, double* iv, int cap, Hook& hook)
    {
        unsigned cand = after_rise<K>(up) & ~up & arrivals<K>(m);
        if (mode != 0) cand = plateau<K, WITH_INTERVALS>(mode == 2 ? -1 : 0, cand, t, m, ring, pk, iv, cap, hook);
        while (cand) {
            const int b = highest_bit(cand);
            const int i = K - 1 - b;
            cand &= ~(1u << b);
            const double a = ring[32 * i], v = ring[32 * i + 32];
            if (a > v) {
                emit<WITH_INTERVALS>(a, t + i, pk, iv, cap, hook);
            } else {
                mode = 1;
                pval = a;
                cand = plateau<K, WITH_INTERVALS>(i + 1, cand, t, m, ring, pk, iv, cap, hook);
            }
        }
        rising = (int)((up >> (K - m)) & 1u);
        prev1 = last;
    }

    // Arrivals whose predecessor rose (bits as in `up`), and the first m arrivals.
    template <int K>
    __host__ __device__ __forceinline__ unsigned after_rise(unsigned up) const
    {
        return (((unsigned)rising << K) | up) >> 1;
    }
    template <int K>
    __host__ __device__ __forceinline__ static unsigned arrivals(int m)
    {
        return ((1u << K) - 1u) & ~((1u << (K - m)) - 1u);
    }

private:
    // Arrivals j, j+1, .. of the block against the running plateau; returns the
    // candidates with the arrival after the plateau's end taken out (SKIP).
    // j = -1: the plateau ended at the last arrival before the block.
    template <int K, bool WITH_INTERVALS, class Hook>
    __host__ __device__ unsigned plateau(int j, unsigned cand, int t, int m, const double* ring, double* pk,
                                         double* iv, int cap, Hook& hook)
    {
        for (; mode == 1 && j < m; ++j) {
            const double v = ring[32 * j + 32];
            if (v == pval) continue;
            if (v < pval) emit<WITH_INTERVALS>(pval, t + j, pk, iv, cap, hook);
            mode = 2;
            break;
        }
        if (mode == 2 && j + 1 < m) {
            mode = 0;
            cand &= ~(1u << (K - 2 - j));
        }
        return cand;
    }

public:
    __host__ __device__ __forceinline__ int emitted() const { return detected > 1 ? detected - 1 : 0; }
};

}  // namespace
}  // namespace cbf
