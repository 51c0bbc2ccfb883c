// Per-point device code of the fused bifurcation kernel: the streaming peak
// finder, the per-point integration and the warp-cooperative KDE / DBSCAN
// epilogues.  Shared by the map kernel (bif.cu) and the batch kernel (batch.cu).
#pragma once

#include <type_traits>

#include "engine.cuh"
#include "peak_stream.cuh"

namespace cbf {
namespace {

constexpr unsigned kFull = 0xffffffffu;

// dbscanCUDAForCalculationOfPeriodicityByOstrovsky (cudaLibrary.cu:628-662):
// the cluster count (dbscanDouble = dbscan as a double) rewritten by the flags.
// A diverged point has flag 3 only: the reference never writes its other flags,
// which are false on zero-filled memory.
__device__ __forceinline__ double ostrovsky_value(int n, bool div, const OstrovskyFlags& f, int clusters)
{
    bool f0, f1, f2, f3, f4;
    if (div) {
        f0 = f1 = f2 = f4 = false;
        f3 = true;
    } else {
        f0 = f.nonInc;
        f1 = f.one && f.zero;
        f2 = !(f.one && !f.zero);
        f3 = (n == 0 || n == 1);
        f4 = f.last > f.thr;
    }
    double out = (double)clusters;
    if (f2) out = -1 * out;
    if (f3) out = f4 ? 1 : -1;
    if (f1) out = 0;
    if (f0) out = out > 0 ? 0.5 : (out == 0 ? 0 : -0.5);
    return out;
}

// Tasks whose peaks carry intervals (DBSCAN on (peak, interval) pairs).
__host__ __device__ constexpr bool task_with_intervals(int task)
{
    return task == CBF_TASK_DBSCAN || task == CBF_TASK_OSTROVSKY;
}

template <int D>
__device__ __forceinline__ double pick(const double (&x)[D], int wv)
{
    double r = x[0];
#pragma unroll
    for (int i = 1; i < D; ++i)
        if (i == wv) r = x[i];
    return r;
}

// The recorded variable of a state, physical; WV >= 0 fixes it at compile time.
template <class S, int WV>
__device__ __forceinline__ double sample_of(const double (&x)[S::DIM], int wv, const typename S::Coef& c)
{
    if constexpr (WV >= 0) return phys_comp<S>(x[WV], WV, c);
    else return phys_comp<S>(pick<S::DIM>(x, wv), wv, c);
}

// Samples per block of the recorded loop, and the shared memory of a warp for
// one block: rows 0..kRing of 32 doubles (row 0: the sample before the block).
constexpr int kRing = 16;
constexpr int kRingWords = (kRing + 1) * 32 * 2;
static_assert(kRingWords % 4 == 0, "every warp's shared words start on a 16-byte boundary");

// What the recorded loop needs of a job.
struct RecordSpec {
    int n, extra;     // samples; steps per sample - 1
    int wv;
    int checkDiv;
    unsigned hiT;     // high word a sample must stay below in a block
    int cap;          // peak slots of pk (and iv)
    double divThresh;
};

template <class S>
struct StateOf {
    double x[S::DIM];
};

// The recorded loop (cudaLibrary.cu:110-114) feeding the peak stream; sample 0
// is the state on entry.  Returns true if the divergence test fired.
//
// Bound: the FP64 step's operand reads.  Judging every sample as it arrives (two
// FP64 comparisons, the divergence test, the state machine's branches) cost more
// than the step: 103 ms for 40 000 samples x 1024^2 Lorenz points where 100 000
// bare steps take 72 ms.  So samples are taken in blocks of kRing: per sample one
// FP64 subtraction whose sign bit (d[i] above d[i-1]) is shifted into a mask
// (RiseMask), one shared-memory store, half a three-input minimum for the mask and
// half a three-input maximum against the threshold; the block's peaks then follow
// from the mask's few candidates (44 ms; the 1024^2 DBSCAN map 256 -> 205 ms, a
// ragged batch 112 -> 86 ms).  A block in which a sample may have reached the
// divergence threshold or is no number is repeated from its first state with the
// exact per-sample code; so is the end of the record.
template <class S, int WV, bool PRE1, bool WITH_INTERVALS, class Hook>
__device__ __forceinline__ bool record_loop(const RecordSpec& R, double (&x)[S::DIM], const typename S::Coef& c,
                                            PeakStream& ps, double* ring, double* pk, double* iv, Hook& hook)
{
    constexpr int D = S::DIM;
    const int n = R.n;
    auto next = [&]() {
        if (!PRE1)
            for (int j = 0; j < R.extra; ++j) S::step(x, c);
        S::step(x, c);
        return sample_of<S, WV>(x, R.wv, c);
    };
    if (n <= 0) return false;
    int t = 0;  // the last sample fed
    ps.push<WITH_INTERVALS>(sample_of<S, WV>(x, R.wv, c), 0, pk, iv, R.cap, hook);
    while (t < n) {  // step t leads to sample t+1; the last one is only tested
        int m = n - t;
        if (m > kRing) {
            double x0[D];
#pragma unroll
            for (int i = 0; i < D; ++i) x0[i] = x[i];
            HiTrack tr;
            tr.init();
            RiseMask<kRing> rises;
            rises.init();
            double p = ps.prev1;
            ring[0] = p;
#pragma unroll (D == 5 ? 1 : 2)
            for (int i = 0; i < kRing; i += 2) {
                const double a = next();
                const int up = rises.add(p, a);
                ring[32 * i + 32] = a;
                p = next();
                rises.seen(up, rises.add(a, p));
                ring[32 * i + 64] = p;
                tr.add2(a, p);
            }
            if (!tr.maybe(R.hiT)) {
                ps.push_block<kRing, WITH_INTERVALS>(rises.mask(kRing, ring), t, kRing, p, ring, pk, iv, R.cap, hook);
                t += kRing;
                continue;
            }
#pragma unroll
            for (int i = 0; i < D; ++i) x[i] = x0[i];
            m = kRing;
        }
        for (int i = 0; i < m; ++i) {
            const double v = next();
            if (R.checkDiv && diverged(v, R.divThresh)) return true;
            if (++t < n) ps.push<WITH_INTERVALS>(v, t, pk, iv, R.cap, hook);
            if (isnan(v)) return false;  // absorbing: no later sample is a peak or passes the test
        }
    }
    return false;
}

// The recorded loop of one point from state `st`: the emitted peak count, -1 if
// the divergence test fired.  A function of its own, called once per point: its
// registers are not those of the epilogues around it, and one copy serves all
// tasks of a kernel.
template <class S, bool WITH_INTERVALS, class Hook>
__device__ __noinline__ int record_point(const RecordSpec R, StateOf<S> st, const typename S::Coef c, double* ring,
                                         double* pk, double* iv, Hook* hookIO)
{
    Hook hook = *hookIO;
    PeakStream ps;
    ps.init();
    bool div;
    auto go = [&](auto wv) {
        constexpr int WV = decltype(wv)::value;
        return R.extra == 0 ? record_loop<S, WV, true, WITH_INTERVALS>(R, st.x, c, ps, ring, pk, iv, hook)
                            : record_loop<S, WV, false, WITH_INTERVALS>(R, st.x, c, ps, ring, pk, iv, hook);
    };
    if constexpr (S::DIM == 3) {
        if (R.wv == 0) div = go(std::integral_constant<int, 0>());
        else if (R.wv == 1) div = go(std::integral_constant<int, 1>());
        else div = go(std::integral_constant<int, 2>());
    } else {
        div = go(std::integral_constant<int, -1>());
    }
    if (R.n > 0) hook.finish(ps.prev1);
    *hookIO = hook;
    return div ? -1 : ps.emitted();
}

// One point: transient (unchecked, cudaLibrary.cu:107-108), then the recorded
// loop (:110-114) feeding the peak stream.  Returns the emitted peak count, 0 on
// divergence (peakFinderCUDA turns the -1 flag into 0, :277-281).  `ring`: this
// lane's column of the warp's kRingWords (not used by TRAJECTORY).
template <class S, int TASK>
__device__ int integrate_point(const DevJob& J, long long g, double* pk, double* iv, int cap,
                               double* traj, int* divFlag, double* ring, OstrovskyFlags* of = nullptr)
{
    constexpr int D = S::DIM;
    StateOf<S> st;
    typename S::Coef c;
    {
        double v[CBF_MAX_VALUES];
        setup_point<D>(J, g, st.x, v);
        c = S::prep(v, J.h);
        to_stored<S>(st.x, c);
    }

#pragma unroll (D == 5 ? 1 : 4)
    for (int i = 0; i < J.nSkip; ++i) S::step(st.x, c);

    if constexpr (TASK == CBF_TASK_TRAJECTORY) {
        const int wv = J.writableVar;
        bool div = false;
        int t = 0;
        for (; t < J.nRecord; ++t) {
            traj[t] = phys_comp<S>(pick<D>(st.x, wv), wv, c);
            for (int j = 0; j < J.preScaller - 1; ++j) S::step(st.x, c);
            S::step(st.x, c);
            if (J.checkDiv && diverged(phys_comp<S>(pick<D>(st.x, wv), wv, c), J.divThresh)) {
                div = true;
                ++t;
                break;
            }
        }
        // Samples after a divergence are never written by the reference; make them NaN.
        for (; t < J.nRecord; ++t) traj[t] = __longlong_as_double(0x7ff8000000000000ll);
        *divFlag = div ? 1 : 0;
        return 0;
    } else {
        const RecordSpec R{J.nRecord, J.preScaller - 1, J.writableVar, J.checkDiv,
                           J.checkDiv ? J.divHi : 0x7f800000u, cap, J.divThresh};
        int n;
        if constexpr (TASK == CBF_TASK_OSTROVSKY) {
            n = record_point<S, true, OstrovskyFlags>(R, st, c, ring, pk, iv, of);
            *divFlag = n < 0 ? 1 : 0;
        } else {
            NoPeakHook hook;
            n = record_point<S, task_with_intervals(TASK), NoPeakHook>(R, st, c, ring, pk, iv, &hook);
        }
        return n < 0 ? 0 : n;
    }
}

// ---------------------------------------------------------------------------
// KDE mode count of one point (kde, cudaLibrary.cu:356-422), whole warp.
//
// The count is a function of the signs of d(w+1) - d(w) alone, d(w) the kernel
// sum at sample w.  The exact sum -- FP64 differences, FP32 expf, a double
// accumulator, the reference's peak order -- costs about 50 issue cycles a term
// (six FP64 instructions and two conversions to and from double, which run at a
// quarter of that rate), and made the map's epilogue three times its integration
// (331 ms of 440 for the 1024^2 Lorenz map with 4 samples per peak).  So the signs
// are first settled by FP32 sums with an error bound (kde_fast_sum: one
// subtraction, one square, one ex2 and one addition a term), over peaks sorted
// once per point so that a chunk of samples meets one window of them; a pair of
// samples whose difference is within the two bounds is settled by the exact
// sums (the same map: 440 -> 302 ms; a point takes 27 chunks and 1400 FP32 terms
// instead of 50 and 7000 exact ones).  Windows of 6 bandwidths first (what lies outside adds at most e^-18 a
// peak), of 16 next (outside, the exact terms are +0 too), the exact sums last.
constexpr int kKdeSortCap = 1024;  // peaks a warp sorts (its ring words hold them)
constexpr double kKdeNear = 6.0, kKdeFar = 16.0;         // window half-widths in bandwidths
constexpr double kKdeScale = 0.84932180028801904;       // sqrt(log2(e) / 2)
constexpr float kKdeDropped = 1.6e-8f;                  // above e^(-kKdeNear^2 / 2)

// The exact sum at this lane's sample `delt`, the warp's samples lying in
// [dlo, dhi].  Rounded subtraction is monotone, so a peak with fl(p - dhi) > skip
// or fl(p - dlo) < -skip has |fl(p - delt)| > skip for every lane, i.e. it adds
// exactly +0 everywhere.  One ballot per 32 peaks drops those; the rest are summed
// in ascending m.  A NaN bound fails both comparisons and keeps every peak.
__device__ __noinline__ double kde_exact_sum(const double* pk, int n, double delt, double dlo, double dhi,
                                             double skip, double H, double invH, bool active, int lane)
{
    double d2 = 0;
    for (int g = 0; g < n; g += 32) {
        const int m = g + lane;
        const double pv = m < n ? pk[m] : 0.0;
        const bool near = m < n && !(pv - dhi > skip) && !(pv - dlo < -skip);
        unsigned mask = __ballot_sync(kFull, near);
        while (mask) {
            const int j = __ffs(mask) - 1;
            mask &= mask - 1;
            const double dd = __shfl_sync(kFull, pv, j) - delt;
            // |dd| > 16|H| makes the FP32 exponent argument <= -128, where expf
            // is exactly +0 (checked exhaustively on the device by
            // cbf_probe_expf_zero), and adding +0 leaves the sum unchanged.
            if (active && !(fabs(dd) > skip)) {
                const double tmp = invH != 0.0 ? dd * invH : dd / H;
                d2 += (double)expf((float)(-((tmp * tmp) / 2)));
            }
        }
    }
    return d2;
}

// Peaks of one point as sorted floats: key[i] = (p - mid) * scale in ascending
// order, scale = kKdeScale / |H| (so a term is 2^-(key - x)^2), padded with +inf
// to P, a power of two >= 32.
struct KdeSorted {
    const float* key;
    int n;
    double mid, scale;
    float qmax;   // largest |key|
    float weight; // peaks per key
};

// Sorts the peaks into key[0..P) (shared); false where the FP32 sums would not
// do: not every value finite, or keys too large for the bound to be of use.
__device__ bool kde_sort(float* key, const double* pk, int n, double H, int lane, KdeSorted& ks)
{
    double lo = INFINITY, hi = -INFINITY;
    bool bad = false;
    for (int m = lane; m < n; m += 32) {
        const double v = pk[m];
        bad |= !isfinite(v);
        lo = fmin(lo, v);
        hi = fmax(hi, v);
    }
    if (__any_sync(kFull, bad)) return false;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo = fmin(lo, __shfl_xor_sync(kFull, lo, o));
        hi = fmax(hi, __shfl_xor_sync(kFull, hi, o));
    }
    ks.n = n;
    ks.key = key;
    ks.mid = lo + (hi - lo) * 0.5;
    ks.scale = kKdeScale / fabs(H);
    const double span = (hi - lo) * ks.scale;
    if (!(span < 1e5) || !(fabs(ks.mid) < 1e100)) return false;
    ks.qmax = (float)(span * 0.5) * 1.001f + 1e-6f;
    ks.weight = 1.0f;
    int P = 32;
    __syncwarp();
    if (span < 0x1p-18) {
        // one value but for its last bits (a fixed point's wobble, thousands of
        // peaks): one key of weight n; |key - 0| <= qmax enters the bound
        key[lane] = lane == 0 ? 0.0f : INFINITY;
        ks.n = 1;
        ks.weight = (float)n;
        __syncwarp();
        return true;
    }
    while (P < n) P <<= 1;
    for (int m = lane; m < P; m += 32) key[m] = m < n ? (float)((pk[m] - ks.mid) * ks.scale) : INFINITY;
    __syncwarp();
    for (int size = 2; size <= P; size <<= 1) {
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            for (int t = lane; t < (P >> 1); t += 32) {
                const int i = 2 * t - (t & (stride - 1));
                const float ki = key[i], kj = key[i + stride];
                const float mn = fminf(ki, kj), mx = fmaxf(ki, kj);
                const bool up = (i & size) == 0;
                key[i] = up ? mn : mx;
                key[i + stride] = up ? mx : mn;
            }
            __syncwarp();
        }
    }
    return true;
}

// Keys below x among key[0..n), whole warp: the last key of each of 32 segments,
// then the same within the first segment whose last key is not below.
__device__ __forceinline__ int kde_below(const KdeSorted& ks, float x, int lane)
{
    int at = 0, len = ks.n;
    for (;;) {
        const int seg = (len + 31) >> 5;
        const int end = min((lane + 1) * seg, len);  // of this lane's segment, if not empty
        const bool below = lane * seg < len && ks.key[at + end - 1] < x;
        const int c = __popc(__ballot_sync(kFull, below)) * seg;
        if (seg == 1 || c >= len) return at + min(c, len);
        at += c;
        len = min(seg, len - c);
    }
}

__device__ __forceinline__ float ex2_ftz(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// The FP32 sum at x over the peaks of key[lo..hi) (and up to three on either
// side, +inf among them: true terms, or 0), four at a time; *least: the smallest
// squared distance met.
__device__ __forceinline__ float kde_fast_sum(const KdeSorted& ks, int lo, int hi, float x, float* least)
{
    float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f, s0 = INFINITY, s1 = INFINITY;
    for (int m = lo & ~3; m < hi; m += 4) {
        const float4 q = *reinterpret_cast<const float4*>(ks.key + m);
        const float u0 = q.x - x, u1 = q.y - x, u2 = q.z - x, u3 = q.w - x;
        const float v0 = u0 * u0, v1 = u1 * u1, v2 = u2 * u2, v3 = u3 * u3;
        s0 = fminf(s0, fminf(v0, v1));
        s1 = fminf(s1, fminf(v2, v3));
        a0 += ex2_ftz(-v0);
        a1 += ex2_ftz(-v1);
        a2 += ex2_ftz(-v2);
        a3 += ex2_ftz(-v3);
    }
    *least = fminf(s0, s1);
    return (a0 + a1) + (a2 + a3);
}

// Bound of |fast sum - exact sum| relative to the sum, for `terms` terms with
// |key - x| <= U, |key| <= Q, |x| <= X, in units of 2^-24:
//   key and x are rounded (Q + X), so is their difference (U), and a key of
//   weight n lies within 64 units of its peaks: the exponent u^2 is off by
//   2U(Q + X + U + 64) and its own rounding U^2; the exact exponent is rounded to
//   FP32 (U^2); ln 2 times that, plus 2^-22 for ex2.approx and 2 ulp for expf
//   (4 + 4), and the additions of four partial sums.
// Terms with U^2 > 126 are at most 2^-126 on either side (absolute bound).
__device__ __forceinline__ float kde_rel_bound(float U, float Q, float X, int terms, float spread)
{
    U = fminf(U, 11.3f);
    const float e = 0.6932f * (2.0f * U * (Q + X + U + spread) + 2.0f * U * U) + 8.0f + 0.25f * (float)terms + 4.0f;
    return 1.05f * 0x1p-24f * e;
}

// What the KDE epilogue needs of a job.
struct KdeSpec {
    double i1, i2, H, skip, invH;
    int maxPeaks, sampling, fixed;
};

__device__ __forceinline__ KdeSpec kde_spec(const DevJob& J)
{
    return KdeSpec{J.kdeI1, J.kdeI2, J.kdeH, J.kdeSkip, J.kdeInvH, J.maxPeaks, J.kdeSampling, J.kdeFixed};
}

// The count of a point that its number of peaks alone decides (-1: it does not).
__device__ __forceinline__ int kde_by_count(int n, int maxPeaks)
{
    return n == 0 ? 0 : n <= 2 ? 1 : n > maxPeaks ? maxPeaks : -1;
}

// `keys`: room for keyCap floats of this warp, a power of two >= 32, 16-byte
// aligned; in shared memory (SHARED) or in global memory.  A function of its own,
// like the recorded loop: its registers are not the integration's.
template <bool SHARED>
__device__ __noinline__ int kde_warp(const KdeSpec J, const double* pk, int n, int lane, float* keys, int keyCap)
{
    float* key = SHARED ? static_cast<float*>(__cvta_shared_to_generic(__cvta_generic_to_shared(keys))) : keys;
    if (n <= 2 || n > J.maxPeaks) return kde_by_count(n, J.maxPeaks);

    const double k1 = J.fixed ? (double)J.sampling : (double)(J.sampling * n);
    const double k2 = (J.i2 - J.i1) / (k1 - 1);
    // `for (int w = 0; w < k1 - 1; ++w)`: k1 is integral, so W = k1 - 1 iterations.
    const int W = (k1 - 1 > 0) ? (int)ceil(k1 - 1) : 0;
    const double skip = J.skip, H = J.H, invH = J.invH;

    // FP32 sums where they can decide: a usable bandwidth and interval, no more
    // peaks than a warp sorts, and a bound of their error well below 1.
    KdeSorted ks;
    bool fast = n <= keyCap && W > 2 && fabs(H) > 1e-30 && fabs(H) < 1e30 && fabs(J.i1) < 1e100 &&
                fabs(J.i2) < 1e100 && k2 != 0 && kde_sort(key, pk, n, H, lane, ks);
    float width = 0.f, spread = 0.f;  // a chunk's extent, and a key's, in key units
    if (fast) {
        width = (float)(31.0 * fabs(k2) * ks.scale);
        spread = ks.n == 1 ? 64.0f : 0.0f;  // 2^-18 in units of 2^-24
        fast = kde_rel_bound(11.3f, ks.qmax, ks.qmax + 14.0f + width, n, spread) < 0x1p-6f;
    }

    int res = 0;
    bool prevUp = false, strange = false, lastUp = false;
    // Samples in chunks of 32, each starting with its predecessor's last: pairs
    // (lane, lane + 1) for lane < cnt - 1.
    for (int base = 0; base < W - 1 || base == 0; base += 31) {
        if (W == 0) break;
        const int w = base + lane;
        const int cnt = min(32, W - base);
        const double delt = w * k2 + J.i1;
        // delt is monotone in w (rounded products and sums are)
        const double dFirst = __shfl_sync(kFull, delt, 0);
        const double dLast = __shfl_sync(kFull, delt, cnt - 1);
        const double dlo = k2 >= 0 ? dFirst : dLast;
        const double dhi = k2 >= 0 ? dLast : dFirst;
        const bool pair = lane < cnt - 1;
        bool up = false, eq = false;
        unsigned open = cnt > 1 ? (0xffffffffu >> (33 - cnt)) : 0u;  // pairs whose sign is not settled
        if (fast) {
            const float x = (float)((delt - ks.mid) * ks.scale);
            const float xlo = (float)((dlo - ks.mid) * ks.scale), xhi = (float)((dhi - ks.mid) * ks.scale);
            // beyond 16 bandwidths (and the roundings of key and x) of every
            // peak the exact sums are +0: all equal
            const float reach = (float)(kKdeFar * kKdeScale) + 0.05f;
            if (fmaxf(-ks.qmax - xhi, xlo - ks.qmax) > reach) {
                eq = pair;
                open = 0;
            }
#pragma unroll 1
            for (int tier = 0; tier < 2 && open; ++tier) {
                const float half = tier == 0 ? (float)(kKdeNear * kKdeScale) : reach;
                const int lo = kde_below(ks, xlo - half, lane);
                const int hi = kde_below(ks, xhi + half, lane);
                float least;
                const float a = kde_fast_sum(ks, lo, hi, x, &least) * ks.weight;
                float e = a * kde_rel_bound(half + width + 1.0f, ks.qmax, ks.qmax + 14.0f + width, hi - lo + 6, spread) +
                          (float)n * 0x1p-125f;
                if (tier == 0) e += (float)(ks.n - (hi - lo)) * ks.weight * kKdeDropped;
                else if (least > reach * reach) e = 0.f;  // no peak in reach: +0, exactly
                const float an = __shfl_down_sync(kFull, a, 1), en = __shfl_down_sync(kFull, e, 1);
                up = an > a;
                eq = a == 0.f && an == 0.f && e == 0.f && en == 0.f;
                // 1.0001: the roundings of e + en and an - a themselves
                const bool sure = eq || fabsf(an - a) > (e + en) * 1.0001f;
                open = __ballot_sync(kFull, pair && !sure);
            }
        }
        bool nan = false;
        if (open || W == 1) {
            // exact sums of the samples of open pairs
            const unsigned act = W == 1 ? 1u : open | (open << 1);
            const double d0 = __shfl_sync(kFull, delt, __ffs(act) - 1);
            const double d1 = __shfl_sync(kFull, delt, highest_bit(act));
            const double d = kde_exact_sum(pk, n, delt, k2 >= 0 ? d0 : d1, k2 >= 0 ? d1 : d0, skip, H, invH,
                                           (act >> lane) & 1u, lane);
            const double dn = __shfl_down_sync(kFull, d, 1);
            if ((open >> lane) & 1u) {
                up = dn > d;
                eq = dn == d;
                nan = !(up || eq || dn < d);
            }
            if (W == 1) lastUp = __shfl_sync(kFull, d, 0) > 0;
        }
        const unsigned pm = cnt > 1 ? (0xffffffffu >> (33 - cnt)) : 0u;
        const unsigned U = __ballot_sync(kFull, up && pair), E = __ballot_sync(kFull, eq && pair);
        const unsigned N = __ballot_sync(kFull, nan && pair);
        if (cnt <= 1) break;
        if (!(E | N) && !strange) {
            // maxima: a rise and then a descent
            res += __popc(((U << 1) | (prevUp ? 1u : 0u)) & ~U & pm);
            prevUp = (U >> (cnt - 2)) & 1u;
        } else if (E == pm) {  // level throughout
            strange |= prevUp;
            prevUp = false;
        } else {
            // the reference's plateau states, pair by pair
            for (int j = 0; j < cnt - 1; ++j) {
                const bool u = (U >> j) & 1u, q = (E >> j) & 1u, d = !u && !q && !((N >> j) & 1u);
                if (strange) {
                    if (u) strange = false;
                    else if (d) { strange = false; ++res; }
                } else if (prevUp && d) {
                    ++res;
                } else if (prevUp && q) {
                    strange = true;
                }
                prevUp = u;
            }
        }
        lastUp = prevUp;
    }
    if (lastUp) ++res;
    return res;
}

// ---------------------------------------------------------------------------
// DBSCAN (dbscan, cudaLibrary.cu:457-529), whole warp per point.
//
// helpfulArray[k] (label, nonzero once set) -> bitset L; helpfulArray[n+k] (the
// "stack", holds k or 0) -> bitset S: popping slot m yields m if set, else 0.
// One scan of a centre c adds to L and S exactly the set
//     {k < n-1 : k != c, k unlabelled, near(c, k)}
// and counts it into the stack depth.  The reference visits k in ascending
// order, but each k once, and nothing it sets is read again within the scan,
// so the order is immaterial.  Three facts make most scans avoidable without
// changing any label, stack bit or count:
//   * a scan of a centre with no near k at all adds nothing ("scan-empty");
//   * a second scan of a centre adds nothing (its near k are all labelled
//     after the first, and labels are never cleared);
//   * once every k < n-1 is labelled, no scan adds anything.
// A neighbour has |fl(p_k - p_c)| < skip (skip = 4 eps bounds the FP32 hypot
// from below), hence p_k in [A, B] = p_c -/+ (2 skip + 4 ulp(p_c)) (rounded).
// The peaks are sorted by a 32-bit key: the top 22 bits of an order-preserving
// encoding of float(p_k) over the 10-bit index k.  Rounding to float and
// truncating are monotone, so every candidate's key lies between the keys of A
// and B: one window of sorted positions.  The scan-empty marks come from a few
// probes per peak, and a real scan tests the window only, each candidate with
// the exact test.  Chaotic points -- hundreds of peaks, almost all of them
// singleton clusters -- then cost a sort and a word-wise walk instead of n
// scans over n peaks.
constexpr int kDbscanIdxBits = 10;
constexpr int kDbscanSortCap = 1 << kDbscanIdxBits;  // scanned peaks (n - 1) a warp sorts
constexpr unsigned kDbscanIdxMask = (1u << kDbscanIdxBits) - 1u;
constexpr int kDbscanProbes = 32;  // per peak, in the scan-empty test; more: not marked

struct DbscanSort {
    unsigned* key = nullptr;  // sorted (coarse value << 10 | index)
    unsigned* E = nullptr;    // scan-empty marks (bitset)
    unsigned* D = nullptr;    // centres scanned once (bitset)
    int cap = 0;              // entries of key; 0: no sorted path
};

// 32-bit words of shared memory per warp: the bitsets L and S of `bitWords`
// words each, and with `sortCap` > 0 (a power of two, 32..1024) also E, D and
// the sort keys.  The recorded loop's ring and the KDE epilogue's sorted peaks lie
// in the same words (a warp's epilogues start when all its lanes have integrated).
// A multiple of four words: every warp's start is 16-byte aligned.
__host__ __device__ inline int dbscan_warp_words(int bitWords, int sortCap)
{
    const int w = ((sortCap > 0 ? 4 * bitWords + sortCap : 2 * bitWords) + 3) & ~3;
    return w > kRingWords ? w : kRingWords;
}

// This lane's column of the ring that starts at the warp's shared words.
__device__ __forceinline__ double* ring_column(unsigned* warpWords, int lane)
{
    return reinterpret_cast<double*>(warpWords) + lane;
}

// Sort keys per warp for peak lists of up to `peakCap` peaks: a power of two
// >= 32, or 0 (no sorted path) when peakCap exceeds kDbscanSortCap.
__host__ __device__ inline int dbscan_sort_cap(int peakCap)
{
    if (peakCap > kDbscanSortCap) return 0;
    int c = 32;
    while (c < peakCap) c <<= 1;
    return c;
}

__device__ inline DbscanSort dbscan_sort_area(unsigned* warpWords, int bitWords, int sortCap)
{
    DbscanSort so;
    if (sortCap > 0) {
        so.E = warpWords + 2 * bitWords;
        so.D = so.E + bitWords;
        so.key = so.D + bitWords;
        so.cap = sortCap;
    }
    return so;
}

// Top 22 bits of an order-preserving encoding of float(v): non-decreasing in v
// (-0 is folded onto +0).
__device__ __forceinline__ unsigned dbscan_coarse(double v)
{
    float f = (float)v;
    if (f == 0.0f) f = 0.0f;
    const unsigned u = __float_as_uint(f);
    return ((u & 0x80000000u) ? ~u : (u | 0x80000000u)) >> kDbscanIdxBits;
}

// distance(...) < eps of the reference (cudaLibrary.cu:445-453) with c = (x1, y1)
// the centre: 0 on exact equality, else the FP32 hypot of the double
// differences.  hypotf(dx, dy) >= max(|dx|, |dy|) up to a few ulps, so a
// coordinate gap >= skip = 4 eps can never be closer than eps.
__device__ __forceinline__ bool dbscan_near(double x1, double y1, double x2, double y2, double eps,
                                            double skip)
{
    if (x1 == x2 && y1 == y2) return 0.0 < eps;
    const double dx = x2 - x1;
    const double dy = y2 - y1;
    if (fabs(dx) >= skip || fabs(dy) >= skip) return false;
    return (double)hypotf((float)dx, (float)dy) < eps;
}

// Bitonic sort of the first P = 2^k >= M keys; the entries past M are
// 0xffffffff and sort last (no finite value reaches that key).  Returns false
// if a value is not finite (the caller then keeps the chunked scans).
__device__ bool dbscan_sort(const DbscanSort& so, const double* pk, int M, int P, int lane)
{
    bool bad = false;
    for (int k = lane; k < P; k += 32) {
        unsigned key = 0xffffffffu;
        if (k < M) {
            const double v = pk[k];
            if (!isfinite(v)) bad = true;
            key = (dbscan_coarse(v) << kDbscanIdxBits) | (unsigned)k;
        }
        so.key[k] = key;
    }
    if (__any_sync(kFull, bad)) return false;
    __syncwarp();
    for (int size = 2; size <= P; size <<= 1) {
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            for (int t = lane; t < (P >> 1); t += 32) {
                const int i = 2 * t - (t & (stride - 1));
                const int j = i + stride;
                const unsigned ki = so.key[i], kj = so.key[j];
                if ((ki > kj) == ((i & size) == 0)) {
                    so.key[i] = kj;
                    so.key[j] = ki;
                }
            }
            __syncwarp();
        }
    }
    return true;
}

// Coarse keys bounding the candidates of a centre at x1 (finite): every k with
// |fl(p_k - x1)| < skip has p_k within x1 -/+ (2 skip + 4 ulp(x1)).
__device__ __forceinline__ void dbscan_bounds(double x1, double skip, unsigned& cA, unsigned& cB)
{
    const double half = 2.0 * skip + fabs(x1) * 0x1p-50;
    cA = dbscan_coarse(x1 - half);
    cB = dbscan_coarse(x1 + half);
}

// Scan-empty marks: E[c] set iff no k < M (k != c) is near c, found by probing
// the sorted neighbours of c outwards while their keys stay within c's bounds.
// A peak with more than kDbscanProbes probes, and the unsorted last peak, stay
// unmarked (their scans run).  E and D are cleared here.
__device__ void dbscan_mark_empty(const DbscanSort& so, const double* pk, const double* iv, int n, int M,
                                  double eps, double skip, int lane)
{
    const int words = (n + 31) >> 5;
    for (int w = lane; w < words; w += 32) {
        so.E[w] = 0u;
        so.D[w] = 0u;
    }
    __syncwarp();
    for (int pos = lane; pos < M; pos += 32) {
        const int c = (int)(so.key[pos] & kDbscanIdxMask);
        const double x1 = pk[c];
        const double y1 = iv[c];
        unsigned cA, cB;
        dbscan_bounds(x1, skip, cA, cB);
        bool near = false;
        int probes = 0;
        for (int q = pos + 1; q < M && !near; ++q) {
            const unsigned kq = so.key[q];
            if ((kq >> kDbscanIdxBits) > cB) break;
            if (++probes > kDbscanProbes) { near = true; break; }
            const int k = (int)(kq & kDbscanIdxMask);
            near = dbscan_near(x1, y1, pk[k], iv[k], eps, skip);
        }
        for (int q = pos - 1; q >= 0 && !near; --q) {
            const unsigned kq = so.key[q];
            if ((kq >> kDbscanIdxBits) < cA) break;
            if (++probes > kDbscanProbes) { near = true; break; }
            const int k = (int)(kq & kDbscanIdxMask);
            near = dbscan_near(x1, y1, pk[k], iv[k], eps, skip);
        }
        if (!near) atomicOr(&so.E[c >> 5], 1u << (c & 31));
    }
    __syncwarp();
}

// Number of sorted positions < M whose coarse value c satisfies pred(c), for a
// predicate true on a prefix: the last entry of each of 32 segments first (the
// non-empty segments whose last entry passes are a prefix of the lanes), then
// the entries of the first segment whose last entry fails.
template <class Pred>
__device__ int dbscan_prefix(const unsigned* key, int M, int lane, Pred pred)
{
    const int seg = (M + 31) >> 5;
    const int first = lane * seg;
    const bool in1 = first < M && pred(key[min(first + seg, M) - 1] >> kDbscanIdxBits);
    const int c = __popc(__ballot_sync(kFull, in1));
    const int pos = c * seg + lane;
    const bool in2 = lane < seg && pos < M && pred(key[pos] >> kDbscanIdxBits);
    return min(M, c * seg + __popc(__ballot_sync(kFull, in2)));
}

// The scan of `center` over k = 0..M-1 in chunks of 32 (label word per chunk).
// Returns the number of indices added to L and S.
__device__ int dbscan_scan_chunked(const double* pk, const double* iv, int M, int center, double x1,
                                   double y1, double eps, double skip, unsigned* L, unsigned* Sb,
                                   int lane)
{
    int added = 0;
    for (int base = 0; base < M; base += 32) {
        const int k = base + lane;
        bool cand = false;
        if (k < M && k != center && !((L[base >> 5] >> lane) & 1u))
            cand = dbscan_near(x1, y1, pk[k], iv[k], eps, skip);
        const unsigned b = __ballot_sync(kFull, cand);
        if (b) {
            if (lane == 0) {
                L[base >> 5] |= b;
                Sb[base >> 5] |= b;
            }
            added += __popc(b);
        }
    }
    return added;
}

// The scan of `center` over the sorted positions [lo, hi) that hold every
// candidate.  Returns the number of indices added to L and S.
__device__ int dbscan_scan_window(const DbscanSort& so, const double* pk, const double* iv, int lo, int hi,
                                  int center, double x1, double y1, double eps, double skip, unsigned* L,
                                  unsigned* Sb, int lane)
{
    int added = 0;
    for (int base = lo; base < hi; base += 32) {
        const int pos = base + lane;
        bool cand = false;
        int k = 0;
        if (pos < hi) {
            k = (int)(so.key[pos] & kDbscanIdxMask);
            if (k != center && !((L[k >> 5] >> (k & 31)) & 1u))
                cand = dbscan_near(x1, y1, pk[k], iv[k], eps, skip);
        }
        const unsigned b = __ballot_sync(kFull, cand);
        if (b) {
            if (cand) {
                atomicOr(&L[k >> 5], 1u << (k & 31));
                atomicOr(&Sb[k >> 5], 1u << (k & 31));
            }
            added += __popc(b);
        }
    }
    return added;
}

// First index j >= i that is unlabelled and not scan-empty, or n.
__device__ int dbscan_next_open(const unsigned* L, const unsigned* E, int n, int i, int lane)
{
    const int words = (n + 31) >> 5;
    for (int w0 = i >> 5; w0 < words; w0 += 32) {
        const int w = w0 + lane;
        unsigned open = 0u;
        if (w < words) {
            open = ~L[w] & ~E[w];
            if (w == (i >> 5)) open &= ~0u << (i & 31);
            if (w == words - 1 && (n & 31)) open &= (1u << (n & 31)) - 1u;
        }
        const unsigned b = __ballot_sync(kFull, open != 0u);
        if (b) {
            const int f = __ffs(b) - 1;
            const unsigned ow = __shfl_sync(kFull, open, f);
            return ((w0 + f) << 5) + __ffs(ow) - 1;
        }
    }
    return n;
}

// The reference's walk over i in [i, j) with an empty stack, where every
// unlabelled index is scan-empty: labelled ones are no-ops, each unlabelled one
// opens a cluster, is labelled, and its scan adds nothing.  Labels them all;
// returns (clusters opened, of which among the scanned indices < M).
__device__ int2 dbscan_open_run(unsigned* L, int i, int j, int M, int lane)
{
    int opened = 0, openedScanned = 0;
    const int wEnd = (j - 1) >> 5;
    for (int w0 = i >> 5; w0 <= wEnd; w0 += 32) {
        const int w = w0 + lane;
        unsigned m = 0u;
        if (w <= wEnd) {
            m = ~L[w];
            if (w == (i >> 5)) m &= ~0u << (i & 31);
            const int top = j - (w << 5);  // >= 1: bits below it lie in [i, j)
            if (top < 32) m &= (1u << top) - 1u;
            if (m) L[w] |= m;
        }
        const int c = __popc(m);
        const int cLast = (w <= wEnd && (M >> 5) == w) ? (int)((m >> (M & 31)) & 1u) : 0;
        opened += __reduce_add_sync(kFull, c);
        openedScanned += __reduce_add_sync(kFull, c - cLast);
    }
    __syncwarp();
    return make_int2(opened, openedScanned);
}

// What the DBSCAN epilogue needs of a job.
struct DbscanSpec {
    double dbEps, dbSkip;
    int maxPeaks;
};

__device__ __forceinline__ DbscanSpec dbscan_spec(const DevJob& J) { return DbscanSpec{J.dbEps, J.dbSkip, J.maxPeaks}; }

// The count of a point that its number of peaks alone decides (-1: it does not).
__device__ __forceinline__ int dbscan_by_count(int n, int maxPeaks)
{
    return n <= 0 ? 0 : n == 1 ? 1 : n > maxPeaks ? 0 : -1;
}

// DBSCAN cluster count of one point; `so` (shared memory of this warp) enables
// the sorted path for points with n - 1 <= so.cap peaks.
__device__ __noinline__ int dbscan_warp(const DbscanSpec J, const double* pk,
                                        const double* iv, int n, int lane, unsigned* L,
                                        unsigned* Sb, int* err, DbscanSort so)
{
    if (n <= 1 || n > J.maxPeaks) return dbscan_by_count(n, J.maxPeaks);

    const int words = (n + 31) >> 5;
    for (int w = lane; w < words; w += 32) {
        L[w] = 0u;
        Sb[w] = 0u;
    }

    const double eps = J.dbEps;
    const double skip = J.dbSkip;
    const int M = n - 1;  // indices 0..n-2 are scanned; the last peak never is
    int P = 32;
    while (P < M) P <<= 1;
    const bool sorted = so.cap > 0 && M <= so.cap && skip > 0 && isfinite(skip) &&
                        dbscan_sort(so, pk, M, P, lane);
    if (sorted) dbscan_mark_empty(so, pk, iv, n, M, eps, skip, lane);
    __syncwarp();

    int cluster = 0;
    int num = 0;
    int nlab = 0;  // labels set among the scanned indices 0..n-2
    long long guard = (long long)n * n + 4ll * n + 16;
    for (int i = 0; i < n; i++) {
        if (--guard < 0) {
            if (lane == 0) atomicExch(err, 1);
            return 0;
        }
        if (sorted && num == 0) {
            const int j = dbscan_next_open(L, so.E, n, i, lane);
            if (j > i) {
                const int2 r = dbscan_open_run(L, i, j, M, lane);
                cluster += r.x;
                nlab += r.y;
                guard -= j - i;
                i = j;
                if (i >= n) break;
            }
        }
        int center = -1;
        if (num >= 1) {
            const int m = num - 1;
            const bool set = (Sb[m >> 5] >> (m & 31)) & 1u;
            __syncwarp();
            if (lane == 0) Sb[m >> 5] &= ~(1u << (m & 31));
            __syncwarp();
            i = set ? m : 0;
            num = num - 1;
            center = i;
        } else if (!((L[i >> 5] >> (i & 31)) & 1u)) {
            num = 0;
            ++cluster;
            __syncwarp();
            if (lane == 0) L[i >> 5] |= 1u << (i & 31);
            __syncwarp();
            center = i;
            if (i < M) ++nlab;
        }
        if (center < 0 || nlab >= M) continue;

        const double x1 = pk[center];
        const double y1 = iv[center];
        int added;
        if (sorted) {
            const unsigned bit = 1u << (center & 31);
            if ((so.E[center >> 5] | so.D[center >> 5]) & bit) continue;
            if (lane == 0) so.D[center >> 5] |= bit;
        }
        if (sorted && isfinite(x1)) {
            unsigned cA, cB;
            dbscan_bounds(x1, skip, cA, cB);
            const int lo = dbscan_prefix(so.key, M, lane, [cA](unsigned c) { return c < cA; });
            const int hi = dbscan_prefix(so.key, M, lane, [cB](unsigned c) { return c <= cB; });
            if (2 * (hi - lo) <= M)
                added = dbscan_scan_window(so, pk, iv, lo, hi, center, x1, y1, eps, skip, L, Sb, lane);
            else
                added = dbscan_scan_chunked(pk, iv, M, center, x1, y1, eps, skip, L, Sb, lane);
        } else {
            added = dbscan_scan_chunked(pk, iv, M, center, x1, y1, eps, skip, L, Sb, lane);
        }
        num += added;
        nlab += added;
        __syncwarp();
    }
    return cluster - 1;
}

// ---------------------------------------------------------------------------
// Epilogues of a tile, shared when the tiles have run out.
//
// A tile's epilogues run one after the other in the warp that integrated it, and
// their cost varies by orders of magnitude (a fixed point's wobble gives a thousand
// peaks within each other's reach), so maps ended with a few warps at work (Lorenz
// 1024^2: KDE 188 -> 176 ms, DBSCAN 156 -> 148 ms; 512^2: KDE 49 -> 37 ms).  Every
// warp therefore publishes its integrated tile, and takes its own points -- and
// the warps that find no tile left take other warps' points -- by an atomic
// counter per warp.  A warp's peak slots are reused only with a new tile, which no
// warp gets once others have found none: nothing a helper reads is overwritten.
//
// Taking a point is an atomic's round trip, so points that their number of peaks alone
// decides are not shared: their lanes write them; and a look through all warps is a
// round trip for every group of 32, so a helper looks only while a tile may have points.
// Maps of next to no work (250^2 Lorenz points, 60 samples) take 62 us (DBSCAN) and 76
// (KDE), 130 when every point was taken and every helper looked, 45 without sharing.
struct EpilogueShare {
    unsigned* next;             // [warps] points taken of the published tile
    unsigned long long* info;   // [warps] published tile: payload << 6 | points
    int* count;                 // [warps * 32] emitted peaks of a point, -1: nothing to do
    unsigned* busy;             // warps that may hold a tile they have not published
    unsigned* open;             // published tiles whose own warp has not taken their last point
    int warps;
};

// Bytes of the share's arrays for `warps` warps; the first `zeroed` of them must
// be zero on entry.
__host__ __device__ inline size_t epilogue_share_bytes(long long warps, size_t* zeroed)
{
    const size_t z = 256 + (size_t)((warps + 31) / 32 * 32) * (sizeof(unsigned) + sizeof(unsigned long long));
    if (zeroed) *zeroed = z;
    return z + (size_t)warps * 32 * sizeof(int);
}

__host__ __device__ inline EpilogueShare epilogue_share(void* mem, long long warps)
{
    const size_t w = (size_t)((warps + 31) / 32 * 32);
    char* p = static_cast<char*>(mem);
    EpilogueShare sh;
    sh.busy = reinterpret_cast<unsigned*>(p);
    sh.open = reinterpret_cast<unsigned*>(p + 128);
    sh.info = reinterpret_cast<unsigned long long*>(p + 256);
    sh.next = reinterpret_cast<unsigned*>(p + 256 + w * sizeof(unsigned long long));
    sh.count = reinterpret_cast<int*>(p + 256 + w * (sizeof(unsigned long long) + sizeof(unsigned)));
    sh.warps = (int)warps;
    return sh;
}

// The warp's next tile from the counter `queue`; one of `tiles` or more: none left.
__device__ __forceinline__ unsigned long long epilogue_next_tile(const EpilogueShare& sh, unsigned long long* queue,
                                                                 unsigned long long tiles, int lane)
{
    unsigned long long t = 0;
    if (lane == 0) {
        atomicAdd(sh.busy, 1u);  // before the tile is taken: helpers that see no busy warp miss none
        __threadfence();
        t = atomicAdd(queue, 1ull);
        if (t >= tiles) atomicSub(sh.busy, 1u);
    }
    return __shfl_sync(kFull, t, 0);
}

// This warp's integrated tile: `n` per lane, `payload` names the tile.  live = 0:
// nothing is left to do, and what was published before has been taken.
__device__ __forceinline__ void epilogue_publish(const EpilogueShare& sh, long long warp, int lane, int n, int live,
                                                 unsigned long long payload)
{
    if (live == 0) {
        if (lane == 0) atomicSub(sh.busy, 1u);
        return;
    }
    sh.count[warp * 32 + lane] = n;
    __threadfence();  // peaks and counts before the tile
    __syncwarp();
    if (lane == 0) {
        atomicAdd(sh.open, 1u);
        *(volatile unsigned long long*)(sh.info + warp) = payload << 6 | (unsigned)live;
        __threadfence();
        atomicExch(sh.next + warp, 0u);
        __threadfence();
        atomicSub(sh.busy, 1u);
    }
}

// The tile's points by the warp itself: item(j) for every point no helper took.
// The next point is taken while one is worked on.
template <class Item>
__device__ __forceinline__ void epilogue_own(const EpilogueShare& sh, long long warp, int lane, int live, Item item)
{
    if (live == 0) return;
    unsigned j = 0;
    if (lane == 0) j = atomicAdd(sh.next + warp, 1u);
    j = __shfl_sync(kFull, j, 0);
    while (j < (unsigned)live) {
        unsigned after = 0;
        if (lane == 0) after = atomicAdd(sh.next + warp, 1u);
        item((int)j);
        j = __shfl_sync(kFull, after, 0);
    }
    if (lane == 0) atomicSub(sh.open, 1u);
    __syncwarp();
}

// No tile is left: other warps' points until no warp holds a tile that it has not
// published, or none has published one for kHelpIdle.  item(warp, payload, j).  A
// helper that leaves early leaves the points to their own warp.  LOOK: groups of 32
// warps looked at at once -- four where a look is most of what helpers do (DBSCAN of
// 496^2 Chen points 206 -> 186 ms, basin maps 2 to 4 % less), one beside the KDE
// epilogue, whose registers are spilled for more (783^2 Rossler points 46 -> 48 ms).
//
// Why leave early: a waiting helper holds its place on the SM, and with it whatever
// else is to run -- another stream's kernel, a batch's other family -- which matters
// where few points take much longer than the rest: a kernel of 0.4 ms on another
// stream took 370 ms beside a batch of 16 such points, and takes 0.4 again.  Maps and
// batches end in a stream of published tiles, so half a millisecond without one is
// rare before the end: 1024^2 maps, 512^2 and 300^2 maps and a batch of 24 take the
// same at 0.1, 0.5, 2 ms and without a limit.
constexpr int kHelpPolls = 1 << 16;
constexpr unsigned long long kHelpIdle = 500000;  // ns
__device__ __forceinline__ unsigned long long now_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}
template <int LOOK, class Item>
__device__ __forceinline__ void epilogue_help(const EpilogueShare& sh, long long warp, int lane, Item item)
{
    unsigned long long since = now_ns();
    for (int poll = 0; poll < kHelpPolls; ++poll) {
        unsigned all = 0, none = 0;
        if (lane == 0) {
            all = *(volatile unsigned*)sh.busy == 0u;
            __threadfence();
            none = all && *(volatile unsigned*)sh.open == 0u;  // as in a map of next to no work
        }
        all = __shfl_sync(kFull, all, 0);  // read before the look: nothing appears after it
        if (__shfl_sync(kFull, none, 0)) return;
        bool found = false;
        // warp `from`'s points, while there are any
        auto take = [&](long long from) {
            for (;;) {
                unsigned j = 0;
                unsigned long long info = 0;
                if (lane == 0) {
                    j = atomicAdd(sh.next + from, 1u);
                    __threadfence();
                    info = *(volatile unsigned long long*)(sh.info + from);
                }
                j = __shfl_sync(kFull, j, 0);
                info = __shfl_sync(kFull, info, 0);
                if (j >= (unsigned)(info & 63u)) break;
                __threadfence();  // the tile before its counts and peaks
                item(from, info >> 6, (int)j);
                found = true;
            }
        };
        // Both start at the warp's own group of 32, so that helpers spread.
        if constexpr (LOOK == 1) {
            for (int base = 0; base < sh.warps; base += 32) {
                long long v = warp / 32 * 32 + base + lane;
                if (v >= (sh.warps + 31) / 32 * 32) v -= (sh.warps + 31) / 32 * 32;
                const bool some = v < sh.warps && *(volatile unsigned*)(sh.next + v) <
                                                      (unsigned)(*(volatile unsigned long long*)(sh.info + v) & 63u);
                unsigned mask = __ballot_sync(kFull, some);
                while (mask) {
                    const int src = __ffs(mask) - 1;
                    mask &= mask - 1;
                    take(__shfl_sync(kFull, v, src));
                }
            }
        } else {
            const int groups = (sh.warps + 31) / 32;
            auto place = [&](int i) {
                const int g = (int)(warp / 32) + i;
                return g < groups ? g : g - groups;
            };
            for (int base = 0; base < groups; base += LOOK) {
                unsigned next[LOOK], live[LOOK], masks[LOOK], any = 0;
#pragma unroll
                for (int k = 0; k < LOOK; ++k) {  // the loads together
                    const int v = place(base + k) * 32 + lane;
                    const bool there = base + k < groups && v < sh.warps;
                    next[k] = there ? *(volatile unsigned*)(sh.next + v) : 0u;
                    live[k] = there ? (unsigned)*(volatile unsigned long long*)(sh.info + v) & 63u : 0u;
                }
#pragma unroll
                for (int k = 0; k < LOOK; ++k) any |= masks[k] = __ballot_sync(kFull, next[k] < live[k]);
                if (!any) continue;
#pragma unroll 1
                for (int k = 0; k < LOOK; ++k) {
                    unsigned mask = masks[0];
#pragma unroll
                    for (int m = 1; m < LOOK; ++m)
                        if (k == m) mask = masks[m];
                    for (; mask; mask &= mask - 1) take(place(base + k) * 32ll + __ffs(mask) - 1);
                }
            }
        }
        if (found) {
            since = now_ns();
        } else {
            if (__shfl_sync(kFull, all || now_ns() - since > kHelpIdle, 0)) return;
            __nanosleep(8000);  // a map of little work ends at once
        }
    }
}

}  // namespace
}  // namespace cbf
