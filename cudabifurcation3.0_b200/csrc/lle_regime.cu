// LLE map with a peak-count regime class per point, in one pass.
//
// The LLE is computed exactly as by the LLE kernels (LLEKernelCUDA semantics,
// cudaLibrary.cu:666-908).  During the first `regimeSteps` steps after the
// transient, the base trajectory's x[writableVar] is sampled before every step
// (the record semantics of loopCalculateDiscreteModel, cudaLibrary.cu:59-62) and
// fed to the streaming peak finder; the class is the reference's DBSCAN cluster
// count of those (peak, interval) pairs (dbscan, cudaLibrary.cu:457-529), with
//   0  when the trajectory diverged inside the window or has no peaks,
//   15 when its LLE exceeds regimeChaosLle (if > 0; no clustering needed), when
//      it has more than maxAmountOfPeaks peaks, or 15 or more clusters.
// A window whose samples span less than regimeMinAmp is class 0 as well: an
// equilibrium reached to FP64 precision can still wobble by an ulp and show
// spurious peaks.  On top of the LLE the window costs a few integer instructions and a
// shared-memory store per step, and the peak states of a block's candidates
// (window_loop); the transient is shared.  This is the plain FP64 method that labels
// the surrogate's training data and recomputes the points it cannot be trusted with.
#include "bif_device.cuh"
#include "lle_device.cuh"

namespace cbf {
namespace {

constexpr int kRegWarps = 4;
constexpr int kRegThreads = kRegWarps * 32;
constexpr int kNumClasses = 16;

// What the window needs of a job, and what it changes.
struct WindowSpec {
    double divThresh, lleEps;
    int nNT, nRecord, wv, checkDiv, cap, amplitude;
    int steps;       // samples in the window: never more than the record has steps
    unsigned hiT;
};

template <class S>
struct WindowState {
    double x[S::DIM], y[S::DIM];
    double result;   // sum of the logarithms
    double amp;      // max - min of the window's samples
    int b, n;        // intervals done; emitted peaks, -1 if the divergence test fired
};

// Renormalisation (cudaLibrary.cu:757-776) after each interval.
template <class S>
__device__ __forceinline__ void renormalise(double (&x)[S::DIM], double (&y)[S::DIM], const typename S::Coef& c,
                                            double lleEps, double& result)
{
    constexpr int D = S::DIM;
    double tt = 0;
#pragma unroll
    for (int l = 0; l < D; ++l) {
        const double d = phys_comp<S>(x[l] - y[l], l, c);
        tt += d * d;
    }
    tt = sqrt(tt) / lleEps;
    result += log(tt);
    if (tt != 0) tt = (1 / tt);
#pragma unroll
    for (int i = 0; i < D; ++i) y[i] = x[i] - ((x[i] - y[i]) * tt);
}

// The intervals that overlap the window: the pair loop with the base trajectory's
// samples fed to the peak stream in blocks of up to kRing steps, as the recorded
// loop of the peak maps does (record_loop, bif_device.cuh).  The window's extremes
// are its ends and its local extremes, which the same mask gives.  A block that
// may reach the divergence threshold, or whose samples are not all numbers, is
// repeated step by step: a trajectory's interval ends at its first failed test
// (loopCalculateDiscreteModel, cudaLibrary.cu:55-74).  A function of its own, so
// that its state does not shape the register use of the pair loop after it.
// Before, the window ran the exact tests and the state machine on every step
// (Chen 600^2, window a tenth of the record: 200 -> 185 ms, and 174 ms with the tile
// counter).  A single sample is no block: intervals of one step, Chen 100^2 with a
// third of the record in the window, take 11.6 ms with the exact tests, 12.1 in blocks.
// Nor are blocks tried once a trajectory is no number (no bound, or an offset of 0):
// each would be repeated (5-D model, 250^2 points without a bound, 13.2 -> 10.2 ms; 12.2
// with the exact tests everywhere).
template <class S, int WV>
__device__ __forceinline__ void window_loop(const WindowSpec& W, WindowState<S>& st, const typename S::Coef& c,
                                            double* ring, double* pk, double* iv)
{
    constexpr int D = S::DIM;
    double x[D], y[D];
    copy_state<D>(x, st.x);
    copy_state<D>(y, st.y);
    double result = st.result;
    PeakStream ps;
    ps.init();
    NoPeakHook hook;
    double lo = INFINITY, hi = -INFINITY;
    bool fired = false, lost = false;  // lost: a trajectory is no number any more
    int b = 0, t = 0;  // t: steps since the transient; sample t is fed, sample t + 1 next
    const int steps = W.steps;
    auto extreme = [&](double v) {
        lo = fmin(lo, v);
        hi = fmax(hi, v);
    };
    if (steps > 0) {
        const double v = sample_of<S, WV>(x, W.wv, c);
        ps.push<true>(v, 0, pk, iv, W.cap, hook);
        extreme(v);
    }
    for (; b < W.nRecord && t < steps; ++b) {
        bool ax = true, ay = true;
        for (int i = 0; i < W.nNT;) {
            const int m = min(kRing, W.nNT - i);
            i += m;
            bool done = false;
            if (!fired && !lost && ax && ay && m > 1) {
                double x0[D], y0[D];
                copy_state<D>(x0, x);
                copy_state<D>(y0, y);
                HiTrack tr, num;
                tr.init();
                num.init();
                RiseMask<kRing> rises;
                rises.init();
                double p = ps.prev1;
                ring[0] = p;
#pragma unroll (D == 5 ? 1 : 4)
                for (int k = 1; k <= m; ++k) {
                    S::step(x, c);
                    S::step(y, c);
                    const double v = sample_of<S, WV>(x, W.wv, c);
                    const int up = rises.add(p, v);
                    rises.seen(up, up);
                    ring[32 * k] = v;
                    p = v;
                    tr.add2(x[0], y[0]);
                    if (WV != 0) num.add1(v);
                }
                done = !tr.maybe(W.hiT) && (WV == 0 || !num.maybe(0x7f800000u));
                if (done) {
                    const int fed = max(0, min(m, steps - 1 - t));  // samples t+1 .. t+fed are in the window
                    if (fed > 0) {
                        const unsigned up = rises.mask(m, ring);
                        if (W.amplitude) {
                            // a sample is a local extreme where it rose and its
                            // successor does not, or the other way round
                            unsigned ext = (ps.after_rise<kRing>(up) ^ up) & PeakStream::arrivals<kRing>(fed);
                            while (ext) {
                                const int e = highest_bit(ext);
                                ext &= ~(1u << e);
                                extreme(ring[32 * (kRing - 1 - e)]);
                            }
                        }
                        ps.push_block<kRing, true>(up, t, fed, ring[32 * fed], ring, pk, iv, W.cap, hook);
                    }
                    t += m;
                } else {
                    copy_state<D>(x, x0);
                    copy_state<D>(y, y0);
                }
            }
            if (!done) {
                if (t < steps && !fired) extreme(ps.prev1);
                for (int k = 0; k < m; ++k, ++t) {
                    if (ax) {
                        S::step(x, c);
                        if (W.checkDiv && diverged(x[0], W.divThresh)) {
                            ax = false;
                            if (t < steps) fired = true;
                        }
                        if (t + 1 < steps && !fired) {
                            const double v = sample_of<S, WV>(x, W.wv, c);
                            ps.push<true>(v, t + 1, pk, iv, W.cap, hook);
                            extreme(v);
                        }
                    }
                    if (ay) {
                        S::step(y, c);
                        if (W.checkDiv && diverged(y[0], W.divThresh)) ay = false;
                    }
                }
                lost = isnan(x[0]) || isnan(y[0]) || isnan(ps.prev1);
            }
        }
        renormalise<S>(x, y, c, W.lleEps, result);
    }
    if (steps > 0) extreme(ps.prev1);  // the last sample
    copy_state<D>(st.x, x);
    copy_state<D>(st.y, y);
    st.result = result;
    st.b = b;
    st.n = fired ? -1 : ps.emitted();
    st.amp = hi - lo;
}

template <class S>
__device__ __noinline__ void run_window(const WindowSpec W, WindowState<S>* st, const typename S::Coef c, double* ring,
                                        double* pk, double* iv)
{
    if constexpr (S::DIM == 3) {
        if (W.wv == 0) window_loop<S, 0>(W, *st, c, ring, pk, iv);
        else if (W.wv == 1) window_loop<S, 1>(W, *st, c, ring, pk, iv);
        else window_loop<S, 2>(W, *st, c, ring, pk, iv);
    } else {
        window_loop<S, -1>(W, *st, c, ring, pk, iv);
    }
}

// One point: returns the LLE; *n = emitted peaks in the window, -1 if the
// divergence test fired inside it; *amp = max - min of the window's samples
// (where regimeMinAmp asks for it).
template <class S, bool IC>
__device__ double lle_regime_point(const DevJob& J, long long g, double* ring, double* pk, double* iv, int cap,
                                   int* nOut, double* amp)
{
    constexpr int D = S::DIM;
    constexpr int UNR = kPointUnroll<S>;
    double x[1][D], y[1][D];
    typename S::Coef c[1];
    {
        double v[CBF_MAX_VALUES];
        setup_point<D>(J, g, x[0], v);
        c[0] = S::prep(v, J.h);
        to_stored<S>(x[0], c[0]);
    }
    run_checked<S, 1, UNR>(x, c, J.nSkip, J);
    double result;
    int b;
    {
        WindowState<S> st;
        double z[D];
        lle_seed<D, IC>(g, J.seedChunk, z);
#pragma unroll
        for (int i = 0; i < D; ++i) {
            st.x[i] = x[0][i];
            st.y[i] = stored_comp<S>(z[i] * J.lleEps, i, c[0]) + x[0][i];
        }
        st.result = 0;
        const WindowSpec W{J.divThresh, J.lleEps, J.nNT, J.nRecord, J.writableVar, J.checkDiv, cap,
                           J.regimeMinAmp > 0 ? 1 : 0,
                           (int)min((long long)J.regimeSteps, (long long)J.nRecord * J.nNT),
                           J.checkDiv ? J.divHi : 0x7f800000u};
        run_window<S>(W, &st, c[0], ring, pk, iv);
        copy_state<D>(x[0], st.x);
        copy_state<D>(y[0], st.y);
        result = st.result;
        b = st.b;
        *nOut = st.n;
        *amp = st.amp;
    }
    for (; b < J.nRecord; ++b) {
        run_pair<S, 1, UNR>(x, y, c, J.nNT, J);
        renormalise<S>(x[0], y[0], c[0], J.lleEps, result);
    }
    return result / J.tMax;
}

// LLE and regime class of the lane's grid point g (`valid` false: the lane idles
// through the integration), the warp cooperating on the DBSCAN epilogues of
// lanes 0..live-1; *lleOut = the lane's LLE.
template <class S, bool IC>
__device__ __forceinline__ int regime_tile(const DevJob& J, long long g, bool valid, int live, int lane,
                                           double* scrPk, double* scrIv, long long slot0, unsigned* L,
                                           unsigned* Sb, const DbscanSort& so, int* err, double* lleOut)
{
    const int cap = J.peakCap;
    double* myPk = scrPk + (slot0 + lane) * (long long)cap;
    double* myIv = scrIv + (slot0 + lane) * (long long)cap;
    int n = 0;
    double lv = 0, amp = 0;
    if (valid) lv = lle_regime_point<S, IC>(J, g, ring_column(L, lane), myPk, myIv, cap, &n, &amp);
    if (J.regimeMinAmp > 0 && amp < J.regimeMinAmp) n = 0;  // no oscillation
    __syncwarp();
    int res = 0;
    for (int j = 0; j < live; ++j) {
        const int nj = __shfl_sync(kFull, n, j);
        const double lj = __shfl_sync(kFull, lv, j);
        int r;
        if (nj <= 0) r = 0;
        else if (J.regimeChaosLle > 0 && lj > J.regimeChaosLle) r = kNumClasses - 1;
        else if (nj > J.maxPeaks) r = kNumClasses - 1;
        else {
            const double* pk = scrPk + (slot0 + j) * (long long)cap;
            const double* iv = scrIv + (slot0 + j) * (long long)cap;
            r = min(dbscan_warp(dbscan_spec(J), pk, iv, nj, lane, L, Sb, err, so), kNumClasses - 1);
        }
        if (lane == j) res = r;
    }
    *lleOut = lv;
    return res;
}

// Blocks per SM, as the LLE map kernel: four for the rescaled Chen/Lorenz step (its
// rounds should end on even counts of warps per scheduler) and for the 5-D model
// (110 registers), six for the 3-D steps that wait for a division.
template <class S>
constexpr int kRegBlocks = S::SCALED || S::DIM == 5 ? 4 : 6;

// nDev (optional): the job's point count read on the device, in place of
// J.nPoints (a point list whose length a previous kernel wrote).
//
// Warps take their tiles from a counter (*queue, zero on entry): a scheduler
// favours its oldest warp, so with as many tiles fixed for each warp the favoured
// ones finished early and the rest ran on too few (the same points, 1024^2 without
// a window: 185 ms fixed, 171 ms where blocks or tiles are handed out).
template <class S, bool IC>
__global__ void __launch_bounds__(kRegThreads, kRegBlocks<S>) lle_regime_kernel(DevJob J, double* __restrict__ lle,
                                                                 int* __restrict__ cls, double* scrPk,
                                                                 double* scrIv, int bitWords, int sortCap,
                                                                 int* err, unsigned long long* queue,
                                                                 const long long* nDev)
{
    extern __shared__ __align__(16) unsigned smem[];
    if (nDev) J.nPoints = *nDev;
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    const long long warpId = (long long)blockIdx.x * kRegWarps + wib;
    const long long nTiles = (J.nPoints + 31) / 32;
    unsigned* L = smem + (size_t)wib * dbscan_warp_words(bitWords, sortCap);
    unsigned* Sb = L + bitWords;
    const DbscanSort so = dbscan_sort_area(L, bitWords, sortCap);
    const long long slot0 = warpId * 32;

    for (;;) {
        unsigned long long next = 0;
        if (lane == 0) next = atomicAdd(queue, 1ull);
        const long long tile = (long long)__shfl_sync(kFull, next, 0);
        if (tile >= nTiles) break;
        const long long p = tile * 32 + lane;
        const bool valid = p < J.nPoints;
        const int live = (int)min(32ll, J.nPoints - tile * 32);
        double lv = 0;
        const int res = regime_tile<S, IC>(J, valid ? grid_index(J, p) : 0, valid, live, lane, scrPk, scrIv,
                                           slot0, L, Sb, so, err, &lv);
        if (valid) {
            lle[p] = lv;
            cls[p] = res;
        }
        __syncwarp();
    }
}

// Blocks of a launch on the current device and its shared memory.
template <class S, bool IC>
cudaError_t regime_shape(const DevJob& J, int* bitWords, int* sortCap, size_t* smem, long long* resident)
{
    auto kern = lle_regime_kernel<S, IC>;
    *bitWords = (J.peakCap + 31) / 32;
    *sortCap = dbscan_sort_cap(J.peakCap);
    *smem = (size_t)kRegWarps * dbscan_warp_words(*bitWords, *sortCap) * sizeof(unsigned);
    cudaError_t e;
    if (*smem > 48 * 1024) {
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)*smem);
        if (e != cudaSuccess) return e;
    }
    int dev = 0, sms = 0, perSm = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, kern, kRegThreads, *smem)) != cudaSuccess)
        return e;
    if (perSm < 1) return cudaErrorInvalidConfiguration;
    *resident = (long long)sms * (perSm < kRegBlocks<S> ? perSm : kRegBlocks<S>);
    return cudaSuccess;
}

template <class S, bool IC>
cudaError_t launch_t(const DevJob& J, double* d_lle, int* d_cls, cudaStream_t s)
{
    const long long nTiles = (J.nPoints + 31) / 32;
    if (nTiles == 0) return cudaSuccess;
    int bitWords = 0, sortCap = 0;
    size_t smemBytes = 0;
    long long resident = 0;
    auto kern = lle_regime_kernel<S, IC>;
    cudaError_t e = regime_shape<S, IC>(J, &bitWords, &sortCap, &smemBytes, &resident);
    if (e != cudaSuccess) return e;
    long long blocks = (nTiles + kRegWarps - 1) / kRegWarps;
    if (blocks > resident) blocks = resident;
    const size_t perBlock = (size_t)kRegThreads * J.peakCap * sizeof(double) * 2;
    size_t freeB = 0, totalB = 0;
    if ((e = cudaMemGetInfo(&freeB, &totalB)) != cudaSuccess) return e;
    size_t budget = freeB / 4;
    if (budget > ((size_t)8 << 30)) budget = (size_t)8 << 30;
    long long fit = (long long)(budget / perBlock);
    if (fit < 1) fit = 1;
    if (blocks > fit) blocks = fit;
    const size_t bytes = (size_t)blocks * perBlock;
    double* scr = nullptr;
    if ((e = cudaMallocAsync((void**)&scr, bytes + 256, s)) != cudaSuccess) return e;
    double* scrIv = scr + (size_t)blocks * kRegThreads * J.peakCap;
    int* err = (int*)((char*)scr + bytes);  // error flag, then the tile counter
    auto* queue = (unsigned long long*)((char*)err + 128);
    if ((e = cudaMemsetAsync(err, 0, 256, s)) == cudaSuccess) {
        kern<<<(unsigned)blocks, kRegThreads, smemBytes, s>>>(J, d_lle, d_cls, scr, scrIv, bitWords, sortCap, err,
                                                              queue, nullptr);
        note_launch();
        e = cudaGetLastError();
    }
    int hostErr = 0;
    cudaError_t e2 = cudaMemcpyAsync(&hostErr, err, sizeof(int), cudaMemcpyDeviceToHost, s);
    cudaError_t e3 = cudaFreeAsync(scr, s);
    if (e == cudaSuccess) e = e2;
    if (e == cudaSuccess) e = e3;
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e == cudaSuccess && hostErr) return cudaErrorAssert;
    return e;
}

template <class S>
cudaError_t launch_s(const DevJob& J, double* d_lle, int* d_cls, cudaStream_t s)
{
    return J.sweepIC ? launch_t<S, true>(J, d_lle, d_cls, s) : launch_t<S, false>(J, d_lle, d_cls, s);
}

// The kernel on a device point list of *nDev <= maxPoints entries: one block per
// resident slot (at most the list's tiles), caller-provided scratch, no
// allocation and no host synchronisation (the caller reads `err`).
template <class S>
cudaError_t launch_list_s(const DevJob& J, const long long* nDev, long long maxPoints, double* d_lle, int* d_cls,
                          double* scratch, size_t scratchBytes, int* err, unsigned long long* queue, cudaStream_t s)
{
    int bitWords = 0, sortCap = 0;
    size_t smemBytes = 0;
    long long resident = 0;
    auto kern = lle_regime_kernel<S, false>;
    cudaError_t e = regime_shape<S, false>(J, &bitWords, &sortCap, &smemBytes, &resident);
    if (e != cudaSuccess) return e;
    long long blocks = (maxPoints + kRegThreads - 1) / kRegThreads;
    if (blocks > resident) blocks = resident;
    const size_t perBlock = (size_t)kRegThreads * J.peakCap * sizeof(double) * 2;
    if ((size_t)blocks * perBlock > scratchBytes) blocks = (long long)(scratchBytes / perBlock);
    if (blocks < 1) return cudaErrorInvalidValue;
    double* scrIv = scratch + (size_t)blocks * kRegThreads * J.peakCap;
    if ((e = cudaMemsetAsync(queue, 0, sizeof(*queue), s)) != cudaSuccess) return e;
    kern<<<(unsigned)blocks, kRegThreads, smemBytes, s>>>(J, d_lle, d_cls, scratch, scrIv, bitWords, sortCap, err,
                                                          queue, nDev);
    note_launch();
    return cudaGetLastError();
}

template <class S>
size_t list_scratch_s(const DevJob& J)
{
    int bitWords = 0, sortCap = 0;
    size_t smem = 0;
    long long resident = 0;
    if (regime_shape<S, false>(J, &bitWords, &sortCap, &smem, &resident) != cudaSuccess) return 0;
    return (size_t)resident * kRegThreads * J.peakCap * sizeof(double) * 2;
}

}  // namespace

// The recompute rounds of the surrogate map are sized by this number, and which
// points a map recomputes follows from the rounds: it stays what it was defined
// by, whatever the kernel's own residency -- six blocks of 128 points per SM, or as
// many as the DBSCAN epilogue's shared memory (bitsets, and sort keys up to 1024
// peaks) leaves room for.
long long lle_regime_round_points(const DevJob& J)
{
    const int bitWords = (J.peakCap + 31) / 32, sortCap = dbscan_sort_cap(J.peakCap);
    const long long words = sortCap > 0 ? 4ll * bitWords + sortCap : 2ll * bitWords;
    int dev = 0, sms = 0, perSm = 0, reserved = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&perSm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev) != cudaSuccess)
        return 0;
    const long long fit = blocks_by_shared_memory(perSm, kRegWarps * words * (long long)sizeof(unsigned), reserved);
    return (long long)sms * (fit < 6 ? fit : 6) * kRegThreads;
}

cudaError_t launch_lle_regime(const DevJob& J, double* d_lle, int* d_cls, cudaStream_t s)
{
    switch (J.system) {
    case CBF_SYS_MEMRISTIVE5: return launch_s<Memristive5>(J, d_lle, d_cls, s);
    case CBF_SYS_ROSSLER: return launch_s<Rossler>(J, d_lle, d_cls, s);
    case CBF_SYS_LORENZ: return J.scaledStep ? (J.unitStep ? launch_s<LorenzScaledU>(J, d_lle, d_cls, s) : launch_s<LorenzScaled>(J, d_lle, d_cls, s)) : launch_s<Lorenz>(J, d_lle, d_cls, s);
    case CBF_SYS_CHEN: return J.scaledStep ? (J.unitStep ? launch_s<ChenScaledU>(J, d_lle, d_cls, s) : launch_s<ChenScaled>(J, d_lle, d_cls, s)) : launch_s<Chen>(J, d_lle, d_cls, s);
    default: return cudaErrorInvalidValue;
    }
}

size_t lle_regime_scratch_bytes(const DevJob& J)
{
    switch (J.system) {
    case CBF_SYS_MEMRISTIVE5: return list_scratch_s<Memristive5>(J);
    case CBF_SYS_ROSSLER: return list_scratch_s<Rossler>(J);
    case CBF_SYS_LORENZ: return J.scaledStep ? (J.unitStep ? list_scratch_s<LorenzScaledU>(J) : list_scratch_s<LorenzScaled>(J)) : list_scratch_s<Lorenz>(J);
    case CBF_SYS_CHEN: return J.scaledStep ? (J.unitStep ? list_scratch_s<ChenScaledU>(J) : list_scratch_s<ChenScaled>(J)) : list_scratch_s<Chen>(J);
    default: return 0;
    }
}

cudaError_t launch_lle_regime_list(const DevJob& J, const long long* nDev, long long maxPoints, double* d_lle,
                                   int* d_cls, double* scratch, size_t scratchBytes, int* err,
                                   unsigned long long* queue, cudaStream_t s)
{
    if (J.sweepIC || !J.pointIndex || maxPoints <= 0) return cudaErrorInvalidValue;
    switch (J.system) {
    case CBF_SYS_ROSSLER: return launch_list_s<Rossler>(J, nDev, maxPoints, d_lle, d_cls, scratch, scratchBytes, err, queue, s);
    case CBF_SYS_LORENZ:
        return J.scaledStep ? (J.unitStep ? launch_list_s<LorenzScaledU>(J, nDev, maxPoints, d_lle, d_cls, scratch, scratchBytes, err, queue, s) : launch_list_s<LorenzScaled>(J, nDev, maxPoints, d_lle, d_cls, scratch, scratchBytes, err, queue, s))
                            : launch_list_s<Lorenz>(J, nDev, maxPoints, d_lle, d_cls, scratch, scratchBytes, err, queue, s);
    case CBF_SYS_CHEN:
        return J.scaledStep ? (J.unitStep ? launch_list_s<ChenScaledU>(J, nDev, maxPoints, d_lle, d_cls, scratch, scratchBytes, err, queue, s) : launch_list_s<ChenScaled>(J, nDev, maxPoints, d_lle, d_cls, scratch, scratchBytes, err, queue, s))
                            : launch_list_s<Chen>(J, nDev, maxPoints, d_lle, d_cls, scratch, scratchBytes, err, queue, s);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace cbf
