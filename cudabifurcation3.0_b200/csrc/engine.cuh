// Internal definitions shared by the kernels and the C-ABI layer.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/cbf.h"
#include "systems.cuh"

namespace cbf {

// A validated job in the form the kernels consume (passed by value).
struct DevJob {
    double ranges[4];
    double ic[CBF_MAX_DIM];
    double values[CBF_MAX_VALUES];
    double h;
    double maxValue;
    double divThresh;   // |x| >= divThresh  <=>  fabsf((float)x) > maxValue
    double lleEps;
    double tMax;
    double kdeI1, kdeI2, kdeH;
    double kdeSkip;     // terms with |peak - delta| > kdeSkip are exactly 0 (see kde epilogue)
    double kdeInvH;     // 1/kdeH when kdeH = +-2^k and 1/kdeH is a normal double, else 0
    double dbEps;
    double dbSkip;      // pairs with |dx| or |dy| >= dbSkip are never neighbours
    long long firstPoint;
    long long nPoints;
    long long seedChunk;
    const long long* pointIndex;  // optional device list of grid indices (see cbf_job)
    int regimeSteps;    // LLE_REGIME: recorded steps after the transient
    double regimeMinAmp;  // LLE_REGIME: window range below this -> class 0
    double regimeChaosLle;  // LLE_REGIME: > 0 and LLE above it -> class 15
    double ostThr;      // OSTROVSKY: periodicity threshold
    int nPts, dims, nIC, nV;
    int idxMut0, idxMut1;
    int writableVar, preScaller;
    int nSkip;          // transient steps: (int)(transientTime / h)
    int nRecord;        // recorded samples (int)(tMax/h/preScaller); LLE: (int)(tMax/NT)
    int nNT;            // LLE steps per renormalisation (int)(size_t)(NT/h)
    int checkDiv;       // maxValue != 0 and can ever fire
    unsigned divHi;     // high word of divThresh (conservative fast check)
    int exactGrid;
    int maxPeaks;
    int kdeSampling;
    int kdeFixed;
    int peakCap;        // peaks stored per point
    int task;
    int system;
    int sweepIC;
    int scaledStep;     // Chen/Lorenz: the rescaled step (systems.cuh, QuadScaled) for this job
    int unitStep;       // ... with k = h1 (s = 1/2): its 8-instruction form
};

// Grid index of the job's k-th point: an explicit list, or a contiguous range.
__device__ __forceinline__ long long grid_index(const DevJob& J, long long k)
{
    return J.pointIndex ? J.pointIndex[k] : J.firstPoint + k;
}

// getValueByIdx (cudaLibrary.cu:210-216): `(int)idx / powf(nPts, v)` is a float
// division, so above 2^24 the index is rounded; exactGrid uses integer math.
__device__ __forceinline__ double grid_value(long long g, int nPts, double start, double finish,
                                             int axis, bool exact)
{
    int cell;
    if (!exact) {
        float p = powf((float)nPts, (float)axis);
        float q = (float)(int)g / p;
        cell = ((int)q) % nPts;
    } else {
        long long d = (axis == 0) ? 1 : (long long)nPts;
        cell = (int)((g / d) % nPts);
    }
    return start + (double)cell * ((double)(finish - start) / (double)(nPts - 1));
}

// Set up one point: ICs and values copied, swept entries overwritten
// (cudaLibrary.cu:96-105; IC variant :183-192).  Fully unrolled so that the
// arrays stay in registers even though the swept indices are runtime values.
template <int DIM>
__device__ __forceinline__ void setup_point(const DevJob& J, long long g, double (&x)[DIM],
                                            double (&v)[CBF_MAX_VALUES])
{
    const bool exact = J.exactGrid != 0;
    const double p0 = grid_value(g, J.nPts, J.ranges[0], J.ranges[1], 0, exact);
    const double p1 = (J.dims > 1) ? grid_value(g, J.nPts, J.ranges[2], J.ranges[3], 1, exact) : 0.0;
    const int m0 = J.idxMut0;
    const int m1 = (J.dims > 1) ? J.idxMut1 : -1;
#pragma unroll
    for (int i = 0; i < DIM; ++i) {
        double t = J.ic[i];
        if (J.sweepIC) {
            if (i == m0) t = p0;
            if (i == m1) t = p1;
        }
        x[i] = t;
    }
#pragma unroll
    for (int i = 0; i < CBF_MAX_VALUES; ++i) {
        double t = J.values[i];
        if (!J.sweepIC) {
            if (i == m0) t = p0;
            if (i == m1) t = p1;
        }
        v[i] = t;
    }
}

// Conservative magnitude tracker of a stream of doubles against a threshold T:
// |v| >= T needs hi(|v|) >= hi(T) (the high word is monotone in the magnitude),
// and the high words compare like the floats of the same bits.  So one
// three-input FP32 maximum of magnitudes (max.abs, sm_100) takes two values of
// either sign per instruction; .NaN makes a high word that is no float number
// (|v| >= 2^1017, infinities, NaNs) stick.  One instruction per two values
// matters: what it reads from the register file delays the FP64 step, which is
// bound by its own operand reads (a chain of the 8-instruction step with a
// signed and an unsigned integer maximum per two values ran at 0.68 of the FP64
// pipe, without any at 0.72).
struct HiTrack {
    float m;
    __device__ __forceinline__ void init() { m = 0.0f; }
    __device__ __forceinline__ void add2(double a, double b)
    {
        asm("max.NaN.abs.f32 %0, %1, %2, %3;"
            : "=f"(m)
            : "f"(m), "f"(__int_as_float(__double2hiint(a))), "f"(__int_as_float(__double2hiint(b))));
    }
    __device__ __forceinline__ void add1(double a) { add2(a, a); }
    // hiT = the threshold's high word without sign (DevJob::divHi); a NaN on
    // either side reads as reached.
    __device__ __forceinline__ bool maybe(unsigned hiT) const { return !(m < __uint_as_float(hiT)); }
};

// Exact divergence test of loopCalculateDiscreteModel (cudaLibrary.cu:69-71).
__device__ __forceinline__ bool diverged(double v, double thresh)
{
    return fabs(v) >= thresh;
}

// Deterministic LLE perturbation direction from the chunk-local thread index
// (cudaLibrary.cu:720-732; IC variant :843-855), normalised in double.
template <int D, bool IC>
__device__ __forceinline__ void lle_seed(long long g, long long seedChunk, double (&z)[D])
{
    const int idx = (int)(seedChunk > 0 ? (g % seedChunk) : g);
    double zPower = 0;
#pragma unroll
    for (int i = 0; i < D; ++i) {
        if (!IC) {
            const unsigned u = (unsigned)idx * ((unsigned)i * (unsigned)idx + 1u) + 1u;
            z[i] = 0.5 * (double)sinf((float)(int)u);
        } else {
            const double arg = 0.2171828 * (i + 1) + idx + (0.2171828 + i * idx);
            z[i] = (double)sinf((float)arg) * 0.5;
        }
        zPower += z[i] * z[i];
    }
    zPower = sqrt(zPower);
#pragma unroll
    for (int i = 0; i < D; ++i) z[i] /= zPower;
}

// Initial perturbation rows of the Lyapunov-spectrum kernel (LSKernelCUDA,
// cudaLibrary.cu:1001-1013): row j, entry i = 0.5 sinf(0.2171828 (i+1)(j+1) + idx
// + (0.2171828 + i j idx)) in the reference's operation order (double sum, FP32
// sinf), idx the chunk-local index; each row normalised to length 1.
template <int D>
__device__ __forceinline__ void ls_seed(long long g, long long seedChunk, double (&z)[D][D])
{
    const int idx = (int)(seedChunk > 0 ? (g % seedChunk) : g);
#pragma unroll
    for (int j = 0; j < D; ++j) {
        double zPower = 0;
#pragma unroll
        for (int i = 0; i < D; ++i) {
            const double arg = 0.2171828 * (i + 1) * (j + 1) + idx + (0.2171828 + i * j * idx);
            z[j][i] = (double)sinf((float)arg) * 0.5;
            zPower += z[j][i] * z[j][i];
        }
        zPower = sqrt(zPower);
#pragma unroll
        for (int i = 0; i < D; ++i) z[j][i] /= zPower;
    }
}

// Kernel launch bookkeeping (defined in capi.cu).
void note_launch(unsigned n = 1);

// Threads per block of the fused bifurcation kernel (bif.cu).
constexpr int kBifBlockThreads = 128;

// Launchers (defined in lle.cu / bif.cu / probes.cu).  All return a CUDA error.
cudaError_t launch_lle(const DevJob& J, double* d_out, cudaStream_t s);
// LLE kernel shapes (lle.cu): the autotuner's search space.
constexpr int kNumLleVariants = CBF_NUM_LLE_VARIANTS;
cudaError_t launch_lle_variant(const DevJob& J, double* d_out, cudaStream_t s, int variant);
// The shape cbf_run uses for `system` on the current device (capi.cu).
int lle_variant_for(int system);
cudaError_t launch_bif(const DevJob& J, void* d_out, int* d_aux, cudaStream_t s);
// Rows of `cap` peak slots, the first min(counts[p], cap) of row p filled, to
// packed[offset[p]..].
cudaError_t launch_pack_peaks(const double* peaks, const int* counts, const long long* offset, long long n, int cap,
                              double* packed, cudaStream_t s);
cudaError_t launch_grid_coords(const DevJob& J, double* d_out, cudaStream_t s);
cudaError_t launch_lle_seeds(const DevJob& J, double* d_out, cudaStream_t s);
// Lyapunov spectrum: nIC exponents per point (d_out[p*nIC + i]); seed rows
// (nIC x nIC per point) for parity checks.
cudaError_t launch_ls(const DevJob& J, double* d_out, cudaStream_t s);
cudaError_t launch_ls_seeds(const DevJob& J, double* d_out, cudaStream_t s);
cudaError_t launch_lle_regime(const DevJob& J, double* d_lle, int* d_class, cudaStream_t s);
// Points of one wave of the surrogate map's recompute rounds on the current device.
long long lle_regime_round_points(const DevJob& J);
// Blocks of `bytes` of dynamic shared memory each that fit an SM's `perSm` bytes: a
// block takes `reserved` bytes more, and whole units of 128 (what the occupancy
// calculator counts: of 233 472 bytes, 45 568 a block are five blocks, 45 584 four).
inline long long blocks_by_shared_memory(long long perSm, long long bytes, long long reserved)
{
    return perSm / ((bytes + reserved + 127) / 128 * 128);
}
// The LLE_REGIME kernel over a device point list (J.pointIndex) whose length
// *nDev (at most maxPoints) a previous kernel wrote, with caller-provided
// scratch of lle_regime_scratch_bytes(J); no allocation, no host
// synchronisation: a device-side check sets *err (zero on entry); *queue is the
// launch's tile counter.
size_t lle_regime_scratch_bytes(const DevJob& J);
cudaError_t launch_lle_regime_list(const DevJob& J, const long long* nDev, long long maxPoints, double* d_lle,
                                   int* d_cls, double* scratch, size_t scratchBytes, int* err,
                                   unsigned long long* queue, cudaStream_t s);

// KDE/DBSCAN with caller-provided scratch (no allocation): `scratch` holds
// `scratchBytes` of peak buffers, `err` one int that must be zero on entry.
// Synchronises `s` to read `err`.
cudaError_t launch_bif_prealloc(const DevJob& J, void* d_out, double* scratch, size_t scratchBytes,
                                int* err, cudaStream_t s);

// Job lowering and error reporting shared with other translation units (capi.cu).
cbf_status lower_job_for(const cbf_job* job, DevJob* d);
// The library's stream for calls given no stream (created once per device).
cbf_status library_default_stream(cudaStream_t* s);
cbf_status report_error(cbf_status st, const char* message);
cbf_status report_cuda_error(cudaError_t e, const char* where);

}  // namespace cbf
