// Ragged batches: many map jobs in one persistent launch per kernel family.
//
// The reference runs one map per host call, one chunk and three kernels at a
// time.  A batch here is any mix of jobs -- systems, tasks (LLE, KDE, DBSCAN,
// 1-D peaks), grid sizes, record lengths, step sizes.  Its jobs form two
// families, LLE jobs and peak-based jobs, each executed by ONE persistent
// kernel compiled with that family's code only (so each gets its tasks'
// register count and occupancy); with both present the two kernels run
// concurrently on forked streams:
//   * every job is cut into tiles of 32 points (one warp: a lane per point; fewer
//     points in a small batch of peak jobs, whose epilogues a warp runs one after
//     the other, shared with the warps that find no tile left);
//   * jobs are ordered by estimated cost per point, longest first, and a prefix
//     table of tile counts maps a global tile number to (job, tile);
//   * each warp takes the next tile number from a device counter (atomicAdd by
//     lane 0), so long and short jobs interleave and the tail is made of the
//     cheapest tiles;
//   * a tile runs exactly the per-point code of the map kernels (lle_device.cuh,
//     bif_device.cuh), so batch results equal one-by-one results bit for bit.
// One batch run is "reset error flag; per family: reset counter, launch" and is
// captured once as a CUDA graph for repeated sweeps.  Each family's grid
// (blocks per SM) is chosen by cbf_batch_autotune on a shortened copy of it.
#include <string.h>

#include <algorithm>
#include <vector>

#include "bif_device.cuh"
#include "lle_device.cuh"

namespace cbf {
namespace {

constexpr int kBatchWarps = 4;
constexpr int kBatchThreads = kBatchWarps * 32;
constexpr int kMaxBatchJobs = 1024;
constexpr int kTile = 32;
constexpr int kFamLle = 0, kFamPeaks = 1;

struct BatchJob {
    DevJob job;
    void* out;
    int* aux;
};

// Peak scratch of a launch: 32 lanes of `stride` slots per warp, and the epilogues
// the warps share (bif_device.cuh).
struct BatchScratch {
    double* peaks;
    double* intervals;
    int stride;
    EpilogueShare share;
};

// What a warp has of its shared memory.
struct WarpArea {
    unsigned* L;
    unsigned* Sb;
    DbscanSort so;
};

// The epilogue of point p (n peaks in the given slot) of a KDE or DBSCAN job.
__device__ __forceinline__ void bif_epilogue(const BatchJob& B, long long p, int n, const BatchScratch& sc,
                                             long long slot, const WarpArea& wa, int lane, int* err)
{
    if (n < 0) return;  // done by its lane
    const double* pk = sc.peaks + slot * sc.stride;
    int r;
    if (B.job.task == CBF_TASK_KDE)
        r = kde_warp<true>(kde_spec(B.job), pk, n, lane, reinterpret_cast<float*>(wa.L), kKdeSortCap);
    else
        r = dbscan_warp(dbscan_spec(B.job), pk, sc.intervals + slot * sc.stride, n, lane, wa.L, wa.Sb, err, wa.so);
    if (lane == 0) ((int*)B.out)[p] = r;
    __syncwarp();
}

// Integrates a tile: the emitted peaks of this lane's point.
template <class S, int TASK>
__device__ __forceinline__ int bif_tile(const DevJob& J, void* out, int* aux, long long p0, int tilePts, int lane,
                                        const BatchScratch& sc, long long warpId, const WarpArea& wa)
{
    const long long p = p0 + lane;
    const bool valid = lane < tilePts && p < J.nPoints;
    const long long g = valid ? grid_index(J, p) : 0;
    double* ring = ring_column(wa.L, lane);
    if (TASK == CBF_TASK_PEAKS) {
        if (valid) {
            double* pk = (double*)out + p * (long long)J.peakCap;
            aux[p] = integrate_point<S, TASK>(J, g, pk, nullptr, J.peakCap, nullptr, nullptr, ring);
        }
        return 0;
    }
    const long long slot = warpId * kTile + lane;
    double* myPk = sc.peaks + slot * sc.stride;
    double* myIv = (TASK == CBF_TASK_DBSCAN) ? sc.intervals + slot * sc.stride : nullptr;
    return valid ? integrate_point<S, TASK>(J, g, myPk, myIv, J.peakCap, nullptr, nullptr, ring) : 0;
}

// FAM: the kernel family -- kFamLle runs LLE jobs only, kFamPeaks the
// peak-based tasks (PEAKS, KDE, DBSCAN).  Each family is compiled with its own
// code only, so its register count and occupancy are those of its tasks.
template <class S, int FAM>
__device__ __forceinline__ int run_tile(const DevJob& J, void* out, int* aux, long long p0, int tilePts, int lane,
                                        const BatchScratch& sc, long long warpId, const WarpArea& wa)
{
    if constexpr (FAM == kFamLle) {
        const long long p = p0 + lane;
        if (p < J.nPoints) {
            const long long g = grid_index(J, p);
            ((double*)out)[p] = J.sweepIC ? lle_point<S, true>(J, g) : lle_point<S, false>(J, g);
        }
        return 0;
    } else {
        switch (J.task) {
        case CBF_TASK_KDE: return bif_tile<S, CBF_TASK_KDE>(J, out, aux, p0, tilePts, lane, sc, warpId, wa);
        case CBF_TASK_DBSCAN: return bif_tile<S, CBF_TASK_DBSCAN>(J, out, aux, p0, tilePts, lane, sc, warpId, wa);
        case CBF_TASK_PEAKS: return bif_tile<S, CBF_TASK_PEAKS>(J, out, aux, p0, tilePts, lane, sc, warpId, wa);
        default: return 0;
        }
    }
}

// WITH_M5: also dispatch the 5-D shipped model.  Its wider state raises the
// register count of the whole kernel, so batches of 3-D systems use the
// instantiation without it.
// Four blocks of 128 threads per SM (128 registers) in both families.  LLE: the FP64
// chains issue best from an even number of warps per scheduler (see lle.cu; at six
// blocks the LLE jobs of a 24-job mix of 64^2 to 256^2 points took 30 ms, at four
// 24).  Peaks: the same mix's peak jobs take 35.1 ms at four, 37.1 at six (80
// registers) and 41.6 at eight (64 registers, 0.6 KB spilled); what a small mix waits
// for is its last tiles, which go slower the more warps share an SM.  Where tiles are
// many the order is another: 24 jobs of 300^2 to 500^2, 182, 164 and 173 ms; a mix of
// 64 jobs, 27 million points, both families, 26.7 s at four and 25.4 at six.  The
// peak jobs' shared epilogues took the small mix's from 43 to 35 ms (the two families
// side by side, two blocks per SM each, were no faster).
template <int FAM, bool WITH_M5>
__global__ void __launch_bounds__(kBatchThreads, 4) batch_kernel(
    const BatchJob* __restrict__ jobs, int nJobs, const long long* __restrict__ tileEnd,
    unsigned long long* counter, const BatchScratch sc, int tilePts, int bitWords, int sortCap, int* err)
{
    extern __shared__ __align__(16) unsigned smem[];
    __shared__ long long sEnd[kMaxBatchJobs];
    for (int i = threadIdx.x; i < nJobs; i += blockDim.x) sEnd[i] = tileEnd[i];
    __syncthreads();
    const unsigned long long total = (unsigned long long)sEnd[nJobs - 1];
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    const long long warpId = (long long)blockIdx.x * kBatchWarps + wib;
    WarpArea wa;
    wa.L = smem + (size_t)wib * dbscan_warp_words(bitWords, sortCap);
    wa.Sb = wa.L + bitWords;
    wa.so = dbscan_sort_area(wa.L, bitWords, sortCap);

    // The job of tile t (the first whose tile range ends after t) and the tile's
    // first point.
    auto job_of = [&](unsigned long long t, long long* p0) {
        int lo = 0, hi = nJobs - 1;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if ((unsigned long long)sEnd[mid] > t) hi = mid;
            else lo = mid + 1;
        }
        *p0 = ((long long)t - (lo ? sEnd[lo - 1] : 0)) * tilePts;
        return lo;
    };

    for (;;) {
        unsigned long long t = 0;
        if constexpr (FAM == kFamPeaks) {
            t = epilogue_next_tile(sc.share, counter, total, lane);
        } else {
            if (lane == 0) t = atomicAdd(counter, 1ull);
            t = __shfl_sync(kFull, t, 0);
        }
        if (t >= total) break;
        long long p0 = 0;
        const int k = job_of(t, &p0);
        void* out = jobs[k].out;
        int* aux = jobs[k].aux;
        auto go = [&](const DevJob& J) -> int {
            switch (J.system) {
            case CBF_SYS_MEMRISTIVE5:
                if (WITH_M5) return run_tile<Memristive5, FAM>(J, out, aux, p0, tilePts, lane, sc, warpId, wa);
                return 0;
            case CBF_SYS_ROSSLER: return run_tile<Rossler, FAM>(J, out, aux, p0, tilePts, lane, sc, warpId, wa);
            case CBF_SYS_LORENZ:
                if (J.scaledStep && J.unitStep)  // the map kernels' 8-instruction form
                    return run_tile<LorenzScaledU, FAM>(J, out, aux, p0, tilePts, lane, sc, warpId, wa);
                if (J.scaledStep) return run_tile<LorenzScaled, FAM>(J, out, aux, p0, tilePts, lane, sc, warpId, wa);
                return run_tile<Lorenz, FAM>(J, out, aux, p0, tilePts, lane, sc, warpId, wa);
            case CBF_SYS_CHEN:
                if (J.scaledStep && J.unitStep)  // the map kernels' 8-instruction form
                    return run_tile<ChenScaledU, FAM>(J, out, aux, p0, tilePts, lane, sc, warpId, wa);
                if (J.scaledStep) return run_tile<ChenScaled, FAM>(J, out, aux, p0, tilePts, lane, sc, warpId, wa);
                return run_tile<Chen, FAM>(J, out, aux, p0, tilePts, lane, sc, warpId, wa);
            default: return 0;
            }
        };
        // The LLE family reads its descriptor in place (read-only cache); the
        // peak family keeps a copy (fewer registers in its epilogues).
        if constexpr (FAM == kFamLle) {
            go(jobs[k].job);
        } else {
            int n = 0, live = 0;
            {
                const DevJob J = jobs[k].job;
                n = go(J);
                if (J.task != CBF_TASK_PEAKS) {
                    // as in the maps: what the number of peaks decides is written at once
                    int r = 0;
                    const bool valid = lane < tilePts && p0 + lane < J.nPoints;
                    if (valid)
                        r = J.task == CBF_TASK_KDE ? kde_by_count(n, J.maxPeaks) : dbscan_by_count(n, J.maxPeaks);
                    if (valid && r >= 0) ((int*)out)[p0 + lane] = r;
                    const unsigned left = __ballot_sync(kFull, r < 0);
                    if (r >= 0) n = -1;
                    live = left ? highest_bit(left) + 1 : 0;
                }
            }
            __syncwarp();
            epilogue_publish(sc.share, warpId, lane, n, live, t);
            epilogue_own(sc.share, warpId, lane, live, [&](int j) {
                bif_epilogue(jobs[k], p0 + j, sc.share.count[warpId * 32 + j], sc, warpId * kTile + j, wa, lane, err);
            });
        }
    }
    if constexpr (FAM == kFamPeaks)
        epilogue_help<4>(sc.share, warpId, lane, [&](long long from, unsigned long long t, int j) {
            long long p0 = 0;
            const int k = job_of(t, &p0);
            bif_epilogue(jobs[k], p0 + j, sc.share.count[from * 32 + j], sc, from * kTile + j, wa, lane, err);
        });
}

// Model steps per point, the batch's cost estimate for ordering.
double steps_per_point(const DevJob& d)
{
    if (d.task == CBF_TASK_LLE) return (double)d.nSkip + 2.0 * d.nRecord * (double)d.nNT;
    return (double)d.nSkip + (double)d.nRecord * d.preScaller;
}

}  // namespace

using BatchKernel = void (*)(const BatchJob*, int, const long long*, unsigned long long*, const BatchScratch, int, int,
                            int, int*);

BatchKernel batch_kernel_for(int fam, bool withM5)
{
    if (fam == kFamLle) return withM5 ? batch_kernel<kFamLle, true> : batch_kernel<kFamLle, false>;
    return withM5 ? batch_kernel<kFamPeaks, true> : batch_kernel<kFamPeaks, false>;
}

// Bytes of the peak family's shared epilogues for a grid of up to `blocks` blocks.
size_t batch_share_bytes(int blocks) { return epilogue_share_bytes((long long)blocks * kBatchWarps, nullptr); }

cudaError_t batch_launch(const void* jobs, int nJobs, const long long* tileEnd,
                         unsigned long long* counter, double* scrPk, double* scrIv, int stride, void* share,
                         int tilePts, int bitWords, int* err, int grid, bool withM5, int fam, cudaStream_t s)
{
    const int sortCap = bitWords > 0 ? dbscan_sort_cap(bitWords * 32) : 0;
    const size_t smem = (size_t)kBatchWarps * dbscan_warp_words(bitWords, sortCap) * sizeof(unsigned);
    auto kern = batch_kernel_for(fam, withM5);
    cudaError_t e;
    if (smem > 48 * 1024) {
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    if ((e = cudaMemsetAsync(counter, 0, sizeof(unsigned long long), s)) != cudaSuccess) return e;
    BatchScratch sc{scrPk, scrIv, stride, EpilogueShare{}};
    if (fam == kFamPeaks) {
        size_t zeroed = 0;
        epilogue_share_bytes((long long)grid * kBatchWarps, &zeroed);
        sc.share = epilogue_share(share, (long long)grid * kBatchWarps);
        if ((e = cudaMemsetAsync(share, 0, zeroed, s)) != cudaSuccess) return e;
    }
    kern<<<grid, kBatchThreads, smem, s>>>((const BatchJob*)jobs, nJobs, tileEnd, counter, sc, tilePts, bitWords,
                                           sortCap, err);
    note_launch();
    return cudaGetLastError();
}

int batch_max_blocks_per_sm(int bitWords, bool withM5, int fam)
{
    const int sortCap = bitWords > 0 ? dbscan_sort_cap(bitWords * 32) : 0;
    const size_t smem = (size_t)kBatchWarps * dbscan_warp_words(bitWords, sortCap) * sizeof(unsigned);
    auto kern = batch_kernel_for(fam, withM5);
    if (smem > 48 * 1024)
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    int perSm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, kern, kBatchThreads, smem) != cudaSuccess)
        return 0;
    return perSm;
}

size_t batch_job_bytes() { return sizeof(BatchJob); }
int batch_threads() { return kBatchThreads; }
int batch_tile() { return kTile; }
int batch_max_jobs() { return kMaxBatchJobs; }

// Host-side plan: order by cost, prefix tile ends, packed device descriptors.
void batch_plan(const DevJob* jobs, void* const* outs, void* const* auxs, int n, int tile,
                std::vector<unsigned char>& packed, std::vector<long long>& tileEnd,
                std::vector<int>& order)
{
    order.resize(n);
    for (int i = 0; i < n; ++i) order[i] = i;
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) {
        return steps_per_point(jobs[a]) > steps_per_point(jobs[b]);
    });
    packed.assign((size_t)n * sizeof(BatchJob), 0);
    tileEnd.resize(n);
    long long acc = 0;
    for (int k = 0; k < n; ++k) {
        const int i = order[k];
        BatchJob b;
        memset(&b, 0, sizeof(b));
        b.job = jobs[i];
        b.out = outs[i];
        b.aux = auxs ? (int*)auxs[i] : nullptr;
        memcpy(packed.data() + (size_t)k * sizeof(BatchJob), &b, sizeof(b));
        acc += (jobs[i].nPoints + tile - 1) / tile;
        tileEnd[k] = acc;
    }
}

}  // namespace cbf
