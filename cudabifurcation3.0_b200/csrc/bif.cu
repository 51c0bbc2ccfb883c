// Bifurcation diagrams and peak-based maps: integrate -> peaks -> KDE / DBSCAN.
//
// Reference pipeline (per chunk of points, three kernels and two HBM round trips
// of the full trajectory): calculateDiscreteModelCUDA writes record doubles per
// point (cudaLibrary.cu:78-117), peakFinderCUDA scans them (:220-284), then
// kdeCUDA (:356-441) or dbscanCUDA (:457-624) reduce each point.
//
// Here one fused kernel does all of it.  Each lane of a warp owns one point and
// keeps the ODE state in registers; the recorded variable is never stored: blocks
// of 16 samples feed a streaming state machine that reproduces peakFinder exactly
// (record_loop, PeakStream), and only the peaks (and intervals) go to a per-warp
// scratch slice in HBM.  Then a warp reduces one point at a time, cooperatively --
// its own tile's, and when the tiles have run out other warps' (EpilogueShare):
//   KDE    -- lanes take 32 consecutive sample positions; the signs of neighbouring
//             sums are settled by FP32 sums with an error bound where those can
//             decide, else by the reference's own sums (a double sum of FP32 expf in
//             its peak order, bit-identical); the plateau state machine then runs
//             over the signs (kde_warp).
//   DBSCAN -- labels and the reference's neighbour "stack" become two bitsets
//             in shared memory; the inner neighbour loop over k is a ballot
//             (its iterations are independent in the reference), popcount
//             updates the neighbour counter.
// A point's result leaves as one 4-byte store when its epilogue ends (OSTROVSKY,
// whose epilogues stay with their warp: one coalesced store per tile).
//
// Tiles are taken from a device counter: how long a point's epilogue takes
// depends on its peaks, and a fixed assignment left the warps with few of them
// idle at the end.  A tile holds 32 points where the map fills the GPU and fewer
// where it does not (tile_points): the steps of a warp's lanes run together, its
// epilogues one after the other.  Lorenz 1024^2: KDE map 302 -> 188 ms, DBSCAN map
// 207 -> 156 ms; where points of very many peaks reach the second pass (recorded
// variable z) 1152 -> 167 ms: a few dozen warps used to do all of them.
#include <algorithm>
#include <type_traits>

#include "bif_device.cuh"

namespace cbf {

namespace {

constexpr int kBifWarps = 4;
constexpr int kBifThreads = kBifWarps * 32;
// Peak slots per lane in the first pass of a KDE/DBSCAN/Ostrovsky map.  The
// reference's bound min(maxAmountOfPeaks, record/2) can be 10 000 and more;
// sizing every lane's scratch for it leaves room for 2-3 blocks per SM.  Points
// with more peaks than this (but not more than maxAmountOfPeaks, which only
// need the count) are listed and recomputed in a second pass at full capacity.
constexpr int kFirstPassPeaks = 1024;

// Sort buffer of the DBSCAN neighbour scans (keys per warp, a power of two
// >= 32): only where the peak capacity is at most kFirstPassPeaks, so that a
// block's shared memory stays at most 18 KB and eight blocks fit an SM.
__host__ __device__ inline int bif_sort_cap(int task, int peakCap)
{
    return task_with_intervals(task) && peakCap <= kFirstPassPeaks ? dbscan_sort_cap(peakCap) : 0;
}

// Points whose first-pass peak list was truncated: grid index and output slot.
struct Overflow {
    long long* g;
    long long* p;
    unsigned long long* count;
};

// ---------------------------------------------------------------------------
// Blocks per SM the kernel is compiled for.  A lane has one chain of FP64 steps,
// and a scheduler issues those best from a multiple of four warps: a bare chain
// of the 8-instruction step reaches 0.71 of the FP64 pipe with 4 or 8 warps per
// scheduler, 0.53 with 5 and 0.59 with 6 (the DBSCAN kernel's transient at 7 and
// at 8 blocks: 72 and 64 ms for 1024^2 x 100 000 steps).
template <class S>
constexpr int kBifMinBlocks = S::DIM == 3 ? 8 : 4;

// Scratch of a launch: peak slots (and intervals) of `tile` points per warp, the
// tile counter, and per warp `keyCap` floats for the KDE epilogue's sorted peaks
// where the shared memory does not hold them (0: none).
struct BifScratch {
    double* peaks;
    double* intervals;
    unsigned long long* queue;
    float* keys;
    int keyCap;
    int* err;
    EpilogueShare share;  // KDE and DBSCAN
};

// Tasks whose epilogues are shared (OSTROVSKY's need the integrating lane's flags).
__host__ __device__ constexpr bool task_shares(int task) { return task == CBF_TASK_KDE || task == CBF_TASK_DBSCAN; }

template <class S, int TASK>
__global__ void __launch_bounds__(kBifThreads, kBifMinBlocks<S>) bif_kernel(const DevJob J, void* __restrict__ d_out,
                                                                            int* __restrict__ d_aux,
                                                                            const BifScratch sc, int bitWords,
                                                                            int sortCap, int tilePts,
                                                                            const Overflow ov)
{
    extern __shared__ __align__(16) unsigned smem[];
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    const long long warpId = (long long)blockIdx.x * kBifWarps + wib;
    const long long nWarps = (long long)gridDim.x * kBifWarps;
    const long long nTiles = (J.nPoints + tilePts - 1) / tilePts;
    const int cap = J.peakCap;
    unsigned* L = smem + (size_t)wib * dbscan_warp_words(bitWords, sortCap);
    unsigned* Sb = L + bitWords;
    const DbscanSort so = dbscan_sort_area(L, bitWords, sortCap);
    double* ring = ring_column(L, lane);
    // Point j of the tile that warp `from` integrated.
    auto epilogue = [&](long long from, long long tile, int j) {
        const int n = sc.share.count[from * 32 + j];
        if (n < 0) return;
        const long long slot = from * tilePts + j;
        const double* pk = sc.peaks + slot * cap;
        int r;
        if constexpr (TASK == CBF_TASK_KDE)
            r = sc.keyCap > 0 ? kde_warp<false>(kde_spec(J), pk, n, lane, sc.keys + warpId * sc.keyCap, sc.keyCap)
                              : kde_warp<true>(kde_spec(J), pk, n, lane, reinterpret_cast<float*>(L), kKdeSortCap);
        else
            r = dbscan_warp(dbscan_spec(J), pk, sc.intervals + slot * cap, n, lane, L, Sb, sc.err, so);
        if (lane == 0) ((int*)d_out)[tile * tilePts + j] = r;
        __syncwarp();
    };

    for (long long next = warpId;; next += nWarps) {
        long long tile = next;
        if constexpr (task_shares(TASK)) {
            tile = (long long)epilogue_next_tile(sc.share, sc.queue, (unsigned long long)nTiles, lane);
        } else if (sc.queue) {
            unsigned long long t = 0;
            if (lane == 0) t = atomicAdd(sc.queue, 1ull);
            tile = (long long)__shfl_sync(kFull, t, 0);
        }
        if (tile >= nTiles) break;
        const long long p = tile * tilePts + lane;
        const bool valid = lane < tilePts && p < J.nPoints;
        const long long g = valid ? grid_index(J, p) : 0;

        if (TASK == CBF_TASK_PEAKS) {
            if (valid) {
                double* pk = (double*)d_out + p * (long long)cap;
                d_aux[p] = integrate_point<S, TASK>(J, g, pk, nullptr, cap, nullptr, nullptr, ring);
            }
            continue;
        }
        if (TASK == CBF_TASK_TRAJECTORY) {
            if (valid) {
                double* tr = (double*)d_out + p * (long long)cap;
                integrate_point<S, TASK>(J, g, nullptr, nullptr, 0, tr, d_aux + p, nullptr);
            }
            continue;
        }

        const long long slot0 = warpId * tilePts;
        double* myPk = sc.peaks + (slot0 + lane) * (long long)cap;
        double* myIv = task_with_intervals(TASK) ? sc.intervals + (slot0 + lane) * (long long)cap : nullptr;
        int n = 0, div = 0;
        OstrovskyFlags of;
        of.init(J.ostThr);
        if (valid) n = integrate_point<S, TASK>(J, g, myPk, myIv, cap, nullptr, &div, ring, &of);
        // A truncated peak list whose result needs every peak goes to the second pass.
        const bool over = valid && ov.count && n > cap && n <= J.maxPeaks;
        if (over) {
            const unsigned long long k = atomicAdd(ov.count, 1ull);
            ov.g[k] = g;
            ov.p[k] = p;
        }
        __syncwarp();

        if constexpr (task_shares(TASK)) {
            // what the number of peaks alone decides is written at once, and only the
            // points up to the last of the others are published
            int r = -1;
            if (valid && !over) r = TASK == CBF_TASK_KDE ? kde_by_count(n, J.maxPeaks) : dbscan_by_count(n, J.maxPeaks);
            if (r >= 0) ((int*)d_out)[p] = r;
            const unsigned left = __ballot_sync(kFull, valid && !over && r < 0);
            const int points = left ? highest_bit(left) + 1 : 0;
            epilogue_publish(sc.share, warpId, lane, (left >> lane) & 1u ? n : -1, points, (unsigned long long)tile);
            epilogue_own(sc.share, warpId, lane, points, [&](int j) { epilogue(warpId, tile, j); });
        } else {
            int res = 0;
            const int live = (int)min((long long)tilePts, J.nPoints - tile * tilePts);
            for (int j = 0; j < live; ++j) {
                const int nj = __shfl_sync(kFull, over ? 0 : n, j);
                const int r = dbscan_warp(dbscan_spec(J), sc.peaks + (slot0 + j) * (long long)cap,
                                          sc.intervals + (slot0 + j) * (long long)cap, nj, lane, L, Sb, sc.err, so);
                if (lane == j) res = r;
            }
            if (valid && !over) ((double*)d_out)[p] = ostrovsky_value(n, div != 0, of, res);
            __syncwarp();
        }
    }
    if constexpr (task_shares(TASK))
        epilogue_help<TASK == CBF_TASK_KDE ? 1 : 4>(sc.share, warpId, lane,
                      [&](long long from, unsigned long long tile, int j) { epilogue(from, (long long)tile, j); });
}

template <class T>
__global__ void scatter_kernel(const T* __restrict__ src, const long long* __restrict__ slot, long long n,
                               T* __restrict__ dst)
{
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) dst[slot[k]] = src[k];
}

// Points per tile of a map of n points: 32, or fewer where that leaves less than
// four warps for each of the SMs' four schedulers.  Up to three warps a scheduler
// the integration is bound by the latency of a lane's own chain (65 cycles a
// step, of which a warp issues 22), so it costs no more when fewer lanes of a
// warp are in use, and the epilogues of a tile -- serial within a warp -- spread
// over more warps (at four warps a step takes 90 cycles; with eight, 180).
// The steps with a division issue for about half their latency: two warps per
// scheduler for the 5-D model and Rossler (40^2 and 100^2 Rossler points, 9000 steps:
// KDE 1.08 and 1.16 ms, with four 1.21 and 1.47; 40^2, 22 000 steps, peaks 2.07 and
// 2.31, in tiles of 32 2.15).
template <class S>
int tile_points(long long n, int sms)
{
    const bool divides = S::DIM == 5 || std::is_same<S, Rossler>::value;
    const long long warps = (divides ? 8ll : 16ll) * sms;
    return (int)std::min(32ll, std::max(1ll, (n + warps - 1) / warps));
}

// Shape of one launch.
struct BifShape {
    int bitWords, sortCap, tile, keyCap;
    size_t smem;
    long long blocks;      // one per resident slot, or fewer
    size_t peakBytes;      // peak slots of a block
    size_t blockBytes;     // ... and its sorted keys
};

template <class S, int TASK>
cudaError_t bif_shape(const DevJob& J, int maxTile, bool keys, BifShape* sh)
{
    auto kern = bif_kernel<S, TASK>;
    sh->bitWords = task_with_intervals(TASK) ? (J.peakCap + 31) / 32 : 0;
    sh->sortCap = bif_sort_cap(TASK, J.peakCap);
    sh->smem = (size_t)kBifWarps * dbscan_warp_words(sh->bitWords, sh->sortCap) * sizeof(unsigned);
    cudaError_t e;
    if (sh->smem > 48 * 1024) {
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh->smem);
        if (e != cudaSuccess) return e;
    }
    int dev = 0, sms = 0, perSm = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, kern, kBifThreads, sh->smem)) != cudaSuccess)
        return e;
    if (perSm < 1) return cudaErrorInvalidConfiguration;
    // Trajectories have no epilogue to spread, and every lane stores each sample: 10 000
    // Rossler points of 6000 samples take 1.20 ms in tiles of 32, 1.55 in tiles of 5.
    sh->tile = TASK == CBF_TASK_TRAJECTORY ? 32 : std::min(maxTile, tile_points<S>(J.nPoints, sms));
    const long long nTiles = (J.nPoints + sh->tile - 1) / sh->tile;
    sh->blocks = std::min((nTiles + kBifWarps - 1) / kBifWarps, (long long)sms * perSm);
    sh->peakBytes = (size_t)kBifWarps * sh->tile * J.peakCap * sizeof(double) * (task_with_intervals(TASK) ? 2 : 1);
    sh->keyCap = 0;
    if (keys && TASK == CBF_TASK_KDE && J.peakCap > kKdeSortCap) {
        sh->keyCap = kKdeSortCap;
        while (sh->keyCap < J.peakCap && sh->keyCap < (1 << 20)) sh->keyCap <<= 1;
    }
    sh->blockBytes = sh->peakBytes + (size_t)kBifWarps * sh->keyCap * sizeof(float);
    return cudaSuccess;
}

// One launch of the fused kernel over the job's points (synchronises `s` where
// it takes scratch).
template <class S, int TASK>
cudaError_t bif_pass(const DevJob& J, void* d_out, int* d_aux, const Overflow& ov, cudaStream_t s)
{
    if (J.nPoints == 0) return cudaSuccess;
    const bool needScratch = (TASK == CBF_TASK_KDE || task_with_intervals(TASK));
    BifShape sh;
    cudaError_t e = bif_shape<S, TASK>(J, 32, true, &sh);
    if (e != cudaSuccess) return e;
    BifScratch sc{};
    char* mem = nullptr;
    if (needScratch) {
        size_t freeB = 0, totalB = 0;
        if ((e = cudaMemGetInfo(&freeB, &totalB)) != cudaSuccess) return e;
        const size_t budget = std::min(freeB / 4, (size_t)8 << 30);
        sh.blocks = std::min(sh.blocks, std::max(1ll, (long long)(budget / sh.blockBytes)));
        // [error flag, counter | shared epilogues | peaks | intervals | keys]
        size_t zeroed = 0;
        const size_t head = 256 + (epilogue_share_bytes(sh.blocks * kBifWarps, &zeroed) + 255) / 256 * 256;
        if ((e = cudaMallocAsync((void**)&mem, head + (size_t)sh.blocks * sh.blockBytes, s)) != cudaSuccess) return e;
        sc.err = (int*)mem;
        sc.queue = (unsigned long long*)(mem + 128);
        sc.share = epilogue_share(mem + 256, sh.blocks * kBifWarps);
        sc.peaks = (double*)(mem + head);
        if (task_with_intervals(TASK)) sc.intervals = sc.peaks + (size_t)sh.blocks * kBifWarps * sh.tile * J.peakCap;
        sc.keys = (float*)(mem + head + (size_t)sh.blocks * sh.peakBytes);
        sc.keyCap = sh.keyCap;
        if ((e = cudaMemsetAsync(mem, 0, 256 + zeroed, s)) != cudaSuccess) {
            cudaFreeAsync(mem, s);
            return e;
        }
    }
    bif_kernel<S, TASK><<<(unsigned)sh.blocks, kBifThreads, sh.smem, s>>>(J, d_out, d_aux, sc, sh.bitWords, sh.sortCap,
                                                                          sh.tile, ov);
    note_launch();
    e = cudaGetLastError();
    if (needScratch) {
        int hostErr = 0;
        cudaError_t e2 = cudaMemcpyAsync(&hostErr, sc.err, sizeof(int), cudaMemcpyDeviceToHost, s);
        cudaError_t e3 = cudaFreeAsync(mem, s);
        if (e == cudaSuccess) e = e2;
        if (e == cudaSuccess) e = e3;
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e == cudaSuccess && hostErr) return cudaErrorAssert;
    }
    return e;
}

// KDE / DBSCAN / Ostrovsky maps whose peak capacity exceeds kFirstPassPeaks run
// a first pass with that capacity -- more blocks per SM -- listing the points
// whose peaks did not fit, then a second pass over that list at full capacity,
// whose results are scattered into place.  Every point runs the same per-point
// code as in a single pass, so the output is identical.
template <class S, int TASK>
cudaError_t launch_bif_t(const DevJob& J, void* d_out, int* d_aux, cudaStream_t s)
{
    constexpr bool split = TASK == CBF_TASK_KDE || TASK == CBF_TASK_DBSCAN || TASK == CBF_TASK_OSTROVSKY;
    if (!split || J.peakCap <= kFirstPassPeaks || J.nPoints == 0)
        return bif_pass<S, TASK>(J, d_out, d_aux, Overflow{nullptr, nullptr, nullptr}, s);
    using Out = typename std::conditional<TASK == CBF_TASK_OSTROVSKY, double, int>::type;
    const long long n = J.nPoints;
    char* mem = nullptr;
    // list of grid indices and slots, count, and the second pass's outputs
    const size_t bytes = (size_t)n * (2 * sizeof(long long) + sizeof(Out)) + 256;
    cudaError_t e = cudaMallocAsync((void**)&mem, bytes, s);
    if (e != cudaSuccess) return e;
    Overflow ov{(long long*)mem, (long long*)mem + n, (unsigned long long*)((long long*)mem + 2 * n)};
    Out* tmp = (Out*)((char*)mem + (size_t)n * 2 * sizeof(long long) + 256);
    unsigned long long count = 0;
    e = cudaMemsetAsync(ov.count, 0, sizeof(unsigned long long), s);
    if (e == cudaSuccess) {
        DevJob J1 = J;
        J1.peakCap = kFirstPassPeaks;
        e = bif_pass<S, TASK>(J1, d_out, d_aux, ov, s);
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(&count, ov.count, sizeof(count), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e == cudaSuccess && count > 0) {
        DevJob J2 = J;
        J2.pointIndex = ov.g;
        J2.firstPoint = 0;
        J2.nPoints = (long long)count;
        e = bif_pass<S, TASK>(J2, tmp, nullptr, Overflow{nullptr, nullptr, nullptr}, s);
        if (e == cudaSuccess) {
            scatter_kernel<Out><<<(unsigned)(((long long)count + 255) / 256), 256, 0, s>>>(tmp, ov.p, (long long)count,
                                                                                         (Out*)d_out);
            note_launch();
            e = cudaGetLastError();
        }
    }
    cudaError_t e2 = cudaFreeAsync(mem, s);
    if (e == cudaSuccess) e = e2;
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    return e;
}

template <class S>
cudaError_t launch_bif_s(const DevJob& J, void* d_out, int* d_aux, cudaStream_t s)
{
    switch (J.task) {
    case CBF_TASK_PEAKS: return launch_bif_t<S, CBF_TASK_PEAKS>(J, d_out, d_aux, s);
    case CBF_TASK_KDE: return launch_bif_t<S, CBF_TASK_KDE>(J, d_out, d_aux, s);
    case CBF_TASK_DBSCAN: return launch_bif_t<S, CBF_TASK_DBSCAN>(J, d_out, d_aux, s);
    case CBF_TASK_TRAJECTORY: return launch_bif_t<S, CBF_TASK_TRAJECTORY>(J, d_out, d_aux, s);
    case CBF_TASK_OSTROVSKY: return launch_bif_t<S, CBF_TASK_OSTROVSKY>(J, d_out, d_aux, s);
    default: return cudaErrorInvalidValue;
    }
}

// One pass of the fused kernel with caller-provided scratch (no allocation);
// synchronises `s` to read the error flag.  The tile counter and the shared
// epilogues come first; where the scratch holds the lanes of few warps, tiles are
// smaller (more warps share it).
template <class S, int TASK>
cudaError_t prealloc_pass(const DevJob& J, void* d_out, double* scratch, size_t scratchBytes, int* err,
                          const Overflow& ov, cudaStream_t s)
{
    if (J.nPoints == 0) return cudaSuccess;
    const size_t perLane = (size_t)J.peakCap * sizeof(double) * (task_with_intervals(TASK) ? 2 : 1);
    int dev = 0, sms = 0;
    cudaError_t e;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    const long long lanes = (long long)(scratchBytes / perLane);
    BifShape sh;
    if ((e = bif_shape<S, TASK>(J, tile_points<S>(2 * lanes, sms), false, &sh)) != cudaSuccess) return e;
    const auto head = [&](long long blocks, size_t* zeroed) {
        return 256 + (epilogue_share_bytes(blocks * kBifWarps, zeroed) + 255) / 256 * 256;
    };
    size_t zeroed = 0;
    sh.blocks = std::min(sh.blocks, (long long)(scratchBytes / sh.peakBytes));
    while (sh.blocks > 0 && head(sh.blocks, &zeroed) + (size_t)sh.blocks * sh.peakBytes > scratchBytes) --sh.blocks;
    if (sh.blocks < 1) return cudaErrorInvalidValue;
    BifScratch sc{};
    sc.err = err;
    sc.queue = (unsigned long long*)scratch;
    sc.share = epilogue_share((char*)scratch + 256, sh.blocks * kBifWarps);
    sc.peaks = (double*)((char*)scratch + head(sh.blocks, &zeroed));
    if (task_with_intervals(TASK)) sc.intervals = sc.peaks + (size_t)sh.blocks * kBifWarps * sh.tile * J.peakCap;
    if ((e = cudaMemsetAsync(scratch, 0, 256 + zeroed, s)) != cudaSuccess) return e;
    bif_kernel<S, TASK><<<(unsigned)sh.blocks, kBifThreads, sh.smem, s>>>(J, d_out, nullptr, sc, sh.bitWords, sh.sortCap,
                                                                          sh.tile, ov);
    note_launch();
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    int hostErr = 0;
    if ((e = cudaMemcpyAsync(&hostErr, err, sizeof(int), cudaMemcpyDeviceToHost, s)) != cudaSuccess) return e;
    if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return e;
    return hostErr ? cudaErrorAssert : cudaSuccess;
}

// KDE / DBSCAN map with caller-provided scratch, in the regular entry point's two
// passes: when the peak capacity exceeds kFirstPassPeaks, a first pass at that
// capacity (many more blocks fit the scratch) lists the points whose peaks did
// not fit, a second pass recomputes them at full capacity and their results are
// scattered into place -- the same per-point code, the same map.  The scratch
// holds the overflow list (grid index and slot, 16 B per point) and the second
// pass's results (4 B per point) of a chunk of points in front of the peak
// buffers; the chunk is sized so that the list takes at most a quarter of the
// scratch and one block still fits at full capacity.  Without room for that,
// every point runs once at full capacity.
template <class S, int TASK>
cudaError_t launch_bif_prealloc_t(const DevJob& J, void* d_out, double* scratch, size_t scratchBytes,
                                  int* err, cudaStream_t s)
{
    const Overflow none{nullptr, nullptr, nullptr};
    if (J.nPoints == 0) return cudaSuccess;
    const size_t perBlockFull = (size_t)kBifThreads * J.peakCap * sizeof(double) * (task_with_intervals(TASK) ? 2 : 1);
    const size_t perPoint = 2 * sizeof(long long) + sizeof(int);
    size_t listBytes = scratchBytes / 4;
    if (scratchBytes < perBlockFull + 1024) listBytes = 0;
    else if (listBytes > scratchBytes - perBlockFull - 1024) listBytes = scratchBytes - perBlockFull - 1024;
    long long chunk = (long long)(listBytes / perPoint);
    if (J.peakCap <= kFirstPassPeaks || chunk < 32)
        return prealloc_pass<S, TASK>(J, d_out, scratch, scratchBytes, err, none, s);
    if (chunk > J.nPoints) chunk = J.nPoints;
    char* base = (char*)scratch;
    long long* listG = (long long*)base;
    long long* listP = listG + chunk;
    int* tmp = (int*)(listP + chunk);
    const size_t countOff = ((size_t)((char*)(tmp + chunk) - base) + 255) / 256 * 256;
    unsigned long long* count = (unsigned long long*)(base + countOff);
    const size_t peakOff = countOff + 256;
    double* peaks = (double*)(base + peakOff);
    const size_t peakBytes = scratchBytes - peakOff;
    cudaError_t e = cudaSuccess;
    for (long long first = 0; first < J.nPoints && e == cudaSuccess; first += chunk) {
        const long long m = (J.nPoints - first < chunk) ? J.nPoints - first : chunk;
        DevJob J1 = J;
        if (J.pointIndex) J1.pointIndex = J.pointIndex + first;
        else J1.firstPoint = J.firstPoint + first;
        J1.nPoints = m;
        J1.peakCap = kFirstPassPeaks;
        int* out = (int*)d_out + first;
        unsigned long long n2 = 0;
        e = cudaMemsetAsync(count, 0, sizeof(unsigned long long), s);
        if (e == cudaSuccess) e = prealloc_pass<S, TASK>(J1, out, peaks, peakBytes, err, Overflow{listG, listP, count}, s);
        if (e == cudaSuccess) e = cudaMemcpyAsync(&n2, count, sizeof(n2), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e == cudaSuccess && n2 > 0) {
            DevJob J2 = J;
            J2.pointIndex = listG;
            J2.firstPoint = 0;
            J2.nPoints = (long long)n2;
            e = prealloc_pass<S, TASK>(J2, tmp, peaks, peakBytes, err, none, s);
            if (e == cudaSuccess) {
                scatter_kernel<int><<<(unsigned)(((long long)n2 + 255) / 256), 256, 0, s>>>(tmp, listP, (long long)n2,
                                                                                         out);
                note_launch();
                e = cudaGetLastError();
            }
        }
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    return e;
}

template <class S>
cudaError_t launch_bif_prealloc_s(const DevJob& J, void* d_out, double* scratch, size_t scratchBytes,
                                  int* err, cudaStream_t s)
{
    switch (J.task) {
    case CBF_TASK_KDE: return launch_bif_prealloc_t<S, CBF_TASK_KDE>(J, d_out, scratch, scratchBytes, err, s);
    case CBF_TASK_DBSCAN: return launch_bif_prealloc_t<S, CBF_TASK_DBSCAN>(J, d_out, scratch, scratchBytes, err, s);
    default: return cudaErrorInvalidValue;
    }
}

static_assert(kBifThreads == kBifBlockThreads, "block size shared with other translation units");

}  // namespace

cudaError_t launch_bif_prealloc(const DevJob& J, void* d_out, double* scratch, size_t scratchBytes,
                                int* err, cudaStream_t s)
{
    switch (J.system) {
    case CBF_SYS_MEMRISTIVE5: return launch_bif_prealloc_s<Memristive5>(J, d_out, scratch, scratchBytes, err, s);
    case CBF_SYS_ROSSLER: return launch_bif_prealloc_s<Rossler>(J, d_out, scratch, scratchBytes, err, s);
    case CBF_SYS_LORENZ: return J.scaledStep ? launch_bif_prealloc_s<LorenzScaled>(J, d_out, scratch, scratchBytes, err, s) : launch_bif_prealloc_s<Lorenz>(J, d_out, scratch, scratchBytes, err, s);
    case CBF_SYS_CHEN: return J.scaledStep ? launch_bif_prealloc_s<ChenScaled>(J, d_out, scratch, scratchBytes, err, s) : launch_bif_prealloc_s<Chen>(J, d_out, scratch, scratchBytes, err, s);
    default: return cudaErrorInvalidValue;
    }
}

namespace {

// A warp per row: the row's first min(count, cap) values to packed[offset[row]..].
__global__ void pack_peaks_kernel(const double* __restrict__ peaks, const int* __restrict__ counts,
                                  const long long* __restrict__ offset, long long n, int cap,
                                  double* __restrict__ packed)
{
    const long long row = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (row >= n) return;
    const int m = min(max(counts[row], 0), cap);
    const double* src = peaks + row * cap;
    double* dst = packed + offset[row];
    for (int k = threadIdx.x & 31; k < m; k += 32) dst[k] = src[k];
}

}  // namespace

cudaError_t launch_pack_peaks(const double* peaks, const int* counts, const long long* offset, long long n, int cap,
                              double* packed, cudaStream_t s)
{
    if (n <= 0) return cudaSuccess;
    pack_peaks_kernel<<<(unsigned)((n + 7) / 8), 256, 0, s>>>(peaks, counts, offset, n, cap, packed);
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_bif(const DevJob& J, void* d_out, int* d_aux, cudaStream_t s)
{
    switch (J.system) {
    case CBF_SYS_MEMRISTIVE5: return launch_bif_s<Memristive5>(J, d_out, d_aux, s);
    case CBF_SYS_ROSSLER: return launch_bif_s<Rossler>(J, d_out, d_aux, s);
    case CBF_SYS_LORENZ: return J.scaledStep ? (J.unitStep ? launch_bif_s<LorenzScaledU>(J, d_out, d_aux, s) : launch_bif_s<LorenzScaled>(J, d_out, d_aux, s)) : launch_bif_s<Lorenz>(J, d_out, d_aux, s);
    case CBF_SYS_CHEN: return J.scaledStep ? (J.unitStep ? launch_bif_s<ChenScaledU>(J, d_out, d_aux, s) : launch_bif_s<ChenScaled>(J, d_out, d_aux, s)) : launch_bif_s<Chen>(J, d_out, d_aux, s);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace cbf
