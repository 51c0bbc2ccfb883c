// The surrogate network: 4 inputs -> fixed Fourier encoding (128) -> 256 -> 256
// -> 256 -> 17 (SiLU), BF16 operands, FP32 accumulation, trained and evaluated
// by this file's kernels.
//
// The 4 inputs are the system code, the two swept parameters mapped to [-1, 1]
// and the third parameter / 10.  The encoding, which is not trained, keeps them
// and adds sin(2 pi p_k), cos(2 pi p_k) of p_k = b_k0 x1 + b_k1 x2 for 62 fixed
// frequencies b_k: on raw coordinates a small MLP learns the smooth part of a
// regime map first and cannot resolve its fine structure, so it lost to the
// nearest coarse label; with the encoding it beats it.
//
// Output 0 is the (normalised) LLE, outputs 1..16 the logits of the 16-way
// peak-count regime class.  Parameters live as FP32 masters (Adam state next to
// them) plus BF16 copies that feed the tensor cores.  A training step is three
// kernels, captured once as a CUDA graph and replayed: minibatch, forward, loss and
// input gradients as one fused tcgen05 kernel, the weight gradients as one launch of
// split-K products, and their sums, the bias sums and Adam (mlp_step.cuh).
// Prediction over a whole grid is one fused tcgen05 kernel (mlp_tc.cuh); explicit
// feature rows run product by product (mlp_gemm_tc.cuh).
#include <cuda.h>
#include <cuda_bf16.h>
#include <math.h>
#include <string.h>

#include <algorithm>
#include <mutex>
#include <vector>

#include "mlp.cuh"

namespace cbf {

// kRaw network inputs, kFreq Fourier frequencies, kIn first-layer inputs
constexpr int kRaw = 4, kFreq = 62, kIn = kRaw + 2 * kFreq, kHid = 256, kOut = 17, kClasses = 16;

namespace {

typedef __nv_bfloat16 bf16;

// Parameter layout of the flat FP32 buffer: W1[256x4] b1 W2[256x256] b2 W3 b3 W4[17x256] b4.
constexpr long long kW1 = 0, kB1 = kW1 + kHid * kIn;
constexpr long long kW2 = kB1 + kHid, kB2 = kW2 + kHid * kHid;
constexpr long long kW3 = kB2 + kHid, kB3 = kW3 + kHid * kHid;
constexpr long long kW4 = kB3 + kHid, kB4 = kW4 + kOut * kHid;
constexpr long long kNumParams = kB4 + kOut;

// Row-major copies of the weights for the products of explicit feature rows: four
// 256 x 256 BF16 slots (row pitch 256), zero outside the weights: W1 (256 x 128),
// W2, W3, W4 (17 x 256, rows padded).
constexpr long long kSlot = (long long)kHid * kHid;
enum { kSlotW1 = 0, kSlotW2, kSlotW3, kSlotW4, kNumSlots };
constexpr int kXPitch = kIn;   // BF16 first-layer input rows
constexpr int kDOutPitch = 32;  // output gradients as an operand: 17 values padded to K = 32

// SiLU z * sigmoid(z) and its derivative.  The sigmoid's quotient uses the
// approximate reciprocal (__fdividef: a few ulp of FP32, far below the BF16
// rounding of every activation) instead of an IEEE division, whose correction
// steps were most of the epilogues' FP32 work; for 1 + e^-z beyond 2^126 it
// returns 0, the limit of z * sigmoid(z) there.
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi)
{
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}

// The encoding's frequencies (cycles per unit of the [-1, 1] axes): per value one
// xorshift64 word (state 0x5EED * 0x9E3779B97F4A7C15 + 1), b = (sum of its four
// low bytes - 510) / 16 -- an Irwin-Hall approximation of a normal distribution
// with standard deviation about 9, exact in FP32 (the oracle rebuilds the same
// table).  Measured on the 8192^2 Chen map (512^2 coarse labels + 65 536 random
// points): raw inputs 97.0 % class agreement, nearest coarse label 97.6 %,
// encoded inputs 98.2 %.
struct FreqTable {
    float b[kFreq][2];
};
constexpr FreqTable make_freqs()
{
    FreqTable t{};
    unsigned long long s = 0x5EEDull * 0x9E3779B97F4A7C15ull + 1ull;
    for (int k = 0; k < kFreq; ++k)
        for (int j = 0; j < 2; ++j) {
            s ^= s << 13;
            s ^= s >> 7;
            s ^= s << 17;
            int m = 0;
            for (int i = 0; i < 4; ++i) m += (int)((s >> (8 * i)) & 255ull);
            t.b[k][j] = (float)(m - 510) / 16.0f;
        }
    return t;
}
__constant__ FreqTable c_freq = make_freqs();

// Encoded first-layer inputs 8j .. 8j+7 of raw features x: e[0..3] = x, then
// e[4 + 2k] = sin(2 pi fs p_k), e[5 + 2k] = cos(2 pi fs p_k), p_k = fl(fl(b_k0 x1)
// + fl(b_k1 x2)), fs the network's frequency scale (a power of two, so 2 fs p_k
// is exact; sincospif: exact argument reduction).
__device__ __forceinline__ void encode8(const float (&x)[kRaw], int j, float fs, float (&e)[8])
{
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
        const int f = 8 * j + i;
        if (f < kRaw) {
            e[i] = x[f];
            e[i + 1] = x[f + 1];
        } else {
            const int k = (f - kRaw) >> 1;
            const float p = __fadd_rn(__fmul_rn(c_freq.b[k][0], x[1]), __fmul_rn(c_freq.b[k][1], x[2]));
            sincospif((2.0f * fs) * p, &e[i], &e[i + 1]);
        }
    }
}

__device__ __forceinline__ float silu(float z) { return __fdividef(z, 1.0f + __expf(-z)); }
__device__ __forceinline__ float silu_grad(float z)
{
    const float s = __fdividef(1.0f, 1.0f + __expf(-z));
    return s * (1.0f + z * (1.0f - s));
}

// ---- element-wise kernels -------------------------------------------------

__device__ __forceinline__ unsigned long long mix64(unsigned long long z)
{
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// Encoded BF16 rows of n raw feature rows X [n x 4].
__global__ void encode_rows_kernel(const float* __restrict__ X, long long n, float fs, bf16* __restrict__ xb)
{
    const long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    float x[kRaw];
#pragma unroll
    for (int f = 0; f < kRaw; ++f) x[f] = X[r * kRaw + f];
#pragma unroll 1
    for (int j = 0; j < kIn / 8; ++j) {
        float e[8];
        encode8(x, j, fs, e);
        reinterpret_cast<uint4*>(xb + r * kXPitch)[j] =
            make_uint4(pack_bf16x2(e[0], e[1]), pack_bf16x2(e[2], e[3]), pack_bf16x2(e[4], e[5]),
                       pack_bf16x2(e[6], e[7]));
    }
}

// Prediction head: LLE (de-normalised), argmax class, softmax confidence.
__global__ void head_kernel(const float* __restrict__ out, long long n, float lleMean, float lleStd,
                            float* __restrict__ lle, int* __restrict__ cls, float* __restrict__ conf)
{
    const long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    const float* o = out + r * kOut;
    int best = 0;
    float mx = o[1];
    for (int c = 1; c < kClasses; ++c)
        if (o[1 + c] > mx) {
            mx = o[1 + c];
            best = c;
        }
    float sum = 0.f;
    for (int c = 0; c < kClasses; ++c) sum += __expf(o[1 + c] - mx);
    if (lle) lle[r] = o[0] * lleStd + lleMean;
    if (cls) cls[r] = best;
    if (conf) conf[r] = 1.0f / sum;
}

__device__ __forceinline__ void point_features(const FeatureSpec& f, long long g, float (&x)[kRaw])
{
    const bool exact = f.J.exactGrid != 0;
    const double p0 = grid_value(g, f.J.nPts, f.J.ranges[0], f.J.ranges[1], 0, exact);
    const double p1 = grid_value(g, f.J.nPts, f.J.ranges[2], f.J.ranges[3], 1, exact);
    x[0] = f.sys;
    x[1] = ((float)p0 - f.lo0) * f.inv0 - 1.0f;
    x[2] = ((float)p1 - f.lo1) * f.inv1 - 1.0f;
    x[3] = f.third;
}

__global__ void features_kernel(const FeatureSpec f, const long long* __restrict__ idx, long long n,
                                float* __restrict__ X)
{
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    float x[kRaw];
    point_features(f, idx[k], x);
#pragma unroll
    for (int i = 0; i < kRaw; ++i) X[k * kRaw + i] = x[i];
}

#include "mlp_tc.cuh"
#include "mlp_gemm_tc.cuh"

__device__ __forceinline__ void put_weight(bf16* __restrict__ tw, unsigned char* __restrict__ wp, long long i, bf16 w);

#include "mlp_step.cuh"

// BF16 weight w = parameter i into its row-major slot (tw) and the operand layouts
// (wp; W2, W3 and W4 transposed too).  Biases have no copy.
__device__ __forceinline__ void put_weight(bf16* __restrict__ tw, unsigned char* __restrict__ wp, long long i, bf16 w)
{
    const auto pack = [&](uint32_t base, int R, int r, int k) { *reinterpret_cast<bf16*>(wp + base + tc_off(R, r, k)) = w; };
    if (i < kB1) {
        const int r = (int)(i / kIn), k = (int)(i % kIn);
        tw[kSlotW1 * kSlot + r * kHid + k] = w;
        pack(kPkW1, kHid, r, k);
    } else if (i >= kW2 && i < kB2) {
        const int r = (int)((i - kW2) / kHid), k = (int)((i - kW2) % kHid);
        tw[kSlotW2 * kSlot + (i - kW2)] = w;
        pack(kPkW2, kHid, r, k);
        pack(kPkW2T, kHid, k, r);
    } else if (i >= kW3 && i < kB3) {
        const int r = (int)((i - kW3) / kHid), k = (int)((i - kW3) % kHid);
        tw[kSlotW3 * kSlot + (i - kW3)] = w;
        pack(kPkW3, kHid, r, k);
        pack(kPkW3T, kHid, k, r);
    } else if (i >= kW4 && i < kB4) {
        const int r = (int)((i - kW4) / kHid), k = (int)((i - kW4) % kHid);
        tw[kSlotW4 * kSlot + (i - kW4)] = w;
        pack(kPkW4, kTcN4, r, k);
        pack(kPkW4T, kHid, k, r);
    }
}

// BF16 copies of the FP32 parameters.
__global__ void expand_params_kernel(const float* __restrict__ p, bf16* __restrict__ tw, unsigned char* __restrict__ wp,
                                     long long n)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) put_weight(tw, wp, i, __float2bfloat16_rn(p[i]));
}

template <class F>
cudaError_t launch1d(long long n, cudaStream_t s, F f)
{
    if (n <= 0) return cudaSuccess;
    const int t = 256;
    const long long b = (n + t - 1) / t;
    f((unsigned)b, t);
    note_launch();
    return cudaGetLastError();
}

}  // namespace

// ---------------------------------------------------------------------------

// Tensor maps of the products of explicit feature rows (fixed buffers, built once).
struct TcMaps {
    // A operands (128-row tiles of the prediction workspace), B operands W
    CUtensorMap pX, pH1, pH2, pH3, bW1, bW2, bW3, bW4;
};

struct Mlp {
    int B = 0;               // training batch
    long long Ba = 0;        // rows of every batch buffer: B rounded up to 128, at least 4096
    unsigned long long seed = 0;
    float encScale = 1.0f;    // frequency scale of the input encoding (a power of two)
    float* params = nullptr;  // FP32 masters (kNumParams)
    float* grads = nullptr;
    float* m1 = nullptr;
    float* m2 = nullptr;
    bf16* tw = nullptr;       // row-major BF16 weights (products of explicit rows)
    unsigned char* wp = nullptr;  // BF16 weights in the shared-memory operand layout (kPkBytes)
    // batch buffers
    float* xraw = nullptr;     // raw feature rows and labels of cbf_mlp_forward_backward
    float* yl = nullptr;
    int* yc = nullptr;
    unsigned char* ops = nullptr;  // the step kernel's operands, tile by tile
    float* out = nullptr;
    float* z = nullptr;        // pre-activations, in the one-CTA step kernel's own order
    int clusters = 0;          // clusters of the step kernel that are resident at once
    float* gradT = nullptr;    // FP32 dOut, dZ3, dZ2, dZ1, transposed, for the bias gradients
    float* loss = nullptr;
    float* ws = nullptr;      // split-K partials, one region per weight gradient
    int* gemmErr = nullptr;   // set by a kernel whose bounded wait ran out
    unsigned long long* step = nullptr;
    unsigned* finished = nullptr;  // blocks of the Adam kernel done
    TcMaps* maps = nullptr;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    const float* gX = nullptr;  // training set the graph was captured for
    const float* gYl = nullptr;
    const int* gYc = nullptr;
    long long gN = 0;
    float gLr = 0.f;
    int gHorizon = 0;
    float gW = 0.f;
    float gScale = 0.f;
    unsigned long long gSeed = 0;
    // prediction workspace (rows per chunk = kPredRows)
    bf16 *pxb = nullptr, *ph1 = nullptr, *ph2 = nullptr, *ph3 = nullptr;
    float* pout = nullptr;
    int* tcErr = nullptr;
};

constexpr int kPredRows = 262144;

namespace {

template <class T>
cudaError_t alloc_zero(T** p, long long n)
{
    const size_t bytes = (size_t)(n > 0 ? n : 1) * sizeof(T);
    cudaError_t e = cudaMalloc((void**)p, bytes);
    if (e == cudaSuccess) e = cudaMemset(*p, 0, bytes);
    return e;
}

cudaError_t pred_workspace(Mlp* m)
{
    if (m->pxb) return cudaSuccess;
    cudaError_t e = alloc_zero(&m->pxb, (long long)kPredRows * kXPitch);
    if (e == cudaSuccess) e = alloc_zero(&m->ph1, (long long)kPredRows * kHid);
    if (e == cudaSuccess) e = alloc_zero(&m->ph2, (long long)kPredRows * kHid);
    if (e == cudaSuccess) e = alloc_zero(&m->ph3, (long long)kPredRows * kHid);
    if (e == cudaSuccess) e = alloc_zero(&m->pout, (long long)kPredRows * kOut);
    TcMaps& mp = *m->maps;
    if (e == cudaSuccess) e = operand_map(&mp.pX, m->pxb, kPredRows, kXPitch, kXPitch, kGtM, 64);
    if (e == cudaSuccess) e = operand_map(&mp.pH1, m->ph1, kPredRows, kHid, kHid, kGtM, 64);
    if (e == cudaSuccess) e = operand_map(&mp.pH2, m->ph2, kPredRows, kHid, kHid, kGtM, 64);
    if (e == cudaSuccess) e = operand_map(&mp.pH3, m->ph3, kPredRows, kHid, kHid, kGtM, 64);
    return e;
}

// Forward on n rows whose BF16 inputs are in the prediction workspace.
cudaError_t forward(Mlp& m, int n, cudaStream_t s)
{
    const TcMaps& mp = *m.maps;
    cudaError_t e;
    TcGemm g = tc_gemm(kEpiHidden, m.gemmErr);
    g.M = n; g.N = kHid; g.BN = 128; g.Mv = n; g.Nv = kHid; g.ldh = kHid;
    g.K = kIn; g.KC = 64;
    g.bias = m.params + kB1; g.Hb = m.ph1;
    if ((e = gemm_tc(mp.pX, mp.bW1, g, s)) != cudaSuccess) return e;
    g.K = kHid;
    g.bias = m.params + kB2; g.Hb = m.ph2;
    if ((e = gemm_tc(mp.pH1, mp.bW2, g, s)) != cudaSuccess) return e;
    g.bias = m.params + kB3; g.Hb = m.ph3;
    if ((e = gemm_tc(mp.pH2, mp.bW3, g, s)) != cudaSuccess) return e;
    g = tc_gemm(kEpiOut, m.gemmErr);
    g.M = n; g.N = 32; g.BN = 32; g.Mv = n; g.Nv = kOut;
    g.K = kHid; g.KC = 64;
    g.bias = m.params + kB4; g.C = m.pout; g.ldc = kOut;
    return gemm_tc(mp.pH3, mp.bW4, g, s);
}

// K slices of the weight-gradient products (K = the batch rows padded to 64):
// 256 rows each, wider when that would exceed kMaxSplit slices.
int wgrad_slice(int K)
{
    int sl = 256;
    while ((K + sl - 1) / sl > kMaxSplit) sl += 64;
    return sl;
}

// Forward, loss and input gradients of n rows (mlp_step.cuh), then the partials of
// the weight gradients; *src is where the gradients are.
cudaError_t step_products(Mlp& m, StepArgs a, cudaStream_t s, GradSource* src)
{
    const int n = a.n;
    const long long tiles = (n + kTcM - 1) / kTcM;
    a.wp = m.wp;
    a.params = m.params;
    a.ops = m.ops;
    a.ld = m.Ba;
    a.gradT = m.gradT;
    a.loss = m.loss;
    a.err = m.gemmErr;
    // one wave of clusters, or one CTA a tile (both measured in mlp_step.cuh)
    if (tiles <= m.clusters) {
        mlp_step_cluster_kernel<<<(unsigned)tiles * kStC, kTcThreads, kStSmem, s>>>(a);
    } else {
        a.z = (float4*)m.z;
        mlp_step_kernel<<<(unsigned)tiles, kTcThreads, kTcSmem, s>>>(a);
    }
    note_launch();
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;

    const int Kb = (n + 63) / 64 * 64, slice = wgrad_slice(Kb), splits = (Kb + slice - 1) / slice;
    const long long wsLayer = (long long)kMaxSplit * kHid * kHid;
    WgradArgs W;
    memset(&W, 0, sizeof(W));
    const uint32_t as[4] = {kOpDOut, kOpDZ3, kOpDZ2, kOpDZ1}, bs[4] = {kOpH3, kOpH2, kOpH1, kOpX};
    const int M[4] = {kOut, kHid, kHid, kHid}, N[4] = {kHid, kHid, kHid, kIn};
    int ctas = 0;
    for (int l = 0; l < 4; ++l) {
        WgradProduct& p = W.p[l];
        p.a = as[l];
        p.b = bs[l];
        p.aBytes = l == 0 ? kTcM * kDOutPitch * 2 : kWgHalf;
        p.M = M[l];
        p.N = N[l];
        p.nx = (M[l] + kTcM - 1) / kTcM;
        p.first = ctas;
        p.ws = m.ws + l * wsLayer;
        ctas += p.nx * splits;
    }
    W.ops = m.ops;
    W.K = Kb;
    W.slice = slice;
    W.err = m.gemmErr;
    mlp_wgrad_kernel<<<ctas, kWgThreads, kWgSmem, s>>>(W);
    note_launch();
    *src = GradSource{m.ws, wsLayer, splits, m.gradT, m.Ba, n};
    return cudaGetLastError();
}

// Reads and clears the products' error flag (call after a synchronisation).
cudaError_t gemm_status(Mlp& m)
{
    int h = 0;
    cudaError_t e = cudaMemcpy(&h, m.gemmErr, sizeof(int), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess && h) {
        cudaMemset(m.gemmErr, 0, sizeof(int));
        e = cudaErrorLaunchTimeout;
    }
    return e;
}

}  // namespace

}  // namespace cbf

using namespace cbf;

struct cbf_mlp : Mlp {};

namespace {

cbf_status mlp_alloc(cbf_mlp* m, int B)
{
    cudaError_t e = cudaSuccess;
    m->B = B;
    const long long Ba = std::max<long long>(4096, ((long long)B + kGtM - 1) / kGtM * kGtM);
    m->Ba = Ba;
#define A_(ptr, n) if (e == cudaSuccess) e = alloc_zero(&m->ptr, (n))
    A_(params, kNumParams); A_(grads, kNumParams); A_(m1, kNumParams); A_(m2, kNumParams);
    A_(tw, kNumSlots * kSlot); A_(wp, (long long)kPkBytes);
    A_(xraw, Ba * kRaw); A_(yl, Ba); A_(yc, Ba);
    A_(ops, Ba / kTcM * kOpTile);
    A_(out, Ba * kOut); A_(gradT, kGradRows * Ba);
    A_(loss, 1); A_(step, 1); A_(finished, 1); A_(gemmErr, 1);
    A_(ws, 4ll * kMaxSplit * kHid * kHid);
#undef A_
    if (e != cudaSuccess) return report_cuda_error(e, "surrogate network buffers");
    m->maps = new TcMaps();
    TcMaps& mp = *m->maps;
    const auto slot = [&](int k) { return m->tw + k * kSlot; };
#define M_(map, p, R, C, ld, rows, kc) if (e == cudaSuccess) e = operand_map(&mp.map, p, R, C, ld, rows, kc)
    M_(bW1, slot(kSlotW1), kHid, kHid, kHid, 128, 64);
    M_(bW2, slot(kSlotW2), kHid, kHid, kHid, 128, 64);
    M_(bW3, slot(kSlotW3), kHid, kHid, kHid, 128, 64);
    M_(bW4, slot(kSlotW4), kHid, kHid, kHid, 32, 64);
#undef M_
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(gemm_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGtMaxSmem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(mlp_wgrad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWgSmem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(mlp_step_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTcSmem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(mlp_step_cluster_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kStSmem);
    if (e == cudaSuccess) {
        cudaLaunchConfig_t c = {};
        cudaLaunchAttribute at;
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = kStC;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        c.gridDim = dim3(kStC);
        c.blockDim = dim3(kTcThreads);
        c.dynamicSmemBytes = kStSmem;
        c.attrs = &at;
        c.numAttrs = 1;
        e = cudaOccupancyMaxActiveClusters(&m->clusters, mlp_step_cluster_kernel, &c);
    }
    if (e == cudaSuccess && Ba / kTcM > m->clusters) e = alloc_zero(&m->z, 3 * Ba * kHid);
    if (e != cudaSuccess) return report_cuda_error(e, "surrogate network tensor maps");
    return CBF_OK;
}

void mlp_free(cbf_mlp* m)
{
    if (m->exec) cudaGraphExecDestroy(m->exec);
    if (m->graph) cudaGraphDestroy(m->graph);
    void* ptrs[] = {m->params, m->grads, m->m1, m->m2, m->tw, m->wp, m->ops, m->xraw, m->yl, m->yc, m->z,
                    m->out, m->gradT, m->loss, m->ws,
                    m->gemmErr, m->step, m->finished, m->pxb, m->ph1, m->ph2, m->ph3, m->pout, m->tcErr};
    for (void* p : ptrs) cudaFree(p);
    delete m->maps;
    m->maps = nullptr;
}

// He-style uniform init from a fixed seed (host side, deterministic).
void init_params(std::vector<float>& p, unsigned long long seed)
{
    p.assign(kNumParams, 0.f);
    unsigned long long st = seed * 0x9E3779B97F4A7C15ull + 1;
    auto rnd = [&]() {
        st ^= st << 13;
        st ^= st >> 7;
        st ^= st << 17;
        return (double)(st >> 11) * (1.0 / 9007199254740992.0) * 2.0 - 1.0;
    };
    auto fill = [&](long long off, long long cnt, int fanIn) {
        const double bound = sqrt(6.0 / fanIn);
        for (long long i = 0; i < cnt; ++i) p[off + i] = (float)(rnd() * bound);
    };
    fill(kW1, (long long)kHid * kIn, kIn);
    fill(kW2, (long long)kHid * kHid, kHid);
    fill(kW3, (long long)kHid * kHid, kHid);
    fill(kW4, (long long)kOut * kHid, kHid);
}

cbf_status upload_params(cbf_mlp* m, const float* host)
{
    cudaError_t e = cudaMemcpy(m->params, host, kNumParams * sizeof(float), cudaMemcpyHostToDevice);
    if (e == cudaSuccess)
        e = launch1d(kNumParams, 0, [&](unsigned b, int t) {
            expand_params_kernel<<<b, t>>>(m->params, m->tw, m->wp, kNumParams);
        });
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e != cudaSuccess) return report_cuda_error(e, "surrogate parameters");
    return CBF_OK;
}

}  // namespace

extern "C" {

int64_t cbf_mlp_num_params(void) { return kNumParams; }

cbf_status cbf_mlp_create(int32_t batch, uint64_t seed, cbf_mlp** out)
{
    if (!out || batch < 1 || batch > (1 << 20))
        return report_error(CBF_ERR_INVALID_ARG, "batch must be in [1, 2^20]");
    cbf_mlp* m = new cbf_mlp();
    m->seed = seed;
    cbf_status st = mlp_alloc(m, batch);
    if (st != CBF_OK) {
        mlp_free(m);
        delete m;
        return st;
    }
    std::vector<float> p;
    init_params(p, seed);
    st = upload_params(m, p.data());
    if (st != CBF_OK) {
        mlp_free(m);
        delete m;
        return st;
    }
    *out = m;
    return CBF_OK;
}

void cbf_mlp_destroy(cbf_mlp* m)
{
    if (!m) return;
    mlp_free(m);
    delete m;
}

cbf_status cbf_mlp_get_params(cbf_mlp* m, float* host, int64_t n)
{
    if (!m || !host || n != kNumParams) return report_error(CBF_ERR_INVALID_ARG, "bad parameter buffer");
    cudaError_t e = cudaMemcpy(host, m->params, kNumParams * sizeof(float), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return report_cuda_error(e, "read parameters");
    return CBF_OK;
}

cbf_status cbf_mlp_set_params(cbf_mlp* m, const float* host, int64_t n)
{
    if (!m || !host || n != kNumParams) return report_error(CBF_ERR_INVALID_ARG, "bad parameter buffer");
    cudaMemset(m->m1, 0, kNumParams * sizeof(float));
    cudaMemset(m->m2, 0, kNumParams * sizeof(float));
    cudaMemset(m->step, 0, sizeof(unsigned long long));
    return upload_params(m, host);
}

// The encoding's frequency table (kFreq x 2 floats, row-major), as the kernels
// hold it in constant memory; n must be kFreq * 2.
cbf_status cbf_mlp_encoding_frequencies(float* out, int32_t n)
{
    if (!out || n != kFreq * 2) return report_error(CBF_ERR_INVALID_ARG, "the table holds 124 floats");
    constexpr FreqTable tab = make_freqs();
    for (int k = 0; k < kFreq; ++k) {
        out[2 * k] = tab.b[k][0];
        out[2 * k + 1] = tab.b[k][1];
    }
    return CBF_OK;
}

// Frequency scale of the input encoding: a power of two in [2^-8, 16].
cbf_status cbf_mlp_set_encoding_scale(cbf_mlp* m, float scale)
{
    int ex = 0;
    if (!m || !(scale >= 0x1p-8f && scale <= 16.0f) || frexpf(scale, &ex) != 0.5f)
        return report_error(CBF_ERR_INVALID_ARG, "encoding scale must be a power of two in [2^-8, 16]");
    m->encScale = scale;
    return CBF_OK;
}

// One forward + backward on host data (n <= batch rows); for gradient checks.
cbf_status cbf_mlp_forward_backward(cbf_mlp* m, const float* hx, const float* hyl, const int32_t* hyc,
                                    int32_t n, float wLle, float* hloss, float* hgrads, float* hout)
{
    if (!m || !hx || !hyl || !hyc || n < 1 || n > m->B)
        return report_error(CBF_ERR_INVALID_ARG, "bad batch");
    cudaError_t e = cudaMemcpy(m->xraw, hx, (size_t)n * kRaw * sizeof(float), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(m->yl, hyl, (size_t)n * sizeof(float), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(m->yc, hyc, (size_t)n * sizeof(int), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemset(m->loss, 0, sizeof(float));
    if (e == cudaSuccess) {
        StepArgs a;
        memset(&a, 0, sizeof(a));
        a.X = m->xraw; a.yl = m->yl; a.yc = m->yc; a.N = n; a.n = n;
        a.fs = m->encScale; a.wLle = wLle;
        a.out = m->out;
        GradSource src;
        e = step_products(*m, a, 0, &src);
        if (e == cudaSuccess) {
            mlp_grads_kernel<<<kParamBlocks + kBiasBlocks, kParamThreads>>>(src, m->grads);
            note_launch();
            e = cudaGetLastError();
        }
    }
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e == cudaSuccess) e = gemm_status(*m);
    if (e == cudaSuccess && hloss) e = cudaMemcpy(hloss, m->loss, sizeof(float), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess && hgrads)
        e = cudaMemcpy(hgrads, m->grads, kNumParams * sizeof(float), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess && hout)
        e = cudaMemcpy(hout, m->out, (size_t)n * kOut * sizeof(float), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return report_cuda_error(e, "forward/backward");
    return CBF_OK;
}

// `steps` Adam steps on minibatches drawn from the device training set
// (X [N x 4] FP32 features, normalised LLE targets, classes 0..15).  One step is
// captured as a CUDA graph on first use and replayed.
cbf_status cbf_mlp_train(cbf_mlp* m, const float* dX, const float* dYl, const int32_t* dYc, int64_t N,
                         int32_t steps, float lr, int32_t horizon, float wLle, float* hLosses,
                         void* stream)
{
    if (!m || !dX || !dYl || !dYc || N < 1 || steps < 0)
        return report_error(CBF_ERR_INVALID_ARG, "bad training arguments");
    cudaStream_t s = (cudaStream_t)stream;
    if (!s) return report_error(CBF_ERR_INVALID_ARG, "training needs a non-default stream");
    const int B = m->B;
    cudaError_t e = cudaSuccess;
    if (!m->exec || m->gX != dX || m->gYl != dYl || m->gYc != (const int*)dYc || m->gN != N || m->gLr != lr || m->gHorizon != horizon ||
        m->gW != wLle || m->gSeed != m->seed || m->gScale != m->encScale) {
        if (m->exec) cudaGraphExecDestroy(m->exec);
        if (m->graph) cudaGraphDestroy(m->graph);
        m->exec = nullptr;
        m->graph = nullptr;
        e = cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal);
        if (e != cudaSuccess) return report_cuda_error(e, "begin capture of the training step");
        StepArgs a;
        memset(&a, 0, sizeof(a));
        a.X = dX; a.yl = dYl; a.yc = (const int*)dYc; a.N = N; a.n = B;
        a.draw = 1; a.step = m->step; a.seed = m->seed;
        a.fs = m->encScale; a.wLle = wLle;
        GradSource src;
        cudaError_t ce = step_products(*m, a, s, &src);
        if (ce == cudaSuccess) {
            mlp_adam_kernel<<<kParamBlocks + kBiasBlocks, kParamThreads, 0, s>>>(src, m->params, m->m1, m->m2, m->tw,
                                                                                 m->wp, lr, horizon, 0.9f, 0.999f,
                                                                                 1e-8f, m->step, m->finished);
            note_launch();
            ce = cudaGetLastError();
        }
        cudaGraph_t gph = nullptr;
        e = cudaStreamEndCapture(s, &gph);
        if (ce != cudaSuccess) {
            if (gph) cudaGraphDestroy(gph);
            return report_cuda_error(ce, "capture of the training step");
        }
        if (e != cudaSuccess) return report_cuda_error(e, "end capture of the training step");
        m->graph = gph;
        e = cudaGraphInstantiate(&m->exec, gph, 0);
        if (e != cudaSuccess) return report_cuda_error(e, "instantiate the training graph");
        m->gX = dX;
        m->gYl = dYl;
        m->gYc = (const int*)dYc;
        m->gN = N;
        m->gLr = lr;
        m->gHorizon = horizon;
        m->gW = wLle;
        m->gScale = m->encScale;
        m->gSeed = m->seed;
    }
    for (int i = 0; i < steps && e == cudaSuccess; ++i) {
        if (hLosses) e = cudaMemsetAsync(m->loss, 0, sizeof(float), s);
        if (e == cudaSuccess) e = cudaGraphLaunch(m->exec, s);
        note_launch();
        if (e == cudaSuccess && hLosses)
            e = cudaMemcpyAsync(&hLosses[i], m->loss, sizeof(float), cudaMemcpyDeviceToHost, s);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e == cudaSuccess) e = gemm_status(*m);
    if (e != cudaSuccess) return report_cuda_error(e, "training");
    return CBF_OK;
}

// Predictions for N feature rows (device X [N x 4] FP32): LLE (de-normalised
// with lleMean/lleStd), class, softmax confidence.  Runs in chunks of kPredRows
// rows through its own workspace, then waits for the stream to read the
// products' error flag.
cbf_status cbf_mlp_predict(cbf_mlp* m, const float* dX, int64_t N, float lleMean, float lleStd,
                           float* dLle, int32_t* dCls, float* dConf, void* stream)
{
    if (!m || !dX || N < 0) return report_error(CBF_ERR_INVALID_ARG, "bad prediction arguments");
    cudaStream_t s = (cudaStream_t)stream;
    cudaError_t e = cudaSuccess;
    if ((e = pred_workspace(m)) != cudaSuccess) return report_cuda_error(e, "prediction workspace");
    for (long long r0 = 0; r0 < N && e == cudaSuccess; r0 += kPredRows) {
        const int n = (int)((N - r0) < kPredRows ? (N - r0) : kPredRows);
        e = launch1d(n, s, [&](unsigned b, int t) {
            encode_rows_kernel<<<b, t, 0, s>>>(dX + r0 * kRaw, n, m->encScale, m->pxb);
        });
        if (e == cudaSuccess) e = forward(*m, n, s);
        if (e == cudaSuccess)
            e = launch1d(n, s, [&](unsigned b, int t) {
                head_kernel<<<b, t, 0, s>>>(m->pout, n, lleMean, lleStd, dLle ? dLle + r0 : nullptr,
                                            dCls ? (int*)dCls + r0 : nullptr, dConf ? dConf + r0 : nullptr);
            });
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e == cudaSuccess) e = gemm_status(*m);
    if (e != cudaSuccess) return report_cuda_error(e, "prediction");
    return CBF_OK;
}

cbf_status cbf_mlp_predict_grid(cbf_mlp* m, const cbf_job* job, float lleMean, float lleStd, double* dLle,
                                int32_t* dCls, float* dConf, void* stream)
{
    if (!m || !job || !dLle || !dCls || !dConf) return report_error(CBF_ERR_INVALID_ARG, "bad prediction arguments");
    cbf::DevJob d;
    cbf_status st = cbf::lower_job_for(job, &d);
    if (st != CBF_OK) return st;
    if (d.dims != 2 || d.nIC != 3) return report_error(CBF_ERR_INVALID_ARG, "grid prediction needs a 2-D sweep of a 3-D system");
    const long long n = (long long)d.nPts * d.nPts;
    cudaError_t e = cbf::mlp_predict_grid(m, cbf::feature_spec(d), n, lleMean, lleStd, dLle, (int*)dCls, dConf,
                                          (cudaStream_t)stream);
    if (e != cudaSuccess) return report_cuda_error(e, "grid prediction");
    return CBF_OK;
}

cbf_status cbf_mlp_grid_features(const cbf_job* job, const int64_t* dIdx, int64_t n, float* dX, void* stream)
{
    if (!job || n < 0 || (n > 0 && (!dIdx || !dX))) return report_error(CBF_ERR_INVALID_ARG, "bad feature arguments");
    cbf::DevJob d;
    cbf_status st = cbf::lower_job_for(job, &d);
    if (st != CBF_OK) return st;
    cudaError_t e = cbf::mlp_features(cbf::feature_spec(d), (const long long*)dIdx, n, dX, (cudaStream_t)stream);
    if (e != cudaSuccess) return report_cuda_error(e, "grid features");
    return CBF_OK;
}

}  // extern "C"

namespace cbf {

FeatureSpec feature_spec(const DevJob& J)
{
    FeatureSpec f;
    memset(&f, 0, sizeof(f));
    f.J = J;
    f.sys = J.system == CBF_SYS_ROSSLER ? -1.0f : (J.system == CBF_SYS_LORENZ ? 0.0f : 1.0f);
    f.lo0 = (float)J.ranges[0];
    f.inv0 = J.ranges[1] != J.ranges[0] ? (float)(2.0 / (J.ranges[1] - J.ranges[0])) : 0.0f;
    f.lo1 = (float)J.ranges[2];
    f.inv1 = J.ranges[3] != J.ranges[2] ? (float)(2.0 / (J.ranges[3] - J.ranges[2])) : 0.0f;
    int third = 1;
    while (third == J.idxMut0 || third == J.idxMut1) ++third;
    f.third = third < 4 ? (float)(J.values[third] * 0.1) : 0.0f;
    return f;
}

cudaError_t mlp_features(const FeatureSpec& f, const long long* idx, long long n, float* X, cudaStream_t s)
{
    return launch1d(n, s, [&](unsigned b, int t) { features_kernel<<<b, t, 0, s>>>(f, idx, n, X); });
}

// One fused tcgen05 kernel over the whole grid (mlp_tc.cuh).  A wait that ran out
// inside the kernel is reported as cudaErrorLaunchTimeout.
cudaError_t mlp_predict_grid(cbf_mlp* m, const FeatureSpec& f, long long nPoints, float lleMean,
                             float lleStd, double* lle, int* cls, float* conf, cudaStream_t s)
{
    if (nPoints <= 0) return cudaSuccess;
    cudaError_t e = cudaSuccess;
    if (!m->tcErr) e = cudaMalloc((void**)&m->tcErr, sizeof(int));
    if (e != cudaSuccess) return e;
    if (e == cudaSuccess) e = cudaMemsetAsync(m->tcErr, 0, sizeof(int), s);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(mlp_predict_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTcSmem);
    int dev = 0, sms = 0;
    if (e == cudaSuccess) e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    const long long tiles = (nPoints + kTcM - 1) / kTcM;
    const unsigned grid = (unsigned)(tiles < sms ? tiles : sms);
    mlp_predict_tc_kernel<<<grid, kTcThreads, kTcSmem, s>>>(f, nPoints, m->encScale, m->wp, m->params, lleMean,
                                                            lleStd, lle, cls, conf, m->tcErr);
    note_launch();
    e = cudaGetLastError();
    int h = 0;
    if (e == cudaSuccess) e = cudaMemcpyAsync(&h, m->tcErr, sizeof(int), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e == cudaSuccess && h) e = cudaErrorLaunchTimeout;
    return e;
}

cudaError_t mlp_reset(cbf_mlp* m, unsigned long long seed)
{
    std::vector<float> p;
    init_params(p, seed);
    m->seed = seed;
    cudaError_t e = cudaMemset(m->m1, 0, kNumParams * sizeof(float));
    if (e == cudaSuccess) e = cudaMemset(m->m2, 0, kNumParams * sizeof(float));
    if (e == cudaSuccess) e = cudaMemset(m->step, 0, sizeof(unsigned long long));
    if (e == cudaSuccess && upload_params(m, p.data()) != CBF_OK) e = cudaErrorUnknown;
    return e;
}

}  // namespace cbf
