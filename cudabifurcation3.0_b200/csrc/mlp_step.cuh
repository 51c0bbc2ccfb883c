// One training step of the surrogate network, apart from the weight gradients, as
// one kernel: a CTA takes 128 minibatch rows through the four forward products, the
// loss and the three input-gradient products.  Included by mlp.cu inside its
// anonymous namespace after mlp_tc.cuh, whose operand layout, helpers and CTA shape
// (512 threads, A and B operands in 192 KB of shared memory, a 128 x 256 FP32
// accumulator in tensor memory) it shares.
//
//   stage  product                  K    N    epilogue
//   0..2   H(l-1) W(l)^T, l = 1..3  128/256 256  z = acc + b, h = SiLU(z)
//   3      H3 W4^T                  256  32   outputs, loss, dOut
//   4      dOut W4                  32   256  dZ3 = acc * SiLU'(z3)
//   5, 6   dZ(l+1) W(l+1), l = 2, 1 256  256  dZl = acc * SiLU'(zl)
//
// Every stage's result is the next one's A operand and stays in shared memory; the
// next weights are copied while the epilogue runs.  What leaves the CTA are those A
// operands as they lie (X, H, dOut, dZ in BF16, by bulk copies while the products
// run) -- the weight gradients read them back as MN-major operands, so nothing is
// transposed --, the FP32 dOut and dZ for the bias gradients, transposed (a warp
// stores a column of 32 rows at once), and z, which the same threads read back
// (stored in their own order).
//
// Before, the step's chain was eleven launches of 6 to 15 us -- gather, four products,
// loss, three products, each with its own descriptor fetch, tensor-memory allocation
// and round trip through L2 -- 147 us a step with the weight gradients beside it, in
// which the tensor pipe was busy for 5 %.  As three kernels: 72 us.

// The weights in the operand layout (tc_off), in the order of the stages.
constexpr uint32_t kPkW1 = 0;
constexpr uint32_t kPkW2 = kPkW1 + kHid * kIn * 2;
constexpr uint32_t kPkW3 = kPkW2 + kHid * kHid * 2;
constexpr uint32_t kPkW4 = kPkW3 + kHid * kHid * 2;          // 32 rows, 17 used
constexpr uint32_t kPkW4T = kPkW4 + kTcN4 * kHid * 2;        // 256 x 32, 17 columns used
constexpr uint32_t kPkW3T = kPkW4T + kHid * kDOutPitch * 2;
constexpr uint32_t kPkW2T = kPkW3T + kHid * kHid * 2;
constexpr uint32_t kPkBytes = kPkW2T + kHid * kHid * 2;

constexpr int kStepStages = 7;
constexpr int kMaxSplit = 16;  // K slices of a weight gradient

// A tile's A operands (128 rows, layout tc_off(128, r, k)) in global memory.
constexpr uint32_t kOpX = 0;
constexpr uint32_t kOpH1 = kOpX + kTcM * kIn * 2;
constexpr uint32_t kOpH2 = kOpH1 + kTcABytes;
constexpr uint32_t kOpH3 = kOpH2 + kTcABytes;
constexpr uint32_t kOpDOut = kOpH3 + kTcABytes;   // 32 columns
constexpr uint32_t kOpDZ3 = kOpDOut + kTcM * kDOutPitch * 2;
constexpr uint32_t kOpDZ2 = kOpDZ3 + kTcABytes;
constexpr uint32_t kOpDZ1 = kOpDZ2 + kTcABytes;
constexpr uint32_t kOpTile = kOpDZ1 + kTcABytes;
constexpr uint32_t kOpGroup = kTcM * 16;          // 8 columns of an operand

// Contiguous shared -> global bulk copy (16-byte aligned, a multiple of 16 bytes),
// in this thread's next bulk group.
__device__ __forceinline__ void bulk_s2g(void* dst, uint32_t src, uint32_t bytes)
{
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(src), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

constexpr int kGradRows = kOut + 3 * kHid;  // rows of StepArgs::gradT: dOut, dZ3, dZ2, dZ1

struct StepArgs {
    const float* X;        // raw feature rows
    const float* yl;
    const int* yc;
    long long N;           // training rows
    int n;                 // minibatch rows
    int draw;              // 1: rows drawn by step and seed; 0: rows 0 .. n-1
    const unsigned long long* step;
    unsigned long long seed;
    float fs, wLle;
    const unsigned char* wp;
    const float* params;
    unsigned char* ops;    // [tiles][kOpTile]: the tile's A operands, in stage order
    long long ld;          // pitch of gradT
    float4* z;             // [3][tiles][16][512]
    float* gradT;          // [kGradRows][ld]
    float* out;            // optional: raw outputs, pitch kOut
    float* loss;
    int* err;
};

// The loss of one row (mean squared error on output 0, the normalised LLE, and
// cross-entropy of outputs 1..16), and its gradient d.
__device__ __forceinline__ float row_loss(const float (&o)[kOut], float yl, int t, float wLle, float invB,
                                          float (&d)[kOut])
{
    const float e = o[0] - yl;
    d[0] = 2.0f * wLle * e * invB;
    float mx = o[1];
#pragma unroll
    for (int c = 1; c < kClasses; ++c) mx = fmaxf(mx, o[1 + c]);
    float sum = 0.f;
#pragma unroll
    for (int c = 0; c < kClasses; ++c) sum += __expf(o[1 + c] - mx);
    float lossCe = 0.f;
#pragma unroll
    for (int c = 0; c < kClasses; ++c) {
        const float p = __expf(o[1 + c] - mx) / sum;
        d[1 + c] = (p - (c == t ? 1.0f : 0.0f)) * invB;
        if (c == t) lossCe = -logf(fmaxf(p, 1e-30f));
    }
    return (wLle * e * e + lossCe) * invB;
}

__global__ void __launch_bounds__(kTcThreads, 1) mlp_step_kernel(const StepArgs S)
{
    extern __shared__ __align__(1024) unsigned char tsm[];
    unsigned char* A = tsm;
    uint64_t* bars = reinterpret_cast<uint64_t*>(tsm + kTcABytes + kTcBBytes);
    uint32_t* tslot = reinterpret_cast<uint32_t*>(bars + 2);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t aAddr = smem_u32(tsm), bAddr = smem_u32(tsm + kTcABytes);
    const uint32_t wbar = smem_u32(&bars[0]), mbar = smem_u32(&bars[1]);

    if (tid == 0) {
        mbar_init(wbar, 1);
        mbar_init(mbar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)),
                     "r"(kTcCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tslot;

    const int q = warp & 3;      // tensor-memory lane quarter: tile rows 32q .. 32q+31
    const int part = warp >> 2;  // column quarter (64 columns) of the epilogues
    const int row = 32 * q + lane;
    const uint32_t laneBase = tmem + ((uint32_t)(32 * q) << 16);
    const long long r = (long long)blockIdx.x * kTcM + row;
    const bool rv = r < S.n;
    const long long tiles = gridDim.x;
    const uint32_t wOff[kStepStages] = {kPkW1, kPkW2, kPkW3, kPkW4, kPkW4T, kPkW3T, kPkW2T};
    const uint32_t wEnd[kStepStages] = {kPkW2, kPkW3, kPkW4, kPkW4T, kPkW3T, kPkW2T, kPkBytes};
    uint32_t wph = 0, mph = 0;

    // thread 0: bring stage s's weights into the B buffer (free by now)
    auto fetch = [&](int s) {
        if (tid != 0) return;
        const uint32_t bytes = wEnd[s] - wOff[s];
        mbar_expect_tx(wbar, bytes);
        for (uint32_t o = 0; o < bytes; o += 16384u)
            bulk_g2s(bAddr + o, S.wp + wOff[s] + o, bytes - o < 16384u ? bytes - o : 16384u, wbar);
    };
    // stage s's products once its weights are in; every thread waits for them
    auto products = [&](int s) -> bool {
        int fail = 0;
        if (tid == 0) {
            if (mbar_wait(wbar, wph)) {
                tc_fence_after();
                const int k = s == 0 ? kIn : (s == 4 ? kDOutPitch : kHid), nn = s == 3 ? kTcN4 : kHid;
                tc_issue(tmem, aAddr, bAddr, k / 16, (uint32_t)nn * 16u, tc_idesc(kTcM, nn));
                tc_commit(mbar);
            } else {
                fail = 1;
            }
        }
        wph ^= 1;
        if (__syncthreads_or(fail)) return false;
        const bool ok = mbar_wait(mbar, mph);
        mph ^= 1;
        tc_fence_after();
        if (tid == 0) bulk_wait_read();  // the A operand has been copied out: its buffer may be written
        return !__syncthreads_or(!ok);
    };
    // tensor-memory reads and A writes before the next products and the copy of the
    // A operand to its place in the tile's operands
    unsigned char* const ops = S.ops + (long long)blockIdx.x * kOpTile;
    auto handoff = [&](uint32_t op, uint32_t bytes) {
        fence_async_smem();
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
        if (tid == 0) {
            bulk_s2g(ops + op, aAddr, bytes);
            bulk_commit();
        }
    };
    // 32 values of this thread's row as 32 columns of the next A operand
    auto to_operand = [&](int col0, const float (&v)[32]) {
        uint32_t pk[16];
#pragma unroll
        for (int j = 0; j < 32; j += 2) pk[j / 2] = pack_bf16x2(v[j], v[j + 1]);
#pragma unroll
        for (int i = 0; i < 4; ++i)
            *reinterpret_cast<uint4*>(A + tc_off(kTcM, row, col0 + 8 * i)) =
                make_uint4(pk[4 * i], pk[4 * i + 1], pk[4 * i + 2], pk[4 * i + 3]);
    };
    fetch(0);
    {
        // the minibatch row and its encoding: column quarter `part` of the inputs
        float x[kRaw] = {0.f, 0.f, 0.f, 0.f};
        if (rv) {
            long long i = r;
            if (S.draw) {
                const unsigned long long h = mix64(S.seed ^ mix64(*S.step * 0x100000001B3ull + (unsigned long long)r));
                i = (long long)(h % (unsigned long long)S.N);
            }
#pragma unroll
            for (int f = 0; f < kRaw; ++f) x[f] = S.X[i * kRaw + f];
        }
        for (int jj = 0; jj < kIn / 32; ++jj) {
            const int j = part * (kIn / 32) + jj;
            float e[8];
            encode8(x, j, S.fs, e);
            if (!rv)
#pragma unroll
                for (int i = 0; i < 8; ++i) e[i] = 0.f;
            *reinterpret_cast<uint4*>(A + tc_off(kTcM, row, 8 * j)) =
                make_uint4(pack_bf16x2(e[0], e[1]), pack_bf16x2(e[2], e[3]), pack_bf16x2(e[4], e[5]),
                           pack_bf16x2(e[6], e[7]));
        }
    }
    handoff(kOpX, kTcM * kIn * 2);

    const uint32_t opOff[kStepStages] = {kOpH1, kOpH2, kOpH3, kOpDOut, kOpDZ3, kOpDZ2, kOpDZ1};
    const float* const bias[3] = {S.params + kB1, S.params + kB2, S.params + kB3};
    bool bad = false;
    for (int s = 0; s < kStepStages; ++s) {
        if (!products(s)) {
            bad = true;
            break;
        }
        if (s + 1 < kStepStages) fetch(s + 1);
        if (s < 3) {
            float4* zt = S.z + ((s * tiles + blockIdx.x) * 16) * kTcThreads + tid;
#pragma unroll 1
            for (int c = 0; c < 2; ++c) {
                const int col0 = part * 64 + c * 32;
                float v[32];
                tmem_ld32(laneBase + (uint32_t)col0, v);
#pragma unroll
                for (int j = 0; j < 32; ++j) v[j] += bias[s][col0 + j];
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    zt[(c * 8 + i) * kTcThreads] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
#pragma unroll
                for (int j = 0; j < 32; ++j) v[j] = silu(v[j]);
                to_operand(col0, v);
            }
        } else if (s == 3) {
            if (part == 0) {
                float v[32];
                tmem_ld32(laneBase, v);
                const float* b4 = S.params + kB4;
                float o[kOut], d[32];
#pragma unroll
                for (int c = 0; c < 32; ++c) d[c] = 0.f;
                float loss = 0.f;
                if (rv) {
#pragma unroll
                    for (int c = 0; c < kOut; ++c) o[c] = v[c] + b4[c];
                    if (S.out)
#pragma unroll
                        for (int c = 0; c < kOut; ++c) S.out[r * kOut + c] = o[c];
                    long long i = r;
                    if (S.draw) {
                        const unsigned long long h =
                            mix64(S.seed ^ mix64(*S.step * 0x100000001B3ull + (unsigned long long)r));
                        i = (long long)(h % (unsigned long long)S.N);
                    }
                    float g[kOut];
                    loss = row_loss(o, S.yl[i], S.yc[i], S.wLle, 1.0f / (float)S.n, g);
#pragma unroll
                    for (int c = 0; c < kOut; ++c) {
                        d[c] = g[c];
                        S.gradT[(long long)c * S.ld + r] = g[c];
                    }
                }
                to_operand(0, d);
#pragma unroll
                for (int m = 16; m > 0; m >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, m);
                if (lane == 0) atomicAdd(S.loss, loss);
            }
        } else {
            const int l = s - 4;  // dZ3, dZ2, dZ1 with z3, z2, z1
            const float4* zt = S.z + (((2 - l) * tiles + blockIdx.x) * 16) * kTcThreads + tid;
            float* gt = S.gradT + (long long)(kOut + l * kHid) * S.ld + r;
#pragma unroll 1
            for (int c = 0; c < 2; ++c) {
                const int col0 = part * 64 + c * 32;
                float v[32];
                tmem_ld32(laneBase + (uint32_t)col0, v);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float4 z = zt[(c * 8 + i) * kTcThreads];
                    v[4 * i] *= silu_grad(z.x);
                    v[4 * i + 1] *= silu_grad(z.y);
                    v[4 * i + 2] *= silu_grad(z.z);
                    v[4 * i + 3] *= silu_grad(z.w);
                }
                if (rv)
#pragma unroll
                    for (int j = 0; j < 32; ++j) gt[(long long)(col0 + j) * S.ld] = v[j];
                to_operand(col0, v);
            }
        }
        handoff(opOff[s], s == 3 ? kTcM * kDOutPitch * 2 : kTcABytes);
    }
    if (tid == 0) bulk_wait();
    if (bad && tid == 0) mbar_wait(wbar, wph ^ 1);  // the weights in flight, again bounded
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTcCols) : "memory");
    if (bad && tid == 0) atomicExch(S.err, 1);
}

// The weight gradients of all four layers, dW = dZ^T H over the minibatch, as one
// launch: tiles of 128 rows and the whole width of the four products side by side,
// split over K (the minibatch rows), partials to each layer's region of ws.  Seven
// tiles, so that sixteen slices are one wave; 128 x 128 tiles would be two.
//
// Both operands are columns of the step kernel's A operands, whose layout for K =
// rows is MN-major without swizzle: 8 columns x 8 rows of 16-byte pieces, 128 bytes
// to the next 8 rows (leading-dimension byte offset), kOpGroup to the next 8 columns
// (stride-dimension byte offset).  128 columns of a tile's 128 rows are one
// contiguous 32 KB copy.  (With the operands transposed in global memory and fetched
// through tensor maps of 16-byte rows, a step of 4096 rows took 89 us instead of 72:
// the transposed two-byte stores of the step kernel cost as much as the products.)
struct WgradProduct {
    uint32_t a, b;       // operands within a tile's operands
    uint32_t aBytes;     // bytes of A's columns (up to 128 of them)
    int M, N;            // result M x N (N 128 or 256)
    int nx, first;       // row tiles, first CTA
    float* ws;
};
struct WgradArgs {
    WgradProduct p[4];
    const unsigned char* ops;
    int K, slice;        // rows (a multiple of 64) and rows of a slice (a multiple of 64)
    int* err;
};

constexpr int kWgThreads = 256, kWgStages = 2;
constexpr uint32_t kWgHalf = 16 * kOpGroup;      // 128 columns of a tile: 32 KB
constexpr uint32_t kWgStage = 3 * kWgHalf;       // A, and B of up to 256 columns
constexpr size_t kWgSmem = (size_t)kWgStages * kWgStage + 64;

__global__ void __launch_bounds__(kWgThreads, 1) mlp_wgrad_kernel(const WgradArgs W)
{
    extern __shared__ __align__(1024) unsigned char tsm[];
    uint64_t* bars = reinterpret_cast<uint64_t*>(tsm + (size_t)kWgStages * kWgStage);  // full[], done
    uint32_t* slot = reinterpret_cast<uint32_t*>(bars + kWgStages + 1);
    int* flag = reinterpret_cast<int*>(slot + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    int l = 0;
    while (l < 3 && (int)blockIdx.x >= W.p[l + 1].first) ++l;
    const WgradProduct& P = W.p[l];
    const int i = (int)blockIdx.x - P.first;
    const int bx = i % P.nx, bz = i / P.nx;
    const int k0 = bz * W.slice, k1 = min(W.K, k0 + W.slice);
    const int t0 = k0 / kTcM, nt = (k1 + kTcM - 1) / kTcM - t0;
    const uint32_t base = smem_u32(tsm), doneBar = smem_u32(&bars[kWgStages]);

    if (tid == 0) {
        for (int j = 0; j <= kWgStages; ++j) mbar_init(smem_u32(&bars[j]), 1);
        *flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)),
                     "r"(256u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *slot;

    if (tid == 0) {
        const uint32_t bBytes = (uint32_t)(P.N / 8) * kOpGroup;
        const uint32_t idesc = tc_idesc(kTcM, P.N) | (1u << 15) | (1u << 16);  // both operands MN-major
        bool ok = true, first = true;
        for (int c = 0, pass = 0; c < nt && ok; c += kWgStages, ++pass) {
            const int cn = min(kWgStages, nt - c);
            const uint32_t par = (uint32_t)(pass & 1);
            for (int j = 0; j < cn; ++j) {
                const uint32_t fb = smem_u32(&bars[j]), at = base + (uint32_t)j * kWgStage;
                const unsigned char* tile = W.ops + (long long)(t0 + c + j) * kOpTile;
                mbar_expect_tx(fb, P.aBytes + bBytes);
                bulk_g2s(at, tile + P.a + (uint32_t)bx * kWgHalf, P.aBytes, fb);
                bulk_g2s(at + kWgHalf, tile + P.b, bBytes, fb);
            }
            int j = 0;
            for (; j < cn; ++j) {
                if (!mbar_wait(smem_u32(&bars[j]), par)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t at = base + (uint32_t)j * kWgStage;
                const int r0 = (t0 + c + j) * kTcM;
                for (int r = max(r0, k0); r < min(r0 + kTcM, k1); r += 16) {
                    const uint32_t off = (uint32_t)((r - r0) / 8) * 128u;
                    tc_mma(tmem, tc_desc(at + off, 128, kOpGroup), tc_desc(at + kWgHalf + off, 128, kOpGroup), idesc,
                           first ? 0u : 1u);
                    first = false;
                }
            }
            // on a failed wait: let the copies still in flight land (bounded)
            if (!ok)
                for (int m = j; m < cn; ++m) mbar_wait(smem_u32(&bars[m]), par);
            tc_commit(doneBar);
            if (!mbar_wait(doneBar, par)) ok = false;  // the products have read every stage
        }
        if (!ok) *flag = 1;
    }
    __syncthreads();
    tc_fence_after();
    const bool bad = *flag != 0;
    if (!bad && nt > 0) {
        const int q = warp & 3, row = bx * kTcM + 32 * q + lane;
        const uint32_t lb = tmem + ((uint32_t)(32 * q) << 16);
        for (int ch = warp >> 2; ch < P.N / 32; ch += 2) {
            float v[32];
            tmem_ld32(lb + (uint32_t)(ch * 32), v);
            if (row < P.M) store_f32x32(P.ws + ((long long)bz * P.M + row) * P.N + ch * 32, v);
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256u) : "memory");
    if (bad && tid == 0) atomicExch(W.err, 1);
}

// Where the gradient of a parameter comes from: the slices of its layer's split-K
// partials, added in order, or for a bias a column sum over the minibatch rows.
struct GradSource {
    const float* ws;
    long long wsLayer;
    int splits;
    const float* gradT;
    long long ld;
    int n;
};

__device__ __forceinline__ float weight_grad(const GradSource& G, long long i)
{
    int l;  // layers 4, 3, 2, 1: ws regions 0 .. 3
    long long at, mn;
    if (i < kB1) { l = 3; at = i - kW1; mn = (long long)kHid * kIn; }
    else if (i < kB2) { l = 2; at = i - kW2; mn = (long long)kHid * kHid; }
    else if (i < kB3) { l = 1; at = i - kW3; mn = (long long)kHid * kHid; }
    else { l = 0; at = i - kW4; mn = (long long)kOut * kHid; }
    const float* p = G.ws + l * G.wsLayer + at;
    float v[kMaxSplit];  // the loads together, the additions in order
#pragma unroll
    for (int z = 0; z < kMaxSplit; ++z) v[z] = z < G.splits ? p[z * mn] : 0.f;
    float acc = 0.f;
#pragma unroll
    for (int z = 0; z < kMaxSplit; ++z)
        if (z < G.splits) acc += v[z];
    return acc;
}

__device__ __forceinline__ bool is_bias(long long i)
{
    return (i >= kB1 && i < kW2) || (i >= kB2 && i < kW3) || (i >= kB3 && i < kW4) || i >= kB4;
}

// Row c of gradT belongs to this bias.
__device__ __forceinline__ long long bias_param(int c)
{
    if (c < kOut) return kB4 + c;
    c -= kOut;
    return (c < kHid ? kB3 : c < 2 * kHid ? kB2 : kB1) + c % kHid;
}

// A warp's sum of column c: lane t adds rows t, t + 32, ..., then the 32 partial
// sums are added in order.
__device__ __forceinline__ float bias_grad(const GradSource& G, int c, int lane)
{
    const float* g = G.gradT + (long long)c * G.ld;
    float s = 0.f;
    int m = lane;
    for (; m + 7 * 32 < G.n; m += 8 * 32) {
        float v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = g[m + 32 * u];
#pragma unroll
        for (int u = 0; u < 8; ++u) s += v[u];
    }
    for (; m < G.n; m += 32) s += g[m];
    float t = 0.f;
#pragma unroll
    for (int r = 0; r < 32; ++r) t += __shfl_sync(0xffffffffu, s, r);
    return t;
}

constexpr int kParamThreads = 256;
constexpr int kParamBlocks = (int)((kNumParams + kParamThreads - 1) / kParamThreads);
constexpr int kBiasBlocks = (kGradRows + kParamThreads / 32 - 1) / (kParamThreads / 32);

// use(i, gradient) for every parameter: a thread per weight, a warp per bias.
template <class Use>
__device__ __forceinline__ void each_gradient(const GradSource& G, Use use)
{
    if ((int)blockIdx.x < kParamBlocks) {
        const long long i = (long long)blockIdx.x * kParamThreads + threadIdx.x;
        if (i < kNumParams && !is_bias(i)) use(i, weight_grad(G, i));
    } else {
        const int c = ((int)blockIdx.x - kParamBlocks) * (kParamThreads / 32) + (int)(threadIdx.x >> 5);
        if (c < kGradRows) {
            const float g = bias_grad(G, c, threadIdx.x & 31);
            if ((threadIdx.x & 31) == 0) use(bias_param(c), g);
        }
    }
}

__global__ void __launch_bounds__(kParamThreads) mlp_grads_kernel(const GradSource G, float* __restrict__ grads)
{
    each_gradient(G, [&](long long i, float g) { grads[i] = g; });
}

// Adam on the flat FP32 parameters; refreshes the BF16 weight copies.  The last
// block to finish advances the step counter (every block has read it by then).
__global__ void __launch_bounds__(kParamThreads) mlp_adam_kernel(const GradSource G, float* __restrict__ p,
                                                                 float* __restrict__ m1, float* __restrict__ m2,
                                                                 bf16* __restrict__ tw, unsigned char* __restrict__ wp,
                                                                 float lr0, int horizon, float b1, float b2, float eps,
                                                                 unsigned long long* step, unsigned* finished)
{
    const unsigned long long at = *(volatile unsigned long long*)step;
    const float t = (float)(at + 1);
    // cosine decay from lr0 to lr0/20 over `horizon` steps (0: constant)
    float lr = lr0;
    if (horizon > 0) {
        const float u = fminf((float)at / (float)horizon, 1.0f);
        lr = lr0 * (0.05f + 0.95f * 0.5f * (1.0f + cospif(u)));
    }
    each_gradient(G, [&](long long i, float gi) {
        const float a = b1 * m1[i] + (1.f - b1) * gi;
        const float v = b2 * m2[i] + (1.f - b2) * gi * gi;
        m1[i] = a;
        m2[i] = v;
        const float ah = a / (1.f - powf(b1, t));
        const float vh = v / (1.f - powf(b2, t));
        const float w = p[i] - lr * ah / (sqrtf(vh) + eps);
        p[i] = w;
        put_weight(tw, wp, i, __float2bfloat16_rn(w));
    });
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(finished, 1u) == gridDim.x - 1) {
            *finished = 0;
            *step = at + 1;
        }
    }
}
