// One training step of the surrogate network, apart from the weight gradients, as
// one kernel: a cluster of four CTAs takes 128 minibatch rows through the four
// forward products, the loss and the three input-gradient products.  Included by
// mlp.cu inside its anonymous namespace after mlp_tc.cuh, whose operand layout and
// helpers it shares.
//
//   stage  product                  K    N    epilogue
//   0..2   H(l-1) W(l)^T, l = 1..3  128/256 256  z = acc + b, h = SiLU(z)
//   3      H3 W4^T                  256  32   outputs, loss, dOut
//   4      dOut W4                  32   256  dZ3 = acc * SiLU'(z3)
//   5, 6   dZ(l+1) W(l+1), l = 2, 1 256  256  dZl = acc * SiLU'(zl)
//
// Each CTA computes 64 of a stage's 256 columns (stage 3, whose result all four
// need, is computed by each) and needs all of them as the next stage's A operand:
// its 64 columns are contiguous 8-column groups of 2 KB in the operand layout, which
// are sent to the other three CTAs, as soon as the four warps that wrote a group meet,
// by bulk copies that complete on the receivers' barriers.  The A
// operand has two buffers, so that no CTA waits for another's products: a slice of
// stage s + 1 goes out when the sender has finished stage s, for which it had every
// CTA's slice of stage s, sent when that CTA had finished stage s - 1, the last to
// read the buffer that stage s + 1 uses (dOut has a buffer of its own; stages 5 and 6
// reuse the buffers of stages 2 and 3).  Weights are copied two stages ahead.
//
// z stays in registers, 16 values per thread and layer.  What leaves the CTA are the
// A operands as they lie (X, H, dOut, dZ in BF16, by bulk copies while the products
// run) -- the weight gradients read them back as MN-major operands, so nothing is
// transposed -- and the FP32 dOut and dZ for the bias gradients, transposed (a warp
// stores a column of 32 rows at once).
//
// What bounds it is the chain of seven stages, not a unit: of the 7400 cycles of a
// middle stage, 2700 are the exchange (48 KB in and out of each SM), 1600 the sixteen
// products, 1500 the epilogue's arithmetic (sent group by group, it overlaps the
// exchange) and the rest waits.  A step of 4096 rows takes 53 us, of which this kernel
// is about 27; with one CTA for a tile (below) 17 us more; as eleven launches -- gather,
// four products, loss, three products, each with its own descriptor fetch,
// tensor-memory allocation and round trip through L2 -- 143 us.

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

// Contiguous copy to another CTA of the cluster, completing on its barrier.
__device__ __forceinline__ void bulk_s2s(uint32_t dst, uint32_t src, uint32_t bytes, uint32_t bar)
{
    asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     dst),
                 "r"(src), "r"(bytes), "r"(bar)
                 : "memory");
}
// `addr` of this CTA's shared memory as the same place in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t map_rank(uint32_t addr, int rank)
{
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
    return a;
}
__device__ __forceinline__ void cluster_sync_all()
{
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// 16 consecutive FP32 columns of this thread's tensor-memory lane.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16])
{
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
}

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
    float4* z;             // [3][tiles][16][512], the one-CTA kernel's
    float* gradT;          // [kGradRows][ld]
    float* out;            // optional: raw outputs, pitch kOut
    float* loss;
    int* err;
};

// The loss of one row (mean squared error on output 0, the normalised LLE, and
// cross-entropy of outputs 1..16), and its gradient d: columns 8 part .. 8 part + 7
// of it, or all (part -1).
__device__ __forceinline__ float row_loss(const float (&o)[kOut], float yl, int t, float wLle, float invB, int part,
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
    float ot = 0.f;
#pragma unroll
    for (int c = 0; c < kClasses; ++c) {
        if (c == t) ot = o[1 + c];
        if (part < 0 || part == (1 + c) / 8) d[1 + c] = (__expf(o[1 + c] - mx) / sum - (c == t ? 1.0f : 0.0f)) * invB;
    }
    const float lossCe = t >= 0 && t < kClasses ? -logf(fmaxf(__expf(ot - mx) / sum, 1e-30f)) : 0.f;
    return (wLle * e * e + lossCe) * invB;
}

constexpr int kStC = 4;                        // CTAs of a cluster
constexpr int kStN = kHid / kStC;              // columns of a CTA
constexpr uint32_t kStBBytes = kStN * kHid * 2;
constexpr uint32_t kStDBytes = kTcM * kDOutPitch * 2;
constexpr uint32_t kStCols = kStN;             // tensor-memory columns
constexpr size_t kStSmem = 2 * (size_t)kTcABytes + kStDBytes + 2 * kStBBytes + 64;
static_assert(kTcW4Bytes <= kStBBytes && kIn / 8 == 4 * kStC && kStN == 4 * 16 && kHid / 8 <= 32, "step kernel tiles");

__global__ void __cluster_dims__(kStC, 1, 1) __launch_bounds__(kTcThreads, 1)
    mlp_step_cluster_kernel(const StepArgs S)
{
    extern __shared__ __align__(1024) unsigned char tsm[];
    unsigned char* const D = tsm + 2 * kTcABytes;
    uint64_t* bars = reinterpret_cast<uint64_t*>(D + kStDBytes + 2 * kStBBytes);
    uint32_t* tslot = reinterpret_cast<uint32_t*>(bars + 5);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rank = (int)blockIdx.x % kStC, tile = (int)blockIdx.x / kStC;
    const uint32_t aAddr = smem_u32(tsm), dAddr = smem_u32(D), bAddr = dAddr + kStDBytes;
    const uint32_t abar = smem_u32(&bars[0]), wbar = smem_u32(&bars[2]), mbar = smem_u32(&bars[4]);

    const int q = warp & 3;      // tensor-memory lane quarter: tile rows 32q .. 32q+31
    const int part = warp >> 2;  // 16 of the CTA's 64 columns
    const int row = 32 * q + lane;
    const int col0 = rank * kStN + part * 16;
    const long long r = (long long)tile * kTcM + row;
    const bool rv = r < S.n;
    // the minibatch row (asked for before the set-up below, which takes as long)
    float x[kRaw] = {0.f, 0.f, 0.f, 0.f}, yl = 0.f;
    int yc = 0;
    if (rv) {
        long long i = r;
        if (S.draw) {
            const unsigned long long h = mix64(S.seed ^ mix64(*S.step * 0x100000001B3ull + (unsigned long long)r));
            i = (long long)(h % (unsigned long long)S.N);
        }
#pragma unroll
        for (int f = 0; f < kRaw; ++f) x[f] = S.X[i * kRaw + f];
        yl = S.yl[i];
        yc = S.yc[i];
    }

    if (tid == 0) {
        for (int i = 0; i < 5; ++i) mbar_init(smem_u32(&bars[i]), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)),
                     "r"(kStCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();  // every CTA's barriers exist before another's copies complete on them
    tc_fence_after();
    const uint32_t tmem = *tslot;

    const uint32_t laneBase = tmem + ((uint32_t)(32 * q) << 16);
    constexpr uint32_t wOff[kStepStages] = {kPkW1, kPkW2, kPkW3, kPkW4, kPkW4T, kPkW3T, kPkW2T};
    constexpr int kLen[kStepStages] = {kIn, kHid, kHid, kHid, kDOutPitch, kHid, kHid};
    int fetched = 0;

    // warp 1: stage s's weights (this CTA's rows of each 8-k group) into B buffer s % 2
    auto fetch = [&](int s) {
        fetched = s + 1;
        if (warp != 1) return;
        const uint32_t bar = wbar + (uint32_t)(s & 1) * 8u, groups = (uint32_t)kLen[s] / 8u;
        const uint32_t rows = s == 3 ? kTcN4 : kHid, piece = (s == 3 ? kTcN4 : kStN) * 16u;
        if (lane == 0) mbar_expect_tx(bar, groups * piece);
        __syncwarp();
        if ((uint32_t)lane < groups)
            bulk_g2s(bAddr + (uint32_t)(s & 1) * kStBBytes + (uint32_t)lane * piece,
                     S.wp + wOff[s] + (uint32_t)lane * rows * 16u + (s == 3 ? 0u : (uint32_t)rank * piece), piece, bar);
    };
    // stage s's products once its weights and its A operand are in (`a`: where it is;
    // `par`: phase of its buffer's barrier, -1: this CTA wrote all of it); every
    // thread waits for them
    auto products = [&](int s, uint32_t a, int par) -> bool {
        if (tid == 0) {
            bool go = mbar_wait(wbar + (uint32_t)(s & 1) * 8u, (uint32_t)(s >> 1) & 1u);
            if (go && par >= 0) go = mbar_wait(abar + (uint32_t)(a != aAddr) * 8u, (uint32_t)par);
            if (go) {
                tc_fence_after();
                const int nn = s == 3 ? kTcN4 : kStN;
                tc_issue(tmem, a, bAddr + (uint32_t)(s & 1) * kStBBytes, kLen[s] / 16, (uint32_t)nn * 16u,
                         tc_idesc(kTcM, nn));
                tc_commit(mbar);
            }
        }
        __syncwarp();
        const bool ok = __all_sync(0xffffffffu, mbar_wait(mbar, (uint32_t)s & 1u));
        tc_fence_after();
        return ok;
    };
    // 8 values of this thread's row as the 8 columns from c0 of the A operand at `base`
    auto to_operand = [&](unsigned char* base, int c0, const float* v) {
        *reinterpret_cast<uint4*>(base + tc_off(kTcM, row, c0)) = make_uint4(
            pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
    };
    // The four warps of a column part have written the 8 columns from c0 of the A
    // operand in `buf`: one of their threads sends them (2 KB) to the other CTAs
    // (exch) and to their place in the tile's operands.
    unsigned char* const ops = S.ops + (long long)tile * kOpTile;
    const bool sender = lane == 0 && (warp & 3) == 0;
    auto send = [&](uint32_t buf, int c0, uint32_t op, bool exch) {
        fence_async_smem();
        asm volatile("bar.sync %0, 128;" ::"r"(1 + part) : "memory");
        if (sender) {
            const uint32_t off = (uint32_t)(c0 / 8) * kOpGroup, src = buf + off;
            const uint32_t bar = abar + (uint32_t)(buf != aAddr) * 8u;
            if (exch)
                for (int t = 1; t < kStC; ++t) {
                    const int to = (rank + t) % kStC;
                    bulk_s2s(map_rank(src, to), src, kOpGroup, map_rank(bar, to));
                }
            bulk_s2g(ops + op + off, src, kOpGroup);
            bulk_commit();
        }
        __syncwarp();
    };
    // The CTA's part of the next A operand is written (exch: `bytes` come from the other
    // CTAs to the buffer of barrier exch).  False if a thread's wait ran out.
    auto handoff = [&](bool ok, int exch, uint32_t bytes) -> bool {
        fence_async_smem();
        tc_fence_before();
        // all but this operand's copies have been read: the operand before is overwritten next
        if (sender) asm volatile("cp.async.bulk.wait_group.read 2;" ::: "memory");
        if (__syncthreads_or(!ok)) return false;
        tc_fence_after();
        if (tid == 0 && exch >= 0) mbar_expect_tx(abar + (uint32_t)exch * 8u, (kStC - 1) * bytes);
        return true;
    };

    fetch(0);
    fetch(1);
    // the encoding of the row: eight of the inputs
    {
        float e[8];
        encode8(x, rank * 4 + part, S.fs, e);
        if (!rv)
#pragma unroll
            for (int i = 0; i < 8; ++i) e[i] = 0.f;
        to_operand(tsm, 8 * (rank * 4 + part), e);
    }
    send(aAddr, 8 * (rank * 4 + part), kOpX, true);
    bool fine = handoff(true, 0, 4 * kOpGroup);

    // A operand of each stage: its buffer (2: dOut) and the phase of its barrier
    constexpr int aBuf[kStepStages + 1] = {0, 1, 0, 1, 2, 0, 1, 0};
    constexpr int aPar[kStepStages] = {0, 0, 1, 1, -1, 0, 0};
    constexpr uint32_t opOff[kStepStages] = {kOpH1, kOpH2, kOpH3, kOpDOut, kOpDZ3, kOpDZ2, kOpDZ1};
    const float* const bias[3] = {S.params + kB1, S.params + kB2, S.params + kB3};
    float z[3][16];
#pragma unroll
    for (int s = 0; s < kStepStages; ++s) {
        if (!fine) break;
        float b[16];
        if (s < 3)
#pragma unroll
            for (int j = 0; j < 16; j += 4) {
                const float4 t = *reinterpret_cast<const float4*>(bias[s < 3 ? s : 0] + col0 + j);
                b[j] = t.x, b[j + 1] = t.y, b[j + 2] = t.z, b[j + 3] = t.w;
            }
        const bool ok = products(s, aBuf[s] == 2 ? dAddr : aAddr + (uint32_t)aBuf[s] * kTcABytes, aPar[s]);
        if (s + 2 < kStepStages && ok) fetch(s + 2);
        if (s == 3) {
            // every part has the whole row and takes eight columns of dOut
            float v[32], d[32];
            tmem_ld32(laneBase, v);
            const float* b4 = S.params + kB4;
#pragma unroll
            for (int c = 0; c < 32; ++c) d[c] = 0.f;
            float loss = 0.f;
            if (rv) {
                float o[kOut], g[kOut];
#pragma unroll
                for (int c = 0; c < kOut; ++c) o[c] = v[c] + b4[c];
                if (S.out && rank == 0 && part == 0)
#pragma unroll
                    for (int c = 0; c < kOut; ++c) S.out[r * kOut + c] = o[c];
                loss = row_loss(o, yl, yc, S.wLle, 1.0f / (float)S.n, part, g);
#pragma unroll
                for (int c = 0; c < kOut; ++c)
                    if (c / 8 == part) {
                        d[c] = g[c];
                        if (rank == 0) S.gradT[(long long)c * S.ld + r] = g[c];
                    }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (i == part) to_operand(D, 8 * i, d + 8 * i);
            if (rank == 0 && part == 0) {
#pragma unroll
                for (int m = 16; m > 0; m >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, m);
                if (lane == 0) atomicAdd(S.loss, loss);
            }
            fine = handoff(ok, -1, 0);
            if (fine && tid == 0 && rank == 0) {
                bulk_s2g(ops + opOff[s], dAddr, kStDBytes);
                bulk_commit();
            }
            continue;
        }
        const uint32_t next = aAddr + (uint32_t)aBuf[s + 1] * kTcABytes;
        float v[16];
        tmem_ld16(laneBase + (uint32_t)(part * 16), v);
#pragma unroll
        for (int h = 0; h < 16; h += 8) {
            if (s < 3) {
#pragma unroll
                for (int j = h; j < h + 8; ++j) {
                    z[s < 3 ? s : 0][j] = v[j] + b[j];
                    v[j] = silu(z[s < 3 ? s : 0][j]);
                }
            } else {
                const int l = s > 3 ? s - 4 : 0;  // dZ3, dZ2, dZ1 with z3, z2, z1
                float* gt = S.gradT + (long long)(kOut + l * kHid + col0) * S.ld + r;
#pragma unroll
                for (int j = h; j < h + 8; ++j) v[j] *= silu_grad(z[2 - l][j]);
                if (rv)
#pragma unroll
                    for (int j = h; j < h + 8; ++j) gt[(long long)j * S.ld] = v[j];
            }
            to_operand(tsm + aBuf[s + 1] * kTcABytes, col0 + h, v + h);
            send(next, col0 + h, opOff[s], s + 1 < kStepStages);
        }
        fine = handoff(ok, s + 1 < kStepStages ? aBuf[s + 1] : -1, (kStN / 8) * kOpGroup);
    }
    if (lane == 0) bulk_wait_read();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    cluster_sync_all();  // every copy between the CTAs has been sent and, where all went well, has landed
    if (!fine) {         // let those in flight land: the weights (bounded), the other CTAs' slices
        if (tid == 32)
            for (int f = fetched > 2 ? fetched - 2 : 0; f < fetched; ++f)
                mbar_wait(wbar + (uint32_t)(f & 1) * 8u, (uint32_t)(f >> 1) & 1u);
        for (int i = 0; i < 1000; ++i) __nanosleep(1000);
        __syncwarp();
    }
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kStCols) : "memory");
    if (!fine && tid == 0) atomicExch(S.err, 1);
}

// The same step with one CTA for 128 rows and all 256 columns (192 KB of operands,
// the weights of one stage at a time, z through global memory in the threads' own
// order): a stage takes longer, but the clusters' exchange -- 192 KB a stage between
// their CTAs -- and the fourfold barriers are saved.  For the batches of more tiles
// than clusters are resident at once: a step of 6144 rows takes 76 us (clusters: 90),
// of 37888 rows 234 (411); of 4096 rows 72 (55), of 256 rows 66 (50).
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
                    loss = row_loss(o, S.yl[i], S.yc[i], S.wLle, 1.0f / (float)S.n, -1, g);
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
// through tensor maps of 16-byte rows, a step took 17 us longer at 4096 rows:
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
// sums are added in order.  Sixteen loads in flight, and the bias warps in the first
// blocks of the grid: the columns of 4096 rows are the longest chain of the kernel
// (a step 55 -> 53 us against eight loads and last blocks; thirty-two take too many
// registers for the grid to be resident).
__device__ __forceinline__ float bias_grad(const GradSource& G, int c, int lane)
{
    const float* g = G.gradT + (long long)c * G.ld;
    float s = 0.f;
    for (int m = lane; m < G.n; m += 16 * 32) {
        float v[16];  // the loads together, the additions in order
#pragma unroll
        for (int u = 0; u < 16; ++u) v[u] = m + 32 * u < G.n ? g[m + 32 * u] : 0.f;
#pragma unroll
        for (int u = 0; u < 16; ++u)
            if (m + 32 * u < G.n) s += v[u];
    }
    float t = 0.f;
#pragma unroll
    for (int r = 0; r < 32; ++r) t += __shfl_sync(0xffffffffu, s, r);
    return t;
}

constexpr int kParamThreads = 256;
constexpr int kParamBlocks = (int)((kNumParams + kParamThreads - 1) / kParamThreads);
constexpr int kBiasBlocks = (kGradRows + kParamThreads / 32 - 1) / (kParamThreads / 32);

// use(i, gradient) for every parameter: a warp per bias (first: they take longest),
// a thread per weight.
template <class Use>
__device__ __forceinline__ void each_gradient(const GradSource& G, Use use)
{
    if ((int)blockIdx.x < kBiasBlocks) {
        const int c = (int)blockIdx.x * (kParamThreads / 32) + (int)(threadIdx.x >> 5);
        if (c < kGradRows) {
            const float g = bias_grad(G, c, threadIdx.x & 31);
            if ((threadIdx.x & 31) == 0) use(bias_param(c), g);
        }
    } else {
        const long long i = (long long)((int)blockIdx.x - kBiasBlocks) * kParamThreads + threadIdx.x;
        if (i < kNumParams && !is_bias(i)) use(i, weight_grad(G, i));
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
