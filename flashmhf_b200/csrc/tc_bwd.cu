// Backward kernels, bf16, sm_100a.  The [T, E*d_e] intermediate is recomputed block by block.
//
//   M = Q K^T, N = Q U^T, sg = sigmoid(M), s = M*sg, dA = dO V^T          (per 64-row weight block)
//   dR_e = rowsum(dA*s*N), dM = dA*(r*N)*(sg + s*(1-sg)), dN = dA*s*r, A = s*N*r
//   dQ += dM K + dN U ;  dK = sum_t dM^T Q ;  dU = sum_t dN^T Q ;  dV = sum_t A^T dO
//
// Three kernels, each the sole owner of its accumulators (no floating-point atomics, bit-reproducible):
//
// bwd_dq_kernel  -- token-stationary.  One CTA owns 128 token rows of one (batch, head): its Q and dO
//   tiles are copied once into tensor memory and all three MMA chains read their A operand from there,
//   the head's weights stream through shared-memory rings (the first lap shares them with the Q and dO tiles).
//   Tensor memory: dQ accumulator (128 cols), Q and dO as bf16 (64 + 64), S = [M|N] (128), dA (64), and the
//   bf16 [dM|dN] operand of the dQ update (64).  Produces dQ (TMA store) and dR (direct stores).
//
// bwd_dw_kernel (d_h = 128)  -- weight-stationary.  One CTA owns one 64-row block of K, U and V of one K/U/V
//   head and a contiguous range of token tiles (the token axis is split `nsplit` ways to fill the
//   machine).  The recompute is transposed (lane = weight row), with K and U stacked in the 128 lanes; {Q, dO} tiles stream
//   through rings of 3.
// bwd_dwt_kernel (d_h = 64, 96)  -- the same with 128 weight rows per CTA, K and U side by side.
//   With more than one split each CTA writes fp32 partial sums to the workspace; dw_reduce_kernel adds the splits in a
//   fixed order and writes bf16 dK, dU, dV.
//
// All use 384 threads: warp 0 TMA producer, warps 1 to 3 MMA issuers (one per chain in bwd_dq_kernel, two chains each in the others, whose
// third, warp 3 of bwd_dw_kernel and warp 2 of bwd_dwt_kernel, fetches routing weights instead; warp 1 owns tensor memory), warps 4-11
// element-wise math (warp % 4 = TMEM lane quarter, (warp-4)/4 = which half of the columns).
#include <atomic>
#include <mutex>

#include "dw_plan.h"
#include "kernels.h"
#include "tc_common.cuh"
#include "tensormap.cuh"

namespace fmhf {
namespace {

// Element-wise warps: 4 lane quarters x two column parts of a 64-column block (a thread = one token row x kCols columns).  The fixed part
// of a block's element-wise step (barrier waits, tensor-memory load and store latencies) does not shrink with narrower threads:
// four parts are 2-4 % slower.
constexpr int kCols = 32;
constexpr int kBT = 128, kBI = 64, kActThreads = 256, kThreads = 128 + kActThreads;
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kTile = kBT * 128;    // one 128-row x 64-col SW128 chunk: 16 KB
constexpr uint32_t kWChunk = kBI * 128;  // one 64-row x 64-col chunk: 8 KB

// dQ/dR: element-wise backward math for two neighbouring intermediate columns of one token row, on packed
// fp32 pairs.  m, n are the raw products Q K^T, Q U^T; with the layer's constants s0 (head), s1 (up),
// s2 (final) the forward is A = silu(s0 m) (s1 n) s2 r.  With t = tanh(s0 m / 2): sg = sigmoid(s0 m) =
// 0.5 + 0.5 t, s = m*sg (so silu(s0 m) = s0 s), silu'(s0 m) = sg + s * s0 (1 - sg).  All three constants
// fold into the per-row factor r2 = s0 s1 s2 r and into the two constants below, at no cost per element:
//   dM = dA r2 n silu'(s0 m),  dN = dA r2 s,  A = s n r2,  dR = s0 s1 s2 * sum dA s n.
struct DqConst {
    f32x2 half_s0, p_half_s0, n_half_s0;  // (s0/2), (s0/2), (-s0/2): tanh argument scale and s0 (1 - sg) = s0/2 - (s0/2) t
};
__device__ __forceinline__ DqConst dq_const(float s0) {
    return DqConst{f2_pack(0.5f * s0, 0.5f * s0), f2_pack(0.5f * s0, 0.5f * s0), f2_pack(-0.5f * s0, -0.5f * s0)};
}
struct DqPair {
    f32x2 dm, dn, sn, da;  // dM, dN, s*N (times r2 gives A, times dA sums to dR / (s0 s1 s2)), dA
};
__device__ __forceinline__ DqPair dq_pair(f32x2 m, f32x2 n, f32x2 da, f32x2 r2, const DqConst &k) {
    const f32x2 half = f2_pack(0.5f, 0.5f);
    const f32x2 t = f2_tanh(f2_mul(m, k.half_s0));
    const f32x2 sg = f2_fma(t, half, half);
    const f32x2 omsg = f2_fma(t, k.n_half_s0, k.p_half_s0);
    const f32x2 s = f2_mul(m, sg);
    const f32x2 dsilu = f2_fma(s, omsg, sg);
    const f32x2 dar = f2_mul(da, r2);
    DqPair o;
    o.sn = f2_mul(s, n);
    o.dn = f2_mul(dar, s);
    o.dm = f2_mul(f2_mul(dar, n), dsilu);
    o.da = da;
    return o;
}

// dK/dU/dV: the same for that kernel, cut where dA comes in.  With h = s0/2, t = tanh(h m):
//   silu(s0 m) = h S with S = m + m t,   2 silu'(s0 m) = D = (1 + h m) + t ((1 + h m) - h S)      (sigmoid = (1 + t) / 2)
// and with the per-row factor rho = h s1 s2 r, carried through (q = rho S, w = n rho D),
//   A = q n,  dN = dA q,  dM = dA w:
// 8 operations before dA, which run while the tensor core still computes it, and 2 after.
struct DwConst {
    f32x2 h, nh;  // h, -h, twice each
};
__device__ __forceinline__ DwConst dw_const(float s0) { return DwConst{f2_pack(0.5f * s0, 0.5f * s0), f2_pack(-0.5f * s0, -0.5f * s0)}; }
struct DwPair {
    f32x2 q, w, a;  // dN = dA q, dM = dA w, A
};
__device__ __forceinline__ DwPair dw_pair(f32x2 m, f32x2 n, f32x2 rho, const DwConst &k) {
    const f32x2 t = f2_tanh(f2_mul(m, k.h));
    const f32x2 mr = f2_mul(m, rho);
    const f32x2 q = f2_fma(mr, t, mr);
    const f32x2 d = f2_fma(mr, k.h, rho);
    const f32x2 e = f2_fma(t, f2_fma(q, k.nh, d), d);
    return DwPair{q, f2_mul(n, e), f2_mul(q, n)};
}

// =============================================================================================
//                                       dQ / dR kernel
// =============================================================================================
template <int DH>
struct DqSmem {
    static constexpr int kChunks = (DH + 63) / 64;
    static constexpr uint32_t kQBytes = kChunks * kTile;
    static constexpr uint32_t kKUStage = kChunks * 2 * kWChunk;  // per chunk: [K;U] = 128 rows
    static constexpr uint32_t kVStage = kChunks * kWChunk;
    // Q and dO are needed in shared memory only until they are copied to tensor memory: they arrive in the last two stages of
    // the [K;U] ring, which joins the ring after that (the ring's first lap waits for it there), and dQ leaves through one of them.
    // With tiles of their own the rings had three and two stages, too few for the way of a stage from L2.
    static constexpr int kKUStages = DH == 64 ? 8 : 5, kVStages = DH == 64 ? 8 : 4;
    static_assert(kQBytes == kKUStage, "a token tile takes one [K;U] stage");
    static constexpr uint32_t kOffKU = 0;
    static constexpr uint32_t kOffQ = kOffKU + (kKUStages - 2) * kKUStage, kOffdO = kOffQ + kQBytes;
    static constexpr uint32_t kOffV = kOffKU + kKUStages * kKUStage;
    static constexpr uint32_t kOffCtl = kOffV + kVStages * kVStage;
    static constexpr uint32_t kCtlBytes = 384 + 2 * 128 * 4;  // barriers + two sets of dR exchange rows
    static constexpr uint32_t kTotal = kOffCtl + kCtlBytes + 1024;
};

// Barriers.  Q and dO are copied once into tensor memory (QT); S, dA and the [dM|dN] operand each have ONE buffer
// there, because the accumulator, Q and dO take half of tensor memory:
//   SFULL (S and dA of the block computed: one commit from each of their issuers), SEMPTY (both are in the
//   element-wise warps' registers), PFULL ([dM|dN] written), PEMPTY (the dQ update that read it is done).
// All of them complete once per block and every waiter waits on every phase, so a one-bit parity is enough.
constexpr int kMaxRing = 8;
enum { DQ_QFULL = 0, DQ_SFULL = 1, DQ_SEMPTY = 2, DQ_PFULL = 3, DQ_PEMPTY = 4, DQ_ACCFULL = 5, DQ_QT = 6, DQ_DRFULL = 7, DQ_DRFREE = 9,
       DQ_KUFULL = 11, DQ_KUEMPTY = DQ_KUFULL + kMaxRing, DQ_VFULL = DQ_KUEMPTY + kMaxRing, DQ_VEMPTY = DQ_VFULL + kMaxRing,
       DQ_BARS = DQ_VEMPTY + kMaxRing };
static_assert(DQ_BARS * 8 + 8 <= 384, "control area");

struct DqArgs {
    const float *R;
    long long r_sb, r_sh, r_ss;
    float *dR;
    long long dr_sb, dr_sh, dr_ss;
    int S, E, De, G;
    // Few token tiles: the sub-networks are split over CTAs, e_per_split each (blockIdx.x = tile * nsplit + split).  A CTA then
    // writes an fp32 partial dQ to `part` ([nsplit][B][H][S][DH], added by the split reduction) and dR of its own sub-networks.
    int nsplit, e_per_split, H, B;
    float *part;
    float s0, c;  // head_scaling; head_scaling * up_scaling * final_scaling
    WaitArgs wait;
};

template <int DH>
__global__ void __maxnreg__(152)
bwd_dq_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmdO,
              const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmU,
              const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdQ, const DqArgs args) {
    using L = DqSmem<DH>;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t *gbase = smem_raw + (base - raw);
    const uint32_t sQ = base + L::kOffQ, sdO = base + L::kOffdO, sKU = base + L::kOffKU, sV = base + L::kOffV,
                   sBar = base + L::kOffCtl;
    volatile uint32_t *tmem_slot = reinterpret_cast<volatile uint32_t *>(gbase + L::kOffCtl + DQ_BARS * 8);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(gbase + L::kOffCtl + DQ_BARS * 8 + 4);
    volatile float *drx = reinterpret_cast<volatile float *>(gbase + L::kOffCtl + 384);  // [2][128]
    auto bar = [&](int i) { return sBar + 8u * i; };

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int isplit = blockIdx.x % args.nsplit, e0 = isplit * args.e_per_split, ne = min(args.E - e0, args.e_per_split);
    const int t0 = (int)(blockIdx.x / args.nsplit) * kBT, h = blockIdx.y, b = blockIdx.z, hk = h / args.G;
    const int bpe = args.De / kBI, nblk = ne * bpe;
    const WaitCtl ctl{abort_flag, args.wait};
    constexpr int W = kKernelBwdDq * 100;
    // Tensor memory: dQ accumulator, Q and dO as bf16 A operands (64 columns each), S = [M | N], dA, [dM | dN] (bf16).
    constexpr uint32_t kColAcc = 0, kColQ = 128, kColdO = 192, kColS = 256, kColdA = 384, kColP = 448;

    if (threadIdx.x == 0) {
        *abort_flag = launch_aborted(args.wait);  // a CTA of this launch gave up: drain fast
        mbar_init(bar(DQ_QFULL), 1);
        for (int s = 0; s < L::kKUStages; ++s) { mbar_init(bar(DQ_KUFULL + s), 1); mbar_init(bar(DQ_KUEMPTY + s), 1); }
        for (int s = 0; s < L::kVStages; ++s) { mbar_init(bar(DQ_VFULL + s), 1); mbar_init(bar(DQ_VEMPTY + s), 1); }
        mbar_init(bar(DQ_SFULL), 2);                          // one commit from each of the two recompute issuers
        mbar_init(bar(DQ_SEMPTY), arrivals_of(kActThreads));  // S and dA are in registers
        mbar_init(bar(DQ_PFULL), arrivals_of(kActThreads));   // [dM|dN] written
        mbar_init(bar(DQ_PEMPTY), 1);                         // the dQ update that read [dM|dN] is done
        mbar_init(bar(DQ_QT), arrivals_of(kActThreads));      // Q and dO copied to tensor memory
        for (int i = 0; i < 2; ++i) {
            mbar_init(bar(DQ_DRFULL + i), arrivals_of(128));  // column part 1 has written its dR_e partial sums
            mbar_init(bar(DQ_DRFREE + i), arrivals_of(128));                 // part 0 has read them: the rows may be reused
        }
        mbar_init(bar(DQ_ACCFULL), 1);
        fence_mbar_init();
    }
    if (warp == 1) tmem_alloc(smem_u32(const_cast<uint32_t *>(tmem_slot)), kTmemCols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    const bool dead = *abort_flag != 0;

    if (dead) {
        // nothing: fall through to the teardown
    } else if (warp == 0) {
        if (lane == 0) {
            tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmdO); tma_prefetch_desc(&tmK);
            tma_prefetch_desc(&tmU); tma_prefetch_desc(&tmV);
            mbar_arrive_expect_tx(bar(DQ_QFULL), 2 * L::kQBytes);
            for (int c = 0; c < L::kChunks; ++c) {
                tma_load_4d(sQ + c * kTile, &tmQ, bar(DQ_QFULL), c * 64, t0, h, b);
                tma_load_4d(sdO + c * kTile, &tmdO, bar(DQ_QFULL), c * 64, t0, h, b);
            }
            int sk = 0, sv = 0;
            uint32_t phk = 1, phv = 1;
            for (int j = 0; j < nblk; ++j) {
                const int row = e0 * args.De + j * kBI;
                // Q and dO are in tensor memory: their tiles join the ring
                if (j == L::kKUStages - 2 && !mbar_wait(bar(DQ_QT), 0, ctl, W + 14)) break;
                if (!mbar_wait(bar(DQ_KUEMPTY + sk), phk, ctl, W + 1)) break;
                const uint32_t fk = bar(DQ_KUFULL + sk);
                mbar_arrive_expect_tx(fk, L::kKUStage);
#pragma unroll
                for (int c = 0; c < L::kChunks; ++c) {
                    const uint32_t d = sKU + sk * L::kKUStage + c * 2 * kWChunk;
                    tma_load_3d(d, &tmK, fk, c * 64, row, hk);
                    tma_load_3d(d + kWChunk, &tmU, fk, c * 64, row, hk);
                }
                if (!mbar_wait(bar(DQ_VEMPTY + sv), phv, ctl, W + 2)) break;
                const uint32_t fv = bar(DQ_VFULL + sv);
                mbar_arrive_expect_tx(fv, L::kVStage);
#pragma unroll
                for (int c = 0; c < L::kChunks; ++c)
                    tma_load_3d(sV + sv * L::kVStage + c * kWChunk, &tmV, fv, c * 64, row, hk);
                if (++sk == L::kKUStages) { sk = 0; phk ^= 1; }
                if (++sv == L::kVStages) { sv = 0; phv ^= 1; }
            }
        }
    } else if (warp == 1) {
        // Three MMA chains, three issuing threads (warps 1, 2, 3), so that none waits on another's barriers and the
        // tensor pipe, which accepts MMAs only a few ahead of execution, is fed by whichever is ready.  Every chain
        // reads its A operand from tensor memory: an MMA with both operands in shared memory takes the SM's whole
        // shared-memory bandwidth (8 KB per 64 clk), which the weight tiles arriving by TMA need as well.
        // Issuer 1: S = Q [K;U]^T.
        if (lane == 0) {
            constexpr uint32_t idS = umma_idesc(128, 2 * kBI, false, false);
            const uint64_t dKU0 = desc_kmajor(sKU);
            constexpr uint64_t kKUStep = L::kKUStage >> 4;
            bool ok = mbar_wait(bar(DQ_QT), 0, ctl, W + 3);
            int sk = 0;
            uint32_t phk = 0;
            for (int j = 0; ok && j < nblk; ++j) {
                if (!mbar_wait(bar(DQ_KUFULL + sk), phk, ctl, W + 4)) break;
                if (j >= 1 && !mbar_wait(bar(DQ_SEMPTY), (j - 1) & 1, ctl, W + 5)) break;
                tc_fence_after();
                const uint64_t dku = dKU0 + sk * kKUStep;
#pragma unroll
                for (int k = 0; k < DH / 16; ++k) {
                    const int c = k >> 2, kk = k & 3;
                    umma_ts(tmem + kColS, tmem + kColQ + k * 8, dku + ((c * 2 * kWChunk + kk * 32) >> 4), idS, k > 0 ? 1u : 0u);
                }
                umma_commit(bar(DQ_SFULL));
                if (++sk == L::kKUStages) { sk = 0; phk ^= 1; }
            }
        }
    } else if (warp == 2) {
        // Issuer 2: dA = dO V^T.
        if (lane == 0) {
            constexpr uint32_t idA = umma_idesc(128, kBI, false, false);
            const uint64_t dV0 = desc_kmajor(sV);
            constexpr uint64_t kVStep = L::kVStage >> 4;
            bool ok = mbar_wait(bar(DQ_QT), 0, ctl, W + 3);
            int sv = 0;
            uint32_t phv = 0;
            for (int j = 0; ok && j < nblk; ++j) {
                if (!mbar_wait(bar(DQ_VFULL + sv), phv, ctl, W + 4)) break;
                if (j >= 1 && !mbar_wait(bar(DQ_SEMPTY), (j - 1) & 1, ctl, W + 5)) break;
                tc_fence_after();
                const uint64_t dv = dV0 + sv * kVStep;
#pragma unroll
                for (int k = 0; k < DH / 16; ++k) {
                    const int c = k >> 2, kk = k & 3;
                    umma_ts(tmem + kColdA, tmem + kColdO + k * 8, dv + ((c * kWChunk + kk * 32) >> 4), idA, k > 0 ? 1u : 0u);
                }
                umma_commit(bar(DQ_VEMPTY + sv));
                umma_commit(bar(DQ_SFULL));
                if (++sv == L::kVStages) { sv = 0; phv ^= 1; }
            }
        }
    } else if (warp == 3) {
        // Issuer 3: dQ += [dM|dN] [K;U], with [dM|dN] read from tensor memory.
        if (lane == 0) {
            constexpr uint32_t idQ = umma_idesc(128, DH, false, true);
            const uint64_t dKUmn0 = desc_mnmajor(sKU, 2 * kWChunk);
            constexpr uint64_t kKUStep = L::kKUStage >> 4;
            int sk = 0;
            bool ok = true;
            for (int j = 0; j < nblk; ++j) {
                if (!mbar_wait(bar(DQ_PFULL), j & 1, ctl, W + 6)) { ok = false; break; }
                tc_fence_after();
                const uint64_t dku = dKUmn0 + sk * kKUStep;
                // [dM|dN] as packed bf16 pairs in 64 columns.  The thread that handled block columns [c, c + kCols) wrote
                // its dM to columns [c, c + kCols/2) and its dN to [c + kCols/2, c + kCols).  K step k (16 values = 8
                // columns; steps 0-3 pair with the K rows of the stage, 4-7 with the U rows) covers block columns
                // [16 (k%4), 16 (k%4) + 16).
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const int bc = 16 * (k & 3);
                    const int col = (bc / kCols) * kCols + (bc % kCols) / 2 + (k >> 2) * (kCols / 2);
                    umma_ts(tmem + kColAcc, tmem + kColP + col, dku + k * 128, idQ, (j > 0 || k > 0) ? 1u : 0u);
                }
                umma_commit(bar(DQ_KUEMPTY + sk));
                umma_commit(bar(DQ_PEMPTY));
                if (++sk == L::kKUStages) sk = 0;
            }
            if (ok) umma_commit(bar(DQ_ACCFULL));
        }
    } else if (warp >= 4) {
        const int quarter = warp & 3, part = (warp - 4) >> 2;  // part: which kCols of the block's 64 columns
        const int row = quarter * 32 + lane, t = t0 + row;
        const bool in_range = t < args.S;
        const float *rrow = args.R + (long long)b * args.r_sb + (long long)h * args.r_sh + (long long)t * args.r_ss + e0;
        float *drrow = args.dR + (long long)b * args.dr_sb + (long long)h * args.dr_sh + (long long)t * args.dr_ss + e0;
        const uint32_t lane_base = tmem + ((uint32_t)(quarter * 32) << 16);
        bool ok = true;
        // Q and dO: shared -> tensor memory, once (thread = token row; column part p copies columns [64p, 64p + 64)
        // of d_h of both tiles).
        if (!mbar_wait(bar(DQ_QFULL), 0, ctl, W + 12)) ok = false;
        if (ok && part * 64 < DH) {
#pragma unroll
            for (int which = 0; which < 2; ++which) {
                uint32_t v32[32];
                const uint8_t *src = gbase + (which ? L::kOffdO : L::kOffQ) + part * kTile;
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const uint4 v = *reinterpret_cast<const uint4 *>(src + sw128_offset(row, c));
                    v32[4 * c] = v.x; v32[4 * c + 1] = v.y; v32[4 * c + 2] = v.z; v32[4 * c + 3] = v.w;
                }
                tmem_st32(lane_base + (which ? kColdO : kColQ) + part * 32, v32);
            }
            tmem_st_wait();
        }
        tc_fence_before();
        warp_arrive(bar(DQ_QT));
        float r_cur = 0.f, r_next = in_range ? __ldg(rrow) : 0.f;
        f32x2 dr2 = f2_pack(0.f, 0.f);  // running dR_e of this thread's columns (two interleaved partial sums)
        const DqConst kc = dq_const(args.s0);
        int in_e = 0, e = 0;  // block index inside the current sub-network; current sub-network
        for (int j = 0; ok && j < nblk; ++j) {
            if (in_e == 0) {
                r_cur = r_next;
                r_next = (in_range && e + 1 < ne) ? __ldg(rrow + e + 1) : 0.f;
                dr2 = f2_pack(0.f, 0.f);
            }
            if (!mbar_wait(bar(DQ_SFULL), j & 1, ctl, W + 7)) { ok = false; break; }
            tc_fence_after();
            const uint32_t tS = lane_base + kColS + part * kCols, tA = lane_base + kColdA + part * kCols;
            uint32_t pm[kCols / 2], pn[kCols / 2];  // packed bf16 pairs of dM, dN for this thread's columns
            const f32x2 r2 = f2_pack(args.c * r_cur, args.c * r_cur);
            // the whole part at once, so that S and dA are free for the next block before any arithmetic
            uint32_t m[kCols], n[kCols], da[kCols];
            tmem_ld32x3_sync(tS, tS + kBI, tA, m, n, da);
            tc_fence_before();
            warp_arrive(bar(DQ_SEMPTY));
#pragma unroll
            for (int i = 0; i < kCols / 2; ++i) {
                const DqPair x = dq_pair(f2_pack_bits(m[2 * i], m[2 * i + 1]), f2_pack_bits(n[2 * i], n[2 * i + 1]),
                                         f2_pack_bits(da[2 * i], da[2 * i + 1]), r2, kc);
                dr2 = f2_fma(x.da, x.sn, dr2);
                pm[i] = f2_to_bf16x2(x.dm);
                pn[i] = f2_to_bf16x2(x.dn);
            }
            // the dQ update of the previous block has read the [dM|dN] buffer
            if (j >= 1 && !mbar_wait(bar(DQ_PEMPTY), (j - 1) & 1, ctl, W + 8)) { ok = false; break; }
            tc_fence_after();
            const uint32_t tP = lane_base + kColP + part * kCols;
            tmem_st16(tP, pm);
            tmem_st16(tP + kCols / 2, pn);
            tmem_st_wait();
            tc_fence_before();
            warp_arrive(bar(DQ_PFULL));
            if (++in_e == bpe) {  // sub-network finished: add the column parts of dR_e, in part order
                const int xb = e & 1;
                float dr_lo, dr_hi;
                f2_unpack(dr2, dr_lo, dr_hi);
                const float dr_acc = (dr_lo + dr_hi) * args.c;
                volatile float *xrow = drx + xb * 128 + row;
                if (part != 0) {
                    // the exchange rows of sub-network e were last used by e - 2: wait until those values have been read
                    if (e >= 2 && !mbar_wait(bar(DQ_DRFREE + xb), ((e >> 1) - 1) & 1, ctl, W + 11)) { ok = false; break; }
                    *xrow = dr_acc;
                    warp_arrive(bar(DQ_DRFULL + xb));
                } else {
                    if (!mbar_wait(bar(DQ_DRFULL + xb), (e >> 1) & 1, ctl, W + 9)) { ok = false; break; }
                    const float sum = dr_acc + *xrow;
                    warp_arrive(bar(DQ_DRFREE + xb));
                    if (in_range) drrow[e] = sum;
                }
                in_e = 0;
                ++e;
            }
        }
        if (ok) ok = mbar_wait(bar(DQ_ACCFULL), 0, ctl, W + 10);
        if (ok) {
            tc_fence_after();
            constexpr int kColsPerHalf = DH / 2;
            const int c0 = part * kColsPerHalf;
            float *pdst = args.part + ((((long long)isplit * args.B + b) * args.H + h) * args.S + t) * DH + c0;
#pragma unroll
            for (int g = 0; g < kColsPerHalf / 16; ++g) {
                uint32_t o[16];
                tmem_ld16_sync(lane_base + kColAcc + c0 + g * 16, o);
                if (args.nsplit > 1) {
                    if (in_range) {
#pragma unroll
                        for (int v = 0; v < 4; ++v)
                            *reinterpret_cast<float4 *>(pdst + g * 16 + v * 4) =
                                make_float4(__uint_as_float(o[4 * v]), __uint_as_float(o[4 * v + 1]),
                                            __uint_as_float(o[4 * v + 2]), __uint_as_float(o[4 * v + 3]));
                    }
                    continue;
                }
#pragma unroll
                for (int v = 0; v < 2; ++v) {
                    const int col = c0 + g * 16 + v * 8;
                    const uint32_t dst = sQ + (col >> 6) * kTile + sw128_offset(row, (col & 63) >> 3);
                    st_shared_v4(dst, pack_bf16(__uint_as_float(o[8 * v + 0]), __uint_as_float(o[8 * v + 1])),
                                 pack_bf16(__uint_as_float(o[8 * v + 2]), __uint_as_float(o[8 * v + 3])),
                                 pack_bf16(__uint_as_float(o[8 * v + 4]), __uint_as_float(o[8 * v + 5])),
                                 pack_bf16(__uint_as_float(o[8 * v + 6]), __uint_as_float(o[8 * v + 7])));
                }
            }
            tc_fence_before();
            fence_async_smem();
        }
        named_bar_sync(1, kActThreads);
        if (ok && warp == 4 && lane == 0 && !*abort_flag && args.nsplit == 1) {
            for (int c = 0; c < L::kChunks; ++c) tma_store_4d(&tmdQ, sQ + c * kTile, c * 64, t0, h, b);
            tma_store_commit();
            tma_store_wait_all();
        }
    }

    __syncwarp();
    // Launched so that it may start under the tail of the dK/dU/dV kernel, whose results it does not read.  Its own end must
    // still come after that kernel's, for whatever follows on the stream: one CTA waits.
    if (blockIdx.x == gridDim.x - 1 && blockIdx.y == gridDim.y - 1 && blockIdx.z == gridDim.z - 1) griddep_wait();
    if (*abort_flag) {
        const long long t_end = clock64() + (1LL << 19);
        while (clock64() < t_end) __nanosleep(256);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, kTmemCols);
    }
}

// =============================================================================================
//                                    dK / dU / dV kernel
// =============================================================================================
// A CTA owns 64 weight rows.  The rows of K and U lie in the 128 lanes of one operand, sixteen of K, sixteen of U and so on, so that
//     S^T = [K;U] Q^T        (128 lanes x 128 tokens: M in lanes 0-15 of each 32, N of the same weight rows in lanes 16-31)
//     dA^T = V dO^T          (64 rows x 128 tokens: an M = 64 product fills sixteen lanes of each 32, here 0-15)
// put M, N and dA of a weight row under one warp, which reads sixteen lanes at a time, and what it writes back, [dM;dN] as bf16, is
// the A operand of
//     [dK;dU] += [dM;dN] Q   (128 x d_h).
// Only A^T goes through shared memory, for dV += A^T dO, an M = 64 product too (lanes 16-31 of dA's columns).  [K;U] are copied to tensor
// memory once.
// Tensor memory (512 columns): [dK;dU] 128, [K;U] 64, S 128, dA and dV 128, [dM;dN] 64.  No product writes where another one reads: of two
// MMAs with different accumulators or shapes, the order in which a thread issues them promises nothing.  As dV^T (M = 128, N = 64) the
// dV update is half as long on the tensor pipe, but then [dM;dN] must lie over dA, and dA of the next tile must wait for the update that
// reads them: 1156 us where this form takes 1017 (32768 tokens of the 370M layer's operator, in a loop at the power limit; ten passes
// 1017 and 891).  [K;U] as an operand in shared memory instead, with dV^T: 1029 to 1039.  dA in two halves of 64 tokens, in lanes 0-15 and
// 16-31 of 64 columns, with dV^T: 1136, since an M = 64 product takes as long at N = 64 as at 128.
// Bound: the tensor pipe (2130 of 2440 clk a tile, 87 %) and with it shared memory, of whose cycles operand reads take 53 % (160 KB a tile),
// the threads' loads and stores 23 % and the fills about 21 % (64 KB), all by counters; and power.
template <int DH>
struct DwSmem {
    static constexpr int kChunks = (DH + 63) / 64;
    static constexpr uint32_t kTok = kChunks * kTile;      // Q or dO of a tile: 128 rows
    static constexpr uint32_t kVBytes = kChunks * kWChunk;
    // [K;U] are needed in shared memory only until they are copied to tensor memory: they arrive in the last stage of the dO ring.
    static constexpr int kQStages = 3, kGStages = 3, kRSlots = 2;
    static constexpr uint32_t kOffQ = 0;
    static constexpr uint32_t kOffG = kOffQ + kQStages * kTok;
    static constexpr uint32_t kOffKU = kOffG + (kGStages - 1) * kTok;
    static constexpr uint32_t kOffV = kOffG + kGStages * kTok;
    static constexpr uint32_t kOffA = kOffV + kVBytes;            // A^T of a tile: 64 weight rows x 128 tokens
    static constexpr uint32_t kOffR = kOffA + 2 * kWChunk;
    static constexpr uint32_t kOffCtl = kOffR + kRSlots * kBT * 4;
    static constexpr uint32_t kTotal = kOffCtl + 256 + 1024;
};

// Barriers.  Each is waited on by one fixed thread (or all element-wise warps) in every phase, so a one-bit parity is enough.
//   KUT: [K;U] copied to tensor memory;  SFULL / SEMPTY, DAFULL / DAEMPTY: S, dA computed / in registers;  AFULL / AEMPTY: A staged /
//   its dV update done;  PFULL / PEMPTY: [dM;dN] written / its update done;  RFULL, REMPTY: routing weights.
enum { DW_WFULL = 0, DW_KUT = 1, DW_SFULL = 2, DW_SEMPTY = 3, DW_DAFULL = 4, DW_AFULL = 5, DW_AEMPTY = 6, DW_PFULL = 7, DW_ACCFULL = 8,
       DW_RFULL = 9, DW_REMPTY = 11, DW_DAEMPTY = 13, DW_PEMPTY = 14, DW_QFULL = 15, DW_QEMPTY = 18, DW_GFULL = 21, DW_GEMPTY = 24,
       DW_BARS = 27 };
static_assert(DW_BARS * 8 + 8 <= 256, "control area");

struct DwArgs {
    const float *R;
    long long r_sb, r_sh, r_ss;
    // fp32 partial sums of the split blocks: [nsplit][3][ws_plane], a plane being the elements of [Hkuv][I][DH] from ws_first on
    float *ws;
    long long ws_plane, ws_first;
    // One part per block: its sums are the results and are written as bf16 at once (dK, dU, dV: head and row strides)
    __nv_bfloat16 *out[3];
    long long o_head[3], o_row[3];
    int S, E, De, G, B, Hkuv;
    int tiles_per_seq, tiles_total, tiles_per_split;
    // CTA -> (weight block, token-tile range).  Blocks [0, n_mixed) are split unevenly into a long part (launched first)
    // and a short part of `small_tiles` tiles (launched last); the others into `nsplit` equal parts, part by part.
    // Blocks [0, n_direct) are whole and written as bf16 results.
    int nblk_j, n_blocks, nsplit, n_direct, n_mixed, small_tiles;
    float s0, c;  // head_scaling; head_scaling * up_scaling * final_scaling / 2
    WaitArgs wait;
};

// This CTA's weight block and token tiles.
__device__ __forceinline__ void dw_range(const DwArgs &args, int &blk, int &split, int &tile_begin, int &tile_end) {
    // in launch order: whole blocks (n_direct), long parts (n_mixed), equal parts part by part, short parts (n_mixed)
    const int cta = (int)blockIdx.x - args.n_direct, first = args.n_direct + args.n_mixed, n_even = args.n_blocks - first;
    if (cta < 0) {
        blk = blockIdx.x; split = 0; tile_begin = 0; tile_end = args.tiles_total;
    } else if (cta < args.n_mixed) {                        // long part of an unevenly split block
        blk = args.n_direct + cta; split = 0; tile_begin = 0; tile_end = args.tiles_total - args.small_tiles;
    } else if (cta < args.n_mixed + n_even * args.nsplit) { // equal parts, part by part
        const int r = cta - args.n_mixed;
        split = r / n_even;
        blk = first + (r - split * n_even);
        tile_begin = split * args.tiles_per_split;
        tile_end = min(tile_begin + args.tiles_per_split, args.tiles_total);
    } else {                                                // short part of an unevenly split block
        blk = args.n_direct + cta - (args.n_mixed + n_even * args.nsplit); split = 1;
        tile_begin = args.tiles_total - args.small_tiles; tile_end = args.tiles_total;
    }
}
// 16 columns of one row of an accumulator: fp32 to the workspace, or the bf16 result.
__device__ __forceinline__ void dw_store16(bool direct, float *dst, __nv_bfloat16 *o16, const uint32_t (&o)[16]) {
    if (direct) {
#pragma unroll
        for (int v = 0; v < 4; ++v)
            *reinterpret_cast<uint2 *>(o16 + v * 4) = make_uint2(pack_bf16(__uint_as_float(o[4 * v]), __uint_as_float(o[4 * v + 1])),
                                                                 pack_bf16(__uint_as_float(o[4 * v + 2]), __uint_as_float(o[4 * v + 3])));
    } else {
#pragma unroll
        for (int v = 0; v < 4; ++v)
            *reinterpret_cast<float4 *>(dst + v * 4) = make_float4(__uint_as_float(o[4 * v]), __uint_as_float(o[4 * v + 1]),
                                                                   __uint_as_float(o[4 * v + 2]), __uint_as_float(o[4 * v + 3]));
    }
}

template <int DH>
__global__ void __launch_bounds__(kThreads, 1)
bwd_dw_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmdO,
              const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmU,
              const __grid_constant__ CUtensorMap tmV, const DwArgs args) {
    using L = DwSmem<DH>;
    static_assert(DH == 128, "the narrower head dimensions have a kernel of their own");
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t *gbase = smem_raw + (base - raw);
    const uint32_t sQ = base + L::kOffQ, sG = base + L::kOffG, sKU = base + L::kOffKU, sV = base + L::kOffV, sA = base + L::kOffA,
                   sBar = base + L::kOffCtl;
    float *rbuf = reinterpret_cast<float *>(gbase + L::kOffR);   // [kRSlots][kBT]
    volatile uint32_t *tmem_slot = reinterpret_cast<volatile uint32_t *>(gbase + L::kOffCtl + DW_BARS * 8);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(gbase + L::kOffCtl + DW_BARS * 8 + 4);
    auto bar = [&](int i) { return sBar + 8u * i; };

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int blk, split, tile_begin, tile_end;
    dw_range(args, blk, split, tile_begin, tile_end);
    const int hk = blk / args.nblk_j, jblk = blk - hk * args.nblk_j;
    const int e = (jblk * kBI) / args.De;
    const int ntiles = tile_end - tile_begin;  // >= 1 by construction of the plan
    const WaitCtl ctl{abort_flag, args.wait};
    constexpr int W = kKernelBwdDw * 100;
    // Columns.  dA and dV share theirs, in lanes 0-15 and 16-31 of each 32.
    constexpr uint32_t kColKU = 0, kColW = kColKU + DH, kColS = kColW + DH / 2, kColdA = kColS + kBT, kColV = kColdA,
                       kColP = kColdA + kBT, kUpper = 16u << 16;
    static_assert(DH <= kBT, "dV fits under dA");
    static_assert(kColP + kBT / 2 <= kTmemCols, "tensor memory");

    auto tile_coords = [&](int i, int &ts, int &hh, int &bb) {  // token tile i of this CTA -> (seq tile, head, batch)
        const int ti = tile_begin + i;
        ts = ti % args.tiles_per_seq;
        const int rest = ti / args.tiles_per_seq;
        hh = hk * args.G + rest % args.G;
        bb = rest / args.G;
    };

    if (threadIdx.x == 0) {
        *abort_flag = launch_aborted(args.wait);  // a CTA of this launch gave up: drain fast
        for (int i : {DW_WFULL, DW_SFULL, DW_DAFULL, DW_AEMPTY, DW_PEMPTY, DW_ACCFULL}) mbar_init(bar(i), 1);
        for (int i : {DW_KUT, DW_SEMPTY, DW_DAEMPTY, DW_AFULL, DW_PFULL}) mbar_init(bar(i), arrivals_of(kActThreads));
        for (int s = 0; s < L::kRSlots; ++s) {
            mbar_init(bar(DW_RFULL + s), arrivals_of(32));
            mbar_init(bar(DW_REMPTY + s), arrivals_of(kActThreads));
        }
        for (int s = 0; s < L::kQStages; ++s) {
            mbar_init(bar(DW_QFULL + s), 1);
            mbar_init(bar(DW_QEMPTY + s), 1);
        }
        for (int s = 0; s < L::kGStages; ++s) {
            mbar_init(bar(DW_GFULL + s), 1);
            mbar_init(bar(DW_GEMPTY + s), 2);   // the dA product and the dV update have read it
        }
        fence_mbar_init();
    }
    if (warp == 1) tmem_alloc(smem_u32(const_cast<uint32_t *>(tmem_slot)), kTmemCols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    const bool dead = *abort_flag != 0;
    griddep_launch_dependents();   // the dQ/dR kernel may take over SMs that this kernel's last CTAs leave idle

    if (dead) {
        // nothing: fall through to the teardown
    } else if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer
        if (lane == 0) {
            tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmdO); tma_prefetch_desc(&tmK);
            tma_prefetch_desc(&tmU); tma_prefetch_desc(&tmV);
            mbar_arrive_expect_tx(bar(DW_WFULL), L::kChunks * kTile + L::kVBytes);
            const int row = jblk * kBI;
            for (int c = 0; c < L::kChunks; ++c) {
                tma_load_3d(sKU + c * kTile, &tmK, bar(DW_WFULL), c * 64, row, hk);
                tma_load_3d(sKU + c * kTile + kWChunk, &tmU, bar(DW_WFULL), c * 64, row, hk);
                tma_load_3d(sV + c * kWChunk, &tmV, bar(DW_WFULL), c * 64, row, hk);
            }
            int sq = 0, sg = 0;
            uint32_t phq = 1, phg = 1;
            for (int i = 0; i < ntiles; ++i) {
                int ts, hh, bb;
                tile_coords(i, ts, hh, bb);
                if (!mbar_wait(bar(DW_QEMPTY + sq), phq, ctl, W + 1)) break;
                mbar_arrive_expect_tx(bar(DW_QFULL + sq), L::kTok);
#pragma unroll
                for (int c = 0; c < L::kChunks; ++c)
                    tma_load_4d(sQ + sq * L::kTok + c * kTile, &tmQ, bar(DW_QFULL + sq), c * 64, ts * kBT, hh, bb);
                if (i == L::kGStages - 1 && !mbar_wait(bar(DW_KUT), 0, ctl, W + 17)) break;   // [K;U] are in tensor memory
                if (!mbar_wait(bar(DW_GEMPTY + sg), phg, ctl, W + 2)) break;
                mbar_arrive_expect_tx(bar(DW_GFULL + sg), L::kTok);
#pragma unroll
                for (int c = 0; c < L::kChunks; ++c)
                    tma_load_4d(sG + sg * L::kTok + c * kTile, &tmdO, bar(DW_GFULL + sg), c * 64, ts * kBT, hh, bb);
                if (++sq == L::kQStages) { sq = 0; phq ^= 1; }
                if (++sg == L::kGStages) { sg = 0; phg ^= 1; }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer 1: S^T of the next tile, dV += A^T dO of this one
        if (lane == 0) {
            constexpr uint32_t idS = umma_idesc(128, kBT, false, false);
            constexpr uint32_t idV = umma_idesc(64, DH, false, true);
            const uint64_t dQ0 = desc_kmajor(sQ), dG0 = desc_mnmajor(sG, kTile), dA0 = desc_kmajor(sA);
            constexpr uint64_t kTokStep = L::kTok >> 4;
            bool ok = mbar_wait(bar(DW_KUT), 0, ctl, W + 3);
            int sq = 0, sg = 0;
            uint32_t phq = 0, phg = 0;
            for (int i = -1; ok && i < ntiles; ++i) {
                const bool more = i + 1 < ntiles;
                if (more && !mbar_wait(bar(DW_QFULL + sq), phq, ctl, W + 4)) break;
                if (more && i >= 0 && !mbar_wait(bar(DW_SEMPTY), i & 1, ctl, W + 5)) break;
                if (more) {
                    tc_fence_after();
                    const uint64_t dq = dQ0 + sq * kTokStep;
#pragma unroll
                    for (int k = 0; k < DH / 16; ++k) {
                        const int c = k >> 2, kk = k & 3;
                        umma_ts(tmem + kColS, tmem + kColW + k * 8, dq + ((c * kTile + kk * 32) >> 4), idS, k > 0 ? 1u : 0u);
                    }
                    umma_commit(bar(DW_SFULL));
                    if (++sq == L::kQStages) { sq = 0; phq ^= 1; }
                }
                if (i < 0) continue;
                if (!mbar_wait(bar(DW_GFULL + sg), phg, ctl, W + 10)) break;   // (A^T does not imply that dO is there)
                if (!mbar_wait(bar(DW_AFULL), i & 1, ctl, W + 6)) break;
                tc_fence_after();
                const uint64_t dg = dG0 + sg * kTokStep;
#pragma unroll
                for (int k = 0; k < kBT / 16; ++k)
                    umma_ss(tmem + kUpper + kColV, dA0 + (((k >> 2) * kWChunk + (k & 3) * 32) >> 4), dg + k * 128, idV, (i > 0 || k > 0) ? 1u : 0u);
                umma_commit(bar(DW_GEMPTY + sg));
                umma_commit(bar(DW_AEMPTY));
                if (++sg == L::kGStages) { sg = 0; phg ^= 1; }
            }
        }
    } else if (warp == 2) {
        // ------------------------------------------------------------------ MMA issuer 2: dA^T of the next tile, [dK;dU] += [dM;dN] Q of this one
        if (lane == 0) {
            constexpr uint32_t idA = umma_idesc(64, kBT, false, false);
            constexpr uint32_t idKU = umma_idesc(128, DH, false, true);
            const uint64_t dV = desc_kmajor(sV), dG0 = desc_kmajor(sG), dQ0 = desc_mnmajor(sQ, kTile);
            constexpr uint64_t kTokStep = L::kTok >> 4;
            bool ok = mbar_wait(bar(DW_WFULL), 0, ctl, W + 3);
            int sq = 0, sg = 0;
            uint32_t phg = 0;
            for (int i = -1; ok && i < ntiles; ++i) {
                if (i + 1 < ntiles) {
                    if (!mbar_wait(bar(DW_GFULL + sg), phg, ctl, W + 4)) { ok = false; break; }
                    if (i >= 0 && !mbar_wait(bar(DW_DAEMPTY), i & 1, ctl, W + 18)) { ok = false; break; }
                    tc_fence_after();
                    const uint64_t dg = dG0 + sg * kTokStep;
#pragma unroll
                    for (int k = 0; k < DH / 16; ++k) {
                        const int c = k >> 2, kk = k & 3;
                        umma_ss(tmem + kColdA, dV + ((c * kWChunk + kk * 32) >> 4), dg + ((c * kTile + kk * 32) >> 4), idA, k > 0 ? 1u : 0u);
                    }
                    umma_commit(bar(DW_DAFULL));
                    umma_commit(bar(DW_GEMPTY + sg));
                    if (++sg == L::kGStages) { sg = 0; phg ^= 1; }
                }
                if (i < 0) continue;
                if (!mbar_wait(bar(DW_PFULL), i & 1, ctl, W + 6)) { ok = false; break; }
                tc_fence_after();
                const uint64_t dq = dQ0 + sq * kTokStep;
#pragma unroll
                for (int k = 0; k < kBT / 16; ++k)
                    umma_ts(tmem + kColKU, tmem + kColP + k * 8, dq + k * 128, idKU, (i > 0 || k > 0) ? 1u : 0u);
                umma_commit(bar(DW_QEMPTY + sq));
                umma_commit(bar(DW_PEMPTY));
                if (++sq == L::kQStages) sq = 0;
            }
            if (ok) umma_commit(bar(DW_ACCFULL));
        }
    } else if (warp == 3) {
        // ------------------------------------------------------------------ routing weights of each tile, times args.c
        for (int i = 0; i < ntiles; ++i) {
            int ts, hh, bb;
            tile_coords(i, ts, hh, bb);
            const float *src = args.R + (long long)bb * args.r_sb + (long long)hh * args.r_sh + e;
            float v[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int t = ts * kBT + k * 32 + lane;
                v[k] = t < args.S ? args.c * __ldg(src + (long long)t * args.r_ss) : 0.f;
            }
            const int slot = i % L::kRSlots;
            if (!mbar_wait(bar(DW_REMPTY + slot), ((uint32_t)(i / L::kRSlots) & 1u) ^ 1u, ctl, W + 13)) break;
#pragma unroll
            for (int k = 0; k < 4; ++k) rbuf[slot * kBT + k * 32 + lane] = v[k];
            warp_arrive(bar(DW_RFULL + slot));
        }
    } else if (warp >= 4) {
        // ------------------------------------------------------------------ element-wise math
        // A warp has sixteen weight rows (M, dA in lanes 0-15 of its quarter, N in lanes 16-31) and 64 tokens; a thread rows lane / 4
        // and lane / 4 + 8 and of each eight tokens the two at 2 (lane % 4).  Pair 2x + rr: tokens 8x.., row lane / 4 + 8 rr.
        const int quarter = warp & 3, part = (warp - 4) >> 2;
        const uint32_t lane_base = tmem + ((uint32_t)(quarter * 32) << 16), lane_up = lane_base + kUpper;
        bool ok = mbar_wait(bar(DW_WFULL), 0, ctl, W + 14);
        if (ok) {   // [K;U]: shared -> tensor memory, once (thread = stacked row; column part p copies columns [64p, 64p + 64) of d_h)
            uint32_t v32[32];
            const int src_row = (lane >> 4) * kBI + quarter * 16 + (lane & 15);   // they arrive as 64 rows of K and 64 of U
            const uint8_t *src = gbase + L::kOffKU + part * kTile;
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const uint4 v = *reinterpret_cast<const uint4 *>(src + sw128_offset(src_row, c));
                v32[4 * c] = v.x; v32[4 * c + 1] = v.y; v32[4 * c + 2] = v.z; v32[4 * c + 3] = v.w;
            }
            tmem_st32(lane_base + kColW + part * 32, v32);
            tmem_st_wait();
        }
        tc_fence_before();
        warp_arrive(bar(DW_KUT));
        const DwConst kc = dw_const(args.s0);
        // stmatrix: lane l gives the row address of matrix l / 8: token group x + l / 16, row (l % 8) + 8 ((l / 8) % 2)
        const int arow = quarter * 16 + (lane & 15);
        const uint32_t a_row = sA + part * kWChunk + arow * 128, a_x = lane >> 4;
        const float *rsrc = rbuf + part * 64 + 2 * (lane & 3);
        for (int i = 0; ok && i < ntiles; ++i) {
            const int slot = i % L::kRSlots;
            const bool r_there = mbar_test(bar(DW_RFULL + slot), (uint32_t)(i / L::kRSlots) & 1u);
            if (!mbar_wait(bar(DW_SFULL), i & 1, ctl, W + 7)) { ok = false; break; }
            if (!r_there && !mbar_wait(bar(DW_RFULL + slot), (uint32_t)(i / L::kRSlots) & 1u, ctl, W + 15)) { ok = false; break; }
            tc_fence_after();
            // first what needs only S: A goes out, and its dV update runs, while dA is still being computed
            f32x2 fq[16], fw[16];
            uint32_t pa[16];
            bool a_free = i == 0;   // asked for ahead of the second half's arithmetic: a wait takes 75 cycles even where nothing is waited for
#pragma unroll
            for (int sub = 0; sub < 2; ++sub) {
                uint32_t m[16], n[16];
                tmem_ld_16x256b_x4x2_sync(lane_base + kColS + part * 64 + sub * 32, lane_up + kColS + part * 64 + sub * 32, m, n);
                if (sub == 1) {   // S is in registers: the buffer can take the next tile
                    tc_fence_before();
                    warp_arrive(bar(DW_SEMPTY));
                    if (i >= 1) a_free = mbar_test(bar(DW_AEMPTY), (i - 1) & 1);
                }
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    const float2 r = *reinterpret_cast<const float2 *>(rsrc + slot * kBT + sub * 32 + x * 8);
#pragma unroll
                    for (int rr = 0; rr < 2; ++rr) {
                        const int q = 2 * x + rr, o = sub * 8 + q;
                        const DwPair d = dw_pair(f2_pack_bits(m[2 * q], m[2 * q + 1]), f2_pack_bits(n[2 * q], n[2 * q + 1]), f2_pack(r.x, r.y), kc);
                        fq[o] = d.q;
                        fw[o] = d.w;
                        pa[o] = f2_to_bf16x2(d.a);
                    }
                }
            }
            warp_arrive(bar(DW_REMPTY + slot));
            if (!a_free && !mbar_wait(bar(DW_AEMPTY), (i - 1) & 1, ctl, W + 8)) { ok = false; break; }
#pragma unroll
            for (int x = 0; x < 8; x += 2)
                stmatrix_x4(a_row + (((x + a_x) ^ (arow & 7)) << 4), pa[2 * x], pa[2 * x + 1], pa[2 * x + 2], pa[2 * x + 3]);
            fence_async_smem();
            warp_arrive(bar(DW_AFULL));
            // then dM and dN
            uint32_t da[32], pm[16], pn[16];
            bool p_free = i == 0;
            if (!mbar_wait(bar(DW_DAFULL), i & 1, ctl, W + 11)) { ok = false; break; }
            tc_fence_after();
            tmem_ld_16x256b_x8_sync(lane_base + kColdA + part * 64, da);
            tc_fence_before();
            warp_arrive(bar(DW_DAEMPTY));
            if (i >= 1) p_free = mbar_test(bar(DW_PEMPTY), (i - 1) & 1);
#pragma unroll
            for (int q = 0; q < 16; ++q) {
                const f32x2 da2 = f2_pack_bits(da[2 * q], da[2 * q + 1]);
                pm[q] = f2_to_bf16x2(f2_mul(da2, fw[q]));
                pn[q] = f2_to_bf16x2(f2_mul(da2, fq[q]));
            }
            if (!p_free && !mbar_wait(bar(DW_PEMPTY), (i - 1) & 1, ctl, W + 19)) { ok = false; break; }
            tc_fence_after();
            tmem_st_16x128b_x8(lane_base + kColP + part * 32, pm);
            tmem_st_16x128b_x8(lane_up + kColP + part * 32, pn);
            tmem_st_wait();
            tc_fence_before();
            warp_arrive(bar(DW_PFULL));
        }
        if (ok) ok = mbar_wait(bar(DW_ACCFULL), 0, ctl, W + 9);
        if (ok && ntiles > 0) ok = mbar_wait(bar(DW_AEMPTY), (ntiles - 1) & 1, ctl, W + 16);
        if (ok) {
            tc_fence_after();
            // fp32 partial sums -> workspace[split][which][hk][row][DH], or bf16 results
            const bool direct = args.nsplit == 1 || blk < args.n_direct;
            const long long I = (long long)args.E * args.De;
            const long long plane = args.ws_plane;
            float *wsb = args.ws + (long long)split * 3 * plane + ((long long)hk * I + (long long)jblk * kBI) * DH - args.ws_first;
            auto out_row = [&](int which, int r) {
                return args.out[which] + hk * args.o_head[which] + ((long long)jblk * kBI + r) * args.o_row[which];
            };
            constexpr int kColsPerHalf = DH / 2;
            const int c0 = part * kColsPerHalf;
            {   // [dK;dU]: sixteen lanes of dK, sixteen of dU, ...
                const int which = lane >> 4, r = quarter * 16 + (lane & 15);
                float *dst = wsb + which * plane + (long long)r * DH + c0;
                __nv_bfloat16 *o16 = out_row(which, r) + c0;
#pragma unroll
                for (int g = 0; g < kColsPerHalf / 16; ++g) {
                    uint32_t o[16];
                    tmem_ld16_sync(lane_base + kColKU + c0 + g * 16, o);
                    dw_store16(direct, dst + g * 16, o16 + g * 16, o);
                }
            }
            {   // dV: lanes 16-31 of each 32
                const int r = quarter * 16 + (lane & 15);
                float *dst = wsb + 2 * plane + (long long)r * DH + c0;
                __nv_bfloat16 *o16 = out_row(2, r) + c0;
#pragma unroll
                for (int g = 0; g < kColsPerHalf / 16; ++g) {
                    uint32_t o[16];
                    tmem_ld16_sync(lane_base + kColV + c0 + g * 16, o);
                    if (lane >= 16) dw_store16(direct, dst + g * 16, o16 + g * 16, o);
                }
            }
            tc_fence_before();
        }
    }

    __syncwarp();
    if (*abort_flag) {
        const long long t_end = clock64() + (1LL << 19);
        while (clock64() < t_end) __nanosleep(256);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, kTmemCols);
    }
}

// =============================================================================================
//                        dK / dU / dV kernel, transposed (d_h = 64 and 96)
// =============================================================================================
// A CTA owns 128 weight rows, and the three recomputed products
//     M^T = K Q^T,  N^T = U Q^T,  dA^T = V dO^T      (128 weight rows x 64 tokens each, lane = weight row)
// come out such that dM^T, dN^T and A^T, written back to tensor memory as bf16, are the A operands of
//     dK += dM^T Q,  dU += dN^T Q,  dV += A^T dO     (128 x d_h each).
// Nothing is staged in shared memory, and a token tile serves twice as many weight rows as above.  Against the lane = token form, which
// moved twice the bytes: 16 x 16 x 192 at d_h = 64, 16384 tokens, 0.795 -> 0.697 ms; 128M layer (d_h = 96), 16384 tokens, 0.377 -> 0.342 ms.
// Against the form above, when its dV was accumulated transposed: d_h = 64 754 against 945 us (its element-wise step is longer: loads of
// sixteen lanes, A through shared memory, and it paces the kernel here), d_h = 96 373.7 against 371.7, at the power limit.
// Tensor memory: three accumulators of d_h columns; d_h = 64: two buffers of [M^T | N^T] (128 columns), whose columns A^T, dM^T and
// dN^T later take, and dA^T; d_h = 96: one [M^T | N^T], given back as soon as it is in registers, dA^T, over which dM^T and dN^T
// are written, and 32 columns for A^T.  (d_h = 128 would need 576 columns.)
// The routing weight now goes with the column: warp 2 fetches the 64 tokens' weights of a tile (of the two sub-networks that
// 128 rows can touch) into a small ring in shared memory, from where the element-wise warps read them as pairs.
constexpr int kTT = 64;    // tokens per tile
constexpr int kTI = 128;   // weight rows per CTA

template <int DH>
struct DwtSmem {
    static constexpr int kChunks = (DH + 63) / 64;
    static constexpr uint32_t kWMat = kChunks * 2 * kWChunk;      // one of K, U, V: 128 rows
    static constexpr uint32_t kTok = kChunks * kWChunk;           // Q or dO of a tile: 64 rows
    // d_h = 96: a fourth token stage fits once the routing-weight ring is halved (231,936 of 232,448 bytes).  Against 3 stages and
    // 4 slots, 128M layer: 377.1 -> 374.9 us, and 730.9 -> 728.0 us with the chip at its power limit.
    static constexpr int kStages = DH == 64 ? 8 : 4;
    static constexpr int kRSlots = DH == 64 ? 4 : 2;
    static constexpr uint32_t kOffW = 0;
    static constexpr uint32_t kOffTok = 3 * kWMat;
    static constexpr uint32_t kOffR = kOffTok + kStages * 2 * kTok;
    static constexpr uint32_t kOffCtl = kOffR + kRSlots * 2 * kTT * 4;
    static constexpr uint32_t kTotal = kOffCtl + 512 + 1024;
};

// Barriers: as in the kernel above, with S = [M^T | N^T] (buffer b = tile % kSB).  SEMPTY[b], DAEMPTY: the buffer may be computed
// into again (d_h = 64: the updates that read [dM|dN] and A from S are done / dA is in registers; d_h = 96: S is in registers /
// the updates that read dM and dN over dA are done).  AEMPTY (d_h = 96): the dV update has read A.  RFULL, REMPTY: routing weights.
constexpr int kMaxTokT = 8;
enum { DT_WFULL = 0, DT_SFULL = 1, DT_SEMPTY = 3, DT_AFULL = 5, DT_PFULL = 7, DT_AEMPTY = 9, DT_DAFULL = 10, DT_DAEMPTY = 11, DT_ACCFULL = 12,
       DT_RFULL = 13, DT_REMPTY = 17, DT_QFULL = 21, DT_GFULL = DT_QFULL + kMaxTokT, DT_QEMPTY = DT_GFULL + kMaxTokT,
       DT_GEMPTY = DT_QEMPTY + kMaxTokT, DT_BARS = DT_GEMPTY + kMaxTokT };
static_assert(DT_BARS * 8 + 8 <= 512, "control area");

template <int DH>
__global__ void __launch_bounds__(kThreads, 1)
bwd_dwt_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmdO,
               const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmU,
               const __grid_constant__ CUtensorMap tmV, const DwArgs args) {
    using L = DwtSmem<DH>;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t *gbase = smem_raw + (base - raw);
    const uint32_t sW = base + L::kOffW, sTok = base + L::kOffTok, sBar = base + L::kOffCtl;
    float *rbuf = reinterpret_cast<float *>(gbase + L::kOffR);   // [kRSlots][2][kTT]
    volatile uint32_t *tmem_slot = reinterpret_cast<volatile uint32_t *>(gbase + L::kOffCtl + DT_BARS * 8);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(gbase + L::kOffCtl + DT_BARS * 8 + 4);
    auto bar = [&](int i) { return sBar + 8u * i; };

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int blk, split, tile_begin, tile_end;
    dw_range(args, blk, split, tile_begin, tile_end);
    const int hk = blk / args.nblk_j, row0 = (blk - hk * args.nblk_j) * kTI;
    const int I = args.E * args.De;
    const int ntiles = tile_end - tile_begin;  // >= 1 by construction of the plan
    const WaitCtl ctl{abort_flag, args.wait};
    constexpr int W = kKernelBwdDw * 100 + 50;
    constexpr int kSB = DH == 64 ? 2 : 1;
    constexpr uint32_t kColAcc = 0, kColS = 3 * DH, kColdA = kColS + kSB * 128, kColA = kColdA + 64;   // kColA: d_h = 96
    static_assert(kColdA + 64 + (kSB == 1 ? 32 : 0) <= kTmemCols, "tensor memory");

    auto tile_coords = [&](int i, int &ts, int &hh, int &bb) {  // token tile i of this CTA -> (seq tile, head, batch)
        const int ti = tile_begin + i;
        ts = ti % args.tiles_per_seq;
        const int rest = ti / args.tiles_per_seq;
        hh = hk * args.G + rest % args.G;
        bb = rest / args.G;
    };

    if (threadIdx.x == 0) {
        *abort_flag = launch_aborted(args.wait);  // a CTA of this launch gave up: drain fast
        for (int i : {DT_WFULL, DT_AEMPTY, DT_DAFULL, DT_ACCFULL}) mbar_init(bar(i), 1);
        mbar_init(bar(DT_DAEMPTY), kSB == 2 ? arrivals_of(kActThreads) : 1);
        for (int b = 0; b < 2; ++b) {
            mbar_init(bar(DT_SFULL + b), 1);
            mbar_init(bar(DT_SEMPTY + b), kSB == 2 ? 1 : arrivals_of(kActThreads));
            mbar_init(bar(DT_AFULL + b), arrivals_of(kActThreads));
            mbar_init(bar(DT_PFULL + b), arrivals_of(kActThreads));
        }
        for (int s = 0; s < L::kRSlots; ++s) {
            mbar_init(bar(DT_RFULL + s), arrivals_of(32));
            mbar_init(bar(DT_REMPTY + s), arrivals_of(kActThreads));
        }
        for (int s = 0; s < L::kStages; ++s) {
            mbar_init(bar(DT_QFULL + s), 1);
            mbar_init(bar(DT_GFULL + s), 1);
            mbar_init(bar(DT_QEMPTY + s), 1);
            mbar_init(bar(DT_GEMPTY + s), 2);   // the dA product and the dV update have read it
        }
        fence_mbar_init();
    }
    if (warp == 1) tmem_alloc(smem_u32(const_cast<uint32_t *>(tmem_slot)), kTmemCols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    const bool dead = *abort_flag != 0;
    griddep_launch_dependents();   // the dQ/dR kernel may take over SMs that this kernel's last CTAs leave idle

    if (dead) {
        // nothing: fall through to the teardown
    } else if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer
        if (lane == 0) {
            tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmdO); tma_prefetch_desc(&tmK);
            tma_prefetch_desc(&tmU); tma_prefetch_desc(&tmV);
            mbar_arrive_expect_tx(bar(DT_WFULL), 3 * L::kWMat);
            for (int c = 0; c < L::kChunks; ++c)
                for (int hf = 0; hf < 2; ++hf) {   // rows beyond the last (an odd number of 64-row blocks) read as zero
                    const uint32_t d = sW + c * 2 * kWChunk + hf * kWChunk;
                    tma_load_3d(d, &tmK, bar(DT_WFULL), c * 64, row0 + hf * 64, hk);
                    tma_load_3d(d + L::kWMat, &tmU, bar(DT_WFULL), c * 64, row0 + hf * 64, hk);
                    tma_load_3d(d + 2 * L::kWMat, &tmV, bar(DT_WFULL), c * 64, row0 + hf * 64, hk);
                }
            int st = 0;
            uint32_t ph = 1;
            for (int i = 0; i < ntiles; ++i) {
                int ts, hh, bb;
                tile_coords(i, ts, hh, bb);
                const uint32_t d = sTok + st * 2 * L::kTok;
                if (!mbar_wait(bar(DT_QEMPTY + st), ph, ctl, W + 1)) break;
                mbar_arrive_expect_tx(bar(DT_QFULL + st), L::kTok);
#pragma unroll
                for (int c = 0; c < L::kChunks; ++c) tma_load_4d(d + c * kWChunk, &tmQ, bar(DT_QFULL + st), c * 64, ts * kTT, hh, bb);
                if (!mbar_wait(bar(DT_GEMPTY + st), ph, ctl, W + 2)) break;
                mbar_arrive_expect_tx(bar(DT_GFULL + st), L::kTok);
#pragma unroll
                for (int c = 0; c < L::kChunks; ++c)
                    tma_load_4d(d + L::kTok + c * kWChunk, &tmdO, bar(DT_GFULL + st), c * 64, ts * kTT, hh, bb);
                if (++st == L::kStages) { st = 0; ph ^= 1; }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer 1: M^T, N^T, dA^T
        if (lane == 0) {
            constexpr uint32_t idS = umma_idesc(128, kTT, false, false);
            const uint64_t dK = desc_kmajor(sW), dU = desc_kmajor(sW + L::kWMat), dV = desc_kmajor(sW + 2 * L::kWMat),
                           dQ0 = desc_kmajor(sTok), dG0 = desc_kmajor(sTok + L::kTok);
            constexpr uint64_t kTokStep = (2 * L::kTok) >> 4;
            bool ok = mbar_wait(bar(DT_WFULL), 0, ctl, W + 3);
            int st = 0;
            uint32_t ph = 0;
            for (int i = 0; ok && i < ntiles; ++i) {
                const int sb = i % kSB;
                if (!mbar_wait(bar(DT_QFULL + st), ph, ctl, W + 4)) break;
                if (!mbar_wait(bar(DT_SEMPTY + sb), ((uint32_t)(i / kSB) & 1u) ^ 1u, ctl, W + 5)) break;
                tc_fence_after();
                const uint64_t dq = dQ0 + st * kTokStep, dg = dG0 + st * kTokStep;
                const uint32_t tS = tmem + kColS + sb * 128;
#pragma unroll
                for (int which = 0; which < 2; ++which)
#pragma unroll
                    for (int k = 0; k < DH / 16; ++k) {
                        const int c = k >> 2, kk = k & 3;
                        umma_ss(tS + which * kTT, (which ? dU : dK) + ((c * 2 * kWChunk + kk * 32) >> 4), dq + ((c * kWChunk + kk * 32) >> 4),
                                idS, k > 0 ? 1u : 0u);
                    }
                umma_commit(bar(DT_SFULL + sb));
                if (!mbar_wait(bar(DT_GFULL + st), ph, ctl, W + 4)) break;
                if (!mbar_wait(bar(DT_DAEMPTY), (i & 1) ^ 1, ctl, W + 10)) break;
                tc_fence_after();
#pragma unroll
                for (int k = 0; k < DH / 16; ++k) {
                    const int c = k >> 2, kk = k & 3;
                    umma_ss(tmem + kColdA, dV + ((c * 2 * kWChunk + kk * 32) >> 4), dg + ((c * kWChunk + kk * 32) >> 4), idS, k > 0 ? 1u : 0u);
                }
                umma_commit(bar(DT_GEMPTY + st));
                umma_commit(bar(DT_DAFULL));
                if (++st == L::kStages) { st = 0; ph ^= 1; }
            }
        }
    } else if (warp == 2) {
        // ------------------------------------------------------------------ routing weights of each tile, times args.c
        const int e_lo = row0 / args.De, e_hi = min((row0 + 64) / args.De, args.E - 1);
        for (int i = 0; i < ntiles; ++i) {
            int ts, hh, bb;
            tile_coords(i, ts, hh, bb);
            const float *src = args.R + (long long)bb * args.r_sb + (long long)hh * args.r_sh;
            float v[2][2];
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const int t = ts * kTT + k * 32 + lane;
                v[0][k] = t < args.S ? args.c * __ldg(src + (long long)t * args.r_ss + e_lo) : 0.f;
                v[1][k] = t < args.S ? args.c * __ldg(src + (long long)t * args.r_ss + e_hi) : 0.f;
            }
            const int slot = i % L::kRSlots;
            if (!mbar_wait(bar(DT_REMPTY + slot), ((uint32_t)(i / L::kRSlots) & 1u) ^ 1u, ctl, W + 12)) break;
            float *dst = rbuf + slot * 2 * kTT;
#pragma unroll
            for (int x = 0; x < 2; ++x)
#pragma unroll
                for (int k = 0; k < 2; ++k) dst[x * kTT + k * 32 + lane] = v[x][k];
            warp_arrive(bar(DT_RFULL + slot));
        }
    } else if (warp == 3) {
        // ------------------------------------------------------------------ MMA issuer 2: dV, dK, dU, their A operands in tensor memory
        if (lane == 0) {
            constexpr uint32_t idA = umma_idesc(128, DH, false, true);
            const uint64_t dQ0 = desc_mnmajor(sTok, kWChunk), dG0 = desc_mnmajor(sTok + L::kTok, kWChunk);
            constexpr uint64_t kTokStep = (2 * L::kTok) >> 4;
            int st = 0;
            uint32_t ph = 0;
            bool ok = true;
            for (int i = 0; i < ntiles; ++i) {
                const int sb = i % kSB;
                const uint32_t sph = (uint32_t)(i / kSB) & 1u;
                const uint64_t dq = dQ0 + st * kTokStep, dg = dG0 + st * kTokStep;
                const uint32_t tS = tmem + kColS + sb * 128;
                if (!mbar_wait(bar(DT_GFULL + st), ph, ctl, W + 14)) { ok = false; break; }   // (A^T does not imply that dO is there)
                // k step of 16 tokens = 8 columns; a thread's 32 tokens (two steps) lie together: see the element-wise warps
                if (!mbar_wait(bar(DT_AFULL + sb), sph, ctl, W + 6)) { ok = false; break; }
                tc_fence_after();
#pragma unroll
                for (int k = 0; k < kTT / 16; ++k) {
                    const uint32_t a = kSB == 2 ? tS + (k >> 1) * 32 + (k & 1) * 8 : tmem + kColA + k * 8;
                    umma_ts(tmem + kColAcc + 2 * DH, a, dg + k * 128, idA, (i > 0 || k > 0) ? 1u : 0u);
                }
                umma_commit(bar(DT_GEMPTY + st));
                if (kSB == 1) umma_commit(bar(DT_AEMPTY));
                if (!mbar_wait(bar(DT_PFULL + sb), sph, ctl, W + 6)) { ok = false; break; }
                tc_fence_after();
#pragma unroll
                for (int k = 0; k < kTT / 16; ++k) {
                    const uint32_t off = (k >> 1) * 32 + (k & 1) * 8;
                    umma_ts(tmem + kColAcc, (kSB == 2 ? tS : tmem + kColdA) + off + (kSB == 2 ? 16 : 0), dq + k * 128, idA,
                            (i > 0 || k > 0) ? 1u : 0u);
                }
#pragma unroll
                for (int k = 0; k < kTT / 16; ++k) {
                    const uint32_t off = (k >> 1) * 32 + (k & 1) * 8;
                    umma_ts(tmem + kColAcc + DH, (kSB == 2 ? tS + kTT : tmem + kColdA + 16) + off, dq + k * 128, idA, (i > 0 || k > 0) ? 1u : 0u);
                }
                umma_commit(bar(DT_QEMPTY + st));
                umma_commit(bar(kSB == 2 ? DT_SEMPTY + sb : (int)DT_DAEMPTY));
                if (++st == L::kStages) { st = 0; ph ^= 1; }
            }
            if (ok) umma_commit(bar(DT_ACCFULL));
        }
    } else if (warp >= 4) {
        // ------------------------------------------------------------------ element-wise math: lane = weight row, 32 tokens a thread
        const int quarter = warp & 3, part = (warp - 4) >> 2;
        const int row = quarter * 32 + lane;
        const uint32_t lane_base = tmem + ((uint32_t)(quarter * 32) << 16);
        const float *rsrc = rbuf + (quarter >> 1) * kTT + part * 32;
        bool ok = true;
        const DwConst kc = dw_const(args.s0);
        for (int i = 0; i < ntiles; ++i) {
            const int sb = i % kSB, slot = i % L::kRSlots;
            if (!mbar_wait(bar(DT_RFULL + slot), (uint32_t)(i / L::kRSlots) & 1u, ctl, W + 13)) { ok = false; break; }
            if (!mbar_wait(bar(DT_SFULL + sb), (uint32_t)(i / kSB) & 1u, ctl, W + 7)) { ok = false; break; }
            tc_fence_after();
            const uint32_t tS = lane_base + kColS + sb * 128 + part * 32, tA = lane_base + kColdA + part * 32;
            const float *rs = rsrc + slot * 2 * kTT;
            // first what needs only S: A goes out, and its dV update runs, while dA is still being computed
            f32x2 fq[16], fw[16];
            uint32_t pa[16];
#pragma unroll
            for (int sub = 0; sub < 2; ++sub) {
                uint32_t m[16], n[16];
                tmem_ld16x2_sync(tS + sub * 16, tS + kTT + sub * 16, m, n);
                if (kSB == 1 && sub == 1) {   // S is in registers: the buffer can take the next tile
                    tc_fence_before();
                    warp_arrive(bar(DT_SEMPTY));
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float4 r4 = *reinterpret_cast<const float4 *>(rs + sub * 16 + q * 4);   // the same address in all lanes
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const int x = q * 2 + u;
                        const DwPair d = dw_pair(f2_pack_bits(m[2 * x], m[2 * x + 1]), f2_pack_bits(n[2 * x], n[2 * x + 1]),
                                                 u ? f2_pack(r4.z, r4.w) : f2_pack(r4.x, r4.y), kc);
                        fq[sub * 8 + x] = d.q;
                        fw[sub * 8 + x] = d.w;
                        pa[sub * 8 + x] = f2_to_bf16x2(d.a);
                    }
                }
            }
            warp_arrive(bar(DT_REMPTY + slot));
            if (kSB == 1 && i >= 1) {
                if (!mbar_wait(bar(DT_AEMPTY), (i - 1) & 1, ctl, W + 8)) { ok = false; break; }
                tc_fence_after();
            }
            tmem_st16(kSB == 2 ? tS : lane_base + kColA + part * 16, pa);
            tmem_st_wait();
            tc_fence_before();
            warp_arrive(bar(DT_AFULL + sb));
            // then dM and dN
            uint32_t da[32], pm[16], pn[16];
            if (!mbar_wait(bar(DT_DAFULL), i & 1, ctl, W + 11)) { ok = false; break; }
            tc_fence_after();
            tmem_ld32_sync(tA, da);
            if (kSB == 2) {
                tc_fence_before();
                warp_arrive(bar(DT_DAEMPTY));
            }
#pragma unroll
            for (int q = 0; q < 16; ++q) {
                const f32x2 da2 = f2_pack_bits(da[2 * q], da[2 * q + 1]);
                pm[q] = f2_to_bf16x2(f2_mul(da2, fw[q]));
                pn[q] = f2_to_bf16x2(f2_mul(da2, fq[q]));
            }
            tmem_st16(kSB == 2 ? tS + 16 : tA, pm);
            tmem_st16(kSB == 2 ? tS + kTT : tA + 16, pn);
            tmem_st_wait();
            tc_fence_before();
            warp_arrive(bar(DT_PFULL + sb));
        }
        if (ok) ok = mbar_wait(bar(DT_ACCFULL), 0, ctl, W + 9);
        if (ok) {
            tc_fence_after();
            const bool in_range = row0 + row < I;
            constexpr int kColsPerHalf = DH / 2;
            const int c0 = part * kColsPerHalf;
#pragma unroll
            for (int which = 0; which < 3; ++which) {
                float *dst = args.ws + ((long long)split * 3 + which) * args.ws_plane + ((long long)hk * I + row0 + row) * DH - args.ws_first + c0;
                __nv_bfloat16 *o16 = args.out[which] + hk * args.o_head[which] + (long long)(row0 + row) * args.o_row[which] + c0;
#pragma unroll
                for (int g = 0; g < kColsPerHalf / 16; ++g) {
                    uint32_t o[16];
                    tmem_ld16_sync(lane_base + kColAcc + which * DH + c0 + g * 16, o);
                    if (in_range) dw_store16(args.nsplit == 1 || blk < args.n_direct, dst + g * 16, o16 + g * 16, o);
                }
            }
            tc_fence_before();
        }
    }

    __syncwarp();
    if (*abort_flag) {
        const long long t_end = clock64() + (1LL << 19);
        while (clock64() < t_end) __nanosleep(256);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, kTmemCols);
    }
}

// Sum the token-axis splits in index order and write bf16 gradients (4 elements per thread, blockIdx.y = dK, dU or dV).
struct ReduceArgs {
    const float *ws;
    __nv_bfloat16 *out[3];
    long long s_head[3], s_row[3];
    long long plane;  // Hkuv * I * DH
    long long first;  // element of a plane where the split blocks begin (those before are written by their CTAs)
    int nsplit, I, DH;
};
// Launched early: what its CTAs have to set up is done when the kernel before it ends.
__global__ void __maxnreg__(48) dw_reduce_kernel(const ReduceArgs a) {
    griddep_launch_dependents();
    griddep_wait();
    const int which = blockIdx.y;
    const unsigned per_row = (unsigned)a.DH / 4;
    const long long n4 = a.plane / 4;
    const long long split4 = 3 * (n4 - a.first / 4);
    const float4 *src = reinterpret_cast<const float4 *>(a.ws) + which * (n4 - a.first / 4) - a.first / 4;
    for (long long idx = a.first / 4 + (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < n4;
         idx += (long long)gridDim.x * blockDim.x) {
        float4 acc = src[idx];
#pragma unroll 4
        for (int s = 1; s < a.nsplit; ++s) {
            const float4 v = src[s * split4 + idx];
            acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
        }
        long long rowi;
        unsigned c;
        if (n4 <= 0x7fffffffLL) { rowi = (unsigned)idx / per_row; c = (unsigned)idx - (unsigned)rowi * per_row; }
        else { rowi = idx / per_row; c = (unsigned)(idx - rowi * per_row); }
        const int hk = (int)(rowi / a.I), r = (int)(rowi - (long long)hk * a.I);
        __nv_bfloat16 *o = a.out[which] + hk * a.s_head[which] + r * a.s_row[which] + c * 4;
        *reinterpret_cast<uint2 *>(o) = make_uint2(pack_bf16(acc.x, acc.y), pack_bf16(acc.z, acc.w));
    }
}

// dQ/dR: with few token tiles the sub-networks are split over CTAs.  In 64-row blocks (about 0.8 us): a CTA costs six besides
// its blocks, the reduction three and its partial sums.  Splits only while the tiles are no more than two waves, and only for
// a gain of a tenth: the split sums dQ in another order than the unsplit kernel.  (The whole backward of 14 shapes of each head
// dimension that split, against never: 1.34x faster at d_h = 64, 1.22x at 96, 1.19x at 128; the rule does not know that unsplit CTAs may fit
// beside a small dK/dU/dV launch: 2 x 125 tokens, 16 heads, d_h = 96, 23 sub-networks of 64, 41 against 31 us.)
struct DqPlan {
    int nsplit, e_per_split;
};
DqPlan dq_plan(const flashmhf_dims &d, int num_sms) {
    const long long tiles = (long long)((d.S + kBT - 1) / kBT) * d.H * d.B;
    const int bpe = d.De / kBI;
    DqPlan best{1, d.E};
    if (tiles > 2LL * num_sms) return best;
    const double plane_blocks = (double)d.B * d.H * d.S * d.Dh * 4 / 3.0e6;
    auto waves = [&](long long n) { return (double)((n + num_sms - 1) / num_sms); };
    double best_cost = 0.9 * waves(tiles) * (6.0 + d.E * bpe);
    for (int eps = d.E - 1; eps >= 1; --eps) {
        const int ns = (d.E + eps - 1) / eps;
        const double cost = waves(tiles * ns) * (6.0 + eps * bpe) + 3.0 + ns * plane_blocks;
        if (cost < best_cost - 1e-9) { best_cost = cost; best = DqPlan{ns, eps}; }
    }
    return best;
}

static_assert(kBI == 64 && kBT == 128 && kTI == 128 && kTT == 64, "dw_shape");
size_t dq_workspace(const flashmhf_dims &d, const DqPlan &pl) {
    return pl.nsplit > 1 ? (size_t)pl.nsplit * d.B * d.H * d.S * d.Dh * sizeof(float) : 0;
}
size_t align256(size_t n) { return (n + 255) & ~(size_t)255; }

template <int DH>
int launch_bwd(const flashmhf_bwd_params &p, cudaStream_t st, int *n_launch) {
    const flashmhf_dims &d = p.d;
    const DeviceCtl *dc = device_ctl();
    if (!dc) return FLASHMHF_ERR_CUDA;
    const bool want_inputs = (p.parts & FLASHMHF_BWD_INPUTS) != 0, want_weights = (p.parts & FLASHMHF_BWD_WEIGHTS) != 0;
    CUtensorMap tmQ, tmdO, tmK, tmU, tmV, tmdQ;
    int rc;
    if ((rc = encode_act_map(&tmQ, p.Q, d, kBT)) != 0) return rc;
    if ((rc = encode_act_map(&tmdO, p.dO, d, kBT)) != 0) return rc;
    if ((rc = encode_weight_map(&tmK, p.K, d, kBI)) != 0) return rc;
    if ((rc = encode_weight_map(&tmU, p.U, d, kBI)) != 0) return rc;
    if ((rc = encode_weight_map(&tmV, p.V, d, kBI)) != 0) return rc;
    if (want_inputs && (rc = encode_act_map(&tmdQ, p.dQ, d, kBT)) != 0) return rc;
    if (want_weights)
        for (const flashmhf_tensor *t : {&p.dK, &p.dU, &p.dV}) {
            if (d.E > 1 && t->stride[1] != (int64_t)d.De * t->stride[2]) return FLASHMHF_ERR_BAD_STRIDE;
            if (t->stride[2] % 4 != 0 || t->stride[0] % 4 != 0) return FLASHMHF_ERR_BAD_STRIDE;
        }
    cudaError_t e;
    {  // the attribute is per device and per kernel: set once for each pair
        static std::atomic<bool> done[64];
        if (!done[dc->device].load(std::memory_order_acquire)) {
            e = cudaFuncSetAttribute(bwd_dq_kernel<DH>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DqSmem<DH>::kTotal);
            if (e == cudaSuccess)
                if constexpr (DH == 128)
                    e = cudaFuncSetAttribute(bwd_dw_kernel<DH>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DwSmem<DH>::kTotal);
                else
                    e = cudaFuncSetAttribute(bwd_dwt_kernel<DH>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DwtSmem<DH>::kTotal);
            if (e != cudaSuccess) { set_cuda_error(e, "cudaFuncSetAttribute(bwd kernels)"); return FLASHMHF_ERR_CUDA; }
            done[dc->device].store(true, std::memory_order_release);
        }
    }
    const int G = d.H / d.Hkuv;
    const float s0 = p.scale.head_scaling, c = p.scale.head_scaling * p.scale.up_scaling * p.scale.final_scaling;

    // Weight gradients first: in data-parallel training their all-reduce can then start while dQ/dR still run.  In a call for
    // everything the dQ/dR kernel is launched so that it may start under the tail of the dK/dU/dV kernel.
    DwPlan pl{};
    if (want_weights) {
        pl = dw_plan(d, dc->num_sms, want_inputs);
        if (dw_workspace(d, pl) > p.workspace_bytes) pl = dw_plan(d, dc->num_sms, want_inputs, p.workspace_bytes);   // (the static array)
    }
    ReduceArgs ra{};
    ra.ws = static_cast<const float *>(p.workspace);
    if (want_weights) {
        const flashmhf_tensor *outs[3] = {&p.dK, &p.dU, &p.dV};
        for (int i = 0; i < 3; ++i) {
            ra.out[i] = static_cast<__nv_bfloat16 *>(outs[i]->ptr);
            ra.s_head[i] = outs[i]->stride[0];
            ra.s_row[i] = outs[i]->stride[2];
        }
        ra.I = d.E * d.De;
        ra.DH = DH;
        ra.plane = (long long)d.Hkuv * ra.I * DH;
        ra.nsplit = pl.nsplit;
        ra.first = dw_first(d, pl);
        const int nblk_j = (d.E * d.De + dw_shape(DH).rows - 1) / dw_shape(DH).rows;
        DwArgs wa{static_cast<const float *>(p.R.ptr), p.R.stride[0], p.R.stride[1], p.R.stride[2],
                  static_cast<float *>(p.workspace), ra.plane - ra.first, ra.first, {ra.out[0], ra.out[1], ra.out[2]}, {ra.s_head[0], ra.s_head[1], ra.s_head[2]},
                  {ra.s_row[0], ra.s_row[1], ra.s_row[2]}, d.S, d.E, d.De, G, d.B, d.Hkuv,
                  pl.tiles_per_seq, pl.tiles_total, pl.tiles_per_split,
                  nblk_j, d.Hkuv * nblk_j, pl.nsplit, pl.n_direct, pl.n_mixed, pl.small_tiles, s0, 0.5f * c, wait_args(dc)};
        const long long ctas = pl.n_direct + (long long)(wa.n_blocks - pl.n_direct) * pl.nsplit;
        if (ctas > 0x7fffffffLL) return FLASHMHF_ERR_BAD_SHAPE;
        dim3 gw((unsigned)ctas);
        prof_mark(st, kMarkStart);
        if constexpr (DH == 128) {
            bwd_dw_kernel<DH><<<gw, kThreads, DwSmem<DH>::kTotal, st>>>(tmQ, tmdO, tmK, tmU, tmV, wa);
        } else {
            CUtensorMap tmQt, tmdOt;
            if ((rc = encode_act_map(&tmQt, p.Q, d, kTT)) != 0) return rc;
            if ((rc = encode_act_map(&tmdOt, p.dO, d, kTT)) != 0) return rc;
            bwd_dwt_kernel<DH><<<gw, kThreads, DwtSmem<DH>::kTotal, st>>>(tmQt, tmdOt, tmK, tmU, tmV, wa);
        }
        prof_mark(st, kMarkBwdDw);
        *n_launch += 1;
        if ((e = cudaGetLastError()) != cudaSuccess) { set_cuda_error(e, "bwd_dw_kernel launch"); return FLASHMHF_ERR_CUDA; }
    }

    DqPlan ql = dq_plan(d, dc->num_sms);
    float *q_part = nullptr;
    if (want_inputs) {
        if (ql.nsplit > 1) {   // the split's partial sums lie behind those of dK, dU, dV; without room for them the kernel runs unsplit
            const size_t off = want_weights ? align256(dw_workspace(d, pl)) : 0;
            if (p.workspace && p.workspace_bytes >= off + dq_workspace(d, ql))
                q_part = reinterpret_cast<float *>(static_cast<char *>(p.workspace) + off);
            else
                ql = DqPlan{1, d.E};
        }
        const DqArgs qa{static_cast<const float *>(p.R.ptr), p.R.stride[0], p.R.stride[1], p.R.stride[2],
                        static_cast<float *>(p.dR.ptr), p.dR.stride[0], p.dR.stride[1], p.dR.stride[2],
                        d.S, d.E, d.De, G, ql.nsplit, ql.e_per_split, d.H, d.B, q_part, s0, c, wait_args(dc)};
        const dim3 gq((unsigned)((d.S + kBT - 1) / kBT * ql.nsplit), d.H, d.B);
        prof_mark(st, kMarkStart);
        e = launch_kernel(want_weights, bwd_dq_kernel<DH>, gq, dim3(kThreads), DqSmem<DH>::kTotal, st, tmQ, tmdO, tmK, tmU, tmV, tmdQ, qa);
        prof_mark(st, kMarkBwdDq);
        *n_launch += 1;
        if (e != cudaSuccess) { set_cuda_error(e, "bwd_dq_kernel launch"); return FLASHMHF_ERR_CUDA; }
    }
    if (want_weights && pl.nsplit > 1) {
        // The addition of the split blocks' partial sums comes last, at full width.  (In front of the dQ/dR kernel, so as to run beside
        // it, its waiting CTAs keep that kernel's off their SMs: over 122 shapes of all head dimensions with up to 45 MB of sums the
        // backward took 5 % longer, up to 40 % where the weights are small: 16 x 1268 tokens, one sub-network of 64 at d_h = 96,
        // 118 against 84 us; 72 token tiles of d_h = 128 won most, 42 against 48 us.)
        const long long n4 = (ra.plane - ra.first) / 4, cap = dc->num_sms * 6;   // per gradient
        const dim3 blocks((unsigned)((n4 + 127) / 128 < cap ? (n4 + 127) / 128 : cap), 3);
        prof_mark(st, kMarkStart);
        e = launch_kernel(true, dw_reduce_kernel, blocks, dim3(128), 0, st, ra);
        prof_mark(st, kMarkBwdReduce);
        *n_launch += 1;
        if (e != cudaSuccess) { set_cuda_error(e, "dw_reduce_kernel launch"); return FLASHMHF_ERR_CUDA; }
    }
    if (want_inputs && ql.nsplit > 1) {
        prof_mark(st, kMarkStart);
        e = launch_o_reduce(q_part, p.dQ, d, ql.nsplit, /*chained=*/false, dc->num_sms, st);
        prof_mark(st, kMarkBwdReduce);
        *n_launch += 1;
        if (e != cudaSuccess) { set_cuda_error(e, "dQ split reduction launch"); return FLASHMHF_ERR_CUDA; }
    }
    return FLASHMHF_OK;
}

}  // namespace

size_t tc_backward_weights_workspace_bytes(const flashmhf_dims &d) {
    const DeviceCtl *dc = device_ctl();
    const int sms = dc ? dc->num_sms : 148;
    const size_t a = dw_workspace(d, dw_plan(d, sms, true)), b = dw_workspace(d, dw_plan(d, sms, false));
    return a > b ? a : b;
}
size_t tc_backward_inputs_workspace_bytes(const flashmhf_dims &d) {
    const DeviceCtl *dc = device_ctl();
    return dq_workspace(d, dq_plan(d, dc ? dc->num_sms : 148));
}
size_t tc_backward_workspace_bytes(const flashmhf_dims &d) {
    const size_t w = tc_backward_weights_workspace_bytes(d), q = tc_backward_inputs_workspace_bytes(d);
    return q ? align256(w) + q : w;
}

void tc_backward_plan(const flashmhf_dims &d, uint32_t parts, flashmhf_backward_plan_info *out) {
    const DeviceCtl *dc = device_ctl();
    const int sms = dc ? dc->num_sms : 148;
    *out = flashmhf_backward_plan_info{};
    if (parts & FLASHMHF_BWD_WEIGHTS) {
        const DwPlan p = dw_plan(d, sms, (parts & FLASHMHF_BWD_INPUTS) != 0);
        out->token_tiles = p.tiles_total;
        out->splits = p.nsplit;
        out->tiles_per_split = p.tiles_per_split;
        out->whole_blocks = p.nsplit > 1 ? p.n_direct : 0;
        out->uneven_blocks = p.n_mixed;
        out->small_tiles = p.small_tiles;
        out->predicted_tiles = p.tiles;
    }
    if (parts & FLASHMHF_BWD_INPUTS) out->dq_splits = dq_plan(d, sms).nsplit;
}

// ---------------------------------------------------------------------------------------------
// Built-in scratch for flashmhf_backward_static_scratch: the split partial sums of dK/dU/dV live in
// this file-scope device array instead of a caller-provided workspace.  One copy per GPU that loads
// the library, held until the process exits.  The dK/dU/dV kernel writes every partial it later
// reads, so nothing here has to start at zero.
constexpr size_t kStaticScratchBytes = FLASHMHF_STATIC_SCRATCH_BYTES;
static __device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];

namespace {
constexpr int kMaxDevices = 64;
std::mutex g_scratch_mu;
void *g_scratch_addr[kMaxDevices] = {nullptr};

// In host code `g_static_scratch` is only a handle for the symbol, not a device address: the
// address is looked up once per device, with that device current, and cached.
int static_scratch_ptr(void **out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
        set_cuda_error(e, "cudaGetDevice (static scratch)");
        return FLASHMHF_ERR_CUDA;
    }
    std::lock_guard<std::mutex> lk(g_scratch_mu);
    if (!g_scratch_addr[dev]) {
        void *ptr = nullptr;
        e = cudaGetSymbolAddress((void **)&ptr, g_static_scratch);
        if (e != cudaSuccess || !ptr) {
            set_cuda_error(e, "cudaGetSymbolAddress(g_static_scratch)");
            return FLASHMHF_ERR_CUDA;
        }
        g_scratch_addr[dev] = ptr;
    }
    *out = g_scratch_addr[dev];
    return FLASHMHF_OK;
}
}  // namespace

int tc_backward_static_scratch(const flashmhf_bwd_params &p, cudaStream_t st, int *n_launch) {
    // one set of partial sums has to fit; a plan that wants more of them than fit gives way to one that does not
    if ((size_t)p.d.Hkuv * p.d.E * p.d.De * p.d.Dh * 3 * sizeof(float) > kStaticScratchBytes) return FLASHMHF_ERR_SCRATCH_LIMIT;
    void *ptr = nullptr;
    const int rc = static_scratch_ptr(&ptr);
    if (rc != FLASHMHF_OK) return rc;
    flashmhf_bwd_params q = p;
    if (p.parts & FLASHMHF_BWD_WEIGHTS) {   // (a call for dQ and dR alone leaves the array to others)
        q.workspace = ptr;
        q.workspace_bytes = kStaticScratchBytes;
    } else {
        q.workspace = nullptr;
        q.workspace_bytes = 0;
    }
    return tc_backward(q, st, n_launch);
}

int tc_backward(const flashmhf_bwd_params &p, cudaStream_t st, int *n_launch) {
    switch (p.d.Dh) {
        case 64: return launch_bwd<64>(p, st, n_launch);
        case 96: return launch_bwd<96>(p, st, n_launch);
        case 128: return launch_bwd<128>(p, st, n_launch);
        default: return FLASHMHF_ERR_BAD_SHAPE;
    }
}

}  // namespace fmhf
