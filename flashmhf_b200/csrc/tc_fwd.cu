// Forward kernel, bf16, sm_100a:  O = sum_e R_e * ((SiLU(Q K_e^T) * (Q U_e^T)) V_e).
//
// One CTA owns one tile of 128 token rows of one (batch, head).  Its Q tile is loaded once; the
// weights of the head stream through shared-memory rings, 64 intermediate rows (one "block": 64
// rows of K_e, U_e and V_e) at a time.  Per block the tensor core computes
//     S = Q [K_blk; U_blk]^T      (128 x 128, one MMA chain, fp32 in tensor memory: M | N)
// the activation warps read S, form A = bf16(SiLU(M) * N * R_e) in registers and write it back into
// tensor memory (two bf16 per column), and the tensor core accumulates, with A read from tensor memory
// and V from shared memory,
//     O += A V_blk                (128 x d_h, fp32 in tensor memory, over all blocks of all e)
// so the [T, E*d_e] intermediate never leaves the SM and A never touches shared memory.
//
// Pipeline.  The hand-off from an MMA to the warps that consume its result costs several hundred
// cycles (commit -> mbarrier -> wake-up) and the tensor pipe accepts MMAs only a few ahead of their
// execution, so nothing on the S path waits for anything on the O path:
//   * Q is copied once from shared into tensor memory and the S chain reads it from there: an MMA with both
//     operands in shared memory uses the whole shared-memory bandwidth of the SM (measured: 128x128x16 takes
//     64.5 clk = 8 KB at 128 B/clk), which the weight tiles arriving by TMA need as well.
//   * S has two buffers.  A thread's first step on a block is to load its part of M and N into registers,
//     after which the buffer is free again -- S of block j+2 may be issued while block j is still being activated.
//   * A has slots of its own (32 columns each), so the O update of a block may lag its activation without
//     holding an S buffer.
//   * The two MMA chains are issued by different threads (S by two threads, one per S buffer, so that each
//     sees every phase of the barriers of its buffer; O by a third).
//
// Pairs of CTAs (CG = 2).  Every CTA reads all of its head's weights, 48 KB a block at d_h = 128 and as much again as the B operand of its
// MMAs.  Two CTAs with a token tile each of one head share them: the first loads K and one half of V's columns, the second U and the
// other half, and one MMA over both (cta_group::2, issued by the first) takes B from both shared memories.  That halves the bytes each
// SM fetches from L2 and reads from shared memory, which is energy: at the power limit 16 x 2048 tokens of the 370M layer (d_h = 128)
// 487 -> 471 us, 8192 tokens of the 1.3B layer 453 -> 435, 8 x 2048 tokens of the 128M layer (d_h = 96) 168.6 -> 157.9.  The pair's
// barriers for its issuing threads lie in the first CTA and take the arrivals of both; its commits go to both.
//
// Warp roles: warp 0 TMA producer, warps 1-2 MMA issuers for S (even / odd blocks; warp 1 owns tensor
// memory), warp 3 MMA issuer for O, then the activation warps (warp % 4 = TMEM lane quarter = 32 token rows).
//
// Tensor memory (512 columns): O at [0, d_h), Q (bf16) at [128, 192), A slots at [192, 256), S buffers at
// [256, 384), [384, 512).
#include <atomic>

#include "kernels.h"
#include "tc_common.cuh"
#include "tensormap.cuh"

namespace fmhf {
namespace {

constexpr int kBT = 128;  // token rows per tile
constexpr int kBI = 64;   // intermediate rows per block
// Shared-memory stages of the [K;U] ring and of the V ring.  The [K;U] ring must have an
// EVEN number of stages: its "full" barriers are waited on by the two S issuers, which own alternate blocks, and a
// barrier's phase is tracked with one parity bit, so each stage must always be waited on by the same issuer (with an
// odd ring an issuer would meet a stage only every other time it fills and could take an old phase for the new one).
// The depth is what hides a stage's way from L2 (about 1000 clk under load, 32 KB per 64-wide chunk row pair): a stage of
// the V ring is asked for again only when the O update that read it is done, so two stages cap the loop at two blocks per
// (load + update + hand-offs).  At d_h = 64 a block is short and shared memory is plentiful; at 96 and 128 the rings
// take what the Q tile leaves.
template <int DH, int CG>
struct FwdRings {
    static constexpr int kKU = CG == 2 ? 8 : DH == 64 ? 6 : 4, kV = CG == 2 ? 7 : DH == 64 ? 6 : 4;
    static_assert(kKU % 2 == 0, "each [K;U] stage must belong to one S issuer");
};
// Activation teams of eight warps (warp % 4 = lane quarter, next bit = which 32 of a block's 64 columns).  With two
// teams, team t owns the blocks j = t (mod 2) and with them S buffer t and A slot t; the two teams are then in
// different phases of their loop (wait, load, arithmetic, store), which keeps the arithmetic pipes busy.
// Two teams at d_h = 64 and 96, where the activation paces the kernel; one at d_h = 128, where the tensor pipe does and the weight tiles from
// L2 (48 KB a block and CTA, 24 of a pair): two teams of pairs there take 470.3 us, one 471.5 (32768 tokens of the 370M layer).
constexpr int kTeamThreads = 256;
__host__ __device__ constexpr int teams_for(int dh) { return dh == 128 ? 1 : 2; }
__host__ __device__ constexpr int threads_for(int dh) { return 128 + teams_for(dh) * kTeamThreads; }
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kColO = 0, kColQ = 128, kColA0 = 192, kColAStride = 32, kColS0 = 256, kColSStride = 128;

template <int DH, int CG>
struct FwdSmem {
    static constexpr int kChunks = (DH + 63) / 64;              // 64-column SW128 chunks per row of d_h
    static constexpr uint32_t kQBytes = kChunks * kBT * 128;    // one Q tile (also the O staging tile of its work item)
    static constexpr uint32_t kWChunk = kBI * 128;              // one 64-row x 64-col weight chunk
    // [K;U]: per chunk K rows then U rows = one 128-row K-major tile; of a pair, the first CTA has the K rows and the second the U rows
    static constexpr uint32_t kKUChunk = (CG == 2 ? 1 : 2) * kWChunk, kKUStage = kChunks * kKUChunk;
    static constexpr uint32_t kVStage = CG == 2 ? kWChunk : kChunks * kWChunk;   // of a pair each CTA has half of V's columns
    // offsets from the 1024-aligned base
    // ONE Q tile: an item's Q is copied to tensor memory before the item ahead of it is written out, so the tile is Q first and
    // that item's O staging tile next.  (A second tile would cost the V ring two of its stages.)
    static constexpr uint32_t kOffQ = 0;
    static constexpr uint32_t kOffKU = kOffQ + kQBytes;
    static constexpr uint32_t kOffV = kOffKU + FwdRings<DH, CG>::kKU * kKUStage;
    static constexpr uint32_t kOffBar = kOffV + FwdRings<DH, CG>::kV * kVStage;
    static constexpr uint32_t kTotal = kOffBar + 384 + 1024;  // + barriers/control + alignment slack
};

// barrier slots (8 bytes each) inside the control area
// QFULL: an item's Q has landed; QFREE: an item's O, staged over the Q of the item after it, has been read by its TMA store;
// SFULL[b]: S computed into buffer b; SEMPTY[b]: every warp of the team working on it has its part in registers;
// AFULL[s]: A written to slot s; AFREE[s]: the O update that read slot s is done; QT: Q copied to tensor memory
// (QTALL: of a pair, by both CTAs);
// SLAST: every S of a work item is computed (one commit from each S issuer; two teams only);
// OFULL: the last O update of a work item is done; OFREE: its accumulator has been read out.
// A CTA walks several work items (token tiles); blocks are counted through all of them (g), buffer and slot of a block
// are g % 2, so every barrier has one fixed set of
// waiters that observes each of its phases and a one-bit phase parity is enough.
constexpr int kMaxRing = 8;
enum { BAR_QFULL = 0, BAR_QFREE = 1, BAR_QT = 2, BAR_SLAST = 3, BAR_SFULL = 4, BAR_SEMPTY = 6, BAR_AFULL = 8, BAR_AFREE = 10, BAR_OFULL = 12,
       BAR_OFREE = 13, BAR_QTALL = 14, BAR_KUFULL = 15, BAR_KUEMPTY = BAR_KUFULL + kMaxRing, BAR_VFULL = BAR_KUEMPTY + kMaxRing,
       BAR_VEMPTY = BAR_VFULL + kMaxRing, BAR_COUNT = BAR_VEMPTY + kMaxRing };
static_assert(BAR_COUNT * 8 + 8 <= 384, "control area");

struct FwdArgs {
    const float *R;
    long long r_sb, r_sh, r_ss;
    int S, E, De, G;
    // Split of the intermediate dimension over CTAs (short token counts, e.g. decode): a work item is (token tile,
    // split) and covers blocks [isplit * blocks_per_split, ...) of the tile; it writes an fp32 partial O.
    int nsplit, blocks_per_split;
    float *part;           // [nsplit][B][H][S][DH] fp32, used when nsplit > 1
    int H, B;
    int tiles_per_seq, n_items;   // work items = tiles_per_seq * H * B * nsplit, dealt round-robin to the CTAs
    float half_s0;  // 0.5 * head_scaling: tanh argument scale, sigmoid(s0 m) = 0.5 + 0.5 tanh(0.5 s0 m)
    float c;        // head_scaling * up_scaling * final_scaling, folded into the routing weight
    // Chained call: launched with programmatic stream serialization.  The CTA may start, and stream weight tiles,
    // while the kernel before it on the stream still runs; Q and R are read, and anything written, only after
    // griddep_wait().
    int chained;
    WaitArgs wait;
};

// Ring position of block j in a ring of N slots: slot j % N and the parity of its lap.
template <int N>
struct RingPos {
    int slot = 0;
    uint32_t lap = 0;
    __device__ __forceinline__ void advance(int by) {
        slot += by;
        if (slot >= N) { slot -= N; lap ^= 1; }
    }
};

// A work item: which token tile of which (batch, head), which blocks of the intermediate dimension.
struct FwdItem {
    int t0, h, b, isplit, j0, nblk;
};
// Of a pair: one head and two token tiles, neighbours in the order (sequence, tile); behind the last tile of the last sequence b == B,
// which reads as zero and is not written.
template <int CG>
__device__ __forceinline__ FwdItem fwd_item(const FwdArgs &a, int item, int nblk_total, uint32_t rank) {
    FwdItem w;
    if (CG == 2) {
        const int pairs = (a.tiles_per_seq * a.B + 1) >> 1;
        w.h = item / pairs;
        const int t = 2 * (item - w.h * pairs) + (int)rank;
        w.b = t / a.tiles_per_seq;
        w.t0 = (t - w.b * a.tiles_per_seq) * kBT;
        w.isplit = w.j0 = 0;
        w.nblk = nblk_total;
        return w;
    }
    w.isplit = item % a.nsplit;
    int t = item / a.nsplit;
    w.t0 = (t % a.tiles_per_seq) * kBT;
    t /= a.tiles_per_seq;
    w.h = t % a.H;
    w.b = t / a.H;
    w.j0 = w.isplit * a.blocks_per_split;
    w.nblk = min(nblk_total - w.j0, a.blocks_per_split);
    return w;
}

// Registers: d_h = 128 at most 152, so that a 128-thread CTA of the split reduction (48 registers) fits beside this one on an SM and is
// resident when it ends; at 154 (allocated as 160) it is not, and a chained 1.3B decode step takes 23.0 instead of 21.9 us.
template <int DH, int CG>
__global__ void __maxnreg__(DH == 128 ? 152 : 96)
fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
           const __grid_constant__ CUtensorMap tmU, const __grid_constant__ CUtensorMap tmV,
           const __grid_constant__ CUtensorMap tmO, const FwdArgs args) {
    using L = FwdSmem<DH, CG>;
    constexpr int kTeams = teams_for(DH), kKURing = FwdRings<DH, CG>::kKU, kVRing = FwdRings<DH, CG>::kV;
    static_assert(kKURing <= kMaxRing && kVRing <= kMaxRing, "barrier slots");
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t *gbase = smem_raw + (base - raw);
    const uint32_t sQ = base + L::kOffQ, sKU = base + L::kOffKU, sV = base + L::kOffV, sBar = base + L::kOffBar;
    volatile uint32_t *tmem_slot = reinterpret_cast<volatile uint32_t *>(gbase + L::kOffBar + BAR_COUNT * 8);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(gbase + L::kOffBar + BAR_COUNT * 8 + 4);
    auto bar = [&](int i) { return sBar + 8u * i; };

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = CG == 2 ? cluster_rank() : 0;
    const int first_item = blockIdx.x / CG, item_step = gridDim.x / CG;
    // Barriers that the issuing CTA waits on and the element-wise warps or copies of both CTAs complete lie in the pair's first CTA.
    const uint32_t sLead = CG == 2 ? cluster_addr(sBar, 0) : sBar;
    auto lead = [&](int i) { return sLead + 8u * i; };
    auto arrive_lead = [&](int i) { if (CG == 2) warp_arrive_cluster(lead(i)); else warp_arrive(bar(i)); };
    auto commit = [&](int i) { if (CG == 2) umma_commit_pair(bar(i)); else umma_commit(bar(i)); };
    auto mma_ts = [&](uint32_t d, uint32_t a, uint64_t b, uint32_t id, uint32_t acc) {
        if (CG == 2) umma_ts_pair(d, a, b, id, acc);
        else umma_ts(d, a, b, id, acc);
    };
    const int blocks_per_e = args.De / kBI, nblk_total = args.E * blocks_per_e;
    const WaitCtl ctl{abort_flag, args.wait};
    constexpr int W = kKernelFwd * 100;
    auto wait_lead = [&](int i, uint32_t parity, int code) { return mbar_wait<CG == 2>(bar(i), parity, ctl, code); };

    if (threadIdx.x == 0) {
        *abort_flag = launch_aborted(args.wait);  // a CTA of this launch gave up: drain fast
        for (int i = 0; i < 2; ++i) {
            mbar_init(bar(BAR_SFULL + i), 1);
            mbar_init(bar(BAR_SEMPTY + i), CG * arrivals_of(kTeamThreads));
            mbar_init(bar(BAR_AFULL + i), CG * arrivals_of(kTeamThreads));
            mbar_init(bar(BAR_AFREE + i), 1);
        }
        for (int i = 0; i < kKURing; ++i) {
            mbar_init(bar(BAR_KUFULL + i), 1);
            mbar_init(bar(BAR_KUEMPTY + i), 1);
        }
        for (int i = 0; i < kVRing; ++i) {
            mbar_init(bar(BAR_VFULL + i), 1);
            mbar_init(bar(BAR_VEMPTY + i), 1);
        }
        mbar_init(bar(BAR_QFULL), 1);
        mbar_init(bar(BAR_QFREE), 1);
        mbar_init(bar(BAR_SLAST), 2);
        mbar_init(bar(BAR_OFULL), 1);
        mbar_init(bar(BAR_OFREE), CG * arrivals_of(kTeamThreads));
        mbar_init(bar(BAR_QT), arrivals_of(kTeamThreads));
        mbar_init(bar(BAR_QTALL), CG * arrivals_of(kTeamThreads));
        fence_mbar_init();
    }
    if (warp == 1) {
        if (CG == 2) tmem_alloc_pair(smem_u32(const_cast<uint32_t *>(tmem_slot)), kTmemCols);
        else tmem_alloc(smem_u32(const_cast<uint32_t *>(tmem_slot)), kTmemCols);
    }
    tc_fence_before();
    __syncthreads();
    if (CG == 2) cluster_sync();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    bool dead = *abort_flag != 0;
    if (CG == 2) {   // both CTAs of a pair give up, or neither
        dead = dead || ld_shared_cluster(cluster_addr(sBar + BAR_COUNT * 8 + 4, rank ^ 1)) != 0;
        cluster_sync();
    }
    // Every launch may start under the end of the kernel before it (a decode step of 8 tokens of the 370M layer 12.3 -> 9.6 us a call);
    // until that kernel has ended only a chained call's producer touches global memory (weight tiles), the others wait below.

    if (dead) {
        // nothing: fall through to the teardown
    } else if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer
        if (lane == 0) {
            tma_prefetch_desc(&tmQ);
            tma_prefetch_desc(&tmK);
            tma_prefetch_desc(&tmU);
            tma_prefetch_desc(&tmV);
            if (!args.chained) griddep_wait();
            RingPos<kKURing> pk;
            RingPos<kVRing> pv;
            bool ok = true;
            int n = 0;  // work items of this CTA so far
            for (int item = first_item; ok && item < args.n_items; item += item_step, ++n) {
                const FwdItem w = fwd_item<CG>(args, item, nblk_total, rank);
                const int hk = w.h / args.G;
                // the tile's last use: Q of item 0 (until it is in tensor memory), then O of item n - 2
                if (n == 1 && !mbar_wait(bar(BAR_QT), 0, ctl, W + 12)) break;
                if (n >= 2 && !mbar_wait(bar(BAR_QFREE), n & 1, ctl, W + 12)) break;
                // (the first Q of a chained call is asked for by the activation warps, once the kernel before this one has
                // completed: this thread touches only the weights and never waits for that)
                if (!(args.chained && n == 0)) {
                    mbar_arrive_expect_tx(bar(BAR_QFULL), L::kQBytes);
                    for (int c = 0; c < L::kChunks; ++c)
                        tma_load_4d(sQ + c * (kBT * 128), &tmQ, bar(BAR_QFULL), c * 64, w.t0, w.h, w.b);
                }
                // [K;U] of block j, then V of block j-2: V is consumed about two blocks later than K and U of
                // the same block, so with this lag the producer never waits on the V ring while a [K;U]
                // stage is free.
                for (int j = 0; j < w.nblk + 2; ++j) {
                    if (j < w.nblk) {
                        if (!mbar_wait(bar(BAR_KUEMPTY + pk.slot), pk.lap ^ 1, ctl, W + 1)) { ok = false; break; }
                        const uint32_t fku = lead(BAR_KUFULL + pk.slot), dku = sKU + pk.slot * L::kKUStage;
                        if (rank == 0) mbar_arrive_expect_tx(bar(BAR_KUFULL + pk.slot), CG * L::kKUStage);
#pragma unroll
                        for (int c = 0; c < L::kChunks; ++c) {
                            if (CG == 2) {
                                tma_load_3d_pair(dku + c * L::kKUChunk, rank ? &tmU : &tmK, fku, c * 64, (w.j0 + j) * kBI, hk);
                                continue;
                            }
                            tma_load_3d(dku + c * 2 * L::kWChunk, &tmK, fku, c * 64, (w.j0 + j) * kBI, hk);
                            tma_load_3d(dku + c * 2 * L::kWChunk + L::kWChunk, &tmU, fku, c * 64, (w.j0 + j) * kBI, hk);
                        }
                        pk.advance(1);
                    }
                    if (j >= 2) {
                        if (!mbar_wait(bar(BAR_VEMPTY + pv.slot), pv.lap ^ 1, ctl, W + 2)) { ok = false; break; }
                        const uint32_t fv = lead(BAR_VFULL + pv.slot), dv = sV + pv.slot * L::kVStage;
                        if (rank == 0) mbar_arrive_expect_tx(bar(BAR_VFULL + pv.slot), CG * L::kVStage);
                        // (d_h = 96: columns 48 to 111, of which those from 96 on are zero and not read)
                        if (CG == 2) tma_load_3d_pair(dv, &tmV, fv, (int)rank * (DH / 2), (w.j0 + j - 2) * kBI, hk);
#pragma unroll
                        for (int c = 0; c < (CG == 2 ? 0 : L::kChunks); ++c)
                            tma_load_3d(dv + c * L::kWChunk, &tmV, fv, c * 64, (w.j0 + j - 2) * kBI, hk);
                        pv.advance(1);
                    }
                }
            }
        }
    } else if (warp == 1 || warp == 2) {
        // ------------------------------------------------------------------ MMA issuers for S = Q [K;U]^T
        // Two threads (warp 1: even blocks into S buffer 0, warp 2: odd blocks into buffer 1; blocks counted through all
        // work items of the CTA): while one is between batches -- barrier polls, commits -- the other keeps the tensor
        // pipe fed.  Q is read from tensor memory.  One thread issues a chain, so its instruction stream is kept
        // minimal: descriptors are built once and advanced by adding constants (the address field counts 16-byte units).
        if (lane == 0 && rank == 0) {
            constexpr uint32_t idesc1 = umma_idesc(CG * 128, 2 * kBI, false, false);
            const uint64_t dKU0 = desc_kmajor(sKU);
            constexpr uint64_t kKUStep = L::kKUStage >> 4;
            const int sb = warp - 1;
            const uint32_t tS = tmem + kColS0 + sb * kColSStride, tQ = tmem + kColQ;
            bool ok = true;
            int g0 = 0, n = 0;   // blocks before this work item; work items so far
            for (int item = first_item; ok && item < args.n_items; item += item_step, ++n) {
                const FwdItem w = fwd_item<CG>(args, item, nblk_total, rank);
                if (!wait_lead(CG == 2 ? BAR_QTALL : BAR_QT, n & 1, W + 3)) break;   // this item's Q is in tensor memory
                for (int j = (g0 + sb) & 1; j < w.nblk; j += 2) {
                    const int g = g0 + j;                                 // g % 2 == sb
                    const int slot = g % kKURing;
                    if (!mbar_wait(bar(BAR_KUFULL + slot), (g / kKURing) & 1, ctl, W + 4)) { ok = false; break; }
                    // the buffer's previous block (g - 2) is in the activation warps' registers
                    if (g >= 2 && !wait_lead(BAR_SEMPTY + sb, ((g >> 1) - 1) & 1, W + 5)) { ok = false; break; }
                    tc_fence_after();
                    const uint64_t dku = dKU0 + slot * kKUStep;
#pragma unroll
                    for (int k = 0; k < DH / 16; ++k) {
                        const int c = k >> 2, kk = k & 3;
                        mma_ts(tS, tQ + k * 8, dku + ((c * L::kKUChunk + kk * 32) >> 4), idesc1, k > 0 ? 1u : 0u);
                    }
                    commit(BAR_KUEMPTY + slot);
                    commit(BAR_SFULL + sb);
                }
                if (kTeams == 2 && ok && item + item_step < args.n_items) commit(BAR_SLAST);   // (read before the next item's Q)
                g0 += w.nblk;
            }
        }
    } else if (warp == 3) {
        // ------------------------------------------------------------------ MMA issuer 2: O += A V
        // A comes from tensor memory (slot g % 2), V from shared memory as an MN-major operand.
        if (lane == 0 && rank == 0) {
            constexpr uint32_t idesc2 = umma_idesc(CG * 128, DH, false, true);
            const uint64_t dV0 = desc_mnmajor(sV, L::kWChunk);
            constexpr uint64_t kVStep = L::kVStage >> 4;
            bool ok = true;
            int g0 = 0, n = 0;
            for (int item = first_item; ok && item < args.n_items; item += item_step, ++n) {
                const FwdItem w = fwd_item<CG>(args, item, nblk_total, rank);
                // the accumulator of the previous work item has been read out
                if (n >= 1 && !wait_lead(BAR_OFREE, (n - 1) & 1, W + 13)) break;
                for (int j = 0; j < w.nblk; ++j) {
                    const int g = g0 + j, slot = g & 1, vs = g % kVRing;
                    if (!mbar_wait(bar(BAR_VFULL + vs), (g / kVRing) & 1, ctl, W + 6)) { ok = false; break; }
                    if (!wait_lead(BAR_AFULL + slot, (g >> 1) & 1, W + 7)) { ok = false; break; }
                    tc_fence_after();
                    const uint64_t dv = dV0 + vs * kVStep;
                    const uint32_t tA = tmem + kColA0 + slot * kColAStride;
#pragma unroll
                    for (int k = 0; k < kBI / 16; ++k)
                        mma_ts(tmem + kColO, tA + k * 8, dv + k * 128, idesc2, (j > 0 || k > 0) ? 1u : 0u);
                    commit(BAR_VEMPTY + vs);
                    commit(BAR_AFREE + slot);
                }
                if (ok) commit(BAR_OFULL);
                g0 += w.nblk;
            }
        }
    } else if (warp >= 4) {
        // ------------------------------------------------------------------ activation + epilogue
        const int quarter = warp & 3, team = (warp - 4) >> 3, group = ((warp - 4) >> 2) & 1;  // group = column half
        const int row = quarter * 32 + lane;
        const uint32_t lane_base = tmem + ((uint32_t)(quarter * 32) << 16);
        const f32x2 half_s0 = f2_pack(args.half_s0, args.half_s0);
        bool ok = true;
        int g0 = 0, n = 0;   // blocks before this work item; work items so far
        griddep_wait();   // these warps read R and write O
        // What follows (the reduction, the next call) may start now, and not before: a chained call reads its weights without waiting
        // and is promised only that the operation directly before it does not write them, so whatever came before this launch
        // must be complete when it starts.  (64 chained tokens of the 1.3B layer 21.5 -> 20.5 us against a trigger before the wait.)
        griddep_launch_dependents();
        if (args.chained) {
            if (warp == 4 && lane == 0 && first_item < args.n_items) {   // the first item's Q (q.v. the producer)
                const FwdItem w = fwd_item<CG>(args, first_item, nblk_total, rank);
                mbar_arrive_expect_tx(bar(BAR_QFULL), L::kQBytes);
                for (int c = 0; c < L::kChunks; ++c)
                    tma_load_4d(sQ + c * (kBT * 128), &tmQ, bar(BAR_QFULL), c * 64, w.t0, w.h, w.b);
            }
            __syncwarp();
        }
        // Copy of a work item's Q tile from shared into tensor memory, by team 0 (thread = token row; its lower four warps
        // copy columns [0, 64) of d_h, the upper four [64, 128)).  Done as soon as the previous item's last S has been
        // computed, i.e. before that item's epilogue, so that the first S of the new item is computed under the epilogue.
        auto copy_q = [&](int nn) -> bool {
            if (!mbar_wait(bar(BAR_QFULL), nn & 1, ctl, W + 11)) return false;
            if (group * 64 < DH) {
                uint32_t qv[32];
                const uint8_t *src = gbase + L::kOffQ + group * (kBT * 128);
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const uint4 v = *reinterpret_cast<const uint4 *>(src + sw128_offset(row, c));
                    qv[4 * c] = v.x; qv[4 * c + 1] = v.y; qv[4 * c + 2] = v.z; qv[4 * c + 3] = v.w;
                }
                tmem_st32(lane_base + kColQ + group * 32, qv);
                tmem_st_wait();
            }
            tc_fence_before();
            if (CG == 2) arrive_lead(BAR_QTALL);
            warp_arrive(bar(BAR_QT));
            return true;
        };
        if (team == 0 && first_item < args.n_items) ok = copy_q(0);
        for (int item = first_item; ok && item < args.n_items; item += item_step, ++n) {
            const FwdItem w = fwd_item<CG>(args, item, nblk_total, rank);
            const int t = w.t0 + row;
            const bool in_range = t < args.S && (CG == 1 || w.b < args.B);
            const float *rrow = args.R + (long long)w.b * args.r_sb + (long long)w.h * args.r_sh + (long long)t * args.r_ss;
            // this team's first block of the item, its sub-network and position inside it; routing weight fetched one ahead
            // (plain loads: the kernel before this one, under which this one may have started, can be the one that wrote R, and a
            // non-coherent load is only for memory that nobody writes while the grid runs)
            const int jfirst = kTeams == 1 ? 0 : ((g0 + team) & 1);
            int e = (w.j0 + jfirst) / blocks_per_e, in_e = (w.j0 + jfirst) - e * blocks_per_e;
            float r_cur = (in_range && e < args.E) ? rrow[e] : 0.f;
            float r_next = (in_range && e + 1 < args.E) ? rrow[e + 1] : 0.f;
            for (int j = jfirst; j < w.nblk; j += kTeams) {
                const int g = g0 + j, sb = g & 1;   // S buffer and A slot of this block
                const float hr = 0.5f * args.c * r_cur;
                const f32x2 half_r = f2_pack(hr, hr);
                if (!mbar_wait(bar(BAR_SFULL + sb), (g >> 1) & 1, ctl, W + 8)) { ok = false; break; }
                tc_fence_after();
                const uint32_t ts = lane_base + kColS0 + sb * kColSStride + group * 32;
                // this thread's 32 columns of M and of N -> 32 bf16 of A.  Two teams have 96 registers a thread: sixteen columns at a
                // time there (d_h = 64, 16384 tokens, 16 x 16 x 192: 381 -> 375 us; with one team no difference)
                constexpr int kPiece = kTeams == 2 ? 16 : 32;
                uint32_t a[16];
#pragma unroll
                for (int sub = 0; sub < 32 / kPiece; ++sub) {
                    uint32_t m[kPiece], nn[kPiece];
                    if constexpr (kPiece == 32) tmem_ld32x2_sync(ts, ts + kBI, m, nn);
                    else tmem_ld16x2_sync(ts + sub * 16, ts + kBI + sub * 16, m, nn);
                    if (sub == 32 / kPiece - 1) {
                        tc_fence_before();
                        arrive_lead(BAR_SEMPTY + sb);  // S is in registers: the buffer may take block g + 2
                    }
#pragma unroll
                    for (int i = 0; i < kPiece / 2; ++i)
                        a[sub * 8 + i] = fwd_act_pair(f2_pack_bits(m[2 * i], m[2 * i + 1]), f2_pack_bits(nn[2 * i], nn[2 * i + 1]), half_r,
                                                      half_s0);
                }
                // the slot's previous block (g - 2) has been consumed by its O update
                if (g >= 2 && !mbar_wait(bar(BAR_AFREE + sb), ((g >> 1) - 1) & 1, ctl, W + 9)) { ok = false; break; }
                tc_fence_after();
                tmem_st16(lane_base + kColA0 + sb * kColAStride + group * 16, a);
                tmem_st_wait();
                tc_fence_before();
                arrive_lead(BAR_AFULL + sb);
#pragma unroll
                for (int k = 0; k < kTeams; ++k)
                    if (++in_e == blocks_per_e) {
                        in_e = 0;
                        ++e;
                        r_cur = r_next;
                        r_next = (in_range && e + 1 < args.E) ? rrow[e + 1] : 0.f;
                    }
            }
            g0 += w.nblk;
            if (!ok || team != 0) continue;   // the rest of the item is team 0's
            // The next item's Q may replace this one's in tensor memory once every S of this item is computed.  One team has read
            // them all by now; of two, team 0 knows of its own blocks only and waits for the others'.  (An issuer begins an item
            // after its Q is there, so it is never a phase ahead of this wait.)
            if (item + item_step < args.n_items) {
                if (kTeams == 2) {
                    if (!mbar_wait(bar(BAR_SLAST), n & 1, ctl, W + 14)) { ok = false; break; }
                    tc_fence_after();
                }
                if (!copy_q(n + 1)) { ok = false; break; }
            }
            // epilogue: O (fp32, tensor memory) -> bf16 -> shared (over this item's Q tile) -> TMA store
            if (!mbar_wait(bar(BAR_OFULL), n & 1, ctl, W + 10)) { ok = false; break; }
            tc_fence_after();
            constexpr int kColsPerGroup = DH / 2;  // 64, 48 or 32 columns per thread
            const int c0 = group * kColsPerGroup;
            const uint32_t sO = sQ;
            if (args.nsplit > 1) {
                // partial O of this item's blocks, fp32, straight from tensor memory to the workspace
                float *dst = args.part + ((((long long)w.isplit * args.B + w.b) * args.H + w.h) * args.S + t) * DH + c0;
#pragma unroll
                for (int gg = 0; gg < kColsPerGroup / 16; ++gg) {
                    uint32_t o[16];
                    tmem_ld16_sync(lane_base + kColO + c0 + gg * 16, o);
                    if (in_range) {
#pragma unroll
                        for (int v = 0; v < 4; ++v)
                            *reinterpret_cast<float4 *>(dst + gg * 16 + v * 4) =
                                make_float4(__uint_as_float(o[4 * v]), __uint_as_float(o[4 * v + 1]),
                                            __uint_as_float(o[4 * v + 2]), __uint_as_float(o[4 * v + 3]));
                    }
                }
                tc_fence_before();
                arrive_lead(BAR_OFREE);
            } else {
                named_bar_sync(2, kTeamThreads);   // the next item's Q has been copied out of the tile by all of the team
#pragma unroll
                for (int gg = 0; gg < kColsPerGroup / 16; ++gg) {
                    uint32_t o[16];
                    tmem_ld16_sync(lane_base + kColO + c0 + gg * 16, o);
#pragma unroll
                    for (int v = 0; v < 2; ++v) {
                        const int col = c0 + gg * 16 + v * 8;  // first of 8 columns -> one 16-byte chunk
                        const uint32_t dst = sO + (col >> 6) * (kBT * 128) + sw128_offset(row, (col & 63) >> 3);
                        st_shared_v4(dst, pack_bf16(__uint_as_float(o[8 * v + 0]), __uint_as_float(o[8 * v + 1])),
                                     pack_bf16(__uint_as_float(o[8 * v + 2]), __uint_as_float(o[8 * v + 3])),
                                     pack_bf16(__uint_as_float(o[8 * v + 4]), __uint_as_float(o[8 * v + 5])),
                                     pack_bf16(__uint_as_float(o[8 * v + 6]), __uint_as_float(o[8 * v + 7])));
                    }
                }
                tc_fence_before();
                arrive_lead(BAR_OFREE);   // the accumulator is in registers / shared memory: the next item may overwrite it
                fence_async_smem();
                named_bar_sync(1, kTeamThreads);
                if (warp == 4 && lane == 0) {
                    for (int c = 0; c < (CG == 2 && w.b >= args.B ? 0 : L::kChunks); ++c) tma_store_4d(&tmO, sO + c * (kBT * 128), c * 64, w.t0, w.h, w.b);
                    tma_store_commit();
                    tma_store_wait_read();          // the tile has been read: it may take the Q of the item after next
                    mbar_arrive(bar(BAR_QFREE));
                }
            }
        }
        if (warp == 4 && lane == 0) tma_store_wait_all();
    }

    // ---------------------------------------------------------------------- teardown
    __syncwarp();
    if (*abort_flag) {
        // a wait ran out somewhere in this CTA: give copies and MMAs still in flight time to land
        // before shared and tensor memory are released
        const long long t_end = clock64() + (1LL << 19);
        while (clock64() < t_end) __nanosleep(256);
    }
    tc_fence_before();
    __syncthreads();
    if (CG == 2) cluster_sync();   // the other CTA arrives on barriers here, and its MMAs read this one's shared and tensor memory
    if (warp == 1) {
        tc_fence_after();
        if (CG == 2) tmem_dealloc_pair(tmem, kTmemCols);
        else tmem_dealloc(tmem, kTmemCols);
    }
}

// O = bf16(sum of the partial O of the splits, in split order); 4 elements per thread.
struct OReduceArgs {
    const float *part;
    long long plane;  // B*H*S*DH
    __nv_bfloat16 *O;
    long long s_b, s_h, s_s;
    int nsplit, H, S, DH;
};
// Measured (one B200): a decode step of 8 tokens of the 370M layer 14.4 -> 12.3 us, of 64 chained tokens 12.0 -> 10.0, against a loop
// that had three splits of two pieces in flight whatever the grid.
// 128 threads and few registers: its CTAs fit beside the forward kernel's on an SM, so a chained launch is resident (and
// has let the next forward launch in turn) long before the forward kernel it waits for ends.
__global__ void __maxnreg__(48) o_reduce_kernel(const OReduceArgs a) {
    griddep_launch_dependents();
    griddep_wait();   // launched early, behind the kernel whose partial sums it adds
    // Eight 16-byte loads of a thread are in flight (the partial sums come from L2 while the next call's weights stream in from
    // HBM: latency is what this kernel is made of): eight splits of one piece of O, or, where the grid is too small to give every
    // thread one piece, of two pieces the first split and then three more at a time; the splits are added in index order.  48
    // registers: 128 threads of it fit beside
    // the d_h = 128 forward CTA.  (a split call has at most a few hundred token tiles: every index fits 32 bits)
    const int n4 = (int)(a.plane / 4), stride = (int)(gridDim.x * blockDim.x);
    const float4 *part4 = reinterpret_cast<const float4 *>(a.part);
    auto add = [](float4 &acc, const float4 &v) { acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w; };
    auto at = [&](int s, int idx) { return __ldcg(part4 + (unsigned)(min(s, a.nsplit - 1) * n4 + idx)); };
    auto store = [&](int idx, const float4 &acc) {
        const int per_row = a.DH / 4;
        const int r1 = idx / per_row, c = (idx - r1 * per_row) * 4;
        const int r2 = r1 / a.S, t = r1 - r2 * a.S;
        const int b = r2 / a.H, h = r2 - b * a.H;
        *reinterpret_cast<uint2 *>(a.O + (long long)b * a.s_b + (long long)h * a.s_h + (long long)t * a.s_s + c) =
            make_uint2(pack_bf16(acc.x, acc.y), pack_bf16(acc.z, acc.w));
    };
    int idx = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    for (; idx + stride < n4; idx += 2 * stride) {
        float4 acc0 = at(0, idx), acc1 = at(0, idx + stride);
        for (int s0 = 1; s0 < a.nsplit; s0 += 3) {
            float4 v0[3], v1[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) { v0[k] = at(s0 + k, idx); v1[k] = at(s0 + k, idx + stride); }
#pragma unroll
            for (int k = 0; k < 3; ++k)
                if (s0 + k < a.nsplit) { add(acc0, v0[k]); add(acc1, v1[k]); }
        }
        store(idx, acc0);
        store(idx + stride, acc1);
    }
    if (idx < n4) {
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int s0 = 0; s0 < a.nsplit; s0 += 8) {
            float4 v[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) v[k] = at(s0 + k, idx);
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (s0 + k < a.nsplit) add(acc, v[k]);
        }
        store(idx, acc);
    }
}

struct FwdPlan {
    int nsplit, blocks_per_split;
};
// With fewer token tiles than about half the SMs (decode-shaped calls) the blocks of the intermediate
// dimension are spread over several CTAs per tile so that the weights stream in at full machine rate.
// All CTAs must run at once: one CTA per SM, so tiles * splits never exceeds the SM count (a second,
// nearly empty wave would double the duration of a call that lasts tens of microseconds).
FwdPlan fwd_plan(const flashmhf_dims &d, int num_sms) {
    const long long tiles = (long long)((d.S + kBT - 1) / kBT) * d.H * d.B;
    const int nblk = d.E * d.De / kBI;
    int ns = 1;
    if (tiles < num_sms / 2) ns = (int)(num_sms / tiles);
    if (ns > nblk) ns = nblk;
    FwdPlan p;
    p.blocks_per_split = (nblk + ns - 1) / ns;
    p.nsplit = (nblk + p.blocks_per_split - 1) / p.blocks_per_split;  // no empty split
    return p;
}

// Pairs of token tiles: those of one head in the order (sequence, tile), two by two.
long long fwd_pairs(const flashmhf_dims &d) { return ((long long)((d.S + kBT - 1) / kBT) * d.B + 1) / 2 * d.H; }
// In pairs at d_h = 96 and 128 (at 64 the activation paces the kernel: 372 us alone, 375 in pairs, 16384 tokens of 16 x 16 x 192), where
// they take no more rounds over the SMs than single tiles (an odd number of tiles of a head leaves half a pair empty).
bool fwd_in_pairs(const flashmhf_dims &d, const FwdPlan &pl, int num_sms) {
    if (pl.nsplit > 1 || d.Dh == 64) return false;
    const long long tiles = (long long)((d.S + kBT - 1) / kBT) * d.H * d.B, pairs = num_sms / 2;
    return (fwd_pairs(d) + pairs - 1) / pairs <= (tiles + num_sms - 1) / num_sms;
}

template <int DH, int CG>
int launch_fwd(const flashmhf_fwd_params &p, const FwdPlan &pl, const DeviceCtl *dc, cudaStream_t st, int *n_launch, bool chained) {
    using L = FwdSmem<DH, CG>;
    CUtensorMap tmQ, tmK, tmU, tmV, tmO;
    int rc;
    if ((rc = encode_act_map(&tmQ, p.Q, p.d, kBT)) != 0) return rc;
    if ((rc = encode_weight_map(&tmK, p.K, p.d, kBI)) != 0) return rc;
    if ((rc = encode_weight_map(&tmU, p.U, p.d, kBI)) != 0) return rc;
    if ((rc = encode_weight_map(&tmV, p.V, p.d, kBI)) != 0) return rc;
    if ((rc = encode_act_map(&tmO, p.O, p.d, kBT)) != 0) return rc;
    {  // the attributes are per device and per kernel: set once for each pair
        static std::atomic<bool> done[64];
        if (!done[dc->device].load(std::memory_order_acquire)) {
            cudaError_t e = cudaFuncSetAttribute(fwd_kernel<DH, CG>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L::kTotal);
            if (e != cudaSuccess) { set_cuda_error(e, "cudaFuncSetAttribute(fwd_kernel)"); return FLASHMHF_ERR_CUDA; }
            done[dc->device].store(true, std::memory_order_release);
        }
    }
    if (pl.nsplit > 1) {
        if (!p.workspace || p.workspace_bytes < tc_forward_workspace_bytes(p.d) ||
            (reinterpret_cast<uintptr_t>(p.workspace) & 255u))
            return FLASHMHF_ERR_WORKSPACE;
        if (p.O.stride[2] % 4 != 0 || p.O.stride[1] % 4 != 0 || p.O.stride[0] % 4 != 0) return FLASHMHF_ERR_BAD_STRIDE;
    }
    FwdArgs a{static_cast<const float *>(p.R.ptr), p.R.stride[0], p.R.stride[1], p.R.stride[2],
              p.d.S, p.d.E, p.d.De, p.d.H / p.d.Hkuv, pl.nsplit, pl.blocks_per_split,
              static_cast<float *>(p.workspace), p.d.H, p.d.B, 0, 0, 0.5f * p.scale.head_scaling,
              p.scale.head_scaling * p.scale.up_scaling * p.scale.final_scaling, chained ? 1 : 0, wait_args(dc)};
    a.tiles_per_seq = (p.d.S + kBT - 1) / kBT;
    const long long tiles = (long long)a.tiles_per_seq * p.d.H * p.d.B * pl.nsplit, items = CG == 2 ? fwd_pairs(p.d) : tiles;
    if (tiles > 0x7fffffffLL) return FLASHMHF_ERR_BAD_SHAPE;   // (in pairs, too: the kernel counts a head's tiles in 32 bits)
    a.n_items = (int)items;
    // one CTA per SM walks the work items round-robin: the next item's Q load, Q copy and first S overlap this item's epilogue
    // (a split call has one item per CTA: tiles * splits <= SMs)
    const unsigned grid = (unsigned)(CG * (items < dc->num_sms / CG ? items : dc->num_sms / CG));
    prof_mark(st, kMarkStart);
    cudaError_t e = launch_kernel(true, CG, fwd_kernel<DH, CG>, dim3(grid), dim3(threads_for(DH)), L::kTotal, st, tmQ, tmK, tmU, tmV, tmO, a);
    prof_mark(st, kMarkFwd);
    *n_launch += 1;
    if (e != cudaSuccess) { set_cuda_error(e, "fwd_kernel launch"); return FLASHMHF_ERR_CUDA; }
    if (pl.nsplit > 1) {
        e = launch_o_reduce(static_cast<const float *>(p.workspace), p.O, p.d, pl.nsplit, chained,
                            dc->num_sms, st);
        prof_mark(st, kMarkFwdReduce);
        *n_launch += 1;
        if (e != cudaSuccess) { set_cuda_error(e, "o_reduce_kernel launch"); return FLASHMHF_ERR_CUDA; }
    }
    return FLASHMHF_OK;
}

}  // namespace

cudaError_t launch_o_reduce(const float *part, const flashmhf_tensor &out, const flashmhf_dims &d, int nsplit, bool chained, int num_sms,
                            cudaStream_t st) {
    const long long plane = (long long)d.B * d.H * d.S * d.Dh, n4 = plane / 4;
    const OReduceArgs ra{part, plane, static_cast<__nv_bfloat16 *>(out.ptr), out.stride[0], out.stride[1], out.stride[2], nsplit, d.H, d.S,
                         d.Dh};
    // chained: at most one (small) CTA per SM, so that all of them are resident beside the forward kernel's
    const long long cap = chained ? (long long)num_sms : (long long)num_sms * 8;
    const int blocks = (int)((n4 + 127) / 128 < cap ? (n4 + 127) / 128 : cap);
    return launch_kernel(true, o_reduce_kernel, dim3(blocks), dim3(128), 0, st, ra);
}

size_t tc_forward_workspace_bytes(const flashmhf_dims &d) {
    const DeviceCtl *dc = device_ctl();
    const FwdPlan pl = fwd_plan(d, dc ? dc->num_sms : 148);
    if (pl.nsplit <= 1) return 0;
    return (size_t)pl.nsplit * (size_t)d.B * d.H * d.S * d.Dh * sizeof(float);
}

template <int DH>
int forward_of(const flashmhf_fwd_params &p, cudaStream_t st, int *n_launch, bool chained) {
    const DeviceCtl *dc = device_ctl();
    if (!dc) return FLASHMHF_ERR_CUDA;
    const FwdPlan pl = fwd_plan(p.d, dc->num_sms);
    if constexpr (DH != 64)
        if (fwd_in_pairs(p.d, pl, dc->num_sms)) return launch_fwd<DH, 2>(p, pl, dc, st, n_launch, chained);
    return launch_fwd<DH, 1>(p, pl, dc, st, n_launch, chained);
}

int tc_forward(const flashmhf_fwd_params &p, cudaStream_t st, int *n_launch, bool chained) {
    switch (p.d.Dh) {
        case 64: return forward_of<64>(p, st, n_launch, chained);
        case 96: return forward_of<96>(p, st, n_launch, chained);
        case 128: return forward_of<128>(p, st, n_launch, chained);
        default: return FLASHMHF_ERR_BAD_SHAPE;
    }
}

}  // namespace fmhf
