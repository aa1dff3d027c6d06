// Histograms of few-bin codes (4-bit codes, at most eight bins) as a contraction on the tensor cores.
//
// For the rows of an era (or of a tile of one) and a threshold t of a feature f,
//     sum over rows of [code_f(row) > t] * [slot(row) == node] * value(row)
// is a matrix product over the rows: A[(f, t)][row] is 0 or 1, B[(node, j)][row] holds the row's value in
// the node's columns and 0 elsewhere.  The values are the four signed base-256 digits of the fixed-point
// gradient and a 1 for the count, so products and sums are whole numbers (8-bit operands, 32-bit
// accumulators) and the sums are exact: |digit| * rows of a tile < 2^22.
//
// A CTA per SM goes through its share of (feature block, tile of rows) tasks; a block is FC = 128 L / TP features
// (TP thresholds of a feature: 4 or 8; L of them per tensor-memory lane).  Its warps:
//   copy     bring codes, frontier slots and gradients of the next 512 rows into shared memory, whole lines;
//   rows     write the B operand: five bytes per row, the five bytes of the row before cleared;
//   codes    turn codes into A: the eight nibbles of a word are the selectors of two byte permutes of the
//            threshold's table, so a permute makes four operand bytes and no nibble is ever unpacked.  A goes to
//            tensor memory, where the lane is (feature, thresholds);
//   issue    one thread each: L tcgen05.mma (M 128, N 5 columns a node, K 32) per 32 rows;
//   flush    read the accumulators of the task before, while the others work on the next one: per-era gains
//            and left sums (summed over the CTA's eras before they go out), or a tile's share of the histogram.
// Operands pass in batches of 64 or 128 rows through three places, each with code and row warps of its own.
//
// Bound: no unit of the SM (ALU pipe 62 % of the time, issue slots 60 %, tensor pipe 16 %; 485 instructions per 32 rows and
// 128 features at one node, 164 of them for A) but the hand-overs between the roles: a batch waits for its stores into
// tensor memory and at two barriers, in one of three places.  What it took:
// the warps of a place wait at one barrier behind one poller (two dozen polling warps made a wait that is over
// cost 350 cycles), the issuers wait at a barrier too (a ready mbarrier costs a thread that issues tcgen05.mma
// 200 cycles, a barrier a few), codes come by cp.async from four warps (bulk copies of a line each: 35 cycles
// each, 416 us where this takes 126), and three places (two: 141 us).
// 2 700 000 rows x 238 features, 574 eras: 172 us by atomics, 126 so, at one node (2.7 TB/s of codes and row
// state, 41 % of measured copy bandwidth); figures by size in hist_rule.h.

#include <stdio.h>
#include <stdlib.h>

#include <type_traits>

#include "common.cuh"
#include "des_math.cuh"
#include "hist_rule.h"
#include "rows.cuh"

namespace pb {

namespace {

constexpr int kSlots = 3;               // places for the operands of a batch; each has four code warps and two row warps,
constexpr int kCodeWarps = 4 * kSlots, kRowWarps = 2 * kSlots, kCopyWarps = 4;   // which make every third batch
// Warp numbers: code, flush, row, issuer, copy.  (A warp reaches the tensor-memory lanes 32 (warp % 4) on.)
__host__ __device__ constexpr int mma_flush_warps(bool groups) { return groups ? 8 : 4; }
__host__ __device__ constexpr int mma_issue_warps(int L) { return L > 1 ? 2 : 1; }
__host__ __device__ constexpr int mma_threads(bool groups, int L) { return 32 * (kCodeWarps + mma_flush_warps(groups) + kRowWarps + mma_issue_warps(L) + kCopyWarps); }
constexpr int kStages = 3;           // blocks of codes on their way
constexpr int kBlock = kCutRows;           // rows of a block: 256 bytes of a feature
constexpr int kPitch = 272;             // bytes per feature of a staged block: lanes that read 16 bytes of
                                        // consecutive features touch every bank
constexpr int kColumns = 512;           // all of the tensor memory: a CTA per SM
constexpr int kMmaTileRows = 32256;     // rows of a tile: sums of its digits stay below 2^22, two of them make 32 bits
constexpr int kTries = 1 << 15;         // eights of tries of a wait, up to 2 us a try

struct MmaArgs {
    const uint8_t* codes;
    int64_t pitch;
    const int32_t* feat_rows;
    int n_feat;
    const int32_t* gq;
    const uint16_t* slot;
    int64_t rows_pad;                   // entries of gq and slot
    const int32_t* era_offsets;
    int n_eras;
    int max_bins;
    int blocks;                         // feature blocks
    Shares shares;                      // of the CTAs
    int era_rows;                       // work of an era beside its rows
    const int32_t* n_nodes_ptr;
    int n_nodes;                        // upper bound
    int node_stride;
    uint32_t* cnt;
    int64_t* gsum;
    int fuse;
    HistFuse fz;
    uint32_t* flags;
    int groups;                         // lanes of a feature: TP / L
    int buffers;                        // accumulators: 2 where they fit
    int failed;                         // 1: as after a wait that ran out
};

__device__ __forceinline__ uint32_t smem_at(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_at(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("{ .reg .b64 s; mbarrier.arrive.shared::cta.b64 s, [%0]; }" ::"r"(smem_at(bar)) : "memory");
}
// Waits for the end of a phase; IDLE: nothing hangs on a microsecond here, and a warp that keeps asking takes issue
// slots from the others.  A wait that runs out marks the launch as failed, after which every wait ends within
// eight tries and no product is issued any more, but each role still goes through all of its steps: no warp decides
// alone to leave.  So the named barriers, which have no limit, are met by all of their warps as often as ever; and
// since nothing else then keeps a place from being handed over twice, its warps wait until the issuing warps, which
// take the places in turn whatever happens, have taken it (s_taken).  The launch ends, its sums are not to be used,
// and the control block says so.
template <bool IDLE = false>
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* fail) {
    const uint32_t at = smem_at(bar);
    for (int i = 0; i < kTries; ++i) {
#pragma unroll 1
        for (int j = 0; j < 8; ++j) {
            uint32_t ok;
            asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, 2000; selp.u32 %0, 1, 0, p; }"
                         : "=r"(ok) : "r"(at), "r"(parity) : "memory");
            if (ok) return true;
            if (IDLE) __nanosleep(500);
        }
        if (*fail) return false;
    }
    *fail = 1;
    return false;
}
// The same for a whole warp, which goes on together.
template <bool IDLE = false>
__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity, volatile int* fail) {
    return __all_sync(0xFFFFFFFFu, mbar_wait<IDLE>(bar, parity, fail));
}
__device__ __forceinline__ bool elect_one() {
    uint32_t e;
    asm volatile("{ .reg .pred p; elect.sync _|p, 0xFFFFFFFF; selp.u32 %0, 1, 0, p; }" : "=r"(e));
    return e != 0u;
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_at(bar)) : "memory");
}

__device__ __forceinline__ void mma_i8(uint32_t d, uint32_t a_at, uint64_t b_desc, uint32_t idesc, uint32_t add) {
    asm volatile("{ .reg .pred p; setp.ne.u32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p; }"
                 ::"r"(d), "r"(a_at), "l"(b_desc), "r"(idesc), "r"(add) : "memory");
}
// `threads` threads meet at a barrier of the CTA.
__device__ __forceinline__ void meet(int barrier, int threads) {
    asm volatile("barrier.cta.sync %0, %1;" ::"r"(barrier), "r"(threads) : "memory");
}
constexpr int kFlushBarrier = 1, kSlotBarrier = 2, kFullBarrier = kSlotBarrier + kSlots;   // (the latter two: one per slot)
constexpr int kSlotThreads = 32 * 6;
// A slot's operands are there: its warps go on, the issuing warp waits for them.  (A wait on an mbarrier that
// is over costs a thread which issues tcgen05.mma some 200 cycles, this one a few.)
__device__ __forceinline__ void hand_over(int slot, int issue_warps) {
    asm volatile("barrier.cta.arrive %0, %1;" ::"r"(kFullBarrier + slot), "r"(kSlotThreads + 32 * issue_warps) : "memory");
}
__device__ __forceinline__ void lds16(uint32_t at, uint32_t (&v)[4]) {
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(at) : "memory");
}
__device__ __forceinline__ void sts8(uint32_t at, uint32_t v) {
    asm volatile("st.shared.b8 [%0], %1;" ::"r"(at), "r"(v) : "memory");
}
__device__ __forceinline__ void copy16(uint32_t to, const void* from) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to), "l"(from) : "memory");
}
// Eight words of this lane to eight neighbouring columns.
__device__ __forceinline__ void tmem_store(uint32_t at, const uint32_t (&v)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(at), "r"(v[0]), "r"(v[1]),
                 "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
}
__device__ __forceinline__ void tmem_load1(uint32_t at, int& v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(v) : "r"(at));
}
__device__ __forceinline__ void tmem_load_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Four neighbouring codes (the low 16 bits of w) looked up in a table of eight bytes.
__device__ __forceinline__ uint32_t lookup4(uint32_t lo, uint32_t hi, uint32_t w) {
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(lo), "r"(hi), "r"(w));
    return r;
}

// Columns of B.  Up to four nodes: eight neighbouring columns a node (its four digits, its count, three that
// stay empty).  More: five groups of eight columns for every eight nodes, a node's column in each.  Either way
// the five columns of a node are a constant apart, in shared memory and in the accumulators.
__host__ __device__ constexpr bool mma_groups(int n_nodes) { return n_nodes > 4; }
__host__ __device__ constexpr int mma_columns(int n_nodes, bool groups) {
    return ((groups ? (n_nodes + 7) / 8 * 40 : 8 * n_nodes) + 15) / 16 * 16;
}
__host__ __device__ constexpr int mma_stage_bytes(int features) { return features * kPitch + kBlock * 6; }

// L: thresholds of a lane; KB: K-steps of a batch; GROUPS: layout of the columns; WIDE: more than 256, two products;
// FUSE: the flush makes the gains
template <int L, int KB, bool GROUPS, bool WIDE, bool FUSE>
__global__ void __launch_bounds__(mma_threads(GROUPS, L), 1) hist_mma_kernel(MmaArgs a) {
    constexpr int kMmaThreads = mma_threads(GROUPS, L), kFlushWarps = mma_flush_warps(GROUPS), kBatch = KB, kBatchRows = 32 * KB;
    constexpr int kUnits = kBlock / kBatchRows;              // batches of a block
    constexpr int kFlushWarp0 = kCodeWarps, kRowWarp0 = kFlushWarp0 + kFlushWarps, kIssueWarp = kRowWarp0 + kRowWarps, kCopyWarp0 = kIssueWarp + mma_issue_warps(L);
    constexpr int kIssueWarps = mma_issue_warps(L), kTilesOf = L / kIssueWarps;   // (accumulators of one issuing warp)
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(8) uint64_t full_c[kStages], empty_c[kStages], empty[kSlots], acc_full[2], acc_empty[2], tot_full[2], last;
    __shared__ uint32_t s_tmem;
    __shared__ volatile int s_fail;
    __shared__ uint32_t s_taken[kSlots];   // times the issuing warps have taken over a place, all together
    __shared__ float4 s_era[64];         // {gradient total, hessian total, parent term, era weight} of a node
    __shared__ long long s_tgq[64];
    __shared__ uint32_t s_tc[64];
    __shared__ int s_kof[8];             // position of a bin among the thresholds, -1: none
    __shared__ int s_cut[2][3];          // where this CTA's rows begin and end: feature block, era, row

    const int n_nodes = a.n_nodes_ptr ? min(*a.n_nodes_ptr, a.n_nodes) : a.n_nodes;
    if (n_nodes <= 0) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int G = a.groups, FC = 128 / G;
    const int N = mma_columns(n_nodes, GROUPS), N_max = mma_columns(a.n_nodes, GROUPS);
    const int k_bytes = N_max * 32, batch_bytes = kBatch * k_bytes;   // of B
    const int stage_bytes = mma_stage_bytes(FC);
    unsigned char* s_codes = smem;                            // [stages]{[FC][kPitch], slots, gradients}
    unsigned char* s_b = smem + kStages * stage_bytes;        // [kSlots][kBatch][N / 8][2][8][16]
    uint32_t* s_tot = reinterpret_cast<uint32_t*>(s_b + kSlots * batch_bytes);   // [buffers][count, low, high][n_nodes][32]: a lane's own cells
    const int tot_plane = a.n_nodes * 32;
    // (fused) left sums over the CTA's eras of a feature block: a flush thread's own, [n_nodes][L][128]
    long long* s_lg = reinterpret_cast<long long*>(s_tot + a.buffers * 3 * tot_plane);
    uint32_t* s_lc = reinterpret_cast<uint32_t*>(s_lg + a.n_nodes * L * 128);

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_at(&s_tmem)), "n"(kColumns) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (threadIdx.x == 32) {
        for (int i = 0; i < kStages; ++i) {
            mbar_init(full_c + i, 32 * kCopyWarps);
            mbar_init(empty_c + i, kCodeWarps + kRowWarps);
        }
        for (int i = 0; i < kSlots; ++i) {
            mbar_init(empty + i, kIssueWarps);
            s_taken[i] = 0u;
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(acc_full + i, kIssueWarps);
            mbar_init(acc_empty + i, kFlushWarps);
            mbar_init(tot_full + i, kRowWarps);
        }
        mbar_init(&last, kIssueWarps);
        s_fail = a.failed;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // The CTAs' shares are ranges of (feature block, row), the block the slowest (totals over the eras gather in a
    // CTA), cut at equal rows, since eras differ in length; with gains in the flush an era is not divided.  (Shares of
    // as many tasks, and tiles counted by the longest era, where this takes, us at one and eight nodes, five bins:
    // 2 700 000 rows x 238 features, 574 eras that grow to 2.8 times the first 163 and 313, now 133 and 264; 2 600 000
    // x 238, 200 eras of gamma(4) lengths 170 and 295, now 109 and 207; 1 100 000 x 57, two eras, one a tenth of the
    // other 41 and 47, now 31 and 38; equal eras 123 and 238, now 123 and 249.)
    const int E = a.n_eras;
#pragma unroll 1
    for (int end = 0; end < 2; ++end) {
        int fb;
        const int64_t at = share_begin(a.shares, (int)blockIdx.x + end, fb);
#pragma unroll 1
        for (int e = kMmaThreads - 1 - threadIdx.x; e <= E; e += kMmaThreads) {   // (the first warp has other things to do)
            int row = 0;
            if (fb == a.blocks ? e == 0 : FUSE ? cut_in_era<true>(a.era_offsets, E, at, a.era_rows, e, row) : cut_in_era<false>(a.era_offsets, E, at, 0, e, row)) {
                s_cut[end][0] = e == E ? fb + 1 : fb;
                s_cut[end][1] = e == E ? 0 : e;
                s_cut[end][2] = e == E ? 0 : row;
            }
        }
    }
    {
        uint4* z = reinterpret_cast<uint4*>(s_b);
        const int n16 = (kSlots * batch_bytes + a.buffers * 3 * tot_plane * 4) / 16;
        for (int i = threadIdx.x; i < n16; i += kMmaThreads) z[i] = make_uint4(0u, 0u, 0u, 0u);
    }
    if (FUSE && threadIdx.x < 8) {
        int k = -1;
        for (int i = 0; i < a.fz.n_thr; ++i)
            if (a.fz.thr_ids[i] == (int)threadIdx.x) k = i;
        s_kof[threadIdx.x] = k;
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    constexpr uint32_t tmem = 0u;        // (all columns are this CTA's)
    const uint32_t a_col = tmem + (uint32_t)(a.buffers * L * N_max);

    // Every role goes through the same tasks.
    auto next_task = [&](RowTask& x) { return next_row_task(a.era_offsets, E, FUSE, s_cut[1], kMmaTileRows, x); };
    RowTask x;
    x.fb = s_cut[0][0];
    x.next = s_cut[0][1];
    x.r1 = s_cut[0][2];

    if (warp < kCodeWarps) {
        // ---- A: this lane's feature and its L thresholds ----
        const int wg = warp >> 2, quarter = warp & 3;
        auto first_unit = [&](int b) { return (int)((uint32_t)(wg + kSlots * kUnits - (b * kUnits) % kSlots) % kSlots); };
        const int row = quarter * 32 + lane, fl = row / G, g = row - fl * G;
        uint32_t lut_lo[L], lut_hi[L];
#pragma unroll
        for (int l = 0; l < L; ++l) {
            const int t = g * L + l;
            lut_lo[l] = lut_hi[l] = 0u;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                if (t < a.max_bins - 1 && c > t) lut_lo[l] |= 1u << (8 * c);
                if (t < a.max_bins - 1 && c + 4 > t) lut_hi[l] |= 1u << (8 * c);
            }
        }
        const uint32_t to = a_col + ((uint32_t)quarter << 21);
        const uint32_t at = to + (uint32_t)(wg * (kBatch * L * 8));
        int stage = 0;
        while (next_task(x)) {
            for (int b = x.b0; b < x.b1; ++b) {
                bool met = false;
#pragma unroll 1
                for (int u = first_unit(b); u < kUnits; u += kSlots) {
                    const int i = u * kBatchRows, r = b * kBlock + i;
                    if (r + kBatchRows <= x.r0 || r >= x.r1) continue;
                    met = true;
                    meet(kSlotBarrier + wg, kSlotThreads);
                    const uint32_t from = smem_at(s_codes + stage * stage_bytes + fl * kPitch + i / 2);
                    tc_fence_after();
#pragma unroll
                    for (int k = 0; k < kBatch; ++k) {
                        uint32_t c[4], up[4];
                        lds16(from + 16 * k, c);
#pragma unroll
                        for (int q = 0; q < 4; ++q) up[q] = c[q] >> 16;
#pragma unroll
                        for (int l = 0; l < L; ++l) {    // (stores read their registers while the next words are made)
                            uint32_t w[8];
#pragma unroll
                            for (int q = 0; q < 4; ++q) {
                                w[2 * q] = lookup4(lut_lo[l], lut_hi[l], c[q]);
                                w[2 * q + 1] = lookup4(lut_lo[l], lut_hi[l], up[q]);
                            }
                            tmem_store(at + (uint32_t)((k * L + l) * 8), w);
                        }
                    }
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                    tc_fence_before();
                    __syncwarp();
                    hand_over(wg, kIssueWarps);
                }
                if (!met) meet(kSlotBarrier + wg, kSlotThreads);   // (a stage is given back only after it came)
                __syncwarp();
                if (lane == 0) mbar_arrive(empty_c + stage);
                if (++stage == kStages) stage = 0;
            }
        }
    } else if (warp < kRowWarp0) {
        // ---- flush ----
        constexpr int U = L == 4 ? 1 : 2;            // nodes at a time
        constexpr int J = GROUPS ? 8 : 1;            // columns between the digits of a node
        const int quarter = warp & 3, fg = (warp - kFlushWarp0) >> 2, row = quarter * 32 + lane, fl = row / G, g = row - fl * G;
        const HistFuse& z = a.fz;
        const float inv_scale = FUSE ? *z.inv_scale_ptr : 0.f;
        const int K = z.n_thr, lanes_total = a.blocks * FC;
        int buf = 0;
        uint32_t phase = 0u;
        while (next_task(x)) {
            const int era = x.era, f = x.fb * FC + fl;
            const bool mine = f < a.n_feat, empty_tile = x.b0 == x.b1;
            // the first and the last of a feature block in this CTA (where the flush makes the gains)
            const bool fresh = era == 0 || (era == s_cut[0][1] && x.fb == s_cut[0][0]), last = x.next == E || (x.next == s_cut[1][1] && x.fb == s_cut[1][0]);
            warp_wait<true>(acc_full + buf, phase, &s_fail);
            warp_wait<true>(tot_full + buf, phase, &s_fail);
            uint32_t* tot = s_tot + buf * 3 * tot_plane;
#pragma unroll 1                                 // (unrolled by four: 2 us a launch for the fetch of its instructions)
            for (int n = warp - kFlushWarp0; n < n_nodes; n += kFlushWarps) {
                uint32_t* at = tot + n * 32 + lane;
                uint32_t tc = at[0];
                long long tg = (long long)(int32_t)at[2 * tot_plane] * 65536ll + (long long)at[tot_plane];
                at[0] = at[tot_plane] = at[2 * tot_plane] = 0u;
                for (int d = 16; d > 0; d >>= 1) {
                    tc += __shfl_xor_sync(0xFFFFFFFFu, tc, d);
                    tg += __shfl_xor_sync(0xFFFFFFFFu, tg, d);
                }
                if (lane == 0) {
                    s_tc[n] = tc;
                    s_tgq[n] = tg;
                    if (FUSE) {
                        const EraTotals e = era_totals(tc, tg, inv_scale, z.lambda_l2, z.era_alpha);
                        s_era[n] = make_float4(e.tg, e.th, e.parent, e.w_era);
                    }
                }
            }
            meet(kFlushBarrier, 32 * kFlushWarps);
            tc_fence_after();
            const uint32_t from = tmem + ((uint32_t)quarter << 21) + (uint32_t)(buf * L * N_max);
            for (int n0 = U * fg; n0 < n_nodes; n0 += U * kFlushWarps / 4) {
                int raw[L][5][U];
#pragma unroll
                for (int l = 0; l < L; ++l)
#pragma unroll
                    for (int j = 0; j < 5; ++j)
#pragma unroll
                        for (int u = 0; u < U; ++u)
                            tmem_load1(from + (uint32_t)(l * N_max + (GROUPS ? (n0 + u) / 8 * 40 + (n0 + u) % 8 : 8 * (n0 + u)) + j * J), raw[l][j][u]);
                tmem_load_wait();
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int n = n0 + u;
                    if (n >= n_nodes) break;
                    uint32_t rc[L];
                    long long rg[L];
#pragma unroll
                    for (int l = 0; l < L; ++l) {
                        rc[l] = empty_tile ? 0u : (uint32_t)raw[l][4][u];
                        const int lo = raw[l][0][u] + raw[l][1][u] * 256, hi = raw[l][2][u] + raw[l][3][u] * 256;
                        rg[l] = empty_tile ? 0ll : (long long)hi * 65536ll + (long long)lo;
                    }
                    const uint32_t tc = s_tc[n];
                    const long long tgq = s_tgq[n];
                    if (FUSE) {
                        if (!mine) continue;
                        const float4 e = s_era[n];
                        const size_t at = (((size_t)f * a.n_eras + era) * a.node_stride + n) * K;
                        const int pa = z.agree ? parent_direction(z.frontier[n].gq) : 0;
                        float2 gain[L];
#pragma unroll
                        for (int l = 0; l < L; ++l) {
                            const int k = z.full_sweep ? g * L + l : s_kof[g * L + l];
                            const uint32_t lc = tc - rc[l];
                            const long long lgq = tgq - rg[l];
                            gain[l] = gain_of(lc, lgq, tc, e.x, e.y, e.z, inv_scale, z.lambda_l2, e.w);
                            if (k < 0 || k >= K) continue;
                            const int own = (n * L + l) * 128 + row;
                            s_lc[own] = fresh ? lc : s_lc[own] + lc;
                            s_lg[own] = fresh ? lgq : s_lg[own] + lgq;
                            if (last) {
                                const size_t tot_at = ((size_t)n * K + k) * lanes_total + f;
                                if (s_lc[own]) atomicAdd(z.lc_tot + tot_at, s_lc[own]);
                                if (s_lg[own]) atomicAdd(reinterpret_cast<unsigned long long*>(z.lg_tot + tot_at), (unsigned long long)s_lg[own]);
                            }
                            if (z.agree)
                                z.agree[at + k] = (uint8_t)agree_code(lc, lgq, e.x, e.y, inv_scale, z.lambda_l2, z.direction_form, pa);
                        }
                        float2* out = z.gw + at;
                        if (L > 1 && z.full_sweep && (K & 1) == 0) {   // rows of an even K start on 16 bytes
#pragma unroll
                            for (int l = 0; l < L; l += 2)
                                if (g * L + l < K)
                                    *reinterpret_cast<float4*>(out + g * L + l) = make_float4(gain[l].x, gain[l].y, gain[(l + 1) % L].x, gain[(l + 1) % L].y);
                        } else {
#pragma unroll
                            for (int l = 0; l < L; ++l) {
                                const int k = z.full_sweep ? g * L + l : s_kof[g * L + l];
                                if (k >= 0 && k < K) out[k] = gain[l];
                            }
                        }
                    } else {
                        // bin t + 1 is what lies right of threshold t but not of t + 1; the next lane holds the
                        // threshold after this lane's last
                        const uint32_t nc = __shfl_down_sync(0xFFFFFFFFu, rc[0], 1);
                        const long long ng = __shfl_down_sync(0xFFFFFFFFu, rg[0], 1);
                        if (!mine) continue;
                        const size_t o = (((size_t)f * a.n_eras + era) * a.node_stride + n) * a.max_bins;
                        auto put = [&](int bin, uint32_t c, long long s) {
                            if (c) atomicAdd(a.cnt + o + bin, c);
                            if (s) atomicAdd(reinterpret_cast<unsigned long long*>(a.gsum + o + bin), (unsigned long long)s);
                        };
                        if (g == 0) put(0, tc - rc[0], tgq - rg[0]);
#pragma unroll
                        for (int l = 0; l < L; ++l) {
                            const int bin = g * L + l + 1;
                            if (bin >= a.max_bins) break;
                            const bool last = l == L - 1;
                            const uint32_t c1 = last ? (g == G - 1 ? 0u : nc) : rc[(l + 1) % L];
                            const long long g1 = last ? (g == G - 1 ? 0ll : ng) : rg[(l + 1) % L];
                            put(bin, rc[l] - c1, rg[l] - g1);
                        }
                    }
                }
                __syncwarp();
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(acc_empty + buf);
            if (++buf == a.buffers) { buf = 0; phase ^= 1u; }
            meet(kFlushBarrier, 32 * kFlushWarps);             // the nodes' totals are read
        }
    } else if (warp < kIssueWarp) {
        // ---- B: a row of two K-steps of each batch ----
        const int wg = (warp - kRowWarp0) >> 1, half = (warp - kRowWarp0) & 1;
        constexpr int kMine = kBatch / 2;
        auto first_unit = [&](int b) { return (int)((uint32_t)(wg + kSlots * kUnits - (b * kUnits) % kSlots) % kSlots); };
        constexpr uint32_t J = GROUPS ? 256u : 16u;  // bytes between the digits of a node
        const uint32_t to = smem_at(s_b) + (uint32_t)(wg * batch_bytes + half * kMine * k_bytes + (lane >> 4) * 128 + (lane & 15));
        uint32_t held[kMine];                        // where these rows' bytes of the last turn lie, 0: none
#pragma unroll
        for (int k = 0; k < kMine; ++k) held[k] = 0u;
        int stage = 0, buf = 0;
        uint32_t turn = 0u, c_phase = 0u, acc_phase = 1u;   // (turn: how often this place was handed over)
        while (next_task(x)) {
            warp_wait(acc_empty + buf, acc_phase, &s_fail);   // the totals of this buffer are zero
            uint32_t* tot = s_tot + buf * 3 * tot_plane + lane;
            for (int b = x.b0; b < x.b1; ++b) {
                bool met = false;
#pragma unroll 1
                for (int u = first_unit(b); u < kUnits; u += kSlots) {
                    const int i = u * kBatchRows, r = b * kBlock + i;
                    if (r + kBatchRows <= x.r0 || r >= x.r1) continue;
                    // the two warps wait for the six of a slot, one for the codes, one for the operands' place
                    if (half != 0) {
                        warp_wait(empty + wg, ~turn & 1u, &s_fail);
                        if (s_fail) {        // a place is not handed over again before all took it
                            const volatile uint32_t* taken = s_taken + wg;
#pragma unroll 1
                            for (int i = 0; i < kTries && *taken != turn * kIssueWarps; ++i) __nanosleep(1000);
                            __syncwarp();
                        }
                    } else if (!met) {
                        warp_wait(full_c + stage, c_phase, &s_fail);
                    }
                    met = true;
                    meet(kSlotBarrier + wg, kSlotThreads);
                    ++turn;
                    const unsigned char* rows = s_codes + stage * stage_bytes + FC * kPitch;
                    const int mine = i + half * kMine * 32 + lane;
                    uint32_t s[kMine], q[kMine];
#pragma unroll
                    for (int k = 0; k < kMine; ++k) {
                        s[k] = reinterpret_cast<const uint16_t*>(rows)[mine + 32 * k];
                        q[k] = reinterpret_cast<const uint32_t*>(rows + kBlock * 2)[mine + 32 * k];
                    }
#pragma unroll
                    for (int k = 0; k < kMine; ++k)
                        if (held[k] != 0u) {
#pragma unroll
                            for (int j = 0; j < 5; ++j) sts8(held[k] + j * J, 0u);
                        }
#pragma unroll
                    for (int k = 0; k < kMine; ++k) {
                        const int row = b * kBlock + mine + 32 * k;
                        const bool ok = row >= x.r0 && row < x.r1 && s[k] < (uint32_t)n_nodes;
                        held[k] = 0u;
                        if (ok) {
                            const uint32_t digits = (q[k] + 0x00808080u) ^ 0x00808080u;   // signed base 256
                            const uint32_t now = to + (uint32_t)(k * k_bytes) + (GROUPS ? (s[k] >> 3) * 1280u + (s[k] & 7u) * 16u : s[k] * 256u);
#pragma unroll
                            for (int j = 0; j < 4; ++j) sts8(now + j * J, digits >> (8 * j));
                            sts8(now + 4 * J, 1u);
                            held[k] = now;
                            atomicAdd(tot + s[k] * 32, 1u);
                            atomicAdd(tot + tot_plane + s[k] * 32, q[k] & 0xFFFFu);
                            atomicAdd(reinterpret_cast<int*>(tot) + 2 * tot_plane + s[k] * 32, (int)q[k] >> 16);
                        }
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    hand_over(wg, kIssueWarps);
                }
                if (!met) {
                    if (half == 0) warp_wait(full_c + stage, c_phase, &s_fail);
                    meet(kSlotBarrier + wg, kSlotThreads);
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(empty_c + stage);
                if (++stage == kStages) { stage = 0; c_phase ^= 1u; }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(tot_full + buf);
            if (++buf == a.buffers) { buf = 0; acc_phase ^= 1u; }
        }
    } else if (warp < kCopyWarp0) {
        // ---- products ----
        const int n1 = WIDE ? min(N, 256) : N, n2 = max(N - n1, 16);   // (of a narrower frontier: columns nobody reads)
        const uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | (8u << 24);   // s32 += s8 * s8, M 128
        const uint32_t idesc1 = idesc | ((uint32_t)(n1 >> 3) << 17), idesc2 = idesc | ((uint32_t)(n2 >> 3) << 17);
        // K-major, no swizzle: 8 x 16-byte core matrices, the two of a K-step 128 bytes apart, eight columns 256
        const uint32_t desc_lo = (smem_at(s_b) >> 4) | (uint32_t)(128 >> 4) << 16, desc_hi = (uint32_t)(256 >> 4) | 1u << 14;
        const uint32_t k16 = (uint32_t)k_bytes >> 4;
        const int first = (warp - kIssueWarp) * kTilesOf;    // of this warp's accumulators
        int buf = 0;
        uint32_t acc_phase = 1u;
        while (next_task(x)) {
            warp_wait(acc_empty + buf, acc_phase, &s_fail);
            uint32_t add = 0u;
            const int u0 = x.r0 / kBatchRows, u1 = x.r0 < x.r1 ? (x.r1 + kBatchRows - 1) / kBatchRows : u0;
            int slot = u0 % kSlots;
            bool lives = s_fail == 0;
            for (int u = u0; u < u1; ++u) {
                asm volatile("barrier.cta.sync.aligned %0, %1;" ::"r"(kFullBarrier + slot), "r"(kSlotThreads + 32 * kIssueWarps) : "memory");
                tc_fence_after();
                if (lane == 0) atomicAdd(s_taken + slot, 1u);
                if (elect_one() && lives) {
                    const uint32_t lo = desc_lo + (uint32_t)(slot * kBatch) * k16, at0 = a_col + (uint32_t)((slot * kBatch * L + first) * 8);
                    const uint32_t d0 = tmem + (uint32_t)((buf * L + first) * N_max);
#pragma unroll
                    for (int k = 0; k < kBatch; ++k) {
                        const uint64_t dk = (uint64_t)desc_hi << 32 | (lo + k * k16);
#pragma unroll
                        for (int l = 0; l < kTilesOf; ++l) {
                            const uint32_t at = at0 + (uint32_t)((k * L + l) * 8), d = d0 + (uint32_t)(l * N_max);
                            mma_i8(d, at, dk, idesc1, k > 0 ? 1u : add);
                            if (WIDE) mma_i8(d + 256u, at, dk + (256 * 32 >> 4), idesc2, k > 0 ? 1u : add);
                        }
                    }
                    tc_commit(empty + slot);
                }
                __syncwarp();
                add = 1u;
                if (++slot == kSlots) slot = 0;
                lives = s_fail == 0;
            }
            if (elect_one() && lives) tc_commit(acc_full + buf);
            __syncwarp();
            if (++buf == a.buffers) { buf = 0; acc_phase ^= 1u; }
        }
    } else {
        // ---- codes, frontier slots and gradients of a block; eight consecutive threads per line ----
        const int cw = warp - kCopyWarp0;
        constexpr int kMine = (128 / 2 + kCopyWarps - 1) / kCopyWarps;   // features of a half warp at most
        const uint32_t pitch = (uint32_t)a.pitch;    // (of fewer than 2^31 rows)
        const int part = lane & 15;
        int stage = 0;
        uint32_t phase = 1u;
        while (next_task(x)) {
            uint32_t rows[kMine];
#pragma unroll
            for (int i = 0; i < kMine; ++i) {
                const int fl = (i * kCopyWarps + cw) * 2 + (lane >> 4);
                rows[i] = fl < FC ? (uint32_t)a.feat_rows[min(x.fb * FC + fl, a.n_feat - 1)] : 0u;
            }
            for (int b = x.b0; b < x.b1; ++b) {
                warp_wait(empty_c + stage, phase, &s_fail);
                const uint32_t to = smem_at(s_codes + stage * stage_bytes);
                const int64_t column = (int64_t)b * (kBlock / 2) + part * 16;
                if (column < a.pitch) {              // (a row is padded to whole lines, not to whole blocks)
                    const uint8_t* base = a.codes + column;
                    const uint32_t mine = to + (uint32_t)((2 * cw + (lane >> 4)) * kPitch + part * 16);
#pragma unroll
                    for (int i = 0; i < kMine; ++i)
                        if ((i * kCopyWarps + cw) * 2 < FC) copy16(mine + (uint32_t)(2 * kCopyWarps * i * kPitch), base + (uint64_t)rows[i] * pitch);
                }
                const uint32_t state = to + (uint32_t)(FC * kPitch);
                const int64_t row0 = (int64_t)b * kBlock;
                for (int i = cw * 32 + lane; i < kBlock * 6 / 16; i += 32 * kCopyWarps) {   // slots, then gradients
                    const bool g = i >= kBlock / 8;
                    const int64_t row = row0 + (g ? (i - kBlock / 8) * 4 : i * 8);
                    if (row < a.rows_pad) copy16(state + (uint32_t)(i * 16), g ? (const void*)(a.gq + row) : (const void*)(a.slot + row));
                }
                asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_at(full_c + stage)) : "memory");
                if (++stage == kStages) { stage = 0; phase ^= 1u; }
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    }
    __syncwarp();
    __syncthreads();
    if (s_fail) {                            // what has been issued ends before the tensor memory goes
        if (a.flags && threadIdx.x == 0) atomicOr(a.flags, kFaultWait);
        if (warp >= kIssueWarp && warp < kCopyWarp0) {
            if (elect_one()) tc_commit(&last);
            __syncwarp();
            int never = 0;
            mbar_wait(&last, 0u, &never);
        }
        __syncthreads();
    }
    tc_fence_after();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(kColumns));
}

struct MmaShape {
    int thresholds_per_lane, batch, groups, features, buffers;
    size_t smem;
};

MmaShape mma_shape(int n_nodes, int n_feat, int max_bins, bool fused) {
    MmaShape s;
    const int N = mma_columns(n_nodes, mma_groups(n_nodes)), L = mma_per_lane(n_nodes, n_feat, max_bins);
    s.thresholds_per_lane = L;
    s.batch = n_nodes > 2 && L == 4 ? 2 : 4;
    s.groups = mma_thresholds(max_bins) / L;
    s.features = mma_features(n_nodes, n_feat, max_bins);
    const int operands = kSlots * s.batch * L * 8;
    s.buffers = 2 * L * N + operands <= kColumns ? 2 : 1;
    const size_t sums = fused ? (size_t)n_nodes * L * 128 * 12 : 0;
    const size_t fixed = (size_t)kSlots * s.batch * N * 32 + sums + (size_t)s.buffers * n_nodes * 32 * 12;
    s.smem = fixed + (size_t)kStages * mma_stage_bytes(s.features);   // (183 KB at most: 64 nodes)
    return s;
}

template <int L, int KB, bool GROUPS, bool WIDE>
int launch_l(const MmaArgs& a, dim3 grid, size_t smem, cudaStream_t stream) {
    if (a.fuse && !WIDE) {
        PB_TRY(allow_shared(hist_mma_kernel<L, KB, GROUPS, false, true>, smem));
        hist_mma_kernel<L, KB, GROUPS, false, true><<<grid, mma_threads(GROUPS, L), smem, stream>>>(a);
    } else {
        PB_TRY(allow_shared(hist_mma_kernel<L, KB, GROUPS, WIDE, false>, smem));
        hist_mma_kernel<L, KB, GROUPS, WIDE, false><<<grid, mma_threads(GROUPS, L), smem, stream>>>(a);
    }
    return PB_OK;
}

}  // namespace

// PACKBOOST_HIST_MMA=0 / 1: nowhere / wherever it can (and a line for each launch), for comparisons.
static int forced_mma() {
    static const int forced = [] {
        const char* e = getenv("PACKBOOST_HIST_MMA");
        if (getenv("PACKBOOST_HIST_SHAPE")) return 0;   // (a shape of the other kernel is asked for)
        return (e && (e[0] == '0' || e[0] == '1') && e[1] == 0) ? e[0] - '0' : -1;
    }();
    return forced;
}

bool hist_mma_takes(const HistLaunch& h) {
#ifdef PB_DEBUG_BOUNDS
    return false;   // codes are no index here: the build that checks them keeps to the kernel where they are
#else
    const bool fused = h.fuse != nullptr, tiled = h.max_era_rows > kTileRowsMax;
    if (forced_mma() == 0 || h.code_bits != 4 || h.max_bins > 8 || h.n_nodes > (fused ? 32 : 64) || fused == tiled) return false;
    if (forced_mma() == 1) return true;
    return mma_pays(fused, h.n_nodes, h.n_feat, h.max_bins, h.n_rows, h.n_eras);
#endif
}

int launch_hist_mma(const HistLaunch& h, cudaStream_t stream) {
    const MmaShape s = mma_shape(h.n_nodes, h.n_feat, h.max_bins, h.fuse != nullptr);
    MmaArgs a;
    memset(&a, 0, sizeof(a));
    a.codes = h.codes;
    a.pitch = h.pitch;
    a.feat_rows = h.feat_rows;
    a.n_feat = h.n_feat;
    a.gq = h.gq;
    a.slot = h.slot;
    a.era_offsets = h.era_offsets;
    a.rows_pad = h.rows_pad;
    a.n_eras = h.n_eras;
    a.max_bins = h.max_bins;
    a.n_nodes_ptr = h.n_nodes_ptr;
    a.n_nodes = h.n_nodes;
    a.node_stride = h.node_stride;
    a.cnt = h.cnt;
    a.gsum = h.gsum;
    a.flags = h.debug_flags;
    a.groups = s.groups;
    a.buffers = s.buffers;
    static const int failed = [] {   // PACKBOOST_WAIT_FAILS=1: launches go the way of a wait that ran out, for the test of it
        const char* e = getenv("PACKBOOST_WAIT_FAILS");
        return (e && e[0] == '1' && e[1] == 0) ? 1 : 0;
    }();
    a.failed = failed;
    const int blocks = (h.n_feat + s.features - 1) / s.features;
    if (!h.fuse && !h.zeroed) {
        const size_t cells = (size_t)h.n_feat * h.node_stride * h.n_eras * h.max_bins;
        PB_CUDA_TRY(cudaMemsetAsync(h.cnt, 0, cells * sizeof(uint32_t), stream));
        PB_CUDA_TRY(cudaMemsetAsync(h.gsum, 0, cells * sizeof(int64_t), stream));
    }
    if (h.fuse) {
        a.fuse = 1;
        h.fuse->tot_fpl = 1;
        h.fuse->tot_lanes = blocks * s.features;
        a.fz = *h.fuse;
        if (!h.zeroed) {
            const size_t tot = (size_t)h.node_stride * a.fz.n_thr * a.fz.tot_lanes;
            PB_CUDA_TRY(cudaMemsetAsync(a.fz.lc_tot, 0, tot * sizeof(uint32_t), stream));
            PB_CUDA_TRY(cudaMemsetAsync(a.fz.lg_tot, 0, tot * sizeof(int64_t), stream));
        }
    }
    a.blocks = blocks;
    // An era costs its flush too, more than its rows where it is short: about 1 200 to 3 300 rows' time by the number of
    // nodes, most of it beside the rows of the next one.
    a.era_rows = !h.fuse ? 0 : h.n_nodes > 8 || h.n_rows < (int64_t)1500 * h.n_eras ? 2048 : 512;
    const int64_t most = (int64_t)blocks * (h.fuse ? h.n_eras : tiles_of(h.n_rows, kCutRows));
    // (A CTA with rows of two feature blocks adds two tiles to a stored histogram: 160 000 rows x 78 features, 64 nodes:
    // 51 us, 36 with blocks of their own.)
    a.shares = shares_of(blocks, h.n_rows + (int64_t)a.era_rows * h.n_eras, (int)(most < 148 ? most : 148), !h.fuse);
    const dim3 grid((unsigned)a.shares.count);
    if (s.smem > kSharedMost) return fail_arg("histogram of %d nodes does not fit shared memory", h.n_nodes);
    if (forced_mma() == 1)
        fprintf(stderr, "hist_mma_kernel<%d,%d,%d,%d> fused=%d nodes=%d features=%d blocks=%d buffers=%d\n", s.thresholds_per_lane, s.batch,
                (int)mma_groups(h.n_nodes), (int)(s.thresholds_per_lane == 1 && mma_columns(h.n_nodes, true) > 256), a.fuse, h.n_nodes, h.n_feat,
                blocks, s.buffers);
    prof_begin(h.prof, kProfHist, stream);
    const int rc = s.thresholds_per_lane == 4 ? (s.batch == 4 ? launch_l<4, 4, false, false>(a, grid, s.smem, stream) : launch_l<4, 2, false, false>(a, grid, s.smem, stream))
                   : s.thresholds_per_lane == 2 ? (mma_groups(h.n_nodes) ? launch_l<2, 4, true, false>(a, grid, s.smem, stream) : launch_l<2, 4, false, false>(a, grid, s.smem, stream))
                                                : mma_columns(h.n_nodes, true) <= 256 ? launch_l<1, 4, true, false>(a, grid, s.smem, stream)
                                                : launch_l<1, 4, true, true>(a, grid, s.smem, stream);
    prof_end(h.prof, kProfHist, stream);
    if (rc) return rc;
    count_launch(1);
    PB_LAUNCH_CHECK("hist_mma_kernel");
    return PB_OK;
}

}  // namespace pb
