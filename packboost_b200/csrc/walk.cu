// Histogram and scorer of one depth in one kernel, for tables of many bins (8-bit codes).
//
// With more than 16 bins a stored histogram is the largest thing a depth moves: 12 bytes per
// (feature, era, node, bin) written and read back, then 8 bytes per threshold of (gain, weight) written
// and read again - 13 GB for one round of 500 000 rows, 256 features, 100 eras, 128 bins and depth 6,
// against 0.9 GB of codes and row state.  None of it outlives its era: the score of a threshold is a
// Welford recursion over the eras in ascending order.  So a CTA owns one feature and a group of frontier
// nodes and walks the eras; the state of the recursion stays in registers to the end, and what leaves the
// CTA is one candidate per node.  Two forms: with fewer nodes than warps the eras go by in batches
// (walk_kernel), from sixteen nodes on a warp owns a node (walk_nodes_kernel, further down).
//
// Cells are the two words of the histogram kernel (sum of low gradient bits << CB | count, sum of high
// bits).  A batch is an (era, node) pair per warp, as many eras at one node as there are warps: (a) all warps add the rows of the batch to its cells; (b) a warp per pair scans the bins (a
// lane per BPL consecutive ones), computes the gains and leaves them in shared memory; (c) a thread per
// threshold advances the recursion through the eras of the batch.  So the latency of the scan, its
// shuffles and divisions, is paid once a batch by all warps side by side.  An era of more rows than
// the count field holds is cut into tiles whose prefix sums are added up before (b) goes on.
//
// Divisions: every divisor of the gains is count + lambda, so an era's divisors and their correctly
// rounded reciprocals come from a table in shared memory, and a quotient takes two corrected products
// instead of a general division (divide.cuh).
//
// Bound: with few nodes the rows (two shared-memory atomics per row and feature take 3.5 wavefronts each
// with 128 bins, 66 % of the shared-memory pipe; without them, or with rows from the L1, they still take 85 %
// of the time: no one thing), with many the gains (issue slots 60 to 64 %).
// 500 000 rows x 256 features, 100 eras, 128 bins, by depth: 0.22, 0.24, 0.29, 0.39, 0.41, 0.62 ms, 2.2 ms a
// round (one form for all depths: 0.50 and 1.01 ms at the last two, 2.7 ms; histogram, gain and chain kernels:
// 4.6); 200 000 x 100, 40 eras, depth 10: 3.0 ms a round (4.8 with the one form), of which 512 nodes 1.23 (2.07).
//
// Float arithmetic as in the scorer: the same separately rounded operations in the same order
// (this file is compiled with -fmad=false), so candidates are bit-identical to the other path's.

#include <stdio.h>
#include <stdlib.h>

#include "common.cuh"
#include "des_math.cuh"
#include "divide.cuh"
#include "rows.cuh"

namespace pb {

namespace {

constexpr int kWalkInv = 4096;           // longest table of era reciprocals

// Four codes, each within the cells of its node (32 BPL of them) whatever the byte: one that is no bin would else be
// counted in another node's cells, or add a sum to counts, which index the table of divisors.
template <int BPL>
__device__ __forceinline__ uint32_t cells_of(uint32_t codes) {
#ifdef PB_DEBUG_BOUNDS
    return codes;                        // (each is looked at where it is used)
#else
    return BPL < 8 ? codes & (uint32_t)(32 * BPL - 1) * 0x01010101u : codes;
#endif
}

struct RowGroup {                        // four consecutive rows
    uint32_t codes;
    uint2 slots;
    int4 gq;
};

__device__ __forceinline__ float sign3(float v) { return v > 0.f ? 1.f : (v < 0.f ? -1.f : v); }

__device__ __forceinline__ float divide_by(float a, float2 dy) { return pb::divide_by(a, dy.x, dy.y); }

// Thresholds of one feature at the count-mass quantiles of its bins over all frontier rows, as the
// reference's compiled split finder takes them (packboost/backends/cpu/frontier_cpu.cpp:35-109): targets
// i / (k - 1) of total * (1 - 1e-12) in float64, a threshold one below the first bin whose cumulative
// mass reaches the target, evenly spaced ids when targets coincide, the k smallest.  Called by all
// threads; s_m: bin masses (cumulated here), s_set: 0 / 1 per bin on return.
__device__ void mass_cut_set(uint32_t* s_m, uint8_t* s_set, int nb, int K) {
    const int max_thr = max(1, nb - 1), kk = max(1, min(K, max_thr));
    const int lane = threadIdx.x & 31;
    __shared__ int s_have;
    if (threadIdx.x < 32) {              // inclusive prefix of up to 256 masses, eight per lane
        uint32_t v[8], run = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            run += (lane * 8 + j < nb) ? s_m[lane * 8 + j] : 0u;
            v[j] = run;
        }
        uint32_t incl = run;
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t up = __shfl_up_sync(0xFFFFFFFFu, incl, d);
            if (lane >= d) incl += up;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (lane * 8 + j < nb) s_m[lane * 8 + j] = v[j] + incl - run;
    }
    for (int b = threadIdx.x; b < 256; b += blockDim.x) s_set[b] = 0;
    if (threadIdx.x == 0) s_have = 0;
    __syncthreads();
    const uint32_t total = s_m[nb - 1];
    if (total > 0) {
        const double upper = (double)total * (1.0 - 1e-12);
        for (int i = threadIdx.x; i < kk; i += blockDim.x) {
            const double alpha = (kk == 1) ? 0.0 : (double)i / (double)(kk - 1);
            const double target = upper * alpha;
            int idx = nb - 1;
            for (int b = 0; b < nb; ++b)
                if (!((double)s_m[b] < target)) {
                    idx = b;
                    break;
                }
            s_set[max(0, min(idx - 1, max_thr - 1))] = 1;
        }
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        int have = 0;
        for (int b = lane; b < max_thr; b += 32) have += s_set[b];
        have = __reduce_add_sync(0xFFFFFFFFu, have);
        if (lane == 0) s_have = have;
    }
    __syncthreads();
    if (s_have < kk) {
        if (kk == 1) {
            if (threadIdx.x == 0) s_set[0] = 1;
        } else {
            const double step = (double)(max_thr - 1) / (double)(kk - 1);
            for (int i = threadIdx.x; i < kk; i += blockDim.x) {
                const long long idx = llround(round((double)i * step));
                s_set[(int)max(0ll, min(idx, (long long)max_thr - 1))] = 1;
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) {          // (more than k ids now: the k smallest stay)
            int w = 0;
            for (int b = 0; b < max_thr; ++b)
                if (s_set[b] && ++w > kk) s_set[b] = 0;
        }
    }
    __syncthreads();
}

// Bin masses of the frontier rows of each feature: counts[f][256] += .  grid (feature, row part).
__global__ void __launch_bounds__(256) mass_count_kernel(WalkLaunch a) {
    __shared__ uint32_t s_m[8][257];
    for (int i = threadIdx.x; i < 8 * 257; i += 256) (&s_m[0][0])[i] = 0u;
    __syncthreads();
    const int n_nodes = min(*a.n_nodes_ptr, a.n_nodes);
    const int warp = threadIdx.x >> 5;
    const uint8_t* codes = a.codes + (int64_t)a.feat_rows[blockIdx.x] * a.pitch;
    // (rows past the end have no slot; the row arrays are padded)
    for (int64_t g = blockIdx.y * 256 + threadIdx.x; 4 * g < a.n_rows; g += gridDim.y * 256) {
        const uint32_t c = *reinterpret_cast<const uint32_t*>(codes + 4 * g);
        const uint2 s = *reinterpret_cast<const uint2*>(a.slot + 4 * g);
        const uint32_t sl[4] = {s.x & 0xFFFFu, s.x >> 16, s.y & 0xFFFFu, s.y >> 16};
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if ((int)sl[j] < n_nodes) atomicAdd(&s_m[warp][(c >> (8 * j)) & 0xFFu], 1u);
    }
    __syncthreads();
    uint32_t t = 0;
    for (int w = 0; w < 8; ++w) t += s_m[w][threadIdx.x];
    if (t) atomicAdd(a.mass + (size_t)blockIdx.x * 256 + threadIdx.x, t);
}

// What the state of a threshold has to hold (its registers decide how many CTAs an SM takes).
constexpr int kUnit = 0;       // era weights 0 / 1, an era is one tile
constexpr int kUnitTiles = 1;  // era weights 0 / 1, eras of several tiles
constexpr int kGeneral = 2;    // any weights, directional term, any eras

// W neighbouring words of a lane, in as few accesses as they take.
template <int W>
__device__ __forceinline__ void take_words(uint32_t* at, uint32_t (&v)[W]) {  // reads, leaves zeros
    if (W >= 4) {
#pragma unroll
        for (int i = 0; i < W; i += 4) {
            const uint4 q = *reinterpret_cast<const uint4*>(at + i);
            v[i] = q.x; v[(i + 1) % W] = q.y; v[(i + 2) % W] = q.z; v[(i + 3) % W] = q.w;
        }
#pragma unroll
        for (int i = 0; i < W; i += 4) *reinterpret_cast<uint4*>(at + i) = make_uint4(0u, 0u, 0u, 0u);
    } else if (W == 2) {
        const uint2 q = *reinterpret_cast<const uint2*>(at);
        v[0] = q.x; v[1 % W] = q.y;
        *reinterpret_cast<uint2*>(at) = make_uint2(0u, 0u);
    } else {
        v[0] = *at;
        *at = 0u;
    }
}

// Shared memory: cells [pairs + 1][NBP][copies] word A, then word B | gains [pairs][NBP] | agreement [pairs][NBP]
// (kGeneral) or 1 / n [eras + 1] | (divisor, reciprocal) [largest era + 1] when an era is one tile.
// A pair's gains lie at i * 32 + lane for bin lane * BPL + i.  COPIES: interleaved copies of the cells.
// WARPS: of a CTA, and (era, node) pairs of a batch and most nodes of a CTA.
template <int BPL, int MODE, int COPIES, int WARPS>
__global__ void __launch_bounds__(32 * WARPS, (BPL <= 4 && MODE != kGeneral && WARPS == 16) ? 2 : 1) walk_kernel(WalkLaunch a) {
    constexpr int kWalkThreads = 32 * WARPS, kWalkNodes = WARPS;
    constexpr bool UNIT = MODE != kGeneral, TILES = MODE != kUnit;
    constexpr int NBP = 32 * BPL;        // bins of a pair's cells
    constexpr int SLOTS = kWalkNodes * NBP / kWalkThreads;   // thresholds a thread may own
    constexpr int plane = kWalkNodes * NBP;
    constexpr int words = (plane + NBP) * COPIES;            // of word A, rows nobody counts included; word B follows
    extern __shared__ __align__(16) uint32_t s_cells[];      // [pairs][NBP][COPIES]
    float2* s_gain = reinterpret_cast<float2*>(s_cells + 2 * words);
    float* s_agree = reinterpret_cast<float*>(s_gain + plane);
    float* s_inv = s_agree;
    float2* s_div = reinterpret_cast<float2*>(s_agree + (UNIT ? (a.n_eras + 2) / 2 * 2 : plane));
    __shared__ uint32_t s_mass[256];
    __shared__ uint8_t s_set[256];
    __shared__ int s_off[kWalkNodes + 2];                    // row ranges of the batch's eras
    const int n_nodes = min(*a.n_nodes_ptr, a.n_nodes);
    const int CN = a.cell_nodes;                             // nodes of a CTA at most: a power of two
    const int node0 = blockIdx.x * CN;
    const int live = min(CN, n_nodes - node0);
    if (live <= 0) return;
    const int f = blockIdx.y;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nb = a.max_bins, E = a.n_eras, K = a.n_thr;
    const int EB = TILES ? 1 : kWalkNodes / CN;              // eras of a batch
    const int CB = a.count_bits, LB = a.lo_bits;
    const uint32_t lo_mask = (1u << LB) - 1u, cmask = (1u << CB) - 1u;
    const float inv_scale = *a.inv_scale_ptr, lam = a.lambda_l2;
    const bool table = a.div_table && division_in_range(inv_scale, lam);

    for (int i = threadIdx.x; i < 2 * words; i += kWalkThreads) s_cells[i] = 0u;
    if (UNIT)
        for (int n = threadIdx.x; n <= E; n += kWalkThreads) s_inv[n] = n > 0 ? f_div(1.f, (float)n) : 0.f;
    if (table)
        for (int n = threadIdx.x; n <= a.max_era_rows; n += kWalkThreads) {
            const float d = f_add((float)n, lam);
            s_div[n] = make_float2(d, f_div(1.f, d));
        }

    // ---- which bins are thresholds ----
    if (a.mass) {
        for (int b = threadIdx.x; b < 256; b += kWalkThreads) s_mass[b] = a.mass[(size_t)f * 256 + b];
        __syncthreads();
        mass_cut_set(s_mass, s_set, nb, K);
    } else {
        for (int b = threadIdx.x; b < 256; b += kWalkThreads) s_set[b] = 0;
        __syncthreads();
        for (int k = threadIdx.x; k < K; k += kWalkThreads) s_set[a.thr_ids[k]] = 1;
        __syncthreads();
    }

    // ---- rows: a warp takes 128 consecutive rows, a lane four of them ----
    const uint8_t* codes = a.codes + (int64_t)a.feat_rows[f] * a.pitch;
    const bool sparse = gridDim.x > 2;   // most rows belong to other CTAs: gradients are read when a row is ours
    constexpr uint32_t PAIR = 4u * NBP * COPIES;             // bytes of a pair's cells
    const uint32_t cells_at = (uint32_t)__cvta_generic_to_shared(s_cells) + 4u * (threadIdx.x & (COPIES - 1));
    // Rows of other CTAs' nodes, and of none, go to cells of their own after the pairs', which nobody reads:
    // an address is chosen, nothing is predicated (a predicate costs a branch each way around the atomics;
    // 500 000 rows x 256 features, one node, rows alone: 204 us with predicates, 190 without)
    const uint32_t trash = cells_at + (uint32_t)kWalkNodes * PAIR;
    const uint32_t one_a = 1u << CB;
    auto load_group = [&](int c, RowGroup& x) {              // chunk c, 128 rows (the row arrays are padded to 256)
        const uint32_t g = 32u * (uint32_t)c + (uint32_t)lane;
        x.codes = reinterpret_cast<const uint32_t*>(codes)[g];
        x.slots = reinterpret_cast<const uint2*>(a.slot)[g];
        if (!sparse) x.gq = reinterpret_cast<const int4*>(a.gq)[g];
    };
    auto add_row = [&](uint32_t base, uint32_t n, uint32_t code, int q) {
#ifdef PB_DEBUG_BOUNDS
        const uint32_t sl = n + (uint32_t)node0;
        if ((sl & 0xFFFFu) != kSlotNone && (int)sl >= a.n_nodes && a.debug_flags) atomicOr(a.debug_flags, kDbgSlot);
        if (n < (uint32_t)live && code >= (uint32_t)nb) {
            if (a.debug_flags) atomicOr(a.debug_flags, kDbgCode);
            return;
        }
#endif
        const uint32_t at = (n < (uint32_t)live ? base + n * PAIR : trash) + code * (4u * COPIES);
        asm volatile("red.shared.add.u32 [%0], %1;\n red.shared.add.u32 [%0 + %3], %2;" ::"r"(at),
                     "r"(((uint32_t)q & lo_mask) * one_a + 1u), "r"(q >> LB), "n"(4 * words) : "memory");
    };
    // `e`, `lim`: era of the batch at the warp's last chunk and where that era ends (rows ascend)
    auto add_group = [&](int c, int r0, int r1, RowGroup& x, int& e, int& lim) {
        x.codes = cells_of<BPL>(x.codes);
        const int first = 128 * c;       // (the warp's: all lanes decide alike)
        if (!TILES)
            while (first >= lim) lim = s_off[++e + 1];
        const uint32_t n0 = (x.slots.x & 0xFFFFu) - (uint32_t)node0, n1 = (x.slots.x >> 16) - (uint32_t)node0;
        const uint32_t n2 = (x.slots.y & 0xFFFFu) - (uint32_t)node0, n3 = (x.slots.y >> 16) - (uint32_t)node0;
        if (sparse) {
            if (min(min(n0, n1), min(n2, n3)) >= (uint32_t)live) return;
            x.gq = reinterpret_cast<const int4*>(a.gq)[32 * c + lane];
        }
        const uint32_t step = (uint32_t)CN * PAIR;
        uint32_t here = cells_at + (TILES ? 0u : (uint32_t)e * step);
        if (first >= r0 && first + 128 <= (TILES ? r1 : lim)) {
            add_row(here, n0, x.codes & 0xFFu, x.gq.x);
            add_row(here, n1, __byte_perm(x.codes, 0u, 0x4441u), x.gq.y);
            add_row(here, n2, __byte_perm(x.codes, 0u, 0x4442u), x.gq.z);
            add_row(here, n3, x.codes >> 24, x.gq.w);
        } else {                         // rows of a neighbouring batch, or of several eras
            int ej = e, end = TILES ? r1 : lim;
            auto one = [&](int r, uint32_t n, uint32_t code, int q) {
                if (r < r0 || r >= r1) return;
                while (r >= end) {
                    end = s_off[++ej + 1];
                    here += step;
                }
                add_row(here, n, code, q);
            };
            const int r = first + 4 * lane;
            one(r, n0, x.codes & 0xFFu, x.gq.x);
            one(r + 1, n1, __byte_perm(x.codes, 0u, 0x4441u), x.gq.y);
            one(r + 2, n2, __byte_perm(x.codes, 0u, 0x4442u), x.gq.z);
            one(r + 3, n3, x.codes >> 24, x.gq.w);
        }
    };

    // ---- the warp's pair: node warp % CN, every EB-th era from warp / CN on ----
    const int my_node = warp & (CN - 1), my_era = warp / CN;
    const bool scans = my_node < live && my_era < EB;
    uint32_t lc_sum[BPL], pc[BPL], tc = 0u;
    long long lg_sum[BPL], pg[BPL], tg = 0ll;
#pragma unroll
    for (int i = 0; i < BPL; ++i) {
        lc_sum[i] = pc[i] = 0u;
        lg_sum[i] = pg[i] = 0ll;
    }
    const long long g_par = scans ? a.frontier[node0 + my_node].gq : 0ll;
    const bool use_dir = !UNIT && a.direction_weight != 0.f && (a.direction_form == 1 || *a.any_dir_ptr != 0);
    const float pa = g_par > 0 ? -1.f : (g_par < 0 ? 1.f : 0.f);  // sign(-G / (H + lambda))

    // ---- state of this thread's thresholds: slots t, t + 512, ... of [node][i * 32 + lane] ----
    float mean[SLOTS], m2[SLOTS], wsum[UNIT ? 1 : SLOTS], a_num[UNIT ? 1 : SLOTS], a_den[UNIT ? 1 : SLOTS];
    int n_valid[UNIT ? SLOTS : 1];
#pragma unroll
    for (int q = 0; q < SLOTS; ++q) {
        mean[q] = m2[q] = 0.f;
        if (UNIT) n_valid[q] = 0;
        else wsum[q] = a_num[q] = a_den[q] = 0.f;
    }
    const int n_slots = live * NBP;

    int e0 = 0, r0 = a.era_offsets[0], r1 = 0, ne = 0;       // eras [e0, e0 + ne), rows [r0, r1) of the batch
    auto batch_end = [&]() {
        ne = min(EB, E - e0);
        const int end = ne > 0 ? a.era_offsets[e0 + ne] : r0;
        r1 = TILES && end - r0 > a.tile_rows ? r0 + a.tile_rows : end;
        return TILES ? r1 >= end : true;                     // the batch completes its eras
    };
    bool complete = batch_end();
    if (threadIdx.x <= kWalkNodes) s_off[threadIdx.x] = a.era_offsets[min((int)threadIdx.x, E)];
    __syncthreads();                     // cells are zero; offsets and tables are there
    while (ne > 0) {
        // ---- (a) ----
        {
            int e = 0, lim = s_off[1], chunk = r0 / 128 + warp;
            const int chunks = (r1 + 127) / 128;             // (128 times a chunk past the last may leave 32 bits)
            RowGroup cur;                // the warp's next chunk of rows
            if (chunk < chunks) load_group(chunk, cur);
            for (; chunk < chunks; chunk += WARPS) {
                RowGroup x = cur;        // (two sets of registers in turn save the copy and spill elsewhere: 215 -> 228 us)
                if (chunk + WARPS < chunks) load_group(chunk + WARPS, cur);
                add_group(chunk, r0, r1, x, e, lim);
            }
        }
        const int n_eras_now = complete ? ne : 0;            // eras that (b) finishes
        if (complete) e0 += ne;
        r0 = r1;
        complete = batch_end();
        __syncthreads();                 // the cells are complete, (c) of the batch before is done
        if (threadIdx.x <= kWalkNodes) s_off[threadIdx.x] = a.era_offsets[min(e0 + (int)threadIdx.x, E)];

        // ---- (b) prefix over the bins; the packed words are added as they are (the rows behind them are
        //      distinct rows of a tile, so no field overflows) ----
        if (scans && (TILES || my_era < n_eras_now)) {
            uint32_t A[BPL], B[BPL];
            uint32_t* at = s_cells + (warp * NBP + lane * BPL) * COPIES;
            uint32_t wa[BPL * COPIES], wb[BPL * COPIES];
            take_words(at, wa);
            take_words(at + words, wb);
#pragma unroll
            for (int i = 0; i < BPL; ++i) {
                A[i] = wa[i * COPIES];
                B[i] = wb[i * COPIES];
#pragma unroll
                for (int c = 1; c < COPIES; ++c) {
                    A[i] += wa[i * COPIES + c];
                    B[i] += wb[i * COPIES + c];
                }
            }
#pragma unroll
            for (int i = 1; i < BPL; ++i) {
                A[i] += A[i - 1];
                B[i] += B[i - 1];
            }
            uint32_t sa = A[BPL - 1], sb = B[BPL - 1];
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t ua = __shfl_up_sync(0xFFFFFFFFu, sa, d), ub = __shfl_up_sync(0xFFFFFFFFu, sb, d);
                if (lane >= d) {
                    sa += ua;
                    sb += ub;
                }
            }
            const uint32_t ta = __shfl_sync(0xFFFFFFFFu, sa, 31), tb = __shfl_sync(0xFFFFFFFFu, sb, 31);
            sa -= A[BPL - 1];
            sb -= B[BPL - 1];
            tc = (TILES ? tc : 0u) + (ta & cmask);
            tg = (TILES ? tg : 0ll) + (long long)(int32_t)tb * (1ll << LB) + (long long)(ta >> CB);
            if (TILES) {
#pragma unroll
                for (int i = 0; i < BPL; ++i) {
                    const uint32_t av = A[i] + sa, bv = B[i] + sb;
                    pc[i] += av & cmask;
                    pg[i] += (long long)(int32_t)bv * (1ll << LB) + (long long)(av >> CB);
                }
            }
            if (!TILES || n_eras_now > 0) {
                float2* out = s_gain + warp * NBP + lane;
                const float w_era = (tc == 0u) ? 0.f : (a.era_alpha > 0.f ? f_add((float)tc, a.era_alpha) : 1.f);
                const float tgf = f_mul(__ll2float_rn(tg), inv_scale);
                // (the operations of era_totals and gain_of, divisions by the table)
                const float parent = table ? divide_by(f_mul(0.5f, f_mul(tgf, tgf)), s_div[tc])
                                           : f_div(f_mul(0.5f, f_mul(tgf, tgf)), f_add((float)tc, lam));
#pragma unroll
                for (int i = 0; i < BPL; ++i) {              // (a threshold at a time: few registers)
                    const uint32_t av = A[i] + sa, bv = B[i] + sb, lc = TILES ? pc[i] : av & cmask, rc = tc - lc;
                    const long long lgq = TILES ? pg[i] : (long long)(int32_t)bv * (1ll << LB) + (long long)(av >> CB);
                    lc_sum[i] += lc;
                    lg_sum[i] += lgq;
                    const float lg = f_mul(__ll2float_rn(lgq), inv_scale), rg = f_sub(tgf, lg);
                    const float ll = f_mul(lg, lg), rr = f_mul(rg, rg);
                    const float dl = f_add((float)lc, lam), dr = f_add(f_sub((float)tc, (float)lc), lam);
                    const float ql = table ? divide_by(ll, s_div[lc]) : f_div(ll, dl);
                    const float qr = table ? divide_by(rr, s_div[rc]) : f_div(rr, dr);
                    out[i * 32] = make_float2(f_sub(f_mul(0.5f, f_add(ql, qr)), parent), (lc > 0u && rc > 0u) ? w_era : 0.f);
                    if (use_dir) {
                        const float vl = f_div(-lg, dl), vr = f_div(-rg, dr);
                        s_agree[warp * NBP + i * 32 + lane] = a.direction_form == 1
                            ? (vl > vr ? 1.f : -1.f)
                            : f_mul(0.5f, f_add(sign3(vl) == pa ? 1.f : 0.f, sign3(vr) == pa ? 1.f : 0.f));  // (an absent era has weight 0)
                    }
                    if (TILES) {
                        pc[i] = 0u;
                        pg[i] = 0ll;
                    }
                }
                if (TILES) {
                    tc = 0u;
                    tg = 0ll;
                }
            }
        }
        __syncthreads();                 // gains are there, cells are zero, offsets are the next batch's

        // ---- (c) recursion ----
#pragma unroll
        for (int q = 0; q < SLOTS; ++q) {
            const int s = threadIdx.x + q * kWalkThreads;
            if (s >= n_slots) break;
            for (int e = 0; e < n_eras_now; ++e) {
                const float2 gw = s_gain[(e * CN) * NBP + s];
                float fac, w;
                if (UNIT) {
                    w = gw.y > 0.f ? 1.f : 0.f;
                    n_valid[q] += gw.y > 0.f ? 1 : 0;
                    fac = gw.y > 0.f ? s_inv[n_valid[q]] : 0.f;
                } else {
                    w = gw.y;
                    wsum[q] = f_add(wsum[q], w);
                    fac = wsum[q] > 0.f ? f_div(w, wsum[q]) : 0.f;
                }
                const float delta = f_sub(gw.x, mean[q]);
                mean[q] = f_add(mean[q], f_mul(fac, delta));
                m2[q] = f_add(m2[q], f_mul(f_mul(w, delta), f_sub(gw.x, mean[q])));
                if (use_dir) {
                    a_num[q] = f_add(a_num[q], f_mul(w, s_agree[(e * CN) * NBP + s]));
                    a_den[q] = f_add(a_den[q], w);
                }
            }
        }
    }
    __syncthreads();

    // ---- left counts and gradient sums over all eras, from the warps that scanned the node ----
    // (the cells are free now: counts in [node][NBP] of word A, 64-bit sums in the gains' place)
    unsigned long long* s_lg = reinterpret_cast<unsigned long long*>(s_gain);
    for (int i = threadIdx.x; i < plane; i += kWalkThreads) {
        s_cells[i] = 0u;
        s_lg[i] = 0ull;
    }
    __syncthreads();
    if (scans) {
#pragma unroll
        for (int i = 0; i < BPL; ++i) {
            const int s = my_node * NBP + i * 32 + lane;
            if (EB == 1) {
                s_cells[s] = lc_sum[i];
                s_lg[s] = (unsigned long long)lg_sum[i];
            } else {
                if (lc_sum[i]) atomicAdd(s_cells + s, lc_sum[i]);
                if (lg_sum[i]) atomicAdd(s_lg + s, (unsigned long long)lg_sum[i]);
            }
        }
    }
    __syncthreads();

    // ---- score of every threshold under the global min_samples_leaf mask ----
    float* s_score = reinterpret_cast<float*>(s_cells + plane);
#pragma unroll
    for (int q = 0; q < SLOTS; ++q) {
        const int s = threadIdx.x + q * kWalkThreads;
        if (s >= n_slots) break;
        const float ws0 = UNIT ? (float)n_valid[q] : wsum[q];
        const float ws = ws0 < 1e-12f ? 1e-12f : ws0;
        float var = f_div(m2[q], ws);
        if (var < 0.f) var = 0.f;        // NaN stays NaN
        float score = f_sub(mean[q], f_mul(a.lambda_dro, __fsqrt_rn(var)));
        if (use_dir) score = f_add(score, f_mul(a.direction_weight, a_den[q] > 0.f ? f_div(a_num[q], a_den[q]) : 0.f));
        const long long lc = s_cells[s], total = a.frontier[node0 + s / NBP].count;
        s_score[s] = (lc >= a.min_samples_leaf && total - lc >= a.min_samples_leaf) ? score : -INFINITY;
    }
    __syncthreads();
    if (warp >= live) return;

    // ---- best threshold of a node: largest score, then largest left count, then the last ----
    float bs = -INFINITY;
    uint32_t bc = 0u, mine = 0u;         // bit i of `mine`: bin lane * BPL + i is a threshold
    int bb = -1;                         // bin of the best threshold
    bool nan = false;
#pragma unroll
    for (int i = 0; i < BPL; ++i) {
        const int bin = lane * BPL + i, s = warp * NBP + i * 32 + lane;
        if (bin >= nb - 1 || !s_set[bin]) continue;
        mine |= 1u << i;
        const float sc = s_score[s];
        const uint32_t lc = s_cells[s];
        if (sc != sc) {
            nan = true;
        } else if (bb < 0 || sc > bs || (sc == bs && lc >= bc)) {
            bs = sc;
            bc = lc;
            bb = bin;
        }
    }
    nan = __any_sync(0xFFFFFFFFu, nan);
    for (int d = 16; d > 0; d >>= 1) {
        const float os = __shfl_xor_sync(0xFFFFFFFFu, bs, d);
        const uint32_t oc = __shfl_xor_sync(0xFFFFFFFFu, bc, d);
        const int ob = __shfl_xor_sync(0xFFFFFFFFu, bb, d);
        if (ob >= 0 && (bb < 0 || os > bs || (os == bs && (oc > bc || (oc == bc && ob > bb))))) {
            bs = os;
            bc = oc;
            bb = ob;
        }
    }
    const int upto = bb - lane * BPL;    // this lane's bins below the best
    const uint32_t below = upto <= 0 ? 0u : (upto >= BPL ? mine : mine & ((1u << upto) - 1u));
    const int k = __reduce_add_sync(0xFFFFFFFFu, __popc(below));
    if (lane == 0) {
        Cand out;
        out.score = bs;
        out.k = bb >= 0 ? k : -1;
        out.left_count = bb >= 0 ? bc : 0u;
        out.flags = (nan ? 1u : 0u) | ((uint32_t)(bb >= 0 ? bb : 0) << 8);
        out.left_gq = bb >= 0 ? (int64_t)s_lg[warp * NBP + bb % BPL * 32 + bb / BPL] : 0ll;
        a.cand[(size_t)a.feat_pos[f] * a.node_stride + node0 + warp] = out;
    }
}

// ---- a warp per node ---------------------------------------------------------------------------------
// Frontiers of as many nodes as a CTA has warps, or more: every warp owns a node for all eras, so the lane that
// scans a threshold also advances its recursion and in the end scores it.  No gain passes through shared
// memory and nothing is waited for but the cells: two eras at a time, the rows of the next two are added to one
// set of cells while the set before is scanned, a barrier per step.  Where the batches spent more time than on
// the gains themselves: the exchange of the gains with its second barrier, 180 of 1 016 us at 32 nodes (500 000
// rows, 256 features), and the rows, which went by once per sixteen nodes, 544.  Now 630.
// (Era weights 0 / 1, eras of one tile.)
template <int BPL, int WARPS>
__global__ void __launch_bounds__(32 * WARPS, (WARPS == 16 && BPL <= 4) ? 2 : 1) walk_nodes_kernel(WalkLaunch a) {
    constexpr int NBP = 32 * BPL, THREADS = 32 * WARPS;
    constexpr int plane = (WARPS + 1) * NBP;                 // of word A; word B follows.  The last pair's cells: rows of no node here
    constexpr uint32_t PAIR = 4u * NBP, ERA = 8u * plane, SET = 2u * ERA;   // bytes
    extern __shared__ __align__(16) uint32_t s_cells[];      // [2 sets][2 eras][2 words][WARPS + 1][NBP] | 1 / n | (divisor, reciprocal)
    float* s_inv = reinterpret_cast<float*>(s_cells + 8 * plane);
    float2* s_div = reinterpret_cast<float2*>(s_inv + (a.n_eras + 2) / 2 * 2);
    __shared__ uint32_t s_mass[256];
    __shared__ uint8_t s_set[256];
    const int n_nodes = min(*a.n_nodes_ptr, a.n_nodes);
    const int node0 = blockIdx.x * WARPS;
    const int live = min(WARPS, n_nodes - node0);
    if (live <= 0) return;
    const int f = blockIdx.y;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nb = a.max_bins, E = a.n_eras, K = a.n_thr;
    const int CB = a.count_bits, LB = a.lo_bits;
    const uint32_t lo_mask = (1u << LB) - 1u, cmask = (1u << CB) - 1u, one_a = 1u << CB;
    const float inv_scale = *a.inv_scale_ptr, lam = a.lambda_l2;
    const bool table = a.div_table && division_in_range(inv_scale, lam);

    for (int i = threadIdx.x; i < 8 * plane; i += THREADS) s_cells[i] = 0u;
    for (int n = threadIdx.x; n <= E; n += THREADS) s_inv[n] = n > 0 ? f_div(1.f, (float)n) : 0.f;
    if (table)
        for (int n = threadIdx.x; n <= a.max_era_rows; n += THREADS) {
            const float d = f_add((float)n, lam);
            s_div[n] = make_float2(d, f_div(1.f, d));
        }
    if (a.mass) {
        for (int b = threadIdx.x; b < 256; b += THREADS) s_mass[b] = a.mass[(size_t)f * 256 + b];
        __syncthreads();
        mass_cut_set(s_mass, s_set, nb, K);
    } else {
        for (int b = threadIdx.x; b < 256; b += THREADS) s_set[b] = 0;
        __syncthreads();
        for (int k = threadIdx.x; k < K; k += THREADS) s_set[a.thr_ids[k]] = 1;
    }
    __syncthreads();

    const uint8_t* codes = a.codes + (int64_t)a.feat_rows[f] * a.pitch;
    const bool sparse = gridDim.x > 2;   // most rows belong to other CTAs: gradients are read when a row is ours
    const uint32_t cells_at = (uint32_t)__cvta_generic_to_shared(s_cells);
    auto load_group = [&](int c, RowGroup& x) {              // chunk c, 128 rows (the row arrays are padded to 256)
        const uint32_t g = 32u * (uint32_t)c + (uint32_t)lane;
        x.codes = reinterpret_cast<const uint32_t*>(codes)[g];
        x.slots = reinterpret_cast<const uint2*>(a.slot)[g];
        if (!sparse) x.gq = reinterpret_cast<const int4*>(a.gq)[g];
    };
    auto add_row = [&](uint32_t here, uint32_t n, uint32_t code, int q) {
#ifdef PB_DEBUG_BOUNDS
        const uint32_t sl = n + (uint32_t)node0;
        if ((sl & 0xFFFFu) != kSlotNone && (int)sl >= a.n_nodes && a.debug_flags) atomicOr(a.debug_flags, kDbgSlot);
        if (n < (uint32_t)live && code >= (uint32_t)nb) {
            if (a.debug_flags) atomicOr(a.debug_flags, kDbgCode);
            return;
        }
#endif
        const uint32_t at = here + min(n, (uint32_t)WARPS) * PAIR + code * 4u;
        asm volatile("red.shared.add.u32 [%0], %1;\n red.shared.add.u32 [%0 + %3], %2;" ::"r"(at),
                     "r"(((uint32_t)q & lo_mask) * one_a + 1u), "r"(q >> LB), "n"(4 * plane) : "memory");
    };
    // rows [r0, r1) of two eras, the second from mid on
    auto add_group = [&](int c, int r0, int mid, int r1, uint32_t set, RowGroup& x) {
        x.codes = cells_of<BPL>(x.codes);
        const int r = 128 * c + 4 * lane;
        const uint32_t n0 = (x.slots.x & 0xFFFFu) - (uint32_t)node0, n1 = (x.slots.x >> 16) - (uint32_t)node0;
        const uint32_t n2 = (x.slots.y & 0xFFFFu) - (uint32_t)node0, n3 = (x.slots.y >> 16) - (uint32_t)node0;
        if (sparse) {
            if (min(min(n0, n1), min(n2, n3)) >= (uint32_t)live) return;
            x.gq = reinterpret_cast<const int4*>(a.gq)[32 * c + lane];
        }
        if (r >= r0 && r + 4 <= r1 && (r >= mid || r + 4 <= mid)) {
            const uint32_t here = set + (r >= mid ? ERA : 0u);
            add_row(here, n0, x.codes & 0xFFu, x.gq.x);
            add_row(here, n1, __byte_perm(x.codes, 0u, 0x4441u), x.gq.y);
            add_row(here, n2, __byte_perm(x.codes, 0u, 0x4442u), x.gq.z);
            add_row(here, n3, x.codes >> 24, x.gq.w);
        } else {                         // rows of other steps, or of both eras
            auto one = [&](int j, uint32_t n, uint32_t code, int q) {
                if (r + j >= r0 && r + j < r1) add_row(set + (r + j >= mid ? ERA : 0u), n, code, q);
            };
            one(0, n0, x.codes & 0xFFu, x.gq.x);
            one(1, n1, __byte_perm(x.codes, 0u, 0x4441u), x.gq.y);
            one(2, n2, __byte_perm(x.codes, 0u, 0x4442u), x.gq.z);
            one(3, n3, x.codes >> 24, x.gq.w);
        }
    };
    auto add_rows = [&](int e, uint32_t set) {               // eras e, e + 1
        if (e >= E) return;
        const int r0 = a.era_offsets[e], mid = a.era_offsets[e + 1], r1 = a.era_offsets[min(e + 2, E)];
        RowGroup cur;
        int c = r0 / 128 + warp;
        const int chunks = (r1 + 127) / 128;
        if (c < chunks) load_group(c, cur);
        for (; c < chunks; c += WARPS) {
            RowGroup x = cur;
            if (c + WARPS < chunks) load_group(c + WARPS, cur);
            add_group(c, r0, mid, r1, set, x);
        }
    };

    float mean[BPL], m2[BPL];
    int n_valid[BPL];
    uint32_t lc_sum[BPL];
    long long lg_sum[BPL];
#pragma unroll
    for (int i = 0; i < BPL; ++i) {
        mean[i] = m2[i] = 0.f;
        n_valid[i] = 0;
        lc_sum[i] = 0u;
        lg_sum[i] = 0ll;
    }
    add_rows(0, cells_at);
    __syncthreads();
    for (int e0 = 0; e0 < E; e0 += 2) {
        add_rows(e0 + 2, cells_at + ((e0 & 2) ? 0u : SET));
        if (warp < live) {
#pragma unroll 1
            for (int e = 0; e < 2 && e0 + e < E; ++e) {
                // prefix over the bins; the packed words are added as they are (the rows behind them are
                // distinct rows of a tile, so no field overflows)
                uint32_t A[BPL], B[BPL];
                uint32_t* at = s_cells + ((e0 & 2) + e) * (2 * plane) + warp * NBP + lane * BPL;
                take_words(at, A);
                take_words(at + plane, B);
#pragma unroll
                for (int i = 1; i < BPL; ++i) {
                    A[i] += A[i - 1];
                    B[i] += B[i - 1];
                }
                uint32_t sa = A[BPL - 1], sb = B[BPL - 1];
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const uint32_t ua = __shfl_up_sync(0xFFFFFFFFu, sa, d), ub = __shfl_up_sync(0xFFFFFFFFu, sb, d);
                    if (lane >= d) {
                        sa += ua;
                        sb += ub;
                    }
                }
                const uint32_t ta = __shfl_sync(0xFFFFFFFFu, sa, 31), tb = __shfl_sync(0xFFFFFFFFu, sb, 31);
                sa -= A[BPL - 1];
                sb -= B[BPL - 1];
                const uint32_t tc = ta & cmask;
                const long long tg = (long long)(int32_t)tb * (1ll << LB) + (long long)(ta >> CB);
                const float tgf = f_mul(__ll2float_rn(tg), inv_scale);
                const float parent = table ? divide_by(f_mul(0.5f, f_mul(tgf, tgf)), s_div[tc])
                                           : f_div(f_mul(0.5f, f_mul(tgf, tgf)), f_add((float)tc, lam));
#pragma unroll
                for (int i = 0; i < BPL; ++i) {              // (the operations of gain_of)
                    const uint32_t av = A[i] + sa, bv = B[i] + sb, lc = av & cmask, rc = tc - lc;
                    const long long lgq = (long long)(int32_t)bv * (1ll << LB) + (long long)(av >> CB);
                    lc_sum[i] += lc;
                    lg_sum[i] += lgq;
                    const float lg = f_mul(__ll2float_rn(lgq), inv_scale), rg = f_sub(tgf, lg);
                    const float ll = f_mul(lg, lg), rr = f_mul(rg, rg);
                    const float ql = table ? divide_by(ll, s_div[lc]) : f_div(ll, f_add((float)lc, lam));
                    const float qr = table ? divide_by(rr, s_div[rc]) : f_div(rr, f_add(f_sub((float)tc, (float)lc), lam));
                    const float gain = f_sub(f_mul(0.5f, f_add(ql, qr)), parent);
                    const bool valid = lc > 0u && rc > 0u;
                    n_valid[i] += valid ? 1 : 0;
                    const float fac = valid ? s_inv[n_valid[i]] : 0.f, delta = f_sub(gain, mean[i]);
                    mean[i] = f_add(mean[i], f_mul(fac, delta));
                    m2[i] = f_add(m2[i], f_mul(f_mul(valid ? 1.f : 0.f, delta), f_sub(gain, mean[i])));
                }
            }
        }
        __syncthreads();                 // the next cells are complete, these are zero
    }
    if (warp >= live) return;

    // ---- score of every threshold under the global min_samples_leaf mask; the best of the node: largest score,
    //      then largest left count, then the last ----
    const int64_t total = a.frontier[node0 + warp].count;
    float bs = -INFINITY;
    uint32_t bc = 0u, mine = 0u;         // bit i of `mine`: bin lane * BPL + i is a threshold
    int bb = -1;                         // bin of the best threshold
    long long bg = 0ll;
    bool nan = false;
#pragma unroll
    for (int i = 0; i < BPL; ++i) {
        const int bin = lane * BPL + i;
        if (bin >= nb - 1 || !s_set[bin]) continue;
        mine |= 1u << i;
        const float ws0 = (float)n_valid[i], ws = ws0 < 1e-12f ? 1e-12f : ws0;
        float var = f_div(m2[i], ws);
        if (var < 0.f) var = 0.f;        // NaN stays NaN
        float sc = f_sub(mean[i], f_mul(a.lambda_dro, __fsqrt_rn(var)));
        const int64_t lc = lc_sum[i];
        if (!(lc >= a.min_samples_leaf && total - lc >= a.min_samples_leaf)) sc = -INFINITY;
        if (sc != sc) {
            nan = true;
        } else if (bb < 0 || sc > bs || (sc == bs && lc_sum[i] >= bc)) {
            bs = sc;
            bc = lc_sum[i];
            bb = bin;
            bg = lg_sum[i];
        }
    }
    nan = __any_sync(0xFFFFFFFFu, nan);
    for (int d = 16; d > 0; d >>= 1) {
        const float os = __shfl_xor_sync(0xFFFFFFFFu, bs, d);
        const uint32_t oc = __shfl_xor_sync(0xFFFFFFFFu, bc, d);
        const int ob = __shfl_xor_sync(0xFFFFFFFFu, bb, d);
        const long long og = __shfl_xor_sync(0xFFFFFFFFu, bg, d);
        if (ob >= 0 && (bb < 0 || os > bs || (os == bs && (oc > bc || (oc == bc && ob > bb))))) {
            bs = os;
            bc = oc;
            bb = ob;
            bg = og;
        }
    }
    const int upto = bb - lane * BPL;    // this lane's bins below the best
    const uint32_t below = upto <= 0 ? 0u : (upto >= BPL ? mine : mine & ((1u << upto) - 1u));
    const int k = __reduce_add_sync(0xFFFFFFFFu, __popc(below));
    if (lane == 0) {
        Cand out;
        out.score = bs;
        out.k = bb >= 0 ? k : -1;
        out.left_count = bb >= 0 ? bc : 0u;
        out.flags = (nan ? 1u : 0u) | ((uint32_t)(bb >= 0 ? bb : 0) << 8);
        out.left_gq = bb >= 0 ? (int64_t)bg : 0ll;
        a.cand[(size_t)a.feat_pos[f] * a.node_stride + node0 + warp] = out;
    }
}

template <int BPL, int WARPS>
int launch_nodes(const WalkLaunch& a, dim3 grid, size_t smem, cudaStream_t stream) {
    PB_TRY(allow_shared(walk_nodes_kernel<BPL, WARPS>, smem));
    walk_nodes_kernel<BPL, WARPS><<<grid, 32 * WARPS, smem, stream>>>(a);
    return PB_OK;
}

template <int BPL, int MODE, int COPIES, int WARPS>
int launch_one(const WalkLaunch& a, dim3 grid, size_t smem, cudaStream_t stream) {
    PB_TRY(allow_shared(walk_kernel<BPL, MODE, COPIES, WARPS>, smem));
    walk_kernel<BPL, MODE, COPIES, WARPS><<<grid, 32 * WARPS, smem, stream>>>(a);
    return PB_OK;
}

template <int BPL>
int launch_bpl(const WalkLaunch& a, int mode, int copies, int warps, bool own, dim3 grid, size_t smem, cudaStream_t stream) {
    constexpr int B = BPL <= 4 ? BPL : 4;
    if (own)
        return warps == 32 ? launch_nodes<B, 32>(a, grid, smem, stream) : launch_nodes<B, 16>(a, grid, smem, stream);
    if (BPL <= 4 && mode == kUnit && warps == 32) {
        return copies == 2 ? launch_one<B, kUnit, 2, 32>(a, grid, smem, stream) : launch_one<B, kUnit, 1, 32>(a, grid, smem, stream);
    }
    if (mode == kUnit) return copies == 2 ? launch_one<BPL, kUnit, 2, 16>(a, grid, smem, stream) : launch_one<BPL, kUnit, 1, 16>(a, grid, smem, stream);
    return mode == kUnitTiles ? launch_one<BPL, kUnitTiles, 1, 16>(a, grid, smem, stream) : launch_one<BPL, kGeneral, 1, 16>(a, grid, smem, stream);
}

}  // namespace

// How a launch is laid out.
struct WalkShape {
    int bpl, mode, copies, warps, cell_nodes, groups;
    bool own;            // a warp per node (walk_nodes_kernel)
    bool div_table;
    size_t smem;
};

// The forms a launch may take: batches of sixteen or thirty-two warps, a warp per node of either.
enum WalkForm { kBatch16 = 0, kBatch32 = 1, kNodes16 = 2, kNodes32 = 3, kWalkForms = 4 };

static bool walk_can(const WalkLaunch& a, int form) {
    const bool unit = a.era_alpha <= 0.f && a.direction_weight == 0.f && a.n_eras < kWalkInv && a.max_era_rows <= a.tile_rows;
    return form == kBatch16 || (unit && a.max_bins <= 128);
}

// PACKBOOST_WALK_FORM=0 .. 3: that form wherever it can be had, and a line for each launch, for comparisons.
static int forced_walk() {
    static const int form = [] {
        const char* e = getenv("PACKBOOST_WALK_FORM");
        return e && e[0] >= '0' && e[0] < '0' + kWalkForms && e[1] == 0 ? e[0] - '0' : -1;
    }();
    return form;
}

static bool walk_takes(const WalkLaunch& a, int form) {
    if (!walk_can(a, form)) return false;
    if (forced_walk() >= 0 && walk_can(a, forced_walk())) return form == forced_walk();
    if (form == kBatch16) return true;
    // (a warp per node of sixteen: from about a hundred rows per era and node on; 20 000 rows, 64 features, 20
    // eras take 40 us that way and 35 as more and smaller CTAs)
    return form == kBatch32 || (form == kNodes16 ? a.n_nodes == 16 && a.n_rows >= (int64_t)1600 * a.n_eras : a.n_nodes >= 32);
}

static WalkShape walk_shape(const WalkLaunch& a, int form) {
    WalkShape s;
    s.bpl = a.max_bins <= 32 ? 1 : a.max_bins <= 64 ? 2 : a.max_bins <= 128 ? 4 : 8;
    const bool unit = a.era_alpha <= 0.f && a.direction_weight == 0.f && a.n_eras < kWalkInv;
    s.mode = !unit ? kGeneral : a.max_era_rows <= a.tile_rows ? kUnit : kUnitTiles;
    s.warps = form == kBatch32 || form == kNodes32 ? 32 : 16;
    s.own = form == kNodes16 || form == kNodes32;
    // Nodes of a batched CTA: fewer while the CTAs do not fill the GPU: the scan and the recursion of an era are
    // then spread over more SMs, each of which goes through the rows of the feature.  That pays up to about
    // 320 rows per era and node of the CTA (20 000 rows, 64 features, 20 eras, 16 nodes: 57 -> 28 us; 200 000
    // rows, 100 features, 40 eras: 16 nodes 152 -> 135, 8 nodes 97 -> 110).
    s.cell_nodes = a.n_nodes < s.warps ? a.n_nodes : s.warps;
    const int64_t places = s.warps == 32 ? 148 : 148 * 2;
    while (!s.own && s.cell_nodes > 1 && (int64_t)a.n_feat * (a.n_nodes / s.cell_nodes) * 2 <= places &&
           a.n_rows <= (int64_t)320 * s.cell_nodes * a.n_eras)
        s.cell_nodes /= 2;
    s.groups = (a.n_nodes + s.cell_nodes - 1) / s.cell_nodes;
    const size_t plane = (size_t)s.warps * 32 * s.bpl * 4, trash = (size_t)32 * s.bpl * 4;
    // Two copies of the cells while few nodes share the rows of a warp: its lanes then meet in the bins of
    // a column of few values, which took twice as long as the others.  With many nodes they meet less and
    // the copies only lengthen the scan (500 000 rows, 256 features: 8 nodes 401 us with copies, 454
    // without, 16 nodes 594 either way, 32 nodes 1 125 and 965).
    s.copies = (s.mode == kUnit && s.bpl <= 4 && a.n_nodes <= 8) ? 2 : 1;
    s.smem = s.own ? 8 * (plane + trash) + (size_t)(a.n_eras + 2) / 2 * 8
                   : 2 * s.copies * (plane + trash) + 2 * plane + (s.mode == kGeneral ? plane : (size_t)(a.n_eras + 2) / 2 * 8);
    // the table of divisors is 8 bytes per row of the largest era: while it leaves room for the SM's CTAs
    s.div_table = a.max_era_rows <= a.tile_rows && s.smem + (size_t)(a.max_era_rows + 1) * 8 <= (s.warps == 32 ? 220 : 110) * 1024;
    if (s.div_table) s.smem += (size_t)(a.max_era_rows + 1) * 8;
    return s;
}

// A CTA goes through all rows of its feature and all eras, whatever the other SMs do, so a launch takes
// that chain once per wave of CTAs; two CTAs on an SM take 1.29 times as long as one (1.7 where each warp owns a
// node).  Constants of the batched form with sixteen warps fitted to 9 000 timed depths (2 000 to 4 million
// rows, 4 to 420 features, 1 to 600 eras, 17 to 256 bins, 1 to 512 nodes, every form of the score); half of the
// estimates were within 13 %.  Those of the other forms from 60 000 to 1 million rows, 8 to 256 features, 20 to
// 574 eras, 63 to 128 bins and 1 to 512 nodes: within 15 %, but for one node over many short eras (121 us, not 92).
static double walk_estimate_us(const WalkLaunch& a, const WalkShape& s) {
    const int64_t tiles = a.max_era_rows <= a.tile_rows ? 1 : tiles_of(a.max_era_rows, a.tile_rows);
    const int eras = s.mode == kUnit ? s.warps / s.cell_nodes : 1;   // of a batch
    const double batches = s.mode == kUnit ? (double)((a.n_eras + eras - 1) / eras) : (double)a.n_eras * tiles;
    const double batch = s.own ? (s.warps == 32 ? 0.41 : 0.23) * s.bpl : s.mode == kUnit ? (s.warps == 32 ? 1.0 + 0.65 * s.bpl : 1.2 + 0.34 * s.bpl)
                         : s.mode == kUnitTiles ? 0.63 + 0.14 * s.bpl
                         : 1.0 + ((a.direction_weight != 0.f && tiles == 1) ? 0.33 : 0.22) * s.bpl;
    const double per_row = s.own ? 3.0e-4 : s.warps == 32 ? 2.05e-4 : 2.9e-4;
    const double chain = per_row * a.n_rows + batches * batch;
    const int per_sm = (s.bpl <= 4 && s.mode != kGeneral && s.warps == 16) ? 2 : 1;
    const int64_t ctas = (int64_t)a.n_feat * s.groups, places = 148 * per_sm;
    const double whole = per_sm == 2 ? (s.own ? 1.7 : 1.29) : 1.0;
    const int64_t rest = ctas % places;
    const double waves = (double)(ctas / places) * whole + (rest == 0 ? 0.0 : rest <= 148 ? 1.0 : whole);
    return (s.warps == 32 || s.own ? 11.0 : 22.0) + waves * chain + (a.mass ? 16.0 + 7.5e-7 * (double)a.n_rows * a.n_feat : 0.0);
}

// The form with the least estimate.  (Measured, batches of sixteen / of thirty-two / a warp per node: 200 000
// rows, 100 features, 40 eras, 128 bins 57 / 53 us at one node, 96 / 83 at eight, 135 / 142 / 107 at sixteen,
// - / 207 / 126 at thirty-two; 500 000 x 256, 100 eras 215 / 236 at one, - / 552 / 414 at sixteen; 131 072 x 8,
// 574 eras, 32 nodes 1 120 with a warp per node, where more and smaller CTAs take a fifth of that.)
static double best_walk(const WalkLaunch& a, WalkShape* best) {
    double us = 1e300;
    for (int form = 0; form < kWalkForms; ++form) {
        if (!walk_takes(a, form)) continue;
        const WalkShape s = walk_shape(a, form);
        const double e = walk_estimate_us(a, s);
        if (e < us) {
            us = e;
            *best = s;
        }
    }
    return us;
}

double walk_estimate_us(const WalkLaunch& a) {
    WalkShape s;
    return best_walk(a, &s);
}

int launch_walk(WalkLaunch a, cudaStream_t stream) {
    if (a.n_feat <= 0 || a.n_nodes <= 0) return PB_OK;
    if (a.max_bins > 256) return fail_arg("max_bins=%d outside [2,256]", a.max_bins);
    WalkShape s;
    best_walk(a, &s);
    if (forced_walk() >= 0)
        fprintf(stderr, "%s<%d> warps=%d mode=%d copies=%d nodes=%d groups=%d table=%d mass=%d\n", s.own ? "walk_nodes_kernel" : "walk_kernel",
                s.bpl, s.warps, s.mode, s.copies, a.n_nodes, s.groups, (int)s.div_table, a.mass ? 1 : 0);
    a.cell_nodes = s.cell_nodes;
    const int bpl = s.bpl, mode = s.mode, copies = s.copies, warps = s.warps;
    const size_t smem = s.smem;
    a.div_table = s.div_table ? 1 : 0;
    dim3 grid((unsigned)s.groups, (unsigned)a.n_feat);
    if (grid.y > 65535u) return fail_arg("too many features in one launch");
    prof_begin(a.prof, kProfHist, stream);
    if (a.mass) {
        PB_CUDA_TRY(cudaMemsetAsync(a.mass, 0, (size_t)a.n_feat * 256 * sizeof(uint32_t), stream));
        int parts = (148 * 8 + a.n_feat - 1) / a.n_feat;   // about eight CTAs per SM
        const int most = tiles_of(a.n_rows, 4096);
        if (parts > most) parts = most;
        if (parts < 1) parts = 1;
        mass_count_kernel<<<dim3((unsigned)a.n_feat, (unsigned)parts), 256, 0, stream>>>(a);
        count_launch(1);
    }
    int rc = bpl == 1 ? launch_bpl<1>(a, mode, copies, warps, s.own, grid, smem, stream)
             : bpl == 2 ? launch_bpl<2>(a, mode, copies, warps, s.own, grid, smem, stream)
             : bpl == 4 ? launch_bpl<4>(a, mode, copies, warps, s.own, grid, smem, stream) : launch_bpl<8>(a, mode, copies, warps, s.own, grid, smem, stream);
    prof_end(a.prof, kProfHist, stream);
    if (rc) return rc;
    count_launch(1);
    PB_LAUNCH_CHECK("walk_kernel");
    return PB_OK;
}

}  // namespace pb
