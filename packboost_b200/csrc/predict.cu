// Tree routing: a row goes left when its code is <= the node's threshold.
//
// Every walk is bounded: it takes at most as many steps as its tree has nodes, a child index must
// stay inside the tree and a feature index inside the row, and a tree that breaks one of these
// rules contributes 0 for that row (the guards of packboost/backends/cuda/frontier_cuda.cu:214-231
// and 953-966).  A malformed ensemble therefore cannot hang the device or read outside its buffers.

#include <stdlib.h>

#include <vector>

#include "common.cuh"

namespace pb {

namespace {

struct PredictRowsArgs {
    const uint8_t* codes;
    int64_t n_rows;
    int64_t pitch_row;
    const int32_t* feature;
    const int32_t* threshold;
    const int32_t* left;
    const int32_t* right;
    const float* value;
    const uint8_t* is_leaf;
    const int32_t* tree_offsets;
    const int32_t* repeat;
    int n_trees;
    float weight;
    float* out;
    const float* init;
    int rows_per_cta;
    int stage;  // 1: the CTA's rows are staged in shared memory
    int n_codes;  // codes held by one row (pitch_row * 8 / code_bits): bound of a feature index
};

template <int BITS>
__device__ __forceinline__ int code_at(const uint8_t* row, int f) {
    if (BITS == 4) return (row[f >> 1] >> ((f & 1) * 4)) & 0xF;
    return row[f];
}

// One thread per row; the ensemble is walked in tree order and the prediction is accumulated
// as out = out + weight * leaf with separately rounded product and sum, which is what a loop
// of float32 tensor operations over the trees produces.
template <int BITS>
__global__ void __launch_bounds__(128) predict_rows_kernel(PredictRowsArgs a) {
    extern __shared__ __align__(16) uint8_t s_rows[];
    const int64_t row0 = (int64_t)blockIdx.x * a.rows_per_cta;
    const int nr = (int)min((int64_t)a.rows_per_cta, a.n_rows - row0);
    if (nr <= 0) return;
    if (a.stage) {
        const int64_t n16 = (int64_t)nr * a.pitch_row / 16;
        const uint4* src = reinterpret_cast<const uint4*>(a.codes + row0 * a.pitch_row);
        uint4* dst = reinterpret_cast<uint4*>(s_rows);
        for (int64_t i = threadIdx.x; i < n16; i += blockDim.x) dst[i] = __ldg(src + i);
        __syncthreads();
    }
    for (int lr = threadIdx.x; lr < nr; lr += blockDim.x) {
        const uint8_t* row = a.stage ? (s_rows + (int64_t)lr * a.pitch_row) : (a.codes + (row0 + lr) * a.pitch_row);
        float acc = a.init ? a.init[row0 + lr] : 0.f;
        for (int t = 0; t < a.n_trees; ++t) {
            const int base = __ldg(a.tree_offsets + t);
            const int n_t = __ldg(a.tree_offsets + t + 1) - base;  // nodes of this tree
            int node = 0, steps = 0;
            bool good = n_t > 0;
            while (good && !__ldg(a.is_leaf + base + node)) {
                const int f = __ldg(a.feature + base + node);
                const int thr = __ldg(a.threshold + base + node);
                if ((unsigned)f >= (unsigned)a.n_codes || ++steps > n_t) { good = false; break; }
                node = (code_at<BITS>(row, f) <= thr) ? __ldg(a.left + base + node) : __ldg(a.right + base + node);
                good = (unsigned)node < (unsigned)n_t;
            }
            const float term = good ? __fmul_rn(a.weight, __ldg(a.value + base + node)) : 0.f;
            const int rep = a.repeat ? __ldg(a.repeat + t) : 1;
            for (int k = 0; k < rep; ++k) acc = __fadd_rn(acc, term);
        }
        a.out[row0 + lr] = acc;
    }
}

// Packed ensemble: one 8-byte word pair per node,
//   x = feature (bits 0-15) | threshold (bits 16-23) | leaf flag (bit 31)
//   y = tree-relative index of the left child (the right child is the next node, which is how
//       the trees are numbered when they are grown) or, for a leaf, the bits of its float value.
// A thread owns one row and walks kWay trees at a time so that their dependent node loads
// overlap; the leaf terms are still added in tree order.
struct PredictPackedArgs {
    const uint8_t* codes;
    int64_t n_rows;
    int64_t pitch_row;
    const uint2* nodes;
    const int32_t* tree_offsets;
    const int32_t* repeat;
    int n_trees;
    float weight;
    float* out;
    const float* init;
    int rows_per_cta;
    int stage;
    int trees_per_batch;
    int n_codes;         // codes held by one row: bound of a feature index
    int max_tree_nodes;  // node count of the largest tree: bound of a walk
};

// kTpr threads share a row (they sit in the same warp): thread q walks trees t0+q, t0+kTpr+q, ...
// of each group of kTpr*kWay consecutive trees, kWay at a time so that their dependent node
// loads overlap, and the leaf terms are then added in tree order by passing them to the row's
// first thread with shuffles — the float32 sum stays the sequential one.
constexpr int kTpr = 4;
constexpr int kWay = 4;

constexpr int kStageNodes = 4096;  // nodes per staged batch of trees (32 KB), two buffers

__device__ __forceinline__ void cp_async8(void* smem_dst, const void* gmem_src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// The CTA keeps its rows' codes in shared memory and streams the ensemble through two
// shared-memory buffers in batches of `trees_per_batch` trees (asynchronous 8-byte copies, the
// next batch in flight while the current one is walked), so a node visit is two shared-memory
// loads instead of a cache-line lookup per lane.
template <int BITS>
__global__ void __launch_bounds__(512) predict_rows_packed_kernel(PredictPackedArgs a) {
    extern __shared__ __align__(16) uint8_t s_rows[];
    const int64_t row0 = (int64_t)blockIdx.x * a.rows_per_cta;
    const int nr = (int)min((int64_t)a.rows_per_cta, a.n_rows - row0);
    if (nr <= 0) return;
    uint2* s_nodes = reinterpret_cast<uint2*>(s_rows + (size_t)a.rows_per_cta * a.pitch_row * (a.stage ? 1 : 0));
    if (a.stage) {
        const int64_t n16 = (int64_t)nr * a.pitch_row / 16;
        const uint4* src = reinterpret_cast<const uint4*>(a.codes + row0 * a.pitch_row);
        uint4* dst = reinterpret_cast<uint4*>(s_rows);
        for (int64_t i = threadIdx.x; i < n16; i += blockDim.x) dst[i] = __ldg(src + i);
    }
    const int TB = a.trees_per_batch;  // 0: trees too large to stage, nodes are read from global memory
    const int q = threadIdx.x % kTpr;
    const int lane = threadIdx.x & 31;
    const int quad_base = lane - q;  // lane of the row's first thread
    const int rows_per_pass = blockDim.x / kTpr;
    const int n_batches = TB ? (a.n_trees + TB - 1) / TB : 1;

    auto prefetch = [&](int b) {
        const int ta = b * TB, tb = min(a.n_trees, ta + TB);
        const int o0 = __ldg(a.tree_offsets + ta), o1 = __ldg(a.tree_offsets + tb);
        uint2* dst = s_nodes + (size_t)(b & 1) * kStageNodes;
        const int n_copy = min(o1 - o0, kStageNodes);
        for (int i = threadIdx.x; i < n_copy; i += blockDim.x) cp_async8(dst + i, a.nodes + o0 + i);
        cp_async_commit();
    };

    // every warp runs the same number of passes, batches and tree groups, so the shuffles below
    // always see all 32 lanes; threads whose row is past the end compute on row 0 and do not store
    for (int lr0 = 0; lr0 < nr; lr0 += rows_per_pass) {
        const int lr_raw = lr0 + threadIdx.x / kTpr;
        const bool has_row = lr_raw < nr;
        const int lr = has_row ? lr_raw : 0;
        const uint8_t* row = a.stage ? (s_rows + (int64_t)lr * a.pitch_row) : (a.codes + (row0 + lr) * a.pitch_row);
        float acc = a.init ? a.init[row0 + lr] : 0.f;
        if (TB) prefetch(0);
        for (int b = 0; b < n_batches; ++b) {
            const int ta = TB ? b * TB : 0, tb = TB ? min(a.n_trees, ta + TB) : a.n_trees;
            const uint2* node_base = a.nodes;
            int off_shift = 0;
            if (TB) {
                if (b + 1 < n_batches) {
                    prefetch(b + 1);
                    cp_async_wait<1>();
                } else {
                    cp_async_wait<0>();
                }
                __syncthreads();  // batch b (and, on the first batch, the rows) are in shared memory
                node_base = s_nodes + (size_t)(b & 1) * kStageNodes;
                off_shift = __ldg(a.tree_offsets + ta);
            } else {
                __syncthreads();
            }
            for (int t0 = ta; t0 < tb; t0 += kTpr * kWay) {
                const uint2* base[kWay];
                uint2 nd[kWay];
                uint32_t lim[kWay];  // nodes of the tree
#pragma unroll
                for (int u = 0; u < kWay; ++u) {
                    const int t = min(t0 + u * kTpr + q, tb - 1);
                    const int o = __ldg(a.tree_offsets + t);
                    lim[u] = (uint32_t)max(__ldg(a.tree_offsets + t + 1) - o, 0);
                    if (TB && ((unsigned)(o - off_shift) > (unsigned)kStageNodes ||
                               lim[u] > (uint32_t)kStageNodes - (uint32_t)(o - off_shift)))
                        lim[u] = 0u;  // not wholly inside the staged batch
                    base[u] = node_base + (o - off_shift);
                    nd[u] = lim[u] ? base[u][0] : make_uint2(0x80000000u, 0u);
                }
                bool any = true;
                for (int steps = 0; any && steps <= a.max_tree_nodes; ++steps) {
                    any = false;
#pragma unroll
                    for (int u = 0; u < kWay; ++u) {
                        if (!(nd[u].x >> 31)) {
                            const int f = nd[u].x & 0xFFFF;
                            const int thr = (nd[u].x >> 16) & 0xFF;
                            const uint32_t child = nd[u].y + ((f < a.n_codes && code_at<BITS>(row, min(f, a.n_codes - 1)) > thr) ? 1u : 0u);
                            // a child outside the tree or a feature outside the row ends the walk with 0
                            const bool good = (child < lim[u]) & (f < a.n_codes);
                            nd[u] = good ? base[u][child] : make_uint2(0x80000000u, 0u);
                            any = true;
                        }
                    }
                }
#pragma unroll
                for (int u = 0; u < kWay; ++u)
                    if (!(nd[u].x >> 31)) nd[u] = make_uint2(0x80000000u, 0u);  // step cap reached: 0
                // ordered accumulation: tree t0 + u*kTpr + qq for u, then qq, ascending
#pragma unroll
                for (int u = 0; u < kWay; ++u) {
                    const float mine = __fmul_rn(a.weight, __uint_as_float(nd[u].y));
#pragma unroll
                    for (int qq = 0; qq < kTpr; ++qq) {
                        const float term = __shfl_sync(0xFFFFFFFFu, mine, quad_base + qq);
                        const int t = t0 + u * kTpr + qq;
                        if (t < tb) {
                            const int rep = a.repeat ? __ldg(a.repeat + t) : 1;
                            for (int k = 0; k < rep; ++k) acc = __fadd_rn(acc, term);
                        }
                    }
                }
            }
            __syncthreads();  // the buffer of batch b may be overwritten by the prefetch of batch b + 2
        }
        if (has_row && q == 0) a.out[row0 + lr] = acc;
    }
}

// The common case of the packed predictor — rows and tree batches both staged in shared memory —
// with every address a 32-bit shared-memory address (the generic form above resolves the address
// space on each of its two loads per node visit and carries 64-bit pointers) and the tree offsets
// of a batch staged next to its nodes, so that a node visit is two shared loads and a handful of
// integer instructions.  Same traversal and the same ordered accumulation as above.
__device__ __forceinline__ uint32_t lds_u8(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u8 %0, [%1];\n" : "=r"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint32_t lds_u32(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];\n" : "=r"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint2 lds_v2(uint32_t addr) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];\n" : "=r"(v.x), "=r"(v.y) : "r"(addr));
    return v;
}
__device__ __forceinline__ void cp_async4(void* smem_dst, const void* gmem_src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(gmem_src) : "memory");
}

constexpr int kStageTrees = 1024;  // most trees of one staged batch (their offsets are staged too)

template <int BITS>
__global__ void __launch_bounds__(512) predict_rows_packed_smem_kernel(PredictPackedArgs a) {
    extern __shared__ __align__(16) uint8_t s_rows[];  // rows | nodes [2][kStageNodes] | offsets [2][kStageTrees + 1]
    const int64_t row0 = (int64_t)blockIdx.x * a.rows_per_cta;
    const int nr = (int)min((int64_t)a.rows_per_cta, a.n_rows - row0);
    if (nr <= 0) return;
    uint2* s_nodes = reinterpret_cast<uint2*>(s_rows + (size_t)a.rows_per_cta * a.pitch_row);
    int32_t* s_offs = reinterpret_cast<int32_t*>(s_nodes + 2 * kStageNodes);
    uint2* s_zero = reinterpret_cast<uint2*>(s_offs + 2 * (kStageTrees + 1));  // a leaf of value 0
    if (threadIdx.x == 0) *s_zero = make_uint2(0x80000000u, 0u);
    {
        const int64_t n16 = (int64_t)nr * a.pitch_row / 16;
        const uint4* src = reinterpret_cast<const uint4*>(a.codes + row0 * a.pitch_row);
        uint4* dst = reinterpret_cast<uint4*>(s_rows);
        for (int64_t i = threadIdx.x; i < n16; i += blockDim.x) dst[i] = __ldg(src + i);
    }
    const uint32_t rows_addr = (uint32_t)__cvta_generic_to_shared(s_rows);
    const uint32_t nodes_addr = (uint32_t)__cvta_generic_to_shared(s_nodes);
    const uint32_t offs_addr = (uint32_t)__cvta_generic_to_shared(s_offs);
    const uint32_t zero_leaf = (uint32_t)__cvta_generic_to_shared(s_zero);
    const uint32_t fmax = (uint32_t)a.n_codes - 1u;
    const int TB = a.trees_per_batch;
    const int q = threadIdx.x % kTpr;
    const int lane = threadIdx.x & 31;
    const int quad_base = lane - q;
    const int rows_per_pass = blockDim.x / kTpr;
    const int n_batches = (a.n_trees + TB - 1) / TB;

    auto prefetch = [&](int b) {
        const int ta = b * TB, tb = min(a.n_trees, ta + TB);
        const int o0 = __ldg(a.tree_offsets + ta), o1 = __ldg(a.tree_offsets + tb);
        uint2* dst = s_nodes + (size_t)(b & 1) * kStageNodes;
        const int n_copy = min(o1 - o0, kStageNodes);  // (a batch larger than the buffer: its tail trees yield 0)
        for (int i = threadIdx.x; i < n_copy; i += blockDim.x) cp_async8(dst + i, a.nodes + o0 + i);
        int32_t* od = s_offs + (size_t)(b & 1) * (kStageTrees + 1);
        for (int i = threadIdx.x; i <= tb - ta; i += blockDim.x) cp_async4(od + i, a.tree_offsets + ta + i);
        cp_async_commit();
    };

    for (int lr0 = 0; lr0 < nr; lr0 += rows_per_pass) {
        const int lr_raw = lr0 + threadIdx.x / kTpr;
        const bool has_row = lr_raw < nr;
        const int lr = has_row ? lr_raw : 0;
        const uint32_t row = rows_addr + (uint32_t)lr * (uint32_t)a.pitch_row;
        float acc = a.init ? a.init[row0 + lr] : 0.f;
        prefetch(0);
        for (int b = 0; b < n_batches; ++b) {
            const int ta = b * TB, tb = min(a.n_trees, ta + TB);
            if (b + 1 < n_batches) {
                prefetch(b + 1);
                cp_async_wait<1>();
            } else {
                cp_async_wait<0>();
            }
            __syncthreads();  // batch b (and, on the first batch, the rows) are in shared memory
            const uint32_t nbase = nodes_addr + (uint32_t)(b & 1) * (kStageNodes * 8u);
            const uint32_t obase = offs_addr + (uint32_t)(b & 1) * ((kStageTrees + 1) * 4u);
            const uint32_t off_shift = lds_u32(obase);
            for (int t0 = ta; t0 < tb; t0 += kTpr * kWay) {
                uint32_t base[kWay];
                uint2 nd[kWay];
                uint32_t lim[kWay];  // nodes of the tree
#pragma unroll
                for (int u = 0; u < kWay; ++u) {
                    const int t = min(t0 + u * kTpr + q, tb - 1);
                    const uint32_t o = lds_u32(obase + (uint32_t)(t - ta) * 4u);
                    const uint32_t rel = o - off_shift;
                    lim[u] = lds_u32(obase + (uint32_t)(t - ta) * 4u + 4u) - o;
                    // a tree that is empty or not wholly inside the staged batch yields 0
                    if (rel > (uint32_t)kStageNodes || lim[u] > (uint32_t)kStageNodes - rel) lim[u] = 0u;
                    base[u] = nbase + rel * 8u;
                    nd[u] = lds_v2(lim[u] ? base[u] : zero_leaf);
                }
                bool any = true;
                for (int steps = 0; any && steps <= a.max_tree_nodes; ++steps) {
                    any = false;
#pragma unroll
                    for (int u = 0; u < kWay; ++u) {
                        if (!(nd[u].x >> 31)) {
                            // a feature index past the row reads the row's last code and ends the walk
                            const uint32_t f = min(nd[u].x & 0xFFFFu, fmax);
                            const uint32_t thr = (nd[u].x >> 16) & 0xFFu;
                            uint32_t code;
                            if (BITS == 4) code = (lds_u8(row + (f >> 1)) >> ((f & 1u) * 4u)) & 0xFu;
                            else code = lds_u8(row + f);
                            const uint32_t child = nd[u].y + ((code > thr) ? 1u : 0u);
                            // a child outside the tree (or a bad feature) ends the walk at the zero leaf
                            const bool good = (child < lim[u]) & ((nd[u].x & 0xFFFFu) <= fmax);
                            nd[u] = lds_v2(good ? base[u] + child * 8u : zero_leaf);
                            any = true;
                        }
                    }
                }
#pragma unroll
                for (int u = 0; u < kWay; ++u)
                    if (!(nd[u].x >> 31)) nd[u] = make_uint2(0x80000000u, 0u);  // step cap reached: 0
#pragma unroll
                for (int u = 0; u < kWay; ++u) {
                    const float mine = __fmul_rn(a.weight, __uint_as_float(nd[u].y));
#pragma unroll
                    for (int qq = 0; qq < kTpr; ++qq) {
                        const float term = __shfl_sync(0xFFFFFFFFu, mine, quad_base + qq);
                        const int t = t0 + u * kTpr + qq;
                        if (t < tb) {
                            if (a.repeat) {
                                const int rep = __ldg(a.repeat + t);
                                for (int k = 0; k < rep; ++k) acc = __fadd_rn(acc, term);
                            } else {
                                acc = __fadd_rn(acc, term);
                            }
                        }
                    }
                }
            }
            __syncthreads();  // the buffers of batch b may be overwritten by the prefetch of batch b + 2
        }
        if (has_row && q == 0) a.out[row0 + lr] = acc;
    }
}


// ---- small trees: every lane a row, every step the same ------------------------------------------------
//
// Trees of at most 256 nodes as slots of `slot` words.  A split is one word, feature << 16 | left
// child << 8 | 255 - threshold (the right child is the next node).  Adding the code of the row to the
// word carries into the child when the code is above the threshold, so a step is two shared-memory
// loads, an add and a byte extraction, without a branch or a comparison.  Every path is exactly
// `depth` splits long - early leaves are led on by splits with threshold 255, which no code exceeds -
// and the word it ends at is the leaf value.  So a walk ends by itself whatever the words hold (child
// indices have eight bits, features are clamped to the row).
//
// The bound of the form above was shared memory: lanes of a warp sat in four trees and eight rows, so
// node loads hit many banks twice and codes of different rows lay a row apart.  Here a warp holds 32
// rows and one tree at a time.  Codes are staged feature-major (the nibbles of 32 rows are 16
// consecutive bytes), so lanes at the same node read one or two wavefronts, and the nodes of a level
// are consecutive words.  The other bound was the ordered sum: a model of 2 000 rounds with packs of
// 32 adds 64 000 numbers one after the other to each prediction, four cycles each, and the walking
// threads did it four times over.  Here `adders` (one warp per 64 rows, two rows per lane and
// instruction; the CTA's first warps, which the scheduler prefers) add the terms of the batch before
// while `walkers` (walk_warps warps per 32 rows) produce those of the next and one warp fetches the
// trees after that; the sum stays the sequential one.
// 500 000 rows x 2 376 features, 2 000 trees of depth 6 added 32 times: 22.2 -> 5.5 ms, of which the
// additions alone take 3.5; 5 417 rows, 1 000 trees: 417 -> 119 us.
struct PredictForestArgs {
    const uint8_t* codes;
    int64_t n_rows;
    int64_t pitch_row;
    int n_features;
    const uint32_t* trees;   // [copies][n_trees][slot]
    int copies;
    int slot;
    int depth;
    const int32_t* repeat;   // per tree, or null: every tree `rep` times
    int rep;
    int n_trees;
    float weight;
    float* out;
    const float* init;
    int groups;              // groups of 32 rows per CTA
    int walk_warps;          // walkers per group
};

constexpr int kTreesPerWalker = 4;  // walked at a time by a lane: independent chains
constexpr int kAddGroup = 8;        // trees whose terms an adder holds; a batch is a multiple of it
// Batches of trees in shared memory: the one being walked and those on their way.
constexpr int kTreeBuffers = 2;
constexpr int kForestShared = 227 * 1024;   // (no static arrays beside it)

// Words per feature.  The words of 32 rows are `bits` neighbouring banks; an odd number of groups puts
// those of different features at every multiple of that, an even one needs a word of padding.
__host__ __device__ constexpr int forest_words(int bits, int groups) { return groups * bits + (groups % 2 == 0 ? 1 : 0); }

__host__ __device__ constexpr int forest_adders(int groups) { return (groups + 1) / 2; }
__host__ __device__ constexpr int forest_threads(int groups, int walk_warps) {
    return 32 * (forest_adders(groups) + groups * walk_warps + 1);
}

// acc += v for two rows at once, each sum rounded like a scalar one
__device__ __forceinline__ void add2(unsigned long long& acc, unsigned long long v) {
    asm("add.rn.f32x2 %0, %0, %1;" : "+l"(acc) : "l"(v));
}

// (an index of a malformed tree may reach 256 words past its slot: the terms and the pad lie there)
inline int64_t forest_smem(int64_t n_features, int bits, int groups, int walk_warps, int64_t slot) {
    const int64_t tb = kTreesPerWalker * walk_warps;
    return ((n_features + 7) / 8 * 8 * forest_words(bits, groups) + 3) / 4 * 16 + kTreeBuffers * tb * slot * 4 + 2 * tb * 32 * groups * 4 + 128 + 1040;
}

template <int REP>
__device__ __forceinline__ void add_times(unsigned long long& acc, const unsigned long long (&v)[kAddGroup]) {
#pragma unroll
    for (int u = 0; u < kAddGroup; ++u)
#pragma unroll
        for (int i = 0; i < REP; ++i) add2(acc, v[u]);
}

template <int BITS>
__global__ void __launch_bounds__(1024) predict_forest_kernel(PredictForestArgs a) {
    extern __shared__ __align__(16) uint32_t s_mem[];
    constexpr int PER = 32 / BITS;                       // codes per word
    const int G = a.groups, R = 32 * G;
    const int W = forest_words(BITS, G);
    const int f_pad = (a.n_features + 7) / 8 * 8;
    const int TB = kTreesPerWalker * a.walk_warps;       // trees per batch
    const int batch_words = TB * a.slot;
    uint32_t* s_codes = s_mem;                           // [f_pad][W]
    uint32_t* s_trees = s_mem + (size_t)(f_pad * W + 3) / 4 * 4;       // [kTreeBuffers][TB][slot]
    const int TR = R;                                    // (the last adder of an odd G reads 32 rows past its terms)
    float* s_term = reinterpret_cast<float*>(s_trees + kTreeBuffers * batch_words);  // [2][TB][TR]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n_warps = blockDim.x >> 5;
    const int64_t row0 = (int64_t)blockIdx.x * R;
    const int nr = (int)min((int64_t)R, a.n_rows - row0);
    const int n_batches = (a.n_trees + TB - 1) / TB;

    // All CTAs ask for the same few lines at the same time, and a line is served by one slice of the L2:
    // 0.9 us per batch of eight trees, more than walking it takes.  The copies spread them.
    const uint32_t* forest = a.trees + (size_t)(blockIdx.x % a.copies) * a.n_trees * a.slot;
    auto fetch = [&](int b) {                            // (one warp) batch b into its buffer
        const int n16 = max(min(TB, a.n_trees - b * TB), 0) * a.slot / 4;
        const uint4* src = reinterpret_cast<const uint4*>(forest + (size_t)b * batch_words);
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(s_trees + (b % kTreeBuffers) * batch_words);
#pragma unroll 4
        for (int i = lane; i < n16; i += 32)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst + 16 * i), "l"(src + i) : "memory");
        cp_async_commit();
    };
    const int A = forest_adders(G);
    const bool adder = warp < A, loader = warp == n_warps - 1;
    if (loader) {
        for (int b = 0; b < kTreeBuffers - 1; ++b) fetch(b);
    }

    // ---- rows: PER x PER blocks of codes turned over (rows of a word's features -> features of rows) ----
    {
        const int row_groups = R / PER;                  // words of a feature
        const int src_words = (a.n_features + PER - 1) / PER;
        const int g_blocks = (row_groups + 7) / 8, w_blocks = (src_words + 3) / 4;
        for (int task = warp; task < g_blocks * w_blocks; task += n_warps) {
            const int g = (task % g_blocks) * 8 + (lane >> 2);
            const int fw = (task / g_blocks) * 4 + (lane & 3);
            if (g >= row_groups || fw >= src_words) continue;
            uint32_t w[PER];
#pragma unroll
            for (int i = 0; i < PER; ++i) {
                const int r = g * PER + i;
                w[i] = r < nr ? __ldg(reinterpret_cast<const uint32_t*>(a.codes + (row0 + r) * a.pitch_row) + fw) : 0u;
            }
            // swap off-diagonal blocks of 1, 2, 4 codes between words 1, 2, 4 apart
#pragma unroll
            for (int d = 1; d < PER; d <<= 1) {
                const int sh = d * BITS;
                const uint32_t m = sh == 4 ? 0x0F0F0F0Fu : (sh == 8 ? 0x00FF00FFu : 0x0000FFFFu);
#pragma unroll
                for (int i = 0; i < PER; ++i)
                    if (!(i & d)) {
                        const uint32_t t = ((w[i] >> sh) ^ w[i + d]) & m;
                        w[i + d] ^= t;
                        w[i] ^= t << sh;
                    }
            }
#pragma unroll
            for (int j = 0; j < PER; ++j) s_codes[(fw * PER + j) * W + g] = w[j];
        }
    }

    if (loader) {
        for (int b = 0; b <= n_batches; ++b) {
            cp_async_wait<kTreeBuffers - 2>();
            __syncthreads();   // batch b is here, the walk of b - 1 and the sums of b - 2 are done
            fetch(b + kTreeBuffers - 1);                 // its buffer held batch b - 1
        }
    } else if (!adder) {
        const int group = (warp - A) % G;
        const int q = (warp - A) / G;                    // trees q * kTreesPerWalker .. of a batch
        const int my_row = group * 32 + lane;
        const uint32_t lane_at = (uint32_t)__cvta_generic_to_shared(s_codes) +
                                 (BITS == 4 ? (uint32_t)(group * 16 + (lane >> 1)) : (uint32_t)my_row);
        const uint32_t nibble = (uint32_t)(lane & 1) * 4u;
        const uint32_t fmax = (uint32_t)a.n_features - 1u, pitch = (uint32_t)W * 4u;
        const uint32_t slot_bytes = (uint32_t)a.slot * 4u;
        const uint32_t first = (uint32_t)__cvta_generic_to_shared(s_trees) + (uint32_t)(q * kTreesPerWalker) * slot_bytes;
        float* term = s_term + (q * kTreesPerWalker) * TR + my_row;
        for (int b = 0; b <= n_batches; ++b) {
            __syncthreads();
            if (b == n_batches) break;
            // (trees past the last one are walked too: what the buffer holds there is never added)
            const uint32_t base = first + (uint32_t)((b % kTreeBuffers) * batch_words) * 4u;
            uint32_t idx[kTreesPerWalker];
#pragma unroll
            for (int u = 0; u < kTreesPerWalker; ++u) idx[u] = 0u;
            for (int s = 0; s < a.depth; ++s) {
                uint32_t w[kTreesPerWalker], c[kTreesPerWalker];
#pragma unroll
                for (int u = 0; u < kTreesPerWalker; ++u) w[u] = lds_u32(base + u * slot_bytes + idx[u] * 4u);
#pragma unroll
                for (int u = 0; u < kTreesPerWalker; ++u) c[u] = lds_u8(min(w[u] >> 16, fmax) * pitch + lane_at);
#pragma unroll
                for (int u = 0; u < kTreesPerWalker; ++u) {
                    const uint32_t code = BITS == 4 ? (c[u] >> nibble) & 0xFu : c[u];
                    idx[u] = __byte_perm(w[u] + code, 0u, 0x4441u);  // (a code above the threshold carries into the child)
                }
            }
            float* out = term + (b & 1) * TB * TR;
#pragma unroll
            for (int u = 0; u < kTreesPerWalker; ++u)
                out[u * TR] = __fmul_rn(a.weight, __uint_as_float(lds_u32(base + u * slot_bytes + idx[u] * 4u)));
        }
    } else {
        const int my_row = warp * 64 + 2 * lane;         // and the next one
        float2 start = make_float2(0.f, 0.f);
        if (a.init) {
            if (my_row < nr) start.x = a.init[row0 + my_row];
            if (my_row + 1 < nr) start.y = a.init[row0 + my_row + 1];
        }
        unsigned long long acc = (unsigned long long)__float_as_uint(start.y) << 32 | __float_as_uint(start.x);
        const unsigned long long* term = reinterpret_cast<const unsigned long long*>(s_term + my_row);
        for (int b = 0; b <= n_batches; ++b) {
            __syncthreads();
            if (b == 0) continue;
            const int t0 = (b - 1) * TB, nt = min(TB, a.n_trees - t0);
            const unsigned long long* in = term + ((b - 1) & 1) * TB * TR / 2;
            for (int k0 = 0; k0 < nt; k0 += kAddGroup) {
                unsigned long long v[kAddGroup];
#pragma unroll
                for (int u = 0; u < kAddGroup; ++u) v[u] = in[(k0 + u) * TR / 2];
                // A lone warp pays some 20 cycles for a branch, five additions' worth: the usual pack sizes
                // run straight through eight trees.
                switch (k0 + kAddGroup <= nt ? a.rep : 0) {
                    case 1: add_times<1>(acc, v); break;
                    case 2: add_times<2>(acc, v); break;
                    case 4: add_times<4>(acc, v); break;
                    case 8: add_times<8>(acc, v); break;
                    case 16: add_times<16>(acc, v); break;
                    case 32: add_times<32>(acc, v); break;
                    case 64: add_times<64>(acc, v); break;
                    default:
                        for (int u = 0; u < kAddGroup && k0 + u < nt; ++u) {
                            int n = a.repeat ? __ldg(a.repeat + t0 + k0 + u) : a.rep;
                            const unsigned long long vu = in[(k0 + u) * TR / 2];
                            for (; n >= 16; n -= 16) {
#pragma unroll
                                for (int i = 0; i < 16; ++i) add2(acc, vu);
                            }
                            for (; n >= 4; n -= 4) {
#pragma unroll
                                for (int i = 0; i < 4; ++i) add2(acc, vu);
                            }
                            for (; n > 0; --n) add2(acc, vu);
                        }
                }
            }
        }
        if (my_row < nr) a.out[row0 + my_row] = __uint_as_float((uint32_t)acc);
        if (my_row + 1 < nr) a.out[row0 + my_row + 1] = __uint_as_float((uint32_t)(acc >> 32));
    }
}

__global__ void __launch_bounds__(256) predict_bins_fm_kernel(
    const uint8_t* __restrict__ bins, int n_features, int64_t n_rows, const int32_t* __restrict__ feature,
    const int32_t* __restrict__ threshold, const int32_t* __restrict__ left, const int32_t* __restrict__ right,
    const float* __restrict__ value, const uint8_t* __restrict__ is_leaf, int n_nodes, float* __restrict__ out) {
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n_rows; r += (int64_t)gridDim.x * blockDim.x) {
        int node = 0, steps = 0;
        bool good = true;
        while (!__ldg(is_leaf + node)) {
            const int f = __ldg(feature + node);
            if ((unsigned)f >= (unsigned)n_features || ++steps > n_nodes) { good = false; break; }
            node = ((int)bins[(int64_t)f * n_rows + r] <= __ldg(threshold + node)) ? __ldg(left + node) : __ldg(right + node);
            if ((unsigned)node >= (unsigned)n_nodes) { good = false; break; }
        }
        out[r] = good ? __ldg(value + node) : 0.f;
    }
}

__global__ void __launch_bounds__(256) predict_pack_fm_kernel(
    const uint8_t* __restrict__ bins, int n_features, int64_t n_rows, const int32_t* __restrict__ feature,
    const int32_t* __restrict__ threshold, const int32_t* __restrict__ left_abs, const int32_t* __restrict__ right_abs,
    const float* __restrict__ value, const uint8_t* __restrict__ is_leaf, const int32_t* __restrict__ offsets,
    int n_trees, float tree_weight, float* __restrict__ out) {
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n_rows; r += (int64_t)gridDim.x * blockDim.x) {
        float sum = 0.f;
        for (int t = 0; t < n_trees; ++t) {
            int node = __ldg(offsets + t);
            const int end = __ldg(offsets + t + 1);
            if (node >= end) continue;
            const int begin = node;
            int steps = 0;
            bool good = true;
            while (!__ldg(is_leaf + node)) {
                const int f = __ldg(feature + node);
                if ((unsigned)f >= (unsigned)n_features || ++steps > end - begin) { good = false; break; }
                node = ((int)bins[(int64_t)f * n_rows + r] <= __ldg(threshold + node)) ? __ldg(left_abs + node)
                                                                                       : __ldg(right_abs + node);
                if (node < begin || node >= end) { good = false; break; }
            }
            if (good) sum = __fadd_rn(sum, __ldg(value + node));
        }
        out[r] = __fmul_rn(tree_weight, sum);
    }
}

}  // namespace
}  // namespace pb

using namespace pb;

extern "C" int pb_predict_rows(const uint8_t* codes, int64_t n_rows, int64_t pitch_row, int64_t code_bits,
                               const int32_t* feature, const int32_t* threshold, const int32_t* left,
                               const int32_t* right, const float* value, const uint8_t* is_leaf,
                               const int32_t* tree_offsets, const int32_t* repeat, int64_t n_trees, float weight,
                               float* out, const float* init, void* stream_) {
    PB_REQUIRE(codes && feature && threshold && left && right && value && is_leaf && tree_offsets && out,
               "null buffer");
    PB_REQUIRE(code_bits == 4 || code_bits == 8, "code_bits must be 4 or 8");
    PB_REQUIRE(pitch_row >= 16 && pitch_row % 16 == 0, "pitch_row must be a positive multiple of 16");
    PB_REQUIRE(((uintptr_t)codes % 16) == 0, "codes must be 16-byte aligned");
    PB_REQUIRE(n_trees >= 0 && n_trees < (1ll << 31), "n_trees out of range");
    if (n_rows <= 0) return PB_OK;
    cudaStream_t stream = (cudaStream_t)stream_;
    PredictRowsArgs a{codes, n_rows, pitch_row, feature, threshold, left, right, value, is_leaf,
                      tree_offsets, repeat, (int)n_trees, weight, out, init, 128, 1,
                      (int)((pitch_row < (1 << 27) ? pitch_row : (1 << 27)) * (code_bits == 4 ? 2 : 1))};
    const int64_t budget = 160 * 1024;
    int rows = (int)(budget / pitch_row);
    if (rows >= 128) rows = 128;
    else rows = rows / 32 * 32;
    size_t smem = 0;
    if (rows < 32) {
        a.stage = 0;
        a.rows_per_cta = 128;
    } else {
        a.rows_per_cta = rows;
        smem = (size_t)rows * pitch_row;
    }
    const unsigned grid = (unsigned)((n_rows + a.rows_per_cta - 1) / a.rows_per_cta);
    if (code_bits == 4) {
        PB_TRY(allow_shared(predict_rows_kernel<4>, smem));
        predict_rows_kernel<4><<<grid, 128, smem, stream>>>(a);
    } else {
        PB_TRY(allow_shared(predict_rows_kernel<8>, smem));
        predict_rows_kernel<8><<<grid, 128, smem, stream>>>(a);
    }
    count_launch(1);
    PB_LAUNCH_CHECK("predict_rows_kernel");
    return PB_OK;
}

static unsigned row_blocks(int64_t n) {
    int64_t b = (n + 255) / 256;
    if (b > 148 * 16) b = 148 * 16;
    return (unsigned)(b < 1 ? 1 : b);
}

extern "C" int pb_predict_bins_fm(const uint8_t* bins, int64_t n_features, int64_t n_rows, const int32_t* feature,
                                  const int32_t* threshold, const int32_t* left, const int32_t* right,
                                  const float* value, const uint8_t* is_leaf, int64_t n_nodes, float* out,
                                  void* stream) {
    PB_REQUIRE(bins && feature && threshold && left && right && value && is_leaf && out, "null buffer");
    PB_REQUIRE(n_features >= 1 && n_nodes >= 1, "bad shape");
    if (n_rows <= 0) return PB_OK;
    PB_REQUIRE(n_features < (1ll << 31) && n_nodes < (1ll << 31), "bad shape");
    predict_bins_fm_kernel<<<row_blocks(n_rows), 256, 0, (cudaStream_t)stream>>>(
        bins, (int)n_features, n_rows, feature, threshold, left, right, value, is_leaf, (int)n_nodes, out);
    count_launch(1);
    PB_LAUNCH_CHECK("predict_bins_fm_kernel");
    return PB_OK;
}

extern "C" int pb_predict_pack_fm(const uint8_t* bins, int64_t n_features, int64_t n_rows, const int32_t* feature,
                                  const int32_t* threshold, const int32_t* left_abs, const int32_t* right_abs,
                                  const float* value, const uint8_t* is_leaf, const int32_t* offsets, int64_t n_trees,
                                  float tree_weight, float* out, void* stream) {
    PB_REQUIRE(bins && feature && threshold && left_abs && right_abs && value && is_leaf && offsets && out,
               "null buffer");
    PB_REQUIRE(n_features >= 1 && n_trees >= 0, "bad shape");
    if (n_rows <= 0) return PB_OK;
    PB_REQUIRE(n_features < (1ll << 31) && n_trees < (1ll << 31), "bad shape");
    predict_pack_fm_kernel<<<row_blocks(n_rows), 256, 0, (cudaStream_t)stream>>>(
        bins, (int)n_features, n_rows, feature, threshold, left_abs, right_abs, value, is_leaf, offsets, (int)n_trees, tree_weight, out);
    count_launch(1);
    PB_LAUNCH_CHECK("predict_pack_fm_kernel");
    return PB_OK;
}

extern "C" int pb_predict_rows_packed(const uint8_t* codes, int64_t n_rows, int64_t pitch_row, int64_t code_bits,
                                      const void* nodes, const int32_t* tree_offsets, const int32_t* repeat,
                                      int64_t n_trees, int64_t max_tree_nodes, float weight, float* out,
                                      const float* init, void* stream_) {
    PB_REQUIRE(codes && nodes && tree_offsets && out, "null buffer");
    PB_REQUIRE(code_bits == 4 || code_bits == 8, "code_bits must be 4 or 8");
    PB_REQUIRE(pitch_row >= 16 && pitch_row % 16 == 0, "pitch_row must be a positive multiple of 16");
    PB_REQUIRE(((uintptr_t)codes % 16) == 0 && ((uintptr_t)nodes % 8) == 0, "codes / nodes are misaligned");
    PB_REQUIRE(n_trees >= 0 && n_trees < (1ll << 31) && max_tree_nodes >= 1, "tree counts out of range");
    if (n_rows <= 0 || n_trees == 0) {
        if (n_rows > 0) {
            if (init) PB_CUDA_TRY(cudaMemcpyAsync(out, init, (size_t)n_rows * 4, cudaMemcpyDeviceToDevice, (cudaStream_t)stream_));
            else PB_CUDA_TRY(cudaMemsetAsync(out, 0, (size_t)n_rows * 4, (cudaStream_t)stream_));
        }
        return PB_OK;
    }
    cudaStream_t stream = (cudaStream_t)stream_;
    PredictPackedArgs a{codes, n_rows, pitch_row, static_cast<const uint2*>(nodes), tree_offsets, repeat,
                        (int)n_trees, weight, out, init, 128, 1, 0,
                        (int)((pitch_row < (1 << 27) ? pitch_row : (1 << 27)) * (code_bits == 4 ? 2 : 1)),
                        (int)(max_tree_nodes < (1 << 30) ? max_tree_nodes : (1 << 30))};
    // trees per staged batch: a multiple of the group walked at once, as many as the buffer holds
    const int group = kTpr * kWay;
    int tb = (int)(kStageNodes / max_tree_nodes) / group * group;
    if (tb > kStageTrees) tb = kStageTrees / group * group;
    a.trees_per_batch = tb;  // 0: no staging
    const size_t stage_bytes = tb ? (size_t)2 * kStageNodes * sizeof(uint2) + (size_t)2 * (kStageTrees + 1) * 4 + 8 : 0;
    const int64_t budget = 224 * 1024 - (int64_t)stage_bytes;
    int rows = (int)(budget / pitch_row);
    if (rows > 128) rows = 128;
    rows = rows / 8 * 8;
    size_t smem = stage_bytes;
    if (rows < 8) {
        a.stage = 0;
        a.rows_per_cta = 128;
    } else {
        a.rows_per_cta = rows;
        smem += (size_t)rows * pitch_row;
    }
    const unsigned grid = (unsigned)((n_rows + a.rows_per_cta - 1) / a.rows_per_cta);
    const int threads = (a.rows_per_cta * kTpr + 31) / 32 * 32;
    if (a.stage && tb > 0) {  // rows and trees both staged: the all-shared-memory form
        if (code_bits == 4) {
            PB_TRY(allow_shared(predict_rows_packed_smem_kernel<4>, smem));
            predict_rows_packed_smem_kernel<4><<<grid, threads, smem, stream>>>(a);
        } else {
            PB_TRY(allow_shared(predict_rows_packed_smem_kernel<8>, smem));
            predict_rows_packed_smem_kernel<8><<<grid, threads, smem, stream>>>(a);
        }
    } else if (code_bits == 4) {
        PB_TRY(allow_shared(predict_rows_packed_kernel<4>, smem));
        predict_rows_packed_kernel<4><<<grid, threads, smem, stream>>>(a);
    } else {
        PB_TRY(allow_shared(predict_rows_packed_kernel<8>, smem));
        predict_rows_packed_kernel<8><<<grid, threads, smem, stream>>>(a);
    }
    count_launch(1);
    PB_LAUNCH_CHECK("predict_rows_packed_kernel");
    return PB_OK;
}

extern "C" int pb_predict_forest(const uint8_t* codes, int64_t n_rows, int64_t pitch_row, int64_t code_bits,
                                 int64_t n_features, const void* trees, int64_t copies, int64_t slot_nodes, int64_t depth,
                                 const int32_t* repeat, int64_t total_repeat, int64_t n_trees, float weight, float* out,
                                 const float* init, void* stream_) {
    PB_REQUIRE(codes && trees && out, "null buffer");
    PB_REQUIRE(code_bits == 4 || code_bits == 8, "code_bits must be 4 or 8");
    PB_REQUIRE(pitch_row >= 16 && pitch_row % 16 == 0, "pitch_row must be a positive multiple of 16");
    PB_REQUIRE(n_features >= 1 && n_features <= pitch_row * (code_bits == 4 ? 2 : 1) && n_features < (1ll << 24),
               "n_features out of range");
    PB_REQUIRE(((uintptr_t)codes % 16) == 0 && ((uintptr_t)trees % 16) == 0, "codes / trees must be 16-byte aligned");
    PB_REQUIRE(slot_nodes >= 4 && slot_nodes <= 256 && slot_nodes % 4 == 0, "slot_nodes must be a multiple of 4 up to 256");
    PB_REQUIRE(depth >= 0 && depth <= 255, "depth out of range");
    PB_REQUIRE(copies >= 1 && copies <= 1024, "copies out of range");
    PB_REQUIRE(n_trees >= 0 && n_trees < (1ll << 31), "n_trees out of range");
    PB_REQUIRE(total_repeat >= 0, "total_repeat out of range");
    cudaStream_t stream = (cudaStream_t)stream_;
    if (n_rows <= 0) return PB_OK;
    if (n_trees == 0) {
        if (init) PB_CUDA_TRY(cudaMemcpyAsync(out, init, (size_t)n_rows * 4, cudaMemcpyDeviceToDevice, stream));
        else PB_CUDA_TRY(cudaMemsetAsync(out, 0, (size_t)n_rows * 4, stream));
        return PB_OK;
    }
    PB_REQUIRE(repeat || (total_repeat % n_trees == 0 && total_repeat / n_trees < (1ll << 31)),
               "without per-tree counts every tree is added total_repeat / n_trees times");
    PredictForestArgs a{codes, n_rows, pitch_row, (int)n_features, static_cast<const uint32_t*>(trees), (int)copies, (int)slot_nodes,
                        (int)depth, repeat, repeat ? 0 : (int)(total_repeat / n_trees), (int)n_trees, weight, out, init, 0, 0};
    // Launch shape: groups of 32 rows per CTA and walkers per group.  Per tree a resident row costs its
    // walkers `depth` steps of about 170 cycles, four trees and walk_warps walkers at a time, and its
    // adder `adds` dependent additions of 4.2 cycles (the two overlap); an SM issues about 10
    // instructions per step and warp and 0.6 per addition, four per cycle, and a batch costs a barrier.
    // The slower of the two sets the time of a wave of CTAs.
    const double adds = (double)total_repeat / (double)n_trees;
    double best = 1e300;
    size_t best_smem = 0;
    for (int g = 1; g <= 8; ++g) {
        for (int ww = kAddGroup / kTreesPerWalker; ww <= 8; ww *= 2) {
            const int threads = forest_threads(g, ww);
            if (threads > 1024) continue;
            const double tb = kTreesPerWalker * ww;
            const int64_t smem = forest_smem(n_features, (int)code_bits, g, ww, slot_nodes);
            if (smem > kForestShared) continue;
            int per_sm = (int)(228 * 1024 / (smem + 1024));
            if (per_sm > 2048 / threads) per_sm = 2048 / threads;
            const double ctas = (double)((n_rows + 32 * g - 1) / (32 * g));
            const double waves = ctas <= 148.0 * per_sm ? 1.0 : ctas / (148.0 * per_sm);
            double here = ctas / 148.0;                 // CTAs an SM holds at a time
            here = here < 1.0 ? 1.0 : (here > per_sm ? per_sm : here);
            const double walk = ((double)depth * 170.0 + 100.0) / tb, sum = adds * 4.2 + 10.0;
            const double issue = here * g * ((10.5 * (double)depth + 12.0) + 0.6 * adds + 8.0) / 4.0;
            const double latency = (walk > sum ? walk : sum) + 80.0 / tb;
            // (every CTA brings the trees in: about 24 bytes a cycle, half of it beside the rest)
            const double cost = waves * ((latency > issue ? latency : issue) + here * (double)slot_nodes * 4.0 / 48.0);
            if (cost < best) {
                best = cost;
                a.groups = g;
                a.walk_warps = ww;
                best_smem = (size_t)smem;
            }
        }
    }
    PB_REQUIRE(a.groups > 0, "a row of %lld features does not fit in shared memory: use pb_predict_rows_packed",
               (long long)n_features);
    static const int* const forced = [] {  // PACKBOOST_FOREST_SHAPE="groups walkers" (tuning)
        static int v[2];
        const char* e = getenv("PACKBOOST_FOREST_SHAPE");
        return (e && sscanf(e, "%d %d", &v[0], &v[1]) == 2) ? v : (const int*)nullptr;
    }();
    if (forced && forced[0] >= 1 && forced[1] >= 1 && forced[1] * kTreesPerWalker % kAddGroup == 0 && forest_threads(forced[0], forced[1]) <= 1024 &&
        forest_smem(n_features, (int)code_bits, forced[0], forced[1], slot_nodes) <= kForestShared) {
        a.groups = forced[0];
        a.walk_warps = forced[1];
        best_smem = (size_t)forest_smem(n_features, (int)code_bits, forced[0], forced[1], slot_nodes);
    }
    const int R = 32 * a.groups;
    const unsigned grid = (unsigned)((n_rows + R - 1) / R);
    const int threads = forest_threads(a.groups, a.walk_warps);
    if (code_bits == 4) {
        PB_TRY(allow_shared(predict_forest_kernel<4>, best_smem, kForestShared));
        predict_forest_kernel<4><<<grid, threads, best_smem, stream>>>(a);
    } else {
        PB_TRY(allow_shared(predict_forest_kernel<8>, best_smem, kForestShared));
        predict_forest_kernel<8><<<grid, threads, best_smem, stream>>>(a);
    }
    count_launch(1);
    PB_LAUNCH_CHECK("predict_forest_kernel");
    return PB_OK;
}

extern "C" int64_t pb_predict_forest_fits(int64_t n_features, int64_t code_bits, int64_t slot_nodes) {
    return forest_smem(n_features, (int)code_bits, 1, kAddGroup / kTreesPerWalker, slot_nodes) <= kForestShared ? 1 : 0;
}

// ---- a whole prediction in one call ----------------------------------------------------------------------

static int64_t up256(int64_t v) { return (v + 255) / 256 * 256; }

// Tables this small are read by the packing kernel from page-locked host memory, and the predictions
// are written there, which saves two copies on the stream (about 10 us of a 64-row call); their codes
// are range-checked on the host.
static const int64_t kTableInPlace = 128 << 10;

struct TablePlan {
    int64_t raw, pitch, in_place, dev_bytes, pinned_bytes, off_codes, off_raw, off_in;
};

static TablePlan table_plan(const pb_model* m, int64_t on_device, int64_t n_rows, int64_t n_features) {
    TablePlan p;
    p.raw = n_rows * n_features * (m->edges ? 4 : 1);
    p.pitch = ((m->code_bits == 4 ? (n_features + 1) / 2 : n_features) + 15) / 16 * 16;
    p.in_place = (!on_device && p.raw <= kTableInPlace) ? 1 : 0;
    p.off_codes = up256(16 + n_rows * 4);   // after the range word and the predictions
    p.off_raw = p.off_codes + up256(n_rows * p.pitch);
    p.dev_bytes = p.off_raw + (on_device || p.in_place ? 0 : up256(p.raw));
    p.off_in = up256(16 + n_rows * 4);
    p.pinned_bytes = p.off_in + (on_device ? 0 : p.in_place ? up256(p.raw) : pb_upload_ring_bytes(p.raw));
    return p;
}

static int check_model(const pb_model* m, int64_t n_rows, int64_t n_features) {
    PB_REQUIRE(m && m->trees && m->n_trees >= 1, "the model has no trees");
    PB_REQUIRE(n_rows >= 1 && n_features >= 1 && n_features < (1ll << 24) && n_rows < (1ll << 40), "bad shape");
    PB_REQUIRE(m->code_bits == 4 || m->code_bits == 8, "code_bits must be 4 or 8");
    return PB_OK;
}

extern "C" int pb_predict_table_bytes(const pb_model* m, int64_t x_on_device, int64_t n_rows, int64_t n_features,
                                      int64_t* dev_bytes, int64_t* pinned_bytes) {
    int rc = check_model(m, n_rows, n_features);
    if (rc) return rc;
    PB_REQUIRE(dev_bytes && pinned_bytes, "null argument");
    const TablePlan p = table_plan(m, x_on_device, n_rows, n_features);
    *dev_bytes = p.dev_bytes;
    *pinned_bytes = p.pinned_bytes;
    return PB_OK;
}

extern "C" int pb_predict_table(const pb_model* m, const void* x, int64_t x_on_device, int64_t n_rows, int64_t n_features,
                                void* dev, int64_t dev_bytes, void* pinned, int64_t pinned_bytes, float* out,
                                int64_t* top, void* stream_) {
    int rc = check_model(m, n_rows, n_features);
    if (rc) return rc;
    PB_REQUIRE(x && dev && pinned && out && top, "null buffer");
    const TablePlan p = table_plan(m, x_on_device, n_rows, n_features);
    PB_REQUIRE(dev_bytes >= p.dev_bytes && pinned_bytes >= p.pinned_bytes, "scratch too small");
    PB_REQUIRE((uintptr_t)dev % 256 == 0 && (uintptr_t)pinned % 16 == 0, "scratch is misaligned");
    cudaStream_t stream = (cudaStream_t)stream_;
    char* d = static_cast<char*>(dev);
    char* h = static_cast<char*>(pinned);
    *top = 0;
    uint32_t* d_top = nullptr;
    const void* src = x;
    float* pred = reinterpret_cast<float*>((p.in_place ? h : d) + 16);
    if (p.in_place) {
        memcpy(h + p.off_in, x, (size_t)p.raw);
        src = h + p.off_in;
        if (!m->edges) {
            const uint8_t* b = static_cast<const uint8_t*>(x);
            uint8_t t = 0;
            for (int64_t i = 0; i < p.raw; ++i) t = b[i] > t ? b[i] : t;
            *top = t;
        }
    } else {
        if (!m->edges) {
            d_top = reinterpret_cast<uint32_t*>(d);
            PB_CUDA_TRY(cudaMemsetAsync(d_top, 0, 16, stream));
        }
        if (!x_on_device) {
            rc = pb_upload(d + p.off_raw, x, p.raw, h + p.off_in, pinned_bytes - p.off_in, stream_);
            src = d + p.off_raw;
        }
    }
    uint8_t* codes = reinterpret_cast<uint8_t*>(d + p.off_codes);
    if (rc == PB_OK)
        rc = pb_pack_rows_top(src, m->edges ? 1 : 0, n_rows, n_features, m->edges, m->n_edges, m->max_bins, codes, p.pitch,
                              m->code_bits, d_top, stream_);
    if (rc == PB_OK)
        rc = pb_predict_forest(codes, n_rows, p.pitch, m->code_bits, n_features, m->trees, m->copies, m->slot_nodes, m->depth,
                               m->repeat, m->total_repeat, m->n_trees, (float)m->weight, pred, nullptr, stream_);
    if (rc == PB_OK && !p.in_place) {
        cudaError_t e = cudaMemcpyAsync(h, d, (size_t)(16 + n_rows * 4), cudaMemcpyDeviceToHost, stream);
        if (e != cudaSuccess) rc = fail_cuda(e, "pb_predict_table");
    }
    // (the scratch is the caller's again after this, also when something failed)
    cudaError_t e = cudaStreamSynchronize(stream);
    if (rc) return rc;
    if (e != cudaSuccess) return fail_cuda(e, "pb_predict_table");
    if (d_top) *top = (int64_t)*reinterpret_cast<uint32_t*>(h);
    memcpy(out, h + 16, (size_t)n_rows * 4);
    return PB_OK;
}

// ---- forests in the one-word form (host) ---------------------------------------------------------------------

// Depths of the nodes of one tree and the words it takes once every path is `depth` splits long; false
// when the tree is not a proper one (children inside the tree and after their parent, ids in range).
static bool tree_depths(const int32_t* feature, const int32_t* threshold, const int32_t* left, const int32_t* right,
                        const uint8_t* is_leaf, int64_t n, std::vector<int32_t>& depth, int32_t* deepest, bool* adjacent) {
    if (n < 1) return false;
    depth.assign((size_t)n, 0);
    for (int64_t i = 0; i < n; ++i) {
        if (is_leaf[i]) continue;
        const int64_t l = left[i], r = right[i];
        if (l <= i || r <= i || l >= n || r >= n || feature[i] < 0 || threshold[i] < 0 || threshold[i] >= 256) return false;
        if (r != l + 1 || feature[i] >= (1 << 16)) *adjacent = false;
        depth[l] = depth[r] = depth[i] + 1;
    }
    // (only nodes that are reached count)
    std::vector<uint8_t> seen((size_t)n, 0);
    seen[0] = 1;
    for (int64_t i = 0; i < n; ++i) {
        if (!seen[i]) {
            depth[i] = -1;
            continue;
        }
        if (is_leaf[i]) *deepest = depth[i] > *deepest ? depth[i] : *deepest;
        else seen[left[i]] = seen[right[i]] = 1;
    }
    return true;
}

static int forest_shape(const int32_t* feature, const int32_t* threshold, const int32_t* left, const int32_t* right,
                        const float* value, const uint8_t* is_leaf, const int32_t* offsets, int64_t n_trees,
                        int64_t* slot_nodes, int64_t* depth_out) {
    PB_REQUIRE(feature && threshold && left && right && value && is_leaf && offsets && slot_nodes && depth_out, "null buffer");
    PB_REQUIRE(n_trees >= 0 && n_trees < (1ll << 31), "n_trees out of range");
    *slot_nodes = 0;
    int32_t deepest = 0;
    bool adjacent = true;
    std::vector<std::vector<int32_t>> depths((size_t)n_trees);
    for (int64_t t = 0; t < n_trees; ++t) {
        const int64_t o = offsets[t], n = (int64_t)offsets[t + 1] - o;
        PB_REQUIRE(n >= 1 && tree_depths(feature + o, threshold + o, left + o, right + o, is_leaf + o, n, depths[t], &deepest, &adjacent),
                   "tree %lld is malformed", (long long)t);
    }
    if (!adjacent || deepest > 16) return PB_OK;
    int64_t most = 0;
    for (int64_t t = 0; t < n_trees; ++t) {
        const int64_t o = offsets[t], n = (int64_t)offsets[t + 1] - o;
        int64_t words = n;
        for (int64_t i = 0; i < n; ++i)
            if (is_leaf[o + i] && depths[t][i] >= 0) words += deepest - depths[t][i];
        most = words > most ? words : most;
        if (most > 256) return PB_OK;
    }
    *slot_nodes = (most + 3) / 4 * 4;
    *depth_out = deepest;
    return PB_OK;
}

static int forest_words(const int32_t* feature, const int32_t* threshold, const int32_t* left, const int32_t* right,
                        const float* value, const uint8_t* is_leaf, const int32_t* offsets, int64_t n_trees,
                        int64_t slot_nodes, int64_t depth, uint32_t* out) {
    PB_REQUIRE(feature && threshold && left && right && value && is_leaf && offsets && out, "null buffer");
    PB_REQUIRE(n_trees >= 0 && n_trees < (1ll << 31) && slot_nodes >= 0, "n_trees or slot_nodes out of range");
    std::vector<int32_t> at;
    memset(out, 0, (size_t)(n_trees * slot_nodes) * 4);
    for (int64_t t = 0; t < n_trees; ++t) {
        const int64_t o = offsets[t], n = (int64_t)offsets[t + 1] - o;
        uint32_t* w = out + t * slot_nodes;
        int32_t deepest = 0;
        bool adjacent = true;
        PB_REQUIRE(n >= 1 && tree_depths(feature + o, threshold + o, left + o, right + o, is_leaf + o, n, at, &deepest, &adjacent) &&
                       adjacent && deepest <= depth,
                   "tree %lld does not have the shape pb_forest_shape found", (long long)t);
        int64_t next = n;   // words of led-on leaves are appended
        for (int64_t i = 0; i < n; ++i) {
            if (at[i] < 0) continue;
            if (!is_leaf[o + i]) {
                w[i] = (uint32_t)feature[o + i] << 16 | (uint32_t)left[o + i] << 8 | (uint32_t)(255 - threshold[o + i]);
                continue;
            }
            int64_t here = i;
            for (int64_t d = at[i]; d < depth; ++d) {
                PB_REQUIRE(next < slot_nodes, "tree %lld needs more than %lld words", (long long)t, (long long)slot_nodes);
                w[here] = (uint32_t)next << 8;
                here = next++;
            }
            memcpy(w + here, value + o + i, 4);
        }
    }
    return PB_OK;
}

extern "C" int pb_forest_shape(const int32_t* feature, const int32_t* threshold, const int32_t* left, const int32_t* right,
                               const float* value, const uint8_t* is_leaf, const int32_t* offsets, int64_t n_trees,
                               int64_t* slot_nodes, int64_t* depth) {
    return no_throw("pb_forest_shape", [&] {
        return forest_shape(feature, threshold, left, right, value, is_leaf, offsets, n_trees, slot_nodes, depth);
    });
}

extern "C" int pb_forest_words(const int32_t* feature, const int32_t* threshold, const int32_t* left, const int32_t* right,
                               const float* value, const uint8_t* is_leaf, const int32_t* offsets, int64_t n_trees,
                               int64_t slot_nodes, int64_t depth, uint32_t* out) {
    return no_throw("pb_forest_words", [&] {
        return forest_words(feature, threshold, left, right, value, is_leaf, offsets, n_trees, slot_nodes, depth, out);
    });
}
