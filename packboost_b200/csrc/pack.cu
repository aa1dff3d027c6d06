// Binning (searchsorted against per-feature edges) and packing of bin codes into the two
// layouts the other kernels read: feature-major (training) and row-major (prediction), each
// with one byte per code or two 4-bit codes per byte.

#include <type_traits>

#include "common.cuh"

namespace pb {

namespace {

constexpr int kTileR = 256;         // rows per tile: one 128-byte line of 4-bit codes per feature
constexpr int kCodeTileF = 128;     // features per tile of byte input: 128 bytes of a row
constexpr int kFloatTileF = 32;     // features per tile of float input: 128 bytes of a row

struct PackArgs {
    const void* x;
    const int32_t* src_rows;        // source row of each destination row, or null: the same
    int64_t n_chunk;
    int64_t n_features;
    int64_t row_offset;
    const float* edges;
    int n_edges;
    int max_bins;
    const int32_t* feature_map;
    uint8_t* codes;
    int64_t pitch;
    uint32_t* top;                  // largest byte seen (atomic maximum), or null
};

// code = number of edges strictly below x (np.searchsorted(edges, x, "left")), clipped to
// max_bins-1; NaN sorts after every edge and gets the last bin.  The edges of a feature are padded
// with +inf to 2^STEPS - 1 entries STRIDE words apart in shared memory, so the search is STEPS
// unconditional probes, each a load at a constant distance from the running address, a comparison
// and a predicated add; the searches of N values are independent and hide each other's latency.  `first`:
// byte offset of a value's lowest edge.
template <int N, int STRIDE, int STEPS>
__device__ __forceinline__ void bins_of(const float* s_edges, const float (&x)[N], const uint32_t (&first)[N], int n_edges,
                                        int max_bins, uint32_t (&code)[N]) {
    uint32_t at[N];
#pragma unroll
    for (int i = 0; i < N; ++i) at[i] = first[i];
#pragma unroll
    for (int s = STEPS - 1; s >= 0; --s) {
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const float e = *reinterpret_cast<const float*>(reinterpret_cast<const char*>(s_edges) + at[i] +
                                                            ((1 << s) - 1) * STRIDE * 4);
            if (e < x[i]) at[i] += (1 << s) * STRIDE * 4;
        }
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const int pos = (int)((at[i] - first[i]) / (STRIDE * 4));
        code[i] = (uint32_t)min((x[i] != x[i]) ? n_edges : pos, max_bins - 1);
    }
}

// m2: two 16-bit maxima (pairs of bytes are compared as 16-bit lanes, which the hardware does in one
// instruction; four byte lanes take about ten)
__device__ __forceinline__ void report_top(uint32_t m2, uint32_t* top) {
    uint32_t m = max(m2 & 0xFFFFu, m2 >> 16);
    m = __reduce_max_sync(0xFFFFFFFFu, m);
    if ((threadIdx.x & 31) == 0 && m > *reinterpret_cast<volatile uint32_t*>(top)) atomicMax(top, m);
}

// Four bytes at `p` (any alignment) of a region that ends at `end`; bytes past the end are zero.
// Only aligned words that hold a byte of the region are read.
__device__ __forceinline__ uint32_t load4(const uint8_t* p, const uint8_t* end) {
    if (p >= end) return 0u;
    const uint32_t m = (uint32_t)(reinterpret_cast<uintptr_t>(p) & 3u);
    const uint8_t* a = p - m;
    const uint32_t lo = __ldg(reinterpret_cast<const uint32_t*>(a));
    const uint32_t hi = (m && a + 4 < end) ? __ldg(reinterpret_cast<const uint32_t*>(a + 4)) : 0u;
    const uint32_t v = __funnelshift_r(lo, hi, 8u * m);
    const int64_t left = end - p;
    return left >= 4 ? v : v & ((1u << (8 * (int)left)) - 1u);
}

// Bytes j of four words as word j.
__device__ __forceinline__ void transpose4(const uint32_t (&t)[4], uint32_t (&o)[4]) {
    const uint32_t a = __byte_perm(t[0], t[1], 0x5140), b = __byte_perm(t[2], t[3], 0x5140);
    const uint32_t c = __byte_perm(t[0], t[1], 0x7362), d = __byte_perm(t[2], t[3], 0x7362);
    o[0] = __byte_perm(a, b, 0x5410);
    o[1] = __byte_perm(a, b, 0x7632);
    o[2] = __byte_perm(c, d, 0x5410);
    o[3] = __byte_perm(c, d, 0x7632);
}

// ---- feature-major, byte input ---------------------------------------------------------------------
// Bound by HBM: n * F bytes in, n * F / 2 out.  A CTA copies 128 bytes of each of 256 rows to shared
// memory with 16-byte asynchronous copies (rows may start on any byte: nine aligned pieces cover
// them), so its whole tile is in flight at once without holding registers.  A lane then takes
// 4 features x 8 rows and turns them over in registers (nibbles of row pairs merged, then a 4 x 4
// byte transposition); the words go through shared memory so that a feature's 256 rows leave as
// whole lines.  1 M x 2 376 codes to
// 4 bits: 0.91 ms, 3.9 TB/s (loads held in registers: 1.39 ms; a byte and a barrier at a time: 2.85).
constexpr int kRowBytes = 144;                // staged bytes of a row: 128 at any of 16 offsets
template <int BITS>
__global__ void __launch_bounds__(256) pack_codes_fm_kernel(PackArgs a) {
    constexpr int W = kTileR * BITS / 32;     // words of a feature's tile rows
    constexpr int P = W + 1;
    extern __shared__ __align__(16) uint32_t tile[];   // [byte j of a lane][lane][P], then the staged rows
    __shared__ uint32_t s_off[kTileR];        // bytes between a row's first staged byte and its first code
    unsigned char* stage = reinterpret_cast<unsigned char*>(tile + kCodeTileF * P);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // neighbouring CTAs take neighbouring features of the same rows: whole rows stream from memory
    const unsigned f_tiles = (unsigned)((a.n_features + kCodeTileF - 1) / kCodeTileF);
    const int64_t f0 = (int64_t)(blockIdx.x % f_tiles) * kCodeTileF;
    const int64_t rt = (int64_t)(blockIdx.x / f_tiles) * kTileR;
    const int nf = (int)min((int64_t)kCodeTileF, a.n_features - f0);
    const int nr = (int)min((int64_t)kTileR, a.n_chunk - rt);
    const uint8_t* x = static_cast<const uint8_t*>(a.x) + f0;
    if (nr < kTileR || nf < kCodeTileF) {     // what is not copied below is code 0
        uint4* z = reinterpret_cast<uint4*>(stage);
        for (int i = threadIdx.x; i < kTileR * kRowBytes / 16; i += 256) z[i] = make_uint4(0u, 0u, 0u, 0u);
    }
    const int my = threadIdx.x < nr ? threadIdx.x : -1;
    s_off[threadIdx.x] = 0u;
    const int64_t my_row = my < 0 ? 0 : (a.src_rows ? (int64_t)__ldg(a.src_rows + rt + my) : rt + my);
    if (my >= 0) s_off[my] = (uint32_t)((reinterpret_cast<uintptr_t>(x) + (uintptr_t)(my_row * a.n_features)) & 15u);
    __syncthreads();
    const uint32_t stage_at = (uint32_t)__cvta_generic_to_shared(stage);
    if (a.src_rows) {
        if (my >= 0) {
            const uint8_t* p = x + my_row * a.n_features - s_off[my];
            const int parts = (int)(s_off[my] + nf + 15) >> 4;   // pieces that hold a code
            for (int j = 0; j < parts; ++j)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(stage_at + my * kRowBytes + 16 * j), "l"(p + 16 * j) : "memory");
        }
    } else {
        for (int c = threadIdx.x; c < nr * 9; c += 256) {
            const int r = c / 9, j = c - r * 9;
            const uint32_t off = s_off[r];
            if (16 * j < (int)off + nf)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(stage_at + r * kRowBytes + 16 * j),
                             "l"(x + (rt + r) * a.n_features - off + 16 * j) : "memory");
        }
    }
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();

    const int keep = nf - 4 * lane;           // bytes of this lane that are features
    const uint32_t mask = keep >= 4 ? 0xFFFFFFFFu : (keep <= 0 ? 0u : (1u << (8 * keep)) - 1u);
    uint32_t top = 0u, top2 = 0u;             // maxima of the even and of the odd bytes, as 16-bit pairs
#pragma unroll 1
    for (int it = 0; it < 4; ++it) {
        const int g = warp * 4 + it;          // group of eight rows
        uint32_t w[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int r = g * 8 + i;
            const uint32_t off = s_off[r];
            const uint32_t* q = reinterpret_cast<const uint32_t*>(stage + r * kRowBytes + (off & ~3u)) + lane;
            // (the second word of the last lane may lie past the row's slot: it is shifted out then)
            w[i] = __funnelshift_r(q[0], q[1], 8u * (off & 3u)) & mask;
            if (r >= nr) w[i] = 0u;
            top = __vmaxu2(top, w[i] & 0x00FF00FFu);
            top2 = __vmaxu2(top2, (w[i] >> 8) & 0x00FF00FFu);
        }
        uint32_t t[4], o[4];
        if (BITS == 4) {
#pragma unroll
            for (int i = 0; i < 4; ++i) t[i] = (w[2 * i] & 0x0F0F0F0Fu) | ((w[2 * i + 1] & 0x0F0F0F0Fu) << 4);
            transpose4(t, o);
#pragma unroll
            for (int j = 0; j < 4; ++j) tile[(j * 32 + lane) * P + g] = o[j];
        } else {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
#pragma unroll
                for (int i = 0; i < 4; ++i) t[i] = w[4 * h + i];
                transpose4(t, o);
#pragma unroll
                for (int j = 0; j < 4; ++j) tile[(j * 32 + lane) * P + 2 * g + h] = o[j];
            }
        }
    }
    if (a.top) report_top(__vmaxu2(top, top2), a.top);
    __syncthreads();
    for (int fl = warp; fl < nf; fl += 8) {
        const int frow = a.feature_map ? a.feature_map[f0 + fl] : (int)(f0 + fl);
        if (frow < 0) continue;
        uint32_t* dst = reinterpret_cast<uint32_t*>(a.codes + (int64_t)frow * a.pitch + (a.row_offset + rt) * BITS / 8);
        const uint32_t* src = tile + ((fl & 3) * 32 + (fl >> 2)) * P;
#pragma unroll
        for (int h = 0; h < W / 32; ++h) dst[h * 32 + lane] = src[h * 32 + lane];
    }
}

// ---- feature-major, float input --------------------------------------------------------------------
// A lane owns a feature, a warp eight rows at a time; the edges of the 32 features sit in shared
// memory with the feature as the bank.  Bound by the probes (steps per value, one shared load each);
// 500 000 x 256 with 127 edges:
// 275 us, 2.3 TB/s (334 with the probe address computed from the position).
template <int BITS, int STEPS>
__global__ void __launch_bounds__(256) pack_floats_fm_kernel(PackArgs a) {
    constexpr int W = kTileR * BITS / 32;
    constexpr int P = W + 1;
    __shared__ uint32_t tile[kFloatTileF * P];
    extern __shared__ float s_edges[];        // [2^STEPS - 1][32]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned f_tiles = (unsigned)((a.n_features + kFloatTileF - 1) / kFloatTileF);
    const int64_t f0 = (int64_t)(blockIdx.x % f_tiles) * kFloatTileF;
    const int64_t f = f0 + lane;
    const int64_t rt = (int64_t)(blockIdx.x / f_tiles) * kTileR;
    const bool f_ok = f < a.n_features;
#pragma unroll 16
    for (int i = warp; i < (1 << STEPS) - 1; i += 8)
        s_edges[i * 32 + lane] = (f_ok && i < a.n_edges) ? __ldg(a.edges + (int64_t)i * a.n_features + f) : INFINITY;
    __syncthreads();
    const float* x = static_cast<const float*>(a.x);
    const uint32_t edges_at = 4u * (uint32_t)lane;
    for (int it = 0; it < 4; ++it) {
        const int g = warp * 4 + it;
        float v[8];
        uint32_t e[8], c[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int64_t r = rt + g * 8 + i;
            e[i] = edges_at;
            v[i] = 0.f;
            if (f_ok && r < a.n_chunk)
                v[i] = __ldg(x + (a.src_rows ? (int64_t)__ldg(a.src_rows + r) : r) * a.n_features + f);
        }
        bins_of<8, 32, STEPS>(s_edges, v, e, a.n_edges, a.max_bins, c);
        const int64_t left = a.n_chunk - rt - g * 8;   // rows past the end are code 0
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (i >= left) c[i] = 0u;
        if (BITS == 4) {
            uint32_t w = 0u;
#pragma unroll
            for (int i = 0; i < 8; ++i) w |= (c[i] & 0xFu) << (4 * i);
            tile[lane * P + g] = w;
        } else {
            tile[lane * P + 2 * g] = c[0] | (c[1] << 8) | (c[2] << 16) | (c[3] << 24);
            tile[lane * P + 2 * g + 1] = c[4] | (c[5] << 8) | (c[6] << 16) | (c[7] << 24);
        }
    }
    __syncthreads();
    for (int fl = warp; fl < kFloatTileF; fl += 8) {
        if (f0 + fl >= a.n_features) break;
        const int frow = a.feature_map ? a.feature_map[f0 + fl] : (int)(f0 + fl);
        if (frow < 0) continue;
        uint32_t* dst = reinterpret_cast<uint32_t*>(a.codes + (int64_t)frow * a.pitch + (a.row_offset + rt) * BITS / 8);
#pragma unroll
        for (int h = 0; h < W / 32; ++h) dst[h * 32 + lane] = tile[fl * P + h * 32 + lane];
    }
}

// ---- row-major (prediction) ------------------------------------------------------------------------

struct PackRowsArgs {
    const void* x;
    int64_t n_rows;
    int64_t n_features;
    const float* edges;
    int n_edges;
    int max_bins;
    uint8_t* out;
    int64_t pitch_row;
    uint32_t* top;
    int rows_per_cta;
};

// Byte input: `lanes` lanes (a power of two) share a row, a lane packs one output word (8 or 4
// codes) per step.  Bound by HBM; 1 M x 2 376 codes: 0.73 ms, 4.9 TB/s
// (1.34 with two loads in flight per lane).
template <int BITS>
__global__ void __launch_bounds__(256) pack_code_rows_kernel(PackRowsArgs a, int lanes) {
    constexpr int PER = 32 / BITS;            // codes per output word
    const int sub = threadIdx.x & (lanes - 1);
    const int words = (int)(a.pitch_row / 4);
    const int64_t step = (int64_t)gridDim.x * (blockDim.x / lanes);
    uint32_t top = 0u;
    for (int64_t r = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / lanes; r < a.n_rows; r += step) {
        const uint8_t* row = static_cast<const uint8_t*>(a.x) + r * a.n_features;
        const uint8_t* end = row + a.n_features;
        uint32_t* out = reinterpret_cast<uint32_t*>(a.out + r * a.pitch_row);
        const int full = (int)(a.n_features / PER);   // words all of whose codes exist
        auto put = [&](int w, uint2 v) {
            if (BITS == 8) {
                top = __vmaxu2(top, __vmaxu2(v.x & 0x00FF00FFu, (v.x >> 8) & 0x00FF00FFu));
                out[w] = v.x;
            } else {
                top = __vmaxu2(top, __vmaxu2(v.x & 0x00FF00FFu, (v.x >> 8) & 0x00FF00FFu));
                top = __vmaxu2(top, __vmaxu2(v.y & 0x00FF00FFu, (v.y >> 8) & 0x00FF00FFu));
                // codes of bytes 0, 1, 2, 3 to nibbles 0 .. 3 of a half word
                const uint32_t lo = v.x & 0x0F0F0F0Fu, hi = v.y & 0x0F0F0F0Fu;
                out[w] = __byte_perm(lo | (lo >> 4), hi | (hi >> 4), 0x6420);
            }
        };
        const uint32_t m = (uint32_t)(reinterpret_cast<uintptr_t>(row) % PER);
        if (m == 0) {
#pragma unroll 8
            for (int w = sub; w < full; w += lanes) {
                if (BITS == 8) put(w, make_uint2(__ldg(reinterpret_cast<const uint32_t*>(row) + w), 0u));
                else put(w, __ldg(reinterpret_cast<const uint2*>(row) + w));
            }
        } else {  // aligned words, shifted together
            const uint32_t sh = 8u * (uint32_t)(reinterpret_cast<uintptr_t>(row) & 3u);
            const uint32_t* q = reinterpret_cast<const uint32_t*>(row - (sh >> 3));
            const int n_q = (int)((end - reinterpret_cast<const uint8_t*>(q) + 3) / 4);  // words that hold a byte of the row
#pragma unroll 8
            for (int w = sub; w < full; w += lanes) {
                const int i = w * (PER / 4);
                const uint32_t q0 = __ldg(q + i), q1 = __ldg(q + min(i + 1, n_q - 1));
                if (BITS == 8) put(w, make_uint2(__funnelshift_r(q0, q1, sh), 0u));
                else put(w, make_uint2(__funnelshift_r(q0, q1, sh), __funnelshift_r(q1, __ldg(q + min(i + 2, n_q - 1)), sh)));
            }
        }
        for (int w = full + (sub + lanes - full % lanes) % lanes; w < words; w += lanes) {
            const uint8_t* p = row + (int64_t)w * PER;
            put(w, make_uint2(load4(p, end), BITS == 8 ? 0u : load4(p + 4, end)));
        }
    }
    if (a.top) report_top(top, a.top);
}

// Float input: a lane owns four consecutive features of a tile of 128 and takes four rows at a time
// (sixteen independent searches); the edges of the tile sit in shared memory, a lane's features 32
// words apart.  Bound by the probes; 300 007 x 256 with 127 edges: 120 us, 3.2 TB/s (514 with the edges
// in global memory).
template <int BITS, int STEPS>
__global__ void __launch_bounds__(256) pack_float_rows_kernel(PackRowsArgs a) {
    extern __shared__ float s_edges[];        // [2^STEPS - 1][4][32]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t f0 = (int64_t)blockIdx.y * 128;
    const int n_pad = (1 << STEPS) - 1;
#pragma unroll 16
    for (int i = threadIdx.x; i < n_pad * 128; i += 256) {
        const int e = i >> 7, fl = i & 127;
        const int64_t f = f0 + fl;
        s_edges[e * 128 + (fl & 3) * 32 + (fl >> 2)] =
            (f < a.n_features && e < a.n_edges) ? __ldg(a.edges + (int64_t)e * a.n_features + f) : INFINITY;
    }
    __syncthreads();
    const int64_t f = f0 + 4 * lane;
    const int64_t out_byte = f * BITS / 8;
    const int n_mine = (int)max((int64_t)0, min((int64_t)4, a.n_features - f));
    const bool even = (a.n_features & 3) == 0 && (reinterpret_cast<uintptr_t>(a.x) & 15) == 0;
    const uint32_t edges_at = 4u * (uint32_t)lane;
    const int64_t r0 = (int64_t)blockIdx.x * a.rows_per_cta;
    const int64_t r1 = min(a.n_rows, r0 + a.rows_per_cta);
    for (int64_t rb = r0 + warp * 4; rb < r1; rb += 32) {
        float v[16];
        uint32_t e[16], c[16];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float* row = static_cast<const float*>(a.x) + (rb + i) * a.n_features + f;
            if (rb + i < r1 && n_mine == 4 && even) {
                const float4 q = __ldg(reinterpret_cast<const float4*>(row));
                v[4 * i] = q.x; v[4 * i + 1] = q.y; v[4 * i + 2] = q.z; v[4 * i + 3] = q.w;
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j) v[4 * i + j] = (rb + i < r1 && j < n_mine) ? __ldg(row + j) : 0.f;
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) e[4 * i + j] = edges_at + j * 128;
        }
        bins_of<16, 128, STEPS>(s_edges, v, e, a.n_edges, a.max_bins, c);
        if (out_byte >= a.pitch_row) continue;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (rb + i >= r1) break;
            uint32_t w = 0u;
#pragma unroll
            for (int j = 0; j < 4; ++j) w |= (j < n_mine ? (BITS == 4 ? c[4 * i + j] & 0xFu : c[4 * i + j]) : 0u) << (BITS * j);
            uint8_t* dst = a.out + (rb + i) * a.pitch_row + out_byte;
            if (BITS == 4) *reinterpret_cast<uint16_t*>(dst) = (uint16_t)w;
            else *reinterpret_cast<uint32_t*>(dst) = w;
        }
    }
}

// calls fn(std::integral_constant<int, steps>) with the probes a search over n_edges edges takes
template <typename F>
int with_steps(int n_edges, F fn) {
    int s = 1;
    while ((1 << s) - 1 < n_edges) ++s;
    switch (s) {
        case 1: return fn(std::integral_constant<int, 1>());
        case 2: return fn(std::integral_constant<int, 2>());
        case 3: return fn(std::integral_constant<int, 3>());
        case 4: return fn(std::integral_constant<int, 4>());
        case 5: return fn(std::integral_constant<int, 5>());
        case 6: return fn(std::integral_constant<int, 6>());
        case 7: return fn(std::integral_constant<int, 7>());
        default: return fn(std::integral_constant<int, 8>());
    }
}

template <int BITS>
int pack_fm(const PackArgs& a, bool f32, cudaStream_t stream) {
    if (a.n_chunk <= 0 || a.n_features <= 0) return PB_OK;
    const int tile_f = f32 ? kFloatTileF : kCodeTileF;
    const int64_t blocks = (a.n_chunk + kTileR - 1) / kTileR * ((a.n_features + tile_f - 1) / tile_f);
    if (blocks >= (1ll << 31)) return fail_arg("table too large to pack in one call");
    int rc = PB_OK;
    if (f32) {
        rc = with_steps(a.n_edges, [&](auto steps) {
            constexpr int S = decltype(steps)::value;
            const size_t smem = sizeof(float) * (size_t)((1 << S) - 1) * kFloatTileF;
            pack_floats_fm_kernel<BITS, S><<<(unsigned)blocks, 256, smem, stream>>>(a);
            return PB_OK;
        });
    } else {
        const size_t smem = sizeof(uint32_t) * kCodeTileF * (kTileR * BITS / 32 + 1) + (size_t)kTileR * kRowBytes + 16;
        PB_TRY(allow_shared(pack_codes_fm_kernel<BITS>, smem));
        pack_codes_fm_kernel<BITS><<<(unsigned)blocks, 256, smem, stream>>>(a);
    }
    if (rc) return rc;
    count_launch(1);
    PB_LAUNCH_CHECK("pack_fm");
    return PB_OK;
}

template <int BITS>
int pack_rows(PackRowsArgs a, bool f32, cudaStream_t stream) {
    int rc = PB_OK;
    if (f32) {
        const int64_t tiles = (a.pitch_row * (8 / BITS) + 127) / 128;
        // a CTA reads its tile's edges once: enough CTAs for three per SM, no fewer than 32 rows each
        int64_t per = (a.n_rows * tiles + 148 * 3 - 1) / (148 * 3);
        per = (per + 31) / 32 * 32;
        a.rows_per_cta = (int)(per < 32 ? 32 : (per > (1 << 20) ? (1 << 20) : per));
        dim3 grid((unsigned)((a.n_rows + a.rows_per_cta - 1) / a.rows_per_cta), (unsigned)tiles);
        if (grid.y > 65535u) return fail_arg("too many features to pack");
        rc = with_steps(a.n_edges, [&](auto steps) {
            constexpr int S = decltype(steps)::value;
            const size_t smem = sizeof(float) * (size_t)((1 << S) - 1) * 128;
            PB_TRY(allow_shared(pack_float_rows_kernel<BITS, S>, smem));
            pack_float_rows_kernel<BITS, S><<<grid, 256, smem, stream>>>(a);
            return PB_OK;
        });
    } else {
        int lanes = 1;
        while (lanes < 32 && lanes < a.pitch_row / 4) lanes *= 2;
        int64_t blocks = (a.n_rows * lanes + 255) / 256;
        if (blocks > 148 * 8) blocks = 148 * 8;
        pack_code_rows_kernel<BITS><<<(unsigned)blocks, 256, 0, stream>>>(a, lanes);
    }
    if (rc) return rc;
    count_launch(1);
    PB_LAUNCH_CHECK("pack_rows");
    return PB_OK;
}

}  // namespace
}  // namespace pb

using namespace pb;

static int check_pack(const void* x, int64_t n_chunk, int64_t n_features, int64_t row_offset, const uint8_t* codes,
                      int64_t pitch, int64_t code_bits, int64_t max_bins) {
    PB_REQUIRE(x && codes, "null buffer");
    PB_REQUIRE(n_chunk >= 0 && n_features >= 1, "bad shape");
    PB_REQUIRE(code_bits == 4 || code_bits == 8, "code_bits must be 4 or 8");
    PB_REQUIRE(code_bits == 8 || max_bins <= 16, "4-bit codes need max_bins <= 16");
    PB_REQUIRE(row_offset % 256 == 0, "row_offset must be a multiple of 256");
    PB_REQUIRE(pitch % 128 == 0, "pitch must be a multiple of 128");
    const int64_t rows_cover = pitch * (code_bits == 4 ? 2 : 1);
    PB_REQUIRE(row_offset + (n_chunk + 255) / 256 * 256 <= rows_cover, "chunk exceeds the padded row range");
    return PB_OK;
}

extern "C" int pb_pack_table(const void* x, int64_t x_is_f32, const int32_t* src_rows, int64_t n_chunk, int64_t n_features,
                             int64_t row_offset, const float* edges, int64_t n_edges, int64_t max_bins,
                             const int32_t* feature_map, uint8_t* codes, int64_t pitch, int64_t code_bits,
                             uint32_t* top, void* stream) {
    int rc = check_pack(x, n_chunk, n_features, row_offset, codes, pitch, code_bits, max_bins);
    if (rc) return rc;
    PB_REQUIRE(!x_is_f32 || (edges && n_edges >= 1 && n_edges <= 255 && max_bins >= 2 && max_bins <= 256), "bad edges / max_bins");
    PackArgs a{x, src_rows, n_chunk, n_features, row_offset, edges, (int)n_edges, (int)max_bins, feature_map, codes, pitch, top};
    return code_bits == 4 ? pack_fm<4>(a, x_is_f32 != 0, (cudaStream_t)stream) : pack_fm<8>(a, x_is_f32 != 0, (cudaStream_t)stream);
}

extern "C" int pb_bin_pack_f32(const float* x, int64_t n_chunk, int64_t n_features, int64_t row_offset,
                               const float* edges, int64_t n_edges, int64_t max_bins, const int32_t* feature_map,
                               uint8_t* codes, int64_t pitch, int64_t code_bits, void* stream) {
    return pb_pack_table(x, 1, nullptr, n_chunk, n_features, row_offset, edges, n_edges, max_bins, feature_map, codes, pitch,
                         code_bits, nullptr, stream);
}

extern "C" int pb_pack_codes_u8(const uint8_t* x, int64_t n_chunk, int64_t n_features, int64_t row_offset,
                                const int32_t* feature_map, uint8_t* codes, int64_t pitch, int64_t code_bits,
                                void* stream) {
    return pb_pack_table(x, 0, nullptr, n_chunk, n_features, row_offset, nullptr, 0, code_bits == 4 ? 16 : 256, feature_map,
                         codes, pitch, code_bits, nullptr, stream);
}

extern "C" int pb_pack_rows_top(const void* x, int64_t x_is_f32, int64_t n_rows, int64_t n_features, const float* edges,
                                int64_t n_edges, int64_t max_bins, uint8_t* out, int64_t pitch_row, int64_t code_bits,
                                uint32_t* top, void* stream) {
    PB_REQUIRE(x && out, "null buffer");
    PB_REQUIRE(code_bits == 4 || code_bits == 8, "code_bits must be 4 or 8");
    PB_REQUIRE(code_bits == 8 || max_bins <= 16, "4-bit codes need max_bins <= 16");
    const int64_t need = (code_bits == 4) ? (n_features + 1) / 2 : n_features;
    PB_REQUIRE(pitch_row >= need && pitch_row % 16 == 0, "pitch_row must cover a row and be a multiple of 16");
    PB_REQUIRE(pitch_row < (1ll << 31), "pitch_row out of range");
    PB_REQUIRE(!x_is_f32 || (edges && n_edges >= 1), "float input needs edges");
    // (edges ascend: those past max_bins - 1 only raise codes that are cut to max_bins - 1)
    if (max_bins >= 2 && n_edges > max_bins - 1) n_edges = max_bins - 1;
    PB_REQUIRE(!x_is_f32 || n_edges <= 255, "float input takes up to 255 edges");
    PB_REQUIRE(((uintptr_t)out % 4) == 0, "out must be 4-byte aligned");
    if (n_rows <= 0) return PB_OK;
    PackRowsArgs a{x, n_rows, n_features, edges, (int)n_edges, (int)max_bins, out, pitch_row, top, 0};
    return code_bits == 4 ? pack_rows<4>(a, x_is_f32 != 0, (cudaStream_t)stream) : pack_rows<8>(a, x_is_f32 != 0, (cudaStream_t)stream);
}

extern "C" int pb_pack_rows(const void* x, int64_t x_is_f32, int64_t n_rows, int64_t n_features, const float* edges,
                            int64_t n_edges, int64_t max_bins, uint8_t* out, int64_t pitch_row, int64_t code_bits,
                            void* stream) {
    return pb_pack_rows_top(x, x_is_f32, n_rows, n_features, edges, n_edges, max_bins, out, pitch_row, code_bits, nullptr,
                            stream);
}
