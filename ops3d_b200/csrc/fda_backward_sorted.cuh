// Cell-sorted backward for 16-bit values with 16, 32, 48 or 64 channels per head.
//
// Every sampling point of a call is sorted by the cell of the pyramid it falls in (and its head); the sorted list is
// then walked run by run of equal cells.  The eight value rows of a cell are read, and its eight rows of the fp32
// gradient image added to, once per RUN instead of once per POINT, and inside a run everything is small matrix products.
//
// Why: a (cell, head) row receives Q*K / cells contributions (9 / 73 / 584 on a 32x64x256 / 16x32x128 / 8x16x64
// pyramid with K = 8 points per level and one query per cell), and the plain and the slab-binned kernels are bound by
// exactly those gathers and reductions (the request path from the SMs to L2), not by HBM.
//
//   fda_sort_clear_kernel     zeroes the counters, one per (batch, level, head, base cell)
//   fda_sort_count_kernel     rows staged like in fda_backward_kernel; rank of every point inside its bin (the one atomic
//                             per point), soft-max statistics of the row
//   fda_scan_*                exclusive scan of the counters (three small kernels, no waiting between blocks)
//   fda_sort_fill_kernel      position = start of the bin + rank; files the point there as one 32-byte record
//   fda_sorted_walk_kernel    grid (x, batch): warps walk spans of the list of the launch's levels; the points' results
//                             {d/dx, d/dy, d/dz, dalpha} in list order
//   fda_sort_finalize_kernel  per row: its points' results, soft-max backward, finished row of grad_sampling_loc_attn
//
// Bins are ordered (batch, level, head, cell): a region of one head reads one head's grad_output rows at random.  A base
// cell may be -1 along an axis (only its upper corners lie inside), so a level of W x H x D cells has (W+1)(H+1)(D+1)
// bins: every point of a bin has the same eight corners.
//
// A launch over a level range that is not the first of a sequence (`resume`) re-uses the list made by the first.
// Nothing here waits on another block.  No counterpart in the reference (its backward is one thread group per query
// and head with atomicAdd per corner and channel, csrc/cuda/flash_deform_col2im_cuda.cuh:248-429).
#pragma once

#include "fda_backward.cuh"
#include "fda_sort_record.cuh"

namespace fda {

constexpr int kScanItems = 8;                         // counters per thread of a scan block
constexpr int kScanThreads = 1024;
constexpr int kScanTile = kScanItems * kScanThreads;  // counters per scan block
constexpr unsigned int kNoPosition = 0xffffffffu;     // a point without a corner inside its level
constexpr unsigned int kNotFinite = 0xfffffff0u;      // the same, and axes (bits x, y, z) whose position is not finite

// Bins of one batch element: level l's start at first[l], head g's inside it at g * cells[l].  first[L] = all of them.
// Bins of a coarse level lie stride[l] counters apart (the ones between stay empty): a level of 21 cells takes 5.7 M atomics
// on 36 lines otherwise, and those on one line are served one after the other (count pass over 28.7 M points 1055 -> 544 us).
struct SortBins {
    unsigned int first[kMaxLevels + 1], cells[kMaxLevels], stride[kMaxLevels];
};
constexpr unsigned int kSpreadBins = 4096;  // counters per head that a coarse level is spread over, at most 32 per bin
__device__ __forceinline__ void build_sort_bins(SortBins &s, const int64_t *shapes, int L, int G, unsigned int spread) {
    unsigned int at = 0;
    for (int l = 0; l < L; ++l) {
        const unsigned int bins = (unsigned int)(shapes[3 * l] + 1) * (unsigned int)(shapes[3 * l + 1] + 1) * (unsigned int)(shapes[3 * l + 2] + 1);
        unsigned int stride = 1;
        while (stride < 32u && bins * stride * 2u <= spread) stride *= 2u;
        s.first[l] = at;
        s.stride[l] = stride;
        s.cells[l] = bins * stride;
        at += s.cells[l] * (unsigned int)G;
    }
    s.first[L] = at;
}

// Base cell of a point from its normalised coordinates, and whether any corner lies inside the level.  A NaN position is
// cell 0, as in the plain kernel's conversion, with fractions of NaN.
struct BaseCell {
    bool ok;
    int x, y, z;        // in [-1, size-1] when ok
    float fx, fy, fz;   // fraction towards the upper corner: upper weight f, lower 1 - f (in range the same value as (floor + 1) - v)
};
__device__ __forceinline__ BaseCell base_cell(const LevelGeom &lv, float x, float y, float z) {
    const float xv = unnormalize(x, lv.fW), yv = unnormalize(y, lv.fH), zv = unnormalize(z, lv.fD);
    const float xf = floorf(xv), yf = floorf(yv), zf = floorf(zv);
    BaseCell c;
    c.x = (int)xf; c.y = (int)yf; c.z = (int)zf;  // saturates
    // an axis has a corner in range iff floor in [-1, size-1]
    c.ok = (unsigned int)c.x + 1u <= (unsigned int)lv.W && (unsigned int)c.y + 1u <= (unsigned int)lv.H && (unsigned int)c.z + 1u <= (unsigned int)lv.D;
    c.fx = __fsub_rn(xv, xf); c.fy = __fsub_rn(yv, yf); c.fz = __fsub_rn(zv, zf);
    return c;
}
// Of a point that is not filed: infinite positions leave weights of infinity minus infinity times zero (the fraction is
// NaN), which its gradients have to show.
__device__ __forceinline__ unsigned int unfiled_code(const BaseCell &c) {
    const unsigned int bad = (isfinite(c.fx) ? 0u : 1u) | (isfinite(c.fy) ? 0u : 2u) | (isfinite(c.fz) ? 0u : 4u);
    return bad ? kNotFinite + bad : kNoPosition;
}
__device__ __forceinline__ unsigned int bin_of(const LevelGeom &lv, const BaseCell &c) {  // inside its level and head
    return ((unsigned int)(c.z + 1) * (unsigned int)(lv.H + 1) + (unsigned int)(c.y + 1)) * (unsigned int)(lv.W + 1) + (unsigned int)(c.x + 1);
}

__global__ void __launch_bounds__(256) fda_sort_clear_kernel(const Problem p) {
    __shared__ SortBins bins;
    if (threadIdx.x == 0) build_sort_bins(bins, p.shapes, p.L, p.G, p.sort_spread);
    __syncthreads();
    const size_t n = (size_t)bins.first[p.L] * p.B + 1;  // one more: after the scan it holds the length of the list
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; 4 * i < n; i += (size_t)gridDim.x * blockDim.x) {
        if (4 * i + 4 <= n) reinterpret_cast<uint4 *>(p.sort_counters)[i] = make_uint4(0u, 0u, 0u, 0u);
        else
            for (size_t k = 4 * i; k < n; ++k) p.sort_counters[k] = 0u;
    }
}

// What the passes tell each other about a row lies where its gradient will: the first 4*L*K of the 8*L*K or more bytes of
// its row of grad_sampling_loc_attn hold the rank of every point inside its bin, then its position in the list
// (kNotFinite and above: not filed); the next eight its soft-max statistics {max, 1 / sum}.
template <typename PT>
__device__ __forceinline__ unsigned int *row_slots(const Problem &p, size_t rowg) {
    return reinterpret_cast<unsigned int *>(static_cast<PT *>(p.grad_packed) + rowg * (size_t)(4 * p.LK));
}
template <typename PT>
__global__ void __launch_bounds__(kThreads) fda_sort_count_kernel(const Problem p) {
    __shared__ LevelGeom geom[kMaxLevels];
    __shared__ SortBins bins;
    extern __shared__ __align__(16) float smem_tile[];
    const int tid = threadIdx.x;
    if (tid == 0) {
        build_level_table(geom, p.shapes, p.lsi, p.L, p.GD, p.value_elem_bytes, false, 0ull);
        build_sort_bins(bins, p.shapes, p.L, p.G, p.sort_spread);
    }
    const int b = blockIdx.y;
    const int gs = 1 << p.gs_log2;
    const int lane = tid & 31, warp = tid >> 5;
    const int lane_c = tid & (gs - 1);
    const int rows_per_block = (int)blockDim.x >> p.gs_log2;
    const int rows_per_warp = 32 >> p.gs_log2;
    const int row = blockIdx.x * rows_per_block + (tid >> p.gs_log2);
    const bool row_ok = row < p.rows_per_b;
    const int LK = p.LK;
    const int first = blockIdx.x * rows_per_block + warp * rows_per_warp;
    float *wtile = smem_tile + warp * rows_per_warp * p.row_stride;
    int nrows = p.rows_per_b - first;
    nrows = nrows < 0 ? 0 : (nrows > rows_per_warp ? rows_per_warp : nrows);
    stage_rows<PT>(static_cast<const PT *>(p.packed) + ((size_t)b * p.rows_per_b + first) * (size_t)(4 * LK), wtile, nrows,
                   LK, p.row_stride, lane);
    __syncthreads();  // level table and this warp's tile visible
    float *trow = wtile + (lane >> p.gs_log2) * p.row_stride;
    const unsigned int g = row_ok ? (unsigned int)(row % p.G) : 0u;
    unsigned int *counters = p.sort_counters + (size_t)b * bins.first[p.L];
    float m = -INFINITY;
    for (int i = lane_c; i < LK; i += gs) m = fmaxf(m, row_ok ? trow[3 * LK + i] : 0.f);
    for (int mask = gs >> 1; mask > 0; mask >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, mask));
    float s = 0.f;
    for (int i = lane_c; i < LK; i += gs) s += row_ok ? __expf(trow[3 * LK + i] - m) : 0.f;
    for (int mask = gs >> 1; mask > 0; mask >>= 1) s += __shfl_xor_sync(0xffffffffu, s, mask);
    if (row_ok && lane_c == 0)
        *reinterpret_cast<float2 *>(row_slots<PT>(p, (size_t)b * p.rows_per_b + row) + LK) = make_float2(m, 1.0f / s);
    // Eight points at a time: all requests go out before the first answer is needed.  The ranks take the place of the
    // logits in the tile (a lane overwrites only slots it owns).
    constexpr int kBatch = 8;
    for (int i0 = lane_c; row_ok && i0 < LK; i0 += kBatch * gs) {
        unsigned int rank[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            const int i = i0 + u * gs;
            rank[u] = kNoPosition;
            if (i < LK) {
                const int l = (i >> 2) >> p.k_shift;
                const LevelGeom lv = geom[l];
                const BaseCell c = base_cell(lv, trow[3 * i], trow[3 * i + 1], trow[3 * i + 2]);
                if (!c.ok) rank[u] = unfiled_code(c);
                else rank[u] = atomicAdd(counters + bins.first[l] + g * bins.cells[l] + bin_of(lv, c) * bins.stride[l], 1u);
            }
        }
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            const int i = i0 + u * gs;
            if (i < LK) trow[3 * LK + i] = __uint_as_float(rank[u]);
        }
    }
    __syncwarp();
    const float inv_vec = 4.0f / (float)LK;
    for (int v = lane; v < nrows * (LK >> 2); v += 32) {
        const int r = row_of_vector(v, inv_vec);
        const int c = (v - r * (LK >> 2)) * 4;
        *reinterpret_cast<float4 *>(row_slots<PT>(p, (size_t)b * p.rows_per_b + first + r) + c) =
            *reinterpret_cast<const float4 *>(wtile + r * p.row_stride + 3 * LK + c);
    }
}

// Files every point at its position: start of its bin + rank, so nothing here depends on the answer of an atomic.  Rows
// are staged like in the count pass; the position takes the place of the rank.
template <typename PT>
__global__ void __launch_bounds__(kThreads) fda_sort_fill_kernel(const Problem p) {
    __shared__ LevelGeom geom[kMaxLevels];
    __shared__ SortBins bins;
    extern __shared__ __align__(16) float smem_tile[];
    const int tid = threadIdx.x;
    if (tid == 0) {
        build_level_table(geom, p.shapes, p.lsi, p.L, p.GD, p.value_elem_bytes, false, 0ull);
        build_sort_bins(bins, p.shapes, p.L, p.G, p.sort_spread);
    }
    const int b = blockIdx.y;
    const int gs = 1 << p.gs_log2;
    const int lane = tid & 31, warp = tid >> 5;
    const int lane_c = tid & (gs - 1);
    const int rows_per_block = (int)blockDim.x >> p.gs_log2;
    const int rows_per_warp = 32 >> p.gs_log2;
    const int row = blockIdx.x * rows_per_block + (tid >> p.gs_log2);
    const int LK = p.LK;
    const int first = blockIdx.x * rows_per_block + warp * rows_per_warp;
    float *wtile = smem_tile + warp * rows_per_warp * p.row_stride;
    int nrows = p.rows_per_b - first;
    nrows = nrows < 0 ? 0 : (nrows > rows_per_warp ? rows_per_warp : nrows);
    stage_rows<PT>(static_cast<const PT *>(p.packed) + ((size_t)b * p.rows_per_b + first) * (size_t)(4 * LK), wtile, nrows,
                   LK, p.row_stride, lane);
    __syncthreads();  // level table and this warp's tile visible
    const unsigned int *starts = p.sort_counters + (size_t)b * bins.first[p.L];
    if (blockIdx.x == 0)  // the walk overwrites the counters with its results; it needs where regions start
        for (int r = tid; r <= p.L * p.G; r += blockDim.x)
            p.sort_regions[(size_t)b * (p.L * p.G + 1) + r] =
                starts[r < p.L * p.G ? bins.first[r / p.G] + (unsigned int)(r % p.G) * bins.cells[r / p.G] : bins.first[p.L]];
    if (row >= p.rows_per_b) return;
    const float *trow = wtile + (lane >> p.gs_log2) * p.row_stride;
    const unsigned int g = (unsigned int)(row % p.G);
    const size_t rowg = (size_t)b * p.rows_per_b + row;
    unsigned int *ranks = row_slots<PT>(p, rowg);
    const float2 stats = *reinterpret_cast<const float2 *>(ranks + LK);
    constexpr int kBatch = 4;  // the starts of four points are requested before the first is used
    for (int i0 = lane_c; i0 < LK; i0 += kBatch * gs) {
        unsigned int pos[kBatch], start[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            const int i = i0 + u * gs;
            pos[u] = i < LK ? ranks[i] : kNoPosition;
            start[u] = 0u;
            if (pos[u] < kNotFinite) {
                const int l = (i >> 2) >> p.k_shift;
                const LevelGeom lv = geom[l];
                start[u] = __ldg(starts + bins.first[l] + g * bins.cells[l] +
                                 bin_of(lv, base_cell(lv, trow[3 * i], trow[3 * i + 1], trow[3 * i + 2])) * bins.stride[l]);
            }
        }
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            const int i = i0 + u * gs;
            if (pos[u] >= kNotFinite) continue;
            const LevelGeom lv = geom[(i >> 2) >> p.k_shift];
            const BaseCell c = base_cell(lv, trow[3 * i], trow[3 * i + 1], trow[3 * i + 2]);
            const uint32_t sx = (uint32_t)p.GD, sy = (uint32_t)lv.W * sx, sz = (uint32_t)lv.H * sy;
            const unsigned int mx = (unsigned int)(c.x >= 0) | (unsigned int)(c.x + 1 < lv.W) << 1;    // corners dx = 0, 1
            const unsigned int mxy = (c.y >= 0 ? mx : 0u) | (c.y + 1 < lv.H ? mx << 2 : 0u);          // dy*2 + dx
            const unsigned int in8 = (c.z >= 0 ? mxy : 0u) | (c.z + 1 < lv.D ? mxy << 4 : 0u);        // dz*4 + dy*2 + dx
            const uint32_t off0 = (uint32_t)c.z * sz + (uint32_t)c.y * sy + (uint32_t)c.x * sx;      // wraps for index -1; + stride wraps back
            const unsigned int at = start[u] + pos[u];
            // one 32-byte record = one whole sector (no read-modify-write behind the store)
            store_record(p.sort_entries + 2 * (size_t)at, make_float4(c.fx, c.fy, c.fz, __expf(trow[3 * LK + i] - stats.x) * stats.y),
                         make_float4(__uint_as_float((unsigned int)rowg), 0.f, __uint_as_float(off0), __uint_as_float(in8)));
            ranks[i] = at;
        }
    }
}

// ---- exclusive scan of n counters, in place: tile sums -> scan of the sums (one block) -> scan of every tile ----
__device__ __forceinline__ unsigned int block_exclusive_scan(unsigned int v, unsigned int *warp_sums, unsigned int &total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned int inc = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const unsigned int t = __shfl_up_sync(0xffffffffu, inc, d);
        if (lane >= d) inc += t;
    }
    if (lane == 31) warp_sums[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        unsigned int w = lane < (int)(blockDim.x >> 5) ? warp_sums[lane] : 0u;
        unsigned int winc = w;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const unsigned int t = __shfl_up_sync(0xffffffffu, winc, d);
            if (lane >= d) winc += t;
        }
        warp_sums[lane] = winc - w;                 // exclusive offset of each warp
        if (lane == 31) warp_sums[32] = winc;       // block total
    }
    __syncthreads();
    total = warp_sums[32];
    const unsigned int r = warp_sums[warp] + inc - v;
    __syncthreads();  // warp_sums may be re-used by the caller's next round
    return r;
}

// The host sizes the counters for the most bins a volume of N cells can have; the kernels find the real number.
__device__ __forceinline__ size_t counters_of(const Problem &p) {
    SortBins bins;
    build_sort_bins(bins, p.shapes, p.L, p.G, p.sort_spread);
    return (size_t)bins.first[p.L] * p.B + 1;
}

__global__ void __launch_bounds__(kScanThreads) fda_scan_tile_sums_kernel(const Problem p) {
    const unsigned int *__restrict__ data = p.sort_counters;
    unsigned int *__restrict__ tile_sums = p.sort_tile_sums;
    const size_t n = counters_of(p);
    if ((size_t)blockIdx.x * kScanTile >= n) return;
    __shared__ unsigned int warp_sums[33];
    const size_t base = (size_t)blockIdx.x * kScanTile + (size_t)threadIdx.x * kScanItems;
    unsigned int s = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) s += base + k < n ? data[base + k] : 0u;
    unsigned int total;
    (void)block_exclusive_scan(s, warp_sums, total);
    if (threadIdx.x == 0) tile_sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(kScanThreads) fda_scan_spine_kernel(const Problem p) {
    unsigned int *tile_sums = p.sort_tile_sums;
    const unsigned int tiles = (unsigned int)((counters_of(p) + kScanTile - 1) / kScanTile);
    __shared__ unsigned int warp_sums[33];
    unsigned int carry = 0;
    for (unsigned int base = 0; base < tiles; base += kScanThreads) {  // uniform trip count
        const unsigned int i = base + threadIdx.x;
        const unsigned int v = i < tiles ? tile_sums[i] : 0u;
        unsigned int total;
        const unsigned int ex = block_exclusive_scan(v, warp_sums, total);
        if (i < tiles) tile_sums[i] = carry + ex;
        carry += total;
    }
}

__global__ void __launch_bounds__(kScanThreads) fda_scan_apply_kernel(const Problem p) {
    unsigned int *__restrict__ data = p.sort_counters;
    const unsigned int *__restrict__ tile_offsets = p.sort_tile_sums;
    const size_t n = counters_of(p);
    if ((size_t)blockIdx.x * kScanTile >= n) return;
    __shared__ unsigned int warp_sums[33];
    const size_t base = (size_t)blockIdx.x * kScanTile + (size_t)threadIdx.x * kScanItems;
    unsigned int v[kScanItems];
    unsigned int s = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        v[k] = base + k < n ? data[base + k] : 0u;
        s += v[k];
    }
    unsigned int total;
    unsigned int run = tile_offsets[blockIdx.x] + block_exclusive_scan(s, warp_sums, total);
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        if (base + k < n) data[base + k] = run;
        run += v[k];
    }
}

// ---- the walk over the sorted list ---------------------------------------------------------------------------
__device__ __forceinline__ void cp_async16_once(void *smem, const void *gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned int)__cvta_generic_to_shared(smem)), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int kPending> __device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(kPending) : "memory");
}

// Warp-level matrix products in the value dtype with fp32 accumulators, and the split of two fp32 weights into three
// 16-bit terms hi + mid + lo.  Three bf16 terms hold all 24 bits of a weight whatever its size; three fp16 terms those above
// fp16's smallest step, 2^-24, so fp16 weights are scaled first and what is left is split again (see `scatter` below).
template <typename VT> struct WarpMma;
#define FDA_WARP_MMA(TYPE)                                                                                                          \
    static __device__ __forceinline__ void k16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,       \
                                               uint32_t b1) {                                                                        \
        asm("mma.sync.aligned.m16n8k16.row.col.f32." TYPE "." TYPE ".f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};" \
            : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));               \
    }                                                                                                                                \
    static __device__ __forceinline__ void k8(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {                               \
        asm("mma.sync.aligned.m16n8k8.row.col.f32." TYPE "." TYPE ".f32 {%0, %1, %2, %3}, {%4, %5}, {%6}, {%0, %1, %2, %3};"         \
            : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(b0));                                          \
    }
template <> struct WarpMma<__nv_bfloat16> {
    FDA_WARP_MMA("bf16")
    static constexpr bool kNarrowExponent = false;
    static __device__ __forceinline__ uint32_t take(float &w0, float &w1) {  // rounds the pair to 16 bits, leaves the remainders
        const __nv_bfloat162 h = __floats2bfloat162_rn(w0, w1);
        const uint32_t r = *reinterpret_cast<const uint32_t *>(&h);
        w0 -= __uint_as_float(r << 16);
        w1 -= __uint_as_float(r & 0xffff0000u);
        return r;
    }
};
template <> struct WarpMma<__half> {
    FDA_WARP_MMA("f16")
    static constexpr bool kNarrowExponent = true;
    static __device__ __forceinline__ uint32_t take(float &w0, float &w1) {
        const __half2 h = __floats2half2_rn(w0, w1);
        const float2 f = __half22float2(h);
        w0 -= f.x;
        w1 -= f.y;
        return *reinterpret_cast<const uint32_t *>(&h);
    }
};
#undef FDA_WARP_MMA
__device__ __forceinline__ uint32_t transpose8x8(uint32_t v) {
    uint32_t r;
    asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
    return r;
}

// A lane's quarter of a head row of D = 16 * KS channels: channels tig * D/4 ... as 2 * KS words.
template <int KS> struct RowWords {
    uint32_t w[2 * KS];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int i = 0; i < 2 * KS; ++i) w[i] = 0u;
    }
    __device__ __forceinline__ void load(const void *p) {
        if constexpr (KS % 2 == 0) {
#pragma unroll
            for (int i = 0; i < KS / 2; ++i) {
                const uint4 r = __ldg(static_cast<const uint4 *>(p) + i);
                w[4 * i] = r.x; w[4 * i + 1] = r.y; w[4 * i + 2] = r.z; w[4 * i + 3] = r.w;
            }
        } else {
#pragma unroll
            for (int i = 0; i < KS; ++i) {
                const uint2 r = __ldg(static_cast<const uint2 *>(p) + i);
                w[2 * i] = r.x; w[2 * i + 1] = r.y;
            }
        }
    }
};

constexpr int kWalkSpan = 128;     // list entries a warp takes at a time
constexpr int kWalkWarps = 4;
constexpr int kWalkRegions = 16384;  // most (level, head) regions of one launch: their tables lie in shared memory
struct WalkBuffer {                // per warp, double-buffered; padded so that a unit may be read past its end
    float4 geo[kWalkSpan + 8];     // fractions along x, y, z, probability
    uint4 tag[kWalkSpan + 8];      // row, (in a unit's first entry) end of the unit, base offset, corner mask
};
struct WalkShared {
    WalkBuffer buf[kWalkWarps][2];
    float4 dots[kWalkWarps][2][kWalkSpan];  // dot products of a point with corners 0-3 / 4-7
};
// followed by the first entry and span of every region, and the end
inline size_t walk_smem_bytes(int regions) { return sizeof(WalkShared) + ((size_t)regions + 1) * sizeof(uint2); }

// The list of a (level, head) region is cut into spans, one warp each; a span into runs of points with the same cell, runs
// into units of at most eight points; a warp takes two units at a time (halves A and B, one cell each).  With the eight
// value rows V of the cell (one per corner), the grad_output rows GO of the unit's points and the points' corner weights
// W, everything is small matrix products:
//
//   dot[point][corner]    = GO  V^T       m16n8k16: rows 0-7 the points of A, 8-15 of B; columns = corners of A's (B's) cell
//   image[channel][corner] += GO^T W      m16n8k8 per half; W in three 16-bit terms (fp16: and more where
//                                         needed), GO^T by 8x8 transpositions
//
// Fragments come straight from 16-byte loads: lane (grp, tig) of a row-major fragment holds row grp's channels
// tig*D/4 ..., for GO and V alike, so the order of the channels inside the product does not matter.  Rows of the next pair
// of units travel while one is computed.  The image accumulators of a run stay in registers from unit to unit (4 * KS per
// lane) and leave with full-line reductions when the run ends.  The dot products go to shared memory; after the span's
// last unit a lane takes a point and turns its eight into the point's gradients.  All branches are uniform over the warp.
//
// 21 instructions per point on the largest pyramid (59 before, one lane group per point with 64 accumulators of its own and
// the groups of a warp changing runs at different times), 33 at 4.5 points per run.  Bound by the L1 request pipe where the
// volume fits L2 (76 % of its wavefronts: one per 64-byte row, two per reduction), by random 64-byte reads of grad_output
// from DRAM on the largest: 4.7 M points 490 -> 263 us, 229.6 M points 19.3 -> 9.7 ms.
//
// A unit of fewer than eight points repeats its last point with weight zero.  An infinite grad_output row gives NaN where a
// scalar sum may give infinity (a weight's terms may be zero or of either sign); both mark the same elements.
template <typename VT, int KS>
__global__ void __launch_bounds__(kWalkWarps * 32, KS <= 2 ? 4 : (KS == 3 ? 3 : 2)) fda_sorted_walk_kernel(const Problem p) {
    static_assert(Vec16<VT>::kCPL == 8, "16-bit value dtypes only");
    using Mma = WarpMma<VT>;
    constexpr int kQuarter = 4 * KS;     // channels of a lane's part of a row
    __shared__ LevelGeom geom[kMaxLevels];
    extern __shared__ __align__(16) unsigned char walk_smem[];
    WalkShared &sm = *reinterpret_cast<WalkShared *>(walk_smem);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int b = blockIdx.y;
    const int level_begin = __ffs(p.level_mask) - 1, level_end = 32 - __clz(p.level_mask);  // a contiguous range
    const int regions = (level_end - level_begin) * p.G;
    uint2 *region_table = reinterpret_cast<uint2 *>(walk_smem + sizeof(WalkShared));  // {first entry, first span}
    if (tid == 0) build_level_table(geom, p.shapes, p.lsi, p.L, p.GD, p.value_elem_bytes, true, p.l2_keep_bytes);
    for (int r = tid; r <= regions; r += blockDim.x) region_table[r].x = p.sort_regions[(size_t)b * (p.L * p.G + 1) + level_begin * p.G + r];
    __syncthreads();
    if (warp == 0) {
        unsigned int carry = 0;
        for (int r0 = 0; r0 <= regions; r0 += 32) {  // uniform trip count
            const int r = r0 + lane;
            const unsigned int n = r < regions ? (region_table[r + 1].x - region_table[r].x + kWalkSpan - 1) / kWalkSpan : 0u;
            unsigned int inc = n;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const unsigned int t = __shfl_up_sync(0xffffffffu, inc, d);
                if (lane >= d) inc += t;
            }
            if (r <= regions) region_table[r].y = carry + inc - n;
            carry += __shfl_sync(0xffffffffu, inc, 31);
        }
    }
    __syncthreads();
    const unsigned int spans = region_table[regions].y;
    const int tig = lane & 3, grp = lane >> 2;
    const uint64_t pol_keep = l2_policy_evict_last(), pol_stream = l2_policy_evict_first();
    const VT *go_base = static_cast<const VT *>(p.grad_out) + tig * kQuarter;
    const bool odd = grp & 1;
    // weight of corner grp along an axis = base + step * fraction
    const float bx = (grp & 1) ? 0.f : 1.f, sx = (grp & 1) ? 1.f : -1.f;
    const float by = (grp & 2) ? 0.f : 1.f, sy = (grp & 2) ? 1.f : -1.f;
    const float bz = (grp & 4) ? 0.f : 1.f, sz = (grp & 4) ? 1.f : -1.f;
    float4 (*dots)[kWalkSpan] = sm.dots[warp];

    float carry[KS][4];  // image of the run that may go on
    auto clear = [&]() {
#pragma unroll
        for (int k = 0; k < KS; ++k) { carry[k][0] = carry[k][1] = carry[k][2] = carry[k][3] = 0.f; }
    };

    auto request_span = [&](unsigned int sp, int r, int which) {  // copies a span's records; commits one (possibly empty) group
        if (sp < spans) {
            const unsigned int w0 = region_table[r].x + (sp - region_table[r].y) * kWalkSpan;
            const unsigned int left = region_table[r + 1].x - w0, wn = left < (unsigned int)kWalkSpan ? left : (unsigned int)kWalkSpan;
            WalkBuffer &bf = sm.buf[warp][which];
            const float4 *src = p.sort_entries + 2 * (size_t)w0;
            void *dst = (lane & 1) ? static_cast<void *>(bf.tag) : static_cast<void *>(bf.geo);
            for (unsigned int v = lane; v < 2 * wn; v += 32) cp_async16_once(static_cast<char *>(dst) + 16 * (v >> 1), src + v);
        }
        cp_async_commit();
    };

    const unsigned int stride = gridDim.x * kWalkWarps;
    unsigned int sp = blockIdx.x * kWalkWarps + warp;
    int region = 0, which = 0;
    while (region < regions && sp >= region_table[region + 1].y) ++region;
    request_span(sp, region, 0);
    for (; sp < spans; sp += stride, which ^= 1) {
        int next_region = region;
        while (next_region < regions && sp + stride >= region_table[next_region + 1].y) ++next_region;
        request_span(sp + stride, next_region, which ^ 1);
        cp_async_wait<1>();
        __syncwarp();
        const unsigned int w0 = region_table[region].x + (sp - region_table[region].y) * kWalkSpan;
        const unsigned int left = region_table[region + 1].x - w0;
        const int wn = (int)(left < (unsigned int)kWalkSpan ? left : (unsigned int)kWalkSpan);
        const float4 *geo = sm.buf[warp][which].geo;
        uint4 *tag = sm.buf[warp][which].tag;

        // the region's level and head: uniform over the span
        const int level = level_begin + region / p.G, head = region % p.G;
        const LevelGeom lv = geom[level];
        const uint32_t ox = (uint32_t)p.GD, oy = (uint32_t)lv.W * ox, oz = (uint32_t)lv.H * oy;
        const size_t slice = (size_t)b * p.N * p.GD + (size_t)lv.start * p.GD + (size_t)head * p.D;
        // value rows: corner grp, this lane's quarter of the channels
        const VT *value_l = static_cast<const VT *>(p.value) + slice + tig * kQuarter;
        const uint32_t corner = ((grp & 4) ? oz : 0u) + ((grp & 2) ? oy : 0u) + ((grp & 1) ? ox : 0u);
        // image rows: corners 2 * tig and 2 * tig + 1, one half of quarter grp / 2
        float *image_l = p.accum + slice + (grp >> 1) * kQuarter + (grp & 1) * (2 * KS);
        const uint32_t corner0 = ((tig & 2) ? oz : 0u) + ((tig & 1) ? oy : 0u);
        const uint64_t pol_image = (lv.keep & 2) ? pol_keep : pol_stream;

        // Sends a run's image.  carry[k][e]: word 2k + e/2 of quarter grp/2, i.e. channels 2 * word + odd, at corner
        // 2 * tig + e%2.  Neighbouring lane groups hold the even and the odd channels; they swap so that each has a
        // contiguous half.
        auto flush = [&](uint32_t off0, unsigned int in8) {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                float out[2 * KS];
#pragma unroll
                for (int j = 0; j < KS; ++j) {   // words j (first half) and KS + j (second half) of the quarter
                    const float first = carry[j >> 1][2 * (j & 1) + e], second = carry[(KS + j) >> 1][2 * ((KS + j) & 1) + e];
                    const float mine = odd ? second : first;
                    const float other = __shfl_xor_sync(0xffffffffu, odd ? first : second, 4);
                    out[2 * j] = odd ? other : mine;
                    out[2 * j + 1] = odd ? mine : other;
                }
                if (in8 >> (2 * tig + e) & 1u) {
                    float *dst = image_l + (uint32_t)(off0 + corner0 + (e ? ox : 0u));
                    if constexpr (KS % 2 == 0) {
#pragma unroll
                        for (int i = 0; i < KS / 2; ++i) red_add_f32x4_hint(dst + 4 * i, out[4 * i], out[4 * i + 1], out[4 * i + 2], out[4 * i + 3], pol_image);
                    } else {
#pragma unroll
                        for (int i = 0; i < KS; ++i) red_add_f32x2_hint(dst + 2 * i, out[2 * i], out[2 * i + 1], pol_image);
                    }
                }
            }
            clear();
        };

        // units: an entry starts one when it is the 1st, 9th, 17th ... of its run; it is told where its unit ends
        unsigned int unit_mask[kWalkSpan / 32];
        int run_start = 0;
#pragma unroll
        for (int g = 0; g < kWalkSpan / 32; ++g) {
            const int e = g * 32 + lane;
            const bool ok = e < wn;
            bool starts = e == 0;
            if (ok && !starts) {
                const uint2 t = *reinterpret_cast<const uint2 *>(&tag[e].z), q = *reinterpret_cast<const uint2 *>(&tag[e - 1].z);
                starts = q.x != t.x || q.y != t.y;
            }
            const unsigned int run_mask = __ballot_sync(0xffffffffu, starts);
            const unsigned int upto = run_mask & (0xffffffffu >> (31 - lane));
            const int mine = upto ? g * 32 + 31 - __clz(upto) : run_start;
            if (run_mask) run_start = g * 32 + 31 - __clz(run_mask);
            unit_mask[g] = __ballot_sync(0xffffffffu, ok && ((e - mine) & 7) == 0);
        }
        int next_first = wn;
#pragma unroll
        for (int g = kWalkSpan / 32 - 1; g >= 0; --g) {
            const unsigned int later = unit_mask[g] & ~(0xffffffffu >> (31 - lane));
            if (unit_mask[g] >> lane & 1u) tag[g * 32 + lane].y = (unsigned int)(later ? g * 32 + __ffs(later) - 1 : next_first);
            if (unit_mask[g]) next_first = g * 32 + __ffs(unit_mask[g]) - 1;
        }
        if (lane == 0) {  // an empty unit behind the last one goes on with its run: half B of an odd last pair
            const uint4 t = tag[wn - 1];
            tag[wn] = make_uint4(t.x, (unsigned int)wn, t.z, t.w);
        }
        __syncwarp();

        struct Half {
            RowWords<KS> go, v;
            int first, last;
            uint2 run;  // base offset, corner mask
            __device__ __forceinline__ bool same(const uint2 &o) const { return run.x == o.x && run.y == o.y; }
        };
        auto request = [&](Half &h, int first) {  // asks for the rows of the unit that starts at entry `first`
            const uint4 t = tag[first];
            h.first = first;
            h.last = (int)t.y;
            h.run = make_uint2(t.z, t.w);
            const int at = min(first + grp, max(h.last - 1, 0));
            h.go.load(go_base + (size_t)tag[at].x * (size_t)p.D);
            h.v.zero();
            if (t.w >> grp & 1u) h.v.load(value_l + (uint32_t)(t.z + corner));
        };
        // image += GO^T W of a unit, into fresh accumulators (no product waits for another unit's), in units of `unit`.
        //
        // fp16: the unit's weights are scaled by the power of two that brings the largest to [2^14, 2^15).  A weight of 2^-15 of
        // that and more lies in its three terms with all its bits.  What is left of smaller ones is scaled again and takes more
        // terms until nothing is left, so that every weight keeps the bits that it has as an fp32 factor (`rest`; one pair of
        // units in seven when points are spread evenly).  Weights scaled by a constant 2^15 alone were off by 9e-7 of themselves at
        // 1e-6 and 9e-3 at 1e-10.  Cost, whole calls:
        // DCNv4, 56.6 M points, 7.63 -> 7.93 ms; 48-channel encoder over 294912 queries 5.45 -> 5.49.
        auto weights = [&](const Half &h, float (&w)[2], float &unit) {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int i = h.first + 2 * tig + e;
                const float4 g = geo[i];
                const float wp = g.w * ((fmaf(sx, g.x, bx) * fmaf(sy, g.y, by)) * fmaf(sz, g.z, bz));
                w[e] = i < h.last ? wp : 0.f;
            }
            if constexpr (Mma::kNarrowExponent) {
                const unsigned int exponent = __reduce_max_sync(0xffffffffu, __float_as_uint(fmaxf(fabsf(w[0]), fabsf(w[1])))) >> 23;
                const unsigned int up = min(268u - exponent, 253u);  // exponent of 2^14 / 2^floor(log2(largest))
                unit = __uint_as_float((254u - up) << 23);
                w[0] *= __uint_as_float(up << 23);
                w[1] *= __uint_as_float(up << 23);
            }
        };
        auto scatter = [&](const Half &h, float (&w)[2], float (&acc)[KS][4]) {
            uint32_t got[2 * KS];
#pragma unroll
            for (int i = 0; i < 2 * KS; ++i) got[i] = transpose8x8(h.go.w[i]);
#pragma unroll
            for (int k = 0; k < KS; ++k) { acc[k][0] = acc[k][1] = acc[k][2] = acc[k][3] = 0.f; }
#pragma unroll
            for (int term = 0; term < 3; ++term) {
                const uint32_t wt = Mma::take(w[0], w[1]);
#pragma unroll
                for (int k = 0; k < KS; ++k) Mma::k8(acc[k], got[2 * k], got[2 * k + 1], wt);
            }
        };
        auto rest = [&](const Half &h, float (&w)[2], float (&acc)[KS][4]) {
            float up = 0x1p39f, down = 0x1p-39f;    // at most half of 2^-24 is left; in later turns half of 2^3
            for (int turn = 0; turn < 16; ++turn) {  // fp32's bits end before; NaN counts as nothing left
                if (!__any_sync(0xffffffffu, fabsf(w[0]) > 0.f || fabsf(w[1]) > 0.f)) break;
                w[0] *= up;
                w[1] *= up;
                const uint32_t wt = Mma::take(w[0], w[1]);
#pragma unroll
                for (int k = 0; k < KS; ++k) {
                    float low[4] = {0.f, 0.f, 0.f, 0.f};
                    Mma::k8(low, transpose8x8(h.go.w[2 * k]), transpose8x8(h.go.w[2 * k + 1]), wt);
#pragma unroll
                    for (int e = 0; e < 4; ++e) acc[k][e] = fmaf(low[e], down, acc[k][e]);
                }
                up = 0x1p11f;
                down *= 0x1p-11f;
            }
        };
        auto add = [&](const float (&acc)[KS][4], float unit) {
#pragma unroll
            for (int k = 0; k < KS; ++k)
#pragma unroll
                for (int e = 0; e < 4; ++e) carry[k][e] = Mma::kNarrowExponent ? fmaf(acc[k][e], unit, carry[k][e]) : carry[k][e] + acc[k][e];
        };
        uint2 run = make_uint2(0u, 0u);  // no run yet: no corner, nothing is sent
        auto pair = [&](const Half &ha, const Half &hb) {
            // Every k-step into fresh accumulators, added as fp32 numbers: the instruction rounds what it adds to its accumulator
            // more coarsely.  Coordinate gradients of 64 channels against 64 bits, relative: fp16 1.35e-7 in one accumulator,
            // 1.04e-7 so, 1.08e-7 the plain kernel (image 1.4e-7, plain 2.9e-7).  Cost: under 1 % of a call.
            float ca[2] = {0.f, 0.f}, cb[2] = {0.f, 0.f};
#pragma unroll
            for (int k = 0; k < KS; ++k) {
                float sa[4] = {0.f, 0.f, 0.f, 0.f}, sb[4] = {0.f, 0.f, 0.f, 0.f};
                Mma::k16(sa, ha.go.w[2 * k], hb.go.w[2 * k], ha.go.w[2 * k + 1], hb.go.w[2 * k + 1], ha.v.w[2 * k], ha.v.w[2 * k + 1]);
                Mma::k16(sb, ha.go.w[2 * k], hb.go.w[2 * k], ha.go.w[2 * k + 1], hb.go.w[2 * k + 1], hb.v.w[2 * k], hb.v.w[2 * k + 1]);
                ca[0] += sa[0]; ca[1] += sa[1];
                cb[0] += sb[2]; cb[1] += sb[3];
            }
            float ia[KS][4], ib[KS][4];
            float wa[2], wb[2], ua = 1.0f, ub = 1.0f;
            weights(ha, wa, ua);
            weights(hb, wb, ub);
            scatter(ha, wa, ia);
            scatter(hb, wb, ib);
            if constexpr (Mma::kNarrowExponent) {
                const unsigned int left = __float_as_uint(wa[0]) | __float_as_uint(wa[1]) | __float_as_uint(wb[0]) | __float_as_uint(wb[1]);
                if (__any_sync(0xffffffffu, (left << 1) != 0u)) {
                    rest(ha, wa, ia);
                    rest(hb, wb, ib);
                }
            }
            // corners 2 * tig and 2 * tig + 1 of point grp
            const int pa = ha.first + grp, pb = hb.first + grp;
            if (pa < ha.last) *(reinterpret_cast<float2 *>(&dots[tig >> 1][pa]) + (tig & 1)) = make_float2(ca[0], ca[1]);
            if (pb < hb.last) *(reinterpret_cast<float2 *>(&dots[tig >> 1][pb]) + (tig & 1)) = make_float2(cb[0], cb[1]);
            if (!ha.same(run)) flush(run.x, run.y);
            add(ia, ua);
            if (!hb.same(ha.run)) flush(ha.run.x, ha.run.y);
            add(ib, ub);
            run = hb.run;
        };
        clear();
        Half h0, h1, h2, h3;
        request(h0, 0);
        request(h1, h0.last);
        for (;;) {  // two pairs per turn: the register sets alternate without copies
            bool more = h1.last < wn;
            if (more) {
                request(h2, h1.last);
                request(h3, h2.last);
            }
            pair(h0, h1);
            if (!more) break;
            more = h3.last < wn;
            if (more) {
                request(h0, h3.last);
                request(h1, h0.last);
            }
            pair(h2, h3);
            if (!more) break;
        }
        flush(run.x, run.y);
        __syncwarp();

        // the points' own gradients, one point per lane
        const float scale_x = p.sort_voxel ? p.sort_scale : lv.fW, scale_y = p.sort_voxel ? p.sort_scale : lv.fH;
        const float scale_z = p.sort_voxel ? p.sort_scale : lv.fD;
        for (int e = lane; e < wn; e += 32) {
            const float4 lo = dots[0][e], hi = dots[1][e], g = geo[e];
            const float x0 = 1.0f - g.x, y0 = 1.0f - g.y, z0 = 1.0f - g.z;
            // along x: interpolated value s and difference d for (z, y) = 00, 01, 10, 11
            const float s00 = fmaf(g.x, lo.y, x0 * lo.x), s01 = fmaf(g.x, lo.w, x0 * lo.z), d00 = lo.y - lo.x, d01 = lo.w - lo.z;
            const float s10 = fmaf(g.x, hi.y, x0 * hi.x), s11 = fmaf(g.x, hi.w, x0 * hi.z), d10 = hi.y - hi.x, d11 = hi.w - hi.z;
            // along y
            const float s0 = fmaf(g.y, s01, y0 * s00), s1 = fmaf(g.y, s11, y0 * s10);
            const float dx0 = fmaf(g.y, d01, y0 * d00), dx1 = fmaf(g.y, d11, y0 * d10);
            const float gx = fmaf(g.z, dx1, z0 * dx0), gy = fmaf(g.z, s11 - s10, z0 * (s01 - s00)), gz = s1 - s0, da = fmaf(g.z, s1, z0 * s0);
            __stcs(p.sort_results + w0 + e, make_float4(g.w * scale_x * gx, g.w * scale_y * gy, g.w * scale_z * gz, da));
        }
        __syncwarp();  // records, units and dot products have been read
        region = next_region;
    }
    cp_async_wait<0>();
}

// Per row: the results of its points from the list, soft-max backward grad_logit_i = p_i * (dalpha_i - sum_j p_j dalpha_j),
// finished row of grad_sampling_loc_attn.  A point that is not filed has no result: its gradients are zero
// (NaN across the axes of an infinite position).  One random
// 16-byte read per point; scattered 16-byte writes in the walk instead cost as much when the results fit L2 and three times
// the DRAM traffic when they do not.
template <typename PT>
__global__ void __launch_bounds__(kThreads) fda_sort_finalize_kernel(const Problem p) {
    extern __shared__ __align__(16) float smem_tile[];
    const int tid = threadIdx.x, b = blockIdx.y;
    const int gs = 1 << p.gs_log2;
    const int lane = tid & 31, warp = tid >> 5;
    const int lane_c = tid & (gs - 1);
    const int rows_per_block = (int)blockDim.x >> p.gs_log2;
    const int rows_per_warp = 32 >> p.gs_log2;
    const int row = blockIdx.x * rows_per_block + (tid >> p.gs_log2);
    const bool row_ok = row < p.rows_per_b;
    const int LK = p.LK;
    const int first = blockIdx.x * rows_per_block + warp * rows_per_warp;
    float *wtile = smem_tile + warp * rows_per_warp * p.row_stride;
    int nrows = p.rows_per_b - first;
    nrows = nrows < 0 ? 0 : (nrows > rows_per_warp ? rows_per_warp : nrows);
    float *trow = wtile + (lane >> p.gs_log2) * p.row_stride;
    const size_t rowg = (size_t)b * p.rows_per_b + (row_ok ? row : 0);
    const unsigned int *positions = row_slots<PT>(p, rowg);  // all read before the first gradient of the row is written
    const PT *logits = static_cast<const PT *>(p.packed) + rowg * (size_t)(4 * LK) + 3 * LK;
    const float2 stats = *reinterpret_cast<const float2 *>(positions + LK);

    // Tile row: [0,3LK) coordinate gradients, [3LK,4LK) dalpha -> logit gradients, [4LK,5LK) probabilities.
    float S = 0.f;
    constexpr int kBatch = 8;  // the results of eight points are requested before the first one is used
    for (int i0 = lane_c; row_ok && i0 < LK; i0 += kBatch * gs) {
        unsigned int at[kBatch];
        float lg[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            const int i = i0 + u * gs;
            at[u] = i < LK ? __ldcs(positions + i) : kNoPosition;
            lg[u] = i < LK ? load1<PT>(logits + i) : 0.f;
        }
        float4 r[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            r[u] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (at[u] < kNotFinite) {
                r[u] = __ldcs(p.sort_results + at[u]);
            } else if (at[u] != kNoPosition) {  // zero times the NaN weights of the other axes
                const unsigned int bad = at[u] - kNotFinite;
                const float nan = __int_as_float(0x7fffffff);
                r[u] = make_float4(bad & 6u ? nan : 0.f, bad & 5u ? nan : 0.f, bad & 3u ? nan : 0.f, nan);
            }
        }
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            const int i = i0 + u * gs;
            if (i < LK) {
                const float a = __expf(lg[u] - stats.x) * stats.y;
                trow[3 * i] = r[u].x; trow[3 * i + 1] = r[u].y; trow[3 * i + 2] = r[u].z;
                trow[3 * LK + i] = r[u].w;
                trow[4 * LK + i] = a;
                S = fmaf(a, r[u].w, S);
            }
        }
    }
    for (int mask = gs >> 1; mask > 0; mask >>= 1) S += __shfl_xor_sync(0xffffffffu, S, mask);
    for (int i = lane_c; row_ok && i < LK; i += gs) trow[3 * LK + i] = trow[4 * LK + i] * (trow[3 * LK + i] - S);
    __syncwarp();
    PT *dst = static_cast<PT *>(p.grad_packed) + ((size_t)b * p.rows_per_b + first) * (size_t)(4 * LK);
    const int nvec = nrows * LK;
    const float inv_lk = 1.0f / (float)LK;
    for (int v = lane; v < nvec; v += 32) {
        const int r = row_of_vector(v, inv_lk);
        const int c = (v - r * LK) * 4;
        store4_stream<PT>(dst + (size_t)v * 4, *reinterpret_cast<const float4 *>(wtile + r * p.row_stride + c));
    }
}

}  // namespace fda
