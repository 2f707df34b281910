// DCNv4-3D (deformable convolution v4, volumetric) for sm_100a: forward and backward.
//
// Replaces forward_kernel_dcn / forward_kernel_dcn_reg (csrc/cuda/dcnv4_im2col_cuda.cuh:49,259),
// backward_kernel_dcn / backward_kernel_dcn_warp_primitive (csrc/cuda/dcnv4_col2im_cuda.cuh:48,319) and
// their host launchers (csrc/cuda/dcnv4_cuda.cu:19-189) of the reference.  Same gather / scatter skeleton
// as Flash Deformable Attention with one level and a fixed stencil:
//
//   out[b, q, g, :] = sum_k m_k * trilinear(value[b], p_k)[g, :]
//   p_k = p0(q) + (stencil_k * dilation + offset_k) * offset_scale          (voxel coordinates)
//
// q = (z, y, x) runs over the output volume, stencil_k over the kernel_w x kernel_h x kernel_d points
// (w outermost, d innermost; the centre point skipped when remove_center), m = mask (soft-maxed over
// the K points when `softmax`).  offset row of (b, q): `padded` elements, per group g a block of
// K*3 offsets (x, y, z per point) followed by K mask values at g*K*4 (csrc/cuda/dcnv4_im2col_cuda.cuh:118).
//
// Thread mapping as in fda_device.cuh: one row = (q, g), its channels over lanes that own one 16-byte
// vector each; the row's 4*K offset/mask values are staged in a warp-private shared-memory tile.
#include "../../include/fda_b200.h"

#include <cstring>

#include "fda_backward.cuh"
#include "fda_config.h"
#include "fda_sort_record.cuh"

namespace {

struct DcnProblem {
    const void *value;       // [B][Din*Hin*Win][G][D]
    const void *offset;      // [B][Q][padded]
    void *out;               // [B][Q][G*D]                      (forward)
    const void *grad_out;    // [B][Q][G*D]                      (backward)
    float *accum;            // fp32 image of grad_value         (backward)
    void *grad_offset;       // [B][Q][padded]                   (backward)
    int B, G, D, Q, K, padded;
    int Din, Hin, Win, Dout, Hout, Wout;
    int kd, kh, kw, sd, sh, sw, pd, ph, pw, dd, dh, dw;
    float offset_scale;
    int remove_center, softmax;
    int gs_log2, lpg, rows_per_b, GD, row_stride;
    int vector_rows;         // offset rows (and their gradients) start on a boundary of four values
    unsigned long long l2_keep_bytes;
};

// Voxel position of stencil point (i, j, k) = (w, h, d index) for output cell (x, y, z), offsets (ox, oy, oz):
// the arithmetic of the reference (dcnv4_im2col_cuda.cuh:178-216), every step in fp32.
struct StencilBase {
    float w, h, d;
};
__device__ __forceinline__ StencilBase stencil_base(const DcnProblem &p, int q) {
    const int x = q % p.Wout, yz = q / p.Wout, y = yz % p.Hout, z = yz / p.Hout;
    const int p0w = ((p.dw * (p.kw - 1)) >> 1) - p.pw + x * p.sw;
    const int p0h = ((p.dh * (p.kh - 1)) >> 1) - p.ph + y * p.sh;
    const int p0d = ((p.dd * (p.kd - 1)) >> 1) - p.pd + z * p.sd;
    StencilBase s;
    s.w = (float)p0w - (float)((p.dw * (p.kw - 1)) >> 1) * p.offset_scale;
    s.h = (float)p0h - (float)((p.dh * (p.kh - 1)) >> 1) * p.offset_scale;
    s.d = (float)p0d - (float)((p.dd * (p.kd - 1)) >> 1) * p.offset_scale;
    return s;
}

// Walks the stencil in the reference's order (w outermost, d innermost), skipping the centre if asked.
struct StencilWalk {
    int i, j, k;
    __device__ __forceinline__ void start(const DcnProblem &p) { i = j = k = 0; skip_centre(p); }
    __device__ __forceinline__ void skip_centre(const DcnProblem &p) {
        if (p.remove_center && i == p.kw / 2 && j == p.kh / 2 && k == p.kd / 2) advance_raw(p);
    }
    __device__ __forceinline__ void advance_raw(const DcnProblem &p) {
        if (++k == p.kd) { k = 0; if (++j == p.kh) { j = 0; ++i; } }
    }
    __device__ __forceinline__ void next(const DcnProblem &p) { advance_raw(p); skip_centre(p); }
};

// Stage the 4*K values of every row of this warp (row = q*G + g -> offset + (b*Q + q)*padded + g*K*4) as fp32.
template <typename T>
__device__ __forceinline__ void stage_dcn_rows(const DcnProblem &p, int b, int first_row, int nrows, float *wtile, int lane) {
    const int per_row = 4 * p.K;
    const T *base = static_cast<const T *>(p.offset) + (size_t)b * p.Q * (size_t)p.padded;
    for (int r = 0; r < nrows; ++r) {
        const int row = first_row + r, q = row / p.G, g = row - q * p.G;
        const T *src = base + (size_t)q * p.padded + (size_t)g * per_row;
        float *dst = wtile + r * p.row_stride;
        if (p.vector_rows) {  // four values per load, one load per lane for 27 points: forward of 56.6 M points 2.85 -> 2.62 ms
            for (int e = 4 * lane; e < per_row; e += 128) {
                const float4 v = fda::load4<T>(src + e);
                dst[e] = v.x; dst[e + 1] = v.y; dst[e + 2] = v.z; dst[e + 3] = v.w;
            }
        } else {
            for (int e = lane; e < per_row; e += 32) dst[e] = fda::load1<T>(src + e);
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(fda::kThreads, 3) dcnv4_forward_kernel(const DcnProblem p) {
    using namespace fda;
    constexpr int CPL = Vec16<T>::kCPL;
    extern __shared__ __align__(16) float smem_tile[];
    const int tid = threadIdx.x, b = blockIdx.y;
    const int gs = 1 << p.gs_log2, lane = tid & 31, warp = tid >> 5;
    const int lane_c = tid & (gs - 1);
    const int rows_per_block = (int)blockDim.x >> p.gs_log2, rows_per_warp = 32 >> p.gs_log2;
    const int row = blockIdx.x * rows_per_block + (tid >> p.gs_log2);
    const bool row_ok = row < p.rows_per_b, active = row_ok && lane_c < p.lpg;
    const int first = blockIdx.x * rows_per_block + warp * rows_per_warp;
    float *wtile = smem_tile + warp * rows_per_warp * p.row_stride;
    int nrows = p.rows_per_b - first;
    nrows = nrows < 0 ? 0 : (nrows > rows_per_warp ? rows_per_warp : nrows);
    stage_dcn_rows<T>(p, b, first, nrows, wtile, lane);
    __syncwarp();
    const float *trow = wtile + (lane >> p.gs_log2) * p.row_stride;
    const int K = p.K;

    float m = 0.f, inv = 1.f;
    if (p.softmax && row_ok) {
        m = -INFINITY;
        for (int k = 0; k < K; ++k) m = fmaxf(m, trow[3 * K + k]);
        float s = 0.f;
        for (int k = 0; k < K; ++k) s += __expf(trow[3 * K + k] - m);
        inv = 1.0f / s;
    }
    LevelGeom lv;
    lv.D = p.Din; lv.H = p.Hin; lv.W = p.Win; lv.start = 0; lv.keep = 0;
    lv.fD = (float)p.Din; lv.fH = (float)p.Hin; lv.fW = (float)p.Win;
    const bool keep = (unsigned long long)p.Din * p.Hin * p.Win * p.GD * sizeof(T) <= p.l2_keep_bytes;
    const uint64_t pol = keep ? l2_policy_evict_last() : l2_policy_evict_normal();
    const int q = row_ok ? row / p.G : 0, g = row_ok ? row - q * p.G : 0;
    const StencilBase sb = stencil_base(p, q);
    const T *value_b = static_cast<const T *>(p.value) + (size_t)b * p.Din * p.Hin * p.Win * (size_t)p.GD + (size_t)g * p.D +
                       (size_t)lane_c * CPL;
    float acc[CPL];
#pragma unroll
    for (int c = 0; c < CPL; ++c) acc[c] = 0.f;
    StencilWalk sw;
    sw.start(p);
    for (int k = 0; k < K; ++k, sw.next(p)) {
        const float ox = row_ok ? trow[3 * k] : 0.f, oy = row_ok ? trow[3 * k + 1] : 0.f, oz = row_ok ? trow[3 * k + 2] : 0.f;
        const float a = row_ok ? (p.softmax ? __expf(trow[3 * K + k] - m) * inv : trow[3 * K + k]) : 0.f;
        const float w_im = sb.w + ((float)(sw.i * p.dw) + ox) * p.offset_scale;
        const float h_im = sb.h + ((float)(sw.j * p.dh) + oy) * p.offset_scale;
        const float d_im = sb.d + ((float)(sw.k * p.dd) + oz) * p.offset_scale;
        PointGeom pg;
        point_geometry_voxel(lv, p.GD, w_im, h_im, d_im, pg);
        uint4 raw[8];
#pragma unroll
        for (int n = 0; n < 8; ++n) {
            const bool in = active && pg.zin[n >> 2] && pg.yin[(n >> 1) & 1] && pg.xin[n & 1];
            raw[n] = in ? ldg16_hint(value_b + pg.off[n], pol) : make_uint4(0u, 0u, 0u, 0u);
        }
#pragma unroll
        for (int n = 0; n < 8; ++n) axpy16<T>(raw[n], a * ((pg.wx[n & 1] * pg.wy[(n >> 1) & 1]) * pg.wz[n >> 2]), acc);
    }
    if (active) {
        T *dst = static_cast<T *>(p.out) + ((size_t)b * p.rows_per_b + row) * (size_t)p.D + (size_t)lane_c * CPL;
        stg16_hint(dst, Vec16<T>::pack(acc), l2_policy_evict_first());
    }
}

// Tile row (fp32): [0,3K) offsets -> offset gradients, [3K,4K) masks -> raw dmask -> mask gradients, [4K,5K) soft-max probabilities.
template <typename T>
__global__ void __launch_bounds__(fda::kThreads, 2) dcnv4_backward_kernel(const DcnProblem p) {
    using namespace fda;
    constexpr int CPL = Vec16<T>::kCPL;
    extern __shared__ __align__(16) float smem_tile[];
    const int tid = threadIdx.x, b = blockIdx.y;
    const int gs = 1 << p.gs_log2, lane = tid & 31, warp = tid >> 5;
    const int lane_c = tid & (gs - 1);
    const int rows_per_block = (int)blockDim.x >> p.gs_log2, rows_per_warp = 32 >> p.gs_log2;
    const int row = blockIdx.x * rows_per_block + (tid >> p.gs_log2);
    const bool row_ok = row < p.rows_per_b, active = row_ok && lane_c < p.lpg;
    const int first = blockIdx.x * rows_per_block + warp * rows_per_warp;
    float *wtile = smem_tile + warp * rows_per_warp * p.row_stride;
    int nrows = p.rows_per_b - first;
    nrows = nrows < 0 ? 0 : (nrows > rows_per_warp ? rows_per_warp : nrows);
    stage_dcn_rows<T>(p, b, first, nrows, wtile, lane);
    __syncwarp();
    float *trow = wtile + (lane >> p.gs_log2) * p.row_stride;
    const int K = p.K;

    if (row_ok) {  // probabilities (or the masks themselves) into [4K, 5K): written by the row's first lane
        float m = -INFINITY, s = 0.f;
        if (p.softmax) {
            for (int k = 0; k < K; ++k) m = fmaxf(m, trow[3 * K + k]);
            for (int k = 0; k < K; ++k) s += __expf(trow[3 * K + k] - m);
        }
        const float inv = p.softmax ? 1.0f / s : 1.f;
        for (int k = lane_c; k < K; k += gs)
            trow[4 * K + k] = p.softmax ? __expf(trow[3 * K + k] - m) * inv : trow[3 * K + k];
    }
    __syncwarp();

    LevelGeom lv;
    lv.D = p.Din; lv.H = p.Hin; lv.W = p.Win; lv.start = 0; lv.keep = 0;
    lv.fD = (float)p.Din; lv.fH = (float)p.Hin; lv.fW = (float)p.Win;
    const size_t cells = (size_t)p.Din * p.Hin * p.Win;
    unsigned long long budget = p.l2_keep_bytes;
    const bool keep_image = cells * p.GD * 4ull <= budget;
    if (keep_image) budget -= cells * p.GD * 4ull;
    const bool keep_value = cells * p.GD * sizeof(T) <= budget;
    const uint64_t pol_keep = l2_policy_evict_last(), pol_stream = l2_policy_evict_first(), pol_norm = l2_policy_evict_normal();
    const uint64_t pol_v = keep_value ? pol_keep : pol_norm, pol_g = keep_image ? pol_keep : pol_norm;
    const int q = row_ok ? row / p.G : 0, g = row_ok ? row - q * p.G : 0;
    const StencilBase sb = stencil_base(p, q);
    const size_t head_elem = (size_t)b * cells * p.GD + (size_t)g * p.D;
    const T *value_b = static_cast<const T *>(p.value) + head_elem + (size_t)lane_c * CPL;
    float *accum_b = p.accum + head_elem + (size_t)lane_c * 4;
    RowGrad<T> go;
    go.load(static_cast<const T *>(p.grad_out) + ((size_t)b * p.rows_per_b + (row_ok ? row : 0)) * (size_t)p.D, lane_c, p.lpg,
            active, pol_stream);
    const int red_stride = 4 * p.lpg;

    StencilWalk sw;
    sw.start(p);
    for (int k = 0; k < K; ++k, sw.next(p)) {
        const float ox = row_ok ? trow[3 * k] : 0.f, oy = row_ok ? trow[3 * k + 1] : 0.f, oz = row_ok ? trow[3 * k + 2] : 0.f;
        const float a = row_ok ? trow[4 * K + k] : 0.f;
        const float w_im = sb.w + ((float)(sw.i * p.dw) + ox) * p.offset_scale;
        const float h_im = sb.h + ((float)(sw.j * p.dh) + oy) * p.offset_scale;
        const float d_im = sb.d + ((float)(sw.k * p.dd) + oz) * p.offset_scale;
        PointGeom pg;
        point_geometry_voxel(lv, p.GD, w_im, h_im, d_im, pg);
        float gx, gy, gz, da;
        point_backward_geom<T, false>(pg, a, value_b, accum_b, go, red_stride, active, gs, pol_v, pol_g, gx, gy, gz, da);
        __syncwarp();  // every lane of the row has read this point's offsets
        if (row_ok && lane_c == 0) {
            // d p / d offset = offset_scale along each axis (csrc/cuda/dcnv4_col2im_cuda.cuh:205)
            trow[3 * k] = a * p.offset_scale * gx;
            trow[3 * k + 1] = a * p.offset_scale * gy;
            trow[3 * k + 2] = a * p.offset_scale * gz;
            trow[3 * K + k] = da;
        }
    }
    __syncwarp();
    if (p.softmax) {  // uniform branch: the warp barrier inside is reached by every lane
        float S = 0.f;  // sum_j m_j * dmask_j
        if (row_ok)
            for (int k = 0; k < K; ++k) S = fmaf(trow[4 * K + k], trow[3 * K + k], S);
        __syncwarp();
        if (row_ok)
            for (int k = lane_c; k < K; k += gs) trow[3 * K + k] = trow[4 * K + k] * (trow[3 * K + k] - S);
    }
    __syncwarp();
    // write the finished gradient rows (the padding of the offset rows is cleared by a memset)
    const int per_row = 4 * K;
    T *gbase = static_cast<T *>(p.grad_offset) + (size_t)b * p.Q * (size_t)p.padded;
    for (int r = 0; r < nrows; ++r) {
        const int rr = first + r, qq = rr / p.G, gg = rr - qq * p.G;
        T *dst = gbase + (size_t)qq * p.padded + (size_t)gg * per_row;
        for (int e = lane; e < per_row; e += 32) fda::store1<T>(dst + e, wtile[r * p.row_stride + e]);
    }
}

// ---- cell-sorted backward (16-bit values) ----------------------------------------------------------------------
// The points of a call are sorted by group and base cell and walked run by run (fda_backward_sorted.cuh): with one output
// cell per input cell and 27 points each, the eight value rows of a cell are read and its eight image rows added to once
// for up to 27 points instead of once per point.  One level; positions come from the stencil instead of normalised
// coordinates.  Rows are taken eight to a warp, their 4*K values staged as fp32; points are dealt to lanes over all the
// warp's rows, so that ranks and positions are read and written as one span.
constexpr int kSortRows = 8;
constexpr int kRowExtra = 6;                          // after a row's 4*K values: base x, y, z, soft-max maximum, 1 / sum, group
constexpr unsigned int kSortNone = 0xffffffffu;       // no corner inside the volume
constexpr unsigned int kSortNotFinite = 0xfffffff0u;  // the same, and axes (bits x, y, z) whose position is not finite

struct DcnSort {
    unsigned int *counters, *ranks, *regions;
    float2 *stats;
    float4 *entries, *results;
    int64_t *shape;  // d, h, w of the volume, 0 (the one level's extents and start)
};

__global__ void __launch_bounds__(256) dcnv4_sort_begin_kernel(const DcnProblem p, const DcnSort s, size_t n) {
    if (blockIdx.x == 0 && threadIdx.x == 0) { s.shape[0] = p.Din; s.shape[1] = p.Hin; s.shape[2] = p.Win; s.shape[3] = 0; }
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) s.counters[i] = 0u;
}

struct SortRows {
    int first, nrows;
    float *tile;
};
// Stencil positions times dilation, by point, in front of the tiles: two integer divisions per point otherwise.  Whole block.
__device__ __forceinline__ float *stencil_table(const DcnProblem &p, float *smem) {
    for (int k = threadIdx.x; k < p.K; k += blockDim.x) {
        const int kk = k + (p.remove_center && k >= ((p.kw / 2) * p.kh + p.kh / 2) * p.kd + p.kd / 2 ? 1 : 0);
        const int ij = kk / p.kd, i = ij / p.kh;
        smem[3 * k] = (float)(i * p.dw);
        smem[3 * k + 1] = (float)((ij - i * p.kh) * p.dh);
        smem[3 * k + 2] = (float)((kk - ij * p.kd) * p.dd);
    }
    return smem;
}
// Stages the warp's rows and each row's stencil base and group.
template <typename T>
__device__ __forceinline__ SortRows sort_rows(const DcnProblem &p, float *smem, int b) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    SortRows s;
    s.first = (blockIdx.x * (blockDim.x >> 5) + warp) * kSortRows;
    s.nrows = max(0, min(kSortRows, p.rows_per_b - s.first));
    s.tile = smem + warp * kSortRows * p.row_stride;
    stage_dcn_rows<T>(p, b, s.first, s.nrows, s.tile, lane);
    if (lane < s.nrows) {
        const int row = s.first + lane, q = row / p.G;
        const StencilBase sb = stencil_base(p, q);
        float *extra = s.tile + lane * p.row_stride + 4 * p.K;
        extra[0] = sb.w; extra[1] = sb.h; extra[2] = sb.d;
        extra[5] = __int_as_float(row - q * p.G);
    }
    return s;
}

// Base cell of stencil point k of a staged row.  Every rounding is spelled out: the count and the fill pass must agree.
struct DcnCell {
    int x, y, z;
    float fx, fy, fz;
    unsigned int code;  // 0: at least one corner inside
    unsigned int bin;   // inside the group
};
__device__ __forceinline__ DcnCell dcn_cell(const DcnProblem &p, const float *stencil, const float *trow, int k) {
    const float *extra = trow + 4 * p.K;
    const float x = __fmaf_rn(__fadd_rn(stencil[3 * k], trow[3 * k]), p.offset_scale, extra[0]);
    const float y = __fmaf_rn(__fadd_rn(stencil[3 * k + 1], trow[3 * k + 1]), p.offset_scale, extra[1]);
    const float z = __fmaf_rn(__fadd_rn(stencil[3 * k + 2], trow[3 * k + 2]), p.offset_scale, extra[2]);
    const float xf = floorf(x), yf = floorf(y), zf = floorf(z);
    DcnCell c;
    c.x = (int)xf; c.y = (int)yf; c.z = (int)zf;  // saturates; NaN is cell 0, its weights stay NaN
    c.fx = __fsub_rn(x, xf); c.fy = __fsub_rn(y, yf); c.fz = __fsub_rn(z, zf);
    const unsigned int ux = (unsigned int)c.x + 1u, uy = (unsigned int)c.y + 1u, uz = (unsigned int)c.z + 1u;
    c.code = 0u;
    c.bin = (uz * (unsigned int)(p.Hin + 1) + uy) * (unsigned int)(p.Win + 1) + ux;
    if (ux > (unsigned int)p.Win || uy > (unsigned int)p.Hin || uz > (unsigned int)p.Din) {
        const unsigned int bad = (isfinite(x) ? 0u : 1u) | (isfinite(y) ? 0u : 2u) | (isfinite(z) ? 0u : 4u);
        c.code = bad ? kSortNotFinite + bad : kSortNone;
    }
    return c;
}

template <typename T>
__global__ void __launch_bounds__(fda::kThreads) dcnv4_sort_count_kernel(const DcnProblem p, const DcnSort s) {
    extern __shared__ __align__(16) float smem_tile[];
    const int lane = threadIdx.x & 31, b = blockIdx.y, K = p.K;
    const float *stencil = stencil_table(p, smem_tile);
    const SortRows rows = sort_rows<T>(p, smem_tile + 3 * p.K, b);
    __syncthreads();
    {   // soft-max statistics, four lanes per row
        const int r = lane >> 2;
        const float *trow = rows.tile + r * p.row_stride + 3 * K;
        float m = 0.f, sum = 1.f;
        if (p.softmax) {
            m = -INFINITY;
            for (int k = lane & 3; r < rows.nrows && k < K; k += 4) m = fmaxf(m, trow[k]);
            m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
            m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
            sum = 0.f;
            for (int k = lane & 3; r < rows.nrows && k < K; k += 4) sum += __expf(trow[k] - m);
            sum += __shfl_xor_sync(0xffffffffu, sum, 1);
            sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        }
        if (r < rows.nrows && (lane & 3) == 0) s.stats[(size_t)b * p.rows_per_b + rows.first + r] = make_float2(m, 1.0f / sum);
    }
    const unsigned int cells = (unsigned int)(p.Din + 1) * (unsigned int)(p.Hin + 1) * (unsigned int)(p.Win + 1);
    unsigned int *counters = s.counters + (size_t)b * p.G * cells;
    unsigned int *ranks = s.ranks + ((size_t)b * p.rows_per_b + rows.first) * (size_t)K;
    const float inv_k = 1.0f / (float)K;
    const int n = rows.nrows * K;
    constexpr int kBatch = 4;  // all requests go out before the first answer is needed
    for (int e0 = lane; e0 < n; e0 += kBatch * 32) {
        unsigned int rank[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            const int e = e0 + 32 * u;
            if (e < n) {
                const int r = fda::row_of_vector(e, inv_k);
                const float *trow = rows.tile + r * p.row_stride;
                const DcnCell c = dcn_cell(p, stencil, trow, e - r * K);
                rank[u] = c.code;
                if (c.code == 0u) rank[u] = atomicAdd(counters + (size_t)__float_as_int(trow[4 * K + 5]) * cells + c.bin, 1u);
            }
        }
#pragma unroll
        for (int u = 0; u < kBatch; ++u)
            if (e0 + 32 * u < n) ranks[e0 + 32 * u] = rank[u];
    }
}

template <typename T>
__global__ void __launch_bounds__(fda::kThreads) dcnv4_sort_fill_kernel(const DcnProblem p, const DcnSort s) {
    extern __shared__ __align__(16) float smem_tile[];
    const int lane = threadIdx.x & 31, b = blockIdx.y, K = p.K;
    const float *stencil = stencil_table(p, smem_tile);
    const SortRows rows = sort_rows<T>(p, smem_tile + 3 * p.K, b);
    if (lane < rows.nrows) {
        const float2 st = s.stats[(size_t)b * p.rows_per_b + rows.first + lane];
        float *extra = rows.tile + lane * p.row_stride + 4 * K;
        extra[3] = st.x; extra[4] = st.y;
    }
    __syncthreads();
    const unsigned int cells = (unsigned int)(p.Din + 1) * (unsigned int)(p.Hin + 1) * (unsigned int)(p.Win + 1);
    const unsigned int *starts = s.counters + (size_t)b * p.G * cells;
    unsigned int *ranks = s.ranks + ((size_t)b * p.rows_per_b + rows.first) * (size_t)K;
    if (blockIdx.x == 0)
        for (int g = threadIdx.x; g <= p.G; g += blockDim.x) s.regions[(size_t)b * (p.G + 1) + g] = starts[(size_t)g * cells];
    const uint32_t sx = (uint32_t)p.GD, sy = (uint32_t)p.Win * sx, sz = (uint32_t)p.Hin * sy;
    const float inv_k = 1.0f / (float)K;
    const int n = rows.nrows * K;
    for (int e = lane; e < n; e += 32) {
        const unsigned int rank = ranks[e];
        if (rank >= kSortNotFinite) continue;
        const int r = fda::row_of_vector(e, inv_k), k = e - r * K;
        const float *trow = rows.tile + r * p.row_stride;
        const DcnCell c = dcn_cell(p, stencil, trow, k);
        const unsigned int at = starts[(size_t)__float_as_int(trow[4 * K + 5]) * cells + c.bin] + rank;
        const unsigned int mx = (unsigned int)(c.x >= 0) | (unsigned int)(c.x + 1 < p.Win) << 1;    // corners dx = 0, 1
        const unsigned int mxy = (c.y >= 0 ? mx : 0u) | (c.y + 1 < p.Hin ? mx << 2 : 0u);          // dy*2 + dx
        const unsigned int in8 = (c.z >= 0 ? mxy : 0u) | (c.z + 1 < p.Din ? mxy << 4 : 0u);        // dz*4 + dy*2 + dx
        const uint32_t off0 = (uint32_t)c.z * sz + (uint32_t)c.y * sy + (uint32_t)c.x * sx;        // wraps for index -1; + stride wraps back
        const float mask = trow[3 * K + k];
        const float a = p.softmax ? __expf(mask - trow[4 * K + 3]) * trow[4 * K + 4] : mask;
        const size_t row = (size_t)b * p.rows_per_b + rows.first + r;
        fda::store_record(s.entries + 2 * (size_t)at, make_float4(c.fx, c.fy, c.fz, a),
                          make_float4(__uint_as_float((unsigned int)row), 0.f, __uint_as_float(off0), __uint_as_float(in8)));
        ranks[e] = at;
    }
}

// Per row: its points' results from the list, soft-max backward, finished row of grad_offset.
template <typename T>
__global__ void __launch_bounds__(fda::kThreads) dcnv4_sort_finalize_kernel(const DcnProblem p, const DcnSort s) {
    extern __shared__ __align__(16) float smem_tile[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, b = blockIdx.y, K = p.K;
    const int first = (blockIdx.x * (blockDim.x >> 5) + warp) * kSortRows;
    const int nrows = max(0, min(kSortRows, p.rows_per_b - first));
    float *tile = smem_tile + warp * kSortRows * p.row_stride;
    const unsigned int *positions = s.ranks + ((size_t)b * p.rows_per_b + first) * (size_t)K;
    const float inv_k = 1.0f / (float)K;
    const int n = nrows * K;
    constexpr int kBatch = 8;  // the results of eight points are requested before the first one is used
    for (int e0 = lane; e0 < n; e0 += kBatch * 32) {
        unsigned int at[kBatch];
        float4 res[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) at[u] = e0 + 32 * u < n ? __ldcs(positions + e0 + 32 * u) : kSortNone;
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            res[u] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (at[u] < kSortNotFinite) {
                res[u] = __ldcs(s.results + at[u]);
            } else if (at[u] != kSortNone) {  // a weight along such an axis times zero
                const unsigned int bad = at[u] - kSortNotFinite;
                const float nan = __int_as_float(0x7fffffff);
                res[u] = make_float4(bad & 6u ? nan : 0.f, bad & 5u ? nan : 0.f, bad & 3u ? nan : 0.f, nan);
            }
        }
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            const int e = e0 + 32 * u;
            if (e < n) {
                const int r = fda::row_of_vector(e, inv_k), k = e - r * K;
                float *trow = tile + r * p.row_stride;
                trow[3 * k] = res[u].x; trow[3 * k + 1] = res[u].y; trow[3 * k + 2] = res[u].z;
                trow[3 * K + k] = res[u].w;
            }
        }
    }
    __syncwarp();
    const T *obase = static_cast<const T *>(p.offset) + (size_t)b * p.Q * (size_t)p.padded;
    T *gbase = static_cast<T *>(p.grad_offset) + (size_t)b * p.Q * (size_t)p.padded;
    if (p.softmax) {  // four lanes per row
        const int r = lane >> 2;
        const bool ok = r < nrows;
        const int row = ok ? first + r : 0, q = row / p.G, g = row - q * p.G;
        const T *masks = obase + (size_t)q * p.padded + (size_t)g * 4 * K + 3 * K;
        const float2 st = s.stats[(size_t)b * p.rows_per_b + row];
        float *trow = tile + r * p.row_stride + 3 * K;
        float S = 0.f;  // sum_j m_j * dmask_j
        for (int k = lane & 3; ok && k < K; k += 4) S = fmaf(__expf(fda::load1<T>(masks + k) - st.x) * st.y, trow[k], S);
        S += __shfl_xor_sync(0xffffffffu, S, 1);
        S += __shfl_xor_sync(0xffffffffu, S, 2);
        for (int k = lane & 3; ok && k < K; k += 4) trow[k] = (__expf(fda::load1<T>(masks + k) - st.x) * st.y) * (trow[k] - S);
    }
    __syncwarp();
    const int per_row = 4 * K;
    for (int r = 0; r < nrows; ++r) {
        const int row = first + r, q = row / p.G, g = row - q * p.G;
        T *dst = gbase + (size_t)q * p.padded + (size_t)g * per_row;
        const float *src = tile + r * p.row_stride;
        if (p.vector_rows)
            for (int e = 4 * lane; e < per_row; e += 128) fda::store4_stream<T>(dst + e, make_float4(src[e], src[e + 1], src[e + 2], src[e + 3]));
        else
            for (int e = lane; e < per_row; e += 32) fda::store1<T>(dst + e, src[e]);
    }
}

inline int dtype_size(int dt) { return dt == FDA_DTYPE_F32 ? 4 : 2; }

int fill_problem(DcnProblem &p, int batch, int depth_in, int height_in, int width_in, int group, int group_channels,
                 const int *kernel, const int *stride, const int *pad, const int *dilation, float offset_scale,
                 int remove_center, int softmax, int padded_offset_dim, int dtype, int im2col_step) {
    if (dtype < 0 || dtype > 2) return FDA_ERR_BAD_DTYPE;
    if (batch <= 0 || depth_in <= 0 || height_in <= 0 || width_in <= 0 || group <= 0 || group_channels <= 0) return FDA_ERR_BAD_SHAPE;
    for (int a = 0; a < 3; ++a)
        if (kernel[a] <= 0 || stride[a] <= 0 || pad[a] < 0 || dilation[a] <= 0) return FDA_ERR_BAD_SHAPE;
    const int cpl = 16 / dtype_size(dtype);
    if (group_channels % cpl != 0 || group_channels / cpl > 32) return FDA_ERR_BAD_HEAD_DIM;
    const int step = batch < im2col_step ? batch : im2col_step;
    if (step <= 0 || batch % step != 0) return FDA_ERR_IM2COL_STEP;
    p.B = batch; p.G = group; p.D = group_channels;
    p.Din = depth_in; p.Hin = height_in; p.Win = width_in;
    p.kd = kernel[0]; p.kh = kernel[1]; p.kw = kernel[2];
    p.sd = stride[0]; p.sh = stride[1]; p.sw = stride[2];
    p.pd = pad[0]; p.ph = pad[1]; p.pw = pad[2];
    p.dd = dilation[0]; p.dh = dilation[1]; p.dw = dilation[2];
    p.Dout = (depth_in + 2 * p.pd - (p.dd * (p.kd - 1) + 1)) / p.sd + 1;
    p.Hout = (height_in + 2 * p.ph - (p.dh * (p.kh - 1) + 1)) / p.sh + 1;
    p.Wout = (width_in + 2 * p.pw - (p.dw * (p.kw - 1) + 1)) / p.sw + 1;
    if (p.Dout <= 0 || p.Hout <= 0 || p.Wout <= 0) return FDA_ERR_BAD_SHAPE;
    p.K = p.kd * p.kh * p.kw - (remove_center ? 1 : 0);
    if (p.K <= 0 || p.K > 343) return FDA_ERR_BAD_POINTS;
    if (padded_offset_dim < group * p.K * 4) return FDA_ERR_BAD_SHAPE;
    const long long Q = (long long)p.Dout * p.Hout * p.Wout;
    if (Q * group >= (1ll << 31) || (long long)depth_in * height_in * width_in * group * group_channels >= (1ll << 31)) return FDA_ERR_BAD_SHAPE;
    if (batch > 65535) return FDA_ERR_BAD_SHAPE;
    p.Q = (int)Q; p.padded = padded_offset_dim;
    p.offset_scale = offset_scale; p.remove_center = remove_center ? 1 : 0; p.softmax = softmax ? 1 : 0;
    p.lpg = group_channels / cpl;
    int lg = 0;
    while ((1 << lg) < p.lpg) ++lg;
    p.gs_log2 = lg;
    p.rows_per_b = p.Q * group;
    p.GD = group * group_channels;
    p.l2_keep_bytes = (unsigned long long)(fda::config().l2_keep_fraction * 126.0 * 1024 * 1024);
    return FDA_OK;
}

template <typename T>
int launch_dcn(const DcnProblem &p0, bool backward, cudaStream_t st) {
    DcnProblem p = p0;
    p.row_stride = (backward ? 5 : 4) * p.K + 1;  // odd: the rows of a warp start in different banks
    int threads = fda::kThreads;
    while (threads > 32 && (size_t)(threads >> p.gs_log2) * p.row_stride * sizeof(float) > 96 * 1024) threads >>= 1;
    const size_t smem = (size_t)(threads >> p.gs_log2) * p.row_stride * sizeof(float);
    if (smem > 200 * 1024) return FDA_ERR_TOO_LARGE_STATIC;
    const int rows_per_block = threads >> p.gs_log2;
    const dim3 grid((unsigned)((p.rows_per_b + rows_per_block - 1) / rows_per_block), (unsigned)p.B, 1);
    auto kern = backward ? dcnv4_backward_kernel<T> : dcnv4_forward_kernel<T>;
    if (smem > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        if (e != cudaSuccess) { fda::record_cuda_error((int)e); return FDA_ERR_CUDA; }
    }
    kern<<<grid, threads, smem, st>>>(p);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) { fda::record_cuda_error((int)e); return FDA_ERR_CUDA; }
    return FDA_OK;
}

inline size_t round256(size_t n) { return (n + 255) & ~(size_t)255; }

// Whether sorting pays.  Measured per point: the plain scatter takes 0.16 / 0.20 / 0.33 ns at 16 / 32 / 48 and more channels,
// the sorted path 0.07 (0.09 above 32 channels) plus 0.19 / 0.27 / 0.55 over the points per cell and group; its launches
// cost 40 us more.  3x3x3, 32 channels: 0.22 M points 81 -> 85 us, 0.44 M 114 -> 97, 3.5 M 720 -> 347, 56.6 M 11.1 -> 4.8 ms;
// with stride 2 (3.4 points per cell) 0.44 M 132 -> 142, 2.7 M 669 -> 489; 64 channels 0.22 M 95 -> 93, 1.8 M 584 -> 257.
bool dcn_sorted_pays(int D, double points, double density) {
    const double plain = D <= 16 ? 0.16 : (D <= 32 ? 0.20 : 0.33);
    const double sorted = (D <= 32 ? 0.07 : 0.09) + (D <= 16 ? 0.19 : (D <= 32 ? 0.27 : 0.55)) / density;
    return points * (plain - sorted) > 40e3;
}

// Scratch of the cell-sorted backward, behind the fp32 image: [shape] [where groups start] [counters] [scan tile sums]
// [soft-max statistics] [ranks] [entries] [results], 52 bytes per point; total 0 when the path is not taken.  A call is sorted `elements` batch
// elements at a time, as many as keep the list at 32 M points, and at least one: the scratch does not grow with the batch, but
// follows an element that is larger than that.  Without memory for it a caller passes the image alone (plain path).
struct DcnSortLayout {
    size_t shape, regions, counters, tile_sums, stats, ranks, entries, results, total;
    int elements;
};
DcnSortLayout dcn_sort_layout(const DcnProblem &p, int dtype) {
    DcnSortLayout s{};
    const int mode = fda::config().sorted;
    if (mode <= 0 || dtype == FDA_DTYPE_F32 || p.D % 16 != 0 || p.D > 64 || p.G > 160 || p.K > 125) return s;
    // the walk splits fp16 weights relative to 1: soft-maxed masks only
    if (dtype == FDA_DTYPE_F16 && !p.softmax) return s;
    const unsigned long long points = (unsigned long long)p.rows_per_b * p.K;
    const unsigned long long bins = (unsigned long long)(p.Din + 1) * (p.Hin + 1) * (p.Win + 1) * p.G;
    if (points >= (1ull << 31) || bins >= (1ull << 30)) return s;
    const double cells = (double)p.Din * p.Hin * p.Win;
    if (mode == 1 && !dcn_sorted_pays(p.D, (double)points * p.B, (double)p.Q * p.K / cells)) return s;
    unsigned long long elements = (32ull << 20) / points;
    elements = elements < 1 ? 1 : (elements > (unsigned long long)p.B ? p.B : elements);
    while (elements > 1 && elements * bins >= (1ull << 30)) --elements;
    s.elements = (int)elements;
    const unsigned long long counters = elements * bins + 1;
    const size_t n = (size_t)(elements * points), rows = (size_t)elements * p.rows_per_b;
    s.shape = 0;
    s.regions = 256;
    s.counters = s.regions + round256((size_t)elements * (p.G + 1) * sizeof(unsigned int));
    s.tile_sums = s.counters + round256(counters * sizeof(unsigned int));
    s.stats = s.tile_sums + round256(fda::sort_scan_tiles(counters) * sizeof(unsigned int));
    s.ranks = s.stats + round256(rows * sizeof(float2));
    s.entries = s.ranks + round256(n * sizeof(unsigned int));
    s.results = s.entries + round256(n * 2 * sizeof(float4));
    s.total = s.results + round256(n * sizeof(float4));
    return s;
}

template <typename T>
int launch_dcn_sorted(const DcnProblem &p0, const DcnSortLayout &lay, char *scratch, int dtype, cudaStream_t st) {
    DcnSort s;
    s.shape = reinterpret_cast<int64_t *>(scratch + lay.shape);
    s.counters = reinterpret_cast<unsigned int *>(scratch + lay.counters);
    s.regions = reinterpret_cast<unsigned int *>(scratch + lay.regions);
    s.stats = reinterpret_cast<float2 *>(scratch + lay.stats);
    s.ranks = reinterpret_cast<unsigned int *>(scratch + lay.ranks);
    s.entries = reinterpret_cast<float4 *>(scratch + lay.entries);
    s.results = reinterpret_cast<float4 *>(scratch + lay.results);
    const size_t cells = (size_t)p0.Din * p0.Hin * p0.Win;
    for (int b0 = 0; b0 < p0.B; b0 += lay.elements) {
        DcnProblem p = p0;
        p.B = p0.B - b0 < lay.elements ? p0.B - b0 : lay.elements;
        p.value = static_cast<const T *>(p0.value) + (size_t)b0 * cells * p0.GD;
        p.offset = static_cast<const T *>(p0.offset) + (size_t)b0 * p0.Q * p0.padded;
        p.grad_out = static_cast<const T *>(p0.grad_out) + (size_t)b0 * p0.Q * p0.GD;
        p.accum = p0.accum + (size_t)b0 * cells * p0.GD;
        p.grad_offset = static_cast<T *>(p0.grad_offset) + (size_t)b0 * p0.Q * p0.padded;
        p.row_stride = (4 * p.K + kRowExtra) | 1;  // odd: the rows of a warp start in different banks
        int warps = fda::kThreads / 32;
        while (warps > 1 && ((size_t)warps * kSortRows * p.row_stride + 3 * p.K) * sizeof(float) > 48 * 1024) warps >>= 1;
        const size_t smem = ((size_t)warps * kSortRows * p.row_stride + 3 * p.K) * sizeof(float);  // K <= 125: at most 16.3 KB per warp
        const int rows_per_block = warps * kSortRows;
        const dim3 grid((unsigned)((p.rows_per_b + rows_per_block - 1) / rows_per_block), (unsigned)p.B, 1);
        const size_t bins = (size_t)(p.Din + 1) * (p.Hin + 1) * (p.Win + 1) * p.G * p.B + 1;
        const size_t blocks = (bins + 1023) / 1024;
        dcnv4_sort_begin_kernel<<<(unsigned)(blocks > 2368 ? 2368 : blocks), 256, 0, st>>>(p, s, bins);
        dcnv4_sort_count_kernel<T><<<grid, warps * 32, smem, st>>>(p, s);
        fda::Problem w;
        std::memset(&w, 0, sizeof(w));
        w.value = p.value; w.grad_out = p.grad_out; w.accum = p.accum;
        w.shapes = s.shape; w.lsi = s.shape + 3;
        w.B = p.B; w.N = (int)cells; w.G = p.G; w.D = p.D; w.L = 1; w.K = p.K; w.Q = p.Q; w.LK = p.K;
        w.rows_per_b = p.rows_per_b; w.GD = p.GD; w.gs_log2 = p.gs_log2; w.lpg = p.lpg; w.head_group = p.G;
        w.l2_keep_bytes = p.l2_keep_bytes; w.value_elem_bytes = sizeof(T); w.level_mask = 1;
        w.sort_counters = s.counters; w.sort_regions = s.regions; w.sort_entries = s.entries;
        w.sort_tile_sums = reinterpret_cast<unsigned int *>(scratch + lay.tile_sums);
        w.sort_results = s.results;
        w.sort_voxel = 1; w.sort_scale = p.offset_scale;
        if (int rc = fda::launch_sort_scan(w, bins, st)) return rc;
        dcnv4_sort_fill_kernel<T><<<grid, warps * 32, smem, st>>>(p, s);
        if (int rc = fda::launch_sort_walk(w, dtype, st)) return rc;
        dcnv4_sort_finalize_kernel<T><<<grid, warps * 32, smem, st>>>(p, s);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) { fda::record_cuda_error((int)e); return FDA_ERR_CUDA; }
    }
    return FDA_OK;
}

int dispatch_dcn(const DcnProblem &p, int dtype, bool backward, cudaStream_t st) {
    if (dtype == FDA_DTYPE_F32) return launch_dcn<float>(p, backward, st);
    if (dtype == FDA_DTYPE_F16) return launch_dcn<__half>(p, backward, st);
    return launch_dcn<__nv_bfloat16>(p, backward, st);
}

// A row's blocks of 4 * K values start at multiples of four values.
inline bool rows_aligned(const void *rows, int padded, int dtype) {
    return padded % 4 == 0 && (reinterpret_cast<uintptr_t>(rows) & (uintptr_t)(4 * dtype_size(dtype) - 1)) == 0;
}

inline bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

}  // namespace

extern "C" int fda_dcnv4_output_size(int depth_in, int height_in, int width_in, const int *kernel, const int *stride,
                                     const int *pad, const int *dilation, int *depth_out, int *height_out, int *width_out) {
    if (!kernel || !stride || !pad || !dilation || !depth_out || !height_out || !width_out) return FDA_ERR_NULL_POINTER;
    for (int a = 0; a < 3; ++a)
        if (kernel[a] <= 0 || stride[a] <= 0 || pad[a] < 0 || dilation[a] <= 0) return FDA_ERR_BAD_SHAPE;
    *depth_out = (depth_in + 2 * pad[0] - (dilation[0] * (kernel[0] - 1) + 1)) / stride[0] + 1;
    *height_out = (height_in + 2 * pad[1] - (dilation[1] * (kernel[1] - 1) + 1)) / stride[1] + 1;
    *width_out = (width_in + 2 * pad[2] - (dilation[2] * (kernel[2] - 1) + 1)) / stride[2] + 1;
    return (*depth_out > 0 && *height_out > 0 && *width_out > 0) ? FDA_OK : FDA_ERR_BAD_SHAPE;
}

extern "C" int fda_dcnv4_forward(const void *value, const void *p_offset, void *output, int batch, int depth_in, int height_in,
                                 int width_in, int group, int group_channels, const int *kernel, const int *stride,
                                 const int *pad, const int *dilation, float offset_scale, int remove_center, int softmax,
                                 int padded_offset_dim, int dtype, int im2col_step, void *stream) {
    if (!value || !p_offset || !output || !kernel || !stride || !pad || !dilation) return FDA_ERR_NULL_POINTER;
    DcnProblem p{};
    if (int rc = fill_problem(p, batch, depth_in, height_in, width_in, group, group_channels, kernel, stride, pad, dilation,
                              offset_scale, remove_center, softmax, padded_offset_dim, dtype, im2col_step))
        return rc;
    if (!aligned16(value) || !aligned16(output)) return FDA_ERR_MISALIGNED;
    p.value = value; p.offset = p_offset; p.out = output;
    p.vector_rows = rows_aligned(p_offset, padded_offset_dim, dtype);
    return dispatch_dcn(p, dtype, false, static_cast<cudaStream_t>(stream));
}

extern "C" size_t fda_dcnv4_backward_workspace_bytes(int batch, int depth_in, int height_in, int width_in, int group,
                                                     int group_channels, int dtype) {
    if (dtype == FDA_DTYPE_F32 || batch <= 0 || depth_in <= 0 || height_in <= 0 || width_in <= 0 || group <= 0 || group_channels <= 0)
        return 0;
    return (size_t)batch * depth_in * height_in * width_in * group * group_channels * sizeof(float);
}

extern "C" size_t fda_dcnv4_backward_scratch_bytes(int batch, int depth_in, int height_in, int width_in, int group,
                                                   int group_channels, const int *kernel, const int *stride, const int *pad,
                                                   const int *dilation, int remove_center, int softmax, int dtype) {
    if (!kernel || !stride || !pad || !dilation) return 0;
    DcnProblem p{};
    if (fill_problem(p, batch, depth_in, height_in, width_in, group, group_channels, kernel, stride, pad, dilation, 1.0f,
                     remove_center, softmax, 0x7fffffff, dtype, 1))
        return 0;
    const size_t image = fda_dcnv4_backward_workspace_bytes(batch, depth_in, height_in, width_in, group, group_channels, dtype);
    const DcnSortLayout lay = dcn_sort_layout(p, dtype);
    return lay.total ? round256(image) + lay.total : image;
}

extern "C" int fda_dcnv4_backward(const void *value, const void *p_offset, const void *grad_output, void *grad_value,
                                  void *grad_offset, void *workspace, size_t workspace_bytes, int batch, int depth_in,
                                  int height_in, int width_in, int group, int group_channels, const int *kernel,
                                  const int *stride, const int *pad, const int *dilation, float offset_scale,
                                  int remove_center, int softmax, int padded_offset_dim, int dtype, int im2col_step,
                                  void *stream) {
    if (!value || !p_offset || !grad_output || !grad_value || !grad_offset || !kernel || !stride || !pad || !dilation)
        return FDA_ERR_NULL_POINTER;
    DcnProblem p{};
    if (int rc = fill_problem(p, batch, depth_in, height_in, width_in, group, group_channels, kernel, stride, pad, dilation,
                              offset_scale, remove_center, softmax, padded_offset_dim, dtype, im2col_step))
        return rc;
    const size_t need = fda_dcnv4_backward_workspace_bytes(batch, depth_in, height_in, width_in, group, group_channels, dtype);
    if (need > 0 && (!workspace || workspace_bytes < need)) return FDA_ERR_WORKSPACE;
    if (!aligned16(value) || !aligned16(grad_output) || !aligned16(grad_value) || (need > 0 && !aligned16(workspace)))
        return FDA_ERR_MISALIGNED;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const size_t n = (size_t)batch * depth_in * height_in * width_in * group * group_channels;
    float *accum = need > 0 ? static_cast<float *>(workspace) : static_cast<float *>(grad_value);
    cudaError_t e = cudaMemsetAsync(accum, 0, n * sizeof(float), st);
    const int used = group * p.K * 4;  // the kernels write these of every offset row; the padding is cleared here
    if (e == cudaSuccess && padded_offset_dim > used)
        e = cudaMemset2DAsync(static_cast<char *>(grad_offset) + (size_t)used * dtype_size(dtype), (size_t)padded_offset_dim * dtype_size(dtype),
                              0, (size_t)(padded_offset_dim - used) * dtype_size(dtype), (size_t)batch * p.Q, st);
    if (e != cudaSuccess) { fda::record_cuda_error((int)e); return FDA_ERR_CUDA; }
    p.value = value; p.offset = p_offset; p.grad_out = grad_output; p.accum = accum; p.grad_offset = grad_offset;
    p.vector_rows = rows_aligned(p_offset, padded_offset_dim, dtype) && rows_aligned(grad_offset, padded_offset_dim, dtype);
    const DcnSortLayout lay = dcn_sort_layout(p, dtype);
    if (lay.total && (reinterpret_cast<uintptr_t>(workspace) & 255u) == 0 && workspace_bytes >= round256(need) + lay.total) {
        char *scratch = static_cast<char *>(workspace) + round256(need);
        if (int rc = dtype == FDA_DTYPE_F16 ? launch_dcn_sorted<__half>(p, lay, scratch, dtype, st)
                                            : launch_dcn_sorted<__nv_bfloat16>(p, lay, scratch, dtype, st))
            return rc;
    } else if (int rc = dispatch_dcn(p, dtype, true, st)) {
        return rc;
    }
    if (need == 0) return FDA_OK;
    return fda_cast_grad_value(accum, grad_value, n, dtype, stream);
}
