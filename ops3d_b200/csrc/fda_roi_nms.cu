// ROI-Align 3D (forward, backward) and NMS 3D for sm_100a: the two small detection-head operators that sit
// beside deformable attention in the reference's extension.
//
// Replaces roi_align_3d_forward_cuda_kernel / roi_align_3d_backward_cuda_kernel
// (csrc/cuda/roi_align_3d_cuda_kernel.cuh:31,110) with their interpolation helpers
// (csrc/cuda/interpolation_helpers_3d.h), and nms_kernel_3d plus the host-side greedy sweep of nms_3d_cuda
// (csrc/cuda/nms_3d_cuda.cu:49-101,133-157).  Differences in structure, not in results:
//   * ROI-Align: a warp per ROI and pair of channels contracts the volume axis after axis with one weight table per axis and
//     ROI; one thread per output element as in the reference where the tables do not fit shared memory.  16-bit features are
//     read directly and accumulated in fp32;
//   * NMS: boxes are ranked by score, the pairwise-IoU bit matrix is built 64 x 64 boxes per block as in the reference,
//     and the greedy sweep runs on the DEVICE in one block, so the matrix never crosses PCIe and the host only reads
//     the number of kept boxes.
#include "../../include/fda_b200.h"

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "fda_config.h"

namespace {

template <typename T> __device__ __forceinline__ float ldf(const T *p);
template <> __device__ __forceinline__ float ldf<float>(const float *p) { return __ldg(p); }
template <> __device__ __forceinline__ float ldf<__half>(const __half *p) { return __half2float(__ldg(p)); }
template <> __device__ __forceinline__ float ldf<__nv_bfloat16>(const __nv_bfloat16 *p) { return __bfloat162float(__ldg(p)); }
template <typename T> __device__ __forceinline__ T cvt_out(float v);
template <> __device__ __forceinline__ float cvt_out<float>(float v) { return v; }
template <> __device__ __forceinline__ __half cvt_out<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 cvt_out<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

// Corner indices and weights of one sample, the reference's rules (interpolation_helpers_3d.h): samples more than
// one voxel outside contribute nothing; coordinates are clamped to [0, size-1]; order 0 picks the nearest corner.
struct Sample {
    int z0, z1, y0, y1, x0, x1;
    float w[8];  // (z0y0x0, z0y0x1, z0y1x0, z0y1x1, z1y0x0, z1y0x1, z1y1x0, z1y1x1)
    bool valid;
};

__device__ __forceinline__ void axis_setup(float v, int size, int &i0, int &i1, float &l, float &h) {
    if (v <= 0.f) v = 0.f;
    i0 = (int)v;
    if (i0 >= size - 1) {
        i1 = i0 = size - 1;
        v = (float)i0;
    } else {
        i1 = i0 + 1;
    }
    l = v - (float)i0;
    h = 1.f - l;
}

__device__ __forceinline__ Sample make_sample(int depth, int height, int width, float z, float y, float x, int order) {
    Sample s;
    s.valid = !(y < -1.0f || y > (float)height || x < -1.0f || x > (float)width || z < -1.0f || z > (float)depth);
    if (!s.valid) {
        s.z0 = s.z1 = s.y0 = s.y1 = s.x0 = s.x1 = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) s.w[i] = 0.f;
        return s;
    }
    float lz, hz, ly, hy, lx, hx;
    axis_setup(z, depth, s.z0, s.z1, lz, hz);
    axis_setup(y, height, s.y0, s.y1, ly, hy);
    axis_setup(x, width, s.x0, s.x1, lx, hx);
    if (order == 0) {  // nearest: all weight on the closer corner along each axis (ties go to the lower one)
        lz = lz > 0.5f ? 1.f : 0.f; hz = 1.f - lz;
        ly = ly > 0.5f ? 1.f : 0.f; hy = 1.f - ly;
        lx = lx > 0.5f ? 1.f : 0.f; hx = 1.f - lx;
    }
    s.w[0] = hz * hy * hx; s.w[1] = hz * hy * lx; s.w[2] = hz * ly * hx; s.w[3] = hz * ly * lx;
    s.w[4] = lz * hy * hx; s.w[5] = lz * hy * lx; s.w[6] = lz * ly * hx; s.w[7] = lz * ly * lx;
    return s;
}

struct RoiGeom {
    int batch;
    float start_w, start_h, start_d, bin_w, bin_h, bin_d;
    int grid_w, grid_h, grid_d;
    float count;
};

template <typename RT>
__device__ __forceinline__ RoiGeom roi_geometry(const RT *roi, float spatial_scale, int sampling_ratio, int pd, int ph, int pw) {
    RoiGeom g;
    g.batch = (int)ldf<RT>(roi);
    g.start_w = ldf<RT>(roi + 1) * spatial_scale;
    g.start_h = ldf<RT>(roi + 2) * spatial_scale;
    g.start_d = ldf<RT>(roi + 3) * spatial_scale;
    const float rw = fmaxf(ldf<RT>(roi + 4) * spatial_scale - g.start_w, 1.f);
    const float rh = fmaxf(ldf<RT>(roi + 5) * spatial_scale - g.start_h, 1.f);
    const float rd = fmaxf(ldf<RT>(roi + 6) * spatial_scale - g.start_d, 1.f);
    g.bin_d = rd / (float)pd; g.bin_h = rh / (float)ph; g.bin_w = rw / (float)pw;
    g.grid_d = sampling_ratio > 0 ? sampling_ratio : (int)ceilf(rd / (float)pd);
    g.grid_h = sampling_ratio > 0 ? sampling_ratio : (int)ceilf(rh / (float)ph);
    g.grid_w = sampling_ratio > 0 ? sampling_ratio : (int)ceilf(rw / (float)pw);
    const int c = g.grid_d * g.grid_h * g.grid_w;
    g.count = (float)(c > 1 ? c : 1);
    return g;
}

template <typename T>
__global__ void __launch_bounds__(256) roi_align3d_forward_kernel(size_t total, const T *__restrict__ features,
                                                                  const T *__restrict__ rois, float spatial_scale,
                                                                  int sampling_ratio, int order, int channels, int depth,
                                                                  int height, int width, int pd, int ph, int pw,
                                                                  T *__restrict__ out) {
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t index = (size_t)blockIdx.x * blockDim.x + threadIdx.x; index < total; index += stride) {
        const int iw = (int)(index % pw);
        const int ih = (int)((index / pw) % ph);
        const int id = (int)((index / pw / ph) % pd);
        const int c = (int)((index / pw / ph / pd) % channels);
        const size_t n = index / pw / ph / pd / channels;
        const RoiGeom g = roi_geometry<T>(rois + n * 7, spatial_scale, sampling_ratio, pd, ph, pw);
        const T *vol = features + ((size_t)g.batch * channels + c) * (size_t)depth * height * width;
        const size_t hw = (size_t)height * width;
        float acc = 0.f;
        for (int iz = 0; iz < g.grid_d; ++iz) {
            const float z = g.start_d + id * g.bin_d + ((float)iz + .5f) * g.bin_d / (float)g.grid_d;
            for (int iy = 0; iy < g.grid_h; ++iy) {
                const float y = g.start_h + ih * g.bin_h + ((float)iy + .5f) * g.bin_h / (float)g.grid_h;
                for (int ix = 0; ix < g.grid_w; ++ix) {
                    const float x = g.start_w + iw * g.bin_w + ((float)ix + .5f) * g.bin_w / (float)g.grid_w;
                    const Sample s = make_sample(depth, height, width, z, y, x, order);
                    if (!s.valid) continue;
                    const T *p0 = vol + s.z0 * hw, *p1 = vol + s.z1 * hw;
                    acc += s.w[0] * ldf<T>(p0 + (size_t)s.y0 * width + s.x0) + s.w[1] * ldf<T>(p0 + (size_t)s.y0 * width + s.x1) +
                           s.w[2] * ldf<T>(p0 + (size_t)s.y1 * width + s.x0) + s.w[3] * ldf<T>(p0 + (size_t)s.y1 * width + s.x1) +
                           s.w[4] * ldf<T>(p1 + (size_t)s.y0 * width + s.x0) + s.w[5] * ldf<T>(p1 + (size_t)s.y0 * width + s.x1) +
                           s.w[6] * ldf<T>(p1 + (size_t)s.y1 * width + s.x0) + s.w[7] * ldf<T>(p1 + (size_t)s.y1 * width + s.x1);
                }
            }
        }
        out[index] = cvt_out<T>(acc / g.count);
    }
}

// grad_features (fp32, pre-zeroed by the caller as in the reference) += scatter of grad_output through the same weights.
template <typename T>
__global__ void __launch_bounds__(256) roi_align3d_backward_kernel(size_t total, const T *__restrict__ grad_out,
                                                                   const float *__restrict__ rois, float spatial_scale,
                                                                   int sampling_ratio, int order, int channels, int depth,
                                                                   int height, int width, int pd, int ph, int pw,
                                                                   float *__restrict__ grad_features) {
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t index = (size_t)blockIdx.x * blockDim.x + threadIdx.x; index < total; index += stride) {
        const int iw = (int)(index % pw);
        const int ih = (int)((index / pw) % ph);
        const int id = (int)((index / pw / ph) % pd);
        const int c = (int)((index / pw / ph / pd) % channels);
        const size_t n = index / pw / ph / pd / channels;
        const RoiGeom g = roi_geometry<float>(rois + n * 7, spatial_scale, sampling_ratio, pd, ph, pw);
        float *vol = grad_features + ((size_t)g.batch * channels + c) * (size_t)depth * height * width;
        const size_t hw = (size_t)height * width;
        const float go = ldf<T>(grad_out + index) / g.count;
        for (int iz = 0; iz < g.grid_d; ++iz) {
            const float z = g.start_d + id * g.bin_d + ((float)iz + .5f) * g.bin_d / (float)g.grid_d;
            for (int iy = 0; iy < g.grid_h; ++iy) {
                const float y = g.start_h + ih * g.bin_h + ((float)iy + .5f) * g.bin_h / (float)g.grid_h;
                for (int ix = 0; ix < g.grid_w; ++ix) {
                    const float x = g.start_w + iw * g.bin_w + ((float)ix + .5f) * g.bin_w / (float)g.grid_w;
                    const Sample s = make_sample(depth, height, width, z, y, x, order);
                    if (!s.valid) continue;
                    float *p0 = vol + s.z0 * hw, *p1 = vol + s.z1 * hw;
                    atomicAdd(p0 + (size_t)s.y0 * width + s.x0, go * s.w[0]);
                    atomicAdd(p0 + (size_t)s.y0 * width + s.x1, go * s.w[1]);
                    atomicAdd(p0 + (size_t)s.y1 * width + s.x0, go * s.w[2]);
                    atomicAdd(p0 + (size_t)s.y1 * width + s.x1, go * s.w[3]);
                    atomicAdd(p1 + (size_t)s.y0 * width + s.x0, go * s.w[4]);
                    atomicAdd(p1 + (size_t)s.y0 * width + s.x1, go * s.w[5]);
                    atomicAdd(p1 + (size_t)s.y1 * width + s.x0, go * s.w[6]);
                    atomicAdd(p1 + (size_t)s.y1 * width + s.x1, go * s.w[7]);
                }
            }
        }
    }
}

// ---- separable form -------------------------------------------------------------------------------------
// A sample's weights are products of one factor per axis, and so is its validity: the samples of a bin average to
//   out[pd][ph][pw] = 1/count * sum_z Wz[pd][z] sum_y Wy[ph][y] sum_x Wx[pw][x] f[z][y][x]
// over the voxels that samples touch, with a small weight table per axis.  A block builds the tables of one ROI once for
// its channels; a warp takes one channel and contracts axis after axis, plane by plane: about 10 x fewer operations than
// eight corners per sample, and in the backward one reduction per touched voxel of the ROI and channel instead of eight per
// sample (7x7x7 bins of 2x2x2 samples on a 9x17x21 ROI: 3.2 k against 22 k).  256 ROIs x 128 channels of a 16x32x64 volume:
// forward 648 -> 143 us, backward 1689 -> 152 us.  What bounds it: shared-memory and L1 accesses of the short dot products.
//
// The tables list the touched voxels only, in order.  A ROI with fewer samples than voxels leaves gaps between them; a voxel
// in a gap is neither read nor added to, whatever it holds (its weight of zero would turn an infinity into NaN), and costs
// nothing (64 ROIs over all of a 32x64x256 volume, 3x3x3 bins of 2x2x2 samples, 128 channels: by ranges of voxels forward 5.8
// ms, backward 2.3; by lists 0.07 and 0.08).  A bin touches a contiguous part of an axis's list: bins and their samples lie in increasing order.
struct AxisTable {
    float *w;     // [bins][size] weight of the i-th touched voxel, zero outside the bin's part
    int *lo, *hi; // [bins] the bin's part of the list (hi < lo: no valid sample)
    int *range;   // [size] first | last << 16 bin that touches the i-th touched voxel
    int *vox;     // [size] the i-th touched voxel
    int bins, size, n;
    __device__ __forceinline__ int first_bin(int i) const { return range[i] & 0xffff; }
    __device__ __forceinline__ int last_bin(int i) const { return (int)((unsigned int)range[i] >> 16); }
};

constexpr int kRoiThreads = 256;
constexpr int kRoiChannels = 2;  // per warp at a time; 1 / 2 / 4: 484 / 317 / 399 us for the two passes below

__host__ __device__ inline int roi_table_words(int bins, int size) { return bins * size + 2 * bins + 2 * size; }
// All tables of a ROI: four words for the lengths of the lists, then x (its weights first, on a 16-byte boundary), y, z.
__host__ __device__ inline int roi_tables_words(int pd, int ph, int pw, int depth, int height, int width) {
    return 4 + roi_table_words(pd, depth) + roi_table_words(ph, height) + roi_table_words(pw, width);
}

__device__ __forceinline__ AxisTable axis_table(float *mem, int bins, int size) {
    AxisTable t;
    t.w = mem;
    t.lo = reinterpret_cast<int *>(mem + bins * size);
    t.hi = t.lo + bins;
    t.range = t.hi + bins;
    t.vox = t.range + size;
    t.bins = bins;
    t.size = size;
    return t;
}

// f(first voxel, second voxel, weight of the second, weight of the first) for the valid samples of bin p along an axis.
template <typename F>
__device__ __forceinline__ void for_axis_samples(int size, int p, float start, float bin, int grid, int order, F f) {
    for (int i = 0; i < grid; ++i) {
        const float v = start + p * bin + ((float)i + .5f) * bin / (float)grid;
        if (v < -1.0f || v > (float)size) continue;
        int i0, i1;
        float l, h;
        axis_setup(v, size, i0, i1, l, h);
        if (order == 0) {
            l = l > 0.5f ? 1.f : 0.f;
            h = 1.f - l;
        }
        f(i0, i1, l, h);
    }
}

// Writes the indices in [0, size) that satisfy `wanted`, in order; returns their number.  By a whole warp.  wanted(i) may
// read list[i]: that place is written only after it.
template <typename F>
__device__ __forceinline__ int list_indices(int size, int *list, F wanted) {
    const int lane = threadIdx.x & 31;
    int n = 0;
    for (int base = 0; base < size; base += 32) {
        const bool is = base + lane < size && wanted(base + lane);
        const unsigned int mask = __ballot_sync(0xffffffffu, is);
        if (is) list[n + __popc(mask & ((1u << lane) - 1u))] = base + lane;
        n += __popc(mask);
    }
    return n;
}

struct RoiTables {
    AxisTable z, y, x;
    float *end;
};

// Called by the whole block; ends with a barrier.  kVec = 0: the forward.  Otherwise the backward, which
// visits rows in vectors of kVec voxels: along x, w and range are by voxel (last < first: not touched), and vox and n list the
// vectors with a touched voxel.
template <typename RT, int kVec>
__device__ __forceinline__ RoiGeom build_roi_tables(RoiTables &t, float *mem, const RT *roi, float spatial_scale, int sampling_ratio,
                                                    int order, int depth, int height, int width, int pd, int ph, int pw) {
    constexpr bool kForward = kVec == 0;
    const RoiGeom g = roi_geometry<RT>(roi, spatial_scale, sampling_ratio, pd, ph, pw);
    int *counts = reinterpret_cast<int *>(mem);
    t.x = axis_table(mem + 4, pw, width);
    t.y = axis_table(reinterpret_cast<float *>(t.x.vox + width), ph, height);
    t.z = axis_table(reinterpret_cast<float *>(t.y.vox + height), pd, depth);
    t.end = reinterpret_cast<float *>(t.z.vox + depth);
    const int tid = threadIdx.x, warp = tid >> 5, warps = blockDim.x >> 5;
    for (int i = tid; mem + i < t.end; i += blockDim.x) mem[i] = 0.f;
    __syncthreads();
    auto axis = [&](int a) {  // a copy: a reference chosen at run time would put the tables into local memory
        AxisTable x = t.x;
        if (a == 1) x = t.y;
        if (a == 2) x = t.z;
        return x;
    };
    auto for_bin_samples = [&](int i, auto f) {  // bin i of all axes' bins: x, then y, then z
        if (i < pw) for_axis_samples(width, i, g.start_w, g.bin_w, g.grid_w, order, [&](int i0, int i1, float l, float h) { f(0, i, i0, i1, l, h); });
        else if (i < pw + ph) for_axis_samples(height, i - pw, g.start_h, g.bin_h, g.grid_h, order, [&](int i0, int i1, float l, float h) { f(1, i - pw, i0, i1, l, h); });
        else for_axis_samples(depth, i - pw - ph, g.start_d, g.bin_d, g.grid_d, order, [&](int i0, int i1, float l, float h) { f(2, i - pw - ph, i0, i1, l, h); });
    };
    // touched voxels, marked in vox
    for (int i = tid; i < pw + ph + pd; i += blockDim.x)
        for_bin_samples(i, [&](int a, int, int i0, int i1, float, float) {
            int *mark = axis(a).vox;
            mark[i0] = 1;
            mark[i1] = 1;
        });
    __syncthreads();
    // their lists, and in range every voxel's place in its list (-1: not touched)
    for (int a = warp; a < 3; a += warps) {
        const AxisTable x = axis(a);
        for (int v = tid & 31; v < x.size; v += 32) x.range[v] = -1;
        const int n = list_indices(x.size, x.vox, [&](int v) { return x.vox[v] != 0; });
        __syncwarp();
        for (int i = tid & 31; i < n; i += 32) x.range[x.vox[i]] = i;
        if ((tid & 31) == 0) counts[a] = n;
    }
    __syncthreads();
    t.x.n = counts[0]; t.y.n = counts[1]; t.z.n = counts[2];
    // weights and every bin's part of the list
    for (int i = tid; i < pw + ph + pd; i += blockDim.x) {
        const AxisTable x = axis(i < pw ? 0 : (i < pw + ph ? 1 : 2));
        const int p = i < pw ? i : (i < pw + ph ? i - pw : i - pw - ph);
        int lo = x.size, hi = -1;
        for_bin_samples(i, [&](int a, int, int i0, int i1, float l, float h) {
            const int j0 = x.range[i0], j1 = x.range[i1];
            lo = min(lo, j0);
            hi = max(hi, j1);
            float *w = x.w + p * x.size;
            w[!kForward && a == 0 ? i0 : j0] += h;
            w[!kForward && a == 0 ? i1 : j1] += l;
        });
        x.lo[p] = lo;
        x.hi[p] = hi;
    }
    __syncthreads();
    // bins by voxel
    auto set_bins = [](const AxisTable &x, int at, int i) {
        int first = 1, last = 0;
        for (int p = 0; p < x.bins; ++p)
            if (x.lo[p] <= i && i <= x.hi[p]) {
                if (last < first) first = p;
                last = p;
            }
        x.range[at] = first | last << 16;
    };
    for (int i = tid; i < t.y.n; i += blockDim.x) set_bins(t.y, i, i);
    for (int i = tid; i < t.z.n; i += blockDim.x) set_bins(t.z, i, i);
    if constexpr (!kForward) {
        for (int v = tid; v < width; v += blockDim.x) set_bins(t.x, v, t.x.range[v]);  // no bin has a place -1
        __syncthreads();
        if (warp == 0) {
            const int n = list_indices(width / kVec, t.x.vox, [&](int i) {
                bool any = false;
#pragma unroll
                for (int e = 0; e < kVec; ++e) any |= t.x.first_bin(i * kVec + e) <= t.x.last_bin(i * kVec + e);
                return any;
            });
            if (tid == 0) counts[3] = n;
        }
    }
    __syncthreads();
    if constexpr (!kForward) t.x.n = counts[3];
    return g;
}

// Grid: (ROI, group of channels_per_block channels).  A warp takes kRoiChannels channels at a time (one weight and one set
// of bin ranges then serve all of them, and their loads overlap).  Per warp and channel: [height][pw] rows contracted
// along x, then the output tile [pd][ph][pw].  Lanes of both contractions: rows_per_step rows x pw bins, so that a lane
// keeps its bin.
template <typename T>
__global__ void __launch_bounds__(kRoiThreads) roi_align3d_forward_separable_kernel(const T *__restrict__ features, const T *__restrict__ rois,
                                                                                   float spatial_scale, int sampling_ratio, int order,
                                                                                   int channels, int depth, int height, int width, int pd,
                                                                                   int ph, int pw, int channels_per_block, T *__restrict__ out) {
    constexpr int kC = kRoiChannels;
    extern __shared__ __align__(16) float roi_smem[];
    const int n = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    RoiTables t;
    const RoiGeom g = build_roi_tables<T, 0>(t, roi_smem, rois + (size_t)n * 7, spatial_scale, sampling_ratio, order, depth, height, width, pd, ph, pw);
    const int bins = pd * ph * pw, rows_size = height * pw;
    float *rows = t.end + warp * kC * (rows_size + bins), *tile = rows + kC * rows_size;
    const int rows_per_step = 32 / pw, lane_row = lane / pw, p = lane - lane_row * pw;
    const bool used = lane_row < rows_per_step;
    const int xlo = used ? t.x.lo[p] : 0, xhi = used ? t.x.hi[p] : -1;
    const float *wx = t.x.w + (used ? p : 0) * width;
    const bool gaps = t.x.n > 0 && t.x.vox[t.x.n - 1] - t.x.vox[0] != t.x.n - 1;
    const int c_end = min(channels, ((int)blockIdx.y + 1) * channels_per_block);
    const size_t volume = (size_t)depth * height * width;
    for (int c = blockIdx.y * channels_per_block + warp * kC; c < c_end; c += warps * kC) {
        const T *vol = features + ((size_t)g.batch * channels + c) * volume;
        size_t of[kC];  // a channel beyond the last one repeats the last one; its result is dropped
#pragma unroll
        for (int k = 0; k < kC; ++k) of[k] = (size_t)min(k, c_end - 1 - c) * volume;
        for (int i = lane; i < kC * bins; i += 32) tile[i] = 0.f;
        for (int z = 0; z < t.z.n; ++z) {
            const T *plane = vol + (size_t)t.z.vox[z] * height * width;
            if (used)
                for (int y = lane_row; y < t.y.n; y += rows_per_step) {
                    const T *src = plane + (size_t)t.y.vox[y] * width;
                    float acc[kC];
#pragma unroll
                    for (int k = 0; k < kC; ++k) acc[k] = 0.f;
                    if (gaps) {
#pragma unroll 2
                        for (int x = xlo; x <= xhi; ++x) {
                            const float w = wx[x];
                            const T *at = src + t.x.vox[x];
#pragma unroll
                            for (int k = 0; k < kC; ++k) acc[k] = fmaf(w, ldf<T>(at + of[k]), acc[k]);
                        }
                    } else {
                        const T *first = src + t.x.vox[0];
#pragma unroll 2
                        for (int x = xlo; x <= xhi; ++x) {
                            const float w = wx[x];
#pragma unroll
                            for (int k = 0; k < kC; ++k) acc[k] = fmaf(w, ldf<T>(first + of[k] + x), acc[k]);
                        }
                    }
#pragma unroll
                    for (int k = 0; k < kC; ++k) rows[k * rows_size + y * pw + p] = acc[k];
                }
            __syncwarp();
            if (used)
                for (int q = lane_row; q < ph; q += rows_per_step) {
                    const float *wy = t.y.w + q * height;
                    float acc[kC];
#pragma unroll
                    for (int k = 0; k < kC; ++k) acc[k] = 0.f;
#pragma unroll 2
                    for (int y = t.y.lo[q]; y <= t.y.hi[q]; ++y) {
                        const float w = wy[y];
#pragma unroll
                        for (int k = 0; k < kC; ++k) acc[k] = fmaf(w, rows[k * rows_size + y * pw + p], acc[k]);
                    }
                    for (int d = t.z.first_bin(z), last = t.z.last_bin(z); d <= last; ++d) {
                        const float w = t.z.w[d * depth + z];
                        float *o = tile + (d * ph + q) * pw + p;
#pragma unroll
                        for (int k = 0; k < kC; ++k) o[k * bins] = fmaf(w, acc[k], o[k * bins]);
                    }
                }
            __syncwarp();
        }
        T *dst = out + ((size_t)n * channels + c) * (size_t)bins;
        const int valid = min(kC, c_end - c) * bins;
        for (int i = lane; i < valid; i += 32) dst[i] = cvt_out<T>(tile[i] / g.count);
        __syncwarp();
    }
}

// The transpose, plane by plane: grad rows contracted along z, expanded along y, then along x into the touched voxels of
// the plane, which are added to grad_features: kVec = 4 consecutive voxels per 16-byte reduction where the rows allow it
// (untouched voxels of such a vector get zeros).
template <typename T, int kVec>
__global__ void __launch_bounds__(kRoiThreads) roi_align3d_backward_separable_kernel(const T *__restrict__ grad_out, const float *__restrict__ rois,
                                                                                    float spatial_scale, int sampling_ratio, int order,
                                                                                    int channels, int depth, int height, int width, int pd,
                                                                                    int ph, int pw, int channels_per_block,
                                                                                    float *__restrict__ grad_features) {
    constexpr int kC = kRoiChannels;
    extern __shared__ __align__(16) float roi_smem[];
    const int n = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    RoiTables t;
    const RoiGeom g = build_roi_tables<float, kVec>(t, roi_smem, rois + (size_t)n * 7, spatial_scale, sampling_ratio, order, depth, height, width, pd, ph, pw);
    const int bins = pd * ph * pw, rows_size = height * pw, plane_size = ph * pw;
    float *rows = t.end + warp * kC * (rows_size + bins + plane_size), *tile = rows + kC * rows_size, *plane = tile + kC * bins;
    const int rows_per_step = 32 / pw, lane_row = lane / pw, p = lane - lane_row * pw;
    const bool used = lane_row < rows_per_step;
    const int ny = t.y.n, nv = t.x.n;
    const int c_end = min(channels, ((int)blockIdx.y + 1) * channels_per_block);
    const size_t volume = (size_t)depth * height * width;
    if (t.z.n == 0 || ny == 0 || nv == 0) return;  // no valid sample (uniform over the block)
    for (int c = blockIdx.y * channels_per_block + warp * kC; c < c_end; c += warps * kC) {
        float *vol = grad_features + ((size_t)g.batch * channels + c) * volume;
        const T *src = grad_out + ((size_t)n * channels + c) * (size_t)bins;
        const int valid = min(kC, c_end - c);
        bool finite = true;
        for (int i = lane; i < kC * bins; i += 32) {
            tile[i] = i < valid * bins ? ldf<T>(src + i) / g.count : 0.f;
            finite &= isfinite(tile[i]);
        }
        finite = __all_sync(0xffffffffu, finite);
        __syncwarp();
        for (int z = 0; z < t.z.n; ++z) {
            for (int i = lane; i < plane_size; i += 32) {
                float acc[kC];
#pragma unroll
                for (int k = 0; k < kC; ++k) acc[k] = 0.f;
                for (int d = t.z.first_bin(z), last = t.z.last_bin(z); d <= last; ++d) {
                    const float w = t.z.w[d * depth + z];
#pragma unroll
                    for (int k = 0; k < kC; ++k) acc[k] = fmaf(w, tile[k * bins + d * plane_size + i], acc[k]);
                }
#pragma unroll
                for (int k = 0; k < kC; ++k) plane[k * plane_size + i] = acc[k];
            }
            __syncwarp();
            if (used)
                for (int y = lane_row; y < ny; y += rows_per_step) {
                    float acc[kC];
#pragma unroll
                    for (int k = 0; k < kC; ++k) acc[k] = 0.f;
                    for (int q = t.y.first_bin(y), last = t.y.last_bin(y); q <= last; ++q) {
                        const float w = t.y.w[q * height + y];
#pragma unroll
                        for (int k = 0; k < kC; ++k) acc[k] = fmaf(w, plane[k * plane_size + q * pw + p], acc[k]);
                    }
#pragma unroll
                    for (int k = 0; k < kC; ++k) rows[k * rows_size + y * pw + p] = acc[k];
                }
            __syncwarp();
            float *plane_dst = vol + (size_t)t.z.vox[z] * height * width;
            int r = lane / nv, v = lane - r * nv;            // row and vector of this lane, advanced without divisions
            const int step_r = 32 / nv, step_v = 32 - step_r * nv;
            while (r < ny) {
                const int x = t.x.vox[v] * kVec;
                float acc[kC][kVec];
#pragma unroll
                for (int k = 0; k < kC; ++k)
#pragma unroll
                    for (int e = 0; e < kVec; ++e) acc[k][e] = 0.f;
                int first = t.x.bins, last = -1;
#pragma unroll
                for (int e = 0; e < kVec; ++e) {
                    const int lo = t.x.first_bin(x + e), hi = t.x.last_bin(x + e);
                    if (lo <= hi) {
                        first = min(first, lo);
                        last = max(last, hi);
                    }
                }
                auto add_bins = [&](auto all_voxels) {
                    for (int b = first; b <= last; ++b) {
                        const float *w = t.x.w + b * width + x;
                        float we[kVec];
                        if constexpr (kVec == 4) {
                            const float4 w4 = *reinterpret_cast<const float4 *>(w);
                            we[0] = w4.x; we[1] = w4.y; we[2] = w4.z; we[3] = w4.w;
                        } else {
                            we[0] = w[0];
                        }
                        bool touched[kVec];
#pragma unroll
                        for (int e = 0; e < kVec; ++e) touched[e] = all_voxels.value || (t.x.first_bin(x + e) <= b && b <= t.x.last_bin(x + e));
#pragma unroll
                        for (int k = 0; k < kC; ++k) {
                            const float u = rows[k * rows_size + r * pw + b];
#pragma unroll
                            for (int e = 0; e < kVec; ++e)
                                if (touched[e]) acc[k][e] = fmaf(we[e], u, acc[k][e]);
                        }
                    }
                };
                if (finite) add_bins(std::true_type{});
                else add_bins(std::false_type{});  // zero times infinity only where the bin touches the voxel
                float *dst = plane_dst + (size_t)t.y.vox[r] * width + x;
#pragma unroll
                for (int k = 0; k < kC; ++k)
                    if (k < valid) {
                        if constexpr (kVec == 4)
                            asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst + k * volume), "f"(acc[k][0]),
                                         "f"(acc[k][1]), "f"(acc[k][2]), "f"(acc[k][3]) : "memory");
                        else
                            atomicAdd(dst + k * volume, acc[k][0]);
                    }
                r += step_r;
                v += step_v;
                if (v >= nv) {
                    v -= nv;
                    ++r;
                }
            }
            __syncwarp();
        }
    }
}

// Whether a call is left to the element-wise kernels: at most 2x2x2 samples per bin and few corners in all.  They start their
// loads at once and use a thread per output element, 5 to 20 us however large the ROIs are; the separable form first builds
// its tables and then walks the planes of a ROI one after the other, 9 us and up.  More samples are a serial chain in a thread
// (4x4x4: 40 us and up), and past these counts of corners the element-wise kernels are bound by them (0.9 ps a load, 2.4 ps a
// reduction).  Measured on 8 and 256 ROIs x 16 and 128 channels of 3 to 100 % of volumes up to 32x64x256, us element-wise
// against separable, 2x2x2 samples: forward 2.8 M corners 9-11 / 17-200, 8 M 13-38 / 12-250, 17 M 39-55 / 32-90, 22 M 27-100 /
// 19-300, 33 M 36-84 / 15-80; backward 1.8 M 12-20 / 13-30, 2.8 M 17-26 / 19-190, 8 M 31-96 / 15-80.  With adaptive sampling the
// host knows only the most samples a bin can have inside the volume.
bool roi_elementwise_pays(int num_rois, int channels, int depth, int height, int width, int pd, int ph, int pw, int sampling_ratio,
                          bool backward) {
    auto along = [&](int size, int bins) { return sampling_ratio > 0 ? (double)sampling_ratio : (double)((size + bins - 1) / bins); };
    const double samples = along(depth, pd) * along(height, ph) * along(width, pw);
    return samples <= 8.0 && (double)num_rois * channels * pd * ph * pw * samples * 8.0 <= (backward ? 3e6 : 16e6);
}

// Launch shape of the separable kernels, or false: a call that the element-wise kernels do faster, a row of bins wider than a
// warp, or tables and tiles beyond shared memory even for one warp.
struct RoiLaunch {
    int threads, channels_per_block;
    size_t smem;
    dim3 grid;
};
bool roi_launch(int num_rois, int channels, int depth, int height, int width, int pd, int ph, int pw, int sampling_ratio, bool backward,
                RoiLaunch &l) {
    const int mode = fda::config().roi_separable;
    if (mode <= 0 || (mode == 1 && roi_elementwise_pays(num_rois, channels, depth, height, width, pd, ph, pw, sampling_ratio, backward))) return false;
    if (pw > 32 || (double)pd * depth + (double)ph * height + (double)pw * width > 40000.0 || (double)pd * ph * pw > 40000.0) return false;
    const size_t tables = (size_t)roi_tables_words(pd, ph, pw, depth, height, width);
    const size_t per_warp = kRoiChannels * ((size_t)height * pw + (size_t)pd * ph * pw + (backward ? (size_t)ph * pw : 0));
    l.threads = kRoiThreads;
    auto bytes = [&]() { return (tables + (size_t)(l.threads / 32) * per_warp) * sizeof(float); };
    while (l.threads > 32 && bytes() > 56 * 1024) l.threads /= 2;  // four blocks of an SM
    l.smem = bytes();
    if (l.smem > 200 * 1024) return false;
    // the tables are shared by a block's channels: up to 64 of them while the SMs still get six blocks each
    l.channels_per_block = l.threads / 32 * kRoiChannels;
    while (l.channels_per_block < 64 && (size_t)num_rois * ((channels + 2 * l.channels_per_block - 1) / (2 * l.channels_per_block)) >= 148 * 6)
        l.channels_per_block *= 2;
    l.grid = dim3((unsigned)num_rois, (unsigned)((channels + l.channels_per_block - 1) / l.channels_per_block));
    return l.grid.y <= 65535;
}

template <typename K>
cudaError_t roi_opt_in(K kernel, size_t smem) {
    return smem > 48 * 1024 ? cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024) : cudaSuccess;
}

// ---------------------------------------------------------------------------------------------------------
// NMS 3D
// ---------------------------------------------------------------------------------------------------------
constexpr int kNmsBlock = 64;  // boxes per block = bits per mask word

__device__ __forceinline__ float intersection3d(const float *a, const float *b) {
    const float left = fmaxf(a[0], b[0]), right = fminf(a[3], b[3]);
    const float top = fmaxf(a[1], b[1]), bottom = fminf(a[4], b[4]);
    const float front = fmaxf(a[2], b[2]), back = fminf(a[5], b[5]);
    const float w = fmaxf(right - left, 0.f), h = fmaxf(bottom - top, 0.f), d = fmaxf(back - front, 0.f);
    return w * h * d;
}

__device__ __forceinline__ float iou3d(const float *a, const float *b) {
    const float inter = intersection3d(a, b);
    const float sa = (a[3] - a[0]) * (a[4] - a[1]) * (a[5] - a[2]);
    const float sb = (b[3] - b[0]) * (b[4] - b[1]) * (b[5] - b[2]);
    return inter / (sa + sb - inter);
}

// Score order without a sort: the rank of box i is the number of boxes with a higher score, plus those with the same
// score that come earlier (what a stable descending sort gives; NaN counts as the highest, -0 as 0).  n^2 comparisons
// of 32-bit keys in shared memory; eight lanes share one box.  Also moves the box to its place.  Replaces a library
// sort, two gathers and their conversions (together 40 us of launches at 4000 boxes, this kernel 11); the comparisons
// grow with n^2, so beyond kRankMaxBoxes the caller sorts.
constexpr int kRankMaxBoxes = 16384;
constexpr int kRankThreads = 512, kRankBoxes = kRankThreads / 8, kRankTile = 4096;

__device__ __forceinline__ unsigned int score_key(float v) {
    if (v != v) return 0xffffffffu;
    const unsigned int u = __float_as_uint(v + 0.0f);
    return (u >> 31) ? ~u : u | 0x80000000u;
}

__global__ void __launch_bounds__(kRankThreads) nms3d_rank_kernel(int n, const float *__restrict__ boxes, long long box_stride,
                                                                  long long coord_stride, const float *__restrict__ scores,
                                                                  long long score_stride, float *__restrict__ sorted,
                                                                  int *__restrict__ order) {
    __shared__ __align__(16) unsigned int keys[kRankTile];
    const int first = blockIdx.x * kRankBoxes, i = first + (int)(threadIdx.x >> 3), sub = threadIdx.x & 7;
    const unsigned int mine = i < n ? score_key(scores[i * score_stride]) : 0u;
    int rank = 0;
    for (int base = 0; base < n; base += kRankTile) {
        const int size = min(n - base, kRankTile), padded = (size + 31) & ~31;
        __syncthreads();  // the previous tile has been read
        for (int j = threadIdx.x; j < padded; j += kRankThreads)
            keys[j] = j < size ? score_key(scores[(base + j) * score_stride]) : 0u;  // padding is never ahead of a box: it comes later
        __syncthreads();
        for (int j = 4 * sub; j < padded; j += 32) {
            const uint4 k = *reinterpret_cast<const uint4 *>(keys + j);
            const int at = base + j - i;  // negative: an earlier box, which also wins a tie
            rank += (k.x > mine) | ((k.x == mine) & (at < 0));
            rank += (k.y > mine) | ((k.y == mine) & (at < -1));
            rank += (k.z > mine) | ((k.z == mine) & (at < -2));
            rank += (k.w > mine) | ((k.w == mine) & (at < -3));
        }
    }
#pragma unroll
    for (int m = 4; m > 0; m >>= 1) rank += __shfl_xor_sync(0xffffffffu, rank, m);
    if (i >= n) return;
    if (sub < 6) sorted[(size_t)rank * 6 + sub] = boxes[i * box_stride + sub * coord_stride];
    if (sub == 6) order[rank] = i;
}

// mask[cb * n + i] for boxes i (score order) of the blocks before column block cb: bit j = box i suppresses box
// cb*64 + j.  On the diagonal the word is the other way round, bit j = box cb*64 + j (< i) suppresses box i: what the
// sweep asks there.  Boxes are [n][6], sorted by score.  Column-major, so that the sweep reads a column's words
// contiguously.  Most pairs do not overlap: their IoU is 0 (or 0/0) and no threshold >= 0 is passed, so the volumes and
// the division are only computed for the pairs that do (35 -> 16 us at 4000 boxes).
__global__ void __launch_bounds__(kNmsBlock) nms3d_mask_kernel(int n, float threshold, const float *__restrict__ boxes,
                                                               unsigned long long *__restrict__ mask) {
    const int row_start = blockIdx.y, col_start = blockIdx.x;
    if (col_start < row_start) return;  // the sweep only reads words at or right of the diagonal
    const int row_size = min(n - row_start * kNmsBlock, kNmsBlock), col_size = min(n - col_start * kNmsBlock, kNmsBlock);
    __shared__ float4 cols_lo[kNmsBlock];
    __shared__ float2 cols_hi[kNmsBlock];
    if ((int)threadIdx.x < col_size) {
        const float *c = boxes + (size_t)(col_start * kNmsBlock + threadIdx.x) * 6;
        cols_lo[threadIdx.x] = make_float4(c[0], c[1], c[2], c[3]);
        cols_hi[threadIdx.x] = make_float2(c[4], c[5]);
    }
    __syncthreads();
    if ((int)threadIdx.x < row_size) {
        const int cur = row_start * kNmsBlock + threadIdx.x;
        float a[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) a[k] = boxes[(size_t)cur * 6 + k];
        const bool diagonal = row_start == col_start, may_skip = threshold >= 0.f;
        unsigned long long t = 0;
        const int end = diagonal ? (int)threadIdx.x : col_size;
        for (int i = 0; i < end; ++i) {
            const float4 lo = cols_lo[i];
            const float2 hi = cols_hi[i];
            const float b[6] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y};
            if (may_skip && intersection3d(a, b) == 0.f) continue;
            if ((diagonal ? iou3d(b, a) : iou3d(a, b)) > threshold) t |= 1ULL << i;
        }
        mask[(size_t)col_start * n + cur] = t;
    }
}

__device__ __forceinline__ unsigned long long warp_or(unsigned long long v) {
    const unsigned int lo = __reduce_or_sync(0xffffffffu, (unsigned int)v), hi = __reduce_or_sync(0xffffffffu, (unsigned int)(v >> 32));
    return (unsigned long long)hi << 32 | lo;
}
__device__ __forceinline__ void cp_async8(void *smem, const void *gmem) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned int)__cvta_generic_to_shared(smem)), "l"(gmem) : "memory");
}

// Greedy sweep in score order, one block; iteration cb decides the 64 boxes of chunk cb.  keep[0 .. *num_keep) = the kept
// boxes (positions in score order, or order[position] when given).  A serial chain of n / 64 iterations, so what counts
// is the length of one:
//   warp 0      resolves chunk cb: boxes removed by chunks 0..cb-2 come from the other warps, by chunk cb-1 from 64
//               words, inside the chunk by rounds (an undecided box that no undecided earlier box suppresses is kept, what
//               it suppresses goes), as many as the longest chain of suppressions, not as there are boxes.  Its words
//               are copied to shared memory kSweepAhead chunks ahead.
//   warps 1..31 meanwhile collect what chunks 0..cb-1 remove from chunk cb+1, from words loaded two iterations before.
// 1256 -> 39 us at 4000 boxes (one thread deciding box after box with a global load each, before).
constexpr int kSweepThreads = 1024, kSweepAhead = 4, kSweepWords = 4;

__global__ void __launch_bounds__(kSweepThreads) nms3d_sweep_kernel(int n, int col_blocks, const unsigned long long *__restrict__ mask,
                                                                    const int *__restrict__ order, long long *__restrict__ keep,
                                                                    int *__restrict__ num_keep) {
    extern __shared__ unsigned long long kept_words[];            // [col_blocks] kept boxes of every decided chunk
    int *kept_before = reinterpret_cast<int *>(kept_words + col_blocks);  // [col_blocks / 2, up] boxes kept before every even chunk
    __shared__ unsigned long long removed_by_far[2][32];          // chunk c: what chunks 0..c-2 remove, by warp, slot c % 2
    __shared__ unsigned long long near_words[kSweepAhead][2 * kNmsBlock];  // chunk c: the words of chunk c-1, then of c itself
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, far_thread = (int)threadIdx.x - 32;
    constexpr int kFarThreads = kSweepThreads - 32;

    auto request_near = [&](int c) {  // warp 0; every lane commits one (possibly empty) group per chunk
        if (c < col_blocks) {
            unsigned long long *slot = near_words[c % kSweepAhead];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int w = lane + 32 * k, row = (c - 1) * kNmsBlock + w;
                if (row >= 0 && row < n) cp_async8(slot + w, mask + (size_t)c * n + row);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    unsigned long long words[2][kSweepWords];
    auto load_far = [&](int c, unsigned long long (&w)[kSweepWords]) {  // the words of chunks 0..c-2 in column c
        const int rows = c < col_blocks ? (c - 1) * kNmsBlock : 0;
#pragma unroll
        for (int k = 0; k < kSweepWords; ++k) {
            const int r = far_thread + k * kFarThreads;
            w[k] = r < rows ? __ldg(mask + (size_t)c * n + r) : 0ull;
        }
    };
    auto collect_far = [&](int c, const unsigned long long (&w)[kSweepWords]) {
        if (c >= col_blocks) return;
        const int rows = (c - 1) * kNmsBlock;
        unsigned long long acc = 0ull;
#pragma unroll
        for (int k = 0; k < kSweepWords; ++k) {
            const int r = far_thread + k * kFarThreads;
            if (r < rows && (kept_words[r >> 6] >> (r & 63) & 1ull)) acc |= w[k];
        }
        for (int r = far_thread + kSweepWords * kFarThreads; r < rows; r += kFarThreads)
            if (kept_words[r >> 6] >> (r & 63) & 1ull) acc |= __ldg(mask + (size_t)c * n + r);
        acc = warp_or(acc);
        if (lane == 0) removed_by_far[c & 1][warp] = acc;
    };

    if (threadIdx.x < 64) removed_by_far[threadIdx.x >> 5][threadIdx.x & 31] = 0ull;  // chunk 0 and warp 0 add nothing
    if (warp == 0) {
        for (int c = 0; c < kSweepAhead - 1; ++c) request_near(c);
    } else {
        load_far(1, words[0]);
        load_far(2, words[1]);
    }
    __syncthreads();
    int total = 0;
    auto iteration = [&](int cb, unsigned long long (&w)[kSweepWords]) {
        if (warp == 0) {
            request_near(cb + kSweepAhead - 1);  // into the slot of chunk cb - 1
            asm volatile("cp.async.wait_group %0;" ::"n"(kSweepAhead - 1) : "memory");
            __syncwarp();
            const unsigned long long *slot = near_words[cb % kSweepAhead];
            const int size = min(n - cb * kNmsBlock, kNmsBlock);
            unsigned long long removed = 0ull;
            if (cb > 0) {
                const unsigned long long prev = kept_words[cb - 1];
                removed = warp_or(((prev >> lane & 1ull) ? slot[lane] : 0ull) | ((prev >> (lane + 32) & 1ull) ? slot[lane + 32] : 0ull) |
                                  removed_by_far[cb & 1][lane]);
            }
            // earlier boxes of the chunk that suppress box lane (low half only) and box lane + 32
            const unsigned int by0 = lane < size ? (unsigned int)slot[kNmsBlock + lane] : 0u;
            const unsigned long long by1 = lane + 32 < size ? slot[kNmsBlock + lane + 32] : 0ull;
            const unsigned int by1_lo = (unsigned int)by1, by1_hi = (unsigned int)(by1 >> 32), bit = 1u << lane;
            const unsigned long long start = ~removed & (size == 64 ? ~0ull : (1ull << size) - 1ull);
            unsigned int lo = (unsigned int)start, hi = (unsigned int)(start >> 32), kept_lo = 0u, kept_hi = 0u;
            while (lo | hi) {
                const bool o0 = lo & bit, o1 = hi & bit;
                const unsigned int sure_lo = __ballot_sync(0xffffffffu, o0 && !(by0 & lo));
                const unsigned int sure_hi = __ballot_sync(0xffffffffu, o1 && !((by1_lo & lo) | (by1_hi & hi)));
                const unsigned int gone_lo = __ballot_sync(0xffffffffu, o0 && (by0 & sure_lo));
                const unsigned int gone_hi = __ballot_sync(0xffffffffu, o1 && ((by1_lo & sure_lo) | (by1_hi & sure_hi)));
                kept_lo |= sure_lo;  // sure is never empty: the first open box is sure
                kept_hi |= sure_hi;
                lo &= ~(sure_lo | gone_lo);
                hi &= ~(sure_hi | gone_hi);
            }
            const unsigned long long kept = (unsigned long long)kept_hi << 32 | kept_lo;
            if (lane == 0) {
                kept_words[cb] = kept;
                if (!(cb & 1)) kept_before[cb >> 1] = total;
            }
            total += __popcll(kept);
        } else {
            collect_far(cb + 1, w);
            load_far(cb + 3, w);
        }
        __syncthreads();
    };
    for (int cb = 0; cb < col_blocks; cb += 2) {
        iteration(cb, words[0]);
        if (cb + 1 < col_blocks) iteration(cb + 1, words[1]);  // uniform over the block
    }
    for (int r = threadIdx.x; r < n; r += kSweepThreads) {
        const unsigned long long kept = kept_words[r >> 6];
        if (kept >> (r & 63) & 1ull) {
            const int before = kept_before[r >> 7] + ((r >> 6 & 1) ? __popcll(kept_words[(r >> 6) - 1]) : 0);
            keep[before + __popcll(kept & ((1ull << (r & 63)) - 1ull))] = order ? order[r] : r;
        }
    }
    if (threadIdx.x == 0) *num_keep = total;
}

inline int status_of(cudaError_t e) {
    if (e == cudaSuccess) return FDA_OK;
    fda::record_cuda_error((int)e);
    return FDA_ERR_CUDA;
}

inline unsigned grid_for(size_t total) {
    size_t blocks = (total + 255) / 256;
    const size_t cap = 148 * 32;  // grid-stride beyond that
    return (unsigned)(blocks > cap ? cap : (blocks ? blocks : 1));
}

}  // namespace

extern "C" int fda_roi_align3d_forward(const void *features, const void *rois, void *output, int num_rois, int channels,
                                       int depth, int height, int width, int pooled_depth, int pooled_height,
                                       int pooled_width, float spatial_scale, int sampling_ratio, int order, int dtype,
                                       void *stream) {
    if (!features || !rois || !output) return FDA_ERR_NULL_POINTER;
    if (dtype < 0 || dtype > 2) return FDA_ERR_BAD_DTYPE;
    if (num_rois < 0 || channels <= 0 || depth <= 0 || height <= 0 || width <= 0 || pooled_depth <= 0 || pooled_height <= 0 ||
        pooled_width <= 0 || (order != 0 && order != 1))
        return FDA_ERR_BAD_SHAPE;
    const size_t total = (size_t)num_rois * channels * pooled_depth * pooled_height * pooled_width;
    if (total == 0) return FDA_OK;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    RoiLaunch l;
    if (roi_launch(num_rois, channels, depth, height, width, pooled_depth, pooled_height, pooled_width, sampling_ratio, false, l)) {
        auto launch = [&](auto kernel, auto *typed) -> int {
            using T = std::remove_pointer_t<decltype(typed)>;
            const cudaError_t e = roi_opt_in(kernel, l.smem);
            if (e != cudaSuccess) return status_of(e);
            kernel<<<l.grid, l.threads, l.smem, st>>>(static_cast<const T *>(features), static_cast<const T *>(rois), spatial_scale,
                                                      sampling_ratio, order, channels, depth, height, width, pooled_depth, pooled_height,
                                                      pooled_width, l.channels_per_block, typed);
            return status_of(cudaGetLastError());
        };
        if (dtype == FDA_DTYPE_F32) return launch(roi_align3d_forward_separable_kernel<float>, static_cast<float *>(output));
        if (dtype == FDA_DTYPE_F16) return launch(roi_align3d_forward_separable_kernel<__half>, static_cast<__half *>(output));
        return launch(roi_align3d_forward_separable_kernel<__nv_bfloat16>, static_cast<__nv_bfloat16 *>(output));
    }
    const unsigned g = grid_for(total);
#define FDA_ROI_FWD(T)                                                                                                     \
    roi_align3d_forward_kernel<T><<<g, 256, 0, st>>>(total, static_cast<const T *>(features), static_cast<const T *>(rois),    \
                                                     spatial_scale, sampling_ratio, order, channels, depth, height, width,   \
                                                     pooled_depth, pooled_height, pooled_width, static_cast<T *>(output))
    if (dtype == FDA_DTYPE_F32) FDA_ROI_FWD(float);
    else if (dtype == FDA_DTYPE_F16) FDA_ROI_FWD(__half);
    else FDA_ROI_FWD(__nv_bfloat16);
#undef FDA_ROI_FWD
    return status_of(cudaGetLastError());
}

extern "C" int fda_roi_align3d_backward(const void *grad_output, const float *rois, float *grad_features, int num_rois,
                                        int channels, int depth, int height, int width, int pooled_depth,
                                        int pooled_height, int pooled_width, float spatial_scale, int sampling_ratio,
                                        int order, int grad_output_dtype, void *stream) {
    if (!grad_output || !rois || !grad_features) return FDA_ERR_NULL_POINTER;
    if (grad_output_dtype < 0 || grad_output_dtype > 2) return FDA_ERR_BAD_DTYPE;
    if (num_rois < 0 || channels <= 0 || depth <= 0 || height <= 0 || width <= 0 || pooled_depth <= 0 || pooled_height <= 0 ||
        pooled_width <= 0 || (order != 0 && order != 1))
        return FDA_ERR_BAD_SHAPE;
    const size_t total = (size_t)num_rois * channels * pooled_depth * pooled_height * pooled_width;
    if (total == 0) return FDA_OK;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    RoiLaunch l;
    if (roi_launch(num_rois, channels, depth, height, width, pooled_depth, pooled_height, pooled_width, sampling_ratio, true, l)) {
        const bool vec = width % 4 == 0 && (reinterpret_cast<uintptr_t>(grad_features) & 15u) == 0;
        auto launch = [&](auto kernel, const auto *typed) -> int {
            const cudaError_t e = roi_opt_in(kernel, l.smem);
            if (e != cudaSuccess) return status_of(e);
            kernel<<<l.grid, l.threads, l.smem, st>>>(typed, rois, spatial_scale, sampling_ratio, order, channels, depth, height, width,
                                                      pooled_depth, pooled_height, pooled_width, l.channels_per_block, grad_features);
            return status_of(cudaGetLastError());
        };
        auto typed_launch = [&](const auto *typed) -> int {
            using T = std::remove_cv_t<std::remove_pointer_t<decltype(typed)>>;
            return vec ? launch(roi_align3d_backward_separable_kernel<T, 4>, typed) : launch(roi_align3d_backward_separable_kernel<T, 1>, typed);
        };
        if (grad_output_dtype == FDA_DTYPE_F32) return typed_launch(static_cast<const float *>(grad_output));
        if (grad_output_dtype == FDA_DTYPE_F16) return typed_launch(static_cast<const __half *>(grad_output));
        return typed_launch(static_cast<const __nv_bfloat16 *>(grad_output));
    }
    const unsigned g = grid_for(total);
#define FDA_ROI_BWD(T)                                                                                                      \
    roi_align3d_backward_kernel<T><<<g, 256, 0, st>>>(total, static_cast<const T *>(grad_output), rois, spatial_scale,           \
                                                      sampling_ratio, order, channels, depth, height, width, pooled_depth,    \
                                                      pooled_height, pooled_width, grad_features)
    if (grad_output_dtype == FDA_DTYPE_F32) FDA_ROI_BWD(float);
    else if (grad_output_dtype == FDA_DTYPE_F16) FDA_ROI_BWD(__half);
    else FDA_ROI_BWD(__nv_bfloat16);
#undef FDA_ROI_BWD
    return status_of(cudaGetLastError());
}

namespace {

size_t nms_mask_bytes(int num_boxes) {
    const size_t col_blocks = ((size_t)num_boxes + kNmsBlock - 1) / kNmsBlock;
    return (size_t)num_boxes * col_blocks * sizeof(unsigned long long);
}

int launch_nms(const float *boxes_sorted, const int *order, int num_boxes, float iou_threshold, unsigned long long *mask,
               long long *keep, int *num_keep, cudaStream_t st) {
    const int col_blocks = (num_boxes + kNmsBlock - 1) / kNmsBlock;
    const size_t smem = (size_t)col_blocks * sizeof(unsigned long long) + ((size_t)col_blocks + 1) / 2 * sizeof(int);
    if (smem > 200 * 1024) return FDA_ERR_TOO_LARGE_STATIC;  // 1.31 M boxes; the matrix of 1.24 M fills the memory of the GPU
    nms3d_mask_kernel<<<dim3((unsigned)col_blocks, (unsigned)col_blocks), kNmsBlock, 0, st>>>(num_boxes, iou_threshold, boxes_sorted, mask);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return status_of(e);
    if (smem > 40 * 1024) {
        e = cudaFuncSetAttribute(nms3d_sweep_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        if (e != cudaSuccess) return status_of(e);
    }
    nms3d_sweep_kernel<<<1, kSweepThreads, smem, st>>>(num_boxes, col_blocks, mask, order, keep, num_keep);
    return status_of(cudaGetLastError());
}

}  // namespace

extern "C" size_t fda_nms3d_workspace_bytes(int num_boxes) { return num_boxes <= 0 ? 0 : nms_mask_bytes(num_boxes); }

extern "C" int fda_nms3d(const float *boxes_sorted, int num_boxes, float iou_threshold, void *workspace,
                         size_t workspace_bytes, long long *keep, int *num_keep, void *stream) {
    if (!boxes_sorted || !keep || !num_keep) return FDA_ERR_NULL_POINTER;
    if (num_boxes < 0) return FDA_ERR_BAD_SHAPE;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (num_boxes == 0) return status_of(cudaMemsetAsync(num_keep, 0, sizeof(int), st));
    if (!workspace || workspace_bytes < nms_mask_bytes(num_boxes)) return FDA_ERR_WORKSPACE;
    return launch_nms(boxes_sorted, nullptr, num_boxes, iou_threshold, static_cast<unsigned long long *>(workspace), keep, num_keep, st);
}

extern "C" size_t fda_nms3d_scored_workspace_bytes(int num_boxes) {
    if (num_boxes <= 0 || num_boxes > kRankMaxBoxes) return 0;
    return nms_mask_bytes(num_boxes) + (size_t)num_boxes * (6 * sizeof(float) + sizeof(int));
}

extern "C" int fda_nms3d_scored(const float *boxes, long long box_stride, long long coord_stride, const float *scores,
                                long long score_stride, int num_boxes, float iou_threshold, void *workspace,
                                size_t workspace_bytes, long long *keep, int *num_keep, void *stream) {
    if (!boxes || !scores || !keep || !num_keep) return FDA_ERR_NULL_POINTER;
    if (num_boxes <= 0) return FDA_ERR_BAD_SHAPE;
    if (num_boxes > kRankMaxBoxes) return FDA_ERR_TOO_LARGE_STATIC;
    if (!workspace || workspace_bytes < fda_nms3d_scored_workspace_bytes(num_boxes)) return FDA_ERR_WORKSPACE;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    auto *mask = static_cast<unsigned long long *>(workspace);
    auto *sorted = reinterpret_cast<float *>(static_cast<char *>(workspace) + nms_mask_bytes(num_boxes));
    auto *order = reinterpret_cast<int *>(sorted + (size_t)num_boxes * 6);
    nms3d_rank_kernel<<<(unsigned)((num_boxes + kRankBoxes - 1) / kRankBoxes), kRankThreads, 0, st>>>(
        num_boxes, boxes, box_stride, coord_stride, scores, score_stride, sorted, order);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return status_of(e);
    return launch_nms(sorted, order, num_boxes, iou_threshold, mask, keep, num_keep, st);
}
