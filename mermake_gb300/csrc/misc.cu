// Small kernels behind the library's general entry points:
//   mirror       fill.py:6-52       in-place reflect about index i along one axis
//   box_1d       blur.cu:1-52       truncated-window mean along one axis (any layout)
//   subtract     math.py:4-33       uint16 saturating / reflecting subtraction
//   sumsq        __main__.py:221    sum of squares for the DAPI RMS (double accumulation)
#include <float.h>
#include <stdint.h>
#include "deconv.cuh"

namespace {

struct NdShape {
    int ndim;
    long long shape[8];
    long long stride[8];  // elements
};

__global__ void k_mirror(float *arr, NdShape s, long long size, int axis, int i, int mode) {
    for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < size;
         idx += (long long)gridDim.x * blockDim.x) {
        long long tmp = idx, off = 0, j = 0;
        for (int d = s.ndim - 1; d >= 0; --d) {
            long long c = tmp % s.shape[d];
            tmp /= s.shape[d];
            off += c * s.stride[d];
            if (d == axis) j = c;
        }
        long long n = s.shape[axis], dist = j - i, src;
        if (mode == 0 && dist > 0) {
            src = i - dist;
            if (src < 0) continue;
        } else if (mode == 1 && dist < 0) {
            src = i - dist;
            if (src >= n) continue;
        } else {
            continue;
        }
        arr[off] = arr[off + (src - j) * s.stride[axis]];
    }
}

// One thread per output voxel; the window is read along `axis` (strides in elements).
__global__ void k_box_1d(const float *__restrict__ in, float *__restrict__ out, int sz, int sx, int sy,
                         long long isz, long long isx, long long isy, long long osz, long long osx, long long osy,
                         int delta, int axis) {
    const long long total = (long long)sz * sx * sy;
    for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (long long)gridDim.x * blockDim.x) {
        int z = (int)(idx / ((long long)sx * sy));
        int x = (int)((idx / sy) % sx);
        int y = (int)(idx % sy);
        int c = axis == 0 ? z : (axis == 1 ? x : y);
        int n = axis == 0 ? sz : (axis == 1 ? sx : sy);
        long long st = axis == 0 ? isz : (axis == 1 ? isx : isy);
        long long b = z * isz + x * isx + y * isy - c * st;
        int s = c - delta < 0 ? 0 : c - delta;
        int e = c + delta > n - 1 ? n - 1 : c + delta;
        float sum = 0.f;
        for (int i = s; i <= e; ++i) sum += in[b + i * st];
        out[z * osz + x * osx + y * osy] = e >= s ? sum / (float)(e - s + 1) : 0.f;
    }
}

__global__ void k_subtract_u16(const uint16_t *__restrict__ x, const uint16_t *__restrict__ y,
                               uint16_t *__restrict__ z, NdShape sx, NdShape sy, NdShape sz, long long size,
                               int mode) {
    for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < size;
         idx += (long long)gridDim.x * blockDim.x) {
        long long tmp = idx, ox = 0, oy = 0, oz = 0;
        for (int d = sx.ndim - 1; d >= 0; --d) {
            long long c = tmp % sx.shape[d];
            tmp /= sx.shape[d];
            ox += c * sx.stride[d];
            oy += c * sy.stride[d];
            oz += c * sz.stride[d];
        }
        uint16_t a = x[ox], b = y[oy];
        // mode 0: subtract_clamp (math.py:4-11); mode 1: subtract_reflect (math.py:20-27)
        z[oz] = mode == 0 ? (uint16_t)(a > b ? a - b : 0) : (uint16_t)(a >= b ? a - b : b - a);
    }
}

// The same where the last axis is dense in all three arrays: a warp per row,
// two pixels per lane and step.  Bound by DRAM (6 bytes a pixel); a pair that
// starts on the second half of a word is read as two half words, so nothing
// outside the row is touched.  49 x 2041 x 2036 pixels: 1.44 ms in the general
// kernel (64-bit divisions per pixel).
__device__ __forceinline__ unsigned two_u16(const uint16_t *p, bool aligned) {
    return aligned ? *reinterpret_cast<const unsigned *>(p) : p[0] | (unsigned)p[1] << 16;
}
struct RowShape {
    long long rows;
    int n, inner;           // row length; rows of the second axis (1 for two axes)
    long long so[3], si[3]; // strides of the outer and the second axis: x, y, z
};
__device__ __forceinline__ unsigned sub_u16x2(unsigned a, unsigned b, int mode) {
    return mode == 0 ? __vsubus2(a, b) : __vabsdiffu2(a, b);
}
constexpr int kSubU = 8;  // words of each array in flight per lane
__global__ void __launch_bounds__(256) k_subtract_rows(const uint16_t *__restrict__ x, const uint16_t *__restrict__ y,
                                                       uint16_t *__restrict__ z, RowShape s, int mode) {
    const int lane = threadIdx.x & 31;
    const long long nw = (long long)gridDim.x * (blockDim.x / 32);
    for (long long r = (long long)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32; r < s.rows; r += nw) {
        const long long o = r / s.inner, i = r - o * s.inner;
        const uint16_t *xr = x + o * s.so[0] + i * s.si[0], *yr = y + o * s.so[1] + i * s.si[1];
        uint16_t *zr = z + o * s.so[2] + i * s.si[2];
        int n = s.n;
        if ((reinterpret_cast<uintptr_t>(zr) & 2) && n > 0) {  // to a word boundary of the result
            if (lane == 0) *zr = (uint16_t)sub_u16x2(*xr, *yr, mode);
            ++xr, ++yr, ++zr, --n;
        }
        const bool xa = (reinterpret_cast<uintptr_t>(xr) & 2) == 0, ya = (reinterpret_cast<uintptr_t>(yr) & 2) == 0;
        const int words = n / 2;
        for (int w0 = lane; w0 < words; w0 += 32 * kSubU) {
            unsigned a[kSubU], b[kSubU];
#pragma unroll
            for (int u = 0; u < kSubU; ++u) {
                const int w = w0 + 32 * u;
                if (w < words) {
                    a[u] = two_u16(xr + 2 * w, xa);
                    b[u] = two_u16(yr + 2 * w, ya);
                }
            }
#pragma unroll
            for (int u = 0; u < kSubU; ++u) {
                const int w = w0 + 32 * u;
                if (w < words) reinterpret_cast<unsigned *>(zr)[w] = sub_u16x2(a[u], b[u], mode);
            }
        }
        if ((n & 1) && lane == 0) zr[n - 1] = (uint16_t)sub_u16x2(xr[n - 1], yr[n - 1], mode);
    }
}

// Sums of squares in a fixed order (the result does not depend on block
// timing): each block writes its partial sum, k_sum_parts adds the partials.
// Four squares are added in float (one 16-byte load) and the group goes into
// the double accumulator, so the FP64 pipe (a small fraction of the FP32 rate
// on this part) sees one add per four elements; the relative error of a
// group is below 3e-7 and the groups add in double.
__global__ void k_sumsq(const float *__restrict__ x, long long n, double *__restrict__ parts) {
    double acc = 0.0;
    const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x, nth = (long long)gridDim.x * blockDim.x;
    long long done = 0;
    if ((reinterpret_cast<uintptr_t>(x) & 15) == 0) {
        const float4 *x4 = reinterpret_cast<const float4 *>(x);
        const long long n4 = n / 4;
        // Conversions to double and additions there bounded the pass at one each
        // per four values (0.103 ms at any grid).  Now four groups of four
        // squares are added without loss, as a float and what its rounding left
        // (two-sum, Knuth), and the left-overs, 2^-24 of the sums, collect in a
        // float.  50 x 1500 x 1302 voxels: the DAPI block's stage 0.123 -> 0.080
        // ms (four CTAs an SM; with eight the kernel alone takes 0.078 for 0.064)
        long long i = tid;
        float rest = 0.f;
        bool fine = true;
        for (; i + 3 * nth < n4; i += 4 * nth) {
            float4 v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) v[u] = x4[i + u * nth];
            float s = 0.f;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const float q = fmaf(v[u].w, v[u].w, fmaf(v[u].z, v[u].z, fmaf(v[u].y, v[u].y, v[u].x * v[u].x)));
                const float t = __fadd_rn(s, q), z = __fsub_rn(t, s);
                rest = __fadd_rn(rest, __fadd_rn(__fsub_rn(s, __fsub_rn(t, z)), __fsub_rn(q, z)));
                s = t;
            }
            fine &= s <= FLT_MAX;
            acc += (double)s;
        }
        acc += (double)rest;
        if (!fine) {  // a sum without a remainder (infinite, NaN): group by group in double
            acc = 0.0;
            i = tid;
        }
        for (; i < n4; i += nth) {
            const float4 v = x4[i];
            acc += (double)fmaf(v.w, v.w, fmaf(v.z, v.z, fmaf(v.y, v.y, v.x * v.x)));
        }
        done = n4 * 4;
    }
    for (long long i = done + tid; i < n; i += nth) {
        const double v = x[i];
        acc += v * v;
    }
    acc = mm_block_sum(acc);
    if (threadIdx.x == 0) parts[blockIdx.x] = acc;
}

__global__ void k_sum_parts(const double *__restrict__ parts, int nparts, double *__restrict__ out) {
    double acc = 0.0;
    for (int i = threadIdx.x; i < nparts; i += blockDim.x) acc += parts[i];
    acc = mm_block_sum(acc);
    if (threadIdx.x == 0) out[0] = acc;
}

// DAPI divisor (__main__.py:221-222): norm = sqrt of the sum of squares rounded
// to float (cp.linalg.norm of a float32 vector), divided in double by sqrt(N)
// (cp.sqrt of the Python int size), then rounded to float when used as the
// divisor of a float32 array.  The sum itself is accumulated in double.
__global__ void k_rms_div(const double *__restrict__ sumsq, long long n, float *__restrict__ div) {
    float norm = sqrtf((float)sumsq[0]);
    div[0] = (float)((double)norm / sqrt((double)n));
}

int grid_for(long long n) {
    long long g = (n + 255) / 256;
    if (g > 152 * 32) g = 152 * 32;
    return g < 1 ? 1 : (int)g;
}

int fill_shape(NdShape &s, int ndim, const int64_t *shape, const int64_t *strides) {
    if (ndim < 1 || ndim > 8) {
        mm_set_error("ndim %d outside [1, 8]", ndim);
        return MM_EINVAL;
    }
    s.ndim = ndim;
    for (int d = 0; d < ndim; ++d) {
        s.shape[d] = shape[d];
        s.stride[d] = strides[d];
    }
    return MM_OK;
}

}  // namespace

extern "C" int mm_reflect_f32(float *arr, int ndim, const int64_t *shape, const int64_t *strides, int axis, int i,
                              int mode, void *stream) {
    NdShape s;
    int rc = fill_shape(s, ndim, shape, strides);
    if (rc) return rc;
    MM_REQUIRE(axis >= 0 && axis < ndim, "axis %d is out of bounds for array of dimension %d", axis, ndim);
    MM_REQUIRE(i >= 0 && i < shape[axis], "index %d is out of bounds for axis %d with size %lld", i, axis,
               (long long)shape[axis]);
    MM_REQUIRE(mode == 0 || mode == 1, "mode must be 'out' (0) or 'in' (1)");
    long long size = 1;
    for (int d = 0; d < ndim; ++d) size *= shape[d];
    if (size == 0) return MM_OK;
    k_mirror<<<grid_for(size), 256, 0, (cudaStream_t)stream>>>(arr, s, size, axis, i, mode);
    MM_CHECK_LAUNCH();
    return MM_OK;
}

extern "C" int mm_box_1d_f32(const float *in, const int64_t *in_strides, float *out, const int64_t *out_strides,
                             int size_z, int size_x, int size_y, int delta, int axis, void *stream) {
    MM_REQUIRE(axis >= 0 && axis <= 2, "axis %d out of range for a (z, x, y) volume", axis);
    MM_REQUIRE(delta >= 0, "negative blur half-width %d", delta);
    long long total = (long long)size_z * size_x * size_y;
    if (total == 0) return MM_OK;
    k_box_1d<<<grid_for(total), 256, 0, (cudaStream_t)stream>>>(
        in, out, size_z, size_x, size_y, in_strides[0], in_strides[1], in_strides[2], out_strides[0],
        out_strides[1], out_strides[2], delta, axis);
    MM_CHECK_LAUNCH();
    return MM_OK;
}

extern "C" int mm_subtract_u16(const uint16_t *x, const int64_t *xs, const uint16_t *y, const int64_t *ys,
                               uint16_t *z, const int64_t *zs, int ndim, const int64_t *shape, int mode,
                               void *stream) {
    NdShape a, b, c;
    int rc;
    if ((rc = fill_shape(a, ndim, shape, xs)) || (rc = fill_shape(b, ndim, shape, ys)) ||
        (rc = fill_shape(c, ndim, shape, zs)))
        return rc;
    MM_REQUIRE(mode == 0 || mode == 1, "mode must be clamp (0) or reflect (1)");
    long long size = 1;
    for (int d = 0; d < ndim; ++d) size *= shape[d];
    if (size == 0) return MM_OK;
    // a dense last axis of at least a warp's words (a shorter row leaves most of
    // the warp idle) and at most three axes: row by row
    if (ndim <= 3 && shape[ndim - 1] >= 64 && shape[ndim - 1] < (1LL << 30) && xs[ndim - 1] == 1 &&
        ys[ndim - 1] == 1 && zs[ndim - 1] == 1) {
        RowShape s = {};
        s.rows = size / shape[ndim - 1];
        s.n = (int)shape[ndim - 1];
        const long long inner = ndim >= 2 ? shape[ndim - 2] : 1;
        const int64_t *st[3] = {xs, ys, zs};
        for (int k = 0; k < 3; ++k) {
            s.si[k] = ndim >= 2 ? st[k][ndim - 2] : 0;
            s.so[k] = ndim == 3 ? st[k][0] : 0;
        }
        if (inner < (1LL << 31)) {
            s.inner = (int)inner;
            const long long blocks = (s.rows + 7) / 8, cap = 152 * 8;
            k_subtract_rows<<<(unsigned)(blocks < cap ? blocks : cap), 256, 0, (cudaStream_t)stream>>>(x, y, z, s, mode);
            MM_CHECK_LAUNCH();
            return MM_OK;
        }
    }
    k_subtract_u16<<<grid_for(size), 256, 0, (cudaStream_t)stream>>>(x, y, z, a, b, c, size, mode);
    MM_CHECK_LAUNCH();
    return MM_OK;
}

int mm_launch_sum_parts(const double *parts, int nparts, double *out, cudaStream_t st) {
    k_sum_parts<<<1, 256, 0, st>>>(parts, nparts, out);
    MM_CHECK_LAUNCH();
    return MM_OK;
}

int mm_launch_sumsq(const float *x, long long n, double *parts, double *out, cudaStream_t st) {
    if (n == 0) {
        MM_CUDA_TRY(cudaMemsetAsync(out, 0, sizeof(double), st));
        return MM_OK;
    }
    // 16 values and more a thread, four CTAs an SM
    int g = grid_for((n + 15) / 16);
    if (g > 152 * 4) g = 152 * 4;
    k_sumsq<<<g, 256, 0, st>>>(x, n, parts);
    MM_CHECK_LAUNCH();
    return mm_launch_sum_parts(parts, g, out, st);
}

int mm_launch_rms_div(const double *sumsq, long long n, float *div, cudaStream_t st) {
    k_rms_div<<<1, 1, 0, st>>>(sumsq, n, div);
    MM_CHECK_LAUNCH();
    return MM_OK;
}

// ---------------------------------------------------------------------------
// Median of a float32 array (cp.median in mermake/io.py:52): the k-th smallest
// value by radix selection over the order-preserving bit pattern of the floats,
// four 8-bit digits, one histogram per digit; an even count averages the two
// middle values in float32 ((a + b) / 2), as the reference's mean does.
// ---------------------------------------------------------------------------
namespace {

__device__ __forceinline__ unsigned f2key(float f) {
    const unsigned u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float key2f(unsigned k) {
    const unsigned u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
    return __uint_as_float(u);
}

// state: [0] prefix, [1] mask, [2] rank still to skip inside the prefix
__global__ void k_select_hist(const float *__restrict__ x, long long n, const unsigned *__restrict__ state,
                              int shift, unsigned *__restrict__ hist) {
    __shared__ unsigned h[256];
    for (int i = threadIdx.x; i < 256; i += blockDim.x) h[i] = 0;
    __syncthreads();
    const unsigned prefix = state[0], mask = state[1];
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const unsigned k = f2key(x[i]);
        if ((k & mask) == prefix) atomicAdd(&h[(k >> shift) & 255u], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 256; i += blockDim.x)
        if (h[i]) atomicAdd(&hist[i], h[i]);
}

__global__ void k_select_pick(unsigned *__restrict__ state, unsigned *__restrict__ hist, int shift) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    unsigned r = state[2];
    int b = 0;
    for (; b < 255; ++b) {
        if (r < hist[b]) break;
        r -= hist[b];
    }
    state[0] |= (unsigned)b << shift;
    state[1] |= 255u << shift;
    state[2] = r;
    for (int i = 0; i < 256; ++i) hist[i] = 0;
}

__global__ void k_select_init(unsigned *__restrict__ state, unsigned long long rank, unsigned *__restrict__ hist) {
    state[0] = 0;
    state[1] = 0;
    state[2] = (unsigned)rank;
    for (int i = 0; i < 256; ++i) hist[i] = 0;
}

__global__ void k_median_finish(const unsigned *__restrict__ s_lo, const unsigned *__restrict__ s_hi, int even,
                                float *__restrict__ med) {
    const float a = key2f(s_lo[0]);
    med[0] = even ? (a + key2f(s_hi[0])) / 2.0f : a;
}

__global__ void k_divide(const float *__restrict__ x, long long n, const float *__restrict__ d, float *__restrict__ out) {
    const float dv = d[0];
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        out[i] = __fdiv_rn(x[i], dv);
}

int select_kth(const float *x, long long n, unsigned long long k, unsigned *state, unsigned *hist, cudaStream_t st) {
    k_select_init<<<1, 1, 0, st>>>(state, k, hist);
    MM_CHECK_LAUNCH();
    for (int shift = 24; shift >= 0; shift -= 8) {
        k_select_hist<<<grid_for(n), 256, 0, st>>>(x, n, state, shift, hist);
        MM_CHECK_LAUNCH();
        k_select_pick<<<1, 1, 0, st>>>(state, hist, shift);
        MM_CHECK_LAUNCH();
    }
    return MM_OK;
}

}  // namespace

int mm_median_impl(const float *x, long long n, unsigned *scratch, float *med_dev, float *out, cudaStream_t st) {
    // scratch: 2 x 4 state words + 256 histogram words
    unsigned *s_lo = scratch, *s_hi = scratch + 4, *hist = scratch + 8;
    int rc;
    const int even = (n % 2) == 0;
    if ((rc = select_kth(x, n, even ? n / 2 - 1 : n / 2, s_lo, hist, st))) return rc;
    if (even && (rc = select_kth(x, n, n / 2, s_hi, hist, st))) return rc;
    k_median_finish<<<1, 1, 0, st>>>(s_lo, s_hi, even, med_dev);
    MM_CHECK_LAUNCH();
    if (out) {
        k_divide<<<grid_for(n), 256, 0, st>>>(x, n, med_dev, out);
        MM_CHECK_LAUNCH();
    }
    return MM_OK;
}
