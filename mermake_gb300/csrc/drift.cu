// Drift alignment of maxima point sets (restating mermake/align.py:12-129 and
// mermake/utils.py:10-36).
//
// Aligner(X_ref, resc, trim, th): rows whose last column exceeds th are kept
// (align.py:121-129), the first three columns are the points.  The reference
// image is the set of voxels round(X/resc) after trimming `trim` voxels from
// the x and y extremes (align.py:37-59); get_best_translation_points splats the
// moving set the same way, takes the argmax of the full linear correlation of
// the two 0/1 images (utils.fftconvolve, align.py:107-111), and refines it with
// five nearest-neighbour rounds at radii linspace(resc, target, 5)
// (align.py:61-77).
//
// The correlation of two 0/1 images at shift s is the number of voxel pairs
// (i in moving, j in reference) with i - j = s, so it is computed exactly by
// counting pair differences, a row of shifts at a time in shared memory,
// instead of an FFT (whose float result rounds to the same integers); the argmax
// takes the first maximal index in C order, as argmax does.  Nearest neighbours are brute force in double precision,
// ties to the lowest reference index.
#include <limits.h>
#include <math.h>
#include <string.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "deconv.cuh"

// per-aligner scratch for the moving sets, grown on demand
struct MmDriftWork {
    float *pts = nullptr;
    int *iv = nullptr, *keep = nullptr, *small = nullptr;
    int *xs = nullptr, *ys = nullptr;  // x and y of the unique voxels, row (z, x) by row
    size_t cap = 0;
    unsigned char *grid = nullptr;
    size_t grid_bytes = 0;
    int *rows = nullptr;      // first voxel of each row, and their number at the end
    size_t rows_cap = 0;
    int *h_small = nullptr;
};

// Uniform cell grid of the reference points for the nearest-neighbour
// refinement: cells of edge cs >= the largest match radius, so every point
// within the radius of a query lies in the query's cell or its neighbours.
struct MmCellGrid {
    int dims[3] = {0, 0, 0};
    float lo[3] = {0, 0, 0};
    float cs = 0;
    int *start = nullptr;     // device, cells + 1: first sorted point of each cell
    float *pts = nullptr;     // device, n x 3: points sorted by cell (index order within a cell)
    int *idx = nullptr;       // device, n: original index of each sorted point
    double *state = nullptr;  // device, two slots: shift (3), integer-shift flag, matched count
    double *parts = nullptr;  // device, two slots: per-block partial sums of a refinement round
};

struct mm_aligner {
    int n;            // reference points kept by the threshold
    float *pts;       // device, n x 3
    int nvox;         // unique reference voxels
    int *rows;        // device, shape[0] x shape[1] + 1: first voxel of each (z, x) row
    int *ys;          // device, nvox: the voxels' y
    int shape[3];     // reference image shape
    int resc, trim;
    float th;         // NaN: no threshold
    MmDriftWork w;
    MmCellGrid cg;
};

namespace {

// stable compaction of the rows whose last column exceeds th (all rows when th is NaN)
__global__ void k_compact_rows(const float *__restrict__ X, int n, int cols, long long ld, float th,
                               float *__restrict__ out, int *__restrict__ nout) {
    __shared__ int warp_tot[32];
    __shared__ int base;
    if (threadIdx.x == 0) base = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int r0 = 0; r0 < n; r0 += blockDim.x) {
        const int r = r0 + threadIdx.x;
        bool keep = false;
        if (r < n) {
            const float last = X[r * ld + cols - 1];
            keep = isnan(th) ? true : (last > th);
        }
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        if (lane == 0) warp_tot[warp] = __popc(m);
        __syncthreads();
        int before = 0;
        for (int w = 0; w < warp; ++w) before += warp_tot[w];
        const int pos = base + before + __popc(m & ((1u << lane) - 1));
        if (keep)
            for (int c = 0; c < 3; ++c) out[pos * 3 + c] = X[r * ld + c];
        __syncthreads();
        if (threadIdx.x == 0) {
            int t = 0;
            for (int w = 0; w < nw; ++w) t += warp_tot[w];
            base += t;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) *nout = base;
}

// round(X / resc) half to even (np.round of a float32 quotient), min/max per axis
__global__ void k_round_minmax(const float *__restrict__ pts, const int *__restrict__ n_p, int resc,
                               int *__restrict__ iv, int *__restrict__ mm) {
    const int n = *n_p;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        for (int c = 0; c < 3; ++c) {
            const int v = (int)rintf(__fdiv_rn(pts[i * 3 + c], (float)resc));
            iv[i * 3 + c] = v;
            atomicMin(&mm[c], v);
            atomicMax(&mm[3 + c], v);
        }
}

// keep = all(Xm + n <= X <= XM - n) with n = (0, trim, trim); max over kept
__global__ void k_trim_max(const int *__restrict__ iv, const int *__restrict__ n_p, const int *__restrict__ mm,
                           int trim, int *__restrict__ keep, int *__restrict__ kmax) {
    const int n = *n_p;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        bool k = true;
        for (int c = 0; c < 3; ++c) {
            const int t = c == 0 ? 0 : trim;
            const int v = iv[i * 3 + c];
            k = k && v <= mm[3 + c] - t && v >= mm[c] + t;
        }
        keep[i] = k;
        if (k)
            for (int c = 0; c < 3; ++c) atomicMax(&kmax[c], iv[i * 3 + c]);
    }
}

// imf[tuple(X.T)] = 1: mark the voxels (negative indices wrap, as NumPy's do)
__global__ void k_mark(const int *__restrict__ iv, const int *__restrict__ keep, const int *__restrict__ n_p,
                       const int *__restrict__ shape, unsigned char *__restrict__ grid) {
    const int n = *n_p;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        if (!keep[i]) continue;
        long long lin = 0;
        bool ok = true;
        for (int c = 0; c < 3; ++c) {
            int v = iv[i * 3 + c];
            if (v < 0) v += shape[c];
            ok = ok && v >= 0 && v < shape[c];
            lin = lin * shape[c] + v;
        }
        if (ok) grid[lin] = 1;
    }
}

// The unique voxels of the grid as rows (z, x): a warp counts a row's, one CTA
// turns the counts into starts (rows[nrows] the total), a warp lists its voxels.
__global__ void k_row_count(const unsigned char *__restrict__ grid, int nrows, int s2, int *__restrict__ rows) {
    const int lane = threadIdx.x & 31;
    for (int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < nrows; r += (gridDim.x * blockDim.x) >> 5) {
        int c = 0;
        for (int y = lane; y < s2; y += 32) c += grid[(long long)r * s2 + y];
        c = __reduce_add_sync(0xffffffffu, c);
        if (lane == 0) rows[r] = c;
    }
}
__global__ void __launch_bounds__(1024) k_row_scan(int *__restrict__ rows, int nrows) {
    __shared__ int part[32];
    __shared__ int base;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) base = 0;
    for (int r0 = 0; r0 < nrows; r0 += 1024) {
        const int r = r0 + threadIdx.x, c = r < nrows ? rows[r] : 0;
        int v = c;
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += t;
        }
        if (lane == 31) part[warp] = v;
        __syncthreads();
        if (warp == 0) {
            int p = part[lane];
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, p, o);
                if (lane >= o) p += t;
            }
            part[lane] = p;
        }
        __syncthreads();
        const int before = base + (warp ? part[warp - 1] : 0) + v - c;
        if (r < nrows) rows[r] = before;
        __syncthreads();
        if (threadIdx.x == 1023) base = before + c;
        __syncthreads();
    }
    if (threadIdx.x == 0) rows[nrows] = base;
}
__global__ void k_row_fill(const unsigned char *__restrict__ grid, int nrows, int s1, int s2,
                           const int *__restrict__ rows, int *__restrict__ xs, int *__restrict__ ys) {
    const int lane = threadIdx.x & 31;
    for (int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < nrows; r += (gridDim.x * blockDim.x) >> 5) {
        int at = rows[r];
        if (at == rows[r + 1]) continue;
        for (int y0 = 0; y0 < s2; y0 += 32) {
            const bool on = y0 + lane < s2 && grid[(long long)r * s2 + y0 + lane];
            const unsigned m = __ballot_sync(0xffffffffu, on);
            if (on) {
                const int v = at + __popc(m & ((1u << lane) - 1));
                xs[v] = r % s1;
                ys[v] = y0 + lane;
            }
            at += __popc(m);
        }
    }
}

// The correlation peak: a CTA takes a row (z, x) of shifts, i.e. the pairs of
// rows (az, ax) of the moving and (az - dz, ax - dx) of the reference voxels,
// counts their y differences in shared memory (kCorrSeg shifts at a time), and
// offers its first largest count, as (count << 32 | ~index).  Counting in one
// histogram of all shifts in global memory took 141 us for 6000 x 6000 voxels
// (36 M additions in L2), clearing and searching it 40 us more.
constexpr int kCorrThreads = 64, kCorrSeg = 1024;
struct CorrShape {
    int a[2], b[2];  // rows of the two sets: (z, x) extents
    int o1, o2;      // extents of the shifts along x and y
    int c2;          // y shift of index 0 (negated)
    long long nout;  // rows of shifts
};
__global__ void __launch_bounds__(kCorrThreads)
k_corr_rows(const int *__restrict__ ra, const int *__restrict__ xa, const int *__restrict__ ya,
            const int *__restrict__ rb, const int *__restrict__ yb, CorrShape s, unsigned long long *__restrict__ best) {
    __shared__ int hist[kCorrSeg];
    unsigned long long mine = 0;
    for (long long out = blockIdx.x; out < s.nout; out += gridDim.x) {
        const int oz = (int)(out / s.o1), ox = (int)(out - (long long)oz * s.o1);
        const int dz = oz - (s.b[0] - 1), dx = ox - (s.b[1] - 1);
        const int z0 = max(0, dz), z1 = min(s.a[0], s.b[0] + dz), x0 = max(0, dx), x1 = min(s.a[1], s.b[1] + dx);
        for (int y0 = 0; y0 < s.o2; y0 += kCorrSeg) {
            const int ny = min(kCorrSeg, s.o2 - y0);
            for (int y = threadIdx.x; y < ny; y += kCorrThreads) hist[y] = 0;
            __syncthreads();
            // the moving voxels of rows (z, x0 .. x1) are consecutive: a thread
            // each, against the voxels of its reference row
            if (ra && x0 < x1)
                for (int z = z0; z < z1; ++z) {
                    const int p1 = ra[z * s.a[1] + x1], jrow = (z - dz) * s.b[1] - dx;
                    for (int p = ra[z * s.a[1] + x0] + threadIdx.x; p < p1; p += kCorrThreads) {
                        const int j = jrow + xa[p], q1 = rb[j + 1], y = ya[p] + s.c2 - y0;
                        for (int q = rb[j]; q < q1; ++q) {
                            const int d = y - yb[q];
                            if ((unsigned)d < (unsigned)ny) atomicAdd(&hist[d], 1);
                        }
                    }
                }
            __syncthreads();
            const long long at = out * s.o2 + y0;
            for (int y = threadIdx.x; y < ny; y += kCorrThreads) {
                const unsigned long long key = ((unsigned long long)(unsigned)hist[y] << 32) | (unsigned)~(unsigned)(at + y);
                mine = key > mine ? key : mine;
            }
            __syncthreads();
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long t = __shfl_xor_sync(0xffffffffu, mine, o);
        mine = t > mine ? t : mine;
    }
    if ((threadIdx.x & 31) == 0) atomicMax(best, mine);
}

// Nearest-neighbour refinement (align.py:55-76, five rounds with radii
// np.linspace(resc, target, 5)), one round per launch over many CTAs.  Each
// moving point X - shift looks for its nearest reference point among the
// cells that its match radius reaches (distance in double, ties to the lower
// reference index: the point a brute-force search over all references would
// pick); if it lies within the round's radius, X - R (float32) is added in
// double.  Eight lanes share a point's rows of cells, since a search is a chain
// of dependent loads, and the cells are found in float, the reach widened by
// more than its rounding, since this part does two double products per SM and
// cycle (a thread per point with double quotients: 22 us a round for 6000
// points).  Blocks write partial sums, which every block of the next round adds
// in the same order into its shift; the shift of round r and its sums are in
// slot r & 1, so that no block of a round writes what another reads.
constexpr int kRefineThreads = 256;
constexpr int kRefineMaxBlocks = 304;
constexpr int kRefineLanes = 8;
constexpr int kState = 8;  // doubles of a slot: shift (3), integer-shift flag, matched count

__global__ void k_refine_init(const unsigned long long *__restrict__ best, int o1, int o2, int sb0, int sb1,
                              int sb2, int resc, double *__restrict__ state) {
    const unsigned long long b = *best;
    const long long idx = (long long)(~(unsigned)(b & 0xffffffffu));
    const long long z = idx / ((long long)o1 * o2), x = (idx / o2) % o1, y = idx % o2;
    state[0] = (double)((z - sb0 + 1) * resc);
    state[1] = (double)((x - sb1 + 1) * resc);
    state[2] = (double)((y - sb2 + 1) * resc);
    state[3] = 1.0;  // the shift is still the integer coarse one
    state[4] = 0.0;
}

// the state after a round: its predecessor `prev` and the blocks' sums, added by
// one warp in a fixed order (s is shared memory of kState doubles; ends with a
// barrier)
__device__ __forceinline__ void refine_state(const double *__restrict__ prev, const double *__restrict__ parts, int nblocks,
                                             double *s) {
    if (threadIdx.x < 32) {
        const int k = threadIdx.x & 3;
        double t = 0;
        for (int b0 = threadIdx.x >> 2; b0 < nblocks; b0 += 64) {
            double v[8];  // loads first: the additions wait for them once
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = b0 + 8 * u < nblocks ? parts[(b0 + 8 * u) * 4 + k] : 0.0;
#pragma unroll
            for (int u = 0; u < 8; ++u) t += v[u];
        }
        for (int o = 4; o < 32; o <<= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        const double cnt = __shfl_sync(0xffffffffu, t, 3);
        // no point kept: the shift stays (align.py:72-74)
        if (threadIdx.x < 3) s[k] = cnt > 0 ? (double)(float)(t / cnt) : prev[k];
        if (threadIdx.x == 3) {
            s[3] = cnt > 0 ? 0.0 : prev[3];
            s[4] = cnt;
        }
    }
    __syncthreads();
}

__global__ void __launch_bounds__(kRefineThreads)
k_refine_round(const float *__restrict__ X, const int *__restrict__ n_p, const float *__restrict__ gp,
               const int *__restrict__ gidx, const int *__restrict__ gstart, int gd0, int gd1, int gd2, float lo0,
               float lo1, float lo2, float cs, double dist_th, int round, double *__restrict__ states,
               double *__restrict__ parts_all) {
    __shared__ double st[kState], wsum[kRefineThreads / 32][4];
    double *parts = parts_all + (round & 1) * 4 * kRefineMaxBlocks;
    if (round == 0) {
        if (threadIdx.x < 4) st[threadIdx.x] = states[threadIdx.x];
        __syncthreads();
    } else {
        refine_state(states + ((round - 1) & 1) * kState, parts_all + ((round - 1) & 1) * 4 * kRefineMaxBlocks, gridDim.x,
                     st);
        if (blockIdx.x == 0 && threadIdx.x < 5) states[(round & 1) * kState + threadIdx.x] = st[threadIdx.x];
    }
    const int n = *n_p;
    const bool tint = st[3] != 0.0;
    const double tz0 = st[0], tz1 = st[1], tz2 = st[2];
    const float t0 = (float)tz0, t1 = (float)tz1, t2 = (float)tz2;
    const float radius = (float)dist_th, inv = 1.f / cs;
    double sum[4] = {0, 0, 0, 0};
    const int sub = threadIdx.x % kRefineLanes;
    const int pb = kRefineThreads / kRefineLanes;  // points of a block at a time
    for (int i0 = blockIdx.x * pb; i0 < n; i0 += gridDim.x * pb) {
        const int i = i0 + threadIdx.x / kRefineLanes;
        double bd = 1e300;
        int bj = 0x7fffffff, bk = -1;
        if (i < n) {
            const float x0 = X[i * 3], x1 = X[i * 3 + 1], x2 = X[i * 3 + 2];
            // the cells within the radius along an axis: the reach is widened
            // by 1e-5 of the coordinates and 0.01, over 40 float roundings each
            int c[3][2];
            auto cells = [&](float x, float t, float lo, int gd, int (&r)[2]) {
                const float w = radius + 0.01f + 1e-5f * (fabsf(x) + fabsf(t) + fabsf(lo)), q = x - t - lo;
                r[0] = max(0, (int)floorf(fminf(fmaxf((q - w) * inv - 0.01f, -1.f), 2e9f)));
                r[1] = min(gd - 1, (int)floorf(fminf(fmaxf((q + w) * inv + 0.01f, -1.f), 2e9f)));
            };
            cells(x0, t0, lo0, gd0, c[0]);
            cells(x1, t1, lo1, gd1, c[1]);
            cells(x2, t2, lo2, gd2, c[2]);
            const int nb = c[1][1] - c[1][0] + 1;
            if (c[0][0] <= c[0][1] && nb > 0 && c[2][0] <= c[2][1])
                for (int r = sub; r < (c[0][1] - c[0][0] + 1) * nb; r += kRefineLanes) {
                    const long long row = ((long long)(c[0][0] + r / nb) * gd1 + c[1][0] + r % nb) * gd2;
                    const int e0 = gstart[row + c[2][0]], e1 = gstart[row + c[2][1] + 1];
                    for (int k = e0; k < e1; ++k) {
                        // XT = X - tzxy: float64 against the integer coarse
                        // shift, float32 after
                        const double q0 = tint ? (double)x0 - tz0 : (double)(x0 - t0);
                        const double q1 = tint ? (double)x1 - tz1 : (double)(x1 - t1);
                        const double q2 = tint ? (double)x2 - tz2 : (double)(x2 - t2);
                        const double d0 = q0 - gp[k * 3], d1 = q1 - gp[k * 3 + 1], d2 = q2 - gp[k * 3 + 2];
                        const double d = d0 * d0 + d1 * d1 + d2 * d2;
                        const int j = gidx[k];
                        if (d < bd || (d == bd && j < bj)) {
                            bd = d;
                            bj = j;
                            bk = k;
                        }
                    }
                }
        }
        for (int o = kRefineLanes / 2; o > 0; o >>= 1) {
            const double d = __shfl_xor_sync(0xffffffffu, bd, o);
            const int j = __shfl_xor_sync(0xffffffffu, bj, o), k = __shfl_xor_sync(0xffffffffu, bk, o);
            if (d < bd || (d == bd && j < bj)) {
                bd = d;
                bj = j;
                bk = k;
            }
        }
        if (sub == 0 && bk >= 0 && sqrt(bd) < dist_th) {
            // X_ - X_ref_ in float32, summed in double
            sum[0] += (double)(X[i * 3] - gp[bk * 3]);
            sum[1] += (double)(X[i * 3 + 1] - gp[bk * 3 + 1]);
            sum[2] += (double)(X[i * 3 + 2] - gp[bk * 3 + 2]);
            sum[3] += 1;
        }
    }
    // lanes 0, 8, 16 and 24 hold a warp's sums
    for (int k = 0; k < 4; ++k) {
        for (int o = kRefineLanes; o < 32; o <<= 1) sum[k] += __shfl_xor_sync(0xffffffffu, sum[k], o);
        if ((threadIdx.x & 31) == 0) wsum[threadIdx.x >> 5][k] = sum[k];
    }
    __syncthreads();
    if (threadIdx.x < 4) {
        double t = 0;
        for (int w = 0; w < kRefineThreads / 32; ++w) t += wsum[w][threadIdx.x];
        parts[blockIdx.x * 4 + threadIdx.x] = t;
    }
}

// the shift after the last round (index `round`), the matched count and the flag
__global__ void k_refine_last(const double *__restrict__ states, const double *__restrict__ parts_all, int nblocks, int round,
                              float *__restrict__ out, int *__restrict__ npts) {
    __shared__ double st[kState];
    refine_state(states + (round & 1) * kState, parts_all + (round & 1) * 4 * kRefineMaxBlocks, nblocks, st);
    if (threadIdx.x == 0) {
        for (int k = 0; k < 3; ++k) out[k] = (float)st[k];
        npts[0] = (int)st[4];
        npts[1] = (int)st[3];
    }
}

struct Splat {
    int shape[3];
    bool any;  // voxels survive the trim
};

// splat of a point set: its unique voxels as rows in w.rows, w.xs and w.ys, their extents on the host
int splat(MmDriftWork &w, const int *n_dev, int n_host, int resc, int trim, int *mm, int *kmax, Splat *out,
          cudaStream_t st) {
    const float *pts_dev = w.pts;
    int *iv = w.iv, *keep = w.keep, *h_small = w.h_small;
    const int init[9] = {INT_MAX, INT_MAX, INT_MAX, INT_MIN, INT_MIN, INT_MIN, INT_MIN, INT_MIN, INT_MIN};
    MM_CUDA_TRY(cudaMemcpyAsync(mm, init, sizeof(int) * 6, cudaMemcpyHostToDevice, st));
    MM_CUDA_TRY(cudaMemcpyAsync(kmax, init + 6, sizeof(int) * 3, cudaMemcpyHostToDevice, st));
    const int g = n_host > 0 ? mm_cdiv(n_host, 256) : 1;
    k_round_minmax<<<g, 256, 0, st>>>(pts_dev, n_dev, resc, iv, mm);
    MM_CHECK_LAUNCH();
    k_trim_max<<<g, 256, 0, st>>>(iv, n_dev, mm, trim, keep, kmax);
    MM_CHECK_LAUNCH();
    MM_CUDA_TRY(cudaMemcpyAsync(h_small, kmax, sizeof(int) * 3, cudaMemcpyDeviceToHost, st));
    MM_CUDA_TRY(cudaStreamSynchronize(st));
    if (h_small[0] == INT_MIN) {  // nothing survives the trim: a (1,1,1) zero image (align.py:51-53)
        out->shape[0] = out->shape[1] = out->shape[2] = 1;
        out->any = false;
        return MM_OK;
    }
    for (int c = 0; c < 3; ++c) out->shape[c] = h_small[c] + 1;
    MM_REQUIRE(out->shape[0] > 0 && out->shape[1] > 0 && out->shape[2] > 0, "negative splat extent");
    const size_t total = (size_t)out->shape[0] * out->shape[1] * out->shape[2];
    if (w.grid_bytes < total) {
        if (w.grid) cudaFree(w.grid);
        w.grid = nullptr;
        w.grid_bytes = 0;
        MM_CUDA_TRY(cudaMalloc(&w.grid, total));
        w.grid_bytes = total;
    }
    MM_REQUIRE((long long)out->shape[0] * out->shape[1] < (1LL << 31) - 64, "splat image of too many rows");
    const int nrows = out->shape[0] * out->shape[1];
    if (w.rows_cap < (size_t)nrows + 1) {
        cudaFree(w.rows);
        w.rows = nullptr;
        w.rows_cap = 0;
        MM_CUDA_TRY(cudaMalloc(&w.rows, sizeof(int) * ((size_t)nrows + 1)));
        w.rows_cap = (size_t)nrows + 1;
    }
    MM_CUDA_TRY(cudaMemsetAsync(w.grid, 0, total, st));
    MM_CUDA_TRY(cudaMemcpyAsync(mm, out->shape, sizeof(int) * 3, cudaMemcpyHostToDevice, st));
    k_mark<<<g, 256, 0, st>>>(iv, keep, n_dev, mm, w.grid);
    MM_CHECK_LAUNCH();
    const int gr = nrows / 8 + 1 < 152 * 8 ? nrows / 8 + 1 : 152 * 8;
    k_row_count<<<gr, 256, 0, st>>>(w.grid, nrows, out->shape[2], w.rows);
    MM_CHECK_LAUNCH();
    k_row_scan<<<1, 1024, 0, st>>>(w.rows, nrows);
    MM_CHECK_LAUNCH();
    k_row_fill<<<gr, 256, 0, st>>>(w.grid, nrows, out->shape[1], out->shape[2], w.rows, w.xs, w.ys);
    MM_CHECK_LAUNCH();
    out->any = true;
    return MM_OK;
}

int work_reserve(MmDriftWork &w, size_t n) {
    if (!w.h_small) MM_CUDA_TRY(cudaMallocHost(&w.h_small, 64 * sizeof(int)));
    if (!w.small) MM_CUDA_TRY(cudaMalloc(&w.small, 64 * sizeof(int)));
    if (n < 16) n = 16;
    if (w.cap >= n) return MM_OK;
    cudaFree(w.pts);
    cudaFree(w.iv);
    cudaFree(w.keep);
    cudaFree(w.xs);
    cudaFree(w.ys);
    w.pts = nullptr; w.iv = w.keep = w.xs = w.ys = nullptr;
    w.cap = 0;
    MM_CUDA_TRY(cudaMalloc(&w.pts, n * 3 * sizeof(float)));
    MM_CUDA_TRY(cudaMalloc(&w.iv, n * 3 * sizeof(int)));
    MM_CUDA_TRY(cudaMalloc(&w.keep, n * sizeof(int)));
    MM_CUDA_TRY(cudaMalloc(&w.xs, n * sizeof(int)));
    MM_CUDA_TRY(cudaMalloc(&w.ys, n * sizeof(int)));
    w.cap = n;
    return MM_OK;
}

void work_free(MmDriftWork &w) {
    cudaFree(w.pts); cudaFree(w.iv); cudaFree(w.keep); cudaFree(w.xs); cudaFree(w.ys); cudaFree(w.small);
    cudaFree(w.grid); cudaFree(w.rows);
    if (w.h_small) cudaFreeHost(w.h_small);
    w = MmDriftWork();
}

// small-buffer slots (ints) inside Work::small
enum { SM_N = 0, SM_MM = 1, SM_KMAX = 8, SM_NPTS = 14, SM_BEST = 16, SM_OUT = 20 };

// The cell grid of the reference points (host-side counting sort, points in
// index order within a cell), and the refinement's small device state.
int cell_grid_build(MmCellGrid &g, const float *pts_dev, int n, float cs_min, cudaStream_t st) {
    std::vector<float> p((size_t)n * 3);
    MM_CUDA_TRY(cudaMemcpyAsync(p.data(), pts_dev, sizeof(float) * 3 * n, cudaMemcpyDeviceToHost, st));
    MM_CUDA_TRY(cudaStreamSynchronize(st));
    float lo[3], hi[3];
    for (int c = 0; c < 3; ++c) lo[c] = hi[c] = p[c];
    for (int i = 0; i < n; ++i)
        for (int c = 0; c < 3; ++c) {
            lo[c] = std::min(lo[c], p[i * 3 + c]);
            hi[c] = std::max(hi[c], p[i * 3 + c]);
        }
    // cells of edge >= cs_min, coarser if the box would need more than 2^24 cells
    double cs = cs_min;
    for (;;) {
        double cells = 1;
        for (int c = 0; c < 3; ++c) cells *= std::floor((hi[c] - lo[c]) / cs) + 1;
        if (cells <= (double)(1 << 24)) break;
        cs *= 1.5;
    }
    g.cs = (float)cs;
    for (int c = 0; c < 3; ++c) {
        g.lo[c] = lo[c];
        g.dims[c] = (int)std::floor((hi[c] - lo[c]) / g.cs) + 1;
    }
    const long long ncell = (long long)g.dims[0] * g.dims[1] * g.dims[2];
    std::vector<int> cell(n), start(ncell + 1, 0), idx(n);
    for (int i = 0; i < n; ++i) {
        int k[3];
        for (int c = 0; c < 3; ++c)
            k[c] = std::min(g.dims[c] - 1, std::max(0, (int)std::floor(((double)p[i * 3 + c] - g.lo[c]) / g.cs)));
        cell[i] = (int)(((long long)k[0] * g.dims[1] + k[1]) * g.dims[2] + k[2]);
        start[cell[i] + 1]++;
    }
    for (long long c = 0; c < ncell; ++c) start[c + 1] += start[c];
    std::vector<int> fill(start.begin(), start.end() - 1);
    std::vector<float> sp((size_t)n * 3);
    for (int i = 0; i < n; ++i) {
        const int at = fill[cell[i]]++;
        idx[at] = i;
        for (int c = 0; c < 3; ++c) sp[at * 3 + c] = p[i * 3 + c];
    }
    MM_CUDA_TRY(cudaMalloc(&g.start, sizeof(int) * (ncell + 1)));
    MM_CUDA_TRY(cudaMalloc(&g.pts, sizeof(float) * 3 * n));
    MM_CUDA_TRY(cudaMalloc(&g.idx, sizeof(int) * n));
    MM_CUDA_TRY(cudaMalloc(&g.state, sizeof(double) * 2 * kState));
    MM_CUDA_TRY(cudaMalloc(&g.parts, sizeof(double) * 2 * 4 * kRefineMaxBlocks));
    MM_CUDA_TRY(cudaMemcpyAsync(g.start, start.data(), sizeof(int) * (ncell + 1), cudaMemcpyHostToDevice, st));
    MM_CUDA_TRY(cudaMemcpyAsync(g.pts, sp.data(), sizeof(float) * 3 * n, cudaMemcpyHostToDevice, st));
    MM_CUDA_TRY(cudaMemcpyAsync(g.idx, idx.data(), sizeof(int) * n, cudaMemcpyHostToDevice, st));
    MM_CUDA_TRY(cudaStreamSynchronize(st));
    return MM_OK;
}

void cell_grid_free(MmCellGrid &g) {
    cudaFree(g.start); cudaFree(g.pts); cudaFree(g.idx); cudaFree(g.state); cudaFree(g.parts);
    g = MmCellGrid();
}

}  // namespace

extern "C" int mm_aligner_create(const float *X_ref, int n, int cols, int64_t ld, float th, int resc, int trim,
                                 mm_aligner **out, void *stream) {
    MM_REQUIRE(out && (X_ref || n == 0), "null argument");
    MM_REQUIRE(n >= 0 && cols >= 3 && ld >= cols, "point rows need at least 3 columns");
    MM_REQUIRE(resc >= 1 && trim >= 0, "resc must be >= 1 and trim >= 0");
    cudaStream_t st = (cudaStream_t)stream;
    mm_aligner *S = new mm_aligner();
    S->pts = nullptr;
    S->rows = S->ys = nullptr;
    S->resc = resc;
    S->trim = trim;
    S->th = th;
    MmDriftWork &w = S->w;
    int rc = work_reserve(w, (size_t)n);
    if (rc) { work_free(w); delete S; return rc; }
    int nkeep = 0;
    if (n > 0) {
        k_compact_rows<<<1, 1024, 0, st>>>(X_ref, n, cols, ld, th, w.pts, w.small + SM_N);
        if (cudaGetLastError() != cudaSuccess || cudaMemcpyAsync(w.h_small, w.small + SM_N, sizeof(int),
                                                                 cudaMemcpyDeviceToHost, st) != cudaSuccess ||
            cudaStreamSynchronize(st) != cudaSuccess) {
            work_free(w); delete S;
            mm_set_error("aligner: compaction failed");
            return MM_EDEVICE;
        }
        mm_launch_counter_add();
        nkeep = w.h_small[0];
    }
    if (nkeep == 0) {
        work_free(w); delete S;
        mm_set_error("No points left after thresholding; cannot build KDTree. Check your data and/or threshold value.");
        return MM_EINVAL;
    }
    S->n = nkeep;
    Splat sp;
    rc = splat(w, w.small + SM_N, nkeep, resc, trim, w.small + SM_MM, w.small + SM_KMAX, &sp, st);
    if (rc) { work_free(w); delete S; return rc; }
    for (int c = 0; c < 3; ++c) S->shape[c] = sp.shape[c];
    const size_t nrows = (size_t)sp.shape[0] * sp.shape[1];
    w.h_small[0] = 0;
    if (sp.any && (cudaMemcpyAsync(w.h_small, w.rows + nrows, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
                   cudaStreamSynchronize(st) != cudaSuccess)) {
        work_free(w); delete S;
        mm_set_error("aligner: splat failed");
        return MM_EDEVICE;
    }
    S->nvox = w.h_small[0];
    // keep the reference points and voxel rows in buffers of their own
    S->pts = nullptr;
    if (cudaMalloc(&S->pts, sizeof(float) * 3 * nkeep) != cudaSuccess ||
        cudaMalloc(&S->rows, sizeof(int) * (nrows + 1)) != cudaSuccess ||
        cudaMalloc(&S->ys, sizeof(int) * (S->nvox > 0 ? S->nvox : 1)) != cudaSuccess) {
        cudaGetLastError();
        cudaFree(S->pts); cudaFree(S->rows); cudaFree(S->ys); work_free(w); delete S;
        mm_set_error("aligner: out of device memory");
        return MM_ENOMEM;
    }
    cudaMemcpyAsync(S->pts, w.pts, sizeof(float) * 3 * nkeep, cudaMemcpyDeviceToDevice, st);
    if (S->nvox) {
        cudaMemcpyAsync(S->rows, w.rows, sizeof(int) * (nrows + 1), cudaMemcpyDeviceToDevice, st);
        cudaMemcpyAsync(S->ys, w.ys, sizeof(int) * S->nvox, cudaMemcpyDeviceToDevice, st);
    }
    MM_CUDA_TRY(cudaStreamSynchronize(st));
    if ((rc = cell_grid_build(S->cg, S->pts, nkeep, (float)resc, st))) {
        cell_grid_free(S->cg); cudaFree(S->pts); cudaFree(S->rows); cudaFree(S->ys); work_free(w); delete S;
        return rc;
    }
    *out = S;
    return MM_OK;
}

extern "C" int mm_aligner_destroy(mm_aligner *S) {
    if (!S) return MM_OK;
    cudaDeviceSynchronize();
    cudaFree(S->pts);
    cudaFree(S->rows);
    cudaFree(S->ys);
    work_free(S->w);
    cell_grid_free(S->cg);
    delete S;
    return MM_OK;
}

extern "C" int mm_aligner_info(const mm_aligner *S, int *n_points, int *n_voxels, int *shape3) {
    MM_REQUIRE(S, "null aligner");
    if (n_points) *n_points = S->n;
    if (n_voxels) *n_voxels = S->nvox;
    if (shape3)
        for (int c = 0; c < 3; ++c) shape3[c] = S->shape[c];
    return MM_OK;
}

extern "C" int mm_aligner_translation(mm_aligner *S, const float *X, int n, int cols, int64_t ld, float target,
                                      float *tzxy, int *npts, void *stream) {
    MM_REQUIRE(S && tzxy && npts && (X || n == 0), "null argument");
    MM_REQUIRE(n >= 0 && cols >= 3 && ld >= cols, "point rows need at least 3 columns");
    const mm_aligner &A = *S;
    MmDriftWork &w = S->w;
    cudaStream_t st = (cudaStream_t)stream;
    int rc = work_reserve(w, (size_t)n);
    if (rc) return rc;
    // get_best_translation_points: threshold on the last column (align.py:97-101)
    int nm = 0;
    if (n > 0) {
        k_compact_rows<<<1, 1024, 0, st>>>(X, n, cols, ld, A.th, w.pts, w.small + SM_N);
        MM_CHECK_LAUNCH();
        MM_CUDA_TRY(cudaMemcpyAsync(w.h_small, w.small + SM_N, sizeof(int), cudaMemcpyDeviceToHost, st));
        MM_CUDA_TRY(cudaStreamSynchronize(st));
        nm = w.h_small[0];
    } else {
        MM_CUDA_TRY(cudaMemsetAsync(w.small + SM_N, 0, sizeof(int), st));
    }
    Splat sp = {{1, 1, 1}, false};
    if (nm > 0) {
        rc = splat(w, w.small + SM_N, nm, A.resc, A.trim, w.small + SM_MM, w.small + SM_KMAX, &sp, st);
        if (rc) return rc;
    }
    // full correlation shape sa + sb - 1
    const int o0 = sp.shape[0] + A.shape[0] - 1, o1 = sp.shape[1] + A.shape[1] - 1, o2 = sp.shape[2] + A.shape[2] - 1;
    unsigned long long *best = reinterpret_cast<unsigned long long *>(w.small + SM_BEST);
    MM_CUDA_TRY(cudaMemsetAsync(best, 0, sizeof(unsigned long long), st));
    const CorrShape cs = {{sp.shape[0], sp.shape[1]}, {A.shape[0], A.shape[1]}, o1, o2, A.shape[2] - 1, (long long)o0 * o1};
    const bool pairs = sp.any && A.nvox > 0;  // none: every count is 0, the first shift is the peak
    k_corr_rows<<<(unsigned)std::min(cs.nout, 152LL * 32), kCorrThreads, 0, st>>>(pairs ? w.rows : nullptr, w.xs, w.ys,
                                                                                  A.rows, A.ys, cs, best);
    MM_CHECK_LAUNCH();
    float *outp = reinterpret_cast<float *>(w.small + SM_OUT);
    const MmCellGrid &G = A.cg;
    k_refine_init<<<1, 1, 0, st>>>(best, o1, o2, A.shape[0], A.shape[1], A.shape[2], A.resc, G.state);
    MM_CHECK_LAUNCH();
    int nb = mm_cdiv((long)nm * kRefineLanes, kRefineThreads);
    nb = std::max(1, std::min(nb, kRefineMaxBlocks));
    for (int it = 0; it < 5; ++it) {
        // np.linspace(resc, target, 5)
        const double dist_th = (double)A.resc + (double)it * (((double)target - (double)A.resc) / 4.0);
        k_refine_round<<<nb, kRefineThreads, 0, st>>>(w.pts, w.small + SM_N, G.pts, G.idx, G.start, G.dims[0],
                                                      G.dims[1], G.dims[2], G.lo[0], G.lo[1], G.lo[2], G.cs, dist_th,
                                                      it, G.state, G.parts);
        MM_CHECK_LAUNCH();
    }
    k_refine_last<<<1, 32, 0, st>>>(G.state, G.parts, nb, 4, outp, w.small + SM_NPTS);
    MM_CHECK_LAUNCH();
    MM_CUDA_TRY(cudaMemcpyAsync(w.h_small, outp, sizeof(float) * 3, cudaMemcpyDeviceToHost, st));
    MM_CUDA_TRY(cudaMemcpyAsync(w.h_small + 4, w.small + SM_NPTS, sizeof(int) * 2, cudaMemcpyDeviceToHost, st));
    MM_CUDA_TRY(cudaStreamSynchronize(st));
    memcpy(tzxy, w.h_small, sizeof(float) * 3);
    npts[0] = w.h_small[4];
    return MM_OK;
}
