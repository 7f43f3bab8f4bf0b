// y passes of the tiled deconvolution for padded tiles of 678 and 478 points:
// the prime-factor transform (fft_pfa.cuh) behind the tile gather, and before
// the windowed stores.  (Other lengths: deconv.cu.)
//
// Rows lie along memory and a transform wants 16 of them side by side, so both
// ends go through shared memory: A[e][line], 17 float2 per element, which a
// warp writes and reads along e without bank conflicts (a row is 136 bytes) and
// across the lines contiguously.  The phases' T lies in the same place: a
// thread holds all its values in registers between reading A and writing T, and
// between reading T and writing A, so a CTA of 16 lines takes 100 KB and two
// share an SM.
#include "deconv.cuh"
#include "fft_pfa.cuh"

namespace {

constexpr int kPitch = kPfaNL + 1;     // float2 per element of A
constexpr int kPitchB = kPitch * 8;    // bytes
template <int N>
constexpr size_t line_bytes() {        // rows 0 .. N - 1, and a row of zeros
    return ((size_t)(N + 1) * kPitchB + 15) & ~(size_t)15;
}

// the transform of the CTA's lines: v holds the inputs of (n1, q2), x0 those of
// n2 = 0 (threads with q1 = 0); the outputs are left in A.  Every thread has
// read A when it calls this; ends without a barrier.
template <int N, bool INV>
__device__ __forceinline__ void pfa_lines(const PfaSmem<N> &s, float2 (&v)[PfaK<N>::C][PfaK<N>::N2],
                                          float2 (&x0)[PfaK<N>::C], int q1, int l) {
    using K = PfaK<N>;
    pfa_first<N, INV>(v);
    __syncthreads();  // A has been read: T may take its place
    pfa_put<N>(s, v, q1, l);
    if (q1 == 0) {
        pfa_dft_c<N, INV>(x0);
#pragma unroll
        for (int c = 0; c < K::C; ++c) s.x0[c * kPfaNL + l] = x0[c];
    }
    __syncthreads();
    pfa_middle<N>(s, q1, l);
    __syncthreads();
#pragma unroll
    for (int c = 0; c < K::C; ++c) pfa_last<N>(s, c, q1, l, v[c]);
    __syncthreads();  // T has been read: A again
    unsigned char *A = reinterpret_cast<unsigned char *>(s.T) + l * 8;
    const int4 *op = reinterpret_cast<const int4 *>(s.tout + q1 * K::ipad);
#pragma unroll
    for (int c = 0; c < K::ipad / 4; ++c) {
        const int4 i4 = op[c];
        const int e[4] = {i4.x, i4.y, i4.z, i4.w};
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (4 * c + u < K::vals)
                *reinterpret_cast<float2 *>(A + e[u]) = v[(4 * c + u) / K::N2][(4 * c + u) % K::N2];
    }
    if (q1 == 0) {
#pragma unroll
        for (int c = 0; c < K::C; ++c) *reinterpret_cast<float2 *>(A + s.out0[c]) = s.y0[c * kPfaNL + l];
    }
}

// reads a thread's inputs at the byte offsets of the input table
template <int N>
__device__ __forceinline__ void pfa_take(const PfaSmem<N> &s, float2 (&v)[PfaK<N>::C][PfaK<N>::N2],
                                         float2 (&x0)[PfaK<N>::C], int q1, int l) {
    using K = PfaK<N>;
    const unsigned char *A = reinterpret_cast<const unsigned char *>(s.T) + l * 8;
    const int4 *ip = reinterpret_cast<const int4 *>(s.tin + q1 * K::ipad);
#pragma unroll
    for (int c = 0; c < K::ipad / 4; ++c) {
        const int4 i4 = ip[c];
        const int e[4] = {i4.x, i4.y, i4.z, i4.w};
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (4 * c + u < K::vals)
                v[(4 * c + u) / K::N2][(4 * c + u) % K::N2] = *reinterpret_cast<const float2 *>(A + e[u]);
    }
#pragma unroll
    for (int c = 0; c < K::C; ++c)
        x0[c] = q1 == 0 ? *reinterpret_cast<const float2 *>(A + s.in0[c]) : make_float2(0.f, 0.f);
}

// ---------------------------------------------------------------------------
// forward: the tile's rows through the pad maps, two real rows (planes 2k and
// 2k + 1 of one x) per complex line, x-major.  A line's raw pixels go to A
// once each, divided by the flat (halved: the unpacking of the two spectra
// takes half sums); the y padding is in the input table, which holds the place
// of the pixel that each padded column copies, or the row of zeros.
// ---------------------------------------------------------------------------
// All of a line's loads are issued before the first is used (U words or pixels
// per lane cover the longest row), so a line waits for memory once, and the
// addresses are a lane's base plus constants.
__device__ __forceinline__ float half_over(float f) { return __fdividef(0.5f, f); }

// 0x4B00xxxx is 2^23 + xxxx: the half word `sel` of a and b as floats, exactly
__device__ __forceinline__ float2 two_pixels(unsigned a, unsigned b, unsigned sel) {
    return psub(make_float2(__uint_as_float(__byte_perm(a, 0x4B000000u, sel)),
                            __uint_as_float(__byte_perm(b, 0x4B000000u, sel))),
                make_float2(8388608.f, 8388608.f));
}
template <int N>
__device__ __forceinline__ void stage_rows(const uint16_t *ra, const uint16_t *rb, const float *fr, const float *hf,
                                           int n, float2 *dst, int lane) {
    // words of two pixels of row a, y = 2 w - off and the next, for the words
    // inside the row; row b the same way, or pixel by pixel where it starts on
    // the other half of a word
    constexpr int U = (N / 2 + 1 + 31) / 32;
    const int off = (int)((reinterpret_cast<uintptr_t>(ra) >> 1) & 1);
    const unsigned *wa = reinterpret_cast<const unsigned *>(ra - off) + lane;
    const int y = 2 * lane - off;
    const unsigned first = lane - off, count = (n + off) / 2 - off;  // word u is inside: first + 32 u < count
    unsigned a[U], b[U];
#pragma unroll
    for (int u = 0; u < U; ++u) a[u] = first + 32 * u < count ? wa[32 * u] : 0u;
    if (!rb) {
#pragma unroll
        for (int u = 0; u < U; ++u) b[u] = 0u;
    } else if (!((reinterpret_cast<uintptr_t>(ra) ^ reinterpret_cast<uintptr_t>(rb)) & 2)) {
        const unsigned *wb = reinterpret_cast<const unsigned *>(rb - off) + lane;
#pragma unroll
        for (int u = 0; u < U; ++u) b[u] = first + 32 * u < count ? wb[32 * u] : 0u;
    } else {
        const uint16_t *pb = rb + y;
#pragma unroll
        for (int u = 0; u < U; ++u)
            b[u] = first + 32 * u < count ? pb[64 * u] | (unsigned)pb[64 * u + 1] << 16 : 0u;
    }
    // the two pixels of a word go out in the order that spreads a half warp's
    // 16 stores over all banks: lanes 8 .. 15 of each half start with the second
    const int sw = (lane >> 3) & 1;
    const unsigned p0 = sw ? 0x7632 : 0x7610, p1 = sw ? 0x7610 : 0x7632;
    float2 *d0 = dst + (y + sw) * kPitch, *d1 = dst + (y + 1 - sw) * kPitch;
    if (hf) {
        const float *f0 = hf + y + sw, *f1 = hf + y + 1 - sw;
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (first + 32 * u < count) {
                d0[64 * u * kPitch] = cscale(two_pixels(a[u], b[u], p0), f0[64 * u]);
                d1[64 * u * kPitch] = cscale(two_pixels(a[u], b[u], p1), f1[64 * u]);
            }
    } else if (fr) {
        const float *f0 = fr + y + sw, *f1 = fr + y + 1 - sw;
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (first + 32 * u < count) {
                d0[64 * u * kPitch] = cscale(two_pixels(a[u], b[u], p0), half_over(f0[64 * u]));
                d1[64 * u * kPitch] = cscale(two_pixels(a[u], b[u], p1), half_over(f1[64 * u]));
            }
    } else {
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (first + 32 * u < count) {
                d0[64 * u * kPitch] = pmul(two_pixels(a[u], b[u], p0), 0.5f);
                d1[64 * u * kPitch] = pmul(two_pixels(a[u], b[u], p1), 0.5f);
            }
    }
    // the pixels of words that reach past the row: the first when it is a
    // second half, the last when it is a first half
    if (lane < 2 && (lane ? (n + off) & 1 : off)) {
        const int e = lane ? n - 1 : 0;
        dst[e * kPitch] = pmul(make_float2((float)ra[e], rb ? (float)rb[e] : 0.f), fr ? half_over(fr[e]) : 0.5f);
    }
}
template <int N>
__device__ __forceinline__ void stage_rows(const float *ra, const float *rb, const float *fr, const float *hf,
                                           int n, float2 *dst, int lane) {
    constexpr int U = (N + 31) / 32;
    float a[U], b[U];
    ra += lane;
    dst += lane * kPitch;
#pragma unroll
    for (int u = 0; u < U; ++u) a[u] = lane + 32 * u < n ? ra[32 * u] : 0.f;
    if (rb) {
        rb += lane;
#pragma unroll
        for (int u = 0; u < U; ++u) b[u] = lane + 32 * u < n ? rb[32 * u] : 0.f;
    } else {
#pragma unroll
        for (int u = 0; u < U; ++u) b[u] = 0.f;
    }
    if (hf) {
        hf += lane;
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (lane + 32 * u < n) dst[32 * u * kPitch] = make_float2(a[u] * hf[32 * u], b[u] * hf[32 * u]);
    } else if (fr) {
        fr += lane;
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (lane + 32 * u < n) dst[32 * u * kPitch] = cscale(make_float2(a[u], b[u]), half_over(fr[32 * u]));
    } else {
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (lane + 32 * u < n) dst[32 * u * kPitch] = pmul(make_float2(a[u], b[u]), 0.5f);
    }
}

// rows of `bytes` bytes at p into L2, a lane per 128 bytes
__device__ __forceinline__ void prefetch_row(const void *p, int bytes, int lane) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(p) & ~(uintptr_t)127, e = reinterpret_cast<uintptr_t>(p) + bytes;
    for (uintptr_t c = a + 128 * lane; c < e; c += 128 * 32) asm volatile("prefetch.global.L2 [%0];" ::"l"(c));
}

// What a line of a group is: planes 2k and 2k + 1 of padded row x of a tile
struct FwdLine {
    long long src;  // element offset of the first plane's row; -1: a row of zeros
    int x, k;       // k < 0: no line (past the tile's last)
    int two;        // the second plane exists
    int fx;         // row of the flat field
    int n;          // pixels of a row
};
constexpr int kFlatRows = 2;  // flat rows kept per group (a group of 16 lines spans two x from 29 planes on)

template <typename T, int N>
__global__ void __launch_bounds__(PfaK<N>::threads, 2)
k_rows_fwd_pfa(TileGeom g, const T *__restrict__ img, const float *__restrict__ flat, float2 *__restrict__ S, FftPlan P,
               int zp, int gx, int ngroups, unsigned *__restrict__ queue) {
    using K = PfaK<N>;
    constexpr int H = N / 2 + 1;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int next;
    __shared__ FwdLine lines[2][kPfaNL];
    __shared__ int any[2];  // the group has a line with pixels
    const PfaSmem<N> s = pfa_layout<N>(smem_raw, line_bytes<N>());
    float *hflat = reinterpret_cast<float *>(smem_raw + line_bytes<N>() + pfa_tail_bytes<N>());  // kFlatRows x N
    float2 *A = s.T;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    constexpr int nw = K::threads / 32;
    const int l = tid % kPfaNL, q1 = tid / kPfaNL;
    const int LT = N * zp;  // lines of a tile
    // line i of group grp (a thread each)
    auto describe = [&](int grp, int i) {
        FwdLine f;
        const int by = grp / gx, L = (grp - by * gx) * kPfaNL + i;
        const TileDesc d = mm_tile_desc(g, g.t0 + by);
        f.x = L / zp;
        f.k = L < LT ? L - f.x * zp : -1;
        f.two = 2 * f.k + 1 < g.Z;
        const int sx = mm_map_xy(f.x, d.x == 0, d.xd, N, g.ov);
        f.fx = d.x0 + sx;
        f.n = d.yd;
        f.src = sx >= 0 ? 2 * f.k * g.isz + (long long)f.fx * g.isx + d.y0 : -1;
        return f;
    };
    pfa_load_tables<N, false>(s, P);
    for (int i = tid; i < kPitch; i += K::threads) A[N * kPitch + i] = make_float2(0.f, 0.f);
    __syncthreads();
    for (int i = tid; i < K::N1 * K::ipad; i += K::threads) s.tout[i] *= kPitchB;
    if (tid < 8) s.out0[tid] *= kPitchB;
    // the half reciprocals of the flat rows of a group, once per pixel: the
    // rows of the first line's x and the next, when those are all
    const bool shared_flat = flat && zp >= kPfaNL - 1;
    auto keep_flat = [&](int grp) {
        const int by = grp / gx, x0 = (grp - by * gx) * kPfaNL / zp;
        const TileDesc d = mm_tile_desc(g, g.t0 + by);
        for (int r = 0; r < kFlatRows; ++r) {
            const int sx = x0 + r < N ? mm_map_xy(x0 + r, d.x == 0, d.xd, N, g.ov) : -1;
            if (sx < 0) continue;
            const float *fr = flat + (long long)(d.x0 + sx) * g.fsx + d.y0;
            for (int y = tid; y < d.yd; y += K::threads) hflat[r * N + y] = half_over(fr[y]);
        }
    };
    auto describe_all = [&](int grp, int b) {  // warp 0
        if (tid >= 32) return;
        bool has = false;
        if (tid < kPfaNL) {
            const FwdLine f = describe(grp, tid);
            lines[b][tid] = f;
            has = f.src >= 0 && f.k >= 0;
        }
        has = __any_sync(0xffffffffu, has);
        if (tid == 0) any[b] = has;
    };
    if ((int)blockIdx.x < ngroups) {
        describe_all(blockIdx.x, 0);
        if (shared_flat) keep_flat(blockIdx.x);
    }
    int tile = -1, buf = 0, yd = 0, y0 = 0;
    __syncthreads();
    for (int grp = blockIdx.x; grp < ngroups; buf ^= 1) {
        const int asked = tid == 0 ? queue_ask(queue, grp) : 0;
        const int by = grp / gx;
        if (by != tile) {
            // the input table of this tile: padded column -> staged pixel
            tile = by;
            const TileDesc d = mm_tile_desc(g, g.t0 + by);
            yd = d.yd;
            y0 = d.y0;
            for (int i = tid; i < K::N1 * K::ipad; i += K::threads) {
                const int m = mm_map_xy(P.pfa_idx[i], d.y == 0, d.yd, N, g.ov);
                s.tin[i] = (m < 0 ? N : m) * kPitchB;
            }
            if (tid < K::C) {
                const int m = mm_map_xy(P.pfa_idx[2 * K::N1 * K::ipad + tid], d.y == 0, d.yd, N, g.ov);
                s.in0[tid] = (m < 0 ? N : m) * kPitchB;
            }
        }
        const FwdLine *ln = lines[buf];
        float2 *Sb = S + (long long)by * g.Z * N * H;
        const bool zero = !any[buf];
        if (!zero)
            for (int q = warp; q < kPfaNL; q += nw) {
                const long long src = ln[q].src;
                float2 *dst = A + q;
                if (src >= 0 && ln[q].k >= 0)
                    stage_rows<N>(img + src, ln[q].two ? img + src + g.isz : nullptr,
                                  flat ? flat + ln[q].fx * g.fsx + y0 : nullptr,
                                  shared_flat ? hflat + (ln[q].x - ln[0].x) * N : nullptr, yd, dst, lane);
                else
                    for (int y = lane; y < yd; y += 32) dst[y * kPitch] = make_float2(0.f, 0.f);
            }
        if (tid == 0) next = asked;
        __syncthreads();
        grp = next;
        if (grp < ngroups) describe_all(grp, buf ^ 1);
        if (!zero) {
            float2 v[K::C][K::N2], x0[K::C];
            pfa_take<N>(s, v, x0, q1, l);
            pfa_lines<N, false>(s, v, x0, q1, l);
        }
        __syncthreads();
        if (grp < ngroups) {
            // the next group's pixel rows into L2
            for (int q = warp; q < kPfaNL; q += nw) {
                const FwdLine &f = lines[buf ^ 1][q];
                if (f.src < 0 || f.k < 0) continue;
                prefetch_row(img + f.src, f.n * (int)sizeof(T), lane);
                if (f.two) prefetch_row(img + f.src + g.isz, f.n * (int)sizeof(T), lane);
            }
            if (shared_flat) keep_flat(grp);
        }
        // the two real rows' half spectra of each line; padded rows beyond the
        // reflected data of a thin tile (deconvolver.py:135-137) are zero
        for (int q = warp; q < kPfaNL; q += nw) {
            if (ln[q].k < 0) break;
            float2 *d0 = Sb + ((long long)(2 * ln[q].k) * N + ln[q].x) * H + lane, *d1 = d0 + (long long)N * H;
            const bool two = ln[q].two;
            const float2 *lo = A + lane * kPitch + q, *hi = A + (N - lane) * kPitch + q;
#pragma unroll
            for (int u = 0; u < (H + 31) / 32; ++u) {
                if (lane + 32 * u >= H) continue;
                float2 a = make_float2(0.f, 0.f), b = a;
                if (!zero) {
                    // element N is element 0
                    const float2 ck = lo[32 * u * kPitch], cn = u == 0 && lane == 0 ? ck : hi[-32 * u * kPitch];
                    a = make_float2(ck.x + cn.x, ck.y - cn.y);
                    b = make_float2(ck.y + cn.y, cn.x - ck.x);
                }
                d0[32 * u] = a;
                if (two) d1[32 * u] = b;
            }
        }
        __syncthreads();
    }
    if (tid == 0) queue_leave(queue);
}

// ---------------------------------------------------------------------------
// inverse: two rows' half spectra -> one complex line -> two real rows.
// Whole rows (WIN false): lines are pairs of consecutive rows of the batch, the
// rows and, with delta >= 0, their box means along y (blur.cu:1-52 semantics)
// are written.  Windows (WIN true): the rows and columns of each tile that the
// caller reads (read_window), into `out` or the stitched buffer; the pairs are
// those of the whole-row pass, so the voxels are the same bits, and a tile's
// lines are numbered through its planes.
// ---------------------------------------------------------------------------
// What a line of a group is: rows `row` and row + 1 of the batch
struct InvLine {
    long long row;
    int z, x;   // plane and first row in it (windows); z < 0: no line
    int store;  // bit 0: the first row is stored, bit 1: the second
};

template <int N, bool WIN>
__global__ void __launch_bounds__(PfaK<N>::threads, 2)
k_rows_inv_pfa(const float2 *__restrict__ S, long long nrows, TileGeom g, int reach, float *__restrict__ out,
               float *__restrict__ blur, int delta, FftPlan P, float *__restrict__ stitch, long long osz, long long osx,
               unsigned *__restrict__ queue) {
    using K = PfaK<N>;
    constexpr int H = N / 2 + 1;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int next;
    __shared__ int cum[WIN ? MM_MAX_WIN_TILES + 1 : 1];  // groups before tile t
    __shared__ InvLine lines[2][kPfaNL];
    const PfaSmem<N> s = pfa_layout<N>(smem_raw, line_bytes<N>());
    float *rtab = reinterpret_cast<float *>(smem_raw + line_bytes<N>() + pfa_tail_bytes<N>());  // 1 / window count
    float2 *A = s.T;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    constexpr int nw = K::threads / 32;
    const int l = tid % kPfaNL, q1 = tid / kPfaNL;
    pfa_load_tables<N, true>(s, P);
    if constexpr (WIN) {
        for (int t = tid; t < g.nt; t += K::threads) {
            int xlo, xhi, ylo, yhi;
            read_window(g, t, reach, xlo, xhi, ylo, yhi);
            const int np = xhi > xlo ? (xhi - (xlo & ~1) + 1) / 2 : 0;
            cum[t + 1] = (g.Z * np + kPfaNL - 1) / kPfaNL;
        }
    } else if (delta >= 0) {
        for (int c = tid; c <= 2 * delta + 1; c += K::threads) rtab[c] = c ? 1.0f / (float)c : 0.f;
    }
    __syncthreads();
    if (WIN && tid == 0) {
        cum[0] = 0;
        for (int t = 0; t < g.nt; ++t) cum[t + 1] += cum[t];
    }
    for (int i = tid; i < 2 * K::N1 * K::ipad + 16; i += K::threads) s.tin[i] *= kPitchB;
    __syncthreads();
    const int ngroups = WIN ? cum[g.nt] : (int)((nrows / 2 + kPfaNL - 1) / kPfaNL);
    // line i of group grp (a thread each), t: a tile at or before the group's
    auto describe = [&](int grp, int i, int t) {
        InvLine f;
        if constexpr (WIN) {
            while (cum[t + 1] <= grp) ++t;
            int xlo, xhi, ylo, yhi;
            read_window(g, t, reach, xlo, xhi, ylo, yhi);
            const int np = (xhi - (xlo & ~1) + 1) / 2, L = (grp - cum[t]) * kPfaNL + i;
            f.z = L < g.Z * np ? L / np : -1;
            f.x = (xlo & ~1) + 2 * (L - L / np * np);
            f.row = ((long long)t * g.Z + f.z) * N + f.x;
            f.store = (f.x >= xlo ? 1 : 0) | (f.x + 1 < xhi ? 2 : 0);
        } else {
            f.row = 2LL * (grp * kPfaNL + i);
            f.z = f.row < nrows ? 0 : -1;
            f.x = 0;
            f.store = 3;
        }
        return f;
    };
    int t = 0, buf = 0, ylo = 0, yhi = N, t_known = -1;
    if ((int)blockIdx.x < ngroups && tid < kPfaNL) lines[0][tid] = describe(blockIdx.x, tid, 0);
    __syncthreads();
    for (int grp = blockIdx.x; grp < ngroups; buf ^= 1) {
        const int asked = tid == 0 ? queue_ask(queue, grp) : 0;
        if constexpr (WIN) {
            while (cum[t + 1] <= grp) ++t;
            if (t != t_known) {
                int xlo, xhi;
                read_window(g, t, reach, xlo, xhi, ylo, yhi);
                t_known = t;
            }
        }
        const InvLine *ln = lines[buf];
        for (int q = warp; q < kPfaNL; q += nw) {
            if (ln[q].z < 0) break;
            const float2 *r0 = S + ln[q].row * H, *r1 = r0 + H;
            // frequencies 1 .. N/2 - 1 give two elements each, all loads first;
            // 0 and N/2 one
            constexpr int U = (H - 2 + 31) / 32;
            float2 a[U], b[U];
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (lane + 32 * u < H - 2) {
                    a[u] = __ldcs(r0 + 1 + lane + 32 * u);
                    b[u] = __ldcs(r1 + 1 + lane + 32 * u);
                }
            float2 *lo = A + (1 + lane) * kPitch + q, *hi = A + (N - 1 - lane) * kPitch + q;
            if (lane < 2) A[lane * (N / 2) * kPitch + q] = make_float2(r0[lane * (N / 2)].x, r1[lane * (N / 2)].x);
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (lane + 32 * u < H - 2) {
                    lo[32 * u * kPitch] = make_float2(a[u].x - b[u].y, a[u].y + b[u].x);
                    hi[-32 * u * kPitch] = make_float2(a[u].x + b[u].y, b[u].x - a[u].y);
                }
        }
        if (tid == 0) next = asked;
        __syncthreads();
        grp = next;
        if (grp < ngroups && tid < kPfaNL) lines[buf ^ 1][tid] = describe(grp, tid, t);
        float2 v[K::C][K::N2], x0[K::C];
        pfa_take<N>(s, v, x0, q1, l);
        pfa_lines<N, true>(s, v, x0, q1, l);
        __syncthreads();
        if (grp < ngroups)
            // the next group's spectrum rows into L2
            for (int q = warp; q < kPfaNL && lines[buf ^ 1][q].z >= 0; q += nw)
                prefetch_row(S + lines[buf ^ 1][q].row * H, 2 * H * 8, lane);
        for (int q = warp; q < kPfaNL; q += nw) {
            if (ln[q].z < 0) break;
            const int z = ln[q].z, x = ln[q].x;
            const long long r0 = ln[q].row;
            const bool first = ln[q].store & 1, second = ln[q].store & 2;
            if (WIN && stitch) {
                // the FOV voxels whose last writer in the reference's order is
                // this tile (Deconvolver.apply, deconvolver.py:179-183): all of
                // its own span, past which each voxel asks. The unrolled loop
                // without a test: 0.253 -> 0.221 ms for a 50x1000x1500 volume
                // of 500-voxel tiles
                const TileDesc d = mm_tile_desc(g, g.t0 + t);
                const int ox = d.x + x - g.ov;
                float *s0 = stitch + z * osz + (long long)ox * osx + (d.y - g.ov), *s1 = s0 + osx;
                const int spanx = min(d.x + g.ts, g.X);
                int e = ylo + lane;
                if (first && second && ox + 1 < spanx) {
                    const int own = min(yhi, min(g.ts, g.Y - d.y) + g.ov);
#pragma unroll 8
                    for (; e < own; e += 32) {
                        const float2 w = A[e * kPitch + q];
                        s0[e] = w.x;
                        s1[e] = w.y;
                    }
                }
                for (; e < yhi; e += 32) {
                    const float2 w = A[e * kPitch + q];
                    const int oy = d.y + e - g.ov;
                    if (oy >= g.Y) break;
                    auto mine = [&](int x) {
                        return x < g.X && ((x < spanx && oy < d.y + g.ts) || mm_stitch_owner(g, x, oy) == g.t0 + t);
                    };
                    if (first && mine(ox)) s0[e] = w.x;
                    if (second && mine(ox + 1)) s1[e] = w.y;
                }
                continue;
            }
            float *o0 = out + r0 * N, *o1 = o0 + N;
            if (first && second) {
#pragma unroll 8
                for (int e = ylo + lane; e < yhi; e += 32) {
                    const float2 w = A[e * kPitch + q];
                    o0[e] = w.x;
                    o1[e] = w.y;
                }
            } else {
                for (int e = ylo + lane; e < yhi; e += 32) {
                    const float2 w = A[e * kPitch + q];
                    if (first) o0[e] = w.x;
                    if (second) o1[e] = w.y;
                }
            }
            if (WIN || delta < 0) continue;
            // y box mean of both rows: each lane slides a window along a
            // segment (an odd number of elements: lanes in distinct banks),
            // and the sums wait in registers until every lane is through
            constexpr int seg = ((N + 31) / 32) | 1;
            const int s0 = lane * seg;
            float2 m[seg], sum = make_float2(0.f, 0.f);
            if (s0 < N)
                for (int i = max(s0 - delta, 0); i <= min(s0 + delta, N - 1); ++i) sum = padd(sum, A[i * kPitch + q]);
            const float2 *pa = A + (s0 + delta) * kPitch + q, *pd = A + (s0 - delta - 1) * kPitch + q;
#pragma unroll
            for (int u = 0; u < seg; ++u) {
                const int e = s0 + u;
                if (u > 0 && e + delta < N) sum = padd(sum, pa[u * kPitch]);
                if (u > 0 && e > delta && e < N) sum = psub(sum, pd[u * kPitch]);
                m[u] = sum;
            }
            __syncwarp();
#pragma unroll
            for (int u = 0; u < seg; ++u) {
                const int e = s0 + u;
                if (e < N) A[e * kPitch + q] = pmul(m[u], rtab[min(e + delta, N - 1) - max(e - delta, 0) + 1]);
            }
            __syncwarp();
            float *b0 = blur + r0 * N, *b1 = b0 + N;
#pragma unroll 4
            for (int e = lane; e < N; e += 32) {
                const float2 w = A[e * kPitch + q];
                b0[e] = w.x;
                b1[e] = w.y;
            }
        }
        __syncthreads();
    }
    if (tid == 0) queue_leave(queue);
}

template <int N>
size_t rows_smem() {
    return line_bytes<N>() + pfa_tail_bytes<N>();
}

template <typename T, int N>
int launch_fwd(const TileGeom &g, const void *img, const float *flat, float2 *S, const FftPlan &P, unsigned *queue,
               cudaStream_t st) {
    using K = PfaK<N>;
    int zp = (g.Z + 1) / 2, gx = mm_cdiv((long)N * zp, kPfaNL), ngroups = gx * g.nt;
    TileGeom ga = g;
    FftPlan Pa = P;
    void *args[] = {&ga, &img, &flat, &S, &Pa, &zp, &gx, &ngroups, &queue};
    return launch_fft_kernel((const void *)k_rows_fwd_pfa<T, N>, dim3(fft_grid(ngroups, {K::threads, 2})),
                             rows_smem<N>() + sizeof(float) * kFlatRows * N, st, args, K::threads);
}

template <int N, bool WIN>
int launch_inv(const float2 *S, long long nrows, const TileGeom &g, int reach, float *out, float *blur, int delta,
               const FftPlan &P, float *stitch, long long osz, long long osx, unsigned *queue, size_t sm, cudaStream_t st) {
    using K = PfaK<N>;
    // an upper bound of the groups (a windowed launch counts them itself)
    const long long ngroups = nrows / 2 / kPfaNL + (WIN ? g.nt : 1);
    TileGeom ga = g;
    FftPlan Pa = P;
    void *args[] = {&S, &nrows, &ga, &reach, &out, &blur, &delta, &Pa, &stitch, &osz, &osx, &queue};
    return launch_fft_kernel((const void *)k_rows_inv_pfa<N, WIN>, dim3(fft_grid(ngroups, {K::threads, 2})), sm, st, args,
                             K::threads);
}

}  // namespace

bool mm_rows_pfa_takes(const FftPlan &P, long long nrows) {
    return P.pfa_idx && nrows < (1LL << 31) - 64 * kPfaNL;
}

int mm_launch_rows_fwd_pfa(const TileGeom &g, const void *img, int dtype, const float *flat, float2 *S, const FftPlan &P,
                           unsigned *queue, cudaStream_t st) {
    if (dtype == MM_DTYPE_U16)
        return P.n == 678 ? launch_fwd<uint16_t, 678>(g, img, flat, S, P, queue, st)
                          : launch_fwd<uint16_t, 478>(g, img, flat, S, P, queue, st);
    return P.n == 678 ? launch_fwd<float, 678>(g, img, flat, S, P, queue, st)
                      : launch_fwd<float, 478>(g, img, flat, S, P, queue, st);
}

// false: the blur's table does not fit beside the lines (the caller takes the
// general pass)
bool mm_rows_inv_pfa_fits(const FftPlan &P, int delta) {
    const size_t rt = delta >= 0 ? sizeof(float) * (2 * (size_t)delta + 2) : 0;
    return (P.n == 678 ? rows_smem<678>() : rows_smem<478>()) + rt <= (size_t)fft_smem_limit({256, 2});
}

int mm_launch_rows_inv_pfa(const float2 *S, long long nrows, float *out, float *blur, int delta, const FftPlan &P,
                           unsigned *queue, cudaStream_t st) {
    const size_t rt = delta >= 0 ? sizeof(float) * (2 * (size_t)delta + 2) : 0;
    const TileGeom g = {};
    if (P.n == 678)
        return launch_inv<678, false>(S, nrows, g, 0, out, blur, delta, P, nullptr, 0, 0, queue, rows_smem<678>() + rt, st);
    return launch_inv<478, false>(S, nrows, g, 0, out, blur, delta, P, nullptr, 0, 0, queue, rows_smem<478>() + rt, st);
}

int mm_launch_rows_inv_win_pfa(const float2 *S, const TileGeom &g, int reach, float *out, float *stitch, long long osz,
                               long long osx, const FftPlan &P, unsigned *queue, cudaStream_t st) {
    const long long nrows = (long long)g.nt * g.Z * g.P;
    if (P.n == 678)
        return launch_inv<678, true>(S, nrows, g, reach, out, nullptr, -1, P, stitch, osz, osx, queue, rows_smem<678>(), st);
    return launch_inv<478, true>(S, nrows, g, reach, out, nullptr, -1, P, stitch, osz, osx, queue, rows_smem<478>(), st);
}
