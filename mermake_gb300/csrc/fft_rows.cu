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
    const int *op = s.tout + q1 * K::ipad;
#pragma unroll
    for (int c = 0; c < K::C; ++c)
#pragma unroll
        for (int q = 0; q < K::N2; ++q) *reinterpret_cast<float2 *>(A + op[c * K::N2 + q]) = v[c][q];
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
// per lane cover the longest row), so a line waits for memory once.
__device__ __forceinline__ float half_over(const float *f) { return f ? __fdividef(0.5f, *f) : 0.5f; }

template <int N>
__device__ __forceinline__ void stage_rows(const uint16_t *ra, const uint16_t *rb, const float *fr, int n,
                                           float2 *dst, int lane) {
    // words of two pixels of row a, y = 2 w - off and the next; the words that
    // reach past either end of the row are read as their one pixel.  Row b
    // comes the same way, or pixel by pixel where it starts on the other half
    // of a word.
    constexpr int U = (N / 2 + 1 + 31) / 32;
    const int off = (int)((reinterpret_cast<uintptr_t>(ra) >> 1) & 1);
    const unsigned *wa = reinterpret_cast<const unsigned *>(ra - off);
    const bool same = rb && !((reinterpret_cast<uintptr_t>(ra) ^ reinterpret_cast<uintptr_t>(rb)) & 2);
    const unsigned *wb = reinterpret_cast<const unsigned *>(rb - off);
    unsigned a[U], b[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int w = lane + 32 * u, y = 2 * w - off;
        const bool lo = y >= 0 && y < n, hi = y + 1 < n;
        a[u] = lo && hi ? wa[w] : lo ? ra[y] : hi ? (unsigned)ra[y + 1] << 16 : 0u;
    }
    if (same) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int w = lane + 32 * u, y = 2 * w - off;
            const bool lo = y >= 0 && y < n, hi = y + 1 < n;
            b[u] = lo && hi ? wb[w] : lo ? rb[y] : hi ? (unsigned)rb[y + 1] << 16 : 0u;
        }
    } else {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int y = 2 * (lane + 32 * u) - off;
            const unsigned lo = rb && y >= 0 && y < n ? rb[y] : 0u, hi = rb && y + 1 < n ? rb[y + 1] : 0u;
            b[u] = lo | hi << 16;
        }
    }
    // the two pixels of a word go out in the order that spreads a half warp's
    // 16 stores over all banks: lanes 8 .. 15 of each half start with the second
    const bool swap = lane & 8;
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int y = 2 * (lane + 32 * u) - off;
        // 0x4B00xxxx is 2^23 + xxxx: the pixel as a float, exactly
        const unsigned p0 = swap ? 0x7632 : 0x7610, p1 = swap ? 0x7610 : 0x7632;
        const int y0 = y + (swap ? 1 : 0), y1 = y + (swap ? 0 : 1);
        const float2 m = make_float2(8388608.f, 8388608.f);
        const float2 v0 = psub(make_float2(__uint_as_float(__byte_perm(a[u], 0x4B000000u, p0)),
                                           __uint_as_float(__byte_perm(b[u], 0x4B000000u, p0))), m);
        const float2 v1 = psub(make_float2(__uint_as_float(__byte_perm(a[u], 0x4B000000u, p1)),
                                           __uint_as_float(__byte_perm(b[u], 0x4B000000u, p1))), m);
        if (y0 >= 0 && y0 < n) dst[y0 * kPitch] = pmul(v0, half_over(fr ? fr + y0 : nullptr));
        if (y1 >= 0 && y1 < n) dst[y1 * kPitch] = pmul(v1, half_over(fr ? fr + y1 : nullptr));
    }
}
template <int N>
__device__ __forceinline__ void stage_rows(const float *ra, const float *rb, const float *fr, int n, float2 *dst,
                                           int lane) {
    constexpr int U = (N + 31) / 32;
    float a[U], b[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int y = lane + 32 * u;
        a[u] = y < n ? ra[y] : 0.f;
        b[u] = rb && y < n ? rb[y] : 0.f;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int y = lane + 32 * u;
        if (y < n) dst[y * kPitch] = pmul(make_float2(a[u], b[u]), half_over(fr ? fr + y : nullptr));
    }
}

// rows of `bytes` bytes at p into L2, a lane per 128 bytes
__device__ __forceinline__ void prefetch_row(const void *p, int bytes, int lane) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(p) & ~(uintptr_t)127, e = reinterpret_cast<uintptr_t>(p) + bytes;
    for (uintptr_t c = a + 128 * lane; c < e; c += 128 * 32) asm volatile("prefetch.global.L2 [%0];" ::"l"(c));
}

template <typename T, int N>
__global__ void __launch_bounds__(PfaK<N>::threads, 2)
k_rows_fwd_pfa(TileGeom g, const T *__restrict__ img, const float *__restrict__ flat, float2 *__restrict__ S, FftPlan P,
               int zp, int gx, int ngroups, unsigned *__restrict__ queue) {
    using K = PfaK<N>;
    constexpr int H = N / 2 + 1;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int next;
    const PfaSmem<N> s = pfa_layout<N>(smem_raw, line_bytes<N>());
    float2 *A = s.T;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    constexpr int nw = K::threads / 32;
    const int l = tid % kPfaNL, q1 = tid / kPfaNL;
    pfa_load_tables<N, false>(s, P);
    for (int i = tid; i < kPitch; i += K::threads) A[N * kPitch + i] = make_float2(0.f, 0.f);
    __syncthreads();
    for (int i = tid; i < K::N1 * K::ipad; i += K::threads) s.tout[i] *= kPitchB;
    if (tid < 8) s.out0[tid] *= kPitchB;
    const int LT = N * zp;  // lines of a tile
    int tile = -1;
    TileDesc d;
    for (int grp = blockIdx.x; grp < ngroups;) {
        const int asked = tid == 0 ? queue_ask(queue, grp) : 0;
        const int by = grp / gx, L0 = (grp - by * gx) * kPfaNL;
        if (by != tile) {
            // the input table of this tile: padded column -> staged pixel
            tile = by;
            d = mm_tile_desc(g, g.t0 + by);
            for (int i = tid; i < K::N1 * K::ipad; i += K::threads) {
                const int m = mm_map_xy(P.pfa_idx[i], d.y == 0, d.yd, N, g.ov);
                s.tin[i] = (m < 0 ? N : m) * kPitchB;
            }
            if (tid < K::C) {
                const int m = mm_map_xy(P.pfa_idx[2 * K::N1 * K::ipad + tid], d.y == 0, d.yd, N, g.ov);
                s.in0[tid] = (m < 0 ? N : m) * kPitchB;
            }
        }
        const int Lend = min(L0 + kPfaNL, LT);
        float2 *Sb = S + (long long)by * g.Z * N * H;
        bool zero = true;
        for (int x = L0 / zp; x <= (Lend - 1) / zp; ++x) zero = zero && mm_map_xy(x, d.x == 0, d.xd, N, g.ov) < 0;
        if (zero) {
            // padded rows beyond the reflected data of a thin tile
            // (deconvolver.py:135-137) transform to zero
            for (int L = L0 + warp; L < Lend; L += nw) {
                const int x = L / zp, k = L - x * zp;
                for (int z = 2 * k; z < min(2 * k + 2, g.Z); ++z)
                    for (int e = lane; e < H; e += 32) Sb[((long long)z * N + x) * H + e] = make_float2(0.f, 0.f);
            }
            if (tid == 0) next = asked;
            __syncthreads();
            grp = next;
            __syncthreads();
            continue;
        }
        for (int q = warp; q < kPfaNL; q += nw) {
            const int L = L0 + q;
            float2 *dst = A + q;
            const T *ra = nullptr, *rb = nullptr;
            const float *fr = nullptr;
            if (L < LT) {
                const int x = L / zp, k = L - x * zp;
                const int sx = mm_map_xy(x, d.x == 0, d.xd, N, g.ov);
                if (sx >= 0) {
                    ra = img + 2 * k * g.isz + (long long)(d.x0 + sx) * g.isx + d.y0;
                    if (2 * k + 1 < g.Z) rb = ra + g.isz;
                    if (flat) fr = flat + (long long)(d.x0 + sx) * g.fsx + d.y0;
                }
            }
            if (ra)
                stage_rows<N>(ra, rb, fr, d.yd, dst, lane);
            else
                for (int y = lane; y < d.yd; y += 32) dst[y * kPitch] = make_float2(0.f, 0.f);
        }
        if (tid == 0) next = asked;
        __syncthreads();
        grp = next;
        if (grp < ngroups && grp / gx == by) {
            // the next group's pixel rows into L2 (past the rows of this one:
            // a group is 16 lines of the same or the next x)
            const int N0 = (grp - by * gx) * kPfaNL;
            for (int q = warp; q < kPfaNL && N0 + q < LT; q += nw) {
                const int x = (N0 + q) / zp, k = N0 + q - x * zp;
                const int sx = mm_map_xy(x, d.x == 0, d.xd, N, g.ov);
                if (sx < 0) continue;
                const T *ra = img + 2 * k * g.isz + (long long)(d.x0 + sx) * g.isx + d.y0;
                prefetch_row(ra, d.yd * (int)sizeof(T), lane);
                if (2 * k + 1 < g.Z) prefetch_row(ra + g.isz, d.yd * (int)sizeof(T), lane);
            }
        }
        float2 v[K::C][K::N2], x0[K::C];
        pfa_take<N>(s, v, x0, q1, l);
        pfa_lines<N, false>(s, v, x0, q1, l);
        __syncthreads();
        // the two real rows' half spectra of each line
        for (int q = warp; q < kPfaNL; q += nw) {
            const int L = L0 + q;
            if (L >= LT) break;
            const int x = L / zp, k = L - x * zp;
            float2 *d0 = Sb + ((long long)(2 * k) * N + x) * H, *d1 = d0 + (long long)N * H;
            const bool two = 2 * k + 1 < g.Z;
#pragma unroll 4
            for (int e = lane; e < H; e += 32) {
                const float2 ck = A[e * kPitch + q], cn = A[(e == 0 ? 0 : N - e) * kPitch + q];
                d0[e] = make_float2(ck.x + cn.x, ck.y - cn.y);
                if (two) d1[e] = make_float2(ck.y + cn.y, cn.x - ck.x);
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
constexpr int kMaxWinTiles = 256;

template <int N, bool WIN>
__global__ void __launch_bounds__(PfaK<N>::threads, 2)
k_rows_inv_pfa(const float2 *__restrict__ S, long long nrows, TileGeom g, int reach, float *__restrict__ out,
               float *__restrict__ blur, int delta, FftPlan P, float *__restrict__ stitch, long long osz, long long osx,
               unsigned *__restrict__ queue) {
    using K = PfaK<N>;
    constexpr int H = N / 2 + 1;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int next;
    __shared__ int cum[WIN ? kMaxWinTiles + 1 : 1];  // groups before tile t
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
    int t = 0;
    for (int grp = blockIdx.x; grp < ngroups;) {
        const int asked = tid == 0 ? queue_ask(queue, grp) : 0;
        // line q of the group: rows row(q) and row(q) + 1 of the batch (the
        // first one even); nl lines exist
        int xlo = 0, xhi = N, ylo = 0, yhi = N, np = 0, nl, L0;
        long long tbase = 0;
        if constexpr (WIN) {
            while (cum[t + 1] <= grp) ++t;
            read_window(g, t, reach, xlo, xhi, ylo, yhi);
            np = (xhi - (xlo & ~1) + 1) / 2;
            L0 = (grp - cum[t]) * kPfaNL;
            nl = min(kPfaNL, g.Z * np - L0);
            tbase = (long long)t * g.Z * N;
        } else {
            L0 = grp * kPfaNL;
            nl = (int)min((long long)kPfaNL, nrows / 2 - L0);
        }
        // plane and first row (in its plane) of line q
        auto line_at = [&](int q, int &z, int &x) {
            z = WIN ? (L0 + q) / np : 0;
            x = WIN ? (xlo & ~1) + 2 * (L0 + q - z * np) : 0;
        };
        auto row_of = [&](int q, int z, int x) { return WIN ? tbase + (long long)z * N + x : 2LL * (L0 + q); };
        for (int q = warp; q < nl; q += nw) {
            int z, x;
            line_at(q, z, x);
            const float2 *r0 = S + row_of(q, z, x) * H, *r1 = r0 + H;
            constexpr int U = 4;
            for (int k0 = lane; k0 < H; k0 += 32 * U) {
                float2 a[U], b[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int k = k0 + 32 * u;
                    a[u] = b[u] = make_float2(0.f, 0.f);
                    if (k < H) {
                        a[u] = __ldcs(r0 + k);
                        b[u] = __ldcs(r1 + k);
                    }
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int k = k0 + 32 * u;
                    if (k >= H) break;
                    if (k == 0 || k == N / 2) {
                        A[k * kPitch + q] = make_float2(a[u].x, b[u].x);
                    } else {
                        A[k * kPitch + q] = make_float2(a[u].x - b[u].y, a[u].y + b[u].x);
                        A[(N - k) * kPitch + q] = make_float2(a[u].x + b[u].y, b[u].x - a[u].y);
                    }
                }
            }
        }
        if (tid == 0) next = asked;
        __syncthreads();
        grp = next;
        if (!WIN || grp < cum[t + 1]) {
            // the next group's spectrum rows into L2
            const int N0 = WIN ? (grp - cum[t]) * kPfaNL : grp * kPfaNL;
            const long long end = WIN ? (long long)g.Z * np : nrows / 2;
            for (int q = warp; q < kPfaNL && N0 + q < end; q += nw) {
                const int z = WIN ? (N0 + q) / np : 0;
                const long long row = WIN ? tbase + (long long)z * N + (xlo & ~1) + 2 * (N0 + q - z * np) : 2LL * (N0 + q);
                prefetch_row(S + row * H, 2 * H * 8, lane);
            }
        }
        float2 v[K::C][K::N2], x0[K::C];
        pfa_take<N>(s, v, x0, q1, l);
        pfa_lines<N, true>(s, v, x0, q1, l);
        __syncthreads();
        for (int q = warp; q < nl; q += nw) {
            int z, x;
            line_at(q, z, x);
            const long long r0 = row_of(q, z, x);
            const bool first = !WIN || x >= xlo, second = !WIN || x + 1 < xhi;
            if (WIN && stitch) {
                // the FOV voxels whose last writer in the reference's order is
                // this tile (Deconvolver.apply, deconvolver.py:179-183)
                const TileDesc d = mm_tile_desc(g, g.t0 + t);
                for (int e = ylo + lane; e < yhi; e += 32) {
                    const float2 w = A[e * kPitch + q];
                    const int oy = d.y + e - g.ov;
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        const int ox = d.x + x + c - g.ov;
                        if (!(c ? second : first) || ox >= g.X || oy >= g.Y) continue;
                        const bool own = ox < d.x + g.ts && oy < d.y + g.ts;
                        if (own || mm_stitch_owner(g, ox, oy) == g.t0 + t)
                            stitch[z * osz + (long long)ox * osx + oy] = c ? w.y : w.x;
                    }
                }
                continue;
            }
            float *o0 = out + r0 * N, *o1 = o0 + N;
#pragma unroll 4
            for (int e = ylo + lane; e < yhi; e += 32) {
                const float2 w = A[e * kPitch + q];
                if (first) o0[e] = w.x;
                if (second) o1[e] = w.y;
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
    return launch_fft_kernel((const void *)k_rows_fwd_pfa<T, N>, dim3(fft_grid(ngroups, {K::threads, 2})), rows_smem<N>(),
                             st, args, K::threads);
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
