// z operator of one Wiener spectrum over a tile batch by short transforms held
// in registers, for the two paddings whose reflections cover whole depths.
//
// Y[t][i][p] = sum_j M_p[i][j] X[t][j][p], with M a Toeplitz matrix plus masked
// Hankel ones (zop_tma.cu).  At zpad = Z - 1 both Hankel parts reach over all j
// but one end each, at 2 zpad = Z - 2 (Zp = 2Z - 2) they are one that reaches
// over all but both ends.  With x~ = x, its first and last planes halved,
//
//   Y[i] = sum_j a[i - j] x~[j] + sum_j b[i + j] x~[j] + (far ends),
//   a[s] = w[s],  b[s] = w[s] (+ w[s - 2Z + 2] at zpad = Z - 1),
//   far ends = x~[0] w[i - 2Z + 2] + x~[Z-1] w[i + Z - 1], at zpad = Z - 1 only,
//
// and both sums are products of transforms of 2N >= 2Z points: with X^ that of
// x~ followed by zeros, Y^[k] = a^[k] X^[k] + b^[k] X^[-k].  The even
// frequencies of a sequence of N values and N zeros are its N-point transform,
// the odd ones that of the sequence times exp(-pi i j / N), and only the first
// half of the inverse is wanted, so a column takes four N-point transforms in
// registers where the matrix form takes Z^2 products and forms the entries.
//
// A CTA (one per SM, persistent) takes groups of 64 consecutive frequencies.
// First its eight warps make the tables a^ and b^ (times the normalisation and
// the folded blur's factor) of the group from the z kernel, a warp for 32
// frequencies of one table's even or odd half.  Then a pair of warps per tile
// and 32 frequencies, a lane each: one does the even frequencies, one the odd,
// and they exchange what the other finishes through shared memory.  A tile's
// planes come by cp.async while the pair works on the tile before.
//
// What bounds it: instruction issue and fetch.  A column is about 7 k
// instructions, nearly all straight-line code, 110 KB in all; warps that ran
// through it apart (jobs taken from a counter, twelve warps) spent half of
// their time waiting for instructions (3.4 ms at 25 tiles).  So the two warps of an SM
// sub-partition run the same steps side by side, one of each half, and all
// warps finish a group together.  At P = 678, Z = 50 (ms per launch, zpad 49 /
// 24, the matrix form in brackets): 4 tiles 0.45 / 0.38 [0.55 / 0.58], 6 tiles
// 0.59 / 0.52 [0.72 / 0.75], 9 tiles 0.88 / 0.80 [1.12 / 1.17], 25 tiles 2.05 /
// 1.94 [2.69 / 2.72].  Three warps a sub-partition with 168 registers took
// 2.3 ms, four threads a column (transforms of N / 2) 2.9 ms at 25 tiles.
//
// Every column is computed alone with the same operations, so a tile's result
// does not depend on the batch.  The largest error against 64-bit sums, over
// random columns at Z = 50, was 5.3e-8 to 8.9e-8 of the largest output where
// the matrix form has 4.7e-8 to 1.2e-7.
#include <type_traits>

#include "deconv.cuh"
#include "fft_pfa.cuh"

namespace {

__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }
// barrier of a pair of warps
__device__ __forceinline__ void pair_sync(int pair) { asm volatile("bar.sync %0, 64;" ::"r"(pair + 1) : "memory"); }
__device__ __forceinline__ float2 cfma(float2 a, float2 b, float2 c) {
    c.x = fmaf(a.x, b.x, c.x);
    c.y = fmaf(a.x, b.y, c.y);
    c.x = fmaf(-a.y, b.y, c.x);
    c.y = fmaf(a.y, b.x, c.y);
    return c;
}

// cos(pi m / N) and sin(pi m / N), m = 0 .. 2N - 1: the Taylor series about 0
// after reduction to [0, pi / 4], at compile time
template <int N>
struct HalfCircle {
    float c[2 * N], s[2 * N];
    static constexpr double series(double x, bool sine) {
        double term = sine ? x : 1.0, sum = term;
        for (int k = sine ? 3 : 2; k < 26; k += 2) {
            term *= -x * x / (k * (k - 1));
            sum += term;
        }
        return sum;
    }
    static constexpr double at(int m, bool sine) {  // sin or cos of pi m / N, 0 <= m < 2N
        if (m >= N) return -at(m - N, sine);
        if (2 * m > N) return sine ? at(N - m, true) : -at(N - m, false);
        constexpr double pi = 3.14159265358979323846;
        return 4 * m > N ? series(pi * (N - 2 * m) / (2 * N), !sine) : series(pi * m / N, sine);
    }
    constexpr HalfCircle() : c(), s() {
        for (int m = 0; m < 2 * N; ++m) {
            c[m] = (float)at(m, false);
            s[m] = (float)at(m, true);
        }
    }
};
template <int N>
__device__ __forceinline__ float2 unit_root(int m) {  // exp(pi i m / N)
    constexpr HalfCircle<N> t;
    return make_float2(t.c[m], t.s[m]);
}

// ---- transforms of registers, natural order in and out ----------------------
template <int N, bool INV>
__device__ __forceinline__ void zdft(float2 *v);

template <bool INV>
__device__ __forceinline__ void zdft5(float2 *v) {
    constexpr float c1 = 0.30901699437494742410f, c2 = -0.80901699437494742410f;
    constexpr float s1 = 0.95105651629515357212f, s2 = 0.58778525229247312917f;
    const float2 a1 = padd(v[1], v[4]), b1 = psub(v[1], v[4]), a2 = padd(v[2], v[3]), b2 = psub(v[2], v[3]);
    const float2 t1 = make_float2(fmaf(c2, a2.x, fmaf(c1, a1.x, v[0].x)), fmaf(c2, a2.y, fmaf(c1, a1.y, v[0].y)));
    const float2 t2 = make_float2(fmaf(c1, a2.x, fmaf(c2, a1.x, v[0].x)), fmaf(c1, a2.y, fmaf(c2, a1.y, v[0].y)));
    const float2 u1 = make_float2(fmaf(s2, b2.x, s1 * b1.x), fmaf(s2, b2.y, s1 * b1.y));
    const float2 u2 = make_float2(fmaf(-s1, b2.x, s2 * b1.x), fmaf(-s1, b2.y, s2 * b1.y));
    v[0] = padd(v[0], padd(a1, a2));
    v[1] = INV ? paddi(t1, u1) : psubi(t1, u1);
    v[4] = INV ? psubi(t1, u1) : paddi(t1, u1);
    v[2] = INV ? paddi(t2, u2) : psubi(t2, u2);
    v[3] = INV ? psubi(t2, u2) : paddi(t2, u2);
}
template <bool INV>
__device__ __forceinline__ void zdft8(float2 *v) {
    float2 e[4], o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        e[j] = padd(v[j], v[j + 4]);
        o[j] = psub(v[j], v[j + 4]);
    }
    o[1] = pw8<INV>(o[1]);
    o[2] = mul_i<INV>(o[2]);
    o[3] = pw8_3<INV>(o[3]);
    pdft4<INV>(e[0], e[1], e[2], e[3]);
    pdft4<INV>(o[0], o[1], o[2], o[3]);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        v[2 * j] = e[j];
        v[2 * j + 1] = o[j];
    }
}
// A and B coprime: inputs B a + A b, outputs by residues (Good 1958)
template <int A, int B, bool INV>
__device__ __forceinline__ void zdft_coprime(float2 *v) {
    constexpr int N = A * B;
    float2 t[A][B];
#pragma unroll
    for (int b = 0; b < B; ++b) {
        float2 u[A];
#pragma unroll
        for (int a = 0; a < A; ++a) u[a] = v[(B * a + A * b) % N];
        zdft<A, INV>(u);
#pragma unroll
        for (int a = 0; a < A; ++a) t[a][b] = u[a];
    }
#pragma unroll
    for (int a = 0; a < A; ++a) zdft<B, INV>(t[a]);
#pragma unroll
    for (int k = 0; k < N; ++k) v[k] = t[k % A][k % B];
}
// R R points with twiddles (Cooley and Tukey 1965)
template <int R, bool INV>
__device__ __forceinline__ void zdft_square(float2 *v) {
    float2 t[R][R];
#pragma unroll
    for (int b = 0; b < R; ++b) {
        float2 u[R];
#pragma unroll
        for (int a = 0; a < R; ++a) u[a] = v[R * a + b];
        zdft<R, INV>(u);
#pragma unroll
        for (int k = 0; k < R; ++k) {
            const float2 w = unit_root<R * R>(2 * b * k % (2 * R * R));
            t[k][b] = b * k == 0 ? u[k] : cmul(u[k], make_float2(w.x, INV ? w.y : -w.y));
        }
    }
#pragma unroll
    for (int k = 0; k < R; ++k) zdft<R, INV>(t[k]);
#pragma unroll
    for (int k = 0; k < R * R; ++k) v[k] = t[k % R][k / R];
}
template <int N, bool INV>
__device__ __forceinline__ void zdft(float2 *v) {
    if constexpr (N == 2) {
        const float2 a = v[0], b = v[1];
        v[0] = padd(a, b);
        v[1] = psub(a, b);
    } else if constexpr (N == 3) {
        pdft3<INV>(v[0], v[1], v[2]);
    } else if constexpr (N == 5) {
        zdft5<INV>(v);
    } else if constexpr (N == 6) {
        pdft6<INV>(v[0], v[1], v[2], v[3], v[4], v[5]);
    } else if constexpr (N == 7) {
        pdft_odd<7, INV>(v);
    } else if constexpr (N == 8) {
        zdft8<INV>(v);
    } else if constexpr (N == 9) {
        zdft_square<3, INV>(v);
    } else if constexpr (N == 25) {
        zdft_square<5, INV>(v);
    } else if constexpr (N == 50) {
        zdft_coprime<2, 25, INV>(v);
    } else if constexpr (N == 56) {
        zdft_coprime<7, 8, INV>(v);
    } else {
        static_assert(N % 5 == 0 && N > 25, "no transform of this length");
        zdft_coprime<5, N / 5, INV>(v);
    }
}

struct ZfArgs {
    int Z, Zp, nt;
    int far;            // zpad = Z - 1
    int ngroups;        // frequency groups
    long long plane;
    const float *fresp;
};
constexpr int kPB = 64;    // frequencies of a group: two rows of a warp
constexpr int kWarps = 8;  // of a CTA
constexpr int kZfMinZ = 26;
constexpr int zf_low(int n) { return n == 30 ? kZfMinZ : n == 56 ? 51 : n == 50 ? 46 : n - 4; }
constexpr size_t zf_tables(int n) { return sizeof(float2) * 4 * n * kPB; }
// rows of the far ends in shared memory, where they fit beside the rest
constexpr size_t zf_far(int n) { return n > 50 ? 0 : sizeof(float2) * (n + 1) * kPB; }
constexpr size_t zf_buffer(int n) { return sizeof(float2) * n * 32; }  // exchanged by a pair of warps

// Y^(p) and Y^(q) from X^(p) and X^(q), q the place of the negative frequency of
// p: even frequencies 2p (H false) have q = -p, odd ones 2p + 1 q = -p - 1.
// Real and imaginary parts change places, so that the forward transform that
// follows is the inverse with its parts in each other's place.
template <int N, bool H, int PB>
__device__ __forceinline__ void zf_mix(float2 *v, const float2 *A, const float2 *B) {
#pragma unroll
    for (int p = 0; p < N; ++p) {
        const int q = H ? N - 1 - p : (N - p) % N;
        if (q < p) continue;
        const float2 xp = v[p], xq = v[q];
        auto make = [&](int k, float2 x, float2 y) {
            const float2 a = A[k * PB], b = B[k * PB];
            float2 r = make_float2(a.x * x.x, a.x * x.y);
            r.x = fmaf(-a.y, x.y, r.x);
            r.y = fmaf(a.y, x.x, r.y);
            r.x = fmaf(b.x, y.x, r.x);
            r.y = fmaf(b.x, y.y, r.y);
            r.x = fmaf(-b.y, y.y, r.x);
            r.y = fmaf(b.y, y.x, r.y);
            return make_float2(r.y, r.x);
        };
        v[p] = make(p, xp, xq);
        if (q != p) v[q] = make(q, xq, xp);
    }
}

// The N values whose transform is one half (even or odd) of the frequencies of
// the generator a (kind 0) or b (kind 1): g[s] + g[s + N] for the even half, g[s]
// - g[s + N] for the odd one.  Each warp of the pair loads one part of it and
// hands over what the other needs (where both loaded all of it a launch took
// 0.04 ms longer).
template <int N>
__device__ __forceinline__ void zf_generator(float2 *v, int kind, int half, const char *wp, unsigned pb8, const ZfArgs &a,
                                             float2 *buf, int pair) {
    constexpr int LO = zf_low(N), M0 = (N + 1) / 2;
    const int Z = a.Z;
    auto wrow = [&](int row) { return __ldg(reinterpret_cast<const float2 *>(wp + (unsigned)row * pb8)); };
    auto load = [&](auto odd) {
        constexpr int H = decltype(odd)::value, S0 = H ? M0 : 0, L = H ? N - M0 : M0;
        float2 lo[L], hi[L];
        auto in = [&](int s) { return s + N <= 2 * LO - 2 || (s + N <= 2 * N - 2 && s + N <= 2 * Z - 2); };
        if (kind == 0) {
#pragma unroll
            for (int i = 0; i < L; ++i) {
                const int s = S0 + i;
                lo[i] = s < LO || s < Z ? wrow(s) : make_float2(0.f, 0.f);
                hi[i] = N - s < LO || N - s < Z ? wrow(a.Zp - N + s) : make_float2(0.f, 0.f);
            }
        } else {
#pragma unroll
            for (int i = 0; i < L; ++i) {
                const int s = S0 + i;
                lo[i] = wrow(s);
                hi[i] = in(s) ? wrow(s + N >= a.Zp ? s + N - a.Zp : s + N) : make_float2(0.f, 0.f);
            }
            if (a.far) {
#pragma unroll
                for (int i = 0; i < L; ++i) {
                    const int s = S0 + i, r = s + N + Z;
                    lo[i] = padd(lo[i], wrow(s + Z));
                    if (in(s)) hi[i] = padd(hi[i], wrow(r >= a.Zp ? r - a.Zp : r));
                }
            }
        }
#pragma unroll
        for (int i = 0; i < L; ++i) {
            const float2 sum = padd(lo[i], hi[i]), dif = psub(lo[i], hi[i]);
            v[S0 + i] = H ? dif : sum;
            buf[(S0 + i) * 32] = H ? sum : dif;
        }
        pair_sync(pair);
        constexpr int T0 = H ? 0 : M0;
#pragma unroll
        for (int i = 0; i < N - L; ++i) v[T0 + i] = buf[(T0 + i) * 32];
    };
    if (half)
        load(std::true_type{});
    else
        load(std::false_type{});
}

template <int N>
__global__ void __launch_bounds__(kWarps * 32, 1)
k_zfft_apply(float2 *__restrict__ S, const float2 *__restrict__ w, const ZfArgs a) {
    constexpr int LO = zf_low(N);
    constexpr int TR = kWarps / 4;  // tiles of a round
    constexpr bool FARS = zf_far(N) > 0;
    extern __shared__ __align__(16) unsigned char zf_smem[];
    const int Z = a.Z, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int half = warp / (kWarps / 2);                 // even or odd frequencies
    const int pair = warp % (kWarps / 2), fsub = pair & 1;
    float2 *xbuf = reinterpret_cast<float2 *>(zf_smem + zf_tables(N)) + pair * N * 32;
    float2 *buf = xbuf + kWarps / 2 * N * 32 + lane;
    float2 *wfar = reinterpret_cast<float2 *>(zf_smem + zf_tables(N) + kWarps * zf_buffer(N));  // rows Z - 1 ..
    const unsigned pb8 = (unsigned)a.plane * 8u;  // bytes of a plane (checked by the launcher)
    const int rounds = (a.nt + TR - 1) / TR;
    for (int grp = blockIdx.x; grp < a.ngroups; grp += gridDim.x) {
        // a tile's planes of the pair's 32 frequencies into xbuf, 16 bytes (two
        // frequencies) per copy; past the plane nothing (not stored either)
        auto stage = [&](int t) {
            const long long q = (long long)grp * kPB + fsub * 32 + 2 * (lane & 15);
            if (q < a.plane) {
                const float2 *src = S + (long long)t * Z * a.plane + q;
                for (int j = half * 2 + (lane >> 4); j < Z; j += 4)
                    cp_async16(xbuf + j * 32 + 2 * (lane & 15), src + (long long)j * a.plane);
            }
        };
        if ((pair >> 1) < a.nt) stage(pair >> 1);
#pragma unroll 1
        for (int item = 0; item <= rounds; ++item) {
            const bool table = item == 0;
            // table job: a^ (kind 0) or b^ (kind 1) of 32 frequencies
            const int kind = pair & 1;
            const int sub = table ? pair >> 1 : fsub;
            const int t = (pair >> 1) + (item - 1) * TR;
            const bool active = table || t < a.nt;
            const long long p = (long long)grp * kPB + sub * 32 + lane;
            const long long pc = p < a.plane ? p : a.plane - 1;
            const char *wp = reinterpret_cast<const char *>(w + pc);
            auto wrow = [&](int row) { return __ldg(reinterpret_cast<const float2 *>(wp + (unsigned)row * pb8)); };
            float2 *tab = reinterpret_cast<float2 *>(zf_smem) + sub * 32 + lane;
            float2 v[N], e0, e1;
            if (active) {
                if (table) {
                    zf_generator<N>(v, kind, half, wp, pb8, a, buf, pair);
                } else {
                    cp_async_wait();
                    pair_sync(pair);
                    const float2 *x = xbuf + lane;
#pragma unroll
                    for (int j = 0; j < N; ++j) v[j] = j < LO || j < Z ? x[j * 32] : make_float2(0.f, 0.f);
                    // the ends halved (planes past the last are zero)
                    e0 = pmul(v[0], 0.5f);
                    e1 = pmul(x[(Z - 1) * 32], 0.5f);
                    v[0] = e0;
#pragma unroll
                    for (int j = LO - 1; j < N; ++j) v[j] = pmul(v[j], j < Z - 1 ? 1.f : 0.5f);
                    pair_sync(pair);
                    if (t + TR < a.nt) stage(t + TR);
                }
                if (half) {
#pragma unroll
                    for (int j = 1; j < N; ++j) v[j] = cmul(v[j], make_float2(unit_root<N>(j).x, -unit_root<N>(j).y));
                }
#pragma unroll 1
                for (int dir = 0;; ++dir) {
                    zdft<N, false>(v);
                    if (table || dir) break;
                    if (half)
                        zf_mix<N, true, kPB>(v, tab + 2 * N * kPB, tab + 3 * N * kPB);
                    else
                        zf_mix<N, false, kPB>(v, tab, tab + N * kPB);
                }
            }
            if (table) {
                __syncthreads();  // the last group's tables are no longer read
                if (FARS && a.far) {
                    const long long q = (long long)grp * kPB + 2 * lane;
                    if (q < a.plane)
                        for (int j = warp; j <= Z; j += kWarps)
                            cp_async16(wfar + j * kPB + 2 * lane, w + (long long)(Z - 1 + j) * a.plane + q);
                    cp_async_wait();
                }
                float scale = 1.0f / (2 * N);
                if (a.fresp) scale *= a.fresp[pc];
                float2 *o = tab + (half * 2 + kind) * N * kPB;
#pragma unroll
                for (int k = 0; k < N; ++k) o[k * kPB] = pmul(v[k], scale);
                __syncthreads();
                // the next group's z kernel into L2
                const long long q = (long long)(grp + gridDim.x) * kPB + 16 * (lane & 3);
                if (q < a.plane)
                    for (int d = threadIdx.x >> 2; d < a.Zp; d += kWarps * 8)
                        asm volatile("prefetch.global.L2 [%0];" ::"l"(w + (long long)d * a.plane + q));
                continue;
            }
            // the even frequencies' warp finishes the first planes, the odd
            // ones' (which have the twiddles) the others: each hands over the
            // other's
            constexpr int M = 3 * N / 5;
            if (!active) continue;
            if (half) {
#pragma unroll
                for (int i = 0; i < M; ++i)
                    buf[i * 32] = cmul(make_float2(unit_root<N>(i).x, unit_root<N>(i).y), make_float2(v[i].y, v[i].x));
            } else {
#pragma unroll
                for (int i = M; i < N; ++i) buf[i * 32] = make_float2(v[i].y, v[i].x);
            }
            pair_sync(pair);
            const float g = a.fresp ? a.fresp[pc] : 1.f;
            const float2 g0 = pmul(e0, g), g1 = pmul(e1, g);
            const float2 *fp = wfar + sub * 32 + lane;
            char *yp = reinterpret_cast<char *>(S + (long long)t * Z * a.plane + pc);
            auto finish = [&](int i, float2 y, float2 &near) {
                if (a.far) {
                    const float2 next = FARS ? fp[(i + 1) * kPB] : wrow(i + Z);
                    y = cfma(g0, next, y);
                    y = cfma(g1, near, y);
                    near = next;
                }
                if (p < a.plane) *reinterpret_cast<float2 *>(yp + (unsigned)i * pb8) = y;
            };
            if (half) {
                float2 near = a.far ? FARS ? fp[M * kPB] : wrow(M + Z - 1) : make_float2(0.f, 0.f);
#pragma unroll
                for (int i = M; i < N; ++i)
                    if (i < LO || i < Z)
                        finish(i, cfma(make_float2(unit_root<N>(i).x, unit_root<N>(i).y), make_float2(v[i].y, v[i].x),
                                       buf[i * 32]), near);
            } else {
                float2 near = a.far ? FARS ? fp[0] : wrow(Z - 1) : make_float2(0.f, 0.f);
#pragma unroll
                for (int i = 0; i < M; ++i) finish(i, padd(make_float2(v[i].y, v[i].x), buf[i * 32]), near);
            }
        }
        // a warp without a tile in the last round would run the next tables' code
        // between the others' rounds, and both would wait for instructions
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// A z kernel per tile (or few tiles): the pair of warps makes its own tables.  An
// item is a tile and 32 frequencies; a warp does its half of both generators, of
// the planes and of the inverse one after the other, with its tables in its own
// rows of shared memory.  The CTA's pairs start their items together (see above).
// Bound like the other kernel, with the loads of the z kernel exposed besides: 16
// tiles of 300 at Z = 37 take 1.16 ms (1.89 with the direct sum; their 3.0 GB a
// copy's 0.45).
// ---------------------------------------------------------------------------
constexpr size_t zt_warp(int n) { return sizeof(float2) * 2 * n * 32; }
constexpr int zt_warps(int n) { return n <= 45 ? 8 : 6; }
constexpr size_t zt_smem(int n) { return zt_warps(n) * zt_warp(n) + zt_warps(n) / 2 * zf_buffer(n); }

template <int N>
__global__ void __launch_bounds__(zt_warps(N) * 32, 1)
k_zfft_tiles(float2 *__restrict__ S, const float2 *__restrict__ w, long long wstride, int t0, int npsf, const ZfArgs a) {
    constexpr int LO = zf_low(N), W = zt_warps(N), NP = W / 2;
    extern __shared__ __align__(16) unsigned char zf_smem[];
    const int Z = a.Z, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int half = warp / NP, pair = warp % NP;
    float2 *tab = reinterpret_cast<float2 *>(zf_smem + warp * zt_warp(N)) + lane;
    float2 *xbuf = reinterpret_cast<float2 *>(zf_smem + W * zt_warp(N)) + pair * N * 32, *buf = xbuf + lane;
    const unsigned pb8 = (unsigned)a.plane * 8u;  // bytes of a plane (checked by the launcher)
    const long long total = (long long)a.ngroups * a.nt;
    for (long long first = (long long)blockIdx.x * NP; first < total; first += (long long)gridDim.x * NP) {
        __syncthreads();
        const long long item = first + pair;
        if (item >= total) continue;
        const int t = (int)(item / a.ngroups), grp = (int)(item - (long long)t * a.ngroups);
        const long long p = (long long)grp * 32 + lane, pc = p < a.plane ? p : a.plane - 1;
        const char *wp = reinterpret_cast<const char *>(w + (npsf > 1 ? (t0 + t) * wstride : 0) + pc);
        auto wrow = [&](int row) { return __ldg(reinterpret_cast<const float2 *>(wp + (unsigned)row * pb8)); };
        const float g = a.fresp ? a.fresp[pc] : 1.f;
        float2 v[N], e0, e1;
#pragma unroll 1
        for (int step = 0; step < 4; ++step) {
            if (step < 2) {
                pair_sync(pair);  // the buffer has been read
                zf_generator<N>(v, step, half, wp, pb8, a, buf, pair);
                if (step == 1) {
                    pair_sync(pair);
                    // the tile's planes, 16 bytes (two frequencies) per copy; past
                    // the last frequency nothing (not stored either)
                    const long long q = (long long)grp * 32 + 2 * (lane & 15);
                    if (q < a.plane) {
                        const float2 *src = S + (long long)t * Z * a.plane + q;
                        for (int j = half * 2 + (lane >> 4); j < Z; j += 4)
                            cp_async16(xbuf + j * 32 + 2 * (lane & 15), src + (long long)j * a.plane);
                    }
                }
            } else if (step == 2) {
                cp_async_wait();
                pair_sync(pair);
#pragma unroll
                for (int j = 0; j < N; ++j) v[j] = j < LO || j < Z ? buf[j * 32] : make_float2(0.f, 0.f);
                // the ends halved (planes past the last are zero)
                e0 = pmul(v[0], 0.5f);
                e1 = pmul(buf[(Z - 1) * 32], 0.5f);
                v[0] = e0;
#pragma unroll
                for (int j = LO - 1; j < N; ++j) v[j] = pmul(v[j], j < Z - 1 ? 1.f : 0.5f);
            }
            if (half && step < 3) {
#pragma unroll
                for (int j = 1; j < N; ++j) v[j] = cmul(v[j], make_float2(unit_root<N>(j).x, -unit_root<N>(j).y));
            }
            zdft<N, false>(v);
            if (step < 2) {
                const float scale = g * (1.0f / (2 * N));
                float2 *o = tab + step * N * 32;
#pragma unroll
                for (int k = 0; k < N; ++k) o[k * 32] = pmul(v[k], scale);
            } else if (step == 2) {
                if (half)
                    zf_mix<N, true, 32>(v, tab, tab + N * 32);
                else
                    zf_mix<N, false, 32>(v, tab, tab + N * 32);
            }
        }
        constexpr int M = 3 * N / 5;
        pair_sync(pair);  // the planes have been read
        if (half) {
#pragma unroll
            for (int i = 0; i < M; ++i)
                buf[i * 32] = cmul(make_float2(unit_root<N>(i).x, unit_root<N>(i).y), make_float2(v[i].y, v[i].x));
        } else {
#pragma unroll
            for (int i = M; i < N; ++i) buf[i * 32] = make_float2(v[i].y, v[i].x);
        }
        pair_sync(pair);
        const float2 g0 = pmul(e0, g), g1 = pmul(e1, g);
        char *yp = reinterpret_cast<char *>(S + (long long)t * Z * a.plane + pc);
        auto finish = [&](int i, float2 y, float2 &near) {
            if (a.far) {
                const float2 next = wrow(i + Z);
                y = cfma(g0, next, y);
                y = cfma(g1, near, y);
                near = next;
            }
            if (p < a.plane) *reinterpret_cast<float2 *>(yp + (unsigned)i * pb8) = y;
        };
        if (half) {
            float2 near = a.far ? wrow(M + Z - 1) : make_float2(0.f, 0.f);
#pragma unroll
            for (int i = M; i < N; ++i)
                if (i < LO || i < Z)
                    finish(i, cfma(make_float2(unit_root<N>(i).x, unit_root<N>(i).y), make_float2(v[i].y, v[i].x), buf[i * 32]),
                           near);
        } else {
            float2 near = a.far ? wrow(Z - 1) : make_float2(0.f, 0.f);
#pragma unroll
            for (int i = 0; i < M; ++i) finish(i, padd(make_float2(v[i].y, v[i].x), buf[i * 32]), near);
        }
    }
}

template <int N>
int zt_launch(float2 *S, const float2 *w, long long wstride, int t0, int npsf, const ZfArgs &args_in, cudaStream_t st) {
    ZfArgs a = args_in;
    const void *fn = (const void *)k_zfft_tiles<N>;
    if (int rc = mm_set_smem(fn, zt_smem(N))) return rc;
    a.ngroups = (int)((a.plane + 31) / 32);
    const long long ctas = ((long long)a.ngroups * a.nt + zt_warps(N) / 2 - 1) / (zt_warps(N) / 2);
    const int grid = ctas < mm_sm_count() ? (int)ctas : mm_sm_count();
    void *args[] = {&S, &w, &wstride, &t0, &npsf, &a};
    MM_CUDA_TRY(cudaLaunchKernel(fn, dim3(grid), dim3(zt_warps(N) * 32), args, zt_smem(N), st));
    mm_launch_counter_add();
    return MM_OK;
}

template <int N>
int zf_launch(float2 *S, const float2 *w, const ZfArgs &args_in, cudaStream_t st) {
    ZfArgs a = args_in;
    const void *fn = (const void *)k_zfft_apply<N>;
    const size_t sm = zf_tables(N) + kWarps * zf_buffer(N) + zf_far(N);
    if (int rc = mm_set_smem(fn, sm)) return rc;
    a.ngroups = (int)((a.plane + kPB - 1) / kPB);
    const int grid = a.ngroups < mm_sm_count() ? a.ngroups : mm_sm_count();
    void *args[] = {&S, &w, &a};
    MM_CUDA_TRY(cudaLaunchKernel(fn, dim3(grid), dim3(kWarps * 32), args, sm, st));
    mm_launch_counter_add();
    return MM_OK;
}

int zf_length(int Z, int zpad) {
    if (Z < kZfMinZ || (zpad != Z - 1 && 2 * zpad != Z - 2)) return 0;
    for (int n : {30, 35, 40, 45, 50, 56})
        if (Z <= n) return n;
    return 0;
}

}  // namespace

int mm_zfft_supported(int Z, int zpad, int nt, long long plane, const void *w) {
    // 16-byte copies of two frequencies, and byte offsets of a column's planes
    // in 32 bits
    return nt >= 1 && plane % 2 == 0 && ((uintptr_t)w & 15) == 0 && plane * 8 * (Z + 2 * zpad) < (1LL << 32) &&
                   zf_length(Z, zpad)
               ? 1
               : 0;
}

int mm_launch_zfft_apply(float2 *S, const float2 *w, int Z, int zpad, int Zp, long long plane, int nt,
                         const float *fresp, cudaStream_t st) {
    MM_REQUIRE(Zp == Z + 2 * zpad && mm_zfft_supported(Z, zpad, nt, plane, w), "z operator: depth %d, padding %d", Z, zpad);
    ZfArgs a = {};
    a.Z = Z;
    a.Zp = Zp;
    a.nt = nt;
    a.far = zpad == Z - 1;
    a.plane = plane;
    a.fresp = fresp;
    switch (zf_length(Z, zpad)) {
        case 30: return zf_launch<30>(S, w, a, st);
        case 35: return zf_launch<35>(S, w, a, st);
        case 40: return zf_launch<40>(S, w, a, st);
        case 45: return zf_launch<45>(S, w, a, st);
        case 56: return zf_launch<56>(S, w, a, st);
        case 50: return zf_launch<50>(S, w, a, st);
    }
    return MM_EINVAL;
}

int mm_launch_zfft_tiles(float2 *S, const float2 *w, long long wstride, int Z, int zpad, int Zp, long long plane, int t0,
                         int nt, int npsf, const float *fresp, cudaStream_t st) {
    MM_REQUIRE(Zp == Z + 2 * zpad && wstride % 2 == 0 && mm_zfft_supported(Z, zpad, nt, plane, w),
               "z operator: depth %d, padding %d", Z, zpad);
    ZfArgs a = {};
    a.Z = Z;
    a.Zp = Zp;
    a.nt = nt;
    a.far = zpad == Z - 1;
    a.plane = plane;
    a.fresp = fresp;
    switch (zf_length(Z, zpad)) {
        case 30: return zt_launch<30>(S, w, wstride, t0, npsf, a, st);
        case 35: return zt_launch<35>(S, w, wstride, t0, npsf, a, st);
        case 40: return zt_launch<40>(S, w, wstride, t0, npsf, a, st);
        case 45: return zt_launch<45>(S, w, wstride, t0, npsf, a, st);
        case 50: return zt_launch<50>(S, w, wstride, t0, npsf, a, st);
        case 56: return zt_launch<56>(S, w, wstride, t0, npsf, a, st);
    }
    return MM_EINVAL;
}
