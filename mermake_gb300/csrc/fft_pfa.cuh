// The transform engine of the two padded lengths the reference's tile sizes
// give (678 = 6 x 113: tile 500, overlap 89; 478 = 2 x 239: tile 300), 16 lines
// per CTA, as prime-factor transforms: no twiddle factor anywhere.
//
// N = C R with C and R coprime and R prime.  With n = (R n1 + C n2) mod N and
// k = k1 (mod C), k2 (mod R), W_N^(n k) = W_C^(n1 k1) W_R^(n2 k2): C-point
// transforms over n1 and R-point transforms over n2 (Good 1958, Thomas 1963).
// The R-point one is Rader's cyclic convolution of length M = R - 1 (g a
// primitive root: n2 = g^-q, k2 = g^m, y[g^m] = x[0] + sum_q x[g^-q] w^(g^(m-q))),
// and M = N1 N2 is a coprime product again (112 = 16 x 7, 238 = 14 x 17), so
// the convolution is two-dimensional over q = (q mod N1, q mod N2):
//   1. a thread (q1, line) takes the C N2 inputs of its q1, does the C-point
//      transforms over n1 and the N2-point transforms over q2, and leaves
//      T[k1][q1][a2];
//   2. per (k1, a2, line): the N1-point transform over q1, the product with
//      the transform H of w^(g^s) / M, the inverse N1-point transform, in place.
//      x[0] enters as an addition to the a1 = a2 = 0 coefficient, and
//      y[0] = x[0] + sum u is that coefficient before the product plus x[0];
//   3. a thread (q1, line): the inverse N2-point transform over a2 gives the
//      outputs k = (k1, g^(q1, q2)).
// All index maps are tables (fft_plan.cu), so a value costs one shared-memory
// write and read per phase boundary and one fused multiply-add of address
// arithmetic at each end.
//
// Complex sums, differences and products with a real constant are issued as
// packed pairs (add/sub/mul/fma.rn.f32x2: one instruction for the real and the
// imaginary part, the same rounding as two).
#pragma once
#include "fft.cuh"

constexpr int kPfaNL = 16;  // lines of a CTA: 128 bytes per element across the lines

template <int N>
struct Pfa;
template <>
struct Pfa<678> {
    static constexpr int R = 113, C = 6, N1 = 16, N2 = 7;
};
template <>
struct Pfa<478> {
    static constexpr int R = 239, C = 2, N1 = 14, N2 = 17;
};
template <int N>
struct PfaK {
    static constexpr int R = Pfa<N>::R, C = Pfa<N>::C, N1 = Pfa<N>::N1, N2 = Pfa<N>::N2;
    static constexpr int M = R - 1;
    static constexpr int threads = N1 * kPfaNL;
    static constexpr int vals = C * N2;               // a thread's values in phases 1 and 3
    static constexpr int ipad = pfa_ipad(vals);       // its index-table row
    static constexpr int trows = C * M;               // rows of T (16 float2 each)
    static constexpr int tab_ints = 2 * N1 * ipad + 2 * 8;  // in, out, then the inputs of n2 = 0 and outputs of k2 = 0
    static_assert(N == C * R && M == N1 * N2, "prime-factor split");
};

// ---- packed arithmetic ----------------------------------------------------
__device__ __forceinline__ float2 padd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 psub(float2 a, float2 b) {
    float2 d;
    asm("{\n\t.reg .b64 x, y, z;\n\t"
        "mov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\t"
        "sub.rn.f32x2 z, x, y;\n\t"
        "mov.b64 {%0, %1}, z;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
__device__ __forceinline__ float2 pmul(float2 a, float s) { return __fmul2_rn(a, make_float2(s, s)); }
__device__ __forceinline__ float2 pfma(float2 a, float s, float2 c) { return __ffma2_rn(a, make_float2(s, s), c); }
// a + i s b and a - i s b (s real)
__device__ __forceinline__ float2 paxpi(float2 a, float s, float2 b) {
    return make_float2(fmaf(-s, b.y, a.x), fmaf(s, b.x, a.y));
}
__device__ __forceinline__ float2 paddi(float2 a, float2 b) { return make_float2(a.x - b.y, a.y + b.x); }
__device__ __forceinline__ float2 psubi(float2 a, float2 b) { return make_float2(a.x + b.y, a.y - b.x); }

// DFT kernels, natural order in and out; sign -1 (INV false) or +1
template <bool INV>
__device__ __forceinline__ void pdft3(float2 &v0, float2 &v1, float2 &v2) {
    constexpr float s = INV ? 0.86602540378443864676f : -0.86602540378443864676f;
    const float2 a = padd(v1, v2), b = psub(v1, v2);
    const float2 t = pfma(a, -0.5f, v0);
    v0 = padd(v0, a);
    v1 = paxpi(t, s, b);
    v2 = paxpi(t, -s, b);
}
// 6 = 2 x 3 (prime-factor order: inputs (3a + 2b) mod 6, outputs by residues)
template <bool INV>
__device__ __forceinline__ void pdft6(float2 &v0, float2 &v1, float2 &v2, float2 &v3, float2 &v4, float2 &v5) {
    float2 s0 = padd(v0, v3), s1 = padd(v2, v5), s2 = padd(v4, v1);
    float2 d0 = psub(v0, v3), d1 = psub(v2, v5), d2 = psub(v4, v1);
    pdft3<INV>(s0, s1, s2);
    pdft3<INV>(d0, d1, d2);
    v0 = s0;
    v4 = s1;
    v2 = s2;
    v3 = d0;
    v1 = d1;
    v5 = d2;
}
// cos(2 pi m / R) and sin(2 pi m / R) for the odd lengths
template <int R>
struct PfaTrig;
template <>
struct PfaTrig<7> {
    __device__ static constexpr float c(int m) {
        constexpr float t[4] = {1.f, 0.62348980185873353053f, -0.22252093395631440429f, -0.90096886790241912624f};
        return t[m];
    }
    __device__ static constexpr float s(int m) {
        constexpr float t[4] = {0.f, 0.78183148246802980871f, 0.97492791218182360702f, 0.43388373911755812048f};
        return t[m];
    }
};
template <>
struct PfaTrig<17> {
    __device__ static constexpr float c(int m) {
        constexpr float t[9] = {1.f,
                                0.93247222940435580457f,
                                0.73900891722065911592f,
                                0.44573835577653826740f,
                                0.09226835946330199524f,
                                -0.27366299007208286354f,
                                -0.60263463637925638918f,
                                -0.85021713572961421569f,
                                -0.98297309968390177828f};
        return t[m];
    }
    __device__ static constexpr float s(int m) {
        constexpr float t[9] = {0.f,
                                0.36124166618715294874f,
                                0.67369564364655721171f,
                                0.89516329135506232207f,
                                0.99573417629503452190f,
                                0.96182564317281907043f,
                                0.79801722728023950333f,
                                0.52643216287735580027f,
                                0.18374951781657033158f};
        return t[m];
    }
};
template <int R, bool INV>
__device__ __forceinline__ void pdft_odd(float2 *v) {
    constexpr int H = (R - 1) / 2;
    float2 a[H], b[H];
#pragma unroll
    for (int r = 1; r <= H; ++r) {
        a[r - 1] = padd(v[r], v[R - r]);
        b[r - 1] = psub(v[r], v[R - r]);
    }
    const float2 x0 = v[0];
    float2 s0 = x0;
#pragma unroll
    for (int r = 0; r < H; ++r) s0 = padd(s0, a[r]);
    v[0] = s0;
#pragma unroll
    for (int k = 1; k <= H; ++k) {
        float2 A = x0, B;
#pragma unroll
        for (int r = 1; r <= H; ++r) {
            const int m = (r * k) % R;
            const float c = m <= H ? PfaTrig<R>::c(m) : PfaTrig<R>::c(R - m);
            const float s = m <= H ? PfaTrig<R>::s(m) : -PfaTrig<R>::s(R - m);
            A = pfma(a[r - 1], c, A);
            B = r == 1 ? pmul(b[0], s) : pfma(b[r - 1], s, B);
        }
        // A -+ i B
        v[k] = INV ? paddi(A, B) : psubi(A, B);
        v[R - k] = INV ? psubi(A, B) : paddi(A, B);
    }
}
template <bool INV>
__device__ __forceinline__ void pdft4(float2 &v0, float2 &v1, float2 &v2, float2 &v3) {
    const float2 s02 = padd(v0, v2), d02 = psub(v0, v2), s13 = padd(v1, v3), d13 = psub(v1, v3);
    v0 = padd(s02, s13);
    v2 = psub(s02, s13);
    v1 = INV ? paddi(d02, d13) : psubi(d02, d13);
    v3 = INV ? psubi(d02, d13) : paddi(d02, d13);
}
// multiply by (r, +-r) / (-r, +-r), r = sqrt(1/2): w8 and w8^3 of the direction
template <bool INV>
__device__ __forceinline__ float2 pw8(float2 a) {
    return pmul(INV ? make_float2(a.x - a.y, a.x + a.y) : make_float2(a.x + a.y, a.y - a.x), 0.70710678118654752440f);
}
template <bool INV>
__device__ __forceinline__ float2 pw8_3(float2 a) {
    return pmul(INV ? make_float2(-a.x - a.y, a.x - a.y) : make_float2(a.y - a.x, -a.x - a.y),
                0.70710678118654752440f);
}
template <bool INV>
__device__ __forceinline__ void pdft16(float2 *v) {
    constexpr float c1 = 0.92387953251128675613f, s1 = 0.38268343236508977173f, sg = INV ? 1.f : -1.f;
#pragma unroll
    for (int n = 0; n < 4; ++n) pdft4<INV>(v[n], v[n + 4], v[n + 8], v[n + 12]);
    // v[n1 + 4 k1] times w16^(n1 k1)
    v[5] = cmul(v[5], make_float2(c1, sg * s1));
    v[9] = pw8<INV>(v[9]);
    v[13] = cmul(v[13], make_float2(s1, sg * c1));
    v[6] = pw8<INV>(v[6]);
    v[10] = mul_i<INV>(v[10]);
    v[14] = pw8_3<INV>(v[14]);
    v[7] = cmul(v[7], make_float2(s1, sg * c1));
    v[11] = pw8_3<INV>(v[11]);
    v[15] = cmul(v[15], make_float2(-c1, -sg * s1));
    float2 o[16];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        float2 t0 = v[4 * k], t1 = v[4 * k + 1], t2 = v[4 * k + 2], t3 = v[4 * k + 3];
        pdft4<INV>(t0, t1, t2, t3);
        o[k] = t0;
        o[k + 4] = t1;
        o[k + 8] = t2;
        o[k + 12] = t3;
    }
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = o[k];
}
// 14 = 2 x 7: inputs (7a + 2b) mod 14, outputs by residues
template <bool INV>
__device__ __forceinline__ void pdft14(float2 *v) {
    float2 s[7], d[7];
#pragma unroll
    for (int b = 0; b < 7; ++b) {
        s[b] = padd(v[2 * b], v[(7 + 2 * b) % 14]);
        d[b] = psub(v[2 * b], v[(7 + 2 * b) % 14]);
    }
    pdft_odd<7, INV>(s);
    pdft_odd<7, INV>(d);
#pragma unroll
    for (int b = 0; b < 7; ++b) {
        v[b % 2 == 0 ? b : b + 7] = s[b];  // even output congruent to b mod 7
        v[b % 2 == 1 ? b : b + 7] = d[b];  // odd output congruent to b mod 7
    }
}
template <int L, bool INV>
__device__ __forceinline__ void pdft(float2 *v) {
    if constexpr (L == 16)
        pdft16<INV>(v);
    else if constexpr (L == 14)
        pdft14<INV>(v);
    else
        pdft_odd<L, INV>(v);
}

// ---- the three phases -----------------------------------------------------
// A CTA's shared memory: T (or a kernel's own line buffer in the same place),
// the x[0] sums, the y[0] outputs, H and the index tables.
template <int N>
struct PfaSmem {
    float2 *T, *x0, *y0, *H;
    int *tin, *tout;   // rows of ipad indices per q1
    int *in0, *out0;   // the C inputs of n2 = 0, the C outputs of k2 = 0
};
// bytes after the line buffer of `rows` rows of `stride` float2
template <int N>
constexpr size_t pfa_tail_bytes() {
    using K = PfaK<N>;
    return sizeof(float2) * (2 * K::C * kPfaNL + K::M) + sizeof(int) * K::tab_ints;
}
template <int N>
__device__ __forceinline__ PfaSmem<N> pfa_layout(unsigned char *base, size_t line_bytes) {
    using K = PfaK<N>;
    PfaSmem<N> s;
    s.T = reinterpret_cast<float2 *>(base);
    s.H = reinterpret_cast<float2 *>(base + line_bytes);
    s.x0 = s.H + K::M;
    s.y0 = s.x0 + K::C * kPfaNL;
    s.tin = reinterpret_cast<int *>(s.y0 + K::C * kPfaNL);
    s.tout = s.tin + K::N1 * K::ipad;
    s.in0 = s.tout + K::N1 * K::ipad;
    s.out0 = s.in0 + 8;
    return s;
}
// tables of the plan into shared memory (all threads; a barrier must follow)
template <int N, bool INV>
__device__ __forceinline__ void pfa_load_tables(const PfaSmem<N> &s, const FftPlan &P) {
    using K = PfaK<N>;
    const float2 *h = P.pfa_h + (INV ? K::M : 0);
    for (int i = threadIdx.x; i < K::M; i += K::threads) s.H[i] = h[i];
    for (int i = threadIdx.x; i < K::tab_ints; i += K::threads) s.tin[i] = P.pfa_idx[i];
}

// phase 1 arithmetic: v[n1][q2] -> v[k1][a2]
template <int N, bool INV>
__device__ __forceinline__ void pfa_first(float2 (&v)[PfaK<N>::C][PfaK<N>::N2]) {
    using K = PfaK<N>;
#pragma unroll
    for (int q = 0; q < K::N2; ++q) {
        if constexpr (K::C == 6) {
            pdft6<INV>(v[0][q], v[1][q], v[2][q], v[3][q], v[4][q], v[5][q]);
        } else {
            const float2 a = v[0][q], b = v[1][q];
            v[0][q] = padd(a, b);
            v[1][q] = psub(a, b);
        }
    }
#pragma unroll
    for (int k = 0; k < K::C; ++k) pdft<K::N2, false>(v[k]);
}
template <int N, bool INV>
__device__ __forceinline__ void pfa_dft_c(float2 (&x)[PfaK<N>::C]) {
    if constexpr (PfaK<N>::C == 6) {
        pdft6<INV>(x[0], x[1], x[2], x[3], x[4], x[5]);
    } else {
        const float2 a = x[0], b = x[1];
        x[0] = padd(a, b);
        x[1] = psub(a, b);
    }
}
template <int N>
__device__ __forceinline__ void pfa_put(const PfaSmem<N> &s, const float2 (&v)[PfaK<N>::C][PfaK<N>::N2], int q1, int l) {
    using K = PfaK<N>;
#pragma unroll
    for (int k = 0; k < K::C; ++k)
#pragma unroll
        for (int a = 0; a < K::N2; ++a) s.T[((k * K::N1 + q1) * K::N2 + a) * kPfaNL + l] = v[k][a];
}
// phase 2, in place; y0[k1][l] gets the output k2 = 0
template <int N>
__device__ __forceinline__ void pfa_middle(const PfaSmem<N> &s, int q1, int l) {
    using K = PfaK<N>;
    for (int r = q1; r < K::vals; r += K::N1) {
        const int k1 = r / K::N2, a2 = r - k1 * K::N2;
        float2 *t = s.T + (k1 * K::N1 * K::N2 + a2) * kPfaNL + l;
        float2 v[K::N1];
#pragma unroll
        for (int a = 0; a < K::N1; ++a) v[a] = t[a * K::N2 * kPfaNL];
        pdft<K::N1, false>(v);
        float2 x0 = make_float2(0.f, 0.f);
        if (a2 == 0) {
            x0 = s.x0[k1 * kPfaNL + l];
            s.y0[k1 * kPfaNL + l] = padd(x0, v[0]);
        }
        const float4 *h = reinterpret_cast<const float4 *>(s.H + a2 * K::N1);
#pragma unroll
        for (int a = 0; a < K::N1; a += 2) {
            const float4 w = h[a / 2];
            v[a] = cmul(v[a], make_float2(w.x, w.y));
            v[a + 1] = cmul(v[a + 1], make_float2(w.z, w.w));
        }
        v[0] = padd(v[0], x0);
        pdft<K::N1, true>(v);
#pragma unroll
        for (int a = 0; a < K::N1; ++a) t[a * K::N2 * kPfaNL] = v[a];
    }
}
// phase 3 of one k1: v[q2] = output (k1, g^(q1, q2))
template <int N>
__device__ __forceinline__ void pfa_last(const PfaSmem<N> &s, int k1, int q1, int l, float2 (&v)[PfaK<N>::N2]) {
    using K = PfaK<N>;
    const float2 *t = s.T + (k1 * K::N1 + q1) * K::N2 * kPfaNL + l;
#pragma unroll
    for (int a = 0; a < K::N2; ++a) v[a] = t[a * kPfaNL];
    pdft<K::N2, true>(v);
}

// ---- dynamic group order --------------------------------------------------
// The persistent CTAs take groups from a counter: SMs finish a group at
// different speeds (on 8 tiles of 678 the static order left the SMs active
// 85 % of the pass on average, the slowest all of it).  queue: two words of
// the context's scratch, zero between launches (the last CTA resets them);
// NULL: every gridDim.x-th group.  Thread 0 asks at a group's start and
// publishes the answer before a later barrier of the group.
__device__ __forceinline__ int queue_ask(unsigned *queue, int grp) {
    return queue ? (int)(gridDim.x + atomicAdd(queue, 1u)) : grp + (int)gridDim.x;
}
__device__ __forceinline__ void queue_leave(unsigned *queue) {
    if (!queue) return;
    __threadfence();
    if (atomicAdd(queue + 1, 1u) == gridDim.x - 1) queue[0] = queue[1] = 0;
}
