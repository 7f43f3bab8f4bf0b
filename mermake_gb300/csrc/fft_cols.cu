// x pass of the tiled deconvolution, and the engine's general strided
// transform: in-place complex FFT along a strided axis (forward or inverse).
#include "deconv.cuh"
#include "fft_pfa.cuh"

namespace {
constexpr FftCfg kColsCfg = kFftPair;

// ---------------------------------------------------------------------------
// strided complex FFT, in place: line l of plane p starts at S + p*plane_stride + l,
// element e at + e*se.  Lines are contiguous, so a CTA's loads are runs of nl,
// staged into shared memory with cp.async.  (Lengths other than 678 and 478.)
// ---------------------------------------------------------------------------
template <bool INV, int LMAX>
__global__ void __launch_bounds__(kColsCfg.threads, kColsCfg.ctas)
k_cols(float2 *__restrict__ S, long long se, int nlines, long long plane_stride, FftPlan P, int nl, int gx,
       int ngroups) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int n = P.n, lnl = log2_pow2(nl);
    const FftSmem L = fft_smem_layout(smem_raw, P, nl);
    fft_load_tables(P, L.tw, L.tab);
    // persistent: the CTAs walk the groups of nl lines (tables loaded once)
    for (int grp = blockIdx.x; grp < ngroups; grp += gridDim.x) {
        const int by = grp / gx, bx = grp - by * gx;
        float2 *base = S + (long long)by * plane_stride;
        const int l0 = bx * nl;
        for (int it = threadIdx.x; it < nl * n; it += blockDim.x) {
            const int l = it & (nl - 1), e = it >> lnl;
            if (l0 + l < nlines)
                cp_async8(&L.A[sidx(e, l, nl)], &base[e * se + l0 + l]);
            else
                L.A[sidx(e, l, nl)] = make_float2(0.f, 0.f);
        }
        cp_async_wait_all();
        __syncthreads();
        float2 *R = fft_lines<INV, LMAX>(L.A, L.B, nl, P, L.tw, L.tab, L.scr);
        for (int it = threadIdx.x; it < nl * n; it += blockDim.x) {
            const int l = it & (nl - 1), e = it >> lnl;
            if (l0 + l < nlines) base[e * se + l0 + l] = R[sidx(e, l, nl)];
        }
        __syncthreads();  // the next group's loads overwrite the line buffers
    }
}

// The same for 678 and 478 points (fft_pfa.cuh).  A thread (q1, line) loads its
// inputs from global memory straight into registers, all in flight at once (16
// lines: 128 contiguous bytes per element), and stores its outputs from
// registers, so shared memory holds only what the phases exchange (T, one
// write and one read per phase boundary).  The lines of all planes are
// numbered through, so a group may span two planes and only the last one of
// the launch is ragged.
template <int N, bool INV>
__global__ void __launch_bounds__(PfaK<N>::threads, 2)
k_cols_pfa(float2 *__restrict__ S, unsigned se8, int nlines, long long plane_stride, int total, int ngroups,
           FftPlan P, unsigned *__restrict__ queue) {
    using K = PfaK<N>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int next;
    const PfaSmem<N> s = pfa_layout<N>(smem_raw, sizeof(float2) * K::trows * kPfaNL);
    pfa_load_tables<N, INV>(s, P);
    __syncthreads();
    const int l = threadIdx.x % kPfaNL, q1 = threadIdx.x / kPfaNL;
    for (int grp = blockIdx.x; grp < ngroups;) {
        const int asked = threadIdx.x == 0 ? queue_ask(queue, grp) : 0;
        // a line past the last one loads the last one and stores nothing
        const int line = min(grp * kPfaNL + l, total - 1);
        const bool mine = grp * kPfaNL + l < total;
        const int plane = line / nlines;
        char *base = reinterpret_cast<char *>(S + plane * plane_stride + (line - plane * nlines));
        auto at = [&](int e) { return reinterpret_cast<float2 *>(base + (unsigned long long)(unsigned)e * se8); };
        float2 v[K::C][K::N2], x0[K::C];
        {
            const int4 *ip = reinterpret_cast<const int4 *>(s.tin + q1 * K::ipad);
#pragma unroll
            for (int c = 0; c < K::ipad / 4; ++c) {
                const int4 i4 = ip[c];
                const int e[4] = {i4.x, i4.y, i4.z, i4.w};
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (4 * c + u < K::vals) v[(4 * c + u) / K::N2][(4 * c + u) % K::N2] = __ldcg(at(e[u]));
            }
        }
        if (q1 == 0) {
#pragma unroll
            for (int c = 0; c < K::C; ++c) x0[c] = __ldcg(at(s.in0[c]));
        }
        pfa_first<N, INV>(v);
        if (q1 == 0) {
            pfa_dft_c<N, INV>(x0);
#pragma unroll
            for (int c = 0; c < K::C; ++c) s.x0[c * kPfaNL + l] = x0[c];
        }
        __syncthreads();  // T is free: the previous group's last phase has read it
        pfa_put<N>(s, v, q1, l);
        if (threadIdx.x == 0) next = asked;
        __syncthreads();
        grp = next;
        if (grp < ngroups) {
            // the next group's 128-byte runs into L2, so that its loads wait
            // for L2 only
            const int n0 = grp * kPfaNL, pl = n0 / nlines;
            const char *nb = reinterpret_cast<const char *>(S + pl * plane_stride + (n0 - pl * nlines));
            for (int e = threadIdx.x; e < N; e += K::threads)
                asm volatile("prefetch.global.L2 [%0];" ::"l"(nb + (unsigned long long)(unsigned)e * se8));
        }
        pfa_middle<N>(s, q1, l);
        __syncthreads();
        const int *op = s.tout + q1 * K::ipad;
#pragma unroll
        for (int c = 0; c < K::C; ++c) {
            float2 y[K::N2];
            pfa_last<N>(s, c, q1, l, y);
#pragma unroll
            for (int q = 0; q < K::N2; ++q)
                if (mine) *at(op[c * K::N2 + q]) = y[q];
        }
        if (q1 == 0 && mine) {
#pragma unroll
            for (int c = 0; c < K::C; ++c) *at(s.out0[c]) = s.y0[c * kPfaNL + l];
        }
    }
    if (threadIdx.x == 0) queue_leave(queue);
}

template <int N>
int launch_pfa(float2 *S, unsigned se8, int nlines, long long plane_stride, int total, bool inv, const FftPlan &P,
               unsigned *queue, cudaStream_t st) {
    using K = PfaK<N>;
    const size_t sm = sizeof(float2) * K::trows * kPfaNL + pfa_tail_bytes<N>();
    int ngroups = mm_cdiv(total, kPfaNL);
    const void *fn = inv ? (const void *)k_cols_pfa<N, true> : (const void *)k_cols_pfa<N, false>;
    FftPlan Pa = P;
    void *args[] = {&S, &se8, &nlines, &plane_stride, &total, &ngroups, &Pa, &queue};
    return launch_fft_kernel(fn, dim3(fft_grid(ngroups, {K::threads, 2})), sm, st, args, K::threads);
}

}  // namespace

int mm_launch_cols(float2 *S, int n, long long se, int nlines, long long plane_stride, int nplanes, bool inv,
                   unsigned *queue, cudaStream_t st) {
    FftPlan P;
    int rc = mm_fft_plan_get(n, &P);
    if (rc) return rc;
    const long long total = (long long)nlines * nplanes;
    // element strides below 4 GB and a line count the kernel's ints hold
    if (P.pfa_idx && se * 8 < (1LL << 32) && total < (1LL << 31) - kPfaNL) {
        if (n == 678) return launch_pfa<678>(S, (unsigned)(se * 8), nlines, plane_stride, (int)total, inv, P, queue, st);
        return launch_pfa<478>(S, (unsigned)(se * 8), nlines, plane_stride, (int)total, inv, P, queue, st);
    }
    int nl = pick_nl(P, 16, kColsCfg);
    size_t sm = fft_smem(P, nl, kColsCfg);
    int gx = mm_cdiv(nlines, nl);
    int ngroups = gx * nplanes;
    // persistent: kColsCfg.ctas CTAs per SM (their line buffers fill its shared memory)
    dim3 grid(fft_grid(ngroups, kColsCfg));
    void *args[] = {&S, &se, &nlines, &plane_stride, &P, &nl, &gx, &ngroups};
    const void *fn = inv ? MM_BY_CLASS(P, k_cols, true,) : MM_BY_CLASS(P, k_cols, false,);
    return launch_fft_kernel(fn, grid, sm, st, args, kColsCfg.threads);
}
