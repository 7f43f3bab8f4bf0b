// z operator of one Wiener spectrum over a tile batch, with the matrix of each
// frequency formed in registers and the operands staged asynchronously (the
// kernel rows by TMA, the spectra by cp.async).
//
// Y[t][i][p] = sum_j M_p[i][j] X[t][j][p] (zop.cu has the derivation).  When
// 1 <= zpad <= Z - 1 every real plane j has at most three padded copies
// (mermake/deconvolver.py:145-148: itself, its reflection about zpad for
// 1 <= j <= zpad, and its reflection about zpad + Z - 1 for
// Z - 1 - zpad <= j <= Z - 2), so with w the z kernel (indices mod Zp)
//
//   M[i][j] = w[i - j] + [1 <= j <= zpad] w[i + j] + [Z-1-zpad <= j <= Z-2] w[i + j - 2Z + 2]:
//
// a Toeplitz matrix plus two masked Hankel matrices.  A thread owns rows
// i0 .. i0 + 4 of TT tiles; along j the direct values w[i - j] and the
// reflected ones slide by one place, so the thread keeps each in a register
// ring of five and loads one new direct value and the one or two reflected ones
// per column (with j unrolled by five the slots are compile-time constants).
// No matrix is stored: shared memory holds only the operands, X (nt x Z rows of
// PB frequencies, copied by cp.async) and the kernel rows w[-kA .. 2Z-2] (two
// TMA boxes of the (Zp, plane) kernel, the negative rows from its top; kA is
// 2Z - 2 rounded up to a multiple of four, so that both boxes land on 128-byte
// boundaries as tiled TMA requires), double buffered.  The persistent CTAs take
// groups of PB consecutive frequencies.  A producer warp issues each group's
// copies once the buffer is free; the compute warps take the group's work in
// warp-sized units from a shared counter, wait only for their buffer to fill
// (its "full" mbarrier completes with the copies: 32 cp.async arrivals and the
// TMA bytes) and release it with one arrive per unit on its "empty" mbarrier,
// so no CTA barrier separates the groups.  Every wait is bounded: a thread that
// gives up records the failure in *err and returns.
//
// Every output sums its columns in ascending order with the same products
// (k_zpt_apply's too), so a tile's result does not depend on the batch it is in.
//
// What bounds it: FP32 issue.  A product needs three register reads; at 25
// tiles, Z = 50 and P = 678 the 115 GFLOP of a launch take 2.69 ms (21.4 T
// products/s of the 40.3 T that 152 SMs have at 2.07 GHz; a loop of products
// with two new operands each reaches 33 T).
#include <cuda.h>
#include <cudaTypedefs.h>

#include <mutex>

#include "deconv.cuh"

namespace {

constexpr int kTI = 5;      // rows of a thread, and the unroll of the column loop
// threads of a CTA at most, and CTAs per SM that the registers are shared out for
constexpr int zth_ctas(int tt, int pb) { return tt == 5 && pb == 8 ? 1 : 2; }
constexpr int zth_max_threads(int tt, int pb) { return 512 / zth_ctas(tt, pb); }
constexpr unsigned kWaitPolls = 1u << 24;

__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t *bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
// true once the barrier's phase with this parity has completed; false after
// kWaitPolls polls
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, unsigned parity) {
    const unsigned a = smem_u32(bar);
    for (unsigned it = 0; it < kWaitPolls; ++it) {
        unsigned done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(a), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}
// 16 bytes global -> shared through L2, completion tracked per thread
__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
// one arrive on *bar (counted in its initial count) once this thread's
// earlier cp.async copies have landed
__device__ __forceinline__ void cp_async_arrive(uint64_t *bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, int c0, int c1, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            smem_u32(dst)),
        "l"(map), "r"(c0), "r"(c1), "r"(smem_u32(bar))
        : "memory");
}

// The accumulators of a thread's kTI rows x TT tiles
template <int TT>
struct ZthAcc {
    float2 v[kTI][TT];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int q = 0; q < kTI; ++q)
#pragma unroll
            for (int b = 0; b < TT; ++b) v[q][b] = make_float2(0.f, 0.f);
    }
    __device__ __forceinline__ void add(const float2 (&m)[kTI], const float2 (&x)[TT]) {
        // an operand of each product is the previous one's: with all operands
        // new, register reads bound the rate (a column of 25 products took 4 %
        // longer in row order, and 10 % with the two products of x[b].x apart)
#pragma unroll
        for (int b = 0; b < TT; ++b) {
#pragma unroll
            for (int q = 0; q < kTI; ++q) v[q][b].x = fmaf(m[q].x, x[b].x, v[q][b].x);
#pragma unroll
            for (int q = 0; q < kTI; ++q) v[q][b].y = fmaf(m[q].y, x[b].x, v[q][b].y);
#pragma unroll
            for (int q = 0; q < kTI; ++q) v[q][b].x = fmaf(-m[q].y, x[b].y, v[q][b].x);
#pragma unroll
            for (int q = 0; q < kTI; ++q) v[q][b].y = fmaf(m[q].x, x[b].y, v[q][b].y);
        }
    }
    __device__ __forceinline__ float2 get(int q, int b) const { return v[q][b]; }
};
struct ZthArgs {
    int Z, Zp, nt;
    int ntc;           // tiles of a chunk (the X box's height)
    int ntg;           // tile groups of TT a CTA computes (ceil(ntc / TT))
    int nchunks;       // chunks the batch's tiles are split into
    long long plane;
    int nitems;        // frequency groups (ceil(plane / PB)) x chunks
    int kA;            // staged row of w[0]: 2Z - 2 rounded up to a multiple of 4
    unsigned wbytesA;  // kernel rows -kA .. -1 (a multiple of 128 bytes)
    unsigned wbytesB;  // kernel rows 0 .. 2Z-2
    unsigned bufstride, woff;  // bytes per buffer, offset of the kernel rows in it
    unsigned zoff;     // bytes: the zero rows (2Z + 3 of them) after the two buffers
    // the columns j in segments of one reflection class: segment k covers
    // [segj[k], segj[k + 1]) (segj[nseg] = Z) with class segc[k]: bit 0 the
    // reflection about zpad (w[i + j]), bit 1 the one about zpad + Z - 1
    // (w[i + j - 2Z + 2])
    int nseg, segj[6], segc[6];
    const float *fresp;
    unsigned *err;
};

// Work item -> frequency group and the first tile of its chunk.  Chunk c
// owns tiles [c * ntc, min((c + 1) * ntc, nt)); its box starts at
// min(c * ntc, nt - ntc) so that every box lies inside the batch (the last
// chunk's box may reach back into the previous chunk, whose tiles it computes
// again but does not store).
__device__ __forceinline__ void zth_item(const ZthArgs &a, int item, int &grp, int &own0, int &box0) {
    grp = item / a.nchunks;
    const int c = item - grp * a.nchunks;
    own0 = c * a.ntc;
    box0 = min(own0, a.nt - a.ntc);
}

// ZC > 0: Z known at compile time (50, the depth of every channel of the
// benchmark FOV); otherwise any depth (the last row group and the last column
// block are cut).  TT: tiles of a thread.  PB: frequencies of a group.  CH: the
// batch is split into several tile chunks (otherwise item == frequency group,
// one box of all nt tiles).
template <int ZC, int TT, int PB, bool CH>
__global__ void __launch_bounds__(zth_max_threads(TT, PB), zth_ctas(TT, PB))
k_zth_apply(float2 *__restrict__ S, const __grid_constant__ CUtensorMap wmapA, const __grid_constant__ CUtensorMap wmapB, const ZthArgs a) {
    constexpr int kLPR = PB / 2;  // 16-byte pieces of a row (copying lanes per row)
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(8) uint64_t full[2], empty[2];
    __shared__ int3 item_of[2];  // (group, first owned tile, box start) of each buffer's item
    __shared__ unsigned unit_next;  // the next (item, warp unit) a compute warp takes
    const int Z = ZC > 0 ? ZC : a.Z;
    const int nig = (Z + kTI - 1) / kTI;
    const int tid = threadIdx.x;
    const int kb = a.kA;              // row of w[0] in the staged kernel rows
    const int ko = kb - (2 * Z - 2);  // row of w[-(2Z-2)], the lowest index the rings read

    // every TMA destination (buffer starts, kernel rows, their second box) is
    // 128-byte aligned given an aligned base: check the base, and give up
    // (recording the failure) rather than issue a misaligned copy
    if ((smem_u32(smem) & 127u) != 0u) {
        if (tid == 0) atomicOr(a.err, 2u);
        return;
    }
    const int lane = tid & 31, warp = tid >> 5;
    const int ncw = (int)(blockDim.x >> 5) - 1;          // compute warps; warp ncw produces
    const int units = (PB * nig * a.ntg + 31) / 32;      // warp units of an item
    if (tid == 0) {
        for (int b = 0; b < 2; ++b) {
            // the producer warp's 32 copy arrivals and the arrive that counts
            // the TMA bytes
            mbar_init(&full[b], 33);
            mbar_init(&empty[b], units);
        }
        unit_next = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    {
        float2 *zr = reinterpret_cast<float2 *>(smem + a.zoff);
        for (int e = tid; e < (2 * Z + 3) * PB; e += blockDim.x) zr[e] = make_float2(0.f, 0.f);
    }
    __syncthreads();

    if (warp == ncw) {
        // producer warp: the copies of item `it` go to buffer it & 1 once the
        // compute warps have released its previous use (item it - 2).  X (the
        // box's nt x Z rows of PB x 8 bytes) by cp.async from all 32 lanes: a
        // tensor copy moves a box row per ~5 SM cycles, which rows this short
        // would make the bound; the kernel rows (2Z - 1 + kA rows) by TMA.
        int grp, own0, box0;
        for (int item = blockIdx.x, it = 0; item < a.nitems; item += gridDim.x, ++it) {
            const int buf = it & 1;
            const bool ok = it < 2 || mbar_wait(&empty[buf], ((it - 2) >> 1) & 1);
            if (!__all_sync(0xffffffffu, ok)) {
                if (lane == 0) atomicOr(a.err, 4u);
                break;
            }
            // order the compute warps' reads of the buffer before the copies
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            unsigned char *b = smem + (size_t)buf * a.bufstride;
            zth_item(a, item, grp, own0, box0);
            const int p0 = grp * PB;
            if (lane == 0) {
                item_of[buf] = make_int3(grp, own0, box0);  // published by the arrives below
                mbar_expect_tx(&full[buf], a.wbytesA + a.wbytesB);
                tma_load_2d(b + a.woff, &wmapA, p0, a.Zp - kb, &full[buf]);
                tma_load_2d(b + a.woff + a.wbytesA, &wmapB, p0, 0, &full[buf]);
            }
            const int nchunk = kLPR * Z * a.ntc;  // 16-byte pieces of the box's rows
            // a piece past the plane (the last group of a plane that is no
            // multiple of PB frequencies) is not copied: its results are not stored
            const long long pc = p0 + 2 * (lane % kLPR);
            if (pc < a.plane) {
                for (int k = lane; k < nchunk; k += 32) {
                    const int row = k / kLPR;  // (tile - box0) * Z + plane
                    cp_async16(b + (size_t)k * 16, S + ((long long)box0 * Z + row) * a.plane + pc);
                }
            }
            cp_async_arrive(&full[buf]);
        }
        // no copy may still be landing when the CTA exits
        asm volatile("cp.async.wait_all;" ::: "memory");
        return;
    }

    // An item's threads (PB x nig x ntg) come in warp units: unit u is threads
    // 32u .. 32u + 31 of the item.  The compute warps (between units and 2 units
    // of them) take the units in order from a shared counter, so a warp on a
    // less loaded SM sub-partition takes more of them, and warps beyond an
    // item's units start the next item's.  The parity wait below passes on this
    // item's own phase: to pass on item it - 2's, a warp would have to take a
    // unit of item it while that item's buffer is unfilled.  The producer
    // fills in order, so no unit of items it - 2 and it - 1 could have
    // finished, and their 2 units would occupy 2 units warps besides the taker,
    // more than the CTA has.
    for (;;) {
        unsigned sq = 0;
        if (lane == 0) sq = atomicAdd(&unit_next, 1u);
        sq = __shfl_sync(0xffffffffu, sq, 0);
        const int it = (int)(sq / (unsigned)units), unit = (int)(sq - (unsigned)it * (unsigned)units);
        const long long item_ll = blockIdx.x + (long long)it * gridDim.x;
        if (item_ll >= a.nitems) break;
        const int item = (int)item_ll;
        const int buf = it & 1;
        if (!mbar_wait(&full[buf], (it >> 1) & 1)) {
            atomicOr(a.err, 1u);
            return;
        }
        const int vt = unit * 32 + lane;
        const int p = vt % PB;
        const int r = vt / PB;
        const int ig = r % nig, tg = r / nig;
        const int i0 = ig * kTI, tl0 = tg * TT;  // first row, first tile of the chunk's box
        const float2 *X = reinterpret_cast<const float2 *>(smem + (size_t)buf * a.bufstride);
        const float2 *W = reinterpret_cast<const float2 *>(smem + (size_t)buf * a.bufstride + a.woff) + p;
        if (tg < a.ntg) {
            ZthAcc<TT> acc;
            acc.clear();
            // rings: the direct value of position q (= row - column) in slot
            // q mod 5; the reflected value of position q (= row + column), the
            // sum of the sources of the column's class (the zero rows stand for
            // an absent one), in slot q mod 5 (i0 and the column blocks are
            // multiples of 5).  A column that starts a segment of another class
            // reloads the reflected ring.
            const int zrow = (int)((a.zoff - (unsigned)buf * a.bufstride - a.woff) / (PB * sizeof(float2)));
            int sk = 0, ra = (a.segc[0] & 1) ? kb : zrow, rb = (a.segc[0] & 2) ? ko : zrow;
            int jnext = a.nseg > 1 ? a.segj[1] : Z;
            float2 rT[kTI], rH[kTI];
#pragma unroll
            for (int q = 1; q < kTI; ++q) rT[q] = W[(i0 + q + kb) * PB];
#pragma unroll
            for (int q = 0; q < kTI - 1; ++q) rH[q] = __fadd2_rn(W[(i0 + q + ra) * PB], W[(i0 + q + rb) * PB]);
            rT[0] = rH[kTI - 1] = make_float2(0.f, 0.f);
            // the box's tiles past ntc read stale buffer contents; their
            // results are not stored
            const float2 *xr = X + ((size_t)tl0 * Z) * PB + p;
            for (int j0 = 0; j0 < Z; j0 += kTI) {
                if (ZC == 0 && j0 + kTI <= min(jnext, Z)) {
                    // five columns of one class: no test between them, so
                    // their loads run ahead of the products (nt = 6: 0.84
                    // against 0.90 ms; five tiles a thread have no registers
                    // to spare for it, and ZC > 0 tests in the columns)
#pragma unroll
                    for (int u = 0; u < kTI; ++u) {
                        const int j = j0 + u;
                        rT[(kTI - u) % kTI] = W[(i0 - j + kb) * PB];
                        rH[(u + kTI - 1) % kTI] =
                            __fadd2_rn(W[(i0 + j + kTI - 1 + ra) * PB], W[(i0 + j + kTI - 1 + rb) * PB]);
                        float2 m[kTI], x[TT];
#pragma unroll
                        for (int q = 0; q < kTI; ++q)
                            m[q] = __fadd2_rn(rT[(q - u + kTI) % kTI], rH[(q + u) % kTI]);
#pragma unroll
                        for (int b = 0; b < TT; ++b) x[b] = xr[((size_t)b * Z + j) * PB];
                        acc.add(m, x);
                    }
                    continue;
                }
                if constexpr (ZC > 0) {
                    static_assert(ZC % kTI == 0, "a depth of whole column blocks");
#pragma unroll
                    for (int u = 0; u < kTI; ++u) {
                        const int j = j0 + u;
                        rT[(kTI - u) % kTI] = W[(i0 - j + kb) * PB];
                        if (j == jnext) {
                            ++sk;
                            ra = (a.segc[sk] & 1) ? kb : zrow;
                            rb = (a.segc[sk] & 2) ? ko : zrow;
                            jnext = sk + 1 < a.nseg ? a.segj[sk + 1] : Z;
#pragma unroll
                            for (int q = 0; q < kTI - 1; ++q)
                                rH[(q + u) % kTI] = __fadd2_rn(W[(i0 + j + q + ra) * PB], W[(i0 + j + q + rb) * PB]);
                        }
                        rH[(u + kTI - 1) % kTI] =
                            __fadd2_rn(W[(i0 + j + kTI - 1 + ra) * PB], W[(i0 + j + kTI - 1 + rb) * PB]);
                        float2 m[kTI], x[TT];
#pragma unroll
                        for (int q = 0; q < kTI; ++q) m[q] = __fadd2_rn(rT[(q - u + kTI) % kTI], rH[(q + u) % kTI]);
#pragma unroll
                        for (int b = 0; b < TT; ++b) x[b] = xr[((size_t)b * Z + j) * PB];
                        acc.add(m, x);
                    }
                } else {
                    // a block with a change of class, or cut at Z: one column
                    // at a time, the rings turned by a place after each
                    const int n = min(kTI, Z - j0);
#pragma unroll 1
                    for (int u = 0; u < n; ++u) {
                        const int j = j0 + u;
                        rT[0] = W[(i0 - j + kb) * PB];
                        if (j == jnext) {
                            ++sk;
                            ra = (a.segc[sk] & 1) ? kb : zrow;
                            rb = (a.segc[sk] & 2) ? ko : zrow;
                            jnext = sk + 1 < a.nseg ? a.segj[sk + 1] : Z;
#pragma unroll
                            for (int q = 0; q < kTI - 1; ++q)
                                rH[q] = __fadd2_rn(W[(i0 + j + q + ra) * PB], W[(i0 + j + q + rb) * PB]);
                        }
                        rH[kTI - 1] = __fadd2_rn(W[(i0 + j + kTI - 1 + ra) * PB], W[(i0 + j + kTI - 1 + rb) * PB]);
                        float2 m[kTI], x[TT];
#pragma unroll
                        for (int q = 0; q < kTI; ++q) m[q] = __fadd2_rn(rT[q], rH[q]);
#pragma unroll
                        for (int b = 0; b < TT; ++b) x[b] = xr[((size_t)b * Z + j) * PB];
                        acc.add(m, x);
                        const float2 t4 = rT[kTI - 1], h0 = rH[0];
#pragma unroll
                        for (int q = kTI - 1; q > 0; --q) rT[q] = rT[q - 1];
#pragma unroll
                        for (int q = 0; q < kTI - 1; ++q) rH[q] = rH[q + 1];
                        rT[0] = t4;
                        rH[kTI - 1] = h0;
                    }
                }
            }
            // the operands are in registers: release the buffer before the stores
            const int3 ii = CH ? item_of[buf] : make_int3(item, 0, 0);
            const int own0 = ii.y, box0 = ii.z;
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty[buf]);
            const long long pg = (long long)ii.x * PB + p;
            if (pg < a.plane) {
                const float f = a.fresp ? a.fresp[pg] : 1.f;
                // box0 + ntc >= t_end: the condition keeps t inside the box
                const int t_end = CH ? min(own0 + a.ntc, a.nt) : a.nt;
#pragma unroll
                for (int b = 0; b < TT; ++b) {
                    const int t = CH ? box0 + tl0 + b : tl0 + b;
                    if ((!CH || t >= own0) && t < t_end) {
#pragma unroll
                        for (int q = 0; q < kTI; ++q)
                            if (ZC > 0 || i0 + q < Z)
                                S[((long long)t * Z + i0 + q) * a.plane + pg] = cscale(acc.get(q, b), f);
                    }
                }
            }
        } else {
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty[buf]);
        }
    }
}

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
    static std::once_flag once;
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    std::call_once(once, [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
        else
            cudaGetLastError();
    });
    return fn;
}

// rows of float2 (8-byte elements), innermost dimension first
int make_map(CUtensorMap *m, const void *base, int rank, const cuuint64_t *dims, const cuuint64_t *strides_bytes,
             const cuuint32_t *box) {
    auto fn = encode_fn();
    MM_REQUIRE(fn != nullptr, "cuTensorMapEncodeTiled is not available");
    cuuint32_t es[3] = {1, 1, 1};
    CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, (cuuint32_t)rank, const_cast<void *>(base), dims,
                    strides_bytes, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        mm_set_error("cuTensorMapEncodeTiled failed (%d)", (int)r);
        return MM_EDEVICE;
    }
    return MM_OK;
}

// warp units of an item (threads PB x ceil(Z / kTI) x ntg)
int zth_units(int Z, int pb, int ntg) { return (pb * ((Z + kTI - 1) / kTI) * ntg + 31) / 32; }
// staged row of w[0]: the rows -(2Z-2) .. -1 rounded up to a multiple of four,
// so that the second kernel box starts on a 128-byte boundary
int zth_ka(int Z) { return (2 * Z - 2 + 3) & ~3; }

// bytes per buffer: X for ntg whole tile groups (the last group's threads
// read tiles past the box, whose results are not stored), then the kernel
// rows -kA .. 2Z - 2 and four more that the cut row group of a depth that is no
// multiple of kTI reads for rows it does not store; both parts start on
// 128-byte boundaries
size_t zth_bufstride(int Z, int pb, int tiles, unsigned *woff) {
    const size_t xb = (size_t)pb * Z * tiles * sizeof(float2);
    const size_t wb = (size_t)pb * (zth_ka(Z) + 2 * Z - 1 + 4) * sizeof(float2);
    const size_t xo = (xb + 127) & ~(size_t)127;
    if (woff) *woff = (unsigned)xo;
    return (xo + wb + 127) & ~(size_t)127;
}

// shared memory of an SM's CTAs
constexpr size_t kSmemMax = 224 * 1024;

// the zero rows after the two buffers
size_t zth_zero_bytes(int Z, int pb) { return ((size_t)(2 * Z + 3) * pb * sizeof(float2) + 127) & ~(size_t)127; }

// How a batch of nt tiles runs: TT tiles per thread, PB frequencies per group,
// and the fewest chunks whose tile groups fit one CTA (threads and shared
// memory), the tiles spread evenly over them.
struct ZthPlan {
    int tt, pb, nchunks, ntc, ntg;
};
bool zth_fits(int Z, int pb, int tt, int ntg) {
    return (zth_units(Z, pb, ntg) + 1) * 32 <= zth_max_threads(tt, pb) &&
           2 * zth_bufstride(Z, pb, ntg * tt, nullptr) + zth_zero_bytes(Z, pb) <= kSmemMax / zth_ctas(tt, pb);
}
bool zth_split(int Z, int nt, int tt, int pb, ZthPlan *pl) {
    const int ntg_all = (nt + tt - 1) / tt;
    int ntg_max = ntg_all;
    while (ntg_max > 0 && !zth_fits(Z, pb, tt, ntg_max)) --ntg_max;
    if (ntg_max == 0) return false;
    pl->tt = tt;
    pl->pb = pb;
    pl->nchunks = (ntg_all + ntg_max - 1) / ntg_max;
    pl->ntc = (nt + pl->nchunks - 1) / pl->nchunks;
    pl->ntg = (pl->ntc + tt - 1) / tt;
    return true;
}
// Measured at P = 678 (ms per launch; the per-tile form, or for Z = 37 the
// direct sum, in brackets): Z = 50, 2 tiles, 16 frequencies of 2 tiles a thread
// 0.29 [0.39]; 3 tiles, 8 x 3 0.45 [0.58]; 4 tiles, 8 x 2 0.58, 8 x 5 0.72
// [0.81]; 6 tiles, 8 x 3 0.75, 8 x 5 1.16 [1.21]; 9 tiles, 8 x 5 1.22, 4 x 5
// 1.26 [2.46 at zpad 24]; Z = 37, 9 tiles, 8 x 3 0.67, 8 x 5 0.72 [2.3].  So up
// to ten tiles the groups are wide (a row of 8 frequencies is 64 bytes), and a
// thread's tiles those with the largest share of products in its work: of its
// places that hold a tile, of its warps' lanes in use, and of a column's
// instructions (20 products and 1 load per tile, 15 to form its entries).  More
// tiles: 5 a thread, on 8 frequencies (25 tiles of Z = 37: 1.78 against 2.05;
// 20 of Z = 56: 2.81 against 3.06) but for the depth with its own kernel (25
// tiles of Z = 50: 4 frequencies 2.83, 8 2.94; 16 tiles 1.97 against 2.21).
bool zth_plan(int Z, int nt, ZthPlan *pl) {
    if (nt <= 2 && zth_split(Z, nt, nt, 16, pl) && pl->nchunks == 1) return true;
    if (nt <= 10) {
        double best = 0;
        ZthPlan c;
        for (int tt : {5, 3, 2}) {
            if (!zth_split(Z, nt, tt, 8, &c) || c.nchunks != 1) continue;
            const double lanes = 8.0 * ((Z + kTI - 1) / kTI) * c.ntg / (32.0 * zth_units(Z, 8, c.ntg));
            const double share = (double)nt / (c.ntg * tt) * lanes * 20.0 * tt / (21.0 * tt + 15.0);
            if (share > best) {
                best = share;
                *pl = c;
            }
        }
        if (best > 0) return true;
    } else if (Z != 50 && zth_split(Z, nt, 5, 8, pl) && pl->nchunks == 1) {
        return true;
    }
    return zth_split(Z, nt, 5, 4, pl);
}

// Threads of a CTA: the producer warp, a compute warp per unit, and more (up to
// two per unit, see the kernel) as far as the CTAs that fit an SM beside each
// other leave registers: a warp beyond an item's units starts the next item (6
// tiles of Z = 50: 0.79 -> 0.75 ms, 16 tiles 2.07 -> 1.97).
int zth_threads(int Z, const ZthPlan &pl, size_t smem) {
    const int units = zth_units(Z, pl.pb, pl.ntg);
    int ctas = 16 / (units + 1);
    if (ctas > (int)(kSmemMax / smem)) ctas = (int)(kSmemMax / smem);
    if (ctas < 1) ctas = 1;
    int w = 16 / ctas - 1;
    if (w > zth_max_threads(pl.tt, pl.pb) / 32 - 1) w = zth_max_threads(pl.tt, pl.pb) / 32 - 1;
    if (w > 2 * units) w = 2 * units;
    return ((w > units ? w : units) + 1) * 32;
}

const void *zth_kernel(int Z, const ZthPlan &pl) {
    if (pl.nchunks > 1) return (const void *)k_zth_apply<0, 5, 4, true>;
    switch (pl.tt * 100 + pl.pb) {
        case 504: return Z == 50 ? (const void *)k_zth_apply<50, 5, 4, false> : (const void *)k_zth_apply<0, 5, 4, false>;
        case 508: return (const void *)k_zth_apply<0, 5, 8, false>;
        case 308: return (const void *)k_zth_apply<0, 3, 8, false>;
        case 208: return (const void *)k_zth_apply<0, 2, 8, false>;
        case 216: return (const void *)k_zth_apply<0, 2, 16, false>;
        case 116: return (const void *)k_zth_apply<0, 1, 16, false>;
    }
    return nullptr;
}

}  // namespace

int mm_zth_supported(int Z, int zpad, int nt, long long plane) {
    if (Z < 2 || zpad < 1 || zpad > Z - 1 || nt < 1 || plane % 2 != 0) return 0;
    if (2 * Z - 1 > 256 || zth_ka(Z) > 256) return 0;  // TMA box height
    ZthPlan pl;
    return zth_plan(Z, nt, &pl) && encode_fn() != nullptr ? pl.nchunks : 0;
}

int mm_launch_zth_apply(float2 *S, const float2 *w, int Z, int zpad, int Zp, long long plane, int nt,
                        const float *fresp, unsigned *err, cudaStream_t st) {
    MM_REQUIRE(Zp == Z + 2 * zpad && mm_zth_supported(Z, zpad, nt, plane),
               "z operator (TMA form) does not take Z %d, zpad %d, %d tiles", Z, zpad, nt);
    MM_REQUIRE(((uintptr_t)S & 15) == 0 && ((uintptr_t)w & 15) == 0, "spectra must be 16-byte aligned");
    ZthPlan pl;
    zth_plan(Z, nt, &pl);
    CUtensorMap wA, wB;
    const cuuint32_t kb = (cuuint32_t)(2 * Z - 2), kA = (cuuint32_t)zth_ka(Z), pb = (cuuint32_t)pl.pb;
    {
        cuuint64_t dims[2] = {(cuuint64_t)plane, (cuuint64_t)Zp};
        cuuint64_t strides[1] = {(cuuint64_t)plane * 8};
        cuuint32_t boxA[2] = {pb, kA}, boxB[2] = {pb, kb + 1};
        if (int rc = make_map(&wA, w, 2, dims, strides, boxA)) return rc;
        if (int rc = make_map(&wB, w, 2, dims, strides, boxB)) return rc;
    }
    ZthArgs a = {};
    a.Z = Z;
    a.Zp = Zp;
    a.nt = nt;
    a.ntc = pl.ntc;
    a.ntg = pl.ntg;
    a.nchunks = pl.nchunks;
    a.plane = plane;
    const long long nitems = ((plane + pl.pb - 1) / pl.pb) * pl.nchunks;
    MM_REQUIRE(nitems < (1LL << 31), "z operator: too many frequency groups");
    a.nitems = (int)nitems;
    // the column segments of one reflection class
    a.nseg = 0;
    for (int j = 0, prev = -1; j < Z; ++j) {
        const bool vin = j >= 1 && j <= zpad, vout = j >= Z - 1 - zpad && j <= Z - 2;
        const int cls = (vin ? 1 : 0) | (vout ? 2 : 0);
        if (cls != prev) {
            MM_REQUIRE(a.nseg < 6, "z operator: more than six column segments");
            a.segj[a.nseg] = j;
            a.segc[a.nseg] = cls;
            ++a.nseg;
            prev = cls;
        }
    }
    a.kA = (int)kA;
    a.wbytesA = (unsigned)(pl.pb * kA * sizeof(float2));
    a.wbytesB = (unsigned)(pl.pb * (kb + 1) * sizeof(float2));
    a.bufstride = (unsigned)zth_bufstride(Z, pl.pb, pl.ntg * pl.tt, &a.woff);
    a.zoff = 2 * a.bufstride;
    MM_REQUIRE(a.bufstride % 128 == 0 && a.woff % 128 == 0 && a.wbytesA % 128 == 0,
               "TMA destinations of the z operator must be 128-byte aligned");
    MM_REQUIRE((size_t)pl.pb * Z * pl.ntc * sizeof(float2) <= a.woff, "z operator: the X box overruns its buffer");
    a.fresp = fresp;
    a.err = err;
    const size_t sm = 2 * (size_t)a.bufstride + zth_zero_bytes(Z, pl.pb);
    const int threads = zth_threads(Z, pl, sm);
    const void *fn = zth_kernel(Z, pl);
    MM_REQUIRE(fn != nullptr, "z operator: no kernel for %d tiles per thread, %d frequencies", pl.tt, pl.pb);
    if (int rc = mm_set_smem(fn, sm)) return rc;
    int per_sm = 0;
    MM_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, sm));
    if (per_sm < 1) per_sm = 1;
    const long long cap = (long long)mm_sm_count() * per_sm;
    const unsigned grid = (unsigned)(a.nitems < cap ? a.nitems : cap);
    void *args[] = {&S, &wA, &wB, &a};
    MM_CUDA_TRY(cudaLaunchKernel(fn, dim3(grid), dim3(threads), args, sm, st));
    mm_launch_counter_add();
    return MM_OK;
}
