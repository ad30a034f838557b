// Device-side reductions shared by the solver kernels and the learned cycle's
// transfer kernels: exact-product accumulators, the deterministic block/grid
// reduction whose last block advances the Krylov scalars (finalize), and the
// early exit of kernels launched after the stop flag was set.
#pragma once
#include "pps_internal.h"

#include <cuda_runtime.h>
#include <math.h>

namespace pps {

// Fused multiply-add for either storage type.
__device__ __forceinline__ float fmx(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fmx(double a, double b, double c) { return __fma_rn(a, b, c); }

// Accumulator of exact products: FP64 FMA for double data; for float data a
// double-float pair (Dekker/Knuth error-free product and sum in FP32), so the
// inner products of the mixed form are FP64-accurate without FP64 arithmetic
// per point (GB300 runs FP64 at 1/64 of the FP32 rate).
template <typename T>
struct Acc;
// float to double on the integer pipe: the FP64 pipe, which also converts, takes 16 clocks a
// warp (measured, one SM with 8 warps and more).  Infinities, NaNs and denormals are left to the conversion instruction.
__device__ __forceinline__ double widen(float f)
{
    const unsigned u = __float_as_uint(f), e = (u >> 23) & 255u;
    if (e - 1u < 254u) return __hiloint2double((int)((u & 0x80000000u) | (((u & 0x7fffffffu) >> 3) + (896u << 20))), (int)(u << 29));
    if ((u << 1) == 0u) return __hiloint2double((int)u, 0);
    return (double)f;
}
template <>
struct Acc<double> {
    double s = 0.0;
    __device__ __forceinline__ void add(double a, double b) { s = fmx(a, b, s); }
    __device__ __forceinline__ double value() const { return s; }
};
template <>
struct Acc<float> {
    float hi = 0.f, lo = 0.f;
    __device__ __forceinline__ void add(float a, float b)
    {
        const float p = __fmul_rn(a, b);
        const float e = __fmaf_rn(a, b, -p);
        const float s = __fadd_rn(hi, p);
        const float bb = __fsub_rn(s, hi);
        const float t = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, bb)), __fsub_rn(p, bb));
        hi = s;
        lo = __fadd_rn(lo, __fadd_rn(t, e));
    }
    __device__ __forceinline__ double value() const { return widen(hi) + widen(lo); }
};

__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

// warp_sum of two values at once, lane 0 receiving a's sum and lane 16 b's: the halves of
// the warp trade values first, so the shared tree takes 5 additions instead of 10.  The
// operands of each addition are warp_sum's, so the sums have the same bits.
__device__ __forceinline__ double warp_sum2(double a, double b)
{
    const bool up = threadIdx.x & 16;
    const double mine = up ? b : a, give = up ? a : b;
    double v = mine + __shfl_xor_sync(0xffffffffu, give, 16);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

// Block sums of NS values per thread, at most 256 threads: warp q (mod the warps) adds sum q,
// eight or fewer values a lane and one shuffle tree.  An SM of GB300
// takes 19 clocks for the FP64 addition of a warp (95 for a tree of five, measured with 8 warps
// and more), so what counts is their number: a tree in every warp took 5 a warp and sum,
// this takes 1 and a last tree (with conversions, 64 -> 20 a block and sum).  Mixed CG on
// 120 x 128 x 90: 17.8 -> 14.3 ms.  st is shared memory; emit(q, sum) runs on one lane per sum.
template <int NS, typename Emit>
__device__ __forceinline__ void block_sums(const double (&v)[NS], double (*st)[256], int tid, int nwarp, Emit emit)
{
#pragma unroll
    for (int q = 0; q < NS; q++) st[q][tid] = v[q];
    __syncthreads();
    const int lane = tid & 31;
    for (int q = tid >> 5; q < NS; q += nwarp) {
        double s = st[q][lane];
        for (int w = 1; w < nwarp; w++) s += st[q][lane + 32 * w];
        s = warp_sum(s);
        if (lane == 0) emit(q, s);
    }
}

static __device__ void finalize(const RedCtx& rc, const double* tot)
{
    DevState* st = rc.st;
    for (int q = 0; q < 4; q++) st->sums[q] = tot[q];
    switch (rc.kind) {
    case FIN_NORMB:
        st->normb = sqrt(tot[0]);
        break;
    case FIN_RES0: {
        const double e0 = sqrt(tot[0]);
        st->err0 = e0;
        st->err = e0;
        if (rc.hist && st->hist_cap > 0) rc.hist[0] = e0 * st->hist_scale;
        st->rho0 = st->rho0_from_r ? tot[0] : st->normb * st->normb;
        st->iter = 0;
        if (!(e0 == e0) || isinf(e0)) {
            st->status = 3;
            st->done = 1;
        } else if (e0 < st->tol_abs) {
            st->status = 0;
            st->done = 1;
        } else {
            st->done = 0;
            st->status = 0;
            // inner solve of a refinement step: reduce by tol_rel, or less if enough
            if (st->tol_relative) st->tol_abs = fmax(st->tol_rel, 0.3 * st->tol_abs / e0) * e0;
        }
        break;
    }
    case FIN_ALPHA: {
        const double a = st->rho0 / tot[0];
        st->alpha = a;
        if (!isfinite(a)) {
            st->status = 2;
            st->done = 1;
        }
        break;
    }
    case FIN_OMEGA: {
        const double w = tot[0] / tot[1];
        st->omega = w;
        if (!isfinite(w) || w == 0.0) {
            st->status = 2;
            st->done = 1;
        }
        break;
    }
    case FIN_CONV: {
        const double err = sqrt(tot[1]);
        const double rho1 = tot[0];
        st->err = err;
        st->beta = rho1 / st->rho0 * st->alpha / st->omega;
        st->rho0 = rho1;
        st->iter += 1;
        if (rc.hist && st->iter < st->hist_cap) rc.hist[st->iter] = err * st->hist_scale;
        if (!isfinite(err)) {
            st->status = 3;
            st->done = 1;
        } else if (err < st->tol_abs) {
            st->status = 0;
            st->done = 1;
        } else if (st->iter >= st->maxit) {
            st->status = 1;
            st->done = 1;
        } else if (!isfinite(st->beta)) {
            st->status = 2;
            st->done = 1;
        }
        break;
    }
    case FIN_CG_ALPHA: {
        st->rho0 = tot[0];                    // r.z
        st->alpha = tot[0] / tot[1];          // r.z / p.Ap
        if (!isfinite(st->alpha)) {
            st->status = 2;
            st->done = 1;
        }
        break;
    }
    case FIN_CG_CONV: {
        const double err = sqrt(tot[1]);
        st->err = err;
        st->beta = tot[0] / st->rho0;         // r_new.z_new / r.z
        st->iter += 1;
        if (rc.hist && st->iter < st->hist_cap) rc.hist[st->iter] = err * st->hist_scale;
        if (!isfinite(err)) {
            st->status = 3;
            st->done = 1;
        } else if (err < st->tol_abs) {
            st->status = 0;
            st->done = 1;
        } else if (st->iter >= st->maxit) {
            st->status = 1;
            st->done = 1;
        }
        break;
    }
    case FIN_FCG_ALPHA: {
        st->alpha = st->rho0 / tot[0];        // z.r / p.Ap
        if (!isfinite(st->alpha)) {
            st->status = 2;
            st->done = 1;
        }
        break;
    }
    case FIN_FCG_SETUP: {
        st->rho0 = tot[0];                    // z.r
        st->beta = 0.0;
        break;
    }
    case FIN_FCG_RES: {
        // flexible CG after x, r: the recursive residual norm and the stop test
        const double err = sqrt(tot[0]);
        st->err = err;
        st->iter += 1;
        if (rc.hist && st->iter < st->hist_cap) rc.hist[st->iter] = err * st->hist_scale;
        if (!isfinite(err)) {
            st->status = 3;
            st->done = 1;
        } else if (err < st->tol_abs) {
            st->status = 0;
            st->done = 1;
        } else if (st->iter >= st->maxit) {
            st->status = 1;
            st->done = 1;
        }
        break;
    }
    case FIN_FCG_CONV: {
        // flexible CG, Polak-Ribiere: beta = z_new.(r_new - r_old) / (z_old.r_old)
        // with r_new - r_old = -alpha Ap
        st->beta = -st->alpha * tot[1] / st->rho0;
        st->rho0 = tot[0];
        if (!isfinite(st->beta)) {
            st->status = 2;
            st->done = 1;
        }
        break;
    }
    case FIN_STORE:
        if (rc.store) {   // byte by byte: a caller's address of any alignment
            unsigned char* to = static_cast<unsigned char*>(rc.store);
            const long long bits = __double_as_longlong(tot[0]);
            for (int q = 0; q < 8; q++) to[q] = (unsigned char)(bits >> (8 * q));
        }
        break;
    default:
        break;
    }
}

// Block reduction of NS partial sums, then the last block reduces all block
// partials in block order and runs the finalizer.  Every thread of every block
// must call this (inactive threads pass zeros).
template <int NS>
__device__ __forceinline__ void reduce_finalize(double (&v)[NS], const RedCtx& rc)
{
    __shared__ double st[NS][256], sm[NS];
    __shared__ int is_last;
    const int tid = threadIdx.x + blockDim.x * threadIdx.y;
    const int nthr = blockDim.x * blockDim.y;
    const int nwarp = nthr >> 5;
    const unsigned nblocks = gridDim.x * gridDim.y;
    const unsigned bid = blockIdx.x + gridDim.x * blockIdx.y;
    block_sums<NS>(v, st, tid, nwarp, [&](int q, double s) {
        rc.partials[(size_t)bid * 4 + q] = s;
        __threadfence();
    });
    __syncthreads();
    if (tid == 0) is_last = count_block(rc.counter, bid, nblocks);
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    double acc[NS];
#pragma unroll
    for (int q = 0; q < NS; q++) acc[q] = 0.0;
    for (unsigned b = tid; b < nblocks; b += nthr) {
#pragma unroll
        for (int q = 0; q < NS; q++) acc[q] += __ldcg(&rc.partials[(size_t)b * 4 + q]);
    }
    block_sums<NS>(acc, st, tid, nwarp, [&](int q, double s) { sm[q] = s; });
    __syncthreads();
    if (tid == 0) {
        double tot[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for (int q = 0; q < NS; q++) tot[q] = sm[q];
        finalize(rc, tot);
    }
}

// Canonical sums: one partial per warp stored as its cell (every lane calls it; rows past
// the last unknown own no cell).
template <int NS>
__device__ __forceinline__ void store_cells(const double (&v)[NS], const RedCtx& rc, const Shape& sh)
{
    static_assert(NS <= 2, "one or two canonical sums");
    const int bx = blockIdx.x % sh.ntx;
    const int row = (blockIdx.x / sh.ntx) * sh.ty + threadIdx.y;
    const double w = NS == 2 ? warp_sum2(v[0], v[NS - 1]) : warp_sum(v[0]);
    if (row < rc.cell_ny && (threadIdx.x & (NS == 2 ? 15 : 31)) == 0) {
        const long long cell = ((long long)blockIdx.y * rc.cell_ny + row) * rc.cell_ntx + bx;
        rc.cells[(threadIdx.x >> 4) * rc.cell_n + cell] = w;
    }
}

// The end of a z-marching kernel on the one-column tiles: canonical sums, or the
// deterministic block reduction.
template <int NS>
__device__ __forceinline__ void reduce_emit(double (&v)[NS], const RedCtx& rc, const Shape& sh)
{
    if (rc.cells) store_cells<NS>(v, rc, sh);
    else reduce_finalize<NS>(v, rc);
}

#define EARLY_EXIT(done)                                      \
    if (done != nullptr && *(volatile const int*)(done) != 0) return;

}  // namespace pps
