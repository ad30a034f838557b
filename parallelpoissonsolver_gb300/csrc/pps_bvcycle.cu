// Batched solves in ONE persistent launch: flexible CG with a multigrid V-cycle per
// problem, FP32 inner iterations inside FP64 iterative refinement.
//
// No reference counterpart (the reference solves one grid per run).  The batch's
// problems are cubes of uneven size (Dirichlet walls, equal spacings).  One
// cooperative kernel (every block resident) runs the whole solve: a fixed program of
// phases per round, all problems advancing together, each phase spread over every
// block as (problem, tile) work items, phases separated by a grid barrier whose wait
// is bounded in time (a wait that runs out sets an error flag, every block returns,
// and the solve reports PPS_TIMEOUT).  The launch, with the state reset before it, is
// captured once as a CUDA graph and replayed.
//
// A round for one problem is either an FCG iteration or a refinement step:
//   A  FCG: p = z + beta p_old, Ap = A p, sum p.Ap -> alpha   | refine: x += e, e = 0
//   B  FCG: e += alpha p, r -= alpha Ap, sum r.r -> stop test | refine: r = b - A x
//      in FP64, ||r|| -> outer stop test, inner target
//   V-cycle z = M r (skipped once the inner solve has converged):
//      level 0: Chebyshev(5) on [lmax/8, lmax]; residual; full-weighting restriction
//      levels 1..k-1: Jacobi-scaled Chebyshev(4) on [2/8, 2] of D^-1 A_l, residual,
//      restriction; level k (at most 32 unknowns per axis): exact inverse by a
//      tensor-product eigen-solve; back up: trilinear prolongation, residual,
//      Jacobi-scaled Chebyshev(4) post-smoothing; level 0: z += P z_1
//   P0 sums z.r, z.Ap -> beta (Polak-Ribiere, -alpha z.Ap / rho), rho = z.r
// The coarse operators are the learned V-cycle's (level l: spacing 2^l h, the upper
// wall one fine spacing above the last unknown).  Reductions are per problem and
// deterministic: one partial per work item, summed in item order by the problem's
// last item, which then advances that problem's scalars.
#include "../../include/pps.h"
#include "pps_internal.h"
#include "pps_reduce.cuh"
#include "pps_unet_internal.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <string>
#include <vector>

namespace pps {
namespace bvc {

constexpr int MAXLEV = 6;          // levels 0..5
constexpr int NT = 256;            // threads per block: 32 x 8 columns of a tile
constexpr int EX_MAX = 32;         // coarsest level: at most 32 unknowns per axis
constexpr int KZ0 = 128, KZ1 = 16;   // longest z chunks of work items: level 0, coarse levels
constexpr double RATIO = 8.0;      // smoothing interval [lmax/RATIO, lmax]

struct Prob {
    int m, k;                      // unknowns per axis on level 0; coarsest level
    long long off;                 // pooled offset of the level-0 guard-padded fields
    long long coff[MAXLEV];        // pooled offset of level l >= 1 (dense n_l^3)
    int n[MAXLEV];                 // unknowns per axis on level l
    int kz[MAXLEV];                // planes per work item on level l
    int lwlog;                     // level 0 in quads of 4 points: log2 of the lanes of a row; 0: one column per thread
    double ih2;                    // 1/h^2 (FP64 residual)
    float fcc[3], fcn[3], fcb[3], fcz[3];   // fine Chebyshev steps: W = cc Y + cn sum(Y nbrs) + cb B + cz Z
    float lih2[MAXLEV], lastm[MAXLEV], lastc[MAXLEV];   // level operators (l >= 1)
    long long mats;                // offset of the coarsest level's eigen-solve matrices
};

struct State {
    double normb, tol_outer, err_outer, target, err;
    double rho, alpha, beta;
    int mode;                      // 0: refinement step next, 1: FCG iteration
    int done, status, skip, par;
    int xnz;                       // the initial x holds a non-zero value the residual reads
    int inner_it, total_it, refinements;
};

// The arrivals' counter and the generation the blocks poll lie on lines of their own.
struct alignas(128) Barrier {
    unsigned count;
    unsigned pad0[31];
    unsigned gen;
    int error;
    unsigned pad1[30];
};

enum : int { PH_NORM = 0, PH_A, PH_B, PH_C1, PH_C2, PH_C3, PH_R0, PH_RS, PH_D1, PH_D2, PH_DR, PH_EX, PH_UP, PH_UR,
             PH_U1, PH_U2, PH_P0 };

struct Phase {
    int type, level;
};

struct Dev {
    const Prob* prob;
    int nprob;
    const long long* toff;         // toff[l * (nprob + 1) + q]: first work item of problem q on level l
    const int4* items[MAXLEV];     // level l's work items: problem, first column along x, y, first plane
    const Phase* phases;
    int nphases;
    State* st;
    double* x;
    const double* b;
    float *r, *z, *pa, *pb, *ap, *e, *y1, *y2, *t0;   // level 0 (guard-padded)
    float *cr, *cz, *ct, *cc1;                        // levels >= 1 (dense)
    const float* mats;
    double* partials;
    unsigned* counters;
    Barrier* bar;
    int* unfinished;
    double tol, inner_tol;
    int inner_maxit, max_refinements, max_rounds;
    float jt, ja1, jb1, ja2, jb2, jc2;   // coarse Jacobi-Chebyshev constants (ph_jcheb)
    unsigned long long limit_ns;
};

__device__ __forceinline__ unsigned long long now_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Grid barrier of the resident blocks.  Thread 0 of each block reads the generation,
// arrives on the counter, and waits for the generation to change; the last block to
// arrive resets the counter and advances the generation.  The wait gives up after
// limit_ns (or as soon as another block gave up): it then sets the error flag and
// every block returns.  Returns false after an error.
__device__ bool grid_barrier(const Dev& D)
{
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        volatile unsigned* gen = &D.bar->gen;
        volatile int* err = &D.bar->error;
        const unsigned g = *gen;
        __threadfence();
        if (atomicAdd(&D.bar->count, 1u) == gridDim.x - 1) {
            D.bar->count = 0u;
            __threadfence();
            atomicAdd(&D.bar->gen, 1u);
        } else {
            const unsigned long long t0 = now_ns();
            for (unsigned spin = 1; *gen == g; spin++) {
                if (spin % 16 == 1 && (*err != 0 || now_ns() - t0 > D.limit_ns)) {
                    atomicExch(&D.bar->error, 1);
                    break;
                }
            }
        }
        __threadfence();
        ok = (*err == 0);
    }
    __syncthreads();
    return ok != 0;
}

// ---- work items ----

struct Item {
    int q;
    int i, j, k0, k1;              // this thread's column (0-based unknown indices; a quad's first) and planes
    int l, lw;                     // quads: this thread's lane of its row, lanes of a row
    bool on;                       // the column lies inside the level
    long long item;                // item index within the phase
};

// quads: level 0 of a problem with lwlog > 0 (a row's quads on 1 << lwlog lanes)
__device__ __forceinline__ Item decode(const Dev& D, int lev, long long item, bool quads)
{
    Item it;
    const int4 w = __ldg(D.items[lev] + item);
    it.q = w.x;
    it.item = item;
    const Prob& P = D.prob[it.q];
    const int n = P.n[lev];
    const int lwlog = quads ? P.lwlog : 0;
    if (lwlog > 0) {
        it.lw = 1 << lwlog;
        it.l = (int)threadIdx.x & (it.lw - 1);
        it.i = w.y + 4 * it.l;
        it.j = w.z + (int)(threadIdx.x >> lwlog);
    } else {
        it.lw = it.l = 0;
        it.i = w.y + (int)(threadIdx.x & 31);
        it.j = w.z + (int)(threadIdx.x >> 5);
    }
    it.k0 = w.w;
    it.k1 = min(it.k0 + P.kz[lev], n);
    it.on = it.i < n && it.j < n;
    return it;
}

// Block sum of NS partials in a fixed order (warp trees, then the eight warps in
// order), stored as this item's partial; the problem's last item sums its items'
// partials in item order (thread t the ones at t + 256 m, then the same block tree)
// and returns true to thread 0 with the totals.
template <int NS>
__device__ bool item_reduce(const Dev& D, const Item& it, long long first, long long count, double (&v)[NS],
                            double (&tot)[2])
{
    __shared__ double sm[8][2];
    __shared__ int last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int s = 0; s < NS; s++) {
        const double w = warp_sum(v[s]);
        if (lane == 0) sm[warp][s] = w;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
        for (int s = 0; s < NS; s++) {
            double t = 0.0;
            for (int w = 0; w < 8; w++) t += sm[w][s];
            D.partials[it.item * 2 + s] = t;
        }
        __threadfence();
        last = atomicAdd(&D.counters[it.q], 1u) == (unsigned)(count - 1);
    }
    __syncthreads();
    if (!last) return false;
    __threadfence();
    double acc[NS];
#pragma unroll
    for (int s = 0; s < NS; s++) acc[s] = 0.0;
    for (long long c = first + threadIdx.x; c < first + count; c += NT) {
#pragma unroll
        for (int s = 0; s < NS; s++) acc[s] += __ldcg(&D.partials[c * 2 + s]);
    }
    __syncthreads();
#pragma unroll
    for (int s = 0; s < NS; s++) {
        const double w = warp_sum(acc[s]);
        if (lane == 0) sm[warp][s] = w;
    }
    __syncthreads();
    bool mine = false;
    if (threadIdx.x == 0) {
        tot[0] = tot[1] = 0.0;
#pragma unroll
        for (int s = 0; s < NS; s++) {
            double t = 0.0;
            for (int w = 0; w < 8; w++) t += sm[w][s];
            tot[s] = t;
        }
        D.counters[it.q] = 0u;
        mine = true;
    }
    __syncthreads();
    return mine;
}

__device__ void finish(const Dev& D, State& S, int status)
{
    S.done = 1;
    S.status = status;
    atomicSub(D.unfinished, 1);
}

// The problem's scalars after a reduction phase (thread 0 of its last item).
__device__ void advance(const Dev& D, int q, int type, const double (&tot)[2])
{
    State& S = D.st[q];
    switch (type) {
    case PH_NORM:
        S.normb = sqrt(tot[0]);
        S.tol_outer = D.tol * S.normb;
        S.mode = 0;
        S.skip = 0;
        if (!(S.normb > 0.0)) finish(D, S, PPS_ERR_ZERO_RHS);
        else if (!isfinite(S.normb)) finish(D, S, PPS_NAN_DETECTED);
        break;
    case PH_A:   // FCG: alpha = rho / p.Ap; the new direction becomes p_old
        S.alpha = S.rho / tot[0];
        S.par ^= 1;
        if (!isfinite(S.alpha)) finish(D, S, PPS_BREAKDOWN);
        break;
    case PH_B:
        if (S.mode == 1) {   // FCG: recursive residual norm, inner stop test
            S.err = sqrt(tot[0]);
            S.inner_it++;
            S.total_it++;
            if (!isfinite(S.err)) {
                finish(D, S, PPS_NAN_DETECTED);
            } else if (S.err < S.target || S.inner_it >= D.inner_maxit) {
                S.skip = 1;    // converged inner solve: no V-cycle; a refinement step next
                S.mode = 0;
            }
        } else {             // refinement: FP64 true residual, outer stop test
            S.err_outer = sqrt(tot[0]);
            if (!isfinite(S.err_outer)) {
                finish(D, S, PPS_NAN_DETECTED);
            } else if (S.err_outer <= S.tol_outer) {
                finish(D, S, PPS_OK);
            } else if (S.refinements >= D.max_refinements) {
                finish(D, S, PPS_NOT_CONVERGED);
            } else {
                S.refinements++;
                S.target = fmax(D.inner_tol, 0.3 * S.tol_outer / S.err_outer) * S.err_outer;
                S.inner_it = 0;
                S.skip = 0;
            }
        }
        break;
    case PH_P0:
        if (S.mode == 0) {   // after a refinement step: the FCG recurrence (re)starts
            S.rho = tot[0];
            S.beta = 0.0;
            S.mode = 1;
        } else {             // Polak-Ribiere: beta = z_new.(r_new - r_old) / rho, r_new - r_old = -alpha Ap
            S.beta = -S.alpha * tot[1] / S.rho;
            S.rho = tot[0];
        }
        if (!isfinite(S.beta) || !isfinite(S.rho)) finish(D, S, PPS_BREAKDOWN);
        break;
    default:
        break;
    }
}

// ---- level 0: guard-padded fields, one column per thread ----

__device__ __forceinline__ long long idx0(const Prob& P, int i, int j, int k)
{
    const long long sj = P.m + 4, sk = sj * sj;
    return P.off + (i + 2) + sj * (j + 2) + sk * (k + 2);
}

// sum of the six neighbours of c (guard and boundary cells of the work fields are 0)
__device__ __forceinline__ float nsum(const float* f, long long c, long long sj, long long sk)
{
    return ((f[c - 1] + f[c + 1]) + (f[c - sj] + f[c + sj])) + (f[c - sk] + f[c + sk]);
}

// ---- levels >= 1: dense n^3, the upper wall one fine spacing above the last unknown ----

// ---- phase bodies ----

// ||b_adj||^2: b minus the Dirichlet nodes' contributions (x on the boundary nodes);
// nz: whether x holds a non-zero value at an unknown or a node next to one
__device__ void ph_norm(const Dev& D, const Item& it, double& acc, unsigned long long& nz)
{
    const Prob& P = D.prob[it.q];
    if (!it.on) return;
    const long long sj = P.m + 4, sk = sj * sj;
    const int m = P.m;
    auto bits = [](double v) { return (unsigned long long)__double_as_longlong(v) << 1; };
    for (int u = 0; u < (it.lw ? 4 : 1); u++) {
        const int i = it.i + u;
        const bool rim = i == 0 || i == m - 1 || it.j == 0 || it.j == m - 1;
        long long c = idx0(P, i, it.j, it.k0);
        for (int k = it.k0; k < it.k1; k++, c += sk) {
            double v = D.b[c];
            nz |= bits(D.x[c]);
            if (rim || k == 0 || k == m - 1) {
                double bd = 0.0;
                auto node = [&](bool at, long long o) {
                    if (!at) return;
                    const double xv = D.x[c + o];
                    nz |= bits(xv);
                    bd += xv;
                };
                node(i == 0, -1);
                node(i == m - 1, 1);
                node(it.j == 0, -sj);
                node(it.j == m - 1, sj);
                node(k == 0, -sk);
                node(k == m - 1, sk);
                v -= bd * P.ih2;
            }
            acc = fma(v, v, acc);
        }
    }
}

// FCG direction: p_out = z + beta p_in at the point and its six neighbours (so p_in
// and p_out are distinct fields), Ap = A p_out, sum p_out.Ap
__device__ void ph_a_fcg(const Dev& D, const Item& it, Acc<float>& acc)
{
    const Prob& P = D.prob[it.q];
    const State& S = D.st[it.q];
    if (!it.on) return;
    const long long sj = P.m + 4, sk = sj * sj;
    const float* pin = S.par ? D.pb : D.pa;
    float* pout = S.par ? D.pa : D.pb;
    const float be = (float)S.beta, ih2 = (float)P.ih2;
    // z and p_in of the planes below and above are carried along the march; the sums
    // keep nsum's operand order
    long long c = idx0(P, it.i, it.j, it.k0);
    float zm = D.z[c - sk], zc = D.z[c], qm = 0.f, qc = 0.f;
    if (be != 0.f) {
        qm = pin[c - sk];
        qc = pin[c];
    }
    for (int k = it.k0; k < it.k1; k++, c += sk) {
        const float zp = D.z[c + sk];
        const float zs = ((D.z[c - 1] + D.z[c + 1]) + (D.z[c - sj] + D.z[c + sj])) + (zm + zp);
        float pc, ps, qp = 0.f;
        if (be == 0.f) {
            pc = zc;
            ps = zs;
        } else {
            qp = pin[c + sk];
            pc = fmaf(be, qc, zc);
            ps = fmaf(be, ((pin[c - 1] + pin[c + 1]) + (pin[c - sj] + pin[c + sj])) + (qm + qp), zs);
        }
        const float a = (ps - 6.f * pc) * ih2;
        pout[c] = pc;
        D.ap[c] = a;
        acc.add(pc, a);
        zm = zc;
        zc = zp;
        qm = qc;
        qc = qp;
    }
}

__device__ void ph_a_refine(const Dev& D, const Item& it)
{
    const Prob& P = D.prob[it.q];
    if (!it.on) return;
    const bool first = D.st[it.q].refinements == 0;   // no correction yet
    for (int k = it.k0; k < it.k1; k++) {
        const long long c = idx0(P, it.i, it.j, k);
        const float ev = D.e[c];
        if (!first && ev != 0.f) D.x[c] += (double)ev;
        D.e[c] = 0.f;
    }
}

__device__ void ph_b_fcg(const Dev& D, const Item& it, Acc<float>& acc)
{
    const Prob& P = D.prob[it.q];
    const State& S = D.st[it.q];
    if (!it.on) return;
    const float* p = S.par ? D.pb : D.pa;   // the direction phase A wrote (its parity flipped since)
    const float al = (float)S.alpha;
    for (int k = it.k0; k < it.k1; k++) {
        const long long c = idx0(P, it.i, it.j, k);
        D.e[c] = fmaf(al, p[c], D.e[c]);
        const float rn = fmaf(-al, D.ap[c], D.r[c]);
        D.r[c] = rn;
        acc.add(rn, rn);
    }
}

// The first residual of a solve that starts from x = 0 is b.
__device__ __forceinline__ bool from_b(const State& S) { return S.refinements == 0 && S.xnz == 0; }

// refinement residual r = b - A x in FP64, stored in FP32; sum of its FP64 squares
__device__ void ph_b_refine(const Dev& D, const Item& it, double& acc)
{
    const Prob& P = D.prob[it.q];
    if (!it.on) return;
    const long long sj = P.m + 4, sk = sj * sj;
    const double* x = D.x;
    long long c = idx0(P, it.i, it.j, it.k0);
    if (from_b(D.st[it.q])) {
        for (int k = it.k0; k < it.k1; k++, c += sk) {
            const double rv = D.b[c];
            D.r[c] = (float)rv;
            acc = fma(rv, rv, acc);
        }
        return;
    }
    double xm = x[c - sk], xc = x[c];   // the planes below and above carried along the march
    for (int k = it.k0; k < it.k1; k++, c += sk) {
        const double xp = x[c + sk];
        const double s6 = ((x[c - 1] + x[c + 1]) + (x[c - sj] + x[c + sj])) + (xm + xp);
        const double rv = D.b[c] - (s6 - 6.0 * xc) * P.ih2;
        D.r[c] = (float)rv;
        acc = fma(rv, rv, acc);
        xm = xc;
        xc = xp;
    }
}

// fine Chebyshev step t: W = cc Y + cn sum(Y nbrs) + cb B + cz Z
// (t = 0: Y = r -> y1; t = 1: Y = y1 -> y2; t = 2: Y = y2, Z = y1 -> z)
__device__ void ph_cheb0(const Dev& D, const Item& it, int t)
{
    const Prob& P = D.prob[it.q];
    if (!it.on) return;
    const long long sj = P.m + 4, sk = sj * sj;
    const float* Y = t == 0 ? D.r : (t == 1 ? D.y1 : D.y2);
    float* W = t == 0 ? D.y1 : (t == 1 ? D.y2 : D.z);
    const float cc = P.fcc[t], cn = P.fcn[t], cb = P.fcb[t], cz = P.fcz[t];
    long long c = idx0(P, it.i, it.j, it.k0);
    float ym = Y[c - sk], yc = Y[c];   // the planes below and above carried along the march
    for (int k = it.k0; k < it.k1; k++, c += sk) {
        const float yp = Y[c + sk];
        float w = fmaf(cn, ((Y[c - 1] + Y[c + 1]) + (Y[c - sj] + Y[c + sj])) + (ym + yp), cc * yc);
        if (t > 0) w = fmaf(cb, D.r[c], w);
        if (t == 2) w = fmaf(cz, D.y1[c], w);
        W[c] = w;
        ym = yc;
        yc = yp;
    }
}

// fine residual t0 = r - A z
__device__ void ph_r0(const Dev& D, const Item& it)
{
    const Prob& P = D.prob[it.q];
    if (!it.on) return;
    const long long sj = P.m + 4, sk = sj * sj;
    const float ih2 = (float)P.ih2;
    long long c = idx0(P, it.i, it.j, it.k0);
    float zm = D.z[c - sk], zc = D.z[c];   // the planes below and above carried along the march
    for (int k = it.k0; k < it.k1; k++, c += sk) {
        const float zp = D.z[c + sk];
        D.t0[c] = D.r[c] - ((((D.z[c - 1] + D.z[c + 1]) + (D.z[c - sj] + D.z[c + sj])) + (zm + zp)) - 6.f * zc) * ih2;
        zm = zc;
        zc = zp;
    }
}

// full-weighting restriction onto level lc (its unknown c on the finer level's 2c+1),
// from t0 (lc = 1) or the finer level's residual ct.  A thread marches its coarse
// column: the weighted 3 x 3 sum of a fine plane serves the coarse planes on either side,
// and the third point of a fine row is the next lane's first.
__device__ void ph_restrict(const Dev& D, const Item& it, int lc)
{
    const Prob& P = D.prob[it.q];
    const int nf = P.n[lc - 1], n = P.n[lc], lane = threadIdx.x & 31;
    const float* f = lc == 1 ? D.t0 : D.ct;
    const long long sj = lc == 1 ? P.m + 4 : nf, sk = sj * sj;
    const long long base = lc == 1 ? idx0(P, 2 * it.i, 2 * it.j, 0) : P.coff[lc - 1] + 2 * it.i + sj * (2 * it.j);
    const bool x2 = 2 * it.i + 2 < nf, y2 = 2 * it.j + 2 < nf;
    auto plane = [&](int k) -> float {
        float s = 0.f;
#pragma unroll
        for (int b = 0; b < 3; b++) {
            const bool in = it.on && k < nf && (b < 2 || y2);
            float u = 0.f, v = 0.f;
            const long long c = base + sj * b + sk * k;
            if (in) {
                const float2 t = *reinterpret_cast<const float2*>(f + c);   // nf and c are even
                u = t.x;
                v = t.y;
            }
            float w = __shfl_down_sync(0xffffffffu, u, 1);
            if (lane == 31) w = in && x2 ? f[c + 2] : 0.f;
            if (!x2) w = 0.f;
            s = fmaf(b == 1 ? 0.5f : 0.25f, fmaf(0.25f, w, fmaf(0.5f, v, 0.25f * u)), s);
        }
        return s;
    };
    float below = plane(2 * it.k0);
    for (int k = it.k0; k < it.k1; k++) {
        const float mid = plane(2 * k + 1), above = plane(2 * k + 2);
        if (it.on)
            D.cr[P.coff[lc] + it.i + (long long)n * (it.j + (long long)n * k)] = fmaf(0.25f, above, fmaf(0.5f, mid, 0.25f * below));
        below = above;
    }
}

// The weights of a level's 7-point operator in one column: a neighbour's is zero where
// it is the wall; the lower neighbour's and the centre's differ at the last unknown of an
// axis.  [e]: e = 1 on the level's last plane.  dinv: 1 / -diag.
struct LCol {
    float xm, xp, ym, yp, zm[2], ndg[2], dinv[2];
};
__device__ __forceinline__ float lvl_ndiag(const Prob& P, int l, bool lx, bool ly, bool lz)
{
    return (lx ? -P.lastc[l] : 2.f * P.lih2[l]) + (ly ? -P.lastc[l] : 2.f * P.lih2[l]) + (lz ? -P.lastc[l] : 2.f * P.lih2[l]);
}
__device__ __forceinline__ LCol lvl_col(const Prob& P, int l, int i, int j)
{
    const int n = P.n[l];
    const bool lx = i == n - 1, ly = j == n - 1;
    LCol C;
    C.xm = i > 0 ? (lx ? P.lastm[l] : P.lih2[l]) : 0.f;
    C.xp = lx ? 0.f : P.lih2[l];
    C.ym = j > 0 ? (ly ? P.lastm[l] : P.lih2[l]) : 0.f;
    C.yp = ly ? 0.f : P.lih2[l];
    C.zm[0] = P.lih2[l];
    C.zm[1] = P.lastm[l];
    for (int e = 0; e < 2; e++) {
        C.ndg[e] = lvl_ndiag(P, l, lx, ly, e);
        C.dinv[e] = 1.f / C.ndg[e];
    }
    return C;
}

// Jacobi-scaled Chebyshev on level l, on the interval [2/RATIO, 2] of D^-1 A_l:
//   s0 = D^-1 b / theta;  s1 = a1 s0 + b1 D^-1 (b + A s0);
//   X = -(a2 s1 + b2 D^-1 (b + A s1) - c2 s0)
// step 1 writes s1 (cc1); step 2 writes X into z (up: adds it).  b is r_l (down leg)
// or t_l (up leg).
__device__ void ph_jcheb(const Dev& D, const Item& it, int l, int step, bool up)
{
    const Prob& P = D.prob[it.q];
    if (!it.on) return;
    const int n = P.n[l];
    const float* b = up ? D.ct : D.cr;
    const float ih2 = P.lih2[l];
    const long long sj = n, sk = (long long)n * n;
    const LCol C = lvl_col(P, l, it.i, it.j);
    long long c = P.coff[l] + it.i + sj * it.j + sk * it.k0;
    if (step == 1) {
        // A s0 needs s0 = D^-1 b / theta at the neighbours, whose D differ where they are
        // the last unknown of an axis: one factor per neighbour and plane kind
        const bool lx = it.i == n - 1, ly = it.j == n - 1;
        float fc[2], fxm[2], fxp[2], fym[2], fyp[2];
        for (int e = 0; e < 2; e++) {
            fc[e] = C.dinv[e] * D.jt;
            fxm[e] = it.i > 0 ? D.jt / lvl_ndiag(P, l, false, ly, e) * C.xm : 0.f;
            fxp[e] = !lx ? D.jt / lvl_ndiag(P, l, it.i + 1 == n - 1, ly, e) * C.xp : 0.f;
            fym[e] = it.j > 0 ? D.jt / lvl_ndiag(P, l, lx, false, e) * C.ym : 0.f;
            fyp[e] = !ly ? D.jt / lvl_ndiag(P, l, lx, it.j + 1 == n - 1, e) * C.yp : 0.f;
        }
        const long long xm = it.i > 0 ? -1 : 0, xp = lx ? 0 : 1, ym = it.j > 0 ? -sj : 0, yp = ly ? 0 : sj;
        float bv = b[c];
        float sm = it.k0 > 0 ? b[c - sk] * fc[0] : 0.f, s0 = bv * fc[it.k0 == n - 1];
        for (int k = it.k0; k < it.k1; k++, c += sk) {
            const int e = k == n - 1;
            const float bn = e ? 0.f : b[c + sk];
            const float sp = bn * fc[k + 1 == n - 1];   // zero above the last plane
            float as = -C.ndg[e] * s0;
            as = fmaf(fxm[e], b[c + xm], as);
            as = fmaf(fxp[e], b[c + xp], as);
            as = fmaf(fym[e], b[c + ym], as);
            as = fmaf(fyp[e], b[c + yp], as);
            as = fmaf(C.zm[e], sm, as);
            as = fmaf(ih2, sp, as);
            D.cc1[c] = fmaf(D.ja1, s0, D.jb1 * C.dinv[e] * (bv + as));
            sm = s0;
            s0 = sp;
            bv = bn;
        }
    } else {
        const float* u = D.cc1;
        const long long xm = it.i > 0 ? -1 : 0, xp = it.i == n - 1 ? 0 : 1, ym = it.j > 0 ? -sj : 0, yp = it.j == n - 1 ? 0 : sj;
        float um = it.k0 > 0 ? u[c - sk] : 0.f, uc = u[c];
        for (int k = it.k0; k < it.k1; k++, c += sk) {
            const int e = k == n - 1;
            const float un = e ? 0.f : u[c + sk], bv = b[c];
            float as = -C.ndg[e] * uc;
            as = fmaf(C.xm, u[c + xm], as);
            as = fmaf(C.xp, u[c + xp], as);
            as = fmaf(C.ym, u[c + ym], as);
            as = fmaf(C.yp, u[c + yp], as);
            as = fmaf(C.zm[e], um, as);
            as = fmaf(ih2, un, as);
            const float X = -(fmaf(D.ja2, uc, D.jb2 * C.dinv[e] * (bv + as)) - D.jc2 * (C.dinv[e] * bv * D.jt));
            D.cz[c] = up ? D.cz[c] + X : X;
            um = uc;
            uc = un;
        }
    }
}

// t_l = r_l - A_l z_l
__device__ void ph_lres(const Dev& D, const Item& it, int l)
{
    const Prob& P = D.prob[it.q];
    if (!it.on) return;
    const int n = P.n[l];
    const long long sj = n, sk = (long long)n * n;
    const LCol C = lvl_col(P, l, it.i, it.j);
    const float* u = D.cz;
    const long long xm = it.i > 0 ? -1 : 0, xp = it.i == n - 1 ? 0 : 1, ym = it.j > 0 ? -sj : 0, yp = it.j == n - 1 ? 0 : sj;
    long long c = P.coff[l] + it.i + sj * it.j + sk * it.k0;
    float um = it.k0 > 0 ? u[c - sk] : 0.f, uc = u[c];
    for (int k = it.k0; k < it.k1; k++, c += sk) {
        const int e = k == n - 1;
        const float un = e ? 0.f : u[c + sk];
        float a = -C.ndg[e] * uc;
        a = fmaf(C.xm, u[c + xm], a);
        a = fmaf(C.xp, u[c + xp], a);
        a = fmaf(C.ym, u[c + ym], a);
        a = fmaf(C.yp, u[c + yp], a);
        a = fmaf(C.zm[e], um, a);
        a = fmaf(P.lih2[l], un, a);
        D.ct[c] = D.cr[c] - a;
        um = uc;
        uc = un;
    }
}

// One column's coarse line in (x, y): fine i odd takes coarse i/2, even the mean of i/2 - 1
// and i/2 (the wall's zero below the first).  The column's value on coarse plane cz.
struct PCol {
    long long aa, ab, ba, bb;
    float waa, wab, wba, wbb;
};
__device__ __forceinline__ PCol pro_col(int nc, int i, int j)
{
    PCol C;
    const int xb = i >> 1, xa = (i & 1) || xb == 0 ? xb : xb - 1, yb = j >> 1, ya = (j & 1) || yb == 0 ? yb : yb - 1;
    const float wxb = i & 1 ? 1.f : 0.5f, wxa = i & 1 || i == 0 ? 0.f : 0.5f;
    const float wyb = j & 1 ? 1.f : 0.5f, wya = j & 1 || j == 0 ? 0.f : 0.5f;
    C.aa = xa + (long long)nc * ya;
    C.ab = xb + (long long)nc * ya;
    C.ba = xa + (long long)nc * yb;
    C.bb = xb + (long long)nc * yb;
    C.waa = wxa * wya;
    C.wab = wxb * wya;
    C.wba = wxa * wyb;
    C.wbb = wxb * wyb;
    return C;
}
__device__ __forceinline__ float pro_plane(const float* zc, const PCol& C)
{
    return fmaf(C.waa, zc[C.aa], fmaf(C.wab, zc[C.ab], fmaf(C.wba, zc[C.ba], C.wbb * zc[C.bb])));
}

// z_l += P z_{l+1} on level l >= 1: a coarse plane is interpolated once for the two fine
// planes it covers
__device__ void ph_up(const Dev& D, const Item& it, int l)
{
    const Prob& P = D.prob[it.q];
    if (!it.on) return;
    const int n = P.n[l], nc = P.n[l + 1];
    const long long sk = (long long)n * n, sc = (long long)nc * nc;
    const PCol C = pro_col(nc, it.i, it.j);
    const float* zc = D.cz + P.coff[l + 1];
    long long c = P.coff[l] + it.i + (long long)n * it.j + sk * it.k0;
    int h = it.k0 >> 1;
    float below = !(it.k0 & 1) && h > 0 ? pro_plane(zc + sc * (h - 1), C) : 0.f;
    float cur = pro_plane(zc + sc * h, C);
    for (int k = it.k0; k < it.k1; k++, c += sk) {
        D.cz[c] += k & 1 ? cur : 0.5f * (below + cur);
        if (k & 1) {
            below = cur;
            h++;
            if (k + 1 < it.k1) cur = pro_plane(zc + sc * h, C);
        }
    }
}

// level 0: z += P z_1, then sums z.r and z.Ap
__device__ void ph_p0(const Dev& D, const Item& it, Acc<float>& a1, Acc<float>& a2)
{
    const Prob& P = D.prob[it.q];
    if (!it.on) return;
    const int nc = P.n[1];
    const long long sk = (long long)(P.m + 4) * (P.m + 4), sc = (long long)nc * nc;
    const PCol C = pro_col(nc, it.i, it.j);
    const float* zc = D.cz + P.coff[1];
    long long c = idx0(P, it.i, it.j, it.k0);
    int h = it.k0 >> 1;
    float below = !(it.k0 & 1) && h > 0 ? pro_plane(zc + sc * (h - 1), C) : 0.f;
    float cur = pro_plane(zc + sc * h, C);
    for (int k = it.k0; k < it.k1; k++, c += sk) {
        const float zv = D.z[c] + (k & 1 ? cur : 0.5f * (below + cur));
        D.z[c] = zv;
        a1.add(zv, D.r[c]);
        a2.add(zv, D.ap[c]);
        if (k & 1) {
            below = cur;
            h++;
            if (k + 1 < it.k1) cur = pro_plane(zc + sc * h, C);
        }
    }
}

// ---- level 0 in quads ----
// Edges that are a multiple of 4: a thread owns four consecutive points of a row, 8, 16 or
// 32 lanes a row (the FP32 pools are shifted so that the first unknown of a row lies on
// a 16-byte boundary).  The x neighbours come by shuffle within the row's lanes, the
// others are quad loads, z carried along the march.  Lanes off the grid take part in
// the shuffles and touch no memory.  (No pointer here is __restrict__: what one phase
// writes the next reads in the same launch, which the read-only load path does not see.)  One column per thread spent 14 scalar loads a point
// on the direction phase alone and was bound by the L1 path.

__device__ __forceinline__ float4 ldq(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void stq(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ float4 operator+(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }
__device__ __forceinline__ float4 fma4(float s, float4 a, float4 b)
{
    return make_float4(fmaf(s, a.x, b.x), fmaf(s, a.y, b.y), fmaf(s, a.z, b.z), fmaf(s, a.w, b.w));
}
__device__ __forceinline__ float4 scale4(float s, float4 a) { return make_float4(s * a.x, s * a.y, s * a.z, s * a.w); }
__device__ __forceinline__ void add4(Acc<float>& acc, float4 a, float4 b)
{
    acc.add(a.x, b.x);
    acc.add(a.y, b.y);
    acc.add(a.z, b.z);
    acc.add(a.w, b.w);
}
// sums of the x neighbours of quad u; beyond the row's lanes: `left` and `right`, read by
// the end lanes (a guard cell's zero, or the next tile of a row longer than 32 quads)
__device__ __forceinline__ float4 xsum4(const Item& it, float4 u, float left, float right)
{
    const float a = __shfl_up_sync(0xffffffffu, u.w, 1, it.lw), b = __shfl_down_sync(0xffffffffu, u.x, 1, it.lw);
    if (it.l != 0) left = a;
    if (it.l != it.lw - 1) right = b;
    return make_float4(left + u.y, u.x + u.z, u.y + u.w, u.z + right);
}

// FCG direction p_out = z + beta p_in, Ap = A p_out, sum p_out.Ap
__device__ void pq_a_fcg(const Dev& D, const Item& it, Acc<float>& acc)
{
    const Prob& P = D.prob[it.q];
    const State& S = D.st[it.q];
    const long long sj = P.m + 4, sk = sj * sj;
    const float* z = D.z;
    const float* pin = S.par ? D.pb : D.pa;
    float* pout = S.par ? D.pa : D.pb;
    const float be = (float)S.beta, ih2 = (float)P.ih2;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const bool on = it.on, plain = be == 0.f;
    const bool el = on && it.l == 0 && it.i > 0, er = on && it.l == it.lw - 1 && it.i + 4 < P.m;
    auto dir = [&](long long c) { return !on ? zero : plain ? ldq(z + c) : fma4(be, ldq(pin + c), ldq(z + c)); };
    auto dir1 = [&](long long c) { return plain ? z[c] : fmaf(be, pin[c], z[c]); };
    long long c = idx0(P, it.i, it.j, it.k0);
    float4 pm = dir(c - sk), pc = dir(c);
    for (int k = it.k0; k < it.k1; k++, c += sk) {
        const float4 pp = dir(c + sk);
        const float4 ya = dir(c - sj), yb = dir(c + sj);
        const float4 s = (xsum4(it, pc, el ? dir1(c - 1) : 0.f, er ? dir1(c + 4) : 0.f) + (ya + yb)) + (pm + pp);
        const float4 a = scale4(ih2, fma4(-6.f, pc, s));
        if (on) {
            stq(pout + c, pc);
            stq(D.ap + c, a);
            add4(acc, pc, a);
        }
        pm = pc;
        pc = pp;
    }
}

__device__ void pq_b_fcg(const Dev& D, const Item& it, Acc<float>& acc)
{
    const Prob& P = D.prob[it.q];
    const State& S = D.st[it.q];
    if (!it.on) return;
    const long long sk = (long long)(P.m + 4) * (P.m + 4);
    const float* p = S.par ? D.pb : D.pa;   // the direction phase A wrote (its parity flipped since)
    const float* ap = D.ap;
    float* e = D.e;
    float* r = D.r;
    const float al = (float)S.alpha;
    long long c = idx0(P, it.i, it.j, it.k0);
#pragma unroll 2
    for (int k = it.k0; k < it.k1; k++, c += sk) {
        const float4 ev = fma4(al, ldq(p + c), ldq(e + c)), rn = fma4(-al, ldq(ap + c), ldq(r + c));
        stq(e + c, ev);
        stq(r + c, rn);
        add4(acc, rn, rn);
    }
}

__device__ void pq_a_refine(const Dev& D, const Item& it)
{
    const Prob& P = D.prob[it.q];
    if (!it.on) return;
    const long long sk = (long long)(P.m + 4) * (P.m + 4);
    long long c = idx0(P, it.i, it.j, it.k0);
    const bool first = D.st[it.q].refinements == 0;   // no correction yet
    for (int k = it.k0; k < it.k1; k++, c += sk) {
        if (!first) {
            const float4 ev = ldq(D.e + c);
            double2* x = reinterpret_cast<double2*>(D.x + c);
            double2 a = x[0], b = x[1];
            if (ev.x != 0.f) a.x += (double)ev.x;
            if (ev.y != 0.f) a.y += (double)ev.y;
            if (ev.z != 0.f) b.x += (double)ev.z;
            if (ev.w != 0.f) b.y += (double)ev.w;
            x[0] = a;
            x[1] = b;
        }
        stq(D.e + c, make_float4(0.f, 0.f, 0.f, 0.f));
    }
}

// refinement residual in FP64, two columns at a time
__device__ void pq_b_refine(const Dev& D, const Item& it, double& acc)
{
    const Prob& P = D.prob[it.q];
    if (!it.on) return;
    const long long sj = P.m + 4, sk = sj * sj;
    const double* x = D.x;
    const double* b = D.b;
    const bool fb = from_b(D.st[it.q]);
    auto ld2 = [](const double* p) { return *reinterpret_cast<const double2*>(p); };
    for (int h = 0; h < 2; h++) {
        long long c = idx0(P, it.i + 2 * h, it.j, it.k0);
        double2 xm = make_double2(0.0, 0.0), xc = xm;
        if (!fb) {
            xm = ld2(x + c - sk);
            xc = ld2(x + c);
        }
        for (int k = it.k0; k < it.k1; k++, c += sk) {
            double2 rv = ld2(b + c);
            if (!fb) {
                const double2 xp = ld2(x + c + sk), ya = ld2(x + c - sj), yb = ld2(x + c + sj);
                const double s0 = ((x[c - 1] + xc.y) + (ya.x + yb.x)) + (xm.x + xp.x);
                const double s1 = ((xc.x + x[c + 2]) + (ya.y + yb.y)) + (xm.y + xp.y);
                rv.x -= (s0 - 6.0 * xc.x) * P.ih2;
                rv.y -= (s1 - 6.0 * xc.y) * P.ih2;
                xm = xc;
                xc = xp;
            }
            *reinterpret_cast<float2*>(D.r + c) = make_float2((float)rv.x, (float)rv.y);
            acc = fma(rv.x, rv.x, acc);
            acc = fma(rv.y, rv.y, acc);
        }
    }
}

// fine Chebyshev step t (ph_cheb0), or, t = 3, the fine residual t0 = r - A z (ph_r0)
template <int t>
__device__ void pq_cheb0(const Dev& D, const Item& it)
{
    const Prob& P = D.prob[it.q];
    const long long sj = P.m + 4, sk = sj * sj;
    const float* Y = t == 0 ? D.r : t == 1 ? D.y1 : t == 2 ? D.y2 : D.z;
    const float* B = D.r;
    const float* Z = D.y1;
    float* W = t == 0 ? D.y1 : t == 1 ? D.y2 : t == 2 ? D.z : D.t0;
    const float cc = t < 3 ? P.fcc[t < 3 ? t : 0] : 6.f * (float)P.ih2, cn = t < 3 ? P.fcn[t < 3 ? t : 0] : -(float)P.ih2;
    const float cb = t < 3 ? P.fcb[t < 3 ? t : 0] : 1.f, cz = t < 3 ? P.fcz[t < 3 ? t : 0] : 0.f;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const bool on = it.on;
    const bool el = on && it.l == 0 && it.i > 0, er = on && it.l == it.lw - 1 && it.i + 4 < P.m;
    auto ld = [&](long long c) { return on ? ldq(Y + c) : zero; };
    long long c = idx0(P, it.i, it.j, it.k0);
    float4 ym = ld(c - sk), yc = ld(c);
    for (int k = it.k0; k < it.k1; k++, c += sk) {
        const float4 yp = ld(c + sk), ya = ld(c - sj), yb = ld(c + sj);
        const float4 s = (xsum4(it, yc, el ? Y[c - 1] : 0.f, er ? Y[c + 4] : 0.f) + (ya + yb)) + (ym + yp);
        float4 w = fma4(cn, s, scale4(cc, yc));
        if (on) {
            if (t > 0) w = fma4(cb, ldq(B + c), w);
            if (t == 2) w = fma4(cz, ldq(Z + c), w);
            stq(W + c, w);
        }
        ym = yc;
        yc = yp;
    }
}

// z += P z_1 and the sums z.r, z.Ap.  The quad at i = 4l takes coarse 2l - 1 .. 2l + 1:
// two from one load, the first from the lane below.
__device__ void pq_p0(const Dev& D, const Item& it, Acc<float>& a1, Acc<float>& a2)
{
    const Prob& P = D.prob[it.q];
    const int nc = P.n[1];
    const long long sk = (long long)(P.m + 4) * (P.m + 4), sc = (long long)nc * nc;
    const bool on = it.on;
    const int h0 = it.i >> 1, yb = it.j >> 1;
    const float wb = it.j & 1 ? 1.f : 0.5f;
    const bool two = !(it.j & 1) && yb > 0;
    const float* zc = D.cz + P.coff[1] + h0 + (long long)nc * yb;
    auto line = [&](int h) -> float4 {   // the quad on coarse plane h
        float2 v = make_float2(0.f, 0.f);
        float left = 0.f;
        if (on) {
            const float* p = zc + sc * h;
            v = *reinterpret_cast<const float2*>(p);
            if (it.l == 0 && h0 > 0) left = p[-1];
            v.x *= wb;
            v.y *= wb;
            left *= wb;
            if (two) {
                const float2 u = *reinterpret_cast<const float2*>(p - nc);
                v.x = fmaf(0.5f, u.x, v.x);
                v.y = fmaf(0.5f, u.y, v.y);
                if (it.l == 0 && h0 > 0) left = fmaf(0.5f, p[-nc - 1], left);
            }
        }
        const float a = __shfl_up_sync(0xffffffffu, v.y, 1, it.lw);
        if (it.l != 0) left = a;
        return make_float4(0.5f * (left + v.x), v.x, 0.5f * (v.x + v.y), v.y);
    };
    const float* r = D.r;
    const float* ap = D.ap;
    float* z = D.z;
    long long c = idx0(P, it.i, it.j, it.k0);
    int h = it.k0 >> 1;
    float4 below = make_float4(0.f, 0.f, 0.f, 0.f), cur = line(h);
    if (!(it.k0 & 1) && h > 0) below = line(h - 1);
    for (int k = it.k0; k < it.k1; k++, c += sk) {
        if (on) {
            const float4 zv = ldq(z + c) + (k & 1 ? cur : scale4(0.5f, below + cur));
            stq(z + c, zv);
            add4(a1, zv, ldq(r + c));
            add4(a2, zv, ldq(ap + c));
        }
        if (k & 1) {
            below = cur;
            h++;
            if (k + 1 < it.k1) cur = line(h);
        }
    }
}

// z_k = A_k^-1 r_k on the coarsest level, the whole level in shared memory (one block):
// passes along x, y, z with V^-1, the eigenvalue division, passes with V
// (matrices as unet::level_exact_data lays them out).  A thread transforms whole lines,
// held in registers (NM >= n; a run-time length left them in local memory); rows have
// an odd pitch, so that lines along x start in different banks, and the matrices' rows a
// multiple of 4, so that one load brings four weights (one a product was the limit).
template <int NM>
__device__ void exact_passes(float* cube, const float* M, int n, int px)
{
    const int tot = n * n * n, pn = (n + 3) & ~3;
    for (int pass = 0; pass < 7; pass++) {
        if (pass == 3) {
            const float* lam = M + 6 * n * pn;
            for (int i = threadIdx.x; i < tot; i += NT) {
                const int xi = i % n, yi = (i / n) % n, zi = i / (n * n);
                float* v = cube + xi + px * (yi + n * zi);
                *v = *v / (lam[xi] + lam[n + yi] + lam[2 * n + zi]);
            }
        } else {
            const int axis = pass < 3 ? pass : pass - 4;
            const float* Mat = M + (pass < 3 ? axis : 3 + axis) * n * pn;
            const int stride = axis == 0 ? 1 : axis == 1 ? px : px * n;
            for (int t = threadIdx.x; t < n * n; t += NT) {
                const int a = t % n, b = t / n;
                float* line = cube + (axis == 0 ? px * t : axis == 1 ? a + px * n * b : a + px * b);
                float v[NM];
#pragma unroll
                for (int m = 0; m < NM; m++) v[m] = m < n ? line[m * stride] : 0.f;
                for (int i = 0; i < n; i++) {
                    float acc = 0.f;
#pragma unroll
                    for (int m = 0; m < NM; m += 4)
                        if (m < n) {   // the padding's weights and values are zero
                            const float4 w = *reinterpret_cast<const float4*>(Mat + i * pn + m);
                            acc = fmaf(w.x, v[m], acc);
                            acc = fmaf(w.y, v[m + 1], acc);
                            acc = fmaf(w.z, v[m + 2], acc);
                            acc = fmaf(w.w, v[m + 3], acc);
                        }
                    line[i * stride] = acc;
                }
            }
        }
        __syncthreads();
    }
}
__device__ void ph_exact(const Dev& D, int q, float* sm)
{
    const Prob& P = D.prob[q];
    const int n = P.n[P.k], px = n | 1, tot = n * n * n;
    float* cube = sm;
    const int pn = (n + 3) & ~3;
    float* M = sm + ((px * n * n + 3) & ~3);
    const float* src = D.mats + P.mats;
    for (int i = threadIdx.x; i < 6 * n * pn; i += NT) M[i] = i % pn < n ? src[i / pn * n + i % pn] : 0.f;
    for (int i = threadIdx.x; i < 3 * n; i += NT) M[6 * n * pn + i] = src[6 * n * n + i];
    const long long base = P.coff[P.k];
    for (int i = threadIdx.x; i < tot; i += NT) cube[i % n + px * (i / n)] = D.cr[base + i];
    __syncthreads();
    if (n <= 8) exact_passes<8>(cube, M, n, px);
    else if (n <= 16) exact_passes<16>(cube, M, n, px);
    else exact_passes<32>(cube, M, n, px);
    for (int i = threadIdx.x; i < tot; i += NT) D.cz[base + i] = cube[i % n + px * (i / n)];
    __syncthreads();
}

// Is problem q part of this phase?  (uniform over a block)
__device__ __forceinline__ bool takes_part(const Dev& D, const Phase& ph, int q)
{
    const State& S = D.st[q];
    if (S.done) return false;
    if (ph.type == PH_NORM || ph.type == PH_A || ph.type == PH_B) return true;
    if (S.skip) return false;
    const int k = D.prob[q].k;
    switch (ph.type) {
    case PH_RS:
        return ph.level + 1 <= k;
    case PH_D1: case PH_D2: case PH_DR: case PH_UP: case PH_UR: case PH_U1: case PH_U2:
        return ph.level < k;
    default:
        return true;
    }
}

// The level whose work items a phase covers.
__device__ __forceinline__ int item_level(const Phase& ph)
{
    switch (ph.type) {
    case PH_RS:
        return ph.level + 1;
    case PH_D1: case PH_D2: case PH_DR: case PH_UP: case PH_UR: case PH_U1: case PH_U2:
        return ph.level;
    default:
        return 0;
    }
}

__device__ void run_phase(const Dev& D, const Phase& ph, float* sm)
{
    if (ph.type == PH_EX) {
        for (int q = blockIdx.x; q < D.nprob; q += gridDim.x)
            if (takes_part(D, ph, q)) ph_exact(D, q, sm);
        return;
    }
    const int lev = item_level(ph);
    const long long* row = D.toff + (long long)lev * (D.nprob + 1);
    const long long total = row[D.nprob];
    for (long long item = blockIdx.x; item < total; item += gridDim.x) {
        const Item it = decode(D, lev, item, ph.type != PH_RS && lev == 0);
        if (!takes_part(D, ph, it.q)) continue;
        const bool quads = it.lw > 0;
        const State& S = D.st[it.q];
        const long long first = row[it.q], count = row[it.q + 1] - row[it.q];
        double tot[2];
        switch (ph.type) {
        case PH_NORM: {
            double v[1] = {0.0};
            unsigned long long nz = 0;
            ph_norm(D, it, v[0], nz);
            if (__syncthreads_or(nz != 0) && threadIdx.x == 0) D.st[it.q].xnz = 1;
            if (item_reduce<1>(D, it, first, count, v, tot)) advance(D, it.q, PH_NORM, tot);
            break;
        }
        case PH_A:
            if (S.mode == 1) {
                Acc<float> a;
                if (quads) pq_a_fcg(D, it, a);
                else ph_a_fcg(D, it, a);
                double v[1] = {a.value()};
                if (item_reduce<1>(D, it, first, count, v, tot)) advance(D, it.q, PH_A, tot);
            } else if (quads) {
                pq_a_refine(D, it);
            } else {
                ph_a_refine(D, it);
            }
            break;
        case PH_B:
            if (S.mode == 1) {
                Acc<float> a;
                if (quads) pq_b_fcg(D, it, a);
                else ph_b_fcg(D, it, a);
                double v[1] = {a.value()};
                if (item_reduce<1>(D, it, first, count, v, tot)) advance(D, it.q, PH_B, tot);
            } else {
                double v[1] = {0.0};
                if (quads) pq_b_refine(D, it, v[0]);
                else ph_b_refine(D, it, v[0]);
                if (item_reduce<1>(D, it, first, count, v, tot)) advance(D, it.q, PH_B, tot);
            }
            break;
        case PH_C1:
            if (quads) pq_cheb0<0>(D, it);
            else ph_cheb0(D, it, 0);
            break;
        case PH_C2:
            if (quads) pq_cheb0<1>(D, it);
            else ph_cheb0(D, it, 1);
            break;
        case PH_C3:
            if (quads) pq_cheb0<2>(D, it);
            else ph_cheb0(D, it, 2);
            break;
        case PH_R0:
            if (quads) pq_cheb0<3>(D, it);
            else ph_r0(D, it);
            break;
        case PH_RS: ph_restrict(D, it, ph.level + 1); break;
        case PH_D1: ph_jcheb(D, it, ph.level, 1, false); break;
        case PH_D2: ph_jcheb(D, it, ph.level, 2, false); break;
        case PH_DR: ph_lres(D, it, ph.level); break;
        case PH_UR: ph_lres(D, it, ph.level); break;
        case PH_UP: ph_up(D, it, ph.level); break;
        case PH_U1: ph_jcheb(D, it, ph.level, 1, true); break;
        case PH_U2: ph_jcheb(D, it, ph.level, 2, true); break;
        case PH_P0: {
            Acc<float> a1, a2;
            if (quads) pq_p0(D, it, a1, a2);
            else ph_p0(D, it, a1, a2);
            double v[2] = {a1.value(), a2.value()};
            if (item_reduce<2>(D, it, first, count, v, tot)) advance(D, it.q, PH_P0, tot);
            break;
        }
        default:
            break;
        }
    }
}

// The persistent solve: the norm phase, then rounds of the phase program until every
// problem has finished (or max_rounds), a grid barrier after every phase.  All blocks
// read `unfinished` after the same barrier, so they leave the loop together.
__global__ void __launch_bounds__(NT, 4) k_bvc_solve(const __grid_constant__ Dev D)
{
    pdl_enter();
    extern __shared__ __align__(16) float sm_ex[];
    run_phase(D, Phase{PH_NORM, 0}, sm_ex);
    if (!grid_barrier(D)) return;
    for (int round = 0; round < D.max_rounds; round++) {
        for (int p = 0; p < D.nphases; p++) {
            run_phase(D, D.phases[p], sm_ex);
            if (!grid_barrier(D)) return;
        }
        if (*(volatile int*)D.unfinished == 0) break;
    }
}

// Initial state of every problem (one thread per problem), counters and barrier.
__global__ void k_bvc_init(Dev D)
{
    pdl_enter();
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q == 0) {
        D.bar->count = 0u;
        D.bar->gen = 0u;
        D.bar->error = 0;
        *D.unfinished = D.nprob;
    }
    if (q < D.nprob) {
        State s;
        memset(&s, 0, sizeof(s));
        D.st[q] = s;
        D.counters[q] = 0u;
    }
}

// ---- host ----

struct Plan {
    int nprob = 0;
    std::vector<Prob> prob;        // in the caller's order
    std::vector<int> slot;         // problem -> its row in the device table (largest first)
    std::vector<long long> toff;
    std::vector<Phase> phases;
    int maxk = 0;
    size_t ex_smem = 0;
    long long max_items = 0;
    Prob* dprob = nullptr;
    long long* dtoff = nullptr;
    int4* ditems = nullptr;
    Phase* dphases = nullptr;
    State* dst = nullptr;
    float *cr = nullptr, *cz = nullptr, *ct = nullptr, *cc1 = nullptr;
    float* dmats = nullptr;
    double* partials = nullptr;
    unsigned* counters = nullptr;
    Barrier* bar = nullptr;
    int* unfinished = nullptr;
    Dev D{};
    int grid = 0;
    double limit_s = 5.0;
    cudaGraphExec_t gexec = nullptr;
    std::vector<State> hst;
};

void free_plan(Plan* p)
{
    if (p->gexec) cudaGraphExecDestroy(p->gexec);
    void* ptrs[] = {p->dprob, p->dtoff, p->ditems, p->dphases, p->dst, p->cr, p->cz, p->ct, p->cc1, p->dmats, p->partials,
                    p->counters, p->bar, p->unfinished};
    for (void* q : ptrs)
        if (q) cudaFree(q);
}

// Chebyshev coefficients of the fine smoother (degree 5 on [lmax/RATIO, lmax] with
// lmax = 12/h^2, the preconditioner's recurrence, output X = -s3) in the form
// W = cc Y + cn sum(Y nbrs) + cb B + cz Z, A Y = (sum(Y nbrs) - 6 Y) / h^2:
//   s1 = (2 rho1 / delta) (2 B + A B / theta)
//   s2 = rho2 (2 sigma s1 + 2/delta (B + A s1)) - rho2 rho1 s0,  s0 = B / theta
//   X  = -(rho3 (2 sigma s2 + 2/delta (B + A s2)) - rho3 rho2 s1)
void fine_coefs(Prob& P, double h)
{
    const double ih2 = 1.0 / (h * h), hi = 12.0 * ih2, lo = hi / RATIO;
    const double theta = 0.5 * (lo + hi), delta = 0.5 * (lo - hi), sigma = theta / delta;
    const double rho0 = 1.0 / sigma, rho1 = 1.0 / (2.0 * sigma - rho0), rho2 = 1.0 / (2.0 * sigma - rho1),
                 rho3 = 1.0 / (2.0 * sigma - rho2);
    const double cy[3] = {4.0 * rho1 / delta, 2.0 * rho2 * sigma, -2.0 * rho3 * sigma};
    const double ca[3] = {2.0 * rho1 / (delta * theta), 2.0 * rho2 / delta, -2.0 * rho3 / delta};
    const double cb[3] = {0.0, 2.0 * rho2 / delta - rho2 * rho1 / theta, -2.0 * rho3 / delta};
    const double cz[3] = {0.0, 0.0, rho3 * rho2};
    for (int t = 0; t < 3; t++) {
        P.fcc[t] = (float)(cy[t] - 6.0 * ca[t] * ih2);
        P.fcn[t] = (float)(ca[t] * ih2);
        P.fcb[t] = (float)cb[t];
        P.fcz[t] = (float)cz[t];
    }
}

}  // namespace bvc

using namespace bvc;

#define VK(call)                                                                                   \
    do {                                                                                           \
        cudaError_t e_ = (call);                                                                   \
        if (e_ != cudaSuccess) {                                                                   \
            err = std::string(#call) + ": " + cudaGetErrorString(e_);                              \
            return fail();                                                                         \
        }                                                                                          \
    } while (0)

bool bvc_create(BvcPlan** out, int nprob, const Geo* geo, const long long* off, const BvcPools& pools, double tol,
                double inner_tol, int inner_maxit, int max_refinements, cudaStream_t s, std::string& err)
{
    *out = nullptr;
    Plan* P = new Plan();
    auto fail = [&]() {
        free_plan(P);
        delete P;
        return false;
    };
    P->nprob = nprob;
    P->prob.resize((size_t)nprob);
    long long cpool = 0;
    std::map<int, long long> mats_of;   // edge -> offset of its eigen-solve matrices
    std::vector<float> mats;
    for (int q = 0; q < nprob; q++) {
        const Geo& g = geo[q];
        const int m = g.n[0] - 2;
        if (g.n[1] != g.n[0] || g.n[2] != g.n[0] || g.ds[1] != g.ds[0] || g.ds[2] != g.ds[0]) {
            err = "the persistent V-cycle batch takes cubes with equal spacings";
            return fail();
        }
        Prob& pr = P->prob[(size_t)q];
        std::memset(&pr, 0, sizeof(pr));
        pr.m = m;
        pr.off = off[q];
        int k = 0, n = m;
        while (n > 16 && n % 2 == 0 && k + 1 < MAXLEV) {
            n /= 2;
            k++;
        }
        if (k < 1 || n > EX_MAX) {
            err = "the persistent V-cycle batch needs edges m = c * 2^k with k >= 1 and c <= 32 (m = " +
                  std::to_string(m) + ")";
            return fail();
        }
        pr.k = k;
        const double h = g.ds[0];
        pr.ih2 = 1.0 / (h * h);
        pr.lwlog = m % 4 != 0 ? 0 : m <= 32 ? 3 : m <= 64 ? 4 : 5;
        fine_coefs(pr, h);
        for (int l = 0; l <= k; l++) {
            const int nl = m >> l;
            pr.n[l] = nl;
            if (l >= 1) {
                const double H = h * (double)(1 << l);
                pr.lih2[l] = (float)(1.0 / (H * H));
                pr.lastm[l] = (float)(2.0 / (H * (H + h)));
                pr.lastc[l] = (float)(-2.0 / (H * h));
                pr.coff[l] = cpool;
                cpool += ((long long)nl * nl * nl + 31) / 32 * 32;
            }
        }
        auto it = mats_of.find(m);
        if (it == mats_of.end()) {
            unet::DLevel L;
            for (int d = 0; d < 3; d++) {
                L.ih2[d] = pr.lih2[k];
                L.last_m[d] = pr.lastm[k];
                L.last_c[d] = pr.lastc[k];
            }
            std::vector<float> mk;
            if (!unet::level_exact_data(unet::Dims{n, n, n}, L, mk)) {
                err = "coarsest level too large for the exact solve";
                return fail();
            }
            it = mats_of.emplace(m, (long long)mats.size()).first;
            mats.insert(mats.end(), mk.begin(), mk.end());
        }
        pr.mats = it->second;
        P->maxk = std::max(P->maxk, k);
        P->ex_smem = std::max(P->ex_smem, sizeof(float) * ((size_t)(n | 1) * n * n + 4 + 6 * (size_t)n * ((n + 3) & ~3) + 3 * (size_t)n));
    }
    // item order: largest problems first, so their items are handed out first
    std::vector<int> order((size_t)nprob);
    for (int q = 0; q < nprob; q++) order[(size_t)q] = q;
    std::stable_sort(order.begin(), order.end(),
                     [&](int a, int b) { return P->prob[(size_t)a].m > P->prob[(size_t)b].m; });
    std::vector<Prob> table((size_t)nprob);
    P->slot.resize((size_t)nprob);
    for (int t = 0; t < nprob; t++) {
        table[(size_t)t] = P->prob[(size_t)order[(size_t)t]];
        P->slot[(size_t)order[(size_t)t]] = t;
    }
    // one resident wave: the grid barrier needs every block resident
    VK(cudaFuncSetAttribute(k_bvc_solve, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)P->ex_smem));
    int per_sm = 0;
    VK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_bvc_solve, NT, P->ex_smem));
    if (per_sm < 1) {
        err = "the persistent kernel does not fit on an SM";
        return fail();
    }
    P->grid = per_sm * sm_count();
    // Work items of every level: a tile of columns (quads on level 0: 256 >> lwlog rows of
    // 1 << lwlog quads; else 32 x 8 columns) by a chunk of planes, block b taking items b,
    // b + grid and so on.  A chunk costs its planes and about 2 more (its start, the plane
    // on either side, the block sum), and the phase ends with its fullest block: of chunks
    // of 128 (coarse levels 16) down to 4 planes the level takes those for which that block
    // has the least to do.  (Chunks that leave 8 items a block, whatever the sizes: 200
    // problems of 26^3 5.32 ms, 30 of 62^3 20.2, 32 of 96^3 14.8; 4.02, 14.6 and 11.6 with
    // this; 250 of 32 to 128 57.8 and 57.4, none of 50 batches slower.  With 4 more planes a
    // chunk instead of 2, 30 of 40 to 80 took 6.67 ms, with 1 100 of 26^3 2.92; 6.21 and 2.17.)
    P->toff.assign((size_t)MAXLEV * (nprob + 1), 0);
    std::vector<int4> items;
    std::vector<size_t> items_at(MAXLEV + 1, 0);
    for (int l = 0; l < MAXLEV; l++) {
        auto tile = [&](const Prob& pr, int& w, int& hgt) {
            const bool quads = l == 0 && pr.lwlog > 0;
            w = quads ? 4 << pr.lwlog : 32;
            hgt = quads ? NT >> pr.lwlog : 8;
        };
        auto fullest = [&](int kz) -> long long {   // planes of the fullest block
            std::vector<long long> load((size_t)P->grid, 0);
            size_t b = 0;
            for (const Prob& pr : table) {
                if (l > pr.k) continue;
                int w, hgt;
                tile(pr, w, hgt);
                const int n = pr.n[l], tiles = ((n + w - 1) / w) * ((n + hgt - 1) / hgt);
                for (int k0 = 0; k0 < n; k0 += kz)
                    for (int q = 0; q < tiles; q++) {
                        load[b] += std::min(kz, n - k0) + 2;
                        b = b + 1 < load.size() ? b + 1 : 0;
                    }
            }
            return *std::max_element(load.begin(), load.end());
        };
        int kz = l == 0 ? KZ0 : KZ1;
        long long least = fullest(kz);
        for (int c = kz / 2; c >= 4; c /= 2) {
            const long long m = fullest(c);
            if (m < least) {
                least = m;
                kz = c;
            }
        }
        items_at[(size_t)l] = items.size();
        for (int t = 0; t < nprob; t++) {
            Prob& pr = table[(size_t)t];
            P->toff[(size_t)l * (nprob + 1) + t] = (long long)(items.size() - items_at[(size_t)l]);
            if (l > pr.k) continue;
            int w, hgt;
            tile(pr, w, hgt);
            const int n = pr.n[l];
            pr.kz[l] = std::min(n, kz);
            for (int k0 = 0; k0 < n; k0 += pr.kz[l])
                for (int j0 = 0; j0 < n; j0 += hgt)
                    for (int i0 = 0; i0 < n; i0 += w) items.push_back(make_int4(t, i0, j0, k0));
        }
        P->toff[(size_t)l * (nprob + 1) + nprob] = (long long)(items.size() - items_at[(size_t)l]);
        P->max_items = std::max(P->max_items, P->toff[(size_t)l * (nprob + 1) + nprob]);
    }
    // the phase program of one round
    auto add = [&](int type, int level) { P->phases.push_back(Phase{type, level}); };
    add(PH_A, 0);
    add(PH_B, 0);
    add(PH_C1, 0);
    add(PH_C2, 0);
    add(PH_C3, 0);
    add(PH_R0, 0);
    add(PH_RS, 0);
    for (int l = 1; l < P->maxk; l++) {
        add(PH_D1, l);
        add(PH_D2, l);
        add(PH_DR, l);
        add(PH_RS, l);
    }
    add(PH_EX, 0);
    for (int l = P->maxk - 1; l >= 1; l--) {
        add(PH_UP, l);
        add(PH_UR, l);
        add(PH_U1, l);
        add(PH_U2, l);
    }
    add(PH_P0, 0);

    const size_t cbytes = sizeof(float) * (size_t)std::max(cpool, 32LL);
    VK(cudaMalloc((void**)&P->dprob, sizeof(Prob) * (size_t)nprob));
    VK(cudaMalloc((void**)&P->dtoff, sizeof(long long) * P->toff.size()));
    VK(cudaMalloc((void**)&P->ditems, sizeof(int4) * std::max<size_t>(items.size(), 1)));
    VK(cudaMemcpyAsync(P->ditems, items.data(), sizeof(int4) * items.size(), cudaMemcpyHostToDevice, s));
    VK(cudaMalloc((void**)&P->dphases, sizeof(Phase) * P->phases.size()));
    VK(cudaMalloc((void**)&P->dst, sizeof(State) * (size_t)nprob));
    for (float** f : {&P->cr, &P->cz, &P->ct, &P->cc1}) {
        VK(cudaMalloc((void**)f, cbytes));
        VK(cudaMemsetAsync(*f, 0, cbytes, s));
    }
    VK(cudaMalloc((void**)&P->dmats, sizeof(float) * std::max<size_t>(mats.size(), 1)));
    VK(cudaMalloc((void**)&P->partials, sizeof(double) * 2 * (size_t)std::max<long long>(P->max_items, 1)));
    VK(cudaMalloc((void**)&P->counters, sizeof(unsigned) * (size_t)nprob));
    VK(cudaMalloc((void**)&P->bar, sizeof(Barrier)));
    VK(cudaMalloc((void**)&P->unfinished, sizeof(int)));
    VK(cudaMemcpyAsync(P->dprob, table.data(), sizeof(Prob) * (size_t)nprob, cudaMemcpyHostToDevice, s));
    VK(cudaMemcpyAsync(P->dtoff, P->toff.data(), sizeof(long long) * P->toff.size(), cudaMemcpyHostToDevice, s));
    VK(cudaMemcpyAsync(P->dphases, P->phases.data(), sizeof(Phase) * P->phases.size(), cudaMemcpyHostToDevice, s));
    if (!mats.empty())
        VK(cudaMemcpyAsync(P->dmats, mats.data(), sizeof(float) * mats.size(), cudaMemcpyHostToDevice, s));
    VK(cudaStreamSynchronize(s));

    // coarse Jacobi-Chebyshev constants on [2/RATIO, 2] (degree 4, output -s2)
    const double lo = 2.0 / RATIO, hi = 2.0, theta = 0.5 * (lo + hi), delta = 0.5 * (lo - hi), sigma = theta / delta;
    const double rho0 = 1.0 / sigma, rho1 = 1.0 / (2.0 * sigma - rho0), rho2 = 1.0 / (2.0 * sigma - rho1);
    Dev& D = P->D;
    D.prob = P->dprob;
    D.nprob = nprob;
    D.toff = P->dtoff;
    for (int l = 0; l < MAXLEV; l++) D.items[l] = P->ditems + items_at[(size_t)l];
    D.phases = P->dphases;
    D.nphases = (int)P->phases.size();
    D.st = P->dst;
    D.x = pools.x;
    D.b = pools.b;
    // two floats in: the first unknown of a row (index 2) then lies on a 16-byte boundary
    D.r = pools.r + 2;
    D.z = pools.z + 2;
    D.pa = pools.pa + 2;
    D.pb = pools.pb + 2;
    D.ap = pools.ap + 2;
    D.e = pools.e + 2;
    D.y1 = pools.y1 + 2;
    D.y2 = pools.y2 + 2;
    D.t0 = pools.t0 + 2;
    D.cr = P->cr;
    D.cz = P->cz;
    D.ct = P->ct;
    D.cc1 = P->cc1;
    D.mats = P->dmats;
    D.partials = P->partials;
    D.counters = P->counters;
    D.bar = P->bar;
    D.unfinished = P->unfinished;
    D.tol = tol;
    D.inner_tol = inner_tol;
    D.inner_maxit = inner_maxit;
    D.max_refinements = max_refinements;
    // a round is one FCG iteration or refinement step of every unfinished problem
    D.max_rounds = (int)std::min<long long>(2000, (long long)(max_refinements + 1) * (inner_maxit + 2));
    D.jt = (float)(1.0 / theta);
    D.ja1 = (float)(2.0 * rho1 * sigma);
    D.jb1 = (float)(2.0 * rho1 / delta);
    D.ja2 = (float)(2.0 * rho2 * sigma);
    D.jb2 = (float)(2.0 * rho2 / delta);
    D.jc2 = (float)(rho2 * rho1);
    P->hst.resize((size_t)nprob);
    *out = reinterpret_cast<BvcPlan*>(P);
    return true;
}

void bvc_destroy(BvcPlan* plan)
{
    if (!plan) return;
    Plan* P = reinterpret_cast<Plan*>(plan);
    free_plan(P);
    delete P;
}

void bvc_set_wait_limit(BvcPlan* plan, double seconds)
{
    Plan* P = reinterpret_cast<Plan*>(plan);
    P->limit_s = seconds;
    if (P->gexec) {   // the captured launch holds the old limit
        cudaGraphExecDestroy(P->gexec);
        P->gexec = nullptr;
    }
}

// Runs the persistent solve (replaying the captured graph), then reads the states.
// PPS_TIMEOUT when a barrier wait ran out; else the first failing problem's status
// (PPS_NOT_CONVERGED for one stopped short), or PPS_OK.
pps_status bvc_solve(BvcPlan* plan, cudaStream_t s, cudaEvent_t ev0, cudaEvent_t ev1, pps_batch_stats* stats,
                     std::string& err)
{
    Plan* P = reinterpret_cast<Plan*>(plan);
    auto ck = [&](cudaError_t e, const char* what) {
        if (e != cudaSuccess) err = std::string(what) + ": " + cudaGetErrorString(e);
        return e == cudaSuccess;
    };
    P->D.limit_ns = (unsigned long long)(P->limit_s * 1e9);
    if (!P->gexec) {
        cudaGraph_t gr = nullptr;
        if (!ck(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal), "cudaStreamBeginCapture"))
            return PPS_ERR_CUDA;
        {
            CaptureGuard cap(s);
            launch_pdl(k_bvc_init, (unsigned)((P->nprob + 255) / 256), 256, 0, s, P->D);
            launch_coop(k_bvc_solve, (unsigned)P->grid, NT, P->ex_smem, s, P->D);
            if (!ck(cap.end(&gr), "cudaStreamEndCapture")) return PPS_ERR_CUDA;
        }
        const cudaError_t ie = cudaGraphInstantiate(&P->gexec, gr, 0);
        cudaGraphDestroy(gr);
        if (ie != cudaSuccess) P->gexec = nullptr;
        if (!ck(ie, "cudaGraphInstantiate")) return PPS_ERR_CUDA;
    }
    if (!ck(cudaEventRecord(ev0, s), "cudaEventRecord")) return PPS_ERR_CUDA;
    if (!ck(cudaGraphLaunch(P->gexec, s), "cudaGraphLaunch")) return PPS_ERR_CUDA;
    if (!ck(cudaEventRecord(ev1, s), "cudaEventRecord")) return PPS_ERR_CUDA;
    if (!ck(cudaEventSynchronize(ev1), "cudaEventSynchronize")) return PPS_ERR_CUDA;
    float ms = 0.f;
    cudaEventElapsedTime(&ms, ev0, ev1);
    std::vector<State> table((size_t)P->nprob);
    Barrier bar;
    std::memset(&bar, 0, sizeof(bar));
    if (!ck(cudaMemcpyAsync(table.data(), P->dst, sizeof(State) * table.size(), cudaMemcpyDeviceToHost, s),
            "cudaMemcpyAsync") ||
        !ck(cudaMemcpyAsync(&bar, P->bar, sizeof(Barrier), cudaMemcpyDeviceToHost, s), "cudaMemcpyAsync") ||
        !ck(cudaStreamSynchronize(s), "cudaStreamSynchronize"))
        return PPS_ERR_CUDA;
    for (int q = 0; q < P->nprob; q++) P->hst[(size_t)q] = table[(size_t)P->slot[(size_t)q]];
    pps_batch_stats& S = *stats;
    std::memset(&S, 0, sizeof(S));
    S.seconds_solve = ms * 1e-3;
    S.kernel_launches = 2;
    S.graph_replays = 1;
    pps_status rc = PPS_OK;
    for (int q = 0; q < P->nprob; q++) {
        const State& st = P->hst[(size_t)q];
        const double e = st.normb > 0 ? st.err_outer / st.normb : 0.0;
        S.max_err_true = std::max(S.max_err_true, e);
        S.max_iterations = std::max(S.max_iterations, st.total_it);
        S.sum_iterations += st.total_it;
        S.max_refinements = std::max(S.max_refinements, st.refinements);
        const double m = (double)P->prob[(size_t)q].m;
        S.unknowns += m * m * m;
        if (st.done && st.status == PPS_OK) S.converged++;
        else if (rc == PPS_OK) rc = st.done && st.status != PPS_OK ? (pps_status)st.status : PPS_NOT_CONVERGED;
    }
    if (bar.error != 0) {
        err = "a grid barrier of the persistent batched solve waited longer than its limit";
        return PPS_TIMEOUT;
    }
    return rc;
}

void bvc_result(const BvcPlan* plan, int q, pps_stats* st)
{
    const Plan* P = reinterpret_cast<const Plan*>(plan);
    const State& s = P->hst[(size_t)q];
    st->iterations = s.total_it;
    st->refinements = s.refinements;
    st->norm_b = s.normb;
    st->err_true = s.normb > 0 ? s.err_outer / s.normb : -1.0;
    st->err_iter = s.normb > 0 ? s.err / s.normb : -1.0;
}

}  // namespace pps
