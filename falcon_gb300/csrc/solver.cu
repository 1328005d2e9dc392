// solver.cu -- GPU multigrid-preconditioned flexible CG on the Yin-Yang grid.
//
// Reference algorithm: ModLinearSolver_Multigrid_CG / _V_cycle / _JCB_CG
// (3_5/ModLinearSolver.f90:86-427) with the 7-point face-coefficient operator
// (:15-84) and the 1-layer face-ghost halo (3_5/ModCommunication.f90:1497-1639).
// GB300 form:
//   - FP64 iterative refinement outside: the true residual r = b - A x, its
//     norms and the update x += d are FP64, and convergence is judged only on
//     the FP64 ||b - A x|| / ||b||;
//   - inside, flexible CG in float-float (FP32 pairs, about 48 bits; GB300's
//     FP64 pipe is too slow for the per-cell work of every iteration) on the
//     correction equation scaled by per-problem powers of two, per-problem
//     dot products reduced into FP64; y = A x of falcon_solver_apply and the
//     coarse training solve stay FP64;
//   - V-cycle preconditioner in FP32: red-black Gauss-Seidel smoothing,
//     restriction R = P^T (sum of 8 children), injection prolongation,
//     Galerkin coarse operators;
//   - every problem of a batch is advanced by the same launches: kernels index
//     block -> problem, scalars are per problem, converged problems freeze.
// The cell kernels' CTAs take chunks of one block's cells, so a CTA never mixes problems
// and its reductions go to one per-problem slot with one atomic; the V-cycle's threads
// take pairs of cells of a row (vcycle.cuh).
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <map>
#include <vector>

#include "../../include/falcon_gb300.h"
#include "ff.cuh"
#include "lcc.h"
#include "solver.h"
#include "uploads.h"
#include "vcycle.cuh"

namespace falcon {
namespace sv {

struct LevelDims {
    int m0, m1, m2;        // interior
    int p0, p1, p2;        // padded (m+2)
    int nint, npad;
    int chunk;             // cells per CTA (a multiple of m0; the solver's tuned tile)
    int tpb;               // threads per CTA (<= 1024, a multiple of 32)
};

struct HaloList {
    int64_t n;
    const int32_t* dst;    // padded global offset
    const int32_t* src;    // padded global offset of the base source cell
    const uint8_t* code;   // bit d set: the weight of direction d is not 0
    const double* w;       // [n][3]
    int32_t sj, sk;        // padded strides of j and k
};

struct Ops64 { const double *Aii, *Ai, *Aj, *Ak; };

// Launch geometry of the cell kernels: CTAs take chunks of d.chunk cells,
// block-major (consecutive CTAs stream consecutive memory); a chunk never
// spans two blocks, so a CTA's reductions go to one problem. The chunk and
// the CTA size are the solver's tile shape, picked by its autotuner.
__device__ __forceinline__ int cell_chunks(const LevelDims& d) { return (d.nint + d.chunk - 1) / d.chunk; }
__device__ __forceinline__ int cell_block(const LevelDims& d) { return (int)(blockIdx.x / (unsigned)cell_chunks(d)); }
__device__ __forceinline__ int cell_first(const LevelDims& d) {
    return (int)(blockIdx.x % (unsigned)cell_chunks(d)) * d.chunk;
}
__device__ __forceinline__ int cell_end(const LevelDims& d) { return min(cell_first(d) + d.chunk, d.nint); }

__device__ __forceinline__ void cell_ijk(const LevelDims& d, int c, int& i, int& j, int& k) {
    i = c % d.m0 + 1;
    j = (c / d.m0) % d.m1 + 1;
    k = c / (d.m0 * d.m1) + 1;
}
__device__ __forceinline__ size_t pidx(const LevelDims& d, int b, int i, int j, int k) {
    return (size_t)b * d.npad + ((size_t)k * d.p1 + j) * d.p0 + i;
}

// y = A x over the interior, reference operand order (3_5/ModLinearSolver.f90:43-50)
template <class T, class O>
__device__ __forceinline__ T apply_A(const O& A, const LevelDims& d, const T* x, int b, int c, int i, int j, int k) {
    const size_t P = pidx(d, b, i, j, k);
    const size_t sj = d.p0, sk = (size_t)d.p0 * d.p1;
    const size_t fi = ((size_t)b * d.m2 * d.m1 + (size_t)(k - 1) * d.m1 + (j - 1)) * (d.m0 + 1) + (i - 1);
    const size_t fj = ((size_t)b * d.m2 * (d.m1 + 1) + (size_t)(k - 1) * (d.m1 + 1) + (j - 1)) * d.m0 + (i - 1);
    const size_t fk = ((size_t)b * (d.m2 + 1) * d.m1 + (size_t)(k - 1) * d.m1 + (j - 1)) * d.m0 + (i - 1);
    return A.Aii[(size_t)b * d.nint + c] * x[P] + A.Ai[fi] * x[P - 1] + A.Ai[fi + 1] * x[P + 1] + A.Aj[fj] * x[P - sj] +
           A.Aj[fj + d.m0] * x[P + sj] + A.Ak[fk] * x[P - sk] + A.Ak[fk + (size_t)d.m0 * d.m1] * x[P + sk];
}

template <class T>
__device__ __forceinline__ void block_sum_atomic(T v, double* slot) {
    double s = (double)v;
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    __shared__ double ws[32];
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += ws[w];
        atomicAdd(slot, t);
    }
    __syncthreads();
}

// ---- halo fill (trilinear from the source interior) ------------------------
// entries whose three weights are exactly zero are plain copies of the base
// cell (a separate index list, no weights)
// one launch for both lists: entries [0, nc) are the copies, the rest the
// interpolated entries of H
template <class T>
__global__ void k_halo(T* v, HaloList H, const int32_t* cdst, const int32_t* csrc, int64_t nc) {
    int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e < nc) {
        v[cdst[e]] = v[csrc[e]];
        return;
    }
    e -= nc;
    if (e >= H.n) return;
    const size_t s = (size_t)H.src[e];
    const int cd = H.code[e];
    const int a = (cd & 1) ? 1 : 0, bq = (cd & 2) ? H.sj : 0, c = (cd & 4) ? H.sk : 0;
    const T wi = H.w[3 * e], wj = H.w[3 * e + 1], wk = H.w[3 * e + 2];
    const T ui = T(1) - wi, uj = T(1) - wj, uk = T(1) - wk;
    const T* f = v + s;
    v[H.dst[e]] = f[0] * ui * uj * uk + f[a] * wi * uj * uk + f[bq] * ui * wj * uk + f[c] * ui * uj * wk +
                  f[a + bq] * wi * wj * uk + f[bq + c] * ui * wj * wk + f[a + c] * wi * uj * wk + f[a + bq + c] * wi * wj * wk;
}

// ---- FP64 outer iteration ----------------------------------------------------
struct Dots {
    double *pAp, *zw, *zAp, *rr, *bb, *ab;   // ab: sum of (|b| + sum_j |A_ij x_j|)^2
    double *pw, *zr;
    const int32_t* active;
    const int32_t* bprob;
};

// y = A x
__global__ void k_spmv(Ops64 A, LevelDims d, const double* x, double* y) {
    const int b = cell_block(d), c0 = cell_first(d), c1 = cell_end(d);
    for (int c = c0 + threadIdx.x; c < c1; c += blockDim.x) {
        int i, j, k;
        cell_ijk(d, c, i, j, k);
        y[(size_t)b * d.nint + c] = apply_A<double>(A, d, x, b, c, i, j, k);
    }
}

// sum_j |A_ij x_j| of one row: the scale of the rounding error of b - A x
__device__ __forceinline__ double abs_row(const Ops64& A, const LevelDims& d, const double* x, int b, int c, int i,
                                          int j, int k) {
    const size_t P = pidx(d, b, i, j, k);
    const size_t sj = d.p0, sk = (size_t)d.p0 * d.p1;
    const size_t fi = ((size_t)b * d.m2 * d.m1 + (size_t)(k - 1) * d.m1 + (j - 1)) * (d.m0 + 1) + (i - 1);
    const size_t fj = ((size_t)b * d.m2 * (d.m1 + 1) + (size_t)(k - 1) * (d.m1 + 1) + (j - 1)) * d.m0 + (i - 1);
    const size_t fk = ((size_t)b * (d.m2 + 1) * d.m1 + (size_t)(k - 1) * d.m1 + (j - 1)) * d.m0 + (i - 1);
    return fabs(A.Aii[(size_t)b * d.nint + c] * x[P]) + fabs(A.Ai[fi] * x[P - 1]) + fabs(A.Ai[fi + 1] * x[P + 1]) +
           fabs(A.Aj[fj] * x[P - sj]) + fabs(A.Aj[fj + d.m0] * x[P + sj]) + fabs(A.Ak[fk] * x[P - sk]) +
           fabs(A.Ak[fk + (size_t)d.m0 * d.m1] * x[P + sk]);
}

// r = b - A x (FP64 true residual); rr += r.r; ab += (|b| + sum|A x|)^2; rf = (float)r
__global__ void k_residual64(Ops64 A, LevelDims d, const double* x, const double* bvec, double* r, float* rf, Dots D,
                             int want_bb) {
    const int b = cell_block(d), c0 = cell_first(d), c1 = cell_end(d);
    double rr = 0, bb = 0, ab = 0;
    for (int c = c0 + threadIdx.x; c < c1; c += blockDim.x) {
        int i, j, k;
        cell_ijk(d, c, i, j, k);
        const size_t q = (size_t)b * d.nint + c;
        const double rv = bvec[q] - apply_A<double>(A, d, x, b, c, i, j, k);
        r[q] = rv;
        rf[q] = (float)rv;
        rr += rv * rv;
        bb += bvec[q] * bvec[q];
        const double s = fabs(bvec[q]) + abs_row(A, d, x, b, c, i, j, k);
        ab += s * s;
    }
    const int pb = D.bprob[b];
    block_sum_atomic(rr, &D.rr[pb]);
    block_sum_atomic(ab, &D.ab[pb]);
    if (want_bb) block_sum_atomic(bb, &D.bb[pb]);
}

// ---- float-float inner iteration -------------------------------------------------
// GB300 runs FP64 at a small fraction of its FP32 rate, and FP64 kernels run
// every iteration are bound by the FP64 pipe. The inner solve of each
// refinement pass therefore runs the flexible CG in float-float: every value
// an FP32 pair (hi, lo), hi + lo with |lo| <= ulp(hi)/2, about 48 significant
// bits, formed with error-free FP32 transformations (this file is compiled
// without FMA contraction; the FMAs below are explicit). FP32's exponent range
// is too narrow for the raw system (b.b reaches 1e54 for conduction), so the
// inner solve works on A' = A / sA, r' = r / sr, d' = d sA / sr per problem
// with sA, sr powers of two (exact): every vector and dot product is O(1).
struct Ops2 { const float2 *Aii, *Ai, *Aj, *Ak; };

__device__ __forceinline__ float2 ff_shfl_xor(float2 v, int o) {
    return make_float2(__shfl_xor_sync(0xffffffffu, v.x, o), __shfl_xor_sync(0xffffffffu, v.y, o));
}
// per-problem FF sums -> one FP64 atomic per CTA and sum (FP64 work once per warp)
__device__ __forceinline__ void block_sum_atomic_ff(float2 v, double* slot) {
    for (int o = 16; o > 0; o >>= 1) v = ff_add(v, ff_shfl_xor(v, o));
    __shared__ double ws[32];
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = ff_to(v);
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += ws[w];
        atomicAdd(slot, t);
    }
}
// four sums at once: each exchange of the first two folds two sums into one
// (the lanes of either half keep their own), 6 FF additions instead of 20
__device__ __forceinline__ void block_sum4_atomic_ff(const float2 (&v)[4], double* const (&slot)[4]) {
    const int lane = threadIdx.x & 31;
    const bool hi = lane & 16, top = lane & 8;
    const float2 a = ff_add(hi ? v[1] : v[0], ff_shfl_xor(hi ? v[0] : v[1], 16));
    const float2 b = ff_add(hi ? v[3] : v[2], ff_shfl_xor(hi ? v[2] : v[3], 16));
    float2 s = ff_add(top ? b : a, ff_shfl_xor(top ? a : b, 8));
    for (int o = 4; o > 0; o >>= 1) s = ff_add(s, ff_shfl_xor(s, o));
    __shared__ double ws[32][4];
    if ((lane & 7) == 0) ws[threadIdx.x >> 5][(hi ? 1 : 0) + (top ? 2 : 0)] = ff_to(s);
    __syncthreads();
    if (threadIdx.x < 4) {
        double t = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += ws[w][threadIdx.x];
        double* p = threadIdx.x == 0 ? slot[0] : threadIdx.x == 1 ? slot[1] : threadIdx.x == 2 ? slot[2] : slot[3];
        atomicAdd(p, t);
    }
}

// The search's z: the preconditioner's FP32 output scaled by the problem's sA, or
// without a preconditioner the residual itself, all of its bits.
struct Z32 {
    const float *__restrict__ z, *__restrict__ scale;
    static constexpr int kUnroll = 2;
    __device__ __forceinline__ float of_problem(int pb) const { return scale[pb]; }
    __device__ __forceinline__ float2 operator()(size_t q, float s) const { return make_float2(z[q] * s, 0.f); }
};
struct ZFF {
    const float2* r;
    static constexpr int kUnroll = 1;
    __device__ __forceinline__ float of_problem(int) const { return 1.f; }
    __device__ __forceinline__ float2 operator()(size_t q, float) const { return r[q]; }
};

// Ghosts of z at the finest level as FF values, one slot per ghost in the layout of
// VLevel::ghost. A copied cell's map weights are 0 or 1 up to eps (about 1e-14, see
// kSnapFF): the ghost is z0 + sum of eps_d (z_d - z0) over the three directions, z_d
// one cell on (eps > 0) or back (eps < 0); second-order terms are below 2^-64. Other
// ghosts sum eight cells with FF weights.
struct GhostFF {
    const int32_t* ghost;   // [slot] >= 0 source cell, -1 none, <= -2 entry -(v + 2)
    const float* eps;       // [slot][3]
    const int32_t* src;     // entry: base source cell
    const uint8_t* code;    // bit d set: the weight of direction d is not 0
    const float2* w8;       // [entry][8] corner weights
    int m;
    int64_t n;              // slots
};
template <class Z>
__global__ void k_ghost_ff(GhostFF H, Z z, const int32_t* bprob, float2* G) {
    const int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= H.n) return;
    const int d = H.ghost[x];
    if (d == -1) return;   // stays 0
    const int m = H.m, mm = m * m;
    const float s = z.of_problem(bprob[x / (6 * mm)]);
    if (d >= 0) {
        const float2 z0 = z((size_t)d, s);
        float lo = 0.f;
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const float ep = H.eps[3 * x + q];
            const int st = q == 0 ? 1 : q == 1 ? m : mm;
            if (ep != 0.f) lo = fmaf(fabsf(ep), z((size_t)(ep > 0.f ? d + st : d - st), s).x - z0.x, lo);
        }
        const float2 t = ff_two_sum(z0.x, lo);
        G[x] = ff_quick(t.x, t.y + z0.y);
        return;
    }
    const int e = -(d + 2), cd = H.code[e];
    const int a = (cd & 1) ? 1 : 0, b = (cd & 2) ? m : 0, c = (cd & 4) ? mm : 0;
    const int off[8] = {0, a, b, c, a + b, b + c, a + c, a + b + c};
    const size_t f = (size_t)H.src[e];
    const float4* w = reinterpret_cast<const float4*>(H.w8 + 8 * (size_t)e);
    FFSum y;
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        const float4 w2 = w[t];
        y.add(make_float2(w2.x, w2.y), z(f + off[2 * t], s));
        y.add(make_float2(w2.z, w2.w), z(f + off[2 * t + 1], s));
    }
    G[x] = y.value();
}

// w = A' z, the reference's operand order, with the four products that the
// step needs: z.w, z.Ap, p.w, z.r. The direction is p' = z + beta p and A' p' = w +
// beta A' p, so that beta, alpha and the update follow from one pass over the operator
// and no halo of p is kept.
template <int M, class Z>   // M: m, or 0
__global__ void __launch_bounds__(512) k_spmv_z_ff(Ops2 A, LevelDims d, Z z, const float2* __restrict__ G,
                                                   const float2* __restrict__ p,
                                                   const float2* __restrict__ r, const float2* __restrict__ Ap,
                                                   float2* __restrict__ w, Dots D) {
    const int b = cell_block(d), c0 = cell_first(d), c1 = cell_end(d), pb = D.bprob[b];
    if (!D.active[pb]) return;
    const int m = M > 0 ? M : d.m0, mm = m * m;
    const float s = z.of_problem(pb);
    const size_t zb = (size_t)b * d.nint;
    const float2* Gb = G + (size_t)b * 6 * mm;
    FFSum zw, za, pw, zr;
    const float2 *__restrict__ Aii = A.Aii, *__restrict__ Ai = A.Ai, *__restrict__ Aj = A.Aj, *__restrict__ Ak = A.Ak;
    // two cells at a time with an FP32 z (the pointers' promise lets their loads overlap)
#pragma unroll Z::kUnroll
    for (int c = c0 + threadIdx.x; c < c1; c += blockDim.x) {
        const int i = c % m, row = c / m, j = row % m, k = row / m;
        const size_t fi = ((size_t)b * mm + row) * (m + 1) + i;
        const size_t fj = ((size_t)b * m * (m + 1) + (size_t)k * (m + 1) + j) * m + i;
        const size_t fk = ((size_t)b * (m + 1) * m + row) * m + i, q = (size_t)b * d.nint + c;
        auto inside = [&](int y) { return z(zb + y, s); };
        const float2 zc = inside(c);
        FFSum y;
        y.add(Aii[q], zc);
        y.add(Ai[fi], i > 0 ? inside(c - 1) : Gb[row]);
        y.add(Ai[fi + 1], i < m - 1 ? inside(c + 1) : Gb[mm + row]);
        y.add(Aj[fj], j > 0 ? inside(c - m) : Gb[2 * mm + k * m + i]);
        y.add(Aj[fj + m], j < m - 1 ? inside(c + m) : Gb[3 * mm + k * m + i]);
        y.add(Ak[fk], k > 0 ? inside(c - mm) : Gb[4 * mm + j * m + i]);
        y.add(Ak[fk + mm], k < m - 1 ? inside(c + mm) : Gb[5 * mm + j * m + i]);
        const float2 wv = y.value();
        w[q] = wv;
        zw.add(zc, wv);
        za.add(zc, Ap[q]);
        pw.add(p[q], wv);
        zr.add(zc, r[q]);
    }
    block_sum4_atomic_ff({zw.value(), za.value(), pw.value(), zr.value()}, {&D.zw[pb], &D.zAp[pb], &D.pw[pb], &D.zr[pb]});
}

// The step's scalars of a problem from k_spmv_z_ff's products: beta = -z.Ap / p.Ap
// (flexible CG, one-term A-orthogonalisation; 0 to restart), p'.Ap' and alpha =
// p'.r / p'.Ap' (p.r = 0 after the step that made r). A direction that vanished
// takes no step.
struct StepFF { double alpha, beta, pAp; };
__device__ __forceinline__ StepFF step_ff(const Dots& D, int pb, int restart) {
    const double pAp = D.pAp[pb], zAp = D.zAp[pb];
    StepFF s;
    s.beta = restart || pAp == 0.0 ? 0.0 : -zAp / pAp;
    s.pAp = D.zw[pb] + s.beta * (zAp + D.pw[pb] + s.beta * pAp);
    s.alpha = s.pAp != 0.0 ? D.zr[pb] / s.pAp : 0.0;
    return s;
}

// p = z + beta p; Ap = w + beta Ap; x += alpha p; r -= alpha Ap; rr += r.r; rf =
// hi(r), the V-cycle's input
template <class Z>
__global__ void __launch_bounds__(512) k_step_ff(LevelDims d, Z z, const float2* w, float2* x,
                                                 float2* p, float2* r, float2* Ap, float* rf, Dots D, int restart) {
    const int b = cell_block(d), c0 = cell_first(d), c1 = cell_end(d), pb = D.bprob[b];
    if (!D.active[pb]) return;
    __shared__ float2 ab[2];   // the scalars' FP64 work once per CTA
    if (threadIdx.x == 0) {
        const StepFF s = step_ff(D, pb, restart);
        ab[0] = ff_from(s.alpha);
        ab[1] = ff_from(s.beta);
    }
    __syncthreads();
    const float2 al = ab[0], be = ab[1], nal = ff_neg(al);
    const float s = z.of_problem(pb);
    FFSum rr;
    for (int c = c0 + threadIdx.x; c < c1; c += blockDim.x) {
        const size_t q = (size_t)b * d.nint + c;
        const float2 pv = ff_add(z(q, s), ff_mul(be, p[q]));   // (z may be r: read before it changes)
        const float2 av = ff_add(w[q], ff_mul(be, Ap[q]));
        const float2 rv = ff_add(r[q], ff_mul(nal, av));
        p[q] = pv;
        Ap[q] = av;
        x[q] = ff_add(x[q], ff_mul(al, pv));
        r[q] = rv;
        rf[q] = rv.x;
        rr.add(rv, rv);
    }
    block_sum_atomic_ff(rr.value(), &D.rr[pb]);
}

// ---- the inner solve's loop control on the device -----------------------------
// One inner solve (an FCG on the correction equation) runs as one graph launch:
// a first iteration, then a WHILE node whose body is one more iteration; the
// last kernel of every iteration decides, on the device, whether the loop goes
// on. The loop is bounded: it counts its iterations and stops at max_it.
struct InnerCtl {
    int32_t it;        // iterations done by this inner solve
    int32_t max_it;    // its iteration limit (<= kInnerCap)
    int32_t stalled;   // the largest relative residual fell by < 5% over 8 iterations
    int32_t nan;       // a non-finite residual
    int32_t cont;      // the loop condition written by the last check
    int32_t pad_;
    double hist[16];   // ring of the largest relative residual per iteration
};
constexpr int32_t kInnerCap = 100000;

// After an iteration's x/r update: each problem's relative recursive residual
// h = sqrt(r.r / r0.r0); a problem at or below its eta leaves the iteration
// (active = 0: no further update). One CTA of 256 threads, problem per thread
// (nproblems <= 256). With `set_cond`, sets the WHILE node's condition.
__global__ void __launch_bounds__(256) k_inner_check(int np, Dots D, int restart, const double* rr0, const double* eta,
                                                     int32_t* active, InnerCtl* ctl, cudaGraphConditionalHandle h,
                                                     int set_cond) {
    __shared__ double smax[256];
    __shared__ int sany[256], snan[256];
    const int q = threadIdx.x;
    double hq = 0.0;
    int still = 0, bad = 0;
    if (q < np && active[q]) {
        hq = sqrt(D.rr[q] / rr0[q]);
        D.pAp[q] = step_ff(D, q, restart).pAp;   // of the direction just taken
        D.zw[q] = D.zAp[q] = D.pw[q] = D.zr[q] = D.rr[q] = 0.0;   // for the next iteration's sums
        if (!(hq == hq) || hq > 1e300) {
            bad = 1;
        } else if (hq <= eta[q]) {
            active[q] = 0;
        } else {
            still = 1;
        }
    }
    smax[q] = hq;
    sany[q] = still;
    snan[q] = bad;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (q < o) {
            smax[q] = fmax(smax[q], smax[q + o]);
            sany[q] |= sany[q + o];
            snan[q] |= snan[q + o];
        }
        __syncthreads();
    }
    if (q == 0) {
        const int it = ctl->it + 1;
        ctl->it = it;
        if (snan[0]) ctl->nan = 1;
        int stalled = ctl->stalled;
        if (sany[0]) {
            ctl->hist[it & 15] = smax[0];
            if (it > 10 && smax[0] > 0.95 * ctl->hist[(it - 8) & 15]) stalled = 1;
        }
        ctl->stalled = stalled;
        const int cap = ctl->max_it < kInnerCap ? ctl->max_it : kInnerCap;
        const int cont = (sany[0] && !stalled && !snan[0] && it < cap) ? 1 : 0;
        ctl->cont = cont;
        if (set_cond) cudaGraphSetConditional(h, (unsigned)cont);
    }
}

// ---- FP64 iterative refinement around the float-float solve ------------------
// r' = r / sr per problem as FF pairs (sr a power of two at or above ||r||_2:
// exact, and |r'| <= 1), its FP32 part for the V-cycle, and rr += r'.r'
__global__ void k_ir_start(LevelDims d, const double* r, const double* inv_sr, float2* r2, float* rf, Dots D) {
    const int b = cell_block(d), c0 = cell_first(d), c1 = cell_end(d);
    const int pb = D.bprob[b];
    const double s = inv_sr[pb];
    float2 rr = make_float2(0.f, 0.f);
    for (int c = c0 + threadIdx.x; c < c1; c += blockDim.x) {
        const size_t q = (size_t)b * d.nint + c;
        const double v = r[q] * s;
        const float h = (float)v;
        const float2 x = make_float2(h, (float)(v - (double)h));
        r2[q] = x;
        rf[q] = h;
        rr = ff_add(rr, ff_mul(x, x));
    }
    block_sum_atomic_ff(rr, &D.rr[pb]);
}

// x += d' * fac per problem (FP64): d' the float-float correction of the
// scaled system, fac = sr / sA (a power of two, so the scaling is exact)
__global__ void k_ir_accum(LevelDims d, const float2* x2, const double* fac, const int32_t* bprob, double* x) {
    const int b = cell_block(d), c0 = cell_first(d), c1 = cell_end(d);
    const double f = fac[bprob[b]];
    for (int c = c0 + threadIdx.x; c < c1; c += blockDim.x) {
        int i, j, k;
        cell_ijk(d, c, i, j, k);
        const size_t P = pidx(d, b, i, j, k);
        x[P] = x[P] + ff_to(x2[(size_t)b * d.nint + c]) * f;
    }
}

// ---- learned coarse correction: coarsest level <-> dense panel grids ---------
// gmap[b][c]: panel-grid voxel of coarse cell c of block b

// static input channels 1..7: the six face couplings / diag, (diag + sum)/diag
__global__ void k_lcc_static(Ops64 A, LevelDims d, const int32_t* gmap, float* feat) {
    const int b = cell_block(d), c0 = cell_first(d), c1 = cell_end(d);
    for (int c = c0 + threadIdx.x; c < c1; c += blockDim.x) {
        int i, j, k;
        cell_ijk(d, c, i, j, k);
        const size_t fi = ((size_t)b * d.m2 * d.m1 + (size_t)(k - 1) * d.m1 + (j - 1)) * (d.m0 + 1) + (i - 1);
        const size_t fj = ((size_t)b * d.m2 * (d.m1 + 1) + (size_t)(k - 1) * (d.m1 + 1) + (j - 1)) * d.m0 + (i - 1);
        const size_t fk = ((size_t)b * (d.m2 + 1) * d.m1 + (size_t)(k - 1) * d.m1 + (j - 1)) * d.m0 + (i - 1);
        const double dg = A.Aii[(size_t)b * d.nint + c];
        const double cpl[6] = {A.Ai[fi], A.Ai[fi + 1], A.Aj[fj], A.Aj[fj + d.m0], A.Ak[fk], A.Ak[fk + (size_t)d.m0 * d.m1]};
        float* f = feat + (size_t)gmap[(size_t)b * d.nint + c] * 8;
        double sum = dg;
        for (int q = 0; q < 6; ++q) { f[1 + q] = (float)(cpl[q] / dg); sum += cpl[q]; }
        f[7] = (float)(sum / dg);
    }
}

// sum over coarse cells of (r/diag)^2
__global__ void k_lcc_sumsq(LevelDims d, const float* r, const float* Aii, double* sum) {
    const int b = cell_block(d), c0 = cell_first(d), c1 = cell_end(d);
    double v = 0.0;
    for (int c = c0 + threadIdx.x; c < c1; c += blockDim.x) {
        const size_t q = (size_t)b * d.nint + c;
        const double x = (double)r[q] / (double)Aii[q];
        v += x * x;
    }
    block_sum_atomic(v, sum);
}

__device__ __forceinline__ double lcc_scale(const double* sum, int64_t n) {
    const double s = sqrt(*sum / (double)n);
    return s > 0.0 ? s : 1.0;
}

// input channel 0: (r/diag)/s, s = RMS of r/diag
__global__ void k_lcc_feat(LevelDims d, const float* r, const float* Aii, const int32_t* gmap, const double* sum,
                           int64_t n, float* feat) {
    const int b = cell_block(d), c0 = cell_first(d), c1 = cell_end(d);
    for (int c = c0 + threadIdx.x; c < c1; c += blockDim.x) {
        const size_t q = (size_t)b * d.nint + c;
        feat[(size_t)gmap[q] * 8] = (float)((double)r[q] / (double)Aii[q] / lcc_scale(sum, n));
    }
}

// coarse correction z = s * y
__global__ void k_lcc_scatter(LevelDims d, const float* y, const int32_t* gmap, const double* sum, int64_t n, float* z) {
    const int b = cell_block(d), c0 = cell_first(d), c1 = cell_end(d);
    for (int c = c0 + threadIdx.x; c < c1; c += blockDim.x) {
        const size_t q = (size_t)b * d.nint + c;
        z[q] = (float)(lcc_scale(sum, n) * (double)y[gmap[q]]);
    }
}

// training target: t = e/s (e: padded FP64 coarse solution)
__global__ void k_lcc_target(LevelDims d, const double* e, const int32_t* gmap, const double* sum, int64_t n, float* t) {
    const int b = cell_block(d), c0 = cell_first(d), c1 = cell_end(d);
    for (int c = c0 + threadIdx.x; c < c1; c += blockDim.x) {
        int i, j, k;
        cell_ijk(d, c, i, j, k);
        t[gmap[(size_t)b * d.nint + c]] = (float)(e[pidx(d, b, i, j, k)] / lcc_scale(sum, n));
    }
}

// ---- Jacobi-preconditioned CG on one level (FP64): exact coarse errors -------
// dots: [0] r.z  [1] p.Ap  [2] r.r (current); nd: the same for the next iterate
__global__ void k_ccg_init(Ops64 A, LevelDims d, const float* rc, double* r, double* z, double* p, double* dots) {
    const int b = cell_block(d), c0 = cell_first(d), c1 = cell_end(d);
    double rz = 0, rr = 0;
    for (int c = c0 + threadIdx.x; c < c1; c += blockDim.x) {
        int i, j, k;
        cell_ijk(d, c, i, j, k);
        const size_t q = (size_t)b * d.nint + c;
        const double rv = (double)rc[q], zv = rv / A.Aii[q];
        r[q] = rv;
        z[q] = zv;
        p[pidx(d, b, i, j, k)] = zv;
        rz += rv * zv;
        rr += rv * rv;
    }
    block_sum_atomic(rz, &dots[0]);
    block_sum_atomic(rr, &dots[2]);
}

__global__ void k_ccg_spmv(Ops64 A, LevelDims d, const double* p, double* Ap, double* dots) {
    const int b = cell_block(d), c0 = cell_first(d), c1 = cell_end(d);
    double pa = 0;
    for (int c = c0 + threadIdx.x; c < c1; c += blockDim.x) {
        int i, j, k;
        cell_ijk(d, c, i, j, k);
        const double y = apply_A<double>(A, d, p, b, c, i, j, k);
        Ap[(size_t)b * d.nint + c] = y;
        pa += p[pidx(d, b, i, j, k)] * y;
    }
    block_sum_atomic(pa, &dots[1]);
}

__global__ void k_ccg_update(Ops64 A, LevelDims d, double* x, const double* p, double* r, const double* Ap, double* z,
                             const double* dots, double* nd) {
    const int b = cell_block(d), c0 = cell_first(d), c1 = cell_end(d);
    const double alpha = dots[0] / dots[1];
    double rz = 0, rr = 0;
    for (int c = c0 + threadIdx.x; c < c1; c += blockDim.x) {
        int i, j, k;
        cell_ijk(d, c, i, j, k);
        const size_t P = pidx(d, b, i, j, k), q = (size_t)b * d.nint + c;
        x[P] += alpha * p[P];
        const double rv = r[q] - alpha * Ap[q], zv = rv / A.Aii[q];
        r[q] = rv;
        z[q] = zv;
        rz += rv * zv;
        rr += rv * rv;
    }
    block_sum_atomic(rz, &nd[0]);
    block_sum_atomic(rr, &nd[2]);
}

__global__ void k_ccg_p(LevelDims d, double* p, const double* z, const double* dots, const double* nd) {
    const int b = cell_block(d), c0 = cell_first(d), c1 = cell_end(d);
    for (int c = c0 + threadIdx.x; c < c1; c += blockDim.x) {
        int i, j, k;
        cell_ijk(d, c, i, j, k);
        const size_t P = pidx(d, b, i, j, k);
        p[P] = z[(size_t)b * d.nint + c] + (nd[0] / dots[0]) * p[P];
    }
}

}  // namespace sv
}  // namespace falcon

using namespace falcon;
using namespace falcon::sv;

struct SvLevel {
    LevelDims d{};
    double *Aii = nullptr, *Ai = nullptr, *Aj = nullptr, *Ak = nullptr;
    float *fAii = nullptr, *fAi = nullptr, *fAj = nullptr, *fAk = nullptr;
    // FP64 halo lists: interpolated entries and plain copies (padded offsets)
    int32_t *hdst = nullptr, *hsrc = nullptr;
    uint8_t* hcode = nullptr;
    double* hw = nullptr;
    int64_t nh = 0;
    int32_t *hcdst = nullptr, *hcsrc = nullptr;
    int64_t nhc = 0;
    // FP32 V-cycle: ghost descriptors and interpolation entries (VLevel)
    int32_t *ghost = nullptr, *isrc = nullptr, *nbr = nullptr;
    uint8_t* icode = nullptr;
    float* iw = nullptr;
    // z: where a V-cycle leaves its result; z and zb take turns inside it
    float *z = nullptr, *zb = nullptr, *r = nullptr, *res = nullptr;
    // level 0: the scaled operator A / sA as FF pairs
    float2 *Aii2 = nullptr, *Ai2 = nullptr, *Aj2 = nullptr, *Ak2 = nullptr;
    HaloList halo() const { return HaloList{nh, hdst, hsrc, hcode, hw, d.p0, d.p0 * d.p1}; }
    Ops2 ops2() const { return Ops2{Aii2, Ai2, Aj2, Ak2}; }
    Ops64 ops64() const { return Ops64{Aii, Ai, Aj, Ak}; }
    VLevel view(int nb) const {
        const uint32_t h = (uint32_t)d.m0 / 2, mh = h * d.m0;
        auto inverse = [](uint32_t x) { return x > 1 ? (uint32_t)((1ull << 32) / x + 1) : 0u; };
        return VLevel{d.m0, d.nint, nb, inverse(h), inverse(mh), fAii, fAi, fAj, fAk, ghost, isrc, icode, iw, nbr};
    }
};

struct falcon_solver {
    SolverProblemSet S;
    std::string err;
    int device = 0;
    cudaStream_t st = nullptr;
    std::vector<SvLevel> lv;
    double *x = nullptr, *p = nullptr, *r = nullptr, *Ap = nullptr, *z = nullptr, *bvec = nullptr;
    // the float-float inner solve (scaled system, see Ops2), interior: w2 = A' z; ghosts of z
    float2 *x2 = nullptr, *p2 = nullptr, *r2 = nullptr, *Ap2 = nullptr, *w2 = nullptr, *ghosts2 = nullptr;
    GhostFF gff{};
    std::vector<double> sA;               // per-problem powers of two (the operator's scale)
    float* dsA = nullptr;                 // sA on the device (FP32: powers of two are exact)
    double* dots = nullptr;       // [8][nproblems]: see Dots
    double* ir_par = nullptr;     // [2][nproblems]: 1/sr and sr/sA of the refinement pass
    int32_t *active = nullptr, *bprob = nullptr;
    std::vector<void*> allocs;
    int nu_pre = 2, nu_post = 2, nu_coarse = 16;
    double dt_conduction = 0;
    uint64_t seed = 0;                    // the spec's seed (problem q: seed + q)
    double r_surface = 0;                 // PFSS: lower boundary radius (cm) of the synthetic magnetogram
    // learned coarse correction
    falcon_lcc* net = nullptr;
    int net_sweeps = 2;
    bool use_net = false;                 // set per V-cycle by the solve
    bool cmap_ok = false;
    int cD = 0, cH = 0, cW = 0;           // dense panel grid of the coarsest level
    int32_t* gmap = nullptr;              // [b][nint_c] -> panel-grid voxel
    float *feat = nullptr, *yout = nullptr;
    double* csum = nullptr;
    double* cdots = nullptr;              // [6] scalars of the coarse CG
    // recording of coarsest-level residuals (falcon_solver_record)
    float* rec = nullptr;
    int rec_max = 0, rec_n = 0;
    // one instantiated CUDA graph per V-cycle shape (smoothing sweeps, network on/off)
    std::map<int64_t, cudaGraphExec_t> vgraphs;
    // one instantiated graph per inner-solve shape: a first iteration and a
    // device-controlled WHILE loop of iterations (the V-cycle inside it)
    std::map<int64_t, cudaGraphExec_t> igraphs;
    bool capturing = false;               // enqueueing into a graph: the V-cycle's kernels inline
    InnerCtl* ictl = nullptr;             // device loop control
    double *rr0 = nullptr, *eta = nullptr;   // device, per problem
    // the coarsest level's sweeps in one launch (k_coarse_sweeps): CTAs per
    // problem (0: one launch per half sweep) and cells per thread and colour
    int coarse_cluster = 0, coarse_r = 1;
    int32_t* first = nullptr;             // [np + 1] first block of each problem
    uint32_t* cghost = nullptr;           // its ghost table and gathered ghosts (CoarseArgs)
    uint2* ceat = nullptr;
    float4* cew = nullptr;
    int4* clist = nullptr;
    int coarse_slots = 0;
    // tile shape of the cell kernels (cells per CTA, threads per CTA), tuned at the first solve
    int tile_chunk = 1024, tile_tpb = 256;
    bool tuned = false;
    double tuned_ms = 0;                  // time of one timed iteration with the chosen tile
    void clear_graphs() {
        for (auto& kv : vgraphs) cudaGraphExecDestroy(kv.second);
        vgraphs.clear();
        for (auto& kv : igraphs) cudaGraphExecDestroy(kv.second);
        igraphs.clear();
    }
    int fail(int c, const std::string& m) { err = m; return c; }
    // zero-filled; the fill completes before returning: the uploads that follow
    // an allocation are plain cudaMemcpy calls, which nothing orders after
    // work on the solver's non-blocking stream
    template <class P> cudaError_t alloc(P** ptr, size_t bytes) {
        cudaError_t e = cudaMalloc((void**)ptr, bytes ? bytes : 16);
        if (e == cudaSuccess) {
            allocs.push_back(*ptr);
            e = cudaMemsetAsync(*ptr, 0, bytes ? bytes : 16, st);
            if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        }
        return e;
    }
    Dots D() const {
        const int n = S.nproblems;
        return Dots{dots, dots + n, dots + 2 * n, dots + 3 * n, dots + 4 * n, dots + 5 * n, dots + 6 * n, dots + 7 * n,
                    active, bprob};
    }
};

#define SCK(call, where)                                                                    \
    do {                                                                                    \
        cudaError_t e_ = (call);                                                            \
        if (e_ != cudaSuccess) return sv->fail(FALCON_ERR_CUDA, std::string(where) + ": " + cudaGetErrorString(e_)); \
    } while (0)

namespace {

// CTAs over (block, chunk of d.chunk cells), block-major: consecutive CTAs
// stream consecutive memory, and each per-problem reduction takes one atomic
// per chunk.
dim3 grid_cells(const LevelDims& d, int nblocks) {
    return dim3((unsigned)nblocks * (unsigned)((d.nint + d.chunk - 1) / d.chunk));
}
unsigned tpb(const LevelDims& d) { return (unsigned)std::min(d.tpb, (std::min(d.nint, d.chunk) + 31) / 32 * 32); }

cudaError_t halo_fill(falcon_solver* sv, int l, double* v) {
    const SvLevel& L = sv->lv[l];
    const int64_t n = L.nhc + L.nh;
    if (n > 0) k_halo<double><<<(unsigned)((n + 255) / 256), 256, 0, sv->st>>>(v, L.halo(), L.hcdst, L.hcsrc, L.nhc);
    return cudaGetLastError();
}

// power of two at or above max |v| over each problem's blocks (1 if all zero)
std::vector<double> problem_scale(const SolverProblemSet& S, const std::vector<double>& v, size_t per_block) {
    std::vector<double> m(S.nproblems, 0.0);
    for (int b = 0; b < S.nblocks; ++b) {
        double& q = m[S.block_problem[b]];
        for (size_t c = 0; c < per_block; ++c) q = std::max(q, std::fabs(v[(size_t)b * per_block + c]));
    }
    for (double& q : m) {
        if (!(q > 0) || !std::isfinite(q)) { q = 1.0; continue; }
        int e;
        std::frexp(q, &e);
        q = std::ldexp(1.0, e);
    }
    return m;
}
std::vector<float2> to_ff(const std::vector<double>& v, const std::vector<double>& scale_of_elem) {
    std::vector<float2> o(v.size());
    for (size_t q = 0; q < v.size(); ++q) {
        const double x = v[q] / scale_of_elem[q];
        const float h = (float)x;
        o[q] = make_float2(h, (float)(x - (double)h));
    }
    return o;
}

// ---- launches of the V-cycle kernels ---------------------------------------------
unsigned vgrid(int64_t threads) { return (unsigned)((threads + kVThreads - 1) / kVThreads); }
template <int M, int MODE>
void vsweep_pairs(falcon_solver* sv, int l, const float* zin, const float* zc, float* zout, int colour) {
    const SvLevel& L = sv->lv[l];
    const VLevel V = L.view(sv->S.nblocks);
    k_vsweep<M, MODE><<<vgrid((int64_t)V.nb * V.nint / 2), kVThreads, 0, sv->st>>>(V, L.r, zin, zc, zout, colour);
}
// of the kernels for any m (Cell)
struct AnyGrid {
    unsigned threads, ctas;
    explicit AnyGrid(const VLevel& V)
        : threads((unsigned)std::min(kVThreads, (V.nint + 31) / 32 * 32)), ctas((unsigned)V.nb * ((V.nint + threads - 1) / threads)) {}
};
// m not a power of two: pairs of cells above 1e5 cells of an even m, else a thread per
// cell with all its ghosts' loads at once. us per iteration by pairs / by cells: levels of
// 83k cells 137 / 109, of 166k 149 / 179, of 384k 126 / 160, of 2.2M 423 / 774
bool even_pairs(const VLevel& V) { return V.m % 2 == 0 && (int64_t)V.nb * V.nint > 100000; }
unsigned even_grid(const VLevel& V) { return (unsigned)V.nb * (((unsigned)V.nint / 2 + kVThreads - 1) / kVThreads); }
template <int MODE>
cudaError_t vsweep(falcon_solver* sv, int l, const float* zin, const float* zc, float* zout, int colour) {
    const SvLevel& L = sv->lv[l];
    switch (L.d.m0) {
    case 2: vsweep_pairs<2, MODE>(sv, l, zin, zc, zout, colour); break;
    case 4: vsweep_pairs<4, MODE>(sv, l, zin, zc, zout, colour); break;
    case 8: vsweep_pairs<8, MODE>(sv, l, zin, zc, zout, colour); break;
    case 16: vsweep_pairs<16, MODE>(sv, l, zin, zc, zout, colour); break;
    case 32: vsweep_pairs<32, MODE>(sv, l, zin, zc, zout, colour); break;
    default: {
        const VLevel V = L.view(sv->S.nblocks);
        const AnyGrid g(V);
        if constexpr (MODE == V_FIRST) {   // the red half sweep into the level's other buffer
            float* red = zout == L.z ? L.zb : L.z;
            k_vfirst_any<<<g.ctas, g.threads, 0, sv->st>>>(V, L.r, red);
            zin = red;
        } else if constexpr (MODE == V_PROLONG) {   // in place where a sweep follows
            float* sum = colour < 0 ? zout : zin == L.z ? L.z : L.zb;
            k_vprolong_any<<<g.ctas, g.threads, 0, sv->st>>>(V, zin, zc, sum);
            if (colour < 0) break;
        }
        if (even_pairs(V)) k_vsweep_even<<<even_grid(V), kVThreads, 0, sv->st>>>(V, L.r, zin, zout, colour);
        else k_vsweep_any<<<g.ctas, g.threads, 0, sv->st>>>(V, L.r, zin, zout, colour);
    }
    }
    return cudaGetLastError();
}
cudaError_t vresid(falcon_solver* sv, int l, const float* z, float* res) {
    const SvLevel& L = sv->lv[l];
    const VLevel V = L.view(sv->S.nblocks);
    const AnyGrid g(V);
    if (even_pairs(V)) k_vresid_even<<<even_grid(V), kVThreads, 0, sv->st>>>(V, L.r, z, res);
    else k_vresid<<<g.ctas, g.threads, 0, sv->st>>>(V, L.r, z, res);
    return cudaGetLastError();
}
// rc = R (r - A z)
template <int M> void vresid_restrict_pairs(falcon_solver* sv, int l, const float* z, float* rc) {
    const SvLevel& L = sv->lv[l];
    const VLevel V = L.view(sv->S.nblocks);
    k_vresid_restrict<M><<<vgrid((int64_t)V.nb * V.nint / 2), kVThreads, 0, sv->st>>>(V, L.r, z, rc);
}
cudaError_t vresid_restrict(falcon_solver* sv, int l, const float* z, float* rc) {
    const SvLevel& L = sv->lv[l];
    switch (L.d.m0) {
    case 2: vresid_restrict_pairs<2>(sv, l, z, rc); break;
    case 4: vresid_restrict_pairs<4>(sv, l, z, rc); break;
    case 8: vresid_restrict_pairs<8>(sv, l, z, rc); break;
    case 16: vresid_restrict_pairs<16>(sv, l, z, rc); break;
    default: {
        const cudaError_t e = vresid(sv, l, z, L.res);
        if (e != cudaSuccess) return e;
        const int64_t nc = (int64_t)sv->S.nblocks * L.d.nint / 8;
        k_vrestrict<<<vgrid(nc), kVThreads, 0, sv->st>>>(L.d.m0, (int)nc, L.res, rc);
    }
    }
    return cudaGetLastError();
}

constexpr size_t coarse_smem(int R, int slots) { return ((size_t)2 * R * kCoarseThreads + 1 + slots) * 4; }
typedef void (*CoarseKernel)(VLevel, CoarseArgs, const float*, float*);
template <int M> CoarseKernel coarse_kernel_m(int R, bool cluster) {
    if (cluster) return R == 1 ? k_coarse_sweeps<M, 1, true> : R == 2 ? k_coarse_sweeps<M, 2, true> : k_coarse_sweeps<M, 4, true>;
    return R == 1 ? k_coarse_sweeps<M, 1, false> : R == 2 ? k_coarse_sweeps<M, 2, false> : k_coarse_sweeps<M, 4, false>;
}
CoarseKernel coarse_kernel(int m, int R, bool cluster) {
    return m == 2 ? coarse_kernel_m<2>(R, cluster) : m == 4 ? coarse_kernel_m<4>(R, cluster) : nullptr;
}
void coarse_config(const falcon_solver* sv, cudaLaunchConfig_t* cfg, cudaLaunchAttribute* at) {
    *cfg = cudaLaunchConfig_t{};
    cfg->gridDim = dim3((unsigned)(sv->S.nproblems * sv->coarse_cluster));
    cfg->blockDim = dim3(kCoarseThreads);
    cfg->dynamicSmemBytes = coarse_smem(sv->coarse_r, sv->coarse_slots);
    cfg->stream = sv->st;
    at->id = cudaLaunchAttributeClusterDimension;
    at->val.clusterDim.x = (unsigned)sv->coarse_cluster;
    at->val.clusterDim.y = at->val.clusterDim.z = 1;
    cfg->attrs = at;
    cfg->numAttrs = sv->coarse_cluster > 1 ? 1 : 0;
}
cudaError_t coarse_sweeps(falcon_solver* sv, int sweeps, float* zout) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at[1];
    coarse_config(sv, &cfg, at);
    const SvLevel& L = sv->lv.back();
    return cudaLaunchKernelEx(&cfg, coarse_kernel(L.d.m0, sv->coarse_r, sv->coarse_cluster > 1), L.view(sv->S.nblocks),
                              CoarseArgs{sv->first, sv->cghost, sv->ceat, sv->cew, sv->clist, sweeps, sv->coarse_cluster},
                              (const float*)L.r, zout);
}
// A kernel's opt-ins hold for every solver of the process, whichever set them last: all
// set the same, the most shared memory that a plan may ask for.
constexpr size_t kCoarseSmemMax = 232448;
cudaError_t allow_coarse(CoarseKernel kern, int cluster) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCoarseSmemMax);
    if (e == cudaSuccess && cluster > 8) e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    return e;
}
// Whether the coarsest level's sweeps run as one launch, and with how many CTAs per
// problem: the cluster with the shortest estimated half sweep -- barriers (a cluster's
// take about three times a CTA's) plus a share per cell of a thread and colour -- times
// the waves that the batch's clusters take, as far as the estimate stays below 4. A launch
// per half sweep advances all problems at once and is as fast from there on. us per
// iteration with 32 sweeps, one launch / launches: 24 x 45 127 / 416, 64 x 180 (16 CTAs of
// four cells) 780 / 916, 16 x 24 x 45 262 / 603, batch of 8 1,012 / 1,180; above the
// limit 16 problems 2,494 / 2,475, 32 problems 4,724 / 4,424. Builds the neighbour words.
int plan_coarse(falcon_solver* sv, const std::vector<int32_t>& ghost, const std::vector<int32_t>& isrc,
                const std::vector<uint8_t>& icode, const std::vector<float>& iw) {
    const SolverProblemSet& S = sv->S;
    sv->coarse_cluster = 0;
    const SvLevel& L = sv->lv.back();
    const int m = L.d.m0, nint = L.d.nint, mm = m * m;
    if (S.nlevels < 2 || !coarse_kernel(m, 1, false)) return FALCON_OK;
    int most = 0;
    for (int p = 0; p < S.nproblems; ++p) most = std::max(most, S.problem_first_block[p + 1] - S.problem_first_block[p]);
    // the cluster with the shortest estimated half sweep, waves of clusters counted
    int cl = 0, R = 1;
    double best = 1e30;
    for (int c = 1; c <= 16; c *= 2) {
        const int64_t cells = (int64_t)((most + c - 1) / c) * nint;
        if (cells > 8 * kCoarseThreads) continue;
        const int r = cells <= 2 * kCoarseThreads ? 1 : cells <= 4 * kCoarseThreads ? 2 : 4;
        sv->coarse_cluster = c;
        const CoarseKernel kern = coarse_kernel(m, r, c > 1);
        int n = 152;
        if (c > 1) {
            cudaLaunchConfig_t cfg;
            cudaLaunchAttribute at[1];
            coarse_config(sv, &cfg, at);
            cfg.dynamicSmemBytes = coarse_smem(r, 4 * kCoarseThreads);
            cudaError_t e = allow_coarse(kern, c);
            if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&n, kern, &cfg);
            if (e != cudaSuccess || n < 1) {
                cudaGetLastError();
                continue;
            }
        }
        const double t = ((S.nproblems + n - 1) / n) * ((c == 1 ? 0.35 : 1.0) + 0.25 * r);
        if (t < best) {
            best = t;
            cl = c;
            R = r;
        }
    }
    sv->coarse_cluster = 0;
    if (cl == 0 || best > 4.0) return FALCON_OK;
    // owner CTA of a block, and the word of a cell
    auto cta = [&](int b) {
        const int p = S.block_problem[b], pb0 = S.problem_first_block[p];
        const int bpc = (S.problem_first_block[p + 1] - pb0 + cl - 1) / cl;
        return p * cl + (b - pb0) / bpc;
    };
    auto colour = [&](int c) { return (c % m + (c / m) % m + c / mm + 1) & 1; };
    auto word = [&](int cell) -> uint32_t {
        const int b = cell / nint, c = cell - b * nint, p = S.block_problem[b], pb0 = S.problem_first_block[p];
        const int bpc = (S.problem_first_block[p + 1] - pb0 + cl - 1) / cl, own = (b - pb0) / bpc;
        return (uint32_t)own << 24 | (uint32_t)((b - pb0 - own * bpc) * nint + c);
    };
    // ghosts by (CTA, colour of the cell inside the face): local copies of the other
    // colour are read in place, the rest gathered
    std::vector<uint32_t> g(ghost.size(), kNone);
    std::vector<uint2> eat;
    std::vector<float4> ew;
    std::vector<int4> list;
    int slots = 0, b = 0;
    for (int c = 0; c < S.nproblems * cl; ++c) {
        int be = b;
        while (be < S.nblocks && cta(be) == c) ++be;
        for (int col = 0; col < 2; ++col) {
            const int start = (int)eat.size();
            std::vector<size_t> place[2];   // ghosts of one entry and of two
            std::vector<CoarseEntry> one[2], two;
            for (int bb = b; bb < be; ++bb)
                for (int f = 0; f < 6; ++f)
                    for (int t = 0; t < mm; ++t) {
                        const int u = t % m, v = t / m, in = (f & 1) ? m - 1 : 0;
                        const int i = f < 2 ? in : u, j = f < 2 ? u : f < 4 ? in : v, k = f < 4 ? v : in;
                        if (((i + j + k + 1) & 1) != col) continue;
                        const size_t q = ((size_t)bb * 6 + f) * mm + t;
                        const int32_t d = ghost[q];
                        if (d == -1) continue;
                        if (d >= 0 && cta(d / nint) == c && colour(d % nint) != col) {
                            g[q] = word(d) & 0xffffu;
                            continue;
                        }
                        CoarseEntry E{make_uint2(0, 0), make_float4(1.f, 0.f, 0.f, 0.f)};
                        bool eight = false;
                        if (d >= 0) {
                            E.at.x = word(d);
                        } else {
                            const size_t e = (size_t)(-2 - d);
                            const float wi = iw[3 * e], wj = iw[3 * e + 1], wk = iw[3 * e + 2], ui = 1.f - wi;
                            const float p[4] = {(1.f - wj) * (1.f - wk), wj * (1.f - wk), (1.f - wj) * wk, wj * wk};
                            E.at.x = word(isrc[e]);
                            if (icode[e] == 1) {
                                E.at.y = 1;
                                E.w = make_float4(ui, wi, 0.f, 0.f);
                            } else {   // offsets whose weight is 0 are never used
                                eight = icode[e] & 1;
                                E.at.y = (uint32_t)(m | mm << 8 | (m + mm) << 16);
                                E.w = make_float4(ui * p[0], ui * p[1], ui * p[2], ui * p[3]);
                                CoarseEntry H = E;
                                H.at.x += 1;
                                H.w = make_float4(wi * p[0], wi * p[1], wi * p[2], wi * p[3]);
                                if (eight) two.push_back(H);
                            }
                        }
                        place[eight].push_back(q);
                        one[eight].push_back(E);
                    }
            int n = 0;
            for (int e = 0; e < 2; ++e)
                for (size_t x = 0; x < place[e].size(); ++x) {
                    g[place[e][x]] = kSlot | (uint32_t)n++;
                    eat.push_back(one[e][x].at);
                    ew.push_back(one[e][x].w);
                }
            for (const CoarseEntry& H : two) {
                eat.push_back(H.at);
                ew.push_back(H.w);
            }
            slots = std::max(slots, n);
            list.push_back(make_int4(start, n, (int)two.size(), 0));
        }
        b = be;
    }
    sv->coarse_cluster = cl;
    sv->coarse_r = R;
    sv->coarse_slots = slots;
    const CoarseKernel kern = coarse_kernel(m, R, cl > 1);
    cudaError_t e = coarse_smem(R, slots) > kCoarseSmemMax || 2 * R * kCoarseThreads + 1 + slots > 65536
                        ? cudaErrorInvalidValue
                        : allow_coarse(kern, cl);
    int n = 1;
    if (e == cudaSuccess && cl > 1) {
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute at[1];
        coarse_config(sv, &cfg, at);
        e = cudaOccupancyMaxActiveClusters(&n, kern, &cfg);
    }
    if (e != cudaSuccess || n < 1) {   // the device does not take this cluster
        cudaGetLastError();
        sv->coarse_cluster = 0;
        return FALCON_OK;
    }
    SCK(sv->alloc(&sv->cghost, g.size() * 4), "coarse words");
    SCK(sv->alloc(&sv->ceat, eat.size() * sizeof(uint2)), "coarse words");
    SCK(sv->alloc(&sv->cew, ew.size() * sizeof(float4)), "coarse words");
    SCK(sv->alloc(&sv->clist, list.size() * sizeof(int4)), "coarse words");
    SCK(cudaMemcpy(sv->cghost, g.data(), g.size() * 4, cudaMemcpyHostToDevice), "coarse words");
    SCK(cudaMemcpy(sv->clist, list.data(), list.size() * sizeof(int4), cudaMemcpyHostToDevice), "coarse words");
    if (!eat.empty()) {
        SCK(cudaMemcpy(sv->ceat, eat.data(), eat.size() * sizeof(uint2), cudaMemcpyHostToDevice), "coarse words");
        SCK(cudaMemcpy(sv->cew, ew.data(), ew.size() * sizeof(float4), cudaMemcpyHostToDevice), "coarse words");
    }
    return FALCON_OK;
}

// Whether `sweeps` red-black sweeps of level l from z = 0 are one launch: on a small
// coarsest level, where several launches are saved
bool sweeps_in_one_launch(const falcon_solver* sv, int l, int sweeps) {
    const int nl = (int)sv->lv.size();
    return l == nl - 1 && nl > 1 && sv->coarse_cluster > 0 && sweeps > 2;
}
// `sweeps` (at least one) red-black sweeps of level l on its r from z = 0. z: the first
// launch's output, next(): the output of each launch after it
template <class F> cudaError_t smooth_from_zero(falcon_solver* sv, int l, int sweeps, float* z, F next) {
    if (sweeps_in_one_launch(sv, l, sweeps)) return coarse_sweeps(sv, sweeps, z);
    cudaError_t e = vsweep<V_FIRST>(sv, l, nullptr, nullptr, z, 1);
    for (int s = 2; s < 2 * sweeps && e == cudaSuccess; ++s) {
        float* out = next();
        e = vsweep<V_PLAIN>(sv, l, z, nullptr, out, s & 1);
        z = out;
    }
    return e;
}

// z_0 = M r_0: one V-cycle on the FP32 residual stored in lv[0].r, into lv[0].z
cudaError_t vcycle_body(falcon_solver* sv) {
    const int nl = (int)sv->lv.size(), nb = sv->S.nblocks;
    cudaError_t e = cudaSuccess;
    // the sweeps are out of place: a level's buffers take turns so that its last write lands in z
    std::vector<int> left(nl);
    std::vector<float*> zc(nl, nullptr);
    auto next = [&](int l) { return --left[l] & 1 ? sv->lv[l].zb : sv->lv[l].z; };
    auto plain = [&](int l, int colour) {
        if (e != cudaSuccess) return;
        float* out = next(l);
        e = vsweep<V_PLAIN>(sv, l, zc[l], nullptr, out, colour);
        zc[l] = out;
    };
    for (int l = 0; l < nl && e == cudaSuccess; ++l) {
        SvLevel& L = sv->lv[l];
        const bool coarsest = l == nl - 1 && nl > 1, net = coarsest && sv->use_net;
        const int sweeps = net ? sv->net_sweeps : l == nl - 1 ? sv->nu_coarse : sv->nu_pre;
        const bool one = !net && sweeps_in_one_launch(sv, l, sweeps);
        left[l] = (net ? 1 + 2 * sweeps : one || sweeps == 0 ? 1 : 2 * sweeps - 1) +
                  (l < nl - 1 ? std::max(1, 2 * sv->nu_post) : 0);
        if (coarsest && sv->rec && sv->rec_n < sv->rec_max)
            e = cudaMemcpyAsync(sv->rec + (size_t)sv->rec_n++ * nb * L.d.nint, L.r, (size_t)nb * L.d.nint * 4,
                                cudaMemcpyDeviceToDevice, sv->st);
        if (e != cudaSuccess) break;
        zc[l] = next(l);
        if (net) {
            // z_c = s * net(r_c / diag / s, operator) then a few sweeps
            const int64_t N = (int64_t)nb * L.d.nint;
            e = cudaMemsetAsync(sv->csum, 0, 8, sv->st);
            if (e == cudaSuccess) {
                k_lcc_sumsq<<<grid_cells(L.d, nb), tpb(L.d), 0, sv->st>>>(L.d, L.r, L.fAii, sv->csum);
                k_lcc_feat<<<grid_cells(L.d, nb), tpb(L.d), 0, sv->st>>>(L.d, L.r, L.fAii, sv->gmap, sv->csum, N, sv->feat);
                e = lcc::forward_device(sv->net, sv->feat, 2, sv->cD, sv->cH, sv->cW, sv->yout, sv->st);
            }
            if (e == cudaSuccess) {
                k_lcc_scatter<<<grid_cells(L.d, nb), tpb(L.d), 0, sv->st>>>(L.d, sv->yout, sv->gmap, sv->csum, N, zc[l]);
                e = cudaGetLastError();
            }
            for (int s = 0; s < 2 * sweeps; ++s) plain(l, s & 1);
        } else if (sweeps == 0) {
            e = cudaMemsetAsync(zc[l], 0, (size_t)nb * L.d.nint * 4, sv->st);
        } else {
            e = smooth_from_zero(sv, l, sweeps, zc[l], [&] { return zc[l] = next(l); });
        }
        if (l + 1 < nl && e == cudaSuccess) e = vresid_restrict(sv, l, zc[l], sv->lv[l + 1].r);
    }
    for (int l = nl - 2; l >= 0 && e == cudaSuccess; --l) {
        float* out = next(l);
        e = vsweep<V_PROLONG>(sv, l, zc[l], zc[l + 1], out, sv->nu_post ? 1 : -1);
        zc[l] = out;
        for (int s = 1; s < 2 * sv->nu_post; ++s) plain(l, 1 - (s & 1));
    }
    return e;
}

// z_0 = M r_0 as one CUDA graph launch: the V-cycle's launches are
// captured once per shape and replayed (recording calls run eagerly: their
// destination changes from call to call)
cudaError_t vcycle(falcon_solver* sv) {
    if (sv->rec || sv->capturing) return vcycle_body(sv);
    const int64_t key = (int64_t)(sv->use_net ? 1 : 0) | ((int64_t)sv->nu_pre << 1) | ((int64_t)sv->nu_post << 8) |
                        ((int64_t)sv->nu_coarse << 15) | ((int64_t)sv->net_sweeps << 28);
    auto it = sv->vgraphs.find(key);
    if (it == sv->vgraphs.end()) {
        cudaGraph_t g = nullptr;
        cudaError_t e = cudaStreamBeginCapture(sv->st, cudaStreamCaptureModeThreadLocal);
        if (e != cudaSuccess) return e;
        const cudaError_t eb = vcycle_body(sv);
        e = cudaStreamEndCapture(sv->st, &g);
        if (eb != cudaSuccess) { if (g) cudaGraphDestroy(g); return eb; }
        if (e != cudaSuccess) return e;
        cudaGraphExec_t x = nullptr;
        e = cudaGraphInstantiate(&x, g, 0);
        cudaGraphDestroy(g);
        if (e != cudaSuccess) return e;
        it = sv->vgraphs.emplace(key, x).first;
    }
    return cudaGraphLaunch(it->second, sv->st);
}

// The tile shape of every cell kernel (all levels); launch shapes are baked
// into the captured graphs, so they go.
void apply_tile(falcon_solver* sv, int chunk, int tpb_) {
    sv->tile_chunk = chunk;
    sv->tile_tpb = tpb_;
    for (SvLevel& L : sv->lv) {
        L.d.chunk = chunk;
        L.d.tpb = tpb_;
    }
    sv->clear_graphs();
}

int setup(falcon_solver* sv) {
    SolverProblemSet& S = sv->S;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return sv->fail(FALCON_ERR_NO_DEVICE, "no CUDA device");
    SCK(cudaSetDevice(sv->device), "cudaSetDevice");
    SCK(cudaStreamCreateWithFlags(&sv->st, cudaStreamNonBlocking), "stream");
    const int nb = S.nblocks;
    sv->lv.resize(S.nlevels);
    for (int l = 0; l < S.nlevels; ++l) {
        const SolverLevel& H = S.L[l];
        SvLevel& L = sv->lv[l];
        L.d.m0 = H.m[0]; L.d.m1 = H.m[1]; L.d.m2 = H.m[2];
        L.d.p0 = H.m[0] + 2; L.d.p1 = H.m[1] + 2; L.d.p2 = H.m[2] + 2;
        L.d.nint = H.nint();
        L.d.npad = L.d.p0 * L.d.p1 * L.d.p2;
        L.d.chunk = sv->tile_chunk;
        L.d.tpb = sv->tile_tpb;
        auto up64 = [&](double** d, const std::vector<double>& h) -> cudaError_t {
            cudaError_t e = sv->alloc(d, h.size() * 8);
            if (e == cudaSuccess) e = cudaMemcpy(*d, h.data(), h.size() * 8, cudaMemcpyHostToDevice);
            return e;
        };
        auto up32 = [&](float** d, const std::vector<double>& h) -> cudaError_t {
            std::vector<float> f(h.begin(), h.end());
            cudaError_t e = sv->alloc(d, f.size() * 4);
            if (e == cudaSuccess) e = cudaMemcpy(*d, f.data(), f.size() * 4, cudaMemcpyHostToDevice);
            return e;
        };
        SCK(up64(&L.Aii, H.Aii), "operator");
        SCK(up64(&L.Ai, H.Ai), "operator");
        SCK(up64(&L.Aj, H.Aj), "operator");
        SCK(up64(&L.Ak, H.Ak), "operator");
        SCK(up32(&L.fAii, H.Aii), "operator");
        SCK(up32(&L.fAi, H.Ai), "operator");
        SCK(up32(&L.fAj, H.Aj), "operator");
        SCK(up32(&L.fAk, H.Ak), "operator");
        // halo entries: the FP64 lists (padded offsets; entries with all
        // weights zero are plain copies, a separate list of 8 bytes each), and
        // the FP32 V-cycle's ghost descriptors (interior cell indices). The
        // map's weights at aligned neighbours are 0 or 1 up to rounding (about
        // 1e-14), seldom exactly: in FP32 a weight within 2^-24 of 0 or 1 changes
        // nothing but the last bit, so those ghosts become copies (one read
        // instead of eight; all but the Yin-Yang seam's).
        const size_t nent = H.halo.size();
        const int m = H.m[0];
        constexpr double kSnap = 1.0 / (1 << 24);
        auto snapped = [](double x) { return x < kSnap ? 0.0 : x > 1.0 - kSnap ? 1.0 : x; };
        std::vector<int32_t> ent(nent), ent32(nent);   // index of an interpolated entry, or -1 - (index of a copy)
        int32_t ni = 0, ncp = 0, ni32 = 0;
        for (size_t q = 0; q < nent; ++q) {
            const double* w = H.halo[q].w;
            ent[q] = w[0] == 0.0 && w[1] == 0.0 && w[2] == 0.0 ? -1 - ncp++ : ni++;
            bool copy = true;
            for (int dd = 0; dd < 3; ++dd) {
                const double x = snapped(w[dd]);
                copy = copy && (x == 0.0 || x == 1.0);
            }
            ent32[q] = copy ? -1 : ni32++;
        }
        const size_t n = (size_t)ni, nc = (size_t)ncp, n32 = (size_t)ni32;
        std::vector<int32_t> dst(n), src(n), cdst(nc), csrc(nc), isrc(n32), ghost((size_t)nb * 6 * m * m, -1);
        std::vector<double> w(3 * n);
        std::vector<uint8_t> code(n), icode(n32);
        std::vector<float> iw(3 * n32);
        std::vector<size_t> slot_of(nent);   // a halo entry's place in the ghost tables
#pragma omp parallel for schedule(static)
        for (int64_t qq = 0; qq < (int64_t)nent; ++qq) {
            const size_t q = (size_t)qq;
            const HaloEntry& h = H.halo[q];
            const int32_t t = (int32_t)(h.tb * (int64_t)L.d.npad + ((int64_t)h.tk * L.d.p1 + h.tj) * L.d.p0 + h.ti);
            const int32_t f = (int32_t)(h.sb * (int64_t)L.d.npad + ((int64_t)h.k0 * L.d.p1 + h.j0) * L.d.p0 + h.i0);
            if (ent[q] < 0) {
                const size_t c = (size_t)(-1 - ent[q]);
                cdst[c] = t;
                csrc[c] = f;
            } else {
                const size_t e = (size_t)ent[q];
                dst[e] = t;
                src[e] = f;
                code[e] = 0;
                for (int dd = 0; dd < 3; ++dd) {
                    w[3 * e + dd] = h.w[dd];
                    if (h.w[dd] != 0.0) code[e] |= (uint8_t)(1 << dd);
                }
            }
            const int32_t step[3] = {1, m, m * m};
            int32_t base = (int32_t)(h.sb * (int64_t)L.d.nint + ((int64_t)(h.k0 - 1) * m + h.j0 - 1) * m + h.i0 - 1);
            uint8_t cd = 0;
            float w3[3];
            for (int dd = 0; dd < 3; ++dd) {
                double x = snapped(h.w[dd]);
                if (x == 1.0) {
                    base += step[dd];
                    x = 0.0;
                }
                w3[dd] = (float)x;
                if (x != 0.0) cd |= (uint8_t)(1 << dd);
            }
            const int axis = h.ti < 1 || h.ti > m ? 0 : h.tj < 1 || h.tj > m ? 1 : 2;
            const int tt[3] = {h.ti, h.tj, h.tk}, hi = tt[axis] > m;
            const int pos = axis == 0 ? (h.tk - 1) * m + h.tj - 1 : axis == 1 ? (h.tk - 1) * m + h.ti - 1 : (h.tj - 1) * m + h.ti - 1;
            const int32_t e32 = ent32[q];
            slot_of[q] = (size_t)h.tb * 6 * m * m + (size_t)(2 * axis + hi) * m * m + pos;
            ghost[slot_of[q]] = e32 < 0 ? base : -2 - e32;
            if (e32 < 0) continue;
            isrc[e32] = base;
            icode[e32] = cd;
            for (int dd = 0; dd < 3; ++dd) iw[3 * (size_t)e32 + dd] = w3[dd];
        }
        L.nh = (int64_t)n;
        L.nhc = (int64_t)nc;
        auto up = [&](auto** dp, const auto& v) -> cudaError_t {
            cudaError_t e = sv->alloc(dp, v.size() * sizeof(v[0]));
            if (e == cudaSuccess && !v.empty()) e = cudaMemcpy(*dp, v.data(), v.size() * sizeof(v[0]), cudaMemcpyHostToDevice);
            return e;
        };
        SCK(up(&L.hdst, dst), "halo");
        SCK(up(&L.hsrc, src), "halo");
        SCK(up(&L.hcode, code), "halo");
        SCK(up(&L.hw, w), "halo");
        SCK(up(&L.hcdst, cdst), "halo");
        SCK(up(&L.hcsrc, csrc), "halo");
        SCK(up(&L.ghost, ghost), "halo");
        SCK(up(&L.isrc, isrc), "halo");
        SCK(up(&L.icode, icode), "halo");
        SCK(up(&L.iw, iw), "halo");
        // faces whose ghosts come from one block, position by position (VLevel::nbr)
        std::vector<int32_t> nbr((size_t)nb * 12, -2);
#pragma omp parallel for schedule(static)
        for (int gb = 0; gb < nb; ++gb)
            for (int f = 0; f < 6; ++f) {
                const int32_t* gf = &ghost[((size_t)gb * 6 + f) * m * m];
                // the entry's base cell and its weight along i; other directions disqualify
                auto base = [&](int t, float& wi) -> int32_t {
                    wi = 0.f;
                    if (gf[t] >= -1) return gf[t];
                    const size_t e = (size_t)(-2 - gf[t]);
                    if (f > 1 || icode[e] != 1) return -1;
                    wi = iw[3 * e];
                    return isrc[e];
                };
                float w0 = 0.f, wt = 0.f;
                const int32_t b0 = base(0, w0);
                const int own = b0 >= 0 ? b0 / L.d.nint : -1, i0 = f < 2 ? b0 % m : 0;
                bool none = true, same = own >= 0;
                for (int t = 0; t < m * m; ++t) {
                    const int u = t % m, v = t / m, in = (f & 1) ? 0 : m - 1;
                    const int i = f < 2 ? i0 : u, j = f < 2 ? u : f < 4 ? in : v, k = f < 4 ? v : in;
                    none = none && gf[t] == -1;
                    same = same && base(t, wt) == own * L.d.nint + (k * m + j) * m + i && wt == w0;
                }
                int32_t* o = &nbr[(size_t)gb * 12];
                o[f] = none ? -2 : same ? own : -1;
                if (f > 1) continue;
                o[6 + f] = i0;
                std::memcpy(&o[8 + f], &w0, 4);
            }
        SCK(up(&L.nbr, nbr), "halo");
        if (l == S.nlevels - 1) {
            const int rc = plan_coarse(sv, ghost, isrc, icode, iw);
            if (rc) return rc;
        }
        if (l == 0) {   // the ghosts of the float-float iteration (GhostFF)
            constexpr double kSnapFF = 1.0 / (1LL << 32);
            const size_t ns = ghost.size();
            std::vector<int32_t> gd(ns, -1), esrc;
            std::vector<float> eps(3 * ns, 0.f);
            std::vector<size_t> two;   // halo entries that stay interpolations
            for (size_t q = 0; q < nent; ++q) {
                const HaloEntry& h = H.halo[q];
                const int32_t st[3] = {1, m, m * m};
                const size_t slot = slot_of[q];
                int32_t base = (int32_t)(h.sb * (int64_t)L.d.nint + ((int64_t)(h.k0 - 1) * m + h.j0 - 1) * m + h.i0 - 1);
                bool copy = true;
                for (int dd = 0; dd < 3; ++dd) copy = copy && (h.w[dd] < kSnapFF || h.w[dd] > 1.0 - kSnapFF);
                if (!copy) {
                    gd[slot] = -2 - (int32_t)two.size();
                    two.push_back(q);
                    esrc.push_back(base);
                    continue;
                }
                for (int dd = 0; dd < 3; ++dd) {
                    if (h.w[dd] > 0.5) {
                        base += st[dd];
                        eps[3 * slot + dd] = -(float)(1.0 - h.w[dd]);
                    } else {
                        eps[3 * slot + dd] = (float)h.w[dd];
                    }
                }
                gd[slot] = base;
            }
            std::vector<float2> w8(8 * two.size());
            std::vector<uint8_t> ecode(two.size());
#pragma omp parallel for schedule(static)
            for (int64_t e = 0; e < (int64_t)two.size(); ++e) {
                const double* hw = H.halo[two[(size_t)e]].w;
                const double wi = hw[0], wj = hw[1], wk = hw[2];
                const double ui = 1.0 - wi, uj = 1.0 - wj, uk = 1.0 - wk;
                const double c8[8] = {ui * uj * uk, wi * uj * uk, ui * wj * uk, ui * uj * wk,
                                      wi * wj * uk, ui * wj * wk, wi * uj * wk, wi * wj * wk};
                for (int t = 0; t < 8; ++t) {
                    const float h = (float)c8[t];
                    w8[8 * (size_t)e + t] = make_float2(h, (float)(c8[t] - (double)h));
                }
                ecode[(size_t)e] = (uint8_t)((wi != 0.0 ? 1 : 0) | (wj != 0.0 ? 2 : 0) | (wk != 0.0 ? 4 : 0));
            }
            int32_t *dg, *ds;
            float* de;
            uint8_t* dc;
            float2* dw;
            SCK(up(&dg, gd), "halo");
            SCK(up(&de, eps), "halo");
            SCK(up(&ds, esrc), "halo");
            SCK(up(&dc, ecode), "halo");
            SCK(up(&dw, w8), "halo");
            SCK(sv->alloc(&sv->ghosts2, ns * sizeof(float2)), "halo");
            sv->gff = GhostFF{dg, de, ds, dc, dw, m, (int64_t)ns};
        }
        SCK(sv->alloc(&L.z, (size_t)nb * L.d.nint * 4), "vectors");
        SCK(sv->alloc(&L.zb, (size_t)nb * L.d.nint * 4), "vectors");
        SCK(sv->alloc(&L.r, (size_t)nb * L.d.nint * 4), "vectors");
        SCK(sv->alloc(&L.res, (size_t)nb * L.d.nint * 4), "vectors");
    }
    const LevelDims& d0 = sv->lv[0].d;
    SCK(sv->alloc(&sv->x, (size_t)nb * d0.npad * 8), "vectors");
    SCK(sv->alloc(&sv->p, (size_t)nb * d0.npad * 8), "vectors");
    SCK(sv->alloc(&sv->r, (size_t)nb * d0.nint * 8), "vectors");
    SCK(sv->alloc(&sv->Ap, (size_t)nb * d0.nint * 8), "vectors");
    SCK(sv->alloc(&sv->z, (size_t)nb * d0.nint * 8), "vectors");
    SCK(sv->alloc(&sv->bvec, (size_t)nb * d0.nint * 8), "vectors");
    SCK(sv->alloc(&sv->dots, (size_t)8 * S.nproblems * 8), "scalars");
    SCK(sv->alloc(&sv->ir_par, (size_t)2 * S.nproblems * 8), "scalars");
    SCK(sv->alloc(&sv->rr0, (size_t)S.nproblems * 8), "scalars");
    SCK(sv->alloc(&sv->eta, (size_t)S.nproblems * 8), "scalars");
    SCK(sv->alloc(&sv->ictl, sizeof(InnerCtl)), "scalars");
    SCK(sv->alloc(&sv->active, (size_t)S.nproblems * 4), "scalars");
    SCK(sv->alloc(&sv->bprob, (size_t)nb * 4), "scalars");
    SCK(cudaMemcpy(sv->bvec, S.b.data(), S.b.size() * 8, cudaMemcpyHostToDevice), "rhs");
    SCK(cudaMemcpy(sv->bprob, S.block_problem.data(), (size_t)nb * 4, cudaMemcpyHostToDevice), "scalars");
    // the float-float solve: A' = A / sA per problem (sA from the diagonal)
    {
        const SolverLevel& H = S.L[0];
        const size_t nint = (size_t)d0.nint;
        sv->sA = problem_scale(S, H.Aii, nint);
        auto upff = [&](float2** dptr, const std::vector<double>& h) -> cudaError_t {
            const size_t per = h.size() / (size_t)nb;   // entries per block
            std::vector<double> sc(h.size());
            for (int b = 0; b < nb; ++b)
                for (size_t c = 0; c < per; ++c) sc[(size_t)b * per + c] = sv->sA[S.block_problem[b]];
            const std::vector<float2> f = to_ff(h, sc);
            cudaError_t e = sv->alloc(dptr, f.size() * sizeof(float2));
            if (e == cudaSuccess) e = cudaMemcpy(*dptr, f.data(), f.size() * sizeof(float2), cudaMemcpyHostToDevice);
            return e;
        };
        SvLevel& L0 = sv->lv[0];
        SCK(upff(&L0.Aii2, H.Aii), "operator");
        SCK(upff(&L0.Ai2, H.Ai), "operator");
        SCK(upff(&L0.Aj2, H.Aj), "operator");
        SCK(upff(&L0.Ak2, H.Ak), "operator");
        for (float2** v : {&sv->x2, &sv->p2, &sv->r2, &sv->Ap2, &sv->w2})
            SCK(sv->alloc(v, (size_t)nb * d0.nint * sizeof(float2)), "vectors");
        std::vector<float> fa(sv->sA.begin(), sv->sA.end());
        SCK(sv->alloc(&sv->dsA, fa.size() * 4), "scalars");
        SCK(cudaMemcpy(sv->dsA, fa.data(), fa.size() * 4, cudaMemcpyHostToDevice), "scalars");
    }
    SCK(sv->alloc(&sv->first, (size_t)(S.nproblems + 1) * 4), "scalars");
    SCK(cudaMemcpy(sv->first, S.problem_first_block.data(), (size_t)(S.nproblems + 1) * 4, cudaMemcpyHostToDevice), "scalars");
    apply_tile(sv, sv->tile_chunk, sv->tile_tpb);
    SCK(uploads_arrived(), "setup");
    SCK(cudaStreamSynchronize(sv->st), "setup");
    return FALCON_OK;
}

// scatter an interior [b][nint] vector into the padded x
template <class T>
__global__ void k_scatter_pad(LevelDims d, const T* v, T* x) {
    const int b = cell_block(d), c0 = cell_first(d), c1 = cell_end(d);
    for (int c = c0 + threadIdx.x; c < c1; c += blockDim.x) {
        int i, j, k;
        cell_ijk(d, c, i, j, k);
        x[pidx(d, b, i, j, k)] = v[(size_t)b * d.nint + c];
    }
}
template <class T>
__global__ void k_gather_pad(LevelDims d, const T* x, T* v) {
    const int b = cell_block(d), c0 = cell_first(d), c1 = cell_end(d);
    for (int c = c0 + threadIdx.x; c < c1; c += blockDim.x) {
        int i, j, k;
        cell_ijk(d, c, i, j, k);
        v[(size_t)b * d.nint + c] = x[pidx(d, b, i, j, k)];
    }
}

// Map the coarsest level onto one dense grid per panel (single problem,
// whole uniform blocks); builds gmap and the static input channels.
int ensure_coarse_map(falcon_solver* sv) {
    if (sv->cmap_ok) return FALCON_OK;
    const SolverProblemSet& S = sv->S;
    if (!sv->st) return sv->fail(FALCON_ERR_NO_DEVICE, "solver created without a device");
    if (S.nproblems != 1) return sv->fail(FALCON_ERR_INVALID_ARG, "learned coarse correction: single-problem solvers only");
    if (S.nlevels < 2) return sv->fail(FALCON_ERR_INVALID_ARG, "learned coarse correction: needs at least 2 levels");
    const int lc = S.nlevels - 1, nb = S.nblocks;
    const SolverLevel& C = S.L[lc];
    const Grid& g = S.grids[0];
    int tiles[2][3] = {{0, 0, 0}, {0, 0, 0}};
    std::vector<int32_t> bt((size_t)nb * 3), bpan(nb);
    for (int pnl = 0; pnl < 2; ++pnl) {
        int count = 0;
        for (int ax = 0; ax < 3; ++ax) {
            std::vector<double> starts;
            for (int b = 0; b < nb; ++b)
                if (((S.block_flags[b] & 1) != 0) == (pnl == 0)) starts.push_back(g.ranges[(size_t)b * 6 + ax * 2]);
            std::sort(starts.begin(), starts.end());
            std::vector<double> uniq;
            for (double v : starts)
                if (uniq.empty() || std::fabs(v - uniq.back()) > 1e-12 * std::max(1.0, std::fabs(v))) uniq.push_back(v);
            tiles[pnl][ax] = (int)uniq.size();
            for (int b = 0; b < nb; ++b) {
                if (((S.block_flags[b] & 1) != 0) != (pnl == 0)) continue;
                const double v = g.ranges[(size_t)b * 6 + ax * 2];
                int idx = 0;
                while (idx + 1 < (int)uniq.size() && v > uniq[idx] + 1e-12 * std::max(1.0, std::fabs(v))) ++idx;
                bt[(size_t)b * 3 + ax] = idx;
                bpan[b] = pnl;
            }
        }
        for (int b = 0; b < nb; ++b) count += ((S.block_flags[b] & 1) != 0) == (pnl == 0);
        if (count != tiles[pnl][0] * tiles[pnl][1] * tiles[pnl][2])
            return sv->fail(FALCON_ERR_INVALID_ARG, "learned coarse correction: blocks do not tile the panels uniformly");
    }
    for (int ax = 0; ax < 3; ++ax)
        if (tiles[0][ax] != tiles[1][ax]) return sv->fail(FALCON_ERR_INVALID_ARG, "learned coarse correction: panels differ");
    const int D = tiles[0][0] * C.m[0], H = tiles[0][1] * C.m[1], W = tiles[0][2] * C.m[2];
    if (D % 8 || H % 8 || W % 8)
        return sv->fail(FALCON_ERR_INVALID_ARG, "learned coarse correction: coarse panel grid " + std::to_string(D) + "x" +
                                                    std::to_string(H) + "x" + std::to_string(W) + " is not a multiple of 8");
    const int nint = C.nint();
    std::vector<int32_t> gm((size_t)nb * nint);
    for (int b = 0; b < nb; ++b)
        for (int c = 0; c < nint; ++c) {
            const int i = c % C.m[0], j = (c / C.m[0]) % C.m[1], k = c / (C.m[0] * C.m[1]);
            const int64_t vox = (int64_t)bpan[b] * D * H * W +
                                ((int64_t)(bt[(size_t)b * 3] * C.m[0] + i) * H + bt[(size_t)b * 3 + 1] * C.m[1] + j) * W +
                                bt[(size_t)b * 3 + 2] * C.m[2] + k;
            gm[(size_t)b * nint + c] = (int32_t)vox;
        }
    // every coarse cell lands on its own voxel of the two panel grids
    {
        std::vector<uint8_t> seen((size_t)2 * D * H * W, 0);
        for (int32_t v : gm) {
            if (v < 0 || (size_t)v >= seen.size() || seen[v])
                return sv->fail(FALCON_ERR_INVALID_ARG, "learned coarse correction: block tiling is not a bijection");
            seen[v] = 1;
        }
    }
    SCK(sv->alloc(&sv->gmap, gm.size() * 4), "coarse map");
    SCK(cudaMemcpy(sv->gmap, gm.data(), gm.size() * 4, cudaMemcpyHostToDevice), "coarse map");
    SCK(uploads_arrived(), "coarse map");
    SCK(sv->alloc(&sv->feat, (size_t)2 * D * H * W * 8 * 4), "coarse features");
    SCK(sv->alloc(&sv->yout, (size_t)2 * D * H * W * 4), "coarse features");
    SCK(sv->alloc(&sv->csum, 8), "coarse features");
    SCK(sv->alloc(&sv->cdots, 6 * 8), "coarse features");
    SvLevel& L = sv->lv[lc];
    k_lcc_static<<<grid_cells(L.d, nb), tpb(L.d), 0, sv->st>>>(L.ops64(), L.d, sv->gmap, sv->feat);
    SCK(cudaGetLastError(), "coarse features");
    SCK(cudaStreamSynchronize(sv->st), "coarse features");
    sv->cD = D; sv->cH = H; sv->cW = W;
    sv->cmap_ok = true;
    return FALCON_OK;
}

// e = A_c^{-1} r_c on the coarsest level (r_c: FP32 [b][nint]) by Jacobi-PCG
// to ||r|| <= 1e-6 ||r_c|| (a training target needs no more: the network's
// own error is near 1e-2); the solution stays in sv->x (padded FP64)
int coarse_solve(falcon_solver* sv, const float* rc) {
    const int lc = sv->S.nlevels - 1, nb = sv->S.nblocks;
    SvLevel& L = sv->lv[lc];
    const dim3 g = grid_cells(L.d, nb);
    double* dots = sv->cdots;      // [0..2] current, [3..5] next
    SCK(cudaMemsetAsync(sv->x, 0, (size_t)nb * L.d.npad * 8, sv->st), "coarse cg");
    SCK(cudaMemsetAsync(sv->p, 0, (size_t)nb * L.d.npad * 8, sv->st), "coarse cg");
    SCK(cudaMemsetAsync(dots, 0, 6 * 8, sv->st), "coarse cg");
    k_ccg_init<<<g, tpb(L.d), 0, sv->st>>>(L.ops64(), L.d, rc, sv->r, sv->z, sv->p, dots);
    double h[6];
    SCK(cudaMemcpyAsync(h, dots, 6 * 8, cudaMemcpyDeviceToHost, sv->st), "coarse cg");
    SCK(cudaStreamSynchronize(sv->st), "coarse cg");
    const double rr0 = h[2];
    if (!(rr0 > 0)) return FALCON_OK;
    for (int it = 0; it < 50000; ++it) {
        SCK(halo_fill(sv, lc, sv->p), "coarse cg");
        SCK(cudaMemsetAsync(dots + 1, 0, 8, sv->st), "coarse cg");
        SCK(cudaMemsetAsync(dots + 3, 0, 3 * 8, sv->st), "coarse cg");
        k_ccg_spmv<<<g, tpb(L.d), 0, sv->st>>>(L.ops64(), L.d, sv->p, sv->Ap, dots);
        k_ccg_update<<<g, tpb(L.d), 0, sv->st>>>(L.ops64(), L.d, sv->x, sv->p, sv->r, sv->Ap, sv->z, dots, dots + 3);
        k_ccg_p<<<g, tpb(L.d), 0, sv->st>>>(L.d, sv->p, sv->z, dots, dots + 3);
        SCK(cudaGetLastError(), "coarse cg");
        SCK(cudaMemcpyAsync(dots, dots + 3, 3 * 8, cudaMemcpyDeviceToDevice, sv->st), "coarse cg");
        SCK(cudaMemcpyAsync(h, dots + 3, 3 * 8, cudaMemcpyDeviceToHost, sv->st), "coarse cg");
        SCK(cudaStreamSynchronize(sv->st), "coarse cg");
        if (h[2] <= 1e-12 * rr0) return FALCON_OK;
    }
    return sv->fail(FALCON_ERR_NOT_CONVERGED, "coarse solve did not reach 1e-6");
}

// The operators of every level on the device again, after the level-0
// operator changed on the host (falcon_solver_set_operator): FP64 and FP32
// copies of each level, the scaled float-float level 0 with its new sA, and
// the learned stage's static input channels. Same sizes, same buffers: the
// captured V-cycle graphs stay valid.
int reupload_operators(falcon_solver* sv) {
    const SolverProblemSet& S = sv->S;
    const int nb = S.nblocks;
    SCK(cudaStreamSynchronize(sv->st), "operator");
    for (int l = 0; l < S.nlevels; ++l) {
        const SolverLevel& H = S.L[l];
        SvLevel& L = sv->lv[l];
        const std::vector<double>* src[4] = {&H.Aii, &H.Ai, &H.Aj, &H.Ak};
        double* d64[4] = {L.Aii, L.Ai, L.Aj, L.Ak};
        float* d32[4] = {L.fAii, L.fAi, L.fAj, L.fAk};
        for (int a = 0; a < 4; ++a) {
            const std::vector<double>& h = *src[a];
            std::vector<float> f(h.begin(), h.end());
            SCK(cudaMemcpy(d64[a], h.data(), h.size() * 8, cudaMemcpyHostToDevice), "operator");
            SCK(cudaMemcpy(d32[a], f.data(), f.size() * 4, cudaMemcpyHostToDevice), "operator");
        }
    }
    const SolverLevel& H = S.L[0];
    const size_t nint = (size_t)sv->lv[0].d.nint;
    sv->sA = problem_scale(S, H.Aii, nint);
    SvLevel& L0 = sv->lv[0];
    const std::vector<double>* src[4] = {&H.Aii, &H.Ai, &H.Aj, &H.Ak};
    float2* dff[4] = {L0.Aii2, L0.Ai2, L0.Aj2, L0.Ak2};
    for (int a = 0; a < 4; ++a) {
        const std::vector<double>& h = *src[a];
        const size_t per = h.size() / (size_t)nb;
        std::vector<double> sc(h.size());
        for (int b = 0; b < nb; ++b)
            for (size_t c = 0; c < per; ++c) sc[(size_t)b * per + c] = sv->sA[S.block_problem[b]];
        const std::vector<float2> f = to_ff(h, sc);
        SCK(cudaMemcpy(dff[a], f.data(), f.size() * sizeof(float2), cudaMemcpyHostToDevice), "operator");
    }
    std::vector<float> fa(sv->sA.begin(), sv->sA.end());
    SCK(cudaMemcpy(sv->dsA, fa.data(), fa.size() * 4, cudaMemcpyHostToDevice), "operator");
    SCK(uploads_arrived(), "operator");
    if (sv->cmap_ok) {
        SvLevel& Lc = sv->lv[S.nlevels - 1];
        k_lcc_static<<<grid_cells(Lc.d, nb), tpb(Lc.d), 0, sv->st>>>(Lc.ops64(), Lc.d, sv->gmap, sv->feat);
        SCK(cudaGetLastError(), "coarse features");
    }
    SCK(cudaStreamSynchronize(sv->st), "operator");
    return FALCON_OK;
}

bool all_finite(const double* v, size_t n) {
    for (size_t q = 0; q < n; ++q)
        if (!std::isfinite(v[q])) return false;
    return true;
}

// ---- the inner solve: one FCG iteration, as a graph or eagerly ----------------
// One iteration unit on the stream: z = M r (r without a preconditioner), its ghosts, w = A z with the products that give beta
// (`first`: 0, a restart) and alpha, the update of p, A p, x and r with r.r, and
// the device-side check (k_inner_check), which sets the WHILE condition when
// `set_cond`. Inactive problems take no step. (Forming p first, with its own
// FF halo of eight weighted reads per ghost, took five kernels and 340 us per
// iteration at 6.3M cells in 16^3 blocks; this takes three.)
cudaError_t enqueue_iteration(falcon_solver* sv, int pc, bool first, cudaGraphConditionalHandle h, int set_cond) {
    const int nb = sv->S.nblocks, np = sv->S.nproblems;
    const LevelDims& d = sv->lv[0].d;
    const dim3 g = grid_cells(d, nb);
    cudaError_t e = cudaSuccess;
    if (pc != FALCON_PRECOND_NONE) {
        sv->use_net = pc == FALCON_PRECOND_MG_LCC;
        e = vcycle(sv);
        sv->use_net = false;
        if (e != cudaSuccess) return e;
    }
    auto step = [&](auto z) {
        using Z = decltype(z);
        const unsigned t = std::min(tpb(d), 512u);
        k_ghost_ff<Z><<<(unsigned)((sv->gff.n + 255) / 256), 256, 0, sv->st>>>(sv->gff, z, sv->bprob, sv->ghosts2);
        const auto spmv = d.m0 == 8 ? k_spmv_z_ff<8, Z> : d.m0 == 16 ? k_spmv_z_ff<16, Z> : k_spmv_z_ff<0, Z>;
        spmv<<<g, t, 0, sv->st>>>(sv->lv[0].ops2(), d, z, sv->ghosts2, sv->p2, sv->r2, sv->Ap2, sv->w2, sv->D());
        k_step_ff<Z><<<g, t, 0, sv->st>>>(d, z, sv->w2, sv->x2, sv->p2, sv->r2, sv->Ap2, sv->lv[0].r, sv->D(), first ? 1 : 0);
    };
    if (pc == FALCON_PRECOND_NONE) step(ZFF{sv->r2});
    else step(Z32{sv->lv[0].z, sv->dsA});   // the V-cycle inverts the unscaled FP32 operator
    k_inner_check<<<1, 256, 0, sv->st>>>(np, sv->D(), first ? 1 : 0, sv->rr0, sv->eta, sv->active, sv->ictl, h, set_cond);
    return cudaGetLastError();
}

// The inner solve as one graph: the first iteration, then a WHILE node whose
// body is a continuing iteration; the loop runs on the device until every
// problem reached its eta, the residual stalls, or max_it (k_inner_check).
cudaError_t build_inner_graph(falcon_solver* sv, int pc, cudaGraphExec_t* out) {
    cudaGraph_t g = nullptr;
    cudaError_t e = cudaGraphCreate(&g, 0);
    if (e != cudaSuccess) return e;
    cudaGraphConditionalHandle h;
    e = cudaGraphConditionalHandleCreate(&h, g, 0, 0);
    sv->capturing = true;
    if (e == cudaSuccess) e = cudaStreamBeginCaptureToGraph(sv->st, g, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal);
    if (e == cudaSuccess) {
        const cudaError_t eb = enqueue_iteration(sv, pc, true, h, 1);
        e = cudaStreamEndCapture(sv->st, &g);
        if (eb != cudaSuccess) e = eb;
    }
    // the captured chain's last node is the check; the WHILE node follows it
    std::vector<cudaGraphNode_t> leaves;
    if (e == cudaSuccess) {
        size_t nn = 0, ne = 0;
        e = cudaGraphGetNodes(g, nullptr, &nn);
        std::vector<cudaGraphNode_t> nodes(nn);
        if (e == cudaSuccess) e = cudaGraphGetNodes(g, nodes.data(), &nn);
        if (e == cudaSuccess) e = cudaGraphGetEdges(g, nullptr, nullptr, nullptr, &ne);
        std::vector<cudaGraphNode_t> from(ne), to(ne);
        if (e == cudaSuccess && ne) e = cudaGraphGetEdges(g, from.data(), to.data(), nullptr, &ne);
        for (cudaGraphNode_t n : nodes)
            if (std::find(from.begin(), from.end(), n) == from.end()) leaves.push_back(n);
    }
    if (e == cudaSuccess) {
        cudaGraphNodeParams p = {};
        p.type = cudaGraphNodeTypeConditional;
        p.conditional.handle = h;
        p.conditional.type = cudaGraphCondTypeWhile;
        p.conditional.size = 1;
        cudaGraphNode_t wn;
        e = cudaGraphAddNode(&wn, g, leaves.data(), nullptr, leaves.size(), &p);
        if (e == cudaSuccess) {
            cudaGraph_t body = p.conditional.phGraph_out[0];
            e = cudaStreamBeginCaptureToGraph(sv->st, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal);
            if (e == cudaSuccess) {
                const cudaError_t eb = enqueue_iteration(sv, pc, false, h, 1);
                e = cudaStreamEndCapture(sv->st, &body);
                if (eb != cudaSuccess) e = eb;
            }
        }
    }
    sv->capturing = false;
    if (e == cudaSuccess) e = cudaGraphInstantiate(out, g, 0);
    if (g) cudaGraphDestroy(g);
    return e;
}

// One inner solve from the current r2 (x2 = 0): the graph when the solve is
// not recording coarse residuals, else the same iterations eagerly with the
// host reading the loop control after each. Fills ctl (host copy).
cudaError_t run_inner(falcon_solver* sv, int pc, int max_it, InnerCtl* ctl) {
    InnerCtl c0;
    std::memset(&c0, 0, sizeof c0);
    c0.max_it = std::max(1, std::min(max_it, kInnerCap));
    cudaError_t e = cudaMemcpyAsync(sv->ictl, &c0, sizeof c0, cudaMemcpyHostToDevice, sv->st);
    if (e != cudaSuccess) return e;
    if (!sv->rec) {
        const int64_t key = (int64_t)pc | ((int64_t)sv->nu_pre << 4) | ((int64_t)sv->nu_post << 12) |
                            ((int64_t)sv->nu_coarse << 20) | ((int64_t)sv->net_sweeps << 34);
        auto it = sv->igraphs.find(key);
        if (it == sv->igraphs.end()) {
            cudaGraphExec_t x = nullptr;
            e = build_inner_graph(sv, pc, &x);
            if (e != cudaSuccess) return e;
            it = sv->igraphs.emplace(key, x).first;
        }
        e = cudaGraphLaunch(it->second, sv->st);
        if (e == cudaSuccess) e = cudaMemcpyAsync(ctl, sv->ictl, sizeof *ctl, cudaMemcpyDeviceToHost, sv->st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(sv->st);
        return e;
    }
    for (bool first = true;; first = false) {
        e = enqueue_iteration(sv, pc, first, 0, 0);
        if (e == cudaSuccess) e = cudaMemcpyAsync(ctl, sv->ictl, sizeof *ctl, cudaMemcpyDeviceToHost, sv->st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(sv->st);
        if (e != cudaSuccess || !ctl->cont) return e;
    }
}

// The solver's autotuner: times two eager FCG iterations for each candidate tile of the
// cell kernels -- cells per CTA in {512, 1024, 2048, 4096}, whole rows, x threads per
// CTA in {128, 256, 512} -- on this solver's own grid, and keeps the fastest. What
// differs between candidates is the operator and the update; the V-cycle, which does
// not use the tile, brings the vectors through the caches between them as in a solve.
// Runs once, at the first solve, on scratch vectors that the solve initialises
// afterwards.
int autotune_tile(falcon_solver* sv) {
    if (sv->tuned) return FALCON_OK;
    const int np = sv->S.nproblems;
    const int m0 = sv->lv[0].d.m0;
    std::vector<int32_t> act(np, 1);
    std::vector<double> ones(np, 1.0), never(np, -1.0);   // no residual is at or below eta: every problem stays active
    SCK(cudaMemcpyAsync(sv->active, act.data(), np * 4, cudaMemcpyHostToDevice, sv->st), "tune");
    SCK(cudaMemcpyAsync(sv->rr0, ones.data(), np * 8, cudaMemcpyHostToDevice, sv->st), "tune");
    SCK(cudaMemcpyAsync(sv->eta, never.data(), np * 8, cudaMemcpyHostToDevice, sv->st), "tune");
    SCK(cudaMemsetAsync(sv->dots, 0, (size_t)8 * np * 8, sv->st), "tune");
    SCK(cudaStreamSynchronize(sv->st), "tune");
    const int pc = sv->S.nlevels > 1 ? FALCON_PRECOND_MG : FALCON_PRECOND_NONE;
    cudaEvent_t a, b;
    cudaEventCreate(&a);
    cudaEventCreate(&b);
    float best = 1e30f;
    int bc = sv->tile_chunk, bt = sv->tile_tpb;
    for (int chunk : {512, 1024, 2048, 4096}) {
        if (chunk % m0) continue;
        for (int t : {128, 256, 512}) {
            apply_tile(sv, chunk, t);
            InnerCtl c0;
            std::memset(&c0, 0, sizeof c0);
            c0.max_it = kInnerCap;
            SCK(cudaMemcpyAsync(sv->ictl, &c0, sizeof c0, cudaMemcpyHostToDevice, sv->st), "tune");
            SCK(enqueue_iteration(sv, pc, false, 0, 0), "tune");   // warm-up
            cudaEventRecord(a, sv->st);
            for (int r = 0; r < 2; ++r) SCK(enqueue_iteration(sv, pc, false, 0, 0), "tune");
            cudaEventRecord(b, sv->st);
            SCK(cudaEventSynchronize(b), "tune");
            float ms = 0;
            cudaEventElapsedTime(&ms, a, b);
            if (ms < best) { best = ms; bc = chunk; bt = t; }
        }
    }
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    apply_tile(sv, bc, bt);
    sv->tuned = true;
    sv->tuned_ms = best / 2.0;
    return FALCON_OK;
}

}  // namespace

extern "C" {

int falcon_solver_set_operator(falcon_solver* sv, const double* Aii, const double* Ai, const double* Aj, const double* Ak) {
    if (!sv || !Aii || !Ai || !Aj || !Ak) return FALCON_ERR_INVALID_ARG;
    SolverProblemSet& S = sv->S;
    SolverLevel& L = S.L[0];
    const double* in[4] = {Aii, Ai, Aj, Ak};
    std::vector<double>* dst[4] = {&L.Aii, &L.Ai, &L.Aj, &L.Ak};
    for (int a = 0; a < 4; ++a)
        if (!all_finite(in[a], dst[a]->size())) return sv->fail(FALCON_ERR_INVALID_ARG, "falcon_solver_set_operator: non-finite coefficient");
    for (size_t q = 0; q < L.Aii.size(); ++q)
        if (!(Aii[q] > 0.0)) return sv->fail(FALCON_ERR_INVALID_ARG, "falcon_solver_set_operator: the diagonal Aii must be positive");
    for (int a = 0; a < 4; ++a) std::memcpy(dst[a]->data(), in[a], dst[a]->size() * 8);
    galerkin_coarsen(S);
    if (!sv->st) return FALCON_OK;
    cudaSetDevice(sv->device);
    return reupload_operators(sv);
}

int falcon_solver_set_magnetogram(falcon_solver* sv, const double* br) {
    if (!sv || !br) return FALCON_ERR_INVALID_ARG;
    SolverProblemSet& S = sv->S;
    if (S.br.empty()) return sv->fail(FALCON_ERR_INVALID_ARG, "falcon_solver_set_magnetogram: not a PFSS solver");
    if (!all_finite(br, S.br.size())) return sv->fail(FALCON_ERR_INVALID_ARG, "falcon_solver_set_magnetogram: non-finite Br");
    std::vector<double> b(br, br + S.br.size());
    for (int gb = 0; gb < S.nblocks; ++gb)   // only bottom blocks carry a magnetogram
        if (!(S.block_flags[gb] & 4)) std::fill(b.begin() + (size_t)gb * (S.br.size() / S.nblocks),
                                                b.begin() + (size_t)(gb + 1) * (S.br.size() / S.nblocks), 0.0);
    pfss_rhs(S, b);
    if (!sv->st) return FALCON_OK;
    cudaSetDevice(sv->device);
    SCK(cudaStreamSynchronize(sv->st), "rhs");
    SCK(cudaMemcpy(sv->bvec, S.b.data(), S.b.size() * 8, cudaMemcpyHostToDevice), "rhs");
    SCK(uploads_arrived(), "rhs");
    return FALCON_OK;
}

int falcon_solver_magnetogram(const falcon_solver* sv, double* br) {
    if (!sv || !br) return FALCON_ERR_INVALID_ARG;
    if (sv->S.br.empty()) return FALCON_ERR_INVALID_ARG;
    std::memcpy(br, sv->S.br.data(), sv->S.br.size() * 8);
    return FALCON_OK;
}

int falcon_solver_vcycle_op(falcon_solver* sv, int32_t op, int32_t level, const float* in0, const float* in1,
                            float* out) {
    if (!sv || !in0 || !out) return FALCON_ERR_INVALID_ARG;
    if (!sv->st) return sv->fail(FALCON_ERR_NO_DEVICE, "solver created without a device");
    const int nl = sv->S.nlevels, nb = sv->S.nblocks;
    const bool needs_coarse = op == FALCON_VCYCLE_RESTRICT || op == FALCON_VCYCLE_PROLONG_ADD ||
                              op == FALCON_VCYCLE_RESIDUAL_RESTRICT || op == FALCON_VCYCLE_PROLONG_SWEEP;
    const bool only_in0 = op == FALCON_VCYCLE_RESTRICT || op == FALCON_VCYCLE_FIRST_SWEEP || op == FALCON_VCYCLE_COARSE_SWEEPS;
    if (op < FALCON_VCYCLE_RESTRICT || op > FALCON_VCYCLE_COARSE_SWEEPS || level < 0 || level >= nl ||
        (needs_coarse && level + 1 >= nl) || (!only_in0 && !in1) ||
        (op == FALCON_VCYCLE_COARSE_SWEEPS && (level == 0 || level != nl - 1 || sv->nu_coarse < 1)))
        return sv->fail(FALCON_ERR_INVALID_ARG, "falcon_solver_vcycle_op: bad operation, level or input");
    cudaSetDevice(sv->device);
    SvLevel& L = sv->lv[level];
    const size_t nf = (size_t)nb * L.d.nint * 4;
    SCK(cudaStreamSynchronize(sv->st), "vcycle op");
    if (op == FALCON_VCYCLE_RESTRICT) {   // the residual of r = in0 at z = 0, restricted
        SvLevel& Cl = sv->lv[level + 1];
        SCK(cudaMemcpyAsync(L.r, in0, nf, cudaMemcpyHostToDevice, sv->st), "vcycle op");
        SCK(cudaMemsetAsync(L.z, 0, nf, sv->st), "vcycle op");
        SCK(vresid_restrict(sv, level, L.z, Cl.r), "vcycle op");
        SCK(cudaMemcpyAsync(out, Cl.r, (size_t)nb * Cl.d.nint * 4, cudaMemcpyDeviceToHost, sv->st), "vcycle op");
    } else if (op == FALCON_VCYCLE_PROLONG_ADD) {
        SvLevel& Cl = sv->lv[level + 1];
        SCK(cudaMemcpyAsync(Cl.z, in0, (size_t)nb * Cl.d.nint * 4, cudaMemcpyHostToDevice, sv->st), "vcycle op");
        SCK(cudaMemcpyAsync(L.z, in1, nf, cudaMemcpyHostToDevice, sv->st), "vcycle op");
        SCK(vsweep<V_PROLONG>(sv, level, L.z, Cl.z, L.zb, -1), "vcycle op");
        SCK(cudaMemcpyAsync(out, L.zb, nf, cudaMemcpyDeviceToHost, sv->st), "vcycle op");
    } else if (op == FALCON_VCYCLE_RESIDUAL_RESTRICT) {
        SvLevel& Cl = sv->lv[level + 1];
        SCK(cudaMemcpyAsync(L.r, in0, nf, cudaMemcpyHostToDevice, sv->st), "vcycle op");
        SCK(cudaMemcpyAsync(L.z, in1, nf, cudaMemcpyHostToDevice, sv->st), "vcycle op");
        SCK(vresid_restrict(sv, level, L.z, Cl.r), "vcycle op");
        SCK(cudaMemcpyAsync(out, Cl.r, (size_t)nb * Cl.d.nint * 4, cudaMemcpyDeviceToHost, sv->st), "vcycle op");
    } else if (op == FALCON_VCYCLE_PROLONG_SWEEP) {
        SvLevel& Cl = sv->lv[level + 1];
        SCK(cudaMemcpyAsync(Cl.z, in0, (size_t)nb * Cl.d.nint * 4, cudaMemcpyHostToDevice, sv->st), "vcycle op");
        SCK(cudaMemcpyAsync(L.r, in1, nf, cudaMemcpyHostToDevice, sv->st), "vcycle op");
        SCK(cudaMemcpyAsync(L.z, in1 + nf / 4, nf, cudaMemcpyHostToDevice, sv->st), "vcycle op");
        SCK(vsweep<V_PROLONG>(sv, level, L.z, Cl.z, L.zb, 1), "vcycle op");
        SCK(cudaMemcpyAsync(out, L.zb, nf, cudaMemcpyDeviceToHost, sv->st), "vcycle op");
    } else if (op == FALCON_VCYCLE_FIRST_SWEEP || op == FALCON_VCYCLE_COARSE_SWEEPS) {
        SCK(cudaMemcpyAsync(L.r, in0, nf, cudaMemcpyHostToDevice, sv->st), "vcycle op");
        float* z = L.z;
        SCK(smooth_from_zero(sv, level, op == FALCON_VCYCLE_FIRST_SWEEP ? 1 : sv->nu_coarse, L.z, [&] {
                z = z == L.z ? L.zb : L.z;
                return z;
            }), "vcycle op");
        SCK(cudaMemcpyAsync(out, z, nf, cudaMemcpyDeviceToHost, sv->st), "vcycle op");
    } else {   // one red-black half sweep of a colour from z = in1, or the residual r - A z
        SCK(cudaMemcpyAsync(L.r, in0, nf, cudaMemcpyHostToDevice, sv->st), "vcycle op");
        SCK(cudaMemcpyAsync(L.z, in1, nf, cudaMemcpyHostToDevice, sv->st), "vcycle op");
        if (op == FALCON_VCYCLE_RESIDUAL) SCK(vresid(sv, level, L.z, L.res), "vcycle op");
        else SCK(vsweep<V_PLAIN>(sv, level, L.z, nullptr, L.zb, op == FALCON_VCYCLE_SMOOTH_RED ? 0 : 1), "vcycle op");
        SCK(cudaMemcpyAsync(out, op == FALCON_VCYCLE_RESIDUAL ? L.res : L.zb, nf, cudaMemcpyDeviceToHost, sv->st), "vcycle op");
    }
    SCK(cudaStreamSynchronize(sv->st), "vcycle op");
    return FALCON_OK;
}

int falcon_solver_tuning(const falcon_solver* sv, int32_t* tile, double* ms_per_iteration) {
    if (!sv || !tile) return FALCON_ERR_INVALID_ARG;
    tile[0] = sv->tile_chunk;
    tile[1] = sv->tile_tpb;
    tile[2] = sv->tuned ? 1 : 0;
    if (ms_per_iteration) *ms_per_iteration = sv->tuned_ms;
    return FALCON_OK;
}

int falcon_solver_coarse_form(const falcon_solver* sv, int32_t* form) {
    if (!sv || !form) return FALCON_ERR_INVALID_ARG;
    form[0] = sv->coarse_cluster;
    form[1] = sv->coarse_cluster ? sv->coarse_r : 0;
    form[2] = sv->coarse_cluster ? sv->coarse_slots : 0;
    return FALCON_OK;
}

int falcon_solver_set_tile(falcon_solver* sv, int32_t cells_per_cta, int32_t threads_per_cta) {
    if (!sv) return FALCON_ERR_INVALID_ARG;
    if (cells_per_cta < 32 || cells_per_cta > (1 << 16) || (cells_per_cta & 31) || threads_per_cta < 32 ||
        threads_per_cta > 1024 || (threads_per_cta & 31))
        return sv->fail(FALCON_ERR_INVALID_ARG,
                        "falcon_solver_set_tile: cells per CTA in [32, 65536] and threads per CTA in [32, 1024], "
                        "both multiples of 32");
    if (sv->st) {
        cudaSetDevice(sv->device);
        SCK(cudaStreamSynchronize(sv->st), "tile");
    }
    apply_tile(sv, cells_per_cta, threads_per_cta);
    sv->tuned = true;   // the caller's shape: no autotuning
    sv->tuned_ms = 0;
    return FALCON_OK;
}

int falcon_solver_block_ranges(const falcon_solver* sv, double* ranges) {
    if (!sv || !ranges) return FALCON_ERR_INVALID_ARG;
    const SolverProblemSet& S = sv->S;
    for (int gb = 0; gb < S.nblocks; ++gb) {
        const int p = S.block_problem[gb];
        const int b = gb - S.problem_first_block[p];
        std::memcpy(ranges + (size_t)gb * 6, &S.grids[p].ranges[(size_t)b * 6], 6 * sizeof(double));
    }
    return FALCON_OK;
}

int falcon_solver_block_flags(const falcon_solver* sv, int32_t* flags) {
    if (!sv || !flags) return FALCON_ERR_INVALID_ARG;
    std::memcpy(flags, sv->S.block_flags.data(), sv->S.block_flags.size() * sizeof(int32_t));
    return FALCON_OK;
}

int falcon_solver_magnetogram_sources(const falcon_solver* sv, int32_t problem, double* xyzq, int32_t cap,
                                      int32_t* n) {
    if (!sv || !n || problem < 0 || problem >= sv->S.nproblems) return FALCON_ERR_INVALID_ARG;
    if (sv->S.br.empty()) return FALCON_ERR_INVALID_ARG;
    Magnetogram M;
    M.init(sv->seed + (uint64_t)problem, sv->r_surface);
    *n = (int32_t)M.q.size();
    if (!xyzq) return FALCON_OK;
    if (cap < *n) return FALCON_ERR_BOUNDS;
    for (size_t c = 0; c < M.q.size(); ++c) {
        xyzq[4 * c] = M.px[c];
        xyzq[4 * c + 1] = M.py[c];
        xyzq[4 * c + 2] = M.pz[c];
        xyzq[4 * c + 3] = M.q[c];
    }
    return FALCON_OK;
}

int falcon_solver_set_guess(falcon_solver* sv, const double* x0) {
    if (!sv || !x0) return FALCON_ERR_INVALID_ARG;
    if (!all_finite(x0, sv->S.x0.size())) return sv->fail(FALCON_ERR_INVALID_ARG, "falcon_solver_set_guess: non-finite value");
    std::memcpy(sv->S.x0.data(), x0, sv->S.x0.size() * 8);
    return FALCON_OK;
}

int falcon_solver_create(falcon_solver** out, const falcon_solver_spec* spec) {
    if (!out || !spec) return FALCON_ERR_INVALID_ARG;
    falcon_solver* sv = new falcon_solver();
    *out = sv;
    if (spec->nproblems < 1 || spec->nproblems > FALCON_MAX_PROBLEMS) return sv->fail(FALCON_ERR_INVALID_ARG, "nproblems out of range");
    if (spec->block < 2 || spec->block > 32 || (spec->block & 1)) return sv->fail(FALCON_ERR_INVALID_ARG, "block must be even, 2..32");
    sv->device = spec->device;
    sv->seed = spec->seed;
    if (spec->kind == FALCON_SOLVER_CONDUCTION) {
        sv->nu_coarse = 4;
    } else {   // PFSS: one sweep each way, 32 on the coarsest level (measured fastest to 1e-10)
        sv->nu_pre = sv->nu_post = 1;
        sv->nu_coarse = 32;
    }
    std::vector<falcon_config> cfgs(spec->nproblems);
    const double kRsun = (double)6.955e10f;
    for (int q = 0; q < spec->nproblems; ++q) {
        falcon_config& c = cfgs[q];
        std::memset(&c, 0, sizeof c);
        falcon_tree_spec& t = c.tree;
        t.ni = t.nj = t.nk = spec->block;
        t.ng = 2;
        const int B = spec->block;
        if (spec->kind == FALCON_SOLVER_PFSS) {
            // (nr, ntheta) -> per panel (nr, ntheta/2, 3 ntheta/2) rounded up to whole blocks
            const int Nr = (spec->nr[q] + B - 1) / B;
            const int Nt = (spec->nt[q] / 2 + B - 1) / B;
            t.root_tiles[0] = Nr; t.root_tiles[1] = Nt; t.root_tiles[2] = 3 * Nt;
            t.radial_levels = 0; t.radial_option = 2; t.n_amr = 0;
        } else {
            // conduction: per panel nr x nt x np cells, uniform radial blocks
            const int Nr = spec->nr[q] / B, Nt = spec->nt[q] / B, Np = spec->np[q] / B;
            if (Nr * B != spec->nr[q] || Nt * B != spec->nt[q] || Np * B != spec->np[q] || Np != 3 * Nt)
                return sv->fail(FALCON_ERR_INVALID_ARG, "conduction grid must be whole blocks with np = 3 nt");
            t.root_tiles[0] = Nr; t.root_tiles[1] = Nt; t.root_tiles[2] = Np;
            t.radial_option = 2;
        }
        t.r_range_rsun[0] = spec->r_range_rsun[0];
        t.r_range_rsun[1] = spec->r_range_rsun[1];
        c.phys.cfl = 0.4;
        c.bg.poly_n = 1.5; c.bg.density_contrast = 100.0; c.bg.mu = 0.6; c.bg.xi_mode = 1;
        c.device = spec->device;
    }
    std::string e = build_solver_levels(sv->S, cfgs, spec->nlevels);
    if (!e.empty()) return sv->fail(FALCON_ERR_INVALID_ARG, e);
    SolverProblemSet& S = sv->S;
    if (spec->kind == FALCON_SOLVER_PFSS) {
        // magnetogram Br at the bottom face centres of bottom blocks (Yin frame)
        const SolverLevel& L = S.L[0];
        const int mj = L.m[1], mk = L.m[2];
        std::vector<double> br((size_t)S.nblocks * mj * mk, 0.0);
        for (int q = 0; q < S.nproblems; ++q) {
            Magnetogram M;
            sv->r_surface = spec->r_range_rsun[0] * kRsun;
            M.init(spec->seed + (uint64_t)q, sv->r_surface);
            for (int gb = S.problem_first_block[q]; gb < S.problem_first_block[q + 1]; ++gb) {
                if (!(S.block_flags[gb] & 4)) continue;
                const bool yin = S.block_flags[gb] & 1;
                const Grid& g = S.grids[q];
                const int b = gb - S.problem_first_block[q];
                const double r0 = g.ranges[(size_t)b * 6 + 0];
                for (int k = 1; k <= mk; ++k)
                    for (int j = 1; j <= mj; ++j) {
                        double t = L.xj[(size_t)gb * (mj + 2) + j], ph = L.xk[(size_t)gb * (mk + 2) + k];
                        if (!yin) {
                            const double a[3] = {r0, t, ph};
                            const double st_ = std::sin(a[1]), ct = std::cos(a[1]), sp = std::sin(a[2]), cp = std::cos(a[2]);
                            t = std::acos(st_ * sp);
                            ph = std::copysign(std::fabs(std::acos(-(st_ * cp) / std::sqrt(st_ * st_ * (cp * cp) + ct * ct))), ct);
                        }
                        br[((size_t)gb * mk + (k - 1)) * mj + (j - 1)] = M.br(r0, t, ph);
                    }
            }
        }
        assemble_pfss(S, br);
    } else {
        ConductionField F;
        F.init(&S.grids[0].bg, spec->seed, S.grids[0].r_range[0]);
        assemble_conduction(S, F, spec->dt_factor > 0 ? spec->dt_factor : 50.0, &sv->dt_conduction);
    }
    galerkin_coarsen(S);
    if (spec->device < 0) return FALCON_OK;
    return setup(sv);
}

void falcon_solver_destroy(falcon_solver* sv) {
    if (!sv) return;
    if (sv->st) {
        cudaSetDevice(sv->device);
        cudaStreamSynchronize(sv->st);
        sv->clear_graphs();
        for (void* q : sv->allocs) cudaFree(q);
        cudaStreamDestroy(sv->st);
    }
    delete sv;
}

int falcon_solver_last_error(const falcon_solver* sv, char* buf, size_t len) {
    if (!sv || !buf || !len) return FALCON_ERR_INVALID_ARG;
    snprintf(buf, len, "%s", sv->err.c_str());
    return FALCON_OK;
}

int falcon_solver_info(const falcon_solver* sv, int32_t* info) {
    if (!sv || !info) return FALCON_ERR_INVALID_ARG;
    info[0] = sv->S.nblocks;
    info[1] = sv->S.nproblems;
    info[2] = sv->S.nlevels;
    for (int d = 0; d < 3; ++d) info[3 + d] = sv->S.nlevels ? sv->S.L[0].m[d] : 0;
    return FALCON_OK;
}

int falcon_solver_problem_blocks(const falcon_solver* sv, int32_t* first) {
    if (!sv || !first) return FALCON_ERR_INVALID_ARG;
    std::memcpy(first, sv->S.problem_first_block.data(), sv->S.problem_first_block.size() * 4);
    return FALCON_OK;
}

int falcon_solver_rhs(const falcon_solver* sv, double* b) {
    if (!sv || !b) return FALCON_ERR_INVALID_ARG;
    std::memcpy(b, sv->S.b.data(), sv->S.b.size() * 8);
    return FALCON_OK;
}

int falcon_solver_operator(const falcon_solver* sv, int32_t level, double* Aii, double* Ai, double* Aj, double* Ak) {
    if (!sv || level < 0 || level >= sv->S.nlevels) return FALCON_ERR_INVALID_ARG;
    const SolverLevel& L = sv->S.L[level];
    if (Aii) std::memcpy(Aii, L.Aii.data(), L.Aii.size() * 8);
    if (Ai) std::memcpy(Ai, L.Ai.data(), L.Ai.size() * 8);
    if (Aj) std::memcpy(Aj, L.Aj.data(), L.Aj.size() * 8);
    if (Ak) std::memcpy(Ak, L.Ak.data(), L.Ak.size() * 8);
    return FALCON_OK;
}

int falcon_solver_halo_count(const falcon_solver* sv, int32_t level, int64_t* n) {
    if (!sv || !n || level < 0 || level >= sv->S.nlevels) return FALCON_ERR_INVALID_ARG;
    *n = (int64_t)sv->S.L[level].halo.size();
    return FALCON_OK;
}

// entries: [n][8] int32 (tb,ti,tj,tk,sb,i0,j0,k0) and [n][6] double (w, src_x)
int falcon_solver_halo_map(const falcon_solver* sv, int32_t level, int32_t* idx, double* wx) {
    if (!sv || level < 0 || level >= sv->S.nlevels) return FALCON_ERR_INVALID_ARG;
    const auto& H = sv->S.L[level].halo;
    for (size_t q = 0; q < H.size(); ++q) {
        const HaloEntry& h = H[q];
        const int32_t v[8] = {h.tb, h.ti, h.tj, h.tk, h.sb, h.i0, h.j0, h.k0};
        std::memcpy(idx + 8 * q, v, sizeof v);
        for (int d = 0; d < 3; ++d) { wx[6 * q + d] = h.w[d]; wx[6 * q + 3 + d] = h.src_x[d]; }
    }
    return FALCON_OK;
}

// y = A x at level 0 on the GPU (x interior [b][nint]; halo filled on the device)
int falcon_solver_apply(falcon_solver* sv, const double* x, double* y) {
    if (!sv || !x || !y) return FALCON_ERR_INVALID_ARG;
    if (!sv->st) return sv->fail(FALCON_ERR_NO_DEVICE, "solver created without a device");
    cudaSetDevice(sv->device);
    const LevelDims& d = sv->lv[0].d;
    const int nb = sv->S.nblocks;
    SCK(cudaMemcpyAsync(sv->z, x, (size_t)nb * d.nint * 8, cudaMemcpyHostToDevice, sv->st), "apply");
    SCK(cudaMemsetAsync(sv->p, 0, (size_t)nb * d.npad * 8, sv->st), "apply");
    k_scatter_pad<double><<<grid_cells(d, nb), tpb(d), 0, sv->st>>>(d, sv->z, sv->p);
    SCK(halo_fill(sv, 0, sv->p), "apply halo");
    k_spmv<<<grid_cells(d, nb), tpb(d), 0, sv->st>>>(sv->lv[0].ops64(), d, sv->p, sv->Ap);
    SCK(cudaGetLastError(), "apply");
    SCK(cudaMemcpyAsync(y, sv->Ap, (size_t)nb * d.nint * 8, cudaMemcpyDeviceToHost, sv->st), "apply");
    SCK(cudaStreamSynchronize(sv->st), "apply");
    return FALCON_OK;
}

int falcon_solver_solve(falcon_solver* sv, double tol, int32_t max_iter, int32_t precond, falcon_solve_report* rep) {
    if (!sv || !rep) return FALCON_ERR_INVALID_ARG;
    if (!sv->st) return sv->fail(FALCON_ERR_NO_DEVICE, "solver created without a device");
    if (precond != FALCON_PRECOND_NONE && precond != FALCON_PRECOND_MG && precond != FALCON_PRECOND_MG_LCC)
        return sv->fail(FALCON_ERR_INVALID_ARG, "unknown preconditioner");
    if (precond == FALCON_PRECOND_MG_LCC && (!sv->net || !sv->cmap_ok))
        return sv->fail(FALCON_ERR_INVALID_ARG, "FALCON_PRECOND_MG_LCC needs falcon_solver_attach_lcc first");
    if (!(tol > 0.0) || max_iter < 0) return sv->fail(FALCON_ERR_INVALID_ARG, "tol must be positive and max_iter >= 0");
    cudaSetDevice(sv->device);
    const SolverProblemSet& S = sv->S;
    const int nb = S.nblocks, np = S.nproblems;
    const LevelDims& d = sv->lv[0].d;
    std::memset(rep, 0, sizeof *rep);
    // Structure (ModLinearSolver_Multigrid_CG, 3_5/ModLinearSolver.f90:313-427,
    // made an FP64 iterative refinement):
    //   outer, FP64: r = b - A x with FP64 dots; a problem is done when
    //     ||r||/||b|| <= tol -- the only convergence test;
    //   inner, float-float FCG + FP32 V-cycle: A' d' = r' on the correction
    //     equation scaled per problem (A' = A / sA, r' = r / sr), to a relative
    //     recursive residual of 0.5 tol ||b|| / ||r|| (at least 2^-40);
    //   x += d' sr / sA in FP64.
    // A problem whose FP64 residual is at the attainable accuracy of b - A x
    // (4 x 8 eps64 (|b| + |A||x|) / ||b||) or that a refinement no longer
    // halves stops unconverged; its residual is reported as floor_residual.
    constexpr double kEps64 = 1.1102230246251565e-16;   // 2^-53
    constexpr double kEtaMin = 9.094947017729282e-13;   // 2^-40: float-float recursive residual limit
    constexpr int kMaxPasses = 30;
    {
        float* rec = sv->rec;   // the tuning iterations record nothing
        sv->rec = nullptr;
        const int rc = autotune_tile(sv);
        sv->rec = rec;
        if (rc) return rc;
    }
    // the launch grid of the tuned tile (the autotuner may just have changed it)
    const dim3 g = grid_cells(d, nb);
    cudaEvent_t t0, t1;
    cudaEventCreate(&t0);
    cudaEventCreate(&t1);
    // x = x0 (FP64, padded; ghost cells 0 until the halo fill)
    SCK(cudaMemcpyAsync(sv->z, S.x0.data(), S.x0.size() * 8, cudaMemcpyHostToDevice, sv->st), "init");
    SCK(cudaMemsetAsync(sv->x, 0, (size_t)nb * d.npad * 8, sv->st), "init");
    SCK(cudaStreamSynchronize(sv->st), "init");
    cudaEventRecord(t0, sv->st);
    k_scatter_pad<double><<<g, tpb(d), 0, sv->st>>>(d, sv->z, sv->x);
    SCK(cudaGetLastError(), "init");
    // per problem: 0 being solved, 1 converged (FP64 residual <= tol), 2 stopped at its floor
    std::vector<int> state(np, 0);
    std::vector<int32_t> act(np, 0);
    std::vector<double> rr(np), bb(np), ab(np), rel(np, 0.0), prev(np, 0.0), rr0(np), eta(np);
    std::vector<double> inv_sr(np, 1.0), fac(np, 1.0);
    int pc = precond;   // FALCON_PRECOND_MG_LCC falls back to FALCON_PRECOND_MG on stagnation
    int it = 0, passes = 0;
    for (bool first = true;; first = false) {
        // FP64 true residual of every problem
        SCK(cudaMemsetAsync(sv->dots + 3 * np, 0, (size_t)(first ? 3 : 1) * np * 8, sv->st), "dots");
        SCK(cudaMemsetAsync(sv->dots + 5 * np, 0, (size_t)np * 8, sv->st), "dots");
        SCK(halo_fill(sv, 0, sv->x), "halo");
        k_residual64<<<g, tpb(d), 0, sv->st>>>(sv->lv[0].ops64(), d, sv->x, sv->bvec, sv->r, sv->lv[0].r, sv->D(),
                                               first ? 1 : 0);
        SCK(cudaGetLastError(), "residual");
        SCK(cudaMemcpyAsync(rr.data(), sv->dots + 3 * np, np * 8, cudaMemcpyDeviceToHost, sv->st), "rr");
        SCK(cudaMemcpyAsync(ab.data(), sv->dots + 5 * np, np * 8, cudaMemcpyDeviceToHost, sv->st), "rr");
        if (first) SCK(cudaMemcpyAsync(bb.data(), sv->dots + 4 * np, np * 8, cudaMemcpyDeviceToHost, sv->st), "bb");
        SCK(cudaStreamSynchronize(sv->st), "rr");
        if (first)
            for (int q = 0; q < np; ++q) if (!(bb[q] > 0)) bb[q] = 1.0;   // b = 0: absolute residual
        bool any = false;
        for (int q = 0; q < np; ++q) {
            if (state[q] != 0) continue;
            const double r_q = std::sqrt(rr[q] / bb[q]);
            if (!std::isfinite(r_q))
                return sv->fail(FALCON_ERR_NAN_DETECTED, "solver: non-finite FP64 residual in problem " + std::to_string(q));
            const double floor_q = 4.0 * 8.0 * kEps64 * std::sqrt(ab[q] / bb[q]);
            rel[q] = r_q;
            if (r_q <= tol) {
                state[q] = 1;
            } else if (r_q <= floor_q || (!first && r_q > 0.5 * prev[q])) {
                state[q] = 2;
                rep->floor_residual = std::max(rep->floor_residual, r_q);
            } else {
                any = true;
            }
            prev[q] = r_q;
        }
        if (!any || it >= max_iter || passes >= kMaxPasses) break;
        // inner solve of A' d' = r' for the problems still being solved
        ++passes;
        for (int q = 0; q < np; ++q) {
            act[q] = state[q] == 0;
            int e2 = 0;
            std::frexp(std::sqrt(rr[q]), &e2);
            const double sr = act[q] && rr[q] > 0 ? std::ldexp(1.0, e2) : 1.0;
            inv_sr[q] = 1.0 / sr;
            fac[q] = sr / sv->sA[q];
            eta[q] = std::max(0.5 * tol / std::max(rel[q], tol), kEtaMin);
        }
        SCK(cudaMemcpyAsync(sv->active, act.data(), np * 4, cudaMemcpyHostToDevice, sv->st), "active");
        SCK(cudaMemcpyAsync(sv->ir_par, inv_sr.data(), np * 8, cudaMemcpyHostToDevice, sv->st), "scale");
        SCK(cudaMemcpyAsync(sv->ir_par + np, fac.data(), np * 8, cudaMemcpyHostToDevice, sv->st), "scale");
        for (float2* v : {sv->x2, sv->p2, sv->Ap2})
            SCK(cudaMemsetAsync(v, 0, (size_t)nb * d.nint * sizeof(float2), sv->st), "init");
        SCK(cudaMemsetAsync(sv->dots, 0, (size_t)8 * np * 8, sv->st), "dots");
        k_ir_start<<<g, tpb(d), 0, sv->st>>>(d, sv->r, sv->ir_par, sv->r2, sv->lv[0].r, sv->D());
        SCK(cudaGetLastError(), "inner start");
        SCK(cudaMemcpyAsync(rr0.data(), sv->dots + 3 * np, np * 8, cudaMemcpyDeviceToHost, sv->st), "rr");
        SCK(cudaMemsetAsync(sv->dots + 3 * np, 0, (size_t)np * 8, sv->st), "dots");
        SCK(cudaStreamSynchronize(sv->st), "rr");
        for (int q = 0; q < np; ++q) if (!(rr0[q] > 0)) { rr0[q] = 1.0; act[q] = 0; }
        SCK(cudaMemcpyAsync(sv->active, act.data(), np * 4, cudaMemcpyHostToDevice, sv->st), "active");
        SCK(cudaMemcpyAsync(sv->rr0, rr0.data(), np * 8, cudaMemcpyHostToDevice, sv->st), "inner start");
        SCK(cudaMemcpyAsync(sv->eta, eta.data(), np * 8, cudaMemcpyHostToDevice, sv->st), "inner start");
        // the inner FCG: one graph launch, its loop controlled on the device
        for (;;) {
            InnerCtl ctl;
            SCK(run_inner(sv, pc, max_iter - it, &ctl), "inner solve");
            it += ctl.it;
            if (pc != FALCON_PRECOND_NONE) rep->vcycles += ctl.it;
            if (ctl.nan) return sv->fail(FALCON_ERR_NAN_DETECTED, "solver: non-finite residual in the inner solve");
            if (ctl.stalled && pc == FALCON_PRECOND_MG_LCC && it < max_iter) {
                // the learned stage stalls: plain MG for the rest, restarted from the current iterate
                pc = FALCON_PRECOND_MG;
                ++rep->fallbacks;
                continue;
            }
            break;   // done, stalled (the refinement restarts from the FP64 residual) or out of iterations
        }
        // x += d' sr / sA (inactive problems: d' = 0)
        k_ir_accum<<<g, tpb(d), 0, sv->st>>>(d, sv->x2, sv->ir_par + np, sv->bprob, sv->x);
        SCK(cudaGetLastError(), "refine");
    }
    cudaEventRecord(t1, sv->st);
    SCK(cudaEventSynchronize(t1), "solve");
    float ms = 0;
    cudaEventElapsedTime(&ms, t0, t1);
    cudaEventDestroy(t0);
    cudaEventDestroy(t1);
    double worst = 0;
    bool done = true;
    for (int q = 0; q < np; ++q) {
        worst = std::max(worst, rel[q]);
        if (state[q] != 1) done = false;
    }
    rep->iterations = it;
    rep->refinements = std::max(0, passes - 1);
    rep->converged = done ? 1 : 0;
    rep->rel_residual = worst;
    rep->ms = ms;
    if (!done) {
        char buf[256];
        snprintf(buf, sizeof buf,
                 "not converged: FP64 relative residual %.3e above tol %.3e (%d inner iterations, %d refinement passes%s)",
                 worst, tol, it, passes, rep->floor_residual > 0 ? "; stopped at the FP64 attainable accuracy" : "");
        sv->err = buf;
        return FALCON_ERR_NOT_CONVERGED;
    }
    return FALCON_OK;
}

int falcon_solver_solution(falcon_solver* sv, double* x) {
    if (!sv || !x) return FALCON_ERR_INVALID_ARG;
    if (!sv->st) return sv->fail(FALCON_ERR_NO_DEVICE, "solver created without a device");
    cudaSetDevice(sv->device);
    const LevelDims& d = sv->lv[0].d;
    const int nb = sv->S.nblocks;
    k_gather_pad<double><<<grid_cells(d, nb), tpb(d), 0, sv->st>>>(d, sv->x, sv->z);
    SCK(cudaMemcpyAsync(x, sv->z, (size_t)nb * d.nint * 8, cudaMemcpyDeviceToHost, sv->st), "solution");
    SCK(cudaStreamSynchronize(sv->st), "solution");
    return FALCON_OK;
}

int falcon_solver_timestep(const falcon_solver* sv, double* dt) {
    if (!sv || !dt) return FALCON_ERR_INVALID_ARG;
    *dt = sv->dt_conduction;
    return FALCON_OK;
}

int falcon_solver_set_smoothing(falcon_solver* sv, int32_t nu_pre, int32_t nu_post, int32_t nu_coarse) {
    if (!sv || nu_pre < 0 || nu_post < 0 || nu_coarse < 0 || nu_pre > 64 || nu_post > 64 || nu_coarse > 4096)
        return FALCON_ERR_INVALID_ARG;
    sv->nu_pre = nu_pre;
    sv->nu_post = nu_post;
    sv->nu_coarse = nu_coarse;
    return FALCON_OK;
}

int falcon_solver_problem_residuals(falcon_solver* sv, double* rel) {
    if (!sv || !rel) return FALCON_ERR_INVALID_ARG;
    if (!sv->st) return sv->fail(FALCON_ERR_NO_DEVICE, "solver created without a device");
    cudaSetDevice(sv->device);
    const int np = sv->S.nproblems, nb = sv->S.nblocks;
    const LevelDims& d = sv->lv[0].d;
    SCK(cudaMemsetAsync(sv->dots, 0, (size_t)6 * np * 8, sv->st), "residuals");
    SCK(halo_fill(sv, 0, sv->x), "residuals");
    k_residual64<<<grid_cells(d, nb), tpb(d), 0, sv->st>>>(sv->lv[0].ops64(), d, sv->x, sv->bvec, sv->r, sv->lv[0].r,
                                                        sv->D(), 1);
    std::vector<double> rr(np), bb(np);
    SCK(cudaMemcpyAsync(rr.data(), sv->dots + 3 * np, np * 8, cudaMemcpyDeviceToHost, sv->st), "residuals");
    SCK(cudaMemcpyAsync(bb.data(), sv->dots + 4 * np, np * 8, cudaMemcpyDeviceToHost, sv->st), "residuals");
    SCK(cudaStreamSynchronize(sv->st), "residuals");
    for (int q = 0; q < np; ++q) rel[q] = bb[q] > 0 ? std::sqrt(rr[q] / bb[q]) : std::sqrt(rr[q]);
    return FALCON_OK;
}

int falcon_solver_set_rhs(falcon_solver* sv, const double* b) {
    if (!sv || !b) return FALCON_ERR_INVALID_ARG;
    std::memcpy(sv->S.b.data(), b, sv->S.b.size() * 8);
    if (sv->st) {
        cudaSetDevice(sv->device);
        SCK(cudaStreamSynchronize(sv->st), "rhs");
        SCK(cudaMemcpy(sv->bvec, b, sv->S.b.size() * 8, cudaMemcpyHostToDevice), "rhs");
        SCK(uploads_arrived(), "rhs");
    }
    return FALCON_OK;
}

int falcon_solver_coarse_shape(falcon_solver* sv, int32_t* shape) {
    if (!sv || !shape) return FALCON_ERR_INVALID_ARG;
    if (sv->st) cudaSetDevice(sv->device);
    const int rc = ensure_coarse_map(sv);
    if (rc) return rc;
    shape[0] = 2; shape[1] = sv->cD; shape[2] = sv->cH; shape[3] = sv->cW;
    return FALCON_OK;
}

int falcon_solver_attach_lcc(falcon_solver* sv, falcon_lcc* net, int32_t sweeps) {
    if (!sv || !net || sweeps < 0 || sweeps > 64) return FALCON_ERR_INVALID_ARG;
    if (sv->st) cudaSetDevice(sv->device);
    const int rc = ensure_coarse_map(sv);
    if (rc) return rc;
    sv->net = net;
    sv->clear_graphs();
    sv->net_sweeps = sweeps;
    // size the network's buffers for this grid now, not inside a timed solve
    SCK(lcc::forward_device(net, sv->feat, 2, sv->cD, sv->cH, sv->cW, sv->yout, sv->st), "lcc");
    SCK(cudaStreamSynchronize(sv->st), "lcc");
    return FALCON_OK;
}

int falcon_solver_record(falcon_solver* sv, double tol, int32_t max_iter, int32_t max_records, float* x, float* t,
                         int32_t* nrecords) {
    if (!sv || !x || !t || !nrecords || max_records < 1) return FALCON_ERR_INVALID_ARG;
    if (sv->st) cudaSetDevice(sv->device);
    int rc = ensure_coarse_map(sv);
    if (rc) return rc;
    const int lc = sv->S.nlevels - 1, nb = sv->S.nblocks;
    SvLevel& L = sv->lv[lc];
    const size_t per = (size_t)nb * L.d.nint;
    float* rec = nullptr;
    SCK(cudaMalloc(&rec, (size_t)max_records * per * 4), "record buffer");
    sv->rec = rec;
    sv->rec_max = max_records;
    sv->rec_n = 0;
    falcon_solve_report rep;
    rc = falcon_solver_solve(sv, tol, max_iter, FALCON_PRECOND_MG, &rep);
    sv->rec = nullptr;
    const int n = sv->rec_n;
    *nrecords = 0;
    if (rc == FALCON_OK || rc == FALCON_ERR_NOT_CONVERGED) {
        rc = FALCON_OK;
        const size_t vox = (size_t)2 * sv->cD * sv->cH * sv->cW;
        float* tdev = nullptr;
        cudaError_t e = cudaMalloc(&tdev, vox * 4);
        for (int q = 0; q < n && rc == FALCON_OK && e == cudaSuccess; ++q) {
            const float* rq = rec + (size_t)q * per;
            rc = coarse_solve(sv, rq);
            if (rc) break;
            const int64_t N = (int64_t)per;
            e = cudaMemsetAsync(sv->csum, 0, 8, sv->st);
            if (e != cudaSuccess) break;
            k_lcc_sumsq<<<grid_cells(L.d, nb), tpb(L.d), 0, sv->st>>>(L.d, rq, L.fAii, sv->csum);
            k_lcc_feat<<<grid_cells(L.d, nb), tpb(L.d), 0, sv->st>>>(L.d, rq, L.fAii, sv->gmap, sv->csum, N, sv->feat);
            k_lcc_target<<<grid_cells(L.d, nb), tpb(L.d), 0, sv->st>>>(L.d, sv->x, sv->gmap, sv->csum, N, tdev);
            e = cudaGetLastError();
            if (e == cudaSuccess) e = cudaMemcpyAsync(x + (size_t)q * vox * 8, sv->feat, vox * 8 * 4, cudaMemcpyDeviceToHost, sv->st);
            if (e == cudaSuccess) e = cudaMemcpyAsync(t + (size_t)q * vox, tdev, vox * 4, cudaMemcpyDeviceToHost, sv->st);
            if (e == cudaSuccess) e = cudaStreamSynchronize(sv->st);
            if (e == cudaSuccess) *nrecords = q + 1;
        }
        cudaFree(tdev);
        if (e != cudaSuccess && rc == FALCON_OK) rc = sv->fail(FALCON_ERR_CUDA, std::string("record: ") + cudaGetErrorString(e));
    }
    cudaStreamSynchronize(sv->st);
    cudaFree(rec);
    return rc;
}

}  // extern "C"
