// vcycle.cuh -- FP32 V-cycle kernels of the solver: red-black Gauss-Seidel
// sweeps, residual with restriction, prolongation, on interior-only arrays
// [block][m][m][m] (blocks are cubes of m cells, m = 2..32, halved per level).
//
// Every kernel pulls its halo: a cell on a block face reads its ghost through
// the level's descriptor table -- the source cell, or an interpolation entry --
// straight from the source block, so no halo is stored and no fill is
// launched. The sweeps are out of place (two z buffers per level): a ghost reads
// the value that the source cell had before the sweep, as a fill before each
// half sweep would leave it.
//
// A thread takes two neighbouring cells of a row, one of each colour: it
// updates one, passes the other on, and all its loads are independent. What
// bounds the kernels: HBM for the finest level (r, four coefficient arrays, z in,
// z out: 28 B per cell and half sweep, the face coefficients read whole
// although one colour is updated -- every face belongs to one red and one black
// cell), launch latency for the others.
#pragma once
#include <cstdint>
#include <type_traits>
#include <cuda_runtime.h>

namespace falcon {
namespace sv {

// explicit FMAs and a fast division (this code is otherwise compiled without
// contraction): the smoother's rounding is free, the outer CG is flexible
__device__ __forceinline__ float gs_value(float r, float off, float aii) { return __fdividef(r - off, aii); }

struct VLevel {
    int m, nint, nb;           // cells per block edge and block, blocks
    uint32_t inv_h, inv_mh;    // 2^32 / (m / 2) and 2^32 / (m^2 / 2), rounded up (EvenPair)
    const float *Aii, *Ai, *Aj, *Ak;
    const int32_t* ghost;      // [nb][6 m^2]: faces i-, i+ [k][j], j-, j+ [k][i], k-, k+ [j][i];
                               // >= 0 source cell, -1 none (0), <= -2 interpolation entry -(v + 2)
    const int32_t* isrc;       // entry: base source cell
    const uint8_t* icode;      // bit d set: the weight of direction d is not 0
    const float* iw;           // [entry][3]
    // [nb][12] faces whose ghosts come from one block, position by position:
    // 0..5 that block, -2 no ghosts (0), -1 mixed (see ghost); j and k faces
    // copy its opposite layer, i faces (blocks of another radial spacing) blend
    // cells i0 and i0 + 1 of each row: 6, 7 i0 of faces i-, i+; 8, 9 the
    // weights of the second cell (float bits; 0: a copy)
    const int32_t* nbr;
};

// What a sweep starts from
enum { V_PLAIN = 0,     // z_in
       V_FIRST = 1,     // z = 0 and the red half sweep from it: r / Aii on red cells, 0 on black ones
       V_PROLONG = 2 }; // z_in plus the coarse correction zc of the cell's parent
template <int M, int MODE>
struct Start {
    const float *r, *Aii, *zin, *zc;
    int m_;
    __device__ __forceinline__ int m() const { return M > 0 ? M : m_; }
    __device__ __forceinline__ float operator()(int q) const {
        if constexpr (MODE == V_PLAIN) return zin[q];
        const int mm = m() * m(), nint = mm * m(), h = m() >> 1;
        const int b = q / nint, c = q - b * nint, i = c % m(), j = (c / m()) % m(), k = c / mm;
        if constexpr (MODE == V_FIRST) return ((i + j + k + 1) & 1) == 0 ? gs_value(r[q], 0.f, Aii[q]) : 0.f;
        return zin[q] + zc[((b * h + (k >> 1)) * h + (j >> 1)) * h + (i >> 1)];
    }
    // of a neighbour inside the block or in one of the same layout: with even m
    // it has the other colour, and V_FIRST asks for red ones only
    __device__ __forceinline__ float near(int q) const {
        if constexpr (MODE == V_FIRST && M > 0) return gs_value(r[q], 0.f, Aii[q]);
        return (*this)(q);
    }
};

// A ghost from the table: the source cell's value, or the sum over an
// interpolation entry's corners. Only the faces at a panel's rim come here, so
// it is a call: inlined six times it would take the sweeps' registers.
template <int M, int MODE>
__device__ __noinline__ float ghost_value(const int32_t* __restrict__ isrc, const uint8_t* __restrict__ icode,
                                          const float* __restrict__ iw, int desc, Start<M, MODE> f) {
    if (desc >= 0) return f(desc);
    if (desc == -1) return 0.f;
    const int m = f.m(), e = -(desc + 2), s = isrc[e], cd = icode[e];
    const int a = (cd & 1) ? 1 : 0, b = (cd & 2) ? m : 0, c = (cd & 4) ? m * m : 0;
    const float wi = iw[3 * e], wj = iw[3 * e + 1], wk = iw[3 * e + 2];
    const float ui = 1.f - wi, uj = 1.f - wj, uk = 1.f - wk;
    if (cd == 1) return f(s) * ui + f(s + 1) * wi;
    if (a == 0)   // aligned in i (the Yin-Yang seam): four corners
        return f(s) * uj * uk + f(s + b) * wj * uk + f(s + c) * uj * wk + f(s + b + c) * wj * wk;
    return f(s) * ui * uj * uk + f(s + a) * wi * uj * uk + f(s + b) * ui * wj * uk + f(s + c) * ui * uj * wk +
           f(s + a + b) * wi * wj * uk + f(s + b + c) * ui * wj * wk + f(s + a + c) * wi * uj * wk +
           f(s + a + b + c) * wi * wj * wk;
}

// The neighbour rows of block b.
struct Faces {
    int nb[6], i0[2];
    float w[2];
    __device__ __forceinline__ Faces(const VLevel& V, int b) {
        const int4* p = reinterpret_cast<const int4*>(V.nbr + 12 * (size_t)b);
        const int4 x = p[0], y = p[1], z = p[2];
        nb[0] = x.x; nb[1] = x.y; nb[2] = x.z; nb[3] = x.w; nb[4] = y.x; nb[5] = y.y;
        i0[0] = y.z; i0[1] = y.w;
        w[0] = __int_as_float(z.x); w[1] = __int_as_float(z.y);
    }
};
// The value of the neighbour of cell q = (i, j, k) of block b across face fc:
// inside the block and across faces with one source block at an address formed
// without a branch; other ghosts through the table.
template <int FC, int M, int MODE>
__device__ __forceinline__ float neighbour(const VLevel& V, const Faces& F, int b, int i, int j, int k, int q,
                                           const Start<M, MODE>& f) {
    constexpr int hi = FC & 1;
    const int m = f.m(), mm = m * m, nint = mm * m;
    const int on = FC < 2 ? i : FC < 4 ? j : k, st = FC < 2 ? 1 : FC < 4 ? m : mm;
    const bool inside = hi ? on < m - 1 : on > 0;
    const int nb = F.nb[FC];
    int src = q + (hi ? st : -st);
    float v;
    if constexpr (FC < 2) {
        if (!inside && nb >= 0) src = q + (nb - b) * nint - i + F.i0[hi];
        const float w = inside || nb < 0 ? 0.f : F.w[hi];
        const bool none = !inside && nb < 0;
        v = inside ? f.near(src) : f(none ? q : src);
        if (w != 0.f) v = v * (1.f - w) + f(src + 1) * w;
    } else {
        // across the face: the same cell of the other block, moved to its opposite layer
        if (!inside) src = nb >= 0 ? q + (nb - b) * nint + (hi ? -(m - 1) * st : (m - 1) * st) : q;
        v = f.near(src);
    }
    if (!inside && nb < 0) {
        const int t = FC < 2 ? k * m + j : FC < 4 ? k * m + i : j * m + i;
        v = nb == -2 ? 0.f : ghost_value(V.isrc, V.icode, V.iw, V.ghost[((size_t)b * 6 + FC) * mm + t], f);
    }
    return v;
}

// the seven coefficients of a cell: faces i-, i+, j-, j+, k-, k+ and the diagonal
struct Coef7 {
    float c[7];
    __device__ __forceinline__ Coef7(const VLevel& V, int m, int b, int i, int j, int k, int q) {
        const int mm = m * m, row = k * m + j;
        const size_t fi = ((size_t)b * mm + row) * (m + 1) + i;
        const size_t fj = ((size_t)b * m * (m + 1) + (size_t)k * (m + 1) + j) * m + i;
        const size_t fk = ((size_t)b * (m + 1) * m + row) * m + i;
        c[0] = V.Ai[fi];
        c[1] = V.Ai[fi + 1];
        c[2] = V.Aj[fj];
        c[3] = V.Aj[fj + m];
        c[4] = V.Ak[fk];
        c[5] = V.Ak[fk + mm];
        c[6] = V.Aii[q];
    }
};

// Cells of the kernels for any m: a thread per cell, CTAs within one block. Lanes without
// a cell (on = false) take part in the warp's votes.
struct Cell {
    int b, i, j, k, q;
    bool on;
    __device__ __forceinline__ Cell(const VLevel& V) {
        const int m = V.m, n = (V.nint + blockDim.x - 1) / blockDim.x;
        b = blockIdx.x / n;
        const int c = (blockIdx.x - b * n) * blockDim.x + threadIdx.x, row = c / m;
        on = c < V.nint;
        i = c - row * m;
        j = row % m;
        k = row / m;
        q = b * V.nint + c;
    }
};
// The six neighbours' values of a cell (0 for lanes that want none). What bounds these
// kernels is latency: a ghost is its descriptor, an entry's fields and its corners, one
// after the other, so each of the three is loaded for all faces at once.
__device__ __forceinline__ void six_neighbours(const VLevel& V, const Cell& C, bool want, const float* __restrict__ z, float (&n)[6]) {
    const int m = V.m, mm = m * m;
    int src[6];
    bool entry = false;
#pragma unroll
    for (int f = 0; f < 6; ++f) {
        const int on = f < 2 ? C.i : f < 4 ? C.j : C.k, st = f < 2 ? 1 : f < 4 ? m : mm;
        const int t = f < 2 ? C.k * m + C.j : f < 4 ? C.k * m + C.i : C.j * m + C.i;
        src[f] = C.q + ((f & 1) ? st : -st);
        if (!((f & 1) ? on < m - 1 : on > 0)) src[f] = want ? V.ghost[((size_t)C.b * 6 + f) * mm + t] : -1;
        entry |= want && src[f] <= -2;
    }
#pragma unroll
    for (int f = 0; f < 6; ++f) n[f] = want && src[f] >= 0 ? z[src[f]] : 0.f;
    if (!__any_sync(0xffffffffu, entry)) return;
    int s[6], cd[6];
    float w[6][3];
#pragma unroll
    for (int f = 0; f < 6; ++f) {
        const bool is = want && src[f] <= -2;
        const int e = is ? -(src[f] + 2) : 0;
        s[f] = is ? V.isrc[e] : 0;
        cd[f] = is ? V.icode[e] : -1;
#pragma unroll
        for (int d = 0; d < 3; ++d) w[f][d] = is ? V.iw[3 * e + d] : 0.f;
    }
    float c[6][8];   // corner t: bit d of t one cell on along d; those of weight 0 are not read
#pragma unroll
    for (int f = 0; f < 6; ++f)
#pragma unroll
        for (int t = 0; t < 8; ++t)
            c[f][t] = cd[f] >= 0 && (t & ~cd[f]) == 0 ? z[s[f] + (t & 1) + (t & 2 ? m : 0) + (t & 4 ? mm : 0)] : 0.f;
#pragma unroll
    for (int f = 0; f < 6; ++f) {
        if (cd[f] < 0) continue;
        const float wi = w[f][0], wj = w[f][1], wk = w[f][2], ui = 1.f - wi, uj = 1.f - wj, uk = 1.f - wk;
        n[f] = c[f][0] * ui * uj * uk + c[f][1] * wi * uj * uk + c[f][2] * ui * wj * uk + c[f][4] * ui * uj * wk +
               c[f][3] * wi * wj * uk + c[f][6] * ui * wj * wk + c[f][5] * wi * uj * wk + c[f][7] * wi * wj * wk;
    }
}

// For m not a power of two: z = r / Aii on red cells, 0 on black ones (the red half sweep
// from 0); z plus the coarse correction of the cell's parent; one half sweep of `colour`
// (0 red: i + j + k even counted from 1) out of place.
__global__ void k_vfirst_any(const __grid_constant__ VLevel V, const float* __restrict__ r, float* __restrict__ z) {
    const Cell C(V);
    if (C.on) z[C.q] = ((C.i + C.j + C.k + 1) & 1) == 0 ? gs_value(r[C.q], 0.f, V.Aii[C.q]) : 0.f;
}
__global__ void k_vprolong_any(const __grid_constant__ VLevel V, const float* zin, const float* __restrict__ zc, float* zout) {
    const Cell C(V);
    const int h = V.m >> 1;
    if (C.on) zout[C.q] = zin[C.q] + zc[((C.b * h + (C.k >> 1)) * h + (C.j >> 1)) * h + (C.i >> 1)];
}
__global__ void k_vsweep_any(const __grid_constant__ VLevel V, const float* __restrict__ r, const float* __restrict__ zin,
                             float* __restrict__ zout, int colour) {
    const Cell C(V);
    const bool upd = C.on && ((C.i + C.j + C.k + 1) & 1) == colour;
    float v = C.on && !upd ? zin[C.q] : 0.f, rq = 0.f, n[6];
    float a[7] = {};
    if (upd) {
        const Coef7 A(V, V.m, C.b, C.i, C.j, C.k, C.q);
#pragma unroll
        for (int f = 0; f < 7; ++f) a[f] = A.c[f];
        rq = r[C.q];
    }
    six_neighbours(V, C, upd, zin, n);
    float off = a[0] * n[0];
#pragma unroll
    for (int f = 1; f < 6; ++f) off = fmaf(a[f], n[f], off);
    if (upd) v = gs_value(rq, off, a[6]);
    if (C.on) zout[C.q] = v;
}

constexpr int kVThreads = 128;   // of a V-cycle kernel's CTA
// The pair of cells 2 ih, 2 ih + 1 of row (j, k) of block b that a thread of the
// power-of-two kernels takes. From m = 8 a CTA lies within one block, from m =
// 16 within one plane: b (and k) are uniform, known before any thread index.
template <int M>
struct Pair {
    int b, k, j, i0, q0;
    __device__ __forceinline__ Pair() {
        constexpr int h = M / 2, per = M * M * h;   // pairs per block
        int y;
        if constexpr (per >= kVThreads) {
            constexpr int n = per / kVThreads;      // CTAs per block
            b = blockIdx.x / n;
            const int c = blockIdx.x % n;
            y = c * kVThreads + threadIdx.x;
            k = M * h >= kVThreads ? c * kVThreads / (M * h) : y / (M * h);
        } else {
            y = threadIdx.x % per;
            b = blockIdx.x * (kVThreads / per) + threadIdx.x / per;
            k = y / (M * h);
        }
        j = y / h % M;
        i0 = 2 * (y % h);
        q0 = ((b * M + k) * M + j) * M + i0;
    }
};

// ... and of any even m: CTAs within one block, divisions by multiplication (exact here:
// the dividends stay below 2^32 / m^2).
struct EvenPair {
    int b, k, j, i0, q0;
    bool on;
    __device__ __forceinline__ EvenPair(const VLevel& V) {
        const int m = V.m, h = m >> 1, per = m * m * h, n = (per + kVThreads - 1) / kVThreads;
        b = blockIdx.x / n;
        const unsigned y = (blockIdx.x - b * n) * kVThreads + threadIdx.x;
        on = y < (unsigned)per;
        k = __umulhi(y, V.inv_mh);
        const unsigned x = y - k * (m * h);
        j = __umulhi(x, V.inv_h);
        i0 = 2 * (x - j * h);
        q0 = ((b * m + k) * m + j) * m + i0;
    }
};

// One half sweep of `colour` (-1: none) on the pair at q0, out of place; with V_FIRST the
// whole first red-black sweep (colour = 1).
template <int M, int MODE>
__device__ __forceinline__ void vsweep_pair(const VLevel& V, const float* __restrict__ r, const float* __restrict__ zin,
                                            const float* __restrict__ zc, float* __restrict__ zout, int colour, int b, int i0,
                                            int j, int k, int q0) {
    const Start<M, MODE> f{r, V.Aii, zin, zc, V.m};
    const int m = f.m(), odd = (colour + j + k + 1) & 1;   // which of the two cells has the colour
    const int i = i0 + odd, q = q0 + odd;
    const Faces F(V, b);
    float2 z;
    if constexpr (MODE == V_FIRST) {
        const int p = q0 + 1 - odd;
        const float v = gs_value(r[p], 0.f, V.Aii[p]);
        z = odd ? make_float2(v, 0.f) : make_float2(0.f, v);
    } else {
        z = *reinterpret_cast<const float2*>(zin + q0);
        if constexpr (MODE == V_PROLONG) {
            const int h = m >> 1;
            const float c = zc[((b * h + (k >> 1)) * h + (j >> 1)) * h + (i0 >> 1)];
            z.x += c;
            z.y += c;
        }
    }
    if (colour >= 0) {
        const Coef7 A(V, m, b, i, j, k, q);
        const float rq = r[q];
        const float o = odd ? neighbour<1>(V, F, b, i, j, k, q, f) : neighbour<0>(V, F, b, i, j, k, q, f);
        const float n2 = neighbour<2>(V, F, b, i, j, k, q, f), n3 = neighbour<3>(V, F, b, i, j, k, q, f);
        const float n4 = neighbour<4>(V, F, b, i, j, k, q, f), n5 = neighbour<5>(V, F, b, i, j, k, q, f);
        float off = A.c[0] * (odd ? z.x : o);   // one i neighbour is the other cell of the pair
        off = fmaf(A.c[1], odd ? o : z.y, off);
        off = fmaf(A.c[2], n2, off);
        off = fmaf(A.c[3], n3, off);
        off = fmaf(A.c[4], n4, off);
        off = fmaf(A.c[5], n5, off);
        const float v = gs_value(rq, off, A.c[6]);
        if (odd) z.y = v;
        else z.x = v;
    }
    *reinterpret_cast<float2*>(zout + q0) = z;
}
template <int M, int MODE>
__global__ void __launch_bounds__(kVThreads)
k_vsweep(const __grid_constant__ VLevel V, const float* __restrict__ r, const float* __restrict__ zin,
         const float* __restrict__ zc, float* __restrict__ zout, int colour) {
    const Pair<M> C;
    if (C.b < V.nb) vsweep_pair<M, MODE>(V, r, zin, zc, zout, colour, C.b, C.i0, C.j, C.k, C.q0);
}
__global__ void __launch_bounds__(kVThreads)
k_vsweep_even(const __grid_constant__ VLevel V, const float* __restrict__ r, const float* __restrict__ zin,
              float* __restrict__ zout, int colour) {
    const EvenPair C(V);
    if (C.on) vsweep_pair<0, V_PLAIN>(V, r, zin, nullptr, zout, colour, C.b, C.i0, C.j, C.k, C.q0);
}

// r - A z at a cell with value z, the reference's operand order
template <int M>
__device__ __forceinline__ float resid_cell(const VLevel& V, const Faces& F, int b, int i, int j, int k, int q, float r,
                                            float z, float n0, float n1, const Start<M, V_PLAIN>& f) {
    const Coef7 A(V, f.m(), b, i, j, k, q);
    float y = A.c[6] * z;
    y = y + A.c[0] * n0;
    y = y + A.c[1] * n1;
    y = y + A.c[2] * neighbour<2>(V, F, b, i, j, k, q, f);
    y = y + A.c[3] * neighbour<3>(V, F, b, i, j, k, q, f);
    y = y + A.c[4] * neighbour<4>(V, F, b, i, j, k, q, f);
    y = y + A.c[5] * neighbour<5>(V, F, b, i, j, k, q, f);
    return r - y;
}

// res = r - A z
__global__ void k_vresid(const __grid_constant__ VLevel V, const float* __restrict__ r, const float* __restrict__ z,
                         float* __restrict__ res) {
    const Cell C(V);
    float n[6];
    six_neighbours(V, C, C.on, z, n);
    if (!C.on) return;
    const Coef7 A(V, V.m, C.b, C.i, C.j, C.k, C.q);
    float y = A.c[6] * z[C.q];
#pragma unroll
    for (int f = 0; f < 6; ++f) y = y + A.c[f] * n[f];
    res[C.q] = r[C.q] - y;
}
// ... on pairs of cells (m even)
template <int M>
__device__ __forceinline__ float2 resid_pair(const VLevel& V, const float* __restrict__ r, const float* __restrict__ z, int b, int i,
                                             int j, int k, int q) {
    const Start<M, V_PLAIN> f{r, V.Aii, z, nullptr, V.m};
    const Faces F(V, b);
    const float2 r2 = *reinterpret_cast<const float2*>(r + q), z2 = *reinterpret_cast<const float2*>(z + q);
    const float v0 = resid_cell(V, F, b, i, j, k, q, r2.x, z2.x, neighbour<0>(V, F, b, i, j, k, q, f), z2.y, f);
    const float v1 = resid_cell(V, F, b, i + 1, j, k, q + 1, r2.y, z2.y, z2.x, neighbour<1>(V, F, b, i + 1, j, k, q + 1, f), f);
    return make_float2(v0, v1);
}
__global__ void __launch_bounds__(kVThreads)
k_vresid_even(const __grid_constant__ VLevel V, const float* __restrict__ r, const float* __restrict__ z, float* __restrict__ res) {
    const EvenPair C(V);
    if (C.on) *reinterpret_cast<float2*>(res + C.q0) = resid_pair<0>(V, r, z, C.b, C.i0, C.j, C.k, C.q0);
}
// rc = the sum of the eight children of res (R = P^T), in the reference's order
__global__ void k_vrestrict(int m, int ncoarse, const float* __restrict__ res, float* __restrict__ rc) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, h = m >> 1;
    if (x >= ncoarse) return;
    const int I = x % h, J = (x / h) % h, K = (x / (h * h)) % h, b = x / (h * h * h);
    float s = 0.f;
#pragma unroll
    for (int q = 0; q < 8; ++q)
        s += res[((b * m + 2 * K + (q >> 2)) * m + 2 * J + ((q >> 1) & 1)) * m + 2 * I + (q & 1)];
    rc[x] = s;
}
// both in one pass for m = 2, 4, 8, 16: a thread takes two cells of a row, the
// four pairs of a coarse cell sit in one warp (lane = pair + m/2 (j & 1 + 2 (k &
// 1)) within a brick of m x 2 x 2 cells), and the residual never goes to HBM.
template <int M>
__global__ void __launch_bounds__(kVThreads)
k_vresid_restrict(const __grid_constant__ VLevel V, const float* __restrict__ r, const float* __restrict__ z,
                  float* __restrict__ rc) {
    constexpr int h = M / 2, per = M * M * h;   // pairs per block
    int b, y;
    if constexpr (per >= kVThreads) {
        b = blockIdx.x / (per / kVThreads);
        y = blockIdx.x % (per / kVThreads) * kVThreads + threadIdx.x;
    } else {
        b = blockIdx.x * (kVThreads / per) + threadIdx.x / per;
        y = threadIdx.x % per;
    }
    const bool on = b < V.nb;
    b = min(b, V.nb - 1);   // every lane takes part in the shuffles
    const int ih = y % h, sub = (y / h) & 3, brick = y / (4 * h), J = brick % h, K = brick / h;
    const int j = 2 * J + (sub & 1), k = 2 * K + (sub >> 1), q = ((b * M + k) * M + j) * M + 2 * ih;
    const float2 v = resid_pair<M>(V, r, z, b, 2 * ih, j, k, q);
    const float v0 = v.x, v1 = v.y;
    float s = 0.f;
    s += v0;
    s += v1;
#pragma unroll
    for (int t = 1; t < 4; ++t) {
        s += __shfl_down_sync(0xffffffffu, v0, t * h);
        s += __shfl_down_sync(0xffffffffu, v1, t * h);
    }
    if (on && sub == 0) rc[((b * h + K) * h + J) * h + ih] = s;
}

// ---- the coarsest level's sweeps in one launch -----------------------------------
// A cluster of CTAs holds one problem's coarsest level: each CTA a run of
// whole blocks, every thread R red and R black cells with their coefficients in
// registers, z in shared memory. A half sweep has two phases: the ghosts that
// are interpolated, lie in another CTA (distributed shared memory) or copy a
// cell of the same colour are gathered into slots, one per thread, then the
// cells of the colour are updated in place from local words of the other
// colour and the slots, without a branch. One launch replaces a launch per
// half sweep: what is left is the chain of half sweeps.
constexpr int kCoarseThreads = 512;
// A gathered ghost: the sum of w[c] times the cells word + (0, off & 255, off >> 8 &
// 255, off >> 16) -- a copy (w[0] = 1), a radial blend (two cells) or the
// Yin-Yang seam's four (of a ghost between the panels' radial layers: two
// entries); cells of weight 0 are not read.
struct CoarseEntry {
    uint2 at;   // word, off
    float4 w;
};
struct CoarseArgs {
    const int32_t* first;      // [problem + 1]: first block
    const uint32_t* ghost;     // the level's ghost table as words
    const uint2* at;           // gathered ghosts (CoarseEntry) per CTA, by colour of the cell that reads them
    const float4* w;
    // [CTA][2 colours] first entry, ghosts, and how many of the last ones sum
    // eight cells: their other four follow the list
    const int4* list;
    int sweeps;                // red-black sweeps
    int cluster;               // CTAs per problem
};
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// A barrier passes a token on; loads of the memory that it orders take the
// token as an operand, so that they stay behind it without being volatile
// and several can be in flight.
template <bool CLUSTER>
__device__ __forceinline__ uint32_t sweep_barrier(uint32_t token) {
    uint32_t t;
    if constexpr (CLUSTER)
        asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\nmov.b32 %0, %1;"
                     : "=r"(t)
                     : "r"(token)
                     : "memory");
    else
        asm volatile("bar.sync 0;\nmov.b32 %0, %1;" : "=r"(t) : "r"(token) : "memory");
    return t;
}
__device__ __forceinline__ float ld_cluster(uint32_t addr, uint32_t rank, uint32_t token) {
    float v;
    asm("{\n.reg .b32 a;\nmapa.shared::cluster.u32 a, %1, %2;\nadd.u32 a, a, %3;\nld.shared::cluster.f32 %0, [a];\n}"
        : "=f"(v)
        : "r"(addr), "r"(rank), "r"(token));
    return v;
}

// A cell's word: owner rank << 24 | cell within the owner. In the ghost
// table a local cell stands without its rank, kSlot | n is gathered slot n; a ghost without a source is kNone.
constexpr uint32_t kNone = 0xffffffffu, kSlot = 0x80000000u;

template <int M, int R, bool CLUSTER>
__global__ void __launch_bounds__(kCoarseThreads, 1)
k_coarse_sweeps(VLevel V, CoarseArgs C, const float* __restrict__ r, float* __restrict__ zout) {
    extern __shared__ float tile[];
    constexpr int CAP = 2 * R * kCoarseThreads;          // cells per CTA
    constexpr int mm = M * M, nint = mm * M, hr = M / 2, half = nint / 2;
    constexpr int ZERO = CAP, SLOT = CAP + 1;
    float* z = tile;   // [CAP], a zero for missing neighbours, the slots
    const int p = blockIdx.x / C.cluster, tid = threadIdx.x;
    const uint32_t rank = CLUSTER ? cluster_rank() : 0u;
    const int pb0 = C.first[p], pnb = C.first[p + 1] - pb0;
    const int bpc = (pnb + C.cluster - 1) / C.cluster;    // blocks per CTA
    const int b0 = min((int)rank * bpc, pnb), nblk = min(bpc, pnb - b0);
    const int q0 = (pb0 + b0) * nint;                     // this CTA's first cell
    for (int x = tid; x <= CAP; x += kCoarseThreads) z[x] = 0.f;
    const int4 lists[2] = {C.list[2 * blockIdx.x], C.list[2 * blockIdx.x + 1]};
    float co[2][R][7], rv[2][R];
    int loc[2][R];
    uint32_t nb[2][R][3];   // the six neighbours' places in z, 16 bits each
#pragma unroll
    for (int col = 0; col < 2; ++col)
#pragma unroll
        for (int s = 0; s < R; ++s) {
            const int hh = tid + s * kCoarseThreads;
            loc[col][s] = -1;
            if (hh >= nblk * half) continue;
            const int lb = hh / half, y = hh % half, row = y / hr, j = row % M, k = row / M;
            const int i = 2 * (y % hr) + ((col + j + k + 1) & 1);
            const int c = row * M + i, b = pb0 + b0 + lb, q = b * nint + c;
            loc[col][s] = lb * nint + c;
            rv[col][s] = r[q];
            const Coef7 A(V, M, b, i, j, k, q);
#pragma unroll
            for (int f = 0; f < 7; ++f) co[col][s][f] = A.c[f];
#pragma unroll
            for (int f = 0; f < 6; ++f) {
                const int on = f < 2 ? i : f < 4 ? j : k, st = f < 2 ? 1 : f < 4 ? M : mm;
                uint32_t w = (uint32_t)(loc[col][s] + ((f & 1) ? st : -st));
                if (!((f & 1) ? on < M - 1 : on > 0)) {
                    w = C.ghost[((size_t)b * 6 + f) * mm + (f < 2 ? k * M + j : f < 4 ? k * M + i : j * M + i)];
                    w = w == kNone ? ZERO : (w & kSlot) ? SLOT + (w & ~kSlot) : w;
                }
                if (f & 1) nb[col][s][f >> 1] |= w << 16;
                else nb[col][s][f >> 1] = w;
            }
        }
    const uint32_t zaddr = (uint32_t)__cvta_generic_to_shared(z);
    uint32_t token = 0;   // always 0
    auto load = [&](uint32_t word, uint32_t off) -> float {
        const uint32_t c = (word & 0xffffu) + off;
        if constexpr (CLUSTER) return ld_cluster(zaddr + 4u * c, word >> 24, token);
        else return z[c];
    };
    auto gather = [&](uint2 at, float4 w) -> float {
        const float v0 = load(at.x, 0u);
        float v1 = 0.f, v2 = 0.f, v3 = 0.f;
        if (w.y != 0.f) v1 = load(at.x, at.y & 255u);
        if (w.z != 0.f) v2 = load(at.x, at.y >> 8 & 255u);
        if (w.w != 0.f) v3 = load(at.x, at.y >> 16);
        return v0 * w.x + v1 * w.y + v2 * w.z + v3 * w.w;
    };
    constexpr int U = 2;   // gathered ghosts in flight per thread
    token = sweep_barrier<CLUSTER>(token);
    for (int s2 = 0; s2 < 2 * C.sweeps; ++s2) {
        auto half_sweep = [&](auto colc) {
            constexpr int col = decltype(colc)::value;
            const int a = lists[col].x, n = lists[col].y, simple = n - lists[col].z;
            for (int x = tid; x < n; x += U * kCoarseThreads) {
                float v[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int y = a + min(x + u * kCoarseThreads, n - 1);
                    v[u] = gather(C.at[y], C.w[y]);
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int y = x + u * kCoarseThreads;
                    if (y >= n) continue;
                    if (y >= simple) v[u] += gather(C.at[a + n + y - simple], C.w[a + n + y - simple]);
                    z[SLOT + y] = v[u];
                }
            }
            token = sweep_barrier<CLUSTER>(token);
#pragma unroll
            for (int s = 0; s < R; ++s) {
                if (loc[col][s] < 0) continue;
                float v[6];
#pragma unroll
                for (int f = 0; f < 6; ++f) v[f] = z[(f & 1) ? nb[col][s][f >> 1] >> 16 : nb[col][s][f >> 1] & 0xffffu];
                float off = co[col][s][0] * v[0];
#pragma unroll
                for (int f = 1; f < 6; ++f) off = fmaf(co[col][s][f], v[f], off);
                z[loc[col][s]] = gs_value(rv[col][s], off, co[col][s][6]);
            }
        };
        if (s2 & 1) half_sweep(std::integral_constant<int, 1>{});
        else half_sweep(std::integral_constant<int, 0>{});
        token = sweep_barrier<CLUSTER>(token);
    }
#pragma unroll
    for (int col = 0; col < 2; ++col)
#pragma unroll
        for (int s = 0; s < R; ++s)
            if (loc[col][s] >= 0) zout[q0 + loc[col][s]] = z[loc[col][s]];
}

}  // namespace sv
}  // namespace falcon
