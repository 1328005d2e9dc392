// mhd_mixed_impl.cuh -- kernels of the mixed step: FP32 state [b][half][cell][4]
// (Layout), u^n compensated by an 8-bit correction [b][interior cell][8].
// Included by mhd_mixed.cu.
#pragma once
#include "mhd_impl.cuh"

namespace falcon {
namespace impl {

// the four values of half `h` of padded cell c of block b
__device__ __forceinline__ size_t quad(int b, int h, int ncell) { return ((size_t)b * 2 + h) * ncell; }
__device__ __forceinline__ const float4* quads(const float* u) { return reinterpret_cast<const float4*>(u); }
__device__ __forceinline__ float4* quads(float* u) { return reinterpret_cast<float4*>(u); }
__device__ __forceinline__ float4 f4(const float* v) { return make_float4(v[0], v[1], v[2], v[3]); }
__device__ __forceinline__ void split(float4 a, float4 b, float (&v)[NV]) {
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}

// ---------------------------------------------------------------------------
// FP32 arithmetic of the mixed step, on pairs of values where it can be (Blackwell's
// two-lane FFMA2/FADD2/FMUL2). The scalar forms give the pairs' bits (a difference
// a - b is formed as fma(b, -1, a), one rounding of the exact difference, as FADD does).
__device__ __forceinline__ float2 f2(float x, float y) { return make_float2(x, y); }
__device__ __forceinline__ float2 f2(float x) { return make_float2(x, x); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, f2(-1.f), a); }

// Half the minmod slope of a cell (3_6/ModLinReconstruct.f90:44-48, halved: the
// fluxes use it so). With da = ur - ul, dr = ur - u, dl = u - ul the reference's
// a = da/2, b = 2 dr, c = 2 dl and its selector max(0, ab) 1e10 max(0, bc) >= 1e-30
// is (|da dr| 1e10) (dr dl) >= 2.5e-31: ab = da dr and bc = 4 dr dl, and of products
// large enough to pass, ab is positive where bc is. The minimum of |a|, |b|, |c| is
// halved likewise, all by powers of two.
__device__ __forceinline__ float half_slope_of(float da, float dr, float dl, float qa, float t, float p) {
    const float m = fminf(fminf(fabsf(qa), fabsf(dr)), fabsf(dl));
    return __fmul_rn(fabsf(t), p) >= 0.25f * 1.e-30f ? copysignf(m, da) : 0.f;
}
__device__ __forceinline__ float half_slope(float ul, float u, float ur) {
    const float da = __fsub_rn(ur, ul), dr = __fsub_rn(ur, u), dl = __fsub_rn(u, ul);
    return half_slope_of(da, dr, dl, __fmul_rn(da, 0.25f), __fmul_rn(__fmul_rn(da, dr), 1.e10f), __fmul_rn(dr, dl));
}
__device__ __forceinline__ float2 half_slope2(float2 ul, float2 u, float2 ur) {
    const float2 da = sub2(ur, ul), dr = sub2(ur, u), dl = sub2(u, ul);
    const float2 qa = __fmul2_rn(da, f2(0.25f)), t = __fmul2_rn(__fmul2_rn(da, dr), f2(1.e10f)), p = __fmul2_rn(dr, dl);
    return f2(half_slope_of(da.x, dr.x, dl.x, qa.x, t.x, p.x), half_slope_of(da.y, dr.y, dl.y, qa.y, t.y, p.y));
}

// The limited flux through a face (3_6/ModDiffusion.f90:40-60) from its two cells'
// values and half slopes: -(phi/2 num) speed/2 with phi = max(0, 1 + 2 (num/den - 1)),
// den = fr - fl, num the jump left between the reconstructions; cc = -2 speed, speed
// the sum of the cells' |v_dir| + c_s. Slopes have den's sign or are 0, so num/den is at
// most 1, and the quotient, num times the approximate reciprocal of den, at most 1 + 2^-22:
// phi/8 saturates to [0, 1] without rounding it again from above; one saturating FMA
// forms it, 0/0 as 0. The reciprocal flushes a denormal den, whose quotient is infinite:
// the bound above makes phi 1 there, the value for slopes of 0, which the selector gives
// (it has den's square) unless the cells' other differences exceed 5e17.
__device__ __forceinline__ float eighth_phi(float r) {
    return fminf(__saturatef(__fmaf_rn(r, 0.25f, -0.125f)), 0.125f * (1.f + 1.f / (1 << 21)));
}
__device__ __forceinline__ float face_flux(float fl, float fr, float hL, float hR, float cc) {
    const float num = __fsub_rn(__fsub_rn(__fsub_rn(fr, hR), fl), hL);
    return __fmul_rn(__fmul_rn(eighth_phi(__fmul_rn(num, rcp_approx(__fsub_rn(fr, fl)))), num), cc);
}
__device__ __forceinline__ float2 face_flux2(float2 fl, float2 fr, float2 hL, float2 hR, float2 cc) {
    const float2 num = sub2(sub2(sub2(fr, hR), fl), hL), den = sub2(fr, fl);
    const float2 r = __fmul2_rn(num, f2(rcp_approx(den.x), rcp_approx(den.y)));
    return __fmul2_rn(__fmul2_rn(f2(eighth_phi(r.x), eighth_phi(r.y)), num), cc);
}
// cc of a face: uL, uR the velocity across it, csL, csR the sound speeds of its cells
__device__ __forceinline__ float face_speed(float uL, float csL, float uR, float csR) {
    return -2.f * ((fabsf(uR) + csR) + (fabsf(uL) + csL));
}

// (hi + q*unit(hi)) + d for four values, rounded to the nearest (hi', q') pairs: two
// error-free FP32 sums (Knuth's TwoSum), no contraction. q: four corrections in a
// word, renewed. A correction q is q + 128 in the low bits of 2^23's float; the
// rounding to the nearest integer, ties to even, is the add of 1.5 * 2^23, whose ulp
// is 1 and whose low byte is then q (the clamp comes first, NaN residuals give -127).
__device__ __forceinline__ float2 ff_add2(float2 hi, float2 q, float2 d, float2& lo) {
    auto unit = [](float x) { return __int_as_float(max((__float_as_int(x) & 0x7f800000) - (31 << 23), 0)); };   // lo_unit
    auto inv_unit = [](float x) {   // lo_inv_unit
        const unsigned t = (unsigned)__float_as_int(x) & 0x7f800000u;
        return __int_as_float((int)(t >= (32u << 23) ? (285u << 23) - t : 0u));
    };
    const float2 l = __fmul2_rn(__fadd2_rn(q, f2(-8388736.f)), f2(unit(hi.x), unit(hi.y)));   // exact
    const float2 s = __fadd2_rn(hi, d);
    const float2 bs = sub2(s, hi);
    const float2 es = __fadd2_rn(sub2(hi, sub2(s, bs)), sub2(d, bs));
    const float2 t = __fadd2_rn(es, l);
    const float2 h = __fadd2_rn(s, t);
    const float2 bh = sub2(h, s);
    const float2 r = __fmul2_rn(__fadd2_rn(sub2(s, sub2(h, bh)), sub2(t, bh)), f2(inv_unit(h.x), inv_unit(h.y)));
    lo = __fadd2_rn(f2(fminf(fmaxf(r.x, -127.f), 127.f), fminf(fmaxf(r.y, -127.f), 127.f)), f2(12582912.f));
    return h;
}
__device__ __forceinline__ void ff_add4(const float* hi, int& q, const float2 (&d)[2], float* o) {
    const unsigned w = (unsigned)q ^ 0x80808080u;
    auto byte = [&](int k) { return __int_as_float((int)__byte_perm(w, 0x4B000000u, 0x7440 + k)); };
    float2 la, lb;
    const float2 a = ff_add2(f2(hi[0], hi[1]), f2(byte(0), byte(1)), d[0], la);
    const float2 b = ff_add2(f2(hi[2], hi[3]), f2(byte(2), byte(3)), d[1], lb);
    o[0] = a.x; o[1] = a.y; o[2] = b.x; o[3] = b.y;
    auto bits = [](float x) { return (unsigned)__float_as_int(x); };
    q = (int)__byte_perm(__byte_perm(bits(la.x), bits(la.y), 0x40), __byte_perm(bits(lb.x), bits(lb.y), 0x40), 0x5410);
}

// v_wave of the CFL ratio (cfl_ratio_f's) at a cell of a column with c_s = cs and
// sqrt(rho0) = d, y = RN(1/d): the quotient sqrt(b2)/d through the reciprocal (P.
// Markstein, IBM J. R&D 34 (1990) 111; the first correction brings q within an ulp).
// RN(h / w) falls as w grows and h is the column's, so its minimum over a column is
// h / max(w): one division a column.
__device__ __forceinline__ float cfl_speed(float v2, float b2, float cs, float d, float y) {
    const float a = __fsqrt_rn(b2);
    float q = __fmul_rn(a, y);
    if (q < INFINITY) {
        q = __fmaf_rn(__fmaf_rn(-d, q, a), y, q);
        q = __fmaf_rn(__fmaf_rn(-d, q, a), y, q);
    }
    return __fadd_rn(__fadd_rn(cs, __fsqrt_rn(v2)), q);
}
// The column's minimum ratio, from its largest speed
__device__ __forceinline__ float cfl_column(float wmax, float r, float sin_t, float dxi, float dxj, float dxk) {
    return __fdiv_rn(fminf(fminf(dxi, __fmul_rn(r, dxj)), __fmul_rn(__fmul_rn(r, sin_t), dxk)), wmax);
}

// Thread 0: bulk-copy planes kp in [lo, hi) of both halves of the block into
// their ring slots (plane kp in slot (kp - p0) % W), completing on `bar`.
template <class S>
__device__ __forceinline__ void issue_quads(const float* blk, float4* tile, int lo, int hi, int p0, uint64_t* bar) {
    mbar_expect_tx(bar, (uint32_t)(2 * (hi - lo)) * S::PL * 16u);
    for (int h = 0; h < 2; ++h)
        for (int kp = lo; kp < hi; ++kp)
            tma_load_1d(tile + ((size_t)h * S::W + (kp - p0) % S::W) * S::PL,
                        quads(blk) + ((size_t)h * S::NKP + kp) * S::PL, S::PL * 16u, bar);
}

// Radial mirror boundary (3_6/ModBoundary.f90:10-55) on planes [lo, hi) of the
// ring, whole rows including their theta ghosts; optionally written back.
template <class S>
__device__ __forceinline__ void apply_bc_quads(float4* tile, int lo, int hi, int p0, int fl, float* wb, int nt) {
    const bool top = fl & 2, bot = fl & 4;
    if (!top && !bot) return;
    const int NI = S::NIP - 4;
    // top mirrors rho1, vt, vp, s1, br and anti-mirrors vr, bt, bp; bottom
    // mirrors rho1, vt, vp, s1, bt, bp and anti-mirrors vr, br
    const int total = (hi - lo) * S::NJP * 4;
    for (int x = threadIdx.x; x < total; x += nt) {
        const int g = x & 1, h = (x >> 1) & 1, rest = x >> 2, j = rest % S::NJP, kp = lo + rest / S::NJP;
        float4* row = tile + ((size_t)h * S::W + (kp - p0) % S::W) * S::PL + j * S::NIP;
        float4* out = wb ? quads(wb) + ((size_t)h * S::NKP + kp) * S::PL + j * S::NIP : nullptr;
        if (top) {   // Fortran i = ni+1+g <- 2*ni+1-i = ni-g ; padded index = Fortran + 1
            float4 s = row[NI - g + 1];
            s = h ? make_float4(s.x, -s.y, -s.z, s.w) : make_float4(s.x, -s.y, s.z, s.w);
            row[NI + 2 + g] = s;
            if (out) out[NI + 2 + g] = s;
        }
        if (bot) {   // Fortran i = -g <- 1-i = 1+g
            float4 s = row[2 + g];
            s = h ? make_float4(-s.x, s.y, s.z, s.w) : make_float4(s.x, -s.y, s.z, s.w);
            row[1 - g] = s;
            if (out) out[1 - g] = s;
        }
    }
}

// Write this cell's new values into the ghost cells of the neighbours whose
// faces are pushed (PushTable), o its values.
// (ii, jj, kp): padded indices. Theta/phi faces: the two interior layers next to
// the side are copied to the target's opposite ghost layers (a shift of one
// block extent). Radial faces: the thread at the first source cell of a ghost
// layer blends it with the next cell along i, taken from the next lane (i is
// the fastest thread index, and the second cell is never beyond the row). Every
// write is whole 16-byte cells, the two layers of a radial face one sector.
// Every thread of the warp calls this (the shuffle needs it).
template <class S>
__device__ __forceinline__ void push_quads(float* out, const PushBlock& P, int ii, int jj, int kp, const float (&o)[NV]) {
    constexpr int NJ = S::NJP - 4, NK = S::NKP - 4;
    const int32_t* tg = P.tgt;
    auto put = [&](int tb, int kt, int jt, int it, const float (&val)[NV]) {
        float4* dst = quads(out) + quad(tb, 0, S::NCELL) + ((size_t)kt * S::NJP + jt) * S::NIP + it;
        dst[0] = f4(val);
        dst[S::NCELL] = f4(val + 4);
    };
    if (jj <= 3 && tg[2] >= 0) put(tg[2], kp, jj + NJ, ii, o);
    if (jj >= NJ && tg[3] >= 0) put(tg[3], kp, jj - NJ, ii, o);
    if (kp <= 3 && tg[4] >= 0) put(tg[4], kp + NK, jj, ii, o);
    if (kp >= NK && tg[5] >= 0) put(tg[5], kp - NK, jj, ii, o);
#pragma unroll
    for (int side = 0; side < 2; ++side) {
        if (tg[side] < 0) continue;   // uniform over the CTA
        const float w0 = P.w[2 * side], w1 = P.w[2 * side + 1];
        const bool l0 = ii == P.src[2 * side], l1 = ii == P.src[2 * side + 1];
        if (w0 == 0.f && w1 == 0.f) {   // copies
            if (l0) put(tg[side], kp, jj, P.dst[2 * side], o);
            if (l1) put(tg[side], kp, jj, P.dst[2 * side + 1], o);
            continue;
        }
        float nx[NV];
#pragma unroll
        for (int v = 0; v < NV; ++v) nx[v] = __shfl_down_sync(0xffffffffu, o[v], 1);
#pragma unroll
        for (int layer = 0; layer < 2; ++layer) {
            if (!(layer ? l1 : l0)) continue;
            const float w = layer ? w1 : w0, uw = 1.f - w;
            float val[NV];
#pragma unroll
            for (int v = 0; v < NV; ++v) val[v] = w == 0.f ? o[v] : blend(o[v], nx[v], uw, w);
            put(tg[side], kp, jj, P.dst[2 * side + layer], val);
        }
    }
}

// ---------------------------------------------------------------------------
// The RK stage: boundary -> RHS (3_6/ModEquation.f90:24-162) ->
// u_out = u^n + dt*R/(5-s) (3_6/ModAdvance.f90:87-93). Two kernels around one cell
// update (stage_cell): the march of 16^3 blocks and the chunks of 8^3 blocks.
//
// The derivatives need rho1 only through p1, so p1 takes rho1's place in the
// shared-memory ring as soon as a plane has arrived (its reads come with the
// velocities'); rho1 of the cells themselves is kept beside it, for the
// buoyancy. The derivatives are formed direction by direction, each from the
// four neighbours' eight values read as two 16-byte accesses.

// Geometry of a block in shared memory: a cell's radial factors in 16-byte
// groups, the theta factors likewise
enum { TI_P1 = 0, TI_R, TI_INV, TI_SRC, TI_COUNT };
struct StageTables {
    float4* ti;   // [TI_COUNT][NIP]: p1 coefficients (hi, lo pairs) | rho0, r^2, r, cs | 1/r, 1/r^2, 1/rho0, 1/Xi^2 | g/rho0, heat
    float4* tj;   // [NJP]: sin, 1/sin, cot of theta
    float* gs;    // [GS_COUNT]
    template <int NIP, int NJP> static constexpr size_t bytes() { return ((size_t)TI_COUNT * NIP + NJP) * 16 + GS_COUNT * 4; }
    __device__ StageTables(unsigned char* m, int nip, int njp)
        : ti(reinterpret_cast<float4*>(m)), tj(ti + TI_COUNT * nip), gs(reinterpret_cast<float*>(tj + njp)) {}
    __device__ void load(const Geometry& g, int b, int nip, int njp, int nt) {
        const float* Gi = g.gi_f + (size_t)b * GI_COUNT * nip;
        const float* Gj = g.gj_f + (size_t)b * GJ_COUNT * njp;
        const double* Gd = g.gi + (size_t)b * GI_COUNT * nip;
        for (int x = threadIdx.x; x < nip; x += nt) {
            // p1's coefficients as FP32 pairs, hi + lo to about 2^-48
            const double a1 = Gd[GI_A1 * nip + x], a2 = Gd[GI_A2 * nip + x];
            const float h1 = (float)a1, h2 = (float)a2;
            ti[TI_P1 * nip + x] = make_float4(h1, (float)(a1 - (double)h1), h2, (float)(a2 - (double)h2));
            ti[TI_R * nip + x] = make_float4(Gi[GI_RHO0 * nip + x], Gi[GI_R2 * nip + x], Gi[GI_R * nip + x], Gi[GI_CS * nip + x]);
            ti[TI_INV * nip + x] = make_float4(Gi[GI_RINV * nip + x], Gi[GI_R2INV * nip + x], Gi[GI_RHO0INV * nip + x], Gi[GI_XI2INV * nip + x]);
            ti[TI_SRC * nip + x] = make_float4(Gi[GI_GOR0 * nip + x], Gi[GI_HEAT * nip + x], 0.f, 0.f);
        }
        for (int x = threadIdx.x; x < njp; x += nt)
            tj[x] = make_float4(Gj[GJ_SIN * njp + x], Gj[GJ_SININV * njp + x], Gj[GJ_COT * njp + x], 0.f);
        if (threadIdx.x < GS_COUNT) gs[threadIdx.x] = g.gs_f[(size_t)b * GS_COUNT + threadIdx.x];
    }
    // p1 = gamma1*(p0/rho0)*rho1 + (gamma3-1)*(rho0*T0)*s1 (3_6/ModEquation.f90:40-46)
    __device__ float p1(int ic, float r1, float s1) const {   // (the p1 group is the first)
        const float4 t = ti[ic];
        return p1_ff(t.x, t.y, t.z, t.w, r1, s1);
    }
};

// The ghost cells of a plane that its interior cells' differences reach (rows
// and columns; corners have no reader), by index y in [0, 4 (NI + NJ)): padded
// cell c and its i. Sizes are powers of two: no divisions.
template <int NI, int NJ, int NIP>
__device__ __forceinline__ void reached_ghost(int y, int& c, int& ic) {
    constexpr int HC = 4 * (NI + NJ);
    static_assert((HC & (HC - 1)) == 0 && NI == NJ, "by shifts and masks");
    // s: which of the four lines, m: along it. Columns: neighbouring lanes on the
    // four lines (the rows of a line lie in two shared-memory banks)
    const bool row = y < HC / 2;
    const int s = row ? y / NI % 4 : y % 4, m = (row ? y % NI : y % (HC / 2) / 4) + 2, e = s < 2 ? s : NI + s;
    c = row ? e * NIP + m : m * NIP + e;
    ic = row ? m : e;
}

// -(f(2) - 8 f(1) + 8 f(-1) - f(-2)): the O4 difference's sum for two values at
// once (packed FP32), negated (every rounding is symmetric)
__device__ __forceinline__ float2 d4neg2(float2 fp2, float2 fp1, float2 fm1, float2 fm2) {
    return __ffma2_rn(fm2, f2(-1.f), __ffma2_rn(fm1, f2(8.f), __ffma2_rn(fp1, f2(-8.f), fp2)));
}

// One cell: (ca, cb) its values with p1 in rho1's place, along_x(h, m) those of
// the neighbour m in {-2, -1, 1, 2} along x, half h; (ua, ub) its u^n and q8 the
// correction (u^n set by before_k at the latest; final_stage: compensated update,
// q8 renewed). o: the new values. No branch between the sums: which products of
// a sum the compiler contracts, and so the last bits, follows from its basic block.
template <int NIP, int PL, int NCELL, int DIVB, class FI, class FJ, class FK, class FG, class FS, class FB>
__device__ __forceinline__ void stage_cell(const StageTables& tab, int b, int ii, int jj, size_t cell, float4 ca, float4 cb,
                                           float rho1, FI along_i, FJ along_j, FK along_k, FG radial, FS sine, FB before_k, const float4& ua,
                                           const float4& ub, int2& q8, bool final_stage, float dtk, const DivBArgs& psi,
                                           float (&o)[NV]) {
    using T = float;
    const T c1 = tab.gs[GS_C1], c2 = tab.gs[GS_C2], c3 = tab.gs[GS_C3];
    const float4 inv = tab.ti[TI_INV * NIP + ii], th = tab.tj[jj];
    const T rinv = inv.x, r2inv = inv.y, rho0inv = inv.z, xi2inv = inv.w, sinv = th.y, cot = th.z;
    const T rho0c = tab.ti[TI_R * NIP + ii].x;
    // ModDerivative_1st_O4_3D (3_6/ModDerivative.f90:16-32)
    auto D = [&](T c, auto f) -> T { return c * (((-f(2) + T(8) * f(1)) - T(8) * f(-1)) + f(-2)); };
    const T vr = ca.y, vt = ca.z, vp = ca.w, br = cb.x, bt = cb.y, bp = cb.z;
    T dA, a_vr, a_vt, a_vp, a_s1, g1, d_bpr, d_btr, q_e3r, q_e2r, dB = T(0);
    {   // along i
        float4 A[5], B[5], G[5];
#pragma unroll
        for (int m = -2; m <= 2; ++m) {
            if (m == 0) continue;
            A[m + 2] = along_i(0, m);
            B[m + 2] = along_i(1, m);
            G[m + 2] = radial(m);   // rho0, r^2, r
        }
        auto E2 = [&](int m) { return A[m + 2].w * B[m + 2].x - A[m + 2].y * B[m + 2].z; };
        auto E3 = [&](int m) { return A[m + 2].y * B[m + 2].y - A[m + 2].z * B[m + 2].x; };
        const float2 d0 = d4neg2(f2(A[4].x, A[4].y), f2(A[3].x, A[3].y), f2(A[1].x, A[1].y), f2(A[0].x, A[0].y));
        const float2 d1 = d4neg2(f2(A[4].z, A[4].w), f2(A[3].z, A[3].w), f2(A[1].z, A[1].w), f2(A[0].z, A[0].w));
        dA = D(c1, [&](int m) { return (G[m + 2].x * A[m + 2].y) * G[m + 2].y; });
        dA = dA * r2inv;
        a_vr = vr * (-c1 * d0.y);
        a_vt = vr * (-c1 * d1.x);
        a_vp = vr * (-c1 * d1.y);
        a_s1 = vr * D(c1, [&](int m) { return B[m + 2].w; });
        g1 = -c1 * d0.x;
        d_bpr = D(c1, [&](int m) { return B[m + 2].z * G[m + 2].z; });
        d_btr = D(c1, [&](int m) { return B[m + 2].y * G[m + 2].z; });
        q_e3r = D(c1, [&](int m) { return E3(m) * G[m + 2].z; });
        q_e2r = D(c1, [&](int m) { return E2(m) * G[m + 2].z; });
        if constexpr (DIVB != 0) dB = D(c1, [&](int m) { return B[m + 2].x * G[m + 2].y; });
    }
    T d23, g2, k1, k3, q1, q3, e23 = T(0);
    {   // along j
        float4 A[5], B[5];
        T sn[5];
#pragma unroll
        for (int m = -2; m <= 2; ++m) {
            if (m == 0) continue;
            A[m + 2] = along_j(0, m);
            B[m + 2] = along_j(1, m);
            sn[m + 2] = sine(m);
        }
        auto E1 = [&](int m) { return A[m + 2].z * B[m + 2].z - A[m + 2].w * B[m + 2].y; };
        auto E3 = [&](int m) { return A[m + 2].y * B[m + 2].y - A[m + 2].z * B[m + 2].x; };
        const float2 d0 = d4neg2(f2(A[4].x, A[4].y), f2(A[3].x, A[3].y), f2(A[1].x, A[1].y), f2(A[0].x, A[0].y));
        const float2 d1 = d4neg2(f2(A[4].z, A[4].w), f2(A[3].z, A[3].w), f2(A[1].z, A[1].w), f2(A[0].z, A[0].w));
        d23 = D(c2, [&](int m) { return (rho0c * A[m + 2].z) * sn[m + 2]; });
        T t = vt * (-c2 * d0.y);
        a_vr = a_vr + t * rinv;
        t = vt * (-c2 * d1.x);
        a_vt = a_vt + t * rinv;
        t = vt * (-c2 * d1.y);
        a_vp = a_vp + t * rinv;
        t = vt * D(c2, [&](int m) { return B[m + 2].w; });
        a_s1 = a_s1 + t * rinv;
        g2 = -c2 * d0.x;
        k1 = D(c2, [&](int m) { return B[m + 2].z * sn[m + 2]; });
        k3 = d_btr - D(c2, [&](int m) { return B[m + 2].x; });
        q1 = D(c2, [&](int m) { return E3(m) * sn[m + 2]; });
        q3 = q_e2r - D(c2, [&](int m) { return E1(m); });
        if constexpr (DIVB != 0) e23 = D(c2, [&](int m) { return B[m + 2].y * sn[m + 2]; });
    }
    before_k();
    T g3, k2, q2;
    {   // along k
        float4 A[5], B[5];
#pragma unroll
        for (int m = -2; m <= 2; ++m) {
            if (m == 0) continue;
            A[m + 2] = along_k(0, m);
            B[m + 2] = along_k(1, m);
        }
        auto E1 = [&](int m) { return A[m + 2].z * B[m + 2].z - A[m + 2].w * B[m + 2].y; };
        auto E2 = [&](int m) { return A[m + 2].w * B[m + 2].x - A[m + 2].y * B[m + 2].z; };
        const float2 d0 = d4neg2(f2(A[4].x, A[4].y), f2(A[3].x, A[3].y), f2(A[1].x, A[1].y), f2(A[0].x, A[0].y));
        const float2 d1 = d4neg2(f2(A[4].z, A[4].w), f2(A[3].z, A[3].w), f2(A[1].z, A[1].w), f2(A[0].z, A[0].w));
        d23 = d23 + D(c3, [&](int m) { return rho0c * A[m + 2].w; });
        T t = vp * (-c3 * d0.y);
        t = t * rinv;
        a_vr = a_vr + sinv * t;
        t = vp * (-c3 * d1.x);
        t = t * rinv;
        a_vt = a_vt + sinv * t;
        t = vp * (-c3 * d1.y);
        t = t * rinv;
        a_vp = a_vp + sinv * t;
        t = vp * D(c3, [&](int m) { return B[m + 2].w; });
        t = t * rinv;
        a_s1 = a_s1 + sinv * t;
        g3 = -c3 * d0.x;
        k1 = k1 - D(c3, [&](int m) { return B[m + 2].y; });
        k2 = D(c3, [&](int m) { return B[m + 2].x * sinv; }) - d_bpr;
        q1 = q1 - D(c3, [&](int m) { return E2(m); });
        q2 = D(c3, [&](int m) { return E1(m) * sinv; }) - q_e3r;
        if constexpr (DIVB != 0) e23 = e23 + D(c3, [&](int m) { return B[m + 2].z; });
    }
    const float4 src = tab.ti[TI_SRC * NIP + ii];
    const T gor0 = src.x, heat = src.y;
    // Mass conservation: -div(rho0 v)/Xi^2 (3_6/ModEquation.f90:50-61, ModSpherical_div :104-159)
    d23 = d23 * sinv;
    d23 = d23 * rinv;
    const T Rrho = -(xi2inv * (dA + d23));
    // Inertial force -(v.grad)v with curvature terms (3_6/ModSpherical.f90:281-343)
    T Rvr, Rvt, Rvp;
    {
        T tmp = -(vt * vt) - vp * vp;
        a_vr = a_vr + tmp * rinv;
        tmp = -(vp * vp);
        tmp = tmp * cot;
        tmp = tmp + vt * vr;
        a_vt = a_vt + tmp * rinv;
        tmp = vp * vt;
        tmp = tmp * cot;
        tmp = tmp + vp * vr;
        a_vp = a_vp + tmp * rinv;
        Rvr = -a_vr; Rvt = -a_vt; Rvp = -a_vp;
    }
    // Pressure gradient -grad(p1)/rho0 (3_6/ModEquation.f90:79-92)
    g2 = g2 * rinv;
    g3 = g3 * rinv;
    g3 = g3 * sinv;
    Rvr = Rvr - g1 * rho0inv;
    Rvt = Rvt - g2 * rho0inv;
    Rvp = Rvp - g3 * rho0inv;
    // Lorentz force (curl B) x B / rho0 (3_6/ModEquation.f90:97-116, curl :38-102)
    {
        k1 = k1 * rinv; k2 = k2 * rinv; k3 = k3 * rinv;
        k1 = k1 * sinv;
        const T x1 = k2 * bp - k3 * bt;
        const T x2 = k3 * br - k1 * bp;
        const T x3 = k1 * bt - k2 * br;
        Rvr = Rvr + x1 * rho0inv;
        Rvt = Rvt + x2 * rho0inv;
        Rvp = Rvp + x3 * rho0inv;
    }
    // Buoyancy -(g/rho0) rho1 (3_6/ModEquation.f90:121-127)
    Rvr = Rvr - gor0 * rho1;
    // Entropy advection and heating (3_6/ModEquation.f90:132-151)
    T Rs = -a_s1;
    Rs = Rs + heat;
    // Induction curl(v x B) (3_6/ModEquation.f90:154-162)
    q1 = q1 * rinv; q2 = q2 * rinv; q3 = q3 * rinv;
    q1 = q1 * sinv;
    T RBr = q1, RBt = q2, RBp = q3;

    // div-B control. GLM cleaning (3_6/ModDivB.f90:13-38), after the
    // equation terms as 3_6/ModAdvance.f90:82-84 orders it: dB += -grad(psi);
    // dpsi = -v_wave^2 div(B) - v_wave/h_LLL psi, v_wave from u^n. Powell
    // (3_5/ModEquation.f90:169-176): dB += -(div B) v.
    T divB = T(0);
    if constexpr (DIVB != 0) {   // ModSpherical_div of B (3_6/ModSpherical.f90:104-159)
        dB = dB * r2inv;
        e23 = e23 * sinv;
        e23 = e23 * rinv;
        divB = dB + e23;
    }
    if constexpr (DIVB == 2) {
        RBr = RBr - divB * vr;
        RBt = RBt - divB * vt;
        RBp = RBp - divB * vp;
    }
    if constexpr (DIVB == 1) {
        const T* P = static_cast<const T*>(psi.in) + (size_t)b * NCELL + cell;
        auto Q = [&](int di, int dj, int dk) -> T { return P[(ptrdiff_t)dk * PL + dj * NIP + di]; };
        // ModSpherical_Grad_f (3_6/ModSpherical.f90:201-239)
        const T h1 = D(c1, [&](int m) { return Q(m, 0, 0); });
        T h2 = D(c2, [&](int m) { return Q(0, m, 0); });
        h2 = h2 * rinv;
        T h3 = D(c3, [&](int m) { return Q(0, 0, m); });
        h3 = h3 * rinv;
        h3 = h3 * sinv;
        RBr = RBr - h1;
        RBt = RBt - h2;
        RBp = RBp - h3;
        // ModWaveSpeed_Dynamo (3_6/ModWaveSpeed.f90:8-27) and h_LLL
        // (3_6/ModBlock.f90:416-425) at this cell, as the CFL pass forms them
        T w = tab.ti[TI_R * NIP + ii].w + sqrt(ua.y * ua.y + ua.z * ua.z + ua.w * ua.w);
        w = w + sqrt(ub.x * ub.x + ub.y * ub.y + ub.z * ub.z) / sqrt(rho0c);
        const T rcell = tab.ti[TI_R * NIP + ii].z;
        const T h = fmin(fmin(tab.gs[GS_DXI], rcell * tab.gs[GS_DXJ]), rcell * th.x * tab.gs[GS_DXK]);
        const T Rpsi = -(w * w * divB) - w / h * Q(0, 0, 0);
        const size_t pc = (size_t)b * NCELL + cell;
        const T pn = static_cast<const T*>(psi.un)[pc];
        static_cast<T*>(psi.out)[pc] = fmaf(dtk, Rpsi, pn);
    }

    // stage update
    const T R[NV] = {Rrho, Rvr, Rvt, Rvp, RBr, RBt, RBp, Rs};
    T u0s[NV];
    split(ua, ub, u0s);
    if (final_stage) {
        // u^{n+1} = u^n + dt*R with u^n and u^{n+1} compensated
        auto dt2 = [&](int v) { return __fmul2_rn(f2(dtk), f2(R[v], R[v + 1])); };
        ff_add4(u0s, q8.x, {dt2(0), dt2(2)}, o);
        ff_add4(u0s + 4, q8.y, {dt2(4), dt2(6)}, o + 4);
    } else {
#pragma unroll
        for (int v = 0; v < NV; ++v) o[v] = fmaf(dtk, R[v], u0s[v]);
    }
}

// Chunks of KPAR planes, a thread per cell: 8^3 blocks. Planes [ch0, ch1) x KPAR of
// block b. The planes of the next chunk, copied during this one, get their
// boundary condition and p1 at its end, so a chunk is one barrier.
// 442k cells (864 blocks): 36.3 -> 34 us per stage.
template <int NI, int NJ, int NK, int KPAR>
struct QShape : Shape<float, NI, NJ, NK, KPAR> {
    using B = Shape<float, NI, NJ, NK, KPAR>;
    // shared memory: mbarriers | tile[2][W][PL] of 16 bytes | rho1[W][PLI] | tables
    static constexpr size_t off_tile = 16;
    static constexpr size_t off_rho = off_tile + (size_t)2 * B::W * B::PL * 16;
    static constexpr size_t off_tab = off_rho + (size_t)B::W * B::PLI * 4;
    static constexpr size_t smem = off_tab + StageTables::bytes<B::NIP, B::NJP>();
    static_assert(off_tab % 16 == 0 && smem <= 232448, "16-byte tables; 227 KB of opt-in shared memory per CTA");
    // as many CTAs per SM as the shared memory holds (228 KB, 1 KB of it reserved
    // and about 0.2 KB static per CTA): the registers must fit them too
    static constexpr int by_smem = (int)(233472 / (smem + 1280));
    static constexpr int reg_cap = 2048 / B::NT;
    static constexpr int min_blocks = by_smem < reg_cap ? by_smem : reg_cap;
};
template <int NI, int NJ, int NK, int KPAR, int DIVB>
__device__ __forceinline__ void stage_chunks(int b, int ch0, int ch1, const float* in, const float* un, float* out,
                                             int8_t* ulo, const PushTable& push, const DivBArgs& psi, const Geometry& g,
                                             StepScalars* sc, int stage, int bc_writeback) {
    using S = QShape<NI, NJ, NK, KPAR>;
    constexpr int NIP = S::NIP, PL = S::PL, W = S::W, NCELL = S::NCELL, HC = 4 * (NI + NJ);
    extern __shared__ __align__(128) unsigned char smem[];
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem);
    float4* tile = reinterpret_cast<float4*>(smem + S::off_tile);   // [2][W][PL]
    float* rho = reinterpret_cast<float*>(smem + S::off_rho);       // [W][PLI]
    StageTables tab(smem + S::off_tab, NIP, S::NJP);
    const int fl = g.flags[b];
    const float* blk_in = in + (size_t)b * NV * NCELL;
    float* wb = bc_writeback ? const_cast<float*>(blk_in) : nullptr;
    __shared__ PushBlock pb;
    load_push_block(push, b, &pb);
    const int tid = threadIdx.x, nch = ch1 - ch0;
    const bool issuer = tid == S::NT - 32;   // requests the copies (the first warp loads the tables)
    step_go();
    if (issuer) {
        mbar_init(&bars[0], 1);
        mbar_init(&bars[1], 1);
        fence_mbar_init();
        step_wait();
        issue_quads<S>(blk_in, tile, ch0 * KPAR, ch0 * KPAR + KPAR + 4, 0, &bars[0]);
    }
    tab.load(g, b, NIP, S::NJP, S::NT);
    step_wait();
    __syncthreads();   // barriers and tables are used by every thread below

    int i, j, kq;
    cell_of_thread<NI, NJ>(tid, i, j, kq);
    const int ii = i + 2, jj = j + 2, c0 = jj * NIP + ii;
    const float dtk = sc->dt_stage_f[stage - 1];
    const int polls = sc->wait_polls;
    const bool final_stage = ulo != nullptr && stage == 4;
    int late = 0;   // a wait of this thread for a chunk's planes ran out

    // planes [lo, lo + np), just copied: boundary condition, p1 in rho1's place
    auto prepare = [&](int lo, int np) {
        if (fl & 6) {   // radial boundary block (uniform over the CTA)
            apply_bc_quads<S>(tile, lo, lo + np, 0, fl, wb, S::NT);
            __syncthreads();
        }
        auto p1_at = [&](int slot, int c, int ic) {
            float4* a = tile + slot * PL + c;
            const float r1 = a->x;
            a->x = tab.p1(ic, r1, tile[(W + slot) * PL + c].w);
            return r1;
        };
        for (int q = kq; q < np; q += KPAR) {
            const int slot = (lo + q) % W;
            rho[slot * S::PLI + j * NI + i] = p1_at(slot, c0, ii);
        }
        for (int x = tid; x < np * HC; x += S::NT) {
            int c, ic;
            reached_ghost<NI, NJ, NIP>(x % HC, c, ic);
            p1_at((lo + x / HC) % W, c, ic);
        }
        fence_proxy_async();   // order these generic writes before later bulk copies into the slots
    };
    late |= mbar_wait(&bars[0], 0u, polls) ? 0 : 1;
    prepare(ch0 * KPAR, KPAR + 4);
    for (int n = 0; n < nch; ++n) {
        const int ch = ch0 + n, next = (ch + 1) * KPAR + 4;   // next: first plane new to the next chunk
        // this chunk's planes are complete and the slots of the next one's are
        // free. A wait that ran out does not leave its chunk (its barriers must be
        // reached by every thread): whatever the slots held was computed on, the
        // step is flagged here and its results are discarded
        if (__syncthreads_or(late)) {
            copy_wait_abort(sc, bars, n, n);
            return;
        }
        if (issuer && n + 1 < nch) issue_quads<S>(blk_in, tile, next, next + KPAR, 0, &bars[(n + 1) & 1]);
        const int kp = ch * KPAR + kq + 2;
        const size_t cell = (size_t)kp * PL + c0;
        int sl[5];
#pragma unroll
        for (int d = 0; d < 5; ++d) sl[d] = (kp + d - 2) % W * PL + c0;
        float4 ua, ub;
        int2* ql = reinterpret_cast<int2*>(ulo + ((size_t)b * S::NINT + ((size_t)(kp - 2) * NJ + j) * NI + i) * NV);
        int2 q8 = make_int2(0, 0);
        if (final_stage) q8 = *ql;
        float o[NV];
        stage_cell<NIP, PL, NCELL, DIVB>(
            tab, b, ii, jj, cell, tile[sl[2]], tile[W * PL + sl[2]], rho[kp % W * S::PLI + j * NI + i],
            [&](int h, int m) { return tile[h * W * PL + sl[2] + m]; },
            [&](int h, int m) { return tile[h * W * PL + sl[2] + m * NIP]; },
            [&](int h, int m) { return tile[h * W * PL + sl[m + 2]]; },
            [&](int m) { return tab.ti[TI_R * NIP + ii + m]; }, [&](int m) { return tab.tj[jj + m].x; },
            // u^n (at stage 1 the input: in L2), loaded here so that the latency
            // overlaps the k derivatives (earlier, the registers spill)
            [&]() {
                ua = quads(un)[quad(b, 0, NCELL) + cell];
                ub = quads(un)[quad(b, 1, NCELL) + cell];
            },
            ua, ub, q8, final_stage, dtk, psi, o);
        if (final_stage) *ql = q8;
        quads(out)[quad(b, 0, NCELL) + cell] = f4(o);
        quads(out)[quad(b, 1, NCELL) + cell] = f4(o + 4);
        if (push.tgt != nullptr) push_quads<S>(out, pb, ii, jj, kp, o);
        if (n + 1 < nch) {
            late |= mbar_wait(&bars[(n + 1) & 1], (uint32_t)(((n + 1) >> 1) & 1), polls) ? 0 : 1;
            prepare(next, KPAR);
        }
    }
    // every copy was waited for before the last chunk's barrier
}

// The march along k: 16^3 blocks, planes [ka, kb) of block b, one thread per (i, j)
// column (256 threads, two CTAs per SM). Planes arrive by bulk copy into a ring of
// 7 slots, an mbarrier each; a plane's boundary condition and p1 (each thread its
// own column, the first 128 a ghost cell as well) are formed one plane before its
// first use, as the neighbour kp + 2, so a plane is one barrier. u^n is read a
// plane ahead, and what depends on the column alone (the neighbours' radial and
// theta factors) stays in registers.
//
// What bounds it: the shared-memory reads (70% of that pipe's cycles) and, with
// 16 warps per SM, the issue (56%). A register window along k spares 8 of the 26
// reads and costs as much in moves (763 us), unrolled by five to avoid those it
// loses to the instruction cache (823); chunks of two planes with 64 registers a
// thread spill (1,006). 21.2M cells: 877 -> 685 us per stage.
template <int NI, int NJ, int NK>
struct SMarch {
    static constexpr int NIP = NI + 4, NJP = NJ + 4, NKP = NK + 4, PL = NIP * NJP, NCELL = PL * NKP, PLI = NI * NJ, NINT = PLI * NK;
    static constexpr int NT = NI * NJ, W = 7;
    // shared memory: mbarriers | tile[2][W][PL] of 16 bytes | rho1[4][PLI] | tables
    static constexpr size_t off_tile = 128, off_rho = off_tile + (size_t)2 * W * PL * 16, off_tab = off_rho + (size_t)4 * PLI * 4;
    static constexpr size_t smem = off_tab + StageTables::bytes<NIP, NJP>();
    static_assert(2 * (smem + 1280) <= 233472, "two CTAs per SM");
};
template <int NI, int NJ, int NK, int DIVB>
__device__ __forceinline__ void stage_march(int b, int ka, int kb, const float* in, const float* un, float* out,
                                            int8_t* ulo, const PushTable& push, const DivBArgs& psi, const Geometry& g,
                                            StepScalars* sc, int stage, int bc_writeback) {
    using S = SMarch<NI, NJ, NK>;
    constexpr int NIP = S::NIP, PL = S::PL, W = S::W, NCELL = S::NCELL, HC = 4 * (NI + NJ);
    static_assert(NI == 16 && HC <= S::NT, "rows of 16 cells: one half-warp per row; a plane's ghost cells in one pass");
    extern __shared__ __align__(128) unsigned char smem[];
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem);   // plane p's: p - p0 counted from the first plane, modulo W
    float4* tile = reinterpret_cast<float4*>(smem + S::off_tile);   // [2][W][PL]
    StageTables tab(smem + S::off_tab, NIP, S::NJP);
    const int fl = g.flags[b];
    const float* blk_in = in + (size_t)b * NV * NCELL;
    float* wb = bc_writeback ? const_cast<float*>(blk_in) : nullptr;
    __shared__ PushBlock pb;
    load_push_block(push, b, &pb);
    const int tid = threadIdx.x, p0 = ka - 2, pe = kb + 2;   // planes [p0, pe) are read
    const bool issuer = tid == S::NT - 32;                   // requests the copies (the first warp loads the tables)
    int issued = p0;                                         // by the issuer: planes [p0, issued)
    auto issue = [&](int last) {
        for (; issued <= last && issued < pe; ++issued)
            issue_quads<S>(blk_in, tile, issued, issued + 1, p0, &bars[(issued - p0) % W]);
    };
    step_go();
    if (issuer) {
        for (int q = 0; q < W; ++q) mbar_init(&bars[q], 1);
        fence_mbar_init();
        step_wait();
        issue(p0 + W - 1);
    }
    tab.load(g, b, NIP, S::NJP, S::NT);
    step_wait();
    __syncthreads();   // barriers and tables are used by every thread below
    const int i = tid % NI, j = tid / NI, ii = i + 2, jj = j + 2, c0 = jj * NIP + ii;
    const float dtk = sc->dt_stage_f[stage - 1];
    const int polls = sc->wait_polls;
    const bool final_stage = ulo != nullptr && stage == 4;
    // a wait of this thread ran out: it computes on whatever the slots hold (and
    // waits no more), the step is flagged and its results are discarded
    int late = 0;
    auto arrived = [&](int p) {
        late |= mbar_wait(&bars[(p - p0) % W], (uint32_t)(((p - p0) / W) & 1), late ? 1 : polls) ? 0 : 1;
    };
    int gc, gic;   // this thread's ghost cell of a plane (the first HC threads)
    reached_ghost<NI, NJ, NIP>(tid % HC, gc, gic);
    float* rho = reinterpret_cast<float*>(smem + S::off_rho) + tid;   // its rho1 of planes kp .. kp + 3, plane p's at p % 4
    // plane p in slot s, just copied: boundary condition, p1 in rho1's place
    auto prepare = [&](int p, int s) {
        if (fl & 6) {   // radial boundary block (uniform over the CTA)
            apply_bc_quads<S>(tile, p, p + 1, p0, fl, wb, S::NT);
            __syncthreads();
        }
        float4* a = tile + s * PL + c0;
        const float r1 = a->x;
        rho[p % 4 * S::PLI] = r1;
        a->x = tab.p1(ii, r1, a[W * PL].w);
        if (tid < HC) {
            a = tile + s * PL + gc;
            a->x = tab.p1(gic, a->x, a[W * PL].w);
        }
        fence_proxy_async();   // order these generic writes before later bulk copies into the slot
    };
#pragma unroll
    for (int m = 0; m < 5; ++m) {
        arrived(p0 + m);
        prepare(p0 + m, m);
    }
    __syncthreads();
    const float4* un_b = quads(un) + quad(b, 0, NCELL);
    float4* out_b = quads(out) + quad(b, 0, NCELL);
    int2* lo_b = reinterpret_cast<int2*>(ulo + ((size_t)b * S::NINT + tid) * NV);
    // the neighbours' radial and theta factors
    float4 gr[5];
    float sn[5];
#pragma unroll
    for (int m = 0; m < 5; ++m) { gr[m] = tab.ti[TI_R * NIP + ii + m - 2]; sn[m] = tab.tj[jj + m - 2].x; }
    float4 na = un_b[ka * PL + c0], nb = un_b[NCELL + ka * PL + c0];
    int s = 2;   // slot of plane kp
    for (int kp = ka; kp < kb; ++kp) {
        // everyone is through with the cells of plane kp - 1: plane kp - 3's slot is free
        if (issuer && !late) issue(kp + W - 3);
        const int cell = kp * PL + c0;
        int2* ql = lo_b + (kp - 2) * S::PLI;
        const float4 ua = na, ub = nb;   // u^n (at stage 1 the input itself, in L2)
        if (kp + 1 < kb) { na = un_b[cell + PL]; nb = un_b[NCELL + cell + PL]; }
        int2 q8 = make_int2(0, 0);
        if (final_stage) q8 = *ql;
        const float4* a = tile + s * PL + c0;
        int sk[5];
#pragma unroll
        for (int d = 0; d < 5; ++d) { const int z = s + d - 2; sk[d] = (z < 0 ? z + W : z >= W ? z - W : z) * PL + c0; }
        float o[NV];
        stage_cell<NIP, PL, NCELL, DIVB>(
            tab, b, ii, jj, cell, a[0], a[W * PL], rho[kp % 4 * S::PLI], [&](int h, int m) { return a[h * W * PL + m]; },
            [&](int h, int m) { return a[h * W * PL + m * NIP]; }, [&](int h, int m) { return tile[h * W * PL + sk[m + 2]]; },
            [&](int m) { return make_float4(gr[m + 2].x, gr[m + 2].y, gr[m + 2].z, 0.f); }, [&](int m) { return sn[m + 2]; },
            []() {}, ua, ub, q8, final_stage, dtk, psi, o);
        if (final_stage) *ql = q8;
        out_b[cell] = f4(o);
        out_b[NCELL + cell] = f4(o + 4);
        if (push.tgt != nullptr) push_quads<S>(out, pb, ii, jj, kp, o);
        if (kp + 1 < kb) {
            arrived(kp + 3);
            prepare(kp + 3, s + 3 < W ? s + 3 : s + 3 - W);
            s = s + 1 < W ? s + 1 : 0;
            __syncthreads();
        }
    }
    if (__syncthreads_or(late) && issuer) {
        atomicOr(&sc->nan_flag, 2);
        for (int p = issued - p0 < W ? p0 : issued - W; p < issued; ++p)   // the copies in flight
            mbar_wait(&bars[(p - p0) % W], (uint32_t)(((p - p0) / W) & 1), kWaitPolls);
    }
    if (issuer)
        for (int q = 0; q < W; ++q) mbar_inval(&bars[q]);
}
// split CTAs per block, each a run of planes
template <int NI, int NJ, int NK, int KPAR, int DIVB>
__global__ void __launch_bounds__(NI* NJ* KPAR, (QShape<NI, NJ, NK, KPAR>::min_blocks))
k_stage_chunks(const float* in, const float* un, float* out, int8_t* ulo, PushTable push, DivBArgs psi, Geometry g,
               StepScalars* sc, int stage, int bc_writeback, int split) {
    const int b = blockIdx.x / split, part = blockIdx.x - b * split, n = NK / KPAR / split;
    stage_chunks<NI, NJ, NK, KPAR, DIVB>(b, part * n, (part + 1) * n, in, un, out, ulo, push, psi, g, sc, stage, bc_writeback);
}
template <int NI, int NJ, int NK, int DIVB>
__global__ void __launch_bounds__(NI* NJ, 2)
k_stage_march(const float* in, const float* un, float* out, int8_t* ulo, PushTable push, DivBArgs psi, Geometry g,
              StepScalars* sc, int stage, int bc_writeback, int split) {
    const int b = blockIdx.x / split, part = blockIdx.x - b * split, n = NK / split;
    stage_march<NI, NJ, NK, DIVB>(b, 2 + part * n, 2 + (part + 1) * n, in, un, out, ulo, push, psi, g, sc, stage, bc_writeback);
}

// ---------------------------------------------------------------------------
// FP32 artificial diffusion (3_6/ModDiffusion.f90:9-150, h = 2) and the update
// u += 0.5*dt*R (3_6/ModAdvance.f90:101-108) of 8^3 blocks, a chunk of KPAR
// planes at a time (a thread per cell). Each face flux is formed once per chunk
// into shared memory: i and j faces of the chunk's planes, and the k faces in a
// ring of KPAR+1 face planes (the last face of a chunk is the first of the
// next). Then each cell sums (F_left - F_right)/den over the three directions,
// in the reference's order. Out of place (out != u) the kernel also writes the
// regular ghost faces of its neighbours in `out` and copies the radial
// physical-boundary ghost columns (set by the boundary condition at stage 1);
// cfl_next: the outputs are the next step's u^n, so it forms the next step's CFL
// minimum and NaN flag from them (k_cfl's formula, cfl_ratio_f).
template <int NI, int NJ, int NK, int KPAR>
struct DShape : Shape<float, NI, NJ, NK, KPAR> {
    using B = Shape<float, NI, NJ, NK, KPAR>;
    static constexpr int NT = NI * NJ * KPAR;
    static constexpr int KS = KPAR + 1;                  // k-face ring slots
    static constexpr int FIP = NI + 1;                   // i-face row pitch
    static constexpr int NFI = NV * KPAR * NJ * FIP;
    static constexpr int NFJ = NV * KPAR * (NJ + 1) * NI;
    static constexpr int NFK = KS * NV * NJ * NI;
    // shared memory: mbarriers | tile[2][W][PL] of 16 bytes | FI | FJ | FK | gi | gj | gs
    static constexpr size_t off_tile = 16;
    static constexpr size_t off_fi = off_tile + (size_t)NV * B::W * B::PL * 4;
    static constexpr size_t off_fj = off_fi + (size_t)NFI * 4;
    static constexpr size_t off_fk = off_fj + (size_t)NFJ * 4;
    static constexpr size_t off_gi = off_fk + (size_t)NFK * 4;
    static constexpr size_t off_gj = off_gi + (size_t)GI_COUNT * B::NIP * 4;
    static constexpr size_t off_gs = off_gj + (size_t)GJ_COUNT * B::NJP * 4;
    static constexpr size_t smem = off_gs + GS_COUNT * 4;
    static_assert(smem <= 232448, "227 KB of opt-in shared memory per CTA");
    static constexpr int by_smem = (int)(233472 / (smem + 1024));
    static constexpr int reg_cap = 2048 / NT;
    static constexpr int min_blocks = by_smem < 2 ? 1 : (by_smem < reg_cap ? by_smem : (reg_cap < 1 ? 1 : reg_cap));
};

// radial boundary ghost columns of planes [plo, phi), tile -> out
template <class S>
__device__ __forceinline__ void copy_bc_columns(const float4* tile, int p0, float* out, int b, int fl, int plo, int phi, int nt) {
    constexpr int NI = S::NIP - 4;
    const int total = (phi - plo) * S::NJP * 8;
    for (int x = threadIdx.x; x < total; x += nt) {
        const int c4 = x & 3, h = (x >> 2) & 1, r = x >> 3, y = r % S::NJP, z = plo + r / S::NJP;
        if (!((c4 < 2) ? (fl & 4) : (fl & 2))) continue;
        const int xi = c4 < 2 ? c4 : NI + c4;   // 0, 1 (bottom) or NI+2, NI+3 (top)
        quads(out)[quad(b, h, S::NCELL) + (size_t)z * S::PL + y * S::NIP + xi] =
            tile[((size_t)h * S::W + (z - p0) % S::W) * S::PL + y * S::NIP + xi];
    }
}

template <int NI, int NJ, int NK, int KPAR>
__global__ void __launch_bounds__(DShape<NI, NJ, NK, KPAR>::NT, (DShape<NI, NJ, NK, KPAR>::min_blocks))
k_diffusion_quads(const float* u, float* out, int8_t* ulo, PushTable push, Geometry g, StepScalars* sc, int cfl_next) {
    using S = DShape<NI, NJ, NK, KPAR>;
    constexpr int NIP = S::NIP, PL = S::PL, W = S::W, NCELL = S::NCELL, KS = S::KS;
    extern __shared__ __align__(128) unsigned char smem[];
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem);
    float4* tile = reinterpret_cast<float4*>(smem + S::off_tile);
    float* FI = reinterpret_cast<float*>(smem + S::off_fi);
    float* FJ = reinterpret_cast<float*>(smem + S::off_fj);
    float* FK = reinterpret_cast<float*>(smem + S::off_fk);
    float* gi = reinterpret_cast<float*>(smem + S::off_gi);
    float* gj = reinterpret_cast<float*>(smem + S::off_gj);
    float* gs = reinterpret_cast<float*>(smem + S::off_gs);
    const int b = blockIdx.x;
    const float* blk = u + (size_t)b * NV * NCELL;
    const int flb = g.flags[b];
    const bool copy_bc = out != u && (flb & 6);
    __shared__ PushBlock pb;
    load_push_block(push, b, &pb);
    const bool issuer = threadIdx.x == S::NT - 32;   // requests the copies
    step_go();
    if (issuer) {
        mbar_init(&bars[0], 1);
        mbar_init(&bars[1], 1);
        fence_mbar_init();
        step_wait();
        issue_quads<S>(blk, tile, 0, KPAR + 4, 0, &bars[0]);
    }
    // the int8 corrections of u^n are read with plain loads: warm L2 one chunk ahead
    auto prefetch_lo = [&](int kp_first) {
        if (ulo != nullptr && threadIdx.x == 0)
            prefetch_l2(ulo + ((size_t)b * S::NINT + (size_t)(kp_first - 2) * S::PLI) * NV, KPAR * S::PLI * NV);
    };
    load_geometry<float, S>(g, b, gi, gj, gs, nullptr);
    step_wait();
    prefetch_lo(2);
    __syncthreads();   // barriers and tables are used by every thread below
    const int tid = threadIdx.x;
    const float* GCS = gi + GI_CS * NIP;
    const int kq = tid / (NI * NJ), i = tid % NI, j = tid / NI % NJ;
    const int ii = i + 2, jj = j + 2;
    const float rc = gi[GI_R * NIP + ii], cs = GCS[ii];
    const float den[3] = {gs[GS_DXI], gs[GS_DXJ] * rc, gs[GS_DXK] * rc * gj[GJ_SIN * S::NJP + jj]};
    const float dinv[3] = {1.f / den[0], 1.f / den[1], 1.f / den[2]};
    const float hdt_f = sc->dt_half_f;
    float wmax = 0.f;   // the largest wave speed of this thread's cells, for the next step's CFL minimum
    int cnan = 0;
    const float srho = __fsqrt_rn(gi[GI_RHO0 * NIP + ii]), srho_inv = __frcp_rn(srho);
    constexpr int nchunk = NK / KPAR;
    const int polls = sc->wait_polls;
    int late = 0;   // a wait of this thread for a chunk's planes ran out
    // variable v of padded cell c in a plane's slot
    auto val = [&](int v, int slot, int c) -> float {
        return reinterpret_cast<const float*>(tile + ((v >> 2) * W + slot) * PL + c)[v & 3];
    };
    for (int ch = 0; ch < nchunk; ++ch) {
        const int k0 = 1 + ch * KPAR;
        const int hi = k0 + KPAR + 3;
        // ring slots and face arrays of the previous chunk are free; a wait of
        // chunk ch-1 that ran out ends the CTA here (chunks ch-1 and ch in flight)
        if (__syncthreads_or(late)) {
            copy_wait_abort(sc, bars, ch - 1, ch);
            return;
        }
        if (issuer && ch + 1 < nchunk) issue_quads<S>(blk, tile, hi, hi + KPAR, 0, &bars[(ch + 1) & 1]);
        if (ch + 1 < nchunk) prefetch_lo(k0 + KPAR + 1);
        const int kp0 = k0 + 1, kp = kp0 + kq;   // padded index of the chunk's first plane, this cell's plane
        // this thread's int8 corrections, loaded now so that their latency
        // overlaps the copy wait and the face phase
        int2* ql = reinterpret_cast<int2*>(ulo + ((size_t)b * S::NINT + ((size_t)(kp - 2) * NJ + j) * NI + i) * NV);
        int2 q8 = make_int2(0, 0);
        if (ulo != nullptr) q8 = *ql;
        // as in the stage kernel: a wait that runs out finishes the chunk on
        // whatever the slots hold; the step is flagged and discarded
        late |= mbar_wait(&bars[ch & 1], (uint32_t)((ch >> 1) & 1), polls) ? 0 : 1;
        if (copy_bc)   // the planes new to this chunk
            copy_bc_columns<S>(tile, 0, out, b, flb, ch == 0 ? 0 : k0 + 3, k0 + KPAR + 3, S::NT);
        // slots of planes kp-1 .. kp+2
        int so[4];
#pragma unroll
        for (int d = 0; d < 4; ++d) so[d] = (kp + d - 1) % W * PL;
        const int c0 = jj * NIP + ii;
        const float4 ca = tile[so[1] + c0], cb = tile[W * PL + so[1] + c0];   // this cell
        // this cell's left i and j faces and right k face
        {
            const float4* tA = tile + c0;
            const float cci = face_speed(tA[so[1] - 1].y, GCS[ii - 1], ca.y, cs);
            const float ccj = face_speed(tA[so[1] - NIP].z, cs, ca.z, cs);
            const float cck = face_speed(ca.w, cs, tA[so[2]].w, cs);
            float* fkw = FK + (size_t)((kp - 1) % KS) * NV * NJ * NI + j * NI + i;
            auto lo2 = [](const float4& x) { return f2(x.x, x.y); };
            auto hi2 = [](const float4& x) { return f2(x.z, x.w); };
            // the fluxes of a half's four values through a face: arrays pitch apart
            auto face4 = [&](const float4& fm, const float4& fl, const float4& fr, const float4& fp, float cc, float* to, int pitch) {
                const float2 a = face_flux2(lo2(fl), lo2(fr), half_slope2(lo2(fm), lo2(fl), lo2(fr)), half_slope2(lo2(fl), lo2(fr), lo2(fp)), f2(cc));
                const float2 b = face_flux2(hi2(fl), hi2(fr), half_slope2(hi2(fm), hi2(fl), hi2(fr)), half_slope2(hi2(fl), hi2(fr), hi2(fp)), f2(cc));
                to[0] = a.x; to[pitch] = a.y; to[2 * pitch] = b.x; to[3 * pitch] = b.y;
            };
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float4* t = tile + h * W * PL + c0;
                const float4 z = t[so[1]];
                face4(t[so[1] - 2], t[so[1] - 1], z, t[so[1] + 1], cci, FI + ((4 * h * KPAR + kq) * NJ + j) * S::FIP + i, KPAR * NJ * S::FIP);
                face4(t[so[1] - 2 * NIP], t[so[1] - NIP], z, t[so[1] + NIP], ccj, FJ + ((4 * h * KPAR + kq) * (NJ + 1) + j) * NI + i,
                      KPAR * (NJ + 1) * NI);
                face4(t[so[0]], z, t[so[2]], t[so[3]], cck, fkw + 4 * h * NJ * NI, NJ * NI);
            }
        }
        // one value's flux from the four around the face
        auto face1 = [&](float fm, float fl, float fr, float fp, float cc) {
            return face_flux(fl, fr, half_slope(fm, fl, fr), half_slope(fl, fr, fp), cc);
        };
        // the right faces of the last cells of i rows and j columns
        constexpr int NXI = NV * KPAR * NJ, NXJ = NV * KPAR * NI;
        for (int x = tid; x < NXI + NXJ; x += S::NT) {
            const bool on_i = x < NXI;
            const int y = on_i ? x : x - NXI, n = on_i ? NJ : NI;
            const int r = y % n + 2, q = (y / n) % KPAR, v = y / (n * KPAR), slot = (kp0 + q) % W;
            const int c = on_i ? r * NIP + NI + 1 : (NJ + 1) * NIP + r, st = on_i ? 1 : NIP;   // last interior cell
            const int vd = on_i ? V_VR : V_VT;
            const float cc = face_speed(val(vd, slot, c), GCS[on_i ? NI + 1 : r], val(vd, slot, c + st), GCS[on_i ? NI + 2 : r]);
            const float f = face1(val(v, slot, c - st), val(v, slot, c), val(v, slot, c + st), val(v, slot, c + 2 * st), cc);
            if (on_i) FI[((v * KPAR + q) * NJ + (r - 2)) * S::FIP + NI] = f;
            else FJ[((v * KPAR + q) * (NJ + 1) + NJ) * NI + (r - 2)] = f;
        }
        // first chunk: the k faces below the first plane (between padded planes 1 and 2)
        if (ch == 0) {
            for (int x = tid; x < NV * NJ * NI; x += S::NT) {
                const int xx = x % NI + 2, y = (x / NI) % NJ + 2, v = x / (NI * NJ), c = y * NIP + xx;
                const float cc = face_speed(val(V_VP, 1, c), GCS[xx], val(V_VP, 2, c), GCS[xx]);
                FK[(v * NJ + (y - 2)) * NI + (xx - 2)] = face1(val(v, 0, c), val(v, 1, c), val(v, 2, c), val(v, 3, c), cc);
            }
        }
        __syncthreads();
        const size_t cell = (size_t)kp * PL + c0;
        const float* fk_l = FK + (size_t)((kp - 2) % KS) * NV * NJ * NI + j * NI + i;
        const float* fk_r = FK + (size_t)((kp - 1) % KS) * NV * NJ * NI + j * NI + i;
        float o[NV], u0[NV], R[NV];
        split(ca, cb, u0);
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            const float* fi = FI + ((v * KPAR + kq) * NJ + j) * S::FIP + i;
            const float* fj = FJ + ((v * KPAR + kq) * (NJ + 1) + j) * NI + i;
            R[v] = __fmul_rn(fi[0] - fi[1], dinv[0]);
            R[v] = __fmaf_rn(fj[0] - fj[NI], dinv[1], R[v]);
            R[v] = __fmaf_rn(fk_l[v * NJ * NI] - fk_r[v * NJ * NI], dinv[2], R[v]);
        }
        if (ulo != nullptr) {
            auto dt2 = [&](int v) { return __fmul2_rn(f2(hdt_f), f2(R[v], R[v + 1])); };
            ff_add4(u0, q8.x, {dt2(0), dt2(2)}, o);
            ff_add4(u0 + 4, q8.y, {dt2(4), dt2(6)}, o + 4);
            *ql = q8;
        } else {
#pragma unroll
            for (int v = 0; v < NV; ++v) o[v] = __fmaf_rn(hdt_f, R[v], u0[v]);
        }
        quads(out)[quad(b, 0, NCELL) + cell] = f4(o);
        quads(out)[quad(b, 1, NCELL) + cell] = f4(o + 4);
        if (push.tgt != nullptr) push_quads<S>(out, pb, ii, jj, kp, o);
        if (cfl_next) {   // uniform over the CTA
#pragma unroll
            for (int v = 0; v < NV; ++v) cnan |= (o[v] != o[v]);
            wmax = fmaxf(wmax, cfl_speed(cfl_sq3(o[V_VR], o[V_VT], o[V_VP]), cfl_sq3(o[V_BR], o[V_BT], o[V_BP]), cs, srho, srho_inv));
        }
    }
    if (__syncthreads_or(late)) {
        copy_wait_abort(sc, bars, nchunk - 1, nchunk - 1);
        return;
    }
    if (cfl_next) cfl_commit(cfl_column(wmax, rc, gj[GJ_SIN * S::NJP + jj], gs[GS_DXI], gs[GS_DXJ], gs[GS_DXK]), cnan, sc);
}

// ---------------------------------------------------------------------------
// FP32 artificial diffusion of one 16^3 block, or of planes [ka, kb) of it, as a
// march along k (same arguments and results as k_diffusion_quads).
//
// One thread per (i, j) column of the block (256 threads), marching k over the
// 16 interior planes. Along k everything stays in registers: the column's
// values at planes kp and kp+1, its k slope at kp and the flux through the
// face below kp; per plane the thread reads one new value per variable (plane
// kp+2, from the ring), forms one k slope and one k face. Across the plane,
// every i and j slope is formed once (phase A, into shared memory, ghost
// columns and rows by the same threads), then every i and j face flux once
// (phase B), then each cell sums its six faces and updates (phase C). Per
// cell and variable that is 3 slopes and 3 fluxes, the minimum; the face
// fluxes are the same functions of the same values as k_diffusion_quads', summed
// in the same order. The arithmetic runs on pairs of variables (packed FP32
// instructions, above), and the slope and face arrays hold the pairs side by
// side, so their shared-memory accesses are 64-bit; a cell's values come from
// the ring four at a time (128-bit).
//
// Planes arrive by bulk copy into a ring of 5 slots, one mbarrier each: the
// column window needs planes kp..kp+2, and the slot of plane kp is refilled
// with plane kp+5 once phase B of plane kp has passed its barrier (planes
// kp+3 and kp+4 are in flight meanwhile). A warp takes rows j and j+4
// (half-warps of 16 cells), so a half-warp holds one row, as the pushed
// radial faces need.
//
// What bounds it is the issue (16 warps per SM, 128 registers a thread): 1,139 warp
// instructions per 32 cells, issued in 58% of the cycles. 21.2M cells: 1,229 ->
// 1,019 us; 442k cells with split blocks: 60 -> 34 us. Two threads per column with
// 64 registers each: 1,367 us (of 1,135 then).
template <int NI, int NJ, int NK>
struct MShape {
    static constexpr int NG = 2, NIP = NI + 4, NJP = NJ + 4, NKP = NK + 4;
    static constexpr int PL = NIP * NJP, NCELL = PL * NKP;
    static constexpr int NT = NI * NJ;
    static constexpr int W = 5;                          // plane ring slots
    static constexpr int PLI = NI * NJ, NINT = PLI * NK;
    static constexpr int NP = NV / 2;                    // variable pairs
    static constexpr int P = 20;                         // row pitch (pairs) of the slope and face arrays
    // per pair (float2): SI[NJ][P] slopes along i of cells i = -1..NI at i + 1;
    // SJ[NJ + 2][P] slopes along j of rows j = -1..NJ at row j + 1;
    // FI[NJ][P] fluxes through faces i - 1/2, i = 0..NI; FJ[NJ + 1][P] likewise along j
    static constexpr int NSI = NJ * P, NSJ = (NJ + 2) * P, NFI = NJ * P, NFJ = (NJ + 1) * P;
    // shared memory: mbarriers | tile[2][W][PL] of 16 bytes | SI | SJ | FI | FJ | gi | gj | gs
    static constexpr size_t off_tile = 64;
    static constexpr size_t off_si = off_tile + (size_t)NV * W * PL * 4;
    static constexpr size_t off_sj = off_si + (size_t)NP * NSI * 8;
    static constexpr size_t off_fi = off_sj + (size_t)NP * NSJ * 8;
    static constexpr size_t off_fj = off_fi + (size_t)NP * NFI * 8;
    static constexpr size_t off_gi = off_fj + (size_t)NP * NFJ * 8;
    static constexpr size_t off_gj = off_gi + (size_t)GI_COUNT * NIP * 4;
    static constexpr size_t off_gs = off_gj + (size_t)GJ_COUNT * NJP * 4;
    static constexpr size_t smem = off_gs + GS_COUNT * 4;
    static_assert(W * 8 <= (int)off_tile, "mbarriers");
    static_assert(off_si % 8 == 0, "float2 arrays");
};

template <int NI, int NJ, int NK>
__device__ __forceinline__ void march_quads(int b, int ka, int kb, const float* u, float* out, int8_t* ulo,
                                            const PushTable& push, const Geometry& g, StepScalars* sc, int cfl_next) {
    using S = MShape<NI, NJ, NK>;
    static_assert(NI == 16 && NJ == 16, "rows of 16 cells: one half-warp per row");
    static_assert(2 * (S::smem + 1024) <= 233472, "two CTAs per SM");
    constexpr int NIP = S::NIP, PL = S::PL, W = S::W, NCELL = S::NCELL, P = S::P, NP = S::NP;
    extern __shared__ __align__(128) unsigned char smem[];
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem);
    float4* tile = reinterpret_cast<float4*>(smem + S::off_tile);   // [2][W][PL]
    float2* SI = reinterpret_cast<float2*>(smem + S::off_si);
    float2* SJ = reinterpret_cast<float2*>(smem + S::off_sj);
    float2* FI = reinterpret_cast<float2*>(smem + S::off_fi);
    float2* FJ = reinterpret_cast<float2*>(smem + S::off_fj);
    float* gi = reinterpret_cast<float*>(smem + S::off_gi);
    float* gj = reinterpret_cast<float*>(smem + S::off_gj);
    float* gs = reinterpret_cast<float*>(smem + S::off_gs);
    const int tid = threadIdx.x;
    const float* blk = u + (size_t)b * NV * NCELL;
    const int flb = g.flags[b];
    const bool copy_bc = out != u && (flb & 6);
    __shared__ PushBlock pb;
    load_push_block(push, b, &pb);
    const bool issuer = tid == S::NT - 32;   // requests the copies
    // planes are counted from pa, the first that [ka, kb) needs; pe: one past the last
    const int pa = ka - 2, pe = kb + 2;
    int issued = pa;   // by the issuer: planes [pa, issued)
    auto issue = [&]() {
        issue_quads<S>(blk, tile, issued, issued + 1, pa, &bars[(issued - pa) % W]);
        ++issued;
    };
    int8_t* blk_lo = ulo != nullptr ? ulo + (size_t)b * NV * S::NINT : nullptr;
    step_go();
    if (issuer) {
        for (int s = 0; s < W; ++s) mbar_init(&bars[s], 1);
        fence_mbar_init();
        step_wait();
        while (issued < pa + W) issue();
        if (blk_lo != nullptr) prefetch_l2(blk_lo + (size_t)(ka - 2) * S::PLI * NV, 2 * S::PLI * NV);
    }
    load_geometry<float, S>(g, b, gi, gj, gs, nullptr);
    step_wait();
    __syncthreads();   // barriers and tables are used by every thread below
    // this thread's column: warp w takes rows (w % 4) + 8 (w / 4) and that + 4
    const int wq = tid >> 5, i = tid & 15;
    const int j = (wq & 3) + 8 * (wq >> 2) + 4 * ((tid >> 4) & 1);
    const int ii = i + 2, jj = j + 2;
    const float* GCS = gi + GI_CS * NIP;
    const float cs = GCS[ii];
    const float rc = gi[GI_R * NIP + ii];
    const float den[3] = {gs[GS_DXI], gs[GS_DXJ] * rc, gs[GS_DXK] * rc * gj[GJ_SIN * S::NJP + jj]};
    const float2 dinv0 = f2(1.f / den[0]), dinv1 = f2(1.f / den[1]), dinv2 = f2(1.f / den[2]);
    const float2 hdt2 = f2(sc->dt_half_f);
    const int polls = sc->wait_polls;
    int late = 0;   // a wait of this thread for a plane ran out
    auto abort_cta = [&]() {   // after a uniform decision: flag, drain the copies in flight
        if (!issuer) return;
        atomicOr(&sc->nan_flag, 2);
        for (int p = issued - pa < W ? 0 : issued - pa - W; p < issued - pa; ++p)
            mbar_wait(&bars[p % W], (uint32_t)((p / W) & 1), kWaitPolls);
        for (int q = 0; q < W; ++q) mbar_inval(&bars[q]);
    };
    auto lo2 = [](const float4& x) { return f2(x.x, x.y); };
    auto hi2 = [](const float4& x) { return f2(x.z, x.w); };
    const int c0 = jj * NIP + ii;
    auto slot_of = [&](int p) { return (p - pa) % W * PL; };
    // the pairs of a cell in a plane's slot
    auto pairs = [&](int slot, int c, float2 (&v)[NP]) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float4 x = tile[h * W * PL + slot + c];
            v[2 * h] = lo2(x);
            v[2 * h + 1] = hi2(x);
        }
    };
    // the column window from planes ka-2 .. ka+1: u at kp = ka and ka + 1, the k
    // slope at ka, the flux through the face between planes ka-1 and ka
    for (int p = 0; p < 4; ++p) late |= mbar_wait(&bars[p], 0u, polls) ? 0 : 1;
    if (copy_bc) copy_bc_columns<S>(tile, pa, out, b, flb, pa, pa + 4, S::NT);
    float2 u0[NP], u1[NP], dk0[NP], fk0[NP];
    {
        const float2 cc = f2(face_speed(tile[PL + c0].w, cs, tile[2 * PL + c0].w, cs));
        float2 a0[NP], a1[NP];
        pairs(0, c0, a0);
        pairs(PL, c0, a1);
        pairs(2 * PL, c0, u0);
        pairs(3 * PL, c0, u1);
#pragma unroll
        for (int q = 0; q < NP; ++q) {
            const float2 d1 = half_slope2(a0[q], a1[q], u0[q]);
            dk0[q] = half_slope2(a1[q], u0[q], u1[q]);
            fk0[q] = face_flux2(a1[q], u0[q], d1, dk0[q], cc);
        }
    }
    float wmax = 0.f;   // the column's largest wave speed, for the next step's CFL minimum
    int cnan = 0;
    const float srho = __fsqrt_rn(gi[GI_RHO0 * NIP + ii]), srho_inv = __frcp_rn(srho);
    for (int kp = ka; kp < kb; ++kp) {
        const int p2 = kp + 2;
        if (blk_lo != nullptr && issuer && kp + 2 < kb)
            prefetch_l2(blk_lo + (size_t)kp * S::PLI * NV, S::PLI * NV);
        // this cell's int8 corrections, loaded before the wait
        int2 q8 = make_int2(0, 0);
        int2* ql = reinterpret_cast<int2*>(blk_lo + (((size_t)(kp - 2) * NJ + j) * NI + i) * NV);
        if (blk_lo != nullptr) q8 = *ql;
        // a wait that runs out finishes the plane on whatever the slot holds;
        // the step is flagged and discarded
        late |= mbar_wait(&bars[(p2 - pa) % W], (uint32_t)(((p2 - pa) / W) & 1), polls) ? 0 : 1;
        if (copy_bc) copy_bc_columns<S>(tile, pa, out, b, flb, p2, p2 + 1, S::NT);
        const int s0 = slot_of(kp), s1 = slot_of(kp + 1), s2 = slot_of(p2);
        // the half with the velocities at this cell
        const float4 vc = tile[s0 + c0], vl = tile[s0 + c0 - 1], vd = tile[s0 + c0 - NIP];
        // ---- phase A: k slope and k face from the window; i and j slopes
        float2 u2[NP], dk1[NP], fk1[NP];
        {
            const float2 cc = f2(face_speed(vc.w, cs, tile[s1 + c0].w, cs));
            pairs(s2, c0, u2);
#pragma unroll
            for (int q = 0; q < NP; ++q) {
                dk1[q] = half_slope2(u0[q], u1[q], u2[q]);
                fk1[q] = face_flux2(u0[q], u1[q], dk0[q], dk1[q], cc);
            }
            float2 l[NP], r[NP];
            pairs(s0, c0 - 1, l);
            pairs(s0, c0 + 1, r);
#pragma unroll
            for (int q = 0; q < NP; ++q) SI[q * S::NSI + j * P + i + 1] = half_slope2(l[q], u0[q], r[q]);
            pairs(s0, c0 - NIP, l);
            pairs(s0, c0 + NIP, r);
#pragma unroll
            for (int q = 0; q < NP; ++q) SJ[q * S::NSJ + (j + 1) * P + i] = half_slope2(l[q], u0[q], r[q]);
        }
        // slopes of the ghost cells next to the block: i = -1, NI of every row
        // (items 0..255) and j = -1, NJ of every column (items 256..511)
#pragma unroll
        for (int x = tid; x < 512; x += S::NT) {
            const int side = x & 1, r = (x >> 1) & 15, v = (x >> 5) & 7;
            const float* a = reinterpret_cast<const float*>(tile + (v >> 2) * W * PL + s0) + (v & 3);
            float* dst;
            float val;
            if (x < 256) {
                const float* q = a + 4 * ((r + 2) * NIP + (side ? NI + 2 : 1));
                val = half_slope(q[-4], q[0], q[4]);
                dst = reinterpret_cast<float*>(SI + (v >> 1) * S::NSI + r * P + (side ? NI + 1 : 0));
            } else {
                const float* q = a + 4 * ((side ? NJ + 2 : 1) * NIP + r + 2);
                val = half_slope(q[-4 * NIP], q[0], q[4 * NIP]);
                dst = reinterpret_cast<float*>(SJ + (v >> 1) * S::NSJ + (side ? NJ + 1 : 0) * P + r);
            }
            dst[v & 1] = val;
        }
        if (__syncthreads_or(late)) {
            abort_cta();
            return;
        }
        // ---- phase B: the faces i - 1/2 and j - 1/2 of this cell, and the
        // last faces of the rows (items 0..127) and columns (128..255)
        float2 fi0[NP], fj0[NP];
        {
            const float2 cci = f2(face_speed(vl.y, GCS[ii - 1], vc.y, cs)), ccj = f2(face_speed(vd.z, cs, vc.z, cs));
            float2 l[NP], d[NP];
            pairs(s0, c0 - 1, l);
            pairs(s0, c0 - NIP, d);
#pragma unroll
            for (int q = 0; q < NP; ++q) {
                const float2* si = SI + q * S::NSI + j * P + i;
                const float2* sj = SJ + q * S::NSJ + j * P + i;
                fi0[q] = face_flux2(l[q], u0[q], si[0], si[1], cci);
                fj0[q] = face_flux2(d[q], u0[q], sj[0], sj[P], ccj);
                FI[q * S::NFI + j * P + i] = fi0[q];
                FJ[q * S::NFJ + j * P + i] = fj0[q];
            }
        }
        if (tid < 256) {
            const int x = tid, r = x & 15, v = (x >> 4) & 7;
            const float* sl = reinterpret_cast<const float*>(x < 128 ? SI + (v >> 1) * S::NSI + r * P + NI
                                                                     : SJ + (v >> 1) * S::NSJ + NJ * P + r);
            if (x < 128) {
                const float* a = reinterpret_cast<const float*>(tile + (v >> 2) * W * PL + s0 + (r + 2) * NIP + NI + 1) + (v & 3);
                const float4* vr = tile + s0 + (r + 2) * NIP + NI + 1;   // last interior cell of row r
                reinterpret_cast<float*>(FI + (v >> 1) * S::NFI + r * P + NI)[v & 1] =
                    face_flux(a[0], a[4], sl[v & 1], sl[2 + (v & 1)], face_speed(vr[0].y, GCS[NI + 1], vr[1].y, GCS[NI + 2]));
            } else {
                const float* a = reinterpret_cast<const float*>(tile + (v >> 2) * W * PL + s0 + (NJ + 1) * NIP + r + 2) + (v & 3);
                const float4* vt = tile + s0 + (NJ + 1) * NIP + r + 2;   // last interior row, column r
                const float c2 = GCS[r + 2];
                reinterpret_cast<float*>(FJ + (v >> 1) * S::NFJ + NJ * P + r)[v & 1] =
                    face_flux(a[0], a[4 * NIP], sl[v & 1], sl[2 * P + (v & 1)], face_speed(vt[0].z, c2, vt[NIP].z, c2));
            }
        }
        __syncthreads();
        // planes below kp + 1 are done with: refill their slots, up to plane
        // kp + W (at kp = 2 that is planes 5, 6, 7; then one plane a step)
        if (issuer)
            while (issued < pe && issued <= kp + W) issue();
        // ---- phase C: sum the six faces in the reference's order, update
        const size_t cell = (size_t)kp * PL + c0;
        float o[NV], u[NV];
        float2 R[NP];
#pragma unroll
        for (int q = 0; q < NP; ++q) {
            R[q] = __fmul2_rn(sub2(fi0[q], FI[q * S::NFI + j * P + i + 1]), dinv0);
            R[q] = __ffma2_rn(sub2(fj0[q], FJ[q * S::NFJ + (j + 1) * P + i]), dinv1, R[q]);
            R[q] = __ffma2_rn(sub2(fk0[q], fk1[q]), dinv2, R[q]);
            u[2 * q] = u0[q].x;
            u[2 * q + 1] = u0[q].y;
        }
        if (ulo != nullptr) {
            ff_add4(u, q8.x, {__fmul2_rn(hdt2, R[0]), __fmul2_rn(hdt2, R[1])}, o);
            ff_add4(u + 4, q8.y, {__fmul2_rn(hdt2, R[2]), __fmul2_rn(hdt2, R[3])}, o + 4);
            *ql = q8;
        } else {
#pragma unroll
            for (int q = 0; q < NP; ++q) {
                const float2 ov = __ffma2_rn(hdt2, R[q], u0[q]);
                o[2 * q] = ov.x;
                o[2 * q + 1] = ov.y;
            }
        }
        quads(out)[quad(b, 0, NCELL) + cell] = f4(o);
        quads(out)[quad(b, 1, NCELL) + cell] = f4(o + 4);
        if (push.tgt != nullptr) push_quads<S>(out, pb, ii, jj, kp, o);
        if (cfl_next) {   // uniform over the CTA
#pragma unroll
            for (int v = 0; v < NV; ++v) cnan |= (o[v] != o[v]);
            wmax = fmaxf(wmax, cfl_speed(cfl_sq3(o[V_VR], o[V_VT], o[V_VP]), cfl_sq3(o[V_BR], o[V_BT], o[V_BP]), cs, srho, srho_inv));
        }
        // the window moves up one plane
#pragma unroll
        for (int q = 0; q < NP; ++q) {
            u0[q] = u1[q];
            u1[q] = u2[q];
            dk0[q] = dk1[q];
            fk0[q] = fk1[q];
        }
    }
    if (__syncthreads_or(late)) {
        abort_cta();
        return;
    }
    if (issuer)   // every copy has been waited for
        for (int q = 0; q < W; ++q) mbar_inval(&bars[q]);
    if (cfl_next) cfl_commit(cfl_column(wmax, rc, gj[GJ_SIN * S::NJP + jj], gs[GS_DXI], gs[GS_DXJ], gs[GS_DXK]), cnan, sc);
}
// split CTAs per block, each a run of planes
template <int NI, int NJ, int NK>
__global__ void __launch_bounds__(NI * NJ, 2)
k_march_quads(const float* u, float* out, int8_t* ulo, PushTable push, Geometry g, StepScalars* sc, int cfl_next, int split) {
    const int b = blockIdx.x / split, part = blockIdx.x - b * split, n = NK / split;
    march_quads<NI, NJ, NK>(b, 2 + part * n, 2 + (part + 1) * n, u, out, ulo, push, g, sc, cfl_next);
}

// ---------------------------------------------------------------------------
// [G][n] to [n][G] in place, an array per CTA through shared memory (a half of a 16^3
// block: 125 KB).
template <class T, int G>
__global__ void __launch_bounds__(512) k_interleave(T* a, int n) {
    extern __shared__ __align__(16) unsigned char smem[];
    int4* s = reinterpret_cast<int4*>(smem);
    int4* g = reinterpret_cast<int4*>(a + (size_t)blockIdx.x * G * n);
    const int vecs = (int)((size_t)G * n * sizeof(T) / 16);
    for (int x = threadIdx.x; x < vecs; x += blockDim.x) s[x] = g[x];
    __syncthreads();
    constexpr int V = 16 / sizeof(T);
    const T* t = reinterpret_cast<const T*>(smem);
    for (int x = threadIdx.x; x < vecs; x += blockDim.x) {
        T o[V];
#pragma unroll
        for (int q = 0; q < V; ++q) {
            const int y = x * V + q;
            o[q] = t[y % G * n + y / G];
        }
        int4 r;
        memcpy(&r, o, 16);
        g[x] = r;
    }
}

// ---------------------------------------------------------------------------
// Every cell outside the core of each block and variable set to 0 (the k ghost
// planes and, in the interior planes, the j ghost rows: per block and
// variable, (NJP-4)*NIP-wide gaps between the core runs). A core upload clears
// them before its exchange refills the listed ones: the mixed interpolations
// read some ghost cells of their source blocks with weight 0, which is
// harmless for finite values only, and the buffer may hold an earlier state
// with NaNs there. Cleared, the uploaded state's ghost cells are the same
// whatever the buffer held (a new context starts with zeros too).
// T: float4 for the state's halves, float for psi; nbv arrays of ncell cells.
template <class T>
__global__ void __launch_bounds__(256) k_clear_outside_core(T* u, int64_t nbv, StepDims d) {
    const int pl = d.nip * d.njp, lead = 2 * pl + 2 * d.nip, gap = 4 * d.nip;
    const int per = 2 * lead + (d.nkp - 5) * gap;   // non-core cells per block and variable
    for (int64_t bv = blockIdx.x; bv < nbv; bv += gridDim.x) {
        T* base = u + bv * d.ncell;
        for (int x = threadIdx.x; x < per; x += blockDim.x) {
            int c;
            if (x < lead) {
                c = x;                                   // planes 0, 1 and rows 0, 1 of plane 2
            } else if (x < per - lead) {
                const int q = (x - lead) / gap, r = (x - lead) - q * gap;
                c = (2 + q) * pl + (d.njp - 2) * d.nip + r;   // rows NJP-2, NJP-1 of plane 2+q, rows 0, 1 of the next
            } else {
                c = d.ncell - lead + (x - (per - lead));   // rows NJP-2, NJP-1 of the last interior plane, 2 ghost planes
            }
            base[c] = T{};
        }
    }
}

// ---------------------------------------------------------------------------
// After the core of a mixed state has been replaced from the host (the core
// upload), what the diffusion pass closing a mixed step leaves besides
// u^{n+1} itself: the regular faces pushed into the neighbours' ghost layers
// (the face entries left to the final exchange follow as a separate launch),
// and the next step's CFL minimum with the NaN scan, each cell's ratio the
// one k_cfl forms. One CTA per block and a thread per (i, j) column marching
// k; a row of NI cells lies in consecutive lanes, as the pushed radial faces
// need.
template <int NI, int NJ, int NK>
__global__ void __launch_bounds__(NI * NJ) k_push_state(float* u, PushTable push, Geometry g, StepScalars* sc) {
    using S = MShape<NI, NJ, NK>;
    constexpr int NIP = S::NIP, NJP = S::NJP;
    static_assert((NI * NJ) % 32 == 0 && 32 % NI == 0, "whole rows in every warp");
    __shared__ PushBlock pb;
    const int b = blockIdx.x, tid = threadIdx.x;
    load_push_block(push, b, &pb);
    __syncthreads();
    const int ii = tid % NI + 2, jj = tid / NI + 2;
    const float* Gi = gi_ptr<float>(g) + (size_t)b * GI_COUNT * NIP;
    const float* Gj = gj_ptr<float>(g) + (size_t)b * GJ_COUNT * NJP;
    const float* Gs = gs_ptr<float>(g) + (size_t)b * GS_COUNT;
    const float cs = Gi[GI_CS * NIP + ii], rho0 = Gi[GI_RHO0 * NIP + ii], r = Gi[GI_R * NIP + ii];
    const float sin_t = Gj[GJ_SIN * NJP + jj], dxi = Gs[GS_DXI], dxj = Gs[GS_DXJ], dxk = Gs[GS_DXK];
    float cmin = INFINITY;
    int cnan = 0;
    constexpr int G = 4;   // planes whose loads are all issued before the first push
    static_assert(NK % G == 0, "whole plane groups");
    for (int k0 = 2; k0 < NK + 2; k0 += G) {
        float o[G][NV];
#pragma unroll
        for (int q = 0; q < G; ++q) {
            const size_t cell = ((size_t)(k0 + q) * NJP + jj) * NIP + ii;
            load_cell<false>(u + Layout<float>::at(b, 0, cell, S::NCELL), S::NCELL, o[q]);
        }
#pragma unroll
        for (int q = 0; q < G; ++q) {
            if (push.tgt != nullptr) push_quads<S>(u, pb, ii, jj, k0 + q, o[q]);
#pragma unroll
            for (int v = 0; v < NV; ++v) cnan |= (o[q][v] != o[q][v]);
            float ratio = cfl_ratio_f(cfl_sq3(o[q][V_VR], o[q][V_VT], o[q][V_VP]),
                                      cfl_sq3(o[q][V_BR], o[q][V_BT], o[q][V_BP]), cs, rho0, r, sin_t, dxi, dxj, dxk);
            if (ratio != ratio) { cnan = 1; ratio = INFINITY; }
            cmin = fminf(cmin, ratio);
        }
    }
    cfl_commit(cmin, cnan, sc);
}

// ---------------------------------------------------------------------------
// A barrier over every CTA of a cooperative launch (all co-resident). Thread
// 0 of each CTA reads the generation, arrives on the counter; the last one
// resets the counter and advances the generation, the others poll it, at most
// `polls` times (a poll that runs out flags the step: bit 1 of nan_flag, the
// host returns FALCON_ERR_TIMEOUT, and the CTA goes on). Fences on both sides
// make every CTA's writes before the barrier visible to every CTA after it.
struct GridBarrier {
    unsigned int* count;   // 0 between barriers
    unsigned int* gen;
    unsigned int* ticket;  // [5]: the next block of each block phase (4 stages, diffusion), 0 at launch
};
__device__ __forceinline__ void grid_sync(const GridBarrier& gb, StepScalars* sc, int polls) {
    // the next phase reads this one's global writes also through bulk copies
    // (the async proxy): order them across the proxies on both sides
    asm volatile("fence.proxy.async.global;" ::: "memory");
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned int g0 = *(volatile unsigned int*)gb.gen;
        __threadfence();
        if (atomicAdd(gb.count, 1u) == gridDim.x - 1) {
            atomicExch(gb.count, 0u);
            __threadfence();
            atomicAdd(gb.gen, 1u);
        } else {
            int it = 0;
            while (*(volatile unsigned int*)gb.gen == g0) {
                if (++it > polls) {
                    atomicOr(&sc->nan_flag, 2);
                    break;
                }
                __nanosleep(64);
            }
        }
        __threadfence();
    }
    __syncthreads();
    asm volatile("fence.proxy.async.global;" ::: "memory");
}

// The pointers of one mixed step: u^n in U, the stage buffer RK, the second
// state buffer R2 (u^{n+1} is written there, then the host swaps U and R2).
struct StepBuffers {
    float* U;
    float* RK;
    float* R2;
    int8_t* ulo;
};

// One mixed RK4 step of 16^3 blocks in one persistent launch: the CTAs take
// the blocks (and, in the exchanges, the ghost entries) in turn and meet at a
// grid barrier between the phases the graph runs as separate launches:
// dt, then per stage s the stage kernel's body into seq[s] (pushing the
// regular ghost faces) and the exchange of the rest (face lists), then the
// diffusion body into R2 (pushes, next step's CFL minimum) and the exchange
// of the remaining entries. The bodies are the separate kernels' own
// (a thread per column: 256 each; every variant computes the same bits), so the
// step equals the graph's bit for bit.
template <int N>
__global__ void __launch_bounds__(256, 2)
k_step_persistent(StepBuffers sb, PushTable push, Geometry g, StepScalars* sc, GhostLists gl_stage,
                  GhostLists gl_final, StepDims d, GridBarrier gb) {
    static_assert(N == 16, "16^3 blocks");
    const int polls = sc->wait_polls;
    if (blockIdx.x == 0 && threadIdx.x == 0) finalize_dt_body(sc);
    grid_sync(gb, sc, polls);
    const int64_t tstride = (int64_t)gridDim.x * blockDim.x;
    const int64_t t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    auto exchange = [&](const GhostLists& G, float* u) {
        for (int64_t e = t0; e < G.ip.n; e += tstride)
            ghost_interp_one<true>(u, G.ip, d.ncell, d.nip, d.nip * d.njp, e);
        for (int64_t e = t0; e < G.ln.n; e += tstride) ghost_lin_one<float, true>(u, G.ln, d.ncell, e);
        for (int64_t e = t0; e < G.cp.n; e += tstride) ghost_copy_one<float, true>(u, G.cp, d.ncell, e);
    };
    // between two bodies in one CTA: the generic writes of the one before
    // are ordered before the bulk copies of the next into the same memory
    auto next_body = [&]() {
        fence_proxy_async();
        __syncthreads();
    };
    // blocks are handed out one at a time from a ticket counter per phase, as
    // the hardware scheduler hands CTAs to SMs: a CTA that finishes early
    // takes the next block instead of waiting at the barrier
    __shared__ int next_b;
    auto take = [&](int phase) -> int {
        if (threadIdx.x == 0) next_b = (int)atomicAdd(&gb.ticket[phase], 1u);
        __syncthreads();
        return next_b;   // read before the next take's write: a body or next_body() barrier lies between
    };
    for (int s = 1; s <= 4; ++s) {
        float* in = s == 1 ? sb.U : (s == 3 ? sb.R2 : sb.RK);
        float* out = s == 4 ? sb.U : (s == 2 ? sb.R2 : sb.RK);   // U -> RK -> R2 -> RK -> U
        for (int b = take(s - 1); b < d.nblocks; b = take(s - 1)) {
            stage_march<16, 16, 16, 0>(b, 2, 18, in, sb.U, out, sb.ulo, push, DivBArgs{nullptr, nullptr, nullptr, 0}, g, sc, s,
                                          1);
            next_body();
        }
        grid_sync(gb, sc, polls);
        exchange(gl_stage, out);
        grid_sync(gb, sc, polls);
    }
    for (int b = take(4); b < d.nblocks; b = take(4)) {
        march_quads<16, 16, 16>(b, 2, 18, sb.U, sb.R2, sb.ulo, push, g, sc, 1);
        next_body();
    }
    grid_sync(gb, sc, polls);
    exchange(gl_final, sb.R2);
}

}  // namespace impl
}  // namespace falcon
