// mhd_impl.cuh -- kernel bodies shared by the FP64 and mixed instantiations.
// Included by mhd_fp64.cu (T=double, -fmad=false) and mhd_mixed.cu (T=float).
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

#include "kernels.cuh"
#include "exact64.cuh"

namespace falcon {
namespace impl {

// Precision policy. Exact: the reference's divisions stay divisions; the
// mixed path multiplies by reciprocals tabulated on the host.
template <class T> struct Pol;
template <> struct Pol<double> {
    static constexpr bool exact = true;
    __device__ static __forceinline__ double mmthr() { return (double)1.e-30f; }
    __device__ static __forceinline__ double mmscale() { return 1.e10; }
    __device__ static __forceinline__ double ratio(double a, double b) { return a / b; }
};
template <> struct Pol<float> {
    static constexpr bool exact = false;
    __device__ static __forceinline__ float mmthr() { return 1.e-30f; }
    __device__ static __forceinline__ float mmscale() { return 1.e10f; }
    // limiter ratio: an approximate quotient is enough (0/0 still gives NaN -> phi = 0)
    __device__ static __forceinline__ float ratio(float a, float b) { return __fdividef(a, b); }
};

// ModLinReconstruct_minmod for one value (3_6/ModLinReconstruct.f90:44-48).
template <class T>
__device__ __forceinline__ T minmod(T ul, T u, T ur) {
    const T a = (ur - ul) * T(0.5);
    const T b = T(2) * (ur - u);
    const T c = T(2) * (u - ul);
    T t;
    if (Pol<T>::exact) {
        t = fmax(T(0), a * b) * fmax(T(0), b * c) * Pol<T>::mmscale() - Pol<T>::mmthr();
    } else {
        // same test, factors reordered so the FP32 product stays in the normal range
        t = (fmax(T(0), a * b) * Pol<T>::mmscale()) * fmax(T(0), b * c) - Pol<T>::mmthr();
    }
    const T s = copysign(T(0.5), t);
    const T m = fmin(fmin(fabs(a), fabs(b)), fabs(c));
    return (s + T(0.5)) * copysign(m, a);
}

// The per-cell CFL ratio h_LLL / v_wave of the mixed path, shared by k_cfl and
// the diffusion pass that forms it for the next step: explicitly rounded FP32
// operations, so both give the same bits whatever the compiler contracts.
__device__ __forceinline__ float cfl_sq3(float x, float y, float z) {
    return __fadd_rn(__fadd_rn(__fmul_rn(x, x), __fmul_rn(y, y)), __fmul_rn(z, z));
}
__device__ __forceinline__ float cfl_ratio_f(float v2, float b2, float cs, float rho0, float r, float sin_t,
                                             float dxi, float dxj, float dxk) {
    // h_LLL = min(dxi, r*dxj, r*sin(theta)*dxk) (3_6/ModBlock.f90:416-425)
    const float h = fminf(fminf(dxi, __fmul_rn(r, dxj)), __fmul_rn(__fmul_rn(r, sin_t), dxk));
    float w = __fadd_rn(cs, __fsqrt_rn(v2));
    w = __fadd_rn(w, __fdiv_rn(__fsqrt_rn(b2), __fsqrt_rn(rho0)));
    return __fdiv_rn(h, w);
}
// block minimum of the ratios (FP64 bit order for positive values) and NaN flag
__device__ __forceinline__ void cfl_commit(float ratio, int nan, StepScalars* sc) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        ratio = fminf(ratio, __shfl_xor_sync(0xffffffffu, ratio, o));
        nan |= __shfl_xor_sync(0xffffffffu, nan, o);
    }
    __shared__ float wmin[32];
    __shared__ int wnan[32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) { wmin[wid] = ratio; wnan[wid] = nan; }
    __syncthreads();
    if (threadIdx.x == 0) {
        float m = wmin[0];
        int n = wnan[0];
        for (int w2 = 1; w2 < (int)(blockDim.x >> 5); ++w2) { m = fminf(m, wmin[w2]); n |= wnan[w2]; }
        atomicMin(&sc->min_ratio_bits, (unsigned long long)__double_as_longlong((double)m));
        if (n) atomicOr(&sc->nan_flag, 1);
    }
}

template <class T> __device__ __forceinline__ const T* gi_ptr(const Geometry& g);
template <> __device__ __forceinline__ const double* gi_ptr<double>(const Geometry& g) { return g.gi; }
template <> __device__ __forceinline__ const float* gi_ptr<float>(const Geometry& g) { return g.gi_f; }
template <class T> __device__ __forceinline__ const T* gj_ptr(const Geometry& g);
template <> __device__ __forceinline__ const double* gj_ptr<double>(const Geometry& g) { return g.gj; }
template <> __device__ __forceinline__ const float* gj_ptr<float>(const Geometry& g) { return g.gj_f; }
template <class T> __device__ __forceinline__ const T* gs_ptr(const Geometry& g);
template <> __device__ __forceinline__ const double* gs_ptr<double>(const Geometry& g) { return g.gs; }
template <> __device__ __forceinline__ const float* gs_ptr<float>(const Geometry& g) { return g.gs_f; }

// ---- TMA (bulk async copy) and mbarrier helpers ---------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
// a barrier object is invalidated before its shared memory is used for
// anything else (the persistent step runs several kernel bodies in one CTA)
__device__ __forceinline__ void mbar_inval(uint64_t* bar) {
    asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
// Programmatic dependent launch of the mixed step's kernels (launch_step): a kernel's
// CTAs may start while the one before drains. What comes before step_wait reads only
// what no kernel of a step writes (geometry, flags, lists, push table) and writes only
// shared memory; after it, the work of every kernel before is complete and visible.
// step_go lets the next kernel's CTAs take the slots that this one's leave.
__device__ __forceinline__ void step_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void step_go() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// 1-D bulk copy global -> shared, completion counted on `bar` (16-byte aligned, size % 16 == 0)
// Hint: pull `bytes` (a multiple of 16, 16-byte aligned) of global memory into
// L2 ahead of plain loads.
__device__ __forceinline__ void prefetch_l2(const void* p, uint32_t bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}
__device__ __forceinline__ void tma_load_1d(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}
// bounded wait on an mbarrier phase; false if it did not complete in max_iter polls
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int max_iter) {
    for (int it = 0; it < max_iter; ++it) {
        uint32_t ok;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(ok)
            : "r"(smem_u32(bar)), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}
constexpr int kWaitPolls = kDefaultWaitPolls;

// A CTA whose wait for a chunk's planes ran out leaves cleanly: every thread
// learns it at the next chunk's leading barrier (__syncthreads_or, so the exit
// is uniform over the CTA and no thread is left at a barrier), then thread 0
// flags the step (bit 1 of nan_flag: the host returns FALCON_ERR_TIMEOUT) and
// waits, with the default bound, for the bulk copies still in flight into
// this CTA's shared memory -- chunks c0..c1 -- before the CTA exits.
__device__ __forceinline__ void copy_wait_abort(StepScalars* sc, uint64_t* bars, int c0, int c1) {
    if (threadIdx.x != 0) return;
    atomicOr(&sc->nan_flag, 2);
    for (int c = c0 < 0 ? 0 : c0; c <= c1; ++c) mbar_wait(&bars[c & 1], (uint32_t)((c >> 1) & 1), kWaitPolls);
    mbar_inval(&bars[0]);
    mbar_inval(&bars[1]);
}

template <class T, int NI, int NJ, int NK, int KPAR>
struct Shape {
    static constexpr int NG = 2, NIP = NI + 4, NJP = NJ + 4, NKP = NK + 4;
    static constexpr int PL = NIP * NJP, NT = NI * NJ * KPAR;
    static constexpr int W = 2 * KPAR + 4;    // ring: current window (KPAR+4) + the prefetched KPAR planes
    static constexpr int WP = KPAR + 4;       // p1 window
    static constexpr int NCELL = PL * NKP;
    static constexpr int PLI = NI * NJ, NINT = PLI * NK;   // the u^n correction's (interior-only) plane and block
    static constexpr uint32_t PLB = PL * (uint32_t)sizeof(T);   // bytes of one variable plane
    static_assert(PLB % 16 == 0, "plane must be a multiple of 16 bytes");
    static_assert(NK % KPAR == 0, "KPAR must divide NK");
    // FP64 path: the fields that several cells' derivatives read, formed once
    // per point instead of at each use. Br/sin(theta) and E_r/sin(theta) (E = v
    // x B; the k-derivatives of the curls divide them by the cell's sin(theta),
    // which its k-neighbours share) and E_theta over the p1 window: [WP][PLI]
    // twice and [WP][NJ][NIP]; E_r and E_phi of the chunk's own planes, on the
    // points that i- and j-derivatives reach: [KPAR][NJP][NI] and [KPAR][PL].
    // With the derivatives' FMAs and the quotients by rho0 and sin(theta)
    // through reciprocals a cell takes 377 FP64 instructions instead of 548
    // (442,368 cells: 477 -> 359 us per stage in 8^3 blocks, 652 -> 482 in 16^3).
    static constexpr bool kPoint = sizeof(T) == 8;
    static constexpr int NXS = kPoint ? 2 * WP * PLI : 0, NE2 = kPoint ? WP * NJ * NIP : 0;
    static constexpr int NE1 = kPoint ? KPAR * NJP * NI : 0, NE3 = kPoint ? KPAR * PL : 0;
    // shared memory: mbarriers | A1/A2 (double) | tile[NV][W][PL] | p1[WP][PL] | xs | e2 | e1 | e3 | gi | gj | gs
    static constexpr size_t off_a12 = 16;
    static constexpr size_t off_tile = off_a12 + ((2 * NIP * sizeof(double) + 15) / 16) * 16;
    static constexpr size_t off_p1 = off_tile + (size_t)NV * W * PL * sizeof(T);
    static constexpr size_t off_xs = off_p1 + (size_t)WP * PL * sizeof(T);
    static constexpr size_t off_e2 = off_xs + (size_t)NXS * sizeof(T);
    static constexpr size_t off_e1 = off_e2 + (size_t)NE2 * sizeof(T);
    static constexpr size_t off_e3 = off_e1 + (size_t)NE1 * sizeof(T);
    static constexpr size_t off_gi = off_e3 + (size_t)NE3 * sizeof(T);
    static constexpr size_t off_gj = off_gi + (size_t)GI_COUNT * NIP * sizeof(T);
    static constexpr size_t off_gs = off_gj + (size_t)GJ_COUNT * NJP * sizeof(T);
    static constexpr size_t smem_stage = off_gs + GS_COUNT * sizeof(T);
};

// Thread 0: bulk-copy planes kp in [lo,hi) of all variables of the block into
// their ring slots, completing on `bar`.
template <class T, class S>
__device__ __forceinline__ void issue_planes(const T* blk, T* tile, int lo, int hi, uint64_t* bar) {
    mbar_expect_tx(bar, (uint32_t)(NV * (hi - lo)) * S::PLB);
    for (int v = 0; v < NV; ++v)
        for (int kp = lo; kp < hi; ++kp)
            tma_load_1d(tile + ((size_t)v * S::W + (kp % S::W)) * S::PL, blk + ((size_t)v * S::NKP + kp) * S::PL,
                        S::PLB, bar);
}

template <class T, class S>
__device__ __forceinline__ void load_geometry(const Geometry& g, int b, T* gi, T* gj, T* gs, double* a12) {
    const T* Gi = gi_ptr<T>(g) + (size_t)b * GI_COUNT * S::NIP;
    const T* Gj = gj_ptr<T>(g) + (size_t)b * GJ_COUNT * S::NJP;
    const T* Gs = gs_ptr<T>(g) + (size_t)b * GS_COUNT;
    for (int x = threadIdx.x; x < GI_COUNT * S::NIP; x += S::NT) gi[x] = Gi[x];
    for (int x = threadIdx.x; x < GJ_COUNT * S::NJP; x += S::NT) gj[x] = Gj[x];
    for (int x = threadIdx.x; x < GS_COUNT; x += S::NT) gs[x] = Gs[x];
    if (a12) {
        const double* Gd = g.gi + (size_t)b * GI_COUNT * S::NIP;
        for (int x = threadIdx.x; x < 2 * S::NIP; x += S::NT) {
            const double a = Gd[(x < S::NIP ? GI_A1 * S::NIP : GI_A2 * S::NIP - S::NIP) + x];
            a12[x] = a;
        }
    }
}

// p1 = a1*rho1 + a2*s1 for the mixed path in float-float arithmetic: the
// two products are formed exactly with FMA (plus the coefficients' low
// parts), summed with an error-free two-sum, and rounded once to FP32. The
// terms nearly cancel, so a plain FP32 sum would lose digits; this keeps the
// accuracy of an FP64 assembly on the FP32 pipe (GB300's FP64 rate is a
// small fraction of its FP32 rate).
__device__ __forceinline__ float p1_ff(float a1h, float a1l, float a2h, float a2l, float r1, float s1) {
    const float ph = __fmul_rn(a1h, r1);
    const float pl = __fmaf_rn(a1h, r1, -ph);
    const float qh = __fmul_rn(a2h, s1);
    const float ql = __fmaf_rn(a2h, s1, -qh);
    const float sh = __fadd_rn(ph, qh);
    const float bb = __fsub_rn(sh, ph);
    const float se = __fadd_rn(__fsub_rn(ph, __fsub_rn(sh, bb)), __fsub_rn(qh, bb));
    const float lo = __fmaf_rn(a1l, r1, __fmaf_rn(a2l, s1, __fadd_rn(pl, ql)));
    return __fadd_rn(sh, __fadd_rn(se, lo));
}

// Radial mirror boundary (3_6/ModBoundary.f90:10-55) on planes [lo,hi) of the
// ring, whole rows including their theta ghosts; optionally written back.
template <class T, class S>
__device__ __forceinline__ void apply_bc(T* tile, int lo, int hi, int fl, T* wb) {
    const bool top = fl & 2, bot = fl & 4;
    if (!top && !bot) return;
    const int np = hi - lo;
    const int NI = S::NIP - 4;
    // per variable sign: top mirrors rho1,vt,vp,s1,br; anti-mirrors vr,bt,bp.
    // bottom mirrors rho1,vt,vp,s1,bt,bp; anti-mirrors vr,br.
    const int total = np * S::NJP * NV * 2;
    for (int x = threadIdx.x; x < total; x += S::NT) {
        const int g = x & 1;
        const int rest = x >> 1;
        const int v = rest % NV;
        const int rest2 = rest / NV;
        const int j = rest2 % S::NJP;
        const int kp = lo + rest2 / S::NJP;
        T* row = tile + ((size_t)v * S::W + (kp % S::W)) * S::PL + j * S::NIP;
        if (top) {
            // Fortran i = ni+1+g <- 2*ni+1-i = ni-g ; padded index = Fortran + 1
            const bool neg = (v == V_VR) || (v == V_BT) || (v == V_BP);
            const T s = row[NI - g + 1];
            const T val = neg ? -s : s;
            row[NI + 2 + g] = val;
            if (wb) wb[((size_t)v * S::NKP + kp) * S::PL + j * S::NIP + NI + 2 + g] = val;
        }
        if (bot) {
            // Fortran i = -g <- 1-i = 1+g ; padded index = Fortran + 1
            const bool neg = (v == V_VR) || (v == V_BR);
            const T s = row[2 + g];
            const T val = neg ? -s : s;
            row[1 - g] = val;
            if (wb) wb[((size_t)v * S::NKP + kp) * S::PL + j * S::NIP + 1 - g] = val;
        }
    }
}

// 1-D blend a*(1-w) + b*w with one fixed rounding sequence, so the ghost
// fill and the stage kernel's pushed faces give identical values
__device__ __forceinline__ float blend(float a, float b, float uw, float w) { return __fmaf_rn(a, uw, __fmul_rn(b, w)); }
__device__ __forceinline__ double blend(double a, double b, double uw, double w) { return a * uw + b * w; }

// The push-table entries of one block, staged in shared memory before the
// kernel's first barrier: they are read at the end of every k-chunk, and as
// global loads their latency held every warp at the chunk's end.
struct PushBlock {
    int32_t tgt[6];
    int32_t src[4], dst[4];   // [side][layer]
    float w[4];
};
__device__ __forceinline__ void load_push_block(const PushTable& P, int b, PushBlock* s) {
    const int t = threadIdx.x;
    if (P.tgt == nullptr) return;
    if (t < 6) {
        s->tgt[t] = P.tgt[6 * b + t];
    } else if (t < 10) {
        const int q = t - 6;
        s->src[q] = P.rad_src[4 * b + q];
        s->dst[q] = P.rad_dst[4 * b + q];
        s->w[q] = P.rad_w[4 * b + q];
    }
}

// Cell (i, j, kq) of a thread in a k-chunk: rows of one plane, then the next plane.
template <int NI, int NJ>
__device__ __forceinline__ void cell_of_thread(int tid, int& i, int& j, int& kq) {
    i = tid % NI;
    j = (tid / NI) % NJ;
    kq = tid / (NI * NJ);
}

// ---------------------------------------------------------------------------
// One RK stage of one block: boundary -> RHS (3_6/ModEquation.f90:24-162) ->
// u_out = u^n + dt*R/(5-s) (3_6/ModAdvance.f90:87-93).
// FP64 (the mixed stage: stage_march, stage_chunks).
template <int NI, int NJ, int NK, int KPAR, int DIVB>
__global__ void __launch_bounds__(NI* NJ* KPAR)
k_stage(const double* in, const double* un, double* out, DivBArgs psi, Geometry g, StepScalars* sc, int stage,
        int bc_writeback) {
    using T = double;
    using S = Shape<T, NI, NJ, NK, KPAR>;
    const int b = blockIdx.x;
    constexpr int NIP = S::NIP, PL = S::PL, W = S::W, WP = S::WP, NCELL = S::NCELL;
    extern __shared__ __align__(128) unsigned char smem[];
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem);
    double* a12 = reinterpret_cast<double*>(smem + S::off_a12);
    T* tile = reinterpret_cast<T*>(smem + S::off_tile);
    T* tp1 = reinterpret_cast<T*>(smem + S::off_p1);
    T* txs = reinterpret_cast<T*>(smem + S::off_xs);   // FP64: [0] Br/sin, [1] E_r/sin (E = v x B)
    T* te2 = reinterpret_cast<T*>(smem + S::off_e2);   // FP64: E_theta, E_r, E_phi
    T* te1 = reinterpret_cast<T*>(smem + S::off_e1);
    T* te3 = reinterpret_cast<T*>(smem + S::off_e3);
    T* gi = reinterpret_cast<T*>(smem + S::off_gi);
    T* gj = reinterpret_cast<T*>(smem + S::off_gj);
    T* gs = reinterpret_cast<T*>(smem + S::off_gs);

    const int fl = g.flags[b];
    const T* blk_in = in + (size_t)b * NV * NCELL;
    T* wb = bc_writeback ? const_cast<T*>(blk_in) : nullptr;
    if (threadIdx.x == 0) {
        mbar_init(&bars[0], 1);
        mbar_init(&bars[1], 1);
        fence_mbar_init();
    }
    __syncthreads();
    if (threadIdx.x == 0) issue_planes<T, S>(blk_in, tile, 0, KPAR + 4, &bars[0]);
    // u^n is read with plain loads at stages 2-4: warm L2 with the planes of the
    // first chunk, then one chunk ahead
    const T* blk_un = un + (size_t)b * NV * NCELL;
    T* blk_out = out + (size_t)b * NV * NCELL;
    auto prefetch_un = [&](int kp_first) {
        if (threadIdx.x >= NV) return;
        const int v = threadIdx.x;
        // the output rows are written in part (interior cells only): their lines into L2 first
        if (out != un || stage == 1) prefetch_l2(blk_out + ((size_t)v * S::NKP + kp_first) * PL, KPAR * S::PLB);
        if (stage == 1) return;
        // u^n is read at interior cells only: its interior rows (2 .. NJ+1 of
        // each plane, one contiguous run) are enough
#pragma unroll
        for (int q = 0; q < KPAR; ++q)
            prefetch_l2(blk_un + ((size_t)v * S::NKP + kp_first + q) * PL + 2 * NIP, (uint32_t)(NJ * NIP * sizeof(T)));
    };
    prefetch_un(2);
    load_geometry<T, S>(g, b, gi, gj, gs, a12);
    __syncthreads();   // the geometry tables are read by every thread below

    const int tid = threadIdx.x;
    int i, j, kq;
    cell_of_thread<NI, NJ>(tid, i, j, kq);
    const int ii = i + 2, jj = j + 2;
    const T c1 = gs[GS_C1], c2 = gs[GS_C2], c3 = gs[GS_C3];
    const T* GR = gi + GI_R * NIP;
    const T* GR2 = gi + GI_R2 * NIP;
    const T* GRHO0 = gi + GI_RHO0 * NIP;
    const T* GSIN = gj + GJ_SIN * S::NJP;
    const T rinv = gi[GI_RINV * NIP + ii], r2inv = gi[GI_R2INV * NIP + ii];
    const T sinv = gj[GJ_SININV * S::NJP + jj], cot = gj[GJ_COT * S::NJP + jj];
    const T rho0c = GRHO0[ii];
    const T gor0 = gi[GI_GOR0 * NIP + ii], heat = gi[GI_HEAT * NIP + ii], xi2inv = gi[GI_XI2INV * NIP + ii];
    const double dt = sc->dt;
    // (dt R) / (5 - stage): for 4, 2, 1 (stages 1, 3, 4) the division is exact and goes
    // into dt, the same bits while dt R / 4 is a normal number; stage 2 divides by 3
    const Divisor three{3.0, 1.0 / 3.0, 1000u};
    const double dts = stage == 2 ? dt : dt / (double)(5.0f - (float)stage);
    auto advance = [&](double R) {   // (dt R) / (5 - stage)
        const double x = dts * R;
        return stage == 2 ? div_by(x, three) : x;
    };
    const Divisor by_rho0 = divisor(rho0c);   // quotients by the cell's rho0
    auto over_rho0 = [&](T x) { return div_by(x, by_rho0); };

    constexpr int nchunk = NK / KPAR;
    const int polls = sc->wait_polls;
    int late = 0;   // a wait of this thread for a chunk's planes ran out
    for (int ch = 0; ch < nchunk; ++ch) {
        const int k0 = 1 + ch * KPAR;  // first Fortran k of the chunk
        const int lo = (ch == 0) ? 0 : k0 + 3;   // first padded plane new to this chunk
        const int hi = k0 + KPAR + 3;            // one past the last plane it needs
        // chunk ch-1 is done with the slots the prefetch below overwrites; a
        // wait of chunk ch-1 that ran out ends the CTA here (chunks ch-1 and ch
        // are in flight)
        if (__syncthreads_or(late)) {
            copy_wait_abort(sc, bars, ch - 1, ch);
            return;
        }
        if (threadIdx.x == 0 && ch + 1 < nchunk)
            issue_planes<T, S>(blk_in, tile, hi, hi + KPAR, &bars[(ch + 1) & 1]);
        if (ch + 1 < nchunk) prefetch_un(k0 + KPAR + 1);
        // a wait that runs out does not leave the chunk (its barriers must be
        // reached by every thread): the chunk computes on whatever the slots
        // hold, the step is flagged and its results are discarded
        late |= mbar_wait(&bars[ch & 1], (uint32_t)((ch >> 1) & 1), polls) ? 0 : 1;
        // u^n for the update (stages 2-4), loaded here so that the latency of
        // these plain loads overlaps the boundary and p1 phases below
        const int kp = k0 + kq + 1;
        const size_t base = (size_t)b * NV * NCELL + (size_t)kp * PL + jj * NIP + ii;
        T u0s[NV];
        if (stage != 1) {
#pragma unroll
            for (int v = 0; v < NV; ++v) u0s[v] = un[base + (size_t)v * NCELL];
        }
        if (fl & 6) {   // radial boundary block (uniform over the CTA)
            apply_bc<T, S>(tile, lo, hi, fl, wb);
            fence_proxy_async();   // order these generic writes before later bulk copies into the slots
            __syncthreads();
        }
        // p1 = gamma1*(p0/rho0)*rho1 + (gamma3-1)*(rho0*T0)*s1, assembled in FP64
        // (3_6/ModEquation.f90:40-46)
        for (int x = tid; x < (hi - lo) * PL; x += S::NT) {
            const int kp = lo + x / PL, c = x % PL, ic = c % NIP;
            const int slot = kp % W;
            const double r1 = tile[(V_RHO1 * W + slot) * PL + c];
            const double s1v = tile[(V_S1 * W + slot) * PL + c];
            tp1[(kp % WP) * PL + c] = a12[ic] * r1 + a12[NIP + ic] * s1v;
            const int jc = c / NIP;
            if (jc >= 2 && jc < NJ + 2) {   // the k-neighbours of interior cells, and E_theta's i-neighbours
                auto at = [&](int v) { return tile[(v * W + slot) * PL + c]; };
                const T vr = at(V_VR), vp = at(V_VP), br = at(V_BR), bp = at(V_BP);
                te2[((kp % WP) * NJ + jc - 2) * NIP + ic] = vp * br - vr * bp;
                if (ic >= 2 && ic < NI + 2) {
                    const Divisor by_sin{gj[GJ_SIN * S::NJP + jc], gj[GJ_SININV * S::NJP + jc], 1000u};
                    T* xs = txs + (kp % WP) * S::PLI + (jc - 2) * NI + ic - 2;
                    xs[0] = div_by(br, by_sin);
                    xs[WP * S::PLI] = div_by(at(V_VT) * bp - vp * at(V_BT), by_sin);
                }
            }
        }
        // E_r and E_phi of the chunk's planes
        for (int x = tid; x < KPAR * PL; x += S::NT) {
            const int q = x / PL, c = x % PL, ic = c % NIP, jc = c / NIP, slot = (k0 + 1 + q) % W;
            const bool in_i = ic >= 2 && ic < NI + 2, in_j = jc >= 2 && jc < NJ + 2;
            if (!in_i && !in_j) continue;
            auto at = [&](int v) { return tile[(v * W + slot) * PL + c]; };
            const T vt = at(V_VT), bt = at(V_BT);
            te3[q * PL + c] = at(V_VR) * bt - vt * at(V_BR);
            if (in_i) te1[(q * S::NJP + jc) * NI + ic - 2] = vt * at(V_BP) - at(V_VP) * bt;
        }
        __syncthreads();

        int sl[5], sp[5];
#pragma unroll
        for (int d = 0; d < 5; ++d) { sl[d] = (kp + d - 2) % W; sp[d] = (kp + d - 2) % WP; }
        auto A = [&](int v, int di, int dj, int dk) -> T {
            return tile[(v * W + sl[dk + 2]) * PL + (jj + dj) * NIP + ii + di];
        };
        auto P = [&](int di, int dj, int dk) -> T { return tp1[sp[dk + 2] * PL + (jj + dj) * NIP + ii + di]; };
        // ModDerivative_1st_O4_3D (3_6/ModDerivative.f90:16-32)
        auto D = [&](T c, auto f) -> T {
            // 8 f is exact, so the FMAs round where the reference's sums do
            return c * (fma(-8.0, f(-1), fma(8.0, f(1), -f(2))) + f(-2));
        };
        const T vr = A(V_VR, 0, 0, 0), vt = A(V_VT, 0, 0, 0), vp = A(V_VP, 0, 0, 0);
        const T br = A(V_BR, 0, 0, 0), bt = A(V_BT, 0, 0, 0), bp = A(V_BP, 0, 0, 0);
        const T rho1 = A(V_RHO1, 0, 0, 0);
        // at stage 1 the input is u^n and sits in the ring
        if (stage == 1) {
#pragma unroll
            for (int v = 0; v < NV; ++v) u0s[v] = A(v, 0, 0, 0);
        }

        // Mass conservation: -div(rho0 v)/Xi^2 (3_6/ModEquation.f90:50-61, ModSpherical_div :104-159)
        T Rrho;
        {
            T dA = D(c1, [&](int m) { return (GRHO0[ii + m] * A(V_VR, m, 0, 0)) * GR2[ii + m]; });
            dA = dA * r2inv;
            T d23 = D(c2, [&](int m) { return (rho0c * A(V_VT, 0, m, 0)) * GSIN[jj + m]; });
            d23 = d23 + D(c3, [&](int m) { return rho0c * A(V_VP, 0, 0, m); });
            d23 = d23 * sinv;
            d23 = d23 * rinv;
            Rrho = -(xi2inv * (dA + d23));
        }
        // A_dot_Grad_f (3_6/ModSpherical.f90:241-279)
        auto adg = [&](int var) -> T {
            T a = vr * D(c1, [&](int m) { return A(var, m, 0, 0); });
            T t = vt * D(c2, [&](int m) { return A(var, 0, m, 0); });
            a = a + t * rinv;
            t = vp * D(c3, [&](int m) { return A(var, 0, 0, m); });
            t = t * rinv;
            a = a + sinv * t;
            return a;
        };
        // Inertial force -(v.grad)v with curvature terms (3_6/ModSpherical.f90:281-343)
        T Rvr, Rvt, Rvp;
        {
            T a1 = adg(V_VR), a2 = adg(V_VT), a3 = adg(V_VP);
            T tmp = -(vt * vt) - vp * vp;
            a1 = a1 + tmp * rinv;
            tmp = -(vp * vp);
            tmp = tmp * cot;
            tmp = tmp + vt * vr;
            a2 = a2 + tmp * rinv;
            tmp = vp * vt;
            tmp = tmp * cot;
            tmp = tmp + vp * vr;
            a3 = a3 + tmp * rinv;
            Rvr = -a1; Rvt = -a2; Rvp = -a3;
        }
        // Pressure gradient -grad(p1)/rho0 (3_6/ModEquation.f90:79-92)
        {
            const T g1 = D(c1, [&](int m) { return P(m, 0, 0); });
            T g2 = D(c2, [&](int m) { return P(0, m, 0); });
            g2 = g2 * rinv;
            T g3 = D(c3, [&](int m) { return P(0, 0, m); });
            g3 = g3 * rinv;
            g3 = g3 * sinv;
            Rvr = Rvr - over_rho0(g1);
            Rvt = Rvt - over_rho0(g2);
            Rvp = Rvp - over_rho0(g3);
        }
        // Lorentz force (curl B) x B / rho0 (3_6/ModEquation.f90:97-116, curl :38-102)
        {
            T k1 = D(c2, [&](int m) { return A(V_BP, 0, m, 0) * GSIN[jj + m]; }) -
                   D(c3, [&](int m) { return A(V_BT, 0, 0, m); });
            // Br / sin(theta) at the k-neighbour m
            auto brs = [&](int m) -> T { return txs[sp[m + 2] * S::PLI + j * NI + i]; };
            T k2 = D(c3, brs) -
                   D(c1, [&](int m) { return A(V_BP, m, 0, 0) * GR[ii + m]; });
            T k3 = D(c1, [&](int m) { return A(V_BT, m, 0, 0) * GR[ii + m]; }) -
                   D(c2, [&](int m) { return A(V_BR, 0, m, 0); });
            k1 = k1 * rinv; k2 = k2 * rinv; k3 = k3 * rinv;
            k1 = k1 * sinv;
            const T x1 = k2 * bp - k3 * bt;
            const T x2 = k3 * br - k1 * bp;
            const T x3 = k1 * bt - k2 * br;
            Rvr = Rvr + over_rho0(x1);
            Rvt = Rvt + over_rho0(x2);
            Rvp = Rvp + over_rho0(x3);
        }
        // Buoyancy -(g/rho0) rho1 (3_6/ModEquation.f90:121-127)
        Rvr = Rvr - gor0 * rho1;
        // Entropy advection and heating (3_6/ModEquation.f90:132-151)
        T Rs = -adg(V_S1);
        Rs = Rs + heat;
        // Induction curl(v x B) (3_6/ModEquation.f90:154-162)
        T RBr, RBt, RBp;
        {
            // from the point arrays: E1 along j, E2 along i and k, E3 along i and j
            auto E1 = [&](int, int bq, int) -> T { return te1[(kq * S::NJP + jj + bq) * NI + i]; };
            auto E2 = [&](int a, int, int c) -> T { return te2[(sp[c + 2] * NJ + j) * NIP + ii + a]; };
            auto E3 = [&](int a, int bq, int) -> T { return te3[kq * PL + (jj + bq) * NIP + ii + a]; };
            T q1 = D(c2, [&](int m) { return E3(0, m, 0) * GSIN[jj + m]; }) - D(c3, [&](int m) { return E2(0, 0, m); });
            // E1 / sin(theta) at the k-neighbour m
            auto e1s = [&](int m) -> T { return txs[(WP + sp[m + 2]) * S::PLI + j * NI + i]; };
            T q2 = D(c3, e1s) -
                   D(c1, [&](int m) { return E3(m, 0, 0) * GR[ii + m]; });
            T q3 = D(c1, [&](int m) { return E2(m, 0, 0) * GR[ii + m]; }) - D(c2, [&](int m) { return E1(0, m, 0); });
            q1 = q1 * rinv; q2 = q2 * rinv; q3 = q3 * rinv;
            q1 = q1 * sinv;
            RBr = q1; RBt = q2; RBp = q3;
        }

        // div-B control. GLM cleaning (3_6/ModDivB.f90:13-38), after the
        // equation terms as 3_6/ModAdvance.f90:82-84 orders it: dB += -grad(psi);
        // dpsi = -v_wave^2 div(B) - v_wave/h_LLL psi, v_wave from u^n. Powell
        // (3_5/ModEquation.f90:169-176): dB += -(div B) v.
        T divB = T(0);
        if constexpr (DIVB != 0) {
            // ModSpherical_div of B (3_6/ModSpherical.f90:104-159)
            T dB = D(c1, [&](int m) { return A(V_BR, m, 0, 0) * GR2[ii + m]; });
            dB = dB * r2inv;
            T e23 = D(c2, [&](int m) { return A(V_BT, 0, m, 0) * GSIN[jj + m]; });
            e23 = e23 + D(c3, [&](int m) { return A(V_BP, 0, 0, m); });
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
            const T* P = static_cast<const T*>(psi.in) + (size_t)b * NCELL + (size_t)kp * PL + jj * NIP + ii;
            auto Q = [&](int di, int dj, int dk) -> T { return P[(size_t)dk * PL + dj * NIP + di]; };
            // ModSpherical_Grad_f (3_6/ModSpherical.f90:201-239)
            const T g1 = D(c1, [&](int m) { return Q(m, 0, 0); });
            T g2 = D(c2, [&](int m) { return Q(0, m, 0); });
            g2 = g2 * rinv;
            T g3 = D(c3, [&](int m) { return Q(0, 0, m); });
            g3 = g3 * rinv;
            g3 = g3 * sinv;
            RBr = RBr - g1;
            RBt = RBt - g2;
            RBp = RBp - g3;
            // ModWaveSpeed_Dynamo (3_6/ModWaveSpeed.f90:8-27) and h_LLL
            // (3_6/ModBlock.f90:416-425) at this cell, as the CFL pass forms them
            T w = gi[GI_CS * NIP + ii] +
                  sqrt(u0s[V_VR] * u0s[V_VR] + u0s[V_VT] * u0s[V_VT] + u0s[V_VP] * u0s[V_VP]);
            w = w + sqrt(u0s[V_BR] * u0s[V_BR] + u0s[V_BT] * u0s[V_BT] + u0s[V_BP] * u0s[V_BP]) / sqrt(rho0c);
            const T rcell = GR[ii];
            const T h = fmin(fmin(gs[GS_DXI], rcell * gs[GS_DXJ]), rcell * GSIN[jj] * gs[GS_DXK]);
            const T Rpsi = -(w * w * divB) - w / h * Q(0, 0, 0);
            const size_t pc = (size_t)b * NCELL + (size_t)kp * PL + jj * NIP + ii;
            const T pn = static_cast<const T*>(psi.un)[pc];
            static_cast<T*>(psi.out)[pc] = pn + advance(Rpsi);
        }

        // stage update
        const T R[NV] = {Rrho, Rvr, Rvt, Rvp, RBr, RBt, RBp, Rs};
#pragma unroll
        for (int v = 0; v < NV; ++v) out[base + (size_t)v * NCELL] = u0s[v] + advance(R[v]);
    }
    if (__syncthreads_or(late)) {
        copy_wait_abort(sc, bars, nchunk - 1, nchunk - 1);
        return;
    }
    if (threadIdx.x == 0) {   // every copy has been waited for
        mbar_inval(&bars[0]);
        mbar_inval(&bars[1]);
    }
}
// ---------------------------------------------------------------------------
// FP64 artificial diffusion (3_6/ModDiffusion.f90:9-150) of one block as a k
// march, in place (the exact path: no pushes, no fused CFL minimum, no u^n
// correction). A thread takes VPT variables of one cell column: 8^3 blocks run
// one variable per thread (512 threads), 16^3 blocks four (512 threads, one
// CTA per SM by shared memory). The k window, slope and face of the thread's
// column stay in registers; across each plane every i and j slope is formed
// once, then every i and j face flux, then each cell sums its six faces in the
// reference's order. Bound by the FP64 pipe, so what counts is FP64
// instructions per cell and variable: the slopes are half_minmod (3 of them
// plus one integer selector, 17 in the formula), a face's difference is the
// slopes' own, its speed sum is formed once for all variables, only faces near
// an extremum divide (face_flux_h) and the sums divide by reciprocals (div_by).
// 442,368 cells, CUDA events: 8^3 blocks 1678 -> 587 us, 16^3 blocks 2385 (chunked
// kernel) -> 731 us (768 and 971 before the limiter's quotient was formed by digits).
template <int NI, int NJ, int NK, int VPT>
struct M64Shape {
    static constexpr int NG = 2, NIP = NI + 4, NJP = NJ + 4, NKP = NK + 4;
    static constexpr int PL = NIP * NJP, NCELL = PL * NKP;
    static constexpr int NCOL = NI * NJ, NT = NCOL * NV / VPT;
    static constexpr int W = 5;                          // plane ring slots
    static constexpr uint32_t PLB = PL * 8u;
    static constexpr int P = NI + 2;                     // row pitch of the slope and face arrays
    // per variable: half slopes SI[NJ][P] (cells i = -1..NI at i + 1), SJ[NJ + 2][P]
    // (rows j = -1..NJ at j + 1), fluxes FI[NJ][P] (faces i - 1/2, i = 0..NI), FJ[NJ + 1][P];
    // speed sums of the plane's faces: VI[NJ][P], VJ[NJ + 1][P], VK[NJ][P] (the face above)
    static constexpr int NSI = NJ * P, NSJ = (NJ + 2) * P, NFI = NJ * P, NFJ = (NJ + 1) * P;
    // shared memory: mbarriers | tile[NV][W][PL] | SI | SJ | FI | FJ | VI | VJ | VK | gi | gj | gs
    static constexpr size_t off_tile = 64;
    static constexpr size_t off_si = off_tile + (size_t)NV * W * PL * 8;
    static constexpr size_t off_sj = off_si + (size_t)NV * NSI * 8;
    static constexpr size_t off_fi = off_sj + (size_t)NV * NSJ * 8;
    static constexpr size_t off_fj = off_fi + (size_t)NV * NFI * 8;
    static constexpr size_t off_vi = off_fj + (size_t)NV * NFJ * 8;
    static constexpr size_t off_vj = off_vi + (size_t)NFI * 8;
    static constexpr size_t off_vk = off_vj + (size_t)NFJ * 8;
    static constexpr size_t off_gi = off_vk + (size_t)NFI * 8;
    static constexpr size_t off_gj = off_gi + (size_t)GI_COUNT * NIP * 8;
    static constexpr size_t off_gs = off_gj + (size_t)GJ_COUNT * NJP * 8;
    static constexpr size_t smem = off_gs + GS_COUNT * 8;
    static_assert(NT <= 1024 && NV % VPT == 0, "whole columns");
    static_assert(smem <= 232448, "227 KB of shared memory per CTA");
};

template <int NI, int NJ, int NK, int VPT>
__global__ void __launch_bounds__(NI * NJ * NV / VPT)
k_diffusion_march64(double* u, Geometry g, StepScalars* sc) {
    using S = M64Shape<NI, NJ, NK, VPT>;
    constexpr int NIP = S::NIP, PL = S::PL, W = S::W, NCELL = S::NCELL, P = S::P;
    extern __shared__ __align__(128) unsigned char smem[];
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem);
    double* tile = reinterpret_cast<double*>(smem + S::off_tile);
    double* SI = reinterpret_cast<double*>(smem + S::off_si);
    double* SJ = reinterpret_cast<double*>(smem + S::off_sj);
    double* FI = reinterpret_cast<double*>(smem + S::off_fi);
    double* FJ = reinterpret_cast<double*>(smem + S::off_fj);
    double* VI = reinterpret_cast<double*>(smem + S::off_vi);
    double* VJ = reinterpret_cast<double*>(smem + S::off_vj);
    double* VK = reinterpret_cast<double*>(smem + S::off_vk);
    double* gi = reinterpret_cast<double*>(smem + S::off_gi);
    double* gj = reinterpret_cast<double*>(smem + S::off_gj);
    double* gs = reinterpret_cast<double*>(smem + S::off_gs);
    const int b = blockIdx.x, tid = threadIdx.x;
    double* blk = u + (size_t)b * NV * NCELL;
    if (tid == 0) {
        for (int q = 0; q < W; ++q) mbar_init(&bars[q], 1);
        fence_mbar_init();
    }
    __syncthreads();
    int issued = 0;   // thread 0: planes [0, issued) have been requested
    if (tid == 0) {
        for (int p = 0; p < W; ++p) issue_planes<double, S>(blk, tile, p, p + 1, &bars[p]);
        issued = W;
    }
    load_geometry<double, S>(g, b, gi, gj, gs, nullptr);
    __syncthreads();
    const int c = tid % S::NCOL, v0 = tid / S::NCOL * VPT;
    const int i = c % NI, j = c / NI, ii = i + 2, jj = j + 2;
    const double* GCS = gi + GI_CS * NIP;
    const double cs = GCS[ii];
    const double rc = gi[GI_R * NIP + ii];
    const Divisor den0 = divisor(gs[GS_DXI]), den1 = divisor(gs[GS_DXJ] * rc),
                  den2 = divisor(gs[GS_DXK] * rc * gj[GJ_SIN * S::NJP + jj]);
    const double hdt = 0.5 * sc->dt;
    const int polls = sc->wait_polls;
    int late = 0;
    auto abort_cta = [&]() {
        if (tid != 0) return;
        atomicOr(&sc->nan_flag, 2);
        for (int p = issued - W < 0 ? 0 : issued - W; p < issued; ++p)
            mbar_wait(&bars[p % W], (uint32_t)((p / W) & 1), kWaitPolls);
        for (int q = 0; q < W; ++q) mbar_inval(&bars[q]);
    };
    const double* col = tile + (size_t)v0 * W * PL + jj * NIP + ii;        // this column, the first variable
    const double* colvp = tile + (size_t)V_VP * W * PL + jj * NIP + ii;    // this column's v_phi
    for (int p = 0; p < 4; ++p) late |= mbar_wait(&bars[p], 0u, polls) ? 0 : 1;
    // per variable: u at kp and kp + 1, their difference, the half slope at kp, the flux below kp
    double u0[VPT], u1[VPT], dk[VPT], hk0[VPT], fk0[VPT];
    {
        const double speed = (fabs(colvp[2 * PL]) + cs) + (fabs(colvp[PL]) + cs);
#pragma unroll
        for (int q = 0; q < VPT; ++q) {
            const double* a = col + q * W * PL;
            const double a0 = a[0], a1 = a[PL], a2 = a[2 * PL], a3 = a[3 * PL];
            const double d0 = a1 - a0, d1 = a2 - a1, d2 = a3 - a2;
            u0[q] = a2;
            u1[q] = a3;
            dk[q] = d2;
            hk0[q] = half_minmod(d1, d2, a3 - a1);
            fk0[q] = face_flux_h(a1, a2, d1, half_minmod(d0, d1, a2 - a0), hk0[q], speed);
        }
    }
    for (int kp = 2; kp < NK + 2; ++kp) {
        const int p2 = kp + 2;
        late |= mbar_wait(&bars[p2 % W], (uint32_t)((p2 / W) & 1), polls) ? 0 : 1;
        const int s0 = (kp % W) * PL, s1 = ((kp + 1) % W) * PL, s2 = (p2 % W) * PL;
        const double* tc = col + s0;   // this cell in plane kp
        // ---- phase A: the k slope of plane kp + 1, the i and j slopes, the speed sums
        double u2[VPT], dk1[VPT], hk1[VPT], dli[VPT], dlj[VPT];
#pragma unroll
        for (int q = 0; q < VPT; ++q) {
            const double* a = tc + q * W * PL;
            u2[q] = col[q * W * PL + s2];
            dk1[q] = u2[q] - u1[q];
            hk1[q] = half_minmod(dk[q], dk1[q], u2[q] - u0[q]);
            const double l = a[-1], r = a[1], d = a[-NIP], t = a[NIP];
            dli[q] = u0[q] - l;
            dlj[q] = u0[q] - d;
            SI[(v0 + q) * S::NSI + j * P + i + 1] = half_minmod(dli[q], r - u0[q], r - l);
            SJ[(v0 + q) * S::NSJ + (j + 1) * P + i] = half_minmod(dlj[q], t - u0[q], t - d);
        }
        // ghost-cell slopes: i = -1, NI of every row, j = -1, NJ of every
        // column; then the faces' speed sums, |v_dir| + c_s on either side
        constexpr int NEI = 2 * NJ * NV, NEJ = 2 * NI * NV;
        constexpr int NVI = NJ * (NI + 1), NVJ = (NJ + 1) * NI, NVK = NJ * NI;
        for (int x = tid; x < NEI + NEJ + NVI + NVJ + NVK; x += S::NT) {
            if (x < NEI + NEJ) {
                const bool on_i = x < NEI;
                const int y = on_i ? x : x - NEI, n = on_i ? NJ : NI;
                const int side = y & 1, r = (y >> 1) % n, w = (y >> 1) / n, st = on_i ? 1 : NIP;
                const double* q = tile + (size_t)w * W * PL + s0 +
                                  (on_i ? (r + 2) * NIP + (side ? NI + 2 : 1) : (side ? NJ + 2 : 1) * NIP + r + 2);
                const double l = q[-st], m = q[0], t = q[st];
                double* dst = on_i ? SI + w * S::NSI + r * P + (side ? NI + 1 : 0)
                                   : SJ + w * S::NSJ + (side ? NJ + 1 : 0) * P + r;
                *dst = half_minmod(m - l, t - m, t - l);
                continue;
            }
            const int y = x - NEI - NEJ;
            if (y < NVI) {
                const int r = y / (NI + 1), e = y % (NI + 1);
                const double* a = tile + (size_t)V_VR * W * PL + s0 + (r + 2) * NIP + e + 1;
                VI[r * P + e] = (fabs(a[1]) + GCS[e + 2]) + (fabs(a[0]) + GCS[e + 1]);
            } else if (y < NVI + NVJ) {
                const int r = (y - NVI) / NI, e = (y - NVI) % NI;
                const double* a = tile + (size_t)V_VT * W * PL + s0 + (r + 1) * NIP + e + 2;
                VJ[r * P + e] = (fabs(a[NIP]) + GCS[e + 2]) + (fabs(a[0]) + GCS[e + 2]);
            } else {
                const int r = (y - NVI - NVJ) / NI, e = (y - NVI - NVJ) % NI;
                const double* a = tile + (size_t)V_VP * W * PL + (r + 2) * NIP + e + 2;
                VK[r * P + e] = (fabs(a[s1]) + GCS[e + 2]) + (fabs(a[s0]) + GCS[e + 2]);
            }
        }
        if (__syncthreads_or(late)) {
            abort_cta();
            return;
        }
        // ---- phase B: the face above this cell and its faces i - 1/2 and j -
        // 1/2; the last faces of the rows and columns
        double fk1[VPT], fi0[VPT], fj0[VPT];
        const double vi = VI[j * P + i], vj = VJ[j * P + i], vk = VK[j * P + i];
#pragma unroll
        for (int q = 0; q < VPT; ++q) {
            const double* a = tc + q * W * PL;
            const double* si = SI + (v0 + q) * S::NSI + j * P + i;
            const double* sj = SJ + (v0 + q) * S::NSJ + j * P + i;
            fk1[q] = face_flux_h(u0[q], u1[q], dk[q], hk0[q], hk1[q], vk);
            fi0[q] = face_flux_h(a[-1], u0[q], dli[q], si[0], si[1], vi);
            fj0[q] = face_flux_h(a[-NIP], u0[q], dlj[q], sj[0], sj[P], vj);
            FI[(v0 + q) * S::NFI + j * P + i] = fi0[q];
            FJ[(v0 + q) * S::NFJ + j * P + i] = fj0[q];
        }
        constexpr int NFE = NJ * NV + NI * NV;
        for (int x = tid; x < NFE; x += S::NT) {
            const bool on_i = x < NJ * NV;
            const int y = on_i ? x : x - NJ * NV, n = on_i ? NJ : NI, r = y % n, w = y / n;
            const double* a = tile + (size_t)w * W * PL + s0 +
                              (on_i ? (r + 2) * NIP + NI + 1 : (NJ + 1) * NIP + r + 2);   // last interior cell
            const double l = a[0], t = on_i ? a[1] : a[NIP];
            const double* h = on_i ? SI + w * S::NSI + r * P + NI : SJ + w * S::NSJ + NJ * P + r;
            const double speed = on_i ? VI[r * P + NI] : VJ[NJ * P + r];
            double* dst = on_i ? FI + w * S::NFI + r * P + NI : FJ + w * S::NFJ + NJ * P + r;
            *dst = face_flux_h(l, t, t - l, h[0], on_i ? h[1] : h[P], speed);
        }
        __syncthreads();
        if (tid == 0) {
            for (; issued < S::NKP && issued <= kp + W; ++issued)
                issue_planes<double, S>(blk, tile, issued, issued + 1, &bars[issued % W]);
        }
        // ---- phase C: the six faces in the reference's order, the update in place
#pragma unroll
        for (int q = 0; q < VPT; ++q) {
            double R = div_by(fi0[q] - FI[(v0 + q) * S::NFI + j * P + i + 1], den0);
            R = R + div_by(fj0[q] - FJ[(v0 + q) * S::NFJ + (j + 1) * P + i], den1);
            R = R + div_by(fk0[q] - fk1[q], den2);
            blk[(size_t)(v0 + q) * NCELL + (size_t)kp * PL + jj * NIP + ii] = u0[q] + hdt * R;
            u0[q] = u1[q];
            u1[q] = u2[q];
            dk[q] = dk1[q];
            hk0[q] = hk1[q];
            fk0[q] = fk1[q];
        }
    }
    if (__syncthreads_or(late)) {
        abort_cta();
        return;
    }
    if (tid == 0)
        for (int q = 0; q < W; ++q) mbar_inval(&bars[q]);
}

// ---------------------------------------------------------------------------
// dt = min(1.e20, CFL*min(h/v_wave)) (3_6/ModTimeStep.f90:20-29); also the
// per-stage FP32 factors of the mixed path and the reset of the accumulator.
// One thread (k_finalize_dt, or the first phase of the persistent step).
__device__ __forceinline__ void finalize_dt_body(StepScalars* sc) {
    const double m = __longlong_as_double((long long)sc->min_ratio_bits);
    const double dt = fmin((double)1.e20f, sc->cfl * m);
    sc->dt = dt;
    for (int s = 1; s <= 4; ++s) sc->dt_stage_f[s - 1] = (float)(dt / (double)(5.0f - (float)s));
    sc->dt_half_f = (float)(0.5 * dt);
    sc->min_ratio_bits = 0x7FF0000000000000ull;   // +inf for the next step
    if (sc->nan_flag && sc->nan_step < 0) sc->nan_step = sc->step_counter;
    sc->step_counter += 1;
}

// The eight values of a cell, p its variable 0 (Layout): FP32 as two 16-byte
// accesses. CG: ld.global.cg (L2 only) -- in the persistent step another SM wrote
// the source cells in the phase before, after this SM may have cached the
// same lines in its L1.
template <bool CG>
__device__ __forceinline__ void load_cell(const double* p, size_t ncell, double (&v)[NV]) {
#pragma unroll
    for (int q = 0; q < NV; ++q) v[q] = CG ? __ldcg(p + q * ncell) : p[q * ncell];
}
template <bool CG>
__device__ __forceinline__ void load_cell(const float* p, size_t ncell, float (&v)[NV]) {
    const float4* f = reinterpret_cast<const float4*>(p);
    const float4 a = CG ? __ldcg(f) : f[0], b = CG ? __ldcg(f + ncell) : f[ncell];
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
__device__ __forceinline__ void store_cell(double* p, size_t ncell, const double (&v)[NV]) {
#pragma unroll
    for (int q = 0; q < NV; ++q) p[q * ncell] = v[q];
}
__device__ __forceinline__ void store_cell(float* p, size_t ncell, const float (&v)[NV]) {
    float4* f = reinterpret_cast<float4*>(p);
    f[0] = make_float4(v[0], v[1], v[2], v[3]);
    f[ncell] = make_float4(v[4], v[5], v[6], v[7]);
}

// ---------------------------------------------------------------------------
// Wave speed (3_6/ModWaveSpeed.f90:8-27), h/v_wave min-reduction
// (3_6/ModTimeStep.f90:10-30) and the NaN scan of 3_6/ModCheck.f90:12-71.
// |x| in FP32, truncated (0 below FP32's range, infinity above and for what is not finite)
__device__ __forceinline__ float magnitude_f(double x) {
    const int hi = __double2hiint(x) & 0x7fffffff, e = (hi >> 20) - 1023 + 127;
    const unsigned m = __funnelshift_l((unsigned)__double2loint(x), (unsigned)hi, 3) & 0x7fffffu;
    return e <= 0 ? 0.f : __int_as_float(e >= 255 ? 0x7f800000 : (int)(m | (unsigned)e << 23));
}
// FP64: the ratio takes about 100 FP64 instructions, and only the smallest counts. An
// FP32 ratio, within 2e-6, first decides which cells can hold the minimum: those
// within 1e-5 of the smallest of their CTA and of what other CTAs have committed so
// far, and cells where FP32's range leaves it open. 442k cells: 67 -> 28 us.
template <class T>
__global__ void __launch_bounds__(256) k_cfl(const T* u, Geometry g, StepScalars* sc, StepDims d) {
    // R: the type the ratio and its block minimum are formed in (FP64 on the
    // exact path, FP32 on the mixed path); the cross-block minimum is FP64.
    using R = T;
    const int nint = d.ni * d.nj * d.nk;
    const int b = blockIdx.y;
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    __shared__ R wmin[8];
    __shared__ int wnan[8];
    R ratio = R(INFINITY);
    int nan = 0;
    const int i = q % d.ni + 2, j = (q / d.ni) % d.nj + 2, k = q / (d.ni * d.nj) + 2;
    const T* Gi = gi_ptr<T>(g) + (size_t)b * GI_COUNT * d.nip + i;
    const T* Gj = gj_ptr<T>(g) + (size_t)b * GJ_COUNT * d.njp + j;
    const T* Gs = gs_ptr<T>(g) + (size_t)b * GS_COUNT;
    T x[NV];
    if (q < nint) load_cell<false>(u + Layout<T>::at(b, 0, ((size_t)k * d.njp + j) * d.nip + i, d.ncell), d.ncell, x);
    if constexpr (Pol<T>::exact) {
        float est = INFINITY;
        bool open = false;
        if (q < nint) {
#pragma unroll
            for (int v = 0; v < NV; ++v) nan |= abs_bits(x[v]) > 0x7ff0000000000000ull;
            const float vr = magnitude_f(x[V_VR]), vt = magnitude_f(x[V_VT]), vp = magnitude_f(x[V_VP]);
            const float br = magnitude_f(x[V_BR]), bt = magnitude_f(x[V_BT]), bp = magnitude_f(x[V_BP]);
            const float r = magnitude_f(Gi[GI_R * d.nip]);
            const float w = magnitude_f(Gi[GI_CS * d.nip]) + sqrtf(vr * vr + vt * vt + vp * vp) +
                            sqrtf(br * br + bt * bt + bp * bp) / sqrtf(magnitude_f(Gi[GI_RHO0 * d.nip]));
            const float h = fminf(fminf(magnitude_f(Gs[GS_DXI]), r * magnitude_f(Gs[GS_DXJ])),
                                  r * magnitude_f(Gj[GJ_SIN * d.njp]) * magnitude_f(Gs[GS_DXK]));
            // (squares that vanished or overflowed in FP32 are too small to count or out of this range)
            open = !(w > 1e-10f && w < 1e15f && h > 1e-15f && h < 1e15f && magnitude_f(Gi[GI_RHO0 * d.nip]) > 1e-20f);
            if (!open) est = h / w;
        }
        float m = est;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = fminf(m, __shfl_xor_sync(0xffffffffu, m, o));
        __shared__ float west[8];
        if (lane == 0) west[wid] = m;
        __syncthreads();
        m = (float)__longlong_as_double((long long)*(volatile unsigned long long*)&sc->min_ratio_bits);
        for (int w2 = 0; w2 < (int)(blockDim.x >> 5); ++w2) m = fminf(m, west[w2]);
        if (q < nint && (open || est <= m * 1.00001f)) {
            // h_LLL = min(dxi, r*dxj, r*sin(theta)*dxk) (3_6/ModBlock.f90:416-425)
            const T r = Gi[GI_R * d.nip];
            const T h = fmin(fmin(Gs[GS_DXI], r * Gs[GS_DXJ]), r * Gj[GJ_SIN * d.njp] * Gs[GS_DXK]);
            T w = Gi[GI_CS * d.nip] + sqrt(x[V_VR] * x[V_VR] + x[V_VT] * x[V_VT] + x[V_VP] * x[V_VP]);
            w = w + sqrt(x[V_BR] * x[V_BR] + x[V_BT] * x[V_BT] + x[V_BP] * x[V_BP]) / sqrt(Gi[GI_RHO0 * d.nip]);
            ratio = h / w;                 // the reference's h_LLL/v_wave
        }
    } else if (q < nint) {
#pragma unroll
        for (int v = 0; v < NV; ++v) nan |= (x[v] != x[v]);
        ratio = cfl_ratio_f(cfl_sq3(x[V_VR], x[V_VT], x[V_VP]), cfl_sq3(x[V_BR], x[V_BT], x[V_BP]), Gi[GI_CS * d.nip],
                            Gi[GI_RHO0 * d.nip], Gi[GI_R * d.nip], Gj[GJ_SIN * d.njp], Gs[GS_DXI], Gs[GS_DXJ], Gs[GS_DXK]);
    }
    if (ratio != ratio) { nan = 1; ratio = R(INFINITY); }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        ratio = fmin(ratio, __shfl_xor_sync(0xffffffffu, ratio, o));
        nan |= __shfl_xor_sync(0xffffffffu, nan, o);
    }
    if (lane == 0) { wmin[wid] = ratio; wnan[wid] = nan; }
    __syncthreads();
    if (threadIdx.x == 0) {
        R m = wmin[0];
        int n = wnan[0];
        for (int w2 = 1; w2 < (int)(blockDim.x >> 5); ++w2) { m = fmin(m, wmin[w2]); n |= wnan[w2]; }
        // positive doubles order like their bit patterns
        if (m < R(INFINITY)) atomicMin(&sc->min_ratio_bits, (unsigned long long)__double_as_longlong((double)m));
        if (n) atomicOr(&sc->nan_flag, 1);
    }
}

// ---------------------------------------------------------------------------
// Ghost fill: the single-GPU form of ModCommunication_SendRecvGC_new
// (3_6/ModCommunication.f90:655-795). Exact copies first, then trilinear
// entries (3_6/ModMath.f90:283-291) with the Yin-Yang vector rotation
// (3_6/ModYinYang.f90:58-60).
// WAIT: step_wait between the entry's own fields and the state.
template <class T, bool CG = false, bool WAIT = false>
__device__ __forceinline__ void ghost_copy_one(T* u, const GhostCopyList& L, int ncell, int64_t e) {
    const size_t src = (size_t)L.src[e], dst = (size_t)L.dst[e];
    if (WAIT) step_wait();
    T v[NV];
    load_cell<CG>(u + src, ncell, v);
    store_cell(u + dst, ncell, v);
}

// one-dimensional linear interpolation (radial neighbours of different
// spacing: the other two weights snapped to exactly 0), mixed path only
template <class T, bool CG = false, bool WAIT = false>
__device__ __forceinline__ void ghost_lin_one(T* u, const GhostLinList& L, int ncell, int64_t e) {
    const T w = (T)L.w[e], uw = T(1) - w;
    const size_t src = (size_t)L.src[e], next = src + (size_t)L.stride[e], dst = (size_t)L.dst[e];
    if (WAIT) step_wait();
    T v[NV], n[NV];
    load_cell<CG>(u + src, ncell, v);
    load_cell<CG>(u + next, ncell, n);
#pragma unroll
    for (int q = 0; q < NV; ++q) v[q] = blend(v[q], n[q], uw, w);
    store_cell(u + dst, ncell, v);
}

template <class T>
__device__ __forceinline__ void ghost_rotate(T (&val)[NV], T a, T c) {
    T x2 = val[V_BT], x3 = val[V_BP];
    val[V_BT] = -(a * x2) - c * x3;
    val[V_BP] = -(a * x3) + c * x2;
    x2 = val[V_VT]; x3 = val[V_VP];
    val[V_VT] = -(a * x2) - c * x3;
    val[V_VP] = -(a * x3) + c * x2;
}
// One interpolated/rotated ghost entry, put(variable, value) for the variables of its
// pairs part, part + parts, .. of four, those that rotate together one after the other
// (a loop, not unrolled: the bodies are long, and two at a time already miss the
// instruction cache).
template <class F>
__device__ __forceinline__ void ghost_interp_each(const double* u, const GhostInterpList& L, int ncell, int nip, int pl,
                                                  int64_t e, F put, int part = 0, int parts = 1) {
    const int kind = L.kind[e];
    const double *f = u + (size_t)L.src[e], *w = L.w + 3 * e;
    const double ra = kind & 2 ? L.rot[2 * e] : 0.0, rc = kind & 2 ? L.rot[2 * e + 1] : 0.0;
    auto each = [&](auto value) {
        double a = 0.0;   // the first of a pair
#pragma unroll 1
        for (int q = 2 * part; q < 8; q += (q & 1) ? 2 * parts - 1 : 1) {   // (rho1, vr), (vt, vp), (bt, bp), (br, s1)
            const int v = 0x74653210 >> (4 * q) & 15;
            double b = value(f + (size_t)v * ncell);
            if ((kind & 2) && (q == 3 || q == 5)) {
                const double x2 = a, x3 = b;
                put(v - 1, -(ra * x2) - rc * x3);
                b = -(ra * x3) + rc * x2;
            }
            if (!((kind & 2) && (q == 2 || q == 4))) put(v, b);
            a = b;
        }
    };
    if (!(kind & 1)) {
        each([&](const double* x) { return x[0]; });
        return;
    }
    const GhostWeights g = ghost_weights(w);
    if (g.near == 7u) {
        const NearEntry n = near_entry(g, nip, pl);
        each([&](const double* x) { return ghost_near(x, w, n, nip, pl); });
    } else if (g.near) {
        const MixedEntry n = mixed_entry(g);
        each([&](const double* x) { return ghost_mixed(x, w, n, nip, pl); });
    } else {
        each([&](const double* x) { return ghost_plain(x, w, nip, pl); });
    }
}
// FP32 weights; the Yin-Yang seam is aligned in r (wi == 0 after snapping), so
// most entries are bilinear in (j, k): four source cells. A cell is two 16-byte
// reads, so an entry's gather touches 8 sectors where [var][cell] order touched 32
// (21.2M cells, all entries of a stage: 114 -> 62 us).
template <bool CG = false, bool WAIT = false>
__device__ __forceinline__ void ghost_interp_vals(const float* u, const GhostInterpList& L, int ncell, int nip, int pl,
                                                  int64_t e, float (&val)[NV]) {
    constexpr int CS = Layout<float>::cell;
    const int kind = L.kind[e];
    const float* s = u + (size_t)L.src[e];
    auto at = [&](int off, float (&v)[NV]) { load_cell<CG>(s + (size_t)CS * off, ncell, v); };
    const float wi = L.wf[3 * e], wj = L.wf[3 * e + 1], wk = L.wf[3 * e + 2];
    const float ui = 1.f - wi, uj = 1.f - wj, uk = 1.f - wk, ra = L.rotf[2 * e], rc = L.rotf[2 * e + 1];
    if (WAIT) step_wait();
    if (!(kind & 1)) {
        at(0, val);
    } else if (wi == 0.f) {
        float f0[NV], f1[NV], f2_[NV], f3[NV];
        at(0, f0); at(nip, f1); at(pl, f2_); at(nip + pl, f3);
#pragma unroll
        for (int v = 0; v < NV; ++v) val[v] = f0[v] * uj * uk + f1[v] * wj * uk + f2_[v] * uj * wk + f3[v] * wj * wk;
    } else {
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            const size_t q = Layout<float>::var(v, ncell);
            auto f = [&](int off) -> float {
                const float* p = s + q + (size_t)CS * off;
                return CG ? __ldcg(p) : *p;
            };
            val[v] = f(0) * ui * uj * uk + f(1) * wi * uj * uk + f(nip) * ui * wj * uk + f(pl) * ui * uj * wk +
                     f(1 + nip) * wi * wj * uk + f(nip + pl) * ui * wj * wk + f(1 + pl) * wi * uj * wk +
                     f(1 + nip + pl) * wi * wj * wk;
        }
    }
    if (kind & 2) ghost_rotate(val, ra, rc);
}
template <bool CG = false, bool WAIT = false>
__device__ __forceinline__ void ghost_interp_one(float* u, const GhostInterpList& L, int ncell, int nip, int pl, int64_t e) {
    float val[NV];
    const size_t dst = (size_t)L.dst[e];
    ghost_interp_vals<CG, WAIT>(u, L, ncell, nip, pl, e, val);
    store_cell(u + dst, ncell, val);
}
template <bool CG = false, bool WAIT = false>
__device__ __forceinline__ void ghost_interp_one(double* u, const GhostInterpList& L, int ncell, int nip, int pl, int64_t e,
                                                 int part = 0, int parts = 1) {
    if (WAIT) step_wait();
    double* to = u + (size_t)L.dst[e];
    ghost_interp_each(u, L, ncell, nip, pl, e, [&](int v, double x) { to[(size_t)v * ncell] = x; }, part, parts);
}

// ---- block sharding: the entries that cross ranks ---------------------------
// The sender evaluates each outgoing ghost entry from its own blocks (the
// same values as the single-GPU ghost fill) into a pack buffer, entry e at
// pack[dst[e]][NV]; the receiver writes pack[e] into its ghost cells (its dst[e], in
// the map's order), as the reference's per-peer send/receive buffers
// (3_6/ModCommunication.f90:725-765).
template <class T>
__global__ void __launch_bounds__(128) k_shard_pack(const T* u, GhostInterpList L, int ncell, int nip, int pl, T* pack, int parts) {
    const int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, e = x >> (parts >> 1);   // parts 1, 2, 4
    if (e >= L.n) return;
    T* to = pack + (size_t)L.dst[e] * NV;
    ghost_interp_each(u, L, ncell, nip, pl, e, [&](int v, T y) { to[v] = y; }, (int)(x & (parts - 1)), parts);
}
template <class T>
__global__ void __launch_bounds__(128) k_shard_unpack(T* u, const int32_t* dst, int64_t n, int ncell, const T* pack) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n) return;
    const size_t d = (size_t)dst[e];
#pragma unroll
    for (int v = 0; v < NV; ++v) u[d + (size_t)v * ncell] = pack[e * NV + v];
}

template <class T>
__global__ void __launch_bounds__(256) k_ghost_copy(T* u, GhostCopyList L, int ncell) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e < L.n) ghost_copy_one(u, L, ncell, e);
}
template <class T>
__global__ void __launch_bounds__(256) k_ghost_lin(T* u, GhostLinList L, int ncell) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e < L.n) ghost_lin_one(u, L, ncell, e);
}
template <class T>
__global__ void __launch_bounds__(128) k_ghost_interp(T* u, GhostInterpList L, int ncell, int nip, int pl) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e < L.n) ghost_interp_one(u, L, ncell, nip, pl, e);
}
// The three lists of one exchange in one launch: every entry reads interior
// cells and writes a ghost cell that no other entry writes, so the lists are
// independent. The interpolated entries (the longest) take the first CTAs, FP64 ones
// `parts` threads each (1, 2 or 4: ghost_parts).
template <class T>
__global__ void __launch_bounds__(128) k_ghost_all(T* u, GhostLists G, int ncell, int nip, int pl, int nb_ip, int nb_ln, int parts) {
    const int bx = blockIdx.x;
    step_go();
    if (bx < nb_ip) {
        const int64_t x = (int64_t)bx * 128 + threadIdx.x;
        if constexpr (sizeof(T) == 8) {
            const int64_t e = x >> (parts >> 1);   // parts 1, 2, 4: shifts 0, 1, 2
            if (e < G.ip.n) ghost_interp_one<false, true>(u, G.ip, ncell, nip, pl, e, (int)(x & (parts - 1)), parts);
        } else {
            if (x < G.ip.n) ghost_interp_one<false, true>(u, G.ip, ncell, nip, pl, x);
        }
    } else if (bx < nb_ip + nb_ln) {
        const int64_t e = (int64_t)(bx - nb_ip) * 128 + threadIdx.x;
        if (e < G.ln.n) ghost_lin_one<T, false, true>(u, G.ln, ncell, e);
    } else {
        const int64_t e = (int64_t)(bx - nb_ip - nb_ln) * 128 + threadIdx.x;
        if (e < G.cp.n) ghost_copy_one<T, false, true>(u, G.cp, ncell, e);
    }
}

// ---------------------------------------------------------------------------
// GLM psi: artificial diffusion (3_6/ModDiffusion.f90:9-150 applies to every
// variable, psi included) into psi_out = psi + dt/2 R_psi, the same formulas
// as the diffusion of u, with psi read from global memory; wave speeds from u.
template <class T>
__global__ void __launch_bounds__(256) k_psi_diffusion(const T* u, const T* psi, T* psi_out, Geometry g,
                                                       StepScalars* sc, StepDims d) {
    const int nint = d.ni * d.nj * d.nk;
    const int b = blockIdx.y;
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= nint) return;
    const int ii = q % d.ni + 2, jj = (q / d.ni) % d.nj + 2, kp = q / (d.ni * d.nj) + 2;
    const size_t pl = (size_t)d.nip * d.njp;
    const size_t c0 = (size_t)b * d.ncell + (size_t)kp * pl + (size_t)jj * d.nip + ii;
    const T* Gi = gi_ptr<T>(g) + (size_t)b * GI_COUNT * d.nip;
    const T* Gj = gj_ptr<T>(g) + (size_t)b * GJ_COUNT * d.njp;
    const T* Gs = gs_ptr<T>(g) + (size_t)b * GS_COUNT;
    const T* GCS = Gi + GI_CS * d.nip;
    const T rc = Gi[GI_R * d.nip + ii];
    const T den[3] = {Gs[GS_DXI], Gs[GS_DXJ] * rc, Gs[GS_DXK] * rc * Gj[GJ_SIN * d.njp + jj]};
    const size_t strides[3] = {1, (size_t)d.nip, pl};
    T R = T(0);
#pragma unroll
    for (int dir = 0; dir < 3; ++dir) {
        const size_t s = strides[dir];
        const T* vd = u + Layout<T>::at(b, V_VR + dir, c0 - (size_t)b * d.ncell, d.ncell);
        const ptrdiff_t vs = (ptrdiff_t)(s * Layout<T>::cell);
        auto at = [&](int m) -> T { return psi[(ptrdiff_t)c0 + (ptrdiff_t)m * (ptrdiff_t)s]; };
        const T csm = dir == 0 ? GCS[ii - 1] : GCS[ii];
        const T cs0 = GCS[ii];
        const T csp = dir == 0 ? GCS[ii + 1] : GCS[ii];
        const T cm = fabs(vd[-vs]) + csm, cz = fabs(vd[0]) + cs0, cp = fabs(vd[vs]) + csp;
        const T fm2 = at(-2), fm1 = at(-1), f0 = at(0), fp1 = at(1), fp2 = at(2);
        const T dm1 = minmod(fm2, fm1, f0);
        const T d0 = minmod(fm1, f0, fp1);
        const T dp1 = minmod(f0, fp1, fp2);
        T num = ((f0 - d0 * T(0.5)) - fm1) - dm1 * T(0.5);
        T phi = fmax(T(0), T(1) + T(2) * (Pol<T>::ratio(num, f0 - fm1) - T(1)));
        T fL = -(T(0.5) * phi * num);
        fL = fL * (cz + cm) * T(0.5);
        num = ((fp1 - dp1 * T(0.5)) - f0) - d0 * T(0.5);
        phi = fmax(T(0), T(1) + T(2) * (Pol<T>::ratio(num, fp1 - f0) - T(1)));
        T fR = -(T(0.5) * phi * num);
        fR = fR * (cp + cz) * T(0.5);
        R = R + (fL - fR) / den[dir];
    }
    const T p0 = psi[c0];
    T o;
    if constexpr (Pol<T>::exact) o = (T)((double)p0 + (0.5 * sc->dt) * (double)R);
    else o = fmaf(sc->dt_half_f, (float)R, (float)p0);
    psi_out[c0] = o;
}

// GLM psi ghost fill with the state's ghost lists (psi is a scalar: no
// rotation). List offsets address var 0 of a cell of the state (Layout); psi's
// array is [b][cell].
template <class T>
__device__ __forceinline__ size_t psi_off(size_t off, int ncell) {
    const size_t b = off / ((size_t)NV * ncell);
    return b * ncell + (off - b * (size_t)NV * ncell) / Layout<T>::cell;
}
template <class T>
__global__ void __launch_bounds__(256) k_psi_ghost(T* psi, GhostLists L, int ncell, int nip, int pl) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t ncp = L.cp.n, nln = L.ln.n, nip_ = L.ip.n;
    if (e < ncp) {
        psi[psi_off<T>(L.cp.dst[e], ncell)] = psi[psi_off<T>(L.cp.src[e], ncell)];
    } else if (e < ncp + nln) {
        const int64_t q = e - ncp;
        const T* f = psi + psi_off<T>(L.ln.src[q], ncell);
        const T w = (T)L.ln.w[q];
        psi[psi_off<T>(L.ln.dst[q], ncell)] = blend(f[0], f[L.ln.stride[q] / Layout<T>::cell], T(1) - w, w);
    } else if (e < ncp + nln + nip_) {
        const int64_t q = e - ncp - nln;
        const T* f = psi + psi_off<T>(L.ip.src[q], ncell);
        T val;
        if (!(L.ip.kind[q] & 1)) {
            val = f[0];
        } else {
            T wi, wj, wk;
            if constexpr (Pol<T>::exact) { wi = L.ip.w[3 * q]; wj = L.ip.w[3 * q + 1]; wk = L.ip.w[3 * q + 2]; }
            else { wi = L.ip.wf[3 * q]; wj = L.ip.wf[3 * q + 1]; wk = L.ip.wf[3 * q + 2]; }
            const T ui = T(1) - wi, uj = T(1) - wj, uk = T(1) - wk;
            val = f[0] * ui * uj * uk + f[1] * wi * uj * uk + f[nip] * ui * wj * uk + f[pl] * ui * uj * wk +
                  f[1 + nip] * wi * wj * uk + f[nip + pl] * ui * wj * wk + f[1 + pl] * wi * uj * wk +
                  f[1 + nip + pl] * wi * wj * wk;
        }
        psi[psi_off<T>(L.ip.dst[q], ncell)] = val;
    }
}

}  // namespace impl
}  // namespace falcon
