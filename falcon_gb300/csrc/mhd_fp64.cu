// mhd_fp64.cu -- FP64 instantiation of the step kernels.
// Compiled with -fmad=false: no multiply-add contraction, so every result is
// rounded exactly where the reference rounds (it is built without FMA).
#include "launch_impl.cuh"

namespace falcon {
using impl::cfl_any;
using impl::ghost_any;

namespace impl {
namespace {
// k-chunk depths (KPAR) instantiated per block size; the context's autotuner
// times them on its own grid and keeps the fastest.
template <int N, int KP, int DIVB>
cudaError_t stage_nd(const StepDims& d, const Geometry& g, const double* in, const double* un, double* out,
                     const DivBArgs& psi, int stage, int bcw, StepScalars* sc, cudaStream_t st) {
    using S = Shape<double, N, N, N, KP>;
    static OncePerDevice once;
    const cudaError_t attr = allow_smem(once, k_stage<N, N, N, KP, DIVB>, S::smem_stage);
    if (attr != cudaSuccess) return attr;
    k_stage<N, N, N, KP, DIVB><<<d.nblocks, S::NT, S::smem_stage, st>>>(in, un, out, psi, g, sc, stage, bcw);
    return cudaGetLastError();
}
// The div-B mode is a template parameter: the plain stage keeps its register
// allocation free of the GLM/Powell terms.
template <int N, int KP>
cudaError_t stage_n(const StepDims& d, const Geometry& g, const double* in, const double* un, double* out,
                    const DivBArgs& psi, int stage, int bcw, StepScalars* sc, cudaStream_t st) {
    switch (psi.mode) {
    case 0: return stage_nd<N, KP, 0>(d, g, in, un, out, psi, stage, bcw, sc, st);
    case 1:
        if (!psi.in || !psi.un || !psi.out) return cudaErrorInvalidValue;
        return stage_nd<N, KP, 1>(d, g, in, un, out, psi, stage, bcw, sc, st);
    case 2: return stage_nd<N, KP, 2>(d, g, in, un, out, psi, stage, bcw, sc, st);
    default: return cudaErrorInvalidValue;
    }
}
// the k march, in place
template <int N, int VPT>
cudaError_t diff_march64(const StepDims& d, const Geometry& g, double* u, StepScalars* sc, cudaStream_t st) {
    using S = M64Shape<N, N, N, VPT>;
    static OncePerDevice once;
    const cudaError_t attr = allow_smem(once, k_diffusion_march64<N, N, N, VPT>, S::smem);
    if (attr != cudaSuccess) return attr;
    k_diffusion_march64<N, N, N, VPT><<<d.nblocks, S::NT, S::smem, st>>>(u, g, sc);
    return cudaGetLastError();
}
}  // namespace
}  // namespace impl

cudaError_t launch_stage_fp64(const StepDims& d, const Geometry& g, const double* in, const double* un, double* out,
                              const DivBArgs& psi, int stage, int bcw, StepScalars* sc, int kpar, cudaStream_t st) {
    if (d.ni != d.nj || d.ni != d.nk) return cudaErrorInvalidValue;
    if (d.ni == 8 && kpar == 2) return impl::stage_n<8, 2>(d, g, in, un, out, psi, stage, bcw, sc, st);
    if (d.ni == 8 && kpar == 4) return impl::stage_n<8, 4>(d, g, in, un, out, psi, stage, bcw, sc, st);
    if (d.ni == 16 && kpar == 1) return impl::stage_n<16, 1>(d, g, in, un, out, psi, stage, bcw, sc, st);
    return cudaErrorInvalidValue;
}
// (any k-chunk depth asked for: the march has one form)
cudaError_t launch_diffusion_fp64(const StepDims& d, const Geometry& g, double* u, StepScalars* sc, cudaStream_t st) {
    if (d.ni != d.nj || d.ni != d.nk) return cudaErrorInvalidValue;
    if (d.ni == 8) return impl::diff_march64<8, 1>(d, g, u, sc, st);
    if (d.ni == 16) return impl::diff_march64<16, 4>(d, g, u, sc, st);
    return cudaErrorInvalidValue;
}
cudaError_t launch_psi_diffusion_fp64(const StepDims& d, const Geometry& g, const double* u, const double* psi,
                                      double* psi_out, StepScalars* sc, cudaStream_t st) {
    return impl::psi_diffusion_any<double>(d, g, u, psi, psi_out, sc, st);
}
cudaError_t launch_psi_ghost_fp64(const StepDims& d, const GhostLists& gl, double* psi, cudaStream_t st) {
    return impl::psi_ghost_any<double>(d, gl, psi, st);
}
cudaError_t launch_cfl_fp64(const StepDims& d, const Geometry& g, const double* u, StepScalars* sc, cudaStream_t st) {
    return cfl_any<double>(d, g, u, sc, st);
}
cudaError_t launch_ghost_fp64(const StepDims& d, const GhostLists& gl, double* u, cudaStream_t st) {
    return ghost_any<double>(d, gl, u, st);
}
cudaError_t launch_shard_pack_fp64(const StepDims& d, const GhostInterpList& L, const double* u, double* pack,
                                   cudaStream_t st) {
    if (L.n == 0) return cudaSuccess;
    const int parts = impl::ghost_parts(L.n);
    impl::k_shard_pack<double><<<(unsigned)((L.n * parts + 127) / 128), 128, 0, st>>>(u, L, d.ncell, d.nip, d.nip * d.njp, pack, parts);
    return cudaGetLastError();
}
cudaError_t launch_shard_unpack_fp64(const StepDims& d, const int32_t* dst, int64_t n, const double* pack, double* u,
                                     cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    impl::k_shard_unpack<double><<<(unsigned)((n + 127) / 128), 128, 0, st>>>(u, dst, n, d.ncell, pack);
    return cudaGetLastError();
}

// dt = min(1.e20, CFL*min(h/v_wave)) (3_6/ModTimeStep.f90:20-29); also the
// per-stage FP32 factors of the mixed path and the reset of the accumulator.
__global__ void k_finalize_dt(StepScalars* sc) {
    impl::step_go();
    impl::finalize_dt_body(sc);
}
cudaError_t launch_finalize_dt(StepScalars* sc, cudaStream_t st) {
    k_finalize_dt<<<1, 1, 0, st>>>(sc);
    return cudaGetLastError();
}

// Host block arrays carry FALCON_NVAR = 9 variables ([b][9][cell], psi last);
// the device state the 8 evolved ones (see Layout) and, with GLM, psi in an
// array of its own ([b][cell]). x counts (block, variable, cell) with the cell fastest.
__device__ __forceinline__ int64_t host_index(int64_t x, int64_t ncell) {   // -> host element
    const int64_t b = x / (NV * ncell);
    return x + b * ncell;
}

// FP64 host array -> compensated FP32 state: hi = RN(u); interior cells get
// the correction of u - hi, ghost cells q = 0
__device__ __forceinline__ void narrow_one(double u, int64_t x, float* d, int8_t* lo, const StepDims& dm) {
    const float hi = (float)u;
    const int64_t bv = x / dm.ncell, b = bv / NV;
    const int v = (int)(bv - b * NV), c = (int)(x - bv * dm.ncell);
    d[Layout<float>::at((size_t)b, v, (size_t)c, (size_t)dm.ncell)] = hi;
    if (lo) {
        const int64_t q = lo_index(b, v, c, dm);
        if (q >= 0) lo[q] = lo_encode64(hi, u - (double)hi);
    }
}
__global__ void k_narrow(const double* s, float* d, int8_t* lo, int64_t n, StepDims dm) {
    for (int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; x < n; x += (int64_t)gridDim.x * blockDim.x)
        narrow_one(s[host_index(x, dm.ncell)], x, d, lo, dm);
}
// psi plane of the host array -> FP32 psi array (mixed GLM)
__global__ void k_narrow_psi(const double* s, float* psi, int64_t nb, int64_t ncell) {
    for (int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; x < nb * ncell; x += (int64_t)gridDim.x * blockDim.x) {
        const int64_t b = x / ncell;
        psi[x] = (float)s[(b * (NV + 1) + NV) * ncell + (x - b * ncell)];
    }
}
// flag = 1 if any psi value of the host array (already on the device) is
// not 0 (NaN counts as not 0)
__global__ void k_psi_nonzero(const double* s, int64_t nb, int64_t ncell, int32_t* flag) {
    int any = 0;
    for (int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; x < nb * ncell; x += (int64_t)gridDim.x * blockDim.x) {
        const int64_t b = x / ncell;
        any |= s[(b * (NV + 1) + NV) * ncell + (x - b * ncell)] != 0.0;
    }
    if (__any_sync(0xffffffffu, any) && (threadIdx.x & 31) == 0) *flag = 1;
}
// Wide forms of the transfer kernels: each thread moves kWide elements per
// pass as kWide/2 16-byte accesses, all issued before any is used (a warp's
// access q covers 512 contiguous bytes), so that many bytes are in flight when
// the FP64 side is host memory read or written in place over the host link. They need 16-byte-aligned FP64
// arrays, an even cell count and even ranges (pairs never straddle a
// variable); the launchers fall back to the one-element kernels otherwise.
constexpr int kWide = 8;
__global__ void k_narrow_wide(const double* s, float* d, int8_t* lo, int64_t n, StepDims dm) {
    const int64_t lane2 = 2 * (threadIdx.x & 31);
    for (int64_t w0 = (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 32 * kWide; w0 < n;
         w0 += (((int64_t)gridDim.x * blockDim.x) >> 5) * 32 * kWide) {
        double2 v[kWide / 2];
#pragma unroll
        for (int q = 0; q < kWide / 2; ++q)
            if ((w0 + 64 * q + lane2) < n) v[q] = *reinterpret_cast<const double2*>(s + host_index((w0 + 64 * q + lane2), dm.ncell));
#pragma unroll
        for (int q = 0; q < kWide / 2; ++q)
            if ((w0 + 64 * q + lane2) < n) {
                narrow_one(v[q].x, (w0 + 64 * q + lane2), d, lo, dm);
                narrow_one(v[q].y, (w0 + 64 * q + lane2) + 1, d, lo, dm);
            }
    }
}
__device__ __forceinline__ int64_t psi_host_index(int64_t x, int64_t ncell) {   // psi element -> host element
    const int64_t b = x / ncell;
    return (b * (NV + 1) + NV) * ncell + (x - b * ncell);
}
__global__ void k_narrow_psi_wide(const double* s, float* psi, int64_t nb, int64_t ncell) {
    const int64_t n = nb * ncell;
    const int64_t lane2 = 2 * (threadIdx.x & 31);
    for (int64_t w0 = (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 32 * kWide; w0 < n;
         w0 += (((int64_t)gridDim.x * blockDim.x) >> 5) * 32 * kWide) {
        double2 v[kWide / 2];
#pragma unroll
        for (int q = 0; q < kWide / 2; ++q)
            if ((w0 + 64 * q + lane2) < n) v[q] = *reinterpret_cast<const double2*>(s + psi_host_index((w0 + 64 * q + lane2), ncell));
#pragma unroll
        for (int q = 0; q < kWide / 2; ++q)
            if ((w0 + 64 * q + lane2) < n) {
                psi[(w0 + 64 * q + lane2)] = (float)v[q].x;
                psi[(w0 + 64 * q + lane2) + 1] = (float)v[q].y;
            }
    }
}
__global__ void k_psi_nonzero_wide(const double* s, int64_t nb, int64_t ncell, int32_t* flag) {
    const int64_t n = nb * ncell;
    int any = 0;
    const int64_t lane2 = 2 * (threadIdx.x & 31);
    for (int64_t w0 = (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 32 * kWide; w0 < n;
         w0 += (((int64_t)gridDim.x * blockDim.x) >> 5) * 32 * kWide) {
        double2 v[kWide / 2];
#pragma unroll
        for (int q = 0; q < kWide / 2; ++q)
            if ((w0 + 64 * q + lane2) < n) v[q] = *reinterpret_cast<const double2*>(s + psi_host_index((w0 + 64 * q + lane2), ncell));
#pragma unroll
        for (int q = 0; q < kWide / 2; ++q)
            if ((w0 + 64 * q + lane2) < n) any |= (v[q].x != 0.0) | (v[q].y != 0.0);
    }
    if (__any_sync(0xffffffffu, any) && (threadIdx.x & 31) == 0) *flag = 1;
}
// host element h as FP64 from the device state (FP32 with its correction, or
// FP64) and psi (nullptr: psi = 0)
template <class T>
__device__ __forceinline__ double gather_one(const T* U, const int8_t* lo, const T* psi, int64_t h, int64_t ncell,
                                             const StepDims& dm) {
    const int64_t b = h / ((NV + 1) * ncell), r = h - b * (NV + 1) * ncell;
    if (r < NV * ncell) {
        if constexpr (sizeof(T) == 8) return U[b * NV * ncell + r];   // the host's order
        const int v = (int)(r / ncell), c = (int)(r - v * ncell);
        const T hi = U[Layout<T>::at((size_t)b, v, (size_t)c, (size_t)ncell)];
        double x = (double)hi;
        if constexpr (sizeof(T) == 4) {
            const int64_t q = lo ? lo_index(b, v, c, dm) : -1;
            if (q >= 0) x += (double)lo[q] * (double)lo_unit((float)hi);
        }
        return x;
    }
    return psi ? (double)psi[b * ncell + (r - NV * ncell)] : 0.0;
}
template <class T>
__global__ void k_gather_host(const T* U, const int8_t* lo, const T* psi, StepDims dm, int64_t first, int64_t count,
                              int64_t ncell, double* out) {
    for (int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; x < count; x += (int64_t)gridDim.x * blockDim.x)
        out[x] = gather_one(U, lo, psi, first + x, ncell, dm);
}
template <class T>
__global__ void k_gather_host_wide(const T* U, const int8_t* lo, const T* psi, StepDims dm, int64_t first,
                                   int64_t count, int64_t ncell, double* out) {
    const int64_t lane2 = 2 * (threadIdx.x & 31);
    for (int64_t w0 = (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 32 * kWide; w0 < count;
         w0 += (((int64_t)gridDim.x * blockDim.x) >> 5) * 32 * kWide) {
        double2 v[kWide / 2];
#pragma unroll
        for (int q = 0; q < kWide / 2; ++q)
            if ((w0 + 64 * q + lane2) < count) {
                v[q].x = gather_one(U, lo, psi, first + (w0 + 64 * q + lane2), ncell, dm);
                v[q].y = gather_one(U, lo, psi, first + (w0 + 64 * q + lane2) + 1, ncell, dm);
            }
#pragma unroll
        for (int q = 0; q < kWide / 2; ++q)
            if ((w0 + 64 * q + lane2) < count) *reinterpret_cast<double2*>(out + (w0 + 64 * q + lane2)) = v[q];
    }
}
bool wide_ok(const void* p, int64_t ncell) { return ((uintptr_t)p % 16) == 0 && ncell % 2 == 0; }

// Core transfers: of every block and variable of the host array (9 per block,
// psi last), the interior planes and within them the interior rows, each
// row whole (its radial ghost columns, which hold the radial boundary
// condition, included). The interior rows of one plane are one contiguous
// run of (NJP-4)*NIP host elements. A warp takes pieces of the runs of one plane of one
// group of a block's variables -- four that the mixed state holds side by side (FP64:
// one), or psi -- so no element pays a 64-bit division (a piece does) and the mixed
// state's side is whole 16-byte cells; a lane's 16-byte host accesses of a piece (two
// cells of every variable, PASS passes) are issued before any is used. Offsets are
// even and NIP is even, so a pair (ip, ip+1) is either two radial ghost columns or
// two interior cells.
template <class T, int PASS> struct CoreRun {
    static constexpr int G = sizeof(T) == 4 ? 4 : 1;    // variables of a group
    static constexpr int NG = NV / G + 1;               // groups, psi last
    static constexpr int kPass = PASS;
    __host__ __device__ static int length(const StepDims& dm) { return (dm.njp - 4) * dm.nip; }
    __host__ __device__ static int pieces(const StepDims& dm) { return (length(dm) + 64 * kPass - 1) / (64 * kPass); }
    int64_t b, cell0;   // block, padded cell of the run's first element
    int g;
    int kp;
    __device__ CoreRun(int64_t r, const StepDims& dm) {
        const int nkc = dm.nkp - 4;
        const int64_t bg = r / nkc;
        b = bg / NG;
        g = (int)(bg - b * NG);
        kp = 2 + (int)(r - bg * nkc);
        cell0 = (int64_t)kp * dm.nip * dm.njp + 2 * dm.nip;
    }
    __device__ bool psi() const { return g == NG - 1; }
    __device__ int vars() const { return psi() ? 1 : G; }
    // host element of variable q of the group at offset o of the run
    __device__ int64_t host(int q, int o, const StepDims& dm) const { return (b * (NV + 1) + g * G + q) * dm.ncell + cell0 + o; }
    // correction of the cells at offset o (mixed): interior cells of the plane's interior rows
    __device__ int64_t lo(int o, const StepDims& dm) const {
        const int jr = o / dm.nip;
        return (((b * dm.nk + (kp - 2)) * dm.nj + jr) * dm.ni + (o - jr * dm.nip - 2)) * NV + g * G;
    }
    __device__ bool interior(int o, const StepDims& dm) const {
        const int ip = o % dm.nip;
        return ip >= 2 && ip < dm.nip - 2;
    }
};
// host core -> device: state cells narrowed (FP32 with its correction) or
// copied (FP64); psi converted into P, or, without P, tested for 0 (flag)
template <class T, int PASS>
__global__ void k_core_up(const double* s, T* U, int8_t* lo, T* P, int32_t* flag, int64_t nruns, StepDims dm) {
    using R = CoreRun<T, PASS>;
    const int lane2 = 2 * (threadIdx.x & 31), len = R::length(dm), pieces = R::pieces(dm);
    int any = 0;
    for (int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < nruns * pieces;
         w += ((int64_t)gridDim.x * blockDim.x) >> 5) {
        const int64_t r = w / pieces;
        const R c(r, dm);
        const int nv = c.vars();
        const int o0 = (int)(w - r * pieces) * 64 * R::kPass;
        double2 v[R::kPass][R::G];
#pragma unroll
        for (int q = 0; q < R::kPass; ++q)
#pragma unroll
            for (int g = 0; g < R::G; ++g)
                if (o0 + 64 * q + lane2 < len && g < nv)
                    v[q][g] = *reinterpret_cast<const double2*>(s + c.host(g, o0 + 64 * q + lane2, dm));
#pragma unroll
        for (int q = 0; q < R::kPass; ++q) {
            const int o = o0 + 64 * q + lane2;
            if (o >= len) continue;
            const int64_t pc = c.b * dm.ncell + c.cell0 + o;   // the cells in a [b][cell] array
            if (c.psi()) {
                if (!P) {
                    any |= (v[q][0].x != 0.0) | (v[q][0].y != 0.0);
                } else if constexpr (sizeof(T) == 4) {
                    *reinterpret_cast<float2*>(P + pc) = make_float2((float)v[q][0].x, (float)v[q][0].y);
                } else {
                    *reinterpret_cast<double2*>(P + pc) = v[q][0];
                }
                continue;
            }
            if constexpr (sizeof(T) == 4) {
                float4* out = reinterpret_cast<float4*>(U) + (c.b * 2 + c.g) * dm.ncell + c.cell0 + o;
                const float4 a = make_float4((float)v[q][0].x, (float)v[q][1].x, (float)v[q][2].x, (float)v[q][3].x);
                const float4 e = make_float4((float)v[q][0].y, (float)v[q][1].y, (float)v[q][2].y, (float)v[q][3].y);
                out[0] = a;
                out[1] = e;
                if (lo && c.interior(o, dm)) {
                    int8_t* l = lo + c.lo(o, dm);
                    *reinterpret_cast<char4*>(l) =
                        make_char4(lo_encode64(a.x, v[q][0].x - (double)a.x), lo_encode64(a.y, v[q][1].x - (double)a.y),
                                   lo_encode64(a.z, v[q][2].x - (double)a.z), lo_encode64(a.w, v[q][3].x - (double)a.w));
                    *reinterpret_cast<char4*>(l + NV) =
                        make_char4(lo_encode64(e.x, v[q][0].y - (double)e.x), lo_encode64(e.y, v[q][1].y - (double)e.y),
                                   lo_encode64(e.z, v[q][2].y - (double)e.z), lo_encode64(e.w, v[q][3].y - (double)e.w));
                }
            } else {
                *reinterpret_cast<double2*>(U + Layout<T>::at((size_t)c.b, c.g, (size_t)(c.cell0 + o), (size_t)dm.ncell)) = v[q][0];
            }
        }
    }
    if (flag && __any_sync(0xffffffffu, any) && (threadIdx.x & 31) == 0) *flag = 1;
}
// device -> host core (psi 0 without P)
template <class T, int PASS>
__global__ void k_core_down(const T* U, const int8_t* lo, const T* P, double* out, int64_t nruns, StepDims dm) {
    using R = CoreRun<T, PASS>;
    const int lane2 = 2 * (threadIdx.x & 31), len = R::length(dm), pieces = R::pieces(dm);
    for (int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < nruns * pieces;
         w += ((int64_t)gridDim.x * blockDim.x) >> 5) {
        const int64_t r = w / pieces;
        const R c(r, dm);
        const int nv = c.vars();
        const int o0 = (int)(w - r * pieces) * 64 * R::kPass;
        double2 v[R::kPass][R::G];
#pragma unroll
        for (int q = 0; q < R::kPass; ++q) {
            const int o = o0 + 64 * q + lane2;
            if (o >= len) continue;
            const int64_t pc = c.b * dm.ncell + c.cell0 + o;
            if (c.psi()) {
                v[q][0] = make_double2(0.0, 0.0);
                if (P) v[q][0] = make_double2((double)P[pc], (double)P[pc + 1]);
                continue;
            }
            if constexpr (sizeof(T) == 4) {
                const float4* in = reinterpret_cast<const float4*>(U) + (c.b * 2 + c.g) * dm.ncell + c.cell0 + o;
                const float4 a = in[0], e = in[1];
                const float h0[4] = {a.x, a.y, a.z, a.w}, h1[4] = {e.x, e.y, e.z, e.w};
                char4 l0 = make_char4(0, 0, 0, 0), l1 = l0;
                const bool add = lo && c.interior(o, dm);
                if (add) {
                    const int8_t* l = lo + c.lo(o, dm);
                    l0 = *reinterpret_cast<const char4*>(l);
                    l1 = *reinterpret_cast<const char4*>(l + NV);
                }
                const int8_t q0[4] = {l0.x, l0.y, l0.z, l0.w}, q1[4] = {l1.x, l1.y, l1.z, l1.w};
#pragma unroll
                for (int g = 0; g < R::G; ++g) {
                    v[q][g] = make_double2((double)h0[g], (double)h1[g]);
                    if (add) {
                        v[q][g].x += (double)q0[g] * (double)lo_unit(h0[g]);
                        v[q][g].y += (double)q1[g] * (double)lo_unit(h1[g]);
                    }
                }
            } else {
                v[q][0] = *reinterpret_cast<const double2*>(U + Layout<T>::at((size_t)c.b, c.g, (size_t)(c.cell0 + o), (size_t)dm.ncell));
            }
        }
#pragma unroll
        for (int g = 0; g < R::G; ++g)
#pragma unroll
            for (int q = 0; q < R::kPass; ++q)
                if (o0 + 64 * q + lane2 < len && g < nv)
                    *reinterpret_cast<double2*>(out + c.host(g, o0 + 64 * q + lane2, dm)) = v[q][g];
    }
}
template <class T> int64_t core_runs(const StepDims& dm) { return (int64_t)dm.nblocks * CoreRun<T, 1>::NG * (dm.nkp - 4); }
constexpr unsigned kCoreGrid = 1216, kCoreThreads = 256;
// Mixed: pieces of two passes while they outnumber the grid's warps, else of one. 12
// blocks of 8^3 to the host 21 / 18 us, 192 blocks 71 / 69; 5,184 blocks of 16^3 from the
// host 10.42 / 10.74 ms. (A whole run per warp: 12 blocks of 16^3 39 us, in pieces 36.)
bool core_short_pieces(const StepDims& dm) {
    return core_runs<float>(dm) * CoreRun<float, 2>::pieces(dm) < (int64_t)kCoreGrid * kCoreThreads / 32;
}
bool core_ok(const void* host, const StepDims& dm) {
    return ((uintptr_t)host % 16) == 0 && dm.ncell % 2 == 0 && dm.nip % 2 == 0;
}

cudaError_t launch_convert_state(const double* src, float* dst, int8_t* lo, int64_t n, const StepDims& dm,
                                 cudaStream_t st) {
    if (wide_ok(src, dm.ncell) && n % 2 == 0) k_narrow_wide<<<1216, 256, 0, st>>>(src, dst, lo, n, dm);
    else k_narrow<<<1216, 256, 0, st>>>(src, dst, lo, n, dm);
    return cudaGetLastError();
}
cudaError_t launch_convert_psi(const double* src, float* psi, int64_t nb, int64_t ncell, cudaStream_t st) {
    if (wide_ok(src, ncell)) k_narrow_psi_wide<<<1216, 256, 0, st>>>(src, psi, nb, ncell);
    else k_narrow_psi<<<1216, 256, 0, st>>>(src, psi, nb, ncell);
    return cudaGetLastError();
}
cudaError_t launch_psi_nonzero(const double* src, int64_t nb, int64_t ncell, int32_t* flag, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(flag, 0, sizeof(int32_t), st);
    if (e != cudaSuccess) return e;
    if (wide_ok(src, ncell)) k_psi_nonzero_wide<<<1216, 256, 0, st>>>(src, nb, ncell, flag);
    else k_psi_nonzero<<<1216, 256, 0, st>>>(src, nb, ncell, flag);
    return cudaGetLastError();
}
cudaError_t launch_gather_host(const void* U, const int8_t* lo, const void* psi, bool fp32, const StepDims& dm,
                               int64_t first, int64_t count, int64_t ncell, double* out, cudaStream_t st) {
    const bool wide = wide_ok(out, ncell) && first % 2 == 0 && count % 2 == 0;
    if (fp32) {
        if (wide)
            k_gather_host_wide<float><<<1216, 256, 0, st>>>((const float*)U, lo, (const float*)psi, dm, first, count, ncell,
                                                            out);
        else k_gather_host<float><<<1216, 256, 0, st>>>((const float*)U, lo, (const float*)psi, dm, first, count, ncell, out);
    } else {
        if (wide)
            k_gather_host_wide<double><<<1216, 256, 0, st>>>((const double*)U, nullptr, (const double*)psi, dm, first, count,
                                                             ncell, out);
        else
            k_gather_host<double><<<1216, 256, 0, st>>>((const double*)U, nullptr, (const double*)psi, dm, first, count,
                                                        ncell, out);
    }
    return cudaGetLastError();
}

cudaError_t launch_core_up(const double* host, void* U, int8_t* lo, void* P, int32_t* flag, bool fp32, const StepDims& dm,
                           cudaStream_t st) {
    if (!core_ok(host, dm)) return cudaErrorInvalidValue;
    if (flag) {
        cudaError_t e = cudaMemsetAsync(flag, 0, sizeof(int32_t), st);
        if (e != cudaSuccess) return e;
    }
    if (fp32) {
        const auto kern = core_short_pieces(dm) ? k_core_up<float, 1> : k_core_up<float, 2>;
        kern<<<kCoreGrid, kCoreThreads, 0, st>>>(host, (float*)U, lo, (float*)P, flag, core_runs<float>(dm), dm);
    } else {
        k_core_up<double, 5><<<kCoreGrid, kCoreThreads, 0, st>>>(host, (double*)U, nullptr, (double*)P, flag,
                                            core_runs<double>(dm), dm);
    }
    return cudaGetLastError();
}
cudaError_t launch_core_down(const void* U, const int8_t* lo, const void* P, bool fp32, double* host, const StepDims& dm,
                             cudaStream_t st) {
    if (!core_ok(host, dm)) return cudaErrorInvalidValue;
    if (fp32) {
        const auto kern = core_short_pieces(dm) ? k_core_down<float, 1> : k_core_down<float, 2>;
        kern<<<kCoreGrid, kCoreThreads, 0, st>>>((const float*)U, lo, (const float*)P, host, core_runs<float>(dm), dm);
    } else {
        k_core_down<double, 5><<<kCoreGrid, kCoreThreads, 0, st>>>((const double*)U, nullptr, (const double*)P, host,
                                            core_runs<double>(dm), dm);
    }
    return cudaGetLastError();
}

int kpar_candidates_fp64(const StepDims& d, int* out) {
    if (d.ni == 16) { out[0] = 1; return 1; }
    if (d.ni == 8) { out[0] = 2; out[1] = 4; return 2; }
    return 0;
}

}  // namespace falcon
