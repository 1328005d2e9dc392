// launch_impl.cuh -- host launchers shared by both precisions (mhd_fp64.cu,
// mhd_mixed.cu): CFL, ghost fill, psi.
#pragma once
#include "mhd_impl.cuh"
#include "once_per_device.h"

namespace falcon {
namespace impl {

// Dynamic shared memory above 48 KB for a kernel, set once per device (`once`: the kernel's own).
template <class K> cudaError_t allow_smem(OncePerDevice& once, K kernel, size_t bytes) {
    int device = 0;
    const cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    return once(device, [&] { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes); });
}

// Launch of a kernel that calls step_wait: with d.overlap (grids of up to 2^20 cells
// without psi, whose kernels run on a branch of their own) it may start while the
// kernel before it in the stream drains (and, if that calls step_go, as soon as all
// its CTAs run). Step without / with: 8^3 blocks, 111k cells 61 / 54 us, 442k 178
// / 174; 16^3, 442k 158 / 153, 885k 290 / 287. Larger grids lose by it, their slots
// taken by waiting CTAs while many remain to run: 16^3, 5.3M cells 1,150 / 1,167, 21M
// 3,982 / 4,074; 8^3, 2.7M 740 / 806.
template <class... P, class... A>
cudaError_t launch_step(const StepDims& d, void (*kernel)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t st,
                        A... args) {
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = d.overlap ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

template <class T>
cudaError_t psi_diffusion_any(const StepDims& d, const Geometry& g, const T* u, const T* psi, T* psi_out,
                              StepScalars* sc, cudaStream_t st) {
    const int nint = d.ni * d.nj * d.nk;
    k_psi_diffusion<T><<<dim3((nint + 255) / 256, d.nblocks), 256, 0, st>>>(u, psi, psi_out, g, sc, d);
    return cudaGetLastError();
}

template <class T>
cudaError_t psi_ghost_any(const StepDims& d, const GhostLists& gl, T* psi, cudaStream_t st) {
    const int64_t n = gl.cp.n + gl.ln.n + gl.ip.n;
    if (n == 0) return cudaSuccess;
    k_psi_ghost<T><<<(unsigned)((n + 255) / 256), 256, 0, st>>>(psi, gl, d.ncell, d.nip, d.nip * d.njp);
    return cudaGetLastError();
}

template <class T>
cudaError_t cfl_any(const StepDims& d, const Geometry& g, const T* u, StepScalars* sc, cudaStream_t st) {
    const int nint = d.ni * d.nj * d.nk;
    dim3 grid((nint + 255) / 256, d.nblocks);
    k_cfl<T><<<grid, 256, 0, st>>>(u, g, sc, d);
    return cudaGetLastError();
}

// Threads per interpolated FP64 entry, each a share of its variables: an entry's eight
// values one after the other are a long chain, which few entries do not hide. us per
// exchange with 1 / 2 / 4 threads: 7.5k entries 31.5 / 20.2 / 12.7, 30k 33 / 24.2 / 22.4,
// 69k 34.8 / 28.4 / 26.0, 152k 53.8 / 47.4 / 47.6, 276k 77.0 / 73.7 / 78.0, 303k 77.8 /
// 75.0 / 83.2, 604k 121.6 / 129.2 / 150.8.
inline int ghost_parts(int64_t n) { return n <= 100000 ? 4 : n <= 320000 ? 2 : 1; }
template <class T>
cudaError_t ghost_any(const StepDims& d, const GhostLists& gl, T* u, cudaStream_t st) {
    const int parts = sizeof(T) == 8 ? ghost_parts(gl.ip.n) : 1;
    const int64_t nb_ip = (gl.ip.n * parts + 127) / 128, nb_ln = (gl.ln.n + 127) / 128, nb_cp = (gl.cp.n + 127) / 128;
    if (nb_ip + nb_ln + nb_cp == 0) return cudaSuccess;
    if (nb_ip + nb_ln + nb_cp < (int64_t)INT32_MAX) {
        return launch_step(d, k_ghost_all<T>, (unsigned)(nb_ip + nb_ln + nb_cp), 128, 0, st, u, gl, d.ncell, d.nip,
                           d.nip * d.njp, (int)nb_ip, (int)nb_ln, parts);
    }
    if (gl.cp.n > 0) {
        k_ghost_copy<T><<<(unsigned)((gl.cp.n + 255) / 256), 256, 0, st>>>(u, gl.cp, d.ncell);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    if (gl.ln.n > 0) {
        k_ghost_lin<T><<<(unsigned)((gl.ln.n + 255) / 256), 256, 0, st>>>(u, gl.ln, d.ncell);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    if (gl.ip.n > 0) {
        k_ghost_interp<T><<<(unsigned)((gl.ip.n + 127) / 128), 128, 0, st>>>(u, gl.ip, d.ncell, d.nip, d.nip * d.njp);
        return cudaGetLastError();
    }
    return cudaSuccess;
}

}  // namespace impl
}  // namespace falcon
