// launch_impl.cuh -- host launchers shared by both precisions (mhd_fp64.cu,
// mhd_mixed.cu): CFL, ghost fill, psi.
#pragma once
#include "mhd_impl.cuh"

namespace falcon {
namespace impl {

// Dynamic shared memory above 48 KB for a kernel, set once per process and kernel.
template <class K> cudaError_t allow_smem(K kernel, size_t bytes) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
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

template <class T>
cudaError_t ghost_any(const StepDims& d, const GhostLists& gl, T* u, cudaStream_t st) {
    const int64_t nb_ip = (gl.ip.n + 127) / 128, nb_ln = (gl.ln.n + 127) / 128, nb_cp = (gl.cp.n + 127) / 128;
    if (nb_ip + nb_ln + nb_cp == 0) return cudaSuccess;
    if (nb_ip + nb_ln + nb_cp < (int64_t)INT32_MAX) {
        k_ghost_all<T><<<(unsigned)(nb_ip + nb_ln + nb_cp), 128, 0, st>>>(u, gl, d.ncell, d.nip, d.nip * d.njp,
                                                                          (int)nb_ip, (int)nb_ln);
        return cudaGetLastError();
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
