// mhd_mixed.cu -- launchers of the mixed-precision step kernels: FP32 state
// (u^n compensated by an 8-bit correction) and stencil RHS; p1 in float-float;
// FP64 CFL reduction and dt.
#include "launch_impl.cuh"
#include "mhd_mixed_impl.cuh"

namespace falcon {
namespace impl {
namespace {
// CTAs per block, each a run of `planes / split` k planes (out of place only: in
// place, a part would overwrite planes that its neighbours still read). A grid
// with few blocks leaves SMs idle or unevenly loaded: the split is the power of
// two that minimises the planes of the busiest SM, counting one more plane per
// part for the ghost planes it rereads. 108 blocks of 16^3: diffusion 50 us whole,
// 41 in two, 37 in four parts (the rule's; 34 now). 864 blocks of 8^3: stage 36.3 us whole
// (the rule's), 41.4 in two.
int split_of(const StepDims& d, int most) {
    auto cost = [&](int s) { return ((int64_t)d.nblocks * s + 151) / 152 * (d.nk / s + 1); };
    int best = 1;
    for (int s = 2; s <= most; s *= 2)
        if (cost(s) < cost(best)) best = s;
    return best;
}

// 8^3 blocks: chunks of KP planes; 16^3 blocks (KP 0): the march
template <int N, int KP, int DIVB>
cudaError_t stage_nd(const StepDims& d, const Geometry& g, const float* in, const float* un, float* out, int8_t* lo,
                     const PushTable& push, const DivBArgs& psi, int stage, int bcw, StepScalars* sc, cudaStream_t st) {
    auto run = [&](auto kernel, size_t smem, int nt, int most) {
        static OncePerDevice once;
        const cudaError_t attr = allow_smem(once, kernel, smem);
        if (attr != cudaSuccess) return attr;
        const int split = in != out ? split_of(d, most) : 1;
        return launch_step(d, kernel, d.nblocks * split, nt, smem, st, in, un, out, lo, push, psi, g, sc, stage, bcw, split);
    };
    if constexpr (KP == 0) return run(k_stage_march<N, N, N, DIVB>, SMarch<N, N, N>::smem, N * N, 8);
    else return run(k_stage_chunks<N, N, N, KP, DIVB>, QShape<N, N, N, KP>::smem, N * N * KP, N / KP);
}
// The div-B mode is a template parameter: the plain stage keeps its register
// allocation free of the GLM/Powell terms.
template <int N, int KP>
cudaError_t stage_n(const StepDims& d, const Geometry& g, const float* in, const float* un, float* out, int8_t* lo,
                    const PushTable& push, const DivBArgs& psi, int stage, int bcw, StepScalars* sc, cudaStream_t st) {
    switch (psi.mode) {
    case 0: return stage_nd<N, KP, 0>(d, g, in, un, out, lo, push, psi, stage, bcw, sc, st);
    case 1:
        if (!psi.in || !psi.un || !psi.out) return cudaErrorInvalidValue;
        return stage_nd<N, KP, 1>(d, g, in, un, out, lo, push, psi, stage, bcw, sc, st);
    case 2: return stage_nd<N, KP, 2>(d, g, in, un, out, lo, push, psi, stage, bcw, sc, st);
    default: return cudaErrorInvalidValue;
    }
}

template <int N, int KP>
cudaError_t diff_n(const StepDims& d, const Geometry& g, const float* u, float* out, int8_t* lo, const PushTable& push,
                   StepScalars* sc, int cfl_next, cudaStream_t st) {
    using S = DShape<N, N, N, KP>;
    static OncePerDevice once;
    const cudaError_t attr = allow_smem(once, k_diffusion_quads<N, N, N, KP>, S::smem);
    if (attr != cudaSuccess) return attr;
    return launch_step(d, k_diffusion_quads<N, N, N, KP>, d.nblocks, S::NT, S::smem, st, u, out, lo, push, g, sc, cfl_next);
}
// 16^3 blocks: the k march
cudaError_t diff_march16(const StepDims& d, const Geometry& g, const float* u, float* out, int8_t* lo,
                         const PushTable& push, StepScalars* sc, int cfl_next, cudaStream_t st) {
    using S = MShape<16, 16, 16>;
    static OncePerDevice once;
    const cudaError_t attr = allow_smem(once, k_march_quads<16, 16, 16>, S::smem);
    if (attr != cudaSuccess) return attr;
    const int split = out != u ? split_of(d, 4) : 1;
    return launch_step(d, k_march_quads<16, 16, 16>, d.nblocks * split, S::NT, S::smem, st, u, out, lo, push, g, sc, cfl_next,
                       split);
}
}  // namespace
}  // namespace impl

// 8^3 blocks: planes per chunk; 16^3 blocks: the march, whatever depth is asked for
cudaError_t launch_stage_mixed(const StepDims& d, const Geometry& g, const float* in, const float* un, float* out,
                               int8_t* lo, const PushTable& push, const DivBArgs& psi, int stage, int bcw, StepScalars* sc,
                               int kpar, cudaStream_t st) {
    if (d.ni != d.nj || d.ni != d.nk) return cudaErrorInvalidValue;
    if (d.ni == 16) return impl::stage_n<16, 0>(d, g, in, un, out, lo, push, psi, stage, bcw, sc, st);
    if (d.ni != 8) return cudaErrorInvalidValue;
    switch (kpar) {
    case 2: return impl::stage_n<8, 2>(d, g, in, un, out, lo, push, psi, stage, bcw, sc, st);
    case 4: return impl::stage_n<8, 4>(d, g, in, un, out, lo, push, psi, stage, bcw, sc, st);
    case 8: return impl::stage_n<8, 8>(d, g, in, un, out, lo, push, psi, stage, bcw, sc, st);
    }
    return cudaErrorInvalidValue;
}
cudaError_t launch_psi_diffusion_mixed(const StepDims& d, const Geometry& g, const float* u, const float* psi,
                                       float* psi_out, StepScalars* sc, cudaStream_t st) {
    return impl::psi_diffusion_any<float>(d, g, u, psi, psi_out, sc, st);
}
cudaError_t launch_psi_ghost_mixed(const StepDims& d, const GhostLists& gl, float* psi, cudaStream_t st) {
    return impl::psi_ghost_any<float>(d, gl, psi, st);
}
// 8^3 blocks: planes per chunk; 16^3 blocks: the march, whatever depth is asked for
cudaError_t launch_diffusion_mixed(const StepDims& d, const Geometry& g, const float* u, float* out, int8_t* lo,
                                   const PushTable& push, StepScalars* sc, int kpar, cudaStream_t st, int cfl_next) {
    if (push.tgt != nullptr && out == u) return cudaErrorInvalidValue;   // pushing needs out != u
    if (d.ni != d.nj || d.ni != d.nk) return cudaErrorInvalidValue;
    if (d.ni == 16) return impl::diff_march16(d, g, u, out, lo, push, sc, cfl_next, st);
    if (d.ni != 8) return cudaErrorInvalidValue;
    switch (kpar) {
    case 2: return impl::diff_n<8, 2>(d, g, u, out, lo, push, sc, cfl_next, st);
    case 4: return impl::diff_n<8, 4>(d, g, u, out, lo, push, sc, cfl_next, st);
    case 8: return impl::diff_n<8, 8>(d, g, u, out, lo, push, sc, cfl_next, st);
    }
    return cudaErrorInvalidValue;
}
cudaError_t launch_cfl_mixed(const StepDims& d, const Geometry& g, const float* u, StepScalars* sc, cudaStream_t st) {
    return impl::cfl_any<float>(d, g, u, sc, st);
}
cudaError_t launch_ghost_mixed(const StepDims& d, const GhostLists& gl, float* u, cudaStream_t st) {
    return impl::ghost_any<float>(d, gl, u, st);
}
// k-chunk depths instantiated per block size; the context's autotuner times
// them on its own grid and keeps the fastest.
int kpar_candidates_mixed(const StepDims& d, int* out) {
    const int first = d.ni == 16 ? 1 : d.ni == 8 ? 2 : 0;
    for (int q = 0; q < 3 && first; ++q) out[q] = first << q;
    return first ? 3 : 0;
}
cudaError_t launch_clear_outside_core_mixed(const StepDims& d, float* u, int nvar, cudaStream_t st) {
    const int64_t n = nvar == NV ? (int64_t)d.nblocks * 2 : d.nblocks;   // the state's halves, or a [b][cell] array
    const unsigned grid = (unsigned)(n < 65535 * 4 ? n : 65535 * 4);
    if (nvar == NV) impl::k_clear_outside_core<float4><<<grid, 256, 0, st>>>(reinterpret_cast<float4*>(u), n, d);
    else if (nvar == 1) impl::k_clear_outside_core<float><<<grid, 256, 0, st>>>(u, n, d);
    else return cudaErrorInvalidValue;
    return cudaGetLastError();
}
namespace impl {
namespace {
template <class T, int G> cudaError_t interleave(T* a, int64_t arrays, int n, cudaStream_t st) {
    const size_t smem = (size_t)G * n * sizeof(T);
    static OncePerDevice once;
    const cudaError_t e = allow_smem(once, k_interleave<T, G>, 232448);
    if (e != cudaSuccess) return e;
    if (smem > 232448 || smem % 16 != 0 || arrays > INT32_MAX) return cudaErrorInvalidValue;
    k_interleave<T, G><<<(unsigned)arrays, 512, smem, st>>>(a, n);
    return cudaGetLastError();
}
}  // namespace
}  // namespace impl
cudaError_t launch_state_from_file(float* U, int8_t* lo, const StepDims& d, cudaStream_t st) {
    const cudaError_t e = impl::interleave<float, 4>(U, (int64_t)d.nblocks * 2, d.ncell, st);
    return e == cudaSuccess && lo ? impl::interleave<int8_t, NV>(lo, d.nblocks, d.ni * d.nj * d.nk, st) : e;
}
cudaError_t launch_push_state_mixed(const StepDims& d, const Geometry& g, float* u, const PushTable& push,
                                    StepScalars* sc, cudaStream_t st) {
    if (d.ni == 16 && d.nj == 16 && d.nk == 16) impl::k_push_state<16, 16, 16><<<d.nblocks, 256, 0, st>>>(u, push, g, sc);
    else if (d.ni == 8 && d.nj == 8 && d.nk == 8) impl::k_push_state<8, 8, 8><<<d.nblocks, 64, 0, st>>>(u, push, g, sc);
    else return cudaErrorInvalidValue;
    return cudaGetLastError();
}


cudaError_t launch_step_persistent_mixed(const StepDims& d, const Geometry& g, float* U, float* RK, float* R2,
                                         int8_t* lo, const PushTable& push, const GhostLists& gl_stage,
                                         const GhostLists& gl_final, StepScalars* sc, unsigned int* bar,
                                         cudaStream_t st) {
    if (d.ni != 16 || d.nj != 16 || d.nk != 16 || !bar) return cudaErrorInvalidValue;
    using SS = impl::SMarch<16, 16, 16>;
    using SD = impl::MShape<16, 16, 16>;
    constexpr size_t smem = SS::smem > SD::smem ? SS::smem : SD::smem;
    // two CTAs of 256 threads per SM, as the separate stage and diffusion
    // launches run (228 KB per SM, 1 KB of it reserved per CTA, and about
    // 0.5 KB of static shared memory in the bodies)
    static_assert(2 * (smem + 512 + 1024) <= 233472, "two CTAs per SM");
    auto kern = impl::k_step_persistent<16>;
    static int grid_cap = 0, dev_cached = -1;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev != dev_cached) {
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        int per_sm = 0, nsm = 0;
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 256, smem);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) return e;
        if (per_sm < 1) return cudaErrorLaunchOutOfResources;
        grid_cap = per_sm * nsm;   // every CTA resident at once: the grid barrier needs it
        dev_cached = dev;
    }
    const unsigned grid = (unsigned)(d.nblocks < grid_cap ? d.nblocks : grid_cap);
    e = cudaMemsetAsync(bar, 0, 8 * sizeof(unsigned int), st);   // arrival counter, generation, block tickets
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, impl::StepBuffers{U, RK, R2, lo}, push, g, sc, gl_stage, gl_final, d,
                              impl::GridBarrier{bar, bar + 1, bar + 2});
}

}  // namespace falcon
