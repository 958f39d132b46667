// reuse.cuh — what the two forms of the FP32-mixed step with neighbour reuse
// (kernels_reuse.cu, kernels_reuse_cell.cu) share.
#pragma once

#include "mixed_common.cuh"
#include "piston.cuh"
#include "step_particle.cuh"

namespace rrsph {

// kernels_reuse_cell.cu: DevParams::reuse == kReuseCell.
void launch_verlet_build_cell(const DevParams& P, const State& S, const Sorted& G, cudaStream_t st);
void launch_density_cell(const DevParams& P, const State& S, const Sorted& G, StepScalars* scal, uint32_t* flags,
                         cudaStream_t st);
void launch_forces_cell(const DevParams& P, const State& S, const Sorted& G, StepScalars* scal,
                        StepScalars* scal_next, uint32_t* flags, cudaStream_t st, bool std_terms, int wv);

// A launch that may start while the stream's previous kernel finishes
// (programmatic dependent launch); the kernel waits for it with
// griddepcontrol.wait before it reads what that kernel wrote.
template <typename... Params, typename... Args>
void launch_after(void (*kernel)(Params...), unsigned blocks, int threads, cudaStream_t st, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, args...);
}

}  // namespace rrsph
