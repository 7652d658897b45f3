// The fixed-point FP64 step as seen by the host engine.
#pragma once
#include "dugks_kernels.cuh"
#include "fixed_kernels.cuh"

namespace dg {

// What a handle keeps for its fixed-point steps: parameters, launch shape and the
// FP64 parameters of the redo kernel.
struct FxPlan {
    FxParams P;
    int fax;          // force axis (3: none)
    int flux_rows, flux_chunks;  // tile rows and z chunks of the flux kernel
    int redo_blocks, redo_kchunk;  // grid and z chunk of the redo kernel
    StepParams<double, double> D;
};

// launch shape of a plan whose P and fax are set
cudaError_t fixed_plan_setup(FxPlan &L);

// One step f_in -> f_out (which may be the same array) in two calls: stage (a);
// flux / update and the FP64 redo that returns at once when the state was in
// range.  words: FXW_WORDS words of the handle, zero at first.
cudaError_t launch_fixed_a(const FxPlan &L, const double *f_in, void *fb, int *words, cudaStream_t st);
cudaError_t launch_fixed_flux(const FxPlan &L, const double *f_in, double *f_out, void *fb, int *words, cudaStream_t st);

// f-bar-plus in FP64 in the layout of StepParams, ghosts included, if the last step left it in
// fixed point, and fixed-point steps run in FP64 from here on.  copy: fb's first
// rs ny nz elements.
cudaError_t launch_fixed_decode(const FxPlan &L, const void *copy, void *fb, int *words, cudaStream_t st);

}  // namespace dg
