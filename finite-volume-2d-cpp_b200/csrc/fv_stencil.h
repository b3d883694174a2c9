// The diffusion kind of the fast modes as one linear stencil per cell.
//
// With V = 1, no limiter and constant geometry, the time derivative of a cell
// (its own and its neighbours' Green-Gauss gradients, the corrected face
// gradient, the flux sum; gradient_for_diffusion, explicit.cpp:70-109, and
// examples/heatTransfer/main.cpp:33-60) is linear in the states of the cell's
// two rings: qt_c = sum_k a_k (q_k - q_c), with at most NF^2 terms for cells of
// NF faces (NF neighbours and NF - 1 further ones of each).  The coefficients
// are laid out once, evaluated and held in FP64 from the stage precision's
// geometry: FP32's rounded coordinates are what its results are exact for.
#pragma once
#include "fv_launch.h"
#include "fv_tile.cuh"

namespace fvgpu {

// Slots of a tile: its T cells, then the two-ring halo.
struct StencilParams {
    Params P;
    const int4* info;        // [n_tiles] {halo_off, n_halo, owned cells, 0}
    const int32_t* halo;     // device cell of each halo slot
    const double* coef;      // [NF * NF][n_real]
    const uint16_t* slot;    // [NF * NF][n_real]: slot, 0x8000 set on a ghost neighbour (the first NF)
    const double* area;      // [n_real]
    int T, nf, max_slots;
};

const void* stencil_run_kernel(bool f32, int nf, int* threads);  // threads: a CTA's at most
void launch_stencil_stage(bool f32, const StencilParams& SP, const TileIO& io, int n_tiles, cudaStream_t st, bool pdl);

}  // namespace fvgpu
