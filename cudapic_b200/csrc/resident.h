// resident.h -- whole ion cycles of a small discharge in one launch
// (kernels_resident.cu), called by the state driver (state.cpp).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "../../include/cudapic.h"

namespace cudapic {

struct ResidentPlanes {
    float *x, *vx, *vy, *vz;
};

// Buffers of a state at the start of an ion cycle; sides and densities by
// their roles there (..._out: by their roles after the steps).
struct ResidentArgs {
    ResidentPlanes e, i[2];                  // electrons' live side; ions: [0] live side, [1] the other
    uint32_t *rng_e[4], *rng_i[4];
    uint32_t *n_e, *n_i, *alive_i;           // counts; the (zero) slot counter of the ion push
    uint32_t *step_counter;
    uint32_t n_sub;
    const float *e_dens_in, *i_collected;    // densities of the present particles
    float *e_dens_out, *i_current_out, *i_collected_out;
    float *pot, *efield;                     // of the last step
    const float *pot0_table;
    const float *sigma_tot_e, *sigma_tot_i, *cs;
    float sigma_max, ion_k;
};

// True when the kernel takes a discharge of this grid (16-byte aligned ion
// planes assumed): capacity and grid fit the cluster's shared memory, FP64
// Poisson sums, at least two steps per ion cycle.
bool resident_fits(const cudapic_grid &g, uint32_t n_sub);
// True when its cluster can be resident where `stream` launches: a stream or a
// process that has a part of the SMs only may hold no cluster of 8 or 16 CTAs
// of one SM each.
bool resident_launchable(const cudapic_grid &g, cudaStream_t stream);
// Enqueues `steps` steps (a positive multiple of n_sub, from the start of an
// ion cycle); resident_launchable for this stream first.
int launch_resident(const ResidentArgs &a, const cudapic_grid &g, uint32_t steps, cudaStream_t stream);

}  // namespace cudapic
