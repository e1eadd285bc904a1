// ppf_particles.h -- launchers of the particle analysis (ppf_particles.cu).
#pragma once

#include <cuda_runtime.h>

#include "ppf_internal.h"

namespace ppf {

// Device scratch of the analysis, parts of one allocation of `ints` ints (none
// needs a value beforehand).
struct ParticleScratch {
    int *lab, *vol, *list;   // `nodes` entries each
    unsigned *bits;          // one per 32-cell word
    int *hist, *counts;      // the sort's counts; list and volume counts
    int64_t nodes, ints;     // nodes: most runs of solid cells a domain can have
};
ParticleScratch particle_scratch(const Geom &g, int *mem);

// Labels the solid (etaS > threshold) of the state whose etaS is `etaS`
// (padded layout), then writes out[0..4] = {particles, sum of equivalent
// radii (cells), solid cells, largest particle (cells), solid/liquid faces}.
// partials: 6 nblocks + 3 num_sms doubles; volumes (nullable): up to `cap`
// particle volumes, in no order; err: a device word, bit 1 set if a retry cap
// was reached.
template <typename T>
cudaError_t launch_particles(const Geom &g, const T *etaS, double threshold, const ParticleScratch &p, double *partials,
                             int nblocks, int num_sms, double *out, int *volumes, int64_t cap, int *err,
                             cudaStream_t s);

// Sorts n >= 1 volumes, none above `largest`, into *sorted (in the scratch of a
// finished analysis); `keys` and `spare` hold n ints each and are overwritten.
cudaError_t launch_sort_volumes(int *keys, int *spare, int64_t n, int64_t largest, const ParticleScratch &p,
                                int64_t **sorted, cudaStream_t s);

}  // namespace ppf
