// ppf_step_fx.h -- launcher of the float64 step in fixed-point arithmetic
// (ppf_step_fx.cu).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include "ppf_fx.h"
#include "ppf_internal.h"
#include "ppf_step_tma.h"

namespace ppf {

// Like launch_step_tma<double>, with the same work items, partial sums and
// scheduler words (no 64-bit offsets: fields of at most 2^32 elements).
// `k` are the float64 coefficients, `in` the input state that `maps`
// describe.  `box` points to two words, one per buffer: word b is not zero
// when the state in buffer b has left the box of ppf_fx.h (set by the step
// or upload that wrote it; sticky until the next upload).  A
// step whose input has left it is computed in float64 arithmetic, straight
// from memory.  `parity`: the buffer of
// the input's c (c changes buffers in every step).
cudaError_t launch_step_fx(const Geom &g, const Coef<double> &k, const fx::FxCoef &kx, const CUtensorMap *maps,
                           Fields<const double> in, Fields<double> out, bool c_only, double *partials,
                           const StepTune &tune, int *err, unsigned long long limit_ns, int inject_stall, int *sched,
                           int *box, int parity, cudaStream_t s);

// Like launch_step_multi<double>, for full steps; each domain's box words
// are in the table.
cudaError_t launch_step_fx_multi(const DomainDesc *table, int ndom, const int *items, const Coef<double> &k,
                                 const fx::FxCoef &kx, int parity, double *partials, int grid, bool pdl, bool split,
                                 int *err, unsigned long long limit_ns, int *sched, cudaStream_t s);

// CTAs of the fixed-point step per SM (its attributes set first); < 1 on failure.
int fx_occupancy(bool multi);

}  // namespace ppf
