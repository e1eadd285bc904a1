// ppf_ctx.h -- the context behind the opaque ppf_ctx of include/ppf.h,
// shared by the C-ABI translation units (ppf_capi.cu, ppf_ensemble.cu).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "ppf.h"
#include "ppf_fx.h"
#include "ppf_internal.h"
#include "ppf_step_tma.h"

// A context replaces the reference's global state (phasefield.c:67-70).
struct ppf_ctx {
    int nz, ny, nx, bc, prec;
    ppf_params p;
    ppf_derived d;
    ppf::Geom g;
    int dev, num_sms;
    cudaStream_t own, stream;
    void *state;          // one allocation: 2 buffers x 3 fields x g.total elements
    void *fld[2][3];      // [buffer][etaS, etaL, c]
    int cur_eta, cur_c;   // buffer holding the current eta / c
    double *staging;      // 3 * cells doubles, compact [z][y][x]
    double *partials;     // partial sums (per work item of the step, per block of other kernels)
    int partials_cap;     // in doubles
    double *dres;         // device results: [0..2] increments, [3..7] observables, [8..12] particles,
                          // [16..19] mass-projection plan; the error word follows at dres + 32
    int *derr;            // device error word set by a kernel whose bounded wait ran out
    int *dsched;          // the step's two scheduler word pairs (dres + 32, after the error word)
    CUtensorMap maps[2][2][3];   // TMA maps of the fields of both buffers, per tile shape [tile][buffer][field]
    ppf::StepTune tune;        // launch choices of the fused step (grid, z chunk, unroll)
    unsigned long long wait_limit_ns;
    int inject;           // test hook: PPF_INJECT_*
    int *pscratch;        // particle analysis (allocated on first use)
    int *plist;           // particle volumes (device), twice plist_cap entries
    int64_t plist_cap;
    int64_t *psorted;     // the last analysis' first pkept volumes in order (in pscratch)
    int64_t pkept;
    int64_t steps;
    int uploaded;
    ppf::Coef<float> kf;
    ppf::Coef<double> kd;
    int eqA;              // AS == AL: the mu reciprocal is a constant
    ppf::fx::FxCoef kx;   // FP64: coefficients of the fixed-point step
    int fx_ok;            // FP64: the parameters and the grid fit the fixed-point step
    int left_box;         // the host knows that the state has left the fixed-point step's box, and
                          // has set both box words
    int shared_box;       // dbox belongs to another slab of the same domain
    int *dbox;            // box words of the two buffers (launch_step_fx): the context's own, behind the
                          // scheduler words, or shared with the slabs of one domain / in the ensemble's array
    ppf::CoefD cd;
};

// helpers of ppf_capi.cu (return PPF_* codes, set ppf_last_error)
int ensure_partials(ppf_ctx *c, int ndoubles);
int do_pack(ppf_ctx *c);        // staging -> state buffer 0 (+ ghosts, box word)
int do_unpack(ppf_ctx *c);      // current state -> staging
int check_device_error(ppf_ctx *c);
// FP64: sets the box words for the state in buffer 0 and learns of them; waits for the stream
int recheck_box(ppf_ctx *c);
inline int *own_box(ppf_ctx *c) { return c->derr + 8; }
// whether the next FP64 step runs in fixed-point arithmetic
inline bool fx_step(const ppf_ctx *c) { return c->fx_ok && !c->left_box; }
