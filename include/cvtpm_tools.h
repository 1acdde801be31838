/*
 * cvtpm_tools.h — measurement helpers exported by libcvtpm.so beside the
 * drop-in ABI of cvtpm.h.  They have no counterpart in the reference: they
 * supply denominators for roofline reporting and show what tests cannot see
 * from results.
 */
#ifndef CVTPM_TOOLS_H
#define CVTPM_TOOLS_H

#include "cvtpm.h"

#ifdef __cplusplus
extern "C" {
#endif

/* FP32 CUDA-core peak of `device`: a grid of independent FFMA chains
 * (2 flops each), timed with CUDA events on `stream`.  Writes TFLOP/s. */
cvtpm_status cvtpm_tool_fp32_peak(int device, void* stream, float* tflops);

/* The blocked PD smoother alone: `steps` (even) steps on the left view's
 * smoother input and edge weights of the last depthMap call on `ctx`, run
 * on `stream` into the context's scratch; writes the time per step (us,
 * best of two timed runs after a warm-up).  depthMap runs the two views'
 * smoothers concurrently, so its per-phase timings cannot give this. */
cvtpm_status cvtpm_tool_pd_time(cvtpm_ctx* ctx, int steps, void* stream, float* us_per_step);

/* The smoother's square roots, reciprocals and divisions against the correctly
 * rounded ones, on `device`; waits.  bad (4 counts): wrong roots or reciprocals
 * that the residual does not flag, right ones that it flags, wrong quotients of
 * the form for any size, of the form for moderate sizes. */
cvtpm_status cvtpm_tool_pd_math_check(int device, void* stream, unsigned long long* bad);

/* The routes that calls of these parameters (patchsize, arith) take for an image
 * size; -1 for a bad argument.  No device is needed.  Routes never change
 * results. */
#define CVTPM_ROUTE_TAPS 1          /* every candidate of a pass tap-parallel */
#define CVTPM_ROUTE_TAP_SWEEPS 2    /* the candidates outside shared windows */
#define CVTPM_ROUTE_WINDOWS 16      /* larger images' passes share plane windows */
#define CVTPM_ROUTE_TAP_COST 4      /* cvtpm_cost_eval */
#define CVTPM_ROUTE_TAP_ADJOINT 8   /* cvtpm_cost_adjoint with image gradients */
int cvtpm_tool_routes(const cvtpm_params* params, int width, int height);

/* Whether a ray cast of dwidth x dheight rays steps over the empty bricks of a
 * volume of this size (1) or marches plainly (0).  No device is needed. */
int cvtpm_tool_tsdf_bricks(int width, int height, int depth, int dwidth, int dheight);

#ifdef __cplusplus
}
#endif
#endif
