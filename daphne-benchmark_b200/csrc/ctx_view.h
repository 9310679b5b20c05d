// Read-only view of a context's evaluation set-up (grid, constants, launch
// shape, stream), for entry points that live outside engine.cu.
#pragma once
#include <cuda_runtime.h>

#include "ndt_types.h"

struct ndt_ctx;

namespace ndt {

struct CtxEvalView {
    GridDev grid;
    double d1, d2;
    int compat;
    int precision;
    int variant;
    int sms;
    int device;
    cudaStream_t stream;
    bool have_map;
};

// Fills *v from the context; returns 0, or NDT_E_ARG for a null argument.
int ctx_eval_view(ndt_ctx *c, CtxEvalView *v);
// NDT scores of B poses on the context's stream (arguments checked by the
// caller): pose b is scored with scan b % scans of the packed d_points /
// d_offsets (scans + 1 entries), total_points >= the scans' points.
int ctx_score_batch(ndt_ctx *c, int B, int scans, const float *d_points, const int *d_offsets, int total_points,
                    const float *d_poses, double *d_score);
// After a wait for the context's stream: NDT_OK, or the error of a map build or
// append whose sort gave up (the context then has no map).
int ctx_map_status(ndt_ctx *c);
// Records an error message on the context (ndt_last_error).
void ctx_set_error(ndt_ctx *c, const char *msg);

}  // namespace ndt
