// pcg3d_stream.cuh — host interface of the 3D pressure PCG that streams its
// vectors once per iteration (pcg3d_stream.cu): F64 and MIXED.
#pragma once

#include <cuda_runtime.h>

#include "gridreduce.cuh"
#include "pcg3d.cuh"
#include "pcg3d_seq.cuh"

namespace flursys {

struct StreamArgs {
    int nx, ny, nz;
    int by, bz, ty, tz;  // blocks per axis, rows and planes of a block
    double ix2, iy2, iz2;
    double *x;
    const double *rhs;   // the system is A x = -rhs
    void *r[2], *d[2], *xi;  // rows padded to whole vectors; xi: the increment of x
    int stop_rule;
    double tol, atol, rtol;
    long long max_iters;
    int replace_every;
    CgSeqState *st;
    RedRecord *records;
    unsigned epoch;
    int fault;           // injected barrier fault
};

struct Pcg3dStreamPlan {
    StreamArgs args{};
    const void *kernel = nullptr;
    int blocks = 0;
    size_t smem = 0;
    void *vectors = nullptr;
    RedRecord *records = nullptr;
    unsigned epoch = 0;
};

// Sets up the solve; false when a block's planes do not fit its shared memory,
// the vectors do not fit the device, or FLURSYS_PCG_RESIDENT asks for another
// form.
bool pcg3d_stream_plan(Pcg3dStreamPlan &plan, const Pcg3dArgs &args, int precision, int device);
// One solve into *state; launches of one plan run one after another.
cudaError_t pcg3d_stream_launch(Pcg3dStreamPlan &plan, CgSeqState *state, cudaStream_t stream);
void pcg3d_stream_destroy(Pcg3dStreamPlan &plan);

}  // namespace flursys
