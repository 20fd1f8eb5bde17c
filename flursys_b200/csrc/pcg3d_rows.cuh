// pcg3d_rows.cuh — host interface of the chip-resident 3D pressure PCG by rows
// (pcg3d_rows.cu): F64 and MIXED.
#pragma once

#include <cuda_runtime.h>

#include "gridreduce.cuh"
#include "pcg3d.cuh"
#include "pcg3d_seq.cuh"

namespace flursys {

struct RowsArgs {
    int nx, ny, nz;
    int by, bz, ty, tz;  // blocks per axis, rows of a block per axis
    double ix2, iy2, iz2;
    double *x;
    const double *rhs;  // the system is A x = -rhs
    int stop_rule;
    double tol, atol, rtol;
    long long max_iters;
    int replace_every;
    CgSeqState *st;
    RedRecord *records;  // grid form
    void *faces;         // grid form: 2 * blocks * slots values
    unsigned epoch;
    int fault;           // injected barrier fault
};

struct Pcg3dRowsPlan {
    RowsArgs args{};
    const void *kernel = nullptr;
    bool cluster = false;
    int blocks = 0, threads = 0;
    size_t smem = 0;
    RedRecord *records = nullptr;
    void *faces = nullptr;
    unsigned epoch = 0;
};

// Sets up the resident solve; false when the grid's rows do not fit the chip
// or FLURSYS_PCG_RESIDENT asks for another form.
bool pcg3d_rows_plan(Pcg3dRowsPlan &plan, const Pcg3dArgs &args, int precision, int device);
// One solve into *state; launches of one plan run one after another.
cudaError_t pcg3d_rows_launch(Pcg3dRowsPlan &plan, CgSeqState *state, cudaStream_t stream);
void pcg3d_rows_destroy(Pcg3dRowsPlan &plan);

}  // namespace flursys
