// pcg2d_res.cuh — host interface of the chip-resident 2D pressure PCG.
#pragma once

#include <cuda_runtime.h>

#include "gridreduce.cuh"
#include "pcg2d.cuh"

namespace flursys {

// How one instance's solve runs with its state on the chip.
struct Pcg2dResPlan {
    bool enabled = false;
    bool cluster = false;  // one thread-block cluster; otherwise a co-resident grid
    int precision = 0;
    int variant = 0;       // kernel instantiation
    int nblocks = 0;
    size_t smem = 0;
    RedRecord *records = nullptr;  // grid form
    unsigned epoch = 0;            // grid form: launches so far
};

// Chooses the form for an nx x ny PCG instance (`plain`: every cell is fluid); plan.enabled is false when its
// state does not fit the chip. Allocates the grid form's records.
cudaError_t pcg2d_res_plan(Pcg2dResPlan &plan, int nx, int ny, bool plain, int precision, int device);
void pcg2d_res_destroy(Pcg2dResPlan &plan);
// Solves *inst_dev (nblocks is the plan's); `result` is the instance's device
// result record.
// Launches of one plan run one after another.
cudaError_t pcg2d_res_launch(Pcg2dResPlan &plan, const Pcg2dInstance *inst_dev, PcgResultDev *result,
                             cudaStream_t stream);

// Batched form: resident clusters take instances from a queue.
struct Pcg2dQueuePlan {
    int clusters = 0;  // 0: not available
    int nblocks = 0;   // blocks per cluster
    size_t smem = 0;   // the largest member's
};
// Whether an instance can be solved by the queue's kernel.
bool pcg2d_queue_fits(int nx, int ny, bool plain, int precision, size_t *smem);
// Pieces (32 vectors' room of a row) per warp of its blocks.
int pcg2d_queue_pieces(int nx, int ny, int precision);
cudaError_t pcg2d_queue_plan(Pcg2dQueuePlan &plan, int precision, size_t smem, int device);
// `order`: `count` instance indices (device); `next`: a device counter that is
// 0 at the launch; instances with resident < 0 are skipped.
cudaError_t pcg2d_queue_launch(const Pcg2dQueuePlan &plan, const Pcg2dInstance *insts, const int *order, int count,
                               unsigned *next, int precision, cudaStream_t stream);

}  // namespace flursys
