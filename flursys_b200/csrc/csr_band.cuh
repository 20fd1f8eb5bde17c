// csr_band.cuh — host interface of the chip-resident CG / Jacobi-PCG for
// banded CSR matrices (csr_band.cu).
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

#include "csr.cuh"
#include "gridreduce.cuh"

namespace flursys {

struct BandArgs {
    int n, rows, band, width;  // rows per block, max |column - row|, entries of the longest row
    const int *ro, *ci;
    const double *va, *inv_diag;  // inv_diag: PCG, or null
    const double *b;
    double *x;
    RedRecord *records;   // 2 * blocks * kRedSlots partial sums, then 2 * n values of the rows
    unsigned epoch;
    CsrResultDev *res;    // device_error is set to 0 by a solve that ends
    double atol, rtol;
    long long max_iters;
};

// The split of an n-row matrix whose rows hold at most `width` entries within
// `band` columns of the diagonal.
BandPlan csr_band_plan(long long n, long long band, long long width, int device);
// Bytes of a plan's records; they are cleared once, and each launch takes a new epoch.
size_t csr_band_record_bytes(const BandPlan &plan, long long n);
cudaError_t csr_band_launch(const BandPlan &plan, const BandArgs &args, cudaStream_t stream);

}  // namespace flursys
