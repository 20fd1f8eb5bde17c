// csr.cuh — device result record of the src/linear CSR solves.
#pragma once

#include <cuda_runtime.h>

#include <string>

#include "common.cuh"
#include "flursys_cuda.h"
#include "gridreduce.cuh"

namespace flursys {

struct CsrResultDev {
    int error;   // FlursysStatus of a failure, 0 when none
    int status;  // FlursysLinearStatus
    long long iterations;
    double initial;
    double final_residual;
    unsigned long long bad_row;  // first non-finite SpMV row (all ones when none)
    unsigned device_error;       // DeviceError bits
    unsigned pad;
};

// The split of a banded matrix over the chip (csr_band.cu).
struct BandPlan {
    int blocks = 0, rows = 0, band = 0, width = 0;  // blocks 0: the matrix does not fit
    size_t smem = 0;
    const void *kernel = nullptr;
};

constexpr int kCsrSlots = 3;  // solves whose results a work area holds at a time

// Work vectors of device-resident CSR solves (grown on demand), for callers
// inside the library that assemble their matrices on the device.
struct CsrDeviceWork {
    int n = 0, grid = 0;
    double *vec = nullptr;       // 10 vectors of n; the others follow in its allocation
    double *inv_diag = nullptr;  // n (PCG)
    double *partials = nullptr;  // grid * 4
    GridBarrier *bar = nullptr;
    CsrResultDev *res = nullptr;   // [0] the solve, [1] the Jacobi set-up (error only)
    CsrResultDev *hres = nullptr;  // pinned copies of both, by the launch's slot
    BandPlan band;                 // CG and PCG of a banded matrix
    RedRecord *records = nullptr;  // its partial sums
    unsigned epoch = 0;
    cudaError_t ensure(int n, int device);
    // Lets CG and PCG solves of matrices with at most `width` entries in a row,
    // all within `band` columns of the diagonal, run on the chip where they fit.
    cudaError_t ensure_band(int n, long long band, long long width, int device, cudaStream_t st);
    void release();
};

// Enqueues one solve on device-resident CSR arrays (32-bit indices, columns
// ascending in each row): method 0 CG, 1 Jacobi-PCG (the inverse diagonal is
// formed on the device; a missing or zero diagonal is reported as an error),
// 2 BiCGSTAB, with the stop rule of src/linear. The result records land in
// w.hres + 2 * slot (slot < kCsrSlots) after the stream is synchronised;
// csr_device_status maps them.
// (b and x are not checked for finiteness beforehand: a non-finite value
// surfaces as FLURSYS_ERR_NON_FINITE from the first SpMV or dot.)
cudaError_t csr_device_launch(int method, int n, const int *ro, const int *ci, const double *va, const double *b,
                              double *x, double atol, double rtol, long long max_iters, CsrDeviceWork &w, int slot,
                              cudaStream_t st);
int32_t csr_device_status(const CsrResultDev *hres, FlursysLinearSolveReport *rep, std::string *err);

}  // namespace flursys
