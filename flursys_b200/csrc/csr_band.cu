// csr_band.cu — CG and Jacobi-PCG of src/linear (solver.rs:62-153) with matrix
// and vectors held on the chip, FP64, for CSR matrices whose rows and their
// band of columns fit the SMs' shared memory.
//
// A block owns `rows` consecutive rows. Their entries lie in shared memory by
// position in the row (entry k of consecutive rows side by side, so that a
// warp's reads do not conflict), and so do d, r and the inverse diagonal of
// every column that the rows can reach (own rows and a band on each side). An
// iteration is one pass q = A d over the own rows, which also forms the
// products d.q, r.Mr, q.Mr, q.Mq and r.r, one grid-wide sum (gridreduce.cuh),
// and one pass that updates x, r and d = M r + beta d on the own rows and, from
// the neighbours' q, on the band, with the owners' arithmetic. beta uses r.Mr - 2 alpha q.Mr + alpha^2 q.Mq of the
// directly summed products. ||r|| is tested where r.r is summed, one pass
// after its update; row sums keep the CSR order.
//
// What bounds it: the round through L2 (about 3 us) and the latency of the
// passes' gathers (262144 rows with a band of 1024: shared memory 47% busy, issue
// slots 37%). Per iteration, against the cooperative kernel with two
// barriers (csr.cu): 32768 rows with a band of 64 17 -> 4.1 us, 262144 rows
// with a band of 1024 18.5 -> 5.4 us. (With q as plain stores behind the
// round's fences instead of records: 7.0 and 6.5 us.)
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "csr_band.cuh"
#include "flursys_cuda.h"

namespace flursys {

namespace {

constexpr int kBandThreads = 512;
constexpr size_t kBandSmemMax = 220 * 1024;  // dynamic; the static part is below 3 KB

size_t band_smem(long long n, long long rows, long long band, long long width) {
    const long long win = std::min(n, rows + 2 * band);
    return (size_t)(24 * win + rows * (16 + 10 * width + 2) + 16);
}

struct BandScalars {
    double alpha, beta;
    int stop;
};

// KW: entries of the longest row (0: a.width, any).
template <int KW>
__global__ void __launch_bounds__(kBandThreads, 1) cg_band_kernel(const __grid_constant__ BandArgs a) {
    constexpr int T = kBandThreads;
    extern __shared__ __align__(16) char dyn[];
    __shared__ GridRedShared<T> red;
    __shared__ BandScalars sc;
    const int tid = threadIdx.x, n = a.n, R = a.rows, width = KW ? KW : a.width;
    const int r0 = blockIdx.x * R, r1 = min(n, r0 + R), nr = r1 - r0;
    const int lo = max(0, r0 - a.band), hi = min(n, r1 + a.band), win = hi - lo, own = r0 - lo;
    const int nh = win - nr;  // columns of the band
    double *dw = reinterpret_cast<double *>(dyn), *rw = dw + win, *iw = rw + win;
    double *qs = iw + win, *xs = qs + R, *va = xs + R;
    unsigned short *co = reinterpret_cast<unsigned short *>(va + (size_t)width * R), *len = co + (size_t)width * R;
    if (tid == 0) red.failed = 0;
    __syncthreads();
    GridGroup<T> grp{&red, a.records, nullptr, (int)gridDim.x, (int)blockIdx.x, 0, 0u, 0u, a.epoch, kRedSpinLimit, false};
    // Rows that another block's band reaches are published as records that
    // carry their round; two sets alternate.
    RedRecord *const values = a.records + 2 * (size_t)gridDim.x * kRedSlots;
    auto published = [&](int r) { return r < a.band || r >= nr - a.band; };
    auto halo = [&](int h) { return h < own ? h : h + nr; };  // window index of band column h
    // the value of a published row: a first look, then the wait
    auto await = [&](const RedRecord *p, double v, unsigned long long t, unsigned long long want) {
        long long spins = 0;
        while (t != want) {
            if (++spins > kRedSpinLimit) {
                red.failed = 1;
                break;
            }
            ld_record(p, v, t);
        }
        return v;
    };
    auto flag_row = [&](int row) { atomicMin(&a.res->bad_row, (unsigned long long)row); };
    auto row_sum = [&](int r) {
        double s = 0.0;
        const int l = len[r];
        if constexpr (KW > 0) {
#pragma unroll
            for (int k = 0; k < KW; ++k)
                if (k < l) s += va[k * R + r] * dw[co[k * R + r]];
        } else {
            for (int k = 0; k < l; ++k) s += va[(size_t)k * R + r] * dw[co[(size_t)k * R + r]];
        }
        return s;
    };

    // ---- matrix and x in; r = b - A x ----
    for (int r = tid; r < nr; r += T) {
        const int e0 = a.ro[r0 + r], l = a.ro[r0 + r + 1] - e0;
        len[r] = (unsigned short)l;
        for (int k = 0; k < l; ++k) {
            va[(size_t)k * R + r] = a.va[e0 + k];
            co[(size_t)k * R + r] = (unsigned short)(a.ci[e0 + k] - lo);
        }
        for (int k = l; k < width; ++k) {
            va[(size_t)k * R + r] = 0.0;
            co[(size_t)k * R + r] = (unsigned short)(own + r);
        }
    }
    for (int c = tid; c < win; c += T) {
        dw[c] = a.x[lo + c];
        iw[c] = a.inv_diag ? a.inv_diag[lo + c] : 1.0;
    }
    __syncthreads();
    double s[kRedSlots];
    auto clear = [&]() {
#pragma unroll
        for (int k = 0; k < kRedSlots; ++k) s[k] = 0.0;
    };
    clear();
    for (int r = tid; r < nr; r += T) {
        const double ax = row_sum(r);
        if (!isfinite(ax)) flag_row(r0 + r);
        const double rv = a.b[r0 + r] - ax;
        rw[own + r] = rv;
        xs[r] = dw[own + r];
        if (published(r)) st_record(values + r0 + r, rv, grp.tag(grp.fround));
        s[4] += rv * rv;
    }
    if (!grp.all(s, false, true)) return;
    double fin = sqrt(s[4]), rz_old = 1.0;
    const double initial = fin, threshold = a.atol + a.rtol * initial;
    int status = FLURSYS_LINEAR_MAX_ITERATIONS, error = 0;
    const int max_it = (int)max(0LL, min(a.max_iters, 2147483000LL));
    int it = 0;
    bool go = true;
    if (!isfinite(initial)) {
        error = FLURSYS_ERR_NON_FINITE;
        go = false;
    } else if (initial <= threshold) {
        status = FLURSYS_LINEAR_CONVERGED;
        go = false;
    }
    if (go) {
        for (int h = tid; h < nh; h += T) {
            const RedRecord *p = values + lo + halo(h);
            rw[halo(h)] = await(p, 0.0, ~0ull, grp.tag(grp.fround - 1u));
        }
        __syncthreads();
        for (int c = tid; c < win; c += T) dw[c] = rw[c] * iw[c];
        __syncthreads();
        clear();
        double sz = 0.0;  // r.Mr alone decides before the first pass
        for (int r = tid; r < nr; r += T) {
            if (!isfinite(dw[own + r])) flag_row(r0 + r);
            sz += rw[own + r] * dw[own + r];
        }
        s[1] = sz;
        if (!grp.all(s, false)) return;
        if (!isfinite(s[1])) {
            error = FLURSYS_ERR_NON_FINITE;
            go = false;
        } else if (max_it == 0) {
            go = false;
        }
    }
    // sums above this do not meet the threshold
    const double above = threshold * threshold * (1.0 + 1.0e-12), big = 1.0e300;
    constexpr int HP = 4;  // band values per thread that are read early
    while (go) {
        // ---- q = A d on the own rows ----
        clear();
        RedRecord *const fq = values + (size_t)(grp.fround & 1u) * n;
        const unsigned long long want = grp.tag(grp.fround);
        for (int r = tid; r < nr; r += T) {
            const double q = row_sum(r);
            if (!isfinite(q)) flag_row(r0 + r);
            qs[r] = q;
            if (published(r)) st_record(fq + r0 + r, q, want);
            const double d = dw[own + r], rv = rw[own + r], iv = iw[own + r], z = rv * iv;
            s[0] += d * q;
            s[1] += rv * z;
            s[2] += q * z;
            s[3] += q * iv * q;
            s[4] += rv * rv;
        }
        double hq[HP];
        unsigned long long ht[HP];
        const bool ok = grp.lead(s, false, true, 0, [&] {
#pragma unroll
            for (int u = 0; u < HP; ++u)
                if (tid + u * T < nh) ld_record(fq + lo + halo(tid + u * T), hq[u], ht[u]);
        });
        if (tid < 32) {
            const double den = s[0], rz = s[1], rr = s[4];
            int stop = 0;
            if (!ok) {
                stop = 2;
            } else {
                if (it > 0) {
                    if (!(rr > above && rr < big)) {
                        fin = sqrt(rr);
                        if (!isfinite(rr)) error = FLURSYS_ERR_NON_FINITE;
                        else if (fin <= threshold) status = FLURSYS_LINEAR_CONVERGED;
                    }
                    if (!error && status != FLURSYS_LINEAR_CONVERGED) {
                        if (!isfinite(rz)) error = FLURSYS_ERR_NON_FINITE;
                        else if (fabs(rz_old) <= 1.0e-30) error = FLURSYS_ERR_BREAKDOWN;
                        else if (fabs(rz) > 1.0e270 && !isfinite(rz / rz_old)) error = FLURSYS_ERR_BREAKDOWN;
                        else if (it >= max_it) stop = 1;
                    }
                    if (error || status == FLURSYS_LINEAR_CONVERGED) stop = 1;
                    if (stop) fin = sqrt(rr);
                }
                if (!stop) {
                    const bool plain = fabs(den) < big && fabs(rz) < big;
                    const double alpha = plain ? quotient(rz, den, fast_recip(den)) : rz / den;
                    double beta = rz + alpha * (alpha * s[3] - 2.0 * s[2]);
                    beta = plain && fabs(rz) > 1.0e-300 ? quotient(beta, rz, fast_recip(rz)) : beta / rz;
                    if (!isfinite(den)) error = FLURSYS_ERR_NON_FINITE;
                    else if (fabs(den) <= 1.0e-30 || !isfinite(alpha)) error = FLURSYS_ERR_BREAKDOWN;
                    if (error) stop = 1;
                    rz_old = rz;
                    if (tid == 0) {
                        sc.alpha = alpha;
                        sc.beta = beta;
                    }
                }
            }
            if (tid == 0) sc.stop = stop;
        }
        __syncthreads();
        const int stop = sc.stop;
        if (stop == 2) return;
        if (stop) break;
        // ---- x += alpha d, r -= alpha q, d = M r + beta d ----
        const double alpha = sc.alpha, beta = sc.beta;
        for (int r = tid; r < nr; r += T) {
            const int c = own + r;
            const double d = dw[c], rv = rw[c] - alpha * qs[r], z = rv * iw[c];
            xs[r] += alpha * d;
            rw[c] = rv;
            if (!isfinite(z)) flag_row(r0 + r);
            dw[c] = z + beta * d;
        }
        auto band = [&](int c, double q) {
            const double rv = rw[c] - alpha * q;
            rw[c] = rv;
            dw[c] = rv * iw[c] + beta * dw[c];
        };
#pragma unroll
        for (int u = 0; u < HP; ++u)
            if (tid + u * T < nh) {
                const int c = halo(tid + u * T);
                band(c, await(fq + lo + c, hq[u], ht[u], want));
            }
        for (int h = tid + HP * T; h < nh; h += T) {
            const int c = halo(h);
            band(c, await(fq + lo + c, 0.0, ~want, want));
        }
        ++it;
        __syncthreads();
    }
    for (int r = tid; r < nr; r += T) a.x[r0 + r] = xs[r];
    if (blockIdx.x == 0 && tid == 0) {
        a.res->error = error;
        a.res->status = status;
        a.res->iterations = status == FLURSYS_LINEAR_CONVERGED ? it : a.max_iters;
        a.res->initial = initial;
        a.res->final_residual = fin;
        a.res->device_error = 0;
    }
}

}  // namespace

BandPlan csr_band_plan(long long n, long long band, long long width, int device) {
    BandPlan p;
    int sms = 0;
    if (n < 1 || width < 1 || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) return p;
    // at least 128 rows per block: a pass over fewer is no shorter. Whatever fits
    // is faster here: the streaming kernel needs 17 us even for 4608 rows.
    const long long most = std::max(1LL, std::min<long long>(std::min(sms, 160), (n + 127) / 128));
    const long long rows = (n + most - 1) / most;
    band = std::min(band, n);
    if (width > 65535 || rows + 2 * band > (1LL << 30) || band_smem(n, rows, band, width) > kBandSmemMax) return p;
    p.rows = (int)rows;
    p.blocks = (int)((n + rows - 1) / rows);
    p.band = (int)band;
    p.width = (int)width;
    p.smem = band_smem(n, rows, band, width);
    p.kernel = width == 5   ? (const void *)cg_band_kernel<5>
               : width == 7 ? (const void *)cg_band_kernel<7>
                            : (const void *)cg_band_kernel<0>;
    int per_sm = 0;
    // the limit is the function's, which solves on several threads share:
    // always the same ceiling, never lowered
    if (cudaFuncSetAttribute(p.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBandSmemMax) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, p.kernel, kBandThreads, p.smem) != cudaSuccess || per_sm < 1) {
        cudaGetLastError();
        return BandPlan{};
    }
    return p;
}

size_t csr_band_record_bytes(const BandPlan &plan, long long n) {
    return sizeof(RedRecord) * 2 * ((size_t)kRedSlots * plan.blocks + (size_t)n);
}

cudaError_t csr_band_launch(const BandPlan &plan, const BandArgs &args, cudaStream_t stream) {
    BandArgs a = args;
    a.rows = plan.rows;
    a.band = plan.band;
    a.width = plan.width;
    void *params[] = {&a};
    return cudaLaunchCooperativeKernel(plan.kernel, dim3(plan.blocks), dim3(kBandThreads), params, plan.smem, stream);
}

}  // namespace flursys
