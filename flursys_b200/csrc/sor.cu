// sor.cu — red-black SOR for the 3D pinned pressure system.
//
// Each sweep updates the cells with (i+j+k) even, then the odd ones, with
// the SOR update of solve_pressure_poisson (src/solver/incompressible_3d.rs:
// 299-322): candidate = (sum of neighbours, a missing neighbour replaced by
// the centre value, minus rhs) / (2(ix2+iy2+iz2)); p += omega (candidate - p);
// p(0,0,0) = 0. After each sweep the reference stop residual
// max |Lap(p) - rhs| over cells other than (0,0,0) (:476-502) is reduced and
// tested against `tol`.
//
// Two kernels. sor3d_res keeps p and rhs on the chip: the grid is cut into
// slabs of z planes, one per block of a thread-block cluster or of a
// co-resident grid, each colour in its own shared array (so a row's cells of
// one colour are consecutive). The residual of a sweep is taken in the pass
// that also forms the next sweep's even cells, from the same neighbour sums,
// into a second array; their faces are sent at once, and the round that
// delivers the faces carries the residual's maximum. Where it meets the
// tolerance the first array holds the result and the sweep that was begun is
// not counted. A sweep so takes one round of the
// group and one exchange with the neighbours. What bounds it is latency: 32^3
// cells took 19.6 us per sweep with three grid barriers.
// The even faces that arrive during a sweep's residual pass go to a buffer of
// their own: a neighbour sends them as soon as it has the odd faces of the sweep
// before, while this block may still be reading the even ones it then received.
// sor3d_kernel streams p through L2, with three bounded grid barriers per
// sweep, for grids whose slabs do not fit.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>

#include "common.cuh"
#include "gridreduce.cuh"
#include "sor.cuh"

namespace flursys {

namespace {

constexpr int kBlock = 256;

struct G {
    int nx, ny, nz;
    long long nxy, n;
    double ix2, iy2, iz2;
};

__device__ __forceinline__ void decode(const G &g, long long c, int &i, int &j, int &k) {
    k = int(c / g.nxy);
    long long rem = c - (long long)k * g.nxy;
    j = int(rem / g.nx);
    i = int(rem - (long long)j * g.nx);
}

__device__ __forceinline__ double nbsum(const G &g, const double *p, long long c, int i, int j, int k,
                                        double pc) {
    const double e = (i + 1 < g.nx) ? __ldcg(p + c + 1) : pc;
    const double w = (i > 0) ? __ldcg(p + c - 1) : pc;
    const double n = (j + 1 < g.ny) ? __ldcg(p + c + g.nx) : pc;
    const double s = (j > 0) ? __ldcg(p + c - g.nx) : pc;
    const double f = (k + 1 < g.nz) ? __ldcg(p + c + g.nxy) : pc;
    const double b = (k > 0) ? __ldcg(p + c - g.nxy) : pc;
    return g.ix2 * (e + w) + g.iy2 * (n + s) + g.iz2 * (f + b);
}

__global__ void __launch_bounds__(kBlock) sor3d_kernel(int nx, int ny, int nz, double ix2, double iy2, double iz2,
                                                       double *p, const double *rhs, double omega, double tol,
                                                       long long max_iters, double *part, GridBarrier *bar,
                                                       PcgResultDev *res) {
    __shared__ double s_red[kBlock / 32];
    const G g{nx, ny, nz, (long long)nx * ny, (long long)nx * ny * nz, ix2, iy2, iz2};
    const double diag = 2.0 * (ix2 + iy2 + iz2);
    const long long stride = (long long)gridDim.x * kBlock;
    const long long tid0 = (long long)blockIdx.x * kBlock + threadIdx.x;
    double residual = INFINITY;
    long long its = 0;
    int error = 0;
    for (long long it = 0; it < max_iters; ++it) {
        its = it + 1;
        for (int color = 0; color < 2; ++color) {
            for (long long c = tid0; c < g.n; c += stride) {
                int i, j, k;
                decode(g, c, i, j, k);
                if (((i + j + k) & 1) != color) continue;
                if (c == 0) { p[0] = 0.0; continue; }
                const double pc = __ldcg(p + c);
                const double cand = (nbsum(g, p, c, i, j, k, pc) - __ldcg(rhs + c)) / diag;
                p[c] = pc + omega * (cand - pc);
            }
            if (!grid_sync_report(bar, gridDim.x, &res->device_error)) return;
        }
        double m = 0.0;
        for (long long c = tid0; c < g.n; c += stride) {
            if (c == 0) continue;
            int i, j, k;
            decode(g, c, i, j, k);
            const double pc = __ldcg(p + c);
            const double lap = nbsum(g, p, c, i, j, k, pc) - diag * pc;
            m = fmax(m, fabs(lap - __ldcg(rhs + c)));
        }
        const double bm = block_max<kBlock>(m, s_red);
        if (threadIdx.x == 0) part[blockIdx.x * 4 + (it & 1)] = bm;
        if (!grid_sync_report(bar, gridDim.x, &res->device_error)) return;
        double s = 0.0;
        for (int b = threadIdx.x; b < (int)gridDim.x; b += kBlock) s = fmax(s, __ldcg(&part[b * 4 + (it & 1)]));
        residual = block_max<kBlock>(s, s_red);
        if (!isfinite(residual)) { error = FLURSYS_ERR_NON_FINITE; break; }
        if (residual < tol) break;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        res->error = error;
        res->status = residual < tol ? FLURSYS_LINEAR_CONVERGED : FLURSYS_LINEAR_MAX_ITERATIONS;
        res->iterations = its;
        res->initial = 0.0;
        res->residual = residual;
        res->true_l2 = 0.0;
        res->initial_l2 = 0.0;
        res->device_error = bar->error;
    }
}

struct SorArgs {
    int nx, ny, nz;
    double ix2, iy2, iz2;
    double *p;
    const double *rhs;
    double omega, tol;
    long long max_iters;
    PcgResultDev *res;
    RedRecord *records, *faces;
    unsigned epoch;
};

constexpr int kResT = 512;

// Cells of one colour in a row, and doubles per plane of one colour.
__host__ __device__ __forceinline__ int half_row(int nx) { return (nx + 1) / 2; }
__host__ __device__ __forceinline__ size_t sor_smem(int nx, int ny, int planes, bool cluster) {
    const size_t hp = (size_t)half_row(nx) * ny;
    // p (the even cells twice) and rhs; two halo planes by colour, in a cluster the even ones twice
    return 8 * hp * (5 * (size_t)planes + (cluster ? 6 : 4));
}

template <bool CLUSTER, typename Group>
__device__ __forceinline__ bool sor3d_solve(const SorArgs &a, Group &grp, char *dyn) {
    const int nx = a.nx, ny = a.ny, nz = a.nz, tid = threadIdx.x, h = half_row(nx), hp = h * ny;
    const int planes = (nz + grp.nb - 1) / grp.nb, k0 = min(grp.rank * planes, nz), np = min(planes, nz - k0);
    const bool has_lo = np > 0 && k0 > 0, has_hi = np > 0 && k0 + np < nz;
    const double diag = 2.0 * (a.ix2 + a.iy2 + a.iz2), inv = 1.0 / diag;
    double *P[2], *R[2], *H[2];  // by colour; H: the planes below and above, as read
    P[0] = reinterpret_cast<double *>(dyn);
    double *next_even = P[0] + (size_t)planes * hp;
    P[1] = next_even + (size_t)planes * hp;
    R[0] = P[1] + (size_t)planes * hp;
    R[1] = R[0] + (size_t)planes * hp;
    H[0] = R[1] + (size_t)planes * hp;
    H[1] = H[0] + 2 * (size_t)hp;
    double *next_even_halo = CLUSTER ? H[1] + 2 * (size_t)hp : H[0];  // CLUSTER: where the coming even faces arrive
    // cells of colour c in plane k (a row of parity s = (c + j + k) & 1 holds i = 2 m + s)
    auto count = [&](int c, int k) {
        const int odd_rows = (c + k) & 1 ? (ny + 1) / 2 : ny / 2;  // rows with s = 1
        return odd_rows * (nx / 2) + (ny - odd_rows) * ((nx + 1) / 2);
    };
    auto bytes = [&](int c) {
        return 8u * (unsigned)((has_lo ? count(c, k0 - 1) : 0) + (has_hi ? count(c, k0 + np) : 0));
    };
    // f(kk, j, m, o) over the slots of one colour; slot o = (kk ny + j) h + m
    const int step_r = kResT / h, step_m = kResT - step_r * h;
    const int r0 = tid / h, m0 = tid - r0 * h, kk0 = r0 / ny, j0 = r0 - kk0 * ny, rows = np * ny;
    auto each = [&](auto f) {
        int m = m0, j = j0, kk = kk0, r = r0;
        while (r < rows) {
            f(kk, j, m, r * h + m);
            m += step_m;
            int dr = step_r;
            if (m >= h) {
                m -= h;
                ++dr;
            }
            r += dr;
            j += dr;
            while (j >= ny) {
                j -= ny;
                ++kk;
            }
        }
    };
    for (int c = 0; c < 2; ++c) {
        each([&](int kk, int j, int m, int o) {
            const int k = k0 + kk, i = 2 * m + ((c + j + k) & 1);
            const bool ok = i < nx;
            const size_t g = ok ? (size_t)i + (size_t)nx * (j + (size_t)ny * k) : 0;
            P[c][o] = ok ? a.p[g] : 0.0;
            R[c][o] = ok ? __ldg(a.rhs + g) : 0.0;
        });
        for (int t = tid; t < 2 * hp; t += kResT) {
            const int side = t >= hp, q = t - side * hp, j = q / h, k = side ? k0 + np : k0 - 1;
            const int i = 2 * (q - j * h) + ((c + j + k) & 1);
            const bool ok = (side ? has_hi : has_lo) && i < nx;
            H[c][t] = ok ? __ldcg(a.p + (size_t)i + (size_t)nx * (j + (size_t)ny * k)) : 0.0;
        }
    }
    if (!grp.barrier()) return false;  // every slab is read before one is written back

    // sum of the neighbours of a cell of colour c, a missing one replaced by pc
    auto nbs = [&](int c, int kk, int j, int m, int o, double pc) -> double {
        const int k = k0 + kk, s = (c + j + k) & 1, i = 2 * m + s, q = j * h + m;
        const double *Q = P[1 - c];
        const double e = i + 1 < nx ? Q[o + s] : pc, w = i > 0 ? Q[o + s - 1] : pc;
        const double n = j + 1 < ny ? Q[o + h] : pc, so = j > 0 ? Q[o - h] : pc;
        const double f = kk + 1 < np ? Q[o + hp] : has_hi ? H[1 - c][hp + q] : pc;
        const double b = kk > 0 ? Q[o - hp] : has_lo ? H[1 - c][q] : pc;
        return a.ix2 * (e + w) + a.iy2 * (n + so) + a.iz2 * (f + b);
    };
    auto send = [&](int c, int kk, int j, int m, double v) {
        const int q = j * h + m;
        if constexpr (CLUSTER) {
            const uint32_t to = smem_addr(c ? H[1] : next_even_halo);
            if (kk == 0 && has_lo) grp.send_to(grp.rank - 1, to + 8u * (uint32_t)(hp + q), v);
            if (kk == np - 1 && has_hi) grp.send_to(grp.rank + 1, to + 8u * (uint32_t)q, v);
        } else {
            if (kk == 0 && has_lo) grp.send(grp.rank - 1, hp + q, v);
            if (kk == np - 1 && has_hi) grp.send(grp.rank + 1, q, v);
        }
    };
    // the halo planes of colour c from the exchange that has ended (grid form;
    // in the cluster form they are there)
    auto take_halo = [&](int c) {
        if constexpr (!CLUSTER) {
            for (int t = tid; t < 2 * hp; t += kResT) {
                const int side = t >= hp, q = t - side * hp, j = q / h, k = side ? k0 + np : k0 - 1;
                if (!(side ? has_hi : has_lo) || 2 * (q - j * h) + ((c + j + k) & 1) >= nx) continue;
                double v;
                unsigned long long tt;
                grp.peek(t, v, tt);
                H[c][t] = grp.take(t, v, tt);
            }
        }
    };

    double residual = INFINITY;  // warp 0's
    long long its = 0;
    int error = 0;
    __shared__ int s_cmd, s_got;
    while (a.max_iters > 0) {
        // ---- the residual of the sweeps so far, and the next even cells ----
        double v[kRedSlots] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0}, mx = 0.0;
        const bool more = its < a.max_iters;
        each([&](int kk, int j, int m, int o) {
            if (2 * m + ((1 + j + k0 + kk) & 1) >= nx) return;
            const double pc = P[1][o];
            mx = fmax(mx, fabs((nbs(1, kk, j, m, o, pc) - diag * pc) - R[1][o]));
        });
        each([&](int kk, int j, int m, int o) {
            const int i = 2 * m + ((j + k0 + kk) & 1);
            if (i >= nx) return;
            const double pc = P[0][o];
            double val = 0.0;  // p(0, 0, 0)
            if (i + j + k0 + kk > 0) {
                const double sum = nbs(0, kk, j, m, o, pc);
                mx = fmax(mx, fabs((sum - diag * pc) - R[0][o]));
                val = pc + a.omega * (rounded_quotient(sum - R[0][o], diag, inv) - pc);
            }
            next_even[o] = val;
            if (more) send(0, kk, j, m, val);
        });
        v[7] = mx;
        const bool ok = grp.lead(v, true, more, bytes(0), [] {});
        if (tid < 32 && its > 0) residual = v[7];
        if (tid == 0) s_cmd = !ok ? 2 : its > 0 && (!isfinite(v[7]) || v[7] < a.tol || !more) ? 1 : 0;
        __syncthreads();
        if (s_cmd == 2) return false;
        if (s_cmd == 1) break;
        double *t = P[0];
        P[0] = next_even;
        next_even = t;
        t = H[0];
        H[0] = next_even_halo;
        next_even_halo = t;
        take_halo(0);
        if (!CLUSTER) __syncthreads();
        // ---- odd cells ----
        each([&](int kk, int j, int m, int o) {
            const int k = k0 + kk;
            if (2 * m + ((1 + j + k) & 1) >= nx) return;
            const double pc = P[1][o];
            const double val = pc + a.omega * (rounded_quotient(nbs(1, kk, j, m, o, pc) - R[1][o], diag, inv) - pc);
            P[1][o] = val;
            send(1, kk, j, m, val);
        });
        const bool got = grp.exchange(bytes(1));
        if (tid == 0) s_got = got;
        take_halo(1);
        __syncthreads();
        if (!s_got) return false;
        ++its;
    }
    __syncthreads();
    if (its > 0 && tid == 0 && !isfinite(residual)) error = FLURSYS_ERR_NON_FINITE;
    for (int c = 0; c < 2; ++c)
        each([&](int kk, int j, int m, int o) {
            const int k = k0 + kk, i = 2 * m + ((c + j + k) & 1);
            if (i < nx) a.p[(size_t)i + (size_t)nx * (j + (size_t)ny * k)] = P[c][o];
        });
    if (grp.rank == 0 && tid == 0) {
        PcgResultDev *res = a.res;
        res->error = error;
        res->status = residual < a.tol ? FLURSYS_LINEAR_CONVERGED : FLURSYS_LINEAR_MAX_ITERATIONS;
        res->iterations = its;
        res->initial = 0.0;
        res->residual = residual;
        res->true_l2 = 0.0;
        res->initial_l2 = 0.0;
    }
    return true;
}

__global__ void __launch_bounds__(kResT, 1) sor3d_res_cluster(SorArgs a) {
    extern __shared__ __align__(16) char dyn[];
    __shared__ ClusterRedShared<kResT> red;
    ClusterGroup<kResT> grp{&red, (int)gridDim.x, (int)blockIdx.x, 0, 0u, 0u, 0u};
    grp.init();
    if (!sor3d_solve<true>(a, grp, dyn) && threadIdx.x == 0)
        atomicOr(&a.res->device_error, (unsigned)kDevErrBarrierTimeout);
    grp.finish();
}

__global__ void __launch_bounds__(kResT, 1) sor3d_res_grid(SorArgs a) {
    extern __shared__ __align__(16) char dyn[];
    __shared__ GridRedShared<kResT> red;
    if (threadIdx.x == 0) red.failed = 0;
    __syncthreads();
    GridGroup<kResT> grp{&red, a.records, a.faces, (int)gridDim.x, (int)blockIdx.x, 2 * half_row(a.nx) * a.ny, 0u, 0u,
                         a.epoch, kRedSpinLimit, false};
    if (!sor3d_solve<false>(a, grp, dyn) && threadIdx.x == 0)
        atomicOr(&a.res->device_error, (unsigned)kDevErrBarrierTimeout);
}

constexpr size_t kSorSmemMax = 222 * 1024;

// Blocks of a slab decomposition into at most `most` blocks; 0 where a slab
// does not fit a block.
int sor_blocks(int nx, int ny, int nz, int most, bool cluster) {
    const int planes = (nz + most - 1) / most;
    if (sor_smem(nx, ny, planes, cluster) > kSorSmemMax) return 0;
    return (nz + planes - 1) / planes;
}

}  // namespace

cudaError_t sor3d_plan(Sor3dPlan &plan, int nx, int ny, int nz, int device) {
    plan = Sor3dPlan{};
    const char *env = std::getenv("FLURSYS_SOR_RESIDENT");
    if (env && std::strcmp(env, "0") == 0) return cudaSuccess;
    const bool may_cluster = !(env && std::strcmp(env, "grid") == 0);
    int sms = 0;
    cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    if (e != cudaSuccess) return e;
    const int nc = may_cluster ? sor_blocks(nx, ny, nz, 16, true) : 0;
    if (nc > 0) {
        plan.smem = sor_smem(nx, ny, (nz + 15) / 16, true);
        // the limit is the function's, which handles on several threads share:
        // always the same ceiling, never lowered
        if (cudaFuncSetAttribute(sor3d_res_cluster, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSorSmemMax) == cudaSuccess &&
            cudaFuncSetAttribute(sor3d_res_cluster, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) {
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = nc;
            attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
            cudaLaunchConfig_t cfg{};
            cfg.gridDim = dim3(nc);
            cfg.blockDim = dim3(kResT);
            cfg.dynamicSmemBytes = plan.smem;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            int active = 0;
            if (cudaOccupancyMaxActiveClusters(&active, (const void *)sor3d_res_cluster, &cfg) == cudaSuccess && active >= 1) {
                plan.blocks = nc;
                plan.cluster = true;
                return cudaSuccess;
            }
        }
        cudaGetLastError();
    }
    const int most = std::min(sms, 160), ng = sor_blocks(nx, ny, nz, most, false);
    if (ng == 0) return cudaSuccess;
    plan.smem = sor_smem(nx, ny, (nz + most - 1) / most, false);
    int per_sm = 0;
    if (cudaFuncSetAttribute(sor3d_res_grid, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSorSmemMax) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, sor3d_res_grid, kResT, plan.smem) != cudaSuccess || per_sm < 1) {
        cudaGetLastError();
        return cudaSuccess;
    }
    const size_t bytes = sizeof(RedRecord) * 2 * ng * (kRedSlots + 2 * (size_t)half_row(nx) * ny);
    if (cudaMalloc(&plan.records, bytes) != cudaSuccess || cudaMemset(plan.records, 0, bytes) != cudaSuccess ||
        cudaStreamSynchronize(nullptr) != cudaSuccess) {  // solves run on streams that do not wait for this one
        sor3d_destroy(plan);  // no room: the streaming kernel serves the solve
        cudaGetLastError();
        return cudaSuccess;
    }
    plan.blocks = ng;
    return cudaSuccess;
}

void sor3d_destroy(Sor3dPlan &plan) {
    cudaFree(plan.records);
    plan = Sor3dPlan{};
}

int32_t run_sor3d(Sor3dPlan &plan, PcgWorkspace &ws, int nx, int ny, int nz, double dx, double dy, double dz, double *p,
                  const double *rhs, double omega, double tol, long long max_iters, cudaStream_t stream,
                  std::string *err) {
    double ix2 = 1.0 / (dx * dx), iy2 = 1.0 / (dy * dy), iz2 = 1.0 / (dz * dz);
    cudaError_t e;
    if (plan.blocks > 0) {
        SorArgs a{nx, ny, nz, ix2, iy2, iz2, p, rhs, omega, tol, max_iters, ws.result, plan.records,
                  plan.records + 2 * (size_t)plan.blocks * kRedSlots, ++plan.epoch};
        e = cudaMemsetAsync(ws.result, 0, sizeof(PcgResultDev), stream);
        void *params[] = {&a};
        cudaLaunchAttribute attr[1];
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(plan.blocks);
        cfg.blockDim = dim3(kResT);
        cfg.dynamicSmemBytes = plan.smem;
        cfg.stream = stream;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        const void *fn = plan.cluster ? (const void *)sor3d_res_cluster : (const void *)sor3d_res_grid;
        if (plan.cluster) {
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = plan.blocks;
            attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        } else {
            attr[0].id = cudaLaunchAttributeCooperative;
            attr[0].val.cooperative = 1;
        }
        if (e == cudaSuccess) e = cudaLaunchKernelExC(&cfg, fn, params);
        if (e != cudaSuccess) return set_cuda_error(err, e, "sor3d launch");
        return FLURSYS_OK;
    }
    int per_sm = 0, sms = 0, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, sor3d_kernel, kBlock, 0);
    int grid = ws.grid;
    if (grid > sms * per_sm) grid = sms * per_sm;
    void *params[] = {&nx, &ny, &nz, &ix2, &iy2, &iz2, &p, &rhs, &omega, &tol, &max_iters, &ws.partials, &ws.barrier,
                      &ws.result};
    e = cudaMemsetAsync(ws.barrier, 0, sizeof(GridBarrier), stream);
    if (e == cudaSuccess)
        e = cudaLaunchCooperativeKernel((const void *)sor3d_kernel, dim3(grid), dim3(kBlock), params, 0, stream);
    if (e != cudaSuccess) return set_cuda_error(err, e, "sor3d launch");
    return FLURSYS_OK;
}

}  // namespace flursys
