// pcg2d_res.cu — the 2D pressure PCG with its state held on the chip for the
// whole solve and one group-wide synchronisation per iteration.
//
// The system, preconditioner, zero-mean projections, stop rules and error
// tests are those of pcg2d.cu (solve_pressure_pcg, src/solver/
// incompressible.rs:1048-1214). Each block of the group owns a run of grid
// rows; r, q = A d, the direction d with a halo row on each side and the FP64
// solution x lie in shared memory. An iteration is
//
//   q = A d; the block's first and last row of q to the neighbours;
//   one reduction of d.q, r.Mr, q.Mr, q.Mq, sum r, sum Mr, sum d and r.r
//   (or max |r|);
//   stop test on r; alpha = r.Mr / d.q; x += alpha (d - mean d);
//   r -= alpha q; beta from r.Mr - 2 alpha q.Mr + alpha^2 q.Mq;
//   d = M r + beta d, on the own rows and, with the neighbours' q, on the halo.
//
// The residual is tested where it is summed, in the reduction after its
// update, so the accepted iterate is the one the two-reduction form accepts.
// Only beta uses the expansion; the next reduction sums r.Mr directly again,
// so nothing accumulates. The halo's r, d are updated with the owner's fused
// operations and stay bit-identical to it. The means that the projections
// remove are those of the reduction before (d's is exact when x uses it), and
// x itself is projected once at the end: A annihilates constants, so these
// shifts are rounding-sized and change no iterate.
//
// MIXED: r, q and d are FP32; every product of the inner products is formed and
// summed in FP64; alpha, beta, the means and 1/diagonal are FP64, r and d are
// updated in FP64 and rounded as they are stored. x is FP64, and r is replaced
// by the FP64 b - A x every replace_every iterations and before convergence is
// accepted (d then exchanges M r_old for M r_new, and the operator pass is
// repeated). The queue's kernel, whose x takes half of the registers, applies the
// scalars and weights rounded to FP32, the same alpha to x and r. Against 64
// bits, as multiples of the streaming kernel's pressure errors: FP32 scalars 1.24
// +- 0.07 for single cavities at 3e-11, where FP64 ones give 1.05, but 0.6 to 1.1
// for batches, where FP64 ones give 1.2 (they stop the solves 4% sooner) and took
// 8 to 15% longer per iteration (a cluster 6%, the grid on 640 x 480 8%, at up to
// 7% fewer iterations).
//
// What bounds it: latency. On small grids that of the block reduction, the
// exchange and the scalars' chain; on large ones also the passes', two warps per
// scheduler (four in the queue) that keep issue slots 25% (55%) busy and wait on
// L2, shared memory and barriers. A lane takes 16 bytes
// of a row at a time, and without solid or outlet cells the direction's ghost
// cells hold the wall cell's own value, so that the operator has no boundary
// case (a pass that derived each cell's position and couplings spent 240
// instructions on a cell and iteration, most of them integer). The passes are
// rolled loops: unrolled
// over a thread's cells with r and q in registers they outgrew the instruction
// cache (on B200 a loop runs at about 1.2 cycles per instruction up to 1000
// instructions and at 3 to 6.6 from 4000 on).
//
// Two forms share the code: a thread-block cluster (partials and faces through
// distributed shared memory) and a co-resident grid (through L2), both with
// the one-hop rounds of gridreduce.cuh.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <type_traits>

#include "pcg2d_res.cuh"

namespace flursys {

namespace {

__device__ __forceinline__ float vfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double vfma(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float vadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double vadd(double a, double b) { return __dadd_rn(a, b); }
// r - alpha q less its mean, and M r + shift + beta d, as they are stored: the
// owner of a cell and the halo copies of it form the same bits. S: the type of the
// scalars and of the arithmetic.
template <typename S, typename V>
__device__ __forceinline__ V next_r(S alpha, V q, V r, S mean) {
    return V(vadd(vfma(-alpha, S(q), S(r)), -mean));
}
template <typename S, typename V>
__device__ __forceinline__ V next_d(S beta, V d, V r, S inv, S shift) {
    return V(vfma(beta, S(d), vfma(S(r), inv, shift)));
}

enum : unsigned { kE = 1, kW = 2, kN = 4, kS = 8, kFluid = 16 };

// Cells of a 16-byte vector.
template <typename V>
constexpr int kVec = 16 / (int)sizeof(V);
// Row pitch of the shared arrays: whole vectors, and one vector in front that
// holds d's ghost column (the ghost behind the row lies in its own last vector
// or in the next row's front).
template <typename V>
__host__ __device__ __forceinline__ int res2d_pitch(int nx) {
    return (nx + kVec<V> - 1) / kVec<V> * kVec<V> + kVec<V>;
}

// Shared-memory footprint of a block that owns `rows` grid rows: r, q and d
// with its halo rows, the halo's r, coupling bits and (cluster) two sets of
// received faces, x unless it is in registers, and the coupling bits unless
// every cell is fluid.
template <typename V, bool CLUSTER>
__host__ __device__ size_t res2d_smem(int rows, int nx, bool xreg, bool plain) {
    const size_t p = res2d_pitch<V>(nx), c = (size_t)rows * p;
    size_t b = (xreg ? 0 : 8 * c) + sizeof(V) * (3 * c + (CLUSTER ? 8 : 4) * p + 2 * kVec<V>) + 2 * p;
    if (!plain) b += c;
    return (b + 15) & ~size_t(15);
}

template <typename V>
__device__ __forceinline__ void ldv(const V *p, V (&a)[kVec<V>]) {
    const uint4 t = *reinterpret_cast<const uint4 *>(p);
    memcpy(a, &t, 16);
}
template <typename V>
__device__ __forceinline__ void stv(V *p, const V (&a)[kVec<V>]) {
    uint4 t;
    memcpy(&t, a, 16);
    *reinterpret_cast<uint4 *>(p) = t;
}

template <int T, bool CLUSTER>
struct Res2dGroup {
    using type = GridGroup<T>;
};
template <int T>
struct Res2dGroup<T, true> {
    using type = ClusterGroup<T>;
};

// 1 / diagonal by coupling bits; 0 marks a row that is not fluid.
struct Res2dTable {
    double inv[32];
    float inv32[32];  // the same where they are FP32 numbers
};
template <typename S>
__device__ __forceinline__ S weight_of(const Res2dTable &t, unsigned bits) {
    if constexpr (sizeof(S) == 4) return t.inv32[bits];
    else return t.inv[bits];
}

// What warp 0 hands the block after an iteration's reduction.
enum : int { kStep = 0, kStop = 1, kRefresh = 2, kFail = 3 };
struct Res2dScalars {
    double alpha, md, mr, beta, shift;  // x += alpha (d - md); r -= alpha q + mr; d = M r + beta d + shift
    int cmd;
};

// The cell's coupling bits.
__device__ __forceinline__ unsigned cell_bits(const Pcg2dInstance &in, bool plain, int g) {
    const int j = g / in.nx, i = g - j * in.nx;
    unsigned b = kFluid;
    if (i + 1 < in.nx) b |= kE;
    if (i > 0) b |= kW;
    if (j + 1 < in.ny) b |= kN;
    if (j > 0) b |= kS;
    if (plain) return b;
    const uint8_t *f = in.flags;
    if (f[g] & 3) return 0u;
    if ((b & kE) && (f[g + 1] & kCellSolid)) b &= ~kE;
    if ((b & kW) && (f[g - 1] & kCellSolid)) b &= ~kW;
    if ((b & kN) && (f[g + in.nx] & kCellSolid)) b &= ~kN;
    if ((b & kS) && (f[g - in.nx] & kCellSolid)) b &= ~kS;
    return b;
}

// One instance on its group of nb blocks; rank is this block's index in it.
// XN > 0: x in registers, at most XN cells per thread. PLAIN: every cell is
// fluid.
template <typename V, int T, int XN, bool CLUSTER, bool PLAIN>
__device__ __forceinline__ bool res2d_solve(const Pcg2dInstance &in, typename Res2dGroup<T, CLUSTER>::type &grp,
                                            char *dyn, Res2dTable &tab, Res2dScalars &sc) {
    constexpr bool MIXED = sizeof(V) == 4;
    constexpr int W = kVec<V>, U = 4 / W;  // cells per vector, vectors per trip
    constexpr int XV = (XN + W - 1) / W;   // vectors of x in registers
    constexpr int NW = T / 32;
    using S = std::conditional_t<XN == 0, double, V>;  // of the scalars as they are applied
    const int nx = in.nx, ny = in.ny, tid = threadIdx.x, lane = tid & 31;
    const int rows = (ny + grp.nb - 1) / grp.nb;
    const int j0 = min(grp.rank * rows, ny), nr = min(rows, ny - j0);
    const int P = res2d_pitch<V>(nx);
    const bool has_lo = nr > 0 && j0 > 0, has_hi = nr > 0 && j0 + nr < ny;
    const bool proj = in.project != 0;
    const bool linf = in.stop_rule != FLURSYS_STOP_REL_L2;
    const double cnt = in.count_fluid > 0 ? double(in.count_fluid) : 1.0;
    const double inv_cnt = proj ? 1.0 / cnt : 0.0;
    const size_t cpad = (size_t)rows * P;
    // Cell (row, i) of the block at row * P + i; d one row and one vector further.
    double *xs = reinterpret_cast<double *>(dyn);
    V *rs = reinterpret_cast<V *>(xs + (XN ? 0 : cpad));
    V *qs = rs + cpad;
    V *ds = qs + cpad;
    V *hr = ds + cpad + 2 * (size_t)P + 2 * W;  // halo: [below, above][P]
    V *hq = hr + 2 * (size_t)P;  // CLUSTER: face values received, by round parity
    uint8_t *hb = reinterpret_cast<uint8_t *>(hq + (CLUSTER ? 4 * (size_t)P : 0));  // the halo's coupling bits
    uint8_t *bs = hb + 2 * (size_t)P;
    V *const dc0 = ds + P + W;  // d of cell (0, 0)
    if constexpr (CLUSTER) {
        grp.face_slots = 2 * P;
        grp.faces = smem_addr(hq);
    }
    // bytes of face data this block receives in a round that sends faces
    const unsigned face_bytes = ((has_lo ? 1u : 0u) + (has_hi ? 1u : 0u)) * (unsigned)(nx * sizeof(V));

    if (tid < 32) {  // 1 / diagonal by coupling bits; 0 marks a row that is not fluid
        const double dg = double((tid & 1) + ((tid >> 1) & 1)) * in.idx2 + double(((tid >> 2) & 1) + ((tid >> 3) & 1)) * in.idy2;
        tab.inv[tid] = (tid & kFluid) ? (dg > 0.0 ? double(S(1.0 / dg)) : 1.0) : 0.0;
        tab.inv32[tid] = float(tab.inv[tid]);
    }
    for (int k = tid; k < (int)cpad + 2 * P + 2 * W; k += T) ds[k] = V(0);
    for (int k = tid; k < (int)cpad; k += T) rs[k] = qs[k] = V(0);
    __syncthreads();
    const V wx = V(in.idx2), wy = V(in.idy2);

    // A warp's walk over its pieces (32 vectors of a row) of the block's rows.
    const int wid = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int nvec = (nx + W - 1) / W, strips = (nvec + 31) >> 5;
    const int step_row = NW / strips, step_strip = NW - step_row * strips;
    struct Walk {
        int row, strip;
    };
    auto first = [&]() { return Walk{wid / strips, wid % strips}; };
    auto next = [&](Walk &w) {
        w.row += step_row;
        w.strip += step_strip;
        if (w.strip >= strips) {
            w.strip -= strips;
            ++w.row;
        }
    };
    // coupling bits of a cell when every cell is fluid
    auto row_bits = [&](int row) -> unsigned {
        return kFluid | (j0 + row + 1 < ny ? kN : 0u) | (j0 + row > 0 ? kS : 0u);
    };
    auto col_bits = [&](int i) -> unsigned { return (i + 1 < nx ? kE : 0u) | (i > 0 ? kW : 0u); };
    // f(row, column, offset, bits) over the own cells
    auto each_cell = [&](auto f) {
        for (int row = wid; row < nr; row += NW)
            for (int i = lane; i < nx; i += 32)
                f(row, i, row * P + i, PLAIN ? row_bits(row) | col_bits(i) : (unsigned)bs[row * P + i]);
    };
    auto fluid = [&](int o) -> bool { return PLAIN || (bs[o] & kFluid); };
    double xr[XN ? XV * W : 1] = {};
    // f(column, row, offset, x) over the own cells, x by reference, each cell
    // by the thread whose vector it is in
    auto each_x = [&](auto f) {
        Walk w = first();
        if constexpr (XN > 0) {
            // opaque, so that the offsets are formed here and not kept in
            // registers across the iteration
            asm volatile("" : "+r"(w.row), "+r"(w.strip));
#pragma unroll
            for (int u = 0; u < XV; ++u) {
                const int i = (w.strip * 32 + lane) * W;
#pragma unroll
                for (int k = 0; k < W; ++k)
                    if (w.row < nr && i + k < nx) f(i + k, w.row, w.row * P + i + k, xr[u * W + k]);
                next(w);
            }
        } else {
            for (; w.row < nr; next(w)) {
                const int i = (w.strip * 32 + lane) * W;
#pragma unroll
                for (int k = 0; k < W; ++k)
                    if (i + k < nx) f(i + k, w.row, w.row * P + i + k, xs[w.row * P + i + k]);
            }
        }
    };
    // Writes d of a cell and, at the domain's walls, its ghosts (PLAIN).
    auto put_d = [&](int row, int i, int o, V v) {
        V *p = dc0 + o;
        *p = v;
        if (PLAIN) {
            if (i == 0) p[-1] = v;
            if (i == nx - 1) p[1] = v;
            if (row == 0 && !has_lo) p[-P] = v;
            if (row == nr - 1 && !has_hi) p[P] = v;
        }
    };
    double s[kRedSlots];
    auto clear = [&]() {
#pragma unroll
        for (int k = 0; k < kRedSlots; ++k) s[k] = 0.0;
    };
    // The block's first row of `a` into the upper halo of the block below, the
    // last row into the lower halo of the block above (after a block barrier
    // that follows the writes of `a`).
    auto send_faces = [&](const V *a) {
        if (has_lo)
            for (int i = tid; i < nx; i += T) grp.send(grp.rank - 1, P + i, a[i]);
        if (has_hi)
            for (int i = tid; i < nx; i += T) grp.send(grp.rank + 1, i, a[(nr - 1) * P + i]);
    };
    // f(halo slot, its d, its value from the last round) over the fluid halo
    // cells; the grid form has already looked at the first two per thread.
    // Halo cell t: column t of the row below, then of the row above.
    const int nlo = has_lo ? nx : 0, nh = nlo + (has_hi ? nx : 0);
    auto hslot = [&](int t) { return t < nlo ? t : P + t - nlo; };
    auto hd = [&](int h) -> V & { return h < P ? dc0[h - P] : dc0[nr * P + h - P]; };
    double pv[2] = {0.0, 0.0};
    unsigned long long pt[2] = {0ull, 0ull};
    auto peek_halo = [&]() {
        if constexpr (!CLUSTER) {
#pragma unroll
            for (int k = 0; k < 2; ++k)
                if (tid + k * T < nh) grp.peek(hslot(tid + k * T), pv[k], pt[k]);
        }
    };
    auto each_halo = [&](auto f) {
        int k = 0;
        for (int t = tid; t < nh; t += T, ++k) {
            const int h = hslot(t);
            V v;
            if constexpr (CLUSTER) {
                v = grp.face(hq, h);
            } else {
                double tv = k == 0 ? pv[0] : pv[1];
                unsigned long long tt = k == 0 ? pt[0] : pt[1];
                if (k > 1) grp.peek(h, tv, tt);
                v = V(grp.take(h, tv, tt));
            }
            if (PLAIN || (hb[h] & kFluid)) f(h, hd(h), v);
        }
    };

    // pressure of a coupled neighbour
    auto xnb = [&](int g) -> double {
        if (!PLAIN && (in.flags[g] & kCellOutlet)) return in.outlet_pressure;
        return __ldcg(in.x + g);
    };

    // ---- set-up: bits, x, the halo's bits; sums of x and b ----
    clear();
    if (!PLAIN) {
        for (int row = wid; row < nr; row += NW)
            for (int i = lane; i < P; i += 32)
                bs[row * P + i] = i < nx ? (uint8_t)cell_bits(in, false, (j0 + row) * nx + i) : (uint8_t)0;
        __syncthreads();
    }
    each_x([&](int i, int row, int o, double &x) {
        const int g = (j0 + row) * nx + i;
        const bool fl = fluid(o);
        x = fl ? in.x[g] : 0.0;
        s[0] += x;
        if (fl) s[1] -= __ldg(in.rhs + g);
    });
    for (int t = tid; t < nh; t += T) {
        const int h = hslot(t), g = h < P ? (j0 - 1) * nx + h : (j0 + nr) * nx + h - P;
        hr[h] = V(0);
        hb[h] = (uint8_t)cell_bits(in, PLAIN, g);
    }
    if (!grp.all(s, false)) return false;
    const double mb = proj ? s[1] / cnt : 0.0;

    // b' - A x of the own cell (row, i) from the global x
    auto true_residual = [&](int row, int i, unsigned b) -> double {
        const int g = (j0 + row) * nx + i;
        const double xc = __ldcg(in.x + g);
        double ax = 0.0;
        if (b & kE) ax += in.idx2 * (xc - xnb(g + 1));
        if (b & kW) ax += in.idx2 * (xc - xnb(g - 1));
        if (b & kN) ax += in.idy2 * (xc - xnb(g + nx));
        if (b & kS) ax += in.idy2 * (xc - xnb(g - nx));
        return -__ldg(in.rhs + g) - mb - ax;
    };
    // r = b' - A x in FP64, rounded to V, mean removed, its faces sent; then
    // slots 1: r.Mr, 4: sum r, 5: sum Mr, 6: r.r, 7: max |r|. With `fix` the
    // direction's M r_old becomes M r_new.
    auto residual_pass = [&](bool fix) -> bool {
        clear();
        each_cell([&](int row, int i, int o, unsigned b) {
            if (!(b & kFluid)) return;
            if (fix) dc0[o] = V(fma(-double(rs[o]), tab.inv[b], double(dc0[o])));
            const double rv = true_residual(row, i, b);
            s[0] += rv;
            rs[o] = V(rv);
        });
        if (fix)
            for (int t = tid; t < nh; t += T) {
                const int h = hslot(t);
                hd(h) = V(fma(-double(hr[h]), tab.inv[hb[h]], double(hd(h))));
            }
        if (!grp.all(s, false)) return false;
        const double mr = proj ? s[0] / cnt : 0.0;
        clear();
        each_cell([&](int row, int i, int o, unsigned b) {
            if (!(b & kFluid)) return;
            const V rv = V(double(rs[o]) - mr);
            rs[o] = rv;
            const double rd = double(rv), zd = rd * tab.inv[b];
            if (fix) put_d(row, i, o, V(fma(rd, tab.inv[b], double(dc0[o]))));
            s[1] = fma(rd, zd, s[1]);
            s[4] += rd;
            s[5] += zd;
            s[6] = fma(rd, rd, s[6]);
            s[7] = fmax(s[7], fabs(rd));
        });
        __syncthreads();
        send_faces(rs);
        if (!grp.all(s, true, true, face_bytes)) return false;
        peek_halo();
        each_halo([&](int h, V &d, V v) {
            hr[h] = v;
            if (fix) d = V(fma(double(v), tab.inv[hb[h]], double(d)));
        });
        return true;
    };

    int status = FLURSYS_LINEAR_MAX_ITERATIONS, error = 0;
    double initial_l2 = 0.0, initial = 0.0, threshold = 0.0, residual = 0.0, rz_old = 1.0;
    // A reduced norm (sum r.r or max |r|) greater than `above` does not meet the
    // threshold: no square root is taken on the way there.
    double above = 0.0, norm = 0.0;
    int since = 0;  // iterations since r was last replaced
    int it = 0, iterations = 0;
    const int max_it = (int)max(0LL, min(in.max_iters, 2147483000LL));
    bool fresh = true, replaced = false, last = false;

    for (;;) {
        if (fresh) {
            // the FP64 residual: of the initial guess, or (MIXED) in place of
            // the recurrence's
            if (!residual_pass(it > 0)) return false;
            fresh = false;
            since = 0;
            norm = linf ? s[7] : s[6];
            residual = linf ? norm : sqrt(norm);
            if (it == 0) {
                initial_l2 = sqrt(s[6]);
                initial = residual;
                threshold = linf ? in.tol : in.atol + in.rtol * initial;
                above = linf ? threshold : threshold * threshold * (1.0 + 1.0e-12);
            } else if (!isfinite(residual)) {
                error = FLURSYS_ERR_NON_FINITE;
                break;
            }
            if (linf ? residual < threshold : residual <= threshold) {
                status = FLURSYS_LINEAR_CONVERGED;
                break;
            }
            if (__syncthreads_or(tid < 32 && last)) break;
            if (it == 0) {  // d = M r less its mean
                const double shift = proj ? -s[5] / cnt : 0.0;
                each_cell([&](int row, int i, int o, unsigned b) {
                    if (b & kFluid) put_d(row, i, o, V(fma(double(rs[o]), tab.inv[b], shift)));
                });
                for (int t = tid; t < nh; t += T) {
                    const int h = hslot(t);
                    if (hb[h] & kFluid) hd(h) = V(fma(double(hr[h]), tab.inv[hb[h]], shift));
                }
            } else {
                replaced = true;
            }
        }
        __syncthreads();
        // ---- q = A d on the own cells, the sums ----
        clear();
        double rr = 0.0;
        for (Walk w = first(); w.row < nr;) {
            // U vectors per trip, their loads before the first use
            V dc[U][W], no[U][W], so[U][W], rv[U][W], ea[U], we[U];
            int row[U], v[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                row[u] = w.row;
                v[u] = w.strip * 32 + lane;
                if (v[u] >= nvec || w.row >= nr) v[u] = -1;
                const int o = v[u] >= 0 ? w.row * P + v[u] * W : 0;
                const V *p = dc0 + o;
                ldv(p, dc[u]);
                ldv(p + P, no[u]);
                ldv(p - P, so[u]);
                ldv(rs + o, rv[u]);
                ea[u] = p[W];
                we[u] = p[-1];
                next(w);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (v[u] < 0) continue;
                const int i = v[u] * W, o = row[u] * P + i;
                V qc[W];
                double md[W];
                if (PLAIN) {
#pragma unroll
                    for (int k = 0; k < W; ++k) {
                        const V e = k < W - 1 ? dc[u][k + 1] : ea[u], wv = k ? dc[u][k - 1] : we[u];
                        qc[k] = vfma(wx, (dc[u][k] - e) + (dc[u][k] - wv),
                                     wy * ((dc[u][k] - no[u][k]) + (dc[u][k] - so[u][k])));
                    }
                    const double mi = tab.inv[row_bits(row[u]) | kE | kW];
#pragma unroll
                    for (int k = 0; k < W; ++k) md[k] = mi;
                    if (v[u] == 0 || v[u] == nvec - 1) {
#pragma unroll
                        for (int k = 0; k < W; ++k) {
                            if (i + k == 0 || i + k == nx - 1) md[k] = tab.inv[row_bits(row[u]) | col_bits(i + k)];
                            if (i + k >= nx) qc[k] = dc[u][k] = V(0);  // behind the row
                        }
                    }
                } else {
#pragma unroll
                    for (int k = 0; k < W; ++k) {
                        const unsigned b = bs[o + k];  // 0 behind the row
                        const V c = dc[u][k], e = k < W - 1 ? dc[u][k + 1] : ea[u], wv = k ? dc[u][k - 1] : we[u];
                        const V de = (b & kE) ? c - e : V(0), dw = (b & kW) ? c - wv : V(0);
                        const V dn = (b & kN) ? c - no[u][k] : V(0), dso = (b & kS) ? c - so[u][k] : V(0);
                        qc[k] = vfma(wx, de + dw, wy * (dn + dso));
                        md[k] = tab.inv[b];
                    }
                }
                stv(qs + o, qc);
#pragma unroll
                for (int k = 0; k < W; ++k) {
                    const double dd = double(dc[u][k]), qd = double(qc[k]), rd = double(rv[u][k]);
                    const double zd = rd * md[k];
                    s[0] = fma(dd, qd, s[0]);
                    s[1] = fma(rd, zd, s[1]);
                    s[2] = fma(qd, zd, s[2]);
                    s[3] = fma(qd * md[k], qd, s[3]);
                    s[4] += rd;
                    s[5] += zd;
                    s[6] += dd;
                    rr = fma(rd, rd, rr);
                    if (linf) s[7] = fmax(s[7], fabs(rd));
                }
            }
        }
        if (!linf) s[7] = rr;
        __syncthreads();
        send_faces(qs);
        const bool ok = grp.lead(s, linf, true, face_bytes, peek_halo);
        if (tid < 32) {  // warp 0: the step's scalars, and the verdict on the current iterate
            const double den = s[0];
            const double mz = s[5] * inv_cnt, md = s[6] * inv_cnt, mr = s[4] * inv_cnt;
            const double rz = s[1] - mz * s[4];
            const double alpha = quotient(rz, den, fast_recip(den));
            const double beta = quotient(s[1] + alpha * (alpha * s[3] - 2.0 * s[2]), rz, fast_recip(rz));
            int cmd = kStep;
            if (!ok) {
                cmd = kFail;
            } else if (it > 0 && !replaced) {
                norm = s[7];
                last = fabs(rz_old) < 1.0e-30 || it >= max_it;
                if (!(norm > above && norm <= 1.7976931348623157e308) || last || (MIXED && since == in.replace_every)) {
                    if (!isfinite(norm)) {
                        error = FLURSYS_ERR_NON_FINITE;
                        cmd = kStop;
                    } else {
                        const bool conv = linf ? norm < threshold : sqrt(norm) <= threshold;
                        if (MIXED && (conv || since == in.replace_every)) {
                            cmd = kRefresh;
                        } else if (conv || last) {
                            if (conv) status = FLURSYS_LINEAR_CONVERGED;
                            cmd = kStop;
                        }
                    }
                }
            } else if (it >= max_it) {
                cmd = kStop;
            }
            if (cmd == kStep) {
                const bool sound = fabs(den) >= 1.0e-30 && fabs(den) <= 1.7976931348623157e308 && isfinite(alpha);
                if (MIXED && !sound && since > 0) {
                    cmd = kRefresh;  // the FP32 recurrence has run out before its replacement was due
                } else {
                    iterations = it + 1;
                    if (!sound) {
                        error = FLURSYS_ERR_BREAKDOWN;
                        cmd = kStop;
                    }
                    rz_old = rz;
                }
            }
            if (tid == 0) {
                sc.alpha = alpha;
                sc.md = md;
                sc.mr = mr;
                sc.beta = beta;
                sc.shift = -mz - beta * md;
                sc.cmd = cmd;
            }
        }
        __syncthreads();
        const int cmd = sc.cmd;
        if (cmd == kFail) return false;
        if (cmd == kStop) break;
        if (MIXED && cmd == kRefresh) {
            // x out, for the FP64 residual at the top of the loop
            each_x([&](int i, int row, int o, double &x) {
                if (fluid(o)) in.x[(j0 + row) * nx + i] = x;
            });
            if (!grp.barrier()) return false;
            fresh = true;
            continue;
        }
        replaced = false;
        const S alpha = S(sc.alpha), mr = S(sc.mr), beta = S(sc.beta), shift = S(sc.shift);
        const double ax = double(alpha), md = sc.md;
        if constexpr (XN > 0) {  // a vector of x at a time; values behind a row are never used
            Walk w = first();
            asm volatile("" : "+r"(w.row), "+r"(w.strip));
#pragma unroll
            for (int u = 0; u < XV; ++u) {
                const int v = w.strip * 32 + lane;
                if (w.row < nr && v < nvec) {
                    V dc[W];
                    ldv(dc0 + w.row * P + v * W, dc);
#pragma unroll
                    for (int k = 0; k < W; ++k) xr[u * W + k] = fma(ax, double(dc[k]) - md, xr[u * W + k]);
                }
                next(w);
            }
        }
        for (Walk w = first(); w.row < nr;) {
            V dc[U][W], qv[U][W], rv[U][W];
            int row[U], v[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                row[u] = w.row;
                v[u] = w.strip * 32 + lane;
                if (v[u] >= nvec || w.row >= nr) v[u] = -1;
                const int o = v[u] >= 0 ? w.row * P + v[u] * W : 0;
                ldv(dc0 + o, dc[u]);
                ldv(qs + o, qv[u]);
                ldv(rs + o, rv[u]);
                next(w);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (v[u] < 0) continue;
                const int i = v[u] * W, o = row[u] * P + i;
                V dn[W];
                S inv[W];
                unsigned b[W];
                const unsigned rb = row_bits(row[u]);
                const S ii = weight_of<S>(tab, rb | kE | kW);
#pragma unroll
                for (int k = 0; k < W; ++k) {
                    b[k] = PLAIN ? 31u : (unsigned)bs[o + k];
                    inv[k] = PLAIN ? ii : weight_of<S>(tab, b[k]);
                }
                const bool edge = v[u] == 0 || v[u] == nvec - 1;
                if (PLAIN && edge) {
#pragma unroll
                    for (int k = 0; k < W; ++k) {
                        b[k] = i + k < nx ? 31u : 0u;
                        if (i + k < nx) inv[k] = weight_of<S>(tab, rb | col_bits(i + k));
                    }
                }
                if (XN == 0) {
#pragma unroll
                    for (int k = 0; k < W; k += 2) {  // x of two cells per 16-byte access
                        double2 *xp = reinterpret_cast<double2 *>(xs + o + k);
                        double2 xv = *xp;
                        xv.x = fma(ax, double(dc[u][k]) - md, xv.x);
                        xv.y = fma(ax, double(dc[u][k + 1]) - md, xv.y);
                        *xp = xv;
                    }
                }
#pragma unroll
                for (int k = 0; k < W; ++k) {
                    const V rn = next_r(alpha, qv[u][k], rv[u][k], mr);
                    dn[k] = next_d(beta, dc[u][k], rn, inv[k], shift);
                    rv[u][k] = (b[k] & kFluid) ? rn : V(0);
                    if (!(b[k] & kFluid)) dn[k] = V(0);
                }
                stv(rs + o, rv[u]);
                V *p = dc0 + o;
                if (PLAIN) {
                    if (edge) {  // the ghost columns; behind the row first, as it may be in this vector
                        if (v[u] == 0) p[-1] = dn[0];
#pragma unroll
                        for (int k = 0; k < W; ++k)
                            if (i + k == nx - 1) {
                                if (k < W - 1) dn[k < W - 1 ? k + 1 : k] = dn[k];
                                else p[W] = dn[k];
                            }
                    }
                    if (row[u] == 0 && !has_lo) stv(p - P, dn);
                    if (row[u] == nr - 1 && !has_hi) stv(p + P, dn);
                }
                stv(p, dn);
            }
        }
        each_halo([&](int h, V &d, V qv) {
            const V hn = next_r(alpha, qv, hr[h], mr);
            hr[h] = hn;
            d = next_d(beta, d, hn, weight_of<S>(tab, hb[h]), shift);
        });
        ++it;
        ++since;
    }

    residual = linf ? norm : sqrt(norm);

    // ---- x' = x - mean x out, then the FP64 ||b' - A x||_2 ----
    clear();
    each_x([&](int, int, int o, double &x) {
        if (fluid(o)) s[0] += x;
    });
    if (!grp.all(s, false)) return false;
    const double mx = proj ? s[0] / cnt : 0.0;
    each_x([&](int i, int row, int o, double &x) {
        const int g = (j0 + row) * nx + i;
        in.x[g] = fluid(o) ? x - mx : (in.flags[g] & kCellOutlet) ? in.outlet_pressure : 0.0;
    });
    if (!grp.barrier()) return false;
    clear();
    each_cell([&](int row, int i, int, unsigned b) {
        if (!(b & kFluid)) return;
        const double t = true_residual(row, i, b);
        s[0] = fma(t, t, s[0]);
    });
    if (!grp.all(s, false)) return false;
    if (grp.rank == 0 && tid == 0) {
        PcgResultDev *res = in.result;
        res->error = error;
        res->status = status;
        res->iterations = iterations;
        res->initial = initial;
        res->residual = residual;
        res->true_l2 = sqrt(s[0]);
        res->initial_l2 = initial_l2;
    }
    return true;
}

template <typename V, int T, int XN, bool CLUSTER>
__device__ __forceinline__ bool res2d_run(const Pcg2dInstance &in, typename Res2dGroup<T, CLUSTER>::type &grp,
                                          char *dyn, Res2dTable &tab, Res2dScalars &sc) {
    if (in.count_fluid == (long long)in.nx * in.ny) return res2d_solve<V, T, XN, CLUSTER, true>(in, grp, dyn, tab, sc);
    return res2d_solve<V, T, XN, CLUSTER, false>(in, grp, dyn, tab, sc);
}

template <typename V, int T, int XN>
__global__ void __launch_bounds__(T, 1) pcg2d_res_cluster(const Pcg2dInstance *__restrict__ inst) {
    extern __shared__ __align__(16) char dyn[];
    __shared__ ClusterRedShared<T> red;
    __shared__ Res2dTable tab;
    __shared__ Res2dScalars sc;
    __shared__ Pcg2dInstance in;
    if (threadIdx.x == 0) in = inst[0];
    __syncthreads();
    ClusterGroup<T> grp{&red, (int)gridDim.x, (int)blockIdx.x, 0, 0u, 0u, 0u};
    grp.init();
    if (!res2d_run<V, T, XN, true>(in, grp, dyn, tab, sc) && threadIdx.x == 0)
        atomicOr(&in.result->device_error, (unsigned)kDevErrBarrierTimeout);
    grp.finish();
}

template <typename V, int T, int XN>
__global__ void __launch_bounds__(T, 1) pcg2d_res_grid(const Pcg2dInstance *__restrict__ inst, RedRecord *records,
                                                       RedRecord *faces, unsigned epoch) {
    extern __shared__ __align__(16) char dyn[];
    __shared__ GridRedShared<T> red;
    __shared__ Res2dTable tab;
    __shared__ Res2dScalars sc;
    __shared__ Pcg2dInstance in;
    if (threadIdx.x == 0) {
        in = inst[0];
        red.failed = 0;
    }
    __syncthreads();
    GridGroup<T> grp{&red, records, faces, (int)gridDim.x, (int)blockIdx.x, 2 * res2d_pitch<V>(in.nx), 0u, 0u, epoch, kRedSpinLimit, false};
    if (!res2d_run<V, T, XN, false>(in, grp, dyn, tab, sc) && threadIdx.x == 0)
        atomicOr(&in.result->device_error, (unsigned)kDevErrBarrierTimeout);
}

// Batched form: each cluster takes instances off the queue until it is empty.
template <typename V, int T, int XN>
__global__ void __launch_bounds__(T, 1) pcg2d_res_queue(const Pcg2dInstance *__restrict__ insts,
                                                        const int *__restrict__ order, int count, unsigned *next) {
    extern __shared__ __align__(16) char dyn[];
    __shared__ ClusterRedShared<T> red;
    __shared__ Res2dTable tab;
    __shared__ Res2dScalars sc;
    __shared__ Pcg2dInstance in;
    __shared__ int slot, gave_up;
    int nb, rank;
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(nb));
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    if (threadIdx.x == 0) gave_up = 0;
    ClusterGroup<T> grp{&red, nb, rank, 0, 0u, 0u, 0u};
    grp.init();
    for (;;) {
        if (rank == 0 && threadIdx.x == 0) {
            const int k = (int)atomicAdd(next, 1u);
            for (int b = 0; b < nb; ++b)
                asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cluster_addr(smem_addr(&slot), b)), "r"(k)
                             : "memory");
        }
        cluster_barrier();
        const int k = slot;
        if (k >= count || gave_up) break;  // the same in every block
        if (threadIdx.x == 0) in = insts[order[k]];
        __syncthreads();
        if (in.resident >= 0) {  // negative: not stepping
            if (rank == 0 && threadIdx.x == 0) in.result->device_error = 0u;
            if (!res2d_run<V, T, XN, true>(in, grp, dyn, tab, sc) && threadIdx.x == 0) {
                atomicOr(&in.result->device_error, (unsigned)kDevErrBarrierTimeout);
                for (int b = 0; b < nb; ++b)
                    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cluster_addr(smem_addr(&gave_up), b)), "r"(1)
                                 : "memory");
            }
        }
        cluster_barrier();  // every block is done with the instance and has read its slot
    }
    grp.finish();
}

// Kernel instantiations: 0: 256 threads, 1: 512 threads, both with x in shared
// memory.
template <bool CLUSTER>
const void *res_fn(int precision, int v) {
    if (CLUSTER) {
        if (precision == FLURSYS_PRECISION_MIXED)
            return v == 0 ? (const void *)pcg2d_res_cluster<float, 256, 0> : (const void *)pcg2d_res_cluster<float, 512, 0>;
        return v == 0 ? (const void *)pcg2d_res_cluster<double, 256, 0> : (const void *)pcg2d_res_cluster<double, 512, 0>;
    }
    if (precision == FLURSYS_PRECISION_MIXED)
        return v == 0 ? (const void *)pcg2d_res_grid<float, 256, 0> : (const void *)pcg2d_res_grid<float, 512, 0>;
    return v == 0 ? (const void *)pcg2d_res_grid<double, 256, 0> : (const void *)pcg2d_res_grid<double, 512, 0>;
}
int variant_threads(int v) { return v == 0 ? 256 : 512; }
// Most pieces (32 vectors of a row) per warp with 256 threads: a block
// reduction of 8 warps is the shorter one, more work per warp the longer. In
// MIXED, whose updates convert to FP64 and back, two pieces take longer than
// twice the warps' reduction (256 and 512 threads, us per iteration: 150 x 120 3.8
// and 3.5, 400 x 300 5.8 and 4.9, 509 x 331 5.9 and 5.1, 700 x 200 6.4 and 5.5).
int small_pieces(int precision) { return precision == FLURSYS_PRECISION_MIXED ? 1 : 2; }
// The queue's kernel keeps x in registers: pieces per warp of 512 threads.
constexpr int kQueuePieces = 8;
int pieces_of(int precision, int v, int rows, int nx) {
    const int warps = variant_threads(v) / 32, w = precision == FLURSYS_PRECISION_MIXED ? kVec<float> : kVec<double>;
    return (rows * (((nx + w - 1) / w + 31) / 32) + warps - 1) / warps;
}
constexpr int kMaxCluster = 16;
constexpr size_t kSmemMax = 222 * 1024;  // dynamic; the static part is below 5 KB

template <bool CLUSTER>
size_t smem_of(int precision, bool xreg, int rows, int nx, bool plain) {
    return precision == FLURSYS_PRECISION_MIXED ? res2d_smem<float, CLUSTER>(rows, nx, xreg, plain)
                                                : res2d_smem<double, CLUSTER>(rows, nx, xreg, plain);
}

// The limit belongs to the function, whose handles may plan and launch on
// several threads: it is set to the same ceiling each time and never lowered.
cudaError_t prepare_fn(const void *fn, bool cluster) {
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax);
    if (e == cudaSuccess && cluster) e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    return e;
}

cudaLaunchConfig_t cluster_config(int grid, int nb, int threads, size_t smem, cudaStream_t st,
                                  cudaLaunchAttribute *attr) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = nb;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}

}  // namespace

cudaError_t pcg2d_res_plan(Pcg2dResPlan &plan, int nx, int ny, bool plain, int precision, int device) {
    plan = Pcg2dResPlan{};
    const char *renv = std::getenv("FLURSYS_2D_RESIDENT");
    plan.precision = precision;
    if (renv && std::strcmp(renv, "0") == 0) return cudaSuccess;
    int sms = 0;
    cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    if (e != cudaSuccess) return e;
    const long long n = (long long)nx * ny;
    const char *cenv = std::getenv("FLURSYS_2D_CLUSTER");
    const bool may_cluster = !(cenv && std::strcmp(cenv, "0") == 0);
    // A cluster's round is shorter than the grid's (about 1300 against 3500
    // cycles), its 16 SMs work longer on a large grid: measured per iteration,
    // cluster and grid take 2.5 and 3.3 us on 128^2, 4.1 and 3.7 us on 180^2
    // in FP64, and 2.3 and 3.2 us on 128^2, 4.2 and 3.4 us on 256^2 in MIXED.
    long long cluster_cells = precision == FLURSYS_PRECISION_MIXED ? 40960 : 28672;
    if (const char *env = std::getenv("FLURSYS_2D_CLUSTER_CELLS")) cluster_cells = std::atoll(env);
    // nb blocks at most; blocks that would get no row are not launched
    auto choose = [&](bool cluster, int nb) {
        const int rows = (ny + nb - 1) / nb;
        plan.smem = cluster ? smem_of<true>(precision, false, rows, nx, plain) : smem_of<false>(precision, false, rows, nx, plain);
        if (plan.smem <= kSmemMax) {
            plan.cluster = cluster;
            plan.variant = pieces_of(precision, 0, rows, nx) <= small_pieces(precision) ? 0 : 1;
            plan.nblocks = (ny + rows - 1) / rows;
            return true;
        }
        return false;
    };
    // Rows of a few vectors leave most lanes of a warp idle, and many of them
    // make a block's passes long: a piece (32 vectors' room) per warp takes 0.85
    // us of an iteration in F64, 1.25 in MIXED. A cluster with more than six
    // leaves the solve to the grid (4 x 5000 F64 18.5 us, grid 10.4), and a grid
    // whose pieces cost more than the streaming kernel's iteration leaves it
    // to that (4 x 100000 MIXED 56.3 us, streaming 26.5; 6 x 100000 F64 41.3 and
    // 33.4; but 16 x 40000 MIXED 26.0 and 34.5).
    auto pieces = [&]() { return pieces_of(precision, plan.variant, (ny + plan.nblocks - 1) / plan.nblocks, nx); };
    if (may_cluster && n <= cluster_cells) {
        const int nb = (int)std::max(1LL, std::min<long long>(kMaxCluster, (n + 255) / 256));
        if (choose(true, nb) && pieces() <= 6) {
            const int nb = plan.nblocks;
            const void *fn = res_fn<true>(precision, plan.variant);
            cudaLaunchAttribute attr[1];
            const cudaLaunchConfig_t cfg = cluster_config(nb, nb, variant_threads(plan.variant), plan.smem, nullptr, attr);
            int active = 0;
            if (prepare_fn(fn, true) == cudaSuccess &&
                cudaOccupancyMaxActiveClusters(&active, fn, &cfg) == cudaSuccess && active >= 1) {
                plan.enabled = true;
                return cudaSuccess;
            }
            cudaGetLastError();
        }
    }
    const int nb = (int)std::max(1LL, std::min<long long>(std::min(sms, 160), (n + 511) / 512));
    const double piece_us = precision == FLURSYS_PRECISION_MIXED ? 1.25 : 0.85;
    if (!choose(false, nb) || 3.5 + piece_us * pieces() > 11.0 + 36.0e-6 * double(n)) {
        plan = Pcg2dResPlan{};
        return cudaSuccess;
    }
    // partial records, then the face records of each block's two halo rows;
    // cleared once (tags carry the launch's number)
    const size_t bytes = sizeof(RedRecord) * 2 * plan.nblocks * (kRedSlots + 2 * (size_t)std::max(res2d_pitch<float>(nx), res2d_pitch<double>(nx)));
    const void *fn = res_fn<false>(precision, plan.variant);
    int per_sm = 0;
    if (prepare_fn(fn, false) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, variant_threads(plan.variant), plan.smem) != cudaSuccess ||
        per_sm < 1) {
        cudaGetLastError();
        plan = Pcg2dResPlan{};
        return cudaSuccess;
    }
    if (cudaMalloc(&plan.records, bytes) != cudaSuccess || cudaMemset(plan.records, 0, bytes) != cudaSuccess ||
        cudaStreamSynchronize(nullptr) != cudaSuccess) {  // solves run on streams that do not wait for this one
        pcg2d_res_destroy(plan);  // no room: the streaming kernel serves the solve
        cudaGetLastError();
        return cudaSuccess;
    }
    plan.enabled = true;
    return cudaSuccess;
}

void pcg2d_res_destroy(Pcg2dResPlan &plan) {
    cudaFree(plan.records);
    plan = Pcg2dResPlan{};
}

cudaError_t pcg2d_res_launch(Pcg2dResPlan &plan, const Pcg2dInstance *inst_dev, PcgResultDev *result,
                             cudaStream_t stream) {
    cudaError_t e = cudaMemsetAsync(result, 0, sizeof(PcgResultDev), stream);
    if (e != cudaSuccess) return e;
    const int threads = variant_threads(plan.variant);
    if (plan.cluster) {
        const void *fn = res_fn<true>(plan.precision, plan.variant);
        cudaLaunchAttribute attr[1];
        const cudaLaunchConfig_t cfg = cluster_config(plan.nblocks, plan.nblocks, threads, plan.smem, stream, attr);
        void *params[] = {&inst_dev};
        return cudaLaunchKernelExC(&cfg, fn, params);
    }
    const void *fn = res_fn<false>(plan.precision, plan.variant);
    RedRecord *records = plan.records, *faces = plan.records + 2 * (size_t)plan.nblocks * kRedSlots;
    unsigned epoch = ++plan.epoch;
    void *params[] = {&inst_dev, &records, &faces, &epoch};
    return cudaLaunchCooperativeKernel(fn, dim3(plan.nblocks), dim3(threads), params, plan.smem, stream);
}

static const void *queue_fn(int precision) {
    return precision == FLURSYS_PRECISION_MIXED ? (const void *)pcg2d_res_queue<float, 512, 32>
                                                : (const void *)pcg2d_res_queue<double, 512, 16>;
}

bool pcg2d_queue_fits(int nx, int ny, bool plain, int precision, size_t *smem) {
    const char *renv = std::getenv("FLURSYS_2D_RESIDENT");
    if (renv && std::strcmp(renv, "0") == 0) return false;
    const int rows = (ny + kMaxCluster - 1) / kMaxCluster;
    if (pieces_of(precision, 1, rows, nx) > kQueuePieces) return false;
    *smem = smem_of<true>(precision, true, rows, nx, plain);
    return *smem <= kSmemMax;
}

int pcg2d_queue_pieces(int nx, int ny, int precision) {
    return pieces_of(precision, 1, (ny + kMaxCluster - 1) / kMaxCluster, nx);
}

cudaError_t pcg2d_queue_plan(Pcg2dQueuePlan &plan, int precision, size_t smem, int device) {
    plan = Pcg2dQueuePlan{};
    (void)device;
    const void *fn = queue_fn(precision);
    cudaLaunchAttribute attr[1];
    const cudaLaunchConfig_t cfg = cluster_config(kMaxCluster, kMaxCluster, 512, smem, nullptr, attr);
    int active = 0;
    if (prepare_fn(fn, true) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&active, fn, &cfg) != cudaSuccess || active < 1) {
        cudaGetLastError();
        return cudaSuccess;
    }
    plan.clusters = active;
    plan.nblocks = kMaxCluster;
    plan.smem = smem;
    return cudaSuccess;
}

cudaError_t pcg2d_queue_launch(const Pcg2dQueuePlan &plan, const Pcg2dInstance *insts, const int *order, int count,
                               unsigned *next, int precision, cudaStream_t stream) {
    const void *fn = queue_fn(precision);
    const int clusters = std::min(plan.clusters, count);
    cudaLaunchAttribute attr[1];
    const cudaLaunchConfig_t cfg = cluster_config(clusters * plan.nblocks, plan.nblocks, 512, plan.smem, stream, attr);
    void *params[] = {&insts, &order, &count, &next};
    return cudaLaunchKernelExC(&cfg, fn, params);
}

}  // namespace flursys
