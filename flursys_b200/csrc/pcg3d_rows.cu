// pcg3d_rows.cu — the 3D pressure PCG with its state held on the chip for the
// whole solve and one group-wide synchronisation per iteration, F64 and MIXED.
//
// The system (the pinned 7-point system of src/solver/incompressible_3d.rs:
// 293-332), the preconditioner, the stop rules and the precisions are those of
// the graph-driven PCG (pcg3d_seq.cu). The iteration is that of the 2D solver
// (pcg2d_res.cu): q = A d; one reduction of d.q, r.Mr, q.Mr, q.Mq and r.r (or
// max |r|) that also delivers the faces of q; stop test where r.r is summed;
// alpha; x, r; beta from r.Mr - 2 alpha q.Mr + alpha^2 q.Mq; d = M r + beta d
// on the block's rows and, from its own copy of the halo's r, on its halo.
// MIXED replaces r by the FP64 b - A x every replace_every iterations and
// before convergence is accepted, after folding the FP32 increment into the
// FP64 pressure; d then exchanges M r_old for M r_new.
//
// A block owns ty x tz rows of x (whole rows: no halo in x, 16-byte vectors
// throughout). d lies in shared memory with a halo row on each side and ghost
// cells that hold the wall cell's own value, so that the operator has no
// boundary case; q, r and x beside it, or, where that does not fit (128^3 in
// MIXED), r and x in registers. Cells per block and faces decide the split:
// see pcg3d_rows_plan().
//
// What bounds it: latency. On small grids the round (partials and faces through
// L2 or, in a cluster, through distributed shared memory); on large ones four
// warps per scheduler that wait on shared memory, L2, their own chains and the
// block's barriers: at 128^3 in MIXED issue slots are 42% busy, shared memory
// 35%, the conversions' unit 11%, FP64 6%. DRAM sees the pressure only at the
// residual replacements. Per iteration, against the graph-driven form:
// 75 x 62 x 51 F64 22.5 -> 6.1 us, 64^3 MIXED 20 -> 4.6, 100^3 F64 39 -> 13.6,
// 128^3 MIXED 30 -> 16.3 (the tile-resident form of pcg3d_res.cu: 20).
//
// MIXED applies alpha and beta rounded to FP32, the same to x and r, as the tile
// form does (the graph rounds beta alone). With alpha in FP64 128^3 took 15%
// longer at the same errors against 64 bits: on average 6% of the graph's and the
// tiles' in the pressure and 75% in the velocities (their operator is a sum that
// does not annihilate a constant exactly).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <type_traits>

#include "pcg3d_rows.cuh"

namespace flursys {

namespace {

template <typename V>
constexpr int kW = 16 / (int)sizeof(V);

__device__ __forceinline__ float rfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double rfma(double a, double b, double c) { return __fma_rn(a, b, c); }

template <typename V>
__device__ __forceinline__ void ldv(const V *p, V (&a)[kW<V>]) {
    const uint4 t = *reinterpret_cast<const uint4 *>(p);
    memcpy(a, &t, 16);
}
template <typename V>
__device__ __forceinline__ void ldv_cg(const V *p, V (&a)[kW<V>]) {
    const uint4 t = __ldcg(reinterpret_cast<const uint4 *>(p));
    memcpy(a, &t, 16);
}
template <typename V>
__device__ __forceinline__ void stv(V *p, const V (&a)[kW<V>]) {
    uint4 t;
    memcpy(&t, a, 16);
    *reinterpret_cast<uint4 *>(p) = t;
}

template <typename V>
__host__ __device__ __forceinline__ int row_pitch(int nx) { return (nx + kW<V> - 1) / kW<V> * kW<V>; }
// Face values of a block: its two y faces, then its two z faces.
template <typename V>
__host__ __device__ __forceinline__ int face_values(int nx, int ty, int tz) { return 2 * (ty + tz) * row_pitch<V>(nx); }

template <typename V>
size_t rows_smem(int nx, int ty, int tz, bool regs, bool cluster) {
    const size_t p = row_pitch<V>(nx), d = (size_t)(ty + 2) * (tz + 2) * (p + kW<V>) + 2 * kW<V>;
    const size_t own = (size_t)ty * tz * p, f = face_values<V>(nx, ty, tz);
    return sizeof(V) * (d + (regs ? 1 : 3) * own + f + (cluster ? 2 * f : 0)) + 8 * (size_t)ty * tz + 16 * 2 * (size_t)(ty + tz);
}

// Per-row facts, formed once: a row's boundary class and, packed beside it,
// whether it is the block's first or last in y and z and where it lies.
enum : int { kYFirst = 1 << 8, kYLast = 1 << 9, kZFirst = 1 << 10, kZLast = 1 << 11, kFaceRow = 15 << 8 };
__device__ __forceinline__ int row_jj(int info) { return (info >> 12) & 1023; }
__device__ __forceinline__ int row_kk(int info) { return (info >> 22) & 1023; }

template <int T, bool CLUSTER>
struct RowsGroup {
    using type = GridGroup<T>;
};
template <int T>
struct RowsGroup<T, true> {
    using type = ClusterGroup<T>;
};

// What warp 0 hands the block after an iteration's reduction.
enum : int { kStep = 0, kStop = 1, kRefresh = 2, kFail = 3 };
template <typename V>
struct RowsScalars {
    V alpha, beta;
    int cmd;
};
template <typename V>
struct RowsTable {  // 1 / diagonal by missing-neighbour class 9 mx + 3 my + mz
    V v[27];
    double d[27];
};

__device__ __forceinline__ unsigned long long now_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

template <typename V, int T, int XV, bool CLUSTER>
__device__ __forceinline__ bool rows_solve(const RowsArgs &a, typename RowsGroup<T, CLUSTER>::type &grp, char *dyn,
                                           RowsTable<V> &tab, RowsScalars<V> &sc) {
    constexpr bool MIXED = sizeof(V) == 4;
    constexpr int W = kW<V>;
    const int nx = a.nx, ny = a.ny, nz = a.nz, tid = threadIdx.x;
    const int bj = grp.rank % a.by, bk = grp.rank / a.by;
    const int j0 = bj * a.ty, k0 = bk * a.tz, nyl = min(a.ty, ny - j0), nzl = min(a.tz, nz - k0);
    const int P = row_pitch<V>(nx), PD = P + W, nvec = P / W, PZ = (a.ty + 2) * PD;
    const bool ylo = j0 > 0, yhi = j0 + nyl < ny, zlo = k0 > 0, zhi = k0 + nzl < nz;
    const bool linf = a.stop_rule != FLURSYS_STOP_REL_L2;
    const int own = a.ty * a.tz * P;
    const int slots = 2 * (a.ty + a.tz) * P;  // face values
    V *ds = reinterpret_cast<V *>(dyn);
    V *qs = ds + (a.ty + 2) * (a.tz + 2) * PD + 2 * W;
    V *rs = qs + own;                   // XV == 0
    V *xs = rs + own;                   // XV == 0: x (F64) or its increment (MIXED)
    V *hr = XV ? qs + own : xs + own;   // r of the halo, as the faces are laid out
    V *hq = hr + slots;                 // CLUSTER: faces received, by exchange parity
    int4 *halot = reinterpret_cast<int4 *>(hq + (CLUSTER ? 2 * slots : 0));  // halo rows: slot, d offset, class
    int2 *rowt = reinterpret_cast<int2 *>(halot + 2 * (a.ty + a.tz));        // own rows: d offset, facts
    V *const dc0 = ds + PZ + PD + W;    // d of cell (0, 0, 0): row (jj, kk) at kk PZ + jj PD
    V *gf = static_cast<V *>(a.faces);
    if constexpr (CLUSTER) {
        grp.face_slots = slots;
        grp.faces = smem_addr(hq);
    }
    const V wx = V(a.ix2), wy = V(a.iy2), wz = V(a.iz2);
    if (tid < 27) {
        const int mx = tid / 9, my = (tid / 3) % 3, mz = tid % 3;
        const double dg = (2 - mx) * a.ix2 + (2 - my) * a.iy2 + (2 - mz) * a.iz2;
        tab.v[tid] = dg > 0.0 ? V(1.0 / dg) : V(0);
        tab.d[tid] = double(tab.v[tid]);
    }
    for (int t = tid; t < (a.ty + 2) * (a.tz + 2) * PD + 2 * W; t += T) ds[t] = V(0);
    for (int t = tid; t < own; t += T) {
        qs[t] = V(0);
        if (XV == 0) rs[t] = xs[t] = V(0);
    }
    for (int t = tid; t < slots; t += T) hr[t] = V(0);
    __syncthreads();

    // A thread's walk over the block's vectors, rows flattened.
    const int rows = nyl * nzl, step_r = T / nvec, step_v = T - step_r * nvec;
    const int r0 = tid / nvec, v0 = tid - r0 * nvec;
    struct Walk {
        int r, v;
    };
    auto first = [&]() { return Walk{r0, v0}; };
    auto next = [&](Walk &w) {
        w.v += step_v;
        w.r += step_r;
        if (w.v >= nvec) {
            w.v -= nvec;
            ++w.r;
        }
    };
    auto row_class = [&](int j, int k) -> int { return 3 * ((j == 0) + (j == ny - 1)) + (k == 0) + (k == nz - 1); };
    auto col_class = [&](int i) -> int { return 9 * ((i == 0) + (i == nx - 1)); };
    for (int r = tid; r < rows; r += T) {
        const int kk = r / nyl, jj = r - kk * nyl;
        rowt[r] = make_int2(kk * PZ + jj * PD, row_class(j0 + jj, k0 + kk) | (jj == 0 ? kYFirst : 0) |
                                                   (jj == nyl - 1 ? kYLast : 0) | (kk == 0 ? kZFirst : 0) |
                                                   (kk == nzl - 1 ? kZLast : 0) | jj << 12 | kk << 22);
    }
    const bool tail = nx % W != 0, pin_block = j0 + k0 == 0;
    auto cell = [&](const Walk &w, int info) -> size_t {  // global index of the vector's first cell
        return (size_t)(w.v * W) + (size_t)nx * ((j0 + row_jj(info)) + (size_t)ny * (k0 + row_kk(info)));
    };
    // m[e] = tab[class of the vector's cells]; rows of a single cell and
    // partial vectors take the general way
    auto weights = [&](const auto *t, int rc, int v, auto &m) {
        const auto in = t[rc];
#pragma unroll
        for (int e = 0; e < W; ++e) m[e] = in;
        if (!tail) {
            const auto edge = t[rc + 9];
            m[0] = v == 0 ? edge : in;
            m[W - 1] = v == nvec - 1 ? edge : m[W - 1];
        } else if (v == 0 || v == nvec - 1) {
#pragma unroll
            for (int e = 0; e < W; ++e)
                if (v * W + e < nx) m[e] = t[rc + col_class(v * W + e)];
        }
    };
    V rr_[XV ? XV : 1][W], xr_[XV ? XV : 1][W];  // XV > 0: r and x of the thread's vectors
    // f(walk, r, x) over the thread's vectors, in the same order in every
    // pass; r and x are written back where WR / WX ask for it
    auto each = [&](auto wr, auto wx_, auto f) {
        Walk w = first();
        if constexpr (XV > 0) {
            asm volatile("" : "+r"(w.r), "+r"(w.v));  // form the offsets here
#pragma unroll
            for (int u = 0; u < XV; ++u) {
                if (w.r < rows) f(w, rr_[u], xr_[u]);
                next(w);
            }
        } else {
            for (; w.r < rows; next(w)) {
                const int o = w.r * P + w.v * W;
                V r[W], x[W];
                ldv(rs + o, r);
                if constexpr (decltype(wx_)::value) ldv(xs + o, x);
                f(w, r, x);
                if constexpr (decltype(wr)::value) stv(rs + o, r);
                if constexpr (decltype(wx_)::value) stv(xs + o, x);
            }
        }
    };
    using Yes = std::true_type;
    using No = std::false_type;
#pragma unroll
    for (int u = 0; u < (XV ? XV : 1); ++u)
#pragma unroll
        for (int k = 0; k < W; ++k) rr_[u][k] = xr_[u][k] = V(0);

    // Writes a vector of d (values behind the row are overwritten) with the
    // ghosts that it gives at the domain's walls.
    auto put_d = [&](int2 ri, int v, V (&dn)[W]) {
        V *p = dc0 + ri.x + v * W;
        if (v == 0) p[-1] = dn[0];
        if (v == nvec - 1) {
            if (!tail) {
                p[W] = dn[W - 1];
            } else {
#pragma unroll
                for (int k = 0; k < W - 1; ++k)
                    if (v * W + k == nx - 1) dn[k + 1] = dn[k];
            }
        }
        stv(p, dn);
        if (ri.y & kFaceRow) {
            if ((ri.y & kYFirst) && !ylo) stv(p - PD, dn);
            if ((ri.y & kYLast) && !yhi) stv(p + PD, dn);
            if ((ri.y & kZFirst) && !zlo) stv(p - PZ, dn);
            if ((ri.y & kZLast) && !zhi) stv(p + PZ, dn);
        }
    };
    // Face slot bases: y faces hold the plane index kk, z faces jj.
    const int fy = a.tz * P, fz = a.ty * P, base[4] = {0, fy, 2 * fy, 2 * fy + fz};
    auto send_vec = [&](int to, int slot, const V (&val)[W]) {
        if constexpr (CLUSTER) {
#pragma unroll
            for (int k = 0; k < W; ++k) grp.send(to, slot + k, val[k]);
        } else {
            stv(gf + ((size_t)(grp.fround & 1u) * grp.nb + to) * slots + slot, val);
        }
    };
    // Sends a boundary row's vector to the blocks whose halo holds it.
    auto send = [&](int info, int v, const V (&val)[W]) {
        if (!(info & kFaceRow)) return;
        const int sy = row_kk(info) * P + v * W, sz = row_jj(info) * P + v * W;
        if ((info & kYFirst) && ylo) send_vec(grp.rank - 1, base[1] + sy, val);
        if ((info & kYLast) && yhi) send_vec(grp.rank + 1, base[0] + sy, val);
        if ((info & kZFirst) && zlo) send_vec(grp.rank - a.by, base[3] + sz, val);
        if ((info & kZLast) && zhi) send_vec(grp.rank + a.by, base[2] + sz, val);
    };
    // Halo rows in the order y-, y+, z-, z+; row h's side, index on it.
    const int n0 = ylo ? nzl : 0, n1 = n0 + (yhi ? nzl : 0), n2 = n1 + (zlo ? nyl : 0), nhr = n2 + (zhi ? nyl : 0);
    const unsigned face_bytes = (unsigned)(nhr * P * (int)sizeof(V));
    for (int h = tid; h < nhr; h += T) {
        const int side = h < n0 ? 0 : h < n1 ? 1 : h < n2 ? 2 : 3;
        const int idx = h - (side == 0 ? 0 : side == 1 ? n0 : side == 2 ? n1 : n2);
        const int jj = side == 0 ? -1 : side == 1 ? nyl : idx, kk = side < 2 ? idx : side == 2 ? -1 : nzl;
        halot[h] = make_int4(base[side] + idx * P, kk * PZ + jj * PD, row_class(j0 + jj, k0 + kk), 0);
    }
    __syncthreads();
    // f(r, d, 1/diagonal, received) over the halo's vectors
    constexpr int HP = 3;  // halo vectors per thread that are looked at early
    V hv[CLUSTER ? 1 : HP][W];
    auto received = [&](int slot, V (&val)[W]) {
        if constexpr (CLUSTER) ldv(hq + ((grp.fround - 1u) & 1u) * (unsigned)slots + slot, val);
        else ldv_cg(gf + ((size_t)((grp.fround - 1u) & 1u) * grp.nb + grp.rank) * slots + slot, val);
    };
    auto peek_halo = [&]() {
        if constexpr (!CLUSTER) {
            Walk w = first();
#pragma unroll
            for (int u = 0; u < HP; ++u) {
                if (w.r < nhr) received(halot[w.r].x + w.v * W, hv[u]);
                next(w);
            }
        }
    };
    auto each_halo = [&](bool recv, auto f) {
        auto one = [&](const Walk &w, bool early, const V (&ev)[W]) {
            const int4 hi = halot[w.r];
            const int slot = hi.x + w.v * W;
            V r[W], d[W], inv[W], val[W];
            V *p = dc0 + hi.y + w.v * W;
            ldv(hr + slot, r);
            ldv(p, d);
            if (early) {
#pragma unroll
                for (int k = 0; k < W; ++k) val[k] = ev[k];
            } else if (recv) {
                received(slot, val);
            }
            weights(tab.v, hi.z, w.v, inv);
            f(r, d, inv, val);
            stv(hr + slot, r);
            stv(p, d);
        };
        Walk w = first();
        if constexpr (!CLUSTER) {
#pragma unroll
            for (int u = 0; u < HP; ++u) {
                if (w.r < nhr) one(w, recv, hv[u]);
                next(w);
            }
        }
        for (; w.r < nhr; next(w)) one(w, false, hv[0]);
    };

    double s[kRedSlots];
    auto clear = [&]() {
#pragma unroll
        for (int k = 0; k < kRedSlots; ++k) s[k] = 0.0;
    };
    // t[e] = b - A x of the vector's cells from the global x (b = -rhs; the
    // pinned cell 0 gives 0). x[0] is 0. Rows of even length are read two
    // values at a time.
    const bool pairs = nx % 2 == 0;
    auto true_residual = [&](const Walk &w, int info, double (&t)[W]) {
        const int j = j0 + row_jj(info), k = k0 + row_kk(info);
        const size_t g = cell(w, info), sy = nx, sz = (size_t)nx * ny;
        const int left = min(W, nx - w.v * W);
        auto row = [&](size_t at, bool there, const double (&other)[W], double (&o)[W]) {
#pragma unroll
            for (int e = 0; e < W; ++e) o[e] = other[e];
            if (!there) return;
            if (pairs) {
#pragma unroll
                for (int e = 0; e < W; e += 2)
                    if (e < left) {
                        const double2 v = __ldcg(reinterpret_cast<const double2 *>(a.x + at + e));
                        o[e] = v.x;
                        o[e + 1] = v.y;
                    }
            } else {
#pragma unroll
                for (int e = 0; e < W; ++e)
                    if (e < left) o[e] = __ldcg(a.x + at + e);
            }
        };
        double zero[W], c[W], no[W], so[W], fo[W], ba[W];
#pragma unroll
        for (int e = 0; e < W; ++e) zero[e] = 0.0;
        row(g, true, zero, c);
        row(g + sy, j + 1 < ny, c, no);
        row(g - sy, j > 0, c, so);
        row(g + sz, k + 1 < nz, c, fo);
        row(g - sz, k > 0, c, ba);
        const double we = w.v > 0 ? __ldcg(a.x + g - 1) : c[0];
        const double ea = w.v * W + W < nx ? __ldcg(a.x + g + W) : 0.0;
#pragma unroll
        for (int e = 0; e < W; ++e) {
            t[e] = 0.0;
            if (e >= left) continue;
            const double xw = e ? c[e - 1] : we;
            const double xe = w.v * W + e == nx - 1 ? c[e] : e < W - 1 ? c[e < W - 1 ? e + 1 : e] : ea;
            const double ax = a.ix2 * ((c[e] - xe) + (c[e] - xw)) + a.iy2 * ((c[e] - no[e]) + (c[e] - so[e])) +
                              a.iz2 * ((c[e] - fo[e]) + (c[e] - ba[e]));
            if (g + e != 0) t[e] = -__ldg(a.rhs + g + e) - ax;
        }
    };
    // r = b - A x in FP64, rounded to V, its faces sent; slots 1: r.Mr, 4: r.r,
    // 7: max |r|. With `fix` the direction's M r_old becomes M r_new.
    auto residual_pass = [&](bool fix) -> bool {
        clear();
        each(Yes{}, No{}, [&](const Walk &w, V (&r)[W], V (&)[W]) {
            const int2 ri = rowt[w.r];
            const int rc = ri.y & 15;
            V dn[W];
            double t[W];
            ldv(dc0 + ri.x + w.v * W, dn);
            true_residual(w, ri.y, t);
#pragma unroll
            for (int e = 0; e < W; ++e) {
                const int i = w.v * W + e;
                if (i >= nx) continue;
                const int c = rc + col_class(i);
                const V rv = V(t[e]);
                if (fix) dn[e] = rfma(rv, tab.v[c], rfma(-r[e], tab.v[c], dn[e]));
                r[e] = rv;
                const double rd = double(rv);
                s[1] = fma(rd * tab.d[c], rd, s[1]);
                s[4] = fma(rd, rd, s[4]);
                s[7] = fmax(s[7], fabs(rd));
            }
            if (fix) put_d(ri, w.v, dn);
            send(ri.y, w.v, r);
        });
        if (!grp.all(s, true, true, face_bytes)) return false;
        peek_halo();
        each_halo(true, [&](V (&r)[W], V (&d)[W], const V (&inv)[W], const V (&val)[W]) {
#pragma unroll
            for (int e = 0; e < W; ++e) {
                if (fix) d[e] = rfma(val[e], inv[e], rfma(-r[e], inv[e], d[e]));
                r[e] = val[e];
            }
        });
        return true;
    };
    // x out: the increment folded into the pressure (MIXED) or x itself (F64).
    auto put_x = [&]() {
        each(No{}, Yes{}, [&](const Walk &w, V (&)[W], V (&x)[W]) {
            const size_t g = cell(w, rowt[w.r].y);
#pragma unroll
            for (int e = 0; e < W; ++e) {
                if (w.v * W + e >= nx) continue;
                if (g + e == 0) a.x[0] = 0.0;
                else if (MIXED) a.x[g + e] += double(x[e]);
                else a.x[g + e] = double(x[e]);
                if (MIXED) x[e] = V(0);
            }
        });
    };

    if (pin_block && tid == 0) a.x[0] = 0.0;
    if (!grp.barrier()) return false;
    if (!MIXED)
        each(No{}, Yes{}, [&](const Walk &w, V (&)[W], V (&x)[W]) {
            const size_t g = cell(w, rowt[w.r].y);
#pragma unroll
            for (int e = 0; e < W; ++e) x[e] = w.v * W + e < nx ? V(__ldcg(a.x + g + e)) : V(0);
        });

    int status = FLURSYS_LINEAR_MAX_ITERATIONS, error = 0;
    double initial_l2 = 0.0, initial = 0.0, threshold = 0.0, residual = 0.0, rz_old = 1.0;
    double above = 0.0, norm = 0.0;  // a reduced norm greater than `above` does not meet the threshold
    int since = 0, it = 0, iterations = 0;
    const int max_it = (int)max(0LL, min(a.max_iters, 2147483000LL));
    bool fresh = true, replaced = false, last = false;
    unsigned long long t_dir = 0, t_op = 0, t_red = 0, t_rep = 0, t_a = 0, t_b = 0;
    const bool clock = tid == 0;
    if (clock) t_a = now_ns();
    auto lap = [&](unsigned long long &acc) {
        if (clock) {
            t_b = now_ns();
            acc += t_b - t_a;
            t_a = t_b;
        }
    };

    for (;;) {
        if (fresh) {
            if (!residual_pass(it > 0)) return false;
            fresh = false;
            since = 0;
            norm = linf ? s[7] : s[4];
            residual = linf ? norm : sqrt(norm);
            if (it == 0) {
                initial_l2 = sqrt(s[4]);
                initial = residual;
                threshold = linf ? a.tol : a.atol + a.rtol * initial;
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
            if (it == 0) {  // d = M r
                each(No{}, No{}, [&](const Walk &w, V (&r)[W], V (&)[W]) {
                    const int2 ri = rowt[w.r];
                    V dn[W];
#pragma unroll
                    for (int e = 0; e < W; ++e)
                        dn[e] = w.v * W + e < nx ? r[e] * tab.v[(ri.y & 15) + col_class(w.v * W + e)] : V(0);
                    put_d(ri, w.v, dn);
                });
                each_halo(false, [&](V (&r)[W], V (&d)[W], const V (&inv)[W], const V (&)[W]) {
#pragma unroll
                    for (int e = 0; e < W; ++e) d[e] = r[e] * inv[e];
                });
            } else {
                replaced = true;
            }
            lap(t_rep);
        }
        __syncthreads();
        // ---- q = A d on the own rows, its faces out, the sums ----
        clear();
        double rr = 0.0;
        each(No{}, No{}, [&](const Walk &w, V (&r)[W], V (&)[W]) {
            const int2 ri = rowt[w.r];
            const V *p = dc0 + ri.x + w.v * W;
            V dc[W], no[W], so[W], fo[W], ba[W], qc[W];
            ldv(p, dc);
            ldv(p + PD, no);
            ldv(p - PD, so);
            ldv(p + PZ, fo);
            ldv(p - PZ, ba);
            const V ea = p[W], we = p[-1];
            double md[W];
            weights(tab.d, ri.y & 15, w.v, md);
#pragma unroll
            for (int e = 0; e < W; ++e) {
                const V xe = e < W - 1 ? dc[e + 1] : ea, xw = e ? dc[e - 1] : we;
                qc[e] = rfma(wx, (dc[e] - xe) + (dc[e] - xw),
                             rfma(wy, (dc[e] - no[e]) + (dc[e] - so[e]), wz * ((dc[e] - fo[e]) + (dc[e] - ba[e]))));
            }
            if (tail && w.v == nvec - 1) {
#pragma unroll
                for (int e = 0; e < W; ++e)
                    if (w.v * W + e >= nx) qc[e] = dc[e] = V(0);  // behind the row
            }
            if (pin_block && w.r == 0 && w.v == 0) qc[0] = V(0);  // the pinned cell
            stv(qs + w.r * P + w.v * W, qc);
            send(ri.y, w.v, qc);
#pragma unroll
            for (int e = 0; e < W; ++e) {
                const double dd = double(dc[e]), qd = double(qc[e]), rd = double(r[e]), zd = rd * md[e];
                s[0] = fma(dd, qd, s[0]);
                s[1] = fma(rd, zd, s[1]);
                s[2] = fma(qd, zd, s[2]);
                s[3] = fma(qd * md[e], qd, s[3]);
                rr = fma(rd, rd, rr);
                if (linf) s[7] = fmax(s[7], fabs(rd));
            }
        });
        if (!linf) s[7] = rr;
        lap(t_op);
        const bool ok = grp.lead(s, linf, true, face_bytes, [] {});
        if (tid < 32) {  // warp 0: the step's scalars, and the verdict on the current iterate
            const double den = s[0], rz = s[1], alpha = quotient(rz, den, fast_recip(den));
            const double beta = quotient(rz + alpha * (alpha * s[3] - 2.0 * s[2]), rz, fast_recip(rz));
            int cmd = kStep;
            if (!ok) {
                cmd = kFail;
            } else if (it > 0 && !replaced) {
                norm = s[7];
                last = fabs(rz_old) < 1.0e-30 || it >= max_it;
                if (!(norm > above && norm <= 1.7976931348623157e308) || last || (MIXED && since == a.replace_every)) {
                    if (!isfinite(norm)) {
                        error = FLURSYS_ERR_NON_FINITE;
                        cmd = kStop;
                    } else {
                        const bool conv = linf ? norm < threshold : sqrt(norm) <= threshold;
                        if (MIXED && (conv || since == a.replace_every)) {
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
                sc.alpha = V(alpha);
                sc.beta = V(beta);
                sc.cmd = cmd;
            }
        }
        __syncthreads();
        const int cmd = sc.cmd;
        if (cmd == kFail) return false;
        if (cmd == kStop) break;
        lap(t_red);
        if (MIXED && cmd == kRefresh) {
            put_x();
            if (!grp.barrier()) return false;
            fresh = true;
            continue;
        }
        replaced = false;
        peek_halo();
        // ---- x += alpha d, r -= alpha q, d = M r + beta d ----
        const V av = sc.alpha, bv = sc.beta;
        each(Yes{}, Yes{}, [&](const Walk &w, V (&r)[W], V (&x)[W]) {
            V dc[W], qv[W], inv[W];
            const int2 ri = rowt[w.r];
            ldv(dc0 + ri.x + w.v * W, dc);
            ldv(qs + w.r * P + w.v * W, qv);
            weights(tab.v, ri.y & 15, w.v, inv);
#pragma unroll
            for (int e = 0; e < W; ++e) {
                x[e] = rfma(av, dc[e], x[e]);  // behind the row: never used
                r[e] = rfma(-av, qv[e], r[e]);  // q is 0 behind the row
                dc[e] = rfma(bv, dc[e], r[e] * inv[e]);
            }
            put_d(ri, w.v, dc);
        });
        each_halo(true, [&](V (&r)[W], V (&d)[W], const V (&inv)[W], const V (&qv)[W]) {
#pragma unroll
            for (int e = 0; e < W; ++e) {
                r[e] = rfma(-av, qv[e], r[e]);
                d[e] = rfma(bv, d[e], r[e] * inv[e]);
            }
        });
        lap(t_dir);
        ++it;
        ++since;
    }
    residual = linf ? norm : sqrt(norm);
    // ---- x out, then the FP64 ||b - A x||_2 ----
    put_x();
    if (!grp.barrier()) return false;
    clear();
    each(No{}, No{}, [&](const Walk &w, V (&)[W], V (&)[W]) {
        double t[W];
        true_residual(w, rowt[w.r].y, t);
#pragma unroll
        for (int e = 0; e < W; ++e) s[0] = fma(t[e], t[e], s[0]);
    });
    if (!grp.all(s, false)) return false;
    lap(t_rep);
    if (grp.rank == 0 && tid == 0) {
        CgSeqState *st = a.st;
        st->error = error;
        st->status = status;
        st->iterations = iterations;
        st->initial = initial;
        st->initial_l2 = initial_l2;
        st->residual = residual;
        st->threshold = threshold;
        st->true_l2 = sqrt(s[0]);
        st->done = 1;
        st->phase_ns[0] = t_dir;
        st->phase_ns[1] = t_op;
        st->phase_ns[2] = t_red;
        st->phase_ns[3] = t_rep;
    }
    if (clock) atomicMax(&a.st->phase_ns[5], t_dir + t_op + t_rep);
    return true;
}

template <typename V, int T, int XV>
__global__ void __launch_bounds__(T, 1) pcg3d_rows_grid(const __grid_constant__ RowsArgs a) {
    extern __shared__ __align__(16) char dyn[];
    __shared__ GridRedShared<T> red;
    __shared__ RowsTable<V> tab;
    __shared__ RowsScalars<V> sc;
    if (threadIdx.x == 0) red.failed = 0;
    __syncthreads();
    GridGroup<T> grp{&red, a.records, nullptr, (int)gridDim.x, (int)blockIdx.x, 0, 0u, 0u, a.epoch,
                     kRedSpinLimit, a.fault != 0, true};
    if (!rows_solve<V, T, XV, false>(a, grp, dyn, tab, sc) && threadIdx.x == 0)
        atomicOr(&a.st->device_error, (unsigned)kDevErrBarrierTimeout);
}

template <typename V, int T>
__global__ void __launch_bounds__(T, 1) pcg3d_rows_cluster(const __grid_constant__ RowsArgs a) {
    extern __shared__ __align__(16) char dyn[];
    __shared__ ClusterRedShared<T> red;
    __shared__ RowsTable<V> tab;
    __shared__ RowsScalars<V> sc;
    ClusterGroup<T> grp{&red, (int)gridDim.x, (int)blockIdx.x, 0, 0u, 0u, 0u, a.fault != 0};
    grp.init();
    if (!rows_solve<V, T, 0, true>(a, grp, dyn, tab, sc) && threadIdx.x == 0)
        atomicOr(&a.st->device_error, (unsigned)kDevErrBarrierTimeout);
    grp.finish();
}

constexpr size_t kRowsSmemMax = 222 * 1024;  // dynamic; the static part is below 5 KB
constexpr int kRowsXV = 8;                   // vectors per thread of 512 with r and x in registers

// The split of the rows into at most `most` blocks with the least work in the
// largest block (its vectors, and its halo's at about a third of their cost);
// false when none fits.
template <typename V>
bool split_rows(int nx, int ny, int nz, int most, bool regs, bool cluster, RowsArgs &a, size_t &smem) {
    double best = 0.0;
    bool found = false;
    for (int by = 1; by <= std::min(ny, most); ++by) {
        const int ty = (ny + by - 1) / by, rby = (ny + ty - 1) / ty;
        const int bz = std::min(nz, most / rby);
        if (bz < 1) continue;
        const int tz = (nz + bz - 1) / bz, rbz = (nz + tz - 1) / tz;
        const size_t need = rows_smem<V>(nx, ty, tz, regs, cluster);
        const long long vecs = (long long)ty * tz * (row_pitch<V>(nx) / kW<V>);
        if (need > kRowsSmemMax || ty > 1023 || tz > 511 || (regs && vecs > 512LL * kRowsXV)) continue;
        const double cost = double(ty) * tz + 0.35 * 2.0 * (ty + tz);
        if (!found || cost < best) {
            found = true;
            best = cost;
            a.by = rby;
            a.bz = rbz;
            a.ty = ty;
            a.tz = tz;
            smem = need;
        }
    }
    return found;
}

template <typename V>
bool choose_rows(Pcg3dRowsPlan &plan, int sms, bool may_cluster, bool may_grid) {
    RowsArgs &a = plan.args;
    const long long n = (long long)a.nx * a.ny * a.nz;
    auto set = [&](bool cluster, int threads, const void *fn) {
        plan.cluster = cluster;
        plan.threads = threads;
        plan.kernel = fn;
        plan.blocks = a.by * a.bz;
        return true;
    };
    // A cluster's round is the shorter one; its 16 SMs work longer on a large
    // grid (us per iteration, cluster | grid; F64: 24^3 2.5 | 5.2, 32^3 3.4 |
    // 4.1, 40 x 40 x 32 4.6 | 4.4; MIXED: 32^3 2.9 | 4.7, 40^3 4.1 | 5.1,
    // 44^3 5.0 | 4.1).
    long long cluster_cells = sizeof(V) == 4 ? 65536 : 40960;
    if (const char *env = std::getenv("FLURSYS_3D_CLUSTER_CELLS")) cluster_cells = std::atoll(env);
    if (may_cluster && n <= cluster_cells && split_rows<V>(a.nx, a.ny, a.nz, 16, false, true, a, plan.smem))
        return set(true, 512, (const void *)pcg3d_rows_cluster<V, 512>);
    if (!may_grid) return false;
    // at least 256 vectors per block: below that a smaller group's round is
    // shorter than what its longer passes cost
    const long long vecs = (long long)a.ny * a.nz * (row_pitch<V>(a.nx) / kW<V>);
    const int most = (int)std::max(1LL, std::min<long long>(std::min(sms, 160), (vecs + 255) / 256));
    if (split_rows<V>(a.nx, a.ny, a.nz, most, false, false, a, plan.smem)) {
        const long long per = (long long)a.ty * a.tz * (row_pitch<V>(a.nx) / kW<V>);
        return per <= 512 ? set(false, 256, (const void *)pcg3d_rows_grid<V, 256, 0>)
                          : set(false, 512, (const void *)pcg3d_rows_grid<V, 512, 0>);
    }
    if (split_rows<V>(a.nx, a.ny, a.nz, std::min(sms, 160), true, false, a, plan.smem))
        return set(false, 512, (const void *)pcg3d_rows_grid<V, 512, kRowsXV>);
    return false;
}

}  // namespace

bool pcg3d_rows_plan(Pcg3dRowsPlan &plan, const Pcg3dArgs &args, int precision, int device) {
    plan = Pcg3dRowsPlan{};
    // FLURSYS_PCG_RESIDENT: 0, 2, "tiles" and "stream" ask for other forms,
    // "grid" for no cluster
    const char *env = std::getenv("FLURSYS_PCG_RESIDENT");
    for (const char *other : {"0", "2", "tiles", "stream"})
        if (env && std::strcmp(env, other) == 0) return false;
    if (args.nz < 2) return false;
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) return false;
    RowsArgs &a = plan.args;
    a.nx = args.nx; a.ny = args.ny; a.nz = args.nz;
    a.ix2 = args.ix2; a.iy2 = args.iy2; a.iz2 = args.iz2;
    a.x = args.x;
    a.rhs = args.rhs;
    a.stop_rule = args.stop_rule;
    a.tol = args.tol; a.atol = args.atol; a.rtol = args.rtol;
    a.max_iters = args.max_iters;
    a.replace_every = args.replace_every > 0 ? args.replace_every : 50;
    const bool mixed = precision == FLURSYS_PRECISION_MIXED;
    bool may_cluster = !(env && std::strcmp(env, "grid") == 0);
    for (;;) {
        if (!(mixed ? choose_rows<float>(plan, sms, may_cluster, true) : choose_rows<double>(plan, sms, may_cluster, true)))
            return false;
        // the limit is the function's, which handles on several threads share:
        // always the same ceiling, never lowered
        bool fits = cudaFuncSetAttribute(plan.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRowsSmemMax) == cudaSuccess;
        if (fits && plan.cluster) {
            fits = cudaFuncSetAttribute(plan.kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = plan.blocks;
            attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
            cudaLaunchConfig_t cfg{};
            cfg.gridDim = dim3(plan.blocks);
            cfg.blockDim = dim3(plan.threads);
            cfg.dynamicSmemBytes = plan.smem;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            int active = 0;
            fits = fits && cudaOccupancyMaxActiveClusters(&active, plan.kernel, &cfg) == cudaSuccess && active >= 1;
        } else if (fits) {
            int per_sm = 0;
            fits = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, plan.kernel, plan.threads, plan.smem) == cudaSuccess &&
                   per_sm >= 1;
        }
        if (fits) break;
        cudaGetLastError();
        if (!plan.cluster) return false;
        may_cluster = false;
    }
    if (!plan.cluster) {
        const size_t rec = sizeof(RedRecord) * 2 * plan.blocks * kRedSlots;
        const size_t slots = mixed ? face_values<float>(a.nx, a.ty, a.tz) : face_values<double>(a.nx, a.ty, a.tz);
        // (the clearing ends here: solves run on streams that do not wait for this one)
        if (cudaMalloc(&plan.records, rec) != cudaSuccess || cudaMemset(plan.records, 0, rec) != cudaSuccess ||
            cudaStreamSynchronize(nullptr) != cudaSuccess ||
            cudaMalloc(&plan.faces, (mixed ? 4 : 8) * 2 * plan.blocks * slots) != cudaSuccess) {
            pcg3d_rows_destroy(plan);
            return false;
        }
    }
    a.records = plan.records;
    a.faces = plan.faces;
    return true;
}

cudaError_t pcg3d_rows_launch(Pcg3dRowsPlan &plan, CgSeqState *state, cudaStream_t stream) {
    RowsArgs a = plan.args;
    a.st = state;
    a.epoch = ++plan.epoch;
    a.fault = take_injected_barrier_fault();
    cudaError_t e = cudaMemsetAsync(state, 0, sizeof(CgSeqState), stream);
    void *params[] = {&a};
    cudaLaunchAttribute attr[1];
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(plan.blocks);
    cfg.blockDim = dim3(plan.threads);
    cfg.dynamicSmemBytes = plan.smem;
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (plan.cluster) {
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = plan.blocks;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    } else {
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
    }
    return e == cudaSuccess ? cudaLaunchKernelExC(&cfg, plan.kernel, params) : e;
}

void pcg3d_rows_destroy(Pcg3dRowsPlan &plan) {
    cudaFree(plan.records);
    cudaFree(plan.faces);
    plan = Pcg3dRowsPlan{};
}

}  // namespace flursys
