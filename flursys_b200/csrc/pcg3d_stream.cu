// pcg3d_stream.cu — the 3D pressure PCG of grids too large for the chip: one
// pass over the vectors and one grid-wide sum per iteration, F64 and MIXED.
//
// The system (the pinned 7-point system of src/solver/incompressible_3d.rs:
// 293-332), the preconditioner, the stop rules and the precisions are those of
// the graph-driven PCG (pcg3d_seq.cu); the iteration is that of the
// chip-resident one (pcg3d_rows.cu). q = A d is never stored: given alpha and
// beta, a pass reads r, d and the increment of x, forms q = A d again, then
//     x += alpha d,  r -= alpha q,  d = M r + beta d
// and, on the new d, the products d.q, r.Mr, q.Mr, q.Mq and r.r that give the
// next alpha and beta. That moves six vectors per iteration where separate
// operand and update passes move ten, and needs no second launch.
//
// A block owns ty rows (of full length in x) by tz planes and marches them in
// z. r and d are read with the one and two rows and planes around the block
// that the new d and its q need; they alternate between two buffers, as a
// neighbour still reads the old values. Planes arrive by bulk copies into
// rings in shared memory (a plane's rows are contiguous, so a plane is one
// copy per vector), several planes ahead. A thread holds the same one or two
// 16-byte columns of vectors throughout: neighbours in z lie in its registers,
// in x in its warp, in y in shared memory. Passes alternate their direction in
// z, so that a pass begins with what the one before left in L2.
//
// What bounds it: the latency of one plane's chain beside DRAM. 256^3 in MIXED
// moves 403 MB per iteration, 62 us at the copy rate; a pass that only moves
// them takes 74 us with its sum, the solve 103 us (two launches per iteration:
// 139 to 147). On 160 x 140 x 120, which lies in L2, issue slots are 49% busy
// and shared memory 34%; the warps wait at the plane's barrier and on their
// loads. One vector column per thread fills the registers of four warps
// per scheduler; two spill some thirty. Per iteration, against the graph:
// 160^3 MIXED 50 -> 30 us, 300 x 200 x 150 MIXED 95 -> 84, 112^3 F64 43 -> 22,
// 200^3 F64 184 -> 124.
//
// MIXED applies alpha and beta rounded to FP32, the same to x and r (the graph
// rounds beta alone; see pcg3d_rows.cu): with alpha in FP64 160 x 140 x 120 took
// 29.1 us instead of 26.5, and the errors against 64 bits are half the graph's in
// the velocities, a twentieth in the pressure, either way.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>

#include "pcg3d_stream.cuh"
#include "tma.cuh"

namespace flursys {

namespace {

template <typename V>
constexpr int kW = 16 / (int)sizeof(V);

constexpr int kT = 512;          // threads per block
constexpr int kD = 4, kR = 3;    // planes in the rings of d, and of r and x
constexpr int kMaxColumns = 2;   // vector columns per thread
constexpr size_t kStreamSmemMax = 222 * 1024;  // dynamic; the static part is below 5 KB

__device__ __forceinline__ float rfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double rfma(double a, double b, double c) { return __fma_rn(a, b, c); }

template <typename V>
__device__ __forceinline__ void ldv(const V *p, V (&a)[kW<V>]) {
    const uint4 t = *reinterpret_cast<const uint4 *>(p);
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

template <typename V>
size_t stream_smem(int nx, int ty) {
    return sizeof(V) * (size_t)row_pitch<V>(nx) * (kD * (ty + 4) + kR * (ty + 2) + kR * ty + 2 * (ty + 2));
}

// Copies `bytes` (a multiple of 16, from a 16-byte boundary) into shared
// memory; completion counts on `bar`.
__device__ __forceinline__ void bulk_load(void *dst, const void *src, unsigned bytes, uint64_t *bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ unsigned long long now_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// What warp 0 hands the block after an iteration's reduction.
enum : int { kStep = 0, kStop = 1, kRefresh = 2, kFail = 3 };
template <typename V>
struct StreamShared {
    GridRedShared<kT> red;
    V inv[27];  // 1 / diagonal by missing-neighbour class 9 mx + 3 my + mz
    double invd[27];
    V alpha, beta;
    int cmd;
    uint64_t dbar[kD], rbar[kR];
    // the solve's scalars and times lie here so that a pass has the registers
    double initial_l2, initial, threshold, residual, rz_old, above, norm;
    unsigned long long t_op, t_red, t_rep, t_last;
};

// U: vector columns per thread. TAIL: a row ends inside a vector.
template <typename V, int U, bool TAIL>
__device__ __forceinline__ bool stream_solve(const StreamArgs &a, StreamShared<V> &sh, char *dyn) {
    constexpr bool MIXED = sizeof(V) == 4;
    constexpr int W = kW<V>, T = kT;
    const int nx = a.nx, ny = a.ny, nz = a.nz, tid = threadIdx.x;
    const int bj = blockIdx.x % a.by, bk = blockIdx.x / a.by;
    const int P = row_pitch<V>(nx), nvec = P / W;
    const size_t plane_n = (size_t)P * ny;
    // own rows and planes, those where the new d is formed, those of the old d
    const int j0 = bj * a.ty, j1 = min(ny, j0 + a.ty), k0 = bk * a.tz, k1 = min(nz, k0 + a.tz);
    const int je0 = max(0, j0 - 1), je1 = min(ny, j1 + 1), jd0 = max(0, j0 - 2), jd1 = min(ny, j1 + 2);
    const int ke0 = max(0, k0 - 1), ke1 = min(nz, k1 + 1), kd0 = max(0, k0 - 2), kd1 = min(nz, k1 + 2);
    const bool linf = a.stop_rule != FLURSYS_STOP_REL_L2;
    const bool pin_block = j0 + k0 == 0;
    const int dslot = P * (a.ty + 4), rslot = P * (a.ty + 2), xslot = P * a.ty;
    V *const ring_d = reinterpret_cast<V *>(dyn), *const ring_r = ring_d + kD * dslot;
    V *const ring_x = ring_r + kR * rslot, *const dn_buf = ring_x + kR * xslot;
    V *rv[2] = {static_cast<V *>(a.r[0]), static_cast<V *>(a.r[1])};
    V *dv[2] = {static_cast<V *>(a.d[0]), static_cast<V *>(a.d[1])};
    V *const xi = static_cast<V *>(a.xi);
    if (tid < 27) {
        const int mx = tid / 9, my = (tid / 3) % 3, mz = tid % 3;
        const double dg = (2 - mx) * a.ix2 + (2 - my) * a.iy2 + (2 - mz) * a.iz2;
        sh.inv[tid] = dg > 0.0 ? V(1.0 / dg) : V(0);
        sh.invd[tid] = double(sh.inv[tid]);
    }
    if (tid == 0) {
        sh.red.failed = 0;
        for (int i = 0; i < kD; ++i) mbar_init(&sh.dbar[i], 1);
        for (int i = 0; i < kR; ++i) mbar_init(&sh.rbar[i], 1);
    }
    __syncthreads();
    GridGroup<T> grp{&sh.red, a.records, nullptr, (int)gridDim.x, (int)blockIdx.x, 0, 0u, 0u, a.epoch,
                     kRedSpinLimit, a.fault != 0, true};
    const V wx = V(a.ix2), wy = V(a.iy2), wz = V(a.iz2);

    const int columns = (je1 - je0) * nvec;
    // ---- the thread's columns: 16 bytes of a row, all planes ----
    enum : int { kIn = 1, kOwn = 2, kFirst = 4, kLast = 8, kPin = 16, kSouth = 32, kNorth = 64 };  // kPin: row 0's first vector
    const int last_lane = TAIL ? (nx - 1) % W : W - 1;
    int off[U], info[U];  // offset of the vector from row je0; facts, class of its row << 8
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int c = tid + u * T, er = c / nvec, v = c - er * nvec, j = je0 + er;
        const bool in = j < je1;
        off[u] = in ? c * W : 0;
        info[u] = in ? kIn | (j >= j0 && j < j1 ? kOwn : 0) | (v == 0 ? kFirst : 0) | (v == nvec - 1 ? kLast : 0) |
                           (j + v == 0 ? kPin : 0) | (j == 0 ? kSouth : 0) | (j == ny - 1 ? kNorth : 0) |
                           (3 * ((j == 0) + (j == ny - 1)) << 8)
                     : kFirst | kLast | kSouth | kNorth;
    }
    const int d_shift = (je0 - jd0) * P, x_shift = (j0 - je0) * P;  // between the rings' rows
    unsigned gd = 0, gr = 0;  // planes taken from the rings by earlier passes
    auto d_ring = [&](int t) { return ring_d + (int)((gd + (unsigned)t) % kD) * dslot; };
    auto r_ring = [&](int s) { return ring_r + (int)((gr + (unsigned)s) % kR) * rslot; };
    auto x_ring = [&](int s) { return ring_x + (int)((gr + (unsigned)s) % kR) * xslot; };
    auto await = [&](uint64_t *bar, unsigned use) {  // use: how often the slot was filled before
        if (mbar_try_wait(bar, use & 1u)) return;
        const unsigned long long t0 = now_ns();
        while (!mbar_try_wait(bar, use & 1u))
            if (now_ns() - t0 > 200'000'000ull) {
                sh.red.failed = 1;
                break;
            }
    };
    auto await_d = [&](int t) { await(&sh.dbar[(gd + (unsigned)t) % kD], (gd + (unsigned)t) / kD); };

    double s[kRedSlots];
    auto clear = [&]() {
#pragma unroll
        for (int k = 0; k < kRedSlots; ++k) s[k] = 0.0;
    };
    // out = A c on the cells of a vector: acc holds wz (c - lo) for the z
    // neighbour already passed and becomes that of hi, the next one; y
    // neighbours no and so, x neighbours in the row at `p` (at a wall the cell
    // itself); 0 on the pinned cell and behind the row.
    auto apply = [&](int u, bool pin, const V *p, const V (&c)[W], const V (&no)[W], const V (&so)[W], V (&acc)[W],
                     const V (&hi)[W], V (&out)[W]) {
        const int f = info[u];
        const V we = p[(f & kFirst) ? 0 : -1], ea = p[(f & kLast) ? W - 1 : W];
        V dw = c[0] - we;  // differences: a constant gives exactly 0
#pragma unroll
        for (int i = 0; i < W; ++i) {
            const V de = c[i] - (i < W - 1 ? c[i < W - 1 ? i + 1 : i] : ea), dz = c[i] - hi[i];
            out[i] = rfma(wx, de + dw, rfma(wy, (c[i] - no[i]) + (c[i] - so[i]), rfma(wz, dz, acc[i])));
            acc[i] = -wz * dz;
            dw = -de;
        }
        if (TAIL && (f & kLast)) {
#pragma unroll
            for (int i = 1; i < W; ++i)
                if (i > last_lane) out[i] = V(0);
        }
        if (pin && (f & kPin)) out[0] = V(0);
    };
    // The weights of a vector's cells from `tab`, on a plane of class z.
    auto weights = [&](int u, int z, const auto *tab, auto &m) {
        const int f = info[u], cls = (f >> 8) + z;
        const auto mid = tab[cls];
#pragma unroll
        for (int i = 0; i < W; ++i) m[i] = mid;
        m[0] = tab[(f & kFirst) ? cls + 9 : cls];
        if constexpr (!TAIL) {
            m[W - 1] = tab[(f & kLast) ? cls + 9 : cls];
        } else if (f & kLast) {
#pragma unroll
            for (int i = 0; i < W; ++i)
                if (i == last_lane) m[i] = tab[cls + 9];
        }
    };
    int cur = 0;
    bool up = true;
    // One iteration: x += alpha d, r -= alpha A d, d = M r + beta d into the
    // other buffers; slots 0: d.q, 1: r.Mr, 2: q.Mr, 3: q.Mq, 4: r.r, 7: max
    // |r| of the new vectors.
    auto pass = [&](const V alpha, const V beta) {
        const V *const rs = rv[cur], *const dsrc = dv[cur];
        V *const rd_ = rv[cur ^ 1], *const dd_ = dv[cur ^ 1];
        const int ns = ke1 - ke0, nd = kd1 - kd0, lead_in = up ? ke0 - kd0 : kd1 - ke1;
        auto plane = [&](int q) { return up ? ke0 + q : ke1 - 1 - q; };
        int issued_d = 0, issued_r = 0;
        auto issue = [&](int to_d, int to_r) {  // one thread
            for (; issued_d < min(nd, to_d); ++issued_d) {
                const int k = up ? kd0 + issued_d : kd1 - 1 - issued_d;
                uint64_t *bar = &sh.dbar[(gd + (unsigned)issued_d) % kD];
                const unsigned bytes = (unsigned)(jd1 - jd0) * P * (unsigned)sizeof(V);
                mbar_expect_tx(bar, bytes);
                bulk_load(d_ring(issued_d), dsrc + (size_t)k * plane_n + (size_t)jd0 * P, bytes, bar);
            }
            for (; issued_r < min(ns, to_r); ++issued_r) {
                const int k = plane(issued_r);
                const bool own = k >= k0 && k < k1;
                uint64_t *bar = &sh.rbar[(gr + (unsigned)issued_r) % kR];
                const unsigned bytes = (unsigned)(je1 - je0) * P * (unsigned)sizeof(V);
                const unsigned xbytes = own ? (unsigned)(j1 - j0) * P * (unsigned)sizeof(V) : 0u;
                mbar_expect_tx(bar, bytes + xbytes);
                bulk_load(r_ring(issued_r), rs + (size_t)k * plane_n + (size_t)je0 * P, bytes, bar);
                if (own) bulk_load(x_ring(issued_r), xi + (size_t)k * plane_n + (size_t)j0 * P, xbytes, bar);
            }
        };
        if (tid == T - 32) {  // in the warp with the least work
            asm volatile("fence.proxy.async;" ::: "memory");  // the vectors were written by plain stores
            issue(kD, kR);
        }
        clear();
        V da[U][W], dc[U][W], ea_[U][W], ec[U][W], rn[U][W];  // old d with its sum so far, the new d likewise, the new r
        for (int t = 0; t <= lead_in; ++t) await_d(t);
#pragma unroll
        for (int u = 0; u < U; ++u) {
#pragma unroll
            for (int i = 0; i < W; ++i) ea_[u][i] = ec[u][i] = rn[u][i] = V(0);
            ldv(d_ring(lead_in) + d_shift + off[u], dc[u]);
            ldv(d_ring(0) + d_shift + off[u], da[u]);  // the same plane at a wall
#pragma unroll
            for (int i = 0; i < W; ++i) da[u][i] = wz * (dc[u][i] - da[u][i]);
        }
        // ring slots of plane q of r and x, and of the old d's current plane
        int slot_r = (int)(gr % kR), slot_d = (int)((gd + (unsigned)lead_in) % kD);
        unsigned use_r = gr / kR, use_d = (gd + (unsigned)lead_in) / kD;
        const ptrdiff_t step = up ? (ptrdiff_t)plane_n : -(ptrdiff_t)plane_n;
        ptrdiff_t gp = (ptrdiff_t)plane(0) * (ptrdiff_t)plane_n + (ptrdiff_t)je0 * P;
        V rmax = V(0);
        // the products of the new vectors of column u; hi: d on the next plane
        auto products = [&](int u, bool pin, int zc, const V *p, const V (&hi)[W]) {
            V no[W], so[W], qv[W];
            double m[W];
            ldv(p + ((info[u] & kNorth) ? 0 : P), no);
            ldv(p - ((info[u] & kSouth) ? 0 : P), so);
            apply(u, pin, p, ec[u], no, so, ea_[u], hi, qv);
            weights(u, zc, sh.invd, m);
#pragma unroll
            for (int i = 0; i < W; ++i) {  // behind the row r and q are 0
                const double qd = double(qv[i]), rd = double(rn[u][i]), zd = rd * m[i];
                s[0] = fma(double(ec[u][i]), qd, s[0]);
                s[1] = fma(rd, zd, s[1]);
                s[2] = fma(qd, zd, s[2]);
                s[3] = fma(qd * m[i], qd, s[3]);
                s[4] = fma(rd, rd, s[4]);
            }
            if (linf)
#pragma unroll
                for (int i = 0; i < W; ++i) rmax = max(rmax, rn[u][i] < V(0) ? -rn[u][i] : rn[u][i]);
        };
        auto wall = [&](int k) { return (k == 0) + (k == nz - 1); };
#pragma unroll(U == 1 ? 2 : 1)
        for (int q = 0; q < ns; ++q, gp += step) {
            const int t = q + lead_in, k = plane(q), ko = plane(q - 1);  // planes of the new d and of its products
            const bool next = t + 1 < nd, own_k = k >= k0 && k < k1, own_ko = q > 0 && ko >= k0 && ko < k1;
            const V *const sd = ring_d + slot_d * dslot + d_shift, *const sr = ring_r + slot_r * rslot;
            if (++slot_d == kD) {
                slot_d = 0;
                ++use_d;
            }
            if (next) await(&sh.dbar[slot_d], use_d);
            await(&sh.rbar[slot_r], use_r);
            const V *const sn = next ? ring_d + slot_d * dslot + d_shift : sd;
            const V *const sx = ring_x + slot_r * xslot - x_shift;
            if (++slot_r == kR) {
                slot_r = 0;
                ++use_r;
            }
            V *const en = dn_buf + (q & 1) * rslot;
            const V *const eo = dn_buf + ((q & 1) ^ 1) * rslot;
            const int zc = wall(k), zo = wall(ko);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (u > 0 && u * T + (tid & ~31) >= columns) continue;  // no lane of the warp has one
                const int o = off[u], f = info[u];
                V e[W], r[W];  // the new d and r of plane k
                {
                    V dx[W], no[W], so[W], qv[W], m[W];
                    ldv(sn + o, dx);
                    ldv(sd + o + ((f & kNorth) ? 0 : P), no);
                    ldv(sd + o - ((f & kSouth) ? 0 : P), so);
                    ldv(sr + o, r);
                    apply(u, k == 0, sd + o, dc[u], no, so, da[u], dx, qv);
                    weights(u, zc, sh.inv, m);
#pragma unroll
                    for (int i = 0; i < W; ++i) {
                        r[i] = rfma(-alpha, qv[i], r[i]);
                        e[i] = rfma(beta, dc[u][i], r[i] * m[i]);
                    }
                    if (TAIL && (f & kLast)) {  // the ghost behind the row
#pragma unroll
                        for (int i = 0; i < W - 1; ++i)
                            if (i >= last_lane) e[i + 1] = e[i];
                    }
                    if (f & kIn) stv(en + o, e);
                    if (own_k && (f & kOwn)) {
                        V x[W];
                        ldv(sx + o, x);
#pragma unroll
                        for (int i = 0; i < W; ++i) x[i] = rfma(alpha, dc[u][i], x[i]);
                        stv(xi + gp + o, x);
                        stv(rd_ + gp + o, r);
                        stv(dd_ + gp + o, e);
                    }
#pragma unroll
                    for (int i = 0; i < W; ++i) dc[u][i] = dx[i];
                }
                if (own_ko && (f & kOwn)) {
                    products(u, ko == 0, zo, eo + o, e);
                } else {  // before a wall the plane itself
#pragma unroll
                    for (int i = 0; i < W; ++i) ea_[u][i] = q == 0 ? V(0) : wz * (e[i] - ec[u][i]);
                }
#pragma unroll
                for (int i = 0; i < W; ++i) {
                    ec[u][i] = e[i];
                    rn[u][i] = r[i];
                }
            }
            __syncthreads();
            if (tid == T - 32) issue(t + 1 + kD, q + 1 + kR);
        }
        if (const int k = plane(ns - 1); k >= k0 && k < k1) {  // the last plane before a wall
            const V *const eo = dn_buf + ((ns - 1) & 1) * rslot;
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (info[u] & kOwn) {
                    V last_d[W];
#pragma unroll
                    for (int i = 0; i < W; ++i) last_d[i] = ec[u][i];
                    products(u, k == 0, wall(k), eo + off[u], last_d);
                }
        }
        s[7] = double(rmax);
        gd += (unsigned)nd;
        gr += (unsigned)ns;
        cur ^= 1;
        up = !up;
        asm volatile("fence.proxy.async;" ::: "memory");  // the next pass reads by bulk copies
    };
    // f(v, j, k, padded offset) over the block's own vectors
    auto each = [&](auto f) {
        const int nyl = j1 - j0, rows = nyl * (k1 - k0);
        int row = tid / nvec, v = tid - row * nvec;
        const int step_r = T / nvec, step_v = T - step_r * nvec;
        while (row < rows) {
            const int kk = row / nyl, j = j0 + row - kk * nyl, k = k0 + kk;
            f(v, j, k, (size_t)k * plane_n + (size_t)j * P + (size_t)v * W);
            v += step_v;
            row += step_r;
            if (v >= nvec) {
                v -= nvec;
                ++row;
            }
        }
    };
    // t[e] = b - A x of the vector's cells from the global x (b = -rhs; the
    // pinned cell 0 gives 0). x[0] is 0. Rows of even length are read two
    // values at a time.
    const bool pairs = nx % 2 == 0;
    auto true_residual = [&](int v, int j, int k, double (&t)[W]) {
        const size_t g = (size_t)(v * W) + (size_t)nx * (j + (size_t)ny * k), sy = nx, sz = (size_t)nx * ny;
        const int left = min(W, nx - v * W);
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
        const double we = v > 0 ? __ldcg(a.x + g - 1) : c[0];
        const double ea = v * W + W < nx ? __ldcg(a.x + g + W) : 0.0;
#pragma unroll
        for (int e = 0; e < W; ++e) {
            t[e] = 0.0;
            if (e >= left) continue;
            const double xw = e ? c[e - 1] : we;
            const double xe = v * W + e == nx - 1 ? c[e] : e < W - 1 ? c[e < W - 1 ? e + 1 : e] : ea;
            const double ax = a.ix2 * ((c[e] - xe) + (c[e] - xw)) + a.iy2 * ((c[e] - no[e]) + (c[e] - so[e])) +
                              a.iz2 * ((c[e] - fo[e]) + (c[e] - ba[e]));
            if (g + e != 0) t[e] = -__ldg(a.rhs + g + e) - ax;
        }
    };
    // r = b - A x in FP64, rounded to V; d becomes d - M r_old, to which the
    // next pass (alpha 0, beta 1) adds M r. `first`: there is no d yet. Slots
    // 4: r.r, 7: max |r|.
    auto residual_pass = [&](bool first) -> bool {
        clear();
        each([&](int v, int j, int k, size_t g) {
            V r[W], d[W], n[W];
            double t[W];
            true_residual(v, j, k, t);
#pragma unroll
            for (int e = 0; e < W; ++e) r[e] = d[e] = V(0);
            if (!first) {
                ldv(rv[cur] + g, r);
                ldv(dv[cur] + g, d);
            }
            const int c0 = 3 * ((j == 0) + (j == ny - 1)) + (k == 0) + (k == nz - 1);
#pragma unroll
            for (int e = 0; e < W; ++e) {
                const int i = v * W + e;
                n[e] = V(0);
                if (i >= nx) continue;
                n[e] = V(t[e]);
                d[e] = rfma(-r[e], sh.inv[c0 + 9 * ((i == 0) + (i == nx - 1))], d[e]);
                const double rd = double(n[e]);
                s[4] = fma(rd, rd, s[4]);
                s[7] = fmax(s[7], fabs(rd));
            }
            stv(rv[cur] + g, n);
            stv(dv[cur] + g, d);
        });
        asm volatile("fence.proxy.async;" ::: "memory");
        return grp.all(s, true, true);
    };
    // The increment folded into x.
    auto put_x = [&]() {
        each([&](int v, int j, int k, size_t g) {
            V x[W], zero[W];
            ldv(xi + g, x);
            const size_t c = (size_t)(v * W) + (size_t)nx * (j + (size_t)ny * k);
#pragma unroll
            for (int e = 0; e < W; ++e) {
                zero[e] = V(0);
                if (v * W + e >= nx) continue;
                if (c + e == 0) a.x[0] = 0.0;
                else a.x[c + e] += double(x[e]);
            }
            stv(xi + g, zero);
        });
        asm volatile("fence.proxy.async;" ::: "memory");
    };

    if (pin_block && tid == 0) a.x[0] = 0.0;
    each([&](int, int, int, size_t g) {
        V zero[W];
#pragma unroll
        for (int e = 0; e < W; ++e) zero[e] = V(0);
        stv(xi + g, zero);
    });
    if (!grp.barrier()) return false;

    int status = FLURSYS_LINEAR_MAX_ITERATIONS, error = 0;
    double &initial_l2 = sh.initial_l2, &initial = sh.initial, &threshold = sh.threshold, &residual = sh.residual;
    double &rz_old = sh.rz_old, &norm = sh.norm;
    double &above = sh.above;  // a reduced norm greater than it does not meet the threshold
    int since = 0, it = 0, iterations = 0;
    const int max_it = (int)max(0LL, min(a.max_iters, 2147483000LL));
    bool fresh = true, replaced = false, last = false;
    const bool clock = tid == 0;
    if (clock) {
        initial_l2 = initial = threshold = residual = above = norm = 0.0;
        rz_old = 1.0;
        sh.t_op = sh.t_red = sh.t_rep = 0;
        sh.t_last = now_ns();
    }
    auto lap = [&](unsigned long long &acc) {
        if (clock) {
            const unsigned long long t = now_ns();
            acc += t - sh.t_last;
            sh.t_last = t;
        }
    };

    V alpha = V(0), beta = V(0);
    for (;;) {
        if (fresh) {
            if (!residual_pass(it == 0)) return false;
            fresh = false;
            since = 0;
            if (clock) {
                norm = linf ? s[7] : s[4];
                residual = linf ? norm : sqrt(norm);
                if (it == 0) {
                    initial_l2 = sqrt(s[4]);
                    initial = residual;
                    threshold = linf ? a.tol : a.atol + a.rtol * initial;
                    above = linf ? threshold : threshold * threshold * (1.0 + 1.0e-12);
                }
            }
            __syncthreads();
            if (it > 0 && !isfinite(residual)) {
                error = FLURSYS_ERR_NON_FINITE;
                break;
            }
            if (linf ? residual < threshold : residual <= threshold) {
                status = FLURSYS_LINEAR_CONVERGED;
                break;
            }
            if (__syncthreads_or(tid < 32 && last)) break;
            alpha = V(0);
            beta = it == 0 ? V(0) : V(1);
            replaced = it > 0;
            lap(sh.t_rep);
        }
        pass(alpha, beta);
        lap(sh.t_op);
        const bool ok = grp.lead(s, linf, true, 0, [] {});
        if (tid < 32) {  // warp 0: the step's scalars, and the verdict on the current iterate
            const double den = s[0], rz = s[1], alpha = quotient(rz, den, fast_recip(den));
            const double beta = quotient(rz + alpha * (alpha * s[3] - 2.0 * s[2]), rz, fast_recip(rz));
            int cmd = kStep;
            if (!ok) {
                cmd = kFail;
            } else if (it > 0 && !replaced) {
                norm = linf ? s[7] : s[4];
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
                sh.alpha = V(alpha);
                sh.beta = V(beta);
                sh.cmd = cmd;
            }
        }
        __syncthreads();
        const int cmd = sh.cmd;
        if (cmd == kFail) return false;
        if (cmd == kStop) break;
        lap(sh.t_red);
        if (MIXED && cmd == kRefresh) {
            put_x();
            if (!grp.barrier()) return false;
            fresh = true;
            continue;
        }
        replaced = false;
        alpha = sh.alpha;
        beta = sh.beta;
        ++it;
        ++since;
    }
    if (clock) residual = linf ? norm : sqrt(norm);
    // ---- x out, then the FP64 ||b - A x||_2 ----
    put_x();
    if (!grp.barrier()) return false;
    clear();
    each([&](int v, int j, int k, size_t) {
        double t[W];
        true_residual(v, j, k, t);
#pragma unroll
        for (int e = 0; e < W; ++e) s[0] = fma(t[e], t[e], s[0]);
    });
    if (!grp.all(s, false)) return false;
    lap(sh.t_rep);
    if (blockIdx.x == 0 && tid == 0) {
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
        st->phase_ns[1] = sh.t_op;
        st->phase_ns[2] = sh.t_red;
        st->phase_ns[3] = sh.t_rep;
    }
    if (clock) atomicMax(&a.st->phase_ns[5], sh.t_op + sh.t_rep);
    return true;
}


template <typename V, int U, bool TAIL>
__global__ void __launch_bounds__(kT, 1) pcg3d_stream_kernel(const __grid_constant__ StreamArgs a) {
    extern __shared__ __align__(16) char dyn[];
    __shared__ StreamShared<V> sh;
    if (!stream_solve<V, U, TAIL>(a, sh, dyn) && threadIdx.x == 0)
        atomicOr(&a.st->device_error, (unsigned)kDevErrBarrierTimeout);
}

// The split into at most `most` blocks with the least work in a block; false
// when a block of four rows does not fit.
template <typename V>
bool choose_stream(Pcg3dStreamPlan &plan, int most) {
    StreamArgs &a = plan.args;
    const int nvec = row_pitch<V>(a.nx) / kW<V>;
    double best = 0.0;
    int columns = 0;
    for (int by = 1; by <= std::min(a.ny, most); ++by) {
        const int ty = (a.ny + by - 1) / by, rby = (a.ny + ty - 1) / ty, bz = std::min(a.nz, most / rby);
        if (bz < 1 || ty < std::min(4, a.ny)) continue;
        const int tz = (a.nz + bz - 1) / bz, u = ((ty + 2) * nvec + kT - 1) / kT;
        if (u > kMaxColumns || stream_smem<V>(a.nx, ty) > kStreamSmemMax) continue;
        // planes with their start-up, rows with their halo; two columns per
        // thread spill (173 against 133 cycles per column)
        const double cost = (tz + 5.0) * (ty + 3.0) * (u == 1 ? 1.0 : 1.3);
        if (columns == 0 || cost < best) {
            best = cost;
            columns = u;
            a.by = rby;
            a.bz = (a.nz + tz - 1) / tz;
            a.ty = ty;
            a.tz = tz;
        }
    }
    if (columns == 0) return false;
    plan.blocks = a.by * a.bz;
    plan.smem = stream_smem<V>(a.nx, a.ty);
    plan.kernel = a.nx % kW<V> ? (columns == 1 ? (const void *)pcg3d_stream_kernel<V, 1, true> : (const void *)pcg3d_stream_kernel<V, 2, true>)
                               : (columns == 1 ? (const void *)pcg3d_stream_kernel<V, 1, false> : (const void *)pcg3d_stream_kernel<V, 2, false>);
    return true;
}

}  // namespace

bool pcg3d_stream_plan(Pcg3dStreamPlan &plan, const Pcg3dArgs &args, int precision, int device) {
    plan = Pcg3dStreamPlan{};
    const char *env = std::getenv("FLURSYS_PCG_RESIDENT");
    if (env && (std::strcmp(env, "0") == 0 || std::strcmp(env, "2") == 0 || std::strcmp(env, "tiles") == 0)) return false;
    int sms = 0, per_sm = 0;
    if (args.nx < 2 || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) return false;
    StreamArgs &a = plan.args;
    a.nx = args.nx; a.ny = args.ny; a.nz = args.nz;
    a.ix2 = args.ix2; a.iy2 = args.iy2; a.iz2 = args.iz2;
    a.x = args.x;
    a.rhs = args.rhs;
    a.stop_rule = args.stop_rule;
    a.tol = args.tol; a.atol = args.atol; a.rtol = args.rtol;
    a.max_iters = args.max_iters;
    a.replace_every = args.replace_every > 0 ? args.replace_every : 50;
    const bool mixed = precision == FLURSYS_PRECISION_MIXED;
    const int most = std::min(sms, 160);
    // The limit keeps what this form and the graph return within 1e-9 of each
    // other (2-norm of the pressure), so that one may stand for the other in
    // a running program; it is not a limit of speed. A MIXED solve by the graph
    // to 1e-12 ends with an error of the pressure's constant part (the pin's
    // tiny eigenvalue) that grows with the grid, and the two forms differ by
    // it: 256^3 1e-10 to 2.4e-9, 144^3 at most 8e-10 (velocities 1e-13).
    if (mixed && !(env && std::strcmp(env, "stream") == 0) && (long long)args.nx * args.ny * args.nz > 3'200'000LL) return false;
    if (!(mixed ? choose_stream<float>(plan, most) : choose_stream<double>(plan, most))) return false;
    const size_t bytes = (mixed ? 4 * (size_t)row_pitch<float>(a.nx) : 8 * (size_t)row_pitch<double>(a.nx)) * a.ny * a.nz;
    const size_t rec = sizeof(RedRecord) * 2 * plan.blocks * kRedSlots;
    // (the limit is the function's, which handles on several threads share:
    // always the same ceiling, never lowered)
    if (cudaFuncSetAttribute(plan.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kStreamSmemMax) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, plan.kernel, kT, plan.smem) != cudaSuccess || per_sm < 1 ||
        cudaMalloc(&plan.records, rec) != cudaSuccess || cudaMemset(plan.records, 0, rec) != cudaSuccess ||
        cudaStreamSynchronize(nullptr) != cudaSuccess ||  // solves run on streams that do not wait for this one
        cudaMalloc(&plan.vectors, 5 * bytes) != cudaSuccess) {
        pcg3d_stream_destroy(plan);
        cudaGetLastError();
        return false;
    }
    char *v = static_cast<char *>(plan.vectors);
    a.r[0] = v;
    a.r[1] = v + bytes;
    a.d[0] = v + 2 * bytes;
    a.d[1] = v + 3 * bytes;
    a.xi = v + 4 * bytes;
    a.records = plan.records;
    return true;
}

cudaError_t pcg3d_stream_launch(Pcg3dStreamPlan &plan, CgSeqState *state, cudaStream_t stream) {
    StreamArgs a = plan.args;
    a.st = state;
    a.epoch = ++plan.epoch;
    a.fault = take_injected_barrier_fault();
    cudaError_t e = cudaMemsetAsync(state, 0, sizeof(CgSeqState), stream);
    void *params[] = {&a};
    return e == cudaSuccess
               ? cudaLaunchCooperativeKernel(plan.kernel, dim3(plan.blocks), dim3(kT), params, plan.smem, stream)
               : e;
}

void pcg3d_stream_destroy(Pcg3dStreamPlan &plan) {
    cudaFree(plan.records);
    cudaFree(plan.vectors);
    plan = Pcg3dStreamPlan{};
}

}  // namespace flursys
