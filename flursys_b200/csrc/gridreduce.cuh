// gridreduce.cuh — one-hop sums over the blocks of a co-resident grid or of a
// thread-block cluster, for solvers that keep their state on the chip and
// synchronise once per iteration.
//
// Up to eight values per thread are summed at a time (slot 7 may be a maximum
// instead). Inside a warp the eight values and the 32 lanes are reduced
// together: each halving step also halves the values a lane carries, so 9
// double shuffles do the work of 40. Every block ends with the same bits,
// because every block adds the same partials in the same order.
//
// Data that travels with a round (the faces of a stencil operand) is sent to
// its reader and carries its own proof of arrival, so no fence orders it
// against the partials:
//
// Grid form: partials and faces are 16-byte {value, round} records, written
// by one relaxed 128-bit store and polled by their reader until they carry
// the round. A reduction is then one store and one load through L2, where an
// atomic barrier is three dependent trips (arrive, poll, read the partials)
// behind a fence. Two record sets alternate by round: a block writes a set
// again two rounds later, when every block has published the round between
// and has therefore read it. `epoch` (the launch's number, from 1) is the high
// half of the tag, so records need clearing only once.
//
// Cluster form: partials and faces are st.async stores into the reader's
// shared memory that count bytes on the reader's mbarrier; two mbarriers
// alternate by round. Measured on a 16-block cluster this replaced remote
// stores and the hardware cluster barrier (about 1500 cycles of a 2500-cycle
// reduction).
//
// lead() gives the totals to warp 0 alone: one warp forms an iteration's
// scalars and hands them to the block through shared memory, which costs less
// than every warp reducing and dividing (on 16 warps about 600 cycles of an
// iteration). all() gives them to every thread.
//
// Faces are counted in rounds of their own (fround): an exchange with the
// neighbours alone (exchange()) needs no reduction, and two reductions with
// exchanges between them still alternate their record sets.
//
// Every wait is bounded; a block whose wait gave up reports false and leaves.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"

namespace flursys {

constexpr int kRedSlots = 8;
// Polls of one wait (each a trip through L2, about half a microsecond): about a second.
constexpr long long kRedSpinLimit = 2'000'000LL;

struct __align__(16) RedRecord {
    double value;
    unsigned long long tag;
};

__device__ __forceinline__ void st_record(RedRecord *p, double v, unsigned long long tag) {
    asm volatile(
        "{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p),
        "l"(__double_as_longlong(v)), "l"(tag)
        : "memory");
}
__device__ __forceinline__ void ld_record(const RedRecord *p, double &v, unsigned long long &tag) {
    long long b;
    asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
                 : "=l"(b), "=l"(tag)
                 : "l"(p)
                 : "memory");
    v = __longlong_as_double(b);
}

template <bool MAX>
__device__ __forceinline__ double red_op(bool is_max, double a, double b) {
    return MAX && is_max ? fmax(a, b) : a + b;
}

// Sums of v[0..7] over the warp (with MAX the maximum of v[7]): lane l
// returns the total of value l >> 2.
template <bool MAX>
__device__ __forceinline__ double warp_reduce8(const double (&v)[kRedSlots]) {
    const int lane = threadIdx.x & 31;
    const bool h4 = lane & 16, h3 = lane & 8, h2 = lane & 4, m = lane >= 28;
    double a[4], b[2];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const double keep = h4 ? v[i + 4] : v[i], send = h4 ? v[i] : v[i + 4];
        a[i] = red_op<MAX>(i == 3 && h4, keep, __shfl_xor_sync(0xffffffffu, send, 16));
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const double keep = h3 ? a[i + 2] : a[i], send = h3 ? a[i] : a[i + 2];
        b[i] = red_op<MAX>(i == 1 && h4 && h3, keep, __shfl_xor_sync(0xffffffffu, send, 8));
    }
    const double keep = h2 ? b[1] : b[0], send = h2 ? b[0] : b[1];
    double c = red_op<MAX>(m, keep, __shfl_xor_sync(0xffffffffu, send, 4));
    c = red_op<MAX>(m, c, __shfl_xor_sync(0xffffffffu, c, 2));
    return red_op<MAX>(m, c, __shfl_xor_sync(0xffffffffu, c, 1));
}
__device__ __forceinline__ double warp_reduce8(const double (&v)[kRedSlots], bool max7) {
    return max7 ? warp_reduce8<true>(v) : warp_reduce8<false>(v);
}

// Totals of `rows` <= 16 rows of eight partials (row-major in shared memory)
// by one warp: lane l returns the total of value l >> 2. The rows of a lane
// are loaded together and added as a tree.
template <bool MAX>
__device__ __forceinline__ double rows_reduce8(const double *rows8, int rows) {
    const int lane = threadIdx.x & 31;
    const bool m = lane >= 28;
    const double *q = rows8 + (lane & 3) * kRedSlots + (lane >> 2);
    double p[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) p[k] = (lane & 3) + 4 * k < rows ? q[4 * k * kRedSlots] : 0.0;
    double t = red_op<MAX>(m, red_op<MAX>(m, p[0], p[1]), red_op<MAX>(m, p[2], p[3]));
    t = red_op<MAX>(m, t, __shfl_xor_sync(0xffffffffu, t, 2));
    return red_op<MAX>(m, t, __shfl_xor_sync(0xffffffffu, t, 1));
}
__device__ __forceinline__ double rows_reduce8(const double *rows8, int rows, bool max7) {
    return max7 ? rows_reduce8<true>(rows8, rows) : rows_reduce8<false>(rows8, rows);
}

__device__ __forceinline__ void spread8(double t, double (&v)[kRedSlots]) {
#pragma unroll
    for (int k = 0; k < kRedSlots; ++k) v[k] = __shfl_sync(0xffffffffu, t, 4 * k);
}

// 1 / x by the Newton-Raphson iteration y + y (1 - x y), which squares the
// relative error, from the hardware's approximate reciprocal, whose result has
// 20 bits behind the point: about 2^-20, 2^-40, then rounding. For x and 1 / x
// that are normal numbers the error is within two units in the last place.
__device__ __forceinline__ double fast_recip(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
#pragma unroll
    for (int k = 0; k < 2; ++k) y = fma(y, fma(-x, y, 1.0), y);
    return y;
}
// a / b from y, nearly 1 / b: the remainder of the product corrects it
// (Markstein 1990), which leaves no more than one unit in the last place. With
// fast_recip() it replaces a division's subroutine in the scalars' chain (three
// divisions and a square root took about 1000 of an iteration's 5000 cycles on
// 128^2). Where a / b is infinite or undefined the result is not finite either.
__device__ __forceinline__ double quotient_step(double q, double a, double b, double y) { return fma(fma(-q, b, a), y, q); }
__device__ __forceinline__ double quotient(double a, double b, double y) { return quotient_step(a * y, a, b, y); }
// a / b rounded as the division rounds it, from y = 1 / b so rounded: the
// second correction starts within one unit in the last place, where Markstein's
// theorem gives the rounded quotient (remainders below the normal range apart).
// An a that is not finite, or too large for a / b, gives what a y is.
__device__ __forceinline__ double rounded_quotient(double a, double b, double y) {
    const double q = a * y;
    if (!(fabs(q) <= 1.7976931348623157e308)) return q;
    return quotient_step(quotient_step(q, a, b, y), a, b, y);
}

// Hands warp 0's totals and its verdict to the block.
__device__ __forceinline__ bool red_share(double *total, bool ok, int &failed, double (&v)[kRedSlots]) {
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 0; k < kRedSlots; ++k) total[k] = v[k];
        if (!ok) failed = 1;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kRedSlots; ++k) v[k] = total[k];
    return failed == 0;
}

template <int T>
struct GridRedShared {
    double warp[T / 32 * kRedSlots];
    double part[T / 32 * kRedSlots];
    double total[kRedSlots];
    int failed;  // cleared before the first round
};

// The co-resident grid of one launch.
template <int T>
struct GridGroup {
    GridRedShared<T> *sm;
    RedRecord *records;           // 2 * nb * kRedSlots partials
    RedRecord *faces;             // 2 * nb * face_slots
    int nb, rank, face_slots;
    unsigned round, fround;       // reductions and exchanges completed
    unsigned epoch;
    long long spin_limit;
    bool fault;                   // injected: every wait gives up at once
    bool plain_faces = false;     // faces are plain global stores, ordered by the round's fences

    __device__ __forceinline__ unsigned long long tag(unsigned r) const {
        return ((unsigned long long)epoch << 32) | (unsigned long long)(r + 1u);
    }
    // Face value for slot h of block `to`, part of the coming exchange.
    template <typename V>
    __device__ __forceinline__ void send(int to, int h, V v) const {
        st_record(faces + ((size_t)(fround & 1u) * nb + to) * face_slots + h, double(v), tag(fround));
    }
    // This block's face slot h of the last exchange (of the coming one inside
    // `look`): a first look, then the wait.
    __device__ __forceinline__ void peek(int h, double &v, unsigned long long &t) const {
        ld_record(faces + ((size_t)((fround - 1u) & 1u) * nb + rank) * face_slots + h, v, t);
    }
    __device__ __forceinline__ double take(int h, double v, unsigned long long t) const {
        long long spins = 0;
        while (t != tag(fround - 1u)) {
            if (++spins > spin_limit) {
                sm->failed = 1;
                break;
            }
            peek(h, v, t);
        }
        return v;
    }
    // Ends an exchange without a reduction; the halo is then taken slot by slot.
    __device__ __forceinline__ bool exchange(unsigned) {
        ++fround;
        return true;
    }
    // Sums of v over the group, in warp 0; false (there) when a wait gave up.
    // With `with_faces` the round also ends an exchange (`face_bytes` is the
    // cluster form's). `look` runs once the partials have
    // arrived: a first look at the faces, which were sent before them, hides
    // their trip behind the rest of the round. Ends behind a block barrier.
    template <typename F>
    __device__ __forceinline__ bool lead(double (&v)[kRedSlots], bool max7, bool with_faces, unsigned face_bytes, F look) {
        (void)face_bytes;
        if (with_faces) ++fround;
        constexpr int kPer = (160 * kRedSlots + T - 1) / T;  // records per thread (at most 160 blocks)
        const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
        const double w = warp_reduce8(v, max7);
        if ((lane & 3) == 0) sm->warp[wid * kRedSlots + (lane >> 2)] = w;
        __syncthreads();
        const unsigned long long want = tag(round);
        RedRecord *set = records + (size_t)(round & 1u) * nb * kRedSlots;
        ++round;
        if (wid == 0) {
            const double t = rows_reduce8(sm->warp, T / 32, max7);
            if (plain_faces && with_faces) asm volatile("fence.acq_rel.gpu;" ::: "memory");
            if ((lane & 3) == 0) st_record(set + (size_t)rank * kRedSlots + (lane >> 2), t, want);
        }
        // value threadIdx & 7 of blocks threadIdx / 8 + i * T / 8; a record
        // that has arrived is not polled again
        const int total = nb * kRedSlots;
        double pv[kPer];
        unsigned long long pt[kPer];
#pragma unroll
        for (int i = 0; i < kPer; ++i) {
            pt[i] = want;
            pv[i] = 0.0;
            if ((int)threadIdx.x + i * T < total) ld_record(set + threadIdx.x + i * T, pv[i], pt[i]);
        }
        long long spins = fault ? spin_limit : 0;
        for (;;) {
            bool all = !fault;
#pragma unroll
            for (int i = 0; i < kPer; ++i)
                if (pt[i] != want) {
                    all = false;
                    ld_record(set + threadIdx.x + i * T, pv[i], pt[i]);
                }
            if (all) break;
            if (++spins > spin_limit) {
                sm->failed = 1;
                break;
            }
        }
        if (plain_faces && with_faces) asm volatile("fence.acq_rel.gpu;" ::: "memory");
        look();
        const bool m = max7 && (threadIdx.x & 7) == 7;
        double t = 0.0;
#pragma unroll
        for (int i = 0; i < kPer; ++i) t = red_op<true>(m, t, pv[i]);
        t = red_op<true>(m, t, __shfl_xor_sync(0xffffffffu, t, 8));
        t = red_op<true>(m, t, __shfl_xor_sync(0xffffffffu, t, 16));
        if (lane < kRedSlots) sm->part[wid * kRedSlots + lane] = t;
        __syncthreads();
        if (wid == 0) spread8(rows_reduce8(sm->part, T / 32, max7), v);
        return sm->failed == 0;
    }
    __device__ __forceinline__ bool all(double (&v)[kRedSlots], bool max7, bool with_faces = false,
                                        unsigned face_bytes = 0) {
        const bool ok = lead(v, max7, with_faces, face_bytes, [] {});
        return red_share(sm->total, ok, sm->failed, v);
    }
    // A round that also orders global memory: what any thread of the group
    // wrote before it is seen by L2 reads after it.
    __device__ __forceinline__ bool barrier() {
        __threadfence();
        double v[kRedSlots] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        const bool ok = all(v, false);
        __threadfence();
        return ok;
    }
};

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t cluster_addr(uint32_t a, int rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void st_async(uint32_t addr, float v, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(addr),
                 "r"(__float_as_uint(v)), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void st_async(uint32_t addr, double v, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(addr),
                 "l"(__double_as_longlong(v)), "r"(bar)
                 : "memory");
}

template <int T>
struct ClusterRedShared {
    double warp[T / 32 * kRedSlots];
    double part[2][16 * kRedSlots];  // by round parity: the blocks' partials
    unsigned long long bar[2], fbar[2];  // partials and faces, by round parity
    double total[kRedSlots];
    int failed;
};

// One thread-block cluster of nb <= 16 blocks. init() runs before the first
// round, finish() before the blocks leave.
template <int T>
struct ClusterGroup {
    ClusterRedShared<T> *sm;
    int nb, rank, face_slots;
    unsigned round, fround;
    uint32_t faces;  // shared address of this block's 2 * face_slots face values
    bool fault = false;  // injected: the first reduction gives up

    __device__ __forceinline__ void init() {
        if (threadIdx.x == 0) {
            sm->failed = 0;
            for (int k = 0; k < 2; ++k) {
                asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&sm->bar[k])) : "memory");
                asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&sm->fbar[k])) : "memory");
            }
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        cluster_barrier();
    }
    __device__ __forceinline__ void finish() { cluster_barrier(); }
    // Face value for address `a` (of this block; the reader's lies alike) of
    // block `to`, part of the coming exchange. A buffer is free for it once its
    // reader has taken part in a round since it last read the buffer.
    template <typename V>
    __device__ __forceinline__ void send_to(int to, uint32_t a, V v) const {
        st_async(cluster_addr(a, to), v, cluster_addr(smem_addr(&sm->fbar[fround & 1u]), to));
    }
    // The same for slot h of the buffer of the exchange's parity.
    template <typename V>
    __device__ __forceinline__ void send(int to, int h, V v) const {
        send_to(to, faces + ((fround & 1u) * (uint32_t)face_slots + (uint32_t)h) * (uint32_t)sizeof(V), v);
    }
    template <typename V>
    __device__ __forceinline__ V face(const V *base, int h) const {
        return base[((fround - 1u) & 1u) * (unsigned)face_slots + (unsigned)h];
    }
    __device__ __forceinline__ void expect(uint32_t bar, unsigned bytes) const {
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
    }
    __device__ __forceinline__ bool wait(uint32_t bar, unsigned phase) const {
        unsigned done = 0;
        unsigned long long t0 = 0;
        for (unsigned spins = 0;; ++spins) {
            asm volatile(
                "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
                "selp.u32 %0, 1, 0, p;\n\t}"
                : "=r"(done)
                : "r"(bar), "r"(phase)
                : "memory");
            if (done) return true;
            if ((spins & 1023u) == 1023u) {  // give up after about two seconds
                unsigned long long now;
                asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
                if (t0 == 0) t0 = now;
                else if (now - t0 > 2000000000ull) return false;
            }
        }
    }
    // Ends an exchange without a reduction, in warp 0 (see lead()).
    __device__ __forceinline__ bool exchange(unsigned face_bytes) {
        const uint32_t bar = smem_addr(&sm->fbar[fround & 1u]);
        const unsigned phase = (fround >> 1) & 1u;
        ++fround;
        if (threadIdx.x >= 32) return true;
        if (threadIdx.x == 0) expect(bar, face_bytes);
        return __all_sync(0xffffffffu, wait(bar, phase));
    }
    // Sums of v over the cluster, in warp 0; false (there) when its wait gave
    // up. With `with_faces` the round also ends an exchange in which other
    // blocks send `face_bytes` here. The other warps return without waiting: a
    // block barrier that warp 0 enters afterwards orders the faces for them.
    template <typename F>
    __device__ __forceinline__ bool lead(double (&v)[kRedSlots], bool max7, bool with_faces, unsigned face_bytes, F) {
        if (fault) return false;
        const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
        const double w = warp_reduce8(v, max7);
        if ((lane & 3) == 0) sm->warp[wid * kRedSlots + (lane >> 2)] = w;
        __syncthreads();
        const unsigned set = round & 1u, phase = (round >> 1) & 1u;
        double *part = sm->part[set];
        const uint32_t bar = smem_addr(&sm->bar[set]);
        ++round;
        const uint32_t fbar = smem_addr(&sm->fbar[fround & 1u]);
        const unsigned fphase = (fround >> 1) & 1u;
        if (with_faces) ++fround;
        if (wid != 0) return true;
        const double t = rows_reduce8(sm->warp, T / 32, max7);
        const uint32_t mine = smem_addr(part + rank * kRedSlots + (lane >> 2));
        for (int b = lane & 3; b < nb; b += 4) st_async(cluster_addr(mine, b), t, cluster_addr(bar, b));
        if (lane == 0) {
            expect(bar, (unsigned)nb * 8u * kRedSlots);
            if (with_faces) expect(fbar, face_bytes);
        }
        bool done = wait(bar, phase);
        if (with_faces) done = wait(fbar, fphase) && done;
        const bool ok = __all_sync(0xffffffffu, done);
        if (ok) spread8(rows_reduce8(part, nb, max7), v);
        return ok;
    }
    __device__ __forceinline__ bool all(double (&v)[kRedSlots], bool max7, bool with_faces = false,
                                        unsigned face_bytes = 0) {
        const bool ok = lead(v, max7, with_faces, face_bytes, [] {});
        return red_share(sm->total, ok, sm->failed, v);
    }
    __device__ __forceinline__ bool barrier() {
        __threadfence();
        double v[kRedSlots] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        const bool ok = all(v, false);
        __threadfence();
        return ok;
    }
};

}  // namespace flursys
