// fcgnet.cu — kernels of the learned FCG preconditioner (fcgnet.cuh):
// forward, backward and Adam, hand-written for sm_100a.
//
//   conv_tc<CIN, COUT, MODE>  3x3x3 convolution as an implicit GEMM on the
//       tensor cores (mma.sync m16n8k16, BF16 operands, FP32 accumulation):
//       M = 16 voxels along x per warp, N = COUT, K = 27 taps x CIN. A block
//       covers 16 x 8 voxels of one z plane; for each of the three input
//       planes it stages the 18 x 10 halo tile and the 9 taps' weights in
//       shared memory (rows padded by 8 BF16 so the fragment loads hit 32
//       distinct banks). MODE fuses the input transform into the staging:
//       PLAIN reads the tensor, POOL averages 2x2x2 cells of the finer level,
//       UPADD adds the nearest-neighbour upsampled coarser tensor to a skip
//       tensor — with the same FP32 sums and BF16 rounding as the separate
//       pool / up_add kernels, so fused and unfused paths agree bit for bit.
//   conv_umma / conv_umma_tma / conv_umma_pair  the convolutions of
//       inference on the 5th-generation tensor cores (tcgen05.mma, FP32
//       accumulators in tensor memory): register-staged input planes, TMA
//       copies with warp-specialised issue and epilogue, and output planes
//       in pairs (see below)
//   conv_first  1 -> 16 channels (FP32 input, CUDA cores; training)
//   conv_last   16 -> 1 channel (FP32 output, CUDA cores, staged tile; training)
//   net_in_fused / net_out_interior + net_out_boundary  the full-resolution layers of inference,
//               collapsed by linearity into composite stencils (see below)
//   wgrad_mma   dW[co][tap][ci] += sum_v dY[v][co] X[v + tap][ci] of the BF16
//               layers (mma.sync, FP32); wgrad_scalar of the layers with one
//               channel on one side (CUDA cores, FP32)
// The data gradient of a layer is the forward convolution with the
// transposed, flipped weights (NetWeights::bwd), so conv_tc serves both.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdlib>

#include "common.cuh"
#include "fcgnet.cuh"
#include "tma.cuh"

namespace flursys {

namespace {

constexpr int kTX = 16, kTY = 8;              // conv tile: 16 x 8 voxels of one plane
constexpr int kHX = kTX + 2, kHY = kTY + 2;   // with the 1-cell halo
constexpr int kConvThreads = 32 * kTY;        // one warp per tile row
constexpr int kPad = 8;                       // BF16 padding of a staged row

enum StageMode { kPlain = 0, kPool = 1, kUpAdd = 2 };

__device__ __forceinline__ float bf2f(uint16_t b) { return __uint_as_float(uint32_t(b) << 16); }

// Asynchronous global-to-shared copies of N = 4, 8 or 16 bytes; a copy with
// `valid` false writes zeros (source size 0, the source address unread).
template <int N>
__device__ __forceinline__ void cp_async_zfill(void *dst, const void *src, bool valid) {
    const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
    if (N == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(valid ? 16 : 0) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(d), "l"(src), "n"(N), "r"(valid ? N : 0)
                     : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}
__device__ __forceinline__ uint16_t f2bf(float f) {
    const __nv_bfloat16 h = __float2bfloat16_rn(f);
    return *reinterpret_cast<const uint16_t *>(&h);
}

// Eight channels of one voxel of a stage source, as FP32.
struct Src {
    const uint16_t *in;      // PLAIN: the tensor; POOL: the finer tensor; UPADD: the skip tensor
    const uint16_t *coarse;  // UPADD: the coarser tensor
};

// 2x2x2 mean of the finer level (dims 2nx, 2ny, 2nz), channels k8*8..+7.
template <int C>
__device__ __forceinline__ void pool8(const uint16_t *fine, int x, int y, int z, int nx, int ny, int k8, float v[8]) {
    const int fx = 2 * nx, fy = 2 * ny;
    #pragma unroll
    for (int c = 0; c < 8; ++c) v[c] = 0.f;
    #pragma unroll
    for (int a = 0; a < 8; ++a) {
        const long long vox = ((long long)(2 * z + (a >> 2)) * fy + (2 * y + ((a >> 1) & 1))) * fx + (2 * x + (a & 1));
        const uint4 q = *reinterpret_cast<const uint4 *>(fine + vox * C + k8 * 8);
        const uint16_t *h = reinterpret_cast<const uint16_t *>(&q);
        #pragma unroll
        for (int c = 0; c < 8; ++c) v[c] += bf2f(h[c]);
    }
    #pragma unroll
    for (int c = 0; c < 8; ++c) v[c] *= 0.125f;
}

// up(coarse) + skip at (x, y, z), channels k8*8..+7.
template <int C>
__device__ __forceinline__ void upadd8(const uint16_t *coarse, const uint16_t *skip, int x, int y, int z, int nx,
                                       int ny, int k8, float v[8]) {
    const int cx = nx >> 1, cy = ny >> 1;
    const long long cv = ((long long)(z >> 1) * cy + (y >> 1)) * cx + (x >> 1);
    const long long fv = ((long long)z * ny + y) * nx + x;
    const uint4 a = *reinterpret_cast<const uint4 *>(coarse + cv * C + k8 * 8);
    const uint4 b = *reinterpret_cast<const uint4 *>(skip + fv * C + k8 * 8);
    const uint16_t *ha = reinterpret_cast<const uint16_t *>(&a);
    const uint16_t *hb = reinterpret_cast<const uint16_t *>(&b);
    #pragma unroll
    for (int c = 0; c < 8; ++c) v[c] = bf2f(ha[c]) + bf2f(hb[c]);
}

// Eight BF16 channels of voxel (x, y, z) of the staged input (zero outside).
template <int C, int MODE>
__device__ __forceinline__ uint4 load8(const Src &s, int x, int y, int z, int nx, int ny, int nz, int k8) {
    if (x < 0 || y < 0 || z < 0 || x >= nx || y >= ny || z >= nz) return make_uint4(0, 0, 0, 0);
    if (MODE == kPlain) return *reinterpret_cast<const uint4 *>(s.in + (((long long)z * ny + y) * nx + x) * C + k8 * 8);
    float v[8];
    if (MODE == kPool) pool8<C>(s.in, x, y, z, nx, ny, k8, v);
    else upadd8<C>(s.coarse, s.in, x, y, z, nx, ny, k8, v);
    uint4 q;
    uint16_t *h = reinterpret_cast<uint16_t *>(&q);
    #pragma unroll
    for (int c = 0; c < 8; ++c) h[c] = f2bf(v[c]);
    return q;
}

// Stages the 18 x 10 halo tile of plane z (row stride C + kPad).
template <int C, int MODE>
__device__ __forceinline__ void stage_tile(uint16_t *sIn, const Src &s, int x0, int y0, int z, int nx, int ny, int nz) {
    constexpr int K8 = C / 8;
    for (int idx = threadIdx.x; idx < kHY * kHX * K8; idx += blockDim.x) {
        const int k8 = idx % K8, cell = idx / K8;
        const int cx = cell % kHX, cy = cell / kHX;
        const uint4 q = load8<C, MODE>(s, x0 - 1 + cx, y0 - 1 + cy, z, nx, ny, nz, k8);
        *reinterpret_cast<uint4 *>(sIn + (cy * kHX + cx) * (C + kPad) + k8 * 8) = q;
    }
}

__device__ __forceinline__ void mma_bf16(float c[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

template <int CIN, int COUT>
constexpr int conv_smem_bytes() {
    return (kHY * kHX * (CIN + kPad) + 9 * COUT * (CIN + kPad)) * 2;
}

__device__ __forceinline__ void ldsm_x4(uint32_t &r0, uint32_t &r1, uint32_t &r2, uint32_t &r3, const void *p) {
    const unsigned a = static_cast<unsigned>(__cvta_generic_to_shared(p));
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(a));
}

// The 9 taps of one staged input plane (sIn: 18 x 10 halo tile, sW: the 9
// taps' weights [t9][COUT][CIN + kPad]) accumulated into this warp's row of
// 16 voxels x COUT channels. Fragments come from ldmatrix.x4: lane l
// addresses row (l & 7) + 8 ((l >> 3) & 1) at k offset 8 (l >> 4) of A
// (voxels x channels), and row (l & 7) + 8 (l >> 4) at k offset
// 8 ((l >> 3) & 1) of two 8-channel blocks of B; rows are 16-byte aligned
// (CIN + kPad is a multiple of 8) and, with the padding, conflict-free.
// Taps alternate between two accumulator sets (acc for even t9, acc2 for
// odd) so that each warp has twice as many independent MMA chains in flight.
template <int CIN, int COUT>
__device__ __forceinline__ void mma_tap(const uint16_t *sIn, const uint16_t *sW, float (&acc)[COUT / 8][4], int warp,
                                        int t9, int a_row, int a_k, int b_row, int b_k) {
    const int dy = t9 / 3, dx = t9 % 3;  // halo-relative offsets 0..2
    const uint16_t *rowA = sIn + ((warp + dy) * kHX + dx) * (CIN + kPad);
    const uint16_t *wt = sW + t9 * COUT * (CIN + kPad);
    #pragma unroll
    for (int kc = 0; kc < CIN; kc += 16) {
        uint32_t a0, a1, a2, a3;
        ldsm_x4(a0, a1, a2, a3, rowA + a_row * (CIN + kPad) + kc + a_k);
        #pragma unroll
        for (int n = 0; n < COUT / 8; n += 2) {
            uint32_t b0, b1, b2, b3;
            ldsm_x4(b0, b1, b2, b3, wt + (n * 8 + b_row) * (CIN + kPad) + kc + b_k);
            mma_bf16(acc[n], a0, a1, a2, a3, b0, b1);
            mma_bf16(acc[n + 1], a0, a1, a2, a3, b2, b3);
        }
    }
}

template <int CIN, int COUT>
__device__ __forceinline__ void mma_plane(const uint16_t *sIn, const uint16_t *sW, float (&acc)[COUT / 8][4],
                                          float (&acc2)[COUT / 8][4], int warp, int g, int tig) {
    static_assert(COUT % 16 == 0, "B fragments are loaded two 8-channel blocks at a time");
    const int lane = threadIdx.x & 31;
    const int a_row = (lane & 7) + 8 * ((lane >> 3) & 1), a_k = 8 * (lane >> 4);
    const int b_row = (lane & 7) + 8 * (lane >> 4), b_k = 8 * ((lane >> 3) & 1);
    #pragma unroll 1
    for (int t9 = 0; t9 < 8; t9 += 2) {
        mma_tap<CIN, COUT>(sIn, sW, acc, warp, t9, a_row, a_k, b_row, b_k);
        mma_tap<CIN, COUT>(sIn, sW, acc2, warp, t9 + 1, a_row, a_k, b_row, b_k);
    }
    mma_tap<CIN, COUT>(sIn, sW, acc, warp, 8, a_row, a_k, b_row, b_k);
}

// Stores this warp's row of 16 voxels x COUT channels of plane z as BF16.
template <int COUT>
__device__ __forceinline__ void store_row(const float (&acc)[COUT / 8][4], uint16_t *out, int x0, int y, int z, int nx,
                                          int ny, int g, int tig) {
    if (y >= ny) return;
    #pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int x = x0 + g + 8 * h;
        if (x >= nx) continue;
        uint16_t *o = out + (((long long)z * ny + y) * nx + x) * COUT;
        #pragma unroll
        for (int n = 0; n < COUT / 8; ++n) {
            const uint32_t pk = uint32_t(f2bf(acc[n][2 * h])) | (uint32_t(f2bf(acc[n][2 * h + 1])) << 16);
            *reinterpret_cast<uint32_t *>(o + n * 8 + tig * 2) = pk;
        }
    }
}

// Raw global data of one staged element (PLAIN: the voxel's 8 channels;
// UPADD: the coarse and skip channels), loaded before it is needed.
struct RawStage {
    uint4 a, b;
};
template <int C, int MODE>
__device__ __forceinline__ RawStage raw_load(const Src &s, int x, int y, int z, int nx, int ny, int nz, int k8) {
    RawStage r;
    r.a = r.b = make_uint4(0, 0, 0, 0);
    if (x < 0 || y < 0 || z < 0 || x >= nx || y >= ny || z >= nz) return r;
    const long long fv = ((long long)z * ny + y) * nx + x;
    if (MODE == kPlain) {
        r.a = *reinterpret_cast<const uint4 *>(s.in + fv * C + k8 * 8);
    } else {
        const int cx = nx >> 1, cy = ny >> 1;
        const long long cv = ((long long)(z >> 1) * cy + (y >> 1)) * cx + (x >> 1);
        r.a = *reinterpret_cast<const uint4 *>(s.coarse + cv * C + k8 * 8);
        r.b = *reinterpret_cast<const uint4 *>(s.in + fv * C + k8 * 8);
    }
    return r;
}
// The staged value of a raw element: the same FP32 sum and BF16 rounding as load8.
template <int MODE>
__device__ __forceinline__ uint4 raw_finish(const RawStage &r) {
    if (MODE == kPlain) return r.a;
    const uint16_t *ha = reinterpret_cast<const uint16_t *>(&r.a);
    const uint16_t *hb = reinterpret_cast<const uint16_t *>(&r.b);
    uint4 q;
    uint16_t *h = reinterpret_cast<uint16_t *>(&q);
    #pragma unroll
    for (int c = 0; c < 8; ++c) h[c] = f2bf(bf2f(ha[c]) + bf2f(hb[c]));
    return q;
}

// Shared memory of conv_tc_z: all 27 taps' weights and a ring of 3 planes.
template <int CIN, int COUT>
constexpr int conv_z_smem_bytes() {
    return (3 * kHY * kHX * (CIN + kPad) + 27 * COUT * (CIN + kPad)) * 2;
}

// The same convolution marching along z: a block owns a 16 x 8 column of kz
// planes, stages the weights of all 27 taps once, and keeps the last three
// input planes in a ring, so each input plane (and its pool / up-add
// transform) is staged once per block instead of three times, and the
// weights once instead of three times per plane.
template <int CIN, int COUT, int MODE>
__global__ void __launch_bounds__(kConvThreads) conv_tc_z(Src src, const uint16_t *__restrict__ W, uint16_t *out,
                                                          int nx, int ny, int nz, int kz) {
    extern __shared__ __align__(16) uint16_t smem[];
    constexpr int kPlane = kHY * kHX * (CIN + kPad);
    uint16_t *sIn = smem;              // [3][kPlane]
    uint16_t *sW = smem + 3 * kPlane;  // [27][COUT][CIN + kPad]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, tig = lane & 3;
    const int x0 = blockIdx.x * kTX, y0 = blockIdx.y * kTY, z0 = blockIdx.z * kz;
    const int z1 = min(z0 + kz, nz);
    constexpr int K8 = CIN / 8;
    for (int idx = threadIdx.x; idx < 27 * COUT * K8; idx += blockDim.x) {
        const int k8 = idx % K8, rest = idx / K8;
        const int co = rest % COUT, t27 = rest / COUT;
        const uint4 q = *reinterpret_cast<const uint4 *>(W + ((long long)co * 27 + t27) * CIN + k8 * 8);
        *reinterpret_cast<uint4 *>(sW + (t27 * COUT + co) * (CIN + kPad) + k8 * 8) = q;
    }
    // ring slot of plane z: (z - z0 + 1) mod 3
    stage_tile<CIN, MODE>(sIn, src, x0, y0, z0 - 1, nx, ny, nz);
    stage_tile<CIN, MODE>(sIn + kPlane, src, x0, y0, z0, nx, ny, nz);
    // PLAIN / UPADD: the global loads of plane z + 2 are issued before the
    // MMAs of plane z and staged after the next barrier (POOL stages directly)
    constexpr bool kPrefetch = MODE != kPool;
    constexpr int kElems = kHY * kHX * K8;
    constexpr int kPer = (kElems + kConvThreads - 1) / kConvThreads;
    RawStage pre[kPrefetch ? kPer : 1];
    auto prefetch = [&](int zz) {
        #pragma unroll
        for (int i = 0; i < (kPrefetch ? kPer : 1); ++i) {
            const int idx = threadIdx.x + i * kConvThreads;
            if (idx < kElems) {
                const int k8 = idx % K8, cell = idx / K8;
                pre[i] = raw_load<CIN, MODE>(src, x0 - 1 + cell % kHX, y0 - 1 + cell / kHX, zz, nx, ny, nz, k8);
            }
        }
    };
    auto stage_pre = [&](uint16_t *dst) {
        #pragma unroll
        for (int i = 0; i < (kPrefetch ? kPer : 1); ++i) {
            const int idx = threadIdx.x + i * kConvThreads;
            if (idx < kElems) {
                const int k8 = idx % K8, cell = idx / K8;
                *reinterpret_cast<uint4 *>(dst + cell * (CIN + kPad) + k8 * 8) = raw_finish<MODE>(pre[i]);
            }
        }
    };
    if (kPrefetch) prefetch(z0 + 1);
    for (int z = z0; z < z1; ++z) {
        if (kPrefetch) stage_pre(sIn + ((z - z0 + 2) % 3) * kPlane);
        else stage_tile<CIN, MODE>(sIn + ((z - z0 + 2) % 3) * kPlane, src, x0, y0, z + 1, nx, ny, nz);
        __syncthreads();
        if (kPrefetch && z + 1 < z1) prefetch(z + 2);
        float acc[COUT / 8][4], acc2[COUT / 8][4];
        #pragma unroll
        for (int n = 0; n < COUT / 8; ++n)
            #pragma unroll
            for (int e = 0; e < 4; ++e) acc[n][e] = acc2[n][e] = 0.f;
        #pragma unroll 1
        for (int dz = 0; dz < 3; ++dz)
            mma_plane<CIN, COUT>(sIn + ((z - z0 + dz) % 3) * kPlane, sW + dz * 9 * COUT * (CIN + kPad), acc, acc2,
                                 warp, g, tig);
        #pragma unroll
        for (int n = 0; n < COUT / 8; ++n)
            #pragma unroll
            for (int e = 0; e < 4; ++e) acc[n][e] += acc2[n][e];
        store_row<COUT>(acc, out, x0, y0 + warp, z, nx, ny, g, tig);
        __syncthreads();  // the slot of plane z - 1 is staged next
    }
}

template <int CIN, int COUT, int MODE>
__global__ void __launch_bounds__(kConvThreads) conv_tc(Src src, const uint16_t *__restrict__ W, uint16_t *out, int nx,
                                                        int ny, int nz) {
    extern __shared__ __align__(16) uint16_t smem[];
    uint16_t *sIn = smem;
    uint16_t *sW = smem + kHY * kHX * (CIN + kPad);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, tig = lane & 3;
    const int x0 = blockIdx.x * kTX, y0 = blockIdx.y * kTY, z = blockIdx.z;
    float acc[COUT / 8][4], acc2[COUT / 8][4];
    #pragma unroll
    for (int n = 0; n < COUT / 8; ++n)
        #pragma unroll
        for (int e = 0; e < 4; ++e) acc[n][e] = acc2[n][e] = 0.f;

    for (int dz = 0; dz < 3; ++dz) {
        __syncthreads();
        stage_tile<CIN, MODE>(sIn, src, x0, y0, z + dz - 1, nx, ny, nz);
        constexpr int K8 = CIN / 8;
        for (int idx = threadIdx.x; idx < 9 * COUT * K8; idx += blockDim.x) {
            const int k8 = idx % K8, rest = idx / K8;
            const int co = rest % COUT, t9 = rest / COUT;
            const uint4 q = *reinterpret_cast<const uint4 *>(W + ((long long)co * 27 + dz * 9 + t9) * CIN + k8 * 8);
            *reinterpret_cast<uint4 *>(sW + (t9 * COUT + co) * (CIN + kPad) + k8 * 8) = q;
        }
        __syncthreads();
        mma_plane<CIN, COUT>(sIn, sW, acc, acc2, warp, g, tig);
    }
    #pragma unroll
    for (int n = 0; n < COUT / 8; ++n)
        #pragma unroll
        for (int e = 0; e < 4; ++e) acc[n][e] += acc2[n][e];
    store_row<COUT>(acc, out, x0, y0 + warp, z, nx, ny, g, tig);
}

// 1 -> 16 channels: out[v][co] = sum_tap W[co][tap] * scale * in[v + tap].
// scale = *scale_ptr (input normalisation) or 1 when scale_ptr is null.
__global__ void __launch_bounds__(256) conv_first(const float *__restrict__ in, const float *__restrict__ W,
                                                  const double *scale_ptr, uint16_t *out, float *scaled_copy, int nx,
                                                  int ny, int nz) {
    __shared__ float sw[16 * 27];
    for (int i = threadIdx.x; i < 16 * 27; i += blockDim.x) sw[i] = W[i];
    __syncthreads();
    const float scale = scale_ptr ? float(scale_ptr[0]) : 1.f;
    const long long n = (long long)nx * ny * nz;
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < n; v += (long long)gridDim.x * blockDim.x) {
        const int x = int(v % nx);
        const long long t = v / nx;
        const int y = int(t % ny), z = int(t / ny);
        float acc[16];
        #pragma unroll
        for (int c = 0; c < 16; ++c) acc[c] = 0.f;
        #pragma unroll
        for (int tap = 0; tap < 27; ++tap) {
            const int xx = x + tap % 3 - 1, yy = y + (tap / 3) % 3 - 1, zz = z + tap / 9 - 1;
            if (xx < 0 || yy < 0 || zz < 0 || xx >= nx || yy >= ny || zz >= nz) continue;
            const float r = in[((long long)zz * ny + yy) * nx + xx] * scale;
            #pragma unroll
            for (int c = 0; c < 16; ++c) acc[c] = fmaf(sw[c * 27 + tap], r, acc[c]);
        }
        uint4 q[2];
        uint16_t *h = reinterpret_cast<uint16_t *>(q);
        #pragma unroll
        for (int c = 0; c < 16; ++c) h[c] = f2bf(acc[c]);
        uint4 *o = reinterpret_cast<uint4 *>(out + v * 16);
        o[0] = q[0];
        o[1] = q[1];
        if (scaled_copy) scaled_copy[v] = in[v] * scale;
    }
}

// 16 -> 1 channel with an FP32 output: out[v] = out_scale * sum W[tap][ci] x[v+tap][ci].
// out_scale = h2 / scale (input normalisation undone), or 1 without scale_ptr.
// The pinned cell 0 is written as 0 when pin0 is set.
template <int MODE>
__global__ void __launch_bounds__(kTX * kTY) conv_last(Src src, const float *__restrict__ W, const double *scale_ptr,
                                                       double h2, float *out, int nx, int ny, int nz, int pin0) {
    __shared__ __align__(16) uint16_t sIn[3][kHY * kHX * (16 + kPad)];
    __shared__ float sw[27 * 16];
    for (int i = threadIdx.x; i < 27 * 16; i += blockDim.x) sw[i] = W[i];
    const int x0 = blockIdx.x * kTX, y0 = blockIdx.y * kTY, z = blockIdx.z;
    for (int p = 0; p < 3; ++p) stage_tile<16, MODE>(sIn[p], src, x0, y0, z + p - 1, nx, ny, nz);
    __syncthreads();
    const int tx = threadIdx.x % kTX, ty = threadIdx.x / kTX;
    const int x = x0 + tx, y = y0 + ty;
    if (x >= nx || y >= ny) return;
    float acc = 0.f;
    #pragma unroll 1
    for (int tap = 0; tap < 27; ++tap) {
        const int dx = tap % 3, dy = (tap / 3) % 3, dz = tap / 9;
        const uint16_t *c = sIn[dz] + ((ty + dy) * kHX + tx + dx) * (16 + kPad);
        #pragma unroll
        for (int k = 0; k < 16; ++k) acc = fmaf(sw[tap * 16 + k], bf2f(c[k]), acc);
    }
    double s = 1.0;
    if (scale_ptr) s = scale_ptr[0] > 0.0 ? h2 / scale_ptr[0] : 0.0;
    const long long v = ((long long)z * ny + y) * nx + x;
    out[v] = (pin0 && v == 0) ? 0.f : float(double(acc) * s);
}

// Mean (factor 0.125) or sum (factor 1) of 2x2x2 fine cells into the coarse level.
template <int C>
__global__ void pool_kernel(const uint16_t *fine, uint16_t *coarse, int cx, int cy, int cz, float factor) {
    const long long n = (long long)cx * cy * cz * (C / 8);
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const int k8 = int(i % (C / 8));
        const long long v = i / (C / 8);
        const int x = int(v % cx);
        const long long t = v / cx;
        const int y = int(t % cy), z = int(t / cy);
        float s[8];
        pool8<C>(fine, x, y, z, cx, cy, k8, s);  // s = mean
        uint4 q;
        uint16_t *h = reinterpret_cast<uint16_t *>(&q);
        #pragma unroll
        for (int c = 0; c < 8; ++c) h[c] = f2bf(factor == 0.125f ? s[c] : s[c] * 8.f * factor);
        *reinterpret_cast<uint4 *>(coarse + v * C + k8 * 8) = q;
    }
}

// out = up(coarse) + skip, or (accumulate) skip += factor * up(coarse) in place.
template <int C>
__global__ void upadd_kernel(const uint16_t *coarse, const uint16_t *skip, uint16_t *out, int nx, int ny, int nz,
                             float factor, int accumulate) {
    const long long n = (long long)nx * ny * nz * (C / 8);
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const int k8 = int(i % (C / 8));
        const long long v = i / (C / 8);
        const int x = int(v % nx);
        const long long t = v / nx;
        const int y = int(t % ny), z = int(t / ny);
        float s[8];
        if (!accumulate) {
            upadd8<C>(coarse, skip, x, y, z, nx, ny, k8, s);
        } else {
            const long long cv = ((long long)(z >> 1) * (ny >> 1) + (y >> 1)) * (nx >> 1) + (x >> 1);
            const uint4 a = *reinterpret_cast<const uint4 *>(coarse + cv * C + k8 * 8);
            const uint4 b = *reinterpret_cast<const uint4 *>(skip + v * C + k8 * 8);
            const uint16_t *ha = reinterpret_cast<const uint16_t *>(&a);
            const uint16_t *hb = reinterpret_cast<const uint16_t *>(&b);
            #pragma unroll
            for (int c = 0; c < 8; ++c) s[c] = bf2f(hb[c]) + factor * bf2f(ha[c]);
        }
        uint4 q;
        uint16_t *h = reinterpret_cast<uint16_t *>(&q);
        #pragma unroll
        for (int c = 0; c < 8; ++c) h[c] = f2bf(s[c]);
        *reinterpret_cast<uint4 *>(out + v * C + k8 * 8) = q;
    }
}

// ---- weight gradients ---------------------------------------------------
// dW[co][tap][ci] += sum over voxels v of dY[v][co] X[v + tap][ci]: for each
// tap a GEMM with M = COUT, N = CIN and the voxels as K, both operands BF16 as
// stored (channels innermost, so both come through transposing ldmatrix).
// A block owns the three taps of one (dz, dy) and marches over its share of
// the rows, 64 voxel slots at a time; the taps dx are the staged row of X read
// one voxel apart. A warp owns 16 output channels of one tap. Rows are cut into
// pieces of at most 64 voxels padded to 16 with zeros, several to a stage where
// they are short; two stages alternate, the next in flight (cp.async) during
// the MMAs. Each piece (at most 4 chained MMAs) is summed from zero and added
// to the FP32 accumulator by the CUDA cores, so that no long chain runs through
// the tensor cores' own accumulation.
// One thread per weight, walking 1024 voxels with two dependent loads per
// product, took 844 us on 64 -> 32 channels at 16^3 and 432 us on 16 -> 32 at
// 32^3: latency, at 0.5 TFLOP/s.
constexpr int kWgSlots = 64;                // voxel slots of a stage
constexpr int kWgXSlots = kWgSlots + 2 * 4;  // with two halo slots for each of at most four pieces

struct WgradGeom {
    int nx, ny, nz;
    int len, padded, pieces, per_stage;  // voxels of a piece, padded to 16; pieces of a row, of a stage
    long long total, stages;             // pieces and stages in all
};

WgradGeom wgrad_geom(int nx, int ny, int nz) {
    WgradGeom g{nx, ny, nz};
    g.pieces = (nx + kWgSlots - 1) / kWgSlots;
    g.len = (nx + g.pieces - 1) / g.pieces;
    g.padded = (g.len + 15) / 16 * 16;
    g.per_stage = kWgSlots / g.padded;
    g.total = (long long)ny * nz * g.pieces;
    g.stages = (g.total + g.per_stage - 1) / g.per_stage;
    return g;
}

__device__ __forceinline__ void ldsm_x4_trans(uint32_t &r0, uint32_t &r1, uint32_t &r2, uint32_t &r3, const void *p) {
    const unsigned a = static_cast<unsigned>(__cvta_generic_to_shared(p));
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(a));
}

template <int CIN, int COUT>
__global__ void __launch_bounds__(6 * COUT) wgrad_mma(const uint16_t *__restrict__ X, const uint16_t *__restrict__ dY,
                                                      float *dW, const WgradGeom g) {
    constexpr int kThreads = 6 * COUT;  // 3 taps x COUT / 16 warps
    constexpr int SY = COUT + kPad, SX = CIN + kPad, NT = CIN / 8;
    __shared__ __align__(16) uint16_t sY[2][kWgSlots * SY];
    __shared__ __align__(16) uint16_t sX[2][kWgXSlots * SX];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int dx = warp % 3, co0 = (warp / 3) * 16;  // dx: halo-relative 0..2
    const int dy = (int)blockIdx.y % 3 - 1, dz = (int)blockIdx.y / 3 - 1;

    auto stage = [&](long long st, int buf) {
        for (int e = threadIdx.x; e < kWgSlots * (COUT / 8); e += kThreads) {
            const int k8 = e % (COUT / 8), v = e / (COUT / 8), u = v / g.padded, xi = v - u * g.padded;
            const long long piece = st * g.per_stage + u, row = piece / g.pieces;
            const int x = (int)(piece - row * g.pieces) * g.len + xi;
            const bool ok = u < g.per_stage && piece < g.total && xi < g.len && x < g.nx;
            cp_async_zfill<16>(&sY[buf][v * SY + k8 * 8], dY + (ok ? (row * g.nx + x) * COUT + k8 * 8 : 0), ok);
        }
        for (int e = threadIdx.x; e < kWgXSlots * (CIN / 8); e += kThreads) {
            const int k8 = e % (CIN / 8), v = e / (CIN / 8), u = v / (g.padded + 2), xi = v - u * (g.padded + 2);
            const long long piece = st * g.per_stage + u, row = piece / g.pieces;
            const int x = (int)(piece - row * g.pieces) * g.len + xi - 1;
            const int y = (int)(row % g.ny) + dy, z = (int)(row / g.ny) + dz;
            const bool ok = u < g.per_stage && piece < g.total && x >= 0 && x < g.nx && y >= 0 && y < g.ny && z >= 0 &&
                            z < g.nz;
            cp_async_zfill<16>(&sX[buf][v * SX + k8 * 8],
                               X + (ok ? (((long long)z * g.ny + y) * g.nx + x) * CIN + k8 * 8 : 0), ok);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    float acc[NT][4];
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[n][e] = 0.f;
    // ldmatrix rows: voxel 8 (i >> 1) + r, channel 8 (i & 1) of A's four
    // matrices i; voxel 8 (i & 1) + r, channel 8 (i >> 1) of two B tiles
    const int mi = lane >> 3, mr = lane & 7;
    const int a_off = (8 * (mi >> 1) + mr) * SY + 8 * (mi & 1) + co0;
    const int b_off = (8 * (mi & 1) + mr + dx) * SX + 8 * (mi >> 1);
    int buf = 0;
    if (blockIdx.x < g.stages) stage(blockIdx.x, 0);
    for (long long st = blockIdx.x; st < g.stages; st += gridDim.x, buf ^= 1) {
        const bool more = st + gridDim.x < g.stages;
        if (more) stage(st + gridDim.x, buf ^ 1);
        if (more) asm volatile("cp.async.wait_group 1;" ::: "memory");
        else asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        for (int u = 0; u < g.per_stage; ++u) {
            float part[NT][4];
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) part[n][e] = 0.f;
            const uint16_t *pa = sY[buf] + u * g.padded * SY + a_off, *pb = sX[buf] + u * (g.padded + 2) * SX + b_off;
            for (int k = 0; k < g.padded; k += 16) {
                uint32_t a0, a1, a2, a3;
                ldsm_x4_trans(a0, a1, a2, a3, pa + k * SY);
#pragma unroll
                for (int n = 0; n < NT; n += 2) {
                    uint32_t b0, b1, b2, b3;
                    ldsm_x4_trans(b0, b1, b2, b3, pb + k * SX + n * 8);
                    mma_bf16(part[n], a0, a1, a2, a3, b0, b1);
                    mma_bf16(part[n + 1], a0, a1, a2, a3, b2, b3);
                }
            }
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[n][e] += part[n][e];
        }
        __syncthreads();
    }
    const int tap = (dz + 1) * 9 + (dy + 1) * 3 + dx, gr = lane >> 2, tc = 2 * (lane & 3);
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e)
            atomicAdd(dW + ((long long)(co0 + gr + 8 * (e >> 1)) * 27 + tap) * CIN + n * 8 + tc + (e & 1), acc[n][e]);
}

// The layers with one channel on one side: T[c][tap] = sum over voxels u of
// Y[u][c] S[u + tap], Y the 16-channel BF16 tensor, S the FP32 scalar one.
// FIRST (1 -> 16): Y = dY, S = X, dW[c][tap]; otherwise (16 -> 1): Y = X, S =
// dY, dW[26 - tap][c], the tap seen from X. A block stages pieces of 64 voxels
// of a row with the nine rows of S around it; a thread owns four channels and
// the three taps dx of one (dz, dy) over an eighth of the piece, S sliding
// through registers (12 products for two shared loads; one thread per weight
// took 357 us at 64^3).
constexpr int kWsLen = 64, kWsGroups = 8, kWsThreads = 36 * kWsGroups;

template <bool FIRST>
__global__ void __launch_bounds__(kWsThreads) wgrad_scalar(const uint16_t *__restrict__ Y, const float *__restrict__ S,
                                                           float *dW, int nx, int ny, int nz) {
    __shared__ float sS[9][kWsLen + 2];
    __shared__ __align__(16) float sY[kWsLen * 16];
    __shared__ float sum[kWsGroups][432];
    const int grp = threadIdx.x / 36, o = threadIdx.x % 36, pair = o >> 2, quad = o & 3;
    const int pieces = (nx + kWsLen - 1) / kWsLen;
    const long long total = (long long)ny * nz * pieces;
    float acc[3][4] = {};
    for (long long p = blockIdx.x; p < total; p += gridDim.x) {
        const long long row = p / pieces;
        const int x0 = (int)(p - row * pieces) * kWsLen, y = (int)(row % ny), z = (int)(row / ny);
        for (int e = threadIdx.x; e < 9 * (kWsLen + 2); e += kWsThreads) {
            const int q = e / (kWsLen + 2), x = x0 + e % (kWsLen + 2) - 1, yy = y + q % 3 - 1, zz = z + q / 3 - 1;
            const bool ok = x >= 0 && x < nx && yy >= 0 && yy < ny && zz >= 0 && zz < nz;
            sS[q][e % (kWsLen + 2)] = ok ? S[((long long)zz * ny + yy) * nx + x] : 0.f;
        }
        for (int e = threadIdx.x; e < kWsLen * 2; e += kWsThreads) {  // eight channels each
            const int v = e >> 1, x = x0 + v;
            uint4 t = make_uint4(0, 0, 0, 0);
            if (x < nx) t = *reinterpret_cast<const uint4 *>(Y + (row * nx + x) * 16 + 8 * (e & 1));
            const uint16_t *h = reinterpret_cast<const uint16_t *>(&t);
#pragma unroll
            for (int c = 0; c < 8; ++c) sY[v * 16 + 8 * (e & 1) + c] = bf2f(h[c]);
        }
        __syncthreads();
        const int v0 = grp * (kWsLen / kWsGroups);
        float s0 = sS[pair][v0], s1 = sS[pair][v0 + 1];
#pragma unroll
        for (int v = v0; v < v0 + kWsLen / kWsGroups; ++v) {
            const float s2 = sS[pair][v + 2];
            const float4 yv = *reinterpret_cast<const float4 *>(sY + v * 16 + quad * 4);
            const float yc[4] = {yv.x, yv.y, yv.z, yv.w};
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                acc[0][c] = fmaf(yc[c], s0, acc[0][c]);
                acc[1][c] = fmaf(yc[c], s1, acc[1][c]);
                acc[2][c] = fmaf(yc[c], s2, acc[2][c]);
            }
            s0 = s1;
            s1 = s2;
        }
        __syncthreads();
    }
#pragma unroll
    for (int t = 0; t < 3; ++t)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int tap = pair * 3 + t, ch = quad * 4 + c;
            sum[grp][FIRST ? ch * 27 + tap : (26 - tap) * 16 + ch] = acc[t][c];
        }
    __syncthreads();
    for (int e = threadIdx.x; e < 432; e += kWsThreads) {
        float t = 0.f;
#pragma unroll
        for (int k = 0; k < kWsGroups; ++k) t += sum[k][e];
        atomicAdd(dW + e, t);
    }
}

// Energy-norm loss of e = out - p_hat on the unit-spacing Neumann operator L:
// gout = 2 L e / norm, loss += e . L e / norm.
__device__ __forceinline__ float neumann_apply(const float *v, int x, int y, int z, int nx, int ny, int nz) {
    const long long c = ((long long)z * ny + y) * nx + x;
    const long long sy = nx, sz = (long long)nx * ny;
    const float e = v[c];
    float q = 0.f;
    if (x > 0) q += e - v[c - 1];
    if (x + 1 < nx) q += e - v[c + 1];
    if (y > 0) q += e - v[c - sy];
    if (y + 1 < ny) q += e - v[c + sy];
    if (z > 0) q += e - v[c - sz];
    if (z + 1 < nz) q += e - v[c + sz];
    return q;
}

// e = out - p_hat into err_out (the loss kernels read e at the neighbours).
__global__ void __launch_bounds__(256) loss_err(const float *out, const float *p_hat, float *err_out, long long n) {
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < n; v += (long long)gridDim.x * blockDim.x)
        err_out[v] = out[v] - p_hat[v];
}

__global__ void __launch_bounds__(256) loss_kernel(const float *e, float *gout, double inv_norm, double *loss, int nx,
                                                   int ny, int nz) {
    __shared__ double red[8];
    const long long n = (long long)nx * ny * nz;
    double part = 0.0;
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < n; v += (long long)gridDim.x * blockDim.x) {
        const int x = int(v % nx);
        const long long t = v / nx;
        const int y = int(t % ny), z = int(t / ny);
        const float q = neumann_apply(e, x, y, z, nx, ny, nz);
        gout[v] = float(2.0 * double(q) * inv_norm);
        part += double(e[v]) * double(q);
    }
    part = block_sum<256>(part, red);
    if (threadIdx.x == 0) atomicAdd(loss, part * inv_norm);
}

// Residual-norm loss, first pass: q = L e into lq, loss += q.q / norm.
__global__ void __launch_bounds__(256) loss_res_kernel(const float *e, float *lq, double inv_norm, double *loss, int nx,
                                                       int ny, int nz) {
    __shared__ double red[8];
    const long long n = (long long)nx * ny * nz;
    double part = 0.0;
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < n; v += (long long)gridDim.x * blockDim.x) {
        const int x = int(v % nx);
        const long long t = v / nx;
        const int y = int(t % ny), z = int(t / ny);
        const float q = neumann_apply(e, x, y, z, nx, ny, nz);
        lq[v] = q;
        part += double(q) * double(q);
    }
    part = block_sum<256>(part, red);
    if (threadIdx.x == 0) atomicAdd(loss, part * inv_norm);
}

// Residual-norm loss, second pass: gout = 2 L q / norm (L is symmetric).
__global__ void __launch_bounds__(256) loss_res_grad(const float *lq, float *gout, double inv_norm, int nx, int ny,
                                                     int nz) {
    const long long n = (long long)nx * ny * nz;
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < n; v += (long long)gridDim.x * blockDim.x) {
        const int x = int(v % nx);
        const long long t = v / nx;
        const int y = int(t % ny), z = int(t / ny);
        gout[v] = float(2.0 * double(neumann_apply(lq, x, y, z, nx, ny, nz)) * inv_norm);
    }
}

// Sum of squares of r into per-block partials; the finalizer turns the total
// into the normalisation scale 1 / rms(r) (0 for r = 0).
__global__ void __launch_bounds__(256) sumsq_kernel(const float *r, long long n, double *partials) {
    __shared__ double red[8];
    double s = 0.0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const double x = r[i];
        s += x * x;
    }
    s = block_sum<256>(s, red);
    if (threadIdx.x == 0) partials[blockIdx.x] = s;
}
__global__ void __launch_bounds__(256) scale_kernel(const double *partials, int np, long long n, double *scale) {
    __shared__ double red[8];
    double s = 0.0;
    for (int i = threadIdx.x; i < np; i += blockDim.x) s += partials[i];
    s = block_sum<256>(s, red);
    if (threadIdx.x == 0) scale[0] = s > 0.0 ? sqrt(double(n) / s) : 0.0;
}

__global__ void pack_kernel(const float *master, uint16_t *fwd, uint16_t *bwd, float *f32, long long total) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        const int cins[kNetLayers] = {1, 16, 32, 64, 64, 32, 16};   // kNetCin
        const int couts[kNetLayers] = {16, 32, 64, 64, 32, 16, 1};  // kNetCout
        int layer = 0;
        long long off = 0;
        while (layer < kNetLayers - 1 && i >= off + 27LL * cins[layer] * couts[layer]) {
            off += 27LL * cins[layer] * couts[layer];
            ++layer;
        }
        const int cin = cins[layer], cout = couts[layer];
        const long long loc = i - off;
        const int co = int(loc / (27 * cin)), rem = int(loc % (27 * cin)), tap = rem / cin, ci = rem % cin;
        const float w = master[i];
        fwd[i] = f2bf(w);
        bwd[off + ((long long)ci * 27 + (26 - tap)) * cout + co] = f2bf(w);
        if (layer == 0) f32[co * 27 + tap] = w;                      // c1 as [16][27]
        if (layer == kNetLayers - 1) {
            f32[432 + tap * 16 + ci] = w;                            // c7 as [27][16]
            f32[864 + ci * 27 + (26 - tap)] = w;                     // c7 transposed as [16][27]
        }
    }
}

// ---- fused full-resolution layers of the inference path ----------------
// The network is linear, so its full-resolution work collapses:
//   x2  = pool(c1 r)          = K2 * r, a 4x4x4 stencil of stride 2 (16 outputs)
//   out = c7(up(b2) + c1 r)   = sum over 8 coarse cells of Wp * b2
//                               + (c7 o c1) r, a 5x5x5 stencil on r
// c7 zero-pads its input a1 = c1 r (not r), so the composite stencil of a
// cell drops the c7 taps that leave the domain: one 5x5x5 stencil per
// boundary class (low boundary / interior / high boundary on each axis,
// 27 classes). With r zero outside the domain every cell then takes the
// same 125-tap path, exactly as the unfused layers compute it (up to FP32
// instead of BF16 rounding of the intermediate a1 and x7).
// up() is nearest-neighbour, so the 27 taps of c7 on up(b2) reach 2x2x2
// coarse cells, with weights Wp that depend on the parity of the fine cell;
// a fine tap leaves the domain exactly when its coarse cell does.
constexpr int kFusedK2 = 0;                         // [16][64], offsets -1..2 from 2V
constexpr int kFusedK125 = kFusedK2 + 16 * 64;      // [27 classes][125], offsets -2..2
constexpr int kFusedWp = kFusedK125 + 27 * 125;     // [8 parities][8 coarse cells][16]
constexpr int kFusedCount = kFusedWp + 8 * 8 * 16;

__global__ void pack_fused(const float *master, long long off_first, long long off_last, float *fz) {
    const float *W1 = master + off_first;  // [16][27][1]
    const float *W7 = master + off_last;   // [1][27][16]
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kFusedCount; i += gridDim.x * blockDim.x) {
        double acc = 0.0;
        if (i < kFusedK125) {  // K2[c][o], o = (oz*4 + oy)*4 + ox
            const int c = i / 64, o = i % 64;
            const int ox = o % 4 - 1, oy = (o / 4) % 4 - 1, oz = o / 16 - 1;
            for (int a = 0; a < 8; ++a)
                for (int t = 0; t < 27; ++t) {
                    const int dx = t % 3 - 1 + (a & 1), dy = (t / 3) % 3 - 1 + ((a >> 1) & 1), dz = t / 9 - 1 + (a >> 2);
                    if (dx == ox && dy == oy && dz == oz) acc += W1[c * 27 + t];
                }
            acc *= 0.125;
        } else if (i < kFusedWp) {  // K125[class][o]; class axis value 0 low, 1 interior, 2 high
            const int k = i - kFusedK125, cls = k / 125, o = k % 125;
            const int ox = o % 5 - 2, oy = (o / 5) % 5 - 2, oz = o / 25 - 2;
            const int clx = cls % 3, cly = (cls / 3) % 3, clz = cls / 9;
            for (int t7 = 0; t7 < 27; ++t7) {
                const int ax = t7 % 3 - 1, ay = (t7 / 3) % 3 - 1, az = t7 / 9 - 1;
                if ((clx == 0 && ax < 0) || (clx == 2 && ax > 0) || (cly == 0 && ay < 0) || (cly == 2 && ay > 0) ||
                    (clz == 0 && az < 0) || (clz == 2 && az > 0))
                    continue;  // this c7 tap leaves the domain
                const int bx = ox - ax, by = oy - ay, bz = oz - az;  // the c1 tap
                if (bx < -1 || bx > 1 || by < -1 || by > 1 || bz < -1 || bz > 1) continue;
                const int t1 = (bz + 1) * 9 + (by + 1) * 3 + (bx + 1);
                for (int ci = 0; ci < 16; ++ci) acc += double(W7[t7 * 16 + ci]) * W1[ci * 27 + t1];
            }
        } else {  // Wp[par][c8][ci]
            const int k = i - kFusedWp, par = k / 128, c8 = (k / 16) % 8, ci = k % 16;
            for (int t7 = 0; t7 < 27; ++t7) {
                bool hit = true;
                for (int ax = 0; ax < 3; ++ax) {
                    const int p = (par >> ax) & 1, d = (ax == 0 ? t7 % 3 : ax == 1 ? (t7 / 3) % 3 : t7 / 9) - 1;
                    const int f = p + d;                                       // fine offset from 2V, -1..2
                    const int cc = (f >= 0 ? f / 2 : -1) - (p == 0 ? -1 : 0);  // coarse cell 0 or 1
                    if (cc != ((c8 >> ax) & 1)) hit = false;
                }
                if (hit) acc += W7[t7 * 16 + ci];
            }
        }
        fz[i] = float(acc);
    }
}

// The up path of the fused output layer as a GEMM on the tensor cores:
// up[cell][par] = sum over the 27 coarse offsets o and 16 channels ci of
// b2[cell + o][ci] * Wo[o][ci][par], with Wo[o][ci][par] = Wp[par][c8][ci]
// when coarse neighbour o feeds fine child par (c8 its bit pattern) and 0
// otherwise. B operands of mma.m16n8k16 (K = ci, N = par) in fragment order,
// each weight split into BF16 hi + lo (hi + lo = the FP32 weight to ~2^-17):
// upfrag[((o * 2 + split) * 32 + lane) * 2 + reg], reg 0 holding
// k = 2 (lane & 3) + {0, 1} and reg 1 k + 8, of column n = lane >> 2, the
// lower k in the low half.
constexpr int kUpFragWords = 27 * 2 * 32 * 2;

__device__ __forceinline__ float up_weight(const float *wp, int o, int n, int k) {
    const int ox = o % 3 - 1, oy = (o / 3) % 3 - 1, oz = o / 9 - 1;
    const int bx = ox + ((n & 1) ? 0 : 1), by = oy + ((n & 2) ? 0 : 1), bz = oz + ((n & 4) ? 0 : 1);
    if (bx < 0 || bx > 1 || by < 0 || by > 1 || bz < 0 || bz > 1) return 0.f;
    return wp[(n * 8 + (bx | (by << 1) | (bz << 2))) * 16 + k];
}

__global__ void pack_upfrag(const float *fz, uint32_t *upfrag) {
    const float *wp = fz + kFusedWp;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kUpFragWords; i += gridDim.x * blockDim.x) {
        const int reg = i & 1, lane = (i >> 1) & 31, split = (i >> 6) & 1, o = i >> 7;
        const int n = lane >> 2, k = 2 * (lane & 3) + 8 * reg;
        uint32_t word = 0;
        for (int e = 0; e < 2; ++e) {
            const float w = up_weight(wp, o, n, k + e);
            const uint16_t hi = f2bf(w);
            const uint16_t v = split ? f2bf(w - bf2f(hi)) : hi;
            word |= uint32_t(v) << (16 * e);
        }
        upfrag[i] = word;
    }
}

// The input layer as a GEMM on the tensor cores: x2[cell][c] = sum over the
// 64 taps o of r[window of cell][o] * K2[c][o], K = 64 taps in four chunks
// of 16 (one oz plane each: k = 4 oy + ox), N = 16 channels in two tiles of
// 8. B operands of mma.m16n8k16 per lane, each weight split into BF16
// hi + lo: infrag[lane * 32 + ((kc * 2 + nt) * 2 + split) * 2 + reg], reg 0
// holding taps 16 kc + 2 (lane & 3) + {0, 1} and reg 1 those + 8, of channel
// 8 nt + (lane >> 2), the lower tap in the low half.
constexpr int kInFragWords = 32 * 32;

__global__ void pack_infrag(const float *fz, uint32_t *infrag) {
    const float *k2 = fz + kFusedK2;  // [16 channels][64 taps]
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kInFragWords; i += gridDim.x * blockDim.x) {
        const int lane = i >> 5, w = i & 31;
        const int reg = w & 1, split = (w >> 1) & 1, nt = (w >> 2) & 1, kc = w >> 3;
        const int c = 8 * nt + (lane >> 2), o = 16 * kc + 2 * (lane & 3) + 8 * reg;
        uint32_t word = 0;
        for (int e = 0; e < 2; ++e) {
            const float v = k2[c * 64 + o + e];
            const uint16_t hi = f2bf(v);
            const uint16_t u = split ? f2bf(v - bf2f(hi)) : hi;
            word |= uint32_t(u) << (16 * e);
        }
        infrag[i] = word;
    }
}

// Two FP32 values as BF16 pairs hi and lo = bf16(v - hi), the lower element
// in the low half.
__device__ __forceinline__ void split_bf16x2(float2 v, uint32_t &hi, uint32_t &lo) {
    const uint16_t h0 = f2bf(v.x), h1 = f2bf(v.y);
    hi = uint32_t(h0) | (uint32_t(h1) << 16);
    lo = uint32_t(f2bf(v.x - bf2f(h0))) | (uint32_t(f2bf(v.y - bf2f(h1))) << 16);
}

// x2 = bf16(scale * K2 * r) on the level-2 grid (cx, cy, cz): a block owns
// 32 x 8 coarse cells of one coarse layer and stages their 4 x 4 x 4
// windows of r as one shared tile (16-byte cp.async copies of whole rows
// from the 16-byte aligned fine column 2 X0 - 4, zeros outside the grid;
// 4-byte copies of the exact window left the load/store unit the
// bottleneck); each
// warp (one row of 32 cells) forms the GEMM [32 cells x 64 taps] x
// [64 taps x 16 channels] as 4 tap chunks x 2 cell tiles x 2 channel tiles
// of mma.m16n8k16, each with the window values and the weights split into
// BF16 hi + lo and the products hi*hi + hi*lo + lo*hi accumulated in FP32
// (the dropped lo*lo term is ~2^-16 of a product, below the BF16 rounding
// of the output). A operands are pairs of adjacent fine cells of the tile
// (taps ox = 0, 1 and 2, 3).
constexpr int kInCX = 32, kInCY = 8;                                        // coarse cells per block
constexpr int kInWX = 2 * kInCX + 8, kInWY = 2 * kInCY + 2, kInWZ = 4;      // fine window, x from 2 X0 - 4
__global__ void __launch_bounds__(kInCX * kInCY) net_in_fused(const float *__restrict__ r, const double *scale_ptr,
                                                              const uint32_t *__restrict__ infrag, uint16_t *x2,
                                                              int cx, int cy, int cz) {
    __shared__ __align__(16) float win[kInWZ][kInWY][kInWX];
    const int nx = 2 * cx, ny = 2 * cy, nz = 2 * cz;
    const int X0 = blockIdx.x * kInCX, Y0 = blockIdx.y * kInCY, Z = blockIdx.z;
    const int x0 = 2 * X0 - 4, y0 = 2 * Y0 - 1, z0 = 2 * Z - 1;
    {  // 16-byte chunks (x0 and nx are multiples of 4, so a chunk is inside or
       // outside the grid as a whole); every copy is in flight before the block waits
        constexpr int kChunks = kInWX / 4, kAll = kInWZ * kInWY * kChunks;
        for (int i = threadIdx.x; i < kAll; i += blockDim.x) {
            const int row = i / kChunks, ch = i - row * kChunks;
            const int wz = row / kInWY, wy = row - wz * kInWY;
            const int y = y0 + wy, z = z0 + wz, x = x0 + 4 * ch;
            const bool ok = y >= 0 && z >= 0 && y < ny && z < nz && x >= 0 && x < nx;
            const float *src = ok ? r + ((long long)z * ny + y) * nx + x : r;
            cp_async_zfill<16>(&win[wz][wy][4 * ch], src, ok);
        }
        cp_async_wait_all();
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, ty = threadIdx.x >> 5;  // warp ty: coarse row Y0 + ty
    const int Y = Y0 + ty;
    const int g = lane >> 2, t = lane & 3;
    uint32_t bfr[32];
    {
        const uint4 *src = reinterpret_cast<const uint4 *>(infrag) + lane * 8;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint4 q = __ldg(src + i);
            bfr[4 * i] = q.x; bfr[4 * i + 1] = q.y; bfr[4 * i + 2] = q.z; bfr[4 * i + 3] = q.w;
        }
    }
    float cf[2][2][4];
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int i = 0; i < 4; ++i) cf[mt][nt][i] = 0.f;
#pragma unroll
    for (int kc = 0; kc < 4; ++kc) {  // tap plane oz = kc
#pragma unroll
        for (int mt = 0; mt < 2; ++mt) {
            // rows g and g + 8 of the tile: cells 16 mt + g (+ 8); taps
            // k = 2 t + {0, 1} (oy = t >> 1, ox = 2 (t & 1) + {0, 1}) and k + 8
            // (oy + 2); tap ox of cell i sits at window column 2 i + ox + 3
            const float *w0 = &win[kc][2 * ty + (t >> 1)][2 * (16 * mt + g) + 2 * (t & 1) + 3];
            const float2 v0 = make_float2(w0[0], w0[1]);
            const float2 v1 = make_float2(w0[16], w0[17]);
            const float2 v2 = make_float2(w0[2 * kInWX], w0[2 * kInWX + 1]);
            const float2 v3 = make_float2(w0[2 * kInWX + 16], w0[2 * kInWX + 17]);
            uint32_t ah[4], al[4];
            split_bf16x2(v0, ah[0], al[0]);
            split_bf16x2(v1, ah[1], al[1]);
            split_bf16x2(v2, ah[2], al[2]);
            split_bf16x2(v3, ah[3], al[3]);
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
                const uint32_t *bh = bfr + ((kc * 2 + nt) * 2) * 2, *bl = bh + 2;
                mma_bf16(cf[mt][nt], ah[0], ah[1], ah[2], ah[3], bh[0], bh[1]);
                mma_bf16(cf[mt][nt], ah[0], ah[1], ah[2], ah[3], bl[0], bl[1]);
                mma_bf16(cf[mt][nt], al[0], al[1], al[2], al[3], bh[0], bh[1]);
            }
        }
    }
    if (Y >= cy) return;
    const float scale = float(scale_ptr[0]);
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int h = 0; h < 2; ++h) {  // accumulator rows g (h = 0) and g + 8
            const int X = X0 + 16 * mt + g + 8 * h;
            if (X >= cx) continue;
            uint32_t *o = reinterpret_cast<uint32_t *>(x2 + (((long long)Z * cy + Y) * cx + X) * 16);
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
                o[4 * nt + t] = uint32_t(f2bf(cf[mt][nt][2 * h] * scale)) |
                                (uint32_t(f2bf(cf[mt][nt][2 * h + 1] * scale)) << 16);
        }
}

// z = (sum over 8 coarse cells of Wp * b2 + scale * K125[class] * r) * h2 / scale,
// in two launches. net_out_interior applies the interior-class stencil to
// every cell: one thread per coarse cell computes its 2 x 2 x 2 fine cells
// from their 6 x 6 x 6 window of r, read once (float2, conflict-free) from a
// shared tile of one coarse layer, all 125 taps unrolled with the weights a
// by-value parameter (constant-bank operands). The up path runs on the
// tensor cores: each warp (one row of 32 coarse cells) takes the GEMM
// [32 cells x (27 offsets x 16 channels)] x [.. x 8 children] as 27 x 2
// mma.m16n8k16 per weight split, A by ldmatrix from the block's staged BF16
// b2 neighbourhood (zeros outside the grid; 8 consecutive cells are 128
// contiguous bytes, conflict-free), B from upfrag, and hands each cell its
// 8 sums through shared memory. net_out_boundary then adds, on the cells of
// the six faces, h2 * (K125[class] - K125[interior]) * r, the taps of c7
// that leave the domain.
constexpr int kOutCX = 32, kOutCY = 8;                       // coarse cells per block
constexpr int kOutWX = 2 * kOutCX + 8, kOutWY = 2 * kOutCY + 4, kOutWZ = 6;  // fine window, x from 2 X0 - 4
constexpr int kFusedInterior = 13;                            // class 1 + 3 * 1 + 9 * 1
constexpr int kOutBX = kOutCX + 2, kOutBY = kOutCY + 2;       // coarse neighbourhood of a block
constexpr int kOutBwin = 3 * kOutBY * 2 * kOutBX;             // its 16-byte units (two per coarse cell)
constexpr int kOutBwinBytes = kOutBwin * 16;
__global__ void __launch_bounds__(kOutCX * kOutCY) net_out_interior(const float *__restrict__ r,
                                                                    const uint16_t *__restrict__ b2,
                                                                    const uint32_t *__restrict__ upfrag,
                                                                    const double *scale_ptr, double h2, float *out,
                                                                    int nx, int ny, int nz,
                                                                    const __grid_constant__ NetOutParams P) {
    __shared__ __align__(16) float win[kOutWZ][kOutWY][kOutWX];
    // the block's coarse neighbourhood of b2, BF16, zero outside the grid:
    // [layer Z-1..Z+1][row][channel half][column] in 16-byte units
    extern __shared__ __align__(16) uint4 bwin[];
    const int cx = nx >> 1, cy = ny >> 1, cz = nz >> 1;
    const int X0 = blockIdx.x * kOutCX, Y0 = blockIdx.y * kOutCY, Z = blockIdx.z;
    const int x0 = 2 * X0 - 4, y0 = 2 * Y0 - 2, z0 = 2 * Z - 2;
    {  // r in 16-byte chunks from the 16-byte aligned column x0 (x0 and nx are
       // multiples of 4, so a chunk is inside or outside the grid as a
       // whole), then the b2 neighbourhood row by row; every copy is in
       // flight before the block waits
        const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
        constexpr int kChunks = kOutWX / 4, kAll = kOutWZ * kOutWY * kChunks;
        for (int i = threadIdx.x; i < kAll; i += blockDim.x) {
            const int row = i / kChunks, ch = i - row * kChunks;
            const int wz = row / kOutWY, wy = row - wz * kOutWY;
            const int y = y0 + wy, z = z0 + wz, x = x0 + 4 * ch;
            const bool ok = y >= 0 && z >= 0 && y < ny && z < nz && x >= 0 && x < nx;
            const float *src = ok ? r + ((long long)z * ny + y) * nx + x : r;
            cp_async_zfill<16>(&win[wz][wy][4 * ch], src, ok);
        }
        for (int row = threadIdx.x >> 5; row < 3 * kOutBY * 2; row += nw) {
            const int h = row & 1, byz = row >> 1;
            const int bz = byz / kOutBY, by = byz - bz * kOutBY;
            const int Yn = Y0 - 1 + by, Zn = Z - 1 + bz;
            const bool yz = Yn >= 0 && Zn >= 0 && Yn < cy && Zn < cz;
            const uint4 *src = reinterpret_cast<const uint4 *>(b2 + ((long long)(yz ? Zn : 0) * cy + (yz ? Yn : 0)) * cx * 16);
#pragma unroll
            for (int bx = lane; bx < kOutBX; bx += 32) {
                const int Xn = X0 - 1 + bx;
                const bool ok = yz && Xn >= 0 && Xn < cx;
                cp_async_zfill<16>(bwin + row * kOutBX + bx, ok ? src + 2 * Xn + h : src, ok);
            }
        }
        cp_async_wait_all();
    }
    __syncthreads();
    const int tx = threadIdx.x % kOutCX, ty = threadIdx.x / kOutCX;  // warp ty, lane tx
    const int X = X0 + tx, Y = Y0 + ty;
    // up path: coarse neighbour (X + ox, Y + oy, Z + oz) feeds child f when
    // o - (f == 0 ? -1 : 0) is 0 or 1 on every axis (that bit picks c8).
    // Every warp runs it (the MMAs are warp-wide; the staged neighbourhood
    // covers cells past the grid's edge as zeros).
    float up[8];
    {
        const int lane = tx;
        float cf[2][4];
#pragma unroll
        for (int mt = 0; mt < 2; ++mt)
#pragma unroll
            for (int i = 0; i < 4; ++i) cf[mt][i] = 0.f;
        // ldmatrix rows: lane l addresses cell (l & 7) + 8 ((l >> 3) & 1) of
        // the 16-cell tile, channel half l >> 4
        const int arow = (lane & 7) + 8 * ((lane >> 3) & 1), ahalf = lane >> 4;
        const uint2 *bf = reinterpret_cast<const uint2 *>(upfrag) + lane;
#pragma unroll 3
        for (int o = 0; o < 27; ++o) {
            const int ox = o % 3 - 1, oy = (o / 3) % 3 - 1, oz = o / 9 - 1;
            const uint2 bh = __ldg(bf + (o * 2) * 32), bl = __ldg(bf + (o * 2 + 1) * 32);
            const uint4 *rowp = bwin + (((oz + 1) * kOutBY + ty + 1 + oy) * 2 + ahalf) * kOutBX + arow + 1 + ox;
#pragma unroll
            for (int mt = 0; mt < 2; ++mt) {
                uint32_t a0, a1, a2, a3;
                ldsm_x4(a0, a1, a2, a3, rowp + 16 * mt);
                mma_bf16(cf[mt], a0, a1, a2, a3, bh.x, bh.y);
                mma_bf16(cf[mt], a0, a1, a2, a3, bl.x, bl.y);
            }
        }
        // accumulator (row g = lane >> 2 and g + 8 of tile mt, columns
        // 2 (lane & 3) + {0, 1}) to the cell's thread: bwin is free once
        // every warp has read it
        __syncthreads();
        float *ex = reinterpret_cast<float *>(bwin) + ty * 32 * 8;
        const int g = lane >> 2, c2 = 2 * (lane & 3);
#pragma unroll
        for (int mt = 0; mt < 2; ++mt) {
            *reinterpret_cast<float2 *>(ex + (16 * mt + g) * 8 + c2) = make_float2(cf[mt][0], cf[mt][1]);
            *reinterpret_cast<float2 *>(ex + (16 * mt + g + 8) * 8 + c2) = make_float2(cf[mt][2], cf[mt][3]);
        }
        __syncwarp();
        const float4 u0 = reinterpret_cast<const float4 *>(ex + lane * 8)[0];
        const float4 u1 = reinterpret_cast<const float4 *>(ex + lane * 8)[1];
        up[0] = u0.x; up[1] = u0.y; up[2] = u0.z; up[3] = u0.w;
        up[4] = u1.x; up[5] = u1.y; up[6] = u1.z; up[7] = u1.w;
    }
    if (X >= cx || Y >= cy) return;
    // skip path: acc[f], f = fx + 2 fy + 4 fz
    float acc[8];
#pragma unroll
    for (int f = 0; f < 8; ++f) acc[f] = 0.f;
#pragma unroll
    for (int pz = 0; pz < 6; ++pz) {
#pragma unroll
        for (int py = 0; py < 6; ++py) {
            const float2 *row = reinterpret_cast<const float2 *>(&win[pz][2 * ty + py][2 * tx + 2]);
            const float2 a = row[0], b = row[1], c = row[2];
            const float v[6] = {a.x, a.y, b.x, b.y, c.x, c.y};
#pragma unroll
            for (int fz = 0; fz < 2; ++fz) {
                const int dz = pz - 2 - fz;
                if (dz < -2 || dz > 2) continue;
#pragma unroll
                for (int fy = 0; fy < 2; ++fy) {
                    const int dy = py - 2 - fy;
                    if (dy < -2 || dy > 2) continue;
#pragma unroll
                    for (int fx = 0; fx < 2; ++fx)
#pragma unroll
                        for (int dx = -2; dx <= 2; ++dx)
                            acc[fx + 2 * fy + 4 * fz] =
                                fmaf(P.k[((dz + 2) * 5 + dy + 2) * 5 + dx + 2], v[fx + dx + 2], acc[fx + 2 * fy + 4 * fz]);
                }
            }
        }
    }
    const double s = scale_ptr[0];
    const double fac = s > 0.0 ? h2 / s : 0.0;
#pragma unroll
    for (int fz = 0; fz < 2; ++fz)
#pragma unroll
        for (int fy = 0; fy < 2; ++fy) {
            const long long v = ((long long)(2 * Z + fz) * ny + 2 * Y + fy) * nx + 2 * X;
            float2 o;
            o.x = float((double(up[2 * fy + 4 * fz]) + s * double(acc[2 * fy + 4 * fz])) * fac);
            o.y = float((double(up[1 + 2 * fy + 4 * fz]) + s * double(acc[1 + 2 * fy + 4 * fz])) * fac);
            *reinterpret_cast<float2 *>(out + v) = o;
        }
}

// Cells of the six faces: out += h2 * (K125[class] - K125[interior]) * r.
__global__ void __launch_bounds__(256) net_out_boundary(const float *__restrict__ r, const float *__restrict__ fz,
                                                        const double *scale_ptr, double h2, float *out, int nx, int ny,
                                                        int nz) {
    // Per boundary class, the taps (in increasing order) whose correction
    // weight is nonzero and that can land inside the grid (a low class on an
    // axis has no reachable tap below it, a high class none above); each warp
    // compacts some classes with ballots.
    __shared__ short tap[27][125];
    __shared__ float wt[27][125];
    __shared__ int cnt[27];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int cls = warp; cls < 27; cls += blockDim.x >> 5) {
        const int clx = cls % 3, cly = (cls / 3) % 3, clz = cls / 9;
        int n = 0;
        for (int o0 = 0; o0 < 125; o0 += 32) {
            const int o = o0 + lane;
            float d = 0.f;
            if (o < 125) {
                const int dx = o % 5 - 2, dy = (o / 5) % 5 - 2, dz = o / 25 - 2;
                const bool reach = !((clx == 0 && dx < 0) || (clx == 2 && dx > 0) || (cly == 0 && dy < 0) ||
                                     (cly == 2 && dy > 0) || (clz == 0 && dz < 0) || (clz == 2 && dz > 0));
                if (reach) d = __ldg(fz + kFusedK125 + cls * 125 + o) - __ldg(fz + kFusedK125 + kFusedInterior * 125 + o);
            }
            const unsigned m = __ballot_sync(0xffffffffu, d != 0.f);
            if (d != 0.f) {
                const int at = n + __popc(m & ((1u << lane) - 1u));
                tap[cls][at] = (short)o;
                wt[cls][at] = d;
            }
            n += __popc(m);
        }
        if (lane == 0) cnt[cls] = n;
    }
    __syncthreads();
    if (!(scale_ptr[0] > 0.0)) return;
    const long long nzf = 2LL * nx * ny, nyf = 2LL * nx * (nz - 2), nxf = 2LL * (ny - 2) * (nz - 2);
    const long long total = nzf + nyf + nxf;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
         t += (long long)gridDim.x * blockDim.x) {
        int x, y, z;
        if (t < nzf) {  // z = 0 and z = nz - 1
            const long long u = t % ((long long)nx * ny);
            x = int(u % nx); y = int(u / nx); z = t < (long long)nx * ny ? 0 : nz - 1;
        } else if (t < nzf + nyf) {  // y = 0 and y = ny - 1, 0 < z < nz - 1
            const long long w = t - nzf, half = (long long)nx * (nz - 2);
            const long long u = w % half;
            x = int(u % nx); z = 1 + int(u / nx); y = w < half ? 0 : ny - 1;
        } else {  // x = 0 and x = nx - 1, 0 < y < ny - 1, 0 < z < nz - 1
            const long long w = t - nzf - nyf, half = (long long)(ny - 2) * (nz - 2);
            const long long u = w % half;
            y = 1 + int(u % (ny - 2)); z = 1 + int(u / (ny - 2)); x = w < half ? 0 : nx - 1;
        }
        const int cls = (x == 0 ? 0 : x + 1 == nx ? 2 : 1) + 3 * (y == 0 ? 0 : y + 1 == ny ? 2 : 1) +
                        9 * (z == 0 ? 0 : z + 1 == nz ? 2 : 1);
        float corr = 0.f;
        const int nt = cnt[cls];
        for (int k = 0; k < nt; ++k) {
            const int o = tap[cls][k];
            const int dx = o % 5 - 2, dy = (o / 5) % 5 - 2, dz = o / 25 - 2;
            const int xx = x + dx, yy = y + dy, zz = z + dz;
            if (xx < 0 || yy < 0 || zz < 0 || xx >= nx || yy >= ny || zz >= nz) continue;
            corr = fmaf(wt[cls][k], __ldg(r + ((long long)zz * ny + yy) * nx + xx), corr);
        }
        const long long v = ((long long)z * ny + y) * nx + x;
        out[v] = float(double(out[v]) + h2 * double(corr));
    }
}

__global__ void adam_kernel(float *w, const float *g, float *m, float *v, long long n, float lr, float b1, float b2,
                            float eps, float c1, float c2, float gs) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float gi = g[i] * gs;
        const float mi = b1 * m[i] + (1.f - b1) * gi;
        const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        w[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    }
}

int grid_1d(long long n, int per = 256) { return (int)std::max<long long>(1, std::min<long long>((n + per - 1) / per, 148LL * 16)); }

// ---------------------------------------------------------------------------
// conv_umma<CIN, COUT, MODE>: the same 3x3x3 convolution on the 5th-generation
// tensor cores. One CTA (4 warps) owns an 8 (x) x 16 (y) column of voxels
// and marches it through kz planes. Per output plane one thread issues
// 27 x CIN/16 tcgen05.mma (kind::f16, M = 128 voxels, N = COUT, K = 16,
// BF16 operands from shared memory, FP32 accumulator in tensor memory),
// commits them to an mbarrier, and the four warps read the accumulator back
// with tcgen05.ld (warp w owns TMEM lanes 32w..32w+31, i.e. voxel rows
// 4w..4w+3) and store it as BF16. Two accumulator buffers alternate between
// planes, and the loop is a software pipeline: while the MMAs of plane z
// run, the CTA stages input plane z + 2, queues the MMAs of plane z + 1
// into the other buffer, and only then waits for plane z and stores it, so
// the tensor pipe has the next plane's work queued during every epilogue.
//
// Operands are in the K-major no-swizzle core-matrix layout (8 rows x 16 B):
//   input ring, 4 planes: [plane][k8][cell] with cell = cy*10 + cx of the
//     10 x 18 halo tile, 16 B = 8 channels per entry. For tap (dy, dx) the
//     A operand of the 128 voxels (row m = 8 y + x) starts at cell
//     dy*10 + dx; 8-row groups (one voxel row) are 10 cells apart (SBO 160 B)
//     and the two 8-channel halves of K = 16 one slice apart (LBO 2880 B).
//   weights: [tap][k8][co] (16 B entries): B is COUT x 16 per MMA, 8-row
//     groups 128 B apart (SBO), K halves COUT * 16 B apart (LBO).
// Every wait is bounded; a CTA whose accumulator never arrives writes NaN
// to its outputs (the solver then sees a non-finite residual and falls back)
// and still frees its tensor memory.
// ---------------------------------------------------------------------------
constexpr int kUX = 8, kUY = 16;                 // voxels per CTA column (M = 128)
constexpr int kUHX = kUX + 2, kUHY = kUY + 2;    // halo tile 10 x 18
constexpr int kUCells = kUHX * kUHY;             // 180
constexpr int kUThreads = 128;

template <int CIN, int COUT>
struct UmmaConv {
    static constexpr int kSlot = (CIN / 8) * kUCells * 16;       // bytes of one staged plane
    static constexpr int kWBytes = 27 * (CIN / 8) * COUT * 16;   // all taps' weights
    static constexpr int kSmem = 4 * kSlot + kWBytes;
    static constexpr int kTmemCols = 2 * COUT < 32 ? 32 : 2 * COUT;  // two accumulator buffers
};

__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFF);
    d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
    d |= (uint64_t)1 << 46;  // descriptor version (bits 46-48 = 0b001); base offset 0, no swizzle
    return d;
}

__device__ __forceinline__ void umma_f16(uint32_t dtmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(dtmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc));
}

__device__ __forceinline__ bool mbar_wait_bounded(uint32_t mbar, uint32_t parity) {
    for (long long spin = 0; spin < (1LL << 26); ++spin) {
        uint32_t done;
        asm volatile(
            "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done)
            : "r"(mbar), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

// Reads N consecutive FP32 accumulator columns of this thread's TMEM lane.
template <int N>
__device__ __forceinline__ void tmem_ld(uint32_t taddr, float (&v)[N]);
template <>
__device__ __forceinline__ void tmem_ld<16>(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}
template <int N>
__device__ __forceinline__ void tmem_ld(uint32_t taddr, float (&v)[N]) {
    static_assert(N % 16 == 0, "16 columns per load");
#pragma unroll
    for (int c = 0; c < N; c += 16) {
        float t[16];
        tmem_ld<16>(taddr + c, t);
#pragma unroll
        for (int i = 0; i < 16; ++i) v[c + i] = t[i];
    }
}

template <int CIN, int COUT, int MODE>
__global__ void __launch_bounds__(kUThreads) conv_umma(Src src, const uint16_t *__restrict__ W, uint16_t *out,
                                                       int nx, int ny, int nz, int kz) {
    using G = UmmaConv<CIN, COUT>;
    extern __shared__ __align__(1024) uint8_t usmem[];
    __shared__ uint32_t s_tmem;
    __shared__ __align__(8) uint64_t s_mbar[2];
    constexpr int K8 = CIN / 8;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int x0 = blockIdx.x * kUX, y0 = blockIdx.y * kUY, z0 = blockIdx.z * kz;
    const int z1 = min(z0 + kz, nz);
    const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(usmem);
    uint8_t *ring = usmem;
    uint8_t *wts = usmem + 4 * G::kSlot;
    // weights [tap][k8][co] from W[co][tap][ci]
    for (int idx = tid; idx < 27 * K8 * COUT; idx += kUThreads) {
        const int co = idx % COUT, rest = idx / COUT;
        const int k8 = rest % K8, t27 = rest / K8;
        const uint4 q = *reinterpret_cast<const uint4 *>(W + ((long long)co * 27 + t27) * CIN + k8 * 8);
        *reinterpret_cast<uint4 *>(wts + ((t27 * K8 + k8) * COUT + co) * 16) = q;
    }
    // input plane p into its ring slot, channels fastest; every load of a
    // thread is issued before its first store
    constexpr int kItems = (kUCells * K8 + kUThreads - 1) / kUThreads;
    auto stage = [&](int p) {
        uint8_t *slot = ring + ((p + 4) & 3) * G::kSlot;
        uint4 v[kItems];
#pragma unroll
        for (int u = 0; u < kItems; ++u) {
            const int idx = tid + u * kUThreads;
            v[u] = make_uint4(0, 0, 0, 0);
            if (idx < kUCells * K8) {
                const int k8 = idx % K8, cell = idx / K8;
                const int cx = cell % kUHX, cy = cell / kUHX;
                v[u] = load8<CIN, MODE>(src, x0 - 1 + cx, y0 - 1 + cy, p, nx, ny, nz, k8);
            }
        }
#pragma unroll
        for (int u = 0; u < kItems; ++u) {
            const int idx = tid + u * kUThreads;
            if (idx < kUCells * K8) {
                const int k8 = idx % K8, cell = idx / K8;
                *reinterpret_cast<uint4 *>(slot + (k8 * kUCells + cell) * 16) = v[u];
            }
        }
    };
    stage(z0 - 1);
    stage(z0);
    if (z0 + 1 <= z1) stage(z0 + 1);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (warp == 0) {
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&s_tmem);
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst),
                     "n"(G::kTmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    const uint32_t mb0 = (uint32_t)__cvta_generic_to_shared(&s_mbar[0]);
    const uint32_t mb1 = (uint32_t)__cvta_generic_to_shared(&s_mbar[1]);
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mb0));
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mb1));
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_tmem;
    // kind::f16 instruction descriptor: FP32 accumulator, BF16 A and B, both
    // K-major, N = COUT, M = 128
    constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(COUT >> 3) << 17) | ((128u >> 4) << 24);
    // The 27 x CIN/16 MMAs of output plane z into accumulator buffer b, then
    // their commit to that buffer's mbarrier (one thread). Descriptors are
    // formed once per input plane; each tap and K chunk adds a constant
    // offset to the start-address field (addresses stay below 2^18 bytes, so
    // the 14-bit field cannot carry).
    auto issue = [&](int z, int b) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t dbuf = tmem + (uint32_t)(b * COUT);
        const uint64_t wdesc = umma_desc(sbase + 4 * G::kSlot, COUT * 16, 128);
#pragma unroll
        for (int dz = 0; dz < 3; ++dz) {
            const uint64_t adesc = umma_desc(sbase + (uint32_t)(((z + dz - 1 + 4) & 3) * G::kSlot), kUCells * 16, kUHX * 16);
#pragma unroll
            for (int t9 = 0; t9 < 9; ++t9) {
#pragma unroll
                for (int kc = 0; kc < CIN / 16; ++kc) {
                    const int dy = t9 / 3, dx = t9 % 3, tap = dz * 9 + t9;
                    const uint64_t a = adesc + (uint64_t)((((dy * kUHX + dx) + 2 * kc * kUCells) * 16) >> 4);
                    const uint64_t w = wdesc + (uint64_t)((((tap * K8 + 2 * kc) * COUT) * 16) >> 4);
                    umma_f16(dbuf, a, w, kIdesc, (dz | t9 | kc) ? 1u : 0u);
                }
            }
        }
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(b ? mb1 : mb0)
                     : "memory");
    };
    if (tid == 0 && z0 < z1) issue(z0, 0);
    const int m = warp * 32 + lane;  // this thread's voxel row of the accumulator
    const int vx = x0 + (m % kUX), vy = y0 + m / kUX;
    bool ok = true;
    int failed_z = -1;
    for (int z = z0; z < z1; ++z) {
        const int b = (z - z0) & 1;
        // Plane z + 2 goes to the slot of plane z - 2, whose last reader (the
        // MMAs of plane z - 1) finished before the previous epilogue; the
        // MMAs of plane z (planes z - 1 .. z + 1) run meanwhile.
        if (z + 2 <= z1) stage(z + 2);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        // The MMAs of plane z + 1 (into the other buffer, free since the
        // epilogue of plane z - 1) queue behind those of plane z.
        if (tid == 0 && z + 1 < z1) issue(z + 1, b ^ 1);
        const bool arrived = mbar_wait_bounded(b ? mb1 : mb0, (uint32_t)(((z - z0) >> 1) & 1));
        ok = ok && arrived;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        float acc[COUT];
        if (arrived) {
            tmem_ld<COUT>(tmem + (uint32_t)(b * COUT) + ((uint32_t)(warp * 32) << 16), acc);
        } else {
#pragma unroll
            for (int c = 0; c < COUT; ++c) acc[c] = __int_as_float(0x7fc00000);
        }
        if (vx < nx && vy < ny) {
            uint16_t *o = out + (((long long)z * ny + vy) * nx + vx) * COUT;
#pragma unroll
            for (int c = 0; c < COUT; c += 8) {
                uint4 q;
                uint16_t *h = reinterpret_cast<uint16_t *>(&q);
#pragma unroll
                for (int e = 0; e < 8; ++e) h[e] = f2bf(acc[c + e]);
                *reinterpret_cast<uint4 *>(o + c) = q;
            }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        if (!__syncthreads_and(ok)) {  // a lost accumulator: stop, free the tensor memory
            failed_z = z;
            break;
        }
    }
    // the group issued for the plane after a lost accumulator gets its own
    // (bounded) wait before the tensor memory is freed
    if (tid == 0 && failed_z >= 0 && failed_z + 1 < z1) {
        const int zz = failed_z + 1;
        (void)mbar_wait_bounded(((zz - z0) & 1) ? mb1 : mb0, (uint32_t)(((zz - z0) >> 1) & 1));
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(G::kTmemCols));
}

// ---------------------------------------------------------------------------
// conv_umma_tma<CIN, COUT, NS>: the tcgen05 convolution of plain inputs with
// TMA staging and warp-specialised roles, 160 threads. Warps 0-3 are the
// epilogue (warp w reads TMEM lanes 32w..32w+31, voxel rows 4w..4w+3); lane 0
// of warp 4 loads and issues. Input planes arrive by cp.async.bulk.tensor,
// one 8-channel slice per copy (the box 8 channels x 10 x 18 cells lands as
// one K-major core-matrix slice; halo cells outside the tensor are
// zero-filled by the copy engine), into a ring of NS plane slots. Every
// hand-off is an mbarrier:
//   full[s]   the plane in slot s has landed (transaction bytes)
//   done[b]   the MMAs of a plane into accumulator buffer b have completed
//   empty[b]  the four epilogue warps have read accumulator buffer b
// The issuer queues the MMAs of plane z once planes z-1..z+1 have landed
// and buffer b is empty, then, once the MMAs of plane z-1 are done, refills
// the slot of plane z-2 (their last reader) with plane z-2+NS, so each copy
// has NS-3 planes of MMAs to land behind. No block-wide barrier runs inside
// the march. Every wait is bounded: on a timeout the epilogue writes NaN
// for its voxels of that plane (the solver then sees a non-finite residual
// and falls back), and the issuer waits (bounded) for its copies and MMAs in
// flight before the tensor memory is freed.
// ---------------------------------------------------------------------------
constexpr int kUSlice = (kUCells * 16 + 127) / 128 * 128;  // one 8-channel slice, 128-byte aligned
constexpr int kUTmaThreads = 160;

template <int CIN, int COUT>
struct UmmaTma {
    static constexpr int kSlot = (CIN / 8) * kUSlice;
    static constexpr int kWBytes = 27 * (CIN / 8) * COUT * 16;
    static constexpr int smem(int ns) { return ns * kSlot + kWBytes; }
    static constexpr int kTmemCols = 2 * COUT < 32 ? 32 : 2 * COUT;
};

// Waits for phase `parity` of an mbarrier for at most about a second of
// device time (%globaltimer, read every 1024 polls); false when it ran out.
__device__ __forceinline__ bool mbar_wait_timed(uint32_t mbar, uint32_t parity) {
    unsigned long long t0 = 0;
    for (unsigned spin = 1;; ++spin) {
        uint32_t done;
        asm volatile(
            "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done)
            : "r"(mbar), "r"(parity)
            : "memory");
        if (done) return true;
        if ((spin & 1023u) == 0) {
            unsigned long long t;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
            if (t0 == 0) t0 = t;
            else if (t - t0 > 1000000000ull) return false;
        }
    }
}

__device__ __forceinline__ void mbar_arrive_cta(uint32_t mbar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(mbar) : "memory");
}

// The copies of input plane p (K8 slices of 8 channels) into its ring slot,
// completion on that slot's full barrier.
template <int K8, int NS, int SLOT>
__device__ __forceinline__ void tma_plane(uint8_t *ring, uint64_t *full, const CUtensorMap *map, int p, int z0, int x0,
                                          int y0) {
    const int s = (p - z0 + 1) % NS;
    mbar_expect_tx(&full[s], K8 * 8 * kUCells * 2);
#pragma unroll
    for (int k8 = 0; k8 < K8; ++k8) tma_load_4d(ring + s * SLOT + k8 * kUSlice, map, 8 * k8, x0 - 1, y0 - 1, p, &full[s]);
}

template <int CIN, int COUT, int NS>
__global__ void __launch_bounds__(kUTmaThreads) conv_umma_tma(const uint16_t *__restrict__ W, uint16_t *out, int nx,
                                                              int ny, int nz, int kz,
                                                              const __grid_constant__ CUtensorMap tmap) {
    using G = UmmaTma<CIN, COUT>;
    extern __shared__ __align__(1024) uint8_t usmem[];
    __shared__ uint32_t s_tmem;
    __shared__ __align__(8) uint64_t s_full[NS], s_done[2], s_empty[2];
    constexpr int K8 = CIN / 8;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int x0 = blockIdx.x * kUX, y0 = blockIdx.y * kUY, z0 = blockIdx.z * kz;
    const int z1 = min(z0 + kz, nz);
    const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(usmem);
    uint8_t *ring = usmem;
    uint8_t *wts = usmem + NS * G::kSlot;
    const bool issuer = tid == 4 * 32;
    // planes z0 - 1 .. z1 pass through the ring in order
    auto slot_of = [&](int p) { return (p - z0 + 1) % NS; };
    auto full_parity = [&](int p) { return (uint32_t)(((p - z0 + 1) / NS) & 1); };
    auto bar = [](const uint64_t &b) { return (uint32_t)__cvta_generic_to_shared(&b); };
    int loaded = z0 - 2;  // issuer: last plane whose copies were issued
    if (issuer) {
        for (int s = 0; s < NS; ++s) mbar_init(&s_full[s], 1);
        for (int b = 0; b < 2; ++b) {
            mbar_init(&s_done[b], 1);
            mbar_init(&s_empty[b], 4);
        }
        // the first planes' copies overlap the weight staging below
        for (int p = z0 - 1; p <= min(z1, z0 - 2 + NS); ++p) {
            tma_plane<K8, NS, G::kSlot>(ring, s_full, &tmap, p, z0, x0, y0);
            loaded = p;
        }
    }
    // weights [tap][k8][co] from W[co][tap][ci]
    for (int idx = tid; idx < 27 * K8 * COUT; idx += kUTmaThreads) {
        const int co = idx % COUT, rest = idx / COUT;
        const int k8 = rest % K8, t27 = rest / K8;
        const uint4 q = *reinterpret_cast<const uint4 *>(W + ((long long)co * 27 + t27) * CIN + k8 * 8);
        *reinterpret_cast<uint4 *>(wts + ((t27 * K8 + k8) * COUT + co) * 16) = q;
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (warp == 0) {
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&s_tmem);
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst),
                     "n"(G::kTmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_tmem;
    if (issuer) {
        constexpr uint32_t kIdesc =
            (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(COUT >> 3) << 17) | ((128u >> 4) << 24);
        bool ok = true;
        int waited = z0 - 2;  // last plane whose arrival was seen
        int issued = z0 - 1;  // last plane whose MMAs were committed
        int confirmed = z0 - 1;  // last plane whose MMAs were seen complete
        for (int z = z0; z < z1 && ok; ++z) {
            const int b = (z - z0) & 1;
            if (z - z0 >= 2) ok = mbar_wait_timed(bar(s_empty[b]), (uint32_t)(((z - z0 - 2) >> 1) & 1));
            for (int p = waited + 1; p <= z + 1 && ok; ++p) {  // planes z - 1 .. z + 1 landed
                ok = mbar_wait_timed(bar(s_full[slot_of(p)]), full_parity(p));
                if (ok) waited = p;
            }
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t dbuf = tmem + (uint32_t)(b * COUT);
            // the weights' descriptor is formed per plane from an opaque copy
            // of its address, so the compiler keeps the 27 x CIN/16 weight
            // descriptors as immediate offsets instead of hoisting them into
            // registers
            uint32_t waddr;
            asm volatile("mov.u32 %0, %1;" : "=r"(waddr) : "r"(sbase + (uint32_t)(NS * G::kSlot)));
            const uint64_t wdesc = umma_desc(waddr, COUT * 16, 128);
#pragma unroll
            for (int dz = 0; dz < 3; ++dz) {
                const uint64_t adesc = umma_desc(sbase + (uint32_t)(slot_of(z + dz - 1) * G::kSlot), kUSlice, kUHX * 16);
#pragma unroll
                for (int t9 = 0; t9 < 9; ++t9) {
#pragma unroll
                    for (int kc = 0; kc < CIN / 16; ++kc) {
                        const int dy = t9 / 3, dx = t9 % 3, tap = dz * 9 + t9;
                        const uint64_t a = adesc + (uint64_t)((((dy * kUHX + dx) * 16) + 2 * kc * kUSlice) >> 4);
                        const uint64_t w = wdesc + (uint64_t)((((tap * K8 + 2 * kc) * COUT) * 16) >> 4);
                        umma_f16(dbuf, a, w, kIdesc, (dz | t9 | kc) ? 1u : 0u);
                    }
                }
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                             bar(s_done[b]))
                         : "memory");
            issued = z;
            if (z > z0) {
                // the MMAs of plane z - 1 were the last readers of plane z - 2
                ok = mbar_wait_timed(bar(s_done[(z - 1 - z0) & 1]), (uint32_t)(((z - 1 - z0) >> 1) & 1));
                if (ok) confirmed = z - 1;
                if (ok && z - 2 + NS <= z1) {
                    tma_plane<K8, NS, G::kSlot>(ring, s_full, &tmap, z - 2 + NS, z0, x0, y0);
                    loaded = z - 2 + NS;
                }
            }
        }
        if (!ok) {
            // drain what is in flight (bounded): copies not yet seen, MMAs not yet confirmed
            for (int p = waited + 1; p <= loaded; ++p)
                (void)mbar_wait_timed(bar(s_full[slot_of(p)]), full_parity(p));
            for (int z = confirmed + 1; z <= issued; ++z)
                (void)mbar_wait_timed(bar(s_done[(z - z0) & 1]), (uint32_t)(((z - z0) >> 1) & 1));
        }
    } else if (warp < 4) {
        const int m = warp * 32 + lane;  // this thread's voxel row of the accumulator
        const int vx = x0 + (m % kUX), vy = y0 + m / kUX;
        for (int z = z0; z < z1; ++z) {
            const int b = (z - z0) & 1;
            const bool arrived =
                __all_sync(0xffffffffu, mbar_wait_timed(bar(s_done[b]), (uint32_t)(((z - z0) >> 1) & 1)));
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            float acc[COUT];
            if (arrived) {
                tmem_ld<COUT>(tmem + (uint32_t)(b * COUT) + ((uint32_t)(warp * 32) << 16), acc);
            } else {
#pragma unroll
                for (int c = 0; c < COUT; ++c) acc[c] = __int_as_float(0x7fc00000);
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (arrived && lane == 0) mbar_arrive_cta(bar(s_empty[b]));
            if (vx < nx && vy < ny) {
                uint16_t *o = out + (((long long)z * ny + vy) * nx + vx) * COUT;
#pragma unroll
                for (int c = 0; c < COUT; c += 8) {
                    uint4 q;
                    uint16_t *h = reinterpret_cast<uint16_t *>(&q);
#pragma unroll
                    for (int e = 0; e < 8; ++e) h[e] = f2bf(acc[c + e]);
                    *reinterpret_cast<uint4 *>(o + c) = q;
                }
            }
            if (!arrived) break;  // a lost accumulator: stop
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(G::kTmemCols));
}

// The 9 x CIN/16 MMAs of one staged input plane (slot at shared address
// `abase`) against the stacked weights starting at row `wrow` of each
// (t9, k8) block (`wbase` = block 0 + wrow * 16 bytes; blocks 3 COUT rows
// apart), into the accumulator at `dtmem`; `first` clears it with the
// first MMA.
template <int K8, int COUT>
__device__ __forceinline__ void umma_plane(uint32_t abase, uint32_t wbase, uint32_t idesc, uint32_t dtmem, bool first) {
    const uint64_t adesc = umma_desc(abase, kUSlice, kUHX * 16);
    const uint64_t wdesc = umma_desc(wbase, 3 * COUT * 16, 128);
#pragma unroll
    for (int t9 = 0; t9 < 9; ++t9) {
#pragma unroll
        for (int kc = 0; kc < K8 / 2; ++kc) {
            const int dy = t9 / 3, dx = t9 % 3;
            const uint64_t a = adesc + (uint64_t)((((dy * kUHX + dx) * 16) + 2 * kc * kUSlice) >> 4);
            const uint64_t w = wdesc + (uint64_t)((((t9 * K8 + 2 * kc) * 3 * COUT) * 16) >> 4);
            umma_f16(dtmem, a, w, idesc, (first && t9 == 0 && kc == 0) ? 0u : 1u);
        }
    }
}

// ---------------------------------------------------------------------------
// conv_umma_pair<CIN, COUT, NS>: conv_umma_tma computing output planes in
// pairs (z, z + 1). An input plane p feeds outputs p - 1, p, p + 1 through
// the weights of taps dz = 2, 1, 0, so the weights are stored per (t9, k8)
// as one stacked block of 3 x COUT rows [W(dz=2); W(dz=1); W(dz=0)] and one
// MMA of N = 2 COUT takes an input plane into both outputs of the pair:
//   plane z      rows W1;W0 -> outputs z, z+1   (N = 2 COUT, first: clears)
//   plane z + 1  rows W2;W1 -> outputs z, z+1   (N = 2 COUT)
//   plane z - 1  rows W0    -> output z         (N = COUT)
//   plane z + 2  rows W2    -> output z + 1     (N = COUT)
// so each 128-voxel A tile is read from shared memory 36 instead of 54
// times per output plane for CIN = 32 (the A reads bound these MMAs of
// small N). Accumulators: two buffers of 2 COUT columns. Ring of NS = 6
// plane slots: once the MMAs of pair z - 2 are done, planes z - 3 and z - 2
// are refilled with z + 3 and z + 4, which the next pair needs. Roles,
// barriers and the bounded waits are those of conv_umma_tma; planes per
// CTA are even.
// ---------------------------------------------------------------------------
template <int CIN, int COUT>
struct UmmaPair {
    static constexpr int kNS = 6;
    static constexpr int kSlot = (CIN / 8) * kUSlice;
    static constexpr int kWBytes = 27 * (CIN / 8) * COUT * 16;
    static constexpr int kSmem = kNS * kSlot + kWBytes;
    static constexpr int kTmemCols = 4 * COUT < 32 ? 32 : 4 * COUT;
};

template <int CIN, int COUT>
__global__ void __launch_bounds__(kUTmaThreads) conv_umma_pair(const uint16_t *__restrict__ W, uint16_t *out, int nx,
                                                               int ny, int nz, int kz,
                                                               const __grid_constant__ CUtensorMap tmap) {
    using G = UmmaPair<CIN, COUT>;
    constexpr int NS = G::kNS;
    extern __shared__ __align__(1024) uint8_t usmem[];
    __shared__ uint32_t s_tmem;
    __shared__ __align__(8) uint64_t s_full[NS], s_done[2], s_empty[2];
    constexpr int K8 = CIN / 8;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int x0 = blockIdx.x * kUX, y0 = blockIdx.y * kUY, z0 = blockIdx.z * kz;
    const int z1 = min(z0 + kz, nz);  // z1 - z0 is even
    const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(usmem);
    uint8_t *ring = usmem;
    uint8_t *wts = usmem + NS * G::kSlot;
    const bool issuer = tid == 4 * 32;
    auto slot_of = [&](int p) { return (p - z0 + 1) % NS; };
    auto full_parity = [&](int p) { return (uint32_t)(((p - z0 + 1) / NS) & 1); };
    auto bar = [](const uint64_t &b) { return (uint32_t)__cvta_generic_to_shared(&b); };
    int loaded = z0 - 2;
    if (issuer) {
        for (int s = 0; s < NS; ++s) mbar_init(&s_full[s], 1);
        for (int b = 0; b < 2; ++b) {
            mbar_init(&s_done[b], 1);
            mbar_init(&s_empty[b], 4);
        }
        for (int p = z0 - 1; p <= min(z1, z0 - 2 + NS); ++p) {
            tma_plane<K8, NS, G::kSlot>(ring, s_full, &tmap, p, z0, x0, y0);
            loaded = p;
        }
    }
    // weights [t9][k8][(2 - dz) * COUT + co] from W[co][dz * 9 + t9][ci]
    for (int idx = tid; idx < 27 * K8 * COUT; idx += kUTmaThreads) {
        const int co = idx % COUT, rest = idx / COUT;
        const int k8 = rest % K8, t27 = rest / K8;
        const int dz = t27 / 9, t9 = t27 % 9;
        const uint4 q = *reinterpret_cast<const uint4 *>(W + ((long long)co * 27 + t27) * CIN + k8 * 8);
        *reinterpret_cast<uint4 *>(wts + ((t9 * K8 + k8) * 3 * COUT + (2 - dz) * COUT + co) * 16) = q;
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (warp == 0) {
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&s_tmem);
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst),
                     "n"(G::kTmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_tmem;
    if (issuer) {
        constexpr uint32_t kIdesc1 =
            (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(COUT >> 3) << 17) | ((128u >> 4) << 24);
        constexpr uint32_t kIdesc2 =
            (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)((2 * COUT) >> 3) << 17) | ((128u >> 4) << 24);
        const int npairs = (z1 - z0) >> 1;
        bool ok = true;
        int waited = z0 - 2;  // last plane whose arrival was seen
        int issued = -1;      // last pair whose MMAs were committed
        int confirmed = -1;   // last pair whose MMAs were seen complete
        for (int j = 0; j < npairs && ok; ++j) {
            const int z = z0 + 2 * j, b = j & 1;
            if (j >= 2) ok = mbar_wait_timed(bar(s_empty[b]), (uint32_t)(((j - 2) >> 1) & 1));
            for (int p = waited + 1; p <= z + 2 && ok; ++p) {  // planes z - 1 .. z + 2 landed
                ok = mbar_wait_timed(bar(s_full[slot_of(p)]), full_parity(p));
                if (ok) waited = p;
            }
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t dbuf = tmem + (uint32_t)(b * 2 * COUT);
            uint32_t waddr;  // opaque copy: the weight offsets stay immediates
            asm volatile("mov.u32 %0, %1;" : "=r"(waddr) : "r"(sbase + (uint32_t)(NS * G::kSlot)));
            const uint32_t rb = sbase;
            umma_plane<K8, COUT>(rb + slot_of(z) * G::kSlot, waddr + COUT * 16, kIdesc2, dbuf, true);
            umma_plane<K8, COUT>(rb + slot_of(z + 1) * G::kSlot, waddr, kIdesc2, dbuf, false);
            umma_plane<K8, COUT>(rb + slot_of(z - 1) * G::kSlot, waddr + 2 * COUT * 16, kIdesc1, dbuf, false);
            umma_plane<K8, COUT>(rb + slot_of(z + 2) * G::kSlot, waddr, kIdesc1, dbuf + COUT, false);
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                             bar(s_done[b]))
                         : "memory");
            issued = j;
            if (j >= 1) {
                // the MMAs of pair j - 1 were the last readers of planes z - 3 and z - 2
                ok = mbar_wait_timed(bar(s_done[(j - 1) & 1]), (uint32_t)(((j - 1) >> 1) & 1));
                if (ok) confirmed = j - 1;
                for (int p = z - 3 + NS; ok && p <= z - 2 + NS && p <= z1; ++p) {
                    tma_plane<K8, NS, G::kSlot>(ring, s_full, &tmap, p, z0, x0, y0);
                    loaded = p;
                }
            }
        }
        if (!ok) {
            for (int p = waited + 1; p <= loaded; ++p) (void)mbar_wait_timed(bar(s_full[slot_of(p)]), full_parity(p));
            for (int j = confirmed + 1; j <= issued; ++j)
                (void)mbar_wait_timed(bar(s_done[j & 1]), (uint32_t)((j >> 1) & 1));
        }
    } else if (warp < 4) {
        const int m = warp * 32 + lane;
        const int vx = x0 + (m % kUX), vy = y0 + m / kUX;
        const int npairs = (z1 - z0) >> 1;
        for (int j = 0; j < npairs; ++j) {
            const int z = z0 + 2 * j, b = j & 1;
            const bool arrived = __all_sync(0xffffffffu, mbar_wait_timed(bar(s_done[b]), (uint32_t)((j >> 1) & 1)));
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
            for (int h = 0; h < 2; ++h) {  // output planes z and z + 1
                float acc[COUT];
                if (arrived) {
                    tmem_ld<COUT>(tmem + (uint32_t)(b * 2 * COUT + h * COUT) + ((uint32_t)(warp * 32) << 16), acc);
                } else {
#pragma unroll
                    for (int c = 0; c < COUT; ++c) acc[c] = __int_as_float(0x7fc00000);
                }
                if (h == 1) {
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (arrived && lane == 0) mbar_arrive_cta(bar(s_empty[b]));
                }
                if (vx < nx && vy < ny) {
                    uint16_t *o = out + (((long long)(z + h) * ny + vy) * nx + vx) * COUT;
#pragma unroll
                    for (int c = 0; c < COUT; c += 8) {
                        uint4 q;
                        uint16_t *hh = reinterpret_cast<uint16_t *>(&q);
#pragma unroll
                        for (int e = 0; e < 8; ++e) hh[e] = f2bf(acc[c + e]);
                        *reinterpret_cast<uint4 *>(o + c) = q;
                    }
                }
            }
            if (!arrived) break;
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(G::kTmemCols));
}

// Planes per block of conv_tc_z: the largest of 8, 4, 2 that still gives
// about two blocks per SM, else 1.
int conv_planes(int nx, int ny, int nz) {
    const long long xy = (long long)((nx + kTX - 1) / kTX) * ((ny + kTY - 1) / kTY);
    for (int kz = 8; kz > 1; kz /= 2)
        if (xy * ((nz + kz - 1) / kz) >= 2 * 148) return kz;
    return 1;
}

template <int CIN, int COUT, int MODE>
cudaError_t launch_conv(const Src &s, const uint16_t *W, uint16_t *out, int nx, int ny, int nz, cudaStream_t st) {
    constexpr int zsmem = conv_z_smem_bytes<CIN, COUT>();
    static int configured = 0;  // per instantiation: 1 plane kernel, 2 z-marching kernel
    // measured on B200: marching pays where the ring and weights leave room
    // for several blocks per SM (the 128^3-level layers of a 256^3 grid);
    // at 160 KB (one block per SM) the plane kernel is faster
    if (zsmem <= 100 * 1024) {
        if (!configured) {
            cudaError_t e = cudaFuncSetAttribute(conv_tc_z<CIN, COUT, MODE>,
                                                 cudaFuncAttributeMaxDynamicSharedMemorySize, zsmem);
            if (e != cudaSuccess) return e;
            configured = 2;
        }
        const int kz = conv_planes(nx, ny, nz);
        dim3 grid((nx + kTX - 1) / kTX, (ny + kTY - 1) / kTY, (nz + kz - 1) / kz);
        conv_tc_z<CIN, COUT, MODE><<<grid, kConvThreads, zsmem, st>>>(s, W, out, nx, ny, nz, kz);
        return cudaGetLastError();
    }
    constexpr int smem = conv_smem_bytes<CIN, COUT>();
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(conv_tc<CIN, COUT, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return e;
        configured = 1;
    }
    dim3 grid((nx + kTX - 1) / kTX, (ny + kTY - 1) / kTY, nz);
    conv_tc<CIN, COUT, MODE><<<grid, kConvThreads, smem, st>>>(s, W, out, nx, ny, nz);
    return cudaGetLastError();
}

// The convolution of inference: on the 5th-generation tensor cores
// (conv_umma, the default) unless FLURSYS_FCG_UMMA=0, which selects the
// mma.sync kernels (measured on B200 at 256^3: 1.47 against 1.74 ms per
// application).
bool umma_enabled() {
    const char *env = std::getenv("FLURSYS_FCG_UMMA");
    return !(env && env[0] == '0');
}

// Resident CTAs per SM and per device of a tcgen05 convolution kernel with
// `smem` bytes of dynamic shared memory, its carveout set to the maximum so
// that as many CTAs as fit by shared and tensor memory share an SM.
cudaError_t umma_occupancy(const void *fn, int smem, int tmem_cols, int &per_sm, int &slots) {
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
    int dev = 0, sms = 0, smem_sm = 0;
    if (e == cudaSuccess) e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
    if (e != cudaSuccess) return e;
    const int by_smem = smem_sm / (smem + 2048);  // + static and reserved shared memory per CTA
    per_sm = std::max(1, std::min(by_smem, 512 / tmem_cols));
    slots = std::max(1, sms * per_sm);
    return cudaSuccess;
}

// Planes per CTA. Where several CTAs share an SM: the longest march that
// still leaves about four CTAs per resident slot over the launch (measured
// on B200: longer marches with fewer CTAs ran up to 2x slower). Where one
// CTA fills an SM (the weights of all taps take most of the shared
// memory): the longest march whose grid fills its last wave to 85% or
// more, so the weights are loaded once per many planes.
int umma_planes(int nx, int ny, int nz, int per_sm, int slots) {
    const long long cols = (long long)((nx + kUX - 1) / kUX) * ((ny + kUY - 1) / kUY);
    int kz = 1;
    if (per_sm > 1) {
        while (kz < nz && cols * ((nz + 2 * kz - 1) / (2 * kz)) >= 4LL * (slots / per_sm)) kz *= 2;
        return kz;
    }
    double best = -1.0;
    for (int t = 1; t <= nz; t *= 2) {
        const long long ctas = cols * ((nz + t - 1) / t);
        const long long waves = (ctas + slots - 1) / slots;
        const double fill = double(ctas) / double(waves * slots);
        if (fill >= 0.85 || fill > best + 1e-9) {
            if (fill >= 0.85 || best < 0.85) kz = t;
            best = std::max(best, fill);
        }
    }
    return kz;
}

// Input staging of the tcgen05 convolutions of plain tensors: TMA copies
// (conv_umma_tma, the default) unless FLURSYS_FCG_TMA=0, which selects the
// register-staged conv_umma. Plane slots of the TMA ring: 5 where that
// keeps as many CTAs per SM as 4, else 4 (FLURSYS_FCG_TMA_SLOTS=4 or 5
// forces one).
bool tma_conv_enabled() {
    const char *env = std::getenv("FLURSYS_FCG_TMA");
    return !(env && env[0] == '0');
}
int tma_conv_slots_forced() {
    const char *env = std::getenv("FLURSYS_FCG_TMA_SLOTS");
    const int v = env ? std::atoi(env) : 0;
    return v == 4 || v == 5 ? v : 0;
}

// Output planes in pairs (conv_umma_pair) where its six-slot ring fits and
// the planes per CTA come out even, unless FLURSYS_FCG_PAIR=0.
bool pair_conv_enabled() {
    const char *env = std::getenv("FLURSYS_FCG_PAIR");
    return !(env && env[0] == '0');
}

template <int CIN, int COUT>
cudaError_t launch_conv_pair(const Src &s, const uint16_t *W, uint16_t *out, int nx, int ny, int nz, int kz,
                             cudaStream_t st) {
    CUtensorMap map;
    if (!tma_map_bf16_cxyz(&map, s.in, CIN, nx, ny, nz, 8, kUHX, kUHY)) return cudaErrorInvalidValue;
    dim3 grid((nx + kUX - 1) / kUX, (ny + kUY - 1) / kUY, (nz + kz - 1) / kz);
    conv_umma_pair<CIN, COUT><<<grid, kUTmaThreads, UmmaPair<CIN, COUT>::kSmem, st>>>(W, out, nx, ny, nz, kz, map);
    return cudaGetLastError();
}

template <int CIN, int COUT, int NS>
cudaError_t launch_conv_tma(const Src &s, const uint16_t *W, uint16_t *out, int nx, int ny, int nz, int per_sm,
                            int slots, cudaStream_t st) {
    CUtensorMap map;
    if (!tma_map_bf16_cxyz(&map, s.in, CIN, nx, ny, nz, 8, kUHX, kUHY)) return cudaErrorInvalidValue;
    const int kz = umma_planes(nx, ny, nz, per_sm, slots);
    dim3 grid((nx + kUX - 1) / kUX, (ny + kUY - 1) / kUY, (nz + kz - 1) / kz);
    conv_umma_tma<CIN, COUT, NS><<<grid, kUTmaThreads, UmmaTma<CIN, COUT>::smem(NS), st>>>(W, out, nx, ny, nz, kz, map);
    return cudaGetLastError();
}

template <int CIN, int COUT, int MODE>
cudaError_t launch_conv_fwd(const Src &s, const uint16_t *W, uint16_t *out, int nx, int ny, int nz, cudaStream_t st) {
    using G = UmmaConv<CIN, COUT>;
    using T = UmmaTma<CIN, COUT>;
    if (!umma_enabled() || G::kSmem > 220 * 1024) return launch_conv<CIN, COUT, MODE>(s, W, out, nx, ny, nz, st);
    if constexpr (MODE == kPlain && T::smem(4) <= 220 * 1024) {
        if constexpr (UmmaPair<CIN, COUT>::kSmem <= 220 * 1024) {
            if (tma_conv_enabled() && pair_conv_enabled() && nz % 2 == 0) {
                using P = UmmaPair<CIN, COUT>;
                static int pper = 0, pslots = 0;  // per instantiation
                if (!pslots) {
                    cudaError_t e = umma_occupancy((const void *)conv_umma_pair<CIN, COUT>, P::kSmem, P::kTmemCols,
                                                   pper, pslots);
                    if (e != cudaSuccess) return e;
                }
                const int kz = umma_planes(nx, ny, nz, pper, pslots);
                if (kz % 2 == 0) return launch_conv_pair<CIN, COUT>(s, W, out, nx, ny, nz, kz, st);
            }
        }
        if (tma_conv_enabled()) {
        // per instantiation: resident CTAs of the 4- and 5-slot rings, and the choice
        static int ns = 0, per4 = 0, slots4 = 0, per5 = 0, slots5 = 0;
        if (!ns) {
            cudaError_t e = umma_occupancy((const void *)conv_umma_tma<CIN, COUT, 4>, T::smem(4), T::kTmemCols, per4, slots4);
            if (e != cudaSuccess) return e;
            ns = 4;
            if (T::smem(5) <= 220 * 1024) {
                e = umma_occupancy((const void *)conv_umma_tma<CIN, COUT, 5>, T::smem(5), T::kTmemCols, per5, slots5);
                if (e != cudaSuccess) return e;
                if (per5 == per4) ns = 5;
            }
            const int forced = tma_conv_slots_forced();
            if (forced == 4 || (forced == 5 && per5 > 0)) ns = forced;
        }
        if (ns == 5) return launch_conv_tma<CIN, COUT, 5>(s, W, out, nx, ny, nz, per5, slots5, st);
        return launch_conv_tma<CIN, COUT, 4>(s, W, out, nx, ny, nz, per4, slots4, st);
        }
    }
    static int slots = 0, per_sm = 0;  // resident CTAs per device and per SM (per instantiation)
    if (!slots) {
        cudaError_t e = umma_occupancy((const void *)conv_umma<CIN, COUT, MODE>, G::kSmem, G::kTmemCols, per_sm, slots);
        if (e != cudaSuccess) return e;
    }
    const int kz = umma_planes(nx, ny, nz, per_sm, slots);
    dim3 grid((nx + kUX - 1) / kUX, (ny + kUY - 1) / kUY, (nz + kz - 1) / kz);
    conv_umma<CIN, COUT, MODE><<<grid, kUThreads, G::kSmem, st>>>(s, W, out, nx, ny, nz, kz);
    return cudaGetLastError();
}

template <int C>
cudaError_t launch_pool(const uint16_t *fine, uint16_t *coarse, int cx, int cy, int cz, float factor, cudaStream_t st) {
    pool_kernel<C><<<grid_1d((long long)cx * cy * cz * (C / 8)), 256, 0, st>>>(fine, coarse, cx, cy, cz, factor);
    return cudaGetLastError();
}
cudaError_t pool_any(int c, const uint16_t *fine, uint16_t *coarse, int cx, int cy, int cz, float factor, cudaStream_t st) {
    switch (c) {
        case 16: return launch_pool<16>(fine, coarse, cx, cy, cz, factor, st);
        case 32: return launch_pool<32>(fine, coarse, cx, cy, cz, factor, st);
        default: return launch_pool<64>(fine, coarse, cx, cy, cz, factor, st);
    }
}
template <int C>
cudaError_t launch_upadd(const uint16_t *coarse, const uint16_t *skip, uint16_t *out, int nx, int ny, int nz,
                         float factor, int acc, cudaStream_t st) {
    upadd_kernel<C><<<grid_1d((long long)nx * ny * nz * (C / 8)), 256, 0, st>>>(coarse, skip, out, nx, ny, nz, factor, acc);
    return cudaGetLastError();
}
cudaError_t upadd_any(int c, const uint16_t *coarse, const uint16_t *skip, uint16_t *out, int nx, int ny, int nz,
                      float factor, int acc, cudaStream_t st) {
    switch (c) {
        case 16: return launch_upadd<16>(coarse, skip, out, nx, ny, nz, factor, acc, st);
        case 32: return launch_upadd<32>(coarse, skip, out, nx, ny, nz, factor, acc, st);
        default: return launch_upadd<64>(coarse, skip, out, nx, ny, nz, factor, acc, st);
    }
}

template <int CIN, int COUT>
cudaError_t launch_wgrad(const uint16_t *X, const uint16_t *dY, float *dW, int nx, int ny, int nz, cudaStream_t st) {
    const WgradGeom g = wgrad_geom(nx, ny, nz);
    // nine (dz, dy) blocks per share of the rows: about four blocks per SM at most
    dim3 grid((unsigned)std::min<long long>(g.stages, 64), 9);
    wgrad_mma<CIN, COUT><<<grid, 6 * COUT, 0, st>>>(X, dY, dW, g);
    return cudaGetLastError();
}
template <bool FIRST>
cudaError_t launch_wgrad_scalar(const uint16_t *Y, const float *S, float *dW, int nx, int ny, int nz, cudaStream_t st) {
    const long long total = (long long)ny * nz * ((nx + kWsLen - 1) / kWsLen);
    wgrad_scalar<FIRST><<<(unsigned)std::min<long long>(total, 148 * 4), kWsThreads, 0, st>>>(Y, S, dW, nx, ny, nz);
    return cudaGetLastError();
}

size_t al(size_t b) { return (b + 255) & ~size_t(255); }

}  // namespace

long long net_param_offset(int layer) {
    long long off = 0;
    for (int l = 0; l < layer; ++l) off += 27LL * kNetCin[l] * kNetCout[l];
    return off;
}
long long net_param_count() { return net_param_offset(kNetLayers); }

cudaError_t NetWorkspace::ensure(int nx_, int ny_, int nz_, bool training_) {
    const long long v1 = (long long)nx_ * ny_ * nz_, v2 = v1 / 8, v3 = v1 / 64, v4 = v1 / 512;
    // element counts (BF16) of every tensor, in declaration order
    // (inference fuses the full-resolution layers, so it keeps x2, a2, a3,
    // a4, b3, b2 and, for the tensor-memory convolutions that stage plain
    // tensors, the pooled / up-added inputs x3, x5, x6)
    const long long tr = training_ ? 1 : 0;
    const long long sizes[24] = {
        tr * v1 * 16, v2 * 16, v2 * 32, v3 * 32, v3 * 64, tr * v4 * 64, v4 * 64,  // a1 x2 a2 x3 a3 x4 a4
        v3 * 64, v3 * 32, v2 * 32, v2 * 16, tr * v1 * 16,                         // x5 b3 x6 b2 x7
        v1 * 16, v2 * 32, v3 * 64, v4 * 64, v3 * 32, v2 * 16,                          // g7 g6 g5 g4 g3 g2
        v2 * 16, v3 * 32, v4 * 64, 0, 0, 0};                                           // gb2 gb3 ga4
    const int ntensor = training_ ? 21 : 12;
    size_t need = 0;
    for (int i = 0; i < ntensor; ++i) need += al(size_t(sizes[i]) * 2);
    const int np = 1024;
    need += al(size_t(v1) * 4) * (training_ ? 3 : 0) + al(8 * 8) + al(size_t(np) * 8);
    if (base && need <= bytes && nx_ == nx && ny_ == ny && nz_ == nz && training == training_) return cudaSuccess;
    if (!base || need > bytes) {
        release();
        cudaError_t e = cudaMalloc(&base, need);
        if (e != cudaSuccess) {
            base = nullptr;
            return e;
        }
        bytes = need;
    }
    nx = nx_; ny = ny_; nz = nz_;
    training = training_;
    char *p = static_cast<char *>(base);
    uint16_t **slots[21] = {&a1, &x2, &a2, &x3, &a3, &x4, &a4, &x5, &b3, &x6, &b2, &x7,
                            &g7, &g6, &g5, &g4, &g3, &g2, &gb2, &gb3, &ga4};
    for (int i = 0; i < 21; ++i) *slots[i] = nullptr;
    for (int i = 0; i < ntensor; ++i) {
        if (sizes[i] == 0) continue;
        *slots[i] = reinterpret_cast<uint16_t *>(p);
        p += al(size_t(sizes[i]) * 2);
    }
    ga3 = g5; ga2 = g6; ga1 = g7;  // skip-path gradients accumulate in place
    out32 = gout = lq = nullptr;
    if (training_) {
        out32 = reinterpret_cast<float *>(p); p += al(size_t(v1) * 4);
        lq = reinterpret_cast<float *>(p); p += al(size_t(v1) * 4);
        gout = reinterpret_cast<float *>(p); p += al(size_t(v1) * 4);
    }
    scalars = reinterpret_cast<double *>(p); p += al(8 * 8);
    partials = reinterpret_cast<double *>(p);
    npartials = np;
    return cudaSuccess;
}

void NetWorkspace::release() {
    if (base) cudaFree(base);
    base = nullptr;
    bytes = 0;
    nx = ny = nz = 0;
}

cudaError_t NetWeights::allocate() {
    const long long n = net_param_count();
    cudaError_t e = cudaMalloc(&fwd, n * 2);
    if (e == cudaSuccess) e = cudaMalloc(&bwd, n * 2);
    if (e == cudaSuccess) e = cudaMalloc(&fwd_f32, 1296 * sizeof(float));
    if (e == cudaSuccess) e = cudaMalloc(&fused, kFusedCount * sizeof(float));
    if (e == cudaSuccess) e = cudaMalloc(&upfrag, kUpFragWords * sizeof(uint32_t));
    if (e == cudaSuccess) e = cudaMalloc(&infrag, kInFragWords * sizeof(uint32_t));
    return e;
}

void NetWeights::release() {
    if (fwd) cudaFree(fwd);
    if (bwd) cudaFree(bwd);
    if (fwd_f32) cudaFree(fwd_f32);
    if (fused) cudaFree(fused);
    if (upfrag) cudaFree(upfrag);
    if (infrag) cudaFree(infrag);
    fwd = bwd = nullptr;
    fwd_f32 = fused = nullptr;
    upfrag = infrag = nullptr;
}

cudaError_t net_pack_weights(const float *master, NetWeights &w, cudaStream_t st) {
    const long long n = net_param_count();
    pack_kernel<<<grid_1d(n), 256, 0, st>>>(master, w.fwd, w.bwd, w.fwd_f32, n);
    pack_fused<<<(kFusedCount + 63) / 64, 64, 0, st>>>(master, net_param_offset(0), net_param_offset(kNetLayers - 1), w.fused);
    pack_upfrag<<<(kUpFragWords + 127) / 128, 128, 0, st>>>(w.fused, w.upfrag);
    pack_infrag<<<(kInFragWords + 127) / 128, 128, 0, st>>>(w.fused, w.infrag);
    w.host_params_valid = false;
    return cudaGetLastError();
}

cudaError_t net_apply(const NetWeights &w, NetWorkspace &ws, int nx, int ny, int nz, double h2, const float *r, float *z,
                      cudaStream_t st) {
    if (nx % 8 || ny % 8 || nz % 8) return cudaErrorInvalidValue;
    cudaError_t e = ws.ensure(nx, ny, nz, false);
    if (e != cudaSuccess) return e;
    const long long n = (long long)nx * ny * nz;
    const int np = std::min(ws.npartials, grid_1d(n));
    sumsq_kernel<<<np, 256, 0, st>>>(r, n, ws.partials);
    scale_kernel<<<1, 256, 0, st>>>(ws.partials, np, n, ws.scalars);
    const int n2x = nx / 2, n2y = ny / 2, n2z = nz / 2, n3x = nx / 4, n3y = ny / 4, n3z = nz / 4;
    const int n4x = nx / 8, n4y = ny / 8, n4z = nz / 8;
    if (!w.host_params_valid) {
        // first application after a repack: bring the output layer's interior stencil to the host
        NetOutParams &P = w.out_params;
        e = cudaMemcpyAsync(P.k, w.fused + kFusedK125 + kFusedInterior * 125, sizeof P.k, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) return e;
        w.host_params_valid = true;
    }
    {
        dim3 grid((n2x + kInCX - 1) / kInCX, (n2y + kInCY - 1) / kInCY, n2z);
        net_in_fused<<<grid, kInCX * kInCY, 0, st>>>(r, ws.scalars, w.infrag, ws.x2, n2x, n2y, n2z);
    }
    e = cudaGetLastError();
    const uint16_t *W = w.fwd;
    if (e == cudaSuccess) e = launch_conv_fwd<16, 32, kPlain>(Src{ws.x2, nullptr}, W + net_param_offset(1), ws.a2, n2x, n2y, n2z, st);
    if (umma_enabled()) {
        // The tensor-memory convolutions stage plain tensors: pool and up-add
        // run as their own passes (same FP32 sums and BF16 rounding as the
        // fused staging of the mma.sync kernels, so the operands are equal).
        if (e == cudaSuccess) e = launch_pool<32>(ws.a2, ws.x3, n3x, n3y, n3z, 0.125f, st);
        if (e == cudaSuccess) e = launch_conv_fwd<32, 64, kPlain>(Src{ws.x3, nullptr}, W + net_param_offset(2), ws.a3, n3x, n3y, n3z, st);
        if (e == cudaSuccess) e = launch_conv_fwd<64, 64, kPool>(Src{ws.a3, nullptr}, W + net_param_offset(3), ws.a4, n4x, n4y, n4z, st);
        if (e == cudaSuccess) e = launch_upadd<64>(ws.a4, ws.a3, ws.x5, n3x, n3y, n3z, 1.f, 0, st);
        if (e == cudaSuccess) e = launch_conv_fwd<64, 32, kPlain>(Src{ws.x5, nullptr}, W + net_param_offset(4), ws.b3, n3x, n3y, n3z, st);
        if (e == cudaSuccess) e = launch_upadd<32>(ws.b3, ws.a2, ws.x6, n2x, n2y, n2z, 1.f, 0, st);
        if (e == cudaSuccess) e = launch_conv_fwd<32, 16, kPlain>(Src{ws.x6, nullptr}, W + net_param_offset(5), ws.b2, n2x, n2y, n2z, st);
    } else {
        if (e == cudaSuccess) e = launch_conv_fwd<32, 64, kPool>(Src{ws.a2, nullptr}, W + net_param_offset(2), ws.a3, n3x, n3y, n3z, st);
        if (e == cudaSuccess) e = launch_conv_fwd<64, 64, kPool>(Src{ws.a3, nullptr}, W + net_param_offset(3), ws.a4, n4x, n4y, n4z, st);
        if (e == cudaSuccess) e = launch_conv_fwd<64, 32, kUpAdd>(Src{ws.a3, ws.a4}, W + net_param_offset(4), ws.b3, n3x, n3y, n3z, st);
        if (e == cudaSuccess) e = launch_conv_fwd<32, 16, kUpAdd>(Src{ws.a2, ws.b3}, W + net_param_offset(5), ws.b2, n2x, n2y, n2z, st);
    }
    if (e == cudaSuccess) {
        dim3 grid((n2x + kOutCX - 1) / kOutCX, (n2y + kOutCY - 1) / kOutCY, n2z);
        static bool configured = false;
        if (!configured) {
            e = cudaFuncSetAttribute(net_out_interior, cudaFuncAttributeMaxDynamicSharedMemorySize, kOutBwinBytes);
            if (e != cudaSuccess) return e;
            configured = true;
        }
        net_out_interior<<<grid, kOutCX * kOutCY, kOutBwinBytes, st>>>(r, ws.b2, w.upfrag, ws.scalars, h2, z, nx,
                                                                       ny, nz, w.out_params);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) {
        const long long faces = 2LL * nx * ny + 2LL * nx * (nz - 2) + 2LL * (ny - 2) * (nz - 2);
        net_out_boundary<<<std::min(grid_1d(faces), 148 * 4), 256, 0, st>>>(r, w.fused, ws.scalars, h2, z, nx, ny, nz);
        e = cudaGetLastError();
    }
    return e;
}

cudaError_t net_train_sample(const NetWeights &w, NetWorkspace &ws, int nx, int ny, int nz, const float *b_hat,
                             const float *p_hat, double norm, int loss_kind, float *grad, double *loss,
                             cudaStream_t st) {
    if (nx % 8 || ny % 8 || nz % 8) return cudaErrorInvalidValue;
    cudaError_t e = ws.ensure(nx, ny, nz, true);
    if (e != cudaSuccess) return e;
    const long long n = (long long)nx * ny * nz;
    const int n2x = nx / 2, n2y = ny / 2, n2z = nz / 2, n3x = nx / 4, n3y = ny / 4, n3z = nz / 4;
    const int n4x = nx / 8, n4y = ny / 8, n4z = nz / 8;
    const uint16_t *W = w.fwd, *Wb = w.bwd;
    auto off = [](int l) { return net_param_offset(l); };
    // ---- forward, every input tensor materialised ----
    conv_first<<<grid_1d(n), 256, 0, st>>>(b_hat, w.fwd_f32, nullptr, ws.a1, nullptr, nx, ny, nz);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = pool_any(16, ws.a1, ws.x2, n2x, n2y, n2z, 0.125f, st);
    if (e == cudaSuccess) e = launch_conv<16, 32, kPlain>(Src{ws.x2, nullptr}, W + off(1), ws.a2, n2x, n2y, n2z, st);
    if (e == cudaSuccess) e = pool_any(32, ws.a2, ws.x3, n3x, n3y, n3z, 0.125f, st);
    if (e == cudaSuccess) e = launch_conv<32, 64, kPlain>(Src{ws.x3, nullptr}, W + off(2), ws.a3, n3x, n3y, n3z, st);
    if (e == cudaSuccess) e = pool_any(64, ws.a3, ws.x4, n4x, n4y, n4z, 0.125f, st);
    if (e == cudaSuccess) e = launch_conv<64, 64, kPlain>(Src{ws.x4, nullptr}, W + off(3), ws.a4, n4x, n4y, n4z, st);
    if (e == cudaSuccess) e = upadd_any(64, ws.a4, ws.a3, ws.x5, n3x, n3y, n3z, 1.f, 0, st);
    if (e == cudaSuccess) e = launch_conv<64, 32, kPlain>(Src{ws.x5, nullptr}, W + off(4), ws.b3, n3x, n3y, n3z, st);
    if (e == cudaSuccess) e = upadd_any(32, ws.b3, ws.a2, ws.x6, n2x, n2y, n2z, 1.f, 0, st);
    if (e == cudaSuccess) e = launch_conv<32, 16, kPlain>(Src{ws.x6, nullptr}, W + off(5), ws.b2, n2x, n2y, n2z, st);
    if (e == cudaSuccess) e = upadd_any(16, ws.b2, ws.a1, ws.x7, nx, ny, nz, 1.f, 0, st);
    if (e == cudaSuccess) {
        dim3 grid((nx + kTX - 1) / kTX, (ny + kTY - 1) / kTY, nz);
        conv_last<kPlain><<<grid, kTX * kTY, 0, st>>>(Src{ws.x7, nullptr}, w.fwd_f32 + 432, nullptr, 1.0, ws.out32, nx,
                                                      ny, nz, 0);
        e = cudaGetLastError();
    }
    // ---- loss and dL/d(output) ----
    if (e == cudaSuccess) {
        loss_err<<<grid_1d(n), 256, 0, st>>>(ws.out32, p_hat, ws.out32, n);  // out32 := e
        if (loss_kind == kNetLossResidual) {
            loss_res_kernel<<<grid_1d(n), 256, 0, st>>>(ws.out32, ws.lq, 1.0 / norm, loss, nx, ny, nz);
            loss_res_grad<<<grid_1d(n), 256, 0, st>>>(ws.lq, ws.gout, 1.0 / norm, nx, ny, nz);
        } else {
            loss_kernel<<<grid_1d(n), 256, 0, st>>>(ws.out32, ws.gout, 1.0 / norm, loss, nx, ny, nz);
        }
        e = cudaGetLastError();
    }
    // ---- backward: weight gradient of each layer, then its data gradient ----
    if (e == cudaSuccess) e = launch_wgrad_scalar<false>(ws.x7, ws.gout, grad + off(6), nx, ny, nz, st);
    if (e == cudaSuccess) {
        conv_first<<<grid_1d(n), 256, 0, st>>>(ws.gout, w.fwd_f32 + 864, nullptr, ws.g7, nullptr, nx, ny, nz);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = pool_any(16, ws.g7, ws.gb2, n2x, n2y, n2z, 1.f, st);
    if (e == cudaSuccess) e = launch_wgrad<32, 16>(ws.x6, ws.gb2, grad + off(5), n2x, n2y, n2z, st);
    if (e == cudaSuccess) e = launch_conv<16, 32, kPlain>(Src{ws.gb2, nullptr}, Wb + off(5), ws.g6, n2x, n2y, n2z, st);
    if (e == cudaSuccess) e = pool_any(32, ws.g6, ws.gb3, n3x, n3y, n3z, 1.f, st);
    if (e == cudaSuccess) e = launch_wgrad<64, 32>(ws.x5, ws.gb3, grad + off(4), n3x, n3y, n3z, st);
    if (e == cudaSuccess) e = launch_conv<32, 64, kPlain>(Src{ws.gb3, nullptr}, Wb + off(4), ws.g5, n3x, n3y, n3z, st);
    if (e == cudaSuccess) e = pool_any(64, ws.g5, ws.ga4, n4x, n4y, n4z, 1.f, st);
    if (e == cudaSuccess) e = launch_wgrad<64, 64>(ws.x4, ws.ga4, grad + off(3), n4x, n4y, n4z, st);
    if (e == cudaSuccess) e = launch_conv<64, 64, kPlain>(Src{ws.ga4, nullptr}, Wb + off(3), ws.g4, n4x, n4y, n4z, st);
    if (e == cudaSuccess) e = upadd_any(64, ws.g4, ws.ga3, ws.ga3, n3x, n3y, n3z, 0.125f, 1, st);
    if (e == cudaSuccess) e = launch_wgrad<32, 64>(ws.x3, ws.ga3, grad + off(2), n3x, n3y, n3z, st);
    if (e == cudaSuccess) e = launch_conv<64, 32, kPlain>(Src{ws.ga3, nullptr}, Wb + off(2), ws.g3, n3x, n3y, n3z, st);
    if (e == cudaSuccess) e = upadd_any(32, ws.g3, ws.ga2, ws.ga2, n2x, n2y, n2z, 0.125f, 1, st);
    if (e == cudaSuccess) e = launch_wgrad<16, 32>(ws.x2, ws.ga2, grad + off(1), n2x, n2y, n2z, st);
    if (e == cudaSuccess) e = launch_conv<32, 16, kPlain>(Src{ws.ga2, nullptr}, Wb + off(1), ws.g2, n2x, n2y, n2z, st);
    if (e == cudaSuccess) e = upadd_any(16, ws.g2, ws.ga1, ws.ga1, nx, ny, nz, 0.125f, 1, st);
    if (e == cudaSuccess) e = launch_wgrad_scalar<true>(ws.ga1, b_hat, grad + off(0), nx, ny, nz, st);
    return e;
}

cudaError_t net_adam(float *w, const float *g, float *m, float *v, long long n, float lr, float beta1, float beta2,
                     float eps, long long t, float grad_scale, cudaStream_t st) {
    const float c1 = 1.f - powf(beta1, float(t)), c2 = 1.f - powf(beta2, float(t));
    adam_kernel<<<grid_1d(n), 256, 0, st>>>(w, g, m, v, n, lr, beta1, beta2, eps, c1, c2, grad_scale);
    return cudaGetLastError();
}

}  // namespace flursys
