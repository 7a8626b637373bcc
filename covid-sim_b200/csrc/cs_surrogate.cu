// Scenario surrogate: a small network mapping 8 intervention/transmission
// parameters to 365 days x 4 daily outputs, trained on trajectories of the GPU
// simulator and used to screen scenario sweeps.  No counterpart in the
// reference, which has no learned model; the layer definitions follow
// oracle/surrogate_ref.py, which the tests use as the reference.
//
//   x [B, 8] -> 4 x (Linear 512 + ReLU) -> Linear 256 + ReLU -> Linear 2944 + ReLU
//   -> [B, 46, 64] -> 3 x (nearest upsample x2 -> Conv1d k=5 pad 2) 64 -> 64 -> 32 -> 4
//      (ReLU after the first two) -> first 365 time points -> y [B, 365, 4]
//
// Every matrix product (the linear layers, and the convolutions as products of
// im2col columns with the weights) runs on the tensor cores in BF16 with FP32
// accumulation: C[M,N] = A[M,K] * B[N,K]^T, both operands row-major BF16 with
// every dimension padded to a multiple of 64 (pads hold zeros, so they add
// nothing).  Master weights, gradients and Adam moments are FP32; the BF16
// weight copies are refreshed after each update.  Gradients are deterministic:
// every reduction has a fixed order.
#include <cuda_runtime.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <thread>
#include <vector>

#include "covidsim_b200.h"

typedef __nv_bfloat16 bf16;

namespace sur {

constexpr int kIn = 8, kWidth = 512, kLatent = 256, kT0 = 46, kC0 = 64, kTap = 5;
constexpr int kTOut = 365, kNOut = 4, kCh = 64;   // conv activations keep 64 channel slots

inline int up64(int x) { return (x + 63) / 64 * 64; }

// ------------------------------------------------------------------- GEMM
// C[M,N] = A[M,K] * B[N,K]^T (+ bias[n]) (ReLU), FP32 out and/or BF16 out.
// M, N multiples of 64; K multiple of 32; leading dimensions multiples of 8.
// 128 threads: a 2 x 2 grid of warps, each a 32 x 32 tile of m16n8k16 products.
__device__ __forceinline__ void mma_bf16(float c[4], const uint32_t a[4], const uint32_t b[2])
{
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 "
        "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// Split K (gridDim.z > 1): slice z covers k in [z * kchunk, min(K, (z + 1) * kchunk))
// and writes its partial product to C + z * cstride (no bias, ReLU or BF16 output).
__global__ void __launch_bounds__(128) k_gemm_nt(const bf16* __restrict__ A, int lda, const bf16* __restrict__ B, int ldb,
                                                 float* __restrict__ C, int ldc, bf16* __restrict__ Cb, int ldcb,
                                                 const float* __restrict__ bias, int relu, int K, int kchunk, size_t cstride,
                                                 const bf16* __restrict__ mask)
{
    if (gridDim.z > 1) {
        const int z = blockIdx.z;
        A += (size_t)z * kchunk;
        B += (size_t)z * kchunk;
        C += (size_t)z * cstride;
        K = min(kchunk, K - z * kchunk);
    }
    __shared__ __align__(16) bf16 As[64][40];
    __shared__ __align__(16) bf16 Bs[64][40];
    const int bm = blockIdx.y * 64, bn = blockIdx.x * 64;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32;
    const int g = lane >> 2, tq = lane & 3;
    float acc[2][4][4];
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int q = 0; q < 4; q++) acc[i][j][q] = 0.f;
    for (int k0 = 0; k0 < K; k0 += 32) {
        for (int i = threadIdx.x; i < 256; i += 128) {
            int r = i >> 2, c = (i & 3) * 8;
            *reinterpret_cast<uint4*>(&As[r][c]) = *reinterpret_cast<const uint4*>(A + (size_t)(bm + r) * lda + k0 + c);
            *reinterpret_cast<uint4*>(&Bs[r][c]) = *reinterpret_cast<const uint4*>(B + (size_t)(bn + r) * ldb + k0 + c);
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < 32; kk += 16) {
            uint32_t a[2][4], b[4][2];
#pragma unroll
            for (int mi = 0; mi < 2; mi++) {
                int r = wm + mi * 16 + g;
                a[mi][0] = *reinterpret_cast<const uint32_t*>(&As[r][kk + tq * 2]);
                a[mi][1] = *reinterpret_cast<const uint32_t*>(&As[r + 8][kk + tq * 2]);
                a[mi][2] = *reinterpret_cast<const uint32_t*>(&As[r][kk + tq * 2 + 8]);
                a[mi][3] = *reinterpret_cast<const uint32_t*>(&As[r + 8][kk + tq * 2 + 8]);
            }
#pragma unroll
            for (int ni = 0; ni < 4; ni++) {
                int n = wn + ni * 8 + g;
                b[ni][0] = *reinterpret_cast<const uint32_t*>(&Bs[n][kk + tq * 2]);
                b[ni][1] = *reinterpret_cast<const uint32_t*>(&Bs[n][kk + tq * 2 + 8]);
            }
#pragma unroll
            for (int mi = 0; mi < 2; mi++)
#pragma unroll
                for (int ni = 0; ni < 4; ni++) mma_bf16(acc[mi][ni], a[mi], b[ni]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int mi = 0; mi < 2; mi++)
#pragma unroll
        for (int ni = 0; ni < 4; ni++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                int r = bm + wm + mi * 16 + g + h * 8;
                int c = bn + wn + ni * 8 + tq * 2;
                float v0 = acc[mi][ni][2 * h], v1 = acc[mi][ni][2 * h + 1];
                if (bias) { v0 += bias[c]; v1 += bias[c + 1]; }
                if (relu) { v0 = fmaxf(v0, 0.f); v1 = fmaxf(v1, 0.f); }
                if (mask) {
                    if (!(__bfloat162float(mask[(size_t)r * ldc + c]) > 0.f)) v0 = 0.f;
                    if (!(__bfloat162float(mask[(size_t)r * ldc + c + 1]) > 0.f)) v1 = 0.f;
                }
                if (C) { C[(size_t)r * ldc + c] = v0; C[(size_t)r * ldc + c + 1] = v1; }
                if (Cb) *reinterpret_cast<__nv_bfloat162*>(Cb + (size_t)r * ldcb + c) = __floats2bfloat162_rn(v0, v1);
            }
}

// ------------------------------------------------------- tcgen05 GEMM
// The same product on the 5th-generation tensor cores.  A block computes a 128 x BN
// tile: its 128 threads copy 64-wide K slices of A and B into shared memory in the
// K-major 128-byte-swizzled layout (cp.async, kStages - 1 slices ahead of the products),
// one thread issues the tcgen05.mma instructions (M = 128, N = BN, K = 16 each, BF16 in,
// FP32 accumulator in tensor memory) and commits them to the stage's mbarrier, and after
// the last slice every warp reads its 32 accumulator rows from tensor memory for the
// epilogue (bias, ReLU, mask, FP32 and/or BF16 stores, 16 bytes each).  Rows of A past M are staged as zeros and not stored.
// Every wait is bounded: on a give-up the block records it in *err, waits (bounded)
// for its issued products, frees its tensor memory and returns.
namespace tc {

constexpr int BM = 128, BK = 64;          // BK bf16 = 128 bytes, one swizzle row
constexpr unsigned kSpin = 1u << 22;      // try_wait rounds before a wait gives up

__host__ __device__ constexpr size_t smem_bytes(int BN, int stages) { return 1024 + stages * (size_t)(BM + BN) * BK * 2; }

__device__ __forceinline__ uint32_t saddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Shared-memory matrix descriptor of a K-major, 128-byte-swizzled operand: start
// address, leading offset 16 B (unused by this layout), 8-row groups 1024 B apart,
// descriptor version 1, layout SWIZZLE_128B.
__device__ __forceinline__ uint64_t sdesc(uint32_t addr)
{
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) |
           ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

// Instruction descriptor of kind::f16: FP32 accumulator, BF16 A and B, both K-major.
__host__ __device__ constexpr uint32_t idesc(int M, int N)
{
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ bool mbar_try(uint64_t* bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(ok) : "r"(saddr(bar)), "r"(parity) : "memory");
    return ok != 0;
}

__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity)
{
    for (unsigned i = 0; i < kSpin; i++)
        if (mbar_try(bar, parity)) return true;
    return false;
}

__device__ __forceinline__ void mma(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t id, uint32_t accumulate)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
                 :: "r"(d_tmem), "l"(a), "l"(b), "r"(id), "r"(accumulate) : "memory");
}

__device__ __forceinline__ void commit(uint64_t* bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(saddr(bar)) : "memory");
}

__device__ __forceinline__ void ld32(uint32_t taddr, uint32_t (&r)[32])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                 "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
                 "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                   "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                   "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// 16 bytes into shared memory, or zeros.
__device__ __forceinline__ void copy16(uint32_t dst, const bf16* src, bool valid)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
}

// A thread's 16-byte chunks of a rows x 64 slice (128-byte-swizzled: chunk j of row r lands
// at r * 128 + ((j ^ (r & 7)) * 16)): chunk j = threadIdx & 7 of every 16th row, the same j
// for all, so what depends on the row is formed once per tile and what depends on k once per
// slice.
template <int kRows>
struct RowSource {   // rows of a row-major matrix; rows at or past nrows are zero
    static constexpr int kN = kRows / 16;
    const bf16 *base, *p;   // base: an address to name where nothing is read
    int ld, left;
    __device__ __forceinline__ RowSource(const bf16* src, int ld_, int r0, int nrows)
        : base(src), p(src + (size_t)(r0 + (int)(threadIdx.x >> 3)) * ld_ + (threadIdx.x & 7) * 8), ld(ld_), left(nrows - r0 - (int)(threadIdx.x >> 3)) {}
    __device__ __forceinline__ void stage(uint32_t dst, int k0) const
    {
        const int r = threadIdx.x >> 3, j = threadIdx.x & 7;
        dst += r * 128 + ((j ^ (r & 7)) << 4);   // r + 16 q has the same low bits
#pragma unroll
        for (int q = 0; q < kN; q++) copy16(dst + q * 2048, 16 * q < left ? p + (size_t)(16 * q) * ld + k0 : base, 16 * q < left);
    }
};

// The A operand of a convolution read straight from its input H [Bn*T, kCh] (no
// column matrix): row m = b*2T + t, column k = tap*Cin + c holds
// H[b*T + (t+tap-2)/2, c] when 0 <= t+tap-2 < 2T, else zero (as k_im2col_up).  Cin is
// a multiple of 8, so a 16-byte chunk never straddles two taps.
struct ConvSource {
    static constexpr int kN = BM / 16;
    const bf16* H;
    int T, Cin, nrows, m0;
    int b[kN], t[kN];
    __device__ __forceinline__ ConvSource(const bf16* H_, int T_, int Cin_, int r0, int nrows_)
        : H(H_), T(T_), Cin(Cin_), nrows(nrows_), m0(r0 + (int)(threadIdx.x >> 3))
    {
#pragma unroll
        for (int q = 0; q < kN; q++) {
            b[q] = (m0 + 16 * q) / (2 * T);
            t[q] = m0 + 16 * q - b[q] * 2 * T;
        }
    }
    __device__ __forceinline__ void stage(uint32_t dst, int k0) const
    {
        const int r = threadIdx.x >> 3, j = threadIdx.x & 7, k = k0 + j * 8, tap = k / Cin, c = k - tap * Cin;
        dst += r * 128 + ((j ^ (r & 7)) << 4);
#pragma unroll
        for (int q = 0; q < kN; q++) {
            const int u = t[q] + tap - kTap / 2;
            const bool on = m0 + 16 * q < nrows && tap < kTap && u >= 0 && u < 2 * T;
            copy16(dst + q * 2048, on ? H + ((size_t)b[q] * T + (u >> 1)) * kCh + c : H, on);
        }
    }
};

}  // namespace tc

// mask (leading dimension ldc, may be null): outputs where it is not positive are zero, the
// backward ReLU of the activation it holds.
// C[M,N] = A[M,K] B[N,K]^T (+ bias) (ReLU) on tcgen05; N a multiple of BN, K of 64;
// split K as k_gemm_nt (gridDim.z slices of kchunk, partial products at C + z * cstride).
// With H set, A is the column matrix of a convolution of H (hT time points, hCin
// channels), generated while staging (not split).
template <int BN, int kStages>
__global__ void __launch_bounds__(128) k_gemm_tc(const bf16* __restrict__ A, int lda, const bf16* __restrict__ B, int ldb,
                                                 float* __restrict__ C, int ldc, bf16* __restrict__ Cb, int ldcb,
                                                 const float* __restrict__ bias, int relu, int M, int K, int kchunk,
                                                 size_t cstride, int* err, const bf16* __restrict__ H, int hT, int hCin,
                                                 const bf16* __restrict__ mask, float* __restrict__ Y, int yn)
{
    using namespace tc;
    constexpr int kCols = BN < 32 ? 32 : BN;   // tensor memory comes in 32 columns at least
    constexpr int kW = BN < 32 ? BN : 32;      // columns of a 32-column read that hold outputs
    extern __shared__ unsigned char smem_raw[];
    __shared__ uint64_t bar[kStages];
    __shared__ uint32_t tmem_base;
    __shared__ int s_ok;
    const uint32_t As = (saddr(smem_raw) + 1023) & ~1023u;   // [kStages][BM * 128 B]
    const uint32_t Bs = As + kStages * BM * BK * 2;          // [kStages][BN * 128 B]
    if (gridDim.z > 1) {
        const int z = blockIdx.z;
        A += (size_t)z * kchunk;
        B += (size_t)z * kchunk;
        C += (size_t)z * cstride;
        K = min(kchunk, K - z * kchunk);
    }
    const int bm = blockIdx.y * BM, bn = blockIdx.x * BN;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nk = K / BK;
    const RowSource<BM> arows(H ? B : A, H ? 0 : lda, H ? 0 : bm, H ? 0 : M);
    const ConvSource aconv(H, H ? hT : 1, H ? hCin : 64, bm, H ? M : 0);
    const RowSource<BN> brows(B, ldb, bn, 1 << 30);
    auto load = [&](int kc) {   // slice kc on its way (an empty group past the last, so that groups count slices)
        if (kc < nk) {
            const uint32_t st = kc % kStages;
            if (H) aconv.stage(As + st * BM * 128, kc * BK);
            else arows.stage(As + st * BM * 128, kc * BK);
            brows.stage(Bs + st * BN * 128, kc * BK);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int kc = 0; kc < kStages - 1; kc++) load(kc);
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(saddr(&tmem_base)), "r"(kCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (threadIdx.x == 0) {
#pragma unroll
        for (int i = 0; i < kStages; i++) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(saddr(&bar[i])));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        s_ok = 1;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tm = tmem_base;
    int issued = 0;                    // slices whose products were committed
    bool ok = true;                    // this thread's waits came through
    for (int kc = 0; kc < nk; kc++) {
        const int st = kc % kStages;
        asm volatile("cp.async.wait_group %0;" :: "n"(kStages - 2) : "memory");   // slice kc is in
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        if (!__syncthreads_and(ok)) break;
        if (threadIdx.x == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t a0 = As + st * BM * 128, b0 = Bs + st * BN * 128;
#pragma unroll
            for (int k = 0; k < BK / 16; k++)
                tc::mma(tm, sdesc(a0 + 32 * k), sdesc(b0 + 32 * k), idesc(BM, BN), (kc | k) != 0);
            commit(&bar[st]);
        }
        issued = kc + 1;
        // the next slice to fetch goes where slice kc - 1 was, once its products are done
        if (kc >= 1 && kc + kStages - 1 < nk) ok = mbar_wait(&bar[(kc - 1) % kStages], ((kc - 1) / kStages) & 1);
        if (ok) load(kc + kStages - 1);
        else asm volatile("cp.async.commit_group;" ::: "memory");
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    // the last committed slice's barrier completes after all earlier products
    if (threadIdx.x == 0 && issued > 0 && !mbar_wait(&bar[(issued - 1) % kStages], ((issued - 1) / kStages) & 1)) s_ok = 0;
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (s_ok && issued == nk) {
        const int row = bm + warp * 32 + lane;
#pragma unroll 1
        for (int c0 = 0; c0 < BN; c0 += 32) {
            uint32_t r[32];
            ld32(tm + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0, r);
            if (row < M) {
                const int col = bn + c0;
                float v[kW];
#pragma unroll
                for (int j = 0; j < kW; j++) v[j] = nk == 0 ? 0.f : __uint_as_float(r[j]);
                if (bias) {
#pragma unroll
                    for (int j = 0; j < kW; j++) v[j] += bias[col + j];
                }
                if (relu) {
#pragma unroll
                    for (int j = 0; j < kW; j++) v[j] = fmaxf(v[j], 0.f);
                }
                if (mask) {
#pragma unroll
                    for (int j = 0; j < kW; j += 8) {
                        const uint4 h4 = *reinterpret_cast<const uint4*>(mask + (size_t)row * ldc + col + j);
                        const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&h4);
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            if (!(__low2float(h[q]) > 0.f)) v[j + 2 * q] = 0.f;
                            if (!(__high2float(h[q]) > 0.f)) v[j + 2 * q + 1] = 0.f;
                        }
                    }
                }
                if (Y && bn + c0 == 0) {   // the network's outputs: [yn, 365, 4] from [yn * 368, ...]
                    const int yb = row / (8 * kT0), yt = row - yb * (8 * kT0);
                    if (yb < yn && yt < kTOut) *reinterpret_cast<float4*>(Y + ((size_t)yb * kTOut + yt) * kNOut) = make_float4(v[0], v[1], v[2], v[3]);
                }
                if (C) {
#pragma unroll
                    for (int j = 0; j < kW; j += 4)
                        *reinterpret_cast<float4*>(C + (size_t)row * ldc + col + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
                }
                if (Cb) {
#pragma unroll
                    for (int j = 0; j < kW; j += 8) {
                        uint4 o4;
                        __nv_bfloat162* o = reinterpret_cast<__nv_bfloat162*>(&o4);
#pragma unroll
                        for (int q = 0; q < 4; q++) o[q] = __floats2bfloat162_rn(v[j + 2 * q], v[j + 2 * q + 1]);
                        *reinterpret_cast<uint4*>(Cb + (size_t)row * ldcb + col + j) = o4;
                    }
                }
            }
        }
    } else if (threadIdx.x == 0) {
        atomicExch(err, 1);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tm), "r"(kCols));
}

// Stages: four put a short product's whole K in flight at once (the linear layers: 64 to 512
// wide, split); with more blocks than two an SM, two leave room for four blocks an SM, which
// hide one another's loads.  BN: the output columns that are there (64, or 32 and 16 for the
// last two convolutions' 32 and 4 channels, whose padding to 64 was product work for nothing).
static int tc_stages(const dim3& grid) { return (size_t)grid.x * grid.y * grid.z <= 296 ? 4 : 2; }
template <int BN, typename... Args>
static void tc_launch(const dim3& grid, cudaStream_t st, Args... args)
{
    if (tc_stages(grid) == 4) k_gemm_tc<BN, 4><<<grid, 128, tc::smem_bytes(BN, 4), st>>>(args...);
    else k_gemm_tc<BN, 2><<<grid, 128, tc::smem_bytes(BN, 2), st>>>(args...);
}
template <int BN>
static cudaError_t tc_enable()
{
    cudaError_t e = cudaFuncSetAttribute(k_gemm_tc<BN, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tc::smem_bytes(BN, 4));
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_gemm_tc<BN, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tc::smem_bytes(BN, 2));
    return e;
}

// C[r, c] = sum over the slices z, in ascending order, of part[z][r, c] ([M, N] each),
// then the product's epilogue (bias, ReLU, FP32 and/or BF16 stores).
__global__ void k_splitk_reduce(const float* __restrict__ part, int nsplit, int M, int N, float* __restrict__ C, int ldc,
                                bf16* __restrict__ Cb, int ldcb, const float* __restrict__ bias, int relu,
                                const bf16* __restrict__ mask)
{
    const size_t MN = (size_t)M * N;
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < MN; e += (size_t)gridDim.x * blockDim.x) {
        float acc = 0.f;
        for (int z = 0; z < nsplit; z++) acc += part[z * MN + e];
        const size_t r = e / N, c = e % N;
        if (bias) acc += bias[c];
        if (relu) acc = fmaxf(acc, 0.f);
        if (mask && !(__bfloat162float(mask[r * ldc + c]) > 0.f)) acc = 0.f;
        if (C) C[r * ldc + c] = acc;
        if (Cb) Cb[r * ldcb + c] = __float2bfloat16_rn(acc);
    }
}

// out[c, r] = in[r, c] for an R x Cc block (both multiples of 32).
__global__ void k_transpose(const bf16* __restrict__ in, int ldi, bf16* __restrict__ out, int ldo, int R, int Cc)
{
    __shared__ bf16 t[32][33];
    int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
    for (int i = threadIdx.y; i < 32; i += blockDim.y) t[i][threadIdx.x] = in[(size_t)(r0 + i) * ldi + c0 + threadIdx.x];
    __syncthreads();
    for (int i = threadIdx.y; i < 32; i += blockDim.y) out[(size_t)(c0 + i) * ldo + r0 + threadIdx.x] = t[threadIdx.x][i];
}

// Columns of the x2 upsampled, zero-padded input: cols[b*2T + t, k*Cin + c] =
// H[b*T + (t+k-2)/2, c] for 0 <= t+k-2 < 2T (channel stride kCh), zero elsewhere
// (and in the pad columns up to ldc).
__global__ void k_im2col_up(const bf16* __restrict__ H, int Bn, int T, int Cin, bf16* __restrict__ cols, int ldc)
{
    const size_t rows = (size_t)Bn * 2 * T;
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < rows * ldc; e += (size_t)gridDim.x * blockDim.x) {
        size_t row = e / ldc;
        int col = (int)(e % ldc);
        bf16 v = __float2bfloat16(0.f);
        if (col < kTap * Cin) {
            int k = col / Cin, c = col % Cin;
            int b = (int)(row / (2 * T)), t = (int)(row % (2 * T));
            int u = t + k - kTap / 2;
            if (u >= 0 && u < 2 * T) v = H[((size_t)b * T + (u >> 1)) * kCh + c];
        }
        cols[e] = v;
    }
}

// The transposed column matrix, colsT[k, m] = cols[m, k] of k_im2col_up, for m < M
// (= Bn*2T, a multiple of 64) and k < ldk (columns past kTap*Cin zero), through a shared tile
// of 32 k by 64 m: a thread reads 8 channels of one tap and writes 8 time points of one
// column, 16 bytes each.  Bound: the matrix' writes (36 MB for 256 rows' last convolution);
// 2 bytes an access took 66 us for that (with the products beside it), now 22.
__global__ void __launch_bounds__(256) k_im2colT_up(const bf16* __restrict__ H, int T, int Cin, bf16* __restrict__ colsT, int M)
{
    __shared__ __align__(16) bf16 tile[32][72];   // rows of 144 B: 16-byte reads, neighbouring columns in other banks
    const int m0 = blockIdx.y * 64, k0 = blockIdx.x * 32;
    {
        const int i = threadIdx.x & 63, m = m0 + i, k = k0 + 8 * (threadIdx.x >> 6), tap = k / Cin;
        union { uint4 q; bf16 h[8]; } u;
        u.q = make_uint4(0, 0, 0, 0);
        if (tap < kTap) {
            const int b = m / (2 * T), t = m - b * 2 * T, v = t + tap - kTap / 2;
            if (v >= 0 && v < 2 * T) u.q = *reinterpret_cast<const uint4*>(H + ((size_t)b * T + (v >> 1)) * kCh + (k - tap * Cin));
        }
#pragma unroll
        for (int j = 0; j < 8; j++) tile[k - k0 + j][i] = u.h[j];
    }
    __syncthreads();
    const int r = threadIdx.x >> 3, c = 8 * (threadIdx.x & 7);
    *reinterpret_cast<uint4*>(colsT + (size_t)(k0 + r) * M + m0 + c) = *reinterpret_cast<const uint4*>(&tile[r][c]);
}

// Adjoint of k_im2col_up, fused with the ReLU mask of H: for channel c < Cin,
// dz[b*T+s, c] = (H > 0) * sum over u in {2s, 2s+1}, k of dcols[b*2T + u-k+2, k*Cin + c];
// FP32 and BF16 copies; channels >= Cin are zero from the start and stay so.
__global__ void k_col2im_up_relu(const float* __restrict__ dcols, int ldd, int Bn, int T, int Cin,
                                 const bf16* __restrict__ H, float* __restrict__ dz, bf16* __restrict__ dzb)
{
    const size_t n = (size_t)Bn * T * Cin;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const int c = (int)(i % Cin);
        const size_t bs = i / Cin, e = bs * kCh + c;
        int b = (int)(bs / T), s = (int)(bs % T);
        float acc = 0.f;
        for (int du = 0; du < 2; du++) {
            int u = 2 * s + du;
            for (int k = 0; k < kTap; k++) {
                int t = u - k + kTap / 2;
                if (t >= 0 && t < 2 * T) acc += dcols[((size_t)b * 2 * T + t) * ldd + k * Cin + c];
            }
        }
        if (!(__bfloat162float(H[e]) > 0.f)) acc = 0.f;
        dz[e] = acc;
        dzb[e] = __float2bfloat16(acc);
    }
}

// Column sums of dz [rows, ld] in a fixed order: part[chunk, col] over row chunks
// of 256, then the chunks in ascending order.
// Column sums of dz [rows, ld] in a fixed order.  Block (x, y) covers 32 columns
// and row chunk y of kColChunk rows; its 8 row lanes each sum every 8th row, then
// a shared-memory tree adds the lanes: part[y, col].  The final pass adds the
// chunks the same way.
constexpr int kColChunk = 2048;
__device__ __forceinline__ float lanes_tree(float v, float (*sh)[33])
{
    sh[threadIdx.y][threadIdx.x] = v;
    __syncthreads();
    for (int o = 4; o > 0; o >>= 1) {
        if ((int)threadIdx.y < o) sh[threadIdx.y][threadIdx.x] += sh[threadIdx.y + o][threadIdx.x];
        __syncthreads();
    }
    return sh[0][threadIdx.x];
}
__global__ void k_colsum_part(const float* __restrict__ dz, int rows, int ld, float* __restrict__ part)
{
    // Bound: the latency of the loads; 16 rows of a thread are on their way at once (and added
    // one by one, in order).  256 rows' three convolutions, with the products beside them:
    // 52 + 38 + 33 us four at a time, at most 39 + 20 + 20 now.
    constexpr int kAhead = 16;
    __shared__ float sh[8][33];
    const int col = blockIdx.x * 32 + threadIdx.x;
    const int r0 = blockIdx.y * kColChunk, r1 = min(rows, r0 + kColChunk);
    float v = 0.f;
    if (col < ld) {
        int r = r0 + threadIdx.y;
        for (; r + 8 * (kAhead - 1) < r1; r += 8 * kAhead) {
            float x[kAhead];
#pragma unroll
            for (int q = 0; q < kAhead; q++) x[q] = dz[(size_t)(r + 8 * q) * ld + col];
#pragma unroll
            for (int q = 0; q < kAhead; q++) v += x[q];
        }
        for (; r < r1; r += 8) v += dz[(size_t)r * ld + col];
    }
    v = lanes_tree(v, sh);
    if (threadIdx.y == 0 && col < ld) part[(size_t)blockIdx.y * ld + col] = v;
}
__global__ void k_colsum_final(const float* __restrict__ part, int nchunks, int ld, float* __restrict__ out)
{
    __shared__ float sh[8][33];
    const int col = blockIdx.x * 32 + threadIdx.x;
    float v = 0.f;
    if (col < ld)
        for (int q = threadIdx.y; q < nchunks; q += 8) v += part[(size_t)q * ld + col];
    v = lanes_tree(v, sh);
    if (threadIdx.y == 0 && col < ld) out[col] = v;
}

// Loss terms and the output gradient (FP32 and BF16): y is [B*368, 64] (channels < 4 used), target
// [n, 365, 4]; rows of samples >= n and time points >= 365 get zero gradient.  A thread per
// row, its four channels in one access; the gradients' other channels are zero from the
// start and stay so.  (All 64 written: 21 us for 256 rows, now 7.)
__global__ void k_mse(const float* __restrict__ y, const float* __restrict__ target, int n, int Bp, float scale,
                      float* __restrict__ dy, bf16* __restrict__ dyb, float* __restrict__ sq)
{
    static_assert(kNOut == 4, "a row's outputs are one 16-byte access");
    const int T = 2 * 2 * 2 * kT0;   // 368
    const size_t total = (size_t)Bp * T;
    for (size_t bt = blockIdx.x * (size_t)blockDim.x + threadIdx.x; bt < total; bt += (size_t)gridDim.x * blockDim.x) {
        const int b = (int)(bt / T), t = (int)(bt % T);
        union F4 { float4 q; float f[4]; };
        F4 g;
        g.q = make_float4(0.f, 0.f, 0.f, 0.f);
        if (t < kTOut && b < n) {
            const size_t at = ((size_t)b * kTOut + t) * kNOut;
            F4 yv, tv, s2;
            yv.q = *reinterpret_cast<const float4*>(y + bt * kCh);
            tv.q = *reinterpret_cast<const float4*>(target + at);
#pragma unroll
            for (int c = 0; c < kNOut; c++) {
                const float d = yv.f[c] - tv.f[c];
                g.f[c] = 2.f * d * scale;
                s2.f[c] = d * d;
            }
            *reinterpret_cast<float4*>(sq + at) = s2.q;
        }
        *reinterpret_cast<float4*>(dy + bt * kCh) = g.q;
        union { uint2 q; bf16 h[4]; } gb;
#pragma unroll
        for (int c = 0; c < kNOut; c++) gb.h[c] = __float2bfloat16(g.f[c]);
        *reinterpret_cast<uint2*>(dyb + bt * kCh) = gb.q;
    }
}

// Adam (Kingma & Ba, 2015) on FP32 master weights; refreshes the BF16 copy.
// Sum of v[0..n) in a fixed order: block b sums its contiguous range (strided by
// thread, then a shared-memory tree), the final pass adds the blocks in order.
__global__ void k_sum_part(const float* __restrict__ v, size_t n, double* __restrict__ part)
{
    __shared__ double sh[256];
    const size_t per = (n + gridDim.x - 1) / gridDim.x, b0 = blockIdx.x * per, e0 = min(n, b0 + per);
    double acc = 0.0;
    for (size_t e = b0 + threadIdx.x; e < e0; e += blockDim.x) acc += v[e];
    sh[threadIdx.x] = acc;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) part[blockIdx.x] = sh[0];
}
__global__ void k_sum_final(const double* __restrict__ part, int n, double* __restrict__ out)
{
    __shared__ double sh[256];
    double a = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) a += part[i];
    sh[threadIdx.x] = a;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) *out = sh[0];
}

__global__ void k_adam(float* __restrict__ w, float* __restrict__ m, float* __restrict__ v, const float* __restrict__ g,
                       bf16* __restrict__ wb, size_t n, float lr, float b1, float b2, float eps, float c1, float c2, float wd,
                       const int* __restrict__ err)
{
    if (*err) return;   // a product of this step gave up: the weights stay
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) {
        float gi = g[e];
        float mi = b1 * m[e] + (1.f - b1) * gi;
        float vi = b2 * v[e] + (1.f - b2) * gi * gi;
        m[e] = mi;
        v[e] = vi;
        // decoupled weight decay (Loshchilov & Hutter, "Decoupled weight decay regularization", 2019)
        float wi = w[e] * (1.f - lr * wd) - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
        w[e] = wi;
        if (wb) wb[e] = __float2bfloat16(wi);
    }
}

__global__ void k_to_bf16(const float* __restrict__ in, bf16* __restrict__ out, size_t n)
{
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x)
        out[e] = __float2bfloat16(in[e]);
}

// x [n, 8] -> BF16 [Bp, 64] (zeros beyond)
__global__ void k_load_x(const float* __restrict__ x, int n, int Bp, bf16* __restrict__ xb)
{
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < Bp * 64; e += gridDim.x * blockDim.x) {
        int b = e / 64, c = e % 64;
        xb[e] = __float2bfloat16((b < n && c < kIn) ? x[b * kIn + c] : 0.f);
    }
}

// y [B*368, 64] -> out [n, 365, 4]
__global__ void k_store_y(const float* __restrict__ y, int n, float* __restrict__ out)
{
    const int T = 8 * kT0;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n * kTOut * kNOut; e += gridDim.x * blockDim.x) {
        int c = e % kNOut, t = (e / kNOut) % kTOut, b = e / (kNOut * kTOut);
        out[e] = y[((size_t)b * T + t) * kCh + c];
    }
}

}  // namespace sur

using namespace sur;

struct Layer {
    int out, in;        // logical
    int outP, inP;      // padded (64)
    bool conv;
    int T;              // conv: output time points; linear: 0
    int cin;            // conv: input channels (logical)
    bool relu;
    size_t wofs, bofs;  // offsets in the padded parameter arrays
};

// A chain of kernels with scratch of its own.  A training step is four such chains: the
// forward pass and the gradients of the activations (0); the weight gradients, alternate
// layers (1 and 2); the bias gradients, transposed weights and loss (3).
constexpr int kLanes = 4;
struct Lane {
    cudaStream_t st = nullptr;
    cudaEvent_t done = nullptr;
    float* kpart = nullptr;                 // split-K partial products
    size_t kpart_n = 0;
    bf16 *dzT = nullptr, *colsT = nullptr;  // transposed operands of a weight gradient
    float* part = nullptr;                  // column sums
};

struct cs_sur {
    int device = 0;
    int bmax = 0;       // batch capacity (multiple of 64)
    cudaStream_t stream = nullptr;
    char err[512] = {0};
    std::vector<Layer> L;
    size_t np = 0;                          // padded parameter count (weights + biases)
    float *w = nullptr, *m = nullptr, *v = nullptr, *g = nullptr;   // FP32, padded layout
    bf16* wb = nullptr;                     // BF16 weights (and biases, unused)
    long long t = 0;                        // Adam step
    // activations and scratch sized for bmax
    std::vector<bf16*> act;                 // act[0] = input, act[l+1] = output of layer l (BF16)
    float* yout = nullptr;                  // last layer output FP32 [bmax*368, 64]
    std::vector<float*> dz;                 // gradient at layer l's output before its ReLU (FP32, BF16); one per
    std::vector<bf16*> dzb;                 // layer, as a layer's weight gradient runs beside the layers below it
    std::vector<bf16*> wT;                  // transposed BF16 weights per layer
    float* dcols = nullptr;
    bf16* cols = nullptr;                   // column matrix of the mma.sync path: one convolution's at a time, in the
                                            // forward pass, which dcols (of the backward pass) leaves to it
    Lane lane[kLanes];                      // [0] the main chain, the others beside it
    cudaEvent_t fork = nullptr;
    std::vector<cudaEvent_t> dz_ready;      // per layer: its dz is written
    double *lpart = nullptr, *lsum = nullptr;   // loss reduction
    int* d_err = nullptr;                   // set by a tensor-core GEMM whose wait gave up; right behind lsum
    int gemm_impl = 0;                      // 0: tcgen05, 1: mma.sync
    float *xdev = nullptr, *tdev = nullptr, *sq = nullptr;
    struct Predict {                        // the prediction path's workspace (predict_space)
        int rows = 0;
        float* dev = nullptr;               // one allocation; the rest points into it
        std::vector<bf16*> act;
        float *xdev[2] = {}, *ydev[2] = {}, *kpart = nullptr;
        size_t kpart_n = 0;
        cudaStream_t copy = nullptr;
        cudaEvent_t ready[2] = {};
    } pred;
    // one training step (or loss and gradient) of n rows as a graph
    struct StepGraph {
        int n = 0;
        bool update = false;
        cudaGraph_t graph = nullptr;
        cudaGraphExec_t exec = nullptr;
        cudaGraphNode_t adam = nullptr;
        cudaKernelNodeParams adam_params{};
        long long used = 0;                 // the step that used it last
    };
    std::vector<StepGraph> graphs;          // kMaxGraphs batch sizes at most
    struct Missed { int n; bool update; long long at; };
    std::vector<Missed> missed;             // sizes that ran without a graph, and the last step that did
    long long steps = 0;
    void* slab = nullptr;                   // the arrays above (Arrays)
};

static int sur_err(cs_sur* s, int code, const char* fmt, ...)
{
    if (s) {
        va_list ap;
        va_start(ap, fmt);
        vsnprintf(s->err, sizeof(s->err), fmt, ap);
        va_end(ap);
    }
    return code;
}

#define SCK(call)                                                                                  \
    do {                                                                                           \
        cudaError_t e_ = (call);                                                                   \
        if (e_ != cudaSuccess) return sur_err(s, CS_E_CUDA, "%s: %s", #call, cudaGetErrorString(e_)); \
    } while (0)

// A network's arrays, asked for one by one and taken as one allocation, zeroed: some sixty
// allocations of their own made creating a network of 256 rows last 22 ms, 18 with the
// thirty-six that it had before its chains ran side by side, 11 now.
struct Arrays {
    struct Item { void** p; size_t bytes; };
    std::vector<Item> items;
    size_t total = 0;
    template <typename T>
    void add(T*& p, size_t n)
    {
        const size_t bytes = (sizeof(T) * std::max<size_t>(n, 1) + 255) / 256 * 256;
        items.push_back({reinterpret_cast<void**>(&p), bytes});
        total += bytes;
    }
    int take(cs_sur* s)
    {
        const cudaError_t e = cudaMalloc(&s->slab, total);
        if (e != cudaSuccess) return sur_err(s, CS_E_CUDA, "cudaMalloc(%zu bytes): %s", total, cudaGetErrorString(e));
        SCK(cudaMemsetAsync(s->slab, 0, total, s->stream));
        char* at = static_cast<char*>(s->slab);
        for (const Item& it : items) {
            *it.p = at;
            at += it.bytes;
        }
        return CS_OK;
    }
};

static void free_predict(cs_sur* s)
{
    cudaFree(s->pred.dev);
    s->pred.dev = nullptr;
    s->pred.rows = 0;
}

static void drop_graphs(cs_sur* s)
{
    for (auto& g : s->graphs) {
        if (g.exec) cudaGraphExecDestroy(g.exec);
        if (g.graph) cudaGraphDestroy(g.graph);
    }
    s->graphs.clear();
    s->missed.clear();
}

static void build_layers(cs_sur* s)
{
    s->L.clear();
    const int lin[6][2] = {{kWidth, kIn}, {kWidth, kWidth}, {kWidth, kWidth}, {kWidth, kWidth}, {kLatent, kWidth}, {kT0 * kC0, kLatent}};
    size_t ofs = 0;
    for (int i = 0; i < 6; i++) {
        Layer l{lin[i][0], lin[i][1], up64(lin[i][0]), up64(lin[i][1]), false, 0, 0, true, 0, 0};
        l.wofs = ofs; ofs += (size_t)l.outP * l.inP;
        l.bofs = ofs; ofs += l.outP;
        s->L.push_back(l);
    }
    const int conv[3][3] = {{64, 64, 1}, {64, 32, 1}, {32, 4, 0}};
    int T = kT0;
    for (int i = 0; i < 3; i++) {
        T *= 2;
        Layer l{conv[i][1], kTap * conv[i][0], up64(conv[i][1]), up64(kTap * conv[i][0]), true, T, conv[i][0], conv[i][2] != 0, 0, 0};
        l.wofs = ofs; ofs += (size_t)l.outP * l.inP;
        l.bofs = ofs; ofs += l.outP;
        s->L.push_back(l);
    }
    s->np = ofs;
}

constexpr int kLossBlocks = 296;

// One product (or, with nsplit > 1, its K slices of kchunk) on the selected path.
static int gemm_launch(cs_sur* s, const Lane& w, const bf16* A, int lda, const bf16* B, int ldb, float* C, int ldc, bf16* Cb,
                       int ldcb, const float* bias, int relu, int M, int N, int K, int nsplit, int kchunk, size_t cstride,
                       const bf16* mask)
{
    if (s->gemm_impl == 0 && K % 64 == 0 && kchunk % 64 == 0) {
        dim3 grid(N / 64, (M + tc::BM - 1) / tc::BM, nsplit);
        tc_launch<64>(grid, w.st, A, lda, B, ldb, C, ldc, Cb, ldcb, bias, relu, M, K, kchunk, cstride, s->d_err,
                      (const bf16*)nullptr, 0, 0, mask, (float*)nullptr, 0);
    } else {
        dim3 grid(N / 64, M / 64, nsplit);
        sur::k_gemm_nt<<<grid, 128, 0, w.st>>>(A, lda, B, ldb, C, ldc, Cb, ldcb, bias, relu, K, kchunk, cstride, mask);
    }
    SCK(cudaGetLastError());
    return CS_OK;
}

// C = A B^T (+ bias) (ReLU) (mask).  A product with few output tiles and a long K (the
// convolutions' weight gradients, K = batch x time points; the linear layers at
// batch sizes of a few hundred) is split along K so that about two blocks per SM
// run; the slices' partial products are then summed in a fixed order and the
// epilogue applied.  Msplit: the rows the split is chosen for, when several batches go
// through as one (their sums must be those of the batch alone).
constexpr int kMaxSplit = 64;

static int gemm(cs_sur* s, const Lane& w, const bf16* A, int lda, const bf16* B, int ldb, float* C, int ldc, bf16* Cb,
                int ldcb, const float* bias, int relu, int M, int N, int K, const bf16* mask = nullptr, int Msplit = 0)
{
    if (M % 64 || N % 64 || K % 32) return sur_err(s, CS_E_ARG, "gemm shape %d x %d x %d not padded", M, N, K);
    const int Mt = Msplit ? Msplit : M;
    const int tiles = (s->gemm_impl == 0 ? (Mt + tc::BM - 1) / tc::BM : Mt / 64) * (N / 64);
    int nsplit = tiles < 74 ? std::min(kMaxSplit, std::max(1, std::min(K / 128, 296 / tiles))) : 1;
    if (nsplit > 1 && K % 64 == 0) {
        const int kchunk = ((K + nsplit - 1) / nsplit + 63) / 64 * 64;
        nsplit = (K + kchunk - 1) / kchunk;
        if (nsplit > 1 && (size_t)nsplit * M * N <= w.kpart_n) {
            int r = gemm_launch(s, w, A, lda, B, ldb, w.kpart, N, nullptr, 0, nullptr, 0, M, N, K, nsplit, kchunk,
                                (size_t)M * N, nullptr);
            if (r) return r;
            const int rg = (int)std::min<size_t>(1184, ((size_t)M * N + 255) / 256);
            sur::k_splitk_reduce<<<rg, 256, 0, w.st>>>(w.kpart, nsplit, M, N, C, ldc, Cb, ldcb, bias, relu, mask);
            SCK(cudaGetLastError());
            return CS_OK;
        }
    }
    return gemm_launch(s, w, A, lda, B, ldb, C, ldc, Cb, ldcb, bias, relu, M, N, K, 1, K, 0, mask);
}


static int transpose(cs_sur* s, const Lane& w, const bf16* in, int ldi, bf16* out, int ldo, int R, int Cc)
{
    dim3 grid(Cc / 32, R / 32), block(32, 8);
    sur::k_transpose<<<grid, block, 0, w.st>>>(in, ldi, out, ldo, R, Cc);
    SCK(cudaGetLastError());
    return CS_OK;
}

static size_t act_elems(const cs_sur* s, int li, int Bp)
{
    // act[li] is the input of layer li: [Bp, inP] for linear layers, [Bp*T_in, 64] for convs
    if (li == 0) return (size_t)Bp * 64;
    const Layer& p = s->L[li - 1];
    return p.conv ? (size_t)Bp * p.T * kCh : (size_t)Bp * p.outP;
}

extern "C" {

size_t cs_sur_num_params(void)
{
    // logical (unpadded) weights and biases, in the flat order of the host interface
    size_t n = 0;
    const int shapes[9][2] = {{kWidth, kIn}, {kWidth, kWidth}, {kWidth, kWidth}, {kWidth, kWidth}, {kLatent, kWidth},
                              {kT0 * kC0, kLatent}, {64, kTap * 64}, {32, kTap * 64}, {4, kTap * 32}};
    for (auto& sh : shapes) n += (size_t)sh[0] * sh[1] + sh[0];
    return n;
}

int cs_sur_create(int max_batch, int device, cs_sur** out)
{
    if (!out) return CS_E_ARG;
    cs_sur* s = new cs_sur();
    *out = s;
    if (max_batch <= 0) return sur_err(s, CS_E_ARG, "max_batch must be positive");
    s->device = device;
    s->bmax = up64(max_batch);
    SCK(cudaSetDevice(device));
    SCK(cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking));
    build_layers(s);
    Arrays arrays;
#define SA(p, n) arrays.add(p, n)
    SA(s->w, s->np); SA(s->m, s->np); SA(s->v, s->np); SA(s->g, s->np); SA(s->wb, s->np);
    const int B = s->bmax;
    s->act.assign(s->L.size() + 1, nullptr);
    size_t maxc = 0, maxcol = 0;
    for (size_t li = 0; li <= s->L.size(); li++) {
        size_t n = act_elems(s, (int)li, B);
        SA(s->act[li], n);
        maxc = std::max(maxc, n);
    }
    for (int i = 0; i < 3; i++) {
        const Layer& l = s->L[6 + i];
        maxcol = std::max(maxcol, (size_t)B * l.T * l.inP);
    }
    SA(s->yout, (size_t)B * 8 * kT0 * kCh);
    SA(s->dcols, maxcol);
    const size_t maxz = std::max(maxc, (size_t)B * 8 * kT0 * kCh);
    s->dz.assign(s->L.size(), nullptr);
    s->dzb.assign(s->L.size(), nullptr);
    s->wT.assign(s->L.size(), nullptr);
    s->dz_ready.assign(s->L.size(), nullptr);
    for (size_t li = 0; li < s->L.size(); li++) {
        const Layer& l = s->L[li];
        const size_t n = l.conv ? (size_t)B * l.T * kCh : (size_t)B * l.outP;
        SA(s->dz[li], n); SA(s->dzb[li], n);
        SA(s->wT[li], (size_t)l.outP * l.inP);
        SCK(cudaEventCreateWithFlags(&s->dz_ready[li], cudaEventDisableTiming));
    }
    SCK(cudaEventCreateWithFlags(&s->fork, cudaEventDisableTiming));
    size_t mn = 0;
    for (int i = 0; i < 3; i++) mn = std::max(mn, (size_t)s->L[6 + i].outP * s->L[6 + i].inP);
    for (int k = 0; k < kLanes; k++) {
        Lane& w = s->lane[k];
        if (k == 0) w.st = s->stream;
        else {
            SCK(cudaStreamCreateWithFlags(&w.st, cudaStreamNonBlocking));
            SCK(cudaEventCreateWithFlags(&w.done, cudaEventDisableTiming));
        }
        if (k < 3) {
            w.kpart_n = std::max(mn * kMaxSplit, (size_t)4 << 20);
            SA(w.kpart, w.kpart_n);
        }
        if (k == 1 || k == 2) {
            SA(w.dzT, maxz);
            SA(w.colsT, std::max(maxcol, maxz));
        }
        if (k == 3) SA(w.part, (size_t)((B * 8 * kT0 + 255) / 256 + 1) * 3000);
    }
    SA(s->lpart, (size_t)kLossBlocks); SA(s->lsum, (size_t)2);
    SA(s->xdev, (size_t)B * kIn); SA(s->tdev, (size_t)B * kTOut * kNOut); SA(s->sq, (size_t)B * kTOut * kNOut);
#undef SA
    if (int r = arrays.take(s)) return r;
    s->cols = reinterpret_cast<bf16*>(s->dcols);
    s->d_err = reinterpret_cast<int*>(s->lsum + 1);
    SCK(tc_enable<64>());
    SCK(tc_enable<32>());
    SCK(tc_enable<16>());
    SCK(cudaStreamSynchronize(s->stream));
    return CS_OK;
}

void cs_sur_destroy(cs_sur* s)
{
    if (!s) return;
    if (s->stream) cudaStreamSynchronize(s->stream);
    drop_graphs(s);
    if (s->pred.copy) { cudaStreamSynchronize(s->pred.copy); cudaStreamDestroy(s->pred.copy); }
    for (cudaEvent_t e : s->pred.ready)
        if (e) cudaEventDestroy(e);
    free_predict(s);
    cudaFree(s->slab);
    for (Lane& w : s->lane) {
        if (w.st && w.st != s->stream) cudaStreamDestroy(w.st);
        if (w.done) cudaEventDestroy(w.done);
    }
    for (cudaEvent_t e : s->dz_ready)
        if (e) cudaEventDestroy(e);
    if (s->fork) cudaEventDestroy(s->fork);
    if (s->stream) cudaStreamDestroy(s->stream);
    delete s;
}

const char* cs_sur_last_error(const cs_sur* s) { return s ? s->err : "null surrogate"; }

int cs_sur_set_params(cs_sur* s, const float* flat)
{
    if (!s || !flat) return CS_E_ARG;
    std::vector<float> h(s->np, 0.f);
    size_t k = 0;
    for (auto& l : s->L) {
        for (int o = 0; o < l.out; o++, k += l.in) memcpy(&h[l.wofs + (size_t)o * l.inP], flat + k, sizeof(float) * l.in);
        memcpy(&h[l.bofs], flat + k, sizeof(float) * l.out);
        k += l.out;
    }
    SCK(cudaMemcpyAsync(s->w, h.data(), sizeof(float) * s->np, cudaMemcpyHostToDevice, s->stream));
    SCK(cudaMemsetAsync(s->m, 0, sizeof(float) * s->np, s->stream));
    SCK(cudaMemsetAsync(s->v, 0, sizeof(float) * s->np, s->stream));
    sur::k_to_bf16<<<256, 256, 0, s->stream>>>(s->w, s->wb, s->np);
    SCK(cudaGetLastError());
    s->t = 0;
    SCK(cudaStreamSynchronize(s->stream));
    return CS_OK;
}

int cs_sur_get_params(cs_sur* s, float* flat)
{
    if (!s || !flat) return CS_E_ARG;
    std::vector<float> h(s->np);
    SCK(cudaMemcpyAsync(h.data(), s->w, sizeof(float) * s->np, cudaMemcpyDeviceToHost, s->stream));
    SCK(cudaStreamSynchronize(s->stream));
    size_t k = 0;
    for (auto& l : s->L) {
        for (int o = 0; o < l.out; o++, k += l.in) memcpy(flat + k, &h[l.wofs + (size_t)o * l.inP], sizeof(float) * l.in);
        memcpy(flat + k, &h[l.bofs], sizeof(float) * l.out);
        k += l.out;
    }
    return CS_OK;
}

}  // extern "C"

// Forward pass of Bp rows (x already in act[0]) through the activation buffers `act`; the
// outputs go to y64 ([Bp*368, 64], channels 0..3) or, for `n` rows, to y ([n, 365, 4]).
// Msplit: the batch size whose summation order the products take (0: Bp).
static int forward(cs_sur* s, const Lane& w, bf16* const* act, int Bp, float* y64, float* y, int n, int Msplit)
{
    int r;
    for (int li = 0; li < 6; li++) {
        const Layer& l = s->L[li];
        if ((r = gemm(s, w, act[li], l.inP, s->wb + l.wofs, l.inP, nullptr, 0, act[li + 1], l.outP,
                      s->w + l.bofs, 1, Bp, l.outP, l.inP, nullptr, Msplit))) return r;
    }
    int T = kT0;
    for (int ci = 0; ci < 3; ci++) {
        const Layer& l = s->L[6 + ci];
        const bool last = ci == 2;
        float* C = last ? y64 : nullptr;
        bf16* Cb = last ? nullptr : act[7 + ci];
        const int M = Bp * 2 * T;
        if (s->gemm_impl == 0) {   // the column matrix is generated while staging
            dim3 grid(1, (M + tc::BM - 1) / tc::BM, 1);
            const bf16 *none = nullptr, *wl = s->wb + l.wofs, *in = act[6 + ci];
            const float* bias = s->w + l.bofs;
            auto args = [&](auto launch) {
                launch(grid, w.st, none, 0, wl, l.inP, C, kCh, Cb, kCh, bias, l.relu ? 1 : 0, M, l.inP, l.inP, (size_t)0,
                       s->d_err, in, T, l.cin, none, last ? y : nullptr, n);
            };
            if (ci == 0) args([](auto... a) { tc_launch<64>(a...); });
            else if (ci == 1) args([](auto... a) { tc_launch<32>(a...); });
            else args([](auto... a) { tc_launch<16>(a...); });
            SCK(cudaGetLastError());
        } else {
            sur::k_im2col_up<<<1184, 256, 0, w.st>>>(act[6 + ci], Bp, T, l.cin, s->cols, l.inP);
            SCK(cudaGetLastError());
            if ((r = gemm(s, w, s->cols, l.inP, s->wb + l.wofs, l.inP, C, kCh, Cb, kCh, s->w + l.bofs, l.relu ? 1 : 0,
                          M, l.outP, l.inP))) return r;
            if (last && y) {
                sur::k_store_y<<<512, 256, 0, w.st>>>(y64, n, y);
                SCK(cudaGetLastError());
            }
        }
        T *= 2;
    }
    return CS_OK;
}

// Sums of the first `cols` columns (the others are padding: zero, as are their sums from the start).
static int colsum(cs_sur* s, const Lane& w, const float* dz, int rows, int ld, int cols, float* out)
{
    const int nch = (rows + kColChunk - 1) / kColChunk;
    const dim3 blk(32, 8);
    sur::k_colsum_part<<<dim3((cols + 31) / 32, nch), blk, 0, w.st>>>(dz, rows, ld, w.part);
    sur::k_colsum_final<<<(cols + 31) / 32, blk, 0, w.st>>>(w.part, nch, ld, out);
    SCK(cudaGetLastError());
    return CS_OK;
}

// The side chains of a step start here: transposed weights for the backward products.
static int begin_lanes(cs_sur* s)
{
    SCK(cudaEventRecord(s->fork, s->stream));
    for (int k = 1; k < kLanes; k++) SCK(cudaStreamWaitEvent(s->lane[k].st, s->fork, 0));
    return CS_OK;
}

// The transposed weights, beside the forward pass.
static int transpose_weights(cs_sur* s)
{
    int r;
    for (size_t li = 1; li < s->L.size(); li++) {
        const Layer& l = s->L[li];
        if ((r = transpose(s, s->lane[3], s->wb + l.wofs, l.inP, s->wT[li], l.outP, l.outP, l.inP))) return r;
    }
    SCK(cudaEventRecord(s->lane[3].done, s->lane[3].st));
    return CS_OK;
}

// Weight and bias gradients of layer li from its dz (rows x outP), beside the main chain.
static int weight_grad(cs_sur* s, int li, int rows, int Tin)
{
    int r;
    const Layer& l = s->L[li];
    const int ld = l.conv ? kCh : l.outP;
    SCK(cudaEventRecord(s->dz_ready[li], s->stream));
    const Lane& w = s->lane[1 + (li & 1)];
    SCK(cudaStreamWaitEvent(w.st, s->dz_ready[li], 0));
    SCK(cudaStreamWaitEvent(s->lane[3].st, s->dz_ready[li], 0));
    // dW = dz^T in: A = dz^T [outP, rows], B = in^T [inP, rows]
    if ((r = transpose(s, w, s->dzb[li], ld, w.dzT, rows, rows, l.outP))) return r;
    if (l.conv) {   // the transposed column matrix of the convolution's input, from the input itself
        sur::k_im2colT_up<<<dim3(l.inP / 32, rows / 64), 256, 0, w.st>>>(s->act[li], Tin, l.cin, w.colsT, rows);
        SCK(cudaGetLastError());
    } else if ((r = transpose(s, w, s->act[li], l.inP, w.colsT, rows, rows, l.inP)))
        return r;
    if ((r = gemm(s, w, w.dzT, rows, w.colsT, rows, s->g + l.wofs, l.inP, nullptr, 0, nullptr, 0, l.outP, l.inP, rows))) return r;
    return colsum(s, s->lane[3], s->dz[li], rows, ld, l.out, s->g + l.bofs);
}

// Backward pass from dy (in the last layer's dz, FP32 and BF16) to gradients in s->g; the
// side chains are joined.
static int backward(cs_sur* s, int Bp)
{
    int r;
    const Lane& w = s->lane[0];
    SCK(cudaStreamWaitEvent(w.st, s->lane[3].done, 0));   // the transposed weights
    // ---- convolutions, last to first
    int T = 8 * kT0;
    for (int li = 8; li >= 6; li--) {
        const Layer& l = s->L[li];
        const int M = Bp * T;
        if ((r = weight_grad(s, li, M, T / 2))) return r;
        // dcols = dz W: A = dz [M, outP], B = W^T [inP, outP]
        if ((r = gemm(s, w, s->dzb[li], kCh, s->wT[li], l.outP, s->dcols, l.inP, nullptr, 0, nullptr, 0, M, l.inP, l.outP))) return r;
        // dz of the layer below: col2im with the ReLU mask of this conv's input
        T /= 2;
        sur::k_col2im_up_relu<<<1184, 256, 0, w.st>>>(s->dcols, l.inP, Bp, T, l.cin, s->act[li], s->dz[li - 1], s->dzb[li - 1]);
        SCK(cudaGetLastError());
    }
    // ---- linear layers, last to first: the product's epilogue applies the ReLU mask of the
    // layer's input and leaves the dz of the layer below
    for (int li = 5; li >= 0; li--) {
        const Layer& l = s->L[li];
        if ((r = weight_grad(s, li, Bp, 0))) return r;
        if (li == 0) break;
        if ((r = gemm(s, w, s->dzb[li], l.outP, s->wT[li], l.outP, s->dz[li - 1], l.inP, s->dzb[li - 1], l.inP, nullptr, 0, Bp,
                      l.inP, l.outP, s->act[li]))) return r;
    }
    for (int k = 1; k < kLanes; k++) {
        SCK(cudaEventRecord(s->lane[k].done, s->lane[k].st));
        SCK(cudaStreamWaitEvent(s->stream, s->lane[k].done, 0));
    }
    return CS_OK;
}

// Wait for the stream; the loss sum of the last step, and an error if a tensor-core GEMM's bounded
// wait gave up (one copy of both).
static int sync_check(cs_sur* s, double* lsum = nullptr)
{
    struct { double lsum; int err, pad; } st = {};   // as they lie on the device
    SCK(cudaMemcpyAsync(&st, s->lsum, sizeof st, cudaMemcpyDeviceToHost, s->stream));
    SCK(cudaStreamSynchronize(s->stream));
    if (lsum) *lsum = st.lsum;
    if (st.err) {
        SCK(cudaMemsetAsync(s->d_err, 0, sizeof(int), s->stream));
        return sur_err(s, CS_E_CUDA, "a tensor-core GEMM gave up waiting for its products");
    }
    return CS_OK;
}

// What the weights' update takes from the step it belongs to.
struct AdamStep {
    float lr = 0.f, b1 = 0.9f, b2 = 0.999f, eps = 1e-8f, c1 = 1.f, c2 = 1.f, wd = 0.f;
};

// The kernels of one step on n rows whose inputs and targets are in xdev and tdev: loss
// terms summed into lsum, gradients in g and, with `update`, the weights' update.
static int enqueue_step(cs_sur* s, int n, bool update, const AdamStep& a)
{
    int r;
    const int Bp = up64(n);
    if ((r = begin_lanes(s))) return r;
    sur::k_load_x<<<(Bp * 64 + 255) / 256, 256, 0, s->stream>>>(s->xdev, n, Bp, s->act[0]);
    SCK(cudaGetLastError());
    if ((r = forward(s, s->lane[0], s->act.data(), Bp, s->yout, nullptr, 0, 0))) return r;
    if ((r = transpose_weights(s))) return r;
    const size_t nsq = (size_t)n * kTOut * kNOut;
    sur::k_mse<<<1184, 256, 0, s->stream>>>(s->yout, s->tdev, n, Bp, 1.f / ((float)n * kTOut * kNOut), s->dz[8], s->dzb[8], s->sq);
    SCK(cudaGetLastError());
    SCK(cudaEventRecord(s->fork, s->stream));
    SCK(cudaStreamWaitEvent(s->lane[3].st, s->fork, 0));
    sur::k_sum_part<<<kLossBlocks, 256, 0, s->lane[3].st>>>(s->sq, nsq, s->lpart);
    sur::k_sum_final<<<1, 256, 0, s->lane[3].st>>>(s->lpart, kLossBlocks, s->lsum);
    SCK(cudaGetLastError());
    if ((r = backward(s, Bp))) return r;
    if (update) {
        sur::k_adam<<<1184, 256, 0, s->stream>>>(s->w, s->m, s->v, s->g, s->wb, s->np, a.lr, a.b1, a.b2, a.eps, a.c1,
                                                  a.c2, a.wd, s->d_err);
        SCK(cudaGetLastError());
    }
    return CS_OK;
}

// The step's graph for n rows, captured on first use, or null: the step then runs as its
// launches.  A step is about 90 launches, most of a few microseconds, in four chains;
// replayed as one graph the chains overlap and the launches leave no gaps (0.93 ms a step of
// 64 rows when launched one after the other, half of it gaps and transposes that nothing had
// to wait for).  Capturing one takes longer than the launches it saves once, so when all
// places are taken a size gets that of the graph unused for longest only if it has itself
// come twice since that was used.  (Twelve sizes in turn, each ninth capture dropping
// the others: 14.7 ms for twelve steps, 11.4 in a single chain, now 4.7.)
constexpr size_t kMaxGraphs = 8;    // batch sizes kept (a training run uses one or two)
constexpr size_t kMaxMissed = 64;   // sizes without one that are remembered
static int step_graph(cs_sur* s, int n, bool update, cs_sur::StepGraph** out)
{
    *out = nullptr;
    const long long now = ++s->steps;
    for (auto& g : s->graphs)
        if (g.n == n && g.update == update) {
            g.used = now;
            *out = &g;
            return CS_OK;
        }
    if (s->graphs.size() >= kMaxGraphs) {
        auto oldest = std::min_element(s->graphs.begin(), s->graphs.end(),
                                       [](const cs_sur::StepGraph& a, const cs_sur::StepGraph& b) { return a.used < b.used; });
        auto m = std::find_if(s->missed.begin(), s->missed.end(),
                              [&](const cs_sur::Missed& x) { return x.n == n && x.update == update; });
        if (m == s->missed.end() || m->at < oldest->used) {
            if (m != s->missed.end()) s->missed.erase(m);
            else if (s->missed.size() >= kMaxMissed) s->missed.erase(s->missed.begin());
            s->missed.push_back({n, update, now});
            return CS_OK;
        }
        s->missed.erase(m);
        SCK(cudaStreamSynchronize(s->stream));
        cudaGraphExecDestroy(oldest->exec);
        cudaGraphDestroy(oldest->graph);
        s->graphs.erase(oldest);
    }
    cs_sur::StepGraph g;
    g.n = n;
    g.update = update;
    g.used = now;
    SCK(cudaStreamBeginCapture(s->stream, cudaStreamCaptureModeThreadLocal));
    int r = enqueue_step(s, n, update, AdamStep());
    cudaError_t e = cudaStreamEndCapture(s->stream, &g.graph);
    if (r || e != cudaSuccess) {
        if (g.graph) cudaGraphDestroy(g.graph);
        (void)cudaGetLastError();
        return r ? r : sur_err(s, CS_E_CUDA, "step graph capture: %s", cudaGetErrorString(e));
    }
    if (update) {
        size_t nn = 0;
        SCK(cudaGraphGetNodes(g.graph, nullptr, &nn));
        std::vector<cudaGraphNode_t> nodes(nn);
        SCK(cudaGraphGetNodes(g.graph, nodes.data(), &nn));
        for (cudaGraphNode_t nd : nodes) {
            cudaGraphNodeType ty;
            SCK(cudaGraphNodeGetType(nd, &ty));
            if (ty != cudaGraphNodeTypeKernel) continue;
            cudaKernelNodeParams kp;
            SCK(cudaGraphKernelNodeGetParams(nd, &kp));
            if (kp.func == (void*)sur::k_adam) { g.adam = nd; g.adam_params = kp; }
        }
    }
    e = cudaGraphInstantiate(&g.exec, g.graph, 0);
    if (e != cudaSuccess) {
        cudaGraphDestroy(g.graph);
        return sur_err(s, CS_E_CUDA, "step graph instantiate: %s", cudaGetErrorString(e));
    }
    s->graphs.push_back(g);
    *out = &s->graphs.back();
    return CS_OK;
}

// One step on the host's batch: inputs and targets to the device, the step's graph, and the
// loss back when asked for (which waits for the step).
static int run_step(cs_sur* s, const float* x, const float* target, int n, float* loss, bool update, float lr, float wd)
{
    if (n <= 0 || n > s->bmax) return sur_err(s, CS_E_RANGE, "batch of %d outside 1..%d", n, s->bmax);
    cs_sur::StepGraph* g;
    int r = step_graph(s, n, update, &g);
    if (r) return r;
    SCK(cudaMemcpyAsync(s->xdev, x, sizeof(float) * n * kIn, cudaMemcpyHostToDevice, s->stream));
    SCK(cudaMemcpyAsync(s->tdev, target, sizeof(float) * n * kTOut * kNOut, cudaMemcpyHostToDevice, s->stream));
    AdamStep a;
    if (update) {
        s->t++;
        a.lr = lr;
        a.wd = wd;
        a.c1 = 1.f - powf(a.b1, (float)s->t);
        a.c2 = 1.f - powf(a.b2, (float)s->t);
    }
    if (!g) {
        if ((r = enqueue_step(s, n, update, a))) return r;
    } else {
        if (update) {
            void* args[] = {&s->w, &s->m, &s->v, &s->g, &s->wb, &s->np, &a.lr, &a.b1, &a.b2, &a.eps, &a.c1, &a.c2, &a.wd, &s->d_err};
            cudaKernelNodeParams kp = g->adam_params;
            kp.kernelParams = args;
            kp.extra = nullptr;
            SCK(cudaGraphExecKernelNodeSetParams(g->exec, g->adam, &kp));
        }
        SCK(cudaGraphLaunch(g->exec, s->stream));
    }
    if (loss) {
        double acc = 0.0;
        if ((r = sync_check(s, &acc))) {
            if (update) s->t--;
            return r;
        }
        *loss = (float)(acc / (double)((size_t)n * kTOut * kNOut));
    }
    return CS_OK;
}

// ---------------------------------------------------------------- prediction
// Workspace of the prediction path: activations for `rows` rows, and two slots of inputs and
// outputs, so that one group of rows is computed while the one before goes to the caller.
// Made for as many rows as the calls so far asked for, up to the largest group.
static cudaError_t make_predict(cs_sur* s, int rows)
{
    cs_sur::Predict& P = s->pred;
    const size_t nx = (size_t)rows * 64, ny = (size_t)rows * kTOut * kNOut;   // rows are 16-byte multiples throughout
    std::vector<size_t> at;   // activations, in floats from the start
    size_t n = 2 * (nx + ny);
    if (rows > s->bmax) {
        for (size_t li = 0; li < s->L.size(); li++) {
            at.push_back(n);
            n += (act_elems(s, (int)li, rows) + 1) / 2;
        }
        size_t wide = 0;   // slices x columns of the widest split: a linear layer has K / 128 slices at most
        for (int li = 0; li < 6; li++) wide = std::max(wide, (size_t)(s->L[li].inP / 128) * s->L[li].outP);
        P.kpart_n = wide * rows;
        P.kpart = nullptr;
        n += P.kpart_n;
    }
    cudaError_t e = cudaMalloc(&P.dev, sizeof(float) * n);
    if (e == cudaSuccess) e = cudaMemsetAsync(P.dev, 0, sizeof(float) * n, s->stream);
    if (e == cudaSuccess && !P.copy) e = cudaStreamCreateWithFlags(&P.copy, cudaStreamNonBlocking);
    for (int k = 0; k < 2; k++) {
        if (e == cudaSuccess && !P.ready[k]) e = cudaEventCreateWithFlags(&P.ready[k], cudaEventDisableTiming);
    }
    if (e != cudaSuccess) return e;
    for (int k = 0; k < 2; k++) {
        P.xdev[k] = P.dev + k * nx;
        P.ydev[k] = P.dev + 2 * nx + k * ny;
    }
    P.act.clear();
    for (size_t a : at) P.act.push_back((bf16*)(P.dev + a));
    if (!at.empty()) P.kpart = P.dev + (n - P.kpart_n);
    P.rows = rows;
    return cudaSuccess;
}

static int predict_space(cs_sur* s, int n)
{
    // as many whole batches as about 2048 rows hold: enough blocks for every product
    const int batches = std::min(std::max(1, 2048 / s->bmax), n / s->bmax);
    const int rows = s->bmax * std::max(1, batches);
    if (rows <= s->pred.rows) return CS_OK;
    if (s->pred.rows) SCK(cudaStreamSynchronize(s->stream));
    free_predict(s);
    if (make_predict(s, rows) == cudaSuccess) return CS_OK;
    cudaGetLastError();   // no memory for a group: one batch at a time
    free_predict(s);
    SCK(make_predict(s, s->bmax));
    return CS_OK;
}

// Has the pages of the caller's output mapped by a few threads while the first groups are
// computed: left to the copies, one page fault after the other takes 20 of the 27 ms that
// 117 MB need to reach memory the caller has just allocated (eight threads: 2.8 ms).  One
// byte a page is written back as it is, before the first copy into the output.
struct PageMapper {
    std::thread th[8];
    PageMapper(float* y, size_t n)
    {
        constexpr size_t kPage = 4096, kLeast = (size_t)4 << 20;
        const size_t bytes = sizeof(float) * n;
        if (bytes < kLeast) return;
        const size_t nt = std::min<size_t>(8, std::max(1u, std::thread::hardware_concurrency()));
        const size_t per = (bytes / nt + kPage) / kPage * kPage;
        volatile char* p = (volatile char*)y;
        try {
            for (size_t t = 0; t < nt; t++)
                th[t] = std::thread([=] {
                    for (size_t i = t * per; i < std::min(bytes, (t + 1) * per); i += kPage) p[i] = p[i];
                });
        } catch (...) {   // no more threads to be had: the copies map what is left
        }
    }
    void done()
    {
        for (std::thread& t : th)
            if (t.joinable()) t.join();
    }
    ~PageMapper() { done(); }
};

// Predictions for n rows in groups of whole batches (several as one pass, each product
// summed as for one batch, so a row's outputs do not depend on the grouping), the rows past
// the last whole batch as a batch of their own.  Bound by the outputs' way into the caller's
// memory: 20,000 rows are 117 MB, 7 ms of copying into mapped pages, beside 2.2 ms of kernels.
static int predict(cs_sur* s, const float* x, int n, float* y)
{
    int r = predict_space(s, n);
    if (r) return r;
    cs_sur::Predict& P = s->pred;
    const size_t ny = (size_t)kTOut * kNOut;
    const bool wide = P.rows > s->bmax && s->gemm_impl == 0;
    PageMapper map(y, (size_t)n * ny);
    struct { int at, rows; } made[2] = {{0, 0}, {0, 0}};
    auto take = [&](int k) -> int {   // slot k's outputs to the caller
        if (made[k].rows == 0) return CS_OK;
        map.done();
        SCK(cudaStreamWaitEvent(P.copy, P.ready[k], 0));
        SCK(cudaMemcpyAsync(y + (size_t)made[k].at * ny, P.ydev[k], sizeof(float) * made[k].rows * ny, cudaMemcpyDeviceToHost,
                            P.copy));
        SCK(cudaStreamSynchronize(P.copy));
        made[k].rows = 0;
        return CS_OK;
    };
    int k = 0;
    for (int at = 0; at < n; k ^= 1) {
        const int left = n - at;
        const int nb = left < s->bmax ? left : wide ? std::min(P.rows, left / s->bmax * s->bmax) : s->bmax;
        const bool group = nb > s->bmax;
        const int Bp = up64(nb);
        SCK(cudaMemcpyAsync(P.xdev[k], x + (size_t)at * kIn, sizeof(float) * nb * kIn, cudaMemcpyHostToDevice, s->stream));
        bf16* const* act = group ? P.act.data() : s->act.data();
        sur::k_load_x<<<(Bp * 64 + 255) / 256, 256, 0, s->stream>>>(P.xdev[k], nb, Bp, act[0]);
        SCK(cudaGetLastError());
        Lane w = s->lane[0];
        if (group) {
            w.kpart = P.kpart;
            w.kpart_n = P.kpart_n;
        }
        if ((r = forward(s, w, act, Bp, s->gemm_impl == 0 ? nullptr : s->yout, P.ydev[k], nb, group ? s->bmax : 0))) return r;
        SCK(cudaEventRecord(P.ready[k], s->stream));
        made[k].at = at;
        made[k].rows = nb;
        at += nb;
        if ((r = take(k ^ 1))) return r;
    }
    return take(k ^ 1);
}

extern "C" {

int cs_sur_forward(cs_sur* s, const float* x, int n, float* y)
{
    if (!s || !x || !y) return CS_E_ARG;
    if (n <= 0) return sync_check(s);
    const int r = predict(s, x, n, y);
    if (r == CS_OK) return sync_check(s);
    cudaStreamSynchronize(s->stream);   // nothing of the call is left in flight
    if (s->pred.copy) cudaStreamSynchronize(s->pred.copy);
    return r;
}

int cs_sur_loss_grad(cs_sur* s, const float* x, const float* target, int n, float* loss, float* grad)
{
    if (!s || !x || !target) return CS_E_ARG;
    int r = run_step(s, x, target, n, loss, false, 0.f, 0.f);
    if (r) return r;
    if (grad) {
        std::vector<float> h(s->np);
        SCK(cudaMemcpyAsync(h.data(), s->g, sizeof(float) * s->np, cudaMemcpyDeviceToHost, s->stream));
        if ((r = sync_check(s))) return r;
        size_t k = 0;
        for (auto& l : s->L) {
            for (int o = 0; o < l.out; o++, k += l.in) memcpy(grad + k, &h[l.wofs + (size_t)o * l.inP], sizeof(float) * l.in);
            memcpy(grad + k, &h[l.bofs], sizeof(float) * l.out);
            k += l.out;
        }
    }
    return CS_OK;
}

int cs_sur_train_step(cs_sur* s, const float* x, const float* target, int n, float lr, float weight_decay, float* loss)
{
    if (!s || !x || !target) return CS_E_ARG;
    int r = run_step(s, x, target, n, loss, true, lr, weight_decay);
    if (r) return r;
    if (loss) return CS_OK;
    if ((r = sync_check(s))) s->t--;
    return r;
}

int cs_sur_set_gemm(cs_sur* s, int impl)
{
    if (!s) return CS_E_ARG;
    if (impl != 0 && impl != 1) return sur_err(s, CS_E_ARG, "GEMM path must be 0 (tcgen05) or 1 (mma.sync)");
    SCK(cudaStreamSynchronize(s->stream));
    drop_graphs(s);
    s->gemm_impl = impl;
    return CS_OK;
}

}  // extern "C"
