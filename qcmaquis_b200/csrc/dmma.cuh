// DMMA (mma.sync m8n8k4 .f64) tile machinery shared by the FP64 kernels: CTA
// tile shapes, a two-stage cp.async staging buffer, warp-level fragments.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace qcm {
namespace dm {

constexpr int BK = 16, PAD = 4, NTHR = 128;

static __device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

// 8-byte asynchronous global->shared copy; a false predicate writes zeros (src-size 0)
static __device__ __forceinline__ void cp8(double* smem, const double* gmem, bool pred) {
    unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(s), "l"(gmem), "r"(pred ? 8 : 0));
}
// 16-byte asynchronous copy (both addresses 16-byte aligned); a false predicate writes zeros
static __device__ __forceinline__ void cp16(void* smem, const void* gmem, bool pred) {
    unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(pred ? 16 : 0));
}
static __device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::); }
static __device__ __forceinline__ void cp_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::); }

// CTA tile = WM x WN warps, each warp FM x FN DMMA fragments of 8 x 8.
template <int WM_, int WN_, int FM_, int FN_>
struct Shape {
    static constexpr int WM = WM_, WN = WN_, FM = FM_, FN = FN_;
    static constexpr int BM = WM * FM * 8, BN = WN * FN * 8;
    static constexpr int A_PER = BM * BK / NTHR, B_PER = BN * BK / NTHR;
    static_assert(WM * WN * 32 == NTHR, "4 warps per CTA");
    // first row of fragment i of a warp in warp row wm: the warp rows take fragments in turn, so that the rows
    // missing from a tile are missing from all warps alike
    __host__ __device__ static constexpr int row(int i, int wm) { return (i * WM + wm) * 8; }
};
using Sh16 = Shape<1, 4, 2, 4>;  // 16 x 128
using Sh32 = Shape<1, 4, 4, 4>;  // 32 x 128
using Sh64 = Shape<2, 2, 4, 4>;  // 64 x 64
using Sh128 = Shape<4, 1, 4, 4>; // 128 x 32

template <class S>
struct __align__(16) Stage {
    double A[BK][S::BM + PAD];
    double B[BK][S::BN + PAD];
};

template <class S>
struct Acc {
    double c[S::FM][S::FN][2];
    __device__ void zero() {
#pragma unroll
        for (int i = 0; i < S::FM; ++i)
#pragma unroll
            for (int j = 0; j < S::FN; ++j) c[i][j][0] = c[i][j][1] = 0.0;
    }
};

template <class S>
static __device__ __forceinline__ void mma_stage(const double (*A)[S::BM + PAD], const double (*B)[S::BN + PAD], Acc<S>& acc,
                                          int warp, int lane) {
    const int r = lane >> 2, q = lane & 3;
    const int wm = warp % S::WM, wn = warp / S::WM;
#pragma unroll
    for (int kk = 0; kk < BK; kk += 4) {
        double a[S::FM], b[S::FN];
#pragma unroll
        for (int i = 0; i < S::FM; ++i) a[i] = A[kk + q][S::row(i, wm) + r];
#pragma unroll
        for (int j = 0; j < S::FN; ++j) b[j] = B[kk + q][wn * S::FN * 8 + j * 8 + r];
#pragma unroll
        for (int i = 0; i < S::FM; ++i)
#pragma unroll
            for (int j = 0; j < S::FN; ++j) dmma(acc.c[i][j], a[i], b[j]);
    }
}

// Same, skipping the 4-slice k groups whose bit in mask is clear (all-zero coefficients)
template <class S>
static __device__ __forceinline__ void mma_stage_masked(const double (*A)[S::BM + PAD], const double (*B)[S::BN + PAD],
                                                 Acc<S>& acc, int warp, int lane, uint32_t mask) {
    const int r = lane >> 2, q = lane & 3;
    const int wm = warp % S::WM, wn = warp / S::WM;
#pragma unroll
    for (int kk = 0; kk < BK; kk += 4) {
        if (!((mask >> (kk / 4)) & 1u)) continue;
        double a[S::FM], b[S::FN];
#pragma unroll
        for (int i = 0; i < S::FM; ++i) a[i] = A[kk + q][S::row(i, wm) + r];
#pragma unroll
        for (int j = 0; j < S::FN; ++j) b[j] = B[kk + q][wn * S::FN * 8 + j * 8 + r];
#pragma unroll
        for (int i = 0; i < S::FM; ++i)
#pragma unroll
            for (int j = 0; j < S::FN; ++j) dmma(acc.c[i][j], a[i], b[j]);
    }
}

// Operand staged with k fastest (its k elements contiguous in memory): element (x, k) of a stage at x * BK +
// (k ^ 4 (x mod 4)).  Rows of 128 bytes without padding; the swizzle puts the 4 k's of 4 neighbouring x's in 16
// different 8-byte banks for the fragment reads, and keeps pairs of k (16-byte copies) together.
static __device__ __forceinline__ int kfast(int x, int k) { return x * BK + (k ^ ((x & 3) << 2)); }

// Staging of one operand of a stage (X x BK elements, X = BM or BN) in one of three ways.  get(x, k): pointer to
// element (x, k); nx, nk: how many x and k of the stage exist (elements past them are zero).
//   k contiguous in memory: k fastest in shared memory (kfast), 16 bytes at a time if v16 (every k pair starts on
//     16 bytes and nk is even), else 8;
//   x contiguous: rows of X + PAD elements per k, 16 bytes at a time if v16 (nx even), else 8.
// UNROLL copies in one loop body.
template <int X, int UNROLL, class Get>
static __device__ __forceinline__ void stage_kfast(double* dst, const double* any, uint32_t nx, uint32_t nk, bool v16, Get get) {
    const int tid = threadIdx.x;
    if (v16) {
        constexpr int CH = X * BK / 2;
        static_assert(CH % NTHR == 0, "whole chunks per thread");
#pragma unroll UNROLL
        for (int rr = 0; rr < CH / NTHR; ++rr) {
            const int e = tid + rr * NTHR, k = 2 * (e % (BK / 2)), x = e / (BK / 2);
            const bool ok = uint32_t(x) < nx && uint32_t(k) < nk;
            cp16(dst + kfast(x, k), ok ? get(x, k) : any, ok);
        }
    } else {
#pragma unroll UNROLL
        for (int rr = 0; rr < X * BK / NTHR; ++rr) {
            const int e = tid + rr * NTHR, k = e % BK, x = e / BK;
            const bool ok = uint32_t(x) < nx && uint32_t(k) < nk;
            cp8(dst + kfast(x, k), ok ? get(x, k) : any, ok);
        }
    }
}
template <int X, int UNROLL, class Get>
static __device__ __forceinline__ void stage_xfast(double* dst, const double* any, uint32_t nx, uint32_t nk, bool v16, Get get) {
    const int tid = threadIdx.x;
    if (v16) {
        constexpr int CH = X * BK / 2;
#pragma unroll UNROLL
        for (int rr = 0; rr < CH / NTHR; ++rr) {
            const int e = tid + rr * NTHR, x = 2 * (e % (X / 2)), k = e / (X / 2);
            const bool ok = uint32_t(x) < nx && uint32_t(k) < nk;
            cp16(dst + k * (X + PAD) + x, ok ? get(x, k) : any, ok);
        }
    } else {
#pragma unroll UNROLL
        for (int rr = 0; rr < X * BK / NTHR; ++rr) {
            const int e = tid + rr * NTHR, x = e % X, k = e / X;
            const bool ok = uint32_t(x) < nx && uint32_t(k) < nk;
            cp8(dst + k * (X + PAD) + x, ok ? get(x, k) : any, ok);
        }
    }
}

// One stage with each operand in either layout (AK, BKF: k fastest), leaving out what lies beyond the operands:
// row fragments past nfm (of the tile's BM / 8) and k groups of 4 past ng.
template <class S, bool AK, bool BKF>
static __device__ __forceinline__ void mma_stage_part(const double* A, const double* B, Acc<S>& acc, int warp, int lane, int nfm,
                                                      int ng) {
    const int r = lane >> 2, q = lane & 3;
    const int wm = warp % S::WM, wn = warp / S::WM;
#pragma unroll
    for (int kk = 0; kk < BK; kk += 4) {
        if (kk >= 4 * ng) break;
        double a[S::FM], b[S::FN];
#pragma unroll
        for (int i = 0; i < S::FM; ++i) {
            const int m = S::row(i, wm) + r;
            a[i] = A[AK ? kfast(m, kk + q) : (kk + q) * (S::BM + PAD) + m];
        }
#pragma unroll
        for (int j = 0; j < S::FN; ++j) {
            const int n = wn * S::FN * 8 + j * 8 + r;
            b[j] = B[BKF ? kfast(n, kk + q) : (kk + q) * (S::BN + PAD) + n];
        }
#pragma unroll
        for (int i = 0; i < S::FM; ++i) {
            if (i * S::WM + wm >= nfm) break;
#pragma unroll
            for (int j = 0; j < S::FN; ++j) dmma(acc.c[i][j], a[i], b[j]);
        }
    }
}

// Visit every accumulator element: f(m, n, value) with tile-local (m, n).
template <class S, class F>
static __device__ __forceinline__ void for_acc(const Acc<S>& acc, int warp, int lane, F f) {
    const int r = lane >> 2, q = lane & 3;
    const int wm = warp % S::WM, wn = warp / S::WM;
#pragma unroll
    for (int i = 0; i < S::FM; ++i)
#pragma unroll
        for (int j = 0; j < S::FN; ++j)
#pragma unroll
            for (int c = 0; c < 2; ++c) f(S::row(i, wm) + r, wn * S::FN * 8 + j * 8 + q * 2 + c, acc.c[i][j][c]);
}


}  // namespace dm
}  // namespace qcm
