// Thin QR and LQ of many blocks at once (the canonisation steps of the sweep).
//
// The reference canonises a site tensor block by block with LAPACK: qr / lq
// (framework/alps/matrix/algorithms.hpp:260-325, geqrf + orgqr, gelqf + orglq), called by
// MPSTensor::normalize_left / normalize_right (mp_tensors/mpstensor.hpp:242-300).  Here every
// block of a site tensor is factorised at the same time, with the unblocked Householder
// method LAPACK's geqr2 / org2r define (a published algorithm; Golub & Van Loan, Algorithm 5.2.1):
//   for j < k = min(m, n): alpha = A(j, j), xnorm = |A(j+1:m, j)|;
//     xnorm = 0: tau_j = 0 (H_j = I);
//     else beta = -sign(alpha) hypot(alpha, xnorm), tau_j = (beta - alpha) / beta,
//          v_j = (1, A(j+1:m, j) / (alpha - beta)), A(j, j) = beta;
//     A(j:m, j+1:n) -= tau_j v_j (v_j^T A(j:m, j+1:n));
//   R = the upper triangle (k x n); Q = H_0 ... H_{k-1} applied to the first k columns of I (m x k).
// One rule is added (the oracle's restatement has it too): a column whose remaining part
// |A(j:m, j)| is at most 64 eps |A|_F -- rounding noise, as in every column after the first of a
// rank-1 block -- is set to exactly zero and gets no reflector, so that the orthonormal completion
// of Q is fixed by the arithmetic rather than by that noise (which LAPACK implementations resolve
// differently).
// LQ is the QR of the transpose (the same reflectors as gelqf): L = R'^T, Q = Q'^T.
//
// An unpivoted block of one CTA's size is factorised by k_qr_one.  The others (k_qr) by a cluster of 1 to
// 16 CTAs each, the columns dealt out to them in turn.  A step reads and writes the whole trailing matrix, so one SM's
// shared memory (or L2, for a block beyond it) binds a large block, and the columns are what a step treats
// independently.  Per step one cluster barrier: each CTA has sent the best
// of its remaining columns as the next pivot (norm, position, leading element; computed while updating them), all
// of them pick the same winner and read its column from the owner's shared memory.  A pivot column is never
// written again in its owner's store (its diagonal and reflector are kept apart), so nobody waits for its readers.
// No column is moved: positions are swapped instead.  Q needs no exchange: each column is the product of
// reflectors with a unit vector, by one warp.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <stdexcept>
#include <vector>

#include "linalg.hpp"

namespace cg = cooperative_groups;

namespace qcm {

namespace {

constexpr int QR_THR = 1024;
constexpr int QR_WARPS = QR_THR / 32;
constexpr uint32_t QR_PIV_MAX = 1024;           // columns of a pivoted factorisation
constexpr uint32_t QR_SMEM_DOUBLES = 28400;     // dynamic shared memory per CTA (222 KiB; 2.4 KiB static)
constexpr uint32_t QR_MAX_CLUSTER = 16;

// CTAs per block, alone: 64 columns of 64 rows are two passes of the 32 warps, about what a step's barriers cost; a cluster's
// barrier costs more than a CTA's, and up to about 112 columns of 112 rows one CTA is the faster (66 to 90 columns:
// 0.37 ms against 0.62 ms).  The pivoted QRs of a two-site truncation at L=24: M=2048 70 ms with one CTA per block, 8.8 ms
// so; M=512 1.54 and 1.1 ms.
inline uint32_t qr_cluster(uint32_t mm, uint32_t nn) {
    const uint64_t e = uint64_t(mm) * nn;
    if (e <= 112 * 112) return 1;
    uint32_t nc = 1;
    while (nc < QR_MAX_CLUSTER && nc * 2 <= nn && e > uint64_t(64 * 64) * nc * nc) nc *= 2;
    return nc;
}

// Shared memory of one CTA (doubles): the current pivot column (mm), the diagonal and scales of R's k steps, the
// positions (nn) and the CTA's own columns' positions, then the CTA's columns if they fit, else they are in
// the block's scratch (L2-resident).  false: not even the fixed part fits, which is then in the scratch too.
struct QrLayout {
    uint32_t ncol;    // columns per CTA
    uint64_t fixed;   // doubles before the columns
    bool cols_smem, fixed_smem;
};
__host__ __device__ inline QrLayout qr_layout(uint32_t mm, uint32_t nn, uint32_t nc, uint32_t smem_doubles) {
    QrLayout l;
    const uint32_t k = mm < nn ? mm : nn;
    l.ncol = (nn + nc - 1) / nc;
    l.fixed = uint64_t(mm) + 2 * uint64_t(k) + (nn + 1) / 2 + (l.ncol + 1) / 2;
    l.fixed_smem = l.fixed <= smem_doubles;
    l.cols_smem = l.fixed_smem && l.fixed + uint64_t(l.ncol) * mm <= smem_doubles;
    return l;
}

__device__ double warp_sum(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

// a pivot candidate: squared norm over the remaining rows, of the rows after the first of them, that first
// element, the column's position and the column
struct QrCand {
    double val, tail, head;
    uint32_t pos, col;
};
__device__ __forceinline__ bool better(double va, uint32_t pa, double vb, uint32_t pb) { return va > vb || (va == vb && pa < pb); }
// the best candidate of each aligned group of n lanes (a power of two), in all of them
__device__ __forceinline__ QrCand warp_best(QrCand c, int n) {
    for (int o = n / 2; o > 0; o >>= 1) {
        QrCand d;
        d.val = __shfl_xor_sync(0xffffffffu, c.val, o);
        d.tail = __shfl_xor_sync(0xffffffffu, c.tail, o);
        d.head = __shfl_xor_sync(0xffffffffu, c.head, o);
        d.pos = __shfl_xor_sync(0xffffffffu, c.pos, o);
        d.col = __shfl_xor_sync(0xffffffffu, c.col, o);
        if (better(d.val, d.pos, c.val, c.pos)) c = d;
    }
    return c;
}

__global__ void __launch_bounds__(QR_THR) k_qr(const QrJob* __restrict__ jobs, const double* __restrict__ A,
                                               double* __restrict__ Q, double* __restrict__ R, double* __restrict__ W,
                                               uint32_t* __restrict__ P, uint32_t smem_doubles) {
    extern __shared__ double qsm[];
    __shared__ QrCand cand[2][QR_MAX_CLUSTER];  // by step parity: every CTA's candidate
    __shared__ QrCand wbest[QR_WARPS];
    __shared__ double red[QR_WARPS];
    __shared__ double fro[QR_MAX_CLUSTER];
    __shared__ double sh_tau, sh_scale;
    cg::cluster_group cl = cg::this_cluster();
    const uint32_t nc = cl.num_blocks(), rank = cl.block_rank();
    const QrJob J = jobs[blockIdx.x / nc];
    const uint32_t nthr = blockDim.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarp = nthr / 32;
    // the matrix factorised: F (mm x nn) = A_j, or A_j^T for an LQ
    const uint32_t mm = J.lq ? J.n : J.m, nn = J.lq ? J.m : J.n, k = mm < nn ? mm : nn;
    const bool pivot = (J.flags & QR_PIVOT) != 0;
    const QrLayout l = qr_layout(mm, nn, nc, smem_doubles);
    // scratch: the reflectors (mm x k, column j of step j), then per CTA its fixed part and columns
    double* Vs = W + J.w_off;
    double* own = Vs + uint64_t(mm) * k + rank * (l.fixed + uint64_t(l.ncol) * mm);
    double* fx = l.fixed_smem ? qsm : own;
    double* vbuf = fx;           // mm: the pivot column, unscaled
    double* diag = vbuf + mm;    // k
    double* taus = diag + k;     // k
    uint32_t* perm = reinterpret_cast<uint32_t*>(taus + k);                        // nn: column at each position
    uint32_t* lpos = reinterpret_cast<uint32_t*>(taus + k + (nn + 1) / 2);         // ncol: position of own columns
    double* F = l.cols_smem ? qsm + l.fixed : own + l.fixed;
    const uint32_t ncl = nn > rank ? (nn - rank + nc - 1) / nc : 0;  // own columns: rank, rank + nc, ...
    auto cluster_sync = [&] {
        if (nc > 1) cluster_sync_all();
        else __syncthreads();
    };
    const double* a = A + J.a_off;
    for (uint64_t e = tid; e < uint64_t(mm) * ncl; e += nthr) {
        const uint32_t i = uint32_t(e % mm), c = rank + uint32_t(e / mm) * nc;
        F[e] = J.lq ? a[c + uint64_t(i) * J.m] : a[i + uint64_t(c) * J.m];
    }
    for (uint32_t c = tid; c < nn; c += nthr) perm[c] = c;
    for (uint32_t c = tid; c < ncl; c += nthr) lpos[c] = rank + c * nc;
    cluster_sync();  // every CTA of the cluster runs: from here on the others may store into its shared memory
    // candidate of this CTA for step `step`, sent to every CTA: `best` of the calling warp's columns
    auto send_candidate = [&](QrCand best, uint32_t step) {
        if (lane == 0) wbest[warp] = best;
        __syncthreads();
        if (warp == 0) {
            QrCand c = wbest[lane < nwarp ? lane : 0];
            if (lane >= nwarp) { c.val = -2.0; c.pos = 0xffffffffu; }
            c = warp_best(c, 32);
            if (nc == 1) {
                if (lane == 0) cand[step & 1][0] = c;
            } else if (lane < nc) {
                cl.map_shared_rank(&cand[step & 1][0], lane)[rank] = c;
            }
        }
        cluster_sync();
    };
    const QrCand none{-1.0, 0.0, 0.0, 0xffffffffu, 0};
    {
        // norms of all columns: the first pivot, and the negligible-column threshold 64 eps |A|_F
        QrCand best = none;
        double f = 0.0;
        for (uint32_t c = warp; c < ncl; c += nwarp) {
            const double* fc = F + uint64_t(c) * mm;
            double t = 0.0;
            for (uint32_t i = 1 + lane; i < mm; i += 32) t = fma(fc[i], fc[i], t);
            t = warp_sum(t);
            const double h = fc[0], v = fma(h, h, t);
            f += v;
            const uint32_t pos = lpos[c];
            if ((pivot || pos == 0) && better(v, pos, best.val, best.pos)) best = QrCand{v, t, h, pos, rank + c * nc};
        }
        if (lane == 0) red[warp] = f;
        __syncthreads();
        if (warp == 0) {
            double t = 0.0;
            for (uint32_t q = 0; q < nwarp; ++q) t += red[q];
            if (nc == 1) {
                if (lane == 0) fro[0] = t;
            } else if (lane < nc) {
                cl.map_shared_rank(&fro[0], lane)[rank] = t;
            }
        }
        send_candidate(best, 0);
    }
    double thr = 0.0;
    for (uint32_t d = 0; d < nc; ++d) thr += fro[d];
    thr = 64.0 * 2.220446049250313e-16 * sqrt(thr);
    for (uint32_t j = 0; j < k; ++j) {
        // the pivot, the same in every warp of every CTA
        QrCand pv = warp_best(cand[j & 1][lane & (nc - 1)], int(nc));
        if (pv.pos >= nn) {
            // no candidate compared (NaN columns remain): the column at position j, its values undefined
            pv.pos = j;
            pv.col = perm[j];  // warp 0 writes the same value below
            pv.head = pv.tail = __longlong_as_double(0x7ff8000000000000ll);
        }
        const uint32_t owner = pv.col % nc;
        if (warp == 0) {
            if (lane == 0) {
                const double alpha = pv.head, xnorm = sqrt(pv.tail), nrm = hypot(alpha, xnorm);
                double tau = 0.0, scale = 1.0, beta = alpha;
                const int zero = nrm <= thr;
                if (!zero && xnorm != 0.0) {
                    beta = -copysign(nrm, alpha);
                    tau = (beta - alpha) / beta;
                    scale = 1.0 / (alpha - beta);
                }
                sh_tau = tau;
                sh_scale = scale;
                taus[j] = tau;
                diag[j] = zero ? 0.0 : beta;  // a negligible column: exactly zero in R, no reflector
                const uint32_t other = perm[j];
                perm[j] = pv.col;
                perm[pv.pos] = other;
                if (other % nc == rank) lpos[other / nc] = pv.pos;
                if (owner == rank) lpos[pv.col / nc] = j;
            }
        } else {
            // the column below the diagonal, from its owner
            const double* src = F + uint64_t(pv.col / nc) * mm;
            if (owner != rank)
                src = l.cols_smem ? cl.map_shared_rank(qsm + l.fixed, owner) + uint64_t(pv.col / nc) * mm
                                  : Vs + uint64_t(mm) * k + owner * (l.fixed + uint64_t(l.ncol) * mm) + l.fixed +
                                        uint64_t(pv.col / nc) * mm;
            for (uint32_t i = j + 1 + (tid - 32); i < mm; i += nthr - 32) vbuf[i] = src[i];
        }
        __syncthreads();
        const double tau = sh_tau, scale = sh_scale;
        if (j % nc == rank && tau != 0.0) {
            double* vj = Vs + uint64_t(j) * mm;
            for (uint32_t i = j + 1 + tid; i < mm; i += nthr) vj[i] = vbuf[i] * scale;
        }
        if (j + 1 == k && nn == k) break;
        // remaining columns, one warp each: F(j:mm, c) -= tau v (v^T F(j:mm, c)), v_j = 1, and their norms over
        // the rows after j
        QrCand best = none;
        for (uint32_t c = warp; c < ncl; c += nwarp) {
            const uint32_t pos = lpos[c];
            if (pos <= j) continue;
            double* fc = F + uint64_t(c) * mm;
            double t = 0.0;
            if (tau != 0.0) {
                const double fj = fc[j];  // read by every lane before lane 0 writes it
                double d = 0.0;
                for (uint32_t i = j + 1 + lane; i < mm; i += 32) d = fma(vbuf[i], fc[i], d);
                d = (warp_sum(d) * scale + fj) * tau;
                if (lane == 0) fc[j] = fj - d;
                const double ds = d * scale;
                for (uint32_t i = j + 1 + lane; i < mm; i += 32) {
                    const double x = fma(-ds, vbuf[i], fc[i]);
                    fc[i] = x;
                    if (i > j + 1) t = fma(x, x, t);
                }
            } else {
                for (uint32_t i = j + 2 + lane; i < mm; i += 32) t = fma(fc[i], fc[i], t);
            }
            t = warp_sum(t);
            __syncwarp();
            if (j + 1 >= k) continue;
            const double h = fc[j + 1], v = fma(h, h, t);
            if ((pivot || pos == j + 1) && better(v, pos, best.val, best.pos)) best = QrCand{v, t, h, pos, rank + c * nc};
        }
        if (j + 1 < k) send_candidate(best, j + 1);
    }
    // every CTA has read the last pivot column, and the reflectors are written
    cluster_sync();
    // R (k x nn, ld k) from the rows above the diagonal; for an LQ, L = R'^T (m x k, ld m)
    double* r = R + J.r_off;
    const bool rt = (J.flags & QR_RT) != 0;
    for (uint64_t e = tid; e < uint64_t(k) * ncl; e += nthr) {
        const uint32_t i = uint32_t(e % k), lc = uint32_t(e / k), c = lpos[lc];
        const double v = i < c ? F[i + uint64_t(lc) * mm] : (i == c ? diag[i] : 0.0);
        if (J.lq) r[c + uint64_t(i) * J.m] = v;
        else if (rt) r[c + uint64_t(i) * nn] = v;
        else r[i + uint64_t(c) * k] = v;
    }
    if (pivot && rank == 0)
        for (uint32_t c = tid; c < nn; c += nthr) P[J.p_off + c] = perm[c];
    __syncthreads();
    // Q' = H_0 ... H_{k-1} I(:, 0:k): columns rank, rank + nc, ... of this CTA in its column store, one warp each,
    // the longest products first; reflectors above a column's index do not touch its unit vector
    double* qo = Q + J.q_off;
    const uint32_t qcl = k > rank ? (k - rank + nc - 1) / nc : 0;
    for (uint32_t x = warp; x < qcl; x += nwarp) {
        const uint32_t lc = qcl - 1 - x, c = rank + lc * nc;
        double* qc = F + uint64_t(lc) * mm;
        for (uint32_t i = lane; i < mm; i += 32) qc[i] = i == c ? 1.0 : 0.0;
        __syncwarp();
        for (int jj = int(c); jj >= 0; --jj) {
            const uint32_t j = uint32_t(jj);
            const double tau = taus[j];
            if (tau == 0.0) continue;
            const double* vj = Vs + uint64_t(j) * mm;
            const double qj = qc[j];
            double d = 0.0;
            for (uint32_t i = j + 1 + lane; i < mm; i += 32) d = fma(vj[i], qc[i], d);
            d = (warp_sum(d) + qj) * tau;
            if (lane == 0) qc[j] = qj - d;
            for (uint32_t i = j + 1 + lane; i < mm; i += 32) qc[i] = fma(-d, vj[i], qc[i]);
            __syncwarp();
        }
        if (J.lq)  // Q = Q'^T (k x n, ld k)
            for (uint32_t i = lane; i < mm; i += 32) qo[c + uint64_t(i) * k] = qc[i];
        else
            for (uint32_t i = lane; i < mm; i += 32) qo[i + uint64_t(c) * mm] = qc[i];
    }
}

__host__ __device__ inline uint64_t qr_one_size(uint32_t m, uint32_t n) { return uint64_t(m) * n + (m < n ? m : n); }

// An unpivoted factorisation by one CTA: no pivot is looked for and nothing is exchanged, so a step is the norm of its
// column, the reflector in place of it, and the trailing columns, one warp each.  Against k_qr with one CTA, which finds
// the norms of all columns and keeps its reflectors in L2: 100 x 100 0.57 against 0.73 ms, 48 x 48 0.21 against 0.26 ms,
// 20 x 400 0.25 against 0.39 ms (whole calls).  Pivoted blocks are the faster in k_qr.  SMEM: the work matrix is in shared
// memory; else in the block's scratch, by all the CTA's 1024 threads, a number known to the compiler (75 blocks of
// 256 x 256: 4.7 ms, 5.3 ms without).
template <bool SMEM>
__global__ void __launch_bounds__(QR_THR) k_qr_one(const QrJob* __restrict__ jobs, const double* __restrict__ A, double* __restrict__ Q,
                                                   double* __restrict__ R, double* __restrict__ W) {
    extern __shared__ double qsm[];
    __shared__ double red[QR_WARPS];
    __shared__ double sh_tau, sh_scale, sh_thr;
    __shared__ int sh_zero;
    const QrJob J = jobs[blockIdx.x];
    const uint32_t nthr = SMEM ? blockDim.x : QR_THR, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarp = nthr / 32;
    // the matrix factorised: F (mm x nn) = A_j, or A_j^T for an LQ
    const uint32_t mm = J.lq ? J.n : J.m, nn = J.lq ? J.m : J.n, k = mm < nn ? mm : nn;
    // F, then R above and the reflectors below the diagonal, with the k reflector scales after it
    const uint64_t fsz = qr_one_size(mm, nn);
    double* w = SMEM ? qsm : W + J.w_off;
    double* taus = w + uint64_t(mm) * nn;
    const double* a = A + J.a_off;
    double f = 0.0;
    for (uint64_t e = tid; e < uint64_t(mm) * nn; e += nthr) {
        const uint32_t i = uint32_t(e % mm), c = uint32_t(e / mm);
        const double x = J.lq ? a[c + uint64_t(i) * J.m] : a[i + uint64_t(c) * J.m];
        w[e] = x;
        f = fma(x, x, f);
    }
    // sum over the CTA in thread 0; red is free again after the barrier that follows
    auto cta_sum = [&](double v) {
        v = warp_sum(v);
        if (lane == 0) red[warp] = v;
        __syncthreads();
        double t = 0.0;
        if (tid == 0)
            for (uint32_t q = 0; q < nwarp; ++q) t += red[q];
        return t;
    };
    f = cta_sum(f);
    if (tid == 0) sh_thr = 64.0 * 2.220446049250313e-16 * sqrt(f);  // negligible columns: 64 eps |A|_F
    __syncthreads();
    for (uint32_t j = 0; j < k; ++j) {
        double* vj = w + uint64_t(j) * mm;
        double s = 0.0;
        for (uint32_t i = j + 1 + tid; i < mm; i += nthr) s = fma(vj[i], vj[i], s);
        s = cta_sum(s);
        if (tid == 0) {
            const double alpha = vj[j], xnorm = sqrt(s), nrm = hypot(alpha, xnorm);
            double tau = 0.0, scale = 1.0;
            const int zero = nrm <= sh_thr;
            if (!zero && xnorm != 0.0) {
                const double beta = -copysign(nrm, alpha);
                tau = (beta - alpha) / beta;
                scale = 1.0 / (alpha - beta);
                vj[j] = beta;
            }
            sh_tau = tau;
            sh_scale = scale;
            sh_zero = zero;
            taus[j] = tau;
        }
        __syncthreads();
        const double tau = sh_tau, scale = sh_scale;
        if (sh_zero)  // a negligible column: exactly zero in R, no reflector
            for (uint32_t i = j + tid; i < mm; i += nthr) vj[i] = 0.0;
        if (tau != 0.0) {
            for (uint32_t i = j + 1 + tid; i < mm; i += nthr) vj[i] *= scale;
            __syncthreads();
            // trailing columns, one warp each: F(j:mm, c) -= tau v (v^T F(j:mm, c)), v_j = 1
            for (uint32_t c = j + 1 + warp; c < nn; c += nwarp) {
                double* fc = w + uint64_t(c) * mm;
                const double fj = fc[j];  // read by every lane before lane 0 writes it
                double d = 0.0;
                for (uint32_t i = j + 1 + lane; i < mm; i += 32) d = fma(vj[i], fc[i], d);
                d = (warp_sum(d) + fj) * tau;
                if (lane == 0) fc[j] = fj - d;
                for (uint32_t i = j + 1 + lane; i < mm; i += 32) fc[i] = fma(-d, vj[i], fc[i]);
            }
        }
        __syncthreads();
    }
    // R (k x nn, ld k) from the upper triangle; for an LQ, L = R'^T (m x k, ld m)
    double* r = R + J.r_off;
    for (uint64_t e = tid; e < uint64_t(k) * nn; e += nthr) {
        const uint32_t i = uint32_t(e % k), c = uint32_t(e / k);
        const double v = i <= c ? w[i + uint64_t(c) * mm] : 0.0;
        if (J.lq) r[c + uint64_t(i) * J.m] = v;
        else if (J.flags & QR_RT) r[c + uint64_t(i) * nn] = v;
        else r[e] = v;
    }
    // Q' = H_0 ... H_{k-1} I(:, 0:k), the reflectors applied from the last to the first; an LQ's in the scratch first
    double* qf = W + J.w_off + fsz;
    double* qo = J.lq ? qf : Q + J.q_off;
    for (uint64_t e = tid; e < uint64_t(mm) * k; e += nthr) {
        const uint32_t i = uint32_t(e % mm), c = uint32_t(e / mm);
        qo[e] = i == c ? 1.0 : 0.0;
    }
    __syncthreads();
    for (int jj = int(k) - 1; jj >= 0; --jj) {
        const uint32_t j = uint32_t(jj);
        const double tau = taus[j];
        if (tau != 0.0) {
            const double* vj = w + uint64_t(j) * mm;
            for (uint32_t c = j + warp; c < k; c += nwarp) {
                double* qc = qo + uint64_t(c) * mm;
                const double qj = qc[j];
                double d = 0.0;
                for (uint32_t i = j + 1 + lane; i < mm; i += 32) d = fma(vj[i], qc[i], d);
                d = (warp_sum(d) + qj) * tau;
                if (lane == 0) qc[j] = qj - d;
                for (uint32_t i = j + 1 + lane; i < mm; i += 32) qc[i] = fma(-d, vj[i], qc[i]);
            }
        }
        __syncthreads();
    }
    if (J.lq)  // Q = Q'^T (k x n, ld k)
        for (uint64_t e = tid; e < uint64_t(mm) * k; e += nthr) {
            const uint32_t i = uint32_t(e % mm), c = uint32_t(e / mm);
            Q[J.q_off + c + uint64_t(i) * k] = qf[e];
        }
}

__global__ void k_permute_rows(const PermJob* __restrict__ jobs, const double* __restrict__ src, double* __restrict__ dst,
                               const uint32_t* __restrict__ perm) {
    const PermJob J = jobs[blockIdx.x];
    const uint64_t n2 = uint64_t(J.n) * J.n;
    for (uint64_t e = threadIdx.x; e < n2; e += blockDim.x) {
        const uint32_t i = uint32_t(e % J.n), j = uint32_t(e / J.n);
        dst[J.dst_off + perm[J.p_off + i] + uint64_t(j) * J.ldd] = src[J.src_off + e];
    }
}

}  // namespace

void batched_permute_rows(const std::vector<PermJob>& jobs, const double* src, uint64_t src_len, double* dst, uint64_t dst_len,
                          const uint32_t* perm, uint64_t p_len, DBuf<PermJob>& jobbuf, cudaStream_t s) {
    if (jobs.empty()) return;
    for (const PermJob& j : jobs) {
        const uint64_t n = j.n;
        if (!n || j.ldd < n || j.src_off + n * n > src_len || j.dst_off + (n - 1) * j.ldd + n > dst_len || j.p_off + n > p_len)
            throw std::runtime_error("row permutation: a block outside its buffers");
    }
    jobbuf.upload(jobs, s);
    k_permute_rows<<<unsigned(jobs.size()), 256, 0, s>>>(jobbuf.get(), src, dst, perm);
    QCM_CUDA(cudaGetLastError());
}

uint64_t qr_scratch(uint32_t m, uint32_t n, bool) {
    // reflectors, and per CTA its fixed part and columns (both rounded up), as k_qr lays them out; F is A or A^T, and the
    // cluster may have to be smaller than it would best be.  k_qr_one's F, scales and Q' (mm nn + k + mm k) are less.
    const uint64_t k = std::min(m, n);
    uint64_t d = 0;
    for (auto [mm, nn] : {std::pair<uint32_t, uint32_t>{m, n}, {n, m}}) {
        for (uint32_t nc = qr_cluster(mm, nn); nc; nc /= 2) {
            const QrLayout l = qr_layout(mm, nn, nc, 0);
            d = std::max<uint64_t>(d, uint64_t(mm) * k + nc * (l.fixed + uint64_t(l.ncol) * mm));
        }
    }
    return d;
}

void batched_qr(const std::vector<QrJob>& jobs, const double* A, uint64_t a_len, double* Q, uint64_t q_len, double* R,
                uint64_t r_len, double* W, uint64_t w_len, DBuf<QrJob>& jobbuf, std::unique_ptr<SideStreams>& side,
                cudaStream_t s, uint32_t max_cluster, uint32_t* P, uint64_t p_len) {
    if (jobs.empty()) return;
    // attributes belong to the functions, for all contexts and host threads: the same values on every call
    for (const void* k : {reinterpret_cast<const void*>(&k_qr), reinterpret_cast<const void*>(&k_qr_one<true>)})
        QCM_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, int(QR_SMEM_DOUBLES * sizeof(double))));
    // time of a block in us by the cluster's size: k steps of a fixed part and of the trailing matrix and Q, dealt out (from
    // single pivoted blocks of 115 to 512 columns, within a fifth)
    std::vector<std::array<double, N_CLUSTER_SIZES>> cost(jobs.size());
    std::vector<uint8_t> size(jobs.size(), 0);
    bool split = false;
    for (std::size_t b = 0; b < jobs.size(); ++b) {
        const QrJob& j = jobs[b];
        const uint32_t mm = j.lq ? j.n : j.m, nn = j.lq ? j.m : j.n;
        while ((2u << size[b]) <= qr_cluster(mm, nn)) ++size[b];
        split = split || size[b];
        for (int i = 0; i < N_CLUSTER_SIZES; ++i)
            cost[b][i] = std::min(mm, nn) * ((i || (j.flags & QR_PIVOT) ? 3.5 : 2.0) + 0.31e-3 * mm * nn / (1 << i));
    }
    if (split) {
        QCM_CUDA(cudaFuncSetAttribute(k_qr, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        size = plan_clusters(cost, size, cluster_slots(reinterpret_cast<const void*>(&k_qr), QR_THR, QR_SMEM_DOUBLES * sizeof(double), max_cluster));
    }
    // 16, 8, 4, 2, 1 CTAs per block, and one CTA unpivoted beyond and in shared memory: a launch each
    constexpr int ONE_L2 = N_CLUSTER_SIZES, ONE = ONE_L2 + 1, NCLS = ONE + 1;
    static_assert(QR_MAX_CLUSTER >> (N_CLUSTER_SIZES - 1) == 1 && SideStreams::N >= NCLS - 1, "a stream per class");
    std::vector<QrJob> cls[NCLS];
    for (std::size_t b = 0; b < jobs.size(); ++b) {
        const QrJob& j = jobs[b];
        const uint64_t k = std::min(j.m, j.n);
        if (!j.m || !j.n || j.a_off + uint64_t(j.m) * j.n > a_len || j.w_off + qr_scratch(j.m, j.n, j.lq != 0) > w_len ||
            j.q_off + k * (j.lq ? j.n : j.m) > q_len || j.r_off + k * (j.lq ? j.m : j.n) > r_len)
            throw std::runtime_error("batched QR: a block outside its buffers");
        const uint32_t nn = j.lq ? j.m : j.n;
        if ((j.flags & QR_RT) && j.lq) throw std::runtime_error("batched QR: a transposed R is for a QR, not an LQ");
        if ((j.flags & QR_PIVOT) && (!P || nn > QR_PIV_MAX || j.p_off + nn > p_len))
            throw std::runtime_error("batched QR: pivoting needs a permutation buffer and at most 1024 columns");
        int i = N_CLUSTER_SIZES - 1 - size[b];
        if (!size[b] && !(j.flags & QR_PIVOT)) i = qr_one_size(j.m, j.n) > QR_SMEM_DOUBLES ? ONE_L2 : ONE;
        cls[i].push_back(j);
    }
    std::vector<QrJob> all;
    int used = 0;
    for (auto& v : cls) {
        // within a launch the largest blocks first
        std::stable_sort(v.begin(), v.end(), [](const QrJob& x, const QrJob& y) {
            return uint64_t(x.m) * x.n > uint64_t(y.m) * y.n;
        });
        all.insert(all.end(), v.begin(), v.end());
        used += !v.empty();
    }
    jobbuf.upload(all, s);
    if (used > 1 && !side) side = std::make_unique<SideStreams>();
    if (used > 1) side->fork(s);
    std::size_t first = 0;
    int lane = -1;  // the first launch stays on s
    cudaError_t err = cudaSuccess;
    for (int i = 0; i < NCLS && err == cudaSuccess; ++i) {
        if (cls[i].empty()) continue;
        const cudaStream_t st = lane < 0 ? s : side->s[lane];
        if (i >= ONE_L2) {
            // shared memory of the largest work matrix, a warp per column and a thread per row
            uint64_t sm = 0, thr = 0;
            for (const QrJob& j : cls[i]) {
                if (i == ONE) sm = std::max(sm, qr_one_size(j.m, j.n));
                thr = std::max<uint64_t>(thr, std::max(32 * uint64_t(j.lq ? j.m : j.n), uint64_t(j.lq ? j.n : j.m)));
            }
            thr = i == ONE_L2 ? QR_THR : std::min<uint64_t>(QR_THR, std::max<uint64_t>(128, (thr + 127) / 128 * 128));
            auto* kernel = i == ONE ? k_qr_one<true> : k_qr_one<false>;
            kernel<<<unsigned(cls[i].size()), unsigned(thr), std::size_t(sm) * sizeof(double), st>>>(jobbuf.get() + first, A, Q, R, W);
            err = cudaGetLastError();
            first += cls[i].size();
            ++lane;
            continue;
        }
        const uint32_t nc = QR_MAX_CLUSTER >> i;
        uint64_t sm = 0;
        uint32_t lanes = 0;  // a warp per column, a thread per row
        for (const QrJob& j : cls[i]) {
            const uint32_t mm = j.lq ? j.n : j.m, nn = j.lq ? j.m : j.n;
            const QrLayout l = qr_layout(mm, nn, nc, QR_SMEM_DOUBLES);
            if (l.fixed_smem) sm = std::max(sm, l.fixed + (l.cols_smem ? uint64_t(l.ncol) * mm : 0));
            lanes = std::max(lanes, std::max(l.ncol * 32, mm));
        }
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(unsigned(cls[i].size()) * nc);
        cfg.blockDim = dim3(std::min<uint32_t>(QR_THR, std::max<uint32_t>(128, (std::min<uint32_t>(lanes, QR_THR) + 127) / 128 * 128)));
        cfg.dynamicSmemBytes = std::size_t(sm) * sizeof(double);
        cfg.stream = st;
        cudaLaunchAttribute at{};
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = nc;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        err = cudaLaunchKernelEx(&cfg, k_qr, static_cast<const QrJob*>(jobbuf.get() + first), A, Q, R, W, P, uint32_t(sm));
        first += cls[i].size();
        ++lane;
    }
    if (used > 1) side->join(s);  // after a failed launch too: the others still use the buffers
    QCM_CUDA(err);
}

}  // namespace qcm
