// One-sided Jacobi SVD (Hestenes) of many blocks, each by a cluster of 1 to 16 CTAs (see linalg.hpp).
//
// G (r x c, ld r) is A when m >= n and A^T otherwise; its columns are rotated pairwise until mutually
// orthogonal, and the rotations accumulate in Q (c x c, starting at I).  Then G = Vg diag(sigma) with
// sigma_j = |G_j|, and A = G Q^T (m >= n: U = G / sigma, V = Q) or A^T = G Q^T (m < n: U = Q, V = G / sigma).
// Column pairs follow the circle (round-robin) ordering, c' - 1 rounds of c'/2 disjoint pairs per sweep
// (c' = c rounded up to even, pairs with the padding column skipped): gamma = G_p . G_q with
// alpha = |G_p|^2, beta = |G_q|^2 tracked in shared memory (recomputed at the start of every sweep, updated
// exactly by alpha -= t gamma, beta += t gamma after a rotation), and if |gamma| > r eps sqrt(alpha beta)
// (the rounding level of a length-r dot product) the rotation with t = sign(zeta) / (|zeta| +
// sqrt(1 + zeta^2)), zeta = (beta - alpha) / (2 gamma), c = rsqrt(1 + t^2), s = c t makes them orthogonal.
// Sweeps end when one performs no rotation (at most JMAX_SWEEPS).
//
// The rows of G and Q are split over the CTAs of the cluster: a round moves ten column lengths per pair
// through shared memory (dot product, two rotations), which binds one SM at 128 B per clock, and rows are
// what can be split without moving columns between SMs.  Each round every CTA sends its partial dot products
// to all of them (distributed shared memory), and after one cluster barrier each CTA adds the partials in rank
// order and derives the same rotations, one thread per pair.  A second cluster barrier per round (the partials
// may be overwritten) is split: it is arrived at before the rotations and waited for after them.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <stdexcept>
#include <string>

#include "linalg.hpp"

namespace cg = cooperative_groups;

namespace qcm {
namespace {

constexpr int JTHR = 1024;
constexpr int JMAX_SWEEPS = 40;
constexpr double JEPS = 2.220446049250313e-16;  // unit roundoff of double
constexpr uint32_t JSMEM_DOUBLES = 28800;       // dynamic shared memory per CTA (225 KiB of the 227)
constexpr uint32_t JMAX_COLS = 1024;
constexpr uint32_t JMAX_CLUSTER = 16;

// Where a block's work arrays live in a cluster of nc CTAs: per CTA hr rows of G and hq rows of Q (even, so
// that columns start on 16 bytes), each in shared memory if it fits there after the fixed part (norms, rotation
// angles, partial dot products, ranks), else in the block's scratch (L2-resident).
struct JacobiLayout {
    uint32_t hr, hq, fixed;
    bool g_smem, q_smem;
};
__host__ __device__ inline JacobiLayout jacobi_layout(uint32_t r, uint32_t c, uint32_t nc, uint32_t smem_doubles) {
    JacobiLayout l;
    l.hr = ((r + nc - 1) / nc + 1) / 2 * 2;
    l.hq = ((c + nc - 1) / nc + 1) / 2 * 2;
    const uint32_t np = (c + 1) / 2;
    l.fixed = (c + 2 * np + nc * np + (c + 1) / 2 + 3) / 2 * 2;
    const uint64_t g = uint64_t(l.hr) * c, q = uint64_t(l.hq) * c;
    l.g_smem = l.fixed + g <= smem_doubles;
    l.q_smem = l.g_smem && l.fixed + g + q <= smem_doubles;
    return l;
}

// CTAs per block: about 36 rows of each column per CTA.  There a round's shared-memory time (under 1 us up to
// 100 columns, 2 us at 500) is near its fixed part (barriers, square root and division chain); splitting
// further only adds CTAs that wait.
inline uint32_t jacobi_cluster(uint32_t r, uint32_t c) {
    if (c <= 48) return 1;
    const uint32_t rows = std::max(r, c);
    uint32_t nc = 2;
    while (nc < JMAX_CLUSTER && rows > 36 * nc) nc *= 2;
    return nc;
}

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory"); }

__device__ __forceinline__ double warp_sum(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
// sum over each aligned group of gs lanes (all 32 lanes call it)
__device__ __forceinline__ double group_sum(double v, uint32_t gs) {
    for (uint32_t o = gs >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, int(o));
    return v;
}

// columns of pair t in round k of the circle ordering of cp players; false if one is the padding column
__device__ __forceinline__ bool pair_of(uint32_t t, uint32_t k, uint32_t cp, uint32_t c, uint32_t& p, uint32_t& q) {
    // (i - 1 + k) mod (cp - 1) + 1 with i - 1 + k < 2 (cp - 1)
    uint32_t xp = t - 1 + k, xq = cp - 2 - t + k;
    xp -= xp >= cp - 1 ? cp - 1 : 0u;
    xq -= xq >= cp - 1 ? cp - 1 : 0u;
    p = t == 0 ? 0 : xp + 1;
    q = xq + 1;
    return p < c && q < c;
}

// x, y: 2 n2 elements of two columns; x = cs x - sn y, y = sn x + cs y by the lanes of a group
__device__ __forceinline__ void rotate(double2* x, double2* y, uint32_t n2, double cs, double sn, uint32_t hl, uint32_t gs) {
    for (uint32_t i = hl; i < n2; i += gs) {
        const double2 a = x[i], b = y[i];
        x[i] = make_double2(cs * a.x - sn * b.x, cs * a.y - sn * b.y);
        y[i] = make_double2(sn * a.x + cs * b.x, sn * a.y + cs * b.y);
    }
}

__global__ void __launch_bounds__(JTHR) k_jacobi_svd(const SvdJob* __restrict__ jobs, const double* __restrict__ A,
                                                     double* __restrict__ U, double* __restrict__ S, double* __restrict__ V,
                                                     double* __restrict__ Wg, uint32_t smem_doubles,
                                                     int* __restrict__ zero_count, int* __restrict__ sweeps_used) {
    extern __shared__ __align__(16) double smem[];
    __shared__ int rotated;
    cg::cluster_group cl = cg::this_cluster();
    const uint32_t nc = cl.num_blocks(), rank = cl.block_rank();
    const SvdJob J = jobs[blockIdx.x / nc];
    const bool tall = J.m >= J.n;
    const uint32_t r = tall ? J.m : J.n, c = tall ? J.n : J.m;
    const JacobiLayout l = jacobi_layout(r, c, nc, smem_doubles);
    const uint32_t hr = l.hr, hq = l.hq, cp = c + (c & 1u), np = cp / 2;
    double* nrm = smem;         // c
    double* rcs = nrm + c;      // np, then np sines
    double* rsn = rcs + np;
    double* part = rsn + np;    // nc x np partial dot products, by rank
    uint32_t* rank_of = reinterpret_cast<uint32_t*>(part + nc * np);  // c
    double* scratch = Wg + J.w_off + uint64_t(rank) * (hr + hq) * c;
    double* G = l.g_smem ? smem + l.fixed : scratch;
    double* Q = l.q_smem ? smem + l.fixed + uint64_t(hr) * c : scratch + uint64_t(hr) * c;
    const uint32_t nthr = blockDim.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarp = nthr / 32;
    const uint32_t r0 = rank * hr, q0 = rank * hq;  // first rows of this CTA
    // G = A or A^T, Q = I
    const double* a = A + J.a_off;
    for (uint32_t i = tid; i < hr * c; i += nthr) {
        const uint32_t col = i / hr, row = r0 + (i - col * hr);
        G[i] = row >= r ? 0.0 : (tall ? a[row + uint64_t(col) * J.m] : a[col + uint64_t(row) * J.m]);
    }
    for (uint32_t i = tid; i < hq * c; i += nthr) {
        const uint32_t col = i / hq;
        Q[i] = q0 + (i - col * hq) == col ? 1.0 : 0.0;
    }
    __syncthreads();
    const double tol2 = (JEPS * double(r)) * (JEPS * double(r));
    auto cluster_sync = [&] {
        if (nc > 1) {
            cluster_arrive();
            cluster_wait();
        } else {
            __syncthreads();
        }
    };
    // a value of rank `rank` at part[rank][t] of every CTA, written by the first nc of the group's lanes
    auto send = [&](uint32_t t, double v, uint32_t hl, uint32_t gs) {
        if (nc == 1) {
            if (hl == 0) part[t] = v;
            return;
        }
        for (uint32_t d = hl; d < nc; d += gs) cl.map_shared_rank(part, d)[rank * np + t] = v;
    };
    auto gather = [&](uint32_t t) {
        double s = part[t];
        for (uint32_t d = 1; d < nc; ++d) s += part[d * np + t];
        return s;
    };
    // nrm[j] = |G_j|^2 over all rows, half the columns at a time (the partials' buffer holds np values)
    auto column_norms = [&] {
        for (uint32_t j0 = 0; j0 < c; j0 += np) {
            const uint32_t j1 = min(c, j0 + np);
            for (uint32_t j = j0 + warp; j < j1; j += nwarp) {
                const double* g = G + uint64_t(j) * hr;
                double x = 0.0;
                for (uint32_t i = lane; i < hr; i += 32) x = fma(g[i], g[i], x);
                send(j - j0, warp_sum(x), lane, 32);
            }
            cluster_sync();
            for (uint32_t j = j0 + tid; j < j1; j += nthr) nrm[j] = gather(j - j0);
            cluster_sync();
        }
    };
    // lanes per pair: enough groups for all pairs of a round in one pass if the columns are long enough to
    // keep the lanes busy (two elements per lane and step)
    uint32_t gs = 16;
    while (gs > 4 && (np * gs > nthr || hr / 2 < gs)) gs >>= 1;
    const uint32_t grp = tid / gs, hl = tid % gs, ngrp = nthr / gs;
    for (int sweep = 0; sweep < JMAX_SWEEPS && c > 1; ++sweep) {
        if (tid == 0) rotated = 0;
        column_norms();
        for (uint32_t k = 0; k + 1 < cp; ++k) {
            // every lane runs the same number of passes so the group shuffles never diverge
            for (uint32_t pass = 0; pass * ngrp < np; ++pass) {
                const uint32_t t = pass * ngrp + grp;
                uint32_t p = 0, q = 0;
                const bool act = t < np && pair_of(t, k, cp, c, p, q);
                double ga = 0.0;
                if (act) {
                    const double2* gp = reinterpret_cast<const double2*>(G + uint64_t(p) * hr);
                    const double2* gq = reinterpret_cast<const double2*>(G + uint64_t(q) * hr);
                    double g2 = 0.0;
                    for (uint32_t i = hl; i < hr / 2; i += gs) {
                        const double2 x = gp[i], y = gq[i];
                        ga = fma(x.x, y.x, ga);
                        g2 = fma(x.y, y.y, g2);
                    }
                    ga += g2;
                }
                ga = group_sum(ga, gs);
                if (pass == 0 && k > 0 && nc > 1) cluster_wait();  // the previous round's partials have been read
                if (act) send(t, ga, hl, gs);
            }
            cluster_sync();
            for (uint32_t t = tid; t < np; t += nthr) {
                uint32_t p = 0, q = 0;
                double cs = 1.0, sn = 0.0;
                if (pair_of(t, k, cp, c, p, q)) {
                    const double ga = gather(t), al = nrm[p], be = nrm[q];
                    if (ga * ga > tol2 * (al * be)) {
                        // t = sign(zeta) / (|zeta| + sqrt(1 + zeta^2)), zeta = d / h, d = beta - alpha, h = 2 gamma,
                        // multiplied through by |h| (one square root and one division) unless d^2 + h^2 could
                        // overflow
                        const double d = be - al, h = 2.0 * ga;
                        double tt;
                        if (fabs(d) < 1e150 && fabs(h) < 1e150) {
                            tt = (d >= 0.0 ? h : -h) / (fabs(d) + sqrt(fma(d, d, h * h)));
                        } else {
                            const double zeta = d / h;
                            tt = (zeta >= 0.0 ? 1.0 : -1.0) / (fabs(zeta) + sqrt(1.0 + zeta * zeta));
                        }
                        cs = rsqrt(1.0 + tt * tt);
                        sn = cs * tt;
                        nrm[p] = al - tt * ga;
                        nrm[q] = be + tt * ga;
                        rotated = 1;
                    }
                }
                rcs[t] = cs;
                rsn[t] = sn;
            }
            __syncwarp();
            if (nc > 1) cluster_arrive();  // waited for before the next partials are sent
            __syncthreads();
            for (uint32_t t = grp; t < np; t += ngrp) {
                const double cs = rcs[t], sn = rsn[t];
                uint32_t p, q;
                if ((cs == 1.0 && sn == 0.0) || !pair_of(t, k, cp, c, p, q)) continue;
                rotate(reinterpret_cast<double2*>(G + uint64_t(p) * hr), reinterpret_cast<double2*>(G + uint64_t(q) * hr),
                       hr / 2, cs, sn, hl, gs);
                rotate(reinterpret_cast<double2*>(Q + uint64_t(p) * hq), reinterpret_cast<double2*>(Q + uint64_t(q) * hq),
                       hq / 2, cs, sn, hl, gs);
            }
            __syncthreads();
        }
        if (nc > 1) cluster_wait();
        const int any = rotated;
        __syncthreads();
        if (sweeps_used && rank == 0 && tid == 0) sweeps_used[J.id] = sweep + 1;
        if (!any) break;
    }
    // sigma_j = |G_j| and its rank in descending order (ties by index)
    column_norms();
    for (uint32_t j = tid; j < c; j += nthr) nrm[j] = sqrt(nrm[j]);
    __syncthreads();
    double* sv = S + J.s_off;
    int zeros = 0;
    for (uint32_t j = tid; j < c; j += nthr) {
        const double x = nrm[j];
        uint32_t rk = 0;
        for (uint32_t i = 0; i < c; ++i) {
            const double y = nrm[i];
            rk += (y > x || (y == x && i < j)) ? 1u : 0u;
        }
        rank_of[j] = rk;
        if (rank == 0) {
            sv[rk] = x;
            zeros += x == 0.0 ? 1 : 0;
        }
    }
    if (zeros) atomicAdd(zero_count + J.id, zeros);
    __syncthreads();
    // outputs in sorted order: this CTA's rows of the normalised G columns and of Q's columns
    double* Gout = tall ? U + J.u_off : V + J.v_off;   // r x c, ld r
    double* Qout = tall ? V + J.v_off : U + J.u_off;   // c x c, ld c
    for (uint32_t i = tid; i < hr * c; i += nthr) {
        const uint32_t col = i / hr, row = r0 + (i - col * hr);
        if (row >= r) continue;
        const double sg = nrm[col];
        Gout[row + uint64_t(rank_of[col]) * r] = sg > 0.0 ? G[i] / sg : 0.0;
    }
    for (uint32_t i = tid; i < hq * c; i += nthr) {
        const uint32_t col = i / hq, row = q0 + (i - col * hq);
        if (row < c) Qout[row + uint64_t(rank_of[col]) * c] = Q[i];
    }
}

}  // namespace

SideStreams::SideStreams() {
    QCM_CUDA(cudaEventCreateWithFlags(&fork_ev, cudaEventDisableTiming));
    for (int i = 0; i < N; ++i) {
        QCM_CUDA(cudaStreamCreateWithFlags(&s[i], cudaStreamNonBlocking));
        QCM_CUDA(cudaEventCreateWithFlags(&done[i], cudaEventDisableTiming));
    }
}

SideStreams::~SideStreams() {
    for (int i = 0; i < N; ++i) {
        if (done[i]) cudaEventDestroy(done[i]);
        if (s[i]) cudaStreamDestroy(s[i]);
    }
    if (fork_ev) cudaEventDestroy(fork_ev);
}

void SideStreams::fork(cudaStream_t from) {
    QCM_CUDA(cudaEventRecord(fork_ev, from));
    for (cudaStream_t x : s) QCM_CUDA(cudaStreamWaitEvent(x, fork_ev, 0));
}

void SideStreams::join(cudaStream_t to) {
    for (int i = 0; i < N; ++i) {
        QCM_CUDA(cudaEventRecord(done[i], s[i]));
        QCM_CUDA(cudaStreamWaitEvent(to, done[i], 0));
    }
}

uint64_t jacobi_svd_scratch(uint32_t m, uint32_t n) {
    const uint64_t r = std::max(m, n), c = std::min(m, n);
    const uint64_t d = (r + c + 4 * JMAX_CLUSTER) * c;  // every CTA's rows rounded up to even
    return (d + 31) / 32 * 32;  // whole multiples of 32 doubles: the next block's scratch stays 16-byte aligned
}

void batched_jacobi_svd(const std::vector<SvdJob>& jobs, const double* A, uint64_t a_len, double* U, uint64_t u_len, double* S,
                        uint64_t s_len, double* V, uint64_t v_len, double* W, uint64_t w_len, int* zero_count,
                        DBuf<SvdJob>& jobbuf, std::unique_ptr<SideStreams>& side, cudaStream_t s, int* sweeps_used) {
    // one launch per cluster size, the largest first (they take longest), each on a stream of its own
    constexpr int NCLS = 5;  // 16, 8, 4, 2, 1 CTAs per block
    static_assert(JMAX_CLUSTER >> (NCLS - 1) == 1 && SideStreams::N >= NCLS - 1, "a stream per class");
    std::vector<SvdJob> cls[NCLS];
    uint32_t nid = 0;
    for (const SvdJob& j : jobs) {
        nid = std::max(nid, j.id + 1);
        const uint64_t k = std::min(j.m, j.n);
        if (!j.m || !j.n) continue;
        if (k > JMAX_COLS) throw std::runtime_error("batched_jacobi_svd: block larger than 1024 in both dimensions");
        if (j.a_off + uint64_t(j.m) * j.n > a_len || j.u_off + uint64_t(j.m) * k > u_len || j.s_off + k > s_len ||
            j.v_off + uint64_t(j.n) * k > v_len || j.w_off + jacobi_svd_scratch(j.m, j.n) > w_len)
            throw std::runtime_error("batched_jacobi_svd: block outside its buffers");
        if (j.w_off % 2) throw std::runtime_error("batched_jacobi_svd: scratch offset not 16-byte aligned");
        if (uint64_t(j.m) * j.n > 0x7fffffffu) throw std::runtime_error("batched_jacobi_svd: block too large");
        const uint32_t nc = jacobi_cluster(std::max(j.m, j.n), uint32_t(k));
        int i = 0;
        for (uint32_t x = JMAX_CLUSTER; x > nc; x /= 2) ++i;
        cls[i].push_back(j);
    }
    if (nid) QCM_CUDA(cudaMemsetAsync(zero_count, 0, nid * sizeof(int), s));
    std::vector<SvdJob> all;
    int used = 0;
    for (auto& v : cls) {
        // within a launch the largest blocks first
        std::stable_sort(v.begin(), v.end(), [](const SvdJob& x, const SvdJob& y) {
            return uint64_t(x.m) * x.n > uint64_t(y.m) * y.n;
        });
        all.insert(all.end(), v.begin(), v.end());
        used += !v.empty();
    }
    if (all.empty()) return;
    jobbuf.upload(all, s);
    QCM_CUDA(cudaFuncSetAttribute(k_jacobi_svd, cudaFuncAttributeMaxDynamicSharedMemorySize, int(JSMEM_DOUBLES * sizeof(double))));
    QCM_CUDA(cudaFuncSetAttribute(k_jacobi_svd, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    if (used > 1 && !side) side = std::make_unique<SideStreams>();
    if (used > 1) side->fork(s);
    std::size_t first = 0;
    int lane = -1;  // the first launch stays on s
    cudaError_t err = cudaSuccess;
    for (int i = 0; i < NCLS && err == cudaSuccess; ++i) {
        if (cls[i].empty()) continue;
        const uint32_t nc = JMAX_CLUSTER >> i;
        // shared memory of the launch's largest block (everything that fits), threads by its pairs per round
        uint64_t sm = 0;
        uint32_t lanes = 0;
        for (const SvdJob& j : cls[i]) {
            const uint32_t r = std::max(j.m, j.n), c = std::min(j.m, j.n);
            const JacobiLayout l = jacobi_layout(r, c, nc, JSMEM_DOUBLES);
            sm = std::max(sm, l.fixed + (l.g_smem ? uint64_t(l.hr) * c : 0) + (l.q_smem ? uint64_t(l.hq) * c : 0));
            lanes = std::max(lanes, (c + 1) / 2 * 8);
        }
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(unsigned(cls[i].size()) * nc);
        cfg.blockDim = dim3(std::min<uint32_t>(JTHR, std::max<uint32_t>(128, (lanes + 127) / 128 * 128)));
        cfg.dynamicSmemBytes = std::size_t(sm) * sizeof(double);
        cfg.stream = lane < 0 ? s : side->s[lane];
        cudaLaunchAttribute at{};
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = nc;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        err = cudaLaunchKernelEx(&cfg, k_jacobi_svd, static_cast<const SvdJob*>(jobbuf.get() + first), A, U, S, V, W,
                                 uint32_t(sm), zero_count, sweeps_used);
        first += cls[i].size();
        ++lane;
    }
    if (used > 1) side->join(s);  // after a failed launch too: the others still use the buffers
    QCM_CUDA(err);
}

}  // namespace qcm
