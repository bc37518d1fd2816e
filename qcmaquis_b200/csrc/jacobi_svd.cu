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
// order and derives the same rotations, one thread per pair.  The partials have two buffers, used in turn, so that a round
// has one barrier; where G leaves room for one only, a second barrier (the partials may be overwritten) is split: it is
// arrived at before the rotations and waited for after them.
//
// The largest blocks (more than about 420 columns on 16 CTAs) leave no shared memory for Q, and rotating it in L2
// took three quarters of their time.  Nothing in the iteration reads Q, and its rows take the same rotations
// independently of one another: these blocks write their rotations to a log, and k_jacobi_rows applies it to slices
// of rows that fit shared memory, LOG_SWEEPS sweeps at a time.
//
// Measured, the blocks of a two-site truncation at L=24: M=2048 (93 blocks, up to 558 columns) 1265 ms with one CTA per
// block, 76 ms with clusters, 58 ms with the log, two buffers and one CTA up to 88 columns, 55 ms with sizes by the batch;
// M=512 (75 blocks, up to 142) 8.5, 3.2, 2.9 and 2.9 ms.  What is left is a round's chain, 9.3 us at 546 columns.
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
// In a cluster the columns are ldg and ldq apart, 64 bytes off a multiple of 128 if that takes at most a quarter more:
// four lanes read a short column, and two neighbouring columns' lanes then share no bank.
// Two buffers of partials (a round needs no second barrier then), or one if G fits only beside one.
struct JacobiLayout {
    uint32_t hr, hq, ldg, ldq, fixed, nbuf;
    bool g_smem, q_smem;
};
__host__ __device__ inline JacobiLayout jacobi_layout(uint32_t r, uint32_t c, uint32_t nc, uint32_t smem_doubles) {
    JacobiLayout l;
    l.hr = ((r + nc - 1) / nc + 1) / 2 * 2;
    l.hq = ((c + nc - 1) / nc + 1) / 2 * 2;
    const uint32_t np = (c + 1) / 2;
    auto padded = [nc](uint32_t h) {
        const uint32_t p = (h + 7) / 16 * 16 + 8;
        return nc > 1 && 4 * p <= 5 * h ? p : h;
    };
    l.ldg = padded(l.hr);
    l.ldq = padded(l.hq);
    const uint64_t g = uint64_t(l.ldg) * c, q = uint64_t(l.ldq) * c;
    for (l.nbuf = nc > 1 ? 2 : 1;; l.nbuf = 1) {
        l.fixed = (c + 2 * np + l.nbuf * nc * (np + (np & 1u)) + (c + 1) / 2 + 3) / 2 * 2;
        l.g_smem = l.fixed + g <= smem_doubles;
        l.q_smem = l.g_smem && l.fixed + g + q <= smem_doubles;
        if (l.g_smem || l.nbuf == 1) return l;
    }
}

// CTAs per block, alone: about 36 rows of each column per CTA.  There a round's shared-memory time (under 1 us up to
// 100 columns, 2 us at 500) is near its fixed part (barriers, square root chain); splitting further only adds
// CTAs that wait: 36 rows 13.8 ms for the blocks of M=1200, 20 or 24 rows 14.9 ms.  Up to 88 columns one CTA, which has no
// exchange and one barrier a round (clusters from 48 columns on made batches of small blocks 0.87 times as fast).
inline uint32_t jacobi_cluster(uint32_t r, uint32_t c) {
    if (c <= 88) return 1;
    const uint32_t rows = std::max(r, c);
    uint32_t nc = 2;
    while (nc < JMAX_CLUSTER && rows > 36 * nc) nc *= 2;
    return nc;
}
// where a launch's blocks keep their work arrays (known at compile time: shared-memory addresses are a third of the
// kernel's instructions): G and Q in one CTA's shared memory; in a cluster's; G there and Q logged; G in the scratch.
// One CTA has an instance without the exchange: 88 x 88 block 2.51 -> 2.21 ms, 64 x 64 1.21 -> 1.07 ms.
enum JacobiMode { J_ONE, J_SMEM, J_LOGGED, J_LOGGED_L2 };
// the instance that a block needs in a cluster of nc CTAs
inline JacobiMode jacobi_mode(uint32_t r, uint32_t c, uint32_t nc) {
    const JacobiLayout l = jacobi_layout(r, c, nc, JSMEM_DOUBLES);
    return l.q_smem ? (nc == 1 ? J_ONE : J_SMEM) : (l.g_smem ? J_LOGGED : J_LOGGED_L2);
}
// time of a sweep of a block in us: c' - 1 rounds of a fixed part (barriers, exchange, square root chain) and of the
// columns' way through shared memory at 128 bytes a clock, dealt out to the CTAs; 2.4 times that for a G in L2; 1.5 us a
// round for k_jacobi_rows (from single blocks of 64 to 512 columns, within a fifth)
inline double jacobi_cost(uint32_t r, uint32_t c, int log2nc) {
    constexpr double fixed[N_CLUSTER_SIZES] = {0.35, 1.2, 1.2, 1.3, 2.3};
    const JacobiMode m = jacobi_mode(r, c, 1u << log2nc);
    const double np = (c + 1) / 2, way = np / 30400.0 / (1 << log2nc);
    const double logged = m == J_LOGGED || m == J_LOGGED_L2 ? 1.5 : 0.0;
    return (2.0 * np - 1.0) * (fixed[log2nc] + logged + way * (logged > 0.0 ? 6.0 * r * (m == J_LOGGED_L2 ? 2.4 : 1.0) : 6.0 * r + 4.0 * c));
}

constexpr int LOG_SWEEPS = 4;       // sweeps per launch of a logged block
constexpr uint32_t ROWS_SLICE = 16;  // rows of Q per CTA of k_jacobi_rows
constexpr int ROWS_THR = 512;
static_assert(JMAX_SWEEPS % LOG_SWEEPS == 0, "whole launches");
// Logged blocks: log: per block (l_off of its job) LOG_SWEEPS sweeps of c' - 1 rounds of c'/2 rotations (cosine, sine);
// meta: per block of the launch the sweeps of this launch and whether the block is done; launch: their number so far.
struct JacobiLog {
    double2* log;
    int* meta;
    int launch;
};

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

// cosine cs and sine sn of the rotation that makes two columns orthogonal, and t = sn / cs, from their squared norms
// al, be and dot product ga: t = sign(zeta) / (|zeta| + sqrt(1 + zeta^2)), zeta = d / h, d = beta - alpha, h = 2 gamma,
// multiplied through by |h| unless d^2 + h^2 is outside the range.  cs and sn come from t alone: cs^2 + sn^2 is 1 to the
// last rounding whatever the error of t, and exactly 1 for small t.  Taken straight from two reciprocal square roots
// (1 % faster) they drifted: after 300 columns' rotations the squared column norms were off by 204 eps rms, against
// 17 eps so, and the singular values by 15.8 eps rms, against 1.2.
__device__ __forceinline__ void rotation(double al, double be, double ga, double& cs, double& sn, double& tt) {
    const double d = be - al, h = 2.0 * ga, dh = fma(d, d, h * h);
    if (dh > 1e-280 && dh < 1e300) {
        tt = (d >= 0.0 ? h : -h) / (fabs(d) + sqrt(dh));
    } else {
        const double zeta = d / h;
        tt = (zeta >= 0.0 ? 1.0 : -1.0) / (fabs(zeta) + sqrt(1.0 + zeta * zeta));
    }
    cs = rsqrt(1.0 + tt * tt);
    sn = cs * tt;
}

// dot product of two columns of 2 n2 elements by a group of gs lanes (all 32 lanes call it; x, y only read if act)
__device__ __forceinline__ double group_dot(const double2* x, const double2* y, uint32_t n2, uint32_t hl, uint32_t gs, bool act) {
    double a = 0.0, b = 0.0;
    if (act)
        for (uint32_t i = hl; i < n2; i += gs) {
            const double2 u = x[i], v = y[i];
            a = fma(u.x, v.x, a);
            b = fma(u.y, v.y, b);
        }
    return group_sum(a + b, gs);
}

template <int MODE>
__global__ void __launch_bounds__(JTHR) k_jacobi_svd(const SvdJob* __restrict__ jobs, const double* __restrict__ A,
                                                     double* __restrict__ U, double* __restrict__ S, double* __restrict__ V,
                                                     double* __restrict__ Wg, int* __restrict__ zero_count,
                                                     int* __restrict__ sweeps_used, JacobiLog lg) {
    extern __shared__ __align__(16) double smem[];
    __shared__ int rotated;
    cg::cluster_group cl = cg::this_cluster();
    const uint32_t nc = MODE == J_ONE ? 1 : cl.num_blocks(), rank = MODE == J_ONE ? 0 : cl.block_rank();
    const SvdJob J = jobs[blockIdx.x / nc];
    constexpr bool logged = MODE == J_LOGGED || MODE == J_LOGGED_L2;
    int* meta = lg.meta + 2 * (blockIdx.x / nc);
    if (logged && lg.launch > 0 && meta[1]) return;  // the whole cluster: done in an earlier launch
    const bool tall = J.m >= J.n;
    const uint32_t r = tall ? J.m : J.n, c = tall ? J.n : J.m;
    const JacobiLayout l = jacobi_layout(r, c, nc, JSMEM_DOUBLES);  // as the launch does
    const uint32_t hr = l.hr, hq = l.hq, ldg = l.ldg, ldq = l.ldq, cp = c + (c & 1u), np = cp / 2, npe = np + (np & 1u);
    double2* rot = reinterpret_cast<double2*>(smem);  // np: the round's rotations (cosine, sine)
    double* part = smem + 2 * np;                     // nbuf x nc x npe partial dot products, by rank
    double* nrm = part + l.nbuf * nc * npe;           // c
    uint32_t* rank_of = reinterpret_cast<uint32_t*>(nrm + c);  // c
    double* scratch = Wg + J.w_off + uint64_t(rank) * (ldg + ldq) * c;
    double* G = MODE == J_LOGGED_L2 ? scratch : smem + l.fixed;
    double* Q = smem + l.fixed + ldg * c;  // unless logged
    const uint32_t nthr = blockDim.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarp = nthr / 32;
    const uint32_t r0 = rank * hr, q0 = rank * hq;  // first rows of this CTA
    // G = A or A^T, Q = I (a logged block goes on from the G it left in the scratch)
    const double* a = A + J.a_off;
    if (!logged || lg.launch == 0) {
        for (uint32_t i = tid; i < hr * c; i += nthr) {
            const uint32_t col = i / hr, k = i - col * hr, row = r0 + k;
            G[col * ldg + k] = row >= r ? 0.0 : (tall ? a[row + uint64_t(col) * J.m] : a[col + uint64_t(row) * J.m]);
        }
    } else if (MODE == J_LOGGED) {
        for (uint32_t i = tid; i < ldg * c; i += nthr) G[i] = scratch[i];
    }
    if (!logged)
        for (uint32_t i = tid; i < hq * c; i += nthr) {
            const uint32_t col = i / hq, k = i - col * hq;
            Q[col * ldq + k] = q0 + k == col ? 1.0 : 0.0;
        }
    const double tol2 = (JEPS * double(r)) * (JEPS * double(r));
    auto cluster_sync = [&] {
        if (nc > 1) {
            cluster_arrive();
            cluster_wait();
        } else {
            __syncthreads();
        }
    };
    cluster_sync();  // every CTA of the cluster runs: from here on the others may store into its shared memory
    // An exchange: every CTA's partial of item t goes to its row of the buffer in all CTAs (put, by the group's lanes);
    // after the barrier (arrived) gather adds them in rank order.  With one buffer it may be filled again once all CTAs
    // have gathered: they arrive at a second barrier then (gathered), waited for before the next put (free).
    uint32_t par = 0;  // this exchange's buffer
    auto put = [&](uint32_t t, double v, uint32_t hl, uint32_t gs) {
        double* b = part + (par * nc + rank) * npe + t;
        for (uint32_t d = hl; d < nc; d += gs) *cl.map_shared_rank(b, d) = v;
    };
    auto gather = [&](uint32_t t) {
        const double* b = part + par * nc * npe + t;
        double s = b[0];
        for (uint32_t d = 1; d < nc; ++d) s += b[d * npe];
        return s;
    };
    bool wait_free = false;  // one buffer: the exchange before is still being gathered
    auto free = [&] {
        if (wait_free) cluster_wait();
        wait_free = false;
    };
    auto gathered = [&] {  // all lanes of a warp together
        if (l.nbuf == 2) {
            par ^= 1;
        } else {
            cluster_arrive();
            wait_free = true;
        }
    };
    // nrm[j] = |G_j|^2 over all rows, half the columns at a time (the partials' buffer holds np values)
    auto column_norms = [&] {
        for (uint32_t j0 = 0; j0 < c; j0 += np) {
            const uint32_t j1 = min(c, j0 + np);
            if (nc > 1) free();
            for (uint32_t j = j0 + warp; j < j1; j += nwarp) {
                const double* g = G + j * ldg;
                double x = 0.0;
                for (uint32_t i = lane; i < hr; i += 32) x = fma(g[i], g[i], x);
                x = warp_sum(x);
                if (nc > 1) put(j - j0, x, lane, 32);
                else if (lane == 0) nrm[j] = x;
            }
            cluster_sync();
            if (nc == 1) continue;
            for (uint32_t j = j0 + tid; j < j1; j += nthr) nrm[j] = gather(j - j0);
            __syncwarp();
            gathered();
        }
        __syncthreads();
    };
    // lanes per pair: the least passes over the pairs times steps along a column (two elements per lane), a pass's
    // fixed part counted as four steps
    uint32_t gs = 16;
    for (uint32_t g = 16, best = 0xffffffffu; g >= 4; g >>= 1) {
        const uint32_t cost = (np * g + nthr - 1) / nthr * ((hr / 2 + g - 1) / g + 4);
        if (cost < best) { best = cost; gs = g; }
    }
    const uint32_t grp = tid / gs, hl = tid % gs, ngrp = nthr / gs;
    const int sweep0 = logged ? lg.launch * LOG_SWEEPS : 0, sweep1 = logged ? sweep0 + LOG_SWEEPS : JMAX_SWEEPS;
    int sweep = sweep0;
    bool done = c <= 1;
    for (; sweep < sweep1 && !done; ++sweep) {
        if (tid == 0) rotated = 0;
        double2* lgs = logged ? lg.log + J.l_off + uint64_t(sweep - sweep0) * (cp - 1) * np : nullptr;
        column_norms();
        for (uint32_t k = 0; k + 1 < cp; ++k) {
            // every lane runs the same number of passes so the group shuffles never diverge
            for (uint32_t pass = 0; pass * ngrp < np; ++pass) {
                const uint32_t t = pass * ngrp + grp;
                uint32_t p = 0, q = 0;
                const bool act = t < np && pair_of(t, k, cp, c, p, q);
                double2* gp = reinterpret_cast<double2*>(G + p * ldg);
                double2* gq = reinterpret_cast<double2*>(G + q * ldg);
                const double ga = group_dot(gp, gq, hr / 2, hl, gs, act);
                if (MODE == J_ONE) {
                    // a block of one CTA needs no exchange: each group rotates its pair at once, one barrier a round
                    const double al = act ? nrm[p] : 0.0, be = act ? nrm[q] : 0.0;
                    if (act && ga * ga > tol2 * (al * be)) {
                        double cs, sn, tt;
                        rotation(al, be, ga, cs, sn, tt);
                        rotate(gp, gq, hr / 2, cs, sn, hl, gs);
                        rotate(reinterpret_cast<double2*>(Q + p * ldq), reinterpret_cast<double2*>(Q + q * ldq),
                               hq / 2, cs, sn, hl, gs);
                        if (hl == 0) {
                            nrm[p] = al - tt * ga;
                            nrm[q] = be + tt * ga;
                            rotated = 1;
                        }
                    }
                    __syncwarp();
                    continue;
                }
                if (pass == 0) free();
                if (act) put(t, ga, hl, gs);
            }
            if (MODE == J_ONE) {
                __syncthreads();
                continue;
            }
            cluster_sync();
            for (uint32_t t = tid; t < np; t += nthr) {
                uint32_t p = 0, q = 0;
                double cs = 1.0, sn = 0.0;
                if (pair_of(t, k, cp, c, p, q)) {
                    const double ga = gather(t), al = nrm[p], be = nrm[q];
                    if (ga * ga > tol2 * (al * be)) {
                        double tt;
                        rotation(al, be, ga, cs, sn, tt);
                        nrm[p] = al - tt * ga;
                        nrm[q] = be + tt * ga;
                        rotated = 1;
                    }
                }
                rot[t] = make_double2(cs, sn);
                if (logged && t % nc == rank) lgs[uint64_t(k) * np + t] = make_double2(cs, sn);
            }
            __syncwarp();
            gathered();
            __syncthreads();
            for (uint32_t t = grp; t < np; t += ngrp) {
                const double2 cs = rot[t];
                uint32_t p, q;
                if ((cs.x == 1.0 && cs.y == 0.0) || !pair_of(t, k, cp, c, p, q)) continue;
                rotate(reinterpret_cast<double2*>(G + p * ldg), reinterpret_cast<double2*>(G + q * ldg),
                       hr / 2, cs.x, cs.y, hl, gs);
                if (!logged)
                    rotate(reinterpret_cast<double2*>(Q + p * ldq), reinterpret_cast<double2*>(Q + q * ldq),
                           hq / 2, cs.x, cs.y, hl, gs);
            }
            __syncthreads();
        }
        const int any = rotated;
        __syncthreads();
        done = !any;
    }
    if (sweeps_used && rank == 0 && tid == 0) sweeps_used[J.id] = sweep;
    if (logged) {
        done = done || sweep == JMAX_SWEEPS;
        if (rank == 0 && tid == 0) { meta[0] = sweep - sweep0; meta[1] = done ? 1 : 0; }
        if (!done) {
            if (MODE == J_LOGGED)
                for (uint32_t i = tid; i < ldg * c; i += nthr) scratch[i] = G[i];
            free();
            return;  // every CTA of the cluster has passed its last exchange
        }
    }
    // sigma_j = |G_j| and its rank in descending order (ties by index)
    column_norms();
    free();
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
            if (logged) lg.log[J.l_off + uint64_t(LOG_SWEEPS) * (cp - 1) * np + j].x = double(rk);
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
        const uint32_t col = i / hr, k = i - col * hr, row = r0 + k;
        if (row >= r) continue;
        const double sg = nrm[col];
        Gout[row + uint64_t(rank_of[col]) * r] = sg > 0.0 ? G[col * ldg + k] / sg : 0.0;
    }
    if (logged) return;
    for (uint32_t i = tid; i < hq * c; i += nthr) {
        const uint32_t col = i / hq, k = i - col * hq, row = q0 + k;
        if (row < c) Qout[row + uint64_t(rank_of[col]) * c] = Q[col * ldq + k];
    }
}

// The logged rotations of k_jacobi_svd's last launch applied to ROWS_SLICE rows of Q (grid: slice, block).  Between
// launches Q waits in its output buffer, its columns in their own order; when its block is done they are written
// in the order of the singular values.  One half-warp per pair, a lane per row: the columns of a pair are two
// conflict-free rows of shared memory, whose bandwidth binds.
__global__ void __launch_bounds__(ROWS_THR) k_jacobi_rows(const SvdJob* __restrict__ jobs, double* __restrict__ U,
                                                          double* __restrict__ V, JacobiLog lg, int launch) {
    extern __shared__ __align__(16) double q[];  // [column][ROWS_SLICE]
    const SvdJob J = jobs[blockIdx.y];
    const bool tall = J.m >= J.n;
    const uint32_t c = tall ? J.n : J.m, cp = c + (c & 1u), np = cp / 2;
    const uint32_t row0 = blockIdx.x * ROWS_SLICE;
    const int nsweeps = lg.meta[2 * blockIdx.y], done = lg.meta[2 * blockIdx.y + 1];
    if (row0 >= c || done > 1) return;  // 2: written by an earlier launch
    double* Qout = tall ? V + J.v_off : U + J.u_off;  // c x c, ld c
    const uint32_t lane = threadIdx.x % ROWS_SLICE, grp = threadIdx.x / ROWS_SLICE, ngrp = ROWS_THR / ROWS_SLICE;
    const uint32_t row = row0 + lane;
    for (uint32_t j = grp; j < c; j += ngrp)
        q[j * ROWS_SLICE + lane] = launch == 0 ? (row == j ? 1.0 : 0.0) : (row < c ? Qout[row + uint64_t(j) * c] : 0.0);
    __syncthreads();
    const double2* log = lg.log + J.l_off;
    for (int sweep = 0; sweep < nsweeps; ++sweep)
        for (uint32_t k = 0; k + 1 < cp; ++k) {
            for (uint32_t t = grp; t < np; t += ngrp) {
                const double2 cs = log[t];
                uint32_t p, r;
                if ((cs.x == 1.0 && cs.y == 0.0) || !pair_of(t, k, cp, c, p, r)) continue;
                const double x = q[p * ROWS_SLICE + lane], y = q[r * ROWS_SLICE + lane];
                q[p * ROWS_SLICE + lane] = cs.x * x - cs.y * y;
                q[r * ROWS_SLICE + lane] = cs.y * x + cs.x * y;
            }
            log += np;
            __syncthreads();
        }
    const double2* rank_of = lg.log + J.l_off + uint64_t(LOG_SWEEPS) * (cp - 1) * np;
    if (row < c)
        for (uint32_t j = grp; j < c; j += ngrp)
            Qout[row + uint64_t(done ? uint32_t(rank_of[j].x) : j) * c] = q[j * ROWS_SLICE + lane];
}

// after k_jacobi_rows: blocks that are done are not touched again
__global__ void k_jacobi_mark(int* meta, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n && meta[2 * i + 1]) meta[2 * i + 1] = 2;
}

// log entries of a block (double2): its rotations, then the rank of every column
uint64_t log_entries(uint32_t c) {
    const uint64_t cp = c + (c & 1u);
    return uint64_t(LOG_SWEEPS) * (cp - 1) * (cp / 2) + c;
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
    const uint64_t d = (r + c + 2 * 18 * JMAX_CLUSTER) * c;  // every CTA's rows, padded (at most 17 each)
    return (d + 31) / 32 * 32;  // whole multiples of 32 doubles: the next block's scratch stays 16-byte aligned
}

void batched_jacobi_svd(const std::vector<SvdJob>& jobs, const double* A, uint64_t a_len, double* U, uint64_t u_len, double* S,
                        uint64_t s_len, double* V, uint64_t v_len, double* W, uint64_t w_len, int* zero_count,
                        DBuf<SvdJob>& jobbuf, std::unique_ptr<SideStreams>& side, cudaStream_t s, uint32_t max_cluster,
                        int* sweeps_used) {
    // attributes belong to the functions, for all contexts and host threads: the same values on every call
    auto allow = [](const void* k, std::size_t bytes) {
        QCM_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes)));
    };
    const std::size_t full = JSMEM_DOUBLES * sizeof(double);
    allow(reinterpret_cast<const void*>(&k_jacobi_svd<J_ONE>), full);
    // cluster sizes: alone, or by the batch; blocks whose Q does not fit one want the most
    std::vector<std::array<double, N_CLUSTER_SIZES>> cost(jobs.size());
    std::vector<uint8_t> size(jobs.size(), 0);
    bool split = false;
    for (std::size_t b = 0; b < jobs.size(); ++b) {
        const uint32_t r = std::max(jobs[b].m, jobs[b].n), c = std::min(jobs[b].m, jobs[b].n);
        if (!c) continue;
        if (c > JMAX_COLS) throw std::runtime_error("batched_jacobi_svd: block larger than 1024 in both dimensions");
        if (uint64_t(r) * c > 0x7fffffffu) throw std::runtime_error("batched_jacobi_svd: block too large");
        const uint32_t nc = jacobi_cluster(r, c), want = jacobi_mode(r, c, nc) >= J_LOGGED ? JMAX_CLUSTER : nc;
        while ((2u << size[b]) <= want) ++size[b];
        split = split || size[b];
        for (int i = 0; i < N_CLUSTER_SIZES; ++i) cost[b][i] = jacobi_cost(r, c, i);
    }
    if (split) {
        for (const void* k : {reinterpret_cast<const void*>(&k_jacobi_svd<J_SMEM>), reinterpret_cast<const void*>(&k_jacobi_svd<J_LOGGED>),
                              reinterpret_cast<const void*>(&k_jacobi_svd<J_LOGGED_L2>)}) {
            allow(k, full);
            QCM_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        }
        allow(reinterpret_cast<const void*>(&k_jacobi_rows), JMAX_COLS * ROWS_SLICE * sizeof(double));
        size = plan_clusters(cost, size, cluster_slots(reinterpret_cast<const void*>(&k_jacobi_svd<J_LOGGED>), JTHR, full, max_cluster));
    }
    // one launch per instance and cluster size, the largest clusters first, each on a stream of its own while they last
    constexpr int NCLS = 4 * N_CLUSTER_SIZES;
    auto cls_of = [](int log2nc, JacobiMode m) { return (N_CLUSTER_SIZES - 1 - log2nc) * 4 + (J_LOGGED_L2 - m); };
    std::vector<SvdJob> cls[NCLS];
    uint64_t log_len = 0;
    uint32_t log_cols = 0, n_logged = 0;
    uint32_t nid = 0;
    for (std::size_t b = 0; b < jobs.size(); ++b) {
        const SvdJob& j = jobs[b];
        nid = std::max(nid, j.id + 1);
        const uint64_t k = std::min(j.m, j.n);
        if (!j.m || !j.n) continue;
        if (j.a_off + uint64_t(j.m) * j.n > a_len || j.u_off + uint64_t(j.m) * k > u_len || j.s_off + k > s_len ||
            j.v_off + uint64_t(j.n) * k > v_len || j.w_off + jacobi_svd_scratch(j.m, j.n) > w_len)
            throw std::runtime_error("batched_jacobi_svd: block outside its buffers");
        if (j.w_off % 2) throw std::runtime_error("batched_jacobi_svd: scratch offset not 16-byte aligned");
        const JacobiMode m = jacobi_mode(std::max(j.m, j.n), uint32_t(k), 1u << size[b]);
        std::vector<SvdJob>& v = cls[cls_of(size[b], m)];
        v.push_back(j);
        if (m >= J_LOGGED) {
            v.back().l_off = log_len;
            log_len += log_entries(uint32_t(k));
            log_cols = std::max(log_cols, uint32_t(k));
            ++n_logged;
        }
    }
    DBuf<double2> log(log_len);
    DBuf<int> metas(2 * n_logged);
    if (metas.size()) QCM_CUDA(cudaMemsetAsync(metas.get(), 0, metas.size() * sizeof(int), s));
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
    if (used > 1 && !side) side = std::make_unique<SideStreams>();
    if (used > 1) side->fork(s);
    std::size_t first = 0, first_logged = 0;
    int lane = -1;  // the first launch stays on s
    cudaError_t err = cudaSuccess;
    for (int i = 0; i < NCLS && err == cudaSuccess; ++i) {
        if (cls[i].empty()) continue;
        const uint32_t nc = 1u << (N_CLUSTER_SIZES - 1 - i / 4);
        const JacobiMode mode = JacobiMode(J_LOGGED_L2 - i % 4);
        // shared memory of the launch's largest block (everything that fits), threads by its pairs per round
        uint64_t sm = 0;
        uint32_t lanes = 0;
        for (const SvdJob& j : cls[i]) {
            const uint32_t r = std::max(j.m, j.n), c = std::min(j.m, j.n);
            const JacobiLayout l = jacobi_layout(r, c, nc, JSMEM_DOUBLES);
            sm = std::max(sm, l.fixed + (mode != J_LOGGED_L2 ? uint64_t(l.ldg) * c : 0) + (mode < J_LOGGED ? uint64_t(l.ldq) * c : 0));
            lanes = std::max(lanes, (c + 1) / 2 * (nc == 1 ? 16 : 8));
        }
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(unsigned(cls[i].size()) * nc);
        cfg.blockDim = dim3(std::min<uint32_t>(JTHR, std::max<uint32_t>(128, (lanes + 127) / 128 * 128)));
        cfg.dynamicSmemBytes = std::size_t(sm) * sizeof(double);
        cfg.stream = lane < 0 ? s : side->s[lane % SideStreams::N];
        cudaLaunchAttribute at{};
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = nc;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        const SvdJob* dj = jobbuf.get() + first;
        if (mode < J_LOGGED) {
            err = cudaLaunchKernelEx(&cfg, mode == J_ONE ? k_jacobi_svd<J_ONE> : k_jacobi_svd<J_SMEM>, dj, A, U, S, V, W, zero_count,
                                     sweeps_used, JacobiLog{nullptr, nullptr, 0});
        } else {
            // LOG_SWEEPS sweeps, then their rotations applied to Q, up to the limit of sweeps (launches after the last
            // block is done return at once)
            const std::size_t qb = std::size_t(log_cols) * ROWS_SLICE * sizeof(double);
            const dim3 qg((log_cols + ROWS_SLICE - 1) / ROWS_SLICE, unsigned(cls[i].size()));
            auto* kernel = mode == J_LOGGED_L2 ? k_jacobi_svd<J_LOGGED_L2> : k_jacobi_svd<J_LOGGED>;
            int* meta = metas.get() + 2 * first_logged;
            first_logged += cls[i].size();
            for (int x = 0; x < JMAX_SWEEPS / LOG_SWEEPS && err == cudaSuccess; ++x) {
                const JacobiLog lg{log.get(), meta, x};
                err = cudaLaunchKernelEx(&cfg, kernel, dj, A, U, S, V, W, zero_count, sweeps_used, lg);
                if (err != cudaSuccess) break;
                k_jacobi_rows<<<qg, ROWS_THR, qb, cfg.stream>>>(dj, U, V, lg, x);
                k_jacobi_mark<<<unsigned((cls[i].size() + 127) / 128), 128, 0, cfg.stream>>>(meta, int(cls[i].size()));
                err = cudaGetLastError();
            }
        }
        first += cls[i].size();
        ++lane;
    }
    if (used > 1) side->join(s);  // after a failed launch too: the others still use the buffers
    QCM_CUDA(err);
}

}  // namespace qcm
