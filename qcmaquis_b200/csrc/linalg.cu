// Dense per-block factorizations on the device (see linalg.hpp).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <functional>
#include <queue>
#include <stdexcept>
#include <string>

#include "linalg.hpp"

#define QCM_SOLVER(call)                                                                                   \
    do {                                                                                                   \
        cusolverStatus_t st_ = (call);                                                                     \
        if (st_ != CUSOLVER_STATUS_SUCCESS)                                                                \
            throw qcm::cuda_error(std::string(#call) + ": cuSOLVER status " + std::to_string(int(st_)));   \
    } while (0)

namespace qcm {
namespace {

constexpr uint32_t INFO_CAP = 4096;

}  // namespace

Solver::Solver() {
    QCM_SOLVER(cusolverDnCreate(&h));
    QCM_SOLVER(cusolverDnCreateGesvdjInfo(&svdp));
    QCM_SOLVER(cusolverDnXgesvdjSetMaxSweeps(svdp, 100));
    QCM_SOLVER(cusolverDnXgesvdjSetSortEig(svdp, 1));
    info.alloc(INFO_CAP);
    QCM_CUDA(cudaEventCreateWithFlags(&fork_ev, cudaEventDisableTiming));
    for (Lane& L : lane) {
        QCM_CUDA(cudaStreamCreateWithFlags(&L.s, cudaStreamNonBlocking));
        register_stream(L.s);
        QCM_CUDA(cudaEventCreateWithFlags(&L.done, cudaEventDisableTiming));
        QCM_SOLVER(cusolverDnCreate(&L.h));
        QCM_SOLVER(cusolverDnSetStream(L.h, L.s));
        QCM_SOLVER(cusolverDnCreateGesvdjInfo(&L.svdp));
        QCM_SOLVER(cusolverDnXgesvdjSetMaxSweeps(L.svdp, 100));
        QCM_SOLVER(cusolverDnXgesvdjSetSortEig(L.svdp, 1));
    }
}

Solver::~Solver() {
    for (Lane& L : lane) {
        if (L.s) cudaStreamSynchronize(L.s);
        L.a.reset();
        L.work.reset();
        if (L.s) {
            cudaStreamSynchronize(L.s);
            retire_stream(L.s);
        }
        if (L.svdp) cusolverDnDestroyGesvdjInfo(L.svdp);
        if (L.h) cusolverDnDestroy(L.h);
        if (L.done) cudaEventDestroy(L.done);
        if (L.s) cudaStreamDestroy(L.s);
    }
    if (fork_ev) cudaEventDestroy(fork_ev);
    if (svdp) cusolverDnDestroyGesvdjInfo(svdp);
    if (h) cusolverDnDestroy(h);
}

void Solver::fork(cudaStream_t s) {
    QCM_CUDA(cudaEventRecord(fork_ev, s));
    for (Lane& L : lane) QCM_CUDA(cudaStreamWaitEvent(L.s, fork_ev, 0));
}

int* Solver::reserve_info(uint32_t n, cudaStream_t s) {
    if (n > INFO_CAP) throw std::runtime_error("too many factorizations in one batch");
    if (n_info + n > INFO_CAP) check(s);
    int* p = info.get() + n_info;
    n_info += n;
    return p;
}

void Solver::join(cudaStream_t s) {
    for (Lane& L : lane) {
        QCM_CUDA(cudaEventRecord(L.done, L.s));
        QCM_CUDA(cudaStreamWaitEvent(s, L.done, 0));
    }
}

void Solver::bind(cudaStream_t s) { QCM_SOLVER(cusolverDnSetStream(h, s)); }

void Solver::check(cudaStream_t s) {
    if (!n_info) return;
    std::vector<int> hi(n_info);
    QCM_CUDA(cudaMemcpyAsync(hi.data(), info.get(), n_info * sizeof(int), cudaMemcpyDeviceToHost, s));
    QCM_CUDA(cudaStreamSynchronize(s));
    n_info = 0;
    for (int v : hi)
        if (v != 0) throw std::runtime_error("device factorization failed (info " + std::to_string(v) + ")");
}

void svd_thin_lane(Solver& sv, int l, const double* A, int m, int n, double* U, double* S, double* V, int* info) {
    if (m == 0 || n == 0) return;
    Solver::Lane& L = sv.lane[l];
    AllocStream scope(L.s);  // a lane's buffers are ordered on the lane's stream
    if (L.a.size() < std::size_t(m) * n) L.a.alloc(std::size_t(m) * n);
    QCM_CUDA(cudaMemcpyAsync(L.a.get(), A, std::size_t(m) * n * sizeof(double), cudaMemcpyDeviceToDevice, L.s));
    int lwork = 0;
    QCM_SOLVER(cusolverDnDgesvdj_bufferSize(L.h, CUSOLVER_EIG_MODE_VECTOR, 1, m, n, L.a.get(), m, S, U, m, V, n, &lwork,
                                            L.svdp));
    if (L.work.size() < std::size_t(lwork)) L.work.alloc(std::size_t(lwork));
    QCM_SOLVER(cusolverDnDgesvdj(L.h, CUSOLVER_EIG_MODE_VECTOR, 1, m, n, L.a.get(), m, S, U, m, V, n, L.work.get(), lwork,
                                 info, L.svdp));
}

ClusterSlots cluster_slots(const void* kernel, uint32_t threads, std::size_t bytes, uint32_t max_cluster) {
    ClusterSlots r{};
    for (int i = 0; i < N_CLUSTER_SIZES && (1u << i) <= max_cluster; ++i) {
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(1u << i);
        cfg.blockDim = dim3(threads);
        cfg.dynamicSmemBytes = bytes;
        cudaLaunchAttribute at{};
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = 1u << i;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) == cudaSuccess) r[i] = uint32_t(std::max(n, 0));
        else cudaGetLastError();  // a size that the device does not know is an error
    }
    r[0] = std::max(r[0], 1u);
    return r;
}

std::vector<uint8_t> plan_clusters(const std::vector<std::array<double, N_CLUSTER_SIZES>>& cost, const std::vector<uint8_t>& want,
                                   const ClusterSlots& slots) {
    const std::size_t n = want.size();
    std::vector<uint8_t> most(want), best;
    double full = 0.0, t0 = 0.0;
    for (std::size_t i = 0; i < n; ++i) {
        while (!slots[most[i]]) --most[i];
        full += 1.0 / slots[most[i]];
        t0 = std::max(t0, *std::min_element(cost[i].begin(), cost[i].begin() + most[i] + 1));
    }
    if (full <= 1.0) return most;
    std::vector<uint8_t> size(n), before;
    std::vector<std::size_t> order(n);
    double end = 0.0, limit = t0;
    for (int step = 0; step < 24; ++step, limit *= 1.25) {
        bool least = true;  // every block at its size of least area
        for (std::size_t i = 0; i < n; ++i) {
            int within = -1, area = 0, fast = 0;
            for (int k = 0; k <= most[i]; ++k) {
                if (!slots[k]) continue;
                const double a = cost[i][k] / slots[k];
                if (a < cost[i][area] / slots[area]) area = k;
                if (cost[i][k] < cost[i][fast]) fast = k;
                if (cost[i][k] <= limit && (within < 0 || a < cost[i][within] / slots[within])) within = k;
            }
            size[i] = uint8_t(within < 0 ? fast : within);
            least = least && size[i] == area;
        }
        if (size != before) {
            before = size;
            for (std::size_t i = 0; i < n; ++i) order[i] = i;
            std::sort(order.begin(), order.end(), [&](std::size_t a, std::size_t b) {
                if (size[a] != size[b]) return size[a] > size[b];
                return cost[a][size[a]] != cost[b][size[b]] ? cost[a][size[a]] > cost[b][size[b]] : a < b;
            });
            // blocks start in this order, each as soon as its share of the device is free
            std::priority_queue<std::pair<double, double>, std::vector<std::pair<double, double>>, std::greater<>> running;
            double now = 0.0, free = 1.0, last = 0.0;
            for (std::size_t i : order) {
                const double share = 1.0 / slots[size[i]];
                while (free < share - 1e-9) {
                    now = running.top().first;
                    free += running.top().second;
                    running.pop();
                }
                free -= share;
                running.push({now + cost[i][size[i]], share});
                last = std::max(last, now + cost[i][size[i]]);
            }
            if (best.empty() || last < end) {
                best = size;
                end = last;
            }
        }
        if (least) break;
    }
    return best;
}

void syevd_lane(Solver& sv, int l, double* A, int n, double* W, int* info) {
    if (n == 0) return;
    Solver::Lane& L = sv.lane[l];
    AllocStream scope(L.s);
    int lwork = 0;
    QCM_SOLVER(cusolverDnDsyevd_bufferSize(L.h, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_LOWER, n, A, n, W, &lwork));
    if (L.work.size() < std::size_t(lwork)) L.work.alloc(std::size_t(lwork));
    QCM_SOLVER(cusolverDnDsyevd(L.h, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_LOWER, n, A, n, W, L.work.get(), lwork, info));
}

void sym_lowest_eigenpair(const double* M, int ldm, int n, double& w, std::vector<double>& z) {
    std::vector<double> A(std::size_t(n) * n), V(std::size_t(n) * n, 0.0);
    for (int j = 0; j < n; ++j)
        for (int i = 0; i <= j; ++i) A[i + std::size_t(j) * n] = A[j + std::size_t(i) * n] = M[i + std::size_t(j) * ldm];
    for (int i = 0; i < n; ++i) V[i + std::size_t(i) * n] = 1.0;
    auto a = [&](int i, int j) -> double& { return A[i + std::size_t(j) * n]; };
    // cyclic Jacobi (Golub & Van Loan, Algorithm 8.5.3) until the off-diagonal part is negligible
    double last = 0.0;  // off-diagonal part of the sweep before
    for (int sweep = 0; sweep < 100; ++sweep) {
        double off = 0.0, tot = 0.0;
        for (int j = 0; j < n; ++j)
            for (int i = 0; i < n; ++i) { tot += a(i, j) * a(i, j); if (i != j) off += a(i, j) * a(i, j); }
        if (jacobi_done(off, tot, last, sweep)) break;
        last = off;
        for (int p = 0; p < n - 1; ++p)
            for (int q = p + 1; q < n; ++q) {
                double apq = a(p, q);
                if (apq == 0.0) continue;
                double tau = (a(q, q) - a(p, p)) / (2.0 * apq);
                double t = (tau >= 0 ? 1.0 : -1.0) / (std::fabs(tau) + std::sqrt(1.0 + tau * tau));
                double c = 1.0 / std::sqrt(1.0 + t * t), s = t * c;
                for (int k = 0; k < n; ++k) {  // A <- A J
                    double akp = a(k, p), akq = a(k, q);
                    a(k, p) = c * akp - s * akq;
                    a(k, q) = s * akp + c * akq;
                }
                for (int k = 0; k < n; ++k) {  // A <- J^T A
                    double apk = a(p, k), aqk = a(q, k);
                    a(p, k) = c * apk - s * aqk;
                    a(q, k) = s * apk + c * aqk;
                }
                for (int k = 0; k < n; ++k) {  // V <- V J
                    double vkp = V[k + std::size_t(p) * n], vkq = V[k + std::size_t(q) * n];
                    V[k + std::size_t(p) * n] = c * vkp - s * vkq;
                    V[k + std::size_t(q) * n] = s * vkp + c * vkq;
                }
            }
    }
    int best = 0;
    for (int i = 1; i < n; ++i) if (a(i, i) < a(best, best)) best = i;
    w = a(best, best);
    z.assign(V.begin() + std::size_t(best) * n, V.begin() + std::size_t(best + 1) * n);
}

}  // namespace qcm
