// Adjoint of the H_eff apply (the differentiation form of the path).  For f = ybar . H_eff(W) x:
//   psi_bar   = H_eff^T ybar = H_eff ybar: the two-site H_eff of a Hermitian MPO is symmetric;
//   coeff_bar = df / d scale_e for every entry e of the plan's two-site MPO tensor.
// f is linear in every scale.  Each coefficient term that k_wgen sums into the dense block W_u
// (lines x slots) of an S-build unit is alpha = o_val * b_cs * (scale_e * line_scale), and the unit's
// S rows are S_u = W_u T_u (create_s_r, tasks.cpp:466-494, as a dense GEMM).  So
//   Sbar      = L_eff^T ybar per L.S segment       (transpose of contract, tasks.cpp:286-313),
//   Wbar_u    = Sbar_u T_u^T per unit              (k_wbar, DMMA, in the coefficient-block layout),
//   coeff_bar = sum over the terms of entry e of Wbar_u(line, slot) * o_val * b_cs * line_scale.
// The last runs k_wgen's traversal backwards.  One thread per (line, entry of its MPO row) writes the
// line's partial sum for the entry (k_wadj).  Then the partials of the lines of the entry's row are added in a
// fixed order (k_entry_sum).  There are no atomics, so the result does not vary from run to run.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <stdexcept>
#include <vector>

#include "dev_ops.hpp"
#include "dmma.cuh"
#include "heff.hpp"
#include "tiles.cuh"
#include "wgen.cuh"

namespace qcm {

struct HeffAdjointWork {
    std::vector<TileD> tiles[N_SHAPES];  // k_wbar: (unit, first line, first slot) per tile of Wbar
    DBuf<TileD> d_tiles[N_SHAPES];
    DBuf<double> d_Wb;          // Wbar, the coefficient-block layout (w_len doubles)
    DBuf<double> d_P;           // per line, one partial per entry of its MPO row
    DBuf<uint64_t> d_pofs;      // per line: offset of its partials in P
    DBuf<uint32_t> d_rl_ptr, d_rl_line, d_e_row;  // lines grouped by MPO row (CSR); MPO row per entry
    DBuf<uint32_t> d_err;
    std::vector<GemmJob> sjobs;  // Sbar = L^T ybar per segment
    DBuf<GemmJob> d_jobs;
    DBuf<uint32_t> d_jtiles;
    uint64_t p_len = 0, n_terms = 0;
};

namespace {

using namespace dm;

// Wbar_u(line, slot) = sum_e Sbar(S row block line_b1[line], element e) * T(slice of slot, e); one CTA per tile (shapes as
// the T-GEMM's, by the unit's lines), K = the unit's elements.  Elements are contiguous in both operands: both are staged
// with k fastest, 16 bytes at a time where the strides are even.  A thread copies the same k of every row, so an
// element's place in its S row (a division) is found once per step.  0.64 ms with 64 x 64 tiles throughout, 8-byte
// copies and a division per element; 0.52 ms so (L=16, M=256: 14 TFLOP/s, K of 91 elements a tile on average).
template <class S>
__device__ __forceinline__ void wbar_tile(Stage<S>* st, uint64_t* soff, uint64_t* lrow, const TileD& tile, const UnitD& U,
                                          const uint32_t* __restrict__ line_b1, const uint64_t* __restrict__ slice_off,
                                          const double* __restrict__ Sb, const double* __restrict__ T, double* __restrict__ Wb) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t nm = min(uint32_t(S::BM), U.nl - tile.m0), nn = min(uint32_t(S::BN), U.nk - tile.n0);
    for (uint32_t c = tid; c < nn; c += NTHR) soff[c] = slice_off[U.slice0 + tile.n0 + c];
    // S row block of each line of the tile (the rows k_sgemm writes for it)
    for (uint32_t c = tid; c < nm; c += NTHR) lrow[c] = U.s_off + uint64_t(line_b1[U.line0 + tile.m0 + c]) * U.line_stride;
    __syncthreads();
    // slices start on 16 bytes; pairs of elements of an S row do if all its strides are even
    const bool a16 = !((U.ne | U.erows | U.col_stride | U.line_stride | U.s_off) & 1u) && !(reinterpret_cast<uintptr_t>(Sb) & 15u);
    const bool b16 = !(U.ne & 1u);
    const uint32_t ka = a16 ? 2 * (tid % (BK / 2)) : tid % BK;  // this thread's k in stage_kfast
    static_assert(NTHR % BK == 0, "the same k in every round");
    const int nfm = int(nm + 7) / 8;
    Acc<S> acc;
    acc.zero();
    const uint32_t nk = (U.ne + BK - 1) / BK;
#pragma unroll 1
    for (int kc = -1; kc < int(nk); ++kc) {
        if (kc >= 0) {
            cp_wait_all();
            __syncthreads();
        }
        if (kc + 1 < int(nk)) {
            Stage<S>& s = st[(kc + 1) & 1];
            const uint32_t k0 = uint32_t(kc + 1) * BK, col = (k0 + ka) / U.erows;
            const uint64_t at = (k0 + ka - col * U.erows) + uint64_t(col) * U.col_stride;
            stage_kfast<S::BM, 4>(&s.A[0][0], Sb, nm, U.ne - k0, a16, [&](int m, int) { return Sb + lrow[m] + at; });
            stage_kfast<S::BN, 4>(&s.B[0][0], T, nn, U.ne - k0, b16, [&](int n, int k) { return T + soff[n] + k0 + k; });
            cp_commit();
        }
        if (kc >= 0) {
            const Stage<S>& s = st[kc & 1];
            mma_stage_part<S, true, true>(&s.A[0][0], &s.B[0][0], acc, warp, lane, nfm,
                                          int(min(uint32_t(BK), U.ne - kc * BK) + 3) / 4);
        }
    }
    for_acc<S>(acc, warp, lane, [&](int m, int n, double v) {
        if (uint32_t(m) < nm && uint32_t(n) < nn) Wb[U.w_off + tile.m0 + m + uint64_t(tile.n0 + n) * U.wld] = v;
    });
}

__global__ void __launch_bounds__(NTHR, 4) k_wbar(TileSet<TileD> set, const UnitD* __restrict__ units,
                                                  const uint32_t* __restrict__ line_b1, const uint64_t* __restrict__ slice_off,
                                                  const double* __restrict__ Sb, const double* __restrict__ T,
                                                  double* __restrict__ Wb) {
    __shared__ __align__(16) unsigned char raw[2 * std::max({sizeof(Stage<Sh16>), sizeof(Stage<Sh32>), sizeof(Stage<Sh64>)})];
    __shared__ uint64_t soff[Sh16::BN], lrow[Sh64::BM];
    static_assert(Sh32::BN <= Sh16::BN && Sh64::BN <= Sh16::BN);
    TileD tile;
    const int sh = set.find(blockIdx.x, tile);
    const UnitD U = units[tile.item];
    if (sh == SHAPE_64) wbar_tile<Sh64>(reinterpret_cast<Stage<Sh64>*>(raw), soff, lrow, tile, U, line_b1, slice_off, Sb, T, Wb);
    else if (sh == SHAPE_32) wbar_tile<Sh32>(reinterpret_cast<Stage<Sh32>*>(raw), soff, lrow, tile, U, line_b1, slice_off, Sb, T, Wb);
    else wbar_tile<Sh16>(reinterpret_cast<Stage<Sh16>*>(raw), soff, lrow, tile, U, line_b1, slice_off, Sb, T, Wb);
}

// Per line: P[pofs[line] + (e - m_ptr[m])] = sum over the terms of entry e (row m of the line) of
// Wbar(line, slot) * o_val * b_cs * line_scale; the traversal and slot lookup of k_wgen, one thread per entry.
__global__ void __launch_bounds__(wg::THR) k_wadj(WGenTab t, const double* __restrict__ Wb, const uint64_t* __restrict__ pofs,
                                                  double* __restrict__ P, uint32_t* __restrict__ err) {
    __shared__ wg::Shared sh;
    const WGenTaskD task = t.tasks[blockIdx.x];
    const WGenUnitD U = t.units[task.unit];
    const wg::Map map = wg::stage(t, U, task.unit, sh);
    const double* Wu = Wb + U.w_off;
    wg::for_entries(t, U, task.i0, sh, [&](uint32_t line, uint32_t e, uint32_t e0, uint32_t) {
        const uint32_t gl = U.line0 + line, x = t.m_other[e];
        const double lsc = t.line_scale[gl];
        const std::size_t q = std::size_t(t.m_op[e]) * t.nst + U.st_out;
        const uint32_t k1 = t.o_ptr[q + 1];
        double acc = 0.0;
        for (uint32_t k = t.o_ptr[q]; k < k1; ++k) {
            const WGenInD g = sh.sin[t.o_in[k]];
            if (g.c == WGEN_NONE) continue;
            const std::size_t bq = std::size_t(g.c) * t.b_aux + x;
            const int32_t pos = t.b_pos[bq];
            if (pos < 0) continue;
            const uint32_t slot = map.slot(g.jbase + uint32_t(pos));
            if (slot == WGEN_NONE) { atomicOr(err, 1u); continue; }
            const double d = __dmul_rn(__dmul_rn(t.o_val[k], t.b_cs[bq]), lsc);  // d alpha / d scale_e
            acc = fma(Wu[line + uint64_t(slot) * U.wld], d, acc);
        }
        P[pofs[gl] + (e - e0)] = acc;
    });
}

// out[e] = sum over the lines of e's MPO row of their partial for e.  A CTA takes 32 entries (a lane each: neighbouring
// entries of a row have neighbouring partials) and its 8 warps an eighth of the lines each, whose sums are added in
// warp order: the order does not vary from run to run.  A row's lines are a chain of dependent reads, thousands for
// some rows: with one thread per entry the longest took 127 us of the 1.9 ms at L=16, M=256.
constexpr int ES_WARPS = 8;
__global__ void __launch_bounds__(32 * ES_WARPS) k_entry_sum(uint64_t n_terms, const uint32_t* __restrict__ e_row,
                                                             const uint32_t* __restrict__ m_ptr, const uint32_t* __restrict__ rl_ptr,
                                                             const uint32_t* __restrict__ rl_line, const uint64_t* __restrict__ pofs,
                                                             const double* __restrict__ P, double* __restrict__ out) {
    __shared__ double part[ES_WARPS][32];
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (uint64_t e0 = uint64_t(blockIdx.x) * 32; e0 < n_terms; e0 += uint64_t(gridDim.x) * 32) {
        const uint64_t e = e0 + lane;
        double s = 0.0;
        if (e < n_terms) {
            const uint32_t m = e_row[e], r0 = rl_ptr[m], nl = rl_ptr[m + 1] - r0, share = (nl + ES_WARPS - 1) / ES_WARPS;
            const uint64_t j = e - m_ptr[m];
            uint32_t t = r0 + min(nl, w * share);
            const uint32_t t1 = r0 + min(nl, (w + 1) * share);
            // eight partials in flight (each is two dependent reads), added in line order
            for (; t + 8 <= t1; t += 8) {
                double v[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) v[i] = P[pofs[rl_line[t + i]] + j];
#pragma unroll
                for (int i = 0; i < 8; ++i) s += v[i];
            }
            for (; t < t1; ++t) s += P[pofs[rl_line[t]] + j];
        }
        part[w][lane] = s;
        __syncthreads();
        if (w == 0 && e < n_terms) {
            for (int i = 1; i < ES_WARPS; ++i) s += part[i][lane];
            out[e] = s;
        }
        __syncthreads();
    }
}

HeffAdjointWork& adjoint_work(HeffPlan& p) {
    if (p.adj) return *p.adj;
    const CoefGen& cg = p.cg;
    if (!cg.by_row || !cg.mt) throw std::runtime_error("heff adjoint: plan without row-major coefficient tables");
    if (!p.L || !p.R) throw std::runtime_error("heff adjoint: plan without boundaries");
    const MPOTables& mt = *cg.mt;
    auto w = std::make_shared<HeffAdjointWork>();
    w->n_terms = mt.row_other.size();
    for (uint32_t i = 0; i < uint32_t(p.units.size()); ++i) {
        const UnitD& u = p.units[i];
        // every Sbar element and T slice element k_wbar reads lies in its buffer
        if (u.nl && u.ne) {
            if (!u.erows) throw std::runtime_error("heff adjoint: unit without element rows");
            auto at = [&](uint32_t e) { return uint64_t(e % u.erows) + uint64_t(e / u.erows) * u.col_stride; };
            uint64_t emax = at(u.ne - 1);
            if (u.ne > u.erows) emax = std::max(emax, at((u.ne - 1) / u.erows * u.erows - 1));
            uint32_t bmax = 0;
            for (uint32_t l = 0; l < u.nl; ++l) bmax = std::max(bmax, p.line_b1.at(std::size_t(u.line0) + l));
            if (u.s_off + uint64_t(bmax) * u.line_stride + emax >= p.s_len)
                throw std::runtime_error("heff adjoint: unit rows outside the S buffer");
            for (uint32_t k = 0; k < u.nk; ++k)
                if (p.slice_off[u.slice0 + k] + u.ne > p.t_len) throw std::runtime_error("heff adjoint: slice outside T");
        }
        const int sh = shape_for_rows(u.nl);
        for (uint32_t m0 = 0; m0 < u.nl; m0 += shape_bm(sh))
            for (uint32_t n0 = 0; n0 < u.nk; n0 += shape_bn(sh)) w->tiles[sh].push_back(TileD{i, m0, n0, 0});
    }
    // partials: per line (global line order), one per entry of its MPO row
    const std::size_t nlines = cg.line_major.size();
    const uint32_t rows = uint32_t(mt.row_ptr.size() - 1);
    std::vector<uint64_t> pofs(nlines);
    std::vector<uint32_t> rl_ptr(std::size_t(rows) + 1, 0), rl_line(nlines), e_row(w->n_terms);
    uint64_t acc = 0;
    for (std::size_t gl = 0; gl < nlines; ++gl) {
        const uint32_t m = cg.line_major[gl];
        if (m >= rows) throw std::runtime_error("heff adjoint: line outside the MPO rows");
        pofs[gl] = acc;
        acc += mt.row_ptr[m + 1] - mt.row_ptr[m];
        rl_ptr[m + 1]++;
    }
    w->p_len = acc;
    for (uint32_t m = 0; m < rows; ++m) rl_ptr[m + 1] += rl_ptr[m];
    {
        std::vector<uint32_t> fill(rl_ptr.begin(), rl_ptr.end() - 1);
        for (std::size_t gl = 0; gl < nlines; ++gl) rl_line[fill[cg.line_major[gl]]++] = uint32_t(gl);
    }
    for (uint32_t m = 0; m < rows; ++m)
        for (uint32_t e = mt.row_ptr[m]; e < mt.row_ptr[m + 1]; ++e) e_row[e] = m;
    // Sbar = L^T ybar per segment (the L.S GEMM's operands, transposed)
    for (const OutD& o : p.outs)
        for (uint32_t k = 0; k < o.seg_count; ++k) {
            const SegD& sg = p.segs[o.seg_start + k];
            GemmJob j{};
            j.a_off = sg.l_off; j.b_off = o.y_off; j.c_off = sg.s_off;
            j.M = sg.nS * sg.ls_in; j.N = o.N; j.K = o.M;
            j.ldb = o.M; j.ldc = sg.nS * sg.ls_in;
            j.tb = 0; j.alpha = 1.0; j.beta = 0.0;
            if (!sg.tr) {
                // L_eff = the cohort's nS blocks (M x ls_in each) side by side: Sbar = L_eff^T ybar
                j.lda = o.M; j.ta = 1;
            } else {
                // a transposed cohort reads its Hermitian partner's blocks (ls_in x M each), so block b of
                // L_eff^T is the stored block itself: row blocks of ls_in rows, block b at b * M * ls_in
                j.lda = sg.ls_in; j.ta = 0;
                j.arb = sg.ls_in; j.a_bs = uint64_t(o.M) * sg.ls_in;
            }
            w->sjobs.push_back(j);
        }
    cudaStream_t s = p.stream;
    for (int sh = 0; sh < N_SHAPES; ++sh) w->d_tiles[sh].upload(w->tiles[sh], s);
    w->d_Wb.alloc(p.w_len ? p.w_len : 1);
    w->d_P.alloc(w->p_len ? w->p_len : 1);
    w->d_pofs.upload(pofs, s);
    w->d_rl_ptr.upload(rl_ptr, s);
    w->d_rl_line.upload(rl_line, s);
    w->d_e_row.upload(e_row, s);
    w->d_err.alloc(1);
    p.adj = w;
    return *w;
}

}  // namespace

uint64_t heff_adjoint_terms(const HeffPlan& p) { return p.cg.mt ? p.cg.mt->row_other.size() : 0; }

void heff_adjoint_device(HeffPlan& p, const double* x, const double* ybar, double* psi_bar, double* coeff_bar) {
    cudaStream_t s = p.stream;
    if (p.sector_chunked()) throw std::runtime_error("heff adjoint: the plan's apply is chunked by ket sector");
    if (psi_bar) heff_apply_device(p, ybar, psi_bar);
    if (!coeff_bar) return;
    HeffAdjointWork& w = adjoint_work(p);
    if (!w.n_terms) return;
    double* T = p.d_T.get();
    double* Sb = p.d_S.get();
    heff_tgemm_device(p, x, T);
    if (!w.sjobs.empty())
        batched_gemm(w.sjobs, p.L->data.get(), p.L->data.size(), ybar, p.x_len, Sb, p.s_len, w.d_jobs, w.d_jtiles, s);
    uint32_t n_tiles;
    const TileSet<TileD> tiles = tile_set(w.d_tiles, w.tiles, n_tiles);
    if (n_tiles)
        k_wbar<<<n_tiles, NTHR, 0, s>>>(tiles, p.d_units.get(), p.d_line_b1.get(), p.d_slice_off.get(), Sb, T, w.d_Wb.get());
    QCM_CUDA(cudaGetLastError());
    const CoefGen& cg = p.cg;
    QCM_CUDA(cudaMemsetAsync(w.d_err.get(), 0, sizeof(uint32_t), s));
    if (!cg.task_ptr.empty() && cg.task_ptr.back())
        k_wadj<<<cg.task_ptr.back(), wg::THR, 0, s>>>(cg.tables(), w.d_Wb.get(), w.d_pofs.get(), w.d_P.get(),
                                                             w.d_err.get());
    QCM_CUDA(cudaGetLastError());
    const unsigned grid = unsigned(std::min<uint64_t>((w.n_terms + 31) / 32, N_SM * 16));
    k_entry_sum<<<grid, 32 * ES_WARPS, 0, s>>>(w.n_terms, w.d_e_row.get(), cg.d_m_ptr.get(), w.d_rl_ptr.get(), w.d_rl_line.get(),
                                     w.d_pofs.get(), w.d_P.get(), coeff_bar);
    QCM_CUDA(cudaGetLastError());
    uint32_t h = 0;
    QCM_CUDA(cudaMemcpyAsync(&h, w.d_err.get(), sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
    QCM_CUDA(cudaStreamSynchronize(s));
    if (h) throw std::runtime_error("heff adjoint: a coefficient term has no slice slot");
}

}  // namespace qcm
