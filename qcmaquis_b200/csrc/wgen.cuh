// Traversal of the coefficient terms of an S-build unit, shared by the generation of its coefficient block
// (k_wgen) and the adjoint's sums over it (k_wadj): one thread per (line, MPO entry) pair.
// Rows of the MPO differ in length by two orders of magnitude, units by three, and a term is a chain of dependent
// table reads: latency binds, so what counts is how many pairs are in flight.  The pairs of a unit are numbered
// through (a scan of the row lengths), cut into tasks of WGEN_PAIRS pairs, a CTA each, and dealt out to its threads
// one by one: neither the longest row nor the largest unit decides, and neighbouring threads read neighbouring
// entries.  An apply that generates its coefficients in 15 chunks (L=20, M=384): 20.9 ms with a thread per line, 10.7 ms
// with a thread per pair and a CTA per unit, 4.2 ms so (46 % of the issue slots, half the stalls on table reads; 3.6 ms
// with the other kernels of the apply as they are now).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "heff.hpp"

namespace qcm {
namespace wg {

constexpr int THR = 256;
constexpr uint32_t SMAP = 2048;   // (slice id, slot) pairs staged in shared memory
constexpr uint32_t NST = 64;      // physical states of the basis (CoefGen::validate bounds nst)
constexpr uint32_t LINES = 1024;  // lines numbered at a time

struct Shared {
    uint32_t sid[SMAP], sslot[SMAP];
    WGenInD sin[NST];
    uint32_t row0[LINES], pre[LINES + 1];  // per line: its row's first entry; entries of the lines before it
};

// Stages the unit's slice map and input states; returns its map (shared or global memory).
struct Map {
    const uint32_t* ids;
    const uint32_t* slots;
    uint32_t n;
    // slot of slice id, or WGEN_NONE
    __device__ __forceinline__ uint32_t slot(uint32_t id) const {
        uint32_t lo = 0, hi = n;
        while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            if (ids[mid] < id) lo = mid + 1;
            else hi = mid;
        }
        return lo < n && ids[lo] == id ? slots[lo] : WGEN_NONE;
    }
};
static __device__ __forceinline__ Map stage(const WGenTab& t, const WGenUnitD& U, uint32_t unit, Shared& sh) {
    const bool staged = U.nk <= SMAP;
    if (staged)
        for (uint32_t i = threadIdx.x; i < U.nk; i += blockDim.x) {
            sh.sid[i] = t.smap_id[U.map0 + i];
            sh.sslot[i] = t.smap_slot[U.map0 + i];
        }
    for (uint32_t i = threadIdx.x; i < t.nst; i += blockDim.x) sh.sin[i] = t.gin[std::size_t(unit) * t.nst + i];
    __syncthreads();
    return Map{staged ? sh.sid : t.smap_id + U.map0, staged ? sh.sslot : t.smap_slot + U.map0, U.nk};
}

// body(line, entry, first entry of the line's row, one past its last) for the pairs [i0, i0 + WGEN_PAIRS) of the unit
template <class Body>
static __device__ __forceinline__ void for_entries(const WGenTab& t, const WGenUnitD& U, uint32_t i0, Shared& sh, Body body) {
    uint32_t base = 0;  // pairs of the lines before l0
    for (uint32_t l0 = 0; l0 < U.nl && base < i0 + WGEN_PAIRS; l0 += LINES) {
        const uint32_t n = min(LINES, U.nl - l0);
        for (uint32_t l = threadIdx.x; l < n; l += blockDim.x) {
            const uint32_t m = t.line_major[U.line0 + l0 + l];
            const uint32_t a = t.m_ptr[m];
            sh.row0[l] = a;
            sh.pre[l + 1] = t.m_ptr[m + 1] - a;
        }
        if (threadIdx.x == 0) sh.pre[0] = 0;
        __syncthreads();
        if (threadIdx.x < 32) {
            uint32_t carry = 0;
            for (uint32_t l = threadIdx.x; l < (n + 31) / 32 * 32; l += 32) {
                uint32_t v = l < n ? sh.pre[l + 1] : 0;
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t w = __shfl_up_sync(0xffffffffu, v, o);
                    if (int(threadIdx.x) >= o) v += w;
                }
                v += carry;
                if (l < n) sh.pre[l + 1] = v;
                carry = __shfl_sync(0xffffffffu, v, 31);
            }
        }
        __syncthreads();
        const uint32_t total = sh.pre[n];
        const uint32_t a0 = i0 > base ? i0 - base : 0, a1 = min(total, i0 + WGEN_PAIRS - base);
        for (uint32_t i = a0 + threadIdx.x; i < a1; i += blockDim.x) {
            uint32_t lo = 0, hi = n;  // the last line with pre[line] <= i (an empty row's successor wins)
            while (hi - lo > 1) {
                const uint32_t mid = (lo + hi) >> 1;
                if (sh.pre[mid] <= i) lo = mid;
                else hi = mid;
            }
            const uint32_t a = sh.row0[lo];
            body(l0 + lo, a + (i - sh.pre[lo]), a, a + (sh.pre[lo + 1] - sh.pre[lo]));
        }
        base += total;
        __syncthreads();
    }
}

}  // namespace wg
}  // namespace qcm
