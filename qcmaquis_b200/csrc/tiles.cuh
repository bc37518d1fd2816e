// The work list of a launch that covers tiles of several shapes.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "device.hpp"
#include "heff.hpp"

namespace qcm {

// The tiles of a phase in all its shapes, one launch: the CTA's tile is looked up by running ends in the order
// 128-, 64-, 32-, 16-row tiles.  A launch per shape left the chip idle at the end of each one: a few long 128-row
// tiles alone took as long as a tenth of the phase (S-GEMM at L=16, M=256 425 -> 333 us, at L=24, M=512 2.72 ->
// 2.50 ms).  Shared memory is the largest shape's; registers are set by the launch bounds in any case.
template <class D>
struct TileSet {
    const D* t[N_SHAPES];
    uint32_t end[N_SHAPES];  // running ends, shapes from 128 rows down
    // shape and tile of CTA b (constant indices: the arrays stay in parameter space)
    __device__ __forceinline__ int find(uint32_t b, D& d) const {
        if (b < end[SHAPE_128]) { d = t[SHAPE_128][b]; return SHAPE_128; }
        if (b < end[SHAPE_64]) { d = t[SHAPE_64][b - end[SHAPE_128]]; return SHAPE_64; }
        if (b < end[SHAPE_32]) { d = t[SHAPE_32][b - end[SHAPE_64]]; return SHAPE_32; }
        d = t[SHAPE_16][b - end[SHAPE_32]];
        return SHAPE_16;
    }
};
// the tiles [a[sh], b[sh]) of every shape (only one shape if `only` >= 0); n: how many in all
template <class D>
inline TileSet<D> tile_set(const DBuf<D>* t, const uint32_t* a, const uint32_t* b, uint32_t& n, int only = -1) {
    TileSet<D> r;
    n = 0;
    for (int sh = N_SHAPES - 1; sh >= 0; --sh) {
        r.t[sh] = t[sh].get() + a[sh];
        if (only < 0 || sh == only) n += b[sh] - a[sh];
        r.end[sh] = n;
    }
    return r;
}
template <class D>
inline TileSet<D> tile_set(const DBuf<D>* t, const std::vector<D>* h, uint32_t& n, int only = -1) {
    uint32_t a[N_SHAPES] = {}, b[N_SHAPES];
    for (int sh = 0; sh < N_SHAPES; ++sh) b[sh] = uint32_t(h[sh].size());
    return tile_set(t, a, b, n, only);
}

}  // namespace qcm
