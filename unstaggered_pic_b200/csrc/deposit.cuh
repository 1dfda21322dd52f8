// Warp-private deposit windows (sm_100a): each warp of a deposit CTA keeps its
// own FP64 sums of the tile's window in shared memory and adds its particles
// to them in order, lane t owning value t = (stencil node, component).
// Only the owning warp touches a window, so plain loads and stores replace
// the grouping of equal cells, the fixed-point conversion and the two 64-bit
// shared atomics that each group of a shared window takes, and the order of
// the additions is that of the particles.  When the CTA leaves the tile, the
// warps' sums are added in warp order and folded into the grid's fixed-point
// accumulators, one conversion and two integer atomics per node and
// component.
#pragma once

#include "kernels.h"
#include "upic_common.cuh"

namespace upic {

// Extents of a private window: the tile window's, an axis that is one whole
// period extended by the stencil's reach, so that stencils never wrap inside
// the window (the fold wraps them).
struct PrivateWindow {
    int ex, ey;
};
UPIC_HD PrivateWindow private_window(const TileGeom& tg, int sx, int sy) {
    return PrivateWindow{tg.full_x ? tg.nx + sx - 1 : tg.wx, tg.full_y ? tg.ny + sy - 1 : tg.wy};
}
UPIC_HD int private_window_doubles(const TileGeom& tg, int sx, int sy, int ncomp) {
    const PrivateWindow w = private_window(tg, sx, sy);
    return w.ex * w.ey * ncomp;
}

// A warp's staged deposits: column k of its 32 particles is
// cols[k * kColStride + lane], the weights first and the deposit values from
// VAL on, zeros for a lane without a deposit.  Storing is conflict-free, and a
// lane reads two particles of a column with one 16-byte load; the stride of 34
// puts neighbouring columns in different banks.
constexpr int kColStride = 34;

// Adds the staged particles to the warp's window.  `key` (per lane): window
// offset in doubles of the particle's first node; valid: lanes with a deposit;
// heads: those of them whose key differs from that of the valid lane before.  Value t of a
// particle is weight ab[t] times value c[t], added at off[t].  The particles
// between two heads are summed in a register.
template <int NV, int VAL, int NPER>
UPIC_D void add_columns(const double* cols, int key, unsigned valid, unsigned heads, double* win,
                        const int (&ab)[NPER], const int (&c)[NPER], const int (&off)[NPER]) {
    const int lane = threadIdx.x & 31;
    const int rows = 32 - __clz(valid);
    int cur = -1;
    double acc[NPER];
    const double *wc[NPER], *vc[NPER];
#pragma unroll
    for (int r = 0; r < NPER; ++r) {
        acc[r] = 0.0;
        wc[r] = cols + ab[r] * kColStride;
        vc[r] = cols + (VAL + c[r]) * kColStride;
    }
    auto next = [&](int j) {
        if (cur >= 0) {
#pragma unroll
            for (int r = 0; r < NPER; ++r)
                if (lane + 32 * r < NV) win[cur + off[r]] += acc[r];
            __syncwarp();
        }
#pragma unroll
        for (int r = 0; r < NPER; ++r) acc[r] = 0.0;
        cur = __shfl_sync(0xffffffffu, key, j);
    };
    for (int j = 0; j < rows; j += 4) {
        double2 w0[NPER], w1[NPER], v0[NPER], v1[NPER];
#pragma unroll
        for (int r = 0; r < NPER; ++r) {
            w0[r] = *reinterpret_cast<const double2*>(wc[r] + j);
            w1[r] = *reinterpret_cast<const double2*>(wc[r] + j + 2);
            v0[r] = *reinterpret_cast<const double2*>(vc[r] + j);
            v1[r] = *reinterpret_cast<const double2*>(vc[r] + j + 2);
        }
        const unsigned h = heads >> j;
        if (h & 1u) next(j);
#pragma unroll
        for (int r = 0; r < NPER; ++r) acc[r] = fma(w0[r].x, v0[r].x, acc[r]);
        if (h & 14u) {
            if (h & 2u) next(j + 1);
#pragma unroll
            for (int r = 0; r < NPER; ++r) acc[r] = fma(w0[r].y, v0[r].y, acc[r]);
            if (h & 4u) next(j + 2);
#pragma unroll
            for (int r = 0; r < NPER; ++r) acc[r] = fma(w1[r].x, v1[r].x, acc[r]);
            if (h & 8u) next(j + 3);
#pragma unroll
            for (int r = 0; r < NPER; ++r) acc[r] = fma(w1[r].y, v1[r].y, acc[r]);
        } else {
#pragma unroll
            for (int r = 0; r < NPER; ++r)
                acc[r] = fma(w1[r].y, v1[r].y, fma(w1[r].x, v1[r].x, fma(w0[r].y, v0[r].y, acc[r])));
        }
    }
    if (cur >= 0) {
#pragma unroll
        for (int r = 0; r < NPER; ++r)
            if (lane + 32 * r < NV) win[cur + off[r]] += acc[r];
    }
    __syncwarp();
}

// Lanes that start a run of equal keys among the valid ones.
UPIC_D unsigned run_heads(int key, unsigned valid) {
    const int lane = threadIdx.x & 31;
    const unsigned before = valid & ((1u << lane) - 1u);
    const int prev = __shfl_sync(0xffffffffu, key, before ? 31 - __clz(before) : lane);
    return __ballot_sync(0xffffffffu, ((valid >> lane) & 1u) && (!before || prev != key));
}

// Adds the warps' windows (consecutive, `size` doubles each) to the grid
// accumulators and clears them.  Called by the whole CTA between barriers.
template <int NC, int WARPS, class Slot>
UPIC_D void fold_private(double* win, int size, const PrivateWindow& w, const TileGeom& tg, int ox, int oy,
                         unsigned long long* acc, const double* scale, Slot slot) {
    const int N = tg.nx * tg.ny;
    for (int i = threadIdx.x; i < size; i += blockDim.x) {
        double s = 0.0;
#pragma unroll
        for (int k = 0; k < WARPS; ++k) {
            s += win[k * size + i];
            win[k * size + i] = 0.0;
        }
        if (s == 0.0) continue;
        const int node = i / NC, c = slot(i - node * NC);
        const int lx = node / w.ey, ly = node - lx * w.ey;
        const int g = wrap_index(tg.full_x ? lx : ox + lx, tg.nx) * tg.ny + wrap_index(tg.full_y ? ly : oy + ly, tg.ny);
        const Fixed2 f = to_fixed(s, scale[c]);
        atomicAdd(&acc[(size_t)(2 * c) * N + g], f.hi);
        atomicAdd(&acc[(size_t)(2 * c + 1) * N + g], f.lo);
    }
}

}  // namespace upic
