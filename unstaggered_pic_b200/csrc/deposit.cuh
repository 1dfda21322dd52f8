// Warp-private deposit windows (sm_100a): each warp of a deposit CTA keeps its
// own sums of the tile's window in shared memory.  It adds up to 32 particles
// at a time, grouped by cell: a group is summed in registers, lane t owning
// value t = (stencil node, component), and then added to the window.  Only the
// owning warp touches a window, so plain loads and stores replace the
// fixed-point conversion and the two 64-bit shared atomics that each group of
// a shared window takes.
// A window sum is an FP64 value and the upper half of another that collects
// the exact errors of the additions to it: 20 bits more than FP64, so that
// what cancels in a window leaves no more behind than in the grid's
// fixed-point accumulators.  When the CTA leaves the tile, the warps' sums are
// added in double-double, in warp order, and folded into the accumulators, two
// conversions and two integer atomics per node and component.
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
// Bytes of `warps` windows: the FP64 sums of all of them, then their lost parts.
UPIC_HD int private_window_bytes(const TileGeom& tg, int sx, int sy, int ncomp, int warps) {
    const PrivateWindow w = private_window(tg, sx, sy);
    return warps * w.ex * w.ey * ncomp * (int)(sizeof(double) + sizeof(int));
}

// A warp's staged deposits: column k of ROWS of its particles is
// cols[k * col_stride(ROWS) + row], the weights first and the deposit values
// from VAL on, zeros for a lane without a deposit.  Storing is conflict-free,
// and a lane reads two particles of a column with one 16-byte load; two rows
// of padding put neighbouring columns in different banks.
constexpr int col_stride(int rows) { return rows + 2; }
constexpr int kNoKey = -1;

// Adds `rows` staged particles to the warp's window.  heads: rows that start a
// group; key (per lane): window offset of the lane's first node; leaders: the
// lanes whose keys the next groups have, consumed; cur: key of the group that
// row 0 continues if it starts none, and of the last one on return.  Value t
// of a particle is weight ab[t] times value c[t], added at off[t].
template <int NV, int VAL, int ROWS, int NPER>
UPIC_D void add_columns(const double* cols, int key, unsigned& leaders, int& cur, int rows, unsigned heads, double* win,
                        int* lost, const int (&ab)[NPER], const int (&c)[NPER], const int (&off)[NPER]) {
    const int lane = threadIdx.x & 31;
    double acc[NPER];
    const double *wc[NPER], *vc[NPER];
#pragma unroll
    for (int r = 0; r < NPER; ++r) {
        acc[r] = 0.0;
        wc[r] = cols + ab[r] * col_stride(ROWS);
        vc[r] = cols + (VAL + c[r]) * col_stride(ROWS);
    }
    // a group's sums are read when it starts, so that their latency lies under
    // its additions
    double was[NPER];
    int part[NPER];
    auto flush = [&]() {
#pragma unroll
        for (int r = 0; r < NPER; ++r) {
            if (lane + 32 * r >= NV) continue;
            const int i = cur + off[r];
            const double s = was[r] + acc[r], d = s - was[r];
            win[i] = s;
            lost[i] = __double2hiint(__hiloint2double(part[r], 0) + ((was[r] - (s - d)) + (acc[r] - d)));
        }
        __syncwarp();
    };
    auto open = [&]() {
#pragma unroll
        for (int r = 0; r < NPER; ++r) {
            acc[r] = 0.0;
            was[r] = win[cur + off[r]];
            part[r] = lost[cur + off[r]];
        }
    };
    bool any = !(heads & 1u);
    if (any) open();
    auto next = [&]() {
        if (any) flush();
        any = true;
        cur = __shfl_sync(0xffffffffu, key, __ffs(leaders) - 1);
        leaders &= leaders - 1;
        open();
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
        if (h & 1u) next();
#pragma unroll
        for (int r = 0; r < NPER; ++r) acc[r] = fma(w0[r].x, v0[r].x, acc[r]);
        if (h & 14u) {
            if (h & 2u) next();
#pragma unroll
            for (int r = 0; r < NPER; ++r) acc[r] = fma(w0[r].y, v0[r].y, acc[r]);
            if (h & 4u) next();
#pragma unroll
            for (int r = 0; r < NPER; ++r) acc[r] = fma(w1[r].x, v1[r].x, acc[r]);
            if (h & 8u) next();
#pragma unroll
            for (int r = 0; r < NPER; ++r) acc[r] = fma(w1[r].y, v1[r].y, acc[r]);
        } else {
#pragma unroll
            for (int r = 0; r < NPER; ++r)
                acc[r] = fma(w1[r].y, v1[r].y, fma(w1[r].x, v1[r].x, fma(w0[r].y, v0[r].y, acc[r])));
        }
    }
    flush();
}

// Rows of a warp's valid lanes grouped by key: groups in the order of their
// first lanes, lanes in order inside a group, the other lanes (whose key must
// be negative) after them.  leaders: the groups' first lanes, in the order of
// the heads.
struct Groups {
    int row;
    unsigned heads, leaders;
};
UPIC_D Groups group_rows(int key, unsigned valid) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    const bool on = (valid >> lane) & 1u;
    const unsigned peers = __match_any_sync(full, on ? key : kNoKey);
    const int leader = __ffs(peers) - 1;
    const bool lead = on && leader == lane;
    int before = lead ? __popc(peers) : 0;
    const int mine = before;
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(full, before, o);
        if (lane >= o) before += y;
    }
    before -= mine;
    const int base = __shfl_sync(full, before, leader);
    Groups g;
    g.row = on ? base + __popc(peers & lt) : __popc(valid) + __popc(~valid & lt);
    g.leaders = __ballot_sync(full, lead);
    g.heads = __reduce_or_sync(full, lead ? 1u << base : 0u);
    return g;
}

// Adds the warps' windows (`size` sums each) to the grid accumulators and
// clears them.  Called by the whole CTA between barriers.
template <int NC, int WARPS, class Slot>
UPIC_D void fold_private(double* win, int* lost, int size, const PrivateWindow& w, const TileGeom& tg, int ox,
                         int oy, unsigned long long* acc, const double* scale, Slot slot) {
    const int N = tg.nx * tg.ny;
    for (int i = threadIdx.x; i < size; i += blockDim.x) {
        DD s{0.0, 0.0};
#pragma unroll
        for (int k = 0; k < WARPS; ++k) {
            s = dd_add(s, win[k * size + i]);
            s.lo += __hiloint2double(lost[k * size + i], 0);
            win[k * size + i] = 0.0;
            lost[k * size + i] = 0;
        }
        const int node = i / NC, c = slot(i - node * NC);
        if (s.hi == 0.0 && s.lo == 0.0) continue;
        const int lx = node / w.ey, ly = node - lx * w.ey;
        const int g = wrap_index(tg.full_x ? lx : ox + lx, tg.nx) * tg.ny + wrap_index(tg.full_y ? ly : oy + ly, tg.ny);
        const Fixed2 f = to_fixed(s.hi, scale[c]), e = to_fixed(s.lo, scale[c]);
        atomicAdd(&acc[(size_t)(2 * c) * N + g], f.hi + e.hi);
        atomicAdd(&acc[(size_t)(2 * c + 1) * N + g], f.lo + e.lo);
    }
}

}  // namespace upic
