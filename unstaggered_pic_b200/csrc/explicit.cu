// Explicit spectral BDF / IAEM step kernels (sm_100a).
//
// Reference: Project2/spectral_pic_part3.cpp (run_simulation :1094-1189).
// One step of the reference is
//   x += dt v; J = deposit(x, v); rho (continuity or redeposit); BDF wave
//   solves for phi, A; spectral grad phi, grad A; IAEM push; diagnostics.
// Here the particle work of a step is one fused kernel (push_deposit_kernel,
// kModePush): it recomputes x^n = wrap(x^{n-1} + dt v^{n-1}), gathers the
// eleven field records at x^n, pushes P and v, stores the step-n state, and
// already deposits the NEXT step's current J^{n+1} at wrap(x^n + dt v^n) with
// v^n (what the reference's next iteration deposits).  The field work of a
// step is a handful of grid kernels in k-space (histories kept as spectra).
#include <map>
#include <mutex>
#include <utility>
#include "deposit.cuh"
#include "kernels.h"
#include "upic_common.cuh"

namespace upic {

namespace {

// Threads per CTA and resident CTAs per SM the push kernel is compiled for
// (register budget 65536 / (threads * CTAs) per thread).
#ifndef UPIC_PUSH_THREADS
#define UPIC_PUSH_THREADS 256
#endif
#ifndef UPIC_PUSH_MIN_BLOCKS
#define UPIC_PUSH_MIN_BLOCKS 3
#endif
constexpr int kPushThreads = UPIC_PUSH_THREADS;
constexpr int kPushWarps = kPushThreads / kWarp;
// With private windows two CTAs fit an SM and their threads keep their values
// in registers.
constexpr int push_min_blocks(bool priv) { return priv ? 2 : UPIC_PUSH_MIN_BLOCKS; }
// Particles staged at a time for private windows: with four components two
// CTAs fit an SM only with half a warp's (107 KB; 120 KB with all).
constexpr int push_rows(int ncomp) { return ncomp == 4 ? 16 : 32; }
constexpr int kKeyNone = -1;
constexpr int kKeyEscape = -2;

// Per-warp staging: one row per particle with its 9 tensor-product stencil
// weights S_ab and its NCOMP deposit values (q v_c / dA, or q / dA).
template <int NCOMP>
struct StageLayout {
    static constexpr int kNV = 9 * NCOMP;   // values reduced per particle
    static constexpr int kRow = 9 + NCOMP;  // doubles staged per particle
    static constexpr int kDoubles = 32 * kRow;
};

UPIC_D int acc_slot(int ncomp, int c) { return ncomp == 1 ? 3 : c; }

// Window-local coordinate of a stencil origin node (tiled axis): -1 when the
// three-node stencil does not fit in the window.
UPIC_D int window_coord(int s, int origin, int n, int w) {
    const int d = (s - origin) & (n - 1);
    return d <= w - 3 ? d : -1;
}

// Fold a CTA's window into the global fixed-point accumulators (integer adds:
// order-independent, hence deterministic).
template <int NCOMP>
UPIC_D void fold_window(const unsigned long long* whi, const unsigned long long* wlo, int WN,
                        const TileGeom& tg, int ox, int oy, unsigned long long* acc) {
    const int N = tg.nx * tg.ny;
    for (int idx = threadIdx.x; idx < NCOMP * WN; idx += blockDim.x) {
        const unsigned long long hi = whi[idx], lo = wlo[idx];
        if ((hi | lo) == 0ull) continue;
        const int cc = idx / WN, widx = idx - cc * WN;
        const int lx = widx / tg.wy, ly = widx - lx * tg.wy;
        const int gx = tg.full_x ? lx : wrap_index(ox + lx, tg.nx);
        const int gy = tg.full_y ? ly : wrap_index(oy + ly, tg.ny);
        const int sl = acc_slot(NCOMP, cc);
        atomicAdd(&acc[(size_t)(2 * sl) * N + gx * tg.ny + gy], hi);
        atomicAdd(&acc[(size_t)(2 * sl + 1) * N + gx * tg.ny + gy], lo);
    }
}

// Bulk L2 prefetch (sm_90+ TMA unit) of elements [i0, i1) of a particle
// array.  The range is widened to 16-byte boundaries; particle arrays carry
// two elements of padding (alloc_soa), so the widened range stays inside
// the allocation.  A prefetch is a hint: it moves no data into the SM.
UPIC_D void prefetch_l2(const double* base, int i0, int i1) {
    if (!base || i1 <= i0) return;
    const unsigned long long a0 = reinterpret_cast<unsigned long long>(base + i0) & ~15ull;
    const unsigned long long a1 = (reinterpret_cast<unsigned long long>(base + i1) + 15ull) & ~15ull;
    const unsigned bytes = (unsigned)(a1 - a0);
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a0), "r"(bytes) : "memory");
}

// Prefetch of the particle state the CTA reads in its next batch of
// kPushThreads particles: the rest of this chunk, else the next chunk.
template <int MODE, bool UNIFORM>
UPIC_D void prefetch_next_batch(const PushArgs& a, const Chunk& ch, int base, int ci, int c_end) {
    int n0, n1;
    if (base + kPushThreads < ch.end) {
        n0 = base + kPushThreads;
        n1 = min(n0 + kPushThreads, ch.end);
    } else if (ci + 1 < c_end) {
        const Chunk nx = a.chunks[ci + 1];
        n0 = nx.start;
        n1 = min(nx.start + kPushThreads, nx.end);
    } else {
        return;
    }
    const int t = threadIdx.x;
    const double* arr = nullptr;
    switch (t) {
        case 0: arr = a.p.x; break;
        case 1: arr = a.p.y; break;
        case 2: arr = a.p.vx; break;
        case 3: arr = a.p.vy; break;
        case 4: arr = a.p.vz; break;
        case 5: arr = MODE == kModePush ? a.p.wx : nullptr; break;
        case 6: arr = MODE == kModePush ? a.p.wy : nullptr; break;
        case 7: arr = MODE == kModePush ? a.p.wz : nullptr; break;
        case 8: arr = MODE == kModePush ? a.p.Px : nullptr; break;
        case 9: arr = MODE == kModePush ? a.p.Py : nullptr; break;
        case 10: arr = MODE == kModePush ? a.p.Pz : nullptr; break;
        case 11: arr = UNIFORM ? nullptr : a.p.q; break;
        case 12: arr = UNIFORM ? nullptr : a.p.m; break;
        default: break;
    }
    prefetch_l2(arr, n0, n1);
}

// PRIV: warp-private windows (deposit.cuh); otherwise the CTA shares one
// window of fixed-point words, to which each group of equal cells of a warp
// adds its sums.
template <int MODE, int NCOMP, bool UNIFORM, bool PRIV>
__global__ void __launch_bounds__(kPushThreads, push_min_blocks(PRIV))
push_deposit_kernel(PushArgs a, TileGeom tg) {
    constexpr int NV = StageLayout<NCOMP>::kNV;
    constexpr int RW = StageLayout<NCOMP>::kRow;
    constexpr int NPER = (NV + 31) / 32;
    extern __shared__ unsigned long long smem_u64[];
    const int WN = tg.wx * tg.wy;
    unsigned long long* whi = smem_u64;
    unsigned long long* wlo = whi + NCOMP * WN;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const PrivateWindow pw = private_window(tg, 3, 3);
    const int psize = pw.ex * pw.ey * NCOMP;
    double* wins = reinterpret_cast<double*>(smem_u64);
    int* lost = reinterpret_cast<int*>(wins + kPushWarps * psize);
    constexpr int ROWS = push_rows(NCOMP), CS = col_stride(ROWS);
    constexpr int STAGE = PRIV ? RW * CS : StageLayout<NCOMP>::kDoubles;  // doubles staged per warp
    const int window_words = PRIV ? (kPushWarps * psize * 3 / 2 + 1) & ~1 : 2 * NCOMP * WN;
    double* sprod = reinterpret_cast<double*>(smem_u64 + window_words) + warp * STAGE;
    int* sgk = reinterpret_cast<int*>(smem_u64 + window_words + kPushWarps * STAGE) + warp * 32;
    // field records of the tile's window (kModePush): the gathers of
    // particles whose stencil lies in the window read them from here
    // (16-byte aligned; an offset from the shared base, so that the pointer
    // keeps the shared state space and the gathers are LDS, not generic
    // loads)
    double2* srec = reinterpret_cast<double2*>(
        smem_u64 + ((window_words + kPushWarps * STAGE + (PRIV ? 0 : kPushWarps * 16) + 1) & ~1));

    const int nx = tg.nx, ny = tg.ny;
    const int N = nx * ny;
    const int nch = *a.nchunks;
    const int c_begin = (int)(((long long)blockIdx.x * nch) / gridDim.x);
    const int c_end = (int)(((long long)(blockIdx.x + 1) * nch) / gridDim.x);

    // values owned by this lane in the segmented reduction: t = lane + 32 r is
    // stencil node ab = t / NCOMP (a = ab/3 along x, b = ab%3 along y) and
    // deposit component c = t % NCOMP
    int t_off[NPER], t_a[NPER], t_b[NPER], t_c[NPER], t_ab[NPER];
#pragma unroll
    for (int r = 0; r < NPER; ++r) {
        const int t = lane + 32 * r;
        const int ab = t < NV ? t / NCOMP : 0;
        t_ab[r] = ab;
        t_a[r] = ab / 3;
        t_b[r] = ab % 3;
        t_c[r] = t < NV ? t - ab * NCOMP : 0;
        t_off[r] = PRIV ? (t_a[r] * pw.ey + t_b[r]) * NCOMP + t_c[r] : t_a[r] * tg.wy + t_b[r];
    }
    if (PRIV) {
        for (int idx = threadIdx.x; idx < window_words; idx += blockDim.x) wins[idx] = 0.0;
        __syncthreads();
    }

    DD kin{0.0, 0.0}, gsum{0.0, 0.0};
    double vmax2 = 0.0;  // largest |v|^2 (sqrt taken once: sqrt is monotonic and correctly rounded)
    const double c2 = a.c * a.c;

    int cur_tile = -1, ox = 0, oy = 0;
    auto fold = [&]() {
        if constexpr (PRIV)
            fold_private<NCOMP, kPushWarps>(wins, lost, psize, pw, tg, ox, oy, a.acc, a.scale,
                                            [](int c) { return acc_slot(NCOMP, c); });
        else
            fold_window<NCOMP>(whi, wlo, WN, tg, ox, oy, a.acc);
    };
    for (int ci = c_begin; ci < c_end; ++ci) {
        const Chunk ch = a.chunks[ci];
        if (ch.tile != cur_tile) {
            __syncthreads();
            if (cur_tile >= 0) {
                fold();
                __syncthreads();
            }
            if (!PRIV)
                for (int idx = threadIdx.x; idx < 2 * NCOMP * WN; idx += blockDim.x) whi[idx] = 0ull;
            cur_tile = ch.tile;
            const int tx = cur_tile / tg.nty, ty = cur_tile - tx * tg.nty;
            ox = tg.full_x ? 0 : tx * tg.tile_x - tg.guard - 1;
            oy = tg.full_y ? 0 : ty * tg.tile_y - tg.guard - 1;
            if (MODE == kModePush) {
                const double2* g2 = reinterpret_cast<const double2*>(a.gfields);
                for (int idx = threadIdx.x; idx < WN * (kGFStride / 2); idx += blockDim.x) {
                    const int node = idx / (kGFStride / 2), f = idx - node * (kGFStride / 2);
                    const int lx = node / tg.wy, ly = node - lx * tg.wy;
                    const int gx = tg.full_x ? lx : ((ox + lx) & (nx - 1));
                    const int gy = tg.full_y ? ly : ((oy + ly) & (ny - 1));
                    srec[idx] = __ldg(g2 + (size_t)(gx * ny + gy) * (kGFStride / 2) + f);
                }
            }
            __syncthreads();
        }
        for (int base = ch.start; base < ch.end; base += kPushThreads) {
            const int p = base + threadIdx.x;
            const bool active = p < ch.end;
            if (threadIdx.x < 13) prefetch_next_batch<MODE, UNIFORM>(a, ch, base, ci, c_end);
            int key = kKeyNone, gx0 = 0, gy0 = 0;
            double dwx[3], dwy[3], dval[NCOMP];
            if (active) {
                const double q = UNIFORM ? a.q0 : a.p.q[p];
                double x = __ldcs(a.p.x + p), y = __ldcs(a.p.y + p);
                double v0 = __ldcs(a.p.vx + p), v1 = __ldcs(a.p.vy + p), v2 = __ldcs(a.p.vz + p);
                if (MODE == kModePush) {
                    // spectral_pic_part3.cpp:1050-1055: x^n = x^{n-1} + dt v^{n-1}
                    x = wrap_periodic(x + a.dt * v0, a.Lx, a.inv_Lx);
                    y = wrap_periodic(y + a.dt * v1, a.Ly, a.inv_Ly);
                    // gather A, grad phi, grad A at x^n (:1063-1078)
                    const Quad1D qx = quadratic_weights(x, a.inv_dx);
                    const Quad1D qy = quadratic_weights(y, a.inv_dy);
                    const double wxs[3] = {qx.w0, qx.w1, qx.w2};
                    const double wys[3] = {qy.w0, qy.w1, qy.w2};
                    double G[12];
#pragma unroll
                    for (int f = 0; f < 12; ++f) G[f] = 0.0;
                    const int lx0 = tg.full_x ? 0 : window_coord(qx.ic - 1, ox, nx, tg.wx);
                    const int ly0 = tg.full_y ? 0 : window_coord(qy.ic - 1, oy, ny, tg.wy);
                    if (lx0 >= 0 && ly0 >= 0) {
#pragma unroll
                        for (int ia = 0; ia < 3; ++ia) {
                            const int wxi = tg.full_x ? wrap_index(qx.ic - 1 + ia, nx) : lx0 + ia;
#pragma unroll
                            for (int ib = 0; ib < 3; ++ib) {
                                const int wyi = tg.full_y ? wrap_index(qy.ic - 1 + ib, ny) : ly0 + ib;
                                const double w = wxs[ia] * wys[ib];
                                const double2* rec = srec + (wxi * tg.wy + wyi) * (kGFStride / 2);
#pragma unroll
                                for (int f2 = 0; f2 < kGF / 2; ++f2) {
                                    const double2 r = rec[f2];
                                    G[2 * f2] = fma(r.x, w, G[2 * f2]);
                                    G[2 * f2 + 1] = fma(r.y, w, G[2 * f2 + 1]);
                                }
                                // the last field alone: the record's padding would
                                // take its share of the shared-memory return path,
                                // which bounds this kernel (71% busy)
                                G[kGF - 1] = fma(reinterpret_cast<const double*>(rec)[kGF - 1], w, G[kGF - 1]);
                            }
                        }
                    } else
#pragma unroll
                    for (int ia = 0; ia < 3; ++ia) {
                        const int gx = wrap_index(qx.ic - 1 + ia, nx);
#pragma unroll
                        for (int ib = 0; ib < 3; ++ib) {
                            const int gy = wrap_index(qy.ic - 1 + ib, ny);
                            const double w = wxs[ia] * wys[ib];
                            const double2* rec = reinterpret_cast<const double2*>(
                                a.gfields + (size_t)(gx * ny + gy) * kGFStride);
#pragma unroll
                            for (int f2 = 0; f2 < kGFStride / 2; ++f2) {
                                const double2 r = __ldg(rec + f2);
                                G[2 * f2] = fma(r.x, w, G[2 * f2]);
                                G[2 * f2 + 1] = fma(r.y, w, G[2 * f2 + 1]);
                            }
                        }
                    }
                    // IAEM momentum update (:1072-1090)
                    const double w0 = __ldcs(a.p.wx + p), w1 = __ldcs(a.p.wy + p), w2 = __ldcs(a.p.wz + p);
                    const double vs0 = 2.0 * v0 - w0, vs1 = 2.0 * v1 - w1, vs2 = 2.0 * v2 - w2;
                    const double gdx = G[5] * vs0 + G[7] * vs1 + G[9] * vs2;
                    const double gdy = G[6] * vs0 + G[8] * vs1 + G[10] * vs2;
                    const double qdt = q * a.dt;
                    const double P0 = __ldcs(a.p.Px + p) + qdt * (gdx - G[3]);
                    const double P1 = __ldcs(a.p.Py + p) + qdt * (gdy - G[4]);
                    const double P2 = __ldcs(a.p.Pz + p);
                    // velocity_from_canonical (:602-607)
                    const double m = UNIFORM ? a.m0 : a.p.m[p];
                    const double p0 = P0 - q * G[0], p1 = P1 - q * G[1], p2 = P2 - q * G[2];
                    const double mc2 = m * c2;
                    const double arg = c2 * (p0 * p0 + p1 * p1 + p2 * p2) + mc2 * mc2;
                    const double s = arg == 0.0 ? 0.0 : c2 * rsqrt(arg);
                    const double n0v = s * p0, n1v = s * p1, n2v = s * p2;
                    __stcs(a.p.x + p, x);
                    __stcs(a.p.y + p, y);
                    __stcs(a.p.Px + p, P0);
                    __stcs(a.p.Py + p, P1);
                    __stcs(a.p.wx + p, v0);
                    __stcs(a.p.wy + p, v1);
                    __stcs(a.p.wz + p, v2);
                    __stcs(a.p.vx + p, n0v);
                    __stcs(a.p.vy + p, n1v);
                    __stcs(a.p.vz + p, n2v);
                    v0 = n0v;
                    v1 = n1v;
                    v2 = n2v;
                }
                // particle diagnostics on the (new) velocity (:950-957)
                if (a.diag_part) {
                    const double m = UNIFORM ? a.m0 : a.p.m[p];
                    const double sp2 = v0 * v0 + v1 * v1 + v2 * v2;
                    const double one_m = 1.0 - sp2 * a.inv_c2;
                    const double gam = rsqrt(one_m > 1.0e-14 ? one_m : 1.0e-14);
                    gsum = dd_add(gsum, gam);
                    kin = dd_add(kin, (gam - 1.0) * m * a.c * a.c);
                    vmax2 = fmax(vmax2, sp2);
                }
                // deposit position: stored x (kModeDeposit) or one step ahead
                if (MODE != kModeDeposit) {
                    x = wrap_periodic(x + a.dt * v0, a.Lx, a.inv_Lx);
                    y = wrap_periodic(y + a.dt * v1, a.Ly, a.inv_Ly);
                }
                const Quad1D dx_ = quadratic_weights(x, a.inv_dx);
                const Quad1D dy_ = quadratic_weights(y, a.inv_dy);
                const double wxs[3] = {dx_.w0, dx_.w1, dx_.w2};
                const double wys[3] = {dy_.w0, dy_.w1, dy_.w2};
                const double qa = q * a.inv_dA;
                if (NCOMP == 1) {
                    dval[0] = qa;
                } else {
                    dval[0] = qa * v0;
                    dval[1] = qa * v1;
                    dval[2] = qa * v2;
                    if (NCOMP == 4) dval[NCOMP - 1] = qa;
                }
                gx0 = wrap_index(dx_.ic - 1, nx);
                gy0 = wrap_index(dy_.ic - 1, ny);
                const int lx = tg.full_x ? gx0 : window_coord(dx_.ic - 1, ox, nx, tg.wx);
                const int ly = tg.full_y ? gy0 : window_coord(dy_.ic - 1, oy, ny, tg.wy);
                key = (lx < 0 || ly < 0) ? kKeyEscape : PRIV ? (lx * pw.ey + ly) * NCOMP : lx * tg.wy + ly;
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    dwx[k] = wxs[k];
                    dwy[k] = wys[k];
                }
            }
            if constexpr (PRIV) {
                // stage S_ab and q v_c / dA column by column
                const unsigned full = 0xffffffffu;
                const unsigned valid = __ballot_sync(full, key >= 0);
                const unsigned esc = __ballot_sync(full, key == kKeyEscape);
                const Groups gr = group_rows(key, valid);
                double* mine = sprod + gr.row % ROWS;
                unsigned leaders = gr.leaders;
                int cur_key = 0;
#pragma unroll
                for (int first = 0; first < 32; first += ROWS) {
                    const bool here = gr.row / ROWS * ROWS == first;
                    if (here) {
#pragma unroll
                        for (int ia = 0; ia < 3; ++ia)
#pragma unroll
                            for (int ib = 0; ib < 3; ++ib)
                                mine[(ia * 3 + ib) * CS] = key == kKeyNone ? 0.0 : dwx[ia] * dwy[ib];
#pragma unroll
                        for (int cc = 0; cc < NCOMP; ++cc) mine[(9 + cc) * CS] = key == kKeyNone ? 0.0 : dval[cc];
                    }
                    __syncwarp();
                    if (esc) {
                        // stencils that leave the window (rare): exact fixed-point
                        // adds straight to the grid, then nothing for the window
                        for (unsigned e = __ballot_sync(full, here && key == kKeyEscape); e; e &= e - 1) {
                            const int l = __ffs(e) - 1, j = __shfl_sync(full, gr.row, l) % ROWS;
                            const int gxj = __shfl_sync(full, gx0, l);
                            const int gyj = __shfl_sync(full, gy0, l);
#pragma unroll
                            for (int r = 0; r < NPER; ++r) {
                                if (lane + 32 * r < NV) {
                                    const double v = sprod[(9 + t_c[r]) * CS + j] * sprod[t_ab[r] * CS + j];
                                    if (v != 0.0) {
                                        const int g = wrap_index(gxj + t_a[r], nx) * ny + wrap_index(gyj + t_b[r], ny);
                                        const int sl = acc_slot(NCOMP, t_c[r]);
                                        const Fixed2 f = to_fixed(v, a.scale[sl]);
                                        atomicAdd(&a.acc[(size_t)(2 * sl) * N + g], f.hi);
                                        atomicAdd(&a.acc[(size_t)(2 * sl + 1) * N + g], f.lo);
                                    }
                                }
                            }
                        }
                        __syncwarp();
                        if (here && key == kKeyEscape)
#pragma unroll
                            for (int cc = 0; cc < NCOMP; ++cc) mine[(9 + cc) * CS] = 0.0;
                        __syncwarp();
                    }
                    const int nrows = min(__popc(valid) - first, ROWS);
                    if (nrows > 0)
                        add_columns<NV, 9, ROWS, NPER>(sprod, key, leaders, cur_key, nrows, gr.heads >> first,
                                                       wins + warp * psize, lost + warp * psize, t_ab, t_c, t_off);
                    __syncwarp();
                }
                continue;
            }
            // Group the warp's particles by window key: groups in the order of
            // their first particle, particles in index order inside a group
            // (deterministic), escapes after all groups.
            const unsigned full = 0xffffffffu;
            const unsigned lt = (1u << lane) - 1u;
            const unsigned valid = __ballot_sync(full, key >= 0);
            const unsigned esc = __ballot_sync(full, key == kKeyEscape);
            const unsigned peers = __match_any_sync(full, key);
            int row = -1, nvalid = 0, ngroups = 0;
            unsigned heads = 0u;
            for (unsigned rem = valid; rem;) {
                const int l = __ffs(rem) - 1;
                const unsigned g = __shfl_sync(full, peers, l);
                const int gk = __shfl_sync(full, key, l);
                if ((g >> lane) & 1u) row = nvalid + __popc(g & lt);
                if (lane == 0) sgk[ngroups] = gk;
                heads |= 1u << nvalid;
                nvalid += __popc(g);
                rem &= ~g;
                ++ngroups;
            }
            if (key == kKeyEscape) row = nvalid + __popc(esc & lt);
            if (row >= 0) {
                // stage S_ab and q v_c / dA of this particle in its row
                double* mine = sprod + row * RW;
#pragma unroll
                for (int ia = 0; ia < 3; ++ia)
#pragma unroll
                    for (int ib = 0; ib < 3; ++ib) mine[ia * 3 + ib] = dwx[ia] * dwy[ib];
#pragma unroll
                for (int cc = 0; cc < NCOMP; ++cc) mine[9 + cc] = dval[cc];
            }
            __syncwarp();
            // Particles whose stencil leaves the window (rare): exact fixed-point
            // adds straight to the grid.
            {
                unsigned e = esc;
                int erow = nvalid;
                while (e) {
                    const int j = __ffs(e) - 1;
                    e &= e - 1;
                    const int gxj = __shfl_sync(full, gx0, j);
                    const int gyj = __shfl_sync(full, gy0, j);
#pragma unroll
                    for (int r = 0; r < NPER; ++r) {
                        const int t = lane + 32 * r;
                        if (t < NV) {
                            const double v = sprod[erow * RW + 9 + t_c[r]] * sprod[erow * RW + t_ab[r]];
                            if (v != 0.0) {
                                const int g = wrap_index(gxj + t_a[r], nx) * ny + wrap_index(gyj + t_b[r], ny);
                                const int sl = acc_slot(NCOMP, t_c[r]);
                                const Fixed2 f = to_fixed(v, a.scale[sl]);
                                atomicAdd(&a.acc[(size_t)(2 * sl) * N + g], f.hi);
                                atomicAdd(&a.acc[(size_t)(2 * sl + 1) * N + g], f.lo);
                            }
                        }
                    }
                    ++erow;
                }
            }
            // Warp-level segmented reduction: lane t owns value t and sums it over
            // the rows of each key group (two interleaved partial sums, fixed
            // order); each group adds its sum to the window once per value.
            {
                unsigned h = heads;
                int gi = 0;
                while (h) {
                    const int rs = __ffs(h) - 1;
                    h &= h - 1;
                    const int re = h ? __ffs(h) - 1 : nvalid;
                    const int k = sgk[gi++];
#pragma unroll
                    for (int r = 0; r < NPER; ++r) {
                        const int t = lane + 32 * r;
                        if (t < NV) {
                            double s0 = 0.0, s1 = 0.0;
                            // rows rs..re-1, two interleaved partial sums
                            const double* pv = sprod + rs * RW + 9 + t_c[r];
                            const double* pw = sprod + rs * RW + t_ab[r];
                            const double* const pe = sprod + re * RW + 9 + t_c[r];
                            for (; pv + RW < pe; pv += 2 * RW, pw += 2 * RW) {
                                s0 = fma(pv[0], pw[0], s0);
                                s1 = fma(pv[RW], pw[RW], s1);
                            }
                            if (pv < pe) s0 = fma(pv[0], pw[0], s0);
                            const double sum = s0 + s1;
                            if (sum != 0.0) {
                                int widx;
                                if (tg.full_x || tg.full_y) {
                                    const int kx = k / tg.wy, ky = k - kx * tg.wy;
                                    int nxl = kx + t_a[r], nyl = ky + t_b[r];
                                    if (tg.full_x) nxl &= tg.wx - 1;
                                    if (tg.full_y) nyl &= tg.wy - 1;
                                    widx = nxl * tg.wy + nyl;
                                } else {
                                    widx = k + t_off[r];
                                }
                                const Fixed2 f = to_fixed(sum, a.scale[acc_slot(NCOMP, t_c[r])]);
                                atomicAdd(&whi[t_c[r] * WN + widx], f.hi);
                                atomicAdd(&wlo[t_c[r] * WN + widx], f.lo);
                            }
                        }
                    }
                }
            }
            __syncwarp();
        }
    }
    __syncthreads();
    if (cur_tile >= 0) fold();
    // particle reductions: fixed order (lanes, then warps in index order)
    if (a.diag_part) {
        kin = warp_sum_dd(kin);
        gsum = warp_sum_dd(gsum);
        const double vmax = warp_max(sqrt(vmax2));
        __syncthreads();
        double* red = reinterpret_cast<double*>(smem_u64);
        if (lane == 0) {
            red[warp * 5 + 0] = kin.hi;
            red[warp * 5 + 1] = kin.lo;
            red[warp * 5 + 2] = gsum.hi;
            red[warp * 5 + 3] = gsum.lo;
            red[warp * 5 + 4] = vmax;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            DD k{0.0, 0.0}, g{0.0, 0.0};
            double vm = 0.0;
            for (int w = 0; w < kPushWarps; ++w) {
                k = dd_add_dd(k, DD{red[w * 5 + 0], red[w * 5 + 1]});
                g = dd_add_dd(g, DD{red[w * 5 + 2], red[w * 5 + 3]});
                vm = fmax(vm, red[w * 5 + 4]);
            }
            double* out = a.diag_part + (size_t)blockIdx.x * kDiagPart;
            out[0] = k.hi;
            out[1] = k.lo;
            out[2] = g.hi;
            out[3] = g.lo;
            out[4] = vm;
        }
    }
}

// acc -> doubles, then clear (kept on device for the next deposit).
__global__ void convert_acc_kernel(unsigned long long* acc, int N, double s0, double s1, double s2,
                                   double s3, double* J, double* rho, double n0, int mask,
                                   const double* bg) {
    for (int id = blockIdx.x * blockDim.x + threadIdx.x; id < N; id += gridDim.x * blockDim.x) {
        if (mask & 1) {
            const double sc[3] = {s0, s1, s2};
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                unsigned long long* h = acc + (size_t)(2 * c) * N;
                unsigned long long* l = acc + (size_t)(2 * c + 1) * N;
                J[(size_t)c * N + id] = from_fixed(h[id], l[id], 1.0 / sc[c]);
                h[id] = 0ull;
                l[id] = 0ull;
            }
        }
        if (mask & 2) {
            unsigned long long* h = acc + (size_t)6 * N;
            unsigned long long* l = acc + (size_t)7 * N;
            rho[id] = (bg ? bg[id] : n0) + from_fixed(h[id], l[id], 1.0 / s3);
            h[id] = 0ull;
            l[id] = 0ull;
        }
    }
}

UPIC_D double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
UPIC_D double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
UPIC_D double2 cscale(double s, double2 a) { return make_double2(s * a.x, s * a.y); }
// i*k*z
UPIC_D double2 cik(double k, double2 z) { return make_double2(-k * z.y, k * z.x); }

// ---- k-space step -----------------------------------------------------------
// Node (i, j)'s wave numbers from the axes' own rows and columns of the
// grid-sized tables (16 B per node less to read): kx depends on i alone, ky
// on j, and k2 = k2(i, 0) + k2(0, j) is the sum the host rounds.
// The BDF combinations' roundings are written out: u - s h in one, so that
// no instance of the kernel contracts them differently (the mixed form's FP32
// records depend on them bit for bit).
UPIC_D double2 cmul_add(double s, double2 h, double2 u) {
    return make_double2(__fma_rn(s, h.x, u.x), __fma_rn(s, h.y, u.y));
}

struct Wave {
    double kx, ky, k2;
};
UPIC_D Wave wave_at(const KGrid& g, int id) {
    const int i = id >> g.lny, j = id & (g.ny - 1);
    Wave w;
    w.kx = __ldg(g.kx + (i << g.lny));
    w.ky = __ldg(g.ky + j);
    w.k2 = g.nx > 1 && g.ny > 1 ? __dadd_rn(__ldg(g.k2 + (i << g.lny)), __ldg(g.k2 + j)) : __ldg(g.k2 + id);
    return w;
}
// Node of -k
UPIC_D int mirror_node(const KGrid& g, int id) {
    const int i = id >> g.lny, j = id & (g.ny - 1);
    return (((g.nx - i) & (g.nx - 1)) << g.lny) + ((g.ny - j) & (g.ny - 1));
}

// k-space BDF step: continuity / naive charge, BDF Helmholtz solves for phi
// and A (spectral_pic_part3.cpp:829-880, 1147-1164), spectra of the eleven
// gathered fields (:1166-1168).  Every field has a transform of its own: two
// real fields that share a complex one (as its real and imaginary parts) both
// take the rounding of the larger, and a field that is zero does not stay
// zero.  NA: BDF coefficients (2 or 3; the Helmholtz solves take 2 NA - 1),
// which fixes the number of history slots, so that all loads of a mode are in
// flight together.
template <int NA>
__global__ void __launch_bounds__(128) bdf_kspace_kernel(KspaceArgs a) {
    constexpr int NB = 2 * NA - 1;
    const int N = a.g.nx * a.g.ny;
    const double scale = 1.0 / (a.c * a.c * a.dt * a.dt);
    const int snew = a.head == 0 ? a.R - 1 : a.head - 1;
    size_t slot[NB - 1];
#pragma unroll
    for (int l = 0; l < NB - 1; ++l) slot[l] = (size_t)(a.head + l < a.R ? a.head + l : a.head + l - a.R) * N;
    const size_t FS = (size_t)a.R * N;  // one field's ring
    for (int id = blockIdx.x * blockDim.x + threadIdx.x; id < N; id += gridDim.x * blockDim.x) {
        const Wave w = wave_at(a.g, id);
        const double kx = w.kx, ky = w.ky;
        double2 J[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) J[c] = a.Jhat[(size_t)c * N + id];
        double2 H[4][NB - 1];
#pragma unroll
        for (int f = 0; f < 4; ++f)
#pragma unroll
            for (int l = 0; l < NB - 1; ++l) H[f][l] = a.hist[f * FS + slot[l] + id];
        double2 rho_new;
        if (a.conserving) {
            const double2 div = cik(1.0, make_double2(kx * J[0].x + ky * J[1].x, kx * J[0].y + ky * J[1].y));
            double2 hs = make_double2(0.0, 0.0);
#pragma unroll
            for (int l = 1; l < NA; ++l) hs = cmul_add(a.a[l], a.hist[4 * FS + slot[l - 1] + id], hs);
            const double2 num = cmul_add(a.dt, div, hs);
            rho_new = make_double2(-num.x / a.a[0], -num.y / a.a[0]);
        } else {
            rho_new = a.rho_dep[id];
        }
        const double denom = scale * a.b[0] + w.k2;
        // (b0 s + k^2) u = source - s sum b_l u^{n+1-l}: phi from rho / eps0, A from mu0 J
        double2 u[4];
        u[0] = make_double2(rho_new.x / a.eps0, rho_new.y / a.eps0);
#pragma unroll
        for (int c = 0; c < 3; ++c)
            u[1 + c] = make_double2(__dmul_rn(a.mu0, J[c].x), __dmul_rn(a.mu0, J[c].y));
#pragma unroll
        for (int f = 0; f < 4; ++f) {
#pragma unroll
            for (int l = 1; l < NB; ++l) u[f] = cmul_add(-(scale * a.b[l]), H[f][l - 1], u[f]);
            u[f] = make_double2(u[f].x / denom, u[f].y / denom);
            a.hist[f * FS + (size_t)snew * N + id] = u[f];
        }
        a.hist[4 * FS + (size_t)snew * N + id] = rho_new;
        double2* g = a.gspec;
#pragma unroll
        for (int c = 0; c < 3; ++c) g[(size_t)c * N + id] = u[1 + c];
#pragma unroll
        for (int f = 0; f < 4; ++f) {
            g[(3 + 2 * f) * (size_t)N + id] = cik(kx, u[f]);
            g[(4 + 2 * f) * (size_t)N + id] = cik(ky, u[f]);
        }
    }
}

// ---- diagnostics --------------------------------------------------------------
// Spectra of one mode's diagnostics fields (spectral_pic_part3.cpp:902-948):
// gauge, E (3), gauss, continuity, B = curl A (3), rho, using BDF first
// derivatives of the histories; J (3) after them.
constexpr int kDiagTerms = 13;

// HERM: of the modes' Hermitian parts (f(k) + conj f(-k)) / 2, the spectra of
// the real fields.
template <bool HERM>
UPIC_D void diag_terms(const DiagArgs& a, int id, double2* o) {
    const int N = a.g.nx * a.g.ny;
    const Wave w = wave_at(a.g, id);
    const double kx = w.kx, ky = w.ky;
    const int mir = HERM ? mirror_node(a.g, id) : id;
    auto val = [&](const double2* __restrict__ f) -> double2 {
        const double2 z = f[id];
        if (!HERM) return z;
        const double2 m = f[mir];
        return make_double2(0.5 * (z.x + m.x), 0.5 * (z.y - m.y));
    };
    auto H = [&](int field, int slot) -> double2 { return val(a.hist + ((size_t)field * a.R + slot) * N); };
    auto ddt = [&](int field) -> double2 {
        double2 r = cscale(a.a[0], H(field, a.slot_new));
        for (int l = 1; l < a.na; ++l) {
            const int sl = a.slot_prev0 + l - 1;
            r = cadd(r, cscale(a.a[l], H(field, sl < a.R ? sl : sl - a.R)));
        }
        return make_double2(r.x / a.dt, r.y / a.dt);
    };
    double2* J = o + 10;
#pragma unroll
    for (int c = 0; c < 3; ++c) J[c] = val(a.Jhat + (size_t)c * N);
    const double2 phi = H(0, a.slot_new);
    const double2 Ax = H(1, a.slot_new), Ay = H(2, a.slot_new), Az = H(3, a.slot_new);
    const double2 rho = H(4, a.slot_new);
    const double2 phit = ddt(0);
    const double2 divA = cik(1.0, make_double2(kx * Ax.x + ky * Ay.x, kx * Ax.y + ky * Ay.y));
    const double c2 = a.c * a.c;
    o[0] = cadd(make_double2(phit.x / c2, phit.y / c2), divA);
    const double2 Atx = ddt(1), Aty = ddt(2), Atz = ddt(3);
    const double2 gpx = cik(kx, phi), gpy = cik(ky, phi);
    o[1] = make_double2(-gpx.x - Atx.x, -gpx.y - Atx.y);
    o[2] = make_double2(-gpy.x - Aty.x, -gpy.y - Aty.y);
    o[3] = make_double2(-Atz.x, -Atz.y);
    const double2 divE = cik(1.0, make_double2(kx * o[1].x + ky * o[2].x, kx * o[1].y + ky * o[2].y));
    o[4] = csub(divE, make_double2(rho.x / a.eps0, rho.y / a.eps0));
    const double2 divJ = cik(1.0, make_double2(kx * J[0].x + ky * J[1].x, kx * J[0].y + ky * J[1].y));
    o[5] = cadd(ddt(4), divJ);
    o[6] = cik(ky, Az);
    o[7] = cik(-kx, Az);
    o[8] = csub(cik(kx, Ay), cik(ky, Ax));
    o[9] = rho;
}

// Spectrum of one diagnostics field (upic_get_field).
__global__ void diag_field_kernel(DiagArgs a, int which, double2* out) {
    const int N = a.g.nx * a.g.ny;
    for (int id = blockIdx.x * blockDim.x + threadIdx.x; id < N; id += gridDim.x * blockDim.x) {
        double2 o[kDiagTerms];
        diag_terms<false>(a, id, o);
        double2 r = o[0];
#pragma unroll
        for (int k = 1; k < 10; ++k)
            if (k == which) r = o[k];
        out[id] = r;
    }
}

constexpr int kRedThreads = 256;
constexpr int kNSums = 8;  // gauge, gauss, cont, Bz, B, E, rho, J

// The diagnostics row.  Sums of squares over the grid are taken in k-space,
// sum_x f^2 = (1/N) sum_k |f_hat|^2 (Parseval; double-double, fixed order), so
// that no field is transformed back: at 64 x 64 the ten inverse transforms,
// the reduction over their results and its one-warp finish took 60 of a
// step's 231 us, this launch takes 11 (512 x 512: 40).  A field is the real
// part of its transform, whose spectrum is (f(k) + conj f(-k)) / 2.  That part
// is taken of the histories and currents that the fields are formed from
// (taking it of the fields costs 4.7 us more a row, 32 x 32 and 64 x 64); of
// the fields themselves on a grid one cell high or wide, where the wave number
// is that of mode -1 at both k and -k (spectral_pic_part3.cpp:320-330), so
// that a derivative of a real field is not one.  One more block adds the push
// kernel's particle partials meanwhile; the last block to finish adds the
// blocks' partials in index order and writes the row (page-locked host
// memory).  A small grid's launch is one chain of latencies, which the
// particle sums were a part of while the last block took them (14.4 -> 10.6 us
// at 32 x 32).
template <bool ONE_CELL>
__global__ void __launch_bounds__(kRedThreads) diag_reduce_kernel(DiagArgs a) {
    const int N = a.g.nx * a.g.ny;
    const int nb = gridDim.x - 1;  // blocks of the field sums
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if ((int)blockIdx.x == nb) {
        __shared__ double part[kRedThreads / kWarp][kDiagPart];
        DD kin{0.0, 0.0}, gs{0.0, 0.0};
        double vmax = 0.0;
        for (int b = threadIdx.x; b < a.pcount; b += blockDim.x) {
            const double* p = a.pdiag + (size_t)b * kDiagPart;
            kin = dd_add_dd(kin, DD{p[0], p[1]});
            gs = dd_add_dd(gs, DD{p[2], p[3]});
            vmax = fmax(vmax, p[4]);
        }
        kin = warp_sum_dd(kin);
        gs = warp_sum_dd(gs);
        vmax = warp_max(vmax);
        if (lane == 0) {
            part[warp][0] = kin.hi;
            part[warp][1] = kin.lo;
            part[warp][2] = gs.hi;
            part[warp][3] = gs.lo;
            part[warp][4] = vmax;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            kin = gs = DD{0.0, 0.0};
            vmax = 0.0;
            for (int w = 0; w < kRedThreads / kWarp; ++w) {
                kin = dd_add_dd(kin, DD{part[w][0], part[w][1]});
                gs = dd_add_dd(gs, DD{part[w][2], part[w][3]});
                vmax = fmax(vmax, part[w][4]);
            }
            double* o = a.partials + (size_t)nb * 16;
            o[0] = kin.hi + kin.lo;
            o[1] = gs.hi + gs.lo;
            o[2] = vmax;
        }
    }
    DD s[kNSums];
#pragma unroll
    for (int k = 0; k < kNSums; ++k) s[k] = DD{0.0, 0.0};
    for (int id = blockIdx.x * blockDim.x + threadIdx.x; id < N && (int)blockIdx.x < nb; id += nb * blockDim.x) {
        double2 o[kDiagTerms];
        diag_terms<!ONE_CELL>(a, id, o);
        if (ONE_CELL) {
            double2 m[kDiagTerms];
            diag_terms<false>(a, mirror_node(a.g, id), m);
#pragma unroll
            for (int k = 0; k < kDiagTerms; ++k) o[k] = make_double2(0.5 * (o[k].x + m[k].x), 0.5 * (o[k].y - m[k].y));
        }
        constexpr int which[kDiagTerms] = {0, 5, 5, 5, 1, 2, 4, 4, 4, 6, 7, 7, 7};
#pragma unroll
        for (int k = 0; k < kDiagTerms; ++k) {
            DD& t = s[which[k]];
            t = dd_add_dd(dd_add_dd(t, dd_sq(o[k].x)), dd_sq(o[k].y));
        }
        s[3] = dd_add_dd(dd_add_dd(s[3], dd_sq(o[8].x)), dd_sq(o[8].y));
    }
    __shared__ double red[kRedThreads / kWarp][kNSums * 2];
#pragma unroll
    for (int k = 0; k < kNSums; ++k) {
        s[k] = warp_sum_dd(s[k]);
        if (lane == 0) {
            red[warp][2 * k] = s[k].hi;
            red[warp][2 * k + 1] = s[k].lo;
        }
    }
    __syncthreads();
    if (threadIdx.x < kNSums && (int)blockIdx.x < nb) {
        DD t{0.0, 0.0};
        for (int w = 0; w < kRedThreads / kWarp; ++w)
            t = dd_add_dd(t, DD{red[w][2 * threadIdx.x], red[w][2 * threadIdx.x + 1]});
        a.partials[(size_t)blockIdx.x * 16 + 2 * threadIdx.x] = t.hi;
        a.partials[(size_t)blockIdx.x * 16 + 2 * threadIdx.x + 1] = t.lo;
    }
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        last = atomicAdd(a.done, 1u) == gridDim.x - 1;
        if (last) *a.done = 0u;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    // one warp per field sum
    __shared__ double sums[kNSums];
    {
        DD t{0.0, 0.0};
        for (int b = lane; b < nb; b += 32) {
            const volatile double* p = a.partials + (size_t)b * 16 + 2 * warp;
            t = dd_add_dd(t, DD{p[0], p[1]});
        }
        t = warp_sum_dd(t);
        if (lane == 0) sums[warp] = t.hi + t.lo;
    }
    __syncthreads();
    const double invN = 1.0 / (double)N;
    auto tot = [&](int k) { return sums[k] * invN; };  // sum over the nodes
    double* r = a.row;
    if (threadIdx.x < kNSums) r[threadIdx.x] = sqrt(tot(threadIdx.x) * invN);
    if (threadIdx.x != kWarp) return;
    const volatile double* p = a.partials + (size_t)nb * 16;
    const double kinetic = p[0], gsum = p[1], vmax = p[2];
    const double field = 0.5 * a.eps0 * (tot(5) * a.dA) + 0.5 / a.mu0 * (tot(4) * a.dA);
    r[8] = field;
    r[9] = kinetic;
    r[10] = field + kinetic;
    r[11] = vmax;
    r[12] = a.np > 0 ? gsum / (double)a.np : 0.0;
}

__global__ void poisson_kspace_kernel(int N, const double* k2, const double2* rh, double eps0,
                                      double2* out) {
    for (int id = blockIdx.x * blockDim.x + threadIdx.x; id < N; id += gridDim.x * blockDim.x) {
        const double kk = k2[id];
        if (kk > 0.0) {
            const double d = eps0 * kk;
            out[id] = make_double2(rh[id].x / d, rh[id].y / d);
        } else {
            out[id] = make_double2(0.0, 0.0);
        }
    }
}

__global__ void derivative_kspace_kernel(int N, const double* k, const double2* in, double2* out) {
    for (int id = blockIdx.x * blockDim.x + threadIdx.x; id < N; id += gridDim.x * blockDim.x)
        out[id] = cik(k[id], in[id]);
}

__global__ void bdf_single_kernel(int N, const double* k2, const double2* src, const double2* hist,
                                  int nb, double b0, double b1, double b2, double b3, double b4,
                                  double scale, double2* out) {
    const double b[5] = {b0, b1, b2, b3, b4};
    for (int id = blockIdx.x * blockDim.x + threadIdx.x; id < N; id += gridDim.x * blockDim.x) {
        double2 r = src[id];
        for (int l = 1; l < nb; ++l) r = csub(r, cscale(scale * b[l], hist[(size_t)(l - 1) * N + id]));
        const double d = scale * b[0] + k2[id];
        out[id] = make_double2(r.x / d, r.y / d);
    }
}

__global__ void gather_scalar_kernel(int nx, int ny, double inv_dx, double inv_dy, const double* f,
                                     long np, const double* x, const double* y, double* out) {
    for (long p = blockIdx.x * (long)blockDim.x + threadIdx.x; p < np; p += (long)gridDim.x * blockDim.x) {
        const Quad1D qx = quadratic_weights(x[p], inv_dx);
        const Quad1D qy = quadratic_weights(y[p], inv_dy);
        const double wxs[3] = {qx.w0, qx.w1, qx.w2};
        const double wys[3] = {qy.w0, qy.w1, qy.w2};
        double v = 0.0;
        for (int ia = 0; ia < 3; ++ia) {
            const int gx = wrap_index(qx.ic - 1 + ia, nx);
            for (int ib = 0; ib < 3; ++ib) {
                const int gy = wrap_index(qy.ic - 1 + ib, ny);
                v = fma(f[gx * ny + gy], wxs[ia] * wys[ib], v);
            }
        }
        out[p] = v;
    }
}

__global__ void fill_hist_kernel(double2* h, int R, int N, const double2* src) {
    for (int id = blockIdx.x * blockDim.x + threadIdx.x; id < N; id += gridDim.x * blockDim.x) {
        const double2 v = src[id];
        for (int s = 0; s < R; ++s) h[(size_t)s * N + id] = v;
    }
}

int grid_for(long n, int threads) {
    long g = (n + threads - 1) / threads;
    if (g > 148 * 16) g = 148 * 16;
    if (g < 1) g = 1;
    return (int)g;
}

// Shared memory of the push kernels with private or shared windows.
int push_smem(const TileGeom& tg, int ncomp, bool priv) {
    const int records = 16 + tg.wx * tg.wy * kGFStride * 8;
    const int windows = priv ? private_window_bytes(tg, 3, 3, ncomp, kPushWarps) + 8 : 2 * ncomp * tg.wx * tg.wy * 8;
    const int stage = priv ? kPushWarps * (9 + ncomp) * col_stride(push_rows(ncomp)) * 8
                           : kPushWarps * (32 * (9 + ncomp) * 8 + 32 * 4);
    const int bytes = windows + stage + records;
    const int red = kPushWarps * 5 * 8;
    return bytes > red ? bytes : red;
}

// Private windows while two CTAs fit an SM, as with the default tile of 8
// cells (99 KB, 107 KB with the charge); larger windows stay shared.  A launch
// with shared windows and chunks of 2048, and one with private windows:
// 32 x 32 x 16 36 and 28 us, 64 x 64 x 64 64 and 29 us, 256 x 128 x 32 with the
// charge 184 and 119 us, 512 x 512 x 64 1480 and 1447 us.
bool push_private(const TileGeom& tg, int ncomp) { return push_smem(tg, ncomp, true) <= 113 * 1024; }

using PushKernel = void (*)(PushArgs, TileGeom);
PushKernel push_kernel(int mode, int ncomp, bool uniform, bool priv) {
#define UPIC_CASE(MODE, NC)                                                                                        \
    if (mode == MODE && ncomp == NC)                                                                               \
        return uniform ? (priv ? push_deposit_kernel<MODE, NC, true, true> : push_deposit_kernel<MODE, NC, true, false>) \
                       : (priv ? push_deposit_kernel<MODE, NC, false, true> : push_deposit_kernel<MODE, NC, false, false>);
    UPIC_CASE(kModeDeposit, 1)
    UPIC_CASE(kModeDeposit, 3)
    UPIC_CASE(kModeDeposit, 4)
    UPIC_CASE(kModeAdvanceDeposit, 3)
    UPIC_CASE(kModeAdvanceDeposit, 4)
    UPIC_CASE(kModePush, 3)
    UPIC_CASE(kModePush, 4)
#undef UPIC_CASE
    return nullptr;
}

}  // namespace

cudaError_t raise_smem_limit(const void* func, int bytes) {
    static std::mutex mu;
    static std::map<std::pair<const void*, int>, int> limit;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lock(mu);
    int& cur = limit[{func, dev}];
    if (bytes <= cur) return cudaSuccess;
    e = cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess) cur = bytes;
    return e;
}

static long g_launches = 0;
void count_launches(long n) { __atomic_fetch_add(&g_launches, n, __ATOMIC_RELAXED); }
long launches_total() { return __atomic_load_n(&g_launches, __ATOMIC_RELAXED); }

cudaError_t push_configure_smem(const TileGeom& tg) {
    for (int mode : {kModeDeposit, kModeAdvanceDeposit, kModePush})
        for (int nc : {1, 3, 4})
            for (bool uniform : {true, false}) {
                const bool priv = push_private(tg, nc);
                const PushKernel k = push_kernel(mode, nc, uniform, priv);
                if (!k) continue;
                const cudaError_t e = raise_smem_limit(reinterpret_cast<const void*>(k), push_smem(tg, nc, priv));
                if (e != cudaSuccess) return e;
            }
    return cudaSuccess;
}

int push_occupancy(const TileGeom& tg, int ncomp) {
    int n = 0;
    const bool priv = push_private(tg, ncomp);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, push_kernel(kModePush, ncomp, true, priv), kPushThreads,
                                                  push_smem(tg, ncomp, priv));
    return n;
}

// IAEM momentum push of a particle list in given fields
// (push_particles_momentum_and_velocity, spectral_pic_part3.cpp:1057-1090):
// quadratic gathers of A, grad phi and grad A at (x, y), P += q dt
// (-grad phi + (grad A) . v*), v* = 2 v - v_prev, then v from the canonical
// momentum (velocity_from_canonical :602).  F: 11 planar fields A (3),
// grad phi (2), dAx/dx, dAx/dy, dAy/dx, dAy/dy, dAz/dx, dAz/dy.  P, v,
// v_prev: xyz triples, updated in place.
__global__ void iaem_push_kernel(long np, const double* __restrict__ x, const double* __restrict__ y,
                                 double* __restrict__ P, double* __restrict__ v, double* __restrict__ vp,
                                 const double* __restrict__ q, const double* __restrict__ m,
                                 const double* __restrict__ F, int nx, int ny, double inv_dx, double inv_dy,
                                 double dt, double c) {
    const int N = nx * ny;
    for (long p = blockIdx.x * (long)blockDim.x + threadIdx.x; p < np; p += (long)gridDim.x * blockDim.x) {
        const Quad1D qx = quadratic_weights(x[p], inv_dx);
        const Quad1D qy = quadratic_weights(y[p], inv_dy);
        const double wx[3] = {qx.w0, qx.w1, qx.w2}, wy[3] = {qy.w0, qy.w1, qy.w2};
        double G[11];
        for (int f = 0; f < 11; ++f) G[f] = 0.0;
        for (int a = 0; a < 3; ++a) {
            const int gx = wrap_index(qx.ic - 1 + a, nx);
            for (int b = 0; b < 3; ++b) {
                const int node = gx * ny + wrap_index(qy.ic - 1 + b, ny);
                for (int f = 0; f < 11; ++f) G[f] += F[(size_t)f * N + node] * wx[a] * wy[b];
            }
        }
        const double vs[3] = {2.0 * v[3 * p] - vp[3 * p], 2.0 * v[3 * p + 1] - vp[3 * p + 1],
                              2.0 * v[3 * p + 2] - vp[3 * p + 2]};
        const double gv[2] = {G[5] * vs[0] + G[7] * vs[1] + G[9] * vs[2], G[6] * vs[0] + G[8] * vs[1] + G[10] * vs[2]};
        const double force[3] = {-G[3] + gv[0], -G[4] + gv[1], 0.0};
        const double qdt = q[p] * dt;
        double Pn[3], pm[3];
        for (int k = 0; k < 3; ++k) {
            Pn[k] = P[3 * p + k] + qdt * force[k];
            pm[k] = Pn[k] - q[p] * G[k];
        }
        const double mc2 = m[p] * c * c;
        const double den = sqrt(c * c * (pm[0] * pm[0] + pm[1] * pm[1] + pm[2] * pm[2]) + mc2 * mc2);
        const double s = den == 0.0 ? 0.0 : c * c / den;
        for (int k = 0; k < 3; ++k) {
            vp[3 * p + k] = v[3 * p + k];
            v[3 * p + k] = s * pm[k];
            P[3 * p + k] = Pn[k];
        }
    }
}

cudaError_t launch_iaem_push(long np, const double* x, const double* y, double* P, double* v, double* vp,
                             const double* q, const double* m, const double* F, int nx, int ny, double inv_dx,
                             double inv_dy, double dt, double c, cudaStream_t st) {
    long g = (np + 127) / 128;
    if (g > 148 * 16) g = 148 * 16;
    iaem_push_kernel<<<(int)(g < 1 ? 1 : g), 128, 0, st>>>(np, x, y, P, v, vp, q, m, F, nx, ny, inv_dx, inv_dy, dt,
                                                           c);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_push_deposit(int mode, int ncomp, bool uniform, const TileGeom& tg,
                                const PushArgs& a, int grid, cudaStream_t st) {
    const bool priv = push_private(tg, ncomp);
    const PushKernel k = push_kernel(mode, ncomp, uniform, priv);
    if (!k) return cudaErrorInvalidValue;
    k<<<grid, kPushThreads, push_smem(tg, ncomp, priv), st>>>(a, tg);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_convert_acc(unsigned long long* acc, int N, const double* scale, double* J,
                               double* rho, double n0, int mask, cudaStream_t st, const double* bg) {
    convert_acc_kernel<<<grid_for(N, 256), 256, 0, st>>>(acc, N, scale[0], scale[1], scale[2],
                                                         scale[3], J, rho, n0, mask, bg);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_bdf_kspace(const KspaceArgs& a, cudaStream_t st) {
    const int grid = grid_for((long)a.g.nx * a.g.ny, 128);
    if (a.na == 3) bdf_kspace_kernel<3><<<grid, 128, 0, st>>>(a);
    else bdf_kspace_kernel<2><<<grid, 128, 0, st>>>(a);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_diag_field(const DiagArgs& a, int which, double2* out, cudaStream_t st) {
    const int grid = grid_for((long)a.g.nx * a.g.ny, 256);
    diag_field_kernel<<<grid, 256, 0, st>>>(a, which, out);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_diag_reduce(const DiagArgs& a, cudaStream_t st) {
    long blocks = ((long)a.g.nx * a.g.ny + kRedThreads - 1) / kRedThreads;
    const int grid = 1 + (int)(blocks < a.max_blocks - 1 ? blocks : a.max_blocks - 1);
    if (a.g.nx > 1 && a.g.ny > 1) diag_reduce_kernel<false><<<grid, kRedThreads, 0, st>>>(a);
    else diag_reduce_kernel<true><<<grid, kRedThreads, 0, st>>>(a);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_poisson_kspace(int N, const double* k2, const double2* rho_hat, double eps0,
                                  double2* out, cudaStream_t st) {
    poisson_kspace_kernel<<<grid_for(N, 256), 256, 0, st>>>(N, k2, rho_hat, eps0, out);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_derivative_kspace(int N, const double* k, const double2* in, double2* out,
                                     cudaStream_t st) {
    derivative_kspace_kernel<<<grid_for(N, 256), 256, 0, st>>>(N, k, in, out);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_bdf_single(int N, const double* k2, const double2* src, const double2* hist,
                              int nb, const double* b, double scale, double2* out,
                              cudaStream_t st) {
    bdf_single_kernel<<<grid_for(N, 256), 256, 0, st>>>(N, k2, src, hist, nb, b[0], b[1], b[2], b[3],
                                                        b[4], scale, out);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_gather_scalar(int nx, int ny, double inv_dx, double inv_dy, const double* f,
                                 long np, const double* x, const double* y, double* out,
                                 cudaStream_t st) {
    gather_scalar_kernel<<<grid_for(np, 256), 256, 0, st>>>(nx, ny, inv_dx, inv_dy, f, np, x, y, out);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_fill_hist(double2* h, int R, int N, const double2* src, cudaStream_t st) {
    fill_hist_kernel<<<grid_for(N, 256), 256, 0, st>>>(h, R, N, src);
    count_launches(1);
    return cudaGetLastError();
}

}  // namespace upic
