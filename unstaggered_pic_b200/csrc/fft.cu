// Batched complex FFT for the collocated periodic grid (sm_100a).
//
// Replaces the reference's fft1d/fft2d (Project2/spectral_pic_part3.cpp:372-424;
// Project3/ec_pic_nyquist_projected.cpp:1566-1670): forward
// f_hat[k] = sum_j f[j] exp(-2 pi i jk/n); the inverse is scaled by 1/n in
// each 1D pass, and a 2D transform is the y-line pass followed by the x-line
// pass, as in the reference.
//
// A line of n points belongs to n/8 threads with eight points each in
// registers.  The log2 n decimation-in-time levels run three at a time (2 2 or
// 2 at the end where 3 does not divide log2 n), with one shared-memory
// exchange between such passes and none before the first (whose eight
// bit-reversed points are a stride apart, so it loads them from global
// memory) or after the last (which ends in natural order).  The levels and
// their twiddles (accurate table, exp(-2 pi i m/n)) are those of the plain
// radix-2 transform, so the results do not depend on the grouping.  A
// 512-point line then takes two exchanges; one level at a time in shared
// memory took nine, and a 64 x 64 grid kept 11 CTAs busy where it now fills
// 44.  Per launch, eleven inverse transforms before and after: 64 x 64
// 13.8-16.2 -> 2.4-3.2 us, 1024 x 1024 226-256 -> 79-125 us.
// Lines that fit a warp exchange without block barriers.  An x pass CTA takes
// a few adjacent columns, so its global accesses are runs along y.
//
// What bounds it: at 1024 x 1024 and above the memory passes (16 B read and
// 16 B written per point and pass), at small grids the latency of one load,
// the passes and one store.
#include "kernels.h"
#include "upic_common.cuh"

namespace upic {

namespace {

constexpr int kFftMaxLog = 13;

// Points per thread and threads per line.
template <int LOGN>
struct Shape {
    static constexpr int n = 1 << LOGN;
    static constexpr int E = n < 8 ? n : 8;
    static constexpr int T = n / E;
    // y pass: lines per CTA for about 128 threads
    static constexpr int ylines = T >= 128 ? 1 : 128 / T;
    static constexpr int ythreads = ylines * T;
    // x pass: columns per CTA for about 256 threads, at most 16
    static constexpr int xcols = T >= 512 ? 1 : T >= 128 ? 2 : T <= 16 ? 16 : 256 / T;
    static constexpr int xthreads = xcols * T;
    static constexpr bool exchanges = LOGN > 3;
};

// a b, its roundings written out so that forward and inverse, whose twiddles
// differ in the sign of the imaginary part, contract alike.
UPIC_D double2 cmul(double2 a, double2 b) {
    return make_double2(__fma_rn(a.x, b.x, -__dmul_rn(a.y, b.y)), __fma_rn(a.x, b.y, __dmul_rn(a.y, b.x)));
}

// Shared-memory slot of point i: the low three bits exclusive-ored with all
// higher groups of three, so that eight points that differ in any three
// adjacent bits (a pass' stores and loads by consecutive threads) lie in
// different 16-byte banks.
UPIC_D int swizzle(int i) { return i ^ (((i >> 3) ^ (i >> 6) ^ (i >> 9) ^ (i >> 12)) & 7); }

template <int BITS>
UPIC_D int reverse_bits(int v) {
    if constexpr (BITS == 0) return 0;
    else return (int)(__brev((unsigned)v) >> (32 - BITS));
}
constexpr int reverse_const(int v, int bits) {
    int r = 0;
    for (int k = 0; k < bits; ++k) r |= ((v >> k) & 1) << (bits - 1 - k);
    return r;
}

// Levels of the decimation-in-time transform of one line from 2^LNS on, RB at
// a time.  A group of 2^RB points that these levels combine is the points
// block 2^(LNS+RB) + j + m 2^LNS of the bit-reversed order, j < 2^LNS; thread
// t holds groups t + h T, point m of group h in v[h + B m].  addr(i): slot of
// point i in shared memory; sync(): barrier of the line's threads.  On entry
// (LNS = 0) v[e] is point t + e T of the input, on return of the output.
template <int LOGN, int LNS, bool INV, class Addr, class Sync>
UPIC_D void line_passes(double2* v, int t, double2* sm, const double2* __restrict__ tw, Addr addr, Sync sync) {
    constexpr int E = Shape<LOGN>::E, T = Shape<LOGN>::T;
    constexpr int REM = LOGN - LNS;
    if constexpr (REM > 0) {
        constexpr int RB = REM == 4 || REM == 2 ? 2 : (REM < 3 ? REM : 3);
        constexpr int R = 1 << RB, B = E / R;
#pragma unroll
        for (int h = 0; h < B; ++h) {
            const int j = (t + h * T) & ((1 << LNS) - 1);
            // the first pass holds its points in input order: point m of the
            // bit-reversed group is input point reverse(m)
            auto at = [&](int m) -> double2& { return v[h + B * (LNS == 0 ? reverse_const(m, RB) : m)]; };
#pragma unroll
            for (int l = 0; l < RB; ++l) {
#pragma unroll
                for (int m = 0; m < R; ++m) {
                    if (m & (1 << l)) continue;
                    // partner m + 2^l, twiddle index (j + (m mod 2^l) 2^LNS) n / 2^(LNS+l+1)
                    double2 w = __ldg(&tw[(j + ((m & ((1 << l) - 1)) << LNS)) << (LOGN - LNS - l - 1)]);
                    if (INV) w.y = -w.y;
                    double2 &a = at(m), &b = at(m + (1 << l));
                    const double2 u = a;
                    const double2 x = cmul(b, w);
                    a = make_double2(u.x + x.x, u.y + x.y);
                    b = make_double2(u.x - x.x, u.y - x.y);
                }
            }
        }
        if constexpr (LNS + RB < LOGN) {
#pragma unroll
            for (int h = 0; h < B; ++h) {
                const int q = t + h * T;
                const int block = LNS == 0 ? reverse_bits<LOGN - RB>(q) : q >> LNS;
                const int base = (block << (LNS + RB)) + (q & ((1 << LNS) - 1));
#pragma unroll
                for (int m = 0; m < R; ++m)
                    sm[addr(base + (m << LNS))] = v[h + B * (LNS == 0 ? reverse_const(m, RB) : m)];
            }
            sync();
            constexpr int LN2 = LNS + RB, REM2 = LOGN - LN2;
            constexpr int RB2 = REM2 == 4 || REM2 == 2 ? 2 : (REM2 < 3 ? REM2 : 3);
            constexpr int R2 = 1 << RB2, B2 = E / R2;
#pragma unroll
            for (int h = 0; h < B2; ++h) {
                const int q = t + h * T;
                const int base = ((q >> LN2) << (LN2 + RB2)) + (q & ((1 << LN2) - 1));
#pragma unroll
                for (int m = 0; m < R2; ++m) v[h + B2 * m] = sm[addr(base + (m << LN2))];
            }
            if constexpr (LN2 + RB2 < LOGN) sync();  // another exchange follows
            line_passes<LOGN, LN2, INV>(v, t, sm, tw, addr, sync);
        } else if constexpr (LNS == 0) {
            // the only pass of a short line: from input to natural order
            double2 o[E];
#pragma unroll
            for (int m = 0; m < E; ++m) o[m] = v[reverse_const(m, RB)];
#pragma unroll
            for (int m = 0; m < E; ++m) v[m] = o[m];
        }
    }
}

struct FftArgs {
    double2* data;
    int nlines;               // y pass: components * nx; x pass: components
    int lognx, logny;
    const double2* tw;
    const double* rin;        // forward: real planar input or null
    int out_mode;             // inverse
    void* rout;
    int rec_stride, comp_offset;
    FftAccIn acc;             // y forward from accumulators
};

enum YPass { kForward = 0, kInverse = 1, kForwardAcc = 2, kForwardAcc1 = 3 };

// Values of component c at E nodes from the accumulators, which are cleared.
// All words are read before the first store, so that the loads overlap (6.4
// -> 3.6 us a launch at 32 x 32, 23 -> 9.6 us at 512 x 512).
template <bool SINGLE, int E>
UPIC_D void take_acc(const FftAccIn& a, int c, size_t N, size_t node, int step, double (&v)[E]) {
    unsigned long long* h = a.acc + (size_t)(2 * c) * N + node;
    unsigned long long hi[E], lo[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
        hi[e] = h[e * step];
        lo[e] = SINGLE ? 0ull : h[N + e * step];
    }
    const double* bg = c == 3 ? a.bg : nullptr;
    const double add = c == 3 ? a.n0 : 0.0;
    double b[E];
#pragma unroll
    for (int e = 0; e < E; ++e) b[e] = bg ? bg[node + e * step] : add;
    double* out = c == 3 ? a.rho + node : a.J + c * N + node;
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const double f = SINGLE ? (double)(long long)hi[e] / a.scale[c] : from_fixed(hi[e], lo[e], 1.0 / a.scale[c]);
        v[e] = c == 3 ? b[e] + f : f;
        h[e * step] = 0ull;
        if (!SINGLE) h[N + e * step] = 0ull;
        out[e * step] = v[e];
    }
}

// y lines (contiguous), the first pass.  Forward: complex, real planar or
// accumulators in; inverse: complex in.  Complex out, in `data`.
template <int LOGN, int PASS>
__global__ void __launch_bounds__(Shape<LOGN>::ythreads) fft_y_kernel(FftArgs a) {
    using S = Shape<LOGN>;
    constexpr bool INV = PASS == kInverse;
    extern __shared__ double2 smem[];
    const int l = threadIdx.x / S::T, t = threadIdx.x % S::T;
    const int line = blockIdx.x * S::ylines + l;
    const bool on = line < a.nlines;
    const int p = line >> a.lognx, row = line & ((1 << a.lognx) - 1);
    const size_t N = (size_t)1 << (a.lognx + LOGN);
    double2* d = a.data + (size_t)line * S::n;
    double2 v[S::E];
#pragma unroll
    for (int e = 0; e < S::E; ++e) v[e] = make_double2(0.0, 0.0);
    if (on) {
        if constexpr (PASS == kForwardAcc || PASS == kForwardAcc1) {
            constexpr bool single = PASS == kForwardAcc1;
            const size_t node = (size_t)row * S::n + t;
            double re[S::E];
            take_acc<single>(a.acc, p, N, node, S::T, re);
#pragma unroll
            for (int e = 0; e < S::E; ++e) v[e].x = re[e];
        } else if (!INV && a.rin) {
            const double* r = a.rin + (size_t)line * S::n;
#pragma unroll
            for (int e = 0; e < S::E; ++e) v[e].x = r[t + e * S::T];
        } else {
#pragma unroll
            for (int e = 0; e < S::E; ++e) v[e] = d[t + e * S::T];
        }
    }
    // lines of fewer than eight threads share a bank phase: they start in different banks
    const int shift = S::T < 8 ? (l * S::T) & 7 : 0;
    line_passes<LOGN, 0, INV>(
        v, t, smem + l * S::n, a.tw, [shift](int i) { return swizzle(i) ^ shift; },
        [] {
            if (S::T <= 32) __syncwarp();
            else __syncthreads();
        });
    if (!on) return;
    constexpr double sc = INV ? 1.0 / (double)S::n : 1.0;
#pragma unroll
    for (int e = 0; e < S::E; ++e) d[t + e * S::T] = make_double2(sc * v[e].x, sc * v[e].y);
}

// x lines, the second pass: element i of column j of transform c is at
// c N + i ny + j; a CTA takes 2^logcols adjacent columns.  Forward: complex in
// place; inverse: out_mode out.
template <int LOGN, bool INV>
__global__ void __launch_bounds__(Shape<LOGN>::xthreads) fft_x_kernel(FftArgs a, int logcols) {
    using S = Shape<LOGN>;
    extern __shared__ double2 smem[];
    const int col = threadIdx.x & ((1 << logcols) - 1), t = threadIdx.x >> logcols;
    const int logblocks = a.logny - logcols;
    const int p = blockIdx.x >> logblocks;
    const int j = ((blockIdx.x & ((1 << logblocks) - 1)) << logcols) + col;
    const size_t N = (size_t)1 << (LOGN + a.logny);
    double2* d = a.data + p * N + j;
    double2 v[S::E];
#pragma unroll
    for (int e = 0; e < S::E; ++e) v[e] = d[(size_t)(t + e * S::T) << a.logny];
    line_passes<LOGN, 0, INV>(
        v, t, smem, a.tw, [logcols, col](int i) { return (swizzle(i) << logcols) + col; }, [] { __syncthreads(); });
    constexpr double sc = INV ? 1.0 / (double)S::n : 1.0;
#pragma unroll
    for (int e = 0; e < S::E; ++e) {
        const size_t at = (size_t)(t + e * S::T) << a.logny, node = at + j;
        const double re = sc * v[e].x, im = sc * v[e].y;
        if (!INV || a.out_mode == 0) {
            d[at] = make_double2(re, im);
        } else if (a.out_mode == 1) {
            static_cast<double*>(a.rout)[p * N + node] = re;
        } else if (a.out_mode == 2) {
            static_cast<double*>(a.rout)[node * a.rec_stride + a.comp_offset + p] = re;
        } else {
            static_cast<float*>(a.rout)[node * a.rec_stride + a.comp_offset + p] = (float)re;
        }
    }
}

int ilog2(int n) {
    int l = 0;
    while ((1 << l) < n) ++l;
    return l;
}

template <int LOGN>
int y_smem() {
    return Shape<LOGN>::exchanges ? (int)sizeof(double2) * Shape<LOGN>::ylines * Shape<LOGN>::n : 0;
}
template <int LOGN>
int x_smem(int cols) {
    return Shape<LOGN>::exchanges ? (int)sizeof(double2) * cols * Shape<LOGN>::n : 0;
}

using YKernel = void (*)(FftArgs);
template <int LOGN>
YKernel y_kernel(int pass) {
    switch (pass) {
        case kInverse: return fft_y_kernel<LOGN, kInverse>;
        case kForwardAcc: return fft_y_kernel<LOGN, kForwardAcc>;
        case kForwardAcc1: return fft_y_kernel<LOGN, kForwardAcc1>;
        default: return fft_y_kernel<LOGN, kForward>;
    }
}

template <int LOGN>
void launch_y(const FftArgs& a, int pass, cudaStream_t st) {
    using S = Shape<LOGN>;
    const int grid = (a.nlines + S::ylines - 1) / S::ylines;
    y_kernel<LOGN>(pass)<<<grid, S::ythreads, y_smem<LOGN>(), st>>>(a);
}

template <int LOGN>
void launch_x(const FftArgs& a, bool inverse, cudaStream_t st) {
    using S = Shape<LOGN>;
    const int ny = 1 << a.logny;
    const int cols = S::xcols < ny ? S::xcols : ny;
    const int grid = a.nlines * (ny / cols);
    if (inverse) fft_x_kernel<LOGN, true><<<grid, cols * S::T, x_smem<LOGN>(cols), st>>>(a, ilog2(cols));
    else fft_x_kernel<LOGN, false><<<grid, cols * S::T, x_smem<LOGN>(cols), st>>>(a, ilog2(cols));
}

template <int LOGN>
cudaError_t raise_one() {
    cudaError_t e = cudaSuccess;
    if constexpr (LOGN >= 0) {
        for (int pass = kForward; pass <= kForwardAcc1 && y_smem<LOGN>() > 48 * 1024 && e == cudaSuccess; ++pass)
            e = raise_smem_limit(reinterpret_cast<const void*>(y_kernel<LOGN>(pass)), y_smem<LOGN>());
        if (x_smem<LOGN>(Shape<LOGN>::xcols) > 48 * 1024) {
            const int b = x_smem<LOGN>(Shape<LOGN>::xcols);
            if (e == cudaSuccess) e = raise_smem_limit(reinterpret_cast<const void*>(fft_x_kernel<LOGN, false>), b);
            if (e == cudaSuccess) e = raise_smem_limit(reinterpret_cast<const void*>(fft_x_kernel<LOGN, true>), b);
        }
        if (e == cudaSuccess) e = raise_one<LOGN - 1>();
    }
    return e;
}

#define UPIC_FFT_SIZES(F) F(0) F(1) F(2) F(3) F(4) F(5) F(6) F(7) F(8) F(9) F(10) F(11) F(12) F(13)

void run_y(int logn, const FftArgs& a, int pass, cudaStream_t st) {
    switch (logn) {
#define UPIC_CASE(L) case L: launch_y<L>(a, pass, st); break;
        UPIC_FFT_SIZES(UPIC_CASE)
#undef UPIC_CASE
    }
}

void run_x(int logn, const FftArgs& a, bool inverse, cudaStream_t st) {
    switch (logn) {
#define UPIC_CASE(L) case L: launch_x<L>(a, inverse, st); break;
        UPIC_FFT_SIZES(UPIC_CASE)
#undef UPIC_CASE
    }
}

}  // namespace

namespace {

// Both passes of `a` (its plan-dependent members are filled in here).
cudaError_t run_2d(const FftPlan& p, FftArgs a, int ncomp, int pass, cudaStream_t st) {
    const int lx = ilog2(p.nx), ly = ilog2(p.ny);
    if (lx > kFftMaxLog || ly > kFftMaxLog) return cudaErrorInvalidValue;
    a.lognx = lx;
    a.logny = ly;
    FftArgs x = a;
    a.nlines = ncomp << lx;
    a.tw = p.tw_y;
    x.nlines = ncomp;
    x.tw = p.tw_x;
    run_y(ly, a, pass, st);
    run_x(lx, x, pass == kInverse, st);
    count_launches(2);
    return cudaGetLastError();
}

}  // namespace

cudaError_t fft2d_batched(const FftPlan& p, double2* data, int ncomp, int inverse, cudaStream_t st,
                          const double* real_in, int out_mode, void* real_out, int rec_stride, int comp_offset) {
    FftArgs a{};
    a.data = data;
    a.rin = inverse ? nullptr : real_in;
    a.out_mode = out_mode;
    a.rout = real_out;
    a.rec_stride = rec_stride;
    a.comp_offset = comp_offset;
    return run_2d(p, a, ncomp, inverse ? kInverse : kForward, st);
}

cudaError_t fft2d_from_acc(const FftPlan& p, double2* data, int ncomp, const FftAccIn& acc, cudaStream_t st) {
    FftArgs a{};
    a.data = data;
    a.acc = acc;
    return run_2d(p, a, ncomp, acc.single ? kForwardAcc1 : kForwardAcc, st);
}

cudaError_t fft_configure_smem() { return raise_one<kFftMaxLog>(); }

}  // namespace upic
