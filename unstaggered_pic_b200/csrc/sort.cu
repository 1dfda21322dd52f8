// Particle ordering for the tiled deposit (sm_100a).
//
// The reference keeps particles in a fixed array order and scatters them one
// by one (Project2/spectral_pic_part3.cpp:747-755); it has no sorting.  Here
// particles are periodically reordered by the nearest-node cell of their next
// gather position, in tile-major cell order, so that a warp's 32 particles
// share a handful of cells (broadcast gathers, long runs in the segmented
// deposit reduction) and a CTA's chunk fits one shared-memory window.  The
// implicit methods order a tile's particles by the number of knots their
// orbits pass before their cells (TileGeom::classes): a warp that walks its
// lanes' segments in rounds otherwise takes two or three rounds for a mean of
// 1.2 segments.
//
// The sort is a stable LSD radix sort of (cell key, index) pairs written for
// this purpose: block histograms, a device-wide exclusive scan, and a scatter
// whose in-block ranks come from warp match/popc and per-warp counts in fixed
// order.  It is therefore deterministic: equal inputs give equal orders, and
// with it the deposit's fixed summation order.
#include "kernels.h"
#include "upic_common.cuh"

namespace upic {

namespace {

constexpr int kSortThreads = 256;
// Keys per thread of a radix pass: 16 (4096-key blocks) for sets that fill the
// GPU with such blocks, 4 below: a 16,384-particle pass then runs 16 blocks of
// four rounds instead of four blocks of sixteen (scatter 16.3 -> 5.7 us).
constexpr int kSortItems = 16, kSortItemsSmall = 4;
constexpr long kSortSmall = 148L * kSortThreads * kSortItems;
constexpr int sort_tile(int items) { return kSortThreads * items; }  // elements per block
constexpr int kSortWarps = kSortThreads / kWarp;
constexpr int kMaxDigits = 256;                       // 8-bit digits at most
constexpr int kScanThreads = 256;
constexpr int kScanItems = 4;
constexpr int kScanTile = kScanThreads * kScanItems;

template <bool CLASSES>
__global__ void make_keys_kernel(TileGeom tg, ParticleSoA p, long np, double Lx, double Ly,
                                 double inv_dx, double inv_dy, double shift, unsigned* keys) {
    for (long q = blockIdx.x * (long)blockDim.x + threadIdx.x; q < np; q += (long)gridDim.x * blockDim.x) {
        double x = p.x[q], y = p.y[q];
        if (shift != 0.0) {
            x = wrap_periodic(x + shift * p.vx[q], Lx, 1.0 / Lx);
            y = wrap_periodic(y + shift * p.vy[q], Ly, 1.0 / Ly);
        }
        const int icx = wrap_index((int)floor((x + tg.key_origin_x) * inv_dx + tg.key_shift), tg.nx);
        const int icy = wrap_index((int)floor((y + tg.key_origin_y) * inv_dy + tg.key_shift), tg.ny);
        const int tx = icx / tg.tile_x, lx = icx - tx * tg.tile_x;
        const int ty = icy / tg.tile_y, ly = icy - ty * tg.tile_y;
        unsigned tile = (unsigned)(tx * tg.nty + ty);
        if (CLASSES) {
            const double ux = (x + tg.key_origin_x) * inv_dx - tg.class_off;
            const double uy = (y + tg.key_origin_y) * inv_dy - tg.class_off;
            const double n = fabs(floor(ux + tg.class_dt * p.vx[q] * inv_dx) - floor(ux)) +
                             fabs(floor(uy + tg.class_dt * p.vy[q] * inv_dy) - floor(uy));
            const double most = (double)(tg.classes - 1);
            tile = tile * (unsigned)tg.classes + (unsigned)(n < most ? n : most);
        }
        keys[q] = tile * (unsigned)(tg.tile_x * tg.tile_y) + (unsigned)(lx * tg.tile_y + ly);
    }
}

// Digit histogram of one block's keys.  Each warp reads its
// ITEMS * 32 keys ahead of counting and adds one shared atomic per
// distinct digit of each 32 (match/popc): the keys of a re-sort are nearly
// sorted already, so most rounds cost one atomic instead of 32 on one word.
template <int ITEMS>
__global__ void __launch_bounds__(kSortThreads)
radix_hist_kernel(const unsigned* __restrict__ keys, long n, int shift, int digits, int nblocks,
                  int* hist) {
    __shared__ int cnt[kMaxDigits];
    for (int d = threadIdx.x; d < digits; d += blockDim.x) cnt[d] = 0;
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    const unsigned mask = (unsigned)digits - 1u;
    const long wbase = (long)blockIdx.x * sort_tile(ITEMS) + (long)warp * (ITEMS * kWarp) + lane;
    unsigned key[ITEMS];
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
        const long e = wbase + r * kWarp;
        key[r] = e < n ? keys[e] : 0u;
    }
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
        const bool valid = wbase + r * kWarp < n;
        const int d = valid ? (int)((key[r] >> shift) & mask) : digits;
        const unsigned peers = __match_any_sync(0xffffffffu, d);
        if (valid && (peers & lt) == 0) atomicAdd(&cnt[d], __popc(peers));
    }
    __syncthreads();
    for (int d = threadIdx.x; d < digits; d += blockDim.x) hist[(long)d * nblocks + blockIdx.x] = cnt[d];
}

// Stable scatter of one digit pass, 256 keys per round: a key's in-block
// rank is the digit's count in the block's earlier rounds, plus its count in
// the round's earlier warps, plus its rank among its own warp's equal digits
// (match/popc); offs holds the scanned histograms (digit-major).  IDENT: the
// values are the source indices (the first pass of a sort, so the key kernel
// writes no values).
template <int ITEMS, bool IDENT>
__global__ void __launch_bounds__(kSortThreads)
radix_scatter_kernel(const unsigned* __restrict__ keys, const int* __restrict__ vals, long n, int shift,
                     int digits, int nblocks, const int* __restrict__ offs, unsigned* __restrict__ okeys,
                     int* __restrict__ ovals) {
    __shared__ int base_cnt[kMaxDigits];
    __shared__ int gofs[kMaxDigits];
    __shared__ int wcnt[kSortWarps][kMaxDigits];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int d = threadIdx.x; d < digits; d += blockDim.x) {
        base_cnt[d] = 0;
        gofs[d] = offs[(long)d * nblocks + blockIdx.x];
    }
    const unsigned mask = (unsigned)digits - 1u;
    const unsigned lt = (1u << lane) - 1u;
    const long base = (long)blockIdx.x * sort_tile(ITEMS);
    for (int r = 0; r < ITEMS; ++r) {
        for (int k = threadIdx.x; k < kSortWarps * kMaxDigits; k += blockDim.x) (&wcnt[0][0])[k] = 0;
        __syncthreads();
        const long e = base + r * kSortThreads + threadIdx.x;
        const bool valid = e < n;
        unsigned key = 0;
        int d = digits;  // sentinel for inactive lanes
        if (valid) {
            key = keys[e];
            d = (int)((key >> shift) & mask);
        }
        const unsigned peers = __match_any_sync(0xffffffffu, d);
        const int lrank = __popc(peers & lt);
        if (valid && lrank == 0) wcnt[warp][d] = __popc(peers);
        __syncthreads();
        if (valid) {
            int rank = base_cnt[d] + lrank;
            for (int w = 0; w < warp; ++w) rank += wcnt[w][d];
            const int dst = gofs[d] + rank;
            okeys[dst] = key;
            ovals[dst] = IDENT ? (int)e : vals[e];
        }
        __syncthreads();
        for (int dd = threadIdx.x; dd < digits; dd += blockDim.x) {
            int s = 0;
            for (int w = 0; w < kSortWarps; ++w) s += wcnt[w][dd];
            base_cnt[dd] += s;
        }
        __syncthreads();
    }
}

// ---- exclusive scan of int arrays ------------------------------------------
__device__ int block_exclusive_scan(int v, int* total) {
    __shared__ int ws[kScanThreads / kWarp];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int x = v;
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) ws[warp] = x;
    __syncthreads();
    if (warp == 0) {
        int s = lane < kScanThreads / kWarp ? ws[lane] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += y;
        }
        if (lane < kScanThreads / kWarp) ws[lane] = s;
    }
    __syncthreads();
    const int warp_excl = warp > 0 ? ws[warp - 1] : 0;
    *total = ws[kScanThreads / kWarp - 1];
    __syncthreads();
    return warp_excl + x - v;
}

__global__ void __launch_bounds__(kScanThreads)
scan_blocks_kernel(const int* in, int* out, long n, int* block_sums) {
    const long base = (long)blockIdx.x * kScanTile + (long)threadIdx.x * kScanItems;
    int v[kScanItems];
    int s = 0;
    for (int k = 0; k < kScanItems; ++k) {
        v[k] = base + k < n ? in[base + k] : 0;
        s += v[k];
    }
    int total;
    int ex = block_exclusive_scan(s, &total);
    for (int k = 0; k < kScanItems; ++k) {
        if (base + k < n) out[base + k] = ex;
        ex += v[k];
    }
    if (threadIdx.x == 0) block_sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(kScanThreads) scan_sums_kernel(int* sums, int nb, int* grand) {
    int carry = 0;
    for (int base = 0; base < nb; base += kScanThreads) {
        const int i = base + threadIdx.x;
        const int v = i < nb ? sums[i] : 0;
        int total;
        const int ex = block_exclusive_scan(v, &total);
        if (i < nb) sums[i] = ex + carry;
        carry += total;
    }
    if (threadIdx.x == 0 && grand) *grand = carry;
}

__global__ void scan_add_kernel(int* out, long n, const int* sums) {
    const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (i < n) out[i] += sums[i / kScanTile];
}

// Exclusive scan by one block, kScanOneItems values per thread at a time.
constexpr int kScanOneThreads = 1024, kScanOneItems = 8;
constexpr long kScanOne = 4096;
__device__ int scan_one_block(const int* in, int* out, int n) {
    __shared__ int ws[kScanOneThreads / kWarp];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int carry = 0;
    for (int base = 0; base < n; base += kScanOneThreads * kScanOneItems) {
        const int at = base + threadIdx.x * kScanOneItems;
        int v[kScanOneItems], s = 0;
#pragma unroll
        for (int k = 0; k < kScanOneItems; ++k) {
            v[k] = at + k < n ? in[at + k] : 0;
            s += v[k];
        }
        int x = s;
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) ws[warp] = x;
        __syncthreads();
        if (warp == 0) {
            int t = ws[lane];
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, t, o);
                if (lane >= o) t += y;
            }
            ws[lane] = t;
        }
        __syncthreads();
        int ex = carry + x - s + (warp > 0 ? ws[warp - 1] : 0);
#pragma unroll
        for (int k = 0; k < kScanOneItems; ++k) {
            if (at + k < n) out[at + k] = ex;
            ex += v[k];
        }
        carry += ws[kScanOneThreads / kWarp - 1];
        __syncthreads();
    }
    return carry;
}

__global__ void __launch_bounds__(kScanOneThreads) scan_one_kernel(const int* in, int* out, int n) {
    scan_one_block(in, out, n);
}

// Up to kScanOne values one block scans them in one launch (2.3 us at 512
// values, 12.8 us at 16,384); more take the three launches of blocks, block
// sums and their addition (5.4 us).
cudaError_t exclusive_scan(const int* in, int* out, long n, int* tmp, int* grand, cudaStream_t st) {
    if (n <= kScanOne && !grand) {
        scan_one_kernel<<<1, kScanOneThreads, 0, st>>>(in, out, (int)n);
        count_launches(1);
        return cudaGetLastError();
    }
    const int nb = (int)((n + kScanTile - 1) / kScanTile);
    scan_blocks_kernel<<<nb, kScanThreads, 0, st>>>(in, out, n, tmp);
    scan_sums_kernel<<<1, kScanThreads, 0, st>>>(tmp, nb, grand);
    scan_add_kernel<<<(int)((n + 255) / 256), 256, 0, st>>>(out, n, tmp);
    count_launches(3);
    return cudaGetLastError();
}

// ---- chunk table ----------------------------------------------------------
// Tile extents of the sorted keys without atomics: position q opens every
// tile in (tile(key[q-1]), tile(key[q])]; tile_start[ntiles] = n.
__global__ void tile_bounds_kernel(const unsigned* keys, long n, unsigned cells_per_tile, int ntiles,
                                   int* tstart) {
    for (long q = blockIdx.x * (long)blockDim.x + threadIdx.x; q <= n; q += (long)gridDim.x * blockDim.x) {
        const int t = q < n ? (int)(keys[q] / cells_per_tile) : ntiles;
        const int tp = q > 0 ? (int)(keys[q - 1] / cells_per_tile) : -1;
        for (int k = tp + 1; k <= t; ++k) tstart[k] = (int)q;
    }
}

__global__ void tile_counts_kernel(const int* tstart, int ntiles, int* cnt) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < ntiles) cnt[t] = tstart[t + 1] - tstart[t];
}

__global__ void tile_chunks_kernel(const int* cnt, int ntiles, int chunk, int* nch) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < ntiles) nch[t] = (cnt[t] + chunk - 1) / chunk;
}

__global__ void fill_chunks_kernel(const int* cnt, const int* tstart, const int* cstart, int ntiles,
                                   int chunk, Chunk* chunks) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= ntiles) return;
    const int c = cnt[t];
    const int s = tstart[t];
    int o = cstart[t];
    for (int k = 0; k < c; k += chunk) {
        Chunk ch;
        ch.start = s + k;
        ch.end = s + (k + chunk < c ? k + chunk : c);
        ch.tile = t;
        chunks[o++] = ch;
    }
}

// The chunk table of up to kTilesOne tiles in one launch of one block (counts,
// chunks per tile, their scan and the table): six launches of 9 us otherwise,
// against 3.3 us at 16 tiles and 37 us at 4096.
constexpr int kTilesOne = 512;
__global__ void __launch_bounds__(kScanOneThreads)
chunk_table_kernel(const int* tstart, int ntiles, int chunk, int* nch, int* nchunks, Chunk* chunks) {
    for (int t = threadIdx.x; t < ntiles; t += blockDim.x) nch[t] = (tstart[t + 1] - tstart[t] + chunk - 1) / chunk;
    __syncthreads();
    const int total = scan_one_block(nch, nch, ntiles);
    if (threadIdx.x == 0) *nchunks = total;
    // warps take the tiles, lanes a tile's chunks
    const int lane = threadIdx.x & 31;
    for (int t = threadIdx.x >> 5; t < ntiles; t += kScanOneThreads / kWarp) {
        const int s = tstart[t], c = tstart[t + 1] - s, o = nch[t];
        for (int k = lane; k * chunk < c; k += kWarp)
            chunks[o + k] = Chunk{s + k * chunk, s + min((k + 1) * chunk, c), t};
    }
}

// All payload arrays of the particle set gathered by one pass over the
// sorted index: dst_k[q] = src_k[idx[q]] for the double arrays present (and
// the original index); the index is read once instead of once per array.
struct GatherSet {
    const double* src[13];
    double* dst[13];
    int narr;
    const int* sid;
    int* did;
};

// One array after the other: each store waits for its load, so a thread
// has one load in flight.  Loading all of a particle's values ahead of the
// stores (13 loads in flight) measured slower on the nearly sorted re-sort
// gathers (7.15-7.21 against 6.85 ms per explicit step at 512x512 x 256).
__global__ void gather_set_kernel(GatherSet g, const int* __restrict__ idx, long n) {
    for (long q = blockIdx.x * (long)blockDim.x + threadIdx.x; q < n; q += (long)gridDim.x * blockDim.x) {
        const int i = idx[q];
#pragma unroll
        for (int k = 0; k < 13; ++k)
            if (k < g.narr) g.dst[k][q] = g.src[k][i];
        if (g.did) g.did[q] = g.sid[i];
    }
}

// ---- caller's order ---------------------------------------------------------
// The read-back gathers each array through the inverse order, so its writes
// are whole lines and its reads, within a few cells of each other, share
// sectors in L2.  Scattering eleven arrays of 16.8M particles by id took 7.3
// ms and the joins into triples 0.7 ms more; the inverse and the gathers
// straight into triples take 2.9 ms together.
__global__ void invert_kernel(const int* __restrict__ id, long n, int* __restrict__ inv) {
    for (long k = blockIdx.x * (long)blockDim.x + threadIdx.x; k < n; k += (long)gridDim.x * blockDim.x)
        inv[id[k]] = (int)k;
}

// Four particles per thread and round, their loads ahead of the stores.
constexpr int kBackItems = 4;

__global__ void gather_pair_kernel(const double* __restrict__ a, const double* __restrict__ b,
                                   const int* __restrict__ inv, long n, double* __restrict__ oa,
                                   double* __restrict__ ob) {
    const long step = (long)gridDim.x * blockDim.x;
    for (long o0 = blockIdx.x * (long)blockDim.x + threadIdx.x; o0 < n; o0 += kBackItems * step) {
        int k[kBackItems];
        double v[kBackItems][2];
#pragma unroll
        for (int i = 0; i < kBackItems; ++i) k[i] = o0 + i * step < n ? inv[o0 + i * step] : 0;
#pragma unroll
        for (int i = 0; i < kBackItems; ++i) {
            v[i][0] = a[k[i]];
            v[i][1] = b[k[i]];
        }
#pragma unroll
        for (int i = 0; i < kBackItems; ++i) {
            const long o = o0 + i * step;
            if (o >= n) break;
            oa[o] = v[i][0];
            ob[o] = v[i][1];
        }
    }
}

__global__ void gather_triple_kernel(const double* __restrict__ a, const double* __restrict__ b,
                                     const double* __restrict__ c, const int* __restrict__ inv, long n,
                                     double* __restrict__ out) {
    const long step = (long)gridDim.x * blockDim.x;
    for (long o0 = blockIdx.x * (long)blockDim.x + threadIdx.x; o0 < n; o0 += kBackItems * step) {
        int k[kBackItems];
        double v[kBackItems][3];
#pragma unroll
        for (int i = 0; i < kBackItems; ++i) k[i] = o0 + i * step < n ? inv[o0 + i * step] : 0;
#pragma unroll
        for (int i = 0; i < kBackItems; ++i) {
            v[i][0] = a[k[i]];
            v[i][1] = b[k[i]];
            v[i][2] = c[k[i]];
        }
#pragma unroll
        for (int i = 0; i < kBackItems; ++i) {
            const long o = o0 + i * step;
            if (o >= n) break;
            out[3 * o] = v[i][0];
            out[3 * o + 1] = v[i][1];
            out[3 * o + 2] = v[i][2];
        }
    }
}

int grid_for(long n) {
    long g = (n + 255) / 256;
    if (g > 148 * 16) g = 148 * 16;
    return g < 1 ? 1 : (int)g;
}

// Digit passes of the radix sort for the grid's cell keys: ceil(bits / 8)
// passes of equal width (at most 8 bits).
int radix_passes(const TileGeom& tg, int* dbits) {
    const long ncells = (long)tg.nx * tg.ny * tg.classes;
    int bits = 0;
    while ((1L << bits) < ncells) ++bits;
    if (bits == 0) bits = 1;
    const int passes = (bits + 7) / 8;
    *dbits = (bits + passes - 1) / passes;
    return passes;
}

}  // namespace

unsigned* sort_key_input(const TileGeom& tg, SortWork& w) {
    int dbits;
    return (radix_passes(tg, &dbits) & 1) ? w.keys_alt : w.keys;
}

cudaError_t sort_particles_by_tile(const TileGeom& tg, const ParticleSoA& p, long np, double Lx,
                                   double Ly, double shift, SortWork& w, cudaStream_t st) {
    if (np <= 0) {
        cudaMemsetAsync(w.nchunks, 0, sizeof(int), st);
        return cudaGetLastError();
    }
    const double inv_dx = (double)tg.nx / Lx, inv_dy = (double)tg.ny / Ly;
    auto make_keys = tg.classes > 1 ? make_keys_kernel<true> : make_keys_kernel<false>;
    make_keys<<<grid_for(np), 256, 0, st>>>(tg, p, np, Lx, Ly, inv_dx, inv_dy, shift, sort_key_input(tg, w));
    count_launches(1);
    return sort_keys_to_chunks(tg, np, w, st);
}

cudaError_t sort_keys_to_chunks(const TileGeom& tg, long np, SortWork& w, cudaStream_t st) {
    if (np <= 0) {
        cudaMemsetAsync(w.nchunks, 0, sizeof(int), st);
        return cudaGetLastError();
    }
    int dbits;
    const int passes = radix_passes(tg, &dbits);
    const int digits = 1 << dbits;
    const bool small = np < kSortSmall;
    const int tile = sort_tile(small ? kSortItemsSmall : kSortItems);
    const int nblocks = (int)((np + tile - 1) / tile);
    // The passes alternate between the two buffers and end in w.keys / w.vals;
    // the key kernel wrote the first pass's input (sort_key_input).
    const bool odd = passes & 1;
    unsigned* kin = odd ? w.keys_alt : w.keys;
    unsigned* kout = odd ? w.keys : w.keys_alt;
    int* vin = nullptr;
    int* vout = odd ? w.vals : w.vals_alt;
    for (int ps = 0; ps < passes; ++ps) {
        const int shift_bits = ps * dbits;
        auto hist = small ? radix_hist_kernel<kSortItemsSmall> : radix_hist_kernel<kSortItems>;
        auto scatter = small ? (ps == 0 ? radix_scatter_kernel<kSortItemsSmall, true>
                                        : radix_scatter_kernel<kSortItemsSmall, false>)
                             : (ps == 0 ? radix_scatter_kernel<kSortItems, true> : radix_scatter_kernel<kSortItems, false>);
        hist<<<nblocks, kSortThreads, 0, st>>>(kin, np, shift_bits, digits, nblocks, w.hist);
        exclusive_scan(w.hist, w.hist, (long)digits * nblocks, w.scan_tmp, nullptr, st);
        scatter<<<nblocks, kSortThreads, 0, st>>>(kin, vin, np, shift_bits, digits, nblocks, w.hist, kout, vout);
        count_launches(2);
        unsigned* tk = kin; kin = kout; kout = tk;
        vin = vout;
        vout = vout == w.vals ? w.vals_alt : w.vals;
    }
    // chunk table
    const int ntiles = tg.ntx * tg.nty;
    tile_bounds_kernel<<<grid_for(np + 1), 256, 0, st>>>(w.keys, np, (unsigned)(tg.tile_x * tg.tile_y * tg.classes),
                                                         ntiles, w.tile_start);
    if (ntiles <= kTilesOne) {
        chunk_table_kernel<<<1, kScanOneThreads, 0, st>>>(w.tile_start, ntiles, tg.chunk, w.tile_chunks, w.nchunks,
                                                          w.chunks);
        count_launches(2);
        return cudaGetLastError();
    }
    tile_counts_kernel<<<(ntiles + 255) / 256, 256, 0, st>>>(w.tile_start, ntiles, w.tile_count);
    count_launches(2);
    tile_chunks_kernel<<<(ntiles + 255) / 256, 256, 0, st>>>(w.tile_count, ntiles, tg.chunk, w.tile_chunks);
    exclusive_scan(w.tile_chunks, w.tile_chunks, ntiles, w.scan_tmp, w.nchunks, st);
    fill_chunks_kernel<<<(ntiles + 255) / 256, 256, 0, st>>>(w.tile_count, w.tile_start, w.tile_chunks,
                                                             ntiles, tg.chunk, w.chunks);
    count_launches(2);
    return cudaGetLastError();
}

cudaError_t permute_particles(const ParticleSoA& s, const ParticleSoA& d, long np, const SortWork& w,
                              cudaStream_t st) {
    const int g = grid_for(np);
    double* const src[13] = {s.x, s.y, s.Px, s.Py, s.Pz, s.vx, s.vy, s.vz, s.wx, s.wy, s.wz, s.q, s.m};
    double* const dst[13] = {d.x, d.y, d.Px, d.Py, d.Pz, d.vx, d.vy, d.vz, d.wx, d.wy, d.wz, d.q, d.m};
    GatherSet gs{};
    for (int k = 0; k < 13; ++k)
        if (src[k] && dst[k]) {
            gs.src[gs.narr] = src[k];
            gs.dst[gs.narr] = dst[k];
            ++gs.narr;
        }
    if (s.id && d.id) {
        gs.sid = s.id;
        gs.did = d.id;
    }
    if (np > 0) {
        gather_set_kernel<<<g, 256, 0, st>>>(gs, w.vals, np);
        count_launches(1);
    }
    return cudaGetLastError();
}

cudaError_t invert_order(const int* id, long np, int* inv, cudaStream_t st) {
    invert_kernel<<<grid_for(np), 256, 0, st>>>(id, np, inv);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t gather_pair(const double* a, const double* b, const int* inv, long np, double* oa, double* ob,
                        cudaStream_t st) {
    gather_pair_kernel<<<grid_for(np), 256, 0, st>>>(a, b, inv, np, oa, ob);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t gather_triple(const double* a, const double* b, const double* c, const int* inv, long np, double* out,
                          cudaStream_t st) {
    gather_triple_kernel<<<grid_for(np), 256, 0, st>>>(a, b, c, inv, np, out);
    count_launches(1);
    return cudaGetLastError();
}

}  // namespace upic
