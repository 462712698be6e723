// assign_owner.cu -- mass assignment for the FP32 / mixed estimator plan:
// owner-computes 16^3 tiles, 64-bit fixed-point accumulation in shared memory,
// FP32 grids written with plain stores.
//
// Same indices and weights as powerI4.f90:68-249 (see assign.cu); the weights
// are evaluated in FP32 from the FP64 cell offset.  Every contribution
// (w_x w_y) w_z weight is rounded once to an integer at scale 2^S (|q| < 2^30,
// 2^-28 resolution for unit weights: far below the FP32 grid's rounding) and
// summed into 64-bit integers with shared-memory atomics, so the grid is
// bit-identical for any particle order and schedule.
//
// 1. count: per particle, the first stencil cell of each grid and the tiles its
//    stencils touch (1 to 8).
// 2. scan, then scatter: the particle is prepared again and one 32-byte record
//    per (particle, touched tile) written in tile order.
// 3. one CTA per tile, one warp per record: the lanes take distinct stencil
//    cells of the record's particle (no two lanes of a warp add to the same
//    cell), keep those inside the tile and add them into the tile's shared
//    accumulator; the tile is then converted to FP32 and stored.  No global
//    atomics, no int64 grid, no memset of the grids.
//
// Tiles are 16^3 cells on grids that are a multiple of 16 and 10 to 16 cells an
// axis on others (TileGeom).
//
// The sort is bound by instruction issue and the FP64 pipe, not by its 25 MB of
// positions (2.1e6 particles in 256^3, PCS on two grids): count 37 us (FP64 pipe
// 67% busy with two operations a coordinate; issue 54%), scatter 75 us (issue 62%).
// With prepared particles written by the count and read back by the scatter, and
// the cells from FP64 arithmetic, the two took 154 us.  The tiles are bound by their
// shared 64-bit atomics: 510 us of 134 M adds at 256^3, 31.5 ms at 10^7 particles in
// 1024^3 (most of it clearing and storing 262,144 tiles of two grids).
#include "assign_owner.cuh"
#include "fixed.cuh"

#include <math.h>
#include <string.h>

#include <algorithm>
#include <type_traits>

namespace pbi4g {

namespace {

constexpr int kT = 16;                  // tile edge
constexpr int kTC = kT * kT * kT;       // 4096 cells
// padded shared layout of a tile's 64-bit sums: cell (x, y, z) at z * kPz + y * kPy + x.
// A stencil step's lanes are (i, j, l) in [0,4) x [0,4) x [0,2), l = lane / 16; a 64-bit
// access takes the bank pair 2 (i + 20 j + 16 l) = 2 i + 8 j (mod 32), so each half-warp
// (one wavefront of 8-byte accesses) touches 16 distinct pairs.
constexpr int kPy = 20, kPz = 336;
constexpr int kTCP = kT * kPz;          // 5376 cells per tile array
constexpr int kThreads = 512;

// One particle's stencil on one grid, relative to one tile (16 bytes): pack =
// base + kBias | x mask << 13 | y mask << 17 | z mask << 21, with base the
// padded offset (z kPz + y kPy + x) of the stencil's first cell from the tile
// origin and bit i of an axis mask set when the stencil's cell i on that axis
// lies inside the tile (pack 0: no cell inside).  The scatter writes them, so
// the tile kernel's lanes test one bit pattern and add one offset per cell.
struct alignas(16) PCell {
    int pack;
    float h[3];
};
struct alignas(16) PTile {              // a sorted record (particle, tile), both grids (32 bytes)
    PCell g[2];
};
// The buffers of an OwnerWork as the kernels see them.  Direct launches take
// them by value; the captured form (IND) reads them from the plan's device block
// (owner_ptrs_host), so its graphs follow the plan to another OwnerWork.  Read
// through the block the tile kernel measured 3% slower at 256^3, which is why
// the direct launches keep the kernel parameters.
struct OwnerPtrs {
    unsigned int *count, *start, *cursor;  // count: [ntiles + 2], the last two the tile counter
    PTile *sorted;
    float *wsorted;
};
static_assert(sizeof(OwnerPtrs) <= kOwnerPtrBytes, "owner pointer block");
constexpr int kBias = 2048;             // a stencil with a cell inside starts at [-3, 15] per axis: base + kBias in [977, 7403]
constexpr int kMX = 13, kMY = 17, kMZ = 21;

// first cell (0-based, in [0,N)) and the offset h that sets the weights
// t mod N for the cell indices: t is in [-2, 2N) for positions in [0, 1]
// (two compares), any other t takes the division
__device__ __forceinline__ int wrap_cell(long long t, int N) {
    if (t >= 0 && t < 2LL * N) return (int)(t >= N ? t - N : t);
    return (int)(t % N);
}

__device__ __forceinline__ void first_and_h(double p, int N, int nintp, bool shifted, bool cic_nint, int &f, float &h) {
    double v = __dadd_rn(__dmul_rn((double)N, p), 1.0);  // two roundings, as in assign.cu
    if (shifted) v = v - 0.5;
    long long iv;
    double hh;
    if (nintp == 4) { iv = (long long)v; f = wrap_cell(iv - 2, N); hh = v - (double)iv; }
    else if (nintp == 3) { iv = llround(v); f = wrap_cell(iv - 2, N); hh = v - (double)iv; }
    else if (nintp == 2) { iv = (long long)v; f = wrap_cell(iv, N); hh = cic_nint ? v - (double)llround(v) : v - (double)iv; }
    else { iv = llround(v); f = wrap_cell(iv - 1, N); hh = 0.0; }
    if (f < 0) f += N;
    if (f < 0 || f >= N) f = 0;
    h = (float)hh;
}

// Weight i of the per-axis stencil at offset h as a cubic in h,
// w_i(h) = c0 + h (c1 + h (c2 + h c3)): the reference's polynomials
// (powerI4.f90) expanded, e.g. PCS w0 = (1-h)^3/6, w1 = 4/6 + (h/2 - 1) h^2,
// w3 = h^3/6 and w2 = 1 - w0 - w1 - w3; TSC w0 = (1/2 - h)^2 / 2, w1 = 3/4 - h^2,
// w2 = 1 - w0 - w1; CIC 1 - h, h.  Each lane's stencil indices are fixed, so it
// picks its coefficients once and evaluates three FMAs per weight.
template <int NI>
__device__ __forceinline__ float4 axis_poly(int i) {
    if constexpr (NI == 4) {
        return i == 0 ? make_float4(1.f / 6.f, -0.5f, 0.5f, -1.f / 6.f)
             : i == 1 ? make_float4(2.f / 3.f, 0.f, -1.f, 0.5f)
             : i == 2 ? make_float4(1.f / 6.f, 0.5f, 0.5f, -0.5f)
                      : make_float4(0.f, 0.f, 0.f, 1.f / 6.f);
    } else if constexpr (NI == 3) {
        return i == 0 ? make_float4(0.125f, -0.5f, 0.5f, 0.f)
             : i == 1 ? make_float4(0.75f, 0.f, -1.f, 0.f)
                      : make_float4(0.125f, 0.5f, 0.5f, 0.f);
    } else if constexpr (NI == 2) {
        return i == 0 ? make_float4(1.f, -1.f, 0.f, 0.f) : make_float4(0.f, 1.f, 0.f, 0.f);
    } else {
        return make_float4(1.f, 0.f, 0.f, 0.f);
    }
}

__device__ __forceinline__ float horner(float4 c, float h) { return fmaf(h, fmaf(h, fmaf(h, c.w, c.z), c.y), c.x); }

// offset of a stencil's first cell from the tile origin, with the stencils that
// wrap past the upper grid edge into tile 0 shifted down by N: the lanes'
// cells are then d + c, inside the tile iff 0 <= d + c < 16 (N >= 32)
__device__ __forceinline__ int tile_offset(int f, int o, int N) {
    const int d = f - o;
    return d >= N - 4 ? d - N : d;
}

// The tiles of one axis.  Grids that are a multiple of 16 have N / 16 tiles of 16 cells;
// others (GEN) ceil(N / 16) tiles of N / nt cells, rounded down or up (10 to 16 for N >= 32,
// so a stencil of up to 5 cells touches at most two): tile t begins at floor(t N / nt), and
// cell f lies in tile floor(((f + 1) nt - 1) / N).  Both quotients are below 2^11 with
// numerators below 2^18 + 2^11, so the product with a float reciprocal of (numerator + 1/2)
// is off by less than 2^-12 of one and never crosses an integer.
struct TileGeom {
    int N, nt;
    float inv_n, inv_nt;
};
template <bool GEN>
__device__ __forceinline__ int tile_of_cell(int f, const TileGeom &g) {
    if constexpr (!GEN) return f / kT;
    return (int)(((float)((f + 1) * g.nt - 1) + 0.5f) * g.inv_n);
}
template <bool GEN>
__device__ __forceinline__ int tile_origin(int t, const TileGeom &g) {
    if constexpr (!GEN) return t * kT;
    return (int)(((float)(t * g.N) + 0.5f) * g.inv_nt);
}

// x 2^-64 rounded to float32 (x as unsigned or two's complement): the top 32 bits below the
// leading one, the rest as a sticky bit, so the 32-bit conversion rounds as the exact value
// does.  (64-bit conversions run on the FP64 pipe, at a 64th of the FP32 rate.)
__device__ __forceinline__ float frac_to_float(unsigned long long x) {
    if (x == 0) return 0.f;
    const int z = __clzll((long long)x);
    const unsigned long long m = x << z;
    const float f = __uint2float_rn((unsigned)(m >> 32) | ((unsigned)m != 0u ? 1u : 0u));
    return f * __int_as_float((127 - 32 - z) << 23);
}
__device__ __forceinline__ float sfrac_to_float(long long x) {
    const float f = frac_to_float((unsigned long long)(x < 0 ? -x : x));
    return x < 0 ? -f : f;
}

// first_and_h for both grids from one FP64 product and sum, v = N p + 1 (the reference's two
// roundings; FP64 is a slow pipe on this part, and these two operations are all it does
// here).  Everything else is read from v's bits: the integer part from its high word, and
// its fraction, aligned to 64 bits, in which the shifted grid's v - 1/2 (exact) flips the top
// bit and nint's offset is the two's complement reading.  Each offset takes the single FP32
// rounding first_and_h gives it, so cells and offsets are bit-identical to it.  v outside
// [1, N + 2) (positions outside [0, 1]) takes first_and_h.
__device__ __forceinline__ void first_cells(double p, int N, int nintp, bool interlaced, int &f0, float &h0, int &f1,
                                            float &h1) {
    const double v = __dadd_rn(__dmul_rn((double)N, p), 1.0);  // two roundings, as in assign.cu
    const unsigned hi = (unsigned)__double2hiint(v);
    // (of no use, and not used, where v is outside)
    const int k = (int)(hi >> 20) - 1023;                            // 2^k <= v < 2^(k+1)
    const int iv = (int)(((hi & 0xFFFFFu) | 0x100000u) >> ((20 - k) & 31));  // floor(v)
    if (hi - 0x3FF00000u >= 0x00C00000u || iv > N + 1) {
        first_and_h(p, N, nintp, false, !interlaced, f0, h0);
        if (interlaced) first_and_h(p, N, nintp, true, false, f1, h1);
        else { f1 = f0; h1 = 0.f; }
        return;
    }
    const unsigned long long fr = (unsigned long long)__double_as_longlong(v) << (12 + k);  // (v - floor(v)) 2^64
    const unsigned long long frs = fr ^ (1ull << 63);                // v - 1/2: the same
    const bool up = (long long)fr < 0;                               // v - floor(v) >= 1/2
    auto cell = [&](int t) { return t < 0 ? t + N : (t >= N ? t - N : t); };
    const int ivs = up ? iv : iv - 1;                                // floor(v - 1/2)
    if (nintp == 4) {
        f0 = cell(iv - 2); h0 = frac_to_float(fr);
        f1 = cell(ivs - 2); h1 = frac_to_float(frs);
    } else if (nintp == 3) {
        // nint(v) = floor(v) + up; nint(v - 1/2) = floor(v)
        f0 = cell(iv + (up ? 1 : 0) - 2); h0 = sfrac_to_float((long long)fr);
        f1 = cell(iv - 2); h1 = sfrac_to_float((long long)frs);
    } else if (nintp == 2) {
        f0 = cell(iv); h0 = interlaced ? frac_to_float(fr) : sfrac_to_float((long long)fr);
        f1 = cell(ivs); h1 = frac_to_float(frs);
    } else {
        f0 = cell(iv + (up ? 1 : 0) - 1); h0 = 0.f;
        f1 = cell(iv - 1); h1 = 0.f;
    }
    if (!interlaced) { f1 = f0; h1 = 0.f; }
}

// One particle: the cells and offsets of both grids, and the lowest first cell per axis
// (the shifted grid starts at the same cell or one below, circularly).
struct Prep {
    int f[2][3], lo[3];
    float h[2][3];
};
__device__ __forceinline__ void prep_particle(const double *__restrict__ pos, int64_t stride, int64_t i, int N,
                                              int nintp, int interlaced, Prep &r) {
#pragma unroll
    for (int c = 0; c < 3; c++) {
        first_cells(__ldg(pos + (size_t)c * stride + i), N, nintp, interlaced != 0, r.f[0][c], r.h[0][c], r.f[1][c],
                    r.h[1][c]);
        r.lo[c] = (interlaced && r.f[1][c] == (r.f[0][c] == 0 ? N - 1 : r.f[0][c] - 1)) ? r.f[1][c] : r.f[0][c];
    }
}

// The tiles that the stencils touch: t[c][0] holds the lowest cell, t[c][1] the last of the
// w cells from it; bit c of the result is set when they differ.
template <bool GEN>
__device__ __forceinline__ int span_tiles(const int lo[3], int w, const TileGeom &g, int t[3][2]) {
    int two = 0;
#pragma unroll
    for (int c = 0; c < 3; c++) {
        int hi = lo[c] + w - 1;
        hi -= hi >= g.N ? g.N : 0;
        t[c][0] = tile_of_cell<GEN>(lo[c], g);
        t[c][1] = tile_of_cell<GEN>(hi, g);
        two |= t[c][1] != t[c][0] ? 1 << c : 0;
    }
    return two;
}

// Grids with few tiles: every block counts its particles in shared memory and adds each
// tile's count once.  Particles in random order otherwise queue on a few addresses
// (100,000 of them on 64 tiles: 31 us for the count alone).
constexpr int kSmallTiles = 2048;
constexpr int kSortThreads = 256;

// particles [b, e) of this block (small grids: a contiguous share; else all, strided by the grid)
__device__ __forceinline__ void block_share(bool small, int64_t n, int64_t &b, int64_t &e, int64_t &step) {
    if (small) {
        b = n * blockIdx.x / gridDim.x;
        e = n * (blockIdx.x + 1) / gridDim.x;
        step = blockDim.x;
    } else {
        b = blockIdx.x * (int64_t)blockDim.x;
        e = n;
        step = (int64_t)gridDim.x * blockDim.x;
    }
}

template <bool IND, bool GEN, bool SMALL>
__global__ void __launch_bounds__(kSortThreads) owner_count_kernel(const TileGeom g, int nintp, int interlaced,
                                                                  int64_t npart, int64_t stride,
                                                                  const BoxPar *__restrict__ bp,
                                                                  const double *__restrict__ pos_arg,
                                                                  const OwnerPtrs ov,
                                                                  const OwnerPtrs *__restrict__ op) {
    // the captured form reads the box's position slot from its BoxPar
    const double *__restrict__ pos = (IND && bp) ? bp->pos : pos_arg;
    unsigned int *__restrict__ count = IND ? op->count : ov.count;
    __shared__ unsigned int hist[SMALL ? kSmallTiles : 1];
    const int w = nintp + (interlaced ? 1 : 0);  // cells spanned from the lowest first cell
    const int ntiles = g.nt * g.nt * g.nt;
    if (SMALL) {
        for (int t = threadIdx.x; t < ntiles; t += blockDim.x) hist[t] = 0u;
        __syncthreads();
    }
    int64_t b, e, step;
    block_share(SMALL, bp ? bp->npart : npart, b, e, step);
    for (int64_t i = b + threadIdx.x; i < e; i += step) {
        Prep r;
        prep_particle(pos, stride, i, g.N, nintp, interlaced, r);
        int t[3][2];
        const int two = span_tiles<GEN>(r.lo, w, g, t);
        const unsigned act = __activemask();
        const int lane = (int)(threadIdx.x & 31);
#pragma unroll
        for (int sl = 0; sl < 8; sl++) {
            const bool has = (sl & ~two) == 0;
            const int id = has ? (t[2][sl >> 2] * g.nt + t[1][(sl >> 1) & 1]) * g.nt + t[0][sl & 1] : -1;
            if (SMALL) {
                if (has) atomicAdd(hist + id, 1u);
                continue;
            }
            // one atomic per distinct tile of the warp (neighbouring particles of a
            // catalogue share their tiles and their tile crossings)
            if (!__any_sync(act, has)) continue;
            const unsigned same = __match_any_sync(act, id);
            if (has && lane == __ffs(same) - 1) atomicAdd(count + id, (unsigned)__popc(same));
        }
    }
    if (SMALL) {
        __syncthreads();
        for (int t = threadIdx.x; t < ntiles; t += blockDim.x)
            if (hist[t]) atomicAdd(count + t, hist[t]);
    }
}

template <bool IND>
__global__ void owner_scan_kernel(int ntiles, const OwnerPtrs ov, const OwnerPtrs *__restrict__ op) {
    const unsigned int *__restrict__ count = IND ? op->count : ov.count;
    unsigned int *__restrict__ start = IND ? op->start : ov.start, *__restrict__ cursor = IND ? op->cursor : ov.cursor;
    __shared__ unsigned int warp_tot[32];
    __shared__ unsigned int carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int base = 0; base < ntiles; base += blockDim.x) {
        const int i = base + threadIdx.x;
        const unsigned v = i < ntiles ? count[i] : 0u;
        unsigned x = v;
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) warp_tot[wid] = x;
        __syncthreads();
        if (wid == 0) {
            unsigned t = lane < (int)(blockDim.x >> 5) ? warp_tot[lane] : 0u;
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned y = __shfl_up_sync(0xffffffffu, t, o);
                if (lane >= o) t += y;
            }
            warp_tot[lane] = t;
        }
        __syncthreads();
        const unsigned excl = carry + x - v + (wid ? warp_tot[wid - 1] : 0u);
        if (i < ntiles) { start[i] = excl; cursor[i] = excl; }
        __syncthreads();
        if (threadIdx.x == blockDim.x - 1) carry = excl + v;
        __syncthreads();
    }
    if (threadIdx.x == 0) start[ntiles] = carry;
}

// Mask of the stencil's NI cells d .. d + NI - 1 that fall inside a tile of tw cells, d the
// offset of its first cell from the tile origin on one axis (tile_offset).
__device__ __forceinline__ unsigned axis_mask(int d, int NI, int tw) {
    const int lo = max(0, -d), hi = min(NI - 1, tw - 1 - d);
    return lo <= hi ? ((2u << hi) - 1u) & ~((1u << lo) - 1u) : 0u;
}

// Scatter: a record per (particle, touched tile).  The positions are read again: preparing
// them costs less than a 32-byte prepared record written by the count and read back.  Per
// axis, grid and tile the cell offset and mask are one addend of PCell::pack, so a record's
// pack is the sum of three.
template <bool IND, bool GEN, bool SMALL>
__global__ void __launch_bounds__(kSortThreads) owner_scatter_kernel(
    const TileGeom g, int nintp, int interlaced, int64_t npart, int64_t stride, const BoxPar *__restrict__ bp,
    const double *__restrict__ pos_arg, const OwnerPtrs ov, const OwnerPtrs *__restrict__ op,
    const double *__restrict__ weight) {
    const double *__restrict__ pos = (IND && bp) ? bp->pos : pos_arg;
    unsigned int *__restrict__ cursor = IND ? op->cursor : ov.cursor;
    PTile *__restrict__ sorted = IND ? op->sorted : ov.sorted;
    float *__restrict__ wsorted = weight ? (IND ? op->wsorted : ov.wsorted) : nullptr;
    __shared__ unsigned int place[SMALL ? kSmallTiles : 1];
    const int w = nintp + (interlaced ? 1 : 0);
    const int ntiles = g.nt * g.nt * g.nt;
    int64_t b, e, step;
    block_share(SMALL, bp ? bp->npart : npart, b, e, step);
    if (SMALL) {
        // the block's records per tile, then a range of places for them: one global atomic a tile
        for (int t = threadIdx.x; t < ntiles; t += blockDim.x) place[t] = 0u;
        __syncthreads();
        for (int64_t i = b + threadIdx.x; i < e; i += step) {
            Prep r;
            prep_particle(pos, stride, i, g.N, nintp, interlaced, r);
            int t[3][2];
            const int two = span_tiles<GEN>(r.lo, w, g, t);
#pragma unroll
            for (int sl = 0; sl < 8; sl++)
                if ((sl & ~two) == 0)
                    atomicAdd(place + (t[2][sl >> 2] * g.nt + t[1][(sl >> 1) & 1]) * g.nt + t[0][sl & 1], 1u);
        }
        __syncthreads();
        for (int t = threadIdx.x; t < ntiles; t += blockDim.x)
            if (place[t]) place[t] = atomicAdd(cursor + t, place[t]);
        __syncthreads();
    }
    for (int64_t i = b + threadIdx.x; i < e; i += step) {
        Prep r;
        prep_particle(pos, stride, i, g.N, nintp, interlaced, r);
        int t[3][2];
        const int two = span_tiles<GEN>(r.lo, w, g, t);
        const unsigned act = __activemask();
        const float wt = weight ? (float)weight[i] : 1.f;
        int x[3][2][2];  // [axis][tile of the axis][grid]
#pragma unroll
        for (int c = 0; c < 3; c++)
#pragma unroll
            for (int k = 0; k < 2; k++) {
                x[c][k][0] = x[c][k][1] = 0;
                if (k == 1 && !__any_sync(act, two >> c & 1)) continue;
                const int cell = c == 0 ? 1 : (c == 1 ? kPy : kPz), msk = c == 0 ? kMX : (c == 1 ? kMY : kMZ);
                const int o = tile_origin<GEN>(t[c][k], g);
                const int tw = GEN ? tile_origin<GEN>(t[c][k] + 1, g) - o : kT;
#pragma unroll
                for (int gr = 0; gr < 2; gr++) {
                    if (gr == 1 && !interlaced) continue;
                    const int d = tile_offset(r.f[gr][c], o, g.N);
                    // no cell in this tile: no offset either (a grid on the other side of the
                    // wrap is up to N cells away, beyond what pack's low bits hold)
                    const unsigned m = axis_mask(d, nintp, tw);
                    x[c][k][gr] = m ? d * cell + (int)(m << msk) : 0;
                }
            }
        // slot by slot (as owner_count_kernel counts them)
#pragma unroll
        for (int sl = 0; sl < 8; sl++) {
            const bool has = (sl & ~two) == 0;
            if (!__any_sync(act, has)) continue;
            const int id = has ? (t[2][sl >> 2] * g.nt + t[1][(sl >> 1) & 1]) * g.nt + t[0][sl & 1] : -1;
            unsigned d;
            if (SMALL) {
                d = has ? atomicAdd(place + id, 1u) : 0u;
            } else {
                // one atomic per distinct tile of the warp; the lanes that share it take
                // consecutive places
                const int lane = (int)(threadIdx.x & 31);
                const unsigned same = __match_any_sync(act, id);
                const int lead = __ffs(same) - 1;
                d = 0;
                if (has && lane == lead) d = atomicAdd(cursor + id, (unsigned)__popc(same));
                d = __shfl_sync(same, d, lead) + (unsigned)__popc(same & ((1u << lane) - 1u));
            }
            if (has) {
                PTile o;
#pragma unroll
                for (int gr = 0; gr < 2; gr++) {
                    const int pk = kBias + x[0][sl & 1][gr] + x[1][(sl >> 1) & 1][gr] + x[2][sl >> 2][gr];
                    const bool in = (pk >> kMX & 15) && (pk >> kMY & 15) && (pk >> kMZ & 15);
                    o.g[gr].pack = in ? pk : 0;
#pragma unroll
                    for (int c = 0; c < 3; c++) o.g[gr].h[c] = r.h[gr][c];
                }
                sorted[d] = o;
                if (wsorted) wsorted[d] = wt;
            }
        }
    }
}

// PCS records in columns: a half-warp takes one (particle, grid) pair of a
// record, lane (j, i) = (l >> 2 & 3, l & 3) of it the z column of cells
// (i, j, 0..3).  The x and y weights and their product are formed once per
// column, the z weights per cell, in the same order as the cell mapping,
// ((w_x w_y) w_z) weight, so every q is the same integer.  Two grids: the
// halves take grids 0 and 1 of one record; one grid: two records.  Each
// half-warp's 16 cells of a z step fall on 16 distinct bank pairs (2 i + 8 j).
// Read-only loads of the sorted records (their pointers come from the pointer
// block, so the compiler cannot infer that the kernel never writes them).
__device__ __forceinline__ PCell ld_cell(const PCell *p) {
    const int4 v = __ldg(reinterpret_cast<const int4 *>(p));
    PCell c;
    c.pack = v.x;
    c.h[0] = __int_as_float(v.y);
    c.h[1] = __int_as_float(v.z);
    c.h[2] = __int_as_float(v.w);
    return c;
}
__device__ __forceinline__ PTile ld_tile(const PTile *p) {
    PTile t;
    t.g[0] = ld_cell(&p->g[0]);
    t.g[1] = ld_cell(&p->g[1]);
    return t;
}

template <int G, bool W, bool GEN>
__device__ __forceinline__ void pcs_columns(unsigned b, unsigned e, int warp, int nwarps, int lane, float scale, int bits,
                                            const PTile *__restrict__ sorted, const float *__restrict__ wsorted,
                                            unsigned long long *acc64) {
    const int half = lane >> 4, ci = lane & 3, cj = (lane >> 2) & 3;
    const int g = G == 2 ? half : 0;
    const float4 px = axis_poly<4>(ci), py = axis_poly<4>(cj);
    float4 pz[4];
#pragma unroll
    for (int l = 0; l < 4; l++) {
        const float4 zc = axis_poly<4>(l);
        pz[l] = make_float4(zc.x * scale, zc.y * scale, zc.z * scale, zc.w * scale);
    }
    const int need = (1 << (kMX + ci)) | (1 << (kMY + cj));  // the column's x and y cells
    const int loff = g * kTCP + cj * kPy + ci - kBias;  // the column's cell offset less the bias
    constexpr int RPW = G == 2 ? 1 : 2;  // records per warp step
    const unsigned step = (unsigned)(RPW * nwarps), off = G == 2 ? 0u : (unsigned)half;
    // the next record of the half-warp is loaded while this one is added
    PCell cn = {};
    float wn = 1.f;
    if (b + (unsigned)(RPW * warp) + off < e) {
        cn = ld_cell(&sorted[b + (unsigned)(RPW * warp) + off].g[g]);
        if (W) wn = __ldg(&wsorted[b + (unsigned)(RPW * warp) + off]);
    }
    for (unsigned k = b + (unsigned)(RPW * warp) + off; k - off < e; k += step) {
        const PCell c = cn;
        const float wt = wn;
        if (k + step < e) {
            cn = ld_cell(&sorted[k + step].g[g]);
            if (W) wn = __ldg(&wsorted[k + step]);
        }
        // k >= e (the second record of a one-grid step past the end): pack 0
        const int pk = k < e ? c.pack : 0;
        const bool okxy = (pk & need) == need;
        const float wxy = horner(px, c.h[0]) * horner(py, c.h[1]);
        unsigned long long *col = acc64 + (loff + (pk & ((1 << kMX) - 1)));
#pragma unroll
        for (int l = 0; l < 4; l++) {
            float wv = wxy * horner(pz[l], c.h[2]);
            if (W) wv *= wt;
            const long long q = GEN ? to_fixed(wv, bits) : (long long)__float2int_rn(wv);
            if (okxy && (pk >> (kMZ + l) & 1)) atomicAdd(col + l * kPz, (unsigned long long)q);
        }
    }
}

// Tile kernel, specialised on the stencil width NI (1..4), the number of
// grids G (2 when interlaced) and the presence of particle weights W: below
// PCS a warp takes one record (particle, tile) and its lanes take the
// G * NI^3 (grid, cell) pairs, so the cell indices and the weight polynomials
// fold to constants and shifts; PCS takes the column mapping above.  The
// fixed-point scale 2^S rides in the z polynomial (a power of two: the
// products are the same bits as scaling at the end).
// GEN (grids that are not a multiple of 16): tiles of 10 to 16 cells an axis, and every
// contribution kept to 2^-bits as one 64-bit integer (scale is then 1), the resolution
// these grids had when their particles were added to a 64-bit grid in global memory.
template <int NI, int G, bool W, bool IND, bool GEN>
__global__ void __launch_bounds__(kThreads, 2) owner_tile_kernel(const TileGeom g, const OwnerPtrs ov,
                                                               const OwnerPtrs *__restrict__ op, float scale,
                                                               int bits, float inv_scale, float *__restrict__ out1,
                                                               float *__restrict__ out2) {
    constexpr int NC = NI * NI * NI;
    extern __shared__ unsigned long long acc64[];  // [G][kTCP]
    const int N = g.N, nt = g.nt, ntiles = nt * nt * nt;
    const unsigned int *__restrict__ start = IND ? op->start : ov.start;
    const PTile *__restrict__ sorted = IND ? op->sorted : ov.sorted;
    const float *__restrict__ wsorted = W ? (IND ? op->wsorted : ov.wsorted) : nullptr;
    unsigned int *next_tile = (IND ? op->count : ov.count) + ntiles + 1;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    __shared__ int s_tile;
    // tiles are handed out dynamically (their particle loads differ by orders of
    // magnitude in clustered boxes); the counter is zeroed before the launch
    for (;;) {
        if (threadIdx.x == 0) s_tile = (int)atomicAdd(next_tile, 1u);
        __syncthreads();
        const int tile = s_tile;
        if (tile >= ntiles) break;
        const int tx = tile % nt, ty = (tile / nt) % nt, tz = tile / (nt * nt);
        const int ox = tile_origin<GEN>(tx, g), oy = tile_origin<GEN>(ty, g), oz = tile_origin<GEN>(tz, g);
        for (int c = threadIdx.x; c < G * kTCP; c += blockDim.x) acc64[c] = 0ull;
        __syncthreads();
        const unsigned b = __ldg(&start[tile]), e = __ldg(&start[tile + 1]);
        if constexpr (NI == 4) {
            pcs_columns<G, W, GEN>(b, e, warp, nwarps, lane, scale, bits, sorted, wsorted, acc64);
        } else {
            // per-lane stencil cells of one grid: NIT steps of 32 cells; the (i, j, l)
            // of a lane, its cell offset, its bit pattern and its weight polynomials
            // are the same for every record
            constexpr int NIT = (NC + 31) / 32;
            int need[NIT], loff[NIT];
            float4 px[NIT], py[NIT], pz[NIT];
#pragma unroll
            for (int it = 0; it < NIT; it++) {
                const int c = it * 32 + lane;
                const int ci = c % NI, cj = (c / NI) % NI, cl = c < NC ? c / (NI * NI) : 0;
                // no cell for this lane at this step: a bit no pack has
                need[it] = c < NC ? (1 << (kMX + ci)) | (1 << (kMY + cj)) | (1 << (kMZ + cl)) : (1 << 30);
                loff[it] = cl * kPz + cj * kPy + ci - kBias;
                px[it] = axis_poly<NI>(ci);
                py[it] = axis_poly<NI>(cj);
                const float4 zc = axis_poly<NI>(cl);
                pz[it] = make_float4(zc.x * scale, zc.y * scale, zc.z * scale, zc.w * scale);
            }
            // the next record of the warp is loaded while this one is added
            PTile rn;
            float wn = 1.f;
            if (b + warp < e) {
                rn = ld_tile(&sorted[b + warp]);
                if (W) wn = __ldg(&wsorted[b + warp]);
            }
            for (unsigned k = b + warp; k < e; k += nwarps) {
                const PTile r = rn;
                const float wt = wn;
                if (k + nwarps < e) {
                    rn = ld_tile(&sorted[k + nwarps]);
                    if (W) wn = __ldg(&wsorted[k + nwarps]);
                }
                int cell[G][NIT];
                long long q[G][NIT];
                bool ok[G][NIT];
#pragma unroll
                for (int gr = 0; gr < G; gr++) {
                    const int pk = r.g[gr].pack;
                    const float hx = r.g[gr].h[0], hy = r.g[gr].h[1], hz = r.g[gr].h[2];
#pragma unroll
                    for (int it = 0; it < NIT; it++) {
                        ok[gr][it] = (pk & need[it]) == need[it];
                        // the reference's product order: ((w_x w_y) w_z) weight; wv * 2^S is exact in
                        // FP32 (a power-of-two scale) and |wv| 2^S < 2^30, so q is one 32-bit integer
                        float wv = horner(px[it], hx) * horner(py[it], hy) * horner(pz[it], hz);
                        if (W) wv *= wt;
                        q[gr][it] = GEN ? to_fixed(wv, bits) : (long long)__float2int_rn(wv);
                        cell[gr][it] = (pk & ((1 << kMX) - 1)) + loff[it];
                    }
                }
                // 64-bit fixed-point adds of the sign-extended q (exact mod 2^64)
#pragma unroll
                for (int gr = 0; gr < G; gr++)
#pragma unroll
                    for (int it = 0; it < NIT; it++)
                        if (ok[gr][it])
                            atomicAdd(acc64 + gr * kTCP + cell[gr][it], (unsigned long long)q[gr][it]);
            }
        }
        __syncthreads();
        for (int c = threadIdx.x; c < G * kTC; c += blockDim.x) {
            const int gr = c / kTC, cc = c % kTC;
            const int x = cc % kT, y = (cc / kT) % kT, z = cc / (kT * kT);
            if (GEN && (x >= tile_origin<GEN>(tx + 1, g) - ox || y >= tile_origin<GEN>(ty + 1, g) - oy ||
                        z >= tile_origin<GEN>(tz + 1, g) - oz))
                continue;
            const int pc = z * kPz + y * kPy + x;
            const long long v = (long long)acc64[gr * kTCP + pc];
            float *out = gr ? out2 : out1;
            out[((size_t)(oz + z) * N + (oy + y)) * N + (ox + x)] = (float)v * inv_scale;
        }
        __syncthreads();
    }
}

template <int NI, int G, bool W, bool IND, bool GEN>
static int launch_tile_w(const TileGeom &g, const OwnerPtrs &ov, const OwnerPtrs *op, int bits, float *out1,
                         float *out2, cudaStream_t st) {
    const size_t smem = sizeof(unsigned long long) * G * kTCP;
    auto kern = owner_tile_kernel<NI, G, W, IND, GEN>;
    PBI4G_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int ntiles = g.nt * g.nt * g.nt;
    int per_sm = 0;
    PBI4G_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kThreads, smem));
    const int grid = std::min(ntiles, 152 * std::max(1, per_sm));
    kern<<<grid, kThreads, smem, st>>>(g, ov, op, GEN ? 1.0f : ldexpf(1.0f, bits), bits, ldexpf(1.0f, -bits), out1,
                                       out2);
    PBI4G_LAUNCH_CHECK();
    return PBI4G_OK;
}

template <int NI, int G>
static int launch_tile(const TileGeom &g, const OwnerPtrs &ov, const OwnerPtrs *op, bool weighted, int bits,
                       float *out1, float *out2, cudaStream_t st) {
    // the captured form takes no weights and only grids that are multiples of 16
    if (op) return launch_tile_w<NI, G, false, true, false>(g, ov, op, bits, out1, out2, st);
    if (g.N % kT)
        return weighted ? launch_tile_w<NI, G, true, false, true>(g, ov, op, bits, out1, out2, st)
                        : launch_tile_w<NI, G, false, false, true>(g, ov, op, bits, out1, out2, st);
    return weighted ? launch_tile_w<NI, G, true, false, false>(g, ov, op, bits, out1, out2, st)
                    : launch_tile_w<NI, G, false, false, false>(g, ov, op, bits, out1, out2, st);
}

// zero the tile counts and the tile counter (through the pointer block)
__global__ void owner_zero_kernel(const OwnerPtrs *__restrict__ op, int n) {  // the captured form
    unsigned int *count = op->count;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) count[i] = 0u;
}

__global__ void owner_wmax_kernel(int64_t n, const double *__restrict__ w, unsigned long long *__restrict__ out) {
    double m = 0.0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        double a = fabs(w[i]);
        if (!(a <= 1e300)) a = 1e308;
        m = fmax(m, a);
    }
    for (int o = 16; o; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(out, (unsigned long long)__double_as_longlong(m));
}

}  // namespace

bool owner_supported(int N) { return N % kT == 0 && N >= 2 * kT && N <= 2048; }

bool owner_direct(int N, int64_t npart) {
    return owner_supported(N) || (N >= 2 * kT && N <= 2048 && npart <= ((int64_t)1 << 26));
}

bool OwnerWork::fits(int N, int64_t npart) const {
    const int nt = (N + kT - 1) / kT;
    const size_t ntiles = (size_t)nt * nt * nt;
    const size_t n = (size_t)(npart > 0 ? npart : 1);
    return count.p && count.bytes >= (ntiles + 2) * 4 && start.bytes >= (ntiles + 1) * 4 &&
           cursor.bytes >= (ntiles + 1) * 4 && sorted.bytes >= 8 * n * sizeof(PTile) && wsorted.bytes >= 8 * n * 4 && wmax.bytes >= 8;
}

int OwnerWork::ensure(int N, int64_t npart) {
    if (fixed) {
        if (fits(N, npart)) return PBI4G_OK;
        return set_error(PBI4G_ERR_RANGE, "shared assignment scratch too small for grid %d, %lld particles", N,
                         (long long)npart);
    }
    const int nt = (N + kT - 1) / kT;
    const size_t ntiles = (size_t)nt * nt * nt;
    const size_t n = (size_t)(npart > 0 ? npart : 1);
    PBI4G_CHECK(count.ensure((ntiles + 2) * 4));  // + the tile kernel's work counter
    PBI4G_CHECK(start.ensure((ntiles + 1) * 4));
    PBI4G_CHECK(cursor.ensure((ntiles + 1) * 4));
    // a record per (particle, touched tile): at most 8 per particle
    PBI4G_CHECK(sorted.ensure(8 * n * sizeof(PTile)));
    PBI4G_CHECK(wsorted.ensure(8 * n * 4));
    PBI4G_CHECK(wmax.ensure(8));
    return PBI4G_OK;
}

void OwnerWork::release() {
    for (DevBuf *b : {&count, &start, &cursor, &sorted, &wsorted, &wmax}) b->release();
}

size_t OwnerWork::footprint(int N, int64_t npart) {
    const size_t nt = (size_t)((N + kT - 1) / kT);
    return 3 * (nt * nt * nt + 2) * 4 + (size_t)npart * 8 * (sizeof(PTile) + 4) + 64;
}

void owner_ptrs_host(const OwnerWork &wk, unsigned char (&block)[kOwnerPtrBytes]) {
    OwnerPtrs o;
    o.count = wk.count.as<unsigned int>();
    o.start = wk.start.as<unsigned int>();
    o.cursor = wk.cursor.as<unsigned int>();
    o.sorted = static_cast<PTile *>(wk.sorted.p);
    o.wsorted = wk.wsorted.as<float>();
    memset(block, 0, kOwnerPtrBytes);
    memcpy(block, &o, sizeof(o));
}

int assign_owner(OwnerWork &wk, const void *d_ptrs, int N, int nintp, bool interlaced, int64_t npart,
                 const double *d_pos, const double *d_weight, float *out, cudaStream_t st, int64_t *launches,
                 int64_t stride, const BoxPar *bp, Prof *prof, int tile_stage, int sort_stage) {
    Prof none;
    Prof &pf = prof ? *prof : none;
    if (stride <= 0) stride = npart;
    if (bp ? !owner_supported(N) : !owner_direct(N, npart))
        return set_error(PBI4G_ERR_UNSUPPORTED, "owner assignment: grid %d, %lld particles", N, (long long)npart);
    if (nintp < 1 || nintp > 4 || npart < 1 || !d_pos || !d_ptrs)
        return set_error(PBI4G_ERR_INVALID, "assign: nintp=%d npart=%lld", nintp, (long long)npart);
    if (npart >= (int64_t)0x1fffffffLL) return set_error(PBI4G_ERR_RANGE, "assign: npart >= 2^29");
    // the caller has sized wk (and, for the captured form, written its pointers to d_ptrs)
    if (!wk.fits(N, npart)) return set_error(PBI4G_ERR_INVALID, "assign: work buffers not sized for this box");
    unsigned char blk[kOwnerPtrBytes];
    owner_ptrs_host(wk, blk);
    OwnerPtrs ov;
    memcpy(&ov, blk, sizeof(ov));
    const OwnerPtrs *op = bp ? static_cast<const OwnerPtrs *>(d_ptrs) : nullptr;  // the captured form
    double wmax = 1.0;
    if (d_weight && bp) return set_error(PBI4G_ERR_UNSUPPORTED, "captured assignment takes no weights");
    if (d_weight) {
        PBI4G_CUDA(cudaMemsetAsync(wk.wmax.p, 0, 8, st));
        owner_wmax_kernel<<<grid_blocks(npart, 256, 152 * 8), 256, 0, st>>>(npart, d_weight,
                                                                            wk.wmax.as<unsigned long long>());
        PBI4G_LAUNCH_CHECK();
        ++*launches;
        unsigned long long bitsw = 0;
        PBI4G_CUDA(cudaMemcpyAsync(&bitsw, wk.wmax.p, 8, cudaMemcpyDeviceToHost, st));
        PBI4G_CUDA(cudaStreamSynchronize(st));
        memcpy(&wmax, &bitsw, 8);
    }
    int bits;
    PBI4G_CHECK(fixed_point_bits(npart, wmax, &bits));
    // grids that are multiples of 16: each contribution is one 32-bit integer,
    // |w_x w_y w_z weight| 2^S <= 3.375 wmax 2^S < 2^30 (the 64-bit tile sums still hold the
    // total); 2^-28 resolution for unit weights
    const bool gen = N % kT != 0;
    if (!gen) {
        bits = std::min(bits, (int)floor(30.0 - log2(4.0 * (wmax > 0 ? wmax : 1.0))));
        if (bits < 8) return set_error(PBI4G_ERR_RANGE, "assign: particle weights up to %g", wmax);
    }
    const int nt = (N + kT - 1) / kT, ntiles = nt * nt * nt;
    const TileGeom geo = {N, nt, 1.0f / (float)N, 1.0f / (float)nt};
    // few tiles: a block counts its share in shared memory, over about two blocks an SM
    const bool small = ntiles <= kSmallTiles;
    const int blocks = small ? (int)std::min<int64_t>(152 * 2, (npart + kSortThreads - 1) / kSortThreads)
                             : grid_blocks(npart, kSortThreads);
    pf.begin(sort_stage, st);
    // counts and the tile counter
    auto sort = [&](auto ind, auto general, auto few) -> int {
        constexpr bool IND = decltype(ind)::value, GEN = decltype(general)::value, SM = decltype(few)::value;
        owner_count_kernel<IND, GEN, SM><<<blocks, kSortThreads, 0, st>>>(geo, nintp, interlaced, npart, stride, bp,
                                                                         d_pos, ov, op);
        PBI4G_LAUNCH_CHECK();
        owner_scan_kernel<IND><<<1, 1024, 0, st>>>(ntiles, ov, op);
        PBI4G_LAUNCH_CHECK();
        owner_scatter_kernel<IND, GEN, SM><<<blocks, kSortThreads, 0, st>>>(geo, nintp, interlaced, npart, stride, bp,
                                                                           d_pos, ov, op, d_weight);
        return PBI4G_OK;
    };
    const std::true_type yes;
    const std::false_type no;
    if (op) {
        owner_zero_kernel<<<grid_blocks(ntiles + 2, 256, 152 * 4), 256, 0, st>>>(op, ntiles + 2);
        PBI4G_LAUNCH_CHECK();
        ++*launches;
        PBI4G_CHECK(small ? sort(yes, no, yes) : sort(yes, no, no));
    } else {
        PBI4G_CUDA(cudaMemsetAsync(wk.count.p, 0, (size_t)(ntiles + 2) * 4, st));
        if (gen) PBI4G_CHECK(small ? sort(no, yes, yes) : sort(no, yes, no));
        else PBI4G_CHECK(small ? sort(no, no, yes) : sort(no, no, no));
    }
    PBI4G_LAUNCH_CHECK();
    const size_t FC = full_cells(N);
    const bool wt = d_weight != nullptr;
    float *o2 = interlaced ? out + FC : nullptr;
    pf.end(st);
    pf.begin(tile_stage, st);
    int rc = PBI4G_OK;
    switch (nintp * 2 + (interlaced ? 1 : 0)) {
        case 2: rc = launch_tile<1, 1>(geo, ov, op, wt, bits, out, o2, st); break;
        case 3: rc = launch_tile<1, 2>(geo, ov, op, wt, bits, out, o2, st); break;
        case 4: rc = launch_tile<2, 1>(geo, ov, op, wt, bits, out, o2, st); break;
        case 5: rc = launch_tile<2, 2>(geo, ov, op, wt, bits, out, o2, st); break;
        case 6: rc = launch_tile<3, 1>(geo, ov, op, wt, bits, out, o2, st); break;
        case 7: rc = launch_tile<3, 2>(geo, ov, op, wt, bits, out, o2, st); break;
        case 8: rc = launch_tile<4, 1>(geo, ov, op, wt, bits, out, o2, st); break;
        default: rc = launch_tile<4, 2>(geo, ov, op, wt, bits, out, o2, st); break;
    }
    pf.end(st);
    PBI4G_CHECK(rc);
    *launches += 4;
    return PBI4G_OK;
}

}  // namespace pbi4g
