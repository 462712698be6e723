// assign_owner.cu -- mass assignment for the FP32 / mixed estimator plan:
// owner-computes tiles, fixed-point sums in 32-bit shared words whose exactness is checked,
// FP32 grids written with plain stores.
//
// Same indices and weights as powerI4.f90:68-249 (see assign.cu); the weights
// are evaluated in FP32 from the FP64 cell offset.  Every contribution
// (w_x w_y) w_z weight is rounded once to an integer at scale 2^S (|q| < 2^30,
// 2^-28 resolution for unit weights: far below the FP32 grid's rounding) and
// summed exactly with shared-memory atomics, so the grid is bit-identical for any
// particle order and schedule.
//
// 1. count: per particle, the first stencil cell of each grid and the tiles its
//    stencils touch (1 to 8).
// 2. scan, then scatter: the particle is prepared again and one 32-byte record
//    per (particle, touched tile) written in tile order.
// 3. one CTA per tile: groups of lanes take the records' stencils column by column and add
//    them into the tile's shared accumulator, halo included; the tile's own cells are then
//    converted to FP32 and stored.  No global atomics, no int64 grid, no memset of the grids.
//
// Tiles are 16^3 cells on grids that are a multiple of 16 and 10 to 16 cells an
// axis on others (TileGeom).
//
// The sort is bound by instruction issue and the FP64 pipe, not by its 50 MB of
// positions, read twice (2.1e6 particles in 256^3, PCS on two grids): count 37 us (FP64 pipe
// 67% busy with two operations a coordinate; issue 54%), scatter 75 us (issue 62%).
// With prepared particles written by the count and read back by the scatter, and
// the cells from FP64 arithmetic, the two took 154 us.  (Of 10^8 particles in random order on the
// same 4096 tiles that form takes 12.5 ms, this one 14; the tiles gain 10 ms there.)
// The tiles are bound by instruction issue (67% at 2 10^6 random particles in 256^3, 266 us;
// 54 instructions a record of two grids) and next by the shared atomics; in dense boxes the
// other way round.  Of the 483 us before, with 64-bit atomics on the cells inside the tile, the
// tests of every cell, its branch and coefficients reloaded for want of registers took half.
// Boxes of few particles are bound by clearing and storing the tiles (512^3: 393 us, 158 of
// them the grids at HBM rate).
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
// Shared layout of a tile's sums: the tile and the NI cells below and above it that the
// stencils of its records reach, so that a stencil is added whole, without a test for each
// cell, and the halo is not stored (the neighbouring tiles have their own records of these
// particles).  Cell (x, y, z) of the tile is word (z + NI) pitch_z + (y + NI) kPy + x + 4;
// x has a halo of 4 for every order (rows of 96 bytes, 16-byte aligned in the tile).  Two
// arrays, arr_words apart.  At order 4 a step's lanes are the columns (i, j) in [0,4) x [0,4)
// of two items (grids 1 and 2 of one record, or two records): 16 columns take the banks
// i + 24 j = i + 8 j' (mod 32), which leaves every second group of four banks to the other
// array (arr_words = 4 mod 8).
constexpr int kPy = 24;
__host__ __device__ constexpr int halo_rows(int ni) { return kT + 2 * ni; }
__host__ __device__ constexpr int pitch_z(int ni) { return kPy * halo_rows(ni); }
__host__ __device__ constexpr int words(int ni) { return pitch_z(ni) * halo_rows(ni); }
__host__ __device__ constexpr int arr_words(int ni) { return words(ni) + 4; }
__host__ __device__ constexpr int origin_word(int ni) { return ni * (pitch_z(ni) + kPy) + 4; }
constexpr size_t tile_smem(int ni) { return sizeof(unsigned) * (size_t)(arr_words(ni) + words(ni)); }
constexpr int kThreads = 512;

// One particle's stencil on one grid, relative to one tile (16 bytes): the offsets that set
// its weights, and in pack the byte offset of its first cell in the tile's shared array
// (below 2^16) with kOut when a coordinate lies outside [0, 1].
struct alignas(16) PCell {
    float h[3];
    int pack;
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
    unsigned int *place;  // few tiles: the first place of each counting block's records, by block and tile
};
static_assert(sizeof(OwnerPtrs) <= kOwnerPtrBytes, "owner pointer block");
constexpr int kOut = 1 << 16;

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

// two float32 in one 64-bit register, and their packed multiply and multiply-add
using F2 = unsigned long long;
__device__ __forceinline__ F2 f2(float lo, float hi) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float f2_lo(F2 a) { return __uint_as_float((unsigned)a); }
__device__ __forceinline__ float f2_hi(F2 a) { return __uint_as_float((unsigned)(a >> 32)); }
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ F2 horner2(const F2 c[4], F2 h) { return fma2(h, fma2(h, fma2(h, c[3], c[2]), c[1]), c[0]); }

// x / 6 rounded to nearest (Markstein's correction of the product with the rounded reciprocal)
__device__ __forceinline__ float sixth(float x) {
    const float c = 1.f / 6.f, q = x * c;
    return fmaf(fmaf(-q, 6.f, x), c, q);
}
// All weights of an axis in the forms of axis_stencil (assign.cu), for GEN: the weights that
// these grids had in the 64-bit grid in global memory, whose rounding the other forms' is not.
template <int NI>
__device__ __forceinline__ void axis_direct(float h, float (&w)[NI]) {
    if constexpr (NI == 4) {
        const float h2 = h * h;
        w[0] = sixth((1.f - h) * (1.f - h) * (1.f - h));
        w[1] = 4.f / 6.f + (0.5f * h - 1.f) * h2;
        w[3] = sixth(h2 * h);
        w[2] = 1.f - w[0] - w[1] - w[3];
    } else if constexpr (NI == 3) {
        w[0] = 0.5f * (0.5f - h) * (0.5f - h);
        w[1] = 0.75f - h * h;
        w[2] = 1.f - w[0] - w[1];
    } else if constexpr (NI == 2) {
        w[0] = 1.f - h;
        w[1] = h;
    } else {
        w[0] = 1.f;
    }
}
template <int NI>
__device__ __forceinline__ float pick_weight(const float (&w)[NI], int i) {
    float r = w[0];
#pragma unroll
    for (int k = 1; k < NI; k++) r = i == k ? w[k] : r;
    return r;
}

// s times all weights of an axis, by pairs: axis_poly's cubics, every operation rounded as the
// single one is, so the three axes err alike (forms of their own for z, though closer to the
// weights, showed as a quadrupole).
template <int NI>
__device__ __forceinline__ void axis_products(float s, float h, float (&w)[NI]) {
    const F2 ss = f2(s, s), hh = f2(h, h);
    if constexpr (NI == 4) {
        const F2 w02 = fma2(hh, fma2(hh, fma2(hh, f2(-1.f / 6.f, -0.5f), f2(0.5f, 0.5f)), f2(-0.5f, 0.5f)),
                            f2(1.f / 6.f, 1.f / 6.f));
        const F2 w13 = fma2(hh, mul2(hh, fma2(hh, f2(0.5f, 1.f / 6.f), f2(-1.f, 0.f))), f2(2.f / 3.f, 0.f));
        const F2 p02 = mul2(ss, w02), p13 = mul2(ss, w13);
        w[0] = f2_lo(p02);
        w[1] = f2_lo(p13);
        w[2] = f2_hi(p02);
        w[3] = f2_hi(p13);
    } else if constexpr (NI == 3) {
        const F2 p02 = mul2(ss, fma2(hh, fma2(hh, f2(0.5f, 0.5f), f2(-0.5f, 0.5f)), f2(0.125f, 0.125f)));
        w[0] = f2_lo(p02);
        w[1] = s * fmaf(-h, h, 0.75f);
        w[2] = f2_hi(p02);
    } else if constexpr (NI == 2) {
        w[0] = s * (1.f - h);
        w[1] = s * h;
    } else {
        w[0] = s;
    }
}

// offset of a stencil's first cell from the origin of a tile that the stencils of its
// particle touch, in [-NI, 16]: the tile and the stencil may lie on either side of the wrap
// (N >= 32, so the three ranges are apart)
__device__ __forceinline__ int tile_offset(int f, int o, int N) {
    const int d = f - o;
    return d + (d < -4 ? N : 0) - (d >= N - 4 ? N : 0);
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
// [1, N + 2) (positions outside [0, 1]) takes first_and_h (and returns true: its offsets may
// make negative weights).
__device__ __forceinline__ bool first_cells(double p, int N, int nintp, bool interlaced, int &f0, float &h0, int &f1,
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
        return true;
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
    return false;
}

// One particle: the cells and offsets of both grids, and the lowest first cell per axis
// (the shifted grid starts at the same cell or one below, circularly).
struct Prep {
    int f[2][3], lo[3];
    float h[2][3];
    int out;  // kOut when a coordinate lies outside [0, 1]
};
__device__ __forceinline__ void prep_particle(const double *__restrict__ pos, int64_t stride, int64_t i, int N,
                                              int nintp, int interlaced, Prep &r) {
    r.out = 0;
#pragma unroll
    for (int c = 0; c < 3; c++) {
        if (first_cells(__ldg(pos + (size_t)c * stride + i), N, nintp, interlaced != 0, r.f[0][c], r.h[0][c], r.f[1][c],
                        r.h[1][c])) {
            r.out = kOut;
            // never further apart than the tiles' halos hold
            if (r.f[1][c] != r.f[0][c] && r.f[1][c] != (r.f[0][c] == 0 ? N - 1 : r.f[0][c] - 1)) r.f[1][c] = r.f[0][c];
        }
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
constexpr int kSortThreads = 256, kSmallThreads = 512, kSmallBlocks = 304;

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
__global__ void __launch_bounds__(SMALL ? kSmallThreads : kSortThreads) owner_count_kernel(const TileGeom g, int nintp, int interlaced,
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
        unsigned int *__restrict__ place = (IND ? op->place : ov.place) + (size_t)blockIdx.x * ntiles;
        for (int t = threadIdx.x; t < ntiles; t += blockDim.x)
            if (hist[t]) place[t] = atomicAdd(count + t, hist[t]);  // (from the tile's start)
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

// Scatter: a record per (particle, touched tile).  The positions are read again: preparing
// them costs less than a 32-byte prepared record written by the count and read back.
template <bool IND, bool GEN, bool SMALL>
__global__ void __launch_bounds__(SMALL ? kSmallThreads : kSortThreads) owner_scatter_kernel(
    const TileGeom g, int nintp, int interlaced, int64_t npart, int64_t stride, const BoxPar *__restrict__ bp,
    const double *__restrict__ pos_arg, const OwnerPtrs ov, const OwnerPtrs *__restrict__ op,
    const double *__restrict__ weight) {
    const double *__restrict__ pos = (IND && bp) ? bp->pos : pos_arg;
    unsigned int *__restrict__ cursor = IND ? op->cursor : ov.cursor;
    PTile *__restrict__ sorted = IND ? op->sorted : ov.sorted;
    float *__restrict__ wsorted = weight ? (IND ? op->wsorted : ov.wsorted) : nullptr;
    __shared__ unsigned int place[SMALL ? kSmallTiles : 1];
    const int w = nintp + (interlaced ? 1 : 0);
    const int pz = pitch_z(nintp), org = 4 * origin_word(nintp);
    const int ntiles = g.nt * g.nt * g.nt;
    int64_t b, e, step;
    block_share(SMALL, bp ? bp->npart : npart, b, e, step);
    if (SMALL) {
        // the block's places of each tile: the particles are those it counted
        const unsigned int *__restrict__ first = (IND ? op->place : ov.place) + (size_t)blockIdx.x * ntiles;
        const unsigned int *__restrict__ start = IND ? op->start : ov.start;
        for (int t = threadIdx.x; t < ntiles; t += blockDim.x) place[t] = start[t] + first[t];
        __syncthreads();
    }
    for (int64_t i = b + threadIdx.x; i < e; i += step) {
        Prep r;
        prep_particle(pos, stride, i, g.N, nintp, interlaced, r);
        int t[3][2];
        const int two = span_tiles<GEN>(r.lo, w, g, t);
        const unsigned act = __activemask();
        const float wt = weight ? (float)weight[i] : 1.f;
        int x[3][2][2];  // byte offset by [axis][tile of the axis][grid]
#pragma unroll
        for (int c = 0; c < 3; c++)
#pragma unroll
            for (int k = 0; k < 2; k++) {
                x[c][k][0] = x[c][k][1] = 0;
                if (k == 1 && !__any_sync(act, two >> c & 1)) continue;
                const int cell = 4 * (c == 0 ? 1 : (c == 1 ? kPy : pz));
                const int o = tile_origin<GEN>(t[c][k], g);
#pragma unroll
                for (int gr = 0; gr < 2; gr++) x[c][k][gr] = tile_offset(r.f[gr][c], o, g.N) * cell;
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
                    o.g[gr].pack = (org + x[0][sl & 1][gr] + x[1][(sl >> 1) & 1][gr] + x[2][sl >> 2][gr]) | r.out;
#pragma unroll
                    for (int c = 0; c < 3; c++) o.g[gr].h[c] = r.h[gr][c];
                }
                sorted[d] = o;
                if (wsorted) wsorted[d] = wt;
            }
        }
    }
}

// Read-only loads of the sorted records (their pointers come from the pointer
// block, so the compiler cannot infer that the kernel never writes them).
__device__ __forceinline__ PCell ld_cell(const PCell *p) {
    const int4 v = __ldg(reinterpret_cast<const int4 *>(p));
    PCell c;
    c.h[0] = __int_as_float(v.x);
    c.h[1] = __int_as_float(v.y);
    c.h[2] = __int_as_float(v.z);
    c.pack = v.w;
    return c;
}

__device__ __forceinline__ unsigned smem_addr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ float ldexp_bits(int e) { return __int_as_float((127 + e) << 23); }  // 2^e
__device__ __forceinline__ void red_shared(unsigned a, unsigned v) {
    asm volatile("red.shared.add.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned atom_shared(unsigned a, unsigned v) {
    unsigned old;
    asm volatile("atom.shared.add.u32 %0, [%1], %2;" : "=r"(old) : "r"(a), "r"(v) : "memory");
    return old;
}

// A tile's sums are kept in 32-bit shared words, whose atomics run at 2.7 times the rate of
// 64-bit ones (3880 against 1440 lanes a ns over the GPU):
//  * SHORT: the sum mod 2^32, biased by kSumBias, both grids at once.  No contribution is
//    below -64 (offsets inside the box make no negative weights but for FP32 rounding), so a
//    cell's sum is at least -kSumBias and a sum beyond 32 bits loses a positive multiple of
//    2^32.  The tile's contributions are also summed in 64-bit registers: the cells hold
//    their true sums exactly when the two totals agree.  If they do not, or a position lay
//    outside the box, or a particle weight is negative, a second pass (HIGH or FLAGGED) sums
//    the contributions' part above 16 bits: with less than 2^16 records, the sum of what is
//    left of them, 0 to 2^16 each, is what the first pass's sum holds beyond it.  HIGH takes
//    the part, at most 2^12, as the floor of the contribution before it is rounded, from the
//    low bits of a sum with 1.5 2^23; contributions that may be anything (FLAGGED) are
//    converted and shifted, at a quarter of that rate.
//    kFree: up to so many records no cell can reach 2^32 (a contribution is at most
//    2^28 times the largest weight of the stencil), and the totals are not compared.
//  * SPLIT: one grid at a time, the integer cut into the part above its low L bits and those
//    bits, neither below -1, whose biased sums fill the two arrays and are checked in the same
//    way.  GEN takes it for contributions of up to 43 bits, with L <= 22; others take it with
//    L = 14 for tiles of more records.
//  * WIDE: one grid at a time as 64-bit sums, low words and high words (array 0 and 1):
//    the low word's atomic returns the old word, from which follows the carry.
// The sums are the same integers in every form.  (2 10^6 particles in 256^3, order 4 on two
// grids: 64-bit words 481 us, SHORT 266; 10^8: 19.9 ms, SHORT 9.7.  Where every tile has a
// cell beyond 16 particles, SHORT and HIGH take 491 against 448 us, and 3.61 against 3.93 ms at
// 2 10^7; with FLAGGED for HIGH 522 us and 3.63 ms.)
constexpr unsigned kSumBias = 1u << 24;
constexpr unsigned kShortRecords = (1u << 16) - 1, kSplitRecords = 1u << 23;
constexpr int kAhead = 4;
__host__ __device__ constexpr unsigned free_records(int ni) { return ni == 4 ? 52u : (ni == 3 ? 36u : 15u); }
enum Form { SHORT, HIGH, FLAGGED, SPLIT, WIDE };

// Add the tile's items: an item is one record's stencil on one grid (NG = 2: both grids in
// turn, each into its own array; NG = 1: grid g0).  LPI lanes take an item, lane (j, i) of
// them the z column of cells (i, j, 0 .. NI - 1): the x and y weights and their product are
// formed once per column, the z weights per cell, in the reference's order
// ((w_x w_y) w_z) weight.  The scale (2^S; 2^(S - 16) in HIGH; with GEN 2^(S - L) in SPLIT and 1 in WIDE) rides in the
// product (a power of two: the same bits as scaling at the end), so a contribution rounds
// straight to an integer below 2^30.  GEN (grids that are not a multiple of 16): every
// contribution is kept to 2^-bits, the resolution these grids had when their particles were
// added to a 64-bit grid in global memory.  Returns the sum of the words added and collects
// the records' pack bits in flags (SHORT, SPLIT).
template <int NI, int NG, bool W, bool GEN, Form F, class Before>
__device__ __forceinline__ long long add_items(unsigned b, unsigned e, int g0, float scale, int bits, int lbits,
                                               const PTile *__restrict__ sorted, const float *__restrict__ wsorted,
                                               unsigned *acc, int &flags, Before &&before) {
    constexpr int LPI = NI * NI, IPW = 32 / LPI;
    constexpr int PZ = 4 * pitch_z(NI), HI = 4 * arr_words(NI);
    const unsigned sub = (threadIdx.x & 31) / LPI;
    const int col = (threadIdx.x & 31) % LPI, ci = col % NI, cj = col / NI;
    const float4 cx = axis_poly<NI>(ci), cy = axis_poly<NI>(cj);
    const F2 pxy[4] = {f2(cx.x, cy.x), f2(cx.y, cy.y), f2(cx.z, cy.z), f2(cx.w, cy.w)};
    const bool idle = sub >= IPW;  // (order 3: three items of 9 columns)
    const unsigned n = (e - b) * NG, step = (blockDim.x >> 5) * IPW;
    const unsigned t0 = (threadIdx.x >> 5) * IPW;
    const int g = NG == 2 ? (int)((t0 + sub) & 1u) : g0;  // (step is even)
    const unsigned base = smem_addr(acc) + 4u * (unsigned)((NG == 2 ? g * arr_words(NI) : 0) + cj * kPy + ci);
    long long tot = 0;
    auto fetch = [&](unsigned t, PCell &c, float &wt, bool all) {
        t += sub;
        if (all || (t < n && !idle)) {
            c = ld_cell(&sorted[b + t / NG].g[g]);
            if (W) wt = __ldg(&wsorted[b + t / NG]);
        }
    };
    auto add = [&](const PCell &c, float wt, bool is) {
        if (IPW > NG && (!is || idle)) return;
        float w[NI];
        if constexpr (GEN) {
            float wx[NI], wy[NI];
            axis_direct<NI>(c.h[0], wx);
            axis_direct<NI>(c.h[1], wy);
            axis_direct<NI>(c.h[2], w);
            const float wxy = pick_weight<NI>(wx, ci) * pick_weight<NI>(wy, cj) * scale;
#pragma unroll
            for (int l = 0; l < NI; l++) w[l] *= wxy;
        } else {
            const F2 wxwy = horner2(pxy, f2(c.h[0], c.h[1]));  // w_x and w_y, each rounded as by single FMAs
            axis_products<NI>(f2_lo(wxwy) * f2_hi(wxwy) * scale, c.h[2], w);
        }
        const unsigned cell = base + (unsigned)(c.pack & (kOut - 1));
        if (F == SHORT || F == SPLIT) {
            flags |= c.pack;
            if (W) flags |= wt >= 0.f ? 0 : kOut;
        }
        int part = 0;
#pragma unroll
        for (int l = 0; l < NI; l++) {
            const float wv = W ? w[l] * wt : w[l];
            if constexpr (F == SHORT) {
                const int q = __float2int_rn(wv);
                red_shared(cell + l * PZ, (unsigned)q);
                part += q;
            } else if constexpr (F == HIGH) {
                red_shared(cell + l * PZ, (unsigned)(__float_as_int(__fadd_rd(wv, 12582912.f)) - 0x4B400000));
            } else if constexpr (F == FLAGGED) {
                red_shared(cell + l * PZ, (unsigned)(__float2int_rn(wv) >> 16));
            } else if constexpr (F == SPLIT) {
                int hi, lo;
                if constexpr (GEN) {
                    // floor(wv) and the rest, rounded at 2^-L: below 2^22 both, so they are
                    // read from the low bits of sums with 1.5 2^23
                    const float m = 12582912.f, f = __fadd_rd(wv, m);
                    hi = __float_as_int(f) - 0x4B400000;
                    lo = __float_as_int(fmaf(wv - (f - m), ldexp_bits(lbits), m)) - 0x4B400000;
                } else {
                    const int q = __float2int_rn(wv);
                    hi = q >> lbits;
                    lo = q & ((1 << lbits) - 1);
                }
                red_shared(cell + l * PZ, (unsigned)lo);
                red_shared(cell + l * PZ + HI, (unsigned)hi);
                part += hi + lo;
            } else {
                const long long q = GEN ? to_fixed(wv, bits) : (long long)__float2int_rn(wv);
                const unsigned old = atom_shared(cell + l * PZ, (unsigned)q);
                const unsigned hi = (unsigned)(q >> 32) + (old + (unsigned)q < old ? 1u : 0u);
                if (hi) red_shared(cell + l * PZ + HI, hi);
            }
        }
        if (F == SHORT || F == SPLIT) tot += part;
    };
    // kAhead records of a warp in flight
    PCell c[kAhead] = {};
    float wt[kAhead];
#pragma unroll
    for (int k = 0; k < kAhead; k++) {
        wt[k] = 1.f;
        fetch(t0 + k * step, c[k], wt[k], false);
    }
    before();
    unsigned t = t0;
    const unsigned round = kAhead * step;
    for (; t < n && n - t >= 2 * round; t += round)  // (no test of the bounds until the end)
#pragma unroll
        for (int k = 0; k < kAhead; k++) {
            add(c[k], wt[k], true);
            fetch(t + (k + kAhead) * step, c[k], wt[k], true);
        }
    for (; t < n; t += round) {
#pragma unroll
        for (int k = 0; k < kAhead; k++) {
            if (t + k * step >= n) break;
            add(c[k], wt[k], t + k * step + sub < n);
            fetch(t + (k + kAhead) * step, c[k], wt[k], false);
        }
    }
    return tot;
}

// Tile kernel, specialised on the stencil width NI (1..4), the number of grids G (2 when
// interlaced) and the presence of particle weights W.  A single CIC grid takes its offset
// from the nearest cell, which makes weights of both signs: it has the WIDE form only.
// lbits: L of the SPLIT form (negative: the contributions have more bits than it holds), and
// split_free its kFree.
template <int NI, int G, bool W, bool IND, bool GEN>
__global__ void __launch_bounds__(kThreads, 2) owner_tile_kernel(const TileGeom g, const OwnerPtrs ov,
                                                               const OwnerPtrs *__restrict__ op, float scale,
                                                               int bits, int lbits, unsigned split_free,
                                                               float inv_scale, float *__restrict__ out1, float *__restrict__ out2) {
    constexpr bool kPositive = !(NI == 2 && G == 1), kShort = kPositive && !GEN;
    constexpr int PZ = pitch_z(NI), ARR = arr_words(NI), ORG = origin_word(NI);
    extern __shared__ __align__(16) unsigned acc[];  // arr_words + words
    const int N = g.N, nt = g.nt, ntiles = nt * nt * nt;
    const unsigned int *__restrict__ start = IND ? op->start : ov.start;
    const PTile *__restrict__ sorted = IND ? op->sorted : ov.sorted;
    const float *__restrict__ wsorted = W ? (IND ? op->wsorted : ov.wsorted) : nullptr;
    unsigned int *next_tile = (IND ? op->count : ov.count) + ntiles + 1;
    __shared__ int s_bad[2][3];  // [tile parity][grid, or 2 for both]
    __shared__ unsigned s_tile[2], s_b[2], s_e[2];
    __shared__ unsigned long long s_chk[2][3];
    uint4 *acc4 = reinterpret_cast<uint4 *>(acc);
    // tiles are handed out dynamically (their particle loads differ by orders of
    // magnitude in clustered boxes); the counter is zeroed before the launch.  A tile is drawn
    // and its records are fetched into L2 while the one before it is done
    auto draw = [&](int slot) {
        const unsigned t = atomicAdd(next_tile, 1u);
        s_tile[slot] = t;
        if (t < (unsigned)ntiles) {
            const unsigned tb = __ldg(&start[t]), te = __ldg(&start[t + 1]);
            s_b[slot] = tb;
            s_e[slot] = te;
            if (te > tb)
                asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(sorted + tb),
                             "r"((unsigned)sizeof(PTile) * min(te - tb, kShortRecords))
                             : "memory");
        }
    };
    if (threadIdx.x == 0) draw(0);
    for (int par = 0;; par ^= 1) {
        if (threadIdx.x == 0) {
#pragma unroll
            for (int k = 0; k < 3; k++) {  // (the other tile's may still be read)
                s_chk[par][k] = 0ull;
                s_bad[par][k] = 0;
            }
        }
        __syncthreads();
        const unsigned tile = s_tile[par];
        if (tile >= (unsigned)ntiles) break;
        const unsigned b = s_b[par], e = s_e[par];
        if (threadIdx.x == 0) draw(par ^ 1);
        const int tx = (int)tile % nt, ty = ((int)tile / nt) % nt, tz = (int)tile / (nt * nt);
        const int ox = tile_origin<GEN>(tx, g), oy = tile_origin<GEN>(ty, g), oz = tile_origin<GEN>(tz, g);
        auto clear = [&](int nwords, unsigned v) {
            for (int c = threadIdx.x; c < nwords / 4; c += blockDim.x) acc4[c] = make_uint4(v, v, v, v);
            __syncthreads();
        };
        // the totals' difference, into s_chk; every word in use was cleared to the bias
        auto compare = [&](long long chk, int nwords, int gr) {
            for (int c = threadIdx.x; c < nwords / 4; c += blockDim.x) {
                const uint4 v = acc4[c];
                chk -= (long long)v.x + v.y + v.z + v.w - 4ll * kSumBias;
            }
            for (int o = 16; o; o >>= 1) chk += __shfl_xor_sync(0xffffffffu, chk, o);
            if ((threadIdx.x & 31) == 0) atomicAdd(&s_chk[par][gr], (unsigned long long)chk);
        };
        if constexpr (kShort) {
            if (e - b <= kShortRecords) {
                constexpr int NW = (G == 2 ? ARR : 0) + words(NI);
                const bool few = e - b <= free_records(NI);
                // the tile's cells in fours, f(words of the accumulator, place in the grid)
                auto cells = [&](auto &&f) {
                    for (int c = threadIdx.x; c < G * kTC / 4; c += blockDim.x) {
                        const int gr = c / (kTC / 4), x = c % 4 * 4, y = c / 4 % kT, z = c / (4 * kT) % kT;
                        f(acc4[(gr * ARR + ORG + z * PZ + y * kPy + x) / 4],
                          reinterpret_cast<float4 *>((gr ? out2 : out1) + ((size_t)(oz + z) * N + (oy + y)) * N + ox + x));
                    }
                };
                int flags = 0;
                const long long tot =
                    add_items<NI, G, W, false, SHORT>(b, e, 0, scale, bits, 0, sorted, wsorted, acc, flags, [&] {
                        if (!few) {
                            clear(NW, kSumBias);
                            return;
                        }
                        cells([](uint4 &v, float4 *) { v = make_uint4(kSumBias, kSumBias, kSumBias, kSumBias); });
                        __syncthreads();
                    });
                __syncthreads();
                if (!few) compare(tot, NW, 2);
                if (flags & kOut) s_bad[par][2] = 1;
                cells([&](uint4 &v, float4 *o) {
                    auto value = [&](unsigned s) {  // the sum, which ranges from -2^24 to beyond 2^31
                        const unsigned d = s - kSumBias;
                        return (s >= kSumBias ? __uint2float_rn(d) : __int2float_rn((int)d)) * inv_scale;
                    };
                    *o = make_float4(value(v.x), value(v.y), value(v.z), value(v.w));
                });
                __syncthreads();
                if (s_chk[par][2] == 0ull && !s_bad[par][2]) continue;
                // the first pass's sums wait in the grid
                cells([&](uint4 &v, float4 *o) { *reinterpret_cast<uint4 *>(o) = v; });
                __syncthreads();
                auto none = [&] { clear(NW, 0u); };
                if (s_bad[par][2])
                    add_items<NI, G, W, false, FLAGGED>(b, e, 0, scale, bits, 0, sorted, wsorted, acc, flags, none);
                else
                    add_items<NI, G, W, false, HIGH>(b, e, 0, scale * ldexp_bits(-16), bits, 0, sorted, wsorted, acc,
                                                     flags, none);
                __syncthreads();
                cells([&](uint4 &v, float4 *o) {
                    const uint4 low = *reinterpret_cast<const uint4 *>(o);
                    auto value = [&](unsigned l, unsigned h) {
                        const long long s = (long long)(int)h * 65536;
                        return sfrac_to_float(s + (unsigned)(l - kSumBias - (unsigned)s)) * inv_scale *
                               18446744073709551616.0f;  // 2^64
                    };
                    *o = make_float4(value(low.x, v.x), value(low.y, v.y), value(low.z, v.z), value(low.w, v.w));
                });
                __syncthreads();
                continue;
            }
        }
        const int wx = GEN ? tile_origin<GEN>(tx + 1, g) - ox : kT, wy = GEN ? tile_origin<GEN>(ty + 1, g) - oy : kT,
                  wz = GEN ? tile_origin<GEN>(tz + 1, g) - oz : kT;
        const float s64 = inv_scale * 18446744073709551616.0f;  // 2^(64 - bits)
        auto store = [&](int gr, auto &&sum) {
            for (int c = threadIdx.x; c < kTC; c += blockDim.x) {
                const int x = c % kT, y = (c / kT) % kT, z = c / (kT * kT);
                if (GEN && (x >= wx || y >= wy || z >= wz)) continue;
                const int pc = ORG + z * PZ + y * kPy + x;
                (gr ? out2 : out1)[((size_t)(oz + z) * N + (oy + y)) * N + (ox + x)] =
                    sfrac_to_float(sum(acc[pc], acc[pc + ARR])) * s64;
            }
            __syncthreads();
        };
        constexpr int NW = ARR + words(NI);
        for (int gr = 0; gr < G; gr++) {
            if constexpr (kPositive) {
                if (lbits >= 0 && e - b <= kSplitRecords) {
                    int flags = 0;
                    const long long tot = add_items<NI, 1, W, GEN, SPLIT>(
                        b, e, gr, GEN ? scale * ldexp_bits(-lbits) : scale, bits, lbits, sorted, wsorted, acc, flags,
                        [&] { clear(NW, kSumBias); });
                    __syncthreads();
                    if (e - b > split_free) compare(tot, NW, gr);
                    if (flags & kOut) s_bad[par][gr] = 1;
                    __syncthreads();
                    if (s_chk[par][gr] == 0ull && !s_bad[par][gr]) {
                        store(gr, [&](unsigned lo, unsigned hi) {
                            return ((long long)hi - kSumBias) * (1ll << lbits) + ((long long)lo - kSumBias);
                        });
                        continue;
                    }
                }
            }
            int flags = 0;
            add_items<NI, 1, W, GEN, WIDE>(b, e, gr, GEN ? 1.f : scale, bits, 0, sorted, wsorted, acc, flags,
                                           [&] { clear(NW, 0u); });
            __syncthreads();
            store(gr, [](unsigned lo, unsigned hi) { return (long long)((unsigned long long)hi << 32 | lo); });
        }
    }
}

template <int NI, int G, bool W, bool IND, bool GEN>
static int launch_tile_w(const TileGeom &g, const OwnerPtrs &ov, const OwnerPtrs *op, int bits, int lbits, float *out1,
                         float *out2, cudaStream_t st) {
    auto kern = owner_tile_kernel<NI, G, W, IND, GEN>;
    const size_t smem = tile_smem(NI);
    PBI4G_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int ntiles = g.nt * g.nt * g.nt;
    int per_sm = 0;
    PBI4G_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kThreads, smem));
    const int grid = std::min(ntiles, 152 * std::max(1, per_sm));
    // parts are at most 2^lbits and 2^21 (GEN) or 2^(28 - lbits)
    const unsigned split_free = lbits < 0 ? 0u : 0xFE000000u >> std::max(lbits, GEN ? 21 : 28 - lbits);
    kern<<<grid, kThreads, smem, st>>>(g, ov, op, ldexpf(1.0f, bits), bits, lbits, split_free,
                                        ldexpf(1.0f, -bits), out1, out2);
    PBI4G_LAUNCH_CHECK();
    return PBI4G_OK;
}

template <int NI, int G>
static int launch_tile(const TileGeom &g, const OwnerPtrs &ov, const OwnerPtrs *op, bool weighted, int bits,
                       int lbits, float *out1, float *out2, cudaStream_t st) {
    // the captured form takes no weights and only grids that are multiples of 16
    if (op) return launch_tile_w<NI, G, false, true, false>(g, ov, op, bits, lbits, out1, out2, st);
    if (g.N % kT)
        return weighted ? launch_tile_w<NI, G, true, false, true>(g, ov, op, bits, lbits, out1, out2, st)
                        : launch_tile_w<NI, G, false, false, true>(g, ov, op, bits, lbits, out1, out2, st);
    return weighted ? launch_tile_w<NI, G, true, false, false>(g, ov, op, bits, lbits, out1, out2, st)
                    : launch_tile_w<NI, G, false, false, false>(g, ov, op, bits, lbits, out1, out2, st);
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

static int small_blocks(int64_t npart) {
    return (int)std::min<int64_t>(kSmallBlocks, (npart + kSmallThreads - 1) / kSmallThreads);
}
// `place` for grids up to N (a shared scratch of a large grid also serves plans of few tiles) and
// up to npart particles: at most 16 bytes a particle and 8 KB
static size_t place_bytes(int N, int64_t npart) {
    const size_t nt = (size_t)((N + kT - 1) / kT);
    return sizeof(unsigned) * (size_t)small_blocks(npart) * std::min<size_t>(nt * nt * nt, kSmallTiles);
}

bool OwnerWork::fits(int N, int64_t npart) const {
    const int nt = (N + kT - 1) / kT;
    const size_t ntiles = (size_t)nt * nt * nt;
    const size_t n = (size_t)(npart > 0 ? npart : 1);
    return count.p && count.bytes >= (ntiles + 2) * 4 && start.bytes >= (ntiles + 1) * 4 &&
           cursor.bytes >= (ntiles + 1) * 4 && sorted.bytes >= 8 * n * sizeof(PTile) && wsorted.bytes >= 8 * n * 4 && wmax.bytes >= 8 &&
           place.bytes >= place_bytes(N, (int64_t)n);
}

int64_t OwnerWork::particles() const { return (int64_t)(sorted.bytes / (8 * sizeof(PTile))); }

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
    PBI4G_CHECK(place.ensure(place_bytes(N, (int64_t)n)));
    return PBI4G_OK;
}

void OwnerWork::release() {
    for (DevBuf *b : {&count, &start, &cursor, &sorted, &wsorted, &wmax, &place}) b->release();
}

size_t OwnerWork::footprint(int N, int64_t npart) {
    const size_t nt = (size_t)((N + kT - 1) / kT);
    // (`place` takes less than 32 bytes a particle from 512 particles on: callers have their
    // budgets from this size, so it stays)
    return 3 * (nt * nt * nt + 2) * 4 + std::max((size_t)npart * 32, place_bytes(N, npart)) +
           (size_t)npart * 8 * (sizeof(PTile) + 4) + 64;
}

void owner_ptrs_host(const OwnerWork &wk, unsigned char (&block)[kOwnerPtrBytes]) {
    OwnerPtrs o;
    o.count = wk.count.as<unsigned int>();
    o.start = wk.start.as<unsigned int>();
    o.cursor = wk.cursor.as<unsigned int>();
    o.sorted = static_cast<PTile *>(wk.sorted.p);
    o.wsorted = wk.wsorted.as<float>();
    o.place = wk.place.as<unsigned int>();
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
    // other grids: 2^-bits in two parts, the upper one below 2^21 for the largest weight
    const int hbits = std::min(bits, (int)floor(21.0 - log2(wmax > 0 ? wmax : 1.0)));
    const int lbits = !gen ? std::min(bits, 14) : (bits - hbits <= 22 ? bits - hbits : -1);
    const int nt = (N + kT - 1) / kT, ntiles = nt * nt * nt;
    const TileGeom geo = {N, nt, 1.0f / (float)N, 1.0f / (float)nt};
    // few tiles: a block counts its share in shared memory, over about two blocks an SM
    const bool small = ntiles <= kSmallTiles;
    const int threads = small ? kSmallThreads : kSortThreads;
    const int blocks = small ? small_blocks(npart) : grid_blocks(npart, threads);
    pf.begin(sort_stage, st);
    // counts and the tile counter
    auto sort = [&](auto ind, auto general, auto few) -> int {
        constexpr bool IND = decltype(ind)::value, GEN = decltype(general)::value, SM = decltype(few)::value;
        owner_count_kernel<IND, GEN, SM><<<blocks, threads, 0, st>>>(geo, nintp, interlaced, npart, stride, bp,
                                                                         d_pos, ov, op);
        PBI4G_LAUNCH_CHECK();
        owner_scan_kernel<IND><<<1, 1024, 0, st>>>(ntiles, ov, op);
        PBI4G_LAUNCH_CHECK();
        owner_scatter_kernel<IND, GEN, SM><<<blocks, threads, 0, st>>>(geo, nintp, interlaced, npart, stride, bp,
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
        case 2: rc = launch_tile<1, 1>(geo, ov, op, wt, bits, lbits, out, o2, st); break;
        case 3: rc = launch_tile<1, 2>(geo, ov, op, wt, bits, lbits, out, o2, st); break;
        case 4: rc = launch_tile<2, 1>(geo, ov, op, wt, bits, lbits, out, o2, st); break;
        case 5: rc = launch_tile<2, 2>(geo, ov, op, wt, bits, lbits, out, o2, st); break;
        case 6: rc = launch_tile<3, 1>(geo, ov, op, wt, bits, lbits, out, o2, st); break;
        case 7: rc = launch_tile<3, 2>(geo, ov, op, wt, bits, lbits, out, o2, st); break;
        case 8: rc = launch_tile<4, 1>(geo, ov, op, wt, bits, lbits, out, o2, st); break;
        default: rc = launch_tile<4, 2>(geo, ov, op, wt, bits, lbits, out, o2, st); break;
    }
    pf.end(st);
    PBI4G_CHECK(rc);
    *launches += 4;
    return PBI4G_OK;
}

}  // namespace pbi4g
