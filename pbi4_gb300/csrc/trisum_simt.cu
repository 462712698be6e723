// trisum_simt.cu -- triangle sums on CUDA cores (the plain FP32 and FP64 forms, the
// cross spectra and the triangle counts).
//
// The "Last sum" loops of measure_bk / measure_bk_multipoles / measure_bk_cross
// (bispectrumI4.f90:160-195, 476-513, 728-757) and count_triangles (884-908):
// S[slot] = sum_x M_f(x) M_g(x) Q(x) over all grid points x, for the (f, g, q) that
// are triangles.
//
// A thread owns a register tile: F consecutive factor maps f, G consecutive maps g and
// Q consecutive shells q of each of the S q sets (every f with every g with every q).
// Triangles l <= i + j + const make the (i, l) entries of one j a staircase that moves
// by one with j; tiles start anywhere on it: at 21 shells 2 x 4 x 2 tiles hold 68%
// triangles, where a dense pairs x maps matrix holds 24%.  The pair products are formed
// in registers from the maps themselves, so only maps are staged.
//
// Points are the contiguous axis of the maps in memory and in shared memory: the FP32
// products and sums are packed pairs of neighbouring points (one packed instruction does
// two FMAs), with no transposition.  Each accumulator half adds at most 32 products (a
// stage) before it is folded into a Kahan-compensated FP32 sum in shared memory.  (Shell
// maps are smooth, so a thread's stages add up coherently and a plain FP32 sum of them rounds
// by more than the stages do: 4 times as much after 32.)  What a fold rounds off is where the
// accumulator begins the next stage, so the compensation takes no room.
//
// What bounds it: the FP32 FMA pipe, and the shared loads next.  A shared load moves 128
// bytes of registers a cycle however many lanes share an address, so a tile is chosen by
// both: a 4-point step of a 2 x 4 x 2 tile at S = 3 takes 224 FMA-pipe cycles a scheduler
// and 192 load cycles an SM for 4 warps (4 x 4 x 1: 208 and 272).  Packed and scalar FMAs
// reach 34 TFMA/s here with three distinct operands; this kernel runs 23.7 TFMA/s of
// them at the 256^3 box (21 shells, 3 sets), 83% in lanes that hold a tile and 68% of
// those triangles: 2.41 ms, against 25.3 ms for 4 x 8 tiles of a pairs x maps matrix with
// the products in shared memory and 44% of their entries triangles.  FP64 at 96^3 points
// and 10 shells: 1.4 ms against 6.7 ms, at the FP64 pipe's rate (0.5 TFMA/s).
#include <algorithm>
#include <iterator>
#include <vector>

#include "bispec.cuh"
#include "widen.cuh"

namespace pbi4g {

namespace {

// Tile shapes F x G x Q.  FP32: 48 packed accumulators at S = 3, 32 at S = 1.  FP64:
// 1 x 2 x 2, since its pipe is 64 times slower than the FP32 one and only the work
// counts: fewer padded entries, fuller warps.
template <class T, int S> struct Shape;
template <> struct Shape<float, 3> { static constexpr int F = 2, G = 4, Q = 2, threads = 384, ctas = 1; };
template <> struct Shape<float, 1> { static constexpr int F = 2, G = 4, Q = 4, threads = 256, ctas = 2; };
template <int S> struct Shape<double, S> { static constexpr int F = 1, G = 2, Q = 2, threads = 256, ctas = 1; };

// a pair of FP32 points, or one FP64 point
template <class T> struct Pack;
template <> struct Pack<float> {
    using P = float2;
    static __device__ __forceinline__ P zero() { return make_float2(0.f, 0.f); }
    static __device__ __forceinline__ P mul(P a, P b) { return __fmul2_rn(a, b); }
    static __device__ __forceinline__ P fma(P a, P b, P c) { return __ffma2_rn(a, b, c); }
    static __device__ __forceinline__ float sum(P a) { return a.x + a.y; }
};
template <> struct Pack<double> {
    using P = double;
    static __device__ __forceinline__ P zero() { return 0.0; }
    static __device__ __forceinline__ P mul(P a, P b) { return a * b; }
    static __device__ __forceinline__ P fma(P a, P b, P c) { return ::fma(a, b, c); }
};

template <class T> struct TriArgs {
    const T *maps;
    size_t mstride;
    unsigned rowlen, rs;   // points of a stored row and its stride (equal: contiguous points)
    long long K;
    int nrows, setrows, nslots;
    int ngroups, ksplit, reps, sub, nstages;  // reps: warp copies, each taking `sub` points of a stage
    int group_warps;
    const int4 *tiles;
    const int2 *groups;
    const int *slots;
    double *partial;       // [ksplit * reps][nslots]
};

__device__ __forceinline__ void cp_async16(void *dst, const void *src, bool valid) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    const int n = valid ? 16 : 0;  // 0: the destination is filled with zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}

// Shared memory: the second-level sums (FP32), then the ring of stages, map row m at
// m * pitch, pitch = points + one 16-byte unit, an odd number of units: 8 consecutive
// rows fall on 8 distinct bank groups.  A tile at the end of the maps reads a few rows
// past the last one (the next stage's, or padding): entries there are no slots.
template <class T, int S>
__global__ void __launch_bounds__(Shape<T, S>::threads, Shape<T, S>::ctas) trisum_kernel(const TriArgs<T> a) {
    constexpr int F = Shape<T, S>::F, G = Shape<T, S>::G, Q = Shape<T, S>::Q, E = F * G * Q * S;
    constexpr int W = 16 / (int)sizeof(T);  // points per 16-byte unit
    constexpr bool FP32 = sizeof(T) == 4;
    static_assert(E % 4 == 0, "second-level sums move as float4");
    using PK = Pack<T>;
    using P = typename PK::P;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nthr = blockDim.x;
    float4 *mid_s = reinterpret_cast<float4 *>(smem_raw) + tid;  // FP32: [E / 4][threads]
    T *sm = reinterpret_cast<T *>(smem_raw + (FP32 ? sizeof(float) * E * nthr : 0));
    const int gi = blockIdx.x % a.ngroups, split = blockIdx.x / a.ngroups;
    const int2 grp = a.groups[gi];
    const int rep = warp / a.group_warps, t = grp.x + (warp - rep * a.group_warps) * 32 + lane;
    const bool active = t < grp.y;
    const bool warp_active = t - lane < grp.y;
    const int4 tile = a.tiles[active ? t : grp.x];
    const int points = a.reps * a.sub;            // per stage
    const int pitch = points + W, stage_elems = a.nrows * pitch;
    const long long nch = (a.K + points - 1) / points;
    const long long cb = nch * split / a.ksplit, ce = nch * (split + 1) / a.ksplit;
    const int n = (int)(ce - cb);

    // copies: a thread takes one unit column of a stage and every row_step-th row (the
    // threads are a multiple of the units of a row)
    const int upr = points / W, row0 = tid / upr, col = (tid - row0 * upr) * W, row_step = nthr / upr;
    auto issue = [&](int i) {  // stage i into ring slot i % nstages
        if (i < n) {
            T *dst = sm + (size_t)(i % a.nstages) * stage_elems + col;
            const long long k = (cb + i) * points + col;
            const bool valid = k < a.K;
            size_t off = (size_t)(valid ? k : 0);
            if (a.rs != a.rowlen) {
                const unsigned q = (unsigned)off / a.rowlen;  // K < 2^32 for padded rows
                off = (size_t)q * a.rs + ((unsigned)off - q * a.rowlen);
            }
            const T *src = a.maps + off;
            for (int row = row0; row < a.nrows; row += row_step)
                cp_async16(dst + row * pitch, src + (size_t)row * a.mstride, valid);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    P acc[E];
    double mid_d[FP32 ? 1 : E];
#pragma unroll
    for (int e = 0; e < E; e++) {
        acc[e] = PK::zero();
        if (!FP32) mid_d[e] = 0.0;
    }
    if (FP32)
        for (int e = 0; e < E / 4; e++) mid_s[(size_t)e * nthr] = make_float4(0.f, 0.f, 0.f, 0.f);

    const int rowoff = rep * a.sub;
    const int fo = tile.x * pitch + rowoff, go = tile.y * pitch + rowoff, qo = tile.z * pitch + rowoff;
    const int so = a.setrows * pitch;
    for (int i = 0; i < a.nstages - 1; i++) issue(i);
    for (int i = 0; i < n; i++) {
        if (a.nstages == 4) asm volatile("cp.async.wait_group 2;" ::: "memory");
        else if (a.nstages == 3) asm volatile("cp.async.wait_group 1;" ::: "memory");
        else asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();  // stage i has landed for all; slot (i - 1) % nstages is free again
        issue(i + a.nstages - 1);
        if (!warp_active) continue;
        const T *st = sm + (size_t)(i % a.nstages) * stage_elems;
        const T *pf = st + fo, *pg = st + go, *pq = st + qo;
        // one step: a pack of every row.  Each value of the next step is loaded right after
        // its last use in this one (the loads past the last step stay in the row's padding
        // or the next copy's points), so no step waits for its own loads.
        auto ld = [](const T *p) { return *reinterpret_cast<const P *>(p); };
        constexpr int U = (int)(sizeof(P) / sizeof(T));  // points of a pack
        P f[F], g[G], q[S * Q];
        const T *pqs[S];
#pragma unroll
        for (int s = 0; s < S; s++) pqs[s] = pq + s * so;
#pragma unroll
        for (int x = 0; x < F; x++) f[x] = ld(pf + x * pitch);
#pragma unroll
        for (int p = 0; p < G; p++) g[p] = ld(pg + p * pitch);
#pragma unroll
        for (int b = 0; b < S * Q; b++) q[b] = ld(pqs[b / Q] + (b % Q) * pitch);
#pragma unroll 2
        for (int k = U; k <= a.sub; k += U) {
            P pr[F * G];
#pragma unroll
            for (int p = 0; p < G; p++)
#pragma unroll
                for (int x = 0; x < F; x++) pr[x * G + p] = PK::mul(f[x], g[p]);
#pragma unroll
            for (int x = 0; x < F; x++) f[x] = ld(pf + x * pitch + k);
#pragma unroll
            for (int p = 0; p < G; p++) g[p] = ld(pg + p * pitch + k);
#pragma unroll
            for (int b = 0; b < S * Q; b++) {
#pragma unroll
                for (int p = 0; p < F * G; p++) acc[b * F * G + p] = PK::fma(pr[p], q[b], acc[b * F * G + p]);
                q[b] = ld(pqs[b / Q] + (b % Q) * pitch + k);
            }
        }
        if constexpr (FP32) {
            // m + c, and c - ((m + c) - m) into the accumulator
            auto fold = [&](float2 m, P &a0, P &a1) {
                const float2 c = make_float2(PK::sum(a0), PK::sum(a1)), t = __fadd2_rn(m, c);
                const float2 d = __fadd2_rn(t, make_float2(-m.x, -m.y));
                const float2 r = __fadd2_rn(c, make_float2(-d.x, -d.y));
                a0 = make_float2(r.x, 0.f);
                a1 = make_float2(r.y, 0.f);
                return t;
            };
#pragma unroll
            for (int e = 0; e < E / 4; e++) {
                const float4 m = mid_s[(size_t)e * nthr];
                const float2 lo = fold(make_float2(m.x, m.y), acc[4 * e], acc[4 * e + 1]);
                const float2 hi = fold(make_float2(m.z, m.w), acc[4 * e + 2], acc[4 * e + 3]);
                mid_s[(size_t)e * nthr] = make_float4(lo.x, lo.y, hi.x, hi.y);
            }
        } else {
#pragma unroll
            for (int e = 0; e < E; e++) {
                mid_d[e] += acc[e];
                acc[e] = PK::zero();
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (!active) return;
    const int *sl = a.slots + (size_t)t * E;
    double *out = a.partial + (size_t)(split * a.reps + rep) * a.nslots;
#pragma unroll
    for (int e = 0; e < E; e++) {
        const int slot = sl[e];
        if (slot < 0) continue;
        double v;
        if constexpr (FP32) {
            // (one conversion on the FP64 pipe, not two: its rate shows in small boxes; sums of the
            // 64^3 box of 86 triangles 34 us, 39 with two)
            v = (double)reinterpret_cast<const float *>(mid_s + (size_t)(e / 4) * nthr)[e % 4] + widen(acc[e].x);
        } else {
            v = mid_d[e];
        }
        out[slot] = v;
    }
}

// S[slot] (+)= sum over the partial results: SL slots a block, the partials dealt to its
// 1024 / SL groups of lanes and the groups' sums added in order (a fixed order for every
// launch).  The loads' latency is all of it (one thread a slot took 52 us for 86 slots x 304
// partials), so few slots take more groups: 86 slots x 1376 partials take 16.6 us with 32 slots a
// block, 8.0 with 8.
template <int SL>
__global__ void __launch_bounds__(1024) reduce_partial_kernel(int nslots, int nparts,
                                                              const double *__restrict__ partial,
                                                              double *__restrict__ S, int accumulate) {
    constexpr int G = 1024 / SL;
    __shared__ double sh[G][SL + 1];
    const int i = threadIdx.x % SL, g = threadIdx.x / SL, s = blockIdx.x * SL + i;
    double v = 0;
    if (s < nslots) {
#pragma unroll 8
        for (int k = g; k < nparts; k += G) v += partial[(size_t)k * nslots + s];
    }
    sh[g][i] = v;
    __syncthreads();
    if (threadIdx.x < 32 * SL) {  // a warp a slot
        const int lane = threadIdx.x & 31, t = threadIdx.x >> 5;
        double r = 0;
#pragma unroll
        for (int k = 0; k < G / 32; k++) r += sh[k * 32 + lane][t];
        for (int o = 16; o; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
        const int d = blockIdx.x * SL + t;
        if (lane == 0 && d < nslots) S[d] = accumulate ? S[d] + r : r;
    }
}

}  // namespace

int reduce_partials(int nslots, int nparts, const double *partial, double *S, bool accumulate, cudaStream_t st) {
    if (nslots <= 8 * 152)  // one round of blocks over the SMs
        reduce_partial_kernel<8><<<(nslots + 7) / 8, 1024, 0, st>>>(nslots, nparts, partial, S, accumulate ? 1 : 0);
    else
        reduce_partial_kernel<32><<<(nslots + 31) / 32, 1024, 0, st>>>(nslots, nparts, partial, S, accumulate ? 1 : 0);
    PBI4G_LAUNCH_CHECK();
    return PBI4G_OK;
}

// ------------------------------------------------------------ TriPlan ---
// Output slot (m, s) = m * nsets + s.  Non-cross: S = sum M_i M_j Q_{s,l}, f = j, g = i,
// q = map qoff + s * nb + l-1.  Cross: S = sum Q_i M_j M_l, f = l, g = j, q = map cross * nb + i-1
// (cross = set index of the q field).
int TriPlan::build(const Shells &sh, int nsets_, int cross, bool dbl, int qoff) {
    nsets = nsets_;
    fp64 = dbl ? 1 : 0;
    if (nsets != 1 && nsets != 3) return set_error(PBI4G_ERR_INVALID, "triangle sums: %d q sets", nsets);
    auto shape = [&](auto s) {
        using Sh = decltype(s);
        tf = Sh::F;
        tg = Sh::G;
        tq = Sh::Q;
        max_warps = Sh::threads / 32;
    };
    if (dbl) shape(Shape<double, 1>{});
    else if (nsets == 3) shape(Shape<float, 3>{});
    else shape(Shape<float, 1>{});
    const int nb = sh.nb;
    setrows = nb;
    nslots = (int)(sh.itot * nsets);
    nrows = cross ? 2 * nb : qoff + nsets * nb;
    // entries (g nb + q shell, triangle) of each factor map f, sorted, and q nb + g, sorted
    std::vector<std::vector<std::pair<int, int>>> ent(nb);
    std::vector<std::vector<int>> by_q(nb);
    const int q0set = cross ? cross * nb : qoff;
    for (int64_t m = 0; m < sh.itot; m++) {
        const int l = sh.tri[3 * m] - 1, j = sh.tri[3 * m + 1] - 1, i = sh.tri[3 * m + 2] - 1;
        const int f = cross ? l : j, g = cross ? j : i, q = cross ? i : l;
        ent[f].push_back({g * nb + q, (int)m});
        by_q[f].push_back(q * nb + g);
    }
    for (int f = 0; f < nb; f++) {  // (one of the two is sorted already)
        if (!std::is_sorted(ent[f].begin(), ent[f].end())) std::sort(ent[f].begin(), ent[f].end());
        if (!std::is_sorted(by_q[f].begin(), by_q[f].end())) std::sort(by_q[f].begin(), by_q[f].end());
    }
    // Cover the entries of one run of factor maps with G x Q windows: strips of Q (or G)
    // columns from the first uncovered one, each cut into windows from its last row down;
    // by columns or by rows, whichever needs fewer windows.
    std::vector<char> row_used(nb, 0);
    auto cover = [&](const std::vector<int> &cells, int R, int C) {  // cells: column nb + row, sorted
        std::vector<std::pair<int, int>> w;  // (first column, first row)
        for (size_t k = 0; k < cells.size();) {
            const int c0 = cells[k] / nb, end = (c0 + C) * nb;
            int lo = nb, hi = -1;
            for (; k < cells.size() && cells[k] < end; k++) {
                const int r = cells[k] % nb;
                row_used[r] = 1;
                lo = std::min(lo, r);
                hi = std::max(hi, r);
            }
            for (int r = hi, first = nb; r >= lo; r--) {
                if (row_used[r] && r < first) w.push_back({c0, first = std::max(0, r - R + 1)});
                row_used[r] = 0;
            }
        }
        return w;
    };
    std::vector<int> qg, gq, tmp;
    auto tiles_from = [&](int first) {  // runs of tf factor maps, the first of `first` maps
        std::vector<int4> tl;
        for (int f0 = 0, f1 = first; f0 < nb; f0 = f1, f1 += tf) {
            qg.clear();
            gq.clear();
            for (int f = f0; f < std::min(f1, nb); f++) {
                tmp.clear();
                std::merge(qg.begin(), qg.end(), by_q[f].begin(), by_q[f].end(), std::back_inserter(tmp));
                qg.swap(tmp);
                const size_t mid = gq.size();
                for (auto &e : ent[f]) gq.push_back(e.first);
                std::inplace_merge(gq.begin(), gq.begin() + mid, gq.end());
            }
            const auto a = cover(qg, tg, tq), b = cover(gq, tq, tg);
            if (a.size() <= b.size())
                for (auto &w : a) tl.push_back(make_int4(f0, w.second, w.first, f1));
            else
                for (auto &w : b) tl.push_back(make_int4(f0, w.first, w.second, f1));
        }
        return tl;
    };
    std::vector<int4> tl = tiles_from(tf);
    for (int first = 1; first < tf; first++) {
        auto t2 = tiles_from(first);
        if (t2.size() < tl.size()) tl = t2;
    }
    // tiles of a warp share their q rows where they can
    std::sort(tl.begin(), tl.end(), [](const int4 &a, const int4 &b) {
        return a.z != b.z ? a.z < b.z : (a.y != b.y ? a.y < b.y : a.x < b.x);
    });
    ntiles = (int)tl.size();
    const int E = tf * tg * tq * nsets;
    std::vector<int> st((size_t)ntiles * E, -1);
    std::vector<std::vector<int>> run(nb);  // first factor map -> tiles
    for (int t = 0; t < ntiles; t++) run[tl[t].x].push_back(t);
    std::vector<int> at((size_t)nb * nb, -1);  // the triangles of one f, by (g, q shell)
    for (int f0 = 0; f0 < nb; f0++) {
        if (run[f0].empty()) continue;
        for (int f = f0; f < std::min(nb, tl[run[f0][0]].w); f++) {
            for (auto &e : ent[f]) at[e.first] = e.second;
            for (int t : run[f0])
                for (int p = 0; p < std::min(tg, nb - tl[t].y); p++)
                    for (int b = 0; b < std::min(tq, nb - tl[t].z); b++) {
                        int &m = at[(tl[t].y + p) * nb + tl[t].z + b];
                        if (m < 0) continue;
                        for (int s = 0; s < nsets; s++)
                            st[(size_t)t * E + ((s * tq + b) * tf + f - f0) * tg + p] = m * nsets + s;
                        m = -1;  // windows may overlap: each triangle belongs to one tile
                    }
        }
    }
    for (auto &t : tl) t.z += q0set;
    // groups of equal size, at most a CTA of tiles each
    const int warps = std::max(1, (ntiles + 31) / 32);
    ngroups = (warps + max_warps - 1) / max_warps;
    std::vector<int2> gl;
    group_warps = 0;
    for (int g = 0; g < ngroups; g++) {
        const int w0 = warps * g / ngroups, w1 = warps * (g + 1) / ngroups;
        gl.push_back(make_int2(std::min(ntiles, 32 * w0), std::min(ntiles, 32 * w1)));
        group_warps = std::max(group_warps, w1 - w0);
    }
    PBI4G_CHECK(tiles.ensure(sizeof(int4) * std::max<size_t>(1, tl.size())));
    PBI4G_CHECK(slots.ensure(sizeof(int) * std::max<size_t>(1, st.size())));
    PBI4G_CHECK(groups.ensure(sizeof(int2) * gl.size()));
    if (ntiles) {
        PBI4G_CUDA(cudaMemcpy(tiles.p, tl.data(), sizeof(int4) * tl.size(), cudaMemcpyHostToDevice));
        PBI4G_CUDA(cudaMemcpy(slots.p, st.data(), sizeof(int) * st.size(), cudaMemcpyHostToDevice));
    }
    PBI4G_CUDA(cudaMemcpy(groups.p, gl.data(), sizeof(int2) * gl.size(), cudaMemcpyHostToDevice));
    return PBI4G_OK;
}

template <class T, int S>
static int launch_trisum(TriPlan &tp, TriArgs<T> &a, DevBuf &partial, double *Sout, bool accumulate, cudaStream_t st,
                         int64_t *launches) {
    using Sh = Shape<T, S>;
    constexpr int E = Sh::F * Sh::G * Sh::Q * S, W = 16 / (int)sizeof(T);
    constexpr int kPad = std::max(Sh::F, std::max(Sh::G, Sh::Q));  // rows a tile may read past the last one
    auto kern = trisum_kernel<T, S>;
    a.nrows = tp.nrows;
    a.group_warps = tp.group_warps;
    // A stage holds `reps` x `sub` points of every row: the most points a thread takes of a
    // stage, then the most warps, then the most stages that fit; where the kernel is
    // compiled for two CTAs an SM, first in half of its shared memory.
    size_t smem = 0;
    bool fits = false;
    const int pref = std::max(1, Sh::threads / 32 / tp.group_warps);
    for (int half = Sh::ctas - 1; half >= 0 && !fits; half--)
        for (int sub = 64; sub >= 16 && !fits; sub /= 2)
            for (int reps = pref; reps >= 1 && !fits; reps--)
                for (int ns = 4; ns >= 2 && !fits; ns--) {
                    const size_t pitch = (size_t)reps * sub + W;
                    smem = sizeof(T) * pitch * ((size_t)ns * tp.nrows + kPad) +
                           (sizeof(T) == 4 ? sizeof(float) * E * 32 * (size_t)tp.group_warps * reps : 0);
                    if (smem > (size_t)(half ? 113 : 226) * 1024) continue;
                    // a thread copies one unit column of a stage
                    if ((32 * tp.group_warps) % (sub / W)) continue;
                    fits = true;
                    a.sub = sub;
                    a.reps = reps;
                    a.nstages = ns;
                }
    if (!fits) return set_error(PBI4G_ERR_UNSUPPORTED, "triangle sums: %d maps exceed shared memory", tp.nrows);
    const int threads = 32 * tp.group_warps * a.reps;
    PBI4G_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int per_sm = 0;
    PBI4G_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem));
    const int ctas = 152 * std::max(1, per_sm);
    const long long nch = (a.K + (long long)a.reps * a.sub - 1) / ((long long)a.reps * a.sub);
    // the K split whose waves x (stages a CTA + a fixed cost of about two) is smallest
    a.ngroups = tp.ngroups;
    long long best = -1;
    a.ksplit = 1;
    for (int k = 1; k <= 4 * ctas / tp.ngroups + 1 && k <= nch; k++) {
        const long long waves = ((long long)tp.ngroups * k + ctas - 1) / ctas;
        const long long cost = waves * ((nch + k - 1) / k + 2);
        if (best < 0 || cost < best) {
            best = cost;
            a.ksplit = k;
        }
    }
    a.setrows = tp.setrows;
    a.nslots = tp.nslots;
    a.tiles = tp.tiles.as<int4>();
    a.groups = tp.groups.as<int2>();
    a.slots = tp.slots.as<int>();
    const int grid = tp.ngroups * a.ksplit, nparts = a.ksplit * a.reps;
    PBI4G_CHECK(partial.ensure(sizeof(double) * (size_t)nparts * tp.nslots));
    a.partial = partial.as<double>();
    kern<<<grid, threads, smem, st>>>(a);
    PBI4G_LAUNCH_CHECK();
    PBI4G_CHECK(reduce_partials(tp.nslots, nparts, partial.as<double>(), Sout, accumulate, st));
    *launches += 2;
    return PBI4G_OK;
}

template <class T>
int triangle_sums(const Shells &sh, TriPlan &tp, const T *maps, size_t mstride, int rowlen, int rs, long long K,
                  DevBuf &partial, double *S, bool accumulate, cudaStream_t st, int64_t *launches) {
    constexpr int W = 16 / (int)sizeof(T);
    if (tp.fp64 != (sizeof(T) == 8))
        return set_error(PBI4G_ERR_INVALID, "triangle sums: plan of another type");
    if (tp.nslots == 0) return PBI4G_OK;
    // 16-byte loads: whole units, none across a row end
    if (K < 1 || K % W || mstride % W || reinterpret_cast<uintptr_t>(maps) % 16 ||
        (rs != rowlen && (rowlen % W || rs % W || K >= (1LL << 32))))
        return set_error(PBI4G_ERR_UNSUPPORTED, "triangle sums: %lld points in rows of %d (stride %d)", K, rowlen, rs);
    TriArgs<T> a;
    a.maps = maps;
    a.mstride = mstride;
    a.rowlen = (unsigned)rowlen;
    a.rs = (unsigned)rs;
    a.K = K;
    if (tp.nsets == 3) return launch_trisum<T, 3>(tp, a, partial, S, accumulate, st, launches);
    return launch_trisum<T, 1>(tp, a, partial, S, accumulate, st, launches);
}

template int triangle_sums<float>(const Shells &, TriPlan &, const float *, size_t, int, int, long long, DevBuf &,
                                  double *, bool, cudaStream_t, int64_t *);
template int triangle_sums<double>(const Shells &, TriPlan &, const double *, size_t, int, int, long long, DevBuf &,
                                   double *, bool, cudaStream_t, int64_t *);

}  // namespace pbi4g
