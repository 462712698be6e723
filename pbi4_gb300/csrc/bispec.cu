// bispec.cu -- shell tables, shell-filtered k-maps, exact triangle counts and
// the bispectrum output rows.
//
// Reference: bispectrumI4.f90 measure_bk (1-198), measure_bk_multipoles
// (200-516), measure_bk_cross (518-761), count_triangles (763-915).
//
// k-maps: the reference expands the kx >= 0 half spectrum to a full Hermitian
// grid, zeroes the imaginary part at the 8 self-conjugate points, and keeps the
// real part of a complex FFT of each shell-masked copy (:116-157).  The real
// part of a complex FFT equals the FFT of the input's Hermitian part, so here
// the masked half spectrum is Hermitian-symmetrised on the kx = 0 and kx = N/2
// planes and transformed with one batched C2R (cuFFT).  The reference's
// FORWARD transform and its x<->z transposed layout map x -> -x and permute
// axes; every output is a sum over all x, which neither changes.
#include "bispec.cuh"

#include <float.h>
#include <math.h>
#include <algorithm>
#include <map>
#include <mutex>
#include <tuple>
#include <vector>

namespace pbi4g {

// ------------------------------------------------------------- Shells ---
// Smallest multiple of 4 above 3 kmax that the map transform handles fast
// (5-smooth, or 7-smooth when that is more than 5% smaller), else N.
int map_grid_for_kmax(int N, int kmax) {
    auto smooth = [](int n, int fmax) {
        for (int f : {2, 3, 5, 7})
            if (f <= fmax)
                while (n % f == 0) n /= f;
        return n == 1;
    };
    int n5 = 0, n7 = 0;
    for (int n = 4; n < N && (!n5 || !n7); n += 4) {
        if (n <= 3 * kmax) continue;
        if (!n7 && smooth(n, 7)) n7 = n;
        if (!n5 && smooth(n, 5)) n5 = n;
    }
    if (n5) return (n7 && n7 < 0.95 * n5) ? n7 : n5;
    return n7 ? n7 : N;
}

int shell_map_grid(int N, float kbin, float kcenter, int nb) {
    const double kck = (double)(kcenter / kbin);
    const int h = N / 2, k2max = 3 * h * h;
    int kmax = 0;
    for (int k2 = 0; k2 <= k2max; k2++) {
        const long long b = llround(sqrt((double)k2) / (double)kbin - kck - (double)FLT_MIN) + 1;
        if (b >= 1 && b <= nb) kmax = std::max(kmax, (int)floor(sqrt((double)k2)));
    }
    return map_grid_for_kmax(N, kmax);
}

int Shells::build(int N_, float kbin_, float kcenter_, int nb_, int iopen_, int cross_, cudaStream_t st) {
    if (N == N_ && kbin == kbin_ && kcenter == kcenter_ && nb == nb_ && iopen == iopen_ && cross == cross_ && lut.p)
        return PBI4G_OK;
    if (nb_ < 1 || nb_ > 4096 || !(kbin_ > 0) || N_ < 4 || (N_ & 1))
        return set_error(PBI4G_ERR_INVALID, "shells: grid=%d nbins=%d kbin=%g", N_, nb_, kbin_);
    N = N_; kbin = kbin_; kcenter = kcenter_; nb = nb_; iopen = iopen_; cross = cross_;
    counts.clear();
    const double kck = (double)(kcenter / kbin);
    const int h = N / 2;
    k2max = 3 * h * h;
    lut_h.assign(k2max + 1, 0);
    int k2top = -1;  // the largest |k|^2 of a shell
    for (int k2 = 0; k2 <= k2max; k2++) {
        // idist = nint(dsqrt(di*di+dj*dj+dl*dl)/kbin - kcenter/kbin - tiny) + 1
        // (bispectrumI4.f90:73); di^2+dj^2+dl^2 is exact, so idist depends on k2 only.
        long long b = llround(sqrt((double)k2) / (double)kbin - kck - (double)FLT_MIN) + 1;
        if (b > nb) break;  // (it never decreases)
        if (b < 1) continue;
        lut_h[k2] = (int)b;
        k2top = k2;
    }
    // Map grid: every shell mode has |k_axis| <= kmax, so the per-axis sum of
    // three of them lies in [-3 kmax, 3 kmax].  On any grid Nm > 3 kmax the
    // condition q1+q2+q3 = 0 (mod Nm) holds only for exact triangles; when
    // 3 kmax < N the reference's N grid has no aliased triangles either, and the
    // sum over x of three maps on the Nm grid equals the reference's sum times
    // (Nm/N)^3.  Otherwise the maps stay on the N grid.
    kmax = k2top > 0 ? (int)floor(sqrt((double)k2top)) : 0;
    // full-grid modes per shell: multiplicity of |k_axis| = d is 1 for d in {0, N/2}, else 2.
    // Only the sphere up to k2top holds any (a walk over the whole octant took 0.3 ms at 128^3).
    nmodes.assign(nb, 0);
    const int top = std::min(h, kmax);
    auto mult = [&](int d) { return d == 0 || d == h ? 1 : 2; };
    for (int dz = 0; dz <= top; dz++)
        for (int dy = 0; dy <= top && dy * dy + dz * dz <= k2top; dy++)
            for (int dx = 0; dx <= top && dx * dx + dy * dy + dz * dz <= k2top; dx++) {
                int b = lut_h[dx * dx + dy * dy + dz * dz];
                if (!b) continue;
                nmodes[b - 1] += mult(dx) * mult(dy) * mult(dz);
            }
    Nm = map_grid_for_kmax(N, kmax);
    ishift = (int)(kcenter / kbin) + (iopen ? 1 : 0);  // bispectrumI4.f90:38-42
    tri.clear();
    for (int l = 1; l <= nb; l++)
        for (int j = 1; j <= l; j++) {
            int imax = cross ? std::min(nb, j + l - 1 + ishift) : j;
            for (int i = std::max(1, l - j + 1 - ishift); i <= imax; i++) {
                tri.push_back(l);
                tri.push_back(j);
                tri.push_back(i);
            }
        }
    itot = (int64_t)tri.size() / 3;
    PBI4G_CHECK(lut.ensure(sizeof(int) * (k2max + 1)));
    PBI4G_CUDA(cudaMemcpyAsync(lut.p, lut_h.data(), sizeof(int) * (k2max + 1), cudaMemcpyHostToDevice, st));
    std::vector<double> nm(nb);
    for (int b = 0; b < nb; b++) nm[b] = (double)nmodes[b];
    PBI4G_CHECK(tri_d.ensure(sizeof(int) * std::max<size_t>(3, tri.size())));
    PBI4G_CUDA(cudaMemcpyAsync(tri_d.p, tri.data(), sizeof(int) * tri.size(), cudaMemcpyHostToDevice, st));
    PBI4G_CHECK(nmodes_d.ensure(sizeof(double) * nb));
    PBI4G_CUDA(cudaMemcpyAsync(nmodes_d.p, nm.data(), sizeof(double) * nb, cudaMemcpyHostToDevice, st));
    PBI4G_CUDA(cudaStreamSynchronize(st));
    return PBI4G_OK;
}

// ------------------------------------------------------- map spectra ---
template <class C> __device__ __forceinline__ C czero() { C c; c.x = 0; c.y = 0; return c; }

constexpr int kMapChunk = 8;  // maps per block row: each block writes 8 contiguous map regions

template <class R>
__global__ void build_map_spectra_kernel(int N, int Nm, int nb, int k2max, const int *__restrict__ lut, int count,
                                         const typename Cx<R>::T *__restrict__ s0,
                                         const typename Cx<R>::T *__restrict__ s1,
                                         const typename Cx<R>::T *__restrict__ s2, int f0, int f1, int f2, double l0,
                                         double l1, double l2, typename Cx<R>::T *__restrict__ out,
                                         double *__restrict__ powsum, int pow_mask) {
    using C = typename Cx<R>::T;
    extern __shared__ double spow[];  // [3][nb] powers sum |H|^2 over the full grid, per set and shell
    if (powsum)
        for (int b = threadIdx.x; b < 3 * nb; b += blockDim.x) spow[b] = 0.0;
    __syncthreads();
    const int NH = N / 2 + 1, NHm = Nm / 2 + 1;
    const size_t HCm = (size_t)Nm * Nm * NHm;
    const int j0 = blockIdx.y * kMapChunk, j1 = min(count, j0 + kMapChunk);
    for (size_t cell = blockIdx.x * (size_t)blockDim.x + threadIdx.x; cell < HCm;
         cell += (size_t)gridDim.x * blockDim.x) {
        const int x = (int)(cell % NHm), y = (int)((cell / NHm) % Nm), z = (int)(cell / ((size_t)NHm * Nm));
        const int ky = kfreq0(y, Nm), kz = kfreq0(z, Nm);
        const int k2 = x * x + ky * ky + kz * kz;
        const int sb = k2 <= k2max ? lut[k2] : 0;
        bool any = false;
        for (int j = j0; j < j1; j++) any |= (j % nb + 1 == sb);
        if (!any) {
            for (int j = j0; j < j1; j++) out[(size_t)j * HCm + cell] = czero<C>();
            continue;
        }
        // source cell on the N grid (same signed frequency), and its mirror -k
        const int yN = ky < 0 ? ky + N : ky, zN = kz < 0 ? kz + N : kz;
        const size_t sc = ((size_t)zN * N + yN) * NH + x;
        const bool herm = (x == 0 || x == Nm / 2);
        const size_t mc = ((size_t)kneg0(zN, N) * N + kneg0(yN, N)) * NH + x;
        const double lk = l0 * x + l1 * ky + l2 * kz;
        const R mu2 = k2 > 0 ? (R)(lk * lk / (double)k2) : (R)0;
        const double wfull = herm ? 1.0 : 2.0;
        for (int j = j0; j < j1; j++) {
            const int s = j / nb, b = j % nb + 1;
            if (b != sb) {
                out[(size_t)j * HCm + cell] = czero<C>();
                continue;
            }
            const C *src = s == 0 ? s0 : (s == 1 ? s1 : s2);
            const int fac = s == 0 ? f0 : (s == 1 ? f1 : f2);
            C v = src[sc];
            if (herm) {
                const C w = src[mc];
                v.x = (v.x + w.x) * (R)0.5;
                v.y = (v.y - w.y) * (R)0.5;
            }
            R L = 1;
            if (fac == 2) L = (R)-0.5 + (R)1.5 * mu2;
            else if (fac == 4) L = (R)0.375 + mu2 * ((R)-3.75 + (R)4.375 * mu2);
            v.x *= L;
            v.y *= L;
            out[(size_t)j * HCm + cell] = v;
            if (powsum && (pow_mask >> s & 1))
                atomicAdd(&spow[s * nb + b - 1], wfull * ((double)v.x * v.x + (double)v.y * v.y));
        }
    }
    if (powsum) {
        __syncthreads();
        for (int b = threadIdx.x; b < 3 * nb; b += blockDim.x)
            if (spow[b] != 0.0) atomicAdd(powsum + b, spow[b]);
    }
}

template <class R>
int build_map_spectra(const Shells &sh, int count, const typename Cx<R>::T *const src[3], const int fac[3],
                      const double los[3], typename Cx<R>::T *out, double *powsum, int pow_mask, cudaStream_t st,
                      int64_t *launches) {
    const size_t smem = powsum ? sizeof(double) * 3 * sh.nb : 0;
    const dim3 grid(grid_blocks(half_cells(sh.Nm), 256, 152 * 2), (count + kMapChunk - 1) / kMapChunk);
    build_map_spectra_kernel<R><<<grid, 256, smem, st>>>(
        sh.N, sh.Nm, sh.nb, sh.k2max, sh.lut.as<int>(), count, src[0], src[1], src[2], fac[0], fac[1], fac[2],
        los ? los[0] : 0, los ? los[1] : 0, los ? los[2] : 0, out, powsum, pow_mask);
    PBI4G_LAUNCH_CHECK();
    ++*launches;
    return PBI4G_OK;
}

template int build_map_spectra<float>(const Shells &, int, const float2 *const[3], const int[3], const double[3],
                                      float2 *, double *, int, cudaStream_t, int64_t *);

template int build_map_spectra<double>(const Shells &, int, const double2 *const[3], const int[3], const double[3],
                                       double2 *, double *, int, cudaStream_t, int64_t *);

template <class R>
__global__ void build_indicator_kernel(int N, int k2max, const int *__restrict__ lut, int m0, int count,
                                       typename Cx<R>::T *__restrict__ out) {
    using C = typename Cx<R>::T;
    const int NH = N / 2 + 1;
    const size_t HC = (size_t)N * N * NH;
    for (size_t cell = blockIdx.x * (size_t)blockDim.x + threadIdx.x; cell < HC;
         cell += (size_t)gridDim.x * blockDim.x) {
        const int x = (int)(cell % NH), ay = kabs0((int)((cell / NH) % N), N),
                  az = kabs0((int)(cell / ((size_t)NH * N)), N);
        const int k2 = x * x + ay * ay + az * az;
        const int sb = k2 <= k2max ? lut[k2] : 0;
        for (int j = 0; j < count; j++) {
            C v = czero<C>();
            if (sb == m0 + j + 1) v.x = 1;
            out[(size_t)j * HC + cell] = v;
        }
    }
}

template <class R>
int build_indicator_spectra(const Shells &sh, int m0, int count, typename Cx<R>::T *out, cudaStream_t st,
                            int64_t *launches) {
    build_indicator_kernel<R><<<grid_blocks(half_cells(sh.Nm), 256, 152 * 8), 256, 0, st>>>(
        sh.Nm, sh.k2max, sh.lut.as<int>(), m0, count, out);
    PBI4G_LAUNCH_CHECK();
    ++*launches;
    return PBI4G_OK;
}
template int build_indicator_spectra<float>(const Shells &, int, int, float2 *, cudaStream_t, int64_t *);
template int build_indicator_spectra<double>(const Shells &, int, int, double2 *, cudaStream_t, int64_t *);

// ------------------------------------------------------------ outputs ---
// Eight lanes a triangle, a quotient or two each: the FP64 divisions one after another were
// most of the time (86 triangles: 7.1 -> 6.6 us).
__global__ void bk_finalize_kernel(int64_t itot, int nb, int nsets, int cross, const int *__restrict__ tri,
                                   const double *__restrict__ S, const double *__restrict__ powsum,
                                   const double *__restrict__ nmodes, double kf3, double powSN, double gridD,
                                   double kcenter, double kbin, const float *__restrict__ counts,
                                   double *__restrict__ bout, double sfac, const BoxPar *__restrict__ bp) {
    if (bp) powSN = bp->pow_sn;
    const double powSN2 = powSN * powSN;
    const int part = threadIdx.x & 7, lane = threadIdx.x & 31;
    const int64_t step = ((int64_t)gridDim.x * blockDim.x) >> 3;
    // whole warps go round together (the lanes exchange values)
    for (int64_t m0 = (blockIdx.x * (int64_t)blockDim.x + (threadIdx.x & ~31)) >> 3; m0 < itot; m0 += step) {
        const int64_t m = m0 + (lane >> 3);
        const bool is = m < itot;
        // parts 0, 1, 2: the sides; 3: B; 4: triangle count; 5, 6: B's multipoles
        double v = 0, t = 0;
        if (is) {
            if (part < 3) {
                const int b = tri[3 * m + part];
                t = kcenter + (double)(b - 1) * kbin;
                // pow(i) = kf3*avg/dble(gridd)/dble(nmodes) - powSN, avg = sum_x m^2 = gridD * sum_k |H|^2
                if (!cross) v = kf3 * (gridD * powsum[b - 1]) / gridD / nmodes[b - 1] - powSN;
            } else if (part == 4) {
                v = (double)(float)((double)counts[m] / gridD);
            } else {
                const int set = part == 3 ? 0 : part - 4;
                if (set < nsets)
                    v = (set == 0 ? kf3 : (set == 1 ? 5 * kf3 : 9 * kf3)) * (sfac * S[m * nsets + set]) / (double)counts[m];
            }
        }
        const int first = lane & ~7;
        const double pl = __shfl_sync(0xffffffffu, v, first), pj = __shfl_sync(0xffffffffu, v, first + 1),
                     pi = __shfl_sync(0xffffffffu, v, first + 2);
        if (!is) continue;
        const int rows = cross ? 5 : (nsets == 3 ? 11 : 9);
        double *o = bout + (size_t)rows * m;
        if (part < 3) o[part] = t;
        if (cross) {
            if (part == 3 || part == 4) o[part] = v;
            continue;
        }
        const double bispSN = (pi + pj + pl) * powSN + powSN2;
        if (part < 3) o[3 + part] = v;
        else if (part == 3) o[6] = v + bispSN;
        else if (part == 4) o[7] = bispSN, o[8] = v;
        else if (nsets == 3 && part < 7) o[4 + part] = v;
    }
}

double bk_pow_sn(float kf, int64_t npart) {
    const float kf3f = kf * kf * kf;
    return 1.0 / (double)npart / (double)kf3f;
}

int bk_finalize(const Shells &sh, int nsets, int cross, const double *S, const double *powsum, float kf,
                int64_t npart, const float *counts_f32, double *bout, cudaStream_t st, int64_t *launches,
                const BoxPar *bp) {
    const float kf3f = kf * kf * kf;
    const double kf3 = (double)kf3f;
    const double powSN = bk_pow_sn(kf, npart);
    const double gridD = (double)sh.N * sh.N * sh.N;
    bk_finalize_kernel<<<grid_blocks(8 * (size_t)sh.itot, 128), 128, 0, st>>>(
        sh.itot, sh.nb, nsets, cross, sh.tri_d.as<int>(), S, powsum, sh.nmodes_d.as<double>(), kf3, powSN, gridD,
        (double)sh.kcenter, (double)sh.kbin, counts_f32, bout,
        // the sums were taken over the Nm^3 map grid: the reference sums over N^3
        ((double)sh.N / sh.Nm) * ((double)sh.N / sh.Nm) * ((double)sh.N / sh.Nm), bp);
    PBI4G_LAUNCH_CHECK();
    ++*launches;
    return PBI4G_OK;
}

// ------------------------------------------------------------- counts ---
// Counts depend only on (grid, kbin, kcenter, nbins, iopen, cross): one
// process-wide copy per binning serves every plan that uses it.
static std::mutex g_counts_mutex;
static std::map<std::tuple<int, float, float, int, int, int>, std::vector<int64_t>> g_counts_cache;

// sh.counts says that counts_f32 holds them: it is set last
static int upload_counts(Shells &sh, const std::vector<int64_t> &counts) {
    const double gridD = (double)sh.N * sh.N * sh.N;
    std::vector<float> c32(sh.itot);
    for (int64_t m = 0; m < sh.itot; m++) c32[m] = (float)(gridD * (double)counts[m]);
    PBI4G_CHECK(sh.counts_f32.ensure(sizeof(float) * std::max<int64_t>(1, sh.itot)));
    PBI4G_CUDA(cudaMemcpy(sh.counts_f32.p, c32.data(), sizeof(float) * sh.itot, cudaMemcpyHostToDevice));
    sh.counts = counts;
    return PBI4G_OK;
}

// Orbit representatives of the map grid under the cube group (the 48 axis
// permutations and sign flips, x_a -> -x_a mod Nm).  A shell indicator map
// I_b(x) = sum over the shell's modes of e^{2 pi i k.x / Nm} is invariant under
// the group (the shell is a set of |k|, and Nm / 2 is no shell frequency since
// Nm > 3 kmax), so sum_x I_l I_j I_i = sum over representatives (a <= b <= c,
// each in [0, Nm/2]) of |orbit| I_l I_j I_i, with |orbit| = 2 per coordinate
// outside {0, Nm/2} times the distinct permutations of (a, b, c) (6, 3 or 1).
// Representatives are packed a | b << 11 | c << 22 and padded with weight-0
// points to a multiple of 64.
static int orbit_points(int Nm, std::vector<unsigned> &pts, long long &nrep) {
    const int h = Nm / 2;
    pts.clear();
    long long wsum = 0;
    for (int a = 0; a <= h; a++)
        for (int b = a; b <= h; b++)
            for (int c = b; c <= h; c++) {
                pts.push_back((unsigned)a | ((unsigned)b << 11) | ((unsigned)c << 22));
                const int sg = (a == 0 || a == h ? 1 : 2) * (b == 0 || b == h ? 1 : 2) * (c == 0 || c == h ? 1 : 2);
                const int pm = (a == b && b == c) ? 1 : ((a == b || b == c) ? 3 : 6);
                wsum += (long long)sg * pm;
            }
    nrep = (long long)pts.size();
    if (wsum != (long long)Nm * Nm * Nm)
        return set_error(PBI4G_ERR_UNSUPPORTED, "orbit weights of grid %d sum to %lld", Nm, wsum);
    while (pts.size() % 64) pts.push_back(0u);
    return PBI4G_OK;
}

__device__ __forceinline__ double orbit_weight(unsigned pk, int h) {
    const int a = pk & 2047, b = (pk >> 11) & 2047, c = pk >> 22;
    const int sg = (a == 0 || a == h ? 1 : 2) * (b == 0 || b == h ? 1 : 2) * (c == 0 || c == h ? 1 : 2);
    const int pm = (a == b && b == c) ? 1 : ((a == b || b == c) ? 3 : 6);
    return (double)(sg * pm);
}

// maps [m0, m0 + count) of the in-place C2R output (map j at real + j * 2 HC,
// point (a, b, c) at (a Nm + b) (2 NH) + c) at the representatives:
// out[m][p] = I_m(rep p), out[nb + m][p] = |orbit p| I_m(rep p)
__global__ void orbit_gather_kernel(int Nm, int nb, int m0, int count, long long nrep, long long npad,
                                    const unsigned *__restrict__ pts, const double *__restrict__ real,
                                    double *__restrict__ out) {
    const int NH = Nm / 2 + 1;
    const size_t HC2 = 2 * (size_t)Nm * Nm * NH;
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < npad;
         p += (long long)gridDim.x * blockDim.x) {
        const unsigned pk = pts[p];
        const bool real_pt = p < nrep;
        const double w = real_pt ? orbit_weight(pk, Nm / 2) : 0.0;
        const size_t off = ((size_t)(pk & 2047) * Nm + ((pk >> 11) & 2047)) * (2 * NH) + (pk >> 22);
        for (int j = 0; j < count; j++) {
            const double v = real_pt ? real[(size_t)j * HC2 + off] : 0.0;
            out[(size_t)(m0 + j) * npad + p] = v;
            out[(size_t)(nb + m0 + j) * npad + p] = w * v;
        }
    }
}

int triangle_counts(Shells &sh, cudaStream_t st, int64_t *launches) {
    if (!sh.counts.empty()) return PBI4G_OK;
    const auto ckey = std::make_tuple(sh.N, sh.kbin, sh.kcenter, sh.nb, sh.iopen, sh.cross);
    {
        std::lock_guard<std::mutex> g(g_counts_mutex);
        auto it = g_counts_cache.find(ckey);
        if (it != g_counts_cache.end()) return upload_counts(sh, it->second);
    }
    const int N = sh.Nm, nb = sh.nb, NH = N / 2 + 1;  // indicator maps on the map grid
    if (N > 2046) return set_error(PBI4G_ERR_UNSUPPORTED, "counts: map grid %d", N);
    const size_t HC = half_cells(N);
    std::vector<unsigned> hpts;
    long long nrep = 0;
    PBI4G_CHECK(orbit_points(N, hpts, nrep));
    const long long npad = (long long)hpts.size();
    DevBuf pts, rep, spec, partial, S;
    PBI4G_CHECK(pts.ensure(sizeof(unsigned) * hpts.size()));
    PBI4G_CUDA(cudaMemcpyAsync(pts.p, hpts.data(), sizeof(unsigned) * hpts.size(), cudaMemcpyHostToDevice, st));
    PBI4G_CHECK(rep.ensure(sizeof(double) * 2 * (size_t)nb * npad));
    // indicator spectra and their FP64 C2R in batches of at most 4 GiB
    const int bsz = (int)std::max<size_t>(1, std::min<size_t>((size_t)nb, ((size_t)4 << 30) / (sizeof(double2) * HC)));
    PBI4G_CHECK(spec.ensure(sizeof(double2) * HC * bsz));
    int n[3] = {N, N, N}, inembed[3] = {N, N, NH}, onembed[3] = {N, N, 2 * NH};
    cufftHandle plan = 0;
    int plan_batch = 0;
    int rc = PBI4G_OK;
    for (int m0 = 0; m0 < nb && rc == PBI4G_OK; m0 += bsz) {
        const int cnt = std::min(bsz, nb - m0);
        if ((rc = build_indicator_spectra<double>(sh, m0, cnt, spec.as<double2>(), st, launches))) break;
        if (plan_batch != cnt) {
            if (plan) cufftDestroy(plan);
            plan = 0;
            if (cufftPlanMany(&plan, 3, n, inembed, 1, (int)HC, onembed, 1, (int)(2 * HC), CUFFT_Z2D, cnt) !=
                CUFFT_SUCCESS) {
                plan = 0;
                rc = set_error(PBI4G_ERR_CUFFT, "counts: cufftPlanMany (%d maps of grid %d)", cnt, N);
                break;
            }
            plan_batch = cnt;
        }
        cufftSetStream(plan, st);
        const cufftResult r = cufftExecZ2D(plan, spec.as<cufftDoubleComplex>(), spec.as<cufftDoubleReal>());
        if (r != CUFFT_SUCCESS) {
            rc = set_error(PBI4G_ERR_CUFFT, "counts: cufftExecZ2D failed (%d)", (int)r);
            break;
        }
        orbit_gather_kernel<<<grid_blocks((size_t)npad, 256, 152 * 8), 256, 0, st>>>(
            N, nb, m0, cnt, nrep, npad, pts.as<unsigned>(), spec.as<double>(), rep.as<double>());
        if (cudaPeekAtLastError() != cudaSuccess) {
            rc = set_error(PBI4G_ERR_CUDA, "counts: gather launch: %s", cudaGetErrorString(cudaGetLastError()));
            break;
        }
        ++*launches;
    }
    if (plan) {
        cudaStreamSynchronize(st);
        cufftDestroy(plan);
    }
    PBI4G_CHECK(rc);
    spec.release();
    // all three factors are indicator maps of the same set (also for the cross
    // enumeration, bispectrumI4.f90:887-896), so the non-cross pair layout
    // applies: pairs from the plain copies [0, nb), q from the weighted copies
    TriPlan tp;
    PBI4G_CHECK(tp.build(sh, 1, 0, true, nb));
    PBI4G_CHECK(S.ensure(sizeof(double) * tp.nslots));
    PBI4G_CHECK(triangle_sums<double>(sh, tp, rep.as<double>(), (size_t)npad, 64, 64, npad, partial, S.as<double>(),
                                      false, st, launches));
    std::vector<double> Sh(tp.nslots);
    PBI4G_CUDA(cudaMemcpyAsync(Sh.data(), S.p, sizeof(double) * tp.nslots, cudaMemcpyDeviceToHost, st));
    PBI4G_CUDA(cudaStreamSynchronize(st));
    const double gridD = (double)N * N * N;
    std::vector<int64_t> counts(sh.itot);
    double maxdev = 0;
    for (int64_t m = 0; m < sh.itot; m++) {
        double v = Sh[m] / gridD;
        long long c = llround(v);
        maxdev = std::max(maxdev, fabs(v - (double)c));
        counts[m] = c;
    }
    if (maxdev > 0.25)
        return set_error(PBI4G_ERR_RANGE, "triangle counts not resolved to integers (max deviation %g)", maxdev);
    {
        std::lock_guard<std::mutex> g(g_counts_mutex);
        g_counts_cache[ckey] = counts;
    }
    return upload_counts(sh, counts);
}

}  // namespace pbi4g
