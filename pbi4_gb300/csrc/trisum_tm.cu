// trisum_tm.cu -- triangle sums on tcgen05 with the pair products in tensor memory.
//
// The "Last sum" loops of measure_bk / measure_bk_multipoles
// (bispectrumI4.f90:160-195, 476-513), S(l,j,i) = sum_x M_i M_j M_l (and the
// B2/B4 sums with the delta_2 / delta_4 maps of shell l), recast as a
// contraction over the grid points x:
//     C[p, q] = sum_x A[p, x] B[q, x],  A[p, x] = M_i(x) M_j(x) for the pair p = (i, j),
//                                       B[q, x] = map q (plane rows: shell-major, set-minor).
// Only the (p, q) entries that are triangles are kept.
//
// Which pairs: a chunk costs a unit (128 pairs x a window of plane rows) about the same
// whatever it holds, so the plan makes few units.  With one q set the three factors of a
// triangle are alike and any of its pairs may be the A row: 489 pairs meet the triangles of
// 48 shells, where the pairs i <= j are 1176 (4 units instead of 10: 5.1 ms against 14.0 ms
// at 300^3 points).  With three sets the pairs are sorted so that a tile's triangles lie in
// a short range of shells, and a unit takes a window of 16 to 64 rows of it (40 shells: 9
// units instead of 14, 7.3 ms against 12.2 ms at 256^3 points).
//
// Operand forms (FP32 accumulation in every form):
//   TF32 split: hi = v with the 13 low mantissa bits cleared (exact in TF32),
//     lo = v - hi; A_hi.B_hi + A_hi.B_lo + A_lo.B_hi with kind::tf32 (K = 8).
//     The FP32 exponent range needs no scaling; every product carries a
//     relative error below 2^-20.
//   FP16 split: every operand scaled by a power of two so |v| <= 2^14 (a
//     per-map bound from Parseval: |M| <= sqrt(nmodes * sum |H|^2)), hi =
//     fp16(v), lo = fp16(v - hi); the same three products with kind::f16 (K = 16).
//   BF16: one bf16 product, kind::f16 with bf16 operands (K = 16).
//
// Data path per chunk of 64 grid points (one CTA per (unit, K range)):
//   * the x pass of the map transform writes the maps as operand planes
//     [row][point] (FP16 hi / lo, BF16, or TF32 hi / lo) plus the set-0 maps in
//     FP32 (the pair factors), so the B tiles need no conversion here;
//   * a TMA warp loads each chunk's B tiles (the window's rows x 64 points, 128-byte
//     swizzled: the K-major operand layout itself) and the FP32 set-0 maps of
//     the chunk into a ring of shared-memory stages, one instruction an operand;
//   * three producer warpgroups take the chunks in turn.  16-bit forms: a thread takes
//     four pair rows that share a map and 16 points of each (the 16x256b layout of
//     tcgen05.st), so the shared map is read once for four products: 20 shared loads
//     for 64 products instead of 32.  It splits the products and stores them straight
//     into a tensor-memory A stage (the A operand never touches shared memory);
//   * two MMA warps issue the MMAs (A in TMEM, B from the stage) of alternate chunks
//     into one of two TMEM accumulators, a fresh one per chunk, and commit them to a
//     per-chunk completion barrier that frees the A stage, the accumulator and
//     (with the producers' release) the shared-memory stage.  The tensor core
//     adds the products of one instruction to the accumulator with truncation,
//     so keeping each accumulation to one chunk keeps that error near 1e-6;
//   * two drain warpgroups (half of the unit's columns each) add each chunk's
//     accumulator into FP32 registers (round to nearest) and fold those into a
//     Kahan-compensated sum every 16 chunks (kept in the TMEM columns the
//     accumulators and A stages leave free), then write the final sums (FP64,
//     scaled back by the FP16 exponents) of the triangle slots.
//
// What bounds it: the latency of the hand-offs around a chunk, 0.49 us a unit and chunk
// (256^3 box, 2 units: 0.81 ms).  Leaving parts out of it took: barriers alone 0.38 ms,
// with the TMA copies 0.51, with the MMAs too 0.60, with the pair products 0.69, with
// their TMEM stores 0.81.  Neither more accumulators (their sums then live in L2 or shared
// memory: 1.25 ms) nor polling waits (0.99 ms) shortened it.
// Every wait is bounded: a wait that runs out sets an abort flag that ends all
// roles, records the error for the host, and the CTA waits (bounded) for its
// own MMAs and copies in flight before it frees its tensor memory.
#include <cuda.h>  // CUtensorMap and its enums (the encoder is fetched through the runtime)
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <queue>
#include <type_traits>
#include <vector>

#include "bispec.cuh"
#include "tc_ptx.cuh"
#include "trisum_tm.cuh"

namespace pbi4g {

namespace {

using namespace tcx;

constexpr int kM = 128;          // pairs per unit (MMA M = TMEM lanes)
constexpr int kN = 64;           // plane rows per unit at most (MMA N: 16, 32, 48 or 64)
constexpr int kKB = 32;          // FP32 values per 128-byte swizzle row (one K block)
constexpr int kBlocks = 2;       // K blocks per chunk
constexpr int kKC = kKB * kBlocks;  // grid points per chunk
constexpr int kMaxStages = 10;   // TMA staging slots (released by the producers and the MMAs)
constexpr int kGroups = 3;       // producer warpgroups, chunks assigned round robin (2: 8% slower at 256^3)
constexpr int kProdWarps = 4 * kGroups;
constexpr int kDrainWarps = 8;   // two warpgroups, 32 accumulator columns each
constexpr int kMmaWarp = kProdWarps + kDrainWarps;
constexpr int kMmaWarps = 2;     // MMA issuers, chunks alternating (a thread's MMAs of a chunk stay in order)
constexpr int kTmaWarp = kMmaWarp + kMmaWarps;
constexpr int kThreads = (kTmaWarp + 1) * 32;  // 736
constexpr int kFold = 16;  // chunks summed in registers before a Kahan fold
constexpr int kAcc = 2;          // TMEM accumulators (one chunk each)
constexpr int kDone = 16;        // per-chunk MMA completion barriers (ring)
constexpr int kMaxAStages = 6;   // producer -> MMA barriers (one per A stage)
constexpr uint32_t kColAcc = 0;  // kAcc accumulators of kN columns, then the A stages
constexpr uint32_t kColA = kAcc * kN;
constexpr uint32_t kTmemCols = 512;
static_assert(kMaxStages <= kDone, "a stage's MMA barrier must not have cycled when the stage is reused");
constexpr uint32_t kTfMask = 0xFFFFE000u;

enum : int { kFormTF32 = 0, kFormF16 = 1, kFormBF16 = 2 };

template <int F> struct Form;
// TF32 split: A stage = 64 hi + 64 lo columns, 8 K-steps of 8, 3 products
template <> struct Form<kFormTF32> {
    static constexpr uint32_t kACols = 2 * kKC;
    static constexpr int kAStages = 2;
    static constexpr int kBTiles = 4;  // hi, hi, lo, lo: 32 FP32 points per 128-byte row
    static constexpr int kKStep = 8;
    static constexpr bool kSplit = true;
    static constexpr uint32_t kIdesc = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(kM >> 4) << 24);  // N to be added (idesc_n)
};
// FP16 split: A stage = 32 hi + 32 lo packed columns, 4 K-steps of 16, 3 products
template <> struct Form<kFormF16> {
    static constexpr uint32_t kACols = kKC;
    static constexpr int kAStages = 4;
    static constexpr int kBTiles = 2;  // hi, lo: 64 FP16 points per 128-byte row
    static constexpr int kKStep = 16;
    static constexpr bool kSplit = true;
    static constexpr uint32_t kIdesc = (1u << 4) | (0u << 7) | (0u << 10) | ((uint32_t)(kM >> 4) << 24);  // N to be added (idesc_n)
};
// BF16: A stage = 32 packed columns, 4 K-steps of 16, 1 product
template <> struct Form<kFormBF16> {
    static constexpr uint32_t kACols = kKC / 2;
    static constexpr int kAStages = 4;
    static constexpr int kBTiles = 1;
    static constexpr int kKStep = 16;
    static constexpr bool kSplit = false;
    static constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kM >> 4) << 24);  // N to be added (idesc_n)
};
// A waiter on an mbarrier names the phase by its parity, so each A stage and each
// accumulator must be consumed by one issuing thread, chunk after chunk: issuer w
// takes chunks w + k kMmaWarps, which use stage (and accumulator) i % count only if
// count is a multiple of kMmaWarps.  Otherwise an issuer two phases ahead of a stage
// would read a stale parity as complete.
static_assert(kAcc % kMmaWarps == 0, "accumulators per issuer");
// the producer -> MMA barriers (one per A stage) are an array of kMaxAStages
static_assert(Form<kFormTF32>::kAStages <= kMaxAStages && Form<kFormF16>::kAStages <= kMaxAStages &&
                  Form<kFormBF16>::kAStages <= kMaxAStages,
              "A stages beyond the barrier array");
static_assert(Form<kFormTF32>::kAStages % kMmaWarps == 0 && Form<kFormF16>::kAStages % kMmaWarps == 0 &&
                  Form<kFormBF16>::kAStages % kMmaWarps == 0,
              "A stages per issuer");
static_assert(kColA + Form<kFormTF32>::kAStages * Form<kFormTF32>::kACols <= kTmemCols, "TMEM budget");
static_assert(kColA + Form<kFormF16>::kAStages * Form<kFormF16>::kACols <= kTmemCols, "TMEM budget");

__device__ __forceinline__ uint32_t idesc_n(int ncols) { return (uint32_t)(ncols >> 3) << 17; }

// D[tmem] (+)= A[tmem] . B[smem]^T
template <int F>
__device__ __forceinline__ void umma_ta(uint32_t d_tmem, uint32_t a_tmem, uint64_t b, uint32_t idesc, uint32_t accum) {
    if constexpr (F == kFormTF32)
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %3, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %4, p;\n\t}" ::"r"(d_tmem),
            "r"(a_tmem), "l"(b), "r"(accum), "r"(idesc)
            : "memory");
    else
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %3, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %4, p;\n\t}" ::"r"(d_tmem),
            "r"(a_tmem), "l"(b), "r"(accum), "r"(idesc)
            : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}

// box at (0, row y, 0, chunk z) of a chunk view (make_chunk_view)
__device__ __forceinline__ void tma_load_chunk(void *dst, const CUtensorMap *tm, int y, int z, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %2, "
        "%4}], [%5];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(tm)), "r"(0), "r"(y), "r"(z), "r"(smem_u32(bar))
        : "memory");
}

// Suspend-time hint of the main-loop waits (ns; 0: plain polling).
#ifndef PBI4G_TM_WAIT_HINT_NS
#define PBI4G_TM_WAIT_HINT_NS 0
#endif

// Bounded wait of the main loop that also gives up once another role has
// aborted: kWaitNs of device time (the abort flag and the timer read every 256
// polls).  The diagnostic instantiation (D) polls `limit` times without
// blocking instead, so that such waits run out on healthy work
// (pbi4g_plan_debug_wait_limit); everything else in the kernel is the same.
template <bool D>
__device__ __forceinline__ bool wait_or_abort(uint64_t *bar, uint32_t parity, volatile int *abort_flag,
                                              uint32_t limit) {
    if constexpr (D) {
        for (uint32_t i = 0; i < limit; i++)
            if (mbar_test_wait(bar, parity)) return true;
        return false;
    } else {
        if (mbar_try_wait(bar, parity)) return true;
        const uint32_t t0 = global_ns();
        for (uint32_t i = 1;; i++) {
            if (PBI4G_TM_WAIT_HINT_NS > 0 ? mbar_try_wait_sleep(bar, parity, PBI4G_TM_WAIT_HINT_NS)
                                          : mbar_try_wait(bar, parity))
                return true;
            if ((i & 255) == 0 && (*abort_flag || global_ns() - t0 > kWaitNs)) return false;
        }
    }
}

// The same, with one answer for the whole warp (the tcgen05 loads and stores
// that follow are warp-collective: every lane takes the same branch).
template <bool D>
__device__ __forceinline__ bool warp_wait(uint64_t *bar, uint32_t parity, volatile int *abort_flag, uint32_t limit) {
    return __all_sync(0xffffffffu, wait_or_abort<D>(bar, parity, abort_flag, limit));
}

// Barrier parity of the completion, for chunk i, of a barrier used every `every` chunks.
__device__ __forceinline__ uint32_t ph(int i, int every) { return (uint32_t)((i / every) & 1); }

// Slot and phase of a ring of `size` barriers, advanced by additions: the roles'
// loops run on a single thread or warp per chunk, where a division by the
// runtime stage count is a long dependent chain.
struct Ring {
    int idx, phase;
    __device__ __forceinline__ Ring(int start, int size) : idx(start % size), phase((start / size) & 1) {}
    __device__ __forceinline__ void step(int k, int size) {  // k <= size
        idx += k;
        if (idx >= size) {
            idx -= size;
            phase ^= 1;
        }
    }
};

// two products u0 v0, u1 v1 -> packed 16-bit hi, and for the FP16 split lo =
// u v - hi (the FMA keeps the product's own rounding error out of lo).  The
// packed FP32 pair instructions round each element as the scalar ones do; they
// made the triangle sums 5% faster at 256^3.
template <int F>
__device__ __forceinline__ void pack_prod2(float u0, float v0, float u1, float v1, uint32_t &hi, uint32_t &lo) {
    if constexpr (F == kFormF16) {
        // packed FP32 pairs: the same roundings as two scalar products and FMAs
        const float2 u = make_float2(u0, u1), v = make_float2(v0, v1);
        const __half2 h = __float22half2_rn(__fmul2_rn(u, v));
        const float2 back = __half22float2(h);
        const __half2 l = __float22half2_rn(__ffma2_rn(u, v, make_float2(-back.x, -back.y)));
        hi = *reinterpret_cast<const uint32_t *>(&h);
        lo = *reinterpret_cast<const uint32_t *>(&l);
    } else {
        const __nv_bfloat162 h = __float22bfloat162_rn(__fmul2_rn(make_float2(u0, u1), make_float2(v0, v1)));
        hi = *reinterpret_cast<const uint32_t *>(&h);
        lo = 0u;
    }
}

// The drain's Kahan sums live in the TMEM columns that two accumulators and the A stages
// leave free: in an L2 scratch beside four accumulators the folds waited on L2 round trips
// (1.08 ms against 1.00 ms at 256^3), and halving the A stages instead took 1.33 ms.
template <int F>
constexpr bool kahan_fits() {
    return kColA + (uint32_t)Form<F>::kAStages * Form<F>::kACols + 2 * kN <= kTmemCols;
}
static_assert(kahan_fits<kFormTF32>() && kahan_fits<kFormF16>() && kahan_fits<kFormBF16>(), "TMEM budget");

struct TmArgs {
    long long nchunks;     // points / kKC, rounded up
    int nunits, ksplit, nslots, nA, nstages, nmaps, nb;
    uint32_t stage_bytes, ablock;  // ablock: bytes of one K block of the pair factors (rows padded to 8)
    const int4 *units;     // (M tile, first plane row, rows, warps of pairs) per unit
    const int2 *prow;      // [tiles][kM] staged rows (u, v) of each pair's factors, (-1, -1) for none
    const int *slots;      // [nunits][kM][kN] output slot or -1
    const int *mexp;       // FP16 form: per-map exponent e, map stored times 2^e (|M| 2^e <= 2^14)
    double *partial;       // [ksplit][nslots]
    int *err;              // set to 1 when a bounded wait gives up
    uint32_t wait_limit;   // polls of a main-loop wait (kWaitLimit unless a diagnostic limit is set)
};

// Tensor maps of one launch: the pair factors, and the B planes (16 bits: hi and lo in bh;
// TF32: in bh and bl) with boxes of 16, 32, 48 and 64 rows (a unit's window).
struct TmMaps {
    CUtensorMap a, bh[4], bl[4];
};

template <int F, bool D>
__global__ void __launch_bounds__(kThreads, 1)
    trisum_tm_kernel(const __grid_constant__ TmMaps tm, const TmArgs a) {
    using FM = Form<F>;
    constexpr int AST = FM::kAStages;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char *base =
        reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const int nst = a.nstages;
    // barriers: full per stage (TMA -> producers, MMA), sfree per stage (producers -> TMA),
    // prod per A stage (producers -> MMA), done per chunk ring (MMA completion -> TMA,
    // producers, drain), accfree per accumulator (drain -> MMA)
    // smem: nst stages | barriers and tables
    uint64_t *bars = reinterpret_cast<uint64_t *>(base + (size_t)nst * a.stage_bytes);
    uint64_t *full = bars, *sfree = full + kMaxStages, *prod = sfree + kMaxStages, *done = prod + kMaxAStages;
    uint64_t *accfree = done + kDone;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(accfree + kAcc);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    int2 *prow_s = reinterpret_cast<int2 *>(tmem_slot + 4);
    int *qexp_s = reinterpret_cast<int *>(prow_s + kM);  // [kN] FP16 exponent of each B row
    // running sums of the drain, then the compensation: TMEM columns kColK .. kColK + 2 kN
    // of the thread's lane
    constexpr uint32_t kColK = kColA + (uint32_t)AST * FM::kACols;

    const int unit = blockIdx.x % a.nunits, split = blockIdx.x / a.nunits;
    const int4 U = a.units[unit];
    const int q0 = U.y, ncols = U.z, nwp = U.w;  // nwp: warps (quadrants of 32 TMEM lanes) that hold pairs
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const long long cb = a.nchunks * split / a.ksplit, ce = a.nchunks * (split + 1) / a.ksplit;
    const int n = (int)(ce - cb);

    for (int r = tid; r < kM; r += kThreads) prow_s[r] = a.prow[(size_t)U.x * kM + r];
    for (int r = tid; r < kN; r += kThreads) {
        const int q = q0 + r, ns = a.nmaps / a.nb;  // plane row -> map
        qexp_s[r] = (F == kFormF16 && q < a.nmaps) ? a.mexp[(q % ns) * a.nb + q / ns] : 0;
    }
    if (tid == 0) {
        for (int s = 0; s < kMaxStages; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&sfree[s], nwp);  // the warpgroup's warps that consumed the stage's pair factors
        }
        for (int s = 0; s < kMaxAStages; s++) mbar_init(&prod[s], nwp);  // one warpgroup per chunk
        for (int s = 0; s < kDone; s++) mbar_init(&done[s], 1);
        for (int s = 0; s < kAcc; s++) mbar_init(&accfree[s], kDrainWarps / 4 * nwp);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        tmem_alloc(tmem_slot, kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    // stage: pair-factor blocks [kBlocks][ablock] (FP32, 32 points a row) | B tiles [kBTiles][rows 128]
    auto stage_ptr = [&](int s) { return base + (size_t)s * a.stage_bytes; };
    auto fail = [&]() {
        *abort_flag = 1;
        atomicExch(a.err, 1);
    };

    if (warp < kProdWarps) {
        // ------------------------------------------------------------ producers
        // (the TMEM rows of quadrants without pairs are never written: their products
        // stay in rows that no slot reads)
        const int quad = warp & 3, grp = warp >> 2;
        const uint32_t lane_addr = tmem + ((uint32_t)(quad * 32) << 16);
        // TF32: thread = row; 16-bit forms: thread = 4 rows (lane / 4 + 8 k) that share the
        // map v, and 4 points of each 16 (lane % 4)
        const int row = quad * 32 + (F == kFormTF32 ? lane : lane >> 2);
        const int2 pr = prow_s[row];
        uint32_t uo[4], vo = 0;  // byte offsets of the thread's first points in a K block
        if constexpr (F != kFormTF32) {
            auto off = [&](int r) { return (uint32_t)(r * 128 + (((lane & 3) ^ (r & 7)) << 4)); };
            vo = off(max(pr.y, 0));
#pragma unroll
            for (int k = 0; k < 4; k++) uo[k] = off(max(prow_s[row + 8 * k].x, 0));
        }
        Ring rs(grp, nst);  // stage and full-barrier phase of chunk i
        for (int i = quad < nwp ? grp : n; i < n; i += kGroups, rs.step(kGroups, nst)) {
            const int s = rs.idx, as = i % AST;
            if (!warp_wait<D>(&full[s], (uint32_t)rs.phase, abort_flag, a.wait_limit)) { fail(); break; }
            // the A stage is free once the MMAs of chunk i - AST completed (MMAs complete in order)
            if (i >= AST && !warp_wait<D>(&done[(i - AST) % kDone], ph(i - AST, kDone), abort_flag, a.wait_limit)) {
                fail();
                break;
            }
            const unsigned char *stg = stage_ptr(s);
            const uint32_t acol = kColA + (uint32_t)as * FM::kACols;
#pragma unroll 1  // (unrolled, its loads do not fit in the registers: spills go to L2 beside 227 KB of shared memory)
            for (int kb = 0; kb < kBlocks; kb++) {
                const unsigned char *blk = stg + kb * a.ablock;
                if constexpr (F == kFormTF32) {
#pragma unroll
                    for (int q8 = 0; q8 < 4; q8++) {
                        uint32_t hi[8], lo[8];
                        if (pr.x >= 0) {
#pragma unroll
                            for (int c4 = 0; c4 < 2; c4++) {
                                const int c = 2 * q8 + c4;
                                const float4 u =
                                    *reinterpret_cast<const float4 *>(blk + pr.x * 128 + ((c ^ (pr.x & 7)) << 4));
                                const float4 v =
                                    *reinterpret_cast<const float4 *>(blk + pr.y * 128 + ((c ^ (pr.y & 7)) << 4));
                                const float2 p01 = __fmul2_rn(make_float2(u.x, u.y), make_float2(v.x, v.y));
                                const float2 p23 = __fmul2_rn(make_float2(u.z, u.w), make_float2(v.z, v.w));
                                const float2 h01 = make_float2(__uint_as_float(__float_as_uint(p01.x) & kTfMask),
                                                               __uint_as_float(__float_as_uint(p01.y) & kTfMask));
                                const float2 h23 = make_float2(__uint_as_float(__float_as_uint(p23.x) & kTfMask),
                                                               __uint_as_float(__float_as_uint(p23.y) & kTfMask));
                                const float2 l01 = __fadd2_rn(p01, make_float2(-h01.x, -h01.y));
                                const float2 l23 = __fadd2_rn(p23, make_float2(-h23.x, -h23.y));
                                hi[4 * c4 + 0] = __float_as_uint(h01.x);
                                hi[4 * c4 + 1] = __float_as_uint(h01.y);
                                hi[4 * c4 + 2] = __float_as_uint(h23.x);
                                hi[4 * c4 + 3] = __float_as_uint(h23.y);
                                lo[4 * c4 + 0] = __float_as_uint(l01.x);
                                lo[4 * c4 + 1] = __float_as_uint(l01.y);
                                lo[4 * c4 + 2] = __float_as_uint(l23.x);
                                lo[4 * c4 + 3] = __float_as_uint(l23.y);
                            }
                        } else {
#pragma unroll
                            for (int e = 0; e < 8; e++) hi[e] = lo[e] = 0u;
                        }
                        const uint32_t col = acol + (uint32_t)(kb * kKB + 8 * q8);
                        tmem_st8(lane_addr + col, hi);
                        tmem_st8(lane_addr + col + kKC, lo);
                    }
                } else {
                    // 32 points -> 16 packed columns (points 2c, 2c + 1 in column c).  Column
                    // block n holds the points 16 n + 4 t .. of lane % 4 = t in columns
                    // 8 n + 2 t, 8 n + 2 t + 1: one 16-byte load a row (XOR 64: the next 16
                    // points under the swizzle), the shared map's loaded once for four rows.
                    const float4 v0 = *reinterpret_cast<const float4 *>(blk + vo);
                    const float4 v1 = *reinterpret_cast<const float4 *>(blk + (vo ^ 64));
                    const uint32_t col = lane_addr + acol + (uint32_t)(kb * (kKB / 2));
#pragma unroll
                    for (int h = 0; h < 2; h++) {  // lanes 0-15, 16-31 of the quadrant: rows k = 2 h, 2 h + 1
                        uint32_t hi[8], lo[8];
#pragma unroll
                        for (int k = 0; k < 2; k++) {
                            const float4 u0 = *reinterpret_cast<const float4 *>(blk + uo[2 * h + k]);
                            const float4 u1 = *reinterpret_cast<const float4 *>(blk + (uo[2 * h + k] ^ 64));
                            pack_prod2<F>(u0.x, v0.x, u0.y, v0.y, hi[2 * k], lo[2 * k]);
                            pack_prod2<F>(u0.z, v0.z, u0.w, v0.w, hi[2 * k + 1], lo[2 * k + 1]);
                            pack_prod2<F>(u1.x, v1.x, u1.y, v1.y, hi[4 + 2 * k], lo[4 + 2 * k]);
                            pack_prod2<F>(u1.z, v1.z, u1.w, v1.w, hi[5 + 2 * k], lo[5 + 2 * k]);
                        }
                        tmem_st_16x256b_x2(col + ((uint32_t)(16 * h) << 16), hi);
                        if (FM::kSplit) tmem_st_16x256b_x2(col + ((uint32_t)(16 * h) << 16) + kKC / 2, lo);
                    }
                }
            }
            __syncwarp();  // one arrival a warp on each barrier
            if (lane == 0) mbar_arrive(&sfree[s]);  // the stage's pair factors are consumed
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&prod[as]);
        }
    } else if (warp < kMmaWarp) {
        // ---------------------------------------------------------------- drain
        // each chunk's accumulator is added into FP32 registers (round to nearest);
        // every kFold chunks those are folded into a Kahan-compensated sum in TMEM, written out
        // at the end
        // (the two warpgroups take half of the unit's columns each, in groups of 8)
        const int quad = warp & 3, cgrp = (warp - kProdWarps) >> 2;
        // NG: groups of 8 columns per warpgroup (a unit of 16 NG columns)
        auto drain = [&](auto ng) {
        constexpr int NG = decltype(ng)::value;
        const int row = quad * 32 + lane, c0 = 8 * NG * cgrp;
        const uint32_t lane_addr = tmem + ((uint32_t)(quad * 32) << 16);
        const uint32_t krun = lane_addr + kColK + (uint32_t)c0, kcomp = krun + kN;
        float mid[8 * NG];
#pragma unroll
        for (int e = 0; e < 8 * NG; e++) mid[e] = 0.f;
        {
            const uint32_t z[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
#pragma unroll
            for (int h = 0; h < 8 * NG; h += 8) {
                tmem_st8(krun + h, z);
                tmem_st8(kcomp + h, z);
            }
            tmem_wait_st();
        }
        bool ok = true;
#pragma unroll 1
        for (int i = 0; i < n; i++) {
            const int b = i % kAcc;
            if (!warp_wait<D>(&done[i % kDone], ph(i, kDone), abort_flag, a.wait_limit)) { fail(); ok = false; break; }
            tc_fence_after();
            const uint32_t src = lane_addr + kColAcc + (uint32_t)b * kN + c0;
#pragma unroll
            for (int h = 0; h < NG; h += 2) {
                uint32_t ac[8], ad[8];
                tmem_ld8(src + 8 * h, ac);
                if (h + 1 < NG) tmem_ld8(src + 8 * h + 8, ad);
                tmem_wait_ld();
#pragma unroll
                for (int e = 0; e < 8; e++) mid[8 * h + e] += __uint_as_float(ac[e]);
                if (h + 1 < NG) {
#pragma unroll
                    for (int e = 0; e < 8; e++) mid[(8 * h + 8 + e) % (8 * NG)] += __uint_as_float(ad[e]);
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&accfree[b]);
            if ((i + 1) % kFold == 0 || i == n - 1) {
#pragma unroll
                for (int h = 0; h < 8 * NG; h += 8) {
                    uint32_t rr[8], cc[8];
                    tmem_ld8(krun + h, rr);
                    tmem_ld8(kcomp + h, cc);
                    tmem_wait_ld();
#pragma unroll
                    for (int e = 0; e < 8; e++) {
                        const float rv = __uint_as_float(rr[e]), y = mid[h + e] - __uint_as_float(cc[e]);
                        const float t2 = rv + y;
                        cc[e] = __float_as_uint((t2 - rv) - y);
                        rr[e] = __float_as_uint(t2);
                        mid[h + e] = 0.f;
                    }
                    tmem_st8(krun + h, rr);
                    tmem_st8(kcomp + h, cc);
                }
                tmem_wait_st();  // the next fold reads these columns back
            }
        }
        if (__all_sync(0xffffffffu, ok && !*abort_flag)) {
            const int *sl = a.slots + ((size_t)unit * kM + row) * kN;
            const int2 pr = prow_s[row];
            const int pe = (F == kFormF16 && pr.x >= 0) ? a.mexp[pr.x] + a.mexp[pr.y] - 14 : 0;
#pragma unroll 1
            for (int h = 0; h < 8 * NG; h += 8) {
                uint32_t rr[8], cc[8];
                tmem_ld8(krun + h, rr);
                tmem_ld8(kcomp + h, cc);
                tmem_wait_ld();
#pragma unroll
                for (int e = 0; e < 8; e++) {
                    const int slot = sl[c0 + h + e];
                    if (slot < 0) continue;
                    const double v = (double)__uint_as_float(rr[e]) - (double)__uint_as_float(cc[e]);
                    a.partial[(size_t)split * a.nslots + slot] =
                        F == kFormF16 ? ldexp(v, -(pe + qexp_s[c0 + h + e])) : v;
                }
            }
        }
        };
        if (quad < nwp) {
            if (ncols == 64) drain(std::integral_constant<int, 4>{});
            else if (ncols == 48) drain(std::integral_constant<int, 3>{});
            else if (ncols == 32) drain(std::integral_constant<int, 2>{});
            else drain(std::integral_constant<int, 1>{});
        }
    } else if (warp < kTmaWarp) {
        // ------------------------------------------ MMA issue (one thread per MMA warp)
        // issuer w takes chunks w, w + kMmaWarps, ...: each chunk has its own
        // accumulator, A stage and completion barrier, and tcgen05.commit tracks the
        // issuing thread's own MMAs, so the two streams need no ordering between them
        if (lane == 0) {
            const int mw = warp - kMmaWarp;
            int last_commit = -1;
            bool ok = true;
            const uint32_t idesc = FM::kIdesc | idesc_n(ncols), btile = (uint32_t)ncols * 128;
            Ring rs(mw, nst);
            for (int i = mw; i < n; i += kMmaWarps, rs.step(kMmaWarps, nst)) {
                const int b = i % kAcc, as = i % AST, s = rs.idx;
                if (i >= kAcc && !wait_or_abort<D>(&accfree[b], ph(i - kAcc, kAcc), abort_flag, a.wait_limit)) { ok = false; break; }
                if (!wait_or_abort<D>(&full[s], (uint32_t)rs.phase, abort_flag, a.wait_limit)) { ok = false; break; }  // B tiles
                if (!wait_or_abort<D>(&prod[as], ph(i, AST), abort_flag, a.wait_limit)) { ok = false; break; }  // A stage
                tc_fence_after();
                // descriptors advance by 16-byte units within the stage (no carry out of the address field)
                const uint64_t db = sw128_desc(smem_u32(stage_ptr(s)) + kBlocks * a.ablock);
                const uint32_t ahi = tmem + kColA + (uint32_t)as * FM::kACols;
                const uint32_t d = tmem + kColAcc + (uint32_t)b * kN;
#pragma unroll
                for (int kk = 0; kk < kKC / FM::kKStep; kk++) {
                    uint64_t dh, dl;
                    uint32_t a_hi, a_lo;
                    if constexpr (F == kFormTF32) {
                        // FP32 rows: K-step of 8 = 32 bytes; tiles hi0, hi1, lo0, lo1
                        dh = db + (((uint32_t)(kk / 4) * btile + (uint32_t)(kk % 4) * 32) >> 4);
                        dl = dh + ((2 * btile) >> 4);
                        a_hi = ahi + 8 * kk;
                        a_lo = a_hi + kKC;
                    } else {
                        // 16-bit rows: K-step of 16 = 32 bytes; tiles hi, lo
                        dh = db + (uint32_t)kk * 2;
                        dl = dh + (btile >> 4);
                        a_hi = ahi + 8 * kk;
                        a_lo = a_hi + kKC / 2;
                    }
                    umma_ta<F>(d, a_hi, dh, idesc, kk == 0 ? 0u : 1u);
                    if (FM::kSplit) {
                        umma_ta<F>(d, a_hi, dl, idesc, 1u);
                        umma_ta<F>(d, a_lo, dh, idesc, 1u);
                    }
                }
                umma_commit(&done[i % kDone]);
                last_commit = i;
            }
            if (!ok) fail();
            // this thread's MMAs still in flight (and their barrier arrival) land before TMEM goes away
            if (last_commit >= 0) mbar_wait(&done[last_commit % kDone], ph(last_commit, kDone));
        }
    } else if (lane == 0) {
        // --------------------------------------------------------- TMA issue (one thread)
        const uint32_t tx = kBlocks * a.ablock + FM::kBTiles * (uint32_t)ncols * 128;
        const CUtensorMap *tmBh = &tm.bh[ncols / 16 - 1], *tmBl = &tm.bl[ncols / 16 - 1];
        int issued = 0;
        bool ok = true;
        Ring rs(0, nst);
        for (int j = 0; j < n; j++, rs.step(1, nst)) {
            const int s = rs.idx;
            // stage s is free once the producers took the pair factors of chunk j - nst
            // (the ring's previous phase) and the MMAs of that chunk (which read its B
            // tiles) completed
            if (j >= nst && (!wait_or_abort<D>(&sfree[s], (uint32_t)(rs.phase ^ 1), abort_flag, a.wait_limit) ||
                             !wait_or_abort<D>(&done[(j - nst) % kDone], ph(j - nst, kDone), abort_flag, a.wait_limit))) {
                ok = false;
                break;
            }
            unsigned char *stg = stage_ptr(s);
            unsigned char *bt = stg + kBlocks * a.ablock;
            mbar_expect_tx(&full[s], tx);
            const int c = (int)(cb + j);  // chunk: 64 consecutive points, one block of every plane
            tma_load_chunk(stg, &tm.a, 0, c, &full[s]);
            tma_load_chunk(bt, tmBh, q0, c, &full[s]);  // 16 bits: hi, and lo after it
            if (F == kFormTF32) tma_load_chunk(bt + 2 * ncols * 128, tmBl, q0, c, &full[s]);
            issued = j + 1;
        }
        if (!ok) fail();
        // copies in flight land (bounded) before the shared memory goes away: after an
        // abort of any role, and (already complete, so at once) at a normal end
        for (int j = std::max(0, issued - nst); j < issued; j++) mbar_wait(&full[j % nst], ph(j, nst));
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, kTmemCols);
    }
}

// Per-map power-of-two scale of the FP16 form: |M(x)| <= sum_k |H(k)| <=
// sqrt(nmodes * sum_k |H(k)|^2) (triangle and Cauchy-Schwarz inequalities over
// the shell's modes).  Sets without their own power use the delta set's times
// max |L_l(mu)| (lfac).
__global__ void map_exponents_kernel(int nmaps, int nb, const double *__restrict__ powsum, int pow_mask,
                                     double lf1, double lf2, const double *__restrict__ nmodes, int *__restrict__ e) {
    for (int m = threadIdx.x; m < nmaps; m += blockDim.x) {
        const int s = m / nb, b = m % nb;
        const double p = (pow_mask >> s & 1) ? powsum[s * nb + b] : powsum[b];
        const double lf = s == 0 ? 1.0 : (s == 1 ? lf1 : lf2);
        const double v = sqrt(nmodes[b] * p) * ((pow_mask >> s & 1) ? 1.0 : lf);
        // scale so that |M| 2^e <= 2^14, clamped to the float exponent range
        int x = v > 0 ? 14 - (int)ceil(log2(v)) : 0;
        e[m] = x < -60 ? -60 : (x > 60 ? 60 : x);
    }
}

// ------------------------------------------------------------- tensor maps ---
using EncodeTiledFn = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                   const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
    static std::once_flag once;
    static EncodeTiledFn fn = nullptr;
    std::call_once(once, [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    });
    return fn;
}

// 4D view of chunk-major operand arrays [nchunks][rows][64 points] (element size esize): a
// box is (128 bytes of points, box_rows rows, all `nblk` blocks, one chunk), 128-byte swizzle
// (the K-major operand layout), one block after the other in shared memory.  The blocks are
// the 128-byte point blocks of the rows (FP32: two, 128 bytes apart) or the hi and lo planes
// (16 bits: `blk_stride` bytes apart), so that one instruction loads a whole operand: the
// issuing thread's loads bounded the chunk loop at four a chunk.  Rows past the last one are
// filled with zeros.
int make_chunk_view(CUtensorMap *tm, const void *base, CUtensorMapDataType dt, int esize, long long nchunks,
                    int rows, int box_rows, int nblk, size_t blk_stride) {
    EncodeTiledFn enc = encode_fn();
    if (!enc) return set_error(PBI4G_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    if (reinterpret_cast<uintptr_t>(base) % 16 || blk_stride % 16)
        return set_error(PBI4G_ERR_INVALID, "operand chunk view: alignment");
    const size_t row_bytes = (size_t)MapPlanes::kChunk * esize;
    const cuuint64_t gdim[4] = {(cuuint64_t)(128 / esize), (cuuint64_t)rows, (cuuint64_t)nblk, (cuuint64_t)nchunks};
    const cuuint64_t gstride[3] = {row_bytes, blk_stride, (cuuint64_t)rows * row_bytes};
    const cuuint32_t box[4] = {(cuuint32_t)(128 / esize), (cuuint32_t)box_rows, (cuuint32_t)nblk, 1};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    const CUresult r = enc(tm, dt, 4, const_cast<void *>(base), gdim, gstride, box, estr,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return set_error(PBI4G_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
    return PBI4G_OK;
}

}  // namespace

// ------------------------------------------------------------- host plan ---
// Pairs of shells (x <= y) that hold every triangle of an equal-set contraction.  With one q
// set the three factors of a triangle are alike, so any of its three pairs may be the A row
// and the third shell the B row: the fewest pairs that meet every triangle are wanted.
// Splitting the shells at `a` and keeping the pairs inside each part covers every triangle
// (two of three shells fall in one part); of those, pairs that no triangle needs are left out,
// the triangles inside a part are covered greedily, and redundant pairs are dropped.  The best
// `a` is taken: 48 shells need 489 pairs of 1176, 24 need 133 of 300.
static std::vector<std::pair<int, int>> covering_pairs(const Shells &sh) {
    const int nb = sh.nb, np = nb * (nb + 1) / 2;
    const size_t nt = (size_t)sh.itot;
    auto id = [](int x, int y) { return x <= y ? y * (y + 1) / 2 + x : x * (x + 1) / 2 + y; };
    std::vector<std::vector<int>> of(np);
    std::vector<int> edge(3 * nt);
    for (size_t t = 0; t < nt; t++) {
        const int l = sh.tri[3 * t] - 1, j = sh.tri[3 * t + 1] - 1, i = sh.tri[3 * t + 2] - 1;
        int e[3] = {id(i, j), id(i, l), id(j, l)};
        for (int k = 0; k < 3; k++) {
            edge[3 * t + k] = e[k];
            bool seen = false;
            for (int m = 0; m < k; m++) seen |= e[m] == e[k];
            if (!seen) of[e[k]].push_back((int)t);
        }
    }
    std::vector<char> best;
    int nbest = 1 << 30;
    std::vector<int> by_size(np);
    for (int e = 0; e < np; e++) by_size[e] = e;
    std::stable_sort(by_size.begin(), by_size.end(), [&](int x, int y) { return of[x].size() < of[y].size(); });
    // splits tried: all of [0, 0.6 nb) for few shells, at least three for many (0.6 s at 256)
    const int amax = std::max(1, (int)(0.6 * nb)),
              ntry = (int)std::min<long long>(amax, std::max<long long>(3, 400000 / std::max<int64_t>(1, sh.itot)));
    for (int k = 0; k < ntry; k++) {
        const int a = ntry == amax ? k : (int)((0.2 + 0.4 * k / std::max(1, ntry - 1)) * nb);
        std::vector<char> keep(np, 0);
        std::vector<int> cov(nt, 0), cnt(np, 0);
        for (size_t t = 0; t < nt; t++) {
            const int l = sh.tri[3 * t] - 1, j = sh.tri[3 * t + 1] - 1, i = sh.tri[3 * t + 2] - 1;
            if (i < a && j < a && l >= a) keep[id(i, j)] = 1;  // i <= j <= l: two low, one high
            if (i < a && j >= a) keep[id(j, l)] = 1;           // one low, two high
        }
        for (int e = 0; e < np; e++)
            if (keep[e])
                for (int t : of[e]) cov[t]++;
        // greedy cover of the rest: the pair that meets most uncovered triangles next (counts
        // only fall, so a stale entry of the queue is pushed back with its present count)
        std::priority_queue<std::pair<int, int>> queue;
        for (int e = 0; e < np; e++) {
            for (int t : of[e]) cnt[e] += cov[t] == 0;
            if (!keep[e] && cnt[e] > 0) queue.push({cnt[e], -e});
        }
        while (!queue.empty()) {
            const auto [c, ne] = queue.top();
            const int b = -ne;
            queue.pop();
            if (cnt[b] <= 0) continue;
            if (cnt[b] < c) {
                queue.push({cnt[b], -b});
                continue;
            }
            keep[b] = 1;
            for (int t : of[b])
                if (cov[t]++ == 0)
                    for (int k3 = 0; k3 < 3; k3++) {
                        const int e = edge[3 * (size_t)t + k3];
                        bool seen = false;
                        for (int m = 0; m < k3; m++) seen |= edge[3 * (size_t)t + m] == e;
                        if (!seen) cnt[e]--;
                    }
        }
        int n = 0;
        for (int e : by_size) {
            if (!keep[e]) continue;
            bool need = false;
            for (int t : of[e]) need |= cov[t] == 1;
            if (need) {
                n++;
                continue;
            }
            keep[e] = 0;
            for (int t : of[e]) cov[t]--;
        }
        if (n < nbest) {
            nbest = n;
            best = keep;
        }
    }
    std::vector<std::pair<int, int>> out;
    for (int y = 0; y < nb; y++)
        for (int x = 0; x <= y; x++)
            if (best[id(x, y)]) out.push_back({x, y});
    return out;
}

int TmPlan::build(const Shells &sh, int nsets_) {
    nsets = nsets_;
    const int nb = sh.nb;
    nA = nb;
    nslots = (int)(sh.itot * nsets);
    // the plane rows and slots of each pair (x <= y): its triangles
    struct E { int q, slot; };
    std::map<std::pair<int, int>, std::vector<E>> ent;
    if (nsets == 1)
        for (auto &p : covering_pairs(sh)) ent[p];
    for (int64_t m = 0; m < sh.itot; m++) {
        const int l = sh.tri[3 * m] - 1, j = sh.tri[3 * m + 1] - 1, i = sh.tri[3 * m + 2] - 1;
        if (nsets == 1) {
            const int c[3][3] = {{i, j, l}, {i, l, j}, {j, l, i}};
            for (auto &t : c) {
                auto it = ent.find({t[0], t[1]});
                if (it == ent.end()) continue;
                it->second.push_back({t[2], (int)m});
                break;
            }
        } else {
            for (int s = 0; s < nsets; s++) ent[{i, j}].push_back({l * nsets + s, (int)(m * nsets + s)});
        }
    }
    for (auto it = ent.begin(); it != ent.end();) it = it->second.empty() ? ent.erase(it) : std::next(it);
    npairs = (int)ent.size();
    // Groups of four pairs that share a map v: every pair belongs to one of its two maps, the
    // larger one at first.  From the last map down, the pairs that do not fill a group of
    // four are handed to their other map (the smallest first, so that neighbouring v give
    // theirs to the same one): nearly all groups come out full.
    std::vector<std::vector<int>> own(nb);  // v -> maps u
    for (auto &kv : ent) own[kv.first.second].push_back(kv.first.first);
    struct G { int v, u[4], n, lo, hi; };
    std::vector<G> groups;
    for (int v = nb - 1; v >= 0; v--) {
        std::sort(own[v].begin(), own[v].end());
        size_t rest = own[v].size() % 4, k = 0;
        std::vector<int> mine;
        for (; k < own[v].size(); k++) {
            const int u = own[v][k];
            if (rest > 0 && u < v) {  // to a map that is still to come
                own[u].push_back(v);
                rest--;
            } else {
                mine.push_back(u);
            }
        }
        std::sort(mine.begin(), mine.end());
        for (size_t m = mine.size(); m > 0;) {  // from the largest down: what is left over is small
            G g = {v, {-1, -1, -1, -1}, 0, 1 << 30, -1};
            for (; g.n < 4 && m > 0; m--) {
                const int u = mine[m - 1];
                g.u[g.n++] = u;
                for (auto &e : ent[{std::min(u, v), std::max(u, v)}]) {
                    g.lo = std::min(g.lo, e.q);
                    g.hi = std::max(g.hi, e.q);
                }
            }
            groups.push_back(g);
        }
    }
    // M tiles: the groups in an order that keeps each tile's range of plane rows short, their
    // warps (8 groups) spread evenly; units: windows of up to 64 rows of a tile's range.  The
    // order with the least cost is taken (a unit's cost per chunk: a fixed part and its rows).
    const int nw = ((int)groups.size() + 7) / 8, nt = (nw + 3) / 4;
    auto first_group = [&](int t) { return std::min((int)groups.size(), 8 * (int)((long long)nw * t / nt)); };
    struct U { int t, q, n; };
    auto layout = [&](const std::vector<G> &gs, std::vector<U> &us) {
        int cost = 0;
        us.clear();
        for (int t = 0; t < nt; t++) {
            std::vector<char> used((size_t)nsets * nb + 1, 0);
            for (int g = first_group(t); g < first_group(t + 1); g++)
                for (int k = 0; k < gs[g].n; k++)
                    for (auto &e : ent[{std::min(gs[g].u[k], gs[g].v), std::max(gs[g].u[k], gs[g].v)}]) used[e.q] = 1;
            for (int q = 0; q < nsets * nb;) {
                if (!used[q]) {
                    q++;
                    continue;
                }
                int last = q;
                for (int r = q; r < std::min(q + kN, nsets * nb); r++)
                    if (used[r]) last = r;
                const int n = (last - q + 16) / 16 * 16;
                us.push_back({t, q, n});
                cost += 96 + n;
                q = last + 1;
            }
        }
        return cost;
    };
    std::vector<G> gbest;
    std::vector<U> ubest, utry;
    int cbest = 1 << 30;
    for (int key = 0; key < 4; key++) {
        std::vector<G> gs = groups;
        std::stable_sort(gs.begin(), gs.end(), [key](const G &a, const G &b) {
            if (key == 0) return a.lo != b.lo ? a.lo < b.lo : a.hi < b.hi;
            if (key == 1) return a.hi != b.hi ? a.hi < b.hi : a.lo < b.lo;
            if (key == 2) return a.lo + a.hi < b.lo + b.hi;
            return a.v != b.v ? a.v < b.v : a.u[0] < b.u[0];
        });
        const int c = layout(gs, utry);
        if (c < cbest) {
            cbest = c;
            gbest = gs;
            ubest = utry;
        }
    }
    ntiles = nt;
    // Rows of a warp: group g takes the TMEM lanes g + 8 k.  Two neighbouring groups read
    // their maps' rows in one shared-memory phase; rows r and r' fall on the same banks when
    // bit 2 of both is the same (128-byte swizzle), so groups are paired, and their maps
    // ordered, to have it differ.
    std::vector<int2> h_prow((size_t)std::max(1, nt) * kM, make_int2(-1, -1));
    std::map<std::pair<int, int>, std::pair<int, int>> at;  // pair -> (tile, row)
    for (int t = 0; t < nt; t++) {
        std::vector<G> gs(gbest.begin() + first_group(t), gbest.begin() + first_group(t + 1));
        auto ones = [](const G &g) {
            int c = 0;
            for (int k = 0; k < g.n; k++) c += g.u[k] >> 2 & 1;
            return c;
        };
        std::stable_sort(gs.begin(), gs.end(), [&](const G &a, const G &b) { return ones(a) < ones(b); });
        std::vector<G> order;
        for (size_t lo = 0, hi = gs.size(); lo < hi;) {
            order.push_back(gs[lo++]);
            if (lo < hi) order.push_back(gs[--hi]);
        }
        for (size_t g = 0; g < order.size(); g++) {
            G &o = order[g];
            std::stable_sort(o.u, o.u + o.n, [g](int a, int b) {
                const int x = a >> 2 & 1, y = b >> 2 & 1;
                return g % 2 ? x > y : x < y;
            });
            for (int k = 0; k < 4; k++) {
                const int row = (int)(g / 8) * 32 + (int)(g % 8) + 8 * k;
                // rows of a short group repeat its shared map (their products go nowhere)
                h_prow[(size_t)t * kM + row] = make_int2(k < o.n ? o.u[k] : o.v, o.v);
                if (k < o.n) at[{std::min(o.u[k], o.v), std::max(o.u[k], o.v)}] = {t, row};
            }
        }
    }
    // the units of one K range are adjacent in the grid
    nunits = (int)ubest.size();
    std::vector<int4> h_units;
    std::vector<int> h_slots((size_t)std::max(1, nunits) * kM * kN, -1);
    max_cols = 16;
    for (auto &u : ubest) {
        h_units.push_back(make_int4(u.t, u.q, u.n, nw * (u.t + 1) / nt - nw * u.t / nt));
        max_cols = std::max(max_cols, u.n);
    }
    std::vector<int> first_unit(nt + 1, 0);  // (the units of a tile are consecutive)
    for (int u = 0; u < nunits; u++) first_unit[ubest[u].t + 1] = u + 1;
    for (auto &kv : ent) {
        const auto [t, row] = at.at(kv.first);
        for (auto &e : kv.second)
            for (int u = first_unit[t]; u < first_unit[t + 1]; u++)
                if (e.q >= ubest[u].q && e.q < ubest[u].q + ubest[u].n) {
                    h_slots[((size_t)u * kM + row) * kN + e.q - ubest[u].q] = e.slot;
                    break;
                }
    }
    PBI4G_CHECK(units.ensure(sizeof(int4) * std::max(1, nunits)));
    PBI4G_CHECK(prow.ensure(sizeof(int2) * h_prow.size()));
    PBI4G_CHECK(slots.ensure(sizeof(int) * h_slots.size()));
    PBI4G_CHECK(err.ensure(sizeof(int)));
    if (nunits) {
        PBI4G_CUDA(cudaMemcpy(units.p, h_units.data(), sizeof(int4) * h_units.size(), cudaMemcpyHostToDevice));
        PBI4G_CUDA(cudaMemcpy(prow.p, h_prow.data(), sizeof(int2) * h_prow.size(), cudaMemcpyHostToDevice));
        PBI4G_CUDA(cudaMemcpy(slots.p, h_slots.data(), sizeof(int) * h_slots.size(), cudaMemcpyHostToDevice));
    }
    return PBI4G_OK;
}

bool tm_supported(const Shells &sh) {
    const long long npts = (long long)sh.Nm * sh.Nm * sh.Nm;
    return sh.nb <= 256 && sh.Nm % 4 == 0 && npts + kKC < (1LL << 31);
}

template <int F>
static int launch_tm(const TmMaps &tm, const TmArgs &a, size_t smem, int grid, cudaStream_t st) {
    auto kern = a.wait_limit < kWaitLimit ? trisum_tm_kernel<F, true> : trisum_tm_kernel<F, false>;
    PBI4G_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kern<<<grid, kThreads, smem, st>>>(tm, a);
    PBI4G_LAUNCH_CHECK();
    return PBI4G_OK;
}

int tm_map_exponents(const Shells &sh, TmPlan &tp, int nmaps, const double *powsum, int pow_mask,
                     const double lfac[3], cudaStream_t st, int64_t *launches) {
    PBI4G_CHECK(tp.mexp.ensure(sizeof(int) * std::max(1, nmaps)));
    map_exponents_kernel<<<1, 256, 0, st>>>(nmaps, sh.nb, powsum, pow_mask, lfac[1], lfac[2],
                                            sh.nmodes_d.as<double>(), tp.mexp.as<int>());
    PBI4G_LAUNCH_CHECK();
    *launches += 1;
    return PBI4G_OK;
}

int triangle_sums_tm(const Shells &sh, TmPlan &tp, const MapPlanes &pl, DevBuf &partial, double *S,
                     bool accumulate, cudaStream_t st, int64_t *launches) {
    const int form = pl.form;
    if (!tm_supported(sh))
        return set_error(PBI4G_ERR_UNSUPPORTED, "tensor-core triangle sums: map grid %d, %d shells", sh.Nm, sh.nb);
    if (form < 0 || form > 2) return set_error(PBI4G_ERR_INVALID, "tensor-core form %d", form);
    if (tp.nunits == 0) return PBI4G_OK;
    if (form == 1 && (!pl.mexp || pl.mexp != tp.mexp.as<int>()))
        return set_error(PBI4G_ERR_INVALID, "tensor-core triangle sums: FP16 planes without the plan's exponents");
    if (pl.nb != sh.nb || pl.npts < kKC || pl.npts > (long long)sh.Nm * sh.Nm * sh.Nm || pl.nchunks * kKC != pl.npts)
        return set_error(PBI4G_ERR_INVALID, "tensor-core triangle sums: operand planes do not match the shells");
    static_assert(MapPlanes::kChunk == kKC, "a planes chunk is a contraction chunk");
    TmMaps tm;
    const long long nc = pl.nchunks;
    const int arows = (tp.nA + 7) / 8 * 8;
    PBI4G_CHECK(make_chunk_view(&tm.a, pl.a32, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, nc, sh.nb, arows, kBlocks, 128));
    for (int b = 0; b < 4; b++) {
        const int n = 16 * (b + 1);
        if (form == 0) {
            PBI4G_CHECK(make_chunk_view(&tm.bh[b], pl.bhi, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, nc, pl.nmaps, n,
                                        kBlocks, 128));
            PBI4G_CHECK(make_chunk_view(&tm.bl[b], pl.blo, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, nc, pl.nmaps, n,
                                        kBlocks, 128));
        } else {
            const size_t lo = form == 1 ? (size_t)((const char *)pl.blo - (const char *)pl.bhi) : 0;
            PBI4G_CHECK(make_chunk_view(&tm.bh[b], pl.bhi,
                                        form == 1 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16,
                                        2, nc, pl.nmaps, n, form == 1 ? 2 : 1, form == 1 ? lo : 128));
            tm.bl[b] = tm.bh[b];  // unused
        }
    }
    TmArgs a;
    a.nchunks = nc;
    a.nunits = tp.nunits;
    // K split: one CTA per SM (152 SMs) in waves; the split minimising waves x
    // (chunks a CTA + a CTA's fixed cost of about 64 chunks), at least 128 chunks a CTA
    {
        long long best_cost = -1;
        a.ksplit = 1;
        for (int k = 1; k <= 152; k++) {
            if (k > 1 && a.nchunks / k < 128) break;
            const long long waves = ((long long)tp.nunits * k + 151) / 152;
            const long long cost = waves * ((a.nchunks + k - 1) / k + 64);
            if (best_cost < 0 || cost < best_cost) {
                best_cost = cost;
                a.ksplit = k;
            }
        }
    }
    a.nslots = tp.nslots;
    a.nA = tp.nA;
    a.nmaps = pl.nmaps;
    a.nb = pl.nb;
    a.ablock = (uint32_t)arows * 128;
    const int btiles = form == 0 ? Form<kFormTF32>::kBTiles : (form == 1 ? Form<kFormF16>::kBTiles : 1);
    a.stage_bytes = kBlocks * a.ablock + (uint32_t)btiles * (uint32_t)tp.max_cols * 128;
    // barriers, TMEM address, abort flag, pair table, B-row exponents
    const size_t fixed =
        1024 + 8 * (2 * kMaxStages + kMaxAStages + kDone + kAcc) + 16 + sizeof(int2) * kM + sizeof(int) * kN;
    a.nstages = kMaxStages;
    while (a.nstages > 3 && fixed + (size_t)a.nstages * a.stage_bytes > 227 * 1024) a.nstages--;
    const size_t smem = fixed + (size_t)a.nstages * a.stage_bytes;
    if (smem > 227 * 1024) return set_error(PBI4G_ERR_UNSUPPORTED, "tensor-core triangle sums: %zu B smem", smem);
    a.units = tp.units.as<int4>();
    a.prow = tp.prow.as<int2>();
    a.slots = tp.slots.as<int>();
    PBI4G_CHECK(tp.mexp.ensure(sizeof(int) * std::max(1, pl.nmaps)));
    a.mexp = tp.mexp.as<int>();
    PBI4G_CHECK(partial.ensure(sizeof(double) * (size_t)a.ksplit * tp.nslots));
    a.partial = partial.as<double>();
    a.err = tp.err.as<int>();
    a.wait_limit = tp.wait_limit > 0 && tp.wait_limit < kWaitLimit ? tp.wait_limit : kWaitLimit;
    PBI4G_CUDA(cudaMemsetAsync(tp.err.p, 0, sizeof(int), st));
    const int grid = tp.nunits * a.ksplit;
    if (form == 0) PBI4G_CHECK(launch_tm<kFormTF32>(tm, a, smem, grid, st));
    else if (form == 1) PBI4G_CHECK(launch_tm<kFormF16>(tm, a, smem, grid, st));
    else PBI4G_CHECK(launch_tm<kFormBF16>(tm, a, smem, grid, st));
    PBI4G_CHECK(reduce_partials(tp.nslots, a.ksplit, partial.as<double>(), S, accumulate, st));
    *launches += 2;
    return PBI4G_OK;
}

int tm_check_error(TmPlan &tp, cudaStream_t st) {
    int h = 0;
    PBI4G_CUDA(cudaMemcpyAsync(&h, tp.err.p, sizeof(int), cudaMemcpyDeviceToHost, st));
    PBI4G_CUDA(cudaStreamSynchronize(st));
    if (h) return set_error(PBI4G_ERR_TIMEOUT, "tensor-core triangle sums: a bounded wait gave up");
    return PBI4G_OK;
}

}  // namespace pbi4g
