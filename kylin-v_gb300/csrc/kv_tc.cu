// Mixed-precision grouped complex GEMM on the 5th-generation tensor cores
// with exact accumulation.
//
// GB300 runs FP64 arithmetic at a small fraction of its FP32 and tensor
// rates, so no FP64 instruction is issued per element of a tile.  Instead:
//
//  1. Slicing (slice_item; one launch per call for both operands).  Every GEMM row of an A
//     block (and every GEMM column of a B block) gets a binary exponent e
//     with max_k |x| < 2^e over that row; each real value becomes the
//     fixed-point integer X = round(x 2^(37-e)), |X| <= 2^37, written as five
//     balanced base-256 digits X = d0 2^32 + d1 2^24 + d2 2^16 + d3 2^8 + d4
//     (|d0| <= 33, |d1..d4| <= 128) in FP16 (exact).  For the 3M complex form
//     three values are sliced per element: re, im and re + im (the last as
//     the exact integer sum X_re + X_im).  Integer arithmetic only.  Where
//     the contracted index runs over parts of very different magnitude (MPO
//     channels, Schmidt values), it is first balanced by exact powers of two
//     (kmax_item, GemmPlan::balance_k; the maxima and the slicing are one
//     launch with a barrier between them, k_slice_coop or k_slice_cluster).  The digits are written directly in the
//     tensor cores' shared-memory panel layout (K-major, no swizzle: 8-row x
//     16-byte core matrices, K-adjacent core matrices 128 B apart, 8-row
//     groups 256 B apart), one 16-deep K panel after another, all 15 digit
//     planes of a panel contiguous, so a pipeline stage is one bulk copy per
//     operand.
//  2. Products (k_gemm_tc).  T1 = Ar Br, T2 = Ai Bi, T3 = As Bs are formed as
//     digit-pair products of orders o = i + j <= 4 (15 per real product; 15
//     tcgen05.mma.kind::f16 of M=128, N=32..160, K=16 per K panel, see
//     mma_panel) into 15 FP32 accumulators in tensor memory.  Every digit product is an integer of
//     at most 2^14 in magnitude, an order sums at most 2^16 of them per K
//     step, and at most 240 K-steps are accumulated between drains, so every
//     accumulator is an integer below 2^24 and the FP32 accumulation is
//     exact.
//  3. Drains (epilogue warps).  At the end of each segment (one block pair)
//     or every 240 K, the accumulators are read with tcgen05.ld, converted to
//     int64 (sum_o P_o 2^(8(4-o)) = X Y / 2^32), combined into Cr = T1 - T2
//     and Ci = T3 - T1 - T2, aligned to the tile's largest row/column
//     exponents and added to int64 running sums; the final sums are converted
//     to FP64 by integer operations (exponent and mantissa assembled
//     directly).
//
// Result: each output element is exact up to the rounding of X (2^-38 of
// the row/column maximum) and the dropped digit orders 5 to 8 (below
// 2^-33 of the same scale), i.e. ~1e-10 relative to max|A_row| max|B_col| K
// (the 30-bit form this replaced left ~1e-8 per product, too much for 20
// time steps of a 160-site chain), with no FP64 arithmetic in the GEMM.
//
// Pipeline: warp 0 (one thread) issues the bulk copies of 3 stages
// (cp.async.bulk completing on mbarriers), warp 1 allocates tensor memory and
// one thread issues the MMAs (tcgen05.commit frees a stage and signals a
// drain), warps 2-17 drain (four per 32-lane quarter of tensor memory, each
// taking a quarter of the tile's columns: the drain is a long chain of
// dependent integer operations per column, so it is spread thin and four
// warps per scheduler hide its latency).
// Every mbarrier wait is bounded; on timeout the CTA records an error, waits
// (bounded) for its copies and MMAs in flight, frees tensor memory and exits.
#include <mutex>
#include <cooperative_groups.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <utility>

#include "kv_internal.h"

namespace kv {

namespace {

constexpr int BM = kMixedTileM, BN = kMixedTileN, BKC = 16;
constexpr int NDIG = 5, NORD = 5, NCOMP = 3;
constexpr int NPL = NCOMP * NDIG;              // digit planes per operand
constexpr int A_PANEL = NPL * BM * BKC;        // FP16 elements per A panel (all planes)
constexpr int B_PANEL = NPL * BN * BKC;
constexpr int A_BYTES = A_PANEL * 2, B_BYTES = B_PANEL * 2;
constexpr int PLANE_A = BM * BKC * 2, PLANE_B = BN * BKC * 2;  // bytes per plane within a panel
constexpr int STAGES = 3;
constexpr int NACC = NCOMP * NORD;             // accumulators of BN columns
constexpr uint32_t TMEM_COLS = 512;            // NACC * BN = 480, rounded to a power of two
constexpr int KDRAIN = 240;                    // K-steps accumulated exactly between drains
constexpr int GKC = KDRAIN / BKC;              // K panels per drain group
constexpr int FRAC = 37;                       // fixed point: X = round(x 2^(FRAC - e)), |X| <= 2^37
// a drained combination sum_o P_o 2^(8(NORD-1-o)) is X Y / 2^COMB_SHIFT
constexpr int COMB_SHIFT = 8 * (2 * (NDIG - 1) - (NORD - 1));
constexpr int kZeroExp = -4000;                // exponent of an all-zero row
constexpr int kErrTimeout = 1, kErrNonFinite = 2;  // bits of the per-device error word
constexpr int kMaxFiniteExp = 1024;            // row / column exponents of finite operands are <= 1024
constexpr long long WAIT_LIMIT = 1ll << 22;   // try_wait polls before a wait gives up
constexpr int EPI_WARPS = 16;                  // four per tensor-memory lane quarter, 8 columns each
constexpr int EPI_COLS = BN / (EPI_WARPS / 4);
constexpr int NTHREADS = 32 * (2 + EPI_WARPS);
constexpr int SMEM_ALIGN = 128;                // stage base alignment (no-swizzle layout, bulk copies)
constexpr int SMEM_BYTES = STAGES * (A_BYTES + B_BYTES) + SMEM_ALIGN + 1024;
static_assert(SMEM_BYTES <= 227 * 1024, "pipeline stages exceed the shared memory of one CTA");

static_assert(NACC * BN <= (int)TMEM_COLS, "accumulators exceed tensor memory");
static_assert(EPI_COLS == 8, "a warp's columns are one multiple of 8 (one piece), loaded 4 at a time");
static_assert(A_BYTES + B_BYTES < (1 << 20), "transaction count per stage");

// ----------------------------------------------------------- slicing
// round(x 2^(FRAC-e)) for |x| < 2^e, from the bits of x (integer operations only)
__device__ __forceinline__ long long fixq(double x, int e) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(x);
    const int E = (int)((u >> 52) & 0x7FF);
    // X = m >> s with m the 53-bit significand; s >= 53 - FRAC when |x| < 2^e
    const int s = 1075 - FRAC + e - E;
    if (E == 0 || s >= 64) return 0;
    long long X;
    if (s < 53 - FRAC) X = 1ll << FRAC;  // only for non-finite input (the exponent came from an inf/NaN row)
    else X = (long long)((((u & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull) + (1ull << (s - 1))) >> s);
    return (u >> 63) ? -X : X;
}

// element offset of (row r, k) inside one plane of a panel 16 deep
__device__ __forceinline__ int panel_off(int r, int k) {
    return (r >> 3) * 128 + (k >> 3) * 64 + (r & 7) * 8 + (k & 7);
}

// The five balanced base-256 digits of X0 and X1 as FP16 pairs.  Adding 128 at
// each of the four low digits makes the digits plus 128 the bytes of Y.  Two
// digits |d| <= 512 as FP16: 1536 + d in the binade [1024, 2048) has unit
// spacing, so its bits are 0x6600 + d; subtracting 1536 is exact.
__device__ __forceinline__ void digit_pairs(long long X0, long long X1, __half2 out[NDIG]) {
    static_assert(NDIG == 5, "four bytes and a leading digit");
    const long long Y0 = X0 + 0x80808080ll, Y1 = X1 + 0x80808080ll;
    const uint32_t l0 = (uint32_t)Y0, l1 = (uint32_t)Y1;
    auto half2_of = [](uint32_t u) {
        __half2 h;
        memcpy(&h, &u, sizeof(h));
        return __hsub2(h, __float2half2_rn(1536.f));
    };
    const uint32_t h0 = (uint32_t)(0x6600 + (int)(Y0 >> 32)), h1 = (uint32_t)(0x6600 + (int)(Y1 >> 32));
    out[0] = half2_of(__byte_perm(h0, h1, 0x5410));
    out[1] = half2_of((__byte_perm(l0, l1, 0x0703) & 0x00FF00FFu) + 0x65806580u);
    out[2] = half2_of((__byte_perm(l0, l1, 0x0602) & 0x00FF00FFu) + 0x65806580u);
    out[3] = half2_of((__byte_perm(l0, l1, 0x0501) & 0x00FF00FFu) + 0x65806580u);
    out[4] = half2_of((__byte_perm(l0, l1, 0x0400) & 0x00FF00FFu) + 0x65806580u);
}

// Balancing of the contracted index k: kmax[k] holds the largest binary
// exponent (biased, 0: none) of re, im in A's column k over the A views of a
// segment component, kmax[kscales + k] that of B's row k.  A's column is scaled
// by 2^s, B's row by 2^-s, with s = floor((E_B - E_A) / 2), so both reach about
// sqrt(max_A max_B) and every digit product is resolved at the same scale.
__device__ __forceinline__ int balance_shift(const int *kmax, int64_t kscales, int64_t k, int b_side) {
    const int ea = __ldcg(kmax + k), eb = __ldcg(kmax + kscales + k);
    if (ea == 0 || eb == 0) return 0;
    const int sh = (eb - ea) >> 1;
    return b_side ? -sh : sh;
}

// x * 2^sh by the exponent field alone (no FP64 arithmetic): exact for
// normal results; results below the normal range become +-0 and results
// beyond it +-inf (as the product would round; a subnormal input stays as it
// is, and fixq reads subnormals as 0 either way)
__device__ __forceinline__ double scale_exp(double x, int sh) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(x);
    const int E = (int)((u >> 52) & 0x7FF);
    if (sh == 0 || E == 0 || E == 0x7FF) return x;
    const int En = E + sh;
    const unsigned long long sign = u & 0x8000000000000000ull;
    if (En <= 0) return __longlong_as_double((long long)sign);
    if (En >= 0x7FF) return __longlong_as_double((long long)(sign | 0x7FF0000000000000ull));
    return __longlong_as_double((long long)((u & ~(0x7FFull << 52)) | ((unsigned long long)En << 52)));
}

// the high word of |x| with its last bit set if only the low word is nonzero:
// ordered by magnitude up to the exponent, zero only for x = 0
__device__ __forceinline__ int magnitude(double x) {
    return (__double2hiint(x) & 0x7FFFFFFF) | (__double2loint(x) != 0 ? 1 : 0);
}

// Slicing works on items of 8 rows (one core matrix high), GW warps an item
// splitting its K range in steps of 8.  Lane l of a warp holds row l / 4 and
// the K positions 2 (l % 4) and + 1 of a step: a step's digits of one plane are
// one 128-byte core matrix, written by one coalesced store (a row a warp wrote
// 16-byte pieces of eight lines), and both operand orders are read in 64 or
// 128-byte pieces.
struct SliceArgs {
    const SliceJob *ajobs, *bjobs;
    const int2 *aitems, *bitems;
    int na, nb;
    const double2 *A, *B;
    __half *ap, *bp;
    int *ae, *be;
    double alpha;
    int step;
    int *err;
    int *kmax;  // null: no balancing
    int64_t kscales;
};

struct SliceLane {
    SliceJob j;
    const double2 *src;
    int64_t base;  // element (row, 0)
    int64_t kst;   // elements per k
    bool on;       // the lane's row exists
    bool is_b;
    int rr;        // row within the panel
};
// the item's job and this lane's row; false: no active segment reads it
__device__ __forceinline__ bool slice_open(const SliceArgs &a, int item, SliceLane &x) {
    x.is_b = item >= a.na;
    const int2 it = x.is_b ? a.bitems[item - a.na] : a.aitems[item];
    x.j = x.is_b ? a.bjobs[it.x] : a.ajobs[it.x];
    if (x.j.entry > a.step) return false;
    const int r = it.y + ((threadIdx.x & 31) >> 2);
    x.on = r < x.j.rows;
    x.rr = x.j.r0 + r;
    const int64_t row = x.j.row0 + r;
    x.src = (x.is_b ? a.B : a.A) + x.j.src_off;
    x.base = x.j.trans ? row : row * x.j.ld;
    x.kst = x.j.trans ? x.j.ld : 1;
    return true;
}
__device__ __forceinline__ double2 slice_raw(const SliceLane &x, int k) {
    return x.on && k < x.j.K ? x.src[x.base + k * x.kst] : make_double2(0.0, 0.0);
}

// largest exponents per k over the item's rows, into kmax
__device__ __forceinline__ void kmax_item(const SliceArgs &a, int item, int w, int GW) {
    SliceLane x;
    if (!slice_open(a, item, x) || x.j.ks_off < 0) return;  // uniform over the item's warps
    const int lane = threadIdx.x & 31;
    int *dst = a.kmax + (x.is_b ? a.kscales : 0) + x.j.ks_off;
    for (int k0 = 8 * w; k0 < x.j.K; k0 += 8 * GW) {
        const int k = k0 + 2 * (lane & 3);
        const double2 v0 = slice_raw(x, k), v1 = slice_raw(x, k + 1);
        const int e0 = max(__double2hiint(v0.x) & 0x7FFFFFFF, __double2hiint(v0.y) & 0x7FFFFFFF) >> 20;
        const int e1 = max(__double2hiint(v1.x) & 0x7FFFFFFF, __double2hiint(v1.y) & 0x7FFFFFFF) >> 20;
        unsigned m = (unsigned)e0 | ((unsigned)e1 << 16);
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) m = __vmaxu2(m, __shfl_xor_sync(0xFFFFFFFFu, m, o));
        if (lane < 4) {
            if (k < x.j.K && (m & 0xFFFF)) atomicMax(dst + k, (int)(m & 0xFFFF));
            if (k + 1 < x.j.K && (m >> 16)) atomicMax(dst + k + 1, (int)(m >> 16));
        }
    }
}

// One item's digits.  A row holding an Inf or NaN sets bit kErrNonFinite of
// *err: fixed point has no code for it, and the digits written for that row are
// meaningless.  red: [GW][8] shared words of the item's warps; bar: their
// named barrier.
__device__ __forceinline__ void slice_item(const SliceArgs &a, int item, int w, int GW, int (*red)[8], int bar) {
    SliceLane x;
    if (!slice_open(a, item, x)) return;  // uniform over the item's warps
    const int lane = threadIdx.x & 31;
    const bool scale = x.is_b && a.alpha != 1.0, bal = a.kmax != nullptr && x.j.ks_off >= 0;
    const int nst = 2 * x.j.nkc;  // steps of 8, zero-padded past K
    auto load = [&](int k) {
        double2 v = slice_raw(x, k);
        if (scale) { v.x *= a.alpha; v.y *= a.alpha; }
        if (x.j.conj) v.y = __hiloint2double(__double2hiint(v.y) ^ (int)0x80000000, __double2loint(v.y));
        if (bal && k < x.j.K) {  // exact power-of-two balancing of the contracted index
            const int sh = balance_shift(a.kmax, a.kscales, x.j.ks_off + k, x.is_b ? 1 : 0);
            v.x = scale_exp(v.x, sh);
            v.y = scale_exp(v.y, sh);
        }
        return v;
    };
    constexpr int KEEP = 4;  // steps whose elements stay in registers between the two passes
    double2 kept[KEEP][2];
    int mx = 0;
#pragma unroll
    for (int i = 0; i < KEEP; ++i) {
        const int st = w + i * GW;
        if (st >= nst) break;  // warp-uniform
        const int k = 8 * st + 2 * (lane & 3);
        kept[i][0] = load(k);
        kept[i][1] = load(k + 1);
        mx = max(mx, max(max(magnitude(kept[i][0].x), magnitude(kept[i][0].y)),
                         max(magnitude(kept[i][1].x), magnitude(kept[i][1].y))));
    }
    for (int st = w + KEEP * GW; st < nst; st += GW) {
        const int k = 8 * st + 2 * (lane & 3);
        const double2 v0 = load(k), v1 = load(k + 1);
        mx = max(mx, max(max(magnitude(v0.x), magnitude(v0.y)), max(magnitude(v1.x), magnitude(v1.y))));
    }
    mx = max(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, 1));
    mx = max(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, 2));
    if (GW > 1) {
        if ((lane & 3) == 0) red[w][lane >> 2] = mx;
        asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(32 * GW) : "memory");
        for (int i = 0; i < GW; ++i) mx = max(mx, red[i][lane >> 2]);
        asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(32 * GW) : "memory");  // red is free for the next item
    }
    const int e = mx ? (mx >> 20) - 1022 : kZeroExp;
    if (w == 0 && (lane & 3) == 0 && x.on) {
        (x.is_b ? a.be : a.ae)[x.j.exp_off + x.rr - x.j.r0] = e;
        if (mx >= 0x7FF00000) atomicOr(a.err, kErrNonFinite);
    }
    // rows past the piece are not written: they only reach output rows /
    // columns the GEMM epilogue never stores
    if (!x.on) return;
    const int plane = x.j.tr * BKC;  // elements of a digit plane
    __half *pan = (x.is_b ? a.bp : a.ap) + x.j.dst_off;
    auto put = [&](int st, double2 v0, double2 v1) {
        const int k = 8 * st + 2 * (lane & 3);
        long long X[2][NCOMP];
        X[0][0] = fixq(v0.x, e);
        X[0][1] = fixq(v0.y, e);
        X[0][2] = X[0][0] + X[0][1];
        X[1][0] = fixq(v1.x, e);
        X[1][1] = fixq(v1.y, e);
        X[1][2] = X[1][0] + X[1][1];
        __half *p = pan + (int64_t)(k / BKC) * (NPL * plane) + panel_off(x.rr, k & (BKC - 1));
#pragma unroll
        for (int c = 0; c < NCOMP; ++c) {
            __half2 d[NDIG];
            digit_pairs(X[0][c], X[1][c], d);
#pragma unroll
            for (int i = 0; i < NDIG; ++i) *reinterpret_cast<__half2 *>(p + (c * NDIG + i) * plane) = d[i];
        }
    };
#pragma unroll
    for (int i = 0; i < KEEP; ++i) {
        const int st = w + i * GW;
        if (st >= nst) break;
        put(st, kept[i][0], kept[i][1]);
    }
    for (int st = w + KEEP * GW; st < nst; st += GW) {
        const int k = 8 * st + 2 * (lane & 3);
        put(st, load(k), load(k + 1));
    }
}

constexpr int kSliceWarps = 8;

// Both operands' slicing (the A items, then the B items), CTA `cta` of `ctas`.
// MAX: the balancing maxima only; otherwise the digits.
template <bool MAX>
__device__ __forceinline__ void slice_walk(const SliceArgs &a, int GW, int cta, int ctas) {
    __shared__ int red[kSliceWarps][8];
    const int warp = threadIdx.x >> 5, per = kSliceWarps / GW, grp = warp / GW, w = warp % GW;
    for (int item = cta * per + grp; item < a.na + a.nb; item += ctas * per) {
        if constexpr (MAX) kmax_item(a, item, w, GW);
        else slice_item(a, item, w, GW, red + grp * GW, 1 + grp);
    }
}

// One launch: the maxima of every contracted index, a barrier, the digits; the
// maxima start from zero (k_gemm_tc of the previous call cleared them).
//  * a grid barrier (cooperative launch) on the main context's stream;
//  * a cluster barrier for few items: a cluster is scheduled whole, so worker
//    streams can use it too.
//  * two launches (k_slice_max, k_slice_put) for many items on worker streams.
// What bounds it: integer instructions and the chain maxima, barrier, row
// maxima for small operands; the panels' traffic (30 B written a complex
// element) for large ones.  Measured (us a launch, a row per warp and three
// grid barriers before): D = 32 12.5 -> 8.8, D = 128 two-site 30.2 -> 24.1 and
// over 8 x 8 blocks 28.2 -> 13.1, D = 512 204 -> 127.
__global__ void __launch_bounds__(32 * kSliceWarps) k_slice_coop(SliceArgs a, int GW, const int *skip) {
    allow_dependents();
    if (skip && *skip) return;  // uniform over the grid: nothing in this launch writes it
    if (a.kmax) {
        slice_walk<true>(a, GW, (int)blockIdx.x, (int)gridDim.x);
        cooperative_groups::this_grid().sync();
    }
    slice_walk<false>(a, GW, (int)blockIdx.x, (int)gridDim.x);
}
__global__ void __launch_bounds__(32 * kSliceWarps) k_slice_cluster(SliceArgs a, int GW, const int *skip) {
    allow_dependents();
    dependency_wait();
    if (skip && *skip) return;
    if (a.kmax) {
        slice_walk<true>(a, GW, (int)blockIdx.x, (int)gridDim.x);
        cooperative_groups::this_cluster().sync();
    }
    slice_walk<false>(a, GW, (int)blockIdx.x, (int)gridDim.x);
}
__global__ void __launch_bounds__(32 * kSliceWarps) k_slice_max(SliceArgs a, int GW, const int *skip) {
    allow_dependents();
    dependency_wait();
    if (skip && *skip) return;
    slice_walk<true>(a, GW, (int)blockIdx.x, (int)gridDim.x);
}
__global__ void __launch_bounds__(32 * kSliceWarps) k_slice_put(SliceArgs a, int GW, const int *skip) {
    allow_dependents();
    dependency_wait();
    if (skip && *skip) return;
    slice_walk<false>(a, GW, (int)blockIdx.x, (int)gridDim.x);
}

// -------------------------------------------------------- tensor-core GEMM
__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// UMMA shared-memory descriptor: start >> 4 (bits 0-13), leading byte offset
// >> 4 (16-29), stride byte offset >> 4 (32-45), descriptor version 1 (46-47),
// base offset 0, layout type 0 = no swizzle (61-63).
__device__ __forceinline__ uint64_t make_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFFu);
    d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
    d |= (uint64_t)1 << 46;
    return d;
}

// instruction descriptor, kind::f16: D = F32 (bits 4-5 = 1), A = B = F16
// (bits 7-9, 10-12 = 0), both K-major, N >> 3 at bit 17, M >> 4 at bit 24
constexpr uint32_t idesc(int n) { return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(BM >> 4) << 24); }

// D (+)= A B over N columns with the accumulate flag fixed at compile time (no per-MMA predicate set-up)
template <bool ACC, int N>
__device__ __forceinline__ void mma_f16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc) {
    if constexpr (ACC)
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.eq.u32 p, 1, 1;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d),
            "l"(adesc), "l"(bdesc), "n"(idesc(N)));
    else
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, 1, 1;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d),
            "l"(adesc), "l"(bdesc), "n"(idesc(N)));
}

// The MMAs of one K panel.  A's digit plane i meets B's planes 0 .. 4-i: those
// planes are consecutive in shared memory (one N axis of 32 (5-i) rows) and
// their orders i .. 4 are consecutive accumulators, so one MMA of N = 32 (5-i)
// does 5-i digit pairs: 15 MMAs a panel, each reading its A plane once (45 of
// N = 32 read A 45 times, and shared memory bounds them: D = 512 two-site
// Lanczos exponential, us a launch: 365 -> 212; D = 128: 34.6 -> 27.2).
// Shared-memory descriptors are the stage's plane-0 descriptors plus plane
// offsets (multiples of 16 bytes, and no address leaves the 14-bit field, so
// adding offset / 16 to the descriptor is adding it to the address); pa: an A
// plane's bytes / 16.  An A plane of fewer than 128 rows is followed by the
// next one, so the MMA's rows beyond it multiply other digits and reach only
// output rows that are not stored.  FIRST: the panel opens a drain group, so A's
// plane 0, which reaches every order, overwrites the accumulators.
template <bool FIRST, int I>
__device__ __forceinline__ void mma_plane(uint32_t tmem, uint64_t da, uint64_t db, uint32_t pa) {
#pragma unroll
    for (int c = 0; c < NCOMP; ++c)
        mma_f16<!(FIRST && I == 0), BN *(NORD - I)>(tmem + (uint32_t)((c * NORD + I) * BN),
                                                    da + (uint64_t)((uint32_t)(c * NDIG + I) * pa),
                                                    db + (uint64_t)(((c * NDIG) * PLANE_B) >> 4));
}
template <bool FIRST>
__device__ __forceinline__ void mma_panel(uint32_t tmem, uint64_t da, uint64_t db, uint32_t pa) {
    static_assert(NDIG == 5 && NORD == 5, "one call per digit plane of A");
    mma_plane<FIRST, 0>(tmem, da, db, pa);
    mma_plane<FIRST, 1>(tmem, da, db, pa);
    mma_plane<FIRST, 2>(tmem, da, db, pa);
    mma_plane<FIRST, 3>(tmem, da, db, pa);
    mma_plane<FIRST, 4>(tmem, da, db, pa);
}

__device__ __forceinline__ void mma_commit(uint32_t mbar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar)
                 : "memory");
}

__device__ __forceinline__ void mbar_init(uint32_t mbar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(mbar), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t mbar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(mbar) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t mbar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mbar), "r"(bytes) : "memory");
}

__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t parity, long long limit = WAIT_LIMIT) {
    for (long long i = 0; i < limit; ++i) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(done)
            : "r"(mbar), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void *src, uint32_t bytes, uint32_t mbar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
        "l"(src), "r"(bytes), "r"(mbar)
        : "memory");
}

__device__ __forceinline__ void tmem_ld4(uint32_t taddr, float *v) {
    uint32_t r0, r1, r2, r3;
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(taddr));
    v[0] = __uint_as_float(r0);
    v[1] = __uint_as_float(r1);
    v[2] = __uint_as_float(r2);
    v[3] = __uint_as_float(r3);
}

__device__ __forceinline__ void epi_bar() { asm volatile("bar.sync 1, %0;" ::"n"(32 * EPI_WARPS) : "memory"); }

// v / 2^sh rounded to nearest, sh >= 0
__device__ __forceinline__ long long sra_round(long long v, int sh) {
    if (sh <= 0) return v;
    if (sh >= 62) return 0;
    return (v + (1ll << (sh - 1))) >> sh;
}

// v 2^sc as FP64, rounded to nearest even, from integer operations
__device__ __forceinline__ double i64_ldexp(long long v, int sc) {
    if (v == 0) return 0.0;
    const unsigned long long neg = v < 0 ? 1ull : 0ull;
    unsigned long long a = neg ? (unsigned long long)(-v) : (unsigned long long)v;
    const int lz = __clzll((long long)a);
    a <<= lz;  // leading one at bit 63
    int ex = 63 - lz + sc;
    unsigned long long mant = a >> 11;
    const unsigned long long rem = a & 0x7FFull;
    if (rem > 0x400ull || (rem == 0x400ull && (mant & 1ull))) {
        ++mant;
        if (mant >> 53) { mant >>= 1; ++ex; }
    }
    const int E = ex + 1023;
    if (E <= 0) return 0.0;
    if (E >= 2047) return __longlong_as_double((long long)((neg << 63) | 0x7FF0000000000000ull));
    return __longlong_as_double((long long)((neg << 63) | ((unsigned long long)E << 52) | (mant & 0xFFFFFFFFFFFFFull)));
}

// sum_o P_o 2^(8(4-o)) from the five order accumulators (exact integers < 2^24)
__device__ __forceinline__ long long combine(const float *p) {
    long long u = __float2int_rn(p[0]);
    u = (u << 8) + __float2int_rn(p[1]);
    u = (u << 8) + __float2int_rn(p[2]);
    u = (u << 8) + __float2int_rn(p[3]);
    return (u << 8) + __float2int_rn(p[4]);
}

// Persistent: CTA b takes tiles b, b + gridDim.x, ...; each role walks the
// same tile sequence and keeps its mbarrier phase counters across tiles, so
// the producer streams the next tile's panels while the current tile drains.
__device__ __forceinline__ bool tile_active(const TcTile &t, const SegX *segs, int step) {
    for (int s = t.seg_begin; s < t.seg_end; ++s)
        if (segs[s].entry <= step) return true;
    return false;
}

__global__ void __launch_bounds__(NTHREADS, 1) k_gemm_tc(const TcTile *__restrict__ tiles, int ntiles,
                                                    const SegX *__restrict__ segs, const int2 *__restrict__ maps,
                                                    const TcPair *__restrict__ pairs,
                                                    const __half *__restrict__ Apl, const __half *__restrict__ Bpl,
                                                    const int *__restrict__ Aexp, const int *__restrict__ Bexp,
                                                    double2 *__restrict__ C, const int *skip, int *err, int step,
                                                    int write_inactive, long long wait_limit, int no_copies,
                                                    int *kmax, int nkmax) {
    // no allow_dependents: its successors' CTAs gain nothing by waiting beside a
    // CTA that holds the SM (D = 512 Lanczos exponential 9.93 ms with, 9.81 without)
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + SMEM_ALIGN - 1) & ~(uintptr_t)(SMEM_ALIGN - 1));
    uint8_t *sA = smem;
    uint8_t *sB = smem + STAGES * A_BYTES;
    uint64_t *bars = (uint64_t *)(smem + STAGES * (A_BYTES + B_BYTES));
    uint64_t *full = bars, *empty = bars + STAGES, *accf = bars + 2 * STAGES, *acce = accf + 1, *mdone = acce + 1;
    uint32_t *tslot = (uint32_t *)(mdone + 1);
    int *s_ecol = (int *)(tslot + 4);  // [BN] largest column exponent over the tile's segments
    int *s_fcol = s_ecol + BN;         // [EPI_WARPS][EPI_COLS] each epilogue warp's copy of a segment's
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)),
                     "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(smem_u32(full + s), 1);
            mbar_init(smem_u32(empty + s), 1);
        }
        mbar_init(smem_u32(accf), 1);
        mbar_init(smem_u32(acce), 32 * EPI_WARPS);
        mbar_init(smem_u32(mdone), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tslot;
    dependency_wait();
    if (skip && *skip) ntiles = 0;  // uniform over the grid: no role has a tile
    else
        // the balancing maxima are used up: zero for the next call's slicing
        for (int i = (int)(blockIdx.x * blockDim.x + threadIdx.x); i < nkmax; i += (int)(gridDim.x * blockDim.x))
            kmax[i] = 0;

    if (warp == 0) {
        // ------------------------------------------------ producer
        if (lane == 0) {
            int it = 0;
            int uses[STAGES] = {0, 0, 0};
            bool ok = true;
            for (int ti = blockIdx.x; ti < ntiles && ok; ti += gridDim.x) {
                const TcTile t = tiles[ti];
                const int a_panel = NPL * BKC * t.rows;  // FP16 elements of one K panel of A
                for (int s = t.seg_begin; s < t.seg_end && ok; ++s) {
                    const SegX g = segs[s];
                    if (g.entry > step) continue;
                    const __half *ap = Apl + g.a_pan;
                    const __half *bp = Bpl + g.b_pan;
                    for (int kc = 0; kc < g.nkc && !no_copies; ++kc, ++it) {
                        const int st = it % STAGES;
                        const uint32_t ph = (uint32_t)(it / STAGES) & 1u;
                        if (!mbar_wait(smem_u32(empty + st), ph ^ 1u, wait_limit)) { ok = false; break; }
                        mbar_expect_tx(smem_u32(full + st), (uint32_t)(2 * a_panel + B_BYTES));
                        bulk_g2s(smem_u32(sA + st * A_BYTES), ap + (int64_t)kc * a_panel, (uint32_t)(2 * a_panel),
                                 smem_u32(full + st));
                        bulk_g2s(smem_u32(sB + st * B_BYTES), bp + (int64_t)kc * B_PANEL, B_BYTES,
                                 smem_u32(full + st));
                        ++uses[st];
                    }
                }
            }
            if (!ok) atomicOr(err, kErrTimeout);
            // no copy may land after the CTA exits: wait (bounded) for the last one into each stage
            for (int st = 0; st < STAGES; ++st)
                if (uses[st]) mbar_wait(smem_u32(full + st), (uint32_t)(uses[st] - 1) & 1u, wait_limit);
        }
    } else if (warp == 1) {
        // ------------------------------------------------ MMA issue
        if (lane == 0) {
            // plane-0 descriptors of stage 0; stage st adds st * bytes / 16 to the address field
            const uint64_t desc_a0 = make_desc(smem_u32(sA), 128, 256), desc_b0 = make_desc(smem_u32(sB), 128, 256);
            int it = 0, grp = 0;
            bool ok = true;
            for (int ti = blockIdx.x; ti < ntiles && ok; ti += gridDim.x) {
                const TcTile t = tiles[ti];
                const uint32_t pa = (uint32_t)(t.rows * BKC * 2) >> 4;
                for (int s = t.seg_begin; s < t.seg_end && ok; ++s) {
                    if (segs[s].entry > step) continue;
                    const int nkc = segs[s].nkc;
                    for (int kc0 = 0; kc0 < nkc && ok; kc0 += GKC, ++grp) {
                        // the epilogue has read the previous group's accumulators
                        if (!mbar_wait(smem_u32(acce), ((uint32_t)grp & 1u) ^ 1u, wait_limit)) { ok = false; break; }
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        const int kc1 = min(nkc, kc0 + GKC);
                        for (int kc = kc0; kc < kc1; ++kc, ++it) {
                            const int st = it % STAGES;
                            const uint32_t ph = (uint32_t)(it / STAGES) & 1u;
                            if (!mbar_wait(smem_u32(full + st), ph, wait_limit)) { ok = false; break; }
                            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                            const uint64_t da = desc_a0 + (uint64_t)(st * (A_BYTES >> 4));
                            const uint64_t db = desc_b0 + (uint64_t)(st * (B_BYTES >> 4));
                            if (t.rows == BM) {  // plane offsets known at compile time
                                if (kc == kc0) mma_panel<true>(tmem, da, db, PLANE_A >> 4);
                                else mma_panel<false>(tmem, da, db, PLANE_A >> 4);
                            } else {
                                if (kc == kc0) mma_panel<true>(tmem, da, db, pa);
                                else mma_panel<false>(tmem, da, db, pa);
                            }
                            mma_commit(smem_u32(empty + st));  // stage free once these MMAs are done
                        }
                        if (!ok) break;
                        mma_commit(smem_u32(accf));  // accumulators ready for the drain
                    }
                }
            }
            if (!ok) atomicOr(err, kErrTimeout);
            // every MMA issued by this thread has completed before tensor memory is freed
            mma_commit(smem_u32(mdone));
            mbar_wait(smem_u32(mdone), 0u, wait_limit);
        }
    } else {
        // ------------------------------------------------ drains and epilogue
        // warp w reads lane quarter w % 4 (the rows it may access in tensor
        // memory) and columns [c_lo, c_lo + EPI_COLS)
        const int q = warp & 3;
        const int c_lo = ((warp - 2) / 4) * EPI_COLS;
        const int m = q * 32 + lane;
        const uint32_t trow = tmem + ((uint32_t)(q * 32) << 16);
        int *fw = s_fcol + (warp - 2) * EPI_COLS;  // this warp's copy of the segment's column exponents
        bool ok = true;  // warp-uniform; after a timed-out wait the warp stops waiting but keeps the barriers
        int grp = 0;
        for (int ti = blockIdx.x; ti < ntiles; ti += gridDim.x) {
            const TcTile t = tiles[ti];
            const bool act = tile_active(t, segs, step);
            const bool used = q * 32 < t.rows;  // warp-uniform: some row of this quarter is stored
            if (!act && !write_inactive) continue;  // the same for every epilogue warp
            const int nseg = t.seg_end - t.seg_begin;
            // where this thread's row and the warp's 8 columns go (pieces start at
            // multiples of 8, so the columns belong to one): read ahead of the drain
            // (row piece, row of its block)
            const int2 rm = m < t.rows ? maps[t.rowmap + m] : make_int2(-1, 0);
            const int2 cm = maps[t.colmap + c_lo + (lane & (EPI_COLS - 1))];
            const int ncol = __popc(__ballot_sync(0xFFFFFFFFu, lane < EPI_COLS && cm.x >= 0));
            const int cpiece = __shfl_sync(0xFFFFFFFFu, cm.x, 0), col0 = __shfl_sync(0xFFFFFFFFu, cm.y, 0);
            TcPair pr{-1, 0, kAllSteps};
            if (rm.x >= 0 && cpiece >= 0) pr = pairs[t.pair + (int64_t)rm.x * t.ncol + cpiece];
            const bool live = act && pr.entry <= step;
            const bool mine = pr.c_off >= 0 && (live || write_inactive);
            int erow = kZeroExp;
            for (int s = t.seg_begin; s < t.seg_end; ++s)
                if (segs[s].entry <= step) erow = max(erow, Aexp[segs[s].a_exp + m]);
            if (warp == 2) {
                int ec = kZeroExp;
                for (int s = t.seg_begin; s < t.seg_end; ++s)
                    if (segs[s].entry <= step) ec = max(ec, Bexp[segs[s].b_exp + lane]);
                s_ecol[lane] = ec;
            }
            epi_bar();  // s_ecol written; reached by every epilogue warp for every tile
            long long cr[EPI_COLS], ci[EPI_COLS];
#pragma unroll
            for (int c = 0; c < EPI_COLS; ++c) cr[c] = ci[c] = 0;
            for (int sl = 0; sl < nseg; ++sl) {
                const SegX g = segs[t.seg_begin + sl];
                if (g.entry > step) continue;
                // column shifts of this segment, into the warp's own shared-memory slots
                if (lane < EPI_COLS) fw[lane] = s_ecol[c_lo + lane] - Bexp[g.b_exp + c_lo + lane];
                __syncwarp();
                const int shr = erow - Aexp[g.a_exp + m];
                for (int kc0 = 0; kc0 < g.nkc; kc0 += GKC, ++grp) {
                    // warp-uniform decision: tcgen05.ld below is a warp-wide instruction
                    if (ok && !__all_sync(0xFFFFFFFFu, mbar_wait(smem_u32(accf), (uint32_t)grp & 1u, wait_limit)))
                        ok = false;
                    if (!ok) continue;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    if (used)
#pragma unroll
                    for (int c0 = 0; c0 < EPI_COLS; c0 += 4) {
                        long long I[NCOMP][4];
#pragma unroll
                        for (int c = 0; c < NCOMP; ++c) {
                            float a[NORD][4];
#pragma unroll
                            for (int o = 0; o < NORD; ++o)
                                tmem_ld4(trow + (uint32_t)((c * NORD + o) * BN + c_lo + c0), a[o]);
                            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                            for (int jx = 0; jx < 4; ++jx) {
                                float p[NORD];
#pragma unroll
                                for (int o = 0; o < NORD; ++o) p[o] = a[o][jx];
                                I[c][jx] = combine(p);
                            }
                        }
#pragma unroll
                        for (int jx = 0; jx < 4; ++jx) {
                            const int col = c0 + jx;
                            const int sh = shr + fw[col];
                            cr[col] += sra_round(I[0][jx] - I[1][jx], sh);
                            ci[col] += sra_round(I[2][jx] - I[0][jx] - I[1][jx], sh);
                        }
                    }
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    mbar_arrive(smem_u32(acce));
                }
                __syncwarp();  // fw is rewritten for the next segment
            }
            if (ok && mine) {
                double2 *crow = C + pr.c_off + (int64_t)rm.y * pr.ldc + col0;
#pragma unroll
                for (int c = 0; c < EPI_COLS; ++c) {
                    if (c >= ncol) break;  // warp-uniform
                    const int ec = s_ecol[c_lo + c];
                    const int sc = erow + ec - 2 * FRAC + COMB_SHIFT;
                    // a row or column holding Inf or NaN (slicer exponent above the
                    // FP64 range) gives NaN, as the FP64 product would
                    crow[c] = !live ? make_double2(0.0, 0.0)
                              : (erow > kMaxFiniteExp || ec > kMaxFiniteExp)
                                  ? make_double2(__longlong_as_double(0x7FF8000000000000ll),
                                                 __longlong_as_double(0x7FF8000000000000ll))
                                  : make_double2(i64_ldexp(cr[c], sc), i64_ldexp(ci[c], sc));
                }
            }
            epi_bar();  // every warp has used s_ecol before the next tile rewrites it
        }
        if (!ok && lane == 0) atomicOr(err, kErrTimeout);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS)
                     : "memory");
    }
}

// Per device: the kernel's shared-memory limit is raised and its error word
// (kErrTimeout | kErrNonFinite bits, cleared when read) allocated once.
constexpr int kMaxDevices = 64;
std::mutex g_dev_mu;
int *g_err[kMaxDevices] = {};
// test hook (kv_debug_gemm_stall): copies withheld and a short wait limit
int g_stall_test = 0;

int *device_err_word(int dev) {
    KV_REQUIRE(dev >= 0 && dev < kMaxDevices, KV_EINVAL, "device index out of range");
    std::lock_guard<std::mutex> lk(g_dev_mu);
    if (!g_err[dev]) {
        KV_CUDA(cudaFuncSetAttribute(k_gemm_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
        int *e = nullptr;
        KV_CUDA(cudaMalloc(&e, sizeof(int)));
        KV_CUDA(cudaMemset(e, 0, sizeof(int)));
        g_err[dev] = e;
    }
    return g_err[dev];
}

}  // namespace

// Tiles, packs and slicing jobs of a tensor-core plan (GemmPlan::tiles holds one
// entry per output block).
//
// A U(1) block-sparse product is a set of dense products cut into small blocks
// (8 x 8 at a D = 128 bond of 17 sectors), and a 128 x 32 tile per output block
// costs the same however little of it is used.  Blocks are therefore packed:
//  * blocks of one segment: A views that meet the same list of B views form a
//    complete bipartite group; their rows and the B views' columns are stacked.
//  * blocks of several segments: blocks with the same list of (B view, entry)
//    share their columns; their rows are stacked (segment by segment).
// Every output element keeps its own segments, row and column exponents, so
// packing does not change a bit of the result.
// The rows a tile takes (128, 64 or 32) follow a cost model: fewer rows make
// more tiles for the SMs to share and smaller operand panels.
// Measured, both GEMM launches of a D = 128 apply over 2992 blocks of 8 x 8 x 8
// (8704 tiles before): 160 -> 32 us; over 62 blocks of 64 x 64: 27.2 -> 23.4 us
// a launch; at D = 512, where blocks fill their tiles: 212 -> 215.
namespace {

struct Pack {
    int begin, end;  // its pieces of the list that it was made in
    int rows;        // with every piece padded to a multiple of 8
};
struct Piece {
    int view, r0, rows, unit;  // rows r0.. of a view; unit: the view's index in the list packed
};

int pad8(int n) { return (n + 7) & ~7; }

// rows of the views in order, cut into packs of at most `most` rows
void make_packs(const std::vector<int> &views, const std::vector<int> &view_rows, int most, std::vector<Pack> *packs,
                std::vector<Piece> *pieces) {
    packs->clear();
    pieces->clear();
    Pack cur{0, 0, 0};
    auto flush = [&] {
        cur.end = (int)pieces->size();
        if (cur.end > cur.begin) packs->push_back(cur);
        cur = Pack{cur.end, cur.end, 0};
    };
    for (size_t u = 0; u < views.size(); ++u)
        for (int r = 0; r < view_rows[u];) {
            if (cur.rows == most) flush();
            const int n = std::min(view_rows[u] - r, most - cur.rows);
            pieces->push_back({views[u], r, n, (int)u});
            cur.rows += pad8(n);
            r += n;
        }
    flush();
}

struct View {
    int64_t key, off;
    int rows, K, ld, trans, conj, ks;
};
struct OutBlock {
    int64_t c_off;
    int ldc, M, N, sb, se;
};
struct Group {
    std::vector<int> rblk;   // row units: A views (one segment) or blocks (several)
    std::vector<int> cview;  // column units: B views (one segment); several: (view, entry) of each segment
    uint64_t hash;           // of cview
    bool multi;
};
struct GroupCost {
    int rows, col_packs, panels, drains;
};
struct Panel {
    int64_t pan;
    int exp;
    int job0, njobs;
};
// ids by 64-bit key, open addressing
struct IdTable {
    std::vector<int> slot;
    size_t mask = 0;
    void reset(size_t n) {
        size_t m = 16;
        while (m < 2 * n) m *= 2;
        slot.assign(m, -1);
        mask = m - 1;
    }
    // the slot of the id for which same(id) holds, or a free one (-1)
    template <class F>
    int &find(uint64_t key, F same) {
        uint64_t h = key * 0x9E3779B97F4A7C15ull;
        h ^= h >> 32;
        for (size_t i = h & mask;; i = (i + 1) & mask)
            if (slot[i] < 0 || same(slot[i])) return slot[i];
    }
};
// The planner's lists, kept by each thread: operations outside the sweep plan on
// every call, and lists grown afresh (page faults of memory that the allocator
// had given back), a node per view and group, and maps of 128 rows for short
// packs took 28 + 69 us of an environment update of 64 + 94 block pairs at
// D = 128, which went from 185 to 125 us without them.  A plan larger than
// kScratchBytes leaves nothing behind.
constexpr size_t kScratchBytes = 4 << 20;
struct Scratch {
    std::vector<View> av, bv;
    std::vector<OutBlock> blocks;
    std::vector<int> sa, sb, zero_blocks, first, of, fill, key, rows, cols, rmap, cmap, bfirst;
    std::vector<Group> groups;
    size_t ngroups = 0;  // of groups in use (the others keep their lists' memory)
    IdTable atab, btab, gtab;
    std::vector<SliceJob> ajobs, bjobs;
    std::vector<SegX> xsegs;
    std::vector<TcTile> tiles;
    std::vector<TcPair> pairs;
    std::vector<int2> maps, aitems, bitems;
    std::vector<Pack> rp, cp;
    std::vector<Piece> rpc, cpc;
    std::vector<Panel> ap, bp, bpanels;
    std::vector<GroupCost> costs;
    void clear() {
        av.clear(), bv.clear(), blocks.clear(), zero_blocks.clear(), bpanels.clear();
        ajobs.clear(), bjobs.clear(), xsegs.clear(), tiles.clear(), pairs.clear(), maps.clear();
        aitems.clear(), bitems.clear();
        ngroups = 0;
    }
    size_t bytes() const {
        return maps.size() * sizeof(int2) + pairs.size() * sizeof(TcPair) + tiles.size() * sizeof(TcTile) +
               xsegs.size() * sizeof(SegX) + (ajobs.size() + bjobs.size()) * sizeof(SliceJob) +
               (aitems.size() + bitems.size()) * sizeof(int2) + (sa.size() + blocks.size()) * 64;
    }
};

}  // namespace

void plan_mixed(GemmPlan &g) {
    thread_local Scratch kept;
    Scratch &w = kept;
    w.clear();
    auto &av = w.av;
    auto &bv = w.bv;
    auto &blocks = w.blocks;
    auto &sa = w.sa, &sb = w.sb;  // views of each segment
    auto &groups = w.groups;
    auto &zero_blocks = w.zero_blocks;
    for (auto &t : g.tiles) blocks.push_back({t.c_off, t.ldc, t.M, t.N, t.seg_begin, t.seg_end});
    // ---- views: one per distinct (block offset, operation) of each operand
    sa.assign(g.segs.size(), -1);
    sb.assign(g.segs.size(), -1);
    w.atab.reset(g.segs.size());
    w.btab.reset(g.segs.size());
    for (auto &b : blocks)
        for (int s = b.sb; s < b.se; ++s) {
            const GemmSeg &sg = g.segs[s];
            const int64_t ka = sg.a_off * 4 + sg.opa, kb = sg.b_off * 4 + sg.opb;
            int &ia = w.atab.find((uint64_t)ka, [&](int i) { return av[i].key == ka; });
            if (ia < 0) {
                ia = (int)av.size();
                av.push_back({ka, sg.a_off, b.M, sg.K, sg.lda, (sg.opa == 1 || sg.opa == 2) ? 1 : 0,
                              (sg.opa == 1 || sg.opa == 3) ? 1 : 0, -1});
            }
            int &ib = w.btab.find((uint64_t)kb, [&](int i) { return bv[i].key == kb; });
            if (ib < 0) {  // B element (n, k) at b[k*ldb + n] for opb 0 and 3
                ib = (int)bv.size();
                bv.push_back({kb, sg.b_off, b.N, sg.K, sg.ldb, (sg.opb == 0 || sg.opb == 3) ? 1 : 0,
                              (sg.opb == 2 || sg.opb == 3) ? 1 : 0, -1});
            }
            sa[s] = ia;
            sb[s] = ib;
            KV_REQUIRE(av[sa[s]].rows == b.M && bv[sb[s]].rows == b.N && av[sa[s]].K == sg.K && bv[sb[s]].K == sg.K,
                       KV_EINVAL, "internal: inconsistent block views in a mixed-precision plan");
        }
    // ---- balancing: A and B views joined by a segment share one vector of
    // per-k scales, so the views of each connected component get one range
    g.k_scales = 0;
    if (g.balance_k) {
        const int na = (int)av.size(), nb = (int)bv.size();
        std::vector<int> parent(na + nb);
        for (int i = 0; i < na + nb; ++i) parent[i] = i;
        auto root = [&](int x) {
            while (parent[x] != x) x = parent[x] = parent[parent[x]];
            return x;
        };
        for (size_t s = 0; s < g.segs.size(); ++s) {
            if (sa[s] < 0) continue;
            const int a = root(sa[s]), b = root(na + sb[s]);
            if (a != b) parent[a] = b;
        }
        std::vector<int64_t> comp_off(na + nb, -1);
        std::vector<int> comp_k(na + nb, -1);
        auto assign = [&](View &v, int id) {
            const int c = root(id);
            if (comp_off[c] < 0) {
                comp_off[c] = g.k_scales;
                comp_k[c] = v.K;
                g.k_scales += v.K;
            }
            KV_REQUIRE(comp_k[c] == v.K, KV_EINVAL, "internal: views of one segment component differ in K");
            v.ks = (int)comp_off[c];
        };
        for (int i = 0; i < na; ++i) assign(av[i], i);
        for (int i = 0; i < nb; ++i) assign(bv[i], na + i);
        KV_REQUIRE(g.k_scales < (1ll << 31), KV_EINVAL, "mixed-precision plan too large");
    }
    // ---- groups
    auto &first = w.first, &of = w.of, &key = w.key;
    {
        w.gtab.reset(blocks.size());
        auto group_of = [&](bool multi) -> Group & {  // the group of `key`, a new one if there is none
            uint64_t h = multi ? 1469598103934665603ull : 0xCBF29CE484222325ull + 2;
            for (int x : key) { h ^= (uint64_t)(uint32_t)x; h *= 1099511628211ull; }
            int &at = w.gtab.find(h, [&](int i) {
                return groups[i].hash == h && groups[i].multi == multi && groups[i].cview == key;
            });
            if (at < 0) {
                at = (int)w.ngroups++;
                if (groups.size() < w.ngroups) groups.emplace_back();
                Group &gr = groups[at];
                gr.rblk.clear();
                gr.cview = key;
                gr.hash = h;
                gr.multi = multi;
            }
            return groups[at];
        };
        // one-segment blocks by A view, in block order
        first.assign(av.size() + 1, 0);
        for (auto &b : blocks)
            if (b.se - b.sb == 1) ++first[sa[b.sb] + 1];
        for (size_t a = 0; a < av.size(); ++a) first[a + 1] += first[a];
        of.resize(first[av.size()]);
        w.fill.assign(first.begin(), first.end() - 1);
        for (size_t b = 0; b < blocks.size(); ++b) {
            const int n = blocks[b].se - blocks[b].sb;
            if (n == 0) zero_blocks.push_back((int)b);
            else if (n == 1) of[w.fill[sa[blocks[b].sb]]++] = (int)b;
            else {
                key.clear();
                for (int s = blocks[b].sb; s < blocks[b].se; ++s) {
                    key.push_back(sb[s]);
                    key.push_back(g.segs[s].entry);
                }
                group_of(true).rblk.push_back((int)b);
            }
        }
        for (size_t a = 0; a < av.size(); ++a) {
            if (first[a] == first[a + 1]) continue;
            key.clear();
            for (int x = first[a]; x < first[a + 1]; ++x) key.push_back(sb[blocks[of[x]].sb]);
            group_of(false).rblk.push_back((int)a);
        }
    }
    // the block of (row unit u, column unit v) of a one-segment group
    auto cell = [&](const Group &gr, int u, int v) -> const OutBlock & { return blocks[of[first[gr.rblk[u]] + v]]; };
    // ---- rows per tile: estimated clocks of the busiest SM.  A K panel costs
    // its operand bytes at about 45 B per clock or the MMAs' shared-memory
    // reads, a drain about 1800 clocks, a tile 600 more (measured on GB300).
    auto group_rows = [&](const Group &gr) {
        int r = 0;
        for (int u : gr.rblk) r += pad8(gr.multi ? blocks[u].M : av[u].rows);
        return r;
    };
    auto group_cols = [&](const Group &gr) {
        if (gr.multi) return bv[gr.cview[0]].rows;
        int c = 0;
        for (int v : gr.cview) c += pad8(bv[v].rows);
        return c;
    };
    int most = BM;
    {
        auto &gc = w.costs;
        gc.resize(w.ngroups);
        for (size_t x = 0; x < w.ngroups; ++x) {
            const Group &gr = groups[x];
            const int s0 = gr.multi ? blocks[gr.rblk[0]].sb : cell(gr, 0, 0).sb;
            const int ns = gr.multi ? (int)gr.cview.size() / 2 : 1;
            GroupCost c{group_rows(gr), (group_cols(gr) + BN - 1) / BN, 0, 0};
            for (int s = s0; s < s0 + ns; ++s) {
                const int nkc = (g.segs[s].K + BKC - 1) / BKC;
                c.panels += nkc;
                c.drains += (nkc + GKC - 1) / GKC;
            }
            gc[x] = c;
        }
        double best = 0.0;
        const double sms = std::max(1, ctx().num_sms);
        for (int log_r : {7, 6, 5}) {
            const int R = 1 << log_r;
            const double panel = std::max(800.0, (R + BN) * NPL * BKC * 2 / 45.0);
            double sum = 0.0, top = 0.0, n = 0.0;
            for (const GroupCost &c : gc) {
                const double cost = 600.0 + c.panels * panel + c.drains * 1800.0;
                const double tiles = (double)((c.rows + R - 1) >> log_r) * c.col_packs;
                sum += tiles * cost;
                n += tiles;
                top = std::max(top, cost);
            }
            const double t = std::max(top, n > 0 ? std::ceil(n / sms) * (sum / n) : 0.0);
            if (R == 128 || t < 0.97 * best) {
                best = t;
                most = R;
            }
        }
    }
    // ---- packs (shared where the same pieces recur), tiles, maps, pairs
    auto &ajobs = w.ajobs, &bjobs = w.bjobs;
    auto &xsegs = w.xsegs;
    auto &tiles = w.tiles;
    auto &pairs = w.pairs;
    auto &maps = w.maps;
    g.a_planes = g.b_planes = g.a_exps = g.b_exps = 0;
    w.bfirst.assign(bv.size(), -1);  // single-piece B packs of each view in bpanels, by first column / BN
    // rows of a pack's panel from its pieces; view_of: the view of a piece
    auto add_pack = [&](const Piece *pc, const Piece *pe, int tall, bool is_b, auto view_of) {
        Panel o;
        const std::vector<View> &vw = is_b ? bv : av;
        std::vector<SliceJob> &jobs = is_b ? bjobs : ajobs;
        const int tr = is_b ? BN : tall, K = vw[view_of(*pc)].K, nkc = (K + BKC - 1) / BKC;
        o.pan = is_b ? g.b_planes : g.a_planes;
        o.exp = (int)(is_b ? g.b_exps : g.a_exps);
        o.job0 = (int)jobs.size();
        o.njobs = (int)(pe - pc);
        int r0 = 0;
        for (; pc != pe; ++pc) {
            const View &v = vw[view_of(*pc)];
            KV_REQUIRE(v.K == K, KV_EINVAL, "internal: a pack's views differ in K");
            jobs.push_back(SliceJob{v.off, o.pan, pc->r0, pc->rows, r0, tr, v.K, v.ld, v.trans, v.conj, o.exp + r0, nkc,
                                    kAllSteps, v.ks});
            r0 += pad8(pc->rows);
        }
        (is_b ? g.b_planes : g.a_planes) += (int64_t)nkc * NPL * BKC * tr;
        (is_b ? g.b_exps : g.a_exps) += is_b ? BN : BM;
        return o;
    };
    auto own_view = [](const Piece &pc) { return pc.view; };
    // a pair reads the pack's piece from step `entry` on (before that its block
    // may not hold data yet)
    auto seen = [&](const Panel &p, bool is_b, int piece, int entry) {
        SliceJob &j = (is_b ? bjobs : ajobs)[p.job0 + piece];
        j.entry = std::min(j.entry, entry);
    };
    // (piece, row) of each of n panel rows; packs of one piece of the same rows share
    // a map (a plan of many blocks that do not pack is mostly such)
    struct {
        int r0, rows, n, at;
    } last[2] = {{0, -1, 0, 0}, {0, -1, 0, 0}};
    auto add_map = [&](const Piece *pc, const Piece *pe, int n, bool is_b) {
        auto &l = last[is_b];
        const bool one = pe - pc == 1;
        if (one && l.r0 == pc->r0 && l.rows == pc->rows && l.n == n) return l.at;
        const int at = (int)maps.size();
        if (one) l = {pc->r0, pc->rows, n, at};
        maps.resize((size_t)at + n);
        int2 *m = maps.data() + at;
        for (int i = 0; pc != pe; ++i, ++pc) {
            int2 *const end = m + pad8(pc->rows);
            for (int r = pc->r0; r < pc->r0 + pc->rows; ++r) *m++ = make_int2(i, r);
            while (m != end) *m++ = make_int2(-1, 0);
        }
        for (int2 *const end = maps.data() + at + n; m != end; ++m) *m = make_int2(-1, 0);
        return at;
    };
    auto &rp = w.rp, &cp = w.cp;
    auto &rpc = w.rpc, &cpc = w.cpc;
    auto &rows = w.rows, &cols = w.cols, &rmap = w.rmap, &cmap = w.cmap;
    auto &ap = w.ap, &bp = w.bp;
    for (size_t x = 0; x < w.ngroups; ++x) {
        const Group &gr = groups[x];
        rows.clear();
        if (!gr.multi && gr.rblk.size() == 1 && gr.cview.size() == 1 && av[gr.rblk[0]].rows <= most &&
            bv[gr.cview[0]].rows <= BN) {  // one block, one tile
            const OutBlock &b = cell(gr, 0, 0);
            const int e = g.segs[b.sb].entry;
            const Piece r{gr.rblk[0], 0, b.M, 0}, c{gr.cview[0], 0, b.N, 0};
            const Panel a1 = add_pack(&r, &r + 1, pad8(b.M), false, own_view);
            const Panel b1 = add_pack(&c, &c + 1, BN, true, own_view);
            ajobs[a1.job0].entry = bjobs[b1.job0].entry = e;
            tiles.push_back({pad8(b.M), (int)xsegs.size(), (int)xsegs.size() + 1, add_map(&r, &r + 1, pad8(b.M), false),
                             add_map(&c, &c + 1, BN, true), (int)pairs.size(), 1});
            xsegs.push_back(SegX{a1.pan, b1.pan, (av[r.view].K + BKC - 1) / BKC, a1.exp, b1.exp, e});
            pairs.push_back({b.c_off, b.ldc, e});
            continue;
        }
        if (!gr.multi) {
            for (int a : gr.rblk) rows.push_back(av[a].rows);
            make_packs(gr.rblk, rows, most, &rp, &rpc);
            cols.clear();
            for (int v : gr.cview) cols.push_back(bv[v].rows);
            make_packs(gr.cview, cols, BN, &cp, &cpc);
            ap.clear(), bp.clear(), rmap.clear(), cmap.clear();
            for (auto &p : rp) {
                ap.push_back(add_pack(rpc.data() + p.begin, rpc.data() + p.end, p.rows, false, own_view));
                rmap.push_back(add_map(rpc.data() + p.begin, rpc.data() + p.end, p.rows, false));
            }
            for (auto &p : cp) {
                bp.push_back(add_pack(cpc.data() + p.begin, cpc.data() + p.end, p.rows, true, own_view));
                cmap.push_back(add_map(cpc.data() + p.begin, cpc.data() + p.end, BN, true));
            }
            const int nkc = (av[gr.rblk[0]].K + BKC - 1) / BKC;
            // kColBatch column packs meet every row pack before the next ones, so
            // the panels of the tiles in flight stay in L2 (all columns a row pack
            // at a time read B's panels from HBM once per row pack)
            constexpr size_t kColBatch = 16;
            int ns = (int)xsegs.size(), nt = (int)tiles.size(), np = (int)pairs.size();
            xsegs.resize(ns + rp.size() * cp.size());
            tiles.resize(nt + rp.size() * cp.size());
            pairs.resize(np + rpc.size() * cpc.size());
            for (size_t j0 = 0; j0 < cp.size(); j0 += kColBatch)
                for (size_t i = 0; i < rp.size(); ++i)
                    for (size_t j = j0; j < std::min(cp.size(), j0 + kColBatch); ++j) {
                        tiles[nt++] = {rp[i].rows, ns, ns + 1, rmap[i], cmap[j], np, cp[j].end - cp[j].begin};
                        int entry = kAllSteps;
                        for (int u = rp[i].begin; u < rp[i].end; ++u)
                            for (int v = cp[j].begin; v < cp[j].end; ++v) {
                                const OutBlock &b = cell(gr, rpc[u].unit, cpc[v].unit);
                                const int e = g.segs[b.sb].entry;
                                pairs[np++] = {b.c_off, b.ldc, e};
                                entry = std::min(entry, e);
                                seen(ap[i], false, u - rp[i].begin, e);
                                seen(bp[j], true, v - cp[j].begin, e);
                            }
                        xsegs[ns++] = SegX{ap[i].pan, bp[j].pan, nkc, ap[i].exp, bp[j].exp, entry};
                    }
            continue;
        }
        for (int b : gr.rblk) rows.push_back(blocks[b].M);
        make_packs(gr.rblk, rows, most, &rp, &rpc);  // pieces name blocks here
        const int ns = (int)gr.cview.size() / 2, N = bv[gr.cview[0]].rows, nb = (N + BN - 1) / BN;
        cmap.clear();
        for (int n0 = 0; n0 < N; n0 += BN) {
            const Piece c{0, n0, std::min(BN, N - n0), 0};
            cmap.push_back(add_map(&c, &c + 1, BN, true));
        }
        for (size_t i = 0; i < rp.size(); ++i) {
            const Piece *p0 = rpc.data() + rp[i].begin, *p1 = rpc.data() + rp[i].end;
            const int rm = add_map(p0, p1, rp[i].rows, false);
            ap.clear();
            for (int s = 0; s < ns; ++s)
                ap.push_back(add_pack(p0, p1, rp[i].rows, false,
                                      [&](const Piece &pc) { return sa[blocks[pc.view].sb + s]; }));
            for (int n0 = 0; n0 < N; n0 += BN) {
                TcTile t{rp[i].rows, (int)xsegs.size(), (int)xsegs.size() + ns, rm, cmap[n0 / BN], (int)pairs.size(), 1};
                int entry = kAllSteps;
                for (int s = 0; s < ns; ++s) {
                    const GemmSeg &sg = g.segs[blocks[gr.rblk[0]].sb + s];
                    const int v = gr.cview[2 * s];
                    if (w.bfirst[v] < 0) {
                        w.bfirst[v] = (int)w.bpanels.size();
                        w.bpanels.resize(w.bpanels.size() + nb, Panel{0, 0, 0, 0});
                    }
                    Panel &pb = w.bpanels[w.bfirst[v] + n0 / BN];
                    if (pb.njobs == 0) {
                        const Piece c{v, n0, std::min(BN, N - n0), 0};
                        pb = add_pack(&c, &c + 1, BN, true, own_view);
                    }
                    xsegs.push_back(SegX{ap[s].pan, pb.pan, (sg.K + BKC - 1) / BKC, ap[s].exp, pb.exp, sg.entry});
                    for (int y = 0; y < ap[s].njobs; ++y) seen(ap[s], false, y, sg.entry);
                    seen(pb, true, 0, sg.entry);
                    entry = std::min(entry, sg.entry);
                }
                for (const Piece *u = p0; u != p1; ++u) {
                    const OutBlock &b = blocks[gr.rblk[u->unit]];
                    pairs.push_back({b.c_off, b.ldc, entry});
                }
                tiles.push_back(t);
            }
        }
    }
    for (int z : zero_blocks) {  // written as zeros (or skipped) by tiles without segments
        const OutBlock &b = blocks[z];
        for (int m0 = 0; m0 < b.M; m0 += BM)
            for (int n0 = 0; n0 < b.N; n0 += BN) {
                const Piece r{0, m0, std::min(BM, b.M - m0), 0}, c{0, n0, std::min(BN, b.N - n0), 0};
                const int rm = add_map(&r, &r + 1, pad8(r.rows), false), cm = add_map(&c, &c + 1, BN, true);
                tiles.push_back(TcTile{pad8(r.rows), (int)xsegs.size(), (int)xsegs.size(), rm, cm,
                                       (int)pairs.size(), 1});
                pairs.push_back({b.c_off, b.ldc, kAllSteps});
            }
    }
    auto &aitems = w.aitems, &bitems = w.bitems;
    auto add_items = [](const std::vector<SliceJob> &jobs, std::vector<int2> &items) {
        size_t n = 0;
        for (auto &j : jobs) n += (j.rows + 7) / 8;
        items.resize(n);
        int2 *o = items.data();
        for (size_t i = 0; i < jobs.size(); ++i)
            for (int r0 = 0; r0 < jobs[i].rows; r0 += 8) *o++ = make_int2((int)i, r0);
    };
    add_items(ajobs, aitems);
    add_items(bjobs, bitems);
    KV_REQUIRE(g.a_exps < (1ll << 31) && g.b_exps < (1ll << 31) && maps.size() < (1ull << 31) &&
                   pairs.size() < (1ull << 31),
               KV_EINVAL, "mixed-precision plan too large");
    g.tc_tiles = (int)tiles.size();
    g.na_items = (int)aitems.size();
    g.nb_items = (int)bitems.size();
    UploadPack u;
    u.add(g.d_tctiles, tiles);
    u.add(g.d_xsegs, xsegs);
    u.add(g.d_maps, maps);
    u.add(g.d_pairs, pairs);
    u.add(g.d_ajobs, ajobs);
    u.add(g.d_bjobs, bjobs);
    u.add(g.d_aitems, aitems);
    u.add(g.d_bitems, bitems);
    g.d_lists = u.upload();
    if (w.bytes() > kScratchBytes) kept = Scratch{};
}

// Per device: the cooperative slicing grid (every CTA resident at once; 0:
// cooperative launches unavailable) and the largest slicing cluster (16, else 8).
struct SliceLimits {
    int grid = 0, cluster = 0;
};
static SliceLimits slice_limits(int device) {
    static std::mutex mu;
    static SliceLimits lim[kMaxDevices];
    KV_REQUIRE(device >= 0 && device < kMaxDevices, KV_EINVAL, "device index out of range");
    std::lock_guard<std::mutex> lk(mu);
    SliceLimits &l = lim[device];
    if (l.cluster == 0) {
        int coop = 0, per_sm = 0, sms = 0;
        KV_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device));
        KV_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
        KV_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_slice_coop, 32 * kSliceWarps, 0));
        l.grid = coop ? per_sm * sms : 0;
        int n = 0;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(16);
        cfg.blockDim = dim3(32 * kSliceWarps);
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = 16;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        const bool ok = cudaFuncSetAttribute((const void *)k_slice_cluster,
                                             cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                        cudaOccupancyMaxActiveClusters(&n, (const void *)k_slice_cluster, &cfg) == cudaSuccess && n > 0;
        if (!ok) (void)cudaGetLastError();
        l.cluster = ok ? 16 : 8;
    }
    return l;
}

// The context's balancing maxima, at least n of them, all zero between calls:
// k_gemm_tc clears what its slicing filled.  Freed with the context.
static int *context_kmax(int64_t n) {
    Context &c = ctx();
    if (c.kmax_n < n) {
        if (c.kmax) KV_CUDA(cudaFreeAsync(c.kmax, c.stream));
        c.kmax = nullptr;
        c.kmax_n = 0;
        const int64_t want = std::max<int64_t>(2 * n, 4096);
        KV_CUDA(cudaMallocAsync(reinterpret_cast<void **>(&c.kmax), want * sizeof(int), c.stream));
        KV_CUDA(cudaMemsetAsync(c.kmax, 0, want * sizeof(int), c.stream));
        c.kmax_n = want;
    }
    return c.kmax;
}

// The context's workspace for sliced panels, at least `bytes` of it; null beyond
// kKeepSlices (such panels are allocated per call).  A context's calls follow
// one another on its stream, so one workspace serves them all; it is freed with
// the context.  Four stream-ordered allocations and frees per GEMM were a
// third of the host's time per call, and contended between worker threads.
constexpr int64_t kKeepSlices = 64ll << 20;
static char *context_slices(int64_t bytes) {
    Context &c = ctx();
    if (bytes > kKeepSlices) return nullptr;
    if (c.slices_n < bytes) {
        if (c.slices) KV_CUDA(cudaFreeAsync(c.slices, c.stream));
        c.slices = nullptr;
        c.slices_n = 0;
        const int64_t want = std::min(kKeepSlices, std::max<int64_t>(2 * bytes, 1 << 20));
        KV_CUDA(cudaMallocAsync(reinterpret_cast<void **>(&c.slices), (size_t)want, c.stream));
        c.slices_n = want;
    }
    return c.slices;
}

void launch_gemm_mixed(const GemmPlan &p, const double2 *A, const double2 *B, double2 *C, double alpha,
                       const int *skip, int step) {
    if (p.tiles.empty()) return;
    KV_REQUIRE(p.tile_m == kMixedBlock && p.tile_n == kMixedBlock && p.tc_tiles > 0, KV_EINVAL,
               "internal: GEMM plan not prepared for the tensor-core path");
    auto &c = ctx();
    int *err = device_err_word(c.device);
    auto up = [](int64_t b) { return (b + 255) & ~(int64_t)255; };
    const int64_t o_bp = up(p.a_planes * (int64_t)sizeof(__half)), o_ae = o_bp + up(p.b_planes * (int64_t)sizeof(__half)),
                  o_be = o_ae + up(p.a_exps * (int64_t)sizeof(int)),
                  bytes = o_be + up(p.b_exps * (int64_t)sizeof(int)) + 256;
    DevBuf large;  // panels beyond the context's workspace
    char *ws = context_slices(bytes);
    if (!ws) {
        large.alloc((size_t)bytes);
        ws = large.as<char>();
    }
    __half *const aph = reinterpret_cast<__half *>(ws), *const bph = reinterpret_cast<__half *>(ws + o_bp);
    int *const aex = reinterpret_cast<int *>(ws + o_ae), *const bex = reinterpret_cast<int *>(ws + o_be);
    int n = 0;
    const bool bal = p.balance_k && p.k_scales > 0 && p.na_items > 0 && p.nb_items > 0;
    const int nkmax = bal ? (int)(2 * p.k_scales) : 0;
    SliceArgs a{p.d_ajobs.as<SliceJob>(), p.d_bjobs.as<SliceJob>(), p.d_aitems.as<int2>(), p.d_bitems.as<int2>(),
                p.na_items, p.nb_items, A, B, aph, bph, aex, bex, alpha, step, err,
                 bal ? context_kmax(nkmax) : nullptr, p.k_scales};
    const int items = p.na_items + p.nb_items;
    if (items > 0) {
        // two K steps of 8 a warp where the longest K allows
        int GW = 1;
        while (GW < kSliceWarps && GW * 16 < p.max_k) GW *= 2;
        const int per = kSliceWarps / GW, ctas = (items + per - 1) / per;
        const SliceLimits lim = slice_limits(c.device);
        const bool main = &c == &main_ctx();
        // Little work, at most two rounds of four steps a warp: one cluster, whose
        // barrier is cheaper than a grid's or a second launch.  More: the whole chip,
        // on the main stream in one cooperative launch (that stream's kernels never
        // overlap, so its grid barrier waits on no other launch).  Measured, us a step
        // with up to 0, 1, 2, 3, 4 and 6 rounds in a cluster: one chain on the main
        // stream, D = 32 one-site 28830, 26860, 26761, 26880, 26837, 26878; D = 96 two-site
        // 91121, 89960, 89831, 90134, 91598, 93476; four chains on worker streams,
        // D = 32 35412, 33615, 34018, 34548, 34728, 34295; D = 96 two-site 121025, 121727,
        // 122222, 122440, 123079, 125065; D = 128 two-site 148949, 148314, 147041, 148498,
        // 148834, 153003.
        const int64_t rounds = (int64_t)((ctas + lim.cluster - 1) / lim.cluster) * ((p.max_k + 32 * GW - 1) / (32 * GW));
        if (!a.kmax) {
            launch_dependent(k_slice_put, (unsigned)ctas, 32 * kSliceWarps, 0, 0, a, GW, skip);
            ++n;
        } else if (rounds <= 2) {
            int size = 1;
            while (size < lim.cluster && size < ctas) size *= 2;
            launch_dependent(k_slice_cluster, (unsigned)size, 32 * kSliceWarps, 0, (unsigned)size, a, GW, skip);
            ++n;
        } else if (main && lim.grid > 0) {
            void *args[] = {&a, &GW, &skip};
            KV_CUDA(cudaLaunchCooperativeKernel((const void *)k_slice_coop, dim3((unsigned)std::min(ctas, lim.grid)),
                                                dim3(32 * kSliceWarps), args, 0, c.stream));
            ++n;
        } else {
            launch_dependent(k_slice_max, (unsigned)ctas, 32 * kSliceWarps, 0, 0, a, GW, skip);
            launch_dependent(k_slice_put, (unsigned)ctas, 32 * kSliceWarps, 0, 0, a, GW, skip);
            n += 2;
        }
    }
    // persistent: one CTA per SM at most (the kernel holds all of an SM's tensor memory)
    const int ntiles = p.tc_tiles;
    launch_dependent(k_gemm_tc, (unsigned)std::min(ntiles, c.num_sms), NTHREADS, SMEM_BYTES, 0,
                     p.d_tctiles.as<TcTile>(), ntiles, p.d_xsegs.as<SegX>(), p.d_maps.as<int2>(),
                     p.d_pairs.as<TcPair>(), aph, bph, aex, bex, C, skip, err, step, p.write_inactive ? 1 : 0,
                     g_stall_test ? (1ll << 10) : WAIT_LIMIT, g_stall_test, a.kmax, nkmax);
    counted(n + 1);
    // large panels are freed stream-ordered after the GEMM
}

// KV_ETIMEOUT if a tensor-core wait gave up, else KV_ENONFINITE if an operand
// held an Inf or NaN, since the last call on this device (then cleared)
int mixed_gemm_status() {
    const int dev = ctx().device;
    int *e = nullptr;
    {
        std::lock_guard<std::mutex> lk(g_dev_mu);
        if (dev >= 0 && dev < kMaxDevices) e = g_err[dev];
    }
    if (!e) return KV_OK;
    int h = 0;
    KV_CUDA(cudaMemcpy(&h, e, sizeof(int), cudaMemcpyDeviceToHost));
    if (h) KV_CUDA(cudaMemset(e, 0, sizeof(int)));
    return (h & kErrTimeout) ? KV_ETIMEOUT : (h & kErrNonFinite) ? KV_ENONFINITE : KV_OK;
}

void set_gemm_stall_test(int on) { g_stall_test = on ? 1 : 0; }

}  // namespace kv
