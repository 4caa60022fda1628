// FP64 device kernels of the contraction engine: grouped block-sparse complex
// GEMM, MPO mixing, block permutation, fills.
#include <algorithm>
#include <cmath>

#include "kv_internal.h"
#include "kv_permute.cuh"

namespace kv {

namespace {

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ void cfma(double2 &acc, double2 a, double2 b) {
    acc.x = fma(a.x, b.x, acc.x);
    acc.x = fma(-a.y, b.y, acc.x);
    acc.y = fma(a.x, b.y, acc.y);
    acc.y = fma(a.y, b.x, acc.y);
}

// ------------------------------------------------------------------ GEMM
// Grouped FP64 GEMM: one CTA per output tile of tm x tn elements (tm tn <=
// NT), each output summed by KS = NT / (tm tn) threads that share the tile's
// K range: the contracted indices of all its segments are numbered
// consecutively and thread slice ks takes those equal to ks mod KS; the KS
// partial sums are added in a fixed tree, so the order is fixed and there are
// no atomics.
// What bounds it: the FP64 unit.  Measured on GB300: a warp's FP64 instruction
// takes 19 clocks of the SM (64 of one warp's time), whatever its active
// lanes, and a complex multiply-add is four, so an operand pair read from
// L1/L2 for every multiply-add is hidden and neither register blocking nor
// shared-memory staging helps; what matters is that all SMs hold equal
// shares of the multiply-adds.  The plan (fp64_tiles) therefore sizes tiles
// by their work, and blocks smaller than a tile leave no thread idle (tm, tn
// are any integers).  Against 32 x 32 tiles with K walked by the whole CTA
// (which left most SMs idle): a D = 96 one-site Lanczos exponential 2047 ->
// 788 us, the energy of 36 such sites 7.73 -> 2.33 ms, the adjoint of a D = 96
// apply (one output of K ~ 5000 per SM) 6.06 -> 0.61 ms.
constexpr int kSegBatch = 32;  // segment descriptors staged in shared memory at a time

// v with its sign flipped if flip is 0x80000000 (no FP64 operation)
__device__ __forceinline__ double flip_sign(double v, int flip) {
    return __hiloint2double(__double2hiint(v) ^ flip, __double2loint(v));
}

template <int NT>
__global__ void __launch_bounds__(NT, NT == 32 ? 8 : 1024 / NT) k_gemm_fp64(const GemmTile *__restrict__ tiles,
                                                  const GemmSeg *__restrict__ segs, const double2 *__restrict__ A,
                                                  const double2 *__restrict__ B, double2 *__restrict__ C, double alpha,
                                                  const int *skip, int step, int write_inactive, int cover,
                                                  int serial_k) {
    allow_dependents();
    __shared__ GemmSeg sg[kSegBatch];
    __shared__ double2 red[NT];
    const GemmTile t = tiles[blockIdx.x];
    dependency_wait();
    if (skip && *skip) return;
    const int tid = threadIdx.x;
    const int tm = t.tm, tn = t.tn, mn = tm * tn, KS = serial_k ? 1 : NT / mn;
    const int ks = tid / mn, m = (tid % mn) / tn, n = tid % tn;
    // cover > 0 (coarse task lists): the CTA walks the cover x cover outputs from (m0, n0) in tm x tn steps
    const int m_end = cover > 0 ? min(t.M, t.m0 + cover) : min(t.M, t.m0 + tm);
    const int n_end = cover > 0 ? min(t.N, t.n0 + cover) : min(t.N, t.n0 + tn);
    for (int mb = t.m0; mb < m_end; mb += tm)
        for (int nb = t.n0; nb < n_end; nb += tn) {
            const int gm = mb + m, gn = nb + n;
            const bool on = ks < KS && gm < m_end && gn < n_end;
            double2 acc = make_double2(0.0, 0.0);
            bool any = false;
            int first = ks;  // this slice's first index within the next segment
            for (int s0 = t.seg_begin; s0 < t.seg_end; s0 += kSegBatch) {
                const int ns = min(kSegBatch, t.seg_end - s0);
                __syncthreads();
                for (int i = tid; i < ns; i += NT) sg[i] = segs[s0 + i];
                __syncthreads();
                for (int i = 0; i < ns; ++i) {
                    if (sg[i].entry > step) continue;  // uniform over the CTA
                    any = true;
                    const int K = sg[i].K, lda = sg[i].lda, ldb = sg[i].ldb, opa = sg[i].opa, opb = sg[i].opb;
                    if (on) {
                        const bool akc = opa == 0 || opa == 3, bnc = opb == 0 || opb == 3;  // contiguous along k / n
                        const int fa = (opa == 1 || opa == 3) ? (int)0x80000000 : 0;
                        const int fb = (opb == 2 || opb == 3) ? (int)0x80000000 : 0;
                        const int64_t da = akc ? 1 : lda, db = bnc ? ldb : 1;
                        const double2 *pa = A + sg[i].a_off + (akc ? (int64_t)gm * lda : gm);
                        const double2 *pb = B + sg[i].b_off + (bnc ? gn : (int64_t)gn * ldb);
                        int k = first;
                        if constexpr (NT == 32) {
                            // a warp alone on its chain: UL operand pairs are read
                            // ahead of the UL being multiplied
                            constexpr int UL = 8;
                            const int64_t sa = (int64_t)KS * da, sb = (int64_t)KS * db;
                            const double2 *qa = pa + first * da, *qb = pb + first * db;
                            if (k + (UL - 1) * KS < K) {
                                double2 a[UL], b[UL];
#pragma unroll
                                for (int u = 0; u < UL; ++u) { a[u] = qa[u * sa]; b[u] = qb[u * sb]; }
                                for (; k + (UL - 1) * KS < K; k += UL * KS) {
                                    double2 an[UL], bn[UL];
                                    qa += UL * sa;
                                    qb += UL * sb;
                                    const bool more = k + (2 * UL - 1) * KS < K;
#pragma unroll
                                    for (int u = 0; u < UL; ++u) {
                                        an[u] = more ? qa[u * sa] : make_double2(0.0, 0.0);
                                        bn[u] = more ? qb[u * sb] : make_double2(0.0, 0.0);
                                    }
#pragma unroll
                                    for (int u = 0; u < UL; ++u) {
                                        a[u].y = flip_sign(a[u].y, fa);
                                        b[u].y = flip_sign(b[u].y, fb);
                                        cfma(acc, a[u], b[u]);
                                        a[u] = an[u];
                                        b[u] = bn[u];
                                    }
                                }
                            }
                        }
#pragma unroll 2
                        for (; k < K; k += KS) {
                            double2 a = pa[k * da], b = pb[k * db];
                            a.y = flip_sign(a.y, fa);
                            b.y = flip_sign(b.y, fb);
                            cfma(acc, a, b);
                        }
                    }
                    // (first - K) mod KS: the next segment continues the numbering
                    if (KS > 1) {
                        first = (first - K) % KS;
                        if (first < 0) first += KS;
                    }
                }
            }
            for (int live = KS; live > 1;) {
                const int half = (live + 1) / 2;
                __syncthreads();
                if (ks < live) red[tid] = acc;
                __syncthreads();
                if (ks < live - half) {
                    acc.x += red[tid + half * mn].x;
                    acc.y += red[tid + half * mn].y;
                }
                live = half;
            }
            if (!any && !write_inactive) return;  // uniform over the CTA
            if (on && ks == 0)
                C[t.c_off + (int64_t)gm * t.ldc + gn] = make_double2(alpha * acc.x, alpha * acc.y);
        }
}

// ------------------------------------------------------------------ mix
// out[k, k2, r, n] = sum_terms sum_kk W[k2, kk, r] in[k, kk, n]; one warp per
// item (a chunk of one job's elements).  An MPO's local operators are mostly
// zeros, real, and often the identity: each warp first compacts its job's
// nonzero W entries, in order, into a list per output (k2, r) in shared
// memory, so an element costs one input per nonzero entry (two fused
// multiply-adds if W is real, none for a leading 1).  What bounds it: the
// elements' traffic once the blocks are large (each element is written once
// and about 1.5 inputs are read), the list's chain of loads (job, terms, W)
// where they are small; a warp per item keeps many such chains in flight.
// For finite inputs the sums equal the four-multiply-add product's over all
// entries up to the sign of a zero.
// Measured (us a launch, against one thread an element over all entries): D =
// 128 two-site blocks 35.6 -> 16.4, D = 512 213 -> 76.
constexpr int kMixWarps = 8;    // warps (items) per CTA
constexpr int kMixTerms = 16;   // terms, outputs (k2, r) and nonzero entries a warp's list holds;
constexpr int kMixOuts = 16;    // larger jobs take mix_direct
constexpr int kMixList = 64;

struct MixEntry {
    double2 w;
    int64_t off;  // of the input element at k = n = 0
    int kst;      // input elements per k
    int kind;     // kUnit, kReal or kComplex (an FP64 comparison per element would cost as much as its sum)
};
enum MixKind { kUnit = 0, kReal = 1, kComplex = 2 };
// acc (first: nothing summed yet) plus the entry's share
__device__ __forceinline__ void mix_add(double2 &acc, const MixEntry &en, double2 x, bool first) {
    if (en.kind == kComplex) {
        cfma(acc, en.w, x);
    } else if (first && en.kind == kUnit) {
        acc = x;
    } else {
        acc.x = fma(en.w.x, x.x, acc.x);
        acc.y = fma(en.w.x, x.y, acc.y);
    }
}
struct MixWarp {
    MixEntry list[kMixList];
    MixTerm term[kMixTerms];
    int start[kMixOuts + 1];
};

// one element straight from the plan and W
__device__ __forceinline__ double2 mix_direct(const MixJob &jb, const MixTerm *__restrict__ terms,
                                              const double2 *__restrict__ in, const double2 *__restrict__ W, int step,
                                              int64_t e) {
    const int64_t n = e % jb.rest, r = (e / jb.rest) % jb.wr, k2 = (e / ((int64_t)jb.rest * jb.wr)) % jb.so;
    const int64_t k = e / ((int64_t)jb.rest * jb.wr * jb.so);
    double2 acc = make_double2(0.0, 0.0);
    for (int ti = jb.term_begin; ti < jb.term_end; ++ti) {
        const MixTerm tm = terms[ti];
        if (tm.entry > step) continue;
        const double2 *w = W + tm.w_off + (k2 * tm.K) * jb.wr + r;
        const double2 *x = in + tm.in_off + (k * tm.K) * jb.rest + n;
        for (int kk = 0; kk < tm.K; ++kk) {
            const double2 wv = w[(int64_t)kk * jb.wr];
            if (wv.x != 0.0 || wv.y != 0.0) cfma(acc, wv, x[(int64_t)kk * jb.rest]);
        }
    }
    return acc;
}

__global__ void __launch_bounds__(32 * kMixWarps) k_mix(const MixItem *__restrict__ items, int nitems, int chunk,
                                                        const MixJob *__restrict__ jobs,
                                                        const MixTerm *__restrict__ terms,
                                                        const double2 *__restrict__ in, const double2 *__restrict__ W,
                                                        double2 *__restrict__ out, const int *skip, int step,
                                                        int write_inactive) {
    allow_dependents();
    __shared__ MixWarp sm[kMixWarps];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int item = blockIdx.x * kMixWarps + warp;
    const MixItem it = items[min(item, nitems - 1)];
    const MixJob jb = jobs[it.job];
    dependency_wait();
    if (skip && *skip) return;
    if (item >= nitems) return;  // warp-uniform, as every branch on the item below
    MixWarp &mw = sm[warp];
    const int nt_all = jb.term_end - jb.term_begin, nout = jb.so * jb.wr;
    const int64_t e1 = min(jb.count, it.start + chunk);
    bool listed = nt_all <= kMixTerms && nout <= kMixOuts && jb.count < (1ll << 31);
    int nt = 0, ktot = 0;  // active terms and their contracted indices
    if (listed) {
        MixTerm tm{};
        const bool act = lane < nt_all && (tm = terms[jb.term_begin + lane]).entry <= step;
        const unsigned m = __ballot_sync(0xFFFFFFFFu, act);
        if (act) mw.term[__popc(m & ((1u << lane) - 1))] = tm;
        nt = __popc(m);
        ktot = __reduce_add_sync(0xFFFFFFFFu, act ? tm.K : 0);
        __syncwarp();
        if (nt == 0 && !write_inactive) return;
        // entries (output o, contracted index kp of the active terms), o major, kept where W is not zero
        int used = 0;
        for (int x0 = 0; x0 < nout * ktot && used <= kMixList; x0 += 32) {
            const int x = x0 + lane;
            MixEntry en{};
            bool nz = false;
            int o = 0, kp = 0;
            if (x < nout * ktot) {
                o = x / ktot;
                kp = x - o * ktot;
                int t = 0, kk = kp;
                while (kk >= mw.term[t].K) kk -= mw.term[t++].K;
                const MixTerm &q = mw.term[t];
                const int k2 = o / jb.wr, r = o - k2 * jb.wr;
                en.w = W[q.w_off + ((int64_t)k2 * q.K + kk) * jb.wr + r];
                en.off = q.in_off + (int64_t)kk * jb.rest;
                en.kst = q.K * jb.rest;
                en.kind = en.w.y != 0.0 ? kComplex : en.w.x == 1.0 ? kUnit : kReal;
                nz = en.w.x != 0.0 || en.w.y != 0.0;
            }
            const unsigned b = __ballot_sync(0xFFFFFFFFu, nz);
            const int at = used + __popc(b & ((1u << lane) - 1));
            if (x < nout * ktot && kp == 0) mw.start[o] = at;
            if (nz && at < kMixList) mw.list[at] = en;
            used += __popc(b);
        }
        if (lane == 0) {
            if (ktot == 0)
                for (int o = 0; o < nout; ++o) mw.start[o] = 0;
            mw.start[nout] = used;
        }
        __syncwarp();
        listed = used <= kMixList;
    } else if (!write_inactive) {
        bool any = false;
        for (int ti = jb.term_begin + lane; ti < jb.term_end; ti += 32) any = any || terms[ti].entry <= step;
        if (!__any_sync(0xFFFFFFFFu, any)) return;
    }
    if (!listed) {
        for (int64_t e = it.start + lane; e < e1; e += 32) out[jb.out_off + e] = mix_direct(jb, terms, in, W, step, e);
        return;
    }
    const unsigned rest = (unsigned)jb.rest, no = (unsigned)nout, ee = (unsigned)e1;
    if (rest > 64) {  // row by row: each entry is read once for up to 4 elements a lane
        for (unsigned e = (unsigned)it.start; e < ee;) {
            const unsigned row = e / rest, n0 = e - row * rest, k = row / no, o = row - k * no;
            const unsigned len = min(min(rest - n0, ee - e), 128u);
            const int i0 = mw.start[o], i1 = mw.start[o + 1];
            double2 acc[4] = {};
            for (int i = i0; i < i1; ++i) {
                const MixEntry &en = mw.list[i];
                const double2 *x = in + en.off + (int64_t)k * en.kst + n0;
                double2 v[4] = {};
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (lane + 32 * j < len) v[j] = x[lane + 32 * j];
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (32 * j < len) mix_add(acc[j], en, v[j], i == i0);
            }
            double2 *y = out + jb.out_off + e;
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (lane + 32 * j < len) y[lane + 32 * j] = acc[j];
            e += len;
        }
        return;
    }
    if (rest > 16) {  // two rows at a time, up to 64 elements of each: four loads in flight a lane
        const unsigned r1 = (ee - 1) / rest;
        for (unsigned row = (unsigned)it.start / rest; row <= r1; row += 2) {
            unsigned k[2];
            int i0[2], cnt[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                k[u] = (row + u) / no;
                const unsigned o = row + u - k[u] * no;
                i0[u] = mw.start[o];
                cnt[u] = row + u <= r1 ? mw.start[o + 1] - i0[u] : 0;
            }
            double2 acc[2][2] = {};
            const int most = max(cnt[0], cnt[1]);
            for (int t = 0; t < most; ++t) {
                double2 v[2][2] = {};
#pragma unroll
                for (int u = 0; u < 2; ++u)
                    if (t < cnt[u]) {
                        const double2 *x = in + mw.list[i0[u] + t].off + (int64_t)k[u] * mw.list[i0[u] + t].kst;
                        if (lane < rest) v[u][0] = x[lane];
                        if (lane + 32 < rest) v[u][1] = x[lane + 32];
                    }
#pragma unroll
                for (int u = 0; u < 2; ++u)
                    if (t < cnt[u]) {
                        mix_add(acc[u][0], mw.list[i0[u] + t], v[u][0], t == 0);
                        if (rest > 32) mix_add(acc[u][1], mw.list[i0[u] + t], v[u][1], t == 0);
                    }
            }
#pragma unroll
            for (int u = 0; u < 2; ++u)
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const unsigned n = lane + 32 * j, e = (row + u) * rest + n;
                    if (n < rest && e >= (unsigned)it.start && e < ee) out[jb.out_off + e] = acc[u][j];
                }
        }
        return;
    }
#pragma unroll 2
    for (unsigned e = (unsigned)it.start + lane; e < ee; e += 32) {
        const unsigned row = e / rest, n = e - row * rest, k = row / no, o = row - k * no;
        double2 acc = make_double2(0.0, 0.0);
        const int i0 = mw.start[o], i1 = mw.start[o + 1];
        for (int i = i0; i < i1; ++i) {
            const MixEntry &en = mw.list[i];
            mix_add(acc, en, in[en.off + (int64_t)k * en.kst + n], i == i0);
        }
        out[jb.out_off + e] = acc;
    }
}

// ------------------------------------------------------------ permute
// desc per block (16 int64): in_off, out_off, size, rank, shape[6], perm[6].
// A CTA takes kPermChunk elements of a block at a time (blockIdx.y, striding
// over the grid), so a tensor of one large block uses the whole chip; 32-bit
// index divisions; an identity permutation is a copy.  A latency-bound copy for
// small blocks: 98 -> 9 us for one of 96 x 5 x 12 x 96 x 5 elements a CTA walked
// alone.
constexpr int kPermChunk = 1024;
static_assert(kMaxRank == kvp::kRank, "axes of a block");
__global__ void __launch_bounds__(256) k_permute(const int64_t *__restrict__ desc, const double2 *__restrict__ in,
                                                 double2 *__restrict__ out) {
    const int64_t *d = desc + 16 * blockIdx.x;
    const int64_t in_off = d[0], out_off = d[1], size = d[2];
    const int rank = (int)d[3];
    if ((int64_t)blockIdx.y * kPermChunk >= size) return;
    const kvp::PermMap map = kvp::perm_map(d + 4, d + 10, rank);
    const bool wide = size >= (1ll << 31);
    for (int64_t c0 = (int64_t)blockIdx.y * kPermChunk; c0 < size; c0 += (int64_t)gridDim.y * kPermChunk) {
        const int64_t c1 = min(size, c0 + kPermChunk);
        for (int64_t e = c0 + threadIdx.x; e < c1; e += 256)
            out[out_off + kvp::perm_index(map, rank, e, wide)] = in[in_off + e];
    }
}

__global__ void k_zero(double2 *p, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        p[i] = make_double2(0.0, 0.0);
}
__global__ void k_copy(double2 *dst, const double2 *src, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        dst[i] = src[i];
}

int grid_for(int64_t n, int threads) {
    int64_t g = (n + threads - 1) / threads;
    int cap = std::max(1, ctx().num_sms * 8);
    return (int)std::max<int64_t>(1, std::min<int64_t>(g, cap));
}

}  // namespace

// Tiles of the FP64 GEMM from one entry per output block (m0 = n0 = 0,
// covering the block).  A tile's cost is its multiply-adds, outputs x K; tiles
// are cut so that none exceeds a quarter of an SM's share of the plan, or
// kMinTile multiply-adds (about 1 us of one SM's FP64 unit, what a CTA costs
// to start), and never more than 256 outputs.  serial_k plans (one thread per
// output, so each sum runs over k in order) take one warp a tile, shaped to
// need the fewest warps.
void fp64_tiles(GemmPlan &g) {
    constexpr double kMinTile = 1024.0;
    std::vector<GemmTile> blocks;
    blocks.swap(g.tiles);
    std::vector<double> K(blocks.size(), 0.0);
    double total = 0.0, top = 0.0;
    int most = 1;
    for (size_t i = 0; i < blocks.size(); ++i) {
        const GemmTile &b = blocks[i];
        for (int s = b.seg_begin; s < b.seg_end; ++s) K[i] += g.segs[s].K;
        total += K[i] * b.M * b.N;
    }
    const double target = std::max(kMinTile, total / (4.0 * std::max(1, ctx().num_sms)));
    for (size_t i = 0; i < blocks.size(); ++i) {
        const GemmTile &b = blocks[i];
        const int area = (int)std::max(1.0, std::min(256.0, target / std::max(1.0, K[i])));
        // nearly square, cut into equal parts
        int tn = std::min(b.N, std::max(1, (int)std::sqrt((double)area)));
        int tm = std::min(b.M, std::max(1, area / tn));
        tn = std::min(b.N, std::max(1, area / tm));
        if (g.serial_k) {
            int64_t fewest = INT64_MAX;
            for (int x = 1; x <= std::min(32, b.N); ++x) {
                const int y = std::min(b.M, 32 / x);
                const int64_t warps = (int64_t)((b.M + y - 1) / y) * ((b.N + x - 1) / x);
                if (warps < fewest) { fewest = warps; tn = x; tm = y; }
            }
        } else {
            tm = (b.M + (b.M + tm - 1) / tm - 1) / ((b.M + tm - 1) / tm);
            tn = (b.N + (b.N + tn - 1) / tn - 1) / ((b.N + tn - 1) / tn);
        }
        GemmTile t = b;
        t.tm = (short)tm;
        t.tn = (short)tn;
        for (t.m0 = 0; t.m0 < b.M; t.m0 += tm)
            for (t.n0 = 0; t.n0 < b.N; t.n0 += tn) g.tiles.push_back(t);
        top = std::max(top, (double)tm * tn * K[i]);
        most = std::max(most, tm * tn);
    }
    if (g.serial_k) g.fp64_threads = 32;
    else g.fp64_threads = top <= 2.0 * kMinTile && most <= 64 ? 64 : 256;
}

void launch_gemm_fp64(const GemmPlan &p, const double2 *A, const double2 *B, double2 *C, double alpha,
                      const int *skip, int step) {
    if (p.tiles.empty()) return;
    KV_REQUIRE(p.tile_m == p.tile_n && (p.tile_m == kFp64Block || p.tile_m == kFp64Coarse), KV_EINVAL,
               "internal: GEMM plan not prepared for the FP64 path");
    const int cover = p.tile_m == kFp64Coarse ? kFp64Coarse : 0;
    const unsigned n = (unsigned)p.tiles.size();
    auto launch = [&](auto kernel, int threads) {
        launch_dependent(kernel, n, (unsigned)threads, 0, 0, p.d_tiles.as<GemmTile>(), p.d_segs.as<GemmSeg>(), A, B, C,
                         alpha, skip, step, p.write_inactive ? 1 : 0, cover, p.serial_k ? 1 : 0);
    };
    if (p.fp64_threads == 32) launch(k_gemm_fp64<32>, 32);
    else if (p.fp64_threads == 64) launch(k_gemm_fp64<64>, 64);
    else launch(k_gemm_fp64<256>, 256);
    counted();
}

void launch_mix(const MixPlan &p, const double2 *in, const double2 *W, double2 *out, const int *skip, int step) {
    if (p.items.empty()) return;
    const int n = (int)p.items.size();
    launch_dependent(k_mix, (unsigned)((n + kMixWarps - 1) / kMixWarps), 32 * kMixWarps, 0, 0, p.d_items.as<MixItem>(),
                     n, p.chunk, p.d_jobs.as<MixJob>(), p.d_terms.as<MixTerm>(), in, W, out, skip, step,
                     p.write_inactive ? 1 : 0);
    counted();
}

void launch_permute(const double2 *in, double2 *out, const std::vector<int64_t> &desc, int nblocks) {
    if (nblocks == 0) return;
    DevBuf d = upload_vec(desc);
    int64_t most = 1;
    for (int b = 0; b < nblocks; ++b) most = std::max(most, desc[16 * (size_t)b + 2]);
    // enough CTAs a block for its chunks, no more in all than eight waves of the chip need
    const int64_t chunks = (most + kPermChunk - 1) / kPermChunk;
    const unsigned gy = (unsigned)std::min<int64_t>(chunks, std::max<int64_t>(1, 64ll * ctx().num_sms / nblocks));
    k_permute<<<dim3((unsigned)nblocks, gy), 256, 0, ctx().stream>>>(d.as<int64_t>(), in, out);
    counted();
    KV_CUDA(cudaGetLastError());
    // d is freed stream-ordered after the kernel
}

void launch_zero(double2 *p, int64_t n) {
    if (n <= 0) return;
    k_zero<<<grid_for(n, 256), 256, 0, ctx().stream>>>(p, n);
    counted();
    KV_CUDA(cudaGetLastError());
}

void launch_copy(double2 *dst, const double2 *src, int64_t n) {
    if (n <= 0) return;
    k_copy<<<grid_for(n, 256), 256, 0, ctx().stream>>>(dst, src, n);
    counted();
    KV_CUDA(cudaGetLastError());
}

}  // namespace kv
