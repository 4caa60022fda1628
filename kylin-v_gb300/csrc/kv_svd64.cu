// FP64 block SVD (svd_impl's factorisation, holstein/svd.h:296-440, in FP64
// mode; the SA-1TDVP split, holstein/svd.h:443-614, in every mode): for each
// charge sector T (p x q, column-major) the p-dimensional left singular
// vectors and the singular values, sorted.  The caller orients T so that these
// are the factor it keeps orthonormal and forms the other factor as the
// projection of the sector matrix onto them.
//
// One thread-block cluster per sector:
//  0. T is scaled by the power of two that brings its largest real or imaginary
//     part to [0.5, 1) (undone on the singular values), so that squared norms
//     neither overflow nor underflow whatever the amplitude of the sector.
//  1. Pivoted Householder reduction of T's rows from the right: at step k the
//     row with the largest trailing norm is reflected onto its position k and
//     the reflector applied to the rows not yet pivoted, so T Q = M is
//     row-pivoted lower triangular (p x r, r <= min(p, q); r is smaller only
//     if the remaining rows are shorter than 1e-130 of the largest element:
//     kNormFloor) and T's left vectors are M's.
//     One-sided Jacobi on such a graded triangular factor converges in fewer
//     sweeps than on T, and a wide T loses its surplus columns (Drmac and
//     Veselic, SIAM J. Matrix Anal. Appl. 29 (2008) 1322).
//  2. One-sided Jacobi on M's columns, round-robin pairs, one barrier a round.
//  3. Column norms = singular values, sorted; normalised columns = vectors.
//     Columns below the floor count as zero, and their vectors are not written;
//     those that a truncation keeps are completed to an orthonormal set
//     (svd_fp64_complete).
//
// What bounds it: the FP64 unit.  GB300 issues two FP64 thread-operations per
// clock per SM, so a warp's FP64 instruction holds its quarter of the SM for
// 64 clocks, and one SM per sector (17 to 32 sectors on 152 SMs) left most of
// the chip idle.  Hence: a cluster of SMs per sector, rows (1) and pairs (2)
// dealt over its SMs, the data in L2 (a round moves a few columns a warp, far
// less time than its arithmetic); no accumulated rotations; sums of several
// values reduced together (each shuffle level halves the values a lane
// carries, then the lanes); and rotation angles from FP32 arithmetic on the
// mantissas -- an angle off by 1e-7 only leaves 1e-7 of the pair's cosine for
// the next sweep -- with (cs, s) completed to a unitary pair in FP64.
// Measured (17 sectors of about 101 x 101, 10 sweeps): 297 ms with one SM a
// sector, accumulated rotations and FP64 angles, 7.5 ms now; the truncated
// product's error against numpy 4.1e-14 -> 2.7e-15.
#include <cooperative_groups.h>

#include <algorithm>
#include <mutex>

#include "kv_internal.h"
#include "kv_rotation64.cuh"
#include "kv_svd.h"

namespace kv {

namespace {

using namespace rot64;

constexpr int NT = 256, NW = NT / 32;
constexpr int kXStage = 4096;  // longest pivot row staged in shared memory

// Squared norms (of the scaled sector) that count as zero.  Above the floor every
// quantity of a reflection or rotation is a normal FP64 number: 1 / |u|^2 <= 1e260,
// and the inner product of two columns at the tolerance is 1e-15 * 1e-260.  The
// squares of such inner products underflow where both columns are short
// (kProductFloor: a b 1e-30 >= 1e-290 above it); those pairs are compared with
// their exponents taken out.
constexpr double kNormFloor = 1e-260, kProductFloor = 1e-130;
// Below it |u_0|^2 gives no phase of modulus one to FP64 rounding (its squares are
// subnormal); u_0 is then under 1e-20 of |u| and is left out of the reflector.
constexpr double kPhaseFloor = 1e-300;

// Data that other CTAs of the cluster read or write goes through L2; a sector of
// one CTA (ONE) keeps it in the SM's L1.
template <bool ONE, class T>
__device__ __forceinline__ T ldg(const T *p) {
    if constexpr (ONE) return *p;
    else return __ldcg(p);
}
template <bool ONE, class T>
__device__ __forceinline__ void stg(T *p, T v) {
    if constexpr (ONE) *p = v;
    else __stcg(p, v);
}

// sums of two / four values over groups of G lanes, every lane of the group
// receiving them: at the first levels a lane passes on half of its values, so
// the four sums cost 2 + 1 + ... additions instead of 4 a level
__device__ __forceinline__ void group_sum2(double &a, double &b, int G) {
    const int lane = threadIdx.x & 31;
    const bool hi = lane & 1;
    double keep = hi ? b : a, give = hi ? a : b;
    keep += __shfl_xor_sync(0xFFFFFFFFu, give, 1);
    for (int o = 2; o < G; o <<= 1) keep += __shfl_xor_sync(0xFFFFFFFFu, keep, o);
    const double other = __shfl_xor_sync(0xFFFFFFFFu, keep, 1);
    a = hi ? other : keep;
    b = hi ? keep : other;
}
template <int G>
__device__ __forceinline__ void group_sum4(double &a, double &b, double &c, double &d) {
    const int lane = threadIdx.x & 31;
    const bool h1 = lane & 1, h2 = lane & 2;
    double k0 = h1 ? c : a, k1 = h1 ? d : b, g0 = h1 ? a : c, g1 = h1 ? b : d;
    k0 += __shfl_xor_sync(0xFFFFFFFFu, g0, 1);
    k1 += __shfl_xor_sync(0xFFFFFFFFu, g1, 1);
    double v = h2 ? k1 : k0;
    v += __shfl_xor_sync(0xFFFFFFFFu, h2 ? k0 : k1, 2);
#pragma unroll
    for (int o = 4; o < G; o <<= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
    // lane bits (h1, h2): (0,0) holds a, (0,1) b, (1,0) c, (1,1) d
    const int base = lane & ~3;
    a = __shfl_sync(0xFFFFFFFFu, v, base);
    c = __shfl_sync(0xFFFFFFFFu, v, base + 1);
    b = __shfl_sync(0xFFFFFFFFu, v, base + 2);
    d = __shfl_sync(0xFFFFFFFFu, v, base + 3);
}

struct Svd64Sector {
    int64_t t_off;   // T, the row workspace and M: p * q elements each
    int64_t s_off;   // q singular values
    int64_t k_off;   // min(p, q) diagonal entries and norms
    int64_t r_off;   // p row flags
    int p, q;
};

// candidate of one CTA for the next pivot row
struct Cand {
    double v;
    int row, bad;
};

template <int G, int EPL, bool ONE>
__global__ void __launch_bounds__(NT) k_svd64(const Svd64Sector *__restrict__ secs, const double2 *__restrict__ T,
                                              double2 *U, double2 *M, double *S, double2 *alph, double *nrm,
                                              int *done, Cand *cand, int *flags, int *status,
                                              int max_sweeps, double tol) {
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    extern __shared__ double2 xs[];  // the pivot row's tail (q <= kXStage)
    __shared__ double wv[NW];
    __shared__ int wi[NW], wbad[NW];
    __shared__ double2 sc[2];  // v0 and (beta, nu) of the step
    __shared__ Cand own[2];    // ONE: the candidates
    auto sync = [&] {
        if constexpr (ONE) __syncthreads();
        else cl.sync();
    };
    auto ldg2 = [](const double2 *p) { return ldg<ONE>(p); };
    auto stg2 = [](double2 *p, double2 v) { stg<ONE>(p, v); };
    const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    const int sec = blockIdx.x / C;
    const Svd64Sector s = secs[sec];
    const int p = s.p, q = s.q, kmax = min(p, q);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const double2 *t = T + s.t_off;
    double2 *w = U + s.t_off;  // row-major workspace, later the sorted vectors
    double2 *m = M + s.t_off;  // column-major p x r
    double2 *al = alph + s.k_off;
    double *nv = nrm + s.k_off;
    int *dn = done + s.r_off;  // step a row was the pivot of, or -1
    Cand *cd = cand + (int64_t)sec * 2 * 16;
    int *fl = flags + sec * 4;

    // best (value, row) of the CTA into slot b; NaN wins, so it is seen
    auto publish = [&](double bv, int bi, int bad, int slot) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const double ov = __shfl_xor_sync(0xFFFFFFFFu, bv, o);
            const int oi = __shfl_xor_sync(0xFFFFFFFFu, bi, o);
            bad |= __shfl_xor_sync(0xFFFFFFFFu, bad, o);
            if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
        }
        if (lane == 0) { wv[warp] = bv; wi[warp] = bi; wbad[warp] = bad; }
        __syncthreads();
        if (tid == 0) {
            for (int x = 1; x < NW; ++x) {
                bad |= wbad[x];
                if (wv[x] > bv || (wv[x] == bv && wi[x] < bi)) { bv = wv[x]; bi = wi[x]; }
            }
            Cand *o = ONE ? own + slot : cd + slot * 16 + rank;
            stg<ONE>(&o->v, bv);
            stg<ONE>(&o->row, bi);
            stg<ONE>(&o->bad, bad);
        }
    };

    // ---- the power of two: the largest exponent, over the cluster by way of the
    // second candidate slot (next written after the barrier that follows its reads)
    int shift;
    {
        int mx = 0;
        const int64_t n = (int64_t)p * q;
        for (int64_t e = (int64_t)rank * NT + tid; e < n; e += (int64_t)C * NT) {
            const double2 v = t[e];
            mx = max(mx, max(__double2hiint(v.x) & 0x7FFFFFFF, __double2hiint(v.y) & 0x7FFFFFFF));
        }
        mx = __reduce_max_sync(0xFFFFFFFFu, mx);
        if (lane == 0) wi[warp] = mx;
        __syncthreads();
        if (tid == 0) {
            for (int x = 1; x < NW; ++x) mx = max(mx, wi[x]);
            stg<ONE>(ONE ? &own[1].row : &cd[16 + rank].row, mx);
        }
        sync();
        mx = 0;
        for (int x = 0; x < C; ++x) mx = max(mx, ldg<ONE>(ONE ? &own[1].row : &cd[16 + x].row));
        const int E = mx >> 20;
        shift = E == 0x7FF ? 0 : 1022 - max(E, 1);  // a non-finite sector is found by its row norms
    }

    // ---- rows i = rank, rank + C, ... belong to this CTA.  A group of lanes takes
    // a row, as many as the row's length keeps busy: a warp's FP64 instruction
    // costs the same for idle lanes.
    auto lanes_for = [](int n) { return n > 64 ? 32 : n > 24 ? 16 : n > 8 ? 8 : 4; };
    {
        double bv = -1.0;
        int bi = 0x7FFFFFFF, bad = 0;
        const int GQ = lanes_for(q), RW = 32 / GQ, sub = lane / GQ, gl = lane % GQ;
        const double up = scalbn(1.0, shift);  // 2^-1024 ... 2^1021: the products are exact
        for (int base = warp * RW; rank + C * base < p; base += NW * RW) {  // warp-uniform
            const int i = rank + C * (base + sub);
            double a = 0.0;
            if (i < p)
                for (int c = gl; c < q; c += GQ) {
                    double2 v = t[i + (int64_t)c * p];
                    v.x *= up;
                    v.y *= up;
                    w[(int64_t)i * q + c] = v;
                    a = fma(v.x, v.x, fma(v.y, v.y, a));
                }
            __syncwarp();
            for (int o = GQ / 2; o > 0; o >>= 1) a += __shfl_xor_sync(0xFFFFFFFFu, a, o);
            if (i < p) {
                if (gl == 0) dn[i] = -1;
                if (!isfinite(a)) bad = 1;
                if (a > bv || (a == bv && i < bi)) { bv = a; bi = i; }
            }
        }
        if (rank == 0 && tid < 4) fl[tid] = 0;
        publish(bv, bi, bad, 0);
    }
    sync();

    // ---- pivoted Householder on the rows
    int r = 0;
    bool nonfinite = false;
    for (int k = 0;; ++k) {
        double mv = -1.0;
        int ip = 0x7FFFFFFF, bad = 0;
        for (int x = 0; x < C; ++x) {  // the same in every CTA
            const Cand *o = ONE ? own + (k & 1) : cd + (k & 1) * 16 + x;
            const double v = ldg<ONE>(&o->v);
            const int i = ldg<ONE>(&o->row);
            bad |= ldg<ONE>(&o->bad);
            if (v > mv || (v == mv && i < ip)) { mv = v; ip = i; }
        }
        if (bad) { nonfinite = true; break; }
        if (k >= kmax || !(mv > kNormFloor) || ip >= p) break;
        r = k + 1;
        const double2 *xr = w + (int64_t)ip * q;
        const bool staged = q <= kXStage;
        if (staged)
            for (int c = k + tid; c < q; c += NT) xs[c] = ldg2(xr + c);
        // u = conj(x), alpha = -e^{i phi} |u| (phi = arg u_0), v = u - alpha e_0,
        // beta = 2 / |v|^2 = 1 / (|u| (|u| + |u_0|))
        if (warp == 0) {
            const double2 x0 = ldg2(xr + k);
            const double n0 = fma(x0.x, x0.x, x0.y * x0.y);
            const double y = newton_rsqrt(mv);
            double nu = mv * y;
            nu = fma(0.5 * y, fma(-nu, nu, mv), nu);
            const bool phase = n0 > kPhaseFloor;
            const double ia = phase ? newton_rsqrt(n0) : 0.0;
            const double a0 = phase ? n0 * ia : 0.0;
            const double beta = newton_reciprocal(nu * (nu + a0));
            const double pr = phase ? x0.x * ia : 1.0, pi = phase ? -x0.y * ia : 0.0;  // e^{i phi}
            if (lane == 0) {
                sc[0] = make_double2(pr * (a0 + nu), pi * (a0 + nu));
                sc[1] = make_double2(beta, 0.0);
                if (ip % C == rank) {
                    al[k] = make_double2(-pr * nu, pi * nu);  // conj(alpha): the pivot row's entry k
                    dn[ip] = k;
                }
            }
        }
        __syncthreads();
        const double2 v0 = sc[0];
        const double beta = sc[1].x;
        double bv = -1.0;
        int bi = 0x7FFFFFFF, isbad = 0;
        const int GQ = lanes_for(q - k), RW = 32 / GQ, sub = lane / GQ, gl = lane % GQ;
        for (int base = warp * RW; rank + C * base < p; base += NW * RW) {  // warp-uniform
            const int i = rank + C * (base + sub);
            const bool live = i < p && dn[i] < 0;
            if (!__any_sync(0xFFFFFFFFu, live)) continue;
            double2 *wr = w + (int64_t)(live ? i : rank) * q;
            double sr = 0.0, si = 0.0;  // sum_c w_c v_c, v_c = conj(x_c) for c > k, v_k = v0
            if (live)
                for (int c = k + gl; c < q; c += GQ) {
                    const double2 xc = staged ? xs[c] : ldg2(xr + c);
                    const double2 vc = c == k ? v0 : make_double2(xc.x, -xc.y);
                    const double2 a = wr[c];
                    sr = fma(a.x, vc.x, fma(-a.y, vc.y, sr));
                    si = fma(a.x, vc.y, fma(a.y, vc.x, si));
                }
            __syncwarp();
            group_sum2(sr, si, GQ);
            const double fr = beta * sr, fi = beta * si;
            double ta = 0.0;
            if (live)
                for (int c = k + gl; c < q; c += GQ) {
                    const double2 xc = staged ? xs[c] : ldg2(xr + c);
                    const double2 cv = c == k ? make_double2(v0.x, -v0.y) : xc;  // conj(v_c)
                    double2 a = wr[c];
                    a.x = fma(-fr, cv.x, fma(fi, cv.y, a.x));
                    a.y = fma(-fr, cv.y, fma(-fi, cv.x, a.y));
                    wr[c] = a;
                    if (c > k) ta = fma(a.x, a.x, fma(a.y, a.y, ta));
                }
            __syncwarp();
            for (int o = GQ / 2; o > 0; o >>= 1) ta += __shfl_xor_sync(0xFFFFFFFFu, ta, o);
            if (live) {
                if (!isfinite(ta)) isbad = 1;
                if (ta > bv || (ta == bv && i < bi)) { bv = ta; bi = i; }
            }
        }
        publish(bv, bi, isbad, (k + 1) & 1);
        sync();
    }
    if (nonfinite) {  // uniform over the cluster: reported by the host
        if (rank == 0)
            for (int j = tid; j < q; j += NT) S[s.s_off + j] = nan("");
        if (rank == 0 && tid == 0) status[sec] = 0;
        return;
    }
    // ---- M, column-major: a row pivoted at step kk has its entry kk and zeros after it
    for (int i = rank + C * warp; i < p; i += C * NW) {
        const int kk = dn[i];
        for (int c = lane; c < r; c += 32) {
            double2 v = w[(int64_t)i * q + c];
            if (kk >= 0 && c >= kk) v = c == kk ? al[kk] : make_double2(0.0, 0.0);
            stg2(m + (int64_t)c * p + i, v);
        }
    }
    sync();

    // ---- one-sided Jacobi on M's r columns: a round's pairs two (G = 16) or
    // one (G = 32) a warp, dealt over the CTAs first
    const int qe = r + (r & 1), m1 = qe - 1, np = qe / 2;
    constexpr int PW = 32 / G;  // pairs a warp
    const int gl = lane % G, sub = lane / G;
    const double tol2 = tol * tol;
    int sweep = 0;
    bool converged = r < 2;
    for (; sweep < max_sweeps && !converged; ++sweep) {
        if (rank == 0 && tid == 0) stg<ONE>(fl + (sweep + 1) % 3, 0);  // last read two sweeps ago
        bool rotated = false;
        for (int rr = 0; rr < m1; ++rr) {
            for (int wt = rank + C * warp; wt * PW < np; wt += C * NW) {  // warp-uniform
                const int pi = wt * PW + sub;
                int c0 = 0, c1 = r;
                if (pi < np) {
                    if (pi > 0) { c0 = pi - 1 + rr; if (c0 >= m1) c0 -= m1; ++c0; }
                    c1 = qe - 2 - pi + rr; if (c1 >= m1) c1 -= m1; ++c1;
                    if (c0 > c1) { const int x = c0; c0 = c1; c1 = x; }
                }
                const bool act = c1 < r;  // group-uniform
                double2 *x = m + (int64_t)c0 * p, *y = m + (int64_t)(act ? c1 : c0) * p;
                double a = 0.0, b = 0.0, cr = 0.0, ci = 0.0;
                double2 xv[EPL > 0 ? EPL : 1], yv[EPL > 0 ? EPL : 1];
                if constexpr (EPL > 0) {
#pragma unroll
                    for (int e = 0; e < EPL; ++e) {
                        const int i = gl + e * G;
                        const bool in = act && i < p;
                        xv[e] = in ? ldg2(x + i) : make_double2(0.0, 0.0);
                        yv[e] = in ? ldg2(y + i) : make_double2(0.0, 0.0);
                    }
#pragma unroll
                    for (int e = 0; e < EPL; ++e) {
                        if (e * G >= p) break;  // uniform
                        a = fma(xv[e].x, xv[e].x, fma(xv[e].y, xv[e].y, a));
                        b = fma(yv[e].x, yv[e].x, fma(yv[e].y, yv[e].y, b));
                        cr = fma(xv[e].x, yv[e].x, fma(xv[e].y, yv[e].y, cr));
                        ci = fma(xv[e].x, yv[e].y, fma(-xv[e].y, yv[e].x, ci));
                    }
                } else {  // four elements in flight a lane (the compiler's own choice: 5 to 15 % longer splits)
                    if (act)
#pragma unroll 4
                        for (int i = gl; i < p; i += G) {
                            const double2 xi = ldg2(x + i), yi = ldg2(y + i);
                            a = fma(xi.x, xi.x, fma(xi.y, xi.y, a));
                            b = fma(yi.x, yi.x, fma(yi.y, yi.y, b));
                            cr = fma(xi.x, yi.x, fma(xi.y, yi.y, cr));
                            ci = fma(xi.x, yi.y, fma(-xi.y, yi.x, ci));
                        }
                    __syncwarp();
                }
                group_sum4<G>(a, b, cr, ci);
                const double ac2 = fma(cr, cr, ci * ci);
                // |c|^2 <= tol^2 a b: the pair is orthogonal to the tolerance; a column below the
                // floor counts as zero (high words: no FP64 instruction)
                const int lo = min(__double2hiint(a), __double2hiint(b));
                if (!act || lo <= __double2hiint(kNormFloor)) continue;
                if (lo > __double2hiint(kProductFloor) ? !(ac2 > tol2 * a * b)
                                                       : !above_tolerance(a, b, cr, ci, tol2))
                    continue;
                double cs, sr, si;
                rotation(a, b, cr, ci, cs, sr, si);
                rotated = true;
                if constexpr (EPL > 0) {
#pragma unroll
                    for (int e = 0; e < EPL; ++e) {
                        const int i = gl + e * G;
                        if (e * G >= p) break;
                        const double2 xo = xv[e], yo = yv[e];
                        const double nxr = fma(cs, xo.x, -fma(sr, yo.x, si * yo.y));
                        const double nxi = fma(cs, xo.y, -fma(sr, yo.y, -si * yo.x));
                        const double nyr = fma(cs, yo.x, fma(sr, xo.x, -si * xo.y));
                        const double nyi = fma(cs, yo.y, fma(sr, xo.y, si * xo.x));
                        if (i < p) {
                            stg2(x + i, make_double2(nxr, nxi));
                            stg2(y + i, make_double2(nyr, nyi));
                        }
                    }
                } else {
#pragma unroll 4
                    for (int i = gl; i < p; i += G) {
                        const double2 xo = ldg2(x + i), yo = ldg2(y + i);
                        stg2(x + i, make_double2(fma(cs, xo.x, -fma(sr, yo.x, si * yo.y)),
                                                 fma(cs, xo.y, -fma(sr, yo.y, -si * yo.x))));
                        stg2(y + i, make_double2(fma(cs, yo.x, fma(sr, xo.x, -si * xo.y)),
                                                 fma(cs, yo.y, fma(sr, xo.y, si * xo.x))));
                    }
                }
            }
            if (rr == m1 - 1 && rotated) stg<ONE>(fl + sweep % 3, 1);
            __syncwarp();
            sync();
        }
        converged = ldg<ONE>(fl + sweep % 3) == 0;  // the same in every CTA
    }
    if (rank == 0 && tid == 0) status[sec] = converged ? sweep : -sweep;

    // ---- norms, then sorted singular values and normalised columns
    for (int j = rank + C * warp; j < kmax; j += C * NW) {
        double a = 0.0;
        if (j < r)
            for (int i = lane; i < p; i += 32) {
                const double2 v = ldg2(m + (int64_t)j * p + i);
                a = fma(v.x, v.x, fma(v.y, v.y, a));
            }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xFFFFFFFFu, a, o);
        if (lane == 0) stg<ONE>(nv + j, a > kNormFloor ? sqrt(a) : 0.0);
    }
    sync();
    for (int j = rank + C * warp; j < kmax; j += C * NW) {
        const double sj = ldg<ONE>(nv + j);
        int pos = 0;
        for (int i = lane; i < kmax; i += 32) {
            const double si = ldg<ONE>(nv + i);
            pos += (si > sj) || (si == sj && i < j);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) pos += __shfl_xor_sync(0xFFFFFFFFu, pos, o);
        const double inv = sj > 0.0 ? 1.0 / sj : 0.0;
        if (sj > 0.0)
            for (int i = lane; i < p; i += 32) {
                const double2 v = ldg2(m + (int64_t)j * p + i);
                stg2(w + (int64_t)pos * p + i, make_double2(v.x * inv, v.y * inv));
            }
        if (lane == 0) S[s.s_off + pos] = scalbn(sj, -shift);
    }
    if (rank == 0)
        for (int j = kmax + tid; j < q; j += NT) S[s.s_off + j] = 0.0;
}

// Completion of a factor's orthonormal columns (svd_fp64_complete): Householder
// reflectors H_0 ... H_{j0-1} of the j0 columns U holds, whose product Q has
// those columns (up to phases) first; Q's columns j0 ... k-1 complete them, each
// for itself.  Only columns that are kept are made, so it runs where a
// truncation keeps singular values of zero (a negative cut-off, the SA split).
// FP64 issue bounds both kernels.  Measured (the split of one 200 x 200 sector,
// kept whole; completion vector by vector in k_svd64 before): all of it zero 132.5
// -> 0.38 ms, half of its rows zero 110.5 -> 15.2 ms, 11.4 of it without
// completion; nothing kept of the zero sector: 132.4 -> 0.19 ms.
struct Fill {
    int64_t t_off, v_off;  // U's columns; the reflectors' vectors, p x j0
    int64_t b_off;         // j0 reflector scales
    int p, j0;
};

__global__ void __launch_bounds__(NT) k_svd64_reflect(const Fill *__restrict__ fills, const double2 *__restrict__ U,
                                                      double2 *V, double *beta) {
    const Fill d = fills[blockIdx.x];
    const int p = d.p, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    double2 *v = V + d.v_off;
    __shared__ double s_beta;
    for (int64_t e = tid; e < (int64_t)p * d.j0; e += NT) v[e] = U[d.t_off + e];
    __syncthreads();
    for (int c = 0; c < d.j0; ++c) {
        double2 *x = v + (int64_t)c * p;
        if (warp == 0) {  // v = x - alpha e_c with alpha = -(x_c / |x_c|) |x|, beta = 2 / |v|^2
            double a = 0.0;
            for (int i = c + lane; i < p; i += 32) a = fma(x[i].x, x[i].x, fma(x[i].y, x[i].y, a));
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xFFFFFFFFu, a, o);
            const double2 xc = x[c];
            const double nu = sqrt(a), n0 = fma(xc.x, xc.x, xc.y * xc.y);
            const bool phase = n0 > kPhaseFloor;
            const double a0 = phase ? sqrt(n0) : 0.0;
            __syncwarp();
            if (lane == 0) {
                x[c] = make_double2(phase ? xc.x / a0 * (a0 + nu) : nu, phase ? xc.y / a0 * (a0 + nu) : 0.0);
                beta[d.b_off + c] = s_beta = 1.0 / (nu * (nu + a0));
            }
        }
        __syncthreads();
        const double b = s_beta;
        for (int y0 = c + 1 + warp; y0 < d.j0; y0 += NW) {
            double2 *y = v + (int64_t)y0 * p;
            double sr = 0.0, si = 0.0;  // v^H y
            for (int i = c + lane; i < p; i += 32) {
                const double2 h = x[i], w = y[i];
                sr = fma(h.x, w.x, fma(h.y, w.y, sr));
                si = fma(h.x, w.y, fma(-h.y, w.x, si));
            }
            __syncwarp();
            group_sum2(sr, si, 32);
            sr *= b;
            si *= b;
            for (int i = c + lane; i < p; i += 32) {
                const double2 h = x[i];
                y[i].x -= h.x * sr - h.y * si;
                y[i].y -= h.x * si + h.y * sr;
            }
        }
        __syncthreads();
    }
}

// one warp per new column: items (fill, column)
__global__ void __launch_bounds__(NT) k_svd64_fill(const Fill *__restrict__ fills, const int2 *__restrict__ items,
                                                   int nitems, const double2 *__restrict__ V,
                                                   const double *__restrict__ beta, double2 *U) {
    const int item = blockIdx.x * NW + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (item >= nitems) return;  // warp-uniform
    const int2 it = items[item];
    const Fill d = fills[it.x];
    double2 *y = U + d.t_off + (int64_t)it.y * d.p;  // a lane reads only elements that it wrote
    for (int i = lane; i < d.p; i += 32) y[i] = make_double2(i == it.y ? 1.0 : 0.0, 0.0);
    for (int c = d.j0 - 1; c >= 0; --c) {
        const double2 *h = V + d.v_off + (int64_t)c * d.p;
        double sr = 0.0, si = 0.0;
        for (int i = lane; i < d.p; i += 32) {
            if (i < c) continue;
            const double2 a = h[i], w = y[i];
            sr = fma(a.x, w.x, fma(a.y, w.y, sr));
            si = fma(a.x, w.y, fma(-a.y, w.x, si));
        }
        __syncwarp();
        group_sum2(sr, si, 32);
        const double b = beta[d.b_off + c];
        sr *= b;
        si *= b;
        for (int i = lane; i < d.p; i += 32) {
            if (i < c) continue;
            const double2 a = h[i];
            y[i].x -= a.x * sr - a.y * si;
            y[i].y -= a.x * si + a.y * sr;
        }
    }
}

constexpr int kMaxDevices = 64;
constexpr int kXBytes = kXStage * (int)sizeof(double2);

// once per device: the kernels may use kXBytes of dynamic shared memory and
// clusters of 16; returns whether a cluster of 16 can be resident
bool svd64_setup(int dev) {
    static std::mutex mu;
    static int state[kMaxDevices] = {};  // 0 unknown, 1: clusters of 16, -1: up to 8
    KV_REQUIRE(dev >= 0 && dev < kMaxDevices, KV_EINVAL, "device index out of range");
    std::lock_guard<std::mutex> lk(mu);
    if (state[dev] == 0) {
        const void *ks[] = {(const void *)k_svd64<16, 4, false>, (const void *)k_svd64<16, 8, false>,
                            (const void *)k_svd64<16, 16, false>, (const void *)k_svd64<16, 0, false>,
                            (const void *)k_svd64<32, 2, false>, (const void *)k_svd64<32, 4, false>,
                            (const void *)k_svd64<32, 8, false>, (const void *)k_svd64<32, 0, false>};
        for (const void *k : {(const void *)k_svd64<16, 4, true>, (const void *)k_svd64<16, 8, true>,
                              (const void *)k_svd64<16, 16, true>, (const void *)k_svd64<16, 0, true>,
                              (const void *)k_svd64<32, 2, true>, (const void *)k_svd64<32, 4, true>,
                              (const void *)k_svd64<32, 8, true>, (const void *)k_svd64<32, 0, true>})
            KV_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kXBytes));
        int ok = 1;
        for (const void *k : ks) {
            KV_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kXBytes));
            if (cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
                (void)cudaGetLastError();
                ok = 0;
                continue;
            }
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(16);
            cfg.blockDim = dim3(NT);
            cfg.dynamicSmemBytes = kXBytes;
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeClusterDimension;
            at[0].val.clusterDim = {16, 1, 1};
            cfg.attrs = at;
            cfg.numAttrs = 1;
            int n = 0;
            if (cudaOccupancyMaxActiveClusters(&n, k, &cfg) != cudaSuccess) {
                (void)cudaGetLastError();
                n = 0;
            }
            if (n < 1) ok = 0;
        }
        state[dev] = ok ? 1 : -1;
    }
    return state[dev] > 0;
}

}  // namespace

void svd_fp64(const SvdPlan &P, const double2 *T, double2 *U, double *S, int *status, int max_sweeps, double tol) {
    if (P.secs.empty()) return;
    const bool c16 = svd64_setup(ctx().device);
    const int nsec = (int)P.secs.size();
    std::vector<Svd64Sector> secs;
    int64_t k_elems = 0, r_elems = 0;
    int max_p = 1, max_q = 1, max_k = 1;
    for (auto &s : P.secs) {
        secs.push_back({s.t_off, s.s_off, k_elems, r_elems, s.p, s.q});
        k_elems += std::min(s.p, s.q);
        r_elems += s.p;
        max_p = std::max(max_p, s.p);
        max_q = std::max(max_q, s.q);
        max_k = std::max(max_k, std::min(s.p, s.q));
    }
    // Cluster size: eight pairs keep one CTA's FP64 units busy (two a warp, a
    // warp per quarter of the SM), and the sectors together should fit one
    // wave of SMs.  Where four pairs a CTA still fit, one pair a warp (G = 32)
    // halves a round's time.
    const int pairs = (max_k + 1) / 2, cmax = c16 ? 16 : 8;
    int C = 1;
    while (C < cmax && C * 8 < pairs && nsec * C * 2 <= ctx().num_sms) C *= 2;
    bool wide = C * 4 >= pairs;
    if (!wide && C < cmax && C * 8 >= pairs && nsec * C * 2 <= ctx().num_sms) {
        C *= 2;
        wide = C * 4 >= pairs;
    }
    // one allocation: sectors, M, diagonal entries, norms, row flags, candidates, sweep flags
    size_t bytes = 0;
    auto carve = [&](size_t n) {
        const size_t o = bytes;
        bytes += (n + 255) & ~size_t(255);
        return o;
    };
    const size_t o_ds = carve(secs.size() * sizeof(Svd64Sector)), o_m = carve((size_t)P.t_elems * sizeof(double2)),
                 o_al = carve((size_t)k_elems * sizeof(double2)), o_nv = carve((size_t)k_elems * sizeof(double)),
                 o_dn = carve((size_t)r_elems * sizeof(int)), o_cd = carve((size_t)nsec * 32 * sizeof(Cand)),
                 o_fl = carve((size_t)nsec * 4 * sizeof(int));
    DevBuf ws(bytes);
    char *wp = ws.as<char>();
    upload_bytes(wp + o_ds, secs.data(), secs.size() * sizeof(Svd64Sector));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(nsec * C));
    cfg.blockDim = dim3(NT);
    cfg.dynamicSmemBytes = (size_t)std::min(max_q, kXStage) * sizeof(double2);
    cfg.stream = ctx().stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)C;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    auto launch = [&](auto kernel) {
        KV_CUDA(cudaLaunchKernelEx(&cfg, kernel, reinterpret_cast<const Svd64Sector *>(wp + o_ds), T, U,
                                   reinterpret_cast<double2 *>(wp + o_m), S, reinterpret_cast<double2 *>(wp + o_al),
                                   reinterpret_cast<double *>(wp + o_nv), reinterpret_cast<int *>(wp + o_dn),
                                   reinterpret_cast<Cand *>(wp + o_cd), reinterpret_cast<int *>(wp + o_fl), status,
                                   max_sweeps, tol));
    };
    // a column's elements stay in registers between the sums and the rotation up to 256 rows
    if (C == 1 && wide) {
        if (max_p <= 64) launch(k_svd64<32, 2, true>);
        else if (max_p <= 128) launch(k_svd64<32, 4, true>);
        else if (max_p <= 256) launch(k_svd64<32, 8, true>);
        else launch(k_svd64<32, 0, true>);
    } else if (C == 1) {
        if (max_p <= 64) launch(k_svd64<16, 4, true>);
        else if (max_p <= 128) launch(k_svd64<16, 8, true>);
        else if (max_p <= 256) launch(k_svd64<16, 16, true>);
        else launch(k_svd64<16, 0, true>);
    } else if (wide) {
        if (max_p <= 64) launch(k_svd64<32, 2, false>);
        else if (max_p <= 128) launch(k_svd64<32, 4, false>);
        else if (max_p <= 256) launch(k_svd64<32, 8, false>);
        else launch(k_svd64<32, 0, false>);
    } else {
        if (max_p <= 64) launch(k_svd64<16, 4, false>);
        else if (max_p <= 128) launch(k_svd64<16, 8, false>);
        else if (max_p <= 256) launch(k_svd64<16, 16, false>);
        else launch(k_svd64<16, 0, false>);
    }
    counted();
}

void svd_fp64_complete(const SvdPlan &P, const std::vector<double> &s, const std::vector<int> &kept, double2 *U) {
    std::vector<Fill> fills;
    std::vector<int2> items;
    int64_t v_elems = 0, b_elems = 0;
    for (size_t i = 0; i < P.secs.size(); ++i) {
        const SvdSector &sc = P.secs[i];
        int j0 = 0;
        while (j0 < kept[i] && s[sc.s_off + j0] > 0.0) ++j0;
        if (j0 >= kept[i]) continue;
        for (int j = j0; j < kept[i]; ++j) items.push_back(make_int2((int)fills.size(), j));
        fills.push_back({sc.t_off, v_elems, b_elems, sc.p, j0});
        v_elems += (int64_t)sc.p * j0;
        b_elems += j0;
    }
    if (fills.empty()) return;
    DevSpan df, di;
    UploadPack u;
    u.add(df, fills);
    u.add(di, items);
    DevBuf lists = u.upload();
    DevBuf V(std::max<int64_t>(1, v_elems) * sizeof(double2)), beta(std::max<int64_t>(1, b_elems) * sizeof(double));
    if (v_elems > 0) {
        k_svd64_reflect<<<(unsigned)fills.size(), NT, 0, ctx().stream>>>(df.as<Fill>(), U, V.as<double2>(),
                                                                         beta.as<double>());
        counted();
    }
    k_svd64_fill<<<(unsigned)((items.size() + NW - 1) / NW), NT, 0, ctx().stream>>>(
        df.as<Fill>(), di.as<int2>(), (int)items.size(), V.as<double2>(), beta.as<double>(), U);
    counted();
    KV_CUDA(cudaGetLastError());
}

}  // namespace kv
