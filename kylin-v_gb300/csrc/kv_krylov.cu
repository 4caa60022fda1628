// FP64 Lanczos kernels for local_krylov (holstein/exponential.h:92-190).
//
// All Krylov vectors share one block layout, so overlaps and updates are flat
// vector operations.  Reductions are two-level and deterministic: each kernel
// writes one partial per CTA (fixed grid, fixed order) and the next kernel
// reduces those partials in a fixed order before using the value, fused with
// the update that needs it (classical Gram-Schmidt in the reference's order:
// beta against v_{k-1} first, then alpha against v_k, then the norm).
#include <cooperative_groups.h>

#include <algorithm>
#include <mutex>

#include "kv_internal.h"

namespace kv {

namespace {

constexpr int KT = 256;
constexpr double kMaxTridiagNorm = 1e5;  // largest ||T||_1 the Taylor sub-stepping accepts

__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }

// GB300's FP64 unit issues two thread-operations per clock per SM, so the
// vector kernels below are bound by their FP64 operation count and latency:
// products are accumulated with fused multiply-adds (two a component), and a
// block's warp sums are combined by a shuffle tree instead of one thread.

// s + conj(x) y, two fused multiply-adds a component
__device__ __forceinline__ double2 cdotc_acc(double2 s, double2 x, double2 y) {
    s.x = fma(x.x, y.x, fma(x.y, y.y, s.x));
    s.y = fma(x.x, y.y, fma(-x.y, y.x, s.y));
    return s;
}

// h - c x
__device__ __forceinline__ double2 csub_mul(double2 h, double2 c, double2 x) {
    h.x = fma(-c.x, x.x, fma(c.y, x.y, h.x));
    h.y = fma(-c.x, x.y, fma(-c.y, x.x, h.y));
    return h;
}

// s + c x
__device__ __forceinline__ double2 cmul_acc(double2 s, double2 c, double2 x) {
    s.x = fma(c.x, x.x, fma(-c.y, x.y, s.x));
    s.y = fma(c.x, x.y, fma(c.y, x.x, s.y));
    return s;
}

// s + |h|^2
__device__ __forceinline__ double norm2_acc(double s, double2 h) { return fma(h.x, h.x, fma(h.y, h.y, s)); }

// The warp's sum over its first W lanes (a shuffle tree, halves added first):
// lane 0 receives the real part, lane W / 2 the imaginary part.  At the first
// level the lower lanes add the real parts and the upper ones the imaginary
// parts, so a complex sum costs log2 W additions a lane instead of twice that
// (a warp's FP64 instruction takes 19 clocks of the SM whatever its active lanes).
template <int W = 32>
__device__ __forceinline__ double warp_sum_split(double2 v) {
    const bool hi = (threadIdx.x & (W / 2)) != 0;
    double k = hi ? v.y : v.x;
    k += __shfl_xor_sync(0xffffffffu, hi ? v.x : v.y, W / 2);
#pragma unroll
    for (int o = W / 4; o > 0; o >>= 1) k += __shfl_down_sync(0xffffffffu, k, o);
    return k;
}

// the block's sum, returned to every thread; a fixed order of adds.  Warps
// from `live` on hold zeros and add nothing.
__device__ double2 block_sum(double2 v, int live = KT / 32) {
    constexpr int NW = KT / 32;
    static_assert(NW <= 32 && (NW & (NW - 1)) == 0, "warp count a power of two");
    __shared__ double red[2 * NW];
    __shared__ double2 out;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    double k = 0.0;
    if (w < live) k = warp_sum_split(v);
    __syncthreads();  // a previous call's readers of red are done
    if ((lane & 15) == 0) red[2 * w + (lane >> 4)] = k;
    __syncthreads();
    if (w == 0) {
        const int x = lane & (NW - 1);
        const double t = warp_sum_split<NW>(make_double2(red[2 * x], red[2 * x + 1]));
        if (lane == 0) out.x = t;
        if (lane == NW / 2) out.y = t;
    }
    __syncthreads();
    return out;
}

// every CTA reduces the same partial array (zero from entry `used` on) in the same order
__device__ double2 reduce_partials(const double2 *parts, int nparts, int used) {
    int i = threadIdx.x;
    double2 v = i < used ? __ldcg(parts + i) : make_double2(0.0, 0.0);
    for (i += KT; i < used; i += KT) v = cadd(v, __ldcg(parts + i));
    return block_sum(v, min(KT, used + 31) / 32);
}
__device__ __forceinline__ double2 reduce_partials(const double2 *parts, int nparts) {
    return reduce_partials(parts, nparts, nparts);
}

__global__ void __launch_bounds__(KT) k_norm_part(const double2 *x, int64_t n, double2 *parts) {
    double s = 0.0;
    for (int64_t i = blockIdx.x * (int64_t)KT + threadIdx.x; i < n; i += (int64_t)gridDim.x * KT)
        s = norm2_acc(s, x[i]);
    double2 r = block_sum(make_double2(s, 0.0));
    if (threadIdx.x == 0) parts[blockIdx.x] = r;
}

// the host-mapped stop flag: visible to the host once the kernel has finished
__device__ __forceinline__ void raise_stop(int *stop) {
    if (stop) {
        *reinterpret_cast<volatile int *>(stop) = 1;
        __threadfence_system();
    }
}

__global__ void __launch_bounds__(KT) k_start(KrylovState *st, const double2 *psi, double2 *v0, int64_t n,
                                              const double2 *parts, int nparts, int *stop) {
    allow_dependents();
    dependency_wait();
    const double n2 = reduce_partials(parts, nparts).x;
    __shared__ double s_inv;
    if (threadIdx.x == 0) {
        const double nrm = sqrt(n2);
        const bool bad = !isfinite(nrm) || nrm == 0.0;
        if (blockIdx.x == 0) {
            st->psi_norm = nrm;
            st->err[0] = 1.0;
            st->done = bad ? 1 : 0;
            st->iters = 0;
            st->status = bad ? KV_ENONFINITE : KV_OK;
            if (bad) raise_stop(stop);
        }
        s_inv = bad ? 0.0 : 1.0 / nrm;
    }
    __syncthreads();
    const double inv = s_inv;
    for (int64_t i = blockIdx.x * (int64_t)KT + threadIdx.x; i < n; i += (int64_t)gridDim.x * KT)
        v0[i] = make_double2(psi[i].x * inv, psi[i].y * inv);
}

// parts[b] = sum conj(x) y
__global__ void __launch_bounds__(KT) k_dot_part(const KrylovState *st, const double2 *x, const double2 *y,
                                                 int64_t n, double2 *parts) {
    if (st->done) return;
    double2 s = make_double2(0.0, 0.0);
    for (int64_t i = blockIdx.x * (int64_t)KT + threadIdx.x; i < n; i += (int64_t)gridDim.x * KT)
        s = cdotc_acc(s, x[i], y[i]);
    double2 r = block_sum(s);
    if (threadIdx.x == 0) parts[blockIdx.x] = r;
}

// c = reduce(pin) (= overlap(v, hv) = <hv|v>);  hv -= c v on [0, n_sub) (v is
// zero beyond);  pout[b] = sum_{i < n_dot} conj(hv) w  (w == nullptr: sum |hv|^2).
// slot receives c.
__global__ void __launch_bounds__(KT) k_sub(KrylovState *st, double2 *hv, const double2 *v, const double2 *w,
                                            int64_t n_sub, int64_t n_dot, const double2 *pin, double2 *pout,
                                            int nparts, double2 *slot) {
    if (st->done) return;
    const double2 c = reduce_partials(pin, nparts);
    if (blockIdx.x == 0 && threadIdx.x == 0) *slot = c;
    double2 s = make_double2(0.0, 0.0);
    for (int64_t i = blockIdx.x * (int64_t)KT + threadIdx.x; i < n_dot; i += (int64_t)gridDim.x * KT) {
        double2 h = hv[i];
        if (i < n_sub) {
            h = csub_mul(h, c, v[i]);
            hv[i] = h;
        }
        if (w) s = cdotc_acc(s, h, w[i]);
        else s.x = norm2_acc(s.x, h);
    }
    double2 r = block_sum(s);
    if (threadIdx.x == 0) pout[blockIdx.x] = r;
}

// err[k+1] = err[k] nrm and the stop test (one thread)
__device__ __forceinline__ void normalize_state(KrylovState *st, double nrm, int k, double tol, int max_iter,
                                                int *stop) {
    const double e = st->err[k] * nrm;
    st->err[k + 1] = e;
    if (!isfinite(nrm)) {
        st->status = KV_ENONFINITE;
        st->done = 1;
        st->iters = k + 1;
        raise_stop(stop);
    } else if (e <= tol || k + 1 >= max_iter - 1) {
        st->done = 1;
        st->iters = k + 1;
        raise_stop(stop);
    }
}

// nrm = sqrt(reduce(pin)); the stop test; vnext = hv / nrm
__global__ void __launch_bounds__(KT) k_normalize(KrylovState *st, const double2 *hv, double2 *vnext, int64_t n,
                                                  const double2 *pin, int nparts, int k, double tol, int max_iter,
                                                  int *stop) {
    if (st->done) return;
    const double n2 = reduce_partials(pin, nparts).x;
    __shared__ double s_inv;
    if (threadIdx.x == 0) {
        const double nrm = sqrt(n2);
        if (blockIdx.x == 0) normalize_state(st, nrm, k, tol, max_iter, stop);
        s_inv = nrm > 0.0 && isfinite(nrm) ? 1.0 / nrm : 0.0;
    }
    __syncthreads();
    const double inv = s_inv;
    if (__double2hiint(inv) == 0) return;  // a zero or non-finite norm
    for (int64_t i = blockIdx.x * (int64_t)KT + threadIdx.x; i < n; i += (int64_t)gridDim.x * KT)
        vnext[i] = make_double2(hv[i].x * inv, hv[i].y * inv);
}

// One Lanczos iteration after hv = (dt/2) H v_k as one launch.  The separate
// kernels (k_dot_part, k_sub, k_sub, k_normalize) are its phases, with a barrier
// where they end.  Their grid of nparts CTAs of KT threads is virtual here:
// CTA `rank` of `size` takes the virtual CTAs rank, rank + size, ..., their warps
// dealt over its PW warps, and virtual CTAs beyond the vectors' ends (whose sums
// are zero) are left out.  The partial sums, their fixed-order reductions and
// every result are the same bits however the work is dealt.
//  * as a grid: one cooperative launch, a CTA an SM, for long vectors; only on
//    the main context's stream.
//  * as a cluster: one cluster of CTAs, for short vectors and for the worker
//    streams (a cluster is scheduled whole, so its barrier waits on no other
//    launch), whose barriers take a fraction of a grid's.
// What bounds it: the FP64 unit for long vectors (20 operations an element),
// the barriers and the chains of sums between them for short ones.
// Measured (us a launch, against a cooperative launch of nparts CTAs): 912
// elements 21.5 -> 13.1, 8496 elements 23.4 -> 18.0 (both cluster), 253952
// elements 32.0 -> 26.8 (grid), 1966080 elements 88.5 -> 89.5 (the FP64 unit:
// 74 us).
constexpr int kMaxLocal = 40;  // virtual CTAs one CTA takes (512 parts over 16 CTAs: 32)

template <int PW, class Sync>
struct LanczosStep {
    Sync &sync;
    int rank, size, nparts;
    double (*red)[16];  // [kMaxLocal] virtual warps' sums, real and imaginary interleaved
    double2 *out;

    __device__ __forceinline__ int vctas(int64_t n) const {
        return (int)min((int64_t)nparts, (n + KT - 1) / KT);
    }
    // f(i) -> value summed into the virtual thread's sum: partial sums of the virtual CTAs into P
    template <class F>
    __device__ __forceinline__ void partial_sums(int64_t n, double2 *P, F f) {
        const int u = vctas(n), warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        const int nloc = u > rank ? (u - rank + size - 1) / size : 0;
        const int64_t di = (int64_t)nparts * KT;
        for (int x = warp; x < 8 * nloc; x += PW) {
            const int j = x >> 3, w = x & 7;
            double2 s = make_double2(0.0, 0.0);
            for (int64_t i = (int64_t)(rank + j * size) * KT + w * 32 + lane; i < n; i += di) s = f(i, s);
            const double k = warp_sum_split(s);
            if ((lane & 15) == 0) red[j][2 * w + (lane >> 4)] = k;
        }
        __syncthreads();
        for (int j = warp; j < nloc; j += PW) {
            const int x = lane & 7;
            const double t = warp_sum_split<8>(make_double2(red[j][2 * x], red[j][2 * x + 1]));
            double *p = reinterpret_cast<double *>(P + rank + j * size);
            if (lane == 0) __stcg(p, t);
            if (lane == 4) __stcg(p + 1, t);
        }
    }
    // the sum of the used partials, to every thread
    __device__ __forceinline__ double2 total(const double2 *P, int64_t n) {
        const int u = vctas(n), warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        if (warp < 8) {
            double k = 0.0;
            if (warp * 32 < u) {
                int i = threadIdx.x;
                double2 v = i < u ? __ldcg(P + i) : make_double2(0.0, 0.0);
                for (i += KT; i < u; i += KT) v = cadd(v, __ldcg(P + i));
                k = warp_sum_split(v);
            }
            if ((lane & 15) == 0) red[0][2 * warp + (lane >> 4)] = k;
        }
        __syncthreads();
        if (warp == 0) {
            const int x = lane & 7;
            const double t = warp_sum_split<8>(make_double2(red[0][2 * x], red[0][2 * x + 1]));
            if (lane == 0) out->x = t;
            if (lane == 4) out->y = t;
        }
        __syncthreads();
        return *out;
    }
    // f(i) for every element of the CTA's virtual threads
    template <class F>
    __device__ __forceinline__ void each(int64_t n, F f) {
        const int u = vctas(n), warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        const int nloc = u > rank ? (u - rank + size - 1) / size : 0;
        const int64_t di = (int64_t)nparts * KT;
        for (int x = warp; x < 8 * nloc; x += PW)
            for (int64_t i = (int64_t)(rank + (x >> 3) * size) * KT + (x & 7) * 32 + lane; i < n; i += di) f(i);
    }

    __device__ __forceinline__ void run(KrylovState *st, int k, double2 *hv, const double2 *vprev, const double2 *vk,
                                        double2 *vnext, int64_t n_prev, int64_t n_k, int64_t n_next, double2 *P0,
                                        double2 *P1, double tol, int max_iter, int *stop) {
        // read once, before the first barrier: this launch sets it only after the last one
        if (*reinterpret_cast<volatile int *>(&st->done)) return;  // uniform over the launch
        const bool lead = rank == 0 && threadIdx.x == 0;
        if (k > 0) {
            partial_sums(n_prev, P0, [&](int64_t i, double2 s) { return cdotc_acc(s, hv[i], vprev[i]); });
            sync.sync();
            const double2 c = total(P0, n_prev);
            if (lead) st->beta[k - 1] = c;
            partial_sums(n_k, P1, [&](int64_t i, double2 s) {
                double2 h = hv[i];
                if (i < n_prev) {
                    h = csub_mul(h, c, vprev[i]);
                    hv[i] = h;
                }
                return cdotc_acc(s, h, vk[i]);
            });
        } else {
            partial_sums(n_k, P1, [&](int64_t i, double2 s) { return cdotc_acc(s, hv[i], vk[i]); });
        }
        sync.sync();
        const double2 c = total(P1, n_k);
        if (lead) st->alpha[k] = c;
        partial_sums(n_next, P0, [&](int64_t i, double2 s) {
            double2 h = hv[i];
            if (i < n_k) {
                h = csub_mul(h, c, vk[i]);
                hv[i] = h;
            }
            s.x = norm2_acc(s.x, h);
            return s;
        });
        sync.sync();
        const double n2 = total(P0, n_next).x;
        // one warp takes the root and the reciprocal: some forty FP64
        // instructions, 0.4 us of the SM for each warp that repeats them
        if (threadIdx.x < 32) {
            const double nrm = sqrt(n2);
            const bool good = nrm > 0.0 && isfinite(nrm);
            if (threadIdx.x == 0) {
                if (lead) normalize_state(st, nrm, k, tol, max_iter, stop);
                *out = make_double2(good ? 1.0 / nrm : 0.0, 0.0);
            }
        }
        __syncthreads();
        const double inv = out->x;
        if (__double2hiint(inv) == 0) return;  // a zero or non-finite norm
        each(n_next, [&](int64_t i) { vnext[i] = make_double2(hv[i].x * inv, hv[i].y * inv); });
    }
};

constexpr int kStepGrid = 512;  // threads a CTA
// cluster form: a virtual CTA each, or (more virtual CTAs than the cluster has) as many warps as a CTA holds
constexpr int kClusterOne = KT, kClusterMany = 1024;

__global__ void __launch_bounds__(kStepGrid) k_lanczos_step(KrylovState *st, int k, double2 *hv, const double2 *vprev,
                                                            const double2 *vk, double2 *vnext, int64_t n_prev,
                                                            int64_t n_k, int64_t n_next, double2 *P0, double2 *P1,
                                                            int nparts, double tol, int max_iter, int *stop) {
    __shared__ double red[kMaxLocal][16];
    __shared__ double2 out;
    allow_dependents();
    cooperative_groups::grid_group g = cooperative_groups::this_grid();
    LanczosStep<kStepGrid / 32, cooperative_groups::grid_group> s{g, (int)blockIdx.x, (int)gridDim.x, nparts, red, &out};
    s.run(st, k, hv, vprev, vk, vnext, n_prev, n_k, n_next, P0, P1, tol, max_iter, stop);
}

template <int NT>
__global__ void __launch_bounds__(NT) k_lanczos_cluster(KrylovState *st, int k, double2 *hv,
                                                                  const double2 *vprev, const double2 *vk,
                                                                  double2 *vnext, int64_t n_prev, int64_t n_k,
                                                                  int64_t n_next, double2 *P0, double2 *P1, int nparts,
                                                                  double tol, int max_iter, int *stop) {
    __shared__ double red[kMaxLocal][16];
    __shared__ double2 out;
    allow_dependents();
    dependency_wait();
    cooperative_groups::cluster_group g = cooperative_groups::this_cluster();
    LanczosStep<NT / 32, cooperative_groups::cluster_group> s{g, (int)blockIdx.x, (int)gridDim.x, nparts, red, &out};
    s.run(st, k, hv, vprev, vk, vnext, n_prev, n_k, n_next, P0, P1, tol, max_iter, stop);
}

// T = tridiag(Re alpha, beta upper); c = exp(img T) e0 with img = -i (forward)
// or +i (reverse).  The reference forms the same vector as
// Z exp(img Lambda) Z^H e0 from a dense eigendecomposition
// (holstein/exponential.h:163-183).  Here it is summed directly: m sub-steps
// with ||T/m||_1 <= 1, each a Taylor series of exp(img T/m) applied to the
// vector (terms t_k = img T t_{k-1} / (m k), stopping once a term falls below
// 1e-18 of the sum), so no term is larger than the vector it is added to.
// One warp; lane i holds component i and takes its neighbours' components
// by shuffles.  The chain of FP64 instructions bounds it (64 clocks each for a
// lone warp), so the stop test runs on integers and the divisions are taken
// once: 57 -> 37 us at dimension 10.
__device__ __forceinline__ double2 shfl_down2(double2 v) {
    return make_double2(__shfl_down_sync(0xFFFFFFFFu, v.x, 1), __shfl_down_sync(0xFFFFFFFFu, v.y, 1));
}

__device__ __forceinline__ double2 shfl_up2(double2 v) {
    return make_double2(__shfl_up_sync(0xFFFFFFFFu, v.x, 1), __shfl_up_sync(0xFFFFFFFFu, v.y, 1));
}

__device__ __forceinline__ double warp_max(double v) {
    for (int o = 16; o; o >>= 1) v = fmax(v, __shfl_xor_sync(0xFFFFFFFFu, v, o));
    return v;
}

// the larger of |re|, |im| by its high word (exponent and leading bits)
__device__ __forceinline__ int part_exponent(double2 v) {
    return max(__double2hiint(v.x) & 0x7FFFFFFF, __double2hiint(v.y) & 0x7FFFFFFF);
}

__global__ void __launch_bounds__(32) k_tridiag_exp(KrylovState *st, int reverse) {
    static_assert(kMaxKrylov <= 32, "one lane per Krylov vector");
    allow_dependents();
    dependency_wait();
    const int lane = threadIdx.x;
    const int n = st->iters;
    if (n <= 0) return;
    if (st->status != KV_OK) {  // a non-finite Lanczos norm: no coefficients
        if (lane < n) st->coef[lane] = make_double2(nan(""), 0.0);
        return;
    }
    const bool on = lane < n;
    const double a = on ? st->alpha[lane].x : 0.0;
    const double2 zero = make_double2(0.0, 0.0);
    const double2 bu = (lane + 1 < n) ? st->beta[lane] : zero;  // T[lane][lane + 1]
    double2 bl = (on && lane >= 1) ? st->beta[lane - 1] : zero;  // T[lane][lane - 1] = conj(beta)
    bl.y = -bl.y;
    const double rs = warp_max(fabs(a) + sqrt(bu.x * bu.x + bu.y * bu.y) + sqrt(bl.x * bl.x + bl.y * bl.y));
    // the sub-step count is ceil(||T||_1): a norm beyond kMaxTridiagNorm (far
    // above any dt * H_eff of a physical chain) is reported as non-finite
    // instead of looping over that many steps
    if (!(rs <= kMaxTridiagNorm)) {
        if (on) st->coef[lane] = make_double2(nan(""), 0.0);
        if (lane == 0) st->status = KV_ENONFINITE;
        return;
    }
    const int m = max(1, (int)ceil(rs));
    const double sg = reverse ? 1.0 : -1.0;
    // term k's factor sg / (m k), lane k - 1 (and k - 33): two divisions a
    // lane instead of one a term
    const double f_lo = sg / ((double)m * (lane + 1)), f_hi = sg / ((double)m * (lane + 33));
    double2 y = make_double2(lane == 0 ? 1.0 : 0.0, 0.0);
    for (int step = 0; step < m; ++step) {
        double2 term = y, acc = y;
        for (int k = 1; k < 64; ++k) {
            const double2 up = shfl_down2(term);  // component lane + 1 (bu = 0 past the end)
            const double2 dn = shfl_up2(term);    // component lane - 1 (bl = 0 on lane 0)
            const double tr = a * term.x + (bu.x * up.x - bu.y * up.y) + (bl.x * dn.x - bl.y * dn.y);
            const double ti = a * term.y + (bu.x * up.y + bu.y * up.x) + (bl.x * dn.y + bl.y * dn.x);
            const double f = __shfl_sync(0xFFFFFFFFu, k <= 32 ? f_lo : f_hi, (k - 1) & 31);  // term <- i f T term
            term = make_double2(-f * ti, f * tr);
            acc.x += term.x;
            acc.y += term.y;
            // max |re| + |im| of the term <= 1e-18 of the sum's?  Their largest
            // parts' exponents bound both within a factor 4 (1e-18 = 2^-59.8),
            // so the FP64 maxima are taken only near the line
            const int eT = __reduce_max_sync(0xFFFFFFFFu, part_exponent(term)) >> 20;
            const int eA = __reduce_max_sync(0xFFFFFFFFu, part_exponent(acc)) >> 20;
            if (eT - eA >= -57) continue;
            if (eT - eA <= -62) break;
            const double tm = warp_max(fabs(term.x) + fabs(term.y));
            const double am = warp_max(fabs(acc.x) + fabs(acc.y));
            if (tm <= 1e-18 * am) break;
        }
        y = acc;
    }
    if (on) st->coef[lane] = y;
}

__global__ void __launch_bounds__(KT) k_combine(const KrylovState *st, double2 *const *V, double2 *out,
                                                KrylovLens nl) {
    allow_dependents();
    dependency_wait();
    const int m = st->iters;
    if (m <= 0) return;
    const int64_t n = nl.n[m - 1];
    for (int64_t i = blockIdx.x * (int64_t)KT + threadIdx.x; i < n; i += (int64_t)gridDim.x * KT) {
        double2 acc = make_double2(0.0, 0.0);
        for (int j = 0; j < m; ++j) {
            if (i >= nl.n[j]) continue;
            acc = cmul_acc(acc, st->coef[j], V[j][i]);
        }
        out[i] = acc;
    }
}

__global__ void k_store_norm2(const double2 *parts, int nparts, double *result) {
    double2 s = reduce_partials(parts, nparts);
    if (threadIdx.x == 0) *result = s.x;
}

}  // namespace

int reduce_parts() { return std::max(1, std::min(512, 2 * ctx().num_sms)); }

void krylov_start(KrylovState *st, const double2 *psi, double2 *v0, int64_t n, double2 *parts, int *stop) {
    const int np = reduce_parts();
    k_norm_part<<<np, KT, 0, ctx().stream>>>(psi, n, parts);
    counted();
    launch_dependent(k_start, (unsigned)np, KT, 0, 0, st, psi, v0, n, parts, np, stop);
    counted();
    KV_CUDA(cudaGetLastError());
}

// Whether the fused step fits one co-resident wave on this device (checked
// once per device).  The fused step runs only on the main context's stream:
// kernels of one stream never overlap, so its grid barrier waits on no
// other launch of this library.
static bool lanczos_step_fused(int device, int np) {
    static std::mutex mu;
    static int ok[64] = {};  // 0 unknown, 1 yes, -1 no
    if (device < 0 || device >= 64) return false;
    std::lock_guard<std::mutex> lk(mu);
    if (ok[device] == 0) {
        int coop = 0, per_sm = 0, sms = 0;
        KV_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device));
        KV_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
        KV_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_lanczos_step, kStepGrid, 0));
        // one CTA an SM takes every virtual CTA
        ok[device] = (coop && per_sm >= 1 && (np + sms - 1) / sms <= kMaxLocal) ? 1 : -1;
    }
    return ok[device] > 0;
}

// Largest cluster (16, else 8) of the cluster form on this device, checked once per device.
static int lanczos_cluster(int device) {
    static std::mutex mu;
    static int size[64] = {};
    if (device < 0 || device >= 64) return 8;
    std::lock_guard<std::mutex> lk(mu);
    if (size[device] == 0) {
        int n = 0;
        bool ok = true;
        auto check = [&](const void *kernel, int threads) {
            if (!ok || cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
                ok = false;
                return;
            }
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(16);
            cfg.blockDim = dim3(threads);
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeClusterDimension;
            at[0].val.clusterDim.x = 16;
            at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
            cfg.attrs = at;
            cfg.numAttrs = 1;
            ok = cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) == cudaSuccess && n > 0;
        };
        check((const void *)k_lanczos_cluster<kClusterOne>, kClusterOne);
        check((const void *)k_lanczos_cluster<kClusterMany>, kClusterMany);
        if (!ok) (void)cudaGetLastError();
        size[device] = ok ? 16 : 8;
    }
    return size[device];
}

// Longest vectors (complex elements) of the cluster form.  On the main stream
// the grid form takes about 22 us however short the vectors; a cluster's 16
// SMs take 18 us at 8496 elements, of which FP64 work (growing with the
// length) is 6.  On a worker stream the alternative is four launches.
constexpr int64_t kClusterMain = 16384, kClusterWorker = 77824;
static_assert(kClusterWorker <= (int64_t)8 * kMaxLocal * KT, "a cluster of 8 takes every virtual CTA");

void krylov_step(KrylovState *st, int k, double2 *hv, const double2 *vprev, const double2 *vk, double2 *vnext,
                 const KrylovLens &nl, double2 *parts, double tol, int max_iter, int *stop) {
    int np = reduce_parts();
    double2 *P0 = parts, *P1 = parts + np;
    cudaStream_t s = ctx().stream;
    int64_t n_prev = k > 0 ? nl.n[k - 1] : 0, n_k = nl.n[k], n_next = nl.n[k + 1];
    const bool main = &ctx() == &main_ctx();
    if (n_next <= (main ? kClusterMain : kClusterWorker)) {
        const int full = lanczos_cluster(ctx().device);
        int size = 1;  // a CTA per virtual one, up to the largest cluster
        while (size < full && (int64_t)size * KT < n_next) size *= 2;
        const bool many = (int64_t)size * KT < n_next;
        launch_dependent(many ? k_lanczos_cluster<kClusterMany> : k_lanczos_cluster<kClusterOne>, (unsigned)size,
                         many ? kClusterMany : kClusterOne, 0, (unsigned)size, st, k, hv, vprev, vk, vnext, n_prev, n_k,
                         n_next, P0, P1, np, tol, max_iter, stop);
        counted();
        return;
    }
    if (main && lanczos_step_fused(ctx().device, np)) {
        void *args[] = {&st, &k, &hv, &vprev, &vk, &vnext, &n_prev, &n_k, &n_next, &P0, &P1, &np, &tol, &max_iter,
                        &stop};
        KV_CUDA(cudaLaunchCooperativeKernel((const void *)k_lanczos_step, dim3(std::min(np, ctx().num_sms)),
                                            dim3(kStepGrid), args, 0, s));
        counted();
        return;
    }
    if (k > 0) {
        k_dot_part<<<np, KT, 0, s>>>(st, hv, vprev, n_prev, P0);
        counted();
        k_sub<<<np, KT, 0, s>>>(st, hv, vprev, vk, n_prev, n_k, P0, P1, np, &st->beta[k - 1]);
        counted();
    } else {
        k_dot_part<<<np, KT, 0, s>>>(st, hv, vk, n_k, P1);
        counted();
    }
    k_sub<<<np, KT, 0, s>>>(st, hv, vk, nullptr, n_k, n_next, P1, P0, np, &st->alpha[k]);
    counted();
    k_normalize<<<np, KT, 0, s>>>(st, hv, vnext, n_next, P0, np, k, tol, max_iter, stop);
    counted();
    KV_CUDA(cudaGetLastError());
}

void tridiag_exp(KrylovState *st, int reverse) {
    launch_dependent(k_tridiag_exp, 1, 32, 0, 0, st, reverse);
    counted();
    KV_CUDA(cudaGetLastError());
}

void krylov_finish(KrylovState *st, double2 *const *dV, double2 *out, const KrylovLens &nl, int reverse) {
    launch_dependent(k_tridiag_exp, 1, 32, 0, 0, st, reverse);
    counted();
    launch_dependent(k_combine, (unsigned)reduce_parts(), KT, 0, 0, st, dV, out, nl);
    counted();
    KV_CUDA(cudaGetLastError());
}

void vec_norm2(const double2 *x, int64_t n, double2 *parts, double *result) {
    const int np = reduce_parts();
    k_norm_part<<<np, KT, 0, ctx().stream>>>(x, n, parts);
    counted();
    k_store_norm2<<<1, KT, 0, ctx().stream>>>(parts, np, result);
    counted();
    KV_CUDA(cudaGetLastError());
}

}  // namespace kv
