// Device arithmetic of the FP64 Jacobi rotations (kv_svd64.cu): reciprocals and
// roots by Newton steps, and the rotation of a column pair.
#pragma once
#include <cstdint>

namespace kv {
namespace rot64 {

// x = m 2^e with |m| in [1, 2) as FP32 (truncated to 24 bits); zero and
// subnormal x give m = 0.  Integer operations only.
__device__ __forceinline__ float mantissa(double x, int &e) {
    const int hi = __double2hiint(x);
    const unsigned lo = (unsigned)__double2loint(x);
    const int E = (hi >> 20) & 0x7FF;
    e = E - 1023;
    if (E == 0) return 0.f;
    return __int_as_float((hi & (int)0x80000000) | (127 << 23) | ((hi & 0xFFFFF) << 3) | (int)(lo >> 29));
}
// 2^e as FP32, e clamped to [-126, 127]
__device__ __forceinline__ float pow2f(int e) { return __int_as_float((min(max(e, -126), 127) + 127) << 23); }
// an FP32 value as FP64 (exact; FP32 subnormals as zero).  Integer operations only.
__device__ __forceinline__ double widen(float x) {
    const int u = __float_as_int(x), E = (u >> 23) & 0xFF, m = u & 0x7FFFFF;
    if (E == 0) return 0.0;
    return __hiloint2double((u & (int)0x80000000) | ((E - 127 + 1023) << 20) | (m >> 3), m << 29);
}

// 1 / sqrt(x) and 1 / x for normal x > 0 away from the range's ends: two Newton
// steps on an FP32 start, about ten FP64 instructions each in place of some
// thirty (64 clocks a warp each), to within two units in the last place
__device__ __forceinline__ double newton_rsqrt(double x) {
    int e;
    float m = mantissa(x, e);
    if (e & 1) m *= 2.f;
    e = (e - (e & 1)) / 2;
    double y = __hiloint2double(__double2hiint(widen(rsqrtf(m))) - (e << 20), __double2loint(widen(rsqrtf(m))));
    y = fma(y * 0.5, fma(-x * y, y, 1.0), y);
    return fma(y * 0.5, fma(-x * y, y, 1.0), y);
}
__device__ __forceinline__ double newton_reciprocal(double x) {
    int e;
    const double r = widen(__fdividef(1.f, mantissa(x, e)));
    double y = __hiloint2double(__double2hiint(r) - (e << 20), __double2loint(r));
    y = fma(y, fma(-x, y, 1.0), y);
    return fma(y, fma(-x, y, 1.0), y);
}

// The Jacobi rotation of a column pair with |x|^2 = a, |y|^2 = b, x^H y = c
// != 0 (x' = cs x - conj(s) y, y' = s x + cs y): tau = t c/|c| with
// t = sign(z) / (|z| + sqrt(1 + z^2)), z = (b - a) / (2|c|), in FP32; then
// cs = 1 / sqrt(1 + |tau|^2) and s = cs tau in FP64 (two Newton steps on the
// FP32 reciprocal square root), unitary to FP64 rounding.
__device__ __forceinline__ void rotation(double a, double b, double cr, double ci, double &cs, double &sr,
                                         double &si) {
    int er, ei, ed;
    const float mr = mantissa(cr, er), mi = mantissa(ci, ei), md = mantissa(b - a, ed);
    const int ec = mr == 0.f ? ei : mi == 0.f ? er : max(er, ei);
    const float fr = mr == 0.f ? 0.f : mr * pow2f(er - ec), fi = mi == 0.f ? 0.f : mi * pow2f(ei - ec);
    const float rn = rsqrtf(fr * fr + fi * fi);  // 1 / (|c| 2^-ec)
    const float z0 = 0.5f * md * rn;             // z 2^(ec - ed), |z0| < 1
    const int ez = ed - ec;
    double tr, ti;
    if (ez > 60) {  // |z| > 2^58: tau = c / (b - a), which may be below FP32's range
        const double inv = 1.0 / (b - a);
        tr = cr * inv;
        ti = ci * inv;
    } else {
        const float z = z0 * pow2f(ez);
        const float t = copysignf(__fdividef(1.f, fabsf(z) + sqrtf(fmaf(z, z, 1.f))), z);
        tr = widen(t * fr * rn);
        ti = widen(t * fi * rn);
    }
    const double w = fma(tr, tr, fma(ti, ti, 1.0));  // in [1, 2]
    cs = newton_rsqrt(w);
    sr = cs * tr;
    si = cs * ti;
}

// |c|^2 > tol2 a b for short columns, whose products would underflow: exponents
// apart, mantissas in FP32 (a tolerance needs no more)
__device__ __forceinline__ bool above_tolerance(double a, double b, double cr, double ci, double tol2) {
    int ea, eb, er, ei;
    const float ma = mantissa(a, ea), mb = mantissa(b, eb), mr = mantissa(cr, er), mi = mantissa(ci, ei);
    const int ec = mr == 0.f ? ei : mi == 0.f ? er : max(er, ei);
    const float fr = mr == 0.f ? 0.f : mr * pow2f(er - ec), fi = mi == 0.f ? 0.f : mi * pow2f(ei - ec);
    return fmaf(fr, fr, fi * fi) * pow2f(2 * ec - ea - eb) > (float)tol2 * ma * mb;
}

}  // namespace rot64
}  // namespace kv
