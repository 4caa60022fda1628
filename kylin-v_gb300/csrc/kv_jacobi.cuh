// Complex Jacobi rotations of the mixed-precision block SVD.
//
// For a Hermitian 2x2 [[a, c], [conj(c), b]] (a, b real) the unitary
//     J = [[cs, s], [-conj(s), cs]],  s = sn * c/|c|
// with t = sign(z)/(|z| + sqrt(1 + z^2)), z = (b - a) / (2|c|),
// cs = 1/sqrt(1 + t^2), sn = t*cs, makes J^H [[a,c],[c*,b]] J diagonal.
// Applied to two columns x, y:  x' = cs x - conj(s) y,  y' = s x + cs y.
// This is the textbook (Hestenes / Rutishauser) Jacobi step; one-sided SVD
// applies it to column pairs with a = |x|^2, b = |y|^2, c = x^H y.
#pragma once

namespace kvj {

template <class T>
struct Rot {
    T cs;
    T s_re, s_im;  // s = sn * exp(i phi)
};

// (x, y) <- (cs x - conj(s) y, s x + cs y) for one complex element pair.
template <class T>
__device__ __forceinline__ void rotate_pair(const Rot<T> &r, T &xr, T &xi, T &yr, T &yi) {
    T nxr = r.cs * xr - (r.s_re * yr + r.s_im * yi);
    T nxi = r.cs * xi - (r.s_re * yi - r.s_im * yr);
    T nyr = (r.s_re * xr - r.s_im * xi) + r.cs * yr;
    T nyi = (r.s_re * xi + r.s_im * xr) + r.cs * yi;
    xr = nxr; xi = nxi; yr = nyr; yi = nyi;
}

}  // namespace kvj
