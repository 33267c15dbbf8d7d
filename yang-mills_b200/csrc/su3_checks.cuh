// su3_checks.cuh -- the gauge-observable units' dense 3x3 helpers and the
// reference's acceptance gates (finite entries, unitarity and determinant
// residuals) shared by stout smearing and blocking.
#pragma once

#include "ym_device.cuh"

namespace ym {

namespace {

constexpr double kAlgebraTol = 2.0e-12;   // ALGEBRA_RESIDUAL_TOLERANCE glueball_smearing.rs:26
constexpr double kSu3Tol = 5.0e-12;       // SU3_ACCEPTANCE_TOLERANCE su3.rs:20
constexpr double kInvSqrt3d = 0.5773502691896258;

constexpr unsigned kErrProjection = 4u;
constexpr unsigned kErrGroup = 8u;
constexpr unsigned kErrNonFiniteStaple = 16u;

__device__ __forceinline__ double norm2(cplx z) { return z.re * z.re + z.im * z.im; }

__device__ __forceinline__ bool finite3(const m3 &m) {
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j)
            if (!isfinite(m.e[i][j].re) || !isfinite(m.e[i][j].im)) return false;
    return true;
}

__device__ __forceinline__ m3 scale_r(const m3 &a, double f) {
    m3 o;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) o.e[i][j] = cmake(a.e[i][j].re * f, a.e[i][j].im * f);
    return o;
}

__device__ __forceinline__ cplx trace3(const m3 &a) { return cadd(cadd(a.e[0][0], a.e[1][1]), a.e[2][2]); }

__device__ __forceinline__ cplx det3(const m3 &m) {
    const cplx t1 = cmul(m.e[0][0], csub(cmul(m.e[1][1], m.e[2][2]), cmul(m.e[1][2], m.e[2][1])));
    const cplx t2 = cmul(m.e[0][1], csub(cmul(m.e[1][0], m.e[2][2]), cmul(m.e[1][2], m.e[2][0])));
    const cplx t3 = cmul(m.e[0][2], csub(cmul(m.e[1][0], m.e[2][1]), cmul(m.e[1][1], m.e[2][0])));
    return cadd(csub(t1, t2), t3);
}

// max |entry|^2 of u u^dag - 1 (ROWS) or u^dag u - 1.  Both are Hermitian, so
// the upper triangle (diagonal included) carries every distinct magnitude;
// only those six entries are formed.
template <bool ROWS>
__device__ __forceinline__ double gram_res2(const m3 &u) {
    double r = 0.0;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = i; j < 3; ++j) {
            cplx g = cmake(i == j ? -1.0 : 0.0, 0.0);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                if (i == j) {
                    const cplx z = ROWS ? u.e[i][k] : u.e[k][i];
                    g.re = fma(z.re, z.re, g.re);
                    g.re = fma(z.im, z.im, g.re);
                } else if (ROWS) {
                    cfma(g, u.e[i][k], cconj(u.e[j][k]));
                } else {
                    cfma(g, cconj(u.e[k][i]), u.e[k][j]);
                }
            }
            r = fmax(r, i == j ? g.re * g.re : norm2(g));
        }
    return r;
}

// Whether Mat3::unitarity_residual (su3.rs:219-223), the larger of
// max |U U^dag - 1| and max |U^dag U - 1|, is at most kSu3Tol.  The two
// deviations have the same singular values, so the largest entry of one is
// at most their common Frobenius norm, at most three times the largest entry
// of the other: below a quarter of the tolerance the first decides both.
__device__ __forceinline__ bool unitary_within(const m3 &u) {
    const double r = gram_res2<true>(u);
    if (r <= kSu3Tol * kSu3Tol * (1.0 / 16.0)) return true;
    return r <= kSu3Tol * kSu3Tol && gram_res2<false>(u) <= kSu3Tol * kSu3Tol;
}

// Su3::from_checked_matrix gate (su3.rs:20, 241-252): finite, unitarity residual
// and |det U - 1| within 5e-12.  The reference also takes |det(U^dag) - 1|,
// which is the same number (det U^dag is the conjugate of det U).
__device__ __forceinline__ bool in_su3(const m3 &u) {
    if (!finite3(u)) return false;
    if (!unitary_within(u)) return false;
    return norm2(csub(det3(u), cmake(1.0, 0.0))) <= kSu3Tol * kSu3Tol;
}

}  // namespace

}  // namespace ym
