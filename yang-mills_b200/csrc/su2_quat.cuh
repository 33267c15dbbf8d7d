// su2_quat.cuh -- SU(2) links as unit quaternions (a0, a1, a2, a3),
// U = a0 I - i a.sigma (reference/rust/src/lib.rs:7-13), stored as two
// double2 planes per direction: (a0, a1) and (a2, a3).  Every product is
// re-normalised exactly as Su2::mul does (lib.rs:106-130, 212-224): divide by
// the largest magnitude, then by the Euclidean norm.  Shared by the sweep
// kernels (su2.cu) and the lattice queries (lattice_ops.cu); include only
// from translation units built with -fmad=false.
#pragma once

#include "ym_device.cuh"

namespace ym {

namespace {

struct q4 {
    double c[4];
};

// The correctly rounded quotient a / b from y, the correctly rounded
// reciprocal of b, by Markstein's method (P. Markstein, IBM J. Res. Dev. 34
// (1990) 111): a quotient within one ulp plus its exactly computed remainder
// times y rounds to RN(a / b).  a y is within two ulps, so one correction
// brings it within one and the second rounds it.  Needs a, b and the
// remainders far from underflow and overflow (common_divisor).
__device__ __forceinline__ double quotient(double a, double b, double y) {
    double q = a * y;
    q = fma(fma(-q, b, a), y, q);
    return fma(fma(-q, b, a), y, q);
}

// Whether every entry lies in [2^-300, 2^300] (zeros do not).
template <int N>
__device__ __forceinline__ bool common_divisor(const double *v) {
    unsigned lo = 0xffffffffu, hi = 0;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const unsigned w = (unsigned)__double2hiint(v[i]) & 0x7fffffffu;
        lo = min(lo, w);
        hi = max(hi, w);
    }
    return lo >= (unsigned)(1023 - 300) << 20 && hi < (unsigned)(1023 + 300) << 20;
}

// normalize_many's vectors outside common_divisor, out of line.  Zeros beside
// entries within it: the quotients in out are right but for the zeros' signs
// (a zero's quotients are zeros, of which the corrections make +0).  An
// identity start is made of such products: its plaquette at 24^4 310 us with
// the plain divisions on top of the quotients, 135 with the signs put back.  Entries
// that are tiny, huge or not finite, or nothing but zeros: plain divisions.
template <int N>
__device__ __noinline__ bool normalize_edge(const double *v, double *out) {
    double scale = 0.0;
    unsigned lo = 0xffffffffu, hi = 0;
    for (int i = 0; i < N; ++i) {
        const unsigned w = (unsigned)__double2hiint(v[i]) & 0x7fffffffu;
        lo = min(lo, v[i] == 0.0 ? 0xffffffffu : w);
        hi = max(hi, w);
    }
    if (lo != 0xffffffffu && lo >= (unsigned)(1023 - 300) << 20 && hi < (unsigned)(1023 + 300) << 20) {
        for (int i = 0; i < N; ++i) out[i] = copysign(out[i], v[i]);
        return true;
    }
    for (int i = 0; i < N; ++i) scale = fmax(scale, fabs(v[i]));
    if (scale == 0.0 || !isfinite(scale)) return false;
    double s[N];
    for (int i = 0; i < N; ++i) s[i] = v[i] / scale;
    double ss = s[0] * s[0];
    for (int i = 1; i < N; ++i) ss = ss + s[i] * s[i];
    const double norm = sqrt(ss);
    if (norm == 0.0 || !isfinite(norm)) return false;
    for (int i = 0; i < N; ++i) out[i] = s[i] / norm;
    return true;
}

// normalize_scaled (lib.rs:106-130) of M independent vectors of N entries:
// divide by the largest magnitude, then by the norm.  The N quotients of each
// division share one reciprocal when the entries' sizes allow it (any vector
// with an entry that is zero, tiny, huge or not finite goes through
// normalize_edge afterwards); both ways round the same.  A division is about 16
// instructions, a quotient 5.  The M chains have no branch between them, so
// they overlap.  Returns whether vector i could be normalised in bit i;
// out[i] is left alone where it could not.
template <int N, int M>
__device__ __forceinline__ unsigned normalize_many(const double (*v)[N], double (*out)[N]) {
    unsigned good = 0;
    double o[M][N];
#pragma unroll
    for (int m = 0; m < M; ++m) {
        good |= common_divisor<N>(v[m]) ? 1u << m : 0u;
        double scale = 0.0;
#pragma unroll
        for (int i = 0; i < N; ++i) scale = fmax(scale, fabs(v[m][i]));
        double s[N];
        const double ys = __drcp_rn(scale);
#pragma unroll
        for (int i = 0; i < N; ++i) s[i] = quotient(v[m][i], scale, ys);
        double ss = s[0] * s[0];
#pragma unroll
        for (int i = 1; i < N; ++i) ss = ss + s[i] * s[i];
        const double norm = sqrt(ss);   // one entry is +-1, so 1 <= norm <= 2
        const double yn = __drcp_rn(norm);
#pragma unroll
        for (int i = 0; i < N; ++i) o[m][i] = quotient(s[i], norm, yn);
    }
    if (good != (1u << M) - 1u) {
#pragma unroll
        for (int m = 0; m < M; ++m)
            if (!(good & (1u << m))) {
                double in[N], edge[N];
#pragma unroll
                for (int i = 0; i < N; ++i) {
                    in[i] = v[m][i];
                    edge[i] = o[m][i];
                }
                const bool ok = normalize_edge<N>(in, edge);
#pragma unroll
                for (int i = 0; i < N; ++i) o[m][i] = ok ? edge[i] : out[m][i];
                good |= ok ? 1u << m : 0u;
            }
    }
#pragma unroll
    for (int m = 0; m < M; ++m)
#pragma unroll
        for (int i = 0; i < N; ++i) out[m][i] = o[m][i];
    return good;
}

template <int N>
__device__ __forceinline__ bool normalize_scaled(const double *v, double *out) {
    double in[1][N], o[1][N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
        in[0][i] = v[i];
        o[0][i] = out[i];
    }
    const bool ok = normalize_many<N, 1>(in, o) != 0;
#pragma unroll
    for (int i = 0; i < N; ++i) out[i] = o[0][i];
    return ok;
}

// Su2::mul (lib.rs:212-224) of M independent pairs; a raw product is kept if
// its normalisation fails, which cannot happen for finite unit inputs (the
// reference panics there).
template <int M>
__device__ __forceinline__ void qmul_many(const q4 *a, const q4 *b, q4 *o) {
    double raw[M][4], n[M][4];
#pragma unroll
    for (int m = 0; m < M; ++m) {
        const double a0 = a[m].c[0], a1 = a[m].c[1], a2 = a[m].c[2], a3 = a[m].c[3];
        const double b0 = b[m].c[0], b1 = b[m].c[1], b2 = b[m].c[2], b3 = b[m].c[3];
        raw[m][0] = a0 * b0 - a1 * b1 - a2 * b2 - a3 * b3;
        raw[m][1] = a0 * b1 + a1 * b0 + a2 * b3 - a3 * b2;
        raw[m][2] = a0 * b2 - a1 * b3 + a2 * b0 + a3 * b1;
        raw[m][3] = a0 * b3 + a1 * b2 - a2 * b1 + a3 * b0;
#pragma unroll
        for (int i = 0; i < 4; ++i) n[m][i] = raw[m][i];
    }
    normalize_many<4, M>(raw, n);
#pragma unroll
    for (int m = 0; m < M; ++m)
#pragma unroll
        for (int i = 0; i < 4; ++i) o[m].c[i] = n[m][i];
}

__device__ __forceinline__ q4 qmul(const q4 &a, const q4 &b) {
    q4 o;
    qmul_many<1>(&a, &b, &o);
    return o;
}

__device__ __forceinline__ q4 qdag(const q4 &a) { return q4{{a.c[0], -a.c[1], -a.c[2], -a.c[3]}}; }

__device__ __forceinline__ q4 load_q(const double2 *__restrict__ links, const ChainInfo &c,
                                     int64_t s, int mu) {
    const double2 *p = links + c.offset + (int64_t)(mu * 2) * c.volume + s;
    const double2 lo = __ldg(p), hi = __ldg(p + c.volume);
    return q4{{lo.x, lo.y, hi.x, hi.y}};
}

__device__ __forceinline__ q4 load_q_rw(const double2 *links, const ChainInfo &c, int64_t s, int mu) {
    const double2 *p = links + c.offset + (int64_t)(mu * 2) * c.volume + s;
    const double2 lo = p[0], hi = p[c.volume];
    return q4{{lo.x, lo.y, hi.x, hi.y}};
}

__device__ __forceinline__ void store_q(double2 *links, const ChainInfo &c, int64_t s, int mu,
                                        const q4 &q) {
    double2 *p = links + c.offset + (int64_t)(mu * 2) * c.volume + s;
    p[0] = make_double2(q.c[0], q.c[1]);
    p[c.volume] = make_double2(q.c[2], q.c[3]);
}

__device__ __forceinline__ q4 link_q(const double2 *links, const ChainInfo &c, const Nb &n, int mu) {
    return load_q(links, c, storage_index(c, n.lex, n.par), mu);
}

}  // namespace

}  // namespace ym
