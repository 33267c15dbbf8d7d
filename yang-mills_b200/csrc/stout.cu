// stout.cu -- spatial stout smearing of SU(3) lattices, one synchronous
// level per launch (glueball_smearing.rs:137-268): for every site and
// spatial mu,
//   C  = rho * sum_{nu spatial != mu} [ U_nu(x) U_mu(x+nu) U_nu(x+mu)^dag
//                                      + U_nu(x-nu)^dag U_mu(x-nu) U_nu(x-nu+mu) ]
//   Om = C U^dag,  A = Om^dag - Om,
//   Q  = (i/2) A - (i/6) Tr(A) 1,           checked Hermitian and traceless,
//   c_a = Re Tr(Q lambda_a),                 checked |Im| <= 2e-12,
//   U' = exp(i sum_a c_a T^a) U             (scale-and-square exponential,
//                                            su3.rs:395-450), checked in SU(3);
// temporal links are copied.  A failed gate sets the device error flag
// (the reference returns an error).  Levels ping-pong between two buffers.
//
// Results are held to a tolerance (1e-14 against the oracle per level, the
// reference goldens' 1e-12), not bitwise, so this unit is compiled with
// fused multiply-adds.
#include <cuda_runtime.h>

#include "su3_checks.cuh"
#include "ym_internal.hpp"

namespace ym {

namespace {

constexpr int T = kSiteThreads;

// A Hermitian 3x3 matrix: its real diagonal and the upper triangle.
struct herm3 {
    double d[3];
    cplx o01, o02, o12;
};

// a 1 + b H + c H^2 times H^2, by Cayley-Hamilton for a traceless Hermitian
// H: H^3 = h H + e 1 with h = Tr(H^2)/2, e = det H, both real.
struct poly3 {
    double a, b, c;
};

__device__ __forceinline__ poly3 times_h2(const poly3 &f, double h, double e) {
    return poly3{f.b * e, fma(f.b, h, f.c * e), fma(f.c, h, f.a)};
}

// Su3::from_algebra_coefficients (su3.rs:255-262, 395-450): exp(i H), H =
// sum_a c_a T^a accumulated in generator order, scaled by 2^-k to 1-norm <=
// 0.5 (the reference's rule), exponentiated, squared k times.  The reference
// sums the dense Taylor series until a term's largest entry is <= 1e-18;
// here exp(i H) = cos H + i sin H, each a polynomial in H reduced by
// Cayley-Hamilton to three real coefficients and summed by Horner's rule
// through order 16 / 17: with the scaled 1-norm <= 0.5 the next terms are
// below 0.5^18 / 18! < 1e-18, so at least the reference's terms are summed,
// and the result agrees with the dense series to rounding (1e-16 per level
// at the coefficient sizes smearing produces).  Real arithmetic on the six
// distinct entries takes about 230 operations, the complex recurrence on
// full matrices took 550.
__device__ __forceinline__ bool from_algebra(const double coef[8], m3 &out) {
#pragma unroll
    for (int a = 0; a < 8; ++a)
        if (!isfinite(coef[a]) || fabs(coef[a]) > 64.0) return false;
    // H = sum_a c_a lambda_a / 2, entries written out
    const double h3 = 0.5 * coef[2], h8 = 0.5 * kInvSqrt3d * coef[7];
    herm3 x{{h3 + h8, -h3 + h8, -2.0 * h8},
            cmake(0.5 * coef[0], -0.5 * coef[1]),
            cmake(0.5 * coef[3], -0.5 * coef[4]),
            cmake(0.5 * coef[5], -0.5 * coef[6])};
    // 1-norm, the largest column sum of |h_rc| (|h_rc| = |h_cr|); |re| + |im|
    // bounds an entry from above, and when that bound is within 0.5 the norm
    // itself is not needed
    auto norm_of = [&](double o01, double o02, double o12) {
        return fmax(fmax((fabs(x.d[0]) + o01) + o02, (o01 + fabs(x.d[1])) + o12), (o02 + o12) + fabs(x.d[2]));
    };
    auto l1 = [](cplx z) { return fabs(z.re) + fabs(z.im); };
    int squarings = 0;
    if (!(norm_of(l1(x.o01), l1(x.o02), l1(x.o12)) <= 0.5)) {
        double norm = norm_of(sqrt(norm2(x.o01)), sqrt(norm2(x.o02)), sqrt(norm2(x.o12)));
        if (!isfinite(norm)) return false;
        while (norm > 0.5) {
            squarings++;
            if (squarings > 32) return false;
            norm *= 0.5;
        }
        const double f = ldexp(1.0, -squarings);
#pragma unroll
        for (int i = 0; i < 3; ++i) x.d[i] *= f;
        x.o01 = cmake(x.o01.re * f, x.o01.im * f);
        x.o02 = cmake(x.o02.re * f, x.o02.im * f);
        x.o12 = cmake(x.o12.re * f, x.o12.im * f);
    }
    // H^2
    const double n01 = norm2(x.o01), n02 = norm2(x.o02), n12 = norm2(x.o12);
    herm3 y;
    y.d[0] = fma(x.d[0], x.d[0], n01 + n02);
    y.d[1] = fma(x.d[1], x.d[1], n01 + n12);
    y.d[2] = fma(x.d[2], x.d[2], n02 + n12);
    auto entry = [](cplx z, double s, cplx p, cplx q) {   // z s + p q
        cplx v = cmake(z.re * s, z.im * s);
        cfma(v, p, q);
        return v;
    };
    y.o01 = entry(x.o01, x.d[0] + x.d[1], x.o02, cconj(x.o12));
    y.o02 = entry(x.o02, x.d[0] + x.d[2], x.o01, x.o12);
    y.o12 = entry(x.o12, x.d[1] + x.d[2], cconj(x.o01), x.o02);
    const double h = 0.5 * ((y.d[0] + y.d[1]) + y.d[2]);
    const cplx p = cmul(x.o01, x.o12);   // h01 h12, times h20 = conj(h02)
    const double e = fma(x.d[0], x.d[1] * x.d[2],
                         2.0 * fma(p.re, x.o02.re, p.im * x.o02.im)) -
                     fma(x.d[0], n12, fma(x.d[1], n02, x.d[2] * n01));
    // cos = 1 - H^2/(1 2) (1 - H^2/(3 4) (...)), sin = H (1 - H^2/(2 3) (...))
    poly3 cs{1.0, 0.0, 0.0}, sn{1.0, 0.0, 0.0};
#pragma unroll
    for (int m = 8; m >= 1; --m) {
        const double ic = -1.0 / ((2 * m - 1) * (2 * m)), is = -1.0 / ((2 * m) * (2 * m + 1));
        const poly3 c = times_h2(cs, h, e), s = times_h2(sn, h, e);
        cs = poly3{fma(c.a, ic, 1.0), c.b * ic, c.c * ic};
        sn = poly3{fma(s.a, is, 1.0), s.b * is, s.c * is};
    }
    // sin's leading factor H: (a + b H + c H^2) H = c e + (a + c h) H + b H^2
    const cplx f0 = cmake(cs.a, sn.c * e), f1 = cmake(cs.b, fma(sn.c, h, sn.a)), f2 = cmake(cs.c, sn.b);
    m3 sum;
    auto place = [&](int i, int j, cplx hx, cplx hy) {
        cplx v = cmul(f1, hx);
        cfma(v, f2, hy);
        sum.e[i][j] = v;
    };
#pragma unroll
    for (int i = 0; i < 3; ++i)
        sum.e[i][i] = cmake(fma(f2.re, y.d[i], fma(f1.re, x.d[i], f0.re)), fma(f2.im, y.d[i], fma(f1.im, x.d[i], f0.im)));
    place(0, 1, x.o01, y.o01);
    place(1, 0, cconj(x.o01), cconj(y.o01));
    place(0, 2, x.o02, y.o02);
    place(2, 0, cconj(x.o02), cconj(y.o02));
    place(1, 2, x.o12, y.o12);
    place(2, 1, cconj(x.o12), cconj(y.o12));
    for (int k = 0; k < squarings; ++k) sum = mul_fma(sum, sum);
    if (!finite3(sum)) return false;
    out = sum;
    return true;
}

// a^dagger b, every entry one chain of cfma() over k = 0, 1, 2 from zero.
__device__ __forceinline__ m3 adj_mul_fma(const m3 &a, const m3 &b) {
    m3 o;
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            cplx v = cmake(0.0, 0.0);
#pragma unroll
            for (int k = 0; k < 3; ++k) cfma(v, cconj(a.e[k][r]), b.e[k][c]);
            o.e[r][c] = v;
        }
    return o;
}

__device__ __forceinline__ m3 lk(const double2 *links, const ChainInfo &c, const Nb &n, int mu) {
    return load_su3(links, c, storage_index(c, n.lex, n.par), mu);
}

// acc += p q, every entry a chain of cfma() over k.
__device__ __forceinline__ void add_product(m3 &acc, const m3 &p, const m3 &q) {
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int k = 0; k < 3; ++k) cfma(acc.e[r][c], p.e[r][k], q.e[k][c]);
}

__device__ __forceinline__ void add_product_adj(m3 &acc, const m3 &p, const m3 &q) {
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int k = 0; k < 3; ++k) cfma(acc.e[r][c], p.e[r][k], cconj(q.e[c][k]));
}

// One thread per (site, spatial mu): block 3 t + mu takes tile t, so the
// three blocks that read the same links run next to each other; the mu = 0
// block also copies the temporal links.
//
// What bounds it: binary64 issue (52 % of the pipe's cycles) with L2 loads
// behind it (3.5 GB per level of 128 x 4^3x10 + 64 x 6^3x12 + 32 x 8^3x16,
// 12.5 TB/s).  That level: 396 us with one thread per site, the complex
// recurrence and both unitarity products, 280 us now; 24^3 x 48 538 -> 348
// us, 9^3 x 15 36 -> 16 us (three times the blocks).  Four blocks per SM at
// 128 registers; three 381 us (24^3 x 48), two 421, five 456.  Also measured
// on 24^3 x 48: the three directions of 32 sites in one block (so that their
// loads might meet in L1) 385 us, factors staged by cp.async 353 (three
// blocks 331, but 1 % slower on the uneven batch).
__global__ void __launch_bounds__(T, 4)
k_stout_level(const ChainInfo *__restrict__ chains, const Tile *__restrict__ tiles,
              const double2 *__restrict__ in, double2 *__restrict__ out, double rho,
              unsigned *__restrict__ err, int reverse) {
    const unsigned b = reverse ? gridDim.x - 1 - blockIdx.x : blockIdx.x;
    const int mu = (int)(b % 3);
    const Tile tile = tiles[b / 3];
    const ChainInfo c = chains[tile.chain];
    const int64_t s = tile.start + threadIdx.x;
    if (s >= c.volume) return;
    const Coord x = decode_storage(c, s);
    const Nb self{x.lex, x.par};
    if (mu == 0) store_su3(out, c, s, 3, load_su3(in, c, s, 3));           // temporal copied
    const Nb pm = step_any(c, x.x, x.lex, x.par, mu, +1);
    m3 staple;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) staple.e[i][j] = cmake(0.0, 0.0);
#pragma unroll 1
    for (int i = 0; i < 2; ++i) {
        const int nu = i + (i >= mu ? 1 : 0);
        const Nb pn = step_any(c, x.x, x.lex, x.par, nu, +1);
        const Nb mn = step_any(c, x.x, x.lex, x.par, nu, -1);
        const Nb mnpm = step_any(c, x.x, mn.lex, mn.par, mu, +1);
        add_product_adj(staple, mul_fma(lk(in, c, self, nu), lk(in, c, pn, mu)), lk(in, c, pm, nu));
        add_product(staple, adj_mul_fma(lk(in, c, mn, nu), lk(in, c, mn, mu)), lk(in, c, mnpm, nu));
    }
    const m3 old = load_su3(in, c, s, mu);
    // stout_q (glueball_smearing.rs:174-193): Om = rho C U^dag, A = Om^dag - Om,
    // Q = (i/2) A - (i/6) Tr(A).  A is anti-Hermitian entry for entry, so Q is
    // exactly Hermitian and the reference's Hermiticity gate cannot fail; a
    // non-finite staple leaves a non-finite Om.
    const m3 omega = mul_adj_fma(scale_r(staple, rho), old);
    bool finite = finite3(omega);
    const double t6 = (2.0 * ((omega.e[0][0].im + omega.e[1][1].im) + omega.e[2][2].im)) * (1.0 / 6.0);
    const double q00 = omega.e[0][0].im - t6, q11 = omega.e[1][1].im - t6, q22 = omega.e[2][2].im - t6;
    // i/2 (conj(om_ji) - om_ij) of an upper entry
    auto upper = [&](int i, int j) {
        return cmake(0.5 * (omega.e[j][i].im + omega.e[i][j].im), 0.5 * (omega.e[j][i].re - omega.e[i][j].re));
    };
    const cplx q01 = upper(0, 1), q02 = upper(0, 2), q12 = upper(1, 2);
    finite = finite && isfinite(q00) && isfinite(q11) && isfinite(q22) && isfinite(q01.re) && isfinite(q01.im) &&
             isfinite(q02.re) && isfinite(q02.im) && isfinite(q12.re) && isfinite(q12.im);
    if (!finite) { atomicOr(err, kErrNonFiniteStaple); return; }
    if (fabs((q00 + q11) + q22) > kAlgebraTol) { atomicOr(err, kErrProjection); return; }
    // q_coefficients (glueball_smearing.rs:195-205): Tr(Q lambda_a), real for
    // a Hermitian Q
    const double coef[8] = {q01.re + q01.re, -(q01.im + q01.im), q00 - q11, q02.re + q02.re, -(q02.im + q02.im),
                            q12.re + q12.re, -(q12.im + q12.im),
                            (q00 + q11) * kInvSqrt3d - q22 * (2.0 * kInvSqrt3d)};
    bool ok = true;
#pragma unroll
    for (int a = 0; a < 8; ++a) ok = ok && isfinite(coef[a]);
    if (!ok) { atomicOr(err, kErrProjection); return; }
    m3 rot;
    if (!from_algebra(coef, rot) || !in_su3(rot)) { atomicOr(err, kErrGroup); return; }
    const m3 upd = mul_fma(rot, old);
    if (!in_su3(upd)) { atomicOr(err, kErrGroup); return; }
    store_su3(out, c, s, mu, upd);
}

}  // namespace

cudaError_t launch_stout_level(ym_ensemble *e, const double2 *in, double2 *out, double rho, int reverse) {
    k_stout_level<<<(unsigned)(3 * e->n_site_tiles), T, 0, e->stream>>>(e->d_chains, e->d_mixed_tiles, in, out,
                                                                 rho, e->d_error, reverse);
    return cudaGetLastError();
}

}  // namespace ym
