// su3_tiled.cuh -- the tiled SU(3) FP64 Metropolis sub-sweep, the engine's
// hot kernels.
//
// One launch updates every link U_mu(x) with x of one checkerboard parity,
// in every chain of the ensemble: staple sum -> eight Metropolis hits ->
// store.  The per-link update rule is the reference's metropolis_sweep
// (reference/rust/src/su3_ensemble.rs:342-391): proposal R = exp(i theta T^a)
// on the paired angle grid, candidate R*U, accept iff u < exp(-max(dS, 0)),
// two stream words per hit.  Links of one parity and direction do not touch
// each other's staples, so all of them update concurrently.
//
// Two translation units compile these kernels:
//   * su3_metropolis.cu (-fmad=false): the reference's bits.  The candidate
//     R*U is the reference's (dense-order products, no fused multiply-add);
//     the staple sum A and the contraction Re Tr(X A) are the engine's own
//     formulation of the action change, dS = (beta/3)(ReTr(U A) - ReTr(U'A)),
//     written as fixed chains of fma() that the CPU oracle repeats bit for
//     bit;
//   * su3_metropolis_fast.cu (YM_TILED_FAST, fused multiply-adds): the same
//     algorithm in binary64 with every product free to round once, and the
//     rotation entries from cos_sin_horner instead of the reference's Taylor
//     recurrence (ym_ensemble_set_fast_sweeps).
//
// Layout: every factor of the six staple terms is copied global -> shared by
// cp.async ahead of its use.  k_su3_metropolis_ring keeps the staple
// accumulator in registers and stages two terms ahead, two persistent
// 128-thread blocks per SM; for the hits the accumulator goes to shared
// memory (nine double2 per thread, conflict-free column layout).
#pragma once
#include <cuda_runtime.h>

#include "su3_exp.cuh"
#include "su3_sites.cuh"
#include "ym_internal.hpp"

// The two compilations live in different namespaces, so that their kernels
// are told apart by name (profilers show ym::tiled_exact::... and
// ym::tiled_fast::...).
#ifdef YM_TILED_FAST
#define YM_TILED_NS tiled_fast
#else
#define YM_TILED_NS tiled_exact
#endif

namespace ym {
namespace YM_TILED_NS {
namespace {

constexpr int T = kSweepThreads;

// A matrix held as nine double2 in memory, entry e at p[e * stride]: a
// thread's column of a [9][T] shared buffer (S = T, offsets are immediates),
// or a link of a chain held in shared memory (S = 0, stride the volume).
template <int S>
struct Col {
    double2 *p;
    int stride;
    __device__ __forceinline__ double2 *at(int e) const { return p + e * (S ? S : stride); }
    __device__ __forceinline__ cplx get(int e) const {
        const double2 v = *at(e);
        return cmake(v.x, v.y);
    }
    __device__ __forceinline__ void put(int e, cplx v) const { *at(e) = make_double2(v.re, v.im); }
    // row i (entries 3 i ..), column i (entries i, 3 + i, 6 + i)
    __device__ __forceinline__ void row(int i, cplx r[3]) const {
#pragma unroll
        for (int k = 0; k < 3; ++k) r[k] = get(3 * i + k);
    }
    __device__ __forceinline__ void column(int i, cplx c[3]) const {
#pragma unroll
        for (int k = 0; k < 3; ++k) c[k] = get(3 * k + i);
    }
};

__device__ __forceinline__ Col<T> column_of(double2 (*buf)[T]) { return Col<T>{&buf[0][threadIdx.x], T}; }

// A link from this thread's column of a staging buffer.
__device__ __forceinline__ m3 staged_link(const double2 (*buf)[T]) {
    m3 o;
#pragma unroll
    for (int e = 0; e < 9; ++e) {
        const double2 v = buf[e][threadIdx.x];
        o.e[e / 3][e % 3] = cmake(v.x, v.y);
    }
    return o;
}

// Fast form only (YM_TILED_FAST): cos h and sin h as polynomials in
// y = h^2 by Horner's rule with fused multiply-adds, the Taylor coefficients
// 1/k! truncated where the next term is below 1e-19 for the half widths
// served: through h^14 / h^15 for K <= 13 (|h| <= 0.231), through h^18 /
// h^19 above (|h| <= 0.578).
template <int K>
__device__ __forceinline__ void cos_sin_horner(double h, double &c, double &s) {
    constexpr int NT = K <= 13 ? 7 : 9;
    constexpr double kc[10] = {1.0, -1.0 / 2, 1.0 / 24, -1.0 / 720, 1.0 / 40320, -1.0 / 3628800,
                               1.0 / 479001600, -1.0 / 87178291200.0, 1.0 / 20922789888000.0,
                               -1.0 / 6402373705728000.0};
    constexpr double ks[10] = {1.0, -1.0 / 6, 1.0 / 120, -1.0 / 5040, 1.0 / 362880, -1.0 / 39916800,
                               1.0 / 6227020800.0, -1.0 / 1307674368000.0, 1.0 / 355687428096000.0,
                               -1.0 / 121645100408832000.0};
    const double y = h * h;
    double pc = kc[NT], ps = ks[NT];
#pragma unroll
    for (int k = NT - 1; k >= 0; --k) {
        pc = fma(pc, y, kc[k]);
        ps = fma(ps, y, ks[k]);
    }
    c = pc;
    s = h * ps;
}

// ---- the hits, software-pipelined ------------------------------------------
// A hit has a link-independent half (its two stream words, the angle, the
// rotation entries from the Taylor chain, the accept threshold) and a
// link-dependent half (candidate rows, Re Tr against the staple, the
// decision).  Every hit's link-independent half is computed next to the
// previous hit's link-dependent half, so each link carries two independent
// dependency chains instead of one.  The values are the reference's, bit for
// bit:
//   * taylor_fixed<K> adds K terms of the reference's recurrence (taylor_chain,
//     su3_exp.cuh), without its 1e-18 stop.  A term past the stop is below 1e-18 |h| / 2, less than
//     half an ulp of both sums (c >= 0.87; s >= 0.95 |h|), so adding it
//     changes no bit, and leaving the test out saves a comparison and a
//     select per term.  K is taken from the proposal half width a: |t_k| <=
//     |h|^k / k! with |h| <= a/2 for generators 1..7 and |h| <= 0.5774 a (at
//     most 0.5 after lambda8's halving) for generator 8, and terms past K
//     must be below half an ulp too: for a <= 0.4, K = 11 (t_12 <=
//     0.231^12/12! = 4.8e-17 < 2^-54 against sums in [0.97, 1), t_13 / s <=
//     0.231^12/13! = 3.7e-18); for a <= 1, K = 14 (t_15 / s <= 0.5^14/15!
//     = 4.7e-17 < 2^-54, t_16 <= 7.3e-19), so the sums are the reference's
//     bit for bit (checked on the CPU against the loop run to the cutoff
//     over millions of grid angles).
//   * the decision is the reference's u < exp(-max(dS, 0))
//     (su3_ensemble.rs:368) through accept_log; the accepted rows are
//     selected, not branched to.
constexpr double kShortRotation = 0.4;   // half widths that eleven terms serve

template <int K>
__device__ __forceinline__ void taylor_fixed(double h, double &c, double &s) {
    double t = h;      // k = 1: t = (1 h) 1, s = 0 + t
    c = 1.0;
    s = h;
#pragma unroll
    for (int k = 2; k <= K; ++k) {
        t = (t * h) * inv_int(k);
        if ((k & 3) == 1) s = s + t;
        else if ((k & 3) == 2) c = c - t;
        else if ((k & 3) == 3) s = s - t;
        else c = c + t;
    }
}

// lambda8_rotation with taylor_chain2's two chains evaluated for K terms;
// |theta| <= 1 needs at most one halving.
template <int K>
__device__ __forceinline__ void lambda8_fixed(double theta, cplx &e1, cplx &e2) {
    const double d1 = (0.5 * kInvSqrt3) * theta;
    const double d2 = (-kInvSqrt3) * theta;
    const bool sq = fmax(fabs(d1), fabs(d2)) > 0.5;
    const double sc = sq ? 0.5 : 1.0;
    taylor_fixed<K>(d1 * sc, e1.re, e1.im);
    taylor_fixed<K>(d2 * sc, e2.re, e2.im);
    const cplx q1 = cmul(e1, e1), q2 = cmul(e2, e2);
    e1 = sq ? q1 : e1;
    e2 = sq ? q2 : e2;
}

// Rotation entries of a hit: the reference's bits (taylor_fixed,
// lambda8_fixed), or in the fast form cos_sin_horner for both generators'
// phases (lambda8's two directly, without halving and squaring).
template <int K>
__device__ __forceinline__ void block_rotation(double h, double &c, double &s) {
#ifdef YM_TILED_FAST
    cos_sin_horner<K>(h, c, s);
#else
    taylor_fixed<K>(h, c, s);
#endif
}

template <int K>
__device__ __forceinline__ void diag_rotation(double theta, cplx &e1, cplx &e2) {
#ifdef YM_TILED_FAST
    double c1, s1, c2, s2;
    cos_sin_horner<K>((0.5 * kInvSqrt3) * theta, c1, s1);
    cos_sin_horner<K>((-kInvSqrt3) * theta, c2, s2);
    e1 = cmake(c1, s1);
    e2 = cmake(c2, s2);
#else
    lambda8_fixed<K>(theta, e1, e2);
#endif
}

struct BlockPre {
    double c, s;
    float logu;        // neg_log_unit of the accept word
};
struct DiagPre {
    cplx e1, e2;
    float logu;
};

template <int K>
__device__ __forceinline__ BlockPre pre_block(uint64_t &state, double angle) {
    BlockPre p;
    block_rotation<K>(0.5 * grid_angle(next_word(state), angle), p.c, p.s);
    p.logu = neg_log_unit(next_word(state));
    return p;
}

template <int K>
__device__ __forceinline__ DiagPre pre_diag(uint64_t &state, double angle) {
    DiagPre p;
    diag_rotation<K>(grid_angle(next_word(state), angle), p.e1, p.e2);
    p.logu = neg_log_unit(next_word(state));
    return p;
}

template <int K>
struct OrderedStream {
    uint64_t state;
    double angle;
    __device__ __forceinline__ BlockPre block() { return pre_block<K>(state, angle); }
    __device__ __forceinline__ DiagPre diag() { return pre_diag<K>(state, angle); }
};

// One row of a link and its Re Tr share.
struct Row {
    cplx e[3];
    double rr;
};

// Candidate entries of an SU(2)-subgroup hit on rows x, y: Mat3::mul's values,
// two rounded products and their sum per entry.
template <int KIND>
__device__ __forceinline__ void block_candidate(const Row &x, const Row &y, double c, double s, cplx n0[3],
                                                cplx n1[3]) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const double x0 = x.e[k].re, y0 = x.e[k].im;
        const double x1 = y.e[k].re, y1 = y.e[k].im;
        if (KIND == 0) {
            n0[k] = cmake(c * x0 - s * y1, c * y0 + s * x1);
            n1[k] = cmake(c * x1 - s * y0, s * x0 + c * y1);
        } else if (KIND == 1) {
            n0[k] = cmake(c * x0 + s * x1, c * y0 + s * y1);
            n1[k] = cmake(c * x1 - s * x0, c * y1 - s * y0);
        } else {
            n0[k] = cmake(c * x0 - s * y0, c * y0 + s * x0);
            n1[k] = cmake(c * x1 + s * y1, c * y1 - s * x1);
        }
    }
}

__device__ __forceinline__ void take_row(Row &r, bool acc, const cplx n[3], double q) {
#pragma unroll
    for (int k = 0; k < 3; ++k) r.e[k] = acc ? n[k] : r.e[k];
    r.rr = acc ? q : r.rr;
}

// An SU(2)-subgroup hit on rows x and y, whose A columns are ca and cb; z is
// the third row.  first: the subgroup is (0, 1), so the trace sums as
// (x + y) + z; else z lies between or before them: (x + z) + y.
template <int KIND, class A>
__device__ __forceinline__ void hit_rows(Row &x, Row &y, const Row &z, const A &a, int ca, int cb, bool first, double &old_tr, const BlockPre &p,
                                         double beta3, unsigned &accepted, uint64_t key, int h) {
    cplx n0[3], n1[3], col[3];
    block_candidate<KIND>(x, y, p.c, p.s, n0, n1);
    a.column(ca, col);
    const double q0 = retr_row_fma(n0, col);
    a.column(cb, col);
    const double q1 = retr_row_fma(n1, col);
    const double mid = first ? q1 : z.rr, end = first ? z.rr : q1;
    const double new_tr = (q0 + mid) + end;
    const bool acc = accept_log(beta3 * (old_tr - new_tr), p.logu, key, h);
    take_row(x, acc, n0, q0);
    take_row(y, acc, n1, q1);
    old_tr = acc ? new_tr : old_tr;
    accepted += acc ? 1u : 0u;
}

__device__ __forceinline__ void swap_rows(Row &x, Row &y) {
    const Row t = x;
    x = y;
    y = t;
}

// The eight ordered hits (generators 1..8, su3_ensemble.rs:361), the three
// SU(2) subgroups (rows (0,1), (0,2), (1,2)) one after the other, unrolled (as
// a loop, with the rows moved between its passes: 32^4 sweep 1373 against
// 1335 us, measured 1433 against 1365, 16^4 95 against 90).  Hit h+1's
// link-independent half is written next to hit h.
// tr receives Re Tr(U' A) of the final link, the sum of its six plaquettes.
// pre gives the hits' link-independent halves in order (OrderedStream, or a
// table made by other threads).
template <class A, class Pre>
__device__ __forceinline__ unsigned visit_ordered(m3 &u, const A &sa, double beta3, uint64_t key, Pre pre, double &tr) {
    Row r[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        cplx col[3];
        sa.column(i, col);
#pragma unroll
        for (int k = 0; k < 3; ++k) r[i].e[k] = u.e[i][k];
        r[i].rr = retr_row_fma(u.e[i], col);
    }
    double old_tr = (r[0].rr + r[1].rr) + r[2].rr;
    unsigned accepted = 0;
    Row x = r[0], y = r[1], z = r[2];
    BlockPre p = pre.block();
#pragma unroll
    for (int it = 0; it < 3; ++it) {
        const int ca = it == 2 ? 1 : 0, cb = it == 0 ? 1 : 2;
        const int h0 = it == 0 ? 0 : 2 * it + 1;   // the pass's first hit
        BlockPre q = pre.block();
        hit_rows<0>(x, y, z, sa, ca, cb, it == 0, old_tr, p, beta3, accepted, key, h0);
        if (it < 2) p = pre.block();
        hit_rows<1>(x, y, z, sa, ca, cb, it == 0, old_tr, q, beta3, accepted, key, h0 + 1);
        if (it == 0) {
            q = pre.block();
            hit_rows<2>(x, y, z, sa, ca, cb, true, old_tr, p, beta3, accepted, key, 2);
            p = q;
            swap_rows(y, z);
        } else if (it == 1) {
            swap_rows(x, z);
        }
    }
    // now x is row 1, y row 2, z row 0
    const DiagPre d = pre.diag();
    cplx n0[3], n1[3], n2[3], col[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        n0[k] = cmul(d.e1, z.e[k]);
        n1[k] = cmul(d.e1, x.e[k]);
        n2[k] = cmul(d.e2, y.e[k]);
    }
    sa.column(0, col);
    const double q0 = retr_row_fma(n0, col);
    sa.column(1, col);
    const double q1 = retr_row_fma(n1, col);
    sa.column(2, col);
    const double q2 = retr_row_fma(n2, col);
    const double new_tr = (q0 + q1) + q2;
    const bool acc = accept_log(beta3 * (old_tr - new_tr), d.logu, key, 7);
    old_tr = acc ? new_tr : old_tr;
    accepted += acc ? 1u : 0u;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        u.e[0][k] = acc ? n0[k] : z.e[k];
        u.e[1][k] = acc ? n1[k] : x.e[k];
        u.e[2][k] = acc ? n2[k] : y.e[k];
    }
    tr = old_tr;
    return accepted;
}

// ---- drawn generators ------------------------------------------------------
// Eight hits whose generator each link draws (bits 52..54 of the angle word).
// One formula serves all eight generators, so a warp whose links drew
// different ones stays converged: with rows r0, r1 of the generator's
// subgroup (lambda3 and lambda8: rows 0, 1) the candidate is
//   n0 = c r0 + s v0,  n1 = c r1 + s' v1,  v = w or i w,
//   lambda1, 4, 6: v0 = i r1, v1 = i r0;   lambda2, 5, 7: v0 = r1, v1 = r0, s' = -s;
//   lambda3: v0 = i r0, v1 = i r1, s' = -s;  lambda8: v0 = i r0, v1 = i r1,
// entry by entry the reference's two rounded products and their sum (a sign
// change is exact).  lambda8's second phase on row 2 is formed for every
// link: a warp has a lambda8 in 98 of 100 hits, and in a branch it would wait
// outside the other products.
// The link's rows and A's columns live in memory (u, a) and are addressed by
// the generator: picking them among registers took twice the instructions
// (10,600 per warp and visit, most of them selects and the two divergent
// sides, against 4,900).
struct DrawnPre {
    cplx e1;         // block rotation c + i s, or lambda8's phase of rows 0 and 1
    cplx e2;         // lambda8's phase of row 2
    float logu;
    int g;
};

template <int K>
__device__ __forceinline__ DrawnPre pre_drawn(uint64_t &state, double angle) {
    DrawnPre p;
    const uint64_t w = next_word(state);
    p.g = (int)((w >> 52) & 7);
    const double theta = grid_angle(w, angle);
    const double d1 = (0.5 * kInvSqrt3) * theta, d2 = (-kInvSqrt3) * theta;
    const bool diag = p.g == 7;
#ifdef YM_TILED_FAST
    const bool sq = false;
#else
    const bool sq = diag && fmax(fabs(d1), fabs(d2)) > 0.5;
#endif
    const double sc = sq ? 0.5 : 1.0;
    block_rotation<K>(diag ? d1 * sc : 0.5 * theta, p.e1.re, p.e1.im);
    block_rotation<K>(d2 * sc, p.e2.re, p.e2.im);
    const cplx q1 = cmul(p.e1, p.e1), q2 = cmul(p.e2, p.e2);
    p.e1 = sq ? q1 : p.e1;
    p.e2 = sq ? q2 : p.e2;
    p.logu = neg_log_unit(next_word(state));
    return p;
}

template <int K>
struct DrawnStream {
    uint64_t state;
    double angle;
    __device__ __forceinline__ DrawnPre next() { return pre_drawn<K>(state, angle); }
};

template <int K, class U, class A, class Pre>
__device__ __forceinline__ unsigned visit_drawn(const U &u, const A &a, double beta3, uint64_t key, Pre pre) {
    double rr[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        cplx row[3], col[3];
        u.row(i, row);
        a.column(i, col);
        rr[i] = retr_row_fma(row, col);
    }
    double old_tr = (rr[0] + rr[1]) + rr[2];
    unsigned accepted = 0;
    DrawnPre nx = pre.next();
#pragma unroll 1
    for (int h = 0; h < 8; ++h) {
        const DrawnPre p = nx;
        if (h < 7) nx = pre.next();
        const int g = p.g;
        const bool diag = g == 7;
        const bool low = g <= 2 || diag;                 // rows 0 and 1
        const int i0 = (g <= 4 || diag) ? 0 : 1, i1 = low ? 1 : 2, i2 = 3 - i0 - i1;
        const bool plain = g == 1 || g == 4 || g == 6;   // v = w, not i w
        const bool cross = !(g == 2 || diag);            // w is the other row
        cplx r0[3], r1[3], n0[3], n1[3], n2[3], col[3];
        u.row(i0, r0);
        u.row(i1, r1);
        const double c = p.e1.re, s = p.e1.im;
        cplx r2[3];
        u.row(2, r2);
        a.column(2, col);
#pragma unroll
        for (int k = 0; k < 3; ++k) n2[k] = cmul(p.e2, r2[k]);
        const double q2 = diag ? retr_row_fma(n2, col) : (i2 == 2 ? rr[2] : (i2 == 1 ? rr[1] : rr[0]));
        const double s1 = (plain || g == 2) ? -s : s;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const cplx w0 = cross ? r1[k] : r0[k], w1 = cross ? r0[k] : r1[k];
            const double v0r = plain ? w0.re : -w0.im, v0i = plain ? w0.im : w0.re;
            const double v1r = plain ? w1.re : -w1.im, v1i = plain ? w1.im : w1.re;
            n0[k] = cmake(c * r0[k].re + s * v0r, c * r0[k].im + s * v0i);
            n1[k] = cmake(c * r1[k].re + s1 * v1r, c * r1[k].im + s1 * v1i);
        }
        a.column(i0, col);
        const double q0 = retr_row_fma(n0, col);
        a.column(i1, col);
        const double q1 = retr_row_fma(n1, col);
        const double mid = low ? q1 : q2, end = low ? q2 : q1;
        const double new_tr = (q0 + mid) + end;
        if (accept_log(beta3 * (old_tr - new_tr), p.logu, key, h)) {
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                u.put(3 * i0 + k, n0[k]);
                u.put(3 * i1 + k, n1[k]);
            }
            if (diag) {
#pragma unroll
                for (int k = 0; k < 3; ++k) u.put(6 + k, n2[k]);
            }
            rr[0] = i0 == 0 ? q0 : rr[0];
            rr[1] = i0 == 1 ? q0 : (i1 == 1 ? q1 : rr[1]);
            rr[2] = i1 == 2 ? q1 : (diag ? q2 : rr[2]);
            old_tr = new_tr;
            accepted++;
        }
    }
    return accepted;
}

// ---- the sub-sweep: two staple terms in flight, two CTAs per SM ----------
// The sub-sweep keeps the staple accumulator in registers and a
// ring of two three-factor staging sets, so term k+2's factors are loading
// while term k multiplies.  Two
// 128-thread CTAs per SM fit (registers and 108 KB of staging each); after
// the staple the accumulator is written once to the second set's memory for
// the hits.  Terms run over the directions nu other than mu in ascending
// order, forward before backward, each product as fma chains (pair_product,
// add_third): the chain-resident kernel's order, so A has the same bits there.
//
// What bounds it: latency, at two warps per scheduler.  Two things cut it.
// (1) The CTAs are persistent, and the next item's first term loads into the
// first set while this item's hits run, so no item starts on an empty
// pipeline (chain table, then links: three dependent trips to L2).  (2) The
// code is small: directions are loops, not copies.  Unrolled
// (66 KB, four directions of it) the warps, which drift apart once they are
// persistent, waited for instructions as long as for data.  Per issued
// instruction on a 32^4 lattice, half width 0.3: unrolled and one tile per
// CTA 1.57 cycles on loads + 0.40 on instruction fetch (168 us per launch
// under the profiler), persistent unrolled 0.85-1.13 + 0.52-0.91 (169 us),
// persistent with looped directions 0.76 + 0.12 (161 us, hits looped too;
// with the ordered hits unrolled again 155).
// Three CTAs per SM (one term ahead, 168 registers with 150 bytes spilled):
// 1.52 + 0.62, 180 us.  Sweep live, start of this design -> now, same
// boxes: 32^4 1487 -> 1319 us at half width 0.3 (of which the shorter
// rotations and accept_log 6 %), 16^4 103 -> 90, 8^4 88 -> 73, 32 chains of
// 6^3 x 10 130 -> 120; drawn generators 2409 -> 1709 (32^4), 230 -> 132 (16^4).
struct TermSet {
    double2 (*f[3])[T];
};

// The three factors of staple term (nu, BWD) of link (x, mu):
//   forward  U_nu(x+mu), U_mu(x+nu), U_nu(x)
//   backward U_nu(x-nu+mu), U_mu(x-nu), U_nu(x-nu)
// mu and nu are run-time values (uniform over the launch), so one copy of
// the code serves every direction.
template <bool BWD>
__device__ __forceinline__ void stage_term3(const TermSet &b, const double2 *base, int64_t v, const Site &x, int par,
                                            int mu, int nu) {
    const int32_t same = par ? x.half : 0, other = par ? 0 : x.half;
    const int32_t up = pick(x.fwd, mu);
    int32_t i1, i2, i3;
    if (!BWD) {
        i1 = other + ((x.lex + up) >> 1);
        i2 = other + ((x.lex + pick(x.fwd, nu)) >> 1);
        i3 = same + (x.lex >> 1);
    } else {
        const int32_t o = x.lex + pick(x.bwd, nu);
        i1 = same + ((o + up) >> 1);
        i2 = i3 = other + (o >> 1);
    }
    const double2 *pn = base + (int64_t)(nu * 9) * v, *pm = base + (int64_t)(mu * 9) * v;
    const double2 *p1 = pn + i1, *p2 = pm + i2, *p3 = pn + i3;
#pragma unroll
    for (int e = 0; e < 9; ++e) {
        cp_async16(&b.f[0][e][threadIdx.x], p1 + (int64_t)e * v);
        cp_async16(&b.f[1][e][threadIdx.x], p2 + (int64_t)e * v);
        cp_async16(&b.f[2][e][threadIdx.x], p3 + (int64_t)e * v);
    }
    cp_async_commit();
}

// A staple term's two products: P = U V^dag (forward) or U^dag V^dag
// (backward) as fma chains from zero, then A += P W^dag or P W.
template <bool BWD>
__device__ __forceinline__ m3 pair_product(const m3 &l1, const m3 &l2) {
    m3 p;
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            cplx v = cmake(0.0, 0.0);
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                if (!BWD) cfma(v, l1.e[r][j], cconj(l2.e[k][j]));
                else cfma(v, cconj(l1.e[j][r]), cconj(l2.e[k][j]));
            }
            p.e[r][k] = v;
        }
    return p;
}

template <bool BWD>
__device__ __forceinline__ void add_third(const m3 &p, const m3 &l3, m3 &a) {
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int col = 0; col < 3; ++col)
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                if (!BWD) cfma(a.e[r][col], p.e[r][k], cconj(l3.e[col][k]));
                else cfma(a.e[r][col], p.e[r][k], l3.e[k][col]);
            }
}

template <bool BWD>
__device__ __forceinline__ void term_accumulate(const TermSet &b, m3 &a) {
    m3 p;
    {
        const m3 l1 = staged_link(b.f[0]), l2 = staged_link(b.f[1]);
        p = pair_product<BWD>(l1, l2);
    }
    add_third<BWD>(p, staged_link(b.f[2]), a);
}

// The staple of link (x, mu); term 0 has been staged into s0.  SAVE (mu = 1
// or 2): `part` receives the accumulator after the directions below mu.
template <bool SAVE>
__device__ __forceinline__ m3 staple_ring(const double2 *base, int64_t v, const Site &x, int par, int mu,
                                          const TermSet &s0, const TermSet &s1, m3 &part) {
    m3 a;
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int k = 0; k < 3; ++k) a.e[r][k] = cmake(0.0, 0.0);
#pragma unroll 1
    for (int i = 0; i < 3; ++i) {
        const int nu = i + (i >= mu ? 1 : 0), nn = i + 1 + (i + 1 >= mu ? 1 : 0);
        stage_term3<true>(s1, base, v, x, par, mu, nu);
        cp_async_wait_one();
        term_accumulate<false>(s0, a);
        if (i < 2) {
            stage_term3<false>(s0, base, v, x, par, mu, nn);
        } else {   // the updated link itself
            const double2 *p = base + (int64_t)(mu * 9) * v + (par ? x.half : 0) + (x.lex >> 1);
#pragma unroll
            for (int e = 0; e < 9; ++e) cp_async16(&s0.f[0][e][threadIdx.x], p + (int64_t)e * v);
            cp_async_commit();
        }
        cp_async_wait_one();
        term_accumulate<true>(s1, a);
        if (SAVE && i + 1 == mu) part = a;
    }
    return a;
}

constexpr int kRingBuffers = 6;   // two sets of three factors

// MEASURE (parity 1, MU = 1, 2 or 3: the last three sub-sweeps of a sweep,
// one chain per CTA): each warp also writes its slot of tr_partial (work
// item b, warp w: b * kSweepWarps + w), the sum over its links of (1/3) Re Tr(U' A_p) with A_p the staple terms of the directions
// nu < MU (MU = 1: nu = 0; MU = 2: nu = 0, 1; MU = 3: all of A).  Once this
// sub-sweep has run, every link of those terms is final (directions below
// MU are done, direction MU's even links were done in parity 0, its odd
// links here), and each plaquette of plane (nu, MU) holds exactly one
// odd-site MU-link, so the three launches' sums are the plaquettes of
// planes (0,1); (0,2), (1,2); (0,3), (1,3), (2,3): all six planes.
template <int K, bool MEASURE, bool DRAWN>
__global__ void __launch_bounds__(T, 2)
k_su3_metropolis_ring(const ChainInfo *__restrict__ chains, const Tile *__restrict__ tiles, int n_ctas,
                      const __grid_constant__ ChainInfo one, double2 *__restrict__ links, int parity, int mu, double angle,
                      const uint64_t *__restrict__ sweep_ptr, unsigned long long *__restrict__ accepts,
                      int log2_item, int reverse, double *__restrict__ tr_partial = nullptr) {
    extern __shared__ __align__(16) double2 ring_mem[];
    auto buf = [&](int i) { return reinterpret_cast<double2 (*)[T]>(ring_mem + (size_t)i * 9 * T); };
    const TermSet s0{{buf(0), buf(1), buf(2)}}, s1{{buf(3), buf(4), buf(5)}};
    const int64_t lane = threadIdx.x & ((1u << log2_item) - 1u);
    const uint64_t sweep = *sweep_ptr;
    int32_t chain;        // of the item in hand
    bool live;
    Site x;
    const double2 *base;  // the chain's links
    int64_t volume;
    double beta;
    uint64_t seed;
    auto take_item = [&](int b) {
        // padding items (chain < 0) read the first chain's geometry and stay idle
        const int64_t item = (int64_t)(reverse ? n_ctas - 1 - b : b) * (T >> log2_item) + (threadIdx.x >> log2_item);
        const ItemChain it = block_of(chains, tiles, one, item, 1 << log2_item);
        const ChainInfo &c = it.c;
        chain = it.chain;
        live = it.chain >= 0 && it.start + lane < c.half;
        x = site_of(c, decode_storage(c, (int64_t)parity * c.half + (live ? it.start + lane : 0)));
        base = links + c.offset;
        volume = c.volume;
        beta = c.beta;
        seed = c.seed;
        if (live) stage_term3<false>(s0, base, volume, x, parity, mu, mu == 0 ? 1 : 0);
    };
    take_item(blockIdx.x);
    for (int b = blockIdx.x; b < n_ctas; b += gridDim.x) {
        unsigned accepted = 0;
        double tr = 0.0;
        const int32_t this_chain = chain;
        const bool this_live = live;
        m3 u, part;
        const Col<T> sa = column_of(s1.f[0]);
        double beta3 = 0.0;
        uint64_t key = 0;
        double2 *dst = links;
        const int64_t this_volume = volume;
        if (live) {
            const m3 a = staple_ring<MEASURE>(base, volume, x, parity, mu, s0, s1, part);
            cp_async_wait_all();
            u = staged_link(s0.f[0]);
            // the accumulator, for the hits, in the second set's (now free) memory
#pragma unroll
            for (int e = 0; e < 9; ++e) sa.put(e, a.e[e / 3][e % 3]);
            key = link_key(seed, sweep, x.lex, mu);
            beta3 = beta / 3.0;
            dst = const_cast<double2 *>(base) + (int64_t)(mu * 9) * volume + (parity ? x.half : 0) + (x.lex >> 1);
        }
        // the next item's first staple term loads while this link's hits run
        if (b + (int)gridDim.x < n_ctas) take_item(b + gridDim.x);
        if (this_live) {
            if (DRAWN) {   // the rows in memory, next to the accumulator
                const Col<T> rows = column_of(s1.f[1]);
#pragma unroll
                for (int e = 0; e < 9; ++e) rows.put(e, u.e[e / 3][e % 3]);
                accepted = visit_drawn<K>(rows, sa, beta3, key, DrawnStream<K>{key, angle});
                u = staged_link(s1.f[1]);
            } else {
                accepted = visit_ordered(u, sa, beta3, key, OrderedStream<K>{key, angle}, tr);
            }
#pragma unroll
            for (int e = 0; e < 9; ++e)
                dst[(int64_t)e * this_volume] = make_double2(u.e[e / 3][e % 3].re, u.e[e / 3][e % 3].im);
            if (MEASURE && mu < 3) {   // Re Tr(U' A_p)
                double q = 0.0;
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    const cplx col[3] = {part.e[0][i], part.e[1][i], part.e[2][i]};
                    q = q + retr_row_fma(u.e[i], col);
                }
                tr = q;
            }
        }
        const unsigned warp_sum = __reduce_add_sync(0xffffffffu, accepted);
        if ((threadIdx.x & 31) == 0 && warp_sum) atomicAdd(accepts + this_chain, (unsigned long long)warp_sum);
        if (MEASURE) {
            double v = this_live ? tr / 3.0 : 0.0;
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
            if ((threadIdx.x & 31) == 0)
                tr_partial[(int64_t)(reverse ? n_ctas - 1 - b : b) * kSweepWarps + (threadIdx.x >> 5)] = v;
        }
    }
}


constexpr size_t kRingBytes = (size_t)kRingBuffers * 9 * T * sizeof(double2);

// Two resident CTAs per SM walk all work items.
unsigned ring_grid(int64_t ctas) {
    static thread_local int sms = 0, dev_seen = -1;
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev != dev_seen) {
        sms = 148;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        dev_seen = dev;
    }
    return (unsigned)(ctas < 2 * sms ? ctas : 2 * sms);
}

// Both launchers take the handle's sweep layout: work items of 2^log2
// sites, chain order or by descending chain volume (all layouts give the
// same bits).
template <int K, bool DRAWN>
void metro_launch_ring(ym_ensemble *e, int parity, int mu, double angle, int reverse) {
    const SweepLayout &L = e->layouts[e->sweep_layout];
    const dim3 grid(ring_grid(L.ctas)), block(T);
    k_su3_metropolis_ring<K, false, DRAWN><<<grid, block, kRingBytes, e->stream>>>(
        e->d_chains, L.d_items, (int)L.ctas, single_chain(e), e->d_links, parity, mu, angle, sweep_index(e), e->d_accepts, L.log2_item,
        reverse, nullptr);
}

// One of a sweep's last three sub-sweeps (parity 1, mu = 1, 2 or 3, ordered
// hits) with its plaquette shares (MEASURE): the handle's layout must put one
// chain in each CTA (128-site items).
template <int K>
void metro_launch_measure(ym_ensemble *e, int mu, double angle, double *tr_partial) {
    const SweepLayout &L = e->layouts[e->sweep_layout];
    const dim3 g(ring_grid(L.ctas)), b(T);
    const int rev = (1 * 4 + mu) & 1;   // the tile order tiled_launch gives (parity 1, mu)
    k_su3_metropolis_ring<K, true, false><<<g, b, kRingBytes, e->stream>>>(
        e->d_chains, L.d_items, (int)L.ctas, single_chain(e), e->d_links, 1, mu, angle, sweep_index(e), e->d_accepts, L.log2_item, rev,
        tr_partial);
}

cudaError_t set_smem(const void *f, size_t bytes) {
    cudaError_t err = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (err == cudaSuccess)
        err = cudaFuncSetAttribute(f, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    return err;
}

// Shared-memory limits of the sub-sweep kernels, set once per device.
cudaError_t configure_kernels() {
    static thread_local int configured_device = -1;
    int dev = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess) return err;
    if (configured_device != dev) {
        const void *ring[6] = {(const void *)k_su3_metropolis_ring<11, false, false>,
                               (const void *)k_su3_metropolis_ring<14, false, false>,
                               (const void *)k_su3_metropolis_ring<11, true, false>,
                               (const void *)k_su3_metropolis_ring<14, true, false>,
                               (const void *)k_su3_metropolis_ring<11, false, true>,
                               (const void *)k_su3_metropolis_ring<14, false, true>};
        for (const void *f : ring)
            if ((err = set_smem(f, kRingBytes)) != cudaSuccess) return err;
        configured_device = dev;
    }
    return cudaSuccess;
}

// One sub-sweep of the handle with the term count the half width allows
// (angles are validated to lie in [1e-8, 1] for binary64 handles).
cudaError_t tiled_launch(ym_ensemble *e, int parity, int mu, double angle, int uniform) {
    if (cudaError_t err = configure_kernels()) return err;
    // Consecutive sub-sweeps walk the lattice in opposite directions (odd
    // ones from the last CTA down), so each starts on the links the previous
    // one touched last and finds its first waves' staple links in L2.  The
    // links of one sub-sweep are independent, so the order changes no bit.
    const int reverse = (parity * 4 + mu) & 1;
    if (uniform && angle <= kShortRotation) metro_launch_ring<11, true>(e, parity, mu, angle, reverse);
    else if (uniform) metro_launch_ring<14, true>(e, parity, mu, angle, reverse);
    else if (angle <= kShortRotation) metro_launch_ring<11, false>(e, parity, mu, angle, reverse);
    else metro_launch_ring<14, false>(e, parity, mu, angle, reverse);
    return cudaGetLastError();
}

// tiled_launch(e, 1, mu, angle, ordered hits), mu = 1, 2 or 3, that also
// writes each warp's plaquette share of the planes (nu, mu), nu < mu, to
// tr_partial[cta * kSweepWarps + warp] (the handle's layout must hold one
// chain per CTA).
cudaError_t tiled_launch_measure(ym_ensemble *e, int mu, double angle, double *tr_partial) {
    if (cudaError_t err = configure_kernels()) return err;
    if (angle <= kShortRotation) metro_launch_measure<11>(e, mu, angle, tr_partial);
    else metro_launch_measure<14>(e, mu, angle, tr_partial);
    return cudaGetLastError();
}

}  // namespace
}  // namespace YM_TILED_NS
}  // namespace ym
