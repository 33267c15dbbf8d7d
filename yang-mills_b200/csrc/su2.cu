// su2.cu -- SU(2) kernels (compiled with -fmad=false): checkerboard
// heat-bath and overrelaxation sub-sweeps, plaquette, unit residual, layout.
//
// Links are unit quaternions (a0, a1, a2, a3), U = a0 I - i a.sigma
// (reference/rust/src/lib.rs:7-13), stored as two double2 planes per
// direction: (a0, a1) and (a2, a3).  Every quaternion product is
// re-normalised exactly as Su2::mul does (lib.rs:106-130, 212-224): divide by
// the largest magnitude, then by the Euclidean norm.
//
// Heat-bath: the reference's sampler (su2_ensemble.rs:220-281) -- r0 from
// the truncated exponential by inverse CDF (exp_m1, ln_1p), the Haar factor
// sqrt(1 - r0^2) by rejection, a uniform direction on S^2, U = R Vhat^dag --
// or, as an alternative, the Kennedy-Pendleton sampler for the same density.
// The attempt loop is bounded; a link that exhausts it keeps its value and
// raises the ensemble's error flag (HeatbathAttemptLimitExceeded).
// Overrelaxation: U <- Vhat^dag U^dag Vhat^dag (su2_ensemble.rs:283-299).
#include <cuda_runtime.h>

#include "su2_quat.cuh"
#include "ym_internal.hpp"

namespace ym {

namespace {

constexpr int T = kSweepThreads;
constexpr double kAlphaZeroLimit = 1.0e-300;   // su2_ensemble.rs:22
constexpr double kTau = 6.283185307179586;     // core::f64::consts::TAU

// Lattice4::staple (lib.rs:507-546): the unnormalised sum of six products,
// nu ascending, forward then backward, components added in order (one
// thread per link).
template <int MU>
__device__ __forceinline__ void su2_staple(const double2 *__restrict__ links, const ChainInfo &c,
                                           const Coord &x, int par, double comp[4]) {
    comp[0] = comp[1] = comp[2] = comp[3] = 0.0;
    const Nb self{x.lex, par};
    const Nb pm = step(c, x.x, x.lex, par, MU, +1);
    // one direction's forward and backward term at a time, side by side
#pragma unroll 1
    for (int i = 0; i < 3; ++i) {
        const int nu = i + (i >= MU ? 1 : 0);
        const Nb pn = step_any(c, x.x, x.lex, par, nu, +1);
        const Nb mn = step_any(c, x.x, x.lex, par, nu, -1);
        const Nb mnpm = step(c, x.x, mn.lex, mn.par, MU, +1);
        const q4 first[2] = {link_q(links, c, pm, nu), qdag(link_q(links, c, mnpm, nu))};
        const q4 second[2] = {qdag(link_q(links, c, pn, MU)), qdag(link_q(links, c, mn, MU))};
        const q4 third[2] = {qdag(link_q(links, c, self, nu)), link_q(links, c, mn, nu)};
        q4 p[2], t[2];
        qmul_many<2>(first, second, p);
        qmul_many<2>(p, third, t);
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int k = 0; k < 4; ++k) comp[k] += t[m].c[k];
    }
}

// The same staple for a link updated by a group of kGroup lanes: lane j < 6
// computes term j (the (j/2)-th direction nu != MU, forward for even j,
// backward for odd j) and every lane of the group then adds the six terms in
// that order, so the sum has the one-thread staple's bits while its twelve
// normalised products run on six lanes at once.
constexpr int kGroup = 8;
constexpr int kGroupLinks = T / kGroup;   // links per 128-thread block

__device__ __forceinline__ q4 qdag_if(const q4 &a, bool d) {
    const double s = d ? -1.0 : 1.0;   // exact sign flip
    return q4{{a.c[0], s * a.c[1], s * a.c[2], s * a.c[3]}};
}

// The three links of term j of the staple of link (x, mu):
//   forward  U_nu(x+mu) U_mu(x+nu)^dag U_nu(x)^dag
//   backward U_nu(x-nu+mu)^dag U_mu(x-nu)^dag U_nu(x-nu)
// mu is a run-time value, so one copy of the code serves a sweep's launches.
struct TermLinks {
    q4 a, b, c;
    bool fwd;
};

__device__ __forceinline__ TermLinks su2_term_links(const double2 *__restrict__ links, const ChainInfo &c,
                                                    const Site &x, int par, int mu, int j) {
    const int k = j >> 1;
    const int nu = k < mu ? k : k + 1;
    const int32_t same = par ? x.half : 0, other = par ? 0 : x.half;
    const int32_t up = pick(x.fwd, mu);
    TermLinks t;
    t.fwd = (j & 1) == 0;
    const int32_t beside = x.lex + (t.fwd ? pick(x.fwd, nu) : pick(x.bwd, nu));   // x + nu or x - nu
    t.a = load_q(links, c, t.fwd ? other + ((x.lex + up) >> 1) : same + ((beside + up) >> 1), nu);
    t.b = load_q(links, c, other + (beside >> 1), mu);
    t.c = load_q(links, c, t.fwd ? same + (x.lex >> 1) : other + (beside >> 1), nu);
    return t;
}

// The group's staple sum (every lane of the group gets it): terms computed
// by lanes 0..5 of the group from the links they hold (`active` false: the
// sum is meaningless), added in term order.
__device__ __forceinline__ void su2_staple_group(const TermLinks &l, bool active, double comp[4]) {
    const int lane = threadIdx.x & 31, j = lane & (kGroup - 1), base = lane - j;
    q4 term{{0.0, 0.0, 0.0, 0.0}};
    if (active && j < 6) term = qmul(qmul(qdag_if(l.a, !l.fwd), qdag(l.b)), qdag_if(l.c, l.fwd));
    comp[0] = comp[1] = comp[2] = comp[3] = 0.0;
#pragma unroll
    for (int jj = 0; jj < 6; ++jj)
#pragma unroll
        for (int i = 0; i < 4; ++i) comp[i] += __shfl_sync(0xffffffffu, term.c[i], base + jj);
}

// staple_norm (su2_ensemble.rs:194-202): sum of squares from -0.0, sqrt.
__device__ __forceinline__ double staple_norm(const double comp[4]) {
    double ss = comp[0] * comp[0];
    ss = ss + comp[1] * comp[1];
    ss = ss + comp[2] * comp[2];
    ss = ss + comp[3] * comp[3];
    return sqrt(ss);
}

// The reference sampler (su2_ensemble.rs:220-254) on the link's stream:
// words 2k, 2k+1 for attempt k+1, then two for the S^2 direction.  The
// direction is drawn after the attempt loop, where the warp has met again:
// inside it, each attempt that some lane accepts would run it once more for
// the whole warp (a warp needs four or five attempts).
__device__ __forceinline__ bool sample_reference(double alpha, uint64_t key, int max_attempts,
                                                 q4 &out, int &attempts) {
    uint64_t j = 0;
    const double mass = alpha <= kAlphaZeroLimit ? 0.0 : -expm1(-2.0 * alpha);
    double r0 = 0.0, radial = 0.0;
    bool found = false;
    int a = 1;
    for (; a <= max_attempts; ++a) {
        const double pu = unit_from(splitmix_at(key, j++));
        if (alpha <= kAlphaZeroLimit) {
            r0 = 2.0 * pu - 1.0;
        } else {
            const double y = -log1p(-pu * mass) / alpha;
            r0 = 1.0 - y;
            r0 = r0 < -1.0 ? -1.0 : (r0 > 1.0 ? 1.0 : r0);
        }
        radial = sqrt(fmax(1.0 - r0 * r0, 0.0));
        if (unit_from(splitmix_at(key, j++)) <= radial) {
            found = true;
            break;
        }
    }
    attempts = found ? a : max_attempts;
    if (!found) return false;
    const double z = 2.0 * unit_from(splitmix_at(key, j)) - 1.0;
    const double phi = kTau * unit_from(splitmix_at(key, j + 1));
    const double planar = sqrt(fmax(1.0 - z * z, 0.0));
    const double v[4] = {r0, radial * (planar * cos(phi)), radial * (planar * sin(phi)), radial * z};
    if (!normalize_scaled<4>(v, out.c)) {
        attempts = 0;
        return false;
    }
    return true;
}

// Kennedy-Pendleton (Phys. Lett. B 156 (1985) 393) for the same density
// exp(alpha r0) sqrt(1 - r0^2): x = -(ln u1 + cos^2(2 pi u2) ln u3)/alpha,
// accept if u4^2 <= 1 - x/2, r0 = 1 - x.  Uniforms in (0, 1].  The direction
// after the loop, as above.
//
// An attempt's draws do not know alpha: `first` is the first attempt's, which
// a caller can make while it waits for the staple's links.
struct KpDraw {
    double num, u4;   // x = num / alpha
};

__device__ __forceinline__ KpDraw kp_draw(uint64_t key, uint64_t j) {
    const double u1 = 1.0 - unit_from(splitmix_at(key, j));
    const double u2 = unit_from(splitmix_at(key, j + 1));
    const double u3 = 1.0 - unit_from(splitmix_at(key, j + 2));
    const double u4 = unit_from(splitmix_at(key, j + 3));
    const double cs = cospi(2.0 * u2);
    return KpDraw{-(log(u1) + cs * cs * log(u3)), u4};
}

__device__ __forceinline__ bool sample_kp(double alpha, uint64_t key, const KpDraw &first, int max_attempts, q4 &out,
                                          int &attempts) {
    if (alpha <= kAlphaZeroLimit) return sample_reference(alpha, key, max_attempts, out, attempts);
    double x = 0.0;
    bool found = false;
    int a = 1;
    KpDraw d = first;
    for (;;) {
        x = d.num / alpha;
        if (d.u4 * d.u4 <= 1.0 - 0.5 * x) {
            found = true;
            break;
        }
        if (++a > max_attempts) break;
        d = kp_draw(key, 4 * (uint64_t)(a - 1));
    }
    const uint64_t j = 4 * (uint64_t)a;
    attempts = found ? a : max_attempts;
    if (!found) return false;
    const double r0 = 1.0 - x;
    const double radial = sqrt(fmax(1.0 - r0 * r0, 0.0));
    const double z = 2.0 * unit_from(splitmix_at(key, j)) - 1.0;
    double sn, cn;
    sincospi(2.0 * unit_from(splitmix_at(key, j + 1)), &sn, &cn);
    const double planar = sqrt(fmax(1.0 - z * z, 0.0));
    const double v[4] = {r0, radial * (planar * cn), radial * (planar * sn), radial * z};
    if (!normalize_scaled<4>(v, out.c)) {
        attempts = 0;
        return false;
    }
    return true;
}

// Error flag bits.
constexpr unsigned kErrAttempts = 1u;
constexpr unsigned kErrNonFinite = 2u;

// One thread per link (large sub-sweeps).  What bounds it: binary64 latency
// and issue of the normalised products.  24^4, per launch under the profiler:
// overrelaxation 48 us with plain divisions and one product at a time, 34 us
// with shared reciprocals and a direction's two terms side by side (binary64
// pipe 36 -> 47 %); heat-bath 75 us to 66, and with the direction drawn after
// the attempt loop a sweep of one heat-bath and one overrelaxation went from
// 758 to 721 us live (918 at first).
template <int MU>
__global__ void __launch_bounds__(T)
k_su2_heatbath_thread(const ChainInfo *__restrict__ chains, const Tile *__restrict__ tiles,
               const __grid_constant__ ChainInfo one, double2 *__restrict__ links, int parity, int max_attempts, int kp,
               const uint64_t *__restrict__ sweep_ptr, unsigned long long *__restrict__ proposals,
               unsigned *__restrict__ err) {
    const ItemChain block = block_of(chains, tiles, one, blockIdx.x, T);
    const ChainInfo &c = block.c;
    const int64_t t = block.start + threadIdx.x;
    unsigned attempts_used = 0;
    if (t < c.half) {
        const int64_t s = (int64_t)parity * c.half + t;
        const Coord x = decode_storage(c, s);
        double comp[4];
        su2_staple<MU>(links, c, x, parity, comp);
        const double norm = staple_norm(comp);
        const double alpha = c.beta * norm;
        if (!isfinite(norm) || !isfinite(alpha)) {
            atomicOr(err, kErrNonFinite);
        } else {
            const uint64_t key = link_key(c.seed, *sweep_ptr, x.lex, MU);
            q4 r;
            int att = 0;
            const bool ok = kp ? sample_kp(alpha, key, kp_draw(key, 0), max_attempts, r, att)
                               : sample_reference(alpha, key, max_attempts, r, att);
            attempts_used = (unsigned)att;
            if (!ok) {
                atomicOr(err, kErrAttempts);
            } else {
                q4 next = r;
                if (norm != 0.0) {
                    q4 vhat;
                    normalize_scaled<4>(comp, vhat.c);
                    next = qmul(r, qdag(vhat));
                }
                store_q(links, c, s, MU, next);
            }
        }
    }
    const unsigned warp_sum = __reduce_add_sync(0xffffffffu, attempts_used);
    if ((threadIdx.x & 31) == 0 && warp_sum)
        atomicAdd(proposals + block.chain, (unsigned long long)warp_sum);
}

template <int MU>
__global__ void __launch_bounds__(T)
k_su2_overrelax_thread(const ChainInfo *__restrict__ chains, const Tile *__restrict__ tiles,
                const __grid_constant__ ChainInfo one, double2 *__restrict__ links, int parity, unsigned *__restrict__ err) {
    const ItemChain block = block_of(chains, tiles, one, blockIdx.x, T);
    const ChainInfo &c = block.c;
    const int64_t t = block.start + threadIdx.x;
    if (t >= c.half) return;
    const int64_t s = (int64_t)parity * c.half + t;
    const Coord x = decode_storage(c, s);
    const q4 u = load_q_rw(links, c, s, MU);
    double comp[4];
    su2_staple<MU>(links, c, x, parity, comp);
    const double norm = staple_norm(comp);
    if (!isfinite(norm)) {
        atomicOr(err, kErrNonFinite);
        return;
    }
    if (norm == 0.0) return;
    q4 vhat;
    normalize_scaled<4>(comp, vhat.c);
    const q4 nd = qdag(vhat);
    store_q(links, c, s, MU, qmul(qmul(nd, qdag(u)), nd));
}

// Grouped form (small sub-sweeps, latency-bound: a 10^4 lattice updates
// 5,000 links per launch, about one warp per SM with one thread per link).
// One block: kGroupLinks links of the tile blockIdx.x / kGroup (sub-block
// blockIdx.x % kGroup), kGroup lanes per link; the update is evaluated by
// every lane of the group alike and written by its first lane.
// What bounds it: the launch and one update's dependency chain (5 to 7 us a
// launch).  The link's words, the first Kennedy-Pendleton attempt's
// logarithms and the overrelaxed link are therefore had while the staple's
// links load, and one copy of the code serves all directions: a measured
// sweep of one heat-bath and three overrelaxations 8^4 158 -> 151 us, 10^4
// 197 -> 195.
__global__ void __launch_bounds__(T)
k_su2_heatbath_group(const ChainInfo *__restrict__ chains, const Tile *__restrict__ tiles,
               const __grid_constant__ ChainInfo one, double2 *__restrict__ links, int parity, int mu, int max_attempts, int kp,
               const uint64_t *__restrict__ sweep_ptr, unsigned long long *__restrict__ proposals,
               unsigned *__restrict__ err) {
    const ItemChain block = block_of(chains, tiles, one, blockIdx.x / kGroup, T);
    const ChainInfo &c = block.c;
    const int64_t t = block.start + (int64_t)(blockIdx.x % kGroup) * kGroupLinks + threadIdx.x / kGroup;
    const bool leader = (threadIdx.x & (kGroup - 1)) == 0;
    const bool active = t < c.half;
    const int64_t s = (int64_t)parity * c.half + (active ? t : 0);
    const Coord x = decode_storage(c, s);
    const uint64_t sweep = *sweep_ptr;
    TermLinks l;
    if (active && (threadIdx.x & (kGroup - 1)) < 6)
        l = su2_term_links(links, c, site_of(c, x), parity, mu, threadIdx.x & (kGroup - 1));
    // made while the links load
    const uint64_t key = link_key(c.seed, sweep, x.lex, mu);
    KpDraw first{0.0, 0.0};
    if (kp) first = kp_draw(key, 0);
    double comp[4];
    su2_staple_group(l, active, comp);
    unsigned attempts_used = 0;
    if (active) {
        const double norm = staple_norm(comp);
        const double alpha = c.beta * norm;
        if (!isfinite(norm) || !isfinite(alpha)) {
            if (leader) atomicOr(err, kErrNonFinite);
        } else {
            q4 r;
            int att = 0;
            const bool ok = kp ? sample_kp(alpha, key, first, max_attempts, r, att)
                               : sample_reference(alpha, key, max_attempts, r, att);
            attempts_used = leader ? (unsigned)att : 0u;
            if (!ok) {
                if (leader) atomicOr(err, kErrAttempts);
            } else {
                q4 next = r;
                if (norm != 0.0) {
                    q4 vhat;
                    normalize_scaled<4>(comp, vhat.c);
                    next = qmul(r, qdag(vhat));
                }
                if (leader) store_q(links, c, s, mu, next);
            }
        }
    }
    const unsigned warp_sum = __reduce_add_sync(0xffffffffu, attempts_used);
    if ((threadIdx.x & 31) == 0 && warp_sum)
        atomicAdd(proposals + block.chain, (unsigned long long)warp_sum);
}

__global__ void __launch_bounds__(T)
k_su2_overrelax_group(const ChainInfo *__restrict__ chains, const Tile *__restrict__ tiles,
                const __grid_constant__ ChainInfo one, double2 *__restrict__ links, int parity, int mu, unsigned *__restrict__ err) {
    const ItemChain block = block_of(chains, tiles, one, blockIdx.x / kGroup, T);
    const ChainInfo &c = block.c;
    const int64_t t = block.start + (int64_t)(blockIdx.x % kGroup) * kGroupLinks + threadIdx.x / kGroup;
    const bool leader = (threadIdx.x & (kGroup - 1)) == 0;
    const bool active = t < c.half;
    const int64_t s = (int64_t)parity * c.half + (active ? t : 0);
    const Coord x = decode_storage(c, s);
    TermLinks l;
    if (active && (threadIdx.x & (kGroup - 1)) < 6)
        l = su2_term_links(links, c, site_of(c, x), parity, mu, threadIdx.x & (kGroup - 1));
    // (an idle group has no link of its own: its slot is another group's,
    // which may be storing to it)
    q4 u{{0.0, 0.0, 0.0, 0.0}};
    if (active) u = load_q_rw(links, c, s, mu);
    double comp[4];
    su2_staple_group(l, active, comp);
    if (!active) return;
    const double norm = staple_norm(comp);
    if (!isfinite(norm)) {
        if (leader) atomicOr(err, kErrNonFinite);
        return;
    }
    if (norm == 0.0) return;
    q4 vhat;
    normalize_scaled<4>(comp, vhat.c);
    const q4 nd = qdag(vhat);
    const q4 next = qmul(qmul(nd, qdag(u)), nd);
    if (leader) store_q(links, c, s, mu, next);
}

// Plaquette half real trace per site, (mu, nu) order as the reference.
__global__ void __launch_bounds__(kSiteThreads)
k_su2_plaquette(const ChainInfo *__restrict__ chains, const Tile *__restrict__ tiles,
                const double2 *__restrict__ links, double *__restrict__ partial) {
    __shared__ double warp_vals[32];
    const Tile tile = tiles[blockIdx.x];
    const ChainInfo c = chains[tile.chain];
    const int64_t s = tile.start + threadIdx.x;
    double v = 0.0;
    if (s < c.volume) {
        const Coord x = decode_storage(c, s);
        const Nb self{x.lex, x.par};
        // planes (0,1),(0,2) then (0,3),(1,2) then (1,3),(2,3), side by side
#pragma unroll 1
        for (int k = 0; k < 3; ++k) {
            const int mu[2] = {k < 2 ? 0 : 1, k == 0 ? 0 : k}, nu[2] = {k == 0 ? 1 : 3, k < 2 ? 2 : 3};
            q4 a[2], b[2], d[2], e[2];
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                const Nb pm = step_any(c, x.x, x.lex, x.par, mu[m], +1);
                const Nb pn = step_any(c, x.x, x.lex, x.par, nu[m], +1);
                a[m] = link_q(links, c, self, mu[m]);
                b[m] = link_q(links, c, pm, nu[m]);
                d[m] = qdag(link_q(links, c, pn, mu[m]));
                e[m] = qdag(link_q(links, c, self, nu[m]));
            }
            qmul_many<2>(a, b, a);
            qmul_many<2>(a, d, a);
            qmul_many<2>(a, e, a);
            v = k == 0 ? a[0].c[0] : v + a[0].c[0];
            v = v + a[1].c[0];
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
    if ((threadIdx.x & 31) == 0) warp_vals[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x < 32) {
        v = threadIdx.x < (blockDim.x >> 5) ? warp_vals[threadIdx.x] : 0.0;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
        if (threadIdx.x == 0) partial[blockIdx.x] = v;
    }
}

// The same for small lattices, eight lanes per site: lane p < 6 evaluates
// plane p (three products deep instead of nine pairs), the site's first lane
// adds them in plane order, and the tile's 128 sites are then summed by
// k_su2_plaquette's tree, so the bits are its.  A 10^4 lattice (79 tiles):
// a measured sweep of one heat-bath and three overrelaxations 205 -> 195 us
// together with the geometry passed by value.
__global__ void __launch_bounds__(kSiteThreads * kGroup)
k_su2_plaquette_group(const ChainInfo *__restrict__ chains, const Tile *__restrict__ tiles,
                      const double2 *__restrict__ links, double *__restrict__ partial) {
    __shared__ double site_vals[kSiteThreads];
    __shared__ double warp_vals[kSiteThreads / 32];
    const Tile tile = tiles[blockIdx.x];
    const ChainInfo c = chains[tile.chain];
    const int site = threadIdx.x / kGroup, lane = threadIdx.x & 31, j = lane & (kGroup - 1), lead = lane - j;
    const int64_t s = tile.start + site;
    const bool active = s < c.volume && j < 6;
    double w = 0.0;
    if (active) {
        const Coord x = decode_storage(c, s);
        const Nb self{x.lex, x.par};
        const int mu = j < 3 ? 0 : (j < 5 ? 1 : 2), nu = j < 3 ? j + 1 : (j < 5 ? j - 1 : 3);
        const Nb pm = step_any(c, x.x, x.lex, x.par, mu, +1);
        const Nb pn = step_any(c, x.x, x.lex, x.par, nu, +1);
        q4 p = qmul(link_q(links, c, self, mu), link_q(links, c, pm, nu));
        p = qmul(p, qdag(link_q(links, c, pn, mu)));
        w = qmul(p, qdag(link_q(links, c, self, nu))).c[0];
    }
    double v = __shfl_sync(0xffffffffu, w, lead);
#pragma unroll
    for (int k = 1; k < 6; ++k) v = v + __shfl_sync(0xffffffffu, w, lead + k);
    if (j == 0) site_vals[site] = s < c.volume ? v : 0.0;
    __syncthreads();
    if (threadIdx.x < kSiteThreads) {
        v = site_vals[threadIdx.x];
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
        if (lane == 0) warp_vals[threadIdx.x >> 5] = v;
    }
    __syncthreads();
    if (threadIdx.x == 0) partial[blockIdx.x] = (warp_vals[0] + warp_vals[2]) + (warp_vals[1] + warp_vals[3]);
}

// max |norm^2 - 1| per tile (Lattice4::max_link_unit_residual lib.rs:726-740).
__global__ void __launch_bounds__(kSiteThreads)
k_su2_unit_residual(const ChainInfo *__restrict__ chains, const Tile *__restrict__ tiles,
                    const double2 *__restrict__ links, double *__restrict__ partial) {
    __shared__ double warp_vals[32];
    const Tile tile = tiles[blockIdx.x];
    const ChainInfo c = chains[tile.chain];
    const int64_t s = tile.start + threadIdx.x;
    double r = 0.0;
    if (s < c.volume) {
        for (int mu = 0; mu < 4; ++mu) {
            const q4 q = load_q(links, c, s, mu);
            double n2 = q.c[0] * q.c[0];
            n2 = n2 + q.c[1] * q.c[1];
            n2 = n2 + q.c[2] * q.c[2];
            n2 = n2 + q.c[3] * q.c[3];
            const double res = isfinite(n2) ? fabs(n2 - 1.0) : INFINITY;
            r = isfinite(res) ? fmax(r, res) : INFINITY;
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) r = fmax(r, __shfl_down_sync(0xffffffffu, r, off));
    if ((threadIdx.x & 31) == 0) warp_vals[threadIdx.x >> 5] = r;
    __syncthreads();
    if (threadIdx.x < 32) {
        r = threadIdx.x < (blockDim.x >> 5) ? warp_vals[threadIdx.x] : 0.0;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) r = fmax(r, __shfl_down_sync(0xffffffffu, r, off));
        if (threadIdx.x == 0) partial[blockIdx.x] = r;
    }
}

// Every chain at once: blockIdx.y picks the chain.
__global__ void k_su2_identity(const ChainInfo *__restrict__ chains, double2 *links) {
    const ChainInfo c = chains[blockIdx.y];
    const int64_t n = 8 * c.volume;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t plane = i / c.volume;
        links[c.offset + i] = make_double2((plane % 2 == 0) ? 1.0 : 0.0, 0.0);
    }
}

__global__ void k_su2_from_aos(const ChainInfo *__restrict__ chains, int chain, double2 *links,
                               const double2 *__restrict__ staging) {
    const ChainInfo c = chains[chain];
    for (int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; s < c.volume;
         s += (int64_t)gridDim.x * blockDim.x) {
        const Coord x = decode_storage(c, s);
        for (int mu = 0; mu < 4; ++mu) {
            const double2 *src = staging + (x.lex * 4 + mu) * 2;
            double2 *dst = links + c.offset + (int64_t)(mu * 2) * c.volume + s;
            dst[0] = src[0];
            dst[c.volume] = src[1];
        }
    }
}

__global__ void k_su2_to_aos(const ChainInfo *__restrict__ chains, int chain,
                             const double2 *__restrict__ links, double2 *staging) {
    const ChainInfo c = chains[chain];
    for (int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; s < c.volume;
         s += (int64_t)gridDim.x * blockDim.x) {
        const Coord x = decode_storage(c, s);
        for (int mu = 0; mu < 4; ++mu) {
            double2 *dst = staging + (x.lex * 4 + mu) * 2;
            const double2 *src = links + c.offset + (int64_t)(mu * 2) * c.volume + s;
            dst[0] = src[0];
            dst[1] = src[c.volume];
        }
    }
}

int grid_for(int64_t n, int threads) {
    int64_t b = (n + threads - 1) / threads;
    if (b > 148 * 16) b = 148 * 16;
    return (int)(b < 1 ? 1 : b);
}

}  // namespace

// The grouped kernels give each link kGroup lanes; they win while a
// sub-sweep has too few links to hide the one-thread kernels' latency
// (measured on B200: 5,000 links per launch 15.5 vs 24.5 us heat-bath,
// 32,768 links 35.4 vs 25.2 us, crossover near 17,000), so up to 96 links
// per SM.
static bool su2_grouped(const ym_ensemble *e) {
    static thread_local int sms = 0, dev_seen = -1;
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev != dev_seen) {
        sms = 148;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        dev_seen = dev;
    }
    return e->n_half_tiles * (int64_t)T <= (int64_t)sms * 96;
}

cudaError_t launch_su2_heatbath(ym_ensemble *e, int parity, int mu, int max_attempts, int kp) {
    auto *ch = e->d_chains;
    auto *tl = e->d_half_tiles;
    const ChainInfo one = single_chain(e);
    const dim3 b(T);
    if (su2_grouped(e)) {
        const dim3 g((unsigned)(e->n_half_tiles * kGroup));
        k_su2_heatbath_group<<<g, b, 0, e->stream>>>(ch, tl, one, e->d_links, parity, mu, max_attempts, kp, sweep_index(e),
                                                     e->d_accepts, e->d_error);
        return cudaGetLastError();
    }
    const dim3 g((unsigned)e->n_half_tiles);
    switch (mu) {
    case 0: k_su2_heatbath_thread<0><<<g, b, 0, e->stream>>>(ch, tl, one, e->d_links, parity, max_attempts, kp, sweep_index(e), e->d_accepts, e->d_error); break;
    case 1: k_su2_heatbath_thread<1><<<g, b, 0, e->stream>>>(ch, tl, one, e->d_links, parity, max_attempts, kp, sweep_index(e), e->d_accepts, e->d_error); break;
    case 2: k_su2_heatbath_thread<2><<<g, b, 0, e->stream>>>(ch, tl, one, e->d_links, parity, max_attempts, kp, sweep_index(e), e->d_accepts, e->d_error); break;
    default: k_su2_heatbath_thread<3><<<g, b, 0, e->stream>>>(ch, tl, one, e->d_links, parity, max_attempts, kp, sweep_index(e), e->d_accepts, e->d_error); break;
    }
    return cudaGetLastError();
}

cudaError_t launch_su2_overrelax(ym_ensemble *e, int parity, int mu) {
    auto *ch = e->d_chains;
    auto *tl = e->d_half_tiles;
    const ChainInfo one = single_chain(e);
    const dim3 b(T);
    if (su2_grouped(e)) {
        const dim3 g((unsigned)(e->n_half_tiles * kGroup));
        k_su2_overrelax_group<<<g, b, 0, e->stream>>>(ch, tl, one, e->d_links, parity, mu, e->d_error);
        return cudaGetLastError();
    }
    const dim3 g((unsigned)e->n_half_tiles);
    switch (mu) {
    case 0: k_su2_overrelax_thread<0><<<g, b, 0, e->stream>>>(ch, tl, one, e->d_links, parity, e->d_error); break;
    case 1: k_su2_overrelax_thread<1><<<g, b, 0, e->stream>>>(ch, tl, one, e->d_links, parity, e->d_error); break;
    case 2: k_su2_overrelax_thread<2><<<g, b, 0, e->stream>>>(ch, tl, one, e->d_links, parity, e->d_error); break;
    default: k_su2_overrelax_thread<3><<<g, b, 0, e->stream>>>(ch, tl, one, e->d_links, parity, e->d_error); break;
    }
    return cudaGetLastError();
}

cudaError_t launch_su2_plaquette_partials(ym_ensemble *e) {
    if (su2_grouped(e)) {
        k_su2_plaquette_group<<<(unsigned)e->n_site_tiles, kSiteThreads * kGroup, 0, e->stream>>>(
            e->d_chains, e->d_site_tiles, e->d_links, e->d_partial);
        return cudaGetLastError();
    }
    k_su2_plaquette<<<(unsigned)e->n_site_tiles, kSiteThreads, 0, e->stream>>>(
        e->d_chains, e->d_site_tiles, e->d_links, e->d_partial);
    return cudaGetLastError();
}

cudaError_t launch_su2_unit_residual_partials(ym_ensemble *e) {
    k_su2_unit_residual<<<(unsigned)e->n_site_tiles, kSiteThreads, 0, e->stream>>>(
        e->d_chains, e->d_site_tiles, e->d_links, e->d_partial);
    return cudaGetLastError();
}

cudaError_t launch_su2_identity(ym_ensemble *e) {
    int64_t vmax = 0;
    for (const ChainInfo &c : e->chains) vmax = c.volume > vmax ? c.volume : vmax;
    for (int64_t first = 0; first < e->n_chains; first += 65535) {   // the grid's y limit
        const int64_t count = e->n_chains - first < 65535 ? e->n_chains - first : 65535;
        const int64_t bx = (grid_for(8 * vmax, 256) + count - 1) / count;
        k_su2_identity<<<dim3((unsigned)(bx < 1 ? 1 : bx), (unsigned)count), 256, 0, e->stream>>>(
            e->d_chains + first, e->d_links);
    }
    return cudaGetLastError();
}

cudaError_t launch_su2_from_aos(ym_ensemble *e, int64_t chain) {
    k_su2_from_aos<<<grid_for(e->chains[chain].volume, 128), 128, 0, e->stream>>>(
        e->d_chains, (int)chain, e->d_links, reinterpret_cast<const double2 *>(e->d_staging));
    return cudaGetLastError();
}

cudaError_t launch_su2_to_aos(ym_ensemble *e, int64_t chain) {
    k_su2_to_aos<<<grid_for(e->chains[chain].volume, 128), 128, 0, e->stream>>>(
        e->d_chains, (int)chain, e->d_links, reinterpret_cast<double2 *>(e->d_staging));
    return cudaGetLastError();
}

}  // namespace ym
