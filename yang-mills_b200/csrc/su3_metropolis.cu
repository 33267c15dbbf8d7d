// su3_metropolis.cu -- the SU(3) FP64 Metropolis sweeps with the
// reference's bits (compiled with -fmad=false): the tiled sub-sweep kernels
// of su3_tiled.cuh, the chain-resident kernel for small chains, and the
// dispatch to the fast form (su3_metropolis_fast.cu) for handles that ask
// for it.
#include "su3_tiled.cuh"

namespace ym {

namespace {

constexpr int T = kSweepThreads;

// ---------------------------------------------------------------------------
// Chain-resident sweeps for small lattices: one CTA per chain copies the
// chain's links into shared memory, runs n_meas x sweeps_per_meas whole
// sweeps there (sub-sweeps separated by block barriers) and writes the links
// back once.  A sweep over a small chain otherwise costs a launch per
// sub-sweep and a global-memory round trip per link; here neither.  Every
// link update is the tiled kernel's arithmetic on the same values
// (tiled_exact::visit_ordered / visit_drawn and the same staple chains), and
// the measured plaquette reproduces ym_average_plaquette's reduction
// (per-site sums, block_reduce's tree per 128-site tile, then the chain
// reduction's tree over the tile partials), so both paths give the same bits.
//
// What bounds it: one link update's latency, at one or two warps per
// scheduler.  The sub-sweep is one copy of code for all directions (the
// unrolled form, four directions of 60 KB, spent more time fetching
// instructions than executing them), each thread owns one link of each
// sub-sweep for the whole launch, and the hits run on the links in place:
// nobody else reads a link that is being updated.  64 chains of 4^4, drawn
// generators, per measured sweep: 247 us in the unrolled form, 82 as one loop
// (2.8 cycles per instruction, of which 1.3 wait for a binary64 result and
// 0.2 for an instruction), 78 with the hits' link-independent halves made by
// the threads that have no link, 72 with lambda8's row outside a branch;
// ordered hits 189, 52 and 46.
constexpr int kResidentThreads = 256;   // resident chains have at most 201 links per sub-sweep

// A link of the chain in shared memory.
__device__ __forceinline__ m3 resident_link(const double2 *p, int v) {
    m3 o;
#pragma unroll
    for (int e = 0; e < 9; ++e) {
        const double2 d = p[e * v];
        o.e[e / 3][e % 3] = cmake(d.x, d.y);
    }
    return o;
}

// a += the staple term (nu, BWD) of link (x, mu): the products of
// tiled_exact::term_accumulate on links read in place.
template <bool BWD>
__device__ __forceinline__ void resident_term(const double2 *sl, int v, const Site &x, int par, int mu,
                                              int nu, m3 &a) {
    const int same = par ? x.half : 0, other = par ? 0 : x.half;
    const int o = BWD ? x.lex + pick(x.bwd, nu) : x.lex;
    const double2 *ln = sl + nu * 9 * v, *lm = sl + mu * 9 * v;
    const int i1 = (BWD ? same : other) + ((o + pick(x.fwd, mu)) >> 1);
    const int i2 = other + ((BWD ? o : x.lex + pick(x.fwd, nu)) >> 1);
    const int i3 = BWD ? i2 : same + (x.lex >> 1);
    m3 p;
    {
        const m3 l1 = resident_link(ln + i1, v), l2 = resident_link(lm + i2, v);
        p = tiled_exact::pair_product<BWD>(l1, l2);
    }
    tiled_exact::add_third<BWD>(p, resident_link(ln + i3, v), a);
}

// The hits' link-independent halves of one sub-sweep, made by the threads that
// have no link of their own while the others form their staples: entry h of
// link t at [h][t].
struct PreTable {
    double2 e1[8][kResidentThreads / 2];   // rotation, or lambda8's phase of rows 0 and 1
    double2 e2[8][kResidentThreads / 2];   // lambda8's phase of row 2
    float logu[8][kResidentThreads / 2];
    int gen[8][kResidentThreads / 2];      // drawn generators
};

template <int K, bool DRAWN>
__device__ __forceinline__ void fill_table(PreTable &tab, int t, uint64_t key, double angle) {
    using namespace tiled_exact;
    uint64_t state = key;
#pragma unroll 1
    for (int h = 0; h < 8; ++h) {
        if (DRAWN) {
            const DrawnPre p = pre_drawn<K>(state, angle);
            tab.e1[h][t] = make_double2(p.e1.re, p.e1.im);
            tab.e2[h][t] = make_double2(p.e2.re, p.e2.im);
            tab.logu[h][t] = p.logu;
            tab.gen[h][t] = p.g;
        } else if (h < 7) {
            const BlockPre p = pre_block<K>(state, angle);
            tab.e1[h][t] = make_double2(p.c, p.s);
            tab.logu[h][t] = p.logu;
        } else {
            const DiagPre p = pre_diag<K>(state, angle);
            tab.e1[h][t] = make_double2(p.e1.re, p.e1.im);
            tab.e2[h][t] = make_double2(p.e2.re, p.e2.im);
            tab.logu[h][t] = p.logu;
        }
    }
}

struct TablePre {
    const PreTable &tab;
    int t, h;
    __device__ __forceinline__ tiled_exact::BlockPre block() {
        const double2 v = tab.e1[h][t];
        return tiled_exact::BlockPre{v.x, v.y, tab.logu[h++][t]};
    }
    __device__ __forceinline__ tiled_exact::DiagPre diag() {
        const double2 v = tab.e1[h][t], w = tab.e2[h][t];
        return tiled_exact::DiagPre{cmake(v.x, v.y), cmake(w.x, w.y), tab.logu[h][t]};
    }
    __device__ __forceinline__ tiled_exact::DrawnPre next() {
        const double2 v = tab.e1[h][t], w = tab.e2[h][t];
        const tiled_exact::DrawnPre p{cmake(v.x, v.y), cmake(w.x, w.y), tab.logu[h][t], tab.gen[h][t]};
        ++h;
        return p;
    }
};

// The three forms: where the staple sum waits for the hits, and who makes the
// hits' link-independent halves.
enum ResidentForm {
    kLocal,     // in local memory (chains that leave no room for it), each thread its own
    kShared,    // in shared memory, each thread its own
    kTable      // in shared memory, the upper half of the block (at most 128 links per sub-sweep)
};

template <int K, bool DRAWN, int FORM>
__global__ void __launch_bounds__(kResidentThreads, 1)
k_su3_resident(const ChainInfo *__restrict__ chains, double2 *__restrict__ links, double angle,
               uint64_t *sweep_ptr, int64_t n_meas, int64_t sweeps_per_meas,
               double *__restrict__ series, int64_t n_chains, unsigned long long *__restrict__ accepts) {
    using namespace tiled_exact;
    extern __shared__ __align__(16) double2 sl[];
    __shared__ double tile_sum[32];
    __shared__ double warp_sum[kResidentThreads / 32];
    const int64_t chain = blockIdx.x;
    const ChainInfo c = chains[chain];
    ChainInfo cs = c;
    cs.offset = 0;
    const int v = (int)c.volume, n = 36 * v, half = (int)c.half;
    for (int i = threadIdx.x; i < n; i += kResidentThreads) cp_async16(sl + i, links + c.offset + i);
    cp_async_commit();
    const int t = threadIdx.x;
    double2 local_a[FORM == kLocal ? 9 : 1];
    constexpr int kLinks = FORM == kTable ? kResidentThreads / 2 : kResidentThreads;
    const Col<FORM == kLocal ? 1 : kLinks> sa{FORM == kLocal ? local_a : sl + n + t % kLinks, 0};
    PreTable &tab = *reinterpret_cast<PreTable *>(sl + n + (FORM == kTable ? 9 * kLinks : 0));
    const bool helper = FORM == kTable && t >= kLinks;   // makes link t - kLinks's table
    const int mine = helper ? t - kLinks : t;
    const bool live = mine < half;
    const double beta3 = c.beta / 3.0;
    cp_async_wait_all();
    __syncthreads();
    const uint64_t sweep0 = *sweep_ptr;
    unsigned accepted = 0;
    for (int64_t m = 0; m < n_meas; ++m) {
        for (int64_t k = 0; k < sweeps_per_meas; ++k) {
            const uint64_t sweep = sweep0 + (uint64_t)(m * sweeps_per_meas + k);
            Site x;
#pragma unroll 1
            for (int sub = 0; sub < 8; ++sub) {
                const int par = sub >> 2, mu = sub & 3;
                uint64_t key = 0;
                if (live) {
                    if (mu == 0) x = site_of(c, decode_storage(c, par * half + mine));
                    key = link_key(c.seed, sweep, x.lex, mu);
                }
                if (helper) {
                    if (live) fill_table<K, DRAWN>(tab, mine, key, angle);
                } else if (live) {
                    m3 a;
#pragma unroll
                    for (int r = 0; r < 3; ++r)
#pragma unroll
                        for (int q = 0; q < 3; ++q) a.e[r][q] = cmake(0.0, 0.0);
#pragma unroll 1
                    for (int i = 0; i < 3; ++i) {
                        const int nu = i + (i >= mu ? 1 : 0);
                        resident_term<false>(sl, v, x, par, mu, nu, a);
                        resident_term<true>(sl, v, x, par, mu, nu, a);
                    }
#pragma unroll
                    for (int e = 0; e < 9; ++e) sa.put(e, a.e[e / 3][e % 3]);
                }
                if (FORM == kTable) __syncthreads();
                if (live && !helper) {
                    double2 *p = sl + mu * 9 * v + (par ? half : 0) + (x.lex >> 1);
                    const Col<0> rows{p, v};
                    if (DRAWN) {
                        accepted += FORM == kTable ? visit_drawn<K>(rows, sa, beta3, key, TablePre{tab, mine, 0})
                                                   : visit_drawn<K>(rows, sa, beta3, key, DrawnStream<K>{key, angle});
                    } else {
                        m3 u = resident_link(p, v);
                        double tr;
                        accepted += FORM == kTable
                                        ? visit_ordered(u, sa, beta3, key, TablePre{tab, mine, 0}, tr)
                                        : visit_ordered(u, sa, beta3, key, OrderedStream<K>{key, angle}, tr);
#pragma unroll
                        for (int e = 0; e < 9; ++e) rows.put(e, u.e[e / 3][e % 3]);
                    }
                }
                __syncthreads();
            }
        }
        if (series) {
            // 128-site tiles, two at a time: each warp's shuffle tree, then
            // block_reduce's tree over the tile's four warps
            const int n_tiles = (v + T - 1) / T;   // at most 32 (resident chains are small)
            for (int tile0 = 0; tile0 < n_tiles; tile0 += kResidentThreads / T) {
                const int s = tile0 * T + t;
                double q = s < v ? site_plaquette_sum<true>(sl, cs, s) : 0.0;
#pragma unroll
                for (int off = 16; off > 0; off >>= 1) q += __shfl_down_sync(0xffffffffu, q, off);
                if ((t & 31) == 0) warp_sum[t >> 5] = q;
                __syncthreads();
                if (t < kResidentThreads / T && tile0 + t < n_tiles) {
                    const double *w = warp_sum + t * (T / 32);
                    tile_sum[tile0 + t] = (w[0] + w[2]) + (w[1] + w[3]);
                }
                __syncthreads();
            }
            if (t < 32) {
                double q = t < n_tiles ? tile_sum[t] : 0.0;
#pragma unroll
                for (int off = 16; off > 0; off >>= 1) q += __shfl_down_sync(0xffffffffu, q, off);
                if (t == 0) series[m * n_chains + chain] = q / (6.0 * (double)c.volume);
            }
            __syncthreads();
        }
    }
    for (int i = threadIdx.x; i < n; i += kResidentThreads) links[c.offset + i] = sl[i];
    const unsigned sum = __reduce_add_sync(0xffffffffu, accepted);
    if ((threadIdx.x & 31) == 0 && sum) atomicAdd(accepts + chain, (unsigned long long)sum);
    __syncthreads();   // every thread has read the sweep counter
    if (threadIdx.x < 32) {
        const int last = threadIdx.x == 0 ? last_block(sweep_ptr + kSweepSlots) : 0;
        if (__shfl_sync(0xffffffffu, last, 0)) sweep_ptr[threadIdx.x] += (uint64_t)(n_meas * sweeps_per_meas);
    }
}

// (kSweepSlots threads)
__global__ void k_advance_sweep(uint64_t *sweep, uint64_t n) { sweep[threadIdx.x] += n; }

}  // namespace

cudaError_t launch_su3_metropolis(ym_ensemble *e, int parity, int mu, double angle, int uniform) {
    if (e->fast_sweeps) return launch_su3_metropolis_fast(e, parity, mu, angle, uniform);
    return tiled_exact::tiled_launch(e, parity, mu, angle, uniform);
}

cudaError_t launch_su3_metropolis_measure(ym_ensemble *e, int mu, double angle, double *tr_partial) {
    if (e->fast_sweeps) return launch_su3_metropolis_measure_fast(e, mu, angle, tr_partial);
    return tiled_exact::tiled_launch_measure(e, mu, angle, tr_partial);
}

size_t resident_smem_bytes(const ym_ensemble *e) {
    int64_t vmax = 0;
    for (const ChainInfo &c : e->chains) vmax = c.volume > vmax ? c.volume : vmax;
    return (size_t)vmax * 36 * sizeof(double2);
}

static int optin_smem() {
    int dev = 0, optin = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) return 0;
    return optin;
}

// static shared memory of the resident kernel (tile and warp sums) and slack
constexpr size_t kResidentFixed = sizeof(double) * (32 + 32) + 1024;
constexpr size_t kResidentAccumulator = (size_t)9 * kResidentThreads * sizeof(double2);

bool resident_fits(const ym_ensemble *e) {
    return resident_smem_bytes(e) + kResidentFixed <= (size_t)optin_smem();
}

// The dynamic shared memory limit of the three forms, set once per device to
// all a block may have.  It belongs to the kernel, not to the handle: set to
// each launch's own size, another thread's launch of a smaller handle could
// lower it between this thread's setting and its launch, which then fails.
template <int K, bool DRAWN>
static cudaError_t configure_resident() {
    static thread_local int configured_device = -1;
    int dev = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess || configured_device == dev) return err;
    const void *forms[3] = {(const void *)k_su3_resident<K, DRAWN, kLocal>,
                            (const void *)k_su3_resident<K, DRAWN, kShared>,
                            (const void *)k_su3_resident<K, DRAWN, kTable>};
    for (const void *f : forms) {
        cudaFuncAttributes at;
        if ((err = cudaFuncGetAttributes(&at, f)) != cudaSuccess) return err;
        err = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   optin_smem() - (int)at.sharedSizeBytes);
        if (err != cudaSuccess) return err;
    }
    configured_device = dev;
    return cudaSuccess;
}

template <int K, bool DRAWN>
static cudaError_t resident_launch(ym_ensemble *e, double angle, int64_t n_meas, int64_t sweeps_per_meas,
                                   double *series) {
    const size_t links = resident_smem_bytes(e);
    int64_t vmax = 0;
    for (const ChainInfo &c : e->chains) vmax = c.volume > vmax ? c.volume : vmax;
    auto kernel = k_su3_resident<K, DRAWN, kLocal>;
    size_t smem = links;
    if (vmax <= kResidentThreads) {   // half as many links per sub-sweep as threads
        kernel = k_su3_resident<K, DRAWN, kTable>;
        smem = links + kResidentAccumulator / 2 + sizeof(PreTable);
    } else if (links + kResidentAccumulator + kResidentFixed <= (size_t)optin_smem()) {
        kernel = k_su3_resident<K, DRAWN, kShared>;
        smem = links + kResidentAccumulator;
    }
    if (const cudaError_t err = configure_resident<K, DRAWN>()) return err;
    kernel<<<(unsigned)e->n_chains, kResidentThreads, smem, e->stream>>>(
        e->d_chains, e->d_links, angle, e->d_sweep, n_meas, sweeps_per_meas, series, e->n_chains, e->d_accepts);
    return cudaGetLastError();
}

cudaError_t launch_su3_resident(ym_ensemble *e, double angle, int uniform, int64_t n_meas,
                                int64_t sweeps_per_meas, double *series) {
    const bool small = angle <= tiled_exact::kShortRotation;
    return uniform ? (small ? resident_launch<11, true>(e, angle, n_meas, sweeps_per_meas, series)
                            : resident_launch<14, true>(e, angle, n_meas, sweeps_per_meas, series))
                   : (small ? resident_launch<11, false>(e, angle, n_meas, sweeps_per_meas, series)
                            : resident_launch<14, false>(e, angle, n_meas, sweeps_per_meas, series));
}

cudaError_t launch_counted_sweeps(ym_ensemble *e) {
    if (e->sweep_slot == 0) return cudaSuccess;
    k_advance_sweep<<<1, kSweepSlots, 0, e->stream>>>(e->d_sweep, (uint64_t)e->sweep_slot);
    const cudaError_t err = cudaGetLastError();
    if (err == cudaSuccess) e->sweep_slot = 0;
    return err;
}

cudaError_t launch_advance_sweep(ym_ensemble *e) {
    ++e->sweep_slot;
    const cudaError_t err = launch_counted_sweeps(e);
    if (err != cudaSuccess) --e->sweep_slot;
    return err;
}

}  // namespace ym
