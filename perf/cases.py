"""Performance cases of the lattice engine: the calls a user's program makes,
over the sizes, storage precisions and options it makes them with.

listed() and draw(rng) give cases, prepare(case, seed) what a program holds
before the call (handles with a field uploaded, host buffers, a model),
run(state) one pass through the public entry points, work(case) what one pass
cannot do without, and exact(case, seed) the same outputs in plain torch in
64 bits.

Kinds of case:
  su3_chain  SU(3) Metropolis chains through Ensemble.measured_sweeps (the
             run_chain cadence: sweeps, a plaquette after each stride), then
             the accept counts and the configurations, as a checkpoint reads
             them; binary64 or two-row binary32 storage, ordered or drawn
             generators.
  su3_run    the loop-measurement cadence of one large lattice through
             Ensemble.measured_run: sweeps with a plaquette each, Wilson
             loops R x T <= 4 x 4 and Polyakov loops after every block, then
             the configuration saved.
  su2_chain  SU(2) heat-bath plus overrelaxation chains through
             Ensemble.su2_measured_sweeps, then counts and configurations.
  glueball   one step of the scalar-glueball production over uneven chain
             groups: sweeps, then Ensemble.glueball_measure (stout levels,
             A1++ operators, stride-2 blocking of the groups that admit it).
  measure    observables of a stored configuration (any extents): upload,
             average plaquette, Wilson and Polyakov loops, and for cubic
             spatial extents the A1++ operators before and after stout.
  learned    learned-proposal sweeps through ProposalModel.measured_sweeps.
  train      ProposalModel.train: sweeps, records, objective gradient, Adam.
"""
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "yang-mills_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)
import ymgpu  # noqa: E402
from ymgpu.learned import N_PARAMS, OFFSETS, ProposalModel  # noqa: E402

MASK64 = (1 << 64) - 1
RHO = 0.1                       # stout coefficient of the production campaigns
BETA_SU3, BETA_SU2 = 6.0, 2.3


def listed():
    return [
        # the smallest call: one sweep and its plaquette on the lattice of the
        # reference's own golden chains
        dict(name="su3_4x4_one_sweep", kind="su3_chain", extents="4x4x4x4", chains=1, precision="f64",
             generators="ordered", angle=0.3, beta=BETA_SU3, measurements=1, stride=1),
        # many small independent chains with drawn generators in one handle
        dict(name="su3_64_chains_4x4", kind="su3_chain", extents="4x4x4x4", chains=64, precision="f64",
             generators="uniform", angle=0.3, beta=BETA_SU3, measurements=40, stride=1),
        # ragged lattices of a production campaign, the run_chain cadence
        dict(name="su3_32_chains_6x6x6x10", kind="su3_chain", extents="6x6x6x10", chains=32, precision="f64",
             generators="ordered", angle=0.35, beta=5.7, measurements=10, stride=4),
        # plain two-row sampling of an ensemble, the ESS comparison's workload
        dict(name="su3_4_chains_16x4_f32", kind="su3_chain", extents="16x16x16x16", chains=4, precision="f32",
             generators="uniform", angle=0.3, beta=BETA_SU3, measurements=20, stride=1),
        # the headline lattice: binary64 sweeps with loops every ten, then saved
        dict(name="su3_32x4_f64_run", kind="su3_run", extents="32x32x32x32", precision="f64", generators="ordered",
             angle=0.3, beta=BETA_SU3, blocks=2, sweeps=10),
        # the same cadence in two-row storage on the other large lattice
        dict(name="su3_24x3x48_f32_run", kind="su3_run", extents="24x24x24x48", precision="f32", generators="ordered",
             angle=0.3, beta=BETA_SU3, blocks=2, sweeps=10),
        # the SU(2) benchmark lattice: one Kennedy-Pendleton heat-bath and
        # three overrelaxation sweeps per measurement
        dict(name="su2_10x4_kp", kind="su2_chain", extents="10x10x10x10", chains=1, sampler="kennedy-pendleton",
             beta=BETA_SU2, overrelaxation=3, measurements=8, stride=1),
        # a large SU(2) lattice with the reference's own sampler
        dict(name="su2_24x4_reference", kind="su2_chain", extents="24x24x24x24", chains=1, sampler="reference",
             beta=BETA_SU2, overrelaxation=1, measurements=16, stride=1),
        # the batched scalar-glueball production: 224 uneven chains
        dict(name="glueball_224_chains", kind="glueball", groups="128:4x10,64:6x12,32:8x16", beta=5.7, angle=0.35,
             sweeps=4, levels="0,5,10"),
        # a stored configuration with odd extents, measured
        dict(name="measure_9x3x15", kind="measure", extents="9x9x9x15", levels="3"),
        # learned-proposal sampling of the lattice it is trained on
        dict(name="learned_4_chains_16x4", kind="learned", extents="16x16x16x16", chains=4, beta=BETA_SU3,
             measurements=10, stride=1),
        # training of the proposal on configurations the sampler generates
        dict(name="train_16x4", kind="train", extents="16x16x16x16", chains=1, beta=BETA_SU3, angle=0.3, steps=20),
    ]


def _log_int(rng, low, high):
    return int(round(np.exp(rng.uniform(np.log(low), np.log(high)))))


def _even_extents(rng, volume):
    """Even extents of about the given volume, not all alike."""
    side = volume ** 0.25
    n = [max(2, 2 * int(round(side * np.exp(rng.uniform(-0.35, 0.35)) / 2))) for _ in range(4)]
    while n[0] * n[1] * n[2] * n[3] > volume * 1.5 and max(n) > 2:
        n[n.index(max(n))] -= 2
    return "x".join(str(max(2, v)) for v in n)


def draw(rng):
    kind = rng.choice(["su3_chain", "su3_chain", "su3_run", "su2_chain", "glueball", "measure", "learned", "train"])
    beta = round(rng.uniform(5.5, 6.5), 2)
    if kind == "su3_chain":
        volume, chains = _log_int(rng, 256, 200000), _log_int(rng, 1, 64)
        while volume * chains > 400000:
            chains = max(1, chains // 2)
        return dict(kind=kind, extents=_even_extents(rng, volume), chains=chains, precision=rng.choice(["f64", "f32"]),
                    generators=rng.choice(["ordered", "uniform"]), angle=round(rng.uniform(0.1, 1.0), 2), beta=beta,
                    measurements=rng.randint(1, 20), stride=rng.randint(1, 2))
    if kind == "su3_run":
        return dict(kind=kind, extents=_even_extents(rng, _log_int(rng, 4096, 700000)),
                    precision=rng.choice(["f64", "f32"]), generators="ordered", angle=round(rng.uniform(0.1, 0.5), 2),
                    beta=beta, blocks=rng.randint(1, 2), sweeps=rng.randint(5, 10))
    if kind == "su2_chain":
        volume, chains = _log_int(rng, 256, 400000), _log_int(rng, 1, 16)
        while volume * chains > 400000:
            chains = max(1, chains // 2)
        over = rng.randint(0, 4)     # overrelaxation amplifies rounding, so the passes with more of it are shorter
        return dict(kind=kind, extents=_even_extents(rng, volume), chains=chains,
                    sampler=rng.choice(["reference", "kennedy-pendleton"]), beta=round(rng.uniform(2.0, 2.6), 2),
                    overrelaxation=over, measurements=rng.randint(1, 20 // (1 + over)), stride=1)
    if kind == "glueball":
        groups = []
        for n in rng.sample([3, 4, 5, 6, 8, 10], rng.randint(1, 3)):
            n = n + (n % 2)         # sweeps need even extents
            if any(g.split(":")[1].startswith("%dx" % n) for g in groups):
                continue
            groups.append("%d:%dx%d" % (_log_int(rng, 2, 48), n, 2 * rng.randint(3, 9)))
        return dict(kind=kind, groups=",".join(groups), beta=round(rng.uniform(5.6, 6.0), 2), angle=0.35,
                    sweeps=rng.randint(1, 8), levels=rng.choice(["0,5,10", "0,1,2", "0,3", "8"]))
    if kind == "measure":
        n = rng.randint(3, 21)
        if rng.random() < 0.7:
            ext = "%dx%dx%dx%d" % (n, n, n, rng.randint(3, 40))
        else:
            ext = "x".join(str(rng.randint(4, 20)) for _ in range(4))
        return dict(kind=kind, extents=ext, levels=str(rng.randint(1, 8)))
    volume = _log_int(rng, 4096, 200000)
    if kind == "learned":
        return dict(kind=kind, extents=_even_extents(rng, volume), chains=rng.randint(1, 3), beta=beta,
                    measurements=rng.randint(2, 10), stride=1)
    return dict(kind=kind, extents=_even_extents(rng, volume), chains=rng.randint(1, 2), beta=beta, angle=0.3,
                steps=rng.randint(5, 20))


# ---------------------------------------------------------------- fields

def _ext(text):
    return [int(v) for v in text.split("x")]


def _groups(case):
    """[(chains, extents)] of a glueball case: '128:4x10' is 128 chains of 4^3 x 10."""
    out = []
    for part in case["groups"].split(","):
        count, size = part.split(":")
        n, t = (int(v) for v in size.split("x"))
        out.append((int(count), [n, n, n, t]))
    return out


def _levels(case):
    return [int(v) for v in case["levels"].split(",")]


def _cubic(ext):
    return ext[0] == ext[1] == ext[2] and ext[0] >= 3


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _neighbours(ext, dev):
    """(forward, backward) site tables [4][V] in lexicographic order, x3 fastest."""
    ids = torch.arange(int(np.prod(ext)), device=dev).reshape(ext)
    return ([torch.roll(ids, -1, d).reshape(-1) for d in range(4)],
            [torch.roll(ids, 1, d).reshape(-1) for d in range(4)])


def _mm(a, b):
    return (a.unsqueeze(-1) * b.unsqueeze(-3)).sum(-2)


def _dag(a):
    return a.conj().transpose(-1, -2)


def _qmul(a, b):
    a0, a1, a2, a3 = a.unbind(-1)
    b0, b1, b2, b3 = b.unbind(-1)
    return torch.stack([a0 * b0 - a1 * b1 - a2 * b2 - a3 * b3, a0 * b1 + a1 * b0 + a2 * b3 - a3 * b2,
                        a0 * b2 - a1 * b3 + a2 * b0 + a3 * b1, a0 * b3 + a1 * b2 - a2 * b1 + a3 * b0], -1)


def _qdag(a):
    return a * torch.tensor([1.0, -1.0, -1.0, -1.0], dtype=a.dtype, device=a.device)


def _special_unitary(m):
    """Gram-Schmidt of rows 0 and 1, row 2 their conjugate cross product."""
    r0 = m[..., 0, :]
    r0 = r0 / r0.abs().square().sum(-1, keepdim=True).sqrt()
    r1 = m[..., 1, :]
    for _ in range(2):
        r1 = r1 - (r0.conj() * r1).sum(-1, keepdim=True) * r0
    r1 = r1 / r1.abs().square().sum(-1, keepdim=True).sqrt()
    return torch.stack([r0, r1, torch.linalg.cross(r0, r1, dim=-1).conj()], -2)


def _field(ext, chains, group, seed):
    """Random links [chain, site, mu, ...] with about the plaquette of an
    equilibrium field (0.6): links near the identity, turned by a random
    gauge transformation, so single links look Haar random."""
    dev = _device()
    g = torch.Generator(device=dev).manual_seed(seed & 0x7FFFFFFF)
    v = int(np.prod(ext))
    fwd, _ = _neighbours(ext, dev)
    out = torch.empty((chains, v, 4, 3, 3) if group == 3 else (chains, v, 4, 4),
                      dtype=torch.complex128 if group == 3 else torch.float64, device=dev)
    for c in range(chains):
        if group == 3:
            def noise(*shape):
                return torch.complex(torch.randn(*shape, generator=g, device=dev, dtype=torch.float64),
                                     torch.randn(*shape, generator=g, device=dev, dtype=torch.float64))
            gauge = _special_unitary(noise(v, 3, 3))
            for mu in range(4):
                h = noise(v, 3, 3)
                w = _special_unitary(torch.eye(3, device=dev, dtype=torch.complex128) + 0.155j * (h + _dag(h)))
                out[c, :, mu] = _mm(_mm(gauge, w), _dag(gauge[fwd[mu]]))
        else:
            def unit(q):
                return q / q.square().sum(-1, keepdim=True).sqrt()
            gauge = unit(torch.randn(v, 4, generator=g, device=dev, dtype=torch.float64))
            for mu in range(4):
                w = 0.29 * torch.randn(v, 4, generator=g, device=dev, dtype=torch.float64)
                w[:, 0] = 1.0
                out[c, :, mu] = unit(_qmul(_qmul(gauge, unit(w)), _qdag(gauge[fwd[mu]])))
    return out


def _seeds(seed, n):
    return [(0x9E3779B97F4A7C15 * (seed + 1) + 0xD1B54A32D192ED03 * (i + 1)) & MASK64 for i in range(n)]


def _host(shape, dtype):
    """A pinned host array, as a program that moves configurations holds."""
    reals = int(np.prod(shape)) * (2 if dtype == np.complex128 else 1)
    return torch.empty(reals, dtype=torch.float64, pin_memory=torch.cuda.is_available()).numpy().view(dtype).reshape(shape)


def _host_links(ext, chains, group):
    links = int(np.prod(ext)) * 4
    return _host((chains, links, 3, 3) if group == 3 else (chains, links, 4),
                 np.complex128 if group == 3 else np.float64)


def _upload(ens, first, field, host):
    host[...] = field.reshape(host.shape).cpu().numpy()
    for c in range(host.shape[0]):
        ens.upload(first + c, host[c])


def _model_params(seed):
    """A network of the size and scale training ends at: small logits and an
    angle half width near 1.6."""
    r = np.random.RandomState(seed & 0x7FFFFFFF)
    p = np.zeros(N_PARAMS, np.float32)
    for name, fan, rows in (("W1", 16, 64), ("W2", 64, 64), ("W3", 64, 9)):
        a = np.sqrt(6.0 / fan) * (0.125 if name == "W3" else 1.0)
        p[OFFSETS[name]:OFFSETS[name] + rows * fan] = r.uniform(-a, a, rows * fan)
    p[OFFSETS["b3"] + 8] = 0.55
    return p


# ---------------------------------------------------------------- preparing and running

def prepare(case, seed):
    kind = case["kind"]
    st = dict(case=case)
    if kind in ("su3_chain", "su2_chain", "learned", "train"):
        ext, n = _ext(case["extents"]), case["chains"]
        group = 2 if kind == "su2_chain" else 3
        two_row = kind in ("learned", "train") or case.get("precision") == "f32"
        ens = ymgpu.Ensemble([ext] * n, case["beta"], _seeds(seed, n), group=group,
                             precision=ymgpu.F32_TWO_ROW if two_row else ymgpu.F64, lift_reference_caps=True)
        st["out"] = _host_links(ext, n, group)
        _upload(ens, 0, _field(ext, n, group, seed), st["out"])
        st["ens"] = ens
        if kind in ("learned", "train"):
            st["model"] = ProposalModel()
            st["model"].params = _model_params(seed)
    elif kind == "su3_run":
        ext = _ext(case["extents"])
        f32 = case["precision"] == "f32"
        ens = ymgpu.Ensemble([ext], case["beta"], _seeds(seed, 1), lift_reference_caps=True,
                             precision=ymgpu.F32_TWO_ROW if f32 else ymgpu.F64)
        st["out"] = _host_links(ext, 1, 3)
        _upload(ens, 0, _field(ext, 1, 3, seed), st["out"])
        st["ens"], st["view"] = ens, ens.like(precision=ymgpu.F64) if f32 else None
    elif kind == "glueball":
        groups = _groups(case)
        exts = [e for count, e in groups for _ in range(count)]
        ens = ymgpu.Ensemble(exts, case["beta"], _seeds(seed, len(exts)), lift_reference_caps=True)
        first, firsts = 0, []
        for k, (count, e) in enumerate(groups):
            _upload(ens, first, _field(e, count, 3, seed + 1000003 * k), _host_links(e, count, 3))
            firsts.append(first)
            first += count
        sm = ens.like()
        blocked = []
        for (count, e), at in zip(groups, firsts):
            if e[0] >= 6:
                fine = sm.subset(range(at, at + count))
                coarse = fine.like([[e[0] // 2, e[1] // 2, e[2] // 2, e[3]]] * count)
                blocked.append((fine, coarse, at))
        ens.glueball_prepare(sm, _levels(case), RHO, blocked)
        st.update(ens=ens, sm=sm, blocked=blocked)
    else:
        ext = _ext(case["extents"])
        st["ens"] = ymgpu.Ensemble([ext], BETA_SU3, _seeds(seed, 1), lift_reference_caps=True)
        st["smeared"] = st["ens"].like()
        st["links"] = _host_links(ext, 1, 3)
        st["links"][...] = _field(ext, 1, 3, seed).reshape(st["links"].shape).cpu().numpy()
    return st


def _save(st, ens):
    """The configurations of every chain, read back as a checkpoint does."""
    for c in range(ens.n_chains):
        ens.download(c, out=st["out"][c])
    return st["out"]


def run(st):
    case, kind, ens = st["case"], st["case"]["kind"], st["ens"]
    if kind == "su3_chain":
        series = ens.measured_sweeps(case["angle"], case["measurements"], case["stride"], case["generators"])
        _, accepts = ens.accounting()
        return dict(plaquette=series, accepts=accepts.astype(np.int64), links=_save(st, ens))
    if kind == "su3_run":
        plaq, wilson, poly = ens.measured_run(case["angle"], case["blocks"], case["sweeps"],
                                              generator_mode=case["generators"], view=st["view"])
        _, accepts = ens.accounting()
        return dict(plaquette=plaq, wilson=wilson, polyakov=poly, accepts=accepts.astype(np.int64),
                    links=_save(st, ens))
    if kind == "su2_chain":
        series = ens.su2_measured_sweeps(case["measurements"], case["stride"], case["overrelaxation"],
                                         sampler=case["sampler"])
        _, attempts = ens.heatbath_accounting()
        return dict(plaquette=series, attempts=attempts.astype(np.int64), links=_save(st, ens))
    if kind == "glueball":
        ens.metropolis_sweeps(case["angle"], case["sweeps"])
        p, r, bp, br = ens.glueball_measure(st["sm"], _levels(case), RHO, st["blocked"])
        return dict(plaquette=p, rectangle=r, blocked_plaquette=bp, blocked_rectangle=br)
    if kind == "measure":
        ens.upload(0, st["links"][0])
        out = dict(plaquette=ens.average_plaquette(), wilson=ens.wilson_loops(), polyakov=ens.polyakov_loops())
        if _cubic(ens.extents[0]):
            out["operators"] = list(ens.scalar_operator_basis()[0])
            ens.stout_smear_into(st["smeared"], RHO, _levels(case)[0])
            out["smeared_operators"] = list(st["smeared"].scalar_operator_basis()[0])
        return out
    if kind == "learned":
        series = st["model"].measured_sweeps(ens, case["measurements"], case["stride"])
        _, accepts = ens.accounting()
        return dict(plaquette=series, accepts=accepts.astype(np.int64), links=_save(st, ens))
    history = st["model"].train(ens, case["steps"], sweeps_per_step=1, plain_angle=case["angle"], lr=3e-3)
    return dict(objective=history, params=st["model"].params, links=_save(st, ens))


# ---------------------------------------------------------------- work

def work(case):
    """Bytes: every sweep reads and writes each link once, every measurement
    reads each once, and the host arrays are moved.  Flops: the matrix
    products (216 per 3 x 3 complex product, 28 per quaternion product)."""
    kind = case["kind"]
    if kind == "glueball":
        links = sum(c * int(np.prod(e)) * 4 for c, e in _groups(case))
        levels = max(_levels(case))
        spatial = links * 0.75
        return dict(bytes=links * 144.0 * (2 * case["sweeps"] + 2 * levels + len(_levels(case))),
                    flops=links * case["sweeps"] * 4800.0 + spatial * levels * 3200.0 +
                    links / 4 * len(_levels(case)) * 24 * 216.0)
    sites = int(np.prod(_ext(case["extents"])))
    if kind == "measure":
        levels = _levels(case)[0] if _cubic(_ext(case["extents"])) else 0
        return dict(bytes=sites * 4 * 144.0 * (5 + 2 * levels),
                    flops=sites * (228 * 216.0 + 13 * 216 + 48 * 216 + levels * 3 * 3200.0))
    links = sites * 4 * case.get("chains", 1)
    if kind == "su2_chain":
        sweeps = case["measurements"] * case["stride"] * (1 + case["overrelaxation"])
        return dict(bytes=links * (64.0 * sweeps + 32 * case["measurements"] + 64),
                    flops=links * (sweeps * 14 * 28.0 + case["measurements"] * 4.5 * 28))
    size = 144.0 if case.get("precision") == "f64" else 48.0
    sweep_flops = 4800.0            # 12 staple products and eight hits
    if kind == "su3_run":
        n = case["blocks"] * case["sweeps"]
        return dict(bytes=links * (2 * size * n + 2 * 144.0 * case["blocks"] + 288.0),
                    flops=links * n * (sweep_flops + 3.5 * 216) + sites * case["blocks"] * 232 * 216.0)
    if kind == "train":
        half = links / 8            # one checkerboard sub-sweep's links per step
        return dict(bytes=case["steps"] * (links * 2 * size + half * 4 * (16 + 18)) + links * 144.0,
                    flops=case["steps"] * (links * sweep_flops + half * (2592.0 + 6 * 6288 * 1.0)))
    n = case["measurements"] * case["stride"]
    net = 2 * 6144.0 if kind == "learned" else 0.0
    return dict(bytes=links * (2 * size * n + 144.0), flops=links * n * (sweep_flops + net) +
                links * case["measurements"] * 3.5 * 216)


# ---------------------------------------------------------------- 64-bit values

_GELL_MANN = np.zeros((8, 3, 3), complex)
for _a, (_i, _j) in ((0, (0, 1)), (3, (0, 2)), (5, (1, 2))):
    _GELL_MANN[_a][_i, _j] = _GELL_MANN[_a][_j, _i] = 1.0
    _GELL_MANN[_a + 1][_i, _j], _GELL_MANN[_a + 1][_j, _i] = -1j, 1j
_GELL_MANN[2] = np.diag([1.0, -1.0, 0.0])
_GELL_MANN[7] = np.diag([1.0, 1.0, -2.0]) / np.sqrt(3.0)


def _s64(v):
    """An unsigned 64-bit constant as torch's signed 64-bit integer."""
    v &= MASK64
    return v - (1 << 64) if v >> 63 else v


def _shr(v, k):
    return (v >> k) & ((1 << (64 - k)) - 1)


def _mix(v):
    v = (v ^ _shr(v, 30)) * _s64(0xBF58476D1CE4E5B9)
    v = (v ^ _shr(v, 27)) * _s64(0x94D049BB133111EB)
    return v ^ _shr(v, 31)


def _word(key, n):
    """Output n of the SplitMix64 stream(s) seeded with key."""
    step = 0x9E3779B97F4A7C15
    return _mix(key + (_s64((n + 1) * step) if isinstance(n, int) else (n + 1) * _s64(step)))


def _unit(w):
    return _shr(w, 11).double() * 2.0 ** -53


class _Chains:
    """Equal-sized chains [chain, site, mu, ...] updated in plain torch."""

    def __init__(self, ext, field, beta, seeds):
        dev = field.device
        self.ext, self.u, self.beta = ext, field, beta
        self.seeds = torch.tensor([_s64(s) for s in seeds], dtype=torch.int64, device=dev)[:, None]
        self.fwd, self.bwd = _neighbours(ext, dev)
        grid = torch.meshgrid(*[torch.arange(n, device=dev) for n in ext], indexing="ij")
        par = (sum(grid) & 1).reshape(-1)
        self.sites = [torch.nonzero(par == p).reshape(-1) for p in (0, 1)]
        self.sweep = 0
        self.lam = torch.tensor(_GELL_MANN, device=dev)

    def keys(self, idx, mu):
        return _word(_word(self.seeds, self.sweep), (4 * idx + mu)[None, :])

    def staple(self, idx, mu, mul, dag):
        u, f, b = self.u, self.fwd, self.bwd
        total = 0
        for nu in range(4):
            if nu == mu:
                continue
            total = total + mul(mul(u[:, f[mu][idx], nu], dag(u[:, f[nu][idx], mu])), dag(u[:, idx, nu]))
            d = b[nu][idx]
            total = total + mul(mul(dag(u[:, f[mu][d], nu]), dag(u[:, d, mu])), u[:, d, nu])
        return total

    def metropolis(self, angle, uniform):
        for par in (0, 1):
            idx = self.sites[par]
            for mu in range(4):
                a = self.staple(idx, mu, _mm, _dag)
                key, link = self.keys(idx, mu), self.u[:, idx, mu]
                old = torch.einsum("...ij,...ji->...", link, a).real
                for h in range(8):
                    w = _word(key, 2 * h)
                    theta = angle * (2 * (w & ((1 << 52) - 1)) + 1).double() * 2.0 ** -53
                    theta = torch.where(w < 0, theta, -theta)
                    gen = _shr(w, 52) & 7 if uniform else torch.full_like(w, h)
                    lam = self.lam[gen]
                    half, phi = 0.5 * theta, theta / (2 * np.sqrt(3.0))
                    # exp(i theta T): cos + i sin lambda on the subgroup's rows, 1 on the other
                    sub = _mm(lam, lam)
                    rot = (torch.eye(3, device=lam.device) - sub) + torch.cos(half)[..., None, None] * sub + \
                        1j * torch.sin(half)[..., None, None] * lam
                    diag = torch.diag_embed(torch.stack([torch.exp(1j * phi), torch.exp(1j * phi),
                                                         torch.exp(-2j * phi)], -1))
                    rot = torch.where((gen == 7)[..., None, None], diag, rot)
                    cand = _mm(rot, link)
                    new = torch.einsum("...ij,...ji->...", cand, a).real
                    ok = _unit(_word(key, 2 * h + 1)) < torch.exp(-torch.clamp(self.beta / 3.0 * (old - new), min=0.0))
                    link = torch.where(ok[..., None, None], cand, link)
                    old = torch.where(ok, new, old)
                self.u[:, idx, mu] = link
        self.sweep += 1

    def su2_sample(self, alpha, key, kp):
        """The heat-bath quaternion of every link, rejection by rejection."""
        shape, alpha, key = alpha.shape, alpha.reshape(-1), key.reshape(-1)
        r0, after = torch.empty_like(alpha), torch.zeros_like(key)
        todo, k = torch.arange(alpha.numel(), device=alpha.device), 0
        while todo.numel():
            al, ky = alpha[todo], key[todo]
            if kp:
                u1, u2, u3, u4 = (_unit(_word(ky, k + i)) for i in range(4))
                x = -(torch.log(1 - u1) + torch.cos(2 * np.pi * u2) ** 2 * torch.log(1 - u3)) / al
                val, ok, k = 1 - x, u4 * u4 <= 1 - 0.5 * x, k + 4
            else:
                val = 1 + torch.log1p(_unit(_word(ky, k)) * torch.expm1(-2 * al)) / al
                val = val.clamp(-1, 1)
                ok, k = _unit(_word(ky, k + 1)) <= (1 - val * val).clamp(min=0).sqrt(), k + 2
            r0[todo[ok]], after[todo[ok]] = val[ok], k
            todo = todo[~ok]
        radial = (1 - r0 * r0).clamp(min=0).sqrt()
        z = 2 * _unit(_word(key, after)) - 1
        phi, planar = 2 * np.pi * _unit(_word(key, after + 1)), (1 - z * z).clamp(min=0).sqrt()
        q = torch.stack([r0, radial * planar * torch.cos(phi), radial * planar * torch.sin(phi), radial * z], -1)
        return (q / q.square().sum(-1, keepdim=True).sqrt()).reshape(*shape, 4)

    def su2_sweep(self, overrelax, kp):
        for par in (0, 1):
            idx = self.sites[par]
            for mu in range(4):
                a = self.staple(idx, mu, _qmul, _qdag)
                norm = a.square().sum(-1, keepdim=True).sqrt()
                r = self.su2_sample(self.beta * norm[..., 0], self.keys(idx, mu), kp)
                self.u[:, idx, mu] = _qmul(r, _qdag(a / norm))
        self.sweep += 1
        for _ in range(overrelax):
            for par in (0, 1):
                idx = self.sites[par]
                for mu in range(4):
                    a = self.staple(idx, mu, _qmul, _qdag)
                    v = _qdag(a / a.square().sum(-1, keepdim=True).sqrt())
                    self.u[:, idx, mu] = _qmul(_qmul(v, _qdag(self.u[:, idx, mu])), v)

    # -------- observables
    def plaquette(self):
        f, u, total = self.fwd, self.u, 0.0
        for mu in range(3):
            for nu in range(mu + 1, 4):
                if u.dim() == 5:
                    p = _mm(u[:, :, mu], u[:, f[mu], nu])
                    q = _mm(u[:, :, nu], u[:, f[nu], mu])
                    total = total + (p * q.conj()).real.sum((-1, -2, -3)) / 3
                else:
                    p = _qmul(u[:, :, mu], u[:, f[mu], nu])
                    q = _qmul(u[:, :, nu], u[:, f[nu], mu])
                    total = total + (p * q).sum((-1, -2))
        return (total / (6.0 * u.shape[1])).cpu().numpy()

    def wilson(self):
        f, u = self.fwd, self.u
        out, plane = np.zeros((u.shape[0], 6, 4, 4)), 0
        for mu in range(3):
            for nu in range(mu + 1, 4):
                d, at, qs = None, torch.arange(u.shape[1], device=u.device), []
                for _ in range(4):
                    link = u[:, at, nu]
                    d = link if d is None else _mm(d, link)
                    qs.append(d)
                    at = f[nu][at]
                a, wa = None, torch.arange(u.shape[1], device=u.device)
                for r in range(4):
                    link = u[:, wa, mu]
                    a = link if a is None else _mm(a, link)
                    wq, wa = wa, f[mu][wa]
                    p, wp = a, wa
                    for t in range(4):
                        p, wp, wq = _mm(p, u[:, wp, nu]), f[nu][wp], f[nu][wq]
                        qs[t] = _mm(qs[t], u[:, wq, mu])
                        out[:, plane, r, t] = ((p * qs[t].conj()).real.sum((-1, -2)) / 3).mean(-1).cpu().numpy()
                plane += 1
        return out

    def polyakov(self, d=3):
        at = torch.arange(self.u.shape[1], device=self.u.device).reshape(self.ext).select(d, 0).reshape(-1)
        h = self.u[:, at, d]
        for _ in range(self.ext[d] - 1):
            at = self.fwd[d][at]
            h = _mm(h, self.u[:, at, d])
        return (torch.einsum("...ii->...", h) / 3).mean(-1).cpu().numpy()

    def operators(self):
        """A1++ plaquette and rectangle means per chain and time slice."""
        f, u = self.fwd, self.u
        here = torch.arange(u.shape[1], device=u.device)

        def loop(mu, nu, r):
            p, at = u[:, here, mu], f[mu]
            for _ in range(r - 1):
                p, at = _mm(p, u[:, at, mu]), f[mu][at]
            p = _mm(p, u[:, at, nu])
            q, at = u[:, here, nu], f[nu]
            for _ in range(r):
                q, at = _mm(q, u[:, at, mu]), f[mu][at]
            return (p * q.conj()).real.sum((-1, -2)) / 3

        pairs = [(0, 1), (0, 2), (1, 2)]
        p = sum(loop(a, b, 1) for a, b in pairs) / 3
        r = sum(loop(a, b, 2) + loop(b, a, 2) for a, b in pairs) / 6
        nt = self.ext[3]
        return (p.reshape(p.shape[0], -1, nt).mean(1).cpu().numpy(), r.reshape(r.shape[0], -1, nt).mean(1).cpu().numpy())

    def copy(self):
        other = object.__new__(_Chains)
        other.__dict__.update(self.__dict__, u=self.u.clone())
        return other

    def stout(self, levels):
        f, b = self.fwd, self.bwd
        for _ in range(levels):
            u, new = self.u, self.u.clone()
            for mu in range(3):
                c = 0
                for nu in range(3):
                    if nu == mu:
                        continue
                    c = c + _mm(_mm(u[:, :, nu], u[:, f[nu], mu]), _dag(u[:, f[mu], nu]))
                    d = b[nu]
                    c = c + _mm(_mm(_dag(u[:, d, nu]), u[:, d, mu]), u[:, f[mu][d], nu])
                om = RHO * _mm(c, _dag(u[:, :, mu]))
                a = _dag(om) - om
                q = 0.5j * a
                q = q - torch.einsum("...ii->...", q)[..., None, None] / 3 * torch.eye(3, device=q.device)
                new[:, :, mu] = _mm(torch.matrix_exp(1j * q), u[:, :, mu])
            self.u = new

    def blocked(self):
        n, t = self.ext[0], self.ext[3]
        even = torch.arange(n * n * n * t, device=self.u.device).reshape(n, n, n, t)[::2, ::2, ::2].reshape(-1)
        v = torch.stack([_mm(self.u[:, even, mu], self.u[:, self.fwd[mu][even], mu]) for mu in range(3)] +
                        [self.u[:, even, 3]], 2)
        other = object.__new__(_Chains)
        ext = [n // 2, n // 2, n // 2, t]
        fwd, bwd = _neighbours(ext, v.device)
        other.__dict__.update(ext=ext, u=v, fwd=fwd, bwd=bwd)
        return other

    def links(self):
        v = self.u.reshape(self.u.shape[0], -1, *self.u.shape[3:])
        return v.cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind in ("learned", "train"):
        return None      # decided by the rounding of BF16 activations and binary32 steps
    if kind == "glueball":
        groups = _groups(case)
        n, first = sum(c for c, _ in groups), 0
        seeds, levels = _seeds(seed, n), _levels(case)
        rows = [[[], [], [], []] for _ in levels]
        for k, (count, e) in enumerate(groups):
            ch = _Chains(e, _field(e, count, 3, seed + 1000003 * k), case["beta"], seeds[first:first + count])
            first += count
            for _ in range(case["sweeps"]):
                ch.metropolis(case["angle"], False)
            done = 0
            for i, lv in enumerate(levels):
                ch.stout(lv - done)
                done = lv
                for j, v in enumerate(ch.operators()):
                    rows[i][j].append(v.reshape(-1))
                if e[0] >= 6:
                    for j, v in enumerate(ch.blocked().operators()):
                        rows[i][2 + j].append(v.reshape(-1))
        p, r, bp, br = (np.stack([np.concatenate(row[j]) if row[j] else np.zeros(0) for row in rows]) for j in range(4))
        return dict(plaquette=p, rectangle=r, blocked_plaquette=bp, blocked_rectangle=br)
    ext = _ext(case["extents"])
    n = case.get("chains", 1)
    ch = _Chains(ext, _field(ext, n, 2 if kind == "su2_chain" else 3, seed), case.get("beta", BETA_SU3), _seeds(seed, n))

    def saved():
        # binary32 decisions near the accept threshold part from the 64-bit
        # ones, and those links with them: no value for two-row storage
        return None if case.get("precision") == "f32" else ch.links()

    if kind == "measure":
        out = dict(plaquette=ch.plaquette(), wilson=ch.wilson(), polyakov=ch.polyakov())
        if _cubic(ext):
            out["operators"] = [v[0] for v in ch.operators()]
            ch.stout(_levels(case)[0])
            out["smeared_operators"] = [v[0] for v in ch.operators()]
        return out
    if kind == "su3_run":
        plaq, wilson, poly = [], [], []
        for _ in range(case["blocks"]):
            for _ in range(case["sweeps"]):
                ch.metropolis(case["angle"], False)
                plaq.append(ch.plaquette())
            wilson.append(ch.wilson())
            poly.append(ch.polyakov())
        return dict(plaquette=np.stack(plaq), wilson=np.stack(wilson), polyakov=np.stack(poly), accepts=None,
                    links=saved())
    plaq = []
    for _ in range(case["measurements"]):
        for _ in range(case["stride"]):
            if kind == "su3_chain":
                ch.metropolis(case["angle"], case["generators"] == "uniform")
            else:
                ch.su2_sweep(case["overrelaxation"], case["sampler"] != "reference")
        plaq.append(ch.plaquette())
    return dict(plaquette=np.stack(plaq), links=saved(),
                **{"accepts" if kind == "su3_chain" else "attempts": None})
