"""The persistent sub-sweep kernel and the chain-resident kernel at the edges
of their work splits, against the oracle bit for bit.

Tiled: two CTAs per SM walk the work items (128 sites each), so the cases are
fewer items than CTAs, a second pass that only some CTAs take, items with
idle threads and several chains per launch.  Resident: one CTA of 256 threads
per chain, the staple sum in shared memory or (chains that leave no room for
it) in local memory.  Both generator modes and both rotation lengths (half
width <= 0.4 and above; 1.0 reaches lambda8's halved angles).  The plaquette
the sweep measures must agree with the oracle's to 1e-12.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MASTER = 0x2C02198105010002


def _check(oracle, extents, chains, angle, mode, path):
    import ymgpu
    seeds = [oracle.derive_su3_chain_seed(MASTER, i) for i in range(chains)]
    with ymgpu.Ensemble([extents] * chains, 5.9, seeds, lift_reference_caps=True) as ens:
        ens.sweep_path = path
        ens.hot_start()
        start = [ens.download(c) for c in range(chains)]
        ens.metropolis_sweeps(angle, 1, mode)
        series = ens.measured_sweeps(angle, 1, 1, mode)
        _, accepts = ens.accounting()
        for c in range(chains):
            ref = start[c].copy()
            acc = sum(oracle.su3_cb_sweep(extents, ref, 5.9, angle, seeds[c], k, mode == "uniform")[1]
                      for k in range(2))
            assert np.array_equal(ens.download(c), ref)
            assert int(accepts[c]) == acc
            plaq = oracle.su3_average_plaquette(extents, ref)
            assert abs(series[0, c] - plaq) <= 1e-12 * abs(plaq)


@pytest.mark.parametrize("mode", ["ordered", "uniform"])
@pytest.mark.parametrize("extents,chains,angle", [
    ([2, 2, 2, 2], 1, 0.3),          # eight live threads
    ([4, 4, 4, 6], 3, 0.4),          # 2 items per chain, the second half empty
    ([4, 4, 4, 4], 2, 1.0),
    ([16, 16, 16, 20], 1, 0.3),      # 320 items: a partial second pass on 148 SMs
    ([6, 6, 6, 10], 40, 0.45),       # 360 items of 40 chains, every ninth partial
])
def test_tiled_sweep_is_the_oracles(oracle, extents, chains, angle, mode):
    _check(oracle, extents, chains, angle, mode, "tiled")


@pytest.mark.parametrize("mode", ["ordered", "uniform"])
@pytest.mark.parametrize("extents,chains,angle", [
    ([2, 2, 2, 2], 1, 0.3),          # eight of 256 threads live
    ([4, 4, 4, 4], 150, 0.3),        # more chains than SMs
    ([4, 4, 2, 10], 2, 1.0),         # 320 sites, three plaquette tiles
    ([4, 4, 4, 6], 2, 0.35),         # 384 sites: no room for the sum in shared memory
])
def test_resident_sweep_is_the_oracles(oracle, extents, chains, angle, mode):
    _check(oracle, extents, chains, angle, mode, "resident")


@pytest.mark.parametrize("extents", [[4, 4, 4, 4], [2, 4, 4, 10]])
def test_short_calls_of_few_chains_match_the_tiled_path(extents):
    """Handles with at most one chain per SM run resident from the first
    call; one sweep, one measurement and a plaquette without a sweep give the
    tiled path's bits and leave the path undecided."""
    import ymgpu
    with ymgpu.Ensemble([extents] * 3, 6.0, [5, 6, 7]) as a, ymgpu.Ensemble([extents] * 3, 6.0, [5, 6, 7]) as b:
        b.sweep_path = "tiled"
        for e in (a, b):
            e.hot_start()
        for call in (lambda e: e.measured_sweeps(0.3, 1, 0), lambda e: e.measured_sweeps(0.3, 1, 1),
                     lambda e: e.measured_sweeps(0.5, 3, 1, "uniform")):
            assert np.array_equal(call(a), call(b))
        for e in (a, b):
            e.metropolis_sweeps(0.3, 1)
        assert a.sweep_path == "auto" and a.sweep_index == b.sweep_index == 5
        for c in range(3):
            assert np.array_equal(a.download(c), b.download(c))
        assert np.array_equal(a.accounting()[1], b.accounting()[1])
