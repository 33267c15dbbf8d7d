"""The persistent ordered-hit sub-sweep at the edges of its work split.

Two CTAs per SM walk the work items (128 sites each), so the cases are fewer
items than CTAs, exactly one pass, a second pass that only some CTAs take,
items with idle threads, several chains per launch and more than one sweep;
both rotation lengths (half width <= 0.3 and above).  Links and accept counts
must be the oracle's bit for bit, and the plaquette the sweep measures must
agree with the oracle's to 1e-12.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MASTER = 0x2C02198105010002


@pytest.mark.parametrize("extents,chains,angle", [
    ([2, 2, 2, 2], 1, 0.3),          # eight live threads
    ([4, 4, 4, 6], 3, 0.35),         # 2 items per chain, the second half empty
    ([16, 16, 16, 20], 1, 0.3),      # 320 items: a partial second pass on 148 SMs
    ([6, 6, 6, 10], 40, 0.35),       # 360 items of 40 chains, every ninth partial
])
def test_ring_sweep_is_the_oracles(oracle, extents, chains, angle):
    import ymgpu
    seeds = [oracle.derive_su3_chain_seed(MASTER, i) for i in range(chains)]
    with ymgpu.Ensemble([extents] * chains, 5.9, seeds, lift_reference_caps=True) as ens:
        ens.sweep_path = "tiled"
        ens.hot_start()
        start = [ens.download(c) for c in range(chains)]
        ens.metropolis_sweeps(angle, 1)
        series = ens.measured_sweeps(angle, 1)
        _, accepts = ens.accounting()
        for c in range(chains):
            ref = start[c].copy()
            acc = sum(oracle.su3_cb_sweep(extents, ref, 5.9, angle, seeds[c], k)[1] for k in range(2))
            assert np.array_equal(ens.download(c), ref)
            assert int(accepts[c]) == acc
            plaq = oracle.su3_average_plaquette(extents, ref)
            assert abs(series[0, c] - plaq) <= 1e-12 * abs(plaq)
