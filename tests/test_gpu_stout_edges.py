"""Stout smearing where the exponential and the work split change regime:
odd and even extents, chains smaller than a tile, and Haar-random fields at
the largest rho, whose generators need scaling and squaring (1-norm above
1/2), beside smooth ones that need none.  Links within 2.5e-14 per level of
the oracle's dense Taylor series (rounding of about a hundred operations of
order one, doubled once per squaring), temporal links copied exactly."""
import numpy as np
import pytest

from test_gpu_su3 import rough_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("extents,rho,levels,haar", [
    ([3, 3, 3, 3], 0.25, 2, True),
    ([5, 5, 5, 7], 0.25, 1, True),
    ([4, 4, 4, 10], 0.2, 2, True),
    ([4, 4, 4, 4], 0.1, 3, False),
    ([6, 6, 6, 5], 0.01, 1, False),
])
def test_stout_levels_match_the_oracle(oracle, extents, rho, levels, haar):
    import ymgpu
    with ymgpu.Ensemble([extents], 6.0, 77, lift_reference_caps=True) as ens, ens.like() as dst:
        if haar:
            ens.hot_start()
        else:
            even = [e + e % 2 for e in extents]
            rough = rough_config(oracle, even, 3, 1).reshape(*even, 4, 3, 3)
            ens.upload(0, rough[:extents[0], :extents[1], :extents[2], :extents[3]].reshape(-1, 3, 3).copy())
        links = ens.download(0)
        ens.stout_smear_into(dst, rho, levels)
        got = dst.download(0)
    ref = oracle.spatial_stout_smear(extents, links, rho, levels)
    assert np.abs(got - ref).max() <= 2.5e-14 * levels
    assert np.array_equal(got.reshape(-1, 4, 3, 3)[:, 3], links.reshape(-1, 4, 3, 3)[:, 3])
