"""Reductions at the sizes where their block size changes: time slices of
fewer and more than 1024 sites (operators), chains of exactly 1024 site tiles
and more (plaquettes), odd extents and remainders of a block's four sites in
flight.  Means of at most 1e6 terms of order one whose partial sums are
exact to 1e-16 of their size: within 1e-12 of the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("extents", [[3, 3, 3, 5], [10, 10, 10, 3], [11, 11, 11, 3], [12, 12, 12, 4]])
def test_operator_slices(oracle, extents):
    import ymgpu
    with ymgpu.Ensemble([extents], 6.0, 5, lift_reference_caps=True) as ens:
        ens.hot_start()
        links = ens.download(0)
        (plaq, rect), = ens.scalar_operator_basis()
    for t in range(extents[3]):
        p, r, _, _ = oracle.scalar_a1pp_operator_basis(extents, links, t)
        assert abs(plaq[t] - p) <= 1e-12 and abs(rect[t] - r) <= 1e-12


@pytest.mark.parametrize("extents", [[16, 16, 16, 32], [16, 16, 18, 30], [15, 17, 23, 23]])
def test_plaquette_of_many_tiles(oracle, extents):
    import ymgpu
    with ymgpu.Ensemble([extents], 6.0, 5, lift_reference_caps=True) as ens:
        ens.hot_start()
        plaq = float(ens.average_plaquette()[0])
        loop = float(ens.wilson_loops(1, 1)[0].reshape(-1, 4, 4)[:, 0, 0].mean())
        links = ens.download(0)
    ref = oracle.su3_average_plaquette(extents, links)
    assert abs(plaq - ref) <= 1e-12
    assert abs(loop - ref) <= 1e-12
