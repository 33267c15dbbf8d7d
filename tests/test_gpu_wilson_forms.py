"""Wilson loops of handles whose tiles reach well past their chains' ends wait
in columns of shared memory, those of other handles are summed warp by warp as
they are made: a chain's loops have the same bits in both, and are the
oracle's plaquette mean at 1 x 1."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("extents", [[2, 2, 2, 2], [3, 3, 3, 3], [3, 3, 3, 5], [4, 4, 4, 3], [5, 5, 5, 5]])
def test_a_ragged_chain_alone_and_among_full_ones(oracle, extents):
    import ymgpu
    with ymgpu.Ensemble([extents], 6.0, [31], lift_reference_caps=True) as alone, \
            ymgpu.Ensemble([[8, 8, 8, 8]] * 2 + [extents], 6.0, [1, 2, 31], lift_reference_caps=True) as batch:
        alone.hot_start()
        batch.hot_start()
        links = alone.download(0)
        assert np.array_equal(links, batch.download(2))
        for rmax in range(1, 5):
            for tmax in range(1, 5):
                assert np.array_equal(alone.wilson_loops(rmax, tmax)[0], batch.wilson_loops(rmax, tmax)[2])
        plaq = float(alone.wilson_loops(1, 1)[0].reshape(-1, 4, 4)[:, 0, 0].mean())
    assert abs(plaq - oracle.su3_average_plaquette(extents, links)) <= 1e-12
