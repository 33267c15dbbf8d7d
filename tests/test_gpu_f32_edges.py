"""Two-row binary32 sweeps at the edges of the tiles: lattices smaller than a
tile, partial last tiles, several uneven chains per launch, both generator
modes.  One sweep stays within the binary32 bars of the binary64 sweep from
the same field (at least 98 % of link entries within 1e-5: a link differs by
more only where a decision within rounding of the accept threshold flipped),
a chain's links do not depend on the chains that share its launches, and the
plaquette agrees with the binary64 plaquette of the same links to 1e-12 (both
are binary64 sums of the stored values)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EXTENTS = [[2, 2, 2, 2], [4, 4, 4, 6], [6, 6, 6, 10], [2, 4, 6, 8]]


@pytest.mark.parametrize("mode", ["ordered", "uniform"])
def test_two_row_sweep_edges(mode):
    import ymgpu
    seeds = [31 + i for i in range(len(EXTENTS))]
    with ymgpu.Ensemble(EXTENTS, 5.8, seeds) as f64, ymgpu.Ensemble(EXTENTS, 5.8, seeds) as view, \
            ymgpu.Ensemble(EXTENTS, 5.8, seeds, precision=ymgpu.F32_TWO_ROW) as f32:
        f64.hot_start()
        f64.metropolis_sweeps(1.0, 5)
        start = [f64.download(c) for c in range(len(EXTENTS))]
        f64.convert_to(f32)
        f32.sweep_index = f64.sweep_index
        first = f64.sweep_index
        f64.metropolis_sweeps(0.4, 1, mode)
        f32.metropolis_sweeps(0.4, 1, mode)
        batch = [f32.download(c) for c in range(len(EXTENTS))]
        for c in range(len(EXTENTS)):
            d = np.abs(batch[c] - f64.download(c)).max((1, 2))
            assert np.mean(d < 1e-5) >= 0.98
        f32.convert_to(view)
        assert np.allclose(f32.average_plaquette(), view.average_plaquette(), rtol=0, atol=1e-12)
    for c, ext in enumerate(EXTENTS):
        with ymgpu.Ensemble([ext], 5.8, seeds[c], precision=ymgpu.F32_TWO_ROW) as one:
            one.upload(0, start[c])
            one.sweep_index = first
            one.metropolis_sweeps(0.4, 1, mode)
            assert np.array_equal(one.download(0), batch[c])
