"""The launch that ends a measurement writes its row and advances the row and
sweep counters for every sweep since the last advance, of which at most 32
are outstanding.  Cadences of fewer, exactly 32 and more sweeps, with one
chain and several, from a sweep index that is not zero, against the same
sweeps made one call at a time: same links, same counter, and the series the
plaquettes those calls see (1e-12: another order of summation)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

START = 2 ** 40 + 3


def _compare(make, cadence, single, stride, n=2):
    with make() as a, make() as b:
        for ens in (a, b):
            ens.sweep_index = START
        got = cadence(a, n, stride)
        for row in range(n):
            for _ in range(stride):
                single(b)
            plaq = b.average_plaquette()
            assert np.all(np.abs(got[row] - plaq) <= 1e-12 * np.abs(plaq))
        assert a.sweep_index == b.sweep_index == START + n * stride
        cadence(a, 1, 0)                                  # a row without a sweep
        assert a.sweep_index == START + n * stride
        for c in range(a.n_chains):
            assert np.array_equal(a.download(c), b.download(c))


@pytest.mark.parametrize("chains", [1, 3])
@pytest.mark.parametrize("stride", [1, 31, 32, 33, 64])
@pytest.mark.parametrize("path", ["tiled", "resident"])
def test_su3_cadence(chains, stride, path):
    import ymgpu

    def make():
        ens = ymgpu.Ensemble([[4, 4, 4, 4]] * chains, 6.0, list(range(5, 5 + chains)))
        ens.sweep_path = path
        return ens
    _compare(make, lambda e, n, s: e.measured_sweeps(0.3, n, s, "ordered"),
             lambda e: e.metropolis_sweeps(0.3, 1, "ordered"), stride)


@pytest.mark.parametrize("chains", [1, 3])
@pytest.mark.parametrize("stride", [1, 32, 33])
def test_two_row_and_su2_cadences(chains, stride):
    import ymgpu
    seeds = list(range(5, 5 + chains))
    _compare(lambda: ymgpu.Ensemble([[4, 4, 4, 4]] * chains, 6.0, seeds, precision=ymgpu.F32_TWO_ROW),
             lambda e, n, s: e.measured_sweeps(0.3, n, s, "uniform"),
             lambda e: e.metropolis_sweeps(0.3, 1, "uniform"), stride)
    _compare(lambda: ymgpu.Ensemble([[4, 4, 4, 4]] * chains, 2.3, seeds, group=ymgpu.SU2),
             lambda e, n, s: e.su2_measured_sweeps(n, s, 1),
             lambda e: e.markov_sweeps(1, 1), stride)
