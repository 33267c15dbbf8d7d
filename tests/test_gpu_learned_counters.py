"""Learned sweeps and training count their sweeps on the host and advance the
device's sweep counter every 32 and at the end of a call: the links and the
counter of one call are those of the same sweeps made one call at a time, for
fewer, exactly 32 and more sweeps, from a sweep index that is not zero."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

START = 2 ** 40 + 3


def _handle(chains):
    import ymgpu
    ens = ymgpu.Ensemble([[4, 4, 4, 4]] * chains, 5.7, list(range(5, 5 + chains)), precision=ymgpu.F32_TWO_ROW)
    ens.hot_start()
    ens.sweep_index = START
    return ens


def _same(a, b, sweeps):
    assert a.sweep_index == b.sweep_index == START + sweeps
    for c in range(a.n_chains):
        assert np.array_equal(a.download(c), b.download(c))


@pytest.mark.parametrize("chains", [1, 3])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 65])
def test_learned_sweeps(chains, n):
    from ymgpu.learned import ProposalModel
    with _handle(chains) as a, _handle(chains) as b, ProposalModel(initial_scale=0.6) as model:
        model.sweeps(a, n)
        for _ in range(n):
            model.sweeps(b, 1)
        _same(a, b, n)
        # a cadence of that stride goes on from the counter
        got = model.measured_sweeps(a, 2, n)
        for row in range(2):
            model.sweeps(b, n)
            plaq = b.average_plaquette()
            assert np.all(np.abs(got[row] - plaq) <= 1e-12 * np.maximum(np.abs(plaq), 1.0))
        _same(a, b, 3 * n)


@pytest.mark.parametrize("steps,sweeps_per_step", [(1, 1), (8, 4), (33, 1), (5, 13)])
def test_training_counts_its_sweeps(steps, sweeps_per_step):
    from ymgpu.learned import ProposalModel
    with _handle(1) as a, _handle(1) as b, ProposalModel(initial_scale=0.6) as model:
        model.train(a, steps, sweeps_per_step, 0.3, 3e-3)
        for _ in range(steps * sweeps_per_step):
            b.metropolis_sweeps(0.3, 1, "uniform")
        _same(a, b, steps * sweeps_per_step)
