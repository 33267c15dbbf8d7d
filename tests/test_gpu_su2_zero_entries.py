"""SU(2) products with entries that are exactly zero, of both signs: they are
normalised by the shared reciprocals and given their sign back, where entries
that are tiny too still take the plain divisions.  Links after overrelaxation
are the oracle's to the last bit, the signs of zeros included, on the grouped
kernels and the one-thread kernels."""
import numpy as np
import pytest

from test_gpu_su2 import cb_overrelax

pytestmark = pytest.mark.gpu


def _identity(n, rng):
    q = np.zeros((n, 4))
    q[:, 0] = 1.0
    return q


def _axes(n, rng):          # a signed unit entry among signed zeros
    q = np.zeros((n, 4)) * rng.choice([-1.0, 1.0], (n, 4))
    q[np.arange(n), rng.integers(0, 4, n)] = rng.choice([-1.0, 1.0], n)
    return q


def _planes(n, rng):        # two or three entries, the others signed zeros
    q = rng.normal(size=(n, 4)) * rng.choice([0.0, 1.0], (n, 4))
    q[np.arange(n), rng.integers(0, 4, n)] = 1.0
    return q / np.sqrt((q * q).sum(1, keepdims=True))


def _tiny(n, rng):          # zeros beside entries past the reciprocals' range
    q = rng.choice([0.0, 5e-324, 2.0 ** -301, 2.0 ** -300, 1e-9], (n, 4)) * rng.choice([-1.0, 1.0], (n, 4))
    q[np.arange(n), rng.integers(0, 4, n)] = 1.0
    return q


@pytest.mark.parametrize("links", [_identity, _axes, _planes, _tiny])
@pytest.mark.parametrize("extents", [[2, 2, 2, 2], [6, 4, 4, 10], [12, 12, 12, 18]])
def test_overrelaxation_keeps_zeros_and_their_signs(oracle, links, extents):
    import ymgpu
    start = links(int(np.prod(extents)) * 4, np.random.default_rng(3))
    with ymgpu.Ensemble([extents], 2.3, 1, group=ymgpu.SU2, lift_reference_caps=True) as ens:
        ens.upload(0, start)
        assert np.array_equal(ens.download(0).view(np.uint64), start.view(np.uint64))
        ens.overrelaxation_sweeps(2)
        got = ens.download(0)
    for _ in range(2):
        cb_overrelax(oracle, extents, start)
    assert np.array_equal(got.view(np.uint64), start.view(np.uint64))
