"""SU(2) products on entries where the shared-reciprocal normalisation hands
over to the plain divisions: zeros, subnormals, tiny entries on both sides of
the 2^-300 limit, and products whose largest entry is far below the others'
ratio.  Overrelaxation must stay the oracle's bit for bit, on the grouped
kernels (small lattices) and the one-thread kernels, and the plaquette within
1e-12."""
import numpy as np
import pytest

from test_gpu_su2 import cb_overrelax

pytestmark = pytest.mark.gpu

EDGES = np.array([0.0, 5e-324, 1e-310, 2.0 ** -301, 2.0 ** -300, 2.0 ** -299 * 1.37, 1e-200, 1e-80, 1e-17,
                  2.0 ** -27, 0.3, 0.9])


def _links(oracle, extents, seed):
    rng = np.random.default_rng(seed)
    n = int(np.prod(extents)) * 4
    q = rng.choice(EDGES, size=(n, 4)) * rng.choice([-1.0, 1.0], size=(n, 4))
    q[np.arange(n), rng.integers(0, 4, n)] = rng.choice([-1.0, 1.0], n)
    return q / np.sqrt((q * q).sum(1, keepdims=True))


@pytest.mark.parametrize("extents", [[4, 4, 4, 4], [6, 4, 4, 10], [12, 12, 12, 18]])
def test_overrelaxation_on_edge_entries_is_the_oracles(oracle, extents):
    import ymgpu
    start = _links(oracle, extents, 11)
    with ymgpu.Ensemble([extents], 2.3, 1, group=ymgpu.SU2, lift_reference_caps=True) as ens:
        ens.upload(0, start)
        assert np.array_equal(ens.download(0), start)
        plaq = float(ens.average_plaquette()[0])
        ref_plaq = oracle.su2_average_plaquette(extents, start)
        assert abs(plaq - ref_plaq) <= 1e-12      # terms of order one
        ens.overrelaxation_sweeps(1)
        got = ens.download(0)
    ref = start.copy()
    cb_overrelax(oracle, extents, ref)
    assert np.array_equal(got, ref)


@pytest.mark.parametrize("extents", [[2, 2, 2, 2], [2, 4, 6, 10], [3, 5, 4, 7], [6, 6, 6, 10]])
def test_plaquette_of_few_and_many_chains_agrees_bitwise(oracle, extents):
    """A small handle measures with eight lanes per site and (one chain) its
    geometry as a launch parameter, a handle of many copies with one thread
    per site: same bits, within 1e-12 of the oracle; and a heat-bath and
    overrelaxation sweep of the copies too."""
    import ymgpu
    start = _links(oracle, extents, 5)
    copies = 1 + 40000 // int(np.prod(extents))
    even = all(e % 2 == 0 for e in extents)
    with ymgpu.Ensemble([extents], 2.3, 9, group=ymgpu.SU2, lift_reference_caps=True) as one, \
            ymgpu.Ensemble([extents] * copies, 2.3, 9, group=ymgpu.SU2, lift_reference_caps=True) as many:
        one.upload(0, start)
        for c in range(copies):
            many.upload(c, start)
        a, b = one.average_plaquette(), many.average_plaquette()
        assert np.all(b == a[0])
        assert abs(a[0] - oracle.su2_average_plaquette(extents, start)) <= 1e-12
        if even:
            for beta, seed in ((2.3, 9), (2.0, 10)):     # the second: a changed chain of the same handle
                for e in (one, many):
                    for c in range(e.n_chains):
                        e.set_chain(c, beta, seed)
                s1 = one.su2_measured_sweeps(2, 1, 1, sampler="kennedy-pendleton")
                s2 = many.su2_measured_sweeps(2, 1, 1, sampler="kennedy-pendleton")
                assert np.all(s2 == s1[:, :1])
            assert np.array_equal(one.download(0), many.download(copies - 1))
