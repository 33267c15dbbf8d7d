"""A chain's plaquette and operators have the same bits alone, in a handle
with many small chains, and in a subset of that handle: the order of a sum
depends on the chain's own number of tiles or sites of a slice, not on the
handle's average.  The large chains lie past 1024 tiles and 1024 sites per
slice, where the width of a reduction changes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SMALL = [4, 4, 4, 4]


@pytest.mark.parametrize("large", [[20, 20, 20, 20], [18, 20, 20, 22]])
@pytest.mark.parametrize("kind", ["f64", "f32", "su2"])
def test_plaquette_alone_and_batched(large, kind):
    import ymgpu
    group = ymgpu.SU2 if kind == "su2" else ymgpu.SU3
    prec = ymgpu.F32_TWO_ROW if kind == "f32" else ymgpu.F64

    def make(exts, seeds):
        ens = ymgpu.Ensemble(exts, 2.3, seeds, group=group, precision=prec, lift_reference_caps=True)
        if kind == "su2":
            ens.markov_sweeps(1, 0)
        else:
            ens.hot_start()
        return ens

    with make([large], [41]) as alone, make([SMALL], [3]) as small, \
            make([SMALL] * 3 + [large] + [SMALL] * 4, [3, 4, 5, 41, 6, 7, 8, 9]) as batch:
        assert np.array_equal(alone.download(0), batch.download(3))
        got = batch.average_plaquette()
        assert got[3] == alone.average_plaquette()[0]
        assert got[0] == small.average_plaquette()[0]


def test_operators_alone_and_batched():
    import ymgpu
    large = [12, 12, 12, 6]                     # 1728 sites per slice
    exts, seeds = [SMALL] * 6 + [large] + [SMALL] * 6, list(range(30, 43))
    with ymgpu.Ensemble(exts, 6.0, seeds, lift_reference_caps=True) as batch, \
            ymgpu.Ensemble([large], 6.0, [36], lift_reference_caps=True) as alone, \
            ymgpu.Ensemble([SMALL], 6.0, [30]) as small:
        for ens in (batch, alone, small):
            ens.hot_start()
        got = batch.scalar_operator_basis()
        for mine, chain in ((alone, 6), (small, 0)):
            (plaq, rect), = mine.scalar_operator_basis()
            assert np.array_equal(got[chain][0], plaq) and np.array_equal(got[chain][1], rect)
        part = batch.subset([1, 6])
        try:
            batch.copy_subset_to([1, 6], part)
            for k, chain in enumerate((1, 6)):
                p, r = part.scalar_operator_basis()[k]
                assert np.array_equal(got[chain][0], p) and np.array_equal(got[chain][1], r)
        finally:
            part.close()
