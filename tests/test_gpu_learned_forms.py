"""Learned sub-sweeps run their hits in registers on handles of at most two
tiles per SM, or of more than four and at most five, and on rows in shared
memory otherwise: a chain's links and accept counts are the same in both, at
those sizes, just past them and far past them, with ragged last tiles."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sweep(extents, copies, n=2):
    import ymgpu
    from ymgpu.learned import ProposalModel
    # the chain under test first; the others fill the handle up
    seeds = [77] + list(range(1000, 1000 + copies - 1))
    with ymgpu.Ensemble([extents] * copies, 5.9, seeds, precision=ymgpu.F32_TWO_ROW,
                        lift_reference_caps=True) as ens, ProposalModel(initial_scale=1.1) as model:
        ens.hot_start()
        model.sweeps(ens, n)
        return ens.download(0), [int(v[0]) for v in ens.accounting()]


@pytest.mark.parametrize("extents", [[4, 4, 4, 4], [4, 4, 4, 6], [6, 6, 6, 10]])
def test_a_chain_is_the_same_in_both_forms(extents):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    tiles = -(-(int(np.prod(extents)) // 2) // 128)
    links, accepted = _sweep(extents, 1)
    for full in (2, 4, 5, 8):
        for copies in (full * sms // tiles, full * sms // tiles + 1):
            got, count = _sweep(extents, copies)
            assert np.array_equal(got, links)
            assert count == accepted
