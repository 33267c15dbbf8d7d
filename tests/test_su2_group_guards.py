"""The grouped SU(2) kernels give eight lanes to a link; the groups past the
end of a sub-sweep keep the first link's slot for their index arithmetic while
that link's own group may be storing to it, so they must not read it.  The
source's loads of the updated link are guarded, and sub-sweeps with idle
groups give the oracle's links."""
import os
import re

import numpy as np
import pytest

SU2 = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "yang-mills_b200", "csrc", "su2.cu")


@pytest.mark.parametrize("kernel", ["k_su2_heatbath_group", "k_su2_overrelax_group"])
def test_loads_of_the_updated_link_are_guarded(kernel):
    with open(SU2) as fh:
        text = fh.read()
    body = text[text.index(kernel + "("):]
    body = body[:body.index("\n}\n")]
    before_exit = body.split("if (!active) return;")[0]
    for line in before_exit.splitlines():
        if re.search(r"\bload_q_rw\(", line):
            assert re.search(r"\bactive\b", line), line


@pytest.mark.gpu
@pytest.mark.parametrize("extents", [[2, 2, 2, 2], [2, 2, 2, 6], [2, 2, 4, 10], [6, 6, 6, 10]])
def test_sub_sweeps_with_idle_groups_are_the_oracles(oracle, extents):
    import ymgpu
    from test_gpu_su2 import cb_overrelax
    rng = np.random.default_rng(17)
    start = rng.normal(size=(int(np.prod(extents)) * 4, 4))
    start /= np.sqrt((start * start).sum(1, keepdims=True))
    with ymgpu.Ensemble([extents], 2.3, 1, group=ymgpu.SU2, lift_reference_caps=True) as ens:
        ens.upload(0, start)
        start = ens.download(0)          # as the handle stores it
        ens.overrelaxation_sweeps(3)
        got = ens.download(0)
    for _ in range(3):
        cb_overrelax(oracle, extents, start)
    assert np.array_equal(got, start)
