"""Chain-resident sweeps of handles of different chain sizes from two host
threads at once.  The kernel's shared-memory limit is the device's, not the
handle's: a small handle's launch must not lower it under a larger one's.
Every call succeeds and the links are those of the same calls one handle
after the other."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CALLS = 1500


@pytest.mark.parametrize("sizes", [([4, 4, 4, 4], [2, 2, 2, 2]), ([4, 4, 4, 6], [2, 2, 8, 10])])
@pytest.mark.parametrize("mode", ["ordered", "uniform"])
def test_handles_of_two_sizes_sweep_concurrently(sizes, mode):
    import ymgpu

    def make(ext):
        ens = ymgpu.Ensemble([ext], 6.0, 23)
        ens.sweep_path = "resident"
        return ens

    expected = []
    for ext in sizes:
        with make(ext) as ens:
            for _ in range(CALLS):
                ens.metropolis_sweeps(0.3, 1, mode)
            expected.append(ens.download(0))

    handles = [make(ext) for ext in sizes]
    start, errors = threading.Barrier(2), []

    def drive(ens):
        start.wait()
        try:
            for _ in range(CALLS):
                ens.metropolis_sweeps(0.3, 1, mode)
        except Exception as exc:   # reported below, in the test's own thread
            errors.append(exc)

    try:
        threads = [threading.Thread(target=drive, args=(ens,)) for ens in handles]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not errors, errors
        for ens, want in zip(handles, expected):
            assert np.array_equal(ens.download(0), want)
    finally:
        for ens in handles:
            ens.close()
