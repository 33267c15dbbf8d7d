"""A lattice of 2^31 sites or more is refused as an allocation that cannot be
made, whatever it stores, before any table or device memory is asked for: the
kernels step between sites in 32 bits.  The reference's link cap, where it is
not lifted, still comes first."""
import ctypes as C

import pytest

ALLOCATION_FAILED, TOO_LARGE = 8, 7


def _create(extents, group, precision, lifted):
    from ymgpu._lib import EnsembleDesc, lib
    ext = (C.c_int64 * 4)(*extents)
    beta, seed = (C.c_double * 1)(2.3), (C.c_uint64 * 1)(1)
    desc = EnsembleDesc(group, precision, 1, ext, beta, seed, lifted, 0)
    handle = C.c_void_p()
    status = lib().ym_ensemble_create(C.byref(desc), C.byref(handle))
    assert not handle.value
    return status


@pytest.mark.parametrize("kind", ["su3", "su3_two_row", "su2"])
@pytest.mark.parametrize("extents", [[1024, 1024, 1024, 2], [2 ** 30, 2, 2, 2], [2 ** 15, 2 ** 15, 2 ** 15, 4]])
def test_2_31_sites_are_refused(kind, extents):
    import ymgpu
    group = ymgpu.SU2 if kind == "su2" else ymgpu.SU3
    precision = ymgpu.F32_TWO_ROW if kind == "su3_two_row" else ymgpu.F64
    assert _create(extents, group, precision, 1) == ALLOCATION_FAILED
    assert _create(extents, group, precision, 0) == TOO_LARGE
