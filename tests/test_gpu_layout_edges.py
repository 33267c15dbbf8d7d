"""Host layout conversions at the edges of their 32-site blocks: fewer sites
than a block, a partial last block, odd extents (lexicographic storage) and a
chain that is not the first of its handle.  Upload then download returns the
same bytes in binary64; in two-row storage the first two rows come back
rounded once and the third is their conjugate cross product."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("extents", [[2, 2, 2, 2], [2, 2, 2, 3], [3, 3, 3, 3], [2, 3, 5, 7], [4, 4, 4, 6], [5, 5, 6, 8]])
def test_upload_download_round_trip(oracle, extents):
    import ymgpu
    other = [2, 2, 2, 4]
    with ymgpu.Ensemble([other, extents], 6.0, [5, 6]) as src, ymgpu.Ensemble([other, extents], 6.0, [1, 2]) as dst, \
            ymgpu.Ensemble([other, extents], 6.0, [1, 2], precision=ymgpu.F32_TWO_ROW) as two:
        src.hot_start()
        links = src.download(1)
        assert abs(links[0] @ links[0].conj().T - np.eye(3)).max() < 1e-13
        for x, mu in (((0, 0, 0, 0), 0), (tuple(e - 1 for e in extents), 3)):
            lex = ((x[0] * extents[1] + x[1]) * extents[2] + x[2]) * extents[3] + x[3]
            assert np.array_equal(src.get_link(1, x, mu), links[lex * 4 + mu])
        dst.upload(1, links)
        assert np.array_equal(dst.download(1), links)
        assert np.array_equal(dst.download(0), np.broadcast_to(np.eye(3), dst.download(0).shape))
        two.upload(1, links)
        back = two.download(1)
        rows = links[:, :2].astype(np.complex64).astype(np.complex128)
        assert np.array_equal(back[:, :2], rows)
        assert np.abs(back[:, 2] - np.cross(rows[:, 0], rows[:, 1]).conj()).max() < 1e-15
