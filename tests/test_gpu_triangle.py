"""Triangle smoothing of the FWI gradient against the oracle's triangle2 on
the unsmoothed gradient, bit for bit: radii of 1, of a few cells and of a
whole line, either axis or both."""
import numpy as np
import pytest

from tests.test_gpu_jobs import _fwi_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rz,rx,doz,dox", [(1, 1, 1, 1), (3, 5, 1, 1), (2, 9, 0, 1), (7, 1, 1, 0),
                                           (0, 0, 1, 1)])
def test_triangle_bitexact(ctx, oracle, rz, rx, doz, dox):
    d, vel, w, shots, _ = _fwi_case()
    n1, n2 = d.g.nz, d.g.nx
    rz, rx = rz or n1, rx or n2            # 0: as long as the line
    d.smooth_rect1, d.smooth_rect2 = rz, rx
    d.smooth_doz = d.smooth_dox = 0
    _, g0, _ = ctx.fwi_fct_gdt(d, vel, w, shots)
    d.smooth_doz, d.smooth_dox = doz, dox
    _, g1, _ = ctx.fwi_fct_gdt(d, vel, w, shots)
    ref = oracle.triangle2(g0, n1, n2, 1, rz, rx, 1, doz, dox, 0)
    assert np.abs(ref).max() > 0
    np.testing.assert_array_equal(g1, ref)
