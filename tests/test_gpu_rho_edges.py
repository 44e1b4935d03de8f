"""The 2D density step's tiles with the absorbing edges: remainders of the
compute domain (ntaper 10: physical size + 20) modulo the tile around the 6
cells that a line needs, one to seven tiles across, against the oracle
bit for bit, traces and the whole padded field."""
import numpy as np
import pytest

import seismic_gb300 as sw
from tests.cases import case2d
from tests.test_gpu_rho import _desc, _rho

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nz,nx", [(44, 44), (54, 54), (53, 53), (44, 53), (118, 54), (180, 90),
                                   (108, 139), (45, 12)])
def test_rho_edges_bitexact(ctx, oracle, nz, nx):
    g, vel, sou, rec, w = case2d(nz=nz, nx=nx, nt=120, ntaper=10, seed=nz)
    sou = np.array([25.0, nx * 5.0, 0.0], np.float32)
    rho = _rho(vel.shape, 7)
    w = sw.rho_wavelet(w, g.lsinc)
    d = _desc(g, injection=sw.INJ_SINC, extraction=sw.EXT_SINC)
    out = []
    for c in (ctx, oracle):
        tr = np.zeros((rec.shape[0], g.nt), np.float32)
        fu = np.zeros(sw.padded_shape(g), np.float32)
        c.propagate(d, vel, sou, w, rec, tr, rho=rho, final_u2=fu)
        out.append((tr, fu))
    for x, y in zip(*out):
        assert np.abs(y).max() > 0
        np.testing.assert_array_equal(x, y)
