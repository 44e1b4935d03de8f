"""The Born source on either stencil grid, through the propagator's own entry
point: traces and the final field equal the oracle's bit for bit (the adjoint
stencil with a Born source is no driver's, but the descriptor is accepted)."""
import numpy as np
import pytest

import seismic_gb300 as sw
from tests.cases import case2d, case3d

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tstep", [1, -1])
@pytest.mark.parametrize("fd", [sw.FD_FORWARD, sw.FD_ADJOINT])
@pytest.mark.parametrize("dim", [2, 3])
def test_born_source_every_grid(ctx, oracle, dim, fd, tstep):
    g, vel, sou, rec, w = (case2d(nz=45, nx=70, nt=120) if dim == 2 else
                           case3d(nz=14, nx=17, ny=13, nt=60))
    rng = np.random.default_rng(6)
    wave = rng.standard_normal((g.nt // g.snapi) * vel.size).astype(np.float32)
    refl = rng.standard_normal(vel.shape).astype(np.float32)
    d = sw.SwPropDesc()
    d.g = g
    d.tmin, d.tmax, d.tstep = (1, g.nt, 1) if tstep > 0 else (g.nt, 1, -1)
    d.fd_scheme, d.imaging, d.extraction = fd, sw.IMG_BORN, sw.EXT_SINC
    d.injection = sw.INJ_SINC
    G = [int(n) + 2 * g.ntaper + 8 for n in ((g.nz, g.nx) if dim == 2 else (g.nz, g.nx, g.ny))]
    out = []
    for f in (ctx.propagate, oracle.propagate):
        tr = np.zeros((len(rec), g.nt), np.float32)
        fu = np.zeros(int(np.prod(G)), np.float32)
        f(d, vel, sou, w[None, :], rec, tr, wave=wave.copy(), ref=refl, final_u2=fu)
        out.append((tr, fu))
    assert np.abs(out[1][0]).max() > 0 and np.abs(out[1][1]).max() > 0
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])
