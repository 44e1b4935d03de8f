"""3D receivers in the absorbing boundary.  The padding cells beside the outer
columns and planes of the compute domain belong to no line of the shared edge
launch, so receivers that gather there take the ordered lines; receivers beside
them, in the flat padding and on the domain's faces are taken too.  Every
record equals the oracle's bit for bit, whatever else the call returns."""
import numpy as np
import pytest

from tests.cases import case3d

pytestmark = pytest.mark.gpu


def _receivers(g, picks):
    """Receivers at compute-domain cells: counted from the near face, or from
    the far one if negative; None is the middle.  A third of a cell beside the
    grid point, so that every cell of the footprint counts."""
    n = (g.nz + 2 * g.ntaper, g.nx + 2 * g.ntaper, g.ny + 2 * g.ntaper)
    out = []
    for p in picks:
        q = [n[a] // 2 if v is None else v if v >= 0 else n[a] + v for a, v in enumerate(p)]
        out.append([(i - g.ntaper + 0.33) * d for i, d in zip(q, (g.dz, g.dx, g.dy))])
    return np.array(out, np.float32)


CORNERS = [[(1, 1, None)], [(1, None, 1)], [(None, 1, 1)], [(-3, -3, None)], [(-3, None, 1)],
           [(None, -3, 1)], [(1, 1, 1), (-3, -3, -3), (1, -3, 1)]]
FLAT = [[(1, None, None), (None, 1, None), (None, None, 1)],
        [(-3, None, None), (None, -3, None), (None, None, -3)],
        [(3, 3, 3), (-4, -4, -4)],                     # the first footprint within the domain
        [(1, 7, 7), (7, 1, 7), (1, 6, 7), (-3, -8, 9), (1, 8, 6)]]


@pytest.mark.parametrize("picks", CORNERS + FLAT)
def test_receivers_in_the_padding(ctx, oracle, picks):
    g, vel, sou, _, w = case3d(nz=16, nx=18, ny=14, nt=150, ntaper=9, seed=2)
    rec = _receivers(g, picks)
    ref, rfu = oracle.modeling(g, vel, sou, w, rec, final_u2=True)
    assert (np.abs(ref).max(axis=1) > 0).all()
    np.testing.assert_array_equal(ctx.modeling(g, vel, sou, w, rec), ref)
    data, fu = ctx.modeling(g, vel, sou, w, rec, final_u2=True)
    np.testing.assert_array_equal(data, ref)
    np.testing.assert_array_equal(fu, rfu)


@pytest.mark.parametrize("lsinc", [3, 5, 9])
def test_sinc_lengths_in_the_padding(ctx, oracle, lsinc):
    g, vel, sou, _, w = case3d(nz=16, nx=18, ny=14, nt=120, ntaper=9, seed=3)
    g.lsinc = lsinc
    lo = max(lsinc // 2 - 4, 0)            # the footprint reaches the padded grid's edge
    for a in range(lo, lsinc // 2 + 1):
        rec = _receivers(g, [(a, a, None), (a, None, a), (None, a, a), (-1 - a, -1 - a, -1 - a)])
        ref = oracle.modeling(g, vel, sou, w, rec)
        assert (np.abs(ref).max(axis=1) > 0).all()
        np.testing.assert_array_equal(ctx.modeling(g, vel, sou, w, rec), ref)


def test_born_receivers_in_the_padding(ctx, oracle):
    g, vel, sou, _, w = case3d(nz=16, nx=18, ny=14, nt=150, ntaper=9, seed=4)
    refl = np.random.default_rng(1).standard_normal(vel.shape).astype(np.float32)
    rec = _receivers(g, [(1, 1, None), (None, 1, 1), (-3, None, -3)])
    ref = oracle.born(g, vel, refl, sou, w, rec)
    assert (np.abs(ref).max(axis=1) > 0).all()
    np.testing.assert_array_equal(ctx.born(g, vel, refl, sou, w, rec), ref)
