"""The 3D chain of launches against the streaming kernel taken step by step:
the edges in one launch (with the corner cells formed by the lines that start
from them), the injection terms of the next step, the snapshots, and the
receiver samples of up to 4 steps together give the same bits, for grids
around the smallest sizes, boundaries too narrow for the shared launch, odd
extents, several sinc lengths and step counts that leave a remainder."""
import numpy as np
import pytest

import seismic_gb300 as sw
from tests.cases import case2d, case3d

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pair():
    a, b = sw.Context(0), sw.Context(0)
    b.set_tuning(step_kernel=1, use_graph=0)
    yield a, b
    a.close()
    b.close()


def _same(x, y):
    for p, q in zip(x if isinstance(x, tuple) else (x,), y if isinstance(y, tuple) else (y,)):
        assert np.abs(q).max() > 0
        np.testing.assert_array_equal(p, q)


FORMS = [  # nz, nx, ny, ntaper, nt, snapi, lsinc
    (12, 13, 12, 8, 41, 4, 7),
    (9, 33, 14, 9, 50, 3, 5),
    (12, 12, 13, 4, 43, 4, 7),        # narrow boundary: lines by themselves
    (47, 30, 21, 8, 62, 1, 7),
    (20, 70, 45, 12, 53, 5, 9),
    (33, 18, 90, 10, 47, 4, 7),
]


@pytest.mark.parametrize("form", FORMS)
def test_step3d_equals_streaming(pair, form):
    nz, nx, ny, ntaper, nt, snapi, lsinc = form
    g, vel, sou, rec, w = case3d(nz, nx, ny, nt, ntaper, seed=nx, snapi=snapi)
    g.lsinc = lsinc
    d = 10.0
    ends = [[z, x, y] for z in (0.0, (nz - 1) * d) for x in (0.0, (nx - 1) * d)
            for y in (0.0, (ny - 1) * d)]
    rec = np.concatenate([rec, np.array(ends, np.float32)]).astype(np.float32)
    rng = np.random.default_rng(ny)
    data = rng.standard_normal((len(rec), nt)).astype(np.float32)
    ref = rng.standard_normal(vel.shape).astype(np.float32)
    out = [(c.modeling(g, vel, sou, w, rec), c.modeling(g, vel, sou, w, rec, final_u2=True),
            c.rtm(g, vel, sou, w, rec, data), c.lsrtm(g, vel, sou, w, rec, data),
            c.born(g, vel, ref, sou, w, rec)) for c in pair]
    for x, y in zip(*out):
        _same(x, y)


@pytest.mark.parametrize("nt", [6, 50, 103])
def test_extraction_of_several_steps_2d(pair, nt):
    g, vel, sou, rec, w = case2d(41, 57, nt, 8, seed=3, snapi=3, nrec=11)
    ref = np.random.default_rng(5).standard_normal(vel.shape).astype(np.float32)
    x, y = (c.born(g, vel, ref, sou, w, rec) for c in pair)
    np.testing.assert_array_equal(x, y)
