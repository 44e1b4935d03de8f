"""The on-chip 2D propagation against the per-step kernels (use_graph = 0
launches every step by itself): the same bits for every form that the on-chip
rule accepts - grids around the smallest and uneven tiles, odd sizes, both
stencils, rigid boundary, mirrors, snapshot intervals, sinc lengths, several
shots of different size and record, and runs of several launches."""
import numpy as np
import pytest

import seismic_gb300 as sw
from tests.cases import case2d, model2d

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pair():
    a, b = sw.Context(0), sw.Context(0)
    b.set_tuning(use_graph=0)
    yield a, b
    a.close()
    b.close()


def _same(x, y):
    for p, q in zip(x if isinstance(x, tuple) else (x,), y if isinstance(y, tuple) else (y,)):
        assert np.abs(q).max() > 0
        np.testing.assert_array_equal(p, q)


FORMS = [  # nz, nx, ntaper, nt, snapi, lsinc, rigid, shot_type, rec_type
    (12, 12, 4, 60, 4, 7, 0, 0, 0),        # smallest padded grid of one tile
    (13, 131, 5, 90, 1, 5, 0, 0, 0),
    (61, 83, 10, 133, 3, 7, 0, 0, 0),
    (64, 96, 8, 100, 2, 3, 0, 0, 0),       # padded extents a multiple of 4 and not
    (119, 57, 12, 90, 5, 7, 1, 0, 0),
    (200, 330, 20, 120, 4, 7, 0, 0, 0),
    (333, 701, 17, 60, 4, 7, 1, 0, 0),
    (90, 150, 16, 150, 4, 7, 0, 1, 1),     # mirror source and receivers
    (40, 1900, 10, 60, 4, 9, 0, 0, 0),     # long and flat
    (701, 40, 10, 60, 4, 7, 0, 0, 0),
]


@pytest.mark.parametrize("form", FORMS)
def test_onchip_equals_per_step(pair, form):
    nz, nx, ntaper, nt, snapi, lsinc, rigid, shot_type, rec_type = form
    g, vel, sou, rec, w = case2d(nz, nx, nt, ntaper, seed=nz, snapi=snapi,
                                 nrec=max(3, nx // (1 + nz % 3)))
    g.lsinc, g.shot_type, g.rec_type = lsinc, shot_type, rec_type
    if shot_type:
        sou[0], rec[:, 0] = 31.3, 22.2     # mirrors inside the grid
    rng = np.random.default_rng(nx)
    data = rng.standard_normal((len(rec), nt)).astype(np.float32)
    ref = rng.standard_normal(vel.shape).astype(np.float32)
    out = []
    for c in pair:
        c.set_boundary(rigid)
        out.append((c.modeling(g, vel, sou, w, rec, final_u2=True), c.rtm(g, vel, sou, w, rec, data),
                    c.lsrtm(g, vel, sou, w, rec, data), c.born(g, vel, ref, sou, w, rec)))
        c.set_boundary(0)
    for x, y in zip(*out):
        _same(x, y)
    # The on-chip path takes these: far fewer launches than steps.
    assert pair[0].stats()["launches_total"] < pair[1].stats()["launches_total"] // 4


def test_onchip_jobs_and_gradient(pair):
    """Shots of different window and record in shared launches (RTM job), the
    FWI gradient with and without checkpoints."""
    nz, nx, d = 70, 260, 10.0
    vel = model2d(nz, nx, d, 9)
    g = sw.make_genpar(nz, nx, 1, dz=d, dx=d, dt=1.5e-3, nt=150, ntaper=9, lsinc=7, snapi=4)
    rng = np.random.default_rng(5)
    w = rng.standard_normal(150).astype(np.float32)
    shots = []
    for q in range(7):
        lo, hi = 3 + 11 * q, 120 + 19 * q
        rec = np.zeros(((hi - lo) // 2, 3), np.float32)
        rec[:, 0], rec[:, 1] = 12.0, np.linspace(lo, hi, len(rec)) * d
        nt = 150 - 13 * q
        shots.append({"sou": np.array([20.5, (lo + hi) * d / 2, 0.0], np.float32), "rec": rec,
                      "data": rng.standard_normal((len(rec), nt)).astype(np.float32)})
    out = []
    for c in pair:
        job = sw.RTMJob(c, g, vel, w, shots, aperture_x=80.0)
        job.run()
        r = job.result()
        m = job.model()
        job.close()
        fs = [dict(s, dobs=np.resize(s["data"], (len(s["rec"]), 150))) for s in shots]
        desc = sw.SwFwiDesc()
        desc.g, desc.illu_pow = g, 1.0
        grads = []
        for k in (0, 5):
            desc.checkpoint_snaps = k
            grads.append(c.fwi_fct_gdt(desc, vel, w, fs[:3]))
        out.append((r, m, grads))
    _same(out[0][0], out[1][0])
    for x, y in zip(out[0][1], out[1][1]):
        np.testing.assert_array_equal(x, y)
    for x, y in zip(out[0][2], out[1][2]):
        assert x[0] == y[0]
        _same(x[1:], y[1:])


def test_onchip_several_launches(pair):
    """A record that one launch's scratch does not hold: the state goes
    through the level buffers between launches."""
    g, vel, sou, rec, w = case2d(420, 610, 2300, 10, seed=4, dt=6e-4, snapi=1,
                                 nrec=200)   # dt: stable up to the model's 5.6 km/s
    rng = np.random.default_rng(8)
    data = rng.standard_normal((len(rec), g.nt)).astype(np.float32)
    _same(*(c.rtm(g, vel, sou, w, rec, data) for c in pair))
