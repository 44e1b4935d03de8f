"""The per-step 2D tile kernel in the form that large grids take (step_kernel
5: captured graphs, programmatic launches, receiver samples of up to 4 steps
together) on small and odd grids, against the oracle bit for bit: records of
every remainder, each imaging condition, batches of unequal shots with fewer
and with more tiles than resident CTAs, and FWI gradients."""
import numpy as np
import pytest

import seismic_gb300 as sw
from tests.cases import case2d, model2d
from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tiles():
    c = sw.Context(0)
    c.set_tuning(step_kernel=5)
    yield c
    c.close()


@pytest.fixture()
def steps(tiles):
    """Fails unless every step of the test was launched by itself."""
    tiles.reset_stats()
    yield
    s = tiles.stats()
    assert s["launches_total"] > s["launches_step"] > 0


@pytest.mark.parametrize("nz,nx", [(41, 57), (9, 200), (130, 45)])
@pytest.mark.parametrize("nt", [6, 33, 50, 103])
def test_records(tiles, steps, oracle, nz, nx, nt):
    g, vel, sou, rec, w = case2d(nz, nx, nt, 8, seed=3, snapi=3, nrec=11)
    rec[:, 0] = 50.0 + 2.3      # within the first steps' reach of the source
    ref = np.random.default_rng(5).standard_normal(vel.shape).astype(np.float32)
    d = oracle.modeling(g, vel, sou, w, rec)
    assert np.abs(d).max() > 0
    np.testing.assert_array_equal(tiles.modeling(g, vel, sou, w, rec), d)
    np.testing.assert_array_equal(tiles.born(g, vel, ref, sou, w, rec),
                                  oracle.born(g, vel, ref, sou, w, rec))


@pytest.mark.parametrize("fd", [sw.FD_FORWARD, sw.FD_ADJOINT])
@pytest.mark.parametrize("imaging", [sw.IMG_RTM, sw.IMG_LSRTM, sw.IMG_AFWI])
@pytest.mark.parametrize("nt,snapi", [(120, 4), (67, 1), (50, 3)])
def test_imaging(tiles, steps, oracle, fd, imaging, nt, snapi):
    g, vel, _, rec, _ = case2d(nz=61, nx=83, nt=nt, ntaper=9, snapi=snapi)
    rng = np.random.default_rng(7)
    wave = rng.standard_normal((nt // snapi) * vel.size).astype(np.float32)
    adj = rng.standard_normal((len(rec), nt)).astype(np.float32)
    d = sw.SwPropDesc()
    d.g, d.tmin, d.tmax, d.tstep = g, nt, 1, -1
    d.fd_scheme, d.imaging = fd, imaging
    d.injection = {sw.IMG_RTM: sw.INJ_SINC, sw.IMG_LSRTM: sw.INJ_LSRTM_SINC,
                   sw.IMG_AFWI: sw.INJ_SIMPLE}[imaging]
    out = []
    for f in (tiles.propagate, oracle.propagate):
        im, il = np.zeros(vel.size, np.float32), np.zeros(vel.size, np.float32)
        f(d, vel, rec, adj, wave=wave.copy(), image=im, illum=il)
        out.append((im, il))
    assert np.abs(out[1][0]).max() > 0
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])


def _shots(nz, nx, sizes, nt):
    """Shots with windows of the given numbers of columns and unequal records."""
    d = 10.0
    rng = np.random.default_rng(nz)
    g = sw.make_genpar(nz, nx, 1, dz=d, dx=d, dt=1.2e-3, nt=nt, ntaper=9, lsinc=7, snapi=4)
    w = rng.standard_normal(nt).astype(np.float32)
    shots = []
    for q, n in enumerate(sizes):
        lo = (37 * q) % (nx - n)
        rec = np.zeros((n // 2, 3), np.float32)
        rec[:, 0], rec[:, 1] = 12.0, np.linspace(lo, lo + n, len(rec)) * d
        data = rng.standard_normal((len(rec), nt - 7 * q)).astype(np.float32)
        shots.append({"sou": np.array([20.5, (lo + n / 2) * d, 0.0], np.float32), "rec": rec,
                      "data": data})
    return g, model2d(nz, nx, d, nz), w, shots


@pytest.mark.parametrize("nz,nx,sizes", [
    (45, 260, (90, 141, 33, 200)),        # fewer tiles than CTAs
    (333, 1300, (1207, 640, 901)),        # several rounds, the last one partial
    (63, 4100, (4001, 333)),              # every tile has edge lines
])
def test_batches_of_unequal_shots(tiles, steps, oracle, nz, nx, sizes):
    g, vel, w, shots = _shots(nz, nx, sizes, 70)
    job = sw.RTMJob(tiles, g, vel, w, shots)
    job.set_batch(len(shots))
    job.run()
    im, il, nm = job.result()
    data = job.model()
    job.close()
    rim, ril, rnm = oracle.rtm_job(g, vel, w, shots)
    assert np.abs(rim).max() > 0
    np.testing.assert_array_equal(im, rim)
    np.testing.assert_array_equal(il, ril)
    assert rel_l2(nm, rnm) < 1e-6          # one FP64 sum in another order
    for s, d in zip(shots, data):          # the shots by themselves, one step per launch
        one = sw.RTMJob(tiles, g, vel, w, [s])
        tiles.set_tuning(use_graph=0)
        np.testing.assert_array_equal(one.model()[0], d)
        tiles.set_tuning(use_graph=1)
        one.close()
        assert np.abs(d).max() > 0


@pytest.mark.parametrize("checkpoint_snaps", [0, 5])
def test_fwi_gradient(tiles, steps, oracle, checkpoint_snaps):
    g, vel, w, shots = _shots(70, 260, (120, 161, 90), 150)
    for s in shots:
        s["dobs"] = np.resize(s.pop("data"), (len(s["rec"]), g.nt))
    desc = sw.SwFwiDesc()
    desc.g, desc.illu_pow, desc.checkpoint_snaps = g, 1.0, checkpoint_snaps
    a = tiles.fwi_fct_gdt(desc, vel, w, shots)
    b = oracle.fwi_fct_gdt(desc, vel, w, shots)
    assert abs(a[0] - b[0]) <= 1e-12 * abs(b[0])
    assert np.abs(b[1]).max() > 0
    for x, y in zip(a[1:], b[1:]):
        assert rel_l2(x, y) < 1e-6         # the misfit's and the illumination's FP64 sums
