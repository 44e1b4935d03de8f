"""What the host code decides for a call, on the CPU (tests/fakecuda.py)."""
import contextlib
import itertools

import numpy as np
import pytest

import seismic_gb300 as sw
from seismic_gb300 import autotune
from tests.cases import case2d, case3d
from tests.fakecuda import Fake


@pytest.fixture()
def fake():
    f = Fake()
    f.reset()
    return f


def _edge_cells(n, shared):
    """Padded cells (4 around n[0] x n[1] x n[2]) that the 3D edge lines write:
    all z, x and y lines, or those that the shared launch keeps."""
    out = np.zeros([m + 8 for m in n], bool)
    ends = [list(range(0, 8)) + list(range(m, m + 8)) for m in n]    # 8 cells of a line
    dom = [range(4, m + 4) for m in n]
    inner = [range(8, m) for m in n]
    z = (inner[1], inner[2]) if shared else (dom[1], dom[2])
    x = (dom[0], inner[2]) if shared else (dom[0], dom[2])
    out[np.ix_(ends[0], *z)] = True
    out[np.ix_(x[0], ends[1], x[1])] = True
    out[np.ix_(dom[0], dom[1], ends[2])] = True
    return out


@pytest.mark.parametrize("lsinc", [3, 7, 15])
def test_receivers_beside_left_out_edge_cells(fake, lsinc):
    """Every receiver whose footprint meets a padding cell that the shared 3D
    edge launch leaves out takes the ordered lines; others mostly do not."""
    g, vel, sou, _, w = case3d(nz=4, nx=5, ny=3, nt=2, ntaper=8)
    g.lsinc = lsinc
    n = (g.nz + 16, g.nx + 16, g.ny + 16)
    missing = _edge_cells(n, False) & ~_edge_cells(n, True)
    assert missing.any()
    h = lsinc // 2
    picks = [sorted({h, h + 1, h + 3, 7, 8, m // 2 + 4, m - 1, m, m + 7 - h - 1, m + 7 - h}
                    & set(range(h, m + 8 - h))) for m in n]
    shared = 0
    with fake.context() as c:
        for p in itertools.product(*picks):
            rec = np.array([[(q - 4 - g.ntaper) * 10.0 for q in p]], np.float32)
            fake.reset()
            c.modeling(g, vel, sou, w, rec)
            ordered = bool(fake.kernels("k_bhiggz"))
            box = tuple(slice(q - h, q + h + 1) for q in p)
            assert ordered or not missing[box].any(), p
            shared += not ordered
    assert shared > 0


def test_onchip_epochs_do_not_wrap(fake):
    """A run of several on-chip launches that starts anywhere near the end of
    the 32-bit epochs never finds a packet of its own epochs in the inbox."""
    g, vel, sou, rec, w = case2d(nz=150, nx=200, nt=260, snapi=1)
    data = np.zeros((len(rec), g.nt), np.float32)
    fake.reset(70 << 20)      # scratch for about 50 steps per launch
    with fake.context() as c:
        c.rtm(g, vel, sou, w, rec, data)
        n = len(fake.kernels("k_onchip2d"))
        first = fake.lib.fake_epoch(c.h)
        c.rtm(g, vel, sou, w, rec, data)
        used = fake.lib.fake_epoch(c.h) - first
        assert n > 3 and used > 2 * g.nt
        for left in [*range(0, 12), *range(used - 12, used + 3), 70, 71, 72, 261, 262, 263]:
            fake.lib.fake_set_epoch(c.h, 2 ** 32 - 1 - left)
            c.rtm(g, vel, sou, w, rec, data)
            assert fake.lib.fake_stale() == 0, left


def test_onchip_inbox_after_a_refused_allocation(fake):
    """Whichever allocation of a call is refused, the next call does not take
    what its memory held before for packets."""
    small = case2d(nz=60, nx=80, nt=40)
    g, vel, sou, rec, w = case2d(nz=200, nx=330, nt=90)
    for k in range(40):
        fake.reset()
        with fake.context() as c:
            c.modeling(*small[:3], small[4], small[3])
            n = len(fake.kernels("k_onchip2d"))
            fake.lib.fake_fail_alloc(k)
            try:
                c.modeling(g, vel, sou, w, rec)
            except sw.SwaveError as e:
                assert e.code == sw.SW_OOM_ADMISSION
            fake.lib.fake_fail_alloc(-1)
            c.modeling(g, vel, sou, w, rec)
            assert len(fake.kernels("k_onchip2d")) > n
            assert fake.lib.fake_stale() == 0, k


CUDA_ERROR_COOPERATIVE_LAUNCH_TOO_LARGE, CUDA_ERROR_LAUNCH_FAILURE = 720, 719


@pytest.mark.parametrize("how", ["residency", "launch"])
def test_onchip_refused_by_the_device(fake, how):
    """Where the CTAs of an on-chip launch are not all resident, or the device
    does not take the launch, the call runs through the per-step kernels;
    shots small enough for the smaller residency stay on the chip, and other
    errors are returned."""
    g, vel, sou, rec, w = case2d(nz=300, nx=600, nt=60)
    data = np.zeros((len(rec), g.nt), np.float32)
    small = case2d(nz=60, nx=80, nt=40)
    with fake.context() as c:
        c.rtm(g, vel, sou, w, rec, data)
        assert fake.kernels("k_onchip2d") and not fake.kernels("k_bstep2d_t")
    fake.reset()
    if how == "residency":
        fake.lib.fake_blocks_per_sm(1)
    else:
        fake.lib.fake_coop_error(CUDA_ERROR_COOPERATIVE_LAUNCH_TOO_LARGE)
    with fake.context() as c:
        c.rtm(g, vel, sou, w, rec, data)
        assert not fake.kernels("k_onchip2d") and fake.kernels("k_bstep2d_t")
        c.modeling(*small[:3], small[4], small[3])
        assert bool(fake.kernels("k_onchip2d")) == (how == "residency")
    if how == "launch":
        fake.lib.fake_coop_error(CUDA_ERROR_LAUNCH_FAILURE)
        with fake.context() as c, pytest.raises(sw.SwaveError) as e:
            c.rtm(g, vel, sou, w, rec, data)
        assert e.value.code == sw.SW_CUDA_ERR


@pytest.mark.parametrize("ntr,nt", [(1, 2), (1, 2_097_153), (3, 2_200_000), (2_097_185, 3)])
def test_bandpass_takes_every_size(fake, ntr, nt):
    with fake.context() as c:
        c.bandpass(np.ones((ntr, nt), np.float32), 2e-3, flo=5.0, fhi=90.0)
    assert len(fake.kernels("k_bp_pad")) == len(fake.kernels("k_bp_cut")) == 1


def _ok(call):
    try:
        call()
        return True
    except sw.SwaveError as e:
        assert e.code == sw.SW_OOM_ADMISSION, e
        return False


def _job(c, g, vel, sou, rec, w, data):
    job = sw.RTMJob(c, g, vel, w, [{"sou": sou, "rec": rec, "data": data}] * 2)
    try:
        job.run()
    finally:
        job.close()


LATER = {   # what runs on a context that has run a 2D shot on the chip
    "nothing": lambda c: None,
    "3d": lambda c: c.modeling(*C3D),
    "network": lambda c: _network(c),
    "job": lambda c: _job(c),
}
C2D = case2d(nz=160, nx=240, nt=60, nrec=240)
C3D = [case3d(nz=60, nx=70, ny=64, nt=4)[q] for q in (0, 1, 2, 4, 3)]


def _network(c):
    with contextlib.closing(sw.CNN(c, [2, 16, 1])) as n:
        n.forward(np.ones((2, 900, 300), np.float32))


def _job(c):
    g, vel, sou, rec, w = C2D
    d = np.zeros((len(rec), g.nt), np.float32)
    shots = [{"sou": sou, "rec": rec, "data": d}] * 2
    with contextlib.closing(sw.RTMJob(c, g, vel, w, shots)) as job:
        job.run()


@pytest.mark.parametrize("later", LATER)
def test_onchip_buffers_make_room(fake, later):
    """What fits into the device's memory with the per-step kernels fits with
    the on-chip path too: a shot by itself, and calls after one whose buffers
    the context still holds."""
    g, vel, sou, rec, w = C2D
    seen = set()
    for quarter in range(4, 600):
        ok = []
        for graph in (0, 1):                 # 0: the per-step kernels
            fake.reset(quarter << 18)
            with fake.context() as c:
                c.set_tuning(use_graph=graph)
                try:
                    c.rtm(g, vel, sou, w, rec, np.zeros((len(rec), g.nt), np.float32))
                    LATER[later](c)
                    ok.append(True)
                except sw.SwaveError as e:
                    assert e.code == sw.SW_OOM_ADMISSION or "cnn create" in str(e), e
                    ok.append(False)
        assert ok[1] or not ok[0], quarter
        seen.add(tuple(ok))
        if ok == [True, True] and fake.kernels("k_onchip2d"):
            break
    assert (False, False) in seen and (True, True) in seen


def test_profiled_bytes_are_of_the_timed_kernel(fake):
    """With profiling on, the bytes of an on-chip migration are those of the
    steps and the saved snapshots; imaging runs in a kernel that is not timed."""
    g, vel, sou, rec, w = case2d(nz=60, nx=80, nt=60)
    data = np.zeros((len(rec), g.nt), np.float32)
    pts = (g.nz + 2 * g.ntaper) * (g.nx + 2 * g.ntaper)
    steps, saved = 2 * g.nt * pts * 24, (g.nt // g.snapi) * vel.size * 4
    with fake.context() as c:
        c.set_profiling(True)
        c.rtm(g, vel, sou, w, rec, data)
        st = c.stats()
        assert fake.kernels("k_oc_image") and st["step_kernel_timed"] == 2 * g.nt
        assert st["step_bytes"] == steps + saved


def test_step_kernel_5_stays_off_the_chip(fake):
    """step_kernel 5 is the per-step tile kernel in the form that large grids
    take: a captured graph, receiver samples of 4 steps per launch."""
    g, vel, sou, rec, w = case2d(nz=60, nx=80, nt=60)
    with fake.context() as c:
        assert c.tuning()["step_kernel"] == 2          # the default: on the chip
        c.modeling(g, vel, sou, w, rec)
        assert fake.kernels("k_onchip2d") and not fake.kernels("k_bstep2d_t")
        fake.reset()
        c.set_tuning(step_kernel=5)
        assert c.tuning()["step_kernel"] == 5
        c.modeling(g, vel, sou, w, rec)
        assert fake.kernels("k_bstep2d_t") and not fake.kernels("k_onchip2d")
        assert len(fake.kernels("graph")) == 4
        assert {k[1][1] for k in fake.kernels("k_bextract")} == {4}
        fake.reset()
        c.set_tuning(graph_chunk=7)                     # another setting keeps it
        c.modeling(g, vel, sou, w, rec)
        assert not fake.kernels("k_onchip2d")
        assert {k[1][1] for k in fake.kernels("k_bextract")} == {4, 3}
        fake.reset()
        c.set_tuning(step_kernel=2)
        c.modeling(g, vel, sou, w, rec)
        assert fake.kernels("k_onchip2d")
        for bad in (-1, 6):
            with pytest.raises(sw.SwaveError):
                c.set_tuning(step_kernel=bad)
        g3, vel3, sou3, rec3, w3 = case3d(nt=4)
        for k in (2, 5):
            fake.reset()
            c.set_tuning(step_kernel=k)
            c.modeling(g3, vel3, sou3, w3, rec3)
            assert fake.kernels("k_bstep3d_t")


def test_tuning_cached_for_other_kernels_is_not_taken(fake, tmp_path):
    """A cache written before the present set of step kernels (its keys name no
    set) neither keeps shots off the chip nor fixes the shots per launch."""
    g, vel, sou, rec, w = case2d(nz=60, nx=80, nt=40)
    shots = [{"sou": sou, "rec": rec, "data": np.zeros((len(rec), g.nt), np.float32)}] * 2
    path = str(tmp_path / "tuning.json")
    n1p, n2p = g.nz + 2 * g.ntaper + 8, g.nx + 2 * g.ntaper + 8
    key = autotune.cache_key("dev", n1p, n2p, 1, 2)
    old = {"step_kernel": 3, "tile_z": 64, "tile_x": 64, "tile_y": 32, "graph_chunk": 16,
           "use_graph": 1}
    autotune.save_cache({key: {"tuning": old}, key + "|batch": {"batch": 77}}, path)
    with fake.context() as c:
        got = autotune.tune_rtm(c, g, vel, w, shots, steps=20, batch="auto", cache_path=path,
                                device_name="dev")
        assert got["batch"] in (1, 2) and got["tried"] == len(autotune.candidates(True))
        again = autotune.tune_rtm(c, g, vel, w, shots, steps=20, batch="auto", cache_path=path,
                                  device_name="dev")
        assert again == got                             # its own entries are


@pytest.mark.parametrize("nz,nx,ny,ok", [(1, 20, 1, False), (20, 1, 1, False), (2, 2, 1, True),
                                         (9, 1, 8, False), (1, 9, 8, False), (9, 9, 1, True)])
def test_density_imaging_of_a_single_row_or_column_is_refused(fake, nz, nx, ny, ok):
    """The differences of SW_IMG_AFWI_RHO on one row or column would start
    before the snapshots' memory."""
    g = sw.make_genpar(nz, nx, ny, dz=10.0, dx=10.0, dy=10.0, dt=1e-3, nt=12, ntaper=10,
                       twoD=ny == 1)
    vel = np.full((ny, nx, nz), 2000.0, np.float32)
    z = lambda: np.zeros(vel.size, np.float32)
    d = sw.SwPropDesc()
    d.g, d.tmin, d.tmax, d.tstep, d.imaging = g, g.nt, 1, -1, sw.IMG_AFWI_RHO
    with fake.context() as c:
        call = lambda: c.propagate(d, vel, wave=np.zeros(3 * vel.size, np.float32), image=z(),
                                   illum=z(), image2=z(), rho=vel)
        if ok:
            call()
        else:
            with pytest.raises(sw.SwaveError) as e:
                call()
            assert e.value.code == sw.SW_BAD_PARAM
            assert not fake.kernels("k_brho") and not fake.kernels("k_bstep")
