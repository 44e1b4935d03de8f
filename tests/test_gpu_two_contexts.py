"""Contexts of several threads on one device at the same time: on-chip launches
(whose CTAs wait for one another's packets) beside each other and beside 3D
steps and network passes give the results they give alone."""
import threading

import numpy as np
import pytest

import seismic_gb300 as sw
from tests.cases import case2d, case3d

pytestmark = pytest.mark.gpu


def _work():
    """Calls and their names; each takes a context and returns arrays."""
    out = {}
    for q, (nz, nx, nt) in enumerate(((60, 80, 300), (201, 401, 250), (420, 610, 120))):
        g, vel, sou, rec, w = case2d(nz, nx, nt, seed=q, dt=1e-3)
        data = np.random.default_rng(q).standard_normal((len(rec), nt)).astype(np.float32)
        out[f"rtm{q}"] = lambda c, a=(g, vel, sou, w, rec, data): c.rtm(*a)
        out[f"model{q}"] = lambda c, a=(g, vel, sou, w, rec): (c.modeling(*a),)
    g3, vel3, sou3, rec3, w3 = case3d(nz=60, nx=70, ny=64, nt=80)
    out["model3d"] = lambda c: (c.modeling(g3, vel3, sou3, w3, rec3),)
    x = np.random.default_rng(9).standard_normal((2, 200, 150)).astype(np.float32)

    def net(c):
        n = sw.CNN(c, [2, 32, 32, 1], seed=3)
        y = n.forward(x)
        n.close()
        return (y,)
    out["network"] = net
    return out


@pytest.mark.parametrize("plans", [
    [["rtm0"] * 12, ["rtm1"] * 6, ["rtm2"] * 6],
    [["rtm2", "model1"] * 4, ["model3d"] * 8, ["network"] * 20],
    [["model2", "rtm0"] * 5] * 4,
])
def test_contexts_side_by_side(plans):
    work = _work()
    with_one = sw.Context(0)
    alone = {k: work[k](with_one) for k in sorted({k for p in plans for k in p})}
    with_one.close()
    for v in alone.values():
        assert all(np.abs(a).max() > 0 for a in v)
    wrong, start = [], threading.Barrier(len(plans))

    def run(plan):
        try:
            c = sw.Context(0)
            start.wait(60)
            for k in plan:
                for a, b in zip(work[k](c), alone[k]):
                    if not np.array_equal(a, b):
                        wrong.append(k)
            c.close()
        except Exception as e:   # a thread's exception would be lost
            wrong.append(repr(e))

    threads = [threading.Thread(target=run, args=(p,)) for p in plans]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120)
    assert not wrong
