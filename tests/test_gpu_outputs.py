"""Host outputs in pages the program has not touched, at odd offsets within
them, hold what they hold in touched ones; what lies beside them stays."""
import mmap

import numpy as np
import pytest

import seismic_gb300 as sw
from tests.cases import case2d

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 4, 8188])
def test_outputs_in_untouched_pages(ctx, offset):
    g, vel, sou, rec, w = case2d(nz=200, nx=390, nt=60)
    data = np.random.default_rng(1).standard_normal((len(rec), g.nt)).astype(np.float32)
    image, illum = ctx.rtm(g, vel, sou, w, rec, data)
    n = image.size
    fresh = []
    for _ in range(2):
        m = mmap.mmap(-1, 4 * n + 16384)
        m[offset + 4 * n] = 77
        fresh.append((m, np.frombuffer(m, np.float32, n, offset)))
    f = sw.fptr
    ctx._check(ctx.lib.sw_rtm(ctx.h, sw.C.byref(g), f(vel), f(sou), f(w), len(rec), f(rec),
                              f(data), f(fresh[0][1]), f(fresh[1][1])))
    for (m, a), b in zip(fresh, (image, illum)):
        np.testing.assert_array_equal(a, b)
        assert m[offset + 4 * n] == 77
