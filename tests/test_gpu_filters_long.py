"""Band-pass of records longer than 65535 blocks of 32 samples, and of more
traces than that many blocks of 32, against the oracle bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ntr,nt,phase", [(1, 2_097_153, 0), (2, 2_100_007, 1), (2_097_185, 3, 1)])
def test_bandpass_long(ctx, oracle, ntr, nt, phase):
    tr = np.random.default_rng(7).standard_normal((ntr, nt)).astype(np.float32)
    a = ctx.bandpass(tr, 2e-3, fhi=90.0, nphi=4, phase=phase)
    b = oracle.bandpass(tr, 2e-3, fhi=90.0, nphi=4, phase=phase)
    assert np.isfinite(b).all() and np.abs(b).max() > 0
    np.testing.assert_array_equal(a, b)
