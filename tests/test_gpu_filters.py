"""Band-pass pass splits (sections are run up to four at a time) and lengths
around its eight-sample blocks, against the oracle bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ntr,nt,nplo,nphi,phase", [
    (1, 2, 14, 14, 0), (5, 9, 2, 1, 0), (33, 61, 14, 30, 1), (32, 64, 64, 6, 0),
    (100, 333, 9, 20, 1), (65, 1001, 3, 14, 0)])
def test_bandpass_sections(ctx, oracle, ntr, nt, nplo, nphi, phase):
    tr = np.random.default_rng(nt).standard_normal((ntr, nt)).astype(np.float32)
    a = ctx.bandpass(tr, 2e-3, flo=40.0, fhi=90.0, nplo=nplo, nphi=nphi, phase=phase)
    b = oracle.bandpass(tr, 2e-3, flo=40.0, fhi=90.0, nplo=nplo, nphi=nphi, phase=phase)
    assert np.isfinite(b).all() and np.abs(b).max() > 0
    np.testing.assert_array_equal(a, b)
