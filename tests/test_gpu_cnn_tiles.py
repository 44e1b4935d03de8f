"""The network kernels at image sizes around their 24 x 16 (convolution) and
16 x 16 (weight gradient) blocks, one and two K steps per tap (16 and 32
stored channels), 2D and 3D, against the float64 reference of test_gpu_cnn
(the same bound: the device sums in FP32 in another order, so a BF16 rounding
lands on the other side now and then)."""
import numpy as np
import pytest

import seismic_gb300 as sw
from tests.conftest import rel_l2
from tests.test_gpu_cnn import TOL, _ref_forward, _ref_gradient

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ch,shape", [
    ([2, 32, 32, 1], (1, 1)), ([2, 32, 32, 1], (16, 24)), ([2, 32, 32, 1], (17, 25)),
    ([1, 16, 16, 1], (33, 8)), ([3, 32, 16, 1], (15, 49)), ([2, 8, 32, 1], (48, 17)),
    ([2, 32, 32, 32, 1], (129, 301)),
    ([2, 16, 32, 1], (5, 17, 25)), ([2, 32, 8, 1], (3, 16, 48))])
def test_cnn_blocks(ctx, ch, shape):
    rng = np.random.default_rng(sum(shape))
    three_d = len(shape) == 3
    x = rng.standard_normal((2, ch[0]) + shape).astype(np.float32)
    t = rng.standard_normal((2,) + shape).astype(np.float32)
    net = sw.CNN(ctx, ch, seed=3, three_d=three_d)
    try:
        w = net.get_weights()
        w += 0.05 * rng.standard_normal(w.size).astype(np.float32)     # biases too
        net.set_weights(w)
        out = net.forward(x[0])
        g, loss = net.gradient(x, t)
    finally:
        net.close()
    ref, _ = _ref_forward(x[0], w, ch, three_d=three_d)
    rg, rl = _ref_gradient(x, t, w, ch, three_d=three_d)
    assert rel_l2(out, ref.detach().numpy()) < TOL
    assert rel_l2(g, rg) < TOL
    assert abs(loss - rl) < TOL * rl
