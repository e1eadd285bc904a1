"""The sums over CTAs of a training step (loss, gradients) where floats do not
hold them: partial sums that are finite and whose total is not, and partial
sums that are infinite."""
import numpy as np
import pytest

import phasefield_coarsening_gb300 as ppf
from helpers import smooth_state
from oracle import surrogate_ref as sr
from test_gpu_surrogate import make_sim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [16, 32])
def test_loss_beyond_the_largest_float(width):
    """A target 1e18 away: the loss is (1e20)^2 / 3, FP32 terms of 1e-7 each and an
    FP64 total; one 1e24 away: infinite in every CTA, and so in total."""
    shape = (61, 40, 128)
    s0 = smooth_state(shape, seed=1)
    far = [x.copy() for x in s0]
    with ppf.Surrogate(width=width) as net, make_sim(shape, s0) as a, make_sim(shape, s0) as b:
        net.set_params(sr.init_params(width, seed=6, last_scale=1.0))
        scale = net.config["out_scale"][0]
        far[0] = s0[0] + 1e18
        b.upload(*far)
        loss, _ = net.loss_grad(a, b)
        want = (np.float64(np.float32(1e18)) / scale) ** 2 / 3
        assert want > 3.5e38 and abs(loss / want - 1) <= 1e-5
        far[0] = s0[0] + 1e24
        b.upload(*far)
        loss, _ = net.loss_grad(a, b)
        assert loss == np.inf
