"""The convolutions at the edges of their work items: items of one, two and
three output rows, CTAs with no item, one, and several of different lengths
(their rows dealt to the epilogue groups across items), two x tiles, both
boundary conditions."""
import numpy as np
import pytest

import phasefield_coarsening_gb300 as ppf
from helpers import smooth_state
from oracle import surrogate_ref as sr
from test_gpu_surrogate import make_sim, perturbed

pytestmark = pytest.mark.gpu

# tolerances as in test_gpu_surrogate.py: BF16 roundings moved by FP32 accumulation order


@pytest.mark.parametrize("width", [16, 32])
@pytest.mark.parametrize("bc", ["periodic", "noflux"])
@pytest.mark.parametrize("shape", [(2, 2, 128), (2, 3, 128), (3, 5, 256), (40, 17, 128), (61, 6, 128)])
def test_forward_over_work_items(width, bc, shape):
    state = smooth_state(shape, seed=sum(shape))
    p = sr.init_params(width, seed=3, last_scale=1.0)
    with ppf.Surrogate(width=width) as net, make_sim(shape, state, bc=bc) as sim:
        net.set_params(p)
        got = net.predict(sim)
        again = net.predict(sim)
        cfg = net.config
    assert np.array_equal(got, again)
    pred, _ = sr.forward(state, p, cfg, bc=bc)
    ref = pred * np.asarray(cfg["out_scale"])[:, None, None, None]
    assert np.abs(got - ref).max() <= 2e-2 * np.abs(ref).max()
    assert np.linalg.norm(got - ref) <= 5e-3 * np.linalg.norm(ref)


@pytest.mark.parametrize("width", [16, 32])
@pytest.mark.parametrize("shape", [(2, 2, 128), (3, 3, 256), (40, 9, 128)])
def test_gradients_over_work_items(width, shape):
    s0 = smooth_state(shape, seed=sum(shape))
    s1 = perturbed(s0, 5)
    p = sr.init_params(width, seed=6, last_scale=1.0)
    with ppf.Surrogate(width=width) as net, make_sim(shape, s0) as a, make_sim(shape, s1) as b:
        net.set_params(p)
        loss, g = net.loss_grad(a, b)
        loss2, g2 = net.loss_grad(a, b)
        cfg = net.config
    assert loss == loss2 and np.array_equal(g, g2)
    rl, rg = sr.loss_and_grad(s0, s1, p, cfg)
    assert abs(loss - rl) <= 1e-3 * rl
    off = 0
    for li, (ci, co) in enumerate(sr.layer_channels(width)):
        for n, what in ((27 * co * ci, "W"), (co, "b")):
            ref = rg[off:off + n]
            assert np.linalg.norm(g[off:off + n] - ref) <= 2e-2 * np.linalg.norm(ref) + 1e-12, (li, what)
            off += n
