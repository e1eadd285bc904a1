"""The solute-mass projection of FP32 states against its rule in exact
arithmetic: compositions that are multiples of 2^-24 below 1, so that every
sum is exact in FP64 and the expected state is known to the bit.  Sizes at the
edges of the kernel's split (four cells per lane, 128 per warp step), both
signs, few and many units per cell, and shifts too wide for one FP32 addend;
the ghosts are checked by a step from the projected and the re-uploaded state."""
import numpy as np
import pytest

import phasefield_coarsening_gb300 as ppf

pytestmark = pytest.mark.gpu

UNIT = 2.0 ** -24


def project(c, target):
    """two passes of the rule, on the flattened (z, y, x) cells"""
    n = c.size
    for _ in range(2):
        units = int(round((target - float(np.sum(c.astype(np.float64)))) / UNIT))
        base, rem = divmod(units, n)
        i = np.arange(n, dtype=object)
        extra = np.array([int(k * rem % n + rem >= n) for k in i], dtype=np.int64)
        c = (c.astype(np.float64) + base * UNIT).astype(np.float32)
        c = (c.astype(np.float64) + extra * UNIT).astype(np.float32)
    return c


@pytest.mark.parametrize("bc", ["periodic", "noflux"])
@pytest.mark.parametrize("shape", [(3, 5, 7), (2, 2, 2), (4, 3, 129), (2, 9, 256), (5, 6, 131), (3, 2, 516)])
def test_projection_follows_its_rule(shape, bc):
    rng = np.random.default_rng(7)
    n = int(np.prod(shape))
    c0 = (rng.integers(1 << 20, 1 << 23, shape) * UNIT)
    eS = rng.uniform(0.4, 0.6, shape)
    eL = rng.uniform(0.4, 0.6, shape)
    m0 = float(c0.sum())
    p = ppf.params_default(dt=1e-4)
    with ppf.Simulation(shape, p, bc, "f32") as a, ppf.Simulation(shape, p, bc, "f32") as b:
        for units in (0, 1, -1, n // 3, -(5 * n + 7), 3 * n + n - 1, 1 - n, (1 << 24) * n + 5):
            a.upload(eS, eL, c0)
            a.mass_project(m0 + units * UNIT)
            got = a.download()
            want = project(c0.astype(np.float32).ravel(), m0 + units * UNIT).reshape(shape)
            assert np.array_equal(np.asarray(got[2], dtype=np.float32), want), units
            b.upload(*got)
            a.step(1)
            b.step(1)
            for x, y in zip(a.download(), b.download()):
                assert np.array_equal(np.asarray(x), np.asarray(y)), units
