"""The float64 step in fixed-point arithmetic on the GPU: states that leave its
box while they run, states and parameters that never fit, and the same bits
from every way of launching it."""
import numpy as np
import pytest

import oracle
import phasefield_coarsening_gb300 as ppf
from helpers import smooth_state

pytestmark = pytest.mark.gpu

DT08 = 0.8 / (6.0 * 1e-14)
# a free energy without a bounded well along etaS = etaL (gamma < -1): both
# phase fields grow, and leave |eta| < 1.75 after some hundred steps
GROW = dict(dt=DT08, AS=300.0, AL=300.0, CS=0.0, CL=0.0, gamma=-1.9)


def growing(shape, seed=0):
    r = np.random.default_rng(seed)
    S = 1.3 + 0.05 * r.random(shape)
    L = 1.3 + 0.05 * r.random(shape)
    return S, L, 0.7 + 0.01 * r.random(shape)


def params(d):
    return ppf.params_default(**d)


def oracle_run(st, n, bc, d, n_iter_init=None):
    p = oracle.reference_params(**d)
    kw = {} if n_iter_init is None else {"n_iter_init": n_iter_init}
    return oracle.run(*st, n, bc=bc, params=p, **kw)


def close(a, b, tol):
    """max error relative to the field's own size"""
    for x, y in zip(a, b):
        assert np.abs(x - y).max() <= tol * np.abs(y).max(), np.abs(x - y).max() / np.abs(y).max()


@pytest.mark.parametrize("shape", [(6, 20, 40), (5, 16, 64)])
@pytest.mark.parametrize("bc", [0, 1])
def test_state_that_leaves_the_box_while_it_runs(shape, bc):
    """One call of many steps, during which the state leaves the box: the later
    steps run in float64 on the device.  Against the oracle; the growth of a
    perturbation is that of the fields (less than tenfold), so 1e-12 holds."""
    st = growing(shape)
    n = 1
    while oracle_run(st, n, bc, GROW)[0].max() < 2.2:
        n += max(1, n // 4)
    before = oracle_run(st, n // 2, bc, GROW)
    assert before[0].max() < 1.75
    ref = oracle_run(st, n, bc, GROW)
    with ppf.Simulation(shape, params(GROW), bc=bc) as s:
        s.upload(*st)
        s.step(n)
        one = s.download()
        g = s.reduce()
        s.step_c_only(3)               # float64 from the host's side now
        s.step(2)
        more = s.download()
        s.upload(*st)                  # back in the box
        s.step(n // 2)
        again = s.download()
    close(one, ref[:3], 1e-12)
    np.testing.assert_allclose([g["sum_dc2"], g["sum_detaS2"], g["sum_detaL2"]], ref[3], rtol=1e-8)
    close(again, before[:3], 1e-12)
    r2 = oracle_run([x for x in ref[:3]], 3, bc, GROW, n_iter_init=0)
    r2 = oracle_run(list(r2[:3]), 2, bc, GROW)
    close(more, r2[:3], 1e-12)


def test_ensemble_and_slabs_of_states_that_leave_the_box():
    """Domains leave the box one by one in an ensemble, and together as slabs of
    one domain: the bits of the undivided contexts."""
    shapes = [(6, 20, 40), (8, 16, 32), (4, 33, 70)]
    states = [growing(s, seed=i) for i, s in enumerate(shapes)]
    states[1] = smooth_state(shapes[1], seed=2)       # stays
    n = 1
    while oracle_run(states[0], n, 0, GROW)[0].max() < 2.2:
        n += max(1, n // 4)
    with ppf.Ensemble(shapes, params(GROW), precision="f64") as e:
        e.upload_all(states)
        e.step(n)
        got = e.download_all()
        red = [e.reduce(d) for d in range(3)]
    for d, shape in enumerate(shapes):
        with ppf.Simulation(shape, params(GROW)) as s:
            s.upload(*states[d])
            s.step(n)
            for a, b in zip(got[d], s.download()):
                assert np.array_equal(a, b)
            r = s.reduce()
            for k in ("sum_dc2", "sum_detaS2", "sum_detaL2"):
                assert abs(red[d][k] - r[k]) <= 1e-12 * abs(r[k])
    with ppf.Simulation(shapes[0], params(GROW)) as s, ppf.Slabs(shapes[0], 3, params(GROW)) as t:
        # one corner grows faster: some slabs hold the first cells outside
        st = [x.copy() for x in states[0]]
        st[0][5, :, :] += 0.2
        s.upload(*st)
        t.upload(*st)
        s.step(n)
        t.step(n)
        for a, b in zip(s.download(), t.download()):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("change", [{}, dict(AL=1.5e9), dict(DS=3e-15), dict(dt=DT08 * 0.3), dict(gamma=2.4)])
@pytest.mark.parametrize("bc", [0, 1])
def test_parameter_sets_against_the_oracle(change, bc):
    """Parameters on both sides of the rule, partial tiles, 40 steps and 5
    c-only ones."""
    d = {"dt": DT08, **change}
    shape = (9, 21, 45)
    st = smooth_state(shape, seed=6)
    with ppf.Simulation(shape, params(d), bc=bc) as s:
        s.upload(*st)
        s.step(40)
        s.step_c_only(5)
        got = s.download()
    ref = oracle_run(st, 45, bc, d, n_iter_init=40)
    assert max(np.abs(a - b).max() for a, b in zip(got, ref[:3])) <= 1e-12


def test_states_that_start_outside_and_copies():
    """A state with an undefined cell (etaS = etaL = 0) and one outside the box
    stay in float64 from their upload on, also through the autotuner and
    ppf_copy_state; a state copied over them returns to the box."""
    shape = (6, 18, 40)
    st = [x.copy() for x in smooth_state(shape, seed=8)]
    good = smooth_state(shape, seed=9)
    st[0][2, 3, 4] = st[1][2, 3, 4] = 0.0
    ref = oracle_run(st, 3, 0, dict(dt=DT08))
    with ppf.Simulation(shape, params(dict(dt=DT08))) as a, ppf.Simulation(shape, params(dict(dt=DT08))) as b, \
            ppf.Simulation(shape, params(dict(dt=DT08))) as c:
        a.upload(*st)
        a.autotune(2)
        b.upload(*good)
        b.copy_from(a)
        c.upload(*st)
        c.copy_from(b)
        for s in (a, b, c):
            s.step(3)
            got = s.download()
            for x, y in zip(got, ref[:3]):
                assert np.array_equal(np.isnan(x), np.isnan(y))
                ok = np.isfinite(y)
                assert np.abs(x[ok] - y[ok]).max() <= 1e-12
        b.upload(*good)
        a.copy_from(b)
        a.step(4)
        b.step(4)
        for x, y in zip(a.download(), b.download()):
            assert np.array_equal(x, y)
