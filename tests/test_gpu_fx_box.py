"""FP64 states outside the fixed-point step's box: they step in float64 inside
the same kernel, at the general kernel's rate, and nothing that shares a
launch, a stream or an autotuner with them changes another domain's bits."""
import time

import numpy as np
import pytest

import phasefield_coarsening_gb300 as ppf
from helpers import smooth_state
from test_gpu_fx import GROW, growing, params

pytestmark = pytest.mark.gpu


def ms_per_step(obj, n=20):
    best = 1e9
    for _ in range(4):
        obj.sync()
        t = time.perf_counter()
        obj.step(n)
        obj.sync()
        best = min(best, (time.perf_counter() - t) * 1e3 / n)
    return best


def test_states_that_left_the_box_step_at_the_general_rate():
    """A domain that leaves the box during a run, in an ensemble, as slabs and
    alone in one long call, against a state known to be outside from its upload
    on: the same arithmetic, so a step may not take half as long again."""
    shape = (96, 128, 128)
    st = growing(shape)
    with ppf.Simulation(shape, params(GROW)) as a, ppf.Ensemble([shape], params(GROW), precision="f64") as e, \
            ppf.Slabs(shape, 2, params(GROW)) as t, ppf.Simulation(shape, params(GROW)) as b:
        for s in (a, t):
            s.upload(*st)
        e.upload_all([st])
        n = 8
        for _ in range(50):
            for s in (a, t, e):
                s.step(n)
            out = a.download()
            if out[0].max() > 1.9:
                break
        assert out[0].max() > 1.9
        b.upload(*out)                   # outside from the start
        general = ms_per_step(b)
        assert ms_per_step(e) <= 1.5 * general
        assert ms_per_step(t) <= 1.5 * general
        a.upload(*st)
        a.step(1)
        a.sync()
        t0 = time.perf_counter()
        a.step(2000)                     # one call, outside for most of it
        a.sync()
        assert (time.perf_counter() - t0) * 1e3 / 2000 <= 1.5 * general


def test_autotuning_leaves_the_state_and_its_arithmetic_alone():
    """Trials that leave the box do not count for the restored state, which is in
    it: bit for bit the steps of a context that was never tuned."""
    shape = (6, 20, 40)
    st = growing(shape)
    with ppf.Simulation(shape, params(GROW)) as a, ppf.Simulation(shape, params(GROW)) as b, \
            ppf.Simulation(shape, params(GROW)) as c:
        for s in (a, b, c):
            s.upload(*st)
        c.step(400)
        assert not c.download()[0].max() < 1.9       # a trial of so many steps leaves the box
        a.autotune(400)
        for n in (1, 2, 5):
            a.step(n)
            b.step(n)
            assert a.reduce()["steps"] == b.reduce()["steps"]
            for x, y in zip(a.download(), b.download()):
                assert np.array_equal(x, y)


def test_ensemble_domains_do_not_depend_on_one_another():
    """A domain that leaves the box while another one is outside from its upload
    on, over an even number of steps; then that one is replaced by a state
    inside.  Every domain has the bits of a context of its own throughout."""
    shape = (6, 20, 40)
    st = growing(shape)
    out = [x.copy() for x in growing(shape, seed=1)]
    out[0][2, 3, 4] = 1.8
    inside = smooth_state(shape, seed=2)
    with ppf.Ensemble([shape, shape], params(GROW), precision="f64") as e, ppf.Simulation(shape, params(GROW)) as a, \
            ppf.Simulation(shape, params(GROW)) as b:
        e.upload_all([out, st])
        a.upload(*out)
        b.upload(*st)

        def same(s, d):
            return all(np.array_equal(x, y) for x, y in zip(s.download(), e.download(d)))

        n = 0
        while n < 100 or not b.download()[0].max() > 1.9:
            for s in (e, a, b):
                s.step(20)
            n += 20
            assert n <= 400
        assert same(a, 0) and same(b, 1)
        e.upload(0, *inside)
        a.upload(*inside)
        for n in (2, 5, 18):
            for s in (e, a, b):
                s.step(n)
            assert same(a, 0) and same(b, 1)
        ra, rb = e.reduce(0), e.reduce(1)
        for r, s in ((ra, a), (rb, b)):
            q = s.reduce()
            for k in ("sum_dc2", "sum_detaS2", "sum_detaL2"):
                assert abs(r[k] - q[k]) <= 1e-12 * abs(q[k])


def test_slabs_that_left_the_box_and_an_upload_back():
    """Slabs learn together that the state has left the box, and that an upload
    brought it back."""
    shape = (9, 20, 40)
    st = growing(shape, seed=4)
    with ppf.Slabs(shape, 3, params(GROW)) as t, ppf.Simulation(shape, params(GROW)) as s:
        for back in (0, 1):
            t.upload(*st)
            s.upload(*st)
            for n in (100, 90, 1, 2):
                t.step(n)
                s.step(n)
                t.sync()
                s.sync()
                for x, y in zip(s.download(), t.download()):
                    assert np.array_equal(x, y)
                assert t.reduce()["steps"] == s.reduce()["steps"]
