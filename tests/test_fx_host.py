"""The fixed-point arithmetic of the float64 step (csrc/ppf_fx.h) on the host,
against extended precision and against float64, over the parameter and state
ranges it accepts; and what it refuses."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import phasefield_coarsening_gb300 as ppf
from helpers import smooth_state

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "phasefield_coarsening_gb300", "csrc")
DT08 = 0.8 / (6.0 * 1e-14)


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("fx") / "fx_host.so")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-I", CSRC,
                    os.path.join(HERE, "fx_host.cpp"), "-o", out], check=True, capture_output=True)
    L = ctypes.CDLL(out)
    L.fx_recip_error.restype = ctypes.c_double
    return L


def coef(p):
    d = ppf.derive(p)
    t1, t3 = -d.L * d.dt, 0.5 * d.dt * d.h2
    return np.array([p.AS, p.cL0, p.cL0 - p.cS0, t3 * d.ML, t3 * (d.MS - d.ML), p.CS - p.CL, p.cS0 - p.cL0, 2 * t1,
                     t1 * d.m, 2 * p.gamma, t1 * d.kappa * d.h2])


def ptr(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def units(host, p):
    u = np.zeros(2)
    k = coef(p)
    ok = host.fx_units(ctypes.c_double(p.AS), ctypes.c_double(p.AL), ptr(k), ptr(u))
    return u if ok else None


def rough_state(shape, seed):
    """Anything in the box: independent cells."""
    r = np.random.default_rng(seed)
    S, L, c = r.uniform(-0.3, 1.3, shape), r.uniform(0.55, 1.5, shape), r.uniform(-1.5, 1.9, shape)
    S.flat[:6] = [0.0, 1.0, -0.0, 1e-300, 1.7499, 2.0 ** -63]
    L.flat[:6] = [1.0, 0.0, 0.5000001, 1.0, 1.0, 0.75]
    c.flat[:4] = [0.0, 1e-12, 1.999, -1.999]
    return S, L, c


PARAMS = {
    "reference": {}, "half_dt": dict(dt=DT08 / 2), "limit": dict(dt=DT08 / 0.8 * (1 - 1e-12)), "solid_diffuses": dict(DS=4e-15),
    "gamma": dict(gamma=0.8), "stiff": dict(AS=300.0, AL=300.0, CS=0.0, CL=0.0), "wide": dict(sigma=0.3, l=12.0),
}


@pytest.mark.parametrize("name", sorted(PARAMS))
@pytest.mark.parametrize("bc", [0, 1])
@pytest.mark.parametrize("kind", ["smooth", "rough"])
def test_fixed_point_step_is_as_exact_as_float64(host, name, bc, kind):
    """One step: before they are rounded and added, the increments are within
    32 units of its increments' scales: 2^(eu-59) for the phase fields
    (drive 8 units, its factors 14, well and Laplacian terms 4, products 1
    each) and 2^(ec-59) for c (w 2.5 units a cell, six faces of slope at most
    1/6).  Its rms error is the float64 step's, up to what those units add."""
    p = ppf.params_default(**{"dt": DT08, **PARAMS[name]})
    u = units(host, p)
    assert u is not None
    shape = (7, 6, 9)
    st = smooth_state(shape, seed=3) if kind == "smooth" else rough_state(shape, 4)
    a = np.concatenate([x.ravel() for x in st])
    diff, rms, drift = np.zeros(3), np.zeros(6), ctypes.c_double()
    k = coef(p)
    out = host.fx_step_errors(*shape, bc, ptr(k), ptr(a), ptr(diff), ptr(rms), ctypes.byref(drift))
    assert out == 0
    unit = np.array([u[1], u[1], u[0]]) * 2.0 ** -59
    assert (diff <= 32 * unit).all(), diff / unit
    assert (rms[:3] <= 1.02 * rms[3:] + 2 * unit).all(), (rms[:3] / rms[3:], unit / rms[3:])
    assert drift.value == 0.0 or abs(drift.value) <= a[2 * len(a) // 3:].size * 2.0 ** -60   # faces cancel exactly


def test_reciprocal(host):
    """Third-order step on a 20-bit estimate: the remainder (2^-20.4)^3 and the
    last unit of 1/s2 @60 for the largest s2 (1/6.2: 2^-57.4)."""
    assert host.fx_recip_error(200000) <= 2.0 ** -57


def test_states_outside_the_box_are_seen(host):
    k, shape = coef(ppf.params_default(dt=DT08)), (2, 3, 4)
    base = smooth_state(shape, seed=1)
    for f, v in ((0, 1.75), (0, -1.76), (1, np.nan), (1, np.inf), (2, 2.0), (2, -2.5), (2, np.nan), (0, -np.inf)):
        st = [x.copy() for x in base]
        st[f][1, 2, 3] = v
        if f < 2 and np.isnan(v):
            st[1 - f][1, 2, 3] = 1.0
        a = np.concatenate([x.ravel() for x in st])
        assert host.fx_step_errors(*shape, 0, ptr(k), ptr(a), ptr(np.zeros(3)), ptr(np.zeros(6)),
                                   ctypes.byref(ctypes.c_double())) == 1, (f, v)
    st = [x.copy() for x in base]
    st[0][0, 0, 0], st[1][0, 0, 0] = 0.3, 0.39          # 0.09 + 0.1521 < 1/4
    st[0][0, 0, 1], st[1][0, 0, 1] = 0.0, 0.0
    st[0][0, 0, 2], st[1][0, 0, 2] = -0.36, 0.36        # 0.2592
    a = np.concatenate([x.ravel() for x in st])
    assert host.fx_step_errors(*shape, 0, ptr(k), ptr(a), ptr(np.zeros(3)), ptr(np.zeros(6)),
                               ctypes.byref(ctypes.c_double())) == 2


@pytest.mark.parametrize("change", [dict(AL=2e9), dict(dt=DT08 * 1.3), dict(gamma=2.5), dict(CS=-1e10), dict(AS=0.5, AL=0.5, CS=0.0, CL=0.0),
                                    dict(DS=2e-14)])
def test_parameters_that_do_not_fit_are_refused(host, change):
    """AS != AL, a step above the explicit limit (by either diffusivity), gamma
    of 2 or more, drives and rates above the scale: left to float64."""
    assert units(host, ppf.params_default(**{"dt": DT08, **change})) is None


def test_other_units_of_c(host):
    """Compositions in other units (c, cS0, cL0 scaled by s, AS by 1/s^2) take
    the same steps: the scale follows the parabola minima."""
    for s in (1e-3, 37.0, 5.2e4):
        p = ppf.params_default(dt=DT08, cS0=0.455 * s, cL0=0.978 * s, cSeq=0.999 * s, cLeq=0.476 * s, AS=1e9 / s ** 2,
                               AL=1e9 / s ** 2)
        u = units(host, p)
        assert u is not None and 0.978 * s <= u[0] < 2 * 0.978 * s
        shape = (5, 5, 6)
        st = smooth_state(shape, seed=9)
        a = np.concatenate([x.ravel() for x in (st[0], st[1], st[2] * s)])
        diff, rms = np.zeros(3), np.zeros(6)
        assert host.fx_step_errors(*shape, 0, ptr(coef(p)), ptr(a), ptr(diff), ptr(rms),
                                   ctypes.byref(ctypes.c_double())) == 0
        unit = np.array([u[1], u[1], u[0]]) * 2.0 ** -59
        assert (diff <= 32 * unit).all(), diff / unit
