"""Phase fields that fall off by orders of magnitude, in the FP64 step that
computes its rates in fixed point: every value keeps float64's relative
precision, however small it is.  On the host against extended precision, and
on the GPU against the oracle."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import oracle
import phasefield_coarsening_gb300 as ppf

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "phasefield_coarsening_gb300", "csrc")
DT08 = 0.8 / (6.0 * 1e-14)


def tails(shape, floor, seed=0):
    """Interfaces whose phase fields decay from 1 to `floor` over the box, with
    a solid and a liquid side, each field the other's tail; noisy, c smooth."""
    r = np.random.default_rng(seed)
    z, y, x = np.meshgrid(*[np.arange(n) for n in shape], indexing="ij")
    t = np.cos(2 * np.pi * x / shape[2]) + 0.2 * np.cos(2 * np.pi * y / shape[1]) + 0.1 * np.sin(2 * np.pi * z / shape[0])
    decade = np.log10(floor) * np.clip(np.abs(t), 0, 1)
    small = 0.5 * 10.0 ** decade * (1 + 0.05 * r.random(shape))
    S = np.where(t > 0, 1 - small, small)
    L = np.where(t > 0, small, 1 - small)
    c = 0.476 * (t > 0) + 0.999 * (t <= 0) + 0.02 * r.random(shape)
    return S, L, c


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("fx") / "fx_tails.so")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-I", CSRC,
                    os.path.join(HERE, "fx_tails.cpp"), "-o", out], check=True, capture_output=True)
    return ctypes.CDLL(out)


def coef(p):
    d = ppf.derive(p)
    t1, t3 = -d.L * d.dt, 0.5 * d.dt * d.h2
    return np.array([p.AS, p.cL0, p.cL0 - p.cS0, t3 * d.ML, t3 * (d.MS - d.ML), p.CS - p.CL, p.cS0 - p.cL0, 2 * t1,
                     t1 * d.m, 2 * p.gamma, t1 * d.kappa * d.h2])


@pytest.mark.parametrize("change", [{}, dict(dt=DT08 / 4), dict(AS=300.0, AL=300.0, CS=0.0, CL=0.0), dict(sigma=0.3, l=12.0)])
@pytest.mark.parametrize("floor", [1e-2, 1e-6, 1e-12, 1e-18, 1e-60, 1e-290])
def test_small_values_keep_their_relative_precision(host, change, floor):
    """Errors relative to the cell's own stencil: at most 2.5 units of 2^-53
    (the rounding of the new value, half; of the neighbours' sum, of the two
    products and their sum, a quarter each at most since a step moves a value by less
    than a quarter; of the rate, 2^-59 of a scale below 1), and on average those of
    float64 arithmetic."""
    shape = (8, 12, 40)
    st = tails(shape, floor)
    i = np.arange(np.prod(shape)).reshape(shape)
    nb = np.stack([np.roll(i, -s, a).ravel() for a in (0, 1, 2) for s in (1, -1)], 1).astype(np.int32).copy()
    a = np.concatenate([x.ravel() for x in st])
    err = np.zeros(4 * i.size)
    k = coef(ppf.params_default(**{"dt": DT08, **change}))
    p = [v.ctypes.data_as(ctypes.c_void_p) for v in (nb, k, a, err)]
    assert host.fx_tail_errors(i.size, *p) == 1
    got, f64 = err.reshape(2, -1)
    assert np.abs(got).max() <= 2.5 * 2.0 ** -53
    assert np.sqrt(np.mean(got ** 2)) <= 1.02 * np.sqrt(np.mean(f64 ** 2))


@pytest.mark.gpu
@pytest.mark.parametrize("bc", [0, 1])
@pytest.mark.parametrize("floor", [1e-6, 1e-12, 1e-25, 1e-200])
def test_small_values_step_as_in_float64(floor, bc):
    """Ten steps against the oracle, value by value: each step's rounding differs
    by a few units of 2^-53 of the largest value of the cell's stencil, which decades
    per cell apart make up to 1e4 times the cell's own after ten steps' spreading;
    the increments' sums of squares, whose largest terms are interface cells', to 1e-10."""
    shape = (8, 18, 70)
    st = tails(shape, floor, seed=3)
    with ppf.Simulation(shape, ppf.params_default(dt=DT08), bc=bc) as s:
        s.upload(*st)
        s.step(10)
        got = s.download()
        g = s.reduce()
    ref = oracle.run(*st, 10, bc=bc, params=oracle.reference_params(dt=DT08))
    for a, b in zip(got[:2], ref[:2]):
        size = np.abs(b)
        for ax in range(3):
            size = np.maximum.reduce([size, np.roll(size, 1, ax), np.roll(size, -1, ax)])
        assert (np.abs(a - b) <= 100 * 2.0 ** -53 * size).all(), (np.abs(a - b) / size).max()
    np.testing.assert_allclose([g["sum_dc2"], g["sum_detaS2"], g["sum_detaL2"]], ref[3], rtol=1e-10)


# a liquid minimum at or near zero: float64 keeps the relative precision of a
# dilute composition
DILUTE = dict(cS0=0.5, cSeq=0.02, cLeq=0.5)


@pytest.mark.parametrize("cL0", [0.0, 1e-12, 1e-3, -0.02])
def test_dilute_liquids_are_left_to_float64(host, cL0):
    shape = (2, 2, 2)
    i = np.arange(8).reshape(shape)
    nb = np.stack([np.roll(i, -s, a).ravel() for a in (0, 1, 2) for s in (1, -1)], 1).astype(np.int32).copy()
    a, err = np.ones(24) * 0.5, np.zeros(32)
    for c, fits in ((cL0, 0), (0.3 + cL0, 1)):
        k = coef(ppf.params_default(dt=DT08, cL0=c, **DILUTE))
        assert host.fx_tail_errors(8, *[v.ctypes.data_as(ctypes.c_void_p) for v in (nb, k, a, err)]) == fits


@pytest.mark.gpu
def test_dilute_compositions_step_as_in_float64():
    """Compositions of 1e-9 beside a liquid minimum of 0: sums of six products of
    relative error 2^-53 and their neighbours' over five steps, 1e-13 of the value."""
    shape = (6, 18, 40)
    r = np.random.default_rng(5)
    p = dict(dt=DT08, cL0=0.0, **DILUTE)
    st = np.zeros(shape), np.ones(shape), 1e-9 * (1 + 0.3 * r.random(shape))
    with ppf.Simulation(shape, ppf.params_default(**p)) as s:
        s.upload(*st)
        s.step(5)
        got = s.download()
    ref = oracle.run(*st, 5, bc=0, params=oracle.reference_params(**p))
    assert np.abs(got[2] / ref[2] - 1).max() <= 1e-13


@pytest.mark.gpu
@pytest.mark.parametrize("S,L", [(1 - 1e-6, 1e-7), (1e-7, 1 - 1e-6), (0.999, 1e-9), (1e-4, 1.01)])
def test_sums_of_the_increments_of_a_bulk_phase(S, L):
    """Uniform phases near their equilibrium, whose increments lie far below an ulp
    of the value: the sums of squares against the oracle's, 1e-9 (float64's own
    error of etaS^2 - 1 is 1e-10 of it at 1e-6 from 1)."""
    shape = (3, 17, 40)
    st = np.full(shape, S), np.full(shape, L), np.full(shape, 0.7)
    with ppf.Simulation(shape, ppf.params_default(dt=DT08)) as s:
        s.upload(*st)
        s.step(1)
        g = s.reduce()
    ref = oracle.run(*st, 1, bc=0, params=oracle.reference_params(dt=DT08))
    np.testing.assert_allclose([g["sum_detaS2"], g["sum_detaL2"]], ref[3][1:], rtol=1e-9)
