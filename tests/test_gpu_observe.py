"""Observables of states whose terms are small, huge or differ by orders of
magnitude: every sum keeps the precision of its own terms."""
import numpy as np
import pytest

import phasefield_coarsening_gb300 as ppf

pytestmark = pytest.mark.gpu

DT08 = 0.8 / (6.0 * 1e-14)
SHAPES = [(6, 18, 40), (5, 7, 33)]


@pytest.mark.parametrize("shape", SHAPES)
def test_fp64_sums_of_small_terms(shape):
    """A dilute liquid with next to no solid: mass and solid relative to
    themselves (a few roundings of 2^-53 a term and a sum of about 5000), and the
    chemical energy of compositions 1e-6 from the minimum (w to 2^-54 of c)."""
    r = np.random.default_rng(1)
    S, L = 1e-9 * (1 + r.random(shape)), np.ones(shape)
    c = 1e-10 * (1 + r.random(shape))
    p = ppf.params_default(dt=DT08, AS=300.0, AL=300.0, CS=0.0, CL=0.0)
    with ppf.Simulation(shape, p) as s:
        s.upload(S, L, c)
        g = s.reduce()
        assert abs(g["mass"] / c.sum() - 1) <= 1e-13
        assert abs(g["solid"] / (S * S / (S * S + L * L)).sum() - 1) <= 1e-13
        c = 0.978 + 1e-6 * (1 + r.random(shape))
        s.upload(np.zeros(shape), L, c)
        w = c.astype(np.longdouble) - np.longdouble(0.978)
        assert abs(s.reduce()["free_energy"] / float((150 * w * w).sum()) - 1) <= 1e-10


def test_fp32_gradient_energy_beside_a_larger_well_energy():
    """Two arrangements of the same values differ by their gradients alone, a third
    of an FP32 ulp of a cell's well energy: the sum has 48 bits of them (a hundredth
    of the difference allowed)."""
    shape = (8, 16, 32)
    d = 8.4e-6
    z, y, x = np.meshgrid(*[np.arange(n) for n in shape], indexing="ij")
    L = np.full(shape, 0.5)
    c = np.full(shape, 0.7)
    p = ppf.params_default(dt=DT08, AS=1e-9, AL=1e-9, CS=0.0, CL=0.0)
    m = ppf.derive(p)
    got, want = [], []
    with ppf.Simulation(shape, p, precision="f32") as s:
        for sign in (np.where((x + y + z) % 2, 1, -1), np.where(x < 16, 1, -1)):
            S = (0.5 + d * sign).astype(np.float32).astype(np.float64)
            s.upload(S, L, c)
            got.append(s.reduce()["free_energy"])
            want.append(0.5 * m.kappa * m.h2 * sum(((np.roll(S, -1, a) - S) ** 2).sum() for a in range(3)))
    assert abs((got[0] - got[1]) / (want[0] - want[1]) - 1) <= 1e-2


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("precision,size,tol", [("f32", 6e-20, 3e-6), ("f32", 1e19, 1e-6), ("f64", 1e-157, 1e-8), ("f64", 1e153, 1e-13)])
def test_solid_fraction_at_the_ends_of_the_range(shape, precision, size, tol):
    """Phase fields whose squares are denormal or near the largest number: the
    ratio etaS^2 / (etaS^2 + etaL^2) is what the type's division gives (a denormal
    square is exact to a unit, 1.4e-45 or 5e-324)."""
    r = np.random.default_rng(3)
    t = np.float32 if precision == "f32" else np.float64
    S, L = ((size * r.uniform(0.7, 1.3, shape)).astype(t) for _ in range(2))
    c = r.uniform(0.4, 1.0, shape)
    with ppf.Simulation(shape, precision=precision) as s:
        s.upload(S.astype(np.float64), L.astype(np.float64), c)
        g = s.reduce()
    S2, s2 = S * S, S * S + L * L
    assert s2.max() < np.finfo(t).max and g["nonfinite"] == 0
    assert abs(g["solid"] / (S2 / s2).astype(np.float64).sum() - 1) <= tol


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("bad", [False, True])
def test_fp32_mass_of_huge_compositions(shape, bad):
    """Finite compositions whose sum no float holds: an FP64 sum of the stored
    values, non-finite cells left out."""
    r = np.random.default_rng(4)
    S, L = r.uniform(0.2, 1.0, shape), r.uniform(0.2, 1.0, shape)
    c = (3e38 * r.uniform(0.5, 1.0, shape)).astype(np.float32).astype(np.float64)
    if bad:
        c[1, 2, 3] = np.inf
        S[2, 3, 5] = np.nan
    with ppf.Simulation(shape, precision="f32") as s:
        s.upload(S, L, c)
        g = s.reduce()
    ok = np.isfinite(S) & np.isfinite(c)
    assert g["nonfinite"] == (~ok).sum()
    assert abs(g["mass"] / c[ok].sum() - 1) <= 1e-12


@pytest.mark.parametrize("precision", ["f32", "f64"])
def test_solid_fraction_of_a_cell_is_its_quotient(precision):
    """One cell's h = etaS^2 / (etaS^2 + etaL^2): the quotient of the rounded squares
    to 0.51 ulp (a correctly rounded division's 0.5), by the one sum of one term.
    (FP64 states in the box have no rounded squares: parameters outside it.)"""
    from fractions import Fraction
    r = np.random.default_rng(6)
    t = np.float32 if precision == "f32" else np.float64
    with ppf.Simulation((1, 1, 1), ppf.params_default(dt=DT08, AL=2e9), precision=precision) as s:
        for _ in range(300):
            S, L = r.uniform(0.05, 1.2, 2).astype(t)
            s.upload(*[np.full((1, 1, 1), float(v)) for v in (S, L, t(0.7))])
            got = s.reduce()["solid"]
            S2 = S * S
            exact = Fraction(float(L)) ** 2 + Fraction(float(S2))
            s2 = float(exact) if precision == "f64" else float(np.float32(float(exact)))
            q = Fraction(float(S2)) / Fraction(s2)
            assert abs(Fraction(got) - q) <= Fraction(51, 100) * Fraction(float(np.spacing(t(float(q)))))
