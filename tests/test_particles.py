"""Particle analysis: the oracle's union-find on CPU, and the GPU labelling
(through the C-ABI) against it."""
import numpy as np
import pytest

import oracle
import phasefield_coarsening_gb300 as ppf
from phasefield_coarsening_gb300 import ic


def _slab_across_x_face(n=16):
    e = np.zeros((n, n, n))
    e[4:8, 4:8, :3] = 1.0      # touches x = 0
    e[4:8, 4:8, -2:] = 1.0     # touches x = n-1
    e[10:12, 10:12, 6:9] = 1.0
    return e


def test_oracle_joins_across_periodic_faces_only():
    e = _slab_across_x_face()
    p = oracle.particles(e, bc=0)
    f = oracle.particles(e, bc=1)
    assert p["count"] == 2 and f["count"] == 3
    assert sorted(p["volumes"]) == [12, 80]
    assert p["solid_volume"] == f["solid_volume"] == 92


def test_oracle_mean_radius_of_spheres():
    eS, _, _, info = ic.generate((48, 48, 48), radius=("uniform", 4, 8), count=10, seed=3)
    p = oracle.particles(eS, bc=0)
    assert p["count"] == 10
    assert abs(p["mean_radius"] - info["mean_radius"]) < 0.05 * info["mean_radius"]


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("bc", [0, 1])
def test_gpu_particles_match_oracle(precision, bc):
    eS, eL, c, _ = ic.generate((40, 36, 70), radius=("uniform", 3, 7), count=25, seed=7 + bc)
    with ppf.Simulation(eS.shape, bc=bc, precision=precision) as s:
        s.upload(eS, eL, c)
        g = s.particles(volumes=True)
        field = s.download()[0]
    o = oracle.particles(field, bc=bc)
    assert g["count"] == o["count"] > 5
    assert np.array_equal(g["volumes"], o["volumes"])
    assert abs(g["mean_radius"] - o["mean_radius"]) <= 1e-12 * o["mean_radius"]
    assert g["solid_volume"] == o["solid_volume"] and g["interface_area"] == o["interface_area"]
    assert g["largest_volume"] == o["largest_volume"]


@pytest.mark.gpu
def test_gpu_particles_wrap_and_edge_cases():
    e = _slab_across_x_face(16)
    for bc, n in ((0, 2), (1, 3)):
        with ppf.Simulation(e.shape, bc=bc) as s:
            s.upload(e, 1.0 - e, np.full(e.shape, 0.9))
            assert s.particles()["count"] == n
    empty = np.zeros((8, 8, 8))
    with ppf.Simulation(empty.shape) as s:
        s.upload(empty, 1.0 - empty, np.full(empty.shape, 0.9))
        st = s.particles(volumes=True)
        assert st["count"] == 0 and st["mean_radius"] == 0.0 and len(st["volumes"]) == 0
    full = np.ones((8, 8, 8))
    with ppf.Simulation(full.shape) as s:
        s.upload(full, 1.0 - full, np.full(full.shape, 0.476))
        st = s.particles()
        assert st["count"] == 1 and st["solid_volume"] == 512 and st["interface_area"] == 0


@pytest.mark.gpu
def test_fp32_mean_radius_within_half_percent_of_fp64():
    """The FP32 path against the FP64 path (itself pinned to the oracle) on
    the 64^3 sphere workload after 2000 steps: R-bar within 0.5 %."""
    from phasefield_coarsening_gb300 import validate
    r = validate.compare((64, 64, 64), "spheres64_uniform4to8", steps=2000, seed=0)
    print(r)
    assert r["rbar_rel_err"] <= 5e-3
    assert r["count_fp32"] == r["count_fp64"]
    # FP32 storage loses increments below half an ulp of c, and the ulp is
    # twice as large in the liquid (c ~ 0.999) as in the solid (c ~ 0.476):
    # a slow systematic drift, 1.5e-8 relative here (6.8e-8 after 10k steps
    # at 256^3); the FP64 path conserves to round-off
    assert abs(r["mass_drift_fp32"]) <= 5e-8
    assert abs(r["mass_drift_fp64"]) <= 1e-13


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 1, 31), (1, 3, 32), (3, 2, 33), (4, 5, 64), (5, 7, 65), (9, 8, 1), (6, 33, 100), (20, 24, 289)])
@pytest.mark.parametrize("bc", [0, 1])
@pytest.mark.parametrize("fill", [0.0, 0.15, 0.31, 0.6, 1.0])
def test_gpu_particles_of_random_cells(shape, bc, fill):
    """Independent random cells: many short runs, single cells, one component
    that fills the box; rows that are one word, several, and ragged.  Exact."""
    r = np.random.default_rng(int(100 * fill) + sum(shape) + bc)
    e = np.where(r.random(shape) < fill, 0.9, 0.1)
    with ppf.Simulation(shape, bc=bc, precision="f32") as s:
        s.upload(e, 1.0 - e, np.full(shape, 0.7))
        g = s.particles(volumes=True)
        few = s.particles()
    o = oracle.particles(e, bc=bc)
    assert g["count"] == few["count"] == o["count"]
    assert np.array_equal(g["volumes"], o["volumes"])
    assert g["solid_volume"] == o["solid_volume"] and g["interface_area"] == o["interface_area"]
    assert g["largest_volume"] == o["largest_volume"]
    assert abs(g["mean_radius"] - o["mean_radius"]) <= 1e-12 * o["mean_radius"]


@pytest.mark.gpu
@pytest.mark.parametrize("bc", [0, 1])
def test_gpu_particles_of_a_spiral(bc):
    """One chain through the whole box (its ends far apart in the labelling), and
    its complement."""
    n = 41
    e = np.zeros((3, n, n))
    lo, hi = 0, n - 1
    y, x = 0, 0
    dy, dx = 0, 1
    seen = np.zeros((n, n), bool)
    seen[0, 0] = True
    while True:                          # a spiral with one-cell gaps
        y2, x2 = y + dy, x + dx
        y3, x3 = y2 + dy, x2 + dx
        blocked = not (0 <= y2 < n and 0 <= x2 < n) or (0 <= y3 < n and 0 <= x3 < n and seen[y3, x3])
        if blocked:
            dy, dx = dx, -dy
            y2, x2 = y + dy, x + dx
            y3, x3 = y2 + dy, x2 + dx
            if not (0 <= y2 < n and 0 <= x2 < n) or seen[y2, x2] or (0 <= y3 < n and 0 <= x3 < n and seen[y3, x3]):
                break
        y, x = y2, x2
        seen[y, x] = True
    e[1][seen] = 1.0
    for f in (e, 1.0 - e):
        with ppf.Simulation(f.shape, bc=bc) as s:
            s.upload(f, 1.0 - f, np.full(f.shape, 0.7))
            g = s.particles(volumes=True)
        o = oracle.particles(f, bc=bc)
        assert g["count"] == o["count"] and np.array_equal(g["volumes"], o["volumes"])
        assert g["interface_area"] == o["interface_area"]


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(19, 35, 300), (40, 33, 40), (70, 18, 20), (8, 16, 128), (9, 17, 129)])
@pytest.mark.parametrize("bc", [0, 1])
@pytest.mark.parametrize("fill", [0.2, 0.31, 0.5])
def test_gpu_particles_over_bricks(shape, bc, fill):
    """Domains of one and of several labelling bricks in every direction, whole
    and ragged; fewer volumes asked for than there are particles."""
    import ctypes
    r = np.random.default_rng(int(100 * fill) + sum(shape) + bc)
    e = np.where(r.random(shape) < fill, 0.9, 0.1)
    o = oracle.particles(e, bc=bc)
    with ppf.Simulation(shape, bc=bc) as s:
        s.upload(e, 1.0 - e, np.full(shape, 0.7))
        g = s.particles(volumes=True)
        few = max(1, o["count"] // 3)
        some = np.full(few + 1, -1, np.int64)
        st, n = ppf.ParticleStats(), ctypes.c_int64(0)
        assert ppf.lib().ppf_particles(s._h, 0.5, ctypes.byref(st), some.ctypes.data, few, ctypes.byref(n)) == 0
    assert g["count"] == o["count"] and np.array_equal(g["volumes"], o["volumes"])
    assert g["interface_area"] == o["interface_area"] and g["solid_volume"] == o["solid_volume"]
    assert n.value == o["count"] and some[few] == -1
    assert np.all(np.diff(some[:few]) >= 0) and np.all(np.isin(some[:few], o["volumes"]))


@pytest.mark.gpu
@pytest.mark.parametrize("fill", [0.3, 0.36])
def test_gpu_particles_repeat(fill):
    """Large branching components over many bricks, analysed again and again with
    other contents of the scratch in between: the same components every time."""
    shape = (64, 64, 256)
    r = np.random.default_rng(int(100 * fill))
    e = np.where(r.random(shape) < fill, 0.9, 0.1)
    o = oracle.particles(e, bc=0)
    with ppf.Simulation(shape, precision="f32") as s:
        s.upload(e, 1.0 - e, np.full(shape, 0.7))
        for k in range(40):
            s.particles(0.05 if k % 2 else 0.95, volumes=True)
            g = s.particles(volumes=True)
            assert g["count"] == o["count"] and np.array_equal(g["volumes"], o["volumes"]), k


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(12, 16, 64), (33, 32, 64), (40, 48, 128), (80, 96, 128)])
def test_gpu_particle_volumes_in_order(shape):
    """Few, some and more volumes than one block sorts (single cells on a lattice,
    one in five of them grown to a row of up to 19 cells in the gap planes)."""
    r = np.random.default_rng(sum(shape))
    e = np.zeros(shape)
    e[::2, ::2, ::2] = 1.0
    for z, y, x in np.argwhere(e > 0):
        if r.random() < 0.2 and z + 1 < shape[0]:
            e[z + 1, y, x:x + r.integers(1, 20)] = 1.0
    o = oracle.particles(e, bc=1)
    with ppf.Simulation(shape, bc=1) as s:
        s.upload(e, 1.0 - e, np.full(shape, 0.7))
        g = s.particles(volumes=True)
    assert g["count"] == o["count"] and np.array_equal(g["volumes"], np.sort(o["volumes"]))


@pytest.mark.gpu
def test_gpu_mean_radius_repeats_and_is_exact():
    """Thousands of particles in an order that differs from call to call: the mean
    radius is the same number every time, the exact sum of the (correctly rounded to
    an ulp) radii to a few ulps."""
    import math
    rng = np.random.default_rng(11)
    shape = (40, 70, 130)
    etaS = np.where(rng.random(shape) < 0.24, 0.9, 0.1)
    with ppf.Simulation(shape, ppf.params_default(dx=0.7), bc="noflux") as s:
        s.upload(etaS, 1 - etaS, np.full(shape, 0.7))
        first = s.particles(volumes=True)
        assert first["count"] > 10000
        for _ in range(60):
            assert s.particles()["mean_radius"] == first["mean_radius"]
    exact = math.fsum(np.cbrt(3 / (4 * math.pi) * first["volumes"])) / first["count"]
    assert abs(first["mean_radius"] / exact - 1) <= 1e-15
