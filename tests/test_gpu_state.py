"""State movement and observables at the edges of their kernels: rows shorter
and longer than a warp, groups of cells that end a row, single planes and
rows, device arrays that the kernels use in place and ones that they cannot.
"""
import numpy as np
import pytest

import oracle
import phasefield_coarsening_gb300 as ppf
from helpers import smooth_state

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (1, 3, 2), (2, 1, 3), (3, 2, 5), (5, 4, 31), (4, 7, 32), (3, 9, 33), (70, 5, 7), (9, 33, 129)]


def cuda(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def download_device(sim, outs):
    rc = ppf.lib().ppf_download_device(sim.handle, *[int(p) for p in outs])
    assert rc == 0, ppf.lib().ppf_last_error()


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("bc", ["periodic", "noflux"])
@pytest.mark.parametrize("precision", ["f64", "f32"])
def test_device_arrays_and_observables(shape, bc, precision):
    """A state uploaded from device arrays steps like one uploaded from the
    host (ghosts included), comes back in device arrays as on the host, bit
    for bit, and has the oracle's observables: FP64 sums to 1e-12; FP32: the
    mass of the stored values to 1e-12, terms of FP32 arithmetic (a few ulps of
    6e-8 each, random) to 1e-6 relative, on an energy scale of its own."""
    import torch
    st = smooth_state(shape, seed=sum(shape))
    dev = [cuda(a) for a in st]
    torch.cuda.synchronize()
    with ppf.Simulation(shape, bc=bc, precision=precision) as a, ppf.Simulation(shape, bc=bc, precision=precision) as b:
        a.upload(*st)
        b.upload_device([t.data_ptr() for t in dev])
        for n in (0, 3):
            a.step(n)
            b.step(n)
            host = a.download()
            out = torch.empty((3, *shape), dtype=torch.float64, device="cuda")
            torch.cuda.synchronize()
            download_device(b, [out[f].data_ptr() for f in range(3)])
            for f in range(3):
                assert np.array_equal(out[f].cpu().numpy(), host[f])
        g = a.reduce()
    o = oracle.observe(*host, bc=0 if bc == "periodic" else 1)
    t = 1e-12 if precision == "f64" else 1e-6
    assert abs(g["mass"] - o["mass"]) <= 1e-12 * abs(o["mass"])
    assert abs(g["solid"] - o["solid"]) <= t * max(o["solid"], 1.0)
    assert g["solid_cells"] == int((host[0] > 0.5).sum())
    scale = abs(o["free_energy"]) + 1e7 * o["solid"]       # the offset CL of every cell, and CS - CL of the solid
    assert abs(g["free_energy"] - o["free_energy"]) <= t * scale
    assert g["nonfinite"] == 0


def test_fp32_values_come_back_exactly():
    """Every kind of float survives the widening to float64: zeros of both
    signs, denormals, the smallest and largest normal numbers, infinities."""
    v = np.array([0.0, -0.0, 1e-45, -1e-45, 1.1754942e-38, 1.17549435e-38, -1.17549435e-38, 1.0, -1.0, 1 + 2.0 ** -23,
                  3.4028235e38, -3.4028235e38, np.inf, -np.inf, 0.1, -0.3], dtype=np.float32)
    shape = (1, 2, 8)
    st = [np.roll(v, k).astype(np.float64).reshape(shape) for k in range(3)]
    with ppf.Simulation(shape, precision="f32") as s:
        s.upload(*st)
        for a, b in zip(s.download(), st):
            assert np.array_equal(a.view(np.uint64), b.view(np.uint64))
    nan = [np.full(shape, np.nan)] * 3
    with ppf.Simulation(shape, precision="f32") as s:
        s.upload(*nan)
        assert all(np.isnan(a).all() for a in s.download())


@pytest.mark.parametrize("precision", ["f64", "f32"])
def test_observables_leave_out_nonfinite_cells(precision):
    """Non-finite cells are counted and add to no sum; their neighbours' cells
    still count towards mass and solid."""
    shape = (4, 5, 22)
    st = [a.copy() for a in smooth_state(shape, seed=3)]
    bad = [(0, 0, 0), (1, 2, 6), (1, 2, 7), (3, 4, 21), (2, 0, 20)]
    for i, p in enumerate(bad):
        st[i % 3][p] = [np.nan, np.inf, -np.inf][i % 3]
    with ppf.Simulation(shape, bc="noflux", precision=precision) as s:
        s.upload(*st)
        host = s.download()
        g = s.reduce()
    ok = np.isfinite(host[0]) & np.isfinite(host[1]) & np.isfinite(host[2])
    assert g["nonfinite"] == len(bad) == int((~ok).sum())
    S, L, c = (a[ok] for a in host)
    assert abs(g["mass"] - c.sum()) <= 1e-12 * c.sum()
    assert abs(g["solid"] - (S * S / (S * S + L * L)).sum()) <= (1e-12 if precision == "f64" else 1e-6) * S.size
    assert g["solid_cells"] == int((S > 0.5).sum())


@pytest.mark.parametrize("precision", ["f64", "f32"])
def test_device_arrays_that_cannot_be_used_in_place(precision):
    """Overlapping destinations and arrays off the 8-byte grid keep the copies'
    behaviour: the last copy wins, any alignment works."""
    import torch
    shape = (6, 9, 40)
    n = int(np.prod(shape))
    st = smooth_state(shape, seed=5)
    with ppf.Simulation(shape, precision=precision) as s:
        s.upload(*st)
        host = s.download()
        out = torch.zeros(2 * n, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        download_device(s, [out.data_ptr(), out.data_ptr(), out.data_ptr() + 8 * n])
        got = out.cpu().numpy()
        assert np.array_equal(got[:n].reshape(shape), host[1]) and np.array_equal(got[n:].reshape(shape), host[2])
        raw = torch.zeros(3 * 8 * n + 64, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        ptr = [raw.data_ptr() + 4 + 8 * n * f for f in range(3)]
        download_device(s, ptr)
        got = raw.cpu().numpy()
        for f in range(3):
            assert np.array_equal(got[4 + 8 * n * f:4 + 8 * n * (f + 1)].view(np.float64).reshape(shape), host[f])
        with ppf.Simulation(shape, precision=precision) as t:
            t.upload_device(ptr)
            assert all(np.array_equal(a, b) for a, b in zip(t.download(), host))
