"""The mixed form's implicit stages away from the measured workloads."""
import ctypes as C

import numpy as np
import pytest

from method_b200 import initial

pytestmark = pytest.mark.gpu


def sheet(integrator, **kw):
    return dict(model="srrmhd", nx=24, ny=40, xmin=-0.5, xmax=0.5, ymin=-1.0, ymax=1.0,
                endTime=3.0, cfl=0.4, Ng=4, gamma=4.0 / 3.0, sigma=1e3, weno=3, bcs="outflow",
                integrator=integrator, **kw)


@pytest.mark.parametrize("integrator", ["ssp2", "ssp3", "ssp2322"])
@pytest.mark.parametrize("cp", [1e154, 1e160, float("inf")])
def test_cleaning_rate_of_any_size(integrator, cp):
    """cp^2 near and beyond the largest double (no divergence cleaning): the
    plain form's result to 1e-6 (L1), without its solver as a fallback."""
    import method_b200 as mb
    p = initial.current_sheet(24, 40, Ng=4, seed=21)
    out = []
    for precision in ("fp64", "mixed"):
        sim = mb.Simulation(precision=precision, **sheet(integrator, cp=cp))
        sim.set_prims(p)
        sim.update_time(3)
        out.append(sim.state()[:2])
        st = sim.stats()
        assert st["status"] == 0 and st["implicit_failed"] == 0 and st["implicit_fallbacks"] == 0
        sim.close()
    for plain, mixed in zip(*out):
        assert np.abs(mixed - plain).sum() < 1e-6 * np.abs(plain).sum()


SOURCED = slice(8, 13)  # E, psi, phi: the planes of S(U1) that the mixed stage 2 writes


def ptr(a):
    return np.ascontiguousarray(a).ctypes.data_as(C.c_void_p)


def test_exact_stage2_reads_the_sourced_planes_alone(kernel_checks):
    """The queued exact solve of stage 2, and the separate combination, with
    NaN in the planes of S(U1) that are identically zero: the bits of the
    launch over all cells, and of the combination, with zeros there."""
    import method_b200 as mb
    cfg = sheet("ssp2")
    dt = 1e-3
    sim = mb.Simulation(**cfg)
    sim.set_prims(initial.current_sheet(24, 40, Ng=4, seed=21))
    sim.step(dt)
    cons, _, aux = sim.state()
    flux, source = sim.flux_F(), sim.source()
    N = cons[0].size
    nan = source.copy()
    nan[:8] = nan[13] = np.nan
    assert not np.any(source[:8]) and not np.any(source[13])
    inside = np.zeros(cons.shape[1:], bool)
    inside[4:-4, 4:-4] = True
    cells = np.flatnonzero(inside.ravel())[::7].astype(np.int32)
    u1 = cons * 1.0
    out = [np.zeros_like(cons), np.zeros_like(cons)]
    for n, s, o in ((-1, source, out[0]), (len(cells), nan, out[1])):
        assert kernel_checks.run_stage2(C.byref(sim.cfg), n, ptr(cells), ptr(cons), ptr(aux),
                                        ptr(u1), ptr(flux), ptr(s), C.c_double(dt),
                                        o.ctypes.data_as(C.c_void_p)) == 0
    every, queued = (o.reshape(14, N) for o in out)
    assert np.array_equal(queued[:, cells], every[:, cells])
    rest = np.setdiff1d(np.arange(N), cells)
    assert not np.any(queued[:, rest])

    out = [cons.copy(), cons.copy()]
    for s, o in ((source, out[0]), (nan, out[1])):
        assert kernel_checks.run_ssp2_combine(C.byref(sim.cfg), o.ctypes.data_as(C.c_void_p),
                                              ptr(flux), ptr(flux), ptr(s), ptr(source),
                                              C.c_double(dt)) == 0
    assert np.array_equal(*out) and not np.array_equal(out[0], cons)
    sim.close()


def strong_field(sim, B):
    """Where B^2 exceeds rho h W^2 and the conductivity is high, the fast solve's
    iteration on E with v frozen does not converge."""
    X, Y, _ = np.meshgrid(*(np.linspace(0, 1, n) for n in (sim.Nx, sim.Ny, sim.Nz)), indexing="ij")
    p = sim.zeros(sim.Nprims)
    p[0] = p[4] = 1.0
    p[1], p[2], p[3] = 0.1 * np.sin(2 * np.pi * Y), -0.1 * np.cos(2 * np.pi * X), 0.05
    p[5], p[6], p[7] = 0.3, B * np.exp(-((X - 0.5) / 0.2) ** 2), 0.2
    p[8] = -(p[2] * p[7] - p[3] * p[6])
    p[9] = -(p[3] * p[5] - p[1] * p[7])
    p[10] = -(p[1] * p[6] - p[2] * p[5])
    return p


@pytest.mark.parametrize("integrator", ["ssp2", "ssp3", "ssp2322"])
@pytest.mark.parametrize("nx,ny,nz", [(24, 40, 0), (50, 0, 0), (12, 6, 5)])
@pytest.mark.parametrize("B", [2.0, 5.0])
def test_cells_that_fall_back_to_the_exact_solve(integrator, nx, ny, nz, B):
    """A part of the cells leaves the fast implicit solves unconverged and is
    solved as in the plain form: its result within the tolerance of those
    solves (1.5e-7 of a cell's state a stage)."""
    import method_b200 as mb
    out = []
    for precision in ("fp64", "mixed"):
        sim = mb.Simulation(precision=precision, **dict(sheet(integrator), nx=nx, ny=ny, nz=nz,
                                                        sigma=1e4))
        sim.set_prims(strong_field(sim, B))
        sim.step(1e-3)
        st = sim.stats()
        assert st["implicit_failed"] == 0 and st["c2p_unconverged"] == 0
        out.append(sim.state()[0])
        sim.close()
    assert 0 < st["implicit_fallbacks"] < st["implicit_cells"]
    plain, mixed = out
    d = np.linalg.norm(mixed - plain, axis=0) / np.linalg.norm(plain, axis=0)
    assert d.max() < 1e-6, d.max()


def test_ensemble_cells_that_fall_back():
    """An ensemble member's queue gives the bits of a single run's."""
    import method_b200 as mb
    cfg = dict(sheet("ssp2", precision="mixed"), sigma=1e4)
    sim = mb.Simulation(**cfg)
    p = strong_field(sim, 5.0)
    sim.set_prims(p)
    sim.update_time(2)
    assert sim.stats()["implicit_fallbacks"] > 0
    ens = mb.Ensemble([cfg, cfg])
    for m in range(2):
        ens.set_prims(m, p)
    ens.step(2)
    for m in range(2):
        for a, b in zip(ens.state(m), sim.state()):
            assert np.array_equal(a, b)
    ens.close()
    sim.close()
