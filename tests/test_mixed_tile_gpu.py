"""The FP32 flux tile in pairs of variables (WENO3/5) against the plain FP64
form, at the edges of its 8 x 32 tile, for an odd and an even number of
variables, and with states scaled by powers of 4 (density, pressure and
energy by s, fields by sqrt(s): a symmetry of the equations), whose smoothness
indicators lie far below, around and above one.

Bound: a reconstructed face is a handful of FP32 operations on values of at
most F = max(|flux|, |U|) (|coefficients| sum to 10/3, about 20 roundings), so a
conserved variable is off by at most dt (1/dx + 1/dy) * 2 faces * 20 * 2^-24 F a
stage; the corrector's inputs carry the predictor's error through the
recovery, allowed for with a factor 6 in all.  The flux of the charge density
is J, whose W sigma (E + v x B - (v.E) v) carries the errors of E, B and v into
the corrector: 8 sigma times the fields' bound, once more dt (1/dx + 1/dy) 2.
(SRRMHD is not scaled up: its
plain recovery's absolute tolerance of 1e-12 is then below rounding.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(8, 32), (7, 31), (9, 33), (4, 4), (33, 95)]


def blast(sim, log4=0):
    s = 4.0 ** log4
    p = sim.zeros(sim.Nprims)
    X, Y = np.meshgrid(np.linspace(0, 1, sim.Nx), np.linspace(0, 1, sim.Ny), indexing="ij")
    X, Y = X[:, :, None], Y[:, :, None]
    hot = (X - 0.5) ** 2 + (Y - 0.4) ** 2 < 0.06
    p[0] = s * np.where(hot, 1.0, 0.2)
    p[4] = s * np.where(hot, 2.0, 0.5)
    p[1], p[2] = 0.3 * np.sin(7 * Y), -0.2 * np.cos(5 * X)
    p[5], p[6], p[7] = 0.4 * 2.0 ** log4, 0.3 * 2.0 ** log4 * np.cos(5 * X), 0.1 * 2.0 ** log4
    if sim.Nprims > 8:
        p[8] = -(p[2] * p[7] - p[3] * p[6])
        p[9] = -(p[3] * p[5] - p[1] * p[7])
        p[10] = -(p[1] * p[6] - p[2] * p[5])
    return p


def config(model, nx, ny, weno, bcs, integrator="rk2", sigma=10.0, **kw):
    return dict(model=model, nx=nx, ny=ny, xmin=0.0, xmax=1.0, ymin=0.0, ymax=1.0, endTime=1.0,
                cfl=0.4, Ng=4, gamma=4.0 / 3.0, sigma=sigma, weno=weno, bcs=bcs,
                integrator=integrator, **kw)


def check(cfg, log4=0, solver=0.0):
    """One step in both forms; every group of variables that scales alike
    within its bound, plus `solver` times its size."""
    import method_b200 as mb
    dt = 0.1 / max(cfg["nx"], cfg["ny"])
    out, F = [], 0.0
    for precision in ("fp64", "mixed"):
        sim = mb.Simulation(precision=precision, **cfg)
        p = blast(sim, log4)
        sim.set_prims(p)
        sim.step(dt)
        out.append(sim.state()[0])
        sim.close()
    # the fluxes' size at the start (the Hybrid model's lie between the two others')
    model = "srmhd" if cfg["model"] == "srmhd" else "srrmhd"
    sim = mb.Simulation(**config(model, cfg["nx"], cfg["ny"], cfg["weno"], cfg["bcs"],
                                 sigma=cfg["sigma"]))
    sim.set_prims(p)
    for dir in (0, 1):
        F = np.maximum(F, np.abs(sim.flux_vector(dir)).max(axis=(1, 2, 3)))
    sim.close()
    plain, mixed = out
    assert np.all(np.isfinite(mixed))
    F = np.maximum(F, np.abs(plain).max(axis=(1, 2, 3)))
    rate = dt * (cfg["nx"] + cfg["ny"]) * 2
    eps = 6 * rate * 20 * 2.0 ** -24 + solver
    # fields and E scale by sqrt(s), the rest by s
    fields = [5, 6, 7, 8] if model == "srmhd" else [5, 6, 7, 8, 9, 10, 11, 12]
    bounds = [(fields, eps * F[fields].max()), ([0, 1, 2, 3, 4], eps * F[:5].max())]
    if model == "srrmhd":
        bounds.append(([13], eps * F[13] + rate * 8 * cfg["sigma"] * bounds[0][1]))
    for group, bound in bounds:
        assert np.abs(mixed[group] - plain[group]).max() <= bound, (group, bound)


@pytest.mark.parametrize("nx,ny", SIZES)
@pytest.mark.parametrize("weno", [3, 5])
@pytest.mark.parametrize("bcs", ["periodic", "outflow", "flow"])
@pytest.mark.parametrize("model,log4", [("srmhd", -10), ("srmhd", 0), ("srmhd", 3),
                                        ("srrmhd", -10), ("srrmhd", 0)])
def test_mixed_step_at_tile_edges(nx, ny, weno, model, bcs, log4):
    check(config(model, nx, ny, weno, bcs), log4)


@pytest.mark.parametrize("nx,ny", SIZES)
@pytest.mark.parametrize("weno", [3, 5])
@pytest.mark.parametrize("model,integrator,sigma,solver",
                         [("srrmhd", "ssp2", 10.0, 2e-6), ("hybrid", "rk2", 170.0, 1e-7),
                          ("hybrid", "rksplit2", 120.0, 1e-7)])
def test_mixed_step_of_other_stages_at_tile_edges(nx, ny, weno, model, integrator, sigma, solver):
    """SSP2's closing combination in the tile's epilogue, and the Hybrid
    model's tile.  Beside the tile's error stand the plain form's solvers:
    hybrd1's tolerance of 1.5e-7 of a cell's state for each of SSP2's two stages,
    magnified by their stiffness, and of 1.4e-8 for the Hybrid's recoveries."""
    kw = dict(useREGIME=False) if model == "hybrid" else {}
    check(config(model, nx, ny, weno, "outflow", integrator, sigma, **kw), 0, solver)
