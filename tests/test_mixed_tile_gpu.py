"""The FP32 flux tile in pairs of variables (WENO3/5) against the plain FP64
form, at the edges of its 8 x 32 tile, for an odd and an even number of
variables, and with states scaled by powers of 4 (density, pressure and
energy by s, fields by sqrt(s): a symmetry of the equations), whose smoothness
indicators lie far below, around and above one.

Bound: a reconstructed face is a handful of FP32 operations on values of at
most F = max|flux| (|coefficients| sum to 10/3, about 20 roundings), so a
conserved variable is off by at most dt (1/dx + 1/dy) * 2 faces * 20 * 2^-24 F a
stage; the corrector's inputs carry the predictor's error through the
recovery, allowed for with a factor 6 in all.  (SRRMHD is not scaled up: its
plain recovery's absolute tolerance of 1e-12 is then below rounding.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(8, 32), (7, 31), (9, 33), (4, 4), (33, 95)])
@pytest.mark.parametrize("weno", [3, 5])
@pytest.mark.parametrize("bcs", ["periodic", "outflow", "flow"])
@pytest.mark.parametrize("model,log4", [("srmhd", -10), ("srmhd", 0), ("srmhd", 3),
                                        ("srrmhd", -10), ("srrmhd", 0)])
def test_mixed_step_at_tile_edges(nx, ny, weno, model, bcs, log4):
    import method_b200 as mb
    s = 4.0 ** log4
    cfg = dict(model=model, nx=nx, ny=ny, xmin=0.0, xmax=1.0, ymin=0.0, ymax=1.0, endTime=1.0,
               cfl=0.4, Ng=4, gamma=4.0 / 3.0, sigma=10.0, weno=weno, bcs=bcs, integrator="rk2")
    dt = 0.1 / max(nx, ny)
    out = []
    for precision in ("fp64", "mixed"):
        sim = mb.Simulation(precision=precision, **cfg)
        p = sim.zeros(sim.Nprims)
        X, Y = np.meshgrid(np.linspace(0, 1, sim.Nx), np.linspace(0, 1, sim.Ny), indexing="ij")
        X, Y = X[:, :, None], Y[:, :, None]
        hot = (X - 0.5) ** 2 + (Y - 0.4) ** 2 < 0.06
        p[0] = s * np.where(hot, 1.0, 0.2)
        p[4] = s * np.where(hot, 2.0, 0.5)
        p[1], p[2] = 0.3 * np.sin(7 * Y), -0.2 * np.cos(5 * X)
        p[5], p[6], p[7] = 0.4 * 2.0 ** log4, 0.3 * 2.0 ** log4 * np.cos(5 * X), 0.1 * 2.0 ** log4
        if model == "srrmhd":
            p[8] = -(p[2] * p[7] - p[3] * p[6])
            p[9] = -(p[3] * p[5] - p[1] * p[7])
            p[10] = -(p[1] * p[6] - p[2] * p[5])
        sim.set_prims(p)
        sim.step(dt)
        out.append(sim.state()[0])
        sim.close()
    plain, mixed = out
    assert np.all(np.isfinite(mixed))
    # fields and E scale by sqrt(s), the rest by s: each group against its own size
    fields = {"srmhd": [5, 6, 7, 8], "srrmhd": [5, 6, 7, 8, 9, 10, 11, 12]}[model]
    rest = [v for v in range(5)]
    for group in (fields, rest):
        F = np.abs(plain[group]).max()
        bound = 6 * dt * (nx + ny) * 2 * 20 * 2.0 ** -24 * F
        assert np.abs(mixed[group] - plain[group]).max() <= bound, (group, F)
