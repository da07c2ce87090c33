"""The mixed form's implicit stages away from the measured workloads."""
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
