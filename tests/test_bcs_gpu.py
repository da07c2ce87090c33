"""Boundary conditions on the device state against the oracle, one to three
dimensions, sizes at and around the ghost depth."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bcs", ["outflow", "periodic", "flow"])
@pytest.mark.parametrize("nx,ny,nz", [(4, 0, 0), (33, 0, 0), (4, 5, 0), (31, 70, 0), (4, 4, 5),
                                      (9, 6, 17)])
@pytest.mark.parametrize("model", ["srmhd", "srrmhd"])
def test_ghost_cells_match_oracle(bcs, nx, ny, nz, model):
    import method_b200 as mb
    from oracle import port
    cfg = dict(model=model, nx=nx, ny=ny, nz=nz, xmin=0.0, xmax=1.0, ymin=0.0, ymax=1.0, zmin=0.0,
               zmax=1.0, endTime=1.0, cfl=0.4, Ng=4, gamma=4.0 / 3.0, sigma=1.0, weno=3, bcs=bcs,
               integrator="rk2")
    sim = mb.Simulation(**cfg)
    rng = np.random.default_rng(1)
    arrays = [rng.random(sim.shape(n)) for n in (sim.Ncons, sim.Nprims, sim.Naux)]
    sim.upload(*arrays)
    sim.apply_bcs()
    got = sim.state()
    sim.close()
    p = np.zeros_like(arrays[1])
    p[0], p[4] = 1.0, 1.0
    o = port.PortSim(p, **cfg)
    want = [a.copy() for a in arrays]
    o.apply_bcs(*want)
    o.close()
    for g, w in zip(got, want):
        assert np.array_equal(g, w)
