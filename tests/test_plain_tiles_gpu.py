"""The plain flux stage in each form that its dispatch by tiles per SM (148 SMs)
chooses -- a CTA per variable, per group of three or five, per tile, and the
grouped tile in passes -- beyond the RK2 WENO3/5 runs of
test_weno_division_gpu.py.  Every form must give the bits of the oracle
(oracle/oracle.c) or, for the Hybrid model, of the per-direction path."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def config(model, nx, ny, weno, integrator="rk2", **kw):
    return dict(model=model, nx=nx, ny=ny, xmin=0.0, xmax=1.0, ymin=0.0, ymax=1.3, endTime=1.0,
                cfl=0.3, Ng=max(4, (weno + 3) // 2), gamma=4.0 / 3.0, weno=weno,
                integrator=integrator, **kw)


def smooth(sim, seed=3):
    r = np.random.default_rng(seed)
    X, Y, _ = np.meshgrid(*(np.linspace(0, 1, n) for n in (sim.Nx, sim.Ny, sim.Nz)), indexing="ij")
    p = sim.zeros(sim.Nprims)
    p[0] = 1.0 + 0.1 * r.random(X.shape)
    p[4] = 1.0 + 0.2 * np.cos(9 * X)
    p[1], p[2], p[3] = 0.3 * np.sin(7 * Y), -0.2 * np.cos(5 * X), 0.1
    p[5], p[6], p[7] = 0.4, 0.3 * np.cos(5 * X), 0.1 * np.sin(3 * Y)
    if sim.Nprims > 8:
        p[8] = -(p[2] * p[7] - p[3] * p[6])
        p[9] = -(p[3] * p[5] - p[1] * p[7])
        p[10] = -(p[1] * p[6] - p[2] * p[5])
    return p


def against_oracle(cfg, dt):
    import method_b200 as mb
    from oracle import port
    sim = mb.Simulation(**cfg)
    p = smooth(sim)
    sim.set_prims(p)
    o = port.PortSim(p, **cfg)
    sim.step(dt)
    o.step_dt(dt)
    for name, got, want in zip(("cons", "prims", "aux"), sim.state(), o.state()):
        assert np.array_equal(got, want), name
    sim.close()
    o.close()


# 4, 130, 280 and 300 tiles of 8 x 32
@pytest.mark.parametrize("nx,ny", [(9, 33), (100, 300), (2240, 5), (2393, 4)])
@pytest.mark.parametrize("weno", [7, 9, 11])
@pytest.mark.parametrize("model", ["srmhd", "srrmhd"])
def test_high_order_step(model, weno, nx, ny):
    against_oracle(config(model, nx, ny, weno, bcs="outflow", sigma=5.0), 0.05 / max(nx, ny))


@pytest.mark.parametrize("nx,ny", [(9, 33), (75, 160), (2393, 4)])
@pytest.mark.parametrize("integrator", ["ssp2", "rksplit"])
def test_resistive_integrators_step(integrator, nx, ny):
    """SSP2's closing combination in the stage's epilogue (a share of the
    variables per CTA), and RKSplit."""
    against_oracle(config("srrmhd", nx, ny, 3, integrator, bcs="outflow", sigma=50.0),
                   0.05 / max(nx, ny))


@pytest.mark.parametrize("nx,ny", [(9, 33), (75, 160), (2393, 4)])
@pytest.mark.parametrize("weno", [3, 5])
@pytest.mark.parametrize("sigma", [120.0, 170.0])
def test_hybrid_step_from_the_per_direction_flux(nx, ny, weno, sigma):
    """RK2 by hand from FVS::F, whose path is the per-direction one, and the
    recovery of the same handle: the fused step's bits."""
    import method_b200 as mb
    cfg = config("hybrid", nx, ny, weno, bcs="outflow", sigma=sigma, useREGIME=False)
    dt = 0.05 / max(nx, ny)
    sim = mb.Simulation(**cfg)
    sim.set_prims(smooth(sim))
    start = sim.state()
    sim.step(dt)
    fused = sim.state()

    n = cfg["Ng"]
    inside = (slice(None), slice(n, -n), slice(n, -n))

    def recovered(cons, prims, aux):
        sim.upload(cons, prims, aux)
        sim.c2p()
        sim.apply_bcs()
        return sim.state()

    sim.upload(*start)
    u1 = start[0].copy()
    u1[inside] = start[0][inside] - dt * sim.flux_F()[inside]
    first = recovered(u1, *start[1:])
    u2 = start[0].copy()
    u2[inside] = 0.5 * (start[0][inside] + first[0][inside] - dt * sim.flux_F()[inside])
    for a, b in zip(fused, recovered(u2, *start[1:])):
        assert np.array_equal(a[inside], b[inside])
    sim.close()
