"""The plain form's WENO3/5 weights and face scaling divide without branches
where the operands allow it (csrc/div64.cuh) and by IEEE division elsewhere;
both must give the bits of the oracle (oracle/oracle.c, plain C), in the
generic path and in both fused tiles, at ragged tile edges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

G = 4.0 / 3.0


def config(nx, ny, nz=0, weno=5, bcs="periodic"):
    return dict(model="srmhd", nx=nx, ny=ny, nz=nz, xmin=0.0, xmax=1.0, ymin=0.0, ymax=1.3,
                zmin=0.0, zmax=0.7, endTime=1.0, cfl=0.3, Ng=4, gamma=G, weno=weno, bcs=bcs,
                integrator="rk2")


@pytest.mark.parametrize("weno", [3, 5])
@pytest.mark.parametrize("nx,ny,nz", [(40, 0, 0), (9, 33, 0), (6, 7, 5)])
@pytest.mark.parametrize("scale", [1.0, 1e-9, 1e-140, 1e66, 1e67, 1e130])
def test_flux_of_any_size_matches_oracle(weno, nx, ny, nz, scale):
    """FVS::F of states whose smoothness indicators are zero (constant
    regions), ordinary, beyond the branch-free range (indicators above 2^448)
    and around its edge."""
    import method_b200 as mb
    from oracle import port
    cfg = config(nx, ny, nz, weno)
    rng = np.random.default_rng(3)
    sim = mb.Simulation(**cfg)
    p, c, a = (sim.zeros(n) for n in (sim.Nprims, sim.Ncons, sim.Naux))
    c[:] = scale * (rng.random(c.shape) - 0.5)
    c[:, : c.shape[1] // 3] = scale  # constant: every indicator is exactly zero
    c[3] = 0.0
    p[1:4] = 0.6 * (rng.random(p[1:4].shape) - 0.5)
    p[4] = scale * rng.random(p[4].shape)
    p[5:7] = rng.random(p[5:7].shape) - 0.5
    a[1] = 1.0 + rng.random(a[1].shape)
    a[4:9] = rng.random(a[4:9].shape) - 0.5
    sim.upload(c, p, a)
    got = sim.flux_F()
    sim.close()
    safe = p.copy()
    safe[0], safe[4] = 1.0, 1.0
    o = port.PortSim(safe, **cfg)
    want = o.flux_F(c, p, a)
    o.close()
    assert np.array_equal(got, want, equal_nan=True)


@pytest.mark.parametrize("weno", [3, 5])
@pytest.mark.parametrize("nx,ny", [(8, 32), (7, 31), (9, 33), (17, 70), (100, 300), (100, 736)])
@pytest.mark.parametrize("model,bcs", [("srmhd", "periodic"), ("srmhd", "outflow"),
                                       ("srrmhd", "flow")])
def test_fused_step_matches_oracle(weno, nx, ny, model, bcs):
    """One RK2 step of a blast with constant regions, by a CTA per variable, by
    CTAs of three (100 x 300: 130 tiles) and by the grouped tile (100 x 736:
    299 tiles)."""
    import method_b200 as mb
    from oracle import port
    cfg = dict(config(nx, ny, 0, weno, bcs), model=model, sigma=5.0)
    sim = mb.Simulation(**cfg)
    p = sim.zeros(sim.Nprims)
    X, Y = np.meshgrid(np.linspace(0, 1, sim.Nx), np.linspace(0, 1, sim.Ny), indexing="ij")
    hot = ((X - 0.5) ** 2 + (Y - 0.4) ** 2 < 0.06)[:, :, None]
    # SRRMHD's secant recovery does not take the strong blast
    p[0] = np.where(hot, 1.0, 0.1 if model == "srmhd" else 0.8)
    p[4] = np.where(hot, 10.0, 0.05) if model == "srmhd" else np.where(hot, 1.0, 0.7)
    p[1] = 0.3 * np.sin(7 * Y)[:, :, None]
    p[5], p[6] = 0.2, 0.1 * np.cos(5 * X)[:, :, None]
    if model == "srrmhd":
        p[9], p[10] = p[1] * p[7], -p[1] * p[6]
    sim.set_prims(p)
    o = port.PortSim(p, **cfg)
    dt = 0.05 / max(nx, ny)
    sim.step(dt)
    o.step_dt(dt)
    for name, got, want in zip(("cons", "prims", "aux"), sim.state(), o.state()):
        assert np.array_equal(got, want), name
    sim.close()
    o.close()


BAND = 2.0 - 2.0 ** -16  # a significand that no branch-free quotient takes


@pytest.mark.parametrize("dx,dy", [(0.0, 0.1), (0.1, 0.0), (-0.1, 0.1), (float("nan"), 0.1),
                                   (float("inf"), 0.1), (BAND, 2.0), (0.125, BAND / 16),
                                   (2.0 ** -99, 2.0 ** -99), (2.0 ** -101, 2.0 ** -101),
                                   (2.0 ** 101, 2.0 ** 101)])
@pytest.mark.parametrize("nx,ny", [(20, 24), (2368, 4)])
def test_cell_size_of_any_kind_matches_oracle(dx, dy, nx, ny):
    """Face fluxes, zeros among them, over cell sizes that are zero, negative,
    NaN or infinite (0 / 0 is NaN), and on either side of the branch-free
    quotients' limits: what IEEE division gives, by a CTA per variable and by
    the grouped tile (296 tiles; few cells, as the retry of failed recoveries is
    serial)."""
    import method_b200 as mb
    from oracle import port
    cfg = dict(config(nx, ny, 0, 3, "outflow"), xmax=dx * nx, ymax=dy * ny)
    dt = 1e-2 * min(d for d in (dx, dy) if d > 0)
    sim = mb.Simulation(**cfg)
    p = sim.zeros(sim.Nprims)
    p[0], p[4] = 1.0, 1.0
    p[1, sim.Nx // 2:] = 0.1 * np.sin(np.arange(sim.Ny))[:, None]
    p[5, sim.Nx // 2:] = 0.3
    sim.set_prims(p)
    o = port.PortSim(p, **cfg)
    sim.step(dt)
    o.step_dt(dt)
    assert np.array_equal(sim.state()[0], o.state()[0], equal_nan=True)
    sim.close()
    o.close()
