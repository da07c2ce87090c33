"""The algorithmic bytes that the step profiler books for SSP2's stages: one
read of each plane a launch needs, one write of each it leaves."""
import pytest

from method_b200 import initial

pytestmark = pytest.mark.gpu

FLUX = 14 + 4 + 6          # cons, prims 1-4, aux 4-8 and 10
CLOSE = FLUX + 3 * 14 + 5  # + flux1, U^n, the sourced planes of S(U1); the state out


@pytest.mark.parametrize("kw,want", [
    (dict(precision="mixed"), dict(fvs2d_fp32=(FLUX + 14 + CLOSE) / 2,
                                   # cons, flux1, 3 of U1, aux 4-6 and 10; state, source
                                   imex_newton_stage2=14 + 14 + 3 + 4 + 14 + 5)),
    (dict(precision="mixed", guess="mlp"),
     # cons, flux1, the source, aux[10], the network's Z; the state
     dict(fvs2d_fp32=(FLUX + 14 + CLOSE) / 2, imex_newton_stage2=14 + 14 + 5 + 1 + 1 + 14)),
    (dict(), dict(fvs2d_fp64=(FLUX + 14 + CLOSE) / 2,
                  # cons, U1, flux1, the source, aux[10]; the state
                  imex_hybrd_stage2=14 + 14 + 14 + 5 + 1 + 14)),
    # cons in and out, both fluxes, the sourced planes of S(U1), S(U2)
    (dict(ny=0), dict(ssp2_combine=28 + 14 + 14 + 5 + 14)),
])
def test_ssp2_bytes(kw, want):
    import method_b200 as mb
    cfg = dict(dict(model="srrmhd", integrator="ssp2", nx=24, ny=40, xmin=-0.5, xmax=0.5, ymin=-1.0,
                    ymax=1.0, gamma=4.0 / 3.0, sigma=100.0, bcs="outflow"), **kw)
    sim = mb.Simulation(**cfg)
    if "guess" in cfg:
        P, S, _ = mb.train_guess(model="srrmhd", iterations=20, n_samples=1 << 14)
        sim.set_mlp(P, S)
    p = initial.current_sheet(24, 40, Ng=4, seed=3)
    sim.set_prims(p if cfg["ny"] else p[:, :, :1])
    got = {k["name"]: k["bytes_per_launch"] for k in sim.profile_step(1e-4, 1)}
    cells = 24 * (cfg["ny"] or 1)
    for name, doubles in want.items():
        assert got[name] == 8 * doubles * cells, (name, got[name] / 8 / cells)
    sim.close()
