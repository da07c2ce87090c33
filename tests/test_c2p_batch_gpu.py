"""Batched SRMHD recovery at the edges of its launches (blocks of 128 cells)."""
import ctypes as C

import numpy as np
import pytest

from method_b200 import initial

pytestmark = pytest.mark.gpu

G = 4.0 / 3.0


def conserved(p):
    rho, v, pr, B = p[0], p[1:4], p[4], p[5:8]
    W = 1 / np.sqrt(1 - (v * v).sum(0))
    h = 1 + pr / rho * (G / (G - 1))
    b0 = W * (v * B).sum(0)
    b = B / W + b0 * v
    bsq = ((B * B).sum(0) + b0 * b0) / (W * W)
    q = (rho * h + bsq) * W * W
    tau = q - (pr + bsq / 2) - b0 * b0 - rho * W
    return np.concatenate([[rho * W], q * v - b0 * b, [tau], B, [0 * rho]]), h


@pytest.mark.parametrize("n", [1, 31, 128, 129, 1000])
@pytest.mark.parametrize("method,guess", [(0, 0), (1, 0), (1, 2)])
def test_batch_recovers_generating_states(n, method, guess):
    """Newton from a previous state 1% off and from a cold start, the Powell
    hybrid from the state itself.  The inversion magnifies the rounding of the
    conserved state by up to W^4 (1 + b^2 / rho) of a few 1e6: 1e-8."""
    import torch

    from method_b200 import _lib
    L = _lib.load()
    p = initial.random_c2p_states(n, seed=n)
    cons, h = conserved(p)
    pg, ag = np.zeros((8, n)), np.zeros((13, n))
    off = 0.0 if method == 0 else 0.01
    pg[0], pg[1:4], ag[0] = p[0] * (1 + off), p[1:4] * (1 - off), h * (1 + off)
    dc, dp, da = (torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (cons, pg, ag))
    st = _lib.C2PBatchStats()
    rc = L.mth_c2p_batch(G, n, dc.data_ptr(), dp.data_ptr(), da.data_ptr(), method, guess, None,
                         None, None, C.byref(st))
    assert rc == 0 and st.cells == n and st.unconverged == 0
    got, aux = dp.cpu().numpy(), da.cpu().numpy()
    assert np.max(np.abs(got[0] - p[0]) / p[0]) < 1e-8
    assert np.max(np.abs(got[1:4] - p[1:4])) < 1e-8
    assert np.array_equal(got[5:8], p[5:8])
    assert np.max(np.abs(aux[0] - h) / h) < 1e-7  # h - 1 is down to 4e-3 of h


@pytest.mark.parametrize("log4,guess", [(-123, 0), (-123, 2), (-100, 0), (100, 0), (122, 2)])
def test_batch_recovers_states_of_any_scale(log4, guess):
    """Newton on states scaled by powers of 4 (density, pressure and energy by s,
    fields by sqrt(s): a symmetry of the equations, exact in binary) up to
    where Z^2 (Z + B^2)^2 spans the range of doubles; same bound as above."""
    import torch

    from method_b200 import _lib
    L = _lib.load()
    n, s = 4096, 4.0 ** log4
    p = initial.random_c2p_states(n, seed=1)
    p[[0, 4]] *= s
    p[5:8] *= 2.0 ** log4
    cons, h = conserved(p)
    pg, ag = np.zeros((8, n)), np.zeros((13, n))
    pg[0], pg[1:4], ag[0] = p[0] * 1.01, p[1:4] * 0.99, h * 1.01
    dc, dp, da = (torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (cons, pg, ag))
    st = _lib.C2PBatchStats()
    rc = L.mth_c2p_batch(G, n, dc.data_ptr(), dp.data_ptr(), da.data_ptr(), 1, guess, None, None,
                         None, C.byref(st))
    assert rc == 0 and st.cells == n and st.unconverged == 0
    got = dp.cpu().numpy()
    assert np.max(np.abs(got[0] - p[0]) / p[0]) < 1e-8
    assert np.max(np.abs(got[1:4] - p[1:4])) < 1e-8


def test_hybrid_register_variants_agree():
    """The Powell hybrid's kernels on either side of their dispatch (16 CTAs of
    128 cells per SM): the same cells give the same bits."""
    import torch

    from method_b200 import _lib
    L = _lib.load()
    line = 16 * 128 * torch.cuda.get_device_properties(0).multi_processor_count
    p = initial.random_c2p_states(line, seed=2)
    cons, h = conserved(p)
    out = []
    for n in (line - 128, line):
        pg, ag = np.zeros((8, n)), np.zeros((13, n))
        pg[:5], ag[0] = p[:5, :n], h[:n]
        dc, dp, da = (torch.from_numpy(np.ascontiguousarray(x)).cuda()
                      for x in (cons[:, :n], pg, ag))
        st = _lib.C2PBatchStats()
        rc = L.mth_c2p_batch(G, n, dc.data_ptr(), dp.data_ptr(), da.data_ptr(), 0, 0, None, None,
                             None, C.byref(st))
        assert rc == 0 and st.unconverged == 0
        out.append((dp.cpu().numpy()[:, :line - 128], da.cpu().numpy()[:, :line - 128]))
    for a, b in zip(*out):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("n", [1, 31, 33, 127, 128, 129, 1000])
@pytest.mark.parametrize("method,guess", [(0, 0), (1, 0), (1, 2)])
@pytest.mark.parametrize("bad", [False, True])
def test_batch_statistics(n, method, guess, bad):
    """n copies of one cell count n times what one counts: cells, iterations and,
    for a cell that does not converge, failures and fallbacks."""
    import torch

    from method_b200 import _lib
    L = _lib.load()
    p = initial.random_c2p_states(1, seed=5)
    cons, h = conserved(p)
    if bad:
        cons[1] = 100 * (cons[0] + cons[4])  # |S| far beyond tau + D
    pg, ag = np.zeros((8, 1)), np.zeros((13, 1))
    pg[:5], ag[0] = p[:5] * (0.99 if method else 1.0), h
    counts = []
    for m in (1, n):
        dc, dp, da = (torch.from_numpy(np.repeat(x, m, axis=1)).cuda() for x in (cons, pg, ag))
        st = _lib.C2PBatchStats()
        rc = L.mth_c2p_batch(G, m, dc.data_ptr(), dp.data_ptr(), da.data_ptr(), method, guess, None,
                             None, None, C.byref(st))
        assert rc == (1 if bad else 0)
        counts.append(np.array([st.cells, st.iterations, st.unconverged, st.fallbacks]))
    assert counts[0][0] == 1 and counts[0][1] > 0 and counts[0][2] == bad
    assert np.array_equal(counts[1], n * counts[0])
