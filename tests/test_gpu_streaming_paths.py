"""The paths that larger grids take, on grids that the oracle solves quickly:
list sweeps with a pre-phase and the window rule, the full-coefficient sweeps,
and the launches of the solve without allocation. A sweep shape named by the
"variant" option, or a grid too large for the scratch array, keeps the solve off
the resident kernel."""
import numpy as np
import pytest

import qesb
from oracle import oracle as O

pytestmark = pytest.mark.gpu

TILED, BULK, ZM, ZMB = 0, 18, 51, 59  # a fused tile shape, bulk-copy rows, tensor-map z-march shapes


def _city(nx, ny, nz, seed=5):
    d = qesb.Domain(nx, ny, nz, 2.0, 2.0, 1.0, qesb.city_dz(nz, 1.0, 1.03))
    c = qesb.city_random(d, seed, 12, fp=(6, 20), h=(4, 20))
    return qesb.city_build(d, c.buildings, c.inflow)


def _check_winds(w, L, out):
    for t, a in zip(out, O.correct(w.domain, w, L)):
        np.testing.assert_array_equal(t.cpu().numpy(), a)


def _winds(ws):
    import torch

    return [[torch.zeros(w.domain.numFaceCentered(), device="cuda") for _ in range(3)] for w in ws]


@pytest.mark.parametrize("variant", [-1, BULK, ZM, ZMB])
def test_batch_phases_and_window_rule(variant):
    """A start stage, a pre-phase and the window rule over a list whose domains
    have all, some and none of them, and leave it one by one. Without a shape
    named (-1) the large domain is the list and the others are resident."""
    dims = [(70, 45, 21), (131, 40, 15), (40, 33, 9), (300, 300, 50)]
    ws = [_city(*g) for g in (dims if variant < 0 else dims[:3])]
    cfg = [((1.6, 5), (1.85, 1e-9, 12)), (None, (1.9, 3e-1, 400)), (None, None), (None, (1.85, 1e-9, 12))]
    K, wtol = 8, 1.0 if variant < 0 else 0.05
    solvers = [qesb.Solver_B200(w.domain, 1e-9) for w in ws]
    out = _winds(ws)
    try:
        for s, w, (start, pre) in zip(solvers, ws, cfg):
            s.set_inputs(w)
            s.set_window_rule(K, wtol)
            if pre:
                s.set_prephase(*pre)
            if start:
                s.set_prephase_start(*start)
        if variant >= 0:
            solvers[0].set_option("variant", variant)
        st = qesb.solve_batch(solvers, 1500, *[[o[q].data_ptr() for o in out] for q in range(3)])
        lams = [s.lambda_ for s in solvers]
    finally:
        for s in solvers:
            s.close()
    for w, (start, pre), x, lam, o in zip(ws, cfg, st, lams, out):
        d = w.domain
        R = O.divergence(d, w)
        L, n_pre = None, 0
        if start:
            L, n, *_ = O.sor(d, w, R, -1.0, start[1], omega=start[0])
            n_pre += n
        if pre:
            L, n, *_ = O.sor(d, w, R, pre[1], pre[2], omega=pre[0], lam=L)
            n_pre += n
        L, it, stop, drift = O.sor_window(d, w, R, 1e-9, 1500, K, wtol, lam=L)
        assert (x["pre_iterations"], x["iterations"], x["converged"], x["window_drift"]) == (n_pre, it, stop, drift)
        assert stop == 2
        np.testing.assert_array_equal(lam, L)
        _check_winds(w, L, o)


def test_batch_runs_the_shape_that_its_tuner_found():
    """The tuned shape, named as the batch's "variant": every domain's sweeps run in it."""
    ws = [_city(70, 45, 21), _city(131, 40, 15), _city(40, 33, 9)]
    solvers = [qesb.Solver_B200(w.domain, 0.05) for w in ws]
    try:
        for s, w in zip(solvers, ws):
            s.set_inputs(w)
        best, _ = qesb.autotune_batch(solvers)
        solvers[0].set_option("variant", best)
        st = qesb.solve_batch(solvers, 1500)
        lams = [s.lambda_ for s in solvers]
    finally:
        for s in solvers:
            s.close()
    for w, x, lam in zip(ws, st, lams):
        L, it, *_ = O.sor(w.domain, w, O.divergence(w.domain, w), 0.05, 1500)
        assert x["iterations"] == it and x["converged"] == 1
        assert x["launches"] >= 2 * max(y["iterations"] for y in st)  # two sweeps an iteration
        np.testing.assert_array_equal(lam, L)


@pytest.mark.parametrize("window", [None, (16, 5e-2)])
def test_full_coefficient_sweeps_stop(window):
    """run by run of 64 iterations, each of four launches: a stop by tolerance,
    a stop by the window rule, and the next solve from the kept lambda."""
    w = _city(72, 56, 24)
    d = w.domain
    R = O.divergence(d, w)
    tol, L = (1e-9, None) if window else (0.01, None)
    with qesb.Solver_B200(d, tol) as s:
        s.set_option("path", 0)
        s.set_option("variant", TILED)
        if window:
            s.set_window_rule(*window)
        for _ in range(2):
            st = s.solve(w, 600)
            if window:
                L, it, stop, drift = O.sor_window(d, w, R, tol, 600, *window, lam=L)
                assert (st["converged"], st["window_drift"]) == (stop, drift) and stop == 2
            else:
                L, it, *_ = O.sor(d, w, R, tol, 600, lam=L)
                assert st["converged"] == 1
            assert (st["path"], st["iterations"], st["launches"]) == (0, it, 2 + 4 * it)
            np.testing.assert_array_equal(s.lambda_, L)


def test_solve_without_allocation_on_a_grid_beyond_the_resident_scratch():
    """By its own launches: a count, then a stop by tolerance past the first 64
    iterations, with a smaller grid's resident solve on the same scratch between."""
    import torch

    big, small = _city(160, 144, 48), _city(70, 45, 21)
    lam0 = np.random.default_rng(3).standard_normal(big.domain.numCellCentered()).astype(np.float32)
    for w, tol, n, start in ((big, 1e-9, 9, lam0), (small, 1e-9, 7, None), (big, 0.05, 600, None)):
        d = w.domain
        if start is None:
            start = np.zeros(d.numCellCentered(), np.float32)
        dev = [torch.from_numpy(a).cuda() for a in (*w.inputs(), start.copy())]
        (out,) = _winds([w])
        torch.cuda.synchronize()
        st = qesb.solve_noalloc(d, tol, n, *[t.data_ptr() for t in dev], *[t.data_ptr() for t in out])
        L, it, fe, _ = O.sor(d, w, O.divergence(d, w), tol, n, lam=start)
        assert st["iterations"] == it and st["converged"] == (n == 600)
        assert (st["launches"] > 4 * it) == (w is big)
        np.testing.assert_array_equal(dev[-1].cpu().numpy(), L)
        _check_winds(w, L, out)
