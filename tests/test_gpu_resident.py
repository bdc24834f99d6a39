"""Solves with lambda resident in shared memory (the default for domains that
fit) against the oracle: grids at the edges of the tiling (one cell, one row or
one plane per tile, ragged rows, one CTA and many), every stop, and batches
whose domains run on groups of CTAs of different sizes. Equal bits everywhere."""
import numpy as np
import pytest

import qesb
from oracle import oracle as O

pytestmark = pytest.mark.gpu

# the smallest grid; single updated rows, planes and columns; rows of one and of many 4-cell groups; sizes off
# every multiple; long x, long y, tall; one that needs every SM
GRIDS = [(3, 3, 2), (3, 40, 5), (40, 3, 9), (9, 7, 2), (10, 9, 3), (17, 12, 4), (47, 41, 20), (64, 33, 17),
         (257, 40, 21), (33, 200, 12), (8, 9, 90), (130, 131, 33), (514, 30, 9), (200, 180, 60)]


def _city(nx, ny, nz, seed=5):
    d = qesb.Domain(nx, ny, nz, 2.0, 2.0, 1.0, qesb.city_dz(nz, 1.0, 1.03))
    if min(nx, ny) < 30:  # no room for the generator's margins: one block in the middle
        b = [qesb.Building(2.0 * (nx // 3), 2.0 * (ny // 3), max(2.0, 2.0 * (nx // 4)), max(2.0, 2.0 * (ny // 4)),
                           max(1.0, nz / 3.0), 0.0)]
        return qesb.city_build(d, b, qesb.Inflow(4.0, 10.0, 0.2, 250.0))
    c = qesb.city_random(d, seed, 12, fp=(6, 20), h=(4, 20))
    return qesb.city_build(d, c.buildings, c.inflow)


def _check_winds(w, L):
    for name, x in zip("uvw", O.correct(w.domain, w, L)):
        np.testing.assert_array_equal(getattr(w, name), x, err_msg=name)


@pytest.mark.parametrize("grid", GRIDS)
def test_fixed_count_from_a_rough_start(grid):
    """A random start (its ground plane not the mirror of plane 1), a count
    that ends the loop: lambda, winds and every iteration's FP64 maximum."""
    w = _city(*grid)
    d = w.domain
    lam0 = np.random.default_rng(3).standard_normal(d.numCellCentered()).astype(np.float32)
    n = 11
    with qesb.Solver_B200(d, 1e-9) as s:
        s.lambda_ = lam0
        st = s.solve(w, n)
        lam, hist = s.lambda_, s.residual_history(n)
    L, it, _, ho = O.sor(d, w, O.divergence(d, w), 1e-9, n, lam=lam0, hist=True)
    assert st["iterations"] == it
    np.testing.assert_array_equal(lam, L)
    np.testing.assert_array_equal(hist[:it], ho[:it])
    assert st["residual"] == ho[it - 1]
    _check_winds(w, L)


@pytest.mark.parametrize("grid", [(10, 9, 3), (47, 41, 20), (130, 61, 33)])
@pytest.mark.parametrize("start", [None, (1.7, 5)])
def test_phases_and_window_rule(grid, start):
    """Start stage, pre-phase to its tolerance and reference loop to the window
    rule, then a second solve from the kept lambda, against the oracle's chain."""
    w = _city(*grid)
    d = w.domain
    R = O.divergence(d, w)
    K, wtol, pre = 8, 5e-3, (1.85, 2e-3, 3000)
    L = None
    with qesb.Solver_B200(d, 1e-9) as s:
        s.set_prephase(*pre)
        s.set_window_rule(K, wtol)
        if start:
            s.set_prephase_start(*start)
        for _ in range(2):
            st = s.solve(w, 4000)
            ns = 0
            if start:
                L, ns, *_ = O.sor(d, w, R, -1.0, start[1], omega=start[0], lam=L)
            L, npre, *_ = O.sor(d, w, R, pre[1], pre[2], omega=pre[0], lam=L)
            L, it, stop, drift = O.sor_window(d, w, R, 1e-9, 4000, K, wtol, lam=L)
            assert (st["pre_iterations"], st["iterations"], st["converged"]) == (ns + npre, it, stop)
            assert st["window_drift"] == drift
            np.testing.assert_array_equal(s.lambda_, L)
            _check_winds(w, L)


@pytest.mark.parametrize("tol", [0.3, 0.05, 2e-3])
def test_stop_on_the_iteration_of_the_rule(tol):
    w = _city(90, 75, 24)
    d = w.domain
    with qesb.Solver_B200(d, tol) as s:
        st = s.solve(w, 5000)
        lam = s.lambda_
    L, it, *_ = O.sor(d, w, O.divergence(d, w), tol, 5000)
    assert (st["iterations"], st["converged"]) == (it, 1)
    np.testing.assert_array_equal(lam, L)


def test_batch_of_uneven_domains_and_group_sizes():
    """Small domains that share a launch, larger ones, and one too large for
    the chip (list sweeps), in one call: each its own oracle result."""
    grids = [(40, 33, 9), (200, 180, 60), (64, 48, 20), (31, 77, 15), (96, 90, 40), (12, 9, 4), (640, 512, 30)]
    ws = [_city(*g, seed=7 + i) for i, g in enumerate(grids)]
    solvers = [qesb.Solver_B200(w.domain, 2e-2) for w in ws]
    try:
        for s, w in zip(solvers, ws):
            s.set_inputs(w)
        st = qesb.solve_batch(solvers, 60)
        lams = [s.lambda_ for s in solvers]
    finally:
        for s in solvers:
            s.close()
    for w, x, lam in zip(ws, st, lams):
        L, it, *_ = O.sor(w.domain, w, O.divergence(w.domain, w), 2e-2, 60)
        assert x["iterations"] == it
        np.testing.assert_array_equal(lam, L)


def test_group_wait_that_runs_out_is_an_error_and_the_handle_recovers():
    w = _city(130, 131, 33)
    d = w.domain
    with qesb.Solver_B200(d, 1e-9) as s:
        s.set_option("wait_limit", 1)
        with pytest.raises(qesb.QesbError, match="gave up"):
            s.solve(w, 50)
        s.set_option("wait_limit", 0)
        s.resetLambda()
        s.solve(w, 20)
        lam = s.lambda_
    L, *_ = O.sor(d, w, O.divergence(d, w), 1e-9, 20)
    np.testing.assert_array_equal(lam, L)


def _cut(w, seed=4):
    """Arbitrary face coefficients beside the walls and in one cell of twenty."""
    d = w.domain
    rng = np.random.default_rng(seed)
    near = (w.e == 0) | (w.g == 0) | (w.m == 0) | (rng.random(w.e.size) < 0.05)
    for name in w.FIELDS_CELL:
        a = getattr(w, name)
        a[near] *= (0.1 + 0.9 * rng.random(near.sum())).astype(np.float32)
        a[near & (a == 0)] = np.float32(1e-3)  # no cell without an open face
    assert d.numCellCentered() == w.e.size
    return w


@pytest.mark.parametrize("grid", [(3, 3, 2), (9, 7, 2), (17, 12, 4), (47, 41, 20), (257, 40, 21), (33, 200, 12),
                                  (130, 131, 33)])
def test_full_coefficients(grid):
    """Cells with six coefficients of their own: the handle's solve (fixed
    count from a rough start, then to the window rule) and the solve without
    allocation, against the oracle."""
    import torch

    w = _cut(_city(*grid))
    d = w.domain
    R = O.divergence(d, w)
    lam0 = np.random.default_rng(3).standard_normal(d.numCellCentered()).astype(np.float32)
    n = 11
    L, it, _, ho = O.sor(d, w, R, 1e-9, n, lam=lam0, hist=True)
    with qesb.Solver_B200(d, 1e-9) as s:
        s.set_option("path", 0)  # the smallest grid's one cell would pass for a wall mask
        s.lambda_ = lam0
        st = s.solve(w, n)
        assert (st["path"], st["iterations"]) == (0, it)
        np.testing.assert_array_equal(s.lambda_, L)
        np.testing.assert_array_equal(s.residual_history(n)[:it], ho[:it])
        _check_winds(w, L)
        s.set_window_rule(8, 1e-2)
        st = s.solve(w, 150, set_inputs=False)  # these random matrices diverge later on, in the oracle too
        Lw, itw, stop, drift = O.sor_window(d, w, R, 1e-9, 150, 8, 1e-2, lam=L)
        assert (st["iterations"], st["converged"], st["window_drift"]) == (itw, stop, drift)
        np.testing.assert_array_equal(s.lambda_, Lw)
    dev = [torch.from_numpy(a).cuda() for a in (*w.inputs(), lam0.copy())]
    out = [torch.empty(d.numFaceCentered(), device="cuda") for _ in range(3)]
    torch.cuda.synchronize()
    st = qesb.solve_noalloc(d, 1e-9, n, *[t.data_ptr() for t in dev], *[t.data_ptr() for t in out])
    assert st["iterations"] == it and st["residual"] == ho[it - 1]
    np.testing.assert_array_equal(dev[-1].cpu().numpy(), L)
    for name, t, x in zip("uvw", out, O.correct(d, w, L)):
        np.testing.assert_array_equal(t.cpu().numpy(), x, err_msg=name)


def _noalloc(d, w, tol, n, lam0):
    """One call on the GPU: its stats, lambda and winds."""
    import torch

    dev = [torch.from_numpy(a).cuda() for a in (*w.inputs(), lam0.copy())]
    out = [torch.empty(d.numFaceCentered(), device="cuda") for _ in range(3)]
    torch.cuda.synchronize()
    st = qesb.solve_noalloc(d, tol, n, *[t.data_ptr() for t in dev], *[t.data_ptr() for t in out])
    return st, dev[-1].cpu().numpy(), [t.cpu().numpy() for t in out]


ROW_GRIDS = [(17, 12, 4), (47, 41, 20), (64, 33, 17), (33, 200, 12), (130, 131, 33)]


@pytest.mark.parametrize("grid", ROW_GRIDS)
def test_no_allocation_calls_of_one_iteration_in_a_row(grid):
    """The scratch array keeps what the last call left in it: calls of one
    iteration, each on other inputs than the last, then one of five; every call
    against the oracle."""
    ws = [_cut(_city(*grid, seed=s), seed=s) for s in (5, 6)]
    d = ws[0].domain
    Rs = [O.divergence(d, w) for w in ws]
    rng = np.random.default_rng(7)
    for call, n in enumerate((1, 1, 1, 5, 1, 5)):
        q = call % 2
        lam0 = rng.standard_normal(d.numCellCentered()).astype(np.float32)
        st, lam, winds = _noalloc(d, ws[q], 1e-9, n, lam0)
        L, it, *_ = O.sor(d, ws[q], Rs[q], 1e-9, n, lam=lam0)
        assert st["iterations"] == it == n
        np.testing.assert_array_equal(lam, L)
        for name, a, x in zip("uvw", winds, O.correct(d, ws[q], L)):
            np.testing.assert_array_equal(a, x, err_msg=name)


@pytest.mark.parametrize("grid", ROW_GRIDS)
def test_no_allocation_call_that_converges_at_once_then_others(grid):
    """A coupling loop's quiet step: the kept lambda meets the tolerance in the
    first iteration; the next steps have other walls and winds."""
    ws = [_city(*grid, seed=s) for s in (5, 6)]
    d = ws[0].domain
    tol, lam = 0.25, np.zeros(d.numCellCentered(), np.float32)
    its = []
    for q in (0, 0, 1, 1, 0):
        w = ws[q]
        if len(its) == 2:
            w.u0 *= np.float32(1.5)  # the smallest grids' cities are alike
        L, it, *_ = O.sor(d, w, O.divergence(d, w), tol, 400, lam=lam)
        st, lam, winds = _noalloc(d, w, tol, 400, lam)
        its.append(it)
        assert st["iterations"] == it and st["converged"] == 1
        np.testing.assert_array_equal(lam, L)
        for name, a, x in zip("uvw", winds, O.correct(d, w, L)):
            np.testing.assert_array_equal(a, x, err_msg=name)
    assert its[1] == its[3] == 1 < its[2]


@pytest.mark.parametrize("grid", [(17, 12, 4), (47, 41, 20), (130, 131, 33)])
@pytest.mark.parametrize("K", [1, 2, 3])
def test_shortest_windows(grid, K):
    """Windows of one to three iterations, whose maxima follow one another
    closely: the stop and the last drift are the oracle's, solve after solve."""
    w = _city(*grid)
    d = w.domain
    R = O.divergence(d, w)
    L = None
    with qesb.Solver_B200(d, 1e-9) as s:
        for wtol in (0.05, 0.0125):
            s.set_window_rule(K, wtol)
            st = s.solve(w, 2000)
            L, it, stop, drift = O.sor_window(d, w, R, 1e-9, 2000, K, wtol, lam=L)
            assert (st["iterations"], st["converged"], st["window_drift"]) == (it, stop, drift) and stop == 2
            np.testing.assert_array_equal(s.lambda_, L)


def test_a_wait_limit_bounds_an_exchange_and_not_the_solve():
    """20000 polls are some ten milliseconds, far more than an exchange takes and
    far less than the solve: a grid of fewer tiles than the GPU has SMs, alone;
    then two domains on groups of one size, one of few tiles, each outlasting
    the limit."""
    ws = [_city(40, 40, 20), _city(47, 41, 20), _city(17, 12, 4)]
    n = 12000
    with qesb.Solver_B200(ws[0].domain, -1.0) as s:
        s.set_option("wait_limit", 20000)
        st = s.solve(ws[0], n)
        assert st["iterations"] == n and st["ms_sor"] > 40.0
    solvers = [qesb.Solver_B200(w.domain, -1.0) for w in ws[1:]]
    try:
        for s, w in zip(solvers, ws[1:]):
            s.set_inputs(w)
        solvers[0].set_option("wait_limit", 20000)
        st = qesb.solve_batch(solvers, n)
        lam = solvers[1].lambda_
    finally:
        for s in solvers:
            s.close()
    assert all(x["iterations"] == n and x["ms_sor"] > 30.0 for x in st)
    w = ws[2]
    np.testing.assert_array_equal(lam, O.sor(w.domain, w, O.divergence(w.domain, w), -1.0, n)[0])


def test_the_first_solve_of_a_handle_allocates_nothing():
    import torch

    w = _city(130, 131, 33)
    d = w.domain
    out = [torch.zeros(d.numFaceCentered(), device="cuda") for _ in range(3)]
    for _ in range(2):  # the first handle's solve loads the kernels
        with qesb.Solver_B200(d, 1e-9) as s:
            s.set_inputs(w)
            torch.cuda.synchronize()
            free = torch.cuda.mem_get_info()[0]
            s.solve_device(5, *[t.data_ptr() for t in out])
            torch.cuda.synchronize()
            used = free - torch.cuda.mem_get_info()[0]
    assert used == 0


def test_full_coefficients_without_room_for_their_split_copies():
    """79 MB of copies that only the resident solve needs, on a GPU with 32 MB
    free: the inputs are taken and solved without it."""
    import torch

    w0 = _city(200, 180, 60)
    w = _cut(_city(200, 180, 60))
    d = w.domain
    out = [torch.zeros(d.numFaceCentered(), device="cuda") for _ in range(3)]
    L = O.sor(d, w, O.divergence(d, w), 1e-9, 5)[0]
    with qesb.Solver_B200(d, 1e-9) as s:
        s.set_option("variant", 0)
        s.set_inputs(w)
        s.solve_device(5, *[t.data_ptr() for t in out])  # loads the kernels
    with qesb.Solver_B200(d, 1e-9) as s:
        s.set_inputs(w0)  # allocates the handle's own copy of the inputs
        torch.cuda.empty_cache()
        full = torch.empty(torch.cuda.mem_get_info()[0] - (32 << 20), dtype=torch.uint8, device="cuda")
        for _ in range(2):
            s.resetLambda()
            s.set_inputs(w)
            st = s.solve_device(5, *[t.data_ptr() for t in out])
            assert (st["iterations"], st["path"]) == (5, 0)
            np.testing.assert_array_equal(s.lambda_, L)
            for t, a in zip(out, O.correct(d, w, L)):
                np.testing.assert_array_equal(t.cpu().numpy(), a)
            del full
            torch.cuda.empty_cache()
            full = None


@pytest.mark.parametrize("variant", [-1, 18])
def test_first_window_counts_the_ground_planes_rim(variant):
    """Full coefficients, a start whose ground plane is not plane 1's mirror on
    the rim alone: the mirror of the first iteration moves those cells by more
    than the window's tolerance, which all others meet at once."""
    w = _city(47, 41, 20)
    d = w.domain
    R = O.divergence(d, w)
    lam0 = O.sor(d, w, R, 1e-9, 60)[0].reshape(21, 41, 47).copy()
    lam0[0, 0, 7] += np.float32(5.0)
    lam0[0, 9, 46] -= np.float32(4.0)
    with qesb.Solver_B200(d, 1e-9) as s:
        s.set_option("path", 0)
        s.set_option("variant", variant)
        s.set_window_rule(4, 3.0)
        s.lambda_ = lam0.ravel()
        st = s.solve(w, 200)
        L, it, stop, drift = O.sor_window(d, w, R, 1e-9, 200, 4, 3.0, lam=lam0.ravel())
        assert (st["iterations"], st["converged"], st["window_drift"]) == (it, stop, drift) and it == 8
        np.testing.assert_array_equal(s.lambda_, L)


@pytest.mark.parametrize("path,variant", [(1, -1), (1, 18), (0, -1), (0, 0)])
def test_window_rule_refuses_a_boundary_that_is_not_a_number(path, variant):
    """A cell on an edge of the box, which no other cell reads."""
    w = _city(47, 41, 20)
    lam0 = np.zeros((21, 41, 47), np.float32)
    lam0[7, 0, 0] = np.nan
    with qesb.Solver_B200(w.domain, 1e-9) as s:
        s.set_option("path", path)
        s.set_option("variant", variant)
        s.lambda_ = lam0.ravel()
        st = s.solve(w, 8)
        assert st["iterations"] == 8
        s.set_window_rule(4, 1e-3)
        with pytest.raises(qesb.QesbError, match="NaN"):
            s.solve(w, 8)


@pytest.mark.parametrize("variant", [-1, 18])
def test_a_tolerance_that_is_not_a_number_stops_the_loop(variant):
    """`max_error > tol` does not hold after the first iteration."""
    w = _city(47, 41, 20)
    with qesb.Solver_B200(w.domain, float("nan")) as s:
        s.set_option("variant", variant)
        st = s.solve(w, 30)
        assert (st["iterations"], st["converged"]) == (1, 1)
