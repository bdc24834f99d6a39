"""Solves beside other work on the GPU. The resident solve needs its CTAs on as
many SMs at once as it has tiles; kernels of other streams may hold some of them.
Such a solve waits until there is room and ends with the oracle's bits. So do
solves from two host threads, one after the other."""
import threading

import numpy as np
import pytest

import qesb
from oracle import oracle as O

pytestmark = pytest.mark.gpu

N = 40


def _city(seed, dims=(128, 128, 48)):
    d = qesb.Domain(*dims, 2.0, 2.0, 1.0, qesb.city_dz(dims[2], 1.0, 1.03))
    c = qesb.city_random(d, seed, 12, fp=(6, 20), h=(4, 20))
    return qesb.city_build(d, c.buildings, c.inflow)


def _oracle(w, n):
    L = O.sor(w.domain, w, O.divergence(w.domain, w), 1e-9, n)[0]
    return L, O.correct(w.domain, w, L)


class _Busy:
    """Four one-thread kernels of 2.5 s on streams of their own: the largest grid
    here has a tile for all SMs but one."""

    def __enter__(self):
        import torch

        self.streams = [torch.cuda.Stream() for _ in range(4)]
        torch.cuda.synchronize()
        for s in self.streams:
            with torch.cuda.stream(s):
                torch.cuda._sleep(int(2.5 * 1.9e9))

    def __exit__(self, *_):
        import torch

        torch.cuda.synchronize()


def test_solve_beside_long_kernels():
    w = _city(5)
    with qesb.Solver_B200(w.domain, 1e-9) as s:
        s.set_inputs(w)
        s.solve(w, N, set_inputs=False)  # a kernel's first launch loads it, which waits for the others
        s.resetLambda()
        with _Busy():
            st = s.solve(w, N, set_inputs=False)
        lam = s.lambda_
    L, winds = _oracle(w, N)
    assert st["iterations"] == N
    np.testing.assert_array_equal(lam, L)
    for name, x in zip("uvw", winds):
        np.testing.assert_array_equal(getattr(w, name), x, err_msg=name)


def test_batch_beside_long_kernels():
    import torch

    ws = [_city(q, dims) for q, dims in enumerate([(96, 80, 24), (70, 45, 21), (131, 40, 15), (300, 300, 50)])]
    out = [[torch.zeros(w.domain.numFaceCentered(), device="cuda") for _ in range(3)] for w in ws]
    pre = (1.8, 1e-9, 9)
    solvers = [qesb.Solver_B200(w.domain, 1e-9) for w in ws]
    try:
        for q, (s, w) in enumerate(zip(solvers, ws)):
            s.set_inputs(w)
            if q % 2:
                s.set_prephase(*pre)
        qesb.solve_batch(solvers, N, *[[o[q].data_ptr() for o in out] for q in range(3)])
        for s in solvers:
            s.resetLambda()
        with _Busy():
            st = qesb.solve_batch(solvers, N, *[[o[q].data_ptr() for o in out] for q in range(3)])
        lams = [s.lambda_ for s in solvers]
    finally:
        for s in solvers:
            s.close()
    for q, (w, x, lam, o) in enumerate(zip(ws, st, lams, out)):
        d = w.domain
        R = O.divergence(d, w)
        L0 = O.sor(d, w, R, pre[1], pre[2], omega=pre[0])[0] if q % 2 else None
        L = O.sor(d, w, R, 1e-9, N, lam=L0)[0]
        assert (x["iterations"], x["pre_iterations"]) == (N, pre[2] * (q % 2))
        np.testing.assert_array_equal(lam, L)
        for t, a in zip(o, O.correct(d, w, L)):
            np.testing.assert_array_equal(t.cpu().numpy(), a)


def test_solve_without_allocation_beside_long_kernels():
    import torch

    w = _city(6, (64, 33, 17))
    d = w.domain
    dev = [torch.from_numpy(a).cuda() for a in (*w.inputs(), np.zeros(d.numCellCentered(), np.float32))]
    out = [torch.empty(d.numFaceCentered(), device="cuda") for _ in range(3)]
    args = [d, 1e-9, N, *[t.data_ptr() for t in dev], *[t.data_ptr() for t in out]]
    qesb.solve_noalloc(*args)
    dev[-1].zero_()
    with _Busy():
        st = qesb.solve_noalloc(*args)
    L, winds = _oracle(w, N)
    assert st["iterations"] == N
    np.testing.assert_array_equal(dev[-1].cpu().numpy(), L)
    for t, a in zip(out, winds):
        np.testing.assert_array_equal(t.cpu().numpy(), a)


def test_two_threads_solve_at_once():
    ws = [_city(8), _city(9, (100, 100, 50))]
    n, calls, errors, lams = 300, 12, [], [None, None]
    ready = threading.Barrier(2)

    def work(q):
        try:
            with qesb.Solver_B200(ws[q].domain, 1e-9) as s:
                s.set_inputs(ws[q])
                ready.wait(60)
                for _ in range(calls):
                    s.resetLambda()
                    st = s.solve(ws[q], n, set_inputs=False)
                    assert st["iterations"] == n
                lams[q] = s.lambda_
        except BaseException as e:  # noqa: BLE001 - shown by the main thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(q,)) for q in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120)
    assert not errors, errors
    for w, lam in zip(ws, lams):
        np.testing.assert_array_equal(lam, _oracle(w, n)[0])
