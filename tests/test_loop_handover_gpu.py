"""Solves that stop just before, at and just after the iteration at which the
captured iteration takes over from the host (8), and a batch whose workspace
fits only once torch's cached memory is given back."""
import numpy as np
import pytest
import torch

from oracle import dda_oracle as O

pytestmark = pytest.mark.gpu


def _problem(n, L, seed, k=10.0):
    from mvp_fft import mvp_fft
    rng = np.random.default_rng(seed)
    address = np.sort(rng.choice(int(np.prod(n)), int(0.7 * np.prod(n)), replace=False))
    N = address.size
    _, _, diag = O.polarizability(np.array([1.5 + 0.01j, 1.55 + 0.01j, 1.45 + 0.02j]), 1.33, 0.03, k, N)
    B = rng.standard_normal((3 * N, L)) + 1j * rng.standard_normal((3 * N, L))
    return n, address, mvp_fft.fft_init(n, 3, 0.03, k), diag, B


@pytest.mark.parametrize("k,stops", [(10.0, 7), (60.0, 99)])
@pytest.mark.parametrize("itermax", [1, 7, 8, 9, 12])
@pytest.mark.parametrize("solver", ["bl_bicgstab_jacobi_mvp_fft", "bl_cocg_rq_jacobi_mvp_fft"])
def test_iteration_limits_around_the_handover(solver, itermax, k, stops):
    """The same kernels in the same order, so the same bits as the host-driven
    loop.  k = 10 meets the tolerance (BiCGSTAB from iteration 7 on), k = 60 never does."""
    from bl_krylov import bl_krylov as bk
    from bdda_b200 import _lib
    p = _problem((9, 8, 11), 8, 1, k)
    runs = []
    try:
        for on in (1, 0):
            _lib.load().bdda_tune_solver_graphs(on)
            h = []
            runs.append(getattr(bk, solver)(p[0], 3, *p[1:], 1e-14, itermax, history=h) + (h,))
    finally:
        _lib.load().bdda_tune_solver_graphs(1)
    (X, it, err, h), (Xh, ith, errh, hh) = runs
    assert it == ith and err == errh and h == hh and len(h) == it + 1
    assert min(itermax - 1, stops) <= it <= itermax - 1
    assert np.array_equal(X, Xh)


@pytest.mark.parametrize("k,stops", [(10.0, 7), (60.0, 99)])
@pytest.mark.parametrize("itermax", [4, 7, 8, 9, 13])
def test_batch_limits_around_the_handover(itermax, k, stops):
    from bl_krylov import bl_krylov as bk
    probs = [_problem((9, 8, 11), 8, 1, k), _problem((10, 12, 8), 8, 2, k)]
    a, b = (bk.bl_bicgstab_jacobi_mvp_fft_batch(probs, 1e-14, itermax, graph=g) for g in (True, False))
    for (X, it, err), (Xd, itd, errd) in zip(a, b):
        assert it == itd and err == errd and np.array_equal(X, Xd)
        assert min(itermax - 1, stops) <= it <= itermax - 1


def test_batch_split_is_decided_with_the_cache_given_back(monkeypatch):
    from bl_krylov import bl_krylov as bk
    probs = [_problem((9, 8, 11), 8, 1), _problem((10, 12, 8), 8, 2)]
    want = bk.bl_bicgstab_jacobi_mvp_fft_batch(probs, 1e-8, 60)
    real, given = torch.cuda.mem_get_info, []
    monkeypatch.setattr(torch.cuda, "empty_cache", lambda: given.append(1))
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda d=None: real(d) if given else (1 << 20, real(d)[1]))
    got = bk.bl_bicgstab_jacobi_mvp_fft_batch(probs, 1e-8, 60)
    assert len(given) == 1   # asked for once, and not after the small workspace
    for (X, it, err), (Xw, itw, errw) in zip(got, want):
        assert it == itw and err == errw and np.array_equal(X, Xw)
