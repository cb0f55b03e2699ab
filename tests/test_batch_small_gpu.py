"""Batches of many small problems: shared launches before the graph, each
problem's own in it; the number of launches shows which run."""
import numpy as np
import pytest

from oracle import dda_oracle as O

pytestmark = pytest.mark.gpu
LF, K = 0.03, 10.0


def _problems(count, L, k=K, sides=(8, 9, 10)):
    from mvp_fft import mvp_fft
    out = []
    for i in range(count):
        rng = np.random.default_rng(i)
        n = (8, sides[i % len(sides)], 8)
        address = np.sort(rng.choice(int(np.prod(n)), int(0.6 * np.prod(n)), replace=False))
        N = address.size
        _, _, diag = O.polarizability(np.array([1.5 + 0.01j, 1.55 + 0.01j, 1.45 + 0.02j]), 1.33, LF, k, N)
        B = rng.standard_normal((3 * N, L)) + 1j * rng.standard_normal((3 * N, L))
        out.append((n, address, mvp_fft.fft_init(n, 3, LF, k), diag, B))
    return out


def _run(problems, *args, **kw):
    from bdda_b200 import _lib
    from bl_krylov import bl_krylov as bk
    before = _lib.load().bdda_launch_count()
    return bk.bl_bicgstab_jacobi_mvp_fft_batch(problems, *args, **kw), _lib.load().bdda_launch_count() - before


@pytest.mark.parametrize("precision", ["c128", "c64", "mixed"])
def test_launches_before_and_after_the_graph(precision):
    """Four iterations of 16 problems take fewer launches than the ten a problem
    and iteration that launches of their own would be; iterations 9 to 12 are
    those.  15 problems, or 16 wider ones, run their own from the first."""
    probs = _problems(16, 8)
    _, four = _run(probs, 1e-30, 4, precision=precision, max_outer=1)
    assert four < 4 * 10 * 16
    late = [_run(probs, 1e-30, n, precision=precision, max_outer=1)[1] for n in (8, 12)]
    assert late[1] - late[0] >= 4 * 10 * 16
    for few in (_problems(15, 8), _problems(16, 32)):
        assert _run(few, 1e-30, 4, precision=precision, max_outer=1)[1] >= 4 * 10 * len(few)


@pytest.mark.parametrize("precision,tol,bound", [("c128", 1e-8, 1e-6), ("mixed", 1e-5, 1e-3)])
@pytest.mark.parametrize("k", [10.0, 60.0])
def test_solutions_across_the_handover(precision, tol, bound, k):
    """The same bits with the graph and without, and the one-problem solver's
    solutions (bounds of the other batch tests) where it converges; k = 60 takes
    more iterations than the direct ones or runs into the limit."""
    from bl_krylov import bl_krylov as bk
    probs = _problems(18, 8, k)
    (a, _), (b, _) = (_run(probs, tol, 40, precision=precision, graph=g) for g in (True, False))
    for p, (X, it, err), (Xd, itd, errd) in zip(probs, a, b):
        assert it == itd and err == errd and np.array_equal(X, Xd)
        Xs, its, errs = bk.bl_bicgstab_jacobi_mvp_fft(p[0], 3, *p[1:], tol, 40, precision=precision)
        if k == 10.0:
            assert err < tol and errs < tol and abs(it - its) <= 3
            assert np.max(np.abs(X - Xs)) < bound * np.max(np.abs(Xs))
        true = O.true_residual(p[0], 3, p[1], O.fft_init(p[0], 3, LF, k), p[3], p[4], X)
        assert abs(true - err) < 1e-3 * err + 1e-9
