"""Batches whose problems run their passes as launches of their own, as
shared launches, or both: axes below the shortest length with kernels of its
own (14), and a long one that keeps its specialised kernels in complex128 (so it
shares the batch's launches there) but not in complex64, against the
one-problem solver and the float64 oracle."""
import numpy as np
import pytest

from oracle import dda_oracle as O

pytestmark = pytest.mark.gpu
LATTICES = [(7, 14, 14), (14, 14, 14), (20, 17, 15), (8, 8, 9), (96, 8, 9)]


def _problems(L, sizes):
    from mvp_fft import mvp_fft
    out = []
    for i, n in enumerate(sizes):
        rng = np.random.default_rng(100 + i)
        address = np.sort(rng.choice(int(np.prod(n)), int((0.4 + 0.1 * i) * np.prod(n)), replace=False))
        N, lf, k = address.size, 0.03, 10.0
        _, _, diag = O.polarizability(np.array([1.5 + 0.01j, 1.55 + 0.01j, 1.45 + 0.02j]), 1.33, lf, k, N)
        B = rng.standard_normal((3 * N, L)) + 1j * rng.standard_normal((3 * N, L))
        out.append((n, address, mvp_fft.fft_init(n, 3, lf, k), diag, B))
    return out


def _rel(a, b):
    return np.max(np.abs(np.asarray(a) - np.asarray(b))) / np.max(np.abs(np.asarray(b)))


@pytest.mark.parametrize("L,sizes", [(8, LATTICES), (16, LATTICES[2:]), (32, LATTICES[1:2]), (8, LATTICES[:1] * 2)])
@pytest.mark.parametrize("precision,tol", [("c128", 1e-8), ("mixed", 1e-5)])
def test_problems_of_both_kinds(L, sizes, precision, tol):
    """Bounds of the other batch tests: X within 1e-6 (complex128) and 1e-3
    (mixed, whose error is the float64 true residual)."""
    from bl_krylov import bl_krylov as bk
    probs = _problems(L, sizes)
    runs = [bk.bl_bicgstab_jacobi_mvp_fft_batch(probs, tol, 300, precision=precision, graph=g) for g in (True, False)]
    for p, (X, it, err), (Xd, itd, errd) in zip(probs, *runs):
        assert it == itd and err == errd and np.array_equal(X, Xd)
        Xs, its, errs = bk.bl_bicgstab_jacobi_mvp_fft(p[0], 3, *p[1:], tol, 300, precision=precision)
        assert err < tol and errs < tol and abs(it - its) <= 3
        assert _rel(X, Xs) < (1e-6 if precision == "c128" else 1e-3)
        true = O.true_residual(p[0], 3, p[1], O.fft_init(p[0], 3, 0.03, 10.0), p[3], p[4], X)
        assert abs(true - err) < 1e-3 * err + 1e-9
    warm = bk.bl_bicgstab_jacobi_mvp_fft_batch([p + (r[0],) for p, r in zip(probs, runs[0])], 100 * tol, 50,
                                               precision=precision)
    for (X, it, err), r in zip(warm, runs[0]):
        assert it == 0 and err < 100 * tol
