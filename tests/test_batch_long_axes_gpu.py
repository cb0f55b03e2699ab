"""Complex128 batches with a long axis: their passes run as launches of each
problem's own, like those of any other length that has two-register-stage kernels."""
import numpy as np
import pytest

from oracle import dda_oracle as O

pytestmark = pytest.mark.gpu


def _problem(n, L, m):
    from mvp_fft import mvp_fft
    rng = np.random.default_rng(n[0])
    address = np.sort(rng.choice(int(np.prod(n)), int(0.6 * np.prod(n)), replace=False))
    N, lf, k = address.size, 0.03, 10.0
    _, _, diag = O.polarizability(np.array([1.5 + 0.01j, 1.55 + 0.01j, 1.45 + 0.02j]), 1.33, lf, k, N)
    B = rng.standard_normal((3 * N, L)) + 1j * rng.standard_normal((3 * N, L))
    return n, address, mvp_fft.fft_init(n, 3, lf, k, m=m), diag, B


@pytest.mark.parametrize("L", [8, 32])
@pytest.mark.parametrize("axis,long,other", [(0, 192, 180), (1, 224, 210), (2, 350, 360)])
def test_the_same_launches_as_other_lengths(axis, long, other, L):
    """Four iterations of two problems, counted: a batch on the long axis and one
    on a length near it; the solutions against the one-problem solver's (rounding
    of the same four iterations, bounds of the other batch tests)."""
    from bdda_b200 import _lib
    from bl_krylov import bl_krylov as bk
    counts = []
    for M in (long, other):
        n, m = [8, 9, 8], [16, 18, 16]
        n[axis], m[axis] = M // 2 - 2, M
        probs = [_problem(tuple(n), L, m), _problem(tuple(n), L, m)]
        before = _lib.load().bdda_launch_count()
        out = bk.bl_bicgstab_jacobi_mvp_fft_batch(probs, 1e-30, 4)
        counts.append(_lib.load().bdda_launch_count() - before)
        for p, (X, it, err) in zip(probs, out):
            Xs, its, errs = bk.bl_bicgstab_jacobi_mvp_fft(p[0], 3, *p[1:], 1e-30, 4)
            assert it == its == 3 and abs(err - errs) < 1e-6 * errs
            assert np.max(np.abs(X - Xs)) < 1e-6 * np.max(np.abs(Xs))
    assert counts[0] == counts[1]
