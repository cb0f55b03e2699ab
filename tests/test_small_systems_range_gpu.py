"""The L x L systems at the ends of the exponent range: a right-hand side scaled
by a power of two scales every quantity of a solve by powers of two, so the
solution is the same bits, scaled, as long as nothing overflows."""
import numpy as np
import pytest

from oracle import dda_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [3, 10, 32])
@pytest.mark.parametrize("top", [1010, -900])
@pytest.mark.parametrize("solver", ["bl_bicgstab_jacobi_mvp_fft", "bl_cocg_rq_jacobi_mvp_fft"])
def test_scaled_right_hand_sides(solver, top, L):
    """||M^-1 B||^2, the size of the first Gram products, just above 2^top: 14
    powers of two below the largest double, or 120 above the smallest normal one."""
    from bl_krylov import bl_krylov as bk
    from mvp_fft import mvp_fft
    n, lf, k = (9, 8, 10), 0.03, 10.0
    rng = np.random.default_rng(L)
    address = np.sort(rng.choice(720, 500, replace=False))
    _, _, diag = O.polarizability(np.array([1.5 + 0.01j, 1.55 + 0.01j, 1.45 + 0.02j]), 1.33, lf, k, 500)
    B = rng.standard_normal((1500, L)) + 1j * rng.standard_normal((1500, L))
    e = (top - int(np.floor(np.log2(np.sum(np.abs(B / diag[:, None]) ** 2))))) // 2
    til = mvp_fft.fft_init(n, 3, lf, k)
    X, it, err = getattr(bk, solver)(n, 3, address, til, diag, B, 1e-6, 12)
    Xs, its, errs = getattr(bk, solver)(n, 3, address, til, diag, np.ldexp(B.real, e) + 1j * np.ldexp(B.imag, e), 1e-6, 12)
    assert it == its and err == errs
    assert np.array_equal(np.ldexp(X.real, e), Xs.real) and np.array_equal(np.ldexp(X.imag, e), Xs.imag)
