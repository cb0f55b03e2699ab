"""Block solvers at block widths around every edge of the Gram, update and
small-system kernels (1, 2, 4, 8, 16, 32, 48 columns are their padded
widths; the division-free elimination ends at 32): X after a fixed three
iterations against the oracle."""
import numpy as np
import pytest

from oracle import dda_oracle as O

pytestmark = pytest.mark.gpu

WIDTHS = [1, 2, 3, 4, 5, 7, 8, 9, 16, 17, 31, 32, 33, 48, 49, 63, 64]


@pytest.mark.parametrize("solver", ["bicgstab", "cocg"])
@pytest.mark.parametrize("L", WIDTHS)
def test_three_iterations_match_the_oracle(solver, L):
    """Three iterations amplify rounding (1e-16) by far less than 1e7, and the
    small systems' condition numbers stay below 1e4: 1e-9, the bound of the other short solves."""
    from bl_krylov import bl_krylov as bk
    from mvp_fft import mvp_fft as mf
    rng = np.random.default_rng(L)
    n = (9, 7, 8)
    address = np.sort(rng.choice(9 * 7 * 8, 401, replace=False))   # 1203 rows: no multiple of any chunk
    N = address.size
    lf, k = 0.045, 2 * np.pi * 1.33 / 0.7
    diag = (rng.standard_normal(3 * N) + 60.0) / lf ** 3 + 1j * rng.standard_normal(3 * N) / lf ** 3
    B = rng.standard_normal((3 * N, L)) + 1j * rng.standard_normal((3 * N, L))
    ours = bk.bl_bicgstab_jacobi_mvp_fft if solver == "bicgstab" else bk.bl_cocg_rq_jacobi_mvp_fft
    theirs = O.bicgstab if solver == "bicgstab" else O.cocg_rq
    h, hr = [], []
    X, it, err = ours(n, 3, address, mf.fft_init(n, 3, lf, k), diag, B, 1e-30, 3, history=h)
    Xr, itr, errr = theirs(n, 3, address, O.fft_init(n, 3, lf, k), diag, B, 1e-30, 3, history=hr)
    assert it == itr == 2
    assert np.max(np.abs(X - Xr)) / np.max(np.abs(Xr)) < 1e-9
    assert h[0] == pytest.approx(hr[0], rel=1e-6)
