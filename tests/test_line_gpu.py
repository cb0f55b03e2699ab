"""The two-register-stage pencil kernels (bdda_line.cuh) of every length they
are compiled for, on each axis: the block product and the dense product
against the oracle, at block widths around the tile sizes."""
import numpy as np
import pytest

from oracle import dda_oracle as O

pytestmark = pytest.mark.gpu

LENGTHS = [m for m in range(16, 541, 2) if 210 ** 9 % m == 0]   # even, 7-smooth
# complex128: rounding of three transforms of at most 540 points and back, a
# few (log2 of the grid) x 1.1e-16 of the largest entry; complex64 the same
# with 6e-8
TOL = {"c128": 1e-13, "c64": 1e-5}


def _rel(a, b):
    return np.max(np.abs(a - b)) / np.max(np.abs(b))


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("L", [1, 3, 8, 13])
def test_every_length_against_the_oracle(axis, L):
    """Axis length M on one axis, the smallest grids on the others; cuboid
    sides M / 2 (every admissible row filled) and an odd one below it."""
    from bl_krylov import bl_krylov as bk
    from mvp_fft import mvp_fft as mf
    assert len(LENGTHS) == 71
    rng = np.random.default_rng(100 * axis + L)
    for i, M in enumerate(LENGTHS):
        n, m = [5, 3, 4], [16, 18, 20]
        n[axis], m[axis] = M // 2 - (i % 2), M
        nc = int(np.prod(n))
        address = np.sort(rng.choice(nc, max(1, nc // 2), replace=False))
        N = address.size
        diag = (rng.standard_normal(3 * N) + 4.0) + 1j * rng.standard_normal(3 * N)
        S = rng.standard_normal((3 * N, L)) + 1j * rng.standard_normal((3 * N, L))
        lf, k = 0.045, 2 * np.pi * 1.33 / 0.7
        ref_til = O.fft_init(n, 3, lf, k)
        idx = O.scatter_index(address, 3)
        ref = O.block_mvp(n, 3, ref_til, idx, diag, S, 1.0 / diag)
        til = mf.fft_init(n, 3, lf, k, m=m)
        P = rng.standard_normal((3 * nc, L)) + 1j * rng.standard_normal((3 * nc, L))
        ref_dense = O.fft_mvp(n, 3, ref_til, P)
        for prec in ("c128", "c64"):
            out = bk._block_mvp(n, 3, til, idx, diag, S, 1.0 / diag, precision=prec)
            assert _rel(out, ref) < TOL[prec], (M, prec)
            assert _rel(mf.fft_mvp(n, 3, til, P, precision=prec), ref_dense) < TOL[prec], (M, prec)
