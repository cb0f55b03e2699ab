"""Which pencil kernels run: the library's choice, a tile width or launch shape
that is asked for, and the two-register-stage kernels by their own id.  The
kernels round differently, so the bits of a product tell them apart."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
LINE, GENERIC = 4096, -2
DTYPE = {0: torch.complex128, 1: torch.complex64}


def _lib():
    from bdda_b200 import _lib
    return _lib.load()


def _product(n, m, L, prec, seed=0):
    """Dense product as a function of the launch choices (its inputs made once)."""
    from mvp_fft import mvp_fft as mf
    til = mf.fft_init(n, 3, 0.045, 10.0, m=m)
    g = torch.Generator(device="cuda").manual_seed(seed)
    P = torch.randn((3 * int(np.prod(n)), L), dtype=DTYPE[prec], device="cuda", generator=g)
    return lambda: mf.fft_mvp(n, 3, til, P, precision=("c128", "c64")[prec]).clone()


def _choose(prec, m, L, lt, variant):
    for kind, M in ((1, m[0]), (0, m[1]), (2, m[1]), (0, m[2]), (2, m[2])):
        assert _lib().bdda_tune_pass(prec, kind, M, L, lt, variant) == 0


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("L", [1, 5, 9])
def test_a_tile_width_selects_the_kernels_of_that_width(prec, L):
    n, m = (20, 23, 27), (48, 50, 60)   # lengths with two-register-stage kernels, none specialised for the radices
    run = _product(n, m, L, prec)
    try:
        own = run()
        _choose(prec, m, L, 8, LINE)
        assert torch.equal(run(), own)
        for lt in (2, 4, 8):
            _choose(prec, m, L, lt, GENERIC)
            want = run()
            assert not torch.equal(want, own)
            _choose(prec, m, L, lt, 0)
            assert torch.equal(run(), want), lt
    finally:
        _choose(prec, m, L, 0, 0)
    assert torch.equal(run(), own)
    assert _lib().bdda_tune_pass(prec, 0, 60, L, 0, LINE + 1) == 3   # BDDA_BAD_ARG


@pytest.mark.parametrize("prec", [0, 1])
def test_a_launch_shape_selects_the_kernels_that_have_one(prec):
    n, m, L = (20, 23, 27), (48, 50, 60), 6
    run = _product(n, m, L, prec)
    budget, threads = C.c_size_t(), C.c_int()
    assert _lib().bdda_tune_get(prec, 0, C.byref(budget), C.byref(threads)) == 0
    own = run()
    try:
        for shape in ((16 * 1024, threads.value), (budget.value, 128)):
            for kind in range(3):
                assert _lib().bdda_tune_set(prec, kind, *shape) == 0
            got = run()
            _choose(prec, m, L, 0, GENERIC)
            assert torch.equal(got, run()) and not torch.equal(got, own), shape
            _choose(prec, m, L, 0, 0)
    finally:
        _choose(prec, m, L, 0, 0)
        for kind in range(3):
            _lib().bdda_tune_set(prec, kind, budget.value, threads.value)
    assert torch.equal(run(), own)


@pytest.mark.parametrize("axis,M", [(0, 192), (1, 224), (2, 350)])
def test_long_complex128_axes_specialised_kernels_from_32_columns(axis, M):
    """Narrower blocks run the two-register-stage kernel of the length."""
    n, m = [10, 11, 9], [20, 24, 18]
    n[axis], m[axis] = M // 2 - 1, M
    for L, line in ((1, True), (4, True), (31, True), (32, False), (64, False)):
        run = _product(n, m, L, 0)
        own = run()
        try:
            for kind in ((1,), (0, 2), (0, 2))[axis]:
                assert _lib().bdda_tune_pass(0, kind, M, L, 0, LINE) == 0
            assert torch.equal(run(), own) == line, L
        finally:
            for kind in range(3):
                _lib().bdda_tune_pass(0, kind, M, L, 0, 0)
