"""The two-register-stage convolution kernel's loop over column tiles."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _dense(n, m, L, dtype, seed):
    from mvp_fft import mvp_fft as mf
    til = mf.fft_init(n, 3, 0.045, 10.0, m=m)
    g = torch.Generator(device="cuda").manual_seed(seed)
    P = torch.randn((3 * int(np.prod(n)), L), dtype=dtype, device="cuda", generator=g)
    prec = "c128" if dtype == torch.complex128 else "c64"
    return lambda: mf.fft_mvp(n, 3, til, P, precision=prec).clone()


@pytest.mark.parametrize("dtype,tol", [(torch.complex128, 1e-13), (torch.complex64, 1e-5)])
@pytest.mark.parametrize("M", [60, 128, 160, 240, 320])
def test_column_tiles_of_the_convolution(M, dtype, tol):
    """2,500 pencils, so that a CTA takes several column tiles of one pencil (the
    last one narrower), over the shapes of the kernel: 8 right-hand sides in
    128, 192 and 256 threads, and 4 (complex128 from 240 on).  Against the
    run-time-radix kernels; tolerances of the length tests."""
    from bdda_b200 import _lib
    n, m = [M // 2 - 1, 24, 25], [M, 50, 50]
    for L in (15, 17, 33, 64):
        run = _dense(n, m, L, dtype, L)
        own = run()
        _lib.load().bdda_tune_fixed(0)
        try:
            generic = run()
        finally:
            _lib.load().bdda_tune_fixed(1)
        assert float((own - generic).abs().max()) <= tol * float(generic.abs().max()), L
