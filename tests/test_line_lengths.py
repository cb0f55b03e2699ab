"""Host-only: the axis lengths with two-register-stage pencil kernels, as the
library's tables hold them."""
import ctypes as C

import pytest

from bdda_b200 import _lib

LENGTHS = [m for m in range(16, 541, 2) if 210 ** 9 % m == 0]   # even, 7-smooth


@pytest.mark.parametrize("prec", [0, 1])
def test_lengths_with_two_register_stage_kernels(prec):
    """Every even 7-smooth length from 16 to 540 but 486 and 490; the X pass, whose
    second factor is at most 10, those up to 320 but 250 and 294.  None outside
    that range, none for odd lengths."""
    lib = _lib.load()
    buf, n = (C.c_int * 4)(), C.c_int()
    for M in LENGTHS + [14, 15, 21, 560, 576, 600]:
        h = C.c_void_p()
        side = (M + 1) // 2
        assert lib.bdda_plan_create((C.c_int * 3)(side, side, side), (C.c_int * 3)(M, M, M), C.byref(h)) == 0
        try:
            for kind, axis in ((0, 2), (0, 1), (1, 0), (2, 1), (2, 2)):
                assert lib.bdda_tune_pass_variants(h, prec, kind, axis, 0, buf, 4, C.byref(n)) == 0
                has = M in LENGTHS and M not in (486, 490) and (axis > 0 or (M <= 320 and M not in (250, 294)))
                assert list(buf[:n.value]) == ([4096] if has else []), (M, kind, axis)
        finally:
            lib.bdda_plan_destroy(h)
