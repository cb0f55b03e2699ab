"""Host-only: the autotuner's rule for near equals."""
import ctypes as C

import pytest

from bdda_b200 import _lib


def choose(keys):
    """keys: (times, default) per pass -> chosen candidates."""
    n = len(keys)
    times = [t for ms, _ in keys for t in ms]
    out = (C.c_int * max(n, 1))(*([-9] * max(n, 1)))
    rc = _lib.load().bdda_tune_choose(n, (C.c_int * max(n, 1))(*[len(ms) for ms, _ in keys]),
                                      (C.c_int * max(n, 1))(*[d for _, d in keys]),
                                      (C.c_double * max(len(times), 1))(*times), out)
    assert rc == 0
    return list(out[:n])


@pytest.mark.parametrize("keys,chosen", [
    ([([1.0, 0.91], 0)], [0]),                                   # under 10 %: the default
    ([([1.0, 0.85], 0)], [1]),
    ([([0.85, 1.0], 1)], [0]),
    ([([1.0, 0.852, 0.850, 0.849], 0)], [1]),                    # near equals: the first
    ([([1.0, 0.90, 0.85], 0)], [2]),                             # 6 % apart: the fastest
    ([([2.0, 1.01, 1.0], -1)], [1]),                             # no default
    ([([], -1), ([1.0], 0)], [-1, 0]),
    ([([2.34, 2.012, 2.017], 0), ([9.4, 11.0], 0), ([8.4], 0)], [0, 0, 0]),     # 1.6 % of the whole: defaults
    ([([21.2, 17.8], 0), ([20.3, 20.0], 0)], [1, 0]),                          # 8 %
    ([([1.0, 0.5], 0), ([100.0, 99.0], 0), ([50.0, 49.5, 10.0], -1)], [0, 0, 2]),   # keys without a default apart
    ([], []),
])
def test_rule(keys, chosen):
    assert choose(keys) == chosen


def test_the_order_of_near_equals_decides_whatever_the_noise():
    for a, b in ((2.012, 2.017), (2.017, 2.012)):
        assert choose([([2.5, a, b], 0)]) == [1]


def test_bad_arguments():
    lib = _lib.load()
    one = (C.c_int * 1)(1)
    assert lib.bdda_tune_choose(-1, None, None, None, None) == _lib.BAD_ARG
    assert lib.bdda_tune_choose(1, one, None, None, None) == _lib.BAD_ARG
    assert lib.bdda_tune_choose(1, one, one, (C.c_double * 1)(1.0), (C.c_int * 1)()) == _lib.BAD_ARG   # default 1 of 1
