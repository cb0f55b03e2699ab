"""How a batch is split into groups: sizes, the memory bound, and that an
unbounded batch is split once (host-only, on a stand-in for the library)."""
import types

import pytest

from bl_krylov import bl_krylov as bk


def _entries(sides):
    return [dict(g=types.SimpleNamespace(plan=types.SimpleNamespace(m=(s, s, s)))) for s in sides]


class _Lib:
    def __init__(self):
        self.calls = 0

    def bdda_batch_workspace_bytes(self, arr, n, mode, L, itermax):
        self.calls += 1
        return 1000 * n


@pytest.fixture
def lib(monkeypatch):
    lib = _Lib()
    monkeypatch.setattr(bk._lib, "load", lambda: lib)
    monkeypatch.setattr(bk, "_batch_struct", lambda entries, mode: None)
    return lib


@pytest.mark.parametrize("sides,limit,groups,bound", [
    ([40, 30, 36], 10 ** 6, [[0, 2, 1]], False),
    ([100, 30, 90], 10 ** 6, [[0, 2], [1]], False),              # longest axes within a factor of 1.6
    ([40] * 5, 2000, [[0, 1], [2, 3], [4]], True),               # memory decides
    ([100, 30, 90], 1000, [[0], [2], [1]], True),
    ([100, 30], 1000, [[0], [1]], False),                        # apart in any case
    ([40] * 1025, 10 ** 9, [list(range(1024)), [1024]], False),
    ([40], 10, [[0]], False),                                     # a problem alone is never cut
])
def test_groups_and_what_ended_them(lib, sides, limit, groups, bound):
    assert bk._batch_groups(_entries(sides), 0, 8, 10, limit) == (groups, bound)
    assert lib.calls == len(sides)
