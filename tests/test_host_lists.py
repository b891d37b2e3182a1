"""Rows of page numbers into int32 tables: the native conversion and the general one agree, and refuse the same."""

import numpy as np
import pytest

from vllm_metal_b200 import host_lists
from vllm_metal_b200.metal.build import build_host


@pytest.mark.parametrize("rows", [
    [[1, 2, 3], [], [2**31 - 1, -2**31]],
    [(4, 5), [6]],
    [np.array([7, 8], dtype=np.int64), [9]],
    [[True, 2], [np.int64(3)]],
    [],
])
@pytest.mark.parametrize("native", [True, False])
def test_rows_as_numpy_fills_them(rows, native, monkeypatch):
    build_host()
    host_lists._lib.cache_clear()
    assert host_lists._lib() is not None
    if not native:
        monkeypatch.setattr(host_lists, "_lib", lambda: None)
    got, want = (np.full((3, 3), -7, dtype=np.int32) for _ in range(2))
    host_lists.fill_rows(got, rows)
    for i, r in enumerate(rows):
        want[i, :len(r)] = r
    assert (got == want).all()
    wide = np.full((3, 6), -7, dtype=np.int32)  # rows apart
    host_lists.fill_rows(wide[:, :3], rows)
    assert (wide[:, :3] == want).all() and (wide[:, 3:] == -7).all()


@pytest.mark.parametrize("rows,error", [([[2**31]], OverflowError), ([[1, 2, 3, 4]], ValueError), ([[1], [2], [3], [4]], IndexError),
                                        ([["x"]], ValueError)])
def test_what_was_refused_stays_refused(rows, error):
    build_host()
    with pytest.raises(error):
        host_lists.fill_rows(np.zeros((3, 3), dtype=np.int32), rows)


def test_slots_of_a_window_of_pages():
    from vllm_metal_b200.attention.context import _slots

    ids = list(range(100, 140))
    for first, count in ((0, 1), (15, 2), (16, 16), (37, 40), (600, 40), (5, 0)):
        want = [ids[p // 16] * 16 + p % 16 for p in range(first, first + count)]
        assert _slots(ids, first, count, 16) == want == _slots(np.array(ids), first, count, 16)
    with pytest.raises(IndexError):
        _slots(ids, 630, 40, 16)
