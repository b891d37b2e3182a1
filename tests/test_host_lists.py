"""Rows of page numbers into int32 tables: the native conversion and the general one agree, and refuse the same."""

import collections

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


@pytest.mark.parametrize("broken", ["compiler", "no compiler", "no source"])
def test_the_library_builds_without_the_converter(broken, monkeypatch, tmp_path):
    """A box with a fresh library, or with nvcc alone, needs no C compiler: lists then go through NumPy."""
    from vllm_metal_b200.metal import build as b

    lib = tmp_path / "lib.so"
    lib.touch()
    monkeypatch.setattr(b, "output_path", lambda component=None: lib)
    monkeypatch.setattr(b, "stale_artifacts", lambda component=None: [])
    monkeypatch.setattr(b, "_PKG_DIR", tmp_path)
    if broken == "no source":
        monkeypatch.setattr(b, "CSRC_DIR", tmp_path)
    else:
        monkeypatch.setenv("CC", "false" if broken == "compiler" else str(tmp_path / "cc"))
    with pytest.warns(RuntimeWarning, match="NumPy"):
        assert b.build() == lib
    assert sorted(tmp_path.iterdir()) == [lib]


def test_the_converter_is_fresh_by_content_and_named_by_interpreter(monkeypatch, tmp_path):
    import os
    import sysconfig

    from vllm_metal_b200.metal import build as b

    monkeypatch.setattr(b, "_PKG_DIR", tmp_path)
    src = tmp_path / "csrc" / "host_lists.c"
    src.parent.mkdir()
    src.write_bytes((b.CSRC_DIR / "host_lists.c").read_bytes())
    monkeypatch.setattr(b, "CSRC_DIR", src.parent)
    out = b.build_host()
    assert sysconfig.get_config_var("SOABI") in out.name
    made = out.stat().st_mtime_ns
    os.utime(src, (out.stat().st_mtime + 100,) * 2)  # a new checkout of the same source
    assert b.build_host().stat().st_mtime_ns == made
    src.write_text(src.read_text() + "\n/* changed */\n")
    os.utime(src, (1, 1))
    assert b.build_host().stat().st_mtime_ns != made
    assert not list(tmp_path.glob(".host_*"))


@pytest.mark.parametrize("values", [[3, -1, 2**31 - 1], [2**32 + 5, 1], np.array([2**32 + 5, -1]), [np.int64(2**32 + 5)], (7, 8), []])
def test_slots_keep_their_64_bits(values):
    from vllm_metal_b200.attention.impls.sdpa import _as_int64

    got = _as_int64(values)
    assert got.dtype == np.int64 and got.tolist() == [int(v) for v in values]


def test_token_ids_as_torch_takes_them():
    import torch

    from vllm_metal_b200.v1.model_runner import _token_ids

    for ids in ([3, 1, 2], (3, 1, 2), np.array([3, 1, 2]), torch.tensor([3, 1, 2]), [torch.tensor(3), np.int64(1), 2]):
        got = _token_ids(ids)
        assert got.dtype == torch.int32 and got.tolist() == [3, 1, 2]
    assert _token_ids([]).shape == (0,)
    for bad in ([2**31], np.array([2**32 + 5]), ["3"], [np.float32(1.5)]):
        with pytest.raises((RuntimeError, ValueError, TypeError)):
            _token_ids(bad)


@pytest.mark.parametrize("kind", [list, tuple, np.array, collections.deque])
@pytest.mark.parametrize("first,count", [(0, 1), (37, 40), (600, 40), (5, 0), (-3, 5)])
def test_slots_of_any_sequence_of_pages(kind, first, count):
    from vllm_metal_b200.attention.context import _slots

    ids = list(range(100, 140))
    want = [ids[p // 16] * 16 + p % 16 for p in range(first, first + count)]
    assert _slots(kind(ids), first, count, 16) == want
