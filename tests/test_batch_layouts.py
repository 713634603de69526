"""The layout that a PRP batch runs on, by words and count (the library's own rule, which needs no GPU)."""
from __future__ import annotations

import ctypes

import pytest


def _layout(pg, words: int, n: int, rounds: int = 1) -> int:
    rule = pg.lib._ZN2pg10pick_batchEjjjPb  # pg::pick_batch(words, n, rounds, &side_by_side)
    rule.restype = ctypes.c_uint32
    rule.argtypes = [ctypes.c_uint32] * 3 + [ctypes.POINTER(ctypes.c_bool)]
    return rule(words, n, rounds, ctypes.byref(ctypes.c_bool()))


def _group(lanes: int, words: int) -> int:
    return lanes << 16 | words


@pytest.mark.parametrize("words,layout", [(16, 16), (17, 20), (18, 20), (19, 20), (20, 20), (24, 24)])
@pytest.mark.parametrize("n", [1, 64, 512, 1536, 2048, 4096, 100_000])
def test_sizes_that_one_thread_fills_stay_on_one_thread(pg, words, layout, n):
    assert _layout(pg, words, n) == layout


@pytest.mark.parametrize("words,n,layout", [(21, 4096, _group(8, 24)), (23, 64, _group(8, 24)), (23, 4097, 23),
                                            (25, 1600, _group(16, 48)), (25, 1601, 28), (47, 64, _group(16, 48)),
                                            (48, 4096, _group(8, 64)), (48, 4097, 48)])
def test_few_longer_numbers_take_groups(pg, words, n, layout):
    assert _layout(pg, words, n) == layout


@pytest.mark.parametrize("words,n,layout", [(16, 1024, 16), (17, 124, _group(8, 24)), (20, 125, 20), (23, 256, _group(8, 24)),
                                            (24, 69, _group(16, 48)), (24, 70, 24), (25, 100, _group(16, 48))])
def test_layouts_of_bases_side_by_side(pg, words, n, layout):
    assert _layout(pg, words, n, 16) == layout
