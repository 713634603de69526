"""The bench's roofline counts the work of the search kernel that ran."""
from __future__ import annotations

import importlib.util
import pathlib

import pytest

ROOT = pathlib.Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def bench():
    spec = importlib.util.spec_from_file_location("bench_work", ROOT / "bench.py")
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


def test_tensor_core_steps_leave_out_the_leading_bits(bench):
    # 703 bits: 9 leading bits in the start, 693 steps of 22 * 23 / 2 + 44 products
    assert bench.tc_steps(703, 22) == 693 and bench.tc_products_per_test(703, 22) == 693 * 297
    assert bench.tc_steps(462, 15) == 461 - 8
    assert bench.tc_steps(1274, 40) == 1273  # from 40 words on every bit is a step


@pytest.mark.parametrize("info,ran_tc,kernel,products", [
    (dict(limbs=28, tc_words=26, tpi=1), True, "k_search_tc<26>", (820 - 1 - 9) * (26 * 27 // 2 + 52)),
    (dict(limbs=28, tc_words=26, tpi=1), False, "k_search_persistent<28>", 819 * (28 * 29 // 2 + 28 * 28 + 28)),
    (dict(limbs=23, tc_words=0, tpi=1), False, "k_search_persistent<23>", 819 * (23 * 24 // 2 + 23 * 23 + 23)),
    (dict(limbs=136, tc_words=0, tpi=8), False, "k_search_persistent_g<136>", 819 * (136 * 137 // 2 + 136 * 136 + 136)),
])
def test_the_kernel_that_ran_is_named_and_counted(bench, info, ran_tc, kernel, products):
    name, count, what = bench.search_work(info, 820, ran_tc)
    assert name == kernel and count == products and str(info["tc_words"] if ran_tc else info["limbs"]) in what
