"""Column sums of the tensor-core search's byte products at their largest, through the 32-bit pair sums that make
words of them."""
from __future__ import annotations

import numpy as np
import pytest

from test_tc_search import SIZES


@pytest.mark.parametrize("L", SIZES)
def test_largest_columns_make_the_exact_words(L):
    """All bytes 255, the operands as long as the kernel has them: every column below 2^24 (above 2^23 from 32 words
    on), every pair with its carry below 2^32, and the words equal the product's."""
    nt, nw = 4 * (L + 4), L + 2
    for a_len, b_len in ((nt, 4 * 48), (4 * (L + 1), 4 * L)):
        a, b = np.full(a_len, 255, np.int64), np.full(b_len, 255, np.int64)
        prod = np.convolve(a, b)
        for off in (0, max(0, len(prod) // 2 - 2 * nw)):  # the lowest columns, and those around the largest
            cols = [int(c) for c in prod[off:off + 4 * nw]]
            cols += [0] * (4 * nw - len(cols))
            assert max(cols) <= nt * 255 * 255 < 1 << 24
            exact, up, carry, words = sum(c << (8 * i) for i, c in enumerate(cols)), 0, 0, []
            for k in range(nw):
                c0, c1, c2, c3 = cols[4 * k:4 * k + 4]
                p1, u = c2 + (c3 << 8), c0 + (c1 << 8) + up
                assert p1 < 1 << 32 and u < 1 << 32
                s = u + (p1 << 16 & 0xffffffff) + carry
                up, carry = p1 >> 16, s >> 32
                words.append(s & 0xffffffff)
            assert sum(w << (32 * k) for k, w in enumerate(words)) == exact & ((1 << 32 * nw) - 1)
