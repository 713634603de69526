"""The enumeration of a prime's lattice finds hits at the very edge of its window, with reciprocals off by all that
their error bound allows (the kernel's arithmetic restated; the limits are read from its header)."""
from __future__ import annotations

import math
import pathlib
import random
import re

import pytest

SRC = pathlib.Path(__file__).resolve().parents[1] / "prime-gap-gpu_b200" / "csrc" / "pg_internal.h"
LAT_W = 1 << 13
RECIPROCAL = 2.0 ** -38


def _limits() -> tuple[int, float]:
    text = SRC.read_text()
    shift = re.search(r"LAT_MAX_M = 1u << (\d+);", text)
    edge = re.search(r"LAT_EDGE = ([0-9.e-]+);", text)
    return 1 << int(shift.group(1)), float(edge.group(1))


def _first(A: int, p: int, lo: int, hi: int) -> int:
    """Smallest x >= 1 with A*x mod p in [lo, hi] (1 <= lo <= hi < p)."""
    A %= p
    if A == 0:
        return 0
    if A * 2 > p:
        return _first(p - A, p, p - hi, p - lo)
    x = -(-lo // A)
    if A * x <= hi:
        return x
    y = _first(p % A and (A - p % A), A, lo % A, hi % A) if A > 1 else 0
    return -(-(lo + p * y) // A)


def _lattice(p: int, A: int) -> tuple[int, int, int, int]:
    """(M, inc, dec, w) of LatC."""
    sa, sb = _first(A, p, 1, LAT_W), _first(A, p, p - LAT_W, p - 1)
    alpha, beta = A * sa % p, p - A * sb % p
    assert sa * beta + sb * alpha == p
    if alpha >= beta:
        return sb, sa % sb, alpha + sa // sb * beta, beta
    d = -(-sb // sa)
    return sa, d * sa - sb, beta + d * alpha, -alpha


def _hits(p, lat, b, W, J, edge, err) -> list[int]:
    """x of every hit that the kernel visits, its reciprocals off by the factor 1 + err."""
    M, inc, dec, w = lat
    inv, rm = (1.0 / p) * (1 + err), (1.0 / M) * (1 + err)
    rM, e = M * inv, float(w) * J * inv
    t = math.floor(rM * b + max(-e, 0.0) + edge)
    t0 = math.ceil(rM * (b - W) - max(e, 0.0) - edge)
    out = []
    if t < t0:
        return out
    Q = math.ceil(float(t) * inc * rm)
    x = Q * M - t * inc
    if x < 0:
        Q, x = Q + 1, x + M
    elif x >= M:
        Q, x = Q - 1, x - M
    assert 0 <= x < M
    u = b - (t * dec + Q * w)
    while t >= t0:
        for k, y in enumerate(range(x, J, M)):
            if 0 <= u - k * w <= W:
                out.append(y)
        t -= 1
        x, u = x + inc, u + dec
        if x >= M:
            x, u = x - M, u + w
    return out


def _missed(max_m: int, edge: float, bits: int, n: int) -> tuple[int, int]:
    """(lattices admitted, edge hits missed) over n primes' residues of about `bits` bits."""
    rng = random.Random(bits)
    admitted = missed = 0
    while n:
        n -= 1
        p = rng.getrandbits(bits) | (1 << (bits - 1)) | 1
        A = rng.randrange(1, p)
        if math.gcd(A, p) != 1:
            continue
        lat = _lattice(p, A)
        if lat[0] >= max_m or lat[2] >= 1 << 32:
            continue
        admitted += 1
        W = rng.choice([600, 7_500, 20_000, 131_070])
        J = min(p // (W + 1), 1 << 20)
        for x in [0, 1, J - 1] + [rng.randrange(min(J, 64)) for _ in range(3)] + [J - 1 - rng.randrange(min(J, 64))]:
            for u in (0, W, rng.randrange(W + 1)):
                b = (u - A * x) % p  # the residue at x = 0 of the sequence that is u at x
                for err in (0.0, RECIPROCAL, -RECIPROCAL):
                    missed += x not in _hits(p, lat, b, W, J, edge, err)
    return admitted, missed


@pytest.mark.parametrize("bits", [27, 31, 33, 34, 36, 37, 40])
def test_edge_hits_are_found(bits):
    max_m, edge = _limits()
    admitted, missed = _missed(max_m, edge, bits, 150)
    assert missed == 0 and (admitted >= 100 or bits > 36)


def test_every_prime_below_2_36_is_admitted():
    max_m, _ = _limits()
    rng = random.Random(3)
    for _ in range(300):
        p = (1 << 36) - 2 * rng.randrange(1 << 20) - 1
        A = rng.randrange(1, p)
        if math.gcd(A, p) == 1:
            assert _lattice(p, A)[0] < max_m


def test_the_limit_is_needed():
    """The same enumeration with M up to 2^30 misses hits of the largest primes accepted."""
    assert _missed(1 << 30, _limits()[1], 40, 150)[1] > 0
