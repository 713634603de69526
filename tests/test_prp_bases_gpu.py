"""Bases side by side: base 2 decides a composite as soon as it would in turn, and the first failing base is the one
reported, whatever order the bases end in."""
from __future__ import annotations

import math
import random

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

MERSENNE = [31, 61, 89, 107, 127, 521, 607, 1279, 2203, 3217, 4253]
SHAPES = [(4, 40), (8, 64), (16, 64), (16, 1024), (17, 124), (20, 125), (22, 12), (23, 257), (24, 69), (24, 70), (28, 300), (25, 296), (25, 297),
          (32, 128), (32, 1024), (40, 161), (47, 189), (48, 257), (64, 40), (96, 20), (136, 12), (144, 5), (144, 74)]


def _ms(pg, ctx, words, values, rounds):
    a = np.stack([np.frombuffer(v.to_bytes(4 * words, "little"), dtype=np.uint32) for v in values])
    x = torch.from_numpy(a.view(np.int32).copy()).cuda()
    out = torch.full((len(values),), -7, dtype=torch.int32, device="cuda")
    stream, best = torch.cuda.Stream(), 1e9
    for _ in range(4):
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            rc = pg.lib.pg_prp_batch_device(ctx.handle, x.data_ptr(), len(values), words, rounds, out.data_ptr(),
                                            stream.cuda_stream)
            e1.record()
        assert rc == pg.PG_OK
        stream.synchronize()
        best = min(best, e0.elapsed_time(e1))
    return best, out.cpu().numpy()


def _one_thread_ms(pg, words, values):
    """Base 2 on one thread per number: a next-prime search of one step."""
    import ctypes
    nxt = pg.lib.pg_next_prime_noalloc
    nxt.argtypes = [ctypes.c_void_p, ctypes.c_uint32, ctypes.c_uint32, ctypes.c_uint32, ctypes.c_void_p, ctypes.c_void_p]
    a = np.stack([np.frombuffer(v.to_bytes(4 * words, "little"), dtype=np.uint32) for v in values])
    x = torch.from_numpy(a.view(np.int32).copy()).cuda()
    steps = torch.empty(len(values), dtype=torch.int32, device="cuda")
    stream, best = torch.cuda.Stream(), 1e9
    stream.wait_stream(torch.cuda.current_stream())
    for _ in range(4):
        with torch.cuda.stream(stream):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            assert nxt(x.data_ptr(), len(values), words, 1, steps.data_ptr(), stream.cuda_stream) == pg.PG_OK
            e1.record()
        stream.synchronize()
        best = min(best, e0.elapsed_time(e1))
    assert (steps.cpu().numpy() == -1).all()
    return best


@pytest.mark.parametrize("words,n", SHAPES)
def test_composites_cost_no_more_than_in_turn(pg, ctx, words, n):
    """A batch without a prime, 16 bases side by side, against base 2 on one thread per number (above 48 words, against
    a batch too large for bases side by side, which still takes the time of one test): a tenth for the clocks, 20 us
    for the launches."""
    rng, values = random.Random(words), []
    small = math.prod(q for q in range(2, 3_000) if all(q % r for r in range(2, int(q ** 0.5) + 1)))
    while len(values) < max(n, 300):  # composites that no trial division finds
        x = (rng.getrandbits(32 * words - 20) | 1 << (32 * words - 21) | 1) * 65_537
        if math.gcd(x, small) == 1:
            values.append(x)
    side, out = _ms(pg, ctx, words, values[:n], 16)
    assert not out.any()
    in_turn = _one_thread_ms(pg, words, values[:n]) if words <= 48 else _ms(pg, ctx, words, values[:300], 16)[0]
    assert side <= 1.1 * in_turn + 0.02


@pytest.mark.parametrize("words,n", [(20, 1025), (21, 1025), (23, 4096), (24, 1025), (25, 1025), (28, 1792), (32, 2048),
                                     (47, 3008), (48, 4096)])
def test_primes_cost_no_more_than_in_turn(pg, ctx, words, n):
    """More numbers than groups take side by side, all prime, 16 bases, against 4 097, which take the bases in turn on
    one thread each and no longer than fewer would: a tenth for the clocks."""
    values = [2 ** max(x for x in MERSENNE if x < 32 * words - 1) - 1] * 4_097
    side, out = _ms(pg, ctx, words, values[:n], 16)
    assert (out == 16).all()
    assert side <= 1.1 * _ms(pg, ctx, words, values, 16)[0]


@pytest.mark.parametrize("words,n", SHAPES)
def test_first_failing_base(pg, ctx, oracle, words, n):
    """Primes, composites, pseudoprimes of the first bases, tiny, even and zero numbers in one batch."""
    fixed = [0, 1, 2, 3, 5, 7, 9, 25, 47, 53, 54, 55, 2047, 3277, 1373653, 25326001, 3215031751, 2152302898747,
             3474749660383, 341550071728321, 3825123056546413051, 2 ** 61 - 1, 2 ** 31 - 1]
    top = 1 << (32 * words - 2)
    e = max(x for x in MERSENNE if x < 32 * words - 1)
    rng = random.Random(n)
    values = (fixed + [2 ** e - 1, top + 1, top - 1, (2 ** e - 1) * 3])[-n:]
    values += [2 ** e - 1 if rng.random() < 0.1 else rng.getrandbits(32 * words - 2) | 1 for _ in range(n - len(values))]
    values = [v for v in values if v < 1 << 128] if words == 4 else values
    rng.shuffle(values)
    cut = range(len(values)) if len(values) <= 80 else sorted(rng.sample(range(len(values)), 80))
    for rounds in (2, 5, 16):
        out = _ms(pg, ctx, words, values, rounds)[1]
        assert [int(out[i]) for i in cut] == [oracle.prp(values[i], rounds) for i in cut]
