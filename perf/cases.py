"""Cases that time the framework's public entry points over the range of work users give it.

listed() names the cases, draw() gives more of the same ranges, prepare()
makes what a program holds before the call (numbers, a context, a job with
its prime tables, a running server), run() is one pass through the public
interface and returns its outputs whole, work() is what a pass cannot do
without, exact() the verdicts of plain Python integers where they are cheap.

Kinds
  prp       strong probable-prime tests of a batch: from host memory
            (Context.prp_words, the reference's test_runner_t::run_test) or
            on device buffers (pg_prp_batch_device)
  search    Job.search of one window of m: previous and next prime gap
  pipeline  the same over consecutive windows, PG_SEARCH_SLOTS in flight
            (Job.submit / Job.wait), each launch capped at 6 warps per SM
  sieve     Job.sieve_interval: the sieve rows of a window
  serve     a mix of requests through a running Server
"""
from __future__ import annotations

import importlib
import math
import random

import numpy as np
import torch

pg = importlib.import_module("prime-gap-gpu_b200")

# the searched configurations: d, search radius, first m of the range, its length
CONFIGS = {
    337: dict(d=2310, sl=7_500, m_lo=10_000_000, m_span=1_000_000, bits=462),
    503: dict(d=2190, sl=10_000, m_lo=1_000_000, m_span=800_000, bits=703),
    907: dict(d=210, sl=18_000, m_lo=1_000_000, m_span=800_000, bits=1274),
    3001: dict(d=2190, sl=40_000, m_lo=1, m_span=90_000, bits=4248),
}
FIRST_PRIMES = (2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31, 37, 41, 43, 47, 53)


def _prp(name, words, n, rounds=1, primes=False, device=False):
    return dict(name=name, kind="prp", words=words, n=n, rounds=rounds, primes=primes, device=device)


def _search(name, P, m_inc, limit, confirm=0.0, plain=False):
    return dict(name=name, kind="search", P=P, m_inc=m_inc, limit=limit, confirm=confirm, plain=plain)


def listed() -> list[dict]:
    return [
        # the ends of a few record gaps checked with 16 bases (as Job.records does), a false one here and there:
        # the smallest call
        _prp("confirm-703b-12", 22, 12, rounds=16, primes=True),
        # a batch of candidates handed over from host memory, the reference's smallest build
        _prp("prp-512b-4096", 16, 4096),
        # a large batch that already lies on the device, 1024 bits
        _prp("prp-1024b-65536", 32, 65_536, device=True),
        # wide operands (the size of P = 3001 candidates), from host memory
        _prp("prp-4352b-2048", 136, 2_048),
        # the small configuration: P = 337, 10 000 m, primes <= 1e8
        _search("search-P337", 337, 10_000, 100_000_000, confirm=20.0),
        # a short request: a few hundred coprime m, where fixed costs and the window's tail count
        _search("search-P503-short", 503, 1_500, 1_000_000_000),
        # the headline window: P = 503, 200 000 m, primes <= 2e9, records above merit 22 confirmed
        _search("search-P503", 503, 200_000, 2_000_000_000, confirm=22.0),
        # a long run as the command line tool makes it: windows one after the other, two in flight
        dict(name="pipeline-P503", kind="pipeline", P=503, m_inc=50_000, windows=4, limit=2_000_000_000,
             confirm=22.0),
        # wider operands and primes above 2^32: P = 907, primes <= 1e10
        _search("search-P907", 907, 20_000, 10_000_000_000, confirm=24.0),
        # the widest operands: a slice of the P = 3001 range, primes <= 1e10
        _search("search-P3001", 3001, 150, 10_000_000_000, confirm=25.0),
        # sieve rows alone, back in host memory
        dict(name="sieve-P503", kind="sieve", P=503, m_inc=20_001, limit=2_000_000_000),
        # a server working through a queue of requests of three operand widths
        dict(name="serve-mix", kind="serve", requests=15, limit=1_000_000_000),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random) -> dict:
    c = _drawn(rng)
    c.pop("name", None)
    return c


def _drawn(rng: random.Random) -> dict:
    kind = rng.choice(["prp", "prp", "prp", "search", "search", "search", "sieve", "pipeline", "serve"])
    if kind == "prp":
        words = _logint(rng, 6, 140)
        if rng.random() < 0.25:  # a few records' ends
            return _prp("", words, rng.randint(8, 40), rounds=16, primes=words <= 48)
        top = max(16, min(200_000, int(3.0e11 / (32 * words) ** 3 * 1000)))
        return _prp("", words, _logint(rng, 8, top), device=rng.random() < 0.4)
    P = rng.choice([337, 503, 503, 907])
    limit = rng.choice([100_000_000, 300_000_000, 1_000_000_000])
    top = {337: 100_000, 503: 100_000, 907: 15_000}[P]
    if kind == "search":
        return _search("", P, _logint(rng, 300, top), limit, confirm=rng.choice([0.0, 20.0]),
                       plain=rng.random() < 0.15)
    if kind == "pipeline":
        return dict(kind="pipeline", P=P, m_inc=_logint(rng, 1_000, top // 4), windows=rng.randint(3, 6), limit=limit,
                    confirm=20.0)
    if kind == "sieve":
        return dict(kind="sieve", P=P, m_inc=_logint(rng, 300, 40_000), limit=limit)
    return dict(kind="serve", requests=rng.randint(4, 15), limit=limit)


# ------------------------------------------------------------------- inputs

def _strong(n: int, base: int) -> bool:
    s = ((n - 1) & (1 - n)).bit_length() - 1
    x = pow(base, (n - 1) >> s, n)
    if x in (1, n - 1):
        return True
    for _ in range(s - 1):
        x = x * x % n
        if x == n - 1:
            return True
    return False


_TRIAL = [q for q in range(3, 2000, 2) if all(q % r for r in range(3, int(q ** 0.5) + 1, 2))]


def _prime_above(n: int) -> int:
    n |= 1
    while any(n % q == 0 for q in _TRIAL) or not _strong(n, 2):
        n += 2
    return n


def _numbers(case: dict, seed: int) -> np.ndarray:
    """(n, words) odd numbers of 32*words - 2 bits: random ones with a few primes among them, as the sieve's
    survivors are, or mostly primes (the ends of record gaps)."""
    words, n = case["words"], case["n"]
    rng = np.random.default_rng([seed, words, n])
    a = rng.integers(0, 2 ** 32, size=(n, words), dtype=np.uint32)
    a[:, 0] |= 1
    a[:, -1] = (a[:, -1] >> 2) | (1 << 29)
    if case["primes"]:
        where = np.nonzero(rng.random(n) < 0.8)[0]
    else:
        where = rng.choice(n, size=rng.integers(1, min(8, n // 2) + 1), replace=False)
    for i in where:
        if not case["primes"]:
            a[i, 22:] = 0  # narrow enough to be found at once
        p = _prime_above(int.from_bytes(a[i].tobytes(), "little"))
        a[i] = np.frombuffer(p.to_bytes(4 * words, "little"), dtype=np.uint32)
    return a


def _window_start(case: dict, seed: int, windows: int = 1) -> int:
    # one residue mod d for every seed: the same number of m coprime to d
    c = CONFIGS[case["P"]]
    room = (c["m_span"] - windows * case["m_inc"]) // c["d"]
    return c["m_lo"] + c["d"] * random.Random(seed * 7919 + case["P"]).randrange(room)


def _job(case: dict, confirm: float):
    c = CONFIGS[case["P"]]
    return pg.Job(case["P"], c["d"], c["sl"], case["limit"], max_m_inc=case["m_inc"],
                  max_m=c["m_lo"] + c["m_span"], confirm_merit=confirm)


SERVED = ((337, 2310, 3_800), (503, 2190, 5_500), (907, 210, 10_200))  # P, d, sl = about 8 ln N


def _requests(case: dict, seed: int) -> list[tuple]:
    """Requests of 500 to 20 000 m from [1e6, 1e9], the three widths in turn."""
    rng = random.Random(seed)
    out = []
    for i in range(case["requests"]):
        P, d, sl = SERVED[i % 3]
        inc = int(500 * 40 ** ((i * 7 % 15) / 14)) + i % 2
        out.append((P, d, sl, case["limit"], 1_000_000 + d * rng.randrange(999_000_000 // d), inc))
    return out


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    st = {"case": case}
    if kind == "prp":
        a = _numbers(case, seed)
        st["ctx"] = pg.Context(0)
        if case["device"]:
            st["numbers"] = torch.from_numpy(a.view(np.int32)).cuda()
            st["passed"] = torch.empty(case["n"], dtype=torch.int32, device="cuda")
            st["stream"] = torch.cuda.Stream()
        else:
            st["numbers"] = a
    elif kind == "serve":
        st["requests"] = _requests(case, seed)
        st["server"] = pg.Server(0, max_sl=max(sl for _, _, sl in SERVED))
        # a running server holds the tables of the widths it serves
        for i in [st["server"].submit(P, d, 1_000, case["limit"], 1_000_001, 200) for P, d, _ in SERVED]:
            st["server"].wait(i)
    else:
        st["job"] = _job(case, case.get("confirm", 0.0))
        st["m_start"] = _window_start(case, seed, case.get("windows", 1))
    return st


# --------------------------------------------------------------------- pass

def run(st: dict):
    case = st["case"]
    kind = case["kind"]
    if kind == "prp":
        if not case["device"]:
            return st["ctx"].prp_words(st["numbers"], case["rounds"])
        rc = pg.lib.pg_prp_batch_device(st["ctx"].handle, st["numbers"].data_ptr(), case["n"], case["words"],
                                        case["rounds"], st["passed"].data_ptr(), st["stream"].cuda_stream)
        if rc != pg.PG_OK:
            raise RuntimeError(pg.lib.pg_last_error().decode())
        return st["passed"]
    if kind == "search":
        r = st["job"].search(st["m_start"], case["m_inc"],
                             pg.PG_SEARCH_PLAIN if case["plain"] else pg.PG_SEARCH_PERSISTENT)
        return {"ms": r.ms, "prev": r.prev_gap, "next": r.next_gap}
    if kind == "pipeline":
        job, tickets, out = st["job"], [], []
        for w in range(case["windows"]):
            if len(tickets) == pg.PG_SEARCH_SLOTS:
                out.append(job.wait(tickets.pop(0)))
            tickets.append(job.submit(st["m_start"] + w * case["m_inc"], case["m_inc"], pg.PG_SEARCH_PERSISTENT,
                                      pg.PG_SUBMIT_WARPS_PER_SM(6)))
        out += [job.wait(t) for t in tickets]
        return [{"ms": r.ms, "prev": r.prev_gap, "next": r.next_gap} for r in out]
    if kind == "sieve":
        ms, rows = st["job"].sieve_interval(st["m_start"], case["m_inc"])
        return {"ms": ms, "rows": rows}
    srv = st["server"]
    res = [srv.wait(i) for i in [srv.submit(*r) for r in st["requests"]]]
    return [{"ms": r.ms, "prev": r.prev_gap, "next": r.next_gap} for r in res]


# --------------------------------------------------------------------- work

def _test_flops(bits: int) -> float:
    """One strong base-2 test: a squaring and a reduction per bit, 1.5 L^2 products of 32-bit words, a multiply
    and an add each."""
    return bits * 1.5 * (bits / 32) ** 2 * 2


def _tests_per_m(bits: int, limit: int) -> float:
    """Candidates tested per m until both primes are found, sieved to `limit` (Mertens)."""
    return 2 * bits * math.log(2) / (1.781 * math.log(limit))


def _primes(limit: int) -> float:
    return limit / math.log(limit) * (1 + 1 / math.log(limit))


def _coprime(m_inc: int, d: int) -> int:
    return max(1, round(m_inc * sum(math.gcd(r, d) == 1 for r in range(d)) / d))


def _search_work(P: int, d: int, bits: int, sl: int, m_inc: int, limit: int, tables: int = 1) -> tuple[float, float]:
    nm = _coprime(m_inc, d)
    prime_bytes = 12 if limit < 2 ** 32 else 24
    return (tables * _primes(limit) * prime_bytes + nm * 16, nm * _tests_per_m(bits, limit) * _test_flops(bits))


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "prp":
        bits = 32 * case["words"] - 2
        tests = case["n"] * (case["rounds"] if case["primes"] else 1)
        return {"bytes": case["n"] * (4 * case["words"] + 4), "flops": tests * _test_flops(bits)}
    if kind == "serve":
        b = f = 0.0
        for P, d, sl, limit, start, inc in _requests(case, 0):
            x, y = _search_work(P, d, CONFIGS[P]["bits"] + (0 if P == 337 else 10), sl, inc, limit)
            b, f = b + x, f + y
        return {"bytes": b, "flops": f}
    c = CONFIGS[case["P"]]
    if kind == "sieve":
        nm = _coprime(case["m_inc"], c["d"])
        prime_bytes = 12 if case["limit"] < 2 ** 32 else 24
        rows = nm * ((c["sl"] // 2 * 2 + 32) // 32) * 4
        # one O(log p) search a prime, a few operations a level
        return {"bytes": _primes(case["limit"]) * prime_bytes + rows, "flops": _primes(case["limit"]) * 40}
    w = case.get("windows", 1)
    b, f = _search_work(case["P"], c["d"], c["bits"], c["sl"], case["m_inc"], case["limit"])
    return {"bytes": w * b, "flops": w * f}


def exact(case: dict, seed: int):
    """The verdicts by Python integers, where they take a few seconds."""
    if case["kind"] != "prp":
        return None
    bits = 32 * case["words"]
    bases = FIRST_PRIMES[:case["rounds"]]
    tests = case["n"] * (len(bases) if case["primes"] else 1)
    if tests * 0.4e-3 * (bits / 703) ** 2.6 > 8:
        return None
    out = []
    for row in _numbers(case, seed):
        n = int.from_bytes(row.tobytes(), "little")
        passed = 0
        for b in bases:
            if not _strong(n, b):
                break
            passed += 1
        out.append(passed)
    return np.array(out, dtype=np.int32)
