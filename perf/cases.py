"""The sieve's work as its users run it, for timing: one dict per case.

  listed()            the cases
  draw(rng)           one more case of the same ranges
  prepare(case, seed) what a user's program holds before the call
  run(state)          one pass through the public entry points
  work(case)          bytes and operations one pass cannot do without
  exact(case, seed)   None: every output is a whole number

Kinds of cases:
  sieve   a resident job over one p window (rsieve.Job.sieve)
  abcd    the same from the job's ABCD text: create, sieve, destroy, as one run
          of the command line does
  batch   many uneven jobs over their own windows (rsieve.Batch)
  primes  the device prime sieve alone (rs_gpu_primes of the C ABI, into the caller's buffer)

The k, the candidates n and the exact start of the p window follow from the
seed; a case fixes base, sign, the number and size of the k, the range of n,
the share of n still in the sieve and about where p lies.
"""
import ctypes
import math
import os
import sys

import numpy as np

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "cuda-riesel-sieve_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import rsieve  # noqa: E402
from rsieve import synth  # noqa: E402

MULS = 19  # 32-bit multiplications of one 64-bit modular product
# A drawn case stays below the largest listed one in modular products and in candidates.
MOST_PRODUCTS = 1.2e11
MOST_N = 2e9  # k times width of the n range
MOST_HITS = 4000.0
ROWS = 8192


def _sieve(name, base, nk, kmax, nmin, width, density, p, window, sign=-1, datless=False, kind="sieve"):
    return {"name": name, "kind": kind, "base": base, "sign": sign, "nk": nk, "kmax": kmax, "nmin": nmin,
            "width": width, "density": density, "p": p, "window": window, "datless": datless}


def listed():
    return [
        # The benchmark's job (base 745, 22 k, n 180000..250000): a few seconds' share of a long run at 1e13.
        _sieve("plain_1e13", 745, 22, 10**6, 180000, 70001, 0.05, 10**13, 10**9),
        # The same job at the start of a sieve's life, where p is below 2^32 and a window has few primes.
        _sieve("plain_1e9", 745, 22, 10**6, 180000, 70001, 0.05, 10**9, 2 * 10**7),
        # The smallest call: a narrow window, as a client that hands out small ranges or resumes asks for.
        _sieve("narrow_1e13", 745, 22, 10**6, 180000, 70001, 0.05, 10**13, 10**5),
        # Every n of the range reported (the reference's -v), where the reference's own default window lies.
        _sieve("datless_1e14", 745, 22, 29587, 182644, 67357, 0.05, 102297149770000, 3 * 10**8, datless=True),
        # One sequence over a wide range of n: the search for a single k.
        _sieve("single_k", 5, 1, 10**5, 10**5, 2 * 10**6, 0.02, 10**15, 10**9),
        # A handful of Sierpinski sequences (k*b^n+1) of middling width.
        _sieve("sierpinski_7k", 13, 7, 10**6, 4 * 10**5, 300000, 0.04, 1 << 52, 5 * 10**8, sign=1),
        # Mixed jobs: an odd number of k, an odd width, large p.
        _sieve("mixed_131k", 97, 131, 10**7, 523457, 187321, 0.03, 1 << 57, 2 * 10**8),
        _sieve("mixed_467k", 230, 467, 10**7, 350003, 911111, 0.07, 1 << 59, 5 * 10**7),
        # The wide job: base 2, 1000 k, n 1e6..3e6 at 2^50.
        _sieve("wide_2_50", 2, 1000, 10**7, 10**6, 2000001, 0.02, 1 << 50, 6 * 10**7),
        # One run of the command line on a short range: text in, factors out.
        _sieve("abcd_1e13", 745, 22, 10**6, 180000, 70001, 0.05, 10**13, 2 * 10**8, kind="abcd"),
        # Many small requests of uneven shape sieved together.
        {"name": "batch_12", "kind": "batch", "jobs": 12, "shape": 1, "window": 2 * 10**7},
        # The prime generator alone.
        {"name": "primes_1e13", "kind": "primes", "p": 10**13, "window": 10**8},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _bases():
    return [b for b in range(2, 1025) if not synth._is_perfect_power(b)]


def draw(rng):
    kind = rng.choices(["sieve", "abcd", "batch", "primes"], [16, 2, 1, 1])[0]
    if kind == "primes":
        return {"kind": kind, "p": int(_log(rng, 10**9, 1 << 50)), "window": int(_log(rng, 10**5, 10**8))}
    if kind == "batch":
        return {"kind": kind, "jobs": rng.randint(2, 12), "shape": rng.randrange(1 << 20),
                "window": int(_log(rng, 10**6, 2 * 10**7))}
    while True:
        nk = round(_log(rng, 1, 60 if kind == "abcd" else 1000))
        width = round(_log(rng, 1e4, 2e6))
        if nk * width > MOST_N:
            continue
        datless = rng.random() < 0.15
        density = rng.uniform(0.01, 0.1)
        # a job of many candidates is sieved at large p: at small p it would have millions of factors
        p = int(_log(rng, 10**9 if nk * width < 3e6 else 10**12, 1 << 60))
        per_prime = 2.0 * math.sqrt(nk * width / 2.0)
        primes = _log(rng, 3000.0, max(4000.0, MOST_PRODUCTS / 2 / per_prime))
        window = min(primes * math.log(p), 10**9, p / 10)
        hits = window / math.log(p) * nk * width * (1.0 if datless else density) / p
        if window < 1000 or hits > MOST_HITS:
            continue
        return {"kind": kind, "base": rng.choice(_bases()), "sign": rng.choice([-1, -1, 1]), "nk": nk,
                "kmax": round(_log(rng, max(2e4, 40 * nk), 1e7)), "nmin": rng.randint(10**5, 10**6),
                "width": width, "density": density, "p": p, "window": int(window), "datless": datless}


def _job(rng, base, sign, nk, kmax, nmin, width, density):
    """ks and their lists of n: distinct odd k, gaps between the n as in a sieved file."""
    ks = np.zeros(0, dtype=np.int64)
    while len(ks) < nk:
        ks = np.unique(np.concatenate([ks, rng.integers(1, kmax // 2, nk, dtype=np.int64) * 2 + 1]))
    ks = np.sort(rng.permutation(ks)[:nk]).astype(np.uint32)
    most = int(width * density + 6 * math.sqrt(width * density) + 16)
    gaps = rng.standard_exponential((nk, most), dtype=np.float32)
    gaps *= np.float32(-1.0 / math.log1p(-density))
    n = np.cumsum(gaps.astype(np.int32) + 1, axis=1, dtype=np.int32)
    n += np.int32(nmin - 1)
    nlists = []
    for row in n:
        row = row[: int(np.searchsorted(row, nmin + width))]
        nlists.append(row.astype(np.uint32) if len(row) else np.array([nmin], dtype=np.uint32))
    return base, sign, ks, nlists


def _shapes(case):
    """The jobs of a batch: the mixed distribution (synth.batch_job), without its few largest."""
    bases, got, i = _bases(), [], 0
    while len(got) < case["jobs"]:
        u = synth.uniform(case["shape"], f"batch{i}", 8)
        i += 1
        nk = max(1, min(1000, round(math.exp(u[1] * math.log(1000.0)))))
        width = round(math.exp(math.log(1e4) + u[3] * (math.log(2e6) - math.log(1e4))))
        if nk * width > 2e8:
            continue
        got.append({"base": bases[int(u[0] * len(bases))], "nk": nk, "nmin": 10**5 + int(u[2] * 9e5), "width": width,
                    "density": 0.01 + u[4] * 0.09, "p": int(1e12 + u[5] * ((1 << 60) - 1e12))})
    return got


def prepare(case, seed):
    rng = np.random.default_rng([seed, 20])
    kind = case["kind"]
    start = lambda p: int(p) + int(rng.integers(0, max(1, int(p) // 1000)))  # noqa: E731
    if kind == "primes":
        p0 = start(case["p"])
        room = int(1.3 * _primes(case["p"], case["window"])) + 1024
        return {"kind": kind, "p0": p0, "p1": p0 + case["window"] - 1, "out": np.zeros(room, dtype=np.int64)}
    if kind == "batch":
        jobs = []
        for s in _shapes(case):
            b, sign, ks, nl = _job(rng, s["base"], -1, s["nk"], 10**7, s["nmin"], s["width"], s["density"])
            p0 = start(s["p"])
            jobs.append((rsieve.Job(base=b, sign=sign, ks=ks, nlists=nl, mem_limit=1 << 29), p0,
                         p0 + case["window"] - 1))
        return {"kind": kind, "jobs": jobs}
    b, sign, ks, nl = _job(rng, case["base"], case["sign"], case["nk"], case["kmax"], case["nmin"], case["width"],
                           case["density"])
    p0 = start(case["p"])
    st = {"kind": kind, "p0": p0, "p1": p0 + case["window"] - 1, "datless": int(case["datless"])}
    if kind == "abcd":
        st["text"] = synth.to_abcd(b, sign, ks, nl).encode()
    else:
        st["job"] = rsieve.Job(base=b, sign=sign, ks=ks, nlists=nl, datless=st["datless"])
    return st


def _out(results):
    """(factors, stats) of one or more jobs: all factors, in room for ROWS of them, and each job's number of primes."""
    got = np.zeros((6, ROWS), dtype=np.int64)
    at = 0
    for i, (f, _) in enumerate(results):
        for row, col in zip(got, ("p", "k", "n", "b", "c")):
            row[at : at + len(f)] = f[col]
        got[5, at : at + len(f)] = i + 1
        at += len(f)
    return {"factors": got, "primes": np.array([st["primes"] for _, st in results], dtype=np.int64)}


def run(state):
    kind = state["kind"]
    if kind == "primes":
        out, count = state["out"], ctypes.c_size_t(0)
        rsieve._check(rsieve.lib().rs_gpu_primes(state["p0"], state["p1"], out.ctypes.data, len(out), count, 0))
        return {"primes": out, "count": count.value}
    if kind == "batch":
        with rsieve.Batch() as batch:
            items = [batch.add(*j) for j in state["jobs"]]
            batch.run()
            return _out([batch.result(i) for i in items])
    if kind == "abcd":
        with rsieve.Job(state["text"], datless=state["datless"]) as job:
            return _out([job.sieve(state["p0"], state["p1"])])
    return _out([state["job"].sieve(state["p0"], state["p1"])])


def _primes(p, window):
    return window / math.log(p)


def work(case):
    """Bytes: candidates as bits, primes or factors out.  Operations: marking the window's composites, and
    2*sqrt(R*X) modular products per prime, R rows of X exponents of which half pass the quadratic character."""
    if case["kind"] == "primes":
        n = _primes(case["p"], case["window"])
        return {"bytes": 8.0 * n, "flops": case["window"] / 2.0 * math.log(math.log(case["p"]))}
    got = {"bytes": 0.0, "flops": 0.0}
    for s in _shapes(case) if case["kind"] == "batch" else [case]:
        n = _primes(s["p"], case["window"])
        got["bytes"] += s["nk"] * s["width"] / 8.0 + 24.0 * n * s["nk"] * s["width"] * s["density"] / s["p"]
        got["flops"] += n * 2.0 * math.sqrt(s["nk"] * s["width"] / 2.0) * MULS
    return got


def exact(case, seed):
    return None
