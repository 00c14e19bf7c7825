"""The framework's work as its users have it done, case by case.

Each case is one call (or one short run of calls) of the public Python entry
points, with inputs made from a seed: a number or a window near the case's
nominal place, so that no two passes ask for the same thing.  ``listed`` gives
the fixed cases, ``draw`` more of the same kinds over the same ranges.

Kinds:

  point    next_prime and prev_prime of one number: the smallest call
  range    range_stats of [a, a + width)
  context  Context(N) and the queries that follow it, as in the README
  count    prime_count(N)
  list     in_range: the primes themselves
  goldbach the smallest p for every even n <= N (histogram, maximum, sum)
  batch    range_stats_batch of a mixed stream of ranges
  server   the same stream submitted to a request server with its four ops
"""
import math

import numpy as np

import voss_gb300 as vg
from voss_gb300 import serve
from voss_gb300.conjectures import goldbach_minp
from voss_gb300.primes import in_range, next_prime, prev_prime, prime_count, range_stats_batch

MAX_END = 10**14

SCALARS = ("a", "b", "count", "twins", "cousins", "sexy", "pi_4_1", "pi_4_3", "pi_3_1", "pi_3_2",
           "first_prime", "last_prime", "max_gap", "max_gap_start", "num_gaps", "large_gaps")


def listed():
    return [
        # A primality-neighbourhood query at a large offset: pure latency, a
        # window of a few thousand integers against all primes to 10^6.
        {"name": "next_prev_1e12", "kind": "point", "x": 1_234_567_890_123},
        # The narrow end of the serving mix: one short odd-sized window.
        {"name": "range_3e5_at_7e10", "kind": "range", "a": 70_000_000_001, "width": 300_007},
        # Every query of a small Context (C1's size), Sophie Germain included.
        {"name": "context_1e7", "kind": "context", "N": 10_000_019, "sophie": True},
        # The reference's second published size (C2).
        {"name": "context_1e10", "kind": "context", "N": 9_999_999_999, "sophie": False},
        # The headline: count, gaps and Chebyshev counts to 10^12.
        {"name": "context_1e12", "kind": "context", "N": 999_900_000_000, "sophie": False},
        # A count alone, which needs no gap scan; between the Context sizes.
        {"name": "count_3e10", "kind": "count", "N": 31_415_926_535},
        # High-offset windows (C3): wide at 10^12, narrower at 10^14.
        {"name": "window_1e10_at_1e12", "kind": "range", "a": 1_000_000_000_000, "width": 10_000_000_000},
        {"name": "window_1e9_at_1e14", "kind": "range", "a": 99_990_000_000_000, "width": 1_000_000_001},
        # The sorted primes of a window (about 3 * 10^5 of them).
        {"name": "list_8e6_at_1e11", "kind": "list", "a": 100_000_000_003, "width": 8_000_000},
        # Every even n to nearly 10^9 (C4).
        {"name": "goldbach_1e9", "kind": "goldbach", "N": 999_900_001},
        # The serving mix as one batched call, and through the server (C5).
        {"name": "batch_300", "kind": "batch", "n": 300},
        {"name": "server_1000", "kind": "server", "n": 1000},
    ]


def _log_int(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    kind = rng.choice(["point", "range", "range", "context", "count", "list", "goldbach", "batch", "server"])
    if kind == "point":
        return {"kind": kind, "x": _log_int(rng, 1e4, 9.9e13)}
    if kind == "range":
        width = _log_int(rng, 1e3, 1e10)
        return {"kind": kind, "a": min(_log_int(rng, 1e4, 9.9e13), MAX_END - 2 * width), "width": width}
    if kind == "context":
        N = _log_int(rng, 1e4, 9e11)
        return {"kind": kind, "N": N, "sophie": N < 10**9 and rng.random() < 0.5}
    if kind == "count":
        return {"kind": kind, "N": _log_int(rng, 1e4, 5e11)}
    if kind == "list":
        return {"kind": kind, "a": _log_int(rng, 1e4, 9.9e13), "width": _log_int(rng, 1e3, 2e7)}
    if kind == "goldbach":
        return {"kind": kind, "N": _log_int(rng, 1e5, 9.9e8)}
    return {"kind": kind, "n": _log_int(rng, 16, 400 if kind == "batch" else 1000)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _numbers(case, seed):
    """The call's own numbers: the case's, moved up by at most a thousandth."""
    r = np.random.default_rng([seed, 7])
    kind = case["kind"]
    if kind == "point":
        return {"x": case["x"] + int(r.integers(0, case["x"] // 1000))}
    if kind in ("range", "list"):
        a = case["a"] + int(r.integers(0, case["width"] + 1000))
        return {"a": a, "b": a + case["width"] + int(r.integers(0, case["width"] // 1000 + 1))}
    if kind in ("context", "count", "goldbach"):
        return {"N": case["N"] + int(r.integers(0, case["N"] // 10000 + 100))}
    return {"requests": serve.serving_mix(case["n"], seed=seed)}


def prepare(case, seed):
    state = dict(case, **_numbers(case, seed))
    if case["kind"] == "batch":
        state["ranges"] = [(q.a, q.b) for q in state["requests"]]
    if case["kind"] == "server":
        state["server"] = serve.Server()      # a long-lived service: made once, kept
    return state


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _stats(results):
    """RangeStats as two whole arrays: the scalars and the gap histograms."""
    return {"scalars": np.array([[getattr(s, n) for n in SCALARS] for s in results], dtype=np.int64),
            "hist": np.array([s.gap_hist for s in results], dtype=np.int64)}


def _padded(rows, room):
    """rows, then zeros up to `room` of them: one shape whatever the window."""
    out = np.zeros((room,) + np.shape(rows)[1:], dtype=np.int64)
    out[:len(rows)] = rows
    return out


def _listed_primes(primes, width):
    # a window of w integers holds fewer than 2 w / ln w primes
    return {"count": len(primes), "primes": _padded(primes, int(2.01 * width / math.log(width)) + 64)}


def _large_gaps(pairs):
    return _padded(np.array(pairs, dtype=np.int64).reshape(-1, 2), 64)     # 11 of them below 10^12


def _context(N, sophie):
    with vg.Context(N) as ctx:
        st = ctx.statistics()
        cb = ctx.chebyshev()
        out = {"pi": ctx.prime_count(), "twins": ctx.twins(), "cousin": ctx.cousin(), "sexy": ctx.sexy(),
               "moments": np.array([st.mean_gap, st.std_dev, st.skewness, st.kurtosis]),
               "total_gaps": st.total_gaps, "pi_4_1": cb.pi_4_1, "pi_4_3": cb.pi_4_3,
               "large": _large_gaps([(g.position, g.gap) for g in ctx.large_gaps()])}
        if sophie:
            out["sophie"] = ctx.sophie_germain()
    return out


def run(state):
    kind = state["kind"]
    if kind == "point":
        return {"next": next_prime(state["x"]), "prev": prev_prime(state["x"])}
    if kind == "range":
        return _stats([vg.range_stats(state["a"], state["b"])])
    if kind == "context":
        return _context(state["N"], state["sophie"])
    if kind == "count":
        return {"pi": prime_count(state["N"])}
    if kind == "list":
        return _listed_primes(in_range(state["a"], state["b"]), state["width"])
    if kind == "goldbach":
        g = goldbach_minp(state["N"], want_array=False)
        return {"hist": g["hist"].astype(np.int64), "max": g["max"], "sum": g["sum"],
                "counterexamples": g["counterexamples"]}
    if kind == "batch":
        return _stats(range_stats_batch(state["ranges"]))
    server = state["server"]
    tickets = [server.submit(q.a, q.b, q.op) for q in state["requests"]]
    return _stats([server.result(t)[0] for t in tickets])


# ---------------------------------------------------------------------------
# the work that no implementation by sieving can do without
# ---------------------------------------------------------------------------
def _sieve_ops(a, b):
    """Candidate clears of the primes above 17 (8 in 30 of the multiples),
    one reduction per sieving prime, and one step per wheel byte."""
    root = max(math.sqrt(b), 18.0)
    clears = (b - a) * (8 / 30) * (math.log(math.log(root)) - math.log(math.log(17.0)))
    return max(clears, 0.0) + root / math.log(root) + (b - a) / 30 + 1


def _union(ranges):
    """The disjoint pieces that ranges cover."""
    out = []
    for a, b in sorted(ranges):
        if out and a <= out[-1][1]:
            out[-1][1] = max(out[-1][1], b)
        else:
            out.append([a, b])
    return out


def work(case):
    kind = case["kind"]
    record = 8.0 * (len(SCALARS) + 202)
    if kind == "point":
        return {"bytes": 24.0, "flops": _sieve_ops(case["x"] - 60, case["x"] + 60)}
    if kind == "range":
        return {"bytes": record, "flops": _sieve_ops(case["a"], case["a"] + case["width"])}
    if kind == "context":
        ops = _sieve_ops(0, case["N"])
        if case["sophie"]:
            ops += _sieve_ops(case["N"], 2 * case["N"])
        return {"bytes": 8.0 * 12, "flops": ops}
    if kind == "count":
        return {"bytes": 16.0, "flops": _sieve_ops(0, case["N"])}
    if kind == "list":
        end = case["a"] + case["width"]
        return {"bytes": 8.0 * case["width"] / math.log(end) + 16, "flops": _sieve_ops(case["a"], end)}
    if kind == "goldbach":
        return {"bytes": 8.0 * 65536, "flops": _sieve_ops(0, case["N"]) + case["N"] / 2}
    mix = serve.serving_mix(case["n"])
    return {"bytes": (record + 20.0) * case["n"],
            "flops": sum(_sieve_ops(a, b) for a, b in _union([(q.a, q.b) for q in mix]))}


# ---------------------------------------------------------------------------
# the same results by a plain numpy sieve
# ---------------------------------------------------------------------------
def _primes(a, b):
    """The primes q with a <= q < b."""
    root = math.isqrt(max(b - 1, 0))
    small = np.ones(root + 1, dtype=bool)
    small[:2] = False
    for i in range(2, math.isqrt(root) + 1):
        if small[i]:
            small[i * i::i] = False
    seg = np.ones(b - a, dtype=bool)
    seg[:max(0, min(2, b) - a)] = False
    for p in np.nonzero(small)[0].tolist():
        first = max(p * p, -(-a // p) * p)
        if first < b:
            seg[first - a::p] = False
    return np.nonzero(seg)[0].astype(np.int64) + a


def _exact_range(a, b):
    q = _primes(a, b)
    g = np.diff(q)
    hist = np.bincount(np.minimum(g // 2, 201), minlength=202)[:202].astype(np.int64)
    top = int(g.max()) if g.size else 0
    # twins, cousins and sexy count the gaps 2, 4 and 6; 2 -> 3 is bin 0
    row = [a, b, q.size, hist[1], hist[2], hist[3],
           np.sum(q % 4 == 1), np.sum(q % 4 == 3), np.sum(q % 3 == 1), np.sum(q % 3 == 2),
           q[0] if q.size else 0, q[-1] if q.size else 0, top, q[int(g.argmax())] if g.size else 0,
           g.size, np.sum(g >= 500)]
    return {"scalars": np.array([row], dtype=np.int64), "hist": hist[None, :]}


def _exact_context(N, sophie):
    q = _primes(0, N + 1)
    g = np.diff(q)
    values, counts = np.unique(g, return_counts=True)
    total = counts.sum()
    mean = float((values * counts).sum()) / float(total)
    d = values.astype(np.float64) - mean
    var, m3, m4 = ((counts * d**k).sum() / total for k in (2, 3, 4))
    big = sorted(((-int(x), int(p)) for x, p in zip(g[g >= 500], q[1:][g >= 500])))
    out = {"pi": int(q.size), "twins": int(np.sum(g == 2)), "cousin": int(np.sum(g == 4)),
           "sexy": int(np.sum(g == 6)),
           "moments": np.array([mean, math.sqrt(var), m3 / var**1.5, m4 / var**2 - 3.0]),
           "total_gaps": int(total), "pi_4_1": int(np.sum(q % 4 == 1)), "pi_4_3": int(np.sum(q % 4 == 3)),
           "large": _large_gaps([(p, -x) for x, p in big])}
    if sophie:
        wide = np.zeros(2 * N + 2, dtype=bool)
        wide[_primes(0, 2 * N + 2)] = True
        out["sophie"] = int(wide[2 * q + 1].sum())
    return out


def exact(case, seed):
    kind, z = case["kind"], _numbers(case, seed) if case["kind"] not in ("batch", "server") else {}
    if kind == "point":
        near = _primes(max(z["x"] - 3000, 0), z["x"] + 3000)
        return {"next": int(near[near > z["x"]][0]), "prev": int(near[near < z["x"]][-1])}
    if kind == "range" and case["width"] <= 2 * 10**7:
        return _exact_range(z["a"], z["b"])
    if kind == "context" and z["N"] <= 2 * 10**8:
        return _exact_context(z["N"], case["sophie"])
    if kind == "count" and z["N"] <= 2 * 10**8:
        return {"pi": int(_primes(0, z["N"] + 1).size)}
    if kind == "list":
        return _listed_primes(_primes(z["a"], z["b"] + 1), case["width"])
    return None          # too long for a plain sieve: over about 20 seconds
