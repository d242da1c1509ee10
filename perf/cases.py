"""The calls that a program makes of this framework, as timed cases.

Every case goes through the Python face of libvoss.so (`voss.Context` and `mr_verify_noalloc`).
A case names its kind, its sizes and where on the number line it works; the seed moves the
inputs inside that neighbourhood, so that no two seeds ask for the same numbers.

  range      [1, N] with every statistic, in the mode that the CSV artifacts are written from
  slice      [lo, lo + len) of a long run that is cut into slices, high up the number line
  intervals  a batch of independent intervals (batched queries, one launch)
  mr         Miller-Rabin of candidates in host memory: half primes, half random odd 64-bit
  mr_device  the same of random odd 64-bit candidates that lie on the GPU, on torch's stream
  gaps       every gap >= min_gap of a window listed, and each proved (verification)
  primes     the first `count` primes from lo on, as an array
  certs      SHA-256 digests of gap certificates
"""
import math
import os
import sys

import numpy as np

_PKG = os.path.abspath("voss-prime-gaps_v1_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

SEG_NUM = 30_000_000_000  # the segment length of the reference's artifacts
LARGE_DTYPE = np.dtype([("position", "<u8"), ("gap", "<i4"), ("merit", "<f4")])  # a record of a gap list
EXACT_SPAN = 1_100_000_000  # longest window that plain numpy sieves in a few seconds


def listed():
    return [
        # one short query: what a single interval costs when nothing hides its latency
        {"name": "interval_one", "kind": "intervals", "count": 1, "start_min": 1e11, "start_max": 1e12,
         "len_min": 1e6, "len_max": 2e6},
        # the smallest published run of the reference: [1, 10^9]
        {"name": "range_1e9", "kind": "range", "n": 1_000_000_000},
        # the headline run: [1, 10^12]
        {"name": "range_1e12", "kind": "range", "n": 1_000_000_000_000},
        # a slice of a run near 10^15, with ends that are multiples of nothing
        {"name": "slice_1e15", "kind": "slice", "lo": 1_000_000_000_000_007, "len": 4_700_000_003},
        # the batched-interval workload: uneven lengths, starts over six decades
        {"name": "intervals_4096", "kind": "intervals", "count": 4096, "start_min": 1e10, "start_max": 1e16,
         "len_min": 1e4, "len_max": 1e8},
        # short queries at high starts
        {"name": "intervals_short_1e18", "kind": "intervals", "count": 1000, "start_min": 1e15, "start_max": 1e18,
         "len_min": 1e3, "len_max": 1e5},
        # a handful of numbers to check
        {"name": "mr_1000", "kind": "mr", "count": 1000, "below": 1_000_000_000_000},
        # a verification batch from host memory
        {"name": "mr_1e7", "kind": "mr", "count": 10_000_000, "below": 1_000_000_000_000},
        # the largest batch that the call without allocations takes, less a ragged end
        {"name": "mr_device_4e6", "kind": "mr_device", "count": 4_000_001},
        # verification of the large gaps of a window near 10^12
        {"name": "gaps_1e12", "kind": "gaps", "lo": 999_000_000_000, "len": 1_000_000_001, "min_gap": 200},
        # a prime list for another program
        {"name": "primes_3e6", "kind": "primes", "lo": 1_000_000_000_003, "count": 3_000_001},
        # the certificates of a list of large gaps
        {"name": "certs_50000", "kind": "certs", "count": 50_000},
    ]


def _log(rng, a, b):
    return 10.0 ** rng.uniform(math.log10(a), math.log10(b))


def draw(rng):
    kind = rng.choice(["range", "slice", "intervals", "intervals", "mr", "mr_device", "gaps", "primes", "certs"])
    if kind == "range":  # shorter than the largest listed one
        return {"kind": kind, "n": int(_log(rng, 1e8, 5e11))}
    if kind == "slice":
        return {"kind": kind, "lo": int(_log(rng, 1e12, 5e15)), "len": int(_log(rng, 1e8, 1e10)) | 1}
    if kind == "intervals":
        count = int(_log(rng, 1, 4096))
        if rng.random() < 0.5:
            return {"kind": kind, "count": count, "start_min": 1e10, "start_max": 1e16, "len_min": 1e4,
                    "len_max": float(int(_log(rng, 1e5, 1e8)))}
        return {"kind": kind, "count": count, "start_min": 1e9, "start_max": 1e18, "len_min": 1e2,
                "len_max": float(int(_log(rng, 1e3, 1e5)))}
    if kind == "mr":
        return {"kind": kind, "count": int(_log(rng, 100, 1e7)), "below": int(_log(rng, 1e10, 5e15))}
    if kind == "mr_device":
        return {"kind": kind, "count": int(_log(rng, 100, 4194304))}
    if kind == "gaps":
        return {"kind": kind, "lo": int(_log(rng, 1e10, 1e13)), "len": int(_log(rng, 1e8, 1e10)) | 1,
                "min_gap": rng.randrange(150, 301, 2)}
    if kind == "primes":
        return {"kind": kind, "lo": int(_log(rng, 1e9, 1e15)), "count": int(_log(rng, 3e3, 6e6)) | 1}
    return {"kind": kind, "count": int(_log(rng, 100, 2e5))}


# A program keeps one context per limit (its base primes lie on the GPU) for all its calls.
_CONTEXTS = {}


def _context(max_hi):
    import voss
    limit = 10**9 + 1
    while limit < max_hi:
        limit = 10 * (limit - 1) + 1
    if limit > 10**18:
        limit = 10**18 + 10**9
    if limit not in _CONTEXTS:
        _CONTEXTS[limit] = voss.Context(limit)
    return _CONTEXTS[limit]


def _rng(seed):
    return np.random.default_rng([20261203, int(seed)])


def _window(case, seed):
    """A window of the case's length (for primes: of that many primes and a tenth more), moved up
    by less than its length over ten."""
    ln = case["len"] if "len" in case else int(1.1 * case["count"] * math.log(2 * case["lo"]))
    lo = case["lo"] + int(_rng(seed).integers(1, ln // 10))
    return lo, lo + ln


def _list_room(case):
    """Room for a case's list of gaps: a program keeps one array for them (the rest of it is zero)."""
    if case["kind"] == "gaps":
        log = math.log(case["lo"])
        return int(1.5 * case["len"] / log * math.exp(-case["min_gap"] / (log - 1))) + 2000
    hi, ln = (case["n"], case["n"]) if case["kind"] == "range" else (case["lo"] + case["len"], case["len"])
    return int(0.3 * ln / math.log(hi) * math.exp(-10)) + 2000


def _into(room, found):
    """The list in the program's own array: its length moves with the seed, the array's does not."""
    room[: found.size] = found
    return room


def _range_end(case, seed):
    """N: at most a thousandth below the case's."""
    return case["n"] - int(_rng(seed).integers(0, case["n"] // 1000))


def prepare(case, seed):
    kind = case["kind"]
    rng = _rng(seed)
    st = {"kind": kind}
    if kind == "range":
        n = _range_end(case, seed)
        st.update(ctx=_context(case["n"] + 1), n=n, large=np.zeros(_list_room(case), dtype=LARGE_DTYPE))
    elif kind in ("slice", "gaps"):
        lo, hi = _window(case, seed)
        st.update(ctx=_context(hi + case["len"]), lo=lo, hi=hi, large=np.zeros(_list_room(case), dtype=LARGE_DTYPE))
        if kind == "gaps":
            st.update(min_gap=case["min_gap"], proved=np.zeros(_list_room(case), dtype=np.uint8))
    elif kind == "primes":
        lo, hi = _window(case, seed)
        st.update(ctx=_context(2 * hi), lo=lo, hi=hi, count=case["count"])
    elif kind == "intervals":
        k = case["count"]
        lo = np.floor(10.0 ** rng.uniform(math.log10(case["start_min"]), math.log10(case["start_max"]), k))
        ln = np.floor(10.0 ** rng.uniform(math.log10(case["len_min"]), math.log10(case["len_max"]), k))
        lo = lo.astype(np.uint64) + rng.integers(0, 1000, size=k, dtype=np.uint64)  # a double's are even up there
        st.update(ctx=_context(int(case["start_max"] + case["len_max"]) + 1000), lo=lo, hi=lo + ln.astype(np.uint64))
    elif kind == "mr":
        ctx = _context(case["below"])
        half = case["count"] // 2
        span = int(half * 1.1 * math.log(case["below"])) + 10**5
        top = case["below"] - int(rng.integers(1, 10**6))
        primes = ctx.primes_range(max(2, top - span), top)[-half:]
        odd = rng.integers(0, 2**63, size=case["count"] - primes.size, dtype=np.uint64) * 2 + 1
        st.update(ctx=ctx, n=rng.permutation(np.concatenate([primes, odd])))
    elif kind == "mr_device":
        import torch
        odd = rng.integers(0, 2**63, size=case["count"], dtype=np.uint64) * 2 + 1
        st.update(n=torch.from_numpy(odd.view(np.int64)).cuda(),
                  ok=torch.empty(case["count"], dtype=torch.uint8, device="cuda"))
    elif kind == "certs":
        p = rng.integers(10**9, 10**12, size=case["count"], dtype=np.uint64)
        g = 2 * rng.integers(100, 350, size=case["count"], dtype=np.uint64)
        merit = g / np.log(p)
        st.update(ctx=_context(10**9),
                  messages=[b"VOSS|%d|%d|%d|%.6f" % (a, a + b, b, m)
                            for a, b, m in zip(p.tolist(), g.tolist(), merit.tolist())])
    return st


def _range_outputs(r, room):
    large = _into(room, r.large)
    return {"prime_count": r.prime_count, "first_prime": r.first_prime, "last_prime": r.last_prime,
            "max_gap": r.max_gap, "max_gap_lo": r.max_gap_lo, "mod4": r.mod4, "modq": r.modq,
            "modq_gap": r.modq_gap, "gap_hist": r.gap_hist, "large_total": r.large_total,
            "large_position": large["position"], "large_gap": large["gap"], "merit": large["merit"]}


_RANGE_KEYS = ("prime_count", "first_prime", "last_prime", "max_gap", "max_gap_lo", "mod4", "modq", "modq_gap",
               "gap_hist", "large_total", "large_position", "large_gap", "merit")


def run(st):
    kind = st["kind"]
    if kind == "range":
        return _range_outputs(st["ctx"].sieve_range(1, st["n"] + 1, compat=True, seg_num=SEG_NUM), st["large"])
    if kind == "slice":
        return _range_outputs(st["ctx"].sieve_range(st["lo"], st["hi"]), st["large"])
    if kind == "intervals":
        out = st["ctx"].sieve_intervals(st["lo"], st["hi"])
        return {k: out[k] for k in out.dtype.names}
    if kind == "mr":
        return st["ctx"].mr_verify(st["n"])
    if kind == "mr_device":
        import torch
        import voss.api
        voss.api.mr_verify_noalloc(st["n"].data_ptr(), st["n"].numel(), st["ok"].data_ptr(),
                                   torch.cuda.current_stream().cuda_stream)
        return st["ok"]
    if kind == "gaps":
        gaps = st["ctx"].gaps_at_least(st["lo"], st["hi"], st["min_gap"])
        proved = st["ctx"].prove_gaps(gaps["position"], gaps["gap"])
        gaps = _into(st["large"], gaps)
        return {"position": gaps["position"], "gap": gaps["gap"], "merit": gaps["merit"],
                "proved": _into(st["proved"], proved)}
    if kind == "primes":
        return st["ctx"].primes_range(st["lo"], st["hi"], st["count"])
    return st["ctx"].sha256_batch(st["messages"])


def _clears(lo, hi):
    """Multiples, coprime to 30, of the primes from 7 to the root of hi in [lo, hi): what a wheel
    sieve strikes out (sum of 1/p by Mertens)."""
    if hi < 49:
        return 0.0
    return (hi - lo) * (8 / 30) * max(0.0, math.log(math.log(math.sqrt(hi))) + 0.2615 - 1 / 2 - 1 / 3 - 1 / 5)


def _root_primes(hi):
    s = math.sqrt(hi)
    return s / max(1.0, math.log(s) - 1.08)


def work(case):
    """bytes: inputs and results, and the base primes once (4 bytes each).  flops: integer
    operations, one for each multiple struck out, one for each prime's statistics, and for
    Miller-Rabin one 64-bit product for each bit of a candidate that needs a test."""
    kind = case["kind"]
    result = 8 * (100_000 + 99 + 1000 + 16)  # the statistics of a range
    if kind == "range":
        n = case["n"]
        return {"bytes": result + 4 * _root_primes(n), "flops": _clears(1, n) + n / math.log(n)}
    if kind == "slice":
        lo, ln = case["lo"], case["len"]
        return {"bytes": result + 4 * _root_primes(lo + ln), "flops": _clears(lo, lo + ln) + ln / math.log(lo)}
    if kind == "intervals":
        mid = math.sqrt(case["start_min"] * case["start_max"])
        a, b = case["len_min"], case["len_max"]
        mean = (b - a) / math.log(b / a) if b > a else a
        return {"bytes": case["count"] * (16 + 8 * (8 + 1024)),
                "flops": case["count"] * (_clears(mid, mid + mean) + mean / math.log(mid))}
    if kind == "mr":
        n = case["count"]
        return {"bytes": 9 * n, "flops": n * (0.5 * math.log2(case["below"]) + 0.5 * 0.27 * 63)}
    if kind == "mr_device":
        return {"bytes": 9 * case["count"], "flops": case["count"] * 0.27 * 63}
    if kind == "gaps":
        lo, ln = case["lo"], case["len"]
        found = ln / math.log(lo) * math.exp(-case["min_gap"] / math.log(lo))
        return {"bytes": 4 * _root_primes(lo + ln) + 17 * found,
                "flops": _clears(lo, lo + ln) + ln / math.log(lo) + found * 0.13 * case["min_gap"] * math.log2(lo)}
    if kind == "primes":
        lo, n = case["lo"], case["count"]
        ln = n * math.log(lo)
        return {"bytes": 4 * _root_primes(lo + ln) + 8 * n, "flops": _clears(lo, lo + ln)}
    return {"bytes": case["count"] * (38 + 32), "flops": case["count"] * 64 * 20}


def _primes_between(lo, hi):
    """The primes of [lo, hi) by a plain sieve over odd numbers, in pieces that fit a cache."""
    root = math.isqrt(hi)
    small = np.ones(root + 1, dtype=bool)
    small[:2] = False
    for p in range(2, math.isqrt(root) + 1):
        if small[p]:
            small[p * p::p] = False
    base = [int(p) for p in np.flatnonzero(small) if p > 2]
    found = [np.array([2], dtype=np.uint64)] if lo <= 2 < hi else []
    lo |= 1
    piece = 1 << 25
    for a in range(lo, hi, 2 * piece):
        size = min(piece, (hi - a + 1) // 2)
        odd = np.ones(size, dtype=bool)  # slot i: the number a + 2 i
        for p in base:
            m = max(p * p, (a + p - 1) // p * p)
            if m % 2 == 0:
                m += p
            odd[(m - a) // 2::p] = False
        if a <= 1:
            odd[(1 - a) // 2] = False
        found.append(np.uint64(a) + 2 * np.flatnonzero(odd).astype(np.uint64))
    return np.concatenate(found)


def exact(case, seed):
    """The merits (gap over the logarithm of the lower prime) of the listed gaps in 64 bits; the
    other outputs are whole numbers and bytes."""
    if case["kind"] == "range" and case["n"] <= EXACT_SPAN:
        p = _primes_between(7, _range_end(case, seed) + 1)
        merit = np.diff(p) / np.log(p[:-1])
        keep = (np.diff(p) > 100) & ((np.diff(p) >= 500) | (merit >= 10.0))
        return {k: _into(np.zeros(_list_room(case)), merit[keep]) if k == "merit" else None for k in _RANGE_KEYS}
    if case["kind"] == "gaps" and case["len"] <= EXACT_SPAN:
        p = _primes_between(*_window(case, seed))
        merit = np.diff(p) / np.log(p[:-1])
        listed_gaps = merit[np.diff(p) >= case["min_gap"]]
        return {"position": None, "gap": None, "merit": _into(np.zeros(_list_room(case)), listed_gaps), "proved": None}
    return None
