"""Performance cases of the sieve, through the package's public entry points.

Four kinds of work that a user of the package has it do:

  resident  a job stays loaded and one p-window after another is sieved:
            Sieve.run + Sieve.factors (what the command line does between two
            checkpoints).  A first pass over a window finds its factors; the
            counters are those of every pass.
  whole     a job from start to end: Sieve.load (the upload), run, factors and
            the final bitmap of candidates that are left.
  batch     several jobs of different shapes resident as templates, one work
            unit of each cloned, run to completion together, collected and
            released (what the serving loop does per unit).
  primes    the prime generator into caller-owned device memory, sorted, as a
            program that wants the primes themselves uses it.

Sizes are those of the benchmark workloads (rssieve_b200.workloads) and the
ranges around them: 1 to 100 sequences, bases 2 to 10, n-ranges of 10^5 to
10^7, p from 10^9 to just below 2^64, windows from 2^16 (the tail of a work
unit) to 2^28 (the command line's first window).  Near 2^50 a window of that
width holds next to no factor of a random job, so a few sequences of each job
are drawn such that a prime of the window divides one of their candidate terms.
"""
import ctypes
import math

import numpy as np
import torch

import rssieve_b200 as rs

# p_lo: the window starts at p_lo + U[0, p_jitter) (from the seed) and is p_width wide
_LISTED = [
    # the headline job: 100 sequences, n-range 6*10^6, p just above 2^50, the
    # command line's first window
    dict(name="hundred_seqs_2p50", kind="resident", base=2, seqs=100, n_lo=4_000_000, n_width=6_000_000, thin=5,
         p_lo=1 << 50, p_jitter=1 << 38, p_width=1 << 28, plant=8),
    # the same job's last few thousand primes: latency of the smallest call
    dict(name="hundred_seqs_tail", kind="resident", base=2, seqs=100, n_lo=4_000_000, n_width=6_000_000, thin=5,
         p_lo=1 << 50, p_jitter=1 << 38, p_width=1 << 16, plant=4),
    # a served unit's file (1..100 sequences) above 2^51, where most of the
    # served p-ranges (2^44..2^62, log-uniform) lie
    dict(name="served_file_2p58", kind="resident", base=2, seqs=61, n_lo=4_000_000, n_width=6_000_000, thin=5,
         p_lo=1 << 58, p_jitter=1 << 50, p_width=1 << 25, plant=6),
    # 20 sequences in base 5 just below 2^64
    dict(name="base5_below_2p64", kind="resident", base=5, seqs=20, n_lo=1_000_000, n_width=2_000_000, thin=4,
         p_lo=(1 << 64) - (1 << 36), p_jitter=1 << 35, p_width=1 << 26, plant=6),
    # many sequences over a short n-range (the mixed-jobs workload's job 15):
    # little search per prime
    dict(name="short_n_base6", kind="resident", base=6, seqs=68, n_lo=1_000_000, n_width=103_125, thin=4,
         p_lo=1_730_000_000_000_000, p_jitter=1 << 40, p_width=1 << 26, plant=8),
    # one sequence over a long n-range, base 10
    dict(name="one_seq_base10", kind="resident", base=10, seqs=1, n_lo=1_000_000, n_width=9_999_991, thin=4,
         p_lo=1 << 45, p_jitter=1 << 40, p_width=(1 << 25) + 12_345, plant=1),
    # a small window, odd everywhere, across the p where the arithmetic changes
    dict(name="odd_window_across_2p51", kind="resident", base=3, seqs=37, n_lo=1_000_001, n_width=777_777, thin=4,
         p_lo=(1 << 51) - 1_300_001, p_jitter=200_000, p_width=2_345_679, plant=5),
    # a small project's whole work unit, from its file to its result: 8
    # sequences k*2^n-1, p from 10^12 over 10^8
    dict(name="whole_unit_8_seqs", kind="whole", base=2, seqs=8, n_lo=100_000, n_width=200_000, thin=4,
         p_lo=10 ** 12, p_jitter=1 << 34, p_width=10 ** 8, plant=8),
    # an early sieve, where terms are still eliminated by the thousand
    dict(name="whole_early_p1e9", kind="whole", base=3, seqs=30, n_lo=50_000, n_width=300_000, thin=2,
         p_lo=10 ** 9, p_jitter=1 << 24, p_width=1 << 22, plant=0),
    # units of twelve jobs of mixed shapes (bases, sequence counts, n-ranges,
    # p from 2^44 to 2^60) at once
    dict(name="batch_12_jobs", kind="batch", jobs=12, job_seed=3, split=2, p_width=1 << 22, plant=3),
    # the generator's widest call
    dict(name="primes_2p22_wide", kind="primes", p_lo=1 << 50, p_jitter=1 << 40, p_width=1 << 22),
]


def listed():
    return [dict(c) for c in _LISTED]


def _log(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    kind = rng.choice(["resident"] * 5 + ["whole"] * 2 + ["batch", "primes"])
    p_lo = int(2 ** rng.uniform(40, 63.9))
    if kind == "primes":
        return dict(kind=kind, p_lo=p_lo, p_jitter=1 << 36, p_width=_log(rng, 10_000, 1 << 22))
    if kind == "batch":
        return dict(kind=kind, jobs=rng.randint(2, 12), job_seed=rng.randrange(1 << 20), split=rng.randint(1, 4),
                    p_width=_log(rng, 1 << 18, 1 << 22), plant=2)
    n_width = _log(rng, 10 ** 5, 10 ** 7) if kind == "resident" else _log(rng, 10 ** 5, 10 ** 6)
    return dict(kind=kind, base=rng.choice([2, 2, 2, 3, 5, 6, 10]), seqs=_log(rng, 1, 100.99),
                n_lo=rng.randint(100_000, 4_000_000), n_width=n_width, thin=rng.randint(3, 5), p_lo=p_lo,
                p_jitter=1 << 36, p_width=_log(rng, 1 << 16, 1 << 26), plant=4)


def _candidates(rng, seqs, n_width, thin):
    """Random bitmap with a density of 2^-thin (3% to 25%), bits past the n-range clear."""
    words = (n_width + 31) // 32
    bits = rng.integers(0, 1 << 32, size=(seqs, words), dtype=np.uint32)
    for _ in range(thin - 1):
        bits &= rng.integers(0, 1 << 32, size=(seqs, words), dtype=np.uint32)
    if n_width % 32:
        bits[:, -1] &= np.uint32((1 << (n_width % 32)) - 1)
    return bits


def _job(rng, base, seqs, n_lo, n_width, thin, p0, p1, plant):
    """Sequences k*b^n+-1 with odd terms, k < 2^32; for `plant` of them k is the residue
    that makes a prime of [p0, p1) divide one candidate term."""
    odd = 1 if base % 2 == 0 else 0
    ks = [int(k) // 2 * 2 + odd for k in rng.integers(4, 1 << 32, size=seqs)]
    cs = [1 if i < seqs // 2 else -1 for i in range(seqs)]
    bits = _candidates(rng, seqs, n_width, thin)
    for i in rng.permutation(seqs)[:plant]:
        p = p0 + int(rng.integers(0, p1 - p0))
        p = min(max(p | 1, p0 | 1), (p1 - 2) | 1)
        while p >= p0 and not rs.is_prime(p):
            p -= 2
        if p < p0:
            continue
        n = n_lo + int(rng.integers(0, n_width - 1000))
        k = -cs[i] * pow(base, -n, p) % p
        while k % 2 != odd:
            n += 1
            k = -cs[i] * pow(base, -n, p) % p
            if n == n_lo + n_width - 1:
                break
        if k % 2 != odd:
            continue
        ks[i] = k
        bits[i, (n - n_lo) >> 5] |= np.uint32(1 << ((n - n_lo) & 31))
    return rs.Seqs.create(base, ks, cs, n_lo, n_lo + n_width - 1, bits)


def _window(case, rng):
    p0 = case["p_lo"] + int(rng.integers(0, case["p_jitter"]))
    return p0, min(p0 + case["p_width"], (1 << 64) - 1)


def _batch_shapes(case):
    """The batch's jobs: shapes from the case alone, as the mixed-jobs workload draws them."""
    g = np.random.default_rng(case["job_seed"])
    return [dict(base=int(g.choice([2, 3, 5, 6, 10])), seqs=int(g.integers(1, 101)), n_lo=1_000_000,
                 n_width=int(math.exp(g.uniform(math.log(10 ** 5), math.log(3 * 10 ** 6)))), thin=int(g.integers(3, 6)),
                 p_lo=int(2 ** g.uniform(44, 60))) for _ in range(case["jobs"])]


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    st = {"case": case}
    if case["kind"] == "primes":
        st["p0"], st["p1"] = _window(case, rng)
        st["out"] = torch.empty((case["p_width"] + 1) // 2 + 1, dtype=torch.int64, device="cuda")
        st["count"] = torch.zeros(1, dtype=torch.int32, device="cuda")
        return st
    if case["kind"] == "batch":
        n = case["jobs"]
        st["batch"] = rs.Batch(0, max_jobs=2 * n, range_slots=5 * n)
        st["units"], st["room"] = [], []
        for s in _batch_shapes(case):
            p0 = s["p_lo"] + int(rng.integers(0, 1 << 36))
            p1 = p0 + case["p_width"]
            seqs = _job(rng, s["base"], s["seqs"], s["n_lo"], s["n_width"], s["thin"], p0, p1, case["plant"])
            st["units"].append((st["batch"].add(seqs, 3, 3), p0, p1))
            st["room"].append(_room(s["seqs"], s["n_width"], s["thin"], s["p_lo"], case["p_width"], case["plant"]))
        return st
    p0, p1 = st["window"] = _window(case, rng)
    st["seqs"] = _job(rng, case["base"], case["seqs"], case["n_lo"], case["n_width"], case["thin"], p0, p1, case["plant"])
    st["room"] = _room(case["seqs"], case["n_width"], case["thin"], case["p_lo"], case["p_width"], case["plant"])
    st["sieve"] = rs.Sieve(0)
    if case["kind"] == "resident":
        st["sieve"].load(st["seqs"])
    return st


def _room(seqs, n_width, thin, p, p_width, plant):
    """Entries that the factors of a window fit in, many times over: expected plus planted."""
    return 64 + 4 * plant + int(2 * seqs * n_width / 2 ** thin * _primes_in(p, p_width) / p)


def _terms(factors, room, with_p=True):
    """The number of factors, and the factors in the order of their terms, each column as an
    array of `room` entries (zeros past the last).  With many factors per window a term may
    have several prime divisors, any of which may claim it: its p is then left out."""
    f = factors[np.lexsort((factors["n"], factors["seq"]))]
    table = np.zeros((3 if with_p else 2, max(room, len(f))), dtype=np.int64)
    for row, column in zip(table, ("seq", "n", "p")):
        row[: len(f)] = f[column].view(np.int64) if column == "p" else f[column]
    return [len(f), table]


def run(state):
    case = state["case"]
    if case["kind"] == "primes":
        out, count = state["out"], state["count"]
        rc = rs.lib().rs_primes_generate_noalloc(state["p0"], state["p1"], out.data_ptr(), out.numel(), count.data_ptr(),
                                                 ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc != rs.RS_OK:
            raise RuntimeError(rs.lib().rs_last_error().decode())
        n = int(count.item())
        sorted_primes = torch.zeros_like(out)                # zeros past the last
        sorted_primes[:n] = torch.sort(out[:n]).values
        return [n, sorted_primes]
    if case["kind"] == "batch":
        b, got = state["batch"], []
        ids = [b.add_clone(src, p0, p1, case["split"]) for src, p0, p1 in state["units"]]
        b.run()
        for j, room in zip(ids, state["room"]):
            _, primes, done = b.job_info(j)
            got.append([int(primes), bool(done)] + _terms(b.factors(j), room))
            b.release(j)
        return {"primes": np.array([g[0] for g in got]), "done": np.array([g[1] for g in got]),
                "factors": np.array([g[2] for g in got]), "terms": np.concatenate([g[3] for g in got], axis=1)}
    s = state["sieve"]
    if case["kind"] == "whole":
        s.load(state["seqs"])
    counters = s.run(*state["window"])
    got = {"primes": counters["primes"], "hits": counters["hits"],
           "terms": _terms(s.factors(), state["room"], case["p_lo"] >= 1 << 39)}
    if case["kind"] == "whole":
        got["left"] = s.bitmap()
    return got


def _primes_in(p, width):
    return width / math.log(p)


def _search(base, seqs, n_width, p, width):
    """Floating-point operations that a search cannot do without, as modular products of nine
    operations: per prime one power per sequence (which classes of n it can divide), and baby and
    giant steps of about 2 sqrt(sequences * n-range / 16) (the split into classes averaged)."""
    per_prime = seqs * math.log2(p) + 2 * math.sqrt(seqs * n_width / 16)
    return 9.0 * per_prime * _primes_in(p, width)


def work(case):
    if case["kind"] == "primes":
        n = _primes_in(case["p_lo"], case["p_width"])
        return {"bytes": 8 * n, "flops": 9.0 * n * 5 * math.log2(case["p_lo"])}
    if case["kind"] == "batch":
        shapes = _batch_shapes(case)
        return {"bytes": 16.0 * case["jobs"] * max(case["plant"], 1),
                "flops": sum(_search(s["base"], s["seqs"], s["n_width"], s["p_lo"], case["p_width"]) for s in shapes)}
    # the whole job's bitmap goes in and comes back; a resident job's (a
    # template's) stays where it is
    moved = 2 * case["seqs"] * case["n_width"] / 8 if case["kind"] == "whole" else 16.0 * max(case["plant"], 1)
    return {"bytes": moved, "flops": _search(case["base"], case["seqs"], case["n_width"], case["p_lo"], case["p_width"])}


def _primes_between(lo, hi):
    """Sieve of Eratosthenes over [lo, hi) by every prime up to sqrt(hi)."""
    root = math.isqrt(hi) + 1
    small = np.ones(root // 2 + 1, dtype=bool)          # index i: 2i + 1
    small[0] = False
    for i in range(1, math.isqrt(root) // 2 + 1):
        if small[i]:
            small[2 * i * (i + 1):: 2 * i + 1] = False
    q = 2 * np.flatnonzero(small).astype(np.int64) + 1
    base = max(lo, 3) | 1
    keep = np.ones(max(0, (hi - base + 1) // 2), dtype=bool)
    first = np.maximum((base + q - 1) // q, q) * q
    first += np.where(first % 2 == 0, q, 0)             # the first odd multiple in the range, from q^2 on
    at = (first - base) // 2
    wide = q > keep.size                                 # at most one multiple in the range
    one = at[wide]
    keep[one[one < keep.size]] = False
    for a, r in zip(at[~wide].tolist(), q[~wide].tolist()):
        keep[a::r] = False
    return base + 2 * np.flatnonzero(keep).astype(np.int64)


def exact(case, seed):
    """The generator's primes by a plain sieve where that takes seconds.  The searches have no
    such value: every term and prime by itself would take hours."""
    if case["kind"] != "primes" or case["p_lo"] + case["p_jitter"] > 1 << 52:
        return None
    p0, p1 = _window(case, np.random.default_rng(seed))
    primes = _primes_between(p0, p1)
    padded = np.zeros((case["p_width"] + 1) // 2 + 1, dtype=np.int64)
    padded[: len(primes)] = primes
    return [len(primes), padded]
