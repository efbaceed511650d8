"""The search kernel at the edges of its classes, segments and filter queue.

A prime is searched by a group of 32 << c threads with 512 << c baby steps
(class c), its giant phase dealt as items of several rounds and, when long, cut
into segments.  Every case compares eliminated terms, bitmap and duplicates
with the brute-force oracle: whole numbers, equal or not.
"""
import numpy as np
import pytest

from rssieve_b200 import workloads as W
from tests.conftest import oracle_job

pytestmark = pytest.mark.gpu

CASES = [
    # kcount, base, n-range, p0, width, Q (0: chosen)
    (1, 2, 40_000, 3, 30_000, 0),                     # orders from 1 to beyond the largest Q'
    (100, 2, 40_000, 500, 2_000, 1024),               # p just above Q': most filter passes true, the queue overflows
    (100, 3, 60_000, 60_000, 4_000, 1024),            # the same with p past the largest class
    (2, 2, 3_000_000, 1_000_000, 2_000, 1024),        # few targets, many chunks: second-level start powers, segments
    (1, 10, 2_000_000, 20_000_000, 20_000, 0),        # one target: G up to its limit
    (100, 2, 1_500_000, 50_000_000, 4_000, 1024),     # segments of many rounds
    (33, 5, 700_001, 10_000_000, 12_000, 0),          # items past the last one in a round
    (64, 6, 1_000, 100_000, 20_000, 0),               # n-range shorter than one giant step
    (100, 2, 900_000, 3_000_000, 4_000, 16384),       # 1024-thread CTAs
]


@pytest.mark.parametrize("kcount,base,width,p0,pw,q", CASES)
def test_search_matches_brute_force(sieve, oracle, kcount, base, width, p0, pw, q):
    job = W.small_job(90 + kcount + base, kcount=kcount, base=base, nmin=1001, nmax=1000 + width, keep=0.2, kmax=1 << 24)
    sieve.set_baby_steps(q)
    try:
        sieve.load(W.seqs_of(job))
        cnt = sieve.run(p0, p0 + pw)
        fac, bm = sieve.factors(), sieve.bitmap()
    finally:
        sieve.set_baby_steps(0)
    plist = oracle.primes(p0, p0 + pw)
    ofac, odups, obm = oracle.brute(oracle_job(oracle, job), plist, ref_skip=True)
    assert cnt["primes"] == len(plist)
    assert oracle.term_set(fac) == oracle.term_set(ofac)
    assert np.array_equal(bm, obm)
    assert cnt["dups"] == odups


@pytest.mark.parametrize("p0", [(1 << 45) + 7, (1 << 51) - 2_000, (1 << 57) + 11, (1 << 62) - 5_000, (1 << 63) + 3])
@pytest.mark.parametrize("kcount,width", [(1, 50_000), (40, 400_000)])
def test_planted_factors_in_every_step_kind(sieve, oracle, p0, kcount, width):
    """Primes of each step kind (FP64, Shoup, Montgomery, and a window across
    2^51): every sequence gets a k that one prime of the window divides a term of."""
    rng = np.random.default_rng(p0 % 1000 + kcount)
    plist = oracle.primes(p0, p0 + 3_000)
    nmin, ks, cs, want = 10_001, [], [], set()
    for i in range(kcount):
        p, c, n = int(rng.choice(plist)), 1 if i % 2 else -1, nmin + int(rng.integers(0, width))
        ks.append(-c * pow(2, -n, p) % p)
        cs.append(c)
        want.add((i, n))
    job = W.job_dict(2, ks, cs, nmin, nmin + width - 1, W.random_bitmap(kcount, nmin, nmin + width - 1, 1.0, 1))
    sieve.load(W.seqs_of(job))
    sieve.run(p0, p0 + 3_000)
    got = oracle.term_set(sieve.factors())
    # a term may be hit by chance as well: at most width * kcount * primes / p, far below one
    assert want == got


def _planted(sieve, oracle, base, kcount, nmin, nmax, p0, p1, seed, q=0):
    """A job whose only candidates are terms that a prime of [p0, p1) divides, one
    per sequence: every one of them has to go, and nothing else."""
    rng = np.random.default_rng(seed)
    plist = oracle.primes(p0, p1)
    ks, cs, want = [], [], set()
    bm = np.zeros((kcount, (nmax - nmin + 32) // 32), dtype=np.uint32)
    for i in range(kcount):
        k, c = base % 2, 1 if i % 2 else -1
        while k % 2 == base % 2:                                # odd terms
            p, n = int(rng.choice(plist)), (nmin, nmax, int(rng.integers(nmin, nmax + 1)))[i % 3]
            k = -c * pow(base, -n, p) % p
        ks.append(k)
        cs.append(c)
        bm[i, (n - nmin) >> 5] |= np.uint32(1 << ((n - nmin) & 31))
        want.add((i, n))
    sieve.set_baby_steps(q)
    try:
        sieve.load(W.seqs_of(W.job_dict(base, ks, cs, nmin, nmax, bm)))
        cnt = sieve.run(p0, p1)
        got = oracle.term_set(sieve.factors())
        left = sieve.bitmap()
    finally:
        sieve.set_baby_steps(0)
    assert cnt["primes"] == len(plist)
    assert got == want
    assert not left.any()


@pytest.mark.parametrize("nmin", [1, 200, 9_000])      # n-ranges of 2^32 - 1 and a little below: L + e - 1, L + Q' - 1 pass 2^32
@pytest.mark.parametrize("p0", [(1 << 47) + 1, (1 << 57) + 1])
def test_n_range_of_32_bits(sieve, oracle, nmin, p0):
    _planted(sieve, oracle, 2, 3, nmin, (1 << 32) - 1, p0, p0 + 2_000, nmin)


# Sequence counts at every step of the set-up's lanes per prime (4, 8, 16, 32) and of
# its last, partial round of powers, shared by four primes of a warp once a chunk has
# about 19000 primes: the window has 25000 or more.
@pytest.mark.parametrize("kcount", [1, 4, 5, 8, 9, 16, 17, 20, 24, 25, 31, 32, 33, 56, 57, 64, 68, 87, 88, 89, 96, 97, 100])
@pytest.mark.parametrize("p0", [(1 << 49) + 5, (1 << 59) + 5])
def test_sequence_counts(sieve, oracle, kcount, p0):
    _planted(sieve, oracle, 3 if kcount % 2 else 10, kcount, 5_001, 25_000, p0, p0 + 1_100_000, kcount)


# The split modulus goes up to 256 from sequences * n-range of 6.5*10^6 (one sequence),
# 8*10^6 (4), 10^7 (8) and 1.4*10^7 (16) on: n-ranges at the line and one past it.
@pytest.mark.parametrize("kcount", [1, 4, 8, 16])
@pytest.mark.parametrize("past", [0, 1])
def test_split_limit_of_few_sequences(sieve, oracle, kcount, past):
    width = (6_000_000 + 500_000 * kcount) // kcount + past
    for p0 in ((1 << 44) + 1, (1 << 56) + 1):
        _planted(sieve, oracle, 2, kcount, 1_001, 1_000 + width, p0, p0 + 20_000, 31 + kcount)
