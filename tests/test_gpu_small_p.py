"""Searches at small p, where solutions are many: filter passes are mostly true, the
queue of passes may overflow, and ord(b^e) often lies below the baby-step count.

Compared with the brute-force oracle: eliminated terms, bitmap and duplicates, whole
numbers, equal or not.
"""
import numpy as np
import pytest

from rssieve_b200 import workloads as W
from tests.conftest import oracle_job

pytestmark = pytest.mark.gpu


def _against_brute(sieve, oracle, job, p0, p1, q):
    sieve.set_baby_steps(q)
    try:
        sieve.load(W.seqs_of(job))
        cnt = sieve.run(p0, p1)
        fac, bm = sieve.factors(), sieve.bitmap()
    finally:
        sieve.set_baby_steps(0)
    plist = oracle.primes(p0, p1)
    ofac, odups, obm = oracle.brute(oracle_job(oracle, job), plist, ref_skip=True)
    assert cnt["primes"] == len(plist)
    assert oracle.term_set(fac) == oracle.term_set(ofac)
    assert np.array_equal(bm, obm)
    assert cnt["dups"] == odups
    return cnt


# kcount, base, n-range, p0, width, Q
CASES = [
    (100, 2, 600_000, 30, 1_000, 0),            # few targets with many claims each, some with none
    (30, 3, 300_000, 1_000, 2_000, 0),          # the order's bound from below Q' to above
    (8, 2, 200_000, 900, 2_500, 1024),          # orders around 512 and 1024 baby steps
    (1, 10, 2_000_000, 3, 5_000, 0),
    (100, 2, 1_000_000, 16_000, 1_500, 8192),   # orders just above the largest Q': nearly every value is there
    (100, 2, 1_000_000, 32_700, 800, 16384),
    (20, 5, 500_000, 100_000, 3_000, 2048),     # passes on one value in ten: segments of one step
    (60, 2, 2_000_000, 1_000_000, 3_000, 4096),
]


@pytest.mark.parametrize("kcount,base,width,p0,pw,q", CASES)
def test_small_p_matches_brute_force(sieve, oracle, kcount, base, width, p0, pw, q):
    job = W.small_job(700 + kcount + base, kcount=kcount, base=base, nmin=1001, nmax=1000 + width, keep=0.2, kmax=1 << 24)
    _against_brute(sieve, oracle, job, p0, p0 + pw, q)


# Large p with a small order of the base (31, 61, 19, 192), one per step kind or more:
# every term of a kept sequence in one class of n is divisible.
@pytest.mark.parametrize("base,p", [(2, (1 << 31) - 1), (2, (1 << 61) - 1), (10, (10 ** 19 - 1) // 9),
                                    (2, (1 << 64) - (1 << 32) + 1)])
@pytest.mark.parametrize("kcount", [3, 40])
def test_small_order_at_large_p(sieve, oracle, base, p, kcount):
    nmin, width, ks, cs = 5_000, 60_000, [], []
    for i in range(kcount):
        c = 1 if i % 2 else -1
        ks.append(-c * pow(base, -(nmin + 7 * i), p) % p if i % 3 else 1_000_003 + 2 * i)
        cs.append(c)
    job = W.job_dict(base, ks, cs, nmin, nmin + width - 1, W.random_bitmap(kcount, nmin, nmin + width - 1, 0.5, 3))
    cnt = _against_brute(sieve, oracle, job, p - 1, p + 1, 0)
    assert cnt["small_order"] == 1 and cnt["hits"] > 0


def test_claims_of_small_orders_fill_the_group(sieve):
    """100 sequences, n-range 6*10^6, the primes from 100 to 1000: 10^8 solutions and
    more, each an atomic on the bitmap.  With the chip full these take 0.04 ns each; 143
    primes, some with many more than others, leave part of it idle.  The bound is five
    times that (32 threads for a prime of up to 10^6 solutions: 0.43)."""
    job = W.small_job(77, kcount=100, base=2, nmin=4_000_000, nmax=9_999_999, keep=0.03, kmax=1 << 32)
    sieve.load(W.seqs_of(job))
    sieve.run(100, 1_000)
    cnt = sieve.run(100, 1_000)
    assert cnt["hits"] > 10 ** 8
    assert sieve.last_timing()["bsgs_ms_avg"] * 1e6 < 0.2 * cnt["hits"]
