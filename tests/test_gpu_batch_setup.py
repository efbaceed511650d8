"""The batch's set-up: primes without a search (they divide the base, or leave no
sequence) beside others, range slots without a prime, and its counters.

Every result is compared with the brute-force oracle or with the single-job path:
whole numbers, equal or not.
"""
from contextlib import closing

import numpy as np
import pytest

from rssieve_b200 import workloads as W
from tests.conftest import oracle_job

pytestmark = pytest.mark.gpu


def _terms(f):
    return set(zip(f["seq"].tolist(), f["n"].tolist()))


def _small_job(base, kcount, seed=0):
    return W.small_job(300 + base + kcount + seed, kcount=kcount, base=base, nmin=1000, nmax=9000, keep=0.3,
                       kmax=1 << 24)


def _check(oracle, job, p0, p1, fac, bitmap):
    plist = oracle.primes(p0, p1)
    ofac, _, obm = oracle.brute(oracle_job(oracle, job), plist, ref_skip=True)
    assert _terms(fac) == _terms(ofac)
    assert np.array_equal(bitmap, obm)
    return len(plist)


@pytest.mark.parametrize("kcount", [1, 8, 20, 68])     # a warp per prime; 20 and 68: four primes may share a round
@pytest.mark.parametrize("base", [3, 6, 10, 15])       # odd primes that divide the base at the start of the range
def test_primes_dividing_the_base(rs, oracle, sieve, base, kcount):
    """The range's first records are primes that divide the base: in a batch that
    has used none of its record slots before, and in the single-job path."""
    job = _small_job(base, kcount)
    with closing(rs.Batch(0, max_jobs=2, range_slots=3)) as b:
        j = b.add(W.seqs_of(job), 3, 60_000)
        assert b.run(0)
        n = _check(oracle, job, 3, 60_000, b.factors(j), b.bitmap(j))
        assert b.job_info(j)[1] == n
    sieve.load(W.seqs_of(job))
    assert sieve.run(3, 60_000)["primes"] == n
    _check(oracle, job, 3, 60_000, sieve.factors(), sieve.bitmap())


def test_first_range_slot_without_a_prime(rs, oracle):
    """Range slot 0 holds no prime in the batch's first round, and a number of
    primes that is no multiple of 32 in the next slot; then slot 0 is reused."""
    empty, job, late = _small_job(2, 5), _small_job(3, 20), _small_job(10, 7, seed=1)
    with closing(rs.Batch(0, max_jobs=4, range_slots=4)) as b:
        e = b.add(W.seqs_of(empty), 24, 28)
        j = b.add(W.seqs_of(job), 3, 1_000)
        assert b.run(0)
        assert b.job_info(e)[1:] == (0, True) and len(b.factors(e)) == 0
        _check(oracle, job, 3, 1_000, b.factors(j), b.bitmap(j))
        b.release(e)
        k = b.add(W.seqs_of(late), 3, 5_000)
        assert b.run(0)
        _check(oracle, late, 3, 5_000, b.factors(k), b.bitmap(k))


# one round and several, one to 100 sequences, primes on both sides of 2^51 (where the
# set-up's launches part) and of 2^63, and primes that divide the base
COUNTED = [(1, 2, 3, 40_000), (3, 3, 3, 200_000), (1, 2, (1 << 51) - 100_000, (1 << 51) + 300_000),
           (20, 3, (1 << 51) - 200_000, (1 << 51) + 200_000), (100, 2, (1 << 58) + 1, (1 << 58) + 100_000),
           (5, 10, (1 << 63) - 200_000, (1 << 63) + 200_000)]


def _check_counters(rs, sieve, jobs):
    want = dict.fromkeys(("primes", "skipped", "full", "parity", "targets", "factors", "dups"), 0)
    for job, p0, p1 in jobs:
        sieve.load(W.seqs_of(job))
        cnt = sieve.run(p0, p1)
        assert cnt["skipped"] + cnt["full"] + cnt["parity"] == cnt["primes"]
        for key in want:
            want[key] += cnt[key]
    with closing(rs.Batch(0, max_jobs=len(jobs), range_slots=2 * len(jobs))) as b:
        for job, p0, p1 in jobs:
            assert b.add(W.seqs_of(job), p0, p1) is not None
        assert b.run(0)
        got = b.counters()
    assert {key: got[key] for key in want} == want


def test_counters_equal_the_single_job_path(rs, sieve):
    _check_counters(rs, sieve, [(_small_job(base, kcount), p0, p1) for kcount, base, p0, p1 in COUNTED])


# From 4 * 4 * 8 * 148 = 18944 primes in a round a warp takes four primes, which may
# share their last, partial round of sequences (20 and 68; 100 has none to share):
# about 17800 and 20300 primes, and a round of two jobs that a warp's four may straddle.
@pytest.mark.parametrize("p0,widths", [(10 ** 7, (288_000, 328_000)), (1 << 52, (642_000, 732_000))])
@pytest.mark.parametrize("kcounts", [(20,), (68,), (100,), (68, 20)])
def test_primes_per_warp(rs, sieve, kcounts, p0, widths):
    for w in widths:
        w = w // len(kcounts)
        _check_counters(rs, sieve, [(_small_job(3, k), p0 + i * w, p0 + (i + 1) * w) for i, k in enumerate(kcounts)])


def test_memory_of_a_range_slot(rs):
    """A range slot holds 2^16 primes' records and scratch: 2420 bytes each or less, so
    that a batch of 1150 slots fits 180 GB."""
    import torch
    free = []
    for slots in (4, 36):
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        with closing(rs.Batch(0, max_jobs=2, range_slots=slots)):
            free.append(before - torch.cuda.mem_get_info()[0])
    # (2 MB granules: one or two per buffer, whatever the number of slots)
    assert (free[1] - free[0]) / 32 <= 2420 * 65536 + (1 << 20)
