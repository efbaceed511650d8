"""Giant phases longer than the start tables' 1024 chunks of one segment each: a
segment then ends inside the chunks.

Results are compared with the brute-force oracle or with planted factors (whole
numbers, equal or not), and the device time of such a search is held against that of
a search whose chunks are whole.
"""
import numpy as np
import pytest

from rssieve_b200 import workloads as W
from tests.conftest import oracle_job
from tests.test_gpu_search import _planted

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kcount,p0", [(1, 20_000), (3, 60_000), (40, 200_000)])
def test_cut_chunks_match_brute_force(sieve, oracle, kcount, p0):
    """Small p: segments of one or a few steps, chunks of up to 6*10^6/(512*1024) = 12."""
    job = W.small_job(400 + kcount, kcount=kcount, base=2, nmin=1001, nmax=6_001_000 // (1 if kcount < 10 else 4),
                      keep=0.05, kmax=1 << 24)
    sieve.set_baby_steps(1024)
    try:
        sieve.load(W.seqs_of(job))
        cnt = sieve.run(p0, p0 + 1_500)
        fac, bm = sieve.factors(), sieve.bitmap()
    finally:
        sieve.set_baby_steps(0)
    plist = oracle.primes(p0, p0 + 1_500)
    ofac, odups, obm = oracle.brute(oracle_job(oracle, job), plist, ref_skip=True)
    assert cnt["primes"] == len(plist)
    assert oracle.term_set(fac) == oracle.term_set(ofac)
    assert np.array_equal(bm, obm)
    assert cnt["dups"] == odups


@pytest.mark.parametrize("p0", [(1 << 47) + 1, (1 << 57) + 1, (1 << 63) + 1])
def test_cut_chunks_in_every_step_kind(sieve, oracle, p0):
    _planted(sieve, oracle, 2, 1, 1, (1 << 32) - 1, p0, p0 + 1_000, 7, q=1024)
    _planted(sieve, oracle, 3, 6, 1, 400_000_000, p0, p0 + 1_000, 8, q=1024)


def test_long_giant_phase_costs_its_steps(sieve):
    """One sequence over 2^32 - 2 exponents near 2^47.  A step costs the same with 512
    or 1024 baby steps as with up to 16384, apart from the baby steps again per
    segment (16 per 62 or more giant steps of a thread) and from the segment's fixed
    work; a bound of four times leaves room for both.  (A queue of filter passes that
    overflows costs 16 products per step instead of one.)"""
    nmax = (1 << 32) - 2
    bm = np.zeros((1, (nmax + 31) // 32), dtype=np.uint32)
    bm[0, 0] = 1
    job = W.seqs_of(W.job_dict(2, [1_234_567], [1], 1, nmax, bm))
    per_step = {}
    try:
        for q in (1024, 16384):
            sieve.set_baby_steps(q)
            sieve.load(job)
            for _ in range(2):
                cnt = sieve.run((1 << 47) + 1, (1 << 47) + 200_001)
            per_step[q] = sieve.last_timing()["bsgs_ms_avg"] / (cnt["baby"] + cnt["giant"])
    finally:
        sieve.set_baby_steps(0)
    assert per_step[1024] < 4 * per_step[16384]
