"""The prime generator at the edges of its sieve blocks.

A window of `nodd` odd numbers is sieved in blocks of 8192 to 131072 odd numbers,
the smallest that two blocks per SM need: the windows below end one number before,
at and after a block, and at the widths where the block size changes (148 SMs), at
p where the base-2 test is in FP64, across 2^51, and in integers.  Whole numbers,
equal to the oracle's or not.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BLOCK = 2 * 8192                    # numbers of the smallest block
STEP = BLOCK * 2 * 148              # the width from which blocks are doubled


@pytest.mark.parametrize("lo", [3, (1 << 45) + 1, (1 << 51) - 20_000, (1 << 58) + 2])
@pytest.mark.parametrize("width", [1, 2, 63, 64, 65, BLOCK - 1, BLOCK, BLOCK + 1, 3 * BLOCK + 7])
def test_windows_around_a_block(sieve, oracle, lo, width):
    assert np.array_equal(np.sort(sieve.primes(lo, lo + width)), oracle.primes(lo, lo + width))


@pytest.mark.parametrize("width", [STEP - 2, STEP, STEP + 2, 2 * STEP + 2])
def test_windows_where_the_block_size_changes(sieve, oracle, width):
    lo = (1 << 50) + 1
    assert np.array_equal(np.sort(sieve.primes(lo, lo + width)), oracle.primes(lo, lo + width))
