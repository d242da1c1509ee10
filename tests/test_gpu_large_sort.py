"""The large-gap list in ascending position order at the edges of its two sorts: as many parts as
SMs, one record per part and fewer, the longest list of the one-launch sort and the next one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def primes():
    flags = np.ones(2_000_000, dtype=bool)
    flags[:2] = False
    for q in range(2, 1415):
        if flags[q]:
            flags[q * q::q] = False
    return np.nonzero(flags)[0]


@pytest.mark.parametrize("first", [10, 100_000])
@pytest.mark.parametrize("count", [1, 2, 147, 148, 149, 1024, 2049, 16_383, 16_384, 16_385])
def test_the_gaps_of_a_window_in_order(gpu_ctx, primes, first, count):
    gap = np.diff(primes)
    upper = first + 1 + np.nonzero(gap[first:] >= 4)[0][:count]  # indices of the gaps' upper primes
    assert upper.size == count
    g = gpu_ctx.gaps_at_least(int(primes[first]), int(primes[upper[-1]]) + 1, 4)
    np.testing.assert_array_equal(g["position"], primes[upper])
    np.testing.assert_array_equal(g["gap"], gap[upper - 1])


def test_a_window_without_such_gaps(gpu_ctx):
    assert len(gpu_ctx.gaps_at_least(10**6, 10**6 + 1000, 500)) == 0
