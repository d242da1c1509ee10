"""Contexts with different tile sizes side by side: the shared memory that a kernel may use is an attribute
of the device's function, not of a context, so one context's smaller tile must not shrink it."""
import pytest

import oracle_lib as O
from test_gpu_sieve import assert_range_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("big,small", [
    (dict(chunk_words=47), dict(chunk_words=1)),
    (dict(block_threads=512, chunk_words=45), dict(block_threads=512, chunk_words=9)),
])
def test_a_smaller_tile_elsewhere_changes_nothing(big, small):
    import voss
    lo, hi = 10**9 - 10**6, 10**9 + 3 * 10**7
    o = O.sieve_range(lo, hi)
    with voss.Context(10**10) as a, voss.Context(10**10) as b:
        a.set_tuning(**big)
        b.set_tuning(**small)
        assert_range_equal(a.sieve_range(lo, hi), o)
        assert_range_equal(b.sieve_range(lo, hi), o)
        with voss.Context(10**10) as c:  # a new context's default tile
            assert_range_equal(c.sieve_range(lo, hi), o)
        assert_range_equal(a.sieve_range(lo, hi), o)
        assert a.primes_range(lo, lo + 10**6).size == O.primes_range(lo, lo + 10**6).size


def test_a_tile_beyond_shared_memory_is_refused():
    import voss
    with voss.Context(10**9) as ctx:
        for words in (55, 57, 61):  # 225 to 250 KB of bitmap: more than a block can have
            with pytest.raises(voss.VossError):
                ctx.set_tuning(chunk_words=words)
        assert ctx.sieve_range(1, 10**7 + 1).prime_count == 664579
