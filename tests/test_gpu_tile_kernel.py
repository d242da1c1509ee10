"""The tile kernel at the sizes where its parts can go wrong, against the CPU oracle (exact): the
last words of a tile, tiles of a few words, tiles without a far gap (the longest gap is then
searched again), primes taken as small, by progressions and by class in every proportion."""
import numpy as np
import pytest

import oracle_lib as O
from test_gpu_sieve import assert_range_equal

pytestmark = pytest.mark.gpu

WORD = 120  # integers per 32-bit bitmap word


# words of the range: around one residue-class period (1001), a warp, the full tile (50176) and two
@pytest.mark.parametrize("words", [1, 2, 31, 33, 1000, 1001, 1002, 50175, 50176, 50177, 100353])
@pytest.mark.parametrize("lo", [120 * 10**4, 10**12 - 77])
def test_tile_lengths(gpu_ctx, lo, words):
    hi = lo + WORD * words - 13
    assert_range_equal(gpu_ctx.sieve_range(lo, hi), O.sieve_range(lo, hi))


@pytest.mark.parametrize("lo,ln", [(10**6, 40), (10**6, 400), (10**9 + 1, 1500), (10**12, 90), (10**12, 5000)])
def test_short_tiles_find_their_longest_gap(gpu_ctx, lo, ln):
    for k in range(12):
        a = lo + 997 * k
        assert_range_equal(gpu_ctx.sieve_range(a, a + ln), O.sieve_range(a, a + ln))


@pytest.mark.parametrize("tuning", [
    dict(coop_div=1),                             # more small primes than records
    dict(coop_div=100000, walk_sixteenths=1),     # none, and the classes from a sixteenth of a tile on
    dict(walk_sixteenths=128),                    # no prime by class
    dict(mult_factor=1, walk_sixteenths=16),      # the classes end at the tile length
    dict(mult_factor=64),
    dict(medium_mode=1),
    dict(block_threads=512, chunk_words=9),
    dict(block_threads=1024, chunk_words=1),
])
def test_tunings(gpu_ctx, tuning):
    lo, hi = 10**13 - 3 * 10**6, 10**13 + 5 * 10**6 + 1
    o = O.sieve_range(lo, hi)
    try:
        gpu_ctx.set_tuning(**tuning)
        assert_range_equal(gpu_ctx.sieve_range(lo, hi), o)
    finally:
        gpu_ctx.set_tuning()


@pytest.mark.parametrize("min_gap", [3, 4, 6, 30, 100, 130])
def test_gap_lists_down_to_the_smallest_gaps(gpu_ctx, min_gap):
    lo, hi = 10**10, 10**10 + 2 * 10**6
    p = O.primes_range(lo, hi)
    want = [(int(b), int(b - a)) for a, b in zip(p[:-1], p[1:]) if b - a >= min_gap]
    got = gpu_ctx.gaps_at_least(lo, hi, min_gap)
    assert [(int(a), int(g)) for a, g in zip(got["position"], got["gap"])] == want


def test_a_range_longer_than_a_prepass_window_equals_its_parts():
    """The large-prime bitmap of a long range is pre-sieved in pieces; ranges of one piece do not."""
    import voss
    lo, cuts = 10**14 + 11, (0, 1_300_000_017, 2_500_000_000, 3_300_000_001)  # 1.5e9 integers per window
    with voss.Context(10**14 + 10**10) as ctx:
        whole = ctx.sieve_range(lo, lo + cuts[-1])
        parts = [ctx.sieve_range(lo + a, lo + b) for a, b in zip(cuts[:-1], cuts[1:])]
        assert_range_equal(voss.merge_stats(parts), whole)


@pytest.mark.parametrize("words", [1, 1024, 1025, 50175, 50176, 50177, 100353])
def test_tile_lengths_in_the_large_tile(gpu_ctx, words):
    """Small launches choose small tiles; the same lengths in the tile that long runs use."""
    lo = 10**12 - 77
    hi = lo + WORD * words - 13
    try:
        gpu_ctx.set_tuning(chunk_words=49)
        assert_range_equal(gpu_ctx.sieve_range(lo, hi), O.sieve_range(lo, hi))
    finally:
        gpu_ctx.set_tuning()


@pytest.mark.parametrize("n,ln", [(1, 10**5), (3, 10**6), (147, 3 * 10**5), (149, 3 * 10**5), (600, 10**5), (900, 10**4)])
def test_chosen_tile_shapes_equal_the_fixed_one(gpu_ctx, n, ln):
    rng = np.random.default_rng(n)
    lo = (10 ** rng.uniform(6, 13, n)).astype(np.uint64)
    hi = lo + rng.integers(0, 2 * ln, n).astype(np.uint64)
    chosen = gpu_ctx.sieve_intervals(lo, hi)
    try:
        gpu_ctx.set_tuning(chunk_words=49)
        fixed = gpu_ctx.sieve_intervals(lo, hi)
    finally:
        gpu_ctx.set_tuning()
    for f in chosen.dtype.names:
        np.testing.assert_array_equal(chosen[f], fixed[f], err_msg=f)


@pytest.mark.parametrize("ln", [10**5, 3 * 10**6, 11 * 10**6, 4 * 10**7, 5 * 10**7, 2 * 10**8])
def test_gap_lists_of_every_sort_in_order(gpu_ctx, ln):
    """Lists around 4096 records (copied with the state), 16384 (ranked) and beyond (radix sorted)."""
    lo = 10**12
    got = gpu_ctx.gaps_at_least(lo, lo + ln, 150)
    p = O.primes_range(lo, lo + ln)
    d = np.diff(p)
    np.testing.assert_array_equal(got["position"], p[1:][d >= 150])
    np.testing.assert_array_equal(got["gap"], d[d >= 150])
    assert gpu_ctx.gaps_at_least(lo, lo + ln, 150, cap=max(1, got.size)).size == got.size


@pytest.mark.parametrize("lo,hi", [(1, 10**6), (10**4, 10**7), (9 * 10**6, 15 * 10**6), (99_000_000, 101_000_000)])
def test_low_ranges_under_a_context_for_high_ones(gpu_ctx_big, lo, hi):
    """The base primes of a context for 10^18 fill the tiles below 10^9; only those that struck
    themselves out are restored."""
    assert_range_equal(gpu_ctx_big.sieve_range(lo, hi), O.sieve_range(lo, hi))


@pytest.mark.parametrize("lo", [26 * 10**11, 8 * 10**12, 16 * 10**12, 17 * 10**12])
def test_long_ranges_around_the_prepass_rule(lo):
    """Ranges whose root lies just above the pre-pass's bound sieve those primes in the tiles; the
    same range through the pre-pass."""
    import voss
    with voss.Context(2 * 10**13) as ctx:
        r = ctx.sieve_range(lo, lo + 3 * 10**9)
        ctx.set_tuning(mult_factor=8)  # a fixed shape: its pre-pass bound is 8 tile lengths
        assert_range_equal(ctx.sieve_range(lo, lo + 3 * 10**9), r)
