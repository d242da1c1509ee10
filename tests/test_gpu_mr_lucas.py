"""The Miller-Rabin entry points at the edges of their two arithmetics and tests, against the
oracle's is_prime_u64: sizes around 2^49 (double-precision products below), 2^63 and 2^64,
perfect squares (no Lucas parameter exists), and composites of the shapes that pass base 2."""
import numpy as np
import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu


def check(ctx, n):
    n = np.asarray(n, dtype=np.uint64)
    np.testing.assert_array_equal(ctx.mr_verify(n), O.mr_batch(n))


def test_every_small_number(gpu_ctx):
    check(gpu_ctx, np.arange(3_000_000, dtype=np.uint64))


@pytest.mark.parametrize("edge", [1 << 31, 1 << 32, 1 << 40, 1 << 48, 1 << 49, 1 << 50, 1 << 53, 1 << 62, 1 << 63,
                                  (1 << 64) - 200_000])
def test_around_powers_of_two(gpu_ctx, edge):
    check(gpu_ctx, np.arange(edge - 150_000, edge + 150_000, dtype=np.uint64))


@pytest.mark.parametrize("bits", [20, 30, 40, 48, 49, 50, 60, 62, 63, 64])
@pytest.mark.parametrize("mult", [(1, 2), (1, 3), (2, 3), (1, 4), (1, 1)])
def test_semiprimes_that_pass_base_two(gpu_ctx, bits, mult):
    # (a k + 1)(b k + 1): most strong pseudoprimes to base 2 are of this shape; a = b: squares
    a, b = mult
    top = int(((2.0**bits - 1) / (a * b)) ** 0.5)
    rng = np.random.default_rng(bits)
    k = rng.integers(max(2, top // 2), top, size=min(200_000, max(1, top // 2)), dtype=np.uint64)
    n = (np.uint64(a) * k + np.uint64(1)) * (np.uint64(b) * k + np.uint64(1))
    check(gpu_ctx, n[n % np.uint64(2) == 1])


def test_squares_that_pass_base_two(gpu_ctx):
    w = [1093, 3511]  # Wieferich primes: their squares are strong pseudoprimes to base 2
    check(gpu_ctx, [w[0] ** 2, w[1] ** 2, (w[0] * w[1]) ** 2, w[0] ** 2 * 41, 41 ** 2, 1681 - 2, 1669, 4294967291**2])


@pytest.mark.parametrize("count", [1, 31, 32, 33, 255, 257, 4097, 606_209])
def test_batch_sizes(gpu_ctx, count):
    # ragged queues of both size classes in one batch
    rng = np.random.default_rng(count)
    n = rng.integers(0, 2**63, size=count, dtype=np.uint64) * 2 + 1
    n[::3] >>= np.uint64(20)
    check(gpu_ctx, n)


@pytest.mark.parametrize("extra", [0, 1])
def test_both_sides_of_the_line_between_inlined_and_called_tests(gpu_ctx, extra):
    # one pass of every block (8 blocks of 256 per SM), and one candidate more
    import torch
    count = torch.cuda.get_device_properties(0).multi_processor_count * 8 * 256 + extra
    rng = np.random.default_rng(count)
    n = rng.integers(0, 2**63, size=count, dtype=np.uint64) * 2 + 1
    n[::2] >>= np.uint64(16)
    n[::5] = (np.uint64(1) << np.uint64(49)) + np.arange(n[::5].size, dtype=np.uint64) - np.uint64(n[::5].size // 2)
    check(gpu_ctx, n)
