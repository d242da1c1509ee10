"""Short intervals by Miller-Rabin in segments of 4096 candidates: lengths around one and several
segments, empty ones and single long ones, bit for bit against the sieve of the same intervals."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SEG = 4096 * 30 // 8  # integers per segment


@pytest.mark.parametrize("lens", [
    [0, 1, 5, 7], [SEG - 30, SEG, SEG + 1, SEG + 30], [2 * SEG - 1, 3 * SEG + 13], [700_000], [10] * 700,
])
def test_segments_equal_the_sieve(gpu_ctx_big, lens):
    rng = np.random.default_rng(len(lens))
    ln = np.asarray(lens, dtype=np.uint64)
    lo = (10**18 - 10**12 + rng.integers(0, 10**11, ln.size)).astype(np.uint64)
    t0 = gpu_ctx_big.tuning()
    routed = gpu_ctx_big.sieve_intervals(lo, lo + ln)
    if ln.min():  # candidates, Miller-Rabin, segments, statistics (an empty interval is not routed: the sieve's kernels run)
        assert gpu_ctx_big.last_phase_ms()[3] == 4
    try:
        gpu_ctx_big.set_tuning(**{**t0, "mr_route": 0xFFFFFFFF})
        k = min(ln.size, 12)  # the sieve walks 50 million base primes per interval up there
        sieved = gpu_ctx_big.sieve_intervals(lo[:k], lo[:k] + ln[:k])
    finally:
        gpu_ctx_big.set_tuning(**t0)
    for f in routed.dtype.names:
        np.testing.assert_array_equal(routed[f][:k], sieved[f], err_msg=f)
