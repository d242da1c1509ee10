"""A call that fails for want of device memory says so and leaves the context, and every other, usable."""
import ctypes

import numpy as np
import pytest

import oracle_lib as O
from test_gpu_sieve import assert_range_equal

pytestmark = pytest.mark.gpu


def test_calls_after_a_failed_allocation():
    import voss
    from voss import _native as N
    n = 25_000_000  # results of 8 KB each: more than the device holds, so nothing is launched or written
    lo = np.full(n, 100, dtype=np.uint64)
    small = np.zeros(1, dtype=voss.api.INTERVAL_DTYPE)
    o = O.sieve_range(1, 10**6)
    with voss.Context(10**9) as ctx, voss.Context(10**9) as other:
        u64 = ctypes.POINTER(ctypes.c_uint64)
        for _ in range(2):
            rc = ctx.lib.voss_sieve_intervals(ctx.handle, lo.ctypes.data_as(u64), lo.ctypes.data_as(u64), n,
                                              small.ctypes.data_as(ctypes.POINTER(N.IntervalStats)))
            assert rc == -3 and b"cudaMalloc" in ctx.lib.voss_last_error()  # VOSS_ERR_NOMEM
            assert_range_equal(other.sieve_range(1, 10**6), o)
            assert_range_equal(ctx.sieve_range(1, 10**6), o)
            assert ctx.mr_verify(np.array([97, 91], dtype=np.uint64)).tolist() == [1, 0]
