"""Ranges sieved on several streams of the caller's in turn: the launches share the context's device memory, so each
has to wait for the one before, and a fetch or another call for the last."""
import pytest

import oracle_lib as O
from test_gpu_sieve import assert_range_equal

pytestmark = pytest.mark.gpu


def test_launches_on_several_streams_follow_each_other():
    import torch
    import voss
    ranges = [(1, 10**8), (10**9, 10**9 + 10**6), (10**8, 4 * 10**8), (5, 10**4), (10**9 - 10**7, 10**9)]
    want = [O.sieve_range(lo, hi) for lo, hi in ranges]
    streams = [torch.cuda.Stream() for _ in range(3)]
    with voss.Context(2 * 10**9) as ctx:
        for last, w in enumerate(want):
            for k in range(last + 1):
                ctx.sieve_range_device(*ranges[k], stream=streams[k % 3].cuda_stream)
            assert_range_equal(ctx.fetch_range(), w)
            ctx.sieve_range_device(*ranges[0], stream=streams[last % 3].cuda_stream)
            assert_range_equal(ctx.sieve_range(*ranges[last]), w)
