"""The end of the primality kernel, where the candidates left in the warps' queues are merged over the
block: batches of which fewer than 32 candidates per warp reach the Lucas test, so that every one
of them goes through that merge.  Each verdict has to be written, whatever was in the output."""
import numpy as np
import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("every", [1, 9, 40])  # one candidate in `every` is prime
@pytest.mark.parametrize("count", [1, 31, 33, 250, 8 * 31, 8 * 32, 5000])
@pytest.mark.parametrize("lo", [10**12, 10**17])  # both arithmetics
def test_every_leftover_gets_its_verdict(gpu_ctx_big, count, every, lo):
    import torch
    import voss.api
    primes = gpu_ctx_big.primes_range(lo, lo + 60 * count + 10_000)
    n = np.full(count, np.uint64(41 * 43), dtype=np.uint64)
    n[::every] = primes[: n[::every].size]
    d_n = torch.from_numpy(n.view(np.int64)).cuda()
    want = O.mr_batch(n)
    for fill in (0, 1, 0xA5):
        d_ok = torch.full((count,), fill, dtype=torch.uint8, device="cuda")
        voss.api.mr_verify_noalloc(d_n.data_ptr(), count, d_ok.data_ptr(), torch.cuda.current_stream().cuda_stream)
        np.testing.assert_array_equal(d_ok.cpu().numpy(), want)
