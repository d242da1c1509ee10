"""The first calls of a process: the library's constant tables and a new context's tables have to be complete
for kernels on any stream, and calls without a context may overlap on several streams and threads.
Each check runs in a process of its own, whose first work on the library it is."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PREAMBLE = """
import sys, threading
sys.path[:0] = [%r, %r]
import numpy as np, torch
import voss, voss.api
import oracle_lib as O
rng = np.random.default_rng(5)
""" % (os.path.join(ROOT, "voss-prime-gaps_v1_b200"), os.path.join(ROOT, "tests"))

NOALLOC = """
n = [(rng.integers(0, 2**(63 - 16 * k), size=100_003 + k, dtype=np.uint64) * 2 + 1) for k in range(4)]
d = [torch.from_numpy(x.view(np.int64)).cuda() for x in n]
ok = [torch.full((x.size,), 7, dtype=torch.uint8, device="cuda") for x in n]
streams = [torch.cuda.Stream() for _ in n]
torch.cuda.synchronize()
go = threading.Barrier(len(n))
def call(k):
    go.wait()
    for _ in range(3):
        voss.api.mr_verify_noalloc(d[k].data_ptr(), n[k].size, ok[k].data_ptr(), streams[k].cuda_stream)
threads = [threading.Thread(target=call, args=(k,)) for k in range(len(n))]
[t.start() for t in threads]
[t.join() for t in threads]
torch.cuda.synchronize()
for x, o in zip(n, ok):
    assert np.array_equal(o.cpu().numpy(), O.mr_batch(x))
"""

CONTEXT = """
with voss.Context(10**16) as ctx:
    r = ctx.sieve_range(10**16 - 2 * 10**6, 10**16)
o = O.sieve_range(10**16 - 2 * 10**6, 10**16)
assert r.prime_count == o.prime_count and np.array_equal(r.gap_hist, o.gap_hist)
"""

DIGESTS = """
import hashlib
with voss.Context(10**9) as ctx:
    msgs = [b"VOSS|%d" % k for k in range(500)]
    got = ctx.sha256_batch(msgs)
assert [bytes(g) for g in got] == [hashlib.sha256(m).digest() for m in msgs]
"""


@pytest.mark.parametrize("body", [NOALLOC, CONTEXT, DIGESTS], ids=["noalloc", "context", "digests"])
def test_the_first_call_of_a_process(body):
    r = subprocess.run([sys.executable, "-c", PREAMBLE + body], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
