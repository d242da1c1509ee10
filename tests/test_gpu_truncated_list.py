"""Gap lists with less room than the range has gaps: the records are those of the tiles that finished first, which
in a long range crowd into a few of the sort's parts (more than a part's list holds).  They come back
sorted, distinct, and each one a gap of the range."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# about a hundred tiles, all at once; and two hundred times that, of which the first wave fills the list
@pytest.mark.parametrize("lo,length,min_gap", [(10**9, 6 * 10**8, 100), (10**12, 6 * 10**8, 100),
                                               (10**12, 2 * 10**11, 200)])
@pytest.mark.parametrize("cap", [1, 2047, 2048, 2049, 4097, 10_000, 16_384, 16_385])
def test_a_list_cut_short(gpu_ctx, lo, length, min_gap, cap):
    from voss import _native as N
    from voss.api import LARGE_DTYPE
    hi = lo + length
    full = gpu_ctx.gaps_at_least(lo, hi, min_gap)
    out = np.zeros(cap, dtype=LARGE_DTYPE)
    n = ctypes.c_uint64()
    N.check(gpu_ctx.lib.voss_gaps_at_least(gpu_ctx.handle, lo, hi, min_gap,
                                           out.ctypes.data_as(ctypes.POINTER(N.LargeGap)), cap, ctypes.byref(n)))
    assert n.value == full.size > cap
    assert np.all(np.diff(out["position"].astype(np.int64)) > 0)
    at = np.searchsorted(full["position"], out["position"])
    np.testing.assert_array_equal(out, full[at])
