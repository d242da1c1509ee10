"""Saving a context's tuning and setting it again keeps the automatic tile shape.  The shape shows in the number
of kernels of a short launch near 10^12: the chosen small tile comes with a pre-pass, the fixed one
without."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LO, HI = 10**12 - 10**7, 10**12


def kernels(ctx):
    ctx.sieve_range(LO, HI)
    return ctx.last_phase_ms()[3]


def test_the_automatic_shape_survives_a_round_trip():
    import voss
    with voss.Context(10**12) as ctx:
        automatic = kernels(ctx)
        ctx.set_tuning(chunk_words=49)
        assert kernels(ctx) != automatic  # what this test tells the two by
        t0 = ctx.set_tuning()
        ctx.set_tuning(**t0)
        assert kernels(ctx) == automatic
        ctx.set_tuning(**{**t0, "mr_route": 0xFFFFFFFF})  # another field changed alone
        assert kernels(ctx) == automatic
        ctx.set_tuning(**{**t0, "coop_div": 64})  # one of the shape's own
        assert kernels(ctx) != automatic
        ctx.set_tuning(**t0)
        assert kernels(ctx) == automatic and ctx.tuning() == t0


def test_the_autotuner_times_the_automatic_shape(tmp_path, monkeypatch):
    import voss
    from voss import autotune
    monkeypatch.setenv("VOSS_TUNE_CACHE", str(tmp_path / "tune.json"))
    with voss.Context(10**12) as ctx:
        automatic = kernels(ctx)
        seen = []
        for cand in autotune.CANDIDATES:
            ctx.set_tuning(**cand)
            seen.append(kernels(ctx))
        assert seen[0] == automatic
        lo = np.array([LO], dtype=np.uint64)
        autotune.tune_intervals(ctx, lo, lo + np.uint64(10**7), candidates=autotune.CANDIDATES[:1])
        assert kernels(ctx) == automatic


def test_a_tie_goes_to_the_automatic_shape(tmp_path, monkeypatch):
    import voss
    from voss import autotune
    monkeypatch.setenv("VOSS_TUNE_CACHE", str(tmp_path / "tune.json"))
    with voss.Context(10**12) as ctx:
        automatic = kernels(ctx)
        times = iter([2.490, 2.488, 2.486])  # each a little faster than the one before
        monkeypatch.setattr(ctx, "last_kernel_ms", lambda: (0.0, next(times)))
        lo = np.array([LO], dtype=np.uint64)
        autotune.tune_intervals(ctx, lo, lo + np.uint64(10**6), reps=1, candidates=autotune.CANDIDATES[:3])
        assert kernels(ctx) == automatic
