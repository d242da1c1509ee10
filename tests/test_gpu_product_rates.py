"""The measured product rates that the primality roofline is set against: they repeat, and the product in
double precision is the fastest of the three."""
import pytest

pytestmark = pytest.mark.gpu


def test_double_products_are_the_fastest(gpu_ctx):
    full, small = gpu_ctx.probe_mulmod()
    dbl = [gpu_ctx.probe_mulmod_double() for _ in range(3)]
    assert min(dbl) > max(full, small) and max(dbl) < 1.2 * min(dbl) < 1e14
