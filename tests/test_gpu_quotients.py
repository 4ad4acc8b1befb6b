"""The quotients and roots that the kernels form by short exact forms (hfb_math.cuh
divBy, rootRecip; sim.cu overRoot), against the device's IEEE operations."""
import ctypes

import pytest

from helpers import small_instance

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from hairfb.lib import Context  # noqa: E402


def test_quotients_by_shared_divisors_equal_ieee_division():
    """Every float as the divisor or under the root, 32 numerators each (16 at the ends of
    the forms' ranges and around the one pair of mantissas that the root's form leaves out)."""
    ctx = Context(small_instance(strands=10).cfg.to_c(), 0)
    out = (ctypes.c_uint64 * 4)()
    ctx.call("hfb_check_shared_quotients", out)
    assert list(out)[:3] == [0, 0, 0]
    # the roots' range has 100 exponents; eight of the edges are numerators that the form takes
    assert out[3] > 8 * 100 * (1 << 23) * 0.99
    ctx.close()
