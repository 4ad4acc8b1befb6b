"""The present pass's tone mapping against float64: every byte is the nearest one
wherever the exact value is not within 2e-3 of a rounding boundary (fp32 powf and
its inputs are good to about 1e-4 there)."""
import numpy as np
import pytest

from helpers import small_instance

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from hairfb import uniforms as UN  # noqa: E402
from hairfb.lib import Context  # noqa: E402
from hairfb.passes import PresentPass, RasterBuffers  # noqa: E402


@pytest.mark.parametrize("gamma", [2.2, 1.0, 3.5, 0.4])
@pytest.mark.parametrize("size", [(1, 700), (1023, 5), (257, 513)])
def test_tone_of_every_kind_of_value(gamma, size):
    w, h = size
    inst = small_instance(strands=4, width=w, height=h)
    u = bytearray(UN.pack_render_uniforms(inst.scene, inst.cfg))
    off = UN.OFF["colorMgmt"]
    u[off:off + 12] = np.array([gamma, 0.85, 0.0], np.float32).tobytes()  # gamma, exposure, no dither
    ctx = Context(inst.cfg.to_c(), 0)
    rb = RasterBuffers(ctx, w, h)
    rng = np.random.default_rng(w)
    c = np.concatenate([rng.uniform(0, 1.5, 3 * w * h // 2), 10.0 ** rng.uniform(-9, 1, 3 * w * h)])[:3 * w * h]
    c[:12] = [0.0, -0.0, 1e-40, 1e-30, 1e-12, 1e30, np.inf, np.nan, -0.2, -1e-6, 1.0, 65504.0]
    px = np.ones((w * h, 4), np.float32)
    px[:, :3] = c.reshape(-1, 3)
    ctx.call("hfb_buffer_upload", rb.rb.rasterizerResult + 16, px.ctypes.data, px.nbytes)
    g = PresentPass(ctx).cmd_draw(bytes(u), rb)
    ctx.sync()
    g = g.cpu().numpy()[::-1].reshape(-1, 4)  # the result is read upside down
    with np.errstate(all="ignore"):
        # over black: alpha 1 leaves the colour, except that 0 * inf and the like are NaN, as in the pass
        x = px[:, :3].astype(np.float64) * np.float64(np.float32(0.85))
        v = x * (2.51 * x + 0.03) / (x * (2.43 * x + 0.59) + 0.14)
        v = np.where(np.abs(x) > 1e18, np.nan, v)  # overflows in fp32: inf / inf saturates to 0
        t = 255.0 * np.clip(np.nan_to_num(v, nan=0.0), 0.0, 1.0) ** (1.0 / np.float64(np.float32(gamma)))
    clear = np.abs(t - np.floor(t) - 0.5) > 2e-3
    assert clear.mean() > 0.98
    assert np.array_equal(g[:, :3][clear], np.rint(t)[clear].astype(np.uint8))
    assert (g[:, 3] == 255).all()


@pytest.mark.parametrize("power", [1.0 / 2.2, 1.0, 0.999, 0.5, 1.0 / 3.5, 0.04, 1e-3, 1e-6, 1e-30, 1e-42])
def test_short_form_gives_the_exact_bytes(power):
    """Every float: a byte that the approximate units decide is the exact operations'."""
    import ctypes
    ctx = Context(small_instance(strands=4).cfg.to_c(), 0)
    out = (ctypes.c_uint64 * 2)()
    ctx.call("hfb_check_tone", power, out)
    assert out[0] == 0, f"{out[0]} bytes differ"
    # about 1 in 1,000 is left to the exact way, and what rounds to a tone below 1e-30
    assert out[1] > 0.6 * np.float32(16.0).view(np.uint32)
    ctx.close()
