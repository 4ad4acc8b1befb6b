"""GTAO at the reference's scale (positions from a shared-memory tile) at sizes
with partial blocks, with numbers of directions that its threads share unevenly or not
at all, and with radii whose samples leave the tile's halo, against
the CPU oracle; the AO test's tolerance (an ulp of a transcendental can move a
sample by a pixel)."""
import numpy as np
import pytest

from helpers import small_instance

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from hairfb import uniforms as UN  # noqa: E402
from hairfb.lib import Context  # noqa: E402
from hairfb.passes import AoPass, _ub  # noqa: E402
from test_gpu_parity import oracle  # noqa: E402,F401


@pytest.mark.parametrize("size", [(64, 16), (131, 37), (1, 50), (322, 241)])
@pytest.mark.parametrize("radius,scale,directions", [(2.0, 0.5, 12), (900.0, 0.5, 5), (2.0, 1.0, 12), (2.0, 0.5, 3),
                                                     (2.0, 0.5, 32), (2.0, 0.5, 33)])
def test_gtao_tile(oracle, size, radius, scale, directions):  # noqa: F811
    w, h = size
    inst = small_instance(strands=4, width=w, height=h)
    u = bytearray(UN.pack_render_uniforms(inst.scene, inst.cfg))
    u[UN.OFF["ao"]:UN.OFF["ao"] + 4] = np.float32(radius).tobytes()
    u[UN.OFF["ao"] + 16:UN.OFF["ao"] + 20] = np.uint32(directions).tobytes()
    rng = np.random.default_rng(w)
    depth = (0.9935 + 0.002 * rng.random(w * h)).astype(np.float32)
    depth[rng.random(w * h) < 0.2] = 1.0
    if w > 200:
        depth.reshape(h, w)[:, 150:] = 1.0  # blocks of sky alone
    normals = rng.random((w * h, 2)).astype(np.float16).astype(np.float32)
    ctx = Context(inst.cfg.to_c(), 0)
    d, n = torch.as_tensor(depth).cuda(), torch.as_tensor(normals).cuda()
    torch.cuda.synchronize()
    g = AoPass(ctx).cmd_calc_ao(bytes(u), d, n, w, h, scale)
    ctx.sync()
    g = g.cpu().numpy()
    o = oracle.gtao(bytes(u), depth, normals, scale).reshape(g.shape)
    err = np.abs(g - o)
    both = np.isnan(g) & np.isnan(o)
    bad = (~both & ~(err <= 4e-3)).sum()
    assert bad <= max(2, 0.005 * g.size), f"{bad} of {g.size} texels differ"
    assert (g > 0).mean() > 0.1


@pytest.mark.parametrize("size", [(64, 16), (131, 37), (1, 50), (2, 3), (17, 33), (322, 241)])
@pytest.mark.parametrize("radius,directions,steps", [(2.0, 12, 8), (900.0, 5, 8), (2.0, 3, 8), (2.0, 32, 3), (2.0, 1, 16),
                                                     (0.0, 12, 1), (2.0, 0, 8)])
def test_tile_kernel_equals_the_kernel_for_any_scale(size, radius, directions, steps):
    """Every texel, the borders of blocks and of the viewport among them: the shared tile changes no bit."""
    w, h = size
    inst = small_instance(strands=4, width=w, height=h)
    u = bytearray(UN.pack_render_uniforms(inst.scene, inst.cfg))
    u[UN.OFF["ao"]:UN.OFF["ao"] + 4] = np.float32(radius).tobytes()
    u[UN.OFF["ao"] + 16:UN.OFF["ao"] + 24] = np.array([directions, steps], np.uint32).tobytes()
    rng = np.random.default_rng(w)
    depth = (0.9935 + 0.002 * rng.random(w * h)).astype(np.float32)
    depth[rng.random(w * h) < 0.2] = 1.0
    if w > 200:
        depth.reshape(h, w)[:, 150:300] = 1.0  # blocks of sky alone, and some past them
    normals = rng.random((w * h, 2)).astype(np.float16).astype(np.float32)
    ctx = Context(inst.cfg.to_c(), 0)
    d, n = torch.as_tensor(depth).cuda(), torch.as_tensor(normals).cuda()
    torch.cuda.synchronize()
    g = AoPass(ctx).cmd_calc_ao(bytes(u), d, n, w, h, 0.5)
    want = torch.empty_like(g)
    ctx.call("hfb_check_gtao", _ub(bytes(u)), d.data_ptr(), n.data_ptr(), 0.5, want.data_ptr())
    ctx.sync()
    assert np.array_equal(g.cpu().numpy().view(np.uint32), want.cpu().numpy().view(np.uint32))
