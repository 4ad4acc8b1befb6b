"""The shading's shadow filter at its default radius, where the gathers share a
window of texels, and at others; lobes with and without weight; against the
CPU oracle with the shading tests' tolerance."""
import numpy as np
import pytest

from helpers import frame_of, small_instance

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from hairfb.passes import HairObject, HairShadingPass  # noqa: E402
from test_gpu_parity import _ctx, oracle  # noqa: E402,F401


@pytest.mark.parametrize("size", [1, 5, 8, 100, 1000, 1024])
@pytest.mark.parametrize("radius,weight_tt", [(3, 0.0), (3, 0.7), (2, 0.0)])
def test_shadow_windows(oracle, size, radius, weight_tt):  # noqa: F811
    """Maps smaller than the window (clamped texels), odd sizes (the gathers'
    coordinates round), and the sizes in use."""
    inst = small_instance(strands=200, shading_points=9)
    inst.scene.pcf_radius = radius
    inst.scene.material.weight_tt = weight_tt
    fr = frame_of(inst)
    hb = inst.hair
    ctx = _ctx(inst)
    hair = HairObject(hb, inst.cfg.shading_points)
    depth = np.full(inst.width * inst.height, 0.9995, np.float32)
    sm = np.random.default_rng(4).uniform(0.2, 0.4, size * size).astype(np.float32)
    HairShadingPass(ctx).cmd_compute_shading_points(fr.uniforms, hair, torch.as_tensor(depth).cuda(),
                                                    shadow_map=torch.as_tensor(sm).cuda(), shadow_size=size)
    ctx.sync()
    o = oracle.shading(inst.cfg, fr.uniforms, hb.hair_data, hb.asset.positions, hb.tangents, depth,
                       hb.asset.strands, shadow_map=sm, shadow_size=size)
    err = np.abs(hair.shading.cpu().numpy() - o)
    assert (err <= 1e-5 + 1e-5 * np.abs(o)).all(), f"max shading error {err.max():.3g}"
