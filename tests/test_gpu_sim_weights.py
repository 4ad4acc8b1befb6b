"""The integration's two ways to hold a strand's constants: a fixed root and
movable points of weight 1 (what assets have), and any other weights, for
strands from the shortest to the longest; one step, bit for bit, against the CPU oracle."""
import numpy as np
import pytest

from helpers import small_instance

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from hairfb import hair_object as HO  # noqa: E402
from hairfb.passes import GridPostSimPass, GridPreSimPass, HairObject, HairSimIntegrationPass, PhysicsGrids, SdfCollider  # noqa: E402
from test_gpu_parity import _ctx, _sim_inputs, oracle  # noqa: E402,F401


@pytest.mark.parametrize("points", [4, 5, 6, 16, 33, 128])
@pytest.mark.parametrize("weights", ["fixed root", "one strand", "all points", "free root"])
def test_one_step_for_any_weights_bit_exact(oracle, points, weights):  # noqa: F811
    inst = small_instance(strands=301, points=points, iterations=3)
    pos = inst.hair.asset.positions.reshape(301, points, 4)
    if weights == "one strand":
        pos[150, -1, 3] = 0.25
    elif weights == "all points":
        pos[:, :, 3] = np.linspace(0.0, 1.0, points, dtype=np.float32)
    elif weights == "free root":
        pos[:, 0, 3] = 1.0
    inst.hair = hb = HO.build_hair_buffers(inst.hair.asset)
    su = _sim_inputs(inst, 3)
    ctx = _ctx(inst)
    hair = HairObject(hb, inst.cfg.shading_points)
    grids = PhysicsGrids(inst.cfg.grid_dims)
    sdf = SdfCollider(inst.sdf)
    rng = np.random.default_rng(2)
    now = hb.asset.positions.copy()
    now[:, :3] += rng.normal(0, 2e-3, now[:, :3].shape).astype(np.float32) * (now[:, 3:] > 0)
    hair.positions.copy_(torch.as_tensor(now))
    GridPostSimPass(ctx).cmd_update_grids_after_sim(su, hair, grids)
    GridPreSimPass(ctx).cmd_update_grids_before_sim(su, grids, sdf)
    HairSimIntegrationPass(ctx).cmd_simulate_hair_positions(su, hair, grids, sdf)
    ctx.sync()
    odv = oracle.grid_post_sim(inst.cfg, su, hb.hair_data, hb.asset.positions, now)
    ogw = oracle.grid_pre_sim(inst.cfg, su, odv, inst.sdf.distances, inst.sdf.dims)
    onew = oracle.sim_integrate(inst.cfg, su, hb.hair_data, hb.asset.positions, now, hb.asset.positions,
                                hb.segment_lengths, odv, ogw, inst.sdf.distances, inst.sdf.dims)
    g = hair.positions.cpu().numpy()
    assert np.array_equal(g.view(np.uint32), onew.view(np.uint32)), f"max abs diff {np.abs(g - onew).max()}"


@pytest.mark.parametrize("points", [4, 16, 65])
def test_a_root_of_weight_minus_zero_keeps_it(oracle, points):  # noqa: F811
    """A root of weight -0 is fixed too, and its weight comes back as it went in, as the
    oracle leaves it."""
    inst = small_instance(strands=301, points=points, iterations=2)
    pos = inst.hair.asset.positions.reshape(301, points, 4)
    pos[::3, 0, 3] = -0.0
    inst.hair = hb = HO.build_hair_buffers(inst.hair.asset)
    su = _sim_inputs(inst, 3)
    ctx = _ctx(inst)
    hair = HairObject(hb, inst.cfg.shading_points)
    grids = PhysicsGrids(inst.cfg.grid_dims)
    sdf = SdfCollider(inst.sdf)
    GridPostSimPass(ctx).cmd_update_grids_after_sim(su, hair, grids)
    GridPreSimPass(ctx).cmd_update_grids_before_sim(su, grids, sdf)
    HairSimIntegrationPass(ctx).cmd_simulate_hair_positions(su, hair, grids, sdf)
    ctx.sync()
    p0 = hb.asset.positions
    odv = oracle.grid_post_sim(inst.cfg, su, hb.hair_data, p0, p0)
    ogw = oracle.grid_pre_sim(inst.cfg, su, odv, inst.sdf.distances, inst.sdf.dims)
    onew = oracle.sim_integrate(inst.cfg, su, hb.hair_data, p0, p0, p0, hb.segment_lengths, odv, ogw,
                                inst.sdf.distances, inst.sdf.dims)
    g = hair.positions.cpu().numpy()
    assert (g.reshape(301, points, 4)[::3, 0, 3].view(np.uint32) == 0x80000000).all()
    assert np.array_equal(g.view(np.uint32), onew.view(np.uint32))
