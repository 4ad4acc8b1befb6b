"""The simulation over numbers of strands where its blocks' sizes change (the
fewest strands per block, a last block of one strand, a second wave of full
blocks; one, two and four points per thread of the grid splat), with points outside the grid and on its nodes; bit for bit, against the
CPU oracle."""
import numpy as np
import pytest

from helpers import small_instance

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from hairfb.passes import GridPostSimPass, GridPreSimPass, HairObject, HairSimIntegrationPass, PhysicsGrids, SdfCollider  # noqa: E402
from test_gpu_parity import _ctx, _sim_inputs, oracle  # noqa: E402,F401


@pytest.mark.parametrize("strands,points", [(1, 4), (3, 65), (4, 128), (455, 16), (1825, 17), (2281, 32), (12001, 16), (59001, 16)])
def test_one_step_for_any_number_of_strands_bit_exact(oracle, strands, points):  # noqa: F811
    inst = small_instance(strands=strands, points=points, iterations=2)
    hb = inst.hair
    su = _sim_inputs(inst, 3)
    ctx = _ctx(inst)
    hair = HairObject(hb, inst.cfg.shading_points)
    grids = PhysicsGrids(inst.cfg.grid_dims)
    sdf = SdfCollider(inst.sdf)
    rng = np.random.default_rng(2)
    now = hb.asset.positions.copy()
    now[:, :3] += rng.normal(0, 2e-3, now[:, :3].shape).astype(np.float32) * (now[:, 3:] > 0)
    now[points - 1::7 * points, :3] *= 50.0  # outside the grid
    now[points - 2::5 * points, 0] = 0.0     # one coordinate of many points in one cell of the grid
    hair.positions.copy_(torch.as_tensor(now))
    GridPostSimPass(ctx).cmd_update_grids_after_sim(su, hair, grids)
    GridPreSimPass(ctx).cmd_update_grids_before_sim(su, grids, sdf)
    HairSimIntegrationPass(ctx).cmd_simulate_hair_positions(su, hair, grids, sdf)
    ctx.sync()
    odv = oracle.grid_post_sim(inst.cfg, su, hb.hair_data, hb.asset.positions, now)
    assert np.array_equal(grids.density_velocity.cpu().numpy().ravel(), np.asarray(odv).ravel())
    ogw = oracle.grid_pre_sim(inst.cfg, su, odv, inst.sdf.distances, inst.sdf.dims)
    onew = oracle.sim_integrate(inst.cfg, su, hb.hair_data, hb.asset.positions, now, hb.asset.positions,
                                hb.segment_lengths, odv, ogw, inst.sdf.distances, inst.sdf.dims)
    g = hair.positions.cpu().numpy()
    assert np.array_equal(g.view(np.uint32), onew.view(np.uint32)), f"max abs diff {np.abs(g - onew).max()}"
