"""The kernels that list a segment's pixels row by row from conservative spans
(raster.cu spanLines): at sizes where the lists, the rounds and the split
tiles' decisions have their edges, against the CPU oracle."""
import numpy as np
import pytest

from helpers import frame_of, small_instance

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from hairfb import hair_object as HO  # noqa: E402
from hairfb.passes import HairObject, HwHairPass, RasterBuffers  # noqa: E402
from test_gpu_parity import _compare_tiles, _ctx, _fine_vs_oracle, _raster_gpu, oracle  # noqa: E402,F401


@pytest.mark.parametrize("tile,slices", [(8, 4), (8, 8), (16, 4), (16, 8), (32, 4), (32, 8)])
@pytest.mark.parametrize("fiber,strands", [(2e-2, 400), (2e-3, 1500), (2e-5, 1500)])
def test_fine_pass_segments_of_every_width(oracle, tile, slices, fiber, strands):  # noqa: F811
    """Segments that cover whole tiles (a round's list fills up before its
    segments do), ordinary ones, and ones thinner than a pixel (most rows'
    spans are empty); a ragged viewport, so edge tiles are partial."""
    inst = small_instance(strands=strands, width=301, height=217, tile_size=tile, slices=slices, fiber_radius=fiber,
                          avg_segments_per_tile=2048)
    cnt, g, o = _fine_vs_oracle(oracle, inst)
    err = np.abs(g - o)
    assert err.max() <= 1.0 / 255.0, f"max pixel error {err.max():.4g} (> 1/255)"
    assert np.array_equal(g[:, 3] > 0, o[:, 3] > 0), "coverage differs"


@pytest.mark.parametrize("tile", [8, 16])
@pytest.mark.parametrize("avg", [4, 9])
def test_fine_pass_split_tiles_near_a_full_pool(oracle, tile, avg):  # noqa: F811
    """Split tiles whose bins hold about a pool's worth of fragments: parts
    that stay clear of it, that are taken again with exact counts, and that
    send the tile to the in-order walk."""
    inst = small_instance(strands=6000, points=32, width=320, height=240, tile_size=tile, depth_bins=4, slices=4)
    inst.cfg.avg_fragments_per_slice = avg
    cnt, g, o = _fine_vs_oracle(oracle, inst)
    assert cnt["fineSplitTiles"] > 0, "no tile was split: the test does not test"
    err = np.abs(g - o)
    assert err.max() <= 1.0 / 255.0, f"max pixel error {err.max():.4g} (> 1/255)"


@pytest.mark.parametrize("tile", [8, 16, 32])
@pytest.mark.parametrize("points,fiber,size", [(2, 5e-4, (640, 480)), (9, 2e-2, (301, 217)), (16, 2e-5, (640, 480)),
                                               (16, 5e-4, (2900, 1700))])
def test_tiles_pass_segments_of_every_size_bit_exact(oracle, tile, points, fiber, size):  # noqa: F811
    """Segments of tens of tiles each (a warp's accumulators hold a few of its
    segments at a time), of one tile, thick and thinner than a pixel; a number
    of segments that ends inside a warp."""
    inst = small_instance(strands=333, points=points, width=size[0], height=size[1], tile_size=tile,
                          fiber_radius=fiber, avg_segments_per_tile=2048)
    fr = frame_of(inst)
    ctx, hair, rb, d = _raster_gpu(inst, fr)
    _compare_tiles(oracle, inst, fr, rb)


@pytest.mark.parametrize("points,fiber,size", [(2, 5e-4, (640, 480)), (9, 2e-2, (301, 217)), (16, 2e-5, (640, 480)),
                                               (16, 5e-4, (2900, 1700)), (16, 2e-3, (64, 1900))])
def test_hair_depth_segments_of_every_size_bit_exact(oracle, points, fiber, size):  # noqa: F811
    """Triangles of one pixel to thousands (drawn by whole blocks), thick and
    thinner than a pixel; a number of points that ends inside a warp."""
    inst = small_instance(strands=333, points=points, width=size[0], height=size[1], fiber_radius=fiber)
    fr = frame_of(inst)
    ctx = _ctx(inst)
    hair = HairObject(inst.hair, inst.cfg.shading_points)
    rb = RasterBuffers(ctx, inst.width, inst.height)
    d = torch.as_tensor(inst.scene_depth).cuda()
    out = torch.empty_like(d)
    HwHairPass(ctx).cmd_draw_hair_depth(fr.uniforms, hair, d, out, rb)
    ctx.sync()
    hb = inst.hair
    o = oracle.hair_depth(fr.uniforms, hb.hair_data, hb.asset.positions, hb.tangents, hb.asset.strands,
                          inst.scene_depth)
    g = out.cpu().numpy()
    assert (g < inst.scene_depth).sum() > 20, "little hair in front: the test does not test"
    assert np.array_equal(g.view(np.uint32), o.view(np.uint32))


def _with_long_strands(strands, points, size, tile, fiber, longer, threshold):
    """Every other strand `longer` times as long."""
    inst = small_instance(strands=strands, points=points, width=size[0], height=size[1], tile_size=tile,
                          fiber_radius=fiber, avg_segments_per_tile=512)
    p = inst.hair.asset.positions.reshape(strands, points, 4)
    p[::2, :, :3] = p[::2, :1, :3] + longer * (p[::2, :, :3] - p[::2, :1, :3])
    inst.hair = HO.build_hair_buffers(inst.hair.asset)
    inst.cfg.invalid_tiles_per_segment_threshold = threshold
    return inst


@pytest.mark.parametrize("tile,size,fiber,longer", [(8, (2900, 1700), 5e-4, 8), (16, (2901, 1697), 5e-4, 12),
                                                    (8, (2160, 1440), 2e-2, 6), (32, (9000, 1200), 5e-4, 300)])
@pytest.mark.parametrize("threshold", [128, 700, 100000])
def test_tiles_pass_segments_past_the_accumulators_bit_exact(oracle, tile, size, fiber, longer, threshold):  # noqa: F811
    """Segments of more tiles than a warp has accumulators, which a threshold above the default lets
    through, some longer than the spans' range, among ordinary ones."""
    inst = _with_long_strands(90, 3, size, tile, fiber, longer, threshold)
    fr = frame_of(inst)
    ctx, hair, rb, d = _raster_gpu(inst, fr)
    _, osg, _ = _compare_tiles(oracle, inst, fr, rb)
    if threshold > 128:
        inst = _with_long_strands(90, 3, size, tile, fiber, longer, 128)
        _, rb128 = _raster_gpu(inst, frame_of(inst))[1:3]
        assert osg[0] > rb128.read_tile_segments()[0], "no segment past the default threshold: the test does not test"


@pytest.mark.parametrize("tile,slices", [(8, 4), (16, 8), (32, 4)])
def test_fine_pass_segments_longer_than_the_spans_range(oracle, tile, slices):  # noqa: F811
    """A viewport and segments above 8,192 px: rows whose edges are out of the spans' range keep the
    whole box."""
    inst = _with_long_strands(60, 3, (9000, 1200), tile, 2e-3, 300, 1 << 20)
    inst.cfg.slices_per_pixel = slices
    cnt, g, o = _fine_vs_oracle(oracle, inst)
    err = np.abs(g - o)
    assert err.max() <= 1.0 / 255.0, f"max pixel error {err.max():.4g} (> 1/255)"
    assert np.array_equal(g[:, 3] > 0, o[:, 3] > 0), "coverage differs"
    assert (o[:, 3] > 0).sum() > 5000
