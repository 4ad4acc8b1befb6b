"""The tile sort, the bins' lists and the fine pass's work items where their
ranges end: tiles per warp of the sort, records per bin (a group of 8 lanes, a
warp, a block, several sorted runs), and split tiles that are drawn in order
from their first group on."""
import numpy as np
import pytest

from helpers import frame_of, small_instance

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from hairfb.passes import HairFinePass, HairTileSortPass  # noqa: E402
from test_gpu_parity import (_compare_tiles, _fine_vs_oracle, _raster_gpu, _shading_input,  # noqa: E402,F401
                             oracle)


@pytest.mark.parametrize("size", [(8, 8), (248, 8), (264, 8), (301, 217), (1361, 767), (2900, 1700)])
@pytest.mark.parametrize("buckets,width", [(1, 16), (7, 1), (64, 16), (256, 3)])
def test_tile_sort_every_tile_count(size, buckets, width):
    """1, 31, 33, 1,064, 16,416 and 77,319 tiles of 8 px; buckets from one to the most."""
    inst = small_instance(strands=1500, width=size[0], height=size[1], tile_size=8, avg_segments_per_tile=2048)
    inst.cfg.sort_buckets = buckets
    inst.cfg.sort_bucket_size = width
    ctx, hair, rb, d = _raster_gpu(inst, frame_of(inst))
    HairTileSortPass(ctx).cmd_sort_hair_tiles(rb)
    ctx.sync()
    count = rb.read_segment_counts()
    bucket = np.minimum(count // width, buckets - 1)
    drawn = np.nonzero(count)[0]
    want = drawn[np.argsort(-bucket[drawn].astype(np.int64), kind="stable")]
    got = rb.read_tile_list()
    assert got[0] == len(want) and np.array_equal(got[1:1 + len(want)], want)
    hist = np.bincount(bucket[drawn], minlength=buckets)
    assert np.array_equal(rb.read_sort_buckets().reshape(-1, 2), np.stack([hist, hist], 1))


@pytest.mark.parametrize("strands,points,size,tile,bins", [
    (40, 4, (320, 240), 16, 8), (1500, 16, (640, 480), 8, 32), (6000, 32, (320, 240), 16, 16),
    (6000, 32, (200, 160), 32, 2), (20000, 32, (64, 48), 32, 1)])
def test_lists_of_every_length(oracle, strands, points, size, tile, bins):  # noqa: F811
    """Bins of one record to more than one sorted run (16,384 records)."""
    tiles = -(-size[0] // tile) * -(-size[1] // tile)
    inst = small_instance(strands=strands, points=points, width=size[0], height=size[1], tile_size=tile,
                          depth_bins=bins, avg_segments_per_tile=-(-4_000_000 // tiles))
    fr = frame_of(inst)
    ctx, hair, rb, d = _raster_gpu(inst, fr)
    _compare_tiles(oracle, inst, fr, rb)


@pytest.mark.parametrize("tile,slices,avg,bins", [(8, 8, 1, 4), (8, 16, 1, 4), (16, 8, 1, 4), (16, 16, 1, 4),
                                                  (16, 8, 6, 4), (8, 8, 6, 4), (32, 8, 1, 4), (16, 4, 1, 2)])
def test_split_tiles_drawn_in_order(oracle, tile, slices, avg, bins):  # noqa: F811
    """Tiles whose later groups fill a pool, drawn in order after their first
    group: the oracle's image, and the same image and counters on every run,
    whichever group finds the full pool first."""
    inst = small_instance(strands=6000, points=32, width=320, height=240, tile_size=tile, depth_bins=bins,
                          slices=slices, avg_segments_per_tile=2048)
    inst.cfg.avg_fragments_per_slice = avg
    cnt, g, o = _fine_vs_oracle(oracle, inst)
    assert cnt["fineSplitTiles"] > 0, "no tile was split: the test does not test"
    err = np.abs(g - o)
    assert err.max() <= 1.0 / 255.0, f"max pixel error {err.max():.4g} (> 1/255)"
    for _ in range(3):
        ctx, hair, rb, d = _raster_gpu(inst, frame_of(inst))
        hair.shading.copy_(torch.as_tensor(_shading_input(inst)))
        HairFinePass(ctx).cmd_rasterize_slices_hair(frame_of(inst).uniforms, hair, d, rb)
        ctx.sync()
        assert np.array_equal(rb.read_result()[4:].reshape(-1, 4), g)
        again = ctx.counters()
        assert all(again[k] == cnt[k] for k in ("fineSplitTiles", "fineSplitRedone", "finePoolFullBins"))


CLASSES = ((1, 8), (9, 32), (33, 256), (257, 1024), (1025, 16384), (16385, 1 << 24))


@pytest.mark.parametrize("strands,points,size,tile,bins,classes", [
    (6000, 32, (320, 240), 16, 16, (0, 1, 2, 3)), (60000, 16, (192, 160), 32, 4, (1, 2, 3, 4, 5))])
def test_lists_of_every_class(oracle, strands, points, size, tile, bins, classes):  # noqa: F811
    """Bins for each way to sort one -- 8 lanes, a warp's registers, its shared memory, a block's, all of
    a block's, sorted runs -- and that they are there."""
    tiles = -(-size[0] // tile) * -(-size[1] // tile)
    inst = small_instance(strands=strands, points=points, width=size[0], height=size[1], tile_size=tile,
                          depth_bins=bins, avg_segments_per_tile=-(-4_000_000 // tiles))
    fr = frame_of(inst)
    ctx, hair, rb, d = _raster_gpu(inst, fr)
    heads = rb.read_tiles().reshape(-1, 4)
    n = heads[heads[:, 2] != 0, 3]  # the lists' lengths
    for k in classes:
        assert ((n >= CLASSES[k][0]) & (n <= CLASSES[k][1])).any(), f"no bin of {CLASSES[k]} records"
    _compare_tiles(oracle, inst, fr, rb)
