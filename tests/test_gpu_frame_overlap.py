"""Whole frames whose hair depth runs beside the tiles and fine passes, and
frames that may not overlap them (the hair's depth drawn over the scene depth
itself, or over another instance's): both give what the passes give in turn."""
import numpy as np
import pytest

from helpers import small_instance

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from hairfb.lib import Context  # noqa: E402
from hairfb.passes import clear_before_render  # noqa: E402
from hairfb.renderer import BatchRenderer, Renderer  # noqa: E402


def _state(r):
    torch.cuda.synchronize()
    return [r.hair.positions.cpu().numpy(), r.grids.density_velocity.cpu().numpy(), r.scene_depth.cpu().numpy(),
            r.hair_depth.cpu().numpy(), r.rb.read_tiles()[:, :2], r.rb.read_segment_counts(), r.hair.shading.cpu().numpy()], \
        r.rb.read_result()[4:]


def _renderer(k, ctx, shared):
    inst = small_instance(seed=k, strands=700 + 300 * k, width=320 + 16 * k, height=240)
    r = Renderer(inst, 0, ctx=ctx, hair_depth=True)
    if shared:  # the hair is drawn over the scene depth that the next frame tests against
        r.hair_depth = r.shading_depth = r.scene_depth
    return r


@pytest.mark.parametrize("shared", [False, True])
@pytest.mark.parametrize("batch", [1, 3])
def test_frames_equal_the_passes_in_turn(shared, batch):
    inst = small_instance()
    ctx = Context(inst.cfg.to_c(), 0)
    got = [_renderer(k, ctx, shared) for k in range(batch)]
    want = [_renderer(k, ctx, shared) for k in range(batch)]
    torch.cuda.synchronize()
    many = BatchRenderer(got)
    for r in got + want:
        r.before_first_frame()
    for _ in range(4):  # the batch's first frames are launches, the later ones a graph
        many.frame() if batch > 1 else got[0].frame_native()
        for r in want:
            r.frame()
        for g, w in zip(got, want):
            (gs, gi), (ws, wi) = _state(g), _state(w)
            for a, b in zip(gs, ws):
                assert np.array_equal(a, b)
            assert np.abs(gi - wi).max() <= 1.0 / 255.0


def test_batch_with_another_instances_depth():
    """Instance 0's hair depth is instance 1's scene depth: the batched frame
    runs each pass for both instances before the next pass."""
    def pair():
        ctx = Context(small_instance().cfg.to_c(), 0)
        rs = [_renderer(1, ctx, False) for _ in range(2)]
        rs[1].scene_depth = rs[0].hair_depth
        torch.cuda.synchronize()
        for r in rs:
            r.before_first_frame()
        return ctx, rs
    _, got = pair()
    many = BatchRenderer(got)
    ctx, want = pair()
    for _ in range(3):
        many.frame()
        for r in want:
            r.simulate()
            clear_before_render(ctx, r.rb)
            r.tiles.cmd_draw_hair_to_tiles(r.uniforms, r.hair, r.scene_depth, r.rb)
            r.sort.cmd_sort_hair_tiles(r.rb)
            r.fine.cmd_rasterize_slices_hair(r.uniforms, r.hair, r.scene_depth, r.rb)
        ctx.sync()
        depth = [r.scene_depth.clone() for r in want]  # both copied before either's hair is drawn
        torch.cuda.synchronize()
        for r, d in zip(want, depth):
            r.hw_hair.cmd_draw_hair_depth(r.uniforms, r.hair, d, r.hair_depth, r.rb)
        for r in want:
            r.shading.cmd_compute_shading_points(r.uniforms, r.hair, r.shading_depth)
            r.frame_idx += 1
        ctx.sync()
        for g, w in zip(got, want):
            a, b = _state(g)[0], _state(w)[0]
            for k in (0, 1, 4, 5):  # positions, grids, tile depths, counts
                assert np.array_equal(a[k], b[k])
    assert np.array_equal(_state(got[0])[0][3], _state(want[0])[0][3])


@pytest.mark.parametrize("batch", [1, 3])
def test_frames_on_changing_streams(batch):
    """Each frame on another stream than the last, the streams ordered by the caller: the work on the
    context's own second stream is joined into the stream that the frame was given."""
    inst = small_instance()
    ctx = Context(inst.cfg.to_c(), 0)
    got = [_renderer(k, ctx, False) for k in range(batch)]
    plain = Context(inst.cfg.to_c(), 0)
    want = [_renderer(k, plain, False) for k in range(batch)]
    torch.cuda.synchronize()
    for r in got + want:
        r.before_first_frame()
    torch.cuda.synchronize()
    many = BatchRenderer(got)
    streams = [torch.cuda.Stream() for _ in range(3)]
    for f in range(7):
        s = streams[f % 3]
        s.wait_stream(streams[(f - 1) % 3])
        ctx.set_stream(s)
        many.frame() if batch > 1 else got[0].frame_native()
        for r in want:
            r.frame()
    torch.cuda.synchronize()
    for g, w in zip(got, want):
        (gs, gi), (ws, wi) = _state(g), _state(w)
        for a, b in zip(gs, ws):
            assert np.array_equal(a, b)
        assert np.abs(gi - wi).max() <= 1.0 / 255.0


def test_frames_captured_by_the_caller():
    """Two frames in a graph of the caller's: nothing runs while they are captured, and a launch of the
    graph gives the two frames."""
    inst = small_instance()
    s = torch.cuda.Stream()
    ctx = Context(inst.cfg.to_c(), 0)
    ctx.set_stream(s)
    first, got = _renderer(1, ctx, False), _renderer(1, ctx, False)
    plain = Context(inst.cfg.to_c(), 0)
    want = _renderer(1, plain, False)
    torch.cuda.synchronize()
    for r in (first, got, want):
        r.before_first_frame()
    first.frame_native()  # the context's buffers grow to these frames' sizes
    torch.cuda.synchronize()
    before = _state(got)[0]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s, capture_error_mode="thread_local"):
        got.frame_native()
        got.frame_native()
    for a, b in zip(before, _state(got)[0]):
        assert np.array_equal(a, b)
    with torch.cuda.stream(s):
        graph.replay()
    want.frame()
    want.frame()
    (gs, gi), (ws, wi) = _state(got), _state(want)
    for a, b in zip(gs, ws):
        assert np.array_equal(a, b)
    assert np.abs(gi - wi).max() <= 1.0 / 255.0
    got.frame_native()  # the context's streams are as they were
    want.frame()
    for a, b in zip(_state(got)[0], _state(want)[0]):
        assert np.array_equal(a, b)


def test_normals_are_cleared_on_the_contexts_stream():
    """A frame with AO on the context's own stream while torch's stream is busy: the normals are
    cleared in turn with the passes, not whenever torch's stream gets to it."""
    inst = small_instance()

    def frames(busy):
        ctx = Context(inst.cfg.to_c(), 0)
        r = Renderer(inst, 0, ctx=ctx, hair_depth=True, ao=True)
        torch.cuda.synchronize()
        r.before_first_frame()
        ctx.sync()
        torch.cuda.synchronize()
        if busy:
            torch.cuda._sleep(100_000_000)  # about 50 ms
        r.frame()
        ctx.sync()
        torch.cuda.synchronize()
        return r.normals.cpu().numpy(), r.ao.cpu().numpy(), r.hair.shading.cpu().numpy()

    want, got = frames(False), frames(True)
    assert (want[0] != 0).any()
    for a, b in zip(want, got):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
