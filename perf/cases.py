"""The work that users have this library do, as cases that can be timed.

Seven kinds of call, each through the public classes of ``hairfb`` (which
forward to ``libhairfb.so``):

- ``frame``    one frame of one hair instance (``Renderer.frame_native``, or
               ``Renderer.frame`` pass by pass with the ambient occlusion)
- ``batch``    one frame of many uneven instances (``BatchRenderer.frame``)
- ``draw``     the raster, hair depth and shading passes of hair at rest
- ``sim``      the three simulation passes
- ``shading``  the strand-space shading with a shadow map and an AO texture
- ``gtao``     the ambient occlusion pass on a depth buffer and normals
- ``present``  the 8-bit images of a batch

Inputs follow ``hairfb.synthetic``'s growth model (roots on the upper half of
a head sphere, random-walk strands, a framing camera, the head's signed
distance field and depth), made on the GPU from the seed.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "frostbitten-hair-webgpu_gb300"))

from hairfb import hair_object as HO, matrices as M, synthetic, uniforms as UN  # noqa: E402
from hairfb.config import HairConfig, SimulationParams  # noqa: E402
from hairfb.formats import SdfVolume  # noqa: E402
from hairfb.lib import Context, ptr, strand_grid_order  # noqa: E402
from hairfb.passes import AoPass, PresentPass, RasterBuffers  # noqa: E402
from hairfb.renderer import BatchRenderer, Renderer  # noqa: E402

HEAD_RADIUS = 0.1
SEGMENT = 0.01


def listed():
    return [
        # the smallest call: one small hair object at VGA, where launches and latency count
        _frame("frame_small", 2000, 16, 640, 480),
        # an ordinary frame: 10k curly strands in wind at full HD
        _frame("frame_full", 10000, 32, 1920, 1080, bins=16, shading_points=16, grid=64, sdf=64, iterations=4,
               curl=True, wind=1.0),
        # the reference's own default constants at the size of its Sintel asset, pass by pass with GTAO
        _frame("frame_reference", 11400, 16, 1920, 1080, tile=8, bins=32, slices=8, shading_points=64, grid=64,
               sdf=64, ao=True),
        # the batched workload: 64 uneven instances in one call, at the constants its autotuner picks
        _batch("batch64", 64, "uniform", 1000, 20000, "16,24,32", "256,512,1024", tile=8, bins=4),
        # one tick of the frame server: a few sessions of very different sizes at the serving constants
        _batch("batch_tick", 6, "log", 500, 50000, "32", "256-2048", tile=16, bins=16),
        # the largest: 200k strands, most in a ponytail, drawn at 4K
        _draw("draw_4k", 200000, 32, 3840, 2160, bins=32, slices=8, shading_points=32, ponytail=0.6),
        # odd sizes and the other options: a ragged viewport, 32 px tiles, part of the strands (LOD)
        _draw("draw_odd", 7001, 23, 1361, 767, tile=32, bins=7, slices=5, shading_points=13, lod=70.0, quadratic=True),
        # the simulation alone: many strands, and a few long ones of an odd length
        _sim("sim_many", 40000, 16, grid=64, sdf=64),
        _sim("sim_long", 1501, 65, grid=64, sdf=32, iterations=5),
        # the shading alone with every input: shadow map, AO, the reference's 64 points per strand
        _shading("shading_lit", 20000, 32, 1920, 1080, shading_points=64, shadow=1024),
        # the ambient occlusion alone
        _gtao("gtao_hd", 1920, 1080),
        # the images of a batched frame, for display or encoding
        _present("present64", 64, "256,512,1024"),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def look():
        return dict(tile=rng.choice([8, 16, 32]), bins=rng.choice([4, 8, 11, 16, 32]), slices=rng.choice([2, 4, 5, 8]),
                    shading_points=rng.choice([8, 13, 16, 32]))

    kind = rng.choice(["frame", "frame", "batch", "draw", "sim", "shading", "gtao", "present"])
    if kind == "frame":
        points, grid = rng.randint(5, 40), rng.choice([48, 64])
        return _frame(None, _settled(log(500, 30000), points, grid), points, log(200, 2048), log(200, 2048), grid=grid,
                      sdf=rng.choice([32, 48, 64]), iterations=rng.randint(2, 8), curl=rng.random() < 0.5,
                      wind=rng.choice([0.0, 1.0]), ao=rng.random() < 0.25, **look())
    if kind == "batch":
        return _batch(None, log(2, 48), "log", 500, 20000, rng.choice(["16,24,32", "32", "11,19,30"]), "256-1024",
                      **look())
    if kind == "draw":
        return _draw(None, log(500, 100000), rng.randint(5, 33), log(200, 3000), log(200, 2160),
                     ponytail=rng.choice([0.0, 0.4]), lod=rng.choice([100.0, 55.0]), quadratic=rng.random() < 0.5,
                     **look())
    if kind == "sim":
        points, grid = rng.choice([8, 15, 16, 31, 32, 64, 101]), rng.choice([48, 64, 96])
        return _sim(None, _settled(log(500, 60000), points, grid), points, grid=grid,
                    sdf=rng.choice([32, 64]), iterations=rng.randint(2, 8))
    if kind == "shading":
        return _shading(None, log(500, 50000), rng.randint(5, 40), log(200, 2048), log(200, 2048),
                        shading_points=rng.choice([7, 16, 64]), shadow=rng.choice([512, 1000, 1024]))
    if kind == "gtao":
        return _gtao(None, log(200, 3840), log(200, 2160))
    return _present(None, log(1, 100), rng.choice(["256,512,1024", "256-2048", "333,501"]))


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------

def _case(name, kind, **kw):
    return {**({"name": name} if name else {}), "kind": kind, **kw}


def _frame(name, strands, points, width, height, *, tile=16, bins=8, slices=4, shading_points=8, grid=32, sdf=32,
           iterations=7, curl=False, wind=0.0, ao=False):
    return _case(name, "frame", strands=strands, points=points, width=width, height=height, tile=tile, bins=bins,
                 slices=slices, shading_points=shading_points, grid=grid, sdf=sdf, iterations=iterations, curl=curl,
                 wind=wind, ao=ao)


def _batch(name, instances, spread, lo, hi, points, sides, *, tile, bins, slices=4, shading_points=8):
    return _case(name, "batch", instances=instances, spread=spread, strands_lo=lo, strands_hi=hi, points=points,
                 sides=sides, tile=tile, bins=bins, slices=slices, shading_points=shading_points, grid=64, sdf=32,
                 iterations=7)


def _draw(name, strands, points, width, height, *, tile=16, bins=8, slices=4, shading_points=8, ponytail=0.0,
          lod=100.0, quadratic=False):
    return _case(name, "draw", strands=strands, points=points, width=width, height=height, tile=tile, bins=bins,
                 slices=slices, shading_points=shading_points, ponytail=ponytail, lod=lod, quadratic=quadratic)


def _sim(name, strands, points, *, grid, sdf, iterations=7):
    return _case(name, "sim", strands=strands, points=points, grid=grid, sdf=sdf, iterations=iterations)


def _shading(name, strands, points, width, height, *, shading_points, shadow):
    return _case(name, "shading", strands=strands, points=points, width=width, height=height,
                 shading_points=shading_points, shadow=shadow)


def _gtao(name, width, height):
    return _case(name, "gtao", width=width, height=height)


def _present(name, images, sides):
    return _case(name, "present", images=images, sides=sides)


def _settled(strands, points, grid):
    """At most the strands that the simulation's 32-bit fixed-point grid can hold at the roots: past about 2,147 its
    density wraps, and the hair blows apart."""
    cell = 4.0 * (HEAD_RADIUS + 0.0085 * points) / (grid - 1)
    return min(strands, int(1500 / (11100 * cell ** 3)))


def _sides(case, rng, count):
    """Square viewports: one of a list, or an area log-uniform between two sides."""
    text = case["sides"]
    if "-" in text:
        lo, hi = (int(v) for v in text.split("-"))
        return [16 * round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / 16) for _ in range(count)]
    return [int(v) for v in rng.choice([int(v) for v in text.split(",")], count)]


def _members(case, seed):
    """The instances of a batch, as (strands, points, side)."""
    n, lo, hi = case["instances"], case["strands_lo"], case["strands_hi"]
    # sizes are the case's own, whatever the seed: the seed changes the values
    rng = np.random.Generator(np.random.PCG64(n))
    if case["spread"] == "log":
        strands = [int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) for _ in range(n)]
    else:
        strands = [int(v) for v in rng.integers(lo, hi + 1, n)]
    points = [int(v) for v in rng.choice([int(v) for v in case["points"].split(",")], n)]
    strands = [_settled(s, p, case["grid"]) for s, p in zip(strands, points)]
    return list(zip(strands, points, _sides(case, rng, n)))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _generator(seed, index=0):
    g = torch.Generator(device="cuda")
    g.manual_seed(1009 * int(seed) + index)
    return g


def _unit(v):
    return v / v.norm(dim=-1, keepdim=True)


def _grow(g, strands, points, curl=False, ponytail=0.0):
    """synthetic.grow_hair's model on the GPU: (S, P, 4) float32 positions, w = isMovable."""
    def rand(*shape):
        return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)

    def randn(*shape):
        return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)

    def perp(d):
        a = randn(*d.shape)
        return _unit(a - (a * d).sum(-1, keepdim=True) * d)

    y, phi = rand(strands), rand(strands) * (2.0 * math.pi)
    s = (1.0 - y * y).clamp_min(0.0).sqrt()
    n = torch.stack([s * phi.cos(), y, s * phi.sin()], -1)
    d = n.clone()
    sigma = torch.full((strands,), 0.2, device="cuda", dtype=torch.float64)
    tail = int(round(ponytail * strands))
    if tail:
        axis = _unit(torch.tensor([0.0, 0.35, -1.0], device="cuda", dtype=torch.float64))
        cone = _unit(torch.tensor([0.0, -1.0, -0.35], device="cuda", dtype=torch.float64))
        n[:tail] = _unit(axis + 0.25 * randn(tail, 3))
        d[:tail] = _unit(cone + 0.08 * randn(tail, 3))
        sigma[:tail] = 0.05
    out = torch.ones(strands, points, 4, device="cuda", dtype=torch.float64)
    p = HEAD_RADIUS * n
    out[:, 0, :3] = p
    out[:, 0, 3] = 0.0
    e1 = perp(n)
    e2 = torch.linalg.cross(n, e1)
    phase = rand(strands) * (2.0 * math.pi)
    for k in range(1, points):
        ang = (randn(strands) * sigma)[:, None]
        d = _unit(ang.cos() * d + ang.sin() * perp(d))
        if curl:
            a = (phase + 0.8 * k)[:, None]
            d = _unit(d + 0.3 * (a.cos() * e1 + a.sin() * e2))
        p = p + SEGMENT * d
        out[:, k, :3] = p
    return out.float()


def _hair(pos):
    """The static buffers of a hair object, as hairfb.hair_object makes them, from (S, P, 4) positions."""
    S, P, _ = pos.shape
    x = pos[..., :3].double()
    d = (x[:, 1:] - x[:, :-1]).float().double()
    tan = torch.zeros_like(pos)
    tan[:, :-1, :3] = _unit(d).float()
    tan[:, -1] = tan[:, -2]
    length = (x[:, 1:] - x[:, :-1]).norm(dim=-1)
    length = torch.cat([length, length[:, -1:]], 1).float()
    flat = pos[..., :3].reshape(-1, 3)
    bmin, bmax = flat.amin(0).cpu().numpy(), flat.amax(0).cpu().numpy()
    center, radius = HO.bounding_sphere(bmin, bmax)
    asset = HO.HairAsset(S, P, pos.reshape(S * P, 4))
    return HO.HairBuffers(asset, tan.reshape(S * P, 4), length.reshape(S * P), (bmin, bmax), center, radius,
                          HO.hair_data_bytes(S, P, center, radius))


def _sdf(dims, bmin, bmax):
    """The head, and at 64^3 and above an ellipsoid below it, at texel centres, x fastest."""
    lo, hi = (torch.as_tensor(np.asarray(b, np.float64), device="cuda") for b in (bmin, bmax))
    t = (torch.arange(dims, device="cuda", dtype=torch.float64) + 0.5) / dims
    z, y, x = torch.meshgrid(t, t, t, indexing="ij")
    p = lo + torch.stack([x, y, z], -1) * (hi - lo)
    d = p.norm(dim=-1) - HEAD_RADIUS
    if dims < 64:
        return SdfVolume(dims, np.asarray(bmin, np.float32), np.asarray(bmax, np.float32), d.float().reshape(-1))
    radii = torch.tensor([0.16, 0.07, 0.09], device="cuda", dtype=torch.float64)
    body = torch.tensor([0.0, -0.17, 0.02], device="cuda", dtype=torch.float64)
    d = torch.minimum(d, (((p - body) / radii).norm(dim=-1) - 1.0) * 0.07)
    return SdfVolume(dims, np.asarray(bmin, np.float32), np.asarray(bmax, np.float32), d.float().reshape(-1))


def _head_depth(width, height, camera):
    """NDC depth of the head (synthetic.sphere_depth), row 0 = top, 1 where nothing is hit."""
    def dev(a):
        return torch.as_tensor(a, device="cuda", dtype=torch.float64)

    vp = M.to_rows(camera.proj(width, height)) @ M.to_rows(camera.view())
    vp, inv = dev(vp), dev(np.linalg.inv(vp))
    xs = (torch.arange(width, device="cuda", dtype=torch.float64) + 0.5) / width * 2.0 - 1.0
    ys = 1.0 - (torch.arange(height, device="cuda", dtype=torch.float64) + 0.5) / height * 2.0
    y, x = torch.meshgrid(ys, xs, indexing="ij")
    one = torch.ones_like(x)
    near = torch.stack([x, y, 0.0 * one, one], -1) @ inv.T
    far = torch.stack([x, y, one, one], -1) @ inv.T
    o = near[..., :3] / near[..., 3:]
    d = _unit(far[..., :3] / far[..., 3:] - o)
    b = (o * d).sum(-1)
    disc = b * b - (o * o).sum(-1) + (0.98 * HEAD_RADIUS) ** 2
    t = -b - disc.clamp_min(0.0).sqrt()
    clip = torch.cat([o + t[..., None] * d, one[..., None]], -1) @ vp.T
    return torch.where((disc >= 0.0) & (t > 0.0), clip[..., 2] / clip[..., 3], one).float().reshape(-1)


def _config(case, **kw):
    return HairConfig(tile_size=case.get("tile", 16), tile_depth_bins=case.get("bins", 8),
                      slices_per_pixel=case.get("slices", 4), shading_points=case.get("shading_points", 8),
                      grid_dims=case.get("grid", 32), alpha_quadratic=case.get("quadratic", False),
                      processor_count=0, **kw)


def _instance(case, g, strands, points, width, height):
    """One hair instance of the case, at rest."""
    pos = _grow(g, strands, points, case.get("curl", False), case.get("ponytail", 0.0))
    hair = _hair(pos)
    sim = SimulationParams(delta_time=1.0 / 60.0, constraint_iterations=case.get("iterations", 7),
                           collision_sphere=(0.0, 0.0, 0.0, HEAD_RADIUS))
    c, r = hair.sphere_center.astype(np.float64), 1.1 * float(hair.sphere_radius)
    sdf = _sdf(case.get("sdf", 32), c - r, c + r)
    camera = synthetic.framing_camera(hair.sphere_center, float(hair.sphere_radius))
    grid = HO.scale_bounding_box(hair.bbox[0], hair.bbox[1], sim.grid_scale)
    scene = UN.SceneParams(width=width, height=height, camera=camera, fiber_radius=5e-4,
                           sdf_bounds=(sdf.bounds_min, sdf.bounds_max), grid_bounds=grid,
                           hair_sphere=(hair.sphere_center, float(hair.sphere_radius)),
                           collision_sphere=sim.collision_sphere, sdf_distance_offset=sim.sdf_distance_offset)
    wind = torch.randn(3, generator=g, device="cuda", dtype=torch.float64)
    return synthetic.Instance(_config(case), sim, hair, sdf, scene, _head_depth(width, height, camera), np.zeros(3),
                              HEAD_RADIUS, _unit(wind).cpu().numpy(), wind_amplitude=case.get("wind", 0.0))


def _device(a):
    return a if isinstance(a, torch.Tensor) else torch.as_tensor(np.ascontiguousarray(a)).cuda()


def _renderer(inst, ctx, **kw):
    a = inst.hair.asset
    order = strand_grid_order(a.positions.cpu().numpy(), a.strands, a.points_per_strand).view(np.int32)
    # a segment pool that holds every record: long thin segments touch a few tiles each
    segments = a.strands * (a.points_per_strand - 1)
    tx, ty = inst.cfg.tile_count(inst.width, inst.height)
    return Renderer(inst, ctx=ctx, max_drawn=6 * segments + tx * ty, pooled=True, upload=_device, grid_order=order,
                    **kw)


def _home(renderers):
    """Keeps the buffers that the passes write in one allocation per kind, as a program does that reads them
    all back; returns them by kind."""
    out = {}

    def take(kind, dtype, sizes):
        whole = torch.zeros(sum(-(-n // 64) * 64 for n in sizes), dtype=dtype, device="cuda")
        views, at = [], 0
        for n in sizes:
            views.append(whole[at:at + n])
            at += -(-n // 64) * 64
        out[kind] = whole
        return views

    def move(kind, get, put):
        old = [get(r) for r in renderers]
        for r, o, v in zip(renderers, old, take(kind, old[0].dtype, [o.numel() for o in old])):
            v.copy_(o.reshape(-1))
            put(r, v.view(o.shape))

    move("positions_0", lambda r: r.hair.positions_0, lambda r, v: setattr(r.hair, "positions_0", v))
    move("positions_1", lambda r: r.hair.positions_1, lambda r, v: setattr(r.hair, "positions_1", v))
    move("shading", lambda r: r.hair.shading, lambda r, v: setattr(r.hair, "shading", v))
    move("density_velocity", lambda r: r.grids.density_velocity, lambda r, v: setattr(r.grids, "density_velocity", v))
    move("density_grad_wind", lambda r: r.grids.density_grad_wind,
         lambda r, v: setattr(r.grids, "density_grad_wind", v))

    def depth(r, v):
        r.hair_depth = r.shading_depth = v

    move("hair_depth", lambda r: r.hair_depth, depth)

    def tiles(r):
        tx, ty = r.cfg.tile_count(r.inst.width, r.inst.height)
        return tx * ty

    sizes = {"tiles": [tiles(r) * r.cfg.tile_depth_bins * 4 for r in renderers],
             "tileSegments": [1 + 2 * r.max_drawn for r in renderers],
             "segmentCountPerTile": [tiles(r) for r in renderers],
             "sortBuckets": [2 * r.cfg.sort_buckets for r in renderers],
             "tileList": [4 + tiles(r) for r in renderers]}
    for kind, n in sizes.items():
        for r, v in zip(renderers, take(kind, torch.int32, n)):
            setattr(r.rb.rb, kind, ptr(v))
    # the image follows a 16-byte header, which holds the pass's own queue
    views = take("image", torch.float32, [r.inst.width * r.inst.height * 4 + 64 for r in renderers])
    for r, v in zip(renderers, views):
        r.rb.rb.rasterizerResult = ptr(v[60:])
    if len(renderers) == 1:
        out["image"] = views[0][64:]
    return out


class _State:
    pass


_queue = []


def _context(cfg):
    """A context on the program's one queue, as the reference submits to one: passes run one after another."""
    if not _queue:
        _queue.append(torch.cuda.Stream())
    ctx = Context(cfg.to_c())
    ctx.set_stream(_queue[0])
    return ctx


# ---------------------------------------------------------------------------
# the interface
# ---------------------------------------------------------------------------

def prepare(case, seed):
    s = _State()
    s.kind = case["kind"]
    g = _generator(seed)
    if s.kind in ("frame", "draw"):
        inst = _instance(case, g, case["strands"], case["points"], case["width"], case["height"])
        s.ao = case.get("ao", False)
        s.ctx = _context(inst.cfg)
        s.renderer = _renderer(inst, s.ctx, hair_depth=True, ao=s.ao)
        s.renderer.hair.lod_render_percent = case.get("lod", 100.0)
        s.out = _home([s.renderer])
        torch.cuda.synchronize()
        with torch.cuda.stream(_queue[0]):  # the passes of a frame with AO clear and allocate with torch
            s.renderer.before_first_frame()
    elif s.kind == "batch":
        cfg = _config(case)
        s.ctx = _context(cfg)
        renderers = [_renderer(_instance(case, _generator(seed, k), S, P, side, side), s.ctx, hair_depth=True)
                     for k, (S, P, side) in enumerate(_members(case, seed))]
        s.out = _home(renderers)
        s.batch = BatchRenderer(renderers)
        torch.cuda.synchronize()
        s.batch.before_first_frame()
    elif s.kind == "sim":
        inst = _instance({**case, "wind": 1.0}, g, case["strands"], case["points"], 64, 64)
        s.ctx = _context(inst.cfg)
        r = s.renderer = _renderer(inst, s.ctx)
        r.hair.positions_0.copy_(_moving(g, inst))
        s.uniforms = _sim_uniforms(inst)
        torch.cuda.synchronize()
        r.grid_post.cmd_update_grids_after_sim(s.uniforms, r.hair, r.grids)
    elif s.kind == "shading":
        inst = _instance(case, g, case["strands"], case["points"], case["width"], case["height"])
        s.ctx = _context(inst.cfg)
        s.renderer = _renderer(inst, s.ctx)
        s.ao, s.shadow = _lighting(case, g)
        s.size, s.shadow_size = (s.ao.shape[1], s.ao.shape[0]), case["shadow"]
    elif s.kind == "gtao":
        s.uniforms, s.depth, s.normals = _ao_inputs(case, g)
        s.ctx = _context(HairConfig())
        s.width, s.height = case["width"], case["height"]
        s.ao = AoPass(s.ctx)
    else:
        rng = np.random.Generator(np.random.PCG64(case["images"]))
        cfg = HairConfig(tile_size=16)
        s.ctx = _context(cfg)
        s.present, s.items, sides = PresentPass(s.ctx), [], _sides(case, rng, case["images"])
        s.pixels = [torch.zeros(4 + 4 * n * n, device="cuda") for n in sides]
        s.image = torch.zeros(sum(n * n for n in sides), 4, dtype=torch.uint8, device="cuda")
        at = 0
        for k, (n, px) in enumerate(zip(sides, s.pixels)):
            rgba = px[4:].view(n * n, 4)
            rgba.uniform_(0.0, 1.2, generator=g)
            hair = torch.rand(n * n, 1, generator=g, device="cuda")
            rgba[:, 3:] = ((hair - 0.4) * 2.0).clamp(0.0, 1.0)  # bare pixels, thin hair, full cover
            rgba *= rgba[:, 3:] > 0
            rb = RasterBuffers(s.ctx, n, n, max_drawn=1, pooled=True)
            rb.rb.rasterizerResult = ptr(px)
            scene = UN.SceneParams(width=n, height=n, camera=UN.Camera(np.array([0.0, 0.0, 1.0]), np.zeros(3)))
            under = torch.rand(n, n, 4, generator=g, device="cuda") if k % 2 else None
            s.items.append((UN.pack_render_uniforms(scene, cfg, 1), rb, under, s.image[at:at + n * n].view(n, n, 4)))
            at += n * n
    torch.cuda.synchronize()
    return s


def run(s):
    if s.kind == "frame":
        if s.ao:
            with torch.cuda.stream(_queue[0]):
                s.renderer.frame()
            return {**s.out, "normals": s.renderer.normals, "ao": s.renderer.ao}
        s.renderer.frame_native()
        return s.out
    if s.kind == "draw":
        s.renderer.draw()
        return s.out
    if s.kind == "batch":
        s.batch.frame()
        return s.out
    if s.kind == "sim":
        r = s.renderer
        r.grid_pre.cmd_update_grids_before_sim(s.uniforms, r.grids, r.sdf)
        r.integrate.cmd_simulate_hair_positions(s.uniforms, r.hair, r.grids, r.sdf)
        r.grid_post.cmd_update_grids_after_sim(s.uniforms, r.hair, r.grids)
        return {"positions": r.hair.positions, "density_grad_wind": r.grids.density_grad_wind,
                "density_velocity": r.grids.density_velocity}
    if s.kind == "shading":
        r = s.renderer
        r.shading.cmd_compute_shading_points(r.uniforms, r.hair, r.scene_depth, s.ao, s.size, s.shadow, s.shadow_size)
        return r.hair.shading
    if s.kind == "gtao":
        with torch.cuda.stream(_queue[0]):
            return s.ao.cmd_calc_ao(s.uniforms, s.depth, s.normals, s.width, s.height)
    s.present.cmd_draw_batch(s.items)
    return s.image


def work(case):
    """Compulsory bytes (inputs read once, outputs written once) and fp32 operations, counted from the passes'
    formulas: a point of the integration ~150 per constraint iteration, a projected segment ~400, a shading point
    ~900, and per pixel what the pass does there once."""
    kind = case["kind"]
    if kind == "batch":
        members = [(S, P, n, n) for S, P, n in _members(case, 0)]
    elif kind == "present":
        rng = np.random.Generator(np.random.PCG64(case["images"]))
        px = [n * n for n in _sides(case, rng, case["images"])]
        return {"bytes": sum(px) * 20 + sum(px[1::2]) * 16, "flops": 60 * sum(px)}
    elif kind == "gtao":
        px = case["width"] * case["height"]
        return {"bytes": px * 12 + px, "flops": px // 4 * 12 * (8 * 2 * 45 + 90)}
    else:
        members = [(case["strands"], case["points"], case.get("width", 0), case.get("height", 0))]
    nbytes = flops = 0
    for S, P, W, H in members:
        n, sp, px = S * P, S * case.get("shading_points", 0), W * H
        grid, sdf = case.get("grid", 0) ** 3, case.get("sdf", 0) ** 3
        if kind in ("frame", "batch", "sim"):  # positions, initial, lengths; the grids and the field
            nbytes += n * (16 * 3 + 4 + 16) + grid * 48 + sdf * 4
            flops += n * (150 * case["iterations"] + 350) + grid * 150
        if kind in ("frame", "batch", "draw"):
            lod = case.get("lod", 100.0) / 100.0
            tiles = -(-W // case["tile"]) * -(-H // case["tile"])
            # tangents (positions too where the simulation has not read them), depth, image, hair depth, lists
            nbytes += n * (16 if kind != "draw" else 32) + px * 24 + tiles * (16 * case["bins"] + 4) + int(n * lod) * 16
            nbytes += sp * 32
            flops += int(n * lod) * 900 + px * 60 + sp * 900
        if kind == "shading":
            nbytes += n * 32 + sp * 16 + px * 5 + case["shadow"] ** 2 * 4
            flops += sp * (900 + 49 * 20)
        if case.get("ao"):
            nbytes += px * 8 + px
            flops += px // 4 * 12 * (8 * 2 * 45 + 90)
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------
# inputs that the single passes take, and what they compute in 64 bits
# ---------------------------------------------------------------------------

def _moving(g, inst):
    """Positions a little after the rest pose, so that there are velocities."""
    now = inst.hair.asset.positions.clone()
    step = torch.randn(now.shape[0], 3, generator=g, device="cuda") * 5e-4
    now[:, :3] += step * now[:, 3:]
    return now


def _sim_uniforms(inst):
    return UN.pack_sim_uniforms(inst.sim, inst.scene.model_matrix, inst.scene.sdf_bounds, inst.scene.grid_bounds, 7,
                                wind_dir=inst.wind_dir, wind_strength=inst.wind_strength(7))


def _lighting(case, g):
    """An AO texture at half resolution and a shadow map in which part of the hair is lit."""
    h, w = math.ceil(case["height"] * 0.5), math.ceil(case["width"] * 0.5)
    ao = 0.2 + 0.8 * torch.rand(h, w, generator=g, device="cuda")
    n = case["shadow"]
    coarse = torch.rand(1, 1, 16, 16, generator=g, device="cuda")
    return ao, (0.2 + 0.2 * torch.nn.functional.interpolate(coarse, (n, n), mode="bilinear")[0, 0]).contiguous()


def _ao_inputs(case, g):
    """The depth and octahedron normals of bumpy hair in front of a head: a wavy surface with thin gaps."""
    W, H = case["width"], case["height"]
    camera = UN.Camera(np.array([0.0, 0.0, 2.0]), np.zeros(3))
    scene = UN.SceneParams(width=W, height=H, camera=camera)
    uniforms = UN.pack_render_uniforms(scene, HairConfig(), 1)
    p = camera.proj(W, H).astype(np.float64)
    coarse = torch.rand(1, 1, 24, 24, generator=g, device="cuda", dtype=torch.float64)
    wave = torch.nn.functional.interpolate(coarse, (H, W), mode="bicubic")[0, 0]
    dist = 1.6 + 0.3 * wave + 0.01 * torch.rand(H, W, generator=g, device="cuda", dtype=torch.float64)
    depth = (-p[10] * dist + p[14]) / dist
    depth = torch.where(torch.rand(H, W, generator=g, device="cuda") < 0.15, torch.ones_like(depth), depth)
    normals = torch.rand(H * W, 2, generator=g, device="cuda").half().float()
    return uniforms, depth.float().reshape(-1), normals


def exact(case, seed):
    g = _generator(seed)
    if case["kind"] == "sim":
        inst = _instance({**case, "wind": 1.0}, g, case["strands"], case["points"], 64, 64)
        pos, gw = _exact_sim(inst, _moving(g, inst))
        return {"positions": pos, "density_grad_wind": gw, "density_velocity": None}
    if case["kind"] == "shading":
        inst = _instance(case, g, case["strands"], case["points"], case["width"], case["height"])
        return _exact_shading(inst, *_lighting(case, g))
    if case["kind"] == "gtao":
        return _exact_gtao(case, *_ao_inputs(case, g))
    return None  # whole frames: coverage and depth tests decide what is computed


def _f64(block, offset, count=1):
    v = torch.as_tensor(np.frombuffer(block, np.float32, count, offset).astype(np.float64), device="cuda")
    return v if count > 1 else float(v)


def _mat(block, offset):
    return _f64(block, offset, 16).view(4, 4)  # rows are the matrix's columns: v @ m applies it


def _apply(m, v):
    return torch.cat([v, torch.ones_like(v[..., :1])], -1) @ m


def _fract(x):
    return x - x.floor()


def _mix(a, b, t):
    return a * (1.0 - t) + b * t


def _sample_sdf(vol, lo, hi, p):
    D = round(vol.numel() ** (1.0 / 3.0))
    t = ((p - lo) / (hi - lo)).clamp(0.0, 1.0) * D - 0.5
    f = t.floor()
    a = t - f
    i0, i1 = f.long().clamp(0, D - 1), (f.long() + 1).clamp(0, D - 1)

    def at(x, y, z):
        return vol[(z * D + y) * D + x]

    x0, y0, z0 = i0.unbind(-1)
    x1, y1, z1 = i1.unbind(-1)
    ax, ay, az = a.unbind(-1)
    c0 = _mix(_mix(at(x0, y0, z0), at(x1, y0, z0), ax), _mix(at(x0, y1, z0), at(x1, y1, z0), ax), ay)
    c1 = _mix(_mix(at(x0, y0, z1), at(x1, y0, z1), ax), _mix(at(x0, y1, z1), at(x1, y1, z1), ax), ay)
    return _mix(c0, c1, az)


def _corners(p, lo, hi, G):
    """(node index, weights, whether the corner exists) of the eight corners of each point's grid cell."""
    q = ((p - lo) / (hi - lo)).clamp(0.0, 1.0) * (G - 1)
    mn, mx = q.floor(), q.ceil()
    for k in range(8):
        off = torch.tensor([k & 1, k >> 1 & 1, k >> 2], device="cuda", dtype=torch.float64)
        node = mn + off
        w = (1.0 - (q - node).abs()).clamp(0.0, 1.0)
        i = node.long().clamp(0, G - 1)
        yield (i[..., 2] * G + i[..., 1]) * G + i[..., 0], w, ((off == 0) | (mx > mn)).all(-1)


def _exact_sim(inst, now):
    u, S, P, G = _sim_uniforms(inst), inst.hair.asset.strands, inst.hair.asset.points_per_strand, inst.cfg.grid_dims
    off = UN.SIM_OFF
    smin, smax = _f64(u, off["sdf"], 3), _f64(u, off["sdf"] + 16, 3)
    gmin, gmax = _f64(u, off["gridData"], 3), _f64(u, off["gridData"] + 16, 3)
    wind, sphere = _f64(u, off["wind"], 4), _f64(u, off["collisionSphere"], 4)
    one = {k: _f64(u, off[k]) for k in off if k not in ("modelMatrix", "modelMatrixInv", "collisionSphere", "wind",
                                                         "sdf", "gridData", "constraintIterations", "frameIdx")}
    sdf_offset, iters = _f64(u, off["sdf"] + 28), inst.sim.constraint_iterations
    vol = inst.sdf.distances.double()
    init = inst.hair.asset.positions.double().view(S, P, 4)
    w, init = init[..., 3], init[..., :3]
    now = now.double().view(S, P, 4)[..., :3]
    # the splat of the positions at hand: velocity and density per node, in millionths
    # (the first pass sees positions that moved from the rest pose)
    dv = torch.zeros(G ** 3, 4, device="cuda", dtype=torch.float64)
    vel = (now - init).reshape(-1, 3)
    for i, cw, ok in _corners(now.reshape(-1, 3), gmin, gmax, G):
        v = torch.cat([vel * cw, cw.norm(dim=-1, keepdim=True)], -1)
        dv.index_add_(0, i[ok], (v[ok] * 1e6).trunc())
    dv = ((dv + 2.0 ** 31) % 2.0 ** 32 - 2.0 ** 31) / 1e6  # the grid holds 32-bit integers, which wrap
    # gradient and wind per node
    ax = torch.arange(G, device="cuda")
    z, y, x = torch.meshgrid(ax, ax, ax, indexing="ij")
    at = gmin + (gmax - gmin) / (G - 1) * torch.stack([x, y, z], -1).double()
    d = _sample_sdf(vol, smin, smax, at)
    trace = at - _unit(wind[:3]) * d[..., None] * one["windColisionTraceOffset"]
    behind = torch.where(_sample_sdf(vol, smin, smax, trace) < 0.0, 0.5, 1.0)
    gust = torch.where(d < 0.0, torch.zeros_like(behind), behind)
    dens = dv[:, 3].view(G, G, G)
    grad = []
    for dim in (2, 1, 0):
        diff = dens.narrow(dim, 0, G - 1) - dens.narrow(dim, 1, G - 1)
        pad = torch.zeros_like(dens.narrow(dim, 0, 1))
        grad.append(torch.cat([diff.clamp_min(0.0), pad], dim) - torch.cat([pad, (-diff).clamp_min(0.0)], dim))
    gw = torch.stack([*grad, gust], -1).view(G ** 3, 4)
    # Verlet with the grid forces
    g, v, str_, den = (torch.zeros(S, P, k, device="cuda", dtype=torch.float64) for k in (3, 3, 1, 1))
    for i, cw, ok in _corners(now, gmin, gmax, G):
        cw = cw * ok[..., None]
        n = cw.norm(dim=-1, keepdim=True)
        g, v = g + cw * gw[i][..., :3], v + cw * dv[i][..., :3]
        str_, den = str_ + n * gw[i][..., 3:], den + n * dv[i][..., 3:]
    strand = torch.arange(S, device="cuda", dtype=torch.float64)
    jitter = _fract((7 * 0.73 + one["windPhaseOffset"] * strand) * one["windStrengthFrequency"])
    jitter = 1.0 + _mix(-0.5 * one["windStrengthJitter"], 0.5 * one["windStrengthJitter"], jitter)
    cell = _mix(one["windStrengthLull"], 1.0, str_).clamp(0.0, 1.0)
    force = wind[:3] * (wind[3] * jitter[:, None, None] * cell).abs() + g * one["volumePreservation"]
    force[..., 1] -= one["gravity"]
    disp = torch.where(den > 0.0, v / den, torch.zeros_like(v))
    nxt = now + _mix(now - init, disp, one["friction"]) + force * one["deltaTime"] ** 2
    pos = _mix(init, nxt, w[..., None])
    pos[:, 0] = now[:, 0]
    # constraints
    length = inst.hair.segment_lengths.double().view(S, P)
    j = torch.arange(P, device="cuda", dtype=torch.float64)
    att = 1.0 - ((j / (P - 1) - one["globalConstrExtent"]) / one["globalConstrFade"]).clamp(0.0, 1.0)
    k_len = one["stiffnessLengthConstr"]
    k_glob, k_loc = one["stiffnessGlobalConstr"] / iters, one["stiffnessLocalConstr"] / iters
    k_coll, k_sdf = one["stiffnessCollisions"] / iters, one["stiffnessSDF"] / iters
    p, ws = list(pos.unbind(1)), [c[:, None] for c in w.unbind(1)]
    for _ in range(iters):
        for i in range(P - 1):
            t = p[i + 1] - p[i]
            c = (1.0 - length[:, i, None] / t.norm(dim=-1, keepdim=True)) * k_len / (ws[i] + ws[i + 1] + 1e-7)
            p[i], p[i + 1] = p[i] + t * c * ws[i], p[i + 1] - t * c * ws[i + 1]
        q = torch.stack(p, 1)
        q[:, 1:] += ((init - q) * w[..., None] * (k_glob * att)[:, None])[:, 1:]
        p = list(q.unbind(1))
        for i in range(max(P - 3, 0)):
            rest = (init[:, i] + init[:, i + 1] + init[:, i + 2]) / 3.0
            h0 = (rest - init[:, i + 1]).norm(dim=-1, keepdim=True)
            total = ws[i] + 2.0 * ws[i + 1] + ws[i + 2]
            hv = p[i + 1] - (p[i] + p[i + 1] + p[i + 2]) / 3.0
            delta = hv * (1.0 - h0 / hv.norm(dim=-1, keepdim=True)) * k_loc
            p[i] = p[i] + delta * (ws[i] / total * 2.0)
            p[i + 1] = p[i + 1] - delta * (ws[i + 1] / total * 4.0)
            p[i + 2] = p[i + 2] + delta * (ws[i + 2] / total * 2.0)
        for i in range(max(P - 3, 1), P):
            p[i] = p[i] + (p[i - 1] + init[:, i] - init[:, i - 1] - p[i]) * k_loc * ws[i]
        q = torch.stack(p, 1)
        away = q[:, 1:] - sphere[:3]
        dist = away.norm(dim=-1, keepdim=True)
        q[:, 1:] += away / dist * (sphere[3] - dist).clamp_min(0.0) * k_coll
        r = q[:, 3:]
        if P > 3:
            d = _sample_sdf(vol, smin, smax, r)
            eps = float(np.float32(0.0033918858971446753 * 0.1))
            slope = torch.stack([_sample_sdf(vol, smin, smax, r + eps * e) - d for e in
                                 torch.eye(3, device="cuda", dtype=torch.float64)], -1)
            inside = (d + sdf_offset < 0.0)[..., None]
            q[:, 3:] = r + torch.where(inside, _unit(slope) * -(d + sdf_offset)[..., None] * k_sdf, 0.0)
        p = list(q.unbind(1))
    return torch.cat([torch.stack(p, 1), w[..., None]], -1).view(S * P, 4), gw


def _dot(a, b):
    return (a * b).sum(-1)


def _marschner(base, material, to_light, to_camera, tangent):
    si, sr = _dot(tangent, to_light), _dot(tangent, to_camera)
    ci, cr = (1.0 - si * si).clamp_min(0.0).sqrt(), (1.0 - sr * sr).clamp_min(0.0).sqrt()

    def half(c):
        return (0.5 + 0.5 * c).clamp(0.0, 1.0).sqrt()

    def fresnel(c, f0=(1.0 - 1.55) ** 2 / (1.0 + 1.55) ** 2):
        return f0 + (1.0 - f0) * (1.0 - c) ** 5

    def lobe(alpha, beta):
        a = si + sr - alpha
        return (-a * a / (2.0 * beta * beta)).exp() / (beta * math.sqrt(2.0 * math.pi))

    cd = half(ci * cr + si * sr)
    lp, cp = to_light - tangent * si[..., None], to_camera - tangent * sr[..., None]
    cphi = _dot(lp, cp) / (lp.norm(dim=-1) * cp.norm(dim=-1) + 1e-4).sqrt()
    chalf = half(cphi)
    spec, tt, trt, shift, rough = (float(v) for v in material)
    r = spec * lobe(-2.0 * shift, rough * rough) * 0.25 * chalf * fresnel(cd)
    a = 1.0 / (1.19 / cd + 0.36 * cd)
    h = (1.0 + a * (0.6 - 0.8 * cphi)) * chalf
    through = base ** ((1.0 - h * h * a * a).sqrt() / (2.0 * cd))[..., None]
    f = fresnel(cd * (1.0 - h * h).clamp(0.0, 1.0).sqrt())
    n_tt = through * ((1.0 - f) ** 2 * (-3.65 * cphi - 3.98).exp())[..., None]
    f = fresnel(cd * 0.5)
    n_trt = base ** (0.8 / cd)[..., None] * ((1.0 - f) ** 2 * f * (17.0 * cphi - 16.78).exp())[..., None]
    return (r[..., None] + n_tt * (tt * lobe(shift, 0.5 * rough * rough))[..., None]
            + n_trt * (trt * lobe(4.0 * shift, 2.0 * rough * rough))[..., None])


def _exact_shading(inst, ao, shadow_map):
    u, off, cfg = UN.pack_render_uniforms(inst.scene, inst.cfg), UN.OFF, inst.cfg
    S, P, SP, W, H = inst.hair.asset.strands, inst.hair.asset.points_per_strand, cfg.shading_points, inst.width, inst.height
    pos = inst.hair.asset.positions.double().view(S, P, 4)[..., :3]
    tan = inst.hair.tangents.double().view(S, P, 4)[..., :3]
    # the points' places are 32-bit fractions of the strand, as the pass states them
    t32 = torch.arange(SP, device="cuda", dtype=torch.float32) / np.float32(SP)
    at = t32 * np.float32(P - 1)
    i0 = at.long().clamp(0, P - 1)
    i1 = (at.long() + 1).clamp(0, P - 1)
    t, ts = t32.double()[:, None], _fract(at).double()[:, None]
    base_o = _mix(pos[:, i0], pos[:, i1], ts)
    tan_o = _mix(_unit(pos[:, i1] - pos[:, i0]), tan[:, i1], ts)
    model = _mat(u, off["modelMatrix"])
    x, tangent = _apply(model, base_o)[..., :3], _apply(model, tan_o)[..., :3]
    clip = _apply(_mat(u, off["vpMatrix"]), x)
    ndc = clip[..., :3] / clip[..., 3:]
    px, py = W * (ndc[..., 0] * 0.5 + 0.5), H * (0.5 - ndc[..., 1] * 0.5)
    m = off["hairMaterial"]
    color0, color1 = _f64(u, m, 3), _f64(u, m + 16, 3)
    spec, shadows = _f64(u, m + 12), _f64(u, m + 28)
    tt, trt, shift, rough, rng, luma, fade = (_f64(u, m + 32 + 4 * k) for k in range(7))
    s32 = torch.arange(S, device="cuda", dtype=torch.float32)
    rnd = torch.stack([_fract(s32 * np.float32(k)) for k in (1.73, 1.17, 1.31)], -1).double()
    base = _mix(_mix(color0, color1, t), rnd[:, None].clamp(0.0, 1.0), rng)
    base = _mix(base, base * _fract(s32 / 255.0).double()[:, None, None], luma)
    to_cam = _unit(_f64(u, off["cameraPosition"], 3) - x)
    # shadow: percentage-closer filtering around the light-space position
    n, sh = shadow_map.shape[0], off["shadows"]
    ls = _apply(_mat(u, sh + 128), x)
    sx, sy, sz = ls[..., 0] * 0.5 + 0.5, 0.5 - ls[..., 1] * 0.5, ls[..., 2]
    radius, source = inst.scene.pcf_radius, _f64(u, sh + 192, 3)
    bias = (_f64(u, sh + 216) * (1.0 - _dot(tangent, _unit(source - x)))).clamp_min(0.0005)
    sm, lit = shadow_map.double(), torch.zeros_like(sx)
    for dx in range(-radius, radius + 1):
        for dy in range(-radius, radius + 1):
            a, b = (sx + dx / n) * n - 0.5, (sy + dy / n) * n - 0.5
            ia, ib = a.floor().long(), b.floor().long()
            avg = sum(sm[(ib + p).clamp(0, n - 1), (ia + q).clamp(0, n - 1)] for p in (0, 1) for q in (0, 1)) / 4.0
            lit += (sz - bias > avg).double()
    dark = lit / (2 * radius + 1) ** 2
    outside = (sz > 1.0) | (sx < 0.0) | (sx > 1.0) | (sy < 0.0) | (sy > 1.0)
    shadow = (1.0 - torch.where(outside, torch.zeros_like(dark), dark)).clamp(1.0 - shadows, 1.0)
    # ambient occlusion and the attenuation by depth
    ah, aw = ao.shape
    aov = ao.double()[(ah * py / H).trunc().long().clamp(0, ah - 1), (aw * px / W).trunc().long().clamp(0, aw - 1)]
    near, far = float(np.float32(cfg.camera_near)), float(np.float32(cfg.camera_far))

    def linear(d):
        return near * far / (far + (near - far) * d)

    z = inst.scene_depth.double().view(H, W)[py.clamp_min(0).long().clamp(0, H - 1), px.clamp_min(0).long().clamp(0, W - 1)]
    term = 1.0 - _mix(1.0, aov, _f64(u, off["ao"] + 24))
    term = (term + (linear(ndc[..., 2]) - linear(z)).abs() * fade).clamp(0.0, 1.0)
    total = torch.zeros_like(x)
    for k in ("light0", "light1", "light2"):
        to_light = _unit(_f64(u, off[k], 3) - x)
        tl = _dot(tangent, to_light)[..., None]
        fake = _unit(to_cam - tangent * _dot(to_cam, tangent)[..., None])
        scatter = (_dot(fake, to_light).clamp(0.0, 1.0) + 1.0) / (4.0 * math.pi)
        grey = _dot(base, torch.tensor([0.2126729, 0.7151522, 0.0721750], device="cuda", dtype=torch.float64))
        tint = (base / grey[..., None]) ** (1.0 - shadow)[..., None]
        diffuse = base * _mix(0.25, 1.0, tl) * base.sqrt() * scatter[..., None] * tint * tl.clamp(0.0, 1.0)
        brdf = diffuse + _marschner(base, (spec, tt, trt, shift, rough), to_light, to_cam, tangent)
        total += brdf * _f64(u, off[k] + 16, 3) * _f64(u, off[k] + 28) * (1.0 - term)[..., None]
    alpha = torch.ones(S, SP, 1, device="cuda", dtype=torch.float64)
    alpha[:, -1] = 0.0
    return torch.cat([total, alpha], -1).view(S * SP, 4)


def _exact_gtao(case, u, depth, normals):
    W, H, off = case["width"], case["height"], UN.OFF
    w, h = math.ceil(W * 0.5), math.ceil(H * 0.5)
    near, far = float(np.float32(0.01)), float(np.float32(100.0))
    inv, view = _mat(u, off["projMatrixInv"]), _mat(u, off["viewMatrix"])
    radius, direction, start, end = (_f64(u, off["ao"] + 4 * k) for k in range(4))
    ndir, nstep = (int(np.frombuffer(u, np.uint32, 1, off["ao"] + 16 + 4 * k)[0]) for k in (0, 1))
    depth = depth.double()
    i = torch.arange(w * h, device="cuda")
    px, py = (i % w).double() * 2.0 + 1.0, (i // w).double() * 2.0 + 1.0

    def reproject(x, y):
        ix, iy = x.clamp_min(0.0).long(), y.clamp_min(0.0).long()
        ok = (ix < W) & (iy < H)
        d = torch.where(ok, depth[(iy * W + ix).clamp(0, W * H - 1)], 0.0)
        c = torch.stack([x / W * 2.0 - 1.0, y / H * 2.0 - 1.0, d, torch.ones_like(d)], -1) @ inv
        return torch.stack([c[:, 0] / c[:, 3], c[:, 1] / c[:, 3], near * far / (far + (near - far) * d)], -1)

    here = reproject(px, py)
    ok = (px.long() < W) & (py.long() < H)
    oct_ = torch.where(ok[:, None], normals.double()[(py.long() * W + px.long()).clamp(0, W * H - 1)], 0.0) * 2.0 - 1.0
    n = torch.cat([oct_, 1.0 - oct_.abs().sum(-1, keepdim=True)], -1)
    t = (-n[:, 2:]).clamp(0.0, 1.0)
    n[:, :2] = torch.where(n[:, :2] >= 0.0, n[:, :2] - t, n[:, :2] + t)
    nv = _apply(view, _unit(n))[:, :3] * torch.tensor([1.0, 1.0, -1.0], device="cuda", dtype=torch.float64)
    to_cam = _unit(-here)
    size = torch.maximum(torch.full_like(px, float(nstep)), radius * here[:, 2] / far) / nstep
    # the noise is a hash of the texel: its 32-bit value is part of the pass
    x32, y32 = px.float(), py.float()
    hash_ = _fract(np.float32(52.9829189) * _fract(x32 * np.float32(0.06711056) + y32 * np.float32(0.00583715)))
    spin = math.pi * hash_.double()
    jitter = _fract((px + py) * 0.25) * size * 0.25
    total = torch.zeros_like(px)
    for k in range(ndir):
        phi = k * math.pi / ndir + direction * math.pi + spin
        dx, dy = phi.cos(), phi.sin()
        step = 1.0 + 0.25 * size + jitter
        horizon = [torch.full_like(px, -1.0), torch.full_like(px, -1.0)]
        for _ in range(nstep):
            ox, oy = (torch.where(v < 0.5, v.floor(), v.ceil()) for v in (dx * step, dy * step))
            for side, sign in ((0, 1.0), (1, -1.0)):
                ws = reproject(px + sign * ox, py + sign * oy) - here
                d2 = ws.norm(dim=-1)
                c = _dot(ws, to_cam) / d2.sqrt() - 2.0 * ((d2 - start) / (end - start)).clamp(0.0, 1.0)
                horizon[side] = torch.fmax(horizon[side], c)
            step = step + size
        h1, h2 = (v.acos() for v in horizon)
        dirv = torch.stack([dx, dy, torch.zeros_like(dx)], -1)
        bit = _unit(torch.linalg.cross(dirv, to_cam))
        tng = torch.linalg.cross(to_cam, bit)
        nx = nv - bit * _dot(nv, bit)[:, None]
        length = nx.norm(dim=-1)
        inverse = 1.0 / (length + 1e-6)
        cosxi = _dot(nx, tng) * inverse
        gamma = cosxi.acos() - math.pi / 2
        cosg, sing2 = _dot(nx, to_cam) * inverse, -2.0 * cosxi
        h1 = gamma + torch.fmax(-h1 - gamma, torch.full_like(h1, -math.pi / 2))
        h2 = gamma + torch.fmin(h2 - gamma, torch.full_like(h2, math.pi / 2))
        arc = sum(a * sing2 + cosg - (2.0 * a - gamma).cos() for a in (h1, h2))
        total += length * 0.25 * arc
    done = here[:, 2] >= 0.999 * far
    return torch.where(done, torch.zeros_like(total), total / ndir).view(h, w)
