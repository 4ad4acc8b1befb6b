// Whole frames: one pass of one instance (framePass, the launches of
// hfb_frame), and hfb_frame_batch's batched frame.
//
// A batched frame runs every pass once for all instances: each pass kind
// is one persistent launch over the "virtual blocks" (the blocks the
// single-instance kernel would launch) of every instance.  The host writes
// one prefix row per pass kind over the instances into a device table with
// the instances' pointers and uniforms; everything that changes from one
// batch to the next is data in device memory, so the kernels' launch
// parameters never change and one captured CUDA graph serves every batch of
// the context.
#include <algorithm>
#include <cstring>
#include <initializer_list>
#include <new>

#define HFB_TU 5
#include "hfb_internal.cuh"

namespace hfb {

static_assert(BATCH_GROUPS_MAX == sizeof(HfbCtx::batchStreams) / sizeof(cudaStream_t), "group stream table");

namespace {

constexpr uint32_t CLEAR_CHUNK = 65536;  // bytes cleared per virtual block

struct Range {
  unsigned char* p;
  size_t bytes;
};
struct Ranges {
  Range r[8];
  uint32_t n;
};

// Zeroes the ranges (whole words): a block per chunk of CLEAR_CHUNK bytes.
__global__ void __launch_bounds__(256) clearRangesKernel(const Ranges a) {
  uint32_t c = blockIdx.x, k = 0;
  for (; k < a.n; k++) {
    const uint32_t ch = (uint32_t)((a.r[k].bytes + CLEAR_CHUNK - 1) / CLEAR_CHUNK);
    if (c < ch) break;
    c -= ch;
  }
  if (k == a.n) return;
  const size_t off = (size_t)c * CLEAR_CHUNK;
  const size_t end = off + CLEAR_CHUNK < a.r[k].bytes ? off + CLEAR_CHUNK : a.r[k].bytes;
  unsigned char* p = a.r[k].p;
  const size_t end16 = (reinterpret_cast<uintptr_t>(p) & 15u) ? off : off + ((end - off) & ~size_t(15));
  for (size_t x = off + threadIdx.x * 16u; x < end16; x += 256u * 16u)
    *HFB_G(reinterpret_cast<uint4*>(p + x)) = make_uint4(0u, 0u, 0u, 0u);
  for (size_t x = end16 + threadIdx.x * 4u; x < end; x += 256u * 4u) *HFB_G(reinterpret_cast<uint32_t*>(p + x)) = 0u;
}

// cmdClearBeforeRender of the tiles, fine and sort passes (hairTilesPass.ts:48-52,
// hairFinePass.ts:50-55, hairTileSortPass.ts:63-68), in one launch instead of six memsets
// (about 2 us each on the frame's critical path); with `tilesPass`, the tiles pass's own
// counters too.
cudaError_t clearRasterRanges(HfbCtx* c, const HfbRasterBuffers& rb, bool tilesPass) {
  HFB_CHECK_BIND(c);
  const HfbConfig& cfg = c->cfg;
  const size_t T = (size_t)divCeil(rb.width, cfg.tileSize) * divCeil(rb.height, cfg.tileSize);
  Ranges a{};
  auto z = [&](void* p, size_t n) { a.r[a.n++] = {(unsigned char*)p, n}; };
  z(rb.tiles, T * cfg.tileDepthBins * 16);
  z(rb.segmentCountPerTile, T * 4);
  z(rb.tileSegments, 4);
  z(rb.rasterizerResult, 16 + (size_t)rb.width * rb.height * 16);
  z(rb.tileList, 4);
  z(rb.sortBuckets, (size_t)cfg.sortBuckets * 8);
  if (tilesPass) {
    const TilesScratch ts = tilesScratchLayout(rb.scratch, cfg, rb.width, rb.height, rb.maxDrawnSegments);
    z(ts.binCount, T * cfg.tileDepthBins * 4);
    z(ts.largeBins, 8);  // its count, and the scan's count of blocks
  }
  uint32_t blocks = 0;
  for (uint32_t k = 0; k < a.n; k++) blocks += (uint32_t)((a.r[k].bytes + CLEAR_CHUNK - 1) / CLEAR_CHUNK);
  clearRangesKernel<<<blocks, 256, 0, c->stream>>>(a);
  HFB_AFTER_LAUNCH(c, "clearRangesKernel");
  c->launches += 1;
  return cudaGetLastError();
}

}  // namespace

cudaError_t clearRaster(HfbCtx* c, const HfbRasterBuffers& rb) { return clearRasterRanges(c, rb, false); }

// One pass of one instance's frame (renderer.ts:171-295).  Integration
// writes positions[1 - current]; every later pass reads those new
// positions, as after HairObject.swapPositionBuffersAfterSimIntegration.
cudaError_t framePass(HfbCtx* c, HfbInstance* in, FramePass p) {
  const HfbSimUniforms& su = *in->simUniforms;
  const HfbUniforms& u = *in->uniforms;
  const HfbHairData& h = in->hair;
  const uint32_t cur = in->current;
  float* prev = in->positions[1u - cur];
  float* now = in->positions[cur];
  HfbRasterBuffers& rb = in->raster;
  switch (p) {
    case FP_GRID_PRE:
      return launchGridPreSim(c, su, in->densityVelocity, in->densityGradWind, in->sdf, in->sdfDims);
    case FP_INTEGRATE:
      if (!h.strandsCount) return cudaSuccess;
      return launchSimIntegrate(c, su, h, prev, now, in->positionsInitial, in->segmentLengths,
                                in->densityVelocity, in->densityGradWind, in->sdf, in->sdfDims);
    case FP_GRID_POST:  // after the swap: "prev" = the old positions, "now" = the new ones
      return launchGridPostSim(c, su, h, now, prev, in->densityVelocity, in->gridOrder);
    case FP_CLEAR:  // with the tiles pass's counters
      return clearRasterRanges(c, rb, true);
    case FP_TILES: {
      // the segments' projections, for this frame's fine pass
      const cudaError_t e = ensureProjCache(c, (size_t)h.strandsCount * (h.pointsPerStrand - 1u));
      if (e != cudaSuccess) return e;
      return launchTilesPass(c, u, h, prev, in->tangents, in->sceneDepth, in->strandsToRender, rb, c->projCache,
                             true);
    }
    case FP_SORT:
      return launchTileSort(c, rb);
    case FP_FINE:
      return launchFinePass(c, u, h, prev, in->tangents, in->shading, in->sceneDepth, rb, c->projCache);
    case FP_HAIR_DEPTH:
      if (!in->hairDepth) return cudaSuccess;
      return launchHairDepth(c, u, h, prev, in->tangents, in->strandsToRender, in->sceneDepth, in->hairDepth, rb);
    case FP_SHADING:
      if (!h.strandsCount) return cudaSuccess;
      return launchShading(c, u, h, prev, in->tangents,
                           in->hairDepth ? in->hairDepth : in->shadingDepth ? in->shadingDepth : in->sceneDepth,
                           in->ao, in->ao ? in->aoWidth : 0u, in->ao ? in->aoHeight : 0u, in->shadowMap,
                           in->shadowMap ? in->shadowMapSize : 0u, in->shading);
    default:
      return cudaErrorInvalidValue;
  }
}

// ---------------------------------------------------------------------------
// What a frame runs beside its main chain of passes, on the context's side
// stream: the raster clears, which wait for nothing of the frame, beside the
// simulation; once the positions are there, the hair depth (read by the shading)
// beside the tiles raster; the tile sort, which needs the raster's counts only,
// beside the lists; and the grid splat (read by the next frame) beside the lists and
// the fine pass.  The main chain alone leaves most of a GPU idle on one instance; each
// pass taken out of it shortens the frame by about its own time (the sort: frame of
// 2,000 x 16 146 -> 142 us, a tick of 6 sessions 1,209 -> 1,198 us).  The hair depth
// may not run beside the tiles and fine passes where they read what it writes: a
// frame whose hairDepth overlaps a sceneDepth keeps everything in turn on the
// caller's stream.
//
// A batch of one group does so at every size, although its persistent kernels fill the GPU
// by themselves: each pass's tail is filled by the others.  In turn against forked, from 0.5 to 121
// integration blocks per SM: ticks of 2, 6, 24 and 96 sessions 420 -> 314 us, 1,276 -> 1,155,
// 4,241 -> 4,098, 17,650 -> 17,400; 4, 16, 64 and 128 instances of the 64-instance mix 1,088 ->
// 977 us, 2,683 -> 2,535, 11,750 -> 11,560, 20,810 -> 20,600; 256 small ones 5,995 -> 5,875.
// ---------------------------------------------------------------------------
enum SideEvent : uint32_t { SE_START = 0, SE_CLEAR, SE_SIM, SE_RASTER, SE_SORT, SE_DONE };
static_assert(SE_DONE + 1 == SIDE_EVENTS, "an event each");

void sideCreate(HfbCtx* c) {
  cudaError_t e = cudaStreamCreateWithFlags(&c->sideStream, cudaStreamNonBlocking);
  for (uint32_t i = 0; i < SIDE_EVENTS && e == cudaSuccess; i++) e = cudaEventCreateWithFlags(&c->sideEvents[i], cudaEventDisableTiming);
  if (e != cudaSuccess) {
    cudaGetLastError();
    sideRelease(c);
  }
}

void sideRelease(HfbCtx* c) {
  for (cudaEvent_t& ev : c->sideEvents) {
    if (ev) cudaEventDestroy(ev);
    ev = nullptr;
  }
  if (c->sideStream) cudaStreamDestroy(c->sideStream);
  c->sideStream = nullptr;
}

// Runs f with the side stream as the context's.
template <class F>
static cudaError_t onSide(HfbCtx* c, F f) {
  const cudaStream_t caller = c->stream;
  c->stream = c->sideStream;
  const cudaError_t e = f();
  c->stream = caller;
  return e;
}

// A frame's passes: start(side), sim(main), depth(side), tiles(main, which records the
// end of its raster), sort(side), fine(main), splat(side), shade(main), with the side
// stream forked from the caller's and joined back into it, also after a failed launch.
template <class Start, class Sim, class Depth, class Tiles, class Sort, class Fine, class Splat, class Shade>
static cudaError_t forkedFrame(HfbCtx* c, Start start, Sim sim, Depth depth, Tiles tiles, Sort sort, Fine fine,
                               Splat splat, Shade shade) {
  const cudaStream_t M = c->stream, S = c->sideStream;
  const cudaEvent_t* ev = c->sideEvents;
  // `to` waits for what `from` has been given so far
  auto after = [&](SideEvent k, cudaStream_t from, cudaStream_t to) {
    const cudaError_t e = cudaEventRecord(ev[k], from);
    return e == cudaSuccess ? cudaStreamWaitEvent(to, ev[k], 0) : e;
  };
  cudaError_t e = after(SE_START, M, S);
  if (e != cudaSuccess) return e;
  e = onSide(c, start);
  if (e == cudaSuccess) e = cudaEventRecord(ev[SE_CLEAR], S);
  if (e == cudaSuccess) e = sim();
  if (e == cudaSuccess) e = after(SE_SIM, M, S);
  if (e == cudaSuccess) e = onSide(c, depth);
  if (e == cudaSuccess) e = cudaStreamWaitEvent(M, ev[SE_CLEAR], 0);
  if (e == cudaSuccess) {
    c->rasterDone = ev[SE_RASTER];
    e = tiles();
    c->rasterDone = nullptr;
  }
  if (e == cudaSuccess) e = cudaStreamWaitEvent(S, ev[SE_RASTER], 0);
  if (e == cudaSuccess) e = onSide(c, sort);
  if (e == cudaSuccess) e = after(SE_SORT, S, M);
  if (e == cudaSuccess) e = fine();
  if (e == cudaSuccess) e = onSide(c, splat);
  const cudaError_t ej = after(SE_DONE, S, M);
  if (e == cudaSuccess) e = ej;
  if (e == cudaSuccess) e = shade();
  return e;
}

// Whether [a, a + an) and [b, b + bn) share a byte.
static bool overlap(const void* a, size_t an, const void* b, size_t bn) {
  const uintptr_t x = (uintptr_t)a, y = (uintptr_t)b;
  return x < y + bn && y < x + an;
}
static size_t depthBytes(const HfbInstance& in) { return (size_t)in.raster.width * in.raster.height * 4; }

// Whether some instance's hairDepth overlaps some instance's sceneDepth.
static bool depthsOverlap(const HfbInstance* in, uint32_t n) {
  if (n == 1)
    return in->hairDepth && overlap(in->hairDepth, depthBytes(*in), in->sceneDepth, depthBytes(*in));
  struct Span {
    uintptr_t p, end;
  };
  Span* scene = new (std::nothrow) Span[n];  // sorted by start; the furthest end up to each
  if (!scene) return true;
  for (uint32_t i = 0; i < n; i++) {
    const uintptr_t p = (uintptr_t)in[i].sceneDepth;
    scene[i] = {p, p + depthBytes(in[i])};
  }
  std::sort(scene, scene + n, [](const Span& a, const Span& b) { return a.p < b.p; });
  for (uint32_t i = 1; i < n; i++) scene[i].end = std::max(scene[i].end, scene[i - 1].end);
  bool found = false;
  for (uint32_t i = 0; i < n && !found; i++) {
    if (!in[i].hairDepth) continue;
    const uintptr_t p = (uintptr_t)in[i].hairDepth, end = p + depthBytes(in[i]);
    // the sceneDepths that start before this one ends
    const Span* it = std::lower_bound(scene, scene + n, end, [](const Span& a, uintptr_t v) { return a.p < v; });
    found = it != scene && (it - 1)->end > p;
  }
  delete[] scene;
  return found;
}

cudaError_t frameOne(HfbCtx* c, HfbInstance* in) {
  auto pass = [&](FramePass p) { return framePass(c, in, p); };
  auto passes = [&](std::initializer_list<FramePass> ps) {
    cudaError_t e = cudaSuccess;
    for (FramePass p : ps)
      if (e == cudaSuccess) e = pass(p);
    return e;
  };
  // grown before the fork: growing waits for the streams
  const cudaError_t e = ensureProjCache(c, (size_t)in->hair.strandsCount * (in->hair.pointsPerStrand - 1u));
  if (e != cudaSuccess) return e;
  if (!c->sideStream || depthsOverlap(in, 1))
    return passes({FP_GRID_PRE, FP_INTEGRATE, FP_GRID_POST, FP_CLEAR, FP_TILES, FP_SORT, FP_FINE, FP_HAIR_DEPTH, FP_SHADING});
  return forkedFrame(c, [&] { return pass(FP_CLEAR); }, [&] { return passes({FP_GRID_PRE, FP_INTEGRATE}); },
                     [&] { return pass(FP_HAIR_DEPTH); }, [&] { return pass(FP_TILES); }, [&] { return pass(FP_SORT); },
                     [&] { return pass(FP_FINE); }, [&] { return pass(FP_GRID_POST); },
                     [&] { return pass(FP_SHADING); });
}

cudaError_t ensureProjCache(HfbCtx* c, size_t segments) {
  const size_t need = segments * SEG_PROJ_VEC4 * sizeof(float4);
  if (need <= c->projCacheBytes) return cudaSuccess;
  // the frames in flight may still read the old cache
  cudaError_t e = cudaStreamSynchronize(c->stream);
  for (int i = 0; i < 2 && e == cudaSuccess; i++)
    if (c->pipeStream[i]) e = cudaStreamSynchronize(c->pipeStream[i]);
  for (uint32_t g = 0; g < BATCH_GROUPS_MAX && e == cudaSuccess; g++)
    if (c->batchStreams[g]) e = cudaStreamSynchronize(c->batchStreams[g]);
  if (e != cudaSuccess) return e;
  if (c->projCache) cudaFree(c->projCache);
  c->projCache = nullptr;
  c->projCacheBytes = 0;
  const size_t bytes = need + need / 4;  // room to grow
  e = cudaMalloc(&c->projCache, bytes);
  if (e != cudaSuccess) {
    c->projCache = nullptr;
    return e;
  }
  c->projCacheBytes = bytes;
  return cudaSuccess;
}

namespace {

// What a frame clears for one instance before the raster passes: the
// reference's cmdClearBeforeRender of the tiles, fine and sort passes
// (hairTilesPass.ts:48-52, hairFinePass.ts:50-55, hairTileSortPass.ts:63-68)
// and the tiles pass's own counters.
__host__ __device__ inline uint32_t frameRanges(const HfbConfig& cfg, const BatchInst& I, Range* r) {
  const size_t TB = (size_t)I.T * cfg.tileDepthBins;
  const TilesScratch ts = tilesScratchLayout(I.scratch, cfg, I.W, I.H, I.maxDrawn);
  r[0] = {(unsigned char*)I.tiles, TB * 16};
  r[1] = {(unsigned char*)I.segCount, (size_t)I.T * 4};
  r[2] = {(unsigned char*)I.segBuf, 4};
  r[3] = {(unsigned char*)I.result, 16 + (size_t)I.W * I.H * 16};
  r[4] = {(unsigned char*)I.tileList, 4};
  r[5] = {(unsigned char*)I.sortBuckets, (size_t)cfg.sortBuckets * 8};
  r[6] = {(unsigned char*)ts.binCount, TB * 4};
  r[7] = {(unsigned char*)ts.largeBins, 4};
  return 8;
}

// clearDensityVelocityBuffer of GridPostSimPass (gridPostSimPass.ts:33-59)
__host__ __device__ inline uint32_t gridRanges(const HfbConfig& cfg, const BatchInst& I, Range* r) {
  r[0] = {(unsigned char*)I.dv, (size_t)cfg.gridDims * cfg.gridDims * cfg.gridDims * 16};
  return 1;
}

__host__ __device__ inline uint32_t clearRanges(const HfbConfig& cfg, const BatchInst& I, uint32_t kind,
                                                Range* r) {
  return kind == BK_CLEAR_FRAME ? frameRanges(cfg, I, r) : gridRanges(cfg, I, r);
}

// Zeroes chunk `local` of the instance's ranges: 16-byte stores, then words
// (every range starts 16-byte aligned and is a whole number of words).
__global__ void __launch_bounds__(256) clearBatch(BatchView b, HfbConfig cfgParam, uint32_t kind) {
  const HfbConfig cfg = cfgParam;
  const uint32_t n = b.hdr->n;
  const uint32_t* row = b.prefix + kind * (BATCH_MAX + 1);
  const uint32_t total = row[n];
  for (uint32_t v = blockIdx.x; v < total; v += gridDim.x) {
    const uint32_t i = batchFind(row, n, v);
    const BatchInst& I = b.insts[i];
    Range r[8];
    const uint32_t nr = clearRanges(cfg, I, kind, r);
    uint32_t c = v - row[i], k = 0;
    for (; k < nr; k++) {
      const uint32_t ch = (uint32_t)((r[k].bytes + CLEAR_CHUNK - 1) / CLEAR_CHUNK);
      if (c < ch) break;
      c -= ch;
    }
    if (k == nr) continue;
    const size_t off = (size_t)c * CLEAR_CHUNK;
    const size_t end = off + CLEAR_CHUNK < r[k].bytes ? off + CLEAR_CHUNK : r[k].bytes;
    unsigned char* p = r[k].p;
    const size_t end16 = off + ((end - off) & ~size_t(15));
    for (size_t x = off + threadIdx.x * 16u; x < end16; x += 256u * 16u)
      *HFB_G(reinterpret_cast<uint4*>(p + x)) = make_uint4(0u, 0u, 0u, 0u);
    for (size_t x = end16 + threadIdx.x * 4u; x < end; x += 256u * 4u) *HFB_G(reinterpret_cast<uint32_t*>(p + x)) = 0u;
  }
}

// sceneDepth -> hairDepth, chunk `local` of the instance's W*H floats; chunk
// 0 also zeroes the count of the hair depth's big-triangle list.
__global__ void __launch_bounds__(256) depthCopyBatch(BatchView b) {
  const uint32_t n = b.hdr->n;
  const uint32_t* row = b.prefix + BK_DEPTH_COPY * (BATCH_MAX + 1);
  const uint32_t total = row[n];
  for (uint32_t v = blockIdx.x; v < total; v += gridDim.x) {
    const uint32_t i = batchFind(row, n, v);
    const BatchInst& I = b.insts[i];
    const size_t bytes = (size_t)I.W * I.H * 4, off = (size_t)(v - row[i]) * CLEAR_CHUNK;
    const size_t end = off + CLEAR_CHUNK < bytes ? off + CLEAR_CHUNK : bytes;
    const unsigned char* src = (const unsigned char*)I.depth;
    unsigned char* dst = (unsigned char*)I.hairDepth;
    for (size_t x = off + threadIdx.x * 4u; x < end; x += 256u * 4u)
      *HFB_G(reinterpret_cast<uint32_t*>(dst + x)) = *HFB_G(reinterpret_cast<const uint32_t*>(src + x));
    if (v == row[i] && threadIdx.x == 0 && I.hdList) *HFB_G(I.hdList) = 0u;
  }
}

}  // namespace

cudaError_t launchBatchDepthCopy(HfbCtx* c, const BatchView& b) {
  HFB_CHECK_BIND(c);
  uint32_t& grid = c->batchGrid[BK_DEPTH_COPY];
  if (!grid) grid = c->smCount * 8u;
  depthCopyBatch<<<batchLaunchGrid(c, grid), 256, 0, c->stream>>>(b);
  HFB_AFTER_LAUNCH(c, "depthCopyBatch");
  c->launches += 1;
  return cudaGetLastError();
}

uint32_t batchBlocks(const HfbConfig& cfg, BatchKind k, const BatchInst& I) {
  const uint32_t G3 = cfg.gridDims * cfg.gridDims * cfg.gridDims;
  const uint32_t TB = I.T * cfg.tileDepthBins;
  const uint32_t nSeg = (I.strandsToRender < I.S ? I.strandsToRender : I.S) * (I.P - 1u);
  switch (k) {
    case BK_CLEAR_FRAME:
    case BK_CLEAR_GRID: {
      Range r[8];
      const uint32_t nr = clearRanges(cfg, I, k, r);
      uint32_t t = 0;
      for (uint32_t j = 0; j < nr; j++) t += (uint32_t)((r[j].bytes + CLEAR_CHUNK - 1) / CLEAR_CHUNK);
      return t;
    }
    case BK_GRID_PRE: return divCeil(G3, 256u);
    case BK_INTEGRATE: return I.S ? divCeil(I.S, I.simNB) : 0u;
    case BK_GRID_POST: return gridPostBlocks(I.S * I.P);
    case BK_RASTER: return divCeil(nSeg, TILES_RASTER_SEGS);
    case BK_SCAN: return divCeil(TB, 2048u);
    case BK_SCAN_SUMS: return 1u;
    case BK_SCATTER: {
      const uint32_t v = divCeil(nSeg, 1024u);
      return v < 1u ? 1u : (v > 256u ? 256u : v);
    }
    case BK_FINALIZE: return divCeil(TB, 32u);  // a warp takes 4 consecutive bins
    case BK_LARGE: {  // a CTA per bin of more than 1,024 records: more segments, more such bins
      const uint32_t v = divCeil(nSeg, 32768u);
      return v < 4u ? 4u : (v > 64u ? 64u : v);
    }
    case BK_SORT: return 1u;
    case BK_SCHEDULE: return 1u;
    case BK_SHADING: return divCeil(I.S * cfg.shadingPoints, 128u);
    case BK_DEPTH_COPY: return I.hairDepth ? divCeil((uint32_t)(((size_t)I.W * I.H * 4 + CLEAR_CHUNK - 1) / CLEAR_CHUNK), 1u) : 0u;
    case BK_HAIR_DEPTH: return I.hairDepth && I.P > 1u ? hairDepthBlocks(I.S * I.P) : 0u;
    default: return 0u;
  }
}

cudaError_t launchBatchClear(HfbCtx* c, const BatchView& b, BatchKind k) {
  HFB_CHECK_BIND(c);
  uint32_t& grid = c->batchGrid[k];
  if (!grid) grid = c->smCount * 8u;
  clearBatch<<<batchLaunchGrid(c, grid), 256, 0, c->stream>>>(b, c->cfg, (uint32_t)k);
  HFB_AFTER_LAUNCH(c, "clearBatch");
  c->launches += 1;
  return cudaGetLastError();
}

// The frame's launch sequence (renderer.ts:171-295 order): the simulation
// passes, then the raster passes.  With `ev`, an event is recorded before the
// first pass and after each of the HFB_FRAME_PASSES passes (grid_pre,
// integrate, grid_post with its grid clear, clear, tiles, sort, fine,
// hair_depth, shading).
static cudaError_t simSequence(HfbCtx* c, const BatchView& b, cudaEvent_t* ev = nullptr) {
  auto mark = [&](int i) { return ev ? cudaEventRecord(ev[i], c->stream) : cudaSuccess; };
  cudaError_t e = mark(0);
  if (e == cudaSuccess) e = launchBatchSim(c, b, BK_GRID_PRE);
  if (e == cudaSuccess) e = mark(1);
  if (e == cudaSuccess) e = launchBatchSim(c, b, BK_INTEGRATE);
  if (e == cudaSuccess) e = mark(2);
  if (e == cudaSuccess) e = launchBatchClear(c, b, BK_CLEAR_GRID);
  if (e == cudaSuccess) e = launchBatchSim(c, b, BK_GRID_POST);
  if (e == cudaSuccess) e = mark(3);
  return e;
}

static cudaError_t rasterSequence(HfbCtx* c, const BatchView& b, cudaEvent_t* ev = nullptr) {
  auto mark = [&](int i) { return ev ? cudaEventRecord(ev[i], c->stream) : cudaSuccess; };
  cudaError_t e = launchBatchClear(c, b, BK_CLEAR_FRAME);
  if (e == cudaSuccess) e = mark(4);
  if (e == cudaSuccess) e = launchBatchTiles(c, b);
  if (e == cudaSuccess) e = mark(5);
  if (e == cudaSuccess) e = launchBatchSort(c, b);
  if (e == cudaSuccess) e = mark(6);
  if (e == cudaSuccess) e = launchBatchFine(c, b);
  if (e == cudaSuccess) e = mark(7);
  if (e == cudaSuccess) e = launchBatchDepthCopy(c, b);
  if (e == cudaSuccess) e = launchBatchHairDepth(c, b);
  if (e == cudaSuccess) e = mark(8);
  if (e == cudaSuccess) e = launchBatchShading(c, b);
  if (e == cudaSuccess) e = mark(9);
  return e;
}

static cudaError_t batchSequence(HfbCtx* c, const BatchView& b, cudaEvent_t* ev = nullptr) {
  cudaError_t e = simSequence(c, b, ev);
  if (e == cudaSuccess) e = rasterSequence(c, b, ev);
  return e;
}

// The same passes, those that need not be in turn on the side stream.
static cudaError_t batchSequenceForked(HfbCtx* c, const BatchView& b) {
  return forkedFrame(
      c,
      [&] {
        const cudaError_t e = launchBatchClear(c, b, BK_CLEAR_FRAME);
        return e == cudaSuccess ? launchBatchDepthCopy(c, b) : e;
      },
      [&] {
        const cudaError_t e = launchBatchSim(c, b, BK_GRID_PRE);
        return e == cudaSuccess ? launchBatchSim(c, b, BK_INTEGRATE) : e;
      },
      [&] { return launchBatchHairDepth(c, b); }, [&] { return launchBatchTiles(c, b); },
      [&] { return launchBatchSort(c, b); }, [&] { return launchBatchFine(c, b); },
      [&] {
        const cudaError_t e = launchBatchClear(c, b, BK_CLEAR_GRID);
        return e == cudaSuccess ? launchBatchSim(c, b, BK_GRID_POST) : e;
      },
      [&] { return launchBatchShading(c, b); });
}

// One instance as the batched kernels read it.
static void fillInstance(const HfbConfig& cfg, const HfbInstance& s, BatchInst& I) {
  memset(&I, 0, sizeof(I));
  memcpy(&I.U, s.uniforms, sizeof(HfbUniforms));
  memcpy(&I.SU, s.simUniforms, sizeof(HfbSimUniforms));
  I.bsphere = make_float4(s.hair.boundingSphere[0], s.hair.boundingSphere[1], s.hair.boundingSphere[2],
                          s.hair.boundingSphere[3]);
  I.S = s.hair.strandsCount;
  I.P = s.hair.pointsPerStrand;
  I.strandsToRender = s.strandsToRender;
  I.sdfDims = s.sdfDims;
  I.W = s.raster.width;
  I.H = s.raster.height;
  I.maxDrawn = s.raster.maxDrawnSegments;
  I.T = divCeil(I.W, cfg.tileSize) * divCeil(I.H, cfg.tileSize);
  I.aoW = s.ao ? s.aoWidth : 0u;
  I.aoH = s.ao ? s.aoHeight : 0u;
  I.smSize = s.shadowMap ? s.shadowMapSize : 0u;
  I.posNew = (float4*)s.positions[1u - s.current];
  I.posOld = (const float4*)s.positions[s.current];
  I.initial = (const float4*)s.positionsInitial;
  I.tan = (const float4*)s.tangents;
  I.segLen = s.segmentLengths;
  I.dv = (int4*)s.densityVelocity;
  I.gw = (float4*)s.densityGradWind;
  I.sdf = s.sdf;
  I.shading = (float4*)s.shading;
  I.depth = s.sceneDepth;
  I.shadingDepth = s.hairDepth ? s.hairDepth : s.shadingDepth ? s.shadingDepth : s.sceneDepth;
  I.hairDepth = s.hairDepth;
  I.gridOrder = s.gridOrder;
  I.ao = s.ao;
  I.sm = s.shadowMap;
  I.tiles = (uint4*)s.raster.tiles;
  I.segBuf = s.raster.tileSegments;
  I.segCount = s.raster.segmentCountPerTile;
  I.sortBuckets = s.raster.sortBuckets;
  I.tileList = s.raster.tileList;
  I.result = s.raster.rasterizerResult;
  I.scratch = (unsigned char*)s.raster.scratch;
  I.scratchBytes = s.raster.scratchBytes;
  I.hdList = s.hairDepth ? hairDepthList(s.raster.scratch, s.raster.scratchBytes,
                                         rasterPassScratchBytes(cfg, I.W, I.H, s.raster.maxDrawnSegments), &I.hdCap)
                         : nullptr;
  if (!I.hdList) I.hdCap = 0;
}

// Rough GPU work of one instance's frame, for balancing the groups: the
// per-point passes and the per-pixel passes.
static double frameWork(const HfbInstance& in) {
  return (double)in.hair.strandsCount * in.hair.pointsPerStrand +
         0.25 * (double)in.raster.width * in.raster.height;
}

static cudaError_t ensureGroupStreams(HfbCtx* c) {
  cudaError_t e = cudaSuccess;
  if (!c->batchFork) e = cudaEventCreateWithFlags(&c->batchFork, cudaEventDisableTiming);
  for (uint32_t g = 0; g < BATCH_GROUPS_MAX && e == cudaSuccess; g++) {
    if (!c->batchStreams[g]) e = cudaStreamCreateWithFlags(&c->batchStreams[g], cudaStreamNonBlocking);
    if (e == cudaSuccess && !c->batchJoin[g]) e = cudaEventCreateWithFlags(&c->batchJoin[g], cudaEventDisableTiming);
  }
  return e;
}

// The launch sequence of NG groups: one group on c->stream, or each group
// on its own worker stream, forked from c->stream and joined back into it.
static cudaError_t groupsSequence(HfbCtx* c, uint32_t NG, bool side) {
  if (NG == 1) return side ? batchSequenceForked(c, batchView(c->batchDev)) : batchSequence(c, batchView(c->batchDev));
  const cudaStream_t caller = c->stream;
  cudaError_t e = cudaEventRecord(c->batchFork, caller);
  for (uint32_t g = 0; g < NG && e == cudaSuccess; g++) e = cudaStreamWaitEvent(c->batchStreams[g], c->batchFork, 0);
  if (e != cudaSuccess) return e;
  c->batchGridDiv = NG;
  for (uint32_t g = 0; g < NG && e == cudaSuccess; g++) {
    c->stream = c->batchStreams[g];
    e = batchSequence(c, batchView((char*)c->batchDev + (size_t)g * BATCH_BYTES));
  }
  c->stream = caller;
  c->batchGridDiv = 1;
  for (uint32_t g = 0; g < NG; g++) {  // also after a failed launch: the streams stay joined
    cudaError_t ej = cudaEventRecord(c->batchJoin[g], c->batchStreams[g]);
    if (ej == cudaSuccess) ej = cudaStreamWaitEvent(caller, c->batchJoin[g], 0);
    if (e == cudaSuccess) e = ej;
  }
  return e;
}

// Pipelined batches: the device table slots after the groups' tables.
static char* pipeTable(HfbCtx* c, uint32_t slot) {
  return (char*)c->batchDev + (size_t)(BATCH_GROUPS_MAX + slot) * BATCH_BYTES;
}

static cudaError_t ensurePipe(HfbCtx* c) {
  cudaError_t e = cudaSuccess;
  for (int i = 0; i < 2 && e == cudaSuccess; i++) {
    if (!c->pipeStream[i]) e = cudaStreamCreateWithFlags(&c->pipeStream[i], cudaStreamNonBlocking);
    if (e == cudaSuccess && !c->pipeSimDone[i]) e = cudaEventCreateWithFlags(&c->pipeSimDone[i], cudaEventDisableTiming);
    if (e == cudaSuccess && !c->pipeRasterDone[i])
      e = cudaEventCreateWithFlags(&c->pipeRasterDone[i], cudaEventDisableTiming);
    if (e == cudaSuccess && !c->pipeCaller[i]) e = cudaEventCreateWithFlags(&c->pipeCaller[i], cudaEventDisableTiming);
  }
  return e;
}

static void batchGraphsRelease(HfbCtx* c) {
  for (cudaGraphExec_t& g : c->batchGraph) {
    if (g) cudaGraphExecDestroy(g);
    g = nullptr;
  }
}

static void pipeGraphsRelease(HfbCtx* c) {
  for (int i = 0; i < 2; i++)
    for (int j = 0; j < 2; j++) {
      if (c->pipeGraph[i][j]) cudaGraphExecDestroy(c->pipeGraph[i][j]);
      c->pipeGraph[i][j] = nullptr;
    }
}

// One half of a pipelined frame (part 0: simulation, 1: raster) on its
// stream: plain launches for the first use of each table slot (they also set
// the kernels' attributes), then the slot's captured graph.
static cudaError_t pipePart(HfbCtx* c, uint32_t part, uint32_t slot) {
  const cudaStream_t caller = c->stream;
  c->stream = c->pipeStream[part];
  const BatchView b = batchView(pipeTable(c, slot));
  auto seq = [&]() { return part == 0u ? simSequence(c, b) : rasterSequence(c, b); };
  cudaError_t e = cudaSuccess;
#ifdef HFB_DEVICE_CHECKS
  const bool plain = true;  // the checked build waits after every launch: no capture
#else
  const bool plain = c->pipeCalls <= 2u;
#endif
  if (plain) {
    e = seq();
  } else {
    cudaGraphExec_t& ge = c->pipeGraph[slot][part];
    if (!ge) {
      cudaGraph_t gr = nullptr;
      e = cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal);
      if (e == cudaSuccess) {
        const uint64_t l0 = c->launches;
        cudaError_t el = seq();
        c->pipeGraphLaunches[slot][part] = c->launches - l0;
        c->launches = l0;
        e = cudaStreamEndCapture(c->stream, &gr);
        if (el != cudaSuccess) e = el;
        if (e == cudaSuccess) e = cudaGraphInstantiate(&ge, gr, 0);
        if (gr) cudaGraphDestroy(gr);
      }
    }
    if (e == cudaSuccess) {
      e = cudaGraphLaunch(ge, c->stream);
      c->launches += c->pipeGraphLaunches[slot][part];
    }
  }
  c->stream = caller;
  return e;
}

// Fills the staging copy (one device table per group), uploads it and runs
// the frame for n validated instances.
cudaError_t frameBatch(HfbCtx* c, HfbInstance* insts, uint32_t n, float* passMs) {
  cudaError_t e = cudaSuccess;
  constexpr size_t TABLES = (size_t)(BATCH_GROUPS_MAX + 2) * BATCH_BYTES;  // groups + two pipeline slots
  if (!c->batchDev) {
    e = cudaMalloc(&c->batchDev, TABLES);
    for (int k = 0; k < 2 && e == cudaSuccess; k++) {
      e = cudaMallocHost(&c->batchHost[k], TABLES);
      if (e == cudaSuccess) e = cudaEventCreateWithFlags(&c->batchCopied[k], cudaEventDisableTiming);
      if (e == cudaSuccess) e = cudaEventRecord(c->batchCopied[k], c->stream);
    }
    if (e == cudaSuccess) e = ensureGroupStreams(c);
    if (e != cudaSuccess) return e;
  }
  // groups: largest instance first, each to the group with the least work so
  // far (the profiling run keeps one group: its passes are timed one by one)
  const bool pipe = c->batchPipeline && !passMs;
  uint32_t NG = (passMs || pipe) ? 1u : (c->batchGroups < n ? c->batchGroups : n);
  if (NG < 1u) NG = 1u;
  uint32_t* group = new uint32_t[n];
  {
    uint32_t* order = new uint32_t[n];
    for (uint32_t i = 0; i < n; i++) order[i] = i;
    std::stable_sort(order, order + n, [&](uint32_t a, uint32_t b) { return frameWork(insts[a]) > frameWork(insts[b]); });
    double load[BATCH_GROUPS_MAX] = {};
    for (uint32_t k = 0; k < n; k++) {
      const uint32_t i = order[k];
      const uint32_t g = (uint32_t)(std::min_element(load, load + NG) - load);
      load[g] += frameWork(insts[i]);
      group[i] = g;
    }
    delete[] order;
  }
  // the staging copy is rewritten once its previous upload has been read
  const uint32_t k = c->batchFlip;
  c->batchFlip ^= 1u;
  e = cudaEventSynchronize(c->batchCopied[k]);
  if (e != cudaSuccess) { delete[] group; return e; }
  const HfbConfig& cfg = c->cfg;
  // the frame's projected segments: one region per instance, written by the
  // tiles pass and read by the fine pass
  size_t segs = 0;
  uint64_t strands = 0;
  for (uint32_t i = 0; i < n; i++) strands += insts[i].hair.strandsCount;
  for (uint32_t i = 0; i < n; i++) segs += (size_t)insts[i].hair.strandsCount * (insts[i].hair.pointsPerStrand - 1u);
  e = ensureProjCache(c, segs);
  if (e != cudaSuccess) { delete[] group; return e; }
  uint32_t ng[BATCH_GROUPS_MAX] = {};
  size_t smem = c->simBatchSmem, segOff = 0;
  for (uint32_t i = 0; i < n; i++) {
    const uint32_t g = group[i];
    char* h = (char*)c->batchHost[k] + (size_t)g * BATCH_BYTES;
    BatchInst& I = ((BatchInst*)(h + BATCH_INSTS_OFF))[ng[g]++];
    fillInstance(cfg, insts[i], I);
    I.proj = c->projCache + segOff * SEG_PROJ_VEC4;
    I.simNB = simStrandsForBatch(strands, I.P, (uint32_t)c->smCount);
    segOff += (size_t)insts[i].hair.strandsCount * (insts[i].hair.pointsPerStrand - 1u);
    const size_t sb = simSmemBytes(insts[i].hair.pointsPerStrand);
    smem = smem > sb ? smem : sb;
  }
  delete[] group;
  // the integration launch stages the longest strands of the batch: a batch
  // with longer strands than any before it re-sizes it (and the graph)
  if (smem > c->simBatchSmem) {
    c->simBatchSmem = smem;
    c->batchGrid[BK_INTEGRATE] = 0;
    e = cudaStreamSynchronize(c->stream);
    for (int i = 0; i < 2 && e == cudaSuccess; i++)
      if (c->pipeStream[i]) e = cudaStreamSynchronize(c->pipeStream[i]);
    if (e != cudaSuccess) return e;
    batchGraphsRelease(c);
    pipeGraphsRelease(c);
  }
  for (uint32_t g = 0; g < NG && e == cudaSuccess; g++) {
    char* h = (char*)c->batchHost[k] + (size_t)g * BATCH_BYTES;
    BatchHdr* hdr = (BatchHdr*)h;
    memset(hdr, 0, sizeof(*hdr));
    hdr->n = ng[g];
    uint32_t* prefix = (uint32_t*)(h + BATCH_PREFIX_OFF);
    const BatchInst* bi = (const BatchInst*)(h + BATCH_INSTS_OFF);
    for (uint32_t kind = 0; kind < BK_COUNT; kind++) {
      uint32_t* row = prefix + (size_t)kind * (BATCH_MAX + 1);
      uint32_t acc = 0;
      for (uint32_t i = 0; i < ng[g]; i++) {
        row[i] = acc;
        acc += batchBlocks(cfg, (BatchKind)kind, bi[i]);
      }
      row[ng[g]] = acc;
    }
    if (pipe) break;  // uploaded on the simulation stream below
    const size_t bytes = BATCH_INSTS_OFF + (size_t)ng[g] * sizeof(BatchInst);
    e = cudaMemcpyAsync((char*)c->batchDev + (size_t)g * BATCH_BYTES, h, bytes, cudaMemcpyHostToDevice, c->stream);
  }
  if (e != cudaSuccess) return e;
  if (pipe) {
    // Table slot k.  The frame's simulation waits for the caller's stream as
    // of the previous call (or this one, the first time) and for the raster
    // passes of the frame before the previous one, which read the table slot
    // and the position buffer this simulation writes; it runs beside the
    // previous frame's raster passes.  The raster passes wait for this
    // simulation and, on their own stream, for the previous raster passes;
    // the caller's stream waits for them.
    e = ensurePipe(c);
    if (e == cudaSuccess) e = cudaEventRecord(c->pipeCaller[k], c->stream);
    const cudaStream_t S = c->pipeStream[0], R = c->pipeStream[1];
    if (e == cudaSuccess) e = cudaStreamWaitEvent(S, c->pipeCaller[c->pipeCalls == 0 ? k : 1u - k], 0);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(S, c->pipeRasterDone[k], 0);
    const size_t bytes = BATCH_INSTS_OFF + (size_t)n * sizeof(BatchInst);
    if (e == cudaSuccess) e = cudaMemcpyAsync(pipeTable(c, k), c->batchHost[k], bytes, cudaMemcpyHostToDevice, S);
    if (e == cudaSuccess) e = cudaEventRecord(c->batchCopied[k], S);
    c->pipeCalls++;
    if (e == cudaSuccess) e = pipePart(c, 0, k);
    if (e == cudaSuccess) e = cudaEventRecord(c->pipeSimDone[k], S);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(R, c->pipeSimDone[k], 0);
    if (e == cudaSuccess) e = pipePart(c, 1, k);
    if (e == cudaSuccess) e = cudaEventRecord(c->pipeRasterDone[k], R);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(c->stream, c->pipeRasterDone[k], 0);
    if (e != cudaSuccess) return e;
    for (uint32_t i = 0; i < n; i++) insts[i].current ^= 1u;
    return cudaGetLastError();
  }
  e = cudaEventRecord(c->batchCopied[k], c->stream);
  if (e != cudaSuccess) return e;

  if (passMs) {  // one group, plain launches with an event between passes
    cudaEvent_t ev[HFB_FRAME_PASSES + 1] = {};
    for (int i = 0; i <= HFB_FRAME_PASSES && e == cudaSuccess; i++) e = cudaEventCreate(&ev[i]);
    if (e == cudaSuccess) e = batchSequence(c, batchView(c->batchDev), ev);
    if (e == cudaSuccess) e = cudaEventSynchronize(ev[HFB_FRAME_PASSES]);
    for (int i = 0; i < HFB_FRAME_PASSES && e == cudaSuccess; i++) e = cudaEventElapsedTime(&passMs[i], ev[i], ev[i + 1]);
    for (int i = 0; i <= HFB_FRAME_PASSES; i++)
      if (ev[i]) cudaEventDestroy(ev[i]);
    if (e != cudaSuccess) return e;
    for (uint32_t i = 0; i < n; i++) insts[i].current ^= 1u;
    return cudaGetLastError();
  }
#ifdef HFB_DEVICE_CHECKS
  c->batchNoGraph = true;  // the checked build waits after every launch: no capture
#endif
  const bool side = NG == 1u && c->sideStream && !depthsOverlap(insts, n);
  cudaGraphExec_t& graph = c->batchGraph[side ? 1 : 0];
  uint64_t& graphLaunches = c->batchGraphLaunches[side ? 1 : 0];
  if (!side && graph && c->batchGraphGroups != NG) {  // made for another number of groups
    e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess) return e;
    cudaGraphExecDestroy(graph);
    graph = nullptr;
  }
  if (c->batchCalls++ == 0 || c->batchNoGraph) {
    // the first batch (which also sets the kernels' attributes), or no graph: plain launches
    e = groupsSequence(c, NG, side);
  } else {
    if (!graph) {
      cudaGraph_t gr = nullptr;
      e = cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal);
      if (e != cudaSuccess) return e;
      const uint64_t l0 = c->launches;
      cudaError_t el = groupsSequence(c, NG, side);
      const uint64_t captured = c->launches - l0;
      c->launches = l0;
      e = cudaStreamEndCapture(c->stream, &gr);
      if (el != cudaSuccess) e = el;
      if (e == cudaSuccess) e = cudaGraphInstantiate(&graph, gr, 0);
      if (gr) cudaGraphDestroy(gr);
      if (e != cudaSuccess) {
        // a stream that cannot be captured (e.g. the legacy default stream): plain launches
        cudaGetLastError();
        graph = nullptr;
        c->batchNoGraph = true;
        e = groupsSequence(c, NG, side);
        if (e != cudaSuccess) return e;
        for (uint32_t i = 0; i < n; i++) insts[i].current ^= 1u;
        return cudaGetLastError();
      }
      graphLaunches = captured;
      if (!side) c->batchGraphGroups = NG;
    }
    e = cudaGraphLaunch(graph, c->stream);
    c->launches += graphLaunches;
  }
  if (e != cudaSuccess) return e;
  for (uint32_t i = 0; i < n; i++) insts[i].current ^= 1u;
  return cudaGetLastError();
}

void frameBatchRelease(HfbCtx* c) {
  pipeGraphsRelease(c);
  for (int i = 0; i < 2; i++) {
    if (c->pipeStream[i]) cudaStreamDestroy(c->pipeStream[i]);
    for (cudaEvent_t* ev : {&c->pipeSimDone[i], &c->pipeRasterDone[i], &c->pipeCaller[i]}) {
      if (*ev) cudaEventDestroy(*ev);
      *ev = nullptr;
    }
    c->pipeStream[i] = nullptr;
  }
  for (uint32_t g = 0; g < BATCH_GROUPS_MAX; g++) {
    if (c->batchJoin[g]) cudaEventDestroy(c->batchJoin[g]);
    if (c->batchStreams[g]) cudaStreamDestroy(c->batchStreams[g]);
    c->batchJoin[g] = nullptr;
    c->batchStreams[g] = nullptr;
  }
  if (c->batchFork) cudaEventDestroy(c->batchFork);
  c->batchFork = nullptr;
  batchGraphsRelease(c);
  for (int k = 0; k < 2; k++) {
    if (c->batchCopied[k]) cudaEventDestroy(c->batchCopied[k]);
    if (c->batchHost[k]) cudaFreeHost(c->batchHost[k]);
  }
  if (c->batchDev) cudaFree(c->batchDev);
  c->batchDev = nullptr;
  if (c->projCache) cudaFree(c->projCache);
  c->projCache = nullptr;
  c->projCacheBytes = 0;
}

}  // namespace hfb
