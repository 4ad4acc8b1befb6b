// Software raster passes: HairTilesPass, HairTileSortPass, HairFinePass.
//
// Reference WGSL: src/passes/swHair/hairTilesPass.wgsl.ts:70-246,
// hairTileSortPass.countTiles.wgsl.ts:21-97, hairTileSortPass.sort.wgsl.ts:35-75,
// hairFinePass.wgsl.ts:41-335 with shaderImpl/{swRasterizeHair,
// processHairSegment,reduceHairSlices,tileUtils}.wgsl.ts and the buffer
// layouts of shared/*.ts.
//
// Tiles pass = 5 kernels:
//   1. tilesRaster   a warp per 32 segments: project, bound, list the pixels of
//                    the box rows' spans, emit one (tile-bin, key) record per
//                    touched tile; the head min/max depth atomics and the
//                    per-tile counts are order independent.
//   2. binScan       exclusive prefix of the per-(tile, bin) record counts (the
//                    batched frame: two kernels).
//   3. binScatter    counting-sort scatter of the record keys into CSR order.
//   4. binFinalize   sort each (tile, bin)'s keys ascending and write the
//                    reference's linked list (head -> largest key): 8 lanes per
//                    bin of at most 8 records, a warp up to WARP_BIN, a block up
//                    to MEDIUM_BIN.
//   5. largeBins     one CTA per bin with more than MEDIUM_BIN records.
// The resulting lists are canonical: they do not depend on atomic order.
#include <cooperative_groups.h>
#include <cuda_fp16.h>
#include <type_traits>

#define HFB_TU 3
#include "hfb_internal.cuh"
#include "hfb_math.cuh"

namespace cg = cooperative_groups;

namespace hfb {
namespace {

constexpr uint32_t INVALID_PTR = 0xffffffffu;
constexpr float F_MAX_U32 = 4294967296.0f;  // f32(MAX_U32)
constexpr uint32_t SMALL_BIN = 32;
constexpr uint32_t WARP_BIN = 256;  // keys of one warp; 8 WARP_BIN >= MEDIUM_BIN words per block
constexpr uint32_t MEDIUM_BIN = 1024;
constexpr uint32_t LARGE_SMEM_KEYS = 16384;
constexpr int SCAN_PER_BLOCK = 2048;

struct TileB { uint32_t x0, y0, x1, y1; };

// getTileBoundsPx, tileUtils.wgsl.ts:43-54
__device__ __forceinline__ TileB tileBoundsPx(uint32_t W, uint32_t H, uint32_t TS, uint32_t tx, uint32_t ty) {
  return {clampu(tx * TS, 0u, W - 1u), clampu(ty * TS, 0u, H - 1u), clampu((tx + 1u) * TS, 0u, W - 1u),
          clampu((ty + 1u) * TS, 0u, H - 1u)};
}

__device__ __forceinline__ ProjSeg projectSegment(const HfbUniforms& U, const float4* __restrict__ pos,
                                                  const float4* __restrict__ tan, uint32_t P, uint32_t strand,
                                                  uint32_t seg, f2 size) {
  ProjSeg r;
  f3 cam = mk3(U.cameraPosition.x, U.cameraPosition.y, U.cameraPosition.z);
  size_t i = (size_t)strand * P + seg;
  projectHairPoint(U.modelMatrix.m, U.vpMatrix.m, cam, ld4(__ldg(HFB_G(&pos[i]))), ld4(__ldg(HFB_G(&tan[i]))), size,
                   U.fiberRadius, r.v00, r.v01, r.depthsProj.x, r.depthsProj.y);
  projectHairPoint(U.modelMatrix.m, U.vpMatrix.m, cam, ld4(__ldg(HFB_G(&pos[i + 1]))), ld4(__ldg(HFB_G(&tan[i + 1]))), size,
                   U.fiberRadius, r.v10, r.v11, r.depthsProj.z, r.depthsProj.w);
  return r;
}

__device__ __forceinline__ bool insideQuad(const ProjSeg& s, f2 p) {
  float C0 = edgeFunction(s.v01, s.v00, p);
  float C1 = edgeFunction(s.v11, s.v01, p);
  float C2 = edgeFunction(s.v10, s.v11, p);
  float C3 = edgeFunction(s.v00, s.v10, p);
  return C0 >= 0.0f && C1 >= 0.0f && C2 >= 0.0f && C3 >= 0.0f;
}

// Candidate pixels of one row of a projected segment quad.  The four edge
// functions are linear in x along a row, so the covered interval follows
// from the edge equations: x = a.x + (y - a.y) * slope per edge.  Edges with
// |slope| > 64 (nearly horizontal, ill conditioned) are skipped, which bounds
// the fp32 error of the solved x by ~0.03 px at 4096 px; a 2-pixel margin
// keeps every pixel the exact fp32 edge test accepts inside the candidate
// range -- the exact test still decides each pixel.
struct RowSpan {
  float ax[4], ay[4], slope[4];
  uint32_t lower;  // bit i: edge i bounds x from below (A > 0), else from above
  uint32_t use;    // bit i: edge i is used
  __device__ __forceinline__ void candidates(float y, uint32_t& x0, uint32_t& x1) const {
    float lo = -1e30f, hi = 1e30f;
#pragma unroll
    for (int i = 0; i < 4; i++) {
      if (!((use >> i) & 1u)) continue;
      float b = ax[i] + (y - ay[i]) * slope[i];
      if ((lower >> i) & 1u) lo = fmaxf(lo, b); else hi = fminf(hi, b);
    }
    if (!(lo <= hi + 4.0f)) { x1 = x0; return; }  // empty row (NaN-safe)
    float l = floorf(lo) - 2.0f, h = ceilf(hi) + 3.0f;
    if (l > (float)x0) x0 = (uint32_t)fminf(l, 4294967040.0f);
    if (h < (float)x1) x1 = h < 0.0f ? 0u : (uint32_t)h;
    if (x1 < x0) x1 = x0;
  }
};

__device__ __forceinline__ RowSpan makeRowSpan(const ProjSeg& s) {
  // edges in the order the test uses: v01->v00, v11->v01, v10->v11, v00->v10
  const f2 a[4] = {s.v01, s.v11, s.v10, s.v00};
  const f2 b[4] = {s.v00, s.v01, s.v11, s.v10};
  RowSpan r;
  r.lower = 0u;
  r.use = 0u;
  bool finite = true;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const float A = b[i].y - a[i].y, Bx = b[i].x - a[i].x;
    r.ax[i] = a[i].x;
    r.ay[i] = a[i].y;
    r.slope[i] = Bx / A;
    if (fabsf(A) * 64.0f >= fabsf(Bx) + 1.0f) r.use |= 1u << i;
    if (A > 0.0f) r.lower |= 1u << i;
    finite = finite && isfinite(a[i].x) && isfinite(a[i].y);
  }
  if (!finite) r.use = 0u;
  return r;
}

// Block-wide exclusive prefix (all threads call; total = block sum).
__device__ __forceinline__ uint32_t blockExclusiveScan(uint32_t v, uint32_t* warpSums, uint32_t& total) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= (uint32_t)o) x += y;
  }
  if (lane == 31) warpSums[warp] = x;
  __syncthreads();
  const uint32_t nw = blockDim.x >> 5;
  if (warp == 0) {
    uint32_t s = lane < nw ? warpSums[lane] : 0u;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t y = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= (uint32_t)o) s += y;
    }
    if (lane < nw) warpSums[lane] = s;
  }
  __syncthreads();
  total = warpSums[nw - 1];
  uint32_t warpPrefix = warp ? warpSums[warp - 1] : 0u;
  __syncthreads();
  return warpPrefix + x - v;
}

// ---------------------------------------------------------------------------
// 1. tilesRaster: HairTilesPass.main + processTile, hairTilesPass.wgsl.ts:70-238
//
// A warp takes 32 consecutive segments, one per lane, and needs no other warp:
// there is no block barrier.  The candidate pixels of a segment are its bounding
// rectangle clipped to the pixels the tiles cover ([0, W - 1) x [0, H - 1):
// getTileBoundsPx clamps the tile ends to W - 1 / H - 1), each belonging to tile
// (x / TS, y / TS).  After projecting, the warp works in rounds of as many of its
// segments as have room for their (segment, tile) accumulators:
//   R  the rectangles' rows are shared out over the lanes (the owner of row i
//      found by a search over the lanes' row counts), each narrowed to its span
//      (spanOf);
//   P  the spans' pixels are shared out over the lanes the same way: the edge
//      tests, interpolated depth, the depth test against the scene and, where the
//      bin does not follow from the depth range (binRange), the view-space depth
//      bin, folded into the (segment, tile) accumulators with shared-memory
//      atomics (min / max over an order-preserving u32 image of the depth, min of
//      the bin): the result does not depend on the order;
//   E  one lane per (segment, tile): the record, as processTile stores it
//      (:220-237).
// A segment of more tiles than there are accumulators is walked by the warp, a tile per
// lane (rasterSegmentTiles).  TR_SLOTS is the default of invalidTilesPerSegmentThreshold:
// such segments exist above it only, and have kernels of their own (WIDE).  A draw of 20,000 x 3 at 4K with 8 px tiles,
// a threshold of 1,024 and every 64th strand ten times as long: 906 us; with each such
// segment walked by its own lane 1,523, with 768 accumulators per block of four warps 1,042.
//
// Bound by issue: an fp32 projection with IEEE roots and quotients per segment,
// then what each row and each covered pixel costs.  Against edge tests of every
// rectangle pixel, four warps sharing one list between block barriers: 92 -> 58 us
// (10,000 x 32 at 1920x1080, 16 px tiles), 98 -> 64 us (11,400 x 16, 8 px tiles),
// 2.65 -> 1.58 ms (200,000 x 32 at 4K), 3.14 -> 2.43 ms (64 instances).
// ---------------------------------------------------------------------------
constexpr uint32_t TR_SEGS = TILES_RASTER_SEGS;  // segments (and threads) per block
// (segment, tile) accumulators per warp.  The raster's gathers live from L1, which is what
// shared memory leaves of the SM's 256 KB: six blocks of 31 KB, not 37 (256 slots), take the
// 64-instance frame from 12.28 to 12.06 ms; 96 the same, 64 slots 12.13 (more rounds), a
// seventh block 12.20.
constexpr uint32_t TR_SLOTS = 128;

struct TrShared {
  float4 ox[TR_SEGS], oy[TR_SEGS], ex[TR_SEGS], ey[TR_SEGS];  // edge tests (insideQuad order)
  float4 dp[TR_SEGS];                                         // depthsProj
  float4 q0[TR_SEGS], q1[TR_SEGS], q2[TR_SEGS];  // QuadConst: sm, ab | d2, lse, wS, wE | d22, QuadRecip
  float4 spanLo[TR_SEGS], spanHi[TR_SEGS];       // SpanLines in the rectangle's pixels
  float2 bin[TR_SEGS];       // depth range over which the bin follows from the depth alone
  uint4 rect[TR_SEGS];       // first column and row, width, tiles per row
  uint2 tile[TR_SEGS];       // first tile's column and row
  uint32_t slotBase[TR_SEGS];
  uint32_t accMin[TR_SEGS / 32][TR_SLOTS], accMax[TR_SEGS / 32][TR_SLOTS], accBin[TR_SEGS / 32][TR_SLOTS];
};

// order-preserving u32 image of a float (NaN excluded by the caller)
__device__ __forceinline__ uint32_t orderedBits(float f) {
  const uint32_t b = __float_as_uint(f);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float orderedFloat(uint32_t u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

// view-space depth bin of a passing pixel (:196-203, getHairDepthBoundsVS :242-246)
__device__ __forceinline__ uint32_t viewDepthBin(const HfbUniforms& U, uint32_t B, float dv0, float dv1, f2 p,
                                                 float hd) {
  const f3 vs = projectVertex(U.projMatrixInv.m, mk4(p.x, p.y, hd, 1.0f));
  return (B - 1u) - getDepthBin(B, dv0, dv1, vs.z);
}

// A (segment, tile) record keeps the smallest bin over its passing pixels.
// When the inverse projection's z row is (0, 0, m10, m14) and its w row
// (0, 0, m11, m15) -- a perspective or orthographic projection -- a pixel's
// view depth does not depend on the pixel: for x, y >= 0 the zero entries
// give signed zeros that the sums absorb, so z = m14 / RN(RN(m11 h) + m15)
// when |m10 h| stays below a quarter ulp of m14 (the z row then rounds to
// m14 exactly).  That is a monotone function of the depth h while the
// denominator keeps one sign, and getDepthBin is monotone in z (u32(NaN)
// is 0), so the smallest bin over a set of depths is the bin of its smallest
// or of its largest depth: the record needs two bins, not one per pixel.
// binRange returns the range [lo, hi] of depths over which that holds for a
// segment (empty when it does not): its four projected depths widened by
// 1e-5 of their magnitude -- the interpolated depths, mixes of the four with
// weights clamped to [0, 1], stay within 1e-6 of it -- checked on both ends.
__device__ __forceinline__ bool binRowsFromDepth(const float* M) {
  return (__float_as_uint(M[2]) << 1) == 0u && (__float_as_uint(M[6]) << 1) == 0u &&
         (__float_as_uint(M[3]) << 1) == 0u && (__float_as_uint(M[7]) << 1) == 0u && M[14] != 0.0f &&
         M[15] != 0.0f && isfinite(M[10]) && isfinite(M[11]) && isfinite(M[14]) && isfinite(M[15]);
}

__device__ __forceinline__ void binRange(const float* M, bool rows, f4 dp, float& lo, float& hi) {
  lo = __int_as_float(0x7f800000);
  hi = -lo;
  if (!rows) return;
  const float a = fminf(fminf(dp.x, dp.y), fminf(dp.z, dp.w)), b = fmaxf(fmaxf(dp.x, dp.y), fmaxf(dp.z, dp.w));
  const bool finite = isfinite(dp.x) && isfinite(dp.y) && isfinite(dp.z) && isfinite(dp.w);
  if (!finite || !(fabsf(a) < 1e30f && fabsf(b) < 1e30f)) return;
  const float m = fadd(fmul(1e-5f, fadd(fabsf(a), fabsf(b))), 1e-30f);
  const float l = fsub(a, m), h = fadd(b, m);
  if (!(fmul(fmul(fabsf(M[10]), fmaxf(fabsf(l), fabsf(h))), 1.0001f) < fmul(fabsf(M[14]), 0x1p-26f))) return;
  const float w0 = fadd(fmul(M[11], l), M[15]), w1 = fadd(fmul(M[11], h), M[15]);
  if (isfinite(w0) && isfinite(w1) && ((w0 > 0.0f && w1 > 0.0f) || (w0 < 0.0f && w1 < 0.0f))) {
    lo = l;
    hi = h;
  }
}

// Stores one (segment, tile) record, :220-237 (warp-aggregated pointer
// allocation; min / max depth as u32 maxima, order independent).
__device__ __forceinline__ void storeTileRecord(uint4* __restrict__ tiles, uint32_t* __restrict__ segBuf,
                                               uint32_t* __restrict__ segCount, uint32_t* __restrict__ binCount,
                                               DeviceCounters* __restrict__ counters, uint32_t maxDrawn,
                                               uint32_t tilesX, uint32_t B, uint32_t tx, uint32_t ty,
                                               uint32_t dbin, float dmin, float dmax, uint32_t key, uint32_t T) {
  if (!HFB_EXPECT(tx < tilesX && ty * tilesX + tx < T && dbin < B)) return;
  cg::coalesced_group g = cg::coalesced_threads();
  uint32_t base = 0;
  if (g.thread_rank() == 0) base = atomicAdd(HFB_G(&segBuf[0]), g.size());
  base = g.shfl(base, 0);
  const uint32_t ptr = base + g.thread_rank();
  if (ptr < maxDrawn) {
    const uint32_t ti = ty * tilesX * B + tx * B + dbin;
    atomicMax(HFB_G(&tiles[ti].x), f2u(fmul(fsub(1.0f, dmin), F_MAX_U32)));  // _storeTileHead
    atomicMax(HFB_G(&tiles[ti].y), f2u(fmul(dmax, F_MAX_U32)));
    atomicAdd(HFB_G(&segCount[ty * tilesX + tx]), 1u);  // _incTileSegmentCount
    atomicAdd(HFB_G(&binCount[ti]), 1u);
    // staging record in the list slot; binFinalize rewrites it
    (*HFB_G(&segBuf[1u + 2u * ptr])) = ti;
    (*HFB_G(&segBuf[2u + 2u * ptr])) = key;
  } else {
    atomicAdd(HFB_G(&counters->tileRecordsDropped), 1ull);
  }
}

// getRasterizedHairBounds, swRasterizeHair.wgsl.ts:111-124: x0, y0, x1, y1
__device__ __forceinline__ uint4 segmentBounds(const ProjSeg& s, f2 size) {
  const float bx1 = fminf(ceilf(fmaxf(fmaxf(s.v00.x, s.v01.x), fmaxf(s.v10.x, s.v11.x))), size.x);
  const float by1 = fminf(ceilf(fmaxf(fmaxf(s.v00.y, s.v01.y), fmaxf(s.v10.y, s.v11.y))), size.y);
  const float bx0 = fmaxf(floorf(fminf(fminf(s.v00.x, s.v01.x), fminf(s.v10.x, s.v11.x))), 0.0f);
  const float by0 = fmaxf(floorf(fminf(fminf(s.v00.y, s.v01.y), fminf(s.v10.y, s.v11.y))), 0.0f);
  return make_uint4(f2u(bx0), f2u(by0), f2u(bx1), f2u(by1));
}

// processTile for every tile of segment gid's tile range, by a warp: lane l takes the
// range's tiles l, l + 32, ... in row-major order.  Projects the segment again: rare, and
// the ordinary segments' rounds then have nothing of it to keep.
// Inlined: U may be a kernel parameter, whose address no function may take.
__device__ __forceinline__ void rasterSegmentTiles(const HfbUniforms& U, uint32_t P, uint32_t gid, uint32_t TS,
                                                   uint32_t B, float dv0, float dv1, uint32_t lane,
                                                   const float4* __restrict__ pos, const float4* __restrict__ tan,
                                                   const float* __restrict__ depth, uint4* __restrict__ tiles,
                                                   uint32_t* __restrict__ segBuf, uint32_t* __restrict__ segCount,
                                                   uint32_t* __restrict__ binCount,
                                                   DeviceCounters* __restrict__ counters) {
  const f2 size = mk2(U.viewport.x, U.viewport.y);
  const uint32_t W = f2u(size.x), H = f2u(size.y), tilesX = divCeil(W, TS), maxDrawn = U.maxDrawnHairSegments;
  const uint32_t strand = gid / (P - 1u), seg = gid - strand * (P - 1u), key = (strand << 8) | seg;
  const ProjSeg s = projectSegment(U, pos, tan, P, strand, seg, size);
  const uint4 u = segmentBounds(s, size);
  const uint32_t tminx = u.x / TS, tminy = u.y / TS, tsx = u.z / TS - tminx + 1u, n = tsx * (u.w / TS - tminy + 1u);
  const RowSpan span = makeRowSpan(s);
  for (uint32_t i = lane; i < n; i += 32u) {
    const uint32_t ty = tminy + i / tsx, tx = tminx + i % tsx;
    TileB tb = tileBoundsPx(W, H, TS, tx, ty);
    // Only pixel corners inside the segment's bounding rectangle can pass
    // the four edge tests, so the walk is restricted to tile x rect, and
    // per row to the candidate span around the covered interval.
    const uint32_t xa = max(tb.x0, u.x), xb = min(tb.x1, u.z + 1u);
    const uint32_t ya = max(tb.y0, u.y), yb = min(tb.y1, u.w + 1u);
    float dmin = 999.0f, dmax = -999.0f;
    uint32_t dbin = B;
    for (uint32_t y = ya; y < yb; y++) {
      uint32_t x0r = xa, x1r = xb;
      span.candidates((float)y, x0r, x1r);
      for (uint32_t x = x0r; x < x1r; x++) {
        f2 p = mk2((float)x, (float)y);
        if (!insideQuad(s, p)) continue;
        f2 w = interpolateHairQuad(s, p);
        float hd = interpolateHairF32(w, s.depthsProj);
        float zb = loadTex2DClamp(depth, W, H, (int)x, (int)H - (int)y);
        if (hd > zb) continue;  // depth test, :193-195
        dmin = fminf(dmin, hd);
        dmax = fmaxf(dmax, hd);
        dbin = min(dbin, viewDepthBin(U, B, dv0, dv1, p, hd));
      }
    }
    if (dmin > 1.0f) continue;
    storeTileRecord(tiles, segBuf, segCount, binCount, counters, maxDrawn, tilesX, B, tx, ty, dbin, dmin, dmax, key,
                    tilesX * divCeil(H, TS));
  }
}

// WIDE: the threshold lets segments of more than TR_SLOTS tiles through.
template <bool WIDE>
__device__ __forceinline__ void tilesRasterBody(const HfbUniforms& U, uint32_t P, uint32_t nStrands, uint32_t TS,
                                                uint32_t B, uint32_t threshold, float4 bsphere,
                                                const float4* __restrict__ pos, const float4* __restrict__ tan,
                                                const float* __restrict__ depth, uint4* __restrict__ tiles,
                                                uint32_t* __restrict__ segBuf, uint32_t* __restrict__ segCount,
                                                uint32_t* __restrict__ binCount,
                                                DeviceCounters* __restrict__ counters, TrShared& sh,
                                                uint32_t blk, float4* __restrict__ projOut) {
  const uint32_t tid = threadIdx.x, lane = tid & 31u, w0 = tid & ~31u;  // w0: the warp's first segment in sh
  const uint32_t segsPerStrand = P - 1u;
  const uint32_t nSeg = nStrands * segsPerStrand;
  const uint32_t gid = blk * TR_SEGS + tid;
  const f2 size = mk2(U.viewport.x, U.viewport.y);
  const uint32_t W = f2u(size.x), H = f2u(size.y);
  const uint32_t tilesX = divCeil(W, TS);
  const uint32_t maxDrawn = U.maxDrawnHairSegments;
  // getHairDepthBoundsVS, :242-246
  const f4 bsVS = m4v(U.modelViewMat.m, mk4(bsphere.x, bsphere.y, bsphere.z, 1.0f));
  const float dv0 = fsub(bsVS.z, bsphere.w), dv1 = fadd(bsVS.z, bsphere.w);
  const uint32_t tsShift = (uint32_t)(__ffs((int)TS) - 1);  // TS is 8, 16 or 32
  uint32_t* const accMin = sh.accMin[tid >> 5];
  uint32_t* const accMax = sh.accMax[tid >> 5];
  uint32_t* const accBin = sh.accBin[tid >> 5];

  // ---- project this lane's segment ----
  uint32_t rows = 0, slots = 0, key = 0;
  bool wide = false;
  if (gid < nSeg) {
    const uint32_t strand = gid / segsPerStrand, seg = gid - strand * segsPerStrand;
    key = (strand << 8) | seg;
    const ProjSeg s = projectSegment(U, pos, tan, P, strand, seg, size);
    if (projOut) {  // for the fine pass of the same frame
      float4* o = projOut + (size_t)gid * SEG_PROJ_VEC4;
      o[0] = make_float4(s.v00.x, s.v00.y, s.v01.x, s.v01.y);
      o[1] = make_float4(s.v10.x, s.v10.y, s.v11.x, s.v11.y);
      o[2] = make_float4(s.depthsProj.x, s.depthsProj.y, s.depthsProj.z, s.depthsProj.w);
    }
    const uint4 ub = segmentBounds(s, size);
    const uint32_t ux0 = ub.x, uy0 = ub.y, ux1 = ub.z, uy1 = ub.w;
    const uint32_t tminx = ux0 >> tsShift, tminy = uy0 >> tsShift, tmaxx = ux1 >> tsShift, tmaxy = uy1 >> tsShift;
    const uint32_t tsx = (tmaxx - tminx) + 1u, tsy = (tmaxy - tminy) + 1u;
    if (tsx * tsy <= threshold) {  // degenerate segment rejection, :111-117
      const uint32_t cx1 = min(ux1 + 1u, W - 1u), cy1 = min(uy1 + 1u, H - 1u);
      const uint32_t cwid = cx1 > ux0 ? cx1 - ux0 : 0u, chei = cy1 > uy0 ? cy1 - uy0 : 0u;
      if (cwid && chei) {
        if (WIDE && tsx * tsy > TR_SLOTS) {
          wide = true;  // walked by the whole warp
        } else {  // at most TR_SLOTS tiles of 32 px either way: 4,096 rows and columns
          rows = chei;
          slots = tsx * tsy;
        }
      }
      if (rows) {
        const f2 o[4] = {s.v01, s.v11, s.v10, s.v00};  // the edge tests in insideQuad's order
        const f2 d[4] = {sub2(s.v00, s.v01), sub2(s.v01, s.v11), sub2(s.v11, s.v10), sub2(s.v10, s.v00)};
        sh.ox[tid] = make_float4(o[0].x, o[1].x, o[2].x, o[3].x);
        sh.oy[tid] = make_float4(o[0].y, o[1].y, o[2].y, o[3].y);
        sh.ex[tid] = make_float4(d[0].x, d[1].x, d[2].x, d[3].x);
        sh.ey[tid] = make_float4(d[0].y, d[1].y, d[2].y, d[3].y);
        sh.dp[tid] = make_float4(s.depthsProj.x, s.depthsProj.y, s.depthsProj.z, s.depthsProj.w);
        const SpanLines sl = spanLines(o, d, (float)ux0, (float)uy0, (float)chei);
        sh.spanLo[tid] = sl.lo;
        sh.spanHi[tid] = sl.hi;
        const QuadConst q = quadConst(s);
        const QuadRecip y = quadRecip(q);
        sh.q0[tid] = make_float4(q.sm.x, q.sm.y, q.ab.x, q.ab.y);
        sh.q1[tid] = make_float4(q.d2, q.lse, q.wS, q.wE);
        sh.q2[tid] = make_float4(q.d22, y.d2, y.lse, y.d22);
        float blo, bhi;
        binRange(U.projMatrixInv.m, binRowsFromDepth(U.projMatrixInv.m), s.depthsProj, blo, bhi);
        sh.bin[tid] = make_float2(blo, bhi);
        sh.rect[tid] = make_uint4(ux0, uy0, cwid, tsx);
        sh.tile[tid] = make_uint2(tminx, tminy);
      }
    }
  }
  const uint32_t slotIncl = warpInclusive(slots, lane);

  // rounds of the lanes [first, end) whose accumulators fit together
  for (uint32_t first = 0; first < 32u;) {
    const uint32_t base = first ? __shfl_sync(0xffffffffu, slotIncl, first - 1u) : 0u;
    const uint32_t fit = __ballot_sync(0xffffffffu, lane >= first && slotIncl - base <= TR_SLOTS);
    const uint32_t end = 32u - (uint32_t)__clz((int)fit);  // slotIncl grows: the fitting lanes are first .. end - 1
    const uint32_t nSlots = __shfl_sync(0xffffffffu, slotIncl, end - 1u) - base;
    const bool mine = lane >= first && lane < end;
    const uint32_t rowIncl = warpInclusive(mine ? rows : 0u, lane);
    const uint32_t nRows = __shfl_sync(0xffffffffu, rowIncl, 31);
    if (mine) sh.slotBase[tid] = slotIncl - slots - base;
    for (uint32_t i = lane; i < nSlots; i += 32u) {
      accMin[i] = 0xffffffffu;
      accMax[i] = 0u;
      accBin[i] = B;
    }
    __syncwarp();
    for (uint32_t r0 = 0; r0 < nRows; r0 += 32u) {
      // ---- R: one row per lane ----
      const uint32_t ri = r0 + lane;
      const uint32_t ro = warpOwner(rowIncl, ri) & 31u;
      const uint32_t row = ri - __shfl_sync(0xffffffffu, rowIncl - (mine ? rows : 0u), ro);
      int xa = 0, xb = -1;
      if (ri < nRows) {
        xb = (int)sh.rect[w0 + ro].z - 1;
        spanOf(sh.spanLo[w0 + ro], sh.spanHi[w0 + ro], (float)row, xa, xb);
      }
      const uint32_t n = xb >= xa ? (uint32_t)(xb - xa + 1) : 0u;
      const uint32_t incl = warpInclusive(n, lane);
      const uint32_t nPix = __shfl_sync(0xffffffffu, incl, 31);
      const uint32_t tag = ro | (row << 5);
      const uint32_t xShift = (uint32_t)xa - (incl - n);
      // ---- P: one pixel per lane ----
      for (uint32_t c0 = 0; c0 < nPix; c0 += 32u) {
        const uint32_t c = c0 + lane;
        const uint32_t src = warpOwner(incl, c) & 31u;
        const uint32_t t = __shfl_sync(0xffffffffu, tag, src), rx = __shfl_sync(0xffffffffu, xShift, src) + c;
        if (c >= nPix) continue;
        const uint32_t k = w0 + (t & 31u);
        const uint4 rect = sh.rect[k];
        const uint32_t x = rect.x + rx, y = rect.y + (t >> 5);
        const f2 p = mk2((float)x, (float)y);
        const float4 ox = sh.ox[k], oy = sh.oy[k], ex = sh.ex[k], ey = sh.ey[k];
        // edgeFunction >= 0 (swRasterizeHair.wgsl.ts:128-130)
        const bool inside = fsub(fmul(fsub(p.x, ox.x), ey.x), fmul(fsub(p.y, oy.x), ex.x)) >= 0.0f &&
                            fsub(fmul(fsub(p.x, ox.y), ey.y), fmul(fsub(p.y, oy.y), ex.y)) >= 0.0f &&
                            fsub(fmul(fsub(p.x, ox.z), ey.z), fmul(fsub(p.y, oy.z), ex.z)) >= 0.0f &&
                            fsub(fmul(fsub(p.x, ox.w), ey.w), fmul(fsub(p.y, oy.w), ex.w)) >= 0.0f;
        if (!inside) continue;
        const float zb = loadTex2DClamp(depth, W, H, (int)x, (int)H - (int)y);
        const float4 q0 = sh.q0[k], q1 = sh.q1[k], q2 = sh.q2[k], dp = sh.dp[k];
        QuadConst qc;
        qc.sm = mk2(q0.x, q0.y);
        qc.ab = mk2(q0.z, q0.w);
        qc.d2 = q1.x; qc.lse = q1.y; qc.wS = q1.z; qc.wE = q1.w;
        qc.ab2 = mk2(ex.w, ey.w);
        qc.d22 = q2.x;
        const f2 wq = interpolateHairQuadPre(qc, {q2.y, q2.z, q2.w}, mk2(ox.w, oy.w), p);
        const float hd = interpolateHairF32(wq, ld4(dp));
        if (hd > zb) continue;  // depth test, :193-195
        const uint2 tl = sh.tile[k];
        const uint32_t slot = sh.slotBase[k] + ((y >> tsShift) - tl.y) * rect.w + ((x >> tsShift) - tl.x);
        if (!HFB_EXPECT(slot < TR_SLOTS)) continue;
        const float2 br = sh.bin[k];
        if (!(hd >= br.x && hd <= br.y))  // else the record's bin comes from its depth range (E)
          atomicMin(&accBin[slot], viewDepthBin(U, B, dv0, dv1, p, hd));
        if (!isnan(hd)) {  // fminf / fmaxf ignore a NaN depth
          atomicMin(&accMin[slot], orderedBits(hd));
          atomicMax(&accMax[slot], orderedBits(hd));
        }
      }
    }
    __syncwarp();
    // ---- E: one record per (segment, tile) that took a pixel ----
    const uint32_t slotEnd = mine ? slotIncl - base : lane < first ? 0u : nSlots;
    for (uint32_t i0 = 0; i0 < nSlots; i0 += 32u) {
      const uint32_t i = i0 + lane;
      const uint32_t so = warpOwner(slotEnd, i) & 31u;
      const uint32_t sKey = __shfl_sync(0xffffffffu, key, so);
      if (i >= nSlots || accMin[i] == 0xffffffffu) continue;  // no pixel with a depth
      const float dmin = orderedFloat(accMin[i]);
      if (dmin > 1.0f) continue;
      const uint32_t k = w0 + so, l = i - sh.slotBase[k], tsx = sh.rect[k].w;
      const uint32_t ty = sh.tile[k].y + l / tsx, tx = sh.tile[k].x + l % tsx;
      const float dmax = orderedFloat(accMax[i]);
      uint32_t bin = accBin[i];
      if (sh.bin[k].x <= sh.bin[k].y) {  // the smallest bin is at one end of the depths (binRange)
        const f2 p0 = mk2(0.0f, 0.0f);
        bin = min(bin, min(viewDepthBin(U, B, dv0, dv1, p0, dmin), viewDepthBin(U, B, dv0, dv1, p0, dmax)));
      }
      storeTileRecord(tiles, segBuf, segCount, binCount, counters, maxDrawn, tilesX, B, tx, ty, bin, dmin, dmax, sKey,
                      tilesX * divCeil(H, TS));
    }
    __syncwarp();  // the accumulators are reused by the next round
    first = end;
  }
  if constexpr (WIDE) {
    for (uint32_t m = __ballot_sync(0xffffffffu, wide); m; m &= m - 1u) {
      rasterSegmentTiles(U, P, blk * TR_SEGS + w0 + (uint32_t)__ffs(m) - 1u, TS, B, dv0, dv1, lane, pos, tan, depth,
                         tiles, segBuf, segCount, binCount, counters);
      __syncwarp();
    }
  }
}

template <bool WIDE>
__global__ void __launch_bounds__(TR_SEGS, 6)
tilesRasterKernel(const HfbUniforms U, uint32_t P, uint32_t nStrands, uint32_t TS, uint32_t B,
                  uint32_t threshold, float4 bsphere, const float4* __restrict__ pos,
                  const float4* __restrict__ tan, const float* __restrict__ depth, uint4* __restrict__ tiles,
                  uint32_t* __restrict__ segBuf, uint32_t* __restrict__ segCount,
                  uint32_t* __restrict__ binCount, DeviceCounters* __restrict__ counters, float4* __restrict__ proj) {
  __shared__ TrShared sh;
  tilesRasterBody<WIDE>(U, P, nStrands, TS, B, threshold, bsphere, pos, tan, depth, tiles, segBuf, segCount, binCount,
                        counters, sh, blockIdx.x, proj);
}

// Whether some segment can need rasterSegmentTiles.
bool rasterWide(const HfbConfig& cfg) { return cfg.invalidTilesPerSegmentThreshold > TR_SLOTS; }

// ---------------------------------------------------------------------------
// 2. binScan: exclusive prefix over T*B counts (block-local + block sums)
// ---------------------------------------------------------------------------
__device__ __forceinline__ void binScanBlocksBody(const uint32_t* __restrict__ cnt, uint32_t* __restrict__ off,
                                                  uint32_t* blockSums, uint32_t n, uint32_t* warpSums,
                                                  uint32_t blk) {
  const uint32_t base = blk * SCAN_PER_BLOCK + threadIdx.x * 4u;
  uint32_t v[4], s = 0;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    v[k] = base + k < n ? (*HFB_G(&cnt[base + k])) : 0u;
    s += v[k];
  }
  uint32_t total;
  uint32_t ex = blockExclusiveScan(s, warpSums, total);
#pragma unroll
  for (int k = 0; k < 4; k++) {
    if (base + k < n) (*HFB_G(&off[base + k])) = ex;
    ex += v[k];
  }
  if (threadIdx.x == 0) (*HFB_G(&blockSums[blk])) = total;
}

__device__ __forceinline__ void binScanSumsBody(uint32_t* blockSums, uint32_t nBlocks,
                                                uint32_t* warpSums) {
  uint32_t carry = 0;
  for (uint32_t b0 = 0; b0 < nBlocks; b0 += blockDim.x) {
    uint32_t i = b0 + threadIdx.x;
    uint32_t v = i < nBlocks ? __ldcg(HFB_G(&blockSums[i])) : 0u;  // other blocks' stores: not from L1
    uint32_t total;
    uint32_t ex = blockExclusiveScan(v, warpSums, total);
    if (i < nBlocks) (*HFB_G(&blockSums[i])) = carry + ex;
    carry += total;
  }
}

// Both in one launch: the block that finishes last scans the sums (arrived, 0 on
// entry, counts the blocks; nobody waits).  A second launch of one block took 4 us.
__global__ void __launch_bounds__(512) binScanKernel(const uint32_t* __restrict__ cnt, uint32_t* __restrict__ off,
                                                     uint32_t* blockSums, uint32_t* __restrict__ arrived, uint32_t n) {
  __shared__ uint32_t warpSums[32], last;
  binScanBlocksBody(cnt, off, blockSums, n, warpSums, blockIdx.x);
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(HFB_G(arrived), 1u) == gridDim.x - 1u;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  binScanSumsBody(blockSums, gridDim.x, warpSums);
}

// ---------------------------------------------------------------------------
// 3. binScatter: keys into CSR order (order inside a bin fixed by step 4)
// ---------------------------------------------------------------------------
__device__ __forceinline__ void binScatterBody(const uint32_t* __restrict__ segBuf, uint32_t maxDrawn,
                                               uint32_t* __restrict__ binOffset,
                                               const uint32_t* __restrict__ blockSums, uint32_t* __restrict__ keys,
                                               DeviceCounters* __restrict__ counters, uint32_t blk, uint32_t nblk,
                                               uint32_t TB) {
  const uint32_t total = (*HFB_G(&segBuf[0]));
  const uint32_t n = min(total, maxDrawn);
  if (blk == 0 && threadIdx.x == 0) atomicAdd(HFB_G(&counters->tileRecords), (unsigned long long)total);
  // The records of a warp come from a few neighbouring segments, so many fall into
  // the same bin, whose counter takes one atomic after the other: one lane adds for
  // all the lanes of its bin.  359,604 records: 18.5 -> 11 us, 7.6 million: 159 -> 105 us;
  // four records per lane in flight gave nothing.
  const uint32_t step = nblk * blockDim.x, lane = threadIdx.x & 31u;
  for (uint64_t r0 = blk * blockDim.x + (threadIdx.x - lane); r0 < n; r0 += step) {
    const uint64_t r = r0 + lane;
    uint32_t ti = r < n ? (*HFB_G(&segBuf[1u + 2u * (uint32_t)r])) : 0xffffffffu;
    const uint32_t key = r < n ? (*HFB_G(&segBuf[2u + 2u * (uint32_t)r])) : 0u;
    if (r < n && !HFB_EXPECT(ti < TB)) ti = 0xffffffffu;
    const uint32_t peers = __match_any_sync(0xffffffffu, ti);
    const uint32_t leader = __ffs(peers) - 1u;
    uint32_t pos = 0;
    if (lane == leader && ti < TB)
      pos = (*HFB_G(&blockSums[ti / SCAN_PER_BLOCK])) + atomicAdd(HFB_G(&binOffset[ti]), (uint32_t)__popc(peers));
    pos = __shfl_sync(0xffffffffu, pos, leader) + __popc(peers & ((1u << lane) - 1u));
    if (ti < TB && HFB_EXPECT(pos < maxDrawn)) (*HFB_G(&keys[pos])) = key;
  }
}

__global__ void __launch_bounds__(256)
binScatterKernel(const uint32_t* __restrict__ segBuf, uint32_t maxDrawn, uint32_t* __restrict__ binOffset,
                 const uint32_t* __restrict__ blockSums, uint32_t* __restrict__ keys,
                 DeviceCounters* __restrict__ counters, uint32_t TB) {
  binScatterBody(segBuf, maxDrawn, binOffset, blockSums, keys, counters, blockIdx.x, gridDim.x, TB);
}

// ---------------------------------------------------------------------------
// 4. binFinalize: per-bin sort + reference linked list (warp per bin)
// ---------------------------------------------------------------------------
__device__ __forceinline__ void writeList(uint32_t* __restrict__ segBuf, uint4* __restrict__ tiles, uint32_t ti,
                                          uint32_t start, uint32_t i, uint32_t n, uint32_t key) {
  // _storeTileSegment encoding: (segment << 24) | strand; next = previous
  // (smaller) key, so the walk from the head visits keys in descending order.
  uint32_t p = start + i;
  (*HFB_G(&segBuf[1u + 2u * p])) = ((key & 0xffu) << 24) | (key >> 8);
  (*HFB_G(&segBuf[2u + 2u * p])) = i == 0 ? INVALID_PTR : p - 1u;
  if (i == n - 1u) {
    (*HFB_G(&tiles[ti])).z = p + 1u;  // head pointer (+1, 0 = empty)
    (*HFB_G(&tiles[ti])).w = n;       // padding0: list length, a hint the fine pass verifies
  }
}

// Bitonic sorting network (Batcher) on N keys in shared memory, ascending, N a
// power of two >= 64.  Stage (k, j) compares the keys at x and x + j for every
// x with bit j clear, ascending where bit k of x is clear.  The stages with
// j <= 32 stay inside aligned runs of 64 keys: a warp holds such a run in
// registers (positions p and p + 32 in lane p % 32; the j = 32 exchange within
// a lane, j <= 16 across lanes by shuffles) and runs all of them between two
// passes over shared memory.

// The j <= 32 stages of the merge steps k = kFrom .. kTo (doubling) on every
// 64-key run; the caller's warps warp0, warp0 + nWarps, ... take the runs.
__device__ __forceinline__ void bitonicRuns64(uint32_t* s, uint32_t N, uint32_t kFrom, uint32_t kTo, uint32_t lane,
                                              uint32_t warp0, uint32_t nWarps) {
  for (uint32_t r = warp0; r < N / 64u; r += nWarps) {
    const uint32_t p0 = r * 64u + lane, p1 = p0 + 32u;
    uint32_t e0 = s[p0], e1 = s[p1];
    for (uint32_t k = kFrom; k <= kTo; k <<= 1) {
      uint32_t j = k >> 1;
      if (j >= 32u) {
        const bool asc = (p0 & k) == 0u;
        const uint32_t lo = min(e0, e1), hi = max(e0, e1);
        e0 = asc ? lo : hi;
        e1 = asc ? hi : lo;
        j = 16u;
      }
      for (; j > 0u; j >>= 1) {
        const uint32_t o0 = __shfl_xor_sync(0xffffffffu, e0, j), o1 = __shfl_xor_sync(0xffffffffu, e1, j);
        const bool low = (lane & j) == 0u;
        e0 = (((p0 & k) == 0u) == low) ? min(e0, o0) : max(e0, o0);
        e1 = (((p1 & k) == 0u) == low) ? min(e1, o1) : max(e1, o1);
      }
    }
    s[p0] = e0;
    s[p1] = e1;
  }
}

// Sorts s[0, N).  BLOCK: every thread of the block calls it (block barriers);
// else one warp does (warp barriers).
template <bool BLOCK>
__device__ __forceinline__ void bitonicSort(uint32_t* s, uint32_t N) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t t0 = BLOCK ? threadIdx.x : lane, nT = BLOCK ? blockDim.x : 32u;
  const uint32_t w0 = BLOCK ? threadIdx.x >> 5 : 0u, nW = BLOCK ? blockDim.x >> 5 : 1u;
  auto sync = [] { if (BLOCK) __syncthreads(); else __syncwarp(); };
  bitonicRuns64(s, N, 2u, 64u, lane, w0, nW);
  sync();
  for (uint32_t k = 128u; k <= N; k <<= 1) {
    for (uint32_t j = k >> 1; j >= 64u; j >>= 1) {
      const uint32_t lj = __ffs(j) - 1u;  // j = 2^lj
      for (uint32_t c = t0; c < N / 2u; c += nT) {
        const uint32_t a = ((c >> lj) << (lj + 1u)) | (c & (j - 1u)), b = a + j;
        const uint32_t x = s[a], y = s[b];
        if ((x > y) == ((a & k) == 0u)) { s[a] = y; s[b] = x; }
      }
      sync();
    }
    bitonicRuns64(s, N, k, k, lane, w0, nW);
    sync();
  }
}

// Bitonic sort of one key per lane across the warp, ascending.
__device__ __forceinline__ uint32_t sortWarp32(uint32_t v, uint32_t lane) {
#pragma unroll
  for (uint32_t k = 2; k <= 32; k <<= 1) {
#pragma unroll
    for (uint32_t j = k >> 1; j > 0; j >>= 1) {
      const uint32_t o = __shfl_xor_sync(0xffffffffu, v, j);
      const bool asc = (lane & k) == 0, low = (lane & j) == 0;
      v = (asc == low) ? min(v, o) : max(v, o);
    }
  }
  return v;
}

// Sorts and links bin ti of at most WARP_BIN records with the whole warp (s: WARP_BIN
// words of the warp's own).
__device__ __forceinline__ void finalizeBinWarp(uint32_t ti, uint32_t n, uint32_t start, uint32_t lane,
                                                const uint32_t* __restrict__ keys, uint32_t* __restrict__ segBuf,
                                                uint4* __restrict__ tiles, uint32_t* s) {
  if (n <= SMALL_BIN) {
    const uint32_t v = sortWarp32(lane < n ? (*HFB_G(&keys[start + lane])) : 0xffffffffu, lane);
    if (lane < n) writeList(segBuf, tiles, ti, start, lane, n, v);
  } else {
    uint32_t N = 64;
    while (N < n) N <<= 1;
    for (uint32_t i = lane; i < N; i += 32) s[i] = i < n ? (*HFB_G(&keys[start + i])) : 0xffffffffu;
    __syncwarp();
    bitonicSort<false>(s, N);
    for (uint32_t i = lane; i < n; i += 32) writeList(segBuf, tiles, ti, start, i, n, s[i]);
    __syncwarp();
  }
}

// Sorts and links bin ti of more than WARP_BIN records with the whole block (s: 8 WARP_BIN
// words), or leaves it to largeBins.  A single warp takes ~16 us for 1,024 records, which
// was the pass's tail.  All threads of the block call it.
__device__ __forceinline__ void finalizeBinBlock(uint32_t ti, uint32_t n, uint32_t start,
                                                 const uint32_t* __restrict__ keys, uint32_t* __restrict__ segBuf,
                                                 uint4* __restrict__ tiles, uint32_t* __restrict__ largeBins,
                                                 uint32_t* s) {
  if (n > MEDIUM_BIN) {
    if (threadIdx.x == 0) {
      const uint32_t slot = atomicAdd(HFB_G(&largeBins[0]), 1u);
      (*HFB_G(&largeBins[1u + slot])) = ti;
    }
    return;
  }
  uint32_t N = 64;
  while (N < n) N <<= 1;
  for (uint32_t i = threadIdx.x; i < N; i += blockDim.x) s[i] = i < n ? (*HFB_G(&keys[start + i])) : 0xffffffffu;
  __syncthreads();
  bitonicSort<true>(s, N);
  for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) writeList(segBuf, tiles, ti, start, i, n, s[i]);
  __syncthreads();
}

// Sorts a bin of at most 8 records across the 8 lanes of a group (gl: the lane
// in its group; 0xffffffff past the bin's end), ascending.  mask: the lanes
// that call it, whole groups.
__device__ __forceinline__ uint32_t sortGroup8(uint32_t v, uint32_t gl, uint32_t mask) {
#pragma unroll
  for (uint32_t k = 2; k <= 8; k <<= 1) {
#pragma unroll
    for (uint32_t j = k >> 1; j > 0; j >>= 1) {
      const uint32_t o = __shfl_xor_sync(mask, v, j);
      const bool asc = (gl & k) == 0, low = (gl & j) == 0;
      v = (asc == low) ? min(v, o) : max(v, o);
    }
  }
  return v;
}

// The warps of the grid stride over the bins (the single-instance launch: a
// fixed grid, where spreading the larger bins over every warp keeps the tail
// short).  Most bins are empty and a bin is a chain of dependent loads, so a
// warp reads 32 of its bins' counts and ends at once, one per lane; it then
// takes the bins of at most 8 records four at a time, 8 lanes each, and the
// others up to WARP_BIN one at a time, the next bins' keys on their way while these are
// sorted; the larger ones wait in a queue for the whole block.  Against a warp that
// walks its bins one by one up to 1,024 records: 1,036,800 bins, 338,890 records of at
// most 80 per bin, 77 -> 18 us; 130,560 bins, 359,604 records of at most 759, 43 -> 21 us.
__device__ __forceinline__ void binFinalizeWarpBody(uint32_t TB, const uint32_t* __restrict__ binCount,
                                                    const uint32_t* __restrict__ binOffset,
                                                    const uint32_t* __restrict__ blockSums,
                                                    uint32_t* __restrict__ keys, uint32_t* __restrict__ segBuf,
                                                    uint4* __restrict__ tiles, uint32_t* __restrict__ largeBins,
                                                    uint32_t* smem, uint32_t* queue, uint32_t blk, uint32_t nblk) {
  constexpr uint32_t ALL = 0xffffffffu;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t grp = lane >> 3, gl = lane & 7u;
  const uint32_t nw = (nblk * blockDim.x) >> 5;
  const uint32_t drawn = (*HFB_G(&segBuf[0]));
  __shared__ uint32_t nQueue;
  if (threadIdx.x == 0) nQueue = 0;
  __syncthreads();
  // a tile's bins, neighbours, go to different blocks: where they are all large, one block
  // would sort them one after the other (a draw of 7,001 x 23 with 32 px tiles: 343 -> 332
  // us; 200,000 x 32 at 4K: 6.40 -> 6.31 ms)
  for (uint64_t base = blk; base < TB; base += 32ull * nw) {  // uniform in the block
    const uint64_t at = base + (uint64_t)warp * nblk + (uint64_t)lane * nw;
    const uint32_t ti = at < TB ? (uint32_t)at : 0u;
    const uint32_t n = at < TB ? (*HFB_G(&binCount[ti])) : 0u;
    const uint32_t end = n ? (*HFB_G(&blockSums[ti / SCAN_PER_BLOCK])) + (*HFB_G(&binOffset[ti])) : 0u;  // bin end
    const bool ok = n != 0u && HFB_EXPECT(n <= end && end <= drawn);
    const uint32_t start = end - n;
    uint32_t few = __ballot_sync(ALL, ok && n <= 8u);
    uint32_t mid = __ballot_sync(ALL, ok && n > 8u && n <= SMALL_BIN);
    uint32_t big = __ballot_sync(ALL, ok && n > SMALL_BIN && n <= WARP_BIN);
    if (ok && n > WARP_BIN) {
      const uint32_t q = atomicAdd(&nQueue, 1u);  // below blockDim.x: one per lane of the block
      queue[3u * q] = ti;
      queue[3u * q + 1u] = n;
      queue[3u * q + 2u] = start;
    }
    // the next four bins of at most 8 records: this lane's bin, count, start and key
    uint32_t bT = 0, bN = 0, bS = 0, bV = ALL;
    auto nextFew = [&]() {
      uint32_t src = 0, have = 0;
#pragma unroll
      for (uint32_t g = 0; g < 4u; g++) {
        if (grp == g && few) { src = __ffs(few) - 1u; have = 1u; }
        few &= few - 1u;
      }
      bT = __shfl_sync(ALL, ti, src);
      bN = __shfl_sync(ALL, n, src) * have;
      bS = __shfl_sync(ALL, start, src);
      bV = gl < bN ? (*HFB_G(&keys[bS + gl])) : ALL;
    };
    // the next bin of 9 .. 32 records
    auto nextMid = [&]() {
      const uint32_t src = (__ffs(mid) - 1u) & 31u;
      bT = __shfl_sync(ALL, ti, src);
      bN = mid ? __shfl_sync(ALL, n, src) : 0u;
      bS = __shfl_sync(ALL, start, src);
      bV = lane < bN ? (*HFB_G(&keys[bS + lane])) : ALL;
      mid &= mid - 1u;
    };
    if (few) {
      nextFew();
      while (true) {
        const bool more = few != 0u;
        const uint32_t T0 = bT, N0 = bN, S0 = bS, V0 = bV;
        if (more) nextFew();
        const uint32_t v = sortGroup8(V0, gl, ALL);
        if (gl < N0) writeList(segBuf, tiles, T0, S0, gl, N0, v);
        if (!more) break;
      }
    }
    if (mid) {
      nextMid();
      while (true) {
        const bool more = mid != 0u;
        const uint32_t T0 = bT, N0 = bN, S0 = bS, V0 = bV;
        if (more) nextMid();
        const uint32_t v = sortWarp32(V0, lane);
        if (lane < N0) writeList(segBuf, tiles, T0, S0, lane, N0, v);
        if (!more) break;
      }
    }
    for (; big; big &= big - 1u) {
      const uint32_t src = __ffs(big) - 1u;
      finalizeBinWarp(__shfl_sync(ALL, ti, src), __shfl_sync(ALL, n, src), __shfl_sync(ALL, start, src), lane, keys,
                      segBuf, tiles, smem + warp * WARP_BIN);
    }
    __syncthreads();
    const uint32_t nq = nQueue;
    for (uint32_t q = 0; q < nq; q++)
      finalizeBinBlock(queue[3u * q], queue[3u * q + 1u], queue[3u * q + 2u], keys, segBuf, tiles, largeBins, smem);
    __syncthreads();
    if (threadIdx.x == 0) nQueue = 0;
    __syncthreads();
  }
}

// A block takes 32 consecutive bins at a time (blockDim 256: 8 warps of 4
// bins): a group of 8 lanes sorts and links a bin of at most 8 records (most
// bins), the larger ones go to a block queue that the warps then share, one
// warp per bin.  All threads of the block call it.  (The batched launch,
// whose persistent blocks take these 32-bin pieces dynamically.)
__device__ __forceinline__ void binFinalizeBody(uint32_t TB, const uint32_t* __restrict__ binCount,
                                                const uint32_t* __restrict__ binOffset,
                                                const uint32_t* __restrict__ blockSums, uint32_t* __restrict__ keys,
                                                uint32_t* __restrict__ segBuf, uint4* __restrict__ tiles,
                                                uint32_t* __restrict__ largeBins, uint32_t* smem,
                                                uint32_t blk, uint32_t nblk) {
  __shared__ uint32_t bigTi[32], bigN[32], bigEnd[32], nBig;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, nWarps = blockDim.x >> 5;
  const uint32_t grp = lane >> 3, gl = lane & 7u;  // four groups of 8 lanes
  const uint32_t perBlock = nWarps * 4u;
  const uint32_t drawn = (*HFB_G(&segBuf[0]));
  for (uint32_t bbase = blk * perBlock; bbase < TB; bbase += nblk * perBlock) {
    if (threadIdx.x == 0) nBig = 0;
    __syncthreads();
    const uint32_t tg = bbase + warp * 4u + grp;
    uint32_t ng = 0, endg = 0;
    if (tg < TB) {
      ng = (*HFB_G(&binCount[tg]));
      if (ng) endg = (*HFB_G(&blockSums[tg / SCAN_PER_BLOCK])) + (*HFB_G(&binOffset[tg]));  // bin end
    }
    const bool ok = ng != 0u && HFB_EXPECT(ng <= endg && endg <= drawn);
    const bool small = ok && ng <= 8u;
    const uint32_t smallLanes = __ballot_sync(0xffffffffu, small);
    if (small) {
      const uint32_t start = endg - ng;
      uint32_t v = gl < ng ? (*HFB_G(&keys[start + gl])) : 0xffffffffu;
      v = sortGroup8(v, gl, smallLanes);
      if (gl < ng) writeList(segBuf, tiles, tg, start, gl, ng, v);
    } else if (ok && gl == 0u) {
      const uint32_t q = atomicAdd(&nBig, 1u);  // < 32: one per group of the block
      bigTi[q] = tg;
      bigN[q] = ng;
      bigEnd[q] = endg;
    }
    __syncthreads();
    const uint32_t nb = nBig;
    for (uint32_t q = warp; q < nb; q += nWarps)
      if (bigN[q] <= WARP_BIN)
        finalizeBinWarp(bigTi[q], bigN[q], bigEnd[q] - bigN[q], lane, keys, segBuf, tiles, smem + warp * WARP_BIN);
    __syncthreads();
    for (uint32_t q = 0; q < nb; q++)  // uniform in the block
      if (bigN[q] > WARP_BIN)
        finalizeBinBlock(bigTi[q], bigN[q], bigEnd[q] - bigN[q], keys, segBuf, tiles, largeBins, smem);
    __syncthreads();  // the queue is rewritten by the next 32 bins
  }
}

__global__ void __launch_bounds__(256)
binFinalizeKernel(uint32_t TB, const uint32_t* __restrict__ binCount, const uint32_t* __restrict__ binOffset,
                  const uint32_t* __restrict__ blockSums, uint32_t* __restrict__ keys,
                  uint32_t* __restrict__ segBuf, uint4* __restrict__ tiles, uint32_t* __restrict__ largeBins) {
  __shared__ uint32_t smem[8 * WARP_BIN], queue[3 * 256];
  binFinalizeWarpBody(TB, binCount, binOffset, blockSums, keys, segBuf, tiles, largeBins, smem, queue, blockIdx.x,
                      gridDim.x);
}

// ---------------------------------------------------------------------------
// 5. largeBins: one CTA per bin with > MEDIUM_BIN records.  A bin of at most
//    LARGE_SMEM_KEYS records is bitonic-sorted in shared memory and linked
//    from there; a larger one in runs of LARGE_SMEM_KEYS, then merged pairwise
//    through the bin's own list slots (free until the final write) by rank
//    search (keys are unique).
// ---------------------------------------------------------------------------
__device__ __forceinline__ void largeBinsBody(const uint32_t* __restrict__ largeBins,
                                              const uint32_t* __restrict__ binCount,
                                              const uint32_t* __restrict__ binOffset,
                                              const uint32_t* __restrict__ blockSums, uint32_t* __restrict__ keys,
                                              uint32_t* __restrict__ segBuf, uint4* __restrict__ tiles, uint32_t* sk,
                                              uint32_t vblk, uint32_t nvblk) {
  const uint32_t nLarge = (*HFB_G(&largeBins[0]));
  for (uint32_t li = vblk; li < nLarge; li += nvblk) {
    const uint32_t ti = (*HFB_G(&largeBins[1u + li]));
    const uint32_t n = (*HFB_G(&binCount[ti]));
    const uint32_t start = (*HFB_G(&blockSums[ti / SCAN_PER_BLOCK])) + (*HFB_G(&binOffset[ti])) - n;
    if (!HFB_EXPECT(start + n <= (*HFB_G(&segBuf[0])) && n > MEDIUM_BIN)) continue;
    uint32_t* a = keys + start;
    uint32_t* tmp = segBuf + 1u + 2u * start;  // 2n free words
    // sort runs in shared memory
    for (uint32_t r0 = 0; r0 < n; r0 += LARGE_SMEM_KEYS) {
      uint32_t m = min(LARGE_SMEM_KEYS, n - r0);
      uint32_t N = 64;
      while (N < m) N <<= 1;
      for (uint32_t i = threadIdx.x; i < N; i += blockDim.x) sk[i] = i < m ? (*HFB_G(&a[r0 + i])) : 0xffffffffu;
      __syncthreads();
      bitonicSort<true>(sk, N);
      if (m == n) break;  // one run: the list is written from shared memory below
      for (uint32_t i = threadIdx.x; i < m; i += blockDim.x) (*HFB_G(&a[r0 + i])) = sk[i];
      __syncthreads();
    }
    if (n <= LARGE_SMEM_KEYS) {
      for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) writeList(segBuf, tiles, ti, start, i, n, sk[i]);
      __syncthreads();
      continue;
    }
    // merge passes (ping-pong between a and tmp)
    uint32_t* src = a;
    uint32_t* dst = tmp;
    for (uint32_t run = LARGE_SMEM_KEYS; run < n; run <<= 1) {
      for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
        uint32_t blk = i / (2u * run);
        uint32_t l0 = blk * 2u * run, l1 = min(l0 + run, n), r1 = min(l0 + 2u * run, n);
        uint32_t v = (*HFB_G(&src[i]));
        bool left = i < l1;
        uint32_t o0 = left ? l1 : l0, o1 = left ? r1 : l1;  // the other run
        uint32_t lo = o0, hi = o1;                           // count of other < v
        while (lo < hi) {
          uint32_t mid = (lo + hi) >> 1;
          if ((*HFB_G(&src[mid])) < v) lo = mid + 1; else hi = mid;
        }
        uint32_t rankOther = lo - o0;
        uint32_t rankSelf = i - (left ? l0 : l1);
        (*HFB_G(&dst[l0 + rankSelf + rankOther])) = v;
      }
      __syncthreads();
      uint32_t* t = src; src = dst; dst = t;
    }
    if (src != a) {
      for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) (*HFB_G(&a[i])) = (*HFB_G(&src[i]));
      __syncthreads();
    }
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) writeList(segBuf, tiles, ti, start, i, n, (*HFB_G(&a[i])));
    __syncthreads();
  }
}

__global__ void __launch_bounds__(1024)
largeBinsKernel(const uint32_t* __restrict__ largeBins, const uint32_t* __restrict__ binCount,
                const uint32_t* __restrict__ binOffset, const uint32_t* __restrict__ blockSums,
                uint32_t* __restrict__ keys, uint32_t* __restrict__ segBuf, uint4* __restrict__ tiles) {
  extern __shared__ uint32_t sk[];
  largeBinsBody(largeBins, binCount, binOffset, blockSums, keys, segBuf, tiles, sk, blockIdx.x, gridDim.x);
}

// ---------------------------------------------------------------------------
// HairTileSortPass (count-tiles + sort) in one CTA, stable inside a bucket.
// ---------------------------------------------------------------------------
constexpr uint32_t SORT_MAX_BUCKETS = 256;

constexpr uint32_t SORT_AHEAD = 8;  // tiles of one lane of the tile sort in flight

struct SortShared {
  uint32_t wcnt[32][SORT_MAX_BUCKETS];  // a warp's tiles per bucket, then its next place in each
  uint32_t warpSums[32];
};

// Warp w takes the w-th contiguous range of tiles, so its counts and its places
// in every bucket are its own: the block meets three times, not four times per
// 1024 tiles.  The pass is bound by the latency of one CTA: a lane has
// SORT_AHEAD tiles on the way.  32,400 tiles: 45 -> 17 us, 8,160: 14 -> 8.4 us.
__device__ __forceinline__ void tileSortBody(uint32_t T, uint32_t NB, uint32_t bucketSize,
                                             const uint32_t* __restrict__ segCount, uint32_t* __restrict__ buckets,
                                             uint32_t* __restrict__ tileList, SortShared& ss) {
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, nWarps = blockDim.x >> 5;
  uint32_t* cnt = ss.wcnt[warp];
  for (uint32_t b = lane; b < NB; b += 32u) cnt[b] = 0;
  __syncwarp();
  const uint32_t perWarp = divCeil(divCeil(T, 32u), nWarps) * 32u;
  const uint32_t t0 = min(warp * perWarp, T), t1 = min(t0 + perWarp, T);
  // calcTileSortBucket, hairTileSortPass.countTiles.wgsl.ts:37-40; NB for an empty tile
  auto load = [&](uint32_t tb, uint32_t* bucket) {
    uint32_t c[SORT_AHEAD];
#pragma unroll
    for (uint32_t k = 0; k < SORT_AHEAD; k++) {
      const uint32_t t = tb + k * 32u + lane;
      c[k] = t < t1 ? (*HFB_G(&segCount[t])) : 0u;
    }
#pragma unroll
    for (uint32_t k = 0; k < SORT_AHEAD; k++) bucket[k] = c[k] ? clampu(c[k] / bucketSize, 0u, NB - 1u) : NB;
  };
  uint32_t bk[SORT_AHEAD];
  for (uint32_t tb = t0; tb < t1; tb += 32u * SORT_AHEAD) {
    load(tb, bk);
#pragma unroll
    for (uint32_t k = 0; k < SORT_AHEAD; k++)
      if (bk[k] < NB) atomicAdd(&cnt[bk[k]], 1u);
  }
  __syncthreads();
  // calculateOffsetsForEachBucket: reverse exclusive scan, sort.wgsl.ts:68-75; thread i
  // takes bucket NB - 1 - i
  const uint32_t b = NB - 1u - tid;  // for tid < NB
  uint32_t sum = 0;
  if (tid < NB)
    for (uint32_t w = 0; w < nWarps; w++) sum += ss.wcnt[w][b];
  uint32_t drawn;
  uint32_t place = blockExclusiveScan(sum, ss.warpSums, drawn);
  if (tid < NB) {
    (*HFB_G(&buckets[2u * b])) = sum;
    (*HFB_G(&buckets[2u * b + 1u])) = sum;  // the in-bucket write counter ends at tileCount
    for (uint32_t w = 0; w < nWarps; w++) {
      const uint32_t x = ss.wcnt[w][b];
      ss.wcnt[w][b] = place;
      place += x;
    }
  }
  if (tid == 0) (*HFB_G(&tileList[0])) = drawn;
  __syncthreads();
  // the scatter, stable: a warp's tiles in order, the warps' ranges in order
  for (uint32_t tb = t0; tb < t1; tb += 32u * SORT_AHEAD) {
    load(tb, bk);
#pragma unroll
    for (uint32_t k = 0; k < SORT_AHEAD; k++) {
      const uint32_t mine = bk[k];
      if (!__any_sync(0xffffffffu, mine < NB)) continue;
      const uint32_t peers = __match_any_sync(0xffffffffu, mine);
      const uint32_t rank = __popc(peers & ((1u << lane) - 1u));
      const uint32_t at = mine < NB ? cnt[mine] + rank : T;
      if (mine < NB && HFB_EXPECT(at < T)) (*HFB_G(&tileList[1u + at])) = tb + k * 32u + lane;
      __syncwarp();
      if (mine < NB && rank == 0u) cnt[mine] = at + __popc(peers);
      __syncwarp();
    }
  }
}

__global__ void __launch_bounds__(1024)
tileSortKernel(uint32_t T, uint32_t NB, uint32_t bucketSize, const uint32_t* __restrict__ segCount,
               uint32_t* __restrict__ buckets, uint32_t* __restrict__ tileList) {
  __shared__ SortShared ss;
  tileSortBody(T, NB, bucketSize, segCount, buckets, tileList, ss);
}

// ---------------------------------------------------------------------------
// HairFinePass: persistent CTAs of TS x TS threads, one tile at a time.
//
// The tile's depth bins are processed in order (processTile per bin,
// hairFinePass.wgsl.ts:205-288).  Their lists are staged in rounds of up to
// STAGE segments -- short bins share a round, a long bin spans several -- and
// each round runs in three phases:
//   A1  one thread per (segment, row of the segment's tile-local bounding
//       box): the row's span (spanOf) without the pixels that are done; the
//       spans' pixels are listed in (segment, row, x) order through a block
//       scan of their counts;
//   A2  one thread per listed pixel: the four edge tests of
//       processHairSegment (:5-20), segment-space interpolation, the depth
//       test and the fragment colour (:21-53), rounded through f16 like
//       pack2x16float (hairSlicesDataBuffer.ts:50-63);
//   B   one thread per pixel: the pixel's fragments in list order, found
//       through a per-pixel bit mask over the round's segments and the place
//       of its row's span in the list.
// A segment covers ~4 of the ~25 pixels of its box at 1080p, so the list holds
// what the edge tests accept and little else, and the phases keep the lanes
// busy where a pixel-per-thread walk of the segments would idle most of them.
// The kernel is bound by issue and by the barriers between the phases: what
// counts is instructions per record and full rounds.  Against edge tests of every
// box pixel, with rounds cut at PAIRS box pixels: 150 -> 109 us (10,000 x 32 at
// 1920x1080, 16 px tiles), 222 -> 154 us (11,400 x 16, 8 px tiles, 8 slices), 320 ->
// 176 us (7,001 x 23 at 1361x767, 32 px), 7.2 -> 4.2 ms (200,000 x 32 at 4K).  Each slice of a pixel keeps the closed form of
// its front-to-back blend (FineSlices): fragments arrive back to front
// (descending key) and acc = f + (1 - f.a) * acc, which equals the
// reference's per-slice linked list reduced front to back
// (reduceHairSlices.wgsl.ts:9-73) -- no fragment pool in memory.
//
// The reference's fragment-pool capacity per bin (SLICE_DATA_PER_PROCESSOR_
// COUNT, processHairSegment.wgsl.ts:33-40, hairFinePass.wgsl.ts:258-264) is
// kept exactly: while an upper bound (edge-test passes) shows that a bin
// cannot fill its pool inside a round, nothing is counted; otherwise the
// round is restricted to that bin, fragments are counted per segment, and the
// segment that fills the pool keeps its first slots in pixel order, after
// which the bin stops.
// ---------------------------------------------------------------------------
constexpr uint32_t MAX_RUNS = 66;           // runs of one round: at most one per depth bin (+1)
constexpr uint32_t EMPTY_BOX = 0x0000ffffu; // x0 = y0 = 255 > x1 = y1 = 0
constexpr uint32_t RUN_ENDS = 1u << 31;
constexpr uint32_t FINE_SPLIT_MIN = 256;  // records: tiles below this are never split

template <int TS> struct FineDims;
// PAIRS: listed pixels of a round (and, in a careful part, box pixels: fineTile); ROWS:
// box rows (a few per thread); NSHADE: shading entries staged per segment; CTAS: CTAs
// per SM that fineScheduleBody shares a frame's records out over, by slices (4, 8, 16) --
// a constant, not the occupancy, so that where a tile is split, and with it the last bits
// of its pixels, does not depend on the build.  At 8 px the sizes leave room for 8 CTAs
// of the batched kernel per SM (28,160 bytes each): 3.10 ms on the 64-instance frame
// against 3.39 at 7.  The single-instance kernel, with 1,184 bytes more for its copy of the
// uniforms, has 7; 256 ROWS would give it the eighth, and the batched one nothing: draws of
// 10,000 x 32 at 1920x1080 353 -> 350 us, of 200,000 x 32 at 4K 6.41 -> 6.75 ms, frames of 11,400 x 16
// 340 -> 348 us, 16 instances in one batch 2.54 -> 2.59 ms.
template <> struct FineDims<8> {
  static constexpr uint32_t STAGE = 64, PAIRS = 768, ROWS = 512, NSHADE = 3, CTAS[3] = {8, 6, 6};
};
template <> struct FineDims<16> {
  static constexpr uint32_t STAGE = 128, PAIRS = 2048, ROWS = 2048, NSHADE = 4, CTAS[3] = {3, 2, 2};  // 96: 2-3 % slower, 160: 4 % slower
};
template <> struct FineDims<32> {
  static constexpr uint32_t STAGE = 256, PAIRS = 4096, ROWS = 4096, NSHADE = 4, CTAS[3] = {1, 1, 1};
};

// A box row's place in the round's list: the row's listed pixels (bit x), and
// the list index of the first.
template <int TS> struct FineRow {
  uint32_t v;  // pixels | first << 16
  __device__ __forceinline__ void set(uint32_t pixels, uint32_t first) { v = pixels | (first << 16); }
  __device__ __forceinline__ uint32_t pixels() const { return v & 0xffffu; }
  __device__ __forceinline__ uint32_t at(uint32_t x) const {
    return (v >> 16) + (uint32_t)__popc(v & ((1u << x) - 1u));
  }
};
template <> struct FineRow<32> {
  uint32_t p, f;
  __device__ __forceinline__ void set(uint32_t pixels, uint32_t first) { p = pixels; f = first; }
  __device__ __forceinline__ uint32_t pixels() const { return p; }
  __device__ __forceinline__ uint32_t at(uint32_t x) const { return f + (uint32_t)__popc(p & ((1u << x) - 1u)); }
};

// Shared inputs of the fine pass.
struct FineArgs {
  uint32_t S, P, B, L, SP, CAP, alphaQuadratic;
  float alphaMul;
  const float4* __restrict__ pos;
  const float4* __restrict__ tan;
  const float4* __restrict__ shading;
  const float* __restrict__ depth;
  const uint4* __restrict__ tiles;
  const uint32_t* __restrict__ segBuf;
  DeviceCounters* counters;
  const float4* __restrict__ proj;  // the tiles pass's projected segments (SEG_PROJ_VEC4 each), or NULL
};

template <int TS>
struct FineSmem {
  static constexpr uint32_t NT = TS * TS, STAGE = FineDims<TS>::STAGE, PAIRS = FineDims<TS>::PAIRS, ROWS = FineDims<TS>::ROWS;
  static_assert(PAIRS >= NT && ROWS >= TS, "any one segment fits in a round");
  static_assert(STAGE <= NT, "a thread per staged segment");
  static_assert(PAIRS <= 65536 && ROWS % NT == 0, "FineRow's first index is 16 bits; rows per thread");
  static_assert(2 * 6 * STAGE * sizeof(float) <= PAIRS * sizeof(uint2), "stagePoint's scratch fits in frag");
  static constexpr uint32_t NSHADE = FineDims<TS>::NSHADE;
  float4 shade[STAGE][NSHADE];   // the shading entries each staged segment can sample
  uint2 frag[PAIRS];             // A1: pixel | segment << 16 of a listed pixel; A2: its fragment's colour as 4 x f16
  float4 spanLo[STAGE], spanHi[STAGE];  // SpanLines in tile pixels
  float4 liveBox;                // box of the tile's pixels that are not done (x0, y0, x1, y1)
  uint8_t slice[PAIRS];          // A2: the fragment's slice
  FineRow<TS> row[ROWS];         // the box rows of the staged segments, segment after segment
  // staged segments, one array per quantity (consecutive segments in consecutive banks)
  float ox[4][STAGE], oy[4][STAGE];  // first vertex of the four edge tests: v01, v11, v10, v00
  float ex[4][STAGE], ey[4][STAGE];  // second - first vertex of each edge test
  float dp[4][STAGE];                // depthsProj
  float qsx[STAGE], qsy[STAGE], qax[STAGE], qay[STAGE], qd2[STAGE], qlse[STAGE], qws[STAGE], qwe[STAGE],
      qd22[STAGE];                   // QuadConst
  float yd2[STAGE], ylse[STAGE], yd22[STAGE];  // QuadRecip
  uint32_t enc[STAGE];               // strand | segment << 24
  uint32_t box[STAGE];               // tile-local pixel box x0 | y0 << 8 | x1 << 16 | y1 << 24
  uint32_t shadeBase[STAGE];         // first staged shading index | count << 16 | depth bin << 24
  uint32_t rowBase[STAGE + 1];       // exclusive prefix of the box heights (A1's items)
  uint32_t rowOff[STAGE];            // rowBase minus the box's first row: tile row y is row[rowOff + y]
  uint32_t cnt[STAGE];               // counted pixels (CAREFUL) or fragments (exact accounting) of each
  uint32_t pixMask[STAGE / 32][NT];  // bit k of pixel p: staged segment k left a fragment at p
  // the tile
  uint4 head[64];                    // HairTileResult per depth bin
  float td0[64], td1[64], tdY[64];   // its depth range (_getTileDepth) and the range's reciprocal (recipOf)
  uint32_t binOff[65];               // tile mode: first entry of each bin in the tile's sequence
  float zbuf[NT];
  uint32_t doneMask[NT / 32];
  // the round
  uint32_t runBin[MAX_RUNS], runOff[MAX_RUNS];
  uint16_t runK0[MAX_RUNS], runK1[MAX_RUNS];
  // tile mode: bit k set where a run with segments starts at staged segment k; the bin of the
  // j-th such run, and its list index plus k
  // (walk mode: each staged segment's place in the list)
  union {
    struct {
      uint32_t runStart[STAGE / 32], startBase[64];
      uint8_t startBin[64];
    };
    uint32_t listIdx[STAGE];
  };
  uint32_t red[32];
  // the work item's instance (written by one thread per item): read where used, so that none of
  // it stays in registers across the tile's rounds
  FineArgs args;
  uint32_t nRuns, nStaged, nSeg, passCount, segLimit, edgePasses, queueIdx, bad, tileMode, total, walkNext;
  uint32_t mode, cutSeg, cutSlots, roundFrags, e0, eLast, arrive;
  uint32_t filled;                   // bins that filled their pool
};

// Block-wide sum (all threads call; every thread gets the total).
template <int NW>
__device__ __forceinline__ uint32_t blockSum(uint32_t v, uint32_t* red, uint32_t lane, uint32_t warp) {
  const uint32_t w = __reduce_add_sync(0xffffffffu, v);
  if (lane == 0) red[warp] = w;
  __syncthreads();
  uint32_t t = 0;
#pragma unroll
  for (int i = 0; i < NW; i++) t += red[i];
  __syncthreads();
  return t;
}

// Block-wide exclusive prefix in thread order (all threads call).
template <int NW>
__device__ __forceinline__ uint32_t blockExclusive(uint32_t v, uint32_t* red, uint32_t lane, uint32_t warp) {
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= (uint32_t)o) x += y;
  }
  if (lane == 31) red[warp] = x;
  __syncthreads();
  uint32_t pre = 0;
  for (uint32_t i = 0; i < warp; i++) pre += red[i];
  __syncthreads();
  return pre + x - v;
}

// The shading entries staged segment (st, sg) can sample (tFull is
// monotonic in the segment coordinate, so they are [i0(t = 0), i1(t = 1)],
// at most NSHADE of them): loads them into sh.shade[k], returns
// first | count << 16.
template <int TS>
__device__ __forceinline__ uint32_t stageShade(FineSmem<TS>& sh, uint32_t k, uint32_t st, uint32_t sg,
                                               const float4* __restrict__ shading, uint32_t P, uint32_t SP) {
  uint32_t a0, a1, b0, b1;
  remapToIndices(SP, fadd((float)sg, 0.0f) / (float)(P - 1u), a0, a1);
  remapToIndices(SP, fadd((float)sg, 1.0f) / (float)(P - 1u), b0, b1);
  const uint32_t ne = min(b1 - a0 + 1u, FineSmem<TS>::NSHADE);
  const size_t sb = (size_t)st * SP;
  float4 v[FineSmem<TS>::NSHADE];
#pragma unroll
  for (uint32_t j = 0; j < FineSmem<TS>::NSHADE; j++)  // all in flight together
    v[j] = j < ne ? __ldg(HFB_G(&shading[sb + a0 + j])) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
  for (uint32_t j = 0; j < FineSmem<TS>::NSHADE; j++)
    if (j < ne) sh.shade[k][j] = v[j];
  return a0 | (ne << 16);
}

// Bounding box of the tile's pixels that are not done (x0, y0, x1, y1; the whole tile
// where none is left), by one warp.  Once most of a tile is opaque, the
// long lists behind it touch the few open pixels only: the rounds of a tile that carries
// on in order take 10.9 -> 9.5 us (200,000 x 32 at 4K); elsewhere it gives less than the
// 0.3 % that it costs.
template <int TS>
__device__ __forceinline__ float4 liveBoxOf(const FineSmem<TS>& sh, uint32_t lane) {
  constexpr uint32_t PER = 32u / TS;  // tile rows in a word of the mask
  constexpr uint32_t ROW = TS == 32 ? 0xffffffffu : (1u << (TS & 31)) - 1u;
  const uint32_t m = lane < TS ? ~(sh.doneMask[lane / PER] >> ((lane % PER) * TS)) & ROW : 0u;  // lane's row
  const uint32_t ys = __ballot_sync(0xffffffffu, m != 0u), xs = __reduce_or_sync(0xffffffffu, m);
  if (ys == 0u) return make_float4(0.0f, 0.0f, (float)(TS - 1), (float)(TS - 1));
  return make_float4((float)(__ffs(xs) - 1), (float)(__ffs(ys) - 1), (float)(31 - __clz(xs)), (float)(31 - __clz(ys)));
}

// Staged segment k from its projection s: edge-test constants, depths, the
// pixel-independent part of interpolateHairQuad, and the tile-local box of
// the pixels that can pass the edge tests ([floor(min), ceil(max)] of the
// vertices), within the tile's live box (liveBoxOf).  shade: first | count << 16 of its staged shading entries
// (stageShade).  Returns the box height (0: no pixel).
template <int TS>
__device__ __forceinline__ uint32_t stageFromProjection(FineSmem<TS>& sh, uint32_t k, uint32_t bin, const ProjSeg& s,
                                                        uint32_t shade, uint32_t x0, uint32_t y0) {
  uint32_t box = EMPTY_BOX, rows = 0, shadeBase = bin << 24;
  float mnx = floorf(fminf(fminf(s.v00.x, s.v01.x), fminf(s.v10.x, s.v11.x))) - (float)x0;
  float mny = floorf(fminf(fminf(s.v00.y, s.v01.y), fminf(s.v10.y, s.v11.y))) - (float)y0;
  float mxx = ceilf(fmaxf(fmaxf(s.v00.x, s.v01.x), fmaxf(s.v10.x, s.v11.x))) - (float)x0;
  float mxy = ceilf(fmaxf(fmaxf(s.v00.y, s.v01.y), fmaxf(s.v10.y, s.v11.y))) - (float)y0;
  const float4 lb = sh.liveBox;
  if (mnx <= mxx && mny <= mxy && mxx >= lb.x && mxy >= lb.y && mnx <= lb.z && mny <= lb.w) {
    const uint32_t bx0 = (uint32_t)fmaxf(mnx, lb.x), by0 = (uint32_t)fmaxf(mny, lb.y);
    const uint32_t bx1 = (uint32_t)fminf(mxx, lb.z), by1 = (uint32_t)fminf(mxy, lb.w);
    box = bx0 | (by0 << 8) | (bx1 << 16) | (by1 << 24);
    rows = by1 - by0 + 1u;
    // edge tests in the order insideQuad evaluates them
    const f2 o[4] = {s.v01, s.v11, s.v10, s.v00};
    const f2 d[4] = {sub2(s.v00, s.v01), sub2(s.v01, s.v11), sub2(s.v11, s.v10), sub2(s.v10, s.v00)};
#pragma unroll
    for (int i = 0; i < 4; i++) {
      sh.ox[i][k] = o[i].x;
      sh.oy[i][k] = o[i].y;
      sh.ex[i][k] = d[i].x;
      sh.ey[i][k] = d[i].y;
    }
    const SpanLines sl = spanLines(o, d, (float)x0, (float)y0, (float)TS);
    sh.spanLo[k] = sl.lo;
    sh.spanHi[k] = sl.hi;
    sh.dp[0][k] = s.depthsProj.x;
    sh.dp[1][k] = s.depthsProj.y;
    sh.dp[2][k] = s.depthsProj.z;
    sh.dp[3][k] = s.depthsProj.w;
    const QuadConst q = quadConst(s);
    sh.qsx[k] = q.sm.x; sh.qsy[k] = q.sm.y; sh.qax[k] = q.ab.x; sh.qay[k] = q.ab.y;
    sh.qd2[k] = q.d2; sh.qlse[k] = q.lse; sh.qws[k] = q.wS; sh.qwe[k] = q.wE; sh.qd22[k] = q.d22;
    const QuadRecip y = quadRecip(q);
    sh.yd2[k] = y.d2; sh.ylse[k] = y.lse; sh.yd22[k] = y.d22;
    shadeBase |= shade;
  }
  sh.box[k] = box;
  sh.shadeBase[k] = shadeBase;
  sh.cnt[k] = 0;
  return rows;
}

// Projects staged segment k (both points, projectSegment) and stages it.
template <int TS>
__device__ __forceinline__ uint32_t stageSegment(FineSmem<TS>& sh, uint32_t k, uint32_t bin, const HfbUniforms& U,
                                                 const float4* __restrict__ pos, const float4* __restrict__ tan,
                                                 const float4* __restrict__ shading, uint32_t S, uint32_t P,
                                                 uint32_t SP, f2 size, uint32_t x0, uint32_t y0) {
  const uint32_t st = sh.enc[k] & 0x00ffffffu, sg = sh.enc[k] >> 24;
  if (st < S && sg + 1u < P) {  // otherwise not a segment of this hair: covers no pixel
    const ProjSeg s = projectSegment(U, pos, tan, P, st, sg, size);
    return stageFromProjection<TS>(sh, k, bin, s, stageShade<TS>(sh, k, st, sg, shading, P, SP), x0, y0);
  }
  sh.box[k] = EMPTY_BOX;
  sh.shadeBase[k] = bin << 24;
  sh.cnt[k] = 0;
  return 0u;
}

// Stages segment k from its projection in the tiles pass's cache.
template <int TS>
__device__ __forceinline__ uint32_t stageCached(FineSmem<TS>& sh, uint32_t k, uint32_t bin,
                                                const float4* __restrict__ proj, const float4* __restrict__ shading,
                                                uint32_t enc, uint32_t S, uint32_t P, uint32_t SP, uint32_t x0,
                                                uint32_t y0) {
  const uint32_t st = enc & 0x00ffffffu, sg = enc >> 24;
  if (st < S && sg + 1u < P) {
    const float4* q = proj + ((size_t)st * (P - 1u) + sg) * SEG_PROJ_VEC4;
    const float4 a = __ldg(HFB_G(&q[0])), b = __ldg(HFB_G(&q[1])), d = __ldg(HFB_G(&q[2]));
    ProjSeg s;
    s.v00 = mk2(a.x, a.y);
    s.v01 = mk2(a.z, a.w);
    s.v10 = mk2(b.x, b.y);
    s.v11 = mk2(b.z, b.w);
    s.depthsProj = mk4(d.x, d.y, d.z, d.w);
    return stageFromProjection<TS>(sh, k, bin, s, stageShade<TS>(sh, k, st, sg, shading, P, SP), x0, y0);
  }
  sh.box[k] = EMPTY_BOX;
  sh.shadeBase[k] = bin << 24;
  sh.cnt[k] = 0;
  return 0u;
}

// With two threads per staged segment: thread `end` of segment k projects
// point sg + end of it (projectHairPoint) into the round's point scratch
// (the fragment list's storage, free until the edge tests); the end-point
// thread also stages the segment's shading entries.
template <int TS>
__device__ __forceinline__ void stagePoint(FineSmem<TS>& sh, uint32_t k, uint32_t end, const HfbUniforms& U,
                                           const float4* __restrict__ pos, const float4* __restrict__ tan,
                                           const float4* __restrict__ shading, uint32_t S, uint32_t P, uint32_t SP,
                                           f2 size) {
  constexpr uint32_t STAGE = FineSmem<TS>::STAGE;
  float* pt = reinterpret_cast<float*>(sh.frag) + end * 6u * STAGE;  // [6][STAGE] per end
  const uint32_t st = sh.enc[k] & 0x00ffffffu, sg = sh.enc[k] >> 24;
  if (!(st < S && sg + 1u < P)) return;
  const size_t i = (size_t)st * P + sg + end;
  f2 o0, o1;
  float z0, z1;
  projectHairPoint(U.modelMatrix.m, U.vpMatrix.m, mk3(U.cameraPosition.x, U.cameraPosition.y, U.cameraPosition.z),
                   ld4(__ldg(HFB_G(&pos[i]))), ld4(__ldg(HFB_G(&tan[i]))), size, U.fiberRadius, o0, o1, z0, z1);
  pt[0u * STAGE + k] = o0.x;
  pt[1u * STAGE + k] = o0.y;
  pt[2u * STAGE + k] = o1.x;
  pt[3u * STAGE + k] = o1.y;
  pt[4u * STAGE + k] = z0;
  pt[5u * STAGE + k] = z1;
  if (end) sh.shadeBase[k] = stageShade<TS>(sh, k, st, sg, shading, P, SP);
}

// Stages segment k from the two points stagePoint left.
template <int TS>
__device__ __forceinline__ uint32_t stageFromPoints(FineSmem<TS>& sh, uint32_t k, uint32_t bin, uint32_t S,
                                                    uint32_t P, uint32_t x0, uint32_t y0) {
  constexpr uint32_t STAGE = FineSmem<TS>::STAGE;
  const uint32_t st = sh.enc[k] & 0x00ffffffu, sg = sh.enc[k] >> 24;
  if (!(st < S && sg + 1u < P)) {
    sh.box[k] = EMPTY_BOX;
    sh.shadeBase[k] = bin << 24;
    sh.cnt[k] = 0;
    return 0u;
  }
  const float* p0 = reinterpret_cast<const float*>(sh.frag);
  const float* p1 = p0 + 6u * STAGE;
  ProjSeg s;
  s.v00 = mk2(p0[0u * STAGE + k], p0[1u * STAGE + k]);
  s.v01 = mk2(p0[2u * STAGE + k], p0[3u * STAGE + k]);
  s.v10 = mk2(p1[0u * STAGE + k], p1[1u * STAGE + k]);
  s.v11 = mk2(p1[2u * STAGE + k], p1[3u * STAGE + k]);
  s.depthsProj = mk4(p0[4u * STAGE + k], p0[5u * STAGE + k], p1[4u * STAGE + k], p1[5u * STAGE + k]);
  return stageFromProjection<TS>(sh, k, bin, s, sh.shadeBase[k], x0, y0);
}

// Fragment colour of staged segment k at segment coordinates w and depth hd
// (processHairSegment.wgsl.ts:43-53 with getAlphaCoverage :60-69 and
// _sampleShading, hairShadingBuffer.ts:28-38), as 4 x f16, and its slice.
template <int TS>
__device__ __forceinline__ uint2 fragmentColour(const FineSmem<TS>& sh, uint32_t k, f2 w, float hd, uint32_t P,
                                                uint32_t SP, uint32_t L, uint32_t bin,
                                                uint32_t alphaQuadratic, float alphaMul,
                                                const float4* __restrict__ shading, uint32_t& slice) {
  float alpha = fsub(1.0f, fabsf(fsub(fmul(w.x, 2.0f), 1.0f)));
  if (alphaQuadratic) alpha = sqrtf(alpha);
  alpha = sat(fmul(alpha, alphaMul));
  // (segment + w.y) / (P - 1).  w.y is a quotient of a length, which is 0 or at least 2^-75, by
  // the segment's: for segments up to 2^25 px it is 0 or at least DIV_TINY, and divBy's quotient is the
  // division's; below (a numerator that only segment 0 has) it may miss one unit of 2^-149,
  // which nothing of a colour in 16 bits (steps of 2^-24 at the least) shows
  const float tFull = divBy(fadd((float)(sh.enc[k] >> 24), w.y), {(float)(P - 1u), 1.0f / (float)(P - 1u)});
  uint32_t i0, i1;
  const float fr = remapToIndices(SP, tFull, i0, i1);
  const uint32_t sbase = sh.shadeBase[k];
  const uint32_t e0 = sbase & 0xffffu, ne = (sbase >> 16) & 0xffu;
  float4 c0, c1;
  if (i0 - e0 < ne && i1 - e0 < ne) {
    c0 = sh.shade[k][i0 - e0];
    c1 = sh.shade[k][i1 - e0];
  } else {
    const size_t sb = (size_t)(sh.enc[k] & 0x00ffffffu) * SP;
    c0 = __ldg(HFB_G(&shading[sb + i0]));
    c1 = __ldg(HFB_G(&shading[sb + i1]));
  }
  f4 c = mix4(ld4(c0), ld4(c1), fr);
  c.w = fmul(c.w, alpha);
  // getSliceIdx: getDepthBin(L, td0, td1, hd); a quotient too tiny for divBy is in slice 0 either way
  const float td0 = sh.td0[bin], span = fabsf(fsub(sh.td1[bin], td0)), x = fsub(hd, td0);
  float t = divBy(x, {span, sh.tdY[bin]});
  if (!(fabsf(t) < 1e30f)) t = x / span;
  slice = clampu(f2u(fmul(t, (float)L)), 0u, L - 1u);
  const uint32_t hx = __half_as_ushort(__float2half_rn(c.x)), hy = __half_as_ushort(__float2half_rn(c.y));
  const uint32_t hz = __half_as_ushort(__float2half_rn(c.z)), hw = __half_as_ushort(__float2half_rn(c.w));
  return make_uint2(hx | (hy << 16), hz | (hw << 16));
}

__device__ __forceinline__ float halfLo(uint32_t v) { return __half2float(__ushort_as_half((unsigned short)(v & 0xffffu))); }
__device__ __forceinline__ float halfHi(uint32_t v) { return __half2float(__ushort_as_half((unsigned short)(v >> 16))); }

// A pixel's slices of the bin at the cursor.  In shared memory, a float4 of every
// pixel per slice, where the CTAs that the registers allow leave room for it: a
// fragment then costs one load and one store, not a predicated blend of every slice,
// and `touched` names the slices that hold anything: 153 -> 131 us on a frame of 11,400
// x 16 at 1920x1080 (8 px tiles, 32 bins, 8 slices).  16 slices at 8 px cost one of 6 CTAs per
// SM and are faster all the same: draws of 10,000 x 32 at 1920x1080 433 -> 385 us, of 200,000 x
// 32 at 4K 7.04 -> 6.46 ms, 16 instances in one batch 2.83 -> 2.69 ms.  Else in registers: 8 px
// tiles with 4 slices would lose one of 8 CTAs per SM, 16 px ones one of 3 (4 slices) or of 2
// (16 slices), and 32 px tiles have no room.
template <int TS, int MAXL>
constexpr bool FINE_SHARED_SLICES = (TS == 8 && MAXL >= 8) || (TS == 16 && MAXL == 8);
template <int TS, int MAXL>
constexpr size_t FINE_SMEM = sizeof(FineSmem<TS>) + (FINE_SHARED_SLICES<TS, MAXL> ? MAXL * TS * TS * sizeof(float4) : 0);

// q + kk * acc with kk = 1 - q.a.  The colours take one rounding (fused) where the reference's product
// and sum take two: no bit of the lists or of coverage depends on them, and a colour is off by less.
// Alpha, which decides when a pixel is done, takes the reference's two.
__device__ __forceinline__ void blendOver(f4& acc, const f4 q, float kk) {
  acc.x = __fmaf_rn(kk, acc.x, q.x);
  acc.y = __fmaf_rn(kk, acc.y, q.y);
  acc.z = __fmaf_rn(kk, acc.z, q.z);
  acc.w = fadd(q.w, fmul(kk, acc.w));
}
__device__ __forceinline__ f4 halfColour(uint2 h) { return mk4(halfLo(h.x), halfHi(h.x), halfLo(h.y), halfHi(h.y)); }
// the slice under what is there, until the pixel is done (reduceHairSlices.wgsl.ts:9-73)
__device__ __forceinline__ void sliceUnder(f4& fin, const f4 acc) {
  if (fin.w < 0.999f) {
    const float kk = fsub(1.0f, fin.w);
    fin.x = fadd(fin.x, fmul(acc.x, kk));
    fin.y = fadd(fin.y, fmul(acc.y, kk));
    fin.z = fadd(fin.z, fmul(acc.z, kk));
    fin.w = fadd(fin.w, fmul(acc.w, kk));
  }
}

template <int TS, int MAXL, bool SHARED = FINE_SHARED_SLICES<TS, MAXL>>
struct FineSlices;
template <int TS, int MAXL>
struct FineSlices<TS, MAXL, true> {
  float4* at;  // this pixel's first slice; the next TS * TS on
  uint32_t touched = 0;
  __device__ __forceinline__ explicit FineSlices(FineSmem<TS>& sh)
      : at(reinterpret_cast<float4*>(&sh + 1) + threadIdx.x) {}
  __device__ __forceinline__ void blend(uint32_t sl, uint2 h) {
    if (!HFB_EXPECT(sl < (uint32_t)MAXL)) return;
    f4 acc = mk4(0.0f, 0.0f, 0.0f, 0.0f);
    if ((touched >> sl) & 1u) acc = ld4(at[sl * TS * TS]);
    touched |= 1u << sl;
    const f4 q = halfColour(h);
    blendOver(acc, q, fsub(1.0f, q.w));
    at[sl * TS * TS] = make_float4(acc.x, acc.y, acc.z, acc.w);
  }
  __device__ __forceinline__ void reduce(f4& fin, uint32_t L) {
    for (uint32_t m = touched; m; m &= m - 1u) {  // an empty slice adds nothing
      const uint32_t si = (uint32_t)__ffs(m) - 1u;
      if (si < L) sliceUnder(fin, ld4(at[si * TS * TS]));
    }
  }
  __device__ __forceinline__ void clear() { touched = 0; }
};
template <int TS, int MAXL>
struct FineSlices<TS, MAXL, false> {
  f4 acc[MAXL];
  __device__ __forceinline__ explicit FineSlices(FineSmem<TS>&) { clear(); }
  __device__ __forceinline__ void blend(uint32_t sl, uint2 h) {
    const f4 q = halfColour(h);  // converted once, not once per slice
    const float kk = fsub(1.0f, q.w);
#pragma unroll
    for (int si = 0; si < MAXL; si++)
      if ((uint32_t)si == sl) blendOver(acc[si], q, kk);
  }
  __device__ __forceinline__ void reduce(f4& fin, uint32_t L) {
#pragma unroll
    for (int si = 0; si < MAXL; si++)
      if ((uint32_t)si < L) sliceUnder(fin, acc[si]);
  }
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int si = 0; si < MAXL; si++) acc[si] = mk4(0.0f, 0.0f, 0.0f, 0.0f);
  }
};

// Tile mode: the runs of the next round, from bin `bin`, entry `off` of its
// list, up to `cap` segments.  Bins without depth (td1 == 0) are skipped as
// the reference skips them; a depth bin with an empty list is a run of zero
// segments (its reduce still runs).  A bin is in the round when fewer than
// `cap` entries lie between the cursor and it (binOff), or exactly `cap` and it
// is empty.  Called by one warp, a lane per bin; sets nRuns, returns the segments.
template <int TS>
__device__ __forceinline__ uint32_t buildRuns(FineSmem<TS>& sh, uint32_t b1, uint32_t bin, uint32_t off, uint32_t cap,
                                              uint32_t lane) {
  if (lane < FineSmem<TS>::STAGE / 32u) sh.runStart[lane] = 0;
  __syncwarp();
  uint32_t n = 0, nStart = 0, used = 0;
  const uint32_t p0 = bin < b1 ? sh.binOff[bin] + off : 0u;
  for (uint32_t c0 = bin & ~31u; c0 < b1; c0 += 32u) {
    const uint32_t bb = c0 + lane;
    uint32_t pre = 0, rem = 0, o = 0, hz = 0;
    bool in = false;
    if (bb >= bin && bb < b1 && sh.head[bb].y != 0u) {
      o = bb == bin ? off : 0u;
      hz = sh.head[bb].z;
      pre = sh.binOff[bb] + o - p0;
      rem = sh.binOff[bb + 1u] - sh.binOff[bb] - o;
      in = pre < cap || (rem == 0u && pre == cap);
    }
    const uint32_t take = in ? min(rem, cap - pre) : 0u, lt = (1u << lane) - 1u;
    const uint32_t m = __ballot_sync(0xffffffffu, in), ms = __ballot_sync(0xffffffffu, take != 0u);
    if (in) {
      const uint32_t r = n + (uint32_t)__popc(m & lt);
      sh.runBin[r] = bb | (take == rem ? RUN_ENDS : 0u);
      sh.runK0[r] = (uint16_t)pre;
      sh.runK1[r] = (uint16_t)(pre + take);
      sh.runOff[r] = o;
    }
    if (take) {
      const uint32_t j = nStart + (uint32_t)__popc(ms & lt);
      sh.startBin[j] = (uint8_t)bb;
      sh.startBase[j] = hz - 1u - o + pre;
      atomicOr(&sh.runStart[pre >> 5], 1u << (pre & 31u));
    }
    n += (uint32_t)__popc(m);
    nStart += (uint32_t)__popc(ms);
    used = max(used, __reduce_max_sync(0xffffffffu, in ? pre + take : 0u));
  }
  if (lane == 0) sh.nRuns = n;
  return used;
}

// Rasterizes depth bins [b0, b1) of tile tileIdx in order, every pixel
// starting from an empty colour (processTile per bin + reduceHairSlices,
// hairFinePass.wgsl.ts:205-288), and leaves each pixel's colour in fin.
// With `part` IN_ORDER the bins start the tile, or carry on from the colours at
// `resume` that the tile's earlier bins left.  Otherwise they are a later part
// of a split tile: every pixel in view takes part, and the call gives up
// (FINE_UNSAFE) where a bin could fill its fragment pool, whose cut would depend
// on which pixels the earlier bins finished.  Where it gives up decides whether
// the tile is merged from its parts or drawn in order, which shows in the pixels
// (up to the 0.001 that a finished pixel still lacks), so the decision must not
// depend on how tight the listed pixels are: CAREFUL takes rounds of at most
// PAIRS box pixels and counts what the edge tests accept, and its running bound
// exceeds a bin's own count by less than PAIRS.  QUICK takes full rounds and bounds
// a bin's count from both sides: the accepted pixels of the rounds that are all the
// bin's, with and without the listed pixels of the others.  Where the lower bound
// exceeds the pool CAREFUL gives up as well, where the upper one stays PAIRS below
// it CAREFUL goes on as well; a bin that ends in between is FINE_AGAIN, for CAREFUL
// to decide.
enum FinePart : uint32_t { FINE_IN_ORDER = 0, FINE_QUICK, FINE_CAREFUL };
// Bits of a split tile's word: parts that arrived; bins of the first part that filled their
// pool; the first part's colours are there; a later part gave up.
constexpr uint32_t FINE_FILLED_SHIFT = 16, FINE_FILLED = 0x7fu << FINE_FILLED_SHIFT, FINE_FIRST = 1u << 30, FINE_REDO = 1u << 31;
enum FineEnd : uint32_t { FINE_OK = 0, FINE_UNSAFE, FINE_AGAIN };
template <int TS, int MAXL>
__device__ __forceinline__ FineEnd fineTile(FineSmem<TS>& sh, const HfbUniforms& U, const FineArgs& a,
                                         uint32_t tileIdx, uint32_t b0, uint32_t b1, FinePart part,
                                         const float4* resume, f4& fin) {
  using SM = FineSmem<TS>;
  constexpr uint32_t NT = SM::NT, STAGE = SM::STAGE, PAIRS = SM::PAIRS, ROWS = SM::ROWS, NW = NT / 32u;
  constexpr uint32_t MODE_FAST = 0, MODE_TIGHTEN = 1, MODE_ABORT = 2;
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  const uint32_t lx = tid % TS, ly = tid / TS;
  const f2 size = mk2(U.viewport.x, U.viewport.y);
  const uint32_t W = f2u(size.x), H = f2u(size.y);
  const uint32_t tilesX = divCeil(W, TS);
  const uint32_t maxDrawn = U.maxDrawnHairSegments;
  const uint32_t maxProcessed = a.S * a.P;  // MAX_PROCESSED_SEGMENTS, hairFinePass.wgsl.ts:212
  const uint32_t dispMode = U.displayMode & 0xffu;
  const uint32_t dbgMax = dispMode == 4u ? ((U.displayMode >> 8) & 0xffffu) : 0u;  // getDbgSlicesModeMaxSlices
  const bool isDbg = dbgMax != 0u;
  const uint32_t tx = tileIdx % tilesX, ty = tileIdx / tilesX;
  const TileB tbp = tileBoundsPx(W, H, TS, tx, ty);
  const uint32_t px = tbp.x0 + lx, py = tbp.y0 + ly;
  // Pixels of a partial edge tile outside the viewport take no part.
  const bool inView = px < W && py < H;
  sh.zbuf[tid] = inView ? loadTex2DClamp(a.depth, W, H, f2i((float)px), f2i(fsub(size.y, (float)py))) : 0.0f;
  bool done = !inView;
  fin = mk4(0.f, 0.f, 0.f, 0.f);  // rasterizerResult was cleared before the pass
  if (resume) {
    const float4 f = __ldcg(HFB_G(&resume[tid]));
    fin = mk4(f.x, f.y, f.z, f.w);
    done = done || fin.w >= 0.999f;
    if (__syncthreads_and(done)) return FINE_OK;
  }
  if (tid == 0) {
    sh.filled = 0;
    sh.liveBox = make_float4(0.0f, 0.0f, (float)(TS - 1), (float)(TS - 1));
  }
  {
    const uint32_t dm = __ballot_sync(0xffffffffu, done);
    if (lane == 0) sh.doneMask[warp] = dm;
  }
  if (tid < a.B) {
    const uint4 h = (*HFB_G(&a.tiles[ty * tilesX * a.B + tx * a.B + tid]));
    sh.head[tid] = h;
    const float d0 = (float)(0xffffffffu - h.x) / F_MAX_U32, d1 = (float)h.y / F_MAX_U32;  // _getTileDepth
    sh.td0[tid] = d0;
    sh.td1[tid] = d1;
    sh.tdY[tid] = recipOf(fabsf(fsub(d1, d0))).y;
  }
  __syncthreads();

  // ---- tile mode: every depth bin's list carries a length hint (padding0,
  // written by the tiles pass) and the lists are the contiguous runs the
  // tiles pass writes; otherwise each list is walked ----
  if (warp == 0) {
    uint32_t ok = 1, sum = 0;
    for (uint32_t c0 = 0; c0 < a.B; c0 += 32) {
      const uint32_t bb = c0 + lane;
      uint32_t nb = 0;
      if (bb >= b0 && bb < b1) {
        const uint4 h = sh.head[bb];
        if (h.y != 0u && h.z != 0u) {
          if (h.w != 0u && h.w <= h.z && h.z <= maxDrawn && h.w <= maxProcessed) nb = h.w; else ok = 0;
        }
      }
      uint32_t incl = nb;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += y;
      }
      if (bb < a.B) sh.binOff[bb] = sum + incl - nb;
      sum += __shfl_sync(0xffffffffu, incl, 31);
    }
    ok = __all_sync(0xffffffffu, ok);
    if (lane == 0) {
      sh.binOff[a.B] = sum;
      sh.total = sum;
      sh.tileMode = ok;
      sh.bad = 0;
    }
  }
  __syncthreads();
  bool tileMode = sh.tileMode != 0u;
  // check every link of the contiguous layout, unless the same frame's tiles pass wrote it
  if (tileMode && a.proj == nullptr) {
    const uint32_t total = sh.total;
    for (uint32_t k = tid; k < total; k += NT) {
      uint32_t lo = 0, hi = a.B;  // bin of k: binOff[lo] <= k < binOff[lo + 1]
      while (hi - lo > 1u) {
        const uint32_t mid = (lo + hi) >> 1;
        if (sh.binOff[mid] <= k) lo = mid; else hi = mid;
      }
      const uint4 h = sh.head[lo];
      const uint32_t j = k - sh.binOff[lo];
      const uint32_t idx = h.z - 1u - j;
      if (!HFB_EXPECT(idx < maxDrawn)) { sh.bad = 1; continue; }
      const uint32_t nxt = __ldg(HFB_G(&a.segBuf[2u + 2u * idx]));
      if (nxt != ((j + 1u == h.w) ? INVALID_PTR : idx - 1u)) sh.bad = 1;
    }
    __syncthreads();
    tileMode = sh.bad == 0u;
  }

  // per-pixel state of the current bin
  FineSlices<TS, MAXL> slices(sh);
  uint32_t nFrag = 0, pending = 0;
  // uniform state: cursor and the pool accounting of the bin at the cursor
  uint32_t bin = b0, off = 0;                    // tile mode: bin, entry of its list
  uint32_t walkPtr = INVALID_PTR, processed = 0;  // walk mode: list pointer, entries processed
  uint32_t running = 0, runningUB = 0;            // slots taken (exact / upper bound)

  while (true) {
    // ---------------- stage the round: a thread per segment ----------------
    uint32_t myBin = 0, myEnc = 0xffffffffu;
    if (resume && warp == 1) {
      const float4 lb = liveBoxOf<TS>(sh, lane);
      if (lane == 0) sh.liveBox = lb;
    }
    if (tileMode) {
      if (warp == 0) {
        const uint32_t used = buildRuns<TS>(sh, b1, bin, off, STAGE, lane);
        if (lane == 0) sh.nStaged = used;
      }
      __syncthreads();
      if (tid < sh.nStaged) {
        uint32_t j = (uint32_t)__popc(sh.runStart[tid >> 5] & (0xffffffffu >> (31u - lane)));
        for (uint32_t w = 0; w < tid >> 5; w++) j += (uint32_t)__popc(sh.runStart[w]);
        myBin = sh.startBin[j - 1u];
        const uint32_t idx = sh.startBase[j - 1u] - tid;
        myEnc = HFB_EXPECT(idx < maxDrawn) ? __ldg(HFB_G(&a.segBuf[1u + 2u * idx])) : 0xffffffffu;
        sh.enc[tid] = myEnc;
      }
    } else {
      while (bin < b1 && sh.head[bin].y == 0u) bin++;  // bins without depth are skipped
      if (bin >= b1) break;
      if (processed == 0u) {
        const uint32_t hz = sh.head[bin].z;
        walkPtr = hz == 0u ? INVALID_PTR : hz - 1u;
      }
      if (warp == 0) {  // speculative contiguous runs, else pointer chasing
        uint32_t p = walkPtr, m = 0;
        while (m < STAGE && p != INVALID_PTR && p < maxDrawn && processed + m < maxProcessed) {
          const uint32_t want = min(min(32u, STAGE - m), maxProcessed - processed - m);
          const uint32_t cand = p - lane;
          const bool inRange = lane < want && lane <= p;
          uint2 e = make_uint2(0u, INVALID_PTR);
          if (inRange) {
            e.x = __ldg(HFB_G(&a.segBuf[1u + 2u * cand]));
            e.y = __ldg(HFB_G(&a.segBuf[2u + 2u * cand]));
          }
          const bool chain = inRange && e.y == cand - 1u;
          const uint32_t brk = __ballot_sync(0xffffffffu, !chain);
          const uint32_t first = brk ? (uint32_t)(__ffs(brk) - 1) : 32u;
          bool firstIn = false;
          uint32_t firstNext = 0u;
          if (first < 32u) {
            firstIn = __shfl_sync(0xffffffffu, inRange, first);
            firstNext = __shfl_sync(0xffffffffu, e.y, first);
          }
          const uint32_t cnt = firstIn ? first + 1u : first;
          if (lane < cnt) {
            sh.enc[m + lane] = e.x;
            sh.listIdx[m + lane] = cand;
          }
          m += cnt;
          p = firstIn ? firstNext : p - cnt;
        }
        if (lane == 0) {
          const bool ends = !(p != INVALID_PTR && p < maxDrawn && processed + m < maxProcessed);
          sh.nStaged = m;
          sh.walkNext = p;
          sh.nRuns = 1;
          sh.runBin[0] = bin | (ends ? RUN_ENDS : 0u);
          sh.runK0[0] = 0;
          sh.runK1[0] = (uint16_t)m;
          sh.runOff[0] = processed;
        }
      }
    }
    // In tile mode the runs were published at the barrier above and each thread
    // projects the segments it staged itself (the cached and the one-thread-per-
    // segment projections): no barrier is needed before the projection.
    if (!(tileMode && (a.proj != nullptr || 2u * STAGE > NT))) __syncthreads();
    uint32_t nRuns = sh.nRuns;
    if (nRuns == 0u) break;  // tile mode: no depth bin left
    const bool fresh = sh.runOff[0] == 0u;  // run 0 starts its bin
    if (fresh) { running = 0; runningUB = 0; }

    // ---------------- project ----------------
    {
      const uint32_t nStaged = sh.nStaged;
#pragma unroll
      for (uint32_t w = 0; w < STAGE / 32; w++) sh.pixMask[w][tid] = 0u;
      if (!tileMode && tid < nStaged) {
        myBin = sh.runBin[0] & 0xffu;
        myEnc = sh.enc[tid];
      }
      if (a.proj) {
        // the tiles pass projected every segment of the frame already
        if (tid < nStaged)
          sh.rowBase[tid] = stageCached<TS>(sh, tid, myBin, a.proj, a.shading, myEnc, a.S, a.P, a.SP, tbp.x0, tbp.y0);
      } else if constexpr (2u * STAGE <= NT) {
        // two threads per segment: one projects its first point, one its second
        if (tid < 2u * nStaged) {
          const uint32_t end = tid >= nStaged ? 1u : 0u;
          stagePoint<TS>(sh, tid - end * nStaged, end, U, a.pos, a.tan, a.shading, a.S, a.P, a.SP, size);
        }
        __syncthreads();
        if (tid < nStaged) sh.rowBase[tid] = stageFromPoints<TS>(sh, tid, myBin, a.S, a.P, tbp.x0, tbp.y0);
      } else {
        if (tid < nStaged)
          sh.rowBase[tid] =
              stageSegment<TS>(sh, tid, myBin, U, a.pos, a.tan, a.shading, a.S, a.P, a.SP, size, tbp.x0, tbp.y0);
      }
      __syncthreads();
      // exclusive prefix of the box heights (low half) and areas (high half) together, all
      // chunks of 32 segments at once (independent shuffle chains); the halves cannot carry
      // into each other: at most STAGE * TS * TS and STAGE * TS, below 2^16 up to 16 px
      // tiles.  The round keeps the longest prefix of segments whose rows fit (and, in a
      // CAREFUL part, at most PAIRS box pixels)
      if (warp == 0) {
        using V = std::conditional_t<(TS <= 16), uint32_t, unsigned long long>;
        constexpr uint32_t SH = TS <= 16 ? 16u : 32u, NC = STAGE / 32u;
        constexpr V LOW = ((V)1 << SH) - 1u;
        V val[NC], incl[NC];
#pragma unroll
        for (uint32_t c = 0; c < NC; c++) {
          const uint32_t k = c * 32u + lane;
          const uint32_t rows = k < nStaged ? sh.rowBase[k] : 0u, box = k < nStaged ? sh.box[k] : 0u;
          val[c] = ((V)(rows ? rows * (((box >> 16) & 0xffu) - (box & 0xffu) + 1u) : 0u) << SH) | rows;
          incl[c] = val[c];
        }
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
          for (uint32_t c = 0; c < NC; c++) {
            const V y = __shfl_up_sync(0xffffffffu, incl[c], o);
            if (lane >= (uint32_t)o) incl[c] += y;
          }
        }
        V carry = 0;
        uint32_t nSeg = nStaged;
#pragma unroll
        for (uint32_t c = 0; c < NC; c++) {
          const uint32_t k = c * 32u + lane;
          const uint32_t ex = (uint32_t)((carry + incl[c] - val[c]) & LOW);
          if (k < nStaged) {
            sh.rowBase[k] = ex;
            sh.rowOff[k] = ex - ((sh.box[k] >> 8) & 0xffu);
          }
          const V end = carry + incl[c];
          const uint32_t over = __ballot_sync(0xffffffffu, k < nStaged && ((uint32_t)(end & LOW) > ROWS ||
                                                                           (part == FINE_CAREFUL && (uint32_t)(end >> SH) > PAIRS)));
          if (over && nSeg == nStaged) nSeg = c * 32u + (uint32_t)(__ffs(over) - 1);
          carry += __shfl_sync(0xffffffffu, incl[c], 31);
        }
        if (lane == 0) {
          sh.rowBase[nStaged] = (uint32_t)(carry & LOW);
          sh.nSeg = nSeg;
          sh.segLimit = nSeg;
          sh.passCount = 0xffffffffu;
          sh.edgePasses = 0;
        }
      }
      __syncthreads();
    }
    uint32_t nSeg = sh.nSeg;

    // ---------------- A1: the box rows' spans, one thread per (segment, row) ----------------
    // Each thread takes consecutive rows: it counts its rows' pixels that are in their
    // span and not done, a block scan places them, and it writes them to the list.  A
    // segment whose pixels do not fit any more ends the round (any first one fits).
    {
      const uint32_t nRows = sh.rowBase[nSeg];
      const uint32_t per = divCeil(nRows, NT);  // at most ROWS / NT
      const uint32_t r0 = min(tid * per, nRows), r1 = min(r0 + per, nRows);
      uint32_t k = 0, kFirst = 0, cnt = 0;
      if (r0 < r1) {
        uint32_t lo = 0, hi = nSeg;  // last k with rowBase[k] <= r0
        while (hi - lo > 1u) {
          const uint32_t mid = (lo + hi) >> 1;
          if (sh.rowBase[mid] <= r0) lo = mid; else hi = mid;
        }
        k = kFirst = lo;
        uint32_t end = sh.rowBase[k + 1u], box = sh.box[k];
        float4 sLo = sh.spanLo[k], sHi = sh.spanHi[k];
        uint32_t off = sh.rowOff[k];
        for (uint32_t r = r0; r < r1; r++) {
          if (r >= end) {  // next segment with rows
            do { end = sh.rowBase[++k + 1u]; } while (end <= r);
            box = sh.box[k];
            sLo = sh.spanLo[k];
            sHi = sh.spanHi[k];
            off = sh.rowOff[k];
          }
          const uint32_t qy = r - off;
          int xa = (int)(box & 0xffu), xb = (int)((box >> 16) & 0xffu);
          spanOf(sLo, sHi, (float)qy, xa, xb);
          uint32_t live = 0;
          if (xa <= xb) {
            const uint32_t rowPix = qy * TS;
            live = (0xffffffffu << xa) & (0xffffffffu >> (31 - xb)) & ~(sh.doneMask[rowPix >> 5] >> (rowPix & 31u));
          }
          sh.row[r].set(live, 0u);
          cnt += (uint32_t)__popc(live);
        }
      }
      // exclusive prefix of the counts in thread order
      uint32_t incl = cnt;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += y;
      }
      if (lane == 31) sh.red[warp] = incl;
      __syncthreads();
      uint32_t pos = incl - cnt;
      for (uint32_t w = 0; w < warp; w++) pos += sh.red[w];
      if (tid == NT - 1u) atomicMin(&sh.passCount, pos + cnt);  // the total: every row's, unless the list fills up
      if (r0 < r1) {
        uint32_t end = sh.rowBase[kFirst + 1u], off = sh.rowOff[kFirst];
        k = kFirst;
        for (uint32_t r = r0; r < r1; r++) {
          if (r >= end) {
            do { end = sh.rowBase[++k + 1u]; } while (end <= r);
            off = sh.rowOff[k];
          }
          uint32_t live = sh.row[r].pixels();
          const uint32_t n = (uint32_t)__popc(live);
          if (pos + n > PAIRS) {  // the rows before this one fit
            atomicMin(&sh.segLimit, k);
            atomicMin(&sh.passCount, pos);
            break;
          }
          sh.row[r].set(live, pos);
          const uint32_t tag = (r - off) * TS | (k << 16);
          while (live) {
            const uint32_t qx = (uint32_t)(__ffs(live) - 1);
            live &= live - 1u;
            if (HFB_EXPECT(pos < PAIRS)) sh.frag[pos].x = tag + qx;
            pos++;
          }
        }
      }
    }
    __syncthreads();
    nSeg = sh.segLimit;
    if (nSeg < sh.nStaged) {  // uniform: drop the segments from nSeg on
      if (tid == 0) sh.nSeg = nSeg;
      if (tileMode) {
        if (warp == 0) buildRuns<TS>(sh, b1, bin, off, nSeg, lane);
      } else if (tid == 0) {
        sh.runK1[0] = (uint16_t)nSeg;
        sh.runBin[0] &= ~RUN_ENDS;
      }
      __syncthreads();
    }
    nRuns = sh.nRuns;

    // ---------------- can a bin fill its pool in this round? ----------------
    // The listed pixels bound the fragments: when those of the whole round, on
    // top of what the cursor's bin may already hold, fit in a pool, no bin can
    // fill its pool and nothing needs counting (the common case: every thread
    // sees passCount after the barrier above).  Otherwise one warp sums the
    // listed pixels run by run.  e0 / eLast carry the bounds of the first and
    // last run (the round's total where it is enough).  A CAREFUL part, and a QUICK
    // one inside a bin, check after A2, which counts what the edge tests accept.
    const uint32_t cap = a.CAP;
    const uint32_t sure = cap > PAIRS ? cap - PAIRS : 0u;  // CAREFUL goes on where QUICK's bound is at most this
    uint32_t mode = MODE_FAST, e0 = sh.passCount, eLast = e0;
    auto sumRuns = [&]() {  // by run, with the warp 0; all threads call
      if (warp == 0) {
        uint32_t wmode = MODE_FAST, keep = nRuns, we0 = 0, weLast = 0;
        for (uint32_t r = 0; r < nRuns; r++) {
          uint32_t e = 0;
          if (part == FINE_CAREFUL) {
            for (uint32_t k = sh.runK0[r] + lane; k < sh.runK1[r]; k += 32) e += sh.cnt[k];
          } else {
            for (uint32_t q = sh.rowBase[sh.runK0[r]] + lane; q < sh.rowBase[sh.runK1[r]]; q += 32)
              e += (uint32_t)__popc(sh.row[q].pixels());
          }
          e = __reduce_add_sync(0xffffffffu, e);
          const uint32_t base = r == 0u ? runningUB : 0u;
          if (r == 0u) we0 = e;
          if (base + e > (part == FINE_QUICK ? sure : cap)) {
            if (r == 0u) { wmode = MODE_TIGHTEN; keep = 1; } else { keep = r; }
            break;
          }
          weLast = e;
        }
        if (part != FINE_IN_ORDER && (wmode == MODE_TIGHTEN || keep < nRuns)) wmode = MODE_ABORT;
        if (lane == 0) {
          sh.mode = wmode;
          sh.e0 = we0;
          sh.eLast = weLast;
          if (keep < nRuns) {  // the round ends where that bin's run starts
            sh.nRuns = keep;
            sh.nSeg = sh.runK1[keep - 1u];
          }
          sh.roundFrags = 0;
        }
      }
      __syncthreads();
      mode = sh.mode;
      e0 = sh.e0;
      eLast = sh.eLast;
      nRuns = sh.nRuns;
      nSeg = sh.nSeg;
    };
    // (QUICK: the bin at the cursor ends, others begin)
    if (part == FINE_IN_ORDER ? runningUB + e0 > cap : part == FINE_QUICK && nRuns > 1u && runningUB + e0 > sure) {
      sumRuns();
      if (mode == MODE_ABORT) return FINE_AGAIN;
    }
    bool exact = false;
    if (mode == MODE_TIGHTEN) {
      running += blockSum<NW>(pending, sh.red, lane, warp);
      pending = 0;
      runningUB = running;
      exact = runningUB + e0 > a.CAP;
    }

    // ---------------- A2: fragments, one thread per listed pixel ----------------
    {
      // the arguments this phase reads, in registers for the phase only
      const uint32_t P = a.P, SP = a.SP, L = a.L, alphaQuadratic = a.alphaQuadratic;
      const float alphaMul = a.alphaMul;
      const float4* __restrict__ shading = a.shading;
      const uint32_t nPass = sh.passCount;
      uint32_t accepted = 0;
      for (uint32_t i = tid; i < nPass; i += NT) {
        const uint32_t e = sh.frag[i].x;
        const uint32_t pix = e & 0xffffu, k = e >> 16;
        if (k >= nSeg) continue;  // dropped from the round
        if (!HFB_EXPECT(i < PAIRS && k < STAGE && pix < NT)) continue;
        const uint32_t qx = pix % TS, qy = pix / TS;
        const f2 pf = mk2((float)(tbp.x0 + qx), (float)(tbp.y0 + qy));
        bool inside = true;
#pragma unroll
        for (int j = 0; j < 4; j++)  // edgeFunction >= 0
          inside = inside && fsub(fmul(fsub(pf.x, sh.ox[j][k]), sh.ey[j][k]), fmul(fsub(pf.y, sh.oy[j][k]), sh.ex[j][k])) >= 0.0f;
        if (!inside) continue;
        accepted++;
        if (part == FINE_CAREFUL) atomicAdd(&sh.cnt[k], 1u);
        QuadConst qc;
        qc.sm = mk2(sh.qsx[k], sh.qsy[k]);
        qc.ab = mk2(sh.qax[k], sh.qay[k]);
        qc.d2 = sh.qd2[k]; qc.lse = sh.qlse[k]; qc.wS = sh.qws[k]; qc.wE = sh.qwe[k];
        qc.ab2 = mk2(sh.ex[3][k], sh.ey[3][k]);
        qc.d22 = sh.qd22[k];
        const f2 w = interpolateHairQuadPre(qc, {sh.yd2[k], sh.ylse[k], sh.yd22[k]}, mk2(sh.ox[3][k], sh.oy[3][k]), pf);
        const float hd = interpolateHairF32(w, mk4(sh.dp[0][k], sh.dp[1][k], sh.dp[2][k], sh.dp[3][k]));
        if (!(hd < sh.zbuf[pix])) continue;  // depth test with GL_LESS (skip when >=)
        const uint32_t kb = sh.shadeBase[k] >> 24;
        uint32_t slice;
        const uint2 col = fragmentColour<TS>(sh, k, w, hd, P, SP, L, kb, alphaQuadratic, alphaMul, shading, slice);
        sh.frag[i] = col;
        sh.slice[i] = (uint8_t)slice;
        atomicOr(&sh.pixMask[k >> 5][pix], 1u << (k & 31u));
        if (exact) atomicAdd(&sh.cnt[k], 1u);
      }
      if (part == FINE_CAREFUL || (part == FINE_QUICK && nRuns == 1u)) {
        accepted = __reduce_add_sync(0xffffffffu, accepted);
        if (lane == 0 && accepted) atomicAdd(&sh.edgePasses, accepted);
      }
    }
    __syncthreads();
    if (part == FINE_QUICK && nRuns == 1u) {  // all the cursor's bin: running and runningUB are its bounds
      e0 = sh.edgePasses;
      running += e0;
      if (running > a.CAP) return FINE_UNSAFE;
      if ((sh.runBin[0] & RUN_ENDS) && runningUB + e0 > sure) return FINE_AGAIN;
    }
    if (part == FINE_CAREFUL) {
      e0 = eLast = sh.edgePasses;
      if (runningUB + e0 > cap) {
        sumRuns();
        if (mode == MODE_ABORT) return FINE_UNSAFE;  // a pool could fill: this part cannot stand alone
      }
    }

    // ---------------- exact accounting: the segment that fills the pool ----------------
    if (exact) {
      if (warp == 0) {  // one run (this bin) in the round
        uint32_t carry = 0, cut = INVALID_PTR, cutSlots = 0;
        for (uint32_t k0 = 0; k0 < nSeg; k0 += 32) {
          const uint32_t k = k0 + lane;
          const uint32_t c = k < nSeg ? sh.cnt[k] : 0u;
          uint32_t incl = c;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= (uint32_t)o) incl += y;
          }
          const uint32_t fb = __ballot_sync(0xffffffffu, k < nSeg && running + carry + incl >= a.CAP);
          if (fb) {
            const uint32_t j = (uint32_t)(__ffs(fb) - 1);
            cut = k0 + j;
            cutSlots = a.CAP - (running + carry + __shfl_sync(0xffffffffu, incl - c, j));
            break;
          }
          carry += __shfl_sync(0xffffffffu, incl, 31);
        }
        if (lane == 0) {
          sh.cutSeg = cut;
          sh.cutSlots = cutSlots;
          sh.roundFrags = carry;
          if (cut != INVALID_PTR) {
            sh.nSeg = cut + 1u;
            sh.runK1[0] = (uint16_t)(cut + 1u);
            sh.runBin[0] |= RUN_ENDS;  // the reference breaks after the filling segment
            sh.filled++;
            atomicAdd(HFB_G(&a.counters->finePoolFullBins), 1ull);
          }
        }
      }
      __syncthreads();
      const uint32_t cut = sh.cutSeg;
      if (cut != INVALID_PTR) {  // slots of the filling segment in pixel order
        const uint32_t b = sh.box[cut], bxa = b & 0xffu, bya = (b >> 8) & 0xffu;
        const uint32_t bw = ((b >> 16) & 0xffu) - bxa + 1u, area = bw * ((b >> 24) - bya + 1u);
        const uint32_t pix = tid < area ? (bya + tid / bw) * TS + bxa + tid % bw : 0u;
        const uint32_t bit = 1u << (cut & 31u);
        const bool has = tid < area && (sh.pixMask[cut >> 5][pix] & bit) != 0u;
        const uint32_t rank = blockExclusive<NW>(has ? 1u : 0u, sh.red, lane, warp);
        if (has && rank >= sh.cutSlots) sh.pixMask[cut >> 5][pix] &= ~bit;  // the pool is full
        __syncthreads();
      }
      nSeg = sh.nSeg;
    }

    // ---------------- B: every pixel blends its fragments in list order ----------------
    const uint32_t L = a.L;
    for (uint32_t r = 0; r < nRuns; r++) {
      const uint32_t rb = sh.runBin[r], k0 = sh.runK0[r], k1 = sh.runK1[r];
      if (!done && k0 < k1) {
        for (uint32_t w = k0 >> 5; w <= (k1 - 1u) >> 5; w++) {
          const uint32_t lo = max(k0, w * 32u) - w * 32u, hi = min(k1, w * 32u + 32u) - w * 32u;
          uint32_t bits = sh.pixMask[w][tid] & (hi == 32u ? 0xffffffffu : ((1u << hi) - 1u)) & ~((1u << lo) - 1u);
          while (bits) {
            const uint32_t j = w * 32u + (uint32_t)(__ffs(bits) - 1);
            bits &= bits - 1u;
            const uint32_t at = sh.row[sh.rowOff[j] + ly].at(lx);
            if (HFB_EXPECT(at < PAIRS)) {
              slices.blend(sh.slice[at], sh.frag[at]);
              nFrag++;
              pending++;
            }
          }
        }
      }
      if (rb & RUN_ENDS) {
        // reduceHairSlices (runs for every bin with depth, as in the reference)
        if (!done) {
          if (isDbg) {
            const uint32_t cntAll = f2u(fmul(fin.x, (float)dbgMax)) + nFrag;
            fin = mk4(sat((float)cntAll / (float)dbgMax), 0.0f, 0.0f, 1.0f);
          } else {
            slices.reduce(fin, L);
            done = fin.w >= 0.999f;  // isPixelDone with ALPHA_CUTOFF
          }
        }
        slices.clear();
        nFrag = 0;
        pending = 0;
      }
    }

    // ---------------- carry the pool state and advance the cursor ----------------
    const uint32_t lastBin = sh.runBin[nRuns - 1u];
    const bool lastEnds = (lastBin & RUN_ENDS) != 0u;
    if (lastEnds) {
      running = 0;
      runningUB = 0;
    } else if (nRuns == 1u) {
      if (exact) {
        running += sh.roundFrags;
        runningUB = running;
        pending = 0;
      } else {
        runningUB += e0;
      }
    } else {
      running = 0;
      runningUB = eLast;
    }
    if (tileMode) {
      const uint32_t lb = lastBin & 0xffu;
      if (lastEnds) { bin = lb + 1u; off = 0; }
      else { off = sh.runOff[nRuns - 1u] + sh.runK1[nRuns - 1u] - sh.runK0[nRuns - 1u]; bin = lb; }
    } else {
      if (lastEnds) { bin++; processed = 0; }
      else {
        walkPtr = nSeg < sh.nStaged ? sh.listIdx[nSeg] : sh.walkNext;
        processed += nSeg;
      }
    }
    {
      const uint32_t dm = __ballot_sync(0xffffffffu, done);
      if (lane == 0) sh.doneMask[warp] = dm;
    }
    // checkAllPixelsInWkgrpDone, :305-327 (also the barrier before the
    // next round rewrites the staged state)
    if (__syncthreads_and(done)) break;
    if (bin >= b1) break;
  }
  return FINE_OK;
}

constexpr uint32_t SCHED_AHEAD = 4;  // tile-list entries of one thread of the schedule in flight
constexpr uint32_t SCHED_HEADS = 8;  // list heads of one tile in flight

// Builds the work list of the fine pass: one item per drawn tile, in the
// tile list's order (most records first), except that a tile with more
// records than a CTA's average share is split into groups of whole depth
// bins, so that no single CTA carries the frame's tail.  Group sizes come
// from the list-length hints; a tile without valid hints is not split.
// One CTA, bound by the latency of its loads: the heads of a tile are read once,
// SCHED_HEADS at a time, and 1024 entries without a split need no scan.  A frame of
// 32,400 tiles: 26 -> 15 us.
__device__ __forceinline__ void fineScheduleBody(const uint32_t* __restrict__ tileList,
                                                 const uint32_t* __restrict__ segCount,
                                                 const uint4* __restrict__ tiles, uint32_t T, uint32_t B,
                                                 uint32_t grid, uint32_t maxDrawn, uint32_t maxProcessed,
                                                 uint32_t allowSplit, const FineScratch& fs,
                                                 DeviceCounters* __restrict__ counters, uint32_t* warpSums,
                                                 uint32_t& total) {
  const uint32_t tid = threadIdx.x;
  const uint32_t drawn = min((*HFB_G(&tileList[0])), T);
  if (tid == 0) total = 0;
  __syncthreads();
  uint32_t mine = 0;
  for (uint32_t q0 = tid; q0 < drawn; q0 += SCHED_AHEAD * blockDim.x) {
    uint32_t t[SCHED_AHEAD];
#pragma unroll
    for (uint32_t k = 0; k < SCHED_AHEAD; k++) {
      const uint32_t q = q0 + k * blockDim.x;
      t[k] = q < drawn ? (*HFB_G(&tileList[1u + q])) : T;
    }
#pragma unroll
    for (uint32_t k = 0; k < SCHED_AHEAD; k++)
      if (t[k] < T) mine += (*HFB_G(&segCount[t[k]]));
  }
  mine = __reduce_add_sync(0xffffffffu, mine);
  if ((tid & 31u) == 0u) atomicAdd(&total, mine);
  __syncthreads();
  const uint32_t thr = max(FINE_SPLIT_MIN, total / max(grid, 1u));
  uint32_t carryItems = 0, carrySlots = 0;
  uint32_t tNext = tid < drawn ? (*HFB_G(&tileList[1u + tid])) : T;
  uint32_t cNext = tNext < T ? (*HFB_G(&segCount[tNext])) : 0u;
  for (uint32_t q0 = 0; q0 < drawn; q0 += blockDim.x) {
    const uint32_t q = q0 + tid;
    const uint32_t t = tNext, c = cNext;  // T, 0 past the list's end
    tNext = q + blockDim.x < drawn ? (*HFB_G(&tileList[1u + q + blockDim.x])) : T;
    cNext = tNext < T ? (*HFB_G(&segCount[tNext])) : 0u;
    uint32_t nG = q < drawn ? 1u : 0u;  // items of this tile-list entry: none past the list's end
    uint64_t starts = 0;                // bins that start a group but the first
    if (allowSplit && t < T && c > thr) {  // the groups of the split
      uint32_t g = 0, acc = 0;
      bool ok = true;
      for (uint32_t b0 = 0; b0 < B; b0 += SCHED_HEADS) {
        uint4 h[SCHED_HEADS];
#pragma unroll
        for (uint32_t k = 0; k < SCHED_HEADS; k++)
          h[k] = b0 + k < B ? (*HFB_G(&tiles[(size_t)t * B + b0 + k])) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (uint32_t k = 0; k < SCHED_HEADS; k++) {
          uint32_t nb = 0;
          if (h[k].y != 0u && h[k].z != 0u) {
            if (h[k].w != 0u && h[k].w <= h[k].z && h[k].z <= maxDrawn && h[k].w <= maxProcessed) nb = h[k].w;
            else ok = false;
          }
          if (nb == 0u) continue;
          if (acc > 0u && acc + nb > thr) {
            g++;
            acc = 0;
            starts |= 1ull << (b0 + k);
          }
          acc += nb;
        }
      }
      if (acc > 0u) g++;
      if (ok && g > 1u) nG = g;
    }
    if (!__syncthreads_or(nG > 1u)) {  // the usual case past the list's front: one item per tile
      if (q < drawn) (*HFB_G(&fs.items[carryItems + tid])) = make_uint4(q, 0u | (B << 8) | (1u << 24), 0u, 0u);
      carryItems += min(drawn - q0, blockDim.x);
      continue;
    }
    uint32_t chunkSlots;
    const uint32_t mySlots = nG > 1u ? nG : 0u;
    const uint32_t slotEnd = carrySlots + blockExclusiveScan(mySlots, warpSums, chunkSlots) + mySlots;
    const bool split = nG > 1u && slotEnd <= fs.maxGroups;
    if (nG > 1u && !split) nG = 1;
    uint32_t chunkItems;
    const uint32_t itemBase = carryItems + blockExclusiveScan(nG, warpSums, chunkItems);
    if (split) {
      const uint32_t slot = slotEnd - nG;
      (*HFB_G(&fs.arrivals[slot])) = 0;
      atomicAdd(HFB_G(&counters->fineSplitTiles), 1ull);
      const uint32_t firstEnd = (uint32_t)__ffsll((long long)starts) - 1u;  // split: at least one later group
      uint32_t start = 0;
      for (uint32_t g = 0; g < nG; g++) {
        const uint32_t end = starts ? (uint32_t)__ffsll((long long)starts) - 1u : B;
        starts &= starts - 1ull;
        (*HFB_G(&fs.items[itemBase + g])) = make_uint4(q, start | (end << 8) | (g << 16) | (nG << 24), slot, firstEnd);
        start = end;
      }
    } else if (nG) {
      (*HFB_G(&fs.items[itemBase])) = make_uint4(q, 0u | (B << 8) | (1u << 24), 0u, 0u);
    }
    carryItems += chunkItems;
    carrySlots += chunkSlots;
  }
  if (tid == 0) (*HFB_G(&fs.hdr[0])) = carryItems;
  __syncthreads();
}

__global__ void __launch_bounds__(1024)
fineScheduleKernel(const uint32_t* __restrict__ tileList, const uint32_t* __restrict__ segCount,
                   const uint4* __restrict__ tiles, uint32_t T, uint32_t B, uint32_t grid, uint32_t maxDrawn,
                   uint32_t maxProcessed, uint32_t allowSplit, FineScratch fs,
                   DeviceCounters* __restrict__ counters) {
  __shared__ uint32_t warpSums[32];
  __shared__ uint32_t total;
  fineScheduleBody(tileList, segCount, tiles, T, B, grid, maxDrawn, maxProcessed, allowSplit, fs, counters,
                   warpSums, total);
}

// One work item of the fine pass: a tile, or one group of depth bins of a
// split tile.  The last group to finish merges the tile; where a later group
// could fill a pool, the tile is drawn in order instead, from the end of the first
// group.  The longest tiles in order are what a frame of long lists waits for
// (200,000 x 32 at 4K: ~160 rounds of 11 us after the first group's ~90): with the
// whole tile drawn again after the last group had taken its bins a second time with
// exact counts, 4.2 ms; from the first group's end, with the undecided groups
// settled from their bounds, 2.6 ms.
template <int TS, int MAXL>
__device__ __forceinline__ void fineItem(FineSmem<TS>& sh, const HfbUniforms& U, const FineArgs& a,
                                         const uint32_t* __restrict__ tileList, float* __restrict__ result,
                                         const FineScratch fs, const uint4 item) {
  using SM = FineSmem<TS>;
  constexpr uint32_t NT = SM::NT;
  const uint32_t tid = threadIdx.x;
  const uint32_t lx = tid % TS, ly = tid / TS;
  const uint32_t W = f2u(U.viewport.x), H = f2u(U.viewport.y);
  const uint32_t tilesX = divCeil(W, TS), tileCount = tilesX * divCeil(H, TS);
  float4* res = reinterpret_cast<float4*>(result + 4);
  {
    if (item.x >= tileCount) {  // not an entry of the tile list: count it and skip
      if (tid == 0) atomicAdd(HFB_G(&a.counters->badWorkItems), 1ull);
      return;
    }
    const uint32_t tileIdx = (*HFB_G(&tileList[1u + item.x]));
    uint32_t b0 = item.y & 0xffu, b1 = (item.y >> 8) & 0xffu;
    const uint32_t g = (item.y >> 16) & 0xffu, nG = item.y >> 24;
    if (tileIdx >= tileCount || b1 > a.B || b0 >= b1) return;
    bool split = nG > 1u, write = true;
    if (split && (g >= nG || item.z >= fs.maxGroups || nG > fs.maxGroups - item.z || item.w == 0u || item.w >= a.B)) {
      // not an item the schedule writes: count it and leave the tile alone
      if (tid == 0) atomicAdd(HFB_G(&a.counters->badWorkItems), 1ull);
      return;
    }
    f4 fin;
    FinePart part = split && g > 0u ? FINE_QUICK : FINE_IN_ORDER;
    const float4* resume = nullptr;
    uint32_t* word = split ? &fs.arrivals[item.z] : nullptr;
    while (true) {
      const FineEnd end = fineTile<TS, MAXL>(sh, U, a, tileIdx, b0, b1, part, resume, fin);
      if (end == FINE_AGAIN) {  // uniform
        part = FINE_CAREFUL;
        __syncthreads();
        continue;
      }
      if (!split) break;
      // A group of a split tile: publish its composite; the last to arrive merges.  Where
      // a later group could fill a pool, the tile is drawn in order instead: from the end
      // of the first group, which is in order already, by whoever finds both that it is
      // there and that a group gave up.
      (*HFB_G(&fs.groups[(size_t)(item.z + g) * NT + tid])) = make_float4(fin.x, fin.y, fin.z, fin.w);
      __threadfence();
      __syncthreads();
      if (tid == 0) {
        uint32_t todo = 0, old;
        if (end != FINE_OK) {  // a later group: the count never fills up, so nobody merges
          old = atomicOr(HFB_G(word), FINE_REDO);
          if ((old & (FINE_FIRST | FINE_REDO)) == FINE_FIRST) todo = 2u;
        } else {
          old = atomicAdd(HFB_G(word), g == 0u ? (FINE_FIRST + 1u) | (sh.filled << FINE_FILLED_SHIFT) : 1u);
          if (old & FINE_REDO) todo = g == 0u ? 2u : 0u;
          else if ((old & 0xffffu) + 1u == nG) todo = 1u;
        }
        const uint32_t filled = g == 0u ? sh.filled : (old & FINE_FILLED) >> FINE_FILLED_SHIFT;
        if (todo == 2u) {
          atomicAdd(HFB_G(&a.counters->fineSplitRedone), 1ull);
          // the bins before the point where the tile is taken up count once more, as if drawn again
          if (filled) atomicAdd(HFB_G(&a.counters->finePoolFullBins), (unsigned long long)filled);
        }
        sh.arrive = todo;
      }
      __syncthreads();
      const uint32_t m = sh.arrive;
      if (m == 0u) { write = false; break; }
      if (m == 2u) {
        __threadfence();
        b0 = item.w;
        b1 = a.B;
        resume = fs.groups + (size_t)item.z * NT;
        split = false;
        part = FINE_IN_ORDER;
        __syncthreads();
        continue;
      }
      __threadfence();
      // front-to-back "over" of the groups' composites, each pixel stopping
      // where the reference stops (isPixelDone, alpha >= 0.999)
      const float4 f0 = __ldcg(HFB_G(&fs.groups[(size_t)item.z * NT + tid]));
      fin = mk4(f0.x, f0.y, f0.z, f0.w);
      for (uint32_t g2 = 1; g2 < nG; g2++) {
        const float4 c = __ldcg(HFB_G(&fs.groups[(size_t)(item.z + g2) * NT + tid]));
        if (fin.w < 0.999f) {
          const float k = fsub(1.0f, fin.w);
          fin.x = fadd(fin.x, fmul(c.x, k));
          fin.y = fadd(fin.y, fmul(c.y, k));
          fin.z = fadd(fin.z, fmul(c.z, k));
          fin.w = fadd(fin.w, fmul(c.w, k));
        }
      }
      break;
    }
    const uint32_t tx = tileIdx % tilesX, ty = tileIdx / tilesX;
    const TileB tbp = tileBoundsPx(W, H, TS, tx, ty);
    const uint32_t px = tbp.x0 + lx, py = tbp.y0 + ly;
    if (write && px < W && py < H) (*HFB_G(&res[(size_t)py * W + px])) = make_float4(fin.x, fin.y, fin.z, fin.w);
  }
}

template <int TS, int MAXL>
__global__ void __launch_bounds__(TS * TS, TS == 8 ? (MAXL <= 4 ? 8 : 6) : TS == 16 ? (MAXL <= 4 ? 3 : 2) : 1)
fineKernel(const HfbUniforms U, const FineArgs a, const uint32_t* __restrict__ tileList, float* __restrict__ result,
           FineScratch fs) {
  using SM = FineSmem<TS>;
  extern __shared__ __align__(16) unsigned char fineSmemRaw[];
  SM& sh = *reinterpret_cast<SM*>(fineSmemRaw);
  const uint32_t nItems = min((*HFB_G(&fs.hdr[0])), fs.maxItems);
  uint32_t* queue = reinterpret_cast<uint32_t*>(result);  // tileQueueAtomicIdx, getNextTileIdx :294-303
  // The device functions get the uniforms and the arguments from shared
  // memory, never an address of a kernel parameter (whose generic address
  // lies in the parameter space, which instructions for global memory
  // reject: error 717, invalid address space).
  __shared__ HfbUniforms Us;
  for (uint32_t w = threadIdx.x; w < sizeof(HfbUniforms) / 4u; w += blockDim.x)
    reinterpret_cast<uint32_t*>(&Us)[w] = reinterpret_cast<const uint32_t*>(&U)[w];
  if (threadIdx.x == 0) sh.args = a;
  while (true) {
    if (threadIdx.x == 0) sh.queueIdx = atomicAdd(HFB_G(queue), 1u);
    __syncthreads();
    const uint32_t it = sh.queueIdx;
    if (it >= nItems) break;
    fineItem<TS, MAXL>(sh, Us, sh.args, tileList, result, fs, (*HFB_G(&fs.items[it])));
    __syncthreads();  // the tile's shared state is rewritten for the next item
  }
}

// batched: one queue over the work items of every instance
template <int TS, int MAXL>
__global__ void __launch_bounds__(TS * TS, TS == 8 ? (MAXL <= 4 ? 8 : 6) : TS == 16 ? (MAXL <= 4 ? 3 : 2) : 1)
fineBatch(BatchView b, FineArgs base, HfbConfig cfgParam) {
  using SM = FineSmem<TS>;
  const HfbConfig cfg = cfgParam;
  extern __shared__ __align__(16) unsigned char fineSmemRaw[];
  SM& sh = *reinterpret_cast<SM*>(fineSmemRaw);
  const uint32_t n = b.hdr->n;
  const uint32_t total = b.itemPrefix[n];
  while (true) {
    if (threadIdx.x == 0) {
      const uint32_t gi = atomicAdd(&b.hdr->fineQueue, 1u);
      sh.queueIdx = gi;
      if (gi < total) {  // the item's instance, for every thread of the CTA
        const BatchInst& I = b.insts[batchFind(b.itemPrefix, n, gi)];
        FineArgs a = base;
        a.S = I.S;
        a.P = I.P;
        a.pos = I.posNew;
        a.tan = I.tan;
        a.shading = I.shading;
        a.depth = I.depth;
        a.tiles = I.tiles;
        a.segBuf = I.segBuf;
        a.proj = I.proj;
        sh.args = a;
      }
    }
    __syncthreads();
    const uint32_t gi = sh.queueIdx;
    if (gi >= total) break;
    const uint32_t i = batchFind(b.itemPrefix, n, gi);
    const BatchInst& I = b.insts[i];
    const FineScratch fs = fineScratchLayout(I.scratch, cfg, I.W, I.H);
    const uint32_t li = gi - b.itemPrefix[i];
    if (li < fs.maxItems) fineItem<TS, MAXL>(sh, I.U, sh.args, I.tileList, I.result, fs, (*HFB_G(&fs.items[li])));
    __syncthreads();
  }
}

// CTAs that the schedule shares a frame's records out over.
template <int TS, int MAXL>
uint32_t fineShare(const HfbCtx* c) {
  return c->cfg.processorCount ? c->cfg.processorCount
                               : FineDims<TS>::CTAS[MAXL == 4 ? 0 : MAXL == 8 ? 1 : 2] * (uint32_t)c->smCount;
}

template <int TS, int MAXL>
cudaError_t launchFineT(HfbCtx* c, const HfbUniforms& u, const HfbHairData& h, const float* pos,
                        const float* tan, const float* shading, const float* depth, HfbRasterBuffers& rb,
                        const float4* proj) {
  HFB_CHECK_BIND(c);
  const HfbConfig& cfg = c->cfg;
  constexpr size_t SMEM = FINE_SMEM<TS, MAXL>;
  int& perSM = c->fineBlocksPerSM[TS == 8 ? 0 : TS == 16 ? 1 : 2][MAXL == 4 ? 0 : MAXL == 8 ? 1 : 2];
  if (perSM == 0) {
    cudaError_t e = cudaFuncSetAttribute(fineKernel<TS, MAXL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM);
    if (e == cudaSuccess)
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, fineKernel<TS, MAXL>, TS * TS, SMEM);
    if (e != cudaSuccess) return e;
    if (perSM < 1) return cudaErrorInvalidConfiguration;
  }
  const uint32_t grid = cfg.processorCount ? cfg.processorCount : (uint32_t)(perSM * c->smCount);
  const uint32_t share = fineShare<TS, MAXL>(c);
  const uint32_t T = divCeil(rb.width, TS) * divCeil(rb.height, TS);
  const uint32_t dispMode = u.displayMode & 0xffu;
  const bool dbg = dispMode == 4u && ((u.displayMode >> 8) & 0xffffu) != 0u;
  FineScratch fs = fineScratchLayout(rb.scratch, cfg, rb.width, rb.height);
  fineScheduleKernel<<<1, 1024, 0, c->stream>>>(rb.tileList, rb.segmentCountPerTile, (const uint4*)rb.tiles, T,
                                                cfg.tileDepthBins, share, rb.maxDrawnSegments,
                                                h.strandsCount * h.pointsPerStrand, dbg ? 0u : 1u, fs,
                                                (DeviceCounters*)c->dCounters);
  HFB_AFTER_LAUNCH(c, "fineScheduleKernel");
  FineArgs a;
  a.S = h.strandsCount;
  a.P = h.pointsPerStrand;
  a.B = cfg.tileDepthBins;
  a.L = cfg.slicesPerPixel;
  a.SP = cfg.shadingPoints;
  a.CAP = cfg.avgFragmentsPerSlice * cfg.slicesPerPixel * cfg.tileSize * cfg.tileSize;
  a.alphaQuadratic = cfg.alphaQuadratic;
  a.alphaMul = cfg.alphaMultiplier;
  a.pos = (const float4*)pos;
  a.tan = (const float4*)tan;
  a.shading = (const float4*)shading;
  a.depth = depth;
  a.tiles = (const uint4*)rb.tiles;
  a.segBuf = rb.tileSegments;
  a.counters = (DeviceCounters*)c->dCounters;
  a.proj = proj;
  fineKernel<TS, MAXL><<<grid, TS * TS, SMEM, c->stream>>>(u, a, rb.tileList, rb.rasterizerResult, fs);
  HFB_AFTER_LAUNCH(c, "fineKernel");
  c->launches += 2;
  return cudaGetLastError();
}


// ---------------------------------------------------------------------------
// Batched tiles pass, tile sort and fine pass: persistent over the virtual
// blocks of every instance (hfb_frame_batch).
// ---------------------------------------------------------------------------
#define BATCH_LOOP(KIND)                                              \
  const uint32_t n = b.hdr->n;                                        \
  const uint32_t* row = b.prefix + (KIND) * (BATCH_MAX + 1);          \
  const uint32_t totalVb = row[n];                                    \
  __shared__ uint32_t vbNext[2];                                      \
  uint32_t vbPar = 0;                                                 \
  for (uint32_t v = batchNext(b.hdr, (KIND), vbNext, vbPar); v < totalVb; \
       v = batchNext(b.hdr, (KIND), vbNext, vbPar)) {                 \
    const uint32_t i = batchFind(row, n, v);                          \
    const BatchInst& I = b.insts[i];                                  \
    if (!HFB_EXPECT(i < n && I.W && I.H && I.W <= 65536 && I.H <= 65536 && I.scratch && I.segBuf && \
                    I.T == divCeil(I.W, cfg.tileSize) * divCeil(I.H, cfg.tileSize))) continue; \
    const uint32_t local = v - row[i], nLocal = row[i + 1] - row[i];  \
    (void)nLocal; (void)local;                                        \
    const TilesScratch ts = tilesScratchLayout(I.scratch, cfg, I.W, I.H, I.maxDrawn); \
    (void)ts;

template <bool WIDE>
__global__ void __launch_bounds__(TR_SEGS, 6) tilesRasterBatch(BatchView b, HfbConfig cfgParam,
                                                             DeviceCounters* __restrict__ counters) {
  const HfbConfig cfg = cfgParam;
  __shared__ TrShared sh;
  BATCH_LOOP(BK_RASTER)
    tilesRasterBody<WIDE>(I.U, I.P, min(I.strandsToRender, I.S), cfg.tileSize, cfg.tileDepthBins,
                    cfg.invalidTilesPerSegmentThreshold, I.bsphere, I.posNew, I.tan, I.depth, I.tiles, I.segBuf,
                    I.segCount, ts.binCount, counters, sh, local, I.proj);
  }
}

__global__ void __launch_bounds__(512) binScanBatch(BatchView b, HfbConfig cfgParam) {
  const HfbConfig cfg = cfgParam;
  __shared__ uint32_t warpSums[32];
  BATCH_LOOP(BK_SCAN)
    binScanBlocksBody(ts.binCount, ts.binOffset, ts.blockSums, I.T * cfg.tileDepthBins, warpSums, local);
  }
}

__global__ void __launch_bounds__(1024) binScanSumsBatch(BatchView b, HfbConfig cfgParam) {
  const HfbConfig cfg = cfgParam;
  __shared__ uint32_t warpSums[32];
  BATCH_LOOP(BK_SCAN_SUMS)
    binScanSumsBody(ts.blockSums, divCeil(I.T * cfg.tileDepthBins, SCAN_PER_BLOCK), warpSums);
    __syncthreads();
  }
}

__global__ void __launch_bounds__(256) binScatterBatch(BatchView b, HfbConfig cfgParam,
                                                        DeviceCounters* __restrict__ counters) {
  const HfbConfig cfg = cfgParam;
  BATCH_LOOP(BK_SCATTER)
    binScatterBody(I.segBuf, I.maxDrawn, ts.binOffset, ts.blockSums, ts.keys, counters, local, nLocal,
                   I.T * cfg.tileDepthBins);
  }
}

__global__ void __launch_bounds__(256) binFinalizeBatch(BatchView b, HfbConfig cfgParam) {
  const HfbConfig cfg = cfgParam;
  __shared__ uint32_t smem[8 * WARP_BIN];
  BATCH_LOOP(BK_FINALIZE)
    binFinalizeBody(I.T * cfg.tileDepthBins, ts.binCount, ts.binOffset, ts.blockSums, ts.keys, I.segBuf, I.tiles,
                    ts.largeBins, smem, local, nLocal);
  }
}

__global__ void __launch_bounds__(1024) largeBinsBatch(BatchView b, HfbConfig cfgParam) {
  const HfbConfig cfg = cfgParam;
  extern __shared__ uint32_t sk[];
  BATCH_LOOP(BK_LARGE)
    largeBinsBody(ts.largeBins, ts.binCount, ts.binOffset, ts.blockSums, ts.keys, I.segBuf, I.tiles, sk, local,
                  nLocal);
  }
}

__global__ void __launch_bounds__(1024) tileSortBatch(BatchView b, HfbConfig cfgParam) {
  const HfbConfig cfg = cfgParam;
  __shared__ SortShared ss;
  BATCH_LOOP(BK_SORT)
    tileSortBody(I.T, cfg.sortBuckets, cfg.sortBucketSize, I.segCount, I.sortBuckets, I.tileList, ss);
    __syncthreads();
  }
}

__global__ void __launch_bounds__(1024) fineScheduleBatch(BatchView b, HfbConfig cfgParam, uint32_t grid,
                                                          DeviceCounters* __restrict__ counters) {
  const HfbConfig cfg = cfgParam;
  __shared__ uint32_t warpSums[32];
  __shared__ uint32_t totalRecords;
  BATCH_LOOP(BK_SCHEDULE)
    const FineScratch fs = fineScratchLayout(I.scratch, cfg, I.W, I.H);
    const uint32_t dispMode = I.U.displayMode & 0xffu;
    const bool dbg = dispMode == 4u && ((I.U.displayMode >> 8) & 0xffffu) != 0u;
    fineScheduleBody(I.tileList, I.segCount, I.tiles, I.T, cfg.tileDepthBins, grid, I.maxDrawn, I.S * I.P,
                     dbg ? 0u : 1u, fs, counters, warpSums, totalRecords);
  }
}

// Exclusive prefix of the instances' work items; resets the batch queue.
__global__ void __launch_bounds__(1024) fineItemPrefixBatch(BatchView b, HfbConfig cfgParam) {
  const HfbConfig cfg = cfgParam;
  __shared__ uint32_t warpSums[32];
  const uint32_t n = b.hdr->n;
  uint32_t carry = 0;
  for (uint32_t i0 = 0; i0 < n; i0 += blockDim.x) {
    const uint32_t i = i0 + threadIdx.x;
    uint32_t items = 0;
    if (i < n) {
      const BatchInst& I = b.insts[i];
      items = (*HFB_G(&fineScratchLayout(I.scratch, cfg, I.W, I.H).hdr[0]));
    }
    uint32_t chunk;
    const uint32_t ex = blockExclusiveScan(items, warpSums, chunk);
    if (i < n) b.itemPrefix[i] = carry + ex;
    carry += chunk;
  }
  if (threadIdx.x == 0) {
    b.itemPrefix[n] = carry;
    b.hdr->fineQueue = 0;
  }
}
#undef BATCH_LOOP

template <int TS, int MAXL>
cudaError_t launchFineBatchT(HfbCtx* c, const BatchView& b) {
  HFB_CHECK_BIND(c);
  const HfbConfig& cfg = c->cfg;
  constexpr size_t SMEM = FINE_SMEM<TS, MAXL>;
  uint32_t& grid = c->batchGrid[BK_COUNT];  // the fine kernel's persistent grid
  if (!grid) {
    cudaError_t e = cudaFuncSetAttribute(fineBatch<TS, MAXL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM);
    int per = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fineBatch<TS, MAXL>, TS * TS, SMEM);
    if (e != cudaSuccess) return e;
    if (per < 1) return cudaErrorInvalidConfiguration;
    grid = cfg.processorCount ? cfg.processorCount : (uint32_t)per * c->smCount;
  }
  DeviceCounters* dc = (DeviceCounters*)c->dCounters;
  uint32_t& sgrid = c->batchGrid[BK_SCHEDULE];
  if (!sgrid) sgrid = c->smCount;
  fineScheduleBatch<<<batchLaunchGrid(c, sgrid), 1024, 0, c->stream>>>(b, cfg, batchLaunchGrid(c, fineShare<TS, MAXL>(c)), dc);
  HFB_AFTER_LAUNCH(c, "fineScheduleBatch");
  fineItemPrefixBatch<<<1, 1024, 0, c->stream>>>(b, cfg);
  HFB_AFTER_LAUNCH(c, "fineItemPrefixBatch");
  FineArgs a{};
  a.B = cfg.tileDepthBins;
  a.L = cfg.slicesPerPixel;
  a.SP = cfg.shadingPoints;
  a.CAP = cfg.avgFragmentsPerSlice * cfg.slicesPerPixel * cfg.tileSize * cfg.tileSize;
  a.alphaQuadratic = cfg.alphaQuadratic;
  a.alphaMul = cfg.alphaMultiplier;
  a.counters = dc;
  fineBatch<TS, MAXL><<<batchLaunchGrid(c, grid), TS * TS, SMEM, c->stream>>>(b, a, cfg);
  HFB_AFTER_LAUNCH(c, "fineBatch");
  c->launches += 3;
  return cudaGetLastError();
}

}  // namespace

cudaError_t launchTilesPass(HfbCtx* c, const HfbUniforms& u, const HfbHairData& h, const float* pos,
                            const float* tan, const float* depth, uint32_t strandsToRender, HfbRasterBuffers& rb,
                            float4* proj, bool cleared) {
  HFB_CHECK_BIND(c);
  const HfbConfig& cfg = c->cfg;
  const uint32_t W = rb.width, H = rb.height, TS = cfg.tileSize, B = cfg.tileDepthBins;
  const uint32_t T = divCeil(W, TS) * divCeil(H, TS);
  const uint32_t TB = T * B;
  TilesScratch s = tilesScratchLayout(rb.scratch, cfg, W, H, rb.maxDrawnSegments);
  cudaError_t e = cudaSuccess;
  if (!cleared) {
    e = cudaMemsetAsync(s.binCount, 0, (size_t)TB * 4, c->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(s.largeBins, 0, 8, c->stream);
    if (e != cudaSuccess) return e;
  }
  const uint32_t nStrands = min(strandsToRender, h.strandsCount);
  const uint32_t nSeg = nStrands * (h.pointsPerStrand - 1u);
  DeviceCounters* dc = (DeviceCounters*)c->dCounters;
  if (nSeg) {
    float4 bs = make_float4(h.boundingSphere[0], h.boundingSphere[1], h.boundingSphere[2], h.boundingSphere[3]);
    (rasterWide(cfg) ? tilesRasterKernel<true> : tilesRasterKernel<false>)<<<divCeil(nSeg, TR_SEGS), TR_SEGS, 0, c->stream>>>(
        u, h.pointsPerStrand, nStrands, TS, B, cfg.invalidTilesPerSegmentThreshold, bs, (const float4*)pos,
        (const float4*)tan, depth, (uint4*)rb.tiles, rb.tileSegments, rb.segmentCountPerTile, s.binCount, dc, proj);
    HFB_AFTER_LAUNCH(c, "tilesRasterKernel");
  }
  if (c->rasterDone && (e = cudaEventRecord(c->rasterDone, c->stream)) != cudaSuccess) return e;
  const uint32_t nBlocks = divCeil(TB, SCAN_PER_BLOCK);
  binScanKernel<<<nBlocks, 512, 0, c->stream>>>(s.binCount, s.binOffset, s.blockSums, &s.largeBins[1], TB);
  HFB_AFTER_LAUNCH(c, "binScanKernel");
  binScatterKernel<<<c->smCount * 8, 256, 0, c->stream>>>(rb.tileSegments, rb.maxDrawnSegments, s.binOffset,
                                                          s.blockSums, s.keys, dc, TB);
  HFB_AFTER_LAUNCH(c, "binScatterKernel");
  binFinalizeKernel<<<min(divCeil(TB, 8), (uint32_t)c->smCount * 7), 256, 0, c->stream>>>(
      TB, s.binCount, s.binOffset, s.blockSums, s.keys, rb.tileSegments, (uint4*)rb.tiles, s.largeBins);
  HFB_AFTER_LAUNCH(c, "binFinalizeKernel");
  if (!c->largeBinsAttrSet) {
    e = cudaFuncSetAttribute(largeBinsKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, LARGE_SMEM_KEYS * 4);
    if (e != cudaSuccess) return e;
    c->largeBinsAttrSet = true;
  }
  // two CTAs of 64 KB per SM: 758 bins of up to 34,187 records 475 -> 400 us
  largeBinsKernel<<<c->smCount * 2, 1024, LARGE_SMEM_KEYS * 4, c->stream>>>(
      s.largeBins, s.binCount, s.binOffset, s.blockSums, s.keys, rb.tileSegments, (uint4*)rb.tiles);
  HFB_AFTER_LAUNCH(c, "largeBinsKernel");
  c->launches += nSeg ? 5 : 4;
  return cudaGetLastError();
}

// Loads the tiles pass's kernels onto the current device and sets the
// large-bins kernel's shared-memory attribute.  CUDA loads device code
// lazily, at a kernel's first launch or attribute query, and loading takes
// device memory for the code; hfb_tiles_pass_noalloc's set-up calls this at
// context creation so that its own launches load (allocate) nothing.
cudaError_t tilesPassLoad(HfbCtx* c) {
  cudaFuncAttributes a;
  cudaError_t e = cudaFuncGetAttributes(&a, rasterWide(c->cfg) ? tilesRasterKernel<true> : tilesRasterKernel<false>);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, binScanKernel);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, binScatterKernel);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, binFinalizeKernel);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, largeBinsKernel);
  if (e == cudaSuccess && !c->largeBinsAttrSet) {
    e = cudaFuncSetAttribute(largeBinsKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, LARGE_SMEM_KEYS * 4);
    if (e == cudaSuccess) c->largeBinsAttrSet = true;
  }
  return e;
}

cudaError_t launchTileSort(HfbCtx* c, HfbRasterBuffers& rb) {
  HFB_CHECK_BIND(c);
  const HfbConfig& cfg = c->cfg;
  const uint32_t T = divCeil(rb.width, cfg.tileSize) * divCeil(rb.height, cfg.tileSize);
  if (cfg.sortBuckets > SORT_MAX_BUCKETS) return cudaErrorInvalidValue;
  tileSortKernel<<<1, 1024, 0, c->stream>>>(T, cfg.sortBuckets, cfg.sortBucketSize, rb.segmentCountPerTile,
                                            rb.sortBuckets, rb.tileList);
  HFB_AFTER_LAUNCH(c, "tileSortKernel");
  c->launches += 1;
  return cudaGetLastError();
}

cudaError_t launchFinePass(HfbCtx* c, const HfbUniforms& u, const HfbHairData& h, const float* pos,
                           const float* tan, const float* shading, const float* depth, HfbRasterBuffers& rb,
                           const float4* proj) {
  const uint32_t TS = c->cfg.tileSize, L = c->cfg.slicesPerPixel;
  if (TS == 8) {
    if (L <= 4) return launchFineT<8, 4>(c, u, h, pos, tan, shading, depth, rb, proj);
    if (L <= 8) return launchFineT<8, 8>(c, u, h, pos, tan, shading, depth, rb, proj);
    return launchFineT<8, 16>(c, u, h, pos, tan, shading, depth, rb, proj);
  }
  if (TS == 16) {
    if (L <= 4) return launchFineT<16, 4>(c, u, h, pos, tan, shading, depth, rb, proj);
    if (L <= 8) return launchFineT<16, 8>(c, u, h, pos, tan, shading, depth, rb, proj);
    return launchFineT<16, 16>(c, u, h, pos, tan, shading, depth, rb, proj);
  }
  if (L <= 4) return launchFineT<32, 4>(c, u, h, pos, tan, shading, depth, rb, proj);
  if (L <= 8) return launchFineT<32, 8>(c, u, h, pos, tan, shading, depth, rb, proj);
  return cudaErrorInvalidValue;  // 32x32 tiles with more than 8 slices: too many registers per pixel
}

}  // namespace hfb

namespace hfb {

cudaError_t launchBatchTiles(HfbCtx* c, const BatchView& b) {
  HFB_CHECK_BIND(c);
  const HfbConfig& cfg = c->cfg;
  DeviceCounters* dc = (DeviceCounters*)c->dCounters;
  uint32_t* g = c->batchGrid;
  const auto raster = rasterWide(cfg) ? tilesRasterBatch<true> : tilesRasterBatch<false>;
  if (!g[BK_RASTER]) {
    int per = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, raster, TR_SEGS, 0);
    if (e != cudaSuccess) return e;
    g[BK_RASTER] = (uint32_t)(per > 0 ? per : 1) * c->smCount;
    g[BK_SCAN] = c->smCount * 4u;
    g[BK_SCAN_SUMS] = c->smCount;
    g[BK_SCATTER] = c->smCount * 8u;
    g[BK_FINALIZE] = c->smCount * 8u;
    g[BK_LARGE] = c->smCount * 2u;
    e = cudaFuncSetAttribute(largeBinsBatch, cudaFuncAttributeMaxDynamicSharedMemorySize, LARGE_SMEM_KEYS * 4);
    if (e != cudaSuccess) return e;
  }
  raster<<<batchLaunchGrid(c, g[BK_RASTER]), TR_SEGS, 0, c->stream>>>(b, cfg, dc);
  HFB_AFTER_LAUNCH(c, "tilesRasterBatch");
  if (c->rasterDone) {
    const cudaError_t e = cudaEventRecord(c->rasterDone, c->stream);
    if (e != cudaSuccess) return e;
  }
  binScanBatch<<<batchLaunchGrid(c, g[BK_SCAN]), 512, 0, c->stream>>>(b, cfg);
  HFB_AFTER_LAUNCH(c, "binScanBatch");
  binScanSumsBatch<<<batchLaunchGrid(c, g[BK_SCAN_SUMS]), 1024, 0, c->stream>>>(b, cfg);
  HFB_AFTER_LAUNCH(c, "binScanSumsBatch");
  binScatterBatch<<<batchLaunchGrid(c, g[BK_SCATTER]), 256, 0, c->stream>>>(b, cfg, dc);
  HFB_AFTER_LAUNCH(c, "binScatterBatch");
  binFinalizeBatch<<<batchLaunchGrid(c, g[BK_FINALIZE]), 256, 0, c->stream>>>(b, cfg);
  HFB_AFTER_LAUNCH(c, "binFinalizeBatch");
  largeBinsBatch<<<batchLaunchGrid(c, g[BK_LARGE]), 1024, LARGE_SMEM_KEYS * 4, c->stream>>>(b, cfg);
  HFB_AFTER_LAUNCH(c, "largeBinsBatch");
  c->launches += 6;
  return cudaGetLastError();
}

cudaError_t launchBatchSort(HfbCtx* c, const BatchView& b) {
  HFB_CHECK_BIND(c);
  if (c->cfg.sortBuckets > SORT_MAX_BUCKETS) return cudaErrorInvalidValue;
  uint32_t& grid = c->batchGrid[BK_SORT];
  if (!grid) grid = c->smCount;
  tileSortBatch<<<batchLaunchGrid(c, grid), 1024, 0, c->stream>>>(b, c->cfg);
  HFB_AFTER_LAUNCH(c, "tileSortBatch");
  c->launches += 1;
  return cudaGetLastError();
}

cudaError_t launchBatchFine(HfbCtx* c, const BatchView& b) {
  const uint32_t TS = c->cfg.tileSize, L = c->cfg.slicesPerPixel;
  if (TS == 8) {
    if (L <= 4) return launchFineBatchT<8, 4>(c, b);
    if (L <= 8) return launchFineBatchT<8, 8>(c, b);
    return launchFineBatchT<8, 16>(c, b);
  }
  if (TS == 16) {
    if (L <= 4) return launchFineBatchT<16, 4>(c, b);
    if (L <= 8) return launchFineBatchT<16, 8>(c, b);
    return launchFineBatchT<16, 16>(c, b);
  }
  if (L <= 4) return launchFineBatchT<32, 4>(c, b);
  if (L <= 8) return launchFineBatchT<32, 8>(c, b);
  return cudaErrorInvalidValue;
}

}  // namespace hfb
