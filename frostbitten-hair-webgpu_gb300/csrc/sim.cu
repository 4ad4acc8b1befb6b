// Simulation passes: GridPreSimPass, HairSimIntegrationPass, GridPostSimPass.
//
// Reference WGSL: src/passes/simulation/{gridPreSimPass,hairSimIntegrationPass,
// gridPostSimPass}.wgsl.ts with shaderImpl/{integration,constraints,
// collisions}.wgsl.ts and grids/*.wgsl.ts.  All arithmetic follows the fixed
// fp32 order of hfb_math.cuh, so results are reproducible run to run; the
// grid splat is integer (i32 fixed point, wrapping adds), hence order-free.
#define HFB_TU 1
#include <algorithm>
#include <atomic>

#include "hfb_internal.cuh"
#include "hfb_math.cuh"

namespace hfb {
namespace {

constexpr float GRID_MUL = 1000000.0f;  // GRID_FLOAT_TO_U32_MUL, grids.wgsl.ts:3
// SDF_SAMPLE_GRAD_OFFSET = SDF_CELL_SIZE * 0.1, collisions.wgsl.ts:23-24
// (abstract-float constant expression, rounded once to f32)
constexpr float SDF_GRAD_OFFSET = (float)(0.0033918858971446753 * 0.1);
constexpr float FLOAT_EPSILON = 1e-7f;

__device__ __forceinline__ int32_t gridEncode(float v) { return f2i(fmul(v, GRID_MUL)); }

// Conversions by an addition, which float <-> integer instructions and roundings run at a
// quarter of the rate of (grid pre-sim 453 -> 414 us, integration 2.75 -> 2.70 ms on the
// 64-instance frame, 159 -> 147 us on 40,000 x 16 alone; the splat's encoding, where they
// take five instructions each, was slower: 1.15 -> 1.26 ms, and keeps the conversion).
// x + 1.5 * 2^23, rounded down or up, has floor(x) or ceil(x) in its low bits and leaves
// it as a float when the constant is taken off again: exact for |x| < 2^22.
constexpr float WHOLE = 12582912.0f;  // 0x4b400000
__device__ __forceinline__ int32_t wholeInt(float t) { return (int32_t)(__float_as_uint(t) - 0x4b400000u); }

// Division by the constants 1e6 and 3 as a correctly rounded multiplication
// by the reciprocal, RN(x * Ch + RN(x * Cl)) with Ch + Cl the reciprocal split
// into two floats (Brisebarre and Muller, "Correctly rounded multiplication by
// arbitrary precision constants", IEEE Trans. Computers 57(2), 2008): one
// multiply and one FMA instead of an IEEE division.  For these two constants
// it gives the IEEE quotient x / d bit for bit for every finite x with
// |x| >= 2^-92 (d = 1e6) and |x| > 2^-123 (d = 3); hfb_check_constant_division
// compares it with the device's division over all 2^32 inputs.
constexpr float RCP_1E6_HI = 0x1.0c6f7ap-20f, RCP_1E6_LO = 0x1.6bdb1ap-49f;
constexpr float RCP_3_HI = 0x1.555556p-2f, RCP_3_LO = -0x1.555556p-27f;
__device__ __forceinline__ float mulRcp(float x, float hi, float lo) { return __fmaf_rn(x, hi, fmul(x, lo)); }

// (float)v / 1e6: a converted i32 is 0 or at least 1 in magnitude
__device__ __forceinline__ float gridDecode(int32_t v) { return mulRcp((float)v, RCP_1E6_HI, RCP_1E6_LO); }
// The same for |v| < 2^22, the conversion by a subtraction.
__device__ __forceinline__ float gridDecodeSmall(int32_t v) {
  return mulRcp(fsub(__uint_as_float(0x4b400000u + (uint32_t)v), WHOLE), RCP_1E6_HI, RCP_1E6_LO);
}

__device__ __forceinline__ float divBy3(float x) {
  const float a = fabsf(x);
  return a > 0x1p-123f && a < INFINITY ? mulRcp(x, RCP_3_HI, RCP_3_LO) : x / 3.0f;
}
__device__ __forceinline__ f3 div3sBy3(f3 v) {
  const float lo = fminf(fminf(fabsf(v.x), fabsf(v.y)), fabsf(v.z)), hi = fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fabsf(v.z));
  if (lo > 0x1p-123f && hi < INFINITY)  // one test for the three
    return {mulRcp(v.x, RCP_3_HI, RCP_3_LO), mulRcp(v.y, RCP_3_HI, RCP_3_LO), mulRcp(v.z, RCP_3_HI, RCP_3_LO)};
  return {divBy3(v.x), divBy3(v.y), divBy3(v.z)};
}

__device__ __forceinline__ uint32_t gridIdx(uint32_t G, uint32_t x, uint32_t y, uint32_t z) {
  return clampu(z, 0u, G - 1u) * G * G + clampu(y, 0u, G - 1u) * G + clampu(x, 0u, G - 1u);
}

struct GridCo {
  uint32_t mn[3], mx[3];
  f3 p;
};

// _getGridCell, grids.wgsl.ts:43-56
__device__ __forceinline__ GridCo gridCell(uint32_t G, f3 bmin, f3 bmax, f3 p) {
  f3 t = sat3(div3(sub3(p, bmin), sub3(bmax, bmin)));
  float g = (float)(G - 1u);
  GridCo r;
  r.p = mul3s(t, g);
  // floor and ceil of coordinates in [0, G - 1]
  r.mn[0] = wholeInt(__fadd_rd(r.p.x, WHOLE)); r.mx[0] = wholeInt(__fadd_ru(r.p.x, WHOLE));
  r.mn[1] = wholeInt(__fadd_rd(r.p.y, WHOLE)); r.mx[1] = wholeInt(__fadd_ru(r.p.y, WHOLE));
  r.mn[2] = wholeInt(__fadd_rd(r.p.z, WHOLE)); r.mx[2] = wholeInt(__fadd_ru(r.p.z, WHOLE));
  return r;
}

// _getGridCellWeights, grids.wgsl.ts:58-66
__device__ __forceinline__ f3 cellWeights(uint32_t x, uint32_t y, uint32_t z, f3 p) {
  return {clampf(fsub(1.0f, fabsf(fsub(p.x, (float)x))), 0.0f, 1.0f),
          clampf(fsub(1.0f, fabsf(fsub(p.y, (float)y))), 0.0f, 1.0f),
          clampf(fsub(1.0f, fabsf(fsub(p.z, (float)z))), 0.0f, 1.0f)};
}

// sampleSDFCollider (sdfCollider.ts:36-44) with the linear / clamp-to-edge
// sampler of sdfUtils.ts:33-42, as an exact fp32 trilinear filter with texel
// centres at (i + 0.5) / D.
__device__ __forceinline__ float sampleSDF(const float* __restrict__ sdf, uint32_t D, f3 bmin, f3 bmax, f3 p) {
  f3 t = sat3(div3(sub3(p, bmin), sub3(bmax, bmin)));
  float fD = (float)D;
  float u = fsub(fmul(t.x, fD), 0.5f), v = fsub(fmul(t.y, fD), 0.5f), w = fsub(fmul(t.z, fD), 0.5f);
  // floor of coordinates in [-0.5, D - 0.5]
  const float tu = __fadd_rd(u, WHOLE), tv = __fadd_rd(v, WHOLE), tw = __fadd_rd(w, WHOLE);
  float ax = fsub(u, fsub(tu, WHOLE)), ay = fsub(v, fsub(tv, WHOLE)), az = fsub(w, fsub(tw, WHOLE));
  int m = (int)D - 1;
  int x0 = wholeInt(tu), y0 = wholeInt(tv), z0 = wholeInt(tw);
  int x1 = min(max(x0 + 1, 0), m), y1 = min(max(y0 + 1, 0), m), z1 = min(max(z0 + 1, 0), m);
  x0 = min(max(x0, 0), m); y0 = min(max(y0, 0), m); z0 = min(max(z0, 0), m);
  // D <= 1024: indices below 2^30
  auto row = [&](int y, int z) { return sdf + (uint32_t)((z * (int)D + y) * (int)D); };
  const float *r00 = row(y0, z0), *r10 = row(y1, z0), *r01 = row(y0, z1), *r11 = row(y1, z1);
  float c00 = mixf(__ldg(HFB_G(r00 + x0)), __ldg(HFB_G(r00 + x1)), ax);
  float c10 = mixf(__ldg(HFB_G(r10 + x0)), __ldg(HFB_G(r10 + x1)), ax);
  float c01 = mixf(__ldg(HFB_G(r01 + x0)), __ldg(HFB_G(r01 + x1)), ax);
  float c11 = mixf(__ldg(HFB_G(r11 + x0)), __ldg(HFB_G(r11 + x1)), ax);
  return mixf(mixf(c00, c10, ay), mixf(c01, c11, ay), az);
}

__device__ __forceinline__ f3 gridMin(const HfbSimUniforms& u) {
  return mk3(u.gridData.boundsMin.x, u.gridData.boundsMin.y, u.gridData.boundsMin.z);
}
__device__ __forceinline__ f3 gridMax(const HfbSimUniforms& u) {
  return mk3(u.gridData.boundsMax[0], u.gridData.boundsMax[1], u.gridData.boundsMax[2]);
}

// ---------------------------------------------------------------------------
// GridPreSimPass.main, gridPreSimPass.wgsl.ts:38-159 (one thread per node)
// ---------------------------------------------------------------------------
__device__ __forceinline__ void gridPreSimBody(const HfbSimUniforms& u, uint32_t G, const int4* __restrict__ dv,
                                               float4* __restrict__ gw, const float* __restrict__ sdf, uint32_t D,
                                               uint32_t id) {
  if (id >= G * G * G) return;
  uint32_t z = id / (G * G);
  uint32_t idXY = id - z * G * G;
  uint32_t y = idXY / G, x = idXY % G;
  f3 gmin = gridMin(u), gmax = gridMax(u);
  f3 cell = div3s(sub3(gmax, gmin), (float)(G - 1u));
  f3 pos = add3(gmin, mul3(cell, mk3((float)x, (float)y, (float)z)));
  f3 smin = mk3(u.sdf.boundsMin.x, u.sdf.boundsMin.y, u.sdf.boundsMin.z);
  f3 smax = mk3(u.sdf.boundsMax.x, u.sdf.boundsMax.y, u.sdf.boundsMax.z);
  // getWindStrength, :89-108
  float wind;
  float d = sampleSDF(sdf, D, smin, smax, pos);
  if (d < 0.0f) {
    wind = 0.0f;
  } else {
    f3 nd = norm3(mk3(u.wind.x, u.wind.y, u.wind.z));
    f3 toward = mk3(-nd.x, -nd.y, -nd.z);
    f3 rp = add3(pos, mul3s(mul3s(toward, d), u.windColisionTraceOffset));
    wind = sampleSDF(sdf, D, smin, smax, rp) < 0.0f ? 0.5f : 1.0f;
  }
  // getDensityGradient, :111-159
  uint32_t idx0 = gridIdx(G, x, y, z);
  float d0 = gridDecode(__ldg(HFB_G(&dv[idx0].w)));
  f3 g = mk3(0.0f, 0.0f, 0.0f);
  const int off[6][3] = {{1, 0, 0}, {-1, 0, 0}, {0, 1, 0}, {0, -1, 0}, {0, 0, 1}, {0, 0, -1}};
#pragma unroll
  for (int k = 0; k < 6; k++) {
    int ox = (int)x + off[k][0], oy = (int)y + off[k][1], oz = (int)z + off[k][2];
    f3 r = mk3(0.0f, 0.0f, 0.0f);
    if (!(ox < 0 || oy < 0 || oz < 0)) {
      uint32_t idxO = gridIdx(G, (uint32_t)ox, (uint32_t)oy, (uint32_t)oz);
      if (idxO != idx0) {
        float dO = gridDecode(__ldg(HFB_G(&dv[idxO].w)));
        float m = fmaxf(fsub(d0, dO), 0.0f);
        r = mul3s(mk3((float)off[k][0], (float)off[k][1], (float)off[k][2]), m);
      }
    }
    g = add3(g, r);
  }
  *HFB_G(&gw[idx0]) = make_float4(g.x, g.y, g.z, wind);
}

__global__ void __launch_bounds__(256) gridPreSimKernel(const HfbSimUniforms u, uint32_t G, const int4* __restrict__ dv,
                                                        float4* __restrict__ gw, const float* __restrict__ sdf,
                                                        uint32_t D) {
  gridPreSimBody(u, G, dv, gw, sdf, D, blockIdx.x * blockDim.x + threadIdx.x);
}

// ---------------------------------------------------------------------------
// HairSimIntegrationPass.main, hairSimIntegrationPass.wgsl.ts:79-273
//
// A block holds NB strands' points in shared memory, laid out
// [strand][point + 1]: one thread per strand walks the Gauss-Seidel chains
// (length and local shape must stay sequential along the strand, as in the
// reference), and the whole block runs the per-point phases (Verlet and
// forces, global shape, sphere and SDF collisions) and the coalesced loads
// and stores.  The padding makes both access patterns conflict-free.
//
// The chains are latency-bound (each step waits on the last through a root and a
// quotient: overRoot), so what sets their speed is how many an SM walks at once,
// which shared memory bounds, and what a step waits for besides: the staged points
// (16 B each) are all that lives there, and where the weights are the usual ones
// (`plain`, below) a step reads nothing else but the segment lengths, four at a time
// where a strand's row is 16-byte aligned, a group ahead.  With other weights the
// bending constants go over the block's own points of the PREV buffer (each thread
// has read its point's previous position by then, and nothing else reads those
// addresses until the final positions overwrite them) and the chain loads them two
// steps ahead.  Against constants in PREV for every block, whose loads came from L2
// and held each bending step for about 340 cycles: 3.15 -> 2.71 ms (64 instances);
// with 256 threads, for the point phases, in the single-instance kernel: 309 -> 222 us
// (40,000 x 16, three passes), 175 -> 137 us (1,501 x 65); 512 threads 250 and 141 us;
// with blocks of a whole wave (simStrandsPerBlockFor) 180 and 132 us.
// Per block of the 64-instance frame (clock counters, before): Verlet 32 %, length
// chain 10 %, global shape 10 %, bending chain 19 %, collisions 29 %.
//
// A block of 128 threads of the batched kernel holds 1,536 points (48 strands of 32, 96
// of 16), seven blocks per SM: 336 strands of 32 points in flight per SM, and 70 KB of its
// L1 left for the Verlet phase's grid gathers.  Six blocks of 2,048 points left 50 KB:
// 12.05 -> 11.88 ms on the 64-instance frame, 1,183 -> 1,160 us on a tick of 6 sessions; six
// of 1,536 11.96, eight 11.98, seven of 1,280 12.09.
// ---------------------------------------------------------------------------
constexpr uint32_t SIM_THREADS = 256;        // threads per block of the single-instance kernel
constexpr uint32_t SIM_BATCH_THREADS = 128;  // and of the batched one (SIM_BATCH_BLOCKS per SM)


// p + z for z a signed zero whose sign is that of c xor the bit in s: p itself
// unless p is -0 and z is +0
__device__ __forceinline__ void zeroSum(float& p, float c, uint32_t s) {
  if (__float_as_uint(p) == 0x80000000u && ((__float_as_uint(c) ^ s) & 0x80000000u) == 0u) p = 0.0f;
}

// Verlet step of one point with the grid forces (:125-162, integration.wgsl.ts:8-28)
__device__ __forceinline__ float4 verletPoint(const HfbSimUniforms& u, uint32_t G, f3 gmin, f3 gmax,
                                              uint32_t strand, f4 posNow, f4 posPrev,
                                              const int4* __restrict__ dv, const float4* __restrict__ gw) {
  f3 force = mk3(0.0f, -u.gravity, 0.0f);
  const f3 pn = xyz(posNow);
  // _getGridDensityGradAndWind + _getGridDensityVelocity (same cell, two grids)
  GridCo co = gridCell(G, gmin, gmax, pn);
  f3 grad = mk3(0.f, 0.f, 0.f), vel = mk3(0.f, 0.f, 0.f);
  float windStr = 0.0f, dens = 0.0f;
  // one corner: node idx, its weights per axis and their length
  auto corner = [&](uint32_t idx, f3 w, float wl) {
    const float4 a = __ldg(HFB_G(&gw[idx]));
    const int4 b = __ldg(HFB_G(&dv[idx]));
    grad = add3(grad, mul3(w, mk3(a.x, a.y, a.z)));
    windStr = fadd(windStr, fmul(wl, a.w));
    // node velocities are small numbers of millionths, as a rule
    const uint32_t lim = 1u << 22;  // |v| < 2^22
    const f3 bv = max(max((uint32_t)b.x + lim, (uint32_t)b.y + lim), (uint32_t)b.z + lim) < 2u * lim
                      ? mk3(gridDecodeSmall(b.x), gridDecodeSmall(b.y), gridDecodeSmall(b.z))
                      : mk3(gridDecode(b.x), gridDecode(b.y), gridDecode(b.z));
    vel = add3(vel, mul3(w, bv));
    dens = fadd(dens, fmul(wl, gridDecode(b.w)));
  };
  if (co.mx[0] > co.mn[0] && co.mx[1] > co.mn[1] && co.mx[2] > co.mn[2]) {
    // inside a cell (no coordinate a whole number): eight corners, whose weights per axis
    // are two numbers in (0, 1) (cellWeights without its clamps) and whose squares are
    // summed once per pair of axes
    const f3 w0 = {fsub(1.0f, fabsf(fsub(co.p.x, (float)co.mn[0]))), fsub(1.0f, fabsf(fsub(co.p.y, (float)co.mn[1]))),
                   fsub(1.0f, fabsf(fsub(co.p.z, (float)co.mn[2])))};
    const f3 w1 = {fsub(1.0f, fabsf(fsub(co.p.x, (float)co.mx[0]))), fsub(1.0f, fabsf(fsub(co.p.y, (float)co.mx[1]))),
                   fsub(1.0f, fabsf(fsub(co.p.z, (float)co.mx[2])))};
    const uint32_t i0 = (co.mn[2] * G + co.mn[1]) * G + co.mn[0];
#pragma unroll
    for (uint32_t k = 0; k < 8u; k++) {
      const f3 w = {(k & 1u) ? w1.x : w0.x, (k & 2u) ? w1.y : w0.y, (k & 4u) ? w1.z : w0.z};
      corner(i0 + (k & 1u) + ((k & 2u) ? G : 0u) + ((k & 4u) ? G * G : 0u), w, len3(w));
    }
  } else {
    for (uint32_t z = co.mn[2]; z <= co.mx[2]; z++)
      for (uint32_t y = co.mn[1]; y <= co.mx[1]; y++)
        for (uint32_t x = co.mn[0]; x <= co.mx[0]; x++) {
          const f3 w = cellWeights(x, y, z, co.p);
          corner(gridIdx(G, x, y, z), w, len3(w));
        }
  }
  float timer = fadd(fmul((float)u.frameIdx, 0.73f), fmul(u.windPhaseOffset, (float)strand));
  float windJitter = fractf(fmul(timer, u.windStrengthFrequency));
  float jitterDelta = mixf(fmul(-0.5f, u.windStrengthJitter), fmul(0.5f, u.windStrengthJitter), windJitter);
  float jitterStr = fadd(1.0f, jitterDelta);
  float windCellStr = sat(mixf(u.windStrengthLull, 1.0f, windStr));
  force = add3(force, mul3s(mk3(u.wind.x, u.wind.y, u.wind.z),
                            fabsf(fmul(fmul(u.wind.w, jitterStr), windCellStr))));
  force = add3(force, mul3s(grad, u.volumePreservation));
  f3 gridDisp = dens > 0.0f ? div3s(vel, dens) : mk3(0.f, 0.f, 0.f);
  float dt = u.deltaTime;
  f3 pd = sub3(pn, xyz(posPrev));
  f3 fpd = mix3(pd, gridDisp, u.friction);
  f3 nxt = add3(add3(pn, fpd), mul3s(mul3s(force, dt), dt));
  f3 r = mix3(xyz(posPrev), nxt, posNow.w);
  return make_float4(r.x, r.y, r.z, posNow.w);
}

// applyCollisionsSphere, collisions.wgsl.ts:4-20: pushes pos out of the sphere by kColl.
__device__ __forceinline__ void sphereCollide(float4& pos, const f4 sph, float kColl, bool kCollFinite) {
  f3 v = mk3(fsub(pos.x, sph.x), fsub(pos.y, sph.y), fsub(pos.z, sph.z));
  const float l = len3(v);
  float dist = fsub(l, sph.w);
  float dts = fmaxf(0.0f, -dist);
  if (dts == 0.0f && l > 0.0f && l < INFINITY && kCollFinite) {
    // outside the sphere the correction (v / l) * dts * kColl is a signed zero, the sign
    // of v's component times those of dts and kColl; adding it changes only a -0
    // coordinate, into +0 when the zero is +0
    const uint32_t sz = (__float_as_uint(dts) ^ __float_as_uint(kColl)) & 0x80000000u;
    zeroSum(pos.x, v.x, sz); zeroSum(pos.y, v.y, sz); zeroSum(pos.z, v.z, sz);
  } else {
    f3 d = mul3s(mul3s(norm3(v), dts), kColl);
    pos.x = fadd(pos.x, d.x); pos.y = fadd(pos.y, d.y); pos.z = fadd(pos.z, d.z);
  }
}

// applyCollisionsSdf, collisions.wgsl.ts:23-61, given the distance d sampled at q (pos's xyz).
__device__ __forceinline__ void sdfPush(float4& pos, const f3 q, float d, const float* __restrict__ sdf, uint32_t D,
                                        const f3 smin, const f3 smax, float sdfOffset, float kSdf) {
  float dOff = fadd(d, sdfOffset);
  if (!(dOff >= 0.0f)) {
    const float o = SDF_GRAD_OFFSET;
    f3 cd;
    cd.x = sampleSDF(sdf, D, smin, smax, add3(q, mk3(fmul(o, 1.0f), fmul(o, 0.0f), fmul(o, 0.0f))));
    cd.y = sampleSDF(sdf, D, smin, smax, add3(q, mk3(fmul(o, 0.0f), fmul(o, 1.0f), fmul(o, 0.0f))));
    cd.z = sampleSDF(sdf, D, smin, smax, add3(q, mk3(fmul(o, 0.0f), fmul(o, 0.0f), fmul(o, 1.0f))));
    cd = sub3(cd, mk3(d, d, d));
    f3 corr = mul3s(norm3(cd), -dOff);
    f3 dd = mul3s(corr, kSdf);
    pos.x = fadd(pos.x, dd.x); pos.y = fadd(pos.y, dd.y); pos.z = fadd(pos.z, dd.z);
  }
}

// x / sqrt(d) for a chain step: root and quotient from one reciprocal square root
// (rootRecip), whose dependent chain is two thirds of an IEEE root and division's.
__device__ __forceinline__ float overRoot(float x, float d) {
  Recip l;
  const bool ok = rootRecip(d, l);
  const float q = divBy(x, l);
  if (ok && x >= DIV_TINY && x <= 0x1p25f) return q;
  return x / sqrtf(d);
}

// lengthStep between two movable points of weight 1: the products by the weights are
// the numbers themselves, and .w, which carries something else, stays as it is.
__device__ __forceinline__ void lengthStepMovable(float4* w, uint32_t j, float4& a, float expected, float kLen) {
  float4 b = w[j + 1u];
  const f3 tng = mk3(fsub(b.x, a.x), fsub(b.y, a.y), fsub(b.z, a.z));
  const float df = fmul(fmul(fsub(1.0f, overRoot(expected, dot3(tng, tng))), kLen), 0.5f);
  const f3 delta = mul3s(tng, df);
  a.x = fadd(a.x, delta.x); a.y = fadd(a.y, delta.y); a.z = fadd(a.z, delta.z);
  b.x = fsub(b.x, delta.x); b.y = fsub(b.y, delta.y); b.z = fsub(b.z, delta.z);
  w[j] = a;
  a = b;
}

// One step of the length chain (applyConstraint_length, constraints.wgsl.ts:5-28):
// segment j between a (point j, carried in registers) and point j + 1 of the
// staged strand w; writes point j and carries point j + 1 on in a.
__device__ __forceinline__ void lengthStep(float4* w, uint32_t j, float4& a, float w0, float w1, float expected,
                                           float kLen) {
  float4 b = w[j + 1u];
  f3 tng = mk3(fsub(b.x, a.x), fsub(b.y, a.y), fsub(b.z, a.z));
  float corr = fsub(1.0f, overRoot(expected, dot3(tng, tng)));
  // two movable points (the common case) make the divisor exactly 2: a halving, exact as a product
  const float num = fmul(corr, kLen), den = fadd(fadd(w0, w1), FLOAT_EPSILON);
  float df = den == 2.0f ? fmul(num, 0.5f) : num / den;
  f3 delta = mul3s(tng, df);
  a.x = fadd(a.x, fmul(delta.x, w0)); a.y = fadd(a.y, fmul(delta.y, w0)); a.z = fadd(a.z, fmul(delta.z, w0));
  b.x = fsub(b.x, fmul(w1, delta.x)); b.y = fsub(b.y, fmul(w1, delta.y)); b.z = fsub(b.z, fmul(w1, delta.z));
  w[j] = a;
  a = b;
}

// h0 of applyConstraint_localShape: the rest distance of a triplet's middle point from its centroid
__device__ __forceinline__ float restHeight(float4 i0, float4 i1, float4 i2) {
  const f3 c = div3sBy3(add3(add3(mk3(i0.x, i0.y, i0.z), mk3(i1.x, i1.y, i1.z)), mk3(i2.x, i2.y, i2.z)));
  return len3(sub3(c, mk3(i1.x, i1.y, i1.z)));
}

// One triplet of the bending chain: p0, p1, p2 move along the middle point's offset from
// the centroid by k0, k1, k2 times it (rest distance h0).
__device__ __forceinline__ void bendStep(float4& p0, float4& p1, float4& p2, float h0, float k0, float k1, float k2) {
  const f3 c = div3sBy3(add3(add3(mk3(p0.x, p0.y, p0.z), mk3(p1.x, p1.y, p1.z)), mk3(p2.x, p2.y, p2.z)));
  const f3 hv = sub3(mk3(p1.x, p1.y, p1.z), c);
  const f3 delta = mul3s(hv, fsub(1.0f, overRoot(h0, dot3(hv, hv))));
  const f3 d0 = mul3s(delta, k0), d1 = mul3s(delta, k1), d2 = mul3s(delta, k2);
  p0.x = fadd(p0.x, d0.x); p0.y = fadd(p0.y, d0.y); p0.z = fadd(p0.z, d0.z);
  p1.x = fadd(p1.x, d1.x); p1.y = fadd(p1.y, d1.y); p1.z = fadd(p1.z, d1.z);
  p2.x = fadd(p2.x, d2.x); p2.y = fadd(p2.y, d2.y); p2.z = fadd(p2.z, d2.z);
}

template <uint32_t NT>
__device__ __forceinline__ void simIntegrateBody(const HfbSimUniforms& u, uint32_t S, uint32_t P, uint32_t G,
                                                 float4* __restrict__ prev, const float4* __restrict__ now,
                                                 const float4* __restrict__ initial, const float* __restrict__ segLen,
                                                 const int4* __restrict__ dv, const float4* __restrict__ gw,
                                                 const float* __restrict__ sdf, uint32_t D, float4* simSmem,
                                                 uint32_t blk, uint32_t NB) {
  const uint32_t R = P + 1u;  // row stride (padded)
  float4* wk = simSmem;                                   // [NB][R] positions
  float* att = reinterpret_cast<float*>(wk + NB * R);     // [P] global-shape attenuation of point index j
  const uint32_t tid = threadIdx.x;
  const uint32_t s0 = blk * NB;
  const uint32_t nStr = min(NB, S - s0);
  const uint32_t nPts = nStr * P;
  const f3 gmin = gridMin(u), gmax = gridMax(u);
  // first point matchInitialTangent moves: the triplet loop ends at P - 3
  const uint32_t jTan = P >= 3u ? P - 3u : 0u;
  // the block's points of the PREV buffer: read once by the Verlet phase, then
  // the chain constants of each point, then the new positions
  float4* const lcg = prev + (size_t)s0 * P;

  // --- Verlet + forces and the chain constants, point-parallel ---
  // Where every strand of the block has a fixed root (weight 0) and movable points of
  // weight 1 (`plain`: what assets have), the weights need no storage: .w of a staged point
  // carries the only bending constant that differs from triplet to triplet, h0.
  bool plain = true;
#pragma unroll 2
  for (uint32_t i = tid; i < nPts; i += NT) {
    const uint32_t ls = i / P, pt = i - ls * P;
    const size_t gi = (size_t)s0 * P + i;
    const f4 posNow = ld4(__ldg(HFB_G(&now[gi])));
    float4 p = pt == 0u ? make_float4(posNow.x, posNow.y, posNow.z, posNow.w)
                        : verletPoint(u, G, gmin, gmax, s0 + ls, posNow, ld4(*HFB_G(&prev[gi])), dv, gw);
    const float4 i0 = __ldg(HFB_G(&initial[gi]));
    const uint32_t weight = pt == 0u ? 0u : 0x3f800000u;  // by the bits: a root of weight -0 keeps its sign
    plain = plain && __float_as_uint(posNow.w) == weight && __float_as_uint(i0.w) == weight;
    if (pt + 3u < P) p.w = restHeight(i0, __ldg(HFB_G(&initial[gi + 1u])), __ldg(HFB_G(&initial[gi + 2u])));
    wk[ls * R + pt] = p;
  }
  for (uint32_t j = tid; j < P; j += NT) {  // applyConstraint_global's attenuation (constraints.wgsl.ts:31-49)
    const float x = (float)j / (float)(P - 1u);
    att[j] = fsub(1.0f, sat(fsub(x, u.globalConstrExtent) / u.globalConstrFade));
  }
  // i / P for the block's points (i < NB * P <= 2048, P <= 256): floor(i * ceil(2^32 / P) / 2^32)
  // is exact there, the error i * (ceil(2^32 / P) * P - 2^32) < 2048 * 256 being far below 2^32
  const uint32_t divP = (uint32_t)((0x100000000ull + P - 1u) / P);
  plain = __syncthreads_and(plain) != 0;
  if (!plain) {  // other weights: .w is the point's, and the chain constants go over the block's points of PREV
    for (uint32_t i = tid; i < nPts; i += NT) {
      const uint32_t ls = i / P, pt = i - ls * P;
      const size_t gi = (size_t)s0 * P + i;
      wk[ls * R + pt].w = __ldg(HFB_G(&now[gi])).w;
      const float4 i0 = __ldg(HFB_G(&initial[gi]));
      float4 c = make_float4(0.f, 0.f, 0.f, 0.f);
      if (pt + 3u < P) {  // applyConstraint_localShape constants (constraints.wgsl.ts:54-99)
        const float4 i1 = __ldg(HFB_G(&initial[gi + 1u])), i2 = __ldg(HFB_G(&initial[gi + 2u]));
        const float wT = fadd(fadd(i0.w, fmul(2.0f, i1.w)), i2.w);
        c = make_float4(restHeight(i0, i1, i2), fmul(i0.w / wT, 2.0f), fmul(i1.w / wT, -4.0f), fmul(i2.w / wT, 2.0f));
      } else if (pt >= jTan && pt >= 1u) {  // applyConstraint_matchInitialTangent (:100-120)
        const float4 im = __ldg(HFB_G(&initial[gi - 1u]));
        c = make_float4(fsub(i0.x, im.x), fsub(i0.y, im.y), fsub(i0.z, im.z), 0.0f);
      }
      *HFB_G(&prev[gi]) = c;
    }
    __syncthreads();  // also makes the constants in PREV visible to the block's chain threads
  }

  const uint32_t iters = u.constraintIterations;
  const f3 smin = mk3(u.sdf.boundsMin.x, u.sdf.boundsMin.y, u.sdf.boundsMin.z);
  const f3 smax = mk3(u.sdf.boundsMax.x, u.sdf.boundsMax.y, u.sdf.boundsMax.z);
  const float sdfOffset = u.sdf.boundsMax.w;
  const f4 sph = mk4(u.collisionSphere.x, u.collisionSphere.y, u.collisionSphere.z, u.collisionSphere.w);
  const float kLen = u.stiffnessLengthConstr;
  // a strand's lengths load as float4s when its row starts on a 16-byte boundary
  const bool len4 = (P & 3u) == 0u && (reinterpret_cast<uintptr_t>(segLen) & 15u) == 0u;
  const float kGlob = u.stiffnessGlobalConstr / (float)iters;
  const float kLoc = u.stiffnessLocalConstr / (float)iters;
  const float kColl = u.stiffnessCollisions / (float)iters;
  const bool kCollFinite = fabsf(kColl) < INFINITY;
  const float kSdf = u.stiffnessSDF / (float)iters;
  for (uint32_t it = 0; it < iters; it++) {
    // length constraint (Gauss-Seidel), :176-190, constraints.wgsl.ts:5-28
    for (uint32_t ls = tid; ls < nStr; ls += NT) {
      float4* w = wk + ls * R;
      const float* L = segLen + (size_t)(s0 + ls) * P;
      float4 a = w[0];
      if (len4) {
        // the lengths of steps 4g .. 4g + 3 in one 16-byte load, the next group's issued
        // before this group's steps: four to seven steps ahead
        const float4* L4 = reinterpret_cast<const float4*>(L);
        const uint32_t NG = P >> 2;
        float4 cur = __ldg(HFB_G(&L4[0]));
        for (uint32_t g = 0; g < NG; g++) {
          const float4 nxt = g + 1u < NG ? __ldg(HFB_G(&L4[g + 1u])) : cur;
          const uint32_t j = g << 2;
          if (plain) {
            if (g) lengthStepMovable(w, j, a, cur.x, kLen); else lengthStep(w, 0u, a, 0.0f, 1.0f, cur.x, kLen);
            lengthStepMovable(w, j + 1u, a, cur.y, kLen);
            lengthStepMovable(w, j + 2u, a, cur.z, kLen);
            if (g + 1u < NG) lengthStepMovable(w, j + 3u, a, cur.w, kLen);  // step P - 1 does not exist
          } else {
            const uint32_t je = g + 1u < NG ? 4u : 3u;
#pragma unroll 1
            for (uint32_t e = 0; e < je; e++)
              lengthStep(w, j + e, a, a.w, w[j + e + 1u].w, e == 0u ? cur.x : e == 1u ? cur.y : e == 2u ? cur.z : cur.w, kLen);
          }
          cur = nxt;
        }
      } else {
        float expected = __ldg(HFB_G(&L[0])), nextExpected = __ldg(HFB_G(&L[1]));  // P >= 2
        for (uint32_t j = 0; j + 1u < P; j++) {
          const float nextExpected2 = j + 2u < P ? __ldg(HFB_G(&L[j + 2u])) : 0.0f;  // two steps ahead
          const float wa = plain ? (j ? 1.0f : 0.0f) : a.w, wb = plain ? 1.0f : w[j + 1u].w;
          lengthStep(w, j, a, wa, wb, expected, kLen);
          expected = nextExpected;
          nextExpected = nextExpected2;
        }
      }
      w[P - 1u] = a;
    }
    __syncthreads();
    // global shape, :193-206, constraints.wgsl.ts:31-49 (point-parallel)
#pragma unroll 2
    for (uint32_t i = tid; i < nPts; i += NT) {
      const uint32_t ls = __umulhi(i, divP), j = i - ls * P;
      if (j == 0u) continue;
      const float4 pi = __ldg(HFB_G(&initial[(size_t)s0 * P + i]));
      const float k = fmul(kGlob, att[j]);
      float4 p = wk[ls * R + j];
      f3 dvv = mk3(fsub(pi.x, p.x), fsub(pi.y, p.y), fsub(pi.z, p.z));
      if (!plain) dvv = mul3s(dvv, p.w);
      f3 d = mul3s(dvv, k);
      p.x = fadd(p.x, d.x); p.y = fadd(p.y, d.y); p.z = fadd(p.z, d.z);
      wk[ls * R + j] = p;
    }
    __syncthreads();
    // local shape (triangle bending, Gauss-Seidel), :209-232, constraints.wgsl.ts:54-120
    for (uint32_t ls = tid; ls < nStr; ls += NT) {
      float4* w = wk + ls * R;
      if (plain) {
        // the last three points' rest positions, for their tangents: loaded before the chain that
        // precedes them (4 <= P: checked by the entry points)
        const float4* E = initial + (size_t)(s0 + ls + 1u) * P - 4u;
        const float4 e0 = __ldg(HFB_G(&E[0])), e1 = __ldg(HFB_G(&E[1])), e2 = __ldg(HFB_G(&E[2])),
                     e3 = __ldg(HFB_G(&E[3]));
        float4 p0 = w[0], p1 = w[1], p2 = w[2];
        // the weights 0, 1, 1 of the triplet at the root; 1, 1, 1 of the others
        bendStep(p0, p1, p2, p0.w, fmul(kLoc, fmul(0.0f / 3.0f, 2.0f)), fmul(kLoc, fmul(1.0f / 3.0f, -4.0f)),
                 fmul(kLoc, fmul(1.0f / 3.0f, 2.0f)));
        w[0] = p0;
        float4 m = p0;  // the point before p1
        p0 = p1;
        p1 = p2;
        const float kEnd = fmul(kLoc, 0.5f), kMid = fmul(kLoc, -1.0f);
        for (uint32_t jj = 1; jj + 3u < P; jj++) {
          p2 = w[jj + 2u];
          bendStep(p0, p1, p2, p0.w, kEnd, kMid, kEnd);
          w[jj] = m = p0;
          p0 = p1;
          p1 = p2;
        }
        // matchInitialTangent of the points P - 3 (p0), P - 2 (p1) and P - 1, each from the one before
        auto tangentStep = [&](float4 p, const float4& ia, const float4& ib, uint32_t j) {
          const f3 proj = add3(mk3(m.x, m.y, m.z), mk3(fsub(ib.x, ia.x), fsub(ib.y, ia.y), fsub(ib.z, ia.z)));
          const f3 d = mul3s(sub3(proj, mk3(p.x, p.y, p.z)), kLoc);
          p.x = fadd(p.x, d.x); p.y = fadd(p.y, d.y); p.z = fadd(p.z, d.z);
          w[j] = m = p;
        };
        tangentStep(p0, e0, e1, P - 3u);
        tangentStep(p1, e1, e2, P - 2u);
        tangentStep(w[P - 1u], e2, e3, P - 1u);
        continue;
      }
      const float4* C = lcg + (size_t)ls * P;
      uint32_t jj = 0;
      if (P >= 3u) {
        float4 p0 = w[0], p1 = w[1];
        // the constants come from L2 (written this frame): loaded two steps ahead
        float4 cc = *HFB_G(&C[0]), ccNext = *HFB_G(&C[1]);
        for (; jj + 3u < P; jj++) {
          const float4 ccNext2 = *HFB_G(&C[jj + 2u]);  // jj + 2 < P
          float4 p2 = w[jj + 2u];
          bendStep(p0, p1, p2, cc.x, fmul(kLoc, cc.y), fmul(kLoc, cc.z), fmul(kLoc, cc.w));
          w[jj] = p0;
          p0 = p1;
          p1 = p2;
          cc = ccNext;
          ccNext = ccNext2;
        }
        w[jj] = p0;
        w[jj + 1u] = p1;
      }
      for (; jj < P; jj++) {  // applyConstraint_matchInitialTangent
        if (jj == 0u) continue;
        const float4 p0 = w[jj - 1u];
        float4 p1 = w[jj];
        const float4 t = *HFB_G(&C[jj]);
        f3 proj = add3(mk3(p0.x, p0.y, p0.z), mk3(t.x, t.y, t.z));
        f3 delta = sub3(proj, mk3(p1.x, p1.y, p1.z));
        f3 d = mul3s(delta, fmul(kLoc, p1.w));
        p1.x = fadd(p1.x, d.x); p1.y = fadd(p1.y, d.y); p1.z = fadd(p1.z, d.z);
        w[jj] = p1;
      }
    }
    __syncthreads();
    // collisions, :236-261, collisions.wgsl.ts:4-61 (point-parallel)
    for (uint32_t i = tid; i < nPts; i += NT) {
      const uint32_t ls = __umulhi(i, divP), j = i - ls * P;
      if (j == 0u) continue;
      float4 pos = wk[ls * R + j];
      sphereCollide(pos, sph, kColl, kCollFinite);
      if (j > 2u) {
        const f3 q = mk3(pos.x, pos.y, pos.z);
        sdfPush(pos, q, sampleSDF(sdf, D, smin, smax, q), sdf, D, smin, smax, sdfOffset, kSdf);
      }
      wk[ls * R + j] = pos;
    }
    __syncthreads();
  }
  // --- write back into the PREV buffer, coalesced (:268-272), over the chain constants ---
  for (uint32_t i = tid; i < nPts; i += NT) {
    const uint32_t ls = i / P, pt = i - ls * P;
    float4 p = wk[ls * R + pt];
    if (plain) p.w = pt == 0u ? 0.0f : 1.0f;
    *HFB_G(&prev[(size_t)s0 * P + i]) = p;
  }
  // the staging is rewritten by the CTA's next strands only after batchNext's barrier
}

__global__ void __launch_bounds__(SIM_THREADS, 3)
simIntegrateKernel(const HfbSimUniforms u, uint32_t S, uint32_t P, uint32_t G,
                   float4* __restrict__ prev, const float4* __restrict__ now,
                   const float4* __restrict__ initial, const float* __restrict__ segLen,
                   const int4* __restrict__ dv, const float4* __restrict__ gw,
                   const float* __restrict__ sdf, uint32_t D, uint32_t NB) {
  extern __shared__ float4 simSmem[];
  simIntegrateBody<SIM_THREADS>(u, S, P, G, prev, now, initial, segLen, dv, gw, sdf, D, simSmem, blockIdx.x, NB);
}

// ---------------------------------------------------------------------------
// GridPostSimPass.main, gridPostSimPass.wgsl.ts:45-72 with
// _addGridDensityVelocity, densityVelocityGrid.wgsl.ts:93-124.
//
// Each point adds to the eight corners of its cell, four wrapping i32 adds
// each.  A block takes GP_THREADS * PPT points, strand after strand in the order
// strandOrder gives (neighbouring strands next to each other: their points
// share grid nodes), a thread PPT consecutive ones: the points of a run
// in one cell sum their corner values in registers, each run's sums merge
// per grid node in a shared-memory hash table, and each node's four sums
// then go to global memory as one set of atomics.
// Wrapping integer sums do not depend on their order, so the grid is
// bit-exact whatever the strand order and the merge; an update that finds no
// free slot within GP_PROBES goes straight to global memory.
// ---------------------------------------------------------------------------
constexpr uint32_t GP_THREADS = 256;
constexpr uint32_t GP_PPT = 4;        // consecutive points per thread, at most
constexpr uint32_t GP_POINTS = GP_PPT * GP_THREADS;  // points per block of the batched kernel
constexpr uint32_t GP_HASH = 2048;    // slots (power of two)
constexpr uint32_t GP_PROBES = 32;
constexpr uint32_t GP_EMPTY = 0xffffffffu;
constexpr uint32_t GP_NO_CELL = 0xffffffffu;
constexpr uint32_t GP_BATCH_BLOCKS = 3;  // blocks per SM of the batched kernel (the run sums need registers)

struct GridPostShared {
  uint32_t key[GP_HASH];
  // the four sums of a slot in four arrays: slot h's words sit in bank h mod 32
  // (one uint4 per slot would put slots h and h + 8 in the same banks)
  unsigned vx[GP_HASH], vy[GP_HASH], vz[GP_HASH], vw[GP_HASH];
};

__device__ __forceinline__ void gridPostClear(GridPostShared& sh) {
  for (uint32_t e = threadIdx.x; e < GP_HASH; e += blockDim.x) {
    sh.key[e] = GP_EMPTY;
    sh.vx[e] = 0u; sh.vy[e] = 0u; sh.vz[e] = 0u; sh.vw[e] = 0u;
  }
}

__device__ __forceinline__ void gridPostAdd(GridPostShared& sh, unsigned* __restrict__ dv, uint32_t idx,
                                            uint4 v) {
  uint32_t h = (idx * 2654435761u) >> (32 - 11);  // Fibonacci hash into GP_HASH = 2^11 slots
  for (uint32_t p = 0; p < GP_PROBES; p++) {
    // a slot's key only ever changes from GP_EMPTY to a node index, so a plain read that finds the
    // node (the common case once its first add is in) needs no compare-and-swap
    uint32_t old = *reinterpret_cast<volatile const uint32_t*>(&sh.key[h]);
    if (old == GP_EMPTY) old = atomicCAS(&sh.key[h], GP_EMPTY, idx);
    if (old == GP_EMPTY || old == idx) {
      atomicAdd(&sh.vx[h], v.x);
      atomicAdd(&sh.vy[h], v.y);
      atomicAdd(&sh.vz[h], v.z);
      atomicAdd(&sh.vw[h], v.w);
      return;
    }
    h = (h + 1u) & (GP_HASH - 1u);
  }
  unsigned* c = reinterpret_cast<unsigned*>(HFB_G(reinterpret_cast<uint4*>(dv + 4u * idx)));
  atomicAdd(c + 0, v.x);
  atomicAdd(c + 1, v.y);
  atomicAdd(c + 2, v.z);
  atomicAdd(c + 3, v.w);
}

// Ordered points [blk * PPT * GP_THREADS, (blk + 1) * PPT * GP_THREADS) of the S * P: the
// ordered point v is point v % P of strand order[v / P].  The table is empty
// on entry and on exit.  All threads of the block call it.
template <uint32_t PPT>
__device__ __forceinline__ void gridPostSimBody(const HfbSimUniforms& u, uint32_t S, uint32_t P, uint32_t G,
                                                const float4* __restrict__ prev, const float4* __restrict__ now,
                                                unsigned* __restrict__ dv, const uint32_t* __restrict__ order,
                                                uint32_t blk, GridPostShared& sh) {
  const uint32_t N = S * P;
  const f3 gmin = gridMin(u), gmax = gridMax(u);
  // a thread's PPT consecutive ordered points: consecutive points that fall in
  // the same cell (mostly neighbours on one strand) add their corner values in
  // registers first (wrapping, as the table and the grid do), and the cell's sums
  // go to the table when the cell changes or the points end -- one set of table
  // adds per run of points.  A corner's share of the velocity's x depends on its x
  // alone, so the run's sums are two numbers per axis, and eight of the weights'
  // lengths; what a point adds to a corner that does not exist is never read
  // (32 sums, four per corner: 40,000 x 16, three passes, 180 -> 177 us; 64 instances
  // 12.32 -> 12.24 ms.  Points loaded one ahead, or 2,048 points per block: slower.)
  unsigned ax[2], ay[2], az[2], aw[8];
  uint32_t c0 = 0, c1 = 0, c2 = 0, cm = GP_NO_CELL;  // the cell being summed; cm: its corner mask
  const uint32_t vb = (blk * GP_THREADS + threadIdx.x) * PPT;
#pragma unroll 1
  for (uint32_t r = 0; r <= PPT; r++) {
    const uint32_t v = vb + r;
    const bool more = r < PPT && v < N;
    GridCo co;
    f3 vel;
    uint32_t m = GP_NO_CELL;
    if (more) {
      const uint32_t ls = v / P, j = v - ls * P;
      const uint32_t s = order ? min(__ldg(HFB_G(&order[ls])), S - 1u) : ls;
      const size_t i = (size_t)s * P + j;
      const float4 a = __ldg(HFB_G(&prev[i])), b = __ldg(HFB_G(&now[i]));
      const f3 pn = mk3(b.x, b.y, b.z);
      vel = sub3(pn, mk3(a.x, a.y, a.z));
      co = gridCell(G, gmin, gmax, pn);
      // corner k = x + 2y + 4z (offsets from mn) exists when each of its offsets is 0 or mx > mn there
      m = (co.mx[0] > co.mn[0] ? 1u : 0u) | (co.mx[1] > co.mn[1] ? 2u : 0u) | (co.mx[2] > co.mn[2] ? 4u : 0u);
    }
    if (!more || m != cm || co.mn[0] != c0 || co.mn[1] != c1 || co.mn[2] != c2) {
      if (cm != GP_NO_CELL) {
#pragma unroll
        for (uint32_t k = 0; k < 8u; k++)
          if ((k & ~cm) == 0u)
            gridPostAdd(sh, dv, gridIdx(G, c0 + (k & 1u), c1 + ((k >> 1) & 1u), c2 + (k >> 2)),
                        make_uint4(ax[k & 1u], ay[(k >> 1) & 1u], az[k >> 2], aw[k]));
      }
      if (!more) break;
#pragma unroll
      for (uint32_t k = 0; k < 2u; k++) ax[k] = ay[k] = az[k] = 0u;
#pragma unroll
      for (uint32_t k = 0; k < 8u; k++) aw[k] = 0u;
      c0 = co.mn[0]; c1 = co.mn[1]; c2 = co.mn[2]; cm = m;
    }
    const f3 w[2] = {cellWeights(co.mn[0], co.mn[1], co.mn[2], co.p),
                     cellWeights(co.mn[0] + 1u, co.mn[1] + 1u, co.mn[2] + 1u, co.p)};
#pragma unroll
    for (uint32_t k = 0; k < 2u; k++) {
      const f3 cv = mul3(vel, w[k]);
      ax[k] += (unsigned)gridEncode(cv.x);
      ay[k] += (unsigned)gridEncode(cv.y);
      az[k] += (unsigned)gridEncode(cv.z);
    }
#pragma unroll
    for (uint32_t k = 0; k < 8u; k++)
      aw[k] += (unsigned)gridEncode(len3(mk3(w[k & 1u].x, w[(k >> 1) & 1u].y, w[k >> 2].z)));
  }
  __syncthreads();
  for (uint32_t e = threadIdx.x; e < GP_HASH; e += blockDim.x) {
    const uint32_t idx = sh.key[e];
    if (idx == GP_EMPTY) continue;
    const uint4 v = make_uint4(sh.vx[e], sh.vy[e], sh.vz[e], sh.vw[e]);
    unsigned* c = reinterpret_cast<unsigned*>(HFB_G(reinterpret_cast<uint4*>(dv + 4u * idx)));
    atomicAdd(c + 0, v.x);
    atomicAdd(c + 1, v.y);
    atomicAdd(c + 2, v.z);
    atomicAdd(c + 3, v.w);
    sh.key[e] = GP_EMPTY;
    sh.vx[e] = 0u; sh.vy[e] = 0u; sh.vz[e] = 0u; sh.vw[e] = 0u;
  }
  // the next points' adds come after batchNext's barrier, with the table empty
}

template <uint32_t PPT>
__global__ void __launch_bounds__(GP_THREADS)
gridPostSimKernel(const HfbSimUniforms u, uint32_t S, uint32_t P, uint32_t G, const float4* __restrict__ prev,
                  const float4* __restrict__ now, unsigned* __restrict__ dv, const uint32_t* __restrict__ order) {
  __shared__ GridPostShared sh;
  gridPostClear(sh);
  __syncthreads();
  gridPostSimBody<PPT>(u, S, P, G, prev, now, dv, order, blockIdx.x, sh);
}

// ---- batched: persistent over the virtual blocks of every instance ----
// 5 blocks per SM (48 registers): 0.45 ms against 0.50 at 4 (64 registers) on the 64-instance frame
__global__ void __launch_bounds__(256, 5) gridPreSimBatch(BatchView b, uint32_t G) {
  const uint32_t n = b.hdr->n;
  const uint32_t* row = b.prefix + BK_GRID_PRE * (BATCH_MAX + 1);
  const uint32_t total = row[n];
  __shared__ uint32_t vbNext[2];
  uint32_t vbPar = 0;
  for (uint32_t v = batchNext(b.hdr, BK_GRID_PRE, vbNext, vbPar); v < total; v = batchNext(b.hdr, BK_GRID_PRE, vbNext, vbPar)) {
    const uint32_t i = batchFind(row, n, v);
    const BatchInst& I = b.insts[i];
    gridPreSimBody(I.SU, G, I.dv, I.gw, I.sdf, I.sdfDims, (v - row[i]) * 256u + threadIdx.x);
  }
}

__global__ void __launch_bounds__(SIM_BATCH_THREADS, SIM_BATCH_BLOCKS) simIntegrateBatch(BatchView b, uint32_t G) {
  extern __shared__ float4 simSmem[];
  const uint32_t n = b.hdr->n;
  const uint32_t* row = b.prefix + BK_INTEGRATE * (BATCH_MAX + 1);
  const uint32_t total = row[n];
  __shared__ uint32_t vbNext[2];
  uint32_t vbPar = 0;
  for (uint32_t v = batchNext(b.hdr, BK_INTEGRATE, vbNext, vbPar); v < total; v = batchNext(b.hdr, BK_INTEGRATE, vbNext, vbPar)) {
    const uint32_t i = batchFind(row, n, v);
    const BatchInst& I = b.insts[i];
    // integration reads positions[1 - current] (prev) and [current] (now), writes the former
    simIntegrateBody<SIM_BATCH_THREADS>(I.SU, I.S, I.P, G, I.posNew, I.posOld, I.initial, I.segLen, I.dv, I.gw, I.sdf, I.sdfDims,
                     simSmem, v - row[i], I.simNB);
  }
}

__global__ void __launch_bounds__(GP_THREADS, GP_BATCH_BLOCKS) gridPostSimBatch(BatchView b, uint32_t G) {
  __shared__ GridPostShared sh;
  gridPostClear(sh);
  __syncthreads();
  const uint32_t n = b.hdr->n;
  const uint32_t* row = b.prefix + BK_GRID_POST * (BATCH_MAX + 1);
  const uint32_t total = row[n];
  __shared__ uint32_t vbNext[2];
  uint32_t vbPar = 0;
  for (uint32_t v = batchNext(b.hdr, BK_GRID_POST, vbNext, vbPar); v < total; v = batchNext(b.hdr, BK_GRID_POST, vbNext, vbPar)) {
    const uint32_t i = batchFind(row, n, v);
    const BatchInst& I = b.insts[i];
    // after the swap: prev = the old current positions, now = the new ones
    gridPostSimBody<GP_PPT>(I.SU, I.S, I.P, G, I.posOld, I.posNew, (unsigned*)I.dv, I.gridOrder, v - row[i], sh);
  }
}


// Compares the reciprocal forms above with the IEEE division over all 2^32
// inputs: cnt[0] x / 3 over every non-NaN float, cnt[1] (float)v / 1e6 over
// every i32 v, cnt[2] x / 1e6 over every finite float with |x| >= 2^-92.
__global__ void __launch_bounds__(256) constDivCheckKernel(unsigned long long* __restrict__ cnt) {
  unsigned long long bad3 = 0, badGrid = 0, bad6 = 0;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < (1ull << 32); i += stride) {
    const uint32_t bits = (uint32_t)i;
    const float x = __uint_as_float(bits);
    if (x == x) {
      bad3 += __float_as_uint(divBy3(x)) != __float_as_uint(x / 3.0f);
      const float a = fabsf(x);
      if (a >= 0x1p-92f && a < INFINITY)
        bad6 += __float_as_uint(mulRcp(x, RCP_1E6_HI, RCP_1E6_LO)) != __float_as_uint(x / GRID_MUL);
    }
    const int32_t v = (int32_t)bits;
    badGrid += __float_as_uint(gridDecode(v)) != __float_as_uint((float)v / GRID_MUL);
  }
  if (bad3) atomicAdd(&cnt[0], bad3);
  if (badGrid) atomicAdd(&cnt[1], badGrid);
  if (bad6) atomicAdd(&cnt[2], bad6);
}

// Compares the quotients by a shared divisor (hfb_math.cuh) and the chains' overRoot with the
// device's IEEE operations, over every float d with numerators from a hash of d's bits and from
// the edges of what the forms take: cnt[0] rootRecip's root against sqrtf, cnt[1] overRoot
// against x / sqrtf(d), cnt[2] divBy against x / d for x in its range, cnt[3] the quotients
// by a root that took the short form (what the first two counts rest on).
constexpr uint32_t QC_EDGES = 16, QC_RANDOM = 16;
__global__ void __launch_bounds__(256) quotientCheckKernel(unsigned long long* __restrict__ cnt) {
  unsigned long long badRoot = 0, badOver = 0, badDiv = 0, shortForm = 0;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  // numerators that differ in their last bits, and at the ends of the ranges
  const uint32_t edges[QC_EDGES] = {0x3f800000u, 0x3f800001u, 0x3fffffffu, 0x3ffffffeu, 0x0d800000u, 0x0d7fffffu,
                                    0x0d800001u, 0x4c000000u, 0x4c000001u, 0x4bffffffu, 0x00000000u, 0x00000001u,
                                    0x007fffffu, 0x7f800000u, 0x7fc00000u, 0xbf800000u};
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < (1ull << 32); i += stride) {
    const float d = __uint_as_float((uint32_t)i);
    Recip l;
    const bool ok = rootRecip(d, l);
    const float root = sqrtf(d);
    if (ok) badRoot += __float_as_uint(l.d) != __float_as_uint(root);
    const Recip r = recipOf(d);
    const bool divides = r.y == r.y;  // d within recipOf's range
    uint32_t h = (uint32_t)i * 0x9e3779b9u + 0x7f4a7c15u;
#pragma unroll 1
    for (uint32_t k = 0; k < QC_EDGES + QC_RANDOM; k++) {
      h ^= h >> 15; h *= 0x2c1b3c6du; h ^= h >> 12; h *= 0x297a2d39u; h ^= h >> 15;
      uint32_t xb = h;
      if (k < QC_EDGES) xb = edges[k];
      const float x = __uint_as_float(xb);
      shortForm += ok && x >= DIV_TINY && x <= 0x1p25f;
      const float q = overRoot(x, d), want = x / root;
      badOver += __float_as_uint(q) != __float_as_uint(want) && (q == q || want == want);
      if (divides) {
        // exponents of x spread over [2^-100, 2^102): the quotients stay finite and normal
        const float y = k < QC_EDGES ? x : __uint_as_float((xb & 0x807fffffu) | ((27u + (xb >> 23) % 202u) << 23));
        const float b = fabsf(y), v = divBy(y, r), w = y / d;
        if (b == 0.0f) badDiv += fabsf(v) != 0.0f;
        else if (b >= DIV_TINY && b < 0x1p102f) badDiv += __float_as_uint(v) != __float_as_uint(w);
      }
    }
  }
  if (badRoot) atomicAdd(&cnt[0], badRoot);
  if (badOver) atomicAdd(&cnt[1], badOver);
  if (badDiv) atomicAdd(&cnt[2], badDiv);
  atomicAdd(&cnt[3], shortForm);
}

}  // namespace

cudaError_t launchQuotientCheck(HfbCtx* c, unsigned long long* cnt) {
  HFB_CHECK_BIND(c);
  cudaError_t e = cudaMemsetAsync(cnt, 0, 4 * sizeof(unsigned long long), c->stream);
  if (e != cudaSuccess) return e;
  quotientCheckKernel<<<c->smCount * 8u, 256, 0, c->stream>>>(cnt);
  HFB_AFTER_LAUNCH(c, "quotientCheckKernel");
  c->launches += 1;
  return cudaGetLastError();
}

cudaError_t launchConstDivCheck(HfbCtx* c, unsigned long long* cnt) {
  HFB_CHECK_BIND(c);
  cudaError_t e = cudaMemsetAsync(cnt, 0, 3 * sizeof(unsigned long long), c->stream);
  if (e != cudaSuccess) return e;
  constDivCheckKernel<<<c->smCount * 8u, 256, 0, c->stream>>>(cnt);
  HFB_AFTER_LAUNCH(c, "constDivCheckKernel");
  c->launches += 1;
  return cudaGetLastError();
}

cudaError_t launchGridPreSim(HfbCtx* c, const HfbSimUniforms& u, const int32_t* dv, float* gw,
                             const float* sdf, uint32_t sdfDims) {
  HFB_CHECK_BIND(c);
  uint32_t G = c->cfg.gridDims;
  uint32_t n = G * G * G;
  gridPreSimKernel<<<divCeil(n, 256), 256, 0, c->stream>>>(u, G, (const int4*)dv, (float4*)gw, sdf, sdfDims);
  HFB_AFTER_LAUNCH(c, "gridPreSimKernel");
  c->launches += 1;
  return cudaGetLastError();
}

// The dynamic shared memory limit of a kernel is a setting of the function
// for the whole process (per device), not of a context: contexts with
// different strand lengths would lower it under one another's launches.  It
// is raised once, to what the longest strands need.
static cudaError_t simSmemLimit(const void* fn, int which) {
  static std::atomic<uint64_t> done[2] = {};  // bit d: set on device d
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const uint64_t bit = 1ull << (dev & 63);
  if (done[which].load() & bit) return cudaSuccess;
  size_t most = 0;
  for (uint32_t P = 2; P <= 256; P++) most = std::max(most, simSmemBytes(P));
  e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
  if (e == cudaSuccess) done[which].fetch_or(bit);
  return e;
}

cudaError_t launchSimIntegrate(HfbCtx* c, const HfbSimUniforms& u, const HfbHairData& h, float* prev,
                               const float* now, const float* initial, const float* segLen,
                               const int32_t* dv, const float* gw, const float* sdf, uint32_t sdfDims) {
  HFB_CHECK_BIND(c);
  const uint32_t S = h.strandsCount, P = h.pointsPerStrand;
  // one instance alone rarely fills the GPU: its blocks take fewer strands (down to
  // 4), in whole waves of three blocks per SM, so that more chains run at once
  const uint32_t NB = simStrandsPerBlockFor(S, P, (uint32_t)c->smCount);
  const size_t smem = (size_t)NB * (P + 1u) * sizeof(float4) + (size_t)P * 4u;
  cudaError_t e = simSmemLimit((const void*)simIntegrateKernel, 0);
  if (e != cudaSuccess) return e;
  simIntegrateKernel<<<divCeil(S, NB), SIM_THREADS, smem, c->stream>>>(
      u, S, P, c->cfg.gridDims, (float4*)prev, (const float4*)now, (const float4*)initial, segLen,
      (const int4*)dv, (const float4*)gw, sdf, sdfDims, NB);
  HFB_AFTER_LAUNCH(c, "simIntegrateKernel");
  c->launches += 1;
  return cudaGetLastError();
}

cudaError_t launchBatchSim(HfbCtx* c, const BatchView& b, BatchKind k) {
  HFB_CHECK_BIND(c);
  const uint32_t G = c->cfg.gridDims;
  uint32_t& grid = c->batchGrid[k];
  if (k == BK_GRID_PRE) {
    if (!grid) grid = c->smCount * 8u;
    gridPreSimBatch<<<batchLaunchGrid(c, grid), 256, 0, c->stream>>>(b, G);
    HFB_AFTER_LAUNCH(c, "gridPreSimBatch");
  } else if (k == BK_INTEGRATE) {
    const size_t smem = c->simBatchSmem;  // the largest staging any batch of the context has needed
    if (!grid) {
      cudaError_t e = simSmemLimit((const void*)simIntegrateBatch, 1);
      int perSM = 0;
      if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, simIntegrateBatch, SIM_BATCH_THREADS, smem);
      if (e != cudaSuccess) return e;
      grid = (uint32_t)(perSM > 0 ? perSM : 1) * c->smCount;
    }
    simIntegrateBatch<<<batchLaunchGrid(c, grid), SIM_BATCH_THREADS, smem, c->stream>>>(b, G);
    HFB_AFTER_LAUNCH(c, "simIntegrateBatch");
  } else if (k == BK_GRID_POST) {
    if (!grid) {
      int perSM = 0;
      cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, gridPostSimBatch, GP_THREADS, 0);
      if (e != cudaSuccess) return e;
      grid = (uint32_t)(perSM > 0 ? perSM : 1) * c->smCount;
    }
    gridPostSimBatch<<<batchLaunchGrid(c, grid), GP_THREADS, 0, c->stream>>>(b, G);
    HFB_AFTER_LAUNCH(c, "gridPostSimBatch");
  } else {
    return cudaErrorInvalidValue;
  }
  c->launches += 1;
  return cudaGetLastError();
}

uint32_t gridPostBlocks(uint32_t points) { return divCeil(points, GP_POINTS); }

cudaError_t launchGridPostSim(HfbCtx* c, const HfbSimUniforms& u, const HfbHairData& h, const float* prev,
                              const float* now, int32_t* dv, const uint32_t* strandOrder) {
  HFB_CHECK_BIND(c);
  uint32_t G = c->cfg.gridDims;
  cudaError_t e = cudaMemsetAsync(dv, 0, (size_t)G * G * G * 16, c->stream);  // clearDensityVelocityBuffer
  if (e != cudaSuccess) return e;
  const uint32_t N = h.strandsCount * h.pointsPerStrand;
  if (N) {
    auto launch = [&](auto kernel, uint32_t ppt) {
      kernel<<<divCeil(N, ppt * GP_THREADS), GP_THREADS, 0, c->stream>>>(
          u, h.strandsCount, h.pointsPerStrand, G, (const float4*)prev, (const float4*)now, (unsigned*)dv, strandOrder);
    };
    // fewer points per thread where more would leave fewer than two blocks per SM: the
    // simulation of 1,501 x 65 (96 blocks of 1,024 points) 131 -> 119 us; from 305 blocks of
    // 1,024 on (10,000 x 32) longer runs are worth more: a frame 337 us, 344 at two points
    const uint32_t few = 2u * (uint32_t)c->smCount * GP_THREADS;  // points of one per thread
    if (N >= 4u * few) launch(gridPostSimKernel<4>, 4u);
    else if (N >= 2u * few) launch(gridPostSimKernel<2>, 2u);
    else launch(gridPostSimKernel<1>, 1u);
    HFB_AFTER_LAUNCH(c, "gridPostSimKernel");
    c->launches += 1;
  }
  return cudaGetLastError();
}

}  // namespace hfb
