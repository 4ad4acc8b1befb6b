// GTAO: AoPass (aoPass.wgsl.ts main_fs, gtao.wgsl.ts) as CUDA.
//
// Per AO texel (the AO texture is the viewport times the reference's
// textureSizeMul, 0.5; at that scale four threads, else one): the texel's full-resolution position
// ((x + 0.5) / scale), the normal there (rg16float octahedron, decoded as
// decodeOctahedronNormal does), and gtao(): for each of numDirections
// directions, numSteps steps each way, every sample reprojected to view
// space from the depth at its pixel (reprojectPositionToVS), the two horizon
// angles, and the cosine-weighted integral over the normal's slice.  The
// result is stored as r16float.  Texel loads outside the textures read 0
// (robust access); a negative coordinate saturates to 0 when converted to
// u32, as WGSL's conversion does.  Transcendentals (cos, sin, acos, inverse
// square root) are the CUDA library's, so results agree with the oracle to
// a tolerance, not bit for bit.
#define HFB_TU 9
#include <cuda_fp16.h>

#include "hfb_internal.cuh"
#include "hfb_math.cuh"

namespace hfb {
namespace {

constexpr float AO_PI = 3.141592653589793f;
constexpr float AO_HALF_PI = 1.5707963267948966f;
constexpr float AO_Z_NEAR = 0.01f;   // camera.projection.near
constexpr float AO_Z_FAR = 100.0f;   // camera.projection.far
constexpr float AO_SKY = 0.999f * AO_Z_FAR;  // view depths from here on are not occluded

struct AoCtx {
  const float* depth;
  uint32_t W, H;
  float vw, vh;
  const float* pinv;  // projMatrixInv
};

__device__ __forceinline__ uint32_t toU32(float v) { return f2u(v); }  // saturating, as WGSL u32(f32)

__device__ __forceinline__ float loadDepth(const AoCtx& a, float px, float py) {
  const uint32_t x = toU32(px), y = toU32(py);
  return x < a.W && y < a.H ? __ldg(HFB_G(&a.depth[(size_t)y * a.W + x])) : 0.0f;
}

// linearizeDepth, linearDepth.wgsl.ts:9-23
__device__ __forceinline__ float linearizeDepth(float d) {
  return fmul(AO_Z_NEAR, AO_Z_FAR) / fadd(AO_Z_FAR, fmul(fsub(AO_Z_NEAR, AO_Z_FAR), d));
}

// reprojectPositionToVS, gtao.wgsl.ts:23-39
__device__ __forceinline__ f3 reproject(const AoCtx& a, float px, float py) {
  const float d = loadDepth(a, px, py);
  const float x = fsub(fmul(px / a.vw, 2.0f), 1.0f), y = fsub(fmul(py / a.vh, 2.0f), 1.0f);
  const f4 c = m4v(a.pinv, mk4(x, y, d, 1.0f));
  return mk3(c.x / c.w, c.y / c.w, linearizeDepth(d));
}

__device__ __forceinline__ float roundF(float v) { return v < 0.5f ? floorf(v) : ceilf(v); }  // round_f

__device__ __forceinline__ f3 decodeOct(float fx0, float fy0) {  // decodeOctahedronNormal
  const float fx = fsub(fmul(fx0, 2.0f), 1.0f), fy = fsub(fmul(fy0, 2.0f), 1.0f);
  f3 n = mk3(fx, fy, fsub(fsub(1.0f, fabsf(fx)), fabsf(fy)));
  const float t = sat(-n.z);
  n.x = n.x >= 0.0f ? fsub(n.x, t) : fadd(n.x, t);
  n.y = n.y >= 0.0f ? fsub(n.y, t) : fadd(n.y, t);
  return norm3(n);
}

// View-space positions of a block's pixels and a halo around them, when the texels
// lie at whole pixels (scale 0.5: pixel 2 i + 1): a sample is then the position of a
// whole pixel, and each of those is reprojected once per block instead of once per
// sample that meets it.  AO_HALO covers the samples of up to 8 steps of one pixel (the
// default radius); farther ones are reprojected.
constexpr int AO_BX = 8, AO_BY = 8, AO_HALO = 10;  // texels of a block
constexpr int AO_TW = 2 * AO_BX + 2 * AO_HALO + 1, AO_TH = 2 * AO_BY + 2 * AO_HALO;  // an odd row stride
constexpr uint32_t AO_SPLIT = 4, AO_TERMS = 8;  // threads per texel, directions of each at most
constexpr uint32_t AO_THREADS = AO_BX * AO_BY * AO_SPLIT;
struct AoTile {
  float x[AO_TH * AO_TW], y[AO_TH * AO_TW], z[AO_TH * AO_TW];
  float term[AO_TERMS][AO_THREADS];  // each thread's directions' terms
};

// The terms of directions [i0, i1) of a texel that is not sky, given to emit in turn.
template <bool TILE, class Emit>
__device__ __forceinline__ void gtao(const HfbUniforms& U, const AoCtx& a, float px, float py, f3 normalWS, f3 posVS,
                                     const AoTile* tile, int at, uint32_t i0, uint32_t i1, Emit emit) {
  const auto& P = U.ao;
  auto tilePos = [&](int i) { return mk3(tile->x[i], tile->y[i], tile->z[i]); };
  f3 nVS = xyz(m4v(U.viewMatrix.m, mk4(normalWS.x, normalWS.y, normalWS.z, 1.0f)));
  nVS.z = -nVS.z;
  const f3 toCam = norm3(mk3(-posVS.x, -posVS.y, -posVS.z));
  const float nSteps = (float)P.numSteps;
  const float radius = fmaxf(nSteps, fmul(P.radius, posVS.z / AO_Z_FAR));
  const float stepSize = radius / nSteps;
  const float rotJitter =
      fmul(AO_PI, fractf(fmul(52.9829189f, fractf(fadd(fmul(px, 0.06711056f), fmul(py, 0.00583715f))))));
  const float jitterMod = fmul(fadd(px, py), 0.25f);
  const float radiusJitter = fmul(fmul(fractf(jitterMod), stepSize), 0.25f);
  // gtaoFalloff's divisor is the same for every sample (divBy on the tile, where its range allows)
  const float s2 = P.falloffStart2, fd = fsub(P.falloffEnd2, s2);
  const Recip fr = s2 >= 1e-6f && s2 <= 1e6f ? recipOf(fd) : Recip{fd, __int_as_float(0x7fffffff)};
  auto horizon = [&](f3 s, float h) {
    const f3 ws = sub3(s, posVS);
    const float d2 = len3(ws);
    const float c = fmul(dot3(ws, toCam), rsqrtf(d2));
    const float n = fsub(d2, s2);
    float q;
    if constexpr (TILE) {
      q = divBy(n, fr);
      if (!(fabsf(q) < 1e30f)) q = n / fd;
    } else {  // hidden behind a sample's reprojection: 33 directions at 1080p 1,446 us, by divBy 1,456
      q = n / fd;
    }
    return fmaxf(h, fsub(c, fmul(2.0f, sat(q))));
  };
  for (uint32_t i = i0; i < i1; i++) {
    float phi = fadd(fmul((float)i, AO_PI / (float)P.numDirections), fmul(P.directionOffset, AO_PI));
    phi = fadd(phi, rotJitter);
    float step = fadd(1.0f, fmul(0.25f, stepSize));
    step = fadd(step, radiusJitter);
    const float dx = cosf(phi), dy = sinf(phi);
    float h1 = -1.0f, h2 = -1.0f;
    for (uint32_t j = 0; j < P.numSteps; j++) {
      const float ox = roundF(fmul(dx, step)), oy = roundF(fmul(dy, step));
      if (TILE && fabsf(ox) <= (float)AO_HALO && fabsf(oy) <= (float)AO_HALO) {
        const int d = (int)oy * AO_TW + (int)ox;
        h1 = horizon(tilePos(at + d), h1);
        h2 = horizon(tilePos(at - d), h2);
      } else {
        h1 = horizon(reproject(a, fadd(px, ox), fadd(py, oy)), h1);
        h2 = horizon(reproject(a, fsub(px, ox), fsub(py, oy)), h2);
      }
      step = fadd(step, stepSize);
    }
    h1 = acosf(h1);
    h2 = acosf(h2);
    const f3 dir = mk3(dx, dy, 0.0f);
    const f3 bit = norm3(cross3(dir, toCam));
    const f3 tng = cross3(toCam, bit);
    const f3 nx = sub3(nVS, mul3s(bit, dot3(nVS, bit)));
    const float nnx = len3(nx);
    const float nnxInv = 1.0f / fadd(nnx, 1e-6f);
    const float cosxi = fmul(dot3(nx, tng), nnxInv);
    const float gamma = fsub(acosf(cosxi), AO_HALF_PI);
    const float cosgamma = fmul(dot3(nx, toCam), nnxInv);
    const float singamma2 = fmul(-2.0f, cosxi);
    h1 = fadd(gamma, fmaxf(fsub(-h1, gamma), -AO_HALF_PI));
    h2 = fadd(gamma, fminf(fsub(h2, gamma), AO_HALF_PI));
    const float t1 = fsub(fadd(fmul(h1, singamma2), cosgamma), cosf(fsub(fmul(2.0f, h1), gamma)));
    const float t2 = fsub(fadd(fmul(h2, singamma2), cosgamma), cosf(fsub(fmul(2.0f, h2), gamma)));
    emit(i, fmul(fmul(nnx, 0.25f), fadd(t1, t2)));
  }
}

// The normal of the pixel under full-resolution position (px, py).
__device__ __forceinline__ f3 normalAt(const AoCtx& a, const float2* __restrict__ normals, float px, float py) {
  const uint32_t nx = toU32(px), ny = toU32(py);
  const float2 no = nx < a.W && ny < a.H ? __ldg(HFB_G(&normals[(size_t)ny * a.W + nx])) : make_float2(0.f, 0.f);
  return decodeOct(no.x, no.y);
}

__device__ __forceinline__ float r16(float v) { return __half2float(__float2half_rn(v)); }  // the r16float texture

__device__ __forceinline__ AoCtx aoCtx(const HfbUniforms& U, const float* depth) {
  AoCtx a;
  a.depth = depth;
  a.W = f2u(U.viewport.x);
  a.H = f2u(U.viewport.y);
  a.vw = U.viewport.x;
  a.vh = U.viewport.y;
  a.pinv = U.projMatrixInv.m;
  return a;
}

// Any scale.
__global__ void __launch_bounds__(128)
gtaoKernel(const HfbUniforms U, const float* __restrict__ depth, const float2* __restrict__ normals, uint32_t aoW,
           uint32_t aoH, float scale, float* __restrict__ out) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= aoW * aoH) return;
  const AoCtx a = aoCtx(U, depth);
  const float px = fadd((float)(i % aoW), 0.5f) / scale, py = fadd((float)(i / aoW), 0.5f) / scale;
  const f3 posVS = reproject(a, px, py);
  float ao = 0.0f;
  if (!(posVS.z >= AO_SKY)) {
    gtao<false>(U, a, px, py, normalAt(a, normals, px, py), posVS, nullptr, 0, 0u, U.ao.numDirections,
                [&](uint32_t, float t) { ao = fadd(ao, t); });
    ao = ao / (float)U.ao.numDirections;
  }
  *HFB_G(&out[i]) = r16(ao);
}

// Scale 0.5, the reference's: a block of 8 x 8 texels with its pixels' positions in
// shared memory, four threads per texel (a quarter of its directions each; the terms
// are summed in the directions' order), so that a frame with little hair still gives
// every SM some.  Bound by issue (81 % of the peak when every one of a texel's 192
// samples was reprojected, ~150 instructions each): 531 -> 309 us at 1920x1080 with every
// texel occluded, 142 -> 48 us where hair covers 6 % of the frame; one thread per texel
// and blocks of 32 x 8: 289 and 94 us.
__global__ void __launch_bounds__(AO_THREADS)
gtaoTileKernel(const HfbUniforms U, const float* __restrict__ depth, const float2* __restrict__ normals, uint32_t aoW,
               uint32_t aoH, float* __restrict__ out) {
  __shared__ AoTile tile;
  const AoCtx a = aoCtx(U, depth);
  const uint32_t texel = threadIdx.x / AO_SPLIT, part = threadIdx.x % AO_SPLIT;
  const uint32_t tx = texel % AO_BX, ty = texel / AO_BX;
  const uint32_t x = blockIdx.x * AO_BX + tx, y = blockIdx.y * AO_BY + ty;
  const bool inside = x < aoW && y < aoH;
  const float px = (float)(2u * x + 1u), py = (float)(2u * y + 1u);
  // blocks of sky alone, most of a frame, need no tile
  const bool sky = !inside || linearizeDepth(loadDepth(a, px, py)) >= AO_SKY;
  if (__syncthreads_and(sky)) {
    if (inside && part == 0u) *HFB_G(&out[(size_t)y * aoW + x]) = 0.0f;
    return;
  }
  // the tile's first pixel: that of the block's first texel, 2 x + 1, less the halo
  const int X0 = 2 * AO_BX * (int)blockIdx.x + 1 - AO_HALO, Y0 = 2 * AO_BY * (int)blockIdx.y + 1 - AO_HALO;
  for (int i = threadIdx.x; i < AO_TW * AO_TH; i += (int)AO_THREADS) {
    const int r = i / AO_TW;
    const f3 p = reproject(a, (float)(X0 + i - r * AO_TW), (float)(Y0 + r));
    tile.x[i] = p.x;
    tile.y[i] = p.y;
    tile.z[i] = p.z;
  }
  __syncthreads();
  const uint32_t n = U.ao.numDirections, per = divCeil(n, AO_SPLIT);  // at most AO_TERMS (launchGtao)
  if (!sky) {
    const int at = (2 * (int)ty + AO_HALO) * AO_TW + 2 * (int)tx + AO_HALO;
    const uint32_t i0 = min(part * per, n), i1 = min(i0 + per, n);
    gtao<true>(U, a, px, py, normalAt(a, normals, px, py), mk3(tile.x[at], tile.y[at], tile.z[at]), &tile, at, i0, i1,
               [&](uint32_t i, float t) { tile.term[i - i0][threadIdx.x] = t; });
  }
  __syncwarp();  // a texel's threads are of one warp
  if (inside && part == 0u) {
    float ao = 0.0f;
    if (!sky) {
      for (uint32_t p = 0, i = 0; p < AO_SPLIT; p++)
        for (uint32_t k = 0; k < per && i < n; k++, i++) ao = fadd(ao, tile.term[k][threadIdx.x + p]);
      ao = ao / (float)n;
    }
    *HFB_G(&out[(size_t)y * aoW + x]) = r16(ao);
  }
}

}  // namespace

uint32_t aoExtent(float viewport, float scale) { return (uint32_t)ceilf(viewport * scale); }

cudaError_t launchGtao(HfbCtx* c, const HfbUniforms& u, const float* depth, const float* normals, float scale,
                       float* ao, bool general) {
  HFB_CHECK_BIND(c);
  const uint32_t aoW = aoExtent(u.viewport.x, scale), aoH = aoExtent(u.viewport.y, scale);
  const uint32_t n = aoW * aoH;
  if (n == 0) return cudaSuccess;
  const uint32_t by = divCeil(aoH, AO_BY);
  if (!general && scale == 0.5f && by <= 65535u && u.ao.numDirections <= AO_SPLIT * AO_TERMS) {
    gtaoTileKernel<<<dim3(divCeil(aoW, AO_BX), by), AO_THREADS, 0, c->stream>>>(u, depth, (const float2*)normals, aoW,
                                                                                aoH, ao);
    HFB_AFTER_LAUNCH(c, "gtaoTileKernel");
  } else {
    gtaoKernel<<<divCeil(n, 128u), 128, 0, c->stream>>>(u, depth, (const float2*)normals, aoW, aoH, scale, ao);
    HFB_AFTER_LAUNCH(c, "gtaoKernel");
  }
  c->launches += 1;
  return cudaGetLastError();
}

}  // namespace hfb
