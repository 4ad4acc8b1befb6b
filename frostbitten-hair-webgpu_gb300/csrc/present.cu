// Composite + present: HairCombinePass and PresentPass as one CUDA pass.
//
// HairCombinePass (hairCombinePass.wgsl.ts:51-89, pipeline blend state
// hairCombinePass.ts:40-52) draws the fine pass's result over the scene
// colour with src-alpha / one-minus-src-alpha, reading the result buffer
// upside down (fragment row y reads result row H - 1 - y).  PresentPass
// (presentPass.wgsl.ts: main_fs, DISPLAY_MODE_FINAL) then dithers (8x8 Bayer,
// dither.wgsl.ts:26-53), applies the exposure, ACES (aces.wgsl.ts:6-13) with
// saturate, and gamma (pow(c, 1 / gamma)); the swap chain stores unorm8,
// c * 255 rounded to nearest.  Out: RGBA8, row 0 at the top, alpha 255.
#define HFB_TU 8
#include "hfb_internal.cuh"
#include "hfb_math.cuh"

namespace hfb {
namespace {

// dither.wgsl.ts:26-53, each entry over 63
#define B8(a, b, c, d, e, f, g, h) a / 63.0f, b / 63.0f, c / 63.0f, d / 63.0f, e / 63.0f, f / 63.0f, g / 63.0f, h / 63.0f
__constant__ float kBayer[64] = {B8(0, 32, 8, 40, 2, 34, 10, 42),  B8(48, 16, 56, 24, 50, 18, 58, 26),
                                 B8(12, 44, 4, 36, 14, 46, 6, 38),  B8(60, 28, 52, 20, 62, 30, 54, 22),
                                 B8(3, 35, 11, 43, 1, 33, 9, 41),   B8(51, 19, 59, 27, 49, 17, 57, 25),
                                 B8(15, 47, 7, 39, 13, 45, 5, 37),  B8(63, 31, 55, 23, 61, 29, 53, 21)};
#undef B8

__device__ __forceinline__ float aces(float x) {  // doACES_Tonemapping, one channel
  const float num = fmul(x, fadd(fmul(2.51f, x), 0.03f));
  const float den = fadd(fmul(x, fadd(fmul(2.43f, x), 0.59f)), 0.14f);
  return sat(num / den);
}

__device__ __forceinline__ uint32_t unorm8(float c) {  // float -> unorm8, round to nearest
  return __float2uint_rn(fmul(sat(c), 255.0f));
}

// Tone mapping, gamma and unorm8 of one channel (x: exposed), as the passes define them.
static __device__ __noinline__ uint32_t toneExact(float x, float power) { return unorm8(powf(aces(x), power)); }

// The same byte from approximate units.  The quotient, logarithm and exponential are good to
// 2^-22 (the logarithm absolutely within (0.5, 2)), so for powers up to 1 the value times 255 is
// off by less than 255 * 2^-22 * (0.7 p + 0.7 * 1.25 * 0.53 + 1 + 0.5 p) < 1.7e-4 (r |log2 r| <=
// 0.53 for r in [0, 1]), and powf and its products by less than 1e-4: farther than 5e-4 from a
// rounding boundary the byte is decided.  One channel in 1,000 is not, and takes the exact way.
constexpr float TONE_MARGIN = 5e-4f;
// False: not decided.  Compared with toneExact over every float by hfb_check_tone.
__device__ __forceinline__ bool toneShort(float x, float power, uint32_t& byte) {
  const float num = fmul(x, fadd(fmul(2.51f, x), 0.03f));
  const float den = fadd(fmul(x, fadd(fmul(2.43f, x), 0.59f)), 0.14f);
  float rcp, lg, r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rcp) : "f"(den));
  const float v = sat(fmul(num, rcp));
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(lg) : "f"(v));
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(fmul(lg, power)));
  const float t = fmul(r, 255.0f);
  const float m = fadd(t, 12582912.0f);  // t rounded to the nearest whole number, in m's low bits
  // den within the approximate reciprocal's accuracy, v not tiny (a zero is exact either way)
  byte = __float_as_uint(m) & 255u;
  return fabsf(den) >= 1e-30f && fabsf(den) <= 1e30f && (v >= 1e-30f || num == 0.0f) &&
         fabsf(fsub(t, fsub(m, 12582912.0f))) < 0.5f - TONE_MARGIN;
}
__device__ __forceinline__ bool toneFast(float power) { return power > 0.0f && power <= 1.0f; }
// fast: toneFast(power)
__device__ __forceinline__ uint32_t tone(float x, float power, bool fast) {
  uint32_t byte;
  return fast && toneShort(x, power, byte) ? byte : toneExact(x, power);
}

// Compares the short form's bytes with toneExact's over every float: cnt[0] the ones that
// differ, cnt[1] the values in [0, 16] that it decided.
__global__ void __launch_bounds__(256) toneCheckKernel(float power, unsigned long long* __restrict__ cnt) {
  unsigned long long bad = 0, decided = 0;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  if (toneFast(power))
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < (1ull << 32); i += stride) {
      const float x = __uint_as_float((uint32_t)i);
      uint32_t byte;
      if (!toneShort(x, power, byte)) continue;
      bad += byte != toneExact(x, power);
      decided += x >= 0.0f && x <= 16.0f;
    }
  if (bad) atomicAdd(&cnt[0], bad);
  if (decided) atomicAdd(&cnt[1], decided);
}

// One image of a launch; it takes the launch's blocks [first, first + blocks).
struct PresentImage {
  float power, exposure, dither;  // power: 1 / gamma
  uint32_t W, H, first;
  const float4* result;
  const float4* scene;
  uchar4* out;
};

// Pixels [blk * PRESENT_PIXELS, (blk + 1) * PRESENT_PIXELS) of an image, row-major, row 0 at
// the top.  20 B per pixel read (36 with a scene) and 4 written: with ~550 instructions per
// pixel (powf, divisions, a search for the pixel's image) the pass ran at 1.8 TB/s on 64
// images; with ~120 it is near the memory's rate.
constexpr uint32_t PRESENT_THREADS = 256, PRESENT_PIXELS = 1024;
__device__ __forceinline__ void presentBlock(const PresentImage m, uint32_t blk, float* bayer) {
  if (threadIdx.x < 64u) bayer[threadIdx.x] = kBayer[threadIdx.x];  // lanes read different entries
  __syncthreads();
  const uint32_t n = m.W * m.H, W = m.W;
  const float power = m.power, exposure = m.exposure, ditherStr = m.dither;
  const bool fast = toneFast(power);
  uint32_t i = blk * PRESENT_PIXELS + threadIdx.x;
  uint32_t y = i / W, x = i - y * W;  // y: row from the top
  const uint32_t dy = PRESENT_THREADS / W, dx = PRESENT_THREADS - dy * W;
#pragma unroll
  for (uint32_t k = 0; k < PRESENT_PIXELS / PRESENT_THREADS; k++) {
    if (i < n) {
      const float4 src = __ldg(HFB_G(&m.result[(size_t)(m.H - 1u - y) * W + x]));
      const float4 dst = m.scene ? __ldg(HFB_G(&m.scene[i])) : make_float4(0.f, 0.f, 0.f, 1.f);
      // blend: src * src.a + dst * (1 - src.a)
      const float ia = fsub(1.0f, src.w);
      const float dither = fmul(fmul(bayer[(y & 7u) * 8u + (x & 7u)], ditherStr), 1.0f / 256.0f);
      const float r = fmul(fadd(fadd(fmul(src.x, src.w), fmul(dst.x, ia)), dither), exposure);
      const float g = fmul(fadd(fadd(fmul(src.y, src.w), fmul(dst.y, ia)), dither), exposure);
      const float b = fmul(fadd(fadd(fmul(src.z, src.w), fmul(dst.z, ia)), dither), exposure);
      *HFB_G(&m.out[i]) = make_uchar4((unsigned char)tone(r, power, fast), (unsigned char)tone(g, power, fast),
                                      (unsigned char)tone(b, power, fast), 255);
    }
    i += PRESENT_THREADS;
    x += dx;
    y += dy;
    if (x >= W) { x -= W; y++; }
  }
}

__global__ void __launch_bounds__(PRESENT_THREADS) presentKernel(const PresentImage m) {
  __shared__ float bayer[64];
  presentBlock(m, blockIdx.x, bayer);
}

// Up to PRESENT_BATCH images in one launch, passed by value (48 B each, inside
// the 4 KB of kernel parameters every launch may carry).
constexpr uint32_t PRESENT_BATCH = 64;
struct PresentBatch {
  uint32_t n, blocks;
  PresentImage im[PRESENT_BATCH];
};
static_assert(sizeof(PresentBatch) <= 4000, "kernel parameters above 4 KB");

__global__ void __launch_bounds__(PRESENT_THREADS) presentBatchKernel(const PresentBatch pb) {
  __shared__ float bayer[64];
  uint32_t lo = 0, hi = pb.n - 1u;  // the last image whose first block is at or before this one
  while (lo < hi) {
    const uint32_t mid = (lo + hi + 1u) >> 1;
    if (pb.im[mid].first <= blockIdx.x) lo = mid; else hi = mid - 1u;
  }
  const PresentImage m = pb.im[lo];
  presentBlock(m, blockIdx.x - m.first, bayer);
}

}  // namespace

cudaError_t launchToneCheck(HfbCtx* c, float power, unsigned long long* cnt) {
  HFB_CHECK_BIND(c);
  cudaError_t e = cudaMemsetAsync(cnt, 0, 2 * sizeof(unsigned long long), c->stream);
  if (e != cudaSuccess) return e;
  toneCheckKernel<<<c->smCount * 8u, 256, 0, c->stream>>>(power, cnt);
  HFB_AFTER_LAUNCH(c, "toneCheckKernel");
  c->launches += 1;
  return cudaGetLastError();
}

cudaError_t launchPresent(HfbCtx* c, const HfbUniforms& u, uint32_t W, uint32_t H, const float* result,
                          const float* scene, uint8_t* rgba) {
  HFB_CHECK_BIND(c);
  const uint32_t n = W * H;
  if (n == 0) return cudaSuccess;
  const PresentImage m = {1.0f / u.colorMgmt.x, u.colorMgmt.y, u.colorMgmt.z, W, H, 0u, (const float4*)result,
                          (const float4*)scene, (uchar4*)rgba};
  presentKernel<<<divCeil(n, PRESENT_PIXELS), PRESENT_THREADS, 0, c->stream>>>(m);
  HFB_AFTER_LAUNCH(c, "presentKernel");
  c->launches += 1;
  return cudaGetLastError();
}

// Images of at most 2^32 - 1 pixels in all per launch of PRESENT_BATCH; the
// caller has checked every item.
cudaError_t launchPresentBatch(HfbCtx* c, const HfbPresentItem* items, uint32_t n) {
  HFB_CHECK_BIND(c);
  for (uint32_t k0 = 0; k0 < n; k0 += PRESENT_BATCH) {
    PresentBatch pb{};
    uint64_t total = 0;
    for (uint32_t k = k0; k < n && k < k0 + PRESENT_BATCH; k++) {
      const HfbPresentItem& it = items[k];
      const uint32_t W = it.rb->width, H = it.rb->height;
      if ((uint64_t)W * H == 0u) continue;
      if (total + (uint64_t)W * H > 0xffffffffull) return cudaErrorInvalidValue;
      pb.im[pb.n++] = {1.0f / it.uniforms->colorMgmt.x, it.uniforms->colorMgmt.y, it.uniforms->colorMgmt.z, W, H,
                       pb.blocks, (const float4*)(it.rb->rasterizerResult + 4), (const float4*)it.sceneColor,
                       (uchar4*)it.rgba};
      pb.blocks += divCeil(W * H, PRESENT_PIXELS);
      total += (uint64_t)W * H;
    }
    if (pb.n == 0) continue;
    presentBatchKernel<<<pb.blocks, PRESENT_THREADS, 0, c->stream>>>(pb);
    HFB_AFTER_LAUNCH(c, "presentBatchKernel");
    c->launches += 1;
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace hfb
