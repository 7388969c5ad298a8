// Post-processing of a film on the GPU: the operations of the reference's
// PostProcessing.cpp (applyExposure :3-6, basicBlur bloom :132-211,
// reinhardTonemap :35-39, acesTonemap :41-52, clampPixels :30-33, applysRGB
// :54-57, flipX :19-28 / flipY :8-17) and its LDR output step (main.cpp:150-158:
// clamp, fastPow(v, 1/2.2) * 255) in one pass over the image, in that order.
// The arithmetic follows the reference's types: double where its
// expressions hold a double literal (ACES, sRGB, the bloom threshold sum),
// float elsewhere.
//
// Defined where the reference reads uninitialised memory: basicBlur leaves
// the alpha of below-threshold pixels and the blur of the border pixels
// (within radius/2 of an edge) unset; here they are 0.
#include <cmath>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "internal.h"

namespace er {
namespace {

struct PostParams {
  int32_t w, h;
  float exposure;
  int32_t tonemap, clamp01, srgb, flip_x, flip_y;
  float threshold, power;
  int32_t blur;  // basicBlur's blurSize; 0 = no bloom
};

__device__ __forceinline__ float clampr(float a, float b, float c) { return a < b ? b : a > c ? c : a; }

// ------------------------------------------------------------ channels --
//
// The reference evaluates ACES, the sRGB power and the 8-bit encoding in
// double.  FP64 runs at a sixty-fourth of the FP32 rate here, and a 1080p
// frame without bloom took 2.08 ms with those expressions (0.07 now; its
// 75 MB take 0.011), so each is computed another way to the same bits:
//  - ACES and the power in pairs of floats (T. J. Dekker, "A floating-point
//    technique for extending the available precision", Numer. Math. 18,
//    1971); if the pair lies within 2^-41 of a point where the rounding to
//    float changes (A. Ziv, "Fast evaluation of elementary mathematical
//    functions with correctly rounded last bit", ACM TOMS 17, 1991), and for
//    arguments out of range, the double expression is evaluated after all
//    (about one value in 2^16).  Over every float that the pairs take, [2^-30,
//    2^30] and [2^-60, 2^16], the largest error of the pair is 2^-44.2 (ACES)
//    and 2^-42.0 (the power, below 2^-16 where its argument is scaled; 2^-43.0
//    elsewhere), and no result differs from the double expression's;
//  - the encoding in integers.

__device__ __noinline__ float aces_exact(float x) {
  const float a = 2.51f, b = 0.03f, c = 2.43f, d = 0.59f, e = 0.14f;
  const double xd = (double)x;
  const double num = xd * 0.6 * ((double)__fmul_rn(a, x) * 0.6 + (double)b);
  const double den = xd * 0.6 * ((double)__fmul_rn(c, x) * 0.6 + (double)d) + (double)e;
  return (float)(num / den);
}
__device__ __forceinline__ float aces(float x) {
  float r;
  if (x >= 0x1p-30f && x <= 0x1p30f) {
    constexpr ff k6 = {(float)0.6, (float)(0.6 - (double)(float)0.6)};
    const ff p = mul(k6, x);
    const ff num = mul(p, add(mul(k6, __fmul_rn(2.51f, x)), 0.03f));
    const ff den = add(mul(p, add(mul(k6, __fmul_rn(2.43f, x)), 0.59f)), 0.14f);
    const float inv = __fdividef(1.0f, den.h), q = num.h * inv;  // (l corrects q)
    const ff back = mul(den, q);
    const float l = __fadd_rn(__fsub_rn(num.h, back.h), __fsub_rn(num.l, back.l)) * inv;
    if (settled(q, l, &r)) return r;
  } else if (x == 0.0f) {
    return x;
  }
  return aces_exact(x);
}

__device__ __noinline__ float root22_exact(float x) { return (float)pow((double)x, 1.0 / 2.2); }
// x^(1/2.2): y^11 = x^5 by one third-order step from an approximate y.  The
// double 1/2.2 differs from 5/11 by 2^-54.7 of it, far below the margin.
// Small x is scaled by 2^44, y then by 2^-20.
__device__ __forceinline__ float root22(float x) {
  if (x >= 0x1p-60f && x <= 0x1p16f) {
    const bool tiny = x < 0x1p-20f;
    const float s = tiny ? x * 0x1p44f : x;
    const float y = __powf(s, 5.0f / 11.0f);
    const ff x2 = two_prod(s, s), x5 = mul(mul(x2, x2), s);
    const ff y2 = two_prod(y, y), y4 = mul(y2, y2), y11 = mul(mul(mul(y4, y4), y2), y);
    const float r = __fdividef(__fadd_rn(__fsub_rn(x5.h, y11.h), __fsub_rn(x5.l, y11.l)), y11.h);
    const float l = y * (r * (1.0f / 11.0f) - (5.0f / 121.0f) * (r * r));
    float v;
    if (settled(y, l, &v)) return tiny ? v * 0x1p-20f : v;
  } else if (x == 0.0f) {
    return 0.0f;
  }
  return root22_exact(x);
}

__device__ __forceinline__ float post_channel(float x, const PostParams& P) {
  if (P.tonemap == ER_TONEMAP_REINHARD) x = __fdiv_rn(x, __fadd_rn(1.0f, x));
  else if (P.tonemap == ER_TONEMAP_ACES) x = clampr(aces(x), 0.0f, 1.0f);
  if (P.clamp01) x = clampr(x, 0.0f, 1.0f);
  if (P.srgb) x = root22(x);
  return x;
}

// trunc(fastPow(v, 1/2.2) * 255), fastPow(a, b) being Ankerl's: the double
// whose high word is trunc(b (hi(a) - K) + K), K = 1072632447.  hi - K is an
// integer, and with b = 1/2.2 the double arithmetic gives exactly
// floor(5 (hi - K) / 11) + K: a non-integral value lies at least 1/11 from an
// integer and the roundings are below 2^-23, an integral one comes out
// exactly because b is within 2^-54.7 of 5/11.  The result's 20-bit mantissa
// times 255 is exact too.  Below 2^-19 the byte is 0.
__device__ __forceinline__ uint8_t ldr_channel(float v) {
  if (!(v >= 0x1p-19f)) return 0;  // (also NaN)
  const int32_t K = 1072632447;
  const uint32_t f = __float_as_uint(fminf(v, 1.0f));
  const int32_t hi = (int32_t)((f >> 3) + ((1023u - 127u) << 20));
  const int32_t o = K - (1 << 24) + (int32_t)((uint32_t)(5 * (hi - K) + 11 * (1 << 24)) / 11u);
  return (uint8_t)((((uint32_t)o & 0xFFFFFu) + 0x100000u) * 255u >> (20 + 1023 - (o >> 20)));
}

__device__ __forceinline__ float4 exposed(float4 v, float e) {
  return make_float4(v.x * e, v.y * e, v.z * e, v.w * e);
}

// basicBlur's threshold: the pixel, or zeros where its mean is below it.
// The reference sums the thirds in double, rounding to float after each;
// only where the plain float sum is within its error of the threshold does
// that decide (and for NaN and infinities).
__device__ __forceinline__ float4 bright(float4 v, float threshold) {
  const float s = (v.x + v.y + v.z) * (1.0f / 3.0f);
  const float m = (fabsf(v.x) + fabsf(v.y) + fabsf(v.z)) * 1e-6f;
  bool below = s < threshold;
  if (!(fabsf(s - threshold) > m)) {
    float t = 0.f;
    t = (float)((double)t + (double)v.x / 3.0);
    t = (float)((double)t + (double)v.y / 3.0);
    t = (float)((double)t + (double)v.z / 3.0);
    below = t < threshold;
  }
  return below ? make_float4(0.f, 0.f, 0.f, 0.f) : v;
}

// Tone map, clamp, sRGB and the float and 8-bit outputs of source pixel
// (x, y), flipped.
__device__ __forceinline__ void finish_pixel(float4 v, int32_t x, int32_t y, float4* out, uchar4* ldr,
                                             const PostParams& P) {
  // one copy of the channel code (the channels rotate through it): four
  // copies, and in the bloom kernel sixteen, are fetched slower than run
#pragma unroll 1
  for (int k = 0; k < 4; k++) v = make_float4(v.y, v.z, v.w, post_channel(v.x, P));
  const int32_t i = (P.flip_x ? P.w - 1 - x : x) + (P.flip_y ? P.h - 1 - y : y) * P.w;
  if (out) out[i] = v;
  if (ldr) ldr[i] = make_uchar4(ldr_channel(v.x), ldr_channel(v.y), ldr_channel(v.z), ldr_channel(v.w));
}

// Without bloom: one read and one write per pixel.  (`in` may be `out` when
// nothing is flipped: every thread reads and writes its own pixel.)
__global__ void k_post(const float4* in, float4* out, uchar4* ldr, PostParams P) {
  const int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= P.w * P.h) return;
  finish_pixel(exposed(in[i], P.exposure), i % P.w, i / P.w, out, ldr, P);
}

// With bloom, blur half-widths up to kTileBlur: a block of 32x8 threads does
// 32x32 pixels.  It reads them with their margin once, holds the thresholded
// pixels in shared memory and every thread sums four pixels of a column, so
// that a value read serves four sums; the sums run over columns, then rows,
// as the reference's do.  FP32 issue bounds it (77 % of the slots).  1080p,
// ACES, sRGB, 8-bit output, per call: half-width 4 136 us, 24 1.95 ms; 2.51
// and 5.59 ms as three passes that read every tap from global memory, with
// the double expressions and an allocation per buffer and call.  320x240 with
// half-width 4: 33 and 310 us.  The weights come as a kernel parameter.  Two
// blocks share an SM up to half-width 23 (78 x 78 pixels and the weights, 115
// KB), one has it from 24 on (122 KB): 1.37 and 1.95 ms, against 3.25 and
// 3.48 with the passes for wider blurs.
constexpr int kTileBlur = 24;
struct BlurWeights {
  float w[(2 * kTileBlur + 1) * (2 * kTileBlur + 1)];
  float one;  // 1 (tap)
};
constexpr int kTile = 32, kRows = 4;
// Tallest image: a grid has 65,535 rows of blocks.  (Taller ones take the
// passes for wide blurs; with the tiles' rows over two dimensions of the grid,
// or all tiles in one, 1080p takes 1 % and 3 % longer.)
constexpr int32_t kTileHeight = 65535 * kTile;
static_assert(kRows == 4, "the four sums of a thread are selected by hand");

__device__ __forceinline__ uint64_t pair(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
// s += t * k, product and sum each rounded, two channels at a time.  The sum
// is a multiply-add by a one the compiler does not know: a packed multiply
// followed by a packed add came out as one multiply-add, rounded once.
__device__ __forceinline__ void tap(uint64_t& s, uint64_t t, uint64_t k, uint64_t one) {
  uint64_t p;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(p) : "l"(t), "l"(k));
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(s) : "l"(p), "l"(one));
}

__global__ void __launch_bounds__(256)
    k_post_bloom(const float4* in, float4* out, uchar4* ldr, PostParams P, const __grid_constant__ BlurWeights W) {
  extern __shared__ float4 tile[];
  const int32_t b = P.blur, ks = 2 * b + 1, tw = kTile + 2 * b;
  uint64_t* wt = (uint64_t*)(tile + tw * tw);  // by column, then row; each weight twice
  const int32_t tid = threadIdx.y * 32 + threadIdx.x;
  const int32_t x0 = blockIdx.x * kTile, y0 = blockIdx.y * kTile;
  for (int32_t k = tid; k < ks * ks; k += 256) {
    const float v = W.w[k / ks + (k % ks) * ks];
    wt[k] = pair(v, v);
  }
  bool any = false;
  for (int32_t k = tid; k < tw * tw; k += 256) {
    const int32_t x = x0 - b + k % tw, y = y0 - b + k / tw;
    float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
    if (x >= 0 && x < P.w && y >= 0 && y < P.h) t = bright(exposed(in[x + y * P.w], P.exposure), P.threshold);
    tile[k] = t;
    // (a pixel of zeros adds +0 to sums that start from +0)
    any |= (__float_as_uint(t.x) | __float_as_uint(t.y) | __float_as_uint(t.z) | __float_as_uint(t.w)) != 0u;
  }
  const uint64_t one = pair(W.one, W.one);
  uint64_t s[kRows][2];
#pragma unroll
  for (int q = 0; q < kRows; q++) s[q][0] = s[q][1] = 0;
  const float4* col = tile + threadIdx.y * kRows * tw + threadIdx.x;
  if (__syncthreads_or(any)) {
    for (int32_t ii = 0; ii < ks; ii++) {
      const uint64_t* wc = wt + ii * ks;
      auto row = [&](int32_t r, bool inside) {
        const float4 t = col[r * tw + ii];
        const uint64_t t0 = pair(t.x, t.y), t1 = pair(t.z, t.w);
#pragma unroll
        for (int q = 0; q < kRows; q++) {
          const int32_t jj = r - q;
          if (inside || (jj >= 0 && jj < ks)) {
            const uint64_t kk = wc[jj];
            tap(s[q][0], t0, kk, one);
            tap(s[q][1], t1, kk, one);
          }
        }
      };
      int32_t r = 0;
      for (; r < kRows - 1; r++) row(r, false);
#pragma unroll 4
      for (; r < ks; r++) row(r, true);
      for (; r < ks + kRows - 1; r++) row(r, false);
    }
  }
  const int32_t x = x0 + threadIdx.x;
  if (x >= P.w) return;
#pragma unroll 1
  for (int q = 0; q < kRows; q++) {
    const int32_t y = y0 + threadIdx.y * kRows + q;
    if (y >= P.h) return;
    const uint64_t s0 = q == 0 ? s[0][0] : q == 1 ? s[1][0] : q == 2 ? s[2][0] : s[3][0];
    const uint64_t s1 = q == 0 ? s[0][1] : q == 1 ? s[1][1] : q == 2 ? s[2][1] : s[3][1];
    float4 v = exposed(in[x + y * P.w], P.exposure);
    if (x >= b && x < P.w - b && y >= b && y < P.h - b) {
      float4 t;
      asm("mov.b64 {%0, %1}, %2;" : "=f"(t.x), "=f"(t.y) : "l"(s0));
      asm("mov.b64 {%0, %1}, %2;" : "=f"(t.z), "=f"(t.w) : "l"(s1));
      v.x = __fadd_rn(v.x, __fmul_rn(t.x, P.power));
      v.y = __fadd_rn(v.y, __fmul_rn(t.y, P.power));
      v.z = __fadd_rn(v.z, __fmul_rn(t.z, P.power));
      v.w = __fadd_rn(v.w, __fmul_rn(t.w, P.power));
    }
    finish_pixel(v, x, y, out, ldr, P);
  }
}

// With bloom of wider blurs, whose margin does not fit in shared memory, and
// of images taller than kTileHeight: the
// thresholded image in global memory, then every tap from it.
__global__ void k_post_bright(const float4* in, float4* thr, PostParams P) {
  const int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < P.w * P.h) thr[i] = bright(exposed(in[i], P.exposure), P.threshold);
}
__global__ void k_post_bloom_wide(const float4* in, const float4* thr, const float* kern, float4* out, uchar4* ldr,
                                  PostParams P) {
  const int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= P.w * P.h) return;
  const int32_t x = i % P.w, y = i / P.w, b = P.blur, ks = 2 * b + 1;
  float4 v = exposed(in[i], P.exposure);
  if (x >= b && x < P.w - b && y >= b && y < P.h - b) {
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int32_t ii = 0; ii < ks; ii++) {
      for (int32_t jj = 0; jj < ks; jj++) {
        const float4 t = thr[(x - b + ii) + (y - b + jj) * P.w];
        const float k = __ldg(kern + ii + jj * ks);
        s.x = __fadd_rn(s.x, __fmul_rn(t.x, k));
        s.y = __fadd_rn(s.y, __fmul_rn(t.y, k));
        s.z = __fadd_rn(s.z, __fmul_rn(t.z, k));
        s.w = __fadd_rn(s.w, __fmul_rn(t.w, k));
      }
    }
    v.x = __fadd_rn(v.x, __fmul_rn(s.x, P.power));
    v.y = __fadd_rn(v.y, __fmul_rn(s.y, P.power));
    v.z = __fadd_rn(v.z, __fmul_rn(s.z, P.power));
    v.w = __fadd_rn(v.w, __fmul_rn(s.w, P.power));
  }
  finish_pixel(v, x, y, out, ldr, P);
}

}  // namespace
}  // namespace er

using namespace er;

extern "C" er_status er_postprocess(const float* rgba_in, int32_t width, int32_t height, const er_post_opts* opts,
                                    float* rgba_out, uint8_t* ldr_out, uint32_t flags) {
  return guarded("er_postprocess", [&]() -> er_status {
    if (!rgba_in || width <= 0 || height <= 0 || (!rgba_out && !ldr_out))
      return fail(ER_ERR_INVALID_ARG, "bad post-processing arguments");
    if ((int64_t)width * height > ((int64_t)1 << 28)) return fail(ER_ERR_INVALID_ARG, "image too large");
    er_post_opts o{};
    o.exposure = 1.0f;
    if (opts) o = *opts;
    if (o.tonemap < ER_TONEMAP_NONE || o.tonemap > ER_TONEMAP_ACES) return fail(ER_ERR_INVALID_ARG, "tonemap");
    if (o.bloom_power != 0.0f && !(o.bloom_radius >= 0.0f && o.bloom_radius <= 256.0f))
      return fail(ER_ERR_INVALID_ARG, "bloom radius out of range");
    int dev = 0;
    ER_CUDA(cudaGetDevice(&dev));
    const bool devp = flags & ER_RENDER_DEVICE_OUT;
    const size_t n = (size_t)width * height;
    PostParams P;
    P.w = width;
    P.h = height;
    P.exposure = o.exposure;
    P.tonemap = o.tonemap;
    P.clamp01 = o.clamp != 0;
    P.srgb = o.srgb != 0;
    P.flip_x = o.flip_x != 0;
    P.flip_y = o.flip_y != 0;
    P.threshold = o.bloom_threshold;
    P.power = o.bloom_power;
    P.blur = o.bloom_power != 0.0f ? (int32_t)(o.bloom_radius / 2) : 0;
    // basicBlur's kernel (PostProcessing.cpp:143-153), built on the host
    const int32_t ks = 2 * P.blur + 1;
    std::vector<float> kern(P.blur > 0 ? (size_t)ks * ks : 1, 0.0f);
    if (P.blur > 0) {
      const float sd = o.bloom_radius;
      const float kernelSize = (float)ks;
      for (int32_t x = 0; x < ks; x++)
        for (int32_t y = 0; y < ks; y++) {
          float t1 = (float)(1.0 / ((2.0 * (double)3.14159265358979323846f) * (double)(sd * sd)));
          float tx = (float)(x - (int32_t)(kernelSize / 2.0));
          float ty = (float)(y - (int32_t)(kernelSize / 2.0));
          float t2 = (float)(-(double)(tx * tx + ty * ty) / (2.0 * (double)sd * (double)sd));
          kern[(size_t)(x + y * ks)] = t1 * std::exp(t2);
        }
    }
    struct Buf {
      std::vector<void*> p;
      ~Buf() {
        for (void* q : p) cudaFree(q);
      }
      er_status get(void** out, size_t bytes) {
        cudaError_t e = cudaMalloc(out, std::max<size_t>(bytes, 16));
        if (e != cudaSuccess) {
          cudaGetLastError();
          return fail(ER_ERR_OOM, "post-processing buffers");
        }
        p.push_back(*out);
        return ER_OK;
      }
    } B;
    er_status st;
    const float4* d_in = (const float4*)rgba_in;
    float4* d_out = nullptr;
    uchar4* d_ldr = nullptr;
    if (!devp) {
      void* p;
      if ((st = B.get(&p, n * 16)) != ER_OK) return st;
      ER_CUDA(cudaMemcpy(p, rgba_in, n * 16, cudaMemcpyHostToDevice));
      d_in = (const float4*)p;
    }
    if (rgba_out) {
      if (devp) d_out = (float4*)rgba_out;
      else if ((st = B.get((void**)&d_out, n * 16)) != ER_OK) return st;
    }
    if (ldr_out) {
      if (devp) d_ldr = (uchar4*)ldr_out;
      else if ((st = B.get((void**)&d_ldr, n * 4)) != ER_OK) return st;
    }
    // Outputs over the input: the same pixels in place need nothing; where a
    // pixel is read after another's output may have replaced it, the passes
    // read a copy of the input.
    const uintptr_t i0 = (uintptr_t)d_in, o0 = (uintptr_t)d_out, l0 = (uintptr_t)d_ldr;
    const bool over_out = d_out && o0 < i0 + n * 16 && i0 < o0 + n * 16;
    const bool over_ldr = d_ldr && l0 < i0 + n * 16 && i0 < l0 + n * 4;
    const bool in_place = o0 == i0 && P.blur == 0 && !P.flip_x && !P.flip_y;
    if (over_ldr || (over_out && !in_place)) {
      void* p;
      if ((st = B.get(&p, n * 16)) != ER_OK) return st;
      ER_CUDA(cudaMemcpyAsync(p, d_in, n * 16, cudaMemcpyDeviceToDevice, 0));
      d_in = (const float4*)p;
    }
    const unsigned blocks = (unsigned)((n + 255) / 256);
    if (P.blur == 0) {
      k_post<<<blocks, 256>>>(d_in, d_out, d_ldr, P);
    } else if (P.blur <= kTileBlur && height <= kTileHeight) {
      BlurWeights W;
      W.one = 1.0f;
      std::memcpy(W.w, kern.data(), kern.size() * sizeof(float));
      const int32_t tw = kTile + 2 * P.blur;
      const size_t smem = (size_t)tw * tw * sizeof(float4) + kern.size() * 2 * sizeof(float);
      // (the same limit from every thread, whatever this call needs)
      constexpr int kMaxSmem = (kTile + 2 * kTileBlur) * (kTile + 2 * kTileBlur) * 16 + 2 * (int)sizeof(BlurWeights);
      ER_CUDA(cudaFuncSetAttribute(k_post_bloom, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem));
      const dim3 grid((unsigned)((width + kTile - 1) / kTile), (unsigned)((height + kTile - 1) / kTile));
      k_post_bloom<<<grid, dim3(32, kTile / kRows), smem>>>(d_in, d_out, d_ldr, P, W);
    } else {
      float4* thr;
      float* d_kern;
      if ((st = B.get((void**)&thr, n * 16)) != ER_OK) return st;
      if ((st = B.get((void**)&d_kern, kern.size() * 4)) != ER_OK) return st;
      ER_CUDA(cudaMemcpy(d_kern, kern.data(), kern.size() * 4, cudaMemcpyHostToDevice));
      k_post_bright<<<blocks, 256>>>(d_in, thr, P);
      k_post_bloom_wide<<<blocks, 256>>>(d_in, thr, d_kern, d_out, d_ldr, P);
    }
    ER_CUDA(cudaGetLastError());
    if (!devp) {
      if (rgba_out) ER_CUDA(cudaMemcpy(rgba_out, d_out, n * 16, cudaMemcpyDeviceToHost));
      if (ldr_out) ER_CUDA(cudaMemcpy(ldr_out, d_ldr, n * 4, cudaMemcpyDeviceToHost));
    }
    ER_CUDA(cudaDeviceSynchronize());
    (void)dev;
    return ER_OK;
  });
}
