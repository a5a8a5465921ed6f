// gi_filters.cu -- the passes after the march: the 5x5 depth/normal bilateral
// filter, the least-squares denoiser (Common/denoiser.frag:72-184), the final
// gather (Common/finalGatherer.frag:42-59), and the deinterleave / interleave
// permutations (Common/deinterleave.frag, Common/interleave.frag).
#include "gi_device.cuh"
#include "gi_internal.h"
#include "gi_kernels.h"

namespace gi {
namespace {

using namespace dev;

constexpr int kTx = 32, kTy = 8;

template <int DCH> __device__ __forceinline__ float depth_at(const float* p, int idx) {
  if (DCH == 2) return __ldg(reinterpret_cast<const float2*>(p) + idx).x;
  return __ldg(p + idx);
}

// Bilateral: taps y outer, x inner over [-2, 2]; w = exp(-|d-d0|*10.5) *
// exp(-|n-n0|^2*20) (weights of denoiser.frag:103,105), evaluated as one
// exponential of the summed exponents; out = sum / (sumW + 1e-7).  A block's halo of
// light, depth and normal is staged in shared memory (clamp-to-edge applied while
// staging), so every tap is a shared-memory read.  Each thread filters two vertically
// adjacent pixels: their windows share tap rows, so a thread reads 6 rows of taps for
// its two outputs instead of 10, and the two pixels' weights and sums are the halves of
// packed operations; each output still sums its taps in the order above, with the same
// roundings.  The fast weights (hardware exponential) are cheap and evaluated per tap;
// the exact ones once for both pixels that share them (bilateral_exact_kernel).
constexpr int kBilRows = 2;
constexpr int kHx = kTx + 4;

// Texels of a 36 x HY halo from (x0, y0) on; xyz of the normal with the depth in w.
// CENTRE: in the light's w (not filtered) the pixel's exact weight to itself, 1, or NaN
// where its normal or depth is not finite.
template <int DCH, int HY, int THREADS, bool CENTRE>
__device__ __forceinline__ void stage_halo(const float* __restrict__ ind, const float* __restrict__ depth,
                                           const float* __restrict__ normal, int w, int h, int x0, int y0,
                                           float4* s_col, float4* s_nrm) {
  // Every load out before the first is stored (fast weights at 1920 x 1080 47.6 -> 42.8 us).
  constexpr int kOwn = (kHx * HY + THREADS - 1) / THREADS;
  float4 c[kOwn], n[kOwn];
#pragma unroll
  for (int k = 0; k < kOwn; k++) {
    const int i = min((int)(threadIdx.y * kTx + threadIdx.x) + k * THREADS, kHx * HY - 1);
    const int q = iclamp(y0 + i / kHx, 0, h - 1) * w + iclamp(x0 + i % kHx, 0, w - 1);
    c[k] = ld4(ind, q);
    n[k] = ld4(normal, q);
    n[k].w = depth_at<DCH>(depth, q);
  }
#pragma unroll
  for (int k = 0; k < kOwn; k++) {
    if (CENTRE)
      c[k].w = 1.0f + ((n[k].x - n[k].x) + (n[k].y - n[k].y) + (n[k].z - n[k].z) + (n[k].w - n[k].w));
    const int i = min((int)(threadIdx.y * kTx + threadIdx.x) + k * THREADS, kHx * HY - 1);
    s_col[i] = c[k];
    s_nrm[i] = n[k];
  }
}

// expf_(-s) of both halves for s >= 0 or NaN, bit for bit.
__device__ __forceinline__ p2 exp_neg(p2 s) {
  // From 104 on expf_ gives 0, as 105 does here.
  float a, b;
  asm("min.NaN.f32 %0, %1, %2;" : "=f"(a) : "f"(lo_(s)), "f"(105.0f));
  asm("min.NaN.f32 %0, %1, %2;" : "=f"(b) : "f"(hi_(s)), "f"(105.0f));
  const p2 x = pk(a, b);
  // n = the nearest integer to -s log2 e (ties to even): the sum's spacing is 1 and its
  // low 8 bits are n + 192, in [40, 192].
  constexpr float kRound = 12582912.0f + 192.0f;
  const p2 t = padd(pmul(x, pk(-kLog2e)), pk(kRound));
  const p2 n = psub(t, pk(kRound));
  // q = -r of expf_, and its series with the signs of the odd terms turned.
  p2 q = pfma(n, pk(kLn2Hi), x);
  q = pfma(n, pk(kLn2Lo), q);
  p2 p = pfma(q, pk(-(1.0f / 40320.0f)), pk(1.0f / 5040.0f));
  p = pfma(q, p, pk(-(1.0f / 720.0f)));
  p = pfma(q, p, pk(1.0f / 120.0f));
  p = pfma(q, p, pk(-(1.0f / 24.0f)));
  p = pfma(q, p, pk(1.0f / 6.0f));
  p = pfma(q, p, pk(-0.5f));
  p = pfma(q, p, pk(1.0f));
  p = pfma(q, p, pk(-1.0f));
  // -p 2^n as (p 2^(n + 65)) 2^-65: one rounding, in the subnormal range, as in ldexp_.
  const p2 scale = pk(__uint_as_float(__float_as_uint(lo_(t)) << 23), __uint_as_float(__float_as_uint(hi_(t)) << 23));
  return pmul(pmul(p, scale), pk(-2.7105054312137611e-20f));
}

__device__ __forceinline__ void store_filtered(float4* at, float x, float y, float z, float w) {
  const float d = w + 1e-7f;
  *at = make_float4(div_(x, d), div_(y, d), div_(z, d), 1.0f);
}

// The fast weights of a tap of each pixel from the differences to their centres.
__device__ __forceinline__ p2 fast_weights(p2 x, p2 y, p2 z, p2 d) {
  const p2 m = pmul(pfma(z, z, pfma(y, y, pmul(x, x))), pk(20.0f));
  return pk(__expf(-fmaf(fabsf(lo_(d)), 10.5f, lo_(m))), __expf(-fmaf(fabsf(hi_(d)), 10.5f, hi_(m))));
}

// The march's fast precision: the weights by fused multiply-adds and the hardware
// exponential, the sums by fused multiply-adds.
template <int DCH>
__global__ void __launch_bounds__(kTx* kTy) bilateral_fast_kernel(const float* __restrict__ ind,
                                                                  const float* __restrict__ depth,
                                                                  const float* __restrict__ normal,
                                                                  float* __restrict__ out, int w, int h) {
  constexpr int kHy = kTy * kBilRows + 4;
  __shared__ float4 s_col[kHy][kHx];
  __shared__ float4 s_nrm[kHy][kHx];  // xyz, w = depth
  stage_halo<DCH, kHy, kTx * kTy, false>(ind, depth, normal, w, h, blockIdx.x * kTx - 2, blockIdx.y * (kTy * kBilRows) - 2,
                                  &s_col[0][0], &s_nrm[0][0]);
  __syncthreads();
  const int tx = threadIdx.x, ty = threadIdx.y * kBilRows;  // the thread's first tap within the tile
  const int x = blockIdx.x * kTx + tx, y = blockIdx.y * (kTy * kBilRows) + ty;
  if (x >= w || y >= h) return;
  const float4 c0 = s_nrm[ty + 2][tx + 2], c1 = s_nrm[ty + 3][tx + 2];
  // Row 0 belongs to the upper pixel alone and row 5 to the lower one: their weights
  // make a pair, and the lower pixel's wait for its last row.
  float sx = 0.0f, sy = 0.0f, sz = 0.0f, sw = 0.0f, last[5];
#pragma unroll
  for (int dx = 0; dx < 5; dx++) {
    const float4 col = s_col[ty][tx + dx], n = s_nrm[ty][tx + dx], m = s_nrm[ty + 5][tx + dx];
    const p2 wt = fast_weights(pk(n.x - c0.x, m.x - c1.x), pk(n.y - c0.y, m.y - c1.y), pk(n.z - c0.z, m.z - c1.z),
                               pk(n.w - c0.w, m.w - c1.w));
    sx = fmaf(col.x, lo_(wt), sx);
    sy = fmaf(col.y, lo_(wt), sy);
    sz = fmaf(col.z, lo_(wt), sz);
    sw = sw + lo_(wt);
    last[dx] = hi_(wt);
  }
  const p2 cx = pk(c0.x, c1.x), cy = pk(c0.y, c1.y), cz = pk(c0.z, c1.z), cd = pk(c0.w, c1.w);
  p2 ax = pk(sx, 0.0f), ay = pk(sy, 0.0f), az = pk(sz, 0.0f), aw = pk(sw, 0.0f);
#pragma unroll
  for (int r = 1; r < 5; r++) {
#pragma unroll
    for (int dx = 0; dx < 5; dx++) {
      const float4 col = s_col[ty + r][tx + dx], n = s_nrm[ty + r][tx + dx];
      const p2 wt = fast_weights(psub(pk(n.x), cx), psub(pk(n.y), cy), psub(pk(n.z), cz), psub(pk(n.w), cd));
      ax = pfma(pk(col.x), wt, ax);
      ay = pfma(pk(col.y), wt, ay);
      az = pfma(pk(col.z), wt, az);
      aw = padd(aw, wt);
    }
  }
  float4* o = reinterpret_cast<float4*>(out) + (size_t)y * w + x;
  store_filtered(o, lo_(ax), lo_(ay), lo_(az), lo_(aw));
  if (y + 1 >= h) return;
  sx = hi_(ax);
  sy = hi_(ay);
  sz = hi_(az);
  sw = hi_(aw);
#pragma unroll
  for (int dx = 0; dx < 5; dx++) {
    const float4 col = s_col[ty + 5][tx + dx];
    sx = fmaf(col.x, last[dx], sx);
    sy = fmaf(col.y, last[dx], sy);
    sz = fmaf(col.z, last[dx], sz);
    sw = sw + last[dx];
  }
  store_filtered(o + w, sx, sy, sz, sw);
}

// The exact weights.  Bound by the arithmetic of the exponentials, of which two pixels
// that lie in each other's window have the same one (the differences change sign, their
// squares and magnitudes do not).  So each pixel's weights to the 12 taps after it --
// (1..2, 0), (-2..2, 1), (-2..2, 2) -- are evaluated once into shared memory, for the
// tile and the two pixels around it on the left, right and above, and an output reads
// its other 12 from the pixels before it.  The tile's height keeps the block within 48
// KB; 8 and 14 rows measured 217 and 209 us against 209 with 12 before the last columns
// of all rows became one warp's.  3840 x 2160: 315 us with scalar weights per tap, 235
// with packed ones, 206 shared; bound by L1's data pipe (82 % busy, shared memory 70 %) now.
constexpr int kExY = 6;                        // rows of threads
constexpr int kExTile = kExY * kBilRows;       // rows of outputs
constexpr int kExHy = kExTile + 4, kExWy = kExTile + 2;  // rows of the halo, and of weights

template <int DCH>
__global__ void __launch_bounds__(kTx* kExY) bilateral_exact_kernel(const float* __restrict__ ind,
                                                                    const float* __restrict__ depth,
                                                                    const float* __restrict__ normal,
                                                                    float* __restrict__ out, int w, int h) {
  constexpr int kThreads = kTx * kExY;
  __shared__ float4 s_col[kExHy][kHx];
  __shared__ float4 s_nrm[kExHy][kHx];  // xyz, w = depth
  __shared__ float s_w[12][kExWy][kHx];
  stage_halo<DCH, kExHy, kThreads, true>(ind, depth, normal, w, h, blockIdx.x * kTx - 2, blockIdx.y * kExTile - 2,
                                   &s_col[0][0], &s_nrm[0][0]);
  __syncthreads();
  // Two rows of a column a lane: a warp takes two rows' first 32 columns, or the last
  // four of all rows.  Taps past the halo's sides belong to pairs that no output has;
  // they read its last column.
  static_assert(kExWy / 2 * 4 <= 32, "the last columns of all rows are one warp's");
  for (int u = threadIdx.y; u <= kExWy / 2; u += kExY) {
    const bool body = u < kExWy / 2;
    const int y = 2 * (body ? u : threadIdx.x / 4), x = body ? threadIdx.x : 32 + threadIdx.x % 4;
    if (y >= kExWy) break;
    const float4 c0 = s_nrm[y][x], c1 = s_nrm[y + 1][x];
    auto weights = [&](int f, const float4& n, const float4& m) {  // taps of the upper and of the lower pixel
      const p2 ex = pk(n.x - c0.x, m.x - c1.x), ey = pk(n.y - c0.y, m.y - c1.y), ez = pk(n.z - c0.z, m.z - c1.z);
      const p2 q = pmul(padd(padd(pmul(ex, ex), pmul(ey, ey)), pmul(ez, ez)), pk(20.0f));
      const p2 d = pmul(pk(n.w - c0.w, m.w - c1.w), pk(10.5f));
      const p2 wt = exp_neg(pk(fabsf(lo_(d)) + lo_(q), fabsf(hi_(d)) + hi_(q)));
      s_w[f][y][x] = lo_(wt);
      s_w[f][y + 1][x] = hi_(wt);
    };
#pragma unroll
    for (int dx = -2; dx <= 2; dx++) {
      const int sx = iclamp(x + dx, 0, kHx - 1);
      const float4 n1 = s_nrm[y + 1][sx], n2 = s_nrm[y + 2][sx], n3 = s_nrm[y + 3][sx];
      if (dx > 0) weights(dx - 1, s_nrm[y][sx], n1);
      weights(4 + dx, n1, n2);
      weights(9 + dx, n2, n3);
    }
  }
  __syncthreads();
  const int tx = threadIdx.x, ty = threadIdx.y * kBilRows;  // the thread's first tap within the tile
  const int x = blockIdx.x * kTx + tx, y = blockIdx.y * kExTile + ty;
  if (x >= w || y >= h) return;
  // Weight of the pixel in halo row py of the thread's column to its tap (dx, dy); to
  // itself: in its light.
  auto weight = [&](int py, int dx, int dy) {
    const int px = tx + 2;
    if (dy == 0) return dx > 0 ? s_w[dx - 1][py][px] : s_w[-dx - 1][py][px + dx];
    if (dy > 0) return s_w[5 * dy - 1 + dx][py][px];
    return s_w[-5 * dy - 1 - dx][py + dy][px + dx];
  };
  float sx = 0.0f, sy = 0.0f, sz = 0.0f, sw = 0.0f;
#pragma unroll
  for (int dx = 0; dx < 5; dx++) {  // row 0: the upper pixel's alone
    const float4 col = s_col[ty][tx + dx];
    const float wt = weight(ty + 2, dx - 2, -2);
    sx = sx + col.x * wt;
    sy = sy + col.y * wt;
    sz = sz + col.z * wt;
    sw = sw + wt;
  }
  p2 ax = pk(sx, 0.0f), ay = pk(sy, 0.0f), az = pk(sz, 0.0f), aw = pk(sw, 0.0f);
#pragma unroll
  for (int r = 1; r < 5; r++) {
#pragma unroll
    for (int dx = 0; dx < 5; dx++) {
      const float4 col = s_col[ty + r][tx + dx];
      const p2 wt = pk(dx == 2 && r == 2 ? col.w : weight(ty + 2, dx - 2, r - 2),
                       dx == 2 && r == 3 ? col.w : weight(ty + 3, dx - 2, r - 3));
      ax = padd(ax, pmul(pk(col.x), wt));
      ay = padd(ay, pmul(pk(col.y), wt));
      az = padd(az, pmul(pk(col.z), wt));
      aw = padd(aw, wt);
    }
  }
  float4* o = reinterpret_cast<float4*>(out) + (size_t)y * w + x;
  store_filtered(o, lo_(ax), lo_(ay), lo_(az), lo_(aw));
  if (y + 1 >= h) return;
  sx = hi_(ax);
  sy = hi_(ay);
  sz = hi_(az);
  sw = hi_(aw);
#pragma unroll
  for (int dx = 0; dx < 5; dx++) {  // row 5: the lower pixel's
    const float4 col = s_col[ty + 5][tx + dx];
    const float wt = weight(ty + 3, dx - 2, 2);
    sx = sx + col.x * wt;
    sy = sy + col.y * wt;
    sz = sz + col.z * wt;
    sw = sw + wt;
  }
  store_filtered(o + w, sx, sy, sz, sw);
}

// denoiser.frag:72-184 with radius 2: 16 equations [depth, 1] -> colour over
// the taps y, x in [-2, 2), Gramian + 1e-7 I, closed-form 2x2 inverse.
template <int DCH> __device__ __forceinline__ float depth_sample(const float* p, int w, int h, float s, float t) {
  Bilin B = bilin(s, t, w, h);
  return blend1(B, depth_at<DCH>(p, B.o00), depth_at<DCH>(p, B.o10), depth_at<DCH>(p, B.o01),
                depth_at<DCH>(p, B.o11));
}

template <int DCH>
__global__ void __launch_bounds__(kTx* kTy) denoise_kernel(const float* __restrict__ noisy,
                                                           const float* __restrict__ depth, float* __restrict__ out,
                                                           int w, int h, int radius) {
  const int x = blockIdx.x * kTx + threadIdx.x, y = blockIdx.y * kTy + threadIdx.y;
  if (x >= w || y >= h) return;
  const float W = (float)w, H = (float)h;
  const float cpx = (float)x + 0.5f, cpy = (float)y + 0.5f;
  if (radius == 0) {
    reinterpret_cast<float4*>(out)[y * w + x] = sample4(noisy, w, h, div_(cpx, W), div_(cpy, H));
    return;
  }
  float p0[16];
  float col[16][3];
  int i = 0;
#pragma unroll
  for (int dy = -2; dy < 2; dy++)
#pragma unroll
    for (int dx = -2; dx < 2; dx++) {
      const float sx = div_(cpx + (float)dx, W), sy = div_(cpy + (float)dy, H);
      p0[i] = depth_sample<DCH>(depth, w, h, sx, sy);
      float4 c = sample4(noisy, w, h, sx, sy);
      col[i][0] = c.x;
      col[i][1] = c.y;
      col[i][2] = c.z;
      i++;
    }
  float g00 = 0.0f, g01 = 0.0f, g10 = 0.0f, g11 = 0.0f;
#pragma unroll
  for (int k = 0; k < 16; k++) g00 = g00 + p0[k] * p0[k];
  g00 = g00 + 1e-7f;
#pragma unroll
  for (int k = 0; k < 16; k++) g01 = g01 + p0[k] * 1.0f;
  g01 = g01 + 0.0f;
#pragma unroll
  for (int k = 0; k < 16; k++) g10 = g10 + 1.0f * p0[k];
  g10 = g10 + 0.0f;
#pragma unroll
  for (int k = 0; k < 16; k++) g11 = g11 + 1.0f * 1.0f;
  g11 = g11 + 1e-7f;
  const float det = g00 * g11 - g01 * g10;
  const float inv00 = div_(g11, det), inv01 = div_(-g01, det), inv10 = div_(-g10, det), inv11 = div_(g00, det);
  const float cp0 = depth_sample<DCH>(depth, w, h, div_(cpx, W), div_(cpy, H));
  float res[3];
#pragma unroll
  for (int ch = 0; ch < 3; ch++) {
    float m0 = 0.0f, m1 = 0.0f;
#pragma unroll
    for (int k = 0; k < 16; k++) m0 = m0 + p0[k] * col[k][ch];
#pragma unroll
    for (int k = 0; k < 16; k++) m1 = m1 + 1.0f * col[k][ch];
    float c0 = 0.0f, c1 = 0.0f;
    c0 = c0 + inv00 * m0;
    c0 = c0 + inv10 * m1;
    c1 = c1 + inv01 * m0;
    c1 = c1 + inv11 * m1;
    float v = 0.0f;
    v = v + c0 * cp0;
    v = v + c1 * 1.0f;
    res[ch] = v;
  }
  reinterpret_cast<float4*>(out)[y * w + x] = make_float4(res[0], res[1], res[2], 1.0f);
}

// finalGatherer.frag:42-59: direct + indirect * albedo (the :50-57 loop adds
// only zero-weighted terms).
// Rows per thread: every thread issues the loads of kRowsPerThread pixels before it
// computes or stores any, which keeps enough bytes in flight per SM to stream at HBM
// speed.  Adjacent rows, whose taps are in part the same (3840 x 2160 97.0 us with rows
// kTy apart, 95.2 so; 114 with one row a thread).
constexpr int kRowsPerThread = 2;

__global__ void __launch_bounds__(kTx* kTy) final_gather_kernel(const float* __restrict__ direct,
                                                                const float* __restrict__ ind,
                                                                const float* __restrict__ albedo,
                                                                float* __restrict__ out, int w, int h) {
  const int x = blockIdx.x * kTx + threadIdx.x;
  const int y0 = (blockIdx.y * kTy + threadIdx.y) * kRowsPerThread;
  if (x >= w) return;
  float4 d[kRowsPerThread][4], i[kRowsPerThread][4], a[kRowsPerThread][4];
  Bilin B[kRowsPerThread];
#pragma unroll
  for (int r = 0; r < kRowsPerThread; r++) {
    const int y = min(y0 + r, h - 1);  // rows past the image repeat the last one; not stored
    const float s = div_((float)x + 0.5f, (float)w), t = div_((float)y + 0.5f, (float)h);
    B[r] = bilin(s, t, w, h);
    const int o[4] = {B[r].o00, B[r].o10, B[r].o01, B[r].o11};
#pragma unroll
    for (int k = 0; k < 4; k++) {
      d[r][k] = ld4(direct, o[k]);
      i[r][k] = ld4(ind, o[k]);
      a[r][k] = ld4(albedo, o[k]);
    }
  }
#pragma unroll
  for (int r = 0; r < kRowsPerThread; r++) {
    const int y = y0 + r;
    if (y >= h) break;
    const float4 dd = blend4(B[r], d[r][0], d[r][1], d[r][2], d[r][3]);
    const float4 ii = blend4(B[r], i[r][0], i[r][1], i[r][2], i[r][3]);
    const float4 aa = blend4(B[r], a[r][0], a[r][1], a[r][2], a[r][3]);
    reinterpret_cast<float4*>(out)[y * w + x] =
        make_float4(dd.x + ii.x * aa.x, dd.y + ii.y * aa.y, dd.z + ii.z * aa.z, dd.w + ii.w * aa.w);
  }
}

// Permutations.  Each thread owns one pixel of the INTERLEAVED image, so reads
// (deinterleave) or writes (interleave) on that side are contiguous, and the
// other side is touched in runs of 32/grid_x consecutive texels per warp.
//   deinterleave.frag: dst[p] = src[InterleavePixel(p)]  ==  dst[DeinterleavePixel(q)] = src[q]
//   interleave.frag:   dst[q] = src[DeinterleavePixel(q)]
// Each thread moves kPermuteRows pixels (kTy rows apart), all loads first.
constexpr int kPermuteRows = 4;

template <int CH> struct Texel;
template <> struct Texel<4> { using T = float4; };
template <> struct Texel<2> { using T = float2; };
template <> struct Texel<1> { using T = float; };

template <int CH, bool INTERLEAVE>
__global__ void __launch_bounds__(kTx* kTy) permute_kernel(const float* __restrict__ src, float* __restrict__ dst,
                                                           int w, int h, int gx, int gy) {
  using T = typename Texel<CH>::T;
  const int x = blockIdx.x * kTx + threadIdx.x;
  const int y0 = blockIdx.y * (kTy * kPermuteRows) + threadIdx.y;
  if (x >= w) return;
  const int dvx = w / gx, dvy = h / gy;
  const int dx = (x % gx) * dvx + x / gx;  // DeinterleavePixel, x part
  T v[kPermuteRows];
  size_t to[kPermuteRows];
#pragma unroll
  for (int r = 0; r < kPermuteRows; r++) {
    const int y = y0 + r * kTy;
    if (y < h) {
      const int dy = (y % gy) * dvy + y / gy;
      const size_t qi = (size_t)y * w + x, di = (size_t)dy * w + dx;
      to[r] = INTERLEAVE ? qi : di;
      v[r] = __ldg(reinterpret_cast<const T*>(src) + (INTERLEAVE ? di : qi));
    }
  }
#pragma unroll
  for (int r = 0; r < kPermuteRows; r++)
    if (y0 + r * kTy < h) reinterpret_cast<T*>(dst)[to[r]] = v[r];
}

dim3 grid2d(int w, int h) { return dim3((w + kTx - 1) / kTx, (h + kTy - 1) / kTy); }

}  // namespace

int launch_bilateral(const float* ind, const float* depth, int depth_ch, const float* normal, float* out, int w, int h,
                     cudaStream_t stream, bool fast) {
  const int rows = fast ? kTy : kExY;
  const dim3 grid((w + kTx - 1) / kTx, (h + rows * kBilRows - 1) / (rows * kBilRows)), block(kTx, rows);
  auto go = [&](auto kernel) { kernel<<<grid, block, 0, stream>>>(ind, depth, normal, out, w, h); };
  if (depth_ch == 2) {
    if (fast) go(bilateral_fast_kernel<2>);
    else go(bilateral_exact_kernel<2>);
  } else {
    if (fast) go(bilateral_fast_kernel<1>);
    else go(bilateral_exact_kernel<1>);
  }
  GI_CHECK_LAUNCH("bilateral_kernel");
  count_launches(1);
  return GI_OK;
}

int launch_final_gather(const float* direct, const float* ind, const float* albedo, float* out, int w, int h,
                        cudaStream_t stream) {
  const dim3 grid((w + kTx - 1) / kTx, (h + kTy * kRowsPerThread - 1) / (kTy * kRowsPerThread));
  final_gather_kernel<<<grid, dim3(kTx, kTy), 0, stream>>>(direct, ind, albedo, out, w, h);
  GI_CHECK_LAUNCH("final_gather_kernel");
  count_launches(1);
  return GI_OK;
}

int launch_deinterleave(const float* src, float* dst, int w, int h, int ch, int gx, int gy, bool inverse,
                        cudaStream_t stream) {
  dim3 g((w + kTx - 1) / kTx, (h + kTy * kPermuteRows - 1) / (kTy * kPermuteRows)), b(kTx, kTy);
  if (inverse) {
    if (ch == 4) permute_kernel<4, true><<<g, b, 0, stream>>>(src, dst, w, h, gx, gy);
    else if (ch == 2) permute_kernel<2, true><<<g, b, 0, stream>>>(src, dst, w, h, gx, gy);
    else permute_kernel<1, true><<<g, b, 0, stream>>>(src, dst, w, h, gx, gy);
  } else {
    if (ch == 4) permute_kernel<4, false><<<g, b, 0, stream>>>(src, dst, w, h, gx, gy);
    else if (ch == 2) permute_kernel<2, false><<<g, b, 0, stream>>>(src, dst, w, h, gx, gy);
    else permute_kernel<1, false><<<g, b, 0, stream>>>(src, dst, w, h, gx, gy);
  }
  GI_CHECK_LAUNCH("permute_kernel");
  count_launches(1);
  return GI_OK;
}

}  // namespace gi

using namespace gi;

extern "C" int gi_deinterleave(const float* src, float* dst, int width, int height, int channels, int grid_x,
                               int grid_y, void* stream) {
  GI_CHECK_ARG(src && dst && src != dst, "gi_deinterleave: null or aliased buffers");
  GI_CHECK_ARG(channels == 1 || channels == 2 || channels == 4, "gi_deinterleave: channels must be 1, 2 or 4");
  GI_CHECK_ARG(grid_x >= 1 && grid_y >= 1 && width >= grid_x && height >= grid_y && width % grid_x == 0 &&
                   height % grid_y == 0,
               "gi_deinterleave: size must be a multiple of the grid");
  GI_CHECK_ARG(aligned16(src) && aligned16(dst), "gi_deinterleave: unaligned buffer");
  return launch_deinterleave(src, dst, width, height, channels, grid_x, grid_y, false, (cudaStream_t)stream);
}

extern "C" int gi_interleave(const float* src, float* dst, int width, int height, int channels, int grid_x, int grid_y,
                             void* stream) {
  GI_CHECK_ARG(src && dst && src != dst, "gi_interleave: null or aliased buffers");
  GI_CHECK_ARG(channels == 1 || channels == 2 || channels == 4, "gi_interleave: channels must be 1, 2 or 4");
  GI_CHECK_ARG(grid_x >= 1 && grid_y >= 1 && width >= grid_x && height >= grid_y && width % grid_x == 0 &&
                   height % grid_y == 0,
               "gi_interleave: size must be a multiple of the grid");
  GI_CHECK_ARG(aligned16(src) && aligned16(dst), "gi_interleave: unaligned buffer");
  return launch_deinterleave(src, dst, width, height, channels, grid_x, grid_y, true, (cudaStream_t)stream);
}

extern "C" int gi_bilateral(const float* indirect, const float* depth_moments, const float* normal, float* out,
                            int width, int height, void* stream) {
  GI_CHECK_ARG(indirect && depth_moments && normal && out && width >= 1 && height >= 1, "gi_bilateral: bad arguments");
  GI_CHECK_ARG(out != indirect, "gi_bilateral: in-place filtering is not supported");
  GI_CHECK_ARG(aligned16(indirect) && aligned16(depth_moments) && aligned16(normal) && aligned16(out),
               "gi_bilateral: unaligned buffer");
  return launch_bilateral(indirect, depth_moments, 2, normal, out, width, height, (cudaStream_t)stream);
}

extern "C" int gi_denoise(const float* noisy, const float* depth_moments, const float* normal, float* out, int width,
                          int height, int radius, void* stream) {
  (void)normal;  // bound by the reference pass (SSVGIRenderer.h:293) but unused by its equations
  GI_CHECK_ARG(noisy && depth_moments && out && width >= 1 && height >= 1, "gi_denoise: bad arguments");
  GI_CHECK_ARG(radius == 0 || radius == 2, "gi_denoise: radius must be 0 or 2 (denoiser.frag:115)");
  GI_CHECK_ARG(out != noisy, "gi_denoise: in-place filtering is not supported");
  GI_CHECK_ARG(aligned16(noisy) && aligned16(depth_moments) && aligned16(out), "gi_denoise: unaligned buffer");
  denoise_kernel<2><<<grid2d(width, height), dim3(kTx, kTy), 0, (cudaStream_t)stream>>>(noisy, depth_moments, out,
                                                                                       width, height, radius);
  GI_CHECK_LAUNCH("denoise_kernel");
  count_launches(1);
  return GI_OK;
}

extern "C" int gi_final_gather(const float* direct, const float* indirect, const float* albedo, float* out, int width,
                               int height, void* stream) {
  GI_CHECK_ARG(direct && indirect && albedo && out && width >= 1 && height >= 1, "gi_final_gather: bad arguments");
  GI_CHECK_ARG(aligned16(direct) && aligned16(indirect) && aligned16(albedo) && aligned16(out),
               "gi_final_gather: unaligned buffer");
  return launch_final_gather(direct, indirect, albedo, out, width, height, (cudaStream_t)stream);
}
