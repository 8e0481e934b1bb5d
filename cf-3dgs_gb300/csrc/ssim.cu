// Fused SSIM (structural similarity) with an 11x11 Gaussian window, forward and
// backward, as the CF-3DGS pose loss uses it: utils/loss_utils.py:23-58 and
// trainer/losses.py:147-251 (window sigma 1.5, zero padding 5, one window per channel,
// C1 = 0.01^2, C2 = 0.03^2, mean over every channel and pixel).
//
// Per channel and pixel p the five windowed moments mu1 = W*x, mu2 = W*y, exx = W*x^2,
// eyy = W*y^2, exy = W*xy give
//   S = (2 mu1 mu2 + C1)(2 s12 + C2) / ((mu1^2 + mu2^2 + C1)(s11 + s22 + C2)),
//   s11 = exx - mu1^2, s22 = eyy - mu2^2, s12 = exy - mu1 mu2.
// The forward writes, besides the partial sums of S, the three maps
//   a = dS/dmu1, b = dS/dexx, c = dS/dexy    (times 1/count: d mean / d S_p)
// and the backward forms dL/dx_q = g (W*a + 2 x_q W*b + y_q W*c)_q with g = dL/dmean
// (the window is symmetric, so the transposed convolution is the same convolution).
//
// Both kernels work on 32x32 output tiles of one channel: the tile and a 5-pixel halo
// are staged in shared memory (zero outside the image); a horizontal 11-tap pass over all
// staged rows and then a vertical pass compute runs of 4 outputs per thread, each input
// loaded once per run and the window slid in registers. They are bound by the issue of
// the taps (127 multiply-adds per output and moment set, against 20 bytes per element of
// traffic that mostly stays in L2), so the taps run on packed pairs — (x, y) and
// (x^2, y^2) in the forward, two of the three maps in the backward — and the horizontal
// sums are stored and loaded as pairs. 3x1080x1920: photometric forward 61 us (issue 67%
// busy, shared-memory pipe 52%), backward 42 us; SSIM alone took 55.7 and 49.2 us with
// scalar taps.
//
// The photometric form (PHOTO) is the whole CF-3DGS image loss of a render x,
//   (1 - lambda) mean |c - y| + lambda (1 - SSIM(c, y)), c = clamp(x, 0, 1)
// (trainer/losses.py:98-136, scene/gaussian_model_cf.py:885), in the same two passes: the
// forward clamps as it reads and also sums |c - y|, the backward adds the L1 sign and
// masks by the clamp. As separate clamp, L1 and SSIM calls the loss and its gradient took
// 21 launches (218 us of kernels) at 3x1080x1920; here 3 launches, 111 us.
#include <cuda.h>  // CUtensorMap and its enumerations (the encoder comes from the runtime)
#include <cudaTypedefs.h>

#include <cmath>

#include "cfgs_internal.cuh"

namespace cfgs {

constexpr int kSsimR = 5;  // window radius
constexpr int kSsimTaps = 2 * kSsimR + 1;
constexpr int kSsimT = 32;                        // output tile: 32 x 32
constexpr int kSsimS = kSsimT + 2 * kSsimR;       // staged rows / columns (42)
constexpr int kSsimSP = 48;  // staged row: columns x0-8 .. x0+39 (a 16-byte-aligned tensor-copy box)
constexpr int kSsimOff = 3;  // staged column of x0 - 5
constexpr uint32_t kSsimBoxBytes = sizeof(float) * kSsimSP * kSsimS;
constexpr int kSsimHP = kSsimT + 1;               // horizontal-result row stride (33)
constexpr int kSsimRun = 4;                       // outputs per thread along a row / column
constexpr int kSsimThreads = 256;
constexpr int kSsimFoldBlocks = 16;  // blocks of the fold of one partial pair per tile at most
constexpr float kSsimC1 = 0.0001f, kSsimC2 = 0.0009f;

__constant__ float c_ssim_w[kSsimTaps];

// Reciprocal to within one unit in the last place (the loss is held to a tolerance).
__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

struct SsimDims {
  int C, H, W, tiles_x, tiles_y;
};

__device__ __forceinline__ float load_or_zero(const float* img, int H, int W, int y, int x) {
  return (y >= 0 && y < H && x >= 0 && x < W) ? img[(size_t)y * W + x] : 0.0f;
}

// One 48 x 42 box of plane z at (x, y) into shared memory by a tensor copy; coordinates
// outside the tensor read as zero.
__device__ __forceinline__ void tma_box(float* dst, const CUtensorMap* map, int x, int y, int z, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
      "[%5];" ::"r"(smem_addr(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(bar)
      : "memory");
}

// Stages `planes` boxes of the tile's rows y0-5 .. y0+36 and columns x0-8 .. x0+39 (zero
// outside the image): by tensor copies (TMA) or by plain loads. Returns false if a
// bounded wait on the copies ran out.
template <bool TMA, int NP>
__device__ __forceinline__ bool stage_planes(float* (&dst)[NP], const float* const (&src)[NP],
                                             const CUtensorMap* const (&maps)[NP], const int (&zidx)[NP], int H,
                                             int W, int x0, int y0, uint64_t* bar_word) {
  if constexpr (TMA) {
    const uint32_t bar = smem_addr(bar_word);
    if (threadIdx.x == 0) mbar_init(bar, 1);
    __syncthreads();
    if (threadIdx.x == 0) {
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(NP * kSsimBoxBytes)
                   : "memory");
#pragma unroll
      for (int p = 0; p < NP; ++p) tma_box(dst[p], maps[p], x0 - 8, y0 - kSsimR, zidx[p], bar);
    }
    return mbar_wait(bar, 0);
  } else {
    for (int i = threadIdx.x; i < kSsimS * kSsimS; i += kSsimThreads) {
      const int r = i / kSsimS, c = i % kSsimS;
#pragma unroll
      for (int p = 0; p < NP; ++p)
        dst[p][r * kSsimSP + kSsimOff + c] = load_or_zero(src[p], H, W, y0 + r - kSsimR, x0 + c - kSsimR);
    }
    return true;
  }
}

// Block-wide float64 sum of one float per thread (kSsimThreads threads), fixed order,
// valid in thread 0. One warp adds the floats from shared memory: the float64 pipe issues
// about two operations per cycle and SM, and a shuffle reduction by every warp kept it
// busy for half of the forward.
__device__ __forceinline__ double block_sum_fixed(float v, float* sh) {
  sh[threadIdx.x] = v;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x < 32) {
#pragma unroll
    for (int w = 0; w < kSsimThreads / 32; ++w) t += (double)sh[threadIdx.x + 32 * w];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  }
  return t;
}

// Block-wide float sum (the precision of the L1 loss's own block sums), fixed order, valid
// in thread 0.
__device__ __forceinline__ float block_sum_float(float v, float* sh) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  float t = 0.0f;
  if (threadIdx.x == 0)
    for (int w = 0; w < kSsimThreads / 32; ++w) t += sh[w];
  return t;
}

// The six distinct weights of the symmetric window as packed pairs.
struct WindowPairs {
  float2 w[kSsimR + 1];
  __device__ __forceinline__ WindowPairs() {
#pragma unroll
    for (int k = 0; k <= kSsimR; ++k) w[k] = splat2(c_ssim_w[k]);
  }
  __device__ __forceinline__ float2 operator[](int tap) const { return w[tap <= kSsimR ? tap : 2 * kSsimR - tap]; }
};

// clamp to [0, 1] that keeps a NaN, as torch.clamp does.
__device__ __forceinline__ float clamp01(float x) { return x != x ? x : fminf(fmaxf(x, 0.0f), 1.0f); }

template <bool TMA, bool PHOTO>
__global__ void __launch_bounds__(kSsimThreads) k_ssim_fwd(SsimDims d, const float* __restrict__ img1,
                                                           const float* __restrict__ img2, float* __restrict__ maps,
                                                           double2* __restrict__ partials,
                                                           unsigned int* __restrict__ fold_counter, float inv_count,
                                                           const __grid_constant__ CUtensorMap t1,
                                                           const __grid_constant__ CUtensorMap t2) {
  __shared__ __align__(128) float s_x[kSsimS * kSsimSP];
  __shared__ __align__(128) float s_y[kSsimS * kSsimSP];
  __shared__ float2 s_hm[kSsimS * kSsimHP];  // horizontal sums of (x, y)
  __shared__ float2 s_hs[kSsimS * kSsimHP];  // of (xx, yy)
  __shared__ float s_hp[kSsimS * kSsimHP];   // of xy
  __shared__ float s_red[kSsimThreads], s_red_l1[kSsimThreads / 32];
  __shared__ __align__(8) uint64_t s_bar;
  const int tile = blockIdx.x, ch = blockIdx.y;
  const int x0 = (tile % d.tiles_x) * kSsimT, y0 = (tile / d.tiles_x) * kSsimT;
  const size_t plane = (size_t)d.H * d.W;
  float* dst[2] = {s_x, s_y};
  const float* const src[2] = {img1 + ch * plane, img2 + ch * plane};
  const CUtensorMap* const tm[2] = {&t1, &t2};
  const int zi[2] = {ch, ch};
  const bool staged = stage_planes<TMA, 2>(dst, src, tm, zi, d.H, d.W, x0, y0, &s_bar);
  const WindowPairs w;
  __syncthreads();
  // horizontal: item = (staged row r, run of 4 output columns)
  for (int it = threadIdx.x; it < kSsimS * (kSsimT / kSsimRun); it += kSsimThreads) {
    const int r = it / (kSsimT / kSsimRun), c0 = (it % (kSsimT / kSsimRun)) * kSsimRun;
    const float* xr = s_x + r * kSsimSP + kSsimOff + c0;
    const float* yr = s_y + r * kSsimSP + kSsimOff + c0;
    float2 m[kSsimRun], q[kSsimRun];
    float p[kSsimRun];
#pragma unroll
    for (int u = 0; u < kSsimRun; ++u) {
      m[u] = q[u] = splat2(0.f);
      p[u] = 0.f;
    }
#pragma unroll
    for (int k = 0; k < kSsimRun + 2 * kSsimR; ++k) {
      const float2 v = make_float2(PHOTO ? clamp01(xr[k]) : xr[k], yr[k]);
      const float2 vv = mul2(v, v);
      const float xy = v.x * v.y;
#pragma unroll
      for (int u = 0; u < kSsimRun; ++u) {
        const int tap = k - u;
        if (tap >= 0 && tap < kSsimTaps) {
          m[u] = fma2(w[tap], v, m[u]);
          q[u] = fma2(w[tap], vv, q[u]);
          p[u] = fmaf(w[tap].x, xy, p[u]);
        }
      }
    }
#pragma unroll
    for (int u = 0; u < kSsimRun; ++u) {
      s_hm[r * kSsimHP + c0 + u] = m[u];
      s_hs[r * kSsimHP + c0 + u] = q[u];
      s_hp[r * kSsimHP + c0 + u] = p[u];
    }
  }
  __syncthreads();
  // vertical: item = (output column c, run of 4 output rows); one item per thread
  float ssum = 0.f, lsum = 0.f;
  {
    const int c = threadIdx.x % kSsimT, r0 = (threadIdx.x / kSsimT) * kSsimRun;
    float2 m[kSsimRun], q[kSsimRun];
    float p[kSsimRun];
#pragma unroll
    for (int u = 0; u < kSsimRun; ++u) {
      m[u] = q[u] = splat2(0.f);
      p[u] = 0.f;
    }
#pragma unroll
    for (int k = 0; k < kSsimRun + 2 * kSsimR; ++k) {
      const float2 vm = s_hm[(r0 + k) * kSsimHP + c], vs = s_hs[(r0 + k) * kSsimHP + c];
      const float vp = s_hp[(r0 + k) * kSsimHP + c];
#pragma unroll
      for (int u = 0; u < kSsimRun; ++u) {
        const int tap = k - u;
        if (tap >= 0 && tap < kSsimTaps) {
          m[u] = fma2(w[tap], vm, m[u]);
          q[u] = fma2(w[tap], vs, q[u]);
          p[u] = fmaf(w[tap].x, vp, p[u]);
        }
      }
    }
    const int px = x0 + c;
#pragma unroll
    for (int u = 0; u < kSsimRun; ++u) {
      const int py = y0 + r0 + u;
      if (py >= d.H || px >= d.W) continue;
      const float mu1 = m[u].x, mu2 = m[u].y, exx = q[u].x, eyy = q[u].y, exy = p[u];
      const float m11 = mu1 * mu1, m22 = mu2 * mu2, m12 = mu1 * mu2;
      const float A = 2.f * m12 + kSsimC1, B = 2.f * (exy - m12) + kSsimC2;
      const float Cc = m11 + m22 + kSsimC1, D = (exx - m11) + (eyy - m22) + kSsimC2;
      const float rA = rcp_approx(A), rB = rcp_approx(B), rC = rcp_approx(Cc), rD = rcp_approx(D);
      const float S = (A * B) * (rC * rD);
      ssum += S;
      if (PHOTO) {
        const int at = (r0 + u + kSsimR) * kSsimSP + kSsimOff + c + kSsimR;
        lsum += fabsf(clamp01(s_x[at]) - s_y[at]);
      }
      const size_t o = ch * plane + (size_t)py * d.W + px;
      // dS/dmu1 = S (2 mu2/A - 2 mu2/B - 2 mu1/C + 2 mu1/D); dS/dexx = -S/D; dS/dexy = 2 S/B
      const float da = S * (2.f * mu2 * (rA - rB) + 2.f * mu1 * (rD - rC));
      maps[o] = inv_count * da;
      maps[(size_t)d.C * plane + o] = inv_count * (-S * rD);
      maps[2 * (size_t)d.C * plane + o] = inv_count * (2.f * S * rB);
    }
  }
  const double t = block_sum_fixed(ssum, s_red);
  const float l = PHOTO ? block_sum_float(lsum, s_red_l1) : 0.0f;
  if (threadIdx.x == 0) {
    // a copy that did not arrive makes the mean NaN (visibly invalid)
    partials[(size_t)ch * gridDim.x + tile] =
        make_double2(staged ? t : __longlong_as_double(0x7ff8000000000000ll), (double)l);
    if (blockIdx.x == 0 && blockIdx.y == 0) *fold_counter = 0u;  // for the fold, the next launch
  }
}

// Mean SSIM and (PHOTO) mean |c - y| from the per-tile partial sums, in a fixed order: out =
// w_l1 mean|c - y| + w_ssim SSIM + constant. Block b sums its share of the partials into
// block_sums[b], the last block to finish adds those in block order. Several blocks,
// because one SM's float64 pipe took 9.4 us for the 6120 pairs of 3x1080x1920; 7.5 us with
// up to 16.
__device__ __forceinline__ double2 block_sum_pair(double2 v, double2* sh) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // after the first exchange lanes below 16 sum v.x, the others v.y
  const bool up = lane & 16;
  double t = (up ? v.y : v.x) + __shfl_xor_sync(0xffffffffu, up ? v.x : v.y, 16);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  if (lane == 0) sh[warp].x = t;
  if (lane == 16) sh[warp].y = t;
  __syncthreads();
  double2 r = make_double2(0.0, 0.0);
  if (threadIdx.x == 0)
    for (int w = 0; w < kSsimThreads / 32; ++w) {
      r.x += sh[w].x;
      r.y += sh[w].y;
    }
  return r;  // valid in thread 0
}

__global__ void __launch_bounds__(kSsimThreads) k_ssim_fold(const double2* __restrict__ partials, int count,
                                                            double2* block_sums, unsigned int* counter,
                                                            double inv_count, double w_l1, double w_ssim,
                                                            double constant, float* __restrict__ out) {
  __shared__ double2 s_red[kSsimThreads / 32];
  double2 v = make_double2(0.0, 0.0);
#pragma unroll 2
  for (int i = blockIdx.x * kSsimThreads + threadIdx.x; i < count; i += gridDim.x * kSsimThreads) {
    const double2 p = partials[i];
    v.x += p.x;
    v.y += p.y;
  }
  v = block_sum_pair(v, s_red);
  if (threadIdx.x != 0) return;
  block_sums[blockIdx.x] = v;
  __threadfence();
  if (atomicAdd(counter, 1u) != gridDim.x - 1) return;
  __threadfence();
  double2 t = make_double2(0.0, 0.0);
  for (unsigned b = 0; b < gridDim.x; ++b) {
    t.x += __ldcg(&block_sums[b].x);
    t.y += __ldcg(&block_sums[b].y);
  }
  *out = (float)(w_ssim * (t.x * inv_count) + w_l1 * (t.y * inv_count) + constant);
}

// dL/dimg1 = g w_ssim (W*a + 2 x W*b + y W*c), g = *dL_dmean; PHOTO: with x clamped, plus
// g w_l1 sign(c - y) / count, where the clamp passes (0 <= x <= 1).
template <bool TMA, bool PHOTO>
__global__ void __launch_bounds__(kSsimThreads) k_ssim_bwd(SsimDims d, const float* __restrict__ img1,
                                                           const float* __restrict__ img2,
                                                           const float* __restrict__ maps,
                                                           const float* __restrict__ dL_dmean, float w_ssim,
                                                           float w_l1_over_count, float* __restrict__ dL_dimg1,
                                                           const __grid_constant__ CUtensorMap tmaps) {
  __shared__ __align__(128) float s_m[3][kSsimS * kSsimSP];
  __shared__ float2 s_hab[kSsimS * kSsimHP];
  __shared__ float s_hc[kSsimS * kSsimHP];
  __shared__ __align__(8) uint64_t s_bar;
  const int tile = blockIdx.x, ch = blockIdx.y;
  const int x0 = (tile % d.tiles_x) * kSsimT, y0 = (tile / d.tiles_x) * kSsimT;
  const size_t plane = (size_t)d.H * d.W;
  float* dst[3] = {s_m[0], s_m[1], s_m[2]};
  const float* const src[3] = {maps + (size_t)ch * plane, maps + ((size_t)d.C + ch) * plane,
                               maps + (2 * (size_t)d.C + ch) * plane};
  const CUtensorMap* const tm[3] = {&tmaps, &tmaps, &tmaps};
  const int zi[3] = {ch, d.C + ch, 2 * d.C + ch};
  const bool staged = stage_planes<TMA, 3>(dst, src, tm, zi, d.H, d.W, x0, y0, &s_bar);
  const WindowPairs w;
  // this thread's pixels of both images, on their way while the taps run
  const int c = threadIdx.x % kSsimT, r0 = (threadIdx.x / kSsimT) * kSsimRun;
  const int px = x0 + c;
  float x[kSsimRun], y[kSsimRun];
#pragma unroll
  for (int u = 0; u < kSsimRun; ++u) {
    const int py = y0 + r0 + u;
    const bool in = py < d.H && px < d.W;
    const size_t o = ch * plane + (size_t)py * d.W + px;
    x[u] = in ? img1[o] : 0.f;
    y[u] = in ? img2[o] : 0.f;
  }
  const float g = *dL_dmean;
  __syncthreads();
  for (int it = threadIdx.x; it < kSsimS * (kSsimT / kSsimRun); it += kSsimThreads) {
    const int r = it / (kSsimT / kSsimRun), c0 = (it % (kSsimT / kSsimRun)) * kSsimRun;
    const int at = r * kSsimSP + kSsimOff + c0;
    float2 ab[kSsimRun];
    float cc[kSsimRun];
#pragma unroll
    for (int u = 0; u < kSsimRun; ++u) {
      ab[u] = splat2(0.f);
      cc[u] = 0.f;
    }
#pragma unroll
    for (int k = 0; k < kSsimRun + 2 * kSsimR; ++k) {
      const float2 v = make_float2(s_m[0][at + k], s_m[1][at + k]);
      const float vc = s_m[2][at + k];
#pragma unroll
      for (int u = 0; u < kSsimRun; ++u) {
        const int tap = k - u;
        if (tap >= 0 && tap < kSsimTaps) {
          ab[u] = fma2(w[tap], v, ab[u]);
          cc[u] = fmaf(w[tap].x, vc, cc[u]);
        }
      }
    }
#pragma unroll
    for (int u = 0; u < kSsimRun; ++u) {
      s_hab[r * kSsimHP + c0 + u] = ab[u];
      s_hc[r * kSsimHP + c0 + u] = cc[u];
    }
  }
  __syncthreads();
  float2 ab[kSsimRun];
  float cc[kSsimRun];
#pragma unroll
  for (int u = 0; u < kSsimRun; ++u) {
    ab[u] = splat2(0.f);
    cc[u] = 0.f;
  }
#pragma unroll
  for (int k = 0; k < kSsimRun + 2 * kSsimR; ++k) {
    const float2 v = s_hab[(r0 + k) * kSsimHP + c];
    const float vc = s_hc[(r0 + k) * kSsimHP + c];
#pragma unroll
    for (int u = 0; u < kSsimRun; ++u) {
      const int tap = k - u;
      if (tap >= 0 && tap < kSsimTaps) {
        ab[u] = fma2(w[tap], v, ab[u]);
        cc[u] = fmaf(w[tap].x, vc, cc[u]);
      }
    }
  }
#pragma unroll
  for (int u = 0; u < kSsimRun; ++u) {
    const int py = y0 + r0 + u;
    if (py >= d.H || px >= d.W) continue;
    const float xc = PHOTO ? clamp01(x[u]) : x[u];
    float v = g * (ab[u].x + 2.f * xc * ab[u].y + y[u] * cc[u]);
    if (PHOTO) {
      const float diff = xc - y[u];
      const float l1 = g * w_l1_over_count;
      v = w_ssim * v + (diff > 0.f ? l1 : (diff < 0.f ? -l1 : 0.f));
      if (!(x[u] >= 0.f && x[u] <= 1.f)) v = 0.f;
    }
    dL_dimg1[ch * plane + (size_t)py * d.W + px] = staged ? v : __int_as_float(0x7fc00000);
  }
}

namespace {

// The window (utils/loss_utils.py:23-29: exp(-(x - 5)^2 / (2 sigma^2)), sigma 1.5,
// normalised to sum 1) goes to constant memory once per device.
bool upload_window(cudaStream_t st) {
  constexpr int kMaxDevices = 64;
  static bool done[kMaxDevices] = {};
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return false;
  if (done[dev]) return true;
  double g[kSsimTaps], sum = 0.0;
  for (int k = 0; k < kSsimTaps; ++k) {
    const double t = (double)(k - kSsimR);
    g[k] = std::exp(-t * t / (2.0 * 1.5 * 1.5));
    sum += g[k];
  }
  float w[kSsimTaps];
  for (int k = 0; k < kSsimTaps; ++k) w[k] = (float)(g[k] / sum);
  if (cudaMemcpyToSymbolAsync(c_ssim_w, w, sizeof(w), 0, cudaMemcpyHostToDevice, st) != cudaSuccess) return false;
  if (cudaStreamSynchronize(st) != cudaSuccess) return false;
  done[dev] = true;
  return true;
}

SsimDims dims(int32_t C, int32_t H, int32_t W) {
  SsimDims d;
  d.C = C;
  d.H = H;
  d.W = W;
  d.tiles_x = (W + kSsimT - 1) / kSsimT;
  d.tiles_y = (H + kSsimT - 1) / kSsimT;
  return d;
}

// Rank-3 tensor map of a [D][H][W] float32 array with the staging box (48 x 42 x 1);
// false when the array cannot be described (width not a multiple of 4 floats, base not
// 16-byte aligned) or the encoder is unavailable — the kernels then stage by plain loads.
bool encode_planes(CUtensorMap* m, const float* base, int W, int H, int D) {
  static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
  static bool looked = false;
  if (!looked) {
    looked = true;
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
  }
  if (!encode || (W % 4) != 0 || (reinterpret_cast<uintptr_t>(base) & 15) != 0) return false;
  const cuuint64_t dim[3] = {(cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)D};
  const cuuint64_t stride[2] = {(cuuint64_t)W * sizeof(float), (cuuint64_t)W * H * sizeof(float)};
  const cuuint32_t box[3] = {(cuuint32_t)kSsimSP, (cuuint32_t)kSsimS, 1};
  const cuuint32_t estride[3] = {1, 1, 1};
  return encode(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(base), dim, stride, box, estride,
                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

bool dims_ok(int32_t C, int32_t H, int32_t W) {
  return C > 0 && H > 0 && W > 0 && C <= 65535 && (int64_t)C * H * W <= ((int64_t)1 << 31);
}

}  // namespace

}  // namespace cfgs

using namespace cfgs;

extern "C" size_t cfgs_ssim_scratch_bytes(int32_t channels, int32_t height, int32_t width) {
  if (!dims_ok(channels, height, width)) return 0;
  const SsimDims d = dims(channels, height, width);
  const size_t maps = sizeof(float) * 3 * (size_t)channels * height * width;
  const size_t parts = sizeof(double2) * (size_t)channels * d.tiles_x * d.tiles_y;
  // the partial sums and what follows them begin at the next 16-byte boundary (aligned16)
  return align256(maps) + align256(parts) + align256(sizeof(double2) * (kSsimFoldBlocks + 1) + kAlignSlack);
}

namespace {

// The forward of the mean SSIM (photo: of the photometric loss with weight lambda).
int ssim_forward(int32_t channels, int32_t height, int32_t width, const float* img1, const float* img2, bool photo,
                 double lambda, void* scratch, float* out, void* stream) {
  if (!dims_ok(channels, height, width) || !img1 || !img2 || !scratch || !out) return CFGS_ERR_INVALID_ARGUMENT;
  cudaStream_t st = (cudaStream_t)stream;
  if (!upload_window(st)) return CFGS_ERR_LAUNCH;
  const SsimDims d = dims(channels, height, width);
  const size_t count = (size_t)channels * height * width;
  float* maps = static_cast<float*>(scratch);
  double2* parts = aligned16<double2>(static_cast<char*>(scratch) + align256(sizeof(float) * 3 * count));
  const int tiles = d.tiles_x * d.tiles_y, pairs = tiles * channels;
  double2* sums = reinterpret_cast<double2*>(reinterpret_cast<char*>(parts) + align256(sizeof(double2) * (size_t)pairs));
  unsigned int* counter = reinterpret_cast<unsigned int*>(sums + kSsimFoldBlocks);
  const float inv = (float)(1.0 / (double)count);
  CUtensorMap t1{}, t2{};
  const bool tma = encode_planes(&t1, img1, width, height, channels) && encode_planes(&t2, img2, width, height, channels);
  auto* kernel = photo ? (tma ? k_ssim_fwd<true, true> : k_ssim_fwd<false, true>)
                       : (tma ? k_ssim_fwd<true, false> : k_ssim_fwd<false, false>);
  kernel<<<dim3(tiles, channels), kSsimThreads, 0, st>>>(d, img1, img2, maps, parts, counter, inv, t1, t2);
  const int fold_blocks = min(kSsimFoldBlocks, div_up(pairs, kSsimThreads));
  k_ssim_fold<<<fold_blocks, kSsimThreads, 0, st>>>(parts, pairs, sums, counter, 1.0 / (double)count,
                                                    photo ? 1.0 - lambda : 0.0, photo ? -lambda : 1.0,
                                                    photo ? lambda : 0.0, out);
  CFGS_CHECK_LAUNCH(0, st);
  return CFGS_OK;
}

int ssim_backward(int32_t channels, int32_t height, int32_t width, const float* img1, const float* img2, bool photo,
                  double lambda, const void* scratch, const float* dL_dout, float* dL_dimg1, void* stream) {
  if (!dims_ok(channels, height, width) || !img1 || !img2 || !scratch || !dL_dout || !dL_dimg1)
    return CFGS_ERR_INVALID_ARGUMENT;
  cudaStream_t st = (cudaStream_t)stream;
  if (!upload_window(st)) return CFGS_ERR_LAUNCH;
  const SsimDims d = dims(channels, height, width);
  const double count = (double)channels * height * width;
  const float* maps = static_cast<const float*>(scratch);
  CUtensorMap tm{};
  const dim3 grid(d.tiles_x * d.tiles_y, channels);
  const bool tma = encode_planes(&tm, maps, width, height, 3 * channels);
  auto* kernel = photo ? (tma ? k_ssim_bwd<true, true> : k_ssim_bwd<false, true>)
                       : (tma ? k_ssim_bwd<true, false> : k_ssim_bwd<false, false>);
  kernel<<<grid, kSsimThreads, 0, st>>>(d, img1, img2, maps, dL_dout, (float)-lambda, (float)((1.0 - lambda) / count),
                                        dL_dimg1, tm);
  CFGS_CHECK_LAUNCH(0, st);
  return CFGS_OK;
}

}  // namespace

extern "C" int cfgs_ssim_forward(int32_t channels, int32_t height, int32_t width, const float* img1,
                                 const float* img2, void* scratch, float* ssim_mean, void* stream) {
  return ssim_forward(channels, height, width, img1, img2, false, 0.0, scratch, ssim_mean, stream);
}

extern "C" int cfgs_ssim_backward(int32_t channels, int32_t height, int32_t width, const float* img1,
                                  const float* img2, const void* scratch, const float* dL_dmean, float* dL_dimg1,
                                  void* stream) {
  return ssim_backward(channels, height, width, img1, img2, false, 0.0, scratch, dL_dmean, dL_dimg1, stream);
}

extern "C" int cfgs_photometric_forward(int32_t channels, int32_t height, int32_t width, const float* img,
                                        const float* target, double lambda_dssim, void* scratch, float* loss,
                                        void* stream) {
  return ssim_forward(channels, height, width, img, target, true, lambda_dssim, scratch, loss, stream);
}

extern "C" int cfgs_photometric_backward(int32_t channels, int32_t height, int32_t width, const float* img,
                                         const float* target, double lambda_dssim, const void* scratch,
                                         const float* dL_dloss, float* dL_dimg, void* stream) {
  return ssim_backward(channels, height, width, img, target, true, lambda_dssim, scratch, dL_dloss, dL_dimg, stream);
}
