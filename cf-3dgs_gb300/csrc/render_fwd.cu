// Forward phase 3: front-to-back alpha compositing of every 16x16 tile over its
// depth-sorted instance list.
//
// The kernel is a template over the scene accessor (one scene for the drop-in path, a
// descriptor table for batched solves); the arithmetic is the same for both.
// Compiled with -fmad=false; the fmaf() calls are the only fused operations, and the
// CPU oracle performs the same sequence.
#include <type_traits>

#include "cfgs_internal.cuh"
#include "kernels.cuh"

namespace cfgs {

// Launch schedules: kRenderBatch instances staged per round and 4 or 8 warps per tile. Every
// schedule gives bit-identical outputs: each pixel sees the same instances in the same
// order with the same arithmetic.
constexpr int kRenderBatch = 128;

// A staged instance as the compositing reads it: every factor twice, so that the packed
// operations take their operands as loaded, without a move per factor.
struct StagedInstance {
  float4 xy;   // (x, x, y, y)
  float4 ab;   // (ca, ca, cb, cb)
  float4 co;   // (cc, cc, opacity, opacity)
};

// Front-to-back state of a lane's two pixels (.x: row r, .y: row r + 4) and one
// compositing step of both: the published loop body per pixel, with the exponential
// skipped below the alpha threshold (exact, see alpha_threshold). The arithmetic runs on
// packed pairs (bit-identical to the scalar operations); each pixel's decisions are its
// own, and a pixel that does not take the step keeps its state: its weight is 0, which adds
// nothing times a finite colour. ODD (a view with a colour or depth that is not finite)
// selects instead.
struct PairFwd {
  float2 T, C0, C1, C2, D;
  uint32_t last0, last1;
  bool done0, done1;
};

template <bool DEPTH, bool ODD>
__device__ __forceinline__ void composite_pair(PairFwd& p, float2 px, float2 py, const StagedInstance& s, float thr,
                                               const float4* s_rgbd, int j, uint32_t pos1) {
  const float2 dx = sub2(make_float2(s.xy.x, s.xy.y), px), dy = sub2(make_float2(s.xy.z, s.xy.w), py);
  const float2 power = gauss_power2(make_float2(s.ab.x, s.ab.y), make_float2(s.ab.z, s.ab.w),
                                    make_float2(s.co.x, s.co.y), dx, dy);
  bool a0 = !p.done0 && !(power.x > 0.0f || power.x < thr);
  bool a1 = !p.done1 && !(power.y > 0.0f || power.y < thr);
  if (!(a0 || a1)) return;
  float2 alpha = mul2(make_float2(s.co.z, s.co.w), exp_ref_inrange2(power));
  alpha.x = fminf(CFGS_ALPHA_MAX, alpha.x);
  alpha.y = fminf(CFGS_ALPHA_MAX, alpha.y);
  a0 = a0 && !(alpha.x < CFGS_ALPHA_MIN);
  a1 = a1 && !(alpha.y < CFGS_ALPHA_MIN);
  if (!(a0 || a1)) return;
  const float2 test_T = mul2(p.T, sub2(splat2(1.0f), alpha));
  const bool end0 = a0 && test_T.x < CFGS_T_MIN, end1 = a1 && test_T.y < CFGS_T_MIN;
  p.done0 = p.done0 || end0;
  p.done1 = p.done1 || end1;
  const float4 c = s_rgbd[j];
  const float2 w = mul2(alpha, p.T);
  const bool u0 = a0 && !end0, u1 = a1 && !end1;
  const float2 wm = ODD ? w : make_float2(u0 ? w.x : 0.0f, u1 ? w.y : 0.0f);
  auto add = [&](float2& C, float v) {
    const float2 sum = fma2(splat2(v), wm, C);
    C = ODD ? make_float2(u0 ? sum.x : C.x, u1 ? sum.y : C.y) : sum;
  };
  add(p.C0, c.x);
  add(p.C1, c.y);
  add(p.C2, c.z);
  if (DEPTH) add(p.D, c.w);
  p.T = make_float2(u0 ? test_T.x : p.T.x, u1 ? test_T.y : p.T.y);
  p.last0 = u0 ? pos1 : p.last0;
  p.last1 = u1 ? pos1 : p.last1;
}

// The same step of one pixel (the 8-warp form's lanes have one each).
struct OneFwd {
  float T, C0, C1, C2, D;
  uint32_t last;
  bool done;
};

template <bool DEPTH, bool ODD>
__device__ __forceinline__ void composite_one(OneFwd& p, float px, float py, const StagedInstance& s, float thr,
                                              const float4* s_rgbd, int j, uint32_t pos1) {
  const float power = gauss_power(s.ab.x, s.ab.z, s.co.x, s.xy.x - px, s.xy.z - py);
  bool a = !p.done && !(power > 0.0f || power < thr);
  if (!a) return;
  const float alpha = fminf(CFGS_ALPHA_MAX, s.co.z * exp_ref_inrange(power));
  if (alpha < CFGS_ALPHA_MIN) return;
  const float test_T = p.T * (1.0f - alpha);
  if (test_T < CFGS_T_MIN) {
    p.done = true;
    return;
  }
  const float4 c = s_rgbd[j];
  const float w = alpha * p.T;
  p.C0 = fmaf(c.x, w, p.C0);
  p.C1 = fmaf(c.y, w, p.C1);
  p.C2 = fmaf(c.z, w, p.C2);
  if (DEPTH) p.D = fmaf(c.w, w, p.D);
  p.T = test_T;
  p.last = pos1;
}

// Warp boxes and pixels of a lane: with 4 warps, warp w covers the 8x8 pixel box
// (8 (w & 1), 8 (w >> 1)) and each lane two pixels of a column, rows r and r + 4, so that
// the stores fill whole 32-byte sectors (with columns c and c + 4 they do not: 1000 Gaussians at
// 1920x1080 31 us against 20, 300,000 at 3840x2160 378 against 365); with 8 warps, warp w
// covers the 8x4 box (8 (w & 1), 4 (w >> 1)) and each lane one pixel.
template <bool DEPTH, bool ODD>
struct PairPixels {
  PairFwd p;
  float2 px, py;
  __device__ __forceinline__ PairPixels(int x, int y, bool in0, bool in1)
      : p{splat2(1.0f), splat2(0.0f), splat2(0.0f), splat2(0.0f), splat2(0.0f), 0u, 0u, !in0, !in1},
        px(splat2((float)x)),
        py(make_float2((float)y, (float)(y + 4))) {}
  __device__ __forceinline__ bool done() const { return p.done0 && p.done1; }
  __device__ __forceinline__ void step(const StagedInstance& s, float thr, const float4* rgbd, int j, uint32_t pos1) {
    composite_pair<DEPTH, ODD>(p, px, py, s, thr, rgbd, j, pos1);
  }
  __device__ __forceinline__ OneFwd pixel(int q) const {
    return q ? OneFwd{p.T.y, p.C0.y, p.C1.y, p.C2.y, p.D.y, p.last1, p.done1}
             : OneFwd{p.T.x, p.C0.x, p.C1.x, p.C2.x, p.D.x, p.last0, p.done0};
  }
};
template <bool DEPTH, bool ODD>
struct OnePixel {
  OneFwd p;
  float px, py;
  __device__ __forceinline__ OnePixel(int x, int y, bool in0, bool)
      : p{1.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0u, !in0}, px((float)x), py((float)y) {}
  __device__ __forceinline__ bool done() const { return p.done; }
  __device__ __forceinline__ void step(const StagedInstance& s, float thr, const float4* rgbd, int j, uint32_t pos1) {
    composite_one<DEPTH, ODD>(p, px, py, s, thr, rgbd, j, pos1);
  }
  __device__ __forceinline__ OneFwd pixel(int) const { return p; }
};

template <int BATCH>
struct FwdShared {
  StagedInstance inst[BATCH];
  float4 rgbd[BATCH];
  float thr[BATCH];
};

template <class Scenes, int BATCH, int WARPS, bool ODD>
__device__ __forceinline__ void composite_tile(const RenderArgs<Scenes>& a, FwdShared<BATCH>& sh) {
  constexpr bool kDepth = !Scenes::kBatched;  // batches ask for no depth
  constexpr int kThreads = 32 * WARPS;
  constexpr int kBoxRows = WARPS == 4 ? 8 : 4;
  constexpr int kPixels = WARPS == 4 ? 2 : 1;
  using Pixels = std::conditional_t<WARPS == 4, PairPixels<kDepth, ODD>, OnePixel<kDepth, ODD>>;
  const int tile = blockIdx.x;
  const SceneDesc& sd = a.scenes.for_tile(tile);
  const int lt = tile - sd.tile_base;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int bx0 = (lt % sd.grid_x) * kTileX + (warp & 1) * 8;
  const int by0 = (lt / sd.grid_x) * kTileY + (warp >> 1) * kBoxRows;
  const int px = bx0 + (lane & 7), py0 = by0 + (lane >> 3);
  const float bxf0 = (float)bx0, bxf1 = (float)(bx0 + 7), byf0 = (float)by0, byf1 = (float)(by0 + kBoxRows - 1);
  const uint32_t lo = a.tile_range[tile];
  const int n = (int)(a.tile_range[tile + 1] - lo);
  Pixels pixels(px, py0, px < sd.W && py0 < sd.H, px < sd.W && py0 + 4 < sd.H);
  for (int base = 0; base < n; base += BATCH) {
    if (__syncthreads_count(pixels.done()) == kThreads) break;
#pragma unroll
    for (int j = threadIdx.x; j < BATCH; j += kThreads) {
      const int i = base + j;
      if (i < n) {
        uint32_t g = a.sorted_gid[lo + i];
        float2 m = a.xy[g];
        float4 co = a.conic_op[g];
        const float ca = -0.5f * co.x, cb = -co.y, cc = -0.5f * co.z;
        sh.inst[j].xy = make_float4(m.x, m.x, m.y, m.y);
        sh.inst[j].ab = make_float4(ca, ca, cb, cb);
        sh.inst[j].co = make_float4(cc, cc, co.w, co.w);
        sh.thr[j] = alpha_threshold(co.w);
        sh.rgbd[j] = a.rgbd[g];
      }
    }
    __syncthreads();
    const int cnt = min(BATCH, n - base);
    uint32_t keep[BATCH / 32];
#pragma unroll
    for (int r = 0; r < BATCH / 32; ++r) {
      const int j = r * 32 + lane;
      bool k = false;
      if (j < cnt) {
        const float4 xy = sh.inst[j].xy, ab = sh.inst[j].ab;
        k = box_may_contribute(make_float2(xy.x, xy.z), ab.x, ab.z, sh.inst[j].co.x, sh.thr[j], bxf0, bxf1, byf0, byf1);
      }
      keep[r] = __ballot_sync(0xffffffffu, k);
    }
#pragma unroll
    for (int r = 0; r < BATCH / 32; ++r) {
      if (__all_sync(0xffffffffu, pixels.done())) break;
      uint32_t mk = keep[r];
      while (mk) {
        const int j = r * 32 + __ffs(mk) - 1;
        mk &= mk - 1;
        pixels.step(sh.inst[j], sh.thr[j], sh.rgbd, j, (uint32_t)(base + j + 1));
      }
    }
  }
  const size_t HW = (size_t)sd.W * sd.H;
  float* col = a.out_color + 3 * (size_t)sd.pix_base;
#pragma unroll
  for (int q = 0; q < kPixels; ++q) {
    const int py = py0 + 4 * q;
    if (px >= sd.W || py >= sd.H) continue;
    const OneFwd p = pixels.pixel(q);
    const size_t pix = (size_t)py * sd.W + px;
    const size_t gp = (size_t)sd.pix_base + pix;
    a.final_T[gp] = p.T;
    a.n_contrib[gp] = p.last;
    col[pix] = fmaf(p.T, __ldg(sd.bg + 0), p.C0);
    col[HW + pix] = fmaf(p.T, __ldg(sd.bg + 1), p.C1);
    col[2 * HW + pix] = fmaf(p.T, __ldg(sd.bg + 2), p.C2);
    if (a.out_depth) a.out_depth[gp] = p.D;
    if (a.out_alpha) a.out_alpha[gp] = 1.0f - p.T;
  }
}

// One block of 32 WARPS threads per 16x16 tile. Batches of BATCH instances are gathered
// into shared memory (per-Gaussian data stays L2-resident).
// Two exact shortcuts skip work whose outcome is known: each warp keeps only the
// instances whose alpha >= 1/255 ellipse can reach its box (box_may_contribute, one test
// per instance and warp), and a pixel skips the exponential when the exponent lies
// below the instance's alpha_threshold. Neither changes a decision of the published
// algorithm, so every output — contributor counts included, which count positions in
// the tile's list — is what the plain per-pixel loop gives. Compositing runs front to
// back; a warp stops when its pixels are saturated and the block when all are.
// Bound by instruction issue (75% busy at 1M Gaussians 1080p), and with few tiles by a
// warp's own chain. Every factor is staged twice and masked weights are added instead of
// results moved under predicates: 489 -> 457 million warp instructions at 1080p (517 us both
// ways, fewer warps ready), 127 -> 121 us for one 640x360 pose solve, 80 -> 74 us for 256
// tiles; the default shapes (resolve_schedule) then take the latter two to 108 and 58 us.
template <class Scenes, int BATCH, int WARPS>
__global__ void __launch_bounds__(32 * WARPS, WARPS == 4 ? 9 : 6) k_render_fwd(RenderArgs<Scenes> a) {
  static_assert(BATCH % 32 == 0 && (WARPS == 4 || WARPS == 8), "whole ballot words; 8x8 or 8x4 warp boxes");
  __shared__ FwdShared<BATCH> sh;
  if ((int64_t)a.counts->num_rendered > a.cap) return;
  if (WARPS == 4 && *nonfinite_word(a.counts)) composite_tile<Scenes, BATCH, WARPS, true>(a, sh);
  else composite_tile<Scenes, BATCH, WARPS, false>(a, sh);
}

template <class Scenes>
void launch_render_fwd(const RenderArgs<Scenes>& a, int tiles, cudaStream_t st) {
  const CfgsRenderSchedule& rs = a.sched;
  if (rs.fwd_warps == 8) {
    if (rs.fwd_batch == 256) k_render_fwd<Scenes, 256, 8><<<tiles, 256, 0, st>>>(a);
    else k_render_fwd<Scenes, 128, 8><<<tiles, 256, 0, st>>>(a);
  } else {
    if (rs.fwd_batch == 64) k_render_fwd<Scenes, 64, 4><<<tiles, 128, 0, st>>>(a);
    else if (rs.fwd_batch == 256) k_render_fwd<Scenes, 256, 4><<<tiles, 128, 0, st>>>(a);
    else k_render_fwd<Scenes, kRenderBatch, 4><<<tiles, 128, 0, st>>>(a);
  }
}
template void launch_render_fwd<SingleScene>(const RenderArgs<SingleScene>&, int, cudaStream_t);
template void launch_render_fwd<SceneTable>(const RenderArgs<SceneTable>&, int, cudaStream_t);

// The default shape. Eight warps of one pixel per lane issue more instructions per pixel
// than four of two, but their 8x4 boxes keep fewer instances, and a warp's chain is
// shorter. They win with at most two tiles per SM, where a tile's longest warp sets the
// time (256 tiles: 58 against 74 us; 304: 63 against 78), and go on winning for some way above
// (1024 tiles with 5 instances per Gaussian 78 against 88; with 11 from 480 tiles on the
// four). And they win with small Gaussians, which reach fewer than four tiles each (one
// 640x360 pose solve, 2.1 tiles each: 108 against 121 us; 16 solves: 1455 against 1535 us; 1024
// tiles, 3.2 each: 67 against 78, but at 1600 tiles 98 against 86). With larger ones four win
// (1M at 1920x1080, 12.4 tiles each: 517 against 649 us; 250,007 at 977x545, 4.5 each: 204 against
// 216 us). `gaussians` are those that touch a tile: 3M of which 95 % are culled have 0.6
// instances each and 12 each of the others (207 us with four warps, 250 with eight). Calls that
// know only how many were given pass 0 and take four.
constexpr int64_t kFewTiles = 2 * 152;
constexpr int64_t kSmallTouch = 4;

bool resolve_schedule(const CfgsRenderSchedule& in, int64_t tiles, int64_t gaussians, int64_t capacity,
                      CfgsRenderSchedule* out) {
  if (in.bin_launch != 0 && in.bin_launch != 1) return false;
  if (in.fwd_batch == 0 && in.fwd_warps == 0 && in.bwd_batch == 0) {
    if (tiles > 0 && (tiles <= kFewTiles || capacity < kSmallTouch * gaussians)) {
      *out = CfgsRenderSchedule{256, 8, 64, in.bin_launch};
      return true;
    }
    *out = CfgsRenderSchedule{kRenderBatch, 4, 64, in.bin_launch};
    return true;
  }
  const bool fwd_ok = in.fwd_warps == 4 ? (in.fwd_batch == 64 || in.fwd_batch == 128 || in.fwd_batch == 256)
                                        : (in.fwd_warps == 8 && (in.fwd_batch == 128 || in.fwd_batch == 256));
  const bool bwd_ok = in.bwd_batch == 32 || in.bwd_batch == 64 || in.bwd_batch == 128;
  if (!fwd_ok || !bwd_ok) return false;
  *out = CfgsRenderSchedule{in.fwd_batch, in.fwd_warps, in.bwd_batch, in.bin_launch};
  return true;
}

}  // namespace cfgs

using namespace cfgs;

extern "C" int cfgs_render_schedule_for(const CfgsRenderSchedule* s, int64_t num_tiles, int64_t num_gaussians,
                                        int64_t capacity, CfgsRenderSchedule* resolved) {
  if (!s || !resolved || num_tiles < 0 || num_gaussians < 0 || capacity < 0) return CFGS_ERR_INVALID_ARGUMENT;
  return resolve_schedule(*s, num_tiles, num_gaussians, capacity, resolved) ? CFGS_OK : CFGS_ERR_INVALID_ARGUMENT;
}

extern "C" int cfgs_render_schedule_check(const CfgsRenderSchedule* s, CfgsRenderSchedule* resolved) {
  if (!s) return CFGS_ERR_INVALID_ARGUMENT;
  CfgsRenderSchedule r;
  if (!resolve_schedule(*s, 0, 0, 0, &r)) return CFGS_ERR_INVALID_ARGUMENT;
  if (resolved) *resolved = r;
  return CFGS_OK;
}

extern "C" int cfgs_composite_forward(const CfgsSettings* s, int32_t num_gaussians, const void* geom, const void* image,
                                      const void* binning, int64_t capacity, float* out_color, float* out_depth,
                                      float* out_alpha, void* stream) {
  if (!s || !geom || !image || !binning || !out_color || capacity < 0 || !s->bg || num_gaussians < 0)
    return CFGS_ERR_INVALID_ARGUMENT;
  if (s->image_width <= 0 || s->image_height <= 0) return CFGS_ERR_INVALID_ARGUMENT;
  if (capacity > 0x7fffffffll) return CFGS_ERR_TOO_LARGE;
  cudaStream_t st = (cudaStream_t)stream;
  ImageLayout IL(s->image_width, s->image_height);
  ImageView iv(const_cast<void*>(image), s->image_width, s->image_height);
  GeomView gv(const_cast<void*>(geom), num_gaussians);
  BinningView bv(const_cast<void*>(binning), capacity);
  RenderArgs<SingleScene> ra;
  ra.scenes.d = single_scene_desc(s, num_gaussians, 0);
  ra.tile_range = iv.tile_range;
  ra.sorted_gid = bv.sorted_gid;
  ra.xy = gv.xy;
  ra.conic_op = gv.conic_op;
  ra.rgbd = gv.rgbd;
  ra.final_T = iv.final_T;
  ra.n_contrib = iv.n_contrib;
  ra.out_color = out_color;
  ra.out_depth = out_depth;
  ra.out_alpha = out_alpha;
  ra.cap = capacity;
  ra.counts = iv.counts;
  if (!resolve_schedule(s->schedule, IL.num_tiles, 0, 0, &ra.sched)) return CFGS_ERR_INVALID_ARGUMENT;
  launch_render_fwd(ra, IL.num_tiles, st);
  CFGS_CHECK_LAUNCH(s->debug, st);
  return CFGS_OK;
}

extern "C" int cfgs_render_forward(const CfgsSettings* s, const CfgsGaussians* g, void* geom, void* image,
                                   void* binning, int64_t capacity, float* out_color, float* out_depth,
                                   float* out_alpha, void* stream) {
  int st = cfgs_bin_forward(s, g, geom, image, binning, capacity, stream);
  if (st != CFGS_OK) return st;
  return cfgs_composite_forward(s, g->num_gaussians, geom, image, binning, capacity, out_color, out_depth, out_alpha,
                                stream);
}
