// Backward, part 1: the per-tile render backward with in-block gradient reduction,
// and the backward entry points (the per-Gaussian part is in preprocess_bwd.cu).
//
// Upstream accumulates every (pixel, Gaussian) gradient with a global atomicAdd.
// Here each tile reduces the gradients of its 256 pixels per instance inside the
// block (eight instances at a time per warp, then a fixed-order sum over the 4 warps) and
// writes one 48-byte record per (Gaussian, tile) instance, at the instance's
// pre-sort index. A Gaussian's instances are contiguous in pre-sort order, so the
// preprocess backward sums its records in a fixed order: no atomics, bit-identical
// results run to run.
#include <mutex>
#include <type_traits>

#include "cfgs_internal.cuh"
#include "kernels.cuh"

namespace cfgs {

constexpr int kBwdThreads = 128;  // 2 pixels per thread, 4 warps per 16x16 tile
constexpr int kWarps = kBwdThreads / 32;
constexpr int kSlots = 8;  // instances a warp reduces at a time, four lanes each

// d/dc of mean |clamp(c, 0, 1) - t| as autograd forms it.
__device__ __forceinline__ float l1_grad(float c, float t, float inv_numel) {
  float d = fminf(fmaxf(c, 0.0f), 1.0f) - t;
  float sgn = d > 0.0f ? 1.0f : (d < 0.0f ? -1.0f : 0.0f);
  return (c >= 0.0f && c <= 1.0f) ? inv_numel * sgn : 0.0f;
}

// Forward results and upstream gradients of one pixel.
struct PixelBwd {
  float T_final, dC0, dC1, dC2, dD, dA_bg;  // dA_bg = dL/dalpha - bg . dL/dcolor
  uint32_t last;
};

// Loads pixel pix's forward state and upstream gradient (zeros outside the image).
template <class Scenes>
__device__ __forceinline__ void load_pixel(PixelBwd& p, const RenderBwdArgs<Scenes>& a, const SceneDesc& sd,
                                           bool inside, size_t pix) {
  const size_t HW = (size_t)sd.W * sd.H;
  const size_t gp = (size_t)sd.pix_base + pix;
  p.T_final = 1.0f;
  p.dC0 = p.dC1 = p.dC2 = p.dD = 0.f;
  float dA = 0.f;
  p.last = 0;
  if (inside) {
    p.T_final = a.final_T[gp];
    p.last = a.n_contrib[gp];
    const size_t cb = 3 * (size_t)sd.pix_base + pix;
    if (a.target) {
      p.dC0 = l1_grad(a.color[cb], a.target[cb], sd.inv_numel);
      p.dC1 = l1_grad(a.color[cb + HW], a.target[cb + HW], sd.inv_numel);
      p.dC2 = l1_grad(a.color[cb + 2 * HW], a.target[cb + 2 * HW], sd.inv_numel);
    } else {
      p.dC0 = a.dL_dcolor[cb];
      p.dC1 = a.dL_dcolor[cb + HW];
      p.dC2 = a.dL_dcolor[cb + 2 * HW];
      if (a.dL_ddepth) p.dD = a.dL_ddepth[gp];
      if (a.dL_dalpha) dA = a.dL_dalpha[gp];
    }
  }
  p.dA_bg = dA - (__ldg(sd.bg + 0) * p.dC0 + __ldg(sd.bg + 1) * p.dC1 + __ldg(sd.bg + 2) * p.dC2);
}

__device__ __forceinline__ bool all_finite(const PixelBwd& p) {
  return isfinite(p.dC0) && isfinite(p.dC1) && isfinite(p.dC2) && isfinite(p.dD) && isfinite(p.dA_bg);
}

// Back-to-front state of a lane's two pixels (.x: column c, .y: column c + 4): upstream
// gradients, the transmittance being unwound, and the colour/depth accumulated behind the
// current instance (updated right after each contributing instance, which gives the
// value upstream forms from the previous instance's alpha and colour).
struct PairBwd {
  float2 T_final, dC0, dC1, dC2, dD, dA_bg;
  float2 T, acc0, acc1, acc2, accd;
  uint32_t last0, last1;
};

__device__ __forceinline__ PairBwd make_pair(const PixelBwd& p, const PixelBwd& q) {
  PairBwd P;
  P.T_final = make_float2(p.T_final, q.T_final);
  P.dC0 = make_float2(p.dC0, q.dC0);
  P.dC1 = make_float2(p.dC1, q.dC1);
  P.dC2 = make_float2(p.dC2, q.dC2);
  P.dD = make_float2(p.dD, q.dD);
  P.dA_bg = make_float2(p.dA_bg, q.dA_bg);
  P.T = P.T_final;
  P.acc0 = P.acc1 = P.acc2 = P.accd = make_float2(0.f, 0.f);
  P.last0 = p.last;
  P.last1 = q.last;
  return P;
}

// A staged instance as the unwinding reads it: every factor twice, so that the packed
// operations take their operands as loaded, without a move per factor.
struct StagedInstance {
  float4 xy;   // (x, x, y, y)
  float4 ab;   // (ca, ca, cb, cb)
  float4 co;   // (cc, cc, opacity, opacity)
  float4 rg;   // (r, r, g, g)
  float4 bd;   // (b, b, depth, depth)
};
__device__ __forceinline__ float2 lo2(const float4& v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(const float4& v) { return make_float2(v.z, v.w); }

// Unwinds one instance at list position c for both pixels: g = G dL/dalpha (G the
// Gaussian's value at the pixel) and w = alpha T, zero where the instance did not
// contribute. A pixel the instance did not reach in the forward pass keeps its state: its
// alpha and G count as 0. Returns whether the instance contributed to either pixel. ODD (a
// tile whose image gradients, or a view whose colours or depths, are not all finite) selects
// where a zero would multiply such a value.
template <bool DEPTH, bool ODD>
__device__ __forceinline__ bool unwind_pair(PairBwd& P, int c, float2 px, float2 py, const StagedInstance& s, float thr,
                                            float2& g, float2& w) {
  const bool in0 = c < (int)P.last0, in1 = c < (int)P.last1;
  const float2 dx = sub2(lo2(s.xy), px), dy = sub2(hi2(s.xy), py);
  const float2 power = gauss_power2(lo2(s.ab), hi2(s.ab), lo2(s.co), dx, dy);
  bool a0 = in0 && !(power.x > 0.0f || power.x < thr);
  bool a1 = in1 && !(power.y > 0.0f || power.y < thr);
  g = w = make_float2(0.f, 0.f);
  if (!(a0 || a1)) return false;
  const float2 G = exp_ref_inrange2(power);
  float2 alpha = mul2(hi2(s.co), G);
  alpha.x = fminf(CFGS_ALPHA_MAX, alpha.x);
  alpha.y = fminf(CFGS_ALPHA_MAX, alpha.y);
  a0 = a0 && !(alpha.x < CFGS_ALPHA_MIN);
  a1 = a1 && !(alpha.y < CFGS_ALPHA_MIN);
  if (!(a0 || a1)) return false;
  const float2 am = make_float2(a0 ? alpha.x : 0.0f, a1 ? alpha.y : 0.0f);
  const float2 om = sub2(splat2(1.0f), am);
  float2 inv;  // 1 where the instance did not contribute (the approximation is exact at 1)
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(inv.x) : "f"(om.x));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(inv.y) : "f"(om.y));
  P.T = mul2(P.T, inv);
  w = mul2(am, P.T);
  const float2 e0 = sub2(lo2(s.rg), P.acc0), e1 = sub2(hi2(s.rg), P.acc1), e2 = sub2(lo2(s.bd), P.acc2);
  float2 dLda = mul2(e0, P.dC0);
  dLda = fma2(e1, P.dC1, dLda);
  dLda = fma2(e2, P.dC2, dLda);
  auto behind = [&](float2& acc, const float2& e) {
    const float2 sum = fma2(am, e, acc);
    acc = ODD ? make_float2(a0 ? sum.x : acc.x, a1 ? sum.y : acc.y) : sum;
  };
  behind(P.acc0, e0);
  behind(P.acc1, e1);
  behind(P.acc2, e2);
  if (DEPTH) {
    const float2 ed = sub2(hi2(s.bd), P.accd);
    dLda = fma2(ed, P.dD, dLda);
    behind(P.accd, ed);
  }
  dLda = mul2(dLda, P.T);
  dLda = fma2(mul2(P.T_final, inv), P.dA_bg, dLda);
  // d/d opacity
  if (ODD) g = make_float2(a0 ? __fmul_rn(G.x, dLda.x) : 0.0f, a1 ? __fmul_rn(G.y, dLda.y) : 0.0f);
  else g = mul2(make_float2(a0 ? G.x : 0.0f, a1 ? G.y : 0.0f), dLda);
  return true;
}

// Record of one instance from its summed terms s (unwind_step) and its (ca, cb, cc,
// opacity): power = ca dx^2 + cb dx dy + cc dy^2 with ca = -A/2, cb = -B, cc = -C/2 for
// the conic (A, B, C), so dL/dpower = opacity g and
//   dL/dmean2D = opacity (2 ca Sx + cb Sy, 2 cc Sy + cb Sx),
//   dL/d(A, B, C) = -opacity (Sxx / 2, Sxy, Syy / 2).
__device__ __forceinline__ void finish_record(float4* rec, const float (&s)[10], const float4& co) {
  const float op = co.w;
  const float dmx = op * fmaf(2.f * co.x, s[0], co.y * s[1]);
  const float dmy = op * fmaf(2.f * co.z, s[1], co.y * s[0]);
  rec[0] = make_float4(dmx, dmy, -0.5f * op * s[2], -op * s[3]);
  rec[1] = make_float4(-0.5f * op * s[4], s[5], s[6], s[7]);
  rec[2] = make_float4(s[8], s[9], 0.f, 0.f);
}

// Shared memory of a block. The gradient terms an instance sums: moments g (dx, dy, dx^2,
// dx dy, dy^2), and unless GEOM g, w dL/drgb, with DEPTH w dL/ddepth.
template <bool DEPTH, int BATCH, bool GEOM>
struct BwdShared {
  static constexpr int kTerms = GEOM ? 5 : (DEPTH ? 10 : 9);
  static constexpr int kPlanes = GEOM ? 0 : (DEPTH ? 4 : 3);
  float4 raw_co[BATCH], raw_rgbd[BATCH];  // the next batch, on its way (cp.async)
  float2 raw_xy[BATCH];
  uint32_t raw_pidx[BATCH];
  StagedInstance inst[BATCH];  // the current batch
  float thr[BATCH];
  uint32_t pidx[BATCH];
  float g[kWarps][kSlots][64];                 // a warp's slots: g per pixel of its 8x8 box (pair_offset)
  float w[kWarps][GEOM ? 1 : kSlots][GEOM ? 4 : 64];
  float image_grad[kWarps][GEOM ? 1 : kPlanes][GEOM ? 4 : 64];  // dL/dcolour (and depth) per pixel
  float part[kWarps][BATCH][kTerms];           // a warp's sums per instance
  uint8_t reached[BATCH][kWarps];              // 1: the instance reached some pixel of the warp
  uint32_t max_last;
};

// Where a warp's 8x8 box keeps a pixel pair (columns q and q + 4 of row y = 4 h + 2 m + l):
// the eight floats of a lane's rows l, l + 2, l + 4, l + 6 in two 16-byte words per l, the
// halves of a word swapped for m = 1. Both the pairs' stores (a half-warp at a time) and
// the 16-byte loads of sum_slots (eight lanes at a time) then meet 32 different banks.
__device__ __forceinline__ int pair_offset(int q, int y) {
  const int h = y >> 2, m = (y >> 1) & 1, l = y & 1;
  return 32 * m + 8 * q + 4 * l + 2 * (h ^ m);
}

// One warp's sums of its n <= 8 pending instances over the 64 pixels of its box. Four lanes
// take an instance: lane 4 s + q sums slot s over columns q and q + 4 (one packed pair per
// row), then the four lanes combine by a transposing exchange. An instance costs about 24
// warp instructions here; forming every pixel's moments in its own lane and reducing each
// instance over all 32 lanes by shuffles took about 70. The order of every sum is the one
// of that reduction — rows y and y + 4, then y and y + 2, y and y + 1, then columns 4, 2
// and 1 apart — so the records keep its bits. Odd slots take the odd rows first (an
// exchange of the operands of one addition), so that loads meet no common bank. ODD: as in
// unwind_pair.
template <bool ODD, bool DEPTH, int BATCH, bool GEOM>
__device__ __forceinline__ void sum_slots(BwdShared<DEPTH, BATCH, GEOM>& sh, int warp, int lane, int n, int j, int bx0,
                                          int by0) {
  using Sh = BwdShared<DEPTH, BATCH, GEOM>;
  constexpr int kTerms = Sh::kTerms, kPlanes = Sh::kPlanes;
  const int slot = lane >> 2, q = lane & 3, odd_first = slot & 1;
  __syncwarp();
  // an image gradient where the instance has a weight, else 0
  auto where = [](float2 d, float2 w) { return ODD ? make_float2(w.x != 0.f ? d.x : 0.f, w.y != 0.f ? d.y : 0.f) : d; };
  float v[10];
#pragma unroll
  for (int k = 0; k < 10; ++k) v[k] = 0.0f;
  if constexpr (!GEOM) {  // w dL/dcolour (and depth), apart from the moments: fewer live registers
    float2 c[kPlanes];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int o = 8 * q + 4 * (i ^ odd_first);
      const float4 wa = *reinterpret_cast<const float4*>(sh.w[warp][slot] + o);
      const float4 wb = *reinterpret_cast<const float4*>(sh.w[warp][slot] + o + 32);
#pragma unroll
      for (int k = 0; k < kPlanes; ++k) {
        const float4 da = *reinterpret_cast<const float4*>(sh.image_grad[warp][k] + o);
        const float4 db = *reinterpret_cast<const float4*>(sh.image_grad[warp][k] + o + 32);
        const float2 u = add2(fma2(where(hi2(da), hi2(wa)), hi2(wa), mul2(where(lo2(da), lo2(wa)), lo2(wa))),
                              fma2(where(lo2(db), lo2(wb)), lo2(wb), mul2(where(hi2(db), hi2(wb)), hi2(wb))));
        c[k] = i ? add2(c[k], u) : u;
      }
    }
#pragma unroll
    for (int k = 0; k < kPlanes; ++k) v[6 + k] = c[k].x + c[k].y;
  }
  __syncwarp();
  {
    const float4 xy = sh.inst[j].xy;
    const float2 dx = sub2(lo2(xy), make_float2((float)(bx0 + q), (float)(bx0 + q + 4)));
    float2 v2[6];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int l = i ^ odd_first;
      const float2 y0 = splat2((float)(by0 + l));
      float2 u[6];
#pragma unroll
      for (int m = 0; m < 2; ++m) {  // rows l + 2 m (x) and l + 2 m + 4 (y) of both columns
        const float4 gv = *reinterpret_cast<const float4*>(sh.g[warp][slot] + 32 * m + 8 * q + 4 * l);
        const float2 gx = m ? hi2(gv) : lo2(gv), gy = m ? lo2(gv) : hi2(gv);
        const float2 dyx = sub2(hi2(xy), m ? add2(y0, splat2(2.0f)) : y0);
        const float2 dyy = sub2(hi2(xy), add2(y0, splat2(m ? 6.0f : 4.0f)));
        const float2 hx = mul2(gx, dyx), hy = mul2(gy, dyy), sg = add2(gx, gy), sx = mul2(sg, dx);
        const float2 t1 = add2(hx, hy);
        const float2 t3 = fma2(mul2(gy, dx), dyy, mul2(mul2(gx, dx), dyx));
        const float2 t4 = fma2(hy, dyy, mul2(hx, dyx));
        // scalar products: a packed one would be fused with the addition
        const float2 t2 = make_float2(__fmul_rn(sx.x, dx.x), __fmul_rn(sx.y, dx.y));
        u[2] = m ? add2(u[2], t2) : t2;
        u[0] = m ? add2(u[0], sx) : sx;
        u[1] = m ? add2(u[1], t1) : t1;
        u[3] = m ? add2(u[3], t3) : t3;
        u[4] = m ? add2(u[4], t4) : t4;
        if (!GEOM) u[5] = m ? add2(u[5], sg) : sg;
      }
#pragma unroll
      for (int k = 0; k < (GEOM ? 5 : 6); ++k) v2[k] = i ? add2(v2[k], u[k]) : u[k];
    }
#pragma unroll
    for (int k = 0; k < (GEOM ? 5 : 6); ++k) v[k] = v2[k].x + v2[k].y;
  }
  // over the four lanes: lane q ends with terms 0-2, 3-4, 5-7, 8-9 of the instance (GEOM:
  // 0-1, 2, 3, 4)
  const bool up = q & 2, odd = q & 1;
  constexpr int kHalf = GEOM ? 3 : 5, kQuarter = GEOM ? 2 : 3;
#pragma unroll
  for (int k = 0; k < kHalf; ++k) {
    const float other = k + kHalf < 10 ? v[k + kHalf] : 0.0f;
    const float send = up ? v[k] : other, keep = up ? other : v[k];
    v[k] = keep + __shfl_xor_sync(0xffffffffu, send, 2);
  }
#pragma unroll
  for (int k = 0; k < kQuarter; ++k) {
    const float other = k + kQuarter < kHalf ? v[k + kQuarter] : 0.0f;
    const float send = odd ? v[k] : other, keep = odd ? other : v[k];
    v[k] = keep + __shfl_xor_sync(0xffffffffu, send, 1);
  }
  if (slot < n) {
    if (q == 0) sh.reached[j][warp] = 1;
    float* part = sh.part[warp][j];
    const int first = (up ? kHalf : 0) + (odd ? kQuarter : 0), end = min(up ? kTerms : kHalf, first + kQuarter);
#pragma unroll
    for (int k = 0; k < kQuarter; ++k)
      if (first + k < end) part[first + k] = v[k];
  }
  __syncwarp();  // the slots are free again
}

// One block of 128 threads per tile with the forward's pixel boxes (warp w: an 8x8 box,
// lane: columns q and q + 4 of a row) and exact shortcuts (box_may_contribute per
// warp and instance, alpha_threshold per pixel). A lane leaves its two pixels' g and w of a
// contributing instance in the warp's next slot; every eight instances the warp sums its
// slots (sum_slots). The cross-warp sum of an instance adds only the warps it contributed
// in (the others' terms are exact zeros). A tile whose image gradients are not all finite, or
// a view with a colour or depth that is not, takes the ODD form, since the sums run over all
// pixels of a box and 0 times such a value is no zero: it stays with the Gaussians that
// contribute to its pixel. BATCH instances are staged per round; the
// records do not depend on it (each instance's sums are formed the same way whatever batch
// it is staged in), so the batch is a schedule choice. GEOM forms only the moments (the
// terms of dL/dmean2D and dL/dconic), the same bits. Bound by instruction issue, and where
// fewer tiles than resident blocks run, by a warp's own chain. BLOCKS is the number of
// resident blocks per SM the registers are cut for (launch_render_bwd_batch). Against the
// per-instance shuffle reduction: 1,000,000 Gaussians at 1920x1080 984 -> 907 us (912 ->
// 711 million warp instructions), 16,384 at 256x256 134 -> 94 us, with depth gradients
// (250,007 at 977x545) 406 -> 313 us, one 640x360 pose solve (GEOM) 218 -> 175 us, 16
// solves 2989 -> 2429 us.
template <class Scenes, bool DEPTH, int BATCH, bool GEOM, int BLOCKS>
__global__ void __launch_bounds__(kBwdThreads, BLOCKS) k_render_bwd(RenderBwdArgs<Scenes> a) {
  static_assert(BATCH % 32 == 0 && BATCH <= kBwdThreads, "whole ballot words, one staged instance per thread");
  using Sh = BwdShared<DEPTH, BATCH, GEOM>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Sh& sh = *reinterpret_cast<Sh*>(smem_raw);
  const bool odd_view = *nonfinite_word(a.counts) != 0;  // on its way with the count and the pixels
  if ((int64_t)a.counts->num_rendered > a.cap) return;
  const int tile = blockIdx.x;
  const SceneDesc& sd = a.scenes.for_tile(tile);
  const int lt = tile - sd.tile_base;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int bx0 = (lt % sd.grid_x) * kTileX + (warp & 1) * 8;
  const int by0 = (lt / sd.grid_x) * kTileY + (warp >> 1) * 8;
  const int px0 = bx0 + (lane & 3), px1 = px0 + 4, py = by0 + (lane >> 2);
  const int slot_at = pair_offset(lane & 3, lane >> 2);
  const float bxf0 = (float)bx0, bxf1 = (float)(bx0 + 7), byf0 = (float)by0, byf1 = (float)(by0 + 7);
  const bool in0 = px0 < sd.W && py < sd.H, in1 = px1 < sd.W && py < sd.H;
  const float2 px = make_float2((float)px0, (float)px1), pyf = splat2((float)py);
  const uint32_t lo = a.tile_range[tile];

  PixelBwd p0, p1;
  load_pixel(p0, a, sd, in0, in0 ? (size_t)py * sd.W + px0 : 0);
  load_pixel(p1, a, sd, in1, in1 ? (size_t)py * sd.W + px1 : 0);
  PairBwd pp = make_pair(p0, p1);
  if constexpr (!GEOM) {
    *reinterpret_cast<float2*>(sh.image_grad[warp][0] + slot_at) = pp.dC0;
    *reinterpret_cast<float2*>(sh.image_grad[warp][1] + slot_at) = pp.dC1;
    *reinterpret_cast<float2*>(sh.image_grad[warp][2] + slot_at) = pp.dC2;
    if (DEPTH) *reinterpret_cast<float2*>(sh.image_grad[warp][3] + slot_at) = pp.dD;
  }
  if (threadIdx.x == 0) sh.max_last = 0;
  // a tile with an image gradient, or a view with a colour or depth, that is not finite
  const bool odd = __syncthreads_or(odd_view || !(all_finite(p0) && all_finite(p1)));
  const uint32_t my_last = max(p0.last, p1.last);
  if (my_last) atomicMax(&sh.max_last, my_last);
  // instances at or past the warp's largest contributor count reach none of its pixels
  const int warp_last = (int)__reduce_max_sync(0xffffffffu, my_last);
  __syncthreads();
  const int max_last = (int)sh.max_last;

  const int t = threadIdx.x;
  auto count_of = [&](int b) { return min(BATCH, max_last - b * BATCH); };
  uint32_t gnext = 0;
  auto load_id = [&](int b) { gnext = t < count_of(b) ? a.sorted_gid[lo + b * BATCH + t] : 0u; };
  auto issue = [&](int b) {
    if (t < count_of(b)) {
      cp_async4(&sh.raw_pidx[t], a.sorted_pidx + lo + (uint32_t)(b * BATCH + t));
      cp_async8(&sh.raw_xy[t], a.xy + gnext);
      cp_async16(&sh.raw_co[t], a.conic_op + gnext);
      cp_async16(&sh.raw_rgbd[t], a.rgbd + gnext);
    }
    cp_async_commit();
  };
  const int nb = (max_last + BATCH - 1) / BATCH;
  if (nb > 0) {
    load_id(nb - 1);
    issue(nb - 1);
    if (nb > 1) load_id(nb - 2);
  }
  // Batch b - 1 is copied asynchronously (its Gaussian ids were loaded a batch earlier)
  // while batch b is unwound; two block barriers per batch (staged, then partial sums
  // complete).
  auto unwind = [&](auto odd_form) {
    constexpr bool ODD = decltype(odd_form)::value;
    for (int b = nb - 1; b >= 0; --b) {
      const int base = b * BATCH;
      const int cnt = count_of(b);
      cp_async_wait_all();
      if (t < cnt) {  // raw values -> render form, own slot
        const float2 m = sh.raw_xy[t];
        const float4 co = sh.raw_co[t], c = sh.raw_rgbd[t];
        StagedInstance& s = sh.inst[t];
        const float ca = -0.5f * co.x, cb = -co.y, cc = -0.5f * co.z;
        s.xy = make_float4(m.x, m.x, m.y, m.y);
        s.ab = make_float4(ca, ca, cb, cb);
        s.co = make_float4(cc, cc, co.w, co.w);
        s.rg = make_float4(c.x, c.x, c.y, c.y);
        s.bd = make_float4(c.z, c.z, c.w, c.w);
        sh.thr[t] = alpha_threshold(co.w);
        sh.pidx[t] = sh.raw_pidx[t];
        *reinterpret_cast<uint32_t*>(sh.reached[t]) = 0u;
      }
      __syncthreads();  // batch b staged; batch b + 1 finished
      if (b > 0) {
        issue(b - 1);  // into this thread's own raw slot, read above
        if (b > 1) load_id(b - 2);
      }
      uint32_t keep[BATCH / 32];
  #pragma unroll
      for (int r = 0; r < BATCH / 32; ++r) {
        const int j = r * 32 + lane;
        bool kp = false;
        if (j < cnt && base + j < warp_last) {
          const StagedInstance& s = sh.inst[j];
          const float4 xy = s.xy, ab = s.ab;
          kp = box_may_contribute(make_float2(xy.x, xy.z), ab.x, ab.z, s.co.x, sh.thr[j], bxf0, bxf1, byf0, byf1);
        }
        keep[r] = __ballot_sync(0xffffffffu, kp);
      }
      // Back to front over the kept instances; the warp sums its slots whenever eight are
      // pending and after the last instance.
      int r = BATCH / 32 - 1;
      uint32_t mk = keep[r];
      for (bool more = true; more;) {
        int used = 0;    // slots pending
        int j_slot = 0;  // the instance in this lane's slot
        while (used < kSlots) {
          if (mk == 0) {
            if (r == 0) {
              more = false;
              break;
            }
            --r;
            mk = keep[0];
  #pragma unroll
            for (int k = 1; k < BATCH / 32; ++k)
              if (k == r) mk = keep[k];
            continue;
          }
          const int bit = 31 - __clz(mk);
          mk &= ~(1u << bit);
          const int j = r * 32 + bit;
          float2 g, w;
          const bool contrib = unwind_pair<DEPTH, ODD>(pp, base + j, px, pyf, sh.inst[j], sh.thr[j], g, w);
          if (!__any_sync(0xffffffffu, contrib)) continue;
          *reinterpret_cast<float2*>(sh.g[warp][used] + slot_at) = g;
          if constexpr (!GEOM) *reinterpret_cast<float2*>(sh.w[warp][used] + slot_at) = w;
          if ((lane >> 2) == used) j_slot = j;
          ++used;
        }
        if (used) sum_slots<ODD>(sh, warp, lane, used, j_slot, bx0, by0);
      }
      __syncthreads();  // every warp's partial sums of batch b are in
      if (t < cnt) {
        float sum[10];
  #pragma unroll
        for (int q = 0; q < 10; ++q) sum[q] = 0.f;
        const uint32_t reached = *reinterpret_cast<const uint32_t*>(sh.reached[t]);
  #pragma unroll
        for (int w = 0; w < kWarps; ++w)
          if ((reached >> (8 * w)) & 0xffu) {
  #pragma unroll
            for (int q = 0; q < Sh::kTerms; ++q) sum[q] += sh.part[w][t][q];
          }
        // An instance that reached no pixel has exact-zero gradients: no record, its byte stays 0.
        if (reached) {
          const uint32_t pidx = sh.pidx[t];
          const float4 ab = sh.inst[t].ab, co = sh.inst[t].co;
          finish_record(a.records + (size_t)kRecordFloat4 * pidx, sum, make_float4(ab.x, ab.z, co.x, co.z));
          a.written[pidx] = 1;
        }
      }
    }
  };
  if (odd) unwind(std::true_type{});
  else unwind(std::false_type{});
  // Instances at or past the tile's last contributor reach no pixel: nothing to write.
}

constexpr int kBwdSms = 152;

template <class Scenes, bool DEPTH, int BATCH, bool GEOM, int BLOCKS>
void launch_render_bwd_blocks(const RenderBwdArgs<Scenes>& a, int tiles, cudaStream_t st) {
  static std::atomic<uint64_t> smem_set{0};
  constexpr int bytes = (int)sizeof(BwdShared<DEPTH, BATCH, GEOM>);
  // a failure of the attribute call surfaces as a launch error
  ensure_dynamic_smem(k_render_bwd<Scenes, DEPTH, BATCH, GEOM, BLOCKS>, bytes, smem_set);
  k_render_bwd<Scenes, DEPTH, BATCH, GEOM, BLOCKS><<<tiles, kBwdThreads, bytes, st>>>(a);
}

// Registers against resident blocks. With fewer tiles than the blocks would fill, the
// registers win (fewer instructions per warp): 256 tiles 94 us at four blocks per SM, 99
// at five; 920 pose tiles 175 us at six, 187 at seven. With many tiles the extra block
// does: 8160 tiles 907 us at five, 987 at four; 20,960 pose tiles 2429 us at seven, 2551 at
// six. Around the lines (608 and 1216 tiles) neither matters much: 625 tiles with 5 instances
// per Gaussian 119 us at four and at five, 800 tiles 121 and 119, 1024 tiles 136 and 129; pose
// form 1024 tiles 119 and 121 us at six and seven, 1280 136 and 134, 1600 149 and 147. The
// depth form, with more live sums, keeps four (2170 tiles: 313 us, 342 at five).
template <class Scenes, bool DEPTH, int BATCH, bool GEOM>
void launch_render_bwd_batch(const RenderBwdArgs<Scenes>& a, int tiles, cudaStream_t st) {
  if constexpr (GEOM) {
    if (tiles <= 8 * kBwdSms) launch_render_bwd_blocks<Scenes, DEPTH, BATCH, GEOM, 6>(a, tiles, st);
    else launch_render_bwd_blocks<Scenes, DEPTH, BATCH, GEOM, 7>(a, tiles, st);
  } else if constexpr (DEPTH) {
    launch_render_bwd_blocks<Scenes, DEPTH, BATCH, GEOM, 4>(a, tiles, st);
  } else {
    if (tiles <= 4 * kBwdSms) launch_render_bwd_blocks<Scenes, DEPTH, BATCH, GEOM, 4>(a, tiles, st);
    else launch_render_bwd_blocks<Scenes, DEPTH, BATCH, GEOM, 5>(a, tiles, st);
  }
}

template <class Scenes, bool DEPTH, bool GEOM = false>
void launch_render_bwd_depth(const RenderBwdArgs<Scenes>& a, int tiles, int batch, cudaStream_t st) {
  if (batch == 32) launch_render_bwd_batch<Scenes, DEPTH, 32, GEOM>(a, tiles, st);
  else if (batch == 128) launch_render_bwd_batch<Scenes, DEPTH, 128, GEOM>(a, tiles, st);
  else launch_render_bwd_batch<Scenes, DEPTH, 64, GEOM>(a, tiles, st);
}

template <class Scenes>
void launch_render_bwd(const RenderBwdArgs<Scenes>& a, int tiles, cudaStream_t st) {
  const int batch = a.sched.bwd_batch;
  if constexpr (Scenes::kBatched) {  // batched solves never ask for depth gradients
    if (a.geom_only) launch_render_bwd_depth<Scenes, false, true>(a, tiles, batch, st);
    else launch_render_bwd_depth<Scenes, false>(a, tiles, batch, st);
  } else {
    if (a.geom_only) launch_render_bwd_depth<Scenes, false, true>(a, tiles, batch, st);
    else if (a.dL_ddepth) launch_render_bwd_depth<Scenes, true>(a, tiles, batch, st);
    else launch_render_bwd_depth<Scenes, false>(a, tiles, batch, st);
  }
}
template void launch_render_bwd<SingleScene>(const RenderBwdArgs<SingleScene>&, int, cudaStream_t);
template void launch_render_bwd<SceneTable>(const RenderBwdArgs<SceneTable>&, int, cudaStream_t);

}  // namespace cfgs

using namespace cfgs;

static int render_backward(const CfgsSettings* s, int32_t num_gaussians, const void* geom, const void* image,
                           const void* binning, int64_t capacity, void* scratch, const float* dL_dcolor,
                           const float* dL_ddepth, const float* dL_dalpha, bool means_only, void* stream) {
  if (!s || !geom || !image || !binning || !scratch || !dL_dcolor || !s->bg || num_gaussians < 0)
    return CFGS_ERR_INVALID_ARGUMENT;
  if (s->image_width <= 0 || s->image_height <= 0) return CFGS_ERR_INVALID_ARGUMENT;
  if (capacity < 0 || capacity > 0x7fffffffll) return CFGS_ERR_INVALID_ARGUMENT;
  cudaStream_t st = (cudaStream_t)stream;
  ImageLayout IL(s->image_width, s->image_height);
  ImageView iv(const_cast<void*>(image), s->image_width, s->image_height);
  GeomView gv(const_cast<void*>(geom), num_gaussians);
  BinningView bv(const_cast<void*>(binning), capacity);
  RenderBwdArgs<SingleScene> ra;
  ra.scenes.d = single_scene_desc(s, num_gaussians, 0);
  ra.tile_range = iv.tile_range;
  ra.sorted_gid = bv.sorted_gid;
  ra.sorted_pidx = bv.sorted_pidx;
  ra.xy = gv.xy;
  ra.conic_op = gv.conic_op;
  ra.rgbd = gv.rgbd;
  ra.final_T = iv.final_T;
  ra.n_contrib = iv.n_contrib;
  ra.dL_dcolor = dL_dcolor;
  ra.dL_ddepth = dL_ddepth;
  ra.dL_dalpha = dL_dalpha;
  ra.color = nullptr;
  ra.target = nullptr;
  const ScratchLayout SL(capacity);
  ra.records = reinterpret_cast<float4*>(static_cast<char*>(scratch) + SL.records);
  ra.written = reinterpret_cast<uint8_t*>(static_cast<char*>(scratch) + SL.written);
  ra.cap = capacity;
  ra.counts = iv.counts;
  if (!resolve_schedule(s->schedule, IL.num_tiles, 0, 0, &ra.sched)) return CFGS_ERR_INVALID_ARGUMENT;
  ra.geom_only = means_only;
  if (capacity > 0 && cudaMemsetAsync(ra.written, 0, (size_t)capacity, st) != cudaSuccess) return CFGS_ERR_LAUNCH;
  launch_render_bwd(ra, IL.num_tiles, st);
  CFGS_CHECK_LAUNCH(s->debug, st);
  return CFGS_OK;
}

extern "C" int cfgs_render_backward(const CfgsSettings* s, int32_t num_gaussians, const void* geom, const void* image,
                                    const void* binning, int64_t capacity, void* scratch, const float* dL_dcolor,
                                    const float* dL_ddepth, const float* dL_dalpha, void* stream) {
  return render_backward(s, num_gaussians, geom, image, binning, capacity, scratch, dL_dcolor, dL_ddepth, dL_dalpha,
                         false, stream);
}

extern "C" int cfgs_render_backward_means(const CfgsSettings* s, int32_t num_gaussians, const void* geom,
                                          const void* image, const void* binning, int64_t capacity, void* scratch,
                                          const float* dL_dcolor, const float* dL_dalpha, void* stream) {
  return render_backward(s, num_gaussians, geom, image, binning, capacity, scratch, dL_dcolor, nullptr, dL_dalpha, true,
                         stream);
}

// Which gradient arrays a caller wants: all eight, those of its inputs, the means'.
enum Wanted { kAllArrays, kInputArrays, kMeansArrays };

static int preprocess_backward(const CfgsSettings* s, const CfgsGaussians* g, const int32_t* radii, const void* geom,
                               const void* image, int64_t capacity, const void* scratch, const CfgsGradients* out,
                               Wanted wanted, void* stream) {
  const bool means_only = wanted == kMeansArrays;
  if (!s || !g || !geom || !image || !scratch || !out || !s->viewmatrix || !s->projmatrix)
    return CFGS_ERR_INVALID_ARGUMENT;
  if (g->num_gaussians == 0) return CFGS_OK;
  if (g->num_gaussians < 0 || !radii || !g->means3D || !g->opacities) return CFGS_ERR_INVALID_ARGUMENT;
  if (!out->dL_dmeans2D || !out->dL_dmeans3D) return CFGS_ERR_INVALID_ARGUMENT;
  if (!means_only && (!out->dL_dopacity || (!g->cov3D_precomp && (!out->dL_dscales || !out->dL_drotations))))
    return CFGS_ERR_INVALID_ARGUMENT;
  if (!means_only && ((!out->dL_dcolors && (wanted == kAllArrays || !g->shs)) ||
                      (!out->dL_dcov3D && (wanted == kAllArrays || g->cov3D_precomp))))
    return CFGS_ERR_INVALID_ARGUMENT;
  if (!g->cov3D_precomp && (!g->scales || !g->rotations)) return CFGS_ERR_INVALID_ARGUMENT;
  if (means_only && g->shs && s->sh_degree != 0) return CFGS_ERR_INVALID_ARGUMENT;
  if ((g->shs == nullptr) == (g->colors_precomp == nullptr)) return CFGS_ERR_INVALID_ARGUMENT;
  if (g->shs && !s->campos) return CFGS_ERR_INVALID_ARGUMENT;
  if (capacity < 0 || capacity > 0x7fffffffll) return CFGS_ERR_INVALID_ARGUMENT;
  cudaStream_t st = (cudaStream_t)stream;
  ImageView iv(const_cast<void*>(image), s->image_width, s->image_height);
  PreBwdArgs<SingleScene> pa;
  pa.scenes.d = single_scene_desc(s, g->num_gaussians, g->sh_coeffs);
  pa.g = *g;
  pa.radii = radii;
  pa.geom = GeomView(const_cast<void*>(geom), g->num_gaussians);
  const ScratchLayout SL(capacity);
  pa.records = reinterpret_cast<const float4*>(static_cast<const char*>(scratch) + SL.records);
  pa.written = reinterpret_cast<const uint8_t*>(static_cast<const char*>(scratch) + SL.written);
  pa.out = *out;
  pa.total_slots = g->num_gaussians;
  pa.cap = capacity;
  pa.counts = iv.counts;
  pa.pose_partials = nullptr;
  pa.flags = &iv.counts->flags;
  pa.sh_bulk = g->shs != nullptr && g->sh_coeffs == CFGS_SH_BULK_COEFFS && (((uintptr_t)g->shs) & 15) == 0 &&
               (out->dL_dsh == nullptr || (((uintptr_t)out->dL_dsh) & 15) == 0);
  pa.means_only = means_only;
  launch_preprocess_bwd(pa, div_up(g->num_gaussians, 256), st);
  CFGS_CHECK_LAUNCH(s->debug, st);
  return CFGS_OK;
}

extern "C" int cfgs_preprocess_backward(const CfgsSettings* s, const CfgsGaussians* g, const int32_t* radii,
                                        const void* geom, const void* image, int64_t capacity, const void* scratch,
                                        const CfgsGradients* out, void* stream) {
  return preprocess_backward(s, g, radii, geom, image, capacity, scratch, out, kAllArrays, stream);
}

extern "C" int cfgs_preprocess_backward_inputs(const CfgsSettings* s, const CfgsGaussians* g, const int32_t* radii,
                                               const void* geom, const void* image, int64_t capacity,
                                               const void* scratch, const CfgsGradients* out, void* stream) {
  return preprocess_backward(s, g, radii, geom, image, capacity, scratch, out, kInputArrays, stream);
}

extern "C" int cfgs_preprocess_backward_means(const CfgsSettings* s, const CfgsGaussians* g, const int32_t* radii,
                                              const void* geom, const void* image, int64_t capacity,
                                              const void* scratch, float* dL_dmeans2D, float* dL_dmeans3D,
                                              void* stream) {
  CfgsGradients out{};
  out.dL_dmeans2D = dL_dmeans2D;
  out.dL_dmeans3D = dL_dmeans3D;
  return preprocess_backward(s, g, radii, geom, image, capacity, scratch, &out, kMeansArrays, stream);
}

extern "C" int cfgs_backward(const CfgsSettings* s, const CfgsGaussians* g, const int32_t* radii, const void* geom,
                             const void* image, const void* binning, int64_t capacity, void* scratch,
                             const float* dL_dcolor, const float* dL_ddepth, const float* dL_dalpha,
                             const CfgsGradients* out, void* stream) {
  if (!g) return CFGS_ERR_INVALID_ARGUMENT;
  if (g->num_gaussians == 0) return CFGS_OK;
  int st = cfgs_render_backward(s, g->num_gaussians, geom, image, binning, capacity, scratch, dL_dcolor, dL_ddepth,
                                dL_dalpha, stream);
  if (st != CFGS_OK) return st;
  return cfgs_preprocess_backward(s, g, radii, geom, image, capacity, scratch, out, stream);
}

// ---- allocation-free backward ----------------------------------------------------
// Some callers cannot allocate device memory when they call the rasteriser: plugin
// hosts that hand a plugin only its input and output buffers, and services that must
// not allocate once they are serving. This entry point runs the same two kernels as
// cfgs_backward, but its per-instance scratch (gradient records and their written
// bytes, the layout cfgs_backward_scratch_bytes sizes) lives in the fixed array below
// instead of a caller-provided buffer. Every GPU that loads this library holds the
// array (30.6 MiB) until the process exits.
constexpr size_t kNoallocRecordBytes = ((size_t)CFGS_NOALLOC_MAX_INSTANCES * 16 * kRecordFloat4 + 255) & ~size_t(255);
constexpr size_t kNoallocScratchBytes = kNoallocRecordBytes + (((size_t)CFGS_NOALLOC_MAX_INSTANCES + 255) & ~size_t(255));
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoallocScratchBytes];

namespace {
// The array's device address belongs to the CUDA context that loaded this library's
// device code: after cudaDeviceReset, or in another context on the same device, the
// module is loaded again and the array may sit elsewhere. So the address is cached per
// context, keyed by the driver's context id (unique for the life of the process, even
// when a new context reuses a freed one's handle), and looked up again for a context
// not seen before. The driver functions come through the runtime's entry-point query,
// so the library does not link the driver library itself.
typedef int (*CtxGetCurrentFn)(void** ctx);
typedef int (*CtxGetIdFn)(void* ctx, unsigned long long* id);
constexpr int kNoallocCacheSize = 64;
struct NoallocEntry {
  unsigned long long ctx_id;
  void* ptr;
};
std::mutex g_noalloc_mutex;
NoallocEntry g_noalloc_cache[kNoallocCacheSize];
int g_noalloc_used = 0, g_noalloc_next = 0;
CtxGetCurrentFn g_ctx_get_current = nullptr;
CtxGetIdFn g_ctx_get_id = nullptr;

bool context_id(unsigned long long* id) {
  void* ctx = nullptr;
  if (g_ctx_get_current(&ctx) != 0 || ctx == nullptr) return false;
  return g_ctx_get_id(ctx, id) == 0;
}

// Device address of g_noalloc_scratch in the current context. The host-side name of
// the array is only a stand-in for it, so the address comes from cudaGetSymbolAddress,
// called with the caller's device current, once per context.
int noalloc_scratch(void** out) {
  std::lock_guard<std::mutex> lock(g_noalloc_mutex);
  if (!g_ctx_get_current || !g_ctx_get_id) {
    cudaDriverEntryPointQueryResult q1, q2;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", reinterpret_cast<void**>(&g_ctx_get_current), 12000,
                                         cudaEnableDefault, &q1) != cudaSuccess ||
        cudaGetDriverEntryPointByVersion("cuCtxGetId", reinterpret_cast<void**>(&g_ctx_get_id), 12000,
                                         cudaEnableDefault, &q2) != cudaSuccess ||
        q1 != cudaDriverEntryPointSuccess || q2 != cudaDriverEntryPointSuccess) {
      g_ctx_get_current = nullptr;
      g_ctx_get_id = nullptr;
      return CFGS_ERR_LAUNCH;
    }
  }
  unsigned long long id = 0;
  const bool have_ctx = context_id(&id);
  if (have_ctx)
    for (int i = 0; i < g_noalloc_used; ++i)
      if (g_noalloc_cache[i].ctx_id == id) {
        *out = g_noalloc_cache[i].ptr;
        return CFGS_OK;
      }
  // Not seen yet (or no context current: the lookup below makes the device's primary
  // context current and loads the module).
  void* p = nullptr;
  if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || p == nullptr) return CFGS_ERR_LAUNCH;
  if (!context_id(&id)) return CFGS_ERR_LAUNCH;
  const int slot = g_noalloc_used < kNoallocCacheSize ? g_noalloc_used++ : (g_noalloc_next++ % kNoallocCacheSize);
  g_noalloc_cache[slot] = NoallocEntry{id, p};
  *out = p;
  return CFGS_OK;
}
}  // namespace

extern "C" int cfgs_backward_noalloc(const CfgsSettings* s, const CfgsGaussians* g, const int32_t* radii,
                                     const void* geom, const void* image, const void* binning, int64_t capacity,
                                     const float* dL_dcolor, const float* dL_ddepth, const float* dL_dalpha,
                                     const CfgsGradients* out, void* stream) {
  if (capacity < 0) return CFGS_ERR_INVALID_ARGUMENT;
  if (capacity > CFGS_NOALLOC_MAX_INSTANCES) return CFGS_ERR_TOO_LARGE;
  void* scratch = nullptr;
  int st = noalloc_scratch(&scratch);
  if (st != CFGS_OK) return st;
  return cfgs_backward(s, g, radii, geom, image, binning, capacity, scratch, dL_dcolor, dL_ddepth, dL_dalpha, out,
                       stream);
}
