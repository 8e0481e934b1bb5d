// Optimisation of the Gaussian parameters (CF-3DGS global refinement and local fitting,
// trainer/cf3dgs_trainer.py:144-170 / 232-259): the Adam step over every parameter
// group, the densification statistics and densify-and-prune of
// scene/gaussian_model_cf.py:242-301 and 605-719, on device-resident arrays.
//
// Adam: one launch for all groups (xyz, f_dc, f_rest, opacity, scaling, rotation) with
// the operation sequence of torch's multi-tensor Adam (non-capturable):
//   m = lerp(m, g, 1 - b1) = fma(1 - b1, g - m, m); v = fma(1 - b2, g * g, v * b2);
//   p = fma(-lr / bc1, m / (sqrt(v) / sqrt(bc2) + eps), p)
// with the per-group scalars formed on the host as torch forms them.
//
// Densify and prune (densify_and_prune with grads = accum / denom, nan -> 0):
//   clone  = |grad| >= max_grad and max(exp(scaling)) <= percent_dense * extent
//   split  = |grad| >= max_grad and max(exp(scaling)) >  percent_dense * extent
//   prune  = sigmoid(opacity) < min_opacity, or (with the screen test enabled)
//            max(exp(scaling)) > 0.1 * extent (the screen-size term is always false
//            then: densification resets max_radii2D to zero)
// The result lists, in this order: the originals that are neither split nor pruned;
// the clones (copies of the raw parameters) whose source is not pruned; then two blocks
// of split children (copy 0 of every split point, then copy 1) not pruned, each child
// at xyz + R(q) (exp(scaling) * z), scaling log(exp(scaling) / 1.6), the rest copied.
// z are the caller's standard-normal draws, [2, splits, 3]. New rows get zero Adam
// moments; the statistics restart at zero.
#include <cmath>

#include "cfgs_internal.cuh"
#include "kernels.cuh"

namespace cfgs {

constexpr int kMaxAdamGroups = 8;

struct AdamGroups {
  float* p[kMaxAdamGroups];
  const float* g[kMaxAdamGroups];
  float* m[kMaxAdamGroups];
  float* v[kMaxAdamGroups];
  int64_t begin[kMaxAdamGroups + 1];  // flattened ranges of 4-element items
  int64_t numel[kMaxAdamGroups];
  float step_size[kMaxAdamGroups];    // -lr / bc1
  float bc2_sqrt[kMaxAdamGroups];
  float eps[kMaxAdamGroups];
  float w1, b2, w2;
  int count;
};

__device__ __forceinline__ void adam_elem(const AdamGroups& a, int k, float g, float& m, float& v, float& p) {
  m = fmaf(a.w1, g - m, m);
  v = v * a.b2;
  v = fmaf(a.w2, g * g, v);
  float denom = sqrtf(v) / a.bc2_sqrt[k];
  denom = denom + a.eps[k];
  p = fmaf(a.step_size[k], m / denom, p);
}

// One thread per 4 consecutive elements of a group (begin[] counts 4-element items, each
// group padded to a whole item): vector loads and stores where the item is whole and the
// arrays 16-byte aligned, scalar ones otherwise.
__global__ void __launch_bounds__(256) k_gaussian_adam(AdamGroups a) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= a.begin[a.count]) return;
  int k = 0;
  while (k + 1 < a.count && t >= a.begin[k + 1]) ++k;
  const int64_t e0 = 4 * (t - a.begin[k]);
  const int64_t numel = a.numel[k];
  float* P = a.p[k];
  const float* G = a.g[k];
  float* Mv = a.m[k];
  float* Vv = a.v[k];
  const bool vec = e0 + 3 < numel && ((((uintptr_t)P) | ((uintptr_t)G) | ((uintptr_t)Mv) | ((uintptr_t)Vv)) & 15) == 0;
  if (vec) {
    const float4 g4 = *reinterpret_cast<const float4*>(G + e0);
    float4 m4 = *reinterpret_cast<float4*>(Mv + e0), v4 = *reinterpret_cast<float4*>(Vv + e0);
    float4 p4 = *reinterpret_cast<float4*>(P + e0);
    adam_elem(a, k, g4.x, m4.x, v4.x, p4.x);
    adam_elem(a, k, g4.y, m4.y, v4.y, p4.y);
    adam_elem(a, k, g4.z, m4.z, v4.z, p4.z);
    adam_elem(a, k, g4.w, m4.w, v4.w, p4.w);
    *reinterpret_cast<float4*>(Mv + e0) = m4;
    *reinterpret_cast<float4*>(Vv + e0) = v4;
    *reinterpret_cast<float4*>(P + e0) = p4;
  } else {
    for (int64_t e = e0; e < min(numel, e0 + 4); ++e) {
      float m = Mv[e], v = Vv[e], p = P[e];
      adam_elem(a, k, G[e], m, v, p);
      Mv[e] = m;
      Vv[e] = v;
      P[e] = p;
    }
  }
}

// xyz_gradient_accum[i] += |grad2D[i, :2]|, denom[i] += 1 where radii[i] > 0
// (add_densification_stats with the visibility filter).
__global__ void __launch_bounds__(256) k_densify_stats(int64_t n, const int32_t* __restrict__ radii,
                                                       const float* __restrict__ grad2D, float* __restrict__ accum,
                                                       float* __restrict__ denom) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n || radii[i] <= 0) return;
  const float gx = grad2D[3 * i], gy = grad2D[3 * i + 1];
  accum[i] += sqrtf(gx * gx + gy * gy);
  denom[i] += 1.0f;
}

struct DensifyParams {
  float max_grad, min_opacity, extent, percent_dense;
  int prune_big;
};

__device__ __forceinline__ float max_scale(const float* s) { return fmaxf(fmaxf(expf(s[0]), expf(s[1])), expf(s[2])); }

// The plan: every point's class bits and every block's counts of them (k_densify_classify,
// 1024 points per block), the exclusive prefix of the block counts (k_densify_prefix, one
// block), then each output row's source (k_densify_map). Ranks inside a block come from
// ballots: a class bit costs one ballot per warp instead of a five-step shuffle scan, and
// the map needs no per-point positions in memory. 1,000,000 points: 84 -> 38 us.
constexpr int kDensBlock = 1024;
constexpr int kDensWarps = kDensBlock / 32;

// Per point: bit 0 keep original, bit 1 kept clone, bit 2 split, bit 3 kept children.
__device__ __forceinline__ uint32_t densify_class(int64_t i, const float* __restrict__ accum,
                                                  const float* __restrict__ denom, const float* __restrict__ scaling,
                                                  const float* __restrict__ opacity, const DensifyParams& d) {
  float g = accum[i] / denom[i];
  if (g != g) g = 0.0f;
  const float smax = max_scale(scaling + 3 * i);
  const float thr = d.percent_dense * d.extent;
  const bool hot = fabsf(g) >= d.max_grad;
  const bool clone = hot && smax <= thr;
  const bool split = hot && smax > thr;
  const float op = 1.0f / (1.0f + expf(-opacity[i]));
  const bool low = op < d.min_opacity;
  const bool big = d.prune_big && smax > 0.1f * d.extent;
  // children: scaling log(exp(s) / 1.6) per axis
  float cs[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) cs[a] = logf(expf(scaling[3 * i + a]) / 1.6f);
  const bool child_big = d.prune_big && max_scale(cs) > 0.1f * d.extent;
  uint32_t c = 0;
  if (!split && !(low || big)) c |= 1u;
  if (clone && !(low || big)) c |= 2u;
  if (split) c |= 4u;
  if (split && !(low || child_big)) c |= 8u;
  return c;
}

__global__ void __launch_bounds__(kDensBlock) k_densify_classify(int64_t n, const float* __restrict__ accum,
                                                                 const float* __restrict__ denom,
                                                                 const float* __restrict__ scaling,
                                                                 const float* __restrict__ opacity, DensifyParams d,
                                                                 uint32_t* __restrict__ cls,
                                                                 uint4* __restrict__ bcount) {
  __shared__ uint32_t s_count[4];
  if (threadIdx.x < 4) s_count[threadIdx.x] = 0;
  __syncthreads();
  const int64_t i = (int64_t)blockIdx.x * kDensBlock + threadIdx.x;
  const uint32_t c = i < n ? densify_class(i, accum, denom, scaling, opacity, d) : 0u;
  if (i < n) cls[i] = c;
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    const unsigned m = __ballot_sync(0xffffffffu, (c >> b) & 1u);
    if ((threadIdx.x & 31) == 0 && m) atomicAdd(&s_count[b], (uint32_t)__popc(m));
  }
  __syncthreads();
  if (threadIdx.x == 0) bcount[blockIdx.x] = make_uint4(s_count[0], s_count[1], s_count[2], s_count[3]);
}

// The block counts become their exclusive prefix in place; the totals go to tot.
__global__ void __launch_bounds__(kDensBlock) k_densify_prefix(int nblocks, uint4* __restrict__ bcount,
                                                               uint4* __restrict__ tot) {
  __shared__ uint4 s_warp[kDensWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint4 carry = make_uint4(0, 0, 0, 0);
  for (int base = 0; base < nblocks; base += kDensBlock) {
    const int j = base + threadIdx.x;
    const uint4 v = j < nblocks ? bcount[j] : make_uint4(0, 0, 0, 0);
    uint4 x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y0 = __shfl_up_sync(0xffffffffu, x.x, o), y1 = __shfl_up_sync(0xffffffffu, x.y, o);
      const uint32_t y2 = __shfl_up_sync(0xffffffffu, x.z, o), y3 = __shfl_up_sync(0xffffffffu, x.w, o);
      if (lane >= o) x = make_uint4(x.x + y0, x.y + y1, x.z + y2, x.w + y3);
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    uint4 before = carry;
    for (int w = 0; w < kDensWarps; ++w) {
      const uint4 t = s_warp[w];
      if (w < warp) before = make_uint4(before.x + t.x, before.y + t.y, before.z + t.z, before.w + t.w);
      carry = make_uint4(carry.x + t.x, carry.y + t.y, carry.z + t.z, carry.w + t.w);
    }
    if (j < nblocks)
      bcount[j] = make_uint4(before.x + x.x - v.x, before.y + x.y - v.y, before.z + x.z - v.z, before.w + x.w - v.w);
    __syncthreads();
  }
  if (threadIdx.x == 0) *tot = carry;
}

// src[r] = source point of output row r: the kept originals, the kept clones, the
// children of copy 0, then of copy 1; split_rank[r] = a child's index among the split
// points.
__global__ void __launch_bounds__(kDensBlock) k_densify_map(int64_t n, const uint32_t* __restrict__ cls,
                                                            const uint4* __restrict__ bprefix,
                                                            const uint4* __restrict__ tot,
                                                            uint32_t* __restrict__ out_src,
                                                            uint32_t* __restrict__ out_split_rank) {
  __shared__ uint32_t s_count[kDensWarps][4];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t i = (int64_t)blockIdx.x * kDensBlock + threadIdx.x;
  const uint32_t c = i < n ? cls[i] : 0u;
  uint32_t rank[4];
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    const unsigned m = __ballot_sync(0xffffffffu, (c >> b) & 1u);
    rank[b] = (uint32_t)__popc(m & ((1u << lane) - 1u));
    if (lane == 0) s_count[warp][b] = (uint32_t)__popc(m);
  }
  __syncthreads();
  if (c == 0) return;
  const uint4 first = bprefix[blockIdx.x], all = *tot;
  rank[0] += first.x;
  rank[1] += first.y;
  rank[2] += first.z;
  rank[3] += first.w;
  for (int w = 0; w < warp; ++w)
#pragma unroll
    for (int b = 0; b < 4; ++b) rank[b] += s_count[w][b];
  if (c & 1u) out_src[rank[0]] = (uint32_t)i;
  if (c & 2u) out_src[all.x + rank[1]] = (uint32_t)i;
  if (c & 8u) {
#pragma unroll
    for (int cp = 0; cp < 2; ++cp) {
      const uint32_t r = all.x + all.y + cp * all.w + rank[3];
      out_src[r] = (uint32_t)i;
      out_split_rank[r] = rank[2];
    }
  }
}

// Rows of several parameter arrays: out[r] = in[src[r]] (zeros for the rows from
// first_new on where an array's new rows are zero, i.e. Adam moments). Bound by HBM:
// each kept float is read and written once. One launch covers all arrays; a block takes
// up to kGatherRows rows of one array (about kGatherFloats floats), holds their sources in
// shared memory and walks the flattened floats, eight loads per thread in flight, with
// both sides coalesced. 1,000,000 Gaussians, 18 arrays of 1 to 45 floats a row (1.2 GB
// moved): 1035 us as one launch per array, a 64-bit division per float and one load in
// flight -> 243 us (4.9 TB/s).
constexpr int kGatherArrays = 24;
constexpr int kGatherThreads = 256;
constexpr int kGatherRows = 2048;
constexpr int kGatherFloats = 8192;
constexpr int kGatherUnroll = 8;

struct GatherArgs {
  const float* in[kGatherArrays];
  float* out[kGatherArrays];
  int64_t rows[kGatherArrays];       // rows written (the child rows of xyz and scaling are k_densify_children's)
  uint32_t first_block[kGatherArrays + 1];
  int32_t width[kGatherArrays];
  int32_t block_rows[kGatherArrays];
  bool zero_new[kGatherArrays];
  int32_t count;
};

__global__ void __launch_bounds__(kGatherThreads) k_densify_gather(GatherArgs a, int64_t first_new,
                                                                   const uint32_t* __restrict__ src) {
  __shared__ uint32_t s_src[kGatherRows];
  constexpr uint32_t kZeroRow = 0xffffffffu;  // sources are below 2^30
  int k = 0;
  while (k + 1 < a.count && blockIdx.x >= a.first_block[k + 1]) ++k;
  const int64_t r0 = (int64_t)(blockIdx.x - a.first_block[k]) * a.block_rows[k];
  const int nr = (int)min((int64_t)a.block_rows[k], a.rows[k] - r0);
  const bool zero_new = a.zero_new[k];
  for (int r = threadIdx.x; r < nr; r += kGatherThreads)
    s_src[r] = zero_new && r0 + r >= first_new ? kZeroRow : src[r0 + r];
  __syncthreads();
  const uint32_t w = (uint32_t)a.width[k];
  // t / w = umulhi(t, magic) for w > 1 and t w < 2^32; a block of several rows has w <= 4096 and t < 8192
  const uint32_t magic = 0xffffffffu / w + 1u;
  const float* __restrict__ in = a.in[k];
  float* __restrict__ out = a.out[k] + (size_t)r0 * w;
  const uint32_t cnt = (uint32_t)nr * w;
  for (uint32_t t0 = threadIdx.x; t0 < cnt; t0 += kGatherThreads * kGatherUnroll) {
    float v[kGatherUnroll];
#pragma unroll
    for (int u = 0; u < kGatherUnroll; ++u) {
      const uint32_t t = t0 + u * kGatherThreads;
      v[u] = 0.0f;
      if (t < cnt) {
        const uint32_t r = w == 1 ? t : (nr > 1 ? __umulhi(t, magic) : 0u);
        const uint32_t s = s_src[r];
        if (s != kZeroRow) v[u] = in[(size_t)s * w + (t - r * w)];
      }
    }
#pragma unroll
    for (int u = 0; u < kGatherUnroll; ++u) {
      const uint32_t t = t0 + u * kGatherThreads;
      if (t < cnt) out[t] = v[u];
    }
  }
}

// Child rows (from row first_child on, copy 0 then copy 1 of `children` points) of xyz:
// xyz + R(normalize(q)) (exp(s) * z), and of scaling: log(exp(s) / 1.6); an output that is
// NULL is not wanted. R as build_rotation (utils/general_utils.py:76-97).
__global__ void __launch_bounds__(256) k_densify_children(int64_t first_child, int64_t children,
                                                          const uint32_t* __restrict__ src,
                                                          const uint32_t* __restrict__ split_rank,
                                                          uint32_t num_split, const float* __restrict__ xyz,
                                                          const float* __restrict__ scaling,
                                                          const float* __restrict__ rotation,
                                                          const float* __restrict__ z, float* __restrict__ out_xyz,
                                                          float* __restrict__ out_scaling) {
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= 2 * children) return;
  const int64_t r = first_child + c;
  const uint32_t i = src[r];
  const int cp = c >= children;
  if (out_scaling) {
#pragma unroll
    for (int a = 0; a < 3; ++a) out_scaling[3 * r + a] = logf(expf(scaling[3 * (size_t)i + a]) / 1.6f);
  }
  if (!out_xyz) return;
  const float* q = rotation + 4 * (size_t)i;
  const float nrm = sqrtf(q[0] * q[0] + q[1] * q[1] + q[2] * q[2] + q[3] * q[3]);
  const float qr = q[0] / nrm, qx = q[1] / nrm, qy = q[2] / nrm, qz = q[3] / nrm;
  const float R[9] = {1.f - 2.f * (qy * qy + qz * qz), 2.f * (qx * qy - qr * qz), 2.f * (qx * qz + qr * qy),
                      2.f * (qx * qy + qr * qz), 1.f - 2.f * (qx * qx + qz * qz), 2.f * (qy * qz - qr * qx),
                      2.f * (qx * qz - qr * qy), 2.f * (qy * qz + qr * qx), 1.f - 2.f * (qx * qx + qy * qy)};
  const float* zz = z + 3 * ((size_t)cp * num_split + split_rank[r]);
  float smp[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) smp[a] = expf(scaling[3 * (size_t)i + a]) * zz[a];
#pragma unroll
  for (int a = 0; a < 3; ++a)
    out_xyz[3 * r + a] =
        (R[3 * a] * smp[0] + R[3 * a + 1] * smp[1] + R[3 * a + 2] * smp[2]) + xyz[3 * (size_t)i + a];
}

// Workspace of a plan: class bits, totals, sources and split ranks of up to 3 n rows, block
// counts. The totals and block counts, of 16-byte words, begin at the next such boundary
// (aligned16).
struct DensifyLayout {
  size_t cls, tot, src, rank, bcount, total;
  explicit DensifyLayout(int64_t num) {
    const size_t n = (size_t)(num > 0 ? num : 1);
    const size_t nb = (n + kDensBlock - 1) / kDensBlock;
    size_t o = 0;
    cls = o;    o = align256(o + sizeof(uint32_t) * n);
    tot = o;    o = align256(o + sizeof(uint4) + kAlignSlack);
    src = o;    o = align256(o + sizeof(uint32_t) * 3 * n);
    rank = o;   o = align256(o + sizeof(uint32_t) * 3 * n);
    bcount = o; o = align256(o + sizeof(uint4) * nb + kAlignSlack);
    total = o;
  }
};

}  // namespace cfgs

using namespace cfgs;

extern "C" int cfgs_gaussian_adam(int32_t num_groups, float* const* params, const float* const* grads,
                                  float* const* exp_avg, float* const* exp_avg_sq, const int64_t* numel,
                                  const double* lr, double beta1, double beta2, double eps, int64_t step,
                                  void* stream) {
  if (num_groups <= 0 || num_groups > kMaxAdamGroups || !params || !grads || !exp_avg || !exp_avg_sq || !numel ||
      !lr || step < 1)
    return CFGS_ERR_INVALID_ARGUMENT;
  AdamGroups a{};
  a.count = num_groups;
  // torch multi-tensor Adam: Python-float bias corrections, float32 operands
  const double bc1 = 1.0 - std::pow(beta1, (double)step);
  const double bc2 = 1.0 - std::pow(beta2, (double)step);
  a.w1 = (float)(1.0 - beta1);
  a.b2 = (float)beta2;
  a.w2 = (float)(1.0 - beta2);
  int64_t off = 0;
  for (int k = 0; k < num_groups; ++k) {
    if (numel[k] < 0 || (numel[k] > 0 && (!params[k] || !grads[k] || !exp_avg[k] || !exp_avg_sq[k])))
      return CFGS_ERR_INVALID_ARGUMENT;
    a.p[k] = params[k];
    a.g[k] = grads[k];
    a.m[k] = exp_avg[k];
    a.v[k] = exp_avg_sq[k];
    a.begin[k] = off;
    a.numel[k] = numel[k];
    off += (numel[k] + 3) / 4;
    a.step_size[k] = (float)(-(lr[k] / bc1));
    a.bc2_sqrt[k] = (float)std::sqrt(bc2);
    a.eps[k] = (float)eps;
  }
  a.begin[num_groups] = off;
  if (off == 0) return CFGS_OK;
  k_gaussian_adam<<<div_up(off, 256), 256, 0, (cudaStream_t)stream>>>(a);
  CFGS_CHECK_LAUNCH(0, stream);
  return CFGS_OK;
}

extern "C" int cfgs_densify_stats(int64_t num_gaussians, const int32_t* radii, const float* grad_means2D,
                                  float* grad_accum, float* denom, void* stream) {
  if (num_gaussians < 0 || (num_gaussians > 0 && (!radii || !grad_means2D || !grad_accum || !denom)))
    return CFGS_ERR_INVALID_ARGUMENT;
  if (num_gaussians == 0) return CFGS_OK;
  k_densify_stats<<<div_up(num_gaussians, 256), 256, 0, (cudaStream_t)stream>>>(num_gaussians, radii, grad_means2D,
                                                                                 grad_accum, denom);
  CFGS_CHECK_LAUNCH(0, stream);
  return CFGS_OK;
}

extern "C" size_t cfgs_densify_workspace_bytes(int64_t num_gaussians) {
  return num_gaussians < 0 ? 0 : DensifyLayout(num_gaussians).total;
}

extern "C" int cfgs_densify_plan(int64_t num_gaussians, const float* grad_accum, const float* denom,
                                 const float* scaling, const float* opacity, float max_grad, float min_opacity,
                                 float extent, float percent_dense, int32_t prune_big, void* workspace,
                                 int64_t counts[4], void* stream) {
  if (num_gaussians < 0 || num_gaussians > 0x3fffffffll || !workspace || !counts) return CFGS_ERR_INVALID_ARGUMENT;
  if (num_gaussians > 0 && (!grad_accum || !denom || !scaling || !opacity)) return CFGS_ERR_INVALID_ARGUMENT;
  for (int b = 0; b < 4; ++b) counts[b] = 0;
  if (num_gaussians == 0) return CFGS_OK;
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t n = num_gaussians;
  const DensifyLayout L(n);
  char* w = static_cast<char*>(workspace);
  uint32_t* cls = reinterpret_cast<uint32_t*>(w + L.cls);
  uint4* tot = aligned16<uint4>(w + L.tot);
  uint4* bcount = aligned16<uint4>(w + L.bcount);
  const int nb = div_up(n, kDensBlock);
  DensifyParams d{max_grad, min_opacity, extent, percent_dense, prune_big};
  k_densify_classify<<<nb, kDensBlock, 0, st>>>(n, grad_accum, denom, scaling, opacity, d, cls, bcount);
  k_densify_prefix<<<1, kDensBlock, 0, st>>>(nb, bcount, tot);
  k_densify_map<<<nb, kDensBlock, 0, st>>>(n, cls, bcount, tot, reinterpret_cast<uint32_t*>(w + L.src),
                                           reinterpret_cast<uint32_t*>(w + L.rank));
  uint32_t h[4];
  if (cudaMemcpyAsync(h, tot, sizeof(h), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess)
    return CFGS_ERR_LAUNCH;
  // kept originals, kept clones, split points, kept children per copy
  for (int b = 0; b < 4; ++b) counts[b] = h[b];
  return CFGS_OK;
}

// Writes parameter arrays of the new model from the row map cfgs_densify_plan left in
// `workspace`: rows = counts[0] + counts[1] + 2 counts[3].
// role 0: plain parameter (copied), 1: Adam moment (zero for new rows), 2: xyz, 3: scaling
// (children computed), z = standard-normal draws [2][counts[2]][3] for roles 2 and 3.
extern "C" int cfgs_densify_write_many(int64_t num_gaussians, void* workspace, const int64_t counts[4],
                                       int32_t num_arrays, const int32_t* widths, const float* const* in,
                                       float* const* out, const int32_t* roles, const float* xyz,
                                       const float* scaling, const float* rotation, const float* z, void* stream) {
  if (num_gaussians <= 0 || !workspace || !counts || num_arrays <= 0 || num_arrays > kGatherArrays || !widths || !in ||
      !out || !roles)
    return CFGS_ERR_INVALID_ARGUMENT;
  const int64_t n = num_gaussians;
  for (int b = 0; b < 4; ++b)
    if (counts[b] < 0 || counts[b] > n) return CFGS_ERR_INVALID_ARGUMENT;
  const int64_t first_child = counts[0] + counts[1], rows = first_child + 2 * counts[3];
  if (rows > 3 * n) return CFGS_ERR_INVALID_ARGUMENT;
  GatherArgs a{};
  a.count = num_arrays;
  int64_t blocks = 0;
  float *out_xyz = nullptr, *out_scaling = nullptr;
  for (int k = 0; k < num_arrays; ++k) {
    if (widths[k] <= 0 || !in[k] || !out[k] || roles[k] < 0 || roles[k] > 3) return CFGS_ERR_INVALID_ARGUMENT;
    if (roles[k] >= 2) {
      if (!xyz || !scaling || !rotation || (counts[3] > 0 && !z) || widths[k] != 3) return CFGS_ERR_INVALID_ARGUMENT;
      float*& dst = roles[k] == 2 ? out_xyz : out_scaling;
      if (dst) return CFGS_ERR_INVALID_ARGUMENT;  // one array per computed role
      dst = out[k];
    }
    a.in[k] = in[k];
    a.out[k] = out[k];
    a.width[k] = widths[k];
    a.zero_new[k] = roles[k] == 1;
    a.rows[k] = roles[k] >= 2 ? first_child : rows;
    const int br = kGatherFloats / widths[k];
    a.block_rows[k] = br < 1 ? 1 : (br > kGatherRows ? kGatherRows : br);
    a.first_block[k] = (uint32_t)blocks;
    blocks += (a.rows[k] + a.block_rows[k] - 1) / a.block_rows[k];
    if (blocks > 0x7fffffffll) return CFGS_ERR_TOO_LARGE;
  }
  a.first_block[num_arrays] = (uint32_t)blocks;
  cudaStream_t st = (cudaStream_t)stream;
  const DensifyLayout L(n);
  char* w = static_cast<char*>(workspace);
  const uint32_t* src = reinterpret_cast<const uint32_t*>(w + L.src);
  if (blocks > 0) k_densify_gather<<<(unsigned)blocks, kGatherThreads, 0, st>>>(a, counts[0], src);
  if ((out_xyz || out_scaling) && counts[3] > 0)
    k_densify_children<<<div_up(2 * counts[3], 256), 256, 0, st>>>(
        first_child, counts[3], src, reinterpret_cast<const uint32_t*>(w + L.rank), (uint32_t)counts[2], xyz, scaling,
        rotation, z, out_xyz, out_scaling);
  CFGS_CHECK_LAUNCH(0, st);
  return CFGS_OK;
}

extern "C" int cfgs_densify_write(int64_t num_gaussians, void* workspace, const int64_t counts[4], int32_t width,
                                  const float* in, float* out, int32_t role, const float* xyz, const float* scaling,
                                  const float* rotation, const float* z, void* stream) {
  return cfgs_densify_write_many(num_gaussians, workspace, counts, 1, &width, &in, &out, &role, xyz, scaling, rotation,
                                 z, stream);
}
