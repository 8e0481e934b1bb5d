// Local-Gaussian initialisation of a CF-3DGS frame (the steps before each pose solve,
// trainer/trainer.py:489-512 and scene/gaussian_model_cf.py:175-210):
//   - depth -> camera-space points: kornia depth_to_3d(normalize_points=False), i.e.
//     ((u - cx) / fx * d, (v - cy) / fy * d, d) at pixel (u, v);
//   - voxel down-sampling: Open3D voxel_down_sample — voxel index
//     floor((p - (min - s/2)) / s) in float64, each voxel's points and colours averaged
//     in float64 in input order; here the voxels come out sorted by their index;
//   - initial scales: simple-knn distCUDA2 — per point the mean squared distance to its
//     three nearest other points (missing neighbours count as FLT_MAX).
// kornia, Open3D and simple-knn are unpinned dependencies of the reference
// (requirements.txt; .gitmodules:1-3); their published algorithms are restated.
//
// kNN search: points sorted by Morton code, cut into boxes of 32 consecutive points and
// super-boxes of 32 boxes, each with its bounding box. A warp takes one box, a lane per
// query. It seeds the queries' best three from the box itself, then tests 32 super-boxes,
// and the 32 boxes of a super-box that may matter, at a time (one per lane, against the
// warp's own box and its worst third-best); a box that can still beat some lane's third-best
// (with a 1e-5 relative margin against rounding) is staged in shared memory, where every
// lane checks its 32 points. The result is the exact three smallest squared distances.
#include <cfloat>
#include <cmath>
#include <cstring>

#include "cfgs_internal.cuh"
#include "kernels.cuh"

namespace cfgs {

constexpr int kKnnBox = 32;
constexpr int kKnnSuper = 32;  // boxes per super-box
constexpr float kKnnMargin = 1.0f + 1e-5f;

// Squared distance with one fixed rounding sequence (the oracle performs the same).
__host__ __device__ __forceinline__ float dist2_ref(float ax, float ay, float az, float bx, float by, float bz) {
  const float dx = ax - bx, dy = ay - by, dz = az - bz;
  return fmaf(dz, dz, fmaf(dy, dy, dx * dx));
}

// ---- depth -> points ---------------------------------------------------------------
__global__ void __launch_bounds__(256) k_depth_to_points(int H, int W, const float* __restrict__ depth, float fx,
                                                         float fy, float cx, float cy, float* __restrict__ xyz) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (int64_t)H * W) return;
  const int u = (int)(i % W), v = (int)(i / W);
  const float d = depth[i];
  xyz[3 * i + 0] = __fmul_rn(__fdiv_rn(__fsub_rn((float)u, cx), fx), d);
  xyz[3 * i + 1] = __fmul_rn(__fdiv_rn(__fsub_rn((float)v, cy), fy), d);
  xyz[3 * i + 2] = d;
}

// ---- bounds ---------------------------------------------------------------------------
// Floats as unsigned integers of the same order, so that blocks combine minima by atomics.
__host__ __device__ __forceinline__ uint32_t ordered_bits(uint32_t u) { return u & 0x80000000u ? ~u : u | 0x80000000u; }
__host__ __device__ __forceinline__ uint32_t unordered_bits(uint32_t o) {
  return o & 0x80000000u ? o & 0x7fffffffu : ~o;
}

// Per-axis bounds of n points, in out[0..5]: ordered minima of x, y, z and of -x, -y, -z
// (set to all ones before the launch). NaN coordinates are passed over. One block over all
// points took 34 us for 230,400 of them; up to 304 blocks take 4.4 us.
constexpr int kBoundsThreads = 256;
constexpr int kBoundsMaxBlocks = 2 * 152;

__global__ void __launch_bounds__(kBoundsThreads) k_bounds(int64_t n, const float* __restrict__ xyz,
                                                           uint32_t* __restrict__ out) {
  __shared__ float sh[6][kBoundsThreads / 32];
  float v[6] = {FLT_MAX, FLT_MAX, FLT_MAX, FLT_MAX, FLT_MAX, FLT_MAX};
  const int64_t stride = (int64_t)gridDim.x * kBoundsThreads;
#pragma unroll 2
  for (int64_t i = (int64_t)blockIdx.x * kBoundsThreads + threadIdx.x; i < n; i += stride) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const float c = xyz[3 * i + a];
      v[a] = fminf(v[a], c);
      v[3 + a] = fminf(v[3 + a], -c);
    }
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int a = 0; a < 6; ++a) {
    float x = v[a];
    for (int o = 16; o > 0; o >>= 1) x = fminf(x, __shfl_xor_sync(0xffffffffu, x, o));
    if (lane == 0) sh[a][warp] = x;
  }
  __syncthreads();
  if (threadIdx.x < 6) {
    float x = sh[threadIdx.x][0];
    for (int w = 1; w < kBoundsThreads / 32; ++w) x = fminf(x, sh[threadIdx.x][w]);
    atomicMin(out + threadIdx.x, ordered_bits(__float_as_uint(x)));
  }
}

// Axis a's bounds (min, max) from k_bounds' output.
__device__ __forceinline__ float2 axis_bounds(const uint32_t* b, int a) {
  return make_float2(__uint_as_float(unordered_bits(b[a])), -__uint_as_float(unordered_bits(b[3 + a])));
}

static bool launch_bounds_pass(int64_t n, const float* xyz, uint32_t* bounds, cudaStream_t st) {
  if (cudaMemsetAsync(bounds, 0xff, 6 * sizeof(uint32_t), st) != cudaSuccess) return false;
  const int64_t blocks = (n + 4 * kBoundsThreads - 1) / (4 * kBoundsThreads);
  k_bounds<<<(int)(blocks < kBoundsMaxBlocks ? blocks : kBoundsMaxBlocks), kBoundsThreads, 0, st>>>(n, xyz, bounds);
  return true;
}

// ---- voxel down-sampling -----------------------------------------------------------
// a / b in float64, correctly rounded, from r = 1 / b correctly rounded: one Newton step on
// the quotient (Markstein, "Computation of elementary functions on the IBM RISC System/6000
// processor", 1990, theorem on division from a correctly rounded reciprocal). Three
// operations instead of a division's twenty-odd on a float64 pipe of about two operations
// per cycle and SM. Non-finite quotients take the division itself.
__device__ __forceinline__ double divide_by(double a, double b, double r) {
  const double q = a * r;
  return isfinite(q) ? fma(fma(-q, b, a), r, q) : a / b;
}

struct VoxelGrid {
  double min_x, min_y, min_z, size, inv_size;
  uint64_t ny, nz;  // voxels along y and z (key = (ix ny + iy) nz + iz)
};

__global__ void __launch_bounds__(256) k_voxel_keys(int64_t n, const float* __restrict__ xyz, VoxelGrid g,
                                                    uint32_t* __restrict__ key_lo, uint32_t* __restrict__ key_hi,
                                                    uint32_t* __restrict__ idx) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double rx = divide_by((double)xyz[3 * i + 0] - g.min_x, g.size, g.inv_size);
  const double ry = divide_by((double)xyz[3 * i + 1] - g.min_y, g.size, g.inv_size);
  const double rz = divide_by((double)xyz[3 * i + 2] - g.min_z, g.size, g.inv_size);
  const uint64_t k = ((uint64_t)floor(rx) * g.ny + (uint64_t)floor(ry)) * g.nz + (uint64_t)floor(rz);
  key_lo[i] = (uint32_t)k;
  if (key_hi) key_hi[i] = (uint32_t)(k >> 32);
  if (idx) idx[i] = (uint32_t)i;
}

__global__ void __launch_bounds__(256) k_gather_u32(int64_t n, const uint32_t* __restrict__ src,
                                                    const uint32_t* __restrict__ idx, uint32_t* __restrict__ dst) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[i] = src[idx[i]];
}

// The voxels are the runs of equal keys in sorted order. A run's number is the count of
// run heads before it: heads per block of 512 positions, an exclusive prefix of those
// (one block), then ballots inside the block. The scan by one block over all positions that
// this replaces took 190 us for 230,400 points; count and prefix take 6.9 us.
constexpr int kVoxelBlock = 512;

__device__ __forceinline__ bool voxel_head(int64_t i, int64_t n, const uint32_t* __restrict__ lo,
                                           const uint32_t* __restrict__ hi) {
  if (i >= n) return false;
  if (i == 0 || lo[i] != lo[i - 1]) return true;
  return hi && hi[i] != hi[i - 1];
}

__global__ void __launch_bounds__(kVoxelBlock) k_voxel_count(int64_t n, const uint32_t* __restrict__ lo,
                                                             const uint32_t* __restrict__ hi,
                                                             uint32_t* __restrict__ bcount) {
  const int64_t i = (int64_t)blockIdx.x * kVoxelBlock + threadIdx.x;
  const int c = __syncthreads_count(voxel_head(i, n, lo, hi));
  if (threadIdx.x == 0) bcount[blockIdx.x] = (uint32_t)c;
}

__global__ void __launch_bounds__(kVoxelBlock) k_voxel_prefix(int nblocks, uint32_t* __restrict__ bcount,
                                                              uint32_t* __restrict__ total) {
  __shared__ uint32_t sh[kVoxelBlock / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t carry = 0;
  for (int base = 0; base < nblocks; base += kVoxelBlock) {
    const int j = base + threadIdx.x;
    const uint32_t v = j < nblocks ? bcount[j] : 0u;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) sh[warp] = x;
    __syncthreads();
    uint32_t before = carry;
    for (int w = 0; w < kVoxelBlock / 32; ++w) {
      const uint32_t t = sh[w];
      if (w < warp) before += t;
      carry += t;
    }
    if (j < nblocks) bcount[j] = before + x - v;
    __syncthreads();
  }
  if (threadIdx.x == 0) *total = carry;
}

// Every voxel's points and colours summed in float64 in input order (the sort is stable),
// averaged and rounded to float. Bound by the float64 pipe, which takes about 16 cycles of
// its SM per warp instruction however few lanes take part, so only the runs of two or more
// points go through it, packed into whole warps; a single point is its own average. The
// block's 512 positions are gathered to shared memory first; a run that goes on into the
// next block reads the rest from memory, one point ahead, which wants 40 registers and so
// three blocks of 512 per SM (two of 1024 leave 32). 230,400 points in 161,225 voxels: 62 us
// with a thread at every run's head -> 20 us. Long runs, whole calls: 20,000 points of which
// two thirds share a voxel 5.7 -> 5.5 ms, 230,400 in 8 voxels 14.3 -> 11.6 ms (6.9 and 17.1 with
// the rest of a run read key by key).
__global__ void __launch_bounds__(kVoxelBlock, 3) k_voxel_average(int64_t n, const uint32_t* __restrict__ lo,
                                                               const uint32_t* __restrict__ hi,
                                                               const uint32_t* __restrict__ bprefix,
                                                               const uint32_t* __restrict__ order,
                                                               const float* __restrict__ xyz,
                                                               const float* __restrict__ rgb,
                                                               float* __restrict__ out_xyz,
                                                               float* __restrict__ out_rgb) {
  __shared__ uint32_t s_run[kVoxelBlock];    // runs of two or more: start | end << 16
  __shared__ uint32_t s_voxel[kVoxelBlock];  // and their voxel numbers
  __shared__ uint32_t s_runs;
  __shared__ float s_val[6][kVoxelBlock];
  __shared__ uint32_t s_heads[kVoxelBlock / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t i = (int64_t)blockIdx.x * kVoxelBlock + threadIdx.x;
  const bool head = voxel_head(i, n, lo, hi);
  if (i < n) {
    const size_t j = order[i];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      s_val[a][threadIdx.x] = xyz[3 * j + a];
      if (rgb) s_val[3 + a][threadIdx.x] = rgb[3 * j + a];
    }
  }
  const unsigned m = __ballot_sync(0xffffffffu, head);
  if (lane == 0) s_heads[warp] = m;
  if (threadIdx.x == 0) s_runs = 0;
  __syncthreads();
  const int64_t first = (int64_t)blockIdx.x * kVoxelBlock;
  const int here = (int)min((int64_t)kVoxelBlock, n - first);
  if (head) {
    uint32_t v = bprefix[blockIdx.x] + (uint32_t)__popc(m & ((1u << lane) - 1u));
    for (int w = 0; w < warp; ++w) v += (uint32_t)__popc(s_heads[w]);
    // the run's end in this block: the next head, or the block's last position
    int end = here;
    const unsigned later = lane < 31 ? m >> (lane + 1) : 0u;
    if (later) {
      end = (int)threadIdx.x + __ffs(later);
    } else {
      for (int w = warp + 1; w < kVoxelBlock / 32; ++w)
        if (s_heads[w]) {
          end = 32 * w + __ffs(s_heads[w]) - 1;
          break;
        }
    }
    const bool goes_on = end == here && first + here < n && !voxel_head(first + here, n, lo, hi);
    if (end - (int)threadIdx.x > 1 || goes_on) {
      const uint32_t at = atomicAdd(&s_runs, 1u);
      s_run[at] = threadIdx.x | ((uint32_t)end << 16);
      s_voxel[at] = v;
    } else {
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        out_xyz[3 * (size_t)v + a] = __fadd_rn(s_val[a][threadIdx.x], 0.0f);  // 0 + x, as the sums start
        if (rgb && out_rgb) out_rgb[3 * (size_t)v + a] = __fadd_rn(s_val[3 + a][threadIdx.x], 0.0f);
      }
    }
  }
  __syncthreads();
  if (threadIdx.x >= s_runs) return;
  const int start = (int)(s_run[threadIdx.x] & 0xffffu), end = (int)(s_run[threadIdx.x] >> 16);
  const size_t v = s_voxel[threadIdx.x];
  double s[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll 2
  for (int t = start; t < end; ++t) {
#pragma unroll
    for (int a = 0; a < 3; ++a) s[a] += (double)s_val[a][t];
    if (rgb) {
#pragma unroll
      for (int a = 0; a < 3; ++a) s[3 + a] += (double)s_val[3 + a][t];
    }
  }
  int64_t k = first + end;
  if (end == here) {
    // its end by steps that double, then halve (the keys are sorted), so that the sums below
    // know their count and load ahead
    const uint32_t klo = lo[first + start], khi = hi ? hi[first + start] : 0u;
    auto inside = [&](int64_t p) { return p < n && lo[p] == klo && (!hi || hi[p] == khi); };
    int64_t last = k - 1, step = 1;
    while (inside(last + step)) {
      last += step;
      step *= 2;
    }
    for (step /= 2; step > 0; step /= 2)
      if (inside(last + step)) last += step;
    // the next point's values and the one after's index are on their way while one is added
    auto load = [&](uint32_t p, float (&v)[6]) {
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        v[a] = xyz[3 * (size_t)p + a];
        v[3 + a] = rgb ? rgb[3 * (size_t)p + a] : 0.f;
      }
    };
    float ahead[6];
    load(order[min(k, last)], ahead);
    uint32_t next = order[min(k + 1, last)];
#pragma unroll 1
    for (; k <= last; ++k) {
      float own[6];
#pragma unroll
      for (int a = 0; a < 6; ++a) own[a] = ahead[a];
      load(next, ahead);
      next = order[min(k + 2, last)];
#pragma unroll
      for (int a = 0; a < 6; ++a) s[a] += (double)own[a];
    }
  }
  const double count = (double)(k - (first + start)), inv = 1.0 / count;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    out_xyz[3 * v + a] = (float)divide_by(s[a], count, inv);
    if (rgb && out_rgb) out_rgb[3 * v + a] = (float)divide_by(s[3 + a], count, inv);
  }
}

// ---- kNN -------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t spread10(uint32_t x) {
  x &= 0x3ffu;
  x = (x | (x << 16)) & 0x030000ffu;
  x = (x | (x << 8)) & 0x0300f00fu;
  x = (x | (x << 4)) & 0x030c30c3u;
  x = (x | (x << 2)) & 0x09249249u;
  return x;
}

__global__ void __launch_bounds__(256) k_morton(int64_t n, const float* __restrict__ xyz,
                                                const uint32_t* __restrict__ bounds, uint32_t* __restrict__ code,
                                                uint32_t* __restrict__ idx) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t q[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float2 b = axis_bounds(bounds, a);
    const float lo = b.x, ext = b.y - lo;
    const float t = ext > 0.f ? (xyz[3 * i + a] - lo) / ext : 0.f;
    q[a] = (uint32_t)fminf(fmaxf(t * 1024.f, 0.f), 1023.f);
  }
  code[i] = spread10(q[0]) | (spread10(q[1]) << 1) | (spread10(q[2]) << 2);
  idx[i] = (uint32_t)i;
}

// Sorted points as float4 (x, y, z, original index bits), the bounding boxes of 32
// consecutive points (one warp each) and of 32 boxes (one block each). Box b = (min.xyz,
// max.xyz) in two float4.
__global__ void __launch_bounds__(kKnnBox* kKnnSuper) k_gather_boxes(int64_t n, const float* __restrict__ xyz,
                                                                      const uint32_t* __restrict__ order,
                                                                      float4* __restrict__ pts,
                                                                      float4* __restrict__ box,
                                                                      float4* __restrict__ sup) {
  __shared__ float s_box[6][kKnnSuper];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t i = (int64_t)blockIdx.x * (kKnnBox * kKnnSuper) + threadIdx.x;
  float v[6] = {FLT_MAX, FLT_MAX, FLT_MAX, FLT_MAX, FLT_MAX, FLT_MAX};  // minima of p and of -p
  if (i < n) {
    const uint32_t j = order[i];
    const float p[3] = {xyz[3 * (size_t)j], xyz[3 * (size_t)j + 1], xyz[3 * (size_t)j + 2]};
    pts[i] = make_float4(p[0], p[1], p[2], __uint_as_float(j));
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      v[a] = fminf(v[a], p[a]);
      v[3 + a] = fminf(v[3 + a], -p[a]);
    }
  }
#pragma unroll
  for (int a = 0; a < 6; ++a) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[a] = fminf(v[a], __shfl_xor_sync(0xffffffffu, v[a], o));
    if (lane == 0) s_box[a][warp] = v[a];
  }
  const int64_t b = (int64_t)blockIdx.x * kKnnSuper + warp;
  if (lane == 0 && b * kKnnBox < n) {
    box[2 * b] = make_float4(v[0], v[1], v[2], 0.f);
    box[2 * b + 1] = make_float4(-v[3], -v[4], -v[5], 0.f);
  }
  __syncthreads();
  if (warp != 0) return;
#pragma unroll
  for (int a = 0; a < 6; ++a) {
    v[a] = s_box[a][lane];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[a] = fminf(v[a], __shfl_xor_sync(0xffffffffu, v[a], o));
  }
  if (lane == 0) {
    sup[2 * (int64_t)blockIdx.x] = make_float4(v[0], v[1], v[2], 0.f);
    sup[2 * (int64_t)blockIdx.x + 1] = make_float4(-v[3], -v[4], -v[5], 0.f);
  }
}

// Squared distance between two boxes (0 where they meet), a lower bound of every pair of
// members'; a point is a box with lo = hi.
__device__ __forceinline__ float box_dist2(const float4& alo, const float4& ahi, const float4& blo, const float4& bhi) {
  const float gx = fmaxf(fmaxf(blo.x - ahi.x, alo.x - bhi.x), 0.f);
  const float gy = fmaxf(fmaxf(blo.y - ahi.y, alo.y - bhi.y), 0.f);
  const float gz = fmaxf(fmaxf(blo.z - ahi.z, alo.z - bhi.z), 0.f);
  return fmaf(gz, gz, fmaf(gy, gy, gx * gx));
}

// The three smallest values so far, b0 <= b1 <= b2 (d < b2: a NaN never enters).
__device__ __forceinline__ void best3_insert(float (&b)[3], float d) {
  if (d < b[2]) {
    b[2] = fminf(b[2], fmaxf(b[1], d));
    b[1] = fminf(b[1], fmaxf(b[0], d));
    b[0] = fminf(b[0], d);
  }
}

// Bound by the distance checks' issue. One thread per query with its own divergent
// traversal waited on one dependent load after another (161,225 points of a 640x360 frame:
// 1671 us); the shared traversal reads each box once per warp: 135 us. Most warps were then
// done after 60; a few whose 32 points span a jump of the curve test hundreds of boxes (892
// of 5,039) one after another. So box tests go four at a time from shared memory, the next
// super-box is loaded ahead, and a box's distances are formed eight at a time before any is
// compared: 105 us. (Tests of parts of the wide box instead: 137; the scan unrolled into each
// of the four tests: 152, instruction fetch.)
constexpr int kKnnWarps = 8, kKnnBatch = 8, kKnnTests = 4;

__global__ void __launch_bounds__(32 * kKnnWarps) k_knn3(int64_t n, const float4* __restrict__ pts,
                                                         const float4* __restrict__ box,
                                                         const float4* __restrict__ sup, float* __restrict__ out) {
  static_assert(kKnnBox == 32 && kKnnSuper == 32, "a lane per query, box and super-box");
  __shared__ float4 s_pts[kKnnWarps][kKnnBox];
  __shared__ float4 s_box[kKnnWarps][kKnnSuper][2];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t nbox = (n + kKnnBox - 1) / kKnnBox;
  const int64_t nsup = (nbox + kKnnSuper - 1) / kKnnSuper;
  const int64_t own = (int64_t)blockIdx.x * kKnnWarps + warp;
  if (own >= nbox) return;
  const int64_t i = own * kKnnBox + lane;
  const bool active = i < n;
  const float4 q = active ? pts[i] : make_float4(0.f, 0.f, 0.f, 0.f);
  const float4 own_lo = box[2 * own], own_hi = box[2 * own + 1];
  float b[3] = {FLT_MAX, FLT_MAX, FLT_MAX};
  if (!active) b[0] = b[1] = b[2] = -1.0f;  // nothing is nearer

  auto stage = [&](int64_t bx) {  // the box's points; slots past the last point are infinitely far
    const int64_t k = bx * kKnnBox + lane;
    __syncwarp();
    s_pts[warp][lane] = k < n ? pts[k] : make_float4(INFINITY, 0.f, 0.f, 0.f);
    __syncwarp();
  };
  // the staged points, but the one at `skip`, kKnnBatch distances at a time: most batches of
  // another box improve no lane's three
  auto scan = [&](int skip) {
#pragma unroll
    for (int j = 0; j < kKnnBox; j += kKnnBatch) {
      float d[kKnnBatch];
#pragma unroll
      for (int k = 0; k < kKnnBatch; ++k) {
        const float4 p = s_pts[warp][j + k];
        d[k] = dist2_ref(q.x, q.y, q.z, p.x, p.y, p.z);
        if (j + k == skip) d[k] = INFINITY;
      }
      float least = d[0];
#pragma unroll
      for (int k = 1; k < kKnnBatch; ++k) least = fminf(least, d[k]);
      if (least < b[2]) {
#pragma unroll
        for (int k = 0; k < kKnnBatch; ++k) best3_insert(b, d[k]);
      }
    }
  };
  stage(own);
  scan(lane);
  auto worst = [&]() {  // the warp's largest third-best, with the margin
    return __uint_as_float(__reduce_max_sync(0xffffffffu, active ? __float_as_uint(b[2]) : 0u)) * kKnnMargin;
  };
  auto load_box = [&](int64_t sb, float4& lo, float4& hi) {  // this lane's box of super-box sb
    const int64_t bx = sb * kKnnSuper + lane;
    if (bx < nbox) {
      lo = box[2 * bx];
      hi = box[2 * bx + 1];
    }
  };
  auto visit = [&](int64_t sb, const float4& lo, const float4& hi, float bound) {  // the boxes of super-box sb
    const int64_t bx = sb * kKnnSuper + lane;
    const bool may = bx < nbox && bx != own && !(box_dist2(own_lo, own_hi, lo, hi) > bound);
    unsigned todo = __ballot_sync(0xffffffffu, may);
    if (!todo) return;
    __syncwarp();
    s_box[warp][lane][0] = lo;
    s_box[warp][lane][1] = hi;
    __syncwarp();
    while (todo) {
      unsigned need = 0;
#pragma unroll
      for (int k = 0; k < kKnnTests; ++k) {
        const unsigned bit = todo & (0u - todo);
        const int l = max(__ffs(todo) - 1, 0);
        todo ^= bit;
        if (__any_sync(0xffffffffu, !(box_dist2(q, q, s_box[warp][l][0], s_box[warp][l][1]) > b[2] * kKnnMargin)))
          need |= bit;
      }
      while (need) {
        const int l = __ffs(need) - 1;
        need &= need - 1;
        stage(sb * kKnnSuper + l);
        scan(-1);
      }
    }
  };
  // its own super-box first, then those within the bound. The next one's boxes are on their
  // way while one is visited.
  const int64_t own_sup = own / kKnnSuper;
  float bound = worst();
  for (int64_t s0 = -32; s0 < nsup; s0 += 32) {
    int64_t base = own_sup;
    unsigned todo = 1u;
    if (s0 >= 0) {
      base = s0;
      const int64_t sb = s0 + lane;
      todo = __ballot_sync(0xffffffffu, sb < nsup && sb != own_sup &&
                                            !(box_dist2(own_lo, own_hi, sup[2 * sb], sup[2 * sb + 1]) > bound));
    }
    float4 lo, hi, next_lo = own_lo, next_hi = own_hi;
    if (todo) load_box(base + __ffs(todo) - 1, next_lo, next_hi);
    while (todo) {
      const int l = __ffs(todo) - 1;
      todo &= todo - 1;
      lo = next_lo;
      hi = next_hi;
      if (todo) load_box(base + __ffs(todo) - 1, next_lo, next_hi);
      visit(base + l, lo, hi, bound);
      bound = worst();
    }
  }
  if (active) out[__float_as_uint(q.w)] = ((b[0] + b[1]) + b[2]) / 3.0f;
}

// ---- initial Gaussians -----------------------------------------------------------------
// The parameters of create_from_pcd (scene/gaussian_model_cf.py:175-210) but the zero
// higher SH bands: positions and DC colours copied, log-scales from the neighbour
// distances, identity rotations, one opacity.
__global__ void __launch_bounds__(256) k_init_gaussians(int64_t n, const float* __restrict__ xyz,
                                                        const float* __restrict__ dc, const float* __restrict__ dist2,
                                                        float opacity, float* __restrict__ out_xyz,
                                                        float* __restrict__ out_dc, float* __restrict__ out_scaling,
                                                        float4* __restrict__ out_rotation,
                                                        float* __restrict__ out_opacity) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float d = dist2[i];
  const float s = logf(sqrtf(d != d ? d : fmaxf(d, 0.0000001f)));
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    out_xyz[3 * i + a] = xyz[3 * i + a];
    out_dc[3 * i + a] = dc[3 * i + a];
    out_scaling[3 * i + a] = s;
  }
  out_rotation[i] = make_float4(1.f, 0.f, 0.f, 0.f);
  out_opacity[i] = opacity;
}

// ---- workspaces ----------------------------------------------------------------------
struct PcLayout {
  size_t keys, vals, extra, extra2, bounds, counts, totals, pts, box, sup, total;
  explicit PcLayout(int64_t n) {
    const size_t c = pingpong_stride(n);
    const int64_t nbox = (n + kKnnBox - 1) / kKnnBox;
    const int64_t nsup = (nbox + kKnnSuper - 1) / kKnnSuper;
    size_t o = 0;
    keys = o;   o = align256(o + sizeof(uint32_t) * 2 * c);
    vals = o;   o = align256(o + sizeof(uint32_t) * 2 * c);
    extra = o;  o = align256(o + sizeof(uint32_t) * (c + 1));
    extra2 = o; o = align256(o + sizeof(uint32_t) * (c + 1));
    bounds = o; o = align256(o + sizeof(float) * 8);
    counts = o; o = align256(o + sizeof(uint32_t) * kSortDigits * (size_t)sort_chunks(n, kTileChunk));
    totals = o; o = align256(o + sizeof(uint32_t) * kSortDigits * kMaxTilePasses);
    pts = o;    o = align256(o + sizeof(float4) * (size_t)(n > 0 ? n : 1));
    box = o;    o = align256(o + 2 * sizeof(float4) * (size_t)(nbox > 0 ? nbox : 1));
    sup = o;    o = align256(o + 2 * sizeof(float4) * (size_t)(nsup > 0 ? nsup : 1));
    total = o;
  }
};

}  // namespace cfgs

using namespace cfgs;

extern "C" int cfgs_depth_to_points(int32_t height, int32_t width, const float* depth, float fx, float fy, float cx,
                                    float cy, float* xyz, void* stream) {
  if (height <= 0 || width <= 0 || !depth || !xyz || (int64_t)height * width > 0x7fffffffll)
    return CFGS_ERR_INVALID_ARGUMENT;
  const int64_t n = (int64_t)height * width;
  k_depth_to_points<<<div_up(n, 256), 256, 0, (cudaStream_t)stream>>>(height, width, depth, fx, fy, cx, cy, xyz);
  CFGS_CHECK_LAUNCH(0, stream);
  return CFGS_OK;
}

extern "C" size_t cfgs_pointcloud_workspace_bytes(int64_t num_points) {
  return num_points < 0 || num_points > 0x7fffffffll ? 0 : PcLayout(num_points).total;
}

extern "C" int cfgs_knn3_mean_dist2(int64_t num_points, const float* xyz, void* workspace, float* dist2,
                                    void* stream) {
  if (num_points < 0 || num_points > 0x7fffffffll || (num_points > 0 && (!xyz || !workspace || !dist2)))
    return CFGS_ERR_INVALID_ARGUMENT;
  const int64_t n = num_points;
  if (n == 0) return CFGS_OK;
  cudaStream_t st = (cudaStream_t)stream;
  PcLayout L(n);
  char* w = static_cast<char*>(workspace);
  const size_t c = pingpong_stride(n);
  uint32_t* keys[2] = {reinterpret_cast<uint32_t*>(w + L.keys), reinterpret_cast<uint32_t*>(w + L.keys) + c};
  uint32_t* vals[2] = {reinterpret_cast<uint32_t*>(w + L.vals), reinterpret_cast<uint32_t*>(w + L.vals) + c};
  uint32_t* bounds = reinterpret_cast<uint32_t*>(w + L.bounds);
  float4* pts = reinterpret_cast<float4*>(w + L.pts);
  float4* box = reinterpret_cast<float4*>(w + L.box);
  float4* sup = reinterpret_cast<float4*>(w + L.sup);
  if (!launch_bounds_pass(n, xyz, bounds, st)) return CFGS_ERR_LAUNCH;
  // 10 bits an axis, four radix passes. 8 bits would save one (160,000 points evenly spread or
  // on a surface: 10 to 13 us of 186 to 361), but a few far points stretch the bounds, and
  // the codes then no longer part the others (one in a thousand 30 times as far out: 3387 us
  // against 556; 262,144 points 9424 against 1069).
  k_morton<<<div_up(n, 256), 256, 0, st>>>(n, xyz, bounds, keys[0], vals[0]);
  int res = 0;
  int s = sort_pairs(keys, vals, n, 30, reinterpret_cast<uint32_t*>(w + L.counts),
                     reinterpret_cast<uint32_t*>(w + L.totals), st, &res);
  if (s != CFGS_OK) return s;
  const int64_t nbox = (n + kKnnBox - 1) / kKnnBox;
  k_gather_boxes<<<div_up(n, kKnnBox * kKnnSuper), kKnnBox * kKnnSuper, 0, st>>>(n, xyz, vals[res], pts, box, sup);
  k_knn3<<<div_up(nbox, kKnnWarps), 32 * kKnnWarps, 0, st>>>(n, pts, box, sup, dist2);
  CFGS_CHECK_LAUNCH(0, st);
  return CFGS_OK;
}

extern "C" int cfgs_init_gaussians(int64_t num_points, int32_t rest_floats, const float* xyz, const float* dc,
                                   const float* dist2, float opacity, float* out_xyz, float* out_dc, float* out_rest,
                                   float* out_scaling, float* out_rotation, float* out_opacity, void* stream) {
  if (num_points < 0 || num_points > 0x7fffffffll || rest_floats < 0) return CFGS_ERR_INVALID_ARGUMENT;
  if (num_points == 0) return CFGS_OK;
  if (!xyz || !dc || !dist2 || !out_xyz || !out_dc || (rest_floats > 0 && !out_rest) || !out_scaling || !out_rotation ||
      !out_opacity || (reinterpret_cast<uintptr_t>(out_rotation) & 15) != 0)
    return CFGS_ERR_INVALID_ARGUMENT;
  cudaStream_t st = (cudaStream_t)stream;
  if (rest_floats > 0 &&
      cudaMemsetAsync(out_rest, 0, sizeof(float) * (size_t)rest_floats * (size_t)num_points, st) != cudaSuccess)
    return CFGS_ERR_LAUNCH;
  k_init_gaussians<<<div_up(num_points, 256), 256, 0, st>>>(num_points, xyz, dc, dist2, opacity, out_xyz, out_dc,
                                                           out_scaling, reinterpret_cast<float4*>(out_rotation),
                                                           out_opacity);
  CFGS_CHECK_LAUNCH(0, st);
  return CFGS_OK;
}

extern "C" int cfgs_voxel_down_sample(int64_t num_points, const float* xyz, const float* rgb, double voxel_size,
                                      void* workspace, float* out_xyz, float* out_rgb, int64_t* num_voxels,
                                      void* stream) {
  if (num_points < 0 || num_points > 0x7fffffffll || !num_voxels || !(voxel_size > 0.0))
    return CFGS_ERR_INVALID_ARGUMENT;
  if (num_points > 0 && (!xyz || !workspace || !out_xyz || (rgb && !out_rgb))) return CFGS_ERR_INVALID_ARGUMENT;
  *num_voxels = 0;
  const int64_t n = num_points;
  if (n == 0) return CFGS_OK;
  cudaStream_t st = (cudaStream_t)stream;
  PcLayout L(n);
  char* w = static_cast<char*>(workspace);
  const size_t c = pingpong_stride(n);
  uint32_t* keys[2] = {reinterpret_cast<uint32_t*>(w + L.keys), reinterpret_cast<uint32_t*>(w + L.keys) + c};
  uint32_t* vals[2] = {reinterpret_cast<uint32_t*>(w + L.vals), reinterpret_cast<uint32_t*>(w + L.vals) + c};
  uint32_t* extra = reinterpret_cast<uint32_t*>(w + L.extra);
  uint32_t* bounds = reinterpret_cast<uint32_t*>(w + L.bounds);
  uint32_t* counts = reinterpret_cast<uint32_t*>(w + L.counts);
  uint32_t* totals = reinterpret_cast<uint32_t*>(w + L.totals);
  if (!launch_bounds_pass(n, xyz, bounds, st)) return CFGS_ERR_LAUNCH;
  uint32_t ordered[6];
  if (cudaMemcpyAsync(ordered, bounds, sizeof(ordered), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess)
    return CFGS_ERR_LAUNCH;
  float hb[6];  // min xyz, max xyz
  for (int a = 0; a < 6; ++a) {
    const uint32_t u = unordered_bits(ordered[a]);
    std::memcpy(&hb[a], &u, sizeof(u));
    if (a >= 3) hb[a] = -hb[a];
  }
  // Open3D: min bound - s/2; the span must index with int
  VoxelGrid g;
  g.size = voxel_size;
  g.inv_size = 1.0 / voxel_size;
  g.min_x = (double)hb[0] - 0.5 * voxel_size;
  g.min_y = (double)hb[1] - 0.5 * voxel_size;
  g.min_z = (double)hb[2] - 0.5 * voxel_size;
  uint64_t dim[3];
  const double lo[3] = {g.min_x, g.min_y, g.min_z};
  for (int a = 0; a < 3; ++a) {
    const double span = ((double)hb[3 + a] + 0.5 * voxel_size - lo[a]) / voxel_size;
    if (!(span < 2147483647.0)) return CFGS_ERR_TOO_LARGE;
    dim[a] = (uint64_t)std::floor(((double)hb[3 + a] - lo[a]) / voxel_size) + 1;
  }
  g.ny = dim[1];
  g.nz = dim[2];
  const double cells = (double)dim[0] * (double)dim[1] * (double)dim[2];
  if (cells >= 18446744073709551615.0) return CFGS_ERR_TOO_LARGE;
  const bool wide = cells > 4294967295.0;
  // keys[0] = low 32 key bits, extra = high 32 bits (wide grids), vals[0] = input index.
  // Wide keys sort as two stable LSD groups: low halves, then high halves; others by the bits
  // that number the grid's cells.
  int bits = 32;
  if (!wide)
    for (bits = 1; bits < 32 && ((uint64_t)1 << bits) < dim[0] * dim[1] * dim[2];) ++bits;
  uint32_t* extra2 = reinterpret_cast<uint32_t*>(w + L.extra2);
  k_voxel_keys<<<div_up(n, 256), 256, 0, st>>>(n, xyz, g, keys[0], wide ? extra : nullptr, vals[0]);
  int r1 = 0;
  int s = sort_pairs(keys, vals, n, bits, counts, totals, st, &r1);
  if (s != CFGS_OK) return s;
  uint32_t *lo_sorted = keys[r1], *hi_sorted = nullptr, *order = vals[r1];
  if (wide) {
    uint32_t* k2[2] = {keys[r1 ^ 1], keys[r1]};
    uint32_t* v2[2] = {vals[r1], vals[r1 ^ 1]};
    k_gather_u32<<<div_up(n, 256), 256, 0, st>>>(n, extra, vals[r1], k2[0]);  // high halves, round-1 order
    int r2 = 0;
    s = sort_pairs(k2, v2, n, 32, counts, totals, st, &r2);
    if (s != CFGS_OK) return s;
    hi_sorted = k2[r2];
    order = v2[r2];
    k_voxel_keys<<<div_up(n, 256), 256, 0, st>>>(n, xyz, g, extra, nullptr, nullptr);  // low halves by input
    lo_sorted = k2[r2 ^ 1];
    k_gather_u32<<<div_up(n, 256), 256, 0, st>>>(n, extra, order, lo_sorted);
  }
  uint32_t* bcount = extra2;  // run heads per block
  uint32_t* dcount = bounds + 6;
  const int nb = div_up(n, kVoxelBlock);
  k_voxel_count<<<nb, kVoxelBlock, 0, st>>>(n, lo_sorted, hi_sorted, bcount);
  k_voxel_prefix<<<1, kVoxelBlock, 0, st>>>(nb, bcount, dcount);
  k_voxel_average<<<nb, kVoxelBlock, 0, st>>>(n, lo_sorted, hi_sorted, bcount, order, xyz, rgb, out_xyz, out_rgb);
  uint32_t hc = 0;
  if (cudaMemcpyAsync(&hc, dcount, sizeof(hc), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess)
    return CFGS_ERR_LAUNCH;
  *num_voxels = hc;
  CFGS_CHECK_LAUNCH(0, st);
  return CFGS_OK;
}
