// CF-3DGS relative-pose path: SE(3) retraction applied to the Gaussians, the fused
// pose-gradient reduction, and the Adam step on the 6-vector tangent.
//
// Parametrisation (the one lietorch's LieGroupParameter(SE3) gives CFGaussianModel,
// scene/gaussian_model_cf.py:123-133 and :328-340): the optimised tensor is a tangent
// xi = (rho, phi) in R^6, initialised at 0; the pose is X = exp(xi) * I with
// R = exp(phi^) and t = J_l(phi) rho (J_l = SO(3) left Jacobian); positions move as
// p' = R p + t. Covariances are not moved by the reference pose
// (scene/gaussian_model_cf.py:119-121); the rotate_cov form (cov' = R cov R^T) is an
// option of this library.
//
// Gradient. With a left perturbation exp(d) X of the pose, dL/dd = (sum g_i,
// sum p'_i x g_i + w_cov), where g_i = dL/dp'_i and w_cov is the rotation gradient of
// the rotated covariances. Since exp(xi + dxi) = exp(J(xi) dxi) exp(xi) with J the
// SE(3) left Jacobian, dL/dxi = J(xi)^T dL/dd. The kernel forms the sums in one pass
// over the Gaussians; the last block to finish folds the per-block partials in a fixed
// pattern (deterministic) and applies J^T in double precision.
#include "cfgs_internal.cuh"

namespace cfgs {

constexpr int kPoseThreads = 256;
constexpr int kPosePartials = 9;  // sum g (3), sum (R p) x g (3), w_cov (3)

__host__ __device__ inline void mm3(const double* A, const double* B, double* C) {
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) C[3 * i + j] = A[3 * i] * B[j] + A[3 * i + 1] * B[3 + j] + A[3 * i + 2] * B[6 + j];
}

// ---- exp(xi) and its Jacobian blocks by one warp ------------------------------------------
// Lane 3 i + j (mod 9) holds element (i, j) of every 3x3 matrix.
struct LanePose {
  double R, t;   // exp(xi): element of the rotation; lane i mod 3: component i of the translation
  double Jl, Q;  // SO(3) left Jacobian of phi, upper-right block of the SE(3) one
};

__device__ __forceinline__ double lane_mm3(double A, double B, int i, int j) {
  const double a0 = __shfl_sync(0xffffffffu, A, 3 * i), a1 = __shfl_sync(0xffffffffu, A, 3 * i + 1),
               a2 = __shfl_sync(0xffffffffu, A, 3 * i + 2);
  const double b0 = __shfl_sync(0xffffffffu, B, j), b1 = __shfl_sync(0xffffffffu, B, 3 + j),
               b2 = __shfl_sync(0xffffffffu, B, 6 + j);
  return a0 * b0 + a1 * b1 + a2 * b2;
}

// Element (i, j) of the cross-product matrix of w.
__device__ __forceinline__ double lane_hat(const double (&w)[3], int i, int j) {
  if (i == j) return 0.0;
  const double v = w[3 - i - j];
  return (j - i + 3) % 3 == 1 ? -v : v;
}

// With theta = |phi|: R = I + a P + b P^2, Jl = I + b P + c P^2 (P the matrix of phi), t = Jl
// rho, and Q(rho, phi) after Barfoot, "State Estimation for Robotics", eq. 7.86. Every lane of
// a warp calls it with the same xi. Bound by latency (a float64 operation takes the pipe 16
// cycles, its result longer): the sine and cosine share their reduction, the five divisions
// run on five lanes at once, the matrices element by element. By single threads, one for exp
// and one for Q, the two took 14,000 and 26,000 cycles, each with its own sines.
__device__ __forceinline__ LanePose lane_pose(const double (&rho)[3], const double (&phi)[3], int lane) {
  const int e = lane % 9, i = e / 3, j = e % 3;
  const double th2 = phi[0] * phi[0] + phi[1] * phi[1] + phi[2] * phi[2];
  double a, b, c, c1, c2, c3;
  // a = sin(th)/th, b = (1-cos th)/th^2, c = c1 = (th - sin th)/th^3, c2 = (th^2 + 2 cos th -
  // 2)/(2 th^4), c3 = (2 th - 3 sin th + th cos th)/(2 th^5), with series near 0
  if (!(th2 < 1e-8)) {
    const double th = sqrt(th2);
    double s, co;
    sincos(th, &s, &co);
    const double th3 = th2 * th, th4 = th2 * th2, th5 = th4 * th;
    double num = s, den = th;
    if (lane == 1) {
      num = 1.0 - co;
      den = th2;
    } else if (lane == 2) {
      num = th - s;
      den = th3;
    } else if (lane == 3) {
      num = th2 + 2.0 * co - 2.0;
      den = 2.0 * th4;
    } else if (lane == 4) {
      num = 2.0 * th - 3.0 * s + th * co;
      den = 2.0 * th5;
    }
    const double q = num / den;
    a = __shfl_sync(0xffffffffu, q, 0);
    b = __shfl_sync(0xffffffffu, q, 1);
    c = c1 = __shfl_sync(0xffffffffu, q, 2);
    c2 = __shfl_sync(0xffffffffu, q, 3);
    c3 = __shfl_sync(0xffffffffu, q, 4);
  } else {
    a = 1.0 - th2 / 6.0;
    b = 0.5 - th2 / 24.0;
    c = 1.0 / 6.0 - th2 / 120.0;
  }
  if (th2 < 1e-6) {
    c1 = 1.0 / 6.0 - th2 / 120.0;
    c2 = 1.0 / 24.0 - th2 / 720.0;
    c3 = 1.0 / 120.0 - th2 / 2520.0;
  }
  const double I = i == j ? 1.0 : 0.0, P = lane_hat(phi, i, j), Rh = lane_hat(rho, i, j);
  const double PP = lane_mm3(P, P, i, j);
  LanePose o;
  o.R = I + a * P + b * PP;
  o.Jl = I + b * P + c * PP;
  const int r = lane % 3;
  const double j0 = __shfl_sync(0xffffffffu, o.Jl, 3 * r), j1 = __shfl_sync(0xffffffffu, o.Jl, 3 * r + 1),
               j2 = __shfl_sync(0xffffffffu, o.Jl, 3 * r + 2);
  o.t = j0 * rho[0] + j1 * rho[1] + j2 * rho[2];
  const double PR = lane_mm3(P, Rh, i, j), RP = lane_mm3(Rh, P, i, j);
  const double PRP = lane_mm3(PR, P, i, j), PPR = lane_mm3(PP, Rh, i, j), RPP = lane_mm3(Rh, PP, i, j);
  const double PRPP = lane_mm3(PRP, P, i, j), PPRP = lane_mm3(P, PRP, i, j);
  o.Q = 0.5 * Rh + c1 * (PR + RP + PRP) + c2 * (PPR + RPP - 3.0 * PRP) + c3 * (PRPP + PPRP);
  return o;
}

// The same into a solve's state.
__device__ __forceinline__ void store_pose_state(const float (&xi)[6], PoseState* ps, int lane) {
  const double rho[3] = {xi[0], xi[1], xi[2]}, phi[3] = {xi[3], xi[4], xi[5]};
  const LanePose o = lane_pose(rho, phi, lane);
  if (lane < 9) {
    ps->R64[lane] = o.R;
    ps->R[lane] = (float)o.R;
    ps->Jl[lane] = o.Jl;
    ps->Q[lane] = o.Q;
  }
  if (lane < 3) {
    ps->t64[lane] = o.t;
    ps->t[lane] = (float)o.t;
  }
}

// Each block's first warp forms exp(xi) in float64 while the others' positions are on
// their way from memory: the chain of double sin, cos and divisions is most of the kernel's
// time, so a block takes kApplyPerThread positions per thread (230,400 positions: 225
// blocks, 16.7 -> 7.6 us; one position per thread ran 900 such chains).
constexpr int kApplyPerThread = 4;

template <bool COV>
__global__ void __launch_bounds__(kPoseThreads) k_pose_apply(int n, const float* xi, const float* xyz,
                                                              const float* cov_in, float* means_out,
                                                              float* cov_out) {
  __shared__ float sR[9], st[3];
  const int64_t i0 = (int64_t)blockIdx.x * (kPoseThreads * kApplyPerThread) + threadIdx.x;
  float p[kApplyPerThread][3];
#pragma unroll
  for (int k = 0; k < kApplyPerThread; ++k) {
    const int64_t i = i0 + k * kPoseThreads;
#pragma unroll
    for (int a = 0; a < 3; ++a) p[k][a] = i < n ? xyz[3 * i + a] : 0.0f;
  }
  if (threadIdx.x < 32) {
    const double rho[3] = {xi[0], xi[1], xi[2]}, phi[3] = {xi[3], xi[4], xi[5]};
    const LanePose o = lane_pose(rho, phi, threadIdx.x);  // (its Q is not used)
    if (threadIdx.x < 9) sR[threadIdx.x] = (float)o.R;
    if (threadIdx.x < 3) st[threadIdx.x] = (float)o.t;
  }
  __syncthreads();
  float R[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) R[k] = sR[k];
#pragma unroll
  for (int k = 0; k < kApplyPerThread; ++k) {
    const int64_t i = i0 + k * kPoseThreads;
    if (i >= n) break;
#pragma unroll
    for (int r = 0; r < 3; ++r)  // ((R0 x + R1 y) + R2 z) + t, each operation rounded once
      means_out[3 * i + r] =
          __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(R[3 * r], p[k][0]), __fmul_rn(R[3 * r + 1], p[k][1])),
                              __fmul_rn(R[3 * r + 2], p[k][2])),
                    st[r]);
    if (COV) {
      const float* c = cov_in + 6 * (size_t)i;
      float C[9] = {c[0], c[1], c[2], c[1], c[3], c[4], c[2], c[4], c[5]};
      float RC[9];
#pragma unroll
      for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b) RC[3 * a + b] = R[3 * a] * C[b] + R[3 * a + 1] * C[3 + b] + R[3 * a + 2] * C[6 + b];
      const int ii[6] = {0, 0, 0, 1, 1, 2}, jj[6] = {0, 1, 2, 1, 2, 2};
#pragma unroll
      for (int q = 0; q < 6; ++q) {
        int a = ii[q], b = jj[q];
        cov_out[6 * (size_t)i + q] = RC[3 * a] * R[3 * b] + RC[3 * a + 1] * R[3 * b + 1] + RC[3 * a + 2] * R[3 * b + 2];
      }
    }
  }
}

// One Adam step on `count` 6-vectors (one per solve), following the operation sequence
// of torch.optim.Adam's default multi-tensor path for float32 CUDA tensors:
//   m = lerp(m, g, 1 - b1);  v = v * b2;  v = addcmul(v, g, g, 1 - b2);
//   denom = sqrt(v) / sqrt(1 - b2^t) + eps;  p = addcdiv(p, m, denom, -lr / (1 - b1^t))
// with the hyper-parameters as float64 scalars rounded to float32 per use, as torch
// passes them, so both optimisers take the same steps. bc1 = 1 - b1^t and
// bc2 = 1 - b2^t are float64, as torch forms them on the host.
// state per solve: m[6], v[6], step, 3 unused floats.
__device__ __forceinline__ double bias_correction(double beta, float step) {
  return 1.0 - pow(beta, (double)step);
}

// The step size and the root of the second correction.
struct AdamScale {
  float step_size, bc2_sqrt;
};
__device__ __forceinline__ AdamScale adam_scale(double lr, double bc1, double bc2) {
  return {(float)(-(lr / bc1)), (float)sqrt(bc2)};
}

__device__ __forceinline__ void adam_component(int k, float* xi, float g, float* st, AdamScale c, double b1, double b2,
                                               double eps) {
  const float w1 = (float)(1.0 - b1), mul2 = (float)b2, w2 = (float)(1.0 - b2);
  const float eps_f = (float)eps;
  float m = st[k], v = st[6 + k];
  m = fmaf(w1, g - m, m);
  v = v * mul2;
  v = fmaf(w2, g * g, v);
  st[k] = m;
  st[6 + k] = v;
  float denom = sqrtf(v) / c.bc2_sqrt;
  denom = denom + eps_f;
  xi[k] = fmaf(c.step_size, m / denom, xi[k]);
}

// One warp per solve: lanes 0 and 1 form the two bias corrections (a double pow each, the
// kernel's longest chain) at the same time, then lanes 0..5 step one component each (10.3 -> 7.9 us).
__global__ void __launch_bounds__(128) k_pose_adam(int count, float* xi, const float* grad, float* state, double lr,
                                                   double b1, double b2, double eps) {
  const int s = blockIdx.x * (int)(blockDim.x >> 5) + (int)(threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (s >= count) return;
  float* st = state + 16 * (size_t)s;
  const float step = st[12] + 1.0f;
  const double bc = bias_correction(lane & 1 ? b2 : b1, step);
  const double bc1 = __shfl_sync(0xffffffffu, bc, 0), bc2 = __shfl_sync(0xffffffffu, bc, 1);
  __syncwarp();  // every lane has read the step count
  if (lane < 6)
    adam_component(lane, xi + 6 * (size_t)s, grad[6 * (size_t)s + lane], st, adam_scale(lr, bc1, bc2), b1, b2, eps);
  if (lane == 0) st[12] = step;
}

// dL/dxi from the left-perturbation sums tot = (sum g, sum (R p) x g, w_cov):
// d_rho = sum g, d_phi = sum (R p + t) x g + w_cov, then dL/dxi = J^T dL/dd with the
// SE(3) left Jacobian J = [[Jl, Q], [0, Jl]] — all in float64, rounded at the end, with
// exp(xi), Jl and Q taken from the solve's state.
__device__ void pose_grad_from_state(const PoseState& ps, const double* tot, float* grad_out) {
  const double gr[3] = {tot[0], tot[1], tot[2]};
  double gp[3];
  gp[0] = tot[3] + (ps.t64[1] * gr[2] - ps.t64[2] * gr[1]) + tot[6];
  gp[1] = tot[4] + (ps.t64[2] * gr[0] - ps.t64[0] * gr[2]) + tot[7];
  gp[2] = tot[5] + (ps.t64[0] * gr[1] - ps.t64[1] * gr[0]) + tot[8];
  const double* Jl = ps.Jl;
  const double* Q = ps.Q;
  for (int j = 0; j < 3; ++j) {
    grad_out[j] = (float)(Jl[j] * gr[0] + Jl[3 + j] * gr[1] + Jl[6 + j] * gr[2]);
    grad_out[3 + j] = (float)(Q[j] * gr[0] + Q[3 + j] * gr[1] + Q[6 + j] * gr[2] + Jl[j] * gp[0] +
                              Jl[3 + j] * gp[1] + Jl[6 + j] * gp[2]);
  }
}

// ---- pose gradient of one solve --------------------------------------------------------
// Sums in float64 of exact float32 x float32 products, so the result is the float64 value
// a float64 autograd of exp(xi).act(p) forms, rounded to float32 at the end: the fused and
// plain solves stay on the same trajectory. With M = sum p g^T, sum (R p) x g is read off
// R M, so the pass over the Gaussians needs neither the rotation nor its products: 12
// float64 accumulations (15 with covariances) per Gaussian. Block 0 forms exp(xi), Jl and Q
// meanwhile; the last block to finish folds the others' partials in a fixed pattern (warp
// w takes rows w, w + 8, ..., one lane per sum) and applies the Jacobian transpose. Bound
// by the float64 pipe (about 2 operations per cycle and SM). 230,400 Gaussians: 371 us
// (one thread folded 900 rows of 9 sums one after another, and every block formed exp(xi))
// -> 22 us.
constexpr int kGradMaxBlocks = 2 * 152;  // two blocks of partial sums per SM at most
constexpr int kGradSums = 16;            // sum g (3), M (9), w_cov (3), unused

struct PoseGradArgs {
  int n;
  const float* xi;
  const float* xyz;
  const float* dL_dmeans;
  const float* cov_rot;
  const float* dL_dcov;
  double* partials;       // [gridDim.x - 1][kGradSums]
  PoseState* state;       // written by block 0
  unsigned int* counter;  // zeroed before launch
  float* grad_out;        // [6]
};

// Sums 16 values per lane over the warp by a transposing reduction (8 + 4 + 2 + 1 exchange
// steps, one plain step): lane 2k ends with the total of value k.
__device__ __forceinline__ double warp_sum16_f64(double (&v)[16], int lane) {
#pragma unroll
  for (int half = 8; half >= 1; half >>= 1) {
    const bool up = lane & (2 * half);
#pragma unroll
    for (int k = 0; k < half; ++k) {
      const double send = up ? v[k] : v[k + half];
      const double keep = up ? v[k + half] : v[k];
      v[k] = keep + __shfl_xor_sync(0xffffffffu, send, 2 * half);
    }
  }
  return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

template <bool COV>
__global__ void __launch_bounds__(kPoseThreads) k_pose_grad(PoseGradArgs a) {
  constexpr int kWarpsPerBlock = kPoseThreads / 32;
  __shared__ double s_red[kWarpsPerBlock][kGradSums];
  __shared__ bool s_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (blockIdx.x == 0) {
    if (warp == 0) {
      const float x[6] = {a.xi[0], a.xi[1], a.xi[2], a.xi[3], a.xi[4], a.xi[5]};
      store_pose_state(x, a.state, lane);
    }
  } else {
    double acc[kGradSums];
#pragma unroll
    for (int k = 0; k < kGradSums; ++k) acc[k] = 0.0;
    const int64_t stride = (int64_t)(gridDim.x - 1) * kPoseThreads;
    for (int64_t i = (int64_t)(blockIdx.x - 1) * kPoseThreads + threadIdx.x; i < a.n; i += stride) {
      double g[3], p[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        p[k] = a.xyz[3 * i + k];
        g[k] = a.dL_dmeans[3 * i + k];
      }
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        acc[k] += g[k];
#pragma unroll
        for (int j = 0; j < 3; ++j) acc[3 + 3 * k + j] = fma(p[k], g[j], acc[3 + 3 * k + j]);
      }
      if (COV) {
        const float* c = a.cov_rot + 6 * (size_t)i;
        const float* d = a.dL_dcov + 6 * (size_t)i;
        float C[9] = {c[0], c[1], c[2], c[1], c[3], c[4], c[2], c[4], c[5]};
        float G[9] = {d[0], 0.5f * d[1], 0.5f * d[2], 0.5f * d[1], d[3], 0.5f * d[4], 0.5f * d[2], 0.5f * d[4], d[5]};
        // w = (M12 - M21, M20 - M02, M01 - M10) of the antisymmetric M = C G - G C, where
        // G C = (C G)^T for symmetric C, G, so M_rs = CG_rs - CG_sr
        float CG[9];
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
          for (int q = 0; q < 3; ++q)
            CG[3 * r + q] = C[3 * r] * G[q] + C[3 * r + 1] * G[3 + q] + C[3 * r + 2] * G[6 + q];
        acc[12] += 2.0 * ((double)CG[5] - (double)CG[7]);
        acc[13] += 2.0 * ((double)CG[6] - (double)CG[2]);
        acc[14] += 2.0 * ((double)CG[1] - (double)CG[3]);
      }
    }
    const double v = warp_sum16_f64(acc, lane);
    if ((lane & 1) == 0) s_red[warp][lane >> 1] = v;
    __syncthreads();
    if (threadIdx.x < kGradSums) {
      double t = 0.0;
      for (int w = 0; w < kWarpsPerBlock; ++w) t += s_red[w][threadIdx.x];
      a.partials[(size_t)(blockIdx.x - 1) * kGradSums + threadIdx.x] = t;
    }
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(a.counter, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  {
    double t = 0.0;
    if (lane < kGradSums) {
#pragma unroll 4
      for (int b = warp; b < (int)gridDim.x - 1; b += kWarpsPerBlock) t += __ldcg(a.partials + (size_t)b * kGradSums + lane);
      s_red[warp][lane] = t;
    }
  }
  __syncthreads();
  if (warp != 0) return;
  {
    double t = 0.0;
    if (lane < kGradSums)
#pragma unroll
      for (int w = 0; w < kWarpsPerBlock; ++w) t += s_red[w][lane];
    __syncwarp();
    if (lane < kGradSums) s_red[0][lane] = t;
    __syncwarp();
  }
  if (lane == 0) {
    const double* s = s_red[0];
    const volatile PoseState* vs = a.state;  // another block's writes
    PoseState ps;
    for (int k = 0; k < 9; ++k) {
      ps.R64[k] = vs->R64[k];
      ps.Jl[k] = vs->Jl[k];
      ps.Q[k] = vs->Q[k];
    }
    for (int k = 0; k < 3; ++k) ps.t64[k] = vs->t64[k];
    double N[9];  // sum (R p) g^T
    mm3(ps.R64, s + 3, N);
    const double tot[kPosePartials] = {s[0],        s[1],        s[2],  N[5] - N[7], N[6] - N[2],
                                       N[1] - N[3], s[12], s[13], s[14]};
    pose_grad_from_state(ps, tot, a.grad_out);
    *a.counter = 0u;
  }
}

// One block per solve: the state of xi by one warp, the next step's bias corrections by two
// others.
__global__ void k_batch_pose_init(const float* xi, const float* adam_state, PoseState* states, double b1,
                                  double b2) {
  const int s = blockIdx.x;
  const float* x = xi + 6 * (size_t)s;
  const float step = adam_state[16 * (size_t)s + 12] + 1.0f;
  if (threadIdx.x < 32) {
    const float xs[6] = {x[0], x[1], x[2], x[3], x[4], x[5]};
    store_pose_state(xs, states + s, threadIdx.x);
  }
  if (threadIdx.x == 64) states[s].bc1 = bias_correction(b1, step);
  if (threadIdx.x == 96) states[s].bc2 = bias_correction(b2, step);
}

// One block per solve: the solve's per-block pose partials summed in a fixed pattern
// (thread i takes blocks i, i+256, ...; then a fixed tree), then by one warp the SE(3)
// Jacobian transpose and the Adam step (a lane per component) with the state's cached
// Jacobian blocks and bias corrections, and the state of the new xi, while two other warps
// form the following step's corrections. A solve's result depends only on its own blocks, so
// it is the same whatever else is in the batch. Bound by the latency of one chain of float64
// operations per solve: 27 -> 13 us (900 partials; 24 us of it one thread's sums, gradient, step
// and then one thread's Q).
constexpr int kUpdateThreads = 256, kUpdateBatch = 4;
__global__ void __launch_bounds__(kUpdateThreads) k_batch_pose_update(const SceneDesc* descs, const double* partials,
                                                                      float* xi, float* adam_state, PoseState* states,
                                                                      const CfgsCounts* counts, int64_t cap, double lr,
                                                                      double b1, double b2, double eps) {
  __shared__ double s_red[8][6];
  if ((int64_t)counts->num_rendered > cap) return;  // overflowed iteration: no update
  const int s = blockIdx.x;
  const SceneDesc& sd = descs[s];
  const int b0 = sd.gauss_base / kPreprocessBlock;
  const int nb = (sd.num_gaussians + kPreprocessBlock - 1) / kPreprocessBlock;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float* x = xi + 6 * (size_t)s;
  float* st = adam_state + 16 * (size_t)s;
  PoseState* ps = states + s;
  const float step = st[12];
  double acc[6] = {0, 0, 0, 0, 0, 0};
  for (int b = threadIdx.x; b < nb; b += kUpdateThreads * kUpdateBatch) {
    double v[kUpdateBatch][6];
#pragma unroll
    for (int q = 0; q < kUpdateBatch; ++q)
#pragma unroll
      for (int k = 0; k < 6; ++k)
        v[q][k] = b + q * kUpdateThreads < nb ? partials[(size_t)(b0 + b + q * kUpdateThreads) * 9 + k] : 0.0;
#pragma unroll
    for (int q = 0; q < kUpdateBatch; ++q)
#pragma unroll
      for (int k = 0; k < 6; ++k) acc[k] += v[q][k];
  }
  // warp 0, before it waits for the sums: what the step needs of the state
  const int j = lane % 3;
  double Jl[3], Q[3], t64[3];
  AdamScale scale{};
  if (warp == 0) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      Jl[k] = ps->Jl[3 * k + j];
      Q[k] = ps->Q[3 * k + j];
      t64[k] = ps->t64[k];
    }
    scale = adam_scale(lr, ps->bc1, ps->bc2);
  }
  {
    const double tot = warp_sum6_f64(acc, lane);  // lane 4k: partial k of the warp
    if ((lane & 3) == 0 && (lane >> 2) < 6) s_red[warp][lane >> 2] = tot;
  }
  __syncthreads();
  if (threadIdx.x == 64) ps->bc1 = bias_correction(b1, (step + 1.0f) + 1.0f);
  if (threadIdx.x == 96) ps->bc2 = bias_correction(b2, (step + 1.0f) + 1.0f);
  if (warp != 0) return;
  double sum = 0.0;
#pragma unroll
  for (int w = 0; w < kUpdateThreads / 32; ++w) sum += s_red[w][lane < 6 ? lane : 0];
  // as pose_grad_from_state: lane j component j, lane 3 + j component 3 + j
  double gr[3], gp[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) gr[k] = __shfl_sync(0xffffffffu, sum, k);
#pragma unroll
  for (int k = 0; k < 3; ++k) gp[k] = __shfl_sync(0xffffffffu, sum, 3 + k);
  gp[0] = gp[0] + (t64[1] * gr[2] - t64[2] * gr[1]);
  gp[1] = gp[1] + (t64[2] * gr[0] - t64[0] * gr[2]);
  gp[2] = gp[2] + (t64[0] * gr[1] - t64[1] * gr[0]);
  const float g_rho = (float)(Jl[0] * gr[0] + Jl[1] * gr[1] + Jl[2] * gr[2]);
  const float g_phi =
      (float)(Q[0] * gr[0] + Q[1] * gr[1] + Q[2] * gr[2] + Jl[0] * gp[0] + Jl[1] * gp[1] + Jl[2] * gp[2]);
  float moved = 0.f;
  if (lane < 6) {
    adam_component(lane, x, lane < 3 ? g_rho : g_phi, st, scale, b1, b2, eps);
    moved = x[lane];
  }
  if (lane == 0) st[12] = step + 1.0f;
  float xs[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) xs[k] = __shfl_sync(0xffffffffu, moved, k);
  store_pose_state(xs, ps, lane);
}

void launch_batch_pose_init(int count, const float* xi, const float* adam_state, PoseState* states, double b1,
                            double b2, cudaStream_t st) {
  k_batch_pose_init<<<count, 128, 0, st>>>(xi, adam_state, states, b1, b2);
}
void launch_batch_pose_update(int count, const SceneDesc* descs, const double* partials, float* xi,
                              float* adam_state, PoseState* states, const CfgsCounts* counts, int64_t cap, double lr,
                              double b1, double b2, double eps, cudaStream_t st) {
  k_batch_pose_update<<<count, kUpdateThreads, 0, st>>>(descs, partials, xi, adam_state, states, counts, cap, lr, b1, b2, eps);
}

}  // namespace cfgs

using namespace cfgs;

// Scratch of cfgs_pose_grad: the blocks' partial sums, the pose state, the block counter.
struct PoseGradLayout {
  size_t partials = 0, state, counter, total;
  PoseGradLayout() {
    state = align256(sizeof(double) * kGradSums * kGradMaxBlocks);
    counter = state + align256(sizeof(PoseState));
    total = counter + 256;
  }
};

extern "C" int cfgs_pose_apply(int32_t n, const float* xi, const float* xyz, const float* cov_in, float* means_out,
                               float* cov_out, void* stream) {
  if (n < 0 || !xi || (n > 0 && (!xyz || !means_out))) return CFGS_ERR_INVALID_ARGUMENT;
  if ((cov_in == nullptr) != (cov_out == nullptr)) return CFGS_ERR_INVALID_ARGUMENT;
  if (n == 0) return CFGS_OK;
  const int blocks = div_up(n, kPoseThreads * kApplyPerThread);
  cudaStream_t st = (cudaStream_t)stream;
  if (cov_in) k_pose_apply<true><<<blocks, kPoseThreads, 0, st>>>(n, xi, xyz, cov_in, means_out, cov_out);
  else k_pose_apply<false><<<blocks, kPoseThreads, 0, st>>>(n, xi, xyz, cov_in, means_out, cov_out);
  CFGS_CHECK_LAUNCH(0, stream);
  return CFGS_OK;
}

extern "C" size_t cfgs_pose_scratch_bytes(int32_t n) {
  (void)n;
  return PoseGradLayout().total;
}

extern "C" int cfgs_pose_grad(int32_t n, const float* xi, const float* xyz, const float* dL_dmeans, const float* cov_rot,
                              const float* dL_dcov, void* scratch, float* grad_out, void* stream) {
  if (n < 0 || !xi || !scratch || !grad_out || (n > 0 && (!xyz || !dL_dmeans))) return CFGS_ERR_INVALID_ARGUMENT;
  if ((cov_rot == nullptr) != (dL_dcov == nullptr)) return CFGS_ERR_INVALID_ARGUMENT;
  cudaStream_t st = (cudaStream_t)stream;
  const PoseGradLayout L;
  char* base = static_cast<char*>(scratch);
  PoseGradArgs a;
  a.n = n;
  a.xi = xi;
  a.xyz = xyz;
  a.dL_dmeans = dL_dmeans;
  a.cov_rot = cov_rot;
  a.dL_dcov = dL_dcov;
  a.partials = reinterpret_cast<double*>(base + L.partials);
  a.state = reinterpret_cast<PoseState*>(base + L.state);
  a.counter = reinterpret_cast<unsigned int*>(base + L.counter);
  a.grad_out = grad_out;
  if (cudaMemsetAsync(a.counter, 0, sizeof(unsigned int), st) != cudaSuccess) return CFGS_ERR_LAUNCH;
  const int sums = div_up(n > 0 ? n : 1, kPoseThreads);
  const int blocks = 1 + (sums < kGradMaxBlocks ? sums : kGradMaxBlocks);  // block 0 forms the pose state
  if (cov_rot) k_pose_grad<true><<<blocks, kPoseThreads, 0, st>>>(a);
  else k_pose_grad<false><<<blocks, kPoseThreads, 0, st>>>(a);
  CFGS_CHECK_LAUNCH(0, st);
  return CFGS_OK;
}

extern "C" int cfgs_pose_adam(int32_t count, float* xi, const float* grad, float* state, double lr, double beta1,
                              double beta2, double eps, void* stream) {
  if (count < 0 || (count > 0 && (!xi || !grad || !state))) return CFGS_ERR_INVALID_ARGUMENT;
  if (count == 0) return CFGS_OK;
  k_pose_adam<<<div_up(count, 4), 128, 0, (cudaStream_t)stream>>>(count, xi, grad, state, lr, beta1, beta2, eps);
  CFGS_CHECK_LAUNCH(0, stream);
  return CFGS_OK;
}
