// Small kernels of the Gram-free leaf range finder (api.cu, HT_LEAF_SKETCH).
//
// A leaf's range finder never forms the mode Gram G = X_(m) X_(m)^T: each
// application Y = G Q runs as two streaming products over the tensor
// (Z = X_(m)^T Q, Y = X_(m) Z).  After the last application the leaf basis
// comes from the Nystrom approximation of G in the test block Q,
//   G ~ Y (Q^T Y)^-1 Y^T,
// taken with a small shift nu for stability (Tropp, Yurtsever, Udell and
// Cevher, "Fixed-rank approximation of a positive-semidefinite matrix from
// streaming data", NeurIPS 2017, Alg. 3): with Y_nu = Y + nu Q = Q1 R1 and
// W = Q^T Y,
//   G + nu I ~ Q1 R1 (W + nu I)^-1 R1^T Q1^T,
// so the leaf basis is Q1 times the top eigenvectors of the s x s matrix
// H = R1 (W + nu I)^-1 R1^T.  The reference's range finder (rsvd,
// third_order_tensor_decompsition/CUDA/Optimized/kernel.cu:595-680) instead
// forms B = C^T A from its sketch C = A Omega and takes the SVD of B.
#include <algorithm>

#include "common.cuh"
#include "engine.h"

namespace htgb {
namespace {

constexpr int NY_MAX = 64;

// nu = nu_rel * tr(W) in FP64, in every lane of the calling warp (the two
// kernels below must agree on it bit for bit).  The diagonal is loaded at once
// and summed as a tree: one thread's chain of loads and FP64 additions took most
// of the shift kernel's 15 us.
HT_DEV double nystrom_nu(const float *W, int s, float nu_rel) {
  const int lane = threadIdx.x & 31;
  double tr = lane < s ? static_cast<double>(W[lane + s * lane]) : 0.0;
  if (lane + 32 < s) tr += static_cast<double>(W[(lane + 32) + s * (lane + 32)]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) tr += __shfl_xor_sync(0xffffffffu, tr, o);
  return static_cast<double>(nu_rel) * (tr > 0.0 ? tr : 0.0);
}

struct NystromShiftBatch {
  NystromShift p[4];
};

// blockIdx.y is the problem (a launch, and a copy of Y, for each mode before).
__global__ void __launch_bounds__(256) nystrom_shift_kernel(const NystromShiftBatch batch, float nu_rel) {
  const NystromShift &p = batch.p[blockIdx.y];
  __shared__ float s_nu;
  if (threadIdx.x < 32) {
    const double nu = nystrom_nu(p.W, p.s, nu_rel);
    if (threadIdx.x == 0) s_nu = static_cast<float>(nu);
  }
  __syncthreads();
  const float nu = s_nu;
  const long long total = p.n * p.s;
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < total; i += gridDim.x * 256ll)
    p.Y[i] = p.Yn[i] = fmaf(nu, p.Q[i], p.Y[i]);
}

// H = R1 (sym(W) + nu I)^-1 R1^T in FP64 (Cholesky of the shifted W; a pivot
// that rounding drove to or below zero is floored at nu).  One CTA.
struct NystromBatch {
  NystromProb p[4];
};

__global__ void __launch_bounds__(256) nystrom_core_kernel(const NystromBatch batch, float nu_rel,
                                                           int *__restrict__ err) {
  const float *__restrict__ W = batch.p[blockIdx.x].W;
  const float *__restrict__ R1 = batch.p[blockIdx.x].R1;
  const int s = batch.p[blockIdx.x].s;
  float *__restrict__ H = batch.p[blockIdx.x].H;
  extern __shared__ double ny_sm[];
  double *L = ny_sm;                       // upper Cholesky factor, row-major: (W + nu I) = L^T L
  double *F = ny_sm + NY_MAX * NY_MAX;     // F = R1 L^-1, row-major
  __shared__ double s_nu, s_inv;
  const int t = threadIdx.x;
  if (t < 32) {
    const double v = nystrom_nu(W, s, nu_rel);
    if (t == 0) s_nu = v;
  }
  __syncthreads();
  const double nu = s_nu;
  for (int e = t; e < s * s; e += 256) {
    const int i = e / s, j = e % s;
    L[i * NY_MAX + j] = 0.5 * (static_cast<double>(W[i + s * j]) + static_cast<double>(W[j + s * i])) +
                        (i == j ? nu : 0.0);
  }
  __syncthreads();
  // F starts as R1 and is solved along with the factorisation: step j scales
  // row j of L and column j of F and updates what lies to their right, 64
  // columns by four rows at a time (FP64 is the scarce unit: one root and one
  // division a step, and each half of a symmetric result once)
  const int col = t & 63, row0 = t >> 6;
  for (int e = t; e < s * s; e += 256) F[(e % s) * NY_MAX + e / s] = static_cast<double>(R1[e]);
  __syncthreads();
  for (int j = 0; j < s; ++j) {
    if (t == 0) {
      double d = L[j * NY_MAX + j];
      if (!isfinite(d)) report_error(err, kErrNonFinite);
      if (!(d > nu)) d = nu > 0.0 ? nu : 1.0;
      s_inv = 1.0 / sqrt(d);
    }
    __syncthreads();
    const double inv = s_inv;
    if (t < 64) {
      if (j + 1 + t < s) L[j * NY_MAX + j + 1 + t] *= inv;
    } else if (t < 128) {
      if (t - 64 < s) F[(t - 64) * NY_MAX + j] *= inv;
    }
    __syncthreads();
    const int c = j + 1 + col;
    if (c < s) {
      const double l = L[j * NY_MAX + c];
      for (int i = j + 1 + row0; i <= c; i += 4) L[i * NY_MAX + c] -= L[j * NY_MAX + i] * l;
      for (int i = row0; i < s; i += 4) F[i * NY_MAX + c] -= F[i * NY_MAX + j] * l;
    }
    __syncthreads();
  }
  for (int e = t; e < s * (s + 1) / 2; e += 256) {   // e = j (j + 1) / 2 + i, i <= j
    int j = static_cast<int>((sqrtf(8.f * e + 1.f) - 1.f) * 0.5f);
    while (j * (j + 1) / 2 > e) --j;
    while ((j + 1) * (j + 2) / 2 <= e) ++j;
    const int i = e - j * (j + 1) / 2;
    double v = 0.0;
    for (int c = 0; c < s; ++c) v = fma(F[i * NY_MAX + c], F[j * NY_MAX + c], v);
    H[i + s * j] = H[j + s * i] = static_cast<float>(v);
  }
}

}  // namespace

cudaError_t nystrom_shift_launch(const NystromShift *probs, int nprob, float nu_rel, cudaStream_t st) {
  if (nprob < 1 || nprob > 4) return cudaErrorInvalidValue;
  NystromShiftBatch b{};
  long long blocks = 1;
  for (int i = 0; i < nprob; ++i) {
    if (probs[i].s < 1 || probs[i].s > NY_MAX) return cudaErrorInvalidValue;
    b.p[i] = probs[i];
    blocks = std::max(blocks, (probs[i].n * probs[i].s + 255) / 256);
  }
  blocks = std::min(blocks, 4ll * device_sm_count());
  nystrom_shift_kernel<<<dim3(static_cast<unsigned>(blocks), nprob), 256, 0, st>>>(b, nu_rel);
  return cudaGetLastError();
}

cudaError_t nystrom_core_launch(const NystromProb *probs, int nprob, float nu_rel, int *err, cudaStream_t st) {
  if (nprob < 1 || nprob > 4) return cudaErrorInvalidValue;
  NystromBatch b;
  for (int i = 0; i < 4; ++i) b.p[i] = NystromProb{nullptr, nullptr, 0, nullptr};
  for (int i = 0; i < nprob; ++i) {
    if (probs[i].s < 1 || probs[i].s > NY_MAX) return cudaErrorInvalidValue;
    b.p[i] = probs[i];
  }
  constexpr int kSmem = 2 * NY_MAX * NY_MAX * sizeof(double);
  static bool attr_set[64] = {};
  const cudaError_t e = opt_in_smem(nystrom_core_kernel, kSmem, attr_set);
  if (e != cudaSuccess) return e;
  nystrom_core_kernel<<<nprob, 256, kSmem, st>>>(b, nu_rel, err);
  return cudaGetLastError();
}

}  // namespace htgb
