// HT tensor layer: a fully connected layer whose weight is held in HT format.
//
// The reference's layer (HT_tensor_layer/FC_MNIST/mnist_ht.py:232-245 and
// Alex_ImageNet/model/alexnet.py:157-170) maps x[z, n0, n1, n2] to
// y[z, m0, m1, m2] through the einsum chain
//   x u1[n0,m0,r3] -> b2[r3,r4,r1] -> u2[n1,m1,r4] -> b1[r1,r2] -> u3[n2,m2,r2],
// i.e. y = x W^T with
//   W[(m0,m1,m2), (n0,n1,n2)] = sum_{r1} P[a, b, r1] Q[c, r1],
//   P[a, b, r1] = sum_{r3,r4} u1[a, r3] u2[b, r4] b2[r3, r4, r1],   a = n0 M0 + m0, b = n1 M1 + m1
//   Q[c, r1]    = sum_{r2} b1[r1, r2] u3[c, r2],                     c = n2 M2 + m2.
// The chain costs more multiply-adds per sample than the dense product at the
// reference's shapes (rank 16 on 8 x 8 x 16 modes), so here the weight is formed
// once per call from the factors (batch-independent, L2-resident) and the batch
// goes through one GEMM; the kernels in this file form P, Q and W, add the
// bias, and carry the gradients back from dW to the factors.
//
// All parameter tensors use the reference's C-order layouts:
// u_j (N_j, M_j, r_j), b2 (r3, r4, r1), b1 (r1, r2), bias (M0, M1, M2).
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "engine.h"

namespace htgb {
namespace {

constexpr int kLayerThreads = 256;

int grid_for_layer(long long n) {
  long long g = (n + kLayerThreads - 1) / kLayerThreads;
  if (g > 32ll * device_sm_count()) g = 32ll * device_sm_count();
  return static_cast<int>(g < 1 ? 1 : g);
}

// dbias[o] = sum_z dy[z, o]: one thread per o, the batch split into `chunks`
// ranges whose partial sums layer_reduce_kernel adds in a fixed order.
HT_DEV void layer_colsum_body(const float *__restrict__ dy, long long batch, long long nout, int chunks,
                              float *__restrict__ part, int blk) {
  const int gx = static_cast<int>((nout + kLayerThreads - 1) / kLayerThreads), chunk = blk / gx;
  const long long o = (blk - chunk * gx) * static_cast<long long>(kLayerThreads) + threadIdx.x;
  if (o >= nout) return;
  const long long per = (batch + chunks - 1) / chunks;
  const long long z0 = per * chunk, z1 = min(batch, z0 + per);
  float s = 0.f;
  for (long long z = z0; z < z1; ++z) s += dy[z * nout + o];
  part[static_cast<long long>(chunk) * nout + o] = s;
}
struct ColsumArgs {
  const float *dy;   // null: none
  long long batch, nout;
  int chunks;
  float *part;
};

// Blocks past P's and Q's: the column sums of a backward's dy, which ride along.
// Blocks [0, A): T1[a] = u1[a, :] b2 (r4 x r1, in shared memory, also written to
// T1g when non-null), then P[a, b, r1] for every b.  Blocks [A, A + qb): Q.
__global__ void __launch_bounds__(kLayerThreads) layer_pq_kernel(const LayerShape sh, const float *__restrict__ u1,
                                                                 const float *__restrict__ u2,
                                                                 const float *__restrict__ u3,
                                                                 const float *__restrict__ b2,
                                                                 const float *__restrict__ b1, float *__restrict__ P,
                                                                 float *__restrict__ Q, float *__restrict__ T1g,
                                                                 int npq, const ColsumArgs cs, int *clear) {
  if (blockIdx.x == 0 && threadIdx.x == 0 && clear) *clear = 0;
  if (static_cast<int>(blockIdx.x) >= npq) {
    layer_colsum_body(cs.dy, cs.batch, cs.nout, cs.chunks, cs.part, blockIdx.x - npq);
    return;
  }
  __shared__ float T1[kLayerMaxRank * kLayerMaxRank];
  const int A = sh.n[0] * sh.m[0], B = sh.n[1] * sh.m[1], C = sh.n[2] * sh.m[2];
  const int R1 = sh.r1, R2 = sh.r2, R3 = sh.r3, R4 = sh.r4;
  if (static_cast<int>(blockIdx.x) < A) {
    const int a = blockIdx.x;
    for (int e = threadIdx.x; e < R4 * R1; e += kLayerThreads) {
      const int r4 = e / R1, r1 = e - r4 * R1;
      float s = 0.f;
      for (int r3 = 0; r3 < R3; ++r3) s = fmaf(u1[a * R3 + r3], b2[(r3 * R4 + r4) * R1 + r1], s);
      T1[e] = s;
      if (T1g) T1g[static_cast<long long>(a) * R4 * R1 + e] = s;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < B * R1; e += kLayerThreads) {
      const int b = e / R1, r1 = e - b * R1;
      float s = 0.f;
      for (int r4 = 0; r4 < R4; ++r4) s = fmaf(T1[r4 * R1 + r1], u2[b * R4 + r4], s);
      P[(static_cast<long long>(a) * B + b) * R1 + r1] = s;
    }
  } else {
    const long long e = static_cast<long long>(blockIdx.x - A) * kLayerThreads + threadIdx.x;
    if (e >= static_cast<long long>(C) * R1) return;
    const int c = static_cast<int>(e / R1), r1 = static_cast<int>(e - static_cast<long long>(c) * R1);
    float s = 0.f;
    for (int r2 = 0; r2 < R2; ++r2) s = fmaf(b1[r1 * R2 + r2], u3[c * R2 + r2], s);
    Q[e] = s;
  }
}

// Where a weight goes: FP32, BF16, or the three BF16 planes of an FP32-accurate
// product (tc3_gemm.cu), the FP32 weight beside them.
struct WeightOut {
  float *w32;
  __nv_bfloat16 *w16, *w3;
  long long plane;
};
enum WeightKind : int { W_FP32 = 0, W_BF16 = 1, W_PLANES = 2 };
template <int KIND>
HT_DEV void put_weight(const WeightOut &W, long long e, float v) {
  if (KIND != W_BF16) W.w32[e] = v;
  if (KIND == W_BF16) W.w16[e] = __float2bfloat16_rn(v);
  if (KIND == W_PLANES) {
    const __nv_bfloat16 h = __float2bfloat16_rn(v);
    const float r = 128.f * (v - __bfloat162float(h));   // planes as in split_pair
    const __nv_bfloat16 m = __float2bfloat16_rn(r);
    W.w3[e] = h;
    W.w3[W.plane + e] = m;
    W.w3[2 * W.plane + e] = __float2bfloat16_rn(128.f * (r - __bfloat162float(m)));
  }
}
// An entry without planes (not finite once rounded to BF16): see split3_launch.
HT_DEV bool no_planes(float v) { return !(fabsf(__bfloat162float(__float2bfloat16_rn(v))) <= 3.4e38f); }

// W[o * Nin + i] = sum_r1 P[a, b, r1] Q[c, r1]; i = (n0 N1 + n1) N2 + n2 runs
// fastest, so consecutive threads share (a, b) and read P's row once.
template <int KIND>
__global__ void __launch_bounds__(kLayerThreads) layer_weight_kernel(const LayerShape sh, const float *__restrict__ P,
                                                                     const float *__restrict__ Q, const WeightOut W,
                                                                     int *flag) {
  const int N1 = sh.n[1], N2 = sh.n[2], M0 = sh.m[0], M1 = sh.m[1], M2 = sh.m[2];
  const long long Nin = static_cast<long long>(sh.n[0]) * N1 * N2, Nout = static_cast<long long>(M0) * M1 * M2;
  const int B = N1 * M1, R1 = sh.r1;
  for (long long e = blockIdx.x * static_cast<long long>(kLayerThreads) + threadIdx.x; e < Nin * Nout;
       e += static_cast<long long>(gridDim.x) * kLayerThreads) {
    const long long o = e / Nin, i = e - o * Nin;
    const int n2 = static_cast<int>(i % N2), n1 = static_cast<int>((i / N2) % N1), n0 = static_cast<int>(i / N2 / N1);
    const int m2 = static_cast<int>(o % M2), m1 = static_cast<int>((o / M2) % M1), m0 = static_cast<int>(o / M2 / M1);
    const int a = n0 * M0 + m0, b = n1 * M1 + m1, c = n2 * M2 + m2;
    const float *p = P + (static_cast<long long>(a) * B + b) * R1;
    const float *q = Q + static_cast<long long>(c) * R1;
    float s = 0.f;
    for (int r = 0; r < R1; ++r) s = fmaf(p[r], q[r], s);
    put_weight<KIND>(W, e, s);
    if (KIND == W_PLANES && no_planes(s)) *flag = 1;
  }
}

// The same W, a block per (m0, m1, group of G m2 rows): a thread keeps its n2 and
// the G x RB entries Q[n2 M2 + m2, :] in registers and walks the pairs, whose
// rows Ps[(n0, n1)][:] of P sit in shared memory: RB / 4 (broadcast) vector loads
// for G x RB multiply-adds, so the FMA pipe is the bound; with Q in shared memory
// its loads were (4096 x 6400 in BF16: 80 -> 63 us).  Consecutive threads write
// consecutive entries of a row.  G x RB = 64: ranks up to 64.
template <int KIND, int RB>
__global__ void __launch_bounds__(kLayerThreads, RB < 64 ? 3 : 1) layer_weight_tiled_kernel(const LayerShape sh,
                                                                           const float *__restrict__ P,
                                                                           const float *__restrict__ Q,
                                                                           const WeightOut W, int *flag) {
  constexpr int G = 64 / RB;
  extern __shared__ __align__(16) float Ps[];   // NP x RB, zero past R1; behind it Qs: N2 rows of 65
  const int N0 = sh.n[0], N1 = sh.n[1], N2 = sh.n[2], M0 = sh.m[0], M1 = sh.m[1], M2 = sh.m[2];
  const int R1 = sh.r1, B = N1 * M1, NP = N0 * N1;
  const long long Nin = static_cast<long long>(NP) * N2;
  const int groups = (M2 + G - 1) / G;
  const int gi = blockIdx.x % groups, mm = blockIdx.x / groups, m1 = mm % M1, m0 = mm / M1;
  const int m2_0 = gi * G, ng = min(G, M2 - m2_0);
  for (int e = threadIdx.x; e < NP * RB; e += kLayerThreads) {
    const int pr = e / RB, r = e % RB, n0 = pr / N1, n1 = pr - n0 * N1;
    Ps[e] = r < R1 ? P[(static_cast<long long>(n0 * M0 + m0) * B + (n1 * M1 + m1)) * R1 + r] : 0.f;
  }
  // Q's rows are G R1 contiguous entries a n2: read along them, then a row per thread
  float *Qs = Ps + NP * RB;
  for (int e = threadIdx.x; e < N2 * 64; e += kLayerThreads) {
    const int n2 = e / 64, g = (e % 64) / RB, r = e % RB;
    Qs[n2 * 65 + (e % 64)] = g < ng && r < R1 ? Q[static_cast<long long>(n2 * M2 + m2_0 + g) * R1 + r] : 0.f;
  }
  __syncthreads();
  const long long o0 = ((static_cast<long long>(m0) * M1 + m1) * M2 + m2_0) * Nin;
  bool bad = false;
  // columns of n2 in turn where a mode is wider than the block
  const int nw = min(N2, kLayerThreads), per = kLayerThreads / nw;   // pairs per sweep of the block
  const int pl = threadIdx.x / nw, nl = threadIdx.x - pl * nw;
  for (int n2 = nl; n2 < N2 && pl < per; n2 += nw) {
    constexpr int GP = (G + 1) / 2;   // rows in pairs (RB = 64: one row, its pair's second half idle)
    float2 q[RB][GP];
#pragma unroll
    for (int r = 0; r < RB; ++r)
#pragma unroll
      for (int g = 0; g < GP; ++g)
        q[r][g] = make_float2(Qs[n2 * 65 + 2 * g * RB + r], 2 * g + 1 < G ? Qs[n2 * 65 + (2 * g + 1) * RB + r] : 0.f);
    for (int p = pl; p < NP; p += per) {
      float2 acc[GP];
#pragma unroll
      for (int g = 0; g < GP; ++g) acc[g] = make_float2(0.f, 0.f);
      const float4 *ps = reinterpret_cast<const float4 *>(Ps + p * RB);
#pragma unroll
      for (int r = 0; r < RB; r += 4) {
        const float4 v = ps[r / 4];
#pragma unroll
        for (int g = 0; g < GP; ++g) {
          fma2(acc[g], make_float2(v.x, v.x), q[r][g]);
          fma2(acc[g], make_float2(v.y, v.y), q[r + 1][g]);
          fma2(acc[g], make_float2(v.z, v.z), q[r + 2][g]);
          fma2(acc[g], make_float2(v.w, v.w), q[r + 3][g]);
        }
      }
      const long long i = o0 + static_cast<long long>(p) * N2 + n2;
#pragma unroll
      for (int g = 0; g < G; ++g)
        if (g < ng) {
          const float v = g & 1 ? acc[g / 2].y : acc[g / 2].x;
          put_weight<KIND>(W, i + g * Nin, v);
          bad |= KIND == W_PLANES && no_planes(v);
        }
    }
  }
  if (KIND == W_PLANES && bad) *flag = 1;
}

// The same W with P's rows as they are and Q's group of kWeightG m2 rows beside
// them, both in shared memory, a thread with kWeightG sums for one input index: where
// the padded rows above do not fit, or cost more than they save (layer_weight_form).
// (12, 64, 32) -> (2, 8, 32) at rank 40: 0.43 ms a forward call, 1.9 with a thread
// per entry of W.
constexpr int kWeightG = 8;
template <int KIND>
__global__ void __launch_bounds__(kLayerThreads) layer_weight_packed_kernel(const LayerShape sh,
                                                                            const float *__restrict__ P,
                                                                            const float *__restrict__ Q,
                                                                            const WeightOut W, int *flag) {
  extern __shared__ __align__(16) float Ps[];   // NP x R1; behind it Qt: R1 x kWeightG x N2
  const int N0 = sh.n[0], N1 = sh.n[1], N2 = sh.n[2], M0 = sh.m[0], M1 = sh.m[1], M2 = sh.m[2];
  const int R1 = sh.r1, B = N1 * M1, NP = N0 * N1;
  const long long Nin = static_cast<long long>(NP) * N2;
  const int groups = (M2 + kWeightG - 1) / kWeightG;
  const int gi = blockIdx.x % groups, mm = blockIdx.x / groups, m1 = mm % M1, m0 = mm / M1;
  const int m2_0 = gi * kWeightG, ng = min(kWeightG, M2 - m2_0);
  float *Qt = Ps + static_cast<size_t>(NP) * R1;
  for (int e = threadIdx.x; e < NP * R1; e += kLayerThreads) {
    const int pr = e / R1, r = e - pr * R1, n0 = pr / N1, n1 = pr - n0 * N1;
    Ps[e] = P[(static_cast<long long>(n0 * M0 + m0) * B + (n1 * M1 + m1)) * R1 + r];
  }
  for (int e = threadIdx.x; e < R1 * kWeightG * N2; e += kLayerThreads) {
    const int n2 = e % N2, g = (e / N2) % kWeightG, r = e / (N2 * kWeightG);
    Qt[e] = g < ng ? Q[static_cast<long long>(n2 * M2 + m2_0 + g) * R1 + r] : 0.f;
  }
  __syncthreads();
  const long long o0 = ((static_cast<long long>(m0) * M1 + m1) * M2 + m2_0) * Nin;
  bool bad = false;
  for (long long i = threadIdx.x; i < Nin; i += kLayerThreads) {
    const int pr = static_cast<int>(i / N2), n2 = static_cast<int>(i - static_cast<long long>(pr) * N2);
    float acc[kWeightG];
#pragma unroll
    for (int g = 0; g < kWeightG; ++g) acc[g] = 0.f;
    const float *ps = Ps + static_cast<size_t>(pr) * R1;
    for (int r = 0; r < R1; ++r) {
      const float pv = ps[r];
      const float *q = Qt + static_cast<size_t>(r) * kWeightG * N2 + n2;
#pragma unroll
      for (int g = 0; g < kWeightG; ++g) acc[g] = fmaf(pv, q[g * N2], acc[g]);
    }
#pragma unroll
    for (int g = 0; g < kWeightG; ++g)
      if (g < ng) {
        put_weight<KIND>(W, o0 + g * Nin + i, acc[g]);
        bad |= KIND == W_PLANES && no_planes(acc[g]);
      }
  }
  if (KIND == W_PLANES && bad) *flag = 1;
}

// y[z, o] = act(y[z, o] + bias[o]), act 0 = identity, 1 = ReLU
__global__ void bias_act_kernel(float *__restrict__ y, const float *__restrict__ bias, long long batch, long long nout,
                                int act) {
  for (long long e = blockIdx.x * static_cast<long long>(kLayerThreads) + threadIdx.x; e < batch * nout;
       e += static_cast<long long>(gridDim.x) * kLayerThreads) {
    float v = y[e];
    if (bias) v += bias[e % nout];
    if (act == 1) v = fmaxf(v, 0.f);
    y[e] = v;
  }
}

// dP[a, b, r1] = sum_{n2, m2} dW[o, i] Q[c, r1] and, in the same pass over dW,
// per-(a, b) block contributions to dQ.  One block per (a, b): the M2 x N2
// sub-block of dW it owns is staged in shared memory.
//   dQpart[(a, b), c, r1] is not formed: dQ is summed by layer_dq_kernel.
__global__ void __launch_bounds__(kLayerThreads) layer_dp_kernel(const LayerShape sh, const float *__restrict__ dW,
                                                                 const float *__restrict__ Q, float *__restrict__ dP) {
  extern __shared__ float sm[];
  const int N1 = sh.n[1], N2 = sh.n[2], M0 = sh.m[0], M1 = sh.m[1], M2 = sh.m[2];
  const long long Nin = static_cast<long long>(sh.n[0]) * N1 * N2;
  const int B = N1 * M1, C = N2 * M2, R1 = sh.r1;
  const int ab = blockIdx.x, a = ab / B, b = ab - a * B;
  const int n0 = a / M0, m0 = a - n0 * M0, n1 = b / M1, m1 = b - n1 * M1;
  float *blk = sm;   // [c = n2 M2 + m2]
  for (int e = threadIdx.x; e < C; e += kLayerThreads) {
    const int n2 = e / M2, m2 = e - n2 * M2;
    const long long o = (static_cast<long long>(m0) * M1 + m1) * M2 + m2;
    const long long i = (static_cast<long long>(n0) * N1 + n1) * N2 + n2;
    blk[e] = dW[o * Nin + i];
  }
  __syncthreads();
  for (int r1 = threadIdx.x; r1 < R1; r1 += kLayerThreads) {
    float s = 0.f;
    for (int c = 0; c < C; ++c) s = fmaf(blk[c], Q[static_cast<long long>(c) * R1 + r1], s);
    dP[static_cast<long long>(ab) * R1 + r1] = s;
  }
}

// dQ[c, r1] = sum_{a, b} dW[o, i] P[a, b, r1]: one block per c, the (a, b)
// range split over the threads, a fixed-order tree reduction at the end.
__global__ void __launch_bounds__(kLayerThreads) layer_dq_kernel(const LayerShape sh, const float *__restrict__ dW,
                                                                 const float *__restrict__ P, float *__restrict__ dQ) {
  __shared__ float red[kLayerThreads / 32][kLayerMaxRank];
  const int N1 = sh.n[1], N2 = sh.n[2], M0 = sh.m[0], M1 = sh.m[1], M2 = sh.m[2];
  const long long Nin = static_cast<long long>(sh.n[0]) * N1 * N2;
  const int A = sh.n[0] * M0, B = N1 * M1, R1 = sh.r1;
  const int c = blockIdx.x, n2 = c / M2, m2 = c - n2 * M2;
  float acc[kLayerMaxRank];
#pragma unroll
  for (int r = 0; r < kLayerMaxRank; ++r) acc[r] = 0.f;
  for (int ab = threadIdx.x; ab < A * B; ab += kLayerThreads) {
    const int a = ab / B, b = ab - a * B;
    const int n0 = a / M0, m0 = a - n0 * M0, n1 = b / M1, m1 = b - n1 * M1;
    const long long o = (static_cast<long long>(m0) * M1 + m1) * M2 + m2;
    const long long i = (static_cast<long long>(n0) * N1 + n1) * N2 + n2;
    const float g = dW[o * Nin + i];
    const float *p = P + static_cast<long long>(ab) * R1;
#pragma unroll
    for (int r = 0; r < kLayerMaxRank; ++r)
      if (r < R1) acc[r] = fmaf(g, p[r], acc[r]);
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int r = 0; r < kLayerMaxRank; ++r) {
    float v = acc[r];
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    if (lane == 0) red[warp][r] = v;
  }
  __syncthreads();
  for (int r = threadIdx.x; r < R1; r += kLayerThreads) {
    float s = 0.f;
    for (int w = 0; w < kLayerThreads / 32; ++w) s += red[w][r];
    dQ[static_cast<long long>(c) * R1 + r] = s;
  }
}

// dP and per-block dQ partials in one pass over dW, a block per (m0, m1) and
// range of m2 (several ranges give dP partials, summed afterwards): the block
// reads its rows o = (m0 M1 + m1) M2 + m2 of dW (coalesced, staged in
// shared memory with an odd pair stride), and with Q (C x R1) and the P slice
// Ps[(n0, n1)][r] resident accumulates
//   dPs[r][(n0, n1)] += sum_n2 dW[o, (n0, n1, n2)] Q[n2 M2 + m2, r]
//   dQpart[blk][n2 M2 + m2][r] = sum_(n0, n1) dW[o, (n0, n1, n2)] Ps[(n0, n1)][r].
// Bound by shared-memory loads, so both products keep a row of outputs in
// registers: dP a thread per pair and RT ranks (one load of the row and RT / 4
// broadcast vectors of Q for RT multiply-adds), dQ a lane per n2 and 16 ranks
// with the pairs spread over the warps (and, for N2 <= 16, over groups of
// lanes), whose partial sums are added in warp order.  With one output per
// thread and two loads per multiply-add the pass over a 6400 x 4096 dW took 454
// us; now 145.  Every sum has a fixed order.
constexpr int kDqRanks = 16;
constexpr int kDqRed = 17;   // floats per lane of the partial sums (odd: no bank conflicts)
template <int RT>
__global__ void __launch_bounds__(kLayerThreads) layer_dpq_kernel(const LayerShape sh, const float *__restrict__ dW,
                                                                  const float *__restrict__ P,
                                                                  const float *__restrict__ Q,
                                                                  float *__restrict__ dP,
                                                                  float *__restrict__ dQpart) {
  extern __shared__ __align__(16) float sm[];
  const int N0 = sh.n[0], N1 = sh.n[1], N2 = sh.n[2], M0 = sh.m[0], M1 = sh.m[1], M2 = sh.m[2];
  const int R1 = sh.r1, RP = (R1 + 3) & ~3, B = N1 * M1, NP = N0 * N1, C = N2 * M2;
  const int rs = N2 | 1;                             // odd stride between pairs: conflict-free column reads
  const long long Nin = static_cast<long long>(NP) * N2;
  const int chunks = gridDim.x / (M0 * M1);             // m2 ranges per (m0, m1): dP partials per range
  const int blk = blockIdx.x / chunks, ch = blockIdx.x - blk * chunks, m1 = blk % M1, m0 = blk / M1;
  const int mg = (M2 + chunks - 1) / chunks, m2_lo = ch * mg, m2_hi = min(M2, m2_lo + mg);
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  float *Qs = sm;                                              // C x RP
  float *Ps = Qs + static_cast<size_t>(C) * RP;                // NP x RP, then 64 spare floats
  float *dPs = Ps + static_cast<size_t>(NP) * RP + 64;         // R1 x NP
  float *red = dPs + static_cast<size_t>(R1) * NP;             // 256 x kDqRed
  float *row = red + kLayerThreads * kDqRed;                   // NP x rs
  for (int e = t; e < C * RP; e += kLayerThreads) {
    const int c = e / RP, r = e - c * RP;
    Qs[e] = r < R1 ? Q[static_cast<long long>(c) * R1 + r] : 0.f;
  }
  for (int e = t; e < NP * RP; e += kLayerThreads) {
    const int pr = e / RP, r = e - pr * RP, n0 = pr / N1, n1 = pr - n0 * N1;
    Ps[e] = r < R1 ? P[(static_cast<long long>(n0 * M0 + m0) * B + (n1 * M1 + m1)) * R1 + r] : 0.f;
  }
  for (int e = t; e < 64; e += kLayerThreads) Ps[NP * RP + e] = 0.f;
  for (int e = t; e < NP * R1; e += kLayerThreads) dPs[e] = 0.f;
  const int dp = kLayerThreads / N2, dn = kLayerThreads - dp * N2;   // steps of (pair, n2) between a thread's entries
  const int nl = min(N2, 32), psub = 32 / nl, ps = lane / nl, ln = lane - ps * nl;
  for (int m2 = m2_lo; m2 < m2_hi; ++m2) {
    __syncthreads();   // previous row fully consumed (and Qs / Ps written on the first pass)
    const float *src = dW + ((static_cast<long long>(m0) * M1 + m1) * M2 + m2) * Nin;
    int pr = t / N2, n2 = t - pr * N2;
    for (long long i = t; i < Nin; i += kLayerThreads) {
      // (asynchronous: every entry of the row is in flight at once)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(row + pr * rs + n2)), "l"(src + i) : "memory");
      pr += dp;
      n2 += dn;
      if (n2 >= N2) {
        n2 -= N2;
        ++pr;
      }
    }
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    for (int e = t; e < NP * ((R1 + RT - 1) / RT); e += kLayerThreads) {
      const int g = e / NP, q = e - g * NP, r0 = g * RT;
      const float *rw = row + q * rs, *qv = Qs + static_cast<size_t>(m2) * RP + r0;
      float2 acc[RT / 2];
#pragma unroll
      for (int r = 0; r < RT / 2; ++r) acc[r] = make_float2(0.f, 0.f);
      for (int c = 0; c < N2; ++c, qv += static_cast<size_t>(M2) * RP) {
        const float x = rw[c];
#pragma unroll
        for (int r = 0; r < RT; r += 4) {   // (vectors past RP read the next row's: their sums are dropped)
          const float4 v = *reinterpret_cast<const float4 *>(qv + r);
          fma2(acc[r / 2], make_float2(x, x), make_float2(v.x, v.y));
          fma2(acc[r / 2 + 1], make_float2(x, x), make_float2(v.z, v.w));
        }
      }
#pragma unroll
      for (int r = 0; r < RT; ++r)
        if (r0 + r < R1) dPs[(r0 + r) * NP + q] += r & 1 ? acc[r / 2].y : acc[r / 2].x;
    }
    for (int nc = 0; nc < N2; nc += 32)
      for (int r0 = 0; r0 < R1; r0 += kDqRanks) {
        float2 acc[kDqRanks / 2];
#pragma unroll
        for (int r = 0; r < kDqRanks / 2; ++r) acc[r] = make_float2(0.f, 0.f);
        if (ps < psub && nc + ln < N2) {
          for (int q = warp * psub + ps; q < NP; q += 8 * psub) {
            const float x = row[q * rs + nc + ln];
            const float *pv = Ps + static_cast<size_t>(q) * RP + r0;
#pragma unroll
            for (int r = 0; r < kDqRanks; r += 4) {
              const float4 v = *reinterpret_cast<const float4 *>(pv + r);
              fma2(acc[r / 2], make_float2(x, x), make_float2(v.x, v.y));
              fma2(acc[r / 2 + 1], make_float2(x, x), make_float2(v.z, v.w));
            }
          }
        }
#pragma unroll
        for (int r = 0; r < kDqRanks; ++r) red[t * kDqRed + r] = r & 1 ? acc[r / 2].y : acc[r / 2].x;
        __syncthreads();
        const int nn = min(nl, N2 - nc), nr = min(kDqRanks, R1 - r0);
        for (int e = t; e < nn * nr; e += kLayerThreads) {
          const int k = e / nr, r = e - k * nr;
          float s = 0.f;
          for (int w = 0; w < 8; ++w)
            for (int g = 0; g < psub; ++g) s += red[(w * 32 + g * nl + k) * kDqRed + r];
          dQpart[(static_cast<long long>(blk) * C + ((nc + k) * M2 + m2)) * R1 + r0 + r] = s;
        }
        __syncthreads();
      }
  }
  __syncthreads();
  // chunks > 1: dP points at the partial buffer [chunks][A B R1]
  float *dPo = dP + static_cast<long long>(ch) * (static_cast<long long>(sh.n[0]) * M0 * B * R1);
  for (int e = t; e < NP * R1; e += kLayerThreads) {
    const int pr = e / R1, r = e - pr * R1, n0 = pr / N1, n1 = pr - n0 * N1;
    dPo[(static_cast<long long>(n0 * M0 + m0) * B + (n1 * M1 + m1)) * R1 + r] = dPs[r * NP + pr];
  }
}

// The same pass without padding and without partial sums in shared memory, an
// output of either product per thread and step, where the kernel above does not fit
// or has too few pairs to keep its threads busy (layer_dpq_form).
__global__ void __launch_bounds__(kLayerThreads) layer_dpq_packed_kernel(const LayerShape sh,
                                                                         const float *__restrict__ dW,
                                                                         const float *__restrict__ P,
                                                                         const float *__restrict__ Q,
                                                                         float *__restrict__ dP,
                                                                         float *__restrict__ dQpart) {
  extern __shared__ __align__(16) float sm[];
  const int N0 = sh.n[0], N1 = sh.n[1], N2 = sh.n[2], M0 = sh.m[0], M1 = sh.m[1], M2 = sh.m[2];
  const int R1 = sh.r1, B = N1 * M1, NP = N0 * N1, C = N2 * M2;
  const int rs = N2 | 1;                             // odd stride between pairs: conflict-free column reads
  const long long Nin = static_cast<long long>(NP) * N2;
  const int chunks = gridDim.x / (M0 * M1);          // m2 ranges per (m0, m1): dP partials per range
  const int blk = blockIdx.x / chunks, ch = blockIdx.x - blk * chunks, m1 = blk % M1, m0 = blk / M1;
  const int mg = (M2 + chunks - 1) / chunks, m2_lo = ch * mg, m2_hi = min(M2, m2_lo + mg);
  float *row = sm;                                   // NP x rs
  float *Qs = row + static_cast<size_t>(NP) * rs;    // C x R1
  float *Ps = Qs + static_cast<size_t>(C) * R1;      // NP x R1
  float *dPs = Ps + static_cast<size_t>(NP) * R1;    // NP x R1
  for (int e = threadIdx.x; e < C * R1; e += kLayerThreads) Qs[e] = Q[e];
  for (int e = threadIdx.x; e < NP * R1; e += kLayerThreads) {
    const int pr = e / R1, r = e - pr * R1, n0 = pr / N1, n1 = pr - n0 * N1;
    Ps[e] = P[(static_cast<long long>(n0 * M0 + m0) * B + (n1 * M1 + m1)) * R1 + r];
    dPs[e] = 0.f;
  }
  for (int m2 = m2_lo; m2 < m2_hi; ++m2) {
    __syncthreads();   // previous row fully consumed (and Qs / Ps written on the first pass)
    const float *src = dW + ((static_cast<long long>(m0) * M1 + m1) * M2 + m2) * Nin;
    for (long long i = threadIdx.x; i < Nin; i += kLayerThreads) {
      const int pr = static_cast<int>(i / N2), n2 = static_cast<int>(i - static_cast<long long>(pr) * N2);
      row[pr * rs + n2] = src[i];
    }
    __syncthreads();
    for (int e = threadIdx.x; e < NP * R1; e += kLayerThreads) {
      const int pr = e / R1, r = e - pr * R1;
      const float *rw = row + pr * rs;
      float s = dPs[e];
      for (int n2 = 0; n2 < N2; ++n2) s = fmaf(rw[n2], Qs[(n2 * M2 + m2) * R1 + r], s);
      dPs[e] = s;
    }
    for (int e = threadIdx.x; e < N2 * R1; e += kLayerThreads) {
      const int r = e / N2, n2 = e - r * N2;
      float s[4] = {0.f, 0.f, 0.f, 0.f};   // four independent chains, combined in a fixed order
      int pr = 0;
      for (; pr + 4 <= NP; pr += 4)
#pragma unroll
        for (int j = 0; j < 4; ++j) s[j] = fmaf(row[(pr + j) * rs + n2], Ps[(pr + j) * R1 + r], s[j]);
      for (; pr < NP; ++pr) s[0] = fmaf(row[pr * rs + n2], Ps[pr * R1 + r], s[0]);
      dQpart[(static_cast<long long>(blk) * C + (n2 * M2 + m2)) * R1 + r] = (s[0] + s[1]) + (s[2] + s[3]);
    }
  }
  __syncthreads();
  // chunks > 1: dP points at the partial buffer [chunks][A B R1]
  float *dPo = dP + static_cast<long long>(ch) * (static_cast<long long>(sh.n[0]) * M0 * B * R1);
  for (int e = threadIdx.x; e < NP * R1; e += kLayerThreads) {
    const int pr = e / R1, r = e - pr * R1, n0 = pr / N1, n1 = pr - n0 * N1;
    dPo[(static_cast<long long>(n0 * M0 + m0) * B + (n1 * M1 + m1)) * R1 + r] = dPs[e];
  }
}

// Sums of partials in a fixed order, several arrays in one launch: out[e] = sum
// over k < n of part[k * count + e].  Few partials (dP): a thread per output.
// Many (dQ, dbias): 32 outputs a block, each warp one contiguous eighth of the
// partials, the eighths added in order.
struct SumJob {
  const float *part;
  float *out;
  long long count;
  int n, blocks;
};
struct SumJobs {
  SumJob j[3];
};
__global__ void __launch_bounds__(kLayerThreads) layer_reduce_kernel(const SumJobs jobs) {
  __shared__ float red[8][32];
  int blk = blockIdx.x, i = 0;
  while (i < 2 && blk >= jobs.j[i].blocks) blk -= jobs.j[i++].blocks;
  const SumJob J = jobs.j[i];
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  if (J.n < 16) {
    const long long e = blk * static_cast<long long>(kLayerThreads) + t;
    if (e >= J.count) return;
    float s = 0.f;
    for (int k = 0; k < J.n; ++k) s += J.part[k * J.count + e];
    J.out[e] = s;
    return;
  }
  const long long e = blk * 32ll + lane;
  const int per = (J.n + 7) / 8, k1 = min(J.n, (warp + 1) * per);
  float s = 0.f;
  if (e < J.count)
    for (int k = warp * per; k < k1; ++k) s += J.part[k * J.count + e];
  red[warp][lane] = s;
  __syncthreads();
  if (warp == 0 && e < J.count) {
    for (int w = 1; w < 8; ++w) s += red[w][lane];
    J.out[e] = s;
  }
}
int sum_blocks(int n, long long count) {
  return static_cast<int>(n < 16 ? (count + kLayerThreads - 1) / kLayerThreads : (count + 31) / 32);
}

// dT1[a, r4, r1] = sum_b u2[b, r4] dP[a, b, r1]: a block per a, the b range
// staged through shared memory in chunks of kDtChunk rows of dP[a] and u2,
// each thread owning fixed (r4, r1) outputs.  Blocks [A, A + du3 blocks):
// du3[c, r2] = sum_r1 dQ[c, r1] b1[r1, r2], a thread per entry.
constexpr int kDtChunk = 64;
HT_DEV void layer_dt1_body(const LayerShape &sh, const float *__restrict__ u2, const float *__restrict__ b1,
                           const float *__restrict__ dP, const float *__restrict__ dQ, float *__restrict__ dT1,
                           float *__restrict__ du3, int blk, float *smem) {
  const int A = sh.n[0] * sh.m[0], B = sh.n[1] * sh.m[1], C = sh.n[2] * sh.m[2];
  const int R1 = sh.r1, R2 = sh.r2, R4 = sh.r4, t = threadIdx.x;
  if (static_cast<int>(blk) >= A) {
    const long long f = (blk - A) * static_cast<long long>(kLayerThreads) + t;
    if (f >= static_cast<long long>(C) * R2) return;
    const int c = static_cast<int>(f / R2), r2 = static_cast<int>(f - static_cast<long long>(c) * R2);
    float v = 0.f;
    for (int r1 = 0; r1 < R1; ++r1) v = fmaf(dQ[static_cast<long long>(c) * R1 + r1], b1[r1 * R2 + r2], v);
    du3[f] = v;
    return;
  }
  float *sP = smem;                                  // [b][r1]
  float *sU = smem + kDtChunk * kLayerMaxRank;       // [b][r4]
  constexpr int kOut = kLayerMaxRank * kLayerMaxRank / kLayerThreads;
  const int a = blk, nout = R4 * R1;
  float acc[kOut];
#pragma unroll
  for (int q = 0; q < kOut; ++q) acc[q] = 0.f;
  for (int b0 = 0; b0 < B; b0 += kDtChunk) {
    const int nb = min(kDtChunk, B - b0);
    __syncthreads();
    for (int e = t; e < nb * R1; e += kLayerThreads) sP[e] = dP[(static_cast<long long>(a) * B + b0) * R1 + e];
    for (int e = t; e < nb * R4; e += kLayerThreads) sU[e] = u2[static_cast<long long>(b0) * R4 + e];
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kOut; ++q) {
      const int o = t + q * kLayerThreads;
      if (o < nout) {
        const int r4 = o / R1, r1 = o - r4 * R1;
        float v = acc[q];
        for (int b = 0; b < nb; ++b) v = fmaf(sU[b * R4 + r4], sP[b * R1 + r1], v);
        acc[q] = v;
      }
    }
  }
#pragma unroll
  for (int q = 0; q < kOut; ++q) {
    const int o = t + q * kLayerThreads;
    if (o < nout) dT1[static_cast<long long>(a) * nout + o] = acc[q];
  }
}

// du1[a, r3] = sum_q dT1[a, q] b2[r3, q] (q = (r4, r1)): a warp per entry,
// lanes striding q, a fixed shuffle tree.  Blocks past the du1 ones:
// db2[r3, q] = sum_a u1[a, r3] dT1[a, q], a thread per entry with four
// independent chains over a combined in a fixed order.
__global__ void __launch_bounds__(kLayerThreads) layer_dt1_back_kernel(const LayerShape sh, const float *__restrict__ u1,
                                                                       const float *__restrict__ b2,
                                                                       const float *__restrict__ dT1,
                                                                       float *__restrict__ du1,
                                                                       float *__restrict__ db2, int du1_blocks) {
  const int A = sh.n[0] * sh.m[0];
  const int R1 = sh.r1, R3 = sh.r3, R4 = sh.r4, Qn = R4 * R1;
  if (static_cast<int>(blockIdx.x) < du1_blocks) {
    const long long w = blockIdx.x * static_cast<long long>(kLayerThreads / 32) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (w >= static_cast<long long>(A) * R3) return;
    const int a = static_cast<int>(w / R3), r3 = static_cast<int>(w - static_cast<long long>(a) * R3);
    const float *d = dT1 + static_cast<long long>(a) * Qn;
    const float *g = b2 + static_cast<long long>(r3) * Qn;
    float v = 0.f;
    for (int q = lane; q < Qn; q += 32) v = fmaf(d[q], g[q], v);
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    if (lane == 0) du1[w] = v;
    return;
  }
  const long long f = (blockIdx.x - du1_blocks) * static_cast<long long>(kLayerThreads) + threadIdx.x;
  if (f >= static_cast<long long>(R3) * Qn) return;
  const int r3 = static_cast<int>(f / Qn), q = static_cast<int>(f - static_cast<long long>(r3) * Qn);
  float s[4] = {0.f, 0.f, 0.f, 0.f};
  int a = 0;
  for (; a + 4 <= A; a += 4)
#pragma unroll
    for (int j = 0; j < 4; ++j) s[j] = fmaf(u1[(a + j) * R3 + r3], dT1[static_cast<long long>(a + j) * Qn + q], s[j]);
  for (; a < A; ++a) s[0] = fmaf(u1[a * R3 + r3], dT1[static_cast<long long>(a) * Qn + q], s[0]);
  db2[f] = (s[0] + s[1]) + (s[2] + s[3]);
}

// The factor gradients from dP, dQ (all small):
//   du3[c, r2] = sum_r1 dQ[c, r1] b1[r1, r2]        db1[r1, r2] = sum_c dQ[c, r1] u3[c, r2]
//   dT1[a, r4, r1] = sum_b dP[a, b, r1] u2[b, r4]   du2[b, r4] = sum_{a, r1} dP[a, b, r1] T1[a, r4, r1]
//   du1[a, r3] = sum_{r4, r1} dT1[a, r4, r1] b2[r3, r4, r1]
//   db2[r3, r4, r1] = sum_a u1[a, r3] dT1[a, r4, r1]
// dT1, du3, du2 and db1 come from layer_grads_kernel, a block range each; du1 and
// db2, which need all of dT1, from layer_dt1_back_kernel.
// du2[b, r4] = sum_{a, r1} dP[a, b, r1] T1[a, r4, r1]: a block per b, the
// (a, r1) pairs split over the threads with R4 accumulators each, then a
// fixed-order reduction (deterministic).
template <int RB>   // rank bound: R4 <= RB
HT_DEV void layer_du2_body(const LayerShape &sh, const float *__restrict__ dP, const float *__restrict__ T1,
                           float *__restrict__ du2, int blk, float *smem) {
  float (*red)[RB] = reinterpret_cast<float (*)[RB]>(smem);
  const int A = sh.n[0] * sh.m[0], B = sh.n[1] * sh.m[1];
  const int R1 = sh.r1, R4 = sh.r4, b = blk;
  float acc[RB];
#pragma unroll
  for (int r = 0; r < RB; ++r) acc[r] = 0.f;
  for (int e = threadIdx.x; e < A * R1; e += kLayerThreads) {
    const int a = e / R1, r1 = e - a * R1;
    const float g = dP[(static_cast<long long>(a) * B + b) * R1 + r1];
    const float *t = T1 + static_cast<long long>(a) * R4 * R1 + r1;
#pragma unroll
    for (int r = 0; r < RB; ++r)
      if (r < R4) acc[r] = fmaf(g, t[r * R1], acc[r]);
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int r = 0; r < RB; ++r) {
    float v = acc[r];
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    if (lane == 0) red[warp][r] = v;
  }
  __syncthreads();
  for (int r = threadIdx.x; r < R4; r += kLayerThreads) {
    float v = 0.f;
    for (int w = 0; w < kLayerThreads / 32; ++w) v += red[w][r];
    du2[static_cast<long long>(b) * R4 + r] = v;
  }
}

// db1[r1, r2] = sum_c dQ[c, r1] u3[c, r2]: a block per r1, c split over the
// threads with R2 accumulators each, fixed-order reduction.
template <int RB>   // rank bound: R2 <= RB
HT_DEV void layer_db1_body(const LayerShape &sh, const float *__restrict__ dQ, const float *__restrict__ u3,
                           float *__restrict__ db1, int blk, float *smem) {
  float (*red)[RB] = reinterpret_cast<float (*)[RB]>(smem);
  const int C = sh.n[2] * sh.m[2], R1 = sh.r1, R2 = sh.r2, r1 = blk;
  float acc[RB];
#pragma unroll
  for (int r = 0; r < RB; ++r) acc[r] = 0.f;
  for (int c = threadIdx.x; c < C; c += kLayerThreads) {
    const float g = dQ[static_cast<long long>(c) * R1 + r1];
    const float *u = u3 + static_cast<long long>(c) * R2;
#pragma unroll
    for (int r = 0; r < RB; ++r)
      if (r < R2) acc[r] = fmaf(g, u[r], acc[r]);
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int r = 0; r < RB; ++r) {
    float v = acc[r];
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    if (lane == 0) red[warp][r] = v;
  }
  __syncthreads();
  for (int r = threadIdx.x; r < R2; r += kLayerThreads) {
    float v = 0.f;
    for (int w = 0; w < kLayerThreads / 32; ++w) v += red[w][r];
    db1[static_cast<long long>(r1) * R2 + r] = v;
  }
}

template <int RB>   // rank bound: R2, R4 <= RB
HT_DEV void layer_grads_body(const LayerShape &sh, const float *__restrict__ u2, const float *__restrict__ u3,
                             const float *__restrict__ b1, const float *__restrict__ T1, const float *__restrict__ dP,
                             const float *__restrict__ dQ, float *__restrict__ dT1, float *__restrict__ du2,
                             float *__restrict__ du3, float *__restrict__ db1, int nb_du2, int nb_dt1) {
  __shared__ float smem[2 * kDtChunk * kLayerMaxRank];
  const int blk = blockIdx.x;
  if (blk < nb_du2) layer_du2_body<RB>(sh, dP, T1, du2, blk, smem);
  else if (blk < nb_du2 + nb_dt1) layer_dt1_body(sh, u2, b1, dP, dQ, dT1, du3, blk - nb_du2, smem);
  else layer_db1_body<RB>(sh, dQ, u3, db1, blk - nb_du2 - nb_dt1, smem);
}

template <int RB>
__global__ void __launch_bounds__(kLayerThreads) layer_grads_kernel(
    const LayerShape sh, const float *__restrict__ u2, const float *__restrict__ u3, const float *__restrict__ b1,
    const float *__restrict__ T1, const float *__restrict__ dP, const float *__restrict__ dQ, float *__restrict__ dT1,
    float *__restrict__ du2, float *__restrict__ du3, float *__restrict__ db1, int nb_du2, int nb_dt1) {
  layer_grads_body<RB>(sh, u2, u3, b1, T1, dP, dQ, dT1, du2, du3, db1, nb_du2, nb_dt1);
}
// du2's RB loads of T1 should all be in flight.  Left to itself the compiler gives
// RB = 32 64 registers, and the kernel then took up to twice as long (A = 256, B = 64,
// rank 32: 287 us a backward, 176 with the 128 registers of two CTAs an SM); at 16
// the bound only costs (up to 1.2 x), at 64 it changes nothing.
__global__ void __launch_bounds__(kLayerThreads, 2) layer_grads32_kernel(
    const LayerShape sh, const float *__restrict__ u2, const float *__restrict__ u3, const float *__restrict__ b1,
    const float *__restrict__ T1, const float *__restrict__ dP, const float *__restrict__ dQ, float *__restrict__ dT1,
    float *__restrict__ du2, float *__restrict__ du3, float *__restrict__ db1, int nb_du2, int nb_dt1) {
  layer_grads_body<32>(sh, u2, u3, b1, T1, dP, dQ, dT1, du2, du3, db1, nb_du2, nb_dt1);
}

}  // namespace

cudaError_t layer_pq_launch(const LayerShape &sh, const float *u1, const float *u2, const float *u3, const float *b2,
                            const float *b1, float *P, float *Q, float *T1, cudaStream_t s, int *clear,
                            const float *dy, long long batch, float *cpart) {
  const int A = sh.n[0] * sh.m[0], C = sh.n[2] * sh.m[2];
  const long long qb = (static_cast<long long>(C) * sh.r1 + kLayerThreads - 1) / kLayerThreads;
  const ColsumArgs cs{dy, batch, static_cast<long long>(sh.m[0]) * sh.m[1] * sh.m[2], layer_colsum_chunks(batch), cpart};
  const long long ncol = dy ? (cs.nout + kLayerThreads - 1) / kLayerThreads * cs.chunks : 0;
  layer_pq_kernel<<<static_cast<unsigned>(A + qb + ncol), kLayerThreads, 0, s>>>(sh, u1, u2, u3, b2, b1, P, Q, T1,
                                                                                static_cast<int>(A + qb), cs, clear);
  return cudaGetLastError();
}

// Rank bound of the tiled weight kernel's instantiation.
int layer_weight_rb(const LayerShape &sh) { return sh.r1 <= 16 ? 16 : (sh.r1 <= 32 ? 32 : 64); }
size_t layer_weight_smem(const LayerShape &sh) {
  return sizeof(float) * (static_cast<size_t>(sh.n[0]) * sh.n[1] * layer_weight_rb(sh) + static_cast<size_t>(sh.n[2]) * 65);
}
size_t layer_weight_packed_smem(const LayerShape &sh) {
  return sizeof(float) * (static_cast<size_t>(sh.n[0]) * sh.n[1] * sh.r1 +
                          static_cast<size_t>(sh.r1) * kWeightG * sh.n[2]);
}

size_t layer_dpq_smem(const LayerShape &sh) {
  const size_t NP = static_cast<size_t>(sh.n[0]) * sh.n[1], C = static_cast<size_t>(sh.n[2]) * sh.m[2];
  const size_t RP = (sh.r1 + 3) & ~3;
  return sizeof(float) *
         (NP * (sh.n[2] | 1) + C * RP + NP * RP + 64 + NP * sh.r1 + static_cast<size_t>(kLayerThreads) * kDqRed);
}
size_t layer_dpq_packed_smem(const LayerShape &sh) {
  const size_t NP = static_cast<size_t>(sh.n[0]) * sh.n[1], C = static_cast<size_t>(sh.n[2]) * sh.m[2];
  return sizeof(float) * (NP * (sh.n[2] | 1) + C * sh.r1 + 2 * NP * sh.r1);
}

constexpr size_t kLayerSmemMax = 200 * 1024, kDpqSmemMax = 224 * 1024;

// Which kernel forms W: the one whose estimated time (us) is the least.  The tiled
// kernel's groups hold 64 / RB rows of W, so at ranks above 16, short N2 and many
// pairs it mostly stages P; the packed one holds eight rows at any rank but has an
// eighth of the threads' work per load; a thread per entry is for weights too few
// to fill the SMs with blocks.  The coefficients are a fit to whole calls on 2617
// shapes (8 to 4096 pairs, N2 of 2 to 800, ranks 2 to 64; median error 12 %); the
// choice takes 1.01 x the best one's time on average, 1.6 x at worst, where tiled
// wherever it fits took 1.22 x and up to 12 x ((12, 64, 8) -> (8, 8, 16) at rank 33:
// 531 us against 133 packed, 217 by entry).
enum WeightForm : int { WEIGHT_TILED, WEIGHT_PACKED, WEIGHT_ENTRIES };
WeightForm layer_weight_form(const LayerShape &sh) {
  const double pairs = static_cast<double>(sh.n[0]) * sh.n[1], n2 = sh.n[2], r = sh.r1;
  const double m01 = static_cast<double>(sh.m[0]) * sh.m[1], entries = pairs * n2 * m01 * sh.m[2];
  const int rb = layer_weight_rb(sh), G = 64 / rb;
  auto waves = [&](int rows) { return std::ceil(m01 * ((sh.m[2] + rows - 1) / rows) / device_sm_count()); };
  double tiled = 1e300, packed = 1e300;
  if (layer_weight_smem(sh) <= kLayerSmemMax)
    tiled = waves(G) * (8.7e-4 * pairs * rb + 7.9e-4 * pairs * n2 + 6.3e-3 * n2 + 0.084);
  if (layer_weight_packed_smem(sh) <= kLayerSmemMax)
    packed = waves(kWeightG) * (7.3e-4 * pairs * r + 2.0e-4 * pairs * n2 * r + 5.2e-4 * pairs * n2 + 6.1e-3 * r * n2);
  const double by_entry = entries * (1.8e-6 * r + 6.7e-7);
  if (tiled <= packed && tiled <= by_entry) return WEIGHT_TILED;
  return packed <= by_entry ? WEIGHT_PACKED : WEIGHT_ENTRIES;
}

// Which of the two fused passes forms dP and dQ.  The tiled one keeps more outputs
// per thread, but pads the ranks to four, holds 17 KB of partial sums and has work
// for pairs x ranks / RT threads only.  Measured against each other over 597 shapes
// (2 to 256 pairs, N2 of 8 to 128, ranks 3 to 64; whole backward calls, with the
// tiled pass up to 2 x as fast at 256 pairs): the packed one is the faster
//   * up to 48 pairs (median 1.02 to 1.1 x, up to 2.9 x where it also lets more
//     CTAs share an SM: (4, 4, 128) -> (8, 8, 64) at rank 5, 1126 us unfused, 614),
//   * up to 128 pairs where twice as many of its CTAs fit an SM, or where the blocks
//     have a row or two each and their setup counts (1.04 to 1.15 x).
// Where the tiled pass does not fit, the packed one is 2 to 4 x as fast as none.
enum DpqForm : int { DPQ_NONE = 0, DPQ_TILED = 1, DPQ_PACKED = 2 };
DpqForm layer_dpq_form(const LayerShape &sh) {
  const size_t st = layer_dpq_smem(sh), sp = layer_dpq_packed_smem(sh);
  if (sp > kLayerSmemMax) return st <= kDpqSmemMax ? DPQ_TILED : DPQ_NONE;
  if (st > kDpqSmemMax) return DPQ_PACKED;
  const long long pairs = static_cast<long long>(sh.n[0]) * sh.n[1];
  const long long rows = static_cast<long long>(sh.m[0]) * sh.m[1] * sh.m[2];
  auto ctas = [](size_t smem) { return std::min<size_t>(8, 227 * 1024 / (smem + 1024)); };   // that share an SM
  const bool packed = pairs <= 48 || (pairs <= 128 && (ctas(sp) >= 2 * ctas(st) || rows <= 2 * device_sm_count()));
  return packed ? DPQ_PACKED : DPQ_TILED;
}

template <class K>
cudaError_t allow_smem(K kernel, size_t bytes) {
  if (bytes <= 48 * 1024) return cudaSuccess;
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
}

// Where the packed kernel's blocks (eight rows of W each) leave SMs idle, the planes'
// three more stores an entry lengthen it, and with few columns the CUDA cores'
// product costs less than that: (12, 64, 32) -> (2, 8, 32) at rank 33, batch 64: 362
// us a forward with planes, 337 without; batch 128: 374, 378; 256: 392, 497.
bool layer_weight_planes(const LayerShape &sh, long long batch) {
  const long long blocks = static_cast<long long>(sh.m[0]) * sh.m[1] * ((sh.m[2] + kWeightG - 1) / kWeightG);
  return batch > 64 || blocks >= device_sm_count() || layer_weight_form(sh) != WEIGHT_PACKED;
}

template <int KIND>
cudaError_t weight_launch(const LayerShape &sh, const float *P, const float *Q, const WeightOut &W, int *flag,
                          cudaStream_t s) {
  const long long total = static_cast<long long>(sh.n[0]) * sh.n[1] * sh.n[2] * sh.m[0] * sh.m[1] * sh.m[2];
  const WeightForm form = layer_weight_form(sh);
  if (form == WEIGHT_TILED) {
    const size_t smem = layer_weight_smem(sh);
    const int rb = layer_weight_rb(sh), G = 64 / rb;
    const unsigned grid = static_cast<unsigned>(sh.m[0]) * sh.m[1] * ((sh.m[2] + G - 1) / G);
    auto launch = [&](auto kernel) -> cudaError_t {
      const cudaError_t e = allow_smem(kernel, smem);
      if (e == cudaSuccess) kernel<<<grid, kLayerThreads, smem, s>>>(sh, P, Q, W, flag);
      return e;
    };
    const cudaError_t e = rb == 16   ? launch(layer_weight_tiled_kernel<KIND, 16>)
                          : rb == 32 ? launch(layer_weight_tiled_kernel<KIND, 32>)
                                     : launch(layer_weight_tiled_kernel<KIND, 64>);
    if (e != cudaSuccess) return e;
  } else if (form == WEIGHT_PACKED) {
    const size_t packed = layer_weight_packed_smem(sh);
    const cudaError_t e = allow_smem(layer_weight_packed_kernel<KIND>, packed);
    if (e != cudaSuccess) return e;
    const unsigned grid = static_cast<unsigned>(sh.m[0]) * sh.m[1] * ((sh.m[2] + kWeightG - 1) / kWeightG);
    layer_weight_packed_kernel<KIND><<<grid, kLayerThreads, packed, s>>>(sh, P, Q, W, flag);
  } else {
    layer_weight_kernel<KIND><<<grid_for_layer(total), kLayerThreads, 0, s>>>(sh, P, Q, W, flag);
  }
  return cudaGetLastError();
}

cudaError_t layer_weight_launch(const LayerShape &sh, const float *P, const float *Q, float *W32, __nv_bfloat16 *W16,
                                __nv_bfloat16 *W3, long long plane, int *flag, cudaStream_t s) {
  const WeightOut W{W32, W16, W3, plane};
  if (W3) return W32 && flag ? weight_launch<W_PLANES>(sh, P, Q, W, flag, s) : cudaErrorInvalidValue;
  if (W32) return weight_launch<W_FP32>(sh, P, Q, W, flag, s);
  return weight_launch<W_BF16>(sh, P, Q, W, flag, s);
}

cudaError_t bias_act_launch(float *y, const float *bias, long long batch, long long nout, int act, cudaStream_t s) {
  bias_act_kernel<<<grid_for_layer(batch * nout), kLayerThreads, 0, s>>>(y, bias, batch, nout, act);
  return cudaGetLastError();
}

int layer_colsum_chunks(long long batch) {
  long long c = (batch + 15) / 16;   // at most 16 rows of dy per thread at small batch
  if (c < 1) c = 1;
  if (c > 64) c = 64;
  return static_cast<int>(c);
}

int layer_dpq_chunks(const LayerShape &sh) {
  const int blocks = sh.m[0] * sh.m[1];
  // a CTA and a half an SM; two of the packed form, of which more share one
  const int ctas = layer_dpq_form(sh) == DPQ_PACKED ? 2 * device_sm_count() : 3 * device_sm_count() / 2;
  int ch = (ctas + blocks - 1) / blocks;
  return ch < 1 ? 1 : (ch > sh.m[2] ? sh.m[2] : ch);
}

size_t layer_dq_part_count(const LayerShape &sh) {
  if (layer_dpq_form(sh) == DPQ_NONE) return 0;
  const size_t dq = static_cast<size_t>(sh.m[0]) * sh.m[1] * sh.n[2] * sh.m[2] * sh.r1;
  const int ch = layer_dpq_chunks(sh);
  const size_t dp = ch > 1 ? static_cast<size_t>(ch) * sh.n[0] * sh.m[0] * sh.n[1] * sh.m[1] * sh.r1 : 0;
  return dq + dp;   // dQ partials, then dP partials
}

cudaError_t layer_factor_grads_launch(const LayerShape &sh, const float *dW, long long batch, const float *u1, const float *u2, const float *u3, const float *b2,
                                      const float *b1, const float *P, const float *Q, const float *T1, float *dP,
                                      float *dQ, float *dT1, float *dQpart, float *cpart, float *du1, float *du2,
                                      float *du3, float *db2, float *db1, float *dbias, cudaStream_t s,
                                      int *launches) {
  const int A = sh.n[0] * sh.m[0], B = sh.n[1] * sh.m[1], C = sh.n[2] * sh.m[2], NP = sh.n[0] * sh.n[1];
  const long long nout = static_cast<long long>(sh.m[0]) * sh.m[1] * sh.m[2];
  const int cchunks = layer_colsum_chunks(batch);
  const DpqForm form = layer_dpq_form(sh);
  const size_t smem_dpq = form == DPQ_PACKED ? layer_dpq_packed_smem(sh) : layer_dpq_smem(sh);
  SumJobs sums{};
  cudaError_t e;
  if (form != DPQ_NONE && dQpart) {
    const int blocks = sh.m[0] * sh.m[1], ch = layer_dpq_chunks(sh);
    float *dPpart = dQpart + static_cast<size_t>(blocks) * C * sh.r1, *dPo = ch > 1 ? dPpart : dP;
    // ranks per thread: as many as leave every thread a pair
    auto launch = [&](auto kernel) -> cudaError_t {
      const cudaError_t r = allow_smem(kernel, smem_dpq);
      if (r != cudaSuccess) return r;
      kernel<<<static_cast<unsigned>(blocks * ch), kLayerThreads, smem_dpq, s>>>(sh, dW, P, Q, dPo, dQpart);
      return cudaGetLastError();
    };
    if (form == DPQ_PACKED) e = launch(layer_dpq_packed_kernel);
    else if (NP * ((sh.r1 + 15) / 16) >= kLayerThreads) e = launch(layer_dpq_kernel<16>);
    else if (NP * ((sh.r1 + 7) / 8) >= kLayerThreads) e = launch(layer_dpq_kernel<8>);
    else e = launch(layer_dpq_kernel<4>);
    if (e != cudaSuccess) return e;
    const long long cnt = static_cast<long long>(C) * sh.r1, pc = static_cast<long long>(A) * B * sh.r1;
    sums.j[0] = SumJob{dQpart, dQ, cnt, blocks, sum_blocks(blocks, cnt)};
    if (ch > 1) sums.j[1] = SumJob{dPpart, dP, pc, ch, sum_blocks(ch, pc)};
    *launches += 1;
  } else {
    const size_t smem = sizeof(float) * static_cast<size_t>(C);
    if (smem > 48 * 1024) return cudaErrorInvalidValue;
    layer_dp_kernel<<<static_cast<unsigned>(A * B), kLayerThreads, smem, s>>>(sh, dW, Q, dP);
    layer_dq_kernel<<<static_cast<unsigned>(C), kLayerThreads, 0, s>>>(sh, dW, P, dQ);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    *launches += 2;
  }
  if (dbias) sums.j[2] = SumJob{cpart, dbias, nout, cchunks, sum_blocks(cchunks, nout)};
  const int nsum = sums.j[0].blocks + sums.j[1].blocks + sums.j[2].blocks;
  if (nsum > 0) {
    layer_reduce_kernel<<<nsum, kLayerThreads, 0, s>>>(sums);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    *launches += 1;
  }
  const int du3_blocks = static_cast<int>((static_cast<long long>(C) * sh.r2 + kLayerThreads - 1) / kLayerThreads);
  const unsigned grid = static_cast<unsigned>(B + A + du3_blocks + sh.r1);
  const int rb = sh.r4 > sh.r2 ? sh.r4 : sh.r2;
  auto grads = [&](auto kernel) {
    kernel<<<grid, kLayerThreads, 0, s>>>(sh, u2, u3, b1, T1, dP, dQ, dT1, du2, du3, db1, B, A + du3_blocks);
  };
  if (rb <= 16) grads(layer_grads_kernel<16>);
  else if (rb <= 32) grads(layer_grads32_kernel);
  else grads(layer_grads_kernel<kLayerMaxRank>);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  const long long du1_blocks = (static_cast<long long>(A) * sh.r3 + kLayerThreads / 32 - 1) / (kLayerThreads / 32);
  const long long db2_blocks =
      (static_cast<long long>(sh.r3) * sh.r4 * sh.r1 + kLayerThreads - 1) / kLayerThreads;
  layer_dt1_back_kernel<<<static_cast<unsigned>(du1_blocks + db2_blocks), kLayerThreads, 0, s>>>(
      sh, u1, b2, dT1, du1, db2, static_cast<int>(du1_blocks));
  *launches += 2;
  return cudaGetLastError();
}

}  // namespace htgb
