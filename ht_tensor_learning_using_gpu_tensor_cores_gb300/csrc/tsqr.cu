// Householder TSQR: the R factor of a tall-skinny FP32 matrix A (m x k,
// k <= 64, column-major), all row blocks in one launch.
//
// Replaces the reference's tsqr_svd / tsqr_svd_half
// (third_order_tensor_decompsition/CUDA/TSQR/kernel.cu:500-949), which splits
// the n^2 x n unfolding into four row blocks on the host, QR-factors each with
// cuSOLVER (geqrf, kernel.cu:326-350), stacks the four R factors and factors
// them again.  Here:
//   * every warp owns a k x k R in shared memory and folds 64-row panels of A
//     into it with Householder reflections on [R; panel] (rows held two per
//     lane, column norms and the reflector-column dot products as warp-shuffle
//     reductions); the reflector of column j touches only row j of R and the
//     panel, because R is upper triangular;
//   * the warps' R factors are combined in a shared-memory binary tree (each
//     partner's R is the next panel);
//   * the CTAs' R factors are combined in a tree of fan-in 8 across the grid:
//     the last CTA of a group to finish (an atomic counter, no waiting) loads
//     the group's R factors and combines them, until one remains.  No CTA ever
//     waits for another, so the launch needs no co-residency.
// The result has a non-negative diagonal (R's rows take the sign of their
// pivot); optionally R^T R is formed in compensated FP32.
#include <cfloat>

#include "common.cuh"
#include "engine.h"

namespace htgb {
namespace {

constexpr int TQ_PROWS = 64;   // rows of a panel (two per lane)
constexpr int TQ_FAN = 8;      // fan-in of the cross-CTA tree

template <int KM>
struct TqCfg {
  static constexpr int WARPS = KM == 32 ? 8 : 4;
  static constexpr int THREADS = WARPS * 32;
  static constexpr int LD = KM + 1;                                  // row stride (floats): conflict-free rows
  static constexpr int WARP_FLOATS = (KM + TQ_PROWS) * LD;           // R (KM rows) + panel (64 rows)
  static constexpr size_t SMEM = size_t(WARPS) * WARP_FLOATS * sizeof(float);
  static constexpr int RPL = KM == 32 ? 4 : 2;                       // panel rows per lane in the main loop
  static constexpr int PANEL = 32 * RPL;                             // main-loop panel height
};

// Sum over the warp, the same value in every lane (lane 0's reduction order).
HT_DEV float warp_sum_bcast(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return __shfl_sync(0xffffffffu, v, 0);
}

// Sum of v[i] over the warp for W (16 or 32) columns i at once (reduce-scatter):
// lane l returns the total of column l (W = 32) or l / 2 (W = 16).  W - 1 or W
// shuffles, all independent per level.
template <int W>
HT_DEV float warp_reduce_scatter(float (&v)[W]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 16, n = W / 2; n >= 1; o >>= 1, n >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < n; ++i) {
      const float send = up ? v[i] : v[i + n];
      const float keep = up ? v[i + n] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  if (W == 16) v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
  return v[0];
}

// [R; P] -> R' with R' upper triangular and R'^T R' = R^T R + P^T P: k
// Householder reflections.  R: k x k row-major (stride LD), P: prow x k
// row-major (stride LD, prow <= 64, destroyed).  One warp; lane l holds panel
// rows l and l + 32 and, while column j is reduced, entries l + 32 b of R's row
// j (the only row of R the reflector changes, R being upper triangular).  For
// each column j the dot products of the reflector with all later columns are
// formed together, 32 columns per reduce-scatter, so the shuffles of different
// columns overlap instead of forming one long dependent chain per column.
template <int KM, int LD>
HT_DEV void warp_qr_fold(float *R, float *P, int prow, int k) {
  constexpr int NB = KM / 32;
  const int lane = threadIdx.x & 31;
  const bool h0 = lane < prow, h1 = lane + 32 < prow;
  float *p0 = P + lane * LD, *p1 = P + (lane + 32) * LD;
  for (int j = 0; j < k; ++j) {
    float r[NB];
#pragma unroll
    for (int b = 0; b < NB; ++b) r[b] = lane + 32 * b < k ? R[j * LD + lane + 32 * b] : 0.f;
    const float x0 = h0 ? p0[j] : 0.f, x1 = h1 ? p1[j] : 0.f;
    const float sig = warp_sum_bcast(fmaf(x0, x0, x1 * x1));
    const float rjj = __shfl_sync(0xffffffffu, NB == 1 || j < 32 ? r[0] : r[NB - 1], j & 31);
    if (sig != 0.f) {   // else the column below the pivot is already zero
      const float nrm = sqrtf(fmaf(rjj, rjj, sig));
      const float alpha = rjj > 0.f ? -nrm : nrm;
      const float v0 = rjj - alpha;            // reflector v = [v0; x], tau = 2 / v^T v
      const float tau = -1.f / (alpha * v0);
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        if (32 * b + 31 <= j) continue;        // every column of this block is done
        float a0[32], a1[32], v[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const int c = 32 * b + i;
          const bool live = c > j && c < k;
          a0[i] = (live && h0) ? p0[c] : 0.f;
          a1[i] = (live && h1) ? p1[c] : 0.f;
          v[i] = fmaf(x0, a0[i], x1 * a1[i]);
        }
        const int cl = 32 * b + lane;        // this lane's column
        const float w = fmaf(v0, r[b], warp_reduce_scatter<32>(v));
        const float tw = (cl > j && cl < k) ? tau * w : 0.f;
        r[b] = fmaf(-tw, v0, r[b]);
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const int c = 32 * b + i;
          const float twi = __shfl_sync(0xffffffffu, tw, i);
          if (c > j && c < k) {
            if (h0) p0[c] = fmaf(-twi, x0, a0[i]);
            if (h1) p1[c] = fmaf(-twi, x1, a1[i]);
          }
        }
      }
      if (lane == (j & 31)) r[NB == 1 ? 0 : j / 32] = alpha;
    }
#pragma unroll
    for (int b = 0; b < NB; ++b)
      if (lane + 32 * b < k) R[j * LD + lane + 32 * b] = r[b];
    __syncwarp();
  }
}

// The same fold for k <= 32 with the panel in registers: lane l holds rows
// l + 32 q in packed pairs of q.  The fold is one dependent chain per column (a
// CTA of the tall case runs 15 folds of 32 columns in a row), so a column is
// kept short: the current column is always index 0 (the update writes column c
// to c - 1, no look-up by j), its norm is the reflector's dot product with
// itself from the same reduce-scatter as the others', the updates' factors are
// shared through W floats of shared memory, and once at most 16 columns are
// left the steps take only those.  261 us to 101 for 409600 rows of 32.
// A column whose squares would underflow or overflow is reflected from a scaled
// copy: a rule on its own size, so that data of any scale folds alike and what
// rounding leaves of a dependent column is just another small column.
constexpr float kQrSmall = 7.8886e-31f;   // 2^-100: squares above it hold 24 bits of every entry that counts
template <int W, int LD, int Q2>
HT_DEV void warp_qr_columns(float *R, float2 (&p)[Q2][32], int j0, int j1, int k, float *fac) {
  const int lane = threadIdx.x & 31, cl = W == 32 ? lane : lane >> 1;   // this lane's column, from j on
  for (int j = j0; j < j1; ++j) {
    const bool live = j + cl < k;
    const float r = live ? R[j * LD + j + cl] : 0.f;
    float2 x[Q2];
#pragma unroll
    for (int q = 0; q < Q2; ++q) x[q] = p[q][0];
    auto dots = [&]() {   // x with itself (index 0) and with the columns behind it
      float v[W];
#pragma unroll
      for (int c = 0; c < W; ++c) {
        float2 a = make_float2(0.f, 0.f);
#pragma unroll
        for (int q = 0; q < Q2; ++q) fma2(a, x[q], c == 0 ? x[q] : p[q][c]);
        v[c] = a.x + a.y;
      }
      return warp_reduce_scatter<W>(v);
    };
    // reflector v = [v0; x], tau = 2 / v^T v = -1 / (alpha v0): the updates' factor
    // and R's row (alpha at the pivot), from a column `down` times this size
    float tw, rn;
    auto reflect = [&](float dot, float sig, float rjj, float n2, float down) {
      const float nrm = sqrtf(n2);
      const float alpha = rjj > 0.f ? -nrm : nrm;
      const float v0 = rjj - alpha;
      tw = 0.f;
      rn = r;
      if (sig != 0.f) {   // otherwise the column below the pivot is zero
        const float tau = -1.f / (alpha * v0);
        if (live && cl > 0) tw = tau * fmaf(v0, r, dot);
        rn = cl > 0 ? fmaf(-tw, v0, r) : alpha * down;
      }
    };
    const float dot = dots();
    const float sig = __shfl_sync(0xffffffffu, dot, 0), rjj = __shfl_sync(0xffffffffu, r, 0);
    const float n2 = fmaf(rjj, rjj, sig);
    reflect(dot, sig, rjj, n2, 1.f);
    // (behind the reflector, whose chain the comparison would lengthen: a call on
    // 409600 x 32 takes 244 us without the rule, 253 with it in front, 251 here)
    if (__builtin_expect(!(n2 >= kQrSmall && n2 <= FLT_MAX), 0)) {
      // the reflector from (pivot, x) times a power of two that takes the largest
      // entry to [1, 2), unless there is nothing to eliminate or no finite column
      float top = fabsf(rjj);
#pragma unroll
      for (int q = 0; q < Q2; ++q) top = fmaxf(top, fmaxf(fabsf(x[q].x), fabsf(x[q].y)));
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
      if (top > 0.f && top < INFINITY) {
        const int e = min(max(ilogbf(top), -126), 126);   // (both powers are normal numbers)
        const float up = scalbnf(1.f, -e);
#pragma unroll
        for (int q = 0; q < Q2; ++q) {
          x[q].x *= up;
          x[q].y *= up;
        }
        const float dots1 = dots(), sig1 = __shfl_sync(0xffffffffu, dots1, 0), rjj1 = up * rjj;
        reflect(dots1, sig1, rjj1, fmaf(rjj1, rjj1, sig1), scalbnf(1.f, e));
      }
    }
    float *f = fac + 32 * (j & 1);   // two buffers: one barrier a column
    f[cl] = -tw;
    if (live && (W == 32 || !(lane & 1))) R[j * LD + j + cl] = rn;
    __syncwarp();
#pragma unroll
    for (int c4 = 0; c4 < W; c4 += 4) {
      const float4 t = *reinterpret_cast<const float4 *>(f + c4);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (c4 + u == 0) continue;
        const float tc = u == 0 ? t.x : u == 1 ? t.y : u == 2 ? t.z : t.w;
#pragma unroll
        for (int q = 0; q < Q2; ++q) {
          float2 y = p[q][c4 + u];
          fma2(y, make_float2(tc, tc), x[q]);
          p[q][c4 + u - 1] = y;
        }
      }
    }
#pragma unroll
    for (int q = 0; q < Q2; ++q) p[q][W - 1] = make_float2(0.f, 0.f);
  }
}

template <int LD, int Q2>
HT_DEV void warp_qr_fold32(float *R, float2 (&p)[Q2][32], int k, float *fac) {
  if (k > 16) warp_qr_columns<32, LD, Q2>(R, p, 0, 16, k, fac);
  warp_qr_columns<16, LD, Q2>(R, p, k > 16 ? 16 : 0, k, k, fac);
  __syncwarp();
}

// Fold a row-major panel in shared memory (prow <= 64 rows, stride LD) into R.
template <int KM, int LD>
HT_DEV void warp_fold_smem(float *R, float *P, int prow, int k, float *fac) {
  if constexpr (KM == 32) {
    const int lane = threadIdx.x & 31;
    float2 p[1][32];
#pragma unroll
    for (int c = 0; c < 32; ++c) {
      p[0][c].x = (lane < prow && c < k) ? P[lane * LD + c] : 0.f;
      p[0][c].y = (lane + 32 < prow && c < k) ? P[(lane + 32) * LD + c] : 0.f;
    }
    warp_qr_fold32<LD, 1>(R, p, k, fac);
  } else {
    warp_qr_fold<KM, LD>(R, P, prow, k);
  }
}

struct TqParams {
  const float *A;
  long long m, lda;
  int k;
  long long rows_per_cta;   // a multiple of warps x panel rows
  float *slots;             // per level: count_l x k x k floats (row-major R)
  long long slot_off[8];    // float offset of level l's slots
  int cnt_off[8];           // offset of level l's group counters
  int *counters;            // zeroed before the launch
  float *R_out;             // k x k column-major (lower triangle zero), diagonal >= 0
  float *RtR_out;           // optional k x k R^T R (compensated FP32)
};

template <int KM>
__global__ void __launch_bounds__(TqCfg<KM>::THREADS, 1) tsqr_kernel(const TqParams p) {
  using C = TqCfg<KM>;
  constexpr int LD = C::LD;
  extern __shared__ float tq_sm[];
  __shared__ int s_last;
  __shared__ __align__(16) float facs[C::WARPS][64];
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int k = p.k;
  float *R = tq_sm + warp * C::WARP_FLOATS;
  float *P = R + KM * LD, *fac = facs[warp];
  for (int e = lane; e < KM * LD; e += 32) R[e] = 0.f;
  __syncwarp();

  // 1. this CTA's rows, in 64-row panels dealt round-robin to the warps
  const long long r_begin = static_cast<long long>(blockIdx.x) * p.rows_per_cta;
  const long long r_end = min(p.m, r_begin + p.rows_per_cta);
  for (long long r0 = r_begin + static_cast<long long>(warp) * C::PANEL; r0 < r_end;
       r0 += static_cast<long long>(C::WARPS) * C::PANEL) {
    const int prow = static_cast<int>(min(static_cast<long long>(C::PANEL), r_end - r0));
    if constexpr (KM == 32) {   // the panel straight into registers
      float2 pr[C::RPL / 2][32];
#pragma unroll
      for (int c = 0; c < 32; ++c) {
        const float *col = p.A + r0 + p.lda * c;
#pragma unroll
        for (int q = 0; q < C::RPL / 2; ++q) {
          pr[q][c].x = (c < k && lane + 64 * q < prow) ? __ldg(col + lane + 64 * q) : 0.f;
          pr[q][c].y = (c < k && lane + 64 * q + 32 < prow) ? __ldg(col + lane + 64 * q + 32) : 0.f;
        }
      }
      warp_qr_fold32<LD, C::RPL / 2>(R, pr, k, fac);
    } else {
#pragma unroll 4
      for (int c = 0; c < k; ++c) {
        const float *col = p.A + r0 + p.lda * c;
        P[lane * LD + c] = lane < prow ? __ldg(col + lane) : 0.f;
        P[(lane + 32) * LD + c] = lane + 32 < prow ? __ldg(col + lane + 32) : 0.f;
      }
      __syncwarp();
      warp_qr_fold<KM, LD>(R, P, prow, k);
    }
  }
  __syncthreads();

  // 2. the warps' R factors, combined pairwise in shared memory
  auto tree = [&]() {
    for (int half = C::WARPS / 2; half >= 1; half >>= 1) {
      if (warp < half) warp_fold_smem<KM, LD>(R, tq_sm + (warp + half) * C::WARP_FLOATS, k, k, fac);
      __syncthreads();
    }
  };
  tree();

  // 3. across CTAs: the last CTA of each group of TQ_FAN combines the group
  float *R0 = tq_sm;   // warp 0's R: the CTA's result
  long long node = blockIdx.x, count = gridDim.x;
  int level = 0;
  while (count > 1) {
    float *slot = p.slots + p.slot_off[level] + node * k * k;
    for (int e = t; e < k * k; e += C::THREADS) slot[e] = R0[(e / k) * LD + e % k];
    __threadfence();
    __syncthreads();
    const long long group = node / TQ_FAN;
    const int gsize = static_cast<int>(min(static_cast<long long>(TQ_FAN), count - group * TQ_FAN));
    if (t == 0) s_last = atomicAdd(p.counters + p.cnt_off[level] + group, 1) == gsize - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    // warp w takes member w into its R (zero when the group is smaller) and
    // folds in members w + WARPS, w + 2 WARPS, ... as panels
    auto load_member = [&](float *dst, long long member) {
      const float *src = p.slots + p.slot_off[level] + member * k * k;
      for (int e = lane; e < KM * LD; e += 32) {
        const int i = e / LD, c = e % LD;
        dst[e] = (i < k && c < k) ? __ldcg(src + i * k + c) : 0.f;
      }
      __syncwarp();
    };
    if (warp < gsize) {
      load_member(R, group * TQ_FAN + warp);
    } else {
      for (int e = lane; e < KM * LD; e += 32) R[e] = 0.f;
      __syncwarp();
    }
    for (int w = warp + C::WARPS; w < gsize; w += C::WARPS) {
      load_member(P, group * TQ_FAN + w);
      warp_fold_smem<KM, LD>(R, P, k, k, fac);
    }
    __syncthreads();
    tree();
    node = group;
    count = (count + TQ_FAN - 1) / TQ_FAN;
    ++level;
  }

  // 4. one R left: non-negative diagonal, column-major out, R^T R if asked
  __shared__ float sgn[64];
  for (int i = t; i < k; i += C::THREADS) sgn[i] = R0[i * LD + i] < 0.f ? -1.f : 1.f;
  __syncthreads();
  for (int e = t; e < k * k; e += C::THREADS) {
    const int i = e % k, j = e / k;
    p.R_out[e] = i <= j ? sgn[i] * R0[i * LD + j] : 0.f;
  }
  if (p.RtR_out) {
    for (int e = t; e < k * k; e += C::THREADS) {
      const int a = e % k, b = e / k;
      Acc2 acc{0.f, 0.f};
      for (int i = 0; i <= min(a, b); ++i) acc2_add_prod(acc, R0[i * LD + a], R0[i * LD + b]);
      p.RtR_out[e] = acc.s + acc.c;
    }
  }
}

int tq_levels(long long count, long long *counts) {
  int L = 0;
  while (count > 1 && L < 8) {
    counts[L++] = count;
    count = (count + TQ_FAN - 1) / TQ_FAN;
  }
  return L;
}

long long tq_grid(long long m) {
  const long long want = (m + 4 * TQ_PROWS - 1) / (4 * TQ_PROWS);   // at least ~4 panels per CTA
  const long long cap = device_sm_count();
  return want < 1 ? 1 : (want < cap ? want : cap);
}

}  // namespace

size_t tsqr_workspace_bytes(long long m, int k) {
  long long counts[8];
  const int L = tq_levels(tq_grid(m), counts);
  size_t floats = 0, ints = 0;
  for (int l = 0; l < L; ++l) {
    floats += static_cast<size_t>(counts[l]) * k * k;
    ints += static_cast<size_t>((counts[l] + TQ_FAN - 1) / TQ_FAN);
  }
  return ((floats * sizeof(float) + 255) & ~size_t(255)) + ((ints * sizeof(int) + 255) & ~size_t(255)) + 256;
}

cudaError_t tsqr_launch(const float *A, long long m, int k, long long lda, float *R, float *RtR, void *ws,
                        size_t ws_bytes, cudaStream_t st, int *launches) {
  if (k < 1 || k > 64 || m < 1 || lda < m) return cudaErrorInvalidValue;
  if (tsqr_workspace_bytes(m, k) > ws_bytes) return cudaErrorInvalidValue;
  TqParams p{};
  p.A = A;
  p.m = m;
  p.lda = lda;
  p.k = k;
  const long long grid = tq_grid(m);
  // a CTA's rows are a whole number of rounds of panels over its warps, so the
  // warps finish together (the tree that follows waits for the slowest)
  const long long round = k <= 32 ? TqCfg<32>::WARPS * TqCfg<32>::PANEL : TqCfg<64>::WARPS * TqCfg<64>::PANEL;
  p.rows_per_cta = ((m + grid - 1) / grid + round - 1) / round * round;
  const long long g = (m + p.rows_per_cta - 1) / p.rows_per_cta;   // CTAs that own rows
  long long counts[8];
  const int L = tq_levels(g, counts);
  if (g > 1 && L >= 8) return cudaErrorInvalidValue;
  size_t floats = 0;
  int ints = 0;
  for (int l = 0; l < L; ++l) {
    p.slot_off[l] = static_cast<long long>(floats);
    p.cnt_off[l] = ints;
    floats += static_cast<size_t>(counts[l]) * k * k;
    ints += static_cast<int>((counts[l] + TQ_FAN - 1) / TQ_FAN);
  }
  char *w = static_cast<char *>(ws);
  p.slots = reinterpret_cast<float *>(w);
  p.counters = reinterpret_cast<int *>(w + ((floats * sizeof(float) + 255) & ~size_t(255)));
  p.R_out = R;
  p.RtR_out = RtR;
  if (ints > 0) {
    const cudaError_t e = cudaMemsetAsync(p.counters, 0, sizeof(int) * ints, st);
    if (e != cudaSuccess) return e;
  }
  static bool attr32[64] = {}, attr64[64] = {};
  if (k <= 32) {
    const cudaError_t e = opt_in_smem(tsqr_kernel<32>, static_cast<int>(TqCfg<32>::SMEM), attr32);
    if (e != cudaSuccess) return e;
    tsqr_kernel<32><<<static_cast<unsigned>(g), TqCfg<32>::THREADS, TqCfg<32>::SMEM, st>>>(p);
  } else {
    const cudaError_t e = opt_in_smem(tsqr_kernel<64>, static_cast<int>(TqCfg<64>::SMEM), attr64);
    if (e != cudaSuccess) return e;
    tsqr_kernel<64><<<static_cast<unsigned>(g), TqCfg<64>::THREADS, TqCfg<64>::SMEM, st>>>(p);
  }
  if (launches) *launches += 1;
  return cudaGetLastError();
}

}  // namespace htgb
