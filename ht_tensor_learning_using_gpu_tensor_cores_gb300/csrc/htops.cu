// Operations on a tensor held in HT format (tree, ranks, leaf bases U_t,
// transfer tensors B_t): full reconstruction and evaluation of single entries.
//
// The reference reconstructs only the whole tensor, with cuBLAS calls on the
// node bases (third_order_tensor_decompsition/CUDA/Optimized/htd_tensorcore.cu:
// 295-331); it has no entry-wise evaluation.  Here the reconstruction is one
// expansion of the interior node basis (api.cu expand2) and one NT product
// written straight into the column-major tensor.  Single entries are read from
// precontracted matrices: every transfer tensor is folded with its parent's
// and one child's factors into a matrix with one row per index of that child's
// mode, so an entry costs one or two k x k row-vector products.
#include <climits>

#include "common.cuh"
#include "engine.h"

namespace htgb {
namespace {

constexpr int RT_M = 128, RT_N = 64, RT_K = 64;

// Slab z of a batch: C_z (m x n, ldc) = A_z (m x k, lda) B^T (B: n x k, ldb),
// k <= 64, column-major, A_z = A + z sA, C_z = C + z sC.  256 threads: thread
// (tx = t % 32, ty = t / 32) owns rows 4 tx .. 4 tx + 3 and columns
// 8 ty .. 8 ty + 7 of the 128 x 64 tile, read from shared memory as one and two
// 16-byte vectors per k step (the column vectors are warp-uniform broadcasts),
// so the loop is bound by the FMA pipe; rows go out as 16-byte stores when the
// output is 16-byte aligned.
__global__ void __launch_bounds__(256) gemm_nt_kernel(const float *__restrict__ A0, long long lda, long long sA,
                                                      const float *__restrict__ B, long long ldb, float *__restrict__ C0,
                                                      long long ldc, long long sC, long long m, long long n, int k,
                                                      long long batch) {
  __shared__ __align__(16) float As[RT_K][RT_M];
  __shared__ __align__(16) float Bs[RT_K][RT_N];
  const long long r0 = static_cast<long long>(blockIdx.x) * RT_M, c0 = static_cast<long long>(blockIdx.y) * RT_N;
  const int t = threadIdx.x, tx = t & 31, ty = t >> 5;
  for (int e = t; e < RT_N * k; e += 256) {
    const int c = e % RT_N, kk = e / RT_N;
    Bs[kk][c] = (c0 + c < n) ? B[(c0 + c) + ldb * kk] : 0.f;
  }
  for (long long z = blockIdx.z; z < batch; z += gridDim.z) {
    const float *A = A0 + z * sA;
    float *C = C0 + z * sC;
    __syncthreads();
    for (int e = t; e < RT_M * k; e += 256) {
      const int r = e % RT_M, kk = e / RT_M;
      As[kk][r] = (r0 + r < m) ? A[(r0 + r) + lda * kk] : 0.f;
    }
    __syncthreads();
    float acc[4][8];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
    for (int kk = 0; kk < k; ++kk) {
      const float4 a = *reinterpret_cast<const float4 *>(&As[kk][4 * tx]);
      const float4 b0 = *reinterpret_cast<const float4 *>(&Bs[kk][8 * ty]);
      const float4 b1 = *reinterpret_cast<const float4 *>(&Bs[kk][8 * ty + 4]);
      const float av[4] = {a.x, a.y, a.z, a.w};
      const float bv[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
    }
    const long long r = r0 + 4 * tx;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const long long c = c0 + 8 * ty + j;
      if (c >= n || r >= m) continue;
      float *dst = C + r + ldc * c;
      if (r + 3 < m && (reinterpret_cast<uintptr_t>(dst) & 15u) == 0) {
        *reinterpret_cast<float4 *>(dst) = make_float4(acc[0][j], acc[1][j], acc[2][j], acc[3][j]);
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (r + i < m) dst[i] = acc[i][j];
      }
    }
  }
}

// out[(c + kc b) + kc kq a] = sum_rt Bt[a + kp b + kp kq rt] M[rt + kt c]
// (M: kt x kc; M null = the identity, kc = kt): a transfer tensor with its
// parent's factor folded in, reordered so that a row of out's product with a
// leaf basis is contiguous in (c, b).
__global__ void eval_core_kernel(const float *__restrict__ Bt, int kp, int kq, int kt, const float *__restrict__ M,
                                 int kc, float *__restrict__ out) {
  const int total = kc * kq * kp;
  for (int e = blockIdx.x * 256 + threadIdx.x; e < total; e += gridDim.x * 256) {
    const int c = e % kc, b = (e / kc) % kq, a = e / (kc * kq);
    float s;
    if (!M) {
      s = Bt[a + kp * b + kp * kq * c];
    } else {
      s = 0.f;
      for (int rt = 0; rt < kt; ++rt) s = fmaf(Bt[a + kp * b + kp * kq * rt], M[rt + kt * c], s);
    }
    out[e] = s;
  }
}

HT_DEV long long eval_index(const long long *idx, long long e, int order, int m, long long dim, int *err, int lane) {
  long long i = idx[e * order + m];
  if (i < 0 || i >= dim) {
    if (lane == 0) atomicOr(err, 1);
    i = i < 0 ? 0 : dim - 1;
  }
  return i;
}

// One warp per entry, lanes over y < ky (two per lane):
//   a[y] = sum_x W0[i_row0][y + ky x] U0v[i_vec0 + n_vec0 x]
//   c[y] = side 1 the same, or U1v[i_vec1 + n_vec1 y] when W1 is null
//   entry = sum_y a[y] c[y].
__global__ void __launch_bounds__(256) evaluate_kernel(const EvalPlan ep, const long long *__restrict__ idx,
                                                       long long count, float *__restrict__ out, int *err) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ky = ep.ky;
  for (long long e = static_cast<long long>(blockIdx.x) * 8 + warp; e < count;
       e += static_cast<long long>(gridDim.x) * 8) {
    float v[2][2];
#pragma unroll
    for (int sd = 0; sd < 2; ++sd) {
      const EvalSide &S = ep.side[sd];
      const long long iv = eval_index(idx, e, ep.order, S.mode_vec, S.n_vec, err, lane);
      if (S.W) {
        const long long ir = eval_index(idx, e, ep.order, S.mode_row, S.n_row, err, lane);
        const float *row = S.W + ir * static_cast<long long>(ky) * S.kx;
        float s0 = 0.f, s1 = 0.f;
        for (int x = 0; x < S.kx; ++x) {
          const float u = __ldg(S.Uv + iv + S.n_vec * x);
          if (lane < ky) s0 = fmaf(row[lane + ky * x], u, s0);
          if (lane + 32 < ky) s1 = fmaf(row[lane + 32 + ky * x], u, s1);
        }
        v[sd][0] = s0;
        v[sd][1] = s1;
      } else {
        v[sd][0] = lane < ky ? S.Uv[iv + S.n_vec * lane] : 0.f;
        v[sd][1] = lane + 32 < ky ? S.Uv[iv + S.n_vec * (lane + 32)] : 0.f;
      }
    }
    float s = v[0][0] * v[1][0] + v[0][1] * v[1][1];
    for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if (lane == 0) out[e] = s;
  }
}

// Many entries of a 3rd-order tensor.  The warp above reads its entry's whole row
// of W (4 KB at rank 32) from L2, which bounds it.  Here the entries are first
// grouped by that row (a counting sort of 16-byte records), so that a block
// stages a row once for all its entries, and a thread forms several entries at
// once from it.
constexpr int kEvalThreads = 128, kEvalPer = 2;   // threads, entries a thread
constexpr int kSortThreads = 1024, kSortEntries = 8 * kSortThreads;   // entries per sorting block

HT_DEV void cp_async16(void *smem_dst, const void *gsrc) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(smem_dst)), "l"(gsrc) : "memory");
}
HT_DEV void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
HT_DEV void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// The leaf bases (n x k, mode-major) with their rows contiguous, padded to a
// multiple of four columns: an entry's row is a few 16-byte loads instead of k
// scattered ones.  Blocks below blocks0 take the first basis.
__global__ void __launch_bounds__(256) eval_rows_kernel(const float *__restrict__ A0, long long n0, int k0,
                                                        float *__restrict__ R0, int blocks0,
                                                        const float *__restrict__ A1, long long n1, int k1,
                                                        float *__restrict__ R1) {
  __shared__ float tile[32][65];
  const bool second = static_cast<int>(blockIdx.x) >= blocks0;
  const float *A = second ? A1 : A0;
  float *R = second ? R1 : R0;
  const long long n = second ? n1 : n0;
  const int k = second ? k1 : k0, kr = (k + 3) / 4 * 4;
  const long long r0 = 32ll * (blockIdx.x - (second ? blocks0 : 0));
  const int nr = static_cast<int>(min(32ll, n - r0));
  for (int e = threadIdx.x; e < 32 * kr; e += 256) {
    const int r = e & 31, c = e >> 5;
    tile[r][c] = r < nr && c < k ? A[r0 + r + n * c] : 0.f;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < nr * kr; e += 256) R[r0 * kr + e] = tile[e / kr][e % kr];
}

// Entries per row of W.
__global__ void __launch_bounds__(kSortThreads) eval_count_kernel(const long long *__restrict__ idx, int count,
                                                                  int order, int mode, int n, int *__restrict__ hist) {
  extern __shared__ int sh[];
  for (int i = threadIdx.x; i < n; i += kSortThreads) sh[i] = 0;
  __syncthreads();
  const long long e0 = static_cast<long long>(blockIdx.x) * kSortEntries;
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const long long e = e0 + u * kSortThreads + threadIdx.x;
    if (e < count) {
      const long long i = idx[e * order + mode];
      atomicAdd(&sh[i < 0 ? 0 : i >= n ? n - 1 : static_cast<int>(i)], 1);
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += kSortThreads)
    if (sh[i]) atomicAdd(&hist[i], sh[i]);
}

// Records (row of U_q, row of U_c, entry, row of W) in order of the row of W.
// Every block sums the counts (n integers), takes room for its own entries of
// each row with one atomic per row and writes them there: the order within a
// row is the blocks' and plays no part in an entry's value.
__global__ void __launch_bounds__(kSortThreads) eval_sort_kernel(const EvalPlan ep, const long long *__restrict__ idx,
                                                                 int count, const int *__restrict__ hist,
                                                                 int *__restrict__ taken, int4 *__restrict__ rec,
                                                                 int *err) {
  extern __shared__ int sh[];   // first[n], mine[n]
  __shared__ int wsum[32];
  const EvalSide &S0 = ep.side[0], &S1 = ep.side[1];
  const int n = static_cast<int>(S0.n_row), t = threadIdx.x, lane = t & 31, warp = t >> 5;
  int *first = sh, *mine = sh + n;
  const int per = (n + kSortThreads - 1) / kSortThreads, lo = min(n, t * per), hi = min(n, lo + per);
  int sum = 0;
  for (int i = lo; i < hi; ++i) {
    sum += hist[i];
    mine[i] = 0;
  }
  int inc = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += v;
  }
  if (lane == 31) wsum[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    int w = wsum[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += v;
    }
    wsum[lane] = w;
  }
  __syncthreads();
  int at = inc - sum + (warp ? wsum[warp - 1] : 0);
  for (int i = lo; i < hi; ++i) {
    first[i] = at;
    at += hist[i];
  }
  __syncthreads();
  const long long e0 = static_cast<long long>(blockIdx.x) * kSortEntries;
  int4 r[8];
  int rank[8];
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const long long e = e0 + u * kSortThreads + t;
    rank[u] = -1;
    if (e < count) {
      r[u].x = static_cast<int>(eval_index(idx, e, ep.order, S0.mode_vec, S0.n_vec, err, 0));
      r[u].y = static_cast<int>(eval_index(idx, e, ep.order, S1.mode_vec, S1.n_vec, err, 0));
      r[u].z = static_cast<int>(e);
      r[u].w = static_cast<int>(eval_index(idx, e, ep.order, S0.mode_row, S0.n_row, err, 0));
      rank[u] = atomicAdd(&mine[r[u].w], 1);
    }
  }
  __syncthreads();
  for (int i = t; i < n; i += kSortThreads)
    if (mine[i]) first[i] += atomicAdd(&taken[i], mine[i]);
  __syncthreads();
#pragma unroll
  for (int u = 0; u < 8; ++u)
    if (rank[u] >= 0) rec[first[r[u].w] + rank[u]] = r[u];
}

// A thread holds two entries' ky <= KB sums over x as packed pairs, so that a
// row's values, broadcast from shared memory, serve two entries each (four
// entries halve those loads but leave eight warps an SM where these two have
// sixteen: 239 us a call against 194 at 1048576 entries, 1024 rows, rank 32).
// A block takes 256 records and stages each row of W that they use in turn; a
// warp fetches the basis rows of its 64 entries with whole-row copies into
// shared memory at an odd pitch of 16 bytes (each thread loading its own rows
// touches 32 lines an instruction).  Entry by entry the call took 881 us.
template <int KB>
__global__ void __launch_bounds__(kEvalThreads) evaluate_grouped_kernel(const EvalPlan ep, const EvalGroups g, int count,
                                                                        float *__restrict__ out) {
  extern __shared__ __align__(16) float4 eval_rows[];   // [warps][32 kEvalPer][pitch]
  __shared__ __align__(16) float Ps[KB][KB];            // [x][y]
  __shared__ int2 row_of[kEvalThreads * kEvalPer];
  __shared__ int last_key[kEvalThreads / 32], runs[kEvalThreads / 32], run_key[kEvalThreads * kEvalPer];
  const int t = threadIdx.x, lane = t & 31, kx = ep.side[0].kx, ky = ep.ky;
  const int lq = (kx + 3) / 4, lc = (ky + 3) / 4, pitch = KB / 4 + 1;
  const int base = blockIdx.x * (kEvalThreads * kEvalPer), end = min(count, base + kEvalThreads * kEvalPer);
  float4 *rows = eval_rows + (t >> 5) * (32 * kEvalPer * pitch);
  int2 *ids = row_of + (t & ~31) * kEvalPer;
  int key[kEvalPer], dst[kEvalPer];
#pragma unroll
  for (int u = 0; u < kEvalPer; ++u) {
    const int e = base + (t & ~31) * kEvalPer + 32 * u + lane;
    const int4 r = e < end ? g.rec[e] : make_int4(0, 0, 0, -1);
    ids[32 * u + lane] = make_int2(r.x, r.y);
    dst[u] = r.z;
    key[u] = r.w;
  }
  // the block's distinct rows of W in order (its records are sorted by them)
  const int warp = t >> 5;
  if (lane == 31) last_key[warp] = key[kEvalPer - 1];
  __syncthreads();
  int before = warp ? last_key[warp - 1] : -1, nrun = 0;
  unsigned heads[kEvalPer];
#pragma unroll
  for (int u = 0; u < kEvalPer; ++u) {
    int prev = __shfl_up_sync(0xffffffffu, key[u], 1);
    if (lane == 0) prev = before;
    before = __shfl_sync(0xffffffffu, key[u], 31);
    heads[u] = __ballot_sync(0xffffffffu, key[u] >= 0 && key[u] != prev);
    nrun += __popc(heads[u]);
  }
  if (lane == 0) runs[warp] = nrun;
  __syncthreads();
  int at = 0, total = 0;
#pragma unroll
  for (int w = 0; w < kEvalThreads / 32; ++w) {
    at += w < warp ? runs[w] : 0;
    total += runs[w];
  }
#pragma unroll
  for (int u = 0; u < kEvalPer; ++u) {
    if ((heads[u] >> lane) & 1u) run_key[at + __popc(heads[u] & ((1u << lane) - 1u))] = key[u];
    at += __popc(heads[u]);
  }
  __syncthreads();
  // rows of U (l 16-byte pieces each) of this warp's entries
  auto fetch = [&](const float *U, int l, bool second) {
    const int dr = 32 / l, dc = 32 - dr * l;
    int r = lane / l, c = lane - r * l;
    while (r < 32 * kEvalPer) {
      const int row = second ? ids[r].y : ids[r].x;
      cp_async16(rows + r * pitch + c, reinterpret_cast<const float4 *>(U) + static_cast<long long>(row) * l + c);
      r += dr;
      c += dc;
      if (c >= l) {
        c -= l;
        ++r;
      }
    }
    cp_async_commit();
  };
  for (int run = 0; run < total; ++run) {
    const int cur = run_key[run];
    bool any = false;
#pragma unroll
    for (int u = 0; u < kEvalPer; ++u) any = any || key[u] == cur;
    any = __any_sync(0xffffffffu, any);
    if (any) fetch(g.Uq, lq, false);
    __syncthreads();
    const float *W = ep.side[0].W + static_cast<long long>(cur) * ky * kx;
    for (int e = t; e < 4 * lq * KB; e += kEvalThreads) {
      const int x = e / KB, y = e - x * KB;
      Ps[x][y] = x < kx && y < ky ? W[y + ky * x] : 0.f;
    }
    cp_async_wait_all();
    __syncthreads();
    if (any) {
      float2 acc[kEvalPer][KB / 2];
#pragma unroll
      for (int u = 0; u < kEvalPer; ++u)
#pragma unroll
        for (int y = 0; y < KB / 2; ++y) acc[u][y] = make_float2(0.f, 0.f);
#pragma unroll 1
      for (int x = 0; x < lq; ++x) {
        float4 q[kEvalPer];
#pragma unroll
        for (int u = 0; u < kEvalPer; ++u) q[u] = rows[(32 * u + lane) * pitch + x];
#pragma unroll
        for (int v = 0; v < 4; ++v) {
#pragma unroll
          for (int y = 0; y < KB; y += 4) {
            const float4 p = *reinterpret_cast<const float4 *>(&Ps[4 * x + v][y]);
#pragma unroll
            for (int u = 0; u < kEvalPer; ++u) {
              const float w = v == 0 ? q[u].x : v == 1 ? q[u].y : v == 2 ? q[u].z : q[u].w;
              fma2(acc[u][y / 2], make_float2(w, w), make_float2(p.x, p.y));
              fma2(acc[u][y / 2 + 1], make_float2(w, w), make_float2(p.z, p.w));
            }
          }
        }
      }
      __syncwarp();
      fetch(g.Uc, lc, true);
      cp_async_wait_all();
      __syncwarp();
#pragma unroll
      for (int u = 0; u < kEvalPer; ++u) {
        float part[KB / 4];   // (columns past ky take no part: 0 times infinity)
#pragma unroll
        for (int y = 0; y < KB; y += 4) {
          part[y / 4] = 0.f;
          if (y < ky) {
            const float4 c = rows[(32 * u + lane) * pitch + (y >> 2)];
            const float2 a = acc[u][y / 2], b = acc[u][y / 2 + 1];
            const float lo = y + 1 < ky ? fmaf(a.y, c.y, a.x * c.x) : a.x * c.x;
            const float hi = y + 2 < ky ? (y + 3 < ky ? fmaf(b.y, c.w, b.x * c.z) : b.x * c.z) : 0.f;
            part[y / 4] = lo + hi;
          }
        }
#pragma unroll
        for (int w = 1; w < KB / 4; w *= 2)
#pragma unroll
          for (int y = 0; y + w < KB / 4; y += 2 * w) part[y] += part[y + w];
        if (key[u] == cur) out[dst[u]] = part[0];
      }
      __syncwarp();
    }
  }
}

template <int KB>
cudaError_t evaluate_grouped_kb(const EvalPlan &ep, const EvalGroups &g, int count, float *out, cudaStream_t s) {
  constexpr int smem = kEvalThreads * kEvalPer * (KB / 4 + 1) * 16;
  const cudaError_t e = cudaFuncSetAttribute(evaluate_grouped_kernel<KB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             smem);
  if (e != cudaSuccess) return e;
  const unsigned grid = static_cast<unsigned>((count + kEvalThreads * kEvalPer - 1) / (kEvalThreads * kEvalPer));
  evaluate_grouped_kernel<KB><<<grid, kEvalThreads, smem, s>>>(ep, g, count, out);
  return cudaGetLastError();
}

}  // namespace

cudaError_t gemm_nt_launch(const float *A, long long lda, long long sA, const float *B, long long ldb, float *C,
                           long long ldc, long long sC, long long m, long long n, int k, long long batch,
                           cudaStream_t s) {
  if (k < 1 || k > RT_K || batch < 1) return cudaErrorInvalidValue;
  const long long gx = (m + RT_M - 1) / RT_M;
  if (gx > 0x7fffffffll) return cudaErrorInvalidValue;
  const long long gz = batch < 65535 ? batch : 65535;
  const long long chunk = 65535ll * RT_N;   // columns per launch (grid y limit)
  for (long long c0 = 0; c0 < n; c0 += chunk) {
    const long long nc = n - c0 < chunk ? n - c0 : chunk;
    const unsigned gy = static_cast<unsigned>((nc + RT_N - 1) / RT_N);
    gemm_nt_kernel<<<dim3(static_cast<unsigned>(gx), gy, static_cast<unsigned>(gz)), 256, 0, s>>>(
        A, lda, sA, B + c0, ldb, C + c0 * ldc, ldc, sC, m, nc, k, batch);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t eval_core_launch(const float *Bt, int kp, int kq, int kt, const float *M, int kc, float *out,
                             cudaStream_t s) {
  const int total = kc * kq * kp;
  int grid = (total + 255) / 256;
  if (grid > 8 * device_sm_count()) grid = 8 * device_sm_count();
  eval_core_kernel<<<grid < 1 ? 1 : grid, 256, 0, s>>>(Bt, kp, kq, kt, M, kc, out);
  return cudaGetLastError();
}

cudaError_t evaluate_launch(const EvalPlan &ep, const long long *idx, long long count, float *out, int *err,
                            cudaStream_t s) {
  if (ep.ky < 1 || ep.ky > 64) return cudaErrorInvalidValue;
  long long grid = (count + 7) / 8;
  if (grid > 16ll * device_sm_count()) grid = 16ll * device_sm_count();
  if (grid < 1) grid = 1;
  evaluate_kernel<<<static_cast<unsigned>(grid), 256, 0, s>>>(ep, idx, count, out, err);
  return cudaGetLastError();
}

// Grouping pays from some count on.  Entry by entry costs ~0.02 ns (kx + 8) an
// entry (1048576 entries at 400^3: 345, 552, 879 us for a whole call at ranks 6,
// 16, 32); grouped, the same take 140, 150, 200 with ~40 us of sorting launches,
// which 65536 entries do not earn back at rank 32 (139 against 156) and just do
// at rank 40 (151 against 144).  With few entries a row the blocks mostly wait
// for the next row: 262144 entries of 1400 rows still gain (299 to 210 at rank
// 32), 65536 lose (143 to 225).
bool evaluate_groups(const EvalPlan &ep, long long count) {
  const EvalSide &S0 = ep.side[0], &S1 = ep.side[1];
  return S0.W && !S1.W && S0.kx <= 64 && ep.ky <= 64 && S0.n_row <= kEvalGroupRows && S0.n_vec <= INT_MAX &&
         S1.n_vec <= INT_MAX && count >= 128 * S0.n_row && count * (S0.kx + 8) >= kEvalGroupMin;
}

cudaError_t evaluate_grouped_launch(const EvalPlan &ep, const EvalGroups &g, const long long *idx, long long count,
                                    float *out, int *err, cudaStream_t s, int *launches) {
  const EvalSide &S0 = ep.side[0], &S1 = ep.side[1];
  const int n = static_cast<int>(S0.n_row);
  const long long b0 = (S0.n_vec + 31) / 32, b1 = (S1.n_vec + 31) / 32;
  if (b0 + b1 > INT_MAX) return cudaErrorInvalidValue;
  eval_rows_kernel<<<static_cast<unsigned>(b0 + b1), 256, 0, s>>>(S0.Uv, S0.n_vec, S0.kx, g.Uq, static_cast<int>(b0),
                                                                  S1.Uv, S1.n_vec, ep.ky, g.Uc);
  ++*launches;
  for (long long e0 = 0; e0 < count; e0 += kEvalChunk) {
    const int cn = static_cast<int>(count - e0 < kEvalChunk ? count - e0 : kEvalChunk);
    const unsigned blocks = static_cast<unsigned>((cn + kSortEntries - 1) / kSortEntries);
    cudaError_t e = cudaMemsetAsync(g.hist, 0, 2 * sizeof(int) * n, s);   // hist, taken
    if (e != cudaSuccess) return e;
    const long long *ix = idx + e0 * ep.order;
    eval_count_kernel<<<blocks, kSortThreads, n * sizeof(int), s>>>(ix, cn, ep.order, S0.mode_row, n, g.hist);
    eval_sort_kernel<<<blocks, kSortThreads, 2 * n * sizeof(int), s>>>(ep, ix, cn, g.hist, g.hist + n, g.rec, err);
    const int k = ep.ky > S0.kx ? ep.ky : S0.kx;
    e = k <= 16   ? evaluate_grouped_kb<16>(ep, g, cn, out + e0, s)
        : k <= 32 ? evaluate_grouped_kb<32>(ep, g, cn, out + e0, s)
        : k <= 48 ? evaluate_grouped_kb<48>(ep, g, cn, out + e0, s)
                  : evaluate_grouped_kb<64>(ep, g, cn, out + e0, s);
    if (e != cudaSuccess) return e;
    *launches += 3;
  }
  return cudaSuccess;
}

}  // namespace htgb
