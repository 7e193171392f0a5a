// FP32-accurate GEMM over tensor matricisations on tcgen05: every FP32 operand
// is held as three BF16 planes, x = h + m / 2^7 + l / 2^14 (8 significant bits
// each), and a product is the six plane products h h', h m', m h', m m', h l',
// l h' (what is left out, m l' and below, is under 2^-24 of |x x'|).  The lower
// planes are stored 2^7 and 2^14 times up, because BF16's smallest subnormal is
// 2^-133 and FP32's last bit 2^-149: the sum is exact for every |x| >= 2^-124 and
// within 2^-148 of x below that (unscaled planes lose bits from 2^-110 down).  The
// tensor core takes the factors out again: its accumulator starts with the
// products 2^14 up and is scaled by 2^-7 as the next group comes in.  |m| and |l|
// stay below |x| / 2 and |x| / 4, so no sum overflows that h h' does not.
//
// What bounds it: the tensor pipe, at six BF16 MMAs per FP32 multiply-add --
// still several times the CUDA cores' FP32 rate, which the plain FP32 path
// (simt_gemm.cu) runs at; measured at about half of the pipe's rate, waiting for
// operand slots.  Three planes rather than two FP16 halves because BF16 has
// FP32's exponent range: no scaling pass, no range where small entries lose bits.
//   y (1024 x 8192) = W x^T, K = 1024       652 -> 97 us (x's planes: 11 us)
//   Gram of a 397-mode, K = 78260          1575 -> 142 us
//   Xhat (1024^3) = W U^T, K = 32          2082 -> 840 us (5.1 TB/s of output)
//   error pass over 301 x 260 x 397, K = 24  121 -> 64 us
// Error against 64 bits: 7e-8 to 2e-7 of the result's norm where the FP32 chains
// had 1.5e-7 to 9e-7.
//
// Accumulation.  tcgen05 adds into its FP32 accumulator with truncation, so a
// long K range summed in TMEM would carry a bias of ~2^-24 per step.  The
// accumulator therefore only ever holds one K block of 64 (the 2^14 products
// m m', h l', l h' first, then h m', m h', the four h h' steps last); the epilogue warps drain it after every K
// block and add it to FP32 sums in registers, rounding to nearest.  Two
// accumulators take turns, so the drain of one overlaps the MMAs of the other.
//
// CTA: warp 0 TMA producer, warp 1 TMEM allocator and MMA issuer, warps 2..17
// (BN = 256; else 2..9) drain (warp w: TMEM lane quarter w % 4, BN / 4 or BN / 2
// columns).  Sixteen drain warps because a K block's or a tile's drain is a long
// serial instruction stream per warp.
// One CTA per SM walks the work items (tiles x K splits): loads, MMAs, drains
// and stores of successive items overlap, so a product with few K blocks runs
// at the speed of its output's bytes.  OUT_SQDIFF stores nothing: the drain
// warps read the matrix the product is compared with and sum the squared
// differences (the error pass of a decomposition).
// Tile 128 x BN; a ring of plane slots (one plane of A and of B, 64 deep in K),
// filled and freed in the order l, m, h, so that a K block's first slots are
// refilled while its last products run.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <mutex>

#include "common.cuh"
#include "engine.h"
#include "tiles.cuh"

namespace htgb {
namespace {

constexpr int T3_BM = 128;
constexpr int T3_BK = 64;

template <int BN, int NSLOT>
struct T3Cfg {
  static constexpr int EW = BN == 256 ? 16 : 8;   // drain warps: 4 lane quarters x column groups
  static constexpr int HC = BN * 4 / EW;          // columns per drain warp
  static constexpr int THREADS = 64 + 32 * EW;
  static constexpr uint32_t A_BYTES = T3_BM * T3_BK * 2;
  static constexpr uint32_t SLOT = A_BYTES + BN * T3_BK * 2;
  static constexpr size_t SMEM = 1024 + size_t(NSLOT) * SLOT + 256;
  static constexpr uint32_t TMEM_COLS = 2 * BN;
};

struct T3Params {
  int a_kind, b_kind;
  int a_lblocks, b_lblocks;
  int num_kb, kb_per_split;
  int num_tiles, work, out_mode;   // work items: tiles x splits, walked by a CTA in steps of the grid
  float *out;                   // OUT_SQDIFF: the matrix the product is compared with (read only)
  long long ld_out;
  int *err;
  double *parts;                // OUT_SQDIFF: one sum of squared differences per CTA
  long long a_len;              // extent of A's contiguous K run: d0 (K-major) or d1 (MN-major)
  Fp32Operand a32, b32;         // read when *guard is set (see t3_fallback)
  const int *guard;
  const float *bias;            // added to row r of a column-major output (bias[out_row + r]), or null
  int relu;
};

HT_DEV void mbar_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

HT_DEV void tma_load_4d(void *smem_dst, const void *tmap, uint64_t *bar, int c0, int c1, int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5, %6}], [%2];" ::"r"(smem_u32(smem_dst)),
      "l"(tmap), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}

// 32 lanes x 16 consecutive 32-bit columns
HT_DEV void tmem_ld_32x32b_x16(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// D = D / 2^7 + A B^T, as umma_f16 otherwise
HT_DEV void umma_f16_down7(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.eq.u32 p, 0, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p, 7;\n\t}" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc)
      : "memory");
}

template <int ROWS>
HT_DEV void t3_load(const CUtensorMap *map, int kind, int lblocks, int kb, int row, int z, int plane, uint8_t *dst,
                    uint64_t *bar) {
  if (kind == OP_MN3) {
#pragma unroll
    for (int c = 0; c < ROWS / 64; ++c) tma_load_4d(dst + c * 8192, map, bar, row + 64 * c, kb * T3_BK, z, plane);
  } else {
    const int lb = kb % lblocks, r = kb / lblocks;
    if (kind == OP_KM3) tma_load_4d(dst, map, bar, lb * T3_BK, row, r, plane);
    else tma_load_4d(dst, map, bar, lb * T3_BK, r, row, plane);
  }
}

HT_DEV uint64_t t3_desc(int kind, uint32_t base, int kk) {
  if (kind == OP_MN3) return make_sdesc_sw128(base + kk * 2048, 8192, 1024);
  return make_sdesc_sw128(base + kk * 32, 16, 1024);
}

// The launch's product from its FP32 operands, when an entry had no planes
// (split3_kernel).  Data with infinities or NaN comes in earnest (a diverged
// training step), so its call has to stay near the CUDA cores' rate: for the
// forward of 8192 x 1024 x 1024 a thread per four outputs straight from global
// memory took 36.9 ms, this takes 0.97 and simt_gemm_kernel's tiles 0.67.
// Parts of SC columns of a tile are walked with 32-deep slices of both operands
// in two shared-memory stages, the next slice (also the next part's first) on its
// way in registers; a thread forms 8 rows x 4 columns.
template <int BN, int NSLOT>
struct T3Fallback {
  using C = T3Cfg<BN, NSLOT>;
  static constexpr int NT = 32 * C::EW, SC = NT / 4, SUB = BN / SC, KC = T3_BK / 2;
  static constexpr int LDA = T3_BM + 4, LDB = SC + 4, STAGE = KC * (LDA + LDB);   // floats
  static_assert(2 * STAGE * sizeof(float) <= size_t(NSLOT) * C::SLOT, "two stages in the ring's memory");
};

// A thread's quads of the ROWS x KC slice of one operand: four consecutive
// entries along whichever index is contiguous, neighbouring threads on
// neighbouring quads.  Entry (i, l) is kept at row l, with the groups of four i
// permuted by l's group, so that storing quads along l meets no bank twice.
HT_DEV int t3_group(int g, int l) { return 4 * (g ^ ((l >> 2) & 7)); }
template <int ROWS, int LD, int THREADS>
struct T3Slice {
  static constexpr int KC = T3_BK / 2, QUADS = ROWS * KC / 4, NV = (QUADS + THREADS - 1) / THREADS;
  float4 v[NV];
  // entries i < n_rows, l < n_l of src (steps rs, ls); zeros past them
  HT_DEV void load(const float *src, long long rs, long long ls, int n_rows, int n_l) {
#pragma unroll
    for (int q = 0; q < NV; ++q) {
      const int e = threadIdx.x + q * THREADS;
      const int i = rs == 1 ? 4 * (e % (ROWS / 4)) : e / (KC / 4), l = rs == 1 ? e / (ROWS / 4) : 4 * (e % (KC / 4));
      v[q] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (e >= QUADS || i >= n_rows || l >= n_l) continue;
      const float *from = src + i * rs + l * ls;
      const int n = rs == 1 ? n_rows - i : n_l - l;   // entries of the quad inside the slice
      if (n >= 4 && (reinterpret_cast<uintptr_t>(from) & 15u) == 0) {
        v[q] = __ldg(reinterpret_cast<const float4 *>(from));
      } else {
        v[q].x = __ldg(from);
        if (n > 1) v[q].y = __ldg(from + 1);
        if (n > 2) v[q].z = __ldg(from + 2);
        if (n > 3) v[q].w = __ldg(from + 3);
      }
    }
  }
  HT_DEV void store(bool rows_contiguous, float *dst) const {
#pragma unroll
    for (int q = 0; q < NV; ++q) {
      const int e = threadIdx.x + q * THREADS;
      if (e >= QUADS) continue;
      if (rows_contiguous) {
        const int l = e / (ROWS / 4);
        *reinterpret_cast<float4 *>(dst + l * LD + t3_group(e % (ROWS / 4), l)) = v[q];
      } else {
        const int i = e / (KC / 4), l = 4 * (e % (KC / 4));
        float *d = dst + l * LD + t3_group(i >> 2, l) + (i & 3);
        d[0] = v[q].x;
        d[LD] = v[q].y;
        d[2 * LD] = v[q].z;
        d[3 * LD] = v[q].w;
      }
    }
  }
};

template <int BN, int NSLOT>
__device__ __noinline__ void t3_fallback(const T3Params &p, const TileGen &gen, float *sm) {
  using F = T3Fallback<BN, NSLOT>;
  constexpr int THREADS = F::C::THREADS;
  const int t = threadIdx.x, rg = t % 16, cg = t / 16;
  const long long ars = p.a32.rs, als = p.a32.ls, brs = p.b32.rs, bls = p.b32.ls;
  // part w: columns [col0, col0 + SC) of item w % work's tile (first every item's
  // first columns: a last tile may have no others)
  auto part = [&](int w, int &col0, int &tile_idx, int &split) {
    const int sub = w / p.work, item = w - sub * p.work;
    col0 = sub * F::SC;
    tile_idx = item % p.num_tiles;
    split = item / p.num_tiles;
    return gen_tile(gen, tile_idx);
  };
  // the slice being fetched: slice i of part w, n deep
  int w = blockIdx.x, i = 0, n = 0, slices = 0, kb0 = 0, rows = 0, cols = 0;
  const float *arow = nullptr, *brow = nullptr;
  const float *a = nullptr, *b = nullptr;
  const int parts = p.work * F::SUB;
  auto locate = [&]() {   // slice i's entries and depth
    const bool amn = p.a_kind == OP_MN3, bmn = p.b_kind == OP_MN3;
    const int kb = kb0 + i / 2, h = (i & 1) * F::KC;
    const int ar = amn ? 0 : kb / p.a_lblocks, br = bmn ? 0 : kb / p.b_lblocks;
    const long long al = (kb - static_cast<long long>(ar) * p.a_lblocks * !amn) * T3_BK + h;
    const long long bl = (kb - static_cast<long long>(br) * p.b_lblocks * !bmn) * T3_BK + h;
    n = static_cast<int>(max(0ll, min(static_cast<long long>(F::KC), min(p.a32.len - al, p.b32.len - bl))));
    a = arow + al * als + ar * p.a32.rr;
    b = brow + bl * bls + br * p.b32.rr;
  };
  auto open = [&]() {   // part w, or the next of this CTA's that has columns
    for (; w < parts; w += gridDim.x) {
      int col0, tile_idx, split;
      const Tile tile = part(w, col0, tile_idx, split);
      if (p.out_mode != OUT_PARTIAL && col0 >= tile.valid_cols) continue;
      rows = tile.valid_rows;
      cols = tile.valid_cols - col0;
      arow = p.a32.p + tile.a_z * p.a32.zs + tile.a_row * ars;
      brow = p.b32.p + (tile.b_row + col0) * brs;
      kb0 = split * p.kb_per_split;
      slices = 2 * max(0, min(p.num_kb, kb0 + p.kb_per_split) - kb0);
      i = n = 0;
      if (slices) locate();   // (a split without K blocks: zeros)
      return;
    }
  };
  auto advance = [&]() {
    while (++i < slices) {
      locate();
      if (n > 0) return;
    }
    w += gridDim.x;
    open();
  };
  T3Slice<T3_BM, F::LDA, THREADS> sa;
  T3Slice<F::SC, F::LDB, THREADS> sb;
  float2 acc[4][4];   // [column][pair of rows: 4 rg, 4 rg + 2, 64 + 4 rg, ...]
  auto clear = [&]() {
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int r = 0; r < 4; ++r) acc[j][r] = make_float2(0.f, 0.f);
  };
  clear();
  open();
  if (w < parts) {
    sa.load(a, ars, als, rows, n);
    sb.load(b, brs, bls, cols, n);
  }
  for (int stage = 0; w < parts; stage ^= 1) {
    float *As = sm + stage * F::STAGE, *Bs = As + F::KC * F::LDA;
    sa.store(ars == 1, As);
    sb.store(brs == 1, Bs);
    __syncthreads();   // (and the other stage's slice is used up)
    const int w0 = w, n0 = n;
    advance();
    if (w < parts) {
      sa.load(a, ars, als, rows, n);
      sb.load(b, brs, bls, cols, n);
    }
    if (t >= F::NT) continue;
#pragma unroll 4
    for (int l = 0; l < n0; ++l) {
      const float4 a0 = *reinterpret_cast<const float4 *>(As + l * F::LDA + t3_group(rg, l));
      const float4 a1 = *reinterpret_cast<const float4 *>(As + l * F::LDA + 64 + t3_group(rg, l));
      const float4 b4 = *reinterpret_cast<const float4 *>(Bs + l * F::LDB + t3_group(cg, l));
      const float bj[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 x = make_float2(bj[j], bj[j]);
        fma2(acc[j][0], x, make_float2(a0.x, a0.y));
        fma2(acc[j][1], x, make_float2(a0.z, a0.w));
        fma2(acc[j][2], x, make_float2(a1.x, a1.y));
        fma2(acc[j][3], x, make_float2(a1.z, a1.w));
      }
    }
    if (w == w0) continue;
    int col0, tile_idx, split;   // that was the part's last slice
    const Tile tile = part(w0, col0, tile_idx, split);
    const int col = col0 + 4 * cg;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const int row = (r < 4 ? 0 : 64) + 4 * rg + (r & 3);
      float v[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = r & 1 ? acc[j][r / 2].y : acc[j][r / 2].x;
      if (p.out_mode == OUT_PARTIAL) {
        float *dst = p.out + ((static_cast<size_t>(split) * p.num_tiles + tile_idx) * T3_BM + row) * BN + col;
        *reinterpret_cast<float4 *>(dst) = make_float4(v[0], v[1], v[2], v[3]);
      } else if (row < tile.valid_rows) {
        const float bias = p.bias ? p.bias[tile.out_row + row] : 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (p.bias) v[j] += bias;
          if (p.relu) v[j] = fmaxf(v[j], 0.f);
          if (col + j < tile.valid_cols)
            p.out[tile.out_row + row + p.ld_out * static_cast<long long>(tile.out_col + col + j)] = v[j];
        }
      }
    }
    clear();
  }
}

template <int BN, int NSLOT>
__global__ void __launch_bounds__((T3Cfg<BN, NSLOT>::THREADS), 1)
    tc3_gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                    const __grid_constant__ T3Params p, const __grid_constant__ TileGen gen) {
  using C = T3Cfg<BN, NSLOT>;
  constexpr int HC = C::HC;
  __shared__ double wsum[C::EW];
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t *full = reinterpret_cast<uint64_t *>(smem + NSLOT * C::SLOT);
  uint64_t *empty = full + NSLOT;
  uint64_t *tfull = empty + NSLOT;
  uint64_t *tempty = tfull + 2;
  uint64_t *idle = tempty + 2;   // an abandoned CTA's MMAs have ended
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(idle + 1);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);

  if (p.guard && *p.guard != 0) {   // the same answer in every thread of the grid
    t3_fallback<BN, NSLOT>(p, gen, reinterpret_cast<float *>(smem));
    return;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // work item w: split w / num_tiles of the K range of tile w % num_tiles
  auto k_begin = [&](int w) { return w / p.num_tiles * p.kb_per_split; };
  auto k_count = [&](int kb0) { return max(0, min(p.num_kb, kb0 + p.kb_per_split) - kb0); };

  if (threadIdx.x == 0) {
    for (int s = 0; s < NSLOT; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&tfull[s], 1);
      mbar_init(&tempty[s], C::EW);
    }
    mbar_init(idle, 1);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, C::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      int it = 0;   // slots filled so far
      for (int w = blockIdx.x; w < p.work && !*abort_flag; w += gridDim.x) {
        const Tile tile = gen_tile(gen, w % p.num_tiles);
        const int kb0 = k_begin(w), n = 3 * k_count(kb0);
        for (int i = 0; i < n; ++i, ++it) {
          const int s = it % NSLOT;
          if (!mbar_wait_bounded(&empty[s], ((it / NSLOT) & 1) ^ 1, abort_flag)) {
            *abort_flag = 1;
            report_error(p.err, kErrTimeout);
            break;
          }
          const int kb = kb0 + i / 3, plane = 2 - i % 3;   // l, m, h
          uint8_t *sa = smem + s * C::SLOT;
          mbar_arrive_expect_tx(&full[s], C::SLOT);
          t3_load<T3_BM>(&tmA, p.a_kind, p.a_lblocks, kb, tile.a_row, tile.a_z, plane, sa, &full[s]);
          t3_load<BN>(&tmB, p.b_kind, p.b_lblocks, kb, tile.b_row, 0, plane, sa + C::A_BYTES, &full[s]);
        }
      }
      if (*abort_flag) {
        // let copies still in flight land before the CTA's shared memory is released
        for (int i = max(0, it - NSLOT); i < it; ++i) {
          int dummy = 0;
          mbar_wait_bounded(&full[i % NSLOT], (i / NSLOT) & 1, &dummy);
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t idesc = make_idesc_bf16(BN, p.a_kind == OP_MN3, p.b_kind == OP_MN3);
      int it = 0, kc = 0;   // slots and K blocks consumed so far
      bool ok = true;
      for (int w = blockIdx.x; w < p.work && ok; w += gridDim.x) {
       const int kb0 = k_begin(w), nk = k_count(kb0);
       for (int i = 0; i < nk; ++i, ++kc, it += 3) {
        ok = false;
        const int set = kc & 1;
        if (!mbar_wait_bounded(&tempty[set], ((kc >> 1) & 1) ^ 1, abort_flag)) {
          *abort_flag = 1;
          report_error(p.err, kErrTimeout);
          break;
        }
        tc_fence_after();
        const uint32_t d = tmem + static_cast<uint32_t>(set * BN);
        const int sl = it % NSLOT, sm = (it + 1) % NSLOT, sh = (it + 2) % NSLOT;
        const uint32_t am = smem_u32(smem + sm * C::SLOT), al = smem_u32(smem + sl * C::SLOT),
                       ah = smem_u32(smem + sh * C::SLOT);
        // 16-wide K steps that hold data (the rest of the block is zero fill)
        const int kb = kb0 + i;
        const long long left = p.a_len - static_cast<long long>(p.a_kind == OP_MN3 ? kb : kb % p.a_lblocks) * T3_BK;
        const int steps = left >= T3_BK ? T3_BK / 16 : max(1, (static_cast<int>(left) + 15) / 16);
        // D = (down ? D / 2^7 : D or nothing) + a b over the block's steps
        auto product = [&](uint32_t a, uint32_t b, bool fresh, bool down) {
          for (int kk = 0; kk < steps; ++kk) {
            const uint64_t da = t3_desc(p.a_kind, a, kk), db = t3_desc(p.b_kind, b + C::A_BYTES, kk);
            if (down && kk == 0) umma_f16_down7(d, da, db, idesc);
            else umma_f16(d, da, db, idesc, fresh && kk == 0 ? 0u : 1u);
          }
        };
        auto ready = [&](int j) {
          if (mbar_wait_bounded(&full[j % NSLOT], (j / NSLOT) & 1, abort_flag)) return true;
          *abort_flag = 1;
          report_error(p.err, kErrTimeout);
          return false;
        };
        if (!ready(it) || !ready(it + 1)) break;
        tc_fence_after();
        product(am, am, true, false);
        if (!ready(it + 2)) break;
        tc_fence_after();
        product(ah, al, false, false);
        product(al, ah, false, false);
        umma_commit(&empty[sl]);
        product(ah, am, false, true);
        product(am, ah, false, false);
        umma_commit(&empty[sm]);
        product(ah, ah, false, true);
        umma_commit(&empty[sh]);
        umma_commit(&tfull[set]);
        ok = true;
       }
      }
      if (!ok) {
        // a wait ran out with products under way: they read this CTA's shared memory
        // and write its accumulators, which are freed only once they have ended (the
        // drain warps wait for none of them)
        int dummy = 0;
        umma_commit(idle);
        mbar_wait_bounded(idle, 0, &dummy);
      }
    }
    __syncwarp();
  } else {
    const int q = warp & 3, c0 = ((warp - 2) >> 2) * HC;
    const int row = q * 32 + lane;
    const uint32_t lane_base = tmem + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>(c0);
    int kc = 0;
    bool ok = true;
    Acc2 sq = {0.f, 0.f};   // OUT_SQDIFF
    for (int w = blockIdx.x; w < p.work && ok; w += gridDim.x) {
      const int tile_idx = w % p.num_tiles, split = w / p.num_tiles;
      const Tile tile = gen_tile(gen, tile_idx);
      const int nk = k_count(k_begin(w));
      const bool in = row < tile.valid_rows;
      const int nc = tile.valid_cols - c0;
      const long long ld = p.ld_out, off = tile.out_row + row + ld * static_cast<long long>(tile.out_col + c0);
      // 16 finished columns c..c+15 of this thread's row
      auto finish = [&](int c, float (&v)[16]) {
        if (p.out_mode == OUT_SQDIFF) {
          const float *src = p.out + off + ld * c;
          float x[16];
          if (in && c + 16 <= nc) {
#pragma unroll
            for (int j = 0; j < 16; ++j, src += ld) x[j] = __ldcs(src);
          } else {
#pragma unroll
            for (int j = 0; j < 16; ++j, src += ld) {
              const bool live = in && c + j < nc;
              x[j] = live ? __ldcs(src) : 0.f;
              if (!live) v[j] = 0.f;
            }
          }
#pragma unroll
          for (int j = 0; j < 16; ++j) acc2_add_prod(sq, x[j] - v[j], x[j] - v[j]);
        } else if (p.out_mode == OUT_PARTIAL) {
          float *dst = p.out + ((static_cast<size_t>(split) * p.num_tiles + tile_idx) * T3_BM + row) * BN + c0 + c;
#pragma unroll
          for (int j = 0; j < 16; j += 4)
            *reinterpret_cast<float4 *>(dst + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
        } else if (in) {
          if (p.bias) {
            const float b = __ldg(p.bias + tile.out_row + row);
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] += b;
          }
          if (p.relu) {
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = fmaxf(v[j], 0.f);
          }
          float *dst = p.out + off + ld * c;
          if (c + 16 <= nc) {
#pragma unroll
            for (int j = 0; j < 16; ++j, dst += ld) *dst = v[j];
          } else {
#pragma unroll
            for (int j = 0; j < 16; ++j, dst += ld)
              if (c + j < nc) *dst = v[j];
          }
        }
      };
      auto drained = [&](int set) {   // this warp has read its part of the accumulator
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&tempty[set]);
      };
      auto filled = [&](int set) {
        ok = __all_sync(0xffffffffu, mbar_wait_bounded(&tfull[set], (kc >> 1) & 1, abort_flag));
        if (!ok && lane == 0) {
          *abort_flag = 1;
          report_error(p.err, kErrTimeout);
        }
        tc_fence_after();
        return ok;
      };
      if (nk == 1) {   // one K block: straight from the accumulator to the output
        const int set = kc & 1;
        if (!filled(set)) break;
        const uint32_t base = lane_base + static_cast<uint32_t>(set * BN);
#pragma unroll 1
        for (int c = 0; c < HC; c += 16) {
          float v[16];
          tmem_ld_32x32b_x16(base + static_cast<uint32_t>(c), v);
          tmem_ld_wait();
          if (c + 16 == HC) drained(set);
          finish(c, v);
        }
        ++kc;
        continue;
      }
      float acc[HC];
#pragma unroll
      for (int j = 0; j < HC; ++j) acc[j] = 0.f;
      for (int i = 0; i < nk; ++i, ++kc) {
        const int set = kc & 1;
        if (!filled(set)) break;
        const uint32_t base = lane_base + static_cast<uint32_t>(set * BN);
#pragma unroll
        for (int c = 0; c < HC; c += 16) {
          float v[16];
          tmem_ld_32x32b_x16(base + static_cast<uint32_t>(c), v);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; ++j) acc[c + j] += v[j];
        }
        drained(set);
      }
#pragma unroll
      for (int c = 0; c < HC; c += 16) {
        float v[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = acc[c + j];
        finish(c, v);
      }
    }
    if (p.out_mode == OUT_SQDIFF) {   // the CTA's sum: lanes, then warps, in a fixed order
      double d = static_cast<double>(sq.s) + static_cast<double>(sq.c);
      for (int o = 16; o > 0; o >>= 1) d += __shfl_down_sync(0xffffffffu, d, o);
      if (lane == 0) wsum[warp - 2] = d;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (p.out_mode == OUT_SQDIFF && threadIdx.x == 0) {
    double d = 0.0;
    for (int i = 0; i < C::EW; ++i) d += wsum[i];
    p.parts[blockIdx.x] = d;
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, C::TMEM_COLS);
  }
}

// ---------------------------------------------------------------- the planes
HT_DEV uint32_t pack2(float a, float b) {
  __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t *>(&v);
}
// (h, m, l) of a pair; each rest is exact, and so are the factors (a rest is at
// most half a unit of its plane's last place)
HT_DEV void split_pair(float x, float y, uint32_t &h, uint32_t &m, uint32_t &l) {
  h = pack2(x, y);
  const float rx = 128.f * (x - __uint_as_float(h << 16)), ry = 128.f * (y - __uint_as_float(h & 0xffff0000u));
  m = pack2(rx, ry);
  l = pack2(128.f * (rx - __uint_as_float(m << 16)), 128.f * (ry - __uint_as_float(m & 0xffff0000u)));
}

// Block sum of the compensated sums of squares -> partials[blockIdx.x].
HT_DEV void block_sumsq(const Acc2 &a, double *partials) {
  __shared__ double red[256];
  red[threadIdx.x] = static_cast<double>(a.s) + static_cast<double>(a.c);
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) partials[blockIdx.x] = red[0];
}

// x (n1 x rest, FP32, first index fastest) -> planes (n1p x rest each, rows
// n1 <= i < n1p zero; n1p a multiple of 8 so that TMA can address the rows).
// An entry whose first plane is not finite (NaN, infinite, or rounded up past
// the largest BF16) has no three-plane form: infinity minus infinity in its
// lower planes would turn every product it meets into NaN.  Such an entry
// sets *flag, which the caller's first launch cleared, and the product's launch
// then takes its FP32 operands instead (t3_fallback).
// A thread forms 8 consecutive elements of all planes: one 16-byte store per
// plane, and two 16-byte loads when x's rows are 16-byte aligned (VEC).  Bound
// by HBM: 4 B read and 6 B written per element.
template <bool VEC, bool SQ>
__global__ void __launch_bounds__(256) split3_kernel(const float *__restrict__ x, __nv_bfloat16 *__restrict__ planes,
                                                     long long plane, long long n1, long long n1p, long long rest,
                                                     double *partials, int *flag) {
  Acc2 a = {0.f, 0.f};
  bool bad = false;
  const long long v1 = n1p / 8, total = v1 * rest;
  for (long long e = blockIdx.x * 256ll + threadIdx.x; e < total; e += gridDim.x * 256ll) {
    float v[8];
    if (VEC) {   // n1 == n1p
      const float4 a0 = __ldg(reinterpret_cast<const float4 *>(x) + 2 * e);
      const float4 a1 = __ldg(reinterpret_cast<const float4 *>(x) + 2 * e + 1);
      v[0] = a0.x; v[1] = a0.y; v[2] = a0.z; v[3] = a0.w;
      v[4] = a1.x; v[5] = a1.y; v[6] = a1.z; v[7] = a1.w;
    } else {
      const long long r = e / v1, i0 = (e - r * v1) * 8;
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = i0 + j < n1 ? __ldg(x + i0 + j + n1 * r) : 0.f;
    }
    uint32_t h[4], m[4], l[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (SQ) {
        acc2_add_prod(a, v[2 * j], v[2 * j]);
        acc2_add_prod(a, v[2 * j + 1], v[2 * j + 1]);
      }
      split_pair(v[2 * j], v[2 * j + 1], h[j], m[j], l[j]);
      bad |= (h[j] & 0x7f800000u) == 0x7f800000u || (h[j] & 0x7f80u) == 0x7f80u;
    }
    *reinterpret_cast<uint4 *>(planes + 8 * e) = make_uint4(h[0], h[1], h[2], h[3]);
    *reinterpret_cast<uint4 *>(planes + plane + 8 * e) = make_uint4(m[0], m[1], m[2], m[3]);
    *reinterpret_cast<uint4 *>(planes + 2 * plane + 8 * e) = make_uint4(l[0], l[1], l[2], l[3]);
  }
  if (flag && bad) *flag = 1;   // every writer stores the same value
  if (SQ) block_sumsq(a, partials);
}

// Two arrays in one launch (a layer's x and dy), 8 elements a thread.
struct SplitJob {
  const float *x;
  __nv_bfloat16 *planes;
  long long plane, n8;
};
__global__ void __launch_bounds__(256) split3_pair_kernel(const SplitJob j0, const SplitJob j1, int *flag) {
  bool bad = false;
  for (long long e = blockIdx.x * 256ll + threadIdx.x; e < j0.n8 + j1.n8; e += gridDim.x * 256ll) {
    const bool second = e >= j0.n8;
    const SplitJob &J = second ? j1 : j0;
    const long long i = second ? e - j0.n8 : e;
    const float4 a0 = __ldg(reinterpret_cast<const float4 *>(J.x) + 2 * i);
    const float4 a1 = __ldg(reinterpret_cast<const float4 *>(J.x) + 2 * i + 1);
    const float v[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
    uint32_t h[4], m[4], l[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      split_pair(v[2 * q], v[2 * q + 1], h[q], m[q], l[q]);
      bad |= (h[q] & 0x7f800000u) == 0x7f800000u || (h[q] & 0x7f80u) == 0x7f80u;
    }
    *reinterpret_cast<uint4 *>(J.planes + 8 * i) = make_uint4(h[0], h[1], h[2], h[3]);
    *reinterpret_cast<uint4 *>(J.planes + J.plane + 8 * i) = make_uint4(m[0], m[1], m[2], m[3]);
    *reinterpret_cast<uint4 *>(J.planes + 2 * J.plane + 8 * i) = make_uint4(l[0], l[1], l[2], l[3]);
  }
  if (flag && bad) *flag = 1;
}

PFN_cuTensorMapEncodeTiled_v12000 t3_encode() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void *f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(f);
  });
  return fn;
}

bool t3_operand_ok(const Operand &o, long long plane) {
  const long long d[3] = {o.d0, o.d1, o.d2};
  for (int i = 0; i < 3; ++i)
    if (d[i] < 1 || d[i] > (1ll << 31) - 1) return false;
  return o.ptr && o.d0 % 8 == 0 && o.s1 % 8 == 0 && o.s2 % 8 == 0 && plane % 8 == 0 && (reinterpret_cast<uintptr_t>(o.ptr) & 15u) == 0;
}

bool t3_map(const Operand &o, long long plane, int rows_box, CUtensorMap *map) {
  auto enc = t3_encode();
  if (!enc) return false;
  cuuint64_t dims[4] = {cuuint64_t(o.d0), cuuint64_t(o.d1), cuuint64_t(o.d2), 3};
  const cuuint64_t s1 = o.s1 ? o.s1 : o.d0, s2 = o.s2 ? o.s2 : cuuint64_t(o.d0) * cuuint64_t(o.d1);
  cuuint64_t strides[3] = {s1 * 2, s2 * 2, cuuint64_t(plane) * 2};
  cuuint32_t box[4] = {T3_BK, 1, 1, 1};
  if (o.kind == OP_KM3) box[1] = rows_box;
  else if (o.kind == OP_KM3Q) box[2] = rows_box;
  else { box[0] = 64; box[1] = T3_BK; }
  cuuint32_t estr[4] = {1, 1, 1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void *>(o.ptr), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

long t3_kblocks(const Operand &o) {
  if (o.kind == OP_MN3) return (o.d1 + T3_BK - 1) / T3_BK;
  return (o.d0 + T3_BK - 1) / T3_BK * (o.kind == OP_KM3 ? o.d2 : o.d1);
}

int tc3_grid(int work) { return std::min(work, device_sm_count()); }

template <int BN, int NSLOT>
cudaError_t t3_launch(const Gemm3Args &g, cudaStream_t s) {
  using C = T3Cfg<BN, NSLOT>;
  if (g.gen.bm != T3_BM || g.gen.bn != BN) return cudaErrorInvalidValue;
  static bool done[64] = {};
  cudaError_t e = opt_in_smem(tc3_gemm_kernel<BN, NSLOT>, int(C::SMEM), done);
  if (e != cudaSuccess) return e;
  CUtensorMap ma, mb;
  if (!t3_map(g.a, g.a_plane, T3_BM, &ma) || !t3_map(g.b, g.b_plane, BN, &mb)) return cudaErrorInvalidValue;
  T3Params p{};
  p.a_kind = g.a.kind;
  p.b_kind = g.b.kind;
  p.a_lblocks = int((g.a.d0 + T3_BK - 1) / T3_BK);
  p.b_lblocks = int((g.b.d0 + T3_BK - 1) / T3_BK);
  p.num_kb = int(t3_kblocks(g.a));
  const int splits = g.splits < 1 ? 1 : g.splits;
  p.kb_per_split = (p.num_kb + splits - 1) / splits;
  p.num_tiles = g.gen.count;
  p.work = g.gen.count * splits;
  p.parts = g.parts;
  p.out_mode = g.out_mode;
  p.out = g.out;
  p.ld_out = g.ld_out;
  p.err = g.err;
  p.a_len = g.a.kind == OP_MN3 ? g.a.d1 : g.a.d0;
  p.a32 = g.a32;
  p.b32 = g.b32;
  p.guard = g.out_mode == OUT_SQDIFF ? nullptr : g.guard;   // (the fallback stores its product)
  p.bias = g.bias;
  p.relu = g.relu;
  // guarded: enough CTAs for the fallback's parts of the tiles
  const int grid = p.guard ? int(std::min<long long>((long long)p.work * T3Fallback<BN, NSLOT>::SUB, device_sm_count()))
                           : tc3_grid(p.work);
  tc3_gemm_kernel<BN, NSLOT><<<grid, C::THREADS, C::SMEM, s>>>(ma, mb, p, g.gen);
  return cudaGetLastError();
}

}  // namespace

int tc3_sq_parts(const Gemm3Args &g) { return tc3_grid(g.gen.count); }

Fp32Operand fp32_operand(const Operand &o) {
  Fp32Operand f;
  f.p = static_cast<const float *>(o.ptr);
  if (o.kind == OP_MN3) {
    f.rs = 1; f.ls = o.d0; f.rr = 0; f.zs = static_cast<long long>(o.d0) * o.d1; f.len = o.d1;
  } else {
    f.ls = 1; f.len = o.d0; f.zs = 0;
    f.rs = o.kind == OP_KM3 ? o.d0 : static_cast<long long>(o.d0) * o.d1;
    f.rr = o.kind == OP_KM3 ? static_cast<long long>(o.d0) * o.d1 : o.d0;
  }
  return f;
}

long tc3_num_kblocks(const Operand &a) { return t3_kblocks(a); }

bool tc3_supported(const Operand &a, long long a_plane, const Operand &b, long long b_plane) {
  return t3_operand_ok(a, a_plane) && t3_operand_ok(b, b_plane) && t3_kblocks(a) == t3_kblocks(b) &&
         t3_kblocks(a) <= (1l << 29) && t3_encode() != nullptr;
}

cudaError_t tc3_gemm_launch(const Gemm3Args &g, cudaStream_t s) {
  switch (g.gen.bn) {
    case 64: return t3_launch<64, 8>(g, s);
    case 128: return t3_launch<128, 6>(g, s);
    case 256: return t3_launch<256, 4>(g, s);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t split3_launch(const float *x, __nv_bfloat16 *planes, long long plane, long long n1, long long n1p,
                          long long rest, double *partials, int num_partials, int *flag, cudaStream_t s) {
  if (n1 < 1 || n1p < n1 || n1p % 8 || rest < 1 || plane % 8 || plane < n1p * rest ||
      (reinterpret_cast<uintptr_t>(planes) & 15u) || (partials && num_partials < 1))
    return cudaErrorInvalidValue;
  const long long total = n1p / 8 * rest;
  const bool vec = n1 == n1p && (reinterpret_cast<uintptr_t>(x) & 15u) == 0;
  int grid = partials ? num_partials
                      : static_cast<int>(std::min<long long>((total + 255) / 256, 8ll * device_sm_count()));
  if (partials) {
    if (vec) split3_kernel<true, true><<<grid, 256, 0, s>>>(x, planes, plane, n1, n1p, rest, partials, flag);
    else split3_kernel<false, true><<<grid, 256, 0, s>>>(x, planes, plane, n1, n1p, rest, partials, flag);
  } else {
    if (vec) split3_kernel<true, false><<<grid, 256, 0, s>>>(x, planes, plane, n1, n1p, rest, nullptr, flag);
    else split3_kernel<false, false><<<grid, 256, 0, s>>>(x, planes, plane, n1, n1p, rest, nullptr, flag);
  }
  return cudaGetLastError();
}

cudaError_t split3_pair_launch(const float *x, __nv_bfloat16 *planes, long long plane, long long n, const float *x2,
                               __nv_bfloat16 *planes2, long long plane2, long long n2, int *flag,
                               cudaStream_t s) {
  if (n % 8 || n2 % 8 || ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(x2)) & 15u))
    return cudaErrorInvalidValue;
  const SplitJob j0{x, planes, plane, n / 8}, j1{x2, planes2, plane2, n2 / 8};
  const int grid = static_cast<int>(std::min<long long>((j0.n8 + j1.n8 + 255) / 256, 8ll * device_sm_count()));
  split3_pair_kernel<<<grid, 256, 0, s>>>(j0, j1, flag);
  return cudaGetLastError();
}

}  // namespace htgb
