// Device code of the eigen-solver (eig.cu), included once per largest block:
// HT_EIG_SMAX (32 or 64) in namespace HT_EIG_NS.  Most leaves of a batch have
// blocks of at most 32, whose solver needs half the shared memory and registers,
// so that four of its CTAs share an SM instead of two: 2.95 ms for the 1536
// leaves of 512 tensors of 32 to 160 a mode with one 64-wide solver, 2.06 with
// the two side by side.
namespace HT_EIG_NS {

constexpr int SMAX = HT_EIG_SMAX;   // largest block
constexpr int ESMAX = SMAX * (SMAX + 1) / 2;   // packed upper triangle
constexpr int GROUP = 8;                        // partials loaded at once by the reduction

// packed upper triangle, column-major: e = j(j+1)/2 + i, i <= j
HT_DEV void tri_index(int e, int &i, int &j) {
  int jj = static_cast<int>((sqrtf(8.f * e + 1.f) - 1.f) * 0.5f);
  while (jj * (jj + 1) / 2 > e) --jj;
  while ((jj + 1) * (jj + 2) / 2 <= e) ++jj;
  j = jj;
  i = e - jj * (jj + 1) / 2;
}

// 16-byte asynchronous global->shared copy; src_bytes < 16 zero-fills the rest.
HT_DEV void cp_async16(void *smem_dst, const void *gsrc, int src_bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(smem_dst)), "l"(gsrc), "r"(src_bytes)
               : "memory");
}
HT_DEV void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
HT_DEV void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Cyclic Jacobi on a symmetric s x s matrix held in shared memory (s <= SMAX),
// 256 or 1024 threads, round-robin ("circle method") ordering: every round rotates up
// to s/2 disjoint pairs.  On return A is diagonal to FP32 rounding, V holds the
// eigenvectors and order[] the indices by descending eigenvalue.  A2 is
// scratch of the same shape.
//
// Rotation rule.  A pair rotates while its coupling is above 2.4e-7 (two FP32
// units of rounding) relative to sqrt(a_pp a_qq), the test that keeps small
// eigenvalues' vectors accurate (Demmel and Veselic, "Jacobi's method is more
// accurate than QR", 1992).  The rotated pair's new diagonal is formed as
// a_pp - t a_pq, a_qq + t a_pq and its coupling set to exactly zero
// (Rutishauser's update), so rounding does not regenerate it and the test
// terminates even between null directions.  Rotations are applied as
// x - s (y + rho x), y + s (x - rho y) with rho = s / (1 + c): for the many
// tiny late rotations c rounds to 1, and the plain c x - s y form would then
// grow every column of V by s^2/2 per rotation (a 1e-5 loss of orthogonality
// after ten sweeps); this form carries that second-order term explicitly.
// The cosine is refined to FP32 rounding for its tangent (jac_choose): one that is
// a few units off makes every rotation slightly non-orthogonal, which the exact
// diagonal update then turns into absolute errors on small eigenvalues.  The
// tangent itself may be a few units off: that only leaves a coupling below the
// update's rounding, which the update sets to zero.
//
// Schedule.  Everything lives in position space: players (indices of the
// matrix) sit at m positions, pair a is positions a ("top") and m - 1 - a
// ("bottom"), and after a round the player of position x + 1 moves to x (x >= 1;
// position 1 goes to m - 1, position 0 stays): the circle method, in which
// player 1 + (x - 1 + round) mod (m - 1) sits at x.  A rotated entry is simply
// stored at its players' next positions, so no round looks up an index.
//
// One round is one phase between two barriers.  Its length is the next
// rotations' dependent chain (loads, four fused operations, square roots and
// reciprocals), which therefore runs beside the update and not between two, as
// long as the update's instructions fit beside it: every thread keeps the same
// 2 x 2 blocks of position space for the whole run, so that all its addresses
// are computed once.
//   blocks     A2 = J^T A J, a thread per block (a, b) of pairs a <= b: only the
//              entries (row, column) with row >= column are stored.
//   V rows     stay in the players' columns; a lane rotates the two of its pair
//              (moving them through registers instead takes two shuffles a row,
//              which at ~3 cycles each made the rows the longest part).
//   last warp  the NEXT round's rotations: lane a forms the three entries of its
//              next pair from the old A with the same arithmetic.
// One-CTA kernels of their own run it with 32 warps, blocks and V rows on
// different ones; the grouped solver, two CTAs to an SM, with 8.
// The iteration stops once m - 1 consecutive rounds (every pair once) chose no
// rotation, i.e. a full sweep left the matrix unchanged.
struct JacRot {   // of a pair's (top, bottom): x - sn (y + rho x), y + sn (x - rho y)
  float rho, sn, tt, rot;
};

// The hardware's approximate reciprocal and roots (a unit or two of rounding).
HT_DEV float approx_rcp(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
HT_DEV float approx_rsqrt(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
HT_DEV float approx_sqrt(float x) {
  float y;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
HT_DEV bool jac_rotates(float att, float abb, float atb) {
  return fabsf(atb) > 1e-30f && fabsf(atb) > 2.4e-7f * approx_sqrt(fabsf(att * abb));
}

// The rotation of the pair with diagonal (att, abb) and coupling atb of a matrix
// scaled to a largest diagonal entry of about one; every lane of the warp calls
// it.  flip: the top player has the larger index; the formulas take the smaller
// index first (which only matters when the diagonals are equal).
// t = 2 b / (d + sign(d) sqrt(d^2 + 4 b^2)) may be a few units of rounding off
// (approximate root and reciprocal): what it leaves of the coupling is below
// the rounding of the update.  The cosine that goes with that tangent is
// refined to FP32 rounding by a Newton step; 1 / (1 + c), c in [0.707, 1], is a
// linear estimate and two Newton steps.
HT_DEV JacRot jac_choose(bool flip, float att, float abb, float atb) {
  const float d = flip ? att - abb : abb - att, b2 = 2.f * atb;
  const float D = __fmaf_rn(d, d, b2 * b2);
  float ta = fabsf(b2) * approx_rcp(fabsf(d) + D * approx_rsqrt(D));
  const bool rot = jac_rotates(att, abb, atb);
  if (__any_sync(0xffffffffu, rot && !(D > 1e-34f))) {   // entries below 1e-17 of the largest: squares would underflow
    const float tau = fabsf(d) * approx_rcp(fabsf(b2));
    const float h = tau < 1.15e18f ? approx_sqrt(__fmaf_rn(tau, tau, 1.f)) : tau;
    if (!(D > 1e-34f)) ta = approx_rcp(tau + h);
  }
  const float tt = ((d >= 0.f) == (b2 >= 0.f) || d == 0.f) != flip ? ta : -ta;
  const float w = __fmaf_rn(ta, ta, 1.f);
  const float c0 = approx_rsqrt(w);
  const float c = __fmaf_rn(0.5f * c0, __fmaf_rn(-w * c0, c0, 1.f), c0);
  float y = __fmaf_rn(-0.29289322f, c, 0.79289322f);
  const float c1 = 1.f + c;
  y = __fmaf_rn(y, __fmaf_rn(-c1, y, 1.f), y);
  y = __fmaf_rn(y, __fmaf_rn(-c1, y, 1.f), y);
  const float sn = tt * c;
  return rot ? JacRot{sn * y, sn, tt, 1.f} : JacRot{0.f, 0.f, 0.f, 0.f};
}

// x - sn (y + rho x) for the top member of a pair (sn, rho as they are) or the
// bottom one (both negated), as explicit fused operations so that every thread
// that evaluates an entry gets the same bits.
HT_DEV float jac_mix(float rho, float sn, float x, float y) { return __fmaf_rn(-sn, __fmaf_rn(rho, x, y), x); }

HT_DEV int jac_player(int x, int round, int m) { return x == 0 ? 0 : 1 + (x - 1 + round) % (m - 1); }

// Position space: entry (x, y) at row max(x, y), column min(x, y) of rows of
// SMAX + 2 floats -- rows, the diagonal and the antidiagonal (a pair's coupling) are free
// of bank conflicts, columns two-way.
constexpr int JLD = SMAX + 2;
constexpr int kJacMat = (SMAX + 1) * (SMAX + 1);   // floats of a matrix buffer that holds it
static_assert((SMAX - 1) * JLD + SMAX <= kJacMat, "position space fits its buffers");
HT_DEV int jac_at(int x, int y) { return max(x, y) * JLD + min(x, y); }

// NT threads: 1024, or 256.  A, A2, V: kJacMat floats each.
template <int NT>
HT_DEV void jacobi_smem(float (*A)[SMAX + 1], float (*A2)[SMAX + 1], float (*V)[SMAX + 1], int s, int *order) {
  constexpr bool SPLIT = NT == 1024;                                  // blocks and V rows on different warps
  constexpr int UW = NT / 32 - 1;                                     // update warps
  constexpr int NBLK = (SMAX / 2) * (SMAX / 2 + 1) / 2;               // blocks of the largest matrix
  constexpr int BPT = SPLIT ? 1 : (NBLK + UW * 32 - 1) / (UW * 32);   // blocks per thread
  __shared__ __align__(16) JacRot Jbuf[2][SMAX / 2];
  __shared__ int s_any[2];
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int m = (s + 1) & ~1;   // even number of players (a dummy index, whose entries stay zero, when s is odd)
  const int np = m / 2, nblk = np * (np + 1) / 2;
  const int vw0 = SPLIT ? (nblk + 31) / 32 : 0, nvw = UW - vw0;
  // next position of the player at position x
  auto moved = [&](int x) { return x == 0 || m == 2 ? x : (x == 1 ? m - 1 : x - 1); };
  // scale by a power of two (exact) to a largest diagonal entry in [1, 2)
  float dmax = 0.f;
  for (int i = lane; i < s; i += 32) dmax = fmaxf(dmax, fabsf(A[i][i]));
  for (int o = 16; o > 0; o >>= 1) dmax = fmaxf(dmax, __shfl_xor_sync(0xffffffffu, dmax, o));
  const int ex = dmax > 0.f && dmax < INFINITY ? ilogbf(dmax) : 0;
  // this thread's blocks: pairs (a, b), where their entries are read and stored;
  // a thread without one works on the unused last words of the buffers
  unsigned ab[BPT], ld01[BPT], ld23[BPT], st01[BPT], st23[BPT];
#pragma unroll
  for (int k = 0; k < BPT; ++k) {
    const int e = t + UW * 32 * k;
    ab[k] = 0u;
    ld01[k] = ld23[k] = st01[k] = st23[k] = (kJacMat - 1) * 0x10001u;
    if (warp < UW && e < nblk) {
      int a, b;
      tri_index(e, a, b);
      const int ta = a, ba = m - 1 - a, tb = b, bb = m - 1 - b;
      ab[k] = static_cast<unsigned>(a | (b << 8));
      ld01[k] = static_cast<unsigned>(jac_at(ta, tb) | (jac_at(ta, bb) << 16));
      ld23[k] = static_cast<unsigned>(jac_at(ba, tb) | (jac_at(ba, bb) << 16));
      st01[k] = static_cast<unsigned>(jac_at(moved(ta), moved(tb)) | (jac_at(moved(ta), moved(bb)) << 16));
      st23[k] = static_cast<unsigned>(jac_at(moved(ba), moved(tb)) | (jac_at(moved(ba), moved(bb)) << 16));
    }
  }
  for (int e = t; e < s * m; e += NT) V[e / m][e % m] = e / m == e % m ? 1.f : 0.f;
  // last warp: the players that come to this lane's positions are at x and y
  const int x = m > 2 && lane > 0 && lane < np ? lane + 1 : 0, y = lane > 0 && lane < np ? m - lane : 1;
  const int ax = x < np ? x : m - 1 - x, ay = y < np ? y : m - 1 - y, px = m - 1 - x, py = m - 1 - y;
  const float gx = x < np ? 1.f : -1.f, gy = y < np ? 1.f : -1.f;
  const bool sw = ax > ay;   // rows: the pair of the smaller index; columns: the other one
  const int o_rc = jac_at(x, y), o_prc = sw ? jac_at(py, x) : jac_at(px, y), o_rpc = sw ? jac_at(y, px) : jac_at(x, py),
            o_prpc = jac_at(px, py);
  // players at this lane's pair, round 0: player x at position x
  int idt = lane < np ? lane : 0, idb = m - 1 - idt;
  auto next_player = [&](int id) { return id == 0 ? 0 : (id == m - 1 ? 1 : id + 1); };
  float *Ac = &A2[0][0], *An = &A[0][0];
  for (int e = t; e < m * m; e += NT) {
    const int i = e / m, j = e - i * m;
    if (i >= j) Ac[i * JLD + j] = i < s && j < s ? scalbnf(A[i][j], -ex) : 0.f;   // (the dummy player's entries are zero)
  }
  __syncthreads();
  if (warp == UW) {
    const int l = lane < np ? lane : 0, o = m - 1 - l;
    const JacRot j0 = jac_choose(false, Ac[jac_at(l, l)], Ac[jac_at(o, o)], Ac[jac_at(l, o)]);
    if (lane < np) Jbuf[0][lane] = j0;
    const int any = __any_sync(0xffffffffu, j0.rot != 0.f);
    if (lane == 0) s_any[0] = any;
  }
  __syncthreads();
  int quiet = 0;   // rounds in a row without a rotation
  const int max_rounds = m > 1 ? 20 * (m - 1) : 0;
  int rr = 0;      // rounds done, modulo m - 1: the players' offset
  for (int round = 0; round < max_rounds; ++round) {
    const JacRot *J = Jbuf[round & 1];
    const int rotates = s_any[round & 1];
    if (warp < UW) {
#pragma unroll
      for (int k = 0; k < BPT; ++k) {
        if (SPLIT && warp >= vw0) break;
        const int a = ab[k] & 255, b = ab[k] >> 8;
        const JacRot ja = J[a], jb = J[b];
        const float w = Ac[ld01[k] & 0xffff], u = Ac[ld01[k] >> 16], v = Ac[ld23[k] & 0xffff], z = Ac[ld23[k] >> 16];
        const float w1 = jac_mix(ja.rho, ja.sn, w, v), v1 = jac_mix(-ja.rho, -ja.sn, v, w);
        const float u1 = jac_mix(ja.rho, ja.sn, u, z), z1 = jac_mix(-ja.rho, -ja.sn, z, u);
        const bool diag = a == b;
        const float off = ja.rot != 0.f ? 0.f : u;
        An[st01[k] & 0xffff] = diag ? __fmaf_rn(-ja.tt, u, w) : jac_mix(jb.rho, jb.sn, w1, u1);
        An[st01[k] >> 16] = diag ? off : jac_mix(-jb.rho, -jb.sn, u1, w1);
        An[st23[k] & 0xffff] = diag ? off : jac_mix(jb.rho, jb.sn, v1, z1);
        An[st23[k] >> 16] = diag ? __fmaf_rn(ja.tt, u, z) : jac_mix(-jb.rho, -jb.sn, z1, v1);
      }
      if ((!SPLIT || warp >= vw0) && rotates && lane < np) {   // V <- V J, two rows at a time
        const JacRot jb = J[lane];
        for (int i = warp - vw0; i < s; i += 2 * nvw) {
          float *v0 = V[i], *v1 = V[i + nvw < s ? i + nvw : SMAX];   // (row SMAX: spare)
          const float p0 = v0[idt], q0 = v0[idb], p1 = v1[idt], q1 = v1[idb];
          v0[idt] = jac_mix(jb.rho, jb.sn, p0, q0);
          v0[idb] = jac_mix(-jb.rho, -jb.sn, q0, p0);
          v1[idt] = jac_mix(jb.rho, jb.sn, p1, q1);
          v1[idb] = jac_mix(-jb.rho, -jb.sn, q1, p1);
        }
      }
      idt = next_player(idt);
      idb = next_player(idb);
    } else {
      idt = next_player(idt);
      idb = next_player(idb);
      const JacRot jx = J[ax], jy = J[ay];
      const float arc = Ac[o_rc], aprc = Ac[o_prc], arpc = Ac[o_rpc], aprpc = Ac[o_prpc];
      const float att = __fmaf_rn(-gx * jx.tt, Ac[jac_at(x, px)], Ac[jac_at(x, x)]);
      const float abb = __fmaf_rn(-gy * jy.tt, Ac[jac_at(y, py)], Ac[jac_at(y, y)]);
      const float r1 = sw ? gy * jy.rho : gx * jx.rho, s1 = sw ? gy * jy.sn : gx * jx.sn;
      const float r2 = sw ? gx * jx.rho : gy * jy.rho, s2 = sw ? gx * jx.sn : gy * jy.sn;
      float atb = jac_mix(r2, s2, jac_mix(r1, s1, arc, aprc), jac_mix(r1, s1, arpc, aprpc));
      if (m == 2) atb = jx.rot != 0.f ? 0.f : arc;   // one pair only
      const JacRot jn = jac_choose(idt > idb, att, abb, atb);
      if (lane < np) Jbuf[(round & 1) ^ 1][lane] = jn;
      const int any = __any_sync(0xffffffffu, lane < np && jn.rot != 0.f);
      if (lane == 0) s_any[(round & 1) ^ 1] = any;
    }
    quiet = rotates ? 0 : quiet + 1;
    __syncthreads();
    rr = rr + 1 == m - 1 ? 0 : rr + 1;
    float *tmp = Ac;
    Ac = An;
    An = tmp;
    // first quiet round: if no pair of the whole matrix would rotate, the
    // remaining quiet rounds of the sweep would change nothing
    if (quiet == 1) {
      int bad = 0;
      for (int e = t; e < m * m; e += NT) {
        const int i = e / m, j = e - i * m;
        if (i > j && jac_rotates(Ac[i * JLD + i], Ac[j * JLD + j], Ac[i * JLD + j])) bad = 1;
      }
      if (!__syncthreads_or(bad)) break;
    }
    if (quiet >= m - 1) break;
  }
  // the diagonal back to the players' indices
  float dg = 0.f;
  if (t < m) dg = scalbnf(Ac[t * JLD + t], ex);
  __syncthreads();
  if (t < m) {
    const int j = jac_player(t, rr, m);
    if (j < s) A[j][j] = dg;
  }
  __syncthreads();
  // rank by counting: descending eigenvalues.  NaN counts as -inf and ties go
  // by index, so the ranks always form a permutation (order[] is used as an
  // index: a hole would be an out-of-range shared-memory access)
  for (int j = t; j < s; j += NT) {
    const float dj = isnan(A[j][j]) ? -INFINITY : A[j][j];
    int rank = 0;
    for (int i = 0; i < s; ++i) {
      const float di = isnan(A[i][i]) ? -INFINITY : A[i][i];
      if (di > dj || (di == dj && i < j)) ++rank;
    }
    order[rank] = j;
  }
  __syncthreads();
}

#if HT_EIG_SMAX == 64
// Transfer-tensor step of the complementary-leaf construction.  WG = W^T G_c W
// (kw x kw, leading dimension kw) for the complementary leaf's Ritz block W;
// V = W[:, :kt].  With GV = V^T G_c V = P diag(lam) P^T:
//   M     = P diag(lam^-1/2)   (columns with lam <= 1e-12 lam_max are zero)
//   Broot = M^T V^T G_c U_c    (kt x kc)
// and the caller forms B_t = C_V M.  On the columns U_c shares with V
// (u < min(kt, kc)) V^T G_c U_c = GV[:, u], so Broot = diag(lam^1/2) P^T there:
// writing it that way makes B_t Broot = C_V P P^T exactly, instead of relying on
// lam^-1 * lam cancelling in FP32, which fails for ill-conditioned Grams.
// Transfer-tensor eigen step on WG (kw x kw, leading dimension kw, global or
// shared memory): the top-kt eigenpairs of sym(WG[:kt, :kt]) by Jacobi give
// M (kt x kt) = V diag(lambda^-1/2) and the root transfer tensor
// Broot (kt x kc, or kc x kt when !t_is_left).
template <int NT>
HT_DEV void transfer_eig_body(const float *WG, int kw, int kt, int kc, int t_is_left, float *M, float *Broot,
                              float (*A)[SMAX + 1], float (*V)[SMAX + 1], float (*A2)[SMAX + 1], int *order,
                              float *inv) {
  const int t = threadIdx.x;
  for (int e = t; e < SMAX * SMAX; e += NT) {
    const int i = e % SMAX, j = e / SMAX;
    A[i][j] = (i < kt && j < kt) ? 0.5f * (WG[i + kw * j] + WG[j + kw * i]) : 0.f;
  }
  __syncthreads();
  jacobi_smem<NT>(A, A2, V, kt, order);
  if (t == 0) {
    const float lmax = A[order[0]][order[0]];
    for (int r = 0; r < kt; ++r) {
      const float l = A[order[r]][order[r]];
      inv[r] = (lmax > 0.f && l > 1e-12f * lmax) ? rsqrtf(l) : 0.f;
    }
  }
  __syncthreads();
  for (int e = t; e < kt * kt; e += NT) {
    const int i = e % kt, r = e / kt;
    M[i + kt * r] = V[i][order[r]] * inv[r];
  }
  __syncthreads();
  for (int e = t; e < kt * kc; e += NT) {
    const int r = e % kt, u = e / kt;
    const int oc = order[r];
    float acc;
    if (u < kt) {
      acc = inv[r] > 0.f ? sqrtf(A[oc][oc]) * V[u][oc] : 0.f;
    } else {
      acc = 0.f;
      for (int c = 0; c < kt; ++c) acc = fmaf(V[c][oc] * inv[r], 0.5f * (WG[c + kw * u] + WG[u + kw * c]), acc);
    }
    if (t_is_left) Broot[r + kt * u] = acc;
    else Broot[u + kc * r] = acc;
  }
}

constexpr int kJacThreads = 1024;   // one-CTA Jacobi kernels

__global__ void __launch_bounds__(kJacThreads) transfer_eig_kernel(const float *WG, int kw, int kt, int kc, int t_is_left,
                                                           float *M, float *Broot) {
  __shared__ float A[SMAX + 1][SMAX + 1];
  __shared__ float V[SMAX + 1][SMAX + 1];
  extern __shared__ float jac_scratch[];   // kJacMat floats
  float (*A2)[SMAX + 1] = reinterpret_cast<float (*)[SMAX + 1]>(jac_scratch);
  __shared__ int order[SMAX];
  __shared__ float inv[SMAX];
  transfer_eig_body<kJacThreads>(WG, kw, kt, kc, t_is_left, M, Broot, A, V, A2, order, inv);
}

// Grouped transfer tail of the batched path, a CTA per tensor:
//   WG = U^T GU (kw x kw, compensated dot products as gemm_tn_small),
//   the transfer eigen step (M, Bkt; Broot = Bkt^T when t is the right child),
//   Bt = C M (kpq x kt, as matmul_nn).
__global__ void __launch_bounds__(256) transfer_tail_grouped_kernel(const TailJob *__restrict__ jobs) {
  __shared__ float A[SMAX + 1][SMAX + 1];
  __shared__ float V[SMAX + 1][SMAX + 1];
  extern __shared__ float tail_sm[];   // A2 (kJacMat), WG (SMAX * SMAX), M (SMAX * SMAX)
  float (*A2)[SMAX + 1] = reinterpret_cast<float (*)[SMAX + 1]>(tail_sm);
  float *WG = tail_sm + kJacMat;
  float *Ms = WG + SMAX * SMAX;
  __shared__ int order[SMAX];
  __shared__ float inv[SMAX];
  __shared__ TailJob J;
  if (threadIdx.x == 0) J = jobs[blockIdx.x];
  __syncthreads();
  const int kw = J.kw, kt = J.kt, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int e = warp; e < kw * kw; e += 8) {
    const int i = e % kw, j = e / kw;
    Acc2 acc = {0.f, 0.f};
    for (int k = lane; k < J.nc; k += 32)
      acc2_add_prod(acc, J.U[k + static_cast<long long>(J.nc) * i], J.GU[k + static_cast<long long>(J.nc) * j]);
    double v = static_cast<double>(acc.s) + static_cast<double>(acc.c);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) WG[i + kw * j] = static_cast<float>(v);
  }
  __syncthreads();
  transfer_eig_body<256>(WG, kw, kt, J.kc, 1, Ms, J.Bkt, A, V, A2, order, inv);
  __syncthreads();
  for (int e = threadIdx.x; e < kt * J.kc && !J.t_is_left; e += 256) {
    const int i = e % kt, j = e / kt;
    J.Broot[j + J.kc * i] = J.Bkt[i + kt * j];
  }
  for (long long idx = threadIdx.x; idx < J.kpq * kt; idx += 256) {
    const long long i = idx % J.kpq;
    const int j = static_cast<int>(idx / J.kpq);
    float sacc = 0.f;
    for (int k = 0; k < kt; ++k) sacc = fmaf(J.C[i + J.kpq * k], Ms[k + kt * j], sacc);
    J.Bt[i + J.kpq * j] = sacc;
  }
}

// SVD of a tall W from its Gram GW = W^T W (s x s): GW = U diag(sigma^2) U^T.
// M1 = U[:, :k1], M2 = U[:, :k2] diag(1/sigma) (zero where sigma <= 1e-6 sigma_1),
// Broot = M1^T GW M2 (k1 x k2).
// Up to four independent problems, one CTA each (blockIdx.x).
struct SvdGramBatch {
  SvdGramProb p[4];
};

__global__ void __launch_bounds__(kJacThreads) svd_from_gram_kernel(const SvdGramBatch batch) {
  const SvdGramProb &pb = batch.p[blockIdx.x];
  const float *GW = pb.GW;
  const int s = pb.s, k1 = pb.k1, k2 = pb.k2;
  float *M1 = pb.M1, *M2 = pb.M2, *Broot = pb.Broot;
  __shared__ float A[SMAX + 1][SMAX + 1];
  __shared__ float V[SMAX + 1][SMAX + 1];
  extern __shared__ float jac_scratch[];   // kJacMat floats
  float (*A2)[SMAX + 1] = reinterpret_cast<float (*)[SMAX + 1]>(jac_scratch);
  __shared__ int order[SMAX];
  __shared__ float inv[SMAX];
  const int t = threadIdx.x;
  for (int e = t; e < SMAX * SMAX; e += kJacThreads) {
    const int i = e % SMAX, j = e / SMAX;
    A[i][j] = (i < s && j < s) ? 0.5f * (GW[i + s * j] + GW[j + s * i]) : 0.f;
  }
  __syncthreads();
  jacobi_smem<kJacThreads>(A, A2, V, s, order);
  if (t == 0) {
    const float s1 = sqrtf(fmaxf(A[order[0]][order[0]], 0.f));
    for (int r = 0; r < s; ++r) {
      const float sg = sqrtf(fmaxf(A[order[r]][order[r]], 0.f));
      inv[r] = (s1 > 0.f && sg > 1e-6f * s1) ? 1.f / sg : 0.f;
    }
  }
  __syncthreads();
  for (int e = t; e < s * k1; e += kJacThreads) {
    const int i = e % s, r = e / s;
    M1[i + s * r] = V[i][order[r]];
  }
  for (int e = t; e < s * k2; e += kJacThreads) {
    const int i = e % s, r = e / s;
    M2[i + s * r] = V[i][order[r]] * inv[r];
  }
  // Broot = M1^T (GW_sym V[:, order[:k2]]) diag(inv): the symmetrised Gram in
  // the Jacobi scratch, the product P = GW_sym V_k2 in A (its diagonal is read
  // above), both in shared memory
  for (int e = t; e < s * s; e += kJacThreads) {
    const int a = e % s, c = e / s;
    A2[a][c] = 0.5f * (GW[a + s * c] + GW[c + s * a]);
  }
  __syncthreads();
  for (int e = t; e < s * k2; e += kJacThreads) {
    const int a = e % s, j = e / s;
    const int oj = order[j];
    float g = 0.f;
    for (int c = 0; c < s; ++c) g = fmaf(A2[a][c], V[c][oj], g);
    A[a][j] = g;
  }
  __syncthreads();
  for (int e = t; e < k1 * k2; e += kJacThreads) {
    const int i = e % k1, j = e / k1;
    const int oi = order[i];
    float acc = 0.f;
    for (int a = 0; a < s; ++a) acc = fmaf(V[a][oi], A[a][j], acc);
    Broot[i + k1 * j] = acc * inv[j];
  }
}
#endif

// ------------------------------------------------------------------------
// Cooperative eigen-solver: the whole subspace iteration of every problem of
// the batch in ONE launch.  CTAs of one problem own consecutive row ranges;
// grid-wide barriers (bounded spins on a counter / generation pair) separate
// the phases, so there is no single-CTA tail per iteration: the s x s Gram
// partials are reduced by all CTAs (each sums a slice of the entries over the
// problem's CTAs, in CTA order) and every CTA of the problem factors the
// reduced Gram itself.  Direct problems (s == n) run in CTAs of their own that
// take no part in the barriers.
constexpr int RBMAX = 32;                 // rows per sub-block
constexpr int CNS = 4;                    // cp.async stages of the G * Y product
constexpr int CLD = 68;                   // padded k length of a staged row
constexpr int kMaxEntPerThread = (ESMAX + 255) / 256;

constexpr size_t kCoopAlias = 2 * ESMAX + 3 * kJacMat;                // Sd (doubles) + A + V + A2
// dynamic shared memory of a solver whose G * Y product runs a `stages`-deep ring
constexpr size_t coop_smem(int stages) {
  return sizeof(float) * (SMAX * SMAX + SMAX + 2 * RBMAX * SMAX +
                          (size_t(stages) * (RBMAX + SMAX) * CLD > kCoopAlias ? size_t(stages) * (RBMAX + SMAX) * CLD
                                                                                : kCoopAlias)) +
         64;
}
constexpr size_t kCoopSmem = coop_smem(CNS);
// the grouped solver (a CTA per problem): a 2-stage ring, so that two CTAs share
// an SM (four at SMAX = 32)
constexpr int kGroupedStages = 2;
constexpr size_t kGroupedSmem = coop_smem(kGroupedStages);
// eig_jacobi_kernel and eig_final_kernel: no ring
constexpr size_t kTailSmem = coop_smem(0);

// Bounded grid barrier over the first `members` CTAs.  False (and the error
// word set) when the wait ran past limit_ns; the caller then returns.
HT_DEV bool grid_barrier(unsigned *bar, unsigned members, int *err, int *s_ok, uint64_t limit_ns = kWaitLimitNs) {
  __syncthreads();
  if (threadIdx.x == 0) {
    volatile unsigned *gen = bar + 1;
    const unsigned g = *gen;
    __threadfence();
    int ok = 1;
    if (atomicAdd(bar, 1u) == members - 1) {
      atomicExch(bar, 0u);
      __threadfence();
      atomicAdd(bar + 1, 1u);
    } else {
      const uint64_t t0 = global_timer_ns();
      while (*gen == g) {
        __nanosleep(64);
        if (global_timer_ns() - t0 > limit_ns) {
          ok = 0;
          break;
        }
      }
    }
    __threadfence();
    if (!ok) report_error(err, kErrTimeout);
    *s_ok = ok;
  }
  __syncthreads();
  return *s_ok != 0;
}

// G * Y product for the CTA's rows, K split across the 8 warps: warp w takes
// k = 8w .. 8w+7 of every 64-wide chunk, lane l columns l and l + 32, and
// every row (RT >= rows, padded); the G operand is a broadcast shared-memory
// load.  The eight partial blocks are summed in a fixed order at the end.
template <int RT, int NC, int NS>
HT_DEV void coop_product_t(const float *G, const float *Y, int n, int s, int r0, int rows, float *ring, float *Zs) {
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const bool vec = (n % 4 == 0) && ((reinterpret_cast<uintptr_t>(G) | reinterpret_cast<uintptr_t>(Y)) & 15u) == 0;
  const int nchunks = (n + 63) / 64;
  constexpr int STAGE = (RBMAX + SMAX) * CLD;
  auto issue = [&](int c) {
    const int kc = c * 64;
    float *Gd = ring + (c % NS) * STAGE, *Yd = Gd + RBMAX * CLD;
    if (vec) {
      for (int idx = t; idx < RT * 16; idx += 256) {
        const int i = idx >> 4, k4 = (idx & 15) * 4, kk = kc + k4;
        const int bytes = (i < rows && kk < n) ? 4 * min(4, n - kk) : 0;
        const float *g = bytes ? G + static_cast<long long>(r0 + i) * n + kk : G;
        cp_async16(Gd + i * CLD + k4, g, bytes);
      }
      for (int idx = t; idx < 32 * NC * 16; idx += 256) {
        const int j = idx >> 4, k4 = (idx & 15) * 4, kk = kc + k4;
        const int bytes = (j < s && kk < n) ? 4 * min(4, n - kk) : 0;
        const float *y = bytes ? Y + static_cast<long long>(j) * n + kk : Y;
        cp_async16(Yd + j * CLD + k4, y, bytes);
      }
    } else {
      for (int idx = t; idx < RT * 64; idx += 256) {
        const int i = idx >> 6, k = idx & 63, kk = kc + k;
        Gd[i * CLD + k] = (i < rows && kk < n) ? __ldcg(G + static_cast<long long>(r0 + i) * n + kk) : 0.f;
      }
      for (int idx = t; idx < 32 * NC * 64; idx += 256) {
        const int j = idx >> 6, k = idx & 63, kk = kc + k;
        Yd[j * CLD + k] = (j < s && kk < n) ? __ldcg(Y + static_cast<long long>(j) * n + kk) : 0.f;
      }
    }
  };
  float acc[RT][NC];
#pragma unroll
  for (int r = 0; r < RT; ++r)
#pragma unroll
    for (int c = 0; c < NC; ++c) acc[r][c] = 0.f;
  for (int c = 0; c < NS - 1; ++c) {
    if (c < nchunks) issue(c);
    cp_async_commit();
  }
  for (int c = 0; c < nchunks; ++c) {
    if (c + NS - 1 < nchunks) issue(c + NS - 1);
    cp_async_commit();
    cp_async_wait<NS - 1>();
    __syncthreads();
    const float *Gd = ring + (c % NS) * STAGE, *Yd = Gd + RBMAX * CLD;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int kk = 8 * warp + 4 * h;
      float4 y[NC];
#pragma unroll
      for (int q = 0; q < NC; ++q) y[q] = *reinterpret_cast<const float4 *>(Yd + (lane + 32 * q) * CLD + kk);
#pragma unroll
      for (int r = 0; r < RT; ++r) {
        const float4 g = *reinterpret_cast<const float4 *>(Gd + r * CLD + kk);
#pragma unroll
        for (int q = 0; q < NC; ++q)
          acc[r][q] = fmaf(g.x, y[q].x, fmaf(g.y, y[q].y, fmaf(g.z, y[q].z, fmaf(g.w, y[q].w, acc[r][q]))));
      }
    }
    __syncthreads();   // this stage is refilled NS-1 chunks later
  }
  cp_async_wait<0>();
  __syncthreads();
  // partials [warp][row][col] in the (now idle) ring, then a fixed-order sum
  float *red = ring;
#pragma unroll
  for (int r = 0; r < RT; ++r)
#pragma unroll
    for (int q = 0; q < NC; ++q) red[(warp * RT + r) * SMAX + lane + 32 * q] = acc[r][q];
  __syncthreads();
  for (int e = t; e < RBMAX * SMAX; e += 256) {
    const int i = e / SMAX, j = e % SMAX;
    float v = 0.f;
    if (i < rows && j < s) {
#pragma unroll
      for (int w = 0; w < 8; ++w) v += red[(w * RT + i) * SMAX + j];
    }
    Zs[e] = v;
  }
  __syncthreads();
}

template <int NS>
HT_DEV void coop_product(const float *G, const float *Y, int n, int s, int r0, int rows, float *ring, float *Zs) {
  if (s <= 32) {
    if (rows <= 8) coop_product_t<8, 1, NS>(G, Y, n, s, r0, rows, ring, Zs);
    else if (rows <= 16) coop_product_t<16, 1, NS>(G, Y, n, s, r0, rows, ring, Zs);
    else if (rows <= 24) coop_product_t<24, 1, NS>(G, Y, n, s, r0, rows, ring, Zs);
    else coop_product_t<32, 1, NS>(G, Y, n, s, r0, rows, ring, Zs);
  } else if constexpr (SMAX > 32) {
    if (rows <= 8) coop_product_t<8, 2, NS>(G, Y, n, s, r0, rows, ring, Zs);
    else if (rows <= 16) coop_product_t<16, 2, NS>(G, Y, n, s, r0, rows, ring, Zs);
    else if (rows <= 24) coop_product_t<24, 2, NS>(G, Y, n, s, r0, rows, ring, Zs);
    else coop_product_t<32, 2, NS>(G, Y, n, s, r0, rows, ring, Zs);
  }
}

// 1 / sqrt(max(x, 1e-24)) in FP64 from an FP32 seed and two Newton steps
// y <- y (3 - x y^2) / 2 (each squares the relative error): a few FP64
// multiplies instead of the FP64 square-root and division sequences, which
// are long on GB300's narrow FP64 pipe.
HT_DEV double frsqrt_fp64(double x) {
  x = fmax(x, 1e-24);
  double y = static_cast<double>(rsqrtf(static_cast<float>(x)));
  y = y * fma(-0.5 * x, y * y, 1.5);
  y = y * fma(-0.5 * x, y * y, 1.5);
  return y;
}

// Pairs of floats (hi + lo, |lo| <= ulp(hi)/2) as a ~48-bit format: sums by
// Knuth's two-sum, products by the FMA two-product (Dekker's double-float
// arithmetic).  The rounded intrinsics keep the compiler from contracting or
// reordering the error terms.
struct DF {
  float h, l;
};
HT_DEV DF df_two_sum(float a, float b) {
  const float s = __fadd_rn(a, b), bb = __fsub_rn(s, a);
  return DF{s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb))};
}
HT_DEV DF df_quick(float a, float b) {
  const float s = __fadd_rn(a, b);
  return DF{s, __fsub_rn(b, __fsub_rn(s, a))};
}
HT_DEV DF df_add(DF x, DF y) {
  DF s = df_two_sum(x.h, y.h);
  const DF t = df_two_sum(x.l, y.l);
  s = df_quick(s.h, __fadd_rn(s.l, t.h));
  return df_quick(s.h, __fadd_rn(s.l, t.l));
}
HT_DEV DF df_mul(DF x, DF y) {
  const float p = __fmul_rn(x.h, y.h);
  float e = __fmaf_rn(x.h, y.h, -p);
  e = __fmaf_rn(x.h, y.l, __fmaf_rn(x.l, y.h, e));
  return df_quick(p, e);
}
HT_DEV DF df_of(double v) {
  const float h = static_cast<float>(v);
  return DF{h, static_cast<float>(v - static_cast<double>(h))};
}
// 1 / sqrt(x) from the FP32 estimate and one Newton step y + y (1 - x y^2) / 2
// in pair arithmetic (the step squares the estimate's ~2^-23 relative error).
// The pair operations on (y0, 0) and (1, 0) are written out without the zero
// words: this is a long dependent chain.
HT_DEV DF df_rsqrt(DF x) {
  const float y0 = rsqrtf(x.h);
  const float p = __fmul_rn(y0, y0);
  const DF r = df_mul(x, df_quick(p, __fmaf_rn(y0, y0, -p)));   // x y0^2
  DF e = df_two_sum(1.f, -r.h);                                  // 1 - x y0^2
  e = df_quick(e.h, __fadd_rn(e.l, -r.l));
  const DF hlf = DF{__fmul_rn(0.5f, e.h), __fmul_rn(0.5f, e.l)};
  const float q = __fmul_rn(y0, hlf.h);
  const DF m = df_quick(q, __fmaf_rn(y0, hlf.l, __fmaf_rn(y0, hlf.h, -q)));
  const DF y = df_two_sum(y0, m.h);
  return df_quick(y.h, __fadd_rn(y.l, m.l));
}
// 1 / x from the hardware's estimate y (x in the normal range): 1 / x =
// y / (1 - e) with e = 1 - x y below 2^-22, so y (1 + e + e^2) leaves 2^-66, and
// the correction's own rounding is below the pair's last bits.
HT_DEV DF df_rcp(DF x) {
  const float y = approx_rcp(x.h);
  const float e = __fmaf_rn(-x.l, y, __fmaf_rn(-x.h, y, 1.f));
  return df_quick(y, __fmul_rn(y, __fmaf_rn(e, e, e)));
}

// Scaled, shifted Cholesky R^T R of the packed s x s matrix Sd followed by the
// explicit transform T = diag(dsc) R^-1 (row-major, stride SMAX, upper
// triangular, FP32) in Ts, so that applying it is a small matrix product.
// ROOT: the plain form.  Otherwise root-free, L D L^T with R = D^1/2 L^T: a
// pair's reciprocal is a third of the dependent operations of its reciprocal
// root.  The subspace iteration takes the root-free form; the CholeskyQR of tall
// blocks, whose result is rounded to BF16 operands where a last bit decides
// which way an entry goes, keeps the plain one.
//
// On numerically rank-deficient blocks the scaled Gram has pivots far below
// FP32 resolution, and an FP32 factor (or a large shift) would discard the weak
// directions every iteration.  The elimination therefore runs in float-pair
// arithmetic (~48 bits) on the unit-diagonal scaled matrix; GB300 issues FP64
// at a small fraction of the FP32 rate and with long latency, pair arithmetic
// runs on the FP32 pipe.  Shifts are tiny (1e-12; 1e-14 in a second refinement
// pass) and pivots are floored at 1e-24, so T stays finite.  The triangular
// inverse runs in FP32 from the factor: T only has to keep the block well
// conditioned; the span is that of Y for any invertible T.
//
// What bounds it: the serial chain of a step (update the next row, reciprocal
// of its pivot or its root, scale it), which warp 0 runs while warps 1-7 apply
// the current row to the rows behind; one barrier a step.
// Every thread keeps the trailing entries it owns in registers for the whole
// elimination: in shared memory, with the packed indices recomputed each step,
// the update was the longer part.  Cycles a step at s = 64 / 48 / 24: 1490 / 1020
// / 630 before, 840 / 700 / 540 now (root-free); the whole transform 66 / 37 / 15
// us before, 32 / 22 / 10 root-free, 34 / 24 / 12 plain.
// W: SMAX x (SMAX + 1) floats, R32: SMAX x SMAX, 16-byte aligned.
template <bool ROOT>
HT_DEV void factor_transform(const double *Sd, int s, double shift, double *A, double *d, float *R32, float *Ts) {
  __shared__ __align__(16) float2 rowa[2][SMAX];   // the last two finished rows of D L^T, or of R (pairs)
  __shared__ __align__(16) float2 rowl[2][SMAX];   // the same of L^T, or of R
  __shared__ __align__(16) float2 pend[2][SMAX];   // a row updated by all finished rows but the last
  __shared__ float dsc[SMAX], rd[SMAX];            // column scales of the block; the pivots, then D^-1/2 or 1 / R's diagonal
  constexpr int OWN = 224;                          // warps 1-7
  constexpr int EPT = (ESMAX + OWN - 1) / OWN;
  const int t = threadIdx.x;
  for (int j = t; j < s; j += 256) {
    const double v = Sd[j * (j + 1) / 2 + j];
    d[j] = v > 1e-300 ? (v >= 1e-24 ? frsqrt_fp64(v) : 1.0 / sqrt(v)) : 0.0;
    dsc[j] = static_cast<float>(d[j]);
  }
  __syncthreads();
  const int E = s * (s + 1) / 2;
  // entry e of an owner: e < L (L + 1) / 2 are the entries of the trailing L x L
  // block, so that the shrinking block stays spread over all owners
  DF v[EPT];
  unsigned ik[EPT];
#pragma unroll
  for (int q = 0; q < EPT; ++q) {
    const int e = t - 32 + OWN * q;
    ik[q] = 0u;
    v[q] = DF{0.f, 0.f};
    if (t >= 32 && e < E) {
      int a, b;
      tri_index(e, a, b);
      const int i = s - 1 - b, k = s - 1 - a;
      ik[q] = static_cast<unsigned>(i | (k << 8));
      double x = Sd[k * (k + 1) / 2 + i] * d[i] * d[k];
      if (i == k) x = (d[k] > 0.0 ? 1.0 : 0.0) + shift;
      v[q] = df_of(x);
      if (i == 0) rowa[1][k] = make_float2(v[q].h, v[q].l);
      if (i == 1) pend[0][k] = make_float2(v[q].h, v[q].l);
    }
  }
  __syncthreads();
  // row j1 (its entries k = j1 + t, j1 + t + 32 in x, its pivot in piv), and the
  // same divided by the pivot, into rowa / rowl [j1 & 1] and R32
  auto finish_row = [&](int j1, DF piv, const DF (&x)[2]) {
    if (!(piv.h >= 1e-24f)) piv = DF{1e-24f, 0.f};
    const DF ri = ROOT ? df_rsqrt(piv) : df_rcp(piv);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int k = j1 + t + 32 * q;
      if (q == 1 && j1 + 32 >= s) break;
      if (k < s) {
        const DF l = df_mul(k == j1 ? piv : x[q], ri);
        rowl[j1 & 1][k] = make_float2(l.h, l.l);
        rowa[j1 & 1][k] = ROOT ? make_float2(l.h, l.l) : make_float2(x[q].h, x[q].l);
        R32[j1 * SMAX + k] = l.h;
      }
    }
    if (!ROOT && t == 0) rd[j1] = piv.h;
  };
  auto pair_at = [](const float2 &p) { return DF{p.x, p.y}; };
  if (t < 32) {
    DF x[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) x[q] = t + 32 * q < s ? pair_at(rowa[1][t + 32 * q]) : DF{0.f, 0.f};
    const DF piv = pair_at(rowa[1][0]);
    __syncwarp();
    finish_row(0, piv, x);
  }
  __syncthreads();
  for (int j = 0; j + 1 < s; ++j) {
    const int j1 = j + 1;
    const float2 *ra = rowa[j & 1], *rl = rowl[j & 1];
    if (t < 32) {
      const float2 *pd = pend[j & 1];
      const DF lj = pair_at(rl[j1]);
      auto updated = [&](int k) {
        const DF p = df_mul(lj, pair_at(ra[k]));
        return df_add(pair_at(pd[k]), DF{-p.h, -p.l});
      };
      DF x[2] = {updated(min(j1 + t, s - 1)), DF{0.f, 0.f}};
      if (j1 + 32 < s) x[1] = updated(min(j1 + t + 32, s - 1));
      const DF piv{__shfl_sync(0xffffffffu, x[0].h, 0), __shfl_sync(0xffffffffu, x[0].l, 0)};
      finish_row(j1, piv, x);
    } else {
      // entries with i >= j + 2 live; dead ones are carried along unused, so that
      // two entries at a time run without a branch between them
      const int nq = ((s - 2 - j) * (s - 1 - j) / 2 + OWN - 1) / OWN;
#pragma unroll
      for (int q0 = 0; q0 < EPT; q0 += 2) {
        if (q0 >= nq) break;
#pragma unroll
        for (int q = q0; q < q0 + 2 && q < EPT; ++q) {
          const DF p = df_mul(pair_at(rl[ik[q] & 255]), pair_at(ra[ik[q] >> 8]));
          v[q] = df_add(v[q], DF{-p.h, -p.l});
        }
#pragma unroll
        for (int q = q0; q < q0 + 2 && q < EPT; ++q)
          if (static_cast<int>(ik[q] & 255) == j + 2) pend[j1 & 1][ik[q] >> 8] = make_float2(v[q].h, v[q].l);
      }
    }
    __syncthreads();
  }
  // W = R^-1 in 32 x 32 blocks, R = [R11 R12; 0 R22] (L^T, unit diagonal, when root-free):
  //   W11 = R11^-1, W22 = R22^-1  (warp 0 / warp 1: lane = column, back substitution
  //                                 with the column in registers, R rows broadcast)
  //   W12 = -W11 (R12 W22)        (two 32 x 32 products over all threads)
  // then T = diag(dsc) W (D^-1/2).
  constexpr int WS = SMAX + 1;
  float *W = reinterpret_cast<float *>(A);
  const int n1 = s < 32 ? s : 32, n2 = s - n1;
  if (t < s) rd[t] = ROOT ? 1.f / R32[t * SMAX + t] : 1.f / sqrtf(rd[t]);
  for (int e = t; e < SMAX * WS; e += 256) W[e] = 0.f;
  __syncthreads();
  if (t < 64) {
    const int w = t >> 5, lane = t & 31, base = 32 * w, nb = w == 0 ? n1 : n2;
    if (lane < nb) {
      // (rows of R are fetched one row ahead of the sums' dependent chain)
      float wv[32], r[2][32];
      auto fetch = [&](int ii, float (&d)[32]) {
#pragma unroll
        for (int j4 = (ii + 1) & ~3; j4 < 32; j4 += 4) {
          const float4 f = *reinterpret_cast<const float4 *>(R32 + (base + ii) * SMAX + base + j4);
          d[j4] = f.x; d[j4 + 1] = f.y; d[j4 + 2] = f.z; d[j4 + 3] = f.w;
        }
      };
      fetch(30, r[1]);
      auto scaled = [&](int ii, float a) { return ROOT ? (ii <= lane ? a * rd[base + (ii < nb ? ii : 0)] : 0.f) : a; };
      wv[31] = scaled(31, lane == 31 ? 1.f : 0.f);
#pragma unroll
      for (int ii = 30; ii >= 0; --ii) {
        if (ii > 0) fetch(ii - 1, r[(ii & 1)]);   // row ii is in r[ii & 1 ^ 1]
        float acc = ii == lane ? 1.f : 0.f;
#pragma unroll
        for (int jj = ii + 1; jj < 32; ++jj) acc = jj <= lane ? fmaf(-r[(ii & 1) ^ 1][jj], wv[jj], acc) : acc;
        wv[ii] = scaled(ii, acc);
      }
#pragma unroll
      for (int ii = 0; ii < 32; ++ii)
        if (ii <= lane) W[(base + ii) * WS + base + lane] = wv[ii];
    }
  }
  __syncthreads();
  if (SMAX > 32 && n2 > 0) {
    // P = R12 W22 (n1 x n2) in Ts (written last), then W12 = -W11 P: thread
    // (lane k, warp w) forms rows w + 8 q of column k, the sums in the order
    // of the columns (entries past a triangle's edge are zero)
    float *Pm = Ts;
    const int k = t & 31, w = t >> 5;
    float o[4] = {0.f, 0.f, 0.f, 0.f};
    for (int j = 0; j < n2; ++j) {
      const float x = W[(32 + j) * WS + 32 + k];
#pragma unroll
      for (int q = 0; q < 4; ++q) o[q] = fmaf(R32[(w + 8 * q) * SMAX + 32 + j], x, o[q]);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) Pm[(w + 8 * q) * SMAX + k] = o[q];
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; ++q) o[q] = 0.f;
    for (int j = 0; j < 32; ++j) {
      const float x = Pm[j * SMAX + k];
#pragma unroll
      for (int q = 0; q < 4; ++q) o[q] = fmaf(W[(w + 8 * q) * WS + j], x, o[q]);
    }
    if (k < n2) {
#pragma unroll
      for (int q = 0; q < 4; ++q) W[(w + 8 * q) * WS + 32 + k] = -o[q];
    }
    __syncthreads();
  }
#pragma unroll
  for (int q = 0; q < SMAX * SMAX / 256; ++q) {
    const int e = t + 256 * q, i = e / SMAX, k = e % SMAX;
    Ts[e] = (i < s && k < s && k >= i) ? W[i * WS + k] * (ROOT ? dsc[i] : dsc[i] * rd[k]) : 0.f;
  }
  __syncthreads();
}

// X (RBMAX x SMAX rows) <- X T for the upper-triangular T (s x s): thread
// (row t / 8, columns t % 8 + 8 b) forms its SMAX / 8 outputs, then writes back.
HT_DEV void coop_apply(float *X, const float *Ts, int s) {
  const int t = threadIdx.x, r = t >> 3, cb = t & 7;
  constexpr int NB = SMAX / 8;
  float o[NB];
#pragma unroll
  for (int b = 0; b < NB; ++b) o[b] = 0.f;
  for (int j = 0; j < s; ++j) {
    const float x = X[r * SMAX + j];
#pragma unroll
    for (int b = 0; b < NB; ++b) o[b] = fmaf(x, Ts[j * SMAX + cb + 8 * b], o[b]);
  }
  __syncthreads();
#pragma unroll
  for (int b = 0; b < NB; ++b) X[r * SMAX + cb + 8 * b] = (cb + 8 * b < s) ? o[b] : 0.f;
  __syncthreads();
}

// Rows [r0, r0 + rows) of an n x s block into X[i * SMAX + j] (zero padded).
HT_DEV void coop_load_rows(const float *src, int n, int s, int r0, int rows, float *X) {
  for (int e = threadIdx.x; e < RBMAX * SMAX; e += 256) {
    const int i = e % RBMAX, j = e / RBMAX;
    X[i * SMAX + j] = (i < rows && j < s) ? __ldcg(src + (r0 + i) + static_cast<long long>(n) * j) : 0.f;
  }
}

HT_DEV void coop_store_rows(const float *X, int n, int s, int r0, int rows, float *dst) {
  for (int e = threadIdx.x; e < RBMAX * SMAX; e += 256) {
    const int i = e % RBMAX, j = e / RBMAX;
    if (i < rows && j < s) dst[(r0 + i) + static_cast<long long>(n) * j] = X[i * SMAX + j];
  }
}

// acc[q] += partial of entry e = t + 256 q (packed upper triangle, i <= j) of L^T R.
HT_DEV void coop_gram_partial(const float *L, const float *R, int s, Acc2 (&acc)[kMaxEntPerThread]) {
  const int E = s * (s + 1) / 2;
#pragma unroll
  for (int q = 0; q < kMaxEntPerThread; ++q) {
    const int e = threadIdx.x + 256 * q;
    if (e < E) {
      int i, j;
      tri_index(e, i, j);
#pragma unroll 8
      for (int r = 0; r < RBMAX; ++r) acc2_add_prod(acc[q], L[r * SMAX + i], R[r * SMAX + j]);
    }
  }
}

HT_DEV void coop_gram_store(const Acc2 (&acc)[kMaxEntPerThread], int s, float *part) {
  const int E = s * (s + 1) / 2;
#pragma unroll
  for (int q = 0; q < kMaxEntPerThread; ++q) {
    const int e = threadIdx.x + 256 * q;
    if (e < E) {
      part[2 * e] = acc[q].s;
      part[2 * e + 1] = acc[q].c;
    }
  }
}

// Every synchronising CTA sums a slice of all problems' entries over the
// problem's CTA partials, in CTA order.
HT_DEV void coop_reduce(const CoopBatch &B) {
  for (int g = blockIdx.x * 256 + threadIdx.x; g < B.ent_total; g += B.nsync * 256) {
    int p = 0;
    while (g >= B.ent_off[p + 1]) ++p;
    const CoopProb &P = B.p[p];
    const int e = g - B.ent_off[p];
    Acc2 acc = {0.f, 0.f};
    for (int c0 = 0; c0 < P.ncta; c0 += GROUP) {
      float hi[GROUP], lo[GROUP];
#pragma unroll
      for (int q = 0; q < GROUP; ++q) {
        const bool ok = c0 + q < P.ncta;
        const float *src = P.part + (static_cast<long long>(c0 + q) * ESMAX + e) * 2;
        hi[q] = ok ? __ldcg(src) : 0.f;
        lo[q] = ok ? __ldcg(src + 1) : 0.f;
      }
#pragma unroll
      for (int q = 0; q < GROUP; ++q) acc2_add(acc, hi[q], lo[q]);
    }
    P.S[e] = static_cast<double>(acc.s) + static_cast<double>(acc.c);
  }
}

HT_DEV void coop_load_S(const CoopProb &P, double *Sd) {
  const int E = P.s * (P.s + 1) / 2;
  for (int e = threadIdx.x; e < E; e += 256) Sd[e] = __ldcg(P.S + e);
  __syncthreads();
}

// One CholeskyQR-type step over the CTA's rows: X = src rows (optionally
// G * src + mu src), apply the current transform Rs (unless identity), store to dst,
// accumulate the Gram partial.  mode 0: ITER, 1: APPLY, 2: RR (also Q rows).
template <int NS>
HT_DEV void coop_step(const CoopProb &P, int cl, int mode, const float *src, float *dst, float *dst2, bool ident,
                      float mu, const float *Rs, float *Zs, float *Qr, float *ring, bool want_s = true) {
  Acc2 acc[kMaxEntPerThread];
#pragma unroll
  for (int q = 0; q < kMaxEntPerThread; ++q) acc[q] = Acc2{0.f, 0.f};
  const int rb = cl * P.rows, re = min(P.n, rb + P.rows);
  for (int r0 = rb; r0 < re; r0 += RBMAX) {
    const int rows = min(RBMAX, re - r0);
    coop_load_rows(src, P.n, P.s, r0, rows, Qr);
    if (mode != 1) {
      coop_product<NS>(P.G, src, P.n, P.s, r0, rows, ring, Zs);
      if (mode == 0)
        for (int e = threadIdx.x; e < RBMAX * SMAX; e += 256) Zs[e] = fmaf(mu, Qr[e], Zs[e]);
    } else {
      __syncthreads();
      for (int e = threadIdx.x; e < RBMAX * SMAX; e += 256) Zs[e] = Qr[e];
    }
    __syncthreads();
    if (!ident) {
      coop_apply(Zs, Rs, P.s);
      if (mode == 2) coop_apply(Qr, Rs, P.s);
    }
    if (mode == 2) {
      coop_store_rows(Qr, P.n, P.s, r0, rows, dst);
      coop_store_rows(Zs, P.n, P.s, r0, rows, dst2);
      coop_gram_partial(Qr, Zs, P.s, acc);
    } else {
      coop_store_rows(Zs, P.n, P.s, r0, rows, dst);
      if (want_s) coop_gram_partial(Zs, Zs, P.s, acc);
    }
    __syncthreads();
  }
  if (want_s) coop_gram_store(acc, P.s, P.part + static_cast<long long>(cl) * ESMAX * 2);
}

// U = Q V[:, :K], GU = Y V[:, :K] on the CTA's rows, column sums of squares of
// GU - theta U into colss[cl].
HT_DEV void coop_final_rows(const CoopProb &P, int cl, int rows_per, const float *Q, const float *Y, float (*Vsm)[SMAX + 1],
                            const float *th, float *Qr, float *Zs) {
  const int t = threadIdx.x, n = P.n, s = P.s, K = P.K;
  __shared__ float colsum[SMAX];
  if (t < SMAX) colsum[t] = 0.f;
  const int rb = cl * rows_per, re = min(n, rb + rows_per);
  for (int r0 = rb; r0 < re; r0 += RBMAX) {
    const int rows = min(RBMAX, re - r0);
    coop_load_rows(Q, n, s, r0, rows, Qr);
    coop_load_rows(Y, n, s, r0, rows, Zs);
    __syncthreads();
    // thread: row i = t / 8 (32 rows), columns j = t % 8 + 8 c
    const int i = t >> 3, jb = t & 7;
    float dsq[SMAX / 8];
#pragma unroll
    for (int c = 0; c < SMAX / 8; ++c) {
      const int j = jb + 8 * c;
      float u = 0.f, gu = 0.f;
      if (j < K && i < rows) {
        for (int k = 0; k < s; ++k) {
          u = fmaf(Qr[i * SMAX + k], Vsm[k][j], u);
          gu = fmaf(Zs[i * SMAX + k], Vsm[k][j], gu);
        }
        P.U[(r0 + i) + static_cast<long long>(n) * j] = u;
        P.GU[(r0 + i) + static_cast<long long>(n) * j] = gu;
      }
      const float d = (j < K && i < rows) ? gu - th[j] * u : 0.f;
      dsq[c] = d * d;
    }
    __syncthreads();
    // column sums over the 32 rows: reuse Qr as scratch [row][col]
#pragma unroll
    for (int c = 0; c < SMAX / 8; ++c) Qr[i * SMAX + jb + 8 * c] = dsq[c];
    __syncthreads();
    if (t < SMAX) {
      float a = 0.f;
      for (int r = 0; r < RBMAX; ++r) a += Qr[r * SMAX + t];
      colsum[t] += a;
    }
    __syncthreads();
  }
  if (t < SMAX) P.colss[static_cast<long long>(cl) * SMAX + t] = colsum[t];
}

// Shared memory of the eigen-solver kernels: the dynamic block (kCoopSmem)
// carved as the cooperative kernel always has, plus small static arrays.
struct EigSmem {
  float *Rs;                    // SMAX*SMAX (upper factor, row-major)
  float *Zs, *Qr;               // RBMAX*SMAX each
  float *ring;                  // product ring, or (aliased) the reducer / Jacobi scratch
  double *Sd;
  float (*A)[SMAX + 1], (*VV)[SMAX + 1], (*A2)[SMAX + 1];
  int *s_ok, *order;
  float *red, *th_sm;
  double *piv64;
};

HT_DEV EigSmem eig_smem(float *sm) {
  __shared__ int s_ok;
  __shared__ int order[SMAX];
  __shared__ float red[256];
  __shared__ float th_sm[SMAX];
  __shared__ double piv64[SMAX];
  EigSmem m;
  m.Rs = sm;
  m.Zs = m.Rs + SMAX * SMAX + SMAX;   // SMAX floats after the factor are reserved
  m.Qr = m.Zs + RBMAX * SMAX;
  m.ring = m.Qr + RBMAX * SMAX;
  m.Sd = reinterpret_cast<double *>(m.ring);
  m.A = reinterpret_cast<float (*)[SMAX + 1]>(m.ring + 2 * ESMAX);
  m.VV = reinterpret_cast<float (*)[SMAX + 1]>(m.ring + 2 * ESMAX + kJacMat);
  m.A2 = reinterpret_cast<float (*)[SMAX + 1]>(m.ring + 2 * ESMAX + 2 * kJacMat);
  m.s_ok = &s_ok;
  m.order = order;
  m.red = red;
  m.th_sm = th_sm;
  m.piv64 = piv64;
  return m;
}

// Direct problem (s == n): Jacobi eigen-decomposition of G itself.
template <int NT>
HT_DEV void eig_direct(const CoopProb &P, const EigSmem &m) {
  const int t = threadIdx.x, n = P.n, K = P.K;
  float (*A)[SMAX + 1] = m.A;
  float (*VV)[SMAX + 1] = m.VV;
  const int *order = m.order;
  for (int e = t; e < SMAX * SMAX; e += NT) {
    const int i = e % SMAX, j = e / SMAX;
    A[i][j] = (i < n && j < n) ? P.G[i + static_cast<long long>(n) * j] : 0.f;
  }
  __syncthreads();
  jacobi_smem<NT>(A, m.A2, VV, n, m.order);
  for (int r = t; r < K; r += NT) P.theta[r] = A[order[r]][order[r]];
  // U = V[:, order[:K]], GU = G U, residual
  for (int e = t; e < n * K; e += NT) {
    const int i = e % n, j = e / n;
    float gu = 0.f;
    for (int k = 0; k < n; ++k) gu = fmaf(P.G[i + static_cast<long long>(n) * k], VV[k][order[j]], gu);
    const float u = VV[i][order[j]];
    P.U[i + static_cast<long long>(n) * j] = u;
    P.GU[i + static_cast<long long>(n) * j] = gu;
    const float d = gu - A[order[j]][order[j]] * u;
    m.Zs[e] = d * d;   // n * K <= 64 * 64 fits Zs + Qr (contiguous)
  }
  __syncthreads();
  if (t == 0) {
    float mx = 0.f;
    for (int j = 0; j < K; ++j) {
      float a = 0.f;
      for (int i = 0; i < n; ++i) a += m.Zs[i + n * j];
      mx = fmaxf(mx, sqrtf(a));
    }
    const float th = A[order[0]][order[0]];
    P.resid[0] = th > 0.f ? mx / th : mx;
  }
}

// Synchronisation of the phases of one problem.  Cooperative: the problem's
// rows are spread over several CTAs of a cooperative grid -- bounded grid
// barriers, and the Gram partials reduced by all CTAs of the grid.  Local:
// the problem is one CTA's (the grouped solver) -- block barriers, and the
// CTA reduces its own partials.
struct CoopSync {
  static constexpr bool kTail = false;
  const CoopBatch *B;
  unsigned members;
  int *s_ok;
  HT_DEV bool bar() const { return grid_barrier(B->bar, members, B->err, s_ok); }
  HT_DEV void reduce() const { coop_reduce(*B); }
};

HT_DEV void coop_reduce_one(const CoopProb &P) {
  const int E = P.s * (P.s + 1) / 2;
  for (int e = threadIdx.x; e < E; e += 256) {
    Acc2 acc = {0.f, 0.f};
    for (int c = 0; c < P.ncta; ++c) {
      const float *src = P.part + (static_cast<long long>(c) * ESMAX + e) * 2;
      acc2_add(acc, __ldcg(src), __ldcg(src + 1));
    }
    P.S[e] = static_cast<double>(acc.s) + static_cast<double>(acc.c);
  }
}

struct LocalSync {
  static constexpr bool kTail = true;
  const CoopProb *P;
  HT_DEV bool bar() const {
    __syncthreads();
    return true;
  }
  HT_DEV void reduce() const { coop_reduce_one(*P); }
};

// Rayleigh-Ritz: H from P.S, its eigenvectors by descending eigenvalue into P.V
// and the leading K eigenvalues into P.theta.
template <int NT>
HT_DEV void ritz(const CoopProb &P, const EigSmem &m) {
  const int t = threadIdx.x, s = P.s;
  for (int e = t; e < s * s; e += NT) {
    const int i = e % s, j = e / s;
    m.A[i][j] = static_cast<float>(__ldcg(P.S + (i <= j ? j * (j + 1) / 2 + i : i * (i + 1) / 2 + j)));
  }
  __syncthreads();
  jacobi_smem<NT>(m.A, m.A2, m.VV, s, m.order);
  for (int e = t; e < s * s; e += NT) {
    const int i = e % s, r = e / s;
    P.V[i + s * r] = m.VV[i][m.order[r]];
  }
  for (int r = t; r < P.K; r += NT) P.theta[r] = m.A[m.order[r]][m.order[r]];
}

// P.V (s x s) into shared memory
template <int NT>
HT_DEV void load_ritz(const CoopProb &P, float (*Vsm)[SMAX + 1]) {
  for (int e = threadIdx.x; e < P.s * P.s; e += NT) Vsm[e % P.s][e / P.s] = __ldcg(P.V + e);
}

// max_j ||G u_j - theta_j u_j|| / theta_1 from the row blocks' column sums
HT_DEV void final_residual(const CoopProb &P, int nblk) {
  __shared__ float nrm[SMAX];
  const int t = threadIdx.x;
  if (t < SMAX) {
    float a = 0.f;
    if (t < P.K)
      for (int c = 0; c < nblk; ++c) a += __ldcg(P.colss + static_cast<long long>(c) * SMAX + t);
    nrm[t] = sqrtf(a);
  }
  __syncthreads();
  if (t == 0) {
    float mx = 0.f;
    for (int j = 0; j < P.K; ++j) mx = fmaxf(mx, nrm[j]);
    const float th = __ldcg(P.theta);
    P.resid[0] = th > 0.f ? mx / th : mx;
  }
}

// Subspace iteration, Rayleigh-Ritz and the final U / GU / residual of one
// problem; CTA `cl` of the problem's P.ncta owns rows [cl * P.rows, ...).
template <class Sync, int NS>
HT_DEV void eig_iterate(const CoopProb &P, int cl, const Sync &sy, int iters, int refine, const EigSmem &m) {
  const int t = threadIdx.x;
  float *Rs = m.Rs, *Zs = m.Zs, *Qr = m.Qr, *ring = m.ring, *red = m.red;
  double *Sd = m.Sd;
  // mu = 1e-9 trace(G), computed identically by every CTA of the problem
  {
    float tr = 0.f;
    for (int i = t; i < P.n; i += 256) tr += __ldg(P.G + i + static_cast<long long>(P.n) * i);
    red[t] = tr;
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
      if (t < w) red[t] += red[t + w];
      __syncthreads();
    }
  }
  const float mu = 1e-9f * fmaxf(red[0], 0.f);
  // start block rows
  {
    const int rb = cl * P.rows, re = min(P.n, rb + P.rows);
    for (int e = t; e < (re - rb) * P.s; e += 256) {
      const int i = rb + e % (re - rb), j = e / (re - rb);
      const long long idx = i + static_cast<long long>(P.n) * j;
      P.buf[0][idx] = P.start ? P.start[idx] : gaussian(P.seed, P.stream_id, static_cast<unsigned long long>(idx));
    }
  }
  if (!sy.bar()) return;

  auto reduce_and_factor = [&](double shift) -> bool {
    if (!sy.bar()) return false;
    sy.reduce();
    if (!sy.bar()) return false;
    coop_load_S(P, Sd);
    double *A64 = Sd + ESMAX;                  // SMAX*SMAX doubles after the reduced Gram
    factor_transform<false>(Sd, P.s, shift, A64, m.piv64, reinterpret_cast<float *>(A64 + SMAX * SMAX), Rs);
    return true;
  };

  int cur = 0;
  bool ident = true;
  for (int it = 0; it < iters; ++it) {
    coop_step<NS>(P, cl, 0, P.buf[cur], P.buf[cur ^ 1], nullptr, ident, mu, Rs, Zs, Qr, ring);
    if (!reduce_and_factor(1e-12)) return;
    ident = false;
    cur ^= 1;
  }
  // Q_L = Y_L T_L -> buffer 2.  The float-pair factor leaves Q_L orthonormal
  // to ~1e-7 (scaled off-diagonal of Q_L^T Q_L, 1e-6 on clustered spectra), so
  // Rayleigh-Ritz takes it as it is: no further CholeskyQR pass.  G Q is formed
  // from Q_L itself, not as (G Y_L) T_L, whose sum over the ill-scaled columns of
  // Y_L loses digits to cancellation.
  // The FP32 path asks for `refine` CholeskyQR passes on Q_L all the same
  // (orthonormal to FP32 rounding, the last digit of its error).
  coop_step<NS>(P, cl, 1, P.buf[cur], P.buf[2], nullptr, ident, 0.f, Rs, Zs, Qr, ring, ident || refine > 0);
  bool rr_ident = true;
  if (ident || refine > 0) {   // ident: no iteration ran, orthonormalise the start block
    if (!reduce_and_factor(1e-12)) return;
    rr_ident = false;
    for (int r = 1; r < refine; ++r) {   // row-local, so in place
      coop_step<NS>(P, cl, 1, P.buf[2], P.buf[2], nullptr, false, 0.f, Rs, Zs, Qr, ring);
      if (!reduce_and_factor(1e-14)) return;
    }
  } else if (!sy.bar()) {
    return;
  }
  // Rayleigh-Ritz: Q -> buf3, G Q -> buf0, H = Q^T G Q
  coop_step<NS>(P, cl, 2, P.buf[2], P.buf[3], P.buf[0], rr_ident, 0.f, Rs, Zs, Qr, ring);
  if (!sy.bar()) return;
  sy.reduce();
  if (!Sync::kTail) return;   // cooperative: eig_jacobi_kernel and eig_final_kernel go on from P.S
  if (!sy.bar()) return;
  ritz<256>(P, m);
  __syncthreads();
  // final: U, GU and the residual
  for (int j = t; j < SMAX; j += 256) m.th_sm[j] = j < P.K ? m.A[m.order[j]][m.order[j]] : 0.f;
  load_ritz<256>(P, m.VV);
  __syncthreads();
  coop_final_rows(P, 0, P.n, P.buf[3], P.buf[0], m.VV, m.th_sm, Qr, Zs);
  __syncthreads();
  final_residual(P, 1);
}

#if HT_EIG_SMAX == 64
__global__ void __launch_bounds__(256, 1) eig_coop_kernel(const __grid_constant__ CoopBatch B) {
  extern __shared__ __align__(16) float sm[];
  const EigSmem m = eig_smem(sm);

  if (static_cast<int>(blockIdx.x) >= B.nsync) {   // past the barrier's members: a direct problem (eig_batched)
    eig_direct<256>(B.p[B.beside[blockIdx.x - B.nsync]], m);
    return;
  }
  int pi = 0;
  while (!(static_cast<int>(blockIdx.x) >= B.p[pi].cta0 && static_cast<int>(blockIdx.x) < B.p[pi].cta0 + B.p[pi].ncta)) ++pi;
  const CoopProb &P = B.p[pi];
  const int cl = blockIdx.x - P.cta0;
  const unsigned members = static_cast<unsigned>(B.nsync);

  if (B.orth_passes > 0) {
    // In-place CholeskyQR of buffer 0 (problems without a Gram): each pass
    // applies the previous transform to the CTA's rows and accumulates their
    // Gram partial, all CTAs reduce, every CTA factors (float pairs, pivots
    // floored, so it cannot break down; the first pass shifted by 1e-12 of the
    // unit diagonal, as the eigen-solver's iterations).  The Gram and the
    // factor carry ~48 bits, so after one pass only the FP32 rounding of the
    // applied transform remains (~u * cond(Y)); a second pass removes it.
    float *Q = P.buf[0];
    double *A64 = m.Sd + ESMAX;
    for (int pass = 0; pass <= B.orth_passes; ++pass) {
      // row-local: in place; the last pass only applies the transform
      coop_step<CNS>(P, cl, 1, Q, Q, nullptr, pass == 0, 0.f, m.Rs, m.Zs, m.Qr, m.ring, pass < B.orth_passes);
      if (pass == B.orth_passes) break;
      if (!grid_barrier(B.bar, members, B.err, m.s_ok)) return;
      coop_reduce(B);
      if (!grid_barrier(B.bar, members, B.err, m.s_ok)) return;
      coop_load_S(P, m.Sd);
      factor_transform<true>(m.Sd, P.s, pass == 0 ? 1e-12 : 0.0, A64, m.piv64, reinterpret_cast<float *>(A64 + SMAX * SMAX),
                       m.Rs);
    }
    return;
  }
  const CoopSync sy{&B, members, m.s_ok};
  eig_iterate<CoopSync, CNS>(P, cl, sy, B.iters, B.refine, m);
}

// The Jacobi step, a CTA per problem: Rayleigh-Ritz of the iterated ones, the
// whole eigen-decomposition of the direct ones (s == n) that the cooperative
// kernel did not take.  A kernel of
// its own so that a round has 32 warps; inside the cooperative kernel, at 8
// warps, the same step took 172 us on the 48 x 48 matrices of a rank-32
// decomposition; here 142.
__global__ void __launch_bounds__(kJacThreads) eig_jacobi_kernel(const __grid_constant__ CoopBatch B) {
  extern __shared__ __align__(16) float sm[];
  const EigSmem m = eig_smem(sm);
  const CoopProb &P = B.p[B.jacobi[blockIdx.x]];
  if (P.s == P.n) eig_direct<kJacThreads>(P, m);
  else ritz<kJacThreads>(P, m);
}

// U = Q V, GU = (G Q) V and the residual of the iterated problems: a CTA per
// block of B.p[i].frows rows; the last one of a problem to finish sums the
// residual's parts (in block order).
__global__ void __launch_bounds__(256) eig_final_kernel(const __grid_constant__ CoopBatch B) {
  extern __shared__ __align__(16) float sm[];
  const EigSmem m = eig_smem(sm);
  int pi = 0;
  while (!(static_cast<int>(blockIdx.x) >= B.p[pi].fcta0 && static_cast<int>(blockIdx.x) < B.p[pi].fcta0 + B.p[pi].fncta)) ++pi;
  const CoopProb &P = B.p[pi];
  for (int j = threadIdx.x; j < SMAX; j += 256) m.th_sm[j] = j < P.K ? __ldcg(P.theta + j) : 0.f;
  load_ritz<256>(P, m.VV);
  __syncthreads();
  coop_final_rows(P, blockIdx.x - P.fcta0, P.frows, P.buf[3], P.buf[0], m.VV, m.th_sm, m.Qr, m.Zs);
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) *m.s_ok = atomicAdd(B.bar + 4 + pi, 1u) == static_cast<unsigned>(P.fncta) - 1u;
  __syncthreads();
  if (*m.s_ok) {
    __threadfence();
    final_residual(P, P.fncta);
  }
}
#endif

// Grouped solver of the batched path: CTA b solves problem tab[b] alone (all
// of its rows, block barriers only), so one ordinary launch covers every leaf
// of every tensor of a batch and no CTA waits on another.
__global__ void __launch_bounds__(256, SMAX > 32 ? 2 : 4) eig_grouped_kernel(const CoopProb *__restrict__ tab, int iters, int refine) {
  extern __shared__ __align__(16) float sm[];
  const EigSmem m = eig_smem(sm);
  __shared__ CoopProb sP;
  if (threadIdx.x == 0) sP = tab[blockIdx.x];
  __syncthreads();
  const CoopProb &P = sP;
  if (P.s == P.n) {
    eig_direct<256>(P, m);
    return;
  }
  const LocalSync sy{&P};
  eig_iterate<LocalSync, kGroupedStages>(P, 0, sy, iters, refine, m);
}

}  // namespace HT_EIG_NS
