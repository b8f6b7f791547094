// Complex128 dense linear algebra of one problem by a team: one CTA of
// kDLThreads threads, or a cluster of up to 8 of them that share the problem
// through global memory (interface and cascade kernels): a tiled GEMM update,
// LU with partial pivoting and the triangular solves that go with it.  Matrices
// are row-major in global memory (leading dimension `ld`).  These replace the
// zgemm / zgesv calls that numpy makes for the reference (np.matrix products
// and np.linalg.solve in backend/stack.py and backend/mode_calcs.py).
// How a team splits the work never changes an entry's arithmetic, so results
// do not depend on its size.
#pragma once
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "emu_cplx.cuh"

namespace emu {

constexpr int kDLThreads = 256;
constexpr int kTM = 64, kTN = 64, kTK = 8;   // GEMM tile
constexpr int kNB = 32;                      // LU / TRSM block

// Shared tiles of cta_gemm_tile.  A: 64 rows x 8 complex columns stored as
// (re, im) pairs; B: 8 complex rows x 64 complex columns stored as the real
// 16 x 128 matrix [[Re, Im], [-Im, Re]] per element, so that the complex
// product is one real product A_r (m x 2k) * B_r (2k x 2n) whose result,
// read in (re, im) pairs, is the complex C.  Row paddings (+4 doubles) make
// the tensor-core fragment reads free of bank conflicts.
constexpr int kAS = 2 * kTK + 4, kBS = 2 * kTN + 4;
struct GemmSmem {
  double As[kTM][kAS];
  double Bs[2 * kTK][kBS];
};

__device__ __forceinline__ cd ldc(const cd *p) { return *p; }

// D = A B + D on the FP64 tensor cores: one 8 x 8 x 4 product per warp
// (PTX mma.sync m8n8k4 f64; lane l holds A[l/4][l%4], B[l%4][l/4] and
// D[l/4][2(l%4) + {0,1}]).
__device__ __forceinline__ void dmma_884(double &d0, double &d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

// The CTAs of one problem.  `sync` orders their global memory too.
struct Team {
  int rank, size;
  __device__ __forceinline__ void sync() const {
    if (size > 1) cooperative_groups::this_cluster().sync();
    else __syncthreads();
  }
  // elementwise loops over the team's threads
  __device__ __forceinline__ int tid() const { return rank * kDLThreads + (int)threadIdx.x; }
  __device__ __forceinline__ int nt() const { return size * kDLThreads; }
  // columns dealt to the CTAs in groups of 8 (128 bytes of a row), so that a few
  // columns still spread over all of them
  __device__ __forceinline__ int col() const {
    return ((((int)threadIdx.x >> 3) * size + rank) << 3) + ((int)threadIdx.x & 7);
  }
};

__device__ __forceinline__ Team cluster_team() {
  namespace cg = cooperative_groups;
  return Team{(int)cg::this_cluster().block_rank(), (int)cg::this_cluster().num_blocks()};
}

// One T x T tile (T = 64 or 32) of a product on the FP64 tensor cores: `fa(r, k)` gives
// A's value at the tile's row r, `fb(k, c)` B's at its column c (both called for k
// below the depth only), `put(r, c, v)` takes the results.  All kDLThreads threads of the
// CTA must call it.  8 warps in a 2 x 4 grid, each owning a T/2 x T/2 block of the real
// T x 2T result in fragments of 8 x 8.  FOLD: the accumulators are folded into a
// running sum every 1 024 values of k, for depths beyond a few thousand.
template <int T, bool FOLD, class FA, class FB, class Put>
static __device__ __forceinline__ void cta_tile(int k, FA &&fa, FB &&fb, Put &&put, GemmSmem &sm) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int wm = warp >> 2, wn = warp & 3;
  constexpr int F = T / 16;        // 8 x 8 fragments of a warp's T/2 x T/2 block, per side
  constexpr int H = T / 32;        // elements of each operand per thread and k-tile
  double acc[F][F][2], sum[FOLD ? F : 1][FOLD ? F : 1][2];
#pragma unroll
  for (int i = 0; i < F; ++i)
#pragma unroll
    for (int j = 0; j < F; ++j) {
      acc[i][j][0] = acc[i][j][1] = 0.0;
      if constexpr (FOLD) sum[i][j][0] = sum[i][j][1] = 0.0;
    }
  // the next k-tile's elements are fetched into registers while the
  // tensor cores work on the current one
  cd va[H], vb[H];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int h = 0; h < H; ++h) {  // A: T x 8 complex
      const int r = tid / 8 + 32 * h, c = tid % 8;
      va[h] = k0 + c < k ? fa(r, k0 + c) : cd{0.0, 0.0};
    }
#pragma unroll
    for (int h = 0; h < H; ++h) {  // B: 8 x T complex
      const int r = tid / T + 8 / H * h, c = tid % T;
      vb[h] = k0 + r < k ? fb(k0 + r, c) : cd{0.0, 0.0};
    }
  };
  if (k > 0) fetch(0);
  for (int k0 = 0; k0 < k; k0 += kTK) {
    // A as (re, im) pairs; B element as the 2 x 2 block [[re, im], [-im, re]]
#pragma unroll
    for (int h = 0; h < H; ++h) {
      const int r = tid / 8 + 32 * h, c = tid % 8;
      sm.As[r][2 * c] = va[h].x;
      sm.As[r][2 * c + 1] = va[h].y;
    }
#pragma unroll
    for (int h = 0; h < H; ++h) {
      const int r = tid / T + 8 / H * h, c = tid % T;
      sm.Bs[2 * r][2 * c] = vb[h].x;
      sm.Bs[2 * r][2 * c + 1] = vb[h].y;
      sm.Bs[2 * r + 1][2 * c] = -vb[h].y;
      sm.Bs[2 * r + 1][2 * c + 1] = vb[h].x;
    }
    __syncthreads();
    if (k0 + kTK < k) fetch(k0 + kTK);
#pragma unroll
    for (int ks = 0; ks < 2 * kTK; ks += 4) {
      double a[F], b[F];
#pragma unroll
      for (int i = 0; i < F; ++i) a[i] = sm.As[wm * (T / 2) + i * 8 + g][ks + t];
#pragma unroll
      for (int j = 0; j < F; ++j) b[j] = sm.Bs[ks + t][wn * (T / 2) + j * 8 + g];
#pragma unroll
      for (int i = 0; i < F; ++i)
#pragma unroll
        for (int j = 0; j < F; ++j) dmma_884(acc[i][j][0], acc[i][j][1], a[i], b[j]);
    }
    __syncthreads();
    if constexpr (FOLD) {
      if ((k0 & 1023) == 1024 - kTK) {
#pragma unroll
        for (int i = 0; i < F; ++i)
#pragma unroll
          for (int j = 0; j < F; ++j)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              sum[i][j][e] += acc[i][j][e];
              acc[i][j][e] = 0.0;
            }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < F; ++i)
#pragma unroll
    for (int j = 0; j < F; ++j) {
      cd v{acc[i][j][0], acc[i][j][1]};
      if constexpr (FOLD) v = cadd(cd{sum[i][j][0], sum[i][j][1]}, v);
      put(wm * (T / 2) + i * 8 + g, wn * (T / 4) + j * 4 + t, v);
    }
}

// One T x T tile of C = alpha * A(m x k) * B(k x n) + beta * C, tile origin (r0, c0).
// If dA is non-null the columns of A are first multiplied by dA[k] (a diagonal factor).
template <int T = kTM>
static __device__ void cta_gemm_tile(int m, int n, int k, cd alpha, const cd *A, int lda, const cd *B,
                              int ldb, cd beta, cd *C, int ldc_, int r0, int c0, GemmSmem &sm,
                              const cd *dA_col = nullptr) {
  const bool zero_beta = beta.x == 0.0 && beta.y == 0.0;
  cta_tile<T, false>(
      k,
      [&](int r, int kk) {
        cd v = cd{0.0, 0.0};
        if (r0 + r < m) {
          v = A[(size_t)(r0 + r) * lda + kk];
          if (dA_col) v = cmul(v, dA_col[kk]);
        }
        return v;
      },
      [&](int kk, int c) { return c0 + c < n ? B[(size_t)kk * ldb + c0 + c] : cd{0.0, 0.0}; },
      [&](int r, int c, cd x) {
        if (r0 + r >= m || c0 + c >= n) return;
        cd v = cmul(alpha, x);
        cd *pc = C + (size_t)(r0 + r) * ldc_ + c0 + c;
        if (!zero_beta) v = cadd(v, cmul(beta, *pc));
        *pc = v;
      },
      sm);
}

// Shared memory of the team routines, at the start of the dynamic allocation:
// the routines are called, not inlined (a cascade calls the GEMM a dozen
// times; inlined, the kernel spilled 4 KB a thread), and find their shared
// memory there instead of through generic pointers.
struct LuSmem {
  cd tri[kNB][kNB];  // a diagonal block, by columns
  cd invd[kNB];      // reciprocals of its diagonal
  cd prow[kNB], jrow[kNB];  // the pivot row of a panel step and the row it replaces
  cd my[2];          // the next pivot: (value, index), reciprocal
  int piv[kNB];      // the block's interchanges
};
struct TeamSmem {
  GemmSmem gs;
  LuSmem ls;
  double red[2 * kDLThreads / 32];
  int next, bad;  // the uneven batch's
};
__device__ __forceinline__ unsigned char *team_dyn() {
  extern __shared__ __align__(16) unsigned char dyn[];
  return dyn;
}
__device__ __forceinline__ TeamSmem &team_shared() { return *reinterpret_cast<TeamSmem *>(team_dyn()); }

// Then what the kernel wants (`extra` bytes), the row bookkeeping of the
// interchanges (two ints per row), and the panel (rows x kPanelLd) when it
// fits.
constexpr int kPanelLd = kNB + 1;
constexpr size_t kTeamFixed = (sizeof(TeamSmem) + 15) / 16 * 16;
constexpr size_t kTeamMaxSmem = 226 * 1024;
struct PanelSmem {
  int panel;    // byte offset of the panel, 0: it stays in global memory
  int src;      // byte offsets: [n] row each row of the current block's interchanges came from
  int perm;     // [n] original row of every row
  __device__ __forceinline__ int *src_p() const { return reinterpret_cast<int *>(team_dyn() + src); }
  __device__ __forceinline__ int *perm_p() const { return reinterpret_cast<int *>(team_dyn() + perm); }
};
__host__ __device__ inline size_t team_ints(int n) { return (2 * sizeof(int) * (size_t)n + 15) / 16 * 16; }
__host__ __device__ inline size_t team_smem(int n, size_t extra = 0) {
  const size_t fixed = kTeamFixed + extra + team_ints(n), pan = (size_t)n * kPanelLd * sizeof(cd);
  return fixed + (fixed + pan <= kTeamMaxSmem ? pan : 0);
}
__device__ __forceinline__ PanelSmem team_panel(int n_max, size_t extra = 0) {
  const size_t at = kTeamFixed + extra, fixed = at + team_ints(n_max);
  const bool fits = fixed + (size_t)n_max * kPanelLd * sizeof(cd) <= kTeamMaxSmem;
  return PanelSmem{fits ? (int)fixed : 0, (int)at, (int)(at + sizeof(int) * (size_t)n_max)};
}

// C = alpha A B + beta C over all tiles, dealt to the team's CTAs (no sync
// before or after).  Tiles of 32 where they leave less padding and fewer CTAs
// idle: a tile of 64 costs four of them, less about a fifth for their
// prologues.
static __device__ __noinline__ void team_gemm(Team tm, int m, int n, int k, cd alpha, const cd *A, int lda, const cd *B,
                                              int ldb, cd beta, cd *C, int ldc_, const cd *dA_col = nullptr) {
  GemmSmem &sm = team_shared().gs;
  const int n64 = (n + 63) / 64, t64 = (m + 63) / 64 * n64, n32 = (n + 31) / 32, t32 = (m + 31) / 32 * n32;
  if (5 * ((t32 + tm.size - 1) / tm.size) >= 16 * ((t64 + tm.size - 1) / tm.size)) {
    for (int t = tm.rank; t < t64; t += tm.size)
      cta_gemm_tile<64>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc_, t / n64 * 64, t % n64 * 64, sm, dA_col);
  } else {
    for (int t = tm.rank; t < t32; t += tm.size)
      cta_gemm_tile<32>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc_, t / n32 * 32, t % n32 * 32, sm, dA_col);
  }
}

// |re| + |im| (LAPACK dcabs1, the pivot measure of izamax)
__device__ __forceinline__ double cabs1(cd a) { return fabs(a.x) + fabs(a.y); }

// Maximum over the warp of non-negative values, the smallest index among
// equals (i = n: no value)
__device__ __forceinline__ void warp_argmax(double &v, int &i, int n) {
  const uint64_t k = i < n ? (uint64_t)__double_as_longlong(v) : 0;
  const uint32_t hi = (uint32_t)(k >> 32), mhi = __reduce_max_sync(0xffffffffu, hi);
  const uint32_t lo = hi == mhi ? (uint32_t)k : 0, mlo = __reduce_max_sync(0xffffffffu, lo);
  i = (int)__reduce_min_sync(0xffffffffu, (hi == mhi && lo == mlo) ? (uint32_t)i : (uint32_t)n);
  v = __longlong_as_double((long long)(((uint64_t)mhi << 32) | mlo));
}

// Columns j0 .. j0 + jb - 1 of the LU of A by one CTA, on rows j0 .. n - 1 of
// these columns only (pointer P to A[j0][j0], leading dimension ldp: shared or
// global memory).  Pivot rule of izamax.  Per column: swap and scale in one
// pass, then warp 0 updates the next column, finds its pivot and inverts it
// while the other warps update the rest.  Returns the first zero pivot + 1.
template <class Ptr>
static __device__ __forceinline__ int cta_panel(int rows, int jb, int j0, Ptr P, int ldp, int *ipiv) {
  LuSmem &ls = team_shared().ls;
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, w = tid >> 5, nw = nt >> 5;
  auto publish = [&](double best, int bi, int c) {
    warp_argmax(best, bi, rows);
    __syncwarp();
    const cd piv = bi < rows ? P[(size_t)bi * ldp + c] : cd{0.0, 0.0};
    const cd r = (piv.x == 0.0 && piv.y == 0.0) ? cd{0.0, 0.0} : crecip(piv);
    if (lane == 0) {
      ls.my[0] = cd{best, __longlong_as_double((long long)bi)};
      ls.my[1] = r;
    }
  };
  if (w == 0) {
    double best = -1.0;
    int bi = rows;
    for (int i = lane; i < rows; i += 32) {
      const double v = cabs1(P[(size_t)i * ldp]);
      if (v > best) {
        best = v;
        bi = i;
      }
    }
    publish(best, bi, 0);
  }
  int first_zero = 0;
  for (int j = 0; j < jb; ++j) {
    __syncthreads();
    int p = (int)__double_as_longlong(ls.my[0].y);
    cd r = ls.my[1];
    const bool none = p >= rows;  // no comparable candidate (NaN column): keep the row
    if (none) {
      p = j;
      r = crecip(P[(size_t)j * ldp + j]);
    }
    if (w == nw - 1 && lane < jb) {
      ls.prow[lane] = P[(size_t)p * ldp + lane];
      ls.jrow[lane] = P[(size_t)j * ldp + lane];
    }
    __syncthreads();
    const cd ajj = ls.prow[j];
    const bool zero = ajj.x == 0.0 && ajj.y == 0.0;
    if (zero && !first_zero) first_zero = j0 + j + 1;
    if (p != j && w == nw - 1 && lane < jb) {
      P[(size_t)j * ldp + lane] = ls.prow[lane];
      if (lane != j) P[(size_t)p * ldp + lane] = ls.jrow[lane];  // column j by the scaling
    }
    if (tid == 0) ipiv[j0 + j] = j0 + p;
    for (int i = j + 1 + tid; i < rows; i += nt) {
      const cd v = (i == p) ? ls.jrow[j] : P[(size_t)i * ldp + j];
      P[(size_t)i * ldp + j] = zero ? v : cmul(v, r);
    }
    __syncthreads();
    for (int c = w == 0 ? j + 1 : j + 1 + w; c < jb; c += w == 0 ? kNB : nw - 1) {
      const cd u = ls.prow[c];
      double best = -1.0;
      int bi = rows;
      for (int i = j + 1 + lane; i < rows; i += 32) {
        cd v = P[(size_t)i * ldp + c];
        if (!zero) {
          v = csub(v, cmul(P[(size_t)i * ldp + j], u));
          P[(size_t)i * ldp + c] = v;
        }
        if (w == 0) {
          const double m = cabs1(v);
          if (m > best) {
            best = m;
            bi = i;
          }
        }
      }
      if (w == 0) publish(best, bi, c);
    }
  }
  __syncthreads();
  return first_zero;
}

// x := L^-1 x for the unit lower block in ls.tri (terms from the first unknown
// to the last), x := U^-1 x for the upper one (from the last to the first); each
// column of the block updates all unknowns, so the multiply-adds overlap.  R:
// unknowns held, rb of them in use.
template <int R>
__device__ __forceinline__ void lower_regs(cd (&x)[R], int rb) {
  const LuSmem &ls = team_shared().ls;
#pragma unroll
  for (int t = 0; t < R - 1; ++t) {
    if (t < rb) {
#pragma unroll
      for (int r = t + 1; r < R; ++r) x[r] = csub(x[r], cmul(ls.tri[t][r], x[t]));
    }
  }
}
template <int R>
__device__ __forceinline__ void upper_regs(cd (&x)[R], int rb) {
  const LuSmem &ls = team_shared().ls;
#pragma unroll
  for (int t = R - 1; t >= 0; --t) {
    if (t < rb) {
      x[t] = cmul(x[t], ls.invd[t]);
#pragma unroll
      for (int r = 0; r < t; ++r) x[r] = csub(x[r], cmul(ls.tri[t][r], x[t]));
    }
  }
}
// the block at rows and columns r0 .. r0 + rb - 1 into ls.tri, zero elsewhere
__device__ __forceinline__ void stage_tri(const cd *A, int lda, int r0, int rb, bool upper) {
  LuSmem &ls = team_shared().ls;
  for (int e = threadIdx.x; e < kNB * kNB; e += blockDim.x) {
    const int r = e / kNB, t = e % kNB;
    ls.tri[t][r] = (r < rb && t < rb && (upper ? r < t : t < r)) ? A[(size_t)(r0 + r) * lda + r0 + t] : cd{0.0, 0.0};
  }
  if (upper && (int)threadIdx.x < rb) ls.invd[threadIdx.x] = crecip(A[(size_t)(r0 + threadIdx.x) * lda + r0 + threadIdx.x]);
  __syncthreads();
}

// unknowns held in registers by a column solve (16 for short blocks)
template <int R>
struct Held {
  char size[R];
};

// In-place LU with partial pivoting of the n x n matrix A (row-major), as
// LAPACK zgetrf: A = P L U, unit L below the diagonal, U on and above;
// ipiv[j] = row swapped with j (0-based).  The first CTA factors each panel;
// then every CTA brings the interchanges to its columns (the block's rows are
// gathered into registers, each other row that moved comes from the block) and
// solves U12 on the way, and the trailing update is dealt out in tiles.
// ps.perm_p()[i] (in every CTA) = original row of row i.  Returns info on rank 0 (0,
// or j+1 for the first exactly-zero pivot; the factorisation continues as
// LAPACK does).  The team must be in sync on entry; it is on return.
static __device__ __noinline__ int team_getrf(Team tm, int n, cd *A, int lda, int *ipiv, PanelSmem ps) {
  LuSmem &ls = team_shared().ls;
  int *src = ps.src_p(), *perm = ps.perm_p();
  const int tid = threadIdx.x, nt = blockDim.x;
  for (int i = tid; i < n; i += nt) perm[i] = i;
  int info = 0;
  for (int j0 = 0; j0 < n; j0 += kNB) {
    const int jb = min(kNB, n - j0), j1 = j0 + jb, rows = n - j0;
    if (tm.rank == 0) {
      int z;
      if (ps.panel) {
        cd *pm = reinterpret_cast<cd *>(team_dyn() + ps.panel);
        for (int e = tid; e < rows * jb; e += nt)
          pm[(e / jb) * kPanelLd + e % jb] = A[(size_t)(j0 + e / jb) * lda + j0 + e % jb];
        __syncthreads();
        z = cta_panel(rows, jb, j0, pm, kPanelLd, ipiv);
        for (int e = tid; e < rows * jb; e += nt)
          A[(size_t)(j0 + e / jb) * lda + j0 + e % jb] = pm[(e / jb) * kPanelLd + e % jb];
      } else {
        z = cta_panel(rows, jb, j0, A + (size_t)j0 * lda + j0, lda, ipiv);
      }
      if (z && !info) info = z;
    }
    for (int i = tid; i < rows; i += nt) src[i] = j0 + i;
    tm.sync();
    if (tid < jb) ls.piv[tid] = ipiv[j0 + tid];
    __syncthreads();
    if (tid == 0)
      for (int j = j0; j < j1; ++j) {
        const int p = ls.piv[j - j0];
        if (p != j) {
          int t = src[j - j0];
          src[j - j0] = src[p - j0];
          src[p - j0] = t;
          t = perm[j];
          perm[j] = perm[p];
          perm[p] = t;
        }
      }
    stage_tri(A, lda, j0, jb, false);
    auto columns = [&](auto held) {
      constexpr int R = sizeof(held);
      for (int t = tm.col(); t < n - jb; t += tm.nt()) {
        const int c = t < j0 ? t : t + jb;
        cd x[R];
#pragma unroll
        for (int r = 0; r < R; ++r) x[r] = r < jb ? A[(size_t)src[r] * lda + c] : cd{0.0, 0.0};
#pragma unroll 8
        for (int r = 0; r < jb; ++r) {
          const int p = ls.piv[r];
          if (p >= j1) A[(size_t)p * lda + c] = A[(size_t)src[p - j0] * lda + c];
        }
        if (c >= j1) lower_regs(x, jb);
#pragma unroll
        for (int r = 0; r < R; ++r)
          if (r < jb) A[(size_t)(j0 + r) * lda + c] = x[r];
      }
    };
    if (jb > kNB / 2) columns(Held<kNB>{});
    else columns(Held<kNB / 2>{});
    tm.sync();
    const int rest = n - j1;
    if (rest > 0) {
      // A22 -= L21 U12
      team_gemm(tm, rest, rest, jb, cd{-1.0, 0.0}, A + (size_t)j1 * lda + j0, lda, A + (size_t)j0 * lda + j1, lda,
                cd{1.0, 0.0}, A + (size_t)j1 * lda + j1, lda);
      tm.sync();
    }
  }
  return info;
}

// X := U^-1 L^-1 X (n x nrhs, its rows already in the factors' order).  In sync
// on entry and on return.
static __device__ __noinline__ void team_getrs(Team tm, int n, int nrhs, const cd *LU, int lda, cd *X, int ldx) {
  const cd one{1.0, 0.0}, mone{-1.0, 0.0};
  auto columns = [&](auto held, int r0, int rb, bool upper) {
    constexpr int R = sizeof(held);
    for (int c = tm.col(); c < nrhs; c += tm.nt()) {
      cd x[R];
#pragma unroll
      for (int r = 0; r < R; ++r) x[r] = r < rb ? X[(size_t)(r0 + r) * ldx + c] : cd{0.0, 0.0};
      if (upper) upper_regs(x, rb);
      else lower_regs(x, rb);
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (r < rb) X[(size_t)(r0 + r) * ldx + c] = x[r];
    }
  };
  auto solve = [&](int r0, int rb, bool upper) {
    stage_tri(LU, lda, r0, rb, upper);
    if (rb > kNB / 2) columns(Held<kNB>{}, r0, rb, upper);
    else columns(Held<kNB / 2>{}, r0, rb, upper);
    tm.sync();
  };
  for (int r0 = 0; r0 < n; r0 += kNB) {
    const int r1 = min(n, r0 + kNB);
    solve(r0, r1 - r0, false);
    if (r1 < n) {
      team_gemm(tm, n - r1, nrhs, r1 - r0, mone, LU + (size_t)r1 * lda + r0, lda, X + (size_t)r0 * ldx, ldx, one,
                X + (size_t)r1 * ldx, ldx);
      tm.sync();
    }
  }
  for (int r1 = n; r1 > 0; r1 -= kNB) {
    const int r0 = max(0, r1 - kNB);
    solve(r0, r1 - r0, true);
    if (r0 > 0) {
      team_gemm(tm, r0, nrhs, r1 - r0, mone, LU + r0, lda, X + (size_t)r0 * ldx, ldx, one, X, ldx);
      tm.sync();
    }
  }
}

// The row interchanges of team_getrf on X, in place (one thread per column).
static __device__ void team_swap_rows(Team tm, int n, int nrhs, const int *ipiv, cd *X, int ldx) {
  for (int c = tm.tid(); c < nrhs; c += tm.nt())
    for (int j = 0; j < n; ++j) {
      const int p = ipiv[j];
      if (p != j) {
        const cd t = X[(size_t)j * ldx + c];
        X[(size_t)j * ldx + c] = X[(size_t)p * ldx + c];
        X[(size_t)p * ldx + c] = t;
      }
    }
  tm.sync();
}

// A X = B of a batch (emu_zgesv_batched), X over B.
struct GesvArgs {
  int n, nrhs, lda, ldb;
  long long sA, sB;
  cd *A;
  cd *B;
  int *ipiv;
  int *info;
};
__device__ __forceinline__ void team_gesv(const GesvArgs &g) {
  const Team tm = cluster_team();
  const int b = blockIdx.x / tm.size;
  cd *A = g.A + b * g.sA;
  cd *B = g.B + b * g.sB;
  int *ipiv = g.ipiv + (size_t)b * g.n;
  const int info = team_getrf(tm, g.n, A, g.lda, ipiv, team_panel(g.n));
  if (g.nrhs > 0) {
    team_swap_rows(tm, g.n, g.nrhs, ipiv, B, g.ldb);
    team_getrs(tm, g.n, g.nrhs, A, g.lda, B, g.ldb);
  }
  if (tm.tid() == 0 && g.info) g.info[b] = info;
}

// CTAs per problem: while all of them are resident at once (the kernels take an
// SM per CTA), at most 8 and no more than a matrix has 32 x 32 tiles.  Measured
// for the chain of 50 problems of P = 58, M = 60 with 1 / 2 / 4 / 8 CTAs each:
// interfaces 0.45 / 0.41 / 0.71 / 1.35 ms, cascades 0.85 / 0.78 / 1.32 / 2.5 ms
// (with 4 and 8 they no longer fit at once).
inline int team_size(int count, int n, int sms) {
  const long long tiles = (long long)((n + 31) / 32) * ((n + 31) / 32);
  int cs = 1;
  while (cs < 8 && 2LL * cs * count <= sms && 2 * cs <= tiles) cs *= 2;
  return cs;
}

// Launches a team kernel: `grid` problems (or slots) of cs CTAs each.  The
// shared-memory limit is set to its largest value, so that threads that launch
// other sizes at once never see a smaller one.
template <class F, class... Args>
inline cudaError_t launch_team(F *kernel, int grid, int cs, size_t smem, cudaStream_t s, Args... args) {
  cudaError_t e = cudaFuncSetAttribute((const void *)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)kTeamMaxSmem);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid * cs);
  cfg.blockDim = dim3(kDLThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cs;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

}  // namespace emu
