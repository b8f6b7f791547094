// Multi-CTA batched dense linear algebra for large interface and cascade
// solves: the steps of the team routines of dense_la.cuh, but every step is its
// own launch over all problems of a batch and spreads each matrix over many
// CTAs.  Small matrices (one block, no residue scratch) keep the teams' tiles,
// panel width and order of operations, and so their bits; larger ones factor
// recursively and compute deep GEMMs as residues on the INT8 tensor cores.
//   LU (zgetrf): per panel of kNB columns, one CTA or one cluster per matrix
//     factors the panel (pivot search, row swaps, rank-1 updates), then a
//     column-parallel unit-lower solve forms U12 and a GEMM updates A22;
//   solve (zgetrs): row interchanges, then blocked forward / backward
//     substitution with column-parallel triangular solves and tiled GEMMs.
// Batched matrices are (base pointer, batch stride in elements, leading
// dimension); problem b is blockIdx.y (.z for the GEMM).
#pragma once
#include <algorithm>
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "dense_la.cuh"
#include "emu_internal.h"
#include "residue_gemm.cuh"

namespace {

using namespace emu;

// ---------------------------------------------------------------- GEMM
struct BGemm {
  int m, n, k;
  cd alpha, beta;
  const cd *A;
  long long sA;
  int lda;
  const cd *B;
  long long sB;
  int ldb;
  cd *C;
  long long sC;
  int ldc;
  const cd *dA;  // optional diagonal scaling of A's columns [b][k]
  long long sdA;
};

__global__ void __launch_bounds__(kDLThreads) bgemm_kernel(BGemm g) {
  __shared__ GemmSmem sm;
  const long long b = blockIdx.z;
  cta_gemm_tile(g.m, g.n, g.k, g.alpha, g.A + b * g.sA, g.lda, g.B + b * g.sB, g.ldb, g.beta,
                g.C + b * g.sC, g.ldc, blockIdx.y * kTM, blockIdx.x * kTN, sm,
                g.dA ? g.dA + b * g.sdA : nullptr);
}

inline void bgemm(int m, int n, int k, cd alpha, const cd *A, long long sA, int lda, const cd *B,
                  long long sB, int ldb, cd beta, cd *C, long long sC, int ldc, int batch,
                  cudaStream_t s, const cd *dA = nullptr, long long sdA = 0) {
  if (m <= 0 || n <= 0 || batch <= 0) return;
  BGemm g{m, n, k, alpha, beta, A, sA, lda, B, sB, ldb, C, sC, ldc, dA, sdA};
  dim3 grid((n + kTN - 1) / kTN, (m + kTM - 1) / kTM, batch);
  bgemm_kernel<<<grid, kDLThreads, 0, s>>>(g);
  note_launch();
}

// ---------------------------------------------------------------- LU
// One CTA per matrix: columns j0 .. j0 + jb - 1 of the LU of A (as the
// inner loop of a team's LU): pivot search, full-row swap, column scaling,
// rank-1 update of the rest of the panel.  info[b] = code + j + 1 for the
// first exactly-zero pivot of this factorisation if info[b] is still 0.
constexpr int kPanelThreads = 1024;
struct WidePanelSmem {
  double val[kPanelThreads / 32];
  int idx[kPanelThreads / 32];
  int piv;
};

__global__ void __launch_bounds__(kPanelThreads) panel_kernel(cd *A_, long long sA, int lda, int n, int j0,
                                                              int jb, int *ipiv_, long long sip,
                                                              int *info, int code) {
  __shared__ WidePanelSmem ls;
  const int tid = threadIdx.x, nt = blockDim.x;
  const long long b = blockIdx.x;
  cd *A = A_ + b * sA;
  int *ipiv = ipiv_ + b * sip;
  for (int j = j0; j < j0 + jb; ++j) {
    double best = -1.0;
    int bi = n;
    for (int i = j + tid; i < n; i += nt) {
      const double v = cabs1(A[(size_t)i * lda + j]);
      if (v > best) {
        best = v;
        bi = i;
      }
    }
    for (int o = 16; o > 0; o >>= 1) {
      const double ov = __shfl_down_sync(0xffffffffu, best, o);
      const int oi = __shfl_down_sync(0xffffffffu, bi, o);
      if (ov > best || (ov == best && oi < bi)) {
        best = ov;
        bi = oi;
      }
    }
    if ((tid & 31) == 0) {
      ls.val[tid >> 5] = best;
      ls.idx[tid >> 5] = bi;
    }
    __syncthreads();
    if (tid == 0) {
      double bv = ls.val[0];
      int bx = ls.idx[0];
      for (int w = 1; w < nt / 32; ++w)
        if (ls.val[w] > bv || (ls.val[w] == bv && ls.idx[w] < bx)) {
          bv = ls.val[w];
          bx = ls.idx[w];
        }
      ls.piv = bx < n ? bx : j;  // no comparable candidate (NaN column): keep the row
    }
    __syncthreads();
    const int p = ls.piv;
    if (tid == 0) ipiv[j] = p;
    if (p != j) {
      for (int c = tid; c < n; c += nt) {
        const cd t = A[(size_t)j * lda + c];
        A[(size_t)j * lda + c] = A[(size_t)p * lda + c];
        A[(size_t)p * lda + c] = t;
      }
    }
    __syncthreads();
    const cd ajj = A[(size_t)j * lda + j];
    const bool zero = ajj.x == 0.0 && ajj.y == 0.0;
    if (zero) {
      if (tid == 0 && info && info[b] == 0) info[b] = code + j + 1;
    } else {
      const cd r = crecip(ajj);
      for (int i = j + 1 + tid; i < n; i += nt) A[(size_t)i * lda + j] = cmul(A[(size_t)i * lda + j], r);
    }
    __syncthreads();
    const int pc = j0 + jb - (j + 1);
    if (!zero && pc > 0) {
      const int rows = n - (j + 1);
      for (int e = tid; e < rows * pc; e += nt) {
        const int i = j + 1 + e / pc, c = j + 1 + e % pc;
        A[(size_t)i * lda + c] = csub(A[(size_t)i * lda + c], cmul(A[(size_t)i * lda + j], A[(size_t)j * lda + c]));
      }
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------- cluster panel
// The same panel factorisation by a thread-block cluster of cs CTAs per
// matrix: CTA q holds panel rows j0 + q, j0 + q + cs, ... (columns j0 ..
// j0+jb-1) in shared memory, one pad entry per row so that neighbouring rows
// start in different banks.  A panel is a chain of column steps, so what
// counts is the length of one step:
//   - every CTA sends its pivot candidate (value, index, reciprocal and whole
//     row) and the owner of row j that row to all CTAs with st.async, which
//     counts the bytes on the receiver's mbarrier: a step waits for its data
//     only, without a cluster barrier and its memory fence.  Two buffers by
//     column parity: nobody can be two columns ahead, because a column's data
//     are sent after the previous column's were received and used;
//   - each CTA picks the winner from its own copies, swaps and scales in one
//     pass, and updates its rows; warp 0 takes the next column, finds its
//     candidate and inverts it while the other warps update the rest.
// Same arithmetic and pivot choice as team_getrf.  The swaps of the columns
// outside the panel are left to laswp_outside_kernel.  Waits are bounded: one
// that gives up is reported through info.
// Measured for 16 panels of 634 x 32 on 8 CTAs each: 148 us with unpadded
// rows, one thread per row and two cluster barriers a column, 114 us with one
// barrier and padded rows, 75 us as it is (6 144 x 32 on 16 CTAs: 244, 164 and
// 100 us).
constexpr int kPanelMaxCS = 8;
constexpr int kPanelCTAThreads = 512;
constexpr int kPanelRow = kNB + 1;
constexpr size_t kPanelMaxSmem = 224 * 1024;
constexpr int kPanelClusterMax = 16;
constexpr int kPanelWaitLimit = 1 << 22;

// rows, 2 candidate rows per CTA of the cluster, 2 copies of row j
__host__ __device__ inline size_t panel_smem(long long rows, int cs) {
  return (size_t)(rows + 2 * cs + 2) * kPanelRow * sizeof(cd);
}

// 16 bytes to the same place in CTA `rank` of the cluster, counted on its
// mbarrier `bar` (both given as this CTA's addresses)
__device__ __forceinline__ void cluster_send(const void *dst, const void *bar, int rank, cd v) {
  asm volatile(
      "{\n\t"
      ".reg .b32 d, m;\n\t"
      "mapa.shared::cluster.u32 d, %0, %2;\n\t"
      "mapa.shared::cluster.u32 m, %1, %2;\n\t"
      "st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [d], {%3, %4}, [m];\n\t"
      "}\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
      "r"((uint32_t)__cvta_generic_to_shared(bar)), "r"(rank), "l"(__double_as_longlong(v.x)),
      "l"(__double_as_longlong(v.y))
      : "memory");
}

__global__ void __launch_bounds__(kPanelCTAThreads) panel_cluster_kernel(cd *A_, long long sA, int lda, int n,
                                                                         int j0, int jb, int *ipiv_,
                                                                         long long sip, int *info, int code) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  extern __shared__ __align__(16) unsigned char psm[];
  __shared__ __align__(16) cd meta[2][kPanelClusterMax][2];  // the cluster's candidates: (value, index), 1 / pivot
  __shared__ __align__(8) uint64_t bar[2];
  __shared__ cd my[2];  // this CTA's candidate, as meta
  const int q = (int)cl.block_rank(), cs = (int)cl.num_blocks();
  const long long b = blockIdx.x / cs;
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, w = tid >> 5, nw = nt >> 5;
  cd *A = A_ + b * sA;
  int *ipiv = ipiv_ + b * sip;
  const int nr = n - j0;                                  // panel rows
  const int my_rows = nr > q ? (nr - q + cs - 1) / cs : 0;
  const int max_rows = (nr + cs - 1) / cs;
  cd *Pm = reinterpret_cast<cd *>(psm);                  // [max_rows][kPanelRow]
  cd *cand = Pm + (size_t)max_rows * kPanelRow;          // [2][cs][kPanelRow]
  cd *jcopy = cand + (size_t)2 * cs * kPanelRow;         // [2][kPanelRow]
  auto grow = [&](int l) { return j0 + q + cs * l; };   // local row l -> matrix row
  if (tid == 0) {
    for (int i = 0; i < 2; ++i)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"((uint32_t)__cvta_generic_to_shared(bar + i)));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int e = tid; e < my_rows * jb; e += nt) {
    const int l = e / jb, c = e % jb;
    Pm[l * kPanelRow + c] = A[(size_t)grow(l) * lda + j0 + c];
  }
  __syncthreads();
  // warp 0: this CTA's candidate in column c from each lane's best
  auto publish = [&](double best, int bi, int c) {
    warp_argmax(best, bi, n);
    __syncwarp();
    const cd piv = bi < n ? Pm[(bi - j0) / cs * kPanelRow + c] : cd{0.0, 0.0};
    const cd r = (piv.x == 0.0 && piv.y == 0.0) ? cd{0.0, 0.0} : crecip(piv);
    if (lane == 0) {
      my[0] = cd{best, __longlong_as_double((long long)bi)};
      my[1] = r;
    }
  };
  if (w == 0) {
    double best = -1.0;
    int bi = n;
    for (int l = lane; l < my_rows; l += 32) {
      const double v = cabs1(Pm[l * kPanelRow]);
      if (v > best) {
        best = v;
        bi = grow(l);
      }
    }
    publish(best, bi, 0);
  }
  cl.sync();  // every CTA's mbarriers are ready before the first send
  int first_zero = 0;
  bool ok = true;
  int jj = 0;
  for (; jj < jb; ++jj) {
    const int j = j0 + jj, par = jj & 1;
    const int qj = jj % cs, lj = jj / cs;
    __syncthreads();  // the previous column's update and `my`
    {
      const int ci = (int)__double_as_longlong(my[0].y);
      const int lc = ci < n ? (ci - j0) / cs : 0;  // without a candidate any row goes: the byte count is fixed
      for (int r = w; r < cs; r += nw) {
        if (lane < jb) {
          cluster_send(cand + ((size_t)par * cs + q) * kPanelRow + lane, bar + par, r, Pm[lc * kPanelRow + lane]);
          if (q == qj) cluster_send(jcopy + par * kPanelRow + lane, bar + par, r, Pm[lj * kPanelRow + lane]);
        }
        if (lane < 2) cluster_send(&meta[par][q][lane], bar + par, r, my[lane]);
      }
      const uint32_t mb = (uint32_t)__cvta_generic_to_shared(bar + par);
      if (tid == 0)
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mb),
                     "r"((uint32_t)((cs * (jb + 2) + jb) * sizeof(cd)))
                     : "memory");
      const uint32_t phase = (uint32_t)(jj >> 1) & 1;
      uint32_t done = 0;
      for (int i = 0; i < kPanelWaitLimit && !done; ++i)
        asm volatile(
            "{\n\t"
            ".reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.b32 %0, 1, 0, p;\n\t"
            "}\n"
            : "=r"(done)
            : "r"(mb), "r"(phase)
            : "memory");
      __syncwarp();
      // the data are here, and every warp has sent its rows: the swap and the
      // scaling below may overwrite them
      ok = __syncthreads_and((int)done) != 0;
    }
    if (!ok) break;  // the candidates may never have come: nothing below may use them
    double bv = lane < cs ? meta[par][lane][0].x : 0.0;
    int p = lane < cs ? (int)__double_as_longlong(meta[par][lane][0].y) : n;
    warp_argmax(bv, p, n);
    const cd *jrow = jcopy + par * kPanelRow;
    const cd *prow = jrow;
    cd r;
    if (p < n) {
      const int qp = (p - j0) % cs;
      prow = cand + ((size_t)par * cs + qp) * kPanelRow;
      r = meta[par][qp][1];
    } else {  // no comparable candidate (NaN column): keep the row
      p = j;
      r = crecip(jrow[jj]);
    }
    const cd ajj = prow[jj];
    const bool zero = ajj.x == 0.0 && ajj.y == 0.0;
    if (zero && !first_zero) first_zero = j + 1;
    // swap (column jj of row p is left to the scaling below)
    const int lp = p != j && q == (p - j0) % cs ? (p - j0) / cs : -1;
    if (p != j && q == qj && w == nw - 1 && lane < jb) Pm[lj * kPanelRow + lane] = prow[lane];
    if (lp >= 0 && w == nw - 2 && lane < jb && lane != jj) Pm[lp * kPanelRow + lane] = jrow[lane];
    if (q == 0 && tid == 0) ipiv[j] = p;
    // rows below j: l >= l0
    const int l0 = q > qj ? lj : lj + 1;
    for (int l = l0 + tid; l < my_rows; l += nt) {
      const cd v = l == lp ? jrow[jj] : Pm[l * kPanelRow + jj];
      Pm[l * kPanelRow + jj] = zero ? v : cmul(v, r);
    }
    __syncthreads();
    // warp 0: column jj + 1 and its candidate; the others share the rest
    for (int c = w == 0 ? jj + 1 : jj + 1 + w; c < jb; c += w == 0 ? kNB : nw - 1) {
      const cd u = prow[c];
      double best = -1.0;
      int bi = n;
      for (int l = l0 + lane; l < my_rows; l += 32) {
        cd v = Pm[l * kPanelRow + c];
        if (!zero) {
          v = csub(v, cmul(Pm[l * kPanelRow + jj], u));
          Pm[l * kPanelRow + c] = v;
        }
        if (w == 0) {
          const double m = cabs1(v);
          if (m > best) {
            best = m;
            bi = grow(l);
          }
        }
      }
      if (w == 0) publish(best, bi, c);
    }
  }
  __syncthreads();
  // a wait that gave up, in whichever CTA: info, NaN factors, and no interchanges
  // in the columns that are left
  if (!ok) {
    first_zero = 1;
    if (q == 0)
      for (int c = jj + tid; c < jb; c += nt) ipiv[j0 + c] = j0 + c;
  }
  if (tid == 0 && info && first_zero && (q == 0 || !ok)) atomicCAS(info + b, 0, code + first_zero);
  for (int e = tid; e < my_rows * jb; e += nt) {
    const int l = e / jb, c = e % jb;
    A[(size_t)grow(l) * lda + j0 + c] = ok ? Pm[l * kPanelRow + c] : cd{nan(""), nan("")};
  }
  cl.sync();  // no CTA leaves while others may still send to it
}

// The panel's row interchanges ipiv[j0 .. j0+jb) applied in order to the
// columns outside the panel, [0, j0) and [j0+jb, n).
__global__ void laswp_outside_kernel(cd *A_, long long sA, int lda, int n, int j0, int jb, const int *ipiv_,
                                     long long sip) {
  const long long b = blockIdx.y;
  cd *A = A_ + b * sA;
  const int *ipiv = ipiv_ + b * sip;
  const int ncols = n - jb;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < ncols; t += gridDim.x * blockDim.x) {
    const int c = t < j0 ? t : t + jb;
    for (int j = j0; j < j0 + jb; ++j) {
      const int p = ipiv[j];
      if (p != j) {
        const cd v = A[(size_t)j * lda + c];
        A[(size_t)j * lda + c] = A[(size_t)p * lda + c];
        A[(size_t)p * lda + c] = v;
      }
    }
  }
}

// The cluster panel's function attributes, set once per device to their
// largest values (kPanelMaxSmem of dynamic shared memory; non-portable
// cluster sizes allowed), never lowered afterwards: host threads that launch
// panels of different sizes at once (two solves on two streams, the server's
// worker threads) then never see a limit another thread set for a smaller
// panel.  Bit 0: the shared-memory limit is set; bit 1: clusters above 8
// CTAs are allowed.  Both threads of a first-call race set the same values.
inline int panel_cluster_attrs() {
  static int state[64] = {};  // 0 = not yet set, else attrs | 4
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  int st = __atomic_load_n(&state[dev], __ATOMIC_ACQUIRE);
  if (st) return st & 3;
  int attrs = 0;
  if (cudaFuncSetAttribute(panel_cluster_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPanelMaxSmem) ==
      cudaSuccess)
    attrs |= 1;
  else
    cudaGetLastError();
  if (cudaFuncSetAttribute(panel_cluster_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess)
    attrs |= 2;
  else
    cudaGetLastError();
  __atomic_store_n(&state[dev], attrs | 4, __ATOMIC_RELEASE);
  return attrs;
}

// Launches the cluster panel; false if it would not beat panel_kernel or
// cannot run (the caller then uses panel_kernel).  Cluster size: enough
// CTAs for the panel to fit in shared memory, and as many more (up to 8) as
// keep all clusters of the batch resident at once; a batch that already
// fills the GPU with one wide CTA per matrix keeps panel_kernel.
inline bool panel_cluster(cd *A, long long sA, int lda, int n, int j0, int jb, int *ipiv, long long sip,
                          int *info, int code, int batch, cudaStream_t s, int max_cs = kPanelMaxCS) {
  const long long nr = n - j0;
  int cs = 0;
  for (int c = max_cs; c >= 1; --c) {
    const size_t smem = panel_smem((nr + c - 1) / c, c);
    if (smem > kPanelMaxSmem) break;
    const long long per_sm = std::min<long long>(2, (long long)(228 * 1024 / (smem + 2048)));
    if ((long long)batch * c <= per_sm * sm_count()) {
      cs = c;
      break;
    }
  }
  if (cs < 2) return false;
  const int attrs = panel_cluster_attrs();
  if (!(attrs & 1)) return false;
  // clusters above 8 CTAs are a non-portable size (the launch fails, and the
  // caller falls back to panel_kernel, where the GPU cannot host them)
  if (cs > 8 && !(attrs & 2)) return false;
  const size_t smem = panel_smem((nr + cs - 1) / cs, cs);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(batch * cs));
  cfg.blockDim = dim3(kPanelCTAThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cs;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cudaLaunchKernelEx(&cfg, panel_cluster_kernel, A, sA, lda, n, j0, jb, ipiv, sip, info, code) !=
      cudaSuccess)
    return false;
  note_launch();
  const int outside = n - jb;
  if (outside > 0) {
    laswp_outside_kernel<<<dim3((unsigned)((outside + 127) / 128), (unsigned)batch), 128, 0, s>>>(
        A, sA, lda, n, j0, jb, ipiv, sip);
    note_launch();
  }
  return true;
}

// X rows r0 .. r0+rb-1 := L11^{-1} X rows (unit lower L11 = L[r0.., r0..],
// rb <= kNB), one thread per column c in [c0, c0 + ncols): the block's L11 is
// staged in shared memory, each column's rb values are held in registers.
// Column by column of L11 (every x[r] takes its terms in the order of
// team_getrf / team_getrs, and those of one column are independent, so the
// multiply-adds overlap: 38 -> 12 us for the upper solve of 16 x 400 columns,
// 13 -> 10 us for the lower one); rows and columns past rb are zero.
constexpr int kTrsmThreads = 64;

__global__ void __launch_bounds__(kTrsmThreads) trsm_lower_kernel(const cd *L_, long long sL, int ldl, int r0, int rb,
                                                                  cd *X_, long long sX, int ldx, int c0, int ncols) {
  __shared__ cd Ls[kNB][kNB];
  const long long b = blockIdx.y;
  const cd *L = L_ + b * sL;
  cd *X = X_ + b * sX;
  for (int e = threadIdx.x; e < kNB * kNB; e += blockDim.x) {
    const int r = e / kNB, t = e % kNB;
    Ls[t][r] = (r < rb && t < r) ? L[(size_t)(r0 + r) * ldl + r0 + t] : cd{0.0, 0.0};
  }
  __syncthreads();
  const int cc = blockIdx.x * blockDim.x + threadIdx.x;
  if (cc >= ncols) return;
  const int c = c0 + cc;
  cd x[kNB];
#pragma unroll
  for (int r = 0; r < kNB; ++r) x[r] = r < rb ? X[(size_t)(r0 + r) * ldx + c] : cd{0.0, 0.0};
#pragma unroll
  for (int t = 0; t < kNB - 1; ++t) {
    if (t < rb) {
#pragma unroll
      for (int r = t + 1; r < kNB; ++r) x[r] = csub(x[r], cmul(Ls[t][r], x[t]));
    }
  }
#pragma unroll
  for (int r = 1; r < kNB; ++r)
    if (r < rb) X[(size_t)(r0 + r) * ldx + c] = x[r];
}

// X rows r0 .. r0+rb-1 := U11^{-1} X rows (upper U11 with its diagonal), from
// the last column of U11 to the first.
__global__ void __launch_bounds__(kTrsmThreads) trsm_upper_kernel(const cd *U_, long long sU, int ldu, int r0, int rb,
                                                                  cd *X_, long long sX, int ldx, int ncols) {
  __shared__ cd Us[kNB][kNB];
  __shared__ cd invd[kNB];
  const long long b = blockIdx.y;
  const cd *U = U_ + b * sU;
  cd *X = X_ + b * sX;
  for (int e = threadIdx.x; e < kNB * kNB; e += blockDim.x) {
    const int r = e / kNB, t = e % kNB;
    Us[t][r] = (t < rb && r < t) ? U[(size_t)(r0 + r) * ldu + r0 + t] : cd{0.0, 0.0};
  }
  if (threadIdx.x < rb) invd[threadIdx.x] = crecip(U[(size_t)(r0 + threadIdx.x) * ldu + r0 + threadIdx.x]);
  __syncthreads();
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncols) return;
  cd x[kNB];
#pragma unroll
  for (int r = 0; r < kNB; ++r) x[r] = r < rb ? X[(size_t)(r0 + r) * ldx + c] : cd{0.0, 0.0};
#pragma unroll
  for (int t = kNB - 1; t >= 0; --t) {
    if (t < rb) {
      x[t] = cmul(x[t], invd[t]);
#pragma unroll
      for (int r = 0; r < t; ++r) x[r] = csub(x[r], cmul(Us[t][r], x[t]));
    }
  }
#pragma unroll
  for (int r = 0; r < kNB; ++r)
    if (r < rb) X[(size_t)(r0 + r) * ldx + c] = x[r];
}

// row interchanges ipiv[0..n) applied in order to the columns of X
__global__ void swap_rows_kernel(cd *X_, long long sX, int ldx, int ncols, const int *ipiv_, long long sip,
                                 int n) {
  const long long b = blockIdx.y;
  cd *X = X_ + b * sX;
  const int *ipiv = ipiv_ + b * sip;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < ncols; c += gridDim.x * blockDim.x) {
    for (int j = 0; j < n; ++j) {
      const int p = ipiv[j];
      if (p != j) {
        const cd t = X[(size_t)j * ldx + c];
        X[(size_t)j * ldx + c] = X[(size_t)p * ldx + c];
        X[(size_t)p * ldx + c] = t;
      }
    }
  }
}

inline dim3 col_grid(int ncols, int batch, int threads = 128) {
  return dim3((unsigned)((ncols + threads - 1) / threads), (unsigned)batch);
}

// Scratch of the residue GEMMs (residue_gemm.cuh); null: every GEMM on the FP64
// tensor cores.  The first error of a residue GEMM goes to *status: the entry
// points return it.
struct RgScratch {
  void *ws;
  size_t bytes;
  int *status;
};

// Sizes from which a GEMM runs as residues on the INT8 tensor cores.  Per
// complex result the residues cost about 30 ps at any depth (their products'
// reduction and the CRT) and 0.03 ps per unit of depth, the FP64 tensor cores
// 0.3 to 0.4 ps per unit.  At depths of 112 to 144 the two are level, at kNB the FP64
// tiles win.  16 interfaces of P = 634, M = 400: 7.6 ms, with FP64 tiles alone 8.3 ms;
// 16 cascades of two such arrays 35.7 and 42.3 ms.
// Few or narrow results leave the launches' time uncovered.  The rule does not look at
// the batch, so that a problem's result does not depend on what it is solved with
// (one interface of P = 226, M = 256: 1.96 ms, with FP64 tiles 2.01; 16 of them 2.69 and
// 2.66 ms).
inline bool gemm_as_residues(int m, int n, int k) {
  return k >= 128 && m >= 96 && n >= 96 && (long long)m * n >= 20000;
}

// Below this dimension a cascade or factorisation asks for no scratch and runs
// in FP64 throughout.
constexpr int kRgMinDim = 256;

inline size_t dense_scratch(int D, int batch) { return D >= kRgMinDim ? rg_dense_scratch(D, D, D, batch) : 0; }

inline void gemm(int m, int n, int k, cd alpha, const cd *A, long long sA, int lda, const cd *B, long long sB, int ldb,
                 cd beta, cd *C, long long sC, int ldc, int batch, const RgScratch &rg, cudaStream_t s,
                 const cd *dA = nullptr, long long sdA = 0) {
  if (m <= 0 || n <= 0 || batch <= 0) return;
  if (rg.ws && gemm_as_residues(m, n, k)) {
    const RgDense g{m, n, k, batch, alpha, beta, A, sA, lda, B, sB, ldb, C, sC, ldc, dA, sdA};
    const int st = rg_dense(g, rg.ws, rg.bytes, s);
    // too little scratch is found before anything is launched; after any other
    // error C may be partly updated
    if (st != EMU_E_WORKSPACE) {
      if (st != EMU_OK && *rg.status == EMU_OK) *rg.status = st;
      return;
    }
  }
  bgemm(m, n, k, alpha, A, sA, lda, B, sB, ldb, beta, C, sC, ldc, batch, s, dA, sdA);
}

// Factorisations and solves recurse on halves down to blocks of kInnerNB: the
// GEMMs between blocks then have depths of n / 2, n / 4, ..., kInnerNB, so the
// matrix is read and written log2(n / kInnerNB) instead of n / kNB times, and
// they run as residues.  Inside a block the updates go panel by panel (depth
// kNB): a recursion down to single panels has many GEMMs and solves of 32 or
// 64 columns, too narrow for their tiles (factor and inverse at n = 6 144 with deep GEMMs
// as residues: 43 against 27 ms in FP64 GEMMs, 22 against 13 ms in solves).  Small matrices
// are one block, in the team kernels' order of operations.
constexpr int kInnerNB = 256;

inline int inner_block(int n, int batch, const RgScratch &rg) {
  return rg.ws || (batch == 1 && n >= 1024) ? kInnerNB : n;
}

// middle of [a, b), whole blocks on its left
inline int half_of(int a, int b) {
  const int blocks = (b - a + kInnerNB - 1) / kInnerNB;
  return a + max(1, blocks / 2) * kInnerNB;
}

struct LuArgs {
  int n;
  cd *A;  // factors
  long long sA;
  int lda, batch;
  RgScratch rg;
  cudaStream_t s;
  int inner;  // blocks of at most this many rows or columns are not halved
};

// X rows [r0, r1) := L^-1 X rows (unit lower triangle of rows and columns [r0,
// r1) of the factors), columns [c0, c0 + nc) of X
inline void lower_solve(const LuArgs &g, int r0, int r1, cd *X, long long sX, int ldx, int c0, int nc) {
  const cd one{1.0, 0.0}, mone{-1.0, 0.0};
  if (nc <= 0) return;
  if (r1 - r0 <= g.inner) {
    for (int r = r0; r < r1; r += kNB) {
      const int e = min(r1, r + kNB);
      trsm_lower_kernel<<<col_grid(nc, g.batch, kTrsmThreads), kTrsmThreads, 0, g.s>>>(g.A, g.sA, g.lda, r, e - r, X, sX,
                                                                                       ldx, c0, nc);
      note_launch();
      bgemm(r1 - e, nc, e - r, mone, g.A + (size_t)e * g.lda + r, g.sA, g.lda, X + (size_t)r * ldx + c0, sX, ldx, one,
            X + (size_t)e * ldx + c0, sX, ldx, g.batch, g.s);
    }
    return;
  }
  const int m = half_of(r0, r1);
  lower_solve(g, r0, m, X, sX, ldx, c0, nc);
  gemm(r1 - m, nc, m - r0, mone, g.A + (size_t)m * g.lda + r0, g.sA, g.lda, X + (size_t)r0 * ldx + c0, sX, ldx, one,
       X + (size_t)m * ldx + c0, sX, ldx, g.batch, g.rg, g.s);
  lower_solve(g, m, r1, X, sX, ldx, c0, nc);
}

// X rows [r0, r1) := U^-1 X rows
inline void upper_solve(const LuArgs &g, int r0, int r1, cd *X, long long sX, int ldx, int nc) {
  const cd one{1.0, 0.0}, mone{-1.0, 0.0};
  if (r1 - r0 <= g.inner) {
    for (int e = r1; e > r0; e -= kNB) {
      const int r = max(r0, e - kNB);
      trsm_upper_kernel<<<col_grid(nc, g.batch, kTrsmThreads), kTrsmThreads, 0, g.s>>>(g.A, g.sA, g.lda, r, e - r, X, sX,
                                                                                       ldx, nc);
      note_launch();
      bgemm(r - r0, nc, e - r, mone, g.A + (size_t)r0 * g.lda + r, g.sA, g.lda, X + (size_t)r * ldx, sX, ldx, one,
            X + (size_t)r0 * ldx, sX, ldx, g.batch, g.s);
    }
    return;
  }
  const int m = half_of(r0, r1);
  upper_solve(g, m, r1, X, sX, ldx, nc);
  gemm(m - r0, nc, r1 - m, mone, g.A + (size_t)r0 * g.lda + m, g.sA, g.lda, X + (size_t)m * ldx, sX, ldx, one,
       X + (size_t)r0 * ldx, sX, ldx, g.batch, g.rg, g.s);
  upper_solve(g, r0, m, X, sX, ldx, nc);
}

inline void factor_panel(const LuArgs &g, int j0, int jb, int *ipiv, long long sip, int *info, int code, int max_cs) {
  // a panel is a latency-bound chain of column steps: a cluster of CTAs
  // keeps the panel in shared memory (one wide CTA through L2 otherwise;
  // the arithmetic is the same)
  if (!panel_cluster(g.A, g.sA, g.lda, g.n, j0, jb, ipiv, sip, info, code, g.batch, g.s, max_cs)) {
    cudaGetLastError();
    panel_kernel<<<g.batch, kPanelThreads, 0, g.s>>>(g.A, g.sA, g.lda, g.n, j0, jb, ipiv, sip, info, code);
    note_launch();
  }
}

// columns [j0, j1) of the factorisation, the columns on their left done
inline void lu_columns(const LuArgs &g, int j0, int j1, int *ipiv, long long sip, int *info, int code, int max_cs) {
  const cd one{1.0, 0.0}, mone{-1.0, 0.0};
  if (j1 - j0 <= g.inner) {
    for (int j = j0; j < j1; j += kNB) {
      const int c = min(j1, j + kNB);
      factor_panel(g, j, c - j, ipiv, sip, info, code, max_cs);
      if (c >= j1) break;
      trsm_lower_kernel<<<col_grid(j1 - c, g.batch, kTrsmThreads), kTrsmThreads, 0, g.s>>>(
          g.A, g.sA, g.lda, j, c - j, g.A, g.sA, g.lda, c, j1 - c);
      note_launch();
      bgemm(g.n - c, j1 - c, c - j, mone, g.A + (size_t)c * g.lda + j, g.sA, g.lda, g.A + (size_t)j * g.lda + c, g.sA,
            g.lda, one, g.A + (size_t)c * g.lda + c, g.sA, g.lda, g.batch, g.s);
    }
    return;
  }
  const int m = half_of(j0, j1);
  lu_columns(g, j0, m, ipiv, sip, info, code, max_cs);
  lower_solve(g, j0, m, g.A, g.sA, g.lda, m, j1 - m);
  gemm(g.n - m, j1 - m, m - j0, mone, g.A + (size_t)m * g.lda + j0, g.sA, g.lda, g.A + (size_t)j0 * g.lda + m, g.sA,
       g.lda, one, g.A + (size_t)m * g.lda + m, g.sA, g.lda, g.batch, g.rg, g.s);
  lu_columns(g, m, j1, ipiv, sip, info, code, max_cs);
}

// In-place LU with partial pivoting of a batch of n x n matrices (team_getrf's
// arithmetic, spread over CTAs).
inline void getrf_multi(int n, cd *A, long long sA, int lda, int *ipiv, long long sip, int *info, int code,
                        int batch, const RgScratch &rg, cudaStream_t s, int max_cs = kPanelMaxCS) {
  lu_columns(LuArgs{n, A, sA, lda, batch, rg, s, inner_block(n, batch, rg)}, 0, n, ipiv, sip, info, code, max_cs);
}

// X := U^-1 L^-1 X (n x nrhs) from getrf_multi's factors, rows already
// interchanged.
inline void lu_solve_multi(int n, int nrhs, const cd *LU, long long sLU, int lda, cd *B, long long sB, int ldb, int batch,
                           const RgScratch &rg, cudaStream_t s) {
  const LuArgs g{n, const_cast<cd *>(LU), sLU, lda, batch, rg, s, inner_block(n, batch, rg)};
  lower_solve(g, 0, n, B, sB, ldb, 0, nrhs);
  upper_solve(g, 0, n, B, sB, ldb, nrhs);
}

// Solve A X = B in place (B n x nrhs) from getrf_multi's factors.
inline void getrs_multi(int n, int nrhs, const cd *LU, long long sLU, int lda, const int *ipiv, long long sip,
                        cd *B, long long sB, int ldb, int batch, const RgScratch &rg, cudaStream_t s) {
  if (nrhs <= 0) return;
  swap_rows_kernel<<<col_grid(nrhs, batch), 128, 0, s>>>(B, sB, ldb, nrhs, ipiv, sip, n);
  note_launch();
  lu_solve_multi(n, nrhs, LU, sLU, lda, B, sB, ldb, batch, rg, s);
}

}  // namespace
