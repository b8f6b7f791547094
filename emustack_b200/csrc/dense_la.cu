// Batched complex128 GEMM and LU solve entry points (the np.matrix products
// and np.linalg.solve / zgesv calls of backend/stack.py and
// backend/mode_calcs.py, as stand-alone batched kernels).
#include <cuda_runtime.h>

#include "dense_la.cuh"
#include "emu_internal.h"

namespace emu {
int zgesv_two_per_sm(const GesvArgs &g, int batch, void *stream);  // dense_la_two.cu
}

namespace {

using namespace emu;

struct GemmArgs {
  int m, n, k, lda, ldb, ldc;
  long long sA, sB, sC;
  cd alpha, beta;
  const cd *A;
  const cd *B;
  cd *C;
};

__global__ void __launch_bounds__(kDLThreads) zgemm_batched_kernel(GemmArgs g) {
  __shared__ GemmSmem sm;
  const int b = blockIdx.z;
  cta_gemm_tile(g.m, g.n, g.k, g.alpha, g.A + b * g.sA, g.lda, g.B + b * g.sB, g.ldb, g.beta,
                g.C + b * g.sC, g.ldc, blockIdx.y * kTM, blockIdx.x * kTN, sm);
}

__global__ void __launch_bounds__(kDLThreads) zgesv_batched_kernel(GesvArgs g) { team_gesv(g); }

}  // namespace

extern "C" int emu_zgemm_batched(int m, int n, int k, emu_c128 alpha, const emu_c128 *A, int lda,
                                 long long strideA, const emu_c128 *B, int ldb, long long strideB,
                                 emu_c128 beta, emu_c128 *C, int ldc, long long strideC, int batch,
                                 void *stream) {
  if (m < 0 || n < 0 || k < 0 || batch < 0) return EMU_E_SHAPE;
  if (m == 0 || n == 0 || batch == 0) return EMU_OK;
  if (!A || !B || !C || lda < k || ldb < n || ldc < n) return EMU_E_ARG;
  if (batch > 65535) return EMU_E_SHAPE;
  GemmArgs g{m, n, k, lda, ldb, ldc, strideA, strideB, strideC, cd{alpha.re, alpha.im},
             cd{beta.re, beta.im}, (const cd *)A, (const cd *)B, (cd *)C};
  dim3 grid((n + kTN - 1) / kTN, (m + kTM - 1) / kTM, batch);
  zgemm_batched_kernel<<<grid, kDLThreads, 0, (cudaStream_t)stream>>>(g);
  emu::note_launch();
  return emu::check_launch();
}

extern "C" int emu_zgesv_batched(int n, int nrhs, emu_c128 *A, int lda, long long strideA,
                                 int32_t *ipiv, emu_c128 *B, int ldb, long long strideB,
                                 int32_t *info, int batch, void *stream) {
  if (n < 0 || nrhs < 0 || batch < 0) return EMU_E_SHAPE;
  if (n == 0 || batch == 0) return EMU_OK;
  if (!A || !ipiv || (nrhs > 0 && !B) || lda < n || (nrhs > 0 && ldb < nrhs)) return EMU_E_ARG;
  GesvArgs g{n, nrhs, lda, ldb, strideA, strideB, (cd *)A, (cd *)B, (int *)ipiv, (int *)info};
  // two systems per SM where they fit, from more systems than SMs on
  if (batch > emu::sm_count() && 2 * (team_smem(n) + 1024) <= 227 * 1024) return zgesv_two_per_sm(g, batch, stream);
  if (launch_team(zgesv_batched_kernel, batch, team_size(batch, n, emu::sm_count()), team_smem(n),
                  (cudaStream_t)stream, g) != cudaSuccess)
    return EMU_E_CUDA;
  emu::note_launch();
  return emu::check_launch();
}
