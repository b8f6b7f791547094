// Batched LU solves with half of the registers, two CTAs per SM.  A file of its own:
// the team routines are called, not inlined, and a kernel's register limit would hold
// for every other caller in its file.
//
// Small systems are chains of barriers and global round trips, so a second CTA on
// the SM pays more than the spills cost.  4 000 systems of n unknowns and n right-hand
// sides, one / two CTAs per SM: n = 8 448 / 276 us, 20 1 301 / 771 us, 40 3 750 / 2 360
// us, 58 5 110 / 3 770 us, 100 14.3 / 10.9 ms; up to as many systems as SMs one CTA wins
// (148 of n = 100 460 / 594 us), and from n of about 115 on two do not fit.
#include <cuda_runtime.h>

#include "dense_la.cuh"
#include "emu_internal.h"

namespace {

using namespace emu;

__global__ void __launch_bounds__(kDLThreads, 2) zgesv_two_kernel(GesvArgs g) { team_gesv(g); }

}  // namespace

namespace emu {

int zgesv_two_per_sm(const GesvArgs &g, int batch, void *stream) {
  if (launch_team(zgesv_two_kernel, batch, 1, team_smem(g.n), (cudaStream_t)stream, g) != cudaSuccess) return EMU_E_CUDA;
  note_launch();
  return check_launch();
}

}  // namespace emu
