// The INT8 GEMMs of the residue-arithmetic complex GEMM (residue_gemm.cuh)
// on the 5th-generation tensor cores.
//
// A persistent kernel: each CTA (one per SM) takes work units (problem, K
// split, modulus or magnitudes, 128-row tile of A, up to 128-row tile of B) round-robin,
// tiles fastest, so that the CTAs of one modulus read the same planes at the
// same time and share them through L2.  192 threads:
//   warp 0 (one lane) streams K stages of 128 bytes by TMA (128-byte swizzle):
//     both planes of A (2 x 128 rows) and the three planes of B;
//   warp 1 (one lane) issues, per 32 bytes of K, two tcgen05.mma kind::i8 of
//     M = 128, N = 2 nt into one accumulator [Cr | Ci]:
//     Ar x [Br | Bi] and Ai x [-Bi | Br]
//     (kind::f8f6f4 with FP32 sums for the magnitudes' planes);
//   warps 2-5 read the finished accumulator (tcgen05.ld), reduce it modulo p
//     and store signed bytes.  Two accumulators of 256 TMEM columns, so that
//     this overlaps the next unit's products.
// Every mbarrier wait is bounded.
#include <cuda.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include "dense_la.cuh"
#include "residue_gemm.cuh"

namespace {

using namespace emu;

constexpr int kThreads = 192;
constexpr int kStages = 3;
constexpr int kABytes = kRgPlanesA * kRgTileM * kRgStageK;  // 32 KB
constexpr uint32_t kTmemCols = 512;
constexpr long long kWaitLimit = 1ll << 26;

struct MmaArgs {
  int mtiles, ntiles, nt, kp, kper, nsplit, units, m, n, ldn, add;
  uint8_t *C;
  int *err;
};

struct Maps {
  CUtensorMap a, b;
};

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// K-major operand in the 128-byte swizzled layout: rows of 128 B, 8-row atoms
// of 1024 B, version 1, layout SWIZZLE_128B
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr) {
  return (uint64_t)((saddr >> 4) & 0x3FFF) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) |
         (2ull << 61);
}

__device__ __forceinline__ void mma_i8(uint32_t d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t"
      "}\n" ::"r"(d),
      "l"(da), "l"(db), "r"(idesc), "r"(acc));
}

// the same on e5m2 operands with FP32 accumulation
__device__ __forceinline__ void mma_f8(uint32_t d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t"
      "}\n" ::"r"(d),
      "l"(da), "l"(db), "r"(idesc), "r"(acc));
}

__device__ __forceinline__ void mma_commit(uint32_t mbar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar)
               : "memory");
}

__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t phase) {
  for (long long i = 0; i < kWaitLimit; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n\t"
        ".reg .pred P1;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, P1;\n\t"
        "}\n"
        : "=r"(ok)
        : "r"(mbar), "r"(phase)
        : "memory");
    if (ok) return true;
  }
  return false;
}

__device__ __forceinline__ void mbar_init(uint32_t mbar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(mbar), "r"(count));
}

__device__ __forceinline__ void mbar_arrive(uint32_t mbar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(mbar) : "memory");
}

__device__ __forceinline__ void tma_load(uint32_t dst, const CUtensorMap *map, int x, int y, int z, uint32_t mbar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(dst), "l"((uint64_t)map), "r"(mbar), "r"(x), "r"(y), "r"(z)
      : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, int *v) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
        "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr));
}

// Waits for the loads above; the registers are valid after it.
__device__ __forceinline__ void tmem_wait(int (&v)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) asm volatile("" : "+r"(v[i]));
}

struct Unit {
  int m0, n0, mod, split, prob;
};

__device__ __forceinline__ Unit decode(const MmaArgs &a, int u) {
  Unit r;
  r.n0 = (u % a.ntiles) * a.nt;
  u /= a.ntiles;
  r.m0 = (u % a.mtiles) * kRgTileM;
  u /= a.mtiles;
  r.mod = u % kRgSlots;
  u /= kRgSlots;
  r.split = u % a.nsplit;
  r.prob = u / a.nsplit;
  return r;
}

__device__ __forceinline__ int unit_stages(const MmaArgs &a, const Unit &u) {
  const int kb = u.split * a.kper, ke = min(a.kp, kb + a.kper);
  return (ke - kb + kRgStageK - 1) / kRgStageK;
}

__global__ void __launch_bounds__(kThreads, 1) rg_mma_kernel(const __grid_constant__ Maps maps, MmaArgs a) {
  extern __shared__ __align__(16) unsigned char sm_raw[];
  __shared__ uint64_t bars[2 * kStages + 5];
  __shared__ uint32_t tslot;
  const uint32_t raw = smem_u32(sm_raw), buf = (raw + 1023u) & ~1023u;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t bbytes = (uint32_t)(kRgPlanesB * a.nt * kRgStageK), stage_bytes = kABytes + bbytes;
  const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + kStages), accf0 = smem_u32(bars + 2 * kStages),
                 acce0 = smem_u32(bars + 2 * kStages + 2), done = smem_u32(bars + 2 * kStages + 4);
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tslot)),
                 "r"(kTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  if (tid == 0) {
    for (int i = 0; i < kStages; ++i) {
      mbar_init(full0 + 8 * i, 1);
      mbar_init(empty0 + 8 * i, 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(accf0 + 8 * i, 1);
      mbar_init(acce0 + 8 * i, 128);
    }
    mbar_init(done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tslot;
  bool ok = true;
  int t = 0;
  if (warp == 0) {
    if (lane == 0) {
      for (int u = blockIdx.x; u < a.units && ok; u += gridDim.x) {
        const Unit w = decode(a, u);
        const int ns = unit_stages(a, w), za = kRgPlanesA * (w.prob * kRgSlots + w.mod),
                  zb = kRgPlanesB * (w.prob * kRgSlots + w.mod);
        for (int j = 0; j < ns; ++j, ++t) {
          const int b = t % kStages;
          if (t >= kStages && !mbar_wait(empty0 + 8 * b, (uint32_t)((t / kStages - 1) & 1))) {
            ok = false;
            break;
          }
          const uint32_t fb = full0 + 8 * b, base = buf + (uint32_t)b * stage_bytes;
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(fb), "r"(stage_bytes)
                       : "memory");
          const int x = w.split * a.kper + j * kRgStageK;
          tma_load(base, &maps.a, x, w.m0, za, fb);
          tma_load(base + kABytes, &maps.b, x, w.n0, zb, fb);
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      // D S32 (2), A and B signed 8-bit (1), K-major, N >> 3 at bit 17, M >> 4 at bit 24
      const uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(2 * a.nt >> 3) << 17) |
                             ((uint32_t)(kRgTileM >> 4) << 24);
      // D F32 (1), A and B e5m2 (1), the rest alike
      const uint32_t idesc8 = idesc - (1u << 4);
      int c = 0;
      for (int u = blockIdx.x; u < a.units && ok; u += gridDim.x, ++c) {
        const Unit w = decode(a, u);
        const int ns = unit_stages(a, w), ab = c & 1;
        if (c >= 2 && !mbar_wait(acce0 + 8 * ab, (uint32_t)((c / 2 - 1) & 1))) {
          ok = false;
          break;
        }
        const uint32_t d = tmem + (uint32_t)ab * 256;
        for (int j = 0; j < ns; ++j, ++t) {
          const int b = t % kStages;
          if (!mbar_wait(full0 + 8 * b, (uint32_t)((t / kStages) & 1))) {
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t ar = buf + (uint32_t)b * stage_bytes, ai = ar + kRgTileM * kRgStageK;
          const uint32_t nb = ar + kABytes, pb = nb + (uint32_t)(a.nt * kRgStageK);  // [-Bi Br Bi]
#pragma unroll
          for (int k = 0; k < kRgStageK / 32; ++k) {
            const uint32_t first = (j == 0 && k == 0) ? 0u : 1u;
            if (w.mod < kRgMods) {
              mma_i8(d, smem_desc(ar + 32 * k), smem_desc(pb + 32 * k), idesc, first);
              mma_i8(d, smem_desc(ai + 32 * k), smem_desc(nb + 32 * k), idesc, 1u);
            } else {
              mma_f8(d, smem_desc(ar + 32 * k), smem_desc(pb + 32 * k), idesc8, first);
              mma_f8(d, smem_desc(ai + 32 * k), smem_desc(nb + 32 * k), idesc8, 1u);
            }
          }
          mma_commit(empty0 + 8 * b);
        }
        if (!ok) break;
        mma_commit(accf0 + 8 * ab);
      }
      mma_commit(done);  // covers every MMA issued, also when a wait gave up
    }
  } else {
    const int q = warp & 3;  // the TMEM lane quarter this warp may read
    int c = 0;
    for (int u = blockIdx.x; u < a.units; u += gridDim.x, ++c) {
      const Unit w = decode(a, u);
      const int ab = c & 1, row = w.m0 + q * 32 + lane;
      if (!__all_sync(0xffffffffu, mbar_wait(accf0 + 8 * ab, (uint32_t)((c / 2) & 1)))) {
        ok = false;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t ta = tmem + (uint32_t)ab * 256 + ((uint32_t)(q * 32) << 16);
      uint8_t *Cz = a.C + ((long long)((w.prob * a.nsplit + w.split) * kRgSlots + w.mod) * 2) * a.m * a.ldn;
      const bool some = unit_stages(a, w) > 0;  // a split without K: nothing was accumulated
      // two chunks of 16 columns at a time; columns [0, nt) are Re C, [nt, 2 nt) Im C.
      // byte(y, prev): what is stored for the sum y over the byte that was there.  The
      // two kinds have loops of their own: this is on the critical path of shallow
      // products (interfaces of P = 634, M = 400: 0.8 ms against 2.4 ms with both in one)
      const int nch = 2 * a.nt / 16;
      auto drain = [&](auto &&byte) {
        for (int h0 = 0; h0 < nch; h0 += 2) {
          int v[32];
          tmem_ld16(ta + 16u * h0, v);
          tmem_ld16(ta + 16u * (h0 + 1), v + 16);
          tmem_wait(v);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int cc = 16 * (h0 + h), pl = cc >= a.nt, col = w.n0 + cc - pl * a.nt;
            const bool in = row < a.m && col < a.ldn;
            uint4 *dst = (uint4 *)(Cz + ((long long)pl * a.m + row) * a.ldn + col);
            uint4 prev = make_uint4(0, 0, 0, 0);
            if (a.add && in) prev = *dst;
            const uint32_t pv[4] = {prev.x, prev.y, prev.z, prev.w};
            uint32_t o[4];
#pragma unroll
            for (int g = 0; g < 4; ++g) {
              uint32_t r[4];
#pragma unroll
              for (int e = 0; e < 4; ++e) r[e] = byte(some ? v[16 * h + 4 * g + e] : 0, pv[g] >> (8 * e));
              o[g] = rg_pack4(r[0], r[1], r[2], r[3]);
            }
            if (in) *dst = make_uint4(o[0], o[1], o[2], o[3]);
          }
        }
      };
      if (w.mod < kRgMods) {
        const int p = c_rg.p[w.mod], c16 = c_rg.c16[w.mod];
        const float ip = c_rg.invp[w.mod];
        drain([&](int y, uint32_t prev) -> uint32_t {
          // y = yh 2^16 + yl; yh (2^16 mod p) + yl on the pattern of 1.5 x 2^23
          const int s = (y >> 16) * c16 + ((y & 0xffff) | 0x4B400000) + (int)(int8_t)prev;
          const float f = __int_as_float(s) - 12582912.0f;
          const int qq = __float_as_int(fmaf(f, ip, 12582912.0f));
          return (uint32_t)(s - qq * p);
        });
      } else {
        drain([&](int y, uint32_t prev) -> uint32_t {
          return rg_code(__int_as_float(y) + rg_uncode(prev & 0xffu));
        });
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      mbar_arrive(acce0 + 8 * ab);
    }
  }
  __syncwarp();
  const bool all_ok = __syncthreads_and(ok) != 0;
  if (!all_ok && tid == 0) {
    atomicExch(a.err, 1);
    // a wait gave up: the copies still in flight land before the CTA leaves
    for (int j = max(0, t - kStages); j < t; ++j) mbar_wait(full0 + 8 * (j % kStages), (uint32_t)((j / kStages) & 1));
  }
  if (tid == 0 && !mbar_wait(done, 0)) atomicExch(a.err, 1);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols));
}

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static const PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      p = nullptr;
    return (PFN_cuTensorMapEncodeTiled_v12000)p;
  }();
  return fn;
}

bool make_map(CUtensorMap *m, const uint8_t *ptr, int kp, int rows, long long planes, int box_rows, int box_planes) {
  auto fn = encode_fn();
  if (!fn) return false;
  const cuuint64_t dims[3] = {(cuuint64_t)kp, (cuuint64_t)rows, (cuuint64_t)planes};
  const cuuint64_t strides[2] = {(cuuint64_t)kp, (cuuint64_t)kp * (cuuint64_t)rows};
  const cuuint32_t box[3] = {(cuuint32_t)kRgStageK, (cuuint32_t)box_rows, (cuuint32_t)box_planes};
  const cuuint32_t estr[3] = {1, 1, 1};
  return fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, (void *)ptr, dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// ---------------------------------------------------------------- dense operands
struct DenseArgs {
  RgDense g;
  int r0, mr;  // rows of A in this pass
  int kp, rblocks;
  RgScale *sa, *sb;  // [batch][mr], [batch][n]
  int *ka, *kb;      // k of the only non-zero value of a row of A, a column of B; -1: not one
  uint8_t *A, *B;
  int *flags;        // [batch][64 x 64 tiles]: the tile holds entries left to FP64 sums
};
__host__ __device__ inline int tiles64(int n) { return (n + 63) / 64; }

// Scales of both operands, one launch: the first `rblocks` blocks of a problem
// take 32 rows of A each (one per warp), the others 32 columns of B.  The first
// block also clears the problem's tile flags.
__global__ void __launch_bounds__(1024) dense_scale_kernel(DenseArgs a) {
  __shared__ double red[2][32][33];
  __shared__ int redi[2][32][33];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long b = blockIdx.y;
  const RgDense &g = a.g;
  if (blockIdx.x == 0) {
    const int tiles = tiles64(a.mr) * tiles64(g.n);
    for (int i = threadIdx.x; i < tiles; i += blockDim.x) a.flags[b * tiles + i] = 0;
  }
  double ss = 0.0, mx = 0.0;
  int cnt = 0, at = -1;  // non-zero values, and the last one's k
  auto add = [&](cd x, int k) {
    ss += fma(x.x, x.x, x.y * x.y);
    mx = fmax(mx, fmax(fabs(x.x), fabs(x.y)));
    if (!cis_zero(x)) {
      ++cnt;
      at = k;
    }
  };
  const bool rows = (int)blockIdx.x < a.rblocks;
  const int r = blockIdx.x * 32 + w, c = (blockIdx.x - a.rblocks) * 32 + lane;
  if (rows) {
    const cd *row = g.A + b * g.sA + (size_t)(a.r0 + r) * g.lda, *d = g.dA ? g.dA + b * g.sdA : nullptr;
    if (r < a.mr)
      for (int k = lane; k < g.k; k += 32) add(d ? cmul(row[k], d[k]) : row[k], k);
  } else {
    const cd *B = g.B + b * g.sB;
    if (c < g.n)
      for (int k = w; k < g.k; k += 32) add(B[(size_t)k * g.ldb + c], k);
    // the column's parts to one warp
    red[0][lane][w] = ss;
    red[1][lane][w] = mx;
    redi[0][lane][w] = cnt;
    redi[1][lane][w] = at;
    __syncthreads();
    ss = red[0][w][lane];
    mx = red[1][w][lane];
    cnt = redi[0][w][lane];
    at = redi[1][w][lane];
  }
  for (int o = 16; o; o >>= 1) {
    ss += __shfl_xor_sync(0xffffffffu, ss, o);
    mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  }
  cnt = __reduce_add_sync(0xffffffffu, cnt);
  at = __reduce_max_sync(0xffffffffu, at);
  if (lane) return;
  const int cw = (blockIdx.x - a.rblocks) * 32 + w;
  if (cnt != 1) at = -1;
  if (rows && r < a.mr) {
    a.sa[b * a.mr + r] = rg_scale(mx, ss);
    a.ka[b * a.mr + r] = at;
  }
  if (!rows && cw < g.n) {
    a.sb[b * g.n + cw] = rg_scale(mx, ss);
    a.kb[b * g.n + cw] = at;
  }
}

constexpr int kDcCols = 32, kDcK = 128;
constexpr int kDcRow = kDcK + kDcK / 8 + 1;  // padded so that runs of 8 k and neighbouring columns differ in bank
constexpr size_t kDcSmem = (size_t)kDcCols * kDcRow * sizeof(cd);

// Residues of both operands: tiles of 32 rows of A (blocks below `rblocks` of
// a problem) or 32 columns of B by 128 k (.y), staged in shared memory, 8
// consecutive k of a row or column per thread.
__global__ void __launch_bounds__(256) dense_residue_kernel(DenseArgs a) {
  extern __shared__ __align__(16) unsigned char dc_smem[];
  cd *v = (cd *)dc_smem;  // [row or column][kDcRow]
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long b = blockIdx.z;
  const RgDense &g = a.g;
  const int k0 = blockIdx.y * kDcK;
  const bool rows = (int)blockIdx.x < a.rblocks;
  const int i0 = 32 * (rows ? (int)blockIdx.x : (int)blockIdx.x - a.rblocks), ni = rows ? a.mr : g.n;
  if (rows) {
    const cd *d = g.dA ? g.dA + b * g.sdA : nullptr;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = i0 + w + 8 * i;
      const cd *row = g.A + b * g.sA + (size_t)(a.r0 + r) * g.lda + k0;
#pragma unroll
      for (int j = 0; j < kDcK / 32; ++j) {
        const int k = lane + 32 * j;
        cd x = cd{0.0, 0.0};
        if (r < ni && k0 + k < g.k) x = d ? cmul(row[k], d[k0 + k]) : row[k];
        v[(w + 8 * i) * kDcRow + k + (k >> 3)] = x;
      }
    }
  } else {
    const cd *B = g.B + b * g.sB + (size_t)k0 * g.ldb + i0 + lane;
#pragma unroll
    for (int i = 0; i < kDcK / 8; ++i) {
      const int k = w + 8 * i;
      v[lane * kDcRow + k + (k >> 3)] =
          (i0 + lane < ni && k0 + k < g.k) ? B[(size_t)k * g.ldb] : cd{0.0, 0.0};
    }
  }
  __syncthreads();
  const RgScale *sc = rows ? a.sa + b * a.mr : a.sb + b * g.n;
  const long long plane = (long long)ni * a.kp;
#pragma unroll
  for (int i = threadIdx.x; i < kDcCols * kDcK / 8; i += 256) {
    const int word = i % (kDcK / 8), ii = i / (kDcK / 8);
    if (i0 + ii >= ni) continue;
    const double up = sc[i0 + ii].up;
    cd x[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] = up != 0.0 ? v[ii * kDcRow + 9 * word + j] : cd{0.0, 0.0};
    const long long off = (long long)(i0 + ii) * a.kp + k0 + 8 * word;
    if (rows) rg_store<kRgPlanesA, 2>(x, up, a.A + b * kRgSlots * kRgPlanesA * plane + off, plane);
    else rg_store<kRgPlanesB, 2>(x, up, a.B + b * kRgSlots * kRgPlanesB * plane + off, plane);
  }
}

// How an entry is computed.  Without a safe scale of its row of A or column of B:
// as an FP64 sum.  If a component's sum of magnitudes is too small for residues: as
// the one product there is, if the row or the column has one non-zero value (a
// diagonal operand, as the reflection of a film substrate), else as an FP64 sum.
enum { kResidues, kProduct, kSum };
__device__ __forceinline__ int dense_way(uint32_t cr, uint32_t ci, double da, double db, int ka, int kb) {
  if (da < 0.0 || db < 0.0) return kSum;
  if (!rg_unsafe(rg_uncode(cr)) && !rg_unsafe(rg_uncode(ci))) return kResidues;
  return ka >= 0 || kb >= 0 ? kProduct : kSum;
}

// C = alpha (integer product, scaled back) + beta C: a thread takes four
// columns of one row.  Entries left to FP64 sums are not touched; their tile is
// flagged.
__global__ void __launch_bounds__(128) dense_crt_kernel(DenseArgs a, const uint8_t *R, int ldn, const int *err) {
  const RgDense &g = a.g;
  const long long b = blockIdx.y, i = blockIdx.x * 128LL + threadIdx.x, plane = (long long)a.mr * ldn;
  const int words = (g.n + 3) / 4;
  if (i >= (long long)a.mr * words) return;
  const int r = (int)(i / words), c0 = (int)(i % words) * 4;
  const double da = a.sa[b * a.mr + r].down;
  const int ka = a.ka[b * a.mr + r];
  const uint8_t *src = R + b * kRgSlots * 2 * plane + (long long)r * ldn + c0;
  cd out[4];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    uint32_t q[kRgMods];
#pragma unroll
    for (int m = 0; m < kRgMods; ++m) q[m] = *(const uint32_t *)(src + (2 * m + h) * plane) ^ 0x80808080u;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const double x = da * rg_crt([&](auto i) { return (q[decltype(i)::value] >> (8 * j)) & 0xffu; }, 128u);
      if (h == 0) out[j].x = x;
      else out[j].y = x;
    }
  }
  const bool failed = *err != 0, zero_beta = g.beta.x == 0.0 && g.beta.y == 0.0;
  const uint32_t sr = *(const uint32_t *)(src + 2 * kRgMods * plane),
                 si = *(const uint32_t *)(src + (2 * kRgMods + 1) * plane);
  bool left = false;
  cd *C = g.C + b * g.sC + (size_t)(a.r0 + r) * g.ldc + c0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    if (c0 + j >= g.n) break;
    const double db = a.sb[b * g.n + c0 + j].down;
    cd x = cscale(out[j], db);
    const int kb = a.kb[b * g.n + c0 + j];
    const int way = dense_way((sr >> (8 * j)) & 0xffu, (si >> (8 * j)) & 0xffu, da, db, ka, kb);
    if (failed) {
      x = cd{nan(""), nan("")};
    } else if (way == kProduct) {
      const int k = ka >= 0 ? ka : kb;
      x = g.A[b * g.sA + (size_t)(a.r0 + r) * g.lda + k];
      if (g.dA) x = cmul(x, g.dA[b * g.sdA + k]);
      x = cmul(x, g.B[b * g.sB + (size_t)k * g.ldb + c0 + j]);
    } else if (way == kSum) {
      left = true;
      continue;
    }
    x = cmul(g.alpha, x);
    C[j] = zero_beta ? x : cadd(x, cmul(g.beta, C[j]));
  }
  if (left) a.flags[b * tiles64(a.mr) * tiles64(g.n) + r / 64 * tiles64(g.n) + c0 / 64] = 1;
}

__device__ __forceinline__ void dense_left_tile(const DenseArgs &a, const uint8_t *R, int ldn, int t, GemmSmem &sm) {
  const RgDense &g = a.g;
  const int tn = tiles64(g.n), tm = tiles64(a.mr), c0 = t % tn * 64, r0 = t / tn % tm * 64;
  const long long b = t / tn / tm;
  const cd *A = g.A + b * g.sA + (size_t)a.r0 * g.lda, *B = g.B + b * g.sB, *d = g.dA ? g.dA + b * g.sdA : nullptr;
  const bool zero_beta = g.beta.x == 0.0 && g.beta.y == 0.0;
  const long long plane = (long long)a.mr * ldn;
  const uint8_t *S = R + (b * kRgSlots + kRgMods) * 2 * plane;
  cd *C = g.C + b * g.sC + (size_t)a.r0 * g.ldc;
  cta_tile<64, false>(
      g.k,
      [&](int r, int k) {
        cd v = r0 + r < a.mr ? A[(size_t)(r0 + r) * g.lda + k] : cd{0.0, 0.0};
        if (d && r0 + r < a.mr) v = cmul(v, d[k]);
        return v;
      },
      [&](int k, int c) { return c0 + c < g.n ? B[(size_t)k * g.ldb + c0 + c] : cd{0.0, 0.0}; },
      [&](int r, int c, cd x) {
        r += r0;
        c += c0;
        if (r >= a.mr || c >= g.n) return;
        const uint8_t *s = S + (long long)r * ldn + c;
        if (dense_way(s[0], s[plane], a.sa[b * a.mr + r].down, a.sb[b * g.n + c].down, a.ka[b * a.mr + r],
                      a.kb[b * g.n + c]) != kSum)
          return;
        x = cmul(g.alpha, x);
        cd *p = C + (size_t)r * g.ldc + c;
        *p = zero_beta ? x : cadd(x, cmul(g.beta, *p));
      },
      sm);
}

// The flagged tiles again in FP64, for the entries left over.
__global__ void __launch_bounds__(kDLThreads) dense_left_kernel(DenseArgs a, const uint8_t *R, int ldn, int tiles) {
  __shared__ GemmSmem sm;
  for (int t0 = blockIdx.x; t0 < tiles; t0 += kDLThreads * gridDim.x) {
    const int mine = t0 + (int)threadIdx.x * gridDim.x;  // most often no tile is flagged
    if (!__syncthreads_or(mine < tiles && a.flags[mine])) continue;
    for (int i = 0, t = t0; i < kDLThreads && t < tiles; ++i, t += gridDim.x)
      if (a.flags[t]) dense_left_tile(a, R, ldn, t, sm);
  }
}

// Deeper products are summed over chunks of this depth in FP64, which bounds
// B's planes (51 bytes per value of B)
constexpr int kDenseDepth = 2048;
constexpr size_t kDenseBytes = (size_t)192 << 20;

struct DenseShape {
  long long kp, ldn, bytesB, perrow;  // bytes of one problem's B, of one row of A with its results
};

DenseShape dense_shape(int n, int k) {
  DenseShape d;
  if (k > kDenseDepth) k = kDenseDepth;
  d.kp = (k + kRgStageK - 1) / kRgStageK * kRgStageK;
  d.ldn = (n + 15) / 16 * 16;
  const long long scale = sizeof(RgScale) + sizeof(int);
  d.bytesB = (long long)kRgSlots * kRgPlanesB * n * d.kp + scale * n;
  d.perrow = (long long)kRgSlots * kRgPlanesA * d.kp + (long long)kRgSlots * 2 * d.ldn + scale +
             (long long)sizeof(int) * tiles64(n);  // flags: enough for a row of tiles each
  return d;
}

constexpr size_t kDenseSlack = 11 * 256;

size_t smem_bytes(int nt) { return (size_t)kStages * (kABytes + kRgPlanesB * nt * kRgStageK) + 1024; }

}  // namespace

namespace emu {

RgPlan rg_plan(int m, int n, int k, int batch, int nsplit) {
  RgPlan p{};
  p.m = m;
  p.n = n;
  p.k = k;
  p.batch = batch;
  p.kp = (k + kRgStageK - 1) / kRgStageK * kRgStageK;
  p.mtiles = (m + kRgTileM - 1) / kRgTileM;
  // three stages fit in shared memory up to 112 rows of B; equal tiles
  p.ntiles = (n + 111) / 112;
  p.nt = ((n + p.ntiles - 1) / p.ntiles + 15) / 16 * 16;
  p.ldn = (n + 15) / 16 * 16;
  // K splits: enough units of one problem for about four waves, each at least 2048
  // deep (by the problem alone: the magnitudes' sums depend on them)
  const long long tiles = (long long)p.mtiles * p.ntiles * kRgSlots;
  long long ns = (4LL * sm_count() + tiles - 1) / tiles;
  const long long most = p.kp / 2048 > 0 ? p.kp / 2048 : 1;
  if (ns > most) ns = most;
  if (ns > kRgMaxSplits) ns = kRgMaxSplits;
  const long long need = (p.kp + kRgMaxK - 1) / kRgMaxK;
  if (ns < need) ns = need;
  if (nsplit > 0) ns = nsplit;
  p.kper = (int)(((p.kp + ns - 1) / ns + kRgStageK - 1) / kRgStageK * kRgStageK);
  p.nsplit = nsplit > 0 ? nsplit : (p.kp + p.kper - 1) / p.kper;
  p.bytesA = (long long)batch * kRgSlots * kRgPlanesA * m * p.kp;
  p.bytesB = (long long)batch * kRgSlots * kRgPlanesB * n * p.kp;
  p.bytesC = (long long)batch * p.nsplit * kRgSlots * 2 * m * p.ldn;
  return p;
}

int rg_mma(const RgPlan &p, const uint8_t *A, const uint8_t *B, uint8_t *C, bool add, int *err, cudaStream_t s) {
  if (((uintptr_t)A | (uintptr_t)B | (uintptr_t)C) & 15) return EMU_E_ARG;
  Maps maps;
  if (!make_map(&maps.a, A, p.kp, p.m, (long long)p.batch * kRgSlots * kRgPlanesA, kRgTileM, kRgPlanesA) ||
      !make_map(&maps.b, B, p.kp, p.n, (long long)p.batch * kRgSlots * kRgPlanesB, p.nt, kRgPlanesB))
    return EMU_E_CUDA;
  MmaArgs a;
  a.mtiles = p.mtiles;
  a.ntiles = p.ntiles;
  a.nt = p.nt;
  a.kp = p.kp;
  a.kper = p.kper;
  a.nsplit = p.nsplit;
  a.units = p.batch * p.nsplit * kRgSlots * p.mtiles * p.ntiles;
  a.m = p.m;
  a.n = p.n;
  a.ldn = p.ldn;
  a.add = add;
  a.C = C;
  a.err = err;
  // the limit is set to its largest value, so that threads launching other
  // tile sizes at once never see a smaller one
  if (cudaFuncSetAttribute(rg_mma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes(112)) !=
      cudaSuccess)
    return EMU_E_CUDA;
  const int grid = a.units < sm_count() ? a.units : sm_count();
  rg_mma_kernel<<<grid, kThreads, smem_bytes(p.nt), s>>>(maps, a);
  note_launch();
  return check_launch();
}

size_t rg_dense_scratch(int m, int n, int k, int batch) {
  if (m < 1 || n < 1 || k < 1 || batch < 1) return 0;
  const DenseShape d = dense_shape(n, k);
  const size_t whole = (size_t)(d.bytesB + (long long)m * d.perrow);
  if (whole <= kDenseBytes) {
    const size_t g = kDenseBytes / whole;
    return whole * (g < (size_t)batch ? g : (size_t)batch) + kDenseSlack;
  }
  long long rows = ((long long)kDenseBytes - d.bytesB) / d.perrow / kRgTileM * kRgTileM;
  if (rows < 4 * kRgTileM) rows = 4 * kRgTileM;
  if (rows > m) rows = m;
  return (size_t)(d.bytesB + rows * d.perrow) + kDenseSlack;
}

int rg_dense(const RgDense &g, void *ws, size_t bytes, cudaStream_t s) {
  if (g.m <= 0 || g.n <= 0 || g.batch <= 0) return EMU_OK;
  if (g.k < 1) return EMU_E_SHAPE;
  if ((uintptr_t)ws & 255) return EMU_E_ARG;
  if (g.k > kDenseDepth) {
    const int nc = (g.k + kDenseDepth - 1) / kDenseDepth;
    const int kc = ((g.k + nc - 1) / nc + kRgStageK - 1) / kRgStageK * kRgStageK;  // <= kDenseDepth
    for (int k0 = 0; k0 < g.k; k0 += kc) {
      RgDense c = g;
      c.k = g.k - k0 < kc ? g.k - k0 : kc;
      c.A += k0;
      c.B += (size_t)k0 * g.ldb;
      if (c.dA) c.dA += k0;
      if (k0) c.beta = cd{1.0, 0.0};
      const int st = rg_dense(c, ws, bytes, s);
      if (st != EMU_OK) return st;
    }
    return EMU_OK;
  }
  const DenseShape d = dense_shape(g.n, g.k);
  if (bytes < kDenseSlack) return EMU_E_WORKSPACE;
  const long long room = (long long)(bytes - kDenseSlack), whole = d.bytesB + g.m * d.perrow;
  long long group = room / whole, rows = g.m;
  if (group < 1) {
    group = 1;
    rows = (room - d.bytesB) / d.perrow / kRgTileM * kRgTileM;
    if (rows < kRgTileM) return EMU_E_WORKSPACE;
    // equal passes
    const long long np = (g.m + rows - 1) / rows;
    rows = ((g.m + np - 1) / np + kRgTileM - 1) / kRgTileM * kRgTileM;
  }
  if (group > g.batch) group = g.batch;
  char *w = (char *)ws;
  auto take = [&](long long n) {
    char *r = w;
    w += align_up((size_t)n, 256);
    return (void *)r;
  };
  int *err = (int *)take(256);
  DenseArgs a;
  a.kp = (int)d.kp;
  a.sa = (RgScale *)take((long long)sizeof(RgScale) * rows * group);
  a.sb = (RgScale *)take((long long)sizeof(RgScale) * g.n * group);
  a.ka = (int *)take((long long)sizeof(int) * rows * group);
  a.kb = (int *)take((long long)sizeof(int) * g.n * group);
  a.A = (uint8_t *)take((long long)kRgSlots * kRgPlanesA * rows * d.kp * group);
  a.B = (uint8_t *)take((long long)kRgSlots * kRgPlanesB * g.n * d.kp * group);
  uint8_t *R = (uint8_t *)take((long long)kRgSlots * 2 * rows * d.ldn * group);
  a.flags = (int *)take((long long)sizeof(int) * tiles64((int)rows) * tiles64(g.n) * group);
  if (cudaMemsetAsync(err, 0, sizeof(int), s) != cudaSuccess) return EMU_E_CUDA;
  if (cudaFuncSetAttribute(dense_residue_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDcSmem) !=
      cudaSuccess)
    return EMU_E_CUDA;
  for (long long b0 = 0; b0 < g.batch; b0 += group) {
    const int nb = (int)(g.batch - b0 < group ? g.batch - b0 : group);
    a.g = g;
    a.g.batch = nb;
    a.g.A += b0 * g.sA;
    a.g.B += b0 * g.sB;
    a.g.C += b0 * g.sC;
    if (g.dA) a.g.dA += b0 * g.sdA;
    for (int r0 = 0; r0 < g.m; r0 += (int)rows) {
      a.r0 = r0;
      a.mr = (int)(g.m - r0 < rows ? g.m - r0 : rows);
      a.rblocks = (a.mr + 31) / 32;
      const int cblocks = r0 == 0 ? (g.n + 31) / 32 : 0;  // B's residues serve all passes
      dense_scale_kernel<<<dim3(a.rblocks + cblocks, nb), 1024, 0, s>>>(a);
      dense_residue_kernel<<<dim3(a.rblocks + cblocks, a.kp / kDcK, nb), 256, kDcSmem, s>>>(a);
      note_launch(2);
      const RgPlan p = rg_plan(a.mr, g.n, g.k, nb, 1);
      const int st = rg_mma(p, a.A, a.B, R, false, err, s);
      if (st != EMU_OK) return st;
      const long long items = (long long)a.mr * ((g.n + 3) / 4);
      dense_crt_kernel<<<dim3((unsigned)((items + 127) / 128), nb), 128, 0, s>>>(a, R, p.ldn, err);
      const int tiles = tiles64(g.n) * tiles64(a.mr) * nb, two = 2 * sm_count();
      dense_left_kernel<<<tiles < two ? tiles : two, kDLThreads, 0, s>>>(a, R, p.ldn, tiles);
      note_launch(2);
    }
  }
  return check_launch();
}

}  // namespace emu
