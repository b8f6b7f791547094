// Electric fields from the GSM amplitudes (vec_coef_down / vec_coef_up of a
// solved stack):
//
//  * plane-wave basis inside a homogeneous layer: the ThinFilm branch of
//    fields_in_plane (backend/plotting.py:1759-1833) and field_values
//    (backend/plotting.py:2857-2996).  For the orders s of the layer (sorted
//    by the air reference's order) with alpha_s, beta_s, gamma_s = k_z,s and
//    index n:
//        norm = sqrt(alpha^2 + beta^2),  k = sqrt(alpha^2 + beta^2 + gamma^2)
//        chi_TE = sqrt(n gamma / k),     chi_TM = sqrt(n k / gamma)
//        e_TE = (beta, -alpha, 0) / norm, e_TM = (alpha / norm, beta / norm,
//        -norm / gamma)
//        eta_{TE,TM} = c_{TE,TM} e_{TE,TM} / chi_{TE,TM}   (c: the amplitude)
//        E(x, y, z) = sum_s eta_down exp(i(alpha x + beta y - gamma (z1 - h)))
//                         + eta_up   exp(i(alpha x + beta y + gamma z1))
//    with z1 = -z in the substrate (layer 0, whose upward amplitudes are
//    zero) and |z| elsewhere, h the layer's height over the period and 0 for
//    a semi-infinite layer.  The TE and TM terms of one order share their
//    exponentials, so they are summed into one coefficient per component.
//
//  * Bloch-mode basis at the six P2 nodes of every element of a 2D
//    nanostructured layer, at one plane hz (measured from the top of the
//    layer, 0 <= hz <= h): field_value_plane
//    (backend/fortran/field_value_plane.f:6-132),
//        E_j(el, i) = sum_m sol(j, i, m, el) c_j(m),
//        c_{x,y} = d_m + u_m, c_z = (u_m - d_m) / beta_m,
//        d_m = v_m exp(i beta_m hz), u_m = v_{m+M} exp(i beta_m (h - hz)).
//
// Both are evaluated in FP64; sums run in another order than the
// reference's, so results agree to rounding, not bit for bit.
#include <cuda_runtime.h>

#include "dense_la.cuh"
#include "emu_cplx.cuh"
#include "emu_internal.h"

namespace {

// ------------------------------------------------------ plane-wave basis
struct PwOrder {  // one order in shared memory (128 bytes)
  double a, b, gr, gi;
  cd d[3], u[3];
};

constexpr int kPwThreads = 256;
constexpr int kPwMaxOrders = 1536;  // 192 KB of shared memory

struct PwArgs {
  int S, Q, grid, nx, ny, nz, substrate, has_up;
  const double *alphas, *betas;
  const int32_t *sort;
  const cd *kz, *n;
  const double *height;
  const cd *vcd, *vcu;
  long long vcd_stride, vcu_stride;
  const double *x, *y, *z;
  cd *E;
  double *E_abs;
};

__device__ __forceinline__ void pw_coefs(cd c_te, cd c_tm, const double ete[3], const cd etm[3],
                                         cd chi_te, cd chi_tm, cd out[3]) {
  for (int j = 0; j < 3; ++j) {
    const cd te = cdiv(cd{c_te.x * ete[j], c_te.y * ete[j]}, chi_te);
    const cd tm = cdiv(cmul(c_tm, etm[j]), chi_tm);
    out[j] = cadd(te, tm);
  }
}

// Order s of stack b: sorted alpha, beta, k_z and the TE + TM coefficients
// of the down and up amplitudes (backend/plotting.py:2896-2941).
__device__ __forceinline__ PwOrder pw_order(const PwArgs &a, int b, int s, cd n) {
  const int S = a.S;
  const int j = a.sort[(size_t)b * S + s];
  const bool ok = j >= 0 && j < S;  // a sort order that is not a permutation gives NaN fields
  const double al = ok ? a.alphas[(size_t)b * S + j] : nan(""), be = ok ? a.betas[(size_t)b * S + j] : nan("");
  const cd g = a.kz[(size_t)b * S + s];
  const double ab2 = al * al + be * be;
  const double norm = sqrt(ab2);
  const cd k = csqrt_p(cd{ab2 + (g.x * g.x - g.y * g.y), 2.0 * g.x * g.y});
  const cd chi_te = csqrt_p(cdiv(cmul(n, g), k));
  const cd chi_tm = csqrt_p(cdiv(cmul(n, k), g));
  const double ete[3] = {be / norm, -al / norm, 0.0};
  const cd etm[3] = {cd{al / norm, 0.0}, cd{be / norm, 0.0}, cdiv(cd{-norm, 0.0}, g)};
  PwOrder o;
  o.a = al;
  o.b = be;
  o.gr = g.x;
  o.gi = g.y;
  const cd *vd = a.vcd + (size_t)b * a.vcd_stride;
  pw_coefs(vd[s], vd[S + s], ete, etm, chi_te, chi_tm, o.d);
  if (a.has_up) {
    const cd *vu = a.vcu + (size_t)b * a.vcu_stride;
    pw_coefs(vu[s], vu[S + s], ete, etm, chi_te, chi_tm, o.u);
  } else {
    for (int c = 0; c < 3; ++c) o.u[c] = cd{0.0, 0.0};
  }
  return o;
}

// Points (x[q], y[q], z[q]): every term evaluated directly.
__global__ void __launch_bounds__(kPwThreads) pw_fields_kernel(PwArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  PwOrder *ord = (PwOrder *)smem_raw;
  const int b = blockIdx.y;
  const int S = a.S;
  const cd n = a.n[b];
  const double h = a.height ? a.height[b] : 0.0;
  for (int s = threadIdx.x; s < S; s += blockDim.x) ord[s] = pw_order(a, b, s, n);
  __syncthreads();

  cd *E = a.E + (size_t)b * 3 * a.Q;
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < a.Q;
       q += (long long)gridDim.x * blockDim.x) {
    double x, y, z;
    if (a.grid) {
      const int iz = (int)(q % a.nz);
      const long long r = q / a.nz;
      x = a.x[r / a.ny];
      y = a.y[r % a.ny];
      z = a.z[iz];
    } else {
      x = a.x[q];
      y = a.y[q];
      z = a.z[q];
    }
    const double z1 = a.substrate ? -z : fabs(z);
    const double dzd = z1 - h;
    cd e[3] = {cd{0.0, 0.0}, cd{0.0, 0.0}, cd{0.0, 0.0}};
    for (int s = 0; s < S; ++s) {
      const PwOrder &o = ord[s];
      const double ph = o.a * x + o.b * y;
      // exp(i (ph - gamma (z1 - h))) = exp(gi (z1 - h)) (cos, sin)(ph - gr (z1 - h))
      double sd, cdn;
      sincos(ph - o.gr * dzd, &sd, &cdn);
      const double md = exp(o.gi * dzd);
      const cd ed{md * cdn, md * sd};
      for (int c = 0; c < 3; ++c) e[c] = cadd(e[c], cmul(o.d[c], ed));
      if (a.has_up) {
        double su, cu;
        sincos(ph + o.gr * z1, &su, &cu);
        const double mu = exp(-o.gi * z1);
        const cd eu{mu * cu, mu * su};
        for (int c = 0; c < 3; ++c) e[c] = cadd(e[c], cmul(o.u[c], eu));
      }
    }
    for (int c = 0; c < 3; ++c) E[(size_t)c * a.Q + q] = e[c];
    if (a.E_abs) a.E_abs[(size_t)b * a.Q + q] = sqrt(cabs2(e[0]) + cabs2(e[1]) + cabs2(e[2]));
  }
}

// Grid x[nx] x y[ny] x z[nz]: the exponential of every term factors as
// exp(i alpha x) exp(i beta y) times a z factor, so per stack three tables
// are formed once,
//   X[ix][s] = exp(i alpha_s x_ix),  Y[iy][s] = exp(i beta_s y_iy),
//   Z[iz][s][c] = eta_down,c exp(-i gamma_s (z1 - h)) + eta_up,c exp(i gamma_s z1),
// and E_c(ix, iy, iz) = sum_s X Y Z is a contraction with no transcendental
// function per term.
__device__ __forceinline__ cd ldg_c(const cd *p) {
  const double2 v = __ldg((const double2 *)p);
  return cd{v.x, v.y};
}

__global__ void __launch_bounds__(kPwThreads) pw_tables_kernel(PwArgs a, cd *ws, long long ws_stride) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  PwOrder *ord = (PwOrder *)smem_raw;
  const int b = blockIdx.x;
  const int S = a.S;
  const cd n = a.n[b];
  const double h = a.height ? a.height[b] : 0.0;
  for (int s = threadIdx.x; s < S; s += blockDim.x) ord[s] = pw_order(a, b, s, n);
  __syncthreads();
  cd *X = ws + (size_t)b * ws_stride;
  cd *Y = X + (size_t)a.nx * S;
  cd *Z = Y + (size_t)a.ny * S;
  for (int i = threadIdx.x; i < a.nx * S; i += blockDim.x) {
    double sn, cs;
    sincos(ord[i % S].a * a.x[i / S], &sn, &cs);
    X[i] = cd{cs, sn};
  }
  for (int i = threadIdx.x; i < a.ny * S; i += blockDim.x) {
    double sn, cs;
    sincos(ord[i % S].b * a.y[i / S], &sn, &cs);
    Y[i] = cd{cs, sn};
  }
  for (int i = threadIdx.x; i < a.nz * S; i += blockDim.x) {
    const PwOrder &o = ord[i % S];
    const double z = a.z[i / S];
    const double z1 = a.substrate ? -z : fabs(z);
    const double dzd = z1 - h;
    double sd, cdn;
    sincos(-o.gr * dzd, &sd, &cdn);
    const double md = exp(o.gi * dzd);
    const cd ed{md * cdn, md * sd};
    cd zc[3];
    for (int c = 0; c < 3; ++c) zc[c] = cmul(o.d[c], ed);
    if (a.has_up) {
      double su, cu;
      sincos(o.gr * z1, &su, &cu);
      const double mu = exp(-o.gi * z1);
      const cd eu{mu * cu, mu * su};
      for (int c = 0; c < 3; ++c) zc[c] = cadd(zc[c], cmul(o.u[c], eu));
    }
    for (int c = 0; c < 3; ++c) Z[(size_t)i * 3 + c] = zc[c];
  }
}

// The contraction over orders on the FP64 tensor cores (mma.sync m8n8k4 f64):
// for one stack and one y, E[ix][(z, component)] = sum_s X[ix][s] W[s][(z, c)]
// with W = Y[iy][s] Z[z][s][c], a product of 8 x 8 fragments per warp: up to 32
// values of x by up to 12 columns, or 24 by 16 (5 z values).  Four orders at a
// time: the lanes' real parts of X against [Re W | Im W], their imaginary parts
// against [-Im W | Re W], so a lane's complex value of X is loaded once.  The
// two have accumulators of their own: in one, the chain of roundings is twice
// as long as in the complex sum and the error 1.13 times as large (8.6e-16
// against 7.6e-16), and with the registers of both, 56 values of x left one CTA
// per SM (386 us).  A CTA's warps take neighbouring y and share the X and Z
// tables in shared memory (ks orders at a time, rows pitched so that fragment
// reads have no bank conflicts); W is formed in registers, two complex products
// per lane and step.  Columns come in groups of 8; four or fewer left over share
// one fragment, [Re | Im].
// 256 stacks x 51 x 51 x 4 points x 81 orders: 460 us for one thread per (x, y)
// on the FP64 pipe, 305 us here; the FP64 tensor rate bounds it (187 us for the
// fragments with their padding).
constexpr int kGx = 32, kGn = 16, kGz = 5, kGs = 84;
constexpr size_t kGridSmem = (size_t)(kGx + kGn) * kGs * sizeof(cd);

struct GridShape {
  int z0, zstep;  // first z and z values of a chunk
  int xr;         // x values of a CTA (a multiple of 8, at most kGx)
  int ks;         // orders at a time and pitch of the tables' rows: 4 modulo 8, at most kGs
};

// FULL groups of 8 columns, HALF a group of up to 4
template <int FULL, int HALF>
__global__ void __launch_bounds__(256, 2) pw_grid_kernel(PwArgs a, const cd *ws, long long ws_stride, GridShape gs) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int ks = gs.ks;
  cd *Xs = (cd *)smem_raw;      // [xr][ks]
  cd *Zs = Xs + gs.xr * ks;     // [columns][ks]
  constexpr int NF = 2 * FULL + HALF, MF = (FULL == 2 ? kGx - 8 : kGx) / 8;  // fragments of a warp
  const int b = blockIdx.y, S = a.S, tid = threadIdx.x, lane = tid & 31, w = tid >> 5, nw = blockDim.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int xchunks = (a.nx + gs.xr - 1) / gs.xr, yg = (a.ny + nw - 1) / nw, chunk = blockIdx.x / yg;
  const int x0 = (chunk % xchunks) * gs.xr, zb = gs.z0 + (chunk / xchunks) * gs.zstep;
  const int mx = min(gs.xr, a.nx - x0), mf = (mx + 7) / 8, zn = min(gs.zstep, a.nz - zb), nn = 3 * zn;
  const int iy = (blockIdx.x % yg) * nw + w;
  const cd *X = ws + (size_t)b * ws_stride;
  const cd *Y = X + (size_t)a.nx * S;
  const cd *Z = Y + (size_t)a.ny * S;
  double acc[MF][NF][2], acc2[MF][NF][2];
#pragma unroll
  for (int f = 0; f < MF; ++f)
#pragma unroll
    for (int j = 0; j < NF; ++j) acc[f][j][0] = acc[f][j][1] = acc2[f][j][0] = acc2[f][j][1] = 0.0;
  for (int s0 = 0; s0 < S; s0 += ks) {
    const int sc = min(ks, S - s0), steps = (sc + 3) / 4;
    __syncthreads();
    for (int i = tid; i < mf * 8 * ks; i += blockDim.x) {
      const int r = i / ks, s = i % ks;
      Xs[i] = (r < mx && s < sc) ? X[(size_t)(x0 + r) * S + s0 + s] : cd{0.0, 0.0};
    }
    for (int i = tid; i < (8 * FULL + 4 * HALF) * ks; i += blockDim.x) {
      const int n = i / ks, s = i % ks;
      Zs[i] = (n < nn && s < sc) ? Z[((size_t)(zb + n / 3) * S + s0 + s) * 3 + n % 3] : cd{0.0, 0.0};
    }
    __syncthreads();
    if (iy >= a.ny) continue;
    const cd *yr = Y + (size_t)iy * S + s0;
    cd yn = t < sc ? ldg_c(yr + t) : cd{0.0, 0.0};
    for (int q = 0; q < steps; ++q) {
      const int s = 4 * q + t;
      const cd y = yn;
      yn = s + 4 < sc ? ldg_c(yr + s + 4) : cd{0.0, 0.0};
      double b1[NF], b2[NF];
#pragma unroll
      for (int j = 0; j < FULL; ++j) {
        const cd wv = cmul(y, Zs[(8 * j + g) * ks + s]);
        b1[2 * j] = wv.x;
        b1[2 * j + 1] = wv.y;
        b2[2 * j] = -wv.y;
        b2[2 * j + 1] = wv.x;
      }
      if (HALF) {
        const cd wv = cmul(y, Zs[(8 * FULL + (g & 3)) * ks + s]);
        b1[NF - 1] = g < 4 ? wv.x : wv.y;
        b2[NF - 1] = g < 4 ? -wv.y : wv.x;
      }
#pragma unroll
      for (int f = 0; f < MF; ++f) {
        if (f < mf) {
          const cd xv = Xs[(8 * f + g) * ks + s];
#pragma unroll
          for (int j = 0; j < NF; ++j) emu::dmma_884(acc[f][j][0], acc[f][j][1], xv.x, b1[j]);
#pragma unroll
          for (int j = 0; j < NF; ++j) emu::dmma_884(acc2[f][j][0], acc2[f][j][1], xv.y, b2[j]);
        }
      }
    }
  }
  // one fragment row block at a time through shared memory (the X table's
  // place): lanes then take (x, z) pairs
  __syncthreads();
  if (iy >= a.ny) return;
  double *st = (double *)smem_raw + (size_t)w * 8 * 2 * kGn;  // [x][component-major column][re, im]
  cd *E = a.E + (size_t)b * 3 * a.Q;
#pragma unroll
  for (int f = 0; f < MF; ++f) {
    if (f >= mf) break;
#pragma unroll
    for (int j = 0; j < NF; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int c = 2 * t + e;  // column of the fragment
        const bool half = j == 2 * FULL;
        const int n = half ? 8 * FULL + (c & 3) : 8 * (j / 2) + c, part = half ? c >> 2 : j & 1;
        st[(g * kGn + n) * 2 + part] = acc[f][j][e] + acc2[f][j][e];
      }
    __syncwarp();
    for (int i = lane; i < 8 * zn; i += 32) {
      const int r = i / zn, z = i % zn, ix = x0 + 8 * f + r;
      if (ix >= a.nx) continue;
      const cd *v = (const cd *)st + r * kGn + 3 * z;
      const size_t q = ((size_t)ix * a.ny + iy) * a.nz + zb + z;
#pragma unroll
      for (int c = 0; c < 3; ++c) E[(size_t)c * a.Q + q] = v[c];
      if (a.E_abs) a.E_abs[(size_t)b * a.Q + q] = sqrt(cabs2(v[0]) + cabs2(v[1]) + cabs2(v[2]));
    }
    __syncwarp();
  }
}

// chunks of `zstep` z values from z0 on, all alike
template <int FULL, int HALF>
int launch_grid(const PwArgs &a, const cd *ws, long long stride, int n_stacks, int z0, int zstep, int chunks,
                cudaStream_t s) {
  if (cudaFuncSetAttribute(pw_grid_kernel<FULL, HALF>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGridSmem) !=
      cudaSuccess)
    return EMU_E_CUDA;
  GridShape gs;
  gs.z0 = z0;
  gs.zstep = zstep;
  // all x values a warp can hold, fewer where that leaves SMs idle
  const long long yg = (a.ny + 7) / 8;
  const int most = FULL == 2 ? kGx - 8 : kGx, nxc = (a.nx + most - 1) / most;
  gs.xr = ((a.nx + nxc - 1) / nxc + 7) / 8 * 8;
  auto xchunks = [&] { return (long long)((a.nx + gs.xr - 1) / gs.xr); };
  while (gs.xr > 8 && n_stacks * chunks * yg * xchunks() < 128) gs.xr = (gs.xr / 8 + 1) / 2 * 8;
  gs.ks = min(kGs, (a.S + 3) / 8 * 8 + 4);
  const size_t stage = 8 * 8 * 2 * kGn * sizeof(double);  // the results' staging, 8 warps
  size_t smem = (size_t)(gs.xr + 8 * FULL + 4 * HALF) * gs.ks * sizeof(cd);
  if (smem < stage) smem = stage;
  pw_grid_kernel<FULL, HALF><<<dim3((unsigned)(yg * xchunks() * chunks), n_stacks), 256, smem, s>>>(a, ws, stride, gs);
  emu::note_launch();
  return EMU_OK;
}

int launch_grids(const PwArgs &a, const cd *ws, long long stride, int n_stacks, cudaStream_t s) {
  const int whole = a.nz / kGz, rest = a.nz % kGz, z1 = whole * kGz;
  int st = EMU_OK;
  if (whole) st = launch_grid<2, 0>(a, ws, stride, n_stacks, 0, kGz, whole, s);
  if (st != EMU_OK) return st;
  switch (rest) {
    case 1: return launch_grid<0, 1>(a, ws, stride, n_stacks, z1, rest, 1, s);
    case 2: return launch_grid<1, 0>(a, ws, stride, n_stacks, z1, rest, 1, s);
    case 3:
    case 4: return launch_grid<1, 1>(a, ws, stride, n_stacks, z1, rest, 1, s);
  }
  return EMU_OK;
}

// ------------------------------------------------------- Bloch-mode basis
constexpr int kNodeVals = 18;  // 6 P2 nodes x 3 components
constexpr int kGroups = 8;     // mode groups per element (partial sums)
constexpr int kBlochThreads = kNodeVals * kGroups;
constexpr int kSolRow = 13 * 3;  // complex values per (element, mode) row

struct BlochArgs {
  int M, nel;
  const cd *sol;
  long long sol_stride;
  const cd *beta, *vc;
  double h, hz;
  cd *E;
};

__global__ void __launch_bounds__(kBlochThreads) bloch_plane_kernel(BlochArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cd *ct = (cd *)smem_raw;  // [M] coefficient of the transverse components
  cd *cz = ct + a.M;        // [M] coefficient of E_z
  cd *red = cz + a.M;       // [kGroups][kNodeVals]
  const int b = blockIdx.y;
  const cd *beta = a.beta + (size_t)b * a.M;
  const cd *vc = a.vc + (size_t)b * 2 * a.M;
  for (int m = threadIdx.x; m < a.M; m += blockDim.x) {
    const cd bm = beta[m];
    const cd dn = cmul(vc[m], cexp_ikh(bm, a.hz));
    const cd up = cmul(vc[m + a.M], cexp_ikh(bm, a.h - a.hz));
    ct[m] = cadd(up, dn);
    cz[m] = cdiv(csub(up, dn), bm);
  }
  __syncthreads();
  const int o = threadIdx.x % kNodeVals, g = threadIdx.x / kNodeVals;
  const cd *coef = (o % 3 == 2) ? cz : ct;
  const cd *sol_b = a.sol + (size_t)b * a.sol_stride;
  for (int el = blockIdx.x; el < a.nel; el += gridDim.x) {
    const cd *row = sol_b + (size_t)el * a.M * kSolRow + o;
    cd acc{0.0, 0.0};
#pragma unroll 4
    for (int m = g; m < a.M; m += kGroups) acc = cadd(acc, cmul(row[(size_t)m * kSolRow], coef[m]));
    red[g * kNodeVals + o] = acc;
    __syncthreads();
    if (g == 0) {
      cd s = red[o];
      for (int k = 1; k < kGroups; ++k) s = cadd(s, red[k * kNodeVals + o]);
      a.E[((size_t)b * a.nel + el) * kNodeVals + o] = s;
    }
    __syncthreads();
  }
}

}  // namespace

namespace {
long long pw_ws_stride(const EmuPwFields *p) {
  return ((long long)p->nx + p->ny + 3LL * p->nz) * p->n_pw;  // complex values per stack
}
}  // namespace

extern "C" size_t emu_pw_fields_workspace_size(const EmuPwFields *p) {
  if (!p || !p->grid || p->n_stacks <= 0 || p->n_pw < 1 || p->nx < 0 || p->ny < 0 || p->nz < 0) return 0;
  return (size_t)p->n_stacks * (size_t)pw_ws_stride(p) * sizeof(cd);
}

extern "C" int emu_pw_fields(const EmuPwFields *p, void *stream) {
  if (!p || p->n_stacks < 0 || p->n_pw < 1 || p->n_pw > kPwMaxOrders) return EMU_E_ARG;
  if (p->nx < 0 || (p->grid && (p->ny < 0 || p->nz < 0))) return EMU_E_ARG;
  const long long Q = p->grid ? (long long)p->nx * p->ny * p->nz : (long long)p->nx;
  if (Q > 0x7fffffffLL || p->n_stacks > 65535) return EMU_E_SHAPE;
  if (p->n_stacks == 0 || Q == 0) return EMU_OK;
  if (!p->d_alphas || !p->d_betas || !p->d_sort || !p->d_kz || !p->d_n || !p->d_vec_coef_down ||
      !p->d_x || !p->d_y || !p->d_z || !p->d_E)
    return EMU_E_ARG;
  if (p->vcd_stride < 2LL * p->n_pw) return EMU_E_ARG;
  const bool has_up = !p->substrate && p->d_vec_coef_up;
  if (has_up && p->vcu_stride < 2LL * p->n_pw) return EMU_E_ARG;
  PwArgs a;
  a.S = p->n_pw;
  a.Q = (int)Q;
  a.grid = p->grid ? 1 : 0;
  a.nx = p->nx;
  a.ny = p->ny;
  a.nz = p->nz;
  a.substrate = p->substrate ? 1 : 0;
  a.has_up = has_up ? 1 : 0;
  a.alphas = p->d_alphas;
  a.betas = p->d_betas;
  a.sort = p->d_sort;
  a.kz = (const cd *)p->d_kz;
  a.n = (const cd *)p->d_n;
  a.height = p->d_height;
  a.vcd = (const cd *)p->d_vec_coef_down;
  a.vcu = (const cd *)p->d_vec_coef_up;
  a.vcd_stride = p->vcd_stride;
  a.vcu_stride = p->vcu_stride;
  a.x = p->d_x;
  a.y = p->d_y;
  a.z = p->d_z;
  a.E = (cd *)p->d_E;
  a.E_abs = p->d_E_abs;
  const size_t smem = sizeof(PwOrder) * (size_t)p->n_pw;
  cudaStream_t st = (cudaStream_t)stream;
  if (p->grid) {
    const size_t need = emu_pw_fields_workspace_size(p);
    if (!p->d_workspace || p->workspace_bytes < need) return EMU_E_WORKSPACE;
    if (smem > 48 * 1024 &&
        cudaFuncSetAttribute(pw_tables_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
            cudaSuccess)
      return EMU_E_CUDA;
    cd *ws = (cd *)p->d_workspace;
    const long long stride = pw_ws_stride(p);
    pw_tables_kernel<<<(unsigned)p->n_stacks, kPwThreads, smem, st>>>(a, ws, stride);
    emu::note_launch();
    const int gst = launch_grids(a, ws, stride, p->n_stacks, st);
    if (gst != EMU_OK) return gst;
    return emu::check_launch();
  }
  if (smem > 48 * 1024 &&
      cudaFuncSetAttribute(pw_fields_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
          cudaSuccess)
    return EMU_E_CUDA;
  // enough blocks per stack to fill the device a few times over, each one
  // sweeping several tiles of points (its order table is built once)
  long long tiles = (Q + kPwThreads - 1) / kPwThreads;
  long long want = (4LL * emu::sm_count() + p->n_stacks - 1) / p->n_stacks;
  if (want < 1) want = 1;
  if (tiles > want) tiles = want;
  pw_fields_kernel<<<dim3((unsigned)tiles, (unsigned)p->n_stacks), kPwThreads, smem, st>>>(a);
  emu::note_launch();
  return emu::check_launch();
}

extern "C" int emu_bloch_fields_plane(const EmuBlochFieldsPlane *p, void *stream) {
  if (!p || p->n_stacks < 0 || p->n_modes < 1 || p->n_elements < 0) return EMU_E_ARG;
  if (!(p->hz >= 0.0 && p->hz <= p->h)) return EMU_E_ARG;  // the routine's own check
  if (p->n_stacks > 65535) return EMU_E_SHAPE;
  if (p->n_stacks == 0 || p->n_elements == 0) return EMU_OK;
  if (!p->d_sol || !p->d_k_z || !p->d_vec_coef || !p->d_E) return EMU_E_ARG;
  if (p->n_stacks > 1 && p->sol_stride < (long long)p->n_elements * p->n_modes * kSolRow) return EMU_E_ARG;
  BlochArgs a;
  a.M = p->n_modes;
  a.nel = p->n_elements;
  a.sol = (const cd *)p->d_sol;
  a.sol_stride = p->sol_stride;
  a.beta = (const cd *)p->d_k_z;
  a.vc = (const cd *)p->d_vec_coef;
  a.h = p->h;
  a.hz = p->hz;
  a.E = (cd *)p->d_E;
  const size_t smem = sizeof(cd) * (2 * (size_t)p->n_modes + kGroups * kNodeVals);
  if (smem > 200 * 1024) return EMU_E_SHAPE;
  if (smem > 48 * 1024 &&
      cudaFuncSetAttribute(bloch_plane_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
          cudaSuccess)
    return EMU_E_CUDA;
  long long blocks = p->n_elements;
  const long long cap = (16LL * emu::sm_count() + p->n_stacks - 1) / p->n_stacks;
  if (blocks > cap) blocks = cap;
  bloch_plane_kernel<<<dim3((unsigned)blocks, (unsigned)p->n_stacks), kBlochThreads, smem,
                       (cudaStream_t)stream>>>(a);
  emu::note_launch();
  return emu::check_launch();
}
