// Bloch-mode / plane-wave overlap integrals J and J_dag
// (backend/fortran/J_overlap.f:92-198, J_dagger_overlap.f:93-199) and the
// Bloch-mode orthogonality / normalisation factors
// (backend/fortran/orthogonal.f:84-248, normalisation.f:15-31).
//
// The reference loops element x quadrature point x plane wave x mode and
// re-interpolates the P2 field for every plane wave.  Here the quadrature
// is folded into a plane-wave table first:
//   E~_s(el, node) = sum_q w_q |det_el| exp(-i k_s . x_q) phi_node(xi_q)
// (16 quadrature points, affine element map), so that
//   G_c[s, n] = sum_{el,node} E~_s(el, node) sol(c, node, n, el),  c = x, y
// is one complex GEMM with K = 6 nel (up to 64 plane waves straight from the
// fields on the FP64 tensor cores, more as residues on the INT8 ones), and
//   J_E = (beta o G_x - alpha o G_y) / |k_s|,  J_K = (alpha o G_x + beta o G_y) / |k_s|
// in the epilogue (rows in the sorted plane-wave order of pw_ordering.f).
// J_dag uses conj(E~) (exp(+i k.x)) and the adjoint fields.
// The exponentials factor as exp(-i(a0 x + b0 y)) (exp(-i 2 pi x / d))^px
// (exp(-i 2 pi y / dy))^py: per quadrature point one base phase and two
// short power tables replace a sine/cosine per plane wave.
#include <cuda_runtime.h>

#include "dense_la.cuh"
#include "emu_internal.h"
#include "residue_gemm.cuh"

namespace {

using namespace emu;

__constant__ double c_wq[16], c_xq[16], c_yq[16];
__constant__ double c_phi2[16][6];       // P2 basis at the quadrature points
__constant__ float c_phi2f[16][6];       // the same, rounded to FP32 (tensor-core operand path)
__constant__ double c_g3[16][2][10];     // P3 gradients (reference triangle)

// 16-point symmetric rule of Lyness & Jespersen (J. Inst. Math. Appl. 15,
// 1975), as tabulated in backend/fortran/quad_triangle.f:56-145.
void quad_table(double *w, double *x, double *y) {
  const double wbar = 1.443156076777862e-1 / 2.0, w1 = 2.852749028018549e-1 / 6.0;
  const double w2 = 9.737549286959440e-2 / 6.0, w3 = 3.096521116041552e-1 / 6.0;
  const double w4 = 1.633818850466092e-1 / 12.0;
  const double cb = 1.0 / 3.0, a1 = 4.592925882927229e-1, b1 = 8.141482341455413e-2;
  const double a2 = 5.054722831703103e-2, b2 = 8.989055433659379e-1;
  const double a3 = 1.705693077517601e-1, b3 = 6.588613844964797e-1;
  const double a4 = 7.284923929554041e-1, b4 = 2.63112829634638689e-1, c4 = 8.394777409957211e-3;
  const double X[16] = {cb, a1, a1, b1, a2, a2, b2, a3, a3, b3, a4, b4, b4, c4, c4, a4};
  const double Y[16] = {cb, a1, b1, a1, a2, b2, a2, a3, b3, a3, b4, a4, c4, b4, a4, c4};
  const double W[16] = {wbar, w1, w1, w1, w2, w2, w2, w3, w3, w3, w4, w4, w4, w4, w4, w4};
  for (int i = 0; i < 16; ++i) {
    w[i] = W[i];
    x[i] = X[i];
    y[i] = Y[i];
  }
}

int upload_tables() {
  static bool done[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && done[dev]) return EMU_OK;
  double w[16], x[16], y[16], phi[16][6], g[16][2][10];
  float phif[16][6];
  quad_table(w, x, y);
  for (int q = 0; q < 16; ++q) {
    const double x0 = x[q], y0 = y[q];
    // P2 basis (backend/fortran/phi2_2d_mat_J.f:17-30)
    phi[q][0] = (-1 + x0 + y0) * (-1 + 2 * x0 + 2 * y0);
    phi[q][1] = x0 * (-1 + 2 * x0);
    phi[q][2] = y0 * (-1 + 2 * y0);
    phi[q][3] = -4 * x0 * (-1 + x0 + y0);
    phi[q][4] = 4 * x0 * y0;
    phi[q][5] = -4 * y0 * (-1 + x0 + y0);
    for (int k = 0; k < 6; ++k) phif[q][k] = (float)phi[q][k];
    // P3 gradients (backend/fortran/phi3_2d_mat.f:17-64)
    const double t = (-11 - 27 * x0 * x0 + x0 * (36 - 54 * y0) + 36 * y0 - 27 * y0 * y0) / 2.;
    g[q][0][0] = t; g[q][1][0] = t;
    g[q][0][1] = 1 - 9 * x0 + (27 * x0 * x0) / 2.; g[q][1][1] = 0;
    g[q][0][2] = 0; g[q][1][2] = 1 - 9 * y0 + (27 * y0 * y0) / 2.;
    g[q][0][3] = (9 * (2 + 9 * x0 * x0 - 5 * y0 + 3 * y0 * y0 + 2 * x0 * (-5 + 6 * y0))) / 2.;
    g[q][1][3] = (9 * x0 * (-5 + 6 * x0 + 6 * y0)) / 2.;
    g[q][0][4] = (-9 * (1 + 9 * x0 * x0 - y0 + x0 * (-8 + 6 * y0))) / 2.;
    g[q][1][4] = (-9 * x0 * (-1 + 3 * x0)) / 2.;
    g[q][0][5] = (9 * (-1 + 6 * x0) * y0) / 2.;
    g[q][1][5] = (9 * x0 * (-1 + 3 * x0)) / 2.;
    g[q][0][6] = (9 * y0 * (-1 + 3 * y0)) / 2.;
    g[q][1][6] = (9 * x0 * (-1 + 6 * y0)) / 2.;
    g[q][0][7] = (-9 * y0 * (-1 + 3 * y0)) / 2.;
    g[q][1][7] = (-9 * (1 - 8 * y0 + 9 * y0 * y0 + x0 * (-1 + 6 * y0))) / 2.;
    g[q][0][8] = (9 * y0 * (-5 + 6 * x0 + 6 * y0)) / 2.;
    g[q][1][8] = (9 * (2 + 3 * x0 * x0 - 10 * y0 + 9 * y0 * y0 + x0 * (-5 + 12 * y0))) / 2.;
    g[q][0][9] = -27 * y0 * (-1 + 2 * x0 + y0);
    g[q][1][9] = -27 * x0 * (-1 + x0 + 2 * y0);
  }
  if (cudaMemcpyToSymbol(c_wq, w, sizeof(w)) != cudaSuccess ||
      cudaMemcpyToSymbol(c_xq, x, sizeof(x)) != cudaSuccess ||
      cudaMemcpyToSymbol(c_yq, y, sizeof(y)) != cudaSuccess ||
      cudaMemcpyToSymbol(c_phi2, phi, sizeof(phi)) != cudaSuccess ||
      cudaMemcpyToSymbol(c_phi2f, phif, sizeof(phif)) != cudaSuccess ||
      cudaMemcpyToSymbol(c_g3, g, sizeof(g)) != cudaSuccess)
    return EMU_E_CUDA;
  if (dev >= 0 && dev < 64) done[dev] = true;
  return EMU_OK;
}

// Element geometry: vertices, affine map x = B xi + x1, |det B| and T = B^-1
// (backend/fortran/jacobian_p1_2d.f:68-133).
struct Geo {
  double x1, y1, B00, B01, B10, B11, adet, T00, T01, T10, T11;
};

__device__ __forceinline__ Geo element_geo(const double *x, const int64_t *tn, long el) {
  const int64_t n1 = tn[el * 6 + 0] - 1, n2 = tn[el * 6 + 1] - 1, n3 = tn[el * 6 + 2] - 1;
  Geo g;
  g.x1 = x[2 * n1];
  g.y1 = x[2 * n1 + 1];
  g.B00 = x[2 * n2] - g.x1;
  g.B01 = x[2 * n3] - g.x1;
  g.B10 = x[2 * n2 + 1] - g.y1;
  g.B11 = x[2 * n3 + 1] - g.y1;
  const double det = g.B00 * g.B11 - g.B01 * g.B10;
  g.adet = fabs(det);
  g.T00 = g.B11 / det;
  g.T01 = -g.B01 / det;
  g.T10 = -g.B10 / det;
  g.T11 = g.B00 / det;
  return g;
}

// ---------------------------------------------------------------- setup
// Plane-wave data per problem: sorted position (pw_ordering.f:54-78 with the
// z_indexx.f key -Re(kz^2)), alpha, beta and 1/|k| by sorted row.
struct PwArgs {
  int batch, npw;
  const int32_t *px, *py;
  double d, dy;
  const double *bloch, *k0;
  int32_t *pos;       // [batch][npw] sorted position of generation-order s
  double *tab;        // [batch][npw][3]: alpha, beta, 1/|k| by sorted row
  int32_t *out_inv;   // optional copy of pos
  int *zero;          // optional word to clear
};

__global__ void pw_setup_kernel(PwArgs a) {
  extern __shared__ double keys[];
  const int b = blockIdx.x;
  if (a.zero && b == 0 && threadIdx.x == 0) *a.zero = 0;
  const double bx = a.bloch[2 * b], by = a.bloch[2 * b + 1], k0 = a.k0[b];
  const double vkx = 2.0 * 3.141592653589793 / a.d, vky = 2.0 * 3.141592653589793 / a.dy;
  for (int s = threadIdx.x; s < a.npw; s += blockDim.x) {
    const double al = bx + vkx * a.px[s], be = by + vky * a.py[s];
    const cd bz = csqrt_p(cd{k0 * k0 - al * al - be * be, 0.0});
    keys[s] = -(bz.x * bz.x - bz.y * bz.y);
  }
  __syncthreads();
  for (int s = threadIdx.x; s < a.npw; s += blockDim.x) {
    const double ks = keys[s];
    int r = 0;
    for (int v = 0; v < a.npw; ++v) r += (keys[v] < ks) || (keys[v] == ks && v < s);
    a.pos[(size_t)b * a.npw + s] = r;
    if (a.out_inv) a.out_inv[(size_t)b * a.npw + s] = r;
    const double al = bx + vkx * a.px[s], be = by + vky * a.py[s];
    double *t = a.tab + ((size_t)b * a.npw + r) * 3;
    t[0] = al;
    t[1] = be;
    t[2] = 1.0 / sqrt(al * al + be * be);
  }
}

// ---------------------------------------------------------------- E~ table
// One warp per element: lanes build the per-quadrature-point phase tables in
// shared memory, then each lane owns plane waves s and accumulates the six
// node sums E~_s(el, node).  Output row = sorted position of s, column
// (el - e0) * 6 + node; rows padded to ldE.
struct EtArgs {
  int npw, mo, e0, ne;
  const int32_t *px, *py, *pos;
  const double *x;
  const int64_t *tn;
  double d, dy;
  const double *bloch;  // this problem's k_parallel * period (2 values)
  cd *E;
  long long ldE, sE;  // sE: E's stride per problem
  // instead of E: [K][re, im][e2p] doubles, plane waves contiguous, columns up
  // to e2n zero past npw; sE doubles per problem
  double *E2;
  int e2p, e2n;
  // tensor-core path: instead of E, the real embedding A (FP32,
  // [2 npw][2 K], K = 6 ne), columns in (element, node, re/im) order:
  // row s = (Re E, -Im E) pairs, row npw + s = (Im E, Re E) pairs
  float *A32;
  // tensor-core path, several problems per launch (blockIdx.y = problem):
  // per-problem strides of pos (ints) and A32 (floats); bloch advances by 2
  int spos;
  long long sA32;
};

constexpr int kEtWarps = 4;
constexpr int kMaxOrd = 24;  // |px|, |py| <= kMaxOrd

// dynamic shared memory per warp: tx[16][no] (times the base phase and weight),
// ty[16][no], and the staging area of 32 plane waves x 6 nodes (+ 1 pad)
constexpr int kEtRow = 7;
__host__ __device__ inline size_t et_warp_bytes(int mo) {
  return sizeof(cd) * (2 * 16 * (size_t)(2 * mo + 1) + 32 * kEtRow);
}

// FP32 tables of the tensor-core operand path: bc[16] (base x weight),
// tx[16][no], ty[16][no] as float2
__host__ __device__ inline size_t et_warp_bytes_f32(int mo) {
  return sizeof(float2) * (16 + 2 * 16 * (size_t)(2 * mo + 1));
}

// kF32: tensor-core operand path.  The phase tables of each element are
// computed in FP64 (arguments, sincos, powers) and stored rounded to FP32
// (relative 6e-8 per entry); the phase products and the 16-point x 6-node
// sums then run in FP32 (~3e-7 relative), below the ~2^-21 relative error of
// the split-TF32 products they feed.  Half the table bytes of the FP64 path,
// so twice the resident warps.
template <bool kF32>
__global__ void __launch_bounds__(32 * kEtWarps) etable_kernel(EtArgs a) {
  extern __shared__ __align__(16) unsigned char et_smem[];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int no = 2 * a.mo + 1;
  if constexpr (kF32) {
    float2 *bc = (float2 *)(et_smem + (size_t)w * et_warp_bytes_f32(a.mo));  // [16]
    float2 *fx = bc + 16;                                                      // [16][no]
    float2 *fy = fx + 16 * no;                                                 // [16][no]
    const int prob = blockIdx.y;
    const double bx = a.bloch[2 * prob], by = a.bloch[2 * prob + 1];
    const int32_t *pos = a.pos + (size_t)prob * a.spos;
    float *A32 = a.A32 + (size_t)prob * a.sA32;
    const long long K = 6LL * a.ne;
    for (long el0 = (long)blockIdx.x * kEtWarps; el0 < a.ne; el0 += (long)gridDim.x * kEtWarps) {
      const long el = el0 + w;
      const bool ok = el < a.ne;
      if (ok && lane < 16) {
        const Geo g = element_geo(a.x, a.tn, a.e0 + el);
        const int q = lane;
        const double xg = g.x1 + g.B00 * c_xq[q] + g.B01 * c_yq[q];
        const double yg = g.y1 + g.B10 * c_xq[q] + g.B11 * c_yq[q];
        const double wq = c_wq[q] * g.adet;
        double s, c;
        sincos(-(bx * xg + by * yg), &s, &c);
        bc[q] = make_float2((float)(c * wq), (float)(s * wq));
        double sx, cx, sy, cy;
        sincos(-2.0 * 3.141592653589793 / a.d * xg, &sx, &cx);
        sincos(-2.0 * 3.141592653589793 / a.dy * yg, &sy, &cy);
        const cd ux = cd{cx, sx}, uy = cd{cy, sy};
        cd px = cd{1.0, 0.0}, py = cd{1.0, 0.0};
        fx[q * no + a.mo] = make_float2(1.f, 0.f);
        fy[q * no + a.mo] = make_float2(1.f, 0.f);
        for (int p = 1; p <= a.mo; ++p) {
          px = cmul(px, ux);
          py = cmul(py, uy);
          fx[q * no + a.mo + p] = make_float2((float)px.x, (float)px.y);
          fx[q * no + a.mo - p] = make_float2((float)px.x, (float)-px.y);
          fy[q * no + a.mo + p] = make_float2((float)py.x, (float)py.y);
          fy[q * no + a.mo - p] = make_float2((float)py.x, (float)-py.y);
        }
      }
      __syncwarp();
      if (ok) {
        for (int s = lane; s < a.npw; s += 32) {
          const int ix = a.px[s] + a.mo, iy = a.py[s] + a.mo;
          float2 acc[6];
#pragma unroll
          for (int k = 0; k < 6; ++k) acc[k] = make_float2(0.f, 0.f);
#pragma unroll 4
          for (int q = 0; q < 16; ++q) {
            const float2 b = bc[q], u = fx[q * no + ix], v = fy[q * no + iy];
            const float2 t = make_float2(b.x * u.x - b.y * u.y, b.x * u.y + b.y * u.x);
            const float ex = t.x * v.x - t.y * v.y, ey = t.x * v.y + t.y * v.x;
#pragma unroll
            for (int k = 0; k < 6; ++k) {
              acc[k].x = fmaf(ex, c_phi2f[q][k], acc[k].x);
              acc[k].y = fmaf(ey, c_phi2f[q][k], acc[k].y);
            }
          }
          // K order (element, node, re/im): 12 contiguous floats per row
          float4 *r0 = (float4 *)(A32 + (size_t)pos[s] * 2 * K + (size_t)el * 12);
          float4 *r1 = (float4 *)((float *)r0 + (size_t)a.npw * 2 * K);
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            r0[k] = make_float4(acc[2 * k].x, -acc[2 * k].y, acc[2 * k + 1].x, -acc[2 * k + 1].y);
            r1[k] = make_float4(acc[2 * k].y, acc[2 * k].x, acc[2 * k + 1].y, acc[2 * k + 1].x);
          }
        }
      }
      __syncwarp();
    }
    return;
  }
  cd *tx = (cd *)(et_smem + (size_t)w * et_warp_bytes(a.mo));  // [16][no]
  cd *ty = tx + 16 * no;                                         // [16][no]
  cd *st = ty + 16 * no;                                         // [32][kEtRow]
  const long long wstride = (long long)(et_warp_bytes(a.mo) / sizeof(cd));
  const int prob = blockIdx.y;
  const double bx = a.bloch[2 * prob], by = a.bloch[2 * prob + 1];
  const int32_t *pos = a.pos + (size_t)prob * a.spos;
  cd *Eo = a.E + (size_t)prob * a.sE;
  for (long el0 = (long)blockIdx.x * kEtWarps; el0 < a.ne; el0 += (long)gridDim.x * kEtWarps) {
    const long el = el0 + w;
    const bool ok = el < a.ne;
    if (ok && lane < 16) {
      const Geo g = element_geo(a.x, a.tn, a.e0 + el);
      const int q = lane;
      const double xg = g.x1 + g.B00 * c_xq[q] + g.B01 * c_yq[q];
      const double yg = g.y1 + g.B10 * c_xq[q] + g.B11 * c_yq[q];
      const double wq = c_wq[q] * g.adet;
      double s, c;
      sincos(-(bx * xg + by * yg), &s, &c);
      const cd base = cd{c * wq, s * wq};
      // powers of exp(-i 2 pi x / d) and exp(-i 2 pi y / dy), exponents -mo..mo
      double sx, cx, sy, cy;
      sincos(-2.0 * 3.141592653589793 / a.d * xg, &sx, &cx);
      sincos(-2.0 * 3.141592653589793 / a.dy * yg, &sy, &cy);
      const cd ux = cd{cx, sx}, uy = cd{cy, sy};
      cd px = cd{1.0, 0.0}, py = cd{1.0, 0.0};
      tx[q * no + a.mo] = base;
      ty[q * no + a.mo] = py;
      for (int p = 1; p <= a.mo; ++p) {
        px = cmul(px, ux);
        py = cmul(py, uy);
        tx[q * no + a.mo + p] = cmul(base, px);
        tx[q * no + a.mo - p] = cmul(base, cconj(px));
        ty[q * no + a.mo + p] = py;
        ty[q * no + a.mo - p] = cconj(py);
      }
    }
    __syncwarp();
    const int nhere = (int)(a.ne - el0 < kEtWarps ? a.ne - el0 : kEtWarps);
    for (int s0 = 0; s0 < (a.E2 ? a.e2n : a.npw); s0 += 32) {
      const int s = s0 + lane;
      if (a.E2 && ok && s >= a.npw && s < a.e2n)
        for (int k = 0; k < 12; ++k) a.E2[(size_t)prob * a.sE + ((size_t)el * 12 + k) * a.e2p + s] = 0.0;
      if (ok && s < a.npw) {
        const int ix = a.px[s] + a.mo, iy = a.py[s] + a.mo;
        cd acc[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) acc[k] = cd{0.0, 0.0};
#pragma unroll 4
        for (int q = 0; q < 16; ++q) {
          const cd e = cmul(tx[q * no + ix], ty[q * no + iy]);
#pragma unroll
          for (int k = 0; k < 6; ++k) {
            acc[k].x = fma(e.x, c_phi2[q][k], acc[k].x);
            acc[k].y = fma(e.y, c_phi2[q][k], acc[k].y);
          }
        }
        if (a.E2) {
          double *o = a.E2 + (size_t)prob * a.sE + (size_t)el * 12 * a.e2p + pos[s];
#pragma unroll
          for (int k = 0; k < 6; ++k) {
            o[2 * k * a.e2p] = acc[k].x;
            o[(2 * k + 1) * a.e2p] = acc[k].y;
          }
          continue;
        }
#pragma unroll
        for (int k = 0; k < 6; ++k) st[lane * kEtRow + k] = acc[k];
      }
      if (a.E2) continue;
      __syncthreads();
      // the CTA's elements are neighbours in every row: runs of kEtWarps x 96 bytes
      for (int i = threadIdx.x; i < 32 * kEtWarps * 6; i += 32 * kEtWarps) {
        const int within = i % (kEtWarps * 6), r = i / (kEtWarps * 6), ew = within / 6;
        if (s0 + r >= a.npw || ew >= nhere) continue;
        const cd *src = (const cd *)et_smem + ew * wstride + 32 * no + r * kEtRow;
        Eo[(size_t)pos[s0 + r] * a.ldE + (size_t)el0 * 6 + within] = src[within % 6];
      }
      __syncthreads();
    }
    __syncwarp();  // the tables are rebuilt for the next element
  }
}

// ---------------------------------------------------------------- epilogue
// J[row][n]: rows 0..npw-1 = J_E, npw..2npw-1 = J_K (sorted order), divided
// by area_norm; J_dag[i][row] uses adjoint column perm[i] scaled by scale[i].
__global__ void epilogue_kernel(const cd *G, const double *tab, int npw, int nval, double inv_area,
                                int dagger, const cd *scale, const int32_t *perm, cd *out) {
  // problem blockIdx.y: every array advances by its per-problem size
  const long long y = blockIdx.y;
  G += y * 2 * npw * (long long)nval;
  tab += y * 3 * npw;
  if (scale) scale += y * nval;
  if (perm) perm += y * nval;
  out += y * 2 * npw * (long long)nval;
  const long total = (long)npw * nval;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
    const int r = (int)(i / nval), n = (int)(i % nval);
    const double al = tab[3 * r], be = tab[3 * r + 1], nm = tab[3 * r + 2];
    const int src = (dagger && perm) ? perm[n] : n;
    const cd gx = G[(size_t)r * 2 * nval + src], gy = G[(size_t)r * 2 * nval + nval + src];
    cd je = cscale(cd{be * gx.x - al * gy.x, be * gx.y - al * gy.y}, nm);
    cd jk = cscale(cd{al * gx.x + be * gy.x, al * gx.y + be * gy.y}, nm);
    if (!dagger) {
      out[(size_t)r * nval + n] = cscale(je, inv_area);
      out[(size_t)(npw + r) * nval + n] = cscale(jk, inv_area);
    } else {
      if (scale) {
        je = cmul(je, scale[n]);
        jk = cmul(jk, scale[n]);
      }
      out[(size_t)n * 2 * npw + r] = je;
      out[(size_t)n * 2 * npw + npw + r] = jk;
    }
  }
}

// ---------------------------------------------------------------- orthogonality
// Per element, the 12 x 22 real matrix of orthogonal.f:110-193 without the
// pp(type_el) / k0 factor: rows (component, P2 node), columns P2 mass part
// (12) then -grad P3 part (10).
__device__ void element_scal(const Geo &g, double ms[12][22]) {
  for (int i = 0; i < 12; ++i)
    for (int j = 0; j < 22; ++j) ms[i][j] = 0.0;
  for (int q = 0; q < 16; ++q) {
    const double c = c_wq[q] * g.adet;
    double g3[2][10];
    for (int j = 0; j < 10; ++j) {
      g3[0][j] = g.T00 * c_g3[q][0][j] + g.T10 * c_g3[q][1][j];
      g3[1][j] = g.T01 * c_g3[q][0][j] + g.T11 * c_g3[q][1][j];
    }
    for (int it = 0; it < 6; ++it) {
      const double pi = c_phi2[q][it] * c;
      for (int jt = 0; jt < 6; ++jt) {
        const double v = pi * c_phi2[q][jt];
        ms[2 * it][2 * jt] += v;
        ms[2 * it + 1][2 * jt + 1] += v;
      }
      for (int jt = 0; jt < 10; ++jt) {
        ms[2 * it][12 + jt] -= pi * g3[0][jt];
        ms[2 * it + 1][12 + jt] -= pi * g3[1][jt];
      }
    }
  }
}

// sol_el_1 entry j of mode n (orthogonal.f:205-227), without the beta factor
__device__ __forceinline__ cd sol1_entry(const cd *s1, int j) {
  if (j < 12) return s1[(j >> 1) * 3 + (j & 1)];
  const int t = j - 12;  // P3 nodes: vertices 0..2, then nodes 6..12
  return s1[(t < 3 ? t : t + 3) * 3 + 2];
}

// Diagonal of the orthogonality matrix for a batch: block (chunk c, problem
// b) stages the element matrices of kDiagChunk elements in shared memory
// (precomputed once per mesh by elem_scal_kernel), then each thread takes
// modes n = tid, tid + 128, ... and sums its chunk's contribution.
constexpr int kDiagChunk = 16;

struct DiagArgs {
  int nval;
  long nel;
  const double *ms_all;  // [nel][12][22]
  const int64_t *type_el;
  const cd *pp, *sol1, *sol2;  // sol: [B][nel][nval][13][3]
  const double *k0;            // [B]
  cd *part;                    // [B][nchunks][nval]
};

__global__ void __launch_bounds__(128) diag_kernel(DiagArgs a) {
  __shared__ double ms[kDiagChunk][264];
  __shared__ cd ppk[kDiagChunk];
  const long c = blockIdx.x, nch = gridDim.x;
  const int b = blockIdx.y;
  const long e0 = c * kDiagChunk;
  const int ne = (int)min((long)kDiagChunk, a.nel - e0);
  for (int i = threadIdx.x; i < ne * 264; i += blockDim.x)
    ms[i / 264][i % 264] = a.ms_all[(size_t)e0 * 264 + i];
  if (threadIdx.x < ne) {
    const cd p = a.pp[a.type_el[e0 + threadIdx.x] - 1];
    ppk[threadIdx.x] = cd{p.x / a.k0[b], p.y / a.k0[b]};
  }
  __syncthreads();
  const size_t sb = (size_t)b * a.nel * a.nval * 39;
  for (int n = threadIdx.x; n < a.nval; n += blockDim.x) {
    cd acc = cd{0.0, 0.0};
    for (int e = 0; e < ne; ++e) {
      const cd *s1 = a.sol1 + sb + ((size_t)(e0 + e) * a.nval + n) * 39;
      const cd *s2 = a.sol2 + sb + ((size_t)(e0 + e) * a.nval + n) * 39;
      cd s1v[22];
#pragma unroll
      for (int j = 0; j < 22; ++j) s1v[j] = sol1_entry(s1, j);
      const double *m = ms[e];
      cd v_e = cd{0.0, 0.0};
#pragma unroll
      for (int i = 0; i < 12; ++i) {
        cd v = cd{0.0, 0.0};
#pragma unroll
        for (int j = 0; j < 22; ++j) {
          v.x = fma(m[i * 22 + j], s1v[j].x, v.x);
          v.y = fma(m[i * 22 + j], s1v[j].y, v.y);
        }
        v_e = cadd(v_e, cmul(v, s2[(i >> 1) * 3 + (i & 1)]));
      }
      acc = cadd(acc, cmul(v_e, ppk[e]));
    }
    a.part[((size_t)b * nch + c) * a.nval + n] = acc;
  }
}

// diag(n) = beta1(n) sum_chunks part ; scale = 1/sqrt(diag)^2 (or 1); one
// thread per (problem, mode)
__global__ void diag_finish_kernel(const cd *part, int nchunks, int nval, int batch, const cd *beta1,
                                   cd *diag, cd *scale, int *n_small) {
  const long total = (long)batch * nval;
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < total; t += (long)gridDim.x * blockDim.x) {
    const int b = (int)(t / nval), n = (int)(t % nval);
    cd s = cd{0.0, 0.0};
    for (int c = 0; c < nchunks; ++c) s = cadd(s, part[((size_t)b * nchunks + c) * nval + n]);
    s = cmul(s, beta1[t]);
    diag[t] = s;
    if (hypot(s.x, s.y) <= 1e-7) atomicAdd(n_small + b, 1);
    const cd z = csqrt_p(s);
    scale[t] = (hypot(z.x, z.y) > 1e-8) ? crecip(cmul(z, z)) : cd{1.0, 0.0};
  }
}

// ---------------------------------------------------------------- tensor-core operands
// Tensor-core path: the complex contractions G = E~ . S1 and
// G_dag = conj(E~) . S2 = conj(E~ . conj(S2)) share one real GEMM
//   C[2 npw][Nb] = A[2 npw][2 K] . B[Nb][2 K]^T
// with A from etable_kernel (A32 output) and B rows, K in (element, node,
// re/im) order,
//   c * M + m          = (Re S1, Im S1) pairs   (c = 0, 1: x, y component)
//   off1 + c * M + m   = (Re S2, -Im S2) pairs  (off1 = 2 M when S1 is present)
// B tile builder: 8 modes x 16 elements per CTA; the 12 transverse values
// (node 0-5, component 0-1) of each (element, mode) record are read with
// consecutive lanes, staged in shared memory and written as rows of
// 192 contiguous floats.
// Field records may be complex128 (the reference's layout) or complex64 in
// the same layout (half the bytes; the B operand is FP32 either way).
constexpr int kBModes = 8, kBElems = 16;
struct cf32 {
  float x, y;
};
__device__ __forceinline__ cd to_cd(const cd &v) { return v; }
__device__ __forceinline__ cd to_cd(const cf32 &v) { return cd{(double)v.x, (double)v.y}; }

template <class Rec>
__global__ void __launch_bounds__(256) make_B_kernel(const Rec *sol_, long long ssol, int nval, long e0, long ne,
                                                     int conj, int row0, float *B_, long long sB) {
  __shared__ cd v[kBModes][kBElems][12];
  const Rec *sol = sol_ + (size_t)blockIdx.z * ssol;  // problem blockIdx.z
  float *B = B_ + (size_t)blockIdx.z * sB;
  const long long K = 6LL * ne;
  const int m0 = blockIdx.x * kBModes;
  const long el0 = (long)blockIdx.y * kBElems;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // load: warp w takes mode m0 + w, two elements per step (lanes 0-23)
  const int m = m0 + w;
  if (lane < 24) {
    const int j = lane % 12, eo = lane / 12;
    const int node = j >> 1, c = j & 1;
#pragma unroll
    for (int e = eo; e < kBElems; e += 2) {
      const long el = el0 + e;
      cd x = cd{0.0, 0.0};
      if (m < nval && el < ne) x = to_cd(sol[((size_t)(e0 + el) * nval + m) * 39 + node * 3 + c]);
      v[w][e][j] = x;
    }
  }
  __syncthreads();
  // write: 16 rows (c, mode) x 192 floats (element, node, re/im)
  const int nel_here = (int)(ne - el0 < kBElems ? ne - el0 : kBElems);
  for (int i = threadIdx.x; i < 2 * kBModes * 192; i += 256) {
    const int within = i % 192, r = i / 192;
    const int c = r / kBModes, mm = r % kBModes;
    const int e = within / 12, node = (within % 12) >> 1, ri = within & 1;
    if (m0 + mm >= nval || e >= nel_here) continue;
    const cd x = v[mm][e][node * 2 + c];
    const float val = ri == 0 ? (float)x.x : (float)(conj ? -x.y : x.y);
    B[(size_t)(row0 + c * nval + m0 + mm) * 2 * K + (size_t)(el0 + e) * 12 + node * 2 + ri] = val;
  }
}

// G (+)= C[:, 0:2M] ; G_dag (+)= conj(C[:, off1:off1+2M]), C = FP64 sum of
// the tensor-core K-split partials Cp[prob][split][2 npw][nb]; problem
// blockIdx.y; G, Gd advance by gsz per problem.
__global__ void pack_G_parts_kernel(const float *Cp, int nsplit, int npw, int nb, int n2, cd *G_, cd *Gd_,
                                    long long gsz, int off1, int first) {
  const long long prob = blockIdx.y;
  const float *C = Cp + prob * nsplit * (long long)2 * npw * nb;
  cd *G = G_ ? G_ + prob * gsz : nullptr;
  cd *Gd = Gd_ ? Gd_ + prob * gsz : nullptr;
  const long long total = (long long)npw * n2, step = (long long)2 * npw * nb;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int s = (int)(i / n2), n = (int)(i % n2);
    double a0 = 0.0, a1 = 0.0, d0 = 0.0, d1 = 0.0;
    for (int sp = 0; sp < nsplit; ++sp) {
      const float *r0 = C + sp * step + (size_t)s * nb, *r1 = C + sp * step + (size_t)(npw + s) * nb;
      if (G) {
        a0 += (double)r0[n];
        a1 += (double)r1[n];
      }
      if (Gd) {
        d0 += (double)r0[off1 + n];
        d1 += (double)r1[off1 + n];
      }
    }
    if (G) G[i] = first ? cd{a0, a1} : cadd(G[i], cd{a0, a1});
    if (Gd) Gd[i] = first ? cd{d0, -d1} : cadd(Gd[i], cd{d0, -d1});
  }
}


// ---------------------------------------------------------------- residue operands
// FP64 contraction on the INT8 tensor cores (residue_gemm.cuh):
//   C[row][s] = sum_k F[row][k] E~[s][k],  k = (element, node)
// with F's rows (set, component, mode): the transverse fields of sol1, then
// the conjugates of sol2's, so that both sets share one E~ operand:
// G = C^T on the first 2 M rows, G_dag = conj(C)^T on the others.
struct FieldArgs {
  const cd *sol1, *sol2;  // this group's fields; null = that set is absent
  long long ssol;         // stride per problem
  int M, nsets, nblk;     // nblk: element blocks of kFnElems
  long e0, ne;
  double *part;           // [prob][2 nsets M][nblk][2]: sum of squares, largest |component|
  RgScale *scale;         // [prob][2 nsets M]
  int *flags;             // [prob][64 x 64 tiles of H]: the tile holds entries left to FP64 sums
  uint8_t *A;             // residue planes
  int kp;
};

__device__ __forceinline__ const cd *field_set(const FieldArgs &a, int set) {
  return (set == 0 && a.sol1) ? a.sol1 : a.sol2;
}
// whether a set's rows are conjugated: the adjoint fields (which may be the prime
// ones' memory)
__device__ __forceinline__ bool field_dag(const FieldArgs &a, int set) { return set == 1 || !a.sol1; }

// Sums of squares and largest components of the rows over blocks of kFnElems
// elements: a warp takes one mode, lanes 0-23 two elements' 12 transverse
// values at a time (288 contiguous bytes of each 624-byte record are read).
constexpr int kFnElems = 128, kFnModes = 8;

__global__ void __launch_bounds__(256) field_norm_kernel(FieldArgs a) {
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m = blockIdx.x * kFnModes + w, set = blockIdx.z % a.nsets, prob = blockIdx.z / a.nsets;
  if (m >= a.M) return;
  const cd *sol = field_set(a, set) + (size_t)prob * a.ssol;
  const long b0 = (long)blockIdx.y * kFnElems, b1 = min(a.ne, b0 + kFnElems);
  const int j = lane % 12, eo = lane / 12, c = j & 1;
  double ss = 0.0, mx = 0.0;
  if (lane < 24) {
#pragma unroll 8
    for (long e = b0 + eo; e < b1; e += 2) {
      const cd x = sol[((size_t)(a.e0 + e) * a.M + m) * 39 + (j >> 1) * 3 + c];
      ss += fma(x.x, x.x, x.y * x.y);
      mx = fmax(mx, fmax(fabs(x.x), fabs(x.y)));
    }
  }
  // lanes of one component: even (x) or odd (y) lanes
#pragma unroll
  for (int o = 16; o >= 2; o >>= 1) {
    ss += __shfl_xor_sync(0xffffffffu, ss, o);
    mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  }
  if (lane < 2) {
    double *p = a.part + ((((size_t)prob * a.nsets + set) * 2 + lane) * a.M + m) * a.nblk * 2 + 2 * blockIdx.y;
    p[0] = ss;
    p[1] = mx;
  }
}

// Scales of both operands' rows from their parts, one warp per row; clears the
// tile flags.
__global__ void __launch_bounds__(256) row_scale_kernel(const double *fp, int fparts, long frows, RgScale *fs,
                                                        const double *ep, int eparts, long erows, RgScale *es,
                                                        int *flags, long nflags) {
  for (long i = blockIdx.x * 256L + threadIdx.x; i < nflags; i += gridDim.x * 256L) flags[i] = 0;
  const long r = blockIdx.x * 8L + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (r >= frows + erows) return;
  const bool e = r >= frows;
  const int n = e ? eparts : fparts;
  const double *p = e ? ep + (r - frows) * 2 * n : fp + r * 2 * n;
  double ss = 0.0, mx = 0.0;
  for (int b = lane; b < n; b += 32) {
    ss += p[2 * b];
    mx = fmax(mx, p[2 * b + 1]);
  }
  for (int o = 16; o; o >>= 1) {
    ss += __shfl_xor_sync(0xffffffffu, ss, o);
    mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  }
  if (lane == 0) (e ? es[r - frows] : fs[r]) = rg_scale(mx, ss);
}

// Residues of the field rows: a CTA stages 8 modes x 32 elements in shared
// memory; each thread then takes 8 consecutive k of one row, so that a row's
// 192 bytes are written together in every plane.
constexpr int kFcModes = 8, kFcElems = 32, kFcThreads = 384;
static_assert(kFcThreads == 2 * kFcModes * kFcElems * 6 / 8, "one item per thread");
constexpr int kFcStep = kFcThreads / (12 * kFcModes);  // elements loaded at a time
// one pad entry per 8 values: the threads' runs of 8 start in different banks
constexpr int kFcRow = kFcElems * 6 + kFcElems * 6 / 8;
constexpr size_t kFcSmem = 2 * kFcModes * kFcRow * sizeof(cd);

__global__ void __launch_bounds__(kFcThreads, 3) field_residue_kernel(FieldArgs a) {
  extern __shared__ __align__(16) unsigned char fc_smem[];
  cd *buf = (cd *)fc_smem;  // [component][mode][kFcRow]
  const int set = blockIdx.z % a.nsets, prob = blockIdx.z / a.nsets;
  const bool conj = field_dag(a, set);
  const int m0 = blockIdx.x * kFcModes;
  const long e0 = (long)blockIdx.y * kFcElems;
  {
    // this thread's value of a record, its mode and first element
    const int lj = threadIdx.x % 12, lm = (threadIdx.x / 12) % kFcModes, le = threadIdx.x / (12 * kFcModes);
    const cd *src = field_set(a, set) + (size_t)prob * a.ssol +
                    ((size_t)(a.e0 + e0 + le) * a.M + m0 + lm) * 39 + (lj >> 1) * 3 + (lj & 1);
    cd *dst = buf + ((lj & 1) * kFcModes + lm) * kFcRow;
    cd x[kFcElems / kFcStep];
#pragma unroll
    for (int t = 0; t < kFcElems / kFcStep; ++t) {
      x[t] = cd{0.0, 0.0};
      if (m0 + lm < a.M && e0 + le + t * kFcStep < a.ne) x[t] = src[(size_t)t * kFcStep * a.M * 39];
    }
#pragma unroll
    for (int t = 0; t < kFcElems / kFcStep; ++t) {
      const int k = (le + t * kFcStep) * 6 + (lj >> 1);
      dst[k + (k >> 3)] = x[t];
    }
  }
  __syncthreads();
  const long long rows = 2LL * a.nsets * a.M, plane = rows * a.kp;
  constexpr int kItems = kFcElems * 6 / 8;
  const int word = threadIdx.x % kItems, r = threadIdx.x / kItems, c = r / kFcModes, mm = r % kFcModes;
  const long long row = (long long)(set * 2 + c) * a.M + m0 + mm, k0 = e0 * 6 + 8 * word;
  if (m0 + mm >= a.M || k0 >= a.kp) return;
  const double up = a.scale[prob * rows + row].up;
  const cd *v = buf + (c * kFcModes + mm) * kFcRow + 9 * word;
  cd x[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    x[j] = up == 0.0 ? cd{0.0, 0.0} : v[j];
    if (conj) x[j].y = -x[j].y;
  }
  rg_store<kRgPlanesA, 2>(x, up, a.A + ((long long)prob * kRgSlots * kRgPlanesA) * plane + row * a.kp + k0, plane);
}

// Sums of squares and largest components of E~'s rows (blockIdx.x) over parts
// (.y) of kErPart values, per problem (.z).
constexpr int kErPart = 2048;

__global__ void __launch_bounds__(256) erow_norm_kernel(const cd *E, long long sE, int npw, long long K, double *part) {
  __shared__ double sh[2][8];
  const cd *row = E + (size_t)blockIdx.z * sE + (size_t)blockIdx.x * K;
  const long long k0 = (long long)blockIdx.y * kErPart, k1 = min(K, k0 + kErPart);
  double ss = 0.0, mx = 0.0;
  for (long long k = k0 + threadIdx.x; k < k1; k += 256) {
    const cd x = row[k];
    ss += fma(x.x, x.x, x.y * x.y);
    mx = fmax(mx, fmax(fabs(x.x), fabs(x.y)));
  }
  for (int o = 16; o; o >>= 1) {
    ss += __shfl_xor_sync(0xffffffffu, ss, o);
    mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  }
  if ((threadIdx.x & 31) == 0) {
    sh[0][threadIdx.x >> 5] = ss;
    sh[1][threadIdx.x >> 5] = mx;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 1; i < 8; ++i) {
      ss += sh[0][i];
      mx = fmax(mx, sh[1][i]);
    }
    double *p = part + (((size_t)blockIdx.z * npw + blockIdx.x) * gridDim.y + blockIdx.y) * 2;
    p[0] = ss;
    p[1] = mx;
  }
}

// Residues of columns [k0, k0 + K) of E~'s rows; a thread takes 4 consecutive k.
__global__ void __launch_bounds__(256) erow_residue_kernel(const cd *E, long long sE, long long ldE, int npw,
                                                           long long K, int kp, const RgScale *scale, uint8_t *B) {
  const int s = blockIdx.x, prob = blockIdx.z;
  const cd *row = E + (size_t)prob * sE + (size_t)s * ldE;
  const double up = scale[(size_t)prob * npw + s].up;
  const long long plane = (long long)npw * kp;
  const long long k0 = ((long long)blockIdx.y * 256 + threadIdx.x) * 4;
  if (k0 >= kp) return;
  cd x[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) x[j] = (k0 + j < K && up != 0.0) ? row[k0 + j] : cd{0.0, 0.0};
  rg_store<kRgPlanesB, 1>(x, up, B + ((long long)prob * kRgSlots * kRgPlanesB) * plane + (long long)s * kp + k0, plane);
}

// An entry left to FP64 sums: a row without a safe scale, or a component whose sum of
// magnitudes is too small for residues; `src` points at its first magnitude code of
// split 0, splits `step` bytes apart.
__device__ __forceinline__ bool field_left(const uint8_t *src, long long plane, long long step, int nsplit, double da,
                                           double db) {
  float sr = 0.0f, si = 0.0f;
  for (int i = 0; i < nsplit; ++i) {
    sr += rg_uncode(src[i * step]);
    si += rg_uncode(src[i * step + plane]);
  }
  return da < 0.0 || db < 0.0 || rg_unsafe(sr) || rg_unsafe(si);
}

// H (+)= C from its residues, conjugated on the rows of sol2 (H = G^T there,
// and G_dag^T): a thread takes one field row and four plane waves.  Entries left
// to FP64 sums are not touched; their tile is flagged.
__global__ void __launch_bounds__(128) field_crt_kernel(FieldArgs a, const uint8_t *C, int ldn, int nsplit, int npw,
                                                        const RgScale *es, cd *H, int first, const int *err) {
  const int prob = blockIdx.y;
  const long long rows = 2LL * a.nsets * a.M, plane = rows * ldn;
  const int words = ldn / 4;
  const long long i = blockIdx.x * 128LL + threadIdx.x;
  if (i >= rows * words) return;
  const long long row = i / words;
  const int s0 = (int)(i % words) * 4;
  const bool dag = field_dag(a, (int)(row / (2 * a.M)));
  const double down = a.scale[prob * rows + row].down;
  cd out[4];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    // residues plus 128 in byte lanes; with K splits as pairs of 16-bit sums
    uint32_t e[kRgMods], o[kRgMods];
#pragma unroll
    for (int m = 0; m < kRgMods; ++m) e[m] = o[m] = 0;
    for (int sp = 0; sp < nsplit; ++sp) {
      const uint8_t *src = C + (((long long)prob * nsplit + sp) * kRgSlots * 2 + h) * plane + row * ldn + s0;
#pragma unroll
      for (int m = 0; m < kRgMods; ++m) {
        const uint32_t w = *(const uint32_t *)(src + 2 * m * plane) ^ 0x80808080u;
        e[m] += w & 0x00ff00ffu;
        o[m] += (w >> 8) & 0x00ff00ffu;
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const double x = down * rg_crt(
          [&](auto i) {
            const uint32_t v = j & 1 ? o[decltype(i)::value] : e[decltype(i)::value];
            return j & 2 ? v >> 16 : v & 0xffffu;
          },
          128u * nsplit);
      if (h == 0) out[j].x = x;
      else out[j].y = x;
    }
  }
  const bool failed = *err != 0;
  const long long step = 2LL * kRgSlots * plane;
  const uint8_t *mags = C + (long long)prob * nsplit * step + 2LL * kRgMods * plane + row * ldn + s0;
  bool left = false;
  cd *Hr = H + (prob * rows + row) * npw;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int s = s0 + j;
    if (s >= npw) break;
    const double ed = es[(size_t)prob * npw + s].down;
    cd c = cscale(out[j], ed);
    if (failed) {
      c = cd{nan(""), nan("")};
    } else if (field_left(mags + j, plane, step, nsplit, down, ed)) {
      left = true;
      continue;
    }
    if (dag) c.y = -c.y;
    Hr[s] = first ? c : cadd(Hr[s], c);
  }
  if (left) a.flags[(prob * ((rows + 63) / 64) + row / 64) * ((npw + 63) / 64) + s0 / 64] = 1;
}

// The flagged tiles again on the FP64 tensor cores, for the entries left over.
__global__ void __launch_bounds__(kDLThreads) field_left_kernel(FieldArgs a, const uint8_t *C, int ldn, int nsplit,
                                                                int npw, const RgScale *es, const cd *E, long long sE,
                                                                cd *H, int first) {
  const long long prob = blockIdx.z, rows = 2LL * a.nsets * a.M, plane = rows * ldn, step = 2LL * kRgSlots * plane;
  if (!a.flags[(prob * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x]) return;
  __shared__ GemmSmem sm;
  const long long r0 = blockIdx.y * 64LL;
  const int s0 = blockIdx.x * 64;
  const long long K = 6LL * a.ne;
  const cd *Ep = E + prob * sE;
  // the one row of A's tile that this thread fetches of each 32
  auto field_row = [&](long long row, bool &dag) -> const cd * {
    const int set = (int)(row / (2 * a.M)), cm = (int)(row % (2 * a.M));
    dag = field_dag(a, set);
    return field_set(a, set) + prob * a.ssol + ((size_t)a.e0 * a.M + cm % a.M) * 39 + cm / a.M;
  };
  cta_tile<64, true>(
      (int)K,
      [&](int r, int k) {
        if (r0 + r >= rows) return cd{0.0, 0.0};
        bool dag;
        const cd *f = field_row(r0 + r, dag);
        cd v = f[(size_t)(k / 6) * a.M * 39 + (k % 6) * 3];
        if (dag) v.y = -v.y;
        return v;
      },
      [&](int k, int c) { return s0 + c < npw ? Ep[(size_t)(s0 + c) * K + k] : cd{0.0, 0.0}; },
      [&](int r, int c, cd v) {
        const long long row = r0 + r;
        const int s = s0 + c;
        if (row >= rows || s >= npw) return;
        const uint8_t *mags = C + prob * nsplit * step + 2LL * kRgMods * plane + row * ldn + s;
        if (!field_left(mags, plane, step, nsplit, a.scale[prob * rows + row].down, es[prob * npw + s].down)) return;
        if (field_dag(a, (int)(row / (2 * a.M)))) v.y = -v.y;
        cd *h = H + (prob * rows + row) * npw + s;
        *h = first ? v : cadd(*h, v);
      },
      sm);
}

// J and J_dag from H (rows component, mode; columns plane waves in sorted
// order), as epilogue_kernel: 32 x 32 tiles (modes x plane waves) through
// shared memory, so that both layouts are read and written in rows.
struct OutArgs {
  const cd *H;         // [problem][rows][npw]
  long long sH;
  const double *tab;
  int npw, nval, nsets;
  double inv_area;
  const cd *scale;
  const int32_t *perm;
  cd *J, *Jd;  // null = that set is absent
};

__global__ void __launch_bounds__(256) rows_epilogue_kernel(OutArgs a) {
  __shared__ cd je[32][33], jk[32][33];
  const int npw = a.npw, nval = a.nval, set = blockIdx.z % a.nsets;
  const long long y = blockIdx.z / a.nsets;
  const bool dagger = set == 1 || !a.J;
  const cd *H = a.H + y * a.sH + (long long)set * 2 * nval * npw;
  const double *tab = a.tab + y * 3 * npw, inv_area = a.inv_area;
  const cd *scale = a.scale ? a.scale + y * nval : nullptr;
  const int32_t *perm = a.perm ? a.perm + y * nval : nullptr;
  cd *out = (dagger ? a.Jd : a.J) + y * 2 * npw * (long long)nval;
  const int n0 = blockIdx.y * 32, s0 = blockIdx.x * 32, tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  for (int i = ty; i < 32; i += 8) {
    const int n = n0 + i, s = s0 + tx;
    if (n >= nval || s >= npw) continue;
    const int src = (dagger && perm) ? perm[n] : n;
    const double al = tab[3 * s], be = tab[3 * s + 1], nm = tab[3 * s + 2];
    const cd gx = H[(size_t)src * npw + s], gy = H[(size_t)(nval + src) * npw + s];
    cd e = cscale(cd{be * gx.x - al * gy.x, be * gx.y - al * gy.y}, nm);
    cd k = cscale(cd{al * gx.x + be * gy.x, al * gx.y + be * gy.y}, nm);
    if (dagger) {
      if (scale) {
        e = cmul(e, scale[n]);
        k = cmul(k, scale[n]);
      }
      out[(size_t)n * 2 * npw + s] = e;
      out[(size_t)n * 2 * npw + npw + s] = k;
    } else {
      je[i][tx] = cscale(e, inv_area);
      jk[i][tx] = cscale(k, inv_area);
    }
  }
  if (dagger) return;
  __syncthreads();
  for (int i = ty; i < 32; i += 8) {
    const int s = s0 + i, n = n0 + tx;
    if (n >= nval || s >= npw) continue;
    out[(size_t)s * nval + n] = je[tx][i];
    out[(size_t)(npw + s) * nval + n] = jk[tx][i];
  }
}

// ---------------------------------------------------------------- direct contraction
// Few plane waves: the contraction on the FP64 tensor cores, straight from the
// fields in the reference's layout.  Residues cost the same per field value
// for any number of plane waves (scaling, 34 bytes written and read back,
// reduced and converted); the FP64 products cost in proportion to it.
//
// A warp takes 8 modes of both components (and of both sets, SETS = 2) and up to
// 8 NT plane waves; a CTA's 8 warps share the E~ tile of 8 elements in shared
// memory (double-buffered, cp.async), whose fragments serve all of the warp's
// rows.  K runs four complex values at a time in the fields' own order: lane
// (mode g, value t) loads the 32 bytes of both components of one node, real
// parts go against [Er | Ei], imaginary parts against [-Ei | Er].  The fields of
// the next element pair are on their way (registers) while one pair is
// summed.  The sum over elements always has the same shape, whatever the batch: folds
// of kOdFold elements, added in order over a segment (64 elements, more for large
// meshes), segments added by reduce_parts_kernel.  A CTA takes some segments, or, where
// that leaves SMs idle, some folds, and writes their sums one by one.
//
// Bound by the FP64 tensor cores: 50 problems of 2 048 elements, 60 modes and 29
// plane waves take 1.65 ms for 40.3 GFLOP of whole fragments (24.4 TFLOP/s of the
// 36.4 that DFMA reaches); repacking, FP64 GEMM and reduction took 7.0 ms, the
// residue kernels 3.6 ms.  Two sets per warp halve the E~ loads per product; at
// more than 32 plane waves their accumulators no longer fit in registers.
// Accumulators are folded into a running sum in shared memory every kOdFold
// elements: chains of 192 products keep the rounding of one accumulator (which
// grows with the chain) at or below that of the 64 partial sums used before.
constexpr int kOdElems = 8, kOdThreads = 256, kOdFold = 16;

struct DirectArgs {
  const cd *sol1, *sol2;
  long long ssol;
  int M, nsets, npw, pitch;
  long e0, ne;      // this span
  long per;         // elements per CTA: whole parts
  int fpp;          // folds per part (a segment, or one)
  const double *E2;
  long long sE;
  cd *H;            // [part][...]
  long long sPart;
  int add;          // later spans add to H (a single part)
};

__host__ __device__ constexpr int od_pitch(int nt) { return 8 * nt + 4; }
// elements per E~ tile: two tiles and the running sums fit in shared memory
__host__ __device__ constexpr int od_elems(int nt) { return nt > 4 ? kOdElems / 2 : kOdElems; }
__host__ __device__ constexpr int od_tile(int nt) { return 12 * od_elems(nt) * od_pitch(nt); }
constexpr size_t od_smem(int nt, int sets) { return sizeof(double) * (2 * od_tile(nt) + 8 * nt * sets * kOdThreads); }

template <int NT, int SETS>
__global__ void __launch_bounds__(kOdThreads, 1) overlap_direct_kernel(DirectArgs a) {
  extern __shared__ __align__(16) unsigned char od_raw[];
  double *tile = (double *)od_raw;  // [2][kOdElems * 6][re, im][pitch]
  constexpr int P = od_pitch(NT), kTile = od_tile(NT), kElems = od_elems(NT);
  double *sum = tile + 2 * kTile + threadIdx.x;  // [accumulator][thread]
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int groups = a.nsets / SETS, prob = blockIdx.z / groups, set0 = blockIdx.z % groups * SETS;
  const int m = (blockIdx.x * 8 + w) * 8 + g;
  const long b0 = (long)blockIdx.y * a.per, b1 = min(a.ne, b0 + a.per);
  const double *E2 = a.E2 + (size_t)prob * a.sE;
  const cd *sol[SETS];
  bool dag[SETS];
#pragma unroll
  for (int i = 0; i < SETS; ++i) {
    dag[i] = set0 + i == 1 || !a.sol1;
    sol[i] = (dag[i] ? a.sol2 : a.sol1) + (size_t)prob * a.ssol + ((size_t)a.e0 * a.M + (m < a.M ? m : 0)) * 39;
  }
  auto load_tile = [&](long el, int buf) {
    const int rows = 12 * (int)min((long)kElems, b1 - el);
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(tile + buf * kTile);
    const double *src = E2 + (size_t)el * 12 * P;
    for (int i = threadIdx.x; i < kTile / 2; i += kOdThreads) {
      const bool in = i < rows * (P / 2);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + 16 * i), "l"(src + (in ? 2 * i : 0)),
                   "r"(in ? 16 : 0)
                   : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // fields of an element pair: step q, this lane's value 4 q + t of the pair's 12
  cd f[3][SETS][2];
  auto load_step = [&](long el, int q) {
    const int idx = 4 * q + t, de = idx / 6, node = idx - 6 * de;
    const bool in = m < a.M && el + de < b1;
#pragma unroll
    for (int i = 0; i < SETS; ++i) {
      const cd *p = sol[i] + (size_t)(el + de) * a.M * 39 + node * 3;
      f[q][i][0] = in ? p[0] : cd{0.0, 0.0};
      f[q][i][1] = in ? p[1] : cd{0.0, 0.0};
    }
  };
  double re[SETS][2][NT][2] = {}, im[SETS][2][NT][2] = {};
  auto fold = [&](bool first) {  // re, im += into the running sums, and restart
#pragma unroll
    for (int i = 0; i < SETS; ++i)
#pragma unroll
      for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            double *p = sum + (size_t)(((i * 2 + c) * NT + j) * 2 + e) * 2 * kOdThreads;
            p[0] = first ? re[i][c][j][e] : p[0] + re[i][c][j][e];
            p[kOdThreads] = first ? im[i][c][j][e] : p[kOdThreads] + im[i][c][j][e];
            re[i][c][j][e] = im[i][c][j][e] = 0.0;
          }
  };
  // the sums into H, over what `folded` has left in the running ones; restarts
  auto emit = [&](long part, bool folded) {
    cd *H = a.H + part * a.sPart + (size_t)prob * 2 * a.nsets * a.M * a.npw;
#pragma unroll
    for (int i = 0; i < SETS; ++i)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        cd *row = H + ((size_t)((set0 + i) * 2 + c) * a.M + m) * a.npw;
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int s = 8 * j + 2 * t + e;
            const double *p = sum + (size_t)(((i * 2 + c) * NT + j) * 2 + e) * 2 * kOdThreads;
            cd v{re[i][c][j][e], im[i][c][j][e]};
            re[i][c][j][e] = im[i][c][j][e] = 0.0;
            if (s >= a.npw || m >= a.M) continue;
            if (folded) v = cadd(cd{p[0], p[kOdThreads]}, v);
            if (dag[i]) v.y = -v.y;
            row[s] = a.add ? cadd(row[s], v) : v;
          }
      }
  };
  if (b0 < b1) {
    load_tile(b0, 0);
#pragma unroll
    for (int q = 0; q < 3; ++q) load_step(b0, q);
  }
  int buf = 0;
  long part = b0 / ((long)kOdFold * a.fpp);
  int done = 0;  // folds of the part
  for (long f0 = b0; f0 < b1; f0 += kOdFold, ++done) {
    if (done == a.fpp) {
      emit(part++, done > 1);
      done = 0;
    } else if (done) {
      fold(done == 1);
    }
#pragma unroll 1
    for (long el = f0; el < min(b1, f0 + kOdFold); el += kElems, buf ^= 1) {
      if (el + kElems < b1) {
        load_tile(el + kElems, buf ^ 1);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
      } else {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
      }
      __syncthreads();
      const double *T = tile + buf * kTile;
#pragma unroll 1
      for (int pr = 0; pr < kElems / 2; ++pr) {
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          double ar[SETS][2], ai[SETS][2];
#pragma unroll
          for (int i = 0; i < SETS; ++i)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
              ar[i][c] = f[q][i][c].x;
              ai[i][c] = dag[i] ? -f[q][i][c].y : f[q][i][c].y;
            }
          load_step(el + 2 * pr + 2, q);
          const double *Er = T + (size_t)(12 * pr + 4 * q + t) * 2 * P + g, *Ei = Er + P;
#pragma unroll
          for (int j = 0; j < NT; ++j) {
            const double er = Er[8 * j], ei = Ei[8 * j];
#pragma unroll
            for (int i = 0; i < SETS; ++i)
#pragma unroll
              for (int c = 0; c < 2; ++c) {
                dmma_884(re[i][c][j][0], re[i][c][j][1], ar[i][c], er);
                dmma_884(im[i][c][j][0], im[i][c][j][1], ar[i][c], ei);
              }
#pragma unroll
            for (int i = 0; i < SETS; ++i)
#pragma unroll
              for (int c = 0; c < 2; ++c) {
                dmma_884(re[i][c][j][0], re[i][c][j][1], -ai[i][c], ei);
                dmma_884(im[i][c][j][0], im[i][c][j][1], ai[i][c], er);
              }
          }
        }
      }
      __syncthreads();
    }
  }
  if (b0 < b1) emit(part, done > 1);
}

template <int NT, int SETS>
cudaError_t launch_direct(const DirectArgs &a, int probs, cudaStream_t s) {
  const cudaError_t e = cudaFuncSetAttribute(overlap_direct_kernel<NT, SETS>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)od_smem(NT, SETS));
  if (e != cudaSuccess) return e;
  overlap_direct_kernel<NT, SETS>
      <<<dim3((a.M + 63) / 64, (unsigned)((a.ne + a.per - 1) / a.per), probs * (a.nsets / SETS)), kOdThreads,
         od_smem(NT, SETS), s>>>(a);
  return cudaSuccess;
}

// H = the sum of the parts (added to it if `add`): `per` parts of a segment in order,
// eight threads per entry for every eighth segment, then the eight sums in order.
__global__ void __launch_bounds__(256) reduce_parts_kernel(cd *H, const cd *part, long long n, int parts, int per,
                                                           int add) {
  __shared__ cd sh[8][32];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const long long i = blockIdx.x * 32LL + tx;
  cd v{0.0, 0.0};
  if (i < n)
    for (int k0 = ty * per; k0 < parts; k0 += 8 * per) {
      cd w = part[k0 * n + i];
#pragma unroll 8
      for (int k = k0 + 1; k < min(parts, k0 + per); ++k) w = cadd(w, part[k * n + i]);
      v = cadd(v, w);
    }
  sh[ty][tx] = v;
  __syncthreads();
  if (ty || i >= n) return;
#pragma unroll
  for (int k = 1; k < 8; ++k) v = cadd(v, sh[k][tx]);
  H[i] = add ? cadd(H[i], v) : v;
}

// fragments held by the kernel that serves npw plane waves (0: none does)
inline int od_frags(int npw) {
  return npw <= 8 ? 1 : npw <= 16 ? 2 : npw <= 32 ? 4 : npw <= 64 ? 8 : 0;
}

cudaError_t launch_direct_any(const DirectArgs &a, int probs, cudaStream_t s) {
  switch (od_frags(a.npw)) {
    case 1: return a.nsets == 2 ? launch_direct<1, 2>(a, probs, s) : launch_direct<1, 1>(a, probs, s);
    case 2: return a.nsets == 2 ? launch_direct<2, 2>(a, probs, s) : launch_direct<2, 1>(a, probs, s);
    case 4: return a.nsets == 2 ? launch_direct<4, 2>(a, probs, s) : launch_direct<4, 1>(a, probs, s);
    case 8: return launch_direct<8, 1>(a, probs, s);
  }
  return cudaErrorInvalidValue;
}

// ---------------------------------------------------------------- pair reordering
// Full adjoint x prime matrix for the conjugate-pair reordering of
// orthogonal.f:252-301 (only run when a diagonal entry vanishes).
__global__ void elem_scal_kernel(const double *x, const int64_t *tn, long nel, double *ms_all) {
  for (long el = blockIdx.x * (long)blockDim.x + threadIdx.x; el < nel; el += (long)gridDim.x * blockDim.x) {
    double ms[12][22];
    element_scal(element_geo(x, tn, el), ms);
    double *o = ms_all + (size_t)el * 264;
    for (int i = 0; i < 12; ++i)
      for (int j = 0; j < 22; ++j) o[i * 22 + j] = ms[i][j];
  }
}

// ovl[i][j] = sum_el (pp_e / k0) sol2_el(:, i)^T ms_el (beta1(j) sol1_el(:, j)); one thread per (i, j).
__global__ void ovl_full_kernel(const double *ms_all, int nval, long nel, const int64_t *type_el,
                                const cd *pp, const double *k0, const cd *beta1, const cd *sol1,
                                const cd *sol2, cd *ovl) {
  const long total = (long)nval * nval;
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < total; t += (long)gridDim.x * blockDim.x) {
    const int i = (int)(t / nval), j = (int)(t % nval);
    cd acc = cd{0.0, 0.0};
    for (long el = 0; el < nel; ++el) {
      const double *ms = ms_all + (size_t)el * 264;
      const cd *s1 = sol1 + ((size_t)el * nval + j) * 39;
      const cd *s2 = sol2 + ((size_t)el * nval + i) * 39;
      cd e = cd{0.0, 0.0};
      for (int r = 0; r < 12; ++r) {
        cd v = cd{0.0, 0.0};
        for (int c = 0; c < 22; ++c) {
          const cd s = sol1_entry(s1, c);
          v.x = fma(ms[r * 22 + c], s.x, v.x);
          v.y = fma(ms[r * 22 + c], s.y, v.y);
        }
        e = cadd(e, cmul(v, s2[(r >> 1) * 3 + (r & 1)]));
      }
      const cd p = pp[type_el[el] - 1];
      acc = cadd(acc, cmul(e, cd{p.x / k0[0], p.y / k0[0]}));
    }
    ovl[t] = cmul(acc, beta1[j]);
  }
}

// The reordering loop itself (one thread): swaps of adjoint modes recorded
// as a permutation; the recomputed diagonal is ovl[perm[i]][i].
__global__ void pair_swap_kernel(const cd *ovl, int nval, int32_t *perm, cd *diag, cd *scale, int32_t *warn) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  for (int i = 0; i < nval; ++i) perm[i] = i;
  int skip = 0, w = 0;
  for (int j = 0; j < nval; ++j) {
    const cd djj = ovl[(size_t)j * nval + j];
    if (hypot(djj.x, djj.y) > 1e-7) continue;
    if (skip == 0) {
      if (j == nval - 1) ++w;
      for (int j2 = j + 1; j2 < nval; ++j2) {
        const cd o = ovl[(size_t)j2 * nval + j];
        if (hypot(o.x, o.y) > 1e-7) {
          const int t = perm[j];
          perm[j] = perm[j2];
          perm[j2] = t;
        }
      }
      skip = 1;
    } else {
      skip = 0;
    }
  }
  for (int i = 0; i < nval; ++i) {
    const cd d = ovl[(size_t)perm[i] * nval + i];
    diag[i] = d;
    const cd z = csqrt_p(d);
    scale[i] = (hypot(z.x, z.y) > 1e-8) ? crecip(cmul(z, z)) : cd{1.0, 0.0};
  }
  *warn = w;
}

}  // namespace

// =============================================================== C ABI
// ---- tensor-core path: problems in groups, one launch per step for a group
struct TcPlan {
  long nec;        // elements per chunk
  long long K2;    // 12 nec: GEMM K of one chunk
  int nb, off1;    // B rows (2M per field set), row of the adjoint set
  int group;       // problems per launch
  int splits;      // K splits of the GEMM
};

constexpr size_t kTcGroupBytes = (size_t)4 << 30;  // scratch budget of one group
// The tensor cores accumulate in FP32 and the sum drifts toward zero by
// about 7e-9 x K relative (measured: 1.9e-6 rms at K = 256, 7.3e-6 at 1024,
// 1.8e-3 at 262144, for random operands).  The GEMM kernel therefore starts
// a fresh tensor-memory accumulation every 256 K values and sums those
// chunk results in FP32 (round to nearest) inside the CTA; a CTA's K range
// holds at most kTcMaxChunksPerCta chunks, and the K splits (CTAs) are
// summed in FP64.
constexpr long long kTcChunkK = 256;
constexpr long long kTcMaxChunksPerCta = 32;
constexpr int kTcMaxSplits = 256;
// element chunk (12 K values per element) of one GEMM
constexpr long kTcMaxChunk = 32768;

static size_t tc_problem_bytes(const EmuOverlap *p, const TcPlan &t) {
  const size_t npw = p->n_pw, M = p->nval;
  return align_up(sizeof(int32_t) * npw, 16) + align_up(sizeof(double) * 3 * npw, 16) +
         2 * align_up(sizeof(cd) * npw * 2 * M, 16) + sizeof(float) * 2 * npw * t.K2 +
         sizeof(float) * t.nb * t.K2 + sizeof(float) * t.splits * 2 * npw * t.nb;
}

static TcPlan tc_plan(const EmuOverlap *p) {
  TcPlan t;
  long chunk = p->elements_per_chunk > 0 ? p->elements_per_chunk : 4096;
  if (chunk > kTcMaxChunk) chunk = kTcMaxChunk;
  t.nec = chunk < p->nel ? chunk : p->nel;
  t.K2 = 12 * (long long)t.nec;
  t.nb = (p->d_sol1 ? 2 * p->nval : 0) + (p->d_sol2 ? 2 * p->nval : 0);
  if (t.nb == 0) t.nb = 2 * p->nval;
  t.off1 = p->d_sol1 ? 2 * p->nval : 0;
  // largest group within the budget (at one split), then splits so that
  // tiles x splits x group fills one wave of CTAs
  t.splits = 1;
  const size_t per = tc_problem_bytes(p, t);
  long long g = (long long)(kTcGroupBytes / (per > 0 ? per : 1));
  if (g < 1) g = 1;
  if (g > p->batch) g = p->batch;
  if (g > 1024) g = 1024;
  t.group = (int)g;
  const int tiles = emu::tc_tiles(2 * p->n_pw, t.nb) * t.group;
  int sp = (emu::sm_count() + tiles - 1) / tiles;
  const int maxsp = (int)(t.K2 / kTcChunkK > 0 ? t.K2 / kTcChunkK : 1);
  if (sp > maxsp) sp = maxsp;
  if (p->tc_splits > 0) sp = p->tc_splits;
  // accuracy floor, also under an explicit choice: no CTA sums more than
  // kTcMaxChunksPerCta chunk results in FP32
  const int need = (int)((t.K2 + kTcChunkK * kTcMaxChunksPerCta - 1) / (kTcChunkK * kTcMaxChunksPerCta));
  if (sp < need) sp = need;
  if (sp > kTcMaxSplits) sp = kTcMaxSplits;
  if (sp * t.group > 65535) sp = 65535 / t.group;
  t.splits = sp < 1 ? 1 : sp;
  return t;
}

// Whether the FP64 contraction runs directly on the FP64 tensor cores.  The
// residues' cost hardly depends on the plane waves, the direct kernel's is in
// steps of 8, 16, 32 and 64.  Direct against residues, whole call: 13 orders,
// 50 problems of 2 048 elements, 60 modes 1.16 against 3.56 ms; 29 orders 1.67
// against 3.78 ms; 49 orders 3.41 against 4.19 ms; one of 20 000 elements, 400
// modes 2.02 against 4.33 ms (29), 3.83 against 4.55 ms (49).  A step of 96 lost:
// 5.54 against 4.85 ms at 81 orders.
constexpr int kDirectOrders = 64;
static bool ov_use_direct(const EmuOverlap *p) { return p->n_pw <= kDirectOrders; }

struct DirectPlan {
  long span, seg;      // elements of one E~ table, of a segment
  long per;            // of a CTA
  int fpp;             // folds per part: a segment's, or one
  int group, nsets, nt;
  int parts(long ne) const { return (int)((ne + (long)kOdFold * fpp - 1) / ((long)kOdFold * fpp)); }
  int per_seg() const { return (int)(seg / ((long)kOdFold * fpp)); }
};

constexpr size_t kDirectGroupBytes = (size_t)1 << 30;  // E~ tables of one group
constexpr size_t kDirectPartBytes = (size_t)1 << 29;   // its parts
constexpr long kOdSeg = 64, kOdSegs = 512;             // elements of a segment; segments before these double

static DirectPlan direct_plan(const EmuOverlap *p) {
  DirectPlan t;
  t.nsets = (p->d_sol1 ? 1 : 0) + (p->d_sol2 ? 1 : 0);
  if (t.nsets == 0) t.nsets = 2;
  t.nt = od_frags(p->n_pw);
  const size_t per_el = sizeof(double) * 12 * od_pitch(t.nt);
  long span = (long)(kDirectGroupBytes / per_el / kOdElems * kOdElems);
  if (p->elements_per_chunk > 0 && span > p->elements_per_chunk)
    span = (p->elements_per_chunk + kOdElems - 1) / kOdElems * kOdElems;
  t.span = span < p->nel ? span : p->nel;
  // segments: by the problem's own sizes, so that its sums do not depend on the batch.
  // With splits chosen for the batch's waves instead, 50 problems of 2 048 elements, 60
  // modes and 29 orders took 1.86 ms (1.67 here), 8 of them 0.33 (0.33), one of 20 000
  // elements and 60 modes 0.37 (0.48)
  const size_t part = sizeof(cd) * 2 * (size_t)t.nsets * p->nval * p->n_pw;
  auto count = [&](long per) { return (t.span + per - 1) / per; };
  t.seg = kOdSeg;
  while (count(t.seg) > 1 && (count(t.seg) > kOdSegs || count(t.seg) * part > kDirectPartBytes)) t.seg *= 2;
  long long g = (long long)std::min(kDirectGroupBytes / (per_el * (size_t)t.span),
                                    kDirectPartBytes / (count(t.seg) * part));
  if (g < 1) g = 1;
  if (g > p->batch) g = p->batch > 0 ? p->batch : 1;
  if (g > 1024) g = 1024;
  t.group = (int)g;
  // whole segments per CTA, or whole folds, whichever waves of CTAs (one per SM) take
  // less time: in elements (some 2 us), with six for a CTA's start and end and four
  // for each part that it writes
  const long long ctas = (long long)((p->nval + 63) / 64) * t.group * (t.nt > 4 ? t.nsets : 1);
  const int sms = emu::sm_count();
  double best = 0.0;
  t.per = 0;
  for (int fpp : {(int)(t.seg / kOdFold), 1}) {
    const long unit = (long)kOdFold * fpp;
    if (fpp == 1 && count(unit) * part * t.group > kDirectPartBytes) break;
    for (long n = 1; n <= 64 && (n == 1 || (n - 1) * unit < t.span); ++n) {
      const long per = n * unit;
      const double time = (double)((count(per) * ctas + sms - 1) / sms) * (double)(std::min(per, t.span) + 6 + 4 * n);
      if (!t.per || time < 0.97 * best) {
        best = time;
        t.per = per;
        t.fpp = fpp;
      }
    }
  }
  return t;
}

static size_t direct_bytes(const EmuOverlap *p, const DirectPlan &t) {
  const size_t npw = p->n_pw, G = t.group, rows = 2 * (size_t)t.nsets * p->nval;
  return align_up(sizeof(int32_t) * npw * G, 256) + align_up(sizeof(double) * 3 * npw * G, 256) +
         align_up(sizeof(cd) * npw * rows * G, 256) +
         (t.parts(t.span) > 1 ? align_up(sizeof(cd) * npw * rows * G * t.parts(t.span), 256) : 0) +
         align_up(sizeof(double) * 12 * od_pitch(t.nt) * t.span * G, 256) + 256;
}

static PwArgs pw_args(const EmuOverlap *p, int g0, int ng, int32_t *pos, double *tab) {
  PwArgs pa;
  pa.batch = ng;
  pa.npw = p->n_pw;
  pa.px = p->d_px;
  pa.py = p->d_py;
  pa.d = p->d;
  pa.dy = p->dy;
  pa.bloch = p->d_bloch + 2 * (size_t)g0;
  pa.k0 = p->d_k0 + g0;
  pa.pos = pos;
  pa.tab = tab;
  pa.zero = nullptr;
  pa.out_inv = p->d_index_pw_inv ? p->d_index_pw_inv + (size_t)g0 * p->n_pw : nullptr;
  return pa;
}

static EtArgs et_args(const EmuOverlap *p, int g0, const int32_t *pos, long e0, long ne) {
  EtArgs ea;
  ea.npw = p->n_pw;
  ea.mo = p->max_order;
  ea.e0 = (int)e0;
  ea.ne = (int)ne;
  ea.px = p->d_px;
  ea.py = p->d_py;
  ea.pos = pos;
  ea.x = p->d_x;
  ea.tn = p->d_table_nod;
  ea.d = p->d;
  ea.dy = p->dy;
  ea.bloch = p->d_bloch + 2 * (size_t)g0;
  ea.E = nullptr;
  ea.ldE = ea.sE = 0;
  ea.E2 = nullptr;
  ea.e2p = ea.e2n = 0;
  ea.A32 = nullptr;
  ea.spos = p->n_pw;
  ea.sA32 = 0;
  return ea;
}

static cudaError_t launch_etable(const EtArgs &ea, int ng, cudaStream_t s) {
  const size_t smem = kEtWarps * et_warp_bytes(ea.mo);
  if (smem > 48 * 1024) {
    const cudaError_t e =
        cudaFuncSetAttribute(etable_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  long long eg = (ea.ne + kEtWarps - 1) / kEtWarps;
  const long long egmax = (16LL * emu::sm_count() + ng - 1) / ng;
  if (eg > egmax) eg = egmax;
  etable_kernel<false><<<dim3((unsigned)eg, (unsigned)ng), 32 * kEtWarps, smem, s>>>(ea);
  return cudaSuccess;
}

static OutArgs out_args(const EmuOverlap *p, int g0, int nsets, const cd *H, const double *tab) {
  const long long M = p->nval, npw = p->n_pw;
  OutArgs o;
  o.H = H;
  o.sH = 2LL * nsets * M * npw;
  o.tab = tab;
  o.npw = (int)npw;
  o.nval = (int)M;
  o.nsets = nsets;
  o.inv_area = 1.0 / p->area_norm;
  o.scale = p->d_scale2 ? (const cd *)p->d_scale2 + (size_t)g0 * M : nullptr;
  o.perm = p->d_perm2 ? p->d_perm2 + (size_t)g0 * M : nullptr;
  o.J = p->d_J ? (cd *)p->d_J + (size_t)g0 * 2 * npw * M : nullptr;
  o.Jd = p->d_J_dag ? (cd *)p->d_J_dag + (size_t)g0 * 2 * npw * M : nullptr;
  return o;
}

static int overlap_direct(const EmuOverlap *p, void *ws, cudaStream_t s) {
  const DirectPlan t = direct_plan(p);
  const int npw = p->n_pw, M = p->nval, Gp = t.group;
  const long long rows = 2LL * t.nsets * M, ssol = (long long)p->nel * M * 39;
  char *w = (char *)ws;
  auto take = [&](size_t bytes) {
    char *r = w;
    w += align_up(bytes, 256);
    return (void *)r;
  };
  int32_t *pos = (int32_t *)take(sizeof(int32_t) * npw * Gp);
  double *tab = (double *)take(sizeof(double) * 3 * npw * Gp);
  cd *H = (cd *)take(sizeof(cd) * rows * npw * Gp);
  const bool many = t.parts(t.span) > 1;
  cd *part = many ? (cd *)take(sizeof(cd) * rows * npw * Gp * t.parts(t.span)) : H;
  double *E2 = (double *)w;
  for (int g0 = 0; g0 < p->batch; g0 += Gp) {
    const int ng = (p->batch - g0) < Gp ? (p->batch - g0) : Gp;
    pw_setup_kernel<<<ng, 256, sizeof(double) * npw, s>>>(pw_args(p, g0, ng, pos, tab));
    DirectArgs a;
    a.sol1 = p->d_sol1 ? (const cd *)p->d_sol1 + (size_t)g0 * ssol : nullptr;
    a.sol2 = p->d_sol2 ? (const cd *)p->d_sol2 + (size_t)g0 * ssol : nullptr;
    a.ssol = ssol;
    a.M = M;
    a.nsets = t.nsets;
    a.npw = npw;
    a.pitch = od_pitch(t.nt);
    a.per = t.per;
    a.fpp = t.fpp;
    a.E2 = E2;
    a.H = part;
    a.sPart = rows * npw * ng;
    for (long s0 = 0; s0 < p->nel; s0 += t.span) {
      a.e0 = s0;
      a.ne = (p->nel - s0) < t.span ? (p->nel - s0) : t.span;
      a.sE = 12LL * a.pitch * a.ne;
      a.add = !many && s0 > 0;
      EtArgs ea = et_args(p, g0, pos, s0, a.ne);
      ea.E2 = E2;
      ea.sE = a.sE;
      ea.e2p = a.pitch;
      ea.e2n = 8 * t.nt;
      if (launch_etable(ea, ng, s) != cudaSuccess) return EMU_E_CUDA;
      if (launch_direct_any(a, ng, s) != cudaSuccess) return EMU_E_CUDA;
      emu::note_launch(2);
      if (many) {
        reduce_parts_kernel<<<(unsigned)((a.sPart + 31) / 32), 256, 0, s>>>(H, part, a.sPart, t.parts(a.ne), t.per_seg(),
                                                                           s0 > 0);
        emu::note_launch();
      }
    }
    rows_epilogue_kernel<<<dim3((npw + 31) / 32, (M + 31) / 32, ng * t.nsets), 256, 0, s>>>(
        out_args(p, g0, t.nsets, H, tab));
    emu::note_launch(2);
  }
  return emu::check_launch();
}

// ---- residue path: problems in groups, one launch per step for a group
// One scale domain is a span of elements: the rows' scales hold over all of
// it, so that its chunks' residues add up and the CRT runs once per span.
struct RgOvPlan {
  long span, nec;  // elements per span (scales, E~) and per chunk (residues, one GEMM)
  int group, nsets, nblk, eparts;
  RgPlan g;        // shapes of a full chunk of a full group
};

constexpr size_t kRgGroupBytes = (size_t)2 << 30;  // E~ and residue planes of one group

static RgOvPlan rg_ov_plan(const EmuOverlap *p) {
  RgOvPlan t;
  t.nsets = (p->d_sol1 ? 1 : 0) + (p->d_sol2 ? 1 : 0);
  if (t.nsets == 0) t.nsets = 2;
  const int rows = 2 * t.nsets * p->nval;
  long chunk = p->elements_per_chunk > 0 ? p->elements_per_chunk : 4096;
  if (chunk > emu::kRgMaxK / 6) chunk = emu::kRgMaxK / 6;
  if (chunk > p->nel) chunk = p->nel;
  const long nch = (p->nel + chunk - 1) / chunk;
  // equal chunks of whole 128-byte lines
  t.nec = ((p->nel + nch - 1) / nch + 63) / 64 * 64;
  if (t.nec > p->nel) t.nec = p->nel;
  const size_t e_el = sizeof(cd) * 6 * (size_t)p->n_pw;
  long span = (long)((kRgGroupBytes / 2) / e_el / (size_t)t.nec) * t.nec;
  if (span < t.nec) span = t.nec;
  t.span = span < p->nel ? span : p->nel;
  const RgPlan one = emu::rg_plan(rows, p->n_pw, (int)(6 * t.nec), 1);
  long long g = (long long)(kRgGroupBytes / (e_el * t.span + (size_t)(one.bytesA + one.bytesB)));
  if (g < 1) g = 1;
  if (g > p->batch) g = p->batch > 0 ? p->batch : 1;
  if (g > 1024) g = 1024;
  t.group = (int)g;
  t.g = emu::rg_plan(rows, p->n_pw, (int)(6 * t.nec), t.group);
  t.nblk = (int)((t.span + kFnElems - 1) / kFnElems);
  t.eparts = (int)((6 * t.span + kErPart - 1) / kErPart);
  return t;
}

static size_t rg_ov_tiles(const EmuOverlap *p, const RgOvPlan &t) {
  return (2 * (size_t)t.nsets * p->nval + 63) / 64 * (((size_t)p->n_pw + 63) / 64);
}

static size_t rg_ov_bytes(const EmuOverlap *p, const RgOvPlan &t) {
  const size_t npw = p->n_pw, G = t.group, rows = 2 * (size_t)t.nsets * p->nval;
  // a smaller last chunk or group may take more K splits: at most kRgMaxSplits
  const size_t bytesC = (size_t)t.g.bytesC / t.g.nsplit * emu::kRgMaxSplits;
  return align_up(sizeof(int32_t) * npw * G, 256) + align_up(sizeof(double) * 3 * npw * G, 256) +
         align_up(sizeof(cd) * npw * rows * G, 256) + align_up(sizeof(cd) * npw * 6 * t.span * G, 256) +
         align_up(sizeof(double) * 2 * rows * t.nblk * G, 256) +
         align_up(sizeof(double) * 2 * npw * t.eparts * G, 256) + align_up(sizeof(RgScale) * rows * G, 256) +
         align_up(sizeof(RgScale) * npw * G, 256) + align_up((size_t)t.g.bytesA, 256) +
         align_up((size_t)t.g.bytesB, 256) + align_up(sizeof(int) * rg_ov_tiles(p, t) * G, 256) +
         align_up(bytesC, 256) + 512;
}

static int overlap_rg(const EmuOverlap *p, void *ws, cudaStream_t s) {
  const RgOvPlan t = rg_ov_plan(p);
  const int npw = p->n_pw, M = p->nval, Gp = t.group;
  const long long rows = 2LL * t.nsets * M;
  char *w = (char *)ws;
  auto take = [&](size_t bytes) {
    char *r = w;
    w += align_up(bytes, 256);
    return (void *)r;
  };
  int32_t *pos = (int32_t *)take(sizeof(int32_t) * npw * Gp);
  double *tab = (double *)take(sizeof(double) * 3 * npw * Gp);
  cd *H = (cd *)take(sizeof(cd) * rows * npw * Gp);
  cd *E = (cd *)take(sizeof(cd) * (size_t)npw * 6 * t.span * Gp);
  double *part = (double *)take(sizeof(double) * 2 * rows * t.nblk * Gp);
  double *epart = (double *)take(sizeof(double) * 2 * npw * t.eparts * Gp);
  RgScale *fs = (RgScale *)take(sizeof(RgScale) * rows * Gp);
  RgScale *es = (RgScale *)take(sizeof(RgScale) * npw * Gp);
  uint8_t *A = (uint8_t *)take((size_t)t.g.bytesA);
  uint8_t *B = (uint8_t *)take((size_t)t.g.bytesB);
  int *err = (int *)take(256);
  const size_t tiles = rg_ov_tiles(p, t);
  int *flags = (int *)take(sizeof(int) * tiles * Gp);
  uint8_t *C = (uint8_t *)w;
  if (cudaFuncSetAttribute(field_residue_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFcSmem) !=
      cudaSuccess)
    return EMU_E_CUDA;
  const long long ssol = (long long)p->nel * M * 39;
  for (int g0 = 0; g0 < p->batch; g0 += Gp) {
    const int ng = (p->batch - g0) < Gp ? (p->batch - g0) : Gp;
    PwArgs pa = pw_args(p, g0, ng, pos, tab);
    pa.zero = g0 == 0 ? err : nullptr;
    pw_setup_kernel<<<ng, 256, sizeof(double) * npw, s>>>(pa);
    emu::note_launch();
    int first = 1;
    for (long s0 = 0; s0 < p->nel; s0 += t.span) {
      const long sn = (p->nel - s0) < t.span ? (p->nel - s0) : t.span;
      FieldArgs f;
      f.sol1 = p->d_sol1 ? (const cd *)p->d_sol1 + (size_t)g0 * ssol : nullptr;
      f.sol2 = p->d_sol2 ? (const cd *)p->d_sol2 + (size_t)g0 * ssol : nullptr;
      f.ssol = ssol;
      f.M = M;
      f.nsets = t.nsets;
      f.nblk = (int)((sn + kFnElems - 1) / kFnElems);
      f.e0 = s0;
      f.ne = sn;
      f.part = part;
      f.scale = fs;
      f.A = A;
      f.flags = flags;
      f.kp = 0;
      field_norm_kernel<<<dim3((M + kFnModes - 1) / kFnModes, f.nblk, ng * t.nsets), 256, 0, s>>>(f);
      EtArgs ea = et_args(p, g0, pos, s0, sn);
      ea.E = E;
      ea.ldE = 6 * sn;
      ea.sE = 6LL * sn * npw;
      if (launch_etable(ea, ng, s) != cudaSuccess) return EMU_E_CUDA;
      const dim3 egrid(npw, (unsigned)((6 * sn + kErPart - 1) / kErPart), ng);
      erow_norm_kernel<<<egrid, 256, 0, s>>>(E, ea.sE, npw, 6LL * sn, epart);
      const long nrow = (long)(rows + npw) * ng;
      row_scale_kernel<<<(int)((nrow + 7) / 8), 256, 0, s>>>(part, f.nblk, (long)rows * ng, fs, epart, (int)egrid.y,
                                                             (long)npw * ng, es, flags, (long)(tiles * ng));
      emu::note_launch(4);
      // chunk by chunk: residues of both operands, then their products, added
      // up modulo p.  All chunks use the K splits of the first one.
      RgPlan gp{};
      for (long c0 = 0; c0 < sn; c0 += t.nec) {
        const long ne = (sn - c0) < t.nec ? (sn - c0) : t.nec;
        const RgPlan cp = emu::rg_plan((int)rows, npw, (int)(6 * ne), ng, c0 ? gp.nsplit : 0);
        if (c0 == 0) gp = cp;
        FieldArgs fc = f;
        fc.e0 = s0 + c0;
        fc.ne = ne;
        fc.kp = cp.kp;
        field_residue_kernel<<<dim3((M + kFcModes - 1) / kFcModes,
                                    (unsigned)((cp.kp + 6 * kFcElems - 1) / (6 * kFcElems)), ng * t.nsets),
                               kFcThreads, kFcSmem, s>>>(fc);
        erow_residue_kernel<<<dim3(npw, (cp.kp + 1023) / 1024, ng), 256, 0, s>>>(E + 6 * c0, ea.sE, ea.ldE, npw,
                                                                                   6LL * ne, cp.kp, es, B);
        emu::note_launch(2);
        const int st = emu::rg_mma(cp, A, B, C, c0 > 0, err, s);
        if (st != EMU_OK) return st;
      }
      const long long items = rows * (gp.ldn / 4);
      field_crt_kernel<<<dim3((unsigned)((items + 127) / 128), (unsigned)ng), 128, 0, s>>>(
          f, C, gp.ldn, gp.nsplit, npw, es, H, first, err);
      field_left_kernel<<<dim3((npw + 63) / 64, (unsigned)((rows + 63) / 64), ng), kDLThreads, 0, s>>>(
          f, C, gp.ldn, gp.nsplit, npw, es, E, ea.sE, H, first);
      emu::note_launch(2);
      first = 0;
    }
    rows_epilogue_kernel<<<dim3((npw + 31) / 32, (M + 31) / 32, ng * t.nsets), 256, 0, s>>>(out_args(p, g0, t.nsets, H, tab));
    emu::note_launch();
  }
  return emu::check_launch();
}

extern "C" size_t emu_overlap_workspace_size(const EmuOverlap *p) {
  if (!p || p->n_pw < 1 || p->nval < 1 || p->nel < 1 || p->batch < 0) return 0;
  if (p->precision == 1) {
    const TcPlan t = tc_plan(p);
    return (size_t)t.group * tc_problem_bytes(p, t) + 16 * 256 + 256;
  }
  return ov_use_direct(p) ? direct_bytes(p, direct_plan(p)) : rg_ov_bytes(p, rg_ov_plan(p));
}

// Tensor-core J / J_dag for all problems, `group` problems per launch: plane
// waves, per element chunk the E~ table (as the FP32 A operand) and B (both
// field sets), one batched tcgen05 GEMM, the split sums folded into G / G_dag,
// then the epilogues.
static int overlap_tc(const EmuOverlap *p, void *ws, cudaStream_t s) {
  const TcPlan t = tc_plan(p);
  const int npw = p->n_pw, M = p->nval, Gp = t.group;
  const long long gsz = (long long)npw * 2 * M;
  char *w = (char *)ws;
  auto take = [&](size_t bytes) {
    char *r = w;
    w += align_up(bytes, 256);
    return (void *)r;
  };
  int32_t *pos = (int32_t *)take(sizeof(int32_t) * npw * Gp);
  double *tab = (double *)take(sizeof(double) * 3 * npw * Gp);
  cd *G = (cd *)take(sizeof(cd) * gsz * Gp);
  cd *Gd = (cd *)take(sizeof(cd) * gsz * Gp);
  float *A32 = (float *)take(sizeof(float) * 2 * npw * t.K2 * Gp);
  float *B32 = (float *)take(sizeof(float) * t.nb * t.K2 * Gp);
  float *Cpart = (float *)take(sizeof(float) * t.splits * 2 * npw * (size_t)t.nb * Gp);
  int *terr = p->d_error ? (int *)p->d_error : (int *)take(256);
  if (!p->d_error && cudaMemsetAsync(terr, 0, sizeof(int), s) != cudaSuccess) return EMU_E_CUDA;
  const int sms = emu::sm_count();
  const size_t et_smem32 = kEtWarps * et_warp_bytes_f32(p->max_order);
  if (et_smem32 > 48 * 1024 &&
      cudaFuncSetAttribute(etable_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)et_smem32) !=
          cudaSuccess)
    return EMU_E_CUDA;
  const long long ssol = (long long)p->nel * M * 39;
  const cd *sol1 = (const cd *)p->d_sol1, *sol2 = (const cd *)p->d_sol2;
  for (int g0 = 0; g0 < p->batch; g0 += Gp) {
    const int ng = (p->batch - g0) < Gp ? (p->batch - g0) : Gp;
    PwArgs pa;
    pa.batch = ng;
    pa.npw = npw;
    pa.px = p->d_px;
    pa.py = p->d_py;
    pa.d = p->d;
    pa.dy = p->dy;
    pa.bloch = p->d_bloch + 2 * (size_t)g0;
    pa.k0 = p->d_k0 + g0;
    pa.pos = pos;
    pa.tab = tab;
    pa.zero = nullptr;
    pa.out_inv = p->d_index_pw_inv ? p->d_index_pw_inv + (size_t)g0 * npw : nullptr;
    pw_setup_kernel<<<ng, 256, sizeof(double) * npw, s>>>(pa);
    emu::note_launch();
    int first = 1;
    for (long e0 = 0; e0 < p->nel; e0 += t.nec) {
      const long ne = (p->nel - e0) < t.nec ? (p->nel - e0) : t.nec;
      const long long K2 = 12 * (long long)ne;
      EtArgs ea;
      ea.npw = npw;
      ea.mo = p->max_order;
      ea.e0 = (int)e0;
      ea.ne = (int)ne;
      ea.px = p->d_px;
      ea.py = p->d_py;
      ea.pos = pos;
      ea.x = p->d_x;
      ea.tn = p->d_table_nod;
      ea.d = p->d;
      ea.dy = p->dy;
      ea.bloch = p->d_bloch + 2 * (size_t)g0;
      ea.E = nullptr;
      ea.ldE = 6 * ne;
      ea.sE = 0;
      ea.E2 = nullptr;
      ea.A32 = A32;
      ea.spos = npw;
      ea.sA32 = 2LL * npw * K2;
      long long eg = (ne + kEtWarps - 1) / kEtWarps;
      const long long egmax = (16LL * sms + ng - 1) / ng;
      if (eg > egmax) eg = egmax;
      etable_kernel<true><<<dim3((unsigned)eg, (unsigned)ng), 32 * kEtWarps, et_smem32, s>>>(ea);
      const dim3 bg((M + kBModes - 1) / kBModes, (unsigned)((ne + kBElems - 1) / kBElems), (unsigned)ng);
      const long long sB = (long long)t.nb * K2;
      if (p->field_c64) {
        const cf32 *f1 = (const cf32 *)p->d_sol1, *f2 = (const cf32 *)p->d_sol2;
        if (f1) make_B_kernel<cf32><<<bg, 256, 0, s>>>(f1 + (size_t)g0 * ssol, ssol, M, e0, ne, 0, 0, B32, sB);
        if (f2)
          make_B_kernel<cf32><<<bg, 256, 0, s>>>(f2 + (size_t)g0 * ssol, ssol, M, e0, ne, 1, t.off1, B32, sB);
      } else {
        if (sol1) make_B_kernel<cd><<<bg, 256, 0, s>>>(sol1 + (size_t)g0 * ssol, ssol, M, e0, ne, 0, 0, B32, sB);
        if (sol2)
          make_B_kernel<cd><<<bg, 256, 0, s>>>(sol2 + (size_t)g0 * ssol, ssol, M, e0, ne, 1, t.off1, B32, sB);
      }
      emu::note_launch(1 + (sol1 ? 1 : 0) + (sol2 ? 1 : 0));
      int used = 0;
      const int tst = emu::tc_gemm_tf32x3_parts(A32, 2LL * npw * K2, B32, sB, 2 * npw, t.nb, (int)K2, ng, t.splits,
                                                Cpart, terr, &used, s);
      if (tst != EMU_OK) return tst;
      long long rgs = (gsz + 255) / 256;
      if (rgs > 1024) rgs = 1024;
      pack_G_parts_kernel<<<dim3((unsigned)rgs, (unsigned)ng), 256, 0, s>>>(
          Cpart, used, npw, t.nb, 2 * M, sol1 ? G : nullptr, sol2 ? Gd : nullptr, gsz, t.off1, first);
      emu::note_launch();
      first = 0;
    }
    long long eb = ((long long)npw * M + 255) / 256;
    if (eb > 1024) eb = 1024;
    if (sol1) {
      epilogue_kernel<<<dim3((unsigned)eb, (unsigned)ng), 256, 0, s>>>(
          G, tab, npw, M, 1.0 / p->area_norm, 0, nullptr, nullptr, (cd *)p->d_J + (size_t)g0 * 2 * npw * M);
      emu::note_launch();
    }
    if (sol2) {
      epilogue_kernel<<<dim3((unsigned)eb, (unsigned)ng), 256, 0, s>>>(
          Gd, tab, npw, M, 1.0, 1, p->d_scale2 ? (const cd *)p->d_scale2 + (size_t)g0 * M : nullptr,
          p->d_perm2 ? p->d_perm2 + (size_t)g0 * M : nullptr, (cd *)p->d_J_dag + (size_t)g0 * 2 * npw * M);
      emu::note_launch();
    }
  }
  return emu::check_launch();
}

// No field set: the plane-wave order alone (d_index_pw_inv).
static int overlap_order(const EmuOverlap *p, void *ws, int group, cudaStream_t s) {
  int32_t *pos = (int32_t *)ws;
  double *tab = (double *)((char *)ws + align_up(sizeof(int32_t) * p->n_pw * (size_t)group, 256));
  for (int g0 = 0; g0 < p->batch; g0 += group) {
    const int ng = p->batch - g0 < group ? p->batch - g0 : group;
    pw_setup_kernel<<<ng, 256, sizeof(double) * p->n_pw, s>>>(pw_args(p, g0, ng, pos, tab));
    emu::note_launch();
  }
  return emu::check_launch();
}

extern "C" int emu_overlap_batch(const EmuOverlap *p, void *d_workspace, size_t workspace_bytes,
                                 void *stream) {
  if (!p) return EMU_E_ARG;
  if (p->batch < 0 || p->nval < 1 || p->nel < 1 || p->npt < 3 || p->n_pw < 1) return EMU_E_SHAPE;
  if (!p->d_px || !p->d_py || !p->d_x || !p->d_table_nod || !p->d_bloch || !p->d_k0) return EMU_E_ARG;
  if (!(p->d > 0) || !(p->dy > 0) || !(p->area_norm > 0)) return EMU_E_ARG;
  if ((p->d_sol1 == nullptr) != (p->d_J == nullptr) || (p->d_sol2 == nullptr) != (p->d_J_dag == nullptr))
    return EMU_E_ARG;
  if (p->max_order < 0 || p->max_order > kMaxOrd) return EMU_E_UNSUPPORTED;
  if (p->precision != 0 && p->precision != 1) return EMU_E_ARG;
  if (p->tc_splits < 0) return EMU_E_ARG;
  if (p->field_c64 != 0 && p->field_c64 != 1) return EMU_E_ARG;
  if (p->field_c64 && p->precision != 1) return EMU_E_UNSUPPORTED;  // the FP64 path reads complex128
  if (p->batch == 0) return EMU_OK;
  if (!d_workspace || workspace_bytes < emu_overlap_workspace_size(p)) return EMU_E_WORKSPACE;
  int st = upload_tables();
  if (st != EMU_OK) return st;
  cudaStream_t s = (cudaStream_t)stream;
  if (!p->d_sol1 && !p->d_sol2) {
    const int group = p->precision == 1 ? tc_plan(p).group
                      : ov_use_direct(p) ? direct_plan(p).group
                                         : rg_ov_plan(p).group;
    return overlap_order(p, d_workspace, group, s);
  }
  if (p->precision == 1) return overlap_tc(p, d_workspace, s);
  return ov_use_direct(p) ? overlap_direct(p, d_workspace, s) : overlap_rg(p, d_workspace, s);
}

// ---------------------------------------------------------------- normalisation
extern "C" size_t emu_mode_overlap_workspace_size(const EmuNormalise *p) {
  if (!p || p->nval < 1 || p->nel < 1 || p->batch < 0) return 0;
  const long long nch = (p->nel + kDiagChunk - 1) / kDiagChunk;
  const long long B = p->batch > 0 ? p->batch : 1;
  return align_up(sizeof(double) * 264 * (size_t)p->nel, 256) +
         align_up(sizeof(cd) * B * nch * p->nval, 256) + 256;
}

extern "C" int emu_mode_overlap_diag(const EmuNormalise *p, void *d_workspace, size_t workspace_bytes,
                                     void *stream) {
  if (!p) return EMU_E_ARG;
  if (p->batch < 0 || p->nval < 1 || p->nel < 1) return EMU_E_SHAPE;
  if (!p->d_x || !p->d_table_nod || !p->d_type_el || !p->d_pp || !p->d_k0 || !p->d_beta1 ||
      !p->d_sol1 || !p->d_sol2 || !p->d_diag || !p->d_scale || !p->d_n_small)
    return EMU_E_ARG;
  if (p->batch == 0) return EMU_OK;
  if (p->batch > 65535) return EMU_E_SHAPE;
  if (!d_workspace || workspace_bytes < emu_mode_overlap_workspace_size(p)) return EMU_E_WORKSPACE;
  int st = upload_tables();
  if (st != EMU_OK) return st;
  cudaStream_t s = (cudaStream_t)stream;
  const long nch = (p->nel + kDiagChunk - 1) / kDiagChunk;
  double *ms_all = (double *)d_workspace;
  cd *part = (cd *)((char *)d_workspace + align_up(sizeof(double) * 264 * (size_t)p->nel, 256));
  if (cudaMemsetAsync(p->d_n_small, 0, sizeof(int32_t) * p->batch, s) != cudaSuccess) return EMU_E_CUDA;
  const int sms = emu::sm_count();
  const long eb = (p->nel + 127) / 128;
  elem_scal_kernel<<<(int)(eb < 8 * sms ? eb : 8 * sms), 128, 0, s>>>(p->d_x, p->d_table_nod, p->nel, ms_all);
  DiagArgs a;
  a.nval = p->nval;
  a.nel = p->nel;
  a.ms_all = ms_all;
  a.type_el = p->d_type_el;
  a.pp = (const cd *)p->d_pp;
  a.sol1 = (const cd *)p->d_sol1;
  a.sol2 = (const cd *)p->d_sol2;
  a.k0 = p->d_k0;
  a.part = part;
  diag_kernel<<<dim3((unsigned)nch, (unsigned)p->batch), 128, 0, s>>>(a);
  const long nt = (long)p->batch * p->nval;
  const long fb = (nt + 127) / 128;
  diag_finish_kernel<<<(int)(fb < 8 * sms ? fb : 8 * sms), 128, 0, s>>>(
      part, (int)nch, p->nval, p->batch, (const cd *)p->d_beta1, (cd *)p->d_diag, (cd *)p->d_scale,
      p->d_n_small);
  emu::note_launch(3);
  return emu::check_launch();
}

extern "C" size_t emu_mode_overlap_reorder_workspace_size(const EmuNormalise *p) {
  if (!p || p->nval < 1 || p->nel < 1) return 0;
  return align_up(sizeof(double) * 264 * (size_t)p->nel, 256) +
         align_up(sizeof(cd) * (size_t)p->nval * p->nval, 256) + 256;
}

extern "C" int emu_mode_overlap_reorder(const EmuNormalise *p, int32_t *d_perm, int32_t *d_warn,
                                        void *d_workspace, size_t workspace_bytes, void *stream) {
  if (!p) return EMU_E_ARG;
  if (p->batch < 0 || p->nval < 1 || p->nel < 1) return EMU_E_SHAPE;
  if (!p->d_x || !p->d_table_nod || !p->d_type_el || !p->d_pp || !p->d_k0 || !p->d_beta1 ||
      !p->d_sol1 || !p->d_sol2 || !p->d_diag || !p->d_scale || !d_perm || !d_warn)
    return EMU_E_ARG;
  if (p->batch == 0) return EMU_OK;
  if (!d_workspace || workspace_bytes < emu_mode_overlap_reorder_workspace_size(p)) return EMU_E_WORKSPACE;
  int st = upload_tables();
  if (st != EMU_OK) return st;
  cudaStream_t s = (cudaStream_t)stream;
  double *ms_all = (double *)d_workspace;
  cd *ovl = (cd *)((char *)d_workspace + align_up(sizeof(double) * 264 * (size_t)p->nel, 256));
  const int sms = emu::sm_count();
  elem_scal_kernel<<<(int)((p->nel + 127) / 128 < 8 * sms ? (p->nel + 127) / 128 : 8 * sms), 128, 0, s>>>(
      p->d_x, p->d_table_nod, p->nel, ms_all);
  emu::note_launch();
  for (int b = 0; b < p->batch; ++b) {
    const size_t off = (size_t)b * p->nel * p->nval * 39;
    const long tot = (long)p->nval * p->nval;
    ovl_full_kernel<<<(int)((tot + 127) / 128 < 16 * sms ? (tot + 127) / 128 : 16 * sms), 128, 0, s>>>(
        ms_all, p->nval, p->nel, p->d_type_el, (const cd *)p->d_pp, p->d_k0 + b,
        (const cd *)p->d_beta1 + (size_t)b * p->nval, (const cd *)p->d_sol1 + off,
        (const cd *)p->d_sol2 + off, ovl);
    pair_swap_kernel<<<1, 32, 0, s>>>(ovl, p->nval, d_perm + (size_t)b * p->nval,
                                       (cd *)p->d_diag + (size_t)b * p->nval,
                                       (cd *)p->d_scale + (size_t)b * p->nval, d_warn + b);
    emu::note_launch(2);
  }
  return emu::check_launch();
}
