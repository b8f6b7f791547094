// Per-order film recursion shared by the film kernels (uniform batches in
// film_stack.cu, heterogeneous batches in film_varlen.cu): impedances,
// Fresnel interfaces, the bottom-to-top cascade of one plane-wave order for
// both polarisations and, for orders carrying incident light, the
// top-to-bottom flux pass (backend/mode_calcs.py:199-218, 451-477;
// backend/stack.py:196-366).
#pragma once
#include "emu_cplx.cuh"
#include "emu_fastmath.cuh"
#include "emu_internal.h"
#include "emu_modes.cuh"

namespace emu {

constexpr int kSave = 5;  // saved scalars per (layer, polarisation)

struct LayerC {
  cd k, zcr, ik;  // wavenumber, 1/n, 1/k
  cd n, nn;       // n, n^2
  cd kk;          // k^2, rounded as kz_arg rounds it
};

// Shared-memory layout of one point's slot (byte offsets); a slot sized for
// (npw, L) also holds any point with fewer orders and layers.
struct SlotSmem {
  int keys, rank, wood, nprop, acc, lay, h, misc, ws, stride;
};

// with_ws: room for the flux-pass scalars of the one order that carries
// light ([L][2][kSave]), for every polarisation but incoming amplitudes
// (whose scalars, one set per order, stay in the global workspace).
__host__ __device__ inline SlotSmem slot_layout(int npw, int L, bool with_ws = true) {
  SlotSmem s;
  int o = 0;
  s.lay = o; o += (int)sizeof(LayerC) * L;
  s.ws = o; o += with_ws ? (int)sizeof(cd) * L * 2 * kSave : 0;
  s.acc = o; o += 16 * (L + 1);
  s.keys = o; o += 8 * npw;
  s.h = o; o += 8 * (L - 1);  // heights, then k_air
  s.rank = o; o += 4 * npw;
  s.nprop = o; o += 4 * (L + 1);
  s.wood = o; o += 4 * ((L + 1 + 31) / 32);
  s.misc = o; o += 16;  // [0] specular order, [1] layer-Wood flag, [2] non-finite list entry
  s.stride = (o + 15) / 16 * 16;
  return s;
}

// any() is a sync() that also returns whether v holds for any thread.
// Thread teams that solve one point together: a whole CTA's slot (uniform
// batches, barriers over the CTA) or one warp (heterogeneous batches).
struct CtaTeam {
  int lt, size;
  __device__ void sync() const { __syncthreads(); }
  __device__ bool any(bool v) const { return __syncthreads_or(v) != 0; }
};
struct WarpTeam {
  int lt;
  static constexpr int size = 32;
  __device__ void sync() const { __syncwarp(); }
  __device__ bool any(bool v) const {
    __syncwarp();
    return __any_sync(0xffffffffu, v) != 0;
  }
};

// A point accessor P (FilmPointCtx-like) exposes, as member functions:
//   L() npw() world_1d() pol() ncoord() slot_per_order() dy() period()
//   inv_sqrt2(), px() py() (order lists), incoming() ([P] or unused),
//   shears() ([L][2] or NULL), ws() ([n_slots][L][2][kSave] workspace),
//   R_net() T_net() ([P]), kz() ([L][npw] or NULL), layer_rt() ([L][2][P]
//   or NULL), vcd() vcu() ([L][P], [L-1][P] or NULL).
// Accessors compute these from kernel parameters on demand, so the
// recursion holds no per-point pointers in registers.
template <class Pt>
__device__ __forceinline__ cd incidence(const Pt &c, int pos, int spec) {
  const int pol = c.pol(), npw = c.npw();
  if (pol == EMU_POL_INCOMING) {
    const emu_c128 v = c.incoming()[pos];
    return cd{v.re, v.im};
  }
  const bool te = (pos == spec), tm = (pos == spec + npw);
  switch (pol) {
    case EMU_POL_TE: return te ? cd{1.0, 0.0} : cd{0.0, 0.0};
    case EMU_POL_TM: return tm ? cd{1.0, 0.0} : cd{0.0, 0.0};
    case EMU_POL_UN: return (te || tm) ? cd{c.inv_sqrt2(), 0.0} : cd{0.0, 0.0};
    case EMU_POL_RCIRC: return te ? cd{c.inv_sqrt2(), 0.0} : (tm ? cd{0.0, c.inv_sqrt2()} : cd{0.0, 0.0});
    case EMU_POL_LCIRC: return te ? cd{c.inv_sqrt2(), 0.0} : (tm ? cd{0.0, -c.inv_sqrt2()} : cd{0.0, 0.0});
  }
  return cd{0.0, 0.0};
}

__device__ __forceinline__ void store_c(emu_c128 *p, size_t i, cd v) {
  p[i] = emu_c128{v.x, v.y};
}

// U-weighted flux contribution of one order and polarisation
// (backend/stack.py:311-321, 351): propagating orders give |f-|^2 - |f+|^2,
// evanescent ones the cross terms with -+i.
__device__ __forceinline__ cd flux_term(cd fm, cd fp, bool prop, bool tm) {
  if (prop) return cd{cabs2(fm) - cabs2(fp), 0.0};
  // TE: conj(fm)(-i)fp + conj(fp)(i)fm ; TM: conj(fm)(i)fp + conj(fp)(-i)fm
  const cd a = cmul(cconj(fm), fp);
  const cd b = cmul(cconj(fp), fm);
  const cd d = csub(b, a);
  const cd te = cd{-d.y, d.x};
  return tm ? cneg(te) : te;
}

// Transmission coefficient T12 = T21 of the air / layer interface for
// polarisation q (0 TE, 1 TM): 2 sqrt(z2) sqrt(z1) / (z2 + z1) with the
// impedances z1 of air and z2 of the layer (backend/mode_calcs.py:199-218,
// 451-477), principal square roots as numpy takes them.
__device__ __forceinline__ cd t12_exact(const LayerC &c, cd kz, double kair, cd kz_air, int q) {
  cd z1, z2;
  if (q == 0) {
    z1 = cscale(crcp_nr(kz_air), kair);
    z2 = cmul(c.zcr, cmul(c.k, crcp_nr(kz)));
  } else {
    z1 = cscale(kz_air, 1.0 / kair);
    z2 = cmul(c.zcr, cmul(kz, c.ik));
  }
  const cd is = crcp_nr(cadd(z2, z1));
  return cmul(cscale(cmul(csqrt_k(z2), csqrt_k(z1)), 2.0), is);
}

// A pair (Z, V) or its companion num outside 2^+-60 is brought back by an exact
// power of two; e collects the exponents.  Called every fourth layer, and before
// and after a layer of |p| >= 2 (see solve_order): between two calls the pair grows by
// at most (8 |t| (|t| + |n^2|))^4, inside the range of a double up to |n| and |t| of
// 1e18, or by 2 |p| |t| (|t| + |n^2|) in one layer.
__device__ __forceinline__ int top_exp(cd a) {
  return max(__double2hiint(a.x) & 0x7fffffff, __double2hiint(a.y) & 0x7fffffff) >> 20;
}
__device__ __forceinline__ double pow2(int e) { return __hiloint2double((1023 + e) << 20, 0); }
__device__ __forceinline__ void renorm(cd &Z, cd &V, cd &num, int &e) {
  const int a = max(top_exp(Z), top_exp(V)), b = top_exp(num);
  if ((unsigned)(a - 963) > 120u && a > 0 && a < 2047) {
    // two halves: a factor itself stays normal
    const int h = (1023 - a) / 2, g = 1023 - a - h;
    const double f = pow2(h), k = pow2(g);
    Z = cscale(cscale(Z, f), k);
    V = cscale(cscale(V, f), k);
    e += 1023 - a;
  }
  if ((unsigned)(b - 963) > 120u && b > 0 && b < 2047) {
    const int h = (1023 - b) / 2, g = 1023 - b - h;
    num = cscale(cscale(num, pow2(h)), pow2(g));
    e -= 1023 - b;
  }
}

// alpha^2 and beta^2 of an order at k_parallel scaled by 1 - 1e-9 (Wood
// anomalies).  Out of line: the cascade keeps its registers for the usual case.
static __device__ __noinline__ double2 wood_squares(int world_1d, double dy, int px, int py, double a0, double b0) {
  double al, be;
  order_ab(world_1d, dy, px, py, (1 - 1e-9) * a0, (1 - 1e-9) * b0, al, be);
  return make_double2(__dmul_rn(al, al), __dmul_rn(be, be));
}

// Cascade of one order (both polarisations) bottom to top, then, if the
// order carries incident light, its flux pass top to bottom.
//
// The reference builds each interface from the impedances z1 of air and z2 of
// the layer, R12 = (z2 - z1)/(z2 + z1), T12 = T21 = 2 sqrt(z2 z1)/(z2 + z1), and
// runs the recursion of backend/stack.py:229-278 on them.  Here:
//  * z2 : z1 = A : B with A = 1, B = t (TE) and A = t, B = n^2 (TM), where
//    t = k_z / k_z,air: a common factor of A and B changes nothing below;
//  * the reflection below a gap is carried as a pair, rnet = (Z - V)/(Z + V).
//    With p = exp(i k_z h) the gap and layer steps of the reference,
//      rg = T12 (1 - R12 rq)^-1 T21 rq - R12,   (air gap, rq = rnet below)
//      rnet' = R12 + T12 p rg p (1 + R12 p rg p)^-1 T21,
//    are then X = A V, Y = B Z, u = X + Y, v = Y - X, w = p^2 v (rg = v/u) and
//      Z' = A (u + w),  V' = B (u - w),
//    without a division;
//  * the transmission through gap and layer is x1 p x2 = 2 A B p (Z + V)/(Z' + V'),
//    so num = tnet (Z + V) takes a factor 2 A B p per layer, and tnet is formed
//    once, in the superstrate.  There and in the substrate the square roots of
//    z1 multiply to z1 itself.
// So a layer costs about 80 FP64 operations for both polarisations where the
// quotient N/D per layer and polarisation took 170, beside the square root for
// k_z and the exponential.  32 768 points x 10 films x 81 orders, 256 threads x 3
// CTAs: 1 040 us before, 840 us now, of which 48 us per film (56 before) and
// 350 us for the phases around the recursion (480 before); the kernel
// is bound by the issue and latency of 16 to 24 warps per SM (54 % of the issue
// slots, 38 % of the FP64 pipe).  Against 64-bit results of higher precision the
// outputs are 4.2e-15 off, with the quotients 4.3e-15.
// The order that carries light also takes the quotients per layer, which the
// flux pass needs; the optional per-layer outputs (layer_rt, vec_coef) take T12
// itself from t12_exact.  Every result is the same whichever optional outputs
// are requested.
// kRare: some layer of the point is at a Wood anomaly, or some film has Im n^2 < 0
// (gain, or a negative real part): its evanescent orders grow, |p| > 1 without bound.
// Such a layer takes u 2^-e, w = (p 2^-e) p v and f = 2 A B p 2^-e with e the exponent
// of |p|: pair and num carry the same exact factor, which cancels in x1 p x2, and
// the pair grows by |p| where p^2 would overflow after a few layers.
// A second copy of the cascade keeps both out of the usual one (862 -> 840 us at the
// size above for the first; 836 us with both).
template <bool kRare, class Pt>
__device__ __forceinline__ void solve_order(const Pt &p, int u, int j, int spec, const LayerC *lay,
                            const double *hsm, const unsigned *wood, bool wood_air,
                            double a0, double b0, int np_air, int np_in, int np_out, cd *acc,
                            int *nprop, bool count, cd *ws_smem) {
  const int L = p.L(), npw = p.npw(), P = 2 * npw;
  const double kair = hsm[L - 2];
  const int px = p.px()[u], py = p.py()[u];
  double al2, be2;
  {
    double al, be;
    order_ab(p.world_1d(), p.dy(), px, py, a0, b0, al, be);
    al2 = __dmul_rn(al, al);
    be2 = __dmul_rn(be, be);
  }
  // alpha^2, beta^2 with k_parallel as given or (at a Wood anomaly) scaled
  auto squares = [&](bool scaled) -> double2 {
    return scaled ? wood_squares(p.world_1d(), p.dy(), px, py, a0, b0) : make_double2(al2, be2);
  };
  cd kz_air;
  {
    const double2 w = squares(wood_air);
    kz_air = csqrt_k(kz_arg_sq(k_squared(cd{kair, 0.0}), w.x, w.y));
  }
  const double *sh = p.shears();
  double al_sh = 0.0, be_sh = 0.0;
  if (sh)
    order_ab(p.world_1d(), p.dy(), p.px()[j], p.py()[j], wood_air ? (1 - 1e-9) * a0 : a0,
             wood_air ? (1 - 1e-9) * b0 : b0, al_sh, be_sh);
  const cd din[2] = {incidence(p, j, spec), incidence(p, j + npw, spec)};
  // k_z,air is real or imaginary: t = k_z / k_z,air with one correction step, so
  // that a layer of air has t = 1 exactly
  const bool ev = kz_air.y != 0.0;
  const double ka = ev ? kz_air.y : kz_air.x, ra = rcp_nr(ka);
  auto ratio = [&](cd kz) -> cd {
    const double x = ev ? kz.y : kz.x, y = ev ? -kz.x : kz.y;
    cd t = cd{x * ra, y * ra};
    t.x = fma(fma(-t.x, ka, x), ra, t.x);
    t.y = fma(fma(-t.y, ka, y), ra, t.y);
    return t;
  };
  const bool active = !cis_zero(din[0]) || !cis_zero(din[1]);
  const bool want_vec = p.vcd() != nullptr;
  const bool all_t = want_vec || p.layer_rt() != nullptr;
  // polarisations whose scalars the flux pass reads
  const bool act[2] = {want_vec ? active : !cis_zero(din[0]), want_vec ? active : !cis_zero(din[1])};
  // flux-pass scalars: in the point's shared-memory slot when one order
  // carries light, else per order in the global workspace
  cd *wsv = p.slot_per_order() ? p.ws() + ((size_t)u * L) * 2 * kSave : ws_smem;
  // k_z of the order in layer l (also stored when requested)
  auto layer_kz = [&](int l) -> cd {
    const double2 w = squares(kRare && ((wood[l >> 5] >> (l & 31)) & 1u));
    const cd kz = csqrt_k(kz_arg_sq(lay[l].kk, w.x, w.y));
    if (p.kz()) store_c(p.kz(), (size_t)l * npw + j, kz);
    return kz;
  };
  // shear phase Q of the gap below layer l and its inverse (backend/stack.py:236-244, 267-275)
  auto shear_q = [&](int l, cd &Q, cd &Qi) {
    Q = cd{1.0, 0.0};
    Qi = cd{1.0, 0.0};
    if (!sh) return;
    double c0, c1;
    if (l < L - 1) {
      c0 = sh[2 * (l - 1)] - sh[2 * l];
      c1 = sh[2 * (l - 1) + 1] - sh[2 * l + 1];
    } else {
      c0 = sh[2 * l];
      c1 = sh[2 * l + 1];
    }
    Q = shear_phase(al_sh, be_sh, c0, c1, p.ncoord());
    Qi = shear_phase(al_sh, be_sh, -1 * c0, -1 * c1, p.ncoord());
  };
  auto store_rt = [&](int l, int q, cd R12, cd T12) {
    if (!p.layer_rt()) return;
    const size_t o = (size_t)l * 2 * P;
    store_c(p.layer_rt(), o + j + q * npw, R12);
    store_c(p.layer_rt(), o + P + j + q * npw, T12);
  };
  // sqrt(z2) (A + B) k_z,air^(1/2) / 2 of an outer layer without its common
  // factors: sqrt(k_z) (TE) and +-sqrt(k_z) n (TM); the sign makes sqrt(k_z) / n the
  // principal root of its square
  auto root = [&](const LayerC &c, cd kz, cd f[2]) {
    f[0] = csqrt_k(kz);
    f[1] = cmul(f[0], c.n);
    if (fma(f[0].x, c.n.x, f[0].y * c.n.y) < 0.0) f[1] = cneg(f[1]);
  };
  // k_z,air^(-1/2), for the order that carries light
  cd isq = cd{0.0, 0.0};
  if (active) {
    const double r = sqrt(fabs(ra));
    isq = ev ? cd{r * 0.70710678118654752440, -copysign(r, ra) * 0.70710678118654752440} : cd{r, 0.0};
  }
  cd Z[2], V[2], num[2], tnet[2], rnet[2];
  int ex[2] = {0, 0};
  // substrate (l = 0)
  {
    const LayerC c = lay[0];
    const cd kz = layer_kz(0);
    cd t = ratio(kz);
    t.x += c.zcr.x - c.zcr.x;  // n = 0 has no impedance
    Z[0] = cd{1.0, 0.0};
    V[0] = t;
    Z[1] = t;
    V[1] = c.nn;
    root(c, kz, num);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      if (!act[q] && !all_t) continue;
      const cd is = crcp_nr(cadd(Z[q], V[q]));
      const cd R12 = cmul(csub(Z[q], V[q]), is);
      if (all_t) store_rt(0, q, R12, t12_exact(c, kz, kair, kz_air, q));
      if (act[q]) {
        cd *sv = wsv + (size_t)q * kSave;
        sv[0] = R12;
        sv[1] = cmul(cscale(cmul(num[q], isq), 2.0), is);  // T12
      }
    }
  }
  // films between air gaps (backend/stack.py:229-262)
  for (int l = 1; l < L - 1; ++l) {
    const cd kz = layer_kz(l);
    if (count && kz.y == 0.0) atomicAdd(&nprop[l], 1);
    const cd t = ratio(kz), nn = lay[l].nn;
    const cd pr = cexp_ikh(kz, hsm[l - 1]);
    cd ps = pr;
    double g = 1.0;
    if constexpr (kRare) {
      const int e = min(top_exp(pr) - 1023, 1022);
      if (e > 0) {
        g = pow2(-e);
        ps = cscale(pr, g);
#pragma unroll
        for (int q = 0; q < 2; ++q) renorm(Z[q], V[q], num[q], ex[q]);
      }
    }
    const cd pr2 = cmul(ps, pr);
    const cd tp = cmul(cscale(t, 2.0), ps);
    cd Q, Qi;
    shear_q(l, Q, Qi);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      if (sh) {
        const cd m = cadd(Z[q], V[q]), n = cmul(cmul(Qi, csub(Z[q], V[q])), Q);
        Z[q] = cscale(cadd(m, n), 0.5);
        V[q] = cscale(csub(m, n), 0.5);
        num[q] = cmul(num[q], Q);
      }
      const cd X = q ? cmul(t, V[q]) : V[q], Y = cmul(q ? nn : t, Z[q]);
      const cd u = cadd(X, Y), v = csub(Y, X);
      const cd w = cmul(pr2, v);
      const cd us = kRare ? cscale(u, g) : u;
      const cd Zn = q ? cmul(t, cadd(us, w)) : cadd(us, w), Vn = cmul(q ? nn : t, csub(us, w));
      const cd f = q ? cmul(nn, tp) : tp;  // 2 A B p
      num[q] = cmul(num[q], f);
      if (act[q] || all_t) {
        const LayerC c = lay[l];
        const cd iD = crcp_nr(cadd(Zn, Vn));
        const cd A = q ? t : cd{1.0, 0.0}, Bz = q ? nn : t, s = cadd(A, Bz);
        cd T12 = cd{0.0, 0.0};
        if (all_t) {
          T12 = t12_exact(c, kz, kair, kz_air, q);
          store_rt(l, q, cmul(csub(A, Bz), crcp_nr(s)), T12);
        }
        if (act[q]) {
          cd *sv = wsv + ((size_t)l * 2 + q) * kSave;
          sv[0] = cmul(cmul(f, cadd(Z[q], V[q])), iD);  // x1 p x2
          sv[2] = pr;
          if (want_vec) {
            sv[1] = cmul(v, crcp_nr(u));                 // rg
            sv[3] = cmul(cmul(T12, cmul(s, us)), iD);    // T12 (1 + R12 p rg p)^-1
          }
          sv[4] = cmul(csub(Zn, Vn), iD);
        }
      }
      Z[q] = Zn;
      V[q] = Vn;
      if ((l & 3) == 3 || (kRare && g != 1.0)) renorm(Z[q], V[q], num[q], ex[q]);
    }
  }
  // superstrate (l = L - 1): the air gap below it (backend/stack.py:263-278)
  {
    const int l = L - 1;
    const LayerC c = lay[l];
    const cd kz = layer_kz(l);
    cd t = ratio(kz);
    t.x += c.zcr.x - c.zcr.x;
    cd Q, Qi, fs[2];
    shear_q(l, Q, Qi);
    root(c, kz, fs);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      renorm(Z[q], V[q], num[q], ex[q]);
      if (sh) {
        const cd m = cadd(Z[q], V[q]), n = cmul(cmul(Qi, csub(Z[q], V[q])), Q);
        Z[q] = cscale(cadd(m, n), 0.5);
        V[q] = cscale(csub(m, n), 0.5);
        num[q] = cmul(num[q], Q);
      }
      const cd X = q ? cmul(t, V[q]) : V[q], Y = cmul(q ? c.nn : t, Z[q]);
      const cd iu = crcp_nr(cadd(X, Y));
      // T12 (A + B) of substrate and superstrate, over 2 u: 2 f_a f_b / (k_z,air u)
      cd tt = cmul(cmul(num[q], fs[q]), iu);
      const double r2 = 2.0 * ra;
      tt = ev ? cd{tt.y * r2, -(tt.x * r2)} : cscale(tt, r2);
      if (ex[q]) tt = cd{scalbn(tt.x, ex[q]), scalbn(tt.y, ex[q])};
      tnet[q] = tt;
      rnet[q] = cmul(csub(Y, X), iu);
      if (all_t) {
        const cd A = q ? t : cd{1.0, 0.0}, Bz = q ? c.nn : t;
        store_rt(l, q, cmul(csub(A, Bz), crcp_nr(cadd(A, Bz))), t12_exact(c, kz, kair, kz_air, q));
      }
      if (act[q]) {
        cd *sv = wsv + ((size_t)l * 2 + q) * kSave;
        sv[0] = cmul(cmul(cmul(fs[q], isq), cadd(Z[q], V[q])), iu);  // T12 (1 - R12 rq)^-1
        sv[1] = rnet[q];
      }
    }
  }
  store_c(p.R_net(), j, rnet[0]);
  store_c(p.R_net(), j + npw, rnet[1]);
  store_c(p.T_net(), j, tnet[0]);
  store_c(p.T_net(), j + npw, tnet[1]);

  // ---- flux pass (backend/stack.py:323-366)
  if (!active) {
    if (want_vec) {
      for (int lv = 0; lv < L; ++lv)
        for (int q = 0; q < 2; ++q) store_c(p.vcd(), (size_t)lv * P + j + q * npw, cd{0.0, 0.0});
      for (int lv = 0; lv < L - 1; ++lv)
        for (int q = 0; q < 2; ++q) store_c(p.vcu(), (size_t)lv * P + j + q * npw, cd{0.0, 0.0});
    }
    return;
  }
  const bool prop = j < np_air;
  double in_sum = 0.0, up_sum = 0.0, out_sum = 0.0;
  for (int q = 0; q < 2; ++q) {
    // a polarisation without incident light (TE or TM incidence) carries
    // zero amplitudes through every layer and adds nothing to the fluxes,
    // unless its coefficients are not finite: 0 times them is NaN, as in the
    // reference's dense products
    if (!want_vec && !act[q]) {
      const double bad = 0.0 * (rnet[q].x + rnet[q].y + tnet[q].x + tnet[q].y);
      if (bad == 0.0) continue;
      if (j < np_in) up_sum += bad;
      for (int i = 0; i < L - 2; ++i) {
        if (p.slot_per_order()) {
          atomicAdd(&acc[1 + i].x, bad);
          atomicAdd(&acc[1 + i].y, bad);
        } else {
          acc[1 + i].x += bad;
          acc[1 + i].y += bad;
        }
      }
      if (j < np_out) out_sum += bad;
      continue;
    }
    const int pos = j + q * npw;
    const cd *top = wsv + ((size_t)(L - 1) * 2 + q) * kSave;
    const cd dp = cmul(top[1], din[q]);  // d_plus = r_top d
    if (j < np_in) {
      in_sum += cabs2(din[q]);
      up_sum += cabs2(dp);
    }
    if (want_vec) {
      store_c(p.vcd(), pos, din[q]);
      store_c(p.vcu(), pos, dp);
    }
    cd f1m = cmul(top[0], din[q]);
    for (int i = 0; i < L - 2; ++i) {
      const int k = L - 2 - i;
      const cd *s = wsv + ((size_t)k * 2 + q) * kSave;
      const cd f1p = cmul(s[4], f1m);
      const cd fl = flux_term(f1m, f1p, prop, q == 1);
      if (p.slot_per_order()) {  // several orders carry light: they add concurrently
        atomicAdd(&acc[1 + i].x, fl.x);
        atomicAdd(&acc[1 + i].y, fl.y);
      } else {                   // the one order that carries light adds alone
        acc[1 + i].x += fl.x;
        acc[1 + i].y += fl.y;
      }
      if (want_vec) {
        const cd f2m = cmul(s[3], f1m);
        const cd f2p = cmul(cmul(s[1], s[2]), f2m);
        store_c(p.vcd(), (size_t)(1 + i) * P + pos, f2m);
        store_c(p.vcu(), (size_t)(1 + i) * P + pos, f2p);
      }
      f1m = cmul(s[0], f1m);
    }
    const cd *s0 = wsv + ((size_t)0 * 2 + q) * kSave;
    const cd f2m = cmul(s0[1], f1m);
    if (want_vec) store_c(p.vcd(), (size_t)(L - 1) * P + pos, f2m);
    if (j < np_out) out_sum += cabs2(f2m);
  }
  atomicAdd(&acc[0].x, in_sum);
  atomicAdd(&acc[L].x, up_sum);
  atomicAdd(&acc[L - 1].x, out_sum);
}

// Sort key of -Re k_z + Im k_z as an unsigned integer with the order of the
// doubles (sign bit flipped for positive values, all bits for negative
// ones; -0 taken as +0, as the double comparison does).
__device__ __forceinline__ unsigned long long sort_key(double k) {
  const long long b = __double_as_longlong(k + 0.0);
  return b < 0 ? ~(unsigned long long)b : (unsigned long long)b | 0x8000000000000000ull;
}

// One point, phases 0-6 (the film kernels' header comments describe them).
// Every thread of the team calls this with the same `valid`, and with
// `valid` false takes the same barriers without touching memory.  The point
// accessor adds, to the fields solve_order uses: wl_nm() kx() ky() (k_pll),
// n(i), height(i), and the optional outputs sort_order() specular()
// num_prop() fluxes() (NULL to skip), and the required a_list() t_list()
// r_list() flags().
template <class Team, class Pt>
__device__ __forceinline__ void film_point(const Team &tm, const Pt &p, bool valid,
                                           unsigned char *base, const SlotSmem &S) {
  LayerC *lay = (LayerC *)(base + S.lay);
  cd *acc = (cd *)(base + S.acc);
  unsigned long long *keys = (unsigned long long *)(base + S.keys);
  double *hsm = (double *)(base + S.h);
  int *rank = (int *)(base + S.rank);
  int *nprop = (int *)(base + S.nprop);
  unsigned *wood = (unsigned *)(base + S.wood);
  cd *ws_smem = (cd *)(base + S.ws);
  int *misc = (int *)(base + S.misc);
  const int lt = tm.lt, team = tm.size;
  const int L = valid ? p.L() : 2, npw = valid ? p.npw() : 1;
  const int wood_words = (L + 1 + 31) / 32;
  const bool count = valid && p.num_prop() != nullptr;
  double a0 = 0.0, b0 = 0.0;
  if (valid) {
    a0 = p.kx() * p.period();
    b0 = p.ky() * p.period();
  }
  // ---------------------------------------------------------- phase 0
  bool grow = false;
  if (valid) {
    for (int i = lt; i <= L; i += team) {
      const double wln = wl_norm(p.wl_nm(), p.period());
      if (i == L) {
        hsm[L - 2] = wavenumber(cd{1.0, 0.0}, wln).x;
        break;
      }
      const emu_c128 v = p.n(i);
      const cd n = cd{v.re, v.im};
      LayerC c;
      c.k = wavenumber(n, wln);
      c.zcr = crcp_nr(n);
      c.ik = crcp_nr(c.k);
      c.n = n;
      c.nn = cmul(n, n);
      c.kk = k_squared(c.k);
      // the sign bit of Im k^2 decides the branch of the evanescent k_z
      grow |= i > 0 && i < L - 1 && signbit(c.kk.y);
      lay[i] = c;
    }
    // a film of index zero has no impedance: its phase, and so every result, is NaN
    for (int i = lt; i < L - 2; i += team) {
      const emu_c128 v = p.n(i + 1);
      hsm[i] = (v.re == 0.0 && v.im == 0.0) ? nan("") : p.height(i) / p.period();
    }
    for (int i = lt; i < L + 1; i += team) {
      acc[i] = cd{0.0, 0.0};
      nprop[i] = 0;
    }
    for (int i = lt; i < wood_words; i += team) wood[i] = 0u;
    if (lt == 0) {
      misc[0] = -1;
      misc[1] = 0;
      misc[2] = 0;
    }
  }
  const bool grows = tm.any(grow);  // of any point of the team: both copies give the same bits
  // ---------------------------------------------------------- phase 1
  // the air's k_z^2 is real, so k_z is the real root of it or i times that of -k_z^2
  auto air_order = [&](int u, double a, double b) -> bool {
    double al, be;
    order_ab(p.world_1d(), p.dy(), p.px()[u], p.py()[u], a, b, al, be);
    const double x = kz_arg(cd{hsm[L - 2], 0.0}, al, be).x;
    const double t = sqrt(fabs(x));
    keys[u] = sort_key(x >= 0.0 ? -1 * t : t);
    if (x >= 0.0) atomicAdd(&nprop[L], 1);
    return x == 0.0;
  };
  bool hit = false;
  if (valid) {
    for (int u = lt; u < npw; u += team)
      if (air_order(u, a0, b0)) {
        atomicOr(&wood[L >> 5], 1u << (L & 31));
        hit = true;
      }
  }
  // ---------------------------------------------------------- phase 2
  const bool some_air = tm.any(hit);
  const bool wood_air = some_air && valid && ((wood[L >> 5] >> (L & 31)) & 1u);
  if (some_air) {
    if (wood_air && lt == 0) nprop[L] = 0;
    tm.sync();
    if (wood_air)
      for (int u = lt; u < npw; u += team) air_order(u, (1 - 1e-9) * a0, (1 - 1e-9) * b0);
    tm.sync();
  }
  // ---------------------------------------------------------- phase 3
  hit = false;
  if (valid) {
    int32_t *so = p.sort_order();
    for (int u = lt; u < npw; u += team) {
      const unsigned long long ku = keys[u];
      // orders below u in the list count on ties, orders above it do not: only
      // the 32 around u need both comparisons
      int r = 0;
      const int v0 = u & ~31, v1 = min(npw, v0 + 32);
#pragma unroll 4
      for (int v = 0; v < v0; v += 2) {
        const ulonglong2 kv = *(const ulonglong2 *)(keys + v);
        r += (kv.x <= ku) + (kv.y <= ku);
      }
#pragma unroll 4
      for (int v = v0; v < v1; ++v) {
        const unsigned long long kv = keys[v];
        r += (kv < ku) | ((kv == ku) & (v < u));
      }
#pragma unroll 4
      for (int v = v1; v < npw; ++v) r += keys[v] < ku;
      rank[u] = r;
      const int pxu = p.px()[u], pyu = p.py()[u];
      const bool zero_order = (pxu == 0) && (p.world_1d() || pyu == 0);
      if (zero_order) misc[0] = r;
      if (so) so[r] = u;
      double al, be;
      order_ab(p.world_1d(), p.dy(), pxu, pyu, a0, b0, al, be);
      const double al2 = __dmul_rn(al, al), be2 = __dmul_rn(be, be);
      if (sqrt_is_real(kz_arg_sq(lay[0].kk, al2, be2))) atomicAdd(&nprop[0], 1);
      if (sqrt_is_real(kz_arg_sq(lay[L - 1].kk, al2, be2))) atomicAdd(&nprop[L - 1], 1);
      // Wood check of every layer: k_z == 0 exactly iff its argument is 0
      for (int l = 0; l < L; ++l) {
        const cd kk = lay[l].kk;
        if (__dsub_rn(kk.x, al2) == be2 && kk.y == 0.0) {
          atomicOr(&wood[l >> 5], 1u << (l & 31));
          misc[1] = 1;
          hit = true;
        }
      }
    }
  }
  // ---------------------------------------------------------- phase 4
  const bool some_layer = tm.any(hit);
  const bool layer_wood = some_layer && valid && misc[1] != 0;
  if (some_layer) {
    // recount substrate / superstrate with the scaled k_parallel where marked
    if (layer_wood && lt == 0) {
      nprop[0] = 0;
      nprop[L - 1] = 0;
    }
    tm.sync();
    if (layer_wood) {
      for (int u = lt; u < npw; u += team) {
        for (int t = 0; t < 2; ++t) {
          const int l = t ? L - 1 : 0;
          const bool wl_l = (wood[l >> 5] >> (l & 31)) & 1u;
          double al, be;
          order_ab(p.world_1d(), p.dy(), p.px()[u], p.py()[u], wl_l ? (1 - 1e-9) * a0 : a0,
                   wl_l ? (1 - 1e-9) * b0 : b0, al, be);
          if (sqrt_is_real(kz_arg(lay[l].k, al, be))) atomicAdd(&nprop[l], 1);
        }
      }
    }
    tm.sync();
  }
  // ---------------------------------------------------------- phase 5
  if (valid) {
    const int spec = misc[0];
    const int np_air = nprop[L], np_in = nprop[L - 1], np_out = nprop[0];
    if (!layer_wood && !grows)
      for (int u = lt; u < npw; u += team)
        solve_order<false>(p, u, rank[u], spec, lay, hsm, wood, wood_air, a0, b0, np_air, np_in, np_out, acc,
                           nprop, count, ws_smem);
    else
      for (int u = lt; u < npw; u += team)
        solve_order<true>(p, u, rank[u], spec, lay, hsm, wood, wood_air, a0, b0, np_air, np_in, np_out, acc,
                          nprop, count, ws_smem);
  }
  tm.sync();
  // ---------------------------------------------------------- phase 6
  // a_list / t_list / r_list (backend/stack.py:368-426), one entry per
  // thread of the team; the flags word once every entry is checked
  int nprop_in0 = 0, nprop_out0 = 0;
  if (valid) {
    const int np_in = nprop[L - 1], np_out = nprop[0];
    nprop_in0 = np_in;
    nprop_out0 = np_out;
    const double df0 = acc[0].x, up0 = acc[L].x, dsub = acc[L - 1].x;
    // |down_fluxes[i]| with down_fluxes = [df0, gap_1..gap_{L-2}, dsub]
    auto dfa = [&](int i) -> double {
      if (i == 0) return fabs(df0);
      if (i == L - 1) return fabs(dsub);
      return acc[i].y == 0.0 ? fabs(acc[i].x) : hypot(acc[i].x, acc[i].y);
    };
    double *al = p.a_list();
    double *tl = p.t_list();
    bool fin = true;
    for (int i = lt; i < L - 1; i += team) {
      double a = 0.0, t = 0.0;
      if (np_out != 0) {
        a = (i < L - 2) ? fabs(dfa(i + 1) - dfa(i + 2)) : fabs(df0 - dsub - up0);
        t = (i < L - 2) ? fabs(dfa(i + 2) / dfa(i)) : fabs(dsub / df0);
      }
      al[i] = a;
      tl[i] = t;
      fin = fin && isfinite(a) && isfinite(t);
    }
    if (lt == 0) {
      const double rr = (np_out != 0) ? fabs(up0 / df0) : 0.0;
      *p.r_list() = rr;
      fin = fin && isfinite(rr);
      if (p.specular()) *p.specular() = misc[0];
    }
    if (!fin) atomicOr(&misc[2], 1);
    if (int32_t *np = p.num_prop())
      for (int i = lt; i <= L; i += team) np[i] = nprop[i];
    if (double *fo = p.fluxes()) {
      for (int i = lt; i <= L; i += team) {
        fo[2 * i] = acc[i].x;
        fo[2 * i + 1] = acc[i].y;
      }
    }
  }
  tm.sync();
  // only misc[2] is read after the barrier, by the thread that resets it in
  // phase 0 of the team's next point
  if (valid && lt == 0) {
    uint32_t flags = 0;
    if (wood_air) flags |= EMU_PT_WOOD_AIR;
    if (layer_wood) flags |= EMU_PT_WOOD_LAYER;
    if (nprop_out0 == 0) flags |= EMU_PT_NO_PROP_SUB;
    if (nprop_in0 == 0) flags |= EMU_PT_NO_PROP_SUP;
    if (misc[2]) flags |= EMU_PT_NONFINITE;
    *p.flags() = flags;
  }
}

}  // namespace emu
