// Mode-space pieces of an RK stage: the nonlinear term from the product spectra, the forces, the
// pressure projection and the stage forms.  Shared by the stage kernel (tg_spectral.cu) and the x-passes
// that end in a stage (tg_xstage.cu).
#pragma once

#include "tg_spectral.cuh"

namespace tg {

template <typename R>
__device__ __forceinline__ cx<double> ldc(const void* p, long long i) {
  return cvt<double>(reinterpret_cast<const cx<R>*>(p)[i]);
}
template <typename R>
__device__ __forceinline__ void stc(void* p, long long i, cx<double> v) {
  reinterpret_cast<cx<R>*>(p)[i] = cvt<R>(v);
}

// The algebra below is written with its roundings (a product and its sum fused, or a product alone), so that
// the compiler has no choice of which products to fuse: the stage gives the same bits in every kernel, and a
// step may take the fused stage kernel or the separate passes by the size of a batch without changing a result.
__device__ __forceinline__ cx<double> mulr(double s, cx<double> a) { return mkc<double>(__dmul_rn(s, a.x), __dmul_rn(s, a.y)); }
__device__ __forceinline__ cx<double> fmar(double s, cx<double> a, cx<double> c) {
  return mkc<double>(__fma_rn(s, a.x, c.x), __fma_rn(s, a.y, c.y));
}
// c + i s a
__device__ __forceinline__ cx<double> ifmar(double s, cx<double> a, cx<double> c) {
  return mkc<double>(__fma_rn(-s, a.y, c.x), __fma_rn(s, a.x, c.y));
}
// |K|^2 of a mode
__device__ __forceinline__ double mode_k2(double kx, double ky, double kz) {
  return __fma_rn(kz, kz, __fma_rn(ky, ky, __dmul_rn(kx, kx)));
}
// nu + nu_h K^2 (nu exactly when the hyper term is off)
__device__ __forceinline__ double mode_nu(double nu, double nuh, double K2) { return nuh != 0.0 ? __fma_rn(nuh, K2, nu) : nu; }

// i (kx a + ky b + kz c)
__device__ __forceinline__ cx<double> ikdot(double kx, double ky, double kz, cx<double> a, cx<double> b, cx<double> c) {
  return ione(fmar(kz, c, fmar(ky, b, mulr(kx, a))));
}

// ------------------------------------------------------------------ nonlinear-term assembly
// Product order of the z-pass (see tg_ctx.cu):
//  fluid : 0 u1u1, 1 u2u2, 2 u3u3, 3 u1u2, 4 u2u3, 5 u3u1        (RSprod.cc:52-105)
//  MHD   : 0 zp1zm1, 1 zp2zm2, 2 zp3zm3, 3 zp1zm2 (v1), 4 zm1zp2 (w1), 5 zp2zm3 (v2),
//          6 zm2zp3 (w2), 7 zp3zm1 (v3), 8 zm3zp1 (w3)              (RSprod.cc:117-194)
//  scalar: fluid 0..5, then 6 u1 th, 7 u2 th, 8 u3 th               (compute_nlin_SF.cc)
// Trace-free form (PX[2] null): the third square is left out and taken from the first two, which changes
// the velocity's term by the gradient of it; the projection takes that gradient out again.
// x-derivative of a coefficient (Xderiv universal_tr.cc:186-210): FOUR i kx; SCFT a real factor
// by the parity of the series, cos -> sin: -kx (Xderiv_Cos_SCFT), sin -> cos: +kx
// (Xderiv_Sin_SCFT, scft_tr.cc:649-672)
struct XDer {
  double kx;
  int scft;
  // c + the derivative of p
  __device__ __forceinline__ cx<double> cos_in(cx<double> p, cx<double> c) const {
    return scft ? fmar(-kx, p, c) : ifmar(kx, p, c);
  }
  __device__ __forceinline__ cx<double> sin_in(cx<double> p, cx<double> c) const {
    return scft ? fmar(kx, p, c) : ifmar(kx, p, c);
  }
};
__device__ __forceinline__ cx<double> iky_ikz(double ky, double kz, cx<double> b, cx<double> c) {
  return ione(fmar(kz, c, mulr(ky, b)));
}

// the products of one mode; the third is zero in the trace-free form
template <typename Rp, int PHYS>
__device__ __forceinline__ void load_products(const void* const* PX, long long idx, cx<double> (&p)[9]) {
#pragma unroll
  for (int q = 0; q < (PHYS == PH_FLUID ? 6 : 9); ++q)
    p[q] = (q != 2 || PX[2]) ? ldc<Rp>(PX[q], idx) : mkc<double>(0, 0);
}

template <int PHYS>
__device__ __forceinline__ void assemble(const cx<double> (&p)[9], const XDer& dx, double ky, double kz, cx<double>* n) {
  if constexpr (PHYS == PH_FLUID || PHYS == PH_SCALAR || PHYS == PH_RB) {
    // parities of the products (RV_Forward_transform_RSprod Rvf.cc:179-186): u1u1, u2u2, u3u3,
    // u2u3 cos; u1u2, u3u1 sin; and u1 th cos, u2 th, u3 th sin (compute_nlin_SF.cc:80-115)
    n[0] = dx.cos_in(p[0], iky_ikz(ky, kz, p[3], p[5]));
    n[1] = dx.sin_in(p[3], iky_ikz(ky, kz, p[1], p[4]));
    n[2] = dx.sin_in(p[5], iky_ikz(ky, kz, p[4], p[2]));
    if constexpr (PHYS != PH_FLUID) n[3] = dx.cos_in(p[6], iky_ikz(ky, kz, p[7], p[8]));
  } else {
    const double kx = dx.kx;
    // Zp.nlin (n) and Zm.nlin (nw)
    const cx<double> n0 = ikdot(kx, ky, kz, p[0], p[3], p[8]);
    const cx<double> n1 = ikdot(kx, ky, kz, p[4], p[1], p[5]);
    const cx<double> n2 = ikdot(kx, ky, kz, p[7], p[6], p[2]);
    const cx<double> w0 = ikdot(kx, ky, kz, p[0], p[4], p[7]);
    const cx<double> w1 = ikdot(kx, ky, kz, p[3], p[1], p[6]);
    const cx<double> w2 = ikdot(kx, ky, kz, p[8], p[5], p[2]);
    // Elsasser_to_UB_nlin (elsasser.cc:118-130)
    n[0] = 0.5 * (n0 + w0);
    n[1] = 0.5 * (n1 + w1);
    n[2] = 0.5 * (n2 + w2);
    n[3] = 0.5 * (n0 - w0);
    n[4] = 0.5 * (n1 - w1);
    n[5] = 0.5 * (n2 - w2);
  }
}

template <int PHYS>
struct NState {
  static constexpr int v = (PHYS == PH_FLUID) ? 3 : (PHYS == PH_MHD ? 6 : 4);
};

// rhs = -[nlin - f + grad p] with p = div(nlin - f)/K^2 on the velocity (Compute_pressure with
// Compute_divergence_nlin: Xderiv of nlin1 with parity 1; Add_pressure_gradient: Xderiv of p
// with parity 0; Compute_rhs); other fields rhs = -(nlin - f).
__device__ __forceinline__ void project_rhs(cx<double>* r, int ns, const XDer& dx, double ky, double kz, double K2) {
  cx<double> p = mkc<double>(0, 0);
  if (K2 > 0) p = mulr(1.0 / K2, dx.sin_in(r[0], iky_ikz(ky, kz, r[1], r[2])));
  r[0] = dx.cos_in(mkc<double>(-p.x, -p.y), mkc<double>(-r[0].x, -r[0].y));
  r[1] = ifmar(-ky, p, mkc<double>(-r[1].x, -r[1].y));
  r[2] = ifmar(-kz, p, mkc<double>(-r[2].x, -r[2].y));
  for (int c = 3; c < ns; ++c) r[c] = mkc<double>(-r[c].x, -r[c].y);
}

// Add_force: nlin -= Force, from the force box and from the stage's fields
template <int PHYS>
__device__ __forceinline__ void sub_forces(const RKArgs& a, long long gi, int kxi, int kyi, int l3, double kx, double ky,
                                           double kz, double K2, cx<double>* r) {
  constexpr int NS = NState<PHYS>::v;
  if (a.FB != nullptr && kxi >= -a.fx && kxi <= a.fx && kyi >= -a.fy && kyi <= a.fy && l3 <= a.fz) {
    const int box = (2 * a.fx + 1) * (2 * a.fy + 1) * (a.fz + 1);
    const int p = ((kxi + a.fx) * (2 * a.fy + 1) + (kyi + a.fy)) * (a.fz + 1) + l3;
#pragma unroll
    for (int c = 0; c < NS; ++c) r[c] = r[c] - a.FB[(long long)c * box + p];
  }
  if (a.coriolis) {
    // Compute_force_Coriolis (compute_force_Coriolis.cc:47-80) from the stage's velocity:
    // Force = V x Omega, then Add_force: nlin -= Force
    cx<double> v[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) v[c] = a.inprec ? ldc<float>(a.IN[c], gi) : ldc<double>(a.IN[c], gi);
    r[0] = r[0] - fmar(a.om[1], v[2], mulr(-a.om[2], v[1]));
    r[1] = r[1] - fmar(a.om[2], v[0], mulr(-a.om[0], v[2]));
    r[2] = r[2] - fmar(a.om[0], v[1], mulr(-a.om[1], v[0]));
  }
  if (a.lm) {
    // Compute_force_Liquid_metal (compute_force_LM.cc:46-70): Force = -(B0 . K)^2/K^2 V
    // (Array_mult_V0_khat_sqr_FOUR four_basic.cc:413-439), then Add_force: nlin -= Force
    const double bk = __fma_rn(a.b0[0], kx, __fma_rn(a.b0[1], ky, __dmul_rn(a.b0[2], kz)));
    const double f = K2 > 0 ? __dmul_rn(bk, bk) / K2 : 0.0;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const cx<double> v = a.inprec ? ldc<float>(a.IN[c], gi) : ldc<double>(a.IN[c], gi);
      r[c] = fmar(f, v, r[c]);
    }
  }
  if constexpr (PHYS == PH_RB) {
    // Compute_force_RB (compute_force_RB.cc:51-105) from the stage's fields, then Add_force:
    // nlin1 -= fu * theta, T.nlin -= ft * u1
    const cx<double> th = a.inprec ? ldc<float>(a.IN[3], gi) : ldc<double>(a.IN[3], gi);
    const cx<double> u1 = a.inprec ? ldc<float>(a.IN[0], gi) : ldc<double>(a.IN[0], gi);
    r[0] = fmar(-a.rb_buoy_u, th, r[0]);
    r[3] = fmar(-a.rb_buoy_t, u1, r[3]);
  }
}

// ------------------------------------------------------------------ RK stage kernel
// IncFluid::Time_advance (time_advance.cc:60-163) with E(a) = exp(-(nu + nu_h K^2) a dt K^2)
// (the hyper term when on, mult_exp_visc.cc:56-165) and Single_time_step(dt, a, b, c) =
// E(b)(E(a - b) u + c dt N) (single_time_step.cc:54-86):
//  RK4 stage 1: u1 = E(1/2)(u0 + dt/2 N0),        tot  = dt/6 E(1) N0
//      stage 2: u2 = E(1/2) u0 + dt/2 N1,         tot += dt/3 E(1/2) N1
//      stage 3: u3 = E(1/2)(E(1/2) u0 + dt N2),   tot += dt/3 E(1/2) N2
//      stage 4: u  = E(1) u0 + tot + dt/6 N3
//  EULER (5):   u  = E(1)(u0 + dt N0)                       Single_time_step(dt, 1, 1, 1)
//  RK2   (7):   u1 = E(1/2)(u0 + dt/2 N0)                   Single_time_step(dt, 1/2, 1/2, 1/2)
//        (6):   u  = E(1/2)(E(1/2) u0 + dt N1)              Single_time_step(dt, 1, 1/2, 1)
// after a final stage (4, 5, 6) the energy of u for the NaN check / Get_dt
// the stage's field and accumulator from u0, the accumulator so far and the right-hand side, for the stages
// that do not end a step (1, 2, 3, 7); eh = E(1/2), e1 = E(1)
template <int STAGE>
__device__ __forceinline__ cx<double> stage_field(cx<double> u0, cx<double> rc, double dt, double eh) {
  if constexpr (STAGE == 1 || STAGE == 7) return mulr(eh, fmar(0.5 * dt, rc, u0));
  else if constexpr (STAGE == 2) return fmar(0.5 * dt, rc, mulr(eh, u0));
  else return mulr(eh, fmar(dt, rc, mulr(eh, u0)));
}
template <int STAGE>
__device__ __forceinline__ cx<double> stage_total(cx<double> tot, cx<double> rc, double dt, double eh, double e1) {
  if constexpr (STAGE == 1) return mulr(dt / 6.0, mulr(e1, rc));
  else return fmar(dt / 3.0, mulr(eh, rc), tot);
}

}  // namespace tg
