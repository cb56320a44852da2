// The push of one particle of the FP64 island (gr.cu), the formulas of
// gr.cu's gr_push_one and of gr_metric.cuh written for the FP64 pipe. GB300
// runs FP64 at 1/64 of the FP32 rate, so the island's time is its count of
// FP64 instructions, and a division or a square root is eight to twelve of
// them. Here the metric at a point takes two reciprocals (of products, from
// which the single ones follow by multiplication) and one square root where
// the component formulas divide ten times, and products and sums that belong
// together are one fma. Each quantity is within a few roundings of 2^-53 of
// gr_metric.cuh's; the results are rounded to FP32.
#pragma once

#include "gr_metric.cuh"

namespace pic {
namespace island {

// 1 / dchi and 1 / deta in 64 bits; QKS holds them rounded to the field type,
// and each formula takes the one that gr_metric.cuh's takes
struct Rcp {
  double chi, eta;
};

// a point's quantities with their reciprocals: S2 = Sg + 2 r = Sg (1 + z)
struct Pt {
  double r, ex, eta, s, c, s2, dtde, Sg, S2, Dl, A;
  double iex, iSg, iS2, is, idt;
  double al, ial;  // lapse = sqrt(Sg / S2) and its reciprocal
};

__device__ __forceinline__ Pt point(const QKS<double>& m, double x1, double x2) {
  Pt p;
  p.ex   = exp(fma(x1, m.dchi, m.chi_min));
  p.r    = m.r0 + p.ex;
  p.eta  = fma(x2, m.deta, m.eta_min);
  p.dtde = m.dtheta_deta(p.eta);
  sincos(m.eta2theta(p.eta), &p.s, &p.c);
  const double a2 = m.a * m.a, rr = fma(p.r, p.r, a2);
  p.s2 = p.s * p.s;
  p.Sg = fma(p.r, p.r, a2 * (p.c * p.c));
  p.S2 = fma(2.0, p.r, p.Sg);
  p.Dl = fma(-2.0, p.r, rr);
  p.A  = fma(rr, rr, -(a2 * p.Dl) * p.s2);
  const double eS = p.ex * p.Sg, i3 = 1.0 / (eS * p.S2), i2 = 1.0 / (p.s * p.dtde);
  p.iex = i3 * (p.Sg * p.S2);
  p.iSg = i3 * (p.ex * p.S2);
  p.iS2 = i3 * eS;
  p.is  = i2 * p.dtde;
  p.idt = i2 * p.s;
  p.ial = sqrt(p.S2 * p.iSg);
  p.al  = p.ial * (p.Sg * p.iS2);
  return p;
}

// h^ij and the shift
struct Up {
  double h11, h22, h33, h13, beta1;
};
__device__ __forceinline__ Up upper(const QKS<double>& m, const Rcp& q, const Pt& p) {
  Up           g;
  const double ei = p.iex * m.dchi_inv, ec = p.iex * q.chi, it = p.idt * q.eta;
  g.h11   = (ec * ec) * (p.A * (p.iSg * p.iS2));
  g.h22   = p.iSg * (it * it);
  g.h33   = p.iSg * (p.is * p.is);
  g.h13   = ei * (m.a * p.iSg);
  g.beta1 = ei * (2.0 * p.r * p.iS2);
  return g;
}

// the orthonormal frame: A0 = sqrt(h^11), q2 = sqrt(h_22), q3 = sqrt(h_33)
struct Frame {
  double A0, q2, q3, iA0, iq2, iq3, h_13;
};
__device__ __forceinline__ Frame frame(const QKS<double>& m, const Rcp& q, const Pt& p) {
  Frame        f;
  const double wS = sqrt(p.Sg), wA = sqrt(p.A), w2 = p.ial * wS;  // w2 = sqrt(S2)
  const double SA = wS * wA, i = 1.0 / (SA * w2);
  const double iS = i * (wA * w2), iA = i * (wS * w2), i2 = i * SA;
  f.A0   = (p.iex * q.chi) * (wA * (iS * i2));
  f.iA0  = (p.ex * m.dchi) * (wS * w2 * iA);
  f.q2   = (m.deta * p.dtde) * wS;
  f.iq2  = (q.eta * p.idt) * iS;
  f.q3   = fabs(p.s) * (wA * iS);
  f.iq3  = fabs(p.is) * (wS * iA);
  f.h_13 = -(m.dchi * p.ex * m.a) * (p.S2 * p.iSg) * p.s2;
  return f;
}

// EMHalfPush (gr.hpp:177-217); Dh, Bh in the frame
__device__ __forceinline__ void half_push(const Frame& f, double al, double ndth, const double* vp,
                                          const double* Dh, const double* Bh, double* vout) {
  const double k  = f.h_13 * f.iq3;
  double       vh[3] = { f.A0 * fma(-vp[2] * f.iq3, k, vp[0]), vp[1] * f.iq2, vp[2] * f.iq3 };
  double       C = ndth * 0.5 * al, D0[3], B[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    D0[c] = Dh[c] * C;
    vh[c] += D0[c];
  }
  C *= rsqrt(fma(vh[0], vh[0], fma(vh[1], vh[1], fma(vh[2], vh[2], 1.0))));
#pragma unroll
  for (int c = 0; c < 3; ++c) B[c] = Bh[c] * C;
  C = 2.0 / fma(B[0], B[0], fma(B[1], B[1], fma(B[2], B[2], 1.0)));
  const double w0 = C * fma(vh[1], B[2], fma(-vh[2], B[1], vh[0]));
  const double w1 = C * fma(vh[2], B[0], fma(-vh[0], B[2], vh[1]));
  const double w2 = C * fma(vh[0], B[1], fma(-vh[1], B[0], vh[2]));
  vh[0] += fma(w1, B[2], fma(-w2, B[1], D0[0]));
  vh[1] += fma(w2, B[0], fma(-w0, B[2], D0[1]));
  vh[2] += fma(w0, B[1], fma(-w1, B[0], D0[2]));
  vout[0] = fma(vh[0], f.iA0, vh[2] * k);
  vout[1] = vh[1] * f.q2;
  vout[2] = vh[2] * f.q3;
}

// v^i of the covariant v, and 1 / gamma; gamma^2 = (massive) + v_i v^i
__device__ __forceinline__ void raise(const Up& g, bool massive, const double* v, double* o,
                                      double& g2, double& ig) {
  o[0] = fma(v[0], g.h11, v[2] * g.h13);
  o[1] = v[1] * g.h22;
  o[2] = fma(v[0], g.h13, v[2] * g.h33);
  g2   = fma(v[0], o[0], fma(v[1], o[1], fma(v[2], o[2], massive ? 1.0 : 0.0)));
  ig   = rsqrt(g2);
}

// GeodesicMomentumPush (gr.hpp:260-331)
template <typename ITER>
__device__ __forceinline__ void momentum(const QKS<double>& m, const Rcp& rc, const Pt& p, const Up& g,
                                         bool massive, double dt, int niter, const double* vp,
                                         double* vu, ITER&& iterate) {
  // derivatives along r and theta (qkerr_schild.h:340-545)
  const double a2 = m.a * m.a, dxdt = m.dx_dt(p.eta);
  const double dx_r = m.dchi * p.ex, dr_S = 2.0 * p.r * dx_r, dr_D = 2.0 * dx_r * (p.r - 1.0);
  const double dr_A = fma(4.0 * p.r * dx_r, fma(p.r, p.r, a2), -a2 * p.s2 * dr_D);
  const double sc = -2.0 * a2 * p.s * p.c * dxdt;
  const double dtS = fabs(sc) <= QKS<double>::eps() ? 0.0 : sc;
  const double dtA0 = sc * p.Dl, dtA = fabs(dtA0) <= QKS<double>::eps() ? 0.0 : dtA0;
  const double iSS = p.iSg * p.iSg, i22 = p.iS2 * p.iS2, iq = p.iSg * p.iS2;
  const double al3 = p.al * p.al * p.al * iSS, ei = p.iex * m.dchi_inv;
  const double ec = p.iex * rc.chi, E = ec * ec;
  const double fr = fma(dx_r, p.Sg, -p.r * dr_S), is2 = p.is * p.is, dti2 = rc.eta * rc.eta;
  const double d_al[2] = { -fr * al3, p.r * sc * al3 };
  const double d_be[2] = { fma(ei * 2.0 * fr, i22, -m.dchi * ei * (2.0 * p.r * p.iS2)),
                           -ei * 2.0 * p.r * dtS * i22 };
  const double A2 = 2.0 * p.A * iq;
  const double d_11[2] = {
    E * iq * fma(-A2, fma(p.r, dr_S, p.Sg * (dr_S + dx_r)), dr_A) - m.dchi * E * A2,
    E * iq * fma(-A2, dtS * (p.r + p.Sg), dtA)
  };
  const double d_22[2] = { -dr_S * iSS * dti2, -dtS * iSS * dti2 };
  const double d_33[2] = { -dr_S * iSS * is2,
                           -fma(2.0 * p.c * p.is * p.Sg, dxdt, dtS) * (iSS * is2) };
  const double d_13[2] = { fma(-m.a * dr_S * iSS, ei, -m.dchi * ei * m.a * p.iSg),
                           -m.a * dtS * iSS * ei };
  vu[0] = vp[0], vu[1] = vp[1], vu[2] = vp[2];
  iterate(niter, vu, [&](int, const double* v, double* o) {
    const double vm[3] = { 0.5 * (vp[0] + v[0]), 0.5 * (vp[1] + v[1]), vp[2] };
    double       vc[3], g2, ig;
    raise(g, massive, vm, vc, g2, ig);
    const double e = g2 * ig, h = 0.5 * p.al * ig;  // alpha u0 = gamma, 1 / u0 = alpha / gamma
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const double q = fma(d_11[k], vm[0] * vm[0],
                           fma(d_22[k], vm[1] * vm[1],
                               fma(d_33[k], vm[2] * vm[2], 2.0 * d_13[k] * vm[0] * vm[2])));
      o[k] = fma(dt, fma(-e, d_al[k], fma(vm[0], d_be[k], -h * q)), vp[k]);
    }
  });
}

// GeodesicCoordinatePush (gr.hpp:333-383); the first pass's point is (p0, g0)
template <typename ITER>
__device__ __forceinline__ void coordinate(const QKS<double>& m, const Rcp& rc, double al0, const Up& g0,
                                           bool massive, double dt, int niter, const double* xp,
                                           const double* vp, double* xu, ITER&& iterate) {
  xu[0] = xp[0], xu[1] = xp[1];
  iterate(niter, xu, [&](int it, const double* x, double* o) {
    Up     g  = g0;
    double al = al0;
    if (it > 0) {
      const Pt p = point(m, 0.5 * (xp[0] + x[0]), m.clamp_x2(0.5 * (xp[1] + x[1])));
      g          = upper(m, rc, p);
      al         = p.al;
    }
    double vc[3], g2, ig;
    raise(g, massive, vp, vc, g2, ig);
    const double iu = al * ig;
    o[0]            = fma(dt, fma(vc[0], iu, -g.beta1), xp[0]);
    o[1]            = fma(dt, vc[1] * iu, xp[1]);
  });
}

template <typename ITER>
__device__ __forceinline__ void push_one(const QKS<double>& m, const Rcp& rc, bool massive,
                                         double ndth, double dt, int niter, const double* xp,
                                         const double* Dc, const double* Bc, const double* u,
                                         double* xo, double* uo, ITER&& iterate) {
  const double xc = m.clamp_x2(xp[1]);
  double       vp[3] = { u[0], u[1], u[2] }, vu[3];
  Pt           p = point(m, xp[0], xp[1]);
  if (massive) {
    const Frame  f  = frame(m, rc, p);
    const double al = p.al, k = f.h_13 * f.iq3;
    const double Dh[3] = { Dc[0] * f.iA0, Dc[1] * f.q2, fma(Dc[2], f.q3, Dc[0] * k) };
    const double Bh[3] = { Bc[0] * f.iA0, Bc[1] * f.q2, fma(Bc[2], f.q3, Bc[0] * k) };
    half_push(f, al, ndth, vp, Dh, Bh, vu);
    vp[0] = vu[0], vp[1] = vu[1], vp[2] = vu[2];
    if (xc != xp[1]) p = point(m, xp[0], xc);
    const Up g = upper(m, rc, p);
    momentum(m, rc, p, g, true, dt, niter, vp, vu, iterate);
    vp[0] = vu[0], vp[1] = vu[1], vp[2] = vu[2];
    half_push(f, al, ndth, vp, Dh, Bh, vu);
    coordinate(m, rc, p.al, g, true, dt, niter, xp, vu, xo, iterate);
  } else {
    Up g = upper(m, rc, p);
    momentum(m, rc, p, g, false, dt, niter, vp, vu, iterate);
    if (xc != xp[1]) p = point(m, xp[0], xc), g = upper(m, rc, p);
    coordinate(m, rc, p.al, g, false, dt, niter, xp, vu, xo, iterate);
  }
  uo[0] = vu[0], uo[1] = vu[1], uo[2] = vu[2];
}

}  // namespace island
}  // namespace pic
