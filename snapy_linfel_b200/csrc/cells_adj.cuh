// cells_adj.cuh — reverse of the face values of a cell (cells.cuh).
#pragma once

#include "cells.cuh"
#include "dual.cuh"

namespace snapb {

// WENO5-JS face value (weno5_face) reversed by hand: g * d out / d (a..e),
// accumulated into gx[0..4].  With omega_k = alpha_k / sum(alpha):
//   d out / d p_k = omega_k,  d out / d beta_k = -2 omega_k (p_k - out) / (beta_k + eps);
// the mean-|phi| scaling adds sign(x_i)/5 * (W - sum_j y_j dW/dy_j).
__device__ __forceinline__ void weno5_face_vjp(double a, double b, double c, double d, double e,
                                               bool scale, double g, double* gx) {
  double x[5] = {a, b, c, d, e};
  double vs = 1.;
  if (scale) {
    vs = (fabs(a) + fabs(b) + fabs(c) + fabs(d) + fabs(e)) / 5.;
    if (vs == 0.) return;  // the forward returns the constant 0
    double iv = 1. / vs;
#pragma unroll
    for (int q = 0; q < 5; ++q) x[q] *= iv;
  }
  const double c16 = 1. / 6., c56 = 5. / 6., c13 = 1. / 3.;
  const double c116 = 11. / 6., c76 = 7. / 6., c1312 = 13. / 12.;
  double y0 = x[0], y1 = x[1], y2 = x[2], y3 = x[3], y4 = x[4];
  double p0 = -c16 * y0 + c56 * y1 + c13 * y2;
  double p1 = c13 * y1 + c56 * y2 - c16 * y3;
  double p2 = c116 * y2 - c76 * y3 + c13 * y4;
  double u0 = y0 - 2. * y1 + y2, v0 = y0 - 4. * y1 + 3. * y2;
  double u1 = y1 - 2. * y2 + y3, v1 = y3 - y1;
  double u2 = y2 - 2. * y3 + y4, v2 = 3. * y2 - 4. * y3 + y4;
  double b0 = c1312 * u0 * u0 + 0.25 * v0 * v0;
  double b1 = c1312 * u1 * u1 + 0.25 * v1 * v1;
  double b2 = c1312 * u2 * u2 + 0.25 * v2 * v2;
  double e0 = b0 + 1e-6, e1 = b1 + 1e-6, e2 = b2 + 1e-6;
  double a0 = 0.3 / (e0 * e0), a1 = 0.6 / (e1 * e1), a2 = 0.1 / (e2 * e2);
  double is = 1. / (a0 + a1 + a2);
  double o0 = a0 * is, o1 = a1 * is, o2 = a2 * is;
  double W = o0 * p0 + o1 * p1 + o2 * p2;
  double gb0 = -2. * o0 * (p0 - W) / e0;
  double gb1 = -2. * o1 * (p1 - W) / e1;
  double gb2 = -2. * o2 * (p2 - W) / e2;
  const double k13 = 13. / 6.;
  double gy[5];
  gy[0] = -c16 * o0 + gb0 * (k13 * u0 + 0.5 * v0);
  gy[1] = c56 * o0 + c13 * o1 + gb0 * (-2. * k13 * u0 - 2. * v0) + gb1 * (k13 * u1 - 0.5 * v1);
  gy[2] = c13 * o0 + c56 * o1 + c116 * o2 + gb0 * (k13 * u0 + 1.5 * v0) +
          gb1 * (-2. * k13 * u1) + gb2 * (k13 * u2 + 1.5 * v2);
  gy[3] = -c16 * o1 - c76 * o2 + gb1 * (k13 * u1 + 0.5 * v1) + gb2 * (-2. * k13 * u2 - 2. * v2);
  gy[4] = c13 * o2 + gb2 * (k13 * u2 + 0.5 * v2);
  if (!scale) {
#pragma unroll
    for (int q = 0; q < 5; ++q) gx[q] += g * gy[q];
    return;
  }
  double ydw = 0.;
#pragma unroll
  for (int q = 0; q < 5; ++q) ydw += x[q] * gy[q];
  double corr = (W - ydw) / 5.;
  double raw[5] = {a, b, c, d, e};
#pragma unroll
  for (int q = 0; q < 5; ++q) gx[q] += g * (gy[q] + (raw[q] < 0. ? -corr : corr));
}

// Reverse of cell_states at WENO5 without scaling: the cotangents glo, ghi of
// the cell's two face values onto its five-cell window.  Both sides share the
// smoothness measures and their reciprocals (five quotients instead of
// fourteen for two weno5_face_vjp).  clip: values below zero are clipped by
// the forward and pass nothing back.
__device__ __forceinline__ void weno5_cell_vjp(const double* q, bool clip, double glo, double ghi,
                                               double* t) {
  const double a = q[0], b = q[1], c = q[2], d = q[3], e = q[4];
  const double c16 = 1. / 6., c56 = 5. / 6., c13 = 1. / 3., c116 = 11. / 6., c76 = 7. / 6.,
               c1312 = 13. / 12., k13 = 13. / 6.;
  const double u0 = a - 2. * b + c, v0 = a - 4. * b + 3. * c;
  const double u1 = b - 2. * c + d, v1 = d - b;
  const double u2 = c - 2. * d + e, v2 = 3. * c - 4. * d + e;
  const double i0 = 1. / (c1312 * u0 * u0 + 0.25 * v0 * v0 + 1e-6);
  const double i1 = 1. / (c1312 * u1 * u1 + 0.25 * v1 * v1 + 1e-6);
  const double i2 = 1. / (c1312 * u2 * u2 + 0.25 * v2 * v2 + 1e-6);
  const double r0 = i0 * i0, r1 = 0.6 * (i1 * i1), r2 = i2 * i2;
  double gb0, gb1, gb2;
  {  // low side: candidates of (a, b, c), (b, c, d), (c, d, e)
    const double p0 = -c16 * a + c56 * b + c13 * c, p1 = c13 * b + c56 * c - c16 * d;
    const double p2 = c116 * c - c76 * d + c13 * e;
    const double a0 = 0.3 * r0, a2 = 0.1 * r2, is = 1. / (a0 + r1 + a2);
    double o0 = a0 * is, o1 = r1 * is, o2 = a2 * is;
    const double W = o0 * p0 + o1 * p1 + o2 * p2;
    if (clip && W < 0.) glo = 0.;
    o0 *= glo, o1 *= glo, o2 *= glo;
    gb0 = -2. * o0 * (p0 - W) * i0;
    gb1 = -2. * o1 * (p1 - W) * i1;
    gb2 = -2. * o2 * (p2 - W) * i2;
    t[0] = -c16 * o0;
    t[1] = c56 * o0 + c13 * o1;
    t[2] = c13 * o0 + c56 * o1 + c116 * o2;
    t[3] = -c16 * o1 - c76 * o2;
    t[4] = c13 * o2;
  }
  {  // high side: mirrored
    const double p0 = -c16 * e + c56 * d + c13 * c, p1 = c13 * d + c56 * c - c16 * b;
    const double p2 = c116 * c - c76 * b + c13 * a;
    const double a0 = 0.3 * r2, a2 = 0.1 * r0, is = 1. / (a0 + r1 + a2);
    double o0 = a0 * is, o1 = r1 * is, o2 = a2 * is;
    const double W = o0 * p0 + o1 * p1 + o2 * p2;
    if (clip && W < 0.) ghi = 0.;
    o0 *= ghi, o1 *= ghi, o2 *= ghi;
    gb2 += -2. * o0 * (p0 - W) * i2;
    gb1 += -2. * o1 * (p1 - W) * i1;
    gb0 += -2. * o2 * (p2 - W) * i0;
    t[4] += -c16 * o0;
    t[3] += c56 * o0 + c13 * o1;
    t[2] += c13 * o0 + c56 * o1 + c116 * o2;
    t[1] += -c16 * o1 - c76 * o2;
    t[0] += c13 * o2;
  }
  t[0] += gb0 * (k13 * u0 + 0.5 * v0);
  t[1] += gb0 * (-2. * k13 * u0 - 2. * v0) + gb1 * (k13 * u1 - 0.5 * v1);
  t[2] += gb0 * (k13 * u0 + 1.5 * v0) + gb1 * (-2. * k13 * u1) + gb2 * (k13 * u2 + 1.5 * v2);
  t[3] += gb1 * (k13 * u1 + 0.5 * v1) + gb2 * (-2. * k13 * u2 - 2. * v2);
  t[4] += gb2 * (k13 * u2 + 0.5 * v2);
}

// the same for every reconstruction of cell_states
__device__ __forceinline__ void cell_states_vjp(int type, bool scale, const double* q, bool clip,
                                                double glo, double ghi, double* t) {
  if (type == SNAPB_RECON_WENO5 && !scale) {
    weno5_cell_vjp(q, clip, glo, ghi, t);
    return;
  }
  if (clip) {
    double lo, hi;
    cell_states(type, scale, q, lo, hi);
    if (lo < 0.) glo = 0.;
    if (hi < 0.) ghi = 0.;
  }
#pragma unroll
  for (int k = 0; k < 5; ++k) t[k] = 0.;
  switch (type) {
    case SNAPB_RECON_WENO5: {
      weno5_face_vjp(q[0], q[1], q[2], q[3], q[4], scale, glo, t);
      double h[5] = {0., 0., 0., 0., 0.};
      weno5_face_vjp(q[4], q[3], q[2], q[1], q[0], scale, ghi, h);
#pragma unroll
      for (int k = 0; k < 5; ++k) t[k] += h[4 - k];
      return;
    }
    case SNAPB_RECON_CP5: {
      const double w[5] = {-1. / 20., 9. / 20., 47. / 60., -13. / 60., 1. / 30.};
#pragma unroll
      for (int k = 0; k < 5; ++k) t[k] = w[k] * glo + w[4 - k] * ghi;
      return;
    }
    case SNAPB_RECON_CP3: {
      const double w[3] = {1. / 3., 5. / 6., -1. / 6.};
#pragma unroll
      for (int k = 0; k < 3; ++k) t[k + 1] = w[k] * glo + w[2 - k] * ghi;
      return;
    }
    case SNAPB_RECON_DC:
      t[2] = glo + ghi;
      return;
    default:
      // WENO3 and PLM: one dual pass per inner window slot
      for (int s = 1; s < 4; ++s) {
        Dual qd[5], lo, hi;
#pragma unroll
        for (int k = 0; k < 5; ++k) qd[k] = Dual(q[k], k == s ? 1. : 0.);
        cell_states<Dual>(type, scale, qd, lo, hi);
        t[s] = glo * lo.d + ghi * hi.d;
      }
  }
}

}  // namespace snapb
