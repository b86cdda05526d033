// cells.cuh — what the cell-centred sweeps of both forms share: the face values
// of a cell and the isentropic x1 ghosts.
#pragma once

#include "common.cuh"
#include "x1_split.cuh"

namespace snapb {

// ---------------------------------------------------------------------------
// Cell-centred reconstruction: from the cells c-2 .. c+2 (q[0..4]) the value
// at the cell's left face (wr of face c) and at its right face (wl of face
// c+1).  The same formulas as face_states (common.cuh); for WENO5 the two
// sides share the three smoothness measures.
// ---------------------------------------------------------------------------
template <class T>
__device__ __forceinline__ void cell_states(int type, bool scale, const T* q, T& lo, T& hi) {
  switch (type) {
    case SNAPB_RECON_WENO5: {
      if constexpr (sizeof(T) != 8) {
        // FP32 (and dual numbers): each side by itself.  Shared measures take
        // 8 to 11 % off the sweeps (384 x 384 x 192: x1 1.25 -> 1.15 ms, x2
        // 0.79 -> 0.69, x3 0.84 -> 0.74), but sum them in another order for one
        // side; the FP32 state then differs in its last bits from the
        // face-centred one, and with it now and then the time step.
        lo = weno5_face(q[0], q[1], q[2], q[3], q[4], scale);
        hi = weno5_face(q[4], q[3], q[2], q[1], q[0], scale);
        break;
      } else {
        // Written so that the reversed window gives lo and hi exchanged, to the
        // bit: at a reflecting wall both sides of the face then hold mirrored
        // states, and its mass flux is zero instead of a rounding error.
        T a = q[0], b = q[1], c = q[2], d = q[3], e = q[4], vs = T(1);
        if (scale) {
          vs = (((fabs(a) + fabs(e)) + (fabs(b) + fabs(d))) + fabs(c)) / T(5);
          if (vs == T(0)) {
            lo = hi = T(0);
            return;
          }
          const T iv = T(1) / vs;
          a *= iv, b *= iv, c *= iv, d *= iv, e *= iv;
        }
        auto M = [](T x, T y) { return __dmul_rn(x, y); };
        auto S = [](T x, T y) { return __dadd_rn(x, y); };
        const T c16 = 1. / 6., c56 = 5. / 6., c13 = 1. / 3., c116 = 11. / 6., c76 = 7. / 6.,
                c1312 = 13. / 12.;
        auto measure = [&](T u, T w) {
          const T t = fma(M(c1312, u), u, fma(M(T(0.25), w), w, T(1e-6)));
          return M(t, t);
        };
        const T s0 = measure(S(fma(T(-2), b, a), c), fma(T(3), c, fma(T(-4), b, a)));
        const T s1 = measure(fma(T(-2), c, S(b, d)), S(d, -b));
        const T s2 = measure(S(fma(T(-2), d, e), c), fma(T(3), c, fma(T(-4), d, e)));
        // weights over the common denominator s0 s1 s2: one division a side
        const T s12 = M(s1, s2), s01 = M(s0, s1), n1 = M(T(0.6), M(s0, s2));
        const T k13 = M(c13, c), k56 = M(c56, c), k116 = M(c116, c);
        auto side = [&](T n0, T n2, T x0, T x1, T x3, T x4) {
          const T p0 = fma(-c16, x0, fma(c56, x1, k13)), p1 = fma(-c16, x3, fma(c13, x1, k56));
          const T p2 = fma(c13, x4, fma(-c76, x3, k116));
          return M(vs, fma(n2, p2, fma(n1, p1, M(n0, p0))) / S(S(n0, n1), n2));
        };
        lo = side(M(T(0.3), s12), M(T(0.1), s01), a, b, d, e);
        hi = side(M(T(0.3), s01), M(T(0.1), s12), e, d, b, a);
        break;
      }
    }
    case SNAPB_RECON_CP5: {
      const T a = T(-1. / 20.), b = T(9. / 20.), c = T(47. / 60.), d = T(-13. / 60.),
              e = T(1. / 30.);
      if constexpr (sizeof(T) == 8) {  // (mirrored to the bit, as above)
        auto side = [&](T x0, T x1, T x3, T x4) {
          return fma(e, x4, fma(d, x3, fma(c, q[2], fma(b, x1, __dmul_rn(a, x0)))));
        };
        lo = side(q[0], q[1], q[3], q[4]);
        hi = side(q[4], q[3], q[1], q[0]);
      } else {
        lo = a * q[0] + b * q[1] + c * q[2] + d * q[3] + e * q[4];
        hi = a * q[4] + b * q[3] + c * q[2] + d * q[1] + e * q[0];
      }
      break;
    }
    case SNAPB_RECON_WENO3:
      lo = weno3_face(q[1], q[2], q[3], scale);
      hi = weno3_face(q[3], q[2], q[1], scale);
      break;
    case SNAPB_RECON_CP3: {
      const T a = T(1. / 3.), b = T(5. / 6.), c = T(-1. / 6.);
      lo = a * q[1] + b * q[2] + c * q[3];
      hi = a * q[3] + b * q[2] + c * q[1];
      break;
    }
    case SNAPB_RECON_PLM: {
      // harmonic-mean slope with FLT_MIN guard, zeroed across extrema
      const T dl = q[2] - q[1], dr = q[3] - q[2], d2 = dl * dr;
      T m = fdiv(T(2) * d2, dl + dr + T(1.1754943508222875e-38));
      m = d2 >= T(0) ? m : T(0);
      lo = q[2] - T(0.5) * m;
      hi = q[2] + T(0.5) * m;
      break;
    }
    default:  // donor cell
      lo = hi = q[2];
  }
}

// Isentropic density and pressure of ghost level n (1 = next to the interior)
// from the edge cell's: with a = (gamma - 1) / gamma the recurrence
// p_{n+1}^a = p_n^a +- a g dz / K^(1/gamma) is linear in p^a, so every level
// follows from the edge directly, and with y = p_n^a / p_e^a = 1 +- n a g dz
// rho_e / p_e (K^(1/gamma) = p_e^(1/gamma) / rho_e and p_e^a p_e^(1/gamma) = p_e)
// p_n = p_e y^(1/a), rho_n = rho_e y^(1/a) / y.  y is near one, so the rounding
// of the exponent does not grow with log p as it does in powers of p itself:
// against 45 digits the pressure is off by 1.7e-16 on average (8e-16 at most), by
// 1.05e-15 (4.1e-15) from powers of p_e.
__device__ __forceinline__ void isentropic_ghost(double gamma, double gdz, int top, int n,
                                                 double pe, double re, double& pn, double& rn) {
  const double a = (gamma - 1.) / gamma;
  // (a negative pressure or density has no adiabat)
  const double y = pe < 0. || re < 0. ? __longlong_as_double(0x7ff8000000000000ll)
                                      : 1. + (top ? -n : n) * a * gdz * re / pe;
  const double z = pow(y, 1. / a);
  pn = pe * z;
  rn = re * z / y;
}

}  // namespace snapb
