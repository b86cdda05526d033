// cells.cuh — what the cell-centred sweeps of both forms share: the face values
// of a cell, the isentropic x1 ghosts, and the split of the x1 sweep.
#pragma once

#include "common.cuh"

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
        T a = q[0], b = q[1], c = q[2], d = q[3], e = q[4], vs = T(1);
        if (scale) {
          vs = (fabs(a) + fabs(b) + fabs(c) + fabs(d) + fabs(e)) / T(5);
          if (vs == T(0)) {
            lo = hi = T(0);
            return;
          }
          const T iv = T(1) / vs;
          a *= iv, b *= iv, c *= iv, d *= iv, e *= iv;
        }
        const T c16 = T(1. / 6.), c56 = T(5. / 6.), c13 = T(1. / 3.), c116 = T(11. / 6.),
                c76 = T(7. / 6.), c1312 = T(13. / 12.), eps = T(1e-6), q4 = T(0.25);
        const T s0 = sqr(c1312 * sqr(a - T(2) * b + c) + q4 * sqr(a - T(4) * b + T(3) * c) + eps);
        const T s1 = sqr(c1312 * sqr(b - T(2) * c + d) + q4 * sqr(d - b) + eps);
        const T s2 = sqr(c1312 * sqr(c - T(2) * d + e) + q4 * sqr(T(3) * c - T(4) * d + e) + eps);
        // weights over the common denominator s0 s1 s2: one division a side
        const T s12 = s1 * s2, s01 = s0 * s1, n1 = T(0.6) * (s0 * s2);
        const T m01 = c56 * b + c13 * c, m10 = c13 * b + c56 * c;  // shared candidate parts
        const T m23 = c56 * c + c13 * d, m32 = c13 * c + c56 * d;
        {
          const T n0 = T(0.3) * s12, n2 = T(0.1) * s01;
          lo = vs * ((n0 * (m01 - c16 * a) + n1 * (m10 - c16 * d) +
                      n2 * (c116 * c - c76 * d + c13 * e)) / (n0 + n1 + n2));
        }
        {
          const T n0 = T(0.3) * s01, n2 = T(0.1) * s12;
          hi = vs * ((n0 * (m32 - c16 * e) + n1 * (m23 - c16 * b) +
                      n2 * (c116 * c - c76 * b + c13 * a)) / (n0 + n1 + n2));
        }
        break;
      }
    }
    case SNAPB_RECON_CP5: {
      const T a = T(-1. / 20.), b = T(9. / 20.), c = T(47. / 60.), d = T(-13. / 60.),
              e = T(1. / 30.);
      lo = a * q[0] + b * q[1] + c * q[2] + d * q[3] + e * q[4];
      hi = a * q[4] + b * q[3] + c * q[2] + d * q[1] + e * q[0];
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

// Split of the x1 sweep over warps: an item is either K whole columns
// (consecutive, so their cells are one contiguous span per variable) or one of
// nseg segments of seglen cells of a single column.
struct X1Split {
  int K, nseg, seglen;
  int pitch;  // doubles per variable row in the warp's shared memory
};

// Isentropic density and pressure of ghost level n (1 = next to the interior)
// from the edge cell's: with a = (gamma - 1) / gamma the recurrence
// p_{n+1}^a = p_n^a +- a g dz / K^(1/gamma) is linear in p^a, so every level
// follows from the edge directly.  With q = p_e^(1/gamma) the other powers
// are quotients (p_e^a = p_e / q, K^(1/gamma) = q / rho_e,
// p^(1/gamma) = p / p^a), which leaves two pow calls per level.
__device__ __forceinline__ void isentropic_ghost(double gamma, double gdz, int top, int n,
                                                 double pe, double re, double& pn, double& rn) {
  const double a = (gamma - 1.) / gamma, q = pow(pe, 1. / gamma);
  const double h = (pe + (top ? -n : n) * a * gdz * re) / q;
  pn = pow(h, 1. / a);
  rn = pn / h * (re / q);
}

// The split for a block: rows of at most row_bytes a warp where some split has
// them, `resident` warps on the GPU at once (whole: no segments).
X1Split x1_split(const Geo& g, int nvt, size_t item, size_t row_bytes, double resident, bool whole);

}  // namespace snapb
