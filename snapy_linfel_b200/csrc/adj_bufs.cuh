// adj_bufs.cuh — device buffers of the reverse of one stage, and the launcher of
// its x2 / x3 sweeps (adj_march.cu).
#pragma once

#include "kernels.cuh"

namespace snapb {

// Buffers of the stage adjoint (all [var][sv], FP64)
struct AdjBufs {
  const double* dt;
  const double* u;   // stage-start state (ghosts filled)
  const double* s;
  const double* W;   // primitives of u with the x1 ghost revision (recomputed)
  const double* R;   // mixing ratios s / rho (recomputed)
  const double* D;   // explicit du (recomputed; implicit solve only)
  double* GD;        // cotangent of du (nvar + ns); rows replaced by the VIC adjoint
  double* GW;        // cotangent of w (nvar) and r (ns), accumulated
  double* gu;        // out: += cotangent of u
  double* gs;        // out: += cotangent of s
  double* vic;       // VIC adjoint scratch
};

cudaError_t launch_march_adj(int axis, const Geo& g, const Phys& p, const AdjBufs& b,
                             cudaStream_t st);

}  // namespace snapb
