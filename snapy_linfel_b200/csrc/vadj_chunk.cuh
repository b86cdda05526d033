// vadj_chunk.cuh — launcher of the one-warp column solves of the implicit
// adjoint (vadj_chunk.cu).
#pragma once

#include "kernels.cuh"

namespace snapb {

struct VadjChunk {
  const double* dt;
  const double* W;   // primitives of the stage input
  const double* R;   // mixing ratios
  const double* D;   // explicit du
  const double* GD;  // cotangents of the stage's du (and scalars)
  double* out;       // [6][columns][layers]: delta rows, then t rows
  double* Z;         // [3][columns]: B_dry / S, g_S, g_B
};

bool vadj_chunk_applies(const Geo& g, const Phys& p);
cudaError_t launch_vadj_chunk(const Geo& g, const Phys& p, const VadjChunk& in, cudaStream_t st);

}  // namespace snapb
