// vic_chunk.cu — launchers of the one-warp implicit solve (vic_chunk.cuh): the
// FP64 form, the FP32 form and the batched ensembles.
#include "vic_chunk.cuh"

namespace snapb {

// CTAs of one warp: nothing is shared between warps, and the shared memory of
// a column length need not divide by more.
template <int G, int NS, class B>
__global__ void __launch_bounds__(32) k_vic_chunk(const __grid_constant__ Geo g,
                                                       const __grid_constant__ Phys p,
                                                       const __grid_constant__ B b, int m) {
  extern __shared__ double chunk_sm[];
  vic_chunk<G, NS, B>(g, p, b, (int64_t)blockIdx.x * (32 / G), m, chunk_sm);
}

// Persistent batched form over the members whose columns take G lanes: an item
// is `chunk_groups` column groups of a member; the next item is claimed while
// the current one is worked on.
template <int G, int NS>
__global__ void __launch_bounds__(32)
    k_vic_chunk_batch(const Member32* __restrict__ mem, const __grid_constant__ Phys p, WorkQueue q,
                      int stage) {
  extern __shared__ double chunk_sm[];
  __shared__ Member32 s_mem;
  constexpr int CW = 32 / G;
  const int lane = threadIdx.x;
  unsigned long long item = 0, ahead = 0;
  if (lane == 0) item = atomicAdd(q.counter, 1ULL);
  item = __shfl_sync(0xffffffffu, item, 0);
  int m = -1;
  while (true) {
    int nm;
    int64_t tile;
    if (!queue_find(q, (int64_t)item, nm, tile)) return;
    if (lane == 0) ahead = atomicAdd(q.counter, 1ULL);
    if (nm != m) {
      __syncwarp();
      load_member_warp(s_mem, mem, nm);
      if (lane == 0) set_stage32(s_mem.b, stage);
      __syncwarp();
      m = nm;
    }
    const Geo& g = s_mem.g;
    const int64_t ncol = (int64_t)(g.ju - g.jl + 1) * (g.ku - g.kl + 1);
    const int rows = (g.nx1 + G - 1) / G;
    const int64_t c0 = tile * s_mem.chunk_groups * CW;
    for (int r = 0; r < s_mem.chunk_groups && c0 + r * CW < ncol; ++r) {
      vic_chunk<G, NS, StageBufs32>(g, p, s_mem.b, c0 + r * CW, rows, chunk_sm);
      __syncwarp();  // the group's shared memory is free
    }
    item = __shfl_sync(0xffffffffu, ahead, 0);
  }
}

template <class B>
static cudaError_t launch_chunk(const Geo& g, const Phys& p, const B& b, cudaStream_t st) {
  const int lanes = chunk_lanes(g.nx1), m = chunk_layers(g.nx1), cw = 32 / lanes;
  const int64_t ncol = (int64_t)(g.ju - g.jl + 1) * (g.ku - g.kl + 1);
  return with_lanes_scalars(lanes, p.nscalar, [&](auto gl, auto ns) {
    constexpr int G = decltype(gl)::value, NS = decltype(ns)::value;
    raise_smem_limit(k_vic_chunk<G, NS, B>, 200 * 1024);
    k_vic_chunk<G, NS, B><<<(unsigned)((ncol + cw - 1) / cw), 32, chunk_smem_bytes(m), st>>>(
        g, p, b, m);
    return cudaGetLastError();
  });
}

bool vic_chunk_applies(const Geo& g, const Phys& p) { return chunk_applies(g, p); }
int vic_chunk_lanes(int nl) { return chunk_lanes(nl); }

cudaError_t launch_vic_chunk(const Geo& g, const Phys& p, const StageBufs& b, cudaStream_t st) {
  return launch_chunk(g, p, b, st);
}
cudaError_t launch_vic_chunk32(const Geo& g, const Phys& p, const StageBufs32& b,
                               cudaStream_t st) {
  return launch_chunk(g, p, b, st);
}

cudaError_t launch_vic_chunk_batch(const Member32* mem, const Phys& p, const WorkQueue& q,
                                   int stage, int lanes, int max_layers, const PersistGrid& pg,
                                   cudaStream_t st) {
  const size_t smem = chunk_smem_bytes((max_layers + lanes - 1) / lanes);
  return with_lanes_scalars(lanes, p.nscalar, [&](auto gl, auto ns) {
    constexpr int G = decltype(gl)::value, NS = decltype(ns)::value;
    raise_smem_limit(k_vic_chunk_batch<G, NS>, 200 * 1024);
    k_vic_chunk_batch<G, NS><<<persistent_grid(k_vic_chunk_batch<G, NS>, 32, smem, pg), 32, smem,
                               st>>>(mem, p, q, stage);
    return cudaGetLastError();
  });
}

}  // namespace snapb
