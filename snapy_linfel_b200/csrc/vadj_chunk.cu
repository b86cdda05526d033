// vadj_chunk.cu — the two column solves of the implicit adjoint (3x3 blocks),
// one warp per group of columns (vic_chunk.cuh): A delta = du / dt again, then
// A^T t = g_delta + (g_fix - V g_B) e_0 with the transposed blocks, both from
// the primitive state.  g_B = Q / S needs only column sums, so the second
// right-hand side is known after the first pass.
//
// Against cyclic reduction by one CTA per column (block_cr.cuh) from blocks
// that an assembly kernel wrote: 512 columns of 256 layers, 151 -> 30 us a
// stage; 3840 columns of 48 layers, 298 -> 38 us.
#include "vadj_chunk.cuh"
#include "vic_chunk.cuh"

namespace snapb {

// The equations of one lane's chunk in one of the two passes: A delta = du / dt,
// or (tr) A^T t = g_delta + (g_fix - V g_B) e_0.
template <int NS>
struct VadjColumn {
  const Geo& g;
  const VadjChunk& in;
  const int cb, l0, m, sv, nl;
  const bool tr;
  double gb, gog, idt;
  ChunkBlocks<double> blocks;
  double raw[5], rawd[3], fix = 0., gi = 0., rc;
  double sum_r2 = 0., sum_du = 0., sum_g = 0.;

  __device__ __forceinline__ void load_w(int l, double (&x)[5]) const {
    const int o = cb + min(l, nl);
#pragma unroll
    for (int v = 0; v < 5; ++v) x[v] = in.W[v * sv + o];
  }
  __device__ __forceinline__ void load_d(int l) {
    const int o = cb + min(l, nl - 1);
    const double* src = tr ? in.GD : in.D;  // right-hand side rows
#pragma unroll
    for (int r = 0; r < 3; ++r) rawd[r] = src[sel<3>(r) * sv + o];
    gi = in.GD[IDN * sv + o];
    if (tr) {
      fix = 0.;
#pragma unroll
      for (int n = 0; n < NS; ++n) fix += in.GD[(5 + n) * sv + o] * in.R[n * sv + o];
    }
  }
  __device__ __forceinline__ void make(const double (&x)[5], ChunkCell<double>& c) const {
    c.set(x[IDN], x[IVX], x[IVY], x[IVZ], x[IPR], gog);
  }
  __device__ __forceinline__ VadjColumn(const Geo& g_, const Phys& p, const VadjChunk& in_, int cb_,
                                        int l0_, int m_, bool tr_, double gb_)
      : g(g_), in(in_), cb(cb_), l0(l0_), m(m_), sv((int)g_.sv), nl(g_.nx1), tr(tr_), gb(gb_) {
    idt = 1. / *in.dt, gog = p.gammad / (p.gammad - 1.);
    blocks.gm1 = p.gammad - 1.;
    blocks.s = g.A1 * (0.5 / g.vol);
    blocks.idt = idt;
    blocks.grav = p.grav1;
    ChunkCell<double> below, cell;
    load_w(l0 - 1, raw);
    make(raw, below);
    load_w(l0, raw);
    make(raw, cell);
    rc = raw[IDN];
    load_w(l0 + 1, raw);
    load_d(l0);
    blocks.start(below, cell);
  }
  __device__ __forceinline__ void operator()(int j, double (&a)[3][3], double (&bl)[3][3],
                                             double (&c)[3][3], double (&rhs)[3]) {
    const int l = l0 + j;
    ChunkCell<double> cn;
    make(raw, cn);
    const double rn = raw[IDN];
#pragma unroll
    for (int r = 0; r < 3; ++r) rhs[r] = l < nl ? (tr ? rawd[r] : rawd[r] * idt) : 0.;
    if (l < nl) {
      if (tr) {
        rhs[0] += fix - g.vol * gb;
      } else {
        sum_r2 += rc * rc;
        sum_du += rawd[0];
        sum_g += gi * rc * rc;
      }
    }
    if (j < m - 1) {
      load_w(l + 2, raw);
      load_d(l + 1);
    }
    blocks.template next<true>(cn, l, nl, tr, a, bl, c);
    rc = rn;
  }
};

// (as chunk_again, vic_chunk.cuh)
template <int G, int NS>
__device__ __noinline__ void vadj_again(const Geo& g, const Phys& p, const VadjChunk& in, int cb,
                                        int m, double* mine, bool tr, double gb, bool again) {
  const int k = threadIdx.x & (G - 1);
  VadjColumn<NS> column(g, p, in, cb, k * m, m, tr, gb);
  chunk_sequence<G>(m, k, mine, again, column);
}

template <int G, int NS>
__global__ void __launch_bounds__(32)
    k_vadj_chunk(const __grid_constant__ Geo g, const __grid_constant__ Phys p,
                 const __grid_constant__ VadjChunk in, int m) {
  extern __shared__ double chunk_sm[];
  constexpr int CW = 32 / G;
  const int lane = threadIdx.x & 31, k = lane & (G - 1), cw = lane / G;
  const int nl = g.nx1, l0 = k * m;
  const int64_t ncol = (int64_t)(g.ju - g.jl + 1) * (g.ku - g.kl + 1);
  const int64_t col0 = (int64_t)blockIdx.x * CW;
  const int cb = (int)column_base(g, min(col0 + cw, ncol - 1));
  double* mine = chunk_sm + lane;
  double gb = 0.;
  // (unrolled: with the passes told apart at run time the second solve's call cost
  // registers, 512 x 256 with the contraction 84 -> 75 us)
#pragma unroll
  for (int pass = 0; pass < 2; ++pass) {
    const bool tr = pass == 1;
    VadjColumn<NS> column(g, p, in, cb, l0, m, tr, gb);
    double sum_x;
    const bool again =
        chunk_solve<G>(m, k, mine, kGrowthLimit<double>, column, [] {}, nl - l0, sum_x);
    if (__any_sync(0xffffffffu, again)) {
      vadj_again<G, NS>(g, p, in, cb, m, mine, tr, gb, again);
      sum_x = chunk_sum(m, mine, nl - l0);
    }
    if (!tr) {
      const double V = g.vol;
      double sum_r2 = column.sum_r2, sum_g = column.sum_g;
      double lost = column.sum_du - sum_x;
#pragma unroll
      for (int h = 1; h < G; h *= 2) {
        lost += __shfl_xor_sync(0xffffffffu, lost, h, G);
        sum_r2 += __shfl_xor_sync(0xffffffffu, sum_r2, h, G);
        sum_g += __shfl_xor_sync(0xffffffffu, sum_g, h, G);
      }
      // B_dry / S, g_S and g_B with S = V^2 sum rho^2, Q = V sum g rho^2
      const double sa2 = V * V * sum_r2, Qs = V * sum_g, bdry = lost * V;
      gb = Qs / sa2;
      if (k == 0 && col0 + cw < ncol) {
        in.Z[col0 + cw] = bdry / sa2;
        in.Z[ncol + col0 + cw] = -Qs * bdry / (sa2 * sa2);
        in.Z[2 * ncol + col0 + cw] = gb;
      }
    }
    __syncwarp();
    // the solution along x1: out [6][ncol][nl], delta rows then t rows
    const int total = (int)min((int64_t)CW, ncol - col0) * nl;
    const int magic = (65536 + m - 1) / m;
    for (int i = lane; i < total; i += 32) {
      int c = 0;
#pragma unroll
      for (int q = 1; q < CW; ++q) c += i >= q * nl;
      const int l = i - c * nl, ch = l * magic >> 16;
      const double* at = chunk_sm + (l - ch * m) * kChunkElems * 32 + c * G + ch;
#pragma unroll
      for (int r = 0; r < 3; ++r)
        in.out[((int64_t)(pass * 3 + r) * ncol + col0 + c) * nl + l] = at[r * 32];
    }
    __syncwarp();
  }
}

bool vadj_chunk_applies(const Geo& g, const Phys& p) { return chunk_applies(g, p); }

cudaError_t launch_vadj_chunk(const Geo& g, const Phys& p, const VadjChunk& in, cudaStream_t st) {
  const int lanes = chunk_lanes(g.nx1), m = chunk_layers(g.nx1), cw = 32 / lanes;
  const int64_t ncol = (int64_t)(g.ju - g.jl + 1) * (g.ku - g.kl + 1);
  return with_lanes_scalars(lanes, p.nscalar, [&](auto gl, auto ns) {
    constexpr int G = decltype(gl)::value, NS = decltype(ns)::value;
    raise_smem_limit(k_vadj_chunk<G, NS>, 200 * 1024);
    k_vadj_chunk<G, NS><<<(unsigned)((ncol + cw - 1) / cw), 32, chunk_smem_bytes(m), st>>>(
        g, p, in, m);
    return cudaGetLastError();
  });
}

}  // namespace snapb
