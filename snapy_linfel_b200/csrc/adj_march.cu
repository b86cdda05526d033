// adj_march.cu — reverse of the FP64 x2 / x3 sweeps of one stage.
#include <algorithm>

#include "adj_bufs.cuh"
#include "cells_adj.cuh"
#include "ring.cuh"
#include "riemann_adj.cuh"

namespace snapb {

constexpr int kAdjThreads = 128;
constexpr int kAdjSlots = 7;  // cells c-3 .. c+2 and the next one

// Reconstruction profile of the reverse: RP 1 the default one (WENO5 for
// density and scalars, the linear 5-point interpolation for velocities and
// pressure), RP 0 every choice at run time.
template <int RP>
__device__ __forceinline__ void adj_states(int type, bool scale, int v, const double* q, double& lo,
                                           double& hi) {
  if constexpr (RP == 1)
    cell_states(v == IDN || v >= 5 ? SNAPB_RECON_WENO5 : SNAPB_RECON_CP5, false, q, lo, hi);
  else
    cell_states(type, scale, q, lo, hi);
  if (v >= 5) {
    lo = lo < 0. ? 0. : lo;
    hi = hi < 0. ? 0. : hi;
  }
}
template <int RP>
__device__ __forceinline__ void adj_states_vjp(int type, bool scale, int v, const double* q,
                                               double glo, double ghi, double* t) {
  if constexpr (RP == 1)
    cell_states_vjp(v == IDN || v >= 5 ? SNAPB_RECON_WENO5 : SNAPB_RECON_CP5, false, q, v >= 5, glo,
                    ghi, t);
  else
    cell_states_vjp(type, scale, q, v >= 5, glo, ghi, t);
}

// Reverse of the fluxes of one face with states L, R (scalars clipped):
// cotangents gF of the NV fluxes onto gL, gR.
template <int NS, int SV>
__device__ __forceinline__ void flux_vjp(const Phys& p, int ivx, const double* L, const double* R,
                                         const double* gFin, double* gL, double* gR) {
#pragma unroll
  for (int v = 0; v < 5 + NS; ++v) gL[v] = gR[v] = 0.;
  double gF[5];
#pragma unroll
  for (int v = 0; v < 5; ++v) gF[v] = gFin[v];
  if constexpr (NS > 0) {
    // scalar upwind flux F_s = F[IDN] * (F[IDN] > 0 ? r_L : r_R)
    double F[5];
    riemann_flux(SV < 0 ? p.riemann : SV, L, R, ivx, p.gammad, F);
#pragma unroll
    for (int n = 0; n < NS; ++n) {
      const double gs = gFin[5 + n];
      const bool up = F[IDN] > 0.;
      gF[IDN] += gs * (up ? L[5 + n] : R[5 + n]);
      gL[5 + n] = up ? gs * F[IDN] : 0.;
      gR[5 + n] = up ? 0. : gs * F[IDN];
    }
  }
  riemann_vjp_rev(SV < 0 ? p.riemann : SV, L, R, ivx, p.gammad, gF, gL, gR);
}

// One thread per (x1 cell, other horizontal index) and segment of cells of the
// sweep axis.  Cell centred: a step forms the face values of cell c, reverses
// the fluxes of face c and then the face values of cell c - 1, whose two face
// cotangents are complete, onto its five-cell window.  The window of
// primitives is the thread's ring in shared memory, the window of cotangents
// five registers a variable, stored when its oldest cell is complete (with
// atomics where another segment adds to the cell too).
//
// Bound: FP64 issue at 8 to 12 warps per SM.  Against a face-centred reverse
// with both six-cell windows in registers: 512 x 256 HLLC 58 -> 39 us, 64 x 60 x
// 48 Roe with two tracers 168 -> 65 us (x2), 62 us (x3).
template <int NS, int AX, int RP, int SV>
__global__ void __launch_bounds__(kAdjThreads, NS == 0 ? 3 : 2)
    k_march_adj(Geo g, Phys p, AdjBufs b, int seglen) {
  constexpr int NV = 5 + NS, SL = NV * kAdjThreads;
  extern __shared__ double adj_ring[];
  const int ni = g.iu - g.il + 1;
  int lo, hi, olo, ohi;
  int64_t st, ost;
  if (AX == 2) {
    lo = g.jl, hi = g.ju, st = g.s2, olo = g.kl, ohi = g.ku, ost = g.s3;
  } else {
    lo = g.kl, hi = g.ku, st = g.s3, olo = g.jl, ohi = g.ju, ost = g.s2;
  }
  const int no = ohi - olo + 1;
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (tid >= (int64_t)ni * no) return;
  const int i = g.il + umod(tid, ni), o = olo + udiv(tid, ni);
  // cells s0 .. s1 of lo-1 .. hi+1 belong to this segment
  const int s0 = lo - 1 + blockIdx.y * seglen;
  if (s0 > hi + 1) return;
  const int s1 = min(s0 + seglen - 1, hi + 1);
  const int64_t base = i + o * ost, sv = g.sv;
  constexpr int ivx = AX == 2 ? IVY : IVZ;
  const bool disabled = (AX == 2 ? p.disable2 : p.disable3) != 0;
  const double cf = *b.dt * (AX == 2 ? g.A2 : g.A3) / g.vol;
  double* ring = adj_ring + threadIdx.x;

  // first cell whose face values are formed: s0 - 1 for the face below s0
  const int cs = max(s0 - 1, lo - 1);
  int64_t src = base + (int64_t)(cs - 2) * st;
  int next = cs - 2;
  auto load = [&](int slot) {  // cell `next`; past the array's end nothing is needed
    if (next <= hi + 3) {
      double* dst = ring + slot * SL;
#pragma unroll
      for (int v = 0; v < 5; ++v) cp_async_bytes8(dst + v * kAdjThreads, b.W + v * sv + src);
#pragma unroll
      for (int n = 0; n < NS; ++n)
        cp_async_bytes8(dst + (5 + n) * kAdjThreads, b.R + n * sv + src);
    }
    cp_async_commit();
    src += st;
    ++next;
  };
#pragma unroll
  for (int t = 1; t < 6; ++t) load(t);  // slots of cells cs-2 .. cs+2 (slot 0: cs-3)
  double H[NV], glo[NV], acc[NV][5], gm[NV];
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    H[v] = glo[v] = 0.;
#pragma unroll
    for (int t = 0; t < 5; ++t) acc[v][t] = 0.;
    gm[v] = cs - 1 >= lo && cs - 1 <= hi ? b.GD[v * sv + base + (int64_t)(cs - 1) * st] : 0.;
  }
  auto flush = [&](int cell, int slot) {
    double* out = b.GW + base + (int64_t)cell * st;
    // cells that no other segment reaches: more than one inside both ends
    const bool own = (cell >= s0 + 2 || s0 == lo - 1) && (cell <= s1 - 2 || s1 == hi + 1);
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      if (acc[v][slot] == 0.) continue;
      if (own)
        out[v * sv] += acc[v][slot];
      else
        atomicAdd(out + v * sv, acc[v][slot]);
    }
  };
  int z = 0;  // slot of cell c - 3
  for (int c = cs; c <= s1 + 1; ++c) {
    int at[kAdjSlots];
#pragma unroll
    for (int t = 0; t < kAdjSlots; ++t) at[t] = z + t >= kAdjSlots ? z + t - kAdjSlots : z + t;
    z = at[1];
    cp_async_wait<0>();  // cell c + 2 has landed
    load(at[6]);
    double gL[NV], gR[NV];
    const bool face = c >= s0 && c >= lo && c <= hi + 1;  // (the face between c - 1 and c)
    double R[NV], Hn[NV];
    if (c <= hi + 1) {
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        double q[5];
#pragma unroll
        for (int t = 0; t < 5; ++t) q[t] = ring[at[t + 1] * SL + v * kAdjThreads];
        const int typ = v >= 5 ? p.rs_type
                               : (p.r23_shock || v == IDN ? p.r23_type : interp2_of(p.r23_type));
        adj_states<RP>(typ, v >= 5 ? p.rs_scale != 0 : p.r23_scale != 0, v, q, R[v], Hn[v]);
      }
    }
    double gp[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v)
      gp[v] = c >= lo && c <= hi ? b.GD[v * sv + base + (int64_t)c * st] : 0.;
    if (face && !disabled) {
      double gF[NV];
#pragma unroll
      for (int v = 0; v < NV; ++v) gF[v] = cf * (gp[v] - gm[v]);
      flux_vjp<NS, SV>(p, ivx, H, R, gF, gL, gR);
    } else {
#pragma unroll
      for (int v = 0; v < NV; ++v) gL[v] = gR[v] = 0.;
    }
    if (c > s0) {  // cell c - 1: both of its faces are done
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        double q[5], t5[5];
#pragma unroll
        for (int t = 0; t < 5; ++t) q[t] = ring[at[t] * SL + v * kAdjThreads];
        const int typ = v >= 5 ? p.rs_type
                               : (p.r23_shock || v == IDN ? p.r23_type : interp2_of(p.r23_type));
        adj_states_vjp<RP>(typ, v >= 5 ? p.rs_scale != 0 : p.r23_scale != 0, v, q, glo[v], gL[v],
                           t5);
#pragma unroll
        for (int t = 0; t < 5; ++t) acc[v][t] += t5[t];
      }
      flush(c - 3, 0);
#pragma unroll
      for (int v = 0; v < NV; ++v) {
#pragma unroll
        for (int t = 0; t < 4; ++t) acc[v][t] = acc[v][t + 1];
        acc[v][4] = 0.;
      }
    }
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      glo[v] = gR[v];
      H[v] = Hn[v];
      gm[v] = gp[v];
    }
  }
  // after the shifts, slot t holds cell s1 - 1 + t
#pragma unroll
  for (int t = 0; t < 4; ++t) flush(s1 - 1 + t, t);
  cp_async_wait<0>();
}

template <int NS, int RP, int SV>
static cudaError_t launch_t(int axis, const Geo& g, const Phys& p, const AdjBufs& b,
                            cudaStream_t st) {
  const int ni = g.iu - g.il + 1, nax = (axis == 2 ? g.nx2 : g.nx3) + 2;
  const int no = axis == 2 ? g.ku - g.kl + 1 : g.ju - g.jl + 1;
  const int64_t lines = (int64_t)ni * no;
  // enough (line, segment) pairs for ~2 waves of 148 SMs x 3 CTAs, segments of
  // at least 8 cells (a segment repeats one face)
  const int64_t want = 148LL * 3 * kAdjThreads * 2;
  int nseg = (int)std::min<int64_t>(std::max<int64_t>(1, want / std::max<int64_t>(lines, 1)),
                                    (nax + 7) / 8);
  const int seglen = std::max(4, (nax + nseg - 1) / nseg);
  nseg = (nax + seglen - 1) / seglen;
  const dim3 grid((unsigned)((lines + kAdjThreads - 1) / kAdjThreads), (unsigned)nseg);
  constexpr size_t smem = (size_t)kAdjSlots * (5 + NS) * kAdjThreads * sizeof(double);
  if (axis == 2) {
    raise_smem_limit(k_march_adj<NS, 2, RP, SV>, smem);
    k_march_adj<NS, 2, RP, SV><<<grid, kAdjThreads, smem, st>>>(g, p, b, seglen);
  } else {
    raise_smem_limit(k_march_adj<NS, 3, RP, SV>, smem);
    k_march_adj<NS, 3, RP, SV><<<grid, kAdjThreads, smem, st>>>(g, p, b, seglen);
  }
  return cudaGetLastError();
}

template <int NS>
static cudaError_t launch_ns(int axis, const Geo& g, const Phys& p, const AdjBufs& b,
                             cudaStream_t st) {
  const bool standard = p.r23_type == SNAPB_RECON_WENO5 && !p.r23_shock && !p.r23_scale &&
                        (NS == 0 || (p.rs_type == SNAPB_RECON_WENO5 && !p.rs_scale));
  if (!standard) return launch_t<NS, 0, -1>(axis, g, p, b, st);
  switch (p.riemann) {
    case SNAPB_RIEMANN_LMARS: return launch_t<NS, 1, SNAPB_RIEMANN_LMARS>(axis, g, p, b, st);
    case SNAPB_RIEMANN_HLLC: return launch_t<NS, 1, SNAPB_RIEMANN_HLLC>(axis, g, p, b, st);
    default: return launch_t<NS, 1, SNAPB_RIEMANN_ROE>(axis, g, p, b, st);
  }
}

cudaError_t launch_march_adj(int axis, const Geo& g, const Phys& p, const AdjBufs& b,
                             cudaStream_t st) {
  switch (p.nscalar) {
    case 0: return launch_ns<0>(axis, g, p, b, st);
    case 1: return launch_ns<1>(axis, g, p, b, st);
    case 2: return launch_ns<2>(axis, g, p, b, st);
    case 3: return launch_ns<3>(axis, g, p, b, st);
  }
  return cudaErrorInvalidValue;
}

}  // namespace snapb
