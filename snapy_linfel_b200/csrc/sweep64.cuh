// sweep64.cuh — the FP64 sweeps of one RK stage as templates over the scalar
// count and the face profile, instantiated by the launchers of stage.cu.
//
//   k_x1     x1 (the contiguous, vertical axis): each WARP works on its own
//            group of x1 columns (or one segment of a long column when there
//            are few): U->W into the warp's shared memory with the isentropic
//            ghost revision, W written back for the other sweeps, then the
//            cells in rounds of 32 lanes.
//   k_march  x2 / x3: one thread per (x1 cell, other horizontal index)
//            marches along the sweep axis; consecutive threads are
//            consecutive x1 cells, so every load is coalesced.
//
// Both are cell centred: a cell's left-face and right-face values come from
// one five-cell window, so the WENO5 smoothness measures (the larger part of
// the reconstruction) are formed once per cell instead of once per face side
// (110 -> 86 FP64 operations per WENO variable and cell), and the face flux
// pairs the cell's left value with its lower neighbour's right value, carried
// in registers (march) or taken from the next lower lane (x1).
#pragma once

#include <type_traits>

#include "cells.cuh"
#include "kernels.cuh"
#include "ring.cuh"

namespace snapb {

// du = -dt*div + forcing for one cell, then the RK combination (or du for the
// implicit solve).  d holds the flux-difference sums of the nvar hydro
// variables followed by the scalars; wc is the cell's primitive state, dtv
// dt / vol.
template <int NS>
__device__ __forceinline__ void finalize_cell(const Geo& g, const Phys& p, const StageBufs& b,
                                              int64_t off, const double* d, const double* wc,
                                              double dt, double dtv) {
  const int64_t sv = g.sv;
  double du[5];
#pragma unroll
  for (int v = 0; v < 5; ++v) du[v] = -dtv * d[v];
  if (p.grav1 != 0.) {
    du[IVX] += dt * wc[IDN] * p.grav1 * p.nh;
    du[IPR] += dt * wc[IDN] * wc[IVX] * p.grav1 * p.nh;
  }
  if (p.grav2 != 0.) {
    du[IVY] += dt * wc[IDN] * p.grav2;
    du[IPR] += dt * wc[IDN] * wc[IVY] * p.grav2;
  }
  if (p.grav3 != 0.) {
    du[IVZ] += dt * wc[IDN] * p.grav3;
    du[IPR] += dt * wc[IDN] * wc[IVZ] * p.grav3;
  }
  if (p.nu > 0. || p.kappa > 0.) {
#pragma unroll
    for (int v = 0; v < 5; ++v) du[v] -= dtv * b.DD[v * sv + off];
  }
  if (uses_rho_grav(g, p)) {
    double rg = b.RG[off];
    du[IVX] += dt * rg * (1. - p.nh);
    du[IPR] += dt * wc[IVX] * rg * (1. - p.nh);
  }
  double ds[NS > 0 ? NS : 1];
#pragma unroll
  for (int n = 0; n < NS; ++n) ds[n] = -dtv * d[5 + n];
  if (b.write_du) {
#pragma unroll
    for (int v = 0; v < 5; ++v) b.D[v * sv + off] = du[v];
#pragma unroll
    for (int n = 0; n < NS; ++n) b.D[(5 + n) * sv + off] = ds[n];
    return;
  }
  double unew_rho = 0.;
#pragma unroll
  for (int v = 0; v < 5; ++v) {
    int64_t o = v * sv + off;
    double uo = b.u[o];
    double u0v;
    if (b.stage == 0) {
      u0v = uo;
      b.u0[o] = uo;
    } else {
      u0v = b.u0[o];
    }
    double un = b.wgt0 * u0v + b.wgt1 * uo + b.wgt2 * du[v];
    b.u[o] = un;
    if (v == IDN) unew_rho = un;
  }
#pragma unroll
  for (int n = 0; n < NS; ++n) {
    int64_t o = n * sv + off;
    double so = b.s[o];
    double s0v;
    if (b.stage == 0) {
      s0v = so;
      b.s0[o] = so;
    } else {
      s0v = b.s0[o];
    }
    double sn = b.wgt0 * s0v + b.wgt1 * so + b.wgt2 * ds[n];
    b.s[o] = sn;
    if (b.r) b.r[o] = sn / unew_rho;
  }
}

// Face profiles: reconstruction RP and solver SV fixed at compile time.
// RP 0 reads every choice at run time; 1: the default (WENO5 for density and
// scalars, the linear 5-point interpolation for velocities and pressure); 2:
// WENO5 for every variable (the shock flag); 3: PLM for every variable; none
// scaled.  SV: a SNAPB_RIEMANN_* value, or -1 at run time.  With the choices
// folded the march of the default profile takes 116 to 128 registers (four
// CTAs per SM) where the run-time form takes 156.
template <int RP>
__device__ __forceinline__ void profile_states(int type, bool scale, int v, const double* q,
                                               double& lo, double& hi) {
  if constexpr (RP == 0)
    cell_states(type, scale, q, lo, hi);
  else if constexpr (RP == 1)
    cell_states(v == IDN || v >= 5 ? SNAPB_RECON_WENO5 : SNAPB_RECON_CP5, false, q, lo, hi);
  else if constexpr (RP == 2)
    cell_states(SNAPB_RECON_WENO5, false, q, lo, hi);
  else
    cell_states(SNAPB_RECON_PLM, false, q, lo, hi);
  if (v >= 5) {
    lo = lo < 0. ? 0. : lo;
    hi = hi < 0. ? 0. : hi;
  }
}
template <int SV>
__device__ __forceinline__ void profile_flux(int solver, const double* L, const double* R, int ivx,
                                             double gamma, double* F) {
  if constexpr (SV < 0)
    riemann_flux(solver, L, R, ivx, gamma, F);
  else
    riemann_flux(SV, L, R, ivx, gamma, F);
}

// ---------------------------------------------------------------------------
// x2 / x3 marching sweeps
// ---------------------------------------------------------------------------
constexpr int kMarchThreads = 128;
constexpr int kMarchSlots = 6;  // five cells of the window and the next one
template <int NS>
constexpr size_t march_smem_bytes() {
  return (size_t)kMarchThreads * kMarchSlots * (5 + NS) * sizeof(double);
}

// Bound: FP64 issue and the latency of its dependent chains.  A window of
// registers (NV x 6 doubles) left 8 warps per SM at 198 registers; each
// thread's window now lives in its own ring of six cells in shared memory
// (layout [slot][variable][thread], no barriers; the incoming cell by cp.async
// a step ahead), which leaves 128 registers and 16 warps.  384 x 384 x 192,
// Roe, two tracers: x2 3.67 -> 1.42 ms, x3 4.19 -> 1.49 ms a stage.  The run-time
// profile needs more than 128 registers: three CTAs, 96^3 with WENO3 x2 69.6 -> 61.9
// us, x3 120 -> 112.
template <int NS, int AX, int RP, int SV>
__global__ void __launch_bounds__(kMarchThreads, RP == 0 ? 3 : 4)
    k_march(Geo g, Phys p, StageBufs b, int seglen, int first, int last) {
  constexpr int NV = 5 + NS;
  constexpr int SL = NV * kMarchThreads;  // doubles per slot
  extern __shared__ double march_ring[];
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
  const int i = g.il + umod(tid, ni);
  const int o = olo + udiv(tid, ni);
  const int f0 = lo + blockIdx.y * seglen;
  if (f0 > hi) return;
  const int f1 = min(f0 + seglen, hi + 1);
  const int64_t sv = g.sv;
  constexpr int ivx = AX == 2 ? IVY : IVZ;
  const double A = AX == 2 ? g.A2 : g.A3;
  const int disabled = AX == 2 ? p.disable2 : p.disable3;

  double* ring = march_ring + threadIdx.x;
  const double* wsrc = b.w + i + o * ost + (int64_t)(f0 - 3) * st;
  const double* rsrc = NS ? b.R + i + o * ost + (int64_t)(f0 - 3) * st : nullptr;
  auto load = [&](int slot) {
    double* dst = ring + slot * SL;
#pragma unroll
    for (int v = 0; v < 5; ++v) cp_async_bytes8(dst + v * kMarchThreads, wsrc + v * sv);
#pragma unroll
    for (int n = 0; n < NS; ++n) cp_async_bytes8(dst + (5 + n) * kMarchThreads, rsrc + n * sv);
    cp_async_commit();
    wsrc += st;
    if (NS) rsrc += st;
  };
#pragma unroll
  for (int t = 0; t < 5; ++t) load(t);
  double L[NV], Fp[NV];
#pragma unroll
  for (int v = 0; v < NV; ++v) L[v] = Fp[v] = 0.;
  int64_t off = i + o * ost + (int64_t)(f0 - 2) * st;  // cell c - 1
  int s0 = 0;                                          // slot of cell c - 2
  for (int c = f0 - 1; c <= f1; ++c, off += st) {
    // slots of the window, oldest first; the sixth takes cell c + 3
    int at[kMarchSlots];
#pragma unroll
    for (int t = 0; t < kMarchSlots; ++t)
      at[t] = s0 + t >= kMarchSlots ? s0 + t - kMarchSlots : s0 + t;
    cp_async_wait<0>();  // cell c + 2 has landed
    if (c < f1) load(at[5]);
    s0 = at[1];
    double R[NV], H[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      double q[5];
#pragma unroll
      for (int t = 0; t < 5; ++t) q[t] = ring[at[t] * SL + v * kMarchThreads];
      const int typ = v >= 5 ? p.rs_type
                             : (p.r23_shock || v == IDN ? p.r23_type : interp2_of(p.r23_type));
      profile_states<RP>(typ, v >= 5 ? p.rs_scale != 0 : p.r23_scale != 0, v, q, R[v], H[v]);
    }
    if (c >= f0) {
      double F[NV];
      if (disabled) {
#pragma unroll
        for (int v = 0; v < 5; ++v) F[v] = 0.;
      } else {
        profile_flux<SV>(p.riemann, L, R, ivx, p.gammad, F);
      }
#pragma unroll
      for (int n = 0; n < NS; ++n)
        F[5 + n] = F[IDN] > 0. ? F[IDN] * L[5 + n] : F[IDN] * R[5 + n];
      if (c > f0) {
        double d[NV];
#pragma unroll
        for (int v = 0; v < NV; ++v) {
          d[v] = A * F[v] - A * Fp[v];
          if (!first) d[v] = b.D[v * sv + off] + d[v];
        }
        if (last) {
          double wc[5];
#pragma unroll
          for (int v = 0; v < 5; ++v) wc[v] = ring[at[1] * SL + v * kMarchThreads];
          const double dt = *b.dt;
          finalize_cell<NS>(g, p, b, off, d, wc, dt, dt / g.vol);
        } else {
#pragma unroll
          for (int v = 0; v < NV; ++v) b.D[v * sv + off] = d[v];
        }
      }
#pragma unroll
      for (int v = 0; v < NV; ++v) Fp[v] = F[v];
    }
#pragma unroll
    for (int v = 0; v < NV; ++v) L[v] = H[v];
  }
}

// ---------------------------------------------------------------------------
// x1 sweep
// ---------------------------------------------------------------------------
// Bound: FP64 issue, as the marches.  One warp per item with its own rows in
// shared memory leaves no CTA barrier (the earlier kernel, one CTA per 16
// columns, waited at four of them and kept face fluxes in shared memory too).
// 384 x 384 x 192, Roe, two tracers: 4.79 -> 2.03 ms a stage; 128^3, LMARS:
// 0.202 -> 0.093 ms; a 1-D block of 1024 cells: 43 -> 6 us.
template <int NS, int RP, int SV>
__global__ void __launch_bounds__(128, 4)
    k_x1(Geo g, Phys p, StageBufs b, X1Split sp, int64_t items) {
  constexpr int NV = 5 + NS;
  extern __shared__ double x1_rows[];
  const int lane = threadIdx.x & 31;
  const int64_t item = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (item >= items) return;  // the whole warp: nothing below synchronizes the CTA
  const int nc1 = g.nc1, il = g.il, iu = g.iu, ng = g.ng;
  const int64_t sv = g.sv, ncol = (int64_t)g.nc2 * g.nc3;
  const int64_t grp = sp.nseg > 1 ? udiv(item, sp.nseg) : item;
  const int seg = sp.nseg > 1 ? umod(item, sp.nseg) : 0;
  const int64_t col0 = grp * sp.K;
  const int K = (int)min((int64_t)sp.K, ncol - col0);
  // cells [c0, c1) are this item's in every column; rows hold [lo, lo + n)
  const int c0 = il + seg * sp.seglen, c1 = min(c0 + sp.seglen, iu + 1);
  const bool bottom = c0 == il, top = c1 == iu + 1;
  const int lo = bottom ? 0 : c0 - 3, n = (top ? nc1 : c1 + 3) - lo;
  double* row = x1_rows + (size_t)(threadIdx.x >> 5) * NV * sp.pitch;
  const int64_t span = col0 * nc1 + lo;  // flat offset of the rows' first cell

  // (1) U -> W of the item's cells (ghosts included), two cells a lane at a
  // time so that both cells' loads are in flight
  for (int e0 = lane; e0 < K * n; e0 += 64) {
    double uc[2][5], sc[2][NS > 0 ? NS : 1];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int64_t off = span + min(e0 + 32 * h, K * n - 1);
#pragma unroll
      for (int v = 0; v < 5; ++v) uc[h][v] = b.u[v * sv + off];
#pragma unroll
      for (int m = 0; m < NS; ++m) sc[h][m] = b.s[m * sv + off];
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int e = e0 + 32 * h;
      if (e >= K * n) break;
      const int64_t off = span + e;
      double wc[5];
      cons2prim_cell(uc[h], wc, p.gammad - 1.);
      const int i = lo + (sp.K > 1 ? umod(e, n) : e);
      const bool own = (i >= c0 || bottom) && (i < c1 || top);
#pragma unroll
      for (int v = 0; v < 5; ++v) {
        row[v * sp.pitch + e] = wc[v];
        if (own) b.w[v * sv + off] = wc[v];
      }
#pragma unroll
      for (int m = 0; m < NS; ++m) {
        const double rr = sc[h][m] / uc[h][IDN];
        row[(5 + m) * sp.pitch + e] = rr;
        if (own) b.R[m * sv + off] = rr;
      }
    }
  }
  __syncwarp();

  // (2) isentropic density and pressure in the x1 ghosts, one lane per
  // (column, end, level)
  if (p.grav1 != 0. && (bottom || top)) {
    for (int slot = lane; slot < 2 * ng * K; slot += 32) {
      const int kk = slot / (2 * ng), rest = slot - kk * 2 * ng;
      const int end = rest >= ng, lev = rest - end * ng + 1;
      if (end ? !top : !bottom) continue;
      const int e = kk * n + (end ? iu : il) - lo, dst = end ? e + lev : e - lev;
      double pn, rn;
      isentropic_ghost(p.gammad, -p.grav1 * g.dx1, end, lev, row[IPR * sp.pitch + e],
                       row[IDN * sp.pitch + e], pn, rn);
      row[IPR * sp.pitch + dst] = pn;
      row[IDN * sp.pitch + dst] = rn;
      b.w[IPR * sv + span + dst] = pn;
      b.w[IDN * sv + span + dst] = rn;
    }
    __syncwarp();
  }

  // (3) cells c0-1 .. c1 of every column, 32 a round, the columns end to end:
  // the lane of cell c forms the flux of face c from its own left value and
  // the lower neighbour's right value (the next lower lane, the previous
  // round's last lane for lane 0) and closes cell c - 1.
  const int nn = c1 - c0 + 2;
  const bool need_rg = uses_rho_grav(g, p);
  double Hc[NV], Fc[NV], rc = 0.;  // lane 0: lane 31 of the previous round
#pragma unroll
  for (int v = 0; v < NV; ++v) Hc[v] = Fc[v] = 0.;
  // which of the item's columns are interior ones
  bool inner = lane < K;
  if (inner) {
    const int j = umod(col0 + lane, g.nc2), k = udiv(col0 + lane, g.nc2);
    inner = j >= g.jl && j <= g.ju && k >= g.kl && k <= g.ku;
  }
  const unsigned columns = __ballot_sync(0xffffffffu, inner);
  int kk = lane / nn, t = lane - kk * nn;
  const int total = K * nn;
  for (int s0 = 0; s0 < total; s0 += 32) {
    const bool act = s0 + lane < total && (columns >> kk & 1);
    if (__any_sync(0xffffffffu, act)) {
      const int c = c0 - 1 + t;
      const double* cell = row + (act ? kk * n + c - lo : 2);
      double L[NV], R[NV];
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        double q[5], H;
#pragma unroll
        for (int m = 0; m < 5; ++m) q[m] = cell[v * sp.pitch + m - 2];
        const int typ = v >= 5 ? p.rs_type
                               : (p.r1_shock || v == IDN ? p.r1_type : interp2_of(p.r1_type));
        profile_states<RP>(typ, v >= 5 ? p.rs_scale != 0 : p.r1_scale != 0, v, q, R[v], H);
        const double below = __shfl_sync(0xffffffffu, H, (lane + 31) & 31);
        L[v] = lane == 0 ? Hc[v] : below;
        Hc[v] = below;
      }
      if (p.grav1 != 0.) {
        if (c == il) {
          L[IPR] = R[IPR];
          L[IDN] = R[IDN];
        }
        if (c == iu + 1) {
          R[IPR] = L[IPR];
          R[IDN] = L[IDN];
        }
      }
      double F[NV];
#pragma unroll
      for (int v = 0; v < 5; ++v) F[v] = 0.;
      if (act && t > 0 && !p.disable1) profile_flux<SV>(p.riemann, L, R, IVX, p.gammad, F);
#pragma unroll
      for (int m = 0; m < NS; ++m)
        F[5 + m] = F[IDN] > 0. ? F[IDN] * L[5 + m] : F[IDN] * R[5 + m];
      double d[NV];
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        const double below = __shfl_sync(0xffffffffu, F[v], (lane + 31) & 31);
        d[v] = g.A1 * F[v] - g.A1 * (lane == 0 ? Fc[v] : below);
        Fc[v] = below;
      }
      double rg = 0.;
      if (need_rg) {
        const double below = __shfl_sync(0xffffffffu, R[IPR], (lane + 31) & 31);
        rg = (L[IPR] - (lane == 0 ? rc : below)) / g.dx1;
        rc = below;
      }
      if (act && t > 1) {
        const int64_t off = (col0 + kk) * nc1 + c - 1;
        if (need_rg) b.RG[off] = rg;
#pragma unroll
        for (int v = 0; v < NV; ++v) b.D[v * sv + off] = d[v];
      }
    }
    t += 32;
    while (t >= nn) {
      t -= nn;
      ++kk;
    }
  }
}

}  // namespace snapb
