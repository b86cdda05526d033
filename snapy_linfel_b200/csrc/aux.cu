// aux.cu — element-wise and reduction kernels around the sweeps: EOS,
// boundary fills, CFL limit, positivity check, and the operator-level
// reconstruct / Riemann entry points (one module call each).
#include <algorithm>
#include <cfloat>
#include <cstring>

#include "kernels.cuh"

namespace snapb {

// ---------------------------------------------------------------------------
// EOS (src/eos/ideal_gas.cpp:67-109)
// ---------------------------------------------------------------------------
__global__ void k_cons2prim(int64_t n, int64_t sv, double gm1, const double* u, double* w) {
  int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  double uc[5], wc[5];
#pragma unroll
  for (int v = 0; v < 5; ++v) uc[v] = u[v * sv + t];
  cons2prim_cell(uc, wc, gm1);
#pragma unroll
  for (int v = 0; v < 5; ++v) w[v * sv + t] = wc[v];
}

__global__ void k_prim2cons(int64_t n, int64_t sv, double gm1, const double* w, double* u) {
  int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  double rho = w[IDN * sv + t];
  double v1 = w[IVX * sv + t], v2 = w[IVY * sv + t], v3 = w[IVZ * sv + t];
  double m1 = v1 * rho, m2 = v2 * rho, m3 = v3 * rho;
  u[IDN * sv + t] = rho;
  u[IVX * sv + t] = m1;
  u[IVY * sv + t] = m2;
  u[IVZ * sv + t] = m3;
  double ke = 0.5 * (v1 * m1 + v2 * m2 + v3 * m3);
  u[IPR * sv + t] = w[IPR * sv + t] / gm1 + ke;
}

cudaError_t launch_cons2prim(const Geo& g, const Phys& p, const double* u, double* w,
                             cudaStream_t st) {
  k_cons2prim<<<(unsigned)((g.sv + 255) / 256), 256, 0, st>>>(g.sv, g.sv, p.gammad - 1., u, w);
  return cudaGetLastError();
}

cudaError_t launch_prim2cons(const Geo& g, const Phys& p, const double* w, double* u,
                             cudaStream_t st) {
  k_prim2cons<<<(unsigned)((g.sv + 255) / 256), 256, 0, st>>>(g.sv, g.sv, p.gammad - 1., w, u);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Boundary fills (src/bc/bc_func.cpp:7-63), applied x1-inner, x1-outer, ...,
// x3-outer (src/mesh/meshblock.cpp:717-730).  Each fill copies from cells
// that are interior along its own axis, so the sequence composes per axis:
// the final value of a cell is var[m3(k)][m2(j)][m1(i)] times the sign flips
// of the reflecting axes it crossed.  One thread per cell of the ghost shell
// (bc_shell_cell enumerates exactly the ghost cells).
// ---------------------------------------------------------------------------
__global__ void k_bc(Geo g, AxisBC a1, AxisBC a2, AxisBC a3, double* var, int nv,
                     int flip_normals) {
  const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= bc_shell_slots(g)) return;
  const int nc1 = g.nc1, nc2 = g.nc2;
  const int64_t sv = g.sv;
  int i, j, k;
  const int64_t t = bc_shell_cell(g, s, i, j, k);
  bool f1, f2, f3;
  int si = bc_map(a1, i, f1), sj = bc_map(a2, j, f2), sk = bc_map(a3, k, f3);
  if (si == i && sj == j && sk == k) return;  // interior (or identity-mapped) cell
  int64_t src = ((int64_t)sk * nc2 + sj) * nc1 + si;
  // loads of a group of variables before its stores (a thread's source cell
  // is never its target; the compiler cannot see that the stores miss it)
  constexpr int kGroup = 8;
  for (int v0 = 0; v0 < nv; v0 += kGroup) {
    double xs[kGroup];
#pragma unroll
    for (int q = 0; q < kGroup; ++q)
      if (v0 + q < nv) xs[q] = var[(v0 + q) * sv + src];
#pragma unroll
    for (int q = 0; q < kGroup; ++q) {
      const int v = v0 + q;
      if (v >= nv) break;
      double x = xs[q];
      if (flip_normals) {
        if ((v == IVX && f1) || (v == IVY && f2) || (v == IVZ && f3)) x = -x;
      }
      var[v * sv + t] = x;
    }
  }
}

cudaError_t launch_bc(const Geo& g, const snapb_hydro_config& c, double* var, int nv, int kind,
                      cudaStream_t st) {
  AxisBC a1{g.nc1, g.ng, c.bc[0], c.bc[1]};
  AxisBC a2{g.nc2, g.ng, c.bc[2], c.bc[3]};
  AxisBC a3{g.nc3, g.ng, c.bc[4], c.bc[5]};
  int flip = (kind == SNAPB_CONSERVED || kind == SNAPB_PRIMITIVE) ? 1 : 0;
  const int64_t n = bc_shell_slots_host(g);
  if (n == 0) return cudaSuccess;
  k_bc<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(g, a1, a2, a3, var, nv, flip);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// CFL limit (src/hydro/hydro.cpp:118-180).  A thread keeps the largest signal
// speed per axis and divides once (cfl32_speeds, kernels.cuh: the quotient is
// monotone, so the minimum is the same to the bit).  Bound: HBM (70 % of the
// copy rate); 384 x 384 x 192: 386 us with a division per cell and axis -> 246.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_cfl(Geo g, double gammad, CflUse use, const double* w,
                                             unsigned long long* slots, double* dt_out) {
  double a1 = 0., a2 = 0., a3 = 0.;
  cfl_cells(g, [&](int64_t o, int) {
    const double rho = w[IDN * g.sv + o], pr = w[IPR * g.sv + o];
    const double cs = sqrt(gammad * pr / rho);
    if (use.use1) a1 = fmax(a1, fabs(w[IVX * g.sv + o]) + cs);
    if (use.use2) a2 = fmax(a2, fabs(w[IVY * g.sv + o]) + cs);
    if (use.use3) a3 = fmax(a3, fabs(w[IVZ * g.sv + o]) + cs);
  });
  cfl_finish(use, fmin(DBL_MAX, g.dx1 / a1), fmin(DBL_MAX, g.dx2 / a2), fmin(DBL_MAX, g.dx3 / a3),
             slots, dt_out);
}

CflUse cfl_use(const Geo& g, const Phys& p) {
  const int scheme = p.implicit_scheme;
  CflUse u{g.nc1 > 1, g.nc2 > 1, g.nc3 > 1, -1.};
  if (scheme != 0) {
    u.use1 = u.use1 && (!(scheme & 1) || (g.nc3 == 1 && g.nc2 == 1));
    u.use2 = u.use2 && !((scheme >> 1) & 1);
    u.use3 = u.use3 && !((scheme >> 2) & 1);
  }
  const double coeff = fmax(p.nu, p.kappa);
  if (coeff > 0.) {
    int ndim = 0;
    double dxm = DBL_MAX;
    if (g.nc1 > 1) ++ndim, dxm = fmin(dxm, g.dx1);
    if (g.nc2 > 1) ++ndim, dxm = fmin(dxm, g.dx2);
    if (g.nc3 > 1) ++ndim, dxm = fmin(dxm, g.dx3);
    if (ndim > 0) u.dt_diff = dxm * dxm / (2. * ndim * coeff);
  }
  return u;
}

cudaError_t launch_cfl(const Geo& g, const Phys& p, const double* w, double* slots,
                       double* dt_out, cudaStream_t st) {
  auto* sl = reinterpret_cast<unsigned long long*>(slots);
  const int blocks = cfl_blocks(g);
  if (blocks > 1) {
    const cudaError_t e = cudaMemsetAsync(sl, 0xff, 4 * sizeof(*sl), st);
    if (e != cudaSuccess) return e;
  }
  k_cfl<<<blocks, 256, 0, st>>>(g, p.gammad, cfl_use(g, p), w, sl, dt_out);
  return cudaGetLastError();
}

__global__ void k_scale_dt(const double* in, double f, double* out) { *out = f * *in; }

cudaError_t launch_scale_dt(const double* dt_in, double cfl, int redo, double* dt_out,
                            cudaStream_t st) {
  // pow(2, -redo) * cfl * dt  (src/mesh/meshblock.cpp:527)
  double f = ldexp(1.0, -redo) * cfl;
  k_scale_dt<<<1, 1, 0, st>>>(dt_in, f, dt_out);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Positivity check (src/mesh/meshblock.cpp:974-1016):
// flags[0] density <= 0, flags[1] total energy <= 0, flags[2] pressure <= 0
// ---------------------------------------------------------------------------
__global__ void k_check(Geo g, double gm1, const double* u, int* flags) {
  const int ni = g.iu - g.il + 1, nj = g.ju - g.jl + 1, nk = g.ku - g.kl + 1;
  const int64_t n = (int64_t)ni * nj * nk;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n;
       t += (int64_t)gridDim.x * blockDim.x) {
    int i = g.il + umod(t, ni);
    int j = g.jl + umod(udiv(t, ni), nj);
    int k = g.kl + udiv(t, (int64_t)ni * nj);
    int64_t o = (int64_t)k * g.s3 + (int64_t)j * g.s2 + i;
    double uc[5], wc[5];
#pragma unroll
    for (int v = 0; v < 5; ++v) uc[v] = u[v * g.sv + o];
    if (!(uc[IDN] > 0.)) atomicOr(&flags[0], 1);
    if (!(uc[IPR] > 0.)) atomicOr(&flags[1], 1);
    cons2prim_cell(uc, wc, gm1);
    if (!(wc[IPR] > 0.)) atomicOr(&flags[2], 1);
  }
}

__global__ void k_zero_int(int* p, int n) {
  if ((int)threadIdx.x < n) p[threadIdx.x] = 0;
}

cudaError_t launch_check_positive(const Geo& g, const Phys& p, const double* u, int* flags,
                                  cudaStream_t st) {
  k_zero_int<<<1, 32, 0, st>>>(flags, 3);
  int64_t n = (int64_t)(g.iu - g.il + 1) * (g.ju - g.jl + 1) * (g.ku - g.kl + 1);
  int blocks = (int)std::min<int64_t>((n + 255) / 256, 148 * 8);
  k_check<<<blocks, 256, 0, st>>>(g, p.gammad - 1., u, flags);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Operator level: ReconstructImpl::forward and RiemannSolverImpl::forward on
// whole arrays, with the reference's edge replication, for parity checks of
// the individual modules.
// ---------------------------------------------------------------------------
__device__ __forceinline__ int stencil_radius(int type) {
  return type == SNAPB_RECON_DC ? 0
         : (type == SNAPB_RECON_WENO5 || type == SNAPB_RECON_CP5) ? 2
                                                                   : 1;
}

__global__ void k_reconstruct(Geo g, Phys p, int dim, int group, const double* w, int nv,
                              double* wlr) {
  int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= g.sv * nv) return;
  int v = udiv(t, g.sv);
  int64_t cell = t - (int64_t)v * g.sv;
  int i = umod(cell, g.nc1);
  int j = umod(udiv(cell, g.nc1), g.nc2);
  int k = udiv(cell, (int64_t)g.nc1 * g.nc2);
  int n, pos;
  int64_t st;
  if (dim == 3) n = g.nc1, pos = i, st = 1;
  else if (dim == 2) n = g.nc2, pos = j, st = g.s2;
  else n = g.nc3, pos = k, st = g.s3;
  int type, shock, scale;
  if (group == 1) type = p.rs_type, shock = 1, scale = p.rs_scale;
  else if (dim == 3) type = p.r1_type, shock = p.r1_shock, scale = p.r1_scale;
  else type = p.r23_type, shock = p.r23_shock, scale = p.r23_scale;
  if (group == 0 && !shock && v >= IVX && v <= IPR) type = interp2_of(type);
  int r = stencil_radius(type);
  int il = r + 1, iu = n - (r + 1);
  const double* line = w + (int64_t)v * g.sv + cell - (int64_t)pos * st;
  auto win = [&](int f, double* q) {  // six cells around face f, clamped
#pragma unroll
    for (int m = 0; m < 6; ++m) q[m] = line[(int64_t)min(max(f - 3 + m, 0), n - 1) * st];
  };
  double q[6], wl, wr;
  // wlr[IRT] slot pos: left face of cell o, o clamped to [il, iu]
  int o = min(max(pos, il), iu);
  if (type == SNAPB_RECON_DC) o = max(pos, il);
  win(o, q);
  face_states(type, scale != 0, q, wl, wr);
  double vr = wr;
  // wlr[ILT] slot pos: right face of cell o-1, o clamped to [il, iu] (dc: to n-1)
  o = min(max(pos, il), iu);
  if (type == SNAPB_RECON_DC) o = max(pos, il);
  win(o, q);
  face_states(type, scale != 0, q, wl, wr);
  double vl = wl;
  if (group == 1) {
    vl = vl < 0. ? 0. : vl;
    vr = vr < 0. ? 0. : vr;
  }
  wlr[t] = vl;                    // ILT
  wlr[(int64_t)nv * g.sv + t] = vr;  // IRT
}

cudaError_t launch_reconstruct(const Geo& g, const Phys& p, int dim, int group, const double* w,
                               int nv, double* wlr, cudaStream_t st) {
  int64_t n = g.sv * nv;
  k_reconstruct<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(g, p, dim, group, w, nv, wlr);
  return cudaGetLastError();
}

__global__ void k_riemann(int64_t sv, int solver, int ivx, double gamma, const double* wl,
                          const double* wr, int nv, double* flx, double* fp, const double* vel) {
  int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= sv) return;
  if (solver == SNAPB_RIEMANN_UPWIND) {
    double ve = vel[t];
    for (int v = 0; v < nv; ++v)
      flx[v * sv + t] = ve > 0. ? ve * wl[v * sv + t] : ve * wr[v * sv + t];
    return;
  }
  double L[5], R[5], F[5], P;
#pragma unroll
  for (int v = 0; v < 5; ++v) {
    L[v] = wl[v * sv + t];
    R[v] = wr[v * sv + t];
  }
  riemann_flux(solver, L, R, ivx, gamma, F, &P);
#pragma unroll
  for (int v = 0; v < 5; ++v) flx[v * sv + t] = F[v];
  if (fp) fp[t] = P;
}

cudaError_t launch_riemann(const Geo& g, const Phys& p, int solver, int dim, const double* wl,
                           const double* wr, int nv, double* flx, double* fp, const double* vel,
                           cudaStream_t st) {
  int ivx = IPR - dim;
  k_riemann<<<(unsigned)((g.sv + 255) / 256), 256, 0, st>>>(g.sv, solver, ivx, p.gammad, wl, wr,
                                                           nv, flx, fp, vel);
  return cudaGetLastError();
}

}  // namespace snapb
