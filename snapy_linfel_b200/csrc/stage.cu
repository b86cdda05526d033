// stage.cu — one RK stage of the FP64 plain form: the launchers of the sweeps
// (sweep64.cuh), and the kernels beside them:
//
//   k_diff      isotropic viscosity / heat-conduction flux differences;
//   k_finalize  the cells of a 1-D block after its x1 sweep (tendency, RK
//               combination and ghost fill).
//
// Reference path: HydroImpl::forward (src/hydro/hydro_forward.cpp:14-217),
// ReconstructImpl::forward (src/recon/reconstruct.cpp:75-154), the Riemann
// solvers (src/riemann/*_impl.h), divergence (src/coord/coordinate.cpp:352-396),
// gravity (src/forcing/const_gravity.cpp:26-45), hydrostatic revisions
// (src/hydro/hydro.cpp:217-269), ScalarImpl::forward (src/scalar/scalar.cpp:50-132).
#include "sweep64.cuh"

namespace snapb {

// Blocks whose x1 column would not fit this many bytes (W and face fluxes of
// every variable, two face pressures) are refused by check_config.
size_t x1_smem_per_column(const Geo& g, int nvt) {
  return (size_t)(2 * nvt + 2) * g.nc1 * sizeof(double);
}

// U -> W (and scalar mixing ratios) when x1 is inactive
template <int NS>
__global__ void k_c2p_r(Geo g, Phys p, StageBufs b) {
  int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= g.sv) return;
  double uc[5], wc[5];
#pragma unroll
  for (int v = 0; v < 5; ++v) uc[v] = b.u[v * g.sv + t];
  cons2prim_cell(uc, wc, p.gammad - 1.);
#pragma unroll
  for (int v = 0; v < 5; ++v) b.w[v * g.sv + t] = wc[v];
#pragma unroll
  for (int n = 0; n < NS; ++n) b.R[n * g.sv + t] = b.s[n * g.sv + t] / uc[IDN];
}

// ---------------------------------------------------------------------------
// diffusion (src/forcing/diffusion.cpp:152-240), uniform Cartesian
// ---------------------------------------------------------------------------
// Isotropic viscosity and heat conduction of the block's active axes (AXES, a
// bit mask), one thread per cell.  With the axes known at compile time every
// loop unrolls, the velocity gradients and temperatures that the cell's faces
// share are formed once, and the spacings enter as reciprocals.  Bound: loads
// in flight (34 of the neighbourhood) and FP64 issue.  1024 x 128 cells: 20.4
// us with run-time axes and quotients -> 8.6 us.
template <int AXES>
struct DiffCell {
  const double* w;
  int64_t sv, st[3];
  double i1[3], i2[3];  // 1 / dx, 1 / (2 dx)
  static constexpr bool on(int a) { return AXES >> a & 1; }
  __device__ __forceinline__ double slope(int v, int a, int64_t t) const {
    return (w[v * sv + t + st[a]] - w[v * sv + t - st[a]]) * i2[a];
  }
  __device__ __forceinline__ double div(int64_t t) const {
    double d = 0.;
#pragma unroll
    for (int a = 0; a < 3; ++a)
      if (on(a)) d += slope(IVX + a, a, t);
    return d;
  }
  // viscous + conductive flux at the face between t - s_a and t
  __device__ __forceinline__ void face(const Phys& p, int a, int64_t t, double div0, double div1,
                                       double T0, double T1, double cv, double* F) const {
    const int64_t s = st[a];
    const double rho0 = w[IDN * sv + t], rho1 = w[IDN * sv + t - s];
#pragma unroll
    for (int v = 0; v < 5; ++v) F[v] = 0.;
    const double rho_face = 0.5 * (rho0 + rho1);
    if (p.nu > 0.) {
      const double div_face = 0.5 * (div0 + div1);
#pragma unroll
      for (int bb = 0; bb < 3; ++bb) {
        const double v0 = w[(IVX + bb) * sv + t], v1 = w[(IVX + bb) * sv + t - s];
        double stress = (v0 - v1) * i1[a];
        if (bb == a)
          stress = 2. * stress - (2. / 3.) * div_face;
        else if (on(bb))
          stress += 0.5 * (slope(IVX + a, bb, t) + slope(IVX + a, bb, t - s));
        const double m = -p.nu * rho_face * stress;
        F[IVX + bb] = m;
        F[IPR] += 0.5 * (v0 + v1) * m;
      }
    }
    if (p.kappa > 0.) F[IPR] -= p.kappa * (0.5 * (rho0 * cv + rho1 * cv)) * ((T0 - T1) * i1[a]);
  }
};

template <int AXES>
__global__ void __launch_bounds__(128) k_diff(Geo g, Phys p, StageBufs b) {
  const int ni = g.iu - g.il + 1, nj = g.ju - g.jl + 1, nk = g.ku - g.kl + 1;
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (tid >= (int64_t)ni * nj * nk) return;
  const int i = g.il + umod(tid, ni);
  const int j = g.jl + umod(udiv(tid, ni), nj);
  const int k = g.kl + udiv(tid, (int64_t)ni * nj);
  const int64_t t = (int64_t)k * g.s3 + (int64_t)j * g.s2 + i;
  using D = DiffCell<AXES>;
  D c;
  c.w = b.w;
  c.sv = g.sv;
  c.st[0] = 1, c.st[1] = g.s2, c.st[2] = g.s3;
  const double dx[3] = {g.dx1, g.dx2, g.dx3}, A[3] = {g.A1, g.A2, g.A3};
#pragma unroll
  for (int a = 0; a < 3; ++a) c.i1[a] = 1. / dx[a], c.i2[a] = 1. / (2. * dx[a]);
  const double cv = p.rgas / (p.gammad - 1.);
  auto temp = [&](int64_t o) { return b.w[IPR * g.sv + o] / (b.w[IDN * g.sv + o] * p.rgas); };
  const double dc = c.div(t), Tc = temp(t);
  double acc[5] = {0., 0., 0., 0., 0.};
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    if (!D::on(a)) continue;
    const int64_t s = c.st[a];
    double Fm[5], Fp[5];
    c.face(p, a, t, dc, c.div(t - s), Tc, temp(t - s), cv, Fm);
    c.face(p, a, t + s, c.div(t + s), dc, temp(t + s), Tc, cv, Fp);
#pragma unroll
    for (int v = 0; v < 5; ++v) acc[v] += A[a] * Fp[v] - A[a] * Fm[v];
  }
#pragma unroll
  for (int v = 0; v < 5; ++v) b.DD[v * g.sv + t] = acc[v];
}

// The cells of a block whose only active axis is x1, after its sweep (whose
// warps share a column, so they may not update u while others read it): the
// tendency, then du or the RK combination; with fill, the thread of a cell
// also writes the ghost cells that are images of it (a ghost fill without its
// own launch; at most 2 ng images a cell).
template <int NS>
__global__ void k_finalize(Geo g, Phys p, StageBufs b, AxisBC a1, int fill) {
  constexpr int NV = 5 + NS;
  const int ni = g.iu - g.il + 1, nj = g.ju - g.jl + 1, nk = g.ku - g.kl + 1;
  int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (tid >= (int64_t)ni * nj * nk) return;
  int i = g.il + umod(tid, ni);
  int j = g.jl + umod(udiv(tid, ni), nj);
  int k = g.kl + udiv(tid, (int64_t)ni * nj);
  const int64_t row = (int64_t)k * g.s3 + (int64_t)j * g.s2, off = row + i;
  double d[NV], wc[5];
#pragma unroll
  for (int v = 0; v < NV; ++v) d[v] = b.D[v * g.sv + off];
#pragma unroll
  for (int v = 0; v < 5; ++v) wc[v] = b.w[v * g.sv + off];
  const double dt = *b.dt;
  finalize_cell<NS>(g, p, b, off, d, wc, dt, dt / g.vol);
  if (!fill) return;
  for (int m = 0; m < 2 * g.ng; ++m) {
    const int gi = m < g.ng ? m : g.nc1 - 2 * g.ng + m;
    bool flip;
    if (bc_map(a1, gi, flip) != i) continue;
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      const double x = b.u[v * g.sv + off];
      b.u[v * g.sv + row + gi] = v == IVX && flip ? -x : x;
    }
#pragma unroll
    for (int n = 0; n < NS; ++n) b.s[n * g.sv + row + gi] = b.s[n * g.sv + off];
  }
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
// Profile of the sweeps along `axis` (sweep64.cuh): the reconstruction profile
// that the options amount to, 0 when none does.
static int recon_profile64(const Phys& p, int axis) {
  const int typ = axis == 1 ? p.r1_type : p.r23_type;
  const int shock = axis == 1 ? p.r1_shock : p.r23_shock;
  const int scale = axis == 1 ? p.r1_scale : p.r23_scale;
  if (scale || (p.nscalar > 0 && (p.rs_type != typ || p.rs_scale))) return 0;
  if (typ == SNAPB_RECON_PLM) return 3;
  if (typ != SNAPB_RECON_WENO5) return 0;
  return shock ? (p.nscalar ? 0 : 2) : 1;
}

// f(NS, RP, SV) as compile-time constants
template <class F>
static cudaError_t with_profile64(const Phys& p, int axis, F&& f) {
  auto with = [&](auto ns) -> cudaError_t {
    using std::integral_constant;
    constexpr int NS = decltype(ns)::value;
    auto solver = [&](auto rp) -> cudaError_t {
      switch (p.riemann) {
        case SNAPB_RIEMANN_LMARS:
          return f(ns, rp, integral_constant<int, SNAPB_RIEMANN_LMARS>{});
        case SNAPB_RIEMANN_HLLC: return f(ns, rp, integral_constant<int, SNAPB_RIEMANN_HLLC>{});
        default: return f(ns, rp, integral_constant<int, SNAPB_RIEMANN_ROE>{});
      }
    };
    switch (recon_profile64(p, axis)) {
      case 1: return solver(integral_constant<int, 1>{});
      case 2:
        if constexpr (NS == 0) return solver(integral_constant<int, 2>{});
        break;
      case 3: return solver(integral_constant<int, 3>{});
    }
    return f(ns, integral_constant<int, 0>{}, integral_constant<int, -1>{});
  };
  switch (p.nscalar) {
    case 0: return with(std::integral_constant<int, 0>{});
    case 1: return with(std::integral_constant<int, 1>{});
    case 2: return with(std::integral_constant<int, 2>{});
    case 3: return with(std::integral_constant<int, 3>{});
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_finalize(const Geo& g, const Phys& p, const StageBufs& b,
                            const snapb_hydro_config* fill, cudaStream_t st) {
  int64_t n = (int64_t)(g.iu - g.il + 1) * (g.ju - g.jl + 1) * (g.ku - g.kl + 1);
  unsigned grid = (unsigned)((n + 127) / 128);
  const AxisBC a1{g.nc1, g.ng, fill ? fill->bc[0] : 0, fill ? fill->bc[1] : 0};
  const int fl = fill ? 1 : 0;
  switch (p.nscalar) {
    case 0: k_finalize<0><<<grid, 128, 0, st>>>(g, p, b, a1, fl); break;
    case 1: k_finalize<1><<<grid, 128, 0, st>>>(g, p, b, a1, fl); break;
    case 2: k_finalize<2><<<grid, 128, 0, st>>>(g, p, b, a1, fl); break;
    case 3: k_finalize<3><<<grid, 128, 0, st>>>(g, p, b, a1, fl); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t launch_x1(const Geo& g, const Phys& p, const StageBufs& b, cudaStream_t st) {
  const X1Split sp = x1_split(g.nx1, g.ng, (int64_t)g.nc2 * g.nc3, 5 + p.nscalar, sizeof(double),
                              14 * 1024, 148. * 16., false);
  const int64_t items = ((int64_t)g.nc2 * g.nc3 + sp.K - 1) / sp.K * sp.nseg;
  const size_t per = (size_t)sp.pitch * (5 + p.nscalar) * sizeof(double);
  // warps per CTA: four, fewer when the items would not reach every SM
  int wpc = items >= 148 * 4 ? 4 : (items >= 148 * 2 ? 2 : 1);
  while (wpc > 1 && wpc * per > 64 * 1024) wpc /= 2;
  if (per > 200 * 1024) return cudaErrorInvalidConfiguration;
  return with_profile64(p, 1, [&](auto ns, auto rp, auto sv) {
    constexpr int NS = decltype(ns)::value, RP = decltype(rp)::value, SV = decltype(sv)::value;
    raise_smem_limit(k_x1<NS, RP, SV>, 200 * 1024);
    k_x1<NS, RP, SV><<<(unsigned)((items + wpc - 1) / wpc), 32 * wpc, wpc * per, st>>>(g, p, b, sp,
                                                                                     items);
    return cudaGetLastError();
  });
}

cudaError_t launch_c2p_only(const Geo& g, const Phys& p, const StageBufs& b, cudaStream_t st) {
  unsigned grid = (unsigned)((g.sv + 255) / 256);
  switch (p.nscalar) {
    case 0: k_c2p_r<0><<<grid, 256, 0, st>>>(g, p, b); break;
    case 1: k_c2p_r<1><<<grid, 256, 0, st>>>(g, p, b); break;
    case 2: k_c2p_r<2><<<grid, 256, 0, st>>>(g, p, b); break;
    case 3: k_c2p_r<3><<<grid, 256, 0, st>>>(g, p, b); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t launch_march(int axis, const Geo& g, const Phys& p, const StageBufs& b, bool first,
                         bool last, cudaStream_t st) {
  const int ni = g.iu - g.il + 1;
  const int no = axis == 2 ? g.ku - g.kl + 1 : g.ju - g.jl + 1;
  const int n = axis == 2 ? g.nx2 : g.nx3;
  int seglen = 32;
  int64_t threads = (int64_t)ni * no;
  // keep at least ~4 waves of threads on 148 SMs: shorter segments for small grids
  while (seglen > 8 && threads * ((n + seglen - 1) / seglen) < 148LL * 1024 * 2) seglen /= 2;
  const dim3 grid((unsigned)((threads + kMarchThreads - 1) / kMarchThreads),
                  (unsigned)((n + seglen - 1) / seglen));
  return with_profile64(p, axis, [&](auto ns, auto rp, auto sv) {
    constexpr int NS = decltype(ns)::value, RP = decltype(rp)::value, SV = decltype(sv)::value;
    constexpr size_t smem = march_smem_bytes<NS>();
    static_assert(smem <= 48 * 1024, "march ring");
    if (axis == 2)
      k_march<NS, 2, RP, SV><<<grid, kMarchThreads, smem, st>>>(g, p, b, seglen, first, last);
    else
      k_march<NS, 3, RP, SV><<<grid, kMarchThreads, smem, st>>>(g, p, b, seglen, first, last);
    return cudaGetLastError();
  });
}

cudaError_t launch_diffusion(const Geo& g, const Phys& p, const StageBufs& b, cudaStream_t st) {
  const int64_t n = (int64_t)(g.iu - g.il + 1) * (g.ju - g.jl + 1) * (g.ku - g.kl + 1);
  const unsigned grid = (unsigned)((n + 127) / 128);
  switch ((g.nc1 > 1 ? 1 : 0) | (g.nc2 > 1 ? 2 : 0) | (g.nc3 > 1 ? 4 : 0)) {
    case 0: k_diff<0><<<grid, 128, 0, st>>>(g, p, b); break;
    case 1: k_diff<1><<<grid, 128, 0, st>>>(g, p, b); break;
    case 2: k_diff<2><<<grid, 128, 0, st>>>(g, p, b); break;
    case 3: k_diff<3><<<grid, 128, 0, st>>>(g, p, b); break;
    case 4: k_diff<4><<<grid, 128, 0, st>>>(g, p, b); break;
    case 5: k_diff<5><<<grid, 128, 0, st>>>(g, p, b); break;
    case 6: k_diff<6><<<grid, 128, 0, st>>>(g, p, b); break;
    case 7: k_diff<7><<<grid, 128, 0, st>>>(g, p, b); break;
  }
  return cudaGetLastError();
}

}  // namespace snapb
