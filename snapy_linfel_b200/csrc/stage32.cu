// stage32.cu — one RK stage in the FP32 perturbation form.
//
// State: u' = u - (rho_bar, 0, 0, 0, p_bar/(gamma-1)) in FP32 over an FP64
// reference profile rho_bar(x1), p_bar(x1) (x1 = vertical).  The sweeps are
// the same fused kernels as the FP64 form (stage.cu) in FP32 arithmetic, with
// three places where FP64 stays:
//   * the reference tables (k_ref32): x1 face reference pressures pf, the
//     offsets of each side's reconstructed reference pressure from pf, and
//     the residual of the reference x1 momentum balance
//     rbar_i = -(A1 pf_{i+1} - A1 pf_i)/V + rho_bar_i g1, formed in FP64 and
//     stored after the cancellation;
//   * the isentropic x1 ghost revision (pow of full values) in FP64, in the
//     x1 sweep;
//   * the implicit column solve (vic.cu, FP64 elimination on full states).
// The momentum fluxes carry the pressure as p' = p - pf (pert.cuh), so the
// large hydrostatic pressure never enters an FP32 difference.
#include <algorithm>
#include <type_traits>

#include "kernels.cuh"
#include "pert.cuh"

namespace snapb {

// ---------------------------------------------------------------------------
// reference tables
// ---------------------------------------------------------------------------
__global__ void k_ref32(Geo g, Phys p, const double* rb_in, const double* pb_in, double* rbw,
                        double* pbw, StageBufs32 b) {
  const int nc1 = g.nc1;
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t <= nc1) {
    // reference pressure at face t from each side, with the x1 pressure
    // interpolation (linear: cp5 / cp3 / dc)
    int typ = (p.r1_shock) ? p.r1_type : interp2_of(p.r1_type);
    double q[6];
    for (int m = 0; m < 6; ++m) {
      int c = min(max(t - 3 + m, 0), nc1 - 1);
      q[m] = pb_in ? pb_in[c] : 0.;
    }
    double pl, pr;
    face_states<double>(typ, false, q, pl, pr);
    if (typ != SNAPB_RECON_CP5 && typ != SNAPB_RECON_CP3 && typ != SNAPB_RECON_DC) {
      pl = pr = q[2];  // non-linear pressure interpolation: only with a zero reference
    }
    double pfv = 0.5 * (pl + pr);
    b.pf[t] = pfv;
    b.offL[t] = (float)(pl - pfv);
    b.offR[t] = (float)(pr - pfv);
  }
  if (t < nc1) {
    double r = rb_in ? rb_in[t] : 0.;
    double pr = pb_in ? pb_in[t] : 0.;
    rbw[t] = r;
    pbw[t] = pr;
    b.rbf[t] = (float)r;
    b.pbf[t] = (float)pr;
  }
}

// second pass: the x1 momentum residual needs pf on both faces of a cell
__global__ void k_ref32_residual(Geo g, Phys p, StageBufs32 b) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= g.nc1) return;
  double res = 0.;
  if (i + 1 <= g.nc1) res = -(g.A1 * b.pf[i + 1] - g.A1 * b.pf[i]) / g.vol;
  res += b.rb[i] * p.grav1;
  b.rbar[i] = (float)res;
}

// ---------------------------------------------------------------------------
// finalize: du' = -dt div'/V + gravity (with the FP64 reference residual),
// then RK on u' or du for the implicit solve
// ---------------------------------------------------------------------------
// What the finish of a cell needs of the descriptors, converted once per CTA
// and member into shared memory (held in registers it made the marches spill:
// 0.75 -> 1.2 ms on the 48 members; read from the descriptors, every cell
// took an FP64 division and nine conversions).
struct Finish32 {
  float dt, ivol, g1, g2, g3, w0, w1, w2;
  bool balance, write_du, stage0;
  const float *rbf, *rbar;
  float *D, *u, *u0, *s, *s0, *r;
  int sv;
  __device__ __forceinline__ void set(const Geo& g, const Phys& p, const StageBufs32& b) {
    dt = (float)*b.dt, ivol = (float)(1.0 / g.vol);
    g1 = (float)p.grav1, g2 = (float)p.grav2, g3 = (float)p.grav3;
    w0 = (float)b.wgt0, w1 = (float)b.wgt1, w2 = (float)b.wgt2;
    balance = g.nc1 > 1, write_du = b.write_du != 0, stage0 = b.stage == 0;
    rbf = b.rbf, rbar = b.rbar, D = b.D, u = b.u, u0 = b.u0, s = b.s, s0 = b.s0, r = b.r;
    sv = (int)g.sv;
  }
};

// A CTA's shared descriptors: the block's (or the current member's), the
// physics and the finish.
struct Shared32 {
  Member32 m;
  Phys p;
  Finish32 fin;
};
// (one variable for the kernels and the functions they call, so that these know its
// address: through a pointer every field was a generic load)
__device__ __forceinline__ Shared32& shared32() {
  __shared__ Shared32 s;
  return s;
}

// UPDATE: the RK combination, else du for the implicit solve
template <int NS, bool UPDATE>
__device__ __forceinline__ void finalize32(const Finish32& c, int off, int xi, const float* d,
                                           const float* wc) {
  const int sv = c.sv;
  const float dt = c.dt;
  float rho = c.rbf[xi] + wc[IDN];
  float du[5];
#pragma unroll
  for (int v = 0; v < 5; ++v) du[v] = -dt * (d[v] * c.ivol);
  if (c.balance) du[IVX] += dt * c.rbar[xi];  // reference pressure gradient + rho_bar g1
  if (c.g1 != 0.f) {
    du[IVX] += dt * wc[IDN] * c.g1;
    du[IPR] += dt * rho * wc[IVX] * c.g1;
  }
  if (c.g2 != 0.f) {
    du[IVY] += dt * rho * c.g2;
    du[IPR] += dt * rho * wc[IVY] * c.g2;
  }
  if (c.g3 != 0.f) {
    du[IVZ] += dt * rho * c.g3;
    du[IPR] += dt * rho * wc[IVZ] * c.g3;
  }
  float ds[NS > 0 ? NS : 1];
#pragma unroll
  for (int n = 0; n < NS; ++n) ds[n] = -dt * (d[5 + n] * c.ivol);
  if constexpr (!UPDATE) {
#pragma unroll
    for (int v = 0; v < 5; ++v) c.D[v * sv + off] = du[v];
#pragma unroll
    for (int n = 0; n < NS; ++n) c.D[(5 + n) * sv + off] = ds[n];
    return;
  }
  // All loads before the first store: the compiler cannot see that the stores miss
  // them and would wait for one load per variable.  x3 of an explicit 96^3 block,
  // Roe 64 -> 37 us, with two tracers 119 -> 57; of 6 members, HLLC 342 -> 149 us.
  float *u = c.u, *u0 = c.u0, *sc = c.s, *sc0 = c.s0, *mix = c.r;
  const float w0 = c.w0, w1 = c.w1, w2 = c.w2, rref = c.rbf[xi];
  const bool stage0 = c.stage0;
  float uo[5], u0v[5], so[NS > 0 ? NS : 1], s0v[NS > 0 ? NS : 1];
#pragma unroll
  for (int v = 0; v < 5; ++v) {
    uo[v] = u[v * sv + off];
    u0v[v] = stage0 ? uo[v] : u0[v * sv + off];
  }
#pragma unroll
  for (int n = 0; n < NS; ++n) {
    so[n] = sc[n * sv + off];
    s0v[n] = stage0 ? so[n] : sc0[n * sv + off];
  }
  float unew_rho = 0.f;
#pragma unroll
  for (int v = 0; v < 5; ++v) {
    const int o = v * sv + off;
    if (stage0) u0[o] = uo[v];
    const float un = fmaf(w2, du[v], fmaf(w1, uo[v], w0 * u0v[v]));
    u[o] = un;
    if (v == IDN) unew_rho = rref + un;
  }
#pragma unroll
  for (int n = 0; n < NS; ++n) {
    const int o = n * sv + off;
    if (stage0) sc0[o] = so[n];
    const float sn = fmaf(w2, ds[n], fmaf(w1, so[n], w0 * s0v[n]));
    sc[o] = sn;
    if (mix) mix[o] = sn / unew_rho;
  }
}

// U' -> W' of one cell at x1 index xi (p' = (gamma-1)(E' - KE): no
// reference-sized cancellation)
__device__ __forceinline__ void cons2prim_pert(const float* u, float* w, float rbar, float gm1) {
  float rho = rbar + u[IDN];
  float ir = fdiv(1.f, rho);
  w[IDN] = u[IDN];
  w[IVX] = u[IVX] * ir;
  w[IVY] = u[IVY] * ir;
  w[IVZ] = u[IVZ] * ir;
  float ke = 0.5f * (w[IVX] * u[IVX] + w[IVY] * u[IVY] + w[IVZ] * u[IVZ]);
  w[IPR] = gm1 * (u[IPR] - ke);
}

// Blocks whose x1 column would not fit this many bytes (every variable twice,
// a density row) are refused by the FP32 entry points.
size_t x1_smem32_per_column(const Geo& g, int nvt) {
  return (size_t)(2 * nvt + 1) * g.nc1 * sizeof(float);
}

// ---------------------------------------------------------------------------
// x1 sweep
// ---------------------------------------------------------------------------
constexpr size_t kX1RowBytes32 = 7 * 1024;  // rows of a warp: shared memory for 24 of them per SM
// warps that the split's rule takes to be resident (the registers hold 20 per SM)
constexpr double kX1Resident32 = 148. * 24.;

// One item (X1Split, cells.cuh) by one warp, with its rows (full density
// rho_bar + rho', v', p', mixing ratios) in shared memory:
//   (1) U' -> W' of the item's cells, W' and the mixing ratios stored;
//   (2) density and pressure of the x1 ghosts from the isentropic revision of
//       the edge cells, on full values in FP64, one lane per (column, end,
//       level);
//   (3) the cells in rounds of 32 lanes, the item's columns end to end: a lane
//       forms the flux of its cell's lower face from its own left value and
//       the next lower lane's right value, and closes the cell below.
// Not inlined: the one-block and the batched kernel run this very code, so a
// member of an ensemble rounds as it does alone.
//
// Bound: instruction issue (72 % active at 20 warps per SM) and the latency of
// the conversion's loads.  Per stage, against a tile of columns per CTA (bulk
// copies into shared memory, barriers, the revision in its own kernel):
// 384 x 384 x 192, Roe, two tracers 1.29 -> 1.25 ms, 512 x 256 21.0 -> 10.7 us,
// 48 members of 64 and 128 layers 1.57 -> 1.22 ms; a 1-D block of 1024 cells, whose
// column is not cut, 90 -> 57 us.
template <int NS, int FP>
__device__ __noinline__ void x1_32_item(int64_t item, int last) {
  constexpr int NV = 5 + NS;
  extern __shared__ float x1_rows32[];
  float* row = x1_rows32;
  const Shared32& sh = shared32();
  const Geo& g = sh.m.g;
  const StageBufs32& b = sh.m.b;
  const Phys& p = sh.p;
  const X1Split sp = sh.m.x1;
  const int lane = threadIdx.x & 31;
  const int nc1 = g.nc1, il = g.il, iu = g.iu, ng = g.ng, pitch = sp.pitch;
  const int sv = (int)g.sv;  // (element indices stay below 2^31: check_config)
  const int ncol = g.nc2 * g.nc3;
  const int grp = sp.nseg > 1 ? udiv(item, sp.nseg) : (int)item;
  const int seg = sp.nseg > 1 ? umod(item, sp.nseg) : 0;
  const int col0 = grp * sp.K, K = min(sp.K, ncol - col0);
  // cells [c0, c1) are this item's in every column; rows hold [lo, lo + n)
  const int c0 = il + seg * sp.seglen, c1 = min(c0 + sp.seglen, iu + 1);
  const bool bottom = c0 == il, top = c1 == iu + 1;
  const int lo = bottom ? 0 : c0 - 3, n = (top ? nc1 : c1 + 3) - lo;
  const int span = col0 * nc1 + lo;
  const float gm1 = (float)(p.gammad - 1.);
  const bool revise = p.grav1 != 0.;
  const float *u = b.u, *s = b.s, *rbf = b.rbf, *offL = b.offL, *offR = b.offR;
  const double* pf = b.pf;
  float *w = b.w, *rr = b.R, *D = b.D;
  // which of the item's columns are interior ones
  bool inner = lane < K;
  if (inner) {
    const int j = umod(col0 + lane, g.nc2), k = udiv(col0 + lane, g.nc2);
    inner = j >= g.jl && j <= g.ju && k >= g.kl && k <= g.ku;
  }
  const unsigned columns = __ballot_sync(0xffffffffu, inner);
  // two cells a lane at a time, so that both cells' loads are in flight
  for (int e0 = lane; e0 < K * n; e0 += 64) {
    float uc[2][5], sc[2][NS > 0 ? NS : 1], rb[2];
    int xi[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int e = min(e0 + 32 * h, K * n - 1), off = span + e;
      xi[h] = lo + (sp.K > 1 ? umod(e, n) : e);
#pragma unroll
      for (int v = 0; v < 5; ++v) uc[h][v] = u[v * sv + off];
#pragma unroll
      for (int m = 0; m < NS; ++m) sc[h][m] = s[m * sv + off];
      rb[h] = rbf[xi[h]];
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int e = e0 + 32 * h, off = span + e;
      if (e >= K * n) break;
      float wc[5];
      cons2prim_pert(uc[h], wc, rb[h], gm1);
      const bool own = (xi[h] >= c0 || bottom) && (xi[h] < c1 || top);
      row[IDN * pitch + e] = rb[h] + wc[IDN];
#pragma unroll
      for (int v = 1; v < 5; ++v) row[v * pitch + e] = wc[v];
      if (own)
#pragma unroll
        for (int v = 0; v < 5; ++v) w[v * sv + off] = wc[v];
#pragma unroll
      for (int m = 0; m < NS; ++m) {
        const float mix = fdiv(sc[h][m], rb[h] + uc[h][IDN]);
        row[(5 + m) * pitch + e] = mix;
        if (own) rr[m * sv + off] = mix;
      }
    }
  }
  __syncwarp();
  if (revise && (bottom || top)) {
    for (int slot = lane; slot < 2 * ng * K; slot += 32) {
      const int kk = slot / (2 * ng), rest = slot - kk * 2 * ng;
      const int end = rest >= ng, lev = rest - end * ng + 1;
      if (end ? !top : !bottom) continue;
      const int edge = end ? iu : il, e = kk * n + edge - lo, dst = end ? e + lev : e - lev;
      const int cell = end ? edge + lev : edge - lev;
      double pn, rn;
      isentropic_ghost(p.gammad, -p.grav1 * g.dx1, end, lev,
                       b.pb[edge] + (double)row[IPR * pitch + e],
                       b.rb[edge] + (double)u[IDN * sv + span + e], pn, rn);
      const float wp = (float)(pn - b.pb[cell]), wr = (float)(rn - b.rb[cell]);
      row[IPR * pitch + dst] = wp;
      row[IDN * pitch + dst] = rbf[cell] + wr;
      w[IPR * sv + span + dst] = wp;
      w[IDN * sv + span + dst] = wr;
    }
    __syncwarp();
  }
  const int nn = c1 - c0 + 2, total = K * nn;
  const float gamma = (float)p.gammad, A1 = (float)g.A1;
  const bool flux = !p.disable1;
  const int ptype = p.r1_shock ? p.r1_type : interp2_of(p.r1_type);
  float Hc[NV], Fc[NV];  // lane 0: lane 31 of the previous round
#pragma unroll
  for (int v = 0; v < NV; ++v) Hc[v] = Fc[v] = 0.f;
  int kk = lane / nn, t = lane - kk * nn;
  for (int s0 = 0; s0 < total; s0 += 32) {
    const bool act = s0 + lane < total && (columns >> kk & 1);
    if (__any_sync(0xffffffffu, act)) {
      const int c = c0 - 1 + t;
      const float* cell = row + (act ? kk * n + c - lo : 2);
      float L[NV], R[NV];
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        float q[5], H;
#pragma unroll
        for (int m = 0; m < 5; ++m) q[m] = cell[v * pitch + m - 2];
        const int typ = v >= 5 ? p.rs_type : (v == IDN ? p.r1_type : ptype);
        sweep_cell_states<FP>(typ, v >= 5 ? p.rs_scale != 0 : p.r1_scale != 0, v, q, R[v], H);
        const float below = __shfl_sync(0xffffffffu, H, (lane + 31) & 31);
        L[v] = lane == 0 ? Hc[v] : below;
        Hc[v] = below;
      }
      const int f = act ? c : il;
      float pl = L[IPR] + offL[f], pr = R[IPR] + offR[f];
      if (revise) {
        if (c == il) {
          pl = pr;
          L[IDN] = R[IDN];
        }
        if (c == iu + 1) {
          pr = pl;
          R[IDN] = L[IDN];
        }
      }
      const float pfv = (float)pf[f];
      L[IPR] = pfv + pl;
      R[IPR] = pfv + pr;
      float F[NV];
#pragma unroll
      for (int v = 0; v < 5; ++v) F[v] = 0.f;
      if (act && t > 0 && flux)
        sweep_riemann<FP>(p.riemann, L, R, pl, pr, pfv, IVX, gamma, F);
#pragma unroll
      for (int m = 0; m < NS; ++m)
        F[5 + m] = F[IDN] > 0.f ? F[IDN] * L[5 + m] : F[IDN] * R[5 + m];
      float d[NV];
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        const float below = __shfl_sync(0xffffffffu, F[v], (lane + 31) & 31);
        d[v] = A1 * F[v] - A1 * (lane == 0 ? Fc[v] : below);
        Fc[v] = below;
      }
      if (act && t > 1) {
        const int off = (col0 + kk) * nc1 + c - 1;
        if (last) {
          float wc[5];
          wc[IDN] = w[IDN * sv + off];
#pragma unroll
          for (int v = 1; v < 5; ++v) wc[v] = cell[v * pitch - 1];
          if (sh.fin.write_du)
            finalize32<NS, false>(sh.fin, off, c - 1, d, wc);
          else
            finalize32<NS, true>(sh.fin, off, c - 1, d, wc);
        } else {
#pragma unroll
          for (int v = 0; v < NV; ++v) D[v * sv + off] = d[v];
        }
      }
    }
    t += 32;
    while (t >= nn) {
      t -= nn;
      ++kk;
    }
  }
}

// one item per CTA of one warp; the block's descriptor goes to shared memory,
// where the batched form has its members'
template <int NS, int FP>
__global__ void __launch_bounds__(32, 20) k_x1_32(Geo g, Phys p, StageBufs32 b, X1Split sp,
                                                  int last) {
  Shared32& sh = shared32();
  if (threadIdx.x == 0) {
    sh.m.g = g;
    sh.m.b = b;
    sh.m.x1 = sp;
    sh.p = p;
    sh.fin.set(g, p, b);
  }
  __syncwarp();
  x1_32_item<NS, FP>(blockIdx.x, last);
}

// ---------------------------------------------------------------------------
// x2 / x3 marching sweeps (reference constant along the sweep)
// ---------------------------------------------------------------------------
// What a march does with a cell's sums: keeps them for the next sweep, forms du for
// the implicit solve, or updates the cell.
enum { kKeep = 0, kTendency = 1, kUpdate = 2 };
inline int march_end(const Phys& p, bool last) {
  return !last ? kKeep : (p.implicit_scheme ? kTendency : kUpdate);
}
// Resident CTAs per SM: the register budget that holds the window of 5 + NS
// variables, and for kUpdate also the cell's old state, without spilling them.
// (With the end read at run time every march held what the update needs: x2 of 6
// members, LMARS, 68 -> 84 us.)
template <int NS, int FP, int END>
constexpr int kMarchCtas32 = END == kUpdate ? (NS >= 2 ? 3 : (FP == 1 && NS == 0 ? 5 : 4))
                                            : (NS >= 2 ? 4 : (FP == 1 ? (NS == 0 ? 6 : 5) : 4));

// One thread's work: line tid (x1 cell x other horizontal index) and face
// segment seg of the sweep axis.  Cell centred (cells.cuh); per stage x2 and x3
// 0.81 + 0.85 -> 0.71 + 0.74 ms on the 48 members, 0.80 + 0.84 -> 0.79 + 0.83 on
// 384 x 384 x 192 with two tracers.  Bound by instruction issue (70 to 74 %
// active).  Not inlined, as x1_32_item: the one-block and the batched kernel round
// alike (inlined into the one-block kernel it rounded Roe fluxes with one tracer
// otherwise), and the descriptor's fields are read from shared memory when they are
// needed instead of being held in registers (copied into registers the batched
// kernel spilled).
template <int NS, int AX, int FP, int END>
__device__ __noinline__ void march32_line(int first, int tid, int seg) {
  const Shared32& sh = shared32();
  const Geo& g = sh.m.g;
  const StageBufs32& b = sh.m.b;
  const Phys& p = sh.p;
  const int seglen = AX == 2 ? sh.m.seglen2 : sh.m.seglen3;
  constexpr int NV = 5 + NS;
  const int ni = g.iu - g.il + 1;
  int lo, hi, olo, ohi;
  int64_t st, ost;
  if (AX == 2) {
    lo = g.jl, hi = g.ju, st = g.s2, olo = g.kl, ohi = g.ku, ost = g.s3;
  } else {
    lo = g.kl, hi = g.ku, st = g.s3, olo = g.jl, ohi = g.ju, ost = g.s2;
  }
  const int no = ohi - olo + 1;
  if (tid >= ni * no) return;
  const int i = g.il + umod(tid, ni);
  const int o = olo + udiv(tid, ni);
  const int f0 = lo + seg * seglen;
  if (f0 > hi) return;
  const int f1 = min(f0 + seglen, hi + 1);
  const int64_t base = i + o * ost;
  const int64_t sv = g.sv;
  const float *w = b.w, *r = b.R;
  float* D = b.D;
  const int ivx = AX == 2 ? IVY : IVZ;
  const float A = (float)(AX == 2 ? g.A2 : g.A3);
  const int disabled = AX == 2 ? p.disable2 : p.disable3;
  const float rref = b.rbf[i], pref = b.pbf[i];
  const float gamma = (float)p.gammad;

  // five-cell window (cells c-2 .. c+2) and the cell after it, loaded a step
  // ahead so that its latency overlaps this step's arithmetic; the stencil
  // stays inside the array (nghost >= 3)
  float q[NV][6];
  int at = (int)base + (f0 - 3) * (int)st;  // (indices stay below 2^31: check_config)
  const int svi = (int)sv, sti = (int)st;
  auto load = [&](int slot) {
#pragma unroll
    for (int v = 0; v < 5; ++v) q[v][slot] = w[v * svi + at];
#pragma unroll
    for (int n = 0; n < NS; ++n) q[5 + n][slot] = r[n * svi + at];
    at += sti;
  };
#pragma unroll
  for (int t = 0; t < 5; ++t) load(t);

  // The face of cell c pairs its left value with the right value of the cell
  // before, carried in L; it closes cell c - 1.
  const int t23 = p.r23_shock ? p.r23_type : interp2_of(p.r23_type);
  float L[NV], Fp[NV];
#pragma unroll
  for (int v = 0; v < NV; ++v) L[v] = Fp[v] = 0.f;
  int off = (int)base + (f0 - 2) * sti;  // cell c - 1
  for (int c = f0 - 1; c <= f1; ++c, off += sti) {
    if (c < f1) load(5);
    // the running sums of cell c - 1, fetched before the face's arithmetic
    float dprev[NV];
    if (c > f0 && !first) {
#pragma unroll
      for (int v = 0; v < NV; ++v) dprev[v] = D[v * svi + off];
    }
    float R[NV], H[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v)
      sweep_cell_states<FP>(v >= 5 ? p.rs_type : (v == IDN ? p.r23_type : t23),
                            v >= 5 ? p.rs_scale != 0 : p.r23_scale != 0, v, q[v], R[v], H[v]);
    if (c >= f0) {
      const float pl = L[IPR], pr = R[IPR];
      L[IDN] += rref;
      R[IDN] += rref;
      L[IPR] += pref;
      R[IPR] += pref;
      float F[NV];
      if (disabled) {
#pragma unroll
        for (int v = 0; v < 5; ++v) F[v] = 0.f;
      } else {
        sweep_riemann<FP>(p.riemann, L, R, pl, pr, pref, ivx, gamma, F);
      }
#pragma unroll
      for (int n = 0; n < NS; ++n)
        F[5 + n] = F[IDN] > 0.f ? F[IDN] * L[5 + n] : F[IDN] * R[5 + n];
      if (c > f0) {
        float d[NV];
#pragma unroll
        for (int v = 0; v < NV; ++v) {
          d[v] = A * F[v] - A * Fp[v];
          if (!first) d[v] = dprev[v] + d[v];
        }
        if constexpr (END == kKeep) {
#pragma unroll
          for (int v = 0; v < NV; ++v) D[v * svi + off] = d[v];
        } else {
          float wc[5];
#pragma unroll
          for (int v = 0; v < 5; ++v) wc[v] = q[v][1];
          finalize32<NS, END == kUpdate>(sh.fin, off, i, d, wc);
        }
      }
#pragma unroll
      for (int v = 0; v < NV; ++v) Fp[v] = F[v];
    }
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      L[v] = H[v];
#pragma unroll
      for (int t = 0; t < 5; ++t) q[v][t] = q[v][t + 1];
    }
  }
}

template <int NS, int AX, int FP, int END>
__global__ void __launch_bounds__(128, kMarchCtas32<NS, FP, END>)
    k_march32(Geo g, Phys p, StageBufs32 b, int seglen, int first) {
  Shared32& sh = shared32();
  // (each of the copies by its own warp: they are one after the other's latency
  // otherwise)
  if (threadIdx.x == 0) {
    sh.m.g = g;
    sh.m.seglen2 = sh.m.seglen3 = seglen;
  } else if (threadIdx.x == 32) {
    sh.m.b = b;
  } else if (threadIdx.x == 64) {
    sh.p = p;
  } else if (threadIdx.x == 96) {
    sh.fin.set(g, p, b);
  }
  __syncthreads();
  march32_line<NS, AX, FP, END>(first, blockIdx.x * blockDim.x + threadIdx.x, blockIdx.y);
}

// ---------------------------------------------------------------------------
// boundary fills of perturbation arrays: as k_bc, plus the x1 offset of the
// reference between the source and the ghost layer (rho, and E or p)
// ---------------------------------------------------------------------------
struct AxisBC32 {
  int n, ng, lo_type, hi_type;
};

__device__ __forceinline__ int bc_map32(const AxisBC32& a, int i, bool& flip) {
  flip = false;
  if (a.n == 1) return i;
  if (i < a.ng) {
    switch (a.lo_type) {
      case SNAPB_BC_REFLECTING: flip = true; return 2 * a.ng - 1 - i;
      case SNAPB_BC_PERIODIC: return a.n - 2 * a.ng + i;
      case SNAPB_BC_OUTFLOW: return a.ng;
      default: return i;
    }
  }
  if (i >= a.n - a.ng) {
    switch (a.hi_type) {
      case SNAPB_BC_REFLECTING: flip = true; return 2 * (a.n - a.ng) - 1 - i;
      case SNAPB_BC_PERIODIC: return i - a.n + 2 * a.ng;
      case SNAPB_BC_OUTFLOW: return a.n - a.ng - 1;
      default: return i;
    }
  }
  return i;
}

// ghost cell t = (i, j, k) of the shell from its image inside the block
__device__ __forceinline__ void bc32_cell(int nc1, int nc2, int64_t sv, AxisBC32 a1,
                                          AxisBC32 a2, AxisBC32 a3, float* var, int nv,
                                          int kind, const double* rb, const double* pb,
                                          double igm1, int64_t t, int i, int j, int k) {
  bool f1, f2, f3;
  int si = bc_map32(a1, i, f1), sj = bc_map32(a2, j, f2), sk = bc_map32(a3, k, f3);
  if (si == i && sj == j && sk == k) return;
  int64_t src = ((int64_t)sk * nc2 + sj) * nc1 + si;
  bool flip = kind != SNAPB_SCALAR;
  // A thread's source cell is never its target, so the loads of a group of
  // variables are issued before its stores: the compiler cannot see that the
  // stores miss the sources and would otherwise wait for one load per
  // variable.
  constexpr int kGroup = 8;
  for (int v0 = 0; v0 < nv; v0 += kGroup) {
    float xs[kGroup];
#pragma unroll
    for (int q = 0; q < kGroup; ++q)
      if (v0 + q < nv) xs[q] = var[(v0 + q) * sv + src];
#pragma unroll
    for (int q = 0; q < kGroup; ++q) {
      const int v = v0 + q;
      if (v >= nv) break;
      double x = xs[q];
      if (flip && ((v == IVX && f1) || (v == IVY && f2) || (v == IVZ && f3))) x = -x;
      if (kind != SNAPB_SCALAR && si != i) {
        if (v == IDN) x += rb[si] - rb[i];
        if (v == IPR) x += (pb[si] - pb[i]) * (kind == SNAPB_CONSERVED ? igm1 : 1.0);
      }
      var[v * sv + t] = (float)x;
    }
  }
}

__global__ void k_bc32(Geo g, AxisBC32 a1, AxisBC32 a2, AxisBC32 a3, float* var, int nv,
                       int kind, const double* rb, const double* pb, double igm1) {
  const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= bc_shell_slots(g)) return;
  int i, j, k;
  const int64_t t = bc_shell_cell(g, s, i, j, k);
  bc32_cell(g.nc1, g.nc2, g.sv, a1, a2, a3, var, nv, kind, rb, pb, igm1, t, i, j, k);
}

// conversions between the FP64 state and the FP32 perturbation
__global__ void k_to_pert(int64_t n, int nc1, int kind, double igm1, const double* in,
                          const double* rb, const double* pb, float* out) {
  int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  int i = umod(t, nc1);
  out[IDN * n + t] = (float)(in[IDN * n + t] - rb[i]);
  out[IVX * n + t] = (float)in[IVX * n + t];
  out[IVY * n + t] = (float)in[IVY * n + t];
  out[IVZ * n + t] = (float)in[IVZ * n + t];
  double pref = kind == SNAPB_CONSERVED ? pb[i] * igm1 : pb[i];
  out[IPR * n + t] = (float)(in[IPR * n + t] - pref);
}

__global__ void k_from_pert(int64_t n, int nc1, int kind, double igm1, const float* in,
                            const double* rb, const double* pb, double* out) {
  int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  int i = umod(t, nc1);
  out[IDN * n + t] = (double)in[IDN * n + t] + rb[i];
  out[IVX * n + t] = in[IVX * n + t];
  out[IVY * n + t] = in[IVY * n + t];
  out[IVZ * n + t] = in[IVZ * n + t];
  double pref = kind == SNAPB_CONSERVED ? pb[i] * igm1 : pb[i];
  out[IPR * n + t] = (double)in[IPR * n + t] + pref;
}

// CFL limit from w'; 384 x 384 x 192: 257 us with four index divisions a cell
// -> 154 us (86 us of HBM traffic)
__global__ void __launch_bounds__(256) k_cfl32(Geo g, double gammad, CflUse use, const float* w,
                                               const float* rbf, const float* pbf,
                                               unsigned long long* slots, double* dt_out) {
  const float gamma = (float)gammad;
  float a[3] = {0.f, 0.f, 0.f};
  cfl_cells(g, [&](int64_t o, int i) { cfl32_speeds(w, g.sv, o, rbf[i], pbf[i], gamma, a); });
  double m1, m2, m3;
  cfl32_limits(g, use.use1, use.use2, use.use3, a, m1, m2, m3);
  // (the value of a used axis without a finite speed, as the batched reduction's)
  const double none = __longlong_as_double(0x7f7f7f7f7f7f7f7fll);
  cfl_finish(use, fmin(m1, none), fmin(m2, none), fmin(m3, none), slots, dt_out);
}

// ---------------------------------------------------------------------------
// persistent batched kernels: every CTA pulls (member, tile) items
// ---------------------------------------------------------------------------
// Persistent batched x1 sweep: CTAs of one warp, the next item claimed while the
// current one is worked on
template <int NS, int FP>
__global__ void __launch_bounds__(32, 20)
    k_x1_32_batch(const Member32* __restrict__ mem, Phys p, WorkQueue q, int stage, int last) {
  Shared32& sh = shared32();
  const int lane = threadIdx.x;
  unsigned long long item = 0, ahead = 0;
  if (lane == 0) {
    sh.p = p;
    item = atomicAdd(q.counter, 1ULL);
  }
  item = __shfl_sync(0xffffffffu, item, 0);
  int m = -1;
  while (true) {
    int nm;
    int64_t tile;
    if (!queue_find(q, (int64_t)item, nm, tile)) return;
    if (lane == 0) ahead = atomicAdd(q.counter, 1ULL);
    __syncwarp();  // the last item's rows and descriptor are read
    if (nm != m) {
      load_member_warp(sh.m, mem, nm);
      if (lane == 0) {
        set_stage32(sh.m.b, stage);
        sh.fin.set(sh.m.g, p, sh.m.b);
      }
      __syncwarp();
      m = nm;
    }
    x1_32_item<NS, FP>(tile, last);
    item = __shfl_sync(0xffffffffu, ahead, 0);
  }
}

template <int NS, int AX, int FP, int END>
__global__ void __launch_bounds__(128, kMarchCtas32<NS, FP, END>)
    k_march32_batch(const Member32* __restrict__ mem, Phys p, WorkQueue q, int stage, int first) {
  Shared32& sh = shared32();
  if (threadIdx.x == 0) sh.p = p;
  int m, have = -1;
  int64_t tile;
  while (queue_next(q, m, tile)) {  // (starts with a barrier: the last tile is done)
    if (m != have) {
      load_member(sh.m, mem, m);
      if (threadIdx.x == 0) {
        set_stage32(sh.m.b, stage);
        sh.fin.set(sh.m.g, p, sh.m.b);
      }
      __syncthreads();
      have = m;
    }
    const int nseg = AX == 2 ? sh.m.nseg2 : sh.m.nseg3;
    const int blk = udiv(tile, nseg);
    march32_line<NS, AX, FP, END>(first, blk * blockDim.x + threadIdx.x,
                             (int)tile - blk * nseg);
  }
}

// boundary fill over the ghost shell only (bc_shell_cell, common.cuh)
__global__ void __launch_bounds__(256) k_bc32_batch(const Member32* __restrict__ mem, Phys p,
                                                    WorkQueue q, int kind, double igm1) {
  int m;
  int64_t tile;
  while (queue_next(q, m, tile)) {
    const Geo& g = mem[m].g;
    const Member32& mb = mem[m];
    AxisBC32 a1{g.nc1, g.ng, mb.bc[0], mb.bc[1]};
    AxisBC32 a2{g.nc2, g.ng, mb.bc[2], mb.bc[3]};
    AxisBC32 a3{g.nc3, g.ng, mb.bc[4], mb.bc[5]};
    float* var = kind == SNAPB_SCALAR ? mb.b.s : mb.b.u;
    const int nv = kind == SNAPB_SCALAR ? p.nscalar : 5;
    const int64_t n = bc_shell_slots(g), s0 = tile * kShellItem;
    for (int64_t slot = s0 + threadIdx.x; slot < min(s0 + kShellItem, n); slot += blockDim.x) {
      int i, j, k;
      const int64_t t = bc_shell_cell(g, slot, i, j, k);
      bc32_cell(g.nc1, g.nc2, g.sv, a1, a2, a3, var, nv, kind, mb.b.rb, mb.b.pb, igm1, t, i, j,
                k);
    }
  }
}

// Face profile of the FP32 sweeps along `axis` (sweep_cell_states, pert.cuh):
// 1, 2, 3 for the default reconstruction with LMARS, HLLC, Roe; 0 otherwise.
int face_profile32(const Phys& p, int axis) {
  const int typ = axis == 1 ? p.r1_type : p.r23_type;
  const int shock = axis == 1 ? p.r1_shock : p.r23_shock;
  const int scale = axis == 1 ? p.r1_scale : p.r23_scale;
  if (typ != SNAPB_RECON_WENO5 || shock || scale) return 0;
  if (p.nscalar > 0 && (p.rs_type != SNAPB_RECON_WENO5 || p.rs_scale)) return 0;
  switch (p.riemann) {
    case SNAPB_RIEMANN_LMARS: return 1;
    case SNAPB_RIEMANN_HLLC: return 2;
    case SNAPB_RIEMANN_ROE: return 3;
  }
  return 0;
}

// f(NS, FP) with the scalar count and the face profile as compile-time constants
template <class F>
static cudaError_t with_ns_profile(int ns, int fp, F&& f) {
#define SNAPB_NF(NS, FP) \
  case NS * 4 + FP:      \
    return f(std::integral_constant<int, NS>{}, std::integral_constant<int, FP>{});
  if (ns < 0 || ns > 3 || fp < 0 || fp > 3) return cudaErrorInvalidValue;
  switch (ns * 4 + fp) {
    SNAPB_NF(0, 0) SNAPB_NF(0, 1) SNAPB_NF(0, 2) SNAPB_NF(0, 3)
    SNAPB_NF(1, 0) SNAPB_NF(1, 1) SNAPB_NF(1, 2) SNAPB_NF(1, 3)
    SNAPB_NF(2, 0) SNAPB_NF(2, 1) SNAPB_NF(2, 2) SNAPB_NF(2, 3)
    SNAPB_NF(3, 0) SNAPB_NF(3, 1) SNAPB_NF(3, 2) SNAPB_NF(3, 3)
  }
#undef SNAPB_NF
  return cudaErrorInvalidValue;
}

cudaError_t launch_x1_32_batch(const Member32* mem, const Phys& p, const WorkQueue& q,
                               int stage, bool last, const PersistGrid& pg, size_t smem,
                               cudaStream_t st) {
  return with_ns_profile(p.nscalar, face_profile32(p, 1), [&](auto ns, auto fp) {
    constexpr int NS = decltype(ns)::value, FP = decltype(fp)::value;
    raise_smem_limit(k_x1_32_batch<NS, FP>, 200 * 1024);
    const int grid = persistent_grid(k_x1_32_batch<NS, FP>, 32, smem, pg);
    k_x1_32_batch<NS, FP><<<grid, 32, smem, st>>>(mem, p, q, stage, last ? 1 : 0);
    return cudaGetLastError();
  });
}

// f(AX, END): the x3 march is the last sweep wherever there is one
template <class F>
static cudaError_t with_axis_end(int axis, int end, F&& f) {
  using std::integral_constant;
  if (axis == 3)
    return end == kUpdate ? f(integral_constant<int, 3>{}, integral_constant<int, kUpdate>{})
                          : f(integral_constant<int, 3>{}, integral_constant<int, kTendency>{});
  switch (end) {
    case kKeep: return f(integral_constant<int, 2>{}, integral_constant<int, kKeep>{});
    case kTendency: return f(integral_constant<int, 2>{}, integral_constant<int, kTendency>{});
    default: return f(integral_constant<int, 2>{}, integral_constant<int, kUpdate>{});
  }
}

cudaError_t launch_march32_batch(int axis, const Member32* mem, const Phys& p,
                                 const WorkQueue& q, int stage, bool first, bool last,
                                 const PersistGrid& pg, cudaStream_t st) {
  return with_ns_profile(p.nscalar, face_profile32(p, axis), [&](auto ns, auto fp) {
    return with_axis_end(axis, march_end(p, last), [&](auto ax, auto end) {
      constexpr int NS = decltype(ns)::value, FP = decltype(fp)::value;
      constexpr int AX = decltype(ax)::value, END = decltype(end)::value;
      const auto kernel = k_march32_batch<NS, AX, FP, END>;
      kernel<<<persistent_grid(kernel, 128, 0, pg), 128, 0, st>>>(mem, p, q, stage, first);
      return cudaGetLastError();
    });
  });
}

cudaError_t launch_bc32_batch(const Member32* mem, const Phys& p, const WorkQueue& q, int kind,
                              double igm1, const PersistGrid& pg, cudaStream_t st) {
  k_bc32_batch<<<persistent_grid(k_bc32_batch, 256, 0, pg), 256, 0, st>>>(mem, p, q, kind, igm1);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// launchers (called from capi32.cu)
// ---------------------------------------------------------------------------
cudaError_t launch_ref32(const Geo& g, const Phys& p, const double* rb, const double* pb,
                         double* rbw, double* pbw, const StageBufs32& b, cudaStream_t st) {
  int n = g.nc1 + 1;
  k_ref32<<<(n + 127) / 128, 128, 0, st>>>(g, p, rb, pb, rbw, pbw, b);
  k_ref32_residual<<<(n + 127) / 128, 128, 0, st>>>(g, p, b);
  return cudaGetLastError();
}

// the split of the x1 sweep of one block; columns > 0 asks for that many per
// item (as far as a warp and its shared memory go).  A 1-D block's cells are finished by
// the sweep itself, so its column is not cut into segments whose halos another
// warp would be updating.
X1Split x1_split32(const Geo& g, int nvt, bool last, int columns, double share) {
  X1Split sp = x1_split(g.nx1, g.ng, (int64_t)g.nc2 * g.nc3, nvt, sizeof(float), kX1RowBytes32,
                        kX1Resident32 * share, last);
  if (columns > 0)
    sp = x1_split_columns(sp, g.nx1, g.ng, nvt, sizeof(float), columns, last);
  return sp;
}
int64_t x1_items32(const Geo& g, const X1Split& sp) {
  return ((int64_t)g.nc2 * g.nc3 + sp.K - 1) / sp.K * sp.nseg;
}

cudaError_t launch_x1_32(const Geo& g, const Phys& p, const StageBufs32& b, bool last,
                         cudaStream_t st) {
  const int nvt = 5 + p.nscalar;
  const X1Split sp = x1_split32(g, nvt, last, 0, 1.);
  const size_t smem = (size_t)sp.pitch * nvt * sizeof(float);
  if (smem > 200 * 1024) return cudaErrorInvalidConfiguration;
  return with_ns_profile(p.nscalar, face_profile32(p, 1), [&](auto ns, auto fp) {
    constexpr int NS = decltype(ns)::value, FP = decltype(fp)::value;
    raise_smem_limit(k_x1_32<NS, FP>, 200 * 1024);
    k_x1_32<NS, FP><<<(unsigned)x1_items32(g, sp), 32, smem, st>>>(g, p, b, sp, last ? 1 : 0);
    return cudaGetLastError();
  });
}

cudaError_t launch_march32(int axis, const Geo& g, const Phys& p, const StageBufs32& b,
                           bool first, bool last, cudaStream_t st) {
  const int ni = g.iu - g.il + 1;
  const int no = axis == 2 ? g.ku - g.kl + 1 : g.ju - g.jl + 1;
  const int n = axis == 2 ? g.nx2 : g.nx3;
  int seglen = 32;
  const int64_t threads = (int64_t)ni * no;
  while (seglen > 8 && threads * ((n + seglen - 1) / seglen) < 148LL * 1024 * 2) seglen /= 2;
  const dim3 grid((unsigned)((threads + 127) / 128), (unsigned)((n + seglen - 1) / seglen));
  return with_ns_profile(p.nscalar, face_profile32(p, axis), [&](auto ns, auto fp) {
    return with_axis_end(axis, march_end(p, last), [&](auto ax, auto end) {
      constexpr int NS = decltype(ns)::value, FP = decltype(fp)::value;
      constexpr int AX = decltype(ax)::value, END = decltype(end)::value;
      k_march32<NS, AX, FP, END><<<grid, 128, 0, st>>>(g, p, b, seglen, first ? 1 : 0);
      return cudaGetLastError();
    });
  });
}

cudaError_t launch_bc32(const Geo& g, const snapb_hydro_config& c, float* var, int nv, int kind,
                        const double* rb, const double* pb, cudaStream_t st) {
  AxisBC32 a1{g.nc1, g.ng, c.bc[0], c.bc[1]};
  AxisBC32 a2{g.nc2, g.ng, c.bc[2], c.bc[3]};
  AxisBC32 a3{g.nc3, g.ng, c.bc[4], c.bc[5]};
  const int64_t n = bc_shell_slots_host(g);
  if (n == 0) return cudaSuccess;
  k_bc32<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(g, a1, a2, a3, var, nv, kind, rb, pb,
                                                     1.0 / (c.gammad - 1.0));
  return cudaGetLastError();
}

cudaError_t launch_to_pert(const Geo& g, const Phys& p, int kind, const double* in,
                           const double* rb, const double* pb, float* out, cudaStream_t st) {
  k_to_pert<<<(unsigned)((g.sv + 255) / 256), 256, 0, st>>>(g.sv, g.nc1, kind,
                                                            1.0 / (p.gammad - 1.0), in, rb, pb,
                                                            out);
  return cudaGetLastError();
}

cudaError_t launch_from_pert(const Geo& g, const Phys& p, int kind, const float* in,
                             const double* rb, const double* pb, double* out, cudaStream_t st) {
  k_from_pert<<<(unsigned)((g.sv + 255) / 256), 256, 0, st>>>(g.sv, g.nc1, kind,
                                                              1.0 / (p.gammad - 1.0), in, rb, pb,
                                                              out);
  return cudaGetLastError();
}

cudaError_t launch_cfl32(const Geo& g, const Phys& p, const float* w, const float* rbf,
                         const float* pbf, unsigned long long* slots, double* dt_out,
                         cudaStream_t st) {
  const int blocks = cfl_blocks(g);
  if (blocks > 1) {
    const cudaError_t e = cudaMemsetAsync(slots, 0xff, 4 * sizeof(*slots), st);
    if (e != cudaSuccess) return e;
  }
  k_cfl32<<<blocks, 256, 0, st>>>(g, p.gammad, cfl_use(g, p), w, rbf, pbf, slots, dt_out);
  return cudaGetLastError();
}

}  // namespace snapb

// No kernel waits on bulk copies any more; kept for the callers of the ABI.
extern "C" int snapb_bulk_copy_timeouts(void) { return 0; }
