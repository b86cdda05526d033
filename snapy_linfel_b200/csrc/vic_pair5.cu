// vic_pair5.cu — the 5x5 implicit solve of the FP64 form: blocks, elimination
// from both column ends at once, and back substitution, sixteen lanes a column.
//
// A 5x5 block with its right-hand sides does not fit one thread's registers
// (the column sweep spilled, and pivoted one row at a time: 27,000 cycles a
// layer).  Here eight lanes share a layer: lane q < 5 owns column q of the
// layer's matrix M and of its coupling to the next layer, lane 5 the right-hand
// side, and M is eliminated by Gauss-Jordan steps with scaled partial pivoting
// whose pivot columns travel by shuffle.  Eight lanes walk up from the bottom
// layer while the other eight walk down from the top one, and the two meet in
// the middle, which halves the chain.  Each lane forms its own column of |A|
// and J, so no block goes through memory; the reduced columns and partial
// solutions go through the workspace (30 doubles a layer, read back by rows).
//
// Bound: instruction issue (51 % active at 13 warps per SM) and the pivot
// chain's latency behind it.  77 x 51 columns of 90 layers: 1340 us (blocks,
// sweep) -> 200 us; three CTAs per SM without spills 243 us (a second wave),
// pivoting on the largest entry at every step instead of by threshold 284 us.
#include "vic_common.cuh"

namespace snapb {

namespace {

constexpr int kPairThreads = 128;  // eight columns a CTA
constexpr int kPairElems = 30;     // A' by rows (25), then the solution (5)

__device__ __forceinline__ double sel5(int q, double a, double b, double c, double d, double e) {
  return q == 0 ? a : (q == 1 ? b : (q == 2 ? c : (q == 3 ? d : e)));
}

// the cell's share of its faces' Roe averages
struct PairCell {
  double rho, u, v, w, sd, ke, hp, H;
  __device__ __forceinline__ void set(const double (&x)[5], double gog) {
    const double is = rsqrt(x[IDN]);
    rho = x[IDN];
    u = x[IVX];
    v = x[IVY];
    w = x[IVZ];
    sd = rho * is;
    hp = gog * x[IPR] * (is * is);
    ke = 0.5 * (u * u + v * v + w * w);
    H = hp + ke;
  }
};

// column q of s |A| at the face of two cells (absA_block, vic_blocks.cuh)
__device__ __forceinline__ void abs_a_col(const PairCell& l, const PairCell& r, int q, double gm1,
                                          double s, double (&A)[5]) {
  const double isd = 1. / (l.sd + r.sd), a = l.sd * isd, b = r.sd * isd;
  const double u = a * l.u + b * r.u, v = a * l.v + b * r.v, w = a * l.w + b * r.w;
  const double H = a * l.H + b * r.H, ke = 0.5 * (u * u + v * v + w * w), hp = H - ke;
  const double c2 = gm1 * hp, ic = rsqrt(c2), c = c2 * ic, ihp = gm1 * (ic * ic);
  const double k = 0.5 * ic * ihp, h = 0.5 * ihp;
  const double lm = s * fabs(u - c), l0 = s * fabs(u), lp = s * fabs(u + c);
  const double cke = c * ke, uhp = u * hp, cu = c * u;
  const double e0 = lm * sel5(q, (cke + uhp) * k, -(hp + cu) * k, -v * h, -w * h, h);
  const double e1 = l0 * sel5(q, (hp - ke) * ihp, u * ihp, v * ihp, w * ihp, -ihp);
  const double e2 = lp * sel5(q, (cke - uhp) * k, (hp - cu) * k, -v * h, -w * h, h);
  const double e3 = l0 * sel5(q, -v, 0., 1., 0., 0.), e4 = l0 * sel5(q, -w, 0., 0., 1., 0.);
  const double sum = e0 + e2, cd = c * (e2 - e0);
  A[0] = sum + e1;
  A[1] = u * A[0] + cd;
  A[2] = v * A[0] + e3;
  A[3] = w * A[0] + e4;
  A[4] = H * sum + u * cd + ke * e1 + v * e3 + w * e4;
}

// column q of s dF/dU of a cell (jac_block)
__device__ __forceinline__ void jac_col(const PairCell& c, int q, double gm1, double s,
                                        double (&J)[5]) {
  const double u = c.u, v = c.v, w = c.w;
  J[0] = q == 1 ? s : 0.;
  J[1] = s * sel5(q, gm1 * c.ke - u * u, (2. - gm1) * u, -gm1 * v, -gm1 * w, gm1);
  J[2] = s * sel5(q, -u * v, v, u, 0., 0.);
  J[3] = s * sel5(q, -u * w, w, 0., u, 0.);
  J[4] = s * sel5(q, ((gm1 - 1.) * c.ke - c.hp) * u, c.H - gm1 * u * u, -gm1 * v * u,
                  -gm1 * w * u, (gm1 + 1.) * u);
}

// M^-1 of X2 (every lane's column, by Gauss-Jordan elimination): lane j < 5 of
// the group of eight holds column j of M in X1.  Threshold pivoting: a step
// takes its diagonal entry unless another row's is more than eight times as
// large under the row weights `lg` (binary logarithms, added to the exponent;
// the implicit scaling of the reference's LU, whose rows differ by powers of
// the sound speed).  Rows are not swapped; a step that pivots elsewhere marks
// its row as taken, and the solution is put in order at the end.  Each group
// chooses its own pivots; the warp's vote only decides whether the step is
// written for the diagonal alone, so that a column's bits depend on no other
// column's.
__device__ __forceinline__ void group_solve(double (&X1)[5], double (&X2)[5], const int (&lg)[5]) {
  unsigned left = 31u;
  int perm[5];
  bool moved = false;  // the same in the whole warp
#pragma unroll
  for (int j = 0; j < 5; ++j) {
    double col[5];
    int mag[5], best = 0;
#pragma unroll
    for (int r = 0; r < 5; ++r) {
      col[r] = __shfl_sync(0xffffffffu, X1[r], j, 8);
      mag[r] = max((__double2hiint(col[r]) & 0x7fffffff) + (lg[r] << 20), 0);
      if (left >> r & 1) best = max(best, mag[r]);
    }
    perm[j] = j;
    const bool diagonal = (left >> j & 1) && mag[j] >= best - (3 << 20);
    if (__all_sync(0xffffffffu, diagonal)) {
      const double rp = 1. / col[j], x1p = X1[j] * rp, x2p = X2[j] * rp;
#pragma unroll
      for (int r = 0; r < 5; ++r) {
        X1[r] = r == j ? x1p : fma(-col[r], x1p, X1[r]);
        X2[r] = r == j ? x2p : fma(-col[r], x2p, X2[r]);
      }
    } else {
      moved = true;
      double piv = 1., x1p = 0., x2p = 0.;
      bool found = false;
#pragma unroll
      for (int r = 0; r < 5; ++r) {
        const bool take = diagonal ? r == j : !found && (left >> r & 1) && mag[r] >= best;
        found = found || take;
        perm[j] = take ? r : perm[j];
        piv = take ? col[r] : piv;
        x1p = take ? X1[r] : x1p;
        x2p = take ? X2[r] : x2p;
      }
      const double rp = 1. / piv;
      x1p *= rp;
      x2p *= rp;
#pragma unroll
      for (int r = 0; r < 5; ++r) {
        X1[r] = r == perm[j] ? x1p : fma(-col[r], x1p, X1[r]);
        X2[r] = r == perm[j] ? x2p : fma(-col[r], x2p, X2[r]);
      }
    }
    left &= ~(1u << perm[j]);
  }
  if (moved) {
    double out[5];
#pragma unroll
    for (int j = 0; j < 5; ++j) out[j] = sel5(perm[j], X2[0], X2[1], X2[2], X2[3], X2[4]);
#pragma unroll
    for (int j = 0; j < 5; ++j) X2[j] = out[j];
  }
}

__global__ void __launch_bounds__(kPairThreads, 4) k_vic_pair5(Geo g, Phys p, StageBufs b) {
  // one matrix per group of eight lanes, 26 doubles apart: the four groups of
  // a warp read different banks
  __shared__ double mats[kPairThreads / 8][26];
  const int lane = threadIdx.x & 31, q = lane & 7, half = lane >> 3 & 1;
  const int64_t ncol = (int64_t)(g.ju - g.jl + 1) * (g.ku - g.kl + 1);
  const int64_t want = (int64_t)blockIdx.x * (kPairThreads / 16) + (threadIdx.x >> 4);
  const bool alive = want < ncol;
  const int64_t col = alive ? want : ncol - 1;
  double* mat = mats[threadIdx.x >> 3];
  const int nl = g.nx1, mid = (nl + 1) / 2, steps = half ? nl - mid : mid;
  const int64_t sv = g.sv, cb = column_base(g, col);
  double* S = b.vic + col * kPairElems;
  const int64_t SL = ncol * kPairElems;  // doubles per layer
  double* Z = b.vic + (int64_t)nl * SL + col;
  const double gm1 = p.gammad - 1., gog = p.gammad / gm1, dt = *b.dt, idt = 1. / dt;
  const double s = g.A1 * (0.5 / g.vol), grav = p.grav1;
  const double sg = half ? -1. : 1.;        // sign of J in the couplings
  const double mir = q == 1 ? -1. : 1.;     // the wall's mirror on column q
  const int dir = half ? -1 : 1, i0 = half ? nl - 1 : 0;

  auto load_w = [&](int i, double (&x)[5]) {  // i in [-1, nl]
#pragma unroll
    for (int v = 0; v < 5; ++v) x[v] = b.w[v * sv + cb + i];
  };
  auto load_d = [&](int i, double (&x)[5]) {
#pragma unroll
    for (int v = 0; v < 5; ++v) x[v] = b.D[v * sv + cb + i];
  };
  // behind: the cell and face already passed; near couples to that side, far
  // to the layer ahead (b and c going up, c and b going down)
  PairCell cc, cn;
  double Ab[5], near[5], Jc[5], raw[5], du[5];
  {
    double x[5];
    load_w(i0 - dir, x);
    cn.set(x, gog);
    load_w(i0, x);
    cc.set(x, gog);
    abs_a_col(cn, cc, q, gm1, s, Ab);
    jac_col(cn, q, gm1, s, near);
    jac_col(cc, q, gm1, s, Jc);
#pragma unroll
    for (int r = 0; r < 5; ++r) near[r] = -(Ab[r] + sg * near[r]);
  }
  load_w(i0 + dir, raw);
  load_d(i0, du);
  // row weights: rows scale with 1, c, c, c, c^2
  int lg[5];
  {
    const int e = ((__double2hiint(gm1 * cc.hp) >> 20) & 0x7ff) - 1023;  // log2 c^2
    const int ec = max(-200, min(200, e / 2));
    lg[0] = 0;
    lg[1] = lg[2] = lg[3] = -ec;
    lg[4] = -2 * ec;
  }
  double X2[5] = {0., 0., 0., 0., 0.};  // A' column (q < 5), partial solution (q = 5)
  double sum_r2 = 0., sum_du = 0.;
  for (int t = 0; t < mid; ++t) {
    const bool on = t < steps;  // (the shorter half idles in the last step)
    const int i = i0 + dir * t;
    cn.set(raw, gog);
    double rhs[5];
#pragma unroll
    for (int r = 0; r < 5; ++r) rhs[r] = du[r] * idt;
    if (on) {
      sum_r2 += cc.rho * cc.rho;
      sum_du += du[IDN];
    }
    const int ahead = t + 1 < steps ? 1 : 0;  // the next step's inputs, ahead of use
    load_w(i + dir * (1 + ahead), raw);
    load_d(i + dir * ahead, du);
    double An[5], Jn[5], far[5], V[5];
    abs_a_col(cc, cn, q, gm1, s, An);
    jac_col(cn, q, gm1, s, Jn);
#pragma unroll
    for (int r = 0; r < 5; ++r) {
      far[r] = sg * Jn[r] - An[r];
      double a = Ab[r] + An[r];
      if ((r == 1 && q == 0) || (r == 4 && q == 1)) a -= grav;
      if (r == q) a += idt;
      if (t == 0) a += mir * near[r];
      V[r] = q == 5 ? rhs[r] : a;
    }
    // V -= near X2(previous): every lane needs the whole coupling matrix
    __syncwarp();
    if (q < 5)
#pragma unroll
      for (int r = 0; r < 5; ++r) mat[r * 5 + q] = near[r];
    __syncwarp();
#pragma unroll
    for (int r = 0; r < 5; ++r)
#pragma unroll
      for (int k = 0; k < 5; ++k) V[r] = fma(-mat[r * 5 + k], X2[k], V[r]);
#pragma unroll
    for (int r = 0; r < 5; ++r) {
      near[r] = -(An[r] + sg * Jc[r]);
      Ab[r] = An[r];
      Jc[r] = Jn[r];
    }
    double Y[5];
#pragma unroll
    for (int r = 0; r < 5; ++r) Y[r] = q == 5 ? V[r] : far[r];
    group_solve(V, Y, lg);
    if (on) {
      cc = cn;
#pragma unroll
      for (int r = 0; r < 5; ++r) X2[r] = Y[r];
      if (alive && q <= 5) {
        double* out = S + i * SL + (q < 5 ? q : 25);
#pragma unroll
        for (int r = 0; r < 5; ++r) out[q < 5 ? r * 5 : r] = Y[r];
      }
    }
  }
  // the middle: x_{mid-1} = p - A' x_mid and x_mid = p' - B' x_{mid-1}, so
  // (I - A' B') x_{mid-1} = p - A' p'
  double x[5];
  {
    __syncwarp();
    if (q < 5)
#pragma unroll
      for (int r = 0; r < 5; ++r) mat[r * 5 + q] = X2[r];
    __syncwarp();
    double V[5], Y[5], other[5];
#pragma unroll
    for (int r = 0; r < 5; ++r) {
      other[r] = __shfl_sync(0xffffffffu, X2[r], lane | 8);  // B' column, p' (upper half)
      V[r] = q == 5 ? X2[r] : (r == q ? 1. : 0.);
    }
#pragma unroll
    for (int r = 0; r < 5; ++r)
#pragma unroll
      for (int k = 0; k < 5; ++k) V[r] = fma(-mat[r * 5 + k], other[k], V[r]);
#pragma unroll
    for (int r = 0; r < 5; ++r) Y[r] = V[r];
    group_solve(V, Y, lg);  // (the upper half's result is not used)
#pragma unroll
    for (int r = 0; r < 5; ++r) x[r] = __shfl_sync(0xffffffffu, Y[r], (lane & 16) | 5);
  }
  // outwards from the middle: lane r takes row r of the layer's A'
  const int r = min(q, 4);
  double sum_x = 0.;
  double row[6];
  auto load_row = [&](int i) {
#pragma unroll
    for (int k = 0; k < 5; ++k) row[k] = S[i * SL + r * 5 + k];
    row[5] = S[i * SL + 25 + r];
  };
  const int j0 = half ? mid : mid - 1, out_dir = -dir;
  __syncwarp();  // the columns written above are visible to the warp
  load_row(min(j0, nl - 1));
  for (int t = 0; t < mid; ++t) {
    const bool on = t < steps;
    const int i = j0 + out_dir * t;
    double v = row[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) v = fma(-row[k], x[k], v);
    if (half == 0 && t == 0) v = sel5(r, x[0], x[1], x[2], x[3], x[4]);  // known already
    if (t + 1 < steps) load_row(i + out_dir);
    if (on && alive && q < 5) S[i * SL + 25 + r] = v;
    if (on && q == 0) sum_x += v;
    double nx[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) nx[k] = __shfl_sync(0xffffffffu, v, k, 8);
#pragma unroll
    for (int k = 0; k < 5; ++k) x[k] = on ? nx[k] : x[k];
  }
  // column sums of the mass redistribution
  double lost = sum_du - sum_x;
  lost += __shfl_xor_sync(0xffffffffu, lost, 8);
  sum_r2 += __shfl_xor_sync(0xffffffffu, sum_r2, 8);
  if (alive && (lane & 15) == 0) {
    Z[0] = sum_r2 * g.vol * g.vol;
    Z[ncol] = lost * g.vol;
  }
}

}  // namespace

cudaError_t launch_vic_pair5(const Geo& g, const Phys& p, const StageBufs& b, cudaStream_t st) {
  const int64_t ncol = (int64_t)(g.ju - g.jl + 1) * (g.ku - g.kl + 1);
  const int per = kPairThreads / 16;
  k_vic_pair5<<<(unsigned)((ncol + per - 1) / per), kPairThreads, 0, st>>>(g, p, b);
  return cudaGetLastError();
}

}  // namespace snapb
