// vic_chunk.cuh — the vertically implicit correction with 3x3 blocks, one warp
// per group of columns: blocks, block-tridiagonal solve, mass redistribution
// and RK combination in one kernel, with nothing of the solve in HBM.
//
// A column's nl layers are cut into G chunks of m layers, one lane each
// (32 / G columns a warp).  A lane eliminates its chunk's first m - 1 layers
// downwards, which expresses them by the last layer of the chunk below (y-)
// and by its own last layer (y):
//     x_j = p_j - A'_j x_{j+1} - f_j y-          (kept in shared memory)
//     x_0 = P - Q y - S y-                       (carried in registers)
// The G last layers then form a block-tridiagonal system of their own, solved
// by parallel cyclic reduction across the lanes (shuffles), and each lane
// substitutes back; columns that this would cost digits are solved again in
// sequence (chunk_solve).  Against the sequential sweep (one thread per column) a
// layer costs 3 to 4 times the FP64 operations, but its chain is m layers and
// log2 G reductions long instead of nl layers, the reduced blocks (96 B a
// layer, written and read back through HBM by the sweep) stay in shared
// memory, and the finish needs no pass of its own.
//
// Bound: instruction issue (about half of it FP64) at 8 resident warps per SM
// (registers).  48 members of 64 and 128 layers, FP32 form: chunks of four
// layers 4.0 ms a stage, of eight 4.75 (twice the shared memory, so five
// warps); a budget of 168 registers for 12 warps spills, 5.4; the reduction
// unrolled over its five levels 5.3 (instruction cache); the finish's inputs
// fetched before the reduction instead of after it 4.5 -> 4.0 (3.79 now, with items
// of several column groups).
#pragma once

#include <type_traits>

#include "kernels.cuh"
#include "vic_blocks.cuh"
#include "vic_common.cuh"

namespace snapb {

// Precision of the blocks (|A|, J and the assembled a, b, c): FP64 for the
// FP64 form, FP32 for the FP32 perturbation form, whose states are FP32; the
// elimination is FP64 in both.
template <class B>
using ChunkBlockT = std::conditional_t<std::is_same_v<B, StageBufs32>, float, double>;

constexpr int kChunkElems = 21;  // p, A', f of a layer
__host__ __device__ constexpr size_t chunk_smem_bytes(int m) {
  return (((size_t)(m - 1) * kChunkElems + 3) * 32 + 4) * sizeof(double) + 4 * sizeof(int);
}

// Lanes per column: chunks of two to four layers up to 128 layers, longer ones
// above (one warp per column at most).  By the column length alone, so that a
// block gives the same bits alone and in an ensemble.
inline int chunk_lanes(int nl) { return nl <= 32 ? 8 : (nl <= 64 ? 16 : 32); }
inline int chunk_layers(int nl) {
  const int G = chunk_lanes(nl);
  return (nl + G - 1) / G;
}
// Chunks whose layers fit in one CTA's shared memory (columns of up to 1216
// layers); the 5x5 form keeps the column sweep.
inline bool chunk_applies(const Geo& g, const Phys& p) {
  return p.implicit_scheme != 0 && vic_n(p) == 3 &&
         chunk_smem_bytes(chunk_layers(g.nx1)) <= 200 * 1024;
}

__device__ __forceinline__ double chunk_rsqrt(double x) { return rsqrt(x); }
__device__ __forceinline__ float chunk_rsqrt(float x) { return rsqrtf(x); }
// A product that is never contracted into a following sum.  Every contraction
// below is spelled out with mul and fma: the one-block and the batched kernels
// must round alike, and the compiler's own choice depends on the code around.
__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }

// What a cell gives to its two faces and to its Jacobian.
template <class T>
struct ChunkCell {
  T u, v, w, sd, ke, hp, H;  // velocities, sqrt(rho), kinetic energy, enthalpy parts
  __device__ __forceinline__ void set(T rho, T vx, T vy, T vz, T p, T gog) {
    const T is = chunk_rsqrt(rho);
    u = vx;
    v = vy;
    w = vz;
    sd = mul(rho, is);
    hp = mul(mul(gog, p), mul(is, is));
    ke = mul(T(0.5), fma(vx, vx, fma(vy, vy, mul(vz, vz))));
    H = hp + ke;
  }
};

// s |A| of the face between two cells: the rows and columns (IDN, IVX, IPR) of
// R |Lambda| R^-1 at the Roe average (absA_block), with the sums over the
// acoustic waves written out: hp = H - ke is c^2 / (gamma - 1), so one
// reciprocal square root gives c, 1 / c and 1 / hp.
template <class T>
__device__ __forceinline__ void chunk_abs_a(const ChunkCell<T>& l, const ChunkCell<T>& r, T gm1,
                                            T s, T (&A)[3][3]) {
  const T isd = fdiv(T(1), l.sd + r.sd), a = mul(l.sd, isd), b = mul(r.sd, isd);
  const T u = fma(a, l.u, mul(b, r.u)), v = fma(a, l.v, mul(b, r.v));
  const T w = fma(a, l.w, mul(b, r.w)), H = fma(a, l.H, mul(b, r.H));
  const T vw = fma(v, v, mul(w, w)), ke = mul(T(0.5), fma(u, u, vw));
  const T hp = H - ke, c2 = mul(gm1, hp);
  const T ic = chunk_rsqrt(c2), c = mul(c2, ic), ihp = mul(gm1, mul(ic, ic));
  const T k = mul(mul(T(0.5), ic), ihp), i2hp = mul(T(0.5), ihp);
  const T lm = mul(s, fabs(u - c)), l0 = mul(s, fabs(u)), lp = mul(s, fabs(u + c));
  const T cke = mul(c, ke), uhp = mul(u, hp), cu = mul(c, u);
  const T lmk = mul(lm, k), lpk = mul(lp, k), l0i = mul(l0, ihp);
  const T Lm[3] = {mul(lmk, cke + uhp), -mul(lmk, hp + cu), mul(lm, i2hp)};
  const T L0[3] = {mul(l0i, hp - ke), mul(l0i, u), -l0i};
  const T Lp[3] = {mul(lpk, cke - uhp), mul(lpk, hp - cu), mul(lp, i2hp)};
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const T sum = Lm[q] + Lp[q], cd = mul(c, Lp[q] - Lm[q]);
    A[0][q] = sum + L0[q];
    A[1][q] = fma(u, A[0][q], cd);
    A[2][q] = fma(H, sum, fma(u, cd, mul(ke, L0[q])));
  }
  A[2][0] = fma(-l0, vw, A[2][0]);
}

// s dF/dU of a cell (jac_block)
template <class T>
__device__ __forceinline__ void chunk_jac(const ChunkCell<T>& c, T gm1, T s, T (&J)[3][3]) {
  const T su = mul(s, c.u), uu = mul(c.u, c.u);
  J[0][0] = T(0);
  J[0][1] = s;
  J[0][2] = T(0);
  J[1][0] = mul(s, fma(gm1, c.ke, -uu));
  J[1][1] = mul(T(2) - gm1, su);
  J[1][2] = mul(s, gm1);
  J[2][0] = mul(fma(gm1 - T(1), c.ke, -c.hp), su);
  J[2][1] = mul(s, fma(-gm1, uu, c.H));
  J[2][2] = mul(gm1 + T(1), su);
}

// The blocks of a column's layers in upward order, in the precision BT:
// b_l = -(|A|_l + J_{l-1}), a_l = |A|_l + |A|_{l+1} + 1/dt - phi and
// c_l = -(|A|_{l+1} - J_{l+1}) (|A|_l at the lower face of layer l, all scaled
// by s = A / 2V), with the walls folded into a at the first and last layers.
template <class BT>
struct ChunkBlocks {
  BT gm1, s, idt, grav;
  ChunkCell<BT> cc;                // the layer's cell
  BT Af[3][3], bf[3][3], Jc[3][3];  // |A| of its lower face, its b, J of its cell
  __device__ __forceinline__ void start(const ChunkCell<BT>& below, const ChunkCell<BT>& cell) {
    BT Jp[3][3];
    cc = cell;
    chunk_abs_a(below, cell, gm1, s, Af);
    chunk_jac(below, gm1, s, Jp);
    chunk_jac(cell, gm1, s, Jc);
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int q = 0; q < 3; ++q) bf[r][q] = -(Af[r][q] + Jp[r][q]);
  }
  // a, b, c of layer l from the cell above it; layers past the column's end
  // are x = 0.  TR: of the transposed system, whose row l holds a_l^T,
  // c_{l-1}^T and b_{l+1}^T, when tr is set.
  template <bool TR>
  __device__ __forceinline__ void next(const ChunkCell<BT>& cn, int l, int nl, bool tr,
                                       double (&a)[3][3], double (&b)[3][3], double (&c)[3][3]) {
    BT An[3][3], Jn[3][3], af[3][3], bv[3][3], cv[3][3], up[3][3];
    chunk_abs_a(cc, cn, gm1, s, An);
    chunk_jac(cn, gm1, s, Jn);
    const bool real = l < nl, first = l == 0, last = l == nl - 1;
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        BT av = Af[r][q] + An[r][q];
        if ((r == 1 && q == 0) || (r == 2 && q == 1)) av -= grav;
        if (r == q) av += idt;
        af[r][q] = av;
        bv[r][q] = bf[r][q];
        cv[r][q] = Jn[r][q] - An[r][q];
        if (TR) up[r][q] = Jc[r][q] - Af[r][q];  // c of the layer below
        bf[r][q] = -(An[r][q] + Jc[r][q]);       // b of the layer above
        Af[r][q] = An[r][q];
        Jc[r][q] = Jn[r][q];
      }
    if (first || l >= nl - 1) {
#pragma unroll
      for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          if (first) af[r][q] += q == 1 ? -bv[r][q] : bv[r][q];
          if (last) af[r][q] += q == 1 ? -cv[r][q] : cv[r][q];
          if (!real) af[r][q] = r == q ? BT(1) : BT(0);
        }
    }
    if (TR) {
#pragma unroll
      for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          if (q > r) {
            const BT x = af[r][q];
            af[r][q] = tr ? af[q][r] : x;
            af[q][r] = tr ? x : af[q][r];
          }
          bv[r][q] = tr ? up[q][r] : bv[r][q];
          cv[r][q] = tr ? bf[q][r] : cv[r][q];
        }
    }
    if (first || l >= nl - 1) {
#pragma unroll
      for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          if (first || !real) bv[r][q] = BT(0);
          if (last || !real) cv[r][q] = BT(0);
        }
    }
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        a[r][q] = (double)af[r][q];
        b[r][q] = (double)bv[r][q];
        c[r][q] = (double)cv[r][q];
      }
    cc = cn;
  }
};

// C -= X Y, c -= X y (three fused operations an entry, no separate sum)
__device__ __forceinline__ void sub_mul3(const double (&X)[3][3], const double (&Y)[3][3],
                                         double (&C)[3][3]) {
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int q = 0; q < 3; ++q)
      C[r][q] = fma(-X[r][2], Y[2][q], fma(-X[r][1], Y[1][q], fma(-X[r][0], Y[0][q], C[r][q])));
}
__device__ __forceinline__ void sub_mul3(const double (&X)[3][3], const double (&y)[3],
                                         double (&c)[3]) {
#pragma unroll
  for (int r = 0; r < 3; ++r)
    c[r] = fma(-X[r][2], y[2], fma(-X[r][1], y[1], fma(-X[r][0], y[0], c[r])));
}
// Z = X Y, z = X y, Z = -X Y
__device__ __forceinline__ void mul3(const double (&X)[3][3], const double (&Y)[3][3],
                                     double (&Z)[3][3]) {
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int q = 0; q < 3; ++q)
      Z[r][q] = fma(X[r][2], Y[2][q], fma(X[r][1], Y[1][q], mul(X[r][0], Y[0][q])));
}
__device__ __forceinline__ void mul3(const double (&X)[3][3], const double (&y)[3],
                                     double (&z)[3]) {
#pragma unroll
  for (int r = 0; r < 3; ++r) z[r] = fma(X[r][2], y[2], fma(X[r][1], y[1], mul(X[r][0], y[0])));
}
__device__ __forceinline__ void neg_mul3(const double (&X)[3][3], const double (&Y)[3][3],
                                         double (&Z)[3][3]) {
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int q = 0; q < 3; ++q)
      Z[r][q] = fma(-X[r][2], Y[2][q], fma(-X[r][1], Y[1][q], mul(-X[r][0], Y[0][q])));
}
// cofactor inverse (inverse3, vic_blocks.cuh)
__device__ __forceinline__ void chunk_inverse(const double (&M)[3][3], double (&inv)[3][3]) {
  double cof[3][3];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const int i1 = (i + 1) % 3, i2 = (i + 2) % 3, j1 = (j + 1) % 3, j2 = (j + 2) % 3;
      cof[i][j] = fma(M[i1][j1], M[i2][j2], -mul(M[i1][j2], M[i2][j1]));
    }
  const double id =
      1. / fma(cof[2][0], M[2][0], fma(cof[1][0], M[1][0], mul(cof[0][0], M[0][0])));
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) inv[i][j] = mul(cof[j][i], id);
}
// the values of lane d of the column
template <int G>
__device__ __forceinline__ void shfl3(const double (&X)[3][3], int d, double (&Y)[3][3]) {
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int q = 0; q < 3; ++q)
      Y[r][q] = __shfl_sync(0xffffffffu, X[r][q], d, G);
}
template <int G>
__device__ __forceinline__ void shfl3(const double (&x)[3], int d, double (&y)[3]) {
#pragma unroll
  for (int r = 0; r < 3; ++r)
    y[r] = __shfl_sync(0xffffffffu, x[r], d, G);
}

// Largest magnitude among the diagonal entries of matrices, as the high word of a
// double (which orders as the value does).
struct Growth {
  int hi = 0;
  __device__ __forceinline__ void note(const double (&X)[3][3]) {
#pragma unroll
    for (int r = 0; r < 3; ++r) hi = max(hi, __double2hiint(X[r][r]) & 0x7fffffff);
  }
};
// The growth from which a column is solved in sequence (chunk_solve), as such a
// word: 1.5 with blocks in FP64, 32 with blocks in FP32, whose own rounding is the
// larger error below that.
template <class BT>
constexpr int kGrowthLimit = sizeof(BT) == 8 ? 0x3ff80000 : (1023 + 5) << 20;

// Solve the block-tridiagonal system of a column, one lane per chunk of m
// layers (lane k of the column's G): eq(j, a, bl, c, rhs), called for j = 0 ..
// m - 1 in turn, gives the equation bl x_{l-1} + a x_l + c x_{l+1} = rhs of the
// lane's j-th layer (bl zero at the column's first layer, c at its last, and
// the identity past its end); mid() is called between the elimination and the
// reduction.  The solution is left in mine[(j * kChunkElems + r) * 32], the sum of
// its first row over the lane's first `left` layers in sum_x.
//
// Returns whether the column is to be solved again by chunk_sequence: chunks and
// the cyclic reduction eliminate stretches of layers that are open at both ends.
// Where a stretch traps a wave (vertical flow converging in it, at vertical
// Courant numbers far above one) its block is nearly singular although the
// column's system is not, and the entries that the elimination makes of it grow by
// as much as its result loses in digits; the elimination from the lower wall up
// meets no such stretch.  So a column goes there whose Q, S or first B and C have
// diagonal entries above `limit`.  Error against 80-bit solutions, 6500 columns of 9
// to 256 layers, Courant numbers 0.5 to 10^4, vertical Mach numbers 3e-4 to 1.5: of
// the columns that stay 1.15 times the sequential solve's in the mean, 3.3 times in
// the worst hundredth, 26 at most; of those that go up to 10^11 times.  None goes at
// Courant numbers up to 10 below Mach 0.1, nor up to 100 below Mach 0.01.  (Watching
// every layer and every level as well kept no better and cost 7 % of the solve.)
template <int G, class Eq, class Mid>
__device__ __forceinline__ bool chunk_solve(int m, int k, double* mine, int limit, Eq&& eq,
                                            Mid&& mid, int left, double& sum_x) {
  Growth growth;
  // ---- elimination inside the chunk ----
  double Ap[3][3] = {}, f[3][3] = {}, pv[3] = {};           // A', f, p of the layer below
  double Q[3][3] = {}, S[3][3] = {}, P[3] = {};             // first layer's relation
#pragma unroll
  for (int r = 0; r < 3; ++r) f[r][r] = Q[r][r] = -1.;      // (none yet: x_0 = x_0)
  double a[3][3], bl[3][3], c[3][3], rhs[3];                // the layer's equation
  for (int j = 0;; ++j) {
    eq(j, a, bl, c, rhs);
    if (j == m - 1) break;
    double inv[3][3], t33[3][3];
    if (j > 0) {
      sub_mul3(bl, Ap, a);
      sub_mul3(bl, pv, rhs);
      mul3(bl, f, t33);
    } else {
#pragma unroll
      for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int q = 0; q < 3; ++q) t33[r][q] = -bl[r][q];
    }
    chunk_inverse(a, inv);
    mul3(inv, c, Ap);
    mul3(inv, rhs, pv);
    neg_mul3(inv, t33, f);
    double* out = mine + (size_t)j * kChunkElems * 32;
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      out[r * 32] = pv[r];
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        out[(3 + r * 3 + q) * 32] = Ap[r][q];
        out[(12 + r * 3 + q) * 32] = f[r][q];
      }
    }
    if (j > 0) {
      sub_mul3(Q, pv, P);
      sub_mul3(Q, f, S);
      neg_mul3(Q, Ap, t33);
#pragma unroll
      for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int q = 0; q < 3; ++q) Q[r][q] = t33[r][q];
    } else {
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        P[r] = pv[r];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          Q[r][q] = Ap[r][q];
          S[r][q] = f[r][q];
        }
      }
    }
  }
  mid();

  // ---- the system of the chunks' last layers ----
  double Bm[3][3], Cm[3][3], y[3];
  {
    double Pn[3], Qn[3][3], Sn[3][3], inv[3][3], t33[3][3];
    shfl3<G>(P, k + 1, Pn);
    shfl3<G>(Q, k + 1, Qn);
    shfl3<G>(S, k + 1, Sn);  // (the last chunk's c is zero)
    sub_mul3(bl, Ap, a);
    sub_mul3(c, Sn, a);
    sub_mul3(bl, pv, rhs);
    sub_mul3(c, Pn, rhs);
    chunk_inverse(a, inv);
    mul3(inv, rhs, y);
    mul3(bl, f, t33);
    neg_mul3(inv, t33, Bm);
    mul3(c, Qn, t33);
    neg_mul3(inv, t33, Cm);
    growth.note(Q);
    growth.note(S);
    growth.note(Bm);
    growth.note(Cm);
  }
  // y_k + B y_{k-h} + C y_{k+h} = r, strides h = 1, 2, 4, ...: a chunk without
  // a neighbour at that distance has a zero block there, so the values that the
  // shuffle wraps around to do not enter
  auto reduce = [&](int h, bool more) {
    double D[3][3] = {}, Xu[3][3], Xd[3][3], xu[3], xd[3], inv[3][3], Bn[3][3], Cn[3][3];
#pragma unroll
    for (int r = 0; r < 3; ++r) D[r][r] = 1.;
    shfl3<G>(Cm, k - h, Xu);
    shfl3<G>(Bm, k + h, Xd);
    sub_mul3(Bm, Xu, D);
    sub_mul3(Cm, Xd, D);
    shfl3<G>(y, k - h, xu);
    shfl3<G>(y, k + h, xd);
    sub_mul3(Bm, xu, y);
    sub_mul3(Cm, xd, y);
    if (more) {
      shfl3<G>(Bm, k - h, Xu);
      shfl3<G>(Cm, k + h, Xd);
      mul3(Bm, Xu, Bn);
      mul3(Cm, Xd, Cn);
    }
    chunk_inverse(D, inv);
    double t[3];
    mul3(inv, y, t);
#pragma unroll
    for (int r = 0; r < 3; ++r) y[r] = t[r];
    if (more) {
      neg_mul3(inv, Bn, Bm);
      neg_mul3(inv, Cn, Cm);
    }
  };
  // (kept a loop: unrolled, its five copies overran the instruction cache)
#pragma unroll 1
  for (int h = 1; 2 * h < G; h *= 2) reduce(h, true);
  reduce(G / 2, false);

  // ---- back substitution; x takes the place of p ----
  double ym[3], x[3];
  shfl3<G>(y, k - 1, ym);
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    if (k == 0) ym[r] = 0.;
    x[r] = y[r];
    mine[((size_t)(m - 1) * kChunkElems + r) * 32] = x[r];
  }
  sum_x = m - 1 < left ? x[0] : 0.;
  for (int j = m - 2; j >= 0; --j) {
    double* at = mine + (size_t)j * kChunkElems * 32;
    double t[3];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      t[r] = at[r * 32];
#pragma unroll
      for (int q = 0; q < 3; ++q) t[r] = fma(-at[(12 + r * 3 + q) * 32], ym[q], t[r]);
#pragma unroll
      for (int q = 0; q < 3; ++q) t[r] = fma(-at[(3 + r * 3 + q) * 32], x[q], t[r]);
    }
#pragma unroll
    for (int r = 0; r < 3; ++r) at[r * 32] = x[r] = t[r];
    if (j < left) sum_x += x[0];
  }
  const unsigned grown = __ballot_sync(0xffffffffu, growth.hi >= limit);
  return grown >> (threadIdx.x & (32 - G)) & (0xffffffffu >> (32 - G));
}

// The same system of the columns that `again` is set for, layer after layer: the
// column's lanes take turns, from the lower wall up and back.  A layer costs a
// whole warp's issue: with every column of the block here, 512 of 256 layers 19 ->
// 189 us (one thread a column, in the column sweep, 239), 16384 of 128 layers 155
// -> 1816 (296).  From both walls at once with the blocks formed beforehand it took
// 1163 us there, but lost a supersonic column (6e-3) and cost the batched kernel 500
// us of 860 in registers.
template <int G, class Eq>
__device__ __forceinline__ void chunk_sequence(int m, int k, double* mine, bool again, Eq&& eq) {
  double Ap[3][3] = {}, pv[3] = {}, a[3][3], bl[3][3], c[3][3], rhs[3];
#pragma unroll 1
  for (int t = 0; t < G; ++t) {
    if (k == t && again) {
#pragma unroll 1
      for (int j = 0; j < m; ++j) {
        double inv[3][3];
        eq(j, a, bl, c, rhs);
        sub_mul3(bl, Ap, a);
        sub_mul3(bl, pv, rhs);
        chunk_inverse(a, inv);
        mul3(inv, c, Ap);
        mul3(inv, rhs, pv);
        if (j == m - 1) break;  // (its p and A' stay in registers)
        double* out = mine + (size_t)j * kChunkElems * 32;
#pragma unroll
        for (int r = 0; r < 3; ++r) {
          out[r * 32] = pv[r];
#pragma unroll
          for (int q = 0; q < 3; ++q) out[(3 + r * 3 + q) * 32] = Ap[r][q];
        }
      }
    }
    double up[3][3], pu[3];
    shfl3<G>(Ap, t, up);
    shfl3<G>(pv, t, pu);
    if (k == t + 1) {
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        pv[r] = pu[r];
#pragma unroll
        for (int q = 0; q < 3; ++q) Ap[r][q] = up[r][q];
      }
    }
  }
  double x[3] = {};  // (the column's last A' is zero)
#pragma unroll 1
  for (int t = G - 1; t >= 0; --t) {
    if (k == t && again) {
      sub_mul3(Ap, x, pv);
#pragma unroll
      for (int r = 0; r < 3; ++r) mine[((size_t)(m - 1) * kChunkElems + r) * 32] = x[r] = pv[r];
#pragma unroll 1
      for (int j = m - 2; j >= 0; --j) {
        double* at = mine + (size_t)j * kChunkElems * 32;
        double y3[3];
#pragma unroll
        for (int r = 0; r < 3; ++r) {
          y3[r] = at[r * 32];
#pragma unroll
          for (int q = 0; q < 3; ++q) y3[r] = fma(-at[(3 + r * 3 + q) * 32], x[q], y3[r]);
        }
#pragma unroll
        for (int r = 0; r < 3; ++r) at[r * 32] = x[r] = y3[r];
      }
    }
    double above[3];
    shfl3<G>(x, t, above);
    if (k == t - 1)
#pragma unroll
      for (int r = 0; r < 3; ++r) x[r] = above[r];
  }
}
// the sum that chunk_solve gives, from the solution
__device__ __forceinline__ double chunk_sum(int m, const double* mine, int left) {
  double sum_x = 0.;
  for (int j = m - 1; j >= 0; --j)
    if (j < left) sum_x += mine[(size_t)j * kChunkElems * 32];
  return sum_x;
}

// The equations of one lane's chunk: layers l0 .. l0 + m - 1 of the column at cb.
template <class B>
struct ChunkColumn {
  using T = std::remove_pointer_t<decltype(B::u)>;  // stored precision
  using BT = ChunkBlockT<B>;
  const Geo& g;
  const Phys& p;
  const B& b;
  const int cb, l0, m, sv, nl;
  ChunkBlocks<BT> blocks;
  BT gog;
  double idt, rc;  // rc: density of the layer
  double sum_r2, sum_du;
  T rawn[5], rawd[3];

  // state of layer l (clamped to the ghost above the column), as stored
  __device__ __forceinline__ void load_w(int l, T (&raw)[5]) const {
    const int o = cb + min(l, nl);
#pragma unroll
    for (int v = 0; v < 5; ++v) raw[v] = b.w[v * sv + o];
  }
  __device__ __forceinline__ void load_d(int l, T (&raw)[3]) const {
    const int o = cb + min(l, nl - 1);
#pragma unroll
    for (int r = 0; r < 3; ++r) raw[r] = b.D[sel<3>(r) * sv + o];
  }
  // full density of the layer (returned in FP64) and its cell quantities
  __device__ __forceinline__ double make(int l, const T (&raw)[5], ChunkCell<BT>& c) const {
    const int xi = g.il + min(l, nl);
    const double rho = vic_full(b, (double)raw[IDN], IDN, xi);
    c.set((BT)rho, (BT)raw[IVX], (BT)raw[IVY], (BT)raw[IVZ], vic_full_blk(b, raw[IPR], IPR, xi),
          gog);
    return rho;
  }
  __device__ __forceinline__ ChunkColumn(const Geo& g_, const Phys& p_, const B& b_, int cb_,
                                         int l0_, int m_)
      : g(g_), p(p_), b(b_), cb(cb_), l0(l0_), m(m_), sv((int)g_.sv), nl(g_.nx1), sum_r2(0.),
        sum_du(0.) {
    idt = 1. / *b.dt;
    gog = (BT)(p.gammad / (p.gammad - 1.));
    blocks.gm1 = (BT)(p.gammad - 1.);
    blocks.s = (BT)g.A1 * (BT)(0.5 / g.vol);
    blocks.idt = (BT)idt;
    blocks.grav = (BT)p.grav1;
    T raw0[5];
    ChunkCell<BT> below, cell;
    load_w(l0 - 1, rawn);
    load_w(l0, raw0);
    load_d(l0, rawd);
    make(l0 - 1, rawn, below);
    load_w(l0 + 1, rawn);
    rc = make(l0, raw0, cell);
    blocks.start(below, cell);
  }
  __device__ __forceinline__ void operator()(int j, double (&a)[3][3], double (&bl)[3][3],
                                             double (&c)[3][3], double (&rhs)[3]) {
    const int l = l0 + j;
    ChunkCell<BT> cn;
    const double rn = make(l + 1, rawn, cn);
    double du[3];
#pragma unroll
    for (int r = 0; r < 3; ++r) du[r] = l < nl ? (double)rawd[r] : 0.;
    if (j < m - 1) {  // the next layer's inputs, ahead of this one's arithmetic
      load_w(l + 2, rawn);
      load_d(l + 1, rawd);
    }
    blocks.template next<false>(cn, l, nl, false, a, bl, c);
#pragma unroll
    for (int r = 0; r < 3; ++r) rhs[r] = mul(du[r], idt);
    if (l < nl) {
      sum_r2 = fma(rc, rc, sum_r2);
      sum_du += du[0];
    }
    rc = rn;
  }
};

// chunk_sequence of a warp's columns.  Not inlined: it is seldom called, and in
// the body of the kernel it cost the chunked solve its registers (128^3: 50 us a
// stage).
template <int G, class B>
__device__ __noinline__ void chunk_again(const Geo& g, const Phys& p, const B& b, int cb, int m,
                                         double* mine, bool again) {
  const int k = threadIdx.x & (G - 1);
  ChunkColumn<B> column(g, p, b, cb, k * m, m);
  chunk_sequence<G>(m, k, mine, again, column);
}

// The columns col0 .. col0 + 32/G - 1 of a block by one warp; sm: the warp's
// chunk_smem_bytes(m).  Ends with the warp's shared memory still in use by
// other lanes: the caller synchronizes the warp before the next group.
template <int G, int NS, class B>
__device__ __forceinline__ void vic_chunk(const Geo& g, const Phys& p, const B& b, int64_t col0,
                                          int m, double* sm) {
  using T = std::remove_pointer_t<decltype(b.u)>;  // stored precision
  using BT = ChunkBlockT<B>;
  constexpr int CW = 32 / G;
  const int lane = threadIdx.x & 31, k = lane & (G - 1), cw = lane / G;
  // (element indices of every array stay below 2^31: check_config)
  const int sv = (int)g.sv, nl = g.nx1, l0 = k * m;
  const int64_t ncol = (int64_t)(g.ju - g.jl + 1) * (g.ku - g.kl + 1);
  const int cb = (int)column_base(g, min(col0 + cw, ncol - 1));
  double* mine = sm + lane;  // element e of layer j at mine[(j * kChunkElems + e) * 32]
  double* backs = sm + ((size_t)(m - 1) * kChunkElems + 3) * 32;  // [4], then the columns' cb
  int* cbs = reinterpret_cast<int*>(backs + 4);

  ChunkColumn<B> column(g, p, b, cb, l0, m);
  // The finish's inputs of the lane's first IT cells, fetched before the
  // reduction so that it hides their latency; further ones batch by batch.
  constexpr int IT = sizeof(T) == 4 ? (NS == 0 ? 4 : 2) : (NS == 0 ? 2 : 1), NSA = NS > 0 ? NS : 1;
  const bool du_only = b.vic_du_only, stage0 = b.stage == 0;
  const int total = (int)min((int64_t)CW, ncol - col0) * nl;
  const int magic = (65536 + m - 1) / m;  // l / m = l * magic >> 16 (l m < 65536)
  T rho[IT], et[IT], dv[IT][2], uo[IT][5], u0o[IT][5];
  T so[IT][NSA], s0o[IT][NSA], ro[IT][NSA], dso[IT][NSA];
  auto place = [&](int idx, int& c, int& l) {  // column and layer of a cell of the warp
    c = 0;
#pragma unroll
    for (int q = 1; q < CW; ++q) c += idx >= q * nl;
    l = idx - c * nl;
  };
  if (k == 0) cbs[cw] = cb;
  __syncwarp();
  auto fetch = [&](int i0) {
#pragma unroll
    for (int q = 0; q < IT; ++q) {
      int cc, l;
      place(min(i0 + 32 * q, total - 1), cc, l);
      const int off = (CW > 1 ? cbs[cc] : cb) + l;
      rho[q] = b.w[IDN * sv + off];
      et[q] = b.D[IDN * sv + off];
      if (du_only) continue;
      dv[q][0] = b.D[IVY * sv + off];
      dv[q][1] = b.D[IVZ * sv + off];
#pragma unroll
      for (int v = 0; v < 5; ++v) {
        uo[q][v] = b.u[v * sv + off];
        u0o[q][v] = stage0 ? T(0) : b.u0[v * sv + off];
      }
#pragma unroll
      for (int n = 0; n < NS; ++n) {
        const int o = n * sv + off;
        so[q][n] = b.s[o];
        s0o[q][n] = stage0 ? T(0) : b.s0[o];
        ro[q][n] = b.r[o];
        dso[q][n] = b.D[(5 + n) * sv + off];
      }
    }
  };
  auto emit = [&](int i0) {
#pragma unroll
    for (int q = 0; q < IT; ++q) {
      if (i0 + 32 * q >= total) break;
      int cc, l;
      place(i0 + 32 * q, cc, l);
      const int ch = l * magic >> 16, j = l - ch * m, xi = g.il + l;
      const double* at = sm + j * kChunkElems * 32 + cc * G + ch;
      const double rhok = vic_full(b, (double)rho[q], IDN, xi);
      const double fix = at[0] - (double)et[q];
      const double du0 = fma(mul(rhok, rhok), backs[cc], at[0]);
      const int off = (CW > 1 ? cbs[cc] : cb) + l;
      if (b.M) b.M[off] = fix;
      if (du_only) {
        vic_set_d(b, IDN * sv + off, du0);
        vic_set_d(b, IVX * sv + off, at[32]);
        vic_set_d(b, IPR * sv + off, at[64]);
        continue;
      }
      const double du[5] = {du0, at[32], (double)dv[q][0], (double)dv[q][1], at[64]};
      double unew_rho = 0.;
#pragma unroll
      for (int v = 0; v < 5; ++v) {
        const double un = vic_rk_from(b.u, b.u0, v * sv + off, stage0, uo[q][v], u0o[q][v], b.wgt0,
                                      b.wgt1, b.wgt2, du[v]);
        if (v == IDN) unew_rho = vic_full_rho(b, un, xi);
      }
#pragma unroll
      for (int n = 0; n < NS; ++n) {
        const int o = n * sv + off;
        const double ds = fma(fix, (double)ro[q][n], (double)dso[q][n]);
        const double sn = vic_rk_from(b.s, b.s0, o, stage0, so[q][n], s0o[q][n], b.wgt0, b.wgt1,
                                      b.wgt2, ds);
        b.r[o] = sn / unew_rho;
      }
    }
  };
  double sum_x;
  const bool again =
      chunk_solve<G>(m, k, mine, kGrowthLimit<BT>, column, [&] { fetch(lane); }, nl - l0, sum_x);
  if (__any_sync(0xffffffffu, again)) {
    chunk_again<G, B>(g, p, b, cb, m, mine, again);
    sum_x = chunk_sum(m, mine, nl - l0);
  }
  double sum_r2 = column.sum_r2;
  double lost = column.sum_du - sum_x;
#pragma unroll
  for (int h = 1; h < G; h *= 2) {
    lost += __shfl_xor_sync(0xffffffffu, lost, h, G);
    sum_r2 += __shfl_xor_sync(0xffffffffu, sum_r2, h, G);
  }
  if (k == 0) backs[cw] = lost / sum_r2;
  __syncwarp();

  // ---- finish: the warp's cells along x1 ----
  for (int i0 = lane;;) {
    emit(i0);
    i0 += 32 * IT;
    if (i0 - lane >= total) break;
    fetch(i0);
  }
}

// f(G, NS) as compile-time constants
template <class F>
static cudaError_t with_lanes_scalars(int lanes, int ns, F&& f) {
#define SNAPB_GN(G, NS) \
  case G * 4 + NS: return f(std::integral_constant<int, G>{}, std::integral_constant<int, NS>{});
  if (ns < 0 || ns > 3) return cudaErrorInvalidValue;
  switch (lanes * 4 + ns) {
    SNAPB_GN(8, 0) SNAPB_GN(8, 1) SNAPB_GN(8, 2) SNAPB_GN(8, 3)
    SNAPB_GN(16, 0) SNAPB_GN(16, 1) SNAPB_GN(16, 2) SNAPB_GN(16, 3)
    SNAPB_GN(32, 0) SNAPB_GN(32, 1) SNAPB_GN(32, 2) SNAPB_GN(32, 3)
  }
#undef SNAPB_GN
  return cudaErrorInvalidValue;
}

}  // namespace snapb
