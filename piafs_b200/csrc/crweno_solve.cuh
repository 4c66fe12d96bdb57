// The CRWENO5 line solve of one (line, component, field) as a device
// function of a whole CTA (crweno_line.cu); the method is
// described in crweno_line.cu.
#pragma once
#include <type_traits>

#include "crweno_common.cuh"

namespace piafs {

// staged slot of a cell or of an output row: one pad slot per M (a thread's M
// consecutive slots are then at compile-time offsets, and threads at a stride
// of M + 1 doubles fall in distinct banks)
template <int M>
__host__ __device__ __forceinline__ int padm(int j) { return j + j / M; }

__host__ __device__ constexpr int line_threads_max() { return 512; }

// threads of a line of N interfaces at M rows per thread (a multiple of 32)
template <int M>
__host__ __device__ constexpr int line_threads_m(int N) {
  return ((N - 1 + M - 1) / M + 31) / 32 * 32;
}

// The WENO5 boundary-row value (optimal weights 0.1, 0.6, 0.3,
// Interp1PrimFifthOrderCRWENO.c:164-175) of bias q at the interface whose six
// cells i-3 .. i+2 are staged at padm<M>(j0) ..., in the arithmetic of the
// weights.
template <int M, int WT, typename R>
__device__ __forceinline__ double crw_edge_staged(const DevParams& P, const double* cs, int j0, int q) {
  R m[5];
#pragma unroll
  for (int r = 0; r < 5; r++) m[r] = (R)cs[padm<M>(j0 + (q == 0 ? r : 5 - r))];
  R w1, w2, w3;
  weno_weights_t<WT>(R(0.1), R(0.6), R(0.3), m[0], m[1], m[2], m[3], m[4], (R)P.eps, w1, w2, w3);
  return (double)weno5_value(w1, w2, w3, m[0], m[1], m[2], m[3], m[4]);
}

// The boundary rows' values on every lane of a warp that holds a line end:
// lanes 0, 1 evaluate interface 0 (both biases) and lanes 2, 3 interface N,
// whose cells are staged from slots j0 and jN (a warp with one end only
// evaluates that one twice).
template <int M, int WT, typename R>
__device__ __forceinline__ void crw_edges(const DevParams& P, const double* cs, int j0, int jN, double (&x0)[2],
                                          double (&xN)[2]) {
  const int lane = threadIdx.x & 31;
  const double e = crw_edge_staged<M, WT, R>(P, cs, (lane & 2) ? jN : j0, lane & 1);
  x0[0] = __shfl_sync(0xffffffffu, e, 0);
  x0[1] = __shfl_sync(0xffffffffu, e, 1);
  xN[0] = __shfl_sync(0xffffffffu, e, 2);
  xN[1] = __shfl_sync(0xffffffffu, e, 3);
}

// Rows s .. s+M-1 of both biases from the staged cells, reduced to the
// chunk's separator: on return x_{s+r} = rh[q][r] - al[q][r] X_s -
// cg[q][r] X_{s+M} for r = 1 .. M-1, and (As, Bs, Cs, Rs) is the separator
// row s.  FULL: every row lies in [1, N-2] (no folding of row N, no identity
// rows).  R: the arithmetic of the nonlinear weights (double, or float in
// mixed precision); the rows' right-hand sides, the rows themselves and their
// elimination are FP64 in both, and in mixed precision each first difference
// and each weight product is converted once and serves both biases' rows.
//
// The line solve issues about as many FP64 instructions as the pipe takes at
// its occupancy, so the rows are formed with few of them: the smoothness
// indicators from first differences g shared by neighbouring windows, with
// eps folded into the curvature term (13 operations a window where the
// three-cell forms take 18), the averages of the right-hand side from 3c and
// g, and the rows scaled so that three coefficients are plain products.
// Measured (B200, 11 variables): 0.876 ms a launch at 2048^2 and 62 us at 512^2;
// with the three-cell forms, all PCR levels, per-row tests of both line ends
// and the end values formed from global memory before the rows 1.097 ms and
// 72 us.
template <int M, int WT, bool FULL, typename R>
__device__ __forceinline__ void crw_chunk(const double* __restrict__ cs, int k, int s, int N, const double* x0,
                                          const double* xN, R eps, double (&As)[2], double (&Bs)[2],
                                          double (&Cs)[2], double (&Rs)[2], double (&al)[2][M],
                                          double (&cg)[2][M], double (&rh)[2][M], int& bad) {
  // cells s-3 .. s+M+1 (staged index = cell + 3)
  double c[M + 5];
#pragma unroll
  for (int r = 0; r < M + 5; r++) c[r] = cs[k * (M + 1) + padm<M>(1 + r)];
  // First differences g[t] = c[t+1] - c[t] and, per window t (cells s-3+t ..
  // s-1+t), the smoothness indicators at 4x (b1: 13/3 d^2 + (a-4b+3c)^2, b2:
  // .. (a-c)^2, b3: .. (3a-4b+c)^2 with d = a-2b+c, each inner form a
  // combination of d and the two differences) and, for Jiang-Shu, q = (beta +
  // eps)^2.  Two-cell averages of the compact right-hand side at 3x for cells
  // (s-3+j, s-2+j): pp = 5/2 left + 1/2 right = 3 left + g/2, qq = 1/2 left +
  // 5/2 right = 3 right - g/2.  Everything is produced in the row loop as the
  // rows need it (row r reads windows up to r+3), which keeps the live range
  // of each value short.
  R gw[M + 4], dw[M + 3], b1[M + 3], b2[M + 3], b3[M + 3], q1[M + 3], q2[M + 3], q3[M + 3];
  double pp[M + 3], qq[M + 3], c3[M + 4];
  auto diff = [&](int t) {
    const double g = c[t + 1] - c[t];
    gw[t] = (R)g;
    if (t >= 1 && t < M + 3) {
      if (t == 1) c3[1] = 3.0 * c[1];
      c3[t + 1] = 3.0 * c[t + 1];
      pp[t] = fma(0.5, g, c3[t]);
      qq[t] = fma(-0.5, g, c3[t + 1]);
    }
  };
  auto window = [&](int t) {
    if (WT != WT_NOLIM) {
      const R g0 = gw[t], g1 = gw[t + 1];
      const R d = g1 - g0;
      dw[t] = d;
      const R e1 = d + R(2) * g1, e2 = g0 + g1, e3 = d - R(2) * g0;
      const R dk = R(13.0 / 3.0) * d;
      if (WT == W_JS) {
        const R dd = dk * d + eps;
        const R s1 = dd + e1 * e1, s2 = dd + e2 * e2, s3 = dd + e3 * e3;
        q1[t] = s1 * s1; q2[t] = s2 * s2; q3[t] = s3 * s3;
      } else {
        const R dd = dk * d;
        b1[t] = dd + e1 * e1;
        b2[t] = dd + e2 * e2;
        b3[t] = dd + e3 * e3;
      }
    }
  };
  // Jiang-Shu products of left-row index j: P23 = q2[j+1] q3[j+2],
  // H13 = 5/2 q1[j] q3[j+2], P12 = q1[j] q2[j+1]; the left row j has the
  // weights (0.2 P23, 0.2 H13, 0.3 P12), the right row j-1 (0.2 P12, 0.2 H13,
  // 0.3 P23)
  double P23[M + 1], H13[M + 1], P12[M + 1];
  auto products = [&](int j) {
    P23[j] = (double)(q2[j + 1] * q3[j + 2]);
    H13[j] = (double)((R(2.5) * q1[j]) * q3[j + 2]);
    P12[j] = (double)(q1[j] * q2[j + 1]);
  };
  diff(0); diff(1); diff(2); diff(3);
  window(0); window(1); window(2);
  if (WT == W_JS) products(0);

#pragma unroll
  for (int r = 0; r < M; r++) {
    const int i = s + r;
    if (r + 4 < M + 4) diff(r + 4);
    window(r + 3);
    if (WT == W_JS) products(r + 1);
#pragma unroll
    for (int q = 0; q < 2; q++) {
      double Ar, Br, Cr, Rr;
      if (WT == W_JS) {
        // rows at 15x: weights (X1, H, 3/2 X3) = 5 (w1, w2, w3), the 3x rows
        // and right-hand side of the general branch times 5
        const double X1 = q == 0 ? P23[r] : P12[r + 1];
        const double Hr = q == 0 ? H13[r] : H13[r + 1];
        const double X3 = q == 0 ? P12[r] : P23[r + 1];
        const double hi = 1.5 * X3, lo = fma(2.0, X1, Hr);
        Br = fma(3.0, X3, fma(2.0, Hr, X1));
        Ar = q == 0 ? lo : hi;
        Cr = q == 0 ? hi : lo;
        Rr = q == 0 ? X1 * qq[r + 1] + Hr * pp[r + 2] + hi * qq[r + 2]
                    : X1 * pp[r + 3] + Hr * qq[r + 2] + hi * pp[r + 2];
      } else {
        R v1, v2, v3, tau = R(0);
        if (q == 0) {
          if (WT == W_BORGES) tau = fabs(b3[r + 2] - b1[r]);
          if (WT == W_YC) { const R t4 = dw[r] - R(2) * dw[r + 1] + dw[r + 2]; tau = R(4) * t4 * t4; }
          crw_weights<WT, R>(b1[r], b2[r + 1], b3[r + 2], tau, eps, v1, v2, v3);
        } else {
          if (WT == W_BORGES) tau = fabs(b1[r + 1] - b3[r + 3]);
          if (WT == W_YC) { const R t4 = dw[r + 1] - R(2) * dw[r + 2] + dw[r + 3]; tau = R(4) * t4 * t4; }
          crw_weights<WT, R>(b3[r + 3], b2[r + 2], b1[r + 1], tau, eps, v1, v2, v3);
        }
        const double w1 = v1, w2 = v2, w3 = v3;
        // rows at 3x: (2 w1 + w2, w1 + 2 w2 + 2 w3, w3) and 3x the
        // right-hand side (pp, qq above)
        const double lo = 2.0 * w1 + w2, hi = w3;
        Br = w1 + 2.0 * (w2 + w3);
        Ar = q == 0 ? lo : hi;
        Cr = q == 0 ? hi : lo;
        Rr = q == 0 ? w1 * qq[r + 1] + w2 * pp[r + 2] + w3 * qq[r + 2]
                    : w1 * pp[r + 3] + w2 * qq[r + 2] + w3 * pp[r + 2];
      }
      if (!FULL) {
        if (i > N - 1) { Ar = 0.0; Br = 1.0; Cr = 0.0; Rr = 0.0; }
        if (i == N - 1) { Rr -= Cr * xN[q]; Cr = 0.0; }
      }
      if (r == 0 && s == 1) { Rr -= Ar * x0[q]; Ar = 0.0; }   // row 1: the line's first separator
      const double A = Ar, B = Br, C = Cr, Rv = Rr;
      if (r == 0) { As[q] = A; Bs[q] = B; Cs[q] = C; Rs[q] = Rv; continue; }
      // rows scaled to a unit diagonal: x_r + cg_r x_{r+1} = rh_r - al_r X_s
      const double be = r == 1 ? B : B - A * cg[q][r - 1];
      bad |= (be == 0.0);
      const double rb = rcp_nr(be);
      const double ta = A * rb;
      cg[q][r] = C * rb;
      if (r == 1) { al[q][1] = ta; rh[q][1] = Rv * rb; }
      else { al[q][r] = -(ta * al[q][r - 1]); rh[q][r] = Rv * rb - ta * rh[q][r - 1]; }
    }
  }
  // upward elimination: x_{s+r} = rh_r - al_r X_s - cg_r X_{s+M}
#pragma unroll
  for (int q = 0; q < 2; q++) {
#pragma unroll
    for (int r = M - 2; r >= 1; r--) {
      const double g = cg[q][r];
      al[q][r] -= g * al[q][r + 1];
      rh[q][r] -= g * rh[q][r + 1];
      cg[q][r] = -(g * cg[q][r + 1]);
    }
  }
}

// Parallel cyclic reduction of the CTA's unit-diagonal separator rows
// a X_{k-1} + X_k + c X_{k+1} = d, both biases (rows in pcA: NC columns a, c,
// d, ... of Pt double2, two buffers; the first row's a and the last row's c
// are zero).  Row k has a = 0 when k < dl (no row k - dl) and c = 0 when k +
// dl >= Pt, and each step keeps these zeros exactly (0 x finite = 0), so the
// neighbour index is clamped into the line and the clamped row's finite
// values are multiplied by those zeros: no predicated loads, no zero fill.
// The columns beyond the third (right-hand sides of unknowns outside the CTA)
// are reduced as d is.
//
// The couplings between separators 2^l chunks apart decay with the distance
// (by 0.55^(8 2^l) and faster where the weights are near their optimal
// values), so from the third level on the CTA votes in the barrier it needs
// anyway and stops once every coupling is below 2^-100 of its diagonal: the
// terms left out are under 1e-30 of a neighbour's value.  Smooth lines stop
// after four levels of eight at 2048 points; lines whose couplings do not
// decay run them all.
template <int NC>
__device__ __forceinline__ void crw_pcr(double2* pcA, int Pt, int k, double (&a)[2], double (&c)[2],
                                        double (&d)[NC - 2][2]) {
  auto small = [](double x) {   // |x| < 2^-100; false for NaN
    return (unsigned)(__double2hiint(x) & 0x7fffffff) < 0x39b00000u;
  };
  int buf = 0;
  for (int dl = 1; dl < Pt; dl <<= 1) {
    const double2* cur = pcA + buf * NC * Pt;
    double2* nxt = pcA + (buf ^ 1) * NC * Pt + k;
    const double2* lo = cur + (k >= dl ? k - dl : k);
    const double2* hi = cur + (k + dl < Pt ? k + dl : k);
    const double2 am = lo[0], cm = lo[Pt], ap = hi[0], cp = hi[Pt];
    double2 dm[NC - 2], dp[NC - 2];
#pragma unroll
    for (int n = 0; n < NC - 2; n++) { dm[n] = lo[(2 + n) * Pt]; dp[n] = hi[(2 + n) * Pt]; }
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const double amq = q ? am.y : am.x, cmq = q ? cm.y : cm.x, apq = q ? ap.y : ap.x, cpq = q ? cp.y : cp.x;
      const double bn = 1.0 - a[q] * cmq - c[q] * apq;
      const double rb = rcp_nr(bn);
      const double an = -(a[q] * amq) * rb, cn = -(c[q] * cpq) * rb;
#pragma unroll
      for (int n = 0; n < NC - 2; n++)
        d[n][q] = (d[n][q] - a[q] * (q ? dm[n].y : dm[n].x) - c[q] * (q ? dp[n].y : dp[n].x)) * rb;
      a[q] = an; c[q] = cn;
    }
    if (2 * dl >= Pt) break;   // the last level: nobody reads its rows
    nxt[0] = make_double2(a[0], a[1]);
    nxt[Pt] = make_double2(c[0], c[1]);
#pragma unroll
    for (int n = 0; n < NC - 2; n++) nxt[(2 + n) * Pt] = make_double2(d[n][0], d[n][1]);
    buf ^= 1;
    if (dl < 4) __syncthreads();
    else if (!__syncthreads_or(!(small(a[0]) && small(a[1]) && small(c[0]) && small(c[1])))) break;
  }
}

// One (line, component, field) of the CRWENO5 reconstruction: both biases'
// tridiagonal systems built from the cells src[-3 .. N+2] (stride st, taken
// relative to `ref`), solved, and their N + 1 interface values staged in
// shared memory: so[q * ostride + padm<M>(i)] for bias q (0 left, 1 right) and
// interface i.  Called by every thread of the CTA (Pt = blockDim.x threads,
// M rows each); returns after a barrier, with the staged values visible to
// the whole CTA.  Shared memory: pcA [2][3][Pt], tp [3][Pt], sy [Pt]
// (double2), the cells cs (padm<M> layout, Pt M + 7 doubles) and the staging
// so, which may alias cs.  Sets bad on a zero pivot.
template <int M, int WT, typename R, typename O>
__device__ __forceinline__ void line_pair_solve(const DevParams& P, const double* __restrict__ src, long long st,
                                                double ref, int N, double* cs, double2* pcA, double2* tp,
                                                double2* sy, O* so, int& bad) {
  const int Pt = blockDim.x, k = threadIdx.x, lane = k & 31;
  const int s = 1 + k * M;          // separator row (interface) of this thread
  const int kN = (N - 2) / M;       // thread owning row N-1
  const R eps = R(4) * (R)P.eps;    // with the smoothness indicators at 4x
  // cells -3 .. N+2 of the line (coalesced for x lines), zero past the last
  // cell any thread reads: all of a thread's loads are issued before the
  // first store (at most M + 1 of them: Pt M + 7 cells over Pt threads)
  {
    const int ncell = Pt * M + 7;
    const double* p = src + (k - 3) * st;
    double cv[M + 1];
#pragma unroll
    for (int it = 0; it <= M; it++) {
      cv[it] = k + it * Pt < N + 6 ? *p - ref : 0.0;
      p += Pt * st;
    }
    double* o = cs + padm<M>(k);
    const int ostep = Pt + Pt / M;   // Pt is a multiple of M
#pragma unroll
    for (int it = 0; it <= M; it++) {
      if (it < M || k + it * Pt < ncell) *o = cv[it];
      o += ostep;
    }
  }
  __syncthreads();
  double x0[2] = {0.0, 0.0}, xN[2] = {0.0, 0.0};
  const int w0 = k - lane;
  if (w0 == 0 || w0 == (kN & ~31)) crw_edges<M, WT, R>(P, cs, w0 == 0 ? 0 : N, w0 == (kN & ~31) ? N : 0, x0, xN);

  double As[2], Bs[2], Cs[2], Rs[2];
  double al[2][M], cg[2][M], rh[2][M];
  // warp-uniform: every chunk of this warp inside rows [1, N-2]
  if ((w0 + 32) * M <= N - 2)
    crw_chunk<M, WT, true, R>(cs, k, s, N, x0, xN, eps, As, Bs, Cs, Rs, al, cg, rh, bad);
  else
    crw_chunk<M, WT, false, R>(cs, k, s, N, x0, xN, eps, As, Bs, Cs, Rs, al, cg, rh, bad);
  tp[k] = make_double2(al[0][M - 1], al[1][M - 1]);
  tp[Pt + k] = make_double2(cg[0][M - 1], cg[1][M - 1]);
  tp[2 * Pt + k] = make_double2(rh[0][M - 1], rh[1][M - 1]);
  __syncthreads();

  // separator equations As x_{s-1} + Bs X_k + Cs x_{s+1} = Rs, with x_{s-1}
  // from the previous chunk's last row and x_{s+1} from row 1, scaled to a
  // unit diagonal: a X_{k-1} + X_k + c X_{k+1} = d
  double a[2], cq[2], d[1][2];
  {
    double2 alp = make_double2(0.0, 0.0), gap = alp, rhp = alp;
    if (k > 0) { alp = tp[k - 1]; gap = tp[Pt + k - 1]; rhp = tp[2 * Pt + k - 1]; }
    const double alq[2] = {alp.x, alp.y}, gaq[2] = {gap.x, gap.y}, rhq[2] = {rhp.x, rhp.y};
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const double b = Bs[q] - As[q] * gaq[q] - Cs[q] * al[q][1];
      bad |= (b == 0.0);
      const double rb = rcp_nr(b);
      a[q] = -(As[q] * alq[q]) * rb;
      cq[q] = -(Cs[q] * cg[q][1]) * rb;
      d[0][q] = (Rs[q] - As[q] * rhq[q] - Cs[q] * rh[q][1]) * rb;
    }
  }
  pcA[k] = make_double2(a[0], a[1]);
  pcA[Pt + k] = make_double2(cq[0], cq[1]);
  pcA[2 * Pt + k] = make_double2(d[0][0], d[0][1]);
  __syncthreads();

  crw_pcr<3>(pcA, Pt, k, a, cq, d);
  sy[k] = make_double2(d[0][0], d[0][1]);
  __syncthreads();

  // recover every row into the output staging (the cells are dead by now);
  // the last row's coefficients come back from tp, which frees their
  // registers across the reduction
  const double2 xn = k + 1 < Pt ? sy[k + 1] : make_double2(0.0, 0.0);
  {
    const double2 l0 = tp[k], l1 = tp[Pt + k], l2 = tp[2 * Pt + k];
    al[0][M - 1] = l0.x; al[1][M - 1] = l0.y;
    cg[0][M - 1] = l1.x; cg[1][M - 1] = l1.y;
    rh[0][M - 1] = l2.x; rh[1][M - 1] = l2.y;
  }
  const int ostride = padm<M>(N) + 1;
  const bool whole = s + M - 1 <= N - 1;   // every row of the chunk lies in the line
#pragma unroll
  for (int q = 0; q < 2; q++) {
    const double Xk = d[0][q], Xn = q == 0 ? xn.x : xn.y;
    O* o = so + q * ostride + k * (M + 1);   // row s + r at padm<M>(1 + r)
    if (whole) {
      o[padm<M>(1)] = (O)Xk;
#pragma unroll
      for (int r = 1; r < M; r++) o[padm<M>(1 + r)] = (O)(rh[q][r] - al[q][r] * Xk - cg[q][r] * Xn);
    } else {
      if (s <= N - 1) o[padm<M>(1)] = (O)Xk;
#pragma unroll
      for (int r = 1; r < M; r++)
        if (s + r <= N - 1) o[padm<M>(1 + r)] = (O)(rh[q][r] - al[q][r] * Xk - cg[q][r] * Xn);
    }
    if (k == 0) so[q * ostride] = (O)x0[q];
    if (k == kN) so[q * ostride + padm<M>(N)] = (O)xN[q];
  }
  __syncthreads();
}

}  // namespace piafs
