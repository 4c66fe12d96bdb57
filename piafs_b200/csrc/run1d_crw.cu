// Whole time steps (or one right-hand side) of a 1D Euler line with CRWENO5 in
// one launch (sm_100a): the counterpart of run1d.cu for the compact scheme
// (Interp1PrimFifthOrderCRWENO on components, FP64).
//
// The line is cut over the CTAs of a cluster, Pt chunks of eight rows each, and
// a CTA solves its part of all six systems (three variables, u and f, both
// biases together), Pt threads a system, by the substructuring of the segment
// kernel (crweno_line.cu): rows and chunk elimination in registers, the
// separators by parallel cyclic reduction with the two unknowns outside the
// CTA as extra columns, and the cluster's first and last separators coupled at
// the end.  Per stage three cluster barriers (the neighbour's last chunk row;
// the first and last separators; the stage's state).  What bounds a stage is
// the latency of this chain, not its work.
// Measured (B200): a step of a 6001-point line with the Yamaleev-Carpenter weights
// and LLF takes 43 us in 12 CTAs of two warps a system; kernel by kernel 58 us
// (the segment solve alone is 13 of a stage's 19).
#include <cooperative_groups.h>

#include "crweno_solve.cuh"
#include "run1d.cuh"

namespace cg = cooperative_groups;

namespace piafs {

namespace {

using namespace line1d;

constexpr int M = 8, NS6 = 2 * NV, MAXC = 16;

// Layout of a CTA's shared memory, in doubles, for Pt threads a system
struct Layout {
  int rows;        // rows of the CTA
  int pS, pP, pR;  // strides: staged cells, plain per-cell values, interface values
  int S0, S1, cf, pr, ub, kd, fi, pc, tp, sy, bnd, ga, total;
  __host__ __device__ Layout(int Pt, int ns) {
    rows = Pt * M;
    pS = padm<M>(rows + 7) + 1;
    pP = rows + 8;
    pR = padm<M>(rows + 2) + 1;
    int o = 0;
    auto take = [&](int n) { const int at = o; o += (n + 1) & ~1; return at; };
    S0 = take(NV * pS); S1 = take(NV * pS); cf = take(NV * pS);
    pr = take(NV * pP); ub = take(NV * pP); kd = take((ns - 1) * NV * pP); fi = take(NV * pP);
    const int pcr = NS6 * 20 * Pt, rec = 4 * NV * pR;   // the values overlay the reduction's rows
    pc = take(pcr > rec ? pcr : rec);
    tp = take(NS6 * 6 * Pt); sy = take(NS6 * 2 * Pt); bnd = take(NS6 * 16); ga = take(NS6 * 12 * MAXC);
    total = o;
  }
};

template <int WT>
__global__ void __launch_bounds__(NS6 * 64, 1) k_run1d_crw(DevParams P, Run1D R, int Pt) {
  extern __shared__ __align__(16) double sm[];
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank(), C = (int)cl.num_blocks();
  const int N = P.N0, tid = threadIdx.x, nt = blockDim.x, ns = R.nstages;
  const Layout L(Pt, ns);
  const int rb = rank * L.rows;                                // rows and cells before the segment
  const bool lastc = rank == C - 1;
  const int n = lastc ? N - rb : L.rows;                       // its cells
  double* cf = sm + L.cf;                                      // staged cell fluxes
  double* pr = sm + L.pr;                                      // velocity, enthalpy, root of the density
  double* ub = sm + L.ub;
  double* kd = sm + L.kd;
  double* fi = sm + L.fi;
  double* rec = sm + L.pc;                                     // [uL uR fL fR][variable][interface - rb]
  const double g = P.gamma;
  const int sys = tid / Pt, k = tid - sys * Pt, lane = tid & 31;
  const int fld = sys >= NV, var = sys - NV * fld;
  double2* pcA = (double2*)(sm + L.pc) + sys * 10 * Pt;
  double2* tp = (double2*)(sm + L.tp) + sys * 3 * Pt;
  double2* sy = (double2*)(sm + L.sy) + sys * Pt;
  double2* bnd = (double2*)(sm + L.bnd) + sys * 8;
  double2* gath = (double2*)(sm + L.ga) + sys * 6 * MAXC;
  const int K = rank * Pt + k, s = 1 + K * M, kN = (N - 2) / M, Kw = K - lane;
  const double eps = 4.0 * P.eps;
  int bad = 0;
  auto at = [&](int i, int m) -> double* {
    return R.rhs ? R.u + (long long)(i + 3) * NV + m : R.u + m * P.ps + pidx(P, i, 0);
  };
  // staged cells past the line stay zero
  for (int e = tid; e < L.pr; e += nt) sm[e] = 0.0;
  __syncthreads();
  for (int c = tid; c < n; c += nt) {
    double u[NV];
#pragma unroll
    for (int m = 0; m < NV; m++) u[m] = *at(rb + c, m);
#pragma unroll
    for (int m = 0; m < NV; m++) { ub[m * L.pP + c] = u[m]; sm[L.S0 + m * L.pS + padm<M>(3 + c)] = u[m]; }
    cell_terms(u, g, cf + padm<M>(3 + c), L.pS, pr + 3 + c, L.pP);
  }
  // the cells beside the segment (as in run1d.cu), threads 0 .. 5
  const int side = tid >= 3, k3 = tid - 3 * side, hc = side ? n + 3 + k3 : k3;
  const bool end = side ? lastc : rank == 0;
  const int type = tid < 6 && end ? R.face[side].type : BC_PERIODIC;
  const int from = side ? (rank + 1) % C : (rank + C - 1) % C;
  const int nf = from == C - 1 ? N - from * L.rows : L.rows;
  const int src = padm<M>(side ? k3 + 3 : nf + k3);
  if (tid < 6) {
#pragma unroll
    for (int m = 0; m < NV; m++)
      sm[L.S0 + m * L.pS + padm<M>(hc)] = sm[L.S1 + m * L.pS + padm<M>(hc)] = *at(side ? N + k3 : k3 - 3, m);
  }
  cl.sync();
  int cur = 0;
  for (int step = 0; step < R.nsteps; step++) {
    for (int st = 0; st < ns; st++) {
      double* S = sm + (cur ? L.S1 : L.S0);
      double* Sn = sm + (cur ? L.S0 : L.S1);
      if (tid < 6) {
        double v[NV];
        if (!end || type == BC_PERIODIC) {
          const double* rs = cl.map_shared_rank(S, from) + src;
#pragma unroll
          for (int m = 0; m < NV; m++) v[m] = rs[m * L.pS];
        } else if (type >= 0) {
          double w[NV];
#pragma unroll
          for (int m = 0; m < NV; m++) w[m] = S[m * L.pS + padm<M>(3 + (side ? n - 1 - k3 : 2 - k3))];
          face_state(P, R.face[side], w, v);
        } else {
#pragma unroll
          for (int m = 0; m < NV; m++) v[m] = S[m * L.pS + padm<M>(hc)];
        }
#pragma unroll
        for (int m = 0; m < NV; m++) S[m * L.pS + padm<M>(hc)] = v[m];
        cell_terms(v, g, cf + padm<M>(hc), L.pS, pr + hc, L.pP);
        // u comes back with the ghosts of the last step's first stage
        if (end && st == 0 && step == R.nsteps - 1)
          for (int m = 0; m < NV; m++) *at(side ? N + k3 : k3 - 3, m) = v[m];
      }
      __syncthreads();

      // rows and their elimination (crw_chunk), this thread's chunk of its system
      const double* cs = fld ? cf + var * L.pS : S + var * L.pS;
      double x0[2] = {0.0, 0.0}, xN[2] = {0.0, 0.0};
      const bool hasN = Kw == kN - (kN & 31);
      if (Kw == 0 || hasN) crw_edges<M, WT, double>(P, cs, Kw == 0 ? 0 : N - rb, hasN ? N - rb : 0, x0, xN);
      double As[2], Bs[2], Cs[2], Rs[2];
      double al[2][M], cgm[2][M], rh[2][M];
      if ((Kw + 32) * M <= N - 2)
        crw_chunk<M, WT, true, double>(cs, k, s, N, x0, xN, eps, As, Bs, Cs, Rs, al, cgm, rh, bad);
      else
        crw_chunk<M, WT, false, double>(cs, k, s, N, x0, xN, eps, As, Bs, Cs, Rs, al, cgm, rh, bad);
      tp[k] = make_double2(al[0][M - 1], al[1][M - 1]);
      tp[Pt + k] = make_double2(cgm[0][M - 1], cgm[1][M - 1]);
      tp[2 * Pt + k] = make_double2(rh[0][M - 1], rh[1][M - 1]);
      cl.sync();   // the previous CTA's last chunk row is read below

      // separator equations with the outside unknowns' columns e, f
      double a[2], cq[2], x[3][2];
      double2 alp = make_double2(0.0, 0.0), gap = alp, rhp = alp;
      if (k > 0) {
        alp = tp[k - 1]; gap = tp[Pt + k - 1]; rhp = tp[2 * Pt + k - 1];
      } else if (rank > 0) {
        const double2* rt = cl.map_shared_rank(tp, rank - 1);
        alp = rt[Pt - 1]; gap = rt[2 * Pt - 1]; rhp = rt[3 * Pt - 1];
      }
      const double alq[2] = {alp.x, alp.y}, gaq[2] = {gap.x, gap.y}, rhq[2] = {rhp.x, rhp.y};
#pragma unroll
      for (int q = 0; q < 2; q++) {
        const double b = Bs[q] - As[q] * gaq[q] - Cs[q] * al[q][1];
        bad |= (b == 0.0);
        const double rbq = rcp_nr(b);
        a[q] = -(As[q] * alq[q]) * rbq;
        cq[q] = -(Cs[q] * cgm[q][1]) * rbq;
        x[0][q] = (Rs[q] - As[q] * rhq[q] - Cs[q] * rh[q][1]) * rbq;
        x[1][q] = 0.0;
        x[2][q] = 0.0;
        if (k == 0) { x[1][q] = a[q]; a[q] = 0.0; }
        if (k == Pt - 1) { x[2][q] = cq[q]; cq[q] = 0.0; }
      }
      pcA[k] = make_double2(a[0], a[1]);
      pcA[Pt + k] = make_double2(cq[0], cq[1]);
#pragma unroll
      for (int c = 0; c < 3; c++) pcA[(2 + c) * Pt + k] = make_double2(x[c][0], x[c][1]);
      __syncthreads();
      crw_pcr<5>(pcA, Pt, k, a, cq, x);
      // X_k = d_k - e_k L - f_k R, L and R the separators beside the CTA
      if (k == 0 || k == Pt - 1) {
        double2* b = bnd + (k == 0 ? 0 : 3);
#pragma unroll
        for (int c = 0; c < 3; c++) b[c] = make_double2(x[c][0], x[c][1]);
      }
      cl.sync();
      for (int e = k; e < 6 * C; e += Pt) gath[e] = cl.map_shared_rank(bnd, e / 6)[e % 6];
      __syncthreads();
      // L = last separator of CTA rank - 1, R = first of CTA rank + 1, from
      //   F_c = d0 - e0 G_{c-1} - f0 F_{c+1},  G_c = dl - el G_{c-1} - fl F_{c+1}
      // A segment's first separator does not feel the unknown beyond its last
      // one, nor the other way round, once the couplings have decayed below
      // 2^-100 over it: the two unknowns either side of a boundary then form a
      // system of their own.  Otherwise the recurrence over all CTAs.
      if (k < 2) {
        const int q = k;
        double* G = (double*)gath;
        auto at6 = [&](int c, int w) -> double& { return G[12 * c + 2 * w + q]; };   // d0 e0 f0 dl el fl
        auto tiny = [](double v) { return (unsigned)(__double2hiint(v) & 0x7fffffff) < 0x39b00000u; };
        bool near = true;
        for (int c = max(rank - 1, 0); c <= min(rank + 1, C - 1); c++) near = near && tiny(at6(c, 2)) && tiny(at6(c, 4));
        double Lv = 0.0, Rv = 0.0;
        if (near) {
          if (rank > 0) {
            const double den = 1.0 - at6(rank - 1, 5) * at6(rank, 1);
            bad |= (den == 0.0);
            Lv = (at6(rank - 1, 3) - at6(rank - 1, 5) * at6(rank, 0)) * rcp_nr(den);
          }
          if (rank < C - 1) {
            const double den = 1.0 - at6(rank, 5) * at6(rank + 1, 1);
            bad |= (den == 0.0);
            Rv = (at6(rank + 1, 0) - at6(rank + 1, 1) * at6(rank, 3)) * rcp_nr(den);
          }
        } else {
          // forward: G_c = al + be F_{c+1}, F_c = ga + de F_{c+1} (kept in place of
          // d0, e0, f0, dl); backward from F_C = 0
          double ap = 0.0, bp = 0.0;
          for (int c = 0; c < C; c++) {
            const double d0 = at6(c, 0), e0 = at6(c, 1), f0 = at6(c, 2), dl = at6(c, 3), el = at6(c, 4), fl = at6(c, 5);
            const double den = 1.0 + e0 * bp;
            bad |= (den == 0.0);
            const double rd = rcp_nr(den);
            const double ga = (d0 - e0 * ap) * rd, de = -f0 * rd;
            const double an = dl - el * (ap + bp * ga), bn = -(el * bp * de + fl);
            at6(c, 0) = ga; at6(c, 1) = de; at6(c, 2) = an; at6(c, 3) = bn;
            ap = an; bp = bn;
          }
          double Fn = 0.0;
          for (int c = C - 1; c >= 0; c--) {
            const double F = at6(c, 0) + at6(c, 1) * Fn;
            if (c == rank + 1) Rv = F;
            if (c == rank - 1) Lv = at6(c, 2) + at6(c, 3) * Fn;
            Fn = F;
          }
        }
        ((double*)(bnd + 6))[q] = Lv;
        ((double*)(bnd + 7))[q] = Rv;
      }
      __syncthreads();
      const double2 Lv = bnd[6], Rv = bnd[7];
      const double Lq[2] = {Lv.x, Lv.y}, Rq[2] = {Rv.x, Rv.y};
      double X[2];
#pragma unroll
      for (int q = 0; q < 2; q++) X[q] = x[0][q] - x[1][q] * Lq[q] - x[2][q] * Rq[q];
      sy[k] = make_double2(X[0], X[1]);
      __syncthreads();
      // every row's value; interface rb from the previous CTA's last chunk row
      const double2 xn = k + 1 < Pt ? sy[k + 1] : Rv;
#pragma unroll
      for (int q = 0; q < 2; q++) {
        double* o = rec + ((2 * fld + q) * NV + var) * L.pR;
        double* w = o + k * (M + 1);
        const double Xn = q == 0 ? xn.x : xn.y;
        if (s <= N - 1) w[padm<M>(1)] = X[q];
#pragma unroll
        for (int r = 1; r < M; r++)
          if (s + r <= N - 1) w[padm<M>(1 + r)] = rh[q][r] - al[q][r] * X[q] - cgm[q][r] * Xn;
        if (k == 0) o[0] = rank == 0 ? x0[q] : rhq[q] - alq[q] * Lq[q] - gaq[q] * X[q];
        if (K == kN) o[padm<M>(N - rb)] = xN[q];
      }
      __syncthreads();

      for (int i = tid; i < n + 1; i += nt) {
        double a4[4], b4[4], c4[4], d4[4], fo[4];
        const int q = padm<M>(i);
#pragma unroll
        for (int m = 0; m < NV; m++) {
          a4[m] = rec[m * L.pR + q]; b4[m] = rec[(NV + m) * L.pR + q];
          c4[m] = rec[(2 * NV + m) * L.pR + q]; d4[m] = rec[(3 * NV + m) * L.pR + q];
        }
        const double *pl = pr + i + 2, *ul = S + padm<M>(i + 2), *ur = S + padm<M>(i + 3);
        switch (P.upwind) {
          case UPW_ROE: iface_flux<UPW_ROE>(a4, b4, c4, d4, pl, pl + 1, L.pP, ul, ur, L.pS, g, fo); break;
          case UPW_RF: iface_flux<UPW_RF>(a4, b4, c4, d4, pl, pl + 1, L.pP, ul, ur, L.pS, g, fo); break;
          case UPW_LLF: iface_flux<UPW_LLF>(a4, b4, c4, d4, pl, pl + 1, L.pP, ul, ur, L.pS, g, fo); break;
          default: iface_flux<UPW_RUSANOV>(a4, b4, c4, d4, pl, pl + 1, L.pP, ul, ur, L.pS, g, fo); break;
        }
#pragma unroll
        for (int m = 0; m < NV; m++) fi[m * L.pP + i] = fo[m];
      }
      __syncthreads();
      if (R.rhs) {                 // the right-hand side alone, zero at the ghosts
        for (int i = tid; i < n; i += nt) {
          const double dxi = R.dxinv[P.ghosts + rb + i];
#pragma unroll
          for (int m = 0; m < NV; m++)
            R.rhs[(long long)(rb + i + 3) * NV + m] = -(dxi * (fi[m * L.pP + i + 1] - fi[m * L.pP + i]));
        }
        if (tid < 3 * NV && rank == 0) R.rhs[tid] = 0.0;
        if (tid < 3 * NV && lastc) R.rhs[(long long)(N + 3) * NV + tid] = 0.0;
        if (bad) atomicOr(R.err, 1);
        cl.sync();                 // the others have read this segment
        return;
      }
      const bool last = st == ns - 1;
      const double* co = last ? R.b : R.a + (st + 1) * MAX_STAGES;
      for (int i = tid; i < n; i += nt) {
        const double dxi = R.dxinv[P.ghosts + rb + i];
        double y[NV];
#pragma unroll
        for (int m = 0; m < NV; m++) {
          const double kk = -(dxi * (fi[m * L.pP + i + 1] - fi[m * L.pP + i]));
          y[m] = ub[m * L.pP + i];
          for (int j = 0; j < st; j++) y[m] = fma_rn(co[j], kd[(j * NV + m) * L.pP + i], y[m]);
          y[m] = fma_rn(co[st], kk, y[m]);
          if (last) ub[m * L.pP + i] = y[m];
          else kd[(st * NV + m) * L.pP + i] = kk;
          Sn[m * L.pS + padm<M>(3 + i)] = y[m];
        }
        cell_terms(y, g, cf + padm<M>(3 + i), L.pS, pr + 3 + i, L.pP);
      }
      // the neighbours read Sn, and tp and bnd are written again, only after
      // this barrier
      cl.sync();
      cur ^= 1;
    }
  }
  if (bad) atomicOr(R.err, 1);
  for (int i = tid; i < n; i += nt)
    for (int m = 0; m < NV; m++) *at(rb + i, m) = ub[m * L.pP + i];
  if (rank == 0 && tid == 0) {
    double t = *R.tdev;
    for (int q = 0; q < R.nsteps; q++) t += P.dt;
    *R.tdev = t;
  }
}

template <int WT>
cudaError_t run_wt(const DevParams& P, const Run1D& R, int C, int Pt, cudaStream_t s, bool probe) {
  const int bytes = Layout(Pt, R.nstages).total * (int)sizeof(double);
  cudaError_t e = cudaFuncSetAttribute(k_run1d_crw<WT>, cudaFuncAttributeMaxDynamicSharedMemorySize, kRun1DCrwSmem);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_run1d_crw<WT>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)C, 1, 1);
  cfg.blockDim = dim3((unsigned)(NS6 * Pt), 1, 1);
  cfg.dynamicSmemBytes = (size_t)bytes;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)C;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (probe) {
    int clusters = 0;
    e = cudaOccupancyMaxActiveClusters(&clusters, k_run1d_crw<WT>, &cfg);
    return e != cudaSuccess ? e : clusters > 0 ? cudaSuccess : cudaErrorInvalidConfiguration;
  }
  return cudaLaunchKernelEx(&cfg, k_run1d_crw<WT>, P, R, Pt);
}

cudaError_t run_any(const DevParams& P, const Run1D& R, int C, int Pt, cudaStream_t s, bool probe) {
  if (P.no_limiting) return run_wt<WT_NOLIM>(P, R, C, Pt, s, probe);
  switch (P.weno_type) {
    case W_MAPPED: return run_wt<W_MAPPED>(P, R, C, Pt, s, probe);
    case W_BORGES: return run_wt<W_BORGES>(P, R, C, Pt, s, probe);
    case W_YC: return run_wt<W_YC>(P, R, C, Pt, s, probe);
    default: return run_wt<W_JS>(P, R, C, Pt, s, probe);
  }
}

}  // namespace

// Threads a system: a warp (256 rows a CTA) while a cluster of 16 covers the
// line so, which keeps a CTA's chains short, else two.
int run1d_crw_threads(int N) { return (N - 1 + M - 1) / M <= 32 * MAXC ? 32 : 64; }

// CTAs of a line, 0 if it is not one of those: at most 16 CTAs, and three cells
// or more in the last (a neighbour's and the boundary's sources)
int run1d_crw_ctas(const DevParams& P, const Run1D& R) {
  const int N = P.N0, Pt = run1d_crw_threads(N), chunks = (N - 1 + M - 1) / M, C = (chunks + Pt - 1) / Pt;
  if (N < 16 || C > MAXC || N - (C - 1) * Pt * M < 3) return 0;
  if (Layout(Pt, R.nstages).total * (int)sizeof(double) > kRun1DCrwSmem) return 0;
  if (run_any(P, R, C, Pt, nullptr, true) != cudaSuccess) {
    cudaGetLastError();   // no such cluster to be had
    return 0;
  }
  return C;
}

cudaError_t launch_run1d_crw(const DevParams& P, const Run1D& R, int ctas, cudaStream_t s) {
  return run_any(P, R, ctas, run1d_crw_threads(P.N0), s, false);
}

}  // namespace piafs
