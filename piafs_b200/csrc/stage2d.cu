// The end of a 2D Runge-Kutta stage in one kernel (sm_100a): upwind fluxes at
// the reconstructed interfaces of a tile (NavierStokes2DUpwind.c), the
// divergence (HyperbolicFunction.c:97-112), the viscous terms
// (NavierStokes2DParabolicFunction.c:41-204 with FirstDerivativeFirstOrder),
// the photochemical source (ChemistrySolve.c:18-115) and the Runge-Kutta
// combination of the stage (TimeRK.c:60-75, :86-99).  The stage derivative and
// the next stage's state are written once each, from registers.
//
// What bounds it: HBM and its latency.  Of the interface arrays it reads 26
// values a point per direction with one chemistry layer and LLF (uL, uR,
// fL + fR of the four flow variables, uL - uR and fL + fR of the seven passive
// ones), and writes 11 (or 22).
// Separate kernels for the upwinding, the viscous terms and source, and the
// combination read and wrote the derivative three times over: at 2048^2 with 11
// variables 0.53 + 0.31 ms and 0.2 ms of combination a stage, where this takes
// 0.67 ms with the combination; a step of the 512^2 run went from 640 to 574 us,
// one of 300 x 217 points from 198 to 161 us.  Three CTAs an SM (80 registers,
// no spills) hide the loads; the 16 x 15 tile of the upwinding alone would put 16 points of
// the viscous fluxes in a second round.
#include <type_traits>

#include "kernels.h"
#include "physics.cuh"
#include "source.cuh"

namespace piafs {

namespace {

// Tile: 16 x 14 points.  With 14 rows the x interfaces (17 x 14), the y
// interfaces (16 x 15) and the points of the viscous fluxes (17 x 15) each fit
// one round of the 256 threads.
constexpr int TI = 16, TJ = 14, LX = TI + 1, LY = TJ + 1;   // LY odd: columns fall in distinct banks
constexpr int NX = LX * TJ, NY = TI * LY;
constexpr int QX = TI + 2, QY = TJ + 2, FX = TI + 1, FY = TJ + 1;

// y interfaces: in the standard layout, in the transposed one, or no
// interfaces but the y term itself (a grid decomposed along y)
enum YMode { Y_STD = 0, Y_TRANSPOSED = 1, Y_GIVEN = 2 };

// CTAs an SM: registers for two 128, three 80, four 64.  Mixed precision four
// (701 x 500: 54.9 us, 62.8 with three); FP64 three (64 registers spill: LLF at
// 2048 x 2048 takes 940 us with four, 703 with three; Roe at 300 x 217 22.1 and
// 18.4); RF's matrices in FP64 two (1201 x 777: 131.1 us, 133.3 with three).
constexpr int stage2d_ctas(int upw, bool mx) { return mx ? 4 : upw == UPW_RF ? 2 : 3; }

// The grid of tiles: rows of tiles in y, ROWS at a time in z (a launch takes 65535
// in either: grids of 917,491 rows of points and more need both).  Tiles that this
// rounds up to beyond the last row have no interface or point inside the grid.
// ROWS is a constant because the row must cost nothing: with the grid's own height
// in its place the 2048^2 launch took 0.630 ms, with this, or without z, 0.611.
constexpr int ROWS = 4096;
dim3 tile_grid(const DevParams& P) {
  const int tx = (P.N0 + TI - 1) / TI, ty = (P.N1 + TJ - 1) / TJ;
  return dim3(tx, ty < ROWS ? ty : ROWS, (ty + ROWS - 1) / ROWS);
}
__device__ __forceinline__ int tile_row() { return blockIdx.y + blockIdx.z * ROWS; }

// Threads a CTA.  Up to one tile an SM 512: x and y interfaces by different
// threads, the chemistry beside the viscous fluxes, a point's variables by two
// threads -- what counts there is the length of one thread's work (64 x 64: two
// warps a scheduler, 7 clocks an instruction).  A step, LLF with chemistry, from
// 256 to 512 threads: 16 x 16 66 -> 55 us, 64 x 64 80 -> 69, 176 x 176 (143 tiles)
// 124 -> 114; Roe, WENO5: 64 x 64 66 -> 56, 176 x 176 88 -> 78.  Past 148 tiles
// the wider CTA, of which an SM holds one (at the 64 registers of two it would
// spill), would need a second round where three of 256 threads need one.
constexpr int WIDE = 512, NARROW = 256;
// the variables of a point from which a wide CTA's second half works on
constexpr int second_half(int nv) { return nv == 11 ? 5 : 2; }

template <typename T>
constexpr size_t stage2d_smem(int nv, bool given, bool visc) {
  // interface fluxes, after velocities and temperature in the same place; the
  // viscous fluxes
  const size_t hyp = (size_t)nv * (NX + (given ? 0 : NY)) * sizeof(T), q = QX * QY * (2 * sizeof(T) + sizeof(double));
  return visc ? (3 * TJ * FX + 3 * FY * TI) * sizeof(T) + (hyp > q ? hyp : q) : hyp;
}

// Upwind flux of all components at interface q into so[m * stride]; cells pL
// / pR are the cells left and right of it in `cells`.  MX: the interface
// arrays hold floats relative to the line's reference values, whose flow
// variables are uref (absolute, FP64); the flux is computed in FP32 in
// deviation form and stored relative to the line's flux reference.  The
// schemes other than RF need only uL - uR and fL + fR besides the states of
// the Roe average (LLF: the interface states), and take them as they are
// packed by the reconstruction (P.pack_sp) or form them here.  NV: the number of
// variables, or 0 for P.nvars; where it is 4 the loop over the passive variables
// must not be there at all -- room for its loads, never issued, spilled 350 to 370
// bytes a thread (132 to 136 in mixed precision with a transposed y pass), which
// cost 0.3 to 1 % of a step at 1201 x 777 (WENO5, Rusanov 668 -> 663 us).  With 11
// a constant end saves 2 % of the launch (2048^2 0.626 -> 0.611 ms).
template <int UPW, int DIR, bool MX, int NV>
__device__ __forceinline__ void iface_upwind(const DevParams& P, const void* __restrict__ uLv,
                                             const void* __restrict__ uRv, const void* __restrict__ fLv,
                                             const void* __restrict__ fRv, long long q,
                                             const double* __restrict__ cells, long long pL, long long pR,
                                             const double* uref,
                                             typename std::conditional<MX, float, double>::type* so, int stride) {
  typedef typename std::conditional<MX, float, double>::type T;
  constexpr int NF = Flow<NS2D>::NF;
  const T* uL = (const T*)uLv + q;
  const T* uR = (const T*)uRv + q;
  const T* fL = (const T*)fLv + q;
  const T* fR = (const T*)fRv + q;
  const long long is = P.pis;
  T fi[4], spa;
  int spm;
  if (UPW == UPW_RF) {
    T a[4], b[4], c[4], d[4];
#pragma unroll
    for (int m = 0; m < NF; m++) { a[m] = uL[m * is]; b[m] = uR[m * is]; c[m] = fL[m * is]; d[m] = fR[m * is]; }
    if (MX) {
      T aL[4], aR[4];
#pragma unroll
      for (int m = 0; m < NF; m++) { const T r = (T)uref[m]; aL[m] = r + a[m]; aR[m] = r + b[m]; }
      upwind_flow_dev<NS2D, UPW, T>(a, b, c, d, aL, aR, a, b, (T)P.gamma, DIR, fi, &spa, &spm);
    } else {
      upwind_flow<NS2D, UPW, T>(a, b, c, d, a, b, (T)P.gamma, DIR, fi, &spa, &spm);
    }
  } else {
    T A[4], B[4], du[4], sf[4];   // LLF: the interface states; else the cell states
    if (UPW == UPW_LLF) {
#pragma unroll
      for (int m = 0; m < NF; m++) { A[m] = uL[m * is]; B[m] = uR[m * is]; sf[m] = fL[m * is]; }
    } else {
#pragma unroll
      for (int m = 0; m < NF; m++) {
        A[m] = (T)cells[m * P.ps + pL]; B[m] = (T)cells[m * P.ps + pR];
        du[m] = uL[m * is]; sf[m] = fL[m * is];
      }
    }
    if (!P.pack_sp) {
#pragma unroll
      for (int m = 0; m < NF; m++) {
        sf[m] += fR[m * is];
        if (UPW != UPW_LLF) du[m] -= uR[m * is];
      }
    }
    if (UPW == UPW_LLF) {
#pragma unroll
      for (int m = 0; m < NF; m++) {
        du[m] = A[m] - B[m];
        if (MX) { const T r = (T)uref[m]; A[m] = r + A[m]; B[m] = r + B[m]; }
      }
    }
    ns2d_upwind_packed<UPW, T>(A, B, du, sf, (T)P.gamma, DIR, fi, &spa, &spm);
  }
#pragma unroll
  for (int m = 0; m < NF; m++) so[m * stride] = fi[m];
  // passive variables seven at a time (a chemistry layer), their loads in flight
  // together: 0.666 ms at 2048^2 where four at a time take 0.697
  const int nv = NV ? NV : P.nvars;
  constexpr int G = 7;
  for (int m = NF; m < nv; m += G) {
    T du[G], sf[G];
    if (P.pack_sp) {
#pragma unroll
      for (int k = 0; k < G; k++)
        if (m + k < nv) { du[k] = uL[(m + k) * is]; sf[k] = fL[(m + k) * is]; }
#pragma unroll
      for (int k = 0; k < G; k++)
        if (m + k < nv) so[(m + k) * stride] = upwind_species_packed(spm, spa, du[k], sf[k]);
    } else {
      T l[G], r[G];
#pragma unroll
      for (int k = 0; k < G; k++)
        if (m + k < nv) {
          l[k] = uL[(m + k) * is]; r[k] = uR[(m + k) * is]; du[k] = fL[(m + k) * is]; sf[k] = fR[(m + k) * is];
        }
#pragma unroll
      for (int k = 0; k < G; k++)
        if (m + k < nv) so[(m + k) * stride] = upwind_species(spm, spa, l[k], r[k], du[k], sf[k]);
    }
  }
}

// NV: the number of variables when it is 11 (one chemistry layer) or 4 (none),
// 0 for any other: the registers hold the point's variables group by group.
// BT: WIDE (NV > 0 only) or NARROW threads.
template <int UPW, int YM, bool MX, int NV, int BT>
__global__ void __launch_bounds__(BT, BT == WIDE ? 1 : stage2d_ctas(UPW, MX)) k_stage2d(DevParams P, Stage2D S) {
  typedef typename std::conditional<MX, float, double>::type T;
  extern __shared__ double sfd[];
  constexpr bool GIVEN = YM == Y_GIVEN;
  const int nv = NV ? NV : P.nvars;
  const int N0 = P.N0, N1 = P.N1, g = P.ghosts;
  const long long ps = P.ps;
  const double* __restrict__ U = S.U;
  const int i0 = blockIdx.x * TI, j0 = tile_row() * TJ;
  const int tid = threadIdx.x;
  const bool visc = S.visc != 0;
  // the thread's point and, in a wide CTA, its half of the point's variables
  const int half = BT == WIDE ? tid / 256 : 0, pt = BT == WIDE ? tid % 256 : tid;
  T* sVx = (T*)sfd;                           // viscous x fluxes [3][TJ][FX]
  T* sVy = sVx + (visc ? 3 * TJ * FX : 0);    // viscous y fluxes [3][FY][TI]
  T* sx = sVy + (visc ? 3 * FY * TI : 0);     // x-interface fluxes [m][row jj][ii = 0..TI]
  T* sy = sx + nv * NX;                       // y-interface fluxes [m][column ii][jj = 0..TJ]
  // before the interface fluxes, in their place: the temperature on the tile
  // and one cell around it [QY][QX], FP64 also in mixed precision (its
  // differences are taken before they are rounded), and u, v [2][QY][QX]
  double* sT_ = (double*)sx;
  T* sQ = (T*)(sT_ + QX * QY);
  if (visc) {
    for (int e = tid; e < QX * QY; e += BT) {
      const int a = e % QX, b = e / QX;
      const int i = i0 - 1 + a, j = j0 - 1 + b;
      double uu = 0.0, vv = 0.0, TT = 0.0;
      if (i < N0 + g && j < N1 + g) {
        const long long p = pidx(P, i, j);
        double rho, e_, pr;
        ns_flowvar(U[p], U[ps + p], U[2 * ps + p], U[3 * ps + p], P.gamma, rho, uu, vv, e_, pr);
        TT = P.gamma * pr / rho;
      }
      sQ[e] = (T)uu; sQ[QX * QY + e] = (T)vv; sT_[e] = TT;
    }
    __syncthreads();
    const T two_third = T(2.0 / 3.0), inv_Re = (T)(1.0 / P.Re), inv_Pr = (T)(1.0 / P.Pr);
    const T igm1 = (T)(1.0 / (P.gamma - 1.0));
    // viscous fluxes on [i0-1, i0+TI) x [j0-1, j0+TJ) (corner cell unused)
    if (tid < FX * FY) {
      const int a = tid % FX, b = tid / FX;
      const int i = i0 - 1 + a, j = j0 - 1 + b;
      const bool need_x = (b >= 1) && (j < N1) && (i < N0);   // x fluxes at interior rows
      const bool need_y = (a >= 1) && (i < N0) && (j < N1);   // y fluxes at interior columns
      if (need_x || need_y) {
        const T* su = sQ + b * QX + a;
        const T* sv = su + QX * QY;
        const double* sT = sT_ + b * QX + a;
        const T dxi = (T)S.dxinv[g + i], dyi = (T)S.dxinv[P.W0 + g + j];
        // interior rows of the whole grid (a row slab's ghost rows inside it
        // are interior rows)
        const bool row_int = (j + P.jg0 >= 0 && j + P.jg0 < P.N1g), col_int = (i >= 0 && i < N0);
        const T uc = su[0], vc = sv[0];
        const double Tc = sT[0];
        // first differences (QDerivX on interior rows, QDerivY on interior
        // columns; zero elsewhere)
        const T ux = row_int ? dxi * (su[1] - uc) : T(0);
        const T vx = row_int ? dxi * (sv[1] - vc) : T(0);
        const T Tx = row_int ? dxi * (T)(sT[1] - Tc) : T(0);
        const T uy = col_int ? dyi * (su[QX] - uc) : T(0);
        const T vy = col_int ? dyi * (sv[QX] - vc) : T(0);
        const T Ty = col_int ? dyi * (T)(sT[QX] - Tc) : T(0);
        T mu, kappa;
        visc_coeffs<T>(P, (T)Tc, mu, kappa);
        const T mre = mu * inv_Re, kre = kappa * inv_Re * igm1 * inv_Pr;
        if (need_x) {
          const T txx = two_third * mre * (T(2) * ux - vy), txy = mre * (uy + vx);
          T* f = sVx + (b - 1) * FX + a;
          f[0] = txx; f[TJ * FX] = txy; f[2 * TJ * FX] = uc * txx + vc * txy + kre * Tx;
        }
        if (need_y) {
          const T tyx = mre * (uy + vx), tyy = two_third * mre * (-ux + T(2) * vy);
          T* f = sVy + b * TI + (a - 1);
          f[0] = tyx; f[FY * TI] = tyy; f[2 * FY * TI] = uc * tyx + vc * tyy + kre * Ty;
        }
      }
    }
  }
  // wide: the chemistry source of point pt by the second half, beside the viscous
  // fluxes; its heat release to the first half
  __shared__ double sH[BT == WIDE && NV == 11 ? TI * TJ : 1];
  T src[5], Q = T(0);
  auto chemistry = [&](int i, int j) {
    const long long p = pidx(P, i, j);
    const double t = *S.tdev + S.cstage * P.dt;
    const T n_hnu = chem_hnu0<T>(P, pulse_factor(P, t), S.imap[p]);
    if (S.hnu) S.hnu[p] = (double)n_hnu;
    const double* s = U + 4 * ps + p;
    chem_layer<T>(P, n_hnu, (T)s[0], (T)s[ps], (T)s[2 * ps], (T)s[3 * ps], (T)s[4 * ps], (T)s[5 * ps],
                  (T)s[6 * ps], src, Q);
  };
  if (BT == WIDE && NV == 11 && S.chem && half && pt < TI * TJ && i0 + pt % TI < N0 && j0 + pt / TI < N1) {
    chemistry(i0 + pt % TI, j0 + pt / TI);
    sH[pt] = (double)Q;
  }
  if (visc) __syncthreads();
  double uref[4];
  if (tid < NX) {                // (TI + 1) x TJ x interfaces
    const int ii = tid % LX, jj = tid / LX;
    const int i = i0 + ii, j = j0 + jj;
    if (i <= N0 && j < N1) {
      const long long pR = pidx(P, i, j);
      if (MX && (UPW == UPW_LLF || UPW == UPW_RF)) {
        const long long p0 = pidx(P, 0, j);
#pragma unroll
        for (int m = 0; m < 4; m++) uref[m] = U[m * ps + p0];
      }
      iface_upwind<UPW, 0, MX, NV>(P, S.xi[0], S.xi[1], S.xi[2], S.xi[3], i + (long long)(N0 + 1) * j, U, pR - 1, pR,
                               uref, sx + jj * LX + ii, NX);
    }
  }
  const int ty = BT == WIDE ? tid - 256 : tid;
  if (!GIVEN && ty >= 0 && ty < NY) {   // TI x (TJ + 1) y interfaces
    int ii, jj;
    if (YM == Y_TRANSPOSED) { jj = ty % LY; ii = ty / LY; }
    else { ii = ty % TI; jj = ty / TI; }
    const int i = i0 + ii, j = j0 + jj;
    if (j <= N1 && i < N0) {
      if (MX && (UPW == UPW_LLF || UPW == UPW_RF)) {
        const long long p0 = pidx(P, i, 0);
#pragma unroll
        for (int m = 0; m < 4; m++) uref[m] = U[m * ps + p0];
      }
      if (YM == Y_TRANSPOSED) {
        const long long pR = (long long)(j + g) + (long long)P.W1 * (i + g);
        iface_upwind<UPW, 1, MX, NV>(P, S.yi[0], S.yi[1], S.yi[2], S.yi[3], j + (long long)(N1 + 1) * i, S.UT, pR - 1,
                                 pR, uref, sy + ii * LY + jj, NY);
      } else {
        const long long pR = pidx(P, i, j);
        iface_upwind<UPW, 1, MX, NV>(P, S.yi[0], S.yi[1], S.yi[2], S.yi[3], i + (long long)N0 * j, U, pR - P.W0, pR,
                                 uref, sy + ii * LY + jj, NY);
      }
    }
  }
  __syncthreads();
  if (pt >= TI * TJ) return;
  const int ii = pt % TI, jj = pt / TI;
  const int i = i0 + ii, j = j0 + jj;
  if (i >= N0 || j >= N1) return;
  const long long p = pidx(P, i, j);
  const T dxi = (T)S.dxinv[g + i], dyi = (T)S.dxinv[P.W0 + g + j];
  // Y_GIVEN: the y term of column i comes from the slab that owns it, as
  // hy[((i / n0) nvars + m) N1 + j) n0 + i % n0] (k_slab_upwind_y)
  const T* hyv = (const T*)S.hy;
  const long long hbase =
      GIVEN ? (long long)(i / S.n0) * nv * N1 * S.n0 + (long long)j * S.n0 + i % S.n0 : 0;
  // hyp = dxinv_x dfx + dxinv_y dfy as dxinv_x dfx fused onto the rounded y
  // term, whether the y term is given or formed here
  auto hyp = [&](int m) -> double {
    const T* ax = sx + m * NX + jj * LX + ii;
    const T dfx = ax[1] - ax[0];
    const T hy = GIVEN ? hyv[hbase + (long long)m * N1 * S.n0]
                       : mul_rn(dyi, sy[m * NY + ii * LY + jj + 1] - sy[m * NY + ii * LY + jj]);
    return (double)fma_rn(dxi, dfx, hy);
  };
  auto par = [&](int m) -> double {      // viscous term of momentum / energy m = 1 .. 3
    const T* vx = sVx + (m - 1) * TJ * FX + jj * FX + ii;
    const T* vy = sVy + (m - 1) * FY * TI + jj * TI + ii;
    return (double)fma_rn(dxi, vx[1] - vx[0], mul_rn(dyi, vy[TI] - vy[0]));
  };
  if (BT == NARROW && NV == 11 && S.chem) chemistry(i, j);
  if (BT == WIDE && NV == 11 && S.chem && !half) Q = (T)sH[pt];
  // the stage derivative of variable m
  auto deriv = [&](int m) -> double {
    double k = S.neg ? -hyp(m) : hyp(m);
    if (visc && m >= 1 && m <= 3) k += par(m);
    if (NV == 11 && S.chem) {
      if (m == 3) k += (double)Q;
      if (m >= 5 && m < 10) k += (double)src[m - 5];
    }
    return k;
  };
  if constexpr (NV > 0) {
    // groups of variables: the loads of the earlier stages' part of the
    // combination in flight together, then the derivatives, then the stores
    constexpr int NG = 4;
    auto group = [&](int m0, int end) {
      double xa[NG];
      if (S.dst) {
#pragma unroll
        for (int w = 0; w < NG; w++)
          if (m0 + w < end) xa[w] = S.u[(m0 + w) * ps + p];
        for (int q = 0; q < S.nprev; q++) {
          const double a = S.a[q];
          const double* d = S.d[q] + p;
          double t[NG];
#pragma unroll
          for (int w = 0; w < NG; w++)
            if (m0 + w < end) t[w] = d[(m0 + w) * ps];
#pragma unroll
          for (int w = 0; w < NG; w++)
            if (m0 + w < end) xa[w] = fma_rn(a, t[w], xa[w]);
        }
      }
#pragma unroll
      for (int w = 0; w < NG; w++)
        if (m0 + w < end) {
          const int m = m0 + w;
          const double k = deriv(m);
          if (S.k) S.k[m * ps + p] = k;
          if (S.dst) S.dst[m * ps + p] = fma_rn(S.as, k, xa[w]);
        }
    };
    if (BT == WIDE) {
      constexpr int MH = second_half(NV);
      if (half) {
#pragma unroll
        for (int m0 = MH; m0 < NV; m0 += NG) group(m0, NV);
      } else {
#pragma unroll
        for (int m0 = 0; m0 < MH; m0 += NG) group(m0, MH);
      }
    } else {
#pragma unroll
      for (int m0 = 0; m0 < NV; m0 += NG) group(m0, NV);
    }
  } else {
    // any number of layers: the derivative through memory
    for (int m = 0; m < nv; m++) S.k[m * ps + p] = deriv(m);
    if (S.chem) {
      const double t = *S.tdev + S.cstage * P.dt;
      chem_source_point<T>(P, U, p, pulse_factor(P, t), S.imap[p], S.k, S.hnu);
    }
    if (S.dst)
      for (int m = 0; m < nv; m++) {
        double x = S.u[m * ps + p];
        for (int q = 0; q < S.nprev; q++) x = fma_rn(S.a[q], S.d[q][m * ps + p], x);
        S.dst[m * ps + p] = fma_rn(S.as, S.k[m * ps + p], x);
      }
  }
}

// The y term of the 2D hyperbolic divergence on a column slab of a grid
// decomposed along y (columns [c0, c0 + N0) of the whole grid, all N1 rows,
// in the transposed layout: cell values from UT, interface q = j + (N1 + 1) c):
// the upwind fluxes at the y interfaces of a tile as in k_stage2d, then
// dyinv_j (fIy[j+1] - fIy[j]) for every variable, written for the row slab
// that owns row j: hy[((r nvars + m) n1 + j - r n1) N0 + c], r = j / n1.  The
// product is rounded on its own; k_stage2d fuses the x term's product onto it.
template <int UPW, bool MX>
__global__ void __launch_bounds__(256, UPW == UPW_RF && !MX ? 2 : 3) k_slab_upwind_y(DevParams P, const double* __restrict__ UT,
                                                       const void* __restrict__ yuL, const void* __restrict__ yuR,
                                                       const void* __restrict__ yfL, const void* __restrict__ yfR,
                                                       const double* __restrict__ dyinv, void* __restrict__ hy,
                                                       int n1) {
  typedef typename std::conditional<MX, float, double>::type T;
  extern __shared__ double sfd[];
  T* sy = (T*)sfd;
  const int nvars = P.nvars, N0 = P.N0, N1 = P.N1, g = P.ghosts;
  const int i0 = blockIdx.x * TI, j0 = tile_row() * TJ;
  const int tid = threadIdx.x;
  double uref[4];
  if (tid < NY) {
    const int jj = tid % LY, ii = tid / LY;
    const int i = i0 + ii, j = j0 + jj;
    if (j <= N1 && i < N0) {
      const long long line = (long long)P.W1 * (i + g);
      if (MX && (UPW == UPW_LLF || UPW == UPW_RF)) {
#pragma unroll
        for (int m = 0; m < 4; m++) uref[m] = UT[m * P.ps + g + line];
      }
      const long long pR = (long long)(j + g) + line;
      iface_upwind<UPW, 1, MX, 0>(P, yuL, yuR, yfL, yfR, j + (long long)(N1 + 1) * i, UT, pR - 1, pR, uref,
                               sy + ii * LY + jj, NY);
    }
  }
  __syncthreads();
  if (tid >= TI * TJ) return;
  const int ii = tid % TI, jj = tid / TI;
  const int i = i0 + ii, j = j0 + jj;
  if (i >= N0 || j >= N1) return;
  const T dyi = (T)dyinv[g + j];
  const int r = j / n1;
  T* out = (T*)hy + ((long long)r * nvars * n1 + (j - (long long)r * n1)) * N0 + i;
  for (int m = 0; m < nvars; m++)
    out[(long long)m * n1 * N0] = mul_rn(dyi, sy[m * NY + ii * LY + jj + 1] - sy[m * NY + ii * LY + jj]);
}

template <int UPW, int YM, bool MX, int NV, int BT>
void stage2d_bt(const DevParams& P, const Stage2D& S, dim3 grid, cudaStream_t s) {
  typedef typename std::conditional<MX, float, double>::type T;
  raise_smem_limit<k_stage2d<UPW, YM, MX, NV, BT>>(200 * 1024);
  k_stage2d<UPW, YM, MX, NV, BT><<<grid, BT, stage2d_smem<T>(P.nvars, YM == Y_GIVEN, S.visc), s>>>(P, S);
}
template <int UPW, int YM, bool MX, int NV>
void stage2d_nv(const DevParams& P, const Stage2D& S, cudaStream_t s) {
  const dim3 grid = tile_grid(P);
  if constexpr (NV > 0 && YM != Y_GIVEN) {
    if (grid.x * grid.y * grid.z <= 148) return stage2d_bt<UPW, YM, MX, NV, WIDE>(P, S, grid, s);
  }
  stage2d_bt<UPW, YM, MX, NV, NARROW>(P, S, grid, s);
}
template <int UPW, int YM, bool MX>
void stage2d_upw(const DevParams& P, const Stage2D& S, cudaStream_t s) {
  if (stage2d_stores_k(P, S.chem)) stage2d_nv<UPW, YM, MX, 0>(P, S, s);
  else if (P.nvars == 4) stage2d_nv<UPW, YM, MX, 4>(P, S, s);
  else stage2d_nv<UPW, YM, MX, 11>(P, S, s);
}
template <int YM, bool MX>
void stage2d_ym(const DevParams& P, const Stage2D& S, cudaStream_t s) {
  switch (P.upwind) {
    case UPW_ROE: stage2d_upw<UPW_ROE, YM, MX>(P, S, s); break;
    case UPW_RF: stage2d_upw<UPW_RF, YM, MX>(P, S, s); break;
    case UPW_RUSANOV: stage2d_upw<UPW_RUSANOV, YM, MX>(P, S, s); break;
    default: stage2d_upw<UPW_LLF, YM, MX>(P, S, s); break;
  }
}
template <bool MX>
void stage2d_mx(const DevParams& P, const Stage2D& S, cudaStream_t s) {
  if (S.hy) stage2d_ym<Y_GIVEN, MX>(P, S, s);
  else if (S.UT) stage2d_ym<Y_TRANSPOSED, MX>(P, S, s);
  else stage2d_ym<Y_STD, MX>(P, S, s);
}

template <int UPW, bool MX>
void slab_upwind_y_u(const DevParams& P, const double* UT, const void* const* yi, const double* dyinv, void* hy,
                     int n1, cudaStream_t s) {
  raise_smem_limit<k_slab_upwind_y<UPW, MX>>(200 * 1024);
  const dim3 grid = tile_grid(P);
  const size_t smem = (size_t)P.nvars * NY * (MX ? sizeof(float) : sizeof(double));
  k_slab_upwind_y<UPW, MX><<<grid, 256, smem, s>>>(P, UT, yi[0], yi[1], yi[2], yi[3], dyinv, hy, n1);
}
template <bool MX>
void slab_upwind_y_m(const DevParams& P, const double* UT, const void* const* yi, const double* dyinv, void* hy,
                     int n1, cudaStream_t s) {
  switch (P.upwind) {
    case UPW_ROE: slab_upwind_y_u<UPW_ROE, MX>(P, UT, yi, dyinv, hy, n1, s); break;
    case UPW_RF: slab_upwind_y_u<UPW_RF, MX>(P, UT, yi, dyinv, hy, n1, s); break;
    case UPW_RUSANOV: slab_upwind_y_u<UPW_RUSANOV, MX>(P, UT, yi, dyinv, hy, n1, s); break;
    default: slab_upwind_y_u<UPW_LLF, MX>(P, UT, yi, dyinv, hy, n1, s); break;
  }
}

}  // namespace

void launch_stage2d(const DevParams& P, const Stage2D& S, cudaStream_t s) {
  if (P.mixed) stage2d_mx<true>(P, S, s);
  else stage2d_mx<false>(P, S, s);
}

void launch_slab_upwind_y(const DevParams& P, const double* UT, const void* const* yi, const double* dyinv, void* hy,
                          int n1, cudaStream_t s) {
  if (P.mixed) slab_upwind_y_m<true>(P, UT, yi, dyinv, hy, n1, s);
  else slab_upwind_y_m<false>(P, UT, yi, dyinv, hy, n1, s);
}

}  // namespace piafs
