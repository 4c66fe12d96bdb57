// Device pieces of the kernels that run whole steps of a 1D Euler line
// (run1d.cu, run1d_crw.cu).
#pragma once
#include "kernels.h"
#include "physics.cuh"

namespace piafs {
namespace line1d {

constexpr int NV = 3;

// Upwind flux at an interface from its reconstructed values; pl, pr point to
// the velocity, enthalpy and root of the density (stride pp) and ul, ur to the
// state (stride ps) of the cells beside it.  Roe (Euler1DUpwind.c, Euler1DUpwindRoe) with the average of the
// cells' velocity and enthalpy (euler1d.h:93-125) taken from what each cell
// formed once, and the dissipation R |lambda| L (uR - uL) / 2 by its three
// wave strengths: one root and two reciprocals in a row, where the matrices of
// the average's conserved variables take some eight quotients and roots one
// after another.  The other schemes as in the other kernels.
template <int UPW>
__device__ __forceinline__ void iface_flux(const double* uL, const double* uR, const double* fL, const double* fR,
                                           const double* pl, const double* pr, int pp, const double* ul,
                                           const double* ur, int ps, double g, double* fo) {
  if (UPW == UPW_ROE) {
    const double tl = pl[2 * pp], tr = pr[2 * pp], inv = rcp_nr(tl + tr);
    const double v = (tl * pl[0] + tr * pr[0]) * inv;
    const double H = (tl * pl[pp] + tr * pr[pp]) * inv;
    const double gm1 = g - 1.0, ek = 0.5 * v * v;
    const double a2 = gm1 * (H - ek), a = sqrt(a2), ia2 = rcp_nr(a2);
    const double d0 = 0.5 * (uR[0] - uL[0]), d1 = 0.5 * (uR[1] - uL[1]), d2 = 0.5 * (uR[2] - uL[2]);
    const double dp = gm1 * (ek * d0 - v * d1 + d2), adu = a * (d1 - v * d0);
    const double w0 = absv(v) * (d0 - dp * ia2);
    const double wm = absv(v - a) * (0.5 * (dp - adu)) * ia2, wp = absv(v + a) * (0.5 * (dp + adu)) * ia2;
    fo[0] = 0.5 * (fL[0] + fR[0]) - (w0 + (wm + wp));
    fo[1] = 0.5 * (fL[1] + fR[1]) - (v * w0 + ((v - a) * wm + (v + a) * wp));
    fo[2] = 0.5 * (fL[2] + fR[2]) - (ek * w0 + ((H - v * a) * wm + (H + v * a) * wp));
    return;
  }
  double cl[4], cr[4], spa;
  int spm;
#pragma unroll
  for (int m = 0; m < NV; m++) { cl[m] = ul[m * ps]; cr[m] = ur[m * ps]; }
  upwind_flow<EULER1D, UPW, double>(uL, uR, fL, fR, cl, cr, g, 0, fo, &spa, &spm);
}

// What a cell's state u gives: its flux (stride fs at f) and the velocity,
// enthalpy and root of the density of the averages (stride pp at p).
__device__ __forceinline__ void cell_terms(const double* u, double g, double* f, int fs, double* p, int pp) {
  double fl[4], vn;
  euler1d_flux(u[0], u[1], u[2], g, fl, vn);
#pragma unroll
  for (int m = 0; m < NV; m++) f[m * fs] = fl[m];
  const double prs = (u[2] - 0.5 * u[0] * vn * vn) * (g - 1.0);
  p[0] = vn;
  p[pp] = (u[2] + prs) * rcp_nr(u[0]);
  p[2 * pp] = sqrt(u[0]);
}

// The ghost state v of a face (BC type, not periodic) from its mirrored
// interior cell w: BCSlipWall.c:24-136 in one dimension, BCDirichlet.c,
// BCReflect.c, BCExtrapolate.c
__device__ __forceinline__ void face_state(const DevParams& P, const Run1D::Face& face, const double* w, double* v) {
  if (face.type == BC_SLIPWALL) {
    double rho, uv, e, p;
    eu_flowvar(w[0], w[1], w[2], P.bc_gamma, rho, uv, e, p);
    const double ug = 2.0 * face.vel - uv, igm1 = 1.0 / (P.bc_gamma - 1.0);
    v[0] = rho; v[1] = rho * ug; v[2] = igm1 * p + 0.5 * rho * ug * ug;
    return;
  }
#pragma unroll
  for (int m = 0; m < NV; m++)
    v[m] = face.type == BC_DIRICHLET ? face.val[m] : face.type == BC_REFLECT ? -1.0 * w[m] : w[m];
}

}  // namespace line1d
}  // namespace piafs
