// Whole time steps (or one right-hand side) of a 1D Euler line in one launch
// (sm_100a): explicit fifth-order schemes (WENO5, upw5) on components, FP64, any of the
// Runge-Kutta tableaux and upwind schemes (TimeRK.c:34-102 with
// HyperbolicFunction.c:34-214 on one dimension).
//
// A 1D step is some twenty kernels of a few microseconds of launch and latency
// each and almost no work.  Here a thread-block cluster holds the line in its
// shared memory, a segment per CTA, and runs the steps without leaving it: per
// stage the three cells beside a segment come from the neighbours' shared
// memory (or the boundary), then cell fluxes, reconstruction (one item per
// interface, variable and field), upwinding and the Runge-Kutta combination
// follow in the CTA, and one cluster barrier ends the stage.  What bounds it
// is the latency of that chain.
// Measured (B200): a step of the 1024-point WENO5 / Roe wave takes 6.9 us in 16
// CTAs of 64 points; kernel by kernel 47 us, 37 with its boundary fill in one
// launch.
#include <cooperative_groups.h>

#include <algorithm>

#include "kernels.h"
#include "run1d.cuh"

namespace cg = cooperative_groups;

namespace piafs {

namespace {

using namespace line1d;

constexpr int T1D = 512;

// shared memory of a CTA for segments of at most n points, in doubles: two
// stage states and the cell fluxes with three cells either side, per cell the
// velocity, enthalpy and root of the density, u, the stage derivatives, the
// four reconstructed values and the interface fluxes
__host__ __device__ constexpr int smem_doubles(int n, int ns) {
  return NV * (4 * (n + 6) + n + ns * n + 5 * (n + 1));
}

__device__ __forceinline__ int seg_start(int N, int C, int r) { return (int)((long long)N * r / C); }

template <int UPW>
__global__ void __launch_bounds__(T1D) k_run1d(DevParams P, Run1D R, int nmax) {
  extern __shared__ double sm[];
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank(), C = (int)cl.num_blocks();
  const int N = P.N0, tid = threadIdx.x, ns = R.nstages;
  const int i0 = seg_start(N, C, rank), n = seg_start(N, C, rank + 1) - i0;
  const int pS = nmax + 6, pI = nmax + 1;
  double* const buf0 = sm;                             // stage states, cell i at i - i0 + 3
  double* const buf1 = sm + NV * pS;
  double* cf = sm + 2 * NV * pS;                       // cell fluxes
  double* pr = cf + NV * pS;                           // velocity, enthalpy, root of the density
  double* ub = pr + NV * pS;                           // u at the step's start
  double* kd = ub + NV * nmax;                         // stage derivatives [stage][variable]
  double* rec = kd + ns * NV * nmax;                   // [uL uR fL fR][variable]
  double* fi = rec + 4 * NV * pI;                      // interface fluxes
  const double g = P.gamma;
  // cell i of variable m of the state: planes, or point-major with rhs
  auto at = [&](int i, int m) -> double* {
    return R.rhs ? R.u + (long long)(i + 3) * NV + m : R.u + m * P.ps + pidx(P, i, 0);
  };
  auto cell = [&](int c, const double* u) { cell_terms(u, g, cf + c, pS, pr + c, pS); };
  for (int c = tid; c < n; c += T1D) {
    double u[NV];
#pragma unroll
    for (int m = 0; m < NV; m++) u[m] = *at(i0 + c, m);
#pragma unroll
    for (int m = 0; m < NV; m++) { ub[m * nmax + c] = u[m]; buf0[m * pS + 3 + c] = u[m]; }
    cell(3 + c, u);
  }
  // the cells beside the segment, threads 0 .. 5: left ones k - 3 (at k), right
  // ones n + k; their sources are cells of a neighbour, or at an end of the
  // line what the boundary says (ghosts of a face no zone sets keep theirs)
  const int side = tid >= 3, k3 = tid - 3 * side, hc = side ? n + 3 + k3 : k3;
  const bool end = side ? rank == C - 1 : rank == 0;
  const int type = tid < 6 && end ? R.face[side].type : BC_PERIODIC;
  const int from = side ? (rank + 1) % C : (rank + C - 1) % C;
  const int src = side ? k3 + 3 : seg_start(N, C, from + 1) - seg_start(N, C, from) + k3;
  if (tid < 6) {
#pragma unroll
    for (int m = 0; m < NV; m++) buf0[m * pS + hc] = buf1[m * pS + hc] = *at(side ? N + k3 : k3 - 3, m);
  }
  cl.sync();
  int cur = 0;
  for (int step = 0; step < R.nsteps; step++) {
    for (int st = 0; st < ns; st++) {
      double* S = cur ? buf1 : buf0;
      double* Sn = cur ? buf0 : buf1;
      if (tid < 6) {
        double v[NV];
        if (!end || type == BC_PERIODIC) {
          const double* rs = cl.map_shared_rank(S, from) + src;
#pragma unroll
          for (int m = 0; m < NV; m++) v[m] = rs[m * pS];
        } else if (type >= 0) {
          double w[NV];
          for (int m = 0; m < NV; m++) w[m] = S[m * pS + 3 + (side ? n - 1 - k3 : 2 - k3)];
          face_state(P, R.face[side], w, v);
        } else {
          for (int m = 0; m < NV; m++) v[m] = S[m * pS + hc];
        }
#pragma unroll
        for (int m = 0; m < NV; m++) S[m * pS + hc] = v[m];
        cell(hc, v);
        // u comes back with the ghosts of the last step's first stage
        if (end && st == 0 && step == R.nsteps - 1)
          for (int m = 0; m < NV; m++) *at(side ? N + k3 : k3 - 3, m) = v[m];
      }
      __syncthreads();
      for (int e = tid; e < 2 * NV * (n + 1); e += T1D) {
        const int fv = e / (n + 1), i = e - fv * (n + 1), fld = fv >= NV;
        const double* s = (fld ? cf + (fv - NV) * pS : S + fv * pS) + i;
        double c[6], vL, vR;
#pragma unroll
        for (int r = 0; r < 6; r++) c[r] = s[r];
        weno5_pair(P, c, vL, vR);
        rec[(fv + fld * NV) * pI + i] = vL;
        rec[(fv + fld * NV + NV) * pI + i] = vR;
      }
      __syncthreads();
      for (int i = tid; i < n + 1; i += T1D) {
        double a[4], b[4], c[4], d[4], fo[4];
#pragma unroll
        for (int m = 0; m < NV; m++) {
          a[m] = rec[m * pI + i]; b[m] = rec[(NV + m) * pI + i];
          c[m] = rec[(2 * NV + m) * pI + i]; d[m] = rec[(3 * NV + m) * pI + i];
        }
        iface_flux<UPW>(a, b, c, d, pr + i + 2, pr + i + 3, pS, S + i + 2, S + i + 3, pS, g, fo);
#pragma unroll
        for (int m = 0; m < NV; m++) fi[m * pI + i] = fo[m];
      }
      __syncthreads();
      if (R.rhs) {                 // the right-hand side alone, zero at the ghosts
        for (int i = tid; i < n; i += T1D) {
          const double dxi = R.dxinv[P.ghosts + i0 + i];
#pragma unroll
          for (int m = 0; m < NV; m++)
            R.rhs[(long long)(i0 + i + 3) * NV + m] = -(dxi * (fi[m * pI + i + 1] - fi[m * pI + i]));
        }
        if (tid < 3 * NV && rank == 0) R.rhs[tid] = 0.0;
        if (tid < 3 * NV && rank == C - 1) R.rhs[(long long)(N + 3) * NV + tid] = 0.0;
        cl.sync();                 // the neighbours have read this segment
        return;
      }
      const bool last = st == ns - 1;
      const double* co = last ? R.b : R.a + (st + 1) * MAX_STAGES;
      for (int i = tid; i < n; i += T1D) {
        const double dxi = R.dxinv[P.ghosts + i0 + i];
        double x[NV];
#pragma unroll
        for (int m = 0; m < NV; m++) {
          const double k = -(dxi * (fi[m * pI + i + 1] - fi[m * pI + i]));
          x[m] = ub[m * nmax + i];
          for (int j = 0; j < st; j++) x[m] = fma_rn(co[j], kd[(j * NV + m) * nmax + i], x[m]);
          x[m] = fma_rn(co[st], k, x[m]);
          kd[(st * NV + m) * nmax + i] = k;
          if (last) ub[m * nmax + i] = x[m];
          Sn[m * pS + 3 + i] = x[m];
        }
        cell(3 + i, x);
      }
      // the neighbours read Sn next; S is written again only after the next
      // barrier, when every reader of it is past
      cl.sync();
      cur ^= 1;
    }
  }
  for (int i = tid; i < n; i += T1D)
    for (int m = 0; m < NV; m++) *at(i0 + i, m) = ub[m * nmax + i];
  if (rank == 0 && tid == 0) {
    double t = *R.tdev;
    for (int k = 0; k < R.nsteps; k++) t += P.dt;
    *R.tdev = t;
  }
}

template <int UPW>
cudaError_t run1d(const DevParams& P, const Run1D& R, int C, cudaStream_t s, bool probe) {
  const int nmax = (P.N0 + C - 1) / C;
  const int bytes = smem_doubles(nmax, R.nstages) * (int)sizeof(double);
  cudaError_t e = cudaFuncSetAttribute(k_run1d<UPW>, cudaFuncAttributeMaxDynamicSharedMemorySize, kRun1DSmem);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_run1d<UPW>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)C, 1, 1);
  cfg.blockDim = dim3(T1D, 1, 1);
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
    e = cudaOccupancyMaxActiveClusters(&clusters, k_run1d<UPW>, &cfg);
    return e != cudaSuccess ? e : clusters > 0 ? cudaSuccess : cudaErrorInvalidConfiguration;
  }
  return cudaLaunchKernelEx(&cfg, k_run1d<UPW>, P, R, nmax);
}

cudaError_t run1d_upw(const DevParams& P, const Run1D& R, int C, cudaStream_t s, bool probe) {
  switch (P.upwind) {
    case UPW_ROE: return run1d<UPW_ROE>(P, R, C, s, probe);
    case UPW_RF: return run1d<UPW_RF>(P, R, C, s, probe);
    case UPW_LLF: return run1d<UPW_LLF>(P, R, C, s, probe);
    default: return run1d<UPW_RUSANOV>(P, R, C, s, probe);
  }
}

}  // namespace

// CTAs of a line: the largest power of two up to 16 that leaves each 64
// points or more (fewer and the reconstruction no longer fills the threads,
// while every stage still pays the cluster barrier).
int run1d_ctas(const DevParams& P, const Run1D& R) {
  if (P.scheme == CRWENO5) return run1d_crw_ctas(P, R);
  int C = 1;
  while (C < 16 && P.N0 / (2 * C) >= 64) C *= 2;
  for (; C >= 1; C /= 2) {
    const int nmax = (P.N0 + C - 1) / C;
    if (smem_doubles(nmax, R.nstages) * (int)sizeof(double) > kRun1DSmem) return 0;
    if (run1d_upw(P, R, C, nullptr, true) == cudaSuccess) return C;
    cudaGetLastError();   // this cluster size is not to be had: try a smaller one
  }
  return 0;
}

cudaError_t launch_run1d(const DevParams& P, const Run1D& R, int ctas, cudaStream_t s) {
  if (P.scheme == CRWENO5) return launch_run1d_crw(P, R, ctas, s);
  return run1d_upw(P, R, ctas, s, false);
}

}  // namespace piafs
