// C ABI of the PIAFS GPU path (include/piafs_gpu.h): simulation object,
// time stepping with CUDA-graph replay, Solve() loop with reference-format
// output, and the operator-level entry points.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/piafs_gpu.h"
#include "deck.h"
#include "kernels.h"
#include "sim.h"

using namespace piafs;

namespace {
thread_local std::string g_err;

int fail(int code, const std::string& msg) {
  g_err = msg;
  return code;
}
}  // namespace

namespace piafs {
int set_last_error(int code, const std::string& msg) { return fail(code, msg); }
}

#define CK(call)                                                                                  \
  do {                                                                                            \
    cudaError_t e_ = (call);                                                                      \
    if (e_ != cudaSuccess)                                                                        \
      return fail(e_ == cudaErrorMemoryAllocation ? PIAFS_ERR_MEMORY : PIAFS_ERR_CUDA,             \
                  std::string(#call) + ": " + cudaGetErrorString(e_));                             \
  } while (0)


static void free_sim(piafs_gpu_sim* s) {
  if (!s) return;
  for (auto& g : s->graph) if (g) cudaGraphExecDestroy(g);
  cudaFree(s->u);
  for (int k = 1; k < MAX_STAGES; k++) cudaFree(s->U[k]);
  for (auto p : s->Ud) cudaFree(p);
  cudaFree(s->fC);
  for (auto p : s->iface) cudaFree(p);
  for (auto p : s->iface_y) cudaFree(p);
  cudaFree(s->scratch);
  cudaFree(s->ut);
  cudaFree(s->dxinv);
  cudaFree(s->imap);
  cudaFree(s->tdev);
  cudaFree(s->top_t);
  cudaFree(s->norm_acc);
  cudaFree(s->cfl_acc);
  cudaFree(s->err);
  cudaFree(s->aos);
  cudaFree(s->hnu);
  cudaFree(s->sponge_buf);
  cudaFree(s->zone_buf);
  cudaFree(s->crwchar);
  if (s->yfork) cudaEventDestroy(s->yfork);
  if (s->yjoin) cudaEventDestroy(s->yjoin);
  if (s->ystream) cudaStreamDestroy(s->ystream);
  if (s->stream) cudaStreamDestroy(s->stream);
  delete s;
}

// -------------------------------------------------------------- the RHS
// Cell-centred flux (into F) and interface values (uL, uR, fL, fR into I) of
// direction d, on the given stream.  The y pass of a 2D CRWENO5 run works on a
// transposed copy of U so that its lines, the tridiagonal systems, are
// contiguous in memory; its interface arrays are then in the transposed layout.
// If `ev` is given, an event is recorded after the flux and after the
// reconstruction.
static void enqueue_recon_on(piafs_gpu_sim* s, const double* U, int d, double* F, double* const* I, cudaStream_t st,
                             cudaEvent_t* ev, int* k) {
  const DevParams& P = s->P;
  auto mark = [&]() { if (ev) cudaEventRecord(ev[++*k], st); };
  if (d == 1 && s->ut) {
    if (P.model == NS2D) {
      launch_transpose_flux_y(P, U, s->ut, F, st);
    } else {
      launch_transpose(P, U, s->ut, st);
      launch_flux(P, s->ut, F, 1, st);
    }
    mark();
    launch_crweno(s->PT, s->ut, F, I[0], I[1], I[2], I[3], 0, s->err, st);
    mark();
    return;
  }
  launch_flux(P, U, F, d, st);
  mark();
  if (P.scheme == CRWENO5 && P.char_interp)
    launch_crweno_char(P, U, F, I[0], I[1], I[2], I[3], d, s->crwchar, s->err, st);
  else if (P.scheme != CRWENO5 && P.char_interp) launch_weno5_char(P, U, F, I[0], I[1], I[2], I[3], d, st);
  else if (P.scheme != CRWENO5) launch_weno5(P, U, F, I[0], I[1], I[2], I[3], d, st);
  else launch_crweno(P, U, F, I[0], I[1], I[2], I[3], d, s->err, st);
  mark();
}

void piafs::enqueue_recon(piafs_gpu_sim* s, const double* U, int d, double* const* I, cudaEvent_t* ev, int* k) {
  enqueue_recon_on(s, U, d, s->fC, I, s->stream, ev, k);
}

// The reconstruction of both directions of a 2D grid: the y pass on its own
// stream and flux array, concurrent with the x pass, where the simulation has
// one (and no phase events are asked for); joined when this returns.  On small
// and middling grids neither pass fills the GPU: the 300 x 217 WENO5 step took
// 148 us with the passes in turn, 141 with both at once.
static void enqueue_recon2d(piafs_gpu_sim* s, const double* U, cudaEvent_t* ev = nullptr, int* k = nullptr) {
  const bool concurrent = s->concurrent_y && !ev;
  if (concurrent) cudaEventRecord(s->yfork, s->stream);
  enqueue_recon(s, U, 0, s->iface, ev, k);
  if (concurrent) {
    // the y pass joins the x pass's stream before the kernel that ends the stage
    cudaStreamWaitEvent(s->ystream, s->yfork, 0);
    enqueue_recon_on(s, U, 1, s->fCy, s->iface_y, s->ystream, nullptr, nullptr);
    cudaEventRecord(s->yjoin, s->ystream);
    cudaStreamWaitEvent(s->stream, s->yjoin, 0);
  } else {
    enqueue_recon(s, U, 1, s->iface_y, ev, k);
  }
}

// What ends a stage from the interface arrays of enqueue_recon2d: -hyp or hyp
// alone into k, until the caller asks for more.
static Stage2D stage2d_args(piafs_gpu_sim* s, const double* U, double* k, bool neg) {
  Stage2D S{};
  S.U = U;
  S.UT = s->ut;
  for (int i = 0; i < 4; i++) { S.xi[i] = s->iface[i]; S.yi[i] = s->iface_y[i]; }
  S.dxinv = s->dxinv;
  S.imap = s->imap;
  S.neg = neg ? 1 : 0;
  S.k = k;
  return S;
}

// the fourth-order viscous terms have their own kernel, the source with them
static bool visc4(const DevParams& P) { return P.viscous && P.par4; }

// HyperbolicFunction (HyperbolicFunction.c:35-119) over all directions into
// out: -hyp (neg, the stage derivative's first term) or hyp.
static void enqueue_hyp(piafs_gpu_sim* s, const double* U, double* out, bool neg, cudaEvent_t* ev = nullptr,
                        int* k = nullptr) {
  const DevParams& P = s->P;
  if (P.ndims == 1) {
    enqueue_recon(s, U, 0, s->iface, ev, k);
    launch_upwind_div(P, U, s->iface[0], s->iface[1], s->iface[2], s->iface[3], s->dxinv, out, 0, neg ? 0 : 2,
                      s->stream);
  } else {
    enqueue_recon2d(s, U, ev, k);
    launch_stage2d(P, stage2d_args(s, U, out, neg), s->stream);
  }
  if (ev) cudaEventRecord(ev[++*k], s->stream);
}

// the sponge zones' source (SourceFunction.c:42-57) added to rhs
static void enqueue_sponge(piafs_gpu_sim* s, const double* U, double* rhs) {
  for (const auto& z : s->sponges)
    launch_sponge(s->P, U, rhs, z.dim, z.is, z.ie, s->sponge_buf + z.sig_off, s->sponge_buf + z.ref_off, s->stream);
}

// The Runge-Kutta combination that follows a stage (TimeRK.c:60-75, :86-99):
// dst = u + sum a[j] d[j] + as * (the stage's derivative).
struct RkNext {
  double* dst;
  int nprev;
  const double* d[MAX_STAGES];
  double a[MAX_STAGES];
  double as;
};

// TimeRHSFunctionExplicit (TimeRHSFunctionExplicit.c:29-77) on SoA arrays:
// rhs = -hyp + par + source; U must have its ghosts filled.
// hnu: where the source stores the photon density of this evaluation (the
// reference's Chemistry::nv_hnu), or nullptr.  next (2D, s->fuse_rk): the
// combination that follows, formed by the same kernel; keep: whether rhs is
// read after it.
static void enqueue_rhs(piafs_gpu_sim* s, double* rhs, const double* U, const double* tdev, double cstage,
                        double* hnu = nullptr, const RkNext* next = nullptr, bool keep = true,
                        cudaEvent_t* ev = nullptr, int* k = nullptr) {
  const DevParams& P = s->P;
  auto mark = [&]() { if (ev) cudaEventRecord(ev[++*k], s->stream); };
  if (P.ndims == 1 || visc4(P)) {
    enqueue_hyp(s, U, rhs, true, ev, k);
    launch_visc_source(P, U, s->dxinv, s->imap, tdev, cstage, rhs, 1, 1, s->stream, hnu);
  } else {
    enqueue_recon2d(s, U, ev, k);
    Stage2D S = stage2d_args(s, U, rhs, true);
    S.visc = P.viscous;
    S.chem = P.chem;
    S.tdev = tdev;
    S.cstage = cstage;
    S.hnu = hnu;
    if (next) {
      S.dst = next->dst;
      S.u = s->u;
      S.nprev = next->nprev;
      for (int j = 0; j < next->nprev; j++) { S.d[j] = next->d[j]; S.a[j] = next->a[j]; }
      S.as = next->as;
      if (!keep && !stage2d_stores_k(P, S.chem)) S.k = nullptr;
    }
    launch_stage2d(P, S, s->stream);
    mark();
  }
  enqueue_sponge(s, U, rhs);
  mark();
}

void piafs::enqueue_bc(piafs_gpu_sim* s, double* u) {
  launch_bc(s->P, u, s->deck.zones.data(), (int)s->deck.zones.size(), s->stream);
}

// One time step: TimePreStep's boundary conditions on u, TimeRK's stages and
// step completion, t += dt.  U[0] aliases u: the reference copies u into
// U[0] and re-applies the (idempotent) boundary conditions to it.  Where the
// kernel that ends a stage forms the combination too, it writes the interior
// points of the next stage's state (ghosts no zone writes keep u's values,
// copied when the state was set); a step that asks for the norm completes
// with the kernel that sums it.
static void enqueue_step(piafs_gpu_sim* s, bool with_norm) {
  const DevParams& P = s->P;
  const Deck& d = s->deck;
  const int ns = d.nstages;
  const long long n = (long long)P.nvars * P.ps;
  // coefficients of the state after stage st: the next stage's, or the step's
  auto coef = [&](int st, int j) { return d.dt * (st < ns - 1 ? d.A[(st + 1) * MAX_STAGES + j] : d.b[j]); };
  enqueue_bc(s, s->u);
  for (int st = 0; st < ns; st++) {
    double* Us = st == 0 ? s->u : s->U[st];
    const bool last = st == ns - 1;
    double* hnu = last ? s->hnu : nullptr;
    if (s->fuse_rk && !(last && with_norm)) {
      RkNext nx{};
      nx.dst = last ? s->u : s->U[st + 1];
      nx.nprev = st;
      for (int j = 0; j < st; j++) { nx.d[j] = s->Ud[j]; nx.a[j] = coef(st, j); }
      nx.as = coef(st, st);
      enqueue_rhs(s, s->Ud[st], Us, s->tdev, d.c[st], hnu, &nx, !last);
      if (!last) enqueue_bc(s, s->U[st + 1]);
      continue;
    }
    enqueue_rhs(s, s->Ud[st], Us, s->tdev, d.c[st], hnu);
    const double* dd[MAX_STAGES];
    double a[MAX_STAGES];
    for (int j = 0; j <= st; j++) { dd[j] = s->Ud[j]; a[j] = coef(st, j); }
    if (!last) {
      launch_stage(n, s->U[st + 1], s->u, dd, a, st + 1, s->stream);
      enqueue_bc(s, s->U[st + 1]);
    } else {
      if (with_norm) cudaMemsetAsync(s->norm_acc, 0, sizeof(double), s->stream);
      launch_update(P, s->u, dd, a, ns, with_norm ? s->norm_acc : nullptr, s->stream);
    }
  }
  launch_advance_time(s->tdev, d.dt, s->stream);
}

// Steps of a 1D line in launches of at most 1024 (7 ms of the 1024-point WENO5
// line, 44 ms of the 6001-point CRWENO5 one).
static int enqueue_run1d(piafs_gpu_sim* s, int nsteps) {
  for (int k = 0; k < nsteps;) {
    Run1D R = s->run1d;
    R.nsteps = std::min(nsteps - k, 1024);
    CK(launch_run1d(s->P, R, s->run1d_ctas, s->stream));
    k += R.nsteps;
  }
  for (int k = 0; k < nsteps; k++) s->t += s->deck.dt;
  s->iter += nsteps;
  return PIAFS_OK;
}

// the line's arguments for enqueue_run1d, where it is one of those
static void setup_run1d(piafs_gpu_sim* s) {
  const DevParams& P = s->P;
  const Deck& d = s->deck;
  if (!(P.ndims == 1 && P.model == EULER1D && !P.chem && P.nvars == 3 && P.ghosts == 3 && !P.mixed &&
        !P.char_interp && s->sponges.empty() && P.N0 >= 16 && d.nstages >= 1))
    return;
  Run1D& R = s->run1d;
  R.u = s->u;
  R.dxinv = s->dxinv;
  R.tdev = s->tdev;
  R.err = s->err;
  R.nstages = d.nstages;
  for (int i = 0; i < MAX_STAGES * MAX_STAGES; i++) R.a[i] = d.dt * d.A[i];
  for (int i = 0; i < MAX_STAGES; i++) R.b[i] = d.dt * d.b[i];
  for (auto& f : R.face) f = {-1, 0.0, nullptr};
  for (const Zone& z : d.zones) {
    if (z.ie[1] <= z.is[1] || z.ie[0] - z.is[0] != P.ghosts) return;   // not a whole face
    if (!bc_per_variable(z.type) && z.type != BC_SLIPWALL) continue;   // acts in two dimensions only
    R.face[z.face == 1 ? 0 : 1] = {z.type, z.vel[0], z.val};
  }
  s->run1d_ctas = run1d_ctas(P, R);
}

static int run_steps(piafs_gpu_sim* s, int nsteps, bool norm_last) {
  int k0 = 0;
  if (s->run1d_ctas > 0) {
    // a step with the norm is one of the same steps, its start kept: the state
    // must not depend on whether the norm is asked for
    k0 = nsteps;
    if (int r = enqueue_run1d(s, norm_last ? nsteps - 1 : nsteps)) return r;
    if (norm_last) {
      CK(cudaMemcpyAsync(s->scratch, s->u, (size_t)s->P.nvars * s->P.ps * sizeof(double), cudaMemcpyDeviceToDevice,
                         s->stream));
      if (int r = enqueue_run1d(s, 1)) return r;
      CK(cudaMemsetAsync(s->norm_acc, 0, sizeof(double), s->stream));
      launch_norm(s->P, s->scratch, s->u, s->norm_acc, s->stream);
    }
  }
  for (int k = k0; k < nsteps; k++) {
    const bool with_norm = norm_last && (k == nsteps - 1);
    const int gi = with_norm ? 1 : 0;
    if (s->use_graph) {
      if (!s->graph[gi]) {
        cudaGraph_t g;
        CK(cudaStreamBeginCapture(s->stream, cudaStreamCaptureModeThreadLocal));
        enqueue_step(s, with_norm);
        CK(cudaStreamEndCapture(s->stream, &g));
        CK(cudaGraphInstantiate(&s->graph[gi], g, 0));
        cudaGraphDestroy(g);
      }
      CK(cudaGraphLaunch(s->graph[gi], s->stream));
    } else {
      enqueue_step(s, with_norm);
    }
    s->t += s->deck.dt;   // same accumulation as the device clock (TimePostStep.c:31)
    s->iter++;
  }
  CK(cudaGetLastError());
  CK(cudaStreamSynchronize(s->stream));
  int e = 0;
  CK(cudaMemcpy(&e, s->err, sizeof(int), cudaMemcpyDeviceToHost));
  if (e) {
    s->singular++;
    cudaMemset(s->err, 0, sizeof(int));
  }
  if (norm_last) {
    double sum = 0.0;
    CK(cudaMemcpy(&sum, s->norm_acc, sizeof(double), cudaMemcpyDeviceToHost));
    double npts = (double)s->P.N0 * (double)s->P.N1;
    s->last_norm = std::sqrt(sum / npts);
  }
  return PIAFS_OK;
}

// ------------------------------------------------------------------ C ABI
extern "C" {

const char* piafs_gpu_last_error(void) { return g_err.c_str(); }

int piafs_gpu_create(const char* deck_dir, int precision, piafs_gpu_sim** out) {
  if (!deck_dir || !out) return fail(PIAFS_ERR_ARGUMENT, "null argument");
  *out = nullptr;
  Deck d;
  std::string err;
  if (int r = read_deck(deck_dir, d, err)) return fail(r, err);
  return piafs::create_sim(std::move(d), precision, out);
}

}  // extern "C"

// A simulation from a parsed (or otherwise filled) deck: device arrays,
// initial state, simulation time restart_iter x dt.
int piafs::create_sim(Deck&& deck, int precision, piafs_gpu_sim** out) {
  if (!out) return fail(PIAFS_ERR_ARGUMENT, "null argument");
  *out = nullptr;
  if (precision != PIAFS_PRECISION_FP64 && precision != PIAFS_PRECISION_MIXED)
    return fail(PIAFS_ERR_ARGUMENT, "precision must be PIAFS_PRECISION_FP64 or PIAFS_PRECISION_MIXED");
  auto* s = new piafs_gpu_sim();
  s->deck = std::move(deck);
  std::string err;
  int r = make_params(s->deck, s->P, err);
  if (r) { delete s; return fail(r, err); }
  s->precision = precision;
  s->P.mixed = precision == PIAFS_PRECISION_MIXED ? 1 : 0;
  {
    // PIAFS_GPU_NO_PACKED_SPECIES=1 keeps the four interface arrays (the
    // same values; for checking the packed form)
    const DevParams& Q = s->P;
    const char* npk = std::getenv("PIAFS_GPU_NO_PACKED_SPECIES");
    s->P.pack_sp = (Q.model == NS2D && Q.ndims == 2 && !Q.char_interp && Q.upwind != UPW_RF &&
                    (Q.scheme != CRWENO5 || (crweno_packs(Q.N0) && crweno_packs(Q.N1))) && !(npk && npk[0] == '1'))
                       ? 1 : 0;
  }
  if (s->P.mixed && s->P.char_interp) {
    delete s;
    return fail(PIAFS_ERR_UNSUPPORTED, "mixed precision runs hyp_interp_type components");
  }
  const char* ng = std::getenv("PIAFS_GPU_NO_GRAPH");
  s->use_graph = !(ng && ng[0] == '1');
  const DevParams& P = s->P;
  const Deck& d = s->deck;
  auto alloc = [&](double** p, size_t n) -> cudaError_t {
    cudaError_t e = cudaMalloc(p, n * sizeof(double));
    if (e == cudaSuccess) e = cudaMemset(*p, 0, n * sizeof(double));
    return e;
  };
  cudaError_t e = cudaGetDevice(&s->device);
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking);
  const size_t planes = (size_t)P.nvars * P.ps, iplanes = (size_t)P.nvars * P.pis;
  if (e == cudaSuccess) e = alloc(&s->u, planes);
  for (int k = 1; k < d.nstages && e == cudaSuccess; k++) e = alloc(&s->U[k], planes);
  for (int k = 0; k < d.nstages && e == cudaSuccess; k++) e = alloc(&s->Ud[k], planes);
  if (e == cudaSuccess) e = alloc(&s->fC, planes);
  for (int k = 0; k < 5 && e == cudaSuccess; k++) e = alloc(&s->iface[k], iplanes);
  for (int k = 0; k < 4 && e == cudaSuccess && P.ndims == 2; k++) e = alloc(&s->iface_y[k], iplanes);
  if (e == cudaSuccess) e = alloc(&s->scratch, planes);
  // transposed y pass: 2D CRWENO5 (PIAFS_GPU_NO_YTRANSPOSE=1 keeps the
  // column-strided kernels instead in the FP64 path; the mixed path has only
  // the transposed one)
  const char* noyt = std::getenv("PIAFS_GPU_NO_YTRANSPOSE");
  if (e == cudaSuccess && P.scheme == CRWENO5 && P.char_interp) e = alloc(&s->crwchar, crweno_char_scratch(P));
  if (e == cudaSuccess && P.ndims == 2 && P.scheme == CRWENO5 && !P.char_interp &&
      (P.mixed || !(noyt && noyt[0] == '1'))) {
    e = alloc(&s->ut, planes);
    s->PT = transposed_params(P);
  }
  if (e == cudaSuccess) e = alloc(&s->dxinv, d.dxinv.size());
  if (e == cudaSuccess) e = alloc(&s->imap, d.imap.size());
  if (e == cudaSuccess) e = alloc(&s->tdev, 1);
  if (e == cudaSuccess) e = alloc(&s->top_t, 1);
  if (e == cudaSuccess) e = alloc(&s->norm_acc, 1);
  if (e == cudaSuccess) e = cudaMalloc(&s->cfl_acc, sizeof(unsigned long long));
  if (e == cudaSuccess) e = cudaMalloc(&s->err, sizeof(int));
  if (e == cudaSuccess) e = cudaMemset(s->err, 0, sizeof(int));
  s->aos_bytes = (size_t)P.npg * P.nvars * sizeof(double);
  // The y pass on a stream of its own (2D Navier-Stokes; the characteristic
  // CRWENO5 solves share one scratch).  Its fluxes go into the array that host
  // transfers are staged in: both are used on the simulation's stream, which a
  // y pass forks from and joins, so never at once.  (An array of its own was one
  // state more of device memory: 94 MB of 1.8 GB at 1024^2 with chemistry.)  Without
  // the stream or an event, and with PIAFS_GPU_NO_CONCURRENT_Y=1, the passes run
  // in turn (the same values).
  const char* ncy = std::getenv("PIAFS_GPU_NO_CONCURRENT_Y");
  const bool ypass = P.ndims == 2 && P.model == NS2D && !s->crwchar && (P.scheme != CRWENO5 || s->ut) &&
                     !(ncy && ncy[0] == '1');
  if (e == cudaSuccess) e = cudaMalloc(&s->aos, ypass ? planes * sizeof(double) : s->aos_bytes);
  if (e == cudaSuccess && ypass) {
    s->concurrent_y = cudaStreamCreateWithFlags(&s->ystream, cudaStreamNonBlocking) == cudaSuccess &&
                      cudaEventCreateWithFlags(&s->yfork, cudaEventDisableTiming) == cudaSuccess &&
                      cudaEventCreateWithFlags(&s->yjoin, cudaEventDisableTiming) == cudaSuccess;
    if (s->concurrent_y) s->fCy = s->aos;
    else cudaGetLastError();
  }
  // the species files carry the photon density of the last RK stage evaluated
  // (zero before the first step, as the reference's calloc'd nv_hnu)
  const bool binary_out = d.op_file_format == "binary" || d.op_file_format == "bin";
  if (e == cudaSuccess && d.write_species && binary_out) e = alloc(&s->hnu, (size_t)P.nz * P.ps);
  if (e == cudaSuccess && !d.sponges.empty()) {
    std::vector<double> hb;
    for (const auto& z : d.sponges) {
      piafs_gpu_sim::SpongeDev sd{};
      sd.dim = z.dim;
      for (int k = 0; k < 2; k++) { sd.is[k] = z.is[k]; sd.ie[k] = z.ie[k]; }
      sd.ref_off = hb.size();
      hb.insert(hb.end(), z.uref.begin(), z.uref.end());
      sd.sig_off = hb.size();
      hb.insert(hb.end(), z.sigma.begin(), z.sigma.end());
      s->sponges.push_back(sd);
    }
    e = alloc(&s->sponge_buf, hb.size());
    if (e == cudaSuccess) e = cudaMemcpy(s->sponge_buf, hb.data(), hb.size() * sizeof(double), cudaMemcpyHostToDevice);
  }
  if (e == cudaSuccess) {
    std::vector<size_t> off;
    const std::vector<double> hv = pack_zone_values(d, off);
    if (!hv.empty()) {
      e = alloc(&s->zone_buf, hv.size());
      if (e == cudaSuccess) e = cudaMemcpy(s->zone_buf, hv.data(), hv.size() * sizeof(double), cudaMemcpyHostToDevice);
      if (e == cudaSuccess) bind_zone_values(d, off, s->zone_buf, s->deck.zones.data());
    }
  }
  if (e == cudaSuccess) e = cudaMemcpy(s->dxinv, d.dxinv.data(), d.dxinv.size() * sizeof(double), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(s->imap, d.imap.data(), d.imap.size() * sizeof(double), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    int code = e == cudaErrorMemoryAllocation ? PIAFS_ERR_MEMORY : PIAFS_ERR_CUDA;
    std::string msg = std::string("device set-up failed: ") + cudaGetErrorString(e);
    free_sim(s);
    return fail(code, msg);
  }
  s->U[0] = s->u;
  // one-stage schemes advance u itself, which other tiles still read as the
  // stage's state: their combination stays a kernel of its own.  So does that
  // of a grid narrower than its ghost layers: its boundary fill reads ghosts of
  // the face across before it writes them, and they must be this step's of u,
  // which only the combination over all points carries into a stage's state
  s->fuse_rk = P.ndims == 2 && !visc4(P) && s->sponges.empty() && d.nstages > 1 && !narrow_grid(P);
  setup_run1d(s);
  // initial solution; restart time waqt = restart_iter * dt (TimeInitialize.c:51)
  int rr = piafs_gpu_set_state(s, d.u0.data(), d.restart_iter * d.dt);
  if (rr) { free_sim(s); return rr; }
  s->iter = d.restart_iter;
  *out = s;
  return PIAFS_OK;
}

extern "C" {

void piafs_gpu_destroy(piafs_gpu_sim* s) { free_sim(s); }

int piafs_gpu_get_photon_density(piafs_gpu_sim* s, double* nv_hnu) {
  if (!s || !nv_hnu) return fail(PIAFS_ERR_ARGUMENT, "null argument");
  if (!s->hnu) return fail(PIAFS_ERR_ARGUMENT, "this simulation keeps no photon density (no species output)");
  const DevParams& P = s->P;
  std::vector<double> h((size_t)P.nz * P.ps);
  CK(cudaMemcpyAsync(h.data(), s->hnu, h.size() * sizeof(double), cudaMemcpyDeviceToHost, s->stream));
  CK(cudaStreamSynchronize(s->stream));
  for (long long p = 0; p < P.npg; p++)
    for (int iz = 0; iz < P.nz; iz++) nv_hnu[(size_t)P.nz * p + iz] = h[(size_t)iz * P.ps + p];
  return PIAFS_OK;
}

int piafs_gpu_get_info(piafs_gpu_sim* s, piafs_gpu_info* info) {
  if (!s || !info) return fail(PIAFS_ERR_ARGUMENT, "null argument");
  const Deck& d = s->deck;
  std::memset(info, 0, sizeof(*info));
  info->ndims = d.ndims; info->nvars = d.nvars; info->ghosts = d.ghosts;
  info->dim[0] = s->P.N0; info->dim[1] = s->P.N1;
  info->n_iter = d.n_iter; info->restart_iter = d.restart_iter;
  info->screen_op_iter = d.screen_op_iter; info->file_op_iter = d.file_op_iter;
  info->iter = s->iter; info->nstages = d.nstages;
  info->dt = d.dt; info->t = s->t;
  info->gamma = d.gamma; info->Re = d.Re; info->Pr = d.Pr;
  info->npoints_ghosted = s->P.npg;
  info->ninterfaces[0] = s->P.nint[0]; info->ninterfaces[1] = s->P.nint[1];
  info->cfl = s->last_cfl; info->norm = s->last_norm; info->singular = s->singular;
  // launches per step: 1 for a 1D line in one launch (which takes up to 1024
  // steps); else the BC launches (nz) of every stage, per stage flux
  // and reconstruction per direction plus the transpose of a transposed y
  // pass and the upwind / stage kernel, the separate source and combination
  // kernels where they are not part of it, and the clock
  const int nz = launch_bc(s->P, nullptr, d.zones.data(), (int)d.zones.size(), nullptr);
  const int vs = (((s->P.ndims == 2 && s->P.viscous) || s->P.chem) && (s->P.ndims == 1 || visc4(s->P))) ? 1 : 0;
  const int tr = (s->ut && s->P.model != NS2D) ? 1 : 0;   // NS2D: the transpose also forms the y flux
  info->launches_per_step = s->run1d_ctas > 0 ? 1 : d.nstages * (nz + 2 * s->P.ndims + 1 + tr + vs + (s->fuse_rk ? 0 : 1)) + 1;
  return PIAFS_OK;
}

int piafs_gpu_set_state(piafs_gpu_sim* s, const double* u_host, double t) {
  if (!s || !u_host) return fail(PIAFS_ERR_ARGUMENT, "null argument");
  CK(cudaMemcpyAsync(s->aos, u_host, s->aos_bytes, cudaMemcpyHostToDevice, s->stream));
  launch_aos_to_soa(s->aos, s->u, s->P.npg, s->P.nvars, s->P.ps, s->stream);
  if (s->fuse_rk) launch_copy_ghosts(s->P, s->u, s->U + 1, s->deck.nstages - 1, s->stream);
  CK(cudaMemcpyAsync(s->tdev, &t, sizeof(double), cudaMemcpyHostToDevice, s->stream));
  CK(cudaStreamSynchronize(s->stream));
  s->t = t;
  return PIAFS_OK;
}

int piafs_gpu_get_state(piafs_gpu_sim* s, double* u_host) {
  if (!s || !u_host) return fail(PIAFS_ERR_ARGUMENT, "null argument");
  launch_soa_to_aos(s->u, s->aos, s->P.npg, s->P.nvars, s->P.ps, s->stream);
  CK(cudaMemcpyAsync(u_host, s->aos, s->aos_bytes, cudaMemcpyDeviceToHost, s->stream));
  CK(cudaStreamSynchronize(s->stream));
  return PIAFS_OK;
}

int piafs_gpu_get_solution(piafs_gpu_sim* s, double* out) {
  if (!s || !out) return fail(PIAFS_ERR_ARGUMENT, "null argument");
  launch_soa_to_interior(s->P, s->u, s->aos, s->stream);
  CK(cudaMemcpyAsync(out, s->aos, (size_t)s->P.N0 * s->P.N1 * s->P.nvars * sizeof(double), cudaMemcpyDeviceToHost,
                     s->stream));
  CK(cudaStreamSynchronize(s->stream));
  return PIAFS_OK;
}

int piafs_gpu_TimeRK(piafs_gpu_sim* s, int nsteps) {
  if (!s || nsteps < 0) return fail(PIAFS_ERR_ARGUMENT, "bad argument");
  return run_steps(s, nsteps, false);
}

int piafs_gpu_TimeRK_async(piafs_gpu_sim* s, int nsteps) {
  if (!s || nsteps < 0) return fail(PIAFS_ERR_ARGUMENT, "bad argument");
  if (s->run1d_ctas > 0) {
    if (int r = enqueue_run1d(s, nsteps)) return r;
    CK(cudaGetLastError());
    return PIAFS_OK;
  }
  for (int k = 0; k < nsteps; k++) {
    if (s->use_graph) {
      if (!s->graph[0]) {
        cudaGraph_t g;
        CK(cudaStreamBeginCapture(s->stream, cudaStreamCaptureModeThreadLocal));
        enqueue_step(s, false);
        CK(cudaStreamEndCapture(s->stream, &g));
        CK(cudaGraphInstantiate(&s->graph[0], g, 0));
        cudaGraphDestroy(g);
      }
      CK(cudaGraphLaunch(s->graph[0], s->stream));
    } else {
      enqueue_step(s, false);
    }
    s->t += s->deck.dt;
    s->iter++;
  }
  CK(cudaGetLastError());
  return PIAFS_OK;
}

int piafs_gpu_get_stream(piafs_gpu_sim* s, void** stream) {
  if (!s || !stream) return fail(PIAFS_ERR_ARGUMENT, "null argument");
  *stream = (void*)s->stream;
  return PIAFS_OK;
}

int piafs_gpu_synchronize(piafs_gpu_sim* s) {
  if (!s) return fail(PIAFS_ERR_ARGUMENT, "null argument");
  CK(cudaStreamSynchronize(s->stream));
  int e = 0;
  CK(cudaMemcpy(&e, s->err, sizeof(int), cudaMemcpyDeviceToHost));
  if (e) { s->singular++; cudaMemset(s->err, 0, sizeof(int)); }
  return PIAFS_OK;
}

int piafs_gpu_profile_rhs(piafs_gpu_sim* s, int reps, double* ms, int* nphases) {
  if (!s || !ms || !nphases || reps < 1) return fail(PIAFS_ERR_ARGUMENT, "bad argument");
  const DevParams& P = s->P;
  const int np = P.ndims == 1 ? 4 : 6;
  if (*nphases < np) return fail(PIAFS_ERR_ARGUMENT, "ms[] too small");
  *nphases = np;
  std::vector<cudaEvent_t> ev(np + 1);
  for (auto& e : ev) CK(cudaEventCreate(&e));
  std::vector<double> acc(np, 0.0);
  double* U = s->u;
  double* R = s->Ud[0];
  // one untimed evaluation first: the first launches of a kernel outside the
  // step graphs carry one-time set-up
  for (int r = -1; r < reps; r++) {
    enqueue_bc(s, U);
    int k = 0;
    CK(cudaEventRecord(ev[0], s->stream));
    enqueue_rhs(s, R, U, s->tdev, 0.0, nullptr, nullptr, true, ev.data(), &k);
    CK(cudaStreamSynchronize(s->stream));
    if (r < 0) continue;
    for (int i = 0; i < np; i++) {
      float t = 0.f;
      CK(cudaEventElapsedTime(&t, ev[i], ev[i + 1]));
      acc[i] += t;
    }
  }
  for (auto& e : ev) cudaEventDestroy(e);
  for (int i = 0; i < np; i++) ms[i] = acc[i] / reps;
  CK(cudaGetLastError());
  return PIAFS_OK;
}

int piafs_gpu_TimeRK_host(piafs_gpu_sim* s, double* u_host, double t) {
  if (int r = piafs_gpu_set_state(s, u_host, t)) return r;
  if (int r = run_steps(s, 1, false)) return r;
  return piafs_gpu_get_state(s, u_host);
}

int piafs_gpu_ComputeCFL(piafs_gpu_sim* s, double* cfl) {
  if (!s || !cfl) return fail(PIAFS_ERR_ARGUMENT, "null argument");
  CK(cudaMemsetAsync(s->cfl_acc, 0, sizeof(unsigned long long), s->stream));
  launch_cfl(s->P, s->u, s->dxinv, s->cfl_acc, s->stream);
  unsigned long long bits = 0;
  CK(cudaMemcpyAsync(&bits, s->cfl_acc, sizeof(bits), cudaMemcpyDeviceToHost, s->stream));
  CK(cudaStreamSynchronize(s->stream));
  std::memcpy(cfl, &bits, sizeof(double));
  s->last_cfl = *cfl;
  return PIAFS_OK;
}

int piafs_gpu_Solve(piafs_gpu_sim* s, const char* output_dir) {
  if (!s || !output_dir) return fail(PIAFS_ERR_ARGUMENT, "null argument");
  const Deck& d = s->deck;
  const bool write = d.op_file_format == "binary" || d.op_file_format == "bin";
  if (!write && d.op_file_format != "none")
    return fail(PIAFS_ERR_UNSUPPORTED, "op_file_format " + d.op_file_format + " is not supported (binary, none)");
  const bool overwrite = d.op_overwrite != "no";
  int index = 0;
  // a restart fast-forwards the output index (InitializeSolvers.c:240-245)
  if (!overwrite)
    for (int t = 0; t < d.restart_iter; t++)
      if ((t + 1) % d.file_op_iter == 0) index++;
  std::vector<double> host((size_t)s->P.N0 * s->P.N1 * d.nvars);
  std::vector<double> hnu_host;
  // ChemistryWriteSpecies (ChemistryWriteSpecies.c:19-90): per layer iz, the
  // seven species of the LAST layer (the reference copies layer z_i for every
  // iz) and the photon density of layer iz, as op_species_z<iz>[_NNNNN].bin,
  // written before the solution file of the same index (Solve.cpp:56-65)
  auto species = [&]() -> int {
    if (!d.write_species || !s->hnu) return PIAFS_OK;
    const DevParams& P = s->P;
    const int nz = P.nz, nsp = 8, z_i = nz - 1;
    hnu_host.resize((size_t)nz * P.ps);
    CK(cudaMemcpyAsync(hnu_host.data(), s->hnu, hnu_host.size() * sizeof(double), cudaMemcpyDeviceToHost,
                       s->stream));
    CK(cudaStreamSynchronize(s->stream));
    const long long npts = (long long)P.N0 * P.N1;
    std::vector<double> sp((size_t)npts * nsp);
    int width = 1;
    for (int q = nz; q >= 10; q /= 10) width++;          // (int)log10(nz) + 1
    for (int iz = d.write_all_zlocs == "no" ? z_i : 0; iz < nz; iz++) {
      for (long long k = 0; k < npts; k++) {
        const int i = (int)(k % P.N0), j = (int)(k / P.N0);
        for (int m = 0; m < nsp - 1; m++) sp[k * nsp + m] = host[k * d.nvars + P.nflow + P.zstride * z_i + m];
        sp[k * nsp + nsp - 1] = hnu_host[(size_t)iz * P.ps + pidx(P, i, j)];
      }
      char name[96];
      if (overwrite) std::snprintf(name, sizeof(name), "op_species_z%0*d.bin", width, iz);
      else std::snprintf(name, sizeof(name), "op_species_z%0*d_%05d.bin", width, iz, index);
      std::string err;
      if (int r = write_binary(std::string(output_dir) + "/" + name, d, sp.data(), err, nsp)) return fail(r, err);
    }
    return PIAFS_OK;
  };
  auto output = [&]() -> int {
    if (!write) return PIAFS_OK;
    if (int r = piafs_gpu_get_solution(s, host.data())) return r;
    if (int r = species()) return r;
    char name[64];
    if (overwrite) std::snprintf(name, sizeof(name), "op.bin");
    else std::snprintf(name, sizeof(name), "op_%05d.bin", index);
    std::string err;
    if (int r = write_binary(std::string(output_dir) + "/" + name, d, host.data(), err)) return fail(r, err);
    if (!overwrite) index++;
    return PIAFS_OK;
  };
  // Solve.cpp:54-95; on screen steps the CFL before the step
  // (TimePreStep.c:54-65), the residual norm after it (TimePostStep.c:36-54)
  // and the TimePrintStep line (TimePrintStep.c:25-37)
  for (int it = s->iter; it < d.n_iter; it++) {
    if (it == 0) if (int r = output()) return r;
    const auto w0 = std::chrono::steady_clock::now();
    const bool screen = ((it + 1) % d.screen_op_iter) == 0;
    if (screen) {
      double c;
      if (int r = piafs_gpu_ComputeCFL(s, &c)) return r;
    }
    if (int r = run_steps(s, 1, screen)) return r;
    if (screen) {
      const double wct = std::chrono::duration<double>(std::chrono::steady_clock::now() - w0).count();
      std::printf("iter=%7d  t=%1.3E  CFL=%1.3E  norm=%1.4E  wctime: %1.1E (s)  \n", it + 1, s->t, s->last_cfl,
                  s->last_norm, wct);
      std::fflush(stdout);
    }
    if (((it + 1) % d.file_op_iter == 0) && (it + 1 < d.n_iter))
      if (int r = output()) return r;
  }
  return output();
}

int piafs_gpu_TimeRK_norm(piafs_gpu_sim* s, int nsteps, double* norm) {
  if (!s || nsteps < 1 || !norm) return fail(PIAFS_ERR_ARGUMENT, "bad argument");
  if (int r = run_steps(s, nsteps, true)) return r;
  *norm = s->last_norm;
  return PIAFS_OK;
}

// SimWriteErrors (SimulationWriteErrors.c:65-80) for one simulation, after
// CalculateError (CalculateError.c:30-120) against exact.inp when the deck
// directory holds one
int piafs_gpu_WriteErrors(piafs_gpu_sim* s, const char* dir, double solver_runtime, double main_runtime) {
  if (!s || !dir) return fail(PIAFS_ERR_ARGUMENT, "null argument");
  const Deck& d = s->deck;
  const DevParams& P = s->P;
  const long long npts = (long long)P.N0 * P.N1;
  std::vector<double> u((size_t)npts * d.nvars);
  if (int r = piafs_gpu_get_solution(s, u.data())) return r;
  double err3[3] = {-1.0, -1.0, -1.0};
  std::vector<double> ex;
  bool found = false;
  std::string msg;
  if (int r = read_exact(dir, d, ex, found, msg)) return fail(r, msg);
  if (found) {
    double nrm[3] = {0, 0, 0}, e[3] = {0, 0, 0};
    for (size_t k = 0; k < u.size(); k++) {
      const double x = ex[k], dd = u[k] - ex[k];
      nrm[0] += std::fabs(x); nrm[1] += x * x; nrm[2] = std::max(nrm[2], std::fabs(x));
      e[0] += std::fabs(dd); e[1] += dd * dd; e[2] = std::max(e[2], std::fabs(dd));
    }
    nrm[0] /= (double)npts; nrm[1] = std::sqrt(nrm[1] / (double)npts);
    e[0] /= (double)npts; e[1] = std::sqrt(e[1] / (double)npts);
    const double tol = 1e-15;
    const bool rel = nrm[0] > tol && nrm[1] > tol && nrm[2] > tol;
    for (int k = 0; k < 3; k++) err3[k] = rel ? e[k] / nrm[k] : e[k];
  }
  const std::string base(dir);
  FILE* f = std::fopen((base + "/errors.dat").c_str(), "w");
  if (!f) return fail(PIAFS_ERR_IO, "cannot write errors.dat");
  for (int k = 0; k < d.ndims; k++) std::fprintf(f, "%4d ", d.size[k]);
  for (int k = 0; k < d.ndims; k++) std::fprintf(f, "%4d ", 1);
  std::fprintf(f, "%1.16E  ", d.dt);
  std::fprintf(f, "%1.16E %1.16E %1.16E   ", err3[0], err3[1], err3[2]);
  std::fprintf(f, "%1.16E %1.16E\n", solver_runtime, main_runtime);
  std::fclose(f);
  // conservation errors: -1 per variable, as the reference leaves them
  // without conservation_check (Initialize.c:195-196)
  f = std::fopen((base + "/conservation.dat").c_str(), "w");
  if (!f) return fail(PIAFS_ERR_IO, "cannot write conservation.dat");
  for (int k = 0; k < d.ndims; k++) std::fprintf(f, "%4d ", d.size[k]);
  for (int k = 0; k < d.ndims; k++) std::fprintf(f, "%4d ", 1);
  std::fprintf(f, "%1.16E  ", d.dt);
  for (int v = 0; v < d.nvars; v++) std::fprintf(f, "%1.16E ", -1.0);
  std::fprintf(f, "\n");
  std::fclose(f);
  // calls of the hyperbolic, parabolic and source functions: one each per
  // RK stage, the parabolic one only for viscous Navier-Stokes
  // (NavierStokes2DParabolicFunction.c:64-65), the source one when the model
  // has a source (both models do, SourceFunction.c:37-39)
  const long long steps = (long long)s->iter - d.restart_iter;
  f = std::fopen((base + "/function_counts.dat").c_str(), "w");
  if (!f) return fail(PIAFS_ERR_IO, "cannot write function_counts.dat");
  std::fprintf(f, "%d\n", d.n_iter);
  std::fprintf(f, "%lld\n", steps * d.nstages);
  std::fprintf(f, "%lld\n", (P.ndims == 2 && P.viscous) ? steps * d.nstages : 0);
  std::fprintf(f, "%lld\n", steps * d.nstages);
  std::fclose(f);
  if (err3[0] >= 0) {
    std::printf("Computed errors for domain %d:\n", 0);
    std::printf("  L1         Error           : %1.16E\n", err3[0]);
    std::printf("  L2         Error           : %1.16E\n", err3[1]);
    std::printf("  Linfinity  Error           : %1.16E\n", err3[2]);
  }
  std::printf("Solver runtime (in seconds): %1.16E\n", solver_runtime);
  std::printf("Total  runtime (in seconds): %1.16E\n", main_runtime);
  return PIAFS_OK;
}

// ------------------------------------------------- operator-level calls
static int to_soa(piafs_gpu_sim* s, const double* aos, double* soa) {
  launch_aos_to_soa(aos, soa, s->P.npg, s->P.nvars, s->P.ps, s->stream);
  return PIAFS_OK;
}
static int set_top_t(piafs_gpu_sim* s, double t) {
  CK(cudaMemcpyAsync(s->top_t, &t, sizeof(double), cudaMemcpyHostToDevice, s->stream));
  return PIAFS_OK;
}
static int finish(piafs_gpu_sim* s) {
  CK(cudaGetLastError());
  CK(cudaStreamSynchronize(s->stream));
  return PIAFS_OK;
}

int piafs_gpu_RHSFunction(piafs_gpu_sim* s, double* rhs, double* u, double t) {
  if (!s || !rhs || !u) return fail(PIAFS_ERR_ARGUMENT, "null argument");
  if (s->run1d_ctas > 0) {
    Run1D R = s->run1d;
    R.u = u;
    R.rhs = rhs;
    R.nsteps = 1;
    CK(launch_run1d(s->P, R, s->run1d_ctas, s->stream));
    return finish(s);
  }
  double* U = s->scratch;
  double* R = s->Ud[0];   // its ghost entries are never written: zero
  to_soa(s, u, U);
  enqueue_bc(s, U);
  if (int r = set_top_t(s, t)) return r;
  enqueue_rhs(s, R, U, s->top_t, 0.0);
  launch_ghosts_to_aos(s->P, U, u, s->stream);   // all that changed in u
  launch_soa_to_aos(R, rhs, s->P.npg, s->P.nvars, s->P.ps, s->stream);
  return finish(s);
}

int piafs_gpu_HyperbolicFunction(piafs_gpu_sim* s, double* hyp, const double* u, double t) {
  if (!s || !hyp || !u) return fail(PIAFS_ERR_ARGUMENT, "null argument");
  const DevParams& P = s->P;
  double* U = s->scratch;
  double* H = s->Ud[0];   // its ghost entries are never written: zero
  to_soa(s, u, U);
  enqueue_hyp(s, U, H, false);
  launch_soa_to_aos(H, hyp, P.npg, P.nvars, P.ps, s->stream);
  return finish(s);
}

static int visc_or_source(piafs_gpu_sim* s, double* out, const double* u, double t, int visc, int chem) {
  if (!s || !out || !u) return fail(PIAFS_ERR_ARGUMENT, "null argument");
  const DevParams& P = s->P;
  double* U = s->scratch;
  double* R = s->Ud[0];
  to_soa(s, u, U);
  CK(cudaMemsetAsync(R, 0, (size_t)P.nvars * P.ps * sizeof(double), s->stream));
  if (int r = set_top_t(s, t)) return r;
  launch_visc_source(P, U, s->dxinv, s->imap, s->top_t, 0.0, R, visc, chem, s->stream);
  if (chem) enqueue_sponge(s, U, R);   // the sponge is part of SourceFunction
  launch_soa_to_aos(R, out, P.npg, P.nvars, P.ps, s->stream);
  return finish(s);
}
int piafs_gpu_ParabolicFunction(piafs_gpu_sim* s, double* par, const double* u, double t) {
  return visc_or_source(s, par, u, t, 1, 0);
}
int piafs_gpu_SourceFunction(piafs_gpu_sim* s, double* src, const double* u, double t) {
  return visc_or_source(s, src, u, t, 0, 1);
}

int piafs_gpu_ApplyBoundaryConditions(piafs_gpu_sim* s, double* u, double) {
  if (!s || !u) return fail(PIAFS_ERR_ARGUMENT, "null argument");
  to_soa(s, u, s->scratch);
  enqueue_bc(s, s->scratch);
  launch_ghosts_to_aos(s->P, s->scratch, u, s->stream);
  return finish(s);
}

int piafs_gpu_FFunction(piafs_gpu_sim* s, double* f, const double* u, int dir, double) {
  if (!s || !f || !u || dir < 0 || dir >= s->P.ndims) return fail(PIAFS_ERR_ARGUMENT, "bad argument");
  to_soa(s, u, s->scratch);
  launch_flux(s->P, s->scratch, s->fC, dir, s->stream);
  launch_soa_to_aos(s->fC, f, s->P.npg, s->P.nvars, s->P.ps, s->stream);
  return finish(s);
}

int piafs_gpu_InterpolateInterfacesHyp(piafs_gpu_sim* s, double* fI, const double* fC, const double* u, int upw,
                                       int dir, int uflag) {
  if (!s || !fI || !fC || !u || dir < 0 || dir >= s->P.ndims) return fail(PIAFS_ERR_ARGUMENT, "bad argument");
  DevParams P = s->P;
  P.mixed = 0;     // operator-level entry points are FP64
  P.pack_sp = 0;   // and return every interface array as the reference forms it
  to_soa(s, u, s->scratch);
  to_soa(s, fC, s->fC);
  if (P.scheme == CRWENO5 && P.char_interp)
    launch_crweno_char(P, s->scratch, s->fC, s->iface[0], s->iface[1], s->iface[2], s->iface[3], dir, s->crwchar,
                       s->err, s->stream);
  else if (P.scheme != CRWENO5 && P.char_interp)
    launch_weno5_char(P, s->scratch, s->fC, s->iface[0], s->iface[1], s->iface[2], s->iface[3], dir, s->stream);
  else if (P.scheme != CRWENO5)
    launch_weno5(P, s->scratch, s->fC, s->iface[0], s->iface[1], s->iface[2], s->iface[3], dir, s->stream);
  else
    launch_crweno(P, s->scratch, s->fC, s->iface[0], s->iface[1], s->iface[2], s->iface[3], dir, s->err, s->stream);
  const double* src = s->iface[(uflag ? 0 : 2) + (upw > 0 ? 0 : 1)];
  launch_iface_soa_to_aos(src, fI, P.nint[dir], P.nvars, P.pis, s->stream);
  return finish(s);
}

int piafs_gpu_Upwind(piafs_gpu_sim* s, double* fI, const double* fL, const double* fR, const double* uL,
                     const double* uR, const double* u, int dir, double) {
  if (!s || !fI || !fL || !fR || !uL || !uR || !u || dir < 0 || dir >= s->P.ndims)
    return fail(PIAFS_ERR_ARGUMENT, "bad argument");
  const DevParams& P = s->P;
  const long long ni = P.nint[dir];
  to_soa(s, u, s->scratch);
  launch_iface_aos_to_soa(uL, s->iface[0], ni, P.nvars, P.pis, s->stream);
  launch_iface_aos_to_soa(uR, s->iface[1], ni, P.nvars, P.pis, s->stream);
  launch_iface_aos_to_soa(fL, s->iface[2], ni, P.nvars, P.pis, s->stream);
  launch_iface_aos_to_soa(fR, s->iface[3], ni, P.nvars, P.pis, s->stream);
  launch_upwind_iface(P, s->scratch, s->iface[0], s->iface[1], s->iface[2], s->iface[3], s->iface[4], dir, s->stream);
  launch_iface_soa_to_aos(s->iface[4], fI, ni, P.nvars, P.pis, s->stream);
  return finish(s);
}

int piafs_gpu_FirstDerivativePar(piafs_gpu_sim* s, double* Df, const double* f, int dir, int bias, int nv) {
  if (!s || !Df || !f || dir < 0 || dir >= s->P.ndims || nv < 1) return fail(PIAFS_ERR_ARGUMENT, "bad argument");
  launch_first_deriv(s->P, Df, f, dir, bias, nv, s->stream);
  return finish(s);
}

int piafs_gpu_tridiagLU(double* a, double* b, double* c, double* x, int n, int ns) {
  if (!a || !b || !c || !x || n < 0 || ns < 0) return fail(PIAFS_ERR_ARGUMENT, "bad argument");
  if (n == 0 || ns == 0) return PIAFS_OK;
  int* err = nullptr;
  CK(cudaMalloc(&err, sizeof(int)));
  CK(cudaMemset(err, 0, sizeof(int)));
  launch_tridiag(a, b, c, x, n, ns, err, 0);
  int h = 0;
  cudaError_t e = cudaMemcpy(&h, err, sizeof(int), cudaMemcpyDeviceToHost);
  cudaFree(err);
  CK(e);
  CK(cudaGetLastError());
  if (h) return fail(PIAFS_ERR_SINGULAR, "zero pivot in tridiagLU");
  return PIAFS_OK;
}

int piafs_gpu_reciprocal(const double* x, double* y, long long n) {
  if (!x || !y || n < 0) return fail(PIAFS_ERR_ARGUMENT, "bad argument");
  if (n == 0) return PIAFS_OK;
  launch_reciprocal(x, y, n, 0);
  CK(cudaGetLastError());
  CK(cudaDeviceSynchronize());
  return PIAFS_OK;
}

}  // extern "C"
