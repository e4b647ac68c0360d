// sgnb_adjoint_api.cu -- C ABI of the adjoint: gauge records of a frozen-dt BS3(2)
// trajectory and their vector-Jacobian product (no reference counterpart).
//
// Parameters: the bathymetry as element means (Nx * Ny, mapped to the depth statics by
// the bilinear cell interpolant, bathy kind 5 of sgnb_setup.cpp) and the initial free
// surface eta0 (Nd nodal values; h0 = H + eta0, zero velocity, w = p = 0).
// Forward: nsteps BS3(2) steps with the given step sizes (src/solver/rk.cpp:41-54 with
// the fused stage kernels of the solver context), recording eta = h - H at the gauge
// nodes after every step, with the state kept every `checkpoint_every` steps.
// Reverse: for each checkpoint segment, from the last to the first, the segment's
// states are recomputed from its checkpoint; then, step by step backwards, the stage
// derivatives k1, k2 are recomputed and the three right-hand-side VJPs of the step run
// (sgnb_adjoint.cu), carrying the state cotangent and accumulating the cotangents of
// the nodal depths and their gradients, which map back to the element means through the
// transpose of the interpolant on the device (sgnb_cells.cu).
#include "sgnb_ctx.h"

#include <cmath>
#include <cstring>
#include <string>
#include <vector>

using namespace sgnb;

struct sgnb_adj {
  sgnb_ctx* c = nullptr;
  long long N = 0;
  int K = 0, ng = 0, nseg = 0;
  std::vector<double> dts;
  std::vector<long long> gnodes;
  bool haveForward = false;
  double* block = nullptr;    // every device buffer below lives in this allocation
  double* dts_dev = nullptr;
  long long* gnodes_dev = nullptr;
  double* ckpt = nullptr;     // nseg states
  double* seg = nullptr;      // K states
  double* u[2] = {nullptr, nullptr};
  double *k1 = nullptr, *k2 = nullptr, *k3 = nullptr;
  double *lam = nullptr, *acc = nullptr, *y3b = nullptr, *y2b = nullptr;
  double* eta_dev = nullptr;
  double* etab_dev = nullptr;
  CtrlState* ctrl = nullptr;
  VjpArgs V{};
  GatherArgs G{};
};

namespace {

int afail(sgnb_ctx* c, int code, const std::string& m) {
  if (c) c->err = m;
  return code;
}

#define SGNB_ACU(c, call)                                                                \
  do {                                                                                   \
    cudaError_t e_ = (call);                                                             \
    if (e_ != cudaSuccess)                                                               \
      return afail(c, e_ == cudaErrorMemoryAllocation ? SGNB_ERR_NOMEM : SGNB_ERR_CUDA,  \
                   std::string(#call) + ": " + cudaGetErrorName(e_));                   \
  } while (0)

FrTablesDev tables_of(const sgnb_ctx* c) {
  FrTablesDev T{};
  for (int k = 0; k < 25; ++k) { T.D[k] = c->tab.D[k]; T.Df[k] = (float)c->tab.D[k]; }
  for (int k = 0; k < 5; ++k) {
    T.gLp[k] = c->tab.gLp[k]; T.gRp[k] = c->tab.gRp[k];
    T.gLpf[k] = (float)c->tab.gLp[k]; T.gRpf[k] = (float)c->tab.gRp[k];
  }
  return T;
}

cudaError_t fused(const sgnb_ctx* c, int mode, const StageArgs& A, cudaStream_t s) {
  return c->precision == SGNB_FP64_EXACT ? dev::launch_fused_exact(mode, c->C, A, s)
                                         : dev::launch_fused_fast(mode, c->C, A, s);
}

// Scratch of one right-hand-side VJP, carved from `p` (advanced past it).
size_t vjp_scratch_doubles(long long Nd, long long ne) {
  return 2 * 5 * (size_t)Nd + 2 * (size_t)Nd + 2 * (size_t)Nd + 4 * 25 * (size_t)ne;
}
void carve_vjp(VjpArgs& V, double*& p, long long Nd, long long ne) {
  for (int d = 0; d < 2; ++d) { V.Ub[d] = p; p += 5 * Nd; }
  for (int d = 0; d < 2; ++d) { V.Hb[d] = p; p += Nd; }
  V.Hxb = p; p += Nd;
  V.Hyb = p; p += Nd;
  for (int d = 0; d < 2; ++d)
    for (int f = 0; f < 2; ++f) { V.Sn[d][f] = p; p += 25 * ne; }
}
size_t stat_doubles(const sgnb_ctx* c) { return 3 * (size_t)c->Nd; }
void carve_stats(GatherArgs& G, double*& p, const sgnb_ctx* c) {
  G.Hacc = p; p += c->Nd;
  G.Hxacc = p; p += c->Nd;
  G.Hyacc = p; p += c->Nd;
}
CellGrid grid_of(const sgnb_ctx* c) {
  CellGrid g{};
  g.Nx = c->desc.Nx; g.Ny = c->desc.Ny;
  g.Lx = c->desc.Lx; g.Ly = c->desc.Ly;
  g.hx = c->mesh.hx; g.hy = c->mesh.hy;
  for (int k = 0; k < 5; ++k) g.nodes[k] = c->tab.nodes[k];
  for (int k = 0; k < 25; ++k) g.D[k] = c->tab.D[k];
  return g;
}

// One BS3(2) step u -> out at step index n (dt read from the device list).
int step(sgnb_adj* a, const double* u, double* out, long long n) {
  sgnb_ctx* c = a->c;
  cudaStream_t s = c->stream;
  SGNB_ACU(c, cudaMemcpyAsync(&a->ctrl->dt, a->dts_dev + n, sizeof(double), cudaMemcpyDeviceToDevice, s));
  StageArgs A{};
  A.U[0] = A.U[1] = const_cast<double*>(u);
  A.K1[0] = A.K1[1] = a->k1;
  A.K2 = a->k2;
  A.K3 = a->k3;
  A.ctrl = a->ctrl;
  A.partials = c->partials;
  A.in = u;
  A.out = a->k1;
  SGNB_ACU(c, fused(c, 0, A, s));
  A.kin_k2 = 0; A.coef = 0.5; A.out = a->k2;
  SGNB_ACU(c, fused(c, 1, A, s));
  A.kin_k2 = 1; A.coef = 0.75; A.out = a->k3;
  SGNB_ACU(c, fused(c, 1, A, s));
  SGNB_ACU(c, dev::launch_rk_update(u, a->k1, a->k2, a->k3, a->dts_dev, n, out, c->ntot, s));
  return SGNB_OK;
}

}  // namespace

extern "C" {

int sgnb_adj_create(sgnb_ctx* c, long long nsteps, const double* dts, int ngauges,
                    const long long* gauge_nodes, int checkpoint_every, sgnb_adj** out) {
  if (!c || !out || nsteps < 1 || !dts || ngauges < 0 || (ngauges > 0 && !gauge_nodes) ||
      checkpoint_every < 1)
    return afail(c, SGNB_ERR_INVALID, "sgnb_adj_create: bad arguments");
  *out = nullptr;
  if (c->mixed) return afail(c, SGNB_ERR_UNSUPPORTED, "the adjoint runs in FP64 modes");
  if (c->desc.Nx_global > 0 || c->C.ghostL || c->C.ghostR)
    return afail(c, SGNB_ERR_UNSUPPORTED, "the adjoint runs on whole meshes");
  if (c->tab.gauss) return afail(c, SGNB_ERR_UNSUPPORTED, "the adjoint runs on GLL points");
  for (int g = 0; g < ngauges; ++g)
    if (gauge_nodes[g] < 0 || gauge_nodes[g] >= c->Nd)
      return afail(c, SGNB_ERR_INVALID, "gauge node out of range");
  for (long long n = 0; n < nsteps; ++n)
    if (!(dts[n] > 0.0)) return afail(c, SGNB_ERR_INVALID, "step sizes must be > 0");
  SGNB_ACU(c, cudaSetDevice(c->device));
  sgnb_adj* a = new sgnb_adj();
  a->c = c;
  a->N = nsteps;
  a->K = checkpoint_every;
  a->ng = ngauges;
  a->nseg = (int)((nsteps + checkpoint_every - 1) / checkpoint_every);
  a->dts.assign(dts, dts + nsteps);
  a->gnodes.assign(gauge_nodes, gauge_nodes + ngauges);
  const long long S = c->ntot, Nd = c->Nd, ne = (long long)c->desc.Nx * c->desc.Ny;
  const long long segStates = (a->K < nsteps) ? a->K : nsteps;
  constexpr size_t kAlign = 32;  // the states start at a multiple of 256 bytes: row copies need 16
  size_t total = nsteps + (size_t)ngauges + 2 * (size_t)nsteps * (ngauges > 0 ? ngauges : 1) +
                 ((size_t)a->nseg + segStates + 9) * S + vjp_scratch_doubles(Nd, ne) +
                 stat_doubles(c) + sizeof(CtrlState) / sizeof(double) + 8 + kAlign;
  cudaError_t e = cudaMalloc(&a->block, total * sizeof(double));
  if (e != cudaSuccess) { delete a; return afail(c, SGNB_ERR_NOMEM, "sgnb_adj_create: cudaMalloc"); }
  double* p = a->block;
  a->ctrl = reinterpret_cast<CtrlState*>(p); p += (sizeof(CtrlState) + 7) / 8 + 1;
  a->dts_dev = p; p += nsteps;
  a->gnodes_dev = reinterpret_cast<long long*>(p); p += ngauges;
  a->eta_dev = p; p += (size_t)nsteps * (ngauges > 0 ? ngauges : 1);
  a->etab_dev = p; p += (size_t)nsteps * (ngauges > 0 ? ngauges : 1);
  p = a->block + ((size_t)(p - a->block) + kAlign - 1) / kAlign * kAlign;
  a->ckpt = p; p += (size_t)a->nseg * S;
  a->seg = p; p += (size_t)segStates * S;
  for (double** q : {&a->u[0], &a->u[1], &a->k1, &a->k2, &a->k3, &a->lam, &a->acc, &a->y3b, &a->y2b}) {
    *q = p;
    p += S;
  }
  carve_vjp(a->V, p, Nd, ne);
  carve_stats(a->G, p, c);
  e = cudaMemset(a->ctrl, 0, sizeof(CtrlState));
  if (e == cudaSuccess) e = cudaMemcpy(a->dts_dev, dts, nsteps * sizeof(double), cudaMemcpyHostToDevice);
  if (e == cudaSuccess && ngauges > 0)
    e = cudaMemcpy(a->gnodes_dev, gauge_nodes, ngauges * sizeof(long long), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    cudaFree(a->block);
    delete a;
    return afail(c, SGNB_ERR_CUDA, "sgnb_adj_create: upload");
  }
  *out = a;
  return SGNB_OK;
}

int sgnb_adj_destroy(sgnb_adj* a) {
  if (!a) return SGNB_OK;
  cudaSetDevice(a->c->device);
  cudaStreamSynchronize(a->c->stream);
  cudaFree(a->block);
  delete a;
  return SGNB_OK;
}

int sgnb_adj_forward(sgnb_adj* a, const double* means, const double* eta0, double* eta_out) {
  if (!a || !means || !eta0) return afail(a ? a->c : nullptr, SGNB_ERR_INVALID, "NULL argument");
  sgnb_ctx* c = a->c;
  SGNB_ACU(c, cudaSetDevice(c->device));
  cudaStream_t s = c->stream;
  const long long Nd = c->Nd, S = c->ntot;
  // statics from the element means and u0 = (H + eta0, 0, 0, 0, 0), in scratch that the run
  // does not use yet
  const long long nm = (long long)c->desc.Nx * c->desc.Ny;
  SGNB_ACU(c, cudaMemcpyAsync(a->y2b, means, nm * sizeof(double), cudaMemcpyHostToDevice, s));
  SGNB_ACU(c, cudaMemcpyAsync(a->y3b, eta0, Nd * sizeof(double), cudaMemcpyHostToDevice, s));
  auto rw = [](const double* q) { return const_cast<double*>(q); };
  SGNB_ACU(c, dev::launch_cells_statics(grid_of(c), a->y2b, a->y3b, rw(c->C.Hnod), rw(c->C.Hx), rw(c->C.Hy),
                                        rw(c->C.HfX), rw(c->C.HfY), rw(c->C.HfXEnd), rw(c->C.HfYEnd),
                                        a->u[0], s));
  int cur = 0;
  for (long long n = 0; n < a->N; ++n) {
    if (n % a->K == 0)
      SGNB_ACU(c, cudaMemcpyAsync(a->ckpt + (n / a->K) * S, a->u[cur], S * sizeof(double),
                                  cudaMemcpyDeviceToDevice, s));
    if (int rc = step(a, a->u[cur], a->u[cur ^ 1], n)) return rc;
    cur ^= 1;
    if (a->ng > 0)
      SGNB_ACU(c, dev::launch_gauges(a->u[cur], c->C.Hnod, a->gnodes_dev, a->ng,
                                     a->eta_dev + n * a->ng, s));
  }
  // the context holds the final state
  SGNB_ACU(c, cudaMemcpyAsync(c->U[c->cur], a->u[cur], S * sizeof(double), cudaMemcpyDeviceToDevice, s));
  if (eta_out && a->ng > 0)
    SGNB_ACU(c, cudaMemcpyAsync(eta_out, a->eta_dev, a->N * a->ng * sizeof(double),
                                cudaMemcpyDeviceToHost, s));
  SGNB_ACU(c, cudaStreamSynchronize(s));
  a->haveForward = true;
  return SGNB_OK;
}

int sgnb_adj_vjp(sgnb_adj* a, const double* eta_bar, double* grad_means, double* grad_eta0) {
  if (!a || !eta_bar) return afail(a ? a->c : nullptr, SGNB_ERR_INVALID, "NULL argument");
  sgnb_ctx* c = a->c;
  if (!a->haveForward) return afail(c, SGNB_ERR_INVALID, "sgnb_adj_vjp before sgnb_adj_forward");
  SGNB_ACU(c, cudaSetDevice(c->device));
  cudaStream_t s = c->stream;
  const long long S = c->ntot, Nd = c->Nd;
  const int ng = a->ng;
  if (ng > 0)
    SGNB_ACU(c, cudaMemcpyAsync(a->etab_dev, eta_bar, a->N * ng * sizeof(double),
                                cudaMemcpyHostToDevice, s));
  SGNB_ACU(c, cudaMemsetAsync(a->G.Hacc, 0, stat_doubles(c) * sizeof(double), s));
  SGNB_ACU(c, cudaMemsetAsync(a->lam, 0, S * sizeof(double), s));
  if (ng > 0)
    SGNB_ACU(c, dev::launch_gauges_back(a->lam, a->gnodes_dev, ng, a->etab_dev + (a->N - 1) * ng, s));
  const FrTablesDev T = tables_of(c);
  double* lam = a->lam;
  double* acc = a->acc;
  for (int sg = a->nseg - 1; sg >= 0; --sg) {
    const long long n0 = (long long)sg * a->K;
    const long long n1 = (n0 + a->K < a->N) ? n0 + a->K : a->N;
    // recompute the segment's states u_n0 .. u_{n1-1}
    SGNB_ACU(c, cudaMemcpyAsync(a->seg, a->ckpt + sg * S, S * sizeof(double), cudaMemcpyDeviceToDevice, s));
    for (long long n = n0; n + 1 < n1; ++n)
      if (int rc = step(a, a->seg + (n - n0) * S, a->seg + (n + 1 - n0) * S, n)) return rc;
    for (long long n = n1 - 1; n >= n0; --n) {
      const double* u = a->seg + (n - n0) * S;
      const double dt = a->dts[n];
      // k1 = R(u), k2 = R(u + dt/2 k1)
      SGNB_ACU(c, cudaMemcpyAsync(&a->ctrl->dt, a->dts_dev + n, sizeof(double), cudaMemcpyDeviceToDevice, s));
      StageArgs A{};
      A.U[0] = A.U[1] = const_cast<double*>(u);
      A.K1[0] = A.K1[1] = a->k1;
      A.K2 = a->k2;
      A.K3 = a->k3;
      A.ctrl = a->ctrl;
      A.partials = c->partials;
      A.in = u;
      A.out = a->k1;
      SGNB_ACU(c, fused(c, 0, A, s));
      A.kin_k2 = 0; A.coef = 0.5; A.out = a->k2;
      SGNB_ACU(c, fused(c, 1, A, s));
      // u_{n+1} = u + dt (2/9 k1 + 1/3 k2 + 4/9 k3), k3 = R(u + 3dt/4 k2), k2 = R(u + dt/2 k1)
      VjpArgs V = a->V;
      GatherArgs G = a->G;
      V.u = u;
      V.k = a->k2; V.acoef = 0.75 * dt;
      V.ra = lam; V.rb = nullptr; V.alpha = (4.0 / 9.0) * dt; V.beta = 0.0;
      G.ybar = a->y3b; G.uacc = acc; G.lam = lam; G.init = 1;
      SGNB_ACU(c, dev::launch_vjp_rhs(c->C, T, V, G, s));
      V.k = a->k1; V.acoef = 0.5 * dt;
      V.ra = lam; V.rb = a->y3b; V.alpha = dt / 3.0; V.beta = 0.75 * dt;
      G.ybar = a->y2b; G.init = 0; G.lam = nullptr;
      SGNB_ACU(c, dev::launch_vjp_rhs(c->C, T, V, G, s));
      V.k = nullptr; V.acoef = 0.0;
      V.ra = lam; V.rb = a->y2b; V.alpha = (2.0 / 9.0) * dt; V.beta = 0.5 * dt;
      G.ybar = nullptr;
      SGNB_ACU(c, dev::launch_vjp_rhs(c->C, T, V, G, s));
      double* t = lam; lam = acc; acc = t;
      if (n >= 1 && ng > 0)
        SGNB_ACU(c, dev::launch_gauges_back(lam, a->gnodes_dev, ng, a->etab_dev + (n - 1) * ng, s));
    }
  }
  // lam = dL/du0; h0 = H + eta0
  if (grad_eta0)
    SGNB_ACU(c, cudaMemcpyAsync(grad_eta0, lam, Nd * sizeof(double), cudaMemcpyDeviceToHost, s));
  if (grad_means) {
    const long long nm = (long long)c->desc.Nx * c->desc.Ny;
    SGNB_ACU(c, dev::launch_cells_back(grid_of(c), a->G, lam, a->gnodes_dev, ng, a->N, a->etab_dev, a->y3b,
                                       a->y2b, s));
    SGNB_ACU(c, cudaMemcpyAsync(grad_means, a->y2b, nm * sizeof(double), cudaMemcpyDeviceToHost, s));
  }
  SGNB_ACU(c, cudaStreamSynchronize(s));
  return SGNB_OK;
}

int sgnb_rhs_vjp(sgnb_ctx* c, const double* U, const double* Rbar, double* Ubar,
                 double* Hnod_bar, double* Hx_bar, double* Hy_bar, double* HfX_bar,
                 double* HfY_bar, double* HfXEnd_bar, double* HfYEnd_bar) {
  if (!c || !U || !Rbar || !Ubar) return afail(c, SGNB_ERR_INVALID, "NULL argument");
  if (c->mixed) return afail(c, SGNB_ERR_UNSUPPORTED, "the adjoint runs in FP64 modes");
  SGNB_ACU(c, cudaSetDevice(c->device));
  cudaStream_t s = c->stream;
  const long long S = c->ntot, Nd = c->Nd, ne = (long long)c->desc.Nx * c->desc.Ny;
  double* block = nullptr;
  const size_t total = 3 * (size_t)S + vjp_scratch_doubles(Nd, ne) + stat_doubles(c);
  SGNB_ACU(c, cudaMalloc(&block, total * sizeof(double)));
  double* p = block;
  double* Ud = p; p += S;
  double* Rd = p; p += S;
  double* Ubd = p; p += S;
  VjpArgs V{};
  GatherArgs G{};
  carve_vjp(V, p, Nd, ne);
  carve_stats(G, p, c);
  cudaError_t e = cudaMemcpyAsync(Ud, U, S * sizeof(double), cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(Rd, Rbar, S * sizeof(double), cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaMemsetAsync(G.Hacc, 0, stat_doubles(c) * sizeof(double), s);
  V.u = Ud; V.k = nullptr; V.acoef = 0.0;
  V.ra = Rd; V.rb = nullptr; V.alpha = 1.0; V.beta = 0.0;
  G.ybar = nullptr; G.uacc = Ubd; G.lam = nullptr; G.init = 1;
  if (e == cudaSuccess) e = dev::launch_vjp_rhs(c->C, tables_of(c), V, G, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(Ubar, Ubd, S * sizeof(double), cudaMemcpyDeviceToHost, s);
  auto down = [&](double* host, const double* dev) {
    if (e == cudaSuccess && host)
      e = cudaMemcpyAsync(host, dev, Nd * sizeof(double), cudaMemcpyDeviceToHost, s);
  };
  down(Hnod_bar, G.Hacc); down(Hx_bar, G.Hxacc); down(Hy_bar, G.Hyacc);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  cudaFree(block);
  if (e != cudaSuccess) return afail(c, SGNB_ERR_CUDA, std::string("sgnb_rhs_vjp: ") + cudaGetErrorName(e));
  // the face depths cancel in R
  auto none = [](double* o, long long n) { if (o) std::memset(o, 0, n * sizeof(double)); };
  none(HfX_bar, 5 * ne); none(HfY_bar, 5 * ne); none(HfXEnd_bar, 5LL * c->desc.Ny); none(HfYEnd_bar, 5LL * c->desc.Nx);
  return SGNB_OK;
}

}  // extern "C"
