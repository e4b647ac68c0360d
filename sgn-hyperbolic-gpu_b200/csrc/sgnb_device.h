// sgnb_device.h -- parameter blocks shared by the host code and the sm_100a kernels.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <utility>

namespace sgnb {

// The GLL differentiation matrix and the g_DG correction derivatives split into their even
// and odd halves (D changes sign when its rows and columns are reversed, gRp is minus the
// reversed gLp): with e_k = F_k + F_{4-k} - 2 F_2 and o_k = F_k - F_{4-k},
//   (D F)_m = E_m + O_m, (D F)_{4-m} = O_m - E_m,
//   E_m = A[2m] e_0 + A[2m+1] e_1 + b[m] (jl + jr)      (m = 0, 1)
//   O_m = B[2m] o_0 + B[2m+1] o_1 + a[m] (jl - jr)      (m = 0, 1, 2)
// including the lifts jl gLp + jr gRp of the face jumps.
struct LineTables {
  double A[4], B[6], a[3], b[2];
};

// Everything the fused right-hand-side kernel needs besides the state: mesh size,
// boundary kinds, the physical constants in the exact forms the reference multiplies
// them in (src/physics/sgn_flux2d.h:89-161), the FR tables, and the bathymetry statics.
struct RhsConsts {
  int Nx, Ny;          // elements per direction
  int bcx, bcy;        // 0 periodic, 1 reflective wall
  long long Nd;        // nodes per field = 25 Nx Ny
  double g;            // gravity
  double halfg;        // 0.5 * g
  double gamma;        // dispersion parameter
  double c2;           // c * c
  double mc2;          // (-c) * c, the ncp coefficient
  double m2c2;         // -2.0 * c2, the relaxation-source coefficient
  double n2g;          // nManning^2 * g: Manning friction (sgn_flux2d.h:135-142)
  int manning;         // friction on (nManning != 0)
  int pad_;
  double Jx, Jy;       // affine Jacobians hx/2, hy/2
  double iJx, iJy;     // 1/Jx, 1/Jy (fast mode)
  double D[25];        // GLL differentiation matrix, row-major
  double gLp[5], gRp[5];  // g_DG correction derivatives
  // bathymetry statics (device pointers)
  const double* Hnod;    // nodal H, Nd
  const double* Hx;      // nodal dH/dx, Nd
  const double* Hy;      // nodal dH/dy, Nd
  const double* HfX;     // H at the left edge of each element, 5 per element
  const double* HfY;     // H at the bottom edge of each element
  const double* HfXEnd;  // H on the right domain edge (walls), 5 per row
  const double* HfYEnd;  // H on the top domain edge (walls), 5 per column
  // slab edges (x decomposition): the neighbours' trace nodes across the left and right
  // edge, [field][row][transverse node], stage inputs formed by the neighbours; NULL: the
  // edge follows bcx (periodic wrap or wall)
  const double* ghostL;
  const double* ghostR;
  // fused edge exchange of the intermediate stages: the next stage's inputs at the slab's
  // edge nodes, written by this launch into the neighbours' ghost arrays (the left
  // neighbour's right ghost, the right neighbour's left ghost; another device's memory in
  // a multi-device run); NULL: none
  double* edgeL;
  double* edgeR;
  // Gauss-Legendre points: face interpolation rows, and the face traces of every element
  // formed by a pre-pass, [face: 0 left, 1 right, 2 bottom, 3 top][field][element][node]
  double lL[5], lR[5];
  double* tr;
  int gauss;
  int pad2_;
  // the differentiation and correction tables rounded to FP32 (the mixed mode's FP32
  // contractions)
  float Df[25], gLpf[5], gRpf[5];
  LineTables eo;  // the line kernels' split tables; sym: the tables have the symmetry they need
  int sym;
  int bulk;       // bulk row copies: the rows of FP64 buffers start and end at multiples of 16
                  // bytes (Nx even)
  int form;       // the exact line kernels' form for this mesh (exact_form)
};

// What the line kernels (fast mode) take of RhsConsts.
struct LineConsts {
  int Nx, Ny, bcx, bcy;
  long long Nd;
  double g, halfg, gamma, c2, n2g, iJx, iJy;
  const double* Hnod;
  const double *ghostL, *ghostR;
  double *edgeL, *edgeR;
  int bulk, pad_;
};
inline LineConsts line_consts(const RhsConsts& C) {
  LineConsts L{};
  L.Nx = C.Nx; L.Ny = C.Ny; L.bcx = C.bcx; L.bcy = C.bcy; L.Nd = C.Nd;
  L.g = C.g; L.halfg = C.halfg; L.gamma = C.gamma; L.c2 = C.c2; L.n2g = C.n2g;
  L.iJx = C.iJx; L.iJy = C.iJy;
  L.Hnod = C.Hnod;
  L.ghostL = C.ghostL; L.ghostR = C.ghostR; L.edgeL = C.edgeL; L.edgeR = C.edgeR;
  L.bulk = C.bulk;
  return L;
}

// Device-resident state of the adaptive integrator: the scalar loop variables of
// src/solver/rk.cpp:67-164 plus the index of the buffer pair that holds u and k1.
struct CtrlState {
  double t, dt, tEnd, errPrev;
  double tReached, dtLast, maxNormLast, errLast;
  long long accepted, rejected, rhsEvals, attempts;
  int cur;     // U[cur] holds u, K1[cur] holds k1
  int done;    // 0 running, 1 reached tEnd, 2 dt fell below dtMin, 3 non-finite error
  int frozen;  // 1: replay the dt list (every attempt accepted)
  int pad;
  double atol, rtol, dtMin, dtMax, safety, facMin, facMax, alpha, beta;
  const double* dtList;  // frozen-dt replay list
  long long nList;
  double* log;           // attempt log: (t, dt, errNorm, accepted) per attempt
  long long logCap;      // capacity of the log in attempts
  long long maxAccepted; // > 0: stop after this many accepted steps
  long long attemptCap;  // the device-side loop hands back to the host at this attempt count
};

#ifdef __CUDACC__
// Programmatic dependent launch: a kernel launched by launch_dependent may start while the
// kernel before it in its stream still runs, once all of that one's CTAs have called
// let_next_start or left; it touches no global memory before wait_for_previous, which returns
// when the kernel before it has completed with its writes visible (every kernel launched this
// way calls it first, in all threads). What that kernel wrote is not read-only over this kernel's
// life, so it is read with ordinary loads, never through the non-coherent path (no ld.global.nc,
// and no const __restrict__ pointers, which let the compiler choose it). Launch latency and the kernel's own set-up then overlap the
// previous kernel's end: a right-hand side of 128 x 64 elements every 8.16 us instead of 10.24
// (8.91 with let_next_start first thing, when the waiting CTAs take room that the running ones'
// L1 would use). Not while a graph is captured: its nodes start faster than these edges
// (20 adaptive steps of that mesh 936 us without, 954 us with them).
__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;\n"); }
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
template <class... P, class... A>
inline cudaError_t launch_dependent(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                                    A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  const cudaError_t e = cudaStreamIsCapturing(s, &capture);
  if (e != cudaSuccess) return e;
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = capture == cudaStreamCaptureStatusNone ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

// The controller's per-launch values (buffer index, dt, tolerances) read again late in a
// stage kernel. The controller, which writes them, is another kernel: the state does not change
// after wait_for_previous, and after the first read on an SM the line comes from L1. Asm
// statements, so the compiler neither merges them with the kernel's first read nor keeps that
// value live in registers in between.
struct CtrlReload {
  int cur;
  double dt, atol, rtol;
};
__device__ __forceinline__ CtrlReload ctrl_reload(const CtrlState* c) {
  CtrlReload r;
  asm volatile("ld.global.s32 %0, [%1];" : "=r"(r.cur) : "l"(&c->cur));
  asm volatile("ld.global.f64 %0, [%1];" : "=d"(r.dt) : "l"(&c->dt));
  asm volatile("ld.global.f64 %0, [%1];" : "=d"(r.atol) : "l"(&c->atol));
  asm volatile("ld.global.f64 %0, [%1];" : "=d"(r.rtol) : "l"(&c->rtol));
  return r;
}

// Block-wide copy of two parameter blocks (W1 and W2 32-bit words) from global to shared
// memory, by NT threads: every load of a thread is issued before its first store, so the
// copy costs one memory round trip however many words a thread moves.
template <int W1, int W2, int NT>
__device__ __forceinline__ void block_copy2(unsigned* d1, const unsigned* s1, unsigned* d2,
                                            const unsigned* s2) {
  constexpr int R1 = (W1 + NT - 1) / NT, R2 = (W2 + NT - 1) / NT;
  unsigned t1[R1], t2[R2];
  const int tid = threadIdx.x;
#pragma unroll
  for (int r = 0; r < R1; ++r)
    if (tid + r * NT < W1) t1[r] = s1[tid + r * NT];
#pragma unroll
  for (int r = 0; r < R2; ++r)
    if (tid + r * NT < W2) t2[r] = s2[tid + r * NT];
#pragma unroll
  for (int r = 0; r < R1; ++r)
    if (tid + r * NT < W1) d1[tid + r * NT] = t1[r];
#pragma unroll
  for (int r = 0; r < R2; ++r)
    if (tid + r * NT < W2) d2[tid + r * NT] = t2[r];
}

// Tile loads by the tensor-memory accelerator, completed on a shared-memory mbarrier
// (one elected thread initialises it and issues the copies; every thread waits on its
// phase with a bounded number of tries). Loads from this device's own buffers only, each
// into the issuing CTA's own shared memory.
__device__ __forceinline__ unsigned smem_addr(const void* p) {
  return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(unsigned mb) {
  asm volatile("mbarrier.init.shared.b64 [%0], 1;\n" ::"r"(mb) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned mb, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared.b64 _, [%0], %1;\n" ::"r"(mb), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned mb, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(mb), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ void mbar_inval(unsigned mb) {
  asm volatile("mbarrier.inval.shared.b64 [%0];\n" ::"r"(mb) : "memory");
}
__device__ __forceinline__ void tma_load_3d(unsigned dst, const CUtensorMap* map, int x, int y,
                                            int z, unsigned mb) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3, %4}], [%5];\n" ::"r"(dst),
      "l"(map), "r"(x), "r"(y), "r"(z), "r"(mb)
      : "memory");
}
__device__ __forceinline__ void tma_load_2d(unsigned dst, const CUtensorMap* map, int x, int y,
                                            unsigned mb) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3}], [%4];\n" ::"r"(dst),
      "l"(map), "r"(x), "r"(y), "r"(mb)
      : "memory");
}
// Tries before a tile-load wait gives up (each try waits a while in hardware): far more
// than any load takes, so a give-up means a fault, reported as a non-finite result.
constexpr int kTmaTries = 1 << 20;
#endif

// The mixed-precision mode's counterparts (intermediate stage): the FP32 stage buffers as
// [field][element row][Nx * 25] with a [1][4][200] box (one field of one tile per copy),
// the nodal depth as for the FP64 kernels.
struct TileMapsM {
  CUtensorMap K1[2], K2, K3, H;
  int ok;
};

// Buffers of one fused launch.
struct StageArgs {
  const double* in;   // MODE_RHS input state
  double* out;        // MODE_RHS / MODE_STAGE output derivative
  double* U[2];       // state ping-pong pair
  double* K1[2];      // k1 / k4 ping-pong pair
  double* K2;
  double* K3;
  int kin_k2;         // MODE_STAGE: add k2 (1) or k1 = K1[cur] (0) to u
  double coef;        // MODE_STAGE, MODE_CAND: 0.5 or 0.75
  const CtrlState* ctrl;
  double* partials;   // MODE_FSAL: 3 doubles per CTA (sum r^2, max |r|, NaN count)
  int cand, pad_;     // MODE_STAGES: the third stage, with the candidate
};

// Whether the rows of every buffer of a launch can move by bulk copies: aligned rows (C.bulk) in
// aligned buffers (the right-hand side's input and output are the caller's).
inline bool bulk_rows(const RhsConsts& C, const StageArgs& A) {
  auto ok = [](const void* p) { return ((unsigned long long)p & 15) == 0; };
  return C.bulk && ok(A.in) && ok(A.out) && ok(A.U[0]) && ok(A.U[1]) && ok(A.K1[0]) && ok(A.K1[1]) &&
         ok(A.K2) && ok(A.K3) && ok(C.Hnod);
}

// Buffers of one mixed-precision launch: FP64 state, FP32 stage derivatives.
struct StageArgsM {
  const double* in;   // MODE_RHS input state
  double* outd;       // MODE_RHS output derivative (FP64)
  float* out;         // MODE_STAGE output derivative
  double* U[2];
  float* K1[2];
  float* K2;
  float* K3;
  int kin_k2;
  double coef;
  const CtrlState* ctrl;
  double* partials;
};

// Differentiation and correction tables (adjoint, mixed batch).
struct FrTablesDev {
  double D[25], gLp[5], gRp[5];
  float Df[25], gLpf[5], gRpf[5];  // FP32 roundings (mixed mode)
};

// Work list of a batched launch: tile t belongs to instance tile_inst[t] and is that
// instance's local tile t - tile_start[inst]; per-instance constants and buffers.
struct BatchArgs {
  LineTables tables;    // shared by every instance (P = 4 GLL)
  const LineConsts* consts;
  const StageArgs* args;
  const int* tile_inst;
  const long long* tile_start;
  long long ntiles;
  int kin_k2;
  double coef;
};

// Vector-Jacobian product of R at a stage input y = u (k == nullptr) or u + acoef k,
// with the cotangent alpha ra + beta rb (rb optional). Scratch written by the line
// kernels and read by the gather kernel:
//   Ub[d]   [5 Nd]   cotangent of each node from its direction-d line
//   Hb[d]   [Nd]     nodal-depth cotangent from the direction-d lines
//   Hxb,Hyb [Nd]     cotangents of dH/dx, dH/dy (x lines: sources)
//   Sn[d][f][5 ne 5] cotangent of the neighbour's trace node across face f (0 low,
//                    1 high) of line (e, j), field-minor
struct VjpArgs {
  const double* u;
  const double* k;
  double acoef;
  const double* ra;
  const double* rb;
  double alpha, beta;
  double* Ub[2];
  double* Hb[2];
  double* Hxb;
  double* Hyb;
  double* Sn[2][2];
};

// Outputs of the gather: ybar (optional) = the node cotangent of R's input;
// uacc = lam + ybar (init; lam optional) or uacc += ybar; statics accumulators +=.
struct GatherArgs {
  double* ybar;
  double* uacc;
  const double* lam;
  int init;
  double* Hacc;
  double* Hxacc;
  double* Hyacc;
};

// Work list of a batched mixed-precision launch (8x4 tiles), as BatchArgs.
struct BatchArgsM {
  FrTablesDev tables;
  const RhsConsts* consts;
  const StageArgsM* args;
  const int* tile_inst;
  const long long* tile_start;
  long long ntiles;
  int kin_k2;
  double coef;
};

// The mesh and tables of the depth interpolant of element means (adjoint), Nx x Ny cells that
// are the mesh's elements.
struct CellGrid {
  int Nx, Ny;
  double Lx, Ly, hx, hy;
  double nodes[5], D[25];
};

namespace dev {
// Batched mixed-precision launch: `blocks` persistent CTAs, or one CTA per tile (0).
cudaError_t launch_mixed_batch(int mode, int blocks, const BatchArgsM& B, cudaStream_t s);
cudaError_t prepare_mixed_batch(int blocks);

// Out-of-range access counts of the checked build, per translation unit.
cudaError_t read_oob_exact(unsigned long long* out, bool reset);
cudaError_t read_oob_fast(unsigned long long* out, bool reset);
cudaError_t read_oob_line(unsigned long long* out, bool reset);
cudaError_t read_oob_batch(unsigned long long* out, bool reset);
cudaError_t read_oob_mixed(unsigned long long* out, bool reset);
cudaError_t read_oob_adjoint(unsigned long long* out, bool reset);
cudaError_t read_oob_cells(unsigned long long* out, bool reset);

// The fast mode's reciprocal (fn 0) and square root (fn 1) elementwise, for tests.
cudaError_t launch_fast_math(int fn, const double* x, double* y, long long n, cudaStream_t s);

// Error partials of every slab of a decomposed mesh, in slab order: slab s holds blocks
// start[s] .. start[s+1]-1 at p[s] (3 doubles per block).
constexpr int kMaxSlabs = 32;
struct SlabPartials {
  const double* p[kMaxSlabs];
  long long start[kMaxSlabs + 1];
  int ns;
};
cudaError_t launch_controller_slabs(CtrlState* c, const SlabPartials& L, long long n,
                                    cudaStream_t s);

// Slab edges: the stage inputs of the first and last element columns' edge nodes
// (a = 0 / a = 4), [field][row][node], for the neighbours' ghosts. mode 0: rhs of in;
// 1: intermediate stage (kin_k2, coef of A); 2: the candidate that the third stage left.
cudaError_t launch_pack_ghosts(int mode, const RhsConsts& C, const StageArgs& A, double* sendL,
                               double* sendR, cudaStream_t s);

// Depth statics of the means (the bits of the host set-up) and the state (H + eta0, 0, 0, 0, 0).
cudaError_t launch_cells_statics(const CellGrid& g, const double* means, const double* eta0, double* Hnod,
                                 double* Hx, double* Hy, double* HfX, double* HfY, double* HfXEnd,
                                 double* HfYEnd, double* u0, cudaStream_t s);
// Their transpose: from the statics' cotangents G, the initial depth's lam (Nd) and the gauge
// records' etab [nsteps][ng] to the gradient of the means. Hb: scratch (Nd).
cudaError_t launch_cells_back(const CellGrid& g, const GatherArgs& G, const double* lam,
                              const long long* gauges, int ng, long long nsteps, const double* etab,
                              double* Hb, double* grad, cudaStream_t s);

// Adjoint kernels (FP64, fast arithmetic).
cudaError_t launch_vjp_rhs(const RhsConsts& C, const FrTablesDev& T, const VjpArgs& A,
                           const GatherArgs& G, cudaStream_t s);
cudaError_t launch_rk_update(const double* u, const double* k1, const double* k2,
                             const double* k3, const double* dts, long long step, double* out,
                             long long n, cudaStream_t s);
cudaError_t launch_gauges(const double* U, const double* Hnod, const long long* nodes, int ng,
                          double* eta, cudaStream_t s);
cudaError_t launch_gauges_back(double* lam, const long long* nodes, int ng, const double* etab,
                               cudaStream_t s);

// Launchers (one translation unit per arithmetic mode).
cudaError_t launch_fused_exact(int mode, const RhsConsts& C, const StageArgs& A, cudaStream_t s);
cudaError_t launch_fused_fast(int mode, const RhsConsts& C, const StageArgs& A, cudaStream_t s);
cudaError_t launch_line(int mode, const RhsConsts& C, const StageArgs& A, cudaStream_t s);
// Raise the shared memory of a context's kernels (its friction and point set; ghost: those with
// slab edges), which loads their code.
cudaError_t prepare_line(const RhsConsts& C, bool ghost);
cudaError_t prepare_fused_exact(const RhsConsts& C, bool ghost);
cudaError_t prepare_fused_fast(const RhsConsts& C, bool ghost);
cudaError_t launch_fused_mixed(int mode, const RhsConsts& C, const StageArgsM& A,
                               cudaStream_t s, const TileMapsM* M = nullptr);
// tma: the stages that add k take their tiles by tensor maps (whole tiles, no friction)
cudaError_t prepare_fused_mixed(const RhsConsts& C, bool tma);
int fused_grid_blocks(int Nx, int Ny);
// Batched launch (fast mode): tile shape shape_id (0: 6x4 elements, 1: 12x2, 2: 24x1);
// `blocks` persistent CTAs looping over the work list, or one CTA per tile when blocks == 0.
cudaError_t launch_fused_batch(int mode, int shape_id, int blocks, const BatchArgs& B,
                               cudaStream_t s);
cudaError_t prepare_fused_batch(int shape_id, int blocks);
int batch_tile_tx(int shape_id);
int batch_tile_ty(int shape_id);
int line_grid_blocks(int Nx, int Ny);
// The exact line kernels' form for a mesh (slab: one of a decomposed one), and the number of its
// tiles.
int exact_form(int Nx, int Ny, bool slab);
int exact_grid_blocks(const RhsConsts& C);
// rk4Step: c->dt = dts[i], and the final update u += dt/6 (k1 + 2 k2 + 2 k3 + k4) over n values
cudaError_t launch_rk4_set_dt(CtrlState* c, const double* dts, long long i, cudaStream_t s);
cudaError_t launch_rk4_update(double* u, const double* k1, const double* k2, const double* k3,
                              const double* k4, const CtrlState* c, long long n, int sms,
                              cudaStream_t s);

// Controller of one adaptive attempt: deterministic reduction of the per-CTA error
// partials, accept/reject, PI step-size update and the next attempt's dt.
// The controller as the last node of the body of a device-side WHILE loop (a conditional
// node of a CUDA graph): it also sets the loop condition, false once the run is done or
// the attempt count has reached attemptCap.
cudaError_t launch_controller_loop(CtrlState* c, const double* partials, int nblk, long long n,
                                   cudaGraphConditionalHandle loop, cudaStream_t s);
// Batched form of the loop controller: block i runs instance i's controller; every block
// counts whether its instance still runs, and the last block to finish (an atomic ticket,
// no waiting) sets the condition (any instance running) and clears the two counters.
cudaError_t launch_controller_batch_loop(CtrlState* ctrls, const double* const* partials,
                                         const int* nblk, const long long* n, int ninst,
                                         int* counters, cudaGraphConditionalHandle loop,
                                         cudaStream_t s);
cudaError_t launch_controller(CtrlState* c, const double* partials, int nblk,
                              long long n, cudaStream_t s);
// Largest eta = h - H inside a window, with its node: (value, index) per block.
cudaError_t launch_eta_max(const RhsConsts& C, const double* U, double x0, double x1, double y0,
                           double y1, double hx, double hy, int ex0, const double* xi,
                           double* out, int nblk, cudaStream_t s);
// Element means of eta, u, v, p, H (out[f * ne + e]), as the reference's VTK writer forms them.
cudaError_t launch_elem_means(const RhsConsts& C, const double* U, const double* qw, double* out,
                              cudaStream_t s);
// eta at the given nodes (gauges).
cudaError_t launch_sample_eta(const double* U, const double* Hnod, const long long* nodes, int n,
                              double* out, cudaStream_t s);
// Reductions over the uploaded state (diagnostics).
cudaError_t launch_reduce_diag(int what, const RhsConsts& C, const double* U,
                               const double* qw, double* out_partials, int nblk,
                               cudaStream_t s);
}  // namespace dev

}  // namespace sgnb
