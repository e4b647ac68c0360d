// sgnb_kernels_fast.cu -- the fast arithmetic mode's dispatch, its Gauss-point kernels and the
// slab packs. Built with -fmad=true: FMA contraction, reciprocals of h and of the Jacobians.
// Agrees with the reference to round-off: one rounding of the hydrostatic flux, times the
// differentiation matrix over J, relative to a field's largest value (1e-13 per field on meshes of
// elements of order one, 2e-13 at J = 0.01). The kernels on GLL points are in
// sgnb_kernels_line.cu.
#define SGNB_EXACT false
#include "sgnb_kernels_inst.cuh"

namespace sgnb {
namespace dev {
cudaError_t launch_fused_fast(int mode, const RhsConsts& C, const StageArgs& A, cudaStream_t s) {
  // FR tables without the reflection symmetry of the GLL ones (given by the caller): the exact
  // mode's kernels, which take any tables
  if (!C.gauss && !C.sym) return launch_fused_exact(mode, C, A, s);
  if (!C.gauss) return launch_line(mode, C, A, s);
  switch (mode) {
    case MODE_RHS: return launch_gauss<MODE_RHS>(C, A, s);
    case MODE_STAGE: return launch_gauss<MODE_STAGE>(C, A, s);
    case MODE_FSAL: return launch_gauss<MODE_FSAL>(C, A, s);
    case MODE_CAND: return launch_gauss<MODE_CAND>(C, A, s);
    default: return cudaErrorInvalidValue;
  }
}
cudaError_t prepare_fused_fast(const RhsConsts& C, bool ghost) {
  if (!C.gauss) return C.sym ? prepare_line(C, ghost) : prepare_fused_exact(C, ghost);
  return C.manning ? prepare_variant<true>() : prepare_variant<false>();
}

// The checked build's out-of-range count of this translation unit's kernels (reset: then
// zero it); cudaErrorNotSupported in the normal build.
cudaError_t read_oob_fast(unsigned long long* out, bool reset) {
#ifdef SGNB_CHECKED
  cudaError_t e = cudaMemcpyFromSymbol(out, g_sgnb_oob, sizeof(*out));
  if (e == cudaSuccess && reset) {
    const unsigned long long z = 0;
    e = cudaMemcpyToSymbol(g_sgnb_oob, &z, sizeof(z));
  }
  return e;
#else
  *out = 0;
  (void)reset;
  return cudaErrorNotSupported;
#endif
}

// The fast mode's reciprocal (fn 0) and square root (fn 1) on a device array, for tests.
__global__ void k_fast_math(int fn, const double* __restrict__ x, double* __restrict__ y,
                            long long n) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] = fn == 0 ? fast_rcp(x[i]) : fast_sqrt(x[i]);
}

cudaError_t launch_fast_math(int fn, const double* x, double* y, long long n, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_fast_math<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(fn, x, y, n);
  return cudaGetLastError();
}

// Slab edges: one thread per (side, field, row, transverse node). Side 0 reads the first
// element column's left nodes (a = 0) into sendL, side 1 the last column's right nodes
// (a = P) into sendR; both [field][row][node]. The stage inputs are formed with the same
// explicitly rounded combinations as the fused kernels' own and halo nodes, so a
// neighbour's ghost holds the bits its own tile would have formed.
__global__ void k_pack_ghosts(int mode, const RhsConsts C, const StageArgs A, double* sendL,
                              double* sendR) {
  const long long per = (long long)NV * C.Ny * NP;
  const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= 2 * per) return;
  if (mode != 0 && A.ctrl->done) return;
  const int side = (int)(q / per);
  const long long r = q - side * per;
  const int t = (int)(r % NP), ey = (int)((r / NP) % C.Ny), v = (int)(r / ((long long)NP * C.Ny));
  const int ex = side == 0 ? 0 : C.Nx - 1, a = side == 0 ? 0 : NP - 1;
  const long long g = (long long)v * C.Nd + ((long long)ex + (long long)C.Nx * ey) * NPP + a + NP * t;
  double val;
  if (mode == 0) {
    val = A.in[g];
  } else {
    const int cur = A.ctrl->cur;
    const double dt = A.ctrl->dt;
    if (mode == 1) {
      const double* k = A.kin_k2 ? A.K2 : A.K1[cur];
      val = stage_axpy(A.U[cur][g], A.coef * dt, k[g]);
    } else {
      val = A.U[cur ^ 1][g];
    }
  }
  (side == 0 ? sendL : sendR)[r] = val;
}

cudaError_t launch_pack_ghosts(int mode, const RhsConsts& C, const StageArgs& A, double* sendL,
                               double* sendR, cudaStream_t s) {
  const long long n = 2LL * NV * C.Ny * NP;
  const int threads = 256;
  k_pack_ghosts<<<(unsigned)((n + threads - 1) / threads), threads, 0, s>>>(mode, C, A, sendL,
                                                                            sendR);
  return cudaGetLastError();
}

}  // namespace dev
}  // namespace sgnb
