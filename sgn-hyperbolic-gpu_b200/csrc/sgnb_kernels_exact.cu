// sgnb_kernels_exact.cu -- kernels in the exact arithmetic mode.
// Built with -fmad=false: every product and sum rounds separately, in the operation
// order of the reference CPU solver, so the results are bit-identical to it.
#define SGNB_EXACT true
#include "sgnb_kernels_inst.cuh"
#include "sgnb_kernels_line.cuh"

namespace sgnb {
namespace dev {
template <int MODE, bool FRIC, bool GHOST>
static cudaError_t launch_variant(const RhsConsts& C, const StageArgs& A, cudaStream_t s) {
  using L = LineTile<1, true>;
  const dim3 grid((C.Nx + L::TX - 1) / L::TX, (C.Ny + L::TY - 1) / L::TY);
  return launch_dependent(k_line_exact<MODE, FRIC, GHOST>, grid, dim3(LTHR), sizeof(typename L::Smem), s, C, A,
                          (int)bulk_rows(C, A));
}

template <int MODE>
static cudaError_t launch_mode(const RhsConsts& C, const StageArgs& A, cudaStream_t s) {
  if (C.gauss) return launch_gauss<MODE>(C, A, s);
  const bool ghost = C.ghostL != nullptr || C.ghostR != nullptr;
  if (C.manning) return ghost ? launch_variant<MODE, true, true>(C, A, s) : launch_variant<MODE, true, false>(C, A, s);
  return ghost ? launch_variant<MODE, false, true>(C, A, s) : launch_variant<MODE, false, false>(C, A, s);
}

cudaError_t launch_fused_exact(int mode, const RhsConsts& C, const StageArgs& A, cudaStream_t s) {
  switch (mode) {
    case MODE_RHS: return launch_mode<MODE_RHS>(C, A, s);
    case MODE_STAGE: return launch_mode<MODE_STAGE>(C, A, s);
    case MODE_FSAL: return launch_mode<MODE_FSAL>(C, A, s);
    case MODE_CAND: return launch_mode<MODE_CAND>(C, A, s);
    default: return cudaErrorInvalidValue;
  }
}

template <bool FRIC, bool GHOST>
static cudaError_t prepare_lines() {
  const size_t bytes = sizeof(LineTile<1, true>::Smem);
  cudaError_t e = raise_smem(k_line_exact<MODE_RHS, FRIC, GHOST>, bytes);
  if (e == cudaSuccess) e = raise_smem(k_line_exact<MODE_STAGE, FRIC, GHOST>, bytes);
  if (e == cudaSuccess) e = raise_smem(k_line_exact<MODE_CAND, FRIC, GHOST>, bytes);
  if (e == cudaSuccess) e = raise_smem(k_line_exact<MODE_FSAL, FRIC, GHOST>, bytes);
  return e;
}

cudaError_t prepare_fused_exact(const RhsConsts& C, bool ghost) {
  if (C.gauss) return C.manning ? prepare_variant<true>() : prepare_variant<false>();
  if (C.manning) return ghost ? prepare_lines<true, true>() : prepare_lines<true, false>();
  return ghost ? prepare_lines<false, true>() : prepare_lines<false, false>();
}
int fused_grid_blocks(int Nx, int Ny) { return ((Nx + 7) / 8) * ((Ny + 3) / 4); }
// The checked build's out-of-range count of this translation unit's kernels (reset: then
// zero it); cudaErrorNotSupported in the normal build.
cudaError_t read_oob_exact(unsigned long long* out, bool reset) {
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

}  // namespace dev
}  // namespace sgnb
