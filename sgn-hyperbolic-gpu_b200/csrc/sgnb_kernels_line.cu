// sgnb_kernels_line.cu -- single-instance and slab kernels of the fast arithmetic mode on GLL
// points. Built with -fmad=true.
#include "sgnb_kernels_line.cuh"

namespace sgnb {
namespace dev {

template <int MODE, bool FRIC, bool GHOST>
static cudaError_t launch_variant(const RhsConsts& C, const StageArgs& A, int bulk, cudaStream_t s) {
  using L = LineTile<1>;
  const dim3 grid((C.Nx + L::TX - 1) / L::TX, (C.Ny + L::TY - 1) / L::TY);
  LineConsts LC = line_consts(C);
  LC.bulk = bulk;
  return launch_dependent(k_line<MODE, FRIC, GHOST>, grid, dim3(LTHR), sizeof(typename L::Smem), s, LC, C.eo, A);
}

template <int MODE>
static cudaError_t launch_mode(const RhsConsts& C, const StageArgs& A, cudaStream_t s) {
  const int bulk = bulk_rows(C, A);
  const bool ghost = C.ghostL != nullptr || C.ghostR != nullptr;
  if (C.manning)
    return ghost ? launch_variant<MODE, true, true>(C, A, bulk, s) : launch_variant<MODE, true, false>(C, A, bulk, s);
  return ghost ? launch_variant<MODE, false, true>(C, A, bulk, s) : launch_variant<MODE, false, false>(C, A, bulk, s);
}
cudaError_t launch_line(int mode, const RhsConsts& C, const StageArgs& A, cudaStream_t s) {
  switch (mode) {
    case MODE_RHS: return launch_mode<MODE_RHS>(C, A, s);
    case MODE_STAGE: return launch_mode<MODE_STAGE>(C, A, s);
    case MODE_FSAL: return launch_mode<MODE_FSAL>(C, A, s);
    case MODE_CAND: return launch_mode<MODE_CAND>(C, A, s);
    default: return cudaErrorInvalidValue;
  }
}
int line_grid_blocks(int Nx, int Ny) {
  using L = LineTile<1>;
  return ((Nx + L::TX - 1) / L::TX) * ((Ny + L::TY - 1) / L::TY);
}

template <bool FRIC, bool GHOST>
static cudaError_t prepare_variant() {
  const int bytes = (int)sizeof(typename LineTile<1>::Smem);
  const auto at = cudaFuncAttributeMaxDynamicSharedMemorySize;
  cudaError_t e = cudaFuncSetAttribute(k_line<MODE_RHS, FRIC, GHOST>, at, bytes);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_line<MODE_STAGE, FRIC, GHOST>, at, bytes);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_line<MODE_FSAL, FRIC, GHOST>, at, bytes);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_line<MODE_CAND, FRIC, GHOST>, at, bytes);
  return e;
}

cudaError_t prepare_line(const RhsConsts& C, bool ghost) {
  if (C.manning) return ghost ? prepare_variant<true, true>() : prepare_variant<true, false>();
  return ghost ? prepare_variant<false, true>() : prepare_variant<false, false>();
}

// The checked build's out-of-range count of this translation unit's kernels (reset: then
// zero it); cudaErrorNotSupported in the normal build.
cudaError_t read_oob_line(unsigned long long* out, bool reset) {
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
