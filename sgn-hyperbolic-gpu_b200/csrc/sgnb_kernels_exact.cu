// sgnb_kernels_exact.cu -- fused kernels in the exact arithmetic mode.
// Built with -fmad=false: every product and sum rounds separately, in the operation
// order of the reference CPU solver, so the results are bit-identical to it.
#define SGNB_EXACT true
#include "sgnb_kernels_inst.cuh"

namespace sgnb {
namespace dev {
template <int MODE>
static cudaError_t launch_mode(const RhsConsts& C, const StageArgs& A, cudaStream_t s,
                               const TileMaps* M) {
  if (C.gauss) return launch_gauss<MODE>(C, A, s);
  const dim3 grid((C.Nx + 7) / 8, (C.Ny + 3) / 4);
  const size_t smem = sizeof(Tile<8, 4, SGNB_EXACT>::Smem);
  cudaError_t e;
  const bool ghost = C.ghostL != nullptr || C.ghostR != nullptr;
  if (C.manning) {
    if (ghost) e = launch_dependent(k_fused<MODE, SGNB_EXACT, true, true>, grid, dim3(NTHR), smem, s, C, A);
    else e = launch_dependent(k_fused<MODE, SGNB_EXACT, true, false>, grid, dim3(NTHR), smem, s, C, A);
  } else {
    const bool full = C.Nx % 8 == 0 && C.Ny % 4 == 0;  // every tile full
    // the own-node tiles by the tensor-memory accelerator where the context's tensor maps
    // describe the buffers (and, for the rhs mode, a map of its input)
    const bool tma = full && M != nullptr && M->ok && (MODE != MODE_RHS || M->inOk);
    if (ghost) {
      if (tma) e = launch_dependent(k_fused_tma<MODE, SGNB_EXACT, true>, grid, dim3(NTHR), smem, s, C, A, *M);
      else if (full) e = launch_dependent(k_fused<MODE, SGNB_EXACT, false, true, false, true>, grid, dim3(NTHR), smem, s, C, A);
      else e = launch_dependent(k_fused<MODE, SGNB_EXACT, false, true>, grid, dim3(NTHR), smem, s, C, A);
    } else if (full) {
      if (tma)
        e = launch_dependent(k_fused_tma<MODE, SGNB_EXACT>, grid, dim3(NTHR), smem, s, C, A, *M);
      else
        e = launch_dependent(k_fused<MODE, SGNB_EXACT, false, false, false, true>, grid, dim3(NTHR), smem, s, C, A);
    } else {
      e = launch_dependent(k_fused<MODE, SGNB_EXACT, false, false>, grid, dim3(NTHR), smem, s, C, A);
    }
  }
  return e;
}

cudaError_t launch_fused_exact(int mode, const RhsConsts& C, const StageArgs& A, cudaStream_t s,
                              const TileMaps* M) {
  switch (mode) {
    case MODE_RHS: return launch_mode<MODE_RHS>(C, A, s, M);
    case MODE_STAGE: return launch_mode<MODE_STAGE>(C, A, s, M);
    case MODE_FSAL: return launch_mode<MODE_FSAL>(C, A, s, M);
    case MODE_CAND: return launch_mode<MODE_CAND>(C, A, s, M);
    default: return cudaErrorInvalidValue;
  }
}

template <bool GHOST>
static cudaError_t prepare_tma() {
  const size_t bytes = sizeof(Tile<8, 4, true>::Smem);
  cudaError_t e = raise_smem(k_fused_tma<MODE_RHS, true, GHOST>, bytes);
  if (e == cudaSuccess) e = raise_smem(k_fused_tma<MODE_STAGE, true, GHOST>, bytes);
  if (e == cudaSuccess) e = raise_smem(k_fused_tma<MODE_CAND, true, GHOST>, bytes);
  if (e == cudaSuccess) e = raise_smem(k_fused_tma<MODE_FSAL, true, GHOST>, bytes);
  return e;
}

cudaError_t prepare_fused_exact() {
  cudaError_t e = prepare_variant<false, false>();
  if (e == cudaSuccess) e = prepare_variant<true, false>();
  if (e == cudaSuccess) e = prepare_variant<false, true>();
  if (e == cudaSuccess) e = prepare_variant<true, true>();
  if (e == cudaSuccess) e = prepare_variant<false, false, true>();
  if (e == cudaSuccess) e = prepare_variant<true, false, true>();
  if (e == cudaSuccess) e = prepare_variant<false, false, false, true>();
  if (e == cudaSuccess) e = prepare_variant<false, true, false, true>();
  if (e == cudaSuccess) e = prepare_tma<false>();
  if (e == cudaSuccess) e = prepare_tma<true>();
  return e;
}
int fused_grid_blocks(int Nx, int Ny) { return ((Nx + 7) / 8) * ((Ny + 3) / 4); }
size_t fused_smem_bytes() { return sizeof(Tile<8, 4, true>::Smem); }
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
