// sgnb_kernels_inst.cuh -- launch helpers of the fused kernels for one arithmetic mode.
// Included by sgnb_kernels_exact.cu (SGNB_EXACT = true, built with -fmad=false) and
// sgnb_kernels_fast.cu (SGNB_EXACT = false, built with -fmad=true).
#pragma once

#include "sgnb_kernels.cuh"

namespace sgnb {
namespace dev {

// Gauss-Legendre points: the trace pre-pass, then the fused kernel.
template <int MODE>
static cudaError_t launch_gauss(const RhsConsts& C, const StageArgs& A, cudaStream_t s) {
  const dim3 grid((C.Nx + 7) / 8, (C.Ny + 3) / 4);
  const size_t smem = sizeof(Tile<8, 4, SGNB_EXACT>::Smem);
  const long long n = 2LL * C.Nx * C.Ny * NP;
  cudaError_t e = launch_dependent(k_traces<MODE, SGNB_EXACT>, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, s, C, A);
  if (e != cudaSuccess) return e;
  if (C.manning) e = launch_dependent(k_fused<MODE, SGNB_EXACT, true>, grid, dim3(NTHR), smem, s, C, A);
  else e = launch_dependent(k_fused<MODE, SGNB_EXACT, false>, grid, dim3(NTHR), smem, s, C, A);
  return e;
}

template <class K>
static cudaError_t raise_smem(K* kernel, size_t bytes) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

template <bool FRIC>
static cudaError_t prepare_variant() {
  const size_t bytes = sizeof(Tile<8, 4, SGNB_EXACT>::Smem);
  cudaError_t e = raise_smem(k_fused<MODE_RHS, SGNB_EXACT, FRIC>, bytes);
  if (e == cudaSuccess) e = raise_smem(k_fused<MODE_STAGE, SGNB_EXACT, FRIC>, bytes);
  if (e == cudaSuccess) e = raise_smem(k_fused<MODE_CAND, SGNB_EXACT, FRIC>, bytes);
  if (e == cudaSuccess) e = raise_smem(k_fused<MODE_FSAL, SGNB_EXACT, FRIC>, bytes);
  return e;
}

}  // namespace dev
}  // namespace sgnb
