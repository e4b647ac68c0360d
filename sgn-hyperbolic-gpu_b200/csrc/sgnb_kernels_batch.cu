// sgnb_kernels_batch.cu -- batched kernels of the fast mode on GLL points: one
// launch per stage over the tiles of many independent instances. Built with -fmad=true.
#include "sgnb_kernels_line.cuh"

namespace sgnb {
namespace dev {

// Batched form: one launch per stage walks the tiles of many independent instances
// (the work list tile_inst / tile_start), each with its own constants, buffers and
// controller. The instance's constants and buffer pointers are copied into shared
// memory once per tile. PERSIST: a fixed grid of CTAs loops over the work list;
// otherwise one CTA per tile (no loop: the compiler then keeps nothing live from one tile
// to the next, which the loop costs in spilled registers).
template <int MODE, int WX>
__device__ __forceinline__ void batch_tile(const BatchArgs& B, long long t,
                                           typename LineTile<WX>::Smem& S, LineConsts& Cs,
                                           StageArgs& As) {
  const int inst = B.tile_inst[t];
  const long long lt = t - B.tile_start[inst];
  __syncthreads();  // the previous tile is done with Cs / As
  {
    // both blocks' loads in flight before the first store (one round trip per tile)
    block_copy2<(int)(sizeof(LineConsts) / 4), (int)(sizeof(StageArgs) / 4), LTHR>(
        reinterpret_cast<unsigned*>(&Cs), reinterpret_cast<const unsigned*>(B.consts + inst),
        reinterpret_cast<unsigned*>(&As), reinterpret_cast<const unsigned*>(B.args + inst));
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    As.kin_k2 = B.kin_k2;
    As.coef = B.coef;
    if (MODE == MODE_STAGE) As.out = As.K2;
  }
  __syncthreads();
  const int ntx = (Cs.Nx + LineTile<WX>::TX - 1) / LineTile<WX>::TX;
  // volatile views: per-instance values are re-read from shared memory at each use
  // rather than held in registers through the passes
  line_tile<MODE, WX, false, false>(
      static_cast<const volatile LineConsts&>(Cs), B.tables, static_cast<const volatile StageArgs&>(As),
      (int)(lt % ntx), (int)(lt / ntx), lt, Cs.bulk != 0, S);
}

template <int MODE, int WX, bool PERSIST>
__global__ void __launch_bounds__(LTHR, (PERSIST ? 3 : kLineCtas<MODE, WX>)) k_line_batch(const BatchArgs B) {
  // FR tables come from the kernel parameters (constant bank): the same for every
  // instance (P = 4 GLL)
  extern __shared__ __align__(128) unsigned char smem_batch[];
  using T = LineTile<WX>;
  typename T::Smem& S = *reinterpret_cast<typename T::Smem*>(smem_batch);
  __shared__ LineConsts Cs;
  __shared__ StageArgs As;
  if (kStash<MODE> && threadIdx.x < 32) stash_alloc(&S.stash);
  if constexpr (PERSIST) {
    for (long long t = blockIdx.x; t < B.ntiles; t += gridDim.x)
      batch_tile<MODE, WX>(B, t, S, Cs, As);
  } else {
    if ((long long)blockIdx.x < B.ntiles) batch_tile<MODE, WX>(B, blockIdx.x, S, Cs, As);
  }
  if constexpr (kStash<MODE>) {
    __syncthreads();
    if (threadIdx.x < 32) stash_free(S.stash);
  }
}

template <int MODE, int WX>
static cudaError_t launch_b(int blocks, const BatchArgs& B, cudaStream_t s) {
  const size_t smem = sizeof(typename LineTile<WX>::Smem);
  if (blocks > 0) {
    k_line_batch<MODE, WX, true><<<blocks, LTHR, smem, s>>>(B);
  } else {
    if (B.ntiles < 1 || B.ntiles > 0x7fffffffLL) return cudaErrorInvalidValue;
    k_line_batch<MODE, WX, false><<<(unsigned)B.ntiles, LTHR, smem, s>>>(B);
  }
  return cudaGetLastError();
}

template <int WX>
static cudaError_t launch_shape(int mode, int blocks, const BatchArgs& B, cudaStream_t s) {
  switch (mode) {
    case MODE_RHS: return launch_b<MODE_RHS, WX>(blocks, B, s);
    case MODE_STAGE: return launch_b<MODE_STAGE, WX>(blocks, B, s);
    case MODE_FSAL: return launch_b<MODE_FSAL, WX>(blocks, B, s);
    case MODE_CAND: return launch_b<MODE_CAND, WX>(blocks, B, s);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_fused_batch(int mode, int shape_id, int blocks, const BatchArgs& B,
                               cudaStream_t s) {
  switch (shape_id) {
    case 0: return launch_shape<1>(mode, blocks, B, s);
    case 1: return launch_shape<2>(mode, blocks, B, s);
    case 2: return launch_shape<4>(mode, blocks, B, s);
    default: return cudaErrorInvalidValue;
  }
}

int batch_tile_tx(int shape_id) { return LROW * (shape_id == 1 ? 2 : (shape_id == 2 ? 4 : 1)); }
int batch_tile_ty(int shape_id) { return shape_id == 1 ? 2 : (shape_id == 2 ? 1 : 4); }

template <int WX, bool PERSIST>
static cudaError_t prepare_form() {
  const int bytes = (int)sizeof(typename LineTile<WX>::Smem);
  const auto at = cudaFuncAttributeMaxDynamicSharedMemorySize;
  cudaError_t e = cudaFuncSetAttribute(k_line_batch<MODE_RHS, WX, PERSIST>, at, bytes);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_line_batch<MODE_STAGE, WX, PERSIST>, at, bytes);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_line_batch<MODE_FSAL, WX, PERSIST>, at, bytes);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_line_batch<MODE_CAND, WX, PERSIST>, at, bytes);
  return e;
}

cudaError_t prepare_fused_batch(int shape_id, int blocks) {
  switch (shape_id) {
    case 0: return blocks > 0 ? prepare_form<1, true>() : prepare_form<1, false>();
    case 1: return blocks > 0 ? prepare_form<2, true>() : prepare_form<2, false>();
    case 2: return blocks > 0 ? prepare_form<4, true>() : prepare_form<4, false>();
    default: return cudaErrorInvalidValue;
  }
}

// The checked build's out-of-range count of this translation unit's kernels (reset: then
// zero it); cudaErrorNotSupported in the normal build.
cudaError_t read_oob_batch(unsigned long long* out, bool reset) {
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
