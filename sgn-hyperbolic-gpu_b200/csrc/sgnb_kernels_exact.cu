// sgnb_kernels_exact.cu -- kernels in the exact arithmetic mode.
// Built with -fmad=false: every product and sum rounds separately, in the operation
// order of the reference CPU solver, so the results are bit-identical to it.
#define SGNB_EXACT true
#include "sgnb_kernels_inst.cuh"
#include "sgnb_kernels_line.cuh"

namespace sgnb {
namespace dev {
// The forms of the line kernels: tiles of 6 x 4 elements with the registers of three or of two CTAs
// per SM, and tiles of 2 x 12 (LineTile's COL).
enum : int { FORM_ROWS = 0, FORM_ROWS2 = 1, FORM_COLUMNS = 2 };
template <bool COL>
static dim3 tiles(int Nx, int Ny) {
  using L = LineTile<1, true, COL>;
  return dim3((Nx + L::TX - 1) / L::TX, (Ny + L::TY - 1) / L::TY);
}
// Columns: rows of six waste lanes where Nx is a little more than a multiple of six; on meshes up to
// 14 elements wide 2 x 12 tiles can be fewer by a fifth and more. Their halo is larger and a warp's
// row takes three copies, so they are taken only where a launch then also needs fewer waves of
// the CTAs that are resident at once (three per SM). us per launch, rhs / stages 2, 3, end point:
// 8 x 4096 elements on rows 123 / 114 139 171, on columns 94 / 97 119 142; 14 x 1500: 70 / 65 79 100
// and 55 / 51 65 79; within one wave, 8 x 256: 23.7 / 19.7 21.8 29.2 and 25.6 / 20.9 24.4 32.5; 10
// x 2048, where columns are fewer by a sixth: rows 69 / 64 76 93. Not for slabs.
// Two CTAs: with 255 registers nothing spills (168: up to 320 bytes per thread), which counts where
// all tiles are resident at once and a launch takes one tile's time; with more tiles three CTAs
// hide more. us per attempt: 96 x 48 elements 87.4 with three, 83.9 with two; 128 x 64 (352 tiles):
// 94.3 and 144.
int exact_form(int Nx, int Ny, bool slab) {
  constexpr long long kSms = 148, kResident = 3 * kSms;
  const dim3 rt = tiles<false>(Nx, Ny), ct = tiles<true>(Nx, Ny);
  const long long r = (long long)rt.x * rt.y, c = (long long)ct.x * ct.y;
  if (r <= 2 * kSms) return FORM_ROWS2;
  if (!slab && 10 * c <= 8 * r && (c + kResident - 1) / kResident < (r + kResident - 1) / kResident)
    return FORM_COLUMNS;
  return FORM_ROWS;
}
int exact_grid_blocks(const RhsConsts& C) {
  const dim3 g = C.form == FORM_COLUMNS ? tiles<true>(C.Nx, C.Ny) : tiles<false>(C.Nx, C.Ny);
  return (int)(g.x * g.y);
}

template <int MODE, bool FRIC, bool GHOST, bool COL, int CTAS>
static cudaError_t launch_form(const RhsConsts& C, const StageArgs& A, cudaStream_t s) {
  return launch_dependent(k_line_exact<MODE, FRIC, GHOST, COL, CTAS>, tiles<COL>(C.Nx, C.Ny), dim3(LTHR),
                          sizeof(typename LineTile<1, true, COL>::Smem), s, C, A, (int)bulk_rows(C, A));
}
template <int MODE, bool FRIC, bool GHOST>
static cudaError_t launch_variant(const RhsConsts& C, const StageArgs& A, cudaStream_t s) {
  switch (C.form) {
    case FORM_ROWS: return launch_form<MODE, FRIC, GHOST, false, 3>(C, A, s);
    case FORM_ROWS2: return launch_form<MODE, FRIC, GHOST, false, 2>(C, A, s);
    case FORM_COLUMNS: return launch_form<MODE, FRIC, GHOST, true, 3>(C, A, s);
    default: return cudaErrorInvalidValue;
  }
}

template <int MODE>
static cudaError_t launch_lines(const RhsConsts& C, const StageArgs& A, cudaStream_t s) {
  const bool ghost = C.ghostL != nullptr || C.ghostR != nullptr;
  if (C.manning) return ghost ? launch_variant<MODE, true, true>(C, A, s) : launch_variant<MODE, true, false>(C, A, s);
  return ghost ? launch_variant<MODE, false, true>(C, A, s) : launch_variant<MODE, false, false>(C, A, s);
}

cudaError_t launch_fused_exact(int mode, const RhsConsts& C, const StageArgs& A, cudaStream_t s) {
  if (C.gauss) {
    switch (mode) {
      case MODE_RHS: return launch_gauss<MODE_RHS>(C, A, s);
      case MODE_STAGE: return launch_gauss<MODE_STAGE>(C, A, s);
      case MODE_FSAL: return launch_gauss<MODE_FSAL>(C, A, s);
      case MODE_CAND: return launch_gauss<MODE_CAND>(C, A, s);
      default: return cudaErrorInvalidValue;
    }
  }
  StageArgs B = A;
  B.cand = mode == MODE_CAND;
  switch (mode) {
    case MODE_RHS: return launch_lines<MODE_RHS>(C, B, s);
    case MODE_STAGE:
    case MODE_CAND: return launch_lines<MODE_STAGES>(C, B, s);
    case MODE_FSAL: return launch_lines<MODE_FSAL>(C, B, s);
    default: return cudaErrorInvalidValue;
  }
}

template <bool FRIC, bool GHOST, bool COL, int CTAS>
static cudaError_t prepare_form() {
  const size_t bytes = sizeof(typename LineTile<1, true, COL>::Smem);
  cudaError_t e = raise_smem(k_line_exact<MODE_RHS, FRIC, GHOST, COL, CTAS>, bytes);
  if (e == cudaSuccess) e = raise_smem(k_line_exact<MODE_STAGES, FRIC, GHOST, COL, CTAS>, bytes);
  if (e == cudaSuccess) e = raise_smem(k_line_exact<MODE_FSAL, FRIC, GHOST, COL, CTAS>, bytes);
  return e;
}
template <bool FRIC, bool GHOST>
static cudaError_t prepare_lines(const RhsConsts& C) {
  switch (C.form) {
    case FORM_ROWS: return prepare_form<FRIC, GHOST, false, 3>();
    case FORM_ROWS2: return prepare_form<FRIC, GHOST, false, 2>();
    case FORM_COLUMNS: return prepare_form<FRIC, GHOST, true, 3>();
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t prepare_fused_exact(const RhsConsts& C, bool ghost) {
  if (C.gauss) return C.manning ? prepare_variant<true>() : prepare_variant<false>();
  if (C.manning) return ghost ? prepare_lines<true, true>(C) : prepare_lines<true, false>(C);
  return ghost ? prepare_lines<false, true>(C) : prepare_lines<false, false>(C);
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
