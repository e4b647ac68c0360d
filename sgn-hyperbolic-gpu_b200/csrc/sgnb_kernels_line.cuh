// sgnb_kernels_line.cuh -- the FP64 modes' fused right-hand-side and stage kernels on
// Gauss-Lobatto points (single instances, slabs; in the fast mode also batches).
//
// Work decomposition. A warp owns a row of six elements and holds one line of solution points per
// lane (30 of 32 lanes): lane (e, j) is line j of element e, first along y (column pass), then
// along x (row pass). All five lines of an element are in one warp, so between the passes a warp
// synchronises with itself only; a CTA of four warps stacks four such rows (or 2 x 2, or 4 x 1)
// and synchronises once, when its tile has landed and every warp has formed its stage inputs.
// With the lanes over 32 elements and one warp per line instead (as the Gauss-point kernels of
// sgnb_kernels.cuh), two of the eight cycles a warp took per instruction were waits at the
// barriers between the passes. On narrow meshes the exact mode's warps hold three rows of two
// elements instead (COL; the rule and its figures are in sgnb_kernels_exact.cu).
//
// The arithmetic is arranged for the fast mode:
//   * every flux component is the normal velocity times a state component, F = u_n U_v (plus
//     the hydrostatic term in the normal discharge; h u_n (p + c^2) in hp), so a line keeps u_n and
//     reads one field at a time from shared memory;
//   * the Rusanov flux minus the element's own face flux is half the flux difference of the
//     two traces plus the dissipation, in which the face depth cancels (both traces take the
//     same one): no face depths are read;
//   * the GLL differentiation matrix changes sign under reflection of its rows and columns and
//     the two correction functions mirror each other, so a 5-point derivative with both
//     lifts splits into an even and an odd half (29 operations instead of 35);
//   * each pass adds its own direction's sources, so no pass differentiates the depth along
//     the other direction, and h_n and H_n of the hp equation share one derivative.
// What bounds it. At 1024 x 512 elements a right-hand side takes 0.224 ms (5.1 TB/s, 80 % of a
// plain copy's rate), the second, third and end-point stage 0.321, 0.515 and 0.508 ms (5.2, 5.3
// and 4.3 TB/s; the end point 0.49 to 0.51 from GPU to GPU); kernels with one warp per GLL line took
// 0.408, 0.497, 0.497 and 0.981 ms (the end point then read four inputs twice). What is left is
// latency: HBM, FP64 issue (62 % busy in the right-hand side) and shared memory (65 %) are all
// within 1.6x of their limits. The right-hand side and the end point run four CTAs of 128
// registers per SM, the stages that add k three: their halos read two arrays, whose sectors only
// stay in L1 if shared memory leaves it more than 24 KB. (Before the derivatives acted on
// differences, which costs 1 %: right-hand side and end point at three CTAs 0.247 and 0.503 ms, at
// four 0.227 and 0.476; the stages at four 0.358 and 0.556, at three 0.320 and 0.508; tiles of
// 2 x 2 or 4 x 1 warps 0.334 and 0.349 ms in the second stage.)
#pragma once

#include "sgnb_kernels.cuh"

namespace sgnb {
namespace dev {

constexpr int LROW = 6;             // elements of a warp's row
constexpr int LWARPS = 4;           // warps of a CTA
constexpr int LTHR = 32 * LWARPS;

// A tile of WX x WY warps, and its shared memory. Field v of the tile's nodes and of the nodes
// across its edges lie in one block, so a line's neighbour is reached with the line's own field
// stride:
//   U[v][i * 25 + a + 5 b]        node (a, b) of tile element i = ix + TX iy
//   U[v][TN + 5 * slot + t]       slots left [TY], right [TY], bottom [TX], top [TX]
// COL: a warp's six elements are three rows of two, the tile 2 x 12 elements.
template <int WX_, bool EXACT_ = false, bool COL = false>
struct LineTile {
  static constexpr int WX = WX_, WY = LWARPS / WX_;
  static constexpr int WR = COL ? 3 : 1, WC = LROW / WR;  // rows of a warp, elements of such a row
  static constexpr int TX = WC * WX, TY = WR * WY;
  static_assert(WX * WY == LWARPS && (!COL || WX == 1), "four warps");
  static constexpr int NHALO = 2 * TY + 2 * TX;
  static constexpr int TN = TX * TY * NPP;        // nodes per tile
  static constexpr int US = TN + NHALO * NP;      // field stride of U
  struct Smem {
    double U[NV][US];
    double H[TN];
    // stage derivative on load; column-pass results (the exact mode: the non-conservative product
    // of hp on its own); then dU
    double G[NV + (EXACT_ ? 1 : 0)][TN];
    double red[LWARPS][3];   // (with the barriers: room for the reads of idle lanes past G)
    unsigned long long mbar[LWARPS];
    unsigned stash;          // base of the CTA's tensor memory
    unsigned pad_;
  };
};
// CTAs per SM that a kernel is compiled for: see the note on what bounds these kernels.
template <int MODE, int WX>
constexpr int kLineCtas = sizeof(typename LineTile<WX>::Smem) <= 57000 && (MODE == MODE_RHS || MODE == MODE_FSAL) ? 4 : 3;
constexpr int LRUN = LROW * NPP;    // nodes of a warp's row per field
// Pairs of neighbouring nodes for element-wise work on a row: lane l < 25 takes pairs l, l + 25,
// l + 50 of every field (constant strides: no index arithmetic per pair; 32 lanes over all 375
// pairs of a row spent 20 integer instructions on each).
constexpr int LPL = 25, LPF = 3;
static_assert(2 * LPL * LPF == LRUN, "pairs of a row");

// Line of a lane in the column pass, 8 e + a. A half-warp's 16 accesses of 8 bytes should hit 16
// different bank pairs: elements lie 25 doubles apart, so line (e, a) starts in pair (9 e + a) mod 16.
// The first 16 lanes cover every pair once, the last 14 collide twice.
__constant__ unsigned char kColumnLane[32] = {
    0, 1, 2, 3, 4, 8, 9, 10, 11, 12, 19, 20, 27, 28, 35, 36,
    16, 17, 18, 24, 25, 26, 32, 33, 34, 40, 41, 42, 43, 44, 0, 0};

// Row copies between global and shared memory by the bulk copy engine. Sizes are multiples
// of 16 bytes and both addresses 16-byte aligned (rows of an even number of elements).
__device__ __forceinline__ void bulk_load(unsigned dst, const void* src, unsigned bytes, unsigned mb) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(dst),
      "l"(src), "r"(bytes), "r"(mb)
      : "memory");
}
// Brings a row to L2.
__device__ __forceinline__ void bulk_prefetch(const void* src, unsigned bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;\n" ::"l"(src), "r"(bytes) : "memory");
}
// Stored with the evict-first policy: a result is next read by another launch, after
// gigabytes of other traffic.
__device__ __forceinline__ void bulk_store(void* dst, unsigned src, unsigned bytes) {
  asm volatile(
      "{\n .reg .b64 pol;\n createpolicy.fractional.L2::evict_first.b64 pol, 1.0;\n"
      " cp.async.bulk.global.shared::cta.bulk_group.L2::cache_hint [%0], [%1], %2, pol;\n}\n" ::"l"(dst),
      "r"(src), "r"(bytes)
      : "memory");
}
__device__ __forceinline__ void bulk_store_wait() {
  asm volatile("cp.async.bulk.commit_group;\n cp.async.bulk.wait_group.read 0;\n" ::: "memory");
}

// Buffer c of a ping-pong pair, by selection: indexing the kernel parameters with a run-time
// value would copy them to local memory.
template <class P>
__device__ __forceinline__ auto pick(const P& p, int c) { return c ? p[1] : p[0]; }

// Tensor memory as a stash. The epilogues of the third and the end-point stage need values that
// the passes have no room for (128 registers, and shared memory that sets the CTAs per SM):
// u and k2 as they were before the stage input replaced them, or u and the embedded part, which
// are best requested at the start, together with the tile. A lane keeps 2 x 30 doubles of its own
// in 120 columns of its lane of tensor memory; four CTAs of 128 columns fill an SM's 512.
// (Read from L2 a second time, one batch of pairs after the other, the two epilogues waited for
// memory in 4.1 and 2.6 of the 10 and 8 cycles a warp took per instruction.)
constexpr unsigned kStashCols = 128;
template <int MODE>
constexpr bool kStash = MODE == MODE_CAND || MODE == MODE_STAGES || MODE == MODE_FSAL;
__device__ __forceinline__ void stash_alloc(unsigned* smem) {  // one warp
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_addr(smem)),
               "r"(kStashCols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
}
__device__ __forceinline__ void stash_free(unsigned base) {  // the same warp
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(base), "r"(kStashCols));
}
// Three pairs of this lane (one field) to 12 columns at addr; the whole warp together.
__device__ __forceinline__ void stash_put(unsigned addr, const double2 (&x)[LPF]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%2, %3, %4, %5, %6, %7, %8, %9};\n"
      "tcgen05.st.sync.aligned.32x32b.x4.b32 [%1], {%10, %11, %12, %13};\n" ::"r"(addr),
      "r"(addr + 8),
      "r"(__double2loint(x[0].x)), "r"(__double2hiint(x[0].x)), "r"(__double2loint(x[0].y)),
        "r"(__double2hiint(x[0].y)), "r"(__double2loint(x[1].x)), "r"(__double2hiint(x[1].x)),
        "r"(__double2loint(x[1].y)), "r"(__double2hiint(x[1].y)), "r"(__double2loint(x[2].x)),
        "r"(__double2hiint(x[2].x)), "r"(__double2loint(x[2].y)), "r"(__double2hiint(x[2].y))
      : "memory");
}
__device__ __forceinline__ void stash_put_wait() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }
// The reads and the wait for them in one statement: nothing may touch the registers in between.
__device__ __forceinline__ void stash_get(unsigned addr, double2 (&x)[LPF]) {
  int r[4 * LPF];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%12];\n"
      "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%8, %9, %10, %11}, [%13];\n"
      "tcgen05.wait::ld.sync.aligned;\n"
      : "=&r"(r[0]), "=&r"(r[1]), "=&r"(r[2]), "=&r"(r[3]), "=&r"(r[4]), "=&r"(r[5]), "=&r"(r[6]),
        "=&r"(r[7]), "=&r"(r[8]), "=&r"(r[9]), "=&r"(r[10]), "=&r"(r[11])
      : "r"(addr), "r"(addr + 8)
      : "memory");
#pragma unroll
  for (int m = 0; m < LPF; ++m)
    x[m] = make_double2(__hiloint2double(r[4 * m + 1], r[4 * m]), __hiloint2double(r[4 * m + 3], r[4 * m + 2]));
}

// Two neighbouring values, in one access where rows start aligned (vec); the second one only if
// two. The same values reach the same lane either way, so both ways give the same sums.
// Streaming (evict-first) accesses: no other CTA reads these lines soon.
__device__ __forceinline__ double2 load_pair(const double* p, bool vec, bool two) {
  if (vec) return __ldcs((const double2*)p);
  double2 r;
  r.x = __ldcs(p);
  r.y = two ? __ldcs(p + 1) : 0.0;
  return r;
}
__device__ __forceinline__ void store_pair(double* p, double2 x, bool vec, bool two) {
  if (vec) {
    __stcs((double2*)p, x);
  } else {
    __stcs(p, x.x);
    if (two) __stcs(p + 1, x.y);
  }
}

// Derivative of the five values F along a line plus the lifts of the face jumps jl, jr, all
// before the division by J. The rows of D sum to zero, so it acts on the differences to the centre
// value, which are exact or nearly so where F varies little along the line; F_0 + F_4 first and
// 2 F_2 off it would round at the size of F itself (two operations less; a right-hand side of 128 x
// 64 elements was then up to 1.35 times as far from the true value in a field).
template <class TE_>
__device__ __forceinline__ void line_derivative(const TE_& T, const double (&F)[NP], double jl,
                                                double jr, double (&d)[NP]) {
  const double o0 = F[0] - F[4], o1 = F[1] - F[3];
  const double e0 = (F[0] - F[2]) + (F[4] - F[2]), e1 = (F[1] - F[2]) + (F[3] - F[2]);
  const double js = jl + jr, jd = jl - jr;
  const double E0 = fma(T.A[0], e0, fma(T.A[1], e1, T.b[0] * js));
  const double E1 = fma(T.A[2], e0, fma(T.A[3], e1, T.b[1] * js));
  const double O0 = fma(T.B[0], o0, fma(T.B[1], o1, T.a[0] * jd));
  const double O1 = fma(T.B[2], o0, fma(T.B[3], o1, T.a[1] * jd));
  d[2] = fma(T.B[4], o0, fma(T.B[5], o1, T.a[2] * jd));
  d[0] = O0 + E0;
  d[4] = O0 - E0;
  d[1] = O1 + E1;
  d[3] = O1 - E1;
}
// The same without face jumps (the still depth).
template <class TE_>
__device__ __forceinline__ void line_derivative(const TE_& T, const double (&F)[NP], double (&d)[NP]) {
  const double o0 = F[0] - F[4], o1 = F[1] - F[3];
  const double e0 = (F[0] - F[2]) + (F[4] - F[2]), e1 = (F[1] - F[2]) + (F[3] - F[2]);
  const double E0 = fma(T.A[0], e0, T.A[1] * e1), E1 = fma(T.A[2], e0, T.A[3] * e1);
  const double O0 = fma(T.B[0], o0, T.B[1] * o1), O1 = fma(T.B[2], o0, T.B[3] * o1);
  d[2] = fma(T.B[4], o0, T.B[5] * o1);
  d[0] = O0 + E0;
  d[4] = O0 - E0;
  d[1] = O1 + E1;
  d[3] = O1 - E1;
}

// One line of direction DIR (0 along x, 1 along y). u: its first node in field 0 (fields US
// apart, nodes SN apart), hl: the nodal depth there, lo / hi: field 0 of the trace across the
// low / high face, with the sign of its normal discharge (-1 across a wall, where lo / hi is
// the line's own end node). Calls emit(v, k, r) with r = the line's share of -dU at node k: the
// divergence of flux v, the non-conservative product and minus the direction's sources; the
// sources without a direction (gamma p, -2 c^2 w) go with y, friction with x.
// LATE: the faces' discharge differences are formed where they are used instead of once. The end
// point, whose other state leaves the passes fewer registers, spills without (1024 x 512 elements:
// 0.495 ms instead of 0.517); the right-hand side is 2.4 % slower with it.
template <int DIR, int US, bool FRIC, bool LATE, class TC, class TE_, class Emit>
__device__ __forceinline__ void line_terms(const TC& C, const TE_& T, const double* u,
                                           const double* hl, const double* lo, const double* hi,
                                           double slo, double shi, Emit&& emit) {
  constexpr int SN = DIR == 0 ? 1 : NP;            // node stride along the line
  constexpr int N = DIR == 0 ? 1 : 2, TG = 3 - N;  // normal and tangential discharge
  const double c2 = C.c2, g = C.g, iJ = DIR == 0 ? C.iJx : C.iJy;
  double h[NP], hn[NP], ih[NP], un[NP], hp[NP];
#pragma unroll
  for (int k = 0; k < NP; ++k) {
    h[k] = u[k * SN];
    hn[k] = u[N * US + k * SN];
    hp[k] = u[4 * US + k * SN];
    ih[k] = fast_rcp(h[k]);
    un[k] = hn[k] * ih[k];
  }
  // across the faces: half the larger wave speed (sgn_flux2d.h:73-86, 169-179)
  const double hL = lo[0], hR = hi[0], hnL = slo * lo[N * US], hnR = shi * hi[N * US];
  const double hpL = lo[4 * US], hpR = hi[4 * US];
  const double ihL = fast_rcp(hL), ihR = fast_rcp(hR);
  const double unL = hnL * ihL, unR = hnR * ihR;
  auto speed = [&](double hh, double pp, double uu) {
    // sqrt(max(a, 0)), with 1e-150 for 0: far below the last bit of c
    const double a = fma(g, hh, pp) + c2;
    return fabs(uu) + fast_sqrt_normal(a > 1e-300 ? a : 1e-300);
  };
  const double lamL = 0.5 * fmax(speed(hL, hpL * ihL, unL), speed(h[0], hp[0] * ih[0], un[0]));
  const double lamR = 0.5 * fmax(speed(h[4], hp[4] * ih[4], un[4]), speed(hR, hpR * ihR, unR));
  double dL = 0.0, dR = 0.0;
  if constexpr (!LATE) {
    dL = hnL - hn[0];
    dR = hnR - hn[4];
  }
  auto dnL = [&] { return LATE ? hnL - hn[0] : dL; };
  auto dnR = [&] { return LATE ? hnR - hn[4] : dR; };
  double F[NP], d[NP];
  // hp: flux h u_n (p + c^2); the non-conservative product -c^2 u_n h_n and the source
  // -2 c^2 u_n H_n together are -c^2 u_n (h - 2 H)_n, h and H each as differences to the centre
  // (h - 2 H itself would round at the size of H)
  {
    double dh[NP];
#pragma unroll
    for (int k = 0; k < NP; ++k) F[k] = k == 2 ? 0.0 : fma(-2.0, hl[k * SN] - hl[2 * SN], h[k] - h[2]);
    line_derivative(T, F, 0.5 * (hL - h[0]), 0.5 * (hR - h[4]), dh);
#pragma unroll
    for (int k = 0; k < NP; ++k) F[k] = hn[k] * fma(hp[k], ih[k], c2);
    const double jl = fma(0.5, fma(hnL, fma(hpL, ihL, c2), -F[0]), lamL * (hpL - hp[0]));
    const double jr = fma(0.5, fma(hnR, fma(hpR, ihR, c2), -F[4]), lamR * (hp[4] - hpR));
    line_derivative(T, F, jl, jr, d);
#pragma unroll
    for (int k = 0; k < NP; ++k) {
      double r = iJ * fma(-c2 * un[k], dh[k], d[k]);
      if constexpr (DIR == 1) r = fma(2.0 * c2, u[3 * US + k * SN] * ih[k], r);
      emit(4, k, r);
    }
  }
  // normal discharge: u_n (h u_n) + g/2 (h^2 - H^2) + hp, source (g (h - H) + gamma p) H_n
  double cf[FRIC ? NP : 1];
  if constexpr (FRIC) {
    // Manning friction n^2 g |vel| vel / h^(1/3) (sgn_flux2d.h:135-142)
#pragma unroll
    for (int k = 0; k < NP; ++k) {
      const double vt = u[TG * US + k * SN] * ih[k];
      cf[k] = C.n2g * fast_sqrt(fma(un[k], un[k], vt * vt)) * rcbrt(h[k]);
    }
  }
  {
    double Hg[NP], Hn[NP];
#pragma unroll
    for (int k = 0; k < NP; ++k) Hn[k] = hl[k * SN];
    line_derivative(T, Hn, Hg);
#pragma unroll
    for (int k = 0; k < NP; ++k)
      F[k] = fma(hn[k], un[k], hydro(C, h[k], Hn[k]) + hp[k]);
    const double fl = fma(unL, hnL, fma(0.5 * g * (hL - h[0]), hL + h[0], (hpL - hp[0]) - un[0] * hn[0]));
    const double fr = fma(unR, hnR, fma(0.5 * g * (hR - h[4]), hR + h[4], (hpR - hp[4]) - un[4] * hn[4]));
    line_derivative(T, F, fma(0.5, fl, lamL * dnL()), fma(0.5, fr, -lamR * dnR()), d);
#pragma unroll
    for (int k = 0; k < NP; ++k) {
      const double bath = fma(g, h[k] - Hn[k], C.gamma * (hp[k] * ih[k]));
      double r = iJ * fma(-bath, Hg[k], d[k]);
      if constexpr (FRIC) r = fma(cf[k], un[k], r);
      emit(N, k, r);
    }
  }
  // hw and the tangential discharge: u_n U_v
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const int v = q == 0 ? 3 : TG;
    double w[NP];
#pragma unroll
    for (int k = 0; k < NP; ++k) w[k] = u[v * US + k * SN];
    const double wL = lo[v * US], wR = hi[v * US];
#pragma unroll
    for (int k = 0; k < NP; ++k) F[k] = un[k] * w[k];
    line_derivative(T, F, fma(0.5, fma(unL, wL, -F[0]), lamL * (wL - w[0])),
                    fma(0.5, fma(unR, wR, -F[4]), lamR * (w[4] - wR)), d);
#pragma unroll
    for (int k = 0; k < NP; ++k) {
      double r = iJ * d[k];
      if constexpr (DIR == 1) {
        if (q == 0) r = fma(-C.gamma, hp[k] * ih[k], r);
      }
      if constexpr (FRIC) {
        if (q == 1) r = fma(cf[k], w[k] * ih[k], r);
      }
      emit(v, k, r);
    }
  }
  // mass: h u_n
  line_derivative(T, hn, fma(0.5, dnL(), lamL * (hL - h[0])), fma(0.5, dnR(), lamR * (h[4] - hR)), d);
#pragma unroll
  for (int k = 0; k < NP; ++k) emit(0, k, iJ * d[k]);
}

// One tile. The CTA holds its stash (S.stash, written before or visible after the first barrier
// here) in the modes that use one. bulk: rows start 16-byte aligned in every buffer (Nx even) and come and go by the bulk
// copy engine; otherwise value by value.
template <int MODE, int WX, bool FRIC, bool GHOST, bool EXACT = false, bool COL = false, class TC, class TE_, class TA>
__device__ __forceinline__ void line_tile(const TC& C, const TE_& T, const TA& A, int bx, int by,
                                          long long blk, const bool bulk,
                                          typename LineTile<WX, EXACT, COL>::Smem& S) {
  using L = LineTile<WX, EXACT, COL>;
  constexpr int TX = L::TX, TY = L::TY, NHALO = L::NHALO, TN = L::TN, US = L::US;
  constexpr int WR = L::WR, WC = L::WC, WRUN = WC * NPP;  // nodes of one row of a warp
  constexpr bool AXPY = MODE == MODE_STAGE || MODE == MODE_CAND || MODE == MODE_STAGES;
  constexpr bool MAYBE_CAND = MODE == MODE_CAND || MODE == MODE_STAGES;
  bool cand = MODE == MODE_CAND;  // the candidate leaves
  if constexpr (MODE == MODE_STAGES) cand = A.cand != 0;

  // ---- controller state -----------------------------------------------------------
  int cur = 0;
  double dt = 0.0, acoef = 0.0;
  if constexpr (MODE != MODE_RHS) {
    if (A.ctrl->done) return;  // uniform across the grid
    cur = A.ctrl->cur;
    dt = A.ctrl->dt;
    acoef = A.coef * dt;
  }
  const double* src = MODE == MODE_RHS ? A.in : (MODE == MODE_FSAL ? pick(A.U, cur ^ 1) : pick(A.U, cur));
  const double* kin = AXPY ? (A.kin_k2 ? A.K2 : pick(A.K1, cur)) : nullptr;

  int tid;
  asm volatile("mov.u32 %0, %%tid.x;" : "=r"(tid));
  const int w = tid >> 5, lane = tid & 31;
  const int wx = WX == 1 ? 0 : w % WX, iy0 = WR * (WX == 1 ? w : w / WX);  // this warp's (first) row of the tile
  const int Nx = C.Nx, Ny = C.Ny;
  const long long Nd = C.Nd;
  const int ex0 = bx * TX, ey0 = by * TY;
  const int TXv = min(TX, Nx - ex0), TYv = min(TY, Ny - ey0);
  // elements of the warp's row in the mesh, and such rows
  const int RXv = iy0 < TYv ? max(0, min(WC, TXv - wx * LROW)) : 0, RYv = COL ? min(WR, TYv - iy0) : 1;
  bool ghostL = false, ghostR = false;
  if constexpr (GHOST) {
    ghostL = C.ghostL != nullptr && ex0 == 0;
    ghostR = C.ghostR != nullptr && ex0 + TXv == Nx;
  }
  const bool wallL = C.bcx && ex0 == 0 && !ghostL, wallR = C.bcx && ex0 + TXv == Nx && !ghostR;
  const bool wallB = C.bcy && ey0 == 0, wallT = C.bcy && ey0 + TYv == Ny;
  const int row0 = (ex0 + wx * LROW + Nx * (ey0 + iy0)) * NPP;  // the row's first node in a field (Nd < 2^31)
  const int s0 = (wx * LROW + TX * iy0) * NPP;                  // and in the tile
  const int rowv = RXv * NPP;                                   // its nodes in the mesh
  const int next_row = Nx * NPP;                                // to the same node one row up
  // column and row in the tile of the warp's element e
  auto el_x = [&](int e) { return COL ? e % WC : wx * LROW + e; };
  auto el_y = [&](int e) { return COL ? iy0 + e / WC : iy0; };

  // ---- the row's own nodes ------------------------------------------------------------
  const unsigned mbar = smem_addr(&S.mbar[w]);
  double* const ks = &S.G[0][0];  // the stage derivative, until the passes
  // pair m of a field: the warp's nodes kp + 2 LPL m and the next one, where in[m] (and two[m]); in
  // the mesh it is step(m) from the first pair (COL: pair m is in row m, 2 LPL nodes long)
  static_assert(!COL || WRUN == 2 * LPL, "a pair per row");
  const int kp = 2 * lane;
  auto step = [&](int m) { return COL ? m * next_row : 2 * LPL * m; };
  bool in[LPF], two[LPF];
#pragma unroll
  for (int m = 0; m < LPF; ++m) {
    const int k = COL ? kp : kp + 2 * LPL * m;
    in[m] = lane < LPL && k < rowv && (!COL || m < RYv);
    two[m] = k + 1 < rowv;
  }
  if (bulk) {
    constexpr int NROW = NV + 1 + (AXPY ? NV : 0);
    const unsigned bytes = (unsigned)rowv * sizeof(double);
    if (lane == 0) {
      mbar_init(mbar);
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
      mbar_expect_tx(mbar, RXv > 0 ? NROW * RYv * bytes : 0u);
    }
    __syncwarp();
    auto copy = [&](int f, int r) {  // array f's row r
      const int sr = s0 + r * WRUN;
      int g = row0 + r * next_row;
      if (!SGNB_INB(g, Nd - rowv + 1)) g = 0;
      if (f < NV) bulk_load(smem_addr(&S.U[f][sr]), src + f * Nd + g, bytes, mbar);
      else if (f == NV) bulk_load(smem_addr(&S.H[sr]), C.Hnod + g, bytes, mbar);
      else bulk_load(smem_addr(ks + (f - NV - 1) * TN + sr), kin + (f - NV - 1) * Nd + g, bytes, mbar);
    };
    if constexpr (COL) {
      for (int q = lane; q < NROW * RYv; q += 32)
        if (RXv > 0) copy(q % NROW, q / NROW);
    } else if (lane < NROW && RXv > 0) {
      copy(lane, 0);
    }
    // what the epilogue reads starts its way to L2
    if ((MAYBE_CAND && cand) || MODE == MODE_FSAL) {
      const int q = COL ? lane : lane - 16;  // (lanes that copy no row)
      const int f = COL ? q % NV : q, r = COL ? q / NV : 0, g = row0 + r * next_row;
      if (f >= 0 && f < NV && r < RYv && RXv > 0 && SGNB_INB(g, Nd - rowv + 1))
        bulk_prefetch((MAYBE_CAND ? pick(A.K1, cur) : A.K3) + f * Nd + g, bytes);
    }
  } else {
#pragma unroll
    for (int m = 0; m < (LRUN + 31) / 32; ++m) {
      const int k = lane + 32 * m, r = COL ? k / WRUN : 0, kr = k - r * WRUN, g = row0 + r * next_row + kr;
      if (kr < rowv && r < RYv && SGNB_INB(g, Nd)) {
        cp_async8(&S.H[s0 + k], C.Hnod + g);
#pragma unroll
        for (int v = 0; v < NV; ++v) {
          cp_async8(&S.U[v][s0 + k], src + v * Nd + g);
          if constexpr (AXPY) cp_async8(ks + v * TN + s0 + k, kin + v * Nd + g);
        }
      }
    }
  }
  // end point: u is requested along with the tile
  static_assert(2 * 4 * LPF * NV <= (int)kStashCols, "two arrays in the stash");
  constexpr int NE = MODE == MODE_FSAL ? NV : 1;
  double2 eu[NE][LPF];
  if constexpr (MODE == MODE_FSAL) {
    const double* u0 = pick(A.U, cur) + row0 + kp;
#pragma unroll
    for (int v = 0; v < NV; ++v)
#pragma unroll
      for (int m = 0; m < LPF; ++m) {
        eu[v][m] = make_double2(0.0, 0.0);
        if (in[m] && SGNB_INB(row0 + kp + step(m), Nd)) eu[v][m] = load_pair(u0 + v * Nd + step(m), bulk, two[m]);
      }
  }
  // ---- nodes across the tile's edges: one (slot, transverse node) per thread, five fields ---
#pragma unroll
  for (int q = tid; q < NHALO * NP; q += LTHR) {
    const int slot = q / NP, t = q - NP * slot;
    const double* gh = nullptr;
    bool ok;
    int ex, ey, node;
    if (slot < 2 * TY) {
      const bool right = slot >= TY;
      const int r = right ? slot - TY : slot;
      ey = ey0 + r;
      ex = right ? (ex0 + TXv == Nx ? 0 : ex0 + TXv) : (ex0 == 0 ? Nx - 1 : ex0 - 1);
      node = (right ? 0 : NP - 1) + NP * t;
      ok = r < TYv && !(right ? wallR : wallL);
      if constexpr (GHOST) gh = right ? (ghostR ? C.ghostR : nullptr) : (ghostL ? C.ghostL : nullptr);
    } else {
      const bool top = slot >= 2 * TY + TX;
      const int r = slot - 2 * TY - (top ? TX : 0);
      ex = ex0 + r;
      ey = top ? (ey0 + TYv == Ny ? 0 : ey0 + TYv) : (ey0 == 0 ? Ny - 1 : ey0 - 1);
      node = t + (top ? 0 : NP * (NP - 1));
      ok = r < TXv && !(top ? wallT : wallB);
    }
    if (ok) {
      double val[NV];
      if (GHOST && gh != nullptr) {
        const long long o = (long long)ey * NP + t, fs = (long long)Ny * NP;
#pragma unroll
        for (int v = 0; v < NV; ++v) val[v] = SGNB_INB(o, fs) ? gh[v * fs + o] : 0.0;
      } else {
        const int g = (ex + Nx * ey) * NPP + node;
        if (SGNB_INB(g, Nd)) {
#pragma unroll
          for (int v = 0; v < NV; ++v) val[v] = src[v * Nd + g];
          if constexpr (AXPY) {
            double kv[NV];
#pragma unroll
            for (int v = 0; v < NV; ++v) kv[v] = kin[v * Nd + g];
#pragma unroll
            for (int v = 0; v < NV; ++v) val[v] = stage_axpy(val[v], acoef, kv[v]);
          }
        }
      }
#pragma unroll
      for (int v = 0; v < NV; ++v) S.U[v][TN + q] = val[v];
    }
  }

  // exact mode: the depths of the faces at both ends of this lane's two lines
  const int ce = kColumnLane[lane] >> 3, cj = kColumnLane[lane] & 7;  // column pass: element, line
  double fy0 = 0.0, fy1 = 0.0, fx0 = 0.0, fx1 = 0.0;
  auto in_mesh = [&](int e) { return COL ? el_x(e) < TXv && el_y(e) < TYv : e < RXv; };
  if constexpr (EXACT) {
    if (lane < LROW * NP && in_mesh(ce)) {
      const int ex = ex0 + el_x(ce), ey = ey0 + el_y(ce);
      const bool end = C.bcy && ey + 1 == Ny;
      const long long f0 = ((long long)ex + (long long)Nx * ey) * NP + cj;
      const long long f1 = end ? (long long)ex * NP + cj
                               : ((long long)ex + (long long)Nx * (ey + 1 == Ny ? 0 : ey + 1)) * NP + cj;
      if (SGNB_INB(f0, Nd / NP)) fy0 = C.HfY[f0];
      if (SGNB_INB(f1, end ? (long long)Nx * NP : Nd / NP)) fy1 = (end ? C.HfYEnd : C.HfY)[f1];
    }
    if (lane < LROW * NP && in_mesh(lane / NP)) {
      const int ex = ex0 + el_x(lane / NP), ey = ey0 + el_y(lane / NP), t = lane % NP;
      const bool end = ex + 1 == Nx && (C.bcx || ghostR);
      const long long f0 = ((long long)ex + (long long)Nx * ey) * NP + t;
      const long long f1 = end ? (long long)ey * NP + t
                               : ((long long)(ex + 1 == Nx ? 0 : ex + 1) + (long long)Nx * ey) * NP + t;
      if (SGNB_INB(f0, Nd / NP)) fx0 = C.HfX[f0];
      if (SGNB_INB(f1, end ? (long long)Ny * NP : Nd / NP)) fx1 = (end ? C.HfXEnd : C.HfX)[f1];
    }
  }

  // ---- this warp's row has landed; stage input u + (c dt) k in place; then the whole tile ---
  const bool cvalid = lane < LROW * NP && in_mesh(ce);
  double* const uc = &S.U[0][s0 + ce * NPP + cj];
  if (!bulk) cp_async_wait_all();
  if (bulk) {
    bool landed = RXv == 0;
    for (int it = 0; it < kTmaTries && !landed; ++it) landed = mbar_try_wait(mbar, 0);
    if (!landed) {
      // the copies did not complete: as long again, so that none lands after this CTA has left its
      // shared memory, and NaN, so that the launch's results are non-finite and the controller
      // ends the run with that error
      for (int it = 0; it < kTmaTries && !landed; ++it) landed = mbar_try_wait(mbar, 0);
      uc[0] = __longlong_as_double(0x7ff8000000000000LL);
    }
  }
  if constexpr (MAYBE_CAND) __syncthreads();  // the stash's address
  else if constexpr (AXPY) __syncwarp();             // the lanes' own copies
  if constexpr (AXPY) {
    // in the linear order of the row (no bank conflicts, 16 bytes per access), the next field's
    // reads ahead of this one's writes
    double2 x[2][LPF], y[2][LPF];
    auto read = [&](int v) {
#pragma unroll
      for (int m = 0; m < LPF; ++m) {
        x[v & 1][m] = y[v & 1][m] = make_double2(0.0, 0.0);
        if (in[m]) {
          x[v & 1][m] = *(const double2*)&S.U[v][s0 + kp + 2 * LPL * m];
          y[v & 1][m] = *(const double2*)&ks[v * TN + s0 + kp + 2 * LPL * m];
        }
      }
    };
    read(0);
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      if (v + 1 < NV) read(v + 1);
      const double2(&xv)[LPF] = x[v & 1];
      const double2(&yv)[LPF] = y[v & 1];
#pragma unroll
      for (int m = 0; m < LPF; ++m)
        if (in[m])
          *(double2*)&S.U[v][s0 + kp + 2 * LPL * m] =
              make_double2(stage_axpy(xv[m].x, acoef, yv[m].x), stage_axpy(xv[m].y, acoef, yv[m].y));
      if (MAYBE_CAND && cand) {
        __syncwarp();
        const unsigned st = S.stash + ((unsigned)w << 21) + 4 * LPF * v;
        stash_put(st, xv);
        stash_put(st + 4 * LPF * NV, yv);
      }
    }
  }
  __syncthreads();
  if constexpr (MODE == MODE_FSAL) {
    const unsigned st = S.stash + ((unsigned)w << 21);
#pragma unroll
    for (int v = 0; v < NV; ++v) stash_put(st + 4 * LPF * v, eu[v]);
  }

  // ---- column pass: y-lines ----------------------------------------------------------
  if (cvalid) {
    const int ix = el_x(ce), iy = el_y(ce);
    const bool mlo = iy == 0 && wallB, mhi = iy + 1 >= TYv && wallT;
    const double* const lo = mlo ? uc : (iy > 0 ? uc - TX * NPP + NP * (NP - 1) : &S.U[0][TN + (2 * TY + ix) * NP + cj]);
    const double* const hi = mhi ? uc + NP * (NP - 1)
                                 : (iy + 1 < TYv ? uc + TX * NPP : &S.U[0][TN + (2 * TY + TX + ix) * NP + cj]);
    const int o = s0 + ce * NPP + cj;
    double* const gp = &S.G[0][o];
    if constexpr (EXACT) {
      double Un[NP][NV], Hn[NP], nLo[NV], nHi[NV];
#pragma unroll
      for (int b = 0; b < NP; ++b) {
#pragma unroll
        for (int v = 0; v < NV; ++v) Un[b][v] = uc[v * US + b * NP];
        Hn[b] = S.H[o + b * NP];
      }
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        nLo[v] = lo[v * US];
        nHi[v] = hi[v * US];
      }
      if (mlo) nLo[2] = -nLo[2];
      if (mhi) nHi[2] = -nHi[2];
      line_pass<true, 1>(
          C, T, Un, Hn, nLo, nHi, fy0, fy1,
          [&](int b, double dh, const Prim<true>& q) { gp[NV * TN + b * NP] = C.mc2 * q.v * dh; },
          [&](int b, int v, double d, const Prim<true>&) { gp[v * TN + b * NP] = d; });
    } else {
      line_terms<1, US, false, MODE == MODE_FSAL>(C, T, uc, &S.H[o], lo, hi, mlo ? -1.0 : 1.0, mhi ? -1.0 : 1.0,
                               [&](int v, int k, double r) { gp[v * TN + k * NP] = r; });
    }
  }
  __syncwarp();
  let_next_start();
  // ---- row pass: x-lines, completes dU --------------------------------------------------
  {
    const int e = lane / NP, j = lane - NP * e, ix = el_x(e), iy = el_y(e);
    if (lane < LROW * NP && in_mesh(e)) {
      const int o = s0 + NP * lane;
      const double* const u = &S.U[0][o];
      const bool mlo = ix == 0 && wallL, mhi = ix + 1 >= TXv && wallR;
      const double* const lo = mlo ? u : (ix > 0 ? u - NPP + (NP - 1) : &S.U[0][TN + iy * NP + j]);
      const double* const hi = mhi ? u + (NP - 1) : (ix + 1 < TXv ? u + NPP : &S.U[0][TN + (TY + iy) * NP + j]);
      double* const gp = &S.G[0][o];
      if constexpr (EXACT) {
        double Un[NP][NV], Hn[NP], nLo[NV], nHi[NV], dhx[NP];
        const double* const He = &S.H[s0 + e * NPP];
#pragma unroll
        for (int a = 0; a < NP; ++a) {
#pragma unroll
          for (int v = 0; v < NV; ++v) Un[a][v] = u[v * US + a];
          Hn[a] = S.H[o + a];
        }
#pragma unroll
        for (int v = 0; v < NV; ++v) {
          nLo[v] = lo[v * US];
          nHi[v] = hi[v * US];
        }
        if (mlo) nLo[1] = -nLo[1];
        if (mhi) nHi[1] = -nHi[1];
        line_pass<true, 0>(
            C, T, Un, Hn, nLo, nHi, fx0, fx1, [&](int a, double dh, const Prim<true>&) { dhx[a] = dh; },
            [&](int a, int v, double d, const Prim<true>& q) {
              gp[v * TN + a] = assemble<true, FRIC>(C, T, Un[a][0], Hn[a], He, a, j, v, d, gp[v * TN + a], dhx[a],
                                                    gp[NV * TN + a], q);
            });
      } else {
        line_terms<0, US, FRIC, MODE == MODE_FSAL>(C, T, u, &S.H[o], lo, hi, mlo ? -1.0 : 1.0, mhi ? -1.0 : 1.0,
                                [&](int v, int k, double r) { gp[v * TN + k] = -r - gp[v * TN + k]; });
      }
    }
  }
  const bool bulk_out = bulk && !cand;
  if (bulk_out) asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  __syncwarp();

  // ---- results ---------------------------------------------------------------------
  if (!(MAYBE_CAND && cand)) {
    double* __restrict__ outp = MODE == MODE_FSAL ? pick(A.K1, cur ^ 1) : A.out;
    if (bulk_out) {
      const int f = COL ? lane % NV : lane, r = COL ? lane / NV : 0, g = row0 + r * next_row;
      if (f < NV && r < RYv && RXv > 0 && SGNB_INB(g, Nd - rowv + 1))
        bulk_store(outp + f * Nd + g, smem_addr(&S.G[f][s0 + r * WRUN]), (unsigned)rowv * sizeof(double));
    } else {
#pragma unroll
      for (int v = 0; v < NV; ++v)
#pragma unroll
        for (int m = 0; m < LPF; ++m)
          if (in[m] && SGNB_INB(row0 + kp + step(m), Nd))
            store_pair(outp + v * Nd + row0 + kp + step(m), *(const double2*)&S.G[v][s0 + kp + 2 * LPL * m],
                       false, two[m]);
    }
  }
  if (MAYBE_CAND && cand) {
    // k3 is used up here: the candidate uNew = u + dt (2/9 k1 + 1/3 k2 + 4/9 k3) and the part
    // 7/24 k1 + 1/4 k2 + 1/3 k3 of the embedded solution leave instead (rk.cpp:106-121)
    const double* k1 = pick(A.K1, cur) + row0 + kp;
    double* __restrict__ un = pick(A.U, cur ^ 1) + row0 + kp;
    double* __restrict__ pe = A.K3 + row0 + kp;
    // a rolled loop over the fields (unrolled, warps waited for instructions), the next field's
    // k1 in flight
    double2 b[LPF], nb[LPF];
    auto load = [&](int v, double2 (&x)[LPF]) {
#pragma unroll
      for (int m = 0; m < LPF; ++m)
        if (in[m] && SGNB_INB(row0 + kp + step(m), Nd)) x[m] = load_pair(k1 + v * Nd + step(m), bulk, two[m]);
    };
    load(0, nb);
    stash_put_wait();
    const unsigned st = S.stash + ((unsigned)w << 21);
#pragma unroll 1
    for (int v = 0; v < NV; ++v) {
#pragma unroll
      for (int m = 0; m < LPF; ++m) b[m] = nb[m];
      if (v + 1 < NV) load(v + 1, nb);
      double2 a[LPF], c[LPF];
      __syncwarp();
      stash_get(st + 4 * LPF * v, a);
      stash_get(st + 4 * LPF * (NV + v), c);
#pragma unroll
      for (int m = 0; m < LPF; ++m) {
        const double2 k3 = *(const double2*)&S.G[v][s0 + kp + 2 * LPL * m];  // (within shared memory)
        double2 x, p;
        x.x = fsal_finish(a[m].x, fsal_part(b[m].x, c[m].x), k3.x, dt);
        x.y = fsal_finish(a[m].y, fsal_part(b[m].y, c[m].y), k3.y, dt);
        p.x = emb_part(b[m].x, c[m].x, k3.x);
        p.y = emb_part(b[m].y, c[m].y, k3.y);
        if (in[m] && SGNB_INB(row0 + kp + step(m), Nd)) {
          store_pair(un + v * Nd + step(m), x, bulk, two[m]);
          store_pair(pe + v * Nd + step(m), p, bulk, two[m]);
        }
      }
    }
  }
  if constexpr (GHOST && AXPY) {
    // Fused edge exchange (as in fused_tile): the next stage's input at the slab's edge nodes of
    // this row, straight into the neighbours' ghost arrays
    const bool outLo = C.edgeL != nullptr && ex0 == 0 && wx == 0;
    const bool outHi = C.edgeR != nullptr && ex0 + wx * LROW + RXv == Nx;
    if (RXv > 0 && (outLo || outHi)) {
      const double* u0 = pick(A.U, cur);
      const double* k1 = pick(A.K1, cur);
      const double* k2 = A.K2;
      for (int q = lane; q < 2 * NV * NP * RYv; q += 32) {
        const int row = q / (2 * NV * NP), qr = q - row * 2 * NV * NP;
        const int side = qr / (NV * NP), r = qr - side * NV * NP, t = r % NP, v = r / NP;
        if (side == 0 ? !outLo : !outHi) continue;
        const int at = side == 0 ? NP * t : (RXv - 1) * NPP + NP - 1 + NP * t;
        const long long g = (long long)v * Nd + row0 + row * next_row + at;
        const double kout = S.G[v][s0 + row * WRUN + at];
        const long long ge = (long long)v * Ny * NP + (long long)(ey0 + iy0 + row) * NP + t;
        if (!SGNB_INB(g, NV * Nd) || !SGNB_INB(ge, (long long)NV * Ny * NP)) continue;
        (side == 0 ? C.edgeL : C.edgeR)[ge] =
            cand ? fsal_finish(u0[g], fsal_part(k1[g], k2[g]), kout, dt) : stage_axpy(u0[g], 0.75 * dt, kout);
      }
    }
  }
  if constexpr (MODE == MODE_FSAL) {
    // scaled embedded error (rk.cpp:118-128) of the row, then of the tile
    const CtrlReload rc = ctrl_reload(A.ctrl);
    double esum = 0.0, emax = 0.0;
    const double* pe = A.K3 + row0 + kp;
    double2 p[LPF], np[LPF];
    auto load = [&](int v, double2 (&x)[LPF]) {
#pragma unroll
      for (int m = 0; m < LPF; ++m)
        if (in[m] && SGNB_INB(row0 + kp + step(m), Nd)) x[m] = load_pair(pe + v * Nd + step(m), bulk, two[m]);
    };
    load(0, np);
    stash_put_wait();
    const unsigned st = S.stash + ((unsigned)w << 21);
    // every lane computes every value, and those outside the mesh are dropped by selection (their
    // operands are whatever shared memory holds): branches would keep the values from overlapping
    auto errors = [&](auto divide) {
      auto err = [&](double u, double q, double un, double k4, bool there) {
        const double au = fabs(u), an = fabs(un), am = au < an ? an : au;
        double rr;
        if constexpr (EXACT) rr = (un - (u + rc.dt * (q + 0.125 * k4))) / (rc.atol + rc.rtol * am);
        else rr = divide(un - fma(rc.dt, fma(0.125, k4, q), u), fma(rc.rtol, am, rc.atol));
        rr = there ? rr : 0.0;
        esum = EXACT ? esum + rr * rr : fma(rr, rr, esum);  // a NaN stays in the sum
        const double ar = fabs(rr);
        emax = emax < ar ? ar : emax;
      };
#pragma unroll 1
      for (int v = 0; v < NV; ++v) {
#pragma unroll
        for (int m = 0; m < LPF; ++m) p[m] = np[m];
        if (v + 1 < NV) load(v + 1, np);
        double2 a[LPF];
        __syncwarp();
        stash_get(st + 4 * LPF * v, a);
#pragma unroll
        for (int m = 0; m < LPF; ++m) {
          const double2 un = *(const double2*)&S.U[v][s0 + kp + 2 * LPL * m];
          const double2 k4 = *(const double2*)&S.G[v][s0 + kp + 2 * LPL * m];
          err(a[m].x, p[m].x, un.x, k4.x, in[m]);
          err(a[m].y, p[m].y, un.y, k4.y, in[m] && two[m]);
        }
      }
    };
    // the fast mode's reciprocal where the scale is a normal number: everywhere if atol is one, else
    // value by value (a purely relative tolerance; a division by every scale instead took 20 steps
    // of 512 x 256 elements from 7.59 to 7.91 ms, this takes 7.83)
    constexpr double kNormal = 2.2250738585072014e-308;
    if (EXACT || rc.atol >= kNormal) errors([](double e, double sc) { return e * fast_rcp(sc); });  // (exact: divides)
    else errors([](double e, double sc) { return sc >= kNormal ? e * fast_rcp(sc) : e / sc; });
    reduce_error<LWARPS>(esum, emax, esum != esum, S.red, A.partials, blk);
  }
  if (bulk_out && lane < NV * WR) bulk_store_wait();  // shared memory is read out
  if (bulk) {
    // a persistent CTA's next tile: its copies write what this one read and wrote, and its
    // warps initialise their barriers again
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    __syncwarp();
    if (lane == 0) mbar_inval(mbar);
  }
}

// FRIC: Manning friction compiled in. GHOST: slab edges compiled in.
template <int MODE, bool FRIC, bool GHOST>
__global__ void __launch_bounds__(LTHR, (kLineCtas<MODE, 1>))
    k_line(const LineConsts C, const LineTables T, const StageArgs A) {
  extern __shared__ __align__(128) unsigned char smem_line[];
  auto& S = *reinterpret_cast<typename LineTile<1>::Smem*>(smem_line);
  if (kStash<MODE> && threadIdx.x < 32) stash_alloc(&S.stash);
  wait_for_previous();
  line_tile<MODE, 1, FRIC, GHOST>(C, T, A, blockIdx.x, blockIdx.y,
                                  (long long)blockIdx.y * gridDim.x + blockIdx.x, C.bulk != 0, S);
  if constexpr (kStash<MODE>) {
    __syncthreads();
    if (threadIdx.x < 32) stash_free(S.stash);
  }
}

// The exact mode's: the reference's operation order and IEEE divisions in the same tiles. At most
// three CTAs per SM fit (62 KB with the sixth field of column results); CTAS: the number that the
// registers are set for. Such a kernel is 115 to 140 KB of instructions, executed once per warp, and
// an attempt's kernels put each other's out of the instruction caches: both stages are one kernel
// (MODE_STAGES; 200 x 100 elements, an attempt: 221 us with two, 211 with one).
template <int MODE, bool FRIC, bool GHOST, bool COL, int CTAS>
__global__ void __launch_bounds__(LTHR, CTAS) k_line_exact(const RhsConsts C, const StageArgs A, const int bulk) {
  extern __shared__ __align__(128) unsigned char smem_line_exact[];
  auto& S = *reinterpret_cast<typename LineTile<1, true, COL>::Smem*>(smem_line_exact);
  if (kStash<MODE> && threadIdx.x < 32) stash_alloc(&S.stash);
  wait_for_previous();
  line_tile<MODE, 1, FRIC, GHOST, true, COL>(C, C, A, blockIdx.x, blockIdx.y,
                                             (long long)blockIdx.y * gridDim.x + blockIdx.x, bulk != 0, S);
  if constexpr (kStash<MODE>) {
    __syncthreads();
    if (threadIdx.x < 32) stash_free(S.stash);
  }
}

}  // namespace dev
}  // namespace sgnb
