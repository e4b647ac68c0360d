// sgnb_kernels_line.cuh -- the fast arithmetic mode's fused right-hand-side and stage
// kernels on Gauss-Lobatto points (single instances, slabs and batches). The mixed mode runs
// the same kernels with its stage derivatives k1, k2, k4 and the embedded part stored in FP32.
//
// Same tile and thread layout as sgnb_kernels.cuh (a CTA of 5 warps owns 32 elements; lane
// i of every warp is tile element i, warp j its j-th line of solution points), with the
// arithmetic arranged for the fast mode:
//   * every flux component is the normal velocity times a state component, F = u_n U_v (plus
//     the hydrostatic term and c^2 h u_n where they belong), so a line keeps u_n and reads one
//     field at a time from shared memory;
//   * the Rusanov flux minus the element's own face flux is half the flux difference of the
//     two traces plus the dissipation, in which the face depth cancels (both traces take the
//     same one): no face depths are read;
//   * the GLL differentiation matrix changes sign under reflection of its rows and columns and
//     the two correction functions mirror each other, so a 5-point derivative with both
//     lifts splits into an even and an odd half (27 operations instead of 35);
//   * each pass adds its own direction's sources, so no pass differentiates the depth along
//     the other direction, and h_n and H_n of the hp equation share one derivative.
// What bounds it: the FP64 pipe and HBM are both within 1.5x of each other at the target
// (about 190 FP64 instructions and 90 to 130 bytes per node), so what matters is enough warps to
// overlap them: 128 registers and 75 KB of shared memory per CTA, three CTAs per SM.
#pragma once

#include "sgnb_kernels.cuh"

namespace sgnb {
namespace dev {

// Shared memory of one tile. Field v of the tile's nodes and of the nodes across its edges lie
// in one block, so a line's neighbour is reached with the line's own field stride:
//   U[v][i * 25 + a + 5 b]        node (a, b) of tile element i
//   U[v][800 + 5 * slot + t]      halo slots as in Tile (left, right, bottom, top)
template <int TX_, int TY_>
struct LineTile {
  static constexpr int TX = TX_, TY = TY_;
  static_assert(TX * TY == TE && TX % 2 == 0, "one tile element per lane, rows of whole pairs");
  static constexpr int NHALO = 2 * TY + 2 * TX;
  static constexpr int TN = TE * NPP;             // nodes per tile
  static constexpr int US = TN + NHALO * NP;      // field stride of U
  static constexpr int RUN = TX * NPP;            // doubles per tile row
  struct Smem {
    double U[NV][US];
    double H[TN];
    double G[NV][TN];        // stage derivative on load; column-pass results; then dU
    double red[NWARP][3];
    unsigned long long mbar;
  };
};

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

// Per-thread asynchronous copy of one value of 4 or 8 bytes.
template <int BYTES>
__device__ __forceinline__ void cp_async(void* smem, const void* gmem) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(smem_addr(smem)), "l"(gmem), "n"(BYTES) : "memory");
}
template <class T> struct Pair;
template <> struct Pair<double> { using type = double2; };
template <> struct Pair<float> { using type = float2; };
// Two neighbouring values, in one access where rows start aligned (vec); the second one only if
// two. The same values reach the same thread either way, so both ways give the same sums.
// Streaming (evict-first) accesses: no other CTA reads these lines soon.
template <class T>
__device__ __forceinline__ typename Pair<T>::type load_pair(const T* p, bool vec, bool two) {
  using T2 = typename Pair<T>::type;
  if (vec) return __ldcs((const T2*)p);
  T2 r;
  r.x = __ldcs(p);
  r.y = two ? __ldcs(p + 1) : T(0);
  return r;
}
template <class T>
__device__ __forceinline__ void store_pair(T* p, typename Pair<T>::type x, bool vec, bool two) {
  if (vec) {
    __stcs((typename Pair<T>::type*)p, x);
  } else {
    __stcs(p, x.x);
    if (two) __stcs(p + 1, x.y);
  }
}

// Derivative of the five values F along a line plus the lifts of the face jumps jl, jr, all
// before the division by J.
template <class TE_>
__device__ __forceinline__ void line_derivative(const TE_& T, const double (&F)[NP], double jl,
                                                double jr, double (&d)[NP]) {
  const double o0 = F[0] - F[4], o1 = F[1] - F[3];
  const double e0 = fma(-2.0, F[2], F[0] + F[4]), e1 = fma(-2.0, F[2], F[1] + F[3]);
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
  const double e0 = fma(-2.0, F[2], F[0] + F[4]), e1 = fma(-2.0, F[2], F[1] + F[3]);
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
template <int DIR, int US, bool FRIC, class TC, class TE_, class Emit>
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
    const double a = fma(g, hh, pp) + c2;
    return fabs(uu) + fast_sqrt(a > 0.0 ? a : 0.0);
  };
  const double lamL = 0.5 * fmax(speed(hL, hpL * ihL, unL), speed(h[0], hp[0] * ih[0], un[0]));
  const double lamR = 0.5 * fmax(speed(h[4], hp[4] * ih[4], un[4]), speed(hR, hpR * ihR, unR));
  const double dnL = hnL - hn[0], dnR = hnR - hn[4];
  double F[NP], d[NP];
  // hp: flux u_n hp + c^2 h u_n; the non-conservative product -c^2 u_n h_n and the source
  // -2 c^2 u_n H_n together are -c^2 u_n (h - 2 H)_n
  {
    double dh[NP];
#pragma unroll
    for (int k = 0; k < NP; ++k) F[k] = fma(-2.0, hl[k * SN], h[k]);
    line_derivative(T, F, 0.5 * (hL - h[0]), 0.5 * (hR - h[4]), dh);
#pragma unroll
    for (int k = 0; k < NP; ++k) F[k] = fma(un[k], hp[k], c2 * hn[k]);
    const double jl = fma(0.5, fma(unL, hpL, fma(c2, dnL, -un[0] * hp[0])), lamL * (hpL - hp[0]));
    const double jr = fma(0.5, fma(unR, hpR, fma(c2, dnR, -un[4] * hp[4])), lamR * (hp[4] - hpR));
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
    line_derivative(T, F, fma(0.5, fl, lamL * dnL), fma(0.5, fr, -lamR * dnR), d);
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
  line_derivative(T, hn, fma(0.5, dnL, lamL * (hL - h[0])), fma(0.5, dnR, lamR * (h[4] - hR)), d);
#pragma unroll
  for (int k = 0; k < NP; ++k) emit(0, k, iJ * d[k]);
}

// One tile. bulk: rows are copied by the bulk copy engine (Nx even, so every row starts
// 16-byte aligned in every buffer); otherwise by per-thread 8-byte copies.
template <int MODE, int TX_, int TY_, bool FRIC, bool GHOST, class K, class TC, class TE_, class TA>
__device__ __forceinline__ void line_tile(const TC& C, const TE_& T, const TA& A, int bx, int by,
                                          long long blk, const bool bulk,
                                          typename LineTile<TX_, TY_>::Smem& S) {
  using L = LineTile<TX_, TY_>;
  constexpr int TX = L::TX, TY = L::TY, NHALO = L::NHALO, TN = L::TN, US = L::US, RUN = L::RUN;
  constexpr bool AXPY = MODE == MODE_STAGE || MODE == MODE_CAND;
  using KT = K;                                  // storage type of the stage derivatives
  constexpr bool K32 = sizeof(KT) == 4;

  // ---- controller state -----------------------------------------------------------
  int cur = 0;
  double dt = 0.0, acoef = 0.0;
  if constexpr (MODE != MODE_RHS) {
    if (A.ctrl->done) return;  // uniform across the grid
    cur = A.ctrl->cur;
    dt = A.ctrl->dt;
    acoef = A.coef * dt;
  }
  const double* __restrict__ src = MODE == MODE_RHS ? A.in : (MODE == MODE_FSAL ? pick(A.U, cur ^ 1) : pick(A.U, cur));
  const KT* __restrict__ kin = AXPY ? (A.kin_k2 ? A.K2 : pick(A.K1, cur)) : nullptr;

  int tid;
  asm volatile("mov.u32 %0, %%tid.x;" : "=r"(tid));
  const int j = tid >> 5, i = tid & 31;  // line index of this warp, tile element of this lane
  const int Nx = C.Nx, Ny = C.Ny;
  const long long Nd = C.Nd;
  const int ex0 = bx * TX, ey0 = by * TY;
  const int TXv = min(TX, Nx - ex0), TYv = min(TY, Ny - ey0);
  bool ghostL = false, ghostR = false;
  if constexpr (GHOST) {
    ghostL = C.ghostL != nullptr && ex0 == 0;
    ghostR = C.ghostR != nullptr && ex0 + TXv == Nx;
  }
  const bool wallL = C.bcx && ex0 == 0 && !ghostL, wallR = C.bcx && ex0 + TXv == Nx && !ghostR;
  const bool wallB = C.bcy && ey0 == 0, wallT = C.bcy && ey0 + TYv == Ny;
  const int row0 = (ex0 + Nx * ey0) * NPP;  // the tile's first node within a field (Nd < 2^31)

  // ---- own nodes ------------------------------------------------------------------
  const unsigned mbar = smem_addr(&S.mbar);
  KT* const ks = reinterpret_cast<KT*>(&S.G[0][0]);  // the stage derivative, until the passes
  if (bulk) {
    const unsigned bytes = (unsigned)TXv * NPP * sizeof(double), kbytes = (unsigned)TXv * NPP * sizeof(KT);
    if (tid == 0) {
      mbar_init(mbar);
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
      mbar_expect_tx(mbar, TYv * ((NV + 1) * bytes + (AXPY ? NV * kbytes : 0)));
    }
    __syncthreads();
    // one row copy per thread, spread over the warps (a warp issues its lanes' copies one by
    // one); the rows that the epilogue reads start their way to L2 as well
    constexpr int NARR = AXPY ? 2 : 1;
    for (int q = i * NWARP + j; q < (NARR * NV + 1) * TY; q += NTHR) {
      const int iy = q % TY, f = q / TY;
      if (iy >= TYv) continue;
      int g = row0 + Nx * NPP * iy;
      if (!SGNB_INB(g, Nd - TXv * NPP + 1)) g = 0;
      if (f == 0) bulk_load(smem_addr(&S.H[iy * RUN]), C.Hnod + g, bytes, mbar);
      else if (f <= NV) bulk_load(smem_addr(&S.U[f - 1][iy * RUN]), src + (f - 1) * Nd + g, bytes, mbar);
      else bulk_load(smem_addr(ks + (f - 1 - NV) * TN + iy * RUN), kin + (f - 1 - NV) * Nd + g, kbytes, mbar);
    }
    if constexpr (MODE == MODE_CAND || MODE == MODE_FSAL) {
      for (int q = i * NWARP + j; q < (MODE == MODE_CAND ? 1 : 2) * NV * TY; q += NTHR) {
        const int iy = q % TY, f = q / TY, v = f % NV;
        const int g = row0 + Nx * NPP * iy;
        if (iy >= TYv || !SGNB_INB(g, Nd - TXv * NPP + 1)) continue;
        if (MODE == MODE_CAND) bulk_prefetch(pick(A.K1, cur) + v * Nd + g, kbytes);
        else if (f < NV) bulk_prefetch(pick(A.U, cur) + v * Nd + g, bytes);
        else bulk_prefetch(A.K3 + v * Nd + g, kbytes);
      }
    }
  } else {
#pragma unroll
    for (int m = 0; m < NIT; ++m) {
      const int q = tid + NTHR * m, iy = q / RUN, k = q - iy * RUN;
      if (iy < TYv && k < TXv * NPP) {
        const int g = row0 + Nx * NPP * iy + k;
        if (!SGNB_INB(g, Nd)) continue;
        cp_async<8>(&S.H[q], C.Hnod + g);
#pragma unroll
        for (int v = 0; v < NV; ++v) {
          cp_async<8>(&S.U[v][q], src + v * Nd + g);
          if constexpr (AXPY) cp_async<sizeof(KT)>(ks + v * TN + q, kin + v * Nd + g);
        }
      }
    }
  }
  // ---- nodes across the tile's edges: one (slot, transverse node) per thread, five fields ---
#pragma unroll
  for (int q = tid; q < NHALO * NP; q += NTHR) {
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
            KT kv[NV];
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
  if (!bulk) cp_async_wait_all();
  __syncthreads();  // halo, per-thread copies and the barrier's initialisation
  bool landed = true;
  if (bulk) {
    landed = false;
    for (int it = 0; it < kTmaTries && !landed; ++it) landed = mbar_try_wait(mbar, 0);
  }

  const int ix = i % TX, iy = i / TX;
  const bool valid = ix < TXv && iy < TYv;

  // ---- column pass: y-line a = j ---------------------------------------------------
  {
    double* const u = &S.U[0][i * NPP + j];
    if constexpr (AXPY) {
      // the stage input u + (c dt) k, in place: this warp alone touches the lines a = j here
      if (valid) {
#pragma unroll
        for (int v = 0; v < NV; ++v)
#pragma unroll
          for (int b = 0; b < NP; ++b)
            u[v * US + b * NP] = stage_axpy(u[v * US + b * NP], acoef, ks[v * TN + i * NPP + j + b * NP]);
      }
      // FP32 derivatives lie elsewhere than the results that overwrite them: every warp has
      // read its own
      if constexpr (K32) __syncthreads(); else __syncwarp();
    }
    // the copies did not complete: NaN, so that the launch's results are non-finite and the
    // controller ends the run with that error
    if (!landed) u[0] = __longlong_as_double(0x7ff8000000000000LL);
    if (valid) {
      const bool mlo = iy == 0 && wallB, mhi = iy + 1 >= TYv && wallT;
      const double* const lo = mlo ? u : (iy > 0 ? u - TX * NPP + NP * (NP - 1) : &S.U[0][TN + (2 * TY + ix) * NP + j]);
      const double* const hi = mhi ? u + NP * (NP - 1)
                                   : (iy + 1 < TYv ? u + TX * NPP : &S.U[0][TN + (2 * TY + TX + ix) * NP + j]);
      double* const gp = &S.G[0][i * NPP + j];
      line_terms<1, US, false>(C, T, u, &S.H[i * NPP + j], lo, hi, mlo ? -1.0 : 1.0, mhi ? -1.0 : 1.0,
                               [&](int v, int k, double r) { gp[v * TN + k * NP] = r; });
    }
  }
  __syncthreads();
  // ---- row pass: x-line b = j, completes dU -------------------------------------------
  if (valid) {
    const double* const u = &S.U[0][i * NPP + NP * j];
    const bool mlo = ix == 0 && wallL, mhi = ix + 1 >= TXv && wallR;
    const double* const lo = mlo ? u : (ix > 0 ? u - NPP + (NP - 1) : &S.U[0][TN + iy * NP + j]);
    const double* const hi = mhi ? u + (NP - 1) : (ix + 1 < TXv ? u + NPP : &S.U[0][TN + (TY + iy) * NP + j]);
    double* const gp = &S.G[0][i * NPP + NP * j];
    line_terms<0, US, FRIC>(C, T, u, &S.H[i * NPP + NP * j], lo, hi, mlo ? -1.0 : 1.0, mhi ? -1.0 : 1.0,
                            [&](int v, int k, double r) { gp[v * TN + k] = -r - gp[v * TN + k]; });
  }
  // the results leave as they lie in shared memory (FP64 rows by bulk copies), or rounded to
  // the storage type of the stage derivatives
  double* out64 = nullptr;
  KT* outk = nullptr;
  if constexpr (MODE == MODE_RHS) {
    if constexpr (K32) { out64 = A.outd; outk = A.out; }  // the head of a run has no outd
    else out64 = A.out;
  } else if constexpr (MODE == MODE_STAGE || MODE == MODE_FSAL) {
    KT* o = MODE == MODE_FSAL ? pick(A.K1, cur ^ 1) : A.out;
    if constexpr (K32) outk = o; else out64 = o;
  }
  const bool bulk_out = bulk && MODE != MODE_CAND && (!K32 || out64 != nullptr);
  if (bulk_out) asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  __syncthreads();

  // ---- results ---------------------------------------------------------------------
  if constexpr (MODE != MODE_CAND) {
    if (bulk_out) {
      if (j == 0) {
        const unsigned bytes = (unsigned)TXv * NPP * sizeof(double);
        for (int q = i; q < NV * TY; q += 32) {
          const int r = q % TY, v = q / TY;
          const int g = row0 + Nx * NPP * r;
          if (r < TYv && SGNB_INB(g, Nd - TXv * NPP + 1))
            bulk_store(out64 + v * Nd + g, smem_addr(&S.G[v][r * RUN]), bytes);
        }
      }
    } else if (K32 && bulk) {
      if constexpr (K32) {
#pragma unroll
        for (int m = 0; m < (TN / 2 + NTHR - 1) / NTHR; ++m) {
          const int q = 2 * (tid + NTHR * m), r = q / RUN, k = q - r * RUN;
          const int g = row0 + Nx * NPP * r + k;
          if (r < TYv && k < TXv * NPP && SGNB_INB(g, Nd - 1)) {
#pragma unroll
            for (int v = 0; v < NV; ++v) {
              const double2 x = *(const double2*)&S.G[v][q];
              __stcs((float2*)(outk + v * Nd + g), make_float2((float)x.x, (float)x.y));
            }
          }
        }
      }
    } else {
#pragma unroll
      for (int m = 0; m < NIT; ++m) {
        const int q = tid + NTHR * m, r = q / RUN, k = q - r * RUN;
        const int g = row0 + Nx * NPP * r + k;
        if (r < TYv && k < TXv * NPP && SGNB_INB(g, Nd)) {
#pragma unroll
          for (int v = 0; v < NV; ++v) {
            if (!K32 || out64 != nullptr) __stcs(&out64[v * Nd + g], S.G[v][q]);
            else __stcs(&outk[v * Nd + g], (KT)S.G[v][q]);
          }
        }
      }
    }
  }
  // pairs of neighbouring nodes of this thread in one field of the tile, at 2 (tid + NTHR m):
  // their offset in the field (-1: outside the mesh)
  constexpr int NPR = (TN / 2 + NTHR - 1) / NTHR;
  int gof[NPR];
  bool two[NPR];
  if constexpr (MODE == MODE_CAND || MODE == MODE_FSAL) {
#pragma unroll
    for (int m = 0; m < NPR; ++m) {
      const int q = 2 * (tid + NTHR * m), r = q / RUN, k = q - r * RUN;
      gof[m] = r < TYv && k < TXv * NPP ? row0 + Nx * NPP * r + k : -1;
      two[m] = k + 1 < TXv * NPP;
    }
  }
  if constexpr (MODE == MODE_CAND) {
    // k3 is used up here: the candidate uNew = u + dt (2/9 k1 + 1/3 k2 + 4/9 k3) and the part
    // 7/24 k1 + 1/4 k2 + 1/3 k3 of the embedded solution leave instead (rk.cpp:106-121)
    const double* __restrict__ u0 = pick(A.U, cur);
    const KT* __restrict__ k1 = pick(A.K1, cur);
    const KT* __restrict__ k2 = A.K2;
    double* __restrict__ un = pick(A.U, cur ^ 1);
    KT* __restrict__ pe = A.K3;
    using KT2 = typename Pair<KT>::type;
    double2 a[NPR], na[NPR];
    KT2 b[NPR], c[NPR], nb[NPR], nc[NPR];
    auto load = [&](int v, double2 (&x)[NPR], KT2 (&y)[NPR], KT2 (&z)[NPR]) {
      const long long o = v * Nd;
#pragma unroll
      for (int m = 0; m < NPR; ++m)
        if (gof[m] >= 0 && SGNB_INB(o + gof[m], NV * Nd)) {
          x[m] = load_pair(u0 + o + gof[m], bulk, two[m]);
          y[m] = load_pair(k1 + o + gof[m], bulk, two[m]);
          z[m] = load_pair(k2 + o + gof[m], bulk, two[m]);
        }
    };
    load(0, a, b, c);
#pragma unroll 1
    for (int v = 0; v < NV; ++v) {
      if (v + 1 < NV) load(v + 1, na, nb, nc);  // the next field's, in flight
      const long long o = v * Nd;
#pragma unroll
      for (int m = 0; m < NPR; ++m)
        if (gof[m] >= 0 && SGNB_INB(o + gof[m], NV * Nd)) {
          const double2 k3 = *(const double2*)&S.G[v][2 * (tid + NTHR * m)];
          double2 x;
          KT2 p;
          x.x = fsal_finish(a[m].x, fsal_part(b[m].x, c[m].x), k3.x, dt);
          x.y = fsal_finish(a[m].y, fsal_part(b[m].y, c[m].y), k3.y, dt);
          p.x = (KT)emb_part(b[m].x, c[m].x, k3.x);
          p.y = (KT)emb_part(b[m].y, c[m].y, k3.y);
          store_pair(un + o + gof[m], x, bulk, two[m]);
          store_pair(pe + o + gof[m], p, bulk, two[m]);
        }
#pragma unroll
      for (int m = 0; m < NPR; ++m) { a[m] = na[m]; b[m] = nb[m]; c[m] = nc[m]; }
    }
  }
  if constexpr (GHOST && AXPY) {
    // Fused edge exchange (as in fused_tile): the next stage's input at the slab's edge
    // nodes, straight into the neighbours' ghost arrays
    const bool outLo = C.edgeL != nullptr && ex0 == 0, outHi = C.edgeR != nullptr && ex0 + TXv == Nx;
    if (outLo || outHi) {
      const double* __restrict__ u0 = pick(A.U, cur);
      const KT* __restrict__ k1 = pick(A.K1, cur);
      const KT* __restrict__ k2 = A.K2;
      const int per = NV * TYv * NP;
      for (int q = tid; q < 2 * per; q += NTHR) {
        const int side = q / per;
        if (side == 0 ? !outLo : !outHi) continue;
        const int r = q - side * per;
        const int t = r % NP, ry = (r / NP) % TYv, v = r / (NP * TYv);
        const int ixe = side == 0 ? 0 : TXv - 1;
        const int node = (side == 0 ? 0 : NP - 1) + NP * t;
        const long long g = (long long)v * Nd + ((long long)(ex0 + ixe) + (long long)Nx * (ey0 + ry)) * NPP + node;
        const double kout = S.G[v][(TX * ry + ixe) * NPP + node];
        const long long ge = (long long)v * Ny * NP + (long long)(ey0 + ry) * NP + t;
        if (!SGNB_INB(g, NV * Nd) || !SGNB_INB(ge, (long long)NV * Ny * NP)) continue;
        (side == 0 ? C.edgeL : C.edgeR)[ge] =
            MODE == MODE_STAGE ? stage_axpy(u0[g], 0.75 * dt, kout)
                               : fsal_finish(u0[g], fsal_part(k1[g], k2[g]), kout, dt);
      }
    }
  }
  if constexpr (MODE == MODE_FSAL) {
    // scaled embedded error (rk.cpp:118-128) of the tile
    const CtrlReload rc = ctrl_reload(A.ctrl);
    const double* __restrict__ u0 = pick(A.U, rc.cur);
    const KT* __restrict__ pe = A.K3;
    using KT2 = typename Pair<KT>::type;
    double esum = 0.0, emax = 0.0;
    // sc >= atol: where that is a normal number, so is sc, and the reciprocal of a few ulp serves
    const bool normal = rc.atol >= 2.2250738585072014e-308;
    auto err = [&](double u, double p, double un, double k4) {
      const double e = un - fma(rc.dt, fma(0.125, k4, p), u);
      const double au = fabs(u), an = fabs(un);
      const double sc = fma(rc.rtol, au < an ? an : au, rc.atol);
      const double rr = normal ? e * fast_rcp(sc) : e / sc;
      esum = fma(rr, rr, esum);  // a NaN stays in the sum
      const double ar = fabs(rr);
      emax = emax < ar ? ar : emax;
    };
    double2 a[NPR], na[NPR];
    KT2 p[NPR], np[NPR];
    auto load = [&](int v, double2 (&x)[NPR], KT2 (&y)[NPR]) {
      const long long o = v * Nd;
#pragma unroll
      for (int m = 0; m < NPR; ++m)
        if (gof[m] >= 0 && SGNB_INB(o + gof[m], NV * Nd)) {
          x[m] = load_pair(u0 + o + gof[m], bulk, two[m]);
          y[m] = load_pair(pe + o + gof[m], bulk, two[m]);
        }
    };
    load(0, a, p);
#pragma unroll 1
    for (int v = 0; v < NV; ++v) {
      if (v + 1 < NV) load(v + 1, na, np);  // the next field's, in flight
#pragma unroll
      for (int m = 0; m < NPR; ++m)
        if (gof[m] >= 0) {
          const int q = 2 * (tid + NTHR * m);
          const double2 un = *(const double2*)&S.U[v][q], k4 = *(const double2*)&S.G[v][q];
          err(a[m].x, p[m].x, un.x, k4.x);
          if (two[m]) err(a[m].y, p[m].y, un.y, k4.y);
        }
#pragma unroll
      for (int m = 0; m < NPR; ++m) { a[m] = na[m]; p[m] = np[m]; }
    }
    const int enan = esum != esum;
    reduce_error(esum, emax, enan, S.red, A.partials, blk);
  }
  if (bulk_out && j == 0) bulk_store_wait();  // shared memory is read out
  if (bulk) {
    // a persistent CTA's next tile: its copies write what this one read and wrote, and its
    // first thread initialises the barrier again
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    __syncthreads();
    if (tid == 0) mbar_inval(mbar);
  }
}

// FRIC: Manning friction compiled in. GHOST: slab edges compiled in. Args: StageArgs (FP64
// stage derivatives) or StageArgsM (FP32).
template <int MODE, bool FRIC, bool GHOST, class Args>
__global__ void __launch_bounds__(NTHR, 3) k_line(const RhsConsts C, const Args A, const int bulk) {
  extern __shared__ __align__(128) unsigned char smem_line[];
  auto& S = *reinterpret_cast<typename LineTile<8, 4>::Smem*>(smem_line);
  line_tile<MODE, 8, 4, FRIC, GHOST, typename Args::K>(C, C.eo, A, blockIdx.x, blockIdx.y,
                                                       (long long)blockIdx.y * gridDim.x + blockIdx.x, bulk != 0, S);
}

}  // namespace dev
}  // namespace sgnb
