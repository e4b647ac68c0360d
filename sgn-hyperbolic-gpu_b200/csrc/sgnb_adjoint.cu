// sgnb_adjoint.cu -- vector-Jacobian products of the right-hand side and of the BS3(2)
// update (no reference counterpart: the reference has no adjoint).
//
// R(U; H) is the FR discretisation of src/solver/sgn2d.cpp:125-290 as the fused kernels
// compute it (sgnb_kernels.cuh, line_pass and the assembly of the row pass): for every
// element and every GLL line in x and in y,
//   nodal fluxes F_k = flux(U_k, H_k)                       (sgn_flux2d.h:89-116)
//   face fluxes: Rusanov with lam = max(ws(s), ws(t))      (sgn_flux2d.h:169-179)
//   j = F* - F(own trace), dF_m = (sum_k D[m,k] F_k + jLo gL'[m] + jHi gR'[m]) / J
//   dh_m likewise with the central common depth            (sgn2d.cpp:265-275)
//   R -= dF; R[hp] -= -c^2 u_n dh  (non-conservative term, sgn_flux2d.h:150-161)
// plus the pointwise sources (sgn_flux2d.h:122-142, Manning friction included). Given a
// cotangent Rb of R, the line kernel reverses one line (one thread per element line and
// direction) and writes:
//   * the cotangent of the line's own nodes, per direction (each node lies on exactly one
//     x line and one y line of its element, so these are plain stores);
//   * the cotangent of the neighbour's trace node across each face (a per-face buffer the
//     gather kernel adds to the neighbour's node) or, at a wall, folded back through the
//     mirror ghost onto the own trace;
//   * the cotangents of the depth statics: nodal H (fluxes and sources) and the nodal dH/dx,
//     dH/dy (sources, x pass); that of the face depths is zero (they cancel in F* - F(own)).
// The gather kernel (one thread per node) sums the two directions and the neighbours'
// face contributions in a fixed order, so the result is deterministic without atomics,
// and folds in the RK-stage combination. Built with -fmad=true like the fast forward.
#include "sgnb_checked.cuh"
#include "sgnb_device.h"
#include "sgnb_fastmath.cuh"

namespace sgnb {
namespace dev {
namespace {

constexpr int NP = 5, NPP = 25, NV = 5;

__device__ __forceinline__ double stage_in(const VjpArgs& A, long long idx) {
  // y = u or u + (c dt) k, with the forward's rounding (stage_axpy of the fused kernels)
  return A.k ? __dadd_rn(A.u[idx], __dmul_rn(A.acoef, A.k[idx])) : A.u[idx];
}

__device__ __forceinline__ double sgn0(double x) { return x > 0.0 ? 1.0 : (x < 0.0 ? -1.0 : 0.0); }

// One line: reverse of its contribution to R (see the file comment). With the forward in the
// form F_v = u_n U_v (plus g/2 (h^2 - H^2) + hp in the normal discharge and c^2 h u_n in hp), the
// cotangent of a field's flux at a node goes to U_v and to u_n, and the fields can be taken one
// after the other: a field's cotangent and state are loaded when its turn comes, and what stays
// live is h, h u_n, hp, 1/h, u_n and their accumulators. (With every field's state, cotangent and
// result live at once the kernels took 254 registers, 8 warps per SM.) The Rusanov flux minus the
// own face flux does not depend on the face depth, so its cotangent is zero.
template <int DIR>
__device__ __forceinline__ void vjp_line(const RhsConsts& C, const FrTablesDev& T, const VjpArgs& A,
                                         long long idx) {
  const long long e = idx / NP;
  const int j = (int)(idx - e * NP);
  const int ex = (int)(e % C.Nx), ey = (int)(e / C.Nx);
  const long long Nd = C.Nd;
  constexpr int N = 1 + DIR, TG = 2 - DIR;  // normal and tangential discharge
  constexpr int SN = DIR == 0 ? 1 : NP;
  const long long g0 = e * NPP + (DIR == 0 ? NP * j : j);  // the line's first node
  const double iJ = DIR == 0 ? C.iJx : C.iJy, c2 = C.c2, gr = C.g;
  [[maybe_unused]] const bool line_ok = SGNB_INB(g0, Nd) && SGNB_INB(g0 + 4 * SN, Nd);
#ifdef SGNB_CHECKED
  if (!line_ok) return;
#endif
  auto state = [&](int v, long long g) { return stage_in(A, v * Nd + g); };
  auto cot = [&](int v, int m) {
    const long long g = v * Nd + g0 + SN * m;
    double r = A.alpha * A.ra[g];
    if (A.rb) r += A.beta * A.rb[g];
    return r;
  };
  // neighbour trace nodes
  const bool wallLo = DIR == 0 ? (C.bcx && ex == 0) : (C.bcy && ey == 0);
  const bool wallHi = DIR == 0 ? (C.bcx && ex == C.Nx - 1) : (C.bcy && ey == C.Ny - 1);
  long long nLo, nHi;
  if (DIR == 0) {
    nLo = ((ex == 0 ? C.Nx - 1 : ex - 1) + (long long)C.Nx * ey) * NPP + (NP - 1) + NP * j;
    nHi = ((ex == C.Nx - 1 ? 0 : ex + 1) + (long long)C.Nx * ey) * NPP + NP * j;
  } else {
    nLo = (ex + (long long)C.Nx * (ey == 0 ? C.Ny - 1 : ey - 1)) * NPP + j + NP * (NP - 1);
    nHi = (ex + (long long)C.Nx * (ey == C.Ny - 1 ? 0 : ey + 1)) * NPP + j;
  }
  if (wallLo) nLo = g0;
  if (wallHi) nHi = g0 + 4 * SN;
#ifdef SGNB_CHECKED
  if (!SGNB_INB(nLo, Nd) || !SGNB_INB(nHi, Nd)) return;
#endif
  const double sgnLo = wallLo ? -1.0 : 1.0, sgnHi = wallHi ? -1.0 : 1.0;

  // ---- forward quantities ---------------------------------------------------------------
  double h[NP], hn[NP], hp[NP], ih[NP], un[NP];
#pragma unroll
  for (int k = 0; k < NP; ++k) {
    const long long g = g0 + SN * k;
    h[k] = state(0, g);
    hn[k] = state(N, g);
    hp[k] = state(4, g);
    ih[k] = fast_rcp(h[k]);
    un[k] = hn[k] * ih[k];
  }
  const double hL = state(0, nLo), hnL = sgnLo * state(N, nLo), hpL = state(4, nLo);
  const double hR = state(0, nHi), hnR = sgnHi * state(N, nHi), hpR = state(4, nHi);
  const double ihL = fast_rcp(hL), ihR = fast_rcp(hR), unL = hnL * ihL, unR = hnR * ihR;
  // root of the wave speed (0 where its argument is not positive: its derivative is dropped then)
  auto root = [&](double hh, double pp) {
    const double a = fma(gr, hh, pp) + c2;
    return a > 0.0 ? fast_sqrt(a) : 0.0;
  };
  const double cLs = root(hL, hpL * ihL), cLt = root(h[0], hp[0] * ih[0]);
  const double cRs = root(hR, hpR * ihR), cRt = root(h[4], hp[4] * ih[4]);
  const double wLs = fabs(unL) + cLs, wLt = fabs(un[0]) + cLt, wRs = fabs(unR) + cRs, wRt = fabs(un[4]) + cRt;
  const bool sideL = wLs >= wLt, sideR = !(wRt >= wRs);  // the neighbour's speed is the larger one
  const double lamL = 0.5 * fmax(wLs, wLt), lamR = 0.5 * fmax(wRs, wRt);

  // accumulators: own nodes, and the neighbours' traces (left L, right R)
  double hb[NP], hnb[NP], hpb[NP], unb[NP], Hb[NP];
  double hLb = 0.0, hnLb = 0.0, hpLb = 0.0, unLb = 0.0, lamLb = 0.0;
  double hRb = 0.0, hnRb = 0.0, hpRb = 0.0, unRb = 0.0, lamRb = 0.0;

  double R[NP], Fb[NP], jL, jR;
  // cotangents of field v's fluxes (nodes; low and high jump) from its cotangent R
  auto flux_cot = [&](int v) {
    jL = 0.0;
    jR = 0.0;
#pragma unroll
    for (int m = 0; m < NP; ++m) {
      R[m] = cot(v, m);
      jL = fma(T.gLp[m], R[m], jL);
      jR = fma(T.gRp[m], R[m], jR);
    }
    jL *= -iJ;
    jR *= -iJ;
#pragma unroll
    for (int k = 0; k < NP; ++k) {
      double s = 0.0;
#pragma unroll
      for (int m = 0; m < NP; ++m) s = fma(T.D[m * NP + k], R[m], s);
      Fb[k] = -iJ * s;
    }
  };
  // the own face fluxes leave with -1/2 of the jump; the wave speed's cotangent
  auto own_faces = [&]() {
    Fb[0] = fma(-0.5, jL, Fb[0]);
    Fb[4] = fma(-0.5, jR, Fb[4]);
  };
  auto lam_cot = [&](double sL, double tL, double sR, double tR) {
    lamLb = fma(0.5 * jL, sL - tL, lamLb);
    lamRb = fma(-0.5 * jR, sR - tR, lamRb);
  };

  // ---- hp: flux u_n hp + c^2 h u_n; R[hp] += c^2 u_n dh ------------------------------------
  flux_cot(4);
  {
    double gh[NP];
    const double jhL = 0.5 * (hL - h[0]), jhR = 0.5 * (hR - h[4]);
    double bL = 0.0, bR = 0.0;
#pragma unroll
    for (int m = 0; m < NP; ++m) {
      double s = fma(jhL, T.gLp[m], jhR * T.gRp[m]);
#pragma unroll
      for (int k = 0; k < NP; ++k) s = fma(T.D[m * NP + k], h[k], s);
      const double r = c2 * iJ * R[m];
      unb[m] = s * r;
      gh[m] = un[m] * r;
      bL = fma(T.gLp[m], gh[m], bL);
      bR = fma(T.gRp[m], gh[m], bR);
    }
#pragma unroll
    for (int k = 0; k < NP; ++k) {
      double s = 0.0;
#pragma unroll
      for (int m = 0; m < NP; ++m) s = fma(T.D[m * NP + k], gh[m], s);
      hb[k] = s;
    }
    hLb = 0.5 * bL;
    hb[0] -= 0.5 * bL;
    hRb = 0.5 * bR;
    hb[4] -= 0.5 * bR;
  }
  own_faces();
#pragma unroll
  for (int k = 0; k < NP; ++k) {
    hpb[k] = un[k] * Fb[k];
    unb[k] = fma(hp[k], Fb[k], unb[k]);
    hnb[k] = c2 * Fb[k];
  }
  hpLb = fma(0.5 * jL, unL, lamL * jL);
  unLb = 0.5 * jL * hpL;
  hnLb = 0.5 * c2 * jL;
  hpb[0] -= lamL * jL;
  hpRb = fma(0.5 * jR, unR, -lamR * jR);
  unRb = 0.5 * jR * hpR;
  hnRb = 0.5 * c2 * jR;
  hpb[4] += lamR * jR;
  lam_cot(hpL, hp[0], hpR, hp[4]);

  // ---- mass: h u_n -----------------------------------------------------------------------
  flux_cot(0);
  own_faces();
#pragma unroll
  for (int k = 0; k < NP; ++k) hnb[k] += Fb[k];
  hnLb = fma(0.5, jL, hnLb);
  hnRb = fma(0.5, jR, hnRb);
  hLb = fma(lamL, jL, hLb);
  hb[0] -= lamL * jL;
  hRb = fma(-lamR, jR, hRb);
  hb[4] += lamR * jR;
  lam_cot(hL, h[0], hR, h[4]);

  // ---- normal discharge: u_n (h u_n) + g/2 (h^2 - H^2) + hp ---------------------------------
  flux_cot(N);
#pragma unroll
  for (int k = 0; k < NP; ++k) Hb[k] = -gr * C.Hnod[g0 + SN * k] * Fb[k];
  own_faces();
#pragma unroll
  for (int k = 0; k < NP; ++k) {
    unb[k] = fma(hn[k], Fb[k], unb[k]);
    hnb[k] = fma(un[k], Fb[k], hnb[k]);
    hb[k] = fma(gr * h[k], Fb[k], hb[k]);
    hpb[k] += Fb[k];
  }
  unLb = fma(0.5 * jL, hnL, unLb);
  hnLb = fma(0.5 * jL, unL, fma(lamL, jL, hnLb));
  hLb = fma(0.5 * jL, gr * hL, hLb);
  hpLb = fma(0.5, jL, hpLb);
  hnb[0] -= lamL * jL;
  unRb = fma(0.5 * jR, hnR, unRb);
  hnRb = fma(0.5 * jR, unR, fma(-lamR, jR, hnRb));
  hRb = fma(0.5 * jR, gr * hR, hRb);
  hpRb = fma(0.5, jR, hpRb);
  hnb[4] += lamR * jR;
  lam_cot(hnL, hn[0], hnR, hn[4]);
  // sources (x pass only; pointwise, sgn_flux2d.h:122-134): (g (h - H) + gamma p) dH/dx and the
  // u dH/dx part of -2 c^2 (w + u dH/dx + v dH/dy)
  if constexpr (DIR == 0) {
#pragma unroll
    for (int k = 0; k < NP; ++k) {
      const long long g = g0 + SN * k;
      const double Hx = C.Hx[g], r4 = C.m2c2 * cot(4, k), p = hp[k] * ih[k];
      const double bath = fma(gr, h[k] - C.Hnod[g], C.gamma * p), s = Hx * R[k];
      hb[k] = fma(gr, s, hb[k]);
      Hb[k] = fma(-gr, s, Hb[k]);
      hpb[k] = fma(C.gamma * s, ih[k], hpb[k]);
      hb[k] = fma(-C.gamma * s * p, ih[k], hb[k]);
      unb[k] = fma(Hx, r4, unb[k]);
      A.Hxb[g] = fma(bath, R[k], un[k] * r4);
    }
  }

  double* const oL = A.Sn[DIR][0] + idx * NV;
  double* const oR = A.Sn[DIR][1] + idx * NV;
  // ---- hw and the tangential discharge: u_n U_v ---------------------------------------------
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const int v = q == 0 ? 3 : TG;
    double w[NP], wb[NP];
#pragma unroll
    for (int k = 0; k < NP; ++k) w[k] = state(v, g0 + SN * k);
    const double wL = state(v, nLo), wR = state(v, nHi);
    flux_cot(v);
    own_faces();
#pragma unroll
    for (int k = 0; k < NP; ++k) {
      wb[k] = un[k] * Fb[k];
      unb[k] = fma(w[k], Fb[k], unb[k]);
    }
    wb[0] -= lamL * jL;
    wb[4] += lamR * jR;
    const double wLb = fma(0.5 * jL, unL, lamL * jL), wRb = fma(0.5 * jR, unR, -lamR * jR);
    unLb = fma(0.5 * jL, wL, unLb);
    unRb = fma(0.5 * jR, wR, unRb);
    lam_cot(wL, w[0], wR, w[4]);
    if constexpr (DIR == 0) {
#pragma unroll
      for (int k = 0; k < NP; ++k) {
        const long long g = g0 + SN * k;
        const double r4 = C.m2c2 * cot(4, k), p = hp[k] * ih[k], x = w[k] * ih[k];
        if (q == 0) {
          // gamma p in hw, w in hp
          wb[k] = fma(r4, ih[k], wb[k]);
          const double pb = C.gamma * R[k];
          hpb[k] = fma(pb, ih[k], hpb[k]);
          hb[k] = fma(-ih[k], fma(r4, x, pb * p), hb[k]);
        } else {
          // (g (h - H) + gamma p) dH/dy, v dH/dy in hp, friction
          const double Hy = C.Hy[g], s = Hy * R[k];
          const double bath = fma(gr, h[k] - C.Hnod[g], C.gamma * p);
          A.Hyb[g] = fma(bath, R[k], x * r4);
          double vb = Hy * r4;
          hb[k] = fma(gr, s, hb[k]);
          Hb[k] = fma(-gr, s, Hb[k]);
          if (C.manning) {
            // (-cf u, -cf v), cf = n^2 g |vel| h^(-1/3)
            const double r1 = cot(1, k), vm = sqrt(un[k] * un[k] + x * x);
            const double kc = C.n2g / cbrt(h[k]), cf = kc * vm, ruv = r1 * un[k] + R[k] * x;
            unb[k] -= r1 * cf;
            vb -= R[k] * cf;
            if (vm > 0.0) {
              unb[k] -= kc * ruv * un[k] / vm;
              vb -= kc * ruv * x / vm;
            }
            hb[k] += ruv * cf / (3.0 * h[k]);  // d/dh of h^(-1/3)
          }
          const double pb = C.gamma * s;
          hpb[k] = fma(pb, ih[k], hpb[k]);
          wb[k] = fma(vb, ih[k], wb[k]);
          hb[k] = fma(-ih[k], fma(vb, x, pb * p), hb[k]);
        }
      }
    }
    // mirror ghosts fold back onto the own trace
    if (wallLo) wb[0] += wLb; else oL[v] = wLb;
    if (wallHi) wb[4] += wRb; else oR[v] = wRb;
#pragma unroll
    for (int k = 0; k < NP; ++k) A.Ub[DIR][v * Nd + g0 + SN * k] = wb[k];
  }

  // ---- wave speed |u_n| + sqrt(g h + p + c^2) of the side that has the larger one; |x|' is
  // sign(x), 0 at 0 (as the central difference) ------------------------------------------------
  auto speed_back = [&](double lb, double cc, double hp_, double ih_, double un_, double& hb_, double& hpb_,
                        double& unb_) {
    unb_ = fma(sgn0(un_), lb, unb_);
    const double ab = cc > 0.0 ? 0.5 * lb * fast_rcp(cc) : 0.0;
    hpb_ = fma(ab, ih_, hpb_);
    hb_ = fma(ab, fma(-hp_ * ih_, ih_, gr), hb_);
  };
  if (sideL) speed_back(lamLb, cLs, hpL, ihL, unL, hLb, hpLb, unLb);
  else speed_back(lamLb, cLt, hp[0], ih[0], un[0], hb[0], hpb[0], unb[0]);
  if (sideR) speed_back(lamRb, cRs, hpR, ihR, unR, hRb, hpRb, unRb);
  else speed_back(lamRb, cRt, hp[4], ih[4], un[4], hb[4], hpb[4], unb[4]);

  // ---- u_n = h u_n / h; results -----------------------------------------------------------
  hnLb = fma(unLb, ihL, hnLb);
  hLb = fma(-unLb * unL, ihL, hLb);
  hnRb = fma(unRb, ihR, hnRb);
  hRb = fma(-unRb * unR, ihR, hRb);
#pragma unroll
  for (int k = 0; k < NP; ++k) {
    hnb[k] = fma(unb[k], ih[k], hnb[k]);
    hb[k] = fma(-unb[k] * un[k], ih[k], hb[k]);
  }
  if (wallLo) {
    hb[0] += hLb;
    hnb[0] -= hnLb;
    hpb[0] += hpLb;
  } else {
    oL[0] = hLb;
    oL[N] = hnLb;
    oL[4] = hpLb;
  }
  if (wallHi) {
    hb[4] += hRb;
    hnb[4] -= hnRb;
    hpb[4] += hpRb;
  } else {
    oR[0] = hRb;
    oR[N] = hnRb;
    oR[4] = hpRb;
  }
#pragma unroll
  for (int k = 0; k < NP; ++k) {
    const long long g = g0 + SN * k;
    A.Ub[DIR][g] = hb[k];
    A.Ub[DIR][N * Nd + g] = hnb[k];
    A.Ub[DIR][4 * Nd + g] = hpb[k];
    A.Hb[DIR][g] = Hb[k];
  }
}

// Both directions' lines in one launch (blockIdx.y: direction).
__global__ void __launch_bounds__(128, 3) k_vjp_lines(const RhsConsts C, const FrTablesDev T, const VjpArgs A) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)C.Nx * C.Ny * NP) return;
  if (blockIdx.y == 0) vjp_line<0>(C, T, A, idx);
  else vjp_line<1>(C, T, A, idx);
}

// One thread per node: the node's cotangent from both directions and from the
// neighbours' faces, the RK-stage combination, and the statics accumulators.
__global__ void __launch_bounds__(256) k_vjp_gather(const RhsConsts C, const VjpArgs A,
                                                    const GatherArgs G) {
  const long long Nd = C.Nd;
  const long long gnode = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gnode >= Nd) return;
  const long long e = gnode / NPP;
  const int loc = (int)(gnode - e * NPP);
  const int a = loc % NP, b = loc / NP;
  const int ex = (int)(e % C.Nx), ey = (int)(e / C.Nx);
  const long long eL = (long long)((ex - 1 + C.Nx) % C.Nx) + (long long)C.Nx * ey;
  const long long eR = (long long)((ex + 1) % C.Nx) + (long long)C.Nx * ey;
  const long long eB = (long long)ex + (long long)C.Nx * ((ey - 1 + C.Ny) % C.Ny);
  const long long eT = (long long)ex + (long long)C.Nx * ((ey + 1) % C.Ny);
  const bool wL = C.bcx && ex == 0, wR = C.bcx && ex == C.Nx - 1;
  const bool wB = C.bcy && ey == 0, wT = C.bcy && ey == C.Ny - 1;
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const long long g = v * Nd + gnode;
    double y = A.Ub[0][g] + A.Ub[1][g];
    // line index of a face entry: (element * 5 + line) * 5 + v
    [[maybe_unused]] const long long nl = (long long)C.Nx * C.Ny * NP * NV;
    if (a == 0 && !wL && SGNB_INB((eL * NP + b) * NV + v, nl)) y += A.Sn[0][1][(eL * NP + b) * NV + v];
    if (a == NP - 1 && !wR && SGNB_INB((eR * NP + b) * NV + v, nl)) y += A.Sn[0][0][(eR * NP + b) * NV + v];
    if (b == 0 && !wB && SGNB_INB((eB * NP + a) * NV + v, nl)) y += A.Sn[1][1][(eB * NP + a) * NV + v];
    if (b == NP - 1 && !wT && SGNB_INB((eT * NP + a) * NV + v, nl)) y += A.Sn[1][0][(eT * NP + a) * NV + v];
    if (G.ybar) G.ybar[g] = y;
    if (G.init) G.uacc[g] = (G.lam ? G.lam[g] : 0.0) + y;
    else G.uacc[g] += y;
  }
  G.Hacc[gnode] += A.Hb[0][gnode] + A.Hb[1][gnode];
  G.Hxacc[gnode] += A.Hxb[gnode];
  G.Hyacc[gnode] += A.Hyb[gnode];
}

// u_new = u + dt ((2/9 k1 + 1/3 k2) + 4/9 k3) with the end-point stage's rounding
// (src/solver/rk.cpp:106-108).
__global__ void k_rk_update(const double* __restrict__ u, const double* __restrict__ k1,
                            const double* __restrict__ k2, const double* __restrict__ k3,
                            const double* __restrict__ dts, long long step,
                            double* __restrict__ out, long long n) {
  const double dt = dts[step];
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const double part = __dadd_rn(__dmul_rn(2.0 / 9.0, k1[i]), __dmul_rn(1.0 / 3.0, k2[i]));
    out[i] = __dadd_rn(u[i], __dmul_rn(dt, __dadd_rn(part, __dmul_rn(4.0 / 9.0, k3[i]))));
  }
}

// eta at the gauges: eta[g] = h(node_g) - H(node_g)
__global__ void k_gauges(const double* __restrict__ U, const double* __restrict__ Hnod,
                         const long long* __restrict__ nodes, int ng, double* __restrict__ eta) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g < ng) eta[g] = U[nodes[g]] - Hnod[nodes[g]];  // nodes checked on the host
}

// lam[h](node_g) += etab[g]
__global__ void k_gauges_back(double* __restrict__ lam, const long long* __restrict__ nodes,
                              int ng, const double* __restrict__ etab) {
  // gauges may share a node: one thread adds all of them, in order
  if (blockIdx.x == 0 && threadIdx.x == 0)
    for (int g = 0; g < ng; ++g) lam[nodes[g]] += etab[g];
}

}  // namespace

// The checked build's out-of-range count of the adjoint kernels (reset: then zero it);
// cudaErrorNotSupported in the normal build.
cudaError_t read_oob_adjoint(unsigned long long* out, bool reset) {
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

cudaError_t launch_vjp_rhs(const RhsConsts& C, const FrTablesDev& T, const VjpArgs& A,
                           const GatherArgs& G, cudaStream_t s) {
  const long long lines = (long long)C.Nx * C.Ny * NP;
  const unsigned nb = (unsigned)((lines + 127) / 128);
  k_vjp_lines<<<dim3(nb, 2), 128, 0, s>>>(C, T, A);
  const unsigned ng = (unsigned)((C.Nd + 255) / 256);
  k_vjp_gather<<<ng, 256, 0, s>>>(C, A, G);
  return cudaGetLastError();
}

cudaError_t launch_rk_update(const double* u, const double* k1, const double* k2,
                             const double* k3, const double* dts, long long step, double* out,
                             long long n, cudaStream_t s) {
  k_rk_update<<<4 * 148, 256, 0, s>>>(u, k1, k2, k3, dts, step, out, n);
  return cudaGetLastError();
}

cudaError_t launch_gauges(const double* U, const double* Hnod, const long long* nodes, int ng,
                          double* eta, cudaStream_t s) {
  k_gauges<<<(ng + 127) / 128, 128, 0, s>>>(U, Hnod, nodes, ng, eta);
  return cudaGetLastError();
}

cudaError_t launch_gauges_back(double* lam, const long long* nodes, int ng, const double* etab,
                               cudaStream_t s) {
  k_gauges_back<<<1, 32, 0, s>>>(lam, nodes, ng, etab);
  return cudaGetLastError();
}

}  // namespace dev
}  // namespace sgnb
