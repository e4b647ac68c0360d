// sgnb_cells.cu -- depth statics of the bilinear interpolant of element means, and its
// transpose, on the device (the adjoint's parameterisation of the bathymetry). Built with
// -fmad=false: the statics have the bits of the host set-up (sgnb_setup.cpp), whose operation
// order these kernels repeat.
//
// Per gradient evaluation the host versions took about 60 ms on 256 x 128 elements (evaluation,
// 26 MB of pageable uploads and as much back, a serial scatter); these kernels take tens of
// microseconds, and only the means, eta0 and the two gradients cross the bus.
#include "sgnb_checked.cuh"
#include "sgnb_device.h"

namespace sgnb {
namespace dev {

namespace {
constexpr int NP = 5, NPP = 25;

// p[i] of n values (the checked build: 0 out of range).
__device__ __forceinline__ double at(const double* p, [[maybe_unused]] long long i, [[maybe_unused]] long long n) {
  return SGNB_INB(i, n) ? p[i] : 0.0;
}
__device__ __forceinline__ void put(double* p, [[maybe_unused]] long long i, [[maybe_unused]] long long n, double v) {
  if (SGNB_INB(i, n)) p[i] = v;
}

// The four cells and the position (tx, ty) between their centres at (x, y): the index
// arithmetic of the host's interpolant.
struct CellAt {
  int i0, i1, j0, j1;
  double tx, ty;
};
__device__ __forceinline__ CellAt cell_at(const CellGrid& g, double x, double y) {
  CellAt c;
  const double cx = g.Lx / g.Nx, cy = g.Ly / g.Ny;
  const double sx = x / cx - 0.5, sy = y / cy - 0.5;
  const double fx0 = floor(sx), fy0 = floor(sy);
  c.tx = sx - fx0;
  c.ty = sy - fy0;
  c.i0 = (int)fx0;
  c.j0 = (int)fy0;
  c.i1 = c.i0 + 1;
  c.j1 = c.j0 + 1;
  c.i0 = ((c.i0 % g.Nx) + g.Nx) % g.Nx;
  c.i1 = ((c.i1 % g.Nx) + g.Nx) % g.Nx;
  c.j0 = ((c.j0 % g.Ny) + g.Ny) % g.Ny;
  c.j1 = ((c.j1 % g.Ny) + g.Ny) % g.Ny;
  return c;
}
__device__ __forceinline__ double depth_at(const CellGrid& g, const double* m, double x, double y) {
  const CellAt c = cell_at(g, x, y);
  const int n = g.Nx * g.Ny;
  const double v00 = at(m, c.i0 + g.Nx * c.j0, n), v10 = at(m, c.i1 + g.Nx * c.j0, n);
  const double v01 = at(m, c.i0 + g.Nx * c.j1, n), v11 = at(m, c.i1 + g.Nx * c.j1, n);
  const double lo = v00 + c.tx * (v10 - v00);
  const double hi = v01 + c.tx * (v11 - v01);
  return lo + c.ty * (hi - lo);
}
__device__ __forceinline__ double node_x(const CellGrid& g, int ex, int a) {
  return ex * g.hx + 0.5 * g.hx * (g.nodes[a] + 1.0);
}
__device__ __forceinline__ double node_y(const CellGrid& g, int ey, int b) {
  return ey * g.hy + 0.5 * g.hy * (g.nodes[b] + 1.0);
}

// Nodal depths, and the state (H + eta0, 0, 0, 0, 0); one thread per node.
__global__ void __launch_bounds__(256) k_cells_depth(const CellGrid g, const double* __restrict__ means,
                                                     const double* __restrict__ eta0,
                                                     double* __restrict__ H, double* __restrict__ u0) {
  const long long Nd = 25LL * g.Nx * g.Ny;
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= Nd) return;
  const int e = (int)(i / NPP), n = (int)(i - (long long)e * NPP);
  const int ey = e / g.Nx, ex = e - ey * g.Nx, b = n / NP, a = n - NP * b;
  const double h = depth_at(g, means, node_x(g, ex, a), node_y(g, ey, b));
  put(H, i, Nd, h);
  put(u0, i, 5 * Nd, h + at(eta0, i, Nd));
#pragma unroll
  for (int v = 1; v < 5; ++v) put(u0, v * Nd + i, 5 * Nd, 0.0);
}

// Nodal depth gradients: the GLL derivative along each line over J; one thread per node.
__global__ void __launch_bounds__(256) k_cells_gradient(const CellGrid g, const double* __restrict__ H,
                                                        double* __restrict__ Hx, double* __restrict__ Hy) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long Nd = 25LL * g.Nx * g.Ny;
  if (i >= Nd) return;
  const long long e = i / NPP;
  const int n = (int)(i - e * NPP), b = n / NP, a = n - NP * b;
  double sx = 0.0, sy = 0.0;
#pragma unroll
  for (int k = 0; k < NP; ++k) {
    sx += g.D[a * NP + k] * at(H, e * NPP + k + NP * b, Nd);
    sy += g.D[b * NP + k] * at(H, e * NPP + a + NP * k, Nd);
  }
  put(Hx, i, Nd, sx / (0.5 * g.hx));
  put(Hy, i, Nd, sy / (0.5 * g.hy));
}

// Face depths: left and bottom edges of every element (5 Nx Ny each), then the right and top
// domain edges (5 Ny, 5 Nx); one thread per edge node.
__global__ void __launch_bounds__(256) k_cells_faces(const CellGrid g, const double* __restrict__ m,
                                                     double* __restrict__ HfX, double* __restrict__ HfY,
                                                     double* __restrict__ HfXEnd, double* __restrict__ HfYEnd) {
  const long long nf = 5LL * g.Nx * g.Ny;
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < nf) {
    const int e = (int)(i / NP), s = (int)(i - (long long)e * NP), ey = e / g.Nx, ex = e - ey * g.Nx;
    put(HfX, i, nf, depth_at(g, m, ex * g.hx, node_y(g, ey, s)));
    put(HfY, i, nf, depth_at(g, m, node_x(g, ex, s), ey * g.hy));
    return;
  }
  i -= nf;
  if (i < NP * g.Ny) {
    put(HfXEnd, i, NP * g.Ny, depth_at(g, m, g.Nx * g.hx, node_y(g, (int)(i / NP), (int)(i % NP))));
  } else if ((i -= NP * g.Ny) < NP * g.Nx) {
    put(HfYEnd, i, NP * g.Nx, depth_at(g, m, node_x(g, (int)(i / NP), (int)(i % NP)), g.Ny * g.hy));
  }
}

// Cotangent of the nodal depths with everything that reaches them: their own, the initial
// depth's (h0 = H + eta0) and, through the gradients' transpose, those of dH/dx and dH/dy. One
// thread per node.
__global__ void __launch_bounds__(256) k_cells_back_nodes(const CellGrid g, const double* __restrict__ Hb,
                                                          const double* __restrict__ lam,
                                                          const double* __restrict__ Hxb,
                                                          const double* __restrict__ Hyb,
                                                          double* __restrict__ out) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long Nd = 25LL * g.Nx * g.Ny;
  if (i >= Nd) return;
  const long long e = i / NPP;
  const int n = (int)(i - e * NPP), b = n / NP, a = n - NP * b;
  double sx = 0.0, sy = 0.0;
#pragma unroll
  for (int k = 0; k < NP; ++k) {
    sx += g.D[k * NP + a] * at(Hxb, e * NPP + k + NP * b, Nd);
    sy += g.D[k * NP + b] * at(Hyb, e * NPP + a + NP * k, Nd);
  }
  put(out, i, Nd, (at(Hb, i, Nd) + at(lam, i, Nd)) + (sx / (0.5 * g.hx) + sy / (0.5 * g.hy)));
}

// eta = h - H at the gauges: the cotangents of a gauge's records leave its node's depth, in
// step order. One thread per gauge; the first of several gauges at one node takes all of them.
__global__ void __launch_bounds__(64) k_cells_back_gauges(const long long Nd, const long long* __restrict__ nodes,
                                                          int ng, long long nsteps,
                                                          const double* __restrict__ etab,
                                                          double* __restrict__ Hb) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= ng) return;
  const long long node = nodes[q];
  for (int p = 0; p < q; ++p)
    if (nodes[p] == node) return;
  int last = q;
  for (int p = q + 1; p < ng; ++p)
    if (nodes[p] == node) last = p;
  if (!SGNB_INB(node, Nd)) return;
  double h = Hb[node];
  for (long long n = 0; n < nsteps; ++n)
    for (int p = q; p <= last; ++p)
      if (nodes[p] == node) h -= at(etab, n * ng + p, nsteps * ng);
  Hb[node] = h;
}

// Gradient of one mean: the weights of its cell at every node around it, in a fixed order. A node
// of element (ex, ey) touches the cells of the elements beside it only, so 3 x 3 elements hold
// every contribution (2 of a direction where the mesh has only two elements along it). One warp
// per mean, lanes over the nodes.
__global__ void __launch_bounds__(256) k_cells_back(const CellGrid g, const double* __restrict__ Hb,
                                                    double* __restrict__ grad) {
  const int cell = (int)(((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (cell >= g.Nx * g.Ny) return;
  const int cj = cell / g.Nx, ci = cell - cj * g.Nx;
  double s = 0.0;
  auto add = [&](double x, double y, double v) {
    const CellAt c = cell_at(g, x, y);
    double w = 0.0;
    if (c.i0 == ci && c.j0 == cj) w += (1.0 - c.tx) * (1.0 - c.ty);
    if (c.i1 == ci && c.j0 == cj) w += c.tx * (1.0 - c.ty);
    if (c.i0 == ci && c.j1 == cj) w += (1.0 - c.tx) * c.ty;
    if (c.i1 == ci && c.j1 == cj) w += c.tx * c.ty;
    if (w != 0.0) s += w * v;
  };
  const int nx3 = g.Nx == 2 ? 2 : 3, ny3 = g.Ny == 2 ? 2 : 3;
  for (int dy = 0; dy < ny3; ++dy)
    for (int dx = 0; dx < nx3; ++dx) {
      const int ex = (ci + dx - 1 + g.Nx) % g.Nx, ey = (cj + dy - 1 + g.Ny) % g.Ny;
      const long long e = ex + (long long)g.Nx * ey;
      // lanes 0..24 the element's nodes (the face depths cancel in R: their cotangents are zero)
      if (lane < NPP) {
        const int b = lane / NP, a = lane - NP * b;
        add(node_x(g, ex, a), node_y(g, ey, b), at(Hb, e * NPP + lane, 25LL * g.Nx * g.Ny));
      }
    }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
  if (lane == 0) grad[cell] = s;
}

unsigned blocks_of(long long n) { return (unsigned)((n + 255) / 256); }
}  // namespace

// The checked build's out-of-range count of this translation unit's kernels (reset: then
// zero it); cudaErrorNotSupported in the normal build.
cudaError_t read_oob_cells(unsigned long long* out, bool reset) {
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

cudaError_t launch_cells_statics(const CellGrid& g, const double* means, const double* eta0, double* Hnod,
                                 double* Hx, double* Hy, double* HfX, double* HfY, double* HfXEnd,
                                 double* HfYEnd, double* u0, cudaStream_t s) {
  const long long Nd = 25LL * g.Nx * g.Ny, nf = 5LL * g.Nx * g.Ny + 5LL * (g.Nx + g.Ny);
  k_cells_depth<<<blocks_of(Nd), 256, 0, s>>>(g, means, eta0, Hnod, u0);
  k_cells_gradient<<<blocks_of(Nd), 256, 0, s>>>(g, Hnod, Hx, Hy);
  k_cells_faces<<<blocks_of(nf), 256, 0, s>>>(g, means, HfX, HfY, HfXEnd, HfYEnd);
  return cudaGetLastError();
}

cudaError_t launch_cells_back(const CellGrid& g, const GatherArgs& G, const double* lam,
                              const long long* gauges, int ng, long long nsteps, const double* etab,
                              double* Hb, double* grad, cudaStream_t s) {
  const long long Nd = 25LL * g.Nx * g.Ny;
  k_cells_back_nodes<<<blocks_of(Nd), 256, 0, s>>>(g, G.Hacc, lam, G.Hxacc, G.Hyacc, Hb);
  if (ng > 0) k_cells_back_gauges<<<(unsigned)((ng + 63) / 64), 64, 0, s>>>(Nd, gauges, ng, nsteps, etab, Hb);
  k_cells_back<<<blocks_of(32LL * g.Nx * g.Ny), 256, 0, s>>>(g, Hb, grad);
  return cudaGetLastError();
}

}  // namespace dev
}  // namespace sgnb
