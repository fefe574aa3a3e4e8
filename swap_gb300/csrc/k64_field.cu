// k64_field.cu -- the FP64 field operators of the drop-in (boundary.f,
// grid_interp.f, gutsf.f), fused between the points where a stencil needs its
// neighbours' results.
//
// Compiled with --fmad=false: every multiply and add is rounded in the
// Fortran's order, so each entry's outputs equal the FP64 CPU restatement bit
// for bit.
//
// What bounds them: GB300 retires two FP64 operations per SM and clock (a warp
// instruction takes 16 clocks), so on grids of 10^5 nodes and more the
// operators are bound by the FP64 pipe, not by HBM, and on small grids by the
// number of launches.  Hence
//  * one kernel per stencil dependency and no more: the periodic fills
//    (boundary.f:9-52) are not passes of their own.  A kernel reads a ghost
//    node at its interior image (wrapped index) and stores an output together
//    with its ghost images.  A subcycle takes 9 launches instead of 44;
//  * no value is computed twice: the neighbours' curl B, cross product and E
//    are read back from memory rather than recomputed, because 8 bytes of HBM
//    traffic cost a tenth of one FP64 operation;
//  * divisions by a grid spacing are exact quotients from a stored reciprocal
//    (quotient(), k64_dev.cuh): one or three operations instead of about nine;
//  * 32-bit index arithmetic (a 64-bit division by the row length is a long
//    emulated sequence).
// 128x64x64 nodes, one subcycle through the three entries curlB, predict_B,
// correct_B: 1.04 -> 0.72 ms, of which on the
// device 0.74 -> 0.36 ms (18x11x14: 0.355 -> 0.211 ms).
#include "k64.cuh"
#include "grid_loop.cuh"
#include "launch_next.cuh"
#include "k64_dev.cuh"

namespace swapk {
namespace {

constexpr int TPB = 128;  // most threads of a block

// Threads per block: a warp instruction of the FP64 pipe holds its SM for 16
// clocks, so small grids are spread over all 152 SMs a warp at a time (2772
// nodes in 11 blocks of 256 took 8.5 us for curl B, in 87 of 32 6.9),
// and middling ones in blocks small enough to even out the SMs' shares.
inline unsigned threads_for(long long n) { return n <= 152 * 64 ? 32u : (n <= 152 * 64 * 64 ? 64u : 128u); }
inline unsigned nblocks(long long n) {
  const long long t = threads_for(n), b = (n + t - 1) / t;
  return (unsigned)(b < 1 ? 1 : b);
}

// Interior thread t -> node (i,j,k) and its offset.
struct Node {
  int i, j, k;
  unsigned o;
};
__device__ __forceinline__ Node node_of(const Geo& g, unsigned t) {
  const unsigned ix = (unsigned)g.nx - 2, iy = (unsigned)g.ny - 2;
  const unsigned r = t / ix, r2 = r / iy;
  Node n;
  n.i = (int)(t - r * ix) + 2;
  n.j = (int)(r - r2 * iy) + 2;
  n.k = (int)r2 + 2;
  n.o = (unsigned)(n.i - 1) + (unsigned)g.nx * ((unsigned)(n.j - 1) + (unsigned)g.ny * (unsigned)(n.k - 1));
  return n;
}

// Offsets from an interior node to its neighbours, at the periodic image
// where the neighbour is a ghost (boundary.f:21-22).
struct Nbr {
  int xm, xp, ym, yp, zm, zp;
};
__device__ __forceinline__ Nbr nbr_of(const Geo& g, const Node& n) {
  const int sy = g.nx, sz = g.nx * g.ny;
  Nbr b;
  b.xm = n.i == 2 ? g.nx - 3 : -1;
  b.xp = n.i == g.nx - 1 ? -(g.nx - 3) : 1;
  b.ym = n.j == 2 ? (g.ny - 3) * sy : -sy;
  b.yp = n.j == g.ny - 1 ? -(g.ny - 3) * sy : sy;
  b.zm = n.k == 2 ? (g.nz - 3) * sz : -sz;
  b.zp = n.k == g.nz - 1 ? -(g.nz - 3) * sz : sz;
  return b;
}

// Whether the node has a ghost image, and the store of a value at every ghost
// node whose image it is (the periodic fill, boundary.f:9-52).
__device__ __forceinline__ bool on_edge(const Geo& g, const Node& n) {
  return n.i == 2 || n.j == 2 || n.k == 2 || n.i == g.nx - 1 || n.j == g.ny - 1 || n.k == g.nz - 1;
}
// ncomp components (v0, v1, v2) of f; one image per axis and side, both sides
// on an axis of a single cell.
__device__ __noinline__ void store_ghosts(int nx, int ny, int nz, long long C, int ncomp, double* f, int i, int j,
                                          int k, double v0, double v1, double v2) {
  const int sy = nx, sz = nx * ny;
  f += (i - 1) + (long long)nx * ((j - 1) + (long long)ny * (k - 1));
  // offset to the image beyond the far end (node 2) and the near end (node n-1)
  const int x[3] = {0, i == 2 ? nx - 2 : 0, i == nx - 1 ? 2 - nx : 0};
  const int y[3] = {0, j == 2 ? (ny - 2) * sy : 0, j == ny - 1 ? (2 - ny) * sy : 0};
  const int z[3] = {0, k == 2 ? (nz - 2) * sz : 0, k == nz - 1 ? (2 - nz) * sz : 0};
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    if (c && !z[c]) continue;
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      if (b && !y[b]) continue;
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        if ((a && !x[a]) || a + b + c == 0) continue;
        double* t = f + (x[a] + y[b] + z[c]);
        t[0] = v0;
        if (ncomp == 3) {
          t[C] = v1;
          t[2 * C] = v2;
        }
      }
    }
  }
}
__device__ __forceinline__ void ghosts3(const Geo& g, const Node& n, double* f, double v0, double v1, double v2) {
  if (on_edge(g, n)) store_ghosts(g.nx, g.ny, g.nz, g.C, 3, f, n.i, n.j, n.k, v0, v1, v2);
}

// The ghost images of an array that the caller sees filled (its periodic()
// in the reference) and this operator does not otherwise write.
__device__ __forceinline__ void fill3(const Geo& g, const Node& n, double* f) {
  if (on_edge(g, n))
    store_ghosts(g.nx, g.ny, g.nz, g.C, 3, f, n.i, n.j, n.k, f[n.o], f[n.o + g.C], f[n.o + 2 * g.C]);
}

// ---- one node of each operator ------------------------------------------------

// curlB (gutsf.f:202-239); the face densities' np is read as it stands (the
// reference does not fill its ghosts here).
// den (may be null): the divisors and their reciprocals (face_density).
__device__ __forceinline__ void face_densities(const Geo& g, const double* np, double alpha, unsigned o,
                                               double (&f)[3]) {
  const double n0 = np[o];
  f[0] = 0.5 * (n0 + np[o + 1]) * alpha;
  f[1] = 0.5 * (n0 + np[o + g.nx]) * alpha;
  f[2] = 0.5 * (n0 + np[o + g.nx * g.ny]) * alpha;
}
template <int SP>
__device__ __forceinline__ void curlB_node(const Geo& g, const Node& n, const Nbr& d, const double* b,
                                           const double* np, const double* den, double alpha, double* aj) {
  const long long C = g.C;
  const unsigned o = n.o;
  const double *B1 = b, *B2 = b + C, *B3 = b + 2 * C;
  const double dx = g.dxc[n.i], dy = g.dyc[n.j], dz = g.dzc[n.k];
  const double rx = g.rdxc[n.i], ry = g.rdyc[n.j], rz = g.rdzc[n.k];
  const double b1 = B1[o], b2 = B2[o], b3 = B3[o];
  const double c1 = quotient<SP>(b3 - B3[o + d.ym], dy, ry) + quotient<SP>(B2[o + d.zm] - b2, dz, rz);
  const double c2 = quotient<SP>(b1 - B1[o + d.zm], dz, rz) + quotient<SP>(B3[o + d.xm] - b3, dx, rx);
  const double c3 = quotient<SP>(b2 - B2[o + d.xm], dx, rx) + quotient<SP>(B1[o + d.ym] - b1, dy, ry);
  if (den) {
    const double a1 = quotient<SPACING_ANY>(c1, den[o], den[o + 3 * C]);
    const double a2 = quotient<SPACING_ANY>(c2, den[o + C], den[o + 4 * C]);
    const double a3 = quotient<SPACING_ANY>(c3, den[o + 2 * C], den[o + 5 * C]);
    aj[o] = a1;
    aj[o + C] = a2;
    aj[o + 2 * C] = a3;
  } else {
    double f[3];
    face_densities(g, np, alpha, o, f);
    aj[o] = c1 / f[0];
    aj[o + C] = c2 / f[1];
    aj[o + 2 * C] = c3 / f[2];
  }
}

// edge_to_center (grid_interp.f:22-57).
__device__ __forceinline__ void e2c_node(const Geo& g, const Node& n, const Nbr& d, const double* bt,
                                         double out[3]) {
  const long long C = g.C;
  const unsigned o = n.o;
  const double xr = g.xr[n.i], yr = g.yr[n.j], zr = g.zr[n.k];
  double a, b1, b2;
  const double* b = bt;  // component 1: y then z
  a = b[o + d.ym];
  b2 = a + yr * (b[o] - a);
  a = b[o + d.ym + d.zm];
  b1 = a + yr * (b[o + d.zm] - a);
  out[0] = b1 + zr * (b2 - b1);
  b = bt + C;  // component 2: x then z
  a = b[o + d.xm];
  b2 = a + xr * (b[o] - a);
  a = b[o + d.xm + d.zm];
  b1 = a + xr * (b[o + d.zm] - a);
  out[1] = b1 + zr * (b2 - b1);
  b = bt + 2 * C;  // component 3: y then x
  a = b[o + d.ym];
  b2 = a + yr * (b[o] - a);
  a = b[o + d.xm + d.ym];
  b1 = a + yr * (b[o + d.xm] - a);
  out[2] = b1 + xr * (b2 - b1);
}

// face_to_center (grid_interp.f:150-171) from a value and its lower neighbour.
__device__ __forceinline__ double f2c(double r, double v, double vm) { return r * (v - vm) + vm; }

// face_to_center(aj - up), B at the centres and the cross product of crossf2
// (gutsf.f:1059-1075, 65-76).  Predictor (CORR false): b is the edge field,
// taken to the centre here.  Corrector: b holds edge_to_center of it, taken
// to the faces (grid_interp.f:123-125) and back to the centres
// (gutsf.f:1268-1269).
template <bool CORR>
__device__ __forceinline__ void ct_node(const Geo& g, const Node& n, const Nbr& d, const double* aj,
                                        const double* up, const double* b,
                                        double* ct) {
  const long long C = g.C;
  const unsigned o = n.o;
  const double xr = g.xr[n.i], yr = g.yr[n.j], zr = g.zr[n.k];
  const double ax = f2c(xr, aj[o] - up[o], aj[o + d.xm] - up[o + d.xm]);
  const double ay = f2c(yr, aj[o + C] - up[o + C], aj[o + C + d.ym] - up[o + C + d.ym]);
  const double az = f2c(zr, aj[o + 2 * C] - up[o + 2 * C], aj[o + 2 * C + d.zm] - up[o + 2 * C + d.zm]);
  double B[3];
  if (!CORR) {
    e2c_node(g, n, d, b, B);
  } else {
    const double x0 = b[o], y0 = b[o + C], z0 = b[o + 2 * C];
    B[0] = f2c(xr, 0.5 * (x0 + b[o + d.xp]), 0.5 * (b[o + d.xm] + x0));
    B[1] = f2c(yr, 0.5 * (y0 + b[o + C + d.yp]), 0.5 * (b[o + C + d.ym] + y0));
    B[2] = f2c(zr, 0.5 * (z0 + b[o + 2 * C + d.zp]), 0.5 * (b[o + 2 * C + d.zm] + z0));
  }
  ct[o] = ay * B[2] - az * B[1];
  ct[o + C] = az * B[0] - ax * B[2];
  ct[o + 2 * C] = ax * B[1] - ay * B[0];
}

// Pressure-gradient extension at the face of component m (see the CPU
// restatement's grad_pe_at); np's ghosts as they stand.
__device__ __forceinline__ double grad_pe_at(const Geo& g, const double* np, double gp, const Node& n, int m) {
  const unsigned o = n.o;
  const unsigned op = o + (m == 0 ? 1u : (m == 1 ? (unsigned)g.nx : (unsigned)(g.nx * g.ny)));
  const double dg = m == 0 ? g.dxg[n.i] : (m == 1 ? g.dyg[n.j] : g.dzg[n.k]);
  const double nf = 0.5 * (np[o] + np[op]);
  return gp * ((np[op] - np[o]) / dg) / nf;
}

// crossf2's face average (gutsf.f:94-96) and E = c + nu*aj (gutsf.f:1082,
// 1282), with E's ghost images.
__device__ __forceinline__ void e_node(const Geo& g, const Node& n, const Nbr& d, const double* ct,
                                       const double* nu, const double* aj,
                                       const double* np, double gp, double* E) {
  const long long C = g.C;
  const unsigned o = n.o;
  const double nuo = nu[o];
  double e[3];
  e[0] = 0.5 * (ct[o] + ct[o + d.xp]) + nuo * aj[o];
  e[1] = 0.5 * (ct[o + C] + ct[o + C + d.yp]) + nuo * aj[o + C];
  e[2] = 0.5 * (ct[o + 2 * C] + ct[o + 2 * C + d.zp]) + nuo * aj[o + 2 * C];
  if (gp != 0.0)
    for (int m = 0; m < 3; ++m) e[m] = e[m] - grad_pe_at(g, np, gp, n, m);
  E[o] = e[0];
  E[o + C] = e[1];
  E[o + 2 * C] = e[2];
  ghosts3(g, n, E, e[0], e[1], e[2]);
}

// curlE (gutsf.f:288-299) and b1p2 = base - coef*curlE (predict_B
// gutsf.f:1158-1159 with coef = 2*dtsub; correct_B :1349-1350 with coef =
// dtsub), with b1p2's ghost images.  half: also the B at m+1/2 of get_Ep1
// (gutsf.f:1210-1219), 0.5*(b1p2 + b1), at the interior nodes.
template <int SP>
__device__ __forceinline__ void b_node(const Geo& g, const Node& n, const Nbr& d, const double* E,
                                       const double* base, double coef, double* b1p2,
                                       const double* b1, double* half) {
  const long long C = g.C;
  const unsigned o = n.o;
  const double *E1 = E, *E2 = E + C, *E3 = E + 2 * C;
  const double dx = g.dxg[n.i], dy = g.dyg[n.j], dz = g.dzg[n.k];
  const double rx = g.rdxg[n.i], ry = g.rdyg[n.j], rz = g.rdzg[n.k];
  const double e1 = E1[o], e2 = E2[o], e3 = E3[o];
  const double ce1 = quotient<SP>(E3[o + d.yp] - e3, dy, ry) + quotient<SP>(e2 - E2[o + d.zp], dz, rz);
  const double ce2 = quotient<SP>(e3 - E3[o + d.xp], dx, rx) + quotient<SP>(E1[o + d.zp] - e1, dz, rz);
  const double ce3 = quotient<SP>(e1 - E1[o + d.yp], dy, ry) + quotient<SP>(E2[o + d.xp] - e2, dx, rx);
  const double v0 = base[o] - coef * ce1;
  const double v1 = base[o + C] - coef * ce2;
  const double v2 = base[o + 2 * C] - coef * ce3;
  if (b1p2) {
    b1p2[o] = v0;
    b1p2[o + C] = v1;
    b1p2[o + 2 * C] = v2;
    ghosts3(g, n, b1p2, v0, v1, v2);
  }
  if (half) {
    half[o] = 0.5 * (v0 + b1[o]);
    half[o + C] = 0.5 * (v1 + b1[o + C]);
    half[o + 2 * C] = 0.5 * (v2 + b1[o + 2 * C]);
  }
}

// ---- kernels --------------------------------------------------------------------

#define NODES(n, d)                                                     \
  const unsigned t_ = blockIdx.x * blockDim.x + threadIdx.x;            \
  if (t_ >= (unsigned)n_interior(g)) return;                            \
  const Node n = node_of(g, t_);                                        \
  const Nbr d = nbr_of(g, n)

// curlB; FILL: b's ghosts too (curlB begins with periodic(b)).  btc (not
// null): edge_to_center of b at the interior nodes, for the corrector.
template <int SP>
__global__ void __launch_bounds__(TPB) k_curlB(Geo g, double* b, const double* np,
                                               const double* den, double alpha,
                                               double* aj, double* btc, bool fill) {
  after_previous();
  NODES(n, d);
  curlB_node<SP>(g, n, d, b, np, den, alpha, aj);
  if (btc) {
    double c[3];
    e2c_node(g, n, d, b, c);
    btc[n.o] = c[0];
    btc[n.o + g.C] = c[1];
    btc[n.o + 2 * g.C] = c[2];
  }
  if (fill) fill3(g, n, b);
}

// The divisors of curlB and their reciprocals: once per field step, where each
// of its 20 curls divided anew (nine operations a quotient).
__global__ void __launch_bounds__(TPB) k_face_density(Geo g, const double* np, double alpha,
                                                      double* den) {
  after_previous();
  const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (unsigned)n_interior(g)) return;
  const unsigned o = node_of(g, t).o;
  double f[3];
  face_densities(g, np, alpha, o, f);
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    den[o + g.C * m] = f[m];
    den[o + g.C * (3 + m)] = reciprocal(f[m]);
  }
}

template <bool CORR>
__global__ void __launch_bounds__(TPB) k_ct(Geo g, const double* aj, const double* up,
                                            double* b, double* ct, bool fill) {
  after_previous();
  NODES(n, d);
  ct_node<CORR>(g, n, d, aj, up, b, ct);
  if (fill) fill3(g, n, b);
}

__global__ void __launch_bounds__(TPB) k_E(Geo g, const double* ct, const double* nu,
                                           const double* aj, const double* np, double gp,
                                           double* E) {
  after_previous();
  NODES(n, d);
  e_node(g, n, d, ct, nu, aj, np, gp, E);
}

template <int SP>
__global__ void __launch_bounds__(TPB) k_B(Geo g, const double* E, const double* base,
                                           double coef, double* b1p2, const double* b1,
                                           double* half) {
  after_previous();
  NODES(n, d);
  b_node<SP>(g, n, d, E, base, coef, b1p2, b1, half);
}

// 0.5*(a + b) at the interior nodes (gutsf.f:1210-1219); the consumers read
// ghosts at their images.
__global__ void __launch_bounds__(TPB) k_half(Geo g, const double* a, const double* b,
                                              double* out) {
  after_previous();
  const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (unsigned)n_interior(g)) return;
  const unsigned o = node_of(g, t).o;
  for (int m = 0; m < 3; ++m) out[o + g.C * m] = 0.5 * (a[o + g.C * m] + b[o + g.C * m]);
}

// edge_to_center (grid_interp.f:10-62): bt's and btc's ghosts too.
__global__ void __launch_bounds__(TPB) k_edge_to_center(Geo g, double* bt, double* btc) {
  after_previous();
  NODES(n, d);
  double c[3];
  e2c_node(g, n, d, bt, c);
  btc[n.o] = c[0];
  btc[n.o + g.C] = c[1];
  btc[n.o + 2 * g.C] = c[2];
  ghosts3(g, n, btc, c[0], c[1], c[2]);
  fill3(g, n, bt);
}

// face_to_center (grid_interp.f:136-176) of v, and of w when given: the
// ghosts of inputs and outputs too.
__global__ void __launch_bounds__(TPB) k_face_to_center(Geo g, double* v, double* vc, double* w,
                                                        double* wc) {
  after_previous();
  NODES(n, d);
  const long long C = g.C;
  const unsigned o = n.o;
  const double xr = g.xr[n.i], yr = g.yr[n.j], zr = g.zr[n.k];
  for (int q = 0; q < 2; ++q) {
    double *in = q ? w : v, *out = q ? wc : vc;
    if (!in) break;
    const double c0 = f2c(xr, in[o], in[o + d.xm]);
    const double c1 = f2c(yr, in[o + C], in[o + C + d.ym]);
    const double c2 = f2c(zr, in[o + 2 * C], in[o + 2 * C + d.zm]);
    out[o] = c0;
    out[o + C] = c1;
    out[o + 2 * C] = c2;
    ghosts3(g, n, out, c0, c1, c2);
    fill3(g, n, in);
  }
}

// The end of update_up (gutsp.f:1825-1839): ct = S/np at the interior (zero
// where no particle deposits, as in the reference) and its face average, with
// up's ghosts.
__device__ __forceinline__ double ct_at(const double* S, const double* np, unsigned o, long long cm) {
  const double n = np[o];
  return n == 0.0 ? 0.0 : S[o + cm] / n;
}
__global__ void __launch_bounds__(TPB) k_up(Geo g, const double* S, double* np,
                                            double* up, bool fill_np) {
  after_previous();
  NODES(n, d);
  const long long C = g.C;
  const unsigned o = n.o;
  const double u0 = 0.5 * (ct_at(S, np, o, 0) + ct_at(S, np, o + d.xp, 0));
  const double u1 = 0.5 * (ct_at(S, np, o, C) + ct_at(S, np, o + d.yp, C));
  const double u2 = 0.5 * (ct_at(S, np, o, 2 * C) + ct_at(S, np, o + d.zp, 2 * C));
  up[o] = u0;
  up[o + C] = u1;
  up[o + 2 * C] = u2;
  ghosts3(g, n, up, u0, u1, u2);
  if (fill_np && on_edge(g, n)) store_ghosts(g.nx, g.ny, g.nz, g.C, 1, np, n.i, n.j, n.k, np[o], 0.0, 0.0);
}

// The particle passes' gather table, six doubles per node (ghosts included):
// face_to_center(aj - up), and edge_to_center(bt) when FULL (otherwise the
// table keeps it).  FULL also stores btc and fills aj's ghosts, as the
// operators it stands for do (edge_to_center, get_Ep's face_to_center(aj)).
// It also clears the velocity sums S, and np when given, for the next pass's
// deposit (at the interior nodes, where deposits go): three clears a step of
// their own cost 10 steps of 64x32x32 cells 0.14 ms of 8.17.
template <bool FULL>
__global__ void __launch_bounds__(TPB) k_kit(Geo g, double* aj, const double* up,
                                             const double* bt, double* btc,
                                             double* kit, double* S, double* np) {
  after_previous();
  NODES(n, d);
  const long long C = g.C;
  const unsigned o = n.o;
  double v[6];
  v[0] = f2c(g.xr[n.i], aj[o] - up[o], aj[o + d.xm] - up[o + d.xm]);
  v[1] = f2c(g.yr[n.j], aj[o + C] - up[o + C], aj[o + C + d.ym] - up[o + C + d.ym]);
  v[2] = f2c(g.zr[n.k], aj[o + 2 * C] - up[o + 2 * C], aj[o + 2 * C + d.zm] - up[o + 2 * C + d.zm]);
  if (FULL) {
    e2c_node(g, n, d, bt, v + 3);
    btc[o] = v[3];
    btc[o + C] = v[4];
    btc[o + 2 * C] = v[5];
    ghosts3(g, n, btc, v[3], v[4], v[5]);
    fill3(g, n, aj);
  }
  S[o] = 0.0;
  S[o + C] = 0.0;
  S[o + 2 * C] = 0.0;
  if (np) np[o] = 0.0;
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  const int is[3] = {n.i, n.i == 2 ? nx : 0, n.i == nx - 1 ? 1 : 0};
  const int js[3] = {n.j, n.j == 2 ? ny : 0, n.j == ny - 1 ? 1 : 0};
  const int ks[3] = {n.k, n.k == 2 ? nz : 0, n.k == nz - 1 ? 1 : 0};
  const int m = on_edge(g, n) ? 3 : 1;
  for (int c = 0; c < m; ++c)
    for (int b = 0; b < m; ++b)
      for (int a = 0; a < m; ++a) {
        if (!is[a] || !js[b] || !ks[c]) continue;
        double* w = kit + 6 * nidx(g, is[a], js[b], ks[c]);
#pragma unroll
        for (int q = 0; q < (FULL ? 6 : 3); ++q) w[q] = v[q];
      }
}

// from to both a and b (f_update_tlev's copies of the new B; 10 steps of 64x32x32
// cells 8.03 -> 7.91 ms against two copies).
__global__ void __launch_bounds__(256) k_copy_both(long long n, const double* from, double* a, double* b) {
  after_previous();
  for (long long t = blockIdx.x * 256LL + threadIdx.x; t < n; t += gridDim.x * 256LL) {
    const double v = from[t];
    a[t] = v;
    b[t] = v;
  }
}

// ---- the whole field step of a small grid in one launch ----
//
// The eight kernels of a subcycle as phases of one cooperative kernel, whose
// blocks meet at a barrier (0.9 us) instead of in a launch: below
// FIELD_LOOP_NODES a phase's FP64 work is about as long as a launch and the
// ramp of its loads.  The same node functions on the same operands: the same
// bits.  A step of 4 ions per cell, loop against launches, in ms: 1k nodes
// 0.390 against 0.396, 33k 0.56 against 0.79, 65k 0.82 against 1.01, 98k 1.14
// against 1.27, 131k 1.38 against 1.64, 164k 1.70 against 1.77, 262k 2.46
// against 2.41 (16 warps per SM then hide less than a full SM): hence
// FIELD_LOOP_NODES.
constexpr int LOOP_TPB = 512;
template <int SP>
__global__ void __launch_bounds__(LOOP_TPB) k_field_loop(Geo g, FieldLoop64 f) {
  // the same in every block: a Courant violation leaves the state as it is
  if (__longlong_as_double((long long)*f.courant) <= f.courant_floor) return;
  loop::Barrier bar{f.bar, f.polls, 0u, true};
  const unsigned nodes = (unsigned)n_interior(g), t0 = blockIdx.x * blockDim.x + threadIdx.x,
                 step = gridDim.x * blockDim.x;
  auto each = [&](auto&& node) {
    for (unsigned t = t0; t < nodes; t += step) {
      const Node n = node_of(g, t);
      node(n, nbr_of(g, n));
    }
    return bar.sync<false>();
  };
  double *now = f.b1, *old = f.b12;
  for (int s = 0; s < f.n; ++s) {
    double* b = s == 0 ? f.bt : now;
    const bool on =
        each([&](const Node& n, const Nbr& d) {
          curlB_node<SP>(g, n, d, b, f.np, f.den, f.alpha, f.aj);
          if (s == 0) fill3(g, n, b);
        }) &&
        each([&](const Node& n, const Nbr& d) { ct_node<false>(g, n, d, f.aj, f.up, b, f.ct); }) &&
        each([&](const Node& n, const Nbr& d) { e_node(g, n, d, f.ct, f.nu, f.aj, f.np, f.gp, f.E); }) &&
        each([&](const Node& n, const Nbr& d) {
          b_node<SP>(g, n, d, f.E, old, 2.0 * f.dtsub, nullptr, now, f.half);
        }) &&
        each([&](const Node& n, const Nbr& d) {
          curlB_node<SP>(g, n, d, f.half, f.np, f.den, f.alpha, f.aj);
          double c[3];
          e2c_node(g, n, d, f.half, c);
          f.btc[n.o] = c[0];
          f.btc[n.o + g.C] = c[1];
          f.btc[n.o + 2 * g.C] = c[2];
        }) &&
        each([&](const Node& n, const Nbr& d) { ct_node<true>(g, n, d, f.aj, f.up, f.btc, f.ct); }) &&
        each([&](const Node& n, const Nbr& d) { e_node(g, n, d, f.ct, f.nu, f.aj, f.np, f.gp, f.E); }) &&
        each([&](const Node& n, const Nbr& d) { b_node<SP>(g, n, d, f.E, now, f.dtsub, old, nullptr, nullptr); });
    if (!on) break;
    double* q = now;
    now = old;
    old = q;
  }
  if (!bar.ok && threadIdx.x == 0) set_err(f.err, KERR_WAIT);
  bar.done();
}

}  // namespace

// ---- launchers --------------------------------------------------------------------

bool field_loop_fits(const Geo& g) { return n_interior(g) <= FIELD_LOOP_NODES; }
cudaError_t field_loop(const Geo& g, const FieldLoop64& f, cudaStream_t st) {
  Geo gg = g;
  FieldLoop64 ff = f;
  void* args[] = {&gg, &ff};
  const void* k = g.spacing == SPACING_UNIT ? reinterpret_cast<const void*>(&k_field_loop<SPACING_UNIT>)
                  : g.spacing == SPACING_P2 ? reinterpret_cast<const void*>(&k_field_loop<SPACING_P2>)
                                            : reinterpret_cast<const void*>(&k_field_loop<SPACING_ANY>);
  // the nodes evenly over the SMs, a block on each, and over the rounds of
  // its threads
  const long long n = n_interior(g), per = (n + 151) / 152, rounds = (per + LOOP_TPB - 1) / LOOP_TPB,
                  t = ((per + rounds - 1) / rounds + 31) / 32 * 32;
  return loop::launch(k, (n + t - 1) / t, (int)t, args, st);
}

#define FL(kern, ...)                                                 \
  do {                                                                \
    return launch_next(kern, nblocks(n_interior(g)), threads_for(n_interior(g)), st, __VA_ARGS__); \
  } while (0)

cudaError_t curlB(const Geo& g, double* b, const double* np, const double* den, double alpha, double* aj,
                  double* btc, bool fill, cudaStream_t st) {
  if (g.spacing == SPACING_UNIT) FL(k_curlB<SPACING_UNIT>, g, b, np, den, alpha, aj, btc, fill);
  if (g.spacing == SPACING_P2) FL(k_curlB<SPACING_P2>, g, b, np, den, alpha, aj, btc, fill);
  FL(k_curlB<SPACING_ANY>, g, b, np, den, alpha, aj, btc, fill);
}
cudaError_t face_density(const Geo& g, const double* np, double alpha, double* den, cudaStream_t st) {
  FL(k_face_density, g, np, alpha, den);
}
cudaError_t cross_ct(const Geo& g, bool corr, const double* aj, const double* up, double* b, double* ct, bool fill,
                     cudaStream_t st) {
  if (corr) FL(k_ct<true>, g, aj, up, b, ct, fill);
  FL(k_ct<false>, g, aj, up, b, ct, fill);
}
cudaError_t e_field(const Geo& g, const double* ct, const double* nu, const double* aj, const double* np, double gp,
                    double* E, cudaStream_t st) {
  FL(k_E, g, ct, nu, aj, np, gp, E);
}
cudaError_t b_advance(const Geo& g, const double* E, const double* base, double coef, double* b1p2, const double* b1,
                      double* half, cudaStream_t st) {
  if (g.spacing == SPACING_UNIT) FL(k_B<SPACING_UNIT>, g, E, base, coef, b1p2, b1, half);
  if (g.spacing == SPACING_P2) FL(k_B<SPACING_P2>, g, E, base, coef, b1p2, b1, half);
  FL(k_B<SPACING_ANY>, g, E, base, coef, b1p2, b1, half);
}
cudaError_t half_sum(const Geo& g, const double* a, const double* b, double* out, cudaStream_t st) {
  FL(k_half, g, a, b, out);
}
cudaError_t edge_to_center(const Geo& g, double* bt, double* btc, cudaStream_t st) {
  FL(k_edge_to_center, g, bt, btc);
}
cudaError_t face_to_center(const Geo& g, double* v, double* vc, double* w, double* wc, cudaStream_t st) {
  FL(k_face_to_center, g, v, vc, w, wc);
}
cudaError_t up_from_sums(const Geo& g, const double* S, double* np, double* up, bool fill_np, cudaStream_t st) {
  FL(k_up, g, S, np, up, fill_np);
}
cudaError_t copy_both(long long n, const double* from, double* a, double* b, cudaStream_t st) {
  const long long blocks = (n + 255) / 256;
  return launch_next(k_copy_both, (unsigned)(blocks < 152 * 8 * 4 ? blocks : 152 * 8 * 4), 256, st, n, from, a, b);
}
cudaError_t gather_kit(const Geo& g, bool full, double* aj, const double* up, const double* bt, double* btc,
                       double* kit, double* S, double* np, cudaStream_t st) {
  if (full) FL(k_kit<true>, g, aj, up, bt, btc, kit, S, np);
  FL(k_kit<false>, g, aj, up, bt, btc, kit, S, np);
}

}  // namespace swapk
