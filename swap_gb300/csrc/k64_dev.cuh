// k64_dev.cuh -- device helpers of the FP64 drop-in's fused kernels.
#pragma once

#include "swap_dev.cuh"

namespace swapk {

// How a quotient by a grid spacing is formed (Geo::spacing, set by the host).
enum Spacing : int {
  SPACING_ANY = 0,
  SPACING_P2 = 1,    // every spacing a power of two: its reciprocal is exact
  SPACING_UNIT = 2,  // every spacing one (lengths in cells): nothing to do
};

// x / d with r = 1/d rounded: exactly the rounded quotient.  A power of two: x
// * r is x / d with the same single rounding.  Otherwise Markstein's
// correction (P. Markstein, IBM J. Res. Dev. 34, 1990): q = x*r, then q + (x -
// q*d)*r in fused operations is the rounded quotient when r is the rounded
// reciprocal and nothing underflows or overflows: three operations instead of
// about nine.  x outside 2^-900..2^900 takes the division; reciprocal() is 0
// where the theorem does not hold (d outside 2^-60..2^60, or with an all-ones
// significand) and d is divided by.
template <int SP>
__device__ __forceinline__ double quotient(double x, double d, double r) {
  if (SP == SPACING_UNIT) return x;
  if (SP == SPACING_P2) return x * r;
  const unsigned e = ((unsigned)__double2hiint(x) >> 20) & 0x7ffu;
  if (e - 123u > 1800u || __double_as_longlong(r) == 0) {
    const bool zero = ((unsigned)__double2hiint(x) << 1 | (unsigned)__double2loint(x)) == 0u;
    return zero && __double_as_longlong(r) != 0 ? x * r : x / d;
  }
  const double q = x * r;
  return __fma_rn(__fma_rn(-q, d, x), r, q);
}
// 1/x for x in [2^-500, 2^500]: the hardware's approximation (within 2^-20) and
// two Newton-Raphson steps, four FP64 operations where a division takes about
// nine.  The second step starts within 2^-40, so what its last operation rounds
// is off by 2^-80 at most: the rounded reciprocal but for ties that close
// (emulated with seeds of 18 to 23 bits, none of 50 million arguments each
// differs from 1/x).
__device__ __forceinline__ double fast_reciprocal(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  r = __fma_rn(__fma_rn(-x, r, 1.0), r, r);
  return __fma_rn(__fma_rn(-x, r, 1.0), r, r);
}
__device__ __forceinline__ bool is_one(double x) { return __double_as_longlong(x) == 0x3ff0000000000000LL; }

__device__ __forceinline__ double reciprocal(double d) {
  const unsigned hi = (unsigned)__double2hiint(d), e = hi >> 20;  // the sign bit puts a negative d out of range
  const bool ones = (hi & 0xfffffu) == 0xfffffu && (unsigned)__double2loint(d) == 0xffffffffu;
  return e - 963u <= 120u && !ones ? 1.0 / d : 0.0;
}

// The bits of a double as an integer that orders like it (-0.0 just below 0.0,
// NaN beyond the infinities): a comparison costs a few integer instructions
// instead of one of the FP64 pipe's 16-clock slots.
__device__ __forceinline__ long long ordered(double x) {
  const long long b = __double_as_longlong(x);
  return b ^ ((b >> 63) & 0x7fffffffffffffffLL);
}
// The same of a position, to be held against ordered() nodes by > and <= alone:
// a zero of either sign as -0.0, so that it is not above a node at -0.0 or 0.0.
__device__ __forceinline__ long long ordered_position(double x) {
  const long long o = ordered(x);
  return o == 0 ? -1 : o;
}

// Cell search of get_interp_weights (gutsp.f:1396-1401): the index i with
// q(i) < x <= q(i+1), i.e. one less than the first node with x <= q(node), 0
// when x is outside (q(1), q(n)] or not a number.  An FP32 guess from the
// uniform spacing is corrected against the node array itself by integer
// comparisons, so the result is the reference's linear search for any
// monotone q.  The guess is bounded while it is a float: of a position far
// outside the conversion alone is the largest int, and one more overflows.
__device__ __forceinline__ int find_cell(const double* __restrict__ q, int n, double x, float q1, float inv_d) {
  const long long xb = ordered_position(x);
  int i = (int)fminf(fmaxf((__double2float_rn(x) - q1) * inv_d, 0.0f), 1.0e9f) + 1;
  i = i > n - 1 ? n - 1 : i;
  while (i > 1 && !(xb > ordered(q[i]))) --i;
  while (i < n - 1 && xb > ordered(q[i + 1])) ++i;
  return xb > ordered(q[i]) && xb <= ordered(q[i + 1]) ? i : 0;
}

// Cell and corner weights of a position (get_interp_weights, gutsp.f:1391-
// 1432), in the reference's order (000,100,001,101,010,110,011,111 over
// x,z,y) and with its products' rounding (their common factors formed once;
// on a uniform grid the cell's inverse volume is given).  Units compiled with
// --fmad=false round every product like the Fortran.  Outside the grid:
// false, cell (1,1,1) and weights of zero.
__device__ __forceinline__ bool weights_at(const Geo& g, double x, double y, double z, int& i, int& j, int& k,
                                           double (&w)[8]) {
  i = find_cell(g.qx, g.nx, x, (float)g.qx[1], (float)g.inv_dx);
  k = find_cell(g.qz, g.nz, z, (float)g.qz[1], (float)g.inv_dz);
  // floor for y >= 0 (any y below is outside either way); a spacing of one
  // needs no quotient
  j = __double2int_rz(is_one(g.rdy) ? y : quotient<SPACING_ANY>(y, g.dy, g.rdy));
  if (!(i >= 1 && j >= 1 && j < g.ny && k >= 1)) {
    i = j = k = 1;
#pragma unroll
    for (int c = 0; c < 8; ++c) w[c] = 0.0;
    return false;
  }
  const double qx = g.qx[i], qxp = g.qx[i + 1], qy = g.qy[j], qyp = g.qy[j + 1], qz = g.qz[k], qzp = g.qz[k + 1];
  const double vol = g.uniform ? g.inv_cell_q : 1.0 / ((qxp - qx) * (qyp - qy) * (qzp - qz));
  const double x1 = fabs(x - qx), x2 = fabs(x - qxp), y1 = fabs(y - qy), y2 = fabs(y - qyp), z1 = fabs(z - qz),
               z2 = fabs(z - qzp);
  const double x2y2 = x2 * y2, x1y2 = x1 * y2, x2y1 = x2 * y1, x1y1 = x1 * y1;
  w[0] = x2y2 * z2;
  w[1] = x1y2 * z2;
  w[2] = x2y2 * z1;
  w[3] = x1y2 * z1;
  w[4] = x2y1 * z2;
  w[5] = x1y1 * z2;
  w[6] = x2y1 * z1;
  w[7] = x1y1 * z1;
  if (!is_one(vol)) {  // (a unit cell: the products are the weights)
#pragma unroll
    for (int c = 0; c < 8; ++c) w[c] = w[c] * vol;
  }
  return true;
}

__device__ __forceinline__ double volume_factor(double cell, double beta, double bp) {
  return 1.0 / (cell * beta * bp);
}

// The density factors of one beta_p on a uniform grid, kept per block (most
// runs have one or two values): update_np's volb and update_up's 1/volb.
struct BlockConst {
  double bp, inv_n, inv_u;
  __device__ __forceinline__ void set(const Geo& g, double beta, double b) {
    bp = b;
    inv_n = volume_factor(g.cell_g, beta, b);
    inv_u = volume_factor(g.cell_q, beta, b);
  }
};

// update_np's 1/(dx_grid dy_grid dz_grid beta beta_p) and update_up's inverse
// volb for a particle of cell (i,j,k).
__device__ __forceinline__ void density_factors(const Geo& g, double beta, double bp, const BlockConst& bc, int i,
                                                int j, int k, double& fn, double& fu) {
  if (!g.uniform) {
    fn = volume_factor(g.dxg[i] * g.dyg[j] * g.dzg[k], beta, bp);
    fu = volume_factor((g.qx[i + 1] - g.qx[i]) * (g.qy[j + 1] - g.qy[j]) * (g.qz[k + 1] - g.qz[k]), beta, bp);
  } else if (__double_as_longlong(bp) == __double_as_longlong(bc.bp)) {
    fn = bc.inv_n;
    fu = bc.inv_u;
  } else {
    fu = volume_factor(g.cell_q, beta, bp);
    fn = g.cell_g == g.cell_q ? fu : volume_factor(g.cell_g, beta, bp);
  }
}

// update_up's factor alone, from the node coordinates.
__device__ __forceinline__ double flow_factor(const Geo& g, double beta, double bp, const BlockConst& bc, int i, int j,
                                              int k) {
  if (!g.uniform)
    return volume_factor((g.qx[i + 1] - g.qx[i]) * (g.qy[j + 1] - g.qy[j]) * (g.qz[k + 1] - g.qz[k]), beta, bp);
  return __double_as_longlong(bp) == __double_as_longlong(bc.bp) ? bc.inv_u : volume_factor(g.cell_q, beta, bp);
}

// ---- the deposits of one warp ----

constexpr int RED_ROW = 34;  // doubles per row: 8 rows a lane group reads at once start on different banks

struct Red {
  double v[12][RED_ROW];        // 8 weights, 4 moments; columns = the warp's ions grouped by cell
  unsigned long long cell[32];  // i | j << 21 | k << 42 per column; ~0 for none
};

// The column of each lane's ion with the warp's ions grouped by cell, and (the
// same in every lane) a bit per column that ends a group.
__device__ __forceinline__ int group_by_cell(unsigned node, unsigned& ends) {
  const int lane = threadIdx.x & 31;
  const unsigned peers = __match_any_sync(0xffffffffu, node);
  const int leader = __ffs(peers) - 1;
  const int mine = lane == leader ? __popc(peers) : 0;
  int incl = mine;
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  const int base = __shfl_sync(0xffffffffu, incl - mine, leader);
  // the column before each group's first ends another group
  ends = (__reduce_or_sync(0xffffffffu, lane == leader ? 1u << base : 0u) >> 1) | 0x80000000u;
  return base + __popc(peers & ((1u << lane) - 1u));
}

// Adds a sum at corner c (x, z, y from the lowest bit) of a packed cell.
__device__ __forceinline__ void add_at_corner(const Geo& g, double* arr, unsigned long long cell, int c, double v) {
  const int i = (int)(cell & 0x1fffffu) + (c & 1), j = (int)(cell >> 21 & 0x1fffffu) + (c >> 2),
            k = (int)(cell >> 42) + (c >> 1 & 1);
  const long long t = fold_target(g, i, j, k);
  if (t >= 0) atomicAdd(arr + t, v);
}

// Adds the warp's ions to the node sums: lane (moment, corner) forms the
// products of its row pair over the columns and adds each group's sum.  w:
// the corner weights; m: the density and velocity moments.  NP false: the
// velocity moments alone.
template <bool NP>
__device__ __forceinline__ void warp_deposit(const Geo& g, Red& s, bool live, int i, int j, int k,
                                             const double (&w)[8], const double (&m)[4], double* __restrict__ np,
                                             double* __restrict__ S) {
  const int lane = threadIdx.x & 31;
  unsigned ends;
  const int pos = group_by_cell(live ? (unsigned)nidx(g, i, j, k) : 0xffffffffu, ends);
#pragma unroll
  for (int c = 0; c < 8; ++c) s.v[c][pos] = live ? w[c] : 0.0;
#pragma unroll
  for (int q = NP ? 0 : 1; q < 4; ++q) s.v[8 + q][pos] = live ? m[q] : 0.0;
  s.cell[pos] = live ? (unsigned long long)i | (unsigned long long)j << 21 | (unsigned long long)k << 42 : ~0ull;
  __syncwarp();
  const int cv = lane & 7;
  if (NP) {
    const int qv = lane >> 3;
    const double2* wr = reinterpret_cast<const double2*>(s.v[cv]);
    const double2* mr = reinterpret_cast<const double2*>(s.v[8 + qv]);
    double* const arr = qv == 0 ? np : S + (qv - 1) * g.C;
    auto flush = [&](int r, double acc) {
      const unsigned long long c = s.cell[r];
      if (c != ~0ull) add_at_corner(g, arr, c, cv, acc);
    };
    double acc = 0.0;
#pragma unroll
    for (int r = 0; r < 16; ++r) {
      const double2 a = wr[r], b = mr[r];
      acc = __fma_rn(a.x, b.x, acc);
      if (ends >> (2 * r) & 1u) {
        flush(2 * r, acc);
        acc = 0.0;
      }
      acc = __fma_rn(a.y, b.y, acc);
      if (ends >> (2 * r + 1) & 1u) {
        flush(2 * r + 1, acc);
        acc = 0.0;
      }
    }
  } else {
    // 24 pairs of rows for 32 lanes: lane < 24 takes columns 0-23 of its
    // pair, lane 24 + corner columns 24-31 of the corner's three pairs; 24
    // operations each where a pair per lane takes 32
    const bool tail = lane >= 24;
    const double* wr = s.v[cv] + (tail ? 24 : 0);
    double acc = 0.0;
#pragma unroll
    for (int b = 0; b < 3; ++b) {  // eight columns at a time
      const int q = tail ? b : lane >> 3, r0 = tail ? 0 : 8 * b;
      const double* mr = s.v[9 + q] + (tail ? 24 : 0);
      const unsigned e8 = ends >> (tail ? 24 : 8 * b) & 0xffu;
#pragma unroll
      for (int r = 0; r < 8; r += 2) {
        const double2 x = *reinterpret_cast<const double2*>(wr + r0 + r), y = *reinterpret_cast<const double2*>(mr + r0 + r);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          acc = __fma_rn(h ? x.y : x.x, h ? y.y : y.x, acc);
          // a group ends, or this lane's columns do
          if ((e8 >> (r + h) & 1u) || (r + h == 7 && (b == 2 || tail))) {
            const unsigned long long c = s.cell[(tail ? 24 : 8 * b) + r + h];
            if (c != ~0ull) add_at_corner(g, S + q * g.C, c, cv, acc);
            acc = 0.0;
          }
        }
      }
    }
  }
  __syncwarp();
}

// One moment alone: lane (quarter, corner) takes eight of the columns.
__device__ __forceinline__ void warp_deposit1(const Geo& g, Red& s, bool live, int i, int j, int k,
                                              const double (&w)[8], double m, double* __restrict__ out) {
  const int lane = threadIdx.x & 31;
  unsigned ends;
  const int pos = group_by_cell(live ? (unsigned)nidx(g, i, j, k) : 0xffffffffu, ends);
#pragma unroll
  for (int c = 0; c < 8; ++c) s.v[c][pos] = live ? w[c] : 0.0;
  s.v[8][pos] = live ? m : 0.0;
  s.cell[pos] = live ? (unsigned long long)i | (unsigned long long)j << 21 | (unsigned long long)k << 42 : ~0ull;
  __syncwarp();
  const int cv = lane & 7, r0 = lane & 24;
  double acc = 0.0;
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    acc = __fma_rn(s.v[cv][r0 + r], s.v[8][r0 + r], acc);
    if (r == 7 || (ends >> (r0 + r) & 1u)) {
      const unsigned long long c = s.cell[r0 + r];
      if (c != ~0ull) add_at_corner(g, out, c, cv, acc);
      acc = 0.0;
    }
  }
  __syncwarp();
}

}  // namespace swapk
