// k64_pass.cu -- the particle half of a fused FP64 ion step (maind.f:385-413
// and the half move of :479) in three passes over the particles:
//   pass 1: weights (gutsp.f:1378-1435), the deposits of update_np and of
//           extrapol_up's 1.5 v - 0.5 vp1 (maind.f:385-386, 399);
//   pass 2: get_Ep, v-/v+ and improve_up's deposit (maind.f:400-402);
//   pass 3: get_Ep with the improved up, v-/v+, get_vp_final, the half move,
//           the weights and both deposits at the new position (maind.f:404-413)
//           and the half move of maind.f:479.
// (maind.f:387's update_up is not deposited: extrapol_up overwrites up before
// anything reads it.)
//
// What bounds them: GB300's FP64 pipe, two operations per SM and clock (a
// warp instruction takes 16 clocks, 527e9 a second measured), so what counts is the number
// of FP64 operations per ion, about 350 here against 930 for the operators
// one by one:
//  * fused multiply-adds wherever the sum's rounding is free;
//  * the difference aj - up is gathered (three components), not both fields;
//    B is gathered once per step and kept (24 B per ion) for pass 3;
//  * the weights are formed once per position and read back (64 B per ion:
//    HBM has room, the FP64 pipe has not);
//  * comparisons and the cell search run on integers (k64_dev.cuh);
//  * a particle's 8 weights and 4 moments go to shared memory and lane (moment,
//    corner) forms the warp's sums: 32 fused operations per 32 ions and no
//    FP64 atomic per ion.  The columns are the warp's ions grouped by cell
//    (__match_any_sync), so a cell's sum leaves as one reduction per value:
//    L2 takes about 200e9 FP64 reductions a second, and 24 + 8 per ion were
//    the deposits' bound.
// 8.4M ions, 128x64x64 cells, ms per step for the particle half: 1.21 + 2.07 + 2.73 = 6.0 (pass
// 1, 2, 3) against 17.3 for the operators one by one.
#include "k64.cuh"
#include "k64_dev.cuh"

namespace swapk {
namespace {

constexpr int TPB = 128, WARPS = TPB / 32;
constexpr int ROW = 34;  // doubles per row: 8 rows a lane group reads at once start on different banks

struct Red {
  double v[12][ROW];            // 8 weights, 4 moments; columns = the warp's ions grouped by cell
  unsigned long long cell[32];  // i | j << 21 | k << 42 per column; ~0 for none
};

__device__ __forceinline__ unsigned long long pack(int i, int j, int k) {
  return (unsigned long long)i | (unsigned long long)j << 21 | (unsigned long long)k << 42;
}

// Adds the warp's ions to the node sums.  w: the corner weights in the
// reference's order (x, z, y from the lowest bit); m: the density and
// velocity moments.  NP false: the velocity moments alone.
template <bool NP>
__device__ __forceinline__ void warp_deposit(const Geo& g, Red& s, bool live, unsigned node, unsigned long long cell,
                                             const double (&w)[8], const double (&m)[4], double* __restrict__ np,
                                             double* __restrict__ S) {
  const int lane = threadIdx.x & 31;
  const unsigned peers = __match_any_sync(0xffffffffu, live ? node : 0xffffffffu);
  const int leader = __ffs(peers) - 1;
  int incl = lane == leader ? __popc(peers) : 0;
  const int mine = incl;
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  const int base = __shfl_sync(0xffffffffu, incl - mine, leader);
  const int pos = base + __popc(peers & ((1u << lane) - 1u));
  // the column after each group is another group's first
  const unsigned heads = __reduce_or_sync(0xffffffffu, lane == leader ? 1u << base : 0u);
  const unsigned ends = (heads >> 1) | 0x80000000u;
#pragma unroll
  for (int c = 0; c < 8; ++c) s.v[c][pos] = live ? w[c] : 0.0;
#pragma unroll
  for (int q = NP ? 0 : 1; q < 4; ++q) s.v[8 + q][pos] = live ? m[q] : 0.0;
  s.cell[pos] = live ? cell : ~0ull;
  __syncwarp();
  const int cv = lane & 7, qv = lane >> 3;
  const bool adds = NP || qv != 0;
  const double2* wr = reinterpret_cast<const double2*>(s.v[cv]);
  const double2* mr = reinterpret_cast<const double2*>(s.v[8 + (adds ? qv : 1)]);
  double* const arr = qv == 0 ? np : S + (qv - 1) * g.C;
  auto flush = [&](int r, double acc) {
    const unsigned long long c = s.cell[r];
    if (c == ~0ull || !adds) return;
    const int i = (int)(c & 0x1fffffu) + (cv & 1), j = (int)(c >> 21 & 0x1fffffu) + (cv >> 2),
              k = (int)(c >> 42) + (cv >> 1 & 1);
    const long long t = fold_target(g, i, j, k);
    if (t >= 0) atomicAdd(arr + t, acc);
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
  __syncwarp();
}

// Constants of the block: the guess of the cell search, and the density
// factors of the first particle's beta_p (most runs have one or two).
struct BlockConst {
  double bp, inv_n, inv_u;  // update_np's volb and update_up's 1/volb for bp
};

__device__ __forceinline__ double volume_factor(double cell, double beta, double bp) {
  return 1.0 / (cell * beta * bp);
}

// Cell and weights at a position (get_interp_weights), stored like the
// reference's COMMON blocks; false when the position is outside the grid.
__device__ __forceinline__ bool locate(const PassArgs& a, long long l, double x, double y, double z, int& i, int& j,
                                       int& k, double (&w)[8]) {
  const Geo& g = a.g;
  const PartDev& p = a.p;
  i = find_cell(g.qx, g.nx, x, (float)g.qx[1], (float)g.inv_dx);
  k = find_cell(g.qz, g.nz, z, (float)g.qz[1], (float)g.inv_dz);
  j = __double2int_rz(quotient<false>(y, g.dy, g.rdy));  // floor for y >= 0; any y below is outside either way
  const bool ok = i >= 1 && j >= 1 && j < g.ny && k >= 1;
  if (!ok) i = j = k = 1;
  p.ijk[l] = i;
  p.ijk[l + p.NM] = j;
  p.ijk[l + 2 * p.NM] = k;
  if (!ok) {
#pragma unroll
    for (int c = 0; c < 8; ++c) p.wght[l + c * p.NM] = w[c] = 0.0;
    return false;
  }
  const double qx = g.qx[i], qxp = g.qx[i + 1], qy = g.qy[j], qyp = g.qy[j + 1], qz = g.qz[k], qzp = g.qz[k + 1];
  const double vol = g.uniform ? g.inv_cell_q : 1.0 / ((qxp - qx) * (qyp - qy) * (qzp - qz));
  const double x1 = fabs(x - qx), x2 = fabs(x - qxp), y1 = fabs(y - qy), y2 = fabs(y - qyp), z1 = fabs(z - qz),
               z2 = fabs(z - qzp);
  const double x2y2 = x2 * y2, x1y2 = x1 * y2, x2y1 = x2 * y1, x1y1 = x1 * y1;
  w[0] = x2y2 * z2 * vol;
  w[1] = x1y2 * z2 * vol;
  w[2] = x2y2 * z1 * vol;
  w[3] = x1y2 * z1 * vol;
  w[4] = x2y1 * z2 * vol;
  w[5] = x1y1 * z2 * vol;
  w[6] = x2y1 * z1 * vol;
  w[7] = x1y1 * z1 * vol;
#pragma unroll
  for (int c = 0; c < 8; ++c) p.wght[l + c * p.NM] = w[c];
  return true;
}

// update_np's 1/(dx_grid dy_grid dz_grid beta beta_p) and update_up's inverse volb.
__device__ __forceinline__ void density_factors(const PassArgs& a, const BlockConst& bc, long long l, int i, int j,
                                                int k, double& fn, double& fu) {
  const Geo& g = a.g;
  const double bp = a.p.beta_p[l];
  if (!g.uniform) {
    fn = volume_factor(g.dxg[i] * g.dyg[j] * g.dzg[k], a.beta, bp);
    fu = volume_factor((g.qx[i + 1] - g.qx[i]) * (g.qy[j + 1] - g.qy[j]) * (g.qz[k + 1] - g.qz[k]), a.beta, bp);
  } else if (__double_as_longlong(bp) == __double_as_longlong(bc.bp)) {
    fn = bc.inv_n;
    fu = bc.inv_u;
  } else {
    fu = volume_factor(g.cell_q, a.beta, bp);
    fn = g.cell_g == g.cell_q ? fu : volume_factor(g.cell_g, a.beta, bp);
  }
}

// The half move of move_ion_half along one axis with its one wrap (gutsp.f:473-510).
__device__ __forceinline__ double half_move(double x, double v, double dth, double q1, double qn, bool wrap) {
  x = x + dth * v;
  if (wrap) {
    const long long b = ordered(x);
    if (b > ordered(qn)) x = q1 + (x - qn);
    else if (b <= ordered(q1)) x = qn - (q1 - x);
  }
  return x;
}

template <int PASS>
__global__ void __launch_bounds__(TPB, 4) k_pass(PassArgs a) {
  __shared__ Red s_red[WARPS];
  __shared__ BlockConst s_bc;
  const Geo& g = a.g;
  const PartDev& p = a.p;
  const long long NM = p.NM;
  if (threadIdx.x == 0) {
    const double bp = p.beta_p[0];
    s_bc.bp = bp;
    s_bc.inv_n = volume_factor(g.cell_g, a.beta, bp);
    s_bc.inv_u = volume_factor(g.cell_q, a.beta, bp);
  }
  __syncthreads();
  Red& red = s_red[threadIdx.x >> 5];
  const long long step = (long long)gridDim.x * TPB;
  // whole warps take part in the deposits
  for (long long base = (long long)blockIdx.x * TPB + (threadIdx.x & ~31); base < a.N; base += step) {
    const long long l = base + (threadIdx.x & 31);
    bool live = l < a.N;
    int i = 1, j = 1, k = 1;
    double w[8], m[4];
#pragma unroll
    for (int c = 0; c < 8; ++c) w[c] = 0.0;
#pragma unroll
    for (int q = 0; q < 4; ++q) m[q] = 0.0;
    if (live && PASS == 1) {
      live = locate(a, l, p.xp[l], p.xp[l + NM], p.xp[l + 2 * NM], i, j, k, w);
      if (!live) set_err(a.err, KERR_DOMAIN);
      double fn, fu;
      density_factors(a, s_bc, l, i, j, k, fn, fu);
      m[0] = fn;
      const double f1 = 1.5 * fu, f2 = -0.5 * fu;
#pragma unroll
      for (int q = 0; q < 3; ++q)  // extrapol_up (gutsp.f:144)
        m[1 + q] = __fma_rn(f1, p.vp[l + q * NM], f2 * p.vp1[l + q * NM]);
    }
    if (live && PASS != 1) {
      i = p.ijk[l];
      j = p.ijk[l + NM];
      k = p.ijk[l + 2 * NM];
#pragma unroll
      for (int c = 0; c < 8; ++c) w[c] = p.wght[l + c * NM];
      const double2* kit = reinterpret_cast<const double2*>(a.kit) + 3 * nidx(g, i, j, k);
      const long long sy = 3LL * g.nx, sz = sy * g.ny;
      double A[3] = {0.0, 0.0, 0.0}, B[3] = {0.0, 0.0, 0.0};
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const double2* t = kit + 3 * (c & 1) + sy * (c >> 2) + sz * (c >> 1 & 1);
        const double2 t0 = t[0];
        A[0] = __fma_rn(w[c], t0.x, A[0]);
        A[1] = __fma_rn(w[c], t0.y, A[1]);
        if (PASS == 2) {
          const double2 t1 = t[1], t2 = t[2];
          A[2] = __fma_rn(w[c], t1.x, A[2]);
          B[0] = __fma_rn(w[c], t1.y, B[0]);
          B[1] = __fma_rn(w[c], t2.x, B[1]);
          B[2] = __fma_rn(w[c], t2.y, B[2]);
        } else {
          A[2] = __fma_rn(w[c], reinterpret_cast<const double*>(t)[2], A[2]);
        }
      }
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        if (PASS == 2) a.b3[l + q * NM] = B[q];
        else B[q] = a.b3[l + q * NM];
      }
      const double mr = p.mrat[l], dt = a.dt, h = 0.5 * dt;
      double v[3], E[3];
#pragma unroll
      for (int q = 0; q < 3; ++q) v[q] = p.vp[l + q * NM];
      // Ep = ((aj - up) x B) mrat (gutsp.f:260-270)
      E[0] = __fma_rn(A[1], B[2], -(A[2] * B[1])) * mr;
      E[1] = __fma_rn(A[2], B[0], -(A[0] * B[2])) * mr;
      E[2] = __fma_rn(A[0], B[1], -(A[1] * B[0])) * mr;
      // v- and the rotation of get_vplus_vminus (gutsp.f:302-397)
      double vm[3], vn[3];
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        vm[q] = __fma_rn(h, E[q], v[q]);
        B[q] = B[q] * mr;
      }
      const double t = 0.25 * dt * dt * __fma_rn(B[0], B[0], __fma_rn(B[1], B[1], B[2] * B[2]));
      const double ad = 1.0 / (1.0 + t), om = 1.0 - t;
      const double kd = 0.5 * dt * dt * __fma_rn(vm[0], B[0], __fma_rn(vm[1], B[1], vm[2] * B[2]));
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        const int q1 = (q + 1) % 3, q2 = (q + 2) % 3;
        const double c = __fma_rn(vm[q1], B[q2], -(vm[q2] * B[q1]));
        vn[q] = ad * __fma_rn(kd, B[q], __fma_rn(dt, c, om * vm[q]));
      }
      double fn, fu;
      if (PASS == 2) {  // improve_up (gutsp.f:422)
        density_factors(a, s_bc, l, i, j, k, fn, fu);
        const double f = 0.5 * fu;
#pragma unroll
        for (int q = 0; q < 3; ++q) m[1 + q] = f * (vn[q] + vm[q]);
      } else {
        // get_vp_final (gutsp.f:442-446)
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          vn[q] = __fma_rn(h, E[q], vn[q]);
          p.vp1[l + q * NM] = v[q];
          p.vp[l + q * NM] = vn[q];
        }
        const double dth = dt / 2.;
        const double qx1 = g.qx[1], qxn = g.qx[g.nx - 1], qy1 = g.qy[1], qyn = g.qy[g.ny - 1], qz1 = g.qz[1],
                     qzn = g.qz[g.nz - 1];
        double x = half_move(p.xp[l], vn[0], dth, qx1, qxn, !a.x_open);
        double y = half_move(p.xp[l + NM], vn[1], dth, qy1, qyn, true);
        double z = half_move(p.xp[l + 2 * NM], vn[2], dth, qz1, qzn, true);
        const bool out = a.x_open && !(ordered(x) > ordered(qx1) && ordered(x) <= ordered(qxn));
        if (out) {  // removed by the caller; its weights are those of no cell
          p.ijk[l] = p.ijk[l + NM] = p.ijk[l + 2 * NM] = 1;
#pragma unroll
          for (int c = 0; c < 8; ++c) p.wght[l + c * NM] = 0.0;
          live = false;
        } else {
          live = locate(a, l, x, y, z, i, j, k, w);
          if (!live) set_err(a.err, KERR_DOMAIN);
          density_factors(a, s_bc, l, i, j, k, fn, fu);
          m[0] = fn;
#pragma unroll
          for (int q = 0; q < 3; ++q) m[1 + q] = fu * vn[q];
        }
        if (a.final_move) {  // maind.f:479
          x = half_move(x, vn[0], dth, qx1, qxn, !a.x_open);
          y = half_move(y, vn[1], dth, qy1, qyn, true);
          z = half_move(z, vn[2], dth, qz1, qzn, true);
        }
        p.xp[l] = x;
        p.xp[l + NM] = y;
        p.xp[l + 2 * NM] = z;
      }
    }
    warp_deposit<PASS != 2>(g, red, live, (unsigned)nidx(g, i, j, k), pack(i, j, k), w, m, a.np, a.S);
  }
}

}  // namespace

cudaError_t particle_pass(int pass, const PassArgs& a, cudaStream_t st) {
  if (a.N <= 0) return cudaSuccess;
  // four blocks of 128 an SM hide the latencies; more blocks than that at
  // once only repeat the block's set-up
  const long long need = (a.N + TPB - 1) / TPB, most = 152LL * 4 * 8;
  const unsigned nb = (unsigned)(need < most ? need : most);
  if (pass == 1) k_pass<1><<<nb, TPB, 0, st>>>(a);
  else if (pass == 2) k_pass<2><<<nb, TPB, 0, st>>>(a);
  else k_pass<3><<<nb, TPB, 0, st>>>(a);
  return cudaGetLastError();
}

}  // namespace swapk
