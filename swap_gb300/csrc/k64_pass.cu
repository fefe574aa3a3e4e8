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
// of FP64 operations per ion, about 340 here against 930 for the operators
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
// 8.4M ions, 128x64x64 cells, ms per step for the particle half: 1.17 + 1.87 +
// 2.59 = 5.6 (pass 1, 2, 3; the FP64 pipe 88 to 92% busy) against 17.3 for the
// operators one by one.
#include "k64.cuh"
#include "k64_dev.cuh"

namespace swapk {
namespace {

constexpr int TPB = 128, WARPS = TPB / 32;

// Cell and weights at a position (get_interp_weights), stored like the
// reference's COMMON blocks; false when the position is outside the grid.
__device__ __forceinline__ bool locate(const PassArgs& a, long long l, double x, double y, double z, int& i, int& j,
                                       int& k, double (&w)[8]) {
  const PartDev& p = a.p;
  const bool ok = weights_at(a.g, x, y, z, i, j, k, w);
  p.ijk[l] = i;
  p.ijk[l + p.NM] = j;
  p.ijk[l + 2 * p.NM] = k;
#pragma unroll
  for (int c = 0; c < 8; ++c) p.wght[l + c * p.NM] = w[c];
  return ok;
}

// The half move of move_ion_half along one axis with its one wrap (gutsp.f:473-510).
__device__ __forceinline__ double half_move(double x, double v, double dth, double q1, double qn, bool wrap) {
  x = x + dth * v;
  if (wrap) {
    const long long b = ordered_position(x);
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
  if (threadIdx.x == 0) s_bc.set(g, a.beta, p.beta_p[0]);
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
      density_factors(g, a.beta, p.beta_p[l], s_bc, i, j, k, fn, fu);
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
      const double mr = p.mrat[l], dt = a.dt;
      double v[3], E[3];
#pragma unroll
      for (int q = 0; q < 3; ++q) v[q] = p.vp[l + q * NM];
      // (aj - up) x B; Ep is mrat times it (gutsp.f:260-270)
      E[0] = __fma_rn(A[1], B[2], -(A[2] * B[1]));
      E[1] = __fma_rn(A[2], B[0], -(A[0] * B[2]));
      E[2] = __fma_rn(A[0], B[1], -(A[1] * B[0]));
      double h = a.half_dt;
      if (!is_one(mr)) {
        h *= mr;
#pragma unroll
        for (int q = 0; q < 3; ++q) B[q] *= mr;
      }
      // v- and the rotation of get_vplus_vminus (gutsp.f:302-397)
      double vm[3], vn[3];
#pragma unroll
      for (int q = 0; q < 3; ++q) vm[q] = __fma_rn(h, E[q], v[q]);
      const double t = a.quarter_dt2 * __fma_rn(B[0], B[0], __fma_rn(B[1], B[1], B[2] * B[2]));
      const double ad = fast_reciprocal(1.0 + t), om = 1.0 - t;
      const double kd = a.half_dt2 * __fma_rn(vm[0], B[0], __fma_rn(vm[1], B[1], vm[2] * B[2]));
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        const int q1 = (q + 1) % 3, q2 = (q + 2) % 3;
        const double c = __fma_rn(vm[q1], B[q2], -(vm[q2] * B[q1]));
        vn[q] = ad * __fma_rn(kd, B[q], __fma_rn(dt, c, om * vm[q]));
      }
      if (PASS == 2) {  // improve_up (gutsp.f:422)
        const double f = 0.5 * flow_factor(g, a.beta, p.beta_p[l], s_bc, i, j, k);
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
        const bool out = a.x_open && !(ordered_position(x) > ordered(qx1) && ordered_position(x) <= ordered(qxn));
        if (out) {  // removed by the caller; its weights are those of no cell
          p.ijk[l] = p.ijk[l + NM] = p.ijk[l + 2 * NM] = 1;
#pragma unroll
          for (int c = 0; c < 8; ++c) p.wght[l + c * NM] = 0.0;
          live = false;
        } else {
          live = locate(a, l, x, y, z, i, j, k, w);
          if (!live) set_err(a.err, KERR_DOMAIN);
          double fn, fu;
          density_factors(g, a.beta, p.beta_p[l], s_bc, i, j, k, fn, fu);
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
    warp_deposit<PASS != 2>(g, red, live, i, j, k, w, m, a.np, a.S);
  }
}

}  // namespace

cudaError_t particle_pass(int pass, PassArgs a, cudaStream_t st) {
  if (a.N <= 0) return cudaSuccess;
  // four blocks of 128 an SM hide the latencies; more blocks than that at
  // once only repeat the block's set-up
  a.half_dt = 0.5 * a.dt;
  a.quarter_dt2 = 0.25 * a.dt * a.dt;
  a.half_dt2 = 0.5 * a.dt * a.dt;
  const long long need = (a.N + TPB - 1) / TPB, most = 152LL * 4 * 8;
  const unsigned nb = (unsigned)(need < most ? need : most);
  if (pass == 1) k_pass<1><<<nb, TPB, 0, st>>>(a);
  else if (pass == 2) k_pass<2><<<nb, TPB, 0, st>>>(a);
  else k_pass<3><<<nb, TPB, 0, st>>>(a);
  return cudaGetLastError();
}

}  // namespace swapk
