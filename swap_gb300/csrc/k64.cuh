// k64.cuh -- launchers of the FP64 kernels (k64.cu).  Every launcher enqueues
// on `st` and returns the launch status.  Grids are device arrays in Fortran
// layout (x fastest, component slowest, stride C); particles are (ni_max,3).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "swap_dev.cuh"

namespace swapk {

struct PartDev {  // device mirrors of the particle arrays
  double *xp, *vp, *vp1, *mrat, *beta_p;
  int32_t* ijk;   // (ni_max,3), 1-based cell indices like ijkp
  double* wght;   // (ni_max,8)
  long long NM;   // leading dimension ni_max
};

// Host: the uniform-grid constants and 1/dy of g (nx, ny, nz and dy set) from
// the host's node coordinates and, when given, dx_grid ... (else cell_g = cell_q).
void set_cell_constants(Geo& g, const double* qx, const double* qy, const double* qz, const double* dxg,
                        const double* dyg, const double* dzg);

// boundary.f
cudaError_t periodic3(const Geo& g, double* b, cudaStream_t st);
cudaError_t periodic1(const Geo& g, double* b, cudaStream_t st);

// The field operators (k64_field.cu).  fill: also write the ghost images of
// the operator's B input, which the caller sees filled.  Every grid output
// is stored with its ghost images unless noted.
// curlB: aj at the interior (ghosts untouched); btc (may be null):
// edge_to_center of b at the interior.  den (may be null): face_density's.
cudaError_t curlB(const Geo& g, double* b, const double* np, const double* den, double alpha, double* aj,
                  double* btc, bool fill, cudaStream_t st);
// Per component the face density times alpha and its reciprocal, [6][C], interior.
cudaError_t face_density(const Geo& g, const double* np, double alpha, double* den, cudaStream_t st);
// ct = face_to_center(aj - up) x B at the centres, interior.  corr: b holds
// curlB's btc, averaged to the faces and back; otherwise the edge field.
cudaError_t cross_ct(const Geo& g, bool corr, const double* aj, const double* up, double* b, double* ct, bool fill,
                     cudaStream_t st);
// E = face average of ct + nu*aj (- the electron-pressure gradient).
cudaError_t e_field(const Geo& g, const double* ct, const double* nu, const double* aj, const double* np, double gp,
                    double* E, cudaStream_t st);
// b1p2 = base - coef*curlE (skipped when null); half (may be null) =
// 0.5*(b1p2 + b1) at the interior.
cudaError_t b_advance(const Geo& g, const double* E, const double* base, double coef, double* b1p2, const double* b1,
                      double* half, cudaStream_t st);
// n subcycles of a small grid in one launch (field_loop_fits): as n rounds of
// the launchers above with b1 and b12 changing places after each.  Nothing is
// done when *courant (a double's bits) <= courant_floor: the caller looks too.
constexpr long long FIELD_LOOP_NODES = 5 << 15;
struct FieldLoop64 {
  int n;
  double *bt, *b1, *b12, *half, *btc, *ct, *E, *aj;
  const double *up, *np, *nu, *den;
  double gp, alpha, dtsub;
  const unsigned long long* courant;
  double courant_floor;
  int* err;       // KERR_WAIT when a barrier's wait runs out
  unsigned* bar;  // two counters, zero between launches
  unsigned polls;
};
bool field_loop_fits(const Geo& g);
cudaError_t field_loop(const Geo& g, const FieldLoop64& f, cudaStream_t st);
// out = 0.5*(a + b) at the interior.
cudaError_t half_sum(const Geo& g, const double* a, const double* b, double* out, cudaStream_t st);
cudaError_t edge_to_center(const Geo& g, double* bt, double* btc, cudaStream_t st);
// vc of v, and wc of w (null: v alone); the inputs' ghosts are filled.
cudaError_t face_to_center(const Geo& g, double* v, double* vc, double* w, double* wc, cudaStream_t st);
// up = face average of S/np (zero where np is zero); fill_np: np's ghosts too.
cudaError_t up_from_sums(const Geo& g, const double* S, double* np, double* up, bool fill_np, cudaStream_t st);
// n values from one array to two others.
cudaError_t copy_both(long long n, const double* from, double* a, double* b, cudaStream_t st);
// The particle passes' gather table, [C][6]: face_to_center(aj - up) and, when
// full, edge_to_center(bt), with btc and aj's ghosts.  Clears S and, when given,
// np at the interior nodes, for the next pass's deposit.
cudaError_t gather_kit(const Geo& g, bool full, double* aj, const double* up, const double* bt, double* btc,
                       double* kit, double* S, double* np, cudaStream_t st);

// The Courant time per node, and the bits of the smallest into *least.
cudaError_t deltat_all(const Geo& g, const double* bt, const double* np, double alpha, double dx, double* dtn,
                       unsigned long long* least, cudaStream_t st);
cudaError_t grad_pe_face_int(const Geo& g, const double* np, double grad_pe, double* gf, cudaStream_t st);

// gutsp.f particle operators
cudaError_t interp_weights(const Geo& g, const PartDev& p, long long N, int* err, cudaStream_t st);
// The cells of the first N particles to another ijkp array, unless *err is set.
cudaError_t copy_cells(const PartDev& p, long long N, int32_t* ijkp, const int* err, cudaStream_t st);
// Deterministic deposits: each added value x goes into a 128-bit fixed-point
// sum in units of 2^-60, as floor(x * 2^28) into a signed 64-bit word (h)
// and the rest * 2^32, rounded, into an unsigned one (l).  Integer adds are
// exact and commutative, so the sum does not depend on the order of the
// GPU's atomics; |x| < 2^25 per value (SWAP_ENONFINITE otherwise).
struct Fix64 {
  long long* h;
  unsigned long long* l;
};
// fix (h, l null: plain FP64 atomics into np) ...
cudaError_t deposit_np(const Geo& g, const PartDev& p, long long N, double beta, double* np, int* err,
                       cudaStream_t st, Fix64 fix = Fix64{nullptr, nullptr});
// out[t] = the fixed-point sums (h[t], l[t]) rounded to FP64, t < n.
cudaError_t fix_to_double(long long n, Fix64 fix, double* out, cudaStream_t st);
// mode: 0 = v, 1 = 1.5 v - 0.5 v1 (extrapol_up), 2 = 0.5 (a + b) (improve_up, also stores into out_v1),
// 3 = (v/sqrt(mrat))^2 and 4 = v/sqrt(mrat) per component (get_temperature)
cudaError_t deposit_u(const Geo& g, const PartDev& p, long long N, double beta, int mode, const double* va,
                      const double* vb, double* out_v1, double* S, int* err, cudaStream_t st,
                      Fix64 fix = Fix64{nullptr, nullptr});
// update_rho deposit (folded into the interior), interior scaling, and the
// temperature of get_temperature from the two face moments.
cudaError_t deposit_rho(const Geo& g, const PartDev& p, long long N, double beta, double* mnp, int* err,
                        cudaStream_t st);
cudaError_t scale_interior(const Geo& g, double* f, double a, cudaStream_t st);
cudaError_t temperature(const Geo& g, const double* up2, const double* upa, double mion, double* temp,
                        cudaStream_t st);
cudaError_t get_Ep(const Geo& g, const PartDev& p, long long N, const double* ajc, const double* upc,
                   const double* btc, const double* gpc, double* Ep, int* err, cudaStream_t st);
cudaError_t vplus_vminus(const Geo& g, const PartDev& p, long long N, double dt, const double* Ep,
                         const double* btc, const double* vp, double* vplus, double* vminus, int* err,
                         cudaStream_t st);
cudaError_t vp_final(const PartDev& p, long long N, double dt, const double* Ep, double* vp, double* vp1,
                     const double* vplus, cudaStream_t st);
// x_open: the x axis does not wrap (particles leaving are removed after the
// move by the caller).
cudaError_t move_half(const Geo& g, const PartDev& p, long long N, double dt, double* xp, const double* vp,
                      bool x_open, cudaStream_t st);

// The particle half of a fused step in three passes (k64_pass.cu).
struct PassArgs {
  Geo g;
  PartDev p;
  long long N;
  double dt, beta;
  const double* kit;  // gather_kit's table
  double* b3;         // (ni_max,3): B at each particle, pass 2 to pass 3
  double *np, *S;     // raw deposit sums (zeroed by the caller); pass 2: S alone
  int* err;
  bool x_open;      // pass 3: the x axis does not wrap, and an ion outside deposits nothing
  bool final_move;  // pass 3: also the half move of maind.f:479
  double half_dt, quarter_dt2, half_dt2;  // set by particle_pass
};
cudaError_t particle_pass(int pass, PassArgs a, cudaStream_t st);

// reductions (FP64)
cudaError_t energy_parts(const Geo& g, const PartDev& p, long long N, double beta, double alpha, const double* vp,
                         const double* b0, const double* b1, const double* E, double* d_acc4, cudaStream_t st);
cudaError_t divb_max(const Geo& g, const double* b, double* d_max, cudaStream_t st);
cudaError_t count_nonfinite(const double* x, long long n, unsigned long long* d_cnt, cudaStream_t st);
// A caller's 4-byte reals to the device's doubles (exact) and back (rounded
// to nearest).
cudaError_t widen_f32(const float* in, double* out, long long n, cudaStream_t st);
cudaError_t narrow_f64(const double* in, float* out, long long n, cudaStream_t st);

}  // namespace swapk
