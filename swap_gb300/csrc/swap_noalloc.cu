// swap_noalloc.cu -- swap_update_up_noalloc: the update_up moment deposit
// (gutsp.f:1649-1842) for callers that cannot allocate device memory.
//
// Who needs it: callers that cannot call cudaMalloc.  One is a host whose
// device memory belongs to another allocator -- for example a process in
// which a framework's caching allocator has already reserved the GPU's
// memory, so a direct cudaMalloc fails or fragments that pool.  Another is a
// caller driving its own asynchronous pipeline on several streams: cudaMalloc
// and cudaFree can synchronize the whole device, every stream of it, which
// such a caller cannot afford inside its time step.  (This entry waits only
// for the one stream it is given: it returns after that stream has finished
// its work, to read the out-of-grid flag.)  Neither caller can create a
// swap_ctx, because swap_init allocates the device mirrors and scratch.  This
// entry takes the caller's own device arrays for every input and output and
// keeps its one scratch array -- the grid coordinates and the per-node
// velocity sums -- in a file-scope __device__ array instead.
//
// Properties:
//  * scratch is static: every GPU that loads this library holds it
//    (SWAP_NOALLOC_SCRATCH_BYTES) until the process exits;
//  * no call can be captured in a CUDA graph: every call reads the flag back
//    and waits for its stream, which a capture does not allow;
//  * the first call on a device looks up the scratch address with
//    cudaGetSymbolAddress (no allocation) and keeps it for the process; do
//    not call the entry again on a device after cudaDeviceReset on it (the
//    module is loaded anew and the kept address is stale);
//  * all calls share the scratch, so calls that overlap on the GPU (two
//    streams, two threads) race; serialize them.  After an error the entry
//    waits for its stream before it returns, so no work of the failed call
//    is still running when the caller tries again;
//  * sizes beyond SWAP_NOALLOC_MAX_NODES nodes or SWAP_NOALLOC_MAX_AXIS
//    nodes on an axis are rejected with SWAP_ECAPACITY.
//
// The cell search, weights and fold are the FP64 drop-in's own
// (k64_dev.cuh), and the unit is compiled with --fmad=false like it, so the
// result equals swap_update_up up to the order of the atomic sums.
#include <cstdint>
#include <mutex>

#include <cuda_runtime.h>

#include "../../include/swap_gpu.h"
#include "k64.cuh"
#include "k64_dev.cuh"

namespace {

constexpr long long kMaxNodes = SWAP_NOALLOC_MAX_NODES;
constexpr int kMaxAxis = SWAP_NOALLOC_MAX_AXIS;
constexpr long long kGeoLen = kMaxAxis + 1;  // 1-based node coordinates
// layout: qx | qy | qz (each kGeoLen, 1-based) | S (3 * kMaxNodes)
constexpr long long kScratchDoubles = 3 * kGeoLen + 3 * kMaxNodes;
static_assert(kScratchDoubles * 8 == SWAP_NOALLOC_SCRATCH_BYTES, "header size out of date");

static __device__ __align__(256) double g_scratch[kScratchDoubles];
static __device__ int g_flag;

constexpr int kMaxDevices = 64;
std::mutex g_mu;
double* g_scratch_addr[kMaxDevices] = {};
int* g_flag_addr[kMaxDevices] = {};

// Once per device, with that device current: resolve the device addresses
// of the static scratch and flag.  Host code may not use the symbols
// themselves as addresses (they are host-side stand-ins).
int setup(double** scratch, int** flag) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return SWAP_ECUDA;
  std::lock_guard<std::mutex> lk(g_mu);
  if (!g_scratch_addr[dev]) {
    void* s = nullptr;
    void* f = nullptr;
    if (cudaGetSymbolAddress(&s, g_scratch) != cudaSuccess) return SWAP_ECUDA;
    if (cudaGetSymbolAddress(&f, g_flag) != cudaSuccess) return SWAP_ECUDA;
    g_scratch_addr[dev] = static_cast<double*>(s);
    g_flag_addr[dev] = static_cast<int*>(f);
  }
  *scratch = g_scratch_addr[dev];
  *flag = g_flag_addr[dev];
  return SWAP_OK;
}

using swapk::Geo;

// Weights (gutsp.f:1414-1429) and the update_up deposit (gutsp.f:1676-1800)
// into S = sum v*w/volb at folded nodes, a warp's ions summed by cell first:
// bound by the FP64 pipe (about 75 operations an ion) instead of by the L2
// reductions of 24 values an ion.  3.9M ions, 96x80x64 cells, the whole call:
// 0.93 -> 0.55 ms.
__global__ void __launch_bounds__(128, 6) k_na_deposit(Geo g, const double* __restrict__ xp,
                                                       const double* __restrict__ vp,
                                                       const double* __restrict__ beta_p, long long N, long long NM,
                                                       double beta, double* __restrict__ S, int* flag) {
  __shared__ swapk::Red s_red[4];
  __shared__ swapk::BlockConst s_bc;
  if (threadIdx.x == 0) s_bc.set(g, beta, beta_p[0]);
  __syncthreads();
  const long long l = blockIdx.x * 128LL + threadIdx.x;
  bool live = l < N;
  int i = 1, j = 1, k = 1;
  double w[8], m[4];
  if (live) {
    live = swapk::weights_at(g, xp[l], xp[l + NM], xp[l + 2 * NM], i, j, k, w);
    if (!live) swapk::set_err(flag, SWAP_EDOMAIN);
    const double fu = swapk::flow_factor(g, beta, beta_p[l], s_bc, i, j, k);
    for (int q = 0; q < 3; ++q) m[1 + q] = vp[l + q * NM] * fu;
  }
  swapk::warp_deposit<false>(g, s_red[threadIdx.x >> 5], live, i, j, k, w, m, nullptr, S);
}

}  // namespace

extern "C" int swap_update_up_noalloc(const swap_dims* dims, const swap_params* params, const swap_coords* coords,
                                      const double* xp, const double* vp, const double* beta_p, int64_t ni_tot,
                                      const double* np, double* up, void* stream) {
  if (!dims || !params || !coords || !coords->qx || !coords->qy || !coords->qz || !np || !up) return SWAP_EINVAL;
  if (ni_tot < 0 || ni_tot > dims->ni_max || (ni_tot > 0 && (!xp || !vp || !beta_p))) return SWAP_EINVAL;
  if (dims->nx < 3 || dims->ny < 3 || dims->nz < 3) return SWAP_EINVAL;
  const long long C = (long long)dims->nx * dims->ny * dims->nz;
  if (dims->nx > kMaxAxis || dims->ny > kMaxAxis || dims->nz > kMaxAxis || C > kMaxNodes) return SWAP_ECAPACITY;
  double* scratch = nullptr;
  int* flag = nullptr;
  int r = setup(&scratch, &flag);
  if (r) return r;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  double* qx = scratch;
  double* qy = scratch + kGeoLen;
  double* qz = scratch + 2 * kGeoLen;
  double* S = scratch + 3 * kGeoLen;
  // The scratch keeps the previous call's contents: load this call's
  // geometry and clear the sums and the flag.  Once anything is queued, an
  // error waits for the stream before returning (see the file's notes).
  auto fail_after_enqueue = [st]() {
    cudaStreamSynchronize(st);
    return SWAP_ECUDA;
  };
  if (cudaMemcpyAsync(qx + 1, coords->qx, dims->nx * sizeof(double), cudaMemcpyHostToDevice, st) != cudaSuccess ||
      cudaMemcpyAsync(qy + 1, coords->qy, dims->ny * sizeof(double), cudaMemcpyHostToDevice, st) != cudaSuccess ||
      cudaMemcpyAsync(qz + 1, coords->qz, dims->nz * sizeof(double), cudaMemcpyHostToDevice, st) != cudaSuccess ||
      cudaMemsetAsync(S, 0, 3 * C * sizeof(double), st) != cudaSuccess ||
      cudaMemsetAsync(flag, 0, sizeof(int), st) != cudaSuccess)
    return fail_after_enqueue();
  Geo g{};
  g.nx = dims->nx; g.ny = dims->ny; g.nz = dims->nz;
  g.C = C;
  g.qx = qx; g.qy = qy; g.qz = qz;
  g.dy = params->dy;
  g.inv_dx = 1.0 / (coords->qx[1] - coords->qx[0]);
  g.inv_dz = 1.0 / (coords->qz[1] - coords->qz[0]);
  swapk::set_cell_constants(g, coords->qx, coords->qy, coords->qz, nullptr, nullptr, nullptr);
  if (ni_tot > 0) {
    const long long blocks = (ni_tot + 127) / 128;
    if (blocks > 0x7fffffffLL) return fail_after_enqueue();  // the unsigned conversion must not wrap
    k_na_deposit<<<(unsigned)blocks, 128, 0, st>>>(g, xp, vp, beta_p, ni_tot, dims->ni_max, params->beta, S, flag);
    if (cudaGetLastError() != cudaSuccess) return fail_after_enqueue();
  }
  // the face average of S/np (gutsp.f:1825-1839) with up's ghosts; np is only read
  if (swapk::up_from_sums(g, S, const_cast<double*>(np), up, false, st) != cudaSuccess) return fail_after_enqueue();
  int hflag = 0;
  if (cudaMemcpyAsync(&hflag, flag, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess)
    return fail_after_enqueue();
  if (cudaStreamSynchronize(st) != cudaSuccess) return SWAP_ECUDA;
  return hflag ? SWAP_EDOMAIN : SWAP_OK;
}
