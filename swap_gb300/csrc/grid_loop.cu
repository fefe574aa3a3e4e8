// grid_loop.cu -- the launch of a kernel whose blocks meet at barriers.
#include "grid_loop.cuh"

#include <mutex>

namespace loop {

namespace {

constexpr int kMaxDevices = 64;
std::mutex g_mu;
cudaEvent_t g_last[kMaxDevices] = {};  // the latest loop queued on each device

}  // namespace

cudaError_t launch(const void* kernel, long long blocks, int threads, void** args, cudaStream_t st) {
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
  // the lock orders wait, launch and record of one loop against another's, on
  // whichever thread and stream
  std::lock_guard<std::mutex> lk(g_mu);
  cudaEvent_t& last = g_last[dev];
  if (last) e = cudaStreamWaitEvent(st, last, 0);
  else e = cudaEventCreateWithFlags(&last, cudaEventDisableTiming);
  if (e != cudaSuccess) return e;
  e = cudaLaunchCooperativeKernel(kernel, dim3((unsigned)(blocks < sms ? blocks : sms)), dim3((unsigned)threads),
                                  args, 0, st);
  if (e != cudaSuccess) return e;
  return cudaEventRecord(last, st);
}

}  // namespace loop
