// The entries that read a handle's control block, on a machine of several GPUs, against a fake CUDA runtime: a handle on
// device 1 is read by a thread whose current device is 0. A launch is refused on a stream of another device than the
// thread's, as CUDA refuses it; copies and waits are accepted from any. Linked with nsf_capi.cpp alone: what these
// entries do not reach is left unresolved. Prints one line per entry: name, status, device of the thread afterwards.
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "nsf_internal.h"
#include "nsf_solver_impl.h"
#include "nsfsi.h"

static int current = 0;
static const int kStreamDevice = 1;
static cudaError_t last = cudaSuccess;

extern "C" {
cudaError_t cudaGetDevice(int* d) {
  *d = current;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int d) {
  current = d;
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  *p = std::calloc(1, n);
  return cudaSuccess;
}
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned) {
  *d = h;
  return cudaSuccess;
}
cudaError_t cudaGetLastError() {
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemcpy2DAsync(void*, size_t, const void*, size_t, size_t, size_t, cudaMemcpyKind, cudaStream_t) {
  return cudaSuccess;
}
const char* cudaGetErrorString(cudaError_t e) { return e == cudaSuccess ? "ok" : "invalid resource handle"; }
}

namespace nsf {
void launch_ctl_out(const StepCtl* ctl, StepCtl* out, void*) {
  if (current != kStreamDevice)
    last = cudaErrorInvalidResourceHandle;
  else
    std::memcpy(static_cast<void*>(out), ctl, sizeof(StepCtl));
}
}  // namespace nsf

int main() {
  nsf_solver s;
  nsf::StepCtl ctl{};
  ctl.t = 1.5;
  ctl.dt = 0.25;
  ctl.level = 6;
  s.device = kStreamDevice;
  s.dCtl = &ctl;
  s.initialized = true;
  double t = 0, dt = 0, host[1] = {0};
  uint64_t level = 0;
  const int time = nsf_get_time(&s, &t, &level, &dt);
  const bool values = t == 1.5 && dt == 0.25 && level == 6;
  std::printf("nsf_get_time %d %d\n", time == 0 && !values ? -1 : time, current);
  std::printf("nsf_sync %d %d\n", nsf_sync(&s), current);
  std::printf("nsf_upload_conserved %d %d\n", nsf_upload_conserved(&s, host), current);
  return 0;
}
