// A CUDA runtime that launches nothing: it keeps kernel attributes per device, as
// the real one does, and refuses a launch whose shared memory was not asked for
// on its device or whose cooperative grid does not fit it. Linked into
// devices_test in the real one's place.
#include <cuda_runtime_api.h>

#include <map>
#include <utility>

struct FakeDevice {
  int sms, coop, per_sm;
};
extern const FakeDevice fake_devices[4] = {{152, 1, 1}, {20, 1, 1}, {152, 0, 1}, {152, 1, 0}};
int fake_current = 0, fake_refused = 0, fake_launches = 0;

namespace {

std::map<std::pair<int, const void *>, size_t> allowed;
struct Config {
  dim3 grid, block;
  size_t smem;
  cudaStream_t s;
} config;

cudaError_t launch(const void *f, dim3 grid, size_t smem, bool coop) {
  ++fake_launches;
  const auto it = allowed.find({fake_current, f});
  const size_t most = it == allowed.end() ? 48 * 1024 : it->second;
  const FakeDevice &d = fake_devices[fake_current];
  if (smem <= most && !(coop && (!d.coop || grid.x > unsigned(d.per_sm * d.sms)))) return cudaSuccess;
  ++fake_refused;
  return cudaErrorInvalidValue;
}

}  // namespace

extern "C" {
cudaError_t cudaGetDevice(int *d) { *d = fake_current; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int d) {
  *v = a == cudaDevAttrMultiProcessorCount ? fake_devices[d].sms : a == cudaDevAttrCooperativeLaunch ? fake_devices[d].coop : 0;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *f, cudaFuncAttribute, int v) {
  allowed[{fake_current, f}] = size_t(v);
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned) {
  *n = fake_devices[fake_current].per_sm;
  return cudaSuccess;
}
cudaError_t cudaLaunchCooperativeKernel(const void *f, dim3 g, dim3, void **, size_t smem, cudaStream_t) {
  return launch(f, g, smem, true);
}
cudaError_t __cudaLaunchKernel(cudaKernel_t f, dim3 g, dim3, void **, size_t smem, cudaStream_t) {
  return launch(f, g, smem, false);
}
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *f) { *k = (cudaKernel_t)f; return cudaSuccess; }
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, cudaStream_t s) { config = {g, b, smem, s}; return 0; }
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *smem, void *s) {
  *g = config.grid; *b = config.block; *smem = config.smem; *static_cast<cudaStream_t *>(s) = config.s;
  return cudaSuccess;
}
void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
char __cudaInitModule(void **) { return 0; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, uint3 *, uint3 *, dim3 *, dim3 *, int *) {}
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "refused"; }
cudaError_t cudaMemsetAsync(void *, int, size_t, cudaStream_t) { return cudaSuccess; }
}
