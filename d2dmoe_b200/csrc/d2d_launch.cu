// Facts of the current device that the launchers need on every call.
#include <mutex>

#include "d2d_common.cuh"

namespace d2d {
namespace {

constexpr int MAX_DEVICES = 64, MAX_KERNELS = 64;
struct OptIn {
  const void* kernel;
  size_t smem;
};
struct DeviceFacts {
  int sms = 0;
  int n = 0;
  OptIn optin[MAX_KERNELS];      // largest dynamic shared memory opted in, per kernel
};
DeviceFacts g_dev[MAX_DEVICES];
std::mutex g_dev_lock;

}  // namespace

// The opt-in (cudaFuncSetAttribute) holds for the current device only, as does the SM count.  kernel null: only that
// count.
int device_launch_facts(const void* kernel, size_t smem, int* sms) {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAX_DEVICES) {
    cudaGetLastError();
    return D2D_ERR_NO_DEVICE;
  }
  std::lock_guard<std::mutex> hold(g_dev_lock);
  DeviceFacts& f = g_dev[dev];
  if (f.sms == 0 &&
      (cudaDeviceGetAttribute(&f.sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
       f.sms <= 0)) {
    cudaGetLastError();
    f.sms = 0;
    return D2D_ERR_NO_DEVICE;
  }
  if (sms) *sms = f.sms;
  if (!kernel) return D2D_OK;
  int i = 0;
  while (i < f.n && f.optin[i].kernel != kernel) ++i;
  if (i == f.n || f.optin[i].smem < smem) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
        cudaSuccess) {
      cudaGetLastError();
      return D2D_ERR_LAUNCH;
    }
    if (i == f.n && f.n < MAX_KERNELS) ++f.n;
    if (i < f.n) f.optin[i] = {kernel, smem};
  }
  return D2D_OK;
}

}  // namespace d2d
