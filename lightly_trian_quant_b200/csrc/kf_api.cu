// Status plumbing of the C-ABI: thread-local last-error text, CUDA error mapping, version, scale-tensor sizes.
#include <atomic>
#include <cstdarg>
#include <cstdio>

#include "../../include/kf_b200_dev.h"
#include "kf_sm100.cuh"

namespace kf {

static thread_local char g_err[512] = "";

void set_error(const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
}

int cuda_status(cudaError_t e, const char* what) {
  if (e == cudaSuccess) return KF_OK;
  set_error("%s: %s (%s)", what, cudaGetErrorName(e), cudaGetErrorString(e));
  return (int)e;
}

// Programmatic dependent launch is taken where the launches are short: the successor's start-up (about 2 us of launch, barrier and
// tensor-memory set-up) then runs under its predecessor.  Over many rows the successor's CTAs, waiting on the SMs, cost more than that.
// Outside a capture it also hides the launch gaps of the stream, so the line lies higher.  Whole models of 640 px images, change of the time from
// plain to dependent (ViT-B MXFP8 / ViT-L NVFP4 / ViT-B bf16):
//   rows        1605               3210           4815               6420   9630          12 840         16 050        19 260
//   captured    -8.3 -7.3 -2.7 %   -3.2 -1.7 %    -4.2 -1.5 -0.8 %   +1.0   +2.5 +2.6 %   +2.3    +1.0   +3.3 +1.8 %   +4.3 +3.3 +1.9 %
//   eager       -22 -20 -15 %      -12 -11 %      -12 -8.4 -8.8 %    -5.3   -4.2 -2.0 %   -1.1    -2.3   +0.0 +0.4 %   +2.4 +1.7 +0.4 %
// and ViT-B 256 px (261 rows) eager 846 -> 612 us.
constexpr int64_t PDL_ROWS_CAPTURED = 5120, PDL_ROWS_EAGER = 14336;
static std::atomic<int> g_pdl{KF_PDL_AUTO};            // kf_set_pdl
bool pdl_for(int64_t rows, cudaStream_t st) {
  const int mode = g_pdl.load(std::memory_order_relaxed);
  if (mode != KF_PDL_AUTO) return mode == KF_PDL_ALL;
  if (rows <= PDL_ROWS_CAPTURED) return true;
  if (rows > PDL_ROWS_EAGER) return false;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  return cudaStreamIsCapturing(st, &cap) == cudaSuccess && cap == cudaStreamCaptureStatusNone;
}

__device__ unsigned int g_dev_error[4];

unsigned int* dev_error_ptr() {
  static PerDevice<unsigned int*> cached;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
  if (unsigned int* known = cached.get(dev)) return known;
  void* p = nullptr;
  if (cudaGetSymbolAddress(&p, g_dev_error) != cudaSuccess) return nullptr;
  cached.put(dev, static_cast<unsigned int*>(p));
  return static_cast<unsigned int*>(p);
}

// A launch that lets its successor start, takes delay_us and then fails: the error word as a bounded wait that ran out leaves it.
__global__ void raise_error_kernel(unsigned int* err, int delay_us) {
  pdl_launch_dependents();
  for (int i = 0; i < delay_us; ++i) __nanosleep(1000);
  if (atomicCAS(&err[0], 0u, (unsigned)(-KF_ERR_DEVICE_WAIT)) == 0u) err[1] = 200;
}

}  // namespace kf

extern "C" int kf_selftest_raise_error(int delay_us, void* stream) {
  KF_REQUIRE(delay_us >= 0 && delay_us <= 1000, "kf_selftest_raise_error: delay of %d us", delay_us);
  unsigned int* err = kf::dev_error_ptr();
  KF_REQUIRE(err != nullptr, "kf_selftest_raise_error: device error word unavailable");
  kf::raise_error_kernel<<<1, 1, 0, static_cast<cudaStream_t>(stream)>>>(err, delay_us);
  return kf::cuda_status(cudaGetLastError(), "kf_selftest_raise_error launch");
}

extern "C" int kf_check_device_error(void) {
  cudaError_t e = cudaDeviceSynchronize();
  if (e != cudaSuccess) return kf::cuda_status(e, "cudaDeviceSynchronize");
  unsigned int h[4] = {0, 0, 0, 0};
  e = cudaMemcpyFromSymbol(h, kf::g_dev_error, sizeof(h));
  if (e != cudaSuccess) return kf::cuda_status(e, "cudaMemcpyFromSymbol");
  if (h[0] == 0) return KF_OK;
  unsigned int z[4] = {0, 0, 0, 0};
  cudaMemcpyToSymbol(kf::g_dev_error, z, sizeof(z));
  kf::set_error("a bounded device wait ran out: code %u at wait site %u in block %u", h[0], h[1], h[2]);
  return KF_ERR_DEVICE_WAIT;
}

extern "C" int kf_set_pdl(int mode) {
  kf::g_pdl.store(mode == KF_PDL_AUTO || mode == KF_PDL_OFF ? mode : KF_PDL_ALL, std::memory_order_relaxed);
  return KF_OK;
}

extern "C" int kf_pdl_choice(int64_t rows, void* stream) { return kf::pdl_for(rows, static_cast<cudaStream_t>(stream)) ? 1 : 0; }

extern "C" const char* kf_version(void) { return "kf_b200 0.1 sm_100a"; }

extern "C" const char* kf_last_error_string(void) { return kf::g_err; }

extern "C" int64_t kf_sf_bytes(int64_t R, int64_t K, int fmt) {
  if (R < 0 || K <= 0 || (fmt != KF_FMT_MX8 && fmt != KF_FMT_NV4 && fmt != KF_FMT_MX4)) {
    kf::set_error("kf_sf_bytes: bad argument R=%lld K=%lld fmt=%d", (long long)R, (long long)K, fmt);
    return KF_ERR_BAD_ARGUMENT;
  }
  int64_t nkb = K / kf::fmt_vec(fmt);
  return ((R + 127) / 128) * ((nkb + 3) / 4) * 512;
}
