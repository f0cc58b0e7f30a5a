// Constant tables on a device: allocation and upload (host code, any caller's state).
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

// Copies `bytes` from host memory to dst on `device`; the bytes have landed when it returns. A
// plain cudaMemcpy from pageable memory may return while its last part is still under way, and is
// ordered only before work of the legacy stream and of the streams that wait for it, which the
// library's own non-blocking streams and many callers' do not.
//
// upload_table allocates as well; nullptr on failure, with nothing left behind. Both work
// whichever device the calling thread has current, and leave it current; and, except where the
// device is out of memory, also while this or another thread captures a stream (the calls that a
// capture would refuse or be broken by are made in the thread's relaxed mode, on a stream that
// takes no part in it).
namespace bbupload {

struct OnDevice {  // makes `device` current and lifts the capture restrictions of this thread
  int before = -1;
  bool ok, relaxed;
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  explicit OnDevice(int device) {
    ok = cudaGetDevice(&before) == cudaSuccess && cudaSetDevice(device) == cudaSuccess;
    relaxed = ok && cudaThreadExchangeStreamCaptureMode(&mode) == cudaSuccess;
    ok = relaxed;
  }
  ~OnDevice() {
    if (relaxed) cudaThreadExchangeStreamCaptureMode(&mode);
    if (before >= 0) cudaSetDevice(before);
  }
  OnDevice(const OnDevice&) = delete;
  OnDevice& operator=(const OnDevice&) = delete;
};

inline cudaError_t copy_and_wait(void* dst, const void* src, size_t bytes) {
  cudaStream_t st = nullptr;
  cudaError_t e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
  if (e != cudaSuccess) return e;
  e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st);
  const cudaError_t w = cudaStreamSynchronize(st);
  cudaStreamDestroy(st);
  return e != cudaSuccess ? e : w;
}

}  // namespace bbupload

inline cudaError_t upload_bytes(int device, void* dst, const void* src, size_t bytes) {
  bbupload::OnDevice on(device);
  return on.ok ? bbupload::copy_and_wait(dst, src, bytes) : cudaErrorInvalidDevice;
}

inline void* upload_table(int device, const void* src, size_t bytes) {
  bbupload::OnDevice on(device);
  void* d = nullptr;
  if (!on.ok || cudaMalloc(&d, bytes) != cudaSuccess) return nullptr;
  if (bbupload::copy_and_wait(d, src, bytes) != cudaSuccess) {
    cudaFree(d);
    d = nullptr;
  }
  return d;
}
