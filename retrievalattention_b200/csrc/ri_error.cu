// Per-thread last-error message, library version, and the status word that kernels report device-side failures in.
#include <stdarg.h>
#include <stdio.h>

#include <mutex>

#include "ri_common.cuh"

static thread_local char g_last_error[512] = "";

int ri_fail(int status, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_last_error, sizeof(g_last_error), fmt, ap);
  va_end(ap);
  return status;
}

extern "C" const char* ri_last_error(void) { return g_last_error; }

extern "C" int ri_version(void) { return 1; }

// Page-locked and mapped for every GPU, so one word serves all devices and streams, a captured call needs no memory of its
// graph, and the host reads it without a copy.  Allocating is allowed while a stream is captured only in relaxed mode.
extern "C" int32_t* ri_status_word(void) {
  static std::mutex lock;
  static int32_t* word = nullptr;
  std::lock_guard<std::mutex> hold(lock);
  if (!word) {
    void* p = nullptr;
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    cudaError_t e = cudaThreadExchangeStreamCaptureMode(&mode);
    if (e == cudaSuccess) {
      e = cudaHostAlloc(&p, sizeof(int32_t), cudaHostAllocPortable | cudaHostAllocMapped);
      cudaThreadExchangeStreamCaptureMode(&mode);
    }
    if (e != cudaSuccess) {
      cudaGetLastError();
      ri_fail(RI_ERR_CUDA, "no page-locked memory for the status word: %s", cudaGetErrorString(e));
      return nullptr;
    }
    *static_cast<int32_t*>(p) = 0;
    word = static_cast<int32_t*>(p);
  }
  return word;
}
