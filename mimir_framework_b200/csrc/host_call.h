// host_call.h — helpers of the synchronous host-pointer entry points (copy in, run, copy out).
#pragma once

#include <vector>

#include "ops.h"

namespace mb {

// Device buffers of one host-pointer call, from the pool of idle buffers; back to it when the call returns (freed, which
// waits for the device, when the call failed before it had synchronised).
struct Temps {
  std::vector<TempBuffer> bufs;
  ErrorWatch errors;
  bool synced = false;
  ~Temps() {
    for (auto& b : bufs) temp_free(b, synced);
  }
  int alloc(void** p, size_t bytes, const char* tag) {
    TempBuffer b;
    MB_TRY(temp_alloc(&b, bytes ? bytes : 4, tag));
    *p = b.p;
    bufs.push_back(b);
    return MIMIR_B200_OK;
  }
  int upload(const float** dev, const float* host, size_t n, const char* tag) {
    void* p;
    MB_TRY(alloc(&p, n * sizeof(float), tag));
    MB_TRY(copy_to_device(p, host, n * sizeof(float), nullptr));
    *dev = static_cast<const float*>(p);
    return MIMIR_B200_OK;
  }
  int out(float** dev, size_t n, const char* tag) {
    void* p;
    MB_TRY(alloc(&p, n * sizeof(float), tag));
    *dev = static_cast<float*>(p);
    return MIMIR_B200_OK;
  }
};

// The last step of a call: result to the host, one synchronisation, device error word.
inline int finish_download(Temps& t, float* host, const float* dev, size_t n) {
  MB_TRY(t.errors.enqueue(nullptr));
  MB_TRY(copy_to_host(host, dev, n * sizeof(float), nullptr));
  MB_CUDA(cudaStreamSynchronize(nullptr));
  t.synced = true;
  return t.errors.read(nullptr);
}

#define MB_REQUIRE_INIT() \
  if (!ctx().initialised) return fail(MIMIR_B200_E_NOT_INIT, "mimir_b200_init has not been called")


}  // namespace mb
