// Device buffers of a context: growth that never loses what it had.
#include <algorithm>

#include "common.hpp"

namespace pwb {

namespace {

// cudaMalloc is forbidden while this thread, or (global mode) any thread,
// captures a stream, unless the calling thread works in relaxed mode; the
// allocation itself does not become part of the graph
struct RelaxedCapture {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
  ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

int device_alloc(void** p, size_t nbytes) {
  const cudaError_t e = cudaMalloc(p, nbytes);
  if (e == cudaSuccess) return PW_OK;
  *p = nullptr;
  cudaGetLastError();     // a later, unrelated check must not report this failure as its own
  set_error(std::string("cudaMalloc failed: ") + cudaGetErrorString(e));
  return PW_ENOMEM;
}

}  // namespace

int DevBuf::alloc(size_t nbytes) {
  if (nbytes <= bytes && p) return PW_OK;
  if (!keep) {
    release();
    if (nbytes == 0) return PW_OK;
    const int rc = device_alloc(&p, nbytes);
    if (!rc) bytes = nbytes;
    return rc;
  }
  if (nbytes == 0) return PW_OK;
  RelaxedCapture guard;
  void* q = nullptr;
  const int rc = device_alloc(&q, nbytes);
  if (rc) return rc;      // the block in use stays in use
  if (p) keep->push_back(p);
  p = q;
  bytes = nbytes;
  return PW_OK;
}

int DevBuf::grow(size_t nbytes) {
  if (nbytes <= bytes && p) return PW_OK;
  if (keep && p && alloc(std::max(nbytes, bytes + bytes / 2)) == PW_OK) return PW_OK;
  return alloc(nbytes);
}

void DevBuf::drop() {
  if (p && keep) {
    keep->push_back(p);
    p = nullptr;
  }
  release();
}

void DevBuf::release() {
  if (p) cudaFree(p);
  p = nullptr;
  bytes = 0;
}

}  // namespace pwb
