// Device memory a context keeps between calls, and allocation that takes it
// back. A kept buffer saves a call the mapping of its memory; nothing but that
// depends on it, so it gives way to every other allocation of the process on
// its device.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace chsga {

// cudaMalloc on the current device; where the device has no room, once more
// after freeing the idle kept buffers there.
cudaError_t device_malloc(void** p, size_t bytes);

// Frees the idle kept buffers of the current device; whether there were any.
bool free_kept_buffers();

// Bytes of the idle kept buffers of a device.
uint64_t kept_bytes(int device);

// One kept buffer. Its owner takes it for a call and puts it back; while it is
// put back, any thread may free it.
class KeptBuffer {
 public:
  KeptBuffer();
  ~KeptBuffer();  // not while taken
  KeptBuffer(const KeptBuffer&) = delete;
  KeptBuffer& operator=(const KeptBuffer&) = delete;
  // At least `bytes` on the current device, contents undefined.
  cudaError_t take(uint64_t bytes, unsigned char** p);
  void put();
  // Frees it, unless it is taken.
  void drop();
  uint64_t idle_bytes() const;

 private:
  friend bool free_kept_buffers();
  friend uint64_t kept_bytes(int device);
  unsigned char* p_ = nullptr;
  uint64_t bytes_ = 0;
  int device_ = 0;
  bool taken_ = false;
};

}  // namespace chsga
