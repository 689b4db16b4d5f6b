// Kept device buffers (device_memory.hpp).
#include "device_memory.hpp"

#include <algorithm>
#include <mutex>
#include <vector>

namespace chsga {

namespace {

// Guards the list and every buffer's fields; never held across a CUDA call
// (cudaFree waits for the device). Both outlive every static object.
std::mutex& mu() {
  static std::mutex& m = *new std::mutex;
  return m;
}
std::vector<KeptBuffer*>& all() {
  static std::vector<KeptBuffer*>& v = *new std::vector<KeptBuffer*>;
  return v;
}

}  // namespace

cudaError_t device_malloc(void** p, size_t bytes) {
  const cudaError_t e = cudaMalloc(p, bytes);
  if (e != cudaErrorMemoryAllocation || !free_kept_buffers()) return e;
  cudaGetLastError();  // the failed attempt's
  return cudaMalloc(p, bytes);
}

bool free_kept_buffers() {
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess) return false;
  std::vector<unsigned char*> gone;
  {
    std::lock_guard<std::mutex> lk(mu());
    gone.reserve(all().size());
    for (KeptBuffer* b : all())
      if (!b->taken_ && b->p_ && b->device_ == device) {
        gone.push_back(b->p_);
        b->p_ = nullptr;
        b->bytes_ = 0;
      }
  }
  for (unsigned char* p : gone) cudaFree(p);
  return !gone.empty();
}

uint64_t kept_bytes(int device) {
  std::lock_guard<std::mutex> lk(mu());
  uint64_t n = 0;
  for (const KeptBuffer* b : all())
    if (!b->taken_ && b->device_ == device) n += b->bytes_;
  return n;
}

KeptBuffer::KeptBuffer() {
  std::lock_guard<std::mutex> lk(mu());
  all().push_back(this);
}

KeptBuffer::~KeptBuffer() {
  {
    std::lock_guard<std::mutex> lk(mu());
    all().erase(std::find(all().begin(), all().end(), this));
  }
  if (p_) cudaFree(p_);
}

cudaError_t KeptBuffer::take(uint64_t bytes, unsigned char** p) {
  unsigned char* small = nullptr;
  {
    std::lock_guard<std::mutex> lk(mu());
    taken_ = true;
    if (p_ && bytes_ < bytes) {
      small = p_;
      p_ = nullptr;
      bytes_ = 0;
    }
  }
  if (small) cudaFree(small);
  if (!p_) {
    const cudaError_t e = device_malloc((void**)&p_, bytes);
    if (e != cudaSuccess) {
      p_ = nullptr;
      put();
      return e;
    }
    bytes_ = bytes;
    cudaGetDevice(&device_);
  }
  *p = p_;
  return cudaSuccess;
}

void KeptBuffer::put() {
  std::lock_guard<std::mutex> lk(mu());
  taken_ = false;
}

void KeptBuffer::drop() {
  unsigned char* p = nullptr;
  {
    std::lock_guard<std::mutex> lk(mu());
    if (taken_) return;
    p = p_;
    p_ = nullptr;
    bytes_ = 0;
  }
  if (p) cudaFree(p);
}

uint64_t KeptBuffer::idle_bytes() const {
  std::lock_guard<std::mutex> lk(mu());
  return taken_ ? 0 : bytes_;
}

}  // namespace chsga
