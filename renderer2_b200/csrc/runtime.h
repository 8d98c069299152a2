// Host runtime pieces shared by the filter and the path tracer: status codes
// (the C ABI returns them; no exception crosses it), an owning device buffer,
// and CUDA error plumbing.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <string>
#include <utility>
#include <vector>

#include "../../include/r2.h"

namespace r2 {

// Error carried inside the C++ runtime; the C ABI converts it to r2_status and
// records the message for r2_last_error().
struct Error {
  r2_status code;
  std::string msg;
};

void set_last_error(const std::string& msg);

#define R2_CUDA(call)                                                                    \
  do {                                                                                   \
    cudaError_t e_ = (call);                                                             \
    if (e_ != cudaSuccess) {                                                             \
      throw ::r2::Error{e_ == cudaErrorMemoryAllocation ? R2_ERR_OUT_OF_MEMORY            \
                                                         : R2_ERR_DEVICE,                \
                        std::string(#call) + ": " + cudaGetErrorString(e_)};             \
    }                                                                                    \
  } while (0)

#define R2_REQUIRE(cond, code, text)                       \
  do {                                                     \
    if (!(cond)) throw ::r2::Error{(code), std::string(text)}; \
  } while (0)

// Device buffer: an allocation of its own (cudaMalloc / cudaFree), or a part of
// another one (reserve_together).
template <typename T>
class DBuf {
 public:
  DBuf() = default;
  explicit DBuf(size_t n) { alloc(n); }
  ~DBuf() { release(); }
  DBuf(const DBuf&) = delete;
  DBuf& operator=(const DBuf&) = delete;
  DBuf(DBuf&& o) noexcept : p_(o.p_), n_(o.n_), part_(o.part_) { o.p_ = nullptr; o.n_ = 0; }
  DBuf& operator=(DBuf&& o) noexcept {
    if (this != &o) { release(); p_ = o.p_; n_ = o.n_; part_ = o.part_; o.p_ = nullptr; o.n_ = 0; }
    return *this;
  }
  void alloc(size_t n) {
    release();
    if (n == 0) return;
    const cudaError_t e = cudaMalloc((void**)&p_, n * sizeof(T));
    if (e != cudaSuccess) {
      p_ = nullptr;
      cudaGetLastError();  // reported here, not by the next launch as well
    }
    R2_CUDA(e);
    n_ = n;
  }
  // Grow-only reallocation (contents are not preserved).
  void reserve(size_t n) { if (n > n_) alloc(n); }
  // Grows to a power of two at least n, so that buffers reused for jobs of
  // varying size reallocate rarely (each cudaFree/cudaMalloc waits for the device).
  void reserve_grow(size_t n) {
    if (n <= n_) return;
    size_t c = 1;
    while (c < n) c <<= 1;
    alloc(c);
  }
  void release() {
    if (p_ && !part_) cudaFree(p_);
    p_ = nullptr;
    n_ = 0;
    part_ = false;
  }
  // Becomes the n elements at p of an allocation that outlives this.
  void view(T* p, size_t n) {
    release();
    p_ = p;
    n_ = n;
    part_ = true;
  }
  void upload(const T* h, size_t n, cudaStream_t s) {
    reserve(n);
    if (n) R2_CUDA(cudaMemcpyAsync(p_, h, n * sizeof(T), cudaMemcpyHostToDevice, s));
  }
  void download(T* h, size_t n, cudaStream_t s) const {
    if (n) R2_CUDA(cudaMemcpyAsync(h, p_, n * sizeof(T), cudaMemcpyDeviceToHost, s));
  }
  T* get() const { return p_; }
  size_t size() const { return n_; }
  size_t bytes() const { return n_ * sizeof(T); }

 private:
  T* p_ = nullptr;
  size_t n_ = 0;
  bool part_ = false;
};

// Gives each buffer at least its number of elements, all of them as parts of
// one allocation (contents are not preserved) unless every one is large enough
// already.  No buffer shrinks, so users that ask for different parts by turns
// allocate once.  An allocation costs about 0.4 ms and its release 0.3 ms whatever
// the size, and a BVH build wants twenty buffers.
template <typename T>
struct DPart {
  DBuf<T>* buf;
  size_t n;
};
template <typename T>
DPart<T> part(DBuf<T>& b, size_t n) { return DPart<T>{&b, n}; }
template <typename... Ts>
void reserve_together(DBuf<uint8_t>& mem, DPart<Ts>... parts) {
  const bool enough = (... && (parts.buf->size() >= parts.n));
  if (enough) return;
  ((parts.n = parts.n > parts.buf->size() ? parts.n : parts.buf->size()), ...);
  const auto bytes = [](auto& p) { return (p.n * sizeof(*p.buf->get()) + 255) / 256 * 256; };
  (parts.buf->release(), ...);
  mem.alloc((size_t(0) + ... + bytes(parts)));
  size_t at = 0;
  const auto place = [&](auto& p) {
    p.buf->view(reinterpret_cast<decltype(p.buf->get())>(mem.get() + at), p.n);
    at += bytes(p);
  };
  (place(parts), ...);
}

inline int sm_count() {
  static int n = 0;
  if (n == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n <= 0) n = 148;
  }
  return n;
}

}  // namespace r2
