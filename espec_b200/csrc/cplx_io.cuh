// cplx_io.cuh -- moving complex arrays between the interface form (separate
// real and imaginary float64 arrays: the reference's U/V and LNZVC columns)
// and the device form (interleaved double2).  Host transfers go through a
// contiguous (re | im) staging block owned by the plan, so each is one linear
// copy; results of up to kStageSmall bytes are written by the kernel straight into
// a page-locked block that the plan holds (HostBlocks) and copied on by the host
// after the caller's synchronisation (a row of a printed table: no device-to-host
// copies, 8 us each); device arguments are (de)interleaved in place by a kernel.
#pragma once
#include <cuda_runtime.h>

#include <cstring>
#include <mutex>

#include "espec_gpu.h"
#include "espec_internal.h"

namespace espec {

constexpr size_t kStageSmall = 64 * 1024;
inline constexpr const char* kPreviousParts =
    "the previous state comes as separate real and imaginary arrays";

// Page-locked blocks of kStageSmall bytes, one for each plan that reads small results;
// a plan holds its block from its first such result until it is destroyed.  Page-locking
// and releasing a block cost 1 to 3 ms, more than a short-lived plan gains (with a block
// of its own, the first result of a new plan took 2.5 ms; 40 us by copies, 20 us through
// a block): all plans share kCount blocks of one allocation, made once and only when
// results have asked kPatience times, by when their copies have cost about as much.  A
// plan that finds no block free has its results copied.
class HostBlocks {
 public:
  static HostBlocks& get() {
    static HostBlocks b;
    return b;
  }
  double* take() {
    std::lock_guard<std::mutex> lock(m_);
    if (!base_ && !allocate()) return nullptr;
    if (!free_) return nullptr;
    int i = 0;
    while (!(free_ >> i & 1)) ++i;
    free_ &= free_ - 1;
    return reinterpret_cast<double*>(base_ + i * kStageSmall);
  }
  void give(double* block) {
    std::lock_guard<std::mutex> lock(m_);
    if (base_) free_ |= 1u << (reinterpret_cast<char*>(block) - base_) / kStageSmall;
  }
  // at the end of the process; plans may still give blocks back afterwards
  ~HostBlocks() {
    if (base_) cudaFreeHost(base_);
    base_ = nullptr;
    asked_ = 0;
  }

 private:
  static constexpr int kCount = 16, kPatience = 64;
  bool allocate() {
    if (++asked_ < kPatience) return false;
    asked_ = 0;
    if (cudaHostAlloc((void**)&base_, kCount * kStageSmall,
                      cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess) {
      (void)cudaGetLastError();
      base_ = nullptr;
      return false;
    }
    free_ = (1u << kCount) - 1;
    return true;
  }
  std::mutex m_;
  char* base_ = nullptr;
  unsigned free_ = 0;  // one bit per block
  int asked_ = 0;
};

struct HostStage {
  double* d = nullptr;
  size_t bytes = 0;
  double* h = nullptr;  // a page-locked block of kStageSmall bytes
  struct Pending {
    double* dst;
    const double* src;
    size_t bytes;
  } pending[4];
  int npending = 0;
  size_t used = 0;  // bytes of h taken by the pending results
  void release() {
    if (d) cudaFree(d);
    if (h) HostBlocks::get().give(h);  // no kernel writes to it: cudaFree has waited
    d = h = nullptr;
    bytes = 0;
  }
  // page-locked space for `size` bytes, or null (too large, or none to be had)
  double* small(size_t size) {
    if (used + size > kStageSmall || npending + 2 > 4) return nullptr;
    if (!h && !(h = HostBlocks::get().take())) return nullptr;
    double* p = h + used / sizeof(double);
    used += size;
    return p;
  }
  void later(double* dst, const double* src, size_t size) {
    if (dst) pending[npending++] = Pending{dst, src, size};
  }
  // before a call's first result, and after its synchronisation
  void drop() {
    npending = 0;
    used = 0;
  }
  void flush() {
    for (int i = 0; i < npending; ++i) std::memcpy(pending[i].dst, pending[i].src, pending[i].bytes);
    drop();
  }
};

namespace {

__global__ void interleave_kernel(const double* re, const double* im, double2* out, size_t n) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    out[i] = make_double2(re[i], im ? im[i] : 0.0);
}

__global__ void deinterleave_kernel(const double2* in, double* re, double* im, size_t n) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    const double2 v = in[i];
    if (re) re[i] = v.x;
    if (im) im[i] = v.y;
  }
}

inline unsigned io_blocks(size_t n) {
  const size_t b = (n + 255) / 256;
  return (unsigned)(b < 148 * 16 ? (b > 0 ? b : 1) : 148 * 16);
}

#define IO_CK(call)                                          \
  do {                                                       \
    cudaError_t e_ = (call);                                 \
    if (e_ != cudaSuccess) return set_cuda_error(#call, e_); \
  } while (0)

inline int stage_reserve(HostStage& s, size_t bytes) {
  if (s.bytes >= bytes) return ESPEC_OK;
  // the device block alone: results of this call may be pending in s.h
  if (s.d) cudaFree(s.d);
  s.d = nullptr;
  s.bytes = 0;
  IO_CK(cudaMalloc(&s.d, bytes));
  s.bytes = bytes;
  return ESPEC_OK;
}

// a user pointer in host memory (synchronous or in-flight copies)
inline bool on_host(int where) { return where == ESPEC_MEM_HOST || where == ESPEC_MEM_HOST_ASYNC; }

inline cudaMemoryType memory_type(const void* p) {
  cudaPointerAttributes at{};
  if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
    (void)cudaGetLastError();
    return cudaMemoryTypeUnregistered;
  }
  return at.type;
}
// ESPEC_MEM_HOST: the caller may reuse its array once the call returns; a copy from
// memory that CUDA knows of (page-locked) is then still in flight
inline int wait_source(const void* p, int where, cudaStream_t st) {
  if (where == ESPEC_MEM_HOST && memory_type(p) != cudaMemoryTypeUnregistered)
    IO_CK(cudaStreamSynchronize(st));
  return ESPEC_OK;
}

// dst (device, n complex) <- (re, im) at `where`; im may be null (zero)
inline int put_complex(HostStage& s, double2* dst, const double* re, const double* im, size_t n,
                       int where, cudaStream_t st) {
  if (n == 0) return ESPEC_OK;
  if (on_host(where)) {
    const int rc = stage_reserve(s, 16 * n);
    if (rc) return rc;
    IO_CK(cudaMemcpyAsync(s.d, re, 8 * n, cudaMemcpyHostToDevice, st));
    if (im) IO_CK(cudaMemcpyAsync(s.d + n, im, 8 * n, cudaMemcpyHostToDevice, st));
    re = s.d;
    im = im ? s.d + n : nullptr;
  }
  interleave_kernel<<<io_blocks(n), 256, 0, st>>>(re, im, dst, n);
  IO_CK(cudaGetLastError());
  return ESPEC_OK;
}

// (re, im) at `where` <- src (device, n complex); either output may be null.
// ESPEC_MEM_HOST: complete once the caller has synchronised the stream and
// called s.flush()
inline int get_complex(HostStage& s, const double2* src, double* re, double* im, size_t n,
                       int where, cudaStream_t st) {
  if ((!re && !im) || n == 0) return ESPEC_OK;
  if (!on_host(where)) {
    deinterleave_kernel<<<io_blocks(n), 256, 0, st>>>(src, re, im, n);
    IO_CK(cudaGetLastError());
    return ESPEC_OK;
  }
  // (device pointers given as host memory are left to the copies below, which take them)
  if (where == ESPEC_MEM_HOST && memory_type(re) != cudaMemoryTypeDevice &&
      memory_type(im) != cudaMemoryTypeDevice) {
    if (double* p = s.small(16 * n)) {
      deinterleave_kernel<<<io_blocks(n), 256, 0, st>>>(src, p, p + n, n);
      IO_CK(cudaGetLastError());
      s.later(re, p, 8 * n);
      s.later(im, p + n, 8 * n);
      return ESPEC_OK;
    }
  }
  const int rc = stage_reserve(s, 16 * n);
  if (rc) return rc;
  deinterleave_kernel<<<io_blocks(n), 256, 0, st>>>(src, s.d, s.d + n, n);
  IO_CK(cudaGetLastError());
  if (re) IO_CK(cudaMemcpyAsync(re, s.d, 8 * n, cudaMemcpyDeviceToHost, st));
  if (im) IO_CK(cudaMemcpyAsync(im, s.d + n, 8 * n, cudaMemcpyDeviceToHost, st));
  return ESPEC_OK;
}

// interleaved user arrays (ESPEC_MEM_INTERLEAVED): one copy as they lie
inline int put_pairs(double2* dst, const double* src, size_t n, int where, cudaStream_t st) {
  if (n == 0) return ESPEC_OK;
  IO_CK(cudaMemcpyAsync(dst, src, 16 * n,
                        on_host(where) ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice, st));
  return wait_source(src, where, st);
}
inline int get_pairs(const double2* src, double* dst, size_t n, int where, cudaStream_t st) {
  if (!dst || n == 0) return ESPEC_OK;
  IO_CK(cudaMemcpyAsync(dst, src, 16 * n,
                        on_host(where) ? cudaMemcpyDeviceToHost : cudaMemcpyDeviceToDevice, st));
  return ESPEC_OK;
}

#undef IO_CK

}  // namespace
}  // namespace espec
