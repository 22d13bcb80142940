// Shared definitions of the GB300 SIMP library: status codes, errors, device
// buffers and launch accounting.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>
#include <cstring>
#include <stdexcept>
#include <string>
#include <utility>
#include <vector>

namespace simp {

using i32 = int32_t;
using i64 = int64_t;

enum Status : int {
  kOk = 0,
  kBadInput = 1,
  kBreakdown = 2,
  kUnderConstrained = 3,
  kMaxIter = 4,
  kNonFinite = 5,
  kCudaError = 6
};

struct Error : std::runtime_error {
  int code;
  Error(int c, const std::string& m) : std::runtime_error(m), code(c) {}
};

#define SIMP_CUDA(expr)                                                                   \
  do {                                                                                    \
    cudaError_t e_ = (expr);                                                              \
    if (e_ != cudaSuccess)                                                                \
      throw ::simp::Error(::simp::kCudaError, std::string(#expr) + ": " + cudaGetErrorString(e_)); \
  } while (0)

// Kernel launches are counted (the library's own kernels only); the
// per-thread count lets a stream capture tell how many kernels it recorded.
extern std::atomic<int64_t> g_launches;
extern thread_local int64_t t_launches;
#define SIMP_LAUNCHED() (++::simp::t_launches, ::simp::g_launches.fetch_add(1, std::memory_order_relaxed))
#define SIMP_CHECK_LAUNCH()             \
  do {                                  \
    SIMP_LAUNCHED();                    \
    SIMP_CUDA(cudaGetLastError());      \
  } while (0)

// SMs of a GB300, where a rule that was measured on one counts blocks, nodes or
// CTAs for each of them.
constexpr int kSms = 152;

// Launch of a kernel whose first statement is chain_start() (kernels.cuh): it
// may be scheduled while the stream's previous kernel drains, and waits there,
// before its first access, until that kernel has completed.  The CG iteration,
// the Lanczos runs and the coarse sweep are chains of kernels of a few
// microseconds each, where the time from one kernel's end to the next one's
// start is a third of the total.  ChainOff turns the overlap off for the
// launches of its scope on the calling thread (bodies of conditional graph
// nodes).
extern thread_local int t_chain_off;
struct ChainOff {
  ChainOff() { ++t_chain_off; }
  ~ChainOff() { --t_chain_off; }
};

template <class... K, class... A>
void chain_launch(void (*kernel)(K...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = &at;
  cfg.numAttrs = t_chain_off ? 0 : 1;
  SIMP_CUDA(cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...));
}

// Owning device array (move-only).
template <class T>
struct DBuf {
  T* p = nullptr;
  size_t n = 0;
  DBuf() = default;
  explicit DBuf(size_t count) { alloc(count); }
  DBuf(const DBuf&) = delete;
  DBuf& operator=(const DBuf&) = delete;
  DBuf(DBuf&& o) noexcept : p(o.p), n(o.n) { o.p = nullptr; o.n = 0; }
  DBuf& operator=(DBuf&& o) noexcept {
    if (this != &o) { release(); p = o.p; n = o.n; o.p = nullptr; o.n = 0; }
    return *this;
  }
  ~DBuf() { release(); }
  void release() {
    if (p) cudaFree(p);
    p = nullptr;
    n = 0;
  }
  void alloc(size_t count) {
    if (count == n && p) return;
    release();
    if (count) SIMP_CUDA(cudaMalloc(&p, count * sizeof(T)));
    n = count;
  }
  void upload(const T* h, size_t count, cudaStream_t s = 0) {
    alloc(count);
    if (count) SIMP_CUDA(cudaMemcpyAsync(p, h, count * sizeof(T), cudaMemcpyHostToDevice, s));
  }
  void upload(const std::vector<T>& h, cudaStream_t s = 0) { upload(h.data(), h.size(), s); }
  void download(T* h, size_t count, cudaStream_t s = 0) const {
    if (count) SIMP_CUDA(cudaMemcpyAsync(h, p, count * sizeof(T), cudaMemcpyDeviceToHost, s));
  }
  std::vector<T> to_host(cudaStream_t s = 0) const {
    std::vector<T> h(n);
    download(h.data(), n, s);
    SIMP_CUDA(cudaStreamSynchronize(s));
    return h;
  }
  void zero(cudaStream_t s = 0) {
    if (n) SIMP_CUDA(cudaMemsetAsync(p, 0, n * sizeof(T), s));
  }
  size_t bytes() const { return n * sizeof(T); }
};

// Owning page-locked host array (copies to and from it do not pass through the
// driver's staging).
template <class T>
struct PinnedBuf {
  T* p = nullptr;
  size_t n = 0;
  PinnedBuf() = default;
  PinnedBuf(const PinnedBuf&) = delete;
  PinnedBuf& operator=(const PinnedBuf&) = delete;
  ~PinnedBuf() {
    if (p) cudaFreeHost(p);
  }
  void alloc(size_t count) {
    if (p && count <= n) return;
    if (p) cudaFreeHost(p);
    p = nullptr;
    n = 0;
    SIMP_CUDA(cudaMallocHost(&p, count * sizeof(T)));
    n = count;
  }
};

// Scalars of a PCG solve in device memory (kernels.cuh).
struct PcgScalars {
  double rz;        // r^T z of the current direction
  double pq;        // p^T A p
  double alpha, beta;
  double rr;        // ||r||^2 after the update
  int status;       // 0 ok, 2 breakdown (p^T A p <= 0 or non-finite)
  int fresh;        // 1: the next direction starts a CG run (beta = 0)
  unsigned ticket;  // grid_sum's
  unsigned seq;     // posts to the host so far
};

// What the host reads after an iteration, in page-locked memory that the last
// block of the update writes: the host polls seq instead of copying and
// synchronising.
struct PcgPost {
  double rr, pq;
  int status;
  unsigned seq;
};

// Sums that a kernel's last block leaves in page-locked memory for the host.
struct SumPost {
  static constexpr int kValues = 7;
  double v[kValues];
  unsigned seq;
};

// Polls a post until it shows `value`.  A fault of the stream, or its end
// without the post, becomes an error.
void wait_for_post(const volatile unsigned* seq, unsigned value, cudaStream_t stream);

// Raises a kernel's dynamic shared-memory limit to at least `bytes` and never
// lowers it: the limit is one value per kernel, shared by every host thread,
// so a thread that set a smaller value could make another thread's larger
// launch fail between its set and its launch.
void raise_dynamic_smem(const void* kernel, size_t bytes);

// dst = a device copy of src (same length)
template <class T>
void copy_device(DBuf<T>& dst, const DBuf<T>& src, cudaStream_t s = 0) {
  dst.alloc(src.n);
  if (src.n) SIMP_CUDA(cudaMemcpyAsync(dst.p, src.p, src.n * sizeof(T), cudaMemcpyDeviceToDevice, s));
}

// Device view of a node-level pattern (see structure.h).
struct NodeView {
  const i32* ptr;   // row-node slot pointer
  const i32* nbr;   // column node per slot
  const i32* off;   // offset of the slot within a scalar row
};

inline int grid_for(i64 work, int block, int max_blocks = 1 << 20) {
  i64 g = (work + block - 1) / block;
  if (g < 1) g = 1;
  if (g > max_blocks) g = max_blocks;
  return static_cast<int>(g);
}

}  // namespace simp
