// Shared definitions for the UW12 B200 engine: status codes, error helpers,
// stream-ordered device buffers and launch accounting.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>
#include <stdexcept>
#include <string>
#include <vector>

namespace uw12b {

// Status codes of the C-ABI (mirrors the exception classes of libuw12).
enum Status : int {
  kOk = 0,
  kErrRuntime = 1,  // std::runtime_error in libuw12 (user-input errors)
  kErrLogic = 2,    // std::logic_error in libuw12 (shape errors)
  kErrCuda = 3,
  kErrAlloc = 4,
  kErrInvalid = 5,
};

struct Error : std::runtime_error {
  int code;
  Error(int c, const std::string& m) : std::runtime_error(m), code(c) {}
};

[[noreturn]] inline void throw_runtime(const std::string& m) { throw Error(kErrRuntime, m); }
[[noreturn]] inline void throw_logic(const std::string& m) { throw Error(kErrLogic, m); }

inline void cuda_check(cudaError_t e, const char* what, const char* file, int line) {
  if (e != cudaSuccess) {
    const int code = (e == cudaErrorMemoryAllocation) ? kErrAlloc : kErrCuda;
    // a failed allocation is reported here: left behind as the thread's last error, it would
    // fail the next launch check, the library's or its caller's
    if (code == kErrAlloc) cudaGetLastError();
    throw Error(code, std::string(what) + ": " + cudaGetErrorString(e) + " (" + file + ":" +
                          std::to_string(line) + ")");
  }
}

#define UW12_CUDA(expr) ::uw12b::cuda_check((expr), #expr, __FILE__, __LINE__)
#define UW12_LAUNCHED() ::uw12b::note_launch(__FILE__, __LINE__)

// Counts this library's kernel launches (used by benchmarks to report how many
// native launches a call made) and surfaces launch-configuration errors.
void note_launch(const char* file, int line);
unsigned long long launch_count();

// Launches a kernel whose threads all call chain_wait: its blocks may be started
// while the stream's previous kernel still drains.
//
// What bounds a chain of small kernels is the drain, launch and fill between two of
// them: 83 kernels of a small Fock matrix (N = 24) 0.50 -> 0.30 ms, 48 of an
// open-shell energy (N = 61) 0.36 -> 0.26, Fock at N = 120 3.07 -> 2.89 ms.
template <typename... P, typename... A>
inline void launch_chained(void (*kernel)(P...), dim3 grid, unsigned block, size_t smem,
                           cudaStream_t s, A... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  UW12_CUDA(cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...));
}

#ifdef __CUDACC__
// Holds the thread until everything before this kernel in its stream has finished
// and its writes are visible; returns at once in a kernel launched otherwise.  Every
// thread of a chained kernel calls it before it exits and before its first access
// to device memory, constant operands included (their buffers are reused): a
// kernel then finishes only after all before it, so its successor need not look
// further back.  Operands read by plain loads are not __restrict__ in such kernels, so
// that no read can be moved ahead of the wait.
__device__ __forceinline__ void chain_wait() {
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
}
// Lets the stream's next kernel, if chained, take free SM slots once every block of
// this one has got here (without it: once every block has finished).  Placed where
// little is left to do: at the start of the GEMM, the waiting blocks held slots that
// the drain of a wide product or another stream could use (N = 61 0.26 -> 0.32 ms,
// N = 120 2.89 -> 2.96, twelve molecules on eight streams 10.4 -> 10.9); in the
// streaming kernels it gained nothing.
__device__ __forceinline__ void chain_release() {
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
}
#endif

// Stream used by every launch of the calling host thread.
cudaStream_t current_stream();
void set_current_stream(cudaStream_t s);

// The library's own stream-ordered memory pool on the current device.  It
// keeps freed memory reserved (release threshold = max) so repeated calls do
// not map and unmap pages; trim_pools() returns it to the system.
cudaMemPool_t library_pool();
void trim_pools();

// One block of the pool that serves the small buffers of an evaluation on this
// host thread and its current stream: a buffer from it costs no driver call (a
// stream-ordered allocation and its release cost about 1.5 us of host time, and
// the smallest evaluations make 80 of them in 0.65 ms).  Buffers are laid one
// after the other; the last one laid is taken back when it is released, the
// others with the arena.  All of them are used on the arena's stream only, so
// memory given out again is reused in stream order.  An arena inside another on
// the same thread and stream does nothing; without memory for its block it
// leaves every buffer to the pool.
class Arena {
 public:
  Arena();
  ~Arena();
  Arena(const Arena&) = delete;
  Arena& operator=(const Arena&) = delete;

  // The calling thread's arena (null: none).
  static Arena* current();
  // n doubles for stream s of the current device, or null when they do not fit or the
  // block is another stream's or device's (a call made by a producer or a sink inside the
  // evaluation may be on either; the default stream is the same handle on every device).
  double* take(size_t n_doubles, cudaStream_t s);
  void give(const double* p, size_t n_doubles) {
    const size_t n = (n_doubles + 31) / 32 * 32;
    if (p + n == base_ + off_) off_ -= n;
  }

 private:
  static constexpr size_t kDoubles = (size_t(32) << 20) / sizeof(double);  // 32 MiB
  double* base_ = nullptr;
  size_t off_ = 0;
  cudaStream_t s_ = nullptr;
  int dev_ = -1;
};

// Device memory from the calling thread's arena, when it fits there, or from the
// library's stream-ordered pool of the current device.
class DevBuf {
 public:
  DevBuf() = default;
  explicit DevBuf(size_t n_doubles, cudaStream_t s = nullptr) { alloc(n_doubles, s); }
  DevBuf(const DevBuf&) = delete;
  DevBuf& operator=(const DevBuf&) = delete;
  DevBuf(DevBuf&& o) noexcept { take(o); }
  DevBuf& operator=(DevBuf&& o) noexcept {
    if (this != &o) {
      release();
      take(o);
    }
    return *this;
  }
  ~DevBuf() { release(); }

  void alloc(size_t n_doubles, cudaStream_t s = nullptr) {
    release();
    s_ = s ? s : current_stream();
    n_ = n_doubles;
    if (!n_) return;
    if (Arena* a = Arena::current()) {
      p_ = a->take(n_, s_);
      if (p_) {
        arena_ = a;
        return;
      }
    }
    UW12_CUDA(cudaMallocFromPoolAsync(reinterpret_cast<void**>(&p_), n_ * sizeof(double),
                                      library_pool(), s_));
  }
  void zero() {
    if (n_) UW12_CUDA(cudaMemsetAsync(p_, 0, n_ * sizeof(double), s_));
  }
  void release() noexcept {
    if (p_ && arena_)
      arena_->give(p_, n_);
    else if (p_)
      cudaFreeAsync(p_, s_);
    p_ = nullptr;
    arena_ = nullptr;
    n_ = 0;
  }
  double* get() const { return p_; }
  size_t size() const { return n_; }

 private:
  void take(DevBuf& o) noexcept {
    p_ = o.p_; n_ = o.n_; s_ = o.s_; arena_ = o.arena_;
    o.p_ = nullptr; o.n_ = 0; o.arena_ = nullptr;
  }
  double* p_ = nullptr;
  size_t n_ = 0;
  cudaStream_t s_ = nullptr;
  Arena* arena_ = nullptr;
};

inline size_t packed_size(size_t n) { return n * (n + 1) / 2; }

}  // namespace uw12b
