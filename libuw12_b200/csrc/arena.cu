// The calling thread's block of small buffers (Arena, common.cuh).
#include "common.cuh"

namespace uw12b {

namespace {
thread_local Arena* t_arena = nullptr;
}  // namespace

Arena::Arena() {
  if (t_arena) return;
  s_ = current_stream();
  void* p = nullptr;
  if (cudaGetDevice(&dev_) != cudaSuccess ||
      cudaMallocFromPoolAsync(&p, kDoubles * sizeof(double), library_pool(), s_) != cudaSuccess) {
    cudaGetLastError();
    return;
  }
  base_ = static_cast<double*>(p);
  t_arena = this;
}

Arena::~Arena() {
  if (t_arena != this) return;
  t_arena = nullptr;
  cudaFreeAsync(base_, s_);
}

Arena* Arena::current() { return t_arena; }

double* Arena::take(size_t n_doubles, cudaStream_t s) {
  const size_t n = (n_doubles + 31) / 32 * 32;  // 256-byte aligned
  int dev = -1;
  if (s != s_ || n > kDoubles - off_ || cudaGetDevice(&dev) != cudaSuccess || dev != dev_)
    return nullptr;
  double* p = base_ + off_;
  off_ += n;
  return p;
}

}  // namespace uw12b
