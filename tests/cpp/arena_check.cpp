// The block of small buffers (csrc/arena.cu, compiled in here) on a fake CUDA runtime of
// two devices: buffers come from the block on its own stream and device only.
#include <cstdio>
#include <cstdlib>

#include "arena.cu"

namespace {
int g_device = 0;
int g_from_pool = 0;
char g_memory[2][1];
cudaStream_t g_stream = nullptr;
}  // namespace

extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = g_device; return cudaSuccess; }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t, cudaStream_t) {
  ++g_from_pool;
  *p = std::malloc(n < 4096 ? 4096 : n);
  return cudaSuccess;
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { std::free(p); return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return ""; }
cudaError_t cudaMemsetAsync(void*, int, size_t, cudaStream_t) { return cudaSuccess; }
}

namespace uw12b {
cudaStream_t current_stream() { return g_stream; }
cudaMemPool_t library_pool() { return reinterpret_cast<cudaMemPool_t>(&g_memory[g_device]); }
}  // namespace uw12b

#define EXPECT(c)                                              \
  do {                                                         \
    if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); return 1; } \
  } while (0)

int main() {
  using namespace uw12b;
  {
    Arena arena;  // device 0, default stream
    EXPECT(g_from_pool == 1);
    DevBuf a(100);
    EXPECT(g_from_pool == 1);
    {
      Arena inner;  // nested on the same thread: does nothing
      DevBuf b(100);
      EXPECT(g_from_pool == 1);
    }
    g_device = 1;  // the same stream handle, another device
    {
      Arena inner;
      DevBuf b(100);
      EXPECT(g_from_pool == 2);
    }
    g_device = 0;
    g_stream = reinterpret_cast<cudaStream_t>(&g_memory[1]);  // another stream
    {
      DevBuf b(100);
      EXPECT(g_from_pool == 3);
    }
    g_stream = nullptr;
    DevBuf c(100);
    EXPECT(g_from_pool == 3);
    EXPECT(c.get() == a.get() + 128);  // laid one after the other, 256-byte steps
  }
  DevBuf d(100);
  EXPECT(g_from_pool == 4);
  std::puts("ok");
  return 0;
}
