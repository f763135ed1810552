// Device buffers against a fake CUDA whose memory runs out: what the library's own pool keeps
// is given back and the allocation tried again, wherever it comes from.
#include <cstdarg>
#include <cstdio>

#include "../../tight_binding_gb300/csrc/tbk_internal.h"

static int trims, mallocs, pool_mallocs, fails, last_error;
static bool full;                                      // until the pool is trimmed
static bool forever;
static char memory[64];

extern "C" {
cudaError_t cudaMalloc(void** p, size_t) {
  ++mallocs;
  if (full || forever) { last_error = 1; return cudaErrorMemoryAllocation; }
  *p = memory;
  return cudaSuccess;
}
cudaError_t cudaMallocFromPoolAsync(void** p, size_t, cudaMemPool_t, cudaStream_t) {
  ++pool_mallocs;
  if (full || forever) { last_error = 1; return cudaErrorMemoryAllocation; }
  *p = memory;
  return cudaSuccess;
}
cudaError_t cudaFree(void*) { return cudaSuccess; }
cudaError_t cudaFreeAsync(void*, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetLastError() { last_error = 0; return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
}
namespace tbk {
thread_local const AsyncAllocCtx* tl_async_alloc = nullptr;
void scratch_trim() { ++trims; full = false; }
cudaMemPool_t scratch_pool() { return reinterpret_cast<cudaMemPool_t>(memory); }
int fail(int code, const char*, ...) { ++fails; return code; }
}  // namespace tbk

#define CHECK(c) do { if (!(c)) { std::printf("FAILED %s:%d %s\n", __FILE__, __LINE__, #c); return 1; } } while (0)

int main() {
  using namespace tbk;
  AsyncAllocCtx own, other;
  own.scratch = true;
  struct { const AsyncAllocCtx* ctx; size_t bytes; } cases[] = {
      {nullptr, 1000}, {&own, 1000}, {&own, kScratchMax + 1}, {&other, 1000}, {&other, size_t(1) << 34}};
  for (const auto& k : cases) {
    tl_async_alloc = k.ctx;
    trims = fails = mallocs = pool_mallocs = 0;
    {
      full = forever = false;
      DevBuf b;
      CHECK(b.alloc(k.bytes) == TBK_OK && b.bytes == k.bytes && trims == 0 && fails == 0);
      CHECK(mallocs + pool_mallocs == 1 && (pool_mallocs == 1) == (k.ctx && (k.ctx != &own || k.bytes <= kScratchMax)));
      CHECK(b.scratch == (pool_mallocs == 1 && k.ctx == &own) && b.ctx == (k.ctx == &other ? &other : nullptr));
    }
    {
      full = true;
      mallocs = 0;
      DevBuf b;
      CHECK(b.alloc(k.bytes) == TBK_OK && b.bytes == k.bytes && trims == 1 && fails == 0 && last_error == 0);
      CHECK(k.ctx != &other || mallocs == 0);          // another pool's budget is not left
    }
    {
      forever = true;
      DevBuf b;
      CHECK(b.alloc(k.bytes) == TBK_ERR_NOMEM && b.p == nullptr && trims == 2 && fails == 1 && last_error == 0);
    }
  }
  std::printf("ALL PASSED\n");
  return 0;
}
