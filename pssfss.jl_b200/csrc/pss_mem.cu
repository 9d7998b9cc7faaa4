// Device memory of the library: one pool per device behind cudaMalloc / cudaFree semantics.
//
// Every analysis uploads its sheets and classes their face pairs anew, some forty buffers of a
// few bytes to hundreds of megabytes; cudaMalloc and cudaFree of those, each with its
// synchronisation and page mapping, took longer than the device work of a small sheet (15 ms of a
// two-sheet stack, 9 ms of a sheet of 1648 faces).  The pool keeps up to kKeep bytes of freed
// memory mapped and is emptied when a context is destroyed or an allocation fails.  A pool's
// release threshold counts the memory in use as well, so it follows that: with a fixed one the
// buffers of a large sweep alone exceeded it, every synchronisation unmapped all that was free,
// and setting a sheet of 3960 faces up took 500 ms instead of 93.
#include "pss_internal.cuh"

namespace {

constexpr unsigned long long kKeep = 2ull << 30;
constexpr int kMaxDevices = 64;

struct Pool {
  cudaMemPool_t pool = nullptr;
  cudaStream_t st = nullptr;  // allocations and frees are ordered on this stream
};
Pool g_pool[kMaxDevices];
DeviceOnce g_once;

int current_pool(Pool **out) {
  int dev = 0;
  PSS_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) { pss_set_error("device %d out of range", dev); return -3; }
  if (int rc = device_once(g_once, [dev] {
        Pool p;
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        PSS_CUDA_TRY(cudaMemPoolCreate(&p.pool, &props));
        unsigned long long keep = kKeep;
        PSS_CUDA_TRY(cudaMemPoolSetAttribute(p.pool, cudaMemPoolAttrReleaseThreshold, &keep));
        PSS_CUDA_TRY(cudaStreamCreateWithFlags(&p.st, cudaStreamNonBlocking));
        g_pool[dev] = p;
        return 0;
      }))
    return rc;
  *out = &g_pool[dev];
  return 0;
}

// At most kKeep bytes beyond what is in use stay mapped.
void follow_use(Pool *q) {
  unsigned long long used = 0;
  if (cudaMemPoolGetAttribute(q->pool, cudaMemPoolAttrUsedMemCurrent, &used) != cudaSuccess) return;
  unsigned long long keep = used + kKeep;
  cudaMemPoolSetAttribute(q->pool, cudaMemPoolAttrReleaseThreshold, &keep);
}

}  // namespace

// Memory of the current device, usable on every stream when the call returns.
int pss_dev_alloc(void **p, size_t bytes) {
  *p = nullptr;
  Pool *q = nullptr;
  if (int rc = current_pool(&q)) return rc;
  cudaError_t e = cudaMallocFromPoolAsync(p, bytes, q->pool, q->st);
  if (e == cudaErrorMemoryAllocation) {  // give the kept memory back and try once more
    cudaGetLastError();
    cudaDeviceSynchronize();
    cudaMemPoolTrimTo(q->pool, 0);
    e = cudaMallocFromPoolAsync(p, bytes, q->pool, q->st);
  }
  if (e == cudaSuccess) {
    follow_use(q);
    e = cudaStreamSynchronize(q->st);
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    *p = nullptr;
    pss_set_error("device allocation of %zu bytes failed: %s", bytes, cudaGetErrorString(e));
    return -3;
  }
  return 0;
}

// As cudaFree: waits for the device, so no stream still uses the memory when it is reused.
void pss_dev_free(void *p) {
  Pool *q = nullptr;
  if (!p || current_pool(&q)) return;
  cudaDeviceSynchronize();
  cudaFreeAsync(p, q->st);
  follow_use(q);
}

void pss_dev_trim() {
  Pool *q = nullptr;
  if (current_pool(&q)) return;
  cudaDeviceSynchronize();
  cudaMemPoolTrimTo(q->pool, 0);
}
