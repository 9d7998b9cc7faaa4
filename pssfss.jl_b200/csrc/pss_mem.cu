// Device memory of the library: one pool per device behind cudaMalloc / cudaFree semantics.
//
// Every analysis uploads its sheets and classes their face pairs anew, some forty buffers of a
// few bytes to hundreds of megabytes; cudaMalloc and cudaFree of those, each with its
// synchronisation and page mapping, took longer than the device work of a small sheet (15 ms of a
// two-sheet stack, 9 ms of a sheet of 1648 faces).  The pool keeps up to kKeep bytes of freed
// memory mapped and is emptied when a context is destroyed, an allocation fails or the caller asks
// (pss_release_memory: no other allocator of the process can use what the pool keeps).  The bound is
// kept by trimming when a buffer is freed.  A pool's own release threshold does not serve: it
// counts the memory in use as well, and once a synchronisation finds it exceeded, all that is free is
// unmapped, not the excess alone - setting up the seven sheets of a gradient (3960 faces each) took
// 0.12 to 0.96 s from call to call, 0.10 now.
//
// A pool and its stream end with their context (a device reset), so both are made anew when the
// device's context is another one than theirs.
#include <cuda.h>

#include "pss_internal.cuh"

namespace {

constexpr unsigned long long kKeep = 2ull << 30;

struct Pool {
  cudaMemPool_t pool = nullptr;
  cudaStream_t st = nullptr;  // allocations and frees are ordered on this stream
};
Pool g_pool[kMaxDevices];
DeviceOnce g_once;

int current_pool(Pool **out) {
  int dev = 0;
  unsigned long long id = 0;
  if (int rc = pss_context_id(&dev, &id)) return rc;
  if (int rc = device_once(g_once, [dev] {
        Pool p;
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        PSS_CUDA_TRY(cudaMemPoolCreate(&p.pool, &props));
        unsigned long long keep = ~0ull;  // pss_dev_free trims
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
void trim_to_keep(Pool *q) {
  unsigned long long used = 0, held = 0;
  if (cudaMemPoolGetAttribute(q->pool, cudaMemPoolAttrUsedMemCurrent, &used) != cudaSuccess ||
      cudaMemPoolGetAttribute(q->pool, cudaMemPoolAttrReservedMemCurrent, &held) != cudaSuccess)
    return;
  if (held <= used + kKeep) return;
  cudaStreamSynchronize(q->st);  // the frees have taken effect
  cudaMemPoolTrimTo(q->pool, used + kKeep);
}

using CtxGetCurrentFn = CUresult (*)(CUcontext *);
using CtxGetIdFn = CUresult (*)(CUcontext, unsigned long long *);
struct DriverFns {
  CtxGetCurrentFn current = nullptr;
  CtxGetIdFn id = nullptr;
};

template <class Fn>
bool driver_fn(const char *name, Fn &out) {
  void *fn = nullptr;
  cudaDriverEntryPointQueryResult q;
  if (cudaGetDriverEntryPoint(name, &fn, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess)
    return false;
  out = (Fn)fn;
  return fn != nullptr;
}

}  // namespace

int pss_context_id(int *dev, unsigned long long *id) {
  static const DriverFns drv = [] {
    DriverFns d;
    if (!driver_fn("cuCtxGetCurrent", d.current) || !driver_fn("cuCtxGetId", d.id)) d = DriverFns{};
    return d;
  }();
  if (!drv.id) { pss_set_error("cuCtxGetCurrent or cuCtxGetId unavailable"); return -3; }
  *dev = -1;
  PSS_CUDA_TRY(cudaGetDevice(dev));
  if (*dev < 0 || *dev >= kMaxDevices) { pss_set_error("device %d out of range", *dev); return -3; }
  auto read = [&] {
    CUcontext ctx = nullptr;
    return drv.current(&ctx) == CUDA_SUCCESS && ctx && drv.id(ctx, id) == CUDA_SUCCESS;
  };
  if (read()) return 0;
  cudaFree(nullptr);  // the device's context is not there yet, or was reset: the runtime makes it
  if (read()) return 0;
  cudaGetLastError();
  pss_set_error("no current CUDA context on device %d", *dev);
  return -3;
}

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
  if (e == cudaSuccess) e = cudaStreamSynchronize(q->st);
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
  trim_to_keep(q);
}

int pss_dev_trim() {
  Pool *q = nullptr;
  if (int rc = current_pool(&q)) return rc;
  PSS_CUDA_TRY(cudaDeviceSynchronize());
  PSS_CUDA_TRY(cudaMemPoolTrimTo(q->pool, 0));
  return 0;
}
