// Thin C entry points over the CUDA runtime, for the host runtime's device plane.
//
// The host library (libpsb200_core.so: Postoffice, vans, KVWorker) does not link against CUDA:
// it must load and run on machines without a GPU.  Its device plane (src/van/nvl_van.cc)
// binds this library at run time and reaches streams, events, copies and allocations through
// the functions below, next to the psdev_* kernels.  Every function returns 0 or a
// cudaError_t value.
#include <cuda.h>
#include <cuda_runtime.h>

#include "ps/device/psdev.h"

extern "C" {

int psdev_rt_device_count(int* n) { return (int)cudaGetDeviceCount(n); }
int psdev_rt_set_device(int device) { return (int)cudaSetDevice(device); }
int psdev_rt_get_device(int* device) { return (int)cudaGetDevice(device); }

int psdev_rt_malloc(void** p, size_t bytes) {
  cudaError_t e = cudaMalloc(p, bytes);
  if (e != cudaSuccess) return (int)e;
  return (int)cudaMemset(*p, 0, bytes);
}
int psdev_rt_free(void* p) { return (int)cudaFree(p); }
int psdev_rt_memset_async(void* p, int value, size_t bytes, void* stream) {
  return (int)cudaMemsetAsync(p, value, bytes, (cudaStream_t)stream);
}

// priority: 0 = default, 1 = highest priority the device offers
int psdev_rt_stream_create(void** stream, int priority) {
  cudaStream_t s;
  int lo = 0, hi = 0;
  cudaDeviceGetStreamPriorityRange(&lo, &hi);
  cudaError_t e = cudaStreamCreateWithPriority(&s, cudaStreamNonBlocking, priority ? hi : lo);
  *stream = s;
  return (int)e;
}
int psdev_rt_stream_destroy(void* stream) { return (int)cudaStreamDestroy((cudaStream_t)stream); }
// An id that no other stream of the process has or will have.  Handles do not tell streams apart:
// the per-thread default stream has one handle in all threads, and the handle of a destroyed stream
// can come back.
int psdev_rt_stream_id(void* stream, unsigned long long* id) {
  return (int)cudaStreamGetId((cudaStream_t)stream, id);
}
int psdev_rt_stream_sync(void* stream) { return (int)cudaStreamSynchronize((cudaStream_t)stream); }

int psdev_rt_event_create(void** event) {
  cudaEvent_t e;
  cudaError_t rc = cudaEventCreateWithFlags(&e, cudaEventDisableTiming);
  *event = e;
  return (int)rc;
}
int psdev_rt_event_destroy(void* event) { return (int)cudaEventDestroy((cudaEvent_t)event); }
int psdev_rt_event_record(void* event, void* stream) {
  return (int)cudaEventRecord((cudaEvent_t)event, (cudaStream_t)stream);
}
int psdev_rt_event_sync(void* event) { return (int)cudaEventSynchronize((cudaEvent_t)event); }
int psdev_rt_stream_wait_event(void* stream, void* event) {
  return (int)cudaStreamWaitEvent((cudaStream_t)stream, (cudaEvent_t)event, 0);
}

// Words that kernels write when they are done: every one in a line of its own, like its counter.
int psdev_done_create(int n, psdev_done_t* done) {
  constexpr size_t kLine = 128;
  if (n < 1 || !done) return PSDEV_ERR_ARG;
  char *host = nullptr, *words = nullptr, *tickets = nullptr;
  cudaError_t e = cudaHostAlloc(reinterpret_cast<void**>(&host), n * kLine,
                                cudaHostAllocMapped | cudaHostAllocPortable);
  if (e != cudaSuccess) return (int)e;
  e = cudaHostGetDevicePointer(reinterpret_cast<void**>(&words), host, 0);
  if (e == cudaSuccess) e = cudaMalloc(reinterpret_cast<void**>(&tickets), n * kLine);
  if (e == cudaSuccess) e = cudaMemset(tickets, 0, n * kLine);
  if (e == cudaSuccess) e = cudaDeviceSynchronize();
  if (e != cudaSuccess) {
    cudaFree(tickets);
    cudaFreeHost(host);
    return (int)e;
  }
  for (int i = 0; i < n; ++i) {
    done[i] = psdev_done_t{};
    done[i].host = reinterpret_cast<volatile uint32_t*>(host + i * kLine);
    *done[i].host = 0;
    done[i].word = reinterpret_cast<uint32_t*>(words + i * kLine);
    done[i].ticket = reinterpret_cast<uint32_t*>(tickets + i * kLine);
  }
  return 0;
}
// (the first entry's addresses are those of the allocations; both calls wait for running kernels)
int psdev_done_destroy(int n, psdev_done_t* done) {
  if (n < 1 || !done) return PSDEV_ERR_ARG;
  const cudaError_t a = cudaFree(done[0].ticket);
  const cudaError_t b = cudaFreeHost(const_cast<uint32_t*>(done[0].host));
  return (int)(a != cudaSuccess ? a : b);
}

// One asynchronous copy; the direction is inferred from the pointers (unified addressing).
int psdev_rt_memcpy_async(void* dst, const void* src, size_t bytes, void* stream) {
  return (int)cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDefault, (cudaStream_t)stream);
}

// 1 if `p` is device memory, 0 if it is host memory (pinned or pageable).
int psdev_rt_is_device_pointer(const void* p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged;
}
// What `p` points at: 0 host memory (pinned or pageable), 1 memory of the GPU *device, 2 managed.
int psdev_rt_memory(const void* p, int* device) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  *device = a.device;
  return a.type == cudaMemoryTypeManaged ? 2 : a.type == cudaMemoryTypeDevice;
}
// 1 if `p` is page-locked host memory that the device can copy from without staging.
int psdev_rt_is_pinned_host(const void* p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return a.type == cudaMemoryTypeHost;
}
// 1 if all of [p, p + bytes) is page-locked host memory that kernels can access; *dev receives
// its address on the device.  The range must lie in one allocation or registration: the ends of
// two of them say nothing about what lies between (all addresses have the same distance on host and
// device), and the driver is asked for the bounds of the one that `p` belongs to.
int psdev_rt_host_mapped(const void* p, size_t bytes, void** dev) {
  cudaPointerAttributes a;
  if (bytes == 0 || cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  if (a.type != cudaMemoryTypeHost || !a.devicePointer) return 0;
  static const auto attribute = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult found;
    if (cudaGetDriverEntryPoint("cuPointerGetAttribute", &f, cudaEnableDefault, &found) !=
            cudaSuccess || found != cudaDriverEntryPointSuccess) {
      cudaGetLastError();
      f = nullptr;
    }
    return reinterpret_cast<CUresult (*)(void*, CUpointer_attribute, CUdeviceptr)>(f);
  }();
  if (!attribute) return 0;
  CUdeviceptr start = 0;
  size_t size = 0;
  const CUdeviceptr at = reinterpret_cast<CUdeviceptr>(a.devicePointer);
  if (attribute(&start, CU_POINTER_ATTRIBUTE_RANGE_START_ADDR, at) != CUDA_SUCCESS ||
      attribute(&size, CU_POINTER_ATTRIBUTE_RANGE_SIZE, at) != CUDA_SUCCESS)
    return 0;
  if (at < start || at - start > size || bytes > size - (at - start)) return 0;
  *dev = a.devicePointer;
  return 1;
}
int psdev_rt_host_alloc(void** p, size_t bytes) {
  return (int)cudaHostAlloc(p, bytes, cudaHostAllocDefault);
}
int psdev_rt_host_free(void* p) { return (int)cudaFreeHost(p); }

}  // extern "C"
