// A host-only stand-in for the CUDA runtime under csrc/vt_api.cu: two devices whose memory is host memory. A
// stream or an event belongs to the device that was current when it was made, an event is recorded on a
// stream of its own device only, and what a device has rendered reaches its memory when that device is
// synchronised. tests/test_context_device.py builds and drives it.
#include <cstdlib>
#include <cstring>
#include <thread>

#include "vt_internal.cuh"

namespace {
thread_local int current = 0;
struct Handle {
  int device;
};
// Per device: the image its queued work will have written, and where to.
struct Pending {
  double *dst = nullptr;
  double value = 0.0;
  size_t n = 0;
} pending[2];
void *take(size_t bytes) { return std::calloc(1, bytes ? bytes : 1); }
template <typename T> cudaError_t make(T *out) {
  *out = reinterpret_cast<T>(new Handle{current});
  return cudaSuccess;
}
}  // namespace

extern "C" {
cudaError_t cudaGetDeviceCount(int *n) { *n = 2; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { current = d; return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = current; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaDeviceSynchronize(void) {
  Pending &p = pending[current];
  for (size_t i = 0; i < p.n; ++i) p.dst[i] = p.value;
  p.n = 0;
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return make(s); }
cudaError_t cudaStreamDestroy(cudaStream_t s) { delete reinterpret_cast<Handle *>(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { return make(e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return make(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { delete reinterpret_cast<Handle *>(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  return reinterpret_cast<Handle *>(e)->device == reinterpret_cast<Handle *>(s)->device ? cudaSuccess : cudaErrorInvalidResourceHandle;
}
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaMalloc(void **p, size_t n) { *p = take(n); return cudaSuccess; }
cudaError_t cudaMallocHost(void **p, size_t n) { *p = take(n); return cudaSuccess; }
cudaError_t cudaFree(void *p) { std::free(p); return cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { std::free(p); return cudaSuccess; }
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { std::free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemset(void *d, int v, size_t n) { std::memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) { std::memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemPoolCreate(cudaMemPool_t *, const cudaMemPoolProps *) { return cudaErrorNotSupported; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *) { return cudaErrorNotSupported; }
cudaError_t cudaMemPoolDestroy(cudaMemPool_t) { return cudaSuccess; }
cudaError_t cudaMallocFromPoolAsync(void **, size_t, cudaMemPool_t, cudaStream_t) { return cudaErrorNotSupported; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *) {
  std::memset(a, 0, sizeof *a);
  a->type = cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t e) { return e == cudaErrorInvalidResourceHandle ? "invalid resource handle" : "fake error"; }
cudaError_t cudaLaunchKernel(const void *, dim3, dim3, void **, size_t, cudaStream_t) { return cudaErrorNotSupported; }
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, CUstream_st *) { return 1u; }
cudaError_t __cudaPopCallConfiguration(dim3 *, dim3 *, size_t *, void *) { return cudaSuccess; }
void **__cudaRegisterFatBinary(void *) { return nullptr; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, uint3 *, uint3 *, dim3 *, dim3 *, int *) {}

// A scene of a w x h image whose every sum becomes `value` once device `device` is synchronised.
void *fake_scene(int device, uint32_t w, uint32_t h, uint32_t samples, double value) {
  vt_scene *s = new vt_scene();
  const size_t n = 3 * (size_t)w * h;
  s->width = w;
  s->height = h;
  s->samples = samples;
  s->d_accum = static_cast<double *>(take(n * sizeof(double)));
  pending[device] = {s->d_accum, value, n};
  return s;
}
}

// What vt_api.cu links against and the test does not reach.
vt_status vt_lbvh_build(vt_ctx *, const vt_face *, uint32_t, const vt_vertex *, uint32_t, const vt_build_options &, vt_mesh *) {
  return VT_ERR_DEVICE;
}
void vt_launch_closest(const vt_mesh *, const vt_ray *, uint32_t, vt_hit *, int, uint32_t *, const uint32_t *, uint32_t *, cudaStream_t,
                       const uint32_t *, bool, bool) {}
void vt_launch_any(const vt_mesh *, const vt_ray *, uint32_t, uint8_t *, int, uint32_t *, const uint32_t *, uint32_t *, cudaStream_t,
                   const uint32_t *, bool, bool) {}
void vt_launch_count(const vt_mesh *, const vt_ray *, uint32_t, int, unsigned long long *, cudaStream_t) {}
