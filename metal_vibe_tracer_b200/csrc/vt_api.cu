// vt_api.cu — the C ABI (include/vt.h): contexts, mesh publish, traversal entry points.
#include <algorithm>
#include <atomic>
#include <cstring>
#include <string>
#include <thread>
#include <vector>

#include "vt_internal.cuh"

// The error of calls made without a context (context creation, host-only entry points).
thread_local std::string g_no_ctx_error;

vt_status vt_fail(vt_ctx *ctx, vt_status code, const std::string &msg) {
  if (ctx) ctx->error = msg; else g_no_ctx_error = msg;
  return code;
}

vt_status vt_cuda_fail(vt_ctx *ctx, cudaError_t err, const char *what) {
  std::string m = std::string(what) + ": " + cudaGetErrorString(err);
  return vt_fail(ctx, err == cudaErrorMemoryAllocation ? VT_ERR_MEMORY : VT_ERR_CUDA, m);
}

cudaError_t vt_pool_alloc(vt_ctx *ctx, void **p, size_t bytes) {
  if (!ctx->pool) {
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = ctx->device;
    cudaMemPool_t pool;
    cudaError_t e = cudaMemPoolCreate(&pool, &props);
    if (e != cudaSuccess) return e;
    uint64_t keep = kPoolKeep;
    e = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
    if (e != cudaSuccess) {
      cudaMemPoolDestroy(pool);
      return e;
    }
    ctx->pool = pool;
  }
  return cudaMallocFromPoolAsync(p, bytes, ctx->pool, ctx->stream);
}

namespace {

// Waits for every use of the mesh first (freeing pool memory does not, unlike plain cudaFree).
void free_mesh(vt_mesh *m) {
  if (!m) return;
  int dev = 0;
  const bool other = cudaGetDevice(&dev) == cudaSuccess && dev != m->device;
  if (other) cudaSetDevice(m->device);
  cudaDeviceSynchronize();
  cudaFree(m->d_nodes);
  cudaFree(m->d_tris);
  cudaFree(m->d_order);
  cudaFree(m->d_codes);
  cudaFree(m->d_sorted);
  cudaFree(m->d_bin_child);
  cudaFree(m->d_bin_box);
  cudaFree(m->d_qnodes);
  cudaFree(m->d_nrm);
  if (other) cudaSetDevice(dev);
  delete m;
}

vt_build_options defaults(const vt_build_options *o) {
  vt_build_options r;
  std::memset(&r, 0, sizeof r);
  if (o) r = *o;
  return r;
}

// Device-side copy of the chunk buffers for host pipelining.
vt_status ensure_chunks(vt_ctx *ctx, size_t in_bytes, size_t out_bytes) {
  if (in_bytes > ctx->chunk_in_bytes) {
    for (int k = 0; k < 2; ++k) {
      cudaFree(ctx->d_chunk_in[k]);
      ctx->d_chunk_in[k] = nullptr;
      VT_CUDA(ctx, cudaMalloc(&ctx->d_chunk_in[k], in_bytes));
    }
    ctx->chunk_in_bytes = in_bytes;
  }
  if (out_bytes > ctx->chunk_out_bytes) {
    for (int k = 0; k < 2; ++k) {
      cudaFree(ctx->d_chunk_out[k]);
      ctx->d_chunk_out[k] = nullptr;
      VT_CUDA(ctx, cudaMalloc(&ctx->d_chunk_out[k], out_bytes));
    }
    ctx->chunk_out_bytes = out_bytes;
  }
  return VT_OK;
}

vt_status check_trace_args(vt_ctx *ctx, const vt_mesh *mesh, const void *rays, const void *out, uint32_t n) {
  if (!ctx) return VT_ERR_INVALID;
  if (!mesh) return vt_fail(ctx, VT_ERR_INVALID, "mesh is null");
  if (n > 0 && (!rays || !out)) return vt_fail(ctx, VT_ERR_INVALID, "rays or output is null");
  if (n > 0 && mesh->nfaces > 0 && !mesh->d_nodes) return vt_fail(ctx, VT_ERR_INVALID, "mesh has no nodes");
  if (mesh->nnodes >= (1u << 29)) return vt_fail(ctx, VT_ERR_LIMIT, "traversal supports up to 2^29 - 1 wide nodes");
  return VT_OK;
}

// Chunk of rays per pipeline stage: 2^22 rays = 128 MB in, 64 MB out.
constexpr uint32_t kChunk = 1u << 22;

__global__ void k_fill_miss(int4 *hits, uint32_t n) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) hits[i] = make_int4(0, 0, 0, -1);
}

}  // namespace

extern "C" {

uint32_t vt_abi_version(void) { return VT_ABI_VERSION; }

vt_status vt_ctx_create(int32_t device, vt_ctx **out) {
  if (!out) return VT_ERR_INVALID;
  *out = nullptr;
  int count = 0;
  cudaError_t e = cudaGetDeviceCount(&count);
  if (e != cudaSuccess || count == 0) {
    g_no_ctx_error = std::string("no CUDA device: ") + cudaGetErrorString(e);
    return VT_ERR_CUDA;
  }
  if (device < 0 || device >= count) return VT_ERR_INVALID;
  vt_ctx *c = new vt_ctx();
  c->device = device;
  if ((e = cudaSetDevice(device)) != cudaSuccess ||
      (e = cudaDeviceGetAttribute(&c->sm_count, cudaDevAttrMultiProcessorCount, device)) != cudaSuccess ||
      (e = cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking)) != cudaSuccess ||
      (e = cudaStreamCreateWithFlags(&c->pipe[0], cudaStreamNonBlocking)) != cudaSuccess ||
      (e = cudaStreamCreateWithFlags(&c->pipe[1], cudaStreamNonBlocking)) != cudaSuccess ||
      (e = cudaEventCreate(&c->ev0)) != cudaSuccess || (e = cudaEventCreate(&c->ev1)) != cudaSuccess ||
      (e = cudaMalloc(&c->d_status, 64)) != cudaSuccess || (e = cudaMalloc(&c->d_counters, kCounterWords * sizeof(uint32_t))) != cudaSuccess) {
    g_no_ctx_error = std::string("context creation: ") + cudaGetErrorString(e);
    vt_ctx_destroy(c);
    return VT_ERR_CUDA;
  }
  cudaMemset(c->d_status, 0, 64);
  *out = c;
  return VT_OK;
}

vt_status vt_ctx_destroy(vt_ctx *ctx) {
  if (!ctx) return VT_OK;
  cudaSetDevice(ctx->device);
  if (ctx->stream) cudaStreamSynchronize(ctx->stream);
  for (int k = 0; k < 2; ++k) {
    if (ctx->pipe[k]) cudaStreamSynchronize(ctx->pipe[k]);
    cudaFree(ctx->d_chunk_in[k]);
    cudaFree(ctx->d_chunk_out[k]);
    if (ctx->pipe[k]) cudaStreamDestroy(ctx->pipe[k]);
  }
  cudaFreeHost(ctx->h_stage_in);
  cudaFreeHost(ctx->h_stage_out);
  for (cudaEvent_t *ev : {ctx->stage_in_ev, ctx->stage_out_ev})
    for (uint32_t k = 0; k < kStageSlots; ++k)
      if (ev[k]) cudaEventDestroy(ev[k]);
  cudaFree(ctx->d_status);
  cudaFree(ctx->d_counters);
  cudaFree(ctx->d_fgrid);
  cudaFree(ctx->d_pbr);
  cudaFree(ctx->d_gnodes);
  if (ctx->pool) cudaMemPoolDestroy(ctx->pool);  // meshes still alive keep their memory until freed
  if (ctx->ev0) cudaEventDestroy(ctx->ev0);
  if (ctx->ev1) cudaEventDestroy(ctx->ev1);
  if (ctx->stream) cudaStreamDestroy(ctx->stream);
  delete ctx;
  return VT_OK;
}

const char *vt_last_error(const vt_ctx *ctx) { return ctx ? ctx->error.c_str() : g_no_ctx_error.c_str(); }

vt_status vt_sync(vt_ctx *ctx) {
  if (!ctx) return VT_ERR_INVALID;
  VT_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return VT_OK;
}

vt_status vt_mesh_build_device(vt_ctx *ctx, const vt_face *faces_dev, uint32_t nfaces,
                               const vt_vertex *verts_dev, uint32_t nverts,
                               const vt_build_options *opts, vt_mesh **out) {
  if (!ctx) return VT_ERR_INVALID;
  if (!out) return vt_fail(ctx, VT_ERR_INVALID, "out is null");
  *out = nullptr;
  if (nfaces > 0 && (!faces_dev || !verts_dev)) return vt_fail(ctx, VT_ERR_INVALID, "faces or vertices is null");
  if (nfaces > (1u << 30)) return vt_fail(ctx, VT_ERR_LIMIT, "more than 2^30 faces");
  VT_CUDA(ctx, cudaSetDevice(ctx->device));
  vt_mesh *m = new vt_mesh();
  m->device = ctx->device;
  vt_build_options o = defaults(opts);
  vt_status st = vt_lbvh_build(ctx, faces_dev, nfaces, verts_dev, nverts, o, m);
  if (st != VT_OK) {
    cudaStreamSynchronize(ctx->stream);
    free_mesh(m);
    return st;
  }
  *out = m;
  return VT_OK;
}

vt_status vt_mesh_build(vt_ctx *ctx, const vt_face *faces, uint32_t nfaces, const vt_vertex *verts,
                        uint32_t nverts, const vt_build_options *opts, vt_mesh **out) {
  if (!ctx) return VT_ERR_INVALID;
  if (nfaces > 0 && (!faces || !verts)) return vt_fail(ctx, VT_ERR_INVALID, "faces or vertices is null");
  VT_CUDA(ctx, cudaSetDevice(ctx->device));
  vt_face *df = nullptr;
  vt_vertex *dv = nullptr;
  if (nfaces > 0) {
    VT_CUDA(ctx, vt_pool_alloc(ctx, reinterpret_cast<void **>(&df), (size_t)nfaces * sizeof(vt_face)));
    cudaError_t e = vt_pool_alloc(ctx, reinterpret_cast<void **>(&dv), (size_t)(nverts ? nverts : 1) * sizeof(vt_vertex));
    if (e != cudaSuccess) { cudaFreeAsync(df, ctx->stream); return vt_cuda_fail(ctx, e, "allocating the vertices"); }
    e = cudaMemcpyAsync(df, faces, (size_t)nfaces * sizeof(vt_face), cudaMemcpyHostToDevice, ctx->stream);
    if (e == cudaSuccess && nverts)
      e = cudaMemcpyAsync(dv, verts, (size_t)nverts * sizeof(vt_vertex), cudaMemcpyHostToDevice, ctx->stream);
    if (e != cudaSuccess) {
      cudaFreeAsync(df, ctx->stream);
      cudaFreeAsync(dv, ctx->stream);
      return vt_cuda_fail(ctx, e, "cudaMemcpyAsync(mesh)");
    }
  }
  vt_status st = vt_mesh_build_device(ctx, df, nfaces, dv, nverts, opts, out);
  cudaStreamSynchronize(ctx->stream);
  if (df) cudaFreeAsync(df, ctx->stream);
  if (dv) cudaFreeAsync(dv, ctx->stream);
  return st;
}

vt_status vt_mesh_destroy(vt_ctx *ctx, vt_mesh *mesh) {
  if (ctx) {
    cudaSetDevice(ctx->device);
    cudaStreamSynchronize(ctx->stream);
  }
  free_mesh(mesh);
  return VT_OK;
}

vt_status vt_mesh_get_info(vt_ctx *ctx, const vt_mesh *mesh, vt_mesh_info *out) {
  if (!ctx) return VT_ERR_INVALID;
  if (!mesh || !out) return vt_fail(ctx, VT_ERR_INVALID, "mesh or out is null");
  out->faces = mesh->nfaces;
  out->wide_nodes = mesh->nnodes;
  out->binary_nodes = mesh->nfaces > 1 ? mesh->nfaces - 1 : 0;
  out->depth = mesh->depth;
  out->sah_cost = mesh->sah;
  out->build_ms = mesh->build_ms;
  for (int k = 0; k < 3; ++k) { out->lo[k] = mesh->lo[k]; out->hi[k] = mesh->hi[k]; }
  return VT_OK;
}

vt_status vt_mesh_get_order(vt_ctx *ctx, const vt_mesh *mesh, int32_t *order, uint32_t n) {
  if (!ctx) return VT_ERR_INVALID;
  if (!mesh || (n && !order)) return vt_fail(ctx, VT_ERR_INVALID, "mesh or order is null");
  if (n != mesh->nfaces) return vt_fail(ctx, VT_ERR_INVALID, "n must equal the face count");
  if (n) VT_CUDA(ctx, cudaMemcpy(order, mesh->d_order, n * sizeof(int32_t), cudaMemcpyDeviceToHost));
  return VT_OK;
}

vt_status vt_mesh_get_nodes(vt_ctx *ctx, const vt_mesh *mesh, vt_wide_node *nodes, uint32_t n) {
  if (!ctx) return VT_ERR_INVALID;
  if (!mesh || (n && !nodes)) return vt_fail(ctx, VT_ERR_INVALID, "mesh or nodes is null");
  if (n != mesh->nnodes) return vt_fail(ctx, VT_ERR_INVALID, "n must equal the wide node count");
  if (n) VT_CUDA(ctx, cudaMemcpy(nodes, mesh->d_nodes, n * sizeof(vt_wide_node), cudaMemcpyDeviceToHost));
  return VT_OK;
}

vt_status vt_mesh_get_morton(vt_ctx *ctx, const vt_mesh *mesh, uint32_t *codes, int32_t *sorted, uint32_t n) {
  if (!ctx) return VT_ERR_INVALID;
  if (!mesh || (n && (!codes || !sorted))) return vt_fail(ctx, VT_ERR_INVALID, "null argument");
  if (n != mesh->nfaces) return vt_fail(ctx, VT_ERR_INVALID, "n must equal the face count");
  if (n) {
    VT_CUDA(ctx, cudaMemcpy(codes, mesh->d_codes, n * sizeof(uint32_t), cudaMemcpyDeviceToHost));
    VT_CUDA(ctx, cudaMemcpy(sorted, mesh->d_sorted, n * sizeof(int32_t), cudaMemcpyDeviceToHost));
  }
  return VT_OK;
}

vt_status vt_mesh_get_binary(vt_ctx *ctx, const vt_mesh *mesh, int32_t *children, float *boxes, uint32_t n) {
  if (!ctx) return VT_ERR_INVALID;
  if (!mesh || (n && (!children || !boxes))) return vt_fail(ctx, VT_ERR_INVALID, "null argument");
  uint32_t expect = mesh->nfaces > 1 ? mesh->nfaces - 1 : 0;
  if (n != expect) return vt_fail(ctx, VT_ERR_INVALID, "n must equal faces - 1");
  if (n) {
    VT_CUDA(ctx, cudaMemcpy(children, mesh->d_bin_child, 2 * (size_t)n * sizeof(int32_t), cudaMemcpyDeviceToHost));
    // Device boxes are (lo xyz, pad, hi xyz, pad); the ABI packs 6 floats.
    float *tmp = new float[8 * (size_t)n];
    cudaError_t e = cudaMemcpy(tmp, mesh->d_bin_box, 8 * (size_t)n * sizeof(float), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) { delete[] tmp; return vt_cuda_fail(ctx, e, "cudaMemcpy(binary boxes)"); }
    for (size_t i = 0; i < n; ++i) {
      boxes[6 * i + 0] = tmp[8 * i + 0]; boxes[6 * i + 1] = tmp[8 * i + 1]; boxes[6 * i + 2] = tmp[8 * i + 2];
      boxes[6 * i + 3] = tmp[8 * i + 4]; boxes[6 * i + 4] = tmp[8 * i + 5]; boxes[6 * i + 5] = tmp[8 * i + 6];
    }
    delete[] tmp;
  }
  return VT_OK;
}

// Shared body of the device-buffer entry points.
static vt_status trace_device(vt_ctx *ctx, const vt_mesh *mesh, const vt_ray *rays_dev, uint32_t n, void *out,
                              bool closest, cudaStream_t s) {
  vt_status st = check_trace_args(ctx, mesh, rays_dev, out, n);
  if (st) return st;
  if (n == 0) return VT_OK;
  if (mesh->nfaces == 0) {
    if (closest) k_fill_miss<<<(n + 255) / 256, 256, 0, s>>>(static_cast<int4 *>(out), n);
    else VT_CUDA(ctx, cudaMemsetAsync(out, 0, n, s));
  } else {
    if (closest) vt_launch_closest(mesh, rays_dev, n, static_cast<vt_hit *>(out), ctx->sm_count, vt_queue_slot(ctx), nullptr, ctx->d_status + 1, s);
    else vt_launch_any(mesh, rays_dev, n, static_cast<uint8_t *>(out), ctx->sm_count, vt_queue_slot(ctx), nullptr, ctx->d_status + 1, s);
  }
  VT_CUDA(ctx, cudaGetLastError());
  return VT_OK;
}

vt_status vt_trace_closest(vt_ctx *ctx, const vt_mesh *mesh, const vt_ray *rays_dev, uint32_t n,
                           vt_hit *hits_dev, void *stream) {
  // NULL stream = the CUDA default stream.
  return trace_device(ctx, mesh, rays_dev, n, hits_dev, true, static_cast<cudaStream_t>(stream));
}

vt_status vt_trace_any(vt_ctx *ctx, const vt_mesh *mesh, const vt_ray *rays_dev, uint32_t n,
                       uint8_t *occluded_dev, void *stream) {
  return trace_device(ctx, mesh, rays_dev, n, occluded_dev, false, static_cast<cudaStream_t>(stream));
}

}  // extern "C"

namespace {

// Pinned staging memory for pageable callers (grown as needed) and the slots' events.
vt_status ensure_stage(vt_ctx *ctx, size_t in_bytes, size_t out_bytes) {
  for (cudaEvent_t *ev : {ctx->stage_in_ev, ctx->stage_out_ev})
    for (uint32_t k = 0; k < kStageSlots; ++k)
      if (!ev[k]) VT_CUDA(ctx, cudaEventCreateWithFlags(&ev[k], cudaEventDisableTiming));
  auto grow = [&](void *&p, size_t &have, size_t bytes) -> vt_status {
    if (bytes <= have) return VT_OK;
    cudaFreeHost(p);
    p = nullptr;
    have = 0;
    VT_CUDA(ctx, cudaMallocHost(&p, bytes));
    have = bytes;
    return VT_OK;
  };
  if (vt_status st = grow(ctx->h_stage_in, ctx->stage_in_bytes, in_bytes)) return st;
  return grow(ctx->h_stage_out, ctx->stage_out_bytes, out_bytes);
}

// Host copies beside GPU work on the caller's chunks. copyIn(c, piece) fills chunk c's staging slot
// (c % kStageSlots), issue(c) enqueues its GPU work and records stage_in_ev[slot] after the copy to the
// device and stage_out_ev[slot] after the copy back, copyOut(c, piece) drains the slot. A few threads
// started once per call take the pieces in one order (chunk c's fill, then chunk c - kStageLag's
// drain), waiting for the slot's event where it needs one; the calling thread issues each chunk as soon
// as it is filled and its slot is drained. Every wait is for something earlier in that order.
//
// Bound: host memory (one core copies, and faults in a new output's pages, at a fraction of the link's
// rate) and the link. Below these bytes starting the threads costs more than they save: closest hits of
// 114,544 rays (5.5 MB) 1.29 ms with them and 0.84 without, 180,000 1.14 and 1.12, 250,000 1.17 and 1.44, any hits
// of 250,000 (8.3 MB) 1.16 and 0.96, 500,000 1.45 and 1.49; an image of 13.5 MB 0.7 and 1.85, of 1.5 MB the same.
constexpr size_t kThreadedBytes = 4u << 20, kThreadedRayBytes = 12u << 20;
template <typename In, typename Issue, typename Out>
vt_status host_pipeline(vt_ctx *ctx, bool threads, uint32_t chunks, uint32_t inPieces, uint32_t outPieces, In copyIn, Issue issue, Out copyOut) {
  constexpr uint32_t kMaxWorkers = 8;
  struct Counts {
    std::atomic<uint32_t> in{0}, out{0};
  };
  Counts slots[kStageSlots];             // pieces done of the slot's chunks so far
  std::atomic<uint32_t> next{0}, issued{0};
  std::atomic<int> error{0};             // a cudaError_t of a worker, or -1: the calling thread gave up
  const uint32_t group = inPieces + outPieces;
  const uint64_t items = (uint64_t)(chunks + kStageLag) * group;
  auto wait_issued = [&](uint32_t c) {
    while (issued.load(std::memory_order_acquire) <= c && !error.load(std::memory_order_relaxed)) std::this_thread::yield();
    return !error.load(std::memory_order_relaxed);
  };
  auto synchronize = [&](cudaEvent_t ev) {
    const cudaError_t e = cudaEventSynchronize(ev);
    if (e != cudaSuccess) error = (int)e;
    return e == cudaSuccess;
  };
  auto work = [&] {
    if (const cudaError_t e = cudaSetDevice(ctx->device); e != cudaSuccess) error = (int)e;
    for (uint64_t q; !error.load(std::memory_order_relaxed) && (q = next.fetch_add(1)) < items;) {
      const uint32_t g = (uint32_t)(q / group), piece = (uint32_t)(q % group);
      if (piece < inPieces) {
        if (g >= chunks) continue;
        if (g >= kStageSlots && !(wait_issued(g - kStageSlots) && synchronize(ctx->stage_in_ev[g % kStageSlots]))) return;
        copyIn(g, piece);
        slots[g % kStageSlots].in.fetch_add(1, std::memory_order_release);
      } else {
        if (g < kStageLag) continue;
        const uint32_t c = g - kStageLag;
        if (!wait_issued(c) || !synchronize(ctx->stage_out_ev[c % kStageSlots])) return;
        copyOut(c, piece - inPieces);
        slots[c % kStageSlots].out.fetch_add(1, std::memory_order_release);
      }
    }
  };
  std::thread workers[kMaxWorkers];
  const uint32_t want = !threads ? 1u : std::min<uint32_t>({kMaxWorkers, std::max(1u, std::thread::hardware_concurrency()), chunks * std::max(inPieces, outPieces)});
  uint32_t started = 0;
  if (want > 1) {
    try {
      for (; started < want; ++started) workers[started] = std::thread(work);
    } catch (...) {  // no more threads: the ones there are do the work
    }
  }
  vt_status st = VT_OK;
  if (started == 0) {
    for (uint32_t c = 0; c < chunks && !st; ++c) {
      for (uint32_t p = 0; p < inPieces; ++p) copyIn(c, p);
      st = issue(c);
      if (!st && !synchronize(ctx->stage_out_ev[c % kStageSlots])) break;
      for (uint32_t p = 0; p < outPieces && !st; ++p) copyOut(c, p);
    }
  } else {
    for (uint32_t c = 0; c < chunks && !st && !error.load(); ++c) {
      const Counts &slot = slots[c % kStageSlots];
      const uint32_t turn = c / kStageSlots;
      while ((slot.in.load(std::memory_order_acquire) < (turn + 1) * inPieces || slot.out.load(std::memory_order_acquire) < turn * outPieces) &&
             !error.load(std::memory_order_relaxed))
        std::this_thread::yield();
      if (error.load()) break;
      st = issue(c);
      if (st) error = -1;
      else issued.store(c + 1, std::memory_order_release);
    }
    for (uint32_t k = 0; k < started; ++k) workers[k].join();
  }
  if (!st && error > 0) st = vt_cuda_fail(ctx, (cudaError_t)error.load(), "host copy pipeline");
  return st;
}

// Whether a host pointer is ordinary (pageable) memory rather than pinned or registered memory.
bool pageable(const void *p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return true;
  }
  return a.type == cudaMemoryTypeUnregistered;
}

// A host copy split over a few threads from 8 MB on (a call of one chunk).
void copy_parallel(void *dst, const void *src, size_t bytes) {
  const size_t parts = std::min<size_t>(std::max(1u, std::thread::hardware_concurrency()), std::max<size_t>(1, bytes >> 22));
  const size_t step = (bytes + parts - 1) / parts;
  std::vector<std::thread> workers;
  size_t done = step;  // [0, step) is this thread's
  try {
    for (; done < bytes; done += step)
      workers.emplace_back([=] { std::memcpy(static_cast<char *>(dst) + done, static_cast<const char *>(src) + done, std::min(step, bytes - done)); });
  } catch (...) {  // no more threads
    std::memcpy(static_cast<char *>(dst) + done, static_cast<const char *>(src) + done, bytes - done);
  }
  std::memcpy(dst, src, std::min(step, bytes));
  for (auto &w : workers) w.join();
}

// Rays of one chunk of the pageable pipeline with threads: a sixth of the call, so that copies in,
// traversal and copies out overlap, but at least 128K (a traversal that fills the GPU; fewer bytes than
// the link's latency is worth) and at most 1M (the slots' pinned memory). Without: the whole call.
uint32_t stage_chunk(uint32_t n) {
  return std::min(n, std::min(1u << 20, std::max(1u << 17, ((n + 5) / 6 + 1023) & ~1023u)));
}

// dst = src x scale for n doubles on the device, to host memory; the device is idle and current. Pageable memory
// goes through the staging slots, scaled by the threads that drain them. Measured on one B200: the
// 50 MB of a 1920 x 1080 image 14.5 -> 3.6 ms, the 13.5 MB of 1001 x 563 1.85 -> 0.7 (one copy into the
// caller's pages by the driver, then a scaling pass by one core).
vt_status read_scaled(vt_ctx *ctx, double *dst, const double *src, size_t n, double scale) {
  constexpr size_t kPiece = kStagePiece / sizeof(double);
  if (n * sizeof(double) < kThreadedBytes || !pageable(dst)) {
    if (n) VT_CUDA(ctx, cudaMemcpy(dst, src, n * sizeof(double), cudaMemcpyDeviceToHost));
    for (size_t i = 0; i < n; ++i) dst[i] *= scale;
    return VT_OK;
  }
  if (vt_status st = ensure_stage(ctx, 0, kStageSlots * kStagePiece)) return st;
  const auto words = [&](uint32_t c) { return std::min(kPiece, n - c * kPiece); };
  const auto slot_of = [&](uint32_t c) { return static_cast<double *>(ctx->h_stage_out) + (c % kStageSlots) * kPiece; };
  return host_pipeline(
      ctx, true, (uint32_t)((n + kPiece - 1) / kPiece), 0, 1, [](uint32_t, uint32_t) {},
      [&](uint32_t c) -> vt_status {
        VT_CUDA(ctx, cudaMemcpyAsync(slot_of(c), src + c * kPiece, words(c) * sizeof(double), cudaMemcpyDeviceToHost, ctx->pipe[0]));
        VT_CUDA(ctx, cudaEventRecord(ctx->stage_out_ev[c % kStageSlots], ctx->pipe[0]));
        return VT_OK;
      },
      [&](uint32_t c, uint32_t) {
        const double *from = slot_of(c);
        double *to = dst + c * kPiece;
        for (size_t i = 0, m = words(c); i < m; ++i) to[i] = from[i] * scale;
      });
}

}  // namespace

extern "C" {

// Host pipeline: chunk c goes on stream c % 2 as copy-in, trace, copy-out; the two streams let
// chunk c + 1's copy-in and chunk c - 1's copy-out overlap chunk c's traversal. Pageable buffers go
// through pinned staging, filled and drained by several host threads (host_pipeline) from 12 MB on. Measured
// on one B200's host, closest hits of rays in ordinary arrays on 200,000 triangles into a new result array:
// 1,000,003 rays 4.0-4.7 -> 2.2-2.6 ms, 4M 15-17 -> 8-11, and whole below, 200,000 1.1 as before (chunks of 4M rays
// with two slots and threads started per copy left nothing to overlap below 8M).
static vt_status trace_host(vt_ctx *ctx, const vt_mesh *mesh, const vt_ray *rays, uint32_t n,
                            void *out, size_t out_stride, bool closest) {
  vt_status st = check_trace_args(ctx, mesh, rays, out, n);
  if (st) return st;
  VT_CUDA(ctx, cudaSetDevice(ctx->device));
  if (n == 0) return VT_OK;
  const bool staged = pageable(rays) || pageable(out);
  const bool threads = n * (sizeof(vt_ray) + out_stride) >= kThreadedRayBytes;
  const uint32_t chunk = staged && threads ? stage_chunk(n) : n < kChunk ? n : kChunk;
  st = ensure_chunks(ctx, (size_t)chunk * sizeof(vt_ray), (size_t)chunk * out_stride);
  if (st) return st;
  // The previous user of these buffers may still be in flight on the other stream.
  VT_CUDA(ctx, cudaStreamSynchronize(ctx->pipe[0]));
  VT_CUDA(ctx, cudaStreamSynchronize(ctx->pipe[1]));
  if (staged) {
    const size_t in_slot = (size_t)chunk * sizeof(vt_ray), out_slot = (size_t)chunk * out_stride;
    const uint32_t slots = threads ? kStageSlots : 1u;
    st = ensure_stage(ctx, slots * in_slot, slots * out_slot);
    if (st) return st;
    const size_t in_size = threads ? kStagePiece : in_slot, out_size = threads ? kStagePiece : out_slot;
    const uint32_t in_pieces = (uint32_t)((in_slot + in_size - 1) / in_size), out_pieces = (uint32_t)((out_slot + out_size - 1) / out_size);
    const auto rays_of = [&](uint32_t c) { return std::min(chunk, n - c * chunk); };
    const auto copy_piece = [](char *dst, const char *src, size_t bytes, uint32_t piece, size_t size) {
      const size_t at = std::min(bytes, piece * size);
      copy_parallel(dst + at, src + at, std::min(bytes - at, size));
    };
    return host_pipeline(
        ctx, threads, (n + chunk - 1) / chunk, in_pieces, out_pieces,
        [&](uint32_t c, uint32_t piece) {
          copy_piece(static_cast<char *>(ctx->h_stage_in) + (c % kStageSlots) * in_slot,
                     reinterpret_cast<const char *>(rays + (size_t)c * chunk), rays_of(c) * sizeof(vt_ray), piece, in_size);
        },
        [&](uint32_t c) -> vt_status {
          const int k = c & 1;
          const uint32_t m = rays_of(c), slot = c % kStageSlots;
          cudaStream_t s = ctx->pipe[k];
          VT_CUDA(ctx, cudaMemcpyAsync(ctx->d_chunk_in[k], static_cast<char *>(ctx->h_stage_in) + slot * in_slot, (size_t)m * sizeof(vt_ray),
                                       cudaMemcpyHostToDevice, s));
          VT_CUDA(ctx, cudaEventRecord(ctx->stage_in_ev[slot], s));
          const vt_status t = trace_device(ctx, mesh, static_cast<const vt_ray *>(ctx->d_chunk_in[k]), m, ctx->d_chunk_out[k], closest, s);
          if (t) return t;
          VT_CUDA(ctx, cudaMemcpyAsync(static_cast<char *>(ctx->h_stage_out) + slot * out_slot, ctx->d_chunk_out[k], (size_t)m * out_stride,
                                       cudaMemcpyDeviceToHost, s));
          VT_CUDA(ctx, cudaEventRecord(ctx->stage_out_ev[slot], s));
          return VT_OK;
        },
        [&](uint32_t c, uint32_t piece) {
          copy_piece(static_cast<char *>(out) + (size_t)c * chunk * out_stride, static_cast<const char *>(ctx->h_stage_out) + (c % kStageSlots) * out_slot,
                     rays_of(c) * out_stride, piece, out_size);
        });
  }
  for (uint32_t c = 0, first = 0; first < n; ++c, first += chunk) {
    const uint32_t m = n - first < chunk ? n - first : chunk;
    const int k = c & 1;
    cudaStream_t s = ctx->pipe[k];
    VT_CUDA(ctx, cudaMemcpyAsync(ctx->d_chunk_in[k], rays + first, (size_t)m * sizeof(vt_ray),
                                 cudaMemcpyHostToDevice, s));
    const vt_ray *dr = static_cast<const vt_ray *>(ctx->d_chunk_in[k]);
    st = trace_device(ctx, mesh, dr, m, ctx->d_chunk_out[k], closest, s);
    if (st) return st;
    VT_CUDA(ctx, cudaMemcpyAsync(static_cast<char *>(out) + (size_t)first * out_stride, ctx->d_chunk_out[k],
                                 (size_t)m * out_stride, cudaMemcpyDeviceToHost, s));
  }
  VT_CUDA(ctx, cudaStreamSynchronize(ctx->pipe[0]));
  VT_CUDA(ctx, cudaStreamSynchronize(ctx->pipe[1]));
  return VT_OK;
}

vt_status vt_trace_closest_host(vt_ctx *ctx, const vt_mesh *mesh, const vt_ray *rays, uint32_t n,
                                vt_hit *hits) {
  return trace_host(ctx, mesh, rays, n, hits, sizeof(vt_hit), true);
}

vt_status vt_trace_any_host(vt_ctx *ctx, const vt_mesh *mesh, const vt_ray *rays, uint32_t n,
                            uint8_t *occluded) {
  return trace_host(ctx, mesh, rays, n, occluded, 1, false);
}

vt_status vt_accum_readback(vt_ctx *ctx, vt_scene *scene, double *rgb, uint32_t n, uint32_t *samples) {
  if (!ctx) return VT_ERR_INVALID;
  if (!scene || !rgb) return vt_fail(ctx, VT_ERR_INVALID, "scene or rgb is null");
  const size_t want = 3 * (size_t)scene->width * scene->height;
  if (n != want) return vt_fail(ctx, VT_ERR_INVALID, "n must equal width * height * 3");
  // The synchronisation and the staging events below are the current device's, which another context's
  // call may have left elsewhere.
  VT_CUDA(ctx, cudaSetDevice(ctx->device));
  VT_CUDA(ctx, cudaDeviceSynchronize());
  {
    uint32_t w[16];
    VT_CUDA(ctx, cudaMemcpy(w, ctx->d_status, sizeof w, cudaMemcpyDeviceToHost));
    if (w[1] & VT_DEV_STACK) {
      VT_CUDA(ctx, cudaMemset(ctx->d_status + 1, 0, sizeof(uint32_t)));
      return vt_fail(ctx, VT_ERR_DEVICE, "a traversal stack would have overflowed; the entries were dropped");
    }
    if (w[2]) {
      VT_CUDA(ctx, cudaMemset(ctx->d_status + 2, 0, sizeof(uint32_t)));
      VT_CUDA(ctx, cudaMemset(ctx->d_status + 8, 0, 3 * sizeof(uint32_t)));
      return vt_fail(ctx, VT_ERR_DEVICE,
                     "the integrator met an out-of-range index (status " + std::to_string(w[2]) +
                         ": 4 hit, 8 cache record, 16 emitter face; first: value " + std::to_string(w[9]) +
                         ", kernel " + std::to_string(w[10] & 0xffu) + "); those accesses were clamped or skipped");
    }
  }
  if (vt_status st = read_scaled(ctx, rgb, scene->d_accum, want, scene->samples ? 1.0 / scene->samples : 0.0)) return st;
  if (samples) *samples = scene->samples;
  return VT_OK;
}

vt_status vt_trace_count(vt_ctx *ctx, const vt_mesh *mesh, const vt_ray *rays_dev, uint32_t n,
                         int32_t closest, uint64_t *nodes_visited, uint64_t *tris_tested) {
  vt_status st = check_trace_args(ctx, mesh, rays_dev, nodes_visited, n);
  if (st) return st;
  if (!tris_tested) return vt_fail(ctx, VT_ERR_INVALID, "tris_tested is null");
  *nodes_visited = 0;
  *tris_tested = 0;
  if (n == 0 || mesh->nfaces == 0) return VT_OK;
  unsigned long long *acc = vt_count_words(ctx);
  VT_CUDA(ctx, cudaMemsetAsync(acc, 0, 2 * sizeof(unsigned long long), ctx->stream));
  vt_launch_count(mesh, rays_dev, n, closest, acc, ctx->stream);
  VT_CUDA(ctx, cudaGetLastError());
  unsigned long long h[2];
  VT_CUDA(ctx, cudaMemcpyAsync(h, acc, sizeof h, cudaMemcpyDeviceToHost, ctx->stream));
  VT_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  *nodes_visited = h[0];
  *tris_tested = h[1];
  return VT_OK;
}

}  // extern "C"
