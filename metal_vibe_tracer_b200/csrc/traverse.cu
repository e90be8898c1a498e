// traverse.cu — closest-hit and any-hit traversal of the 4-wide BVH with the watertight
// triangle test.
//
// Reference: blas_closest / blas_any (main.swift:1788-1838), wide_ray / wide_node_hit /
// wide_order (main.swift:1758-1785), watertight_ray / watertight_edge / intersect_mesh_triangle
// (main.swift:1536-1582).
//
// Layout: a node is the 64-byte quantised copy of the reference's MeshWideNode (qnode.cu), fetched as two
// 32-byte vector loads; a triangle is three float4 in BVH order (vertex a carries the input face index
// in .w, vertex c the mark of its leaf's last triangle), 48 bytes fetched as three 16-byte loads. The
// whole structure of a 1M-triangle mesh (19 MB nodes + 48 MB triangles) sits in the 126 MB L2.
//
// The watertight arithmetic is written with explicitly rounded intrinsics in one fixed order
// (each product and sum rounded on its own; the exact FMA fallback on edge ties), which the CPU
// oracle reproduces, so hits compare bit for bit.
#include <algorithm>

#include "trace_common.cuh"
#include "vt_internal.cuh"

namespace {
using namespace vtd;

// ---- persistent traversal -----------------------------------------------------------------------
// Rays vary a lot in length (65 node visits on average for the incoherent set, with a long tail), so
// a thread-per-ray grid leaves most lanes of a warp idle while its longest ray finishes.
// Persistent traversal (k_closest, k_any): each warp stays resident and refills idle lanes from a
// global ray counter: one warp-aggregated atomicAdd hands out as many rays as there are idle lanes,
// whenever at least kRefill lanes are idle. Each loop iteration handles one stack entry per active
// lane (a node visit or a leaf's triangles) with the per-ray order of the single-ray form, so
// the hits equal those of the single-ray form bit for bit. Rays are read and hits written with
// streaming cache hints so that the ray stream does not evict the BVH from L2.
//
// Bound: issue (ALU) and the latency of dependent loads, not bandwidth. A node visit goes straight on to
// its nearest hit child, kept in a register, and a warp in its node phase takes up to kSteps nodes per
// lane before it votes again (a vote costs about a tenth of a visit, and the lanes that meet a leaf
// earlier wait): of 1, 2, 3, 4, 8 and 16 steps, 4 (closest) and 2 (any hit) measured best. The node
// test's keys, links and steps are laid out so that a visit needs no index arithmetic (qnode.cu).
// 8 and 9 blocks per SM (64 and 56 registers) beat 5 to 7 and 10: the loads' latency needs the warps.
// Measured on one B200, 1M-triangle soup: closest hit of 4M random rays 5.30 -> 4.17 ms, any hit
// 3.55 -> 2.92 ms; 1080p camera rays 1.37 -> 1.12 and 0.75 -> 0.66 ms; 4,096 rays on 20,000 triangles
// 110 -> 93 us. Tried and dropped: entry distances on the stack to drop entries beyond a closer hit
// unvisited (5.76 against 5.20 ms: the larger stacks cost more L1 than the visits saved), loading the
// next node before pushing the others (5.11 against 4.26 ms).
//
// Few rays (lanes_used) go one or two to a warp: a ray then waits for no others' node and leaf phases, and the
// chip has room. Measured on one B200 (the whole call): 4,096 rays on 20,000 triangles, closest hit
// 90 -> 79 us and any hit 72 -> 58; 1,000 rays on 1M triangles 237 -> 184 and 167 -> 111. Spread further it
// loses: 20,000 rays on 16 warps an SM 99 -> 112 us, on 8 108, on 4 107.
constexpr unsigned kFull = 0xffffffffu;
// Refill once this many lanes are idle (measured at 4, 8, 12 and 16).
constexpr int kRefill = 4, kRefillAny = 8;
constexpr int kSteps = 4, kStepsAny = 2;  // nodes per lane between votes
constexpr int kBlock = 128;
constexpr int kMinBlocks = 8, kMinBlocksAny = 9;  // register budget: 65536 / (kBlock * blocks)

// The rays of a launch and where the results go: perm (null: all rays in order) lists the rays, count (when
// not null) holds the list's length on the device (at most n), counter the next to hand out.
template <typename Out>
struct RaySet {
  const float4 *rays;
  uint32_t n;
  Out *out;
  uint32_t *counter;
  const uint32_t *perm, *count;
  uint32_t sms;
};

// Lanes of each warp that take rays (kFew: a launch of possibly few rays): one or two while that gives every
// ray of the launch a place in kFewWarps warps an SM, else all.
constexpr uint32_t kFewWarps = 16, kFewLanes = 2;
template <bool kFew>
__device__ __forceinline__ unsigned lanes_used(uint32_t n, uint32_t sms) {
  if (!kFew) return kFull;
  const uint32_t warps = min(gridDim.x * (kBlock / 32u), sms * kFewWarps), lanes = (n + warps - 1u) / warps;
  return lanes > kFewLanes ? kFull : (1u << lanes) - 1u;
}

struct RayState {
  WRay wr;
  QRay qr;
  float tMin, tMax;
};

__device__ __forceinline__ void load_ray(const float4 *__restrict__ rays, uint32_t r, RayState &s,
                                         float rootMax) {
  const float4 r0 = __ldcs(rays + 2 * (size_t)r), r1 = __ldcs(rays + 2 * (size_t)r + 1);
  s.wr = make_wray(r0.x, r0.y, r0.z, r1.x, r1.y, r1.z);
  s.qr = make_qray(r0.x, r0.y, r0.z, r1.x, r1.y, r1.z, rootMax);
  s.tMin = r0.w;
  s.tMax = r1.w;
}

// Hands rays [base, base + idle lanes) to the idle lanes of the warp. Returns the lane's ray
// index, or n if it got none; *exhausted is set (warp-uniformly) once the pool is empty.
__device__ __forceinline__ uint32_t refill(unsigned idle, uint32_t *counter, uint32_t n, bool &exhausted) {
  const unsigned lane = threadIdx.x & 31u;
  uint32_t base = 0;
  if (lane == 0) base = atomicAdd(counter, (uint32_t)__popc(idle));
  base = __shfl_sync(kFull, base, 0);
  if (base + (uint32_t)__popc(idle) >= n) exhausted = true;
  const uint32_t r = base + (uint32_t)__popc(idle & ((1u << lane) - 1u));
  return (idle >> lane & 1u) && r < n ? r : n;
}

// The traversal stack lives in shared memory, one column per thread: entry d of thread t is
// word d * kBlock + t, so every lane of a warp hits its own bank whatever its stack depth.
__device__ __forceinline__ int *stack_slot(int *sstack, int d) { return sstack + d * kBlock + threadIdx.x; }

// Entries: an inner node is its index (>= 0), a leaf ~(its first triangle); kIdle marks a lane
// without a ray. A lane's current entry stays in a register: a node visit goes straight on to its
// nearest hit child and pushes only the others.
constexpr int kIdle = 0x7fffffff;

// Per lane, one iteration handles the current entry: a node visit (its hit children, leaves
// included, near first) or one leaf's triangle tests. The warp runs only the kind more of its lanes
// need this iteration; the others wait one iteration. A ray's own order (LIFO over its stack) does
// not depend on the warp.
// kPos: a hit reports the triangle's BVH position instead of its input face (the integrator's
// hit record).
template <bool kPos, bool kFew>
__device__ __forceinline__ void closest_rays(const float4 *__restrict__ nodes, const float4 *__restrict__ tris, float rootMax,
                                             const RaySet<int4> &R, int stackSize, uint32_t *status, int *sstack) {
  const uint32_t n = R.count ? min(R.n, *R.count) : R.n;
  const unsigned mine = lanes_used<kFew>(n, R.sms);  // of this warp
  int cur = kIdle, top = 0;
  uint32_t rid = 0;
  RayState s;
  float closest = 0.0f, hb1 = 0.0f, hb2 = 0.0f;
  int prim = -1;
  bool exhausted = false;  // warp-uniform
  while (true) {
    const unsigned idle = __ballot_sync(kFull, cur == kIdle) & mine;
    if (!exhausted && (__popc(idle) >= kRefill || (kFew && idle == mine))) {
      const uint32_t r = refill(idle, R.counter, n, exhausted);
      if (r < n) {
        rid = R.perm ? __ldcs(R.perm + r) : r;
        load_ray(R.rays, rid, s, rootMax);
        s.tMin = __fadd_rn(s.tMin, 0.0f);  // -0 to +0 (sort_qchildren)
        closest = s.tMax;
        prim = -1;
        cur = 0;
        top = 0;
      }
    }
    const bool leaf = cur < 0;
    const unsigned leaves = __ballot_sync(kFull, leaf), active = __ballot_sync(kFull, cur != kIdle);
    if (exhausted && active == 0u) break;
    const bool leafPhase = 2 * __popc(leaves) >= __popc(active);
    if (cur == kIdle || leaf != leafPhase) continue;
    auto pop = [&] { cur = top > 0 ? *stack_slot(sstack, --top) : kIdle; };
    if (leaf) {
      if (cur != kEmptyChild) {
        int at = ~cur;
        const float4 *tp = tris + 3 * (size_t)at;
        for (int q = 0; q < kMaxLeafTris; ++q, tp += 3, ++at) {
          const float4 a = __ldg(tp), b = __ldg(tp + 1), cc = __ldg(tp + 2);
          float t, b1, b2;
          if (intersect_tri(s.wr, a, b, cc, s.tMin, closest, t, b1, b2)) {
            closest = t; hb1 = b1; hb2 = b2; prim = kPos ? at : __float_as_int(a.w);
          }
          if (leaf_ends(cc)) break;
        }
      }
      pop();
    } else {
      QNode nd;
      load_qnode(nodes, cur, nd);
#pragma unroll 1
      for (int step = 1;; ++step) {
        float nearT[4];
        bool hit[4];
        uint32_t key[4];
        qnode_test(nd, s.qr, s.tMin, closest, nearT, hit);
        sort_qchildren(hit, nearT, s.tMin >= 0.0f, key);
        // At most three pushes per level of the tree: a full stack means a corrupted tree.
        if (top + 3 > stackSize) {
          atomicOr(status, (uint32_t)VT_DEV_STACK);
          top = stackSize - 3;
        }
#pragma unroll
        for (int j = 3; j >= 1; --j) {
          if (key[j] == kMissKey) continue;
          *stack_slot(sstack, top++) = pick4(nd.child, key[j] & 3u);
        }
        if (key[0] != kMissKey) cur = pick4(nd.child, key[0] & 3u);
        else pop();
        if (cur < 0 || cur == kIdle || step >= kSteps) break;
        load_qnode(nodes, cur, nd);
      }
    }
    if (cur == kIdle) {
      const int4 out = prim >= 0 ? make_int4(__float_as_int(closest), __float_as_int(hb1), __float_as_int(hb2), prim)
                                 : make_int4(0, 0, 0, -1);
      __stcs(R.out + rid, out);
    }
  }
}

// kSlack: each triangle's own rounding bound comes off tmax (the integrator's shadow rays in
// imported scenes, scene_occluded main.swift:2066-2069).
template <bool kSlack, bool kFew>
__device__ __forceinline__ void any_rays(const float4 *__restrict__ nodes, const float4 *__restrict__ tris, float rootMax,
                                         const RaySet<uint8_t> &R, int stackSize, uint32_t *status, int *sstack) {
  const uint32_t n = R.count ? min(R.n, *R.count) : R.n;
  const unsigned mine = lanes_used<kFew>(n, R.sms);  // of this warp
  int cur = kIdle, top = 0;
  uint32_t rid = 0;
  RayState s;
  bool exhausted = false;
  while (true) {
    const unsigned idle = __ballot_sync(kFull, cur == kIdle) & mine;
    if (!exhausted && (__popc(idle) >= kRefillAny || (kFew && idle == mine))) {
      const uint32_t r = refill(idle, R.counter, n, exhausted);
      if (r < n) {
        rid = R.perm ? __ldcs(R.perm + r) : r;
        load_ray(R.rays, rid, s, rootMax);
        cur = 0;
        top = 0;
      }
    }
    const bool leaf = cur < 0;
    const unsigned leaves = __ballot_sync(kFull, leaf), active = __ballot_sync(kFull, cur != kIdle);
    if (exhausted && active == 0u) break;
    const bool leafPhase = 2 * __popc(leaves) >= __popc(active);
    if (cur == kIdle || leaf != leafPhase) continue;
    bool hit = false;
    auto pop = [&] { cur = top > 0 ? *stack_slot(sstack, --top) : kIdle; };
    if (leaf) {
      if (cur != kEmptyChild) {
        const float4 *tp = tris + 3 * (size_t)(~cur);
        for (int q = 0; q < kMaxLeafTris; ++q, tp += 3) {
          const float4 a = __ldg(tp), b = __ldg(tp + 1), cc = __ldg(tp + 2);
          float t, b1, b2;
          const float tMax = kSlack ? s.tMax - tri_error_bound(a, b, cc) : s.tMax;
          if (intersect_tri(s.wr, a, b, cc, s.tMin, tMax, t, b1, b2)) { hit = true; break; }
          if (leaf_ends(cc)) break;
        }
      }
      if (hit) cur = kIdle;
      else pop();
    } else {
#pragma unroll 1
      for (int step = 0; step < kStepsAny; ++step) {
        QNode nd;
        load_qnode(nodes, cur, nd);
        float nearT[4];
        bool meets[4];
        qnode_test(nd, s.qr, s.tMin, s.tMax, nearT, meets);
        if (top + 3 > stackSize) {
          atomicOr(status, (uint32_t)VT_DEV_STACK);
          top = stackSize - 3;
        }
        int next = kIdle;
#pragma unroll
        for (int k = 3; k >= 0; --k) {
          if (!meets[k]) continue;
          if (next != kIdle) *stack_slot(sstack, top++) = next;
          next = i4(nd.child, k);
        }
        if (next != kIdle) cur = next;
        else pop();
        if (cur < 0 || cur == kIdle) break;
      }
    }
    if (cur == kIdle) R.out[rid] = hit ? 1 : 0;
  }
}

template <bool kPos, bool kFew>
__global__ void __launch_bounds__(kBlock, kMinBlocks) k_closest(const float4 *__restrict__ nodes, const float4 *__restrict__ tris,
                                                                float rootMax, const __grid_constant__ RaySet<int4> R, int stackSize, uint32_t *status) {
  extern __shared__ int sstack[];
  closest_rays<kPos, kFew>(nodes, tris, rootMax, R, stackSize, status, sstack);
}
template <bool kSlack, bool kFew>
__global__ void __launch_bounds__(kBlock, kMinBlocksAny) k_any(const float4 *__restrict__ nodes, const float4 *__restrict__ tris,
                                                               float rootMax, const __grid_constant__ RaySet<uint8_t> R, int stackSize, uint32_t *status) {
  extern __shared__ int sstack[];
  any_rays<kSlack, kFew>(nodes, tris, rootMax, R, stackSize, status, sstack);
}

// A bounce's shadow rays and the next bounce's rays in one launch (the integrator's stages): even blocks
// begin with the one, odd blocks with the other, and whoever is done helps with the rest. Either set
// alone ends in a few long rays while most of the chip idles (some 100 us a launch). Measured on one B200, device
// time of whole frames: 1080p production of 4 samples 18.9 -> 17.5 ms, four 1001 x 563 ReSTIR frames
// 16.7 -> 15.6, a 1000 x 600 Lambert frame 4.66 -> 4.27. (7 blocks an SM instead of 8: the same.)
template <bool kSlack>
__global__ void __launch_bounds__(kBlock, kMinBlocks) k_closest_any(const float4 *__restrict__ nodes, const float4 *__restrict__ tris,
                                                                    float rootMax, const __grid_constant__ RaySet<int4> C,
                                                                    const __grid_constant__ RaySet<uint8_t> O, int stackSize,
                                                                    uint32_t *status) {
  extern __shared__ int sstack[];
#pragma unroll 1
  for (uint32_t turn = 0; turn < 2u; ++turn) {
    if ((turn ^ blockIdx.x) & 1u) any_rays<kSlack, true>(nodes, tris, rootMax, O, stackSize, status, sstack);
    else closest_rays<true, true>(nodes, tris, rootMax, C, stackSize, status, sstack);
  }
}

__global__ void __launch_bounds__(128) k_count(const float4 *__restrict__ nodes,
                                                const float4 *__restrict__ tris, float rootMax,
                                                const float4 *__restrict__ rays, uint32_t n,
                                                int closest, unsigned long long *acc) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t nv = 0, nt = 0;
  if (i < n) {
    const float4 r0 = __ldg(rays + 2 * (size_t)i), r1 = __ldg(rays + 2 * (size_t)i + 1);
    if (closest) {
      count_closest(nodes, tris, rootMax, r0, r1, nv, nt);
    } else {
      count_any(nodes, tris, rootMax, r0, r1, nv, nt);
    }
  }
  unsigned long long a = nv, b = nt;
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(acc, a);
    atomicAdd(acc + 1, b);
  }
}

}  // namespace

namespace {
// Stack entries a traversal of a tree of `depth` levels needs: a visit goes on to one child and
// pushes at most three.
inline int stack_entries(uint32_t depth) { return 3 * (int)depth; }

// Launches a persistent traversal of n rays: a warp per ray where they are few (lanes_used), else per 32, and as
// many blocks as fit the chip; `smem` bytes of stacks in each. (With a warp per ray whatever the count,
// the idle warps' draws on the ray counter cost 20,000 rays 9 us and 65,536 19 us.)
template <typename K, typename... Args>
void launch_persistent(K kernel, const vt_mesh *mesh, uint64_t n, bool few, int sm_count, cudaStream_t s, uint32_t *status, Args... rays) {
  const int S = stack_entries(mesh->depth);
  const size_t smem = (size_t)S * kBlock * sizeof(int);
  if (smem > 48 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  int resident = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, kernel, kBlock, smem) != cudaSuccess || resident < 1) resident = 1;
  const uint64_t perBlock = (kBlock / 32) * (few ? 1u : 32u);
  const uint32_t grid = (uint32_t)std::min<uint64_t>((n + perBlock - 1) / perBlock, (uint64_t)resident * sm_count);
  kernel<<<grid, kBlock, smem, s>>>(reinterpret_cast<const float4 *>(mesh->d_qnodes), mesh->d_tris, mesh->root_max, rays..., S, status);
}
template <typename Out, typename T>
RaySet<Out> ray_set(const vt_ray *rays, uint32_t n, T *out, uint32_t *counter, const uint32_t *perm, const uint32_t *count, int sm_count) {
  return {reinterpret_cast<const float4 *>(rays), n, reinterpret_cast<Out *>(out), counter, perm, count, (uint32_t)sm_count};
}
}  // namespace

void vt_launch_closest(const vt_mesh *mesh, const vt_ray *rays, uint32_t n, vt_hit *hits, int sm_count,
                       uint32_t *counter, const uint32_t *perm, uint32_t *status, cudaStream_t s,
                       const uint32_t *count, bool bvhPos, bool cleared) {
  if (n == 0) return;
  if (!cleared) cudaMemsetAsync(counter, 0, sizeof(uint32_t), s);
  const bool small = n <= kFewLanes * kFewWarps * (uint32_t)sm_count, few = count || small;
  launch_persistent(bvhPos ? (few ? k_closest<true, true> : k_closest<true, false>) : few ? k_closest<false, true> : k_closest<false, false>, mesh, n, small, sm_count, s, status,
                    ray_set<int4>(rays, n, hits, counter, perm, count, sm_count));
}

void vt_launch_any(const vt_mesh *mesh, const vt_ray *rays, uint32_t n, uint8_t *occ, int sm_count,
                   uint32_t *counter, const uint32_t *perm, uint32_t *status, cudaStream_t s,
                   const uint32_t *count, bool slack, bool cleared) {
  if (n == 0) return;
  if (!cleared) cudaMemsetAsync(counter, 0, sizeof(uint32_t), s);
  const bool small = n <= kFewLanes * kFewWarps * (uint32_t)sm_count, few = count || small;
  // (Shadow rays with slack come from queues only, so they need no form for a launch of many rays.)
  launch_persistent(slack ? k_any<true, true> : few ? k_any<false, true> : k_any<false, false>, mesh, n, small, sm_count, s, status,
                    ray_set<uint8_t>(rays, n, occ, counter, perm, count, sm_count));
}

void vt_launch_closest_any(const vt_mesh *mesh, const vt_ray_queue &closest, vt_hit *hits, const vt_ray_queue &any, uint8_t *occ,
                           uint32_t n, int sm_count, uint32_t *status, cudaStream_t s, bool slack) {
  if (n == 0) return;
  launch_persistent(slack ? k_closest_any<true> : k_closest_any<false>, mesh, 2 * (uint64_t)n, n <= 2u * kFewLanes * kFewWarps * (uint32_t)sm_count,
                    sm_count, s, status,
                    ray_set<int4>(closest.rays, n, hits, closest.head, closest.list, closest.count, sm_count),
                    ray_set<uint8_t>(any.rays, n, occ, any.head, any.list, any.count, sm_count));
}

void vt_launch_count(const vt_mesh *mesh, const vt_ray *rays, uint32_t n, int closest,
                     unsigned long long *acc, cudaStream_t s) {
  if (n == 0) return;
  k_count<<<(n + 127) / 128, 128, 0, s>>>(reinterpret_cast<const float4 *>(mesh->d_qnodes), mesh->d_tris,
                                         mesh->root_max, reinterpret_cast<const float4 *>(rays), n,
                                         closest, acc);
}
