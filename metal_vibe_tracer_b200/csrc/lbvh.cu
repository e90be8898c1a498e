// lbvh.cu — GPU acceleration-structure build: LBVH (30-bit Morton codes, stable radix sort,
// Karras hierarchy), bottom-up refit, SAH treelet restructuring and the collapse to the
// reference's 4-wide node layout (MeshWideNode, main.swift:617; Sources/Acceleration.swift:23-30).
//
// Replaces the reference's CPU binned-SAH WideBVH.build (Sources/Acceleration.swift:106-352).
// Every arithmetic step that decides topology is written with explicitly rounded intrinsics
// (__fadd_rn, __fmul_rn, __fdiv_rn) so the CPU oracle (oracle/vt_oracle.cpp, built with
// -ffp-contract=off) reproduces Morton codes, sorted order and topology bit for bit.
#include <algorithm>
#include <cfloat>
#include <climits>
#include <vector>

#include "vt_internal.cuh"

namespace {

constexpr float kCi = 1.2f, kCt = 1.0f;  // treelet costs: internal node, triangle
constexpr int kMaxTreelet = 8;

struct Box { float3 lo, hi; };

__device__ __forceinline__ float box_area(float3 lo, float3 hi) {
  float ex = fmaxf(__fsub_rn(hi.x, lo.x), 0.0f), ey = fmaxf(__fsub_rn(hi.y, lo.y), 0.0f),
        ez = fmaxf(__fsub_rn(hi.z, lo.z), 0.0f);
  return __fadd_rn(__fadd_rn(__fmul_rn(ex, ey), __fmul_rn(ey, ez)), __fmul_rn(ez, ex));
}
__device__ __forceinline__ Box box_union(const Box &a, const Box &b) {
  return {make_float3(fminf(a.lo.x, b.lo.x), fminf(a.lo.y, b.lo.y), fminf(a.lo.z, b.lo.z)),
          make_float3(fmaxf(a.hi.x, b.hi.x), fmaxf(a.hi.y, b.hi.y), fmaxf(a.hi.z, b.hi.z))};
}
// Boxes live as two float4 (lo.xyz, hi.xyz). L2 loads (.cg) because other threads of the same
// launch write them in the bottom-up passes.
__device__ __forceinline__ Box load_box_cg(const float4 *b, int i) {
  float4 l = __ldcg(b + 2 * i), h = __ldcg(b + 2 * i + 1);
  return {make_float3(l.x, l.y, l.z), make_float3(h.x, h.y, h.z)};
}
__device__ __forceinline__ void store_box(float4 *b, int i, const Box &x) {
  __stcg(b + 2 * i, make_float4(x.lo.x, x.lo.y, x.lo.z, 0.0f));
  __stcg(b + 2 * i + 1, make_float4(x.hi.x, x.hi.y, x.hi.z, 0.0f));
}

// Order-preserving float <-> uint map for atomic min/max of the scene bounds.
__device__ __forceinline__ uint32_t f2ord(float f) {
  uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__host__ __device__ inline float ord2f(uint32_t u) {
  uint32_t b = (u & 0x80000000u) ? (u & 0x7fffffffu) : ~u;
#ifdef __CUDA_ARCH__
  return __uint_as_float(b);
#else
  float f;
  memcpy(&f, &b, 4);
  return f;
#endif
}

// ---- stage 1: face boxes, centroid bounds, scene bounds, validation ---------------------------
// bounds[0..5] = centroid lo xyz, hi xyz; bounds[6..11] = scene lo xyz, hi xyz (ordered uints).
__global__ void k_init_bounds(uint32_t *bounds) {
  int i = threadIdx.x;
  if (i < 12) bounds[i] = (i % 6) < 3 ? 0xffffffffu : 0u;
}

__global__ void __launch_bounds__(256) k_face_boxes(const vt_face *faces, uint32_t nfaces,
                                                      const vt_vertex *verts, uint32_t nverts,
                                                      float4 *boxes, uint32_t *bounds,
                                                      uint32_t *status) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  float3 clo = make_float3(FLT_MAX, FLT_MAX, FLT_MAX), chi = make_float3(-FLT_MAX, -FLT_MAX, -FLT_MAX);
  float3 slo = clo, shi = chi;
  bool smooth = false;
  if (i < nfaces) {
    vt_face f = faces[i];
    Box b{make_float3(0, 0, 0), make_float3(0, 0, 0)};
    if (f.a >= nverts || f.b >= nverts || f.c >= nverts) {
      atomicOr(status, (uint32_t)VT_DEV_BAD_INDEX);
    } else {
      const vt_vertex &va = verts[f.a], &vb = verts[f.b], &vc = verts[f.c];
      float3 a = make_float3(va.px, va.py, va.pz), p = make_float3(vb.px, vb.py, vb.pz),
             q = make_float3(vc.px, vc.py, vc.pz);
      smooth = va.nx != 0.0f || va.ny != 0.0f || va.nz != 0.0f || vb.nx != 0.0f || vb.ny != 0.0f || vb.nz != 0.0f ||
               vc.nx != 0.0f || vc.ny != 0.0f || vc.nz != 0.0f;
      bool finite = isfinite(a.x) && isfinite(a.y) && isfinite(a.z) && isfinite(p.x) &&
                    isfinite(p.y) && isfinite(p.z) && isfinite(q.x) && isfinite(q.y) && isfinite(q.z);
      if (!finite) {
        atomicOr(status, (uint32_t)VT_DEV_NONFINITE);
      } else {
        b.lo = make_float3(fminf(fminf(a.x, p.x), q.x), fminf(fminf(a.y, p.y), q.y), fminf(fminf(a.z, p.z), q.z));
        b.hi = make_float3(fmaxf(fmaxf(a.x, p.x), q.x), fmaxf(fmaxf(a.y, p.y), q.y), fmaxf(fmaxf(a.z, p.z), q.z));
      }
    }
    boxes[2 * i] = make_float4(b.lo.x, b.lo.y, b.lo.z, 0.0f);
    boxes[2 * i + 1] = make_float4(b.hi.x, b.hi.y, b.hi.z, 0.0f);
    float3 c = make_float3(__fmul_rn(__fadd_rn(b.lo.x, b.hi.x), 0.5f), __fmul_rn(__fadd_rn(b.lo.y, b.hi.y), 0.5f),
                           __fmul_rn(__fadd_rn(b.lo.z, b.hi.z), 0.5f));
    clo = chi = c;
    slo = b.lo;
    shi = b.hi;
  }
  // Warp then block reduction of the 12 bounds, one atomic per block per bound.
  float v[12] = {clo.x, clo.y, clo.z, chi.x, chi.y, chi.z, slo.x, slo.y, slo.z, shi.x, shi.y, shi.z};
#pragma unroll
  for (int k = 0; k < 12; ++k) {
    const bool isMin = (k % 6) < 3;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      float u = __shfl_xor_sync(0xffffffffu, v[k], o);
      v[k] = isMin ? fminf(v[k], u) : fmaxf(v[k], u);
    }
  }
  __shared__ float red[8][12];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < 12; ++k) red[warp][k] = v[k];
  if (__syncthreads_or(smooth) && threadIdx.x == 0 && !(__ldcg(status) & (uint32_t)VT_DEV_NORMALS))
    atomicOr(status, (uint32_t)VT_DEV_NORMALS);
  if (threadIdx.x < 12) {
    const int k = threadIdx.x;
    const bool isMin = (k % 6) < 3;
    float x = red[0][k];
    for (int w = 1; w < (int)(blockDim.x / 32); ++w) x = isMin ? fminf(x, red[w][k]) : fmaxf(x, red[w][k]);
    if (isMin) atomicMin(&bounds[k], f2ord(x));
    else atomicMax(&bounds[k], f2ord(x));
  }
}

// ---- stage 2: Morton codes --------------------------------------------------------------------
__device__ __forceinline__ uint32_t expand_bits(uint32_t v) {
  v = (v * 0x00010001u) & 0xFF0000FFu;
  v = (v * 0x00000101u) & 0x0F00F00Fu;
  v = (v * 0x00000011u) & 0xC30C30C3u;
  v = (v * 0x00000005u) & 0x49249249u;
  return v;
}
// q = min(uint((c - clo) * (1024 / (chi - clo))), 1023), 0 on a flat axis.
__device__ __forceinline__ uint32_t quantize(float c, float clo, float chi) {
  float ext = __fsub_rn(chi, clo);
  if (!(ext > 0.0f)) return 0u;
  float scale = __fdiv_rn(1024.0f, ext);
  float f = __fmul_rn(__fsub_rn(c, clo), scale);
  return f >= 1023.0f ? 1023u : (uint32_t)f;
}

__global__ void k_morton(const float4 *boxes, uint32_t n, const uint32_t *bounds, uint32_t *codes,
                         uint32_t *vals) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float4 l = boxes[2 * i], h = boxes[2 * i + 1];
  float cx = __fmul_rn(__fadd_rn(l.x, h.x), 0.5f), cy = __fmul_rn(__fadd_rn(l.y, h.y), 0.5f),
        cz = __fmul_rn(__fadd_rn(l.z, h.z), 0.5f);
  uint32_t qx = quantize(cx, ord2f(bounds[0]), ord2f(bounds[3]));
  uint32_t qy = quantize(cy, ord2f(bounds[1]), ord2f(bounds[4]));
  uint32_t qz = quantize(cz, ord2f(bounds[2]), ord2f(bounds[5]));
  codes[i] = (expand_bits(qx) << 2) | (expand_bits(qy) << 1) | expand_bits(qz);
  vals[i] = i;
}

// ---- stage 3: Karras hierarchy (HPG 2012) -----------------------------------------------------
// Children: internal index >= 0, leaf = -(sorted position + 1). parent[] holds internal nodes at
// [0, n-1) and leaves at n - 1 + position; the root's parent is -1.
__device__ __forceinline__ int delta(const uint32_t *codes, int n, int i, int j) {
  if (j < 0 || j > n - 1) return -1;
  uint32_t a = codes[i], b = codes[j];
  if (a != b) return __clz(a ^ b);
  return 32 + __clz((uint32_t)i ^ (uint32_t)j);
}

// Whether the sort gave up: its face indices are then any numbers and nothing is built on them. k_hierarchy leaves
// every leaf without a parent, so that the treelet walks end where they start, the collapse has no level, and the
// build reports the error.
__device__ __forceinline__ bool unsorted(const uint32_t *status) { return (__ldcg(status) & (uint32_t)VT_DEV_SORT) != 0u; }

// One thread per sorted position: its leaf box gathered, and internal node i's hierarchy with its
// visit counter cleared.
__global__ void k_hierarchy(const uint32_t *codes, const float4 *boxes, const uint32_t *sorted, int n, float4 *leaf, int2 *child,
                            int32_t *parent, uint32_t *flags, const uint32_t *status) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (unsorted(status)) {
    parent[n - 1 + i] = -1;
    return;
  }
  const uint32_t f = sorted[i];
  leaf[2 * (size_t)i] = boxes[2 * (size_t)f];
  leaf[2 * (size_t)i + 1] = boxes[2 * (size_t)f + 1];
  if (i == 0) parent[0] = -1;
  if (i >= n - 1) return;
  flags[i] = 0u;
  const int d = delta(codes, n, i, i + 1) - delta(codes, n, i, i - 1) > 0 ? 1 : -1;
  const int dmin = delta(codes, n, i, i - d);
  int lmax = 2;
  while (delta(codes, n, i, i + lmax * d) > dmin) lmax *= 2;
  int l = 0;
  for (int s = lmax / 2; s >= 1; s /= 2)
    if (delta(codes, n, i, i + (l + s) * d) > dmin) l += s;
  const int j = i + l * d;
  const int dnode = delta(codes, n, i, j);
  int s = 0;
  for (int div = 2;; div *= 2) {
    const int step = (l + div - 1) / div;
    if (delta(codes, n, i, i + (s + step) * d) > dnode) s += step;
    if (step <= 1) break;
  }
  const int gamma = i + s * d + min(d, 0);
  const int lo = min(i, j), hi = max(i, j);
  const int left = lo == gamma ? -(gamma + 1) : gamma;
  const int right = hi == gamma + 1 ? -(gamma + 2) : gamma + 1;
  child[i] = make_int2(left, right);
  parent[left >= 0 ? left : (n - 1 + gamma)] = i;
  parent[right >= 0 ? right : (n - 1 + gamma + 1)] = i;
}

// ---- bottom-up passes ---------------------------------------------------------------------------
struct TreeView {
  int n;
  int2 *child;
  int32_t *parent;
  const float4 *leafBox;
  float4 *nodeBox;
  uint32_t *count;
  float *cost;
};

__device__ __forceinline__ int2 load_child(const TreeView &t, int i) {
  return __ldcg(t.child + i);
}
__device__ __forceinline__ Box child_box(const TreeView &t, int c) {
  return c >= 0 ? load_box_cg(t.nodeBox, c) : load_box_cg(t.leafBox, -c - 1);
}
__device__ __forceinline__ float child_cost(const TreeView &t, int c) {
  if (c >= 0) return __ldcg(t.cost + c);
  Box b = load_box_cg(t.leafBox, -c - 1);
  return __fmul_rn(kCt, box_area(b.lo, b.hi));
}
__device__ __forceinline__ uint32_t child_count(const TreeView &t, int c) {
  return c >= 0 ? __ldcg(t.count + c) : 1u;
}
__device__ __forceinline__ void refit_node(const TreeView &t, int i) {
  int2 ch = load_child(t, i);
  Box b = box_union(child_box(t, ch.x), child_box(t, ch.y));
  store_box(t.nodeBox, i, b);
  __stcg(t.count + i, child_count(t, ch.x) + child_count(t, ch.y));
  __stcg(t.cost + i, __fadd_rn(__fmul_rn(kCi, box_area(b.lo, b.hi)),
                               __fadd_rn(child_cost(t, ch.x), child_cost(t, ch.y))));
}

// Treelet restructuring at internal node `root` (Karras and Aila, HPG 2013), in the
// deterministic form the oracle restates: grow the treelet by opening its largest-area internal
// leaf (first in list order on ties; opened node replaced in place by its left child, right child
// appended), DP over subsets (partitions p = (p - 1) & s downwards, strict improvement), rebuild
// only on a strict cost improvement, internal nodes reassigned depth first, left = the side with
// the lowest leaf bit.
//
// A warp takes one treelet (Karras and Aila's warp-wide DP): lane q holds treelet leaf q while the
// treelet grows (its box, children, cost and leaf count loaded in one round trip, the largest area
// chosen by a warp reduction that keeps the first slot on ties). The DP visits the subsets by size,
// one or more lanes a subset. A partition and its complement cost the same, and the serial loop meets
// the one with the subset's highest leaf first: only those are tried, the largest of equal cost kept.
// A subset's box is the union of two table entries (of the low and of the high four leaves). The
// rebuilt nodes need no second pass: a node's cost is its subset's optimum, whose sums are the same.
//
// Bound: latency of the chain of treelets from the leaves to the root (loads of a growing treelet, the
// DP's shared-memory reads) and, for large meshes, issue. Measured on one B200, whole builds with
// three rounds of treelets of 7: 1,000 triangles 0.84 -> 0.60 ms, 20,480 1.31 -> 0.88, 200,000
// 2.16 -> 1.42, 1M 6.16 -> 3.72, 4M 21.0 -> 12.0. Before, small treelets near the leaves were taken by
// single threads (divergent, arrays in local memory), the DP tried every partition with a box
// recomputed per subset, and the rebuilt nodes were refitted one by one.
struct TreeletScratch {
  float4 tabLo[32], tabHi[32];  // boxes of the subsets of leaves 0-3 (entries 0-15) and of 4-7 (16-31)
  float4 leafLo[kMaxTreelet], leafHi[kMaxTreelet];
  float copt[1 << kMaxTreelet];
  uint8_t part[1 << kMaxTreelet];
  int leaves[kMaxTreelet], internals[kMaxTreelet];
  uint32_t lcount[kMaxTreelet];
  int2 kid[kMaxTreelet];        // rebuilt node j's children: >= 0 internal index, else -(leaf slot + 1)
  uint8_t set[kMaxTreelet];     // rebuilt node j's subset
  int ok;
};

// The nonempty subsets of 8 leaves grouped by size, increasing within a size, so that for k leaves each
// group's first C(k, size) entries are the subsets of those; copied to shared memory once per block.
struct alignas(4) SubsetTable {
  uint8_t list[256];
  int start[kMaxTreelet + 2];
};
constexpr SubsetTable make_subsets() {
  SubsetTable t{};
  int at = 0;
  for (int size = 1; size <= kMaxTreelet; ++size) {
    t.start[size] = at;
    for (int s = 1; s < 256; ++s) {
      int bits = 0;
      for (int r = s; r; r &= r - 1) ++bits;
      if (bits == size) t.list[at++] = (uint8_t)s;
    }
  }
  t.start[kMaxTreelet + 1] = at;
  return t;
}
__device__ const SubsetTable kSubsets = make_subsets();

__device__ __forceinline__ Box subset_box(const TreeletScratch &w, int s) {
  const float4 al = w.tabLo[s & 15], ah = w.tabHi[s & 15], bl = w.tabLo[16 + (s >> 4)], bh = w.tabHi[16 + (s >> 4)];
  return box_union(Box{make_float3(al.x, al.y, al.z), make_float3(ah.x, ah.y, ah.z)},
                   Box{make_float3(bl.x, bl.y, bl.z), make_float3(bh.x, bh.y, bh.z)});
}

__device__ void restructure_warp(const TreeView &t, int root, int size, uint32_t *status, TreeletScratch &w, const SubsetTable &sets) {
  const unsigned kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const float rootCost = __ldcg(t.cost + root);
  const int2 rc = load_child(t, root);
  // Lane q < nl holds treelet leaf q: its node, box, children, cost and leaf count.
  int myLeaf = lane == 0 ? rc.x : rc.y;
  bool dirty = lane < 2;
  Box myBox{};
  int2 myKids = make_int2(0, 0);
  float myCost = 0.0f;
  uint32_t myCount = 1u, myKey = 0u;  // key: area bits + 1 of a leaf that can be opened
  int myInternal = lane == 0 ? root : -1;
  int nl = 2, ni = 1;
  while (true) {
    if (dirty) {
      if (myLeaf >= 0) {
        myBox = load_box_cg(t.nodeBox, myLeaf);
        myKids = load_child(t, myLeaf);
        myCost = __ldcg(t.cost + myLeaf);
        myCount = __ldcg(t.count + myLeaf);
        myKey = __float_as_uint(box_area(myBox.lo, myBox.hi)) + 1u;
      } else {  // a primitive is never opened
        myBox = load_box_cg(t.leafBox, -myLeaf - 1);
        myCost = __fmul_rn(kCt, box_area(myBox.lo, myBox.hi));
        myCount = 1u;
        myKey = 0u;
      }
      dirty = false;
    }
    if (nl >= size) break;
    const uint32_t largest = __reduce_max_sync(kAll, lane < nl ? myKey : 0u);
    if (largest == 0u) break;  // no internal node left to open
    const int q = __ffs(__ballot_sync(kAll, lane < nl && myKey == largest)) - 1;
    const int c = __shfl_sync(kAll, myLeaf, q);
    const int cx = __shfl_sync(kAll, myKids.x, q), cy = __shfl_sync(kAll, myKids.y, q);
    if (lane == ni) myInternal = c;
    if (lane == q) { myLeaf = cx; dirty = true; }
    if (lane == nl) { myLeaf = cy; dirty = true; }
    ++ni;
    ++nl;
  }
  const int k = nl;
  if (k < 3) return;
  const int full = (1 << k) - 1;
  if (lane < k) {
    w.leaves[lane] = myLeaf;
    w.leafLo[lane] = make_float4(myBox.lo.x, myBox.lo.y, myBox.lo.z, 0.0f);
    w.leafHi[lane] = make_float4(myBox.hi.x, myBox.hi.y, myBox.hi.z, 0.0f);
    w.copt[1 << lane] = myCost;
    w.lcount[lane] = myCount;
  }
  if (lane < ni) w.internals[lane] = myInternal;
  __syncwarp();
  {
    Box b{make_float3(INFINITY, INFINITY, INFINITY), make_float3(-INFINITY, -INFINITY, -INFINITY)};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int leaf = (lane >> 4) * 4 + q;
      if ((lane >> q & 1) && leaf < k) {
        const float4 l = w.leafLo[leaf], h = w.leafHi[leaf];
        b = box_union(b, Box{make_float3(l.x, l.y, l.z), make_float3(h.x, h.y, h.z)});
      }
    }
    w.tabLo[lane] = make_float4(b.lo.x, b.lo.y, b.lo.z, 0.0f);
    w.tabHi[lane] = make_float4(b.hi.x, b.hi.y, b.hi.z, 0.0f);
  }
  __syncwarp();
  int nsub = k;  // C(k, sz)
  for (int sz = 2; sz <= k; ++sz) {
    nsub = nsub * (k - sz + 1) / sz;
    // 2^g lanes a subset (as many as keep all subsets in one round, at most one per partition half).
    int g = 0;
    while (g < sz - 1 && (nsub << (g + 1)) <= 32) ++g;
    for (int j0 = 0; j0 < nsub; j0 += 32 >> g) {
      const int j = j0 + (lane >> g);
      const bool active = j < nsub;
      const int s = active ? sets.list[sets.start[sz] + j] : full;
      const int top = 1 << (31 - __clz(s)), rest = s ^ top;
      // This lane fixes the g lowest leaves of the rest by its place in the group and tries every choice
      // of the others.
      int fixed = 0, open = rest;
      for (int q = 0; q < g; ++q) {
        const int bit = open & -open;
        open ^= bit;
        if (lane >> q & 1) fixed |= bit;
      }
      float best = FLT_MAX;
      int bp = 0;
      if (active) {
        for (int sub = open;; sub = (sub - 1) & open) {
          const int p = top | fixed | sub;
          if (p != s) {
            const float c = __fadd_rn(w.copt[p], w.copt[s ^ p]);
            if (c < best || (c == best && bp != 0 && p > bp)) { best = c; bp = p; }
          }
          if (sub == 0) break;
        }
      }
      for (int off = 1; off < (1 << g); off <<= 1) {
        const float ob = __shfl_xor_sync(kAll, best, off);
        const int op = __shfl_xor_sync(kAll, bp, off);
        if (ob < best || (ob == best && op > bp)) { best = ob; bp = op; }
      }
      if (active && (lane & ((1 << g) - 1)) == 0) {
        const Box b = subset_box(w, s);
        w.copt[s] = __fadd_rn(__fmul_rn(kCi, box_area(b.lo, b.hi)), best);
        w.part[s] = (uint8_t)bp;
      }
    }
    __syncwarp();
  }
  if (!(w.copt[full] < rootCost)) return;
  if (lane == 0) {
    // Depth-first assignment of the internal nodes: index j in assignment order, a stack of 4-bit indices.
    int next = 1, depth = 1;
    uint32_t stack = 0u;
    w.set[0] = (uint8_t)full;
    w.ok = 1;
    while (depth > 0) {
      const int j = (int)(stack & 15u);
      stack >>= 4;
      --depth;
      const int s = w.set[j], p = w.part[s], q = s ^ p;
      const int lowbit = s & -s;
      const int left = (p & lowbit) ? p : q, right = (p & lowbit) ? q : p;
      int2 ref;
      const bool li = (left & (left - 1)) != 0, ri = (right & (right - 1)) != 0;
      if (next + (li ? 1 : 0) + (ri ? 1 : 0) > ni) { w.ok = 0; break; }
      ref.x = li ? next++ : -__ffs(left);  // -(leaf slot + 1)
      ref.y = ri ? next++ : -__ffs(right);
      w.kid[j] = ref;
      if (ri) { w.set[ref.y] = (uint8_t)right; stack = stack << 4 | (uint32_t)ref.y; ++depth; }
      if (li) { w.set[ref.x] = (uint8_t)left; stack = stack << 4 | (uint32_t)ref.x; ++depth; }
    }
    if (!w.ok) atomicOr(status, (uint32_t)VT_DEV_TREELET);
  }
  __syncwarp();
  if (!w.ok || lane >= ni) return;
  const int node = w.internals[lane], s = w.set[lane];
  const int2 r = w.kid[lane];
  const int kx = r.x >= 0 ? w.internals[r.x] : w.leaves[-r.x - 1];
  const int ky = r.y >= 0 ? w.internals[r.y] : w.leaves[-r.y - 1];
  uint32_t count = 0;
  for (int q = 0; q < k; ++q) count += (s >> q & 1) ? w.lcount[q] : 0u;
  __stcg(t.child + node, make_int2(kx, ky));
  store_box(t.nodeBox, node, subset_box(w, s));
  __stcg(t.count + node, count);
  __stcg(t.cost + node, w.copt[s]);
  __stcg(t.parent + (kx >= 0 ? kx : (t.n - 1 + (-kx - 1))), node);
  __stcg(t.parent + (ky >= 0 ? ky : (t.n - 1 + (-ky - 1))), node);
}

constexpr int kMaxWalk = 1 << 14;

// A visit of a node's counter: everything this thread (and, after a __syncwarp, its warp) wrote below
// the node is visible to the visitor that comes second, which sees an odd count.
__device__ __forceinline__ bool second_visit(uint32_t *flag) {
  uint32_t before;
  asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(before) : "l"(flag) : "memory");
  return (before & 1u) != 0u;
}

// One thread per leaf walks to the root; the second thread to reach a node owns it (its two
// subtrees are final) and refits it. A pass visits every node twice, so flags[] starts each pass even
// and the first visitor sees an even count: it is cleared once, by k_hierarchy.
__global__ void __launch_bounds__(128) k_bottom_up(TreeView t, uint32_t *flags, uint32_t *status) {
  const int leaf = blockIdx.x * blockDim.x + threadIdx.x;
  if (leaf >= t.n) return;
  int node = __ldcg(t.parent + (t.n - 1 + leaf));
  // A walk longer than any tree of 30-bit codes and 32-bit positions is deep means a corrupted parent
  // chain: stop and report.
  for (int guard = 0; node >= 0; ++guard) {
    if (guard >= kMaxWalk) { atomicOr(status, (uint32_t)VT_DEV_TREELET); return; }
    if (!second_visit(&flags[node])) return;
    refit_node(t, node);
    node = __ldcg(t.parent + node);
  }
}

// The cost of the tree as the first pass found it, kept beside t.cost: a node's restructuring decision
// compares against its cost before any restructuring below it.
__device__ __forceinline__ void refit_first(const TreeView &t, float *firstCost, int i) {
  const int2 ch = load_child(t, i);
  const Box b = box_union(child_box(t, ch.x), child_box(t, ch.y));
  auto first = [&](int c) { return c >= 0 ? __ldcg(firstCost + c) : child_cost(t, c); };
  const float cost = __fadd_rn(__fmul_rn(kCi, box_area(b.lo, b.hi)), __fadd_rn(first(ch.x), first(ch.y)));
  store_box(t.nodeBox, i, b);
  __stcg(t.count + i, child_count(t, ch.x) + child_count(t, ch.y));
  __stcg(t.cost + i, cost);
  __stcg(firstCost + i, cost);
}

// The same walk for restructuring; the first round (firstCost not null) refits each node as it comes
// to own it, which saves a pass of its own. Nodes owned by lanes of one warp in the same step are
// disjoint subtrees (an owner's subtrees are final), so the warp takes those with >= size leaves one
// after another in any order.
// Blocks of two warps: a block's slots stay taken until its longest walk ends (128 threads 0.839 and 3.50 ms
// for whole builds of 20,480 and 1M triangles, 64 0.813 and 3.46, 32 0.866 and 3.52).
constexpr int kRestructureBlock = 64;
__global__ void __launch_bounds__(kRestructureBlock) k_restructure(TreeView t, uint32_t *flags, int size, float *firstCost, uint32_t *status) {
  __shared__ TreeletScratch scratch[kRestructureBlock / 32];
  __shared__ SubsetTable sets;
  for (uint32_t q = threadIdx.x; q < sizeof(SubsetTable) / 4; q += blockDim.x)
    reinterpret_cast<uint32_t *>(&sets)[q] = reinterpret_cast<const uint32_t *>(&kSubsets)[q];
  __syncthreads();
  TreeletScratch &w = scratch[threadIdx.x >> 5];
  const unsigned kAll = 0xffffffffu;
  const int leaf = blockIdx.x * blockDim.x + threadIdx.x;
  int node = leaf < t.n ? __ldcg(t.parent + (t.n - 1 + leaf)) : -1;
  for (int guard = 0;; ++guard) {
    bool own = false;
    if (node >= 0) {
      if (guard >= kMaxWalk) {
        atomicOr(status, (uint32_t)VT_DEV_TREELET);
        node = -1;
      } else {
        own = second_visit(&flags[node]);
        if (!own) node = -1;
      }
    }
    if (own && firstCost) refit_first(t, firstCost, node);
    __syncwarp();
    unsigned work = __ballot_sync(kAll, own && __ldcg(t.count + node) >= (uint32_t)size);
    while (work) {
      const int src = __ffs(work) - 1;
      work &= work - 1;
      restructure_warp(t, __shfl_sync(kAll, node, src), size, status, w, sets);
      __syncwarp();
    }
    if (own) node = __ldcg(t.parent + node);
    if (!__any_sync(kAll, node >= 0)) break;
  }
}

// ---- collapse to 4-wide -------------------------------------------------------------------------
// A wide node rooted at binary node b starts with children [b] and splits the child of largest
// area among those with more than leafSize leaves (the reference's rule,
// Sources/Acceleration.swift:255-263) until four children.
// The children of the wide node at binary node `root`; returns their number.
__device__ __forceinline__ int collapse_children(const TreeView &t, int root, int leafSize, int ch[4], uint32_t &inner, uint32_t &prims) {
  uint32_t cnt[4];
  ch[0] = root;
  cnt[0] = child_count(t, root);
  int m = 1;
  while (m < 4) {
    int best = -1;
    float bestA = 0.0f;
    for (int k = 0; k < m; ++k) {
      if (cnt[k] <= (uint32_t)leafSize) continue;
      Box b = child_box(t, ch[k]);
      float a = box_area(b.lo, b.hi);
      if (best < 0 || a > bestA) { best = k; bestA = a; }
    }
    if (best < 0) break;
    const int c = ch[best];
    for (int k = m; k > best + 1; --k) { ch[k] = ch[k - 1]; cnt[k] = cnt[k - 1]; }
    int2 cc = load_child(t, c);
    ch[best] = cc.x;
    ch[best + 1] = cc.y;
    cnt[best] = child_count(t, cc.x);
    cnt[best + 1] = child_count(t, cc.y);
    ++m;
  }
  inner = prims = 0;
  for (int k = 0; k < m; ++k) {
    if (cnt[k] <= (uint32_t)leafSize) prims += cnt[k];
    else ++inner;
  }
  return m;
}

// Wide node `at` with children ch (unused slots INT_MIN, which no leaf encoding reaches): its inner
// children get nodes from nextBase + inner on and entries from nextLevel[inner] on, its leaves'
// triangles BVH positions from prim on (order: the face, with kLastOfLeaf on a leaf's last).
constexpr uint32_t kLastOfLeaf = 0x80000000u;
__device__ __forceinline__ void collapse_emit(const TreeView &t, int leafSize, const int4 c4, uint32_t inner, uint32_t prim,
                                              uint32_t at, uint32_t nextBase, vt_wide_node *nodes, int32_t *nextLevel,
                                              const uint32_t *sorted, int32_t *order, uint32_t *status) {
  int ch[4] = {c4.x, c4.y, c4.z, c4.w};
  vt_wide_node nd;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    nd.lox[k] = nd.loy[k] = nd.loz[k] = nd.hix[k] = nd.hiy[k] = nd.hiz[k] = 0.0f;
    nd.child[k] = 0;
    nd.count[k] = 0;
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (ch[k] == INT_MIN) break;
    Box b = child_box(t, ch[k]);
    nd.lox[k] = b.lo.x; nd.loy[k] = b.lo.y; nd.loz[k] = b.lo.z;
    nd.hix[k] = b.hi.x; nd.hiy[k] = b.hi.y; nd.hiz[k] = b.hi.z;
    uint32_t cnt = child_count(t, ch[k]);
    if (cnt <= (uint32_t)leafSize) {
      nd.child[k] = -(int32_t)(prim + 1);
      nd.count[k] = (int32_t)cnt;
      // Leaves of the binary subtree, depth first, left first.
      int st[2 * 8 + 2];
      int top = 0;
      st[top++] = ch[k];
      while (top) {
        int c = st[--top];
        if (c < 0) {
          if (prim >= (uint32_t)t.n) { atomicOr(status, (uint32_t)VT_DEV_TREELET); return; }
          order[prim++] = (int32_t)(sorted[-c - 1] | (top == 0 ? kLastOfLeaf : 0u));
          continue;
        }
        if (top + 2 > 2 * 8 + 2) { atomicOr(status, (uint32_t)VT_DEV_TREELET); return; }
        int2 cc = load_child(t, c);
        st[top++] = cc.y;
        st[top++] = cc.x;
      }
    } else {
      nd.child[k] = (int32_t)(nextBase + inner);
      __stcg(nextLevel + inner, ch[k]);
      ++inner;
    }
  }
  nodes[at] = nd;
}

// One thread per BVH position: its triangle gathered from the input, once the collapse has placed it. Bound: the
// scattered reads. In the collapse these were three dependent loads a triangle inside every level's serial
// chain: whole builds on one B200 0.884 -> 0.858 ms at 20,480 triangles, 3.72 -> 3.59 at 1M, 12.0 -> 11.5
// at 4M.
__global__ void k_triangles(const vt_face *faces, uint32_t n, const vt_vertex *verts, uint32_t nverts, int32_t *order, float4 *tris,
                            float4 *nrm, int markLeaves) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t placed = (uint32_t)order[i], f = placed & ~kLastOfLeaf;
  if (f >= n) return;  // a collapse that stopped early: the build reports its error
  // The traversal's leaf loop ends at the triangle marked as its leaf's last.
  const float last = markLeaves && (placed & kLastOfLeaf) ? 1.0f : 0.0f;
  const size_t p3 = 3 * (size_t)i;
  order[i] = (int32_t)f;
  const vt_face fc = faces[f];
  if (fc.a >= nverts || fc.b >= nverts || fc.c >= nverts) {
    // k_face_boxes flagged this face already; its vertices are not read (the build then
    // returns VT_ERR_INVALID), the slot gets a degenerate triangle at the origin.
    const float4 z = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    tris[p3] = make_float4(0.0f, 0.0f, 0.0f, __int_as_float((int)f));
    tris[p3 + 1] = z;
    tris[p3 + 2] = make_float4(0.0f, 0.0f, 0.0f, last);
    if (nrm) nrm[p3] = nrm[p3 + 1] = nrm[p3 + 2] = z;
    return;
  }
  const vt_vertex va = verts[fc.a], vb = verts[fc.b], vc = verts[fc.c];
  tris[p3] = make_float4(va.px, va.py, va.pz, __int_as_float((int)f));
  tris[p3 + 1] = make_float4(vb.px, vb.py, vb.pz, __uint_as_float(fc.tag));
  tris[p3 + 2] = make_float4(vc.px, vc.py, vc.pz, last);
  if (nrm) {  // vertex normals for smooth shading (mesh_hit_attributes)
    nrm[p3] = make_float4(va.nx, va.ny, va.nz, 0.0f);
    nrm[p3 + 1] = make_float4(vb.nx, vb.ny, vb.nz, 0.0f);
    nrm[p3 + 2] = make_float4(vc.nx, vc.ny, vc.nz, 0.0f);
  }
}

// What a build reports back, in one copy.
struct BuildReport {
  uint32_t bounds[12];                 // k_face_boxes'
  uint32_t nodes, depth, prims, code;  // the collapse's (code: kCollapse*)
  uint32_t status, done, pad[2];       // done: 1 once the collapse has run to its end
};
enum : uint32_t { kCollapseOk = 0, kCollapseDepth = 1, kCollapseNodes = 2 };

constexpr int kCollapseBlock = 128;
constexpr uint32_t kBarrierSpins = 1u << 21;  // polls before a grid barrier gives up (VT_DEV_BARRIER)

// Barrier over the grid of a cooperative launch: bar[0] counts arrivals over the kernel's whole life,
// bar[1] is set when a block gave up. False (block-uniform) once any block did.
__device__ bool grid_barrier(uint32_t *bar, uint32_t &round, uint32_t *status) {
  __shared__ bool alive;
  ++round;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(bar, 1u);
    const uint32_t target = round * gridDim.x;
    uint32_t spins = 0;
    while (vt_poll(bar) < target && vt_poll(bar + 1) == 0u && ++spins < kBarrierSpins) {}
    if (spins >= kBarrierSpins) {
      atomicOr(status, (uint32_t)VT_DEV_BARRIER);
      atomicExch(bar + 1, 1u);
    }
    __threadfence();
    alive = vt_poll(bar + 1) == 0u;
  }
  __syncthreads();
  return alive;
}

// Sum over the block (every thread gets it).
__device__ __forceinline__ uint32_t block_sum(uint32_t v, uint32_t *ws) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = v;
  __syncthreads();
  return ws[0] + ws[1] + ws[2] + ws[3];
}

// The whole collapse in one cooperative launch. Bound: latency (per level a few dependent loads and two
// grid barriers); a launch per step with the level's size read back by the host spent 60-100 us a
// level instead (rebuilding and tracing 20,480 triangles: 4.1 -> 1.6 ms with the sort and the pool). Per
// level each block takes a contiguous part: it counts its wide nodes' inner children and triangles, and
// after a barrier prefixes the blocks' sums to place its own nodes, children and triangles in the level
// order of a serial pass.
__global__ void __launch_bounds__(kCollapseBlock) k_collapse(TreeView t, int leafSize, int maxDepth, uint32_t maxNodes, int32_t *levelA,
                                                             int32_t *levelB, int4 *children, uint32_t *packed, uint2 *blockSums,
                                                             uint32_t *bar, vt_wide_node *nodes, const uint32_t *sorted, int32_t *order,
                                                             const uint32_t *bounds, BuildReport *report, uint32_t *status) {
  __shared__ uint32_t ws[kCollapseBlock / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t L = unsorted(status) ? 0u : 1u, base = 0, primBase = 0, depth = 0, code = kCollapseOk, round = 0;
  int32_t *level = levelA, *nextLevel = levelB;
  while (L > 0) {
    if ((int)depth >= maxDepth) { code = kCollapseDepth; break; }
    ++depth;
    const uint32_t per = ((L + gridDim.x - 1) / gridDim.x + kCollapseBlock - 1) / kCollapseBlock * kCollapseBlock;
    const uint32_t w0 = min((uint64_t)L, (uint64_t)blockIdx.x * per), w1 = min(L, w0 + per);
    uint32_t sumI = 0, sumP = 0;
    for (uint32_t w = w0 + threadIdx.x; w < w1; w += kCollapseBlock) {
      const int root = depth == 1 ? (t.n >= 2 ? 0 : -1) : __ldcg(level + w);
      int ch[4];
      uint32_t inner, prims;
      const int m = collapse_children(t, root, leafSize, ch, inner, prims);
      children[w] = make_int4(ch[0], m > 1 ? ch[1] : INT_MIN, m > 2 ? ch[2] : INT_MIN, m > 3 ? ch[3] : INT_MIN);
      packed[w] = inner | prims << 16;
      sumI += inner;
      sumP += prims;
    }
    sumI = block_sum(sumI, ws);
    sumP = block_sum(sumP, ws);
    if (threadIdx.x == 0) __stcg(blockSums + blockIdx.x, make_uint2(sumI, sumP));
    if (!grid_barrier(bar, round, status)) return;
    uint32_t allI = 0, allP = 0, runI = 0, runP = 0;
    for (uint32_t q = threadIdx.x; q < gridDim.x; q += kCollapseBlock) {
      const uint2 v = __ldcg(blockSums + q);  // ordered by the barrier
      allI += v.x;
      allP += v.y;
      if (q < blockIdx.x) { runI += v.x; runP += v.y; }
    }
    allI = block_sum(allI, ws);
    allP = block_sum(allP, ws);
    runI = block_sum(runI, ws);
    runP = block_sum(runP, ws);
    const uint32_t nextBase = base + L;
    for (uint32_t tile = w0; tile < w1; tile += kCollapseBlock) {  // w0, w1 are block-uniform
      const uint32_t w = tile + threadIdx.x;
      // Exclusive prefix of (inner, triangles) over the tile: 16 bits hold either sum.
      const uint32_t v = w < w1 ? packed[w] : 0u;
      uint32_t inc = v;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += u;
      }
      __syncthreads();
      if (lane == 31) ws[warp] = inc;
      __syncthreads();
      uint32_t before = 0, all = 0;
#pragma unroll
      for (int k = 0; k < kCollapseBlock / 32; ++k) {
        before += k < warp ? ws[k] : 0u;
        all += ws[k];
      }
      before += inc - v;
      if (w < w1)
        collapse_emit(t, leafSize, children[w], runI + (before & 0xffffu), primBase + runP + (before >> 16), base + w, nextBase,
                      nodes, nextLevel, sorted, order, status);
      runI += all & 0xffffu;
      runP += all >> 16;
    }
    if (!grid_barrier(bar, round, status)) return;
    // No block writes status before the next barrier, so all of them read the same.
    const uint32_t st = vt_poll(status);
    primBase += allP;
    base = nextBase;
    L = allI;
    int32_t *x = level; level = nextLevel; nextLevel = x;
    if (st & (uint32_t)(VT_DEV_TREELET | VT_DEV_BAD_INDEX | VT_DEV_NONFINITE)) break;
    if (base + L > maxNodes) { code = kCollapseNodes; break; }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    for (int k = 0; k < 12; ++k) report->bounds[k] = bounds[k];
    report->nodes = base;
    report->depth = depth;
    report->prims = primBase;
    report->code = code;
    report->status = vt_poll(status);
    report->done = 1u;
  }
}

// SAH cost of the wide tree (node cost 1, triangle cost 1, areas over the root box's area).
__global__ void k_sah(const vt_wide_node *nodes, uint32_t nn, double *acc) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  const vt_wide_node &r = nodes[0];
  float3 lo = make_float3(FLT_MAX, FLT_MAX, FLT_MAX), hi = make_float3(-FLT_MAX, -FLT_MAX, -FLT_MAX);
  for (int k = 0; k < 4; ++k) {
    if (r.child[k] == 0) continue;
    lo = make_float3(fminf(lo.x, r.lox[k]), fminf(lo.y, r.loy[k]), fminf(lo.z, r.loz[k]));
    hi = make_float3(fmaxf(hi.x, r.hix[k]), fmaxf(hi.y, r.hiy[k]), fmaxf(hi.z, r.hiz[k]));
  }
  auto dA = [](double lx, double ly, double lz, double hx, double hy, double hz) {
    double ex = fmax(0.0, hx - lx), ey = fmax(0.0, hy - ly), ez = fmax(0.0, hz - lz);
    return ex * ey + ey * ez + ez * ex;
  };
  double A0 = dA(lo.x, lo.y, lo.z, hi.x, hi.y, hi.z);
  if (!(A0 > 0.0)) A0 = 1.0;
  double v = 0.0;
  if (i < nn) {
    if (i == 0) v += 1.0;
    const vt_wide_node &nd = nodes[i];
    for (int k = 0; k < 4; ++k) {
      if (nd.child[k] == 0) continue;
      double a = dA(nd.lox[k], nd.loy[k], nd.loz[k], nd.hix[k], nd.hiy[k], nd.hiz[k]) / A0;
      v += nd.child[k] > 0 ? a : a * nd.count[k];
    }
  }
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) atomicAdd(acc, v);
}

inline uint32_t blocks(uint32_t n, uint32_t t) { return (n + t - 1) / t; }

// Bump allocator over one device buffer (256-byte aligned regions). With base == nullptr it only
// measures.
struct ScratchCarve {
  unsigned char *base;
  size_t off = 0;
  template <typename T> T *take(size_t count) {
    size_t bytes = (count * sizeof(T) + 16 + 255) & ~size_t(255);
    T *p = base ? reinterpret_cast<T *>(base + off) : nullptr;
    off += bytes;
    return p;
  }
};

// Temporaries of a build of n faces.
struct BuildScratch {
  float4 *boxes, *leafBox;
  uint32_t *bounds, *codesAlt, *valsAlt, *sortTemp, *flags, *count, *packed, *bar;
  int32_t *parent, *levelA, *levelB;
  float *cost, *firstCost;
  int4 *children;
  uint2 *blockSums;
  BuildReport *report;
  double *sah;
};

constexpr uint32_t kCollapseBlocksMax = 592;  // 4 per SM: more blocks make the barriers and the prefix dearer

void carve_build(ScratchCarve &c, uint32_t n, BuildScratch &b) {
  const uint32_t ni = n > 1 ? n - 1 : 1;
  b.boxes = c.take<float4>(2 * (size_t)n);
  b.leafBox = c.take<float4>(2 * (size_t)n);
  b.bounds = c.take<uint32_t>(16);
  b.codesAlt = c.take<uint32_t>(n);
  b.valsAlt = c.take<uint32_t>(n);
  b.sortTemp = c.take<uint32_t>(vt_radix_temp_words(n));
  b.flags = c.take<uint32_t>(ni);
  b.count = c.take<uint32_t>(ni);
  b.parent = c.take<int32_t>(2 * (size_t)n);
  b.cost = c.take<float>(ni);
  b.firstCost = c.take<float>(ni);
  b.levelA = c.take<int32_t>(n);
  b.levelB = c.take<int32_t>(n);
  b.children = c.take<int4>(n);
  b.packed = c.take<uint32_t>(n);
  b.blockSums = c.take<uint2>(kCollapseBlocksMax);
  b.bar = c.take<uint32_t>(2);
  b.report = c.take<BuildReport>(1);
  b.sah = c.take<double>(1);
}

// The build's outputs and the binary hierarchy they come from (either the mesh's own buffers or the
// caller's).
struct BuildBuffers {
  uint32_t *codes, *sorted;  // Morton codes and face indices, sorted
  int2 *child;               // binary hierarchy: children and boxes per internal node
  float4 *nodeBox;
  vt_wide_node *nodes;
  uint32_t maxNodes;
  int32_t *order;
  float4 *tris, *nrm;        // nrm may be null
  bool markLeaves;           // set the traversal's leaf marks (leaf_ends)
};

// Queues the build up to the collapse on stream s; the report then holds its outcome.
cudaError_t queue_build(const vt_face *faces, uint32_t n, const vt_vertex *verts, uint32_t nverts, int leafSize, int treelet,
                        int rounds, int maxDepth, const BuildBuffers &o, const BuildScratch &b, uint32_t *status, cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(status, 0, sizeof(uint32_t), s);
  if (e == cudaSuccess) e = cudaMemsetAsync(b.bar, 0, 2 * sizeof(uint32_t), s);
  if (e == cudaSuccess) e = cudaMemsetAsync(b.report, 0, sizeof(BuildReport), s);
  if (e != cudaSuccess) return e;
  k_init_bounds<<<1, 32, 0, s>>>(b.bounds);
  k_face_boxes<<<blocks(n, 256), 256, 0, s>>>(faces, n, verts, nverts, b.boxes, b.bounds, status);
  k_morton<<<blocks(n, 256), 256, 0, s>>>(b.boxes, n, b.bounds, o.codes, o.sorted);
  vt_radix_sort_pairs(o.codes, o.sorted, b.codesAlt, b.valsAlt, n, 30, b.sortTemp, status, s);
  k_hierarchy<<<blocks(n, 256), 256, 0, s>>>(o.codes, b.boxes, o.sorted, (int)n, b.leafBox, o.child, b.parent, b.flags, status);
  TreeView t{(int)n, o.child, b.parent, b.leafBox, o.nodeBox, b.count, b.cost};
  if (n >= 3 && treelet > 0) {
    for (int r = 0; r < rounds; ++r)
      k_restructure<<<blocks(n, kRestructureBlock), kRestructureBlock, 0, s>>>(t, b.flags, treelet, r == 0 ? b.firstCost : nullptr, status);
  } else if (n >= 2) {
    k_bottom_up<<<blocks(n, 128), 128, 0, s>>>(t, b.flags, status);
  }
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  // Cooperative (its blocks wait on one another): as many blocks as the widest levels can use, at most
  // what the device holds at once.
  int dev = 0, sms = 0, per = 0;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess || (e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess ||
      (e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_collapse, kCollapseBlock, 0)) != cudaSuccess)
    return e;
  const uint32_t most = std::min<uint32_t>(kCollapseBlocksMax, (uint32_t)(sms * std::max(1, per)));
  const uint32_t grid = std::max(1u, std::min(most, blocks(n, 4 * kCollapseBlock)));
  uint32_t maxNodes = o.maxNodes, *bounds = b.bounds;
  int leaf = leafSize, depth = maxDepth;
  BuildBuffers ob = o;
  BuildScratch sb = b;
  void *args[] = {&t, &leaf, &depth, &maxNodes, &sb.levelA, &sb.levelB, &sb.children, &sb.packed, &sb.blockSums, &sb.bar,
                  &ob.nodes, &ob.sorted, &ob.order, &bounds, &sb.report, &status};
  if ((e = cudaLaunchCooperativeKernel(k_collapse, dim3(grid), dim3(kCollapseBlock), args, 0, s)) != cudaSuccess) return e;
  k_triangles<<<blocks(n, 256), 256, 0, s>>>(faces, n, verts, nverts, o.order, o.tris, o.nrm, o.markLeaves ? 1 : 0);
  return cudaGetLastError();
}

}  // namespace

vt_status vt_lbvh_build(vt_ctx *ctx, const vt_face *faces, uint32_t nfaces, const vt_vertex *verts,
                        uint32_t nverts, const vt_build_options &opt, vt_mesh *mesh) {
  cudaStream_t s = ctx->stream;
  const uint32_t n = nfaces;
  mesh->nfaces = n;
  if (n == 0) { mesh->nnodes = 0; mesh->depth = 0; return VT_OK; }
  int leafSize = opt.leaf_size > 0 ? opt.leaf_size : 2;
  int treelet = opt.treelet_size == 0 ? 7 : opt.treelet_size;
  int rounds = opt.refine_rounds > 0 ? opt.refine_rounds : 2;
  int maxDepth = opt.max_depth > 0 ? opt.max_depth : 31;
  if (leafSize > 8) return vt_fail(ctx, VT_ERR_INVALID, "leaf_size must be in 1..8");
  if (treelet > kMaxTreelet) treelet = kMaxTreelet;
  if (treelet > 0 && treelet < 3) treelet = 3;

  // Temporaries in one buffer of the context's pool, returned to it on every way out.
  struct Temp {
    cudaStream_t s;
    void *p = nullptr;
    ~Temp() {
      if (p) cudaFreeAsync(p, s);
    }
  } temp{s};
  ScratchCarve probe{nullptr};
  BuildScratch b;
  carve_build(probe, n, b);
  VT_CUDA(ctx, vt_pool_alloc(ctx, &temp.p, probe.off));
  ScratchCarve carve{static_cast<unsigned char *>(temp.p)};
  carve_build(carve, n, b);
  // Outputs kept by the mesh (the binary hierarchy for parity checks). The wide node count is bounded by
  // the binary internal count (each wide inner node consumes at least one) plus the root.
  const uint32_t ni = n > 1 ? n - 1 : 1, maxNodes = ni + 1;
  auto keep = [&](auto **p, size_t count) { return vt_pool_alloc(ctx, reinterpret_cast<void **>(p), count * sizeof(**p)); };
  VT_CUDA(ctx, keep(&mesh->d_codes, n));
  VT_CUDA(ctx, keep(&mesh->d_sorted, n));
  VT_CUDA(ctx, keep(&mesh->d_order, n));
  VT_CUDA(ctx, keep(&mesh->d_tris, 3 * (size_t)n));
  VT_CUDA(ctx, keep(&mesh->d_nrm, 3 * (size_t)n));
  VT_CUDA(ctx, keep(&mesh->d_nodes, maxNodes));
  VT_CUDA(ctx, keep(&mesh->d_bin_child, 2 * (size_t)ni));
  VT_CUDA(ctx, keep(&mesh->d_bin_box, 8 * (size_t)ni));
  const BuildBuffers o{mesh->d_codes, reinterpret_cast<uint32_t *>(mesh->d_sorted), reinterpret_cast<int2 *>(mesh->d_bin_child),
                       reinterpret_cast<float4 *>(mesh->d_bin_box), mesh->d_nodes, maxNodes, mesh->d_order, mesh->d_tris,
                       mesh->d_nrm, true};
  VT_CUDA(ctx, cudaEventRecord(ctx->ev0, s));
  VT_CUDA(ctx, queue_build(faces, n, verts, nverts, leafSize, treelet, rounds, maxDepth, o, b, ctx->d_status, s));
  BuildReport r;
  VT_CUDA(ctx, cudaMemcpyAsync(&r, b.report, sizeof r, cudaMemcpyDeviceToHost, s));
  VT_CUDA(ctx, cudaStreamSynchronize(s));
  if (!r.done) return vt_fail(ctx, VT_ERR_DEVICE, "the collapse's grid barrier timed out");
  if (r.status & VT_DEV_SORT) return vt_fail(ctx, VT_ERR_DEVICE, "the Morton sort's look-back timed out");
  if (r.status & VT_DEV_TREELET) return vt_fail(ctx, VT_ERR_DEVICE, "hierarchy inconsistency during the collapse");
  if (r.status & VT_DEV_BAD_INDEX) return vt_fail(ctx, VT_ERR_INVALID, "a face indexes past the vertex array");
  if (r.status & VT_DEV_NONFINITE) return vt_fail(ctx, VT_ERR_INVALID, "a vertex position is not finite");
  if (r.code == kCollapseDepth)
    return vt_fail(ctx, VT_ERR_LIMIT, "BVH depth exceeds max_depth (" + std::to_string(maxDepth) + ")");
  if (r.code == kCollapseNodes) return vt_fail(ctx, VT_ERR_LIMIT, "wide node count exceeds its bound");
  if (r.prims != n) return vt_fail(ctx, VT_ERR_DEVICE, "collapse emitted " + std::to_string(r.prims) + " of " + std::to_string(n) + " triangles");
  mesh->nnodes = r.nodes;
  mesh->depth = r.depth;
  // A mesh without vertex normals shades with geometric normals: no normal buffer to read.
  if (!(r.status & VT_DEV_NORMALS)) {
    VT_CUDA(ctx, cudaFreeAsync(mesh->d_nrm, s));
    mesh->d_nrm = nullptr;
  }
  if (n < 2) {  // no binary hierarchy
    VT_CUDA(ctx, cudaFreeAsync(mesh->d_bin_child, s));
    VT_CUDA(ctx, cudaFreeAsync(mesh->d_bin_box, s));
    mesh->d_bin_child = nullptr;
    mesh->d_bin_box = nullptr;
  }
  {
    const vt_status qs = vt_quantize_nodes(ctx, mesh, s);
    if (qs != VT_OK) return qs;
  }
  VT_CUDA(ctx, cudaMemsetAsync(b.sah, 0, sizeof(double), s));
  k_sah<<<blocks(mesh->nnodes, 256), 256, 0, s>>>(mesh->d_nodes, mesh->nnodes, b.sah);
  VT_CUDA(ctx, cudaEventRecord(ctx->ev1, s));
  double hsah = 0.0;
  VT_CUDA(ctx, cudaMemcpyAsync(&hsah, b.sah, sizeof(double), cudaMemcpyDeviceToHost, s));
  VT_CUDA(ctx, cudaStreamSynchronize(s));
  float ms = 0.0f;
  cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
  mesh->build_ms = ms;
  mesh->sah = (float)hsah;
  float m = 0.0f;
  for (int k = 0; k < 3; ++k) {
    mesh->lo[k] = ord2f(r.bounds[6 + k]);
    mesh->hi[k] = ord2f(r.bounds[9 + k]);
    m = fmaxf(m, fmaxf(fabsf(mesh->lo[k]), fabsf(mesh->hi[k])));
  }
  mesh->root_max = m;
  return VT_OK;
}

// =============================================================================================
// Allocation-free build (vt_mesh_build_noalloc). No counterpart in the reference.
//
// For callers that cannot call cudaMalloc: hosts that run under a fixed device-memory budget
// owned elsewhere (their own arena, or a framework's caching allocator holding the GPU memory),
// and loops that must not pay cudaMalloc/cudaFree's implicit device synchronisation. The caller
// passes the faces, vertices and the output buffers; every temporary of the build comes from
// g_build_scratch, a file-scope device array of kNoAllocScratchBytes that every GPU loading this
// library holds until the process exits. It fits VT_NOALLOC_MAX_FACES faces; larger meshes are
// rejected. The first call on a device looks the array's address up (cudaGetSymbolAddress, with
// that device current) and caches it, so that first call should come before any stream capture.
// Every call blocks the host until its build has finished: it synchronises its stream after the
// collapse (for the node count) and at the end, and on an error after its first launch it still
// waits for the work it queued before returning.
// All calls share the one array and find the previous call's contents in it: every region the
// build needs zeroed is cleared on the call's stream, and two calls overlapping on the GPU (other
// streams or other host threads) race on it.
#include <chrono>
#include <cstring>
#include <mutex>

namespace {

constexpr size_t kNoAllocScratchBytes = size_t(6) << 20;  // 6 MiB per GPU
static __device__ __align__(256) unsigned char g_build_scratch[kNoAllocScratchBytes];

constexpr int kNoAllocMaxDevices = 64;
std::mutex g_scratch_mutex;
unsigned char *g_scratch_addr[kNoAllocMaxDevices] = {};

struct NoAllocBuffers {
  BuildScratch scratch;
  float4 *nodeBox;
  int2 *child;
  uint32_t *codes, *vals, *status;
};

size_t carve_noalloc(unsigned char *base, uint32_t n, NoAllocBuffers &b) {
  ScratchCarve c{base};
  const uint32_t ni = n > 1 ? n - 1 : 1;
  carve_build(c, n, b.scratch);
  b.nodeBox = c.take<float4>(2 * (size_t)ni);
  b.child = c.take<int2>(ni);
  b.codes = c.take<uint32_t>(n);
  b.vals = c.take<uint32_t>(n);
  b.status = c.take<uint32_t>(4);
  return c.off;
}

vt_status noalloc_fail(char *error, uint32_t capacity, vt_status code, const std::string &msg) {
  if (error && capacity) {
    std::strncpy(error, msg.c_str(), capacity - 1);
    error[capacity - 1] = '\0';
  }
  return code;
}

}  // namespace

extern "C" vt_status vt_mesh_build_noalloc(const vt_face *faces, uint32_t nfaces, const vt_vertex *verts,
                                           uint32_t nverts, const vt_build_options *opts,
                                           vt_wide_node *nodes, uint32_t nodes_capacity, float *tris,
                                           int32_t *order, vt_mesh_info *info, void *stream,
                                           char *error, uint32_t error_capacity) {
  auto t_start = std::chrono::steady_clock::now();
  if (error && error_capacity) error[0] = '\0';
  // Once work is queued on the stream, a failing call first waits for it (ignoring the result), so
  // that no kernel of this call still writes the shared scratch array after the call returns.
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  bool queued = false;
  auto fail = [&](vt_status code, const std::string &msg) {
    if (queued) (void)cudaStreamSynchronize(s);
    return noalloc_fail(error, error_capacity, code, msg);
  };
  if (nfaces > VT_NOALLOC_MAX_FACES)
    return fail(VT_ERR_LIMIT, "vt_mesh_build_noalloc: " + std::to_string(nfaces) + " faces exceed the limit of " +
                                  std::to_string(VT_NOALLOC_MAX_FACES) + " (the library's static build scratch)");
  if (!info) return fail(VT_ERR_INVALID, "vt_mesh_build_noalloc: info is null");
  std::memset(info, 0, sizeof *info);
  if (nfaces == 0) return VT_OK;
  if (!faces || !verts || !nodes || !tris || !order)
    return fail(VT_ERR_INVALID, "vt_mesh_build_noalloc: null input or output pointer");
  if (nodes_capacity < nfaces)
    return fail(VT_ERR_INVALID, "vt_mesh_build_noalloc: nodes_capacity must be at least nfaces");
  if ((reinterpret_cast<uintptr_t>(nodes) | reinterpret_cast<uintptr_t>(tris)) & 15u)
    return fail(VT_ERR_INVALID, "vt_mesh_build_noalloc: nodes and tris must be 16-byte aligned");
  vt_build_options o;
  std::memset(&o, 0, sizeof o);
  if (opts) o = *opts;
  const int leafSize = o.leaf_size > 0 ? o.leaf_size : 2;
  int treelet = o.treelet_size == 0 ? 7 : o.treelet_size;
  const int rounds = o.refine_rounds > 0 ? o.refine_rounds : 2;
  const int maxDepth = o.max_depth > 0 ? o.max_depth : 31;
  if (leafSize > 8) return fail(VT_ERR_INVALID, "vt_mesh_build_noalloc: leaf_size must be in 1..8");
  if (treelet > kMaxTreelet) treelet = kMaxTreelet;
  if (treelet > 0 && treelet < 3) treelet = 3;

  // Per-device set-up: the scratch array's device address, looked up once with the device current.
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return fail(VT_ERR_CUDA, std::string("cudaGetDevice: ") + cudaGetErrorString(e));
  if (dev < 0 || dev >= kNoAllocMaxDevices) return fail(VT_ERR_LIMIT, "vt_mesh_build_noalloc: device index too large");
  unsigned char *scratch = nullptr;
  {
    std::lock_guard<std::mutex> lock(g_scratch_mutex);
    if (!g_scratch_addr[dev]) {
      void *p = nullptr;
      e = cudaGetSymbolAddress(&p, g_build_scratch);
      if (e != cudaSuccess) return fail(VT_ERR_CUDA, std::string("cudaGetSymbolAddress(build scratch): ") + cudaGetErrorString(e));
      NoAllocBuffers probe;
      if (carve_noalloc(nullptr, VT_NOALLOC_MAX_FACES, probe) > kNoAllocScratchBytes)
        return fail(VT_ERR_LIMIT, "vt_mesh_build_noalloc: static scratch smaller than the face limit needs");
      g_scratch_addr[dev] = static_cast<unsigned char *>(p);
    }
    scratch = g_scratch_addr[dev];
  }
  NoAllocBuffers b;
  carve_noalloc(scratch, nfaces, b);

  const uint32_t n = nfaces;
#define VT_NA(call)                                                                  \
  do {                                                                               \
    cudaError_t _e = (call);                                                         \
    if (_e != cudaSuccess) return fail(VT_ERR_CUDA, std::string(#call ": ") + cudaGetErrorString(_e)); \
  } while (0)
  queued = true;
  const BuildBuffers out{b.codes, b.vals, b.child, b.nodeBox, nodes, nodes_capacity, order, reinterpret_cast<float4 *>(tris), nullptr, false};
  VT_NA(queue_build(faces, n, verts, nverts, leafSize, treelet, rounds, maxDepth, out, b.scratch, b.status, s));
  BuildReport r;
  VT_NA(cudaMemcpyAsync(&r, b.scratch.report, sizeof r, cudaMemcpyDeviceToHost, s));
  VT_NA(cudaStreamSynchronize(s));
  if (!r.done) return fail(VT_ERR_DEVICE, "vt_mesh_build_noalloc: the collapse's grid barrier timed out");
  if (r.status & VT_DEV_SORT) return fail(VT_ERR_DEVICE, "vt_mesh_build_noalloc: the Morton sort's look-back timed out");
  if (r.status & VT_DEV_BAD_INDEX) return fail(VT_ERR_INVALID, "vt_mesh_build_noalloc: a face indexes past the vertex array");
  if (r.status & VT_DEV_NONFINITE) return fail(VT_ERR_INVALID, "vt_mesh_build_noalloc: a vertex position is not finite");
  if (r.status & VT_DEV_TREELET) return fail(VT_ERR_DEVICE, "vt_mesh_build_noalloc: hierarchy inconsistency");
  if (r.code == kCollapseDepth) return fail(VT_ERR_LIMIT, "vt_mesh_build_noalloc: BVH depth exceeds max_depth");
  if (r.code == kCollapseNodes) return fail(VT_ERR_LIMIT, "vt_mesh_build_noalloc: wide nodes exceed nodes_capacity");
  if (r.prims != n) return fail(VT_ERR_DEVICE, "vt_mesh_build_noalloc: collapse emitted too few triangles");
  VT_NA(cudaMemsetAsync(b.scratch.sah, 0, sizeof(double), s));
  k_sah<<<blocks(r.nodes, 256), 256, 0, s>>>(nodes, r.nodes, b.scratch.sah);
  VT_NA(cudaGetLastError());
  double hsah = 0.0;
  VT_NA(cudaMemcpyAsync(&hsah, b.scratch.sah, sizeof(double), cudaMemcpyDeviceToHost, s));
  VT_NA(cudaStreamSynchronize(s));
#undef VT_NA
  info->faces = n;
  info->wide_nodes = r.nodes;
  info->binary_nodes = n - 1;
  info->depth = r.depth;
  info->sah_cost = (float)hsah;
  for (int k = 0; k < 3; ++k) {
    info->lo[k] = ord2f(r.bounds[6 + k]);
    info->hi[k] = ord2f(r.bounds[9 + k]);
  }
  info->build_ms = std::chrono::duration<float, std::milli>(std::chrono::steady_clock::now() - t_start).count();
  return VT_OK;
}
