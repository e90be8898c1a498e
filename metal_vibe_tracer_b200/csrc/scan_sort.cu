// scan_sort.cu — the stable LSD radix sort of the LBVH build.
//
// Bound: HBM, or launches for small inputs. One pass over the keys counts the digits of every pass; then
// each 8-bit digit takes one launch that reads and writes the pairs once (four passes for 30-bit Morton
// codes): the tiles' running digit offsets come from a decoupled look-back over the tiles before it (Merrill
// and Garland, "Single-pass Parallel Prefix Scan with Decoupled Look-back", 2016; in a digit sort Adinets and
// Merrill, "Onesweep", 2022) instead of a histogram launch, a scan and a scatter per digit. Within a tile the
// pairs are ranked by (digit, warp, item, lane), the order they appear in memory, so the sort is stable, and
// are reordered in shared memory so that each digit's run is stored contiguously. Eight 4-bit passes of
// histogram, scan and scatter launches took 391 us for 1M pairs (44 launches) before.
#include "vt_internal.cuh"

namespace {

constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kSortItems = 12;
constexpr int kSortTile = kSortThreads * kSortItems;  // 3072 pairs per tile
constexpr int kDigits = 256;
constexpr int kMaxPasses = 4;
// Tile states of the look-back, in the two top bits of a word whose low bits hold a count (pairs
// number fewer than 2^30).
constexpr uint32_t kPartial = 1u << 30, kPrefix = 2u << 30, kCountMask = kPartial - 1u;
// Look-back polls before a tile gives up (a tile's predecessors have all started, so this is never
// reached unless a launch is broken); the sort then reports VT_DEV_SORT, and its output holds some pairs twice
// and others' slots unwritten. (0: every look-back gives up, for the test of that.)
#ifndef VT_SORT_SPIN_LIMIT
#define VT_SORT_SPIN_LIMIT (1u << 21)
#endif
constexpr uint32_t kSpinLimit = VT_SORT_SPIN_LIMIT;

// Temporary words: digit counts of each pass, tile tickets, then the tile states of each pass.
constexpr uint32_t kTicketAt = kMaxPasses * kDigits, kStateAt = kTicketAt + 64;

__device__ __forceinline__ uint32_t digit_of(uint32_t key, int shift) { return (key >> shift) & (kDigits - 1); }

__global__ void __launch_bounds__(kSortThreads) k_radix_count(const uint32_t *__restrict__ keys, uint32_t n, int passes,
                                                                uint32_t *temp) {
  __shared__ uint32_t cnt[kMaxPasses][kDigits];
  for (int p = 0; p < passes; ++p) cnt[p][threadIdx.x] = 0;
  __syncthreads();
  for (uint32_t i = blockIdx.x * kSortThreads + threadIdx.x; i < n; i += gridDim.x * kSortThreads) {
    const uint32_t k = keys[i];
    for (int p = 0; p < passes; ++p) atomicAdd(&cnt[p][digit_of(k, 8 * p)], 1u);
  }
  __syncthreads();
  for (int p = 0; p < passes; ++p)
    if (cnt[p][threadIdx.x]) atomicAdd(temp + p * kDigits + threadIdx.x, cnt[p][threadIdx.x]);
}

// Exclusive prefix over the block of one value per thread.
__device__ __forceinline__ uint32_t block_exclusive(uint32_t v, uint32_t *warpSums) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t u = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += u;
  }
  if (lane == 31) warpSums[warp] = inc;
  __syncthreads();
  uint32_t before = 0;
#pragma unroll
  for (int w = 0; w < kSortWarps; ++w) before += w < warp ? warpSums[w] : 0u;
  __syncthreads();
  return before + inc - v;
}

__global__ void __launch_bounds__(kSortThreads) k_radix_pass(const uint32_t *__restrict__ keys, const uint32_t *__restrict__ vals,
                                                               uint32_t n, int pass, uint32_t *temp, uint32_t tiles,
                                                               uint32_t *__restrict__ keysOut, uint32_t *__restrict__ valsOut,
                                                               uint32_t *status) {
  __shared__ uint32_t cnt[kSortWarps][kDigits];  // per warp: running digit counts, then offsets in the tile
  __shared__ uint32_t sKeys[kSortTile], sVals[kSortTile];
  __shared__ uint32_t out[kDigits];              // destination of a digit's run minus its place in the tile
  __shared__ uint32_t warpSums[kSortWarps];
  __shared__ uint32_t sTile;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5, shift = 8 * pass;
  if (t == 0) sTile = atomicAdd(temp + kTicketAt + pass, 1u);  // tiles in the order they start
#pragma unroll
  for (int w = 0; w < kSortWarps; ++w) cnt[w][t] = 0;
  __syncthreads();
  const uint32_t tile = sTile, base = tile * kSortTile, valid = min((uint32_t)kSortTile, n - base);
  // Item j of lane l of warp w is pair (w * items + j) * 32 + l of the tile.
  uint32_t key[kSortItems], val[kSortItems];
#pragma unroll
  for (int j = 0; j < kSortItems; ++j) {
    const uint32_t at = (uint32_t)(warp * kSortItems + j) * 32u + lane;
    key[j] = at < valid ? keys[base + at] : 0xffffffffu;
    val[j] = at < valid ? vals[base + at] : 0u;
  }
  uint32_t rank[kSortItems];
#pragma unroll
  for (int j = 0; j < kSortItems; ++j) {
    const bool in = (uint32_t)(warp * kSortItems + j) * 32u + lane < valid;
    const uint32_t d = digit_of(key[j], shift);
    const unsigned peers = __match_any_sync(0xffffffffu, in ? d : kDigits);  // past-the-end lanes among themselves
    const uint32_t before = __popc(peers & ((1u << lane) - 1u));
    rank[j] = in ? cnt[warp][d] + before : 0u;
    __syncwarp();
    if (in && before == 0) cnt[warp][d] += __popc(peers);
    __syncwarp();
  }
  __syncthreads();
  // Thread d owns digit d: the warps' counts become offsets, their sum the tile's count.
  uint32_t total = 0;
#pragma unroll
  for (int w = 0; w < kSortWarps; ++w) {
    const uint32_t c = cnt[w][t];
    cnt[w][t] = total;
    total += c;
  }
  uint32_t *state = temp + kStateAt + ((size_t)pass * tiles + tile) * kDigits + t;
  atomicExch(state, (tile == 0 ? kPrefix : kPartial) | total);
  const uint32_t start = block_exclusive(total, warpSums);                           // the digit's place in the tile
  const uint32_t first = block_exclusive(__ldcg(temp + pass * kDigits + t), warpSums);  // and in the output
  // Pairs of this digit in the tiles before this one.
  uint32_t before = 0;
  for (uint32_t p = tile; p > 0;) {
    uint32_t s = 0;
    for (uint32_t spins = 0; spins < kSpinLimit && (s & ~kCountMask) == 0u; ++spins)
      s = vt_poll(temp + kStateAt + ((size_t)pass * tiles + (p - 1)) * kDigits + t);
    if ((s & ~kCountMask) == 0u) {
      atomicOr(status, (uint32_t)VT_DEV_SORT);
      break;
    }
    before += s & kCountMask;
    if (s & kPrefix) break;
    --p;
  }
  if (tile > 0) atomicExch(state, kPrefix | (before + total));
  out[t] = first + before - start;
#pragma unroll
  for (int w = 0; w < kSortWarps; ++w) cnt[w][t] += start;
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kSortItems; ++j) {
    if ((uint32_t)(warp * kSortItems + j) * 32u + lane >= valid) continue;
    const uint32_t at = cnt[warp][digit_of(key[j], shift)] + rank[j];
    sKeys[at] = key[j];
    sVals[at] = val[j];
  }
  __syncthreads();
  for (uint32_t at = t; at < valid; at += kSortThreads) {
    const uint32_t k = sKeys[at], to = out[digit_of(k, shift)] + at;
    if (to < n) {  // holds unless a look-back gave up
      keysOut[to] = k;
      valsOut[to] = sVals[at];
    }
  }
}

}  // namespace

size_t vt_radix_temp_words(uint32_t n) {
  const size_t tiles = ((size_t)n + kSortTile - 1) / kSortTile;
  return kStateAt + (size_t)kMaxPasses * tiles * kDigits;
}

void vt_radix_sort_pairs(uint32_t *keys, uint32_t *vals, uint32_t *keys_alt, uint32_t *vals_alt,
                         uint32_t n, int bits, uint32_t *temp, uint32_t *status, cudaStream_t s) {
  if (n <= 1) return;
  const uint32_t tiles = (n + kSortTile - 1) / kSortTile;
  const int passes = (bits + 7) / 8;
  cudaMemsetAsync(temp, 0, (kStateAt + (size_t)passes * tiles * kDigits) * sizeof(uint32_t), s);
  k_radix_count<<<tiles < 592u ? tiles : 592u, kSortThreads, 0, s>>>(keys, n, passes, temp);
  uint32_t *srcK = keys, *srcV = vals, *dstK = keys_alt, *dstV = vals_alt;
  for (int p = 0; p < passes; ++p) {
    k_radix_pass<<<tiles, kSortThreads, 0, s>>>(srcK, srcV, n, p, temp, tiles, dstK, dstV, status);
    uint32_t *tk = srcK, *tv = srcV;
    srcK = dstK; srcV = dstV; dstK = tk; dstV = tv;
  }
  if (srcK != keys) {
    cudaMemcpyAsync(keys, srcK, n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, s);
    cudaMemcpyAsync(vals, srcV, n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, s);
  }
}
