// Stable LSD radix sort of (64-bit key, 32-bit value) pairs, one digit of at
// most 8 bits per pass, as three launches per pass:
//   count    every tile of kSortTile pairs counts its digits (one count per
//            digit and tile, digit-major)
//   scan     one block per digit scans that digit's counts over the tiles
//   scatter  every tile ranks its pairs (stable: warps own consecutive
//            segments and rank equal digits by match groups), lays them out
//            in digit order in shared memory and writes each digit's run to
//            its place: full sectors instead of one 12-byte store per pair
// The first pass takes its pairs from a source functor (the edge list), so
// they are not written before they are sorted, and may drop some: the later
// passes run on what is left.  Tiles do not wait on one another.
// What bounds it: 24 bytes moved per pair and pass by the scatter and 8 by the
// count, and the instructions and shared-memory accesses of a tile's phases
// (ranks, digit places, staging): of RMAT-20's pairs the scatter moves 0.72 GB
// to and from HBM and has L1 and shared memory at 69%, its issue slots at 61%
// and HBM at 42%; the count is at 41% of HBM, waiting for its loads.
// It replaced one cooperative kernel whose CTAs sorted their ranges 512 pairs
// a round behind four block barriers: RMAT-20's edge list (33.5 M entries)
// 7.2 -> 2.0 ms with the compaction.
#pragma once

#include "engine_common.cuh"

namespace sgb {
namespace rsort {

using u64 = unsigned long long;
using sygraph::detail::kFullMask;

// 384 threads of 8 pairs, three blocks an SM: 56 registers without spills.
// Of 33.5 M pairs a scatter took 236 us (0.81 GB of pairs read and written, 3.4 TB/s) against 395
// us for 512 threads of 16 pairs (two blocks an SM, spills), 258 us for 512 x
// 8 at three blocks (spills), 250 us for 512 x 8 at two and 247 us for 384 x 8
// at four; the lanes' equal digits by eight votes or by match instructions
// made no difference.
constexpr uint32_t kSortThreads = 384, kSortWarps = kSortThreads / 32;
constexpr uint32_t kSortItems = 8;
constexpr uint32_t kSortBlocks = 3;  // per SM
constexpr uint32_t kSortTile = kSortThreads * kSortItems;
constexpr uint32_t kDigits = 256;

// Pairs that an earlier pass wrote.
struct ArraySource {
  const u64* key;
  const uint32_t* val;
  const uint32_t* count;  // device word: pairs left after the first pass
  __device__ __forceinline__ uint32_t size() const { return *count; }
  __device__ __forceinline__ bool key_at(uint32_t i, u64* k) const {
    *k = key[i];
    return true;
  }
  __device__ __forceinline__ uint32_t val_at(uint32_t i) const { return val[i]; }
};

template <class Source>
__global__ void __launch_bounds__(kSortThreads) count_kernel(Source src, uint32_t shift, uint32_t mask,
                                                             uint32_t tiles, uint32_t* __restrict__ hist) {
  __shared__ uint32_t s_cnt[kSortWarps / 4][kDigits];  // one histogram per four warps
  for (uint32_t x = threadIdx.x; x < kSortWarps / 4 * kDigits; x += kSortThreads) (&s_cnt[0][0])[x] = 0u;
  __syncthreads();
  const uint32_t n = src.size();
  const uint64_t base = (uint64_t)blockIdx.x * kSortTile;
  uint32_t* mine = s_cnt[threadIdx.x >> 7];
#pragma unroll
  for (uint32_t r = 0; r < kSortItems; r++) {
    const uint64_t i = base + r * kSortThreads + threadIdx.x;
    u64 k = 0;
    if (i < n && src.key_at((uint32_t)i, &k)) atomicAdd(mine + ((uint32_t)(k >> shift) & mask), 1u);
  }
  __syncthreads();
  if (threadIdx.x <= mask) {
    uint32_t c = 0;
#pragma unroll
    for (uint32_t h = 0; h < kSortWarps / 4; h++) c += s_cnt[h][threadIdx.x];
    hist[(size_t)threadIdx.x * tiles + blockIdx.x] = c;
  }
}

// Block d: exclusive scan of digit d's counts over the tiles, in place, and
// their sum.
__global__ void __launch_bounds__(kSortThreads) scan_kernel(uint32_t tiles, uint32_t* __restrict__ hist,
                                                            uint32_t* __restrict__ total) {
  __shared__ uint32_t s_scan[32];
  uint32_t* h = hist + (size_t)blockIdx.x * tiles;
  uint32_t carry = 0;
  for (uint32_t t0 = 0; t0 < tiles; t0 += kSortThreads * 8) {
    uint32_t x[8], sum = 0;
#pragma unroll
    for (uint32_t k = 0; k < 8; k++) {
      const uint32_t t = t0 + threadIdx.x * 8 + k;
      x[k] = t < tiles ? h[t] : 0u;
      sum += x[k];
    }
    uint32_t all;
    uint32_t run = carry + sygraph::detail::block_excl_scan(sum, &all, s_scan);
#pragma unroll
    for (uint32_t k = 0; k < 8; k++) {
      const uint32_t t = t0 + threadIdx.x * 8 + k;
      if (t < tiles) h[t] = run;
      run += x[k];
    }
    carry += all;
  }
  if (threadIdx.x == 0) total[blockIdx.x] = carry;
}

struct ScatterShared {
  u64 key[kSortTile];
  uint32_t val[kSortTile];
  uint32_t start[kDigits];  // first place of a digit in the tile
  uint32_t out[kDigits];    // its place in the output, less `start`
  uint32_t scan[32];
};
static_assert(sizeof(u64) * kSortTile >= sizeof(uint32_t) * kSortWarps * kDigits, "the counts share the key staging");

template <class Source>
__global__ void __launch_bounds__(kSortThreads, kSortBlocks) scatter_kernel(Source src, uint32_t shift, uint32_t mask,
                                                                  uint32_t tiles, const uint32_t* __restrict__ hist,
                                                                  const uint32_t* __restrict__ total,
                                                                  u64* __restrict__ kout, uint32_t* __restrict__ vout,
                                                                  uint32_t* count_out) {
  extern __shared__ __align__(16) unsigned char s_raw[];
  ScatterShared& S = *reinterpret_cast<ScatterShared*>(s_raw);
  uint32_t(*cnt)[kDigits] = reinterpret_cast<uint32_t(*)[kDigits]>(S.key);  // before the keys are staged
  const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
  const uint32_t n = src.size(), first = blockIdx.x * kSortTile;
  const uint32_t here = n > first ? n - first : 0u;  // pairs from the tile's start on
  const uint32_t at0 = warp * (32 * kSortItems) + lane;
  for (uint32_t x = t; x < kSortWarps * kDigits; x += kSortThreads) (&cnt[0][0])[x] = 0u;
  u64 k[kSortItems];
  uint32_t valid = 0;
#pragma unroll
  for (uint32_t r = 0; r < kSortItems; r++) {
    k[r] = 0;
    if (at0 + r * 32 < here && src.key_at(first + at0 + r * 32, &k[r])) valid |= 1u << r;
  }
  const uint32_t whole = t <= mask ? total[t] : 0u;
  const uint32_t tile_before = t <= mask ? hist[(size_t)t * tiles + blockIdx.x] : 0u;
  __syncthreads();
  // rank of each pair among the warp's earlier ones of its digit, two in a word
  uint32_t rank[kSortItems / 2];
#pragma unroll
  for (uint32_t r = 0; r < kSortItems; r++) {
    const bool in = (valid >> r) & 1u;
    const uint32_t d = (uint32_t)(k[r] >> shift) & mask;
    // the lanes of the same digit, by eight votes
    uint32_t grp = __ballot_sync(kFullMask, in);
#pragma unroll
    for (uint32_t bit = 0; bit < 8; bit++) {
      const bool one = (d >> bit) & 1u;
      const uint32_t ones = __ballot_sync(kFullMask, one);
      grp &= one ? ones : ~ones;
    }
    const uint32_t before = in ? cnt[warp][d] : 0u;
    __syncwarp();
    if (in && (grp >> lane) == 1u) cnt[warp][d] = before + __popc(grp);  // the group's last lane
    __syncwarp();
    const uint32_t x = before + __popc(grp & ((1u << lane) - 1u));
    rank[r / 2] = r & 1 ? rank[r / 2] | x << 16 : x;
  }
  uint32_t val[kSortItems];  // on their way while the digits are placed
#pragma unroll
  for (uint32_t r = 0; r < kSortItems; r++) val[r] = (valid >> r) & 1u ? src.val_at(first + at0 + r * 32) : 0u;
  __syncthreads();
  // digit starts in the tile and in the output
  uint32_t sum = 0;
  if (t < kDigits) {
#pragma unroll
    for (uint32_t w = 0; w < kSortWarps; w++) {
      const uint32_t x = cnt[w][t];
      cnt[w][t] = sum;
      sum += x;
    }
  }
  uint32_t staged, all;
  const uint32_t start = sygraph::detail::block_excl_scan(t < kDigits ? sum : 0u, &staged, S.scan);
  const uint32_t gbase = sygraph::detail::block_excl_scan(whole, &all, S.scan);
  if (t < kDigits) {
    S.start[t] = start;
    S.out[t] = gbase + tile_before - start;
  }
  if (count_out && blockIdx.x == 0 && t == 0) *count_out = all;
  __syncthreads();
#pragma unroll
  for (uint32_t r = 0; r < kSortItems; r++) {
    const uint32_t d = (uint32_t)(k[r] >> shift) & mask;
    rank[r / 2] += (cnt[warp][d] + S.start[d]) << (r & 1 ? 16 : 0);
  }
  __syncthreads();  // the counts are read: the keys take their place
#pragma unroll
  for (uint32_t r = 0; r < kSortItems; r++) {
    if ((valid >> r) & 1u) {
      const uint32_t at = rank[r / 2] >> (r & 1 ? 16 : 0) & 0xffffu;
      S.key[at] = k[r];
      S.val[at] = val[r];
    }
  }
  __syncthreads();
#pragma unroll
  for (uint32_t r = 0; r < kSortItems; r++) {
    const uint32_t i = r * kSortThreads + t;
    if (i < staged) {
      const u64 key = S.key[i];
      const uint32_t at = S.out[(uint32_t)(key >> shift) & mask] + i;
      kout[at] = key;
      vout[at] = S.val[i];
    }
  }
}

inline uint32_t tiles_of(uint64_t entries) { return entries ? (uint32_t)((entries - 1) / kSortTile + 1) : 1u; }
// Words of scratch of a sort of `entries` pairs: the tile counts, the digit
// totals and the count of pairs left.
inline uint64_t scratch_words(uint64_t entries) { return (uint64_t)kDigits * tiles_of(entries) + kDigits + 1; }

// Sorts what `src` yields (at most `entries` pairs) on key bits [0, bits);
// k[1] / v[1] take the first pass's output, k[0] / v[0] the second's, and so
// on: the sorted pairs end in k[passes & 1].  *left points at the device word
// with their number.
template <class Source>
sg_status sort_pairs(const Source& src, uint64_t entries, uint32_t bits, u64* (&k)[2], uint32_t* (&v)[2],
                     uint32_t* scratch, cudaStream_t st, uint32_t* passes_out, uint32_t** left) {
  const uint32_t tiles = tiles_of(entries), passes = bits ? (bits + 7) / 8 : 1;
  uint32_t *hist = scratch, *total = hist + (uint64_t)kDigits * tiles, *count = total + kDigits;
  // a scatter block holds its tile in shared memory; the attribute is per
  // function and device, and cheap to set again
  SG_CUDA(cudaFuncSetAttribute(scatter_kernel<Source>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)sizeof(ScatterShared)));
  SG_CUDA(cudaFuncSetAttribute(scatter_kernel<ArraySource>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)sizeof(ScatterShared)));
  uint32_t shift = 0;
  for (uint32_t p = 0; p < passes; p++) {
    const uint32_t width = (bits - shift + (passes - p) - 1) / (passes - p);  // digits of about equal width
    const uint32_t mask = (1u << width) - 1u;
    u64* ko = k[(p + 1) & 1];
    uint32_t* vo = v[(p + 1) & 1];
    if (p == 0) {
      count_kernel<<<tiles, kSortThreads, 0, st>>>(src, shift, mask, tiles, hist);
    } else {
      const ArraySource a{k[p & 1], v[p & 1], count};
      count_kernel<<<tiles, kSortThreads, 0, st>>>(a, shift, mask, tiles, hist);
    }
    SG_CHECK_LAUNCH();
    scan_kernel<<<mask + 1, kSortThreads, 0, st>>>(tiles, hist, total);
    SG_CHECK_LAUNCH();
    if (p == 0) {
      scatter_kernel<<<tiles, kSortThreads, sizeof(ScatterShared), st>>>(src, shift, mask, tiles, hist, total, ko, vo,
                                                                        count);
    } else {
      const ArraySource a{k[p & 1], v[p & 1], count};
      scatter_kernel<<<tiles, kSortThreads, sizeof(ScatterShared), st>>>(a, shift, mask, tiles, hist, total, ko, vo,
                                                                        (uint32_t*)nullptr);
    }
    SG_CHECK_LAUNCH();
    shift += width;
  }
  *passes_out = passes;
  *left = count;
  return SG_OK;
}

}  // namespace rsort
}  // namespace sgb
