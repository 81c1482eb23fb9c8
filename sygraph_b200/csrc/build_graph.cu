// Graph construction on the device: edge list -> CSR (forward, and the
// inverse for directed graphs).  The reference builds on the host:
// io::csr::fromCOO (io/read_csr.hpp:260-300), formats::CSR::invert
// (formats/csr.hpp:179-209) and the upload of GraphCSR
// (graph/impls/graph_csr.hpp:394-426); sg_csr_from_edges is that host path.
// Here:
//   sort    entry 2i / 2i+1 (or i) = (u, v) / (v, u) of edge i as the key
//           u * 2^b + v (2^b >= n), by a stable radix sort (radix_sort.cuh)
//           whose first pass makes the entries from the edge list and leaves
//           the dropped ones out (a self-loop when they are dropped, the
//           reverse of a self-loop); equal keys keep their insertion order
//   compact the first entry of every run of equal keys (every entry without
//           de-duplication) is kept, in order: columns, values, and the row
//           offset of each non-empty row; empty rows take the next row's
//           offset by a backward minimum scan
// The result is bit-identical to the host path's (stable sort by key, keep
// the first of equal keys).
#include <algorithm>
#include <cstring>
#include <mutex>
#include <vector>

#include "radix_sort.cuh"

namespace sgb {
namespace gb {

using rsort::u64;
using sygraph::detail::kFullMask;

// The entries of an edge list, in insertion order.
struct EdgeSource {
  const uint32_t* src;
  const uint32_t* dst;
  const uint32_t* val;  // nullptr: every value is `one`
  uint32_t entries;
  uint32_t n;
  uint32_t b;  // bits per endpoint (2^b >= n)
  uint32_t one;
  int symmetrize, drop_self_loops;
  uint32_t* bad;  // an endpoint was >= n
  __device__ __forceinline__ uint32_t size() const { return entries; }
  __device__ __forceinline__ bool key_at(uint32_t i, u64* k) const {
    const uint32_t j = symmetrize ? i >> 1 : i;
    const bool rev = symmetrize && (i & 1u);
    const uint32_t u = src[j], v = dst[j];
    if (u >= n || v >= n) {
      *bad = 1u;
      return false;
    }
    *k = rev ? ((u64)v << b) | u : ((u64)u << b) | v;
    return u != v || !(drop_self_loops || rev);
  }
  __device__ __forceinline__ uint32_t val_at(uint32_t i) const { return val ? val[symmetrize ? i >> 1 : i] : one; }
};

// Sorted keys are compacted in tiles, one bit per kept entry (the first of
// its run of equal keys, or every entry without de-duplication).
constexpr uint32_t kKeepThreads = 512, kKeepItems = 8, kKeepTile = kKeepThreads * kKeepItems;

// Bit r: entry base + 32 r is kept; `base` is the lane's first entry.
__device__ __forceinline__ uint32_t keep_bits(const u64* __restrict__ key, uint32_t count, int dedupe, uint64_t base) {
  uint32_t bits = 0;
#pragma unroll
  for (uint32_t r = 0; r < kKeepItems; r++) {
    const uint64_t i = base + 32 * r;
    if (i < count && (!dedupe || i == 0 || key[i - 1] != key[i])) bits |= 1u << r;
  }
  return bits;
}

__global__ void __launch_bounds__(kKeepThreads) keep_count_kernel(const u64* __restrict__ key, const uint32_t* count,
                                                                  int dedupe, uint32_t* __restrict__ tile_kept) {
  __shared__ uint32_t s_red[32];
  const uint64_t base =
      (uint64_t)blockIdx.x * kKeepTile + (threadIdx.x >> 5) * (32 * kKeepItems) + (threadIdx.x & 31u);
  const uint32_t kept = sygraph::detail::block_sum<uint32_t>(__popc(keep_bits(key, *count, dedupe, base)), s_red);
  if (threadIdx.x == 0) tile_kept[blockIdx.x] = kept;
}

__global__ void __launch_bounds__(kKeepThreads) keep_write_kernel(const u64* __restrict__ key,
                                                                  const uint32_t* __restrict__ val,
                                                                  const uint32_t* count, int dedupe, uint32_t b,
                                                                  const uint32_t* __restrict__ tile_first,
                                                                  const uint32_t* kept_total, uint32_t n,
                                                                  uint32_t* __restrict__ ro, uint32_t* __restrict__ col,
                                                                  uint32_t* __restrict__ oval) {
  __shared__ uint32_t s_scan[32];
  const uint32_t lane = threadIdx.x & 31u;
  const uint64_t base = (uint64_t)blockIdx.x * kKeepTile + (threadIdx.x >> 5) * (32 * kKeepItems) + lane;
  const uint32_t bits = keep_bits(key, *count, dedupe, base);
  // kept entries before the warp's segment
  const uint32_t mine = sygraph::detail::warp_sum(__popc(bits));
  uint32_t all;
  uint32_t pos = sygraph::detail::block_excl_scan(lane == 0 ? mine : 0u, &all, s_scan);
  pos = tile_first[blockIdx.x] + __shfl_sync(kFullMask, pos, 0);
#pragma unroll
  for (uint32_t r = 0; r < kKeepItems; r++) {
    const bool keep = (bits >> r) & 1u;
    const uint32_t m = __ballot_sync(kFullMask, keep);
    if (keep) {
      const uint64_t i = base + 32 * r;
      const uint32_t at = pos + __popc(m & ((1u << lane) - 1u));
      const u64 k = key[i];
      const uint32_t s = (uint32_t)(k >> b);
      col[at] = (uint32_t)k & (uint32_t)((1ull << b) - 1u);
      oval[at] = val[i];
      // first kept entry of row s: nothing before it in the sorted order
      // shares its row (a duplicate of the same key shares it and is not kept)
      if (i == 0 || (uint32_t)(key[i - 1] >> b) != s) ro[s] = at;
    }
    pos += __popc(m);
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) ro[n] = *kept_total;
}

// Rows without edges hold the all-ones word; they take the offset of the next
// row that has some: a suffix minimum over ro[0, n] (ro[n] = m is set), by
// tile minima, their suffix minima in one block, and the tiles again.
__device__ __forceinline__ uint32_t block_suffix_min(uint32_t x, uint32_t* s_min) {
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t y = __shfl_down_sync(kFullMask, x, d);
    if (lane + d < 32) x = min(x, y);
  }
  if (lane == 0) s_min[warp] = x;
  __syncthreads();
  uint32_t later = 0xffffffffu;
  for (uint32_t w = warp + 1; w < nw; w++) later = min(later, s_min[w]);
  __syncthreads();
  return min(x, later);
}

__global__ void __launch_bounds__(kKeepThreads) row_min_kernel(const uint32_t* __restrict__ ro, uint64_t rows,
                                                               uint32_t* __restrict__ tile_min) {
  __shared__ uint32_t s_min[32];
  uint32_t mn = 0xffffffffu;
#pragma unroll
  for (uint32_t r = 0; r < kKeepItems; r++) {
    const uint64_t v = (uint64_t)blockIdx.x * kKeepTile + r * kKeepThreads + threadIdx.x;
    if (v < rows) mn = min(mn, ro[v]);
  }
  mn = block_suffix_min(mn, s_min);
  if (threadIdx.x == 0) tile_min[blockIdx.x] = mn;
}

// One block: tile_min[t] = minimum over the tiles after t.
__global__ void __launch_bounds__(1024) row_carry_kernel(uint32_t* __restrict__ tile_min, uint32_t tiles) {
  __shared__ uint32_t s_min[32], s_all;
  uint32_t carry = 0xffffffffu;
  for (uint32_t end = tiles; end;) {
    const uint32_t beg = end > blockDim.x ? end - blockDim.x : 0u, t = beg + threadIdx.x;
    const uint32_t x = t < end ? tile_min[t] : 0xffffffffu;
    // suffix minimum of the tiles after t: shift by one
    const uint32_t later = t + 1 < end ? tile_min[t + 1] : 0xffffffffu;
    const uint32_t y = min(block_suffix_min(later, s_min), carry);
    if (threadIdx.x == 0) s_all = min(min(x, y), carry);
    __syncthreads();
    if (t < end) tile_min[t] = y;
    carry = s_all;
    __syncthreads();
    end = beg;
  }
}

__global__ void __launch_bounds__(kKeepThreads) row_fill_kernel(uint32_t* __restrict__ ro, uint64_t rows,
                                                                const uint32_t* __restrict__ tile_later) {
  __shared__ uint32_t s_min[32], s_all;
  uint32_t carry = tile_later[blockIdx.x];
  for (uint32_t r = kKeepItems; r--;) {
    const uint64_t v = (uint64_t)blockIdx.x * kKeepTile + r * kKeepThreads + threadIdx.x;
    const uint32_t x = v < rows ? ro[v] : 0xffffffffu;
    const uint32_t y = min(block_suffix_min(x, s_min), carry);
    if (v < rows && x != y) ro[v] = y;
    if (threadIdx.x == 0) s_all = y;
    __syncthreads();
    carry = s_all;
    __syncthreads();
  }
}

// ---- weight-sorted adjacency (delta-stepping SSSP) ---------------------------
//
// Every row of the forward CSR sorted by weight, on the device: the pairs
// (row << 32 | weight bits, column) of all edges, filled in row order, are
// radix-sorted (stable, so equal weights keep their column order); weights
// are non-negative float32 or uint32, whose bit patterns order like the
// values.  The fill also checks whether the weighted adjacency is symmetric
// (each row strictly increasing in column, every edge's reverse present with
// the same weight), which the pull phases of delta-stepping need.
//
// Of the two edges between u and v it is the one towards the smaller end (by
// degree, then id) whose reverse is looked up, by a binary search of the
// smaller row; where all of those have theirs and there are as many edges
// towards the larger end, every edge has.
struct WsortParams {
  const uint32_t* ro;
  const uint32_t* col;
  const uint32_t* val;
  uint32_t n, m;
  u64* k0;
  uint32_t* v0;
  uint32_t* asym;       // set when a row is not increasing or a reverse is missing
  u64* towards;         // edges towards their smaller end, and towards their larger one
};

// A warp takes up to kWsRun runs of 32 edges in a row, a lane per edge.  (A thread
// per short row and a warp per long one took 10 ms on RMAT-22 and another 42
// for its largest hub; this form 6.)
constexpr uint32_t kWsRun = 32;

__global__ void __launch_bounds__(256) ws_fill_kernel(WsortParams P) {
  __shared__ u64 s_red[32];
  const uint32_t lane = threadIdx.x & 31u, words = (P.m - 1) / 32 + 1;
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  const uint32_t run = min(kWsRun, max(1u, words / nwarps));
  bool bad = false;
  u64 smaller = 0, larger = 0;
  for (uint32_t w0 = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * run; w0 < words; w0 += nwarps * run) {
    uint32_t row = eng::row_of_edge(P.ro, P.n, w0 * 32u);
    for (uint32_t w = w0; w < min(w0 + run, words); w++) {
      const uint32_t e0 = w * 32u;
      const uint32_t v = eng::word_source(P.ro, P.n, P.m, row, e0);
      row = __shfl_sync(kFullMask, v, 31);
      if (lane > P.m - 1u - e0) continue;  // the last word; no collective follows in this turn
      const uint32_t i = e0 + lane, u = P.col[i], x = P.val[i];
      P.k0[i] = ((u64)v << 32) | x;
      P.v0[i] = u;
      const uint32_t vb = P.ro[v], ve = P.ro[v + 1], end = P.ro[u + 1];
      uint32_t lo = P.ro[u], hi = end;
      if (i + 1 < ve && u >= P.col[i + 1]) bad = true;
      const uint32_t dv = ve - vb, du = end - lo;
      if (du > dv || (du == dv && u > v)) {
        larger++;
      } else if (u != v) {
        smaller++;
        while (lo < hi) {  // v in row u (sorted): lower bound
          const uint32_t mid = lo + ((hi - lo) >> 1);
          if (P.col[mid] < v)
            lo = mid + 1;
          else
            hi = mid;
        }
        if (lo == end || P.col[lo] != v || P.val[lo] != x) bad = true;
      }
    }
  }
  if (bad) *P.asym = 1u;
  const u64 a = sygraph::detail::block_sum<u64>(smaller, s_red), b = sygraph::detail::block_sum<u64>(larger, s_red);
  if (threadIdx.x == 0) {
    if (a) atomicAdd(P.towards, a);
    if (b) atomicAdd(P.towards + 1, b);
  }
}

__global__ void __launch_bounds__(256) low_words_kernel(const u64* __restrict__ key, uint64_t m,
                                                        uint32_t* __restrict__ out) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (uint64_t)gridDim.x * blockDim.x)
    out[i] = (uint32_t)key[i];
}

}  // namespace gb

namespace {

uint32_t bit_length(uint32_t x) { return x ? 32u - (uint32_t)__builtin_clz(x) : 1u; }

}  // namespace

// Builds g->wcol / g->wval (rows of the forward CSR sorted by weight) and
// g->wsym once per graph, on the device.
sg_status graph_weight_sorted(sg_graph g) {
  using rsort::u64;
  std::lock_guard<std::mutex> lk(g->wsort_mu);
  if (g->wcol) return SG_OK;
  SG_REQUIRE(g->fwd.val && g->value_type != SG_WEIGHT_NONE, SG_ERR_INVALID, "the graph has no weights");
  const uint32_t n = g->n;
  const uint64_t m = g->m, ma = m ? m : 1;
  cudaStream_t st = g->stream;
  const uint32_t bits = 32 + bit_length(n - 1), passes = (bits + 7) / 8;
  Carve c;
  const uint64_t k0 = c.reserve(8 * ma), k1 = c.reserve(8 * ma), v = c.reserve(4 * ma), words = c.reserve(24),
                 scratch = c.reserve(4 * rsort::scratch_words(m));
  uint32_t *wc = nullptr, *wv = nullptr;
  sg_status s = SG_OK;
  do {
    if ((s = dev_alloc(&c.base, c.bytes)) || (s = dev_alloc(&wc, ma)) || (s = dev_alloc(&wv, ma))) break;
    u64* k[2] = {c.at<u64>(k0), c.at<u64>(k1)};
    uint32_t* vals[2] = {c.at<uint32_t>(v), c.at<uint32_t>(v)};
    vals[passes & 1] = wc;  // the sorted columns stay where the last pass puts them
    struct {
      u64 towards[2];
      uint32_t asym, m;
    } flags = {{0, 0}, 0, (uint32_t)m};
    static_assert(sizeof(flags) == 24, "reserved above");
    char* dev = c.at<char>(words);
    const gb::WsortParams P{g->fwd.ro,  g->fwd.col, reinterpret_cast<const uint32_t*>(g->fwd.val),
                            n,          (uint32_t)m, k[0], vals[0], reinterpret_cast<uint32_t*>(dev + 16),
                            reinterpret_cast<u64*>(dev)};
    cudaError_t e = cudaMemcpyAsync(dev, &flags, sizeof(flags), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess && m) {
      gb::ws_fill_kernel<<<grid_for((m - 1) / 32 + 1, 8, 8), 256, 0, st>>>(P);
      count_launch();
      uint32_t done, *left;
      const rsort::ArraySource src{k[0], vals[0], reinterpret_cast<uint32_t*>(dev + 20)};
      if ((s = rsort::sort_pairs(src, m, bits, k, vals, c.at<uint32_t>(scratch), st, &done, &left)) != SG_OK) break;
      gb::low_words_kernel<<<grid_for(m, 256, 8), 256, 0, st>>>(k[passes & 1], m, wv);
      e = cudaGetLastError();
      count_launch();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(&flags, dev, sizeof(flags), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) {
      s = cuda_fail(e, "weight sort", __FILE__, __LINE__);
      break;
    }
    g->wcol = wc;
    g->wval = wv;
    wc = wv = nullptr;
    g->wsym = flags.asym == 0 && flags.towards[0] == flags.towards[1];
    g->bytes += 8ull * m;
  } while (0);
  dev_free(c.base);
  dev_free(wc);
  dev_free(wv);
  return s;
}

namespace {

// One direction (forward, or with src / dst swapped the inverse) of a build;
// out gets device arrays ro (n+1), col and val (m each) in one allocation.
sg_status build_direction(const uint32_t* dsrc, const uint32_t* ddst, const uint32_t* dval, uint64_t count,
                          uint32_t n, uint32_t one, int symmetrize, int dedupe, int drop_self_loops,
                          cudaStream_t stream, GraphDir* out, uint64_t* m_out) {
  using rsort::u64;
  const uint64_t E = symmetrize ? 2 * count : count, Ea = E ? E : 1;  // below 2^32
  const uint32_t b = bit_length(n - 1);
  const uint32_t tiles = (uint32_t)((Ea - 1) / gb::kKeepTile + 1);
  const uint64_t rows = (uint64_t)n + 1;
  const uint32_t row_tiles = (uint32_t)((rows - 1) / gb::kKeepTile + 1);
  Carve c;
  const uint64_t k0 = c.reserve(8 * Ea), k1 = c.reserve(8 * Ea), v0 = c.reserve(4 * Ea), v1 = c.reserve(4 * Ea),
                 scratch = c.reserve(4 * rsort::scratch_words(E)), tile_kept = c.reserve(4ull * tiles),
                 tile_min = c.reserve(4ull * row_tiles), words = c.reserve(8);
  void* block = nullptr;
  sg_status s = SG_OK;
  do {
    if ((s = dev_alloc(&c.base, c.bytes))) break;
    uint32_t* flags = c.at<uint32_t>(words);  // edges kept, an endpoint was out of range
    cudaError_t e = cudaMemsetAsync(flags, 0, 8, stream);
    if (e != cudaSuccess) {
      s = cuda_fail(e, "memset", __FILE__, __LINE__);
      break;
    }
    const gb::EdgeSource src{dsrc, ddst, dval, (uint32_t)E, n, b, one, symmetrize, drop_self_loops, flags + 1};
    u64* k[2] = {c.at<u64>(k0), c.at<u64>(k1)};
    uint32_t* v[2] = {c.at<uint32_t>(v0), c.at<uint32_t>(v1)};
    uint32_t passes, *left;
    if ((s = rsort::sort_pairs(src, E, 2 * b, k, v, c.at<uint32_t>(scratch), stream, &passes, &left)) != SG_OK) break;
    const u64* key = k[passes & 1];
    uint32_t* kept = c.at<uint32_t>(tile_kept);
    gb::keep_count_kernel<<<tiles, gb::kKeepThreads, 0, stream>>>(key, left, dedupe, kept);
    rsort::scan_kernel<<<1, rsort::kSortThreads, 0, stream>>>(tiles, kept, flags);
    count_launch(2);
    uint32_t hf[2];
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(hf, flags, sizeof(hf), cudaMemcpyDeviceToHost, stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    if (e != cudaSuccess) {
      s = cuda_fail(e, "graph build", __FILE__, __LINE__);
      break;
    }
    if (hf[1]) {
      s = fail(SG_ERR_INVALID, "edge endpoint out of range");
      break;
    }
    const uint64_t m = hf[0], ma = m ? m : 1;
    Carve o;
    const uint64_t ro = o.reserve(4 * rows), col = o.reserve(4 * ma), val = o.reserve(4 * ma), units = o.reserve(4),
                   unit = o.reserve(sizeof(uint2) * hub_units_capacity(m));
    if ((s = dev_alloc(&o.base, o.bytes))) break;
    block = o.base;
    e = cudaMemsetAsync(o.at<uint32_t>(ro), 0xff, 4 * rows, stream);
    gb::keep_write_kernel<<<tiles, gb::kKeepThreads, 0, stream>>>(key, v[passes & 1], left, dedupe, b, kept, flags, n,
                                                                  o.at<uint32_t>(ro), o.at<uint32_t>(col),
                                                                  o.at<uint32_t>(val));
    gb::row_min_kernel<<<row_tiles, gb::kKeepThreads, 0, stream>>>(o.at<uint32_t>(ro), rows, c.at<uint32_t>(tile_min));
    gb::row_carry_kernel<<<1, 1024, 0, stream>>>(c.at<uint32_t>(tile_min), row_tiles);
    gb::row_fill_kernel<<<row_tiles, gb::kKeepThreads, 0, stream>>>(o.at<uint32_t>(ro), rows, c.at<uint32_t>(tile_min));
    count_launch(4);
    GraphDir d{o.at<uint32_t>(ro), o.at<uint32_t>(col), o.at<uint32_t>(val), block, o.at<uint32_t>(units),
               o.at<uint2>(unit)};
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e == cudaSuccess && (s = build_hub_units(d, n, stream)) != SG_OK) break;
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    if (e != cudaSuccess) {
      s = cuda_fail(e, "graph build", __FILE__, __LINE__);
      break;
    }
    *out = d;
    *m_out = m;
    block = nullptr;
  } while (0);
  dev_free(c.base);
  if (block) cudaFree(block);
  return s;
}

}  // namespace
}  // namespace sgb

using namespace sgb;

extern "C" {

sg_status sg_graph_create_coo(const uint32_t* src, const uint32_t* dst, const void* values, int value_type,
                              uint32_t n, uint64_t count, int symmetrize, int dedupe, int drop_self_loops,
                              int device_pointers, void* stream, sg_graph* out) {
  clear_error();
  SG_REQUIRE(out, SG_ERR_INVALID, "out is NULL");
  *out = nullptr;
  SG_REQUIRE(count == 0 || (src && dst), SG_ERR_INVALID, "NULL edge array");
  SG_REQUIRE(n > 0 && n < 0x7fffffffu, SG_ERR_INVALID, "vertex count must be in [1, 2^31)");
  SG_REQUIRE(value_type == SG_WEIGHT_NONE || value_type == SG_WEIGHT_F32 || value_type == SG_WEIGHT_U32,
             SG_ERR_INVALID, "unknown value_type");
  SG_REQUIRE((symmetrize ? 2 * count : count) < (1ull << 32), SG_ERR_INVALID,
             "edge entries (twice the edges when symmetrised) must be below 2^32");
  cudaStream_t st = (cudaStream_t)stream;
  const bool weighted = value_type != SG_WEIGHT_NONE && values;
  // missing weights are ones, as sg_graph_create_csr stores them
  uint32_t one = 1u;
  if (value_type == SG_WEIGHT_F32) {
    const float f = 1.0f;
    memcpy(&one, &f, 4);
  }
  const uint32_t* dsrc = src;
  const uint32_t* ddst = dst;
  const uint32_t* dval = weighted ? (const uint32_t*)values : nullptr;
  uint32_t* own[3] = {nullptr, nullptr, nullptr};
  sg_status s = SG_OK;
  if (!device_pointers && count) {
    if ((s = dev_alloc(&own[0], count)) || (s = dev_alloc(&own[1], count)) ||
        (weighted && (s = dev_alloc(&own[2], count)))) {
      for (auto* p : own) dev_free(p);
      return s;
    }
    cudaError_t e = cudaMemcpyAsync(own[0], src, 4 * count, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(own[1], dst, 4 * count, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess && weighted) e = cudaMemcpyAsync(own[2], values, 4 * count, cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) {
      for (auto* p : own) dev_free(p);
      return cuda_fail(e, "edge upload", __FILE__, __LINE__);
    }
    dsrc = own[0];
    ddst = own[1];
    dval = weighted ? own[2] : nullptr;
  }
  sg_graph g = new sg_graph_s();
  g->n = n;
  g->flags = (symmetrize ? 0u : SG_GRAPH_DIRECTED) | (value_type != SG_WEIGHT_NONE ? SG_GRAPH_WEIGHTED : 0u);
  g->stream = st;
  g->value_type = value_type == SG_WEIGHT_NONE ? SG_WEIGHT_U32 : value_type;
  uint64_t m = 0;
  s = build_direction(dsrc, ddst, dval, count, n, one, symmetrize, dedupe, drop_self_loops, st, &g->fwd, &m);
  if (s == SG_OK) {
    g->m = m;
    g->bytes = sizeof(uint32_t) * ((uint64_t)n + 1 + 2 * m) + sizeof(uint2) * hub_units_capacity(m);
    if (symmetrize) {
      g->inv = g->fwd;
      g->owns_inverse = false;
    } else {
      uint64_t mi = 0;
      s = build_direction(ddst, dsrc, dval, count, n, one, 0, dedupe, drop_self_loops, st, &g->inv, &mi);
      if (s == SG_OK) {
        g->owns_inverse = true;
        g->bytes *= 2;
      }
    }
  }
  for (auto* p : own) dev_free(p);
  if (s != SG_OK) {
    release_graph(g);
    return s;
  }
  *out = g;
  return SG_OK;
}

sg_status sg_graph_weight_sorted(sg_graph g, uint32_t* host_column_indices, void* host_values, int* symmetric) {
  clear_error();
  SG_REQUIRE(g, SG_ERR_INVALID, "graph is NULL");
  SG_TRY(graph_weight_sorted(g));
  if (host_column_indices && g->m)
    SG_CUDA(cudaMemcpyAsync(host_column_indices, g->wcol, sizeof(uint32_t) * g->m, cudaMemcpyDeviceToHost, g->stream));
  if (host_values && g->m)
    SG_CUDA(cudaMemcpyAsync(host_values, g->wval, sizeof(uint32_t) * g->m, cudaMemcpyDeviceToHost, g->stream));
  SG_CUDA(cudaStreamSynchronize(g->stream));
  if (symmetric) *symmetric = g->wsym ? 1 : 0;
  return SG_OK;
}

}  // extern "C"
