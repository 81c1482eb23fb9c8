// Generic advance kernels: advance::frontier<Direction, Lb, InView, OutView>
// (operators/advance/advance.hpp:116-218) for any device functor
// bool f(src, dst, edge, weight).  The C ABI instantiates them with its
// built-in functors; the C++ header API instantiates them with user lambdas.
//
// Semantics kept from operators/advance/common.hpp:49-75:
//   candidates   push: vertices in the input frontier; pull / pull_all: the
//                vertices NOT in it; graph view: every vertex < limit
//   neighbours   push: every out-edge; pull: in-edges (the inverse graph)
//                whose endpoint is in the input frontier
//   insert       push: dst; pull: src (the candidate)
//   short-circuit (pull only): a candidate stops at its first successful edge
//
// Candidate vertices are enumerated through the input frontier's compacted
// word list (offsets[0 .. *offsets_size), written by the compaction kernel);
// the count is read on the device, so no launch needs a host round trip.
#pragma once

#include <cstdint>

#include "primitives.cuh"

namespace sygraph {
namespace detail {

enum AdvDir : int { kPush = 0, kPull = 1, kPullAll = 2 };
enum AdvView : int { kViewGraph = 0, kViewVertex = 1, kViewEdge = 2, kViewNone = 3 };

// Device view of a two-level bitmap frontier (MLBDevice,
// frontier/impls/mlb_frontier.hpp:58-153): level 0 has one bit per element,
// level 1 one bit per level-0 word.
struct MLBDev {
  uint32_t num_elems;
  uint32_t words0;
  uint32_t words1;
  uint32_t* l0;
  uint32_t* l1;
  int32_t* offsets;
  uint32_t* offsets_size;

  __device__ __forceinline__ bool check(uint32_t i) const { return (ld_cg(l0 + (i >> 5)) >> (i & 31)) & 1u; }
  // MLBDevice::insert (mlb:86-97): read first, atomicOr only when the bit is clear.
  __device__ __forceinline__ void insert(uint32_t i) const {
    const uint32_t b0 = 1u << (i & 31);
    uint32_t* w0 = l0 + (i >> 5);
    if (!(ld_cg(w0) & b0)) atomicOr(w0, b0);
    const uint32_t j = i >> 5;
    const uint32_t b1 = 1u << (j & 31);
    uint32_t* w1 = l1 + (j >> 5);
    if (!(ld_cg(w1) & b1)) atomicOr(w1, b1);
  }
  // MLBDevice::remove (mlb:99-103): level 0 only.
  __device__ __forceinline__ void remove(uint32_t i) const { atomicAnd(l0 + (i >> 5), ~(1u << (i & 31))); }
};

template <typename W>
struct GraphDev {
  uint32_t n;
  uint64_t m;
  const uint32_t* ro;
  const uint32_t* col;
  const W* val;
};

struct AdvanceArgs {
  int in_view;
  int out_view;
  uint32_t limit;  // number of vertices
  MLBDev in;
  MLBDev out;
  // The graph direction's long rows (kHubDegree edges or more) cut in units of
  // kHubUnit edges, as (vertex, first edge), or null: then every row is its
  // candidate's CTA's work.
  const uint2* hub_units = nullptr;
  const uint32_t* n_hub_units = nullptr;

  __device__ __forceinline__ uint32_t num_words() const {
    return in_view == kViewVertex ? ld_cg(in.offsets_size) : (limit + 31) / 32;
  }
  __device__ __forceinline__ uint32_t word_at(uint32_t i) const {
    return in_view == kViewVertex ? (uint32_t)ld_cg(in.offsets + i) : i;
  }
  template <int Dir>
  __device__ __forceinline__ bool check(uint32_t v) const {
    if (v >= limit) return false;
    if (in_view == kViewGraph) return true;
    if (in_view != kViewVertex) return false;
    return (Dir == kPush) == in.check(v);
  }
  template <int Dir>
  __device__ __forceinline__ bool valid_neighbor(uint32_t u) const {
    return Dir == kPush ? true : in.check(u);
  }
  template <int Dir>
  __device__ __forceinline__ void insert(uint32_t v, uint32_t u) const {
    if (out_view == kViewVertex) out.insert(Dir == kPush ? u : v);
  }
};

// Rows that a CTA does not walk alone.  On an RMAT graph of 300 K vertices one
// CTA walked a hub's 100 K edges 256 at a time while the others had finished:
// 206 us for that level's advance, 67 with the rows in units.
// Below 512 edges a row is two rounds of its CTA; a unit is four.  The list is
// looked through whatever the frontier holds: an advance of one vertex takes
// 10.3 us with its compaction instead of 9.2 (RMAT-18).
constexpr uint32_t kHubDegree = 512, kHubUnit = 1024;

// The units of the candidates among the long rows, spread over the grid: a
// CTA's 256 threads look at 256 units at once, then the CTA walks the active
// ones.  Not for short-circuit pulls, whose candidates stop at their first
// successful edge.  Every thread of the CTA calls it; s_unit holds 256.
template <int Dir, typename W, typename F>
__device__ __forceinline__ void walk_hub_units(const GraphDev<W>& g, const AdvanceArgs& a, const F& f, uint2* s_unit,
                                               uint32_t* s_count) {
  const uint32_t t = threadIdx.x, units = *a.n_hub_units;
  for (uint32_t i0 = blockIdx.x; i0 < units; i0 += gridDim.x * blockDim.x) {
    if (t == 0) *s_count = 0;
    __syncthreads();
    const uint64_t i = i0 + (uint64_t)t * gridDim.x;
    if (i < units) {
      const uint2 u = a.hub_units[i];
      if (a.template check<Dir>(u.x)) s_unit[atomicAdd(s_count, 1u)] = u;
    }
    __syncthreads();
    for (uint32_t k = 0; k < *s_count; k++) {
      const uint32_t v = s_unit[k].x, b = s_unit[k].y, left = g.ro[v + 1] - b;
      const uint32_t len = left < kHubUnit ? left : kHubUnit;
      uint32_t u[kHubUnit / 256];
#pragma unroll
      for (uint32_t q = 0; q < kHubUnit / 256; q++) u[q] = q * 256 + t < len ? g.col[b + q * 256 + t] : 0u;
#pragma unroll
      for (uint32_t q = 0; q < kHubUnit / 256; q++) {
        const uint32_t e = b + q * 256 + t;
        if (q * 256 + t < len && a.template valid_neighbor<Dir>(u[q]) && f(v, u[q], e, g.val[e]))
          a.template insert<Dir>(v, u[q]);
      }
    }
    __syncthreads();
  }
}

// ---- work-item mapped: one thread per candidate vertex, serial neighbour loop
template <int Dir, typename W, typename F>
__global__ void __launch_bounds__(256) advance_workitem_kernel(GraphDev<W> g, AdvanceArgs a, F f) {
  const uint64_t total = (uint64_t)a.num_words() * 32;
  for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < total; t += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t v = a.word_at((uint32_t)(t >> 5)) * 32 + (uint32_t)(t & 31);
    if (!a.template check<Dir>(v)) continue;
    const uint32_t end = g.ro[v + 1];
    for (uint32_t e = g.ro[v]; e < end; e++) {
      const uint32_t u = g.col[e];
      if (!a.template valid_neighbor<Dir>(u)) continue;
      if (!f(v, u, e, g.val[e])) continue;
      a.template insert<Dir>(v, u);
      if (Dir == kPull) break;
    }
  }
}

// ---- sub-group mapped: a warp walks each candidate of its word in turn,
// 32 neighbours per step (coalesced column loads).
template <int Dir, typename W, typename F>
__global__ void __launch_bounds__(256) advance_subgroup_kernel(GraphDev<W> g, AdvanceArgs a, F f) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t nw = a.num_words();
  const uint32_t gwarp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t wi = gwarp; wi < nw; wi += nwarps) {
    const uint32_t v0 = a.word_at(wi) * 32;
    uint32_t cand = __ballot_sync(kFullMask, a.template check<Dir>(v0 + lane));
    while (cand) {
      const uint32_t v = v0 + __ffs(cand) - 1;
      cand &= cand - 1;
      const uint32_t b = g.ro[v], en = g.ro[v + 1];
      for (uint32_t eb = b; eb < en; eb += 32) {
        const uint32_t e = eb + lane;
        bool ok = false;
        if (e < en) {
          const uint32_t u = g.col[e];
          if (a.template valid_neighbor<Dir>(u) && f(v, u, e, g.val[e])) {
            a.template insert<Dir>(v, u);
            ok = true;
          }
        }
        if (Dir == kPull && __any_sync(kFullMask, ok)) break;
      }
    }
  }
}

// ---- work-group mapped: a 256-thread CTA takes 8 words (256 candidates),
// scans their degrees, and walks the combined edge range; each thread finds
// its source by binary search over the inclusive degree scan (of the
// candidates that have edges) in shared memory.  Long rows go in units.
template <int Dir, typename W, typename F>
__global__ void __launch_bounds__(256) advance_workgroup_kernel(GraphDev<W> g, AdvanceArgs a, F f) {
  constexpr uint32_t kB = 256;
  __shared__ uint32_t s_v[kB], s_beg[kB], s_incl[kB], s_scan[32], s_count;
  __shared__ volatile uint32_t s_done[kB];
  __shared__ uint2 s_unit[Dir == kPull ? 1 : kB];
  const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const uint32_t nw = a.num_words();
  const bool hubs = Dir != kPull && a.hub_units;
  for (uint32_t chunk = blockIdx.x; chunk * (kB / 32) < nw; chunk += gridDim.x) {
    const uint32_t wi = chunk * (kB / 32) + warp;
    uint32_t v = 0xffffffffu;
    bool act = false;
    if (wi < nw) {
      v = a.word_at(wi) * 32 + lane;
      act = a.template check<Dir>(v);
    }
    const uint32_t beg = act ? g.ro[v] : 0u;
    uint32_t deg = act ? g.ro[v + 1] - beg : 0u;
    if (hubs && deg >= kHubDegree) deg = 0;  // walked in units
    uint32_t total, slots;
    const uint32_t excl = block_excl_scan(deg, &total, s_scan);
    const uint32_t mine = block_excl_scan(deg != 0, &slots, s_scan);
    if (deg) {
      s_v[mine] = v;
      s_beg[mine] = beg;
      s_incl[mine] = excl + deg;
      s_done[mine] = 0;
    }
    __syncthreads();
    for (uint32_t r = t; r < total; r += kB) {
      uint32_t lo = 0, hi = slots;
      while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (s_incl[mid] <= r)
          lo = mid + 1;
        else
          hi = mid;
      }
      const uint32_t slot = lo;
      if (Dir == kPull && s_done[slot]) continue;
      const uint32_t before = slot ? s_incl[slot - 1] : 0u;
      const uint32_t e = s_beg[slot] + (r - before);
      const uint32_t src = s_v[slot];
      const uint32_t u = g.col[e];
      if (!a.template valid_neighbor<Dir>(u)) continue;
      if (!f(src, u, e, g.val[e])) continue;
      a.template insert<Dir>(src, u);
      if (Dir == kPull) s_done[slot] = 1;
    }
    __syncthreads();
  }
  if constexpr (Dir != kPull) {
    if (hubs) walk_hub_units<Dir>(g, a, f, s_unit, &s_count);
  }
}

// ---- bucketing: each candidate by degree goes to its lane (< 32), its warp
// (< kHubDegree, or < kCtaDegree without units) or the whole CTA (the rest;
// long rows in units).
template <int Dir, typename W, typename F>
__global__ void __launch_bounds__(256) advance_bucketing_kernel(GraphDev<W> g, AdvanceArgs a, F f) {
  constexpr uint32_t kB = 256, kCtaDegree = 2048;
  __shared__ uint32_t s_big[kB];
  __shared__ uint32_t s_nbig;
  __shared__ uint2 s_unit[Dir == kPull ? 1 : kB];
  const bool hubs = Dir != kPull && a.hub_units;
  __shared__ volatile uint32_t s_claimed;
  const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const uint32_t nw = a.num_words();
  for (uint32_t chunk = blockIdx.x; chunk * (kB / 32) < nw; chunk += gridDim.x) {
    if (t == 0) s_nbig = 0;
    __syncthreads();
    const uint32_t wi = chunk * (kB / 32) + warp;
    uint32_t v = 0;
    bool act = false;
    if (wi < nw) {
      v = a.word_at(wi) * 32 + lane;
      act = a.template check<Dir>(v);
    }
    const uint32_t beg = act ? g.ro[v] : 0u;
    const uint32_t deg = act ? g.ro[v + 1] - beg : 0u;
    const bool unit = act && hubs && deg >= kHubDegree;  // walked in units below
    const bool big = act && !unit && deg >= kCtaDegree;
    const bool mid = act && !unit && !big && deg >= 32;
    const bool small = act && deg < 32;
    if (big) s_big[atomicAdd(&s_nbig, 1u)] = v;
    // warp bucket
    uint32_t mids = __ballot_sync(kFullMask, mid);
    while (mids) {
      const uint32_t j = __ffs(mids) - 1;
      mids &= mids - 1;
      const uint32_t vj = __shfl_sync(kFullMask, v, j);
      const uint32_t bj = __shfl_sync(kFullMask, beg, j);
      const uint32_t ej = bj + __shfl_sync(kFullMask, deg, j);
      for (uint32_t eb = bj; eb < ej; eb += 32) {
        const uint32_t e = eb + lane;
        bool ok = false;
        if (e < ej) {
          const uint32_t u = g.col[e];
          if (a.template valid_neighbor<Dir>(u) && f(vj, u, e, g.val[e])) {
            a.template insert<Dir>(vj, u);
            ok = true;
          }
        }
        if (Dir == kPull && __any_sync(kFullMask, ok)) break;
      }
    }
    // lane bucket: serial, stops at the first success in pull mode
    if (small) {
      for (uint32_t e = beg; e < beg + deg; e++) {
        const uint32_t u = g.col[e];
        if (!a.template valid_neighbor<Dir>(u)) continue;
        if (!f(v, u, e, g.val[e])) continue;
        a.template insert<Dir>(v, u);
        if (Dir == kPull) break;
      }
    }
    __syncthreads();
    // CTA bucket
    const uint32_t nbig = s_nbig;
    for (uint32_t i = 0; i < nbig; i++) {
      const uint32_t vb = s_big[i];
      const uint32_t b = g.ro[vb], en = g.ro[vb + 1];
      if (t == 0) s_claimed = 0;
      __syncthreads();
      for (uint32_t e = b + t; e < en; e += kB) {
        if (Dir == kPull && s_claimed) break;
        const uint32_t u = g.col[e];
        if (!a.template valid_neighbor<Dir>(u)) continue;
        if (!f(vb, u, e, g.val[e])) continue;
        a.template insert<Dir>(vb, u);
        if (Dir == kPull) s_claimed = 1;
      }
      __syncthreads();
    }
  }
  if constexpr (Dir != kPull) {
    __syncthreads();  // s_nbig is read by the last chunk's CTA bucket
    if (hubs) walk_hub_units<Dir>(g, a, f, s_unit, &s_nbig);
  }
}

// Host launcher; lb follows operators/config.hpp (0 workitem, 1 subgroup,
// 2 workgroup, 3 bucketing).  Returns the CUDA launch status.
template <int Dir, typename W, typename F>
inline cudaError_t launch_advance(int lb, const GraphDev<W>& g, const AdvanceArgs& a, const F& f, unsigned grid,
                                  cudaStream_t stream) {
  switch (lb) {
    case 0: advance_workitem_kernel<Dir, W, F><<<grid, 256, 0, stream>>>(g, a, f); break;
    case 1: advance_subgroup_kernel<Dir, W, F><<<grid, 256, 0, stream>>>(g, a, f); break;
    case 2: advance_workgroup_kernel<Dir, W, F><<<grid, 256, 0, stream>>>(g, a, f); break;
    case 3: advance_bucketing_kernel<Dir, W, F><<<grid, 256, 0, stream>>>(g, a, f); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

// ---- frontier-wide helpers used by filter / compute (one thread per
// candidate of the compacted input).
template <typename P>
__global__ void __launch_bounds__(256) filter_external_kernel(MLBDev in, MLBDev out, uint32_t limit, P pred) {
  const uint64_t total = (uint64_t)ld_cg(in.offsets_size) * 32;
  for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < total; t += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t v = (uint32_t)ld_cg(in.offsets + (t >> 5)) * 32 + (uint32_t)(t & 31);
    if (v < limit && in.check(v) && pred(v)) out.insert(v);
  }
}

template <typename P>
__global__ void __launch_bounds__(256) filter_inplace_kernel(MLBDev f, uint32_t limit, P pred) {
  const uint64_t total = (uint64_t)ld_cg(f.offsets_size) * 32;
  for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < total; t += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t v = (uint32_t)ld_cg(f.offsets + (t >> 5)) * 32 + (uint32_t)(t & 31);
    if (v < limit && f.check(v) && pred(v)) f.remove(v);
  }
}

template <typename Fn>
__global__ void __launch_bounds__(256) compute_execute_kernel(MLBDev f, uint32_t limit, Fn fn) {
  const uint64_t total = (uint64_t)ld_cg(f.offsets_size) * 32;
  for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < total; t += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t v = (uint32_t)ld_cg(f.offsets + (t >> 5)) * 32 + (uint32_t)(t & 31);
    if (v < limit && f.check(v)) fn(v);
  }
}

// Sum of fn(v) over the active vertices; one atomic per CTA.
template <typename Fn>
__global__ void __launch_bounds__(256) compute_reduce_kernel(MLBDev f, uint32_t limit, Fn fn,
                                                             unsigned long long* out) {
  __shared__ unsigned long long s_red[32];
  const uint64_t total = (uint64_t)ld_cg(f.offsets_size) * 32;
  unsigned long long acc = 0;
  for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < total; t += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t v = (uint32_t)ld_cg(f.offsets + (t >> 5)) * 32 + (uint32_t)(t & 31);
    if (v < limit && f.check(v)) acc += fn(v);
  }
  acc = block_sum(acc, s_red);
  if (threadIdx.x == 0 && acc) atomicAdd(out, acc);
}

}  // namespace detail
}  // namespace sygraph
