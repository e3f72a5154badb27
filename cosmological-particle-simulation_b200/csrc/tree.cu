// tree.cu — octree build from sorted octant keys (tree.rs:171-250). The walk is in walk.cu.
//
// Build. Particles are sorted by their 63-bit octant key (21 digits of the reference's descent,
// tree.rs:186-250), or by the Hilbert key of the same cubes (the simulation's order), so every
// node of the reference's tree is a contiguous range of the sorted array: the particles whose
// first d digits equal the node's prefix. One kernel per level splits each node of that level
// that holds more than LEAF_SIZE particles: the 8 sub-ranges are found on digit d+1 (sorted
// within the node: a thread per node on wide levels, a warp per node on levels with few nodes),
// and the non-empty ones become children, allocated contiguously in digit order; a child's octant
// (its centre, and the node's octant mask that the walk's children[0] rule reads) is the octant
// digit of its first particle. Node centres are built with the reference's
// f32 arithmetic (centre +- half/2), so they are bit-identical. A node deeper than the 21 key
// digits that still holds more than LEAF_SIZE particles stays a leaf (the reference would keep
// splitting to depth 40); such nodes are counted.
//
// Centres of mass are FP64 sums of the sorted positions over a node's range, divided by the count
// and rounded once to f32. (The reference sums in f32 sequentially in input order; the difference is
// f32 round-off of that sum.)
#include <cooperative_groups.h>

#include <algorithm>
#include <vector>

#include "cpm_internal.cuh"

namespace cpm {

constexpr int BUILD_THREADS = 256;
constexpr int BUILD_BLOCKS = 148 * 4;
constexpr int TOP_LEVEL = 3;             // the levels down to it are made in one launch
constexpr size_t CLUSTER_TAIL = 262144;  // particles up to which the deep levels start early in one cluster

// counters layout (u32): [0..KEY_LEVELS+1] per-level node counts (level 0 = root),
// [32] nodes that hit the key-depth limit with > LEAF_SIZE particles, [33] max depth, [34] the level that
// k_tree_cluster left to k_tree_com (0: none), [40..41] the phases of those.
constexpr int CNT_DEPTH_LIMIT = 32;
constexpr int CNT_MAX_DEPTH = 33;
constexpr int CNT_WIDE = 34;
constexpr int CNT_PHASES = 40;
constexpr int CNT_WORDS = 64;

__device__ __forceinline__ uint32_t digit_at(uint64_t key, int shift) { return (uint32_t)(key >> shift) & 7u; }

// The seven boundaries of a range [s, e) of more than 32 keys whose digits at `shift` do not decrease:
// lane 4 o (o = 1..7) returns the first index whose digit is >= o (e if none). One round of 32 evenly
// spaced probes narrows all of them to a 32nd of the range, then each group of four lanes narrows its own
// to a fifth per round: a range of 32,768 keys takes 6 dependent loads instead of 21.
__device__ __forceinline__ uint32_t warp_boundaries(const uint64_t* __restrict__ keys, uint32_t s, uint32_t e,
                                                    int shift, int lane) {
  const unsigned FULL = 0xffffffffu;
  const uint32_t o = (uint32_t)lane >> 2, c = e - s;
  const uint32_t mine = digit_at(__ldg(keys + s + (uint32_t)(((uint64_t)c * (uint32_t)lane) >> 5)), shift);
  uint32_t below = 0;  // probes with a digit below o: the boundary lies after the last of them
#pragma unroll
  for (uint32_t q = 1; q < 8; ++q) {
    const uint32_t m = __ballot_sync(FULL, mine < q);
    if (o == q) below = (uint32_t)__popc(m);
  }
  uint32_t lo = s, hi = s;
  if (o != 0u && below != 0u) {
    lo = s + (uint32_t)(((uint64_t)c * (below - 1u)) >> 5) + 1u;
    hi = below < 32u ? s + (uint32_t)(((uint64_t)c * below) >> 5) : e;
  }
  while (__any_sync(FULL, lo < hi)) {
    const uint32_t len = hi - lo, j = (uint32_t)lane & 3u;
    const uint32_t p = lo + (uint32_t)(((uint64_t)len * (j + 1u)) / 5u);  // p < hi
    const bool lt = lo < hi && digit_at(__ldg(keys + p), shift) < o;
    const uint32_t k = (uint32_t)__popc((__ballot_sync(FULL, lt) >> (lane & ~3)) & 15u);  // probes below
    const uint32_t nlo = k ? lo + (uint32_t)(((uint64_t)len * k) / 5u) + 1u : lo;
    const uint32_t nhi = k < 4u ? lo + (uint32_t)(((uint64_t)len * (k + 1u)) / 5u) : hi;
    if (lo < hi) {
      lo = nlo;
      hi = nhi;
    }
  }
  return lo;
}

// The root of every box (one box, or a batch of `roots` boxes of n_box particles each, sorted box by
// box): node b covers the particles of box b, the cube [0, L]^3 of its own box. One CTA.
__device__ __forceinline__ void make_roots(uint4* link, float4* geo, uint32_t* counters, uint32_t n, float half0,
                                           uint32_t roots, uint32_t n_box) {
  for (uint32_t b = threadIdx.x; b < roots; b += blockDim.x) {
    const uint32_t s0 = roots > 1 ? b * n_box : 0u, e0 = roots > 1 ? min(n, (b + 1) * n_box) : n;
    __stcg(link + b, make_uint4(s0, e0, 0u, 0u));
    __stcg(geo + b, make_float4(half0, half0, half0, half0));
  }
  if (threadIdx.x < CNT_WORDS) __stcg(counters + threadIdx.x, threadIdx.x == 0 ? roots : 0u);
}

// Splits the nodes of level d. A level with more nodes than the grid has warps takes one node
// per thread: the 8 octant sub-ranges by counting the digits d+1 of a small node's keys, larger
// nodes by the warp. A smaller level (the top levels, and the sparse deep levels of clustered
// states) takes one node per warp.
constexpr uint32_t SMALL_NODE = 256;
constexpr uint32_t SCAN_NODE = 32;  // thread path: nodes up to this size count their digits

// The octant of a position against a node's centre (tree.rs:186-190), the digit that the descent
// gives it there.
__device__ __forceinline__ uint32_t octant_of(const float4& x, const float4& G) {
  return (uint32_t)(x.x >= G.x) | ((uint32_t)(x.y >= G.y) << 1) | ((uint32_t)(x.z >= G.z) << 2);
}

// The boundaries of a node's eight sub-ranges, by a warp: lane o (1..7) returns the first index whose
// digit is >= o. Nodes of up to SMALL_NODE particles count the digits of all their keys (coalesced
// loads, a ballot per octant).
__device__ __forceinline__ uint32_t node_boundaries(const uint64_t* __restrict__ keys, uint32_t s, uint32_t e, int shift,
                                                    int lane) {
  const unsigned FULL = 0xffffffffu;
  if (e - s > SMALL_NODE) {
    const uint32_t bo = warp_boundaries(keys, s, e, shift, lane);
    return __shfl_sync(FULL, bo, (lane & 7) * 4);
  }
  uint32_t below = 0;  // lane o: keys with digit < o
  for (uint32_t i0 = s; i0 < e; i0 += 32) {
    const uint32_t i = i0 + (uint32_t)lane;
    const uint32_t dg = i < e ? digit_at(__ldg(keys + i), shift) : 8u;
#pragma unroll
    for (uint32_t o = 1; o < 8; ++o) {
      const uint32_t bal = __ballot_sync(FULL, dg < o);
      if ((uint32_t)lane == o) below += (uint32_t)__popc(bal);
    }
  }
  return s + below;
}

// After a capacity failure: the counted nodes from `first` on that are still in the arrays become empty
// leaves (the next levels read every counted node).
__device__ __forceinline__ void clear_nodes(uint4* link, float4* geo, uint32_t first, uint32_t capacity) {
  for (uint32_t q = first; q < min(first + 8u, capacity); ++q) {
    __stcg(link + q, make_uint4(0u, 0u, 0u, 0u));
    __stcg(geo + q, make_float4(0.0f, 0.0f, 0.0f, 0.0f));
  }
}

// Room for the children of a CTA's nodes, `want` by this warp: one atomic per CTA and round on the
// level's counter (one per warp, or per node on levels of a node per warp, come to 4,000 and more on one
// address: 20 us a level at 91,125 clustered particles). Returns the warp's first.
__device__ __forceinline__ uint32_t claim_nodes(uint32_t want, uint32_t* counter) {
  __shared__ uint32_t part[32];
  const unsigned FULL = 0xffffffffu;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  if (lane == 0) part[warp] = want;
  __syncthreads();
  if (warp == 0) {
    const uint32_t v = lane < warps ? part[lane] : 0u;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(FULL, incl, o);
      if (lane >= (uint32_t)o) incl += y;
    }
    uint32_t base = 0;
    if (lane == 31 && incl > 0u) base = atomicAdd(counter, incl);
    base = __shfl_sync(FULL, base, 31);
    if (lane < warps) part[lane] = base + incl - v;
  }
  __syncthreads();
  return part[warp];
}

// keys: the sort keys (octant or Hilbert digits split the node); a child's octant is that of its
// first particle.
// lb, cnt: the level's first node and its size. The level is shared by nblocks CTAs, of which this is
// number `block`; nodes are written and read past L1, since one launch may build several levels.
__device__ __forceinline__ void split_level(int d, int levels, uint32_t lb, uint32_t cnt,
                                            const uint64_t* __restrict__ keys, const float4* __restrict__ x4,
                                            uint4* link, float4* geo, uint32_t* counters, uint32_t capacity,
                                            DevStatus* st, uint32_t block, uint32_t nblocks) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const uint32_t next_base = lb + cnt;
  // After a capacity failure the counters overshoot; never touch nodes past the arrays.
  const uint32_t level_end = min(next_base, capacity);
  const int shift = 3 * (levels - 1 - d);
  const uint32_t warps = blockDim.x >> 5, warp = threadIdx.x >> 5;
  bool any_split = false;
  if (cnt > nblocks * warps) {
    // Thread per node. A warp's nodes are a stride apart: large nodes lie next to one another, and a
    // warp takes its large ones in turn.
    const uint32_t stride = nblocks * warps;
    for (uint32_t base = lb + block * warps + warp; base - (block * warps + warp) < level_end; base += 32u * stride) {
      const uint32_t node = base + (uint32_t)lane * stride;
      const bool valid = node < level_end;
      const uint4 L = valid ? __ldcg(link + node) : make_uint4(0u, 0u, 0u, 0u);
      const uint32_t s = L.x, e = L.y, c = e - s;
      bool split = false;
      if (valid) {
        if (c <= (uint32_t)LEAF_SIZE || d >= MAX_DEPTH) {
          __stcg(link + node, make_uint4(s, e, 0u, (uint32_t)d << 8));
        } else if (d >= levels) {
          atomicAdd(&counters[CNT_DEPTH_LIMIT], 1u);
          __stcg(link + node, make_uint4(s, e, 0u, (uint32_t)d << 8));
        } else {
          split = true;
        }
      }
      uint32_t b[9];
      b[0] = s;
      b[8] = e;
      uint32_t mask = 0;
      if (split) {
        if (c <= SCAN_NODE) {
          // Small node: read its keys in order and count each digit (eight 8-bit counters in
          // one word); a few sectors instead of the scattered probes of a search.
          unsigned long long counts = 0ull;
#pragma unroll 4
          for (uint32_t i = s; i < e; ++i) counts += 1ull << (8u * digit_at(__ldg(keys + i), shift));
#pragma unroll
          for (int o = 1; o < 8; ++o) b[o] = b[o - 1] + (uint32_t)((counts >> (8 * (o - 1))) & 0xFFull);
        }
      }
      // The warp's larger nodes, one after another by the whole warp (a thread's own binary searches
      // are 50 and more dependent loads).
      for (uint32_t big = __ballot_sync(FULL, split && c > SCAN_NODE); big; big &= big - 1) {
        const int owner = __ffs(big) - 1;
        const uint32_t bo = node_boundaries(keys, __shfl_sync(FULL, s, owner), __shfl_sync(FULL, e, owner), shift, lane);
#pragma unroll
        for (int o = 1; o < 8; ++o) {
          const uint32_t v = __shfl_sync(FULL, bo, o);
          if (lane == owner) b[o] = v;
        }
      }
      if (split) {
#pragma unroll
        for (int o = 0; o < 8; ++o)
          if (b[o + 1] > b[o]) mask |= 1u << o;
      }
      // octant of each non-empty sub-range (its first particle's octant digit)
      uint32_t octmask = 0, octs = 0;
      float4 G = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (split) {
        G = __ldcg(geo + node);
#pragma unroll
        for (int o = 0; o < 8; ++o)
          if (mask & (1u << o)) {
            const uint32_t oc = octant_of(__ldg(x4 + b[o]), G);
            octmask |= 1u << oc;
            octs |= oc << (3 * o);
          }
      }
      // Children of the warp's nodes: an inclusive scan of their counts.
      const uint32_t nch = (uint32_t)__popc(mask);
      uint32_t incl = nch;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(FULL, incl, o);
        if (lane >= o) incl += y;
      }
      const uint32_t wbase = claim_nodes(__shfl_sync(FULL, incl, 31), &counters[d + 1]);
      any_split |= split;
      if (!split) continue;
      const uint32_t first = next_base + wbase + incl - nch;
      if (first + nch > capacity) {
        dev_fail(st, DEV_NODE_CAPACITY, (int)(first + nch));
        __stcg(link + node, make_uint4(s, e, 0u, (uint32_t)d << 8));
        clear_nodes(link, geo, first, capacity);
        continue;
      }
      const float q = G.w * 0.5f;  // half / 2.0
      uint32_t r = 0;
#pragma unroll
      for (int o = 0; o < 8; ++o) {
        if (!(mask & (1u << o))) continue;
        const uint32_t child = first + r++;
        const uint32_t oc = (octs >> (3 * o)) & 7u;
        __stcg(link + child, make_uint4(b[o], b[o + 1], 0u, 0u));
        __stcg(geo + child, make_float4(__fadd_rn(G.x, (oc & 1) ? q : -q), __fadd_rn(G.y, (oc & 2) ? q : -q),
                                 __fadd_rn(G.z, (oc & 4) ? q : -q), q));
      }
      __stcg(link + node, make_uint4(s, e, first, octmask | ((uint32_t)d << 8)));
    }
  } else {
    // Warp per node.
    for (uint32_t base = lb + block * warps; base < level_end; base += nblocks * warps) {
      const uint32_t node = base + warp;
      const uint4 L = node < level_end ? __ldcg(link + node) : make_uint4(0u, 0u, 0u, 0u);
      const uint32_t s = L.x, e = L.y, c = e - s;
      const bool split = c > (uint32_t)LEAF_SIZE && d < MAX_DEPTH && d < levels;
      if (lane == 0 && node < level_end && !split) {
        if (c > (uint32_t)LEAF_SIZE && d < MAX_DEPTH) atomicAdd(&counters[CNT_DEPTH_LIMIT], 1u);
        __stcg(link + node, make_uint4(s, e, 0u, (uint32_t)d << 8));
      }
      // Lane o < 8: octant o's range [olo, ohi) (lane o >= 1: first index whose digit is >= o).
      uint32_t olo = 0, ohi = 0;
      if (split) {
        const uint32_t bo = node_boundaries(keys, s, e, shift, lane);
        const uint32_t nb = __shfl_sync(FULL, bo, (lane + 1) & 31);
        olo = lane == 0 ? s : bo;
        ohi = lane == 7 ? e : nb;
      }
      const uint32_t mask = __ballot_sync(FULL, lane < 8 && ohi > olo);
      const uint32_t nch = (uint32_t)__popc(mask);
      const uint32_t first = next_base + claim_nodes(nch, &counters[d + 1]);
      any_split |= split;
      if (!split) continue;
      if (first + nch > capacity) {
        if (lane == 0) {
          dev_fail(st, DEV_NODE_CAPACITY, (int)(first + nch));
          __stcg(link + node, make_uint4(s, e, 0u, (uint32_t)d << 8));
          clear_nodes(link, geo, first, capacity);
        }
        continue;
      }
      // lane o: the octant of sub-range o (its first particle's octant digit)
      const bool live = lane < 8 && ((mask >> lane) & 1u);
      const float4 G = __ldcg(geo + node);
      const uint32_t oc = live ? octant_of(__ldg(x4 + olo), G) : 0u;
      const uint32_t octmask = __reduce_or_sync(FULL, live ? 1u << oc : 0u);
      if (live) {
        const float q = G.w * 0.5f;  // half / 2.0
        const uint32_t child = first + (uint32_t)__popc(mask & ((1u << lane) - 1u));
        __stcg(link + child, make_uint4(olo, ohi, 0u, 0u));
        __stcg(geo + child, make_float4(__fadd_rn(G.x, (oc & 1) ? q : -q), __fadd_rn(G.y, (oc & 2) ? q : -q),
                                        __fadd_rn(G.z, (oc & 4) ? q : -q), q));
      }
      if (lane == 0) __stcg(link + node, make_uint4(s, e, first, octmask | ((uint32_t)d << 8)));
    }
  }
  if (__syncthreads_or(any_split) && threadIdx.x == 0) atomicMax(&counters[CNT_MAX_DEPTH], (uint32_t)(d + 1));
}

__global__ void __launch_bounds__(BUILD_THREADS) k_tree_level(int d, int levels, const uint64_t* __restrict__ keys,
                                                              const float4* __restrict__ x4, uint4* link,
                                                              float4* geo, uint32_t* counters, uint32_t capacity,
                                                              DevStatus* st) {
  uint32_t lb = 0;
  for (int j = 0; j < d; ++j) lb += counters[j];
  split_level(d, levels, lb, counters[d], keys, x4, link, geo, counters, capacity, st, blockIdx.x, gridDim.x);
}

// ---------------------------------------------------------------------------------------------
// Centres of mass: FP64 sums of the sorted positions over each node's range. A node of up to
// SUM_DIRECT particles adds them itself; a larger one takes the difference of prefix sums, kept per
// CHUNK of particles (the partial chunk at either end is added by the node), chunk prefixes within
// tiles of CHUNKS_PER_TILE and tile prefixes apart. A prefix sum per particle instead (24 bytes each)
// cost 0.49 ms of FP64 stores and reads at 256^3 particles.
// ---------------------------------------------------------------------------------------------
constexpr uint32_t SUM_DIRECT = 32;
constexpr uint32_t CHUNK = 32;
constexpr uint32_t CHUNKS_PER_TILE = 32;
constexpr uint32_t SUM_TILE = CHUNK * CHUNKS_PER_TILE;

struct D3 {
  double x, y, z;
};
__device__ __forceinline__ D3 d3add(D3 a, D3 b) { return D3{a.x + b.x, a.y + b.y, a.z + b.z}; }

__device__ __forceinline__ D3 shfl_up_d3(D3 v, int o) {
  return D3{__shfl_up_sync(0xffffffffu, v.x, o), __shfl_up_sync(0xffffffffu, v.y, o),
            __shfl_up_sync(0xffffffffu, v.z, o)};
}

// Sum of the positions a .. b - 1.
__device__ __forceinline__ D3 sum_range(const float4* __restrict__ x4, uint32_t a, uint32_t b) {
  D3 s{0.0, 0.0, 0.0};
#pragma unroll 4
  for (uint32_t i = a; i < b; ++i) {
    const float4 x = __ldg(x4 + i);
    s = d3add(s, D3{(double)x.x, (double)x.y, (double)x.z});
  }
  return s;
}

// Inclusive scan over the warp.
__device__ __forceinline__ D3 warp_scan_d3(D3 x, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const D3 y = shfl_up_d3(x, o);
    if (lane >= o) x = d3add(x, y);
  }
  return x;
}

// One warp per tile: lane c sums chunk c, then the exclusive scan over the tile's chunks and the
// tile's total.
__device__ __forceinline__ void sum_tile(const float4* __restrict__ x4, uint32_t n, uint32_t tile, D3* chunk,
                                         D3* totals) {
  const int lane = threadIdx.x & 31;
  const uint32_t i0 = min(n, tile * SUM_TILE + (uint32_t)lane * CHUNK), i1 = min(n, i0 + CHUNK);
  const D3 s = sum_range(x4, i0, i1);
  const D3 incl = warp_scan_d3(s, lane);
  chunk[(size_t)tile * CHUNKS_PER_TILE + lane] = D3{incl.x - s.x, incl.y - s.y, incl.z - s.z};
  if (lane == 31) totals[tile] = incl;
}

__global__ void __launch_bounds__(BUILD_THREADS) k_sum_tiles(const float4* __restrict__ x4, uint32_t n, D3* chunk,
                                                             D3* totals, uint32_t tiles) {
  for (uint32_t t = blockIdx.x * (BUILD_THREADS / 32) + (threadIdx.x >> 5); t < tiles;
       t += gridDim.x * (BUILD_THREADS / 32))
    sum_tile(x4, n, t, chunk, totals);
}

// Exclusive scan of the tile totals in place, one CTA of up to 1024 threads, four tiles per thread and
// round.
__device__ __forceinline__ void scan_tiles(D3* totals, uint32_t tiles, D3* ws) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  D3 carry{0.0, 0.0, 0.0};
  for (uint32_t c0 = 0; c0 < tiles; c0 += 4 * blockDim.x) {
    const uint32_t i = c0 + 4 * threadIdx.x;
    D3 v[4], sum{0.0, 0.0, 0.0};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      v[q] = i + q < tiles ? totals[i + q] : D3{0.0, 0.0, 0.0};
      sum = d3add(sum, v[q]);
    }
    const D3 x = warp_scan_d3(sum, lane);
    if (lane == 31) ws[warp] = x;
    __syncthreads();
    if (warp == 0) {
      const D3 w = warp_scan_d3(lane < warps ? ws[lane] : D3{0.0, 0.0, 0.0}, lane);
      if (lane < warps) ws[lane] = w;
    }
    __syncthreads();
    D3 run = d3add(carry, D3{x.x - sum.x, x.y - sum.y, x.z - sum.z});
    if (warp) run = d3add(run, ws[warp - 1]);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (i + q < tiles) totals[i + q] = run;
      run = d3add(run, v[q]);
    }
    carry = d3add(carry, ws[warps - 1]);
    __syncthreads();
  }
}

// The prefix sum of the whole chunks before particle i.
__device__ __forceinline__ D3 chunk_prefix(const D3* chunk, const D3* totals, uint32_t c) {
  return d3add(totals[c / CHUNKS_PER_TILE], chunk[c]);
}

// Centre of mass of one node, and NODE_FLAT for an inner node whose children all have no octant-0
// child (bit 0 of the mask, which the flag's store leaves as it is for the parents that read it).
__device__ __forceinline__ void finish_node(uint32_t node, uint4* link, const float4* __restrict__ x4, const D3* chunk,
                                            const D3* totals, float4* mass, uint32_t dense_depth, uint32_t n_box,
                                            uint32_t* words) {
  const uint4 L = __ldcg(link + node);
  D3 s;
  if (L.y - L.x <= SUM_DIRECT) {
    s = sum_range(x4, L.x, L.y);
  } else {
    const uint32_t c0 = (L.x + CHUNK - 1) / CHUNK, c1 = L.y / CHUNK;  // whole chunks c0 .. c1 - 1
    const D3 p0 = chunk_prefix(chunk, totals, c0), p1 = chunk_prefix(chunk, totals, c1);
    s = d3add(D3{p1.x - p0.x, p1.y - p0.y, p1.z - p0.z},
              d3add(sum_range(x4, L.x, c0 * CHUNK), sum_range(x4, c1 * CHUNK, L.y)));
  }
  const double c = (double)(L.y - L.x);
  mass[node] = make_float4((float)(s.x / c), (float)(s.y / c), (float)(s.z / c), (float)(L.y - L.x));
  if ((L.w & 0xFFu) != 0u && ((L.w >> 8) & 0x7Fu) >= dense_depth) words[WALK_DENSE + (n_box ? L.x / n_box : 0u)] = 1u;
  if (L.w & 1u) {
    const uint32_t nch = (uint32_t)__popc(L.w & 0xFFu);
    uint32_t any = 0;
    for (uint32_t q = 0; q < nch; ++q) any |= __ldcg(&link[L.z + q].w);
    if ((any & 1u) == 0u) __stcg(&link[node].w, L.w | NODE_FLAT);
  }
}

// The centres of mass of all nodes, after the levels from counters[CNT_WIDE] on that k_tree_cluster found too wide
// for itself, each a phase over all CTAs.
__global__ void __launch_bounds__(BUILD_THREADS, 5) k_tree_com(int levels, const uint64_t* __restrict__ keys, uint4* link,
                                                            float4* geo, const float4* __restrict__ x4,
                                                            const D3* chunk, const D3* totals, float4* mass,
                                                            uint32_t* counters, uint32_t capacity,
                                                            uint32_t dense_depth, uint32_t n_box, uint32_t* words,
                                                            DevStatus* st) {
  if (const int wide = (int)counters[CNT_WIDE]) {
    Phases phases(counters + CNT_PHASES);
    uint32_t lb = 0, cnt = __ldcg(counters + wide);
    for (int d = 0; d < wide; ++d) lb += __ldcg(counters + d);
    for (int d = wide; d <= levels && cnt; ++d) {
      const uint32_t blocks = min(gridDim.x, (cnt + BUILD_THREADS / 32 - 1) / (BUILD_THREADS / 32));
      uint32_t item;
      while (phases.take(blocks, item)) {
        split_level(d, levels, lb, cnt, keys, x4, link, geo, counters, capacity, st, item, blocks);
        phases.done();
      }
      if (!phases.next(blocks)) {
        if (threadIdx.x == 0) dev_fail(st, DEV_WAIT_LIMIT, d);
        return;
      }
      lb += cnt;
      cnt = __ldcg(counters + d + 1);
    }
  }
  uint32_t total = 0;
  for (int j = 0; j <= KEY_LEVELS; ++j) total += counters[j];
  total = min(total, capacity);
  for (uint32_t node = blockIdx.x * blockDim.x + threadIdx.x; node < total; node += gridDim.x * blockDim.x)
    finish_node(node, link, x4, chunk, totals, mass, dense_depth, n_box, words);
}

// The top of a single box's tree: CTA 0 finds where each of the 8^TOP_LEVEL cells of level TOP_LEVEL
// starts in the sorted keys (all searches at once), from which the nodes of the levels above follow
// without another look at the keys, and makes them down to level TOP_LEVEL. The other CTAs form the
// prefix sums' tiles meanwhile. As a level per launch, or per barrier of one cluster, the same
// levels are a chain of searches: 60 us at 32,768 particles. (One level more, 4096 cells, is 44 us: its
// probes are more than one SM fetches quickly.)
constexpr int TOP_CELLS = 1 << (3 * TOP_LEVEL);
constexpr int TOP_THREADS = 512;
constexpr int TOP_PARENTS = TOP_CELLS / 8;  // nodes of the last level that is split here
__global__ void __launch_bounds__(TOP_THREADS) k_tree_top(int levels, const uint64_t* __restrict__ keys,
                                                          const float4* __restrict__ x4, uint32_t n, float half0,
                                                          uint4* link, float4* geo, uint32_t* counters,
                                                          uint32_t capacity, D3* chunk, D3* totals, uint32_t tiles,
                                                          DevStatus* st) {
  if (blockIdx.x > 0) {
    for (uint32_t t = (blockIdx.x - 1) * (TOP_THREADS / 32) + (threadIdx.x >> 5); t < tiles;
         t += (gridDim.x - 1) * (TOP_THREADS / 32))
      sum_tile(x4, n, t, chunk, totals);
    return;
  }
  __shared__ uint32_t start[TOP_CELLS + 1];
  __shared__ uint16_t prefix[2][TOP_PARENTS];  // of the level's nodes
  __shared__ float4 centre[2][TOP_PARENTS];
  __shared__ uint32_t ws[TOP_THREADS / 32];
  static_assert(TOP_PARENTS <= TOP_THREADS && TOP_PARENTS <= 65536, "a thread per node");
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  {
    // The first key of cell q or after: seven probes a round, a thread's cells side by side.
    constexpr int PER = TOP_CELLS / TOP_THREADS;
    const int shift = 3 * (levels - TOP_LEVEL);
    uint32_t lo[PER], hi[PER];
#pragma unroll
    for (int c = 0; c < PER; ++c) {
      lo[c] = 0;
      hi[c] = n;
    }
    for (uint32_t left = n; left > 0; left >>= 3) {  // a round leaves an eighth of the range
#pragma unroll
      for (int c = 0; c < PER; ++c) {
        const uint32_t len = hi[c] - lo[c], q = (uint32_t)(t + c * TOP_THREADS);
        uint32_t k = 0;
        if (len) {
#pragma unroll
          for (uint32_t j = 1; j < 8; ++j)
            k += (uint32_t)((__ldg(keys + lo[c] + (uint32_t)(((uint64_t)len * j) >> 3)) >> shift) < (uint64_t)q);
        }
        const uint32_t nlo = k ? lo[c] + (uint32_t)(((uint64_t)len * k) >> 3) + 1u : lo[c];
        if (k < 7u) hi[c] = lo[c] + (uint32_t)(((uint64_t)len * (k + 1u)) >> 3);
        lo[c] = nlo;
      }
    }
#pragma unroll
    for (int c = 0; c < PER; ++c) start[t + c * TOP_THREADS] = lo[c];
    if (t == 0) start[TOP_CELLS] = n;
  }
  if (t < CNT_WORDS) __stcg(counters + t, t == 0 ? 1u : 0u);
  if (t == 0) {
    prefix[0][0] = 0;
    centre[0][0] = make_float4(half0, half0, half0, half0);
    geo[0] = centre[0][0];
    link[0] = make_uint4(0u, n, 0u, 0u);
  }
  __syncthreads();
  uint32_t lb = 0, cnt = 1;
  for (int d = 0; d < TOP_LEVEL && cnt; ++d) {
    const int cur = d & 1, below = 3 * (TOP_LEVEL - 1 - d);  // a child's cells: 2^below
    uint32_t b[9], mask = 0;
    bool split = false;
    const uint32_t node = lb + (uint32_t)t;
    uint32_t p = 0;
    float4 G = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if ((uint32_t)t < cnt) {
      p = prefix[cur][t];
      G = centre[cur][t];
#pragma unroll
      for (int o = 0; o < 9; ++o) b[o] = start[((p << 3) + o) << below];
      split = b[8] - b[0] > (uint32_t)LEAF_SIZE;
      if (split) {
#pragma unroll
        for (int o = 0; o < 8; ++o)
          if (b[o + 1] > b[o]) mask |= 1u << o;
      }
    }
    const uint32_t nch = (uint32_t)__popc(mask);
    uint32_t incl = nch;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) ws[warp] = incl;
    __syncthreads();
    uint32_t before = 0, total = 0;
    for (int w = 0; w < TOP_THREADS / 32; ++w) {
      before += w < warp ? ws[w] : 0u;
      total += ws[w];
    }
    const uint32_t base = lb + cnt, slot = before + incl - nch, first = base + slot;
    if ((uint32_t)t < cnt) {
      uint32_t octmask = 0, r = 0;
      if (split && first + nch > capacity) {
        dev_fail(st, DEV_NODE_CAPACITY, (int)(first + nch));
        clear_nodes(link, geo, first, capacity);
        split = false;
      }
      if (split) {
        const float q = G.w * 0.5f;  // half / 2.0
#pragma unroll
        for (int o = 0; o < 8; ++o) {
          if (!(mask & (1u << o))) continue;
          const uint32_t oc = octant_of(__ldg(x4 + b[o]), G);
          const float4 C = make_float4(__fadd_rn(G.x, (oc & 1) ? q : -q), __fadd_rn(G.y, (oc & 2) ? q : -q),
                                       __fadd_rn(G.z, (oc & 4) ? q : -q), q);
          octmask |= 1u << oc;
          link[first + r] = make_uint4(b[o], b[o + 1], 0u, 0u);
          geo[first + r] = C;
          if (d + 1 < TOP_LEVEL) {
            prefix[cur ^ 1][slot + r] = (uint16_t)((p << 3) + o);
            centre[cur ^ 1][slot + r] = C;
          }
          ++r;
        }
        link[node] = make_uint4(b[0], b[8], first, octmask | ((uint32_t)d << 8));
      } else {
        link[node] = make_uint4(b[0], b[8], 0u, (uint32_t)d << 8);
      }
    }
    if (t == 0 && total) {
      counters[d + 1] = total;
      counters[CNT_MAX_DEPTH] = (uint32_t)(d + 1);
    }
    __syncthreads();
    lb += cnt;
    cnt = lb + total <= capacity ? total : 0u;
  }
}

// Levels first .. last of the build by one cluster of CTAs in one launch, a level per cluster barrier,
// ending at the deepest level there is: the top levels of a batch, and the levels below every node of a
// smooth distribution, of which a clustered one has some and a smooth one none (as launches of their
// own they are 2 to 4 us each). A level of more than WIDE_LEVEL nodes ends it and is left to k_tree_com with all
// below: 65,536 particles in 100 haloes take 0.142 ms with levels of up to 16,384 nodes here and 0.171 with up
// to 8192, larger levels want the chip (4e6 particles in haloes of 1500 0.48 ms, all levels here 2.2).
// first = 0 makes the roots (and no level is too wide); with `totals` one CTA scans the tile totals.
constexpr uint32_t WIDE_LEVEL = 16384;
constexpr int CLUSTER_CTAS = 8;
constexpr int CLUSTER_THREADS = 1024;
__global__ void __cluster_dims__(CLUSTER_CTAS, 1, 1) __launch_bounds__(CLUSTER_THREADS)
    k_tree_cluster(int first, int last, int levels, const uint64_t* __restrict__ keys, const float4* __restrict__ x4,
                   uint32_t n, float half0, uint32_t roots, uint32_t n_box, uint4* link, float4* geo,
                   uint32_t* counters, uint32_t capacity, D3* totals, uint32_t tiles, DevStatus* st) {
  __shared__ D3 ws[32];
  const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const uint32_t block = blockIdx.x;
  if (first == 0) {
    if (block == 0) make_roots(link, geo, counters, n, half0, roots, n_box);
    cluster.sync();
  }
  if (totals && block == CLUSTER_CTAS - 1) scan_tiles(totals, tiles, ws);
  uint32_t lb = 0;
  for (int d = 0; d < first; ++d) lb += __ldcg(counters + d);
  for (int d = first; d <= last; ++d) {
    const uint32_t cnt = __ldcg(counters + d);
    if (cnt == 0) break;
    if (first > 0 && cnt > WIDE_LEVEL) {
      if (block == 0 && threadIdx.x == 0) counters[CNT_WIDE] = (uint32_t)d;
      break;
    }
    split_level(d, levels, lb, cnt, keys, x4, link, geo, counters, capacity, st, block, CLUSTER_CTAS);
    lb += cnt;
    cluster.sync();
  }
}

// Packs AoS positions into float4 (x, y, z, 0); words[WALK_OUTSIDE] becomes 1 when a position lies
// outside [0, L] (zeroed by the caller).
__global__ void k_pack4(const float* __restrict__ x3, size_t n, float box, float4* __restrict__ x4,
                        uint32_t* __restrict__ words) {
  bool out = false;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const float a = x3[3 * i], b = x3[3 * i + 1], c = x3[3 * i + 2];
    x4[i] = make_float4(a, b, c, 0.0f);
    out |= outside_box(a, b, c, box);
  }
  if (__any_sync(0xffffffffu, out) && (threadIdx.x & 31) == 0) words[WALK_OUTSIDE] = 1u;
}

// Second moments about the centre of mass, T = sum_j (x_j - com)(x_j - com)^T over the node's
// particles (unit masses), one warp per node with FP64 sums; stored as (Txx, Tyy, Tzz, Txy),
// (Txz, Tyz, 0, 0). Nodes with half >= half_max are never accepted by the walk and get zeros.
// No counterpart in the reference, whose tree carries monopoles only (tree.rs:68-80).
__global__ void k_tree_quad(const uint4* __restrict__ link, const float4* __restrict__ geo,
                            const float4* __restrict__ mass, const float* __restrict__ x3, float4* __restrict__ quad,
                            const uint32_t* __restrict__ counters, uint32_t capacity, float half_max) {
  uint32_t total = 0;
  for (int j = 0; j <= KEY_LEVELS; ++j) total += counters[j];
  total = min(total, capacity);
  const int lane = threadIdx.x & 31;
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  for (uint32_t node = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); node < total; node += warps) {
    double t[6] = {0, 0, 0, 0, 0, 0};
    if (geo[node].w < half_max) {
      const uint4 L = link[node];
      const float4 M = mass[node];
      for (uint32_t i = L.x + lane; i < L.y; i += 32) {
        const double dx = (double)x3[3 * (size_t)i] - M.x, dy = (double)x3[3 * (size_t)i + 1] - M.y,
                     dz = (double)x3[3 * (size_t)i + 2] - M.z;
        t[0] += dx * dx;
        t[1] += dy * dy;
        t[2] += dz * dz;
        t[3] += dx * dy;
        t[4] += dx * dz;
        t[5] += dy * dz;
      }
#pragma unroll
      for (int k = 0; k < 6; ++k)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t[k] += __shfl_xor_sync(0xffffffffu, t[k], o);
    }
    if (lane == 0) {
      quad[2 * (size_t)node] = make_float4((float)t[0], (float)t[1], (float)t[2], (float)t[3]);
      quad[2 * (size_t)node + 1] = make_float4((float)t[4], (float)t[5], 0.0f, 0.0f);
    }
  }
}

cudaError_t tree_positions(TreeNodes& t, size_t n, cudaStream_t s) {
  cudaError_t e = ensure(t.x4, n * sizeof(float4) + WALK_WORDS * sizeof(uint32_t));
  if (e != cudaSuccess) return e;
  return cudaMemsetAsync(tree_words(t, n), 0, WALK_WORDS * sizeof(uint32_t), s);
}

cudaError_t tree_pack(TreeNodes& t, const float* sorted_x3, size_t n, float box, cudaStream_t s) {
  cudaError_t e = tree_positions(t, n, s);
  if (e != cudaSuccess || n == 0) return e;
  count_launch();
  k_pack4<<<(unsigned)std::min<size_t>((n + 255) / 256, 148 * 16), 256, 0, s>>>(sorted_x3, n, box, as<float4>(t.x4),
                                                                               tree_words(t, n));
  return cudaGetLastError();
}

cudaError_t tree_build(TreeNodes& t, const uint64_t* sorted_keys, const float* sorted_x3, size_t n, float box,
                       DevStatus* st, cudaStream_t s, float quad_half_max, int levels, size_t n_box) {
  if (n == 0) return cudaSuccess;
  const size_t cap = 2 * n + 64;
  cudaError_t e;
  if (t.capacity < cap || !t.link.p) {
    if ((e = ensure(t.geo, cap * sizeof(float4))) != cudaSuccess) return e;
    if ((e = ensure(t.mass, cap * sizeof(float4))) != cudaSuccess) return e;
    if ((e = ensure(t.link, cap * sizeof(uint4))) != cudaSuccess) return e;
    t.capacity = cap;
  }
  if ((e = ensure(t.counters, CNT_WORDS * sizeof(uint32_t))) != cudaSuccess) return e;
  const uint32_t tiles = (uint32_t)(n / SUM_TILE + 1);  // the last one may be empty: prefixes up to n
  if ((e = ensure(t.prefix, (size_t)tiles * (CHUNKS_PER_TILE + 1) * sizeof(D3))) != cudaSuccess) return e;

  uint4* link = as<uint4>(t.link);
  float4 *geo = as<float4>(t.geo), *mass = as<float4>(t.mass);
  uint32_t* counters = as<uint32_t>(t.counters);
  D3 *chunk = as<D3>(t.prefix), *totals = chunk + (size_t)tiles * CHUNKS_PER_TILE;
  const uint32_t roots = n_box ? (uint32_t)((n + n_box - 1) / n_box) : 1u, capacity = (uint32_t)t.capacity;
  const float4* x4 = as<float4>(t.x4);
  // The cells of level `spread` are about as many as the particles, so that a smooth distribution has
  // nothing to split below it; a clustered one has, fewer and fewer: their first levels still fill
  // launches (1.0 ms of 2.4 at 256^3 clustered particles went into one cluster from level spread + 3 on).
  int spread = 0;
  for (size_t c = n; c > 1; c >>= 3) ++spread;
  const int tail = std::min(levels, std::max(TOP_LEVEL + 1, spread + (n > CLUSTER_TAIL ? 6 : 3)));
  count_launch();
  if (roots == 1) {
    const unsigned sums = std::min(148u, (tiles + TOP_THREADS / 32 - 1) / (TOP_THREADS / 32));
    k_tree_top<<<1 + sums, TOP_THREADS, 0, s>>>(levels, sorted_keys, x4, (uint32_t)n, box / 2.0f, link, geo, counters,
                                                capacity, chunk, totals, tiles, st);
  } else {
    k_tree_cluster<<<CLUSTER_CTAS, CLUSTER_THREADS, 0, s>>>(0, TOP_LEVEL - 1, levels, sorted_keys, x4, (uint32_t)n,
                                                            box / 2.0f, roots, (uint32_t)n_box, link, geo, counters,
                                                            capacity, nullptr, 0, st);
    count_launch();
    k_sum_tiles<<<BUILD_BLOCKS, BUILD_THREADS, 0, s>>>(x4, (uint32_t)n, chunk, totals, tiles);
  }
  for (int d = TOP_LEVEL; d < tail; ++d) {
    count_launch();
    k_tree_level<<<BUILD_BLOCKS, BUILD_THREADS, 0, s>>>(d, levels, sorted_keys, x4, link, geo, counters, capacity, st);
  }
  count_launch();
  k_tree_cluster<<<CLUSTER_CTAS, CLUSTER_THREADS, 0, s>>>(tail, levels, levels, sorted_keys, x4, (uint32_t)n, box / 2.0f,
                                                          roots, (uint32_t)n_box, link, geo, counters, capacity, totals,
                                                          tiles, st);
  count_launch();
  // a node split at level d or below marks its box dense
  int box_spread = 0;
  for (size_t c = n_box ? n_box : n; c > 1; c >>= 3) ++box_spread;
  const uint32_t dense_depth = (n_box ? n_box : n) <= ORDERED_PARTICLES ? (uint32_t)(box_spread + ORDERED_DEPTH) : 0x80u;
  k_tree_com<<<2 * BUILD_BLOCKS, BUILD_THREADS, 0, s>>>(levels, sorted_keys, link, geo, x4, chunk, totals, mass, counters,
                                                        capacity, dense_depth, (uint32_t)n_box, tree_words(t, n), st);
  t.has_quad = quad_half_max > 0.0f;
  if (t.has_quad) {
    if ((e = ensure(t.quad, 2 * t.capacity * sizeof(float4))) != cudaSuccess) return e;
    count_launch();
    k_tree_quad<<<BUILD_BLOCKS, BUILD_THREADS, 0, s>>>(link, geo, as<float4>(t.mass), sorted_x3, as<float4>(t.quad),
                                                       counters, capacity, quad_half_max);
  }
  return cudaGetLastError();
}

}  // namespace cpm
