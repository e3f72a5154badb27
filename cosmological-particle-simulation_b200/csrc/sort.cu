// sort.cu — octant and Hilbert keys of the tree descent, the stable radix sort of u64 keys, and
// exclusive scans. HBM-bound integer work: coalesced tiles, per-warp ranking with ballots, no
// tensor cores.
#include <cooperative_groups.h>

#include <algorithm>
#include <atomic>
#include <mutex>
#include <vector>

#include "cpm_host.h"
#include "cpm_internal.cuh"

namespace cpm {

constexpr int HFSM_STATES = 24;  // orientations of a cube: an upper bound on the Hilbert curve's states

static std::atomic<unsigned long long> g_launches{0};
unsigned long long launch_count() { return g_launches.load(std::memory_order_relaxed); }
void count_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }

cudaError_t ensure(DevBuf& b, size_t bytes) {
  if (b.p != nullptr && b.bytes >= bytes) return cudaSuccess;
  release(b);
  const size_t want = bytes ? bytes : 16;
  cudaError_t e = cudaMalloc(&b.p, want);
  if (e != cudaSuccess) {
    b.p = nullptr;
    b.bytes = 0;
    return e;
  }
  b.bytes = want;
  return cudaSuccess;
}

void release(DevBuf& b) {
  if (b.p) cudaFree(b.p);
  b.p = nullptr;
  b.bytes = 0;
}

// ---------------------------------------------------------------------------------------------
// Octant keys: tree.rs:186-250 descent. At depth d the octant is (x>=cx)|(y>=cy)<<1|(z>=cz)<<2
// against the node centre; the child centre is centre +- half/2, in f32. The first digit is the
// most significant. Comparisons and additions only, so the digits are bit-exact.
// ---------------------------------------------------------------------------------------------
// With a batch of boxes (n_box > 0: particle i belongs to box i / n_box, boxes one after another),
// the box index goes above the octant digits (bit `box_shift` up), so sorting keeps every box's
// particles together and in box order.
//
// With hkeys, also the particle's Hilbert key over the same cubes: the octant digits are the bits of
// integer coordinates (digit d holds bit levels-1-d of each axis), which J. Skilling's transform
// of axes to the transposed Hilbert index ("Programming the Hilbert curve", AIP Conf. Proc. 707,
// 381, 2004) maps to a key whose first 3d bits name the same level-d cube as the octant key's:
// sorting by it keeps every octree node's particles contiguous and orders the nodes, and the
// particles, along a Hilbert curve.
template <int BITS>
__host__ __device__ __forceinline__ uint64_t hilbert_from_axes(uint32_t X0, uint32_t X1, uint32_t X2) {
  uint32_t X[3] = {X0, X1, X2};
#pragma unroll
  for (int b = BITS - 1; b >= 1; --b) {  // undo excess work, Q = 2^b
    const uint32_t Q = 1u << b, P = Q - 1;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const uint32_t t = (X[0] ^ X[i]) & P;
      const bool inv = (X[i] & Q) != 0u;
      X[0] ^= inv ? P : t;  // invert the low bits of X[0], or exchange them with X[i]'s
      if (i) X[i] ^= inv ? 0u : t;
    }
  }
  X[1] ^= X[0];  // Gray encode
  X[2] ^= X[1];
  uint32_t t = 0;
#pragma unroll
  for (int b = BITS - 1; b >= 1; --b)
    if (X[2] & (1u << b)) t ^= (1u << b) - 1u;
  X[0] ^= t;
  X[1] ^= t;
  X[2] ^= t;
  uint64_t key = 0;
#pragma unroll
  for (int j = BITS - 1; j >= 0; --j)
    key = (key << 3) | (uint64_t)((((X[0] >> j) & 1u) << 2) | (((X[1] >> j) & 1u) << 1) | ((X[2] >> j) & 1u));
  return key;
}

// The same keys digit by digit: because a key's first 3d bits depend only on the first d octant
// digits, digit d is a function of the octant at depth d and of a state (the orientation of the
// curve in the depth-d cube) that the previous digits determine. The state machine is derived on
// the host from hilbert_from_axes itself (states told apart by the order in which they visit the
// eight octants; each transition read off from a representative prefix) and used only after it
// reproduces the transform on every prefix of up to four digits and on 2^16 random coordinates.
// Entry [state * 8 + octant] = digit | next state << 3.
struct HilbertFsm {
  unsigned char t[HFSM_STATES * 8];
  int start = 0;
  int states = 0;
  int ok = 0;
};

static uint64_t hilbert_host(int bits, uint32_t a0, uint32_t a1, uint32_t a2) {
  return bits == KEY_LEVELS ? hilbert_from_axes<KEY_LEVELS>(a0, a1, a2)
                            : hilbert_from_axes<KEY_LEVELS - 2>(a0, a1, a2);
}

static uint64_t hilbert_fsm_host(const HilbertFsm& f, int bits, uint32_t a0, uint32_t a1, uint32_t a2) {
  uint32_t st = (uint32_t)f.start;
  uint64_t key = 0;
  for (int d = 0; d < bits; ++d) {
    const int j = bits - 1 - d;
    const uint32_t o = ((a0 >> j) & 1u) | (((a1 >> j) & 1u) << 1) | (((a2 >> j) & 1u) << 2);
    const uint32_t e = f.t[st * 8 + o];
    key = (key << 3) | (e & 7u);
    st = e >> 3;
  }
  return key;
}

static HilbertFsm derive_hilbert_fsm(int bits) {
  HilbertFsm f;
  // key of the point whose first digits are `pre` (octants, most significant first), zeros after
  auto key_of = [&](const std::vector<uint32_t>& pre) {
    uint32_t a0 = 0, a1 = 0, a2 = 0;
    for (int d = 0; d < bits; ++d) {
      const uint32_t o = d < (int)pre.size() ? pre[d] : 0u;
      a0 = (a0 << 1) | (o & 1u);
      a1 = (a1 << 1) | ((o >> 1) & 1u);
      a2 = (a2 << 1) | ((o >> 2) & 1u);
    }
    return hilbert_host(bits, a0, a1, a2);
  };
  // the digits of the eight octants below prefix `pre`: the state's signature
  auto order_of = [&](std::vector<uint32_t> pre) {
    const int d = (int)pre.size();
    uint32_t sig = 0;
    pre.push_back(0);
    for (uint32_t o = 0; o < 8; ++o) {
      pre.back() = o;
      sig |= (uint32_t)((key_of(pre) >> (3 * (bits - 1 - d))) & 7u) << (3 * o);
    }
    return sig;
  };
  std::vector<uint32_t> sigs;
  std::vector<std::vector<uint32_t>> reps;
  sigs.push_back(order_of({}));
  reps.push_back({});
  for (size_t q = 0; q < sigs.size(); ++q) {
    if ((int)reps[q].size() + 2 > bits || sigs.size() > (size_t)HFSM_STATES) return f;
    for (uint32_t o = 0; o < 8; ++o) {
      std::vector<uint32_t> child = reps[q];
      child.push_back(o);
      const uint32_t sig = order_of(child);
      size_t id = std::find(sigs.begin(), sigs.end(), sig) - sigs.begin();
      if (id == sigs.size()) {
        if (sigs.size() == (size_t)HFSM_STATES) return f;
        sigs.push_back(sig);
        reps.push_back(child);
      }
      f.t[q * 8 + o] = (unsigned char)(((sigs[q] >> (3 * o)) & 7u) | (id << 3));
    }
  }
  f.states = (int)sigs.size();
  // every prefix of up to four digits (the rest zero), then random coordinates
  for (uint32_t p = 0; p < 4096u; ++p)
    for (int len = 1; len <= 4; ++len) {
      std::vector<uint32_t> pre;
      for (int d = 0; d < len; ++d) pre.push_back((p >> (3 * d)) & 7u);
      uint32_t a0 = 0, a1 = 0, a2 = 0;
      for (int d = 0; d < bits; ++d) {
        const uint32_t o = d < len ? pre[d] : 0u;
        a0 = (a0 << 1) | (o & 1u);
        a1 = (a1 << 1) | ((o >> 1) & 1u);
        a2 = (a2 << 1) | ((o >> 2) & 1u);
      }
      if (hilbert_fsm_host(f, bits, a0, a1, a2) != hilbert_host(bits, a0, a1, a2)) return f;
    }
  uint64_t r = 0x9E3779B97F4A7C15ull;
  const uint32_t mask = (1u << bits) - 1u;
  for (int k = 0; k < (1 << 16); ++k) {
    r ^= r << 13;
    r ^= r >> 7;
    r ^= r << 17;
    const uint32_t a0 = (uint32_t)r & mask, a1 = (uint32_t)(r >> 21) & mask, a2 = (uint32_t)(r >> 42) & mask;
    if (hilbert_fsm_host(f, bits, a0, a1, a2) != hilbert_host(bits, a0, a1, a2)) return f;
  }
  f.ok = 1;
  return f;
}

// The state machines of the two key depths in use (21 digits; 19 under a batch of boxes), derived once.
static const HilbertFsm& hilbert_fsm(int bits) {
  static std::once_flag once;
  static HilbertFsm f21, f19;
  std::call_once(once, [] {
    f21 = derive_hilbert_fsm(KEY_LEVELS);
    f19 = derive_hilbert_fsm(KEY_LEVELS - 2);
  });
  return bits == KEY_LEVELS ? f21 : f19;
}

__global__ void k_octant_keys(const float* __restrict__ x3, size_t n, float half0, int levels,
                              uint64_t* __restrict__ keys, DevStatus* st, size_t n_box,
                              int box_shift, uint64_t* __restrict__ hkeys, HilbertFsm fsm) {
  __shared__ unsigned char table[HFSM_STATES * 8];
  const bool use_fsm = hkeys && fsm.ok;
  if (use_fsm) {
    for (int j = threadIdx.x; j < HFSM_STATES * 8; j += blockDim.x) table[j] = fsm.t[j];
    __syncthreads();
  }
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float p0 = x3[3 * i], p1 = x3[3 * i + 1], p2 = x3[3 * i + 2];
  if (!(isfinite(p0) && isfinite(p1) && isfinite(p2))) dev_fail(st, DEV_NONFINITE, (int)i);
  float half = half0, c0 = half0, c1 = half0, c2 = half0;
  uint64_t key = 0, hkey = 0;
  uint32_t a0 = 0, a1 = 0, a2 = 0;  // the digits' bits per axis
  uint32_t state = (uint32_t)fsm.start;
  for (int d = 0; d < levels; ++d) {
    const uint32_t o = (uint32_t)(p0 >= c0) | ((uint32_t)(p1 >= c1) << 1) | ((uint32_t)(p2 >= c2) << 2);
    key = (key << 3) | o;
    if (use_fsm) {
      const uint32_t e = table[state * 8 + o];
      hkey = (hkey << 3) | (e & 7u);
      state = e >> 3;
    } else {
      a0 = (a0 << 1) | (o & 1u);
      a1 = (a1 << 1) | ((o >> 1) & 1u);
      a2 = (a2 << 1) | ((o >> 2) & 1u);
    }
    const float q = half * 0.5f;  // == half / 2.0 exactly
    c0 = __fadd_rn(c0, (o & 1u) ? q : -q);
    c1 = __fadd_rn(c1, (o & 2u) ? q : -q);
    c2 = __fadd_rn(c2, (o & 4u) ? q : -q);
    half = q;
  }
  const uint64_t boxbits = n_box ? (uint64_t)(i / n_box) << box_shift : 0ull;
  if (keys) keys[i] = key | boxbits;
  if (hkeys) {
    const uint64_t h = use_fsm ? hkey
                               : (levels == KEY_LEVELS ? hilbert_from_axes<KEY_LEVELS>(a0, a1, a2)
                                                       : hilbert_from_axes<KEY_LEVELS - 2>(a0, a1, a2));
    hkeys[i] = h | boxbits;
  }
}

void launch_octant_keys(const float* x3, size_t n, float box, int levels, uint64_t* keys, DevStatus* st,
                        cudaStream_t s, size_t n_box, uint64_t* hkeys) {
  if (n == 0) return;
  const int T = 256;
  count_launch();
  HilbertFsm fsm;  // ok = 0: the direct transform
  if (hkeys && (levels == KEY_LEVELS || levels == KEY_LEVELS - 2)) fsm = hilbert_fsm(levels);
  k_octant_keys<<<(unsigned)((n + T - 1) / T), T, 0, s>>>(x3, n, box / 2.0f, levels, keys, st, n_box, 3 * levels,
                                                          hkeys, fsm);
}

// ---------------------------------------------------------------------------------------------
// Exclusive scan of u32: tiles of 2048 (256 threads x 8 items), multi-level for large n.
// ---------------------------------------------------------------------------------------------
constexpr int SC_THREADS = 256;
constexpr int SC_ITEMS = 8;
constexpr int SC_TILE = SC_THREADS * SC_ITEMS;

__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* total, uint32_t* warp_sums) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_sums[warp] = x;
  __syncthreads();
  if (warp == 0) {
    uint32_t w = lane < (SC_THREADS / 32) ? warp_sums[lane] : 0u;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    if (lane < (SC_THREADS / 32)) warp_sums[lane] = w;
  }
  __syncthreads();
  const uint32_t warp_prefix = warp ? warp_sums[warp - 1] : 0u;
  *total = warp_sums[SC_THREADS / 32 - 1];
  return warp_prefix + x - v;
}

__global__ void __launch_bounds__(SC_THREADS) k_scan_reduce(const uint32_t* __restrict__ in, size_t n,
                                                            uint32_t* __restrict__ partial) {
  __shared__ uint32_t ws[SC_THREADS / 32];
  const size_t base = (size_t)blockIdx.x * SC_TILE;
  uint32_t sum = 0;
#pragma unroll
  for (int j = 0; j < SC_ITEMS; ++j) {
    const size_t i = base + (size_t)j * SC_THREADS + threadIdx.x;
    if (i < n) sum += in[i];
  }
  uint32_t total;
  block_exclusive_scan(sum, &total, ws);
  if (threadIdx.x == 0) partial[blockIdx.x] = total;
}

__global__ void __launch_bounds__(SC_THREADS) k_scan_tile(const uint32_t* __restrict__ in, uint32_t* out, size_t n,
                                                          const uint32_t* __restrict__ block_offsets) {
  __shared__ uint32_t ws[SC_THREADS / 32];
  const size_t base = (size_t)blockIdx.x * SC_TILE + (size_t)threadIdx.x * SC_ITEMS;
  uint32_t v[SC_ITEMS];
  uint32_t sum = 0;
#pragma unroll
  for (int j = 0; j < SC_ITEMS; ++j) {
    const size_t i = base + j;
    v[j] = i < n ? in[i] : 0u;
    sum += v[j];
  }
  uint32_t total;
  uint32_t run = block_exclusive_scan(sum, &total, ws);
  if (block_offsets) run += block_offsets[blockIdx.x];
#pragma unroll
  for (int j = 0; j < SC_ITEMS; ++j) {
    const size_t i = base + j;
    if (i < n) out[i] = run;
    run += v[j];
  }
}

static size_t scan_tmp_words(size_t n) {
  size_t total = 0;
  while (n > (size_t)SC_TILE) {
    n = (n + SC_TILE - 1) / SC_TILE;
    total += n + 64;
  }
  return total + 64;
}

static void scan_rec(const uint32_t* in, uint32_t* out, size_t n, uint32_t* tmp, cudaStream_t s) {
  if (n == 0) return;
  if (n <= (size_t)SC_TILE) {
    count_launch();
    k_scan_tile<<<1, SC_THREADS, 0, s>>>(in, out, n, nullptr);
    return;
  }
  const size_t nb = (n + SC_TILE - 1) / SC_TILE;
  uint32_t* partial = tmp;
  count_launch();
  k_scan_reduce<<<(unsigned)nb, SC_THREADS, 0, s>>>(in, n, partial);
  scan_rec(partial, partial, nb, tmp + nb + 64, s);
  count_launch();
  k_scan_tile<<<(unsigned)nb, SC_THREADS, 0, s>>>(in, out, n, partial);
}

cudaError_t exclusive_scan_u32(const uint32_t* in, uint32_t* out, size_t n, DevBuf& tmp, cudaStream_t s) {
  cudaError_t e = ensure(tmp, scan_tmp_words(n) * sizeof(uint32_t));
  if (e != cudaSuccess) return e;
  scan_rec(in, out, n, as<uint32_t>(tmp), s);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
// Stable radix sort of u64 keys, 8-bit digits, giving the sorted keys and the permutation.
//
// Only the upper 32 bits of the keys go through LSD passes, as 8-byte elements (those bits and the
// 32-bit index); the last pass fetches each element's whole key. The particles of a simulation then
// are in order but for short runs that share a cube of level 10 or 11 (0.16 of the mean spacing at
// 256^3 particles; a handful of particles, a few hundred in the core of a cluster): a run of up to
// RUN_SHORT elements is put in order by one thread, of up to RUN_MID by one warp, of up to RUN_BLOCK by one
// CTA, and longer ones by LSD passes of the whole chip over these runs. At 256^3 the scatters move 1.3 GB and
// the counts read 0.5; eight passes of (u64 key, u32 index) moved 3.2 and 1.1.
//
// Per pass: digit counts per tile of 4096 (digit-major), their exclusive scan (one CTA per digit), then
// a stable scatter. Within a tile each warp ranks a contiguous sub-tile in warp-striped rounds (lanes with
// equal digits found by ballots), so equal digits keep their input order.
//
// Up to SMALL_SORT keys go through the passes of their upper 24 bits in one launch of one cluster of
// CTAs.
// ---------------------------------------------------------------------------------------------
constexpr int RS_THREADS = 256;
constexpr int RS_ITEMS = 16;
constexpr int RS_TILE = RS_THREADS * RS_ITEMS;
constexpr int RS_WARPS = RS_THREADS / 32;
constexpr int RS_BINS = 256;
static_assert(RS_THREADS == RS_BINS, "one thread per digit");

constexpr int RUN_SHORT = 8;
constexpr int RUN_MID = 256;
constexpr int RUN_BLOCK_BITS = 12;
constexpr int RUN_BLOCK = 1 << RUN_BLOCK_BITS;

// The lists of runs: RUNS_LISTED of more than RUN_SHORT elements, their starts from RUNS_WORDS on; RUNS_LONG of
// more than RUN_MID, their starts from the end downwards. Then the words of k_long_runs: its phases, and the
// number of runs over RUN_BLOCK (upper half) and of their tiles.
constexpr int RUNS_LISTED = 0, RUNS_LONG = 1, RUNS_PHASES = 2, RUNS_TILES = 4, RUNS_WORDS = 6;

// The lanes whose 9-bit value d equals this lane's (a digit, or 0x100 | lane for a lane without
// an element): one ballot per bit, the same mask as __match_any_sync.
__device__ __forceinline__ uint32_t match_digit(uint32_t d) {
  uint32_t peers = 0xffffffffu;
#pragma unroll
  for (int b = 0; b < 9; ++b) {
    const uint32_t bal = __ballot_sync(0xffffffffu, (d >> b) & 1u);
    peers &= ((d >> b) & 1u) ? bal : ~bal;
  }
  return peers;
}

// Digit counts of each tile, by shared-memory atomics: the elements are in no order by the digit that
// is counted, so lanes seldom meet. FIRST: the elements are the keys themselves, in their order
// (neighbours share their upper digits then, which `same` takes out).
template <bool FIRST>
__global__ void __launch_bounds__(RS_THREADS) k_radix_hist(const uint64_t* __restrict__ keys, int drop,
                                                           const uint2* __restrict__ in, size_t n, int shift,
                                                           uint32_t* __restrict__ tile_hist, int ntiles,
                                                           uint32_t* __restrict__ runs) {
  __shared__ uint32_t h[RS_BINS];
  h[threadIdx.x] = 0;
  if (runs && blockIdx.x == 0 && threadIdx.x < RUNS_WORDS) runs[threadIdx.x] = 0;
  __syncthreads();
  const size_t base = (size_t)blockIdx.x * RS_TILE;
  uint32_t v[RS_ITEMS];
#pragma unroll
  for (int j = 0; j < RS_ITEMS; ++j) {
    const size_t i = base + (size_t)j * RS_THREADS + threadIdx.x;
    v[j] = i >= n ? 0u : FIRST ? (uint32_t)(keys[i] >> drop) : in[i].x;
  }
#pragma unroll
  for (int j = 0; j < RS_ITEMS; ++j) {
    const bool valid = base + (size_t)j * RS_THREADS + threadIdx.x < n;
    const uint32_t d = (v[j] >> shift) & (RS_BINS - 1);
    const uint32_t d0 = __shfl_sync(0xffffffffu, d, 0);
    const bool same = __all_sync(0xffffffffu, valid && d == d0);
    if (same ? (threadIdx.x & 31) == 0 : valid) atomicAdd(&h[d], same ? 32u : 1u);
  }
  __syncthreads();
  tile_hist[(size_t)threadIdx.x * ntiles + blockIdx.x] = h[threadIdx.x];
}

// Exclusive scan of the tile counts of digit blockIdx.x, in place; its total to totals[digit].
__global__ void __launch_bounds__(SC_THREADS) k_radix_scan(uint32_t* __restrict__ tile_hist, int ntiles,
                                                           uint32_t* __restrict__ totals) {
  __shared__ uint32_t ws[SC_THREADS / 32];
  uint32_t* row = tile_hist + (size_t)blockIdx.x * ntiles;
  uint32_t carry = 0;
  for (int c0 = 0; c0 < ntiles; c0 += SC_TILE) {
    const int i0 = c0 + threadIdx.x * SC_ITEMS;
    uint32_t v[SC_ITEMS], sum = 0;
#pragma unroll
    for (int j = 0; j < SC_ITEMS; ++j) {
      v[j] = i0 + j < ntiles ? row[i0 + j] : 0u;
      sum += v[j];
    }
    uint32_t total;
    uint32_t run = carry + block_exclusive_scan(sum, &total, ws);
#pragma unroll
    for (int j = 0; j < SC_ITEMS; ++j) {
      if (i0 + j < ntiles) row[i0 + j] = run;
      run += v[j];
    }
    carry += total;
    __syncthreads();  // the next round reuses the warp sums
  }
  if (threadIdx.x == 0) totals[blockIdx.x] = carry;
}

// One stable pass: the tile is ranked by digit (per warp with match_digit, warps in order),
// reordered in shared memory, and each digit's run is written out contiguously, so consecutive
// threads store consecutive addresses. LAST: whole keys and indices are written.
template <bool FIRST, bool LAST>
__global__ void __launch_bounds__(RS_THREADS) k_radix_scatter(const uint64_t* __restrict__ keys, int drop,
                                                              const uint2* __restrict__ in, uint2* __restrict__ out,
                                                              uint64_t* __restrict__ kout, uint32_t* __restrict__ vout,
                                                              size_t n, int shift,
                                                              const uint32_t* __restrict__ tile_hist,
                                                              const uint32_t* __restrict__ totals, int ntiles) {
  __shared__ uint2 se[RS_TILE];
  __shared__ uint32_t wc[RS_WARPS][RS_BINS];
  __shared__ uint32_t gbase[RS_BINS];
  __shared__ uint32_t ws[SC_THREADS / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, t = threadIdx.x;
#pragma unroll
  for (int q = 0; q < RS_WARPS; ++q) wc[q][t] = 0;
  __syncthreads();
  const unsigned lt_mask = (1u << lane) - 1u;
  const size_t tile0 = (size_t)blockIdx.x * RS_TILE;
  const size_t wbase = tile0 + (size_t)warp * 32 * RS_ITEMS;
  uint2 e[RS_ITEMS];
  uint32_t rank[RS_ITEMS];
#pragma unroll
  for (int j = 0; j < RS_ITEMS; ++j) {
    const size_t i = wbase + (size_t)j * 32 + lane;
    e[j] = make_uint2(0u, 0u);
    if (i < n) e[j] = FIRST ? make_uint2((uint32_t)(keys[i] >> drop), (uint32_t)i) : in[i];
  }
  // Thread t = digit t: where its elements of this tile start in the output.
  uint32_t sum;
  const uint32_t before = tile_hist[(size_t)t * ntiles + blockIdx.x] + block_exclusive_scan(totals[t], &sum, ws);
#pragma unroll
  for (int j = 0; j < RS_ITEMS; ++j) {
    const bool valid = wbase + (size_t)j * 32 + lane < n;
    const uint32_t d = valid ? (e[j].x >> shift) & (RS_BINS - 1) : (0x100u | (uint32_t)lane);
    const uint32_t peers = match_digit(d);
    uint32_t prev = 0;
    if (valid) prev = wc[warp][d];
    __syncwarp();
    if (valid) {
      rank[j] = prev + (uint32_t)__popc(peers & lt_mask);
      if ((__ffs(peers) - 1) == lane) wc[warp][d] = prev + (uint32_t)__popc(peers);
    }
    __syncwarp();
  }
  __syncthreads();
  // Thread t = digit t: its tile total, then the exclusive scan over digits (tile-local starts).
  uint32_t tot = 0;
#pragma unroll
  for (int w = 0; w < RS_WARPS; ++w) tot += wc[w][t];
  const uint32_t start = block_exclusive_scan(tot, &sum, ws);
  gbase[t] = before - start;
  uint32_t run = start;
#pragma unroll
  for (int w = 0; w < RS_WARPS; ++w) {
    const uint32_t c = wc[w][t];
    wc[w][t] = run;
    run += c;
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < RS_ITEMS; ++j)
    if (wbase + (size_t)j * 32 + lane < n) se[wc[warp][(e[j].x >> shift) & (RS_BINS - 1)] + rank[j]] = e[j];
  __syncthreads();
  const uint32_t count = (uint32_t)min((size_t)RS_TILE, n - tile0);
#pragma unroll 4
  for (uint32_t q = t; q < count; q += RS_THREADS) {
    const uint2 v = se[q];
    const uint32_t pos = gbase[(v.x >> shift) & (RS_BINS - 1)] + q;
    if constexpr (LAST) {
      kout[pos] = __ldg(keys + v.y);
      vout[pos] = v.y;
    } else {
      out[pos] = v;
    }
  }
}

// ---------------------------------------------------------------------------------------------
// The runs of elements that share key >> drop, put in order by their lower bits (stable: a run arrives
// in input order).
// ---------------------------------------------------------------------------------------------
// The thread of a run's first element sorts it by insertion, or lists it.
__global__ void k_short_runs(uint64_t* sorted, uint32_t* perm, size_t n, int drop, uint32_t* runs) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i + 1 >= n) return;
  // (another thread's insertions leave the upper bits of its run's slots as they are)
  const volatile uint64_t* keys = sorted;
  const uint64_t h = keys[i] >> drop;
  if ((keys[i + 1] >> drop) != h || (i > 0 && (keys[i - 1] >> drop) == h)) return;
  int len = 2;
  while (len <= RUN_SHORT && i + len < n && (keys[i + len] >> drop) == h) ++len;
  if (len > RUN_SHORT) {
    runs[RUNS_WORDS + atomicAdd(&runs[RUNS_LISTED], 1u)] = (uint32_t)i;
    return;
  }
  uint64_t* k = sorted + i;
  uint32_t* v = perm + i;
  for (int a = 1; a < len; ++a) {
    const uint64_t key = k[a];
    const uint32_t val = v[a];
    int b = a;
    for (; b > 0 && k[b - 1] > key; --b) {
      k[b] = k[b - 1];
      v[b] = v[b - 1];
    }
    k[b] = key;
    v[b] = val;
  }
}

// One warp per listed run of up to RUN_MID elements, RUN_MID / 32 to a lane: every element's place is
// the number of elements before it.
__global__ void __launch_bounds__(256) k_mid_runs(uint64_t* sorted, uint32_t* perm, size_t n, int drop, uint32_t* runs,
                                                  uint32_t runs_end) {
  constexpr int PER = RUN_MID / 32;
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const uint32_t count = runs[RUNS_LISTED];
  for (uint32_t r = blockIdx.x * 8 + (threadIdx.x >> 5); r < count; r += gridDim.x * 8) {
    const size_t start = runs[RUNS_WORDS + r];
    const uint64_t h = sorted[start] >> drop;
    uint64_t k[PER];
    uint32_t v[PER];
    int len = 0;
#pragma unroll
    for (int q = 0; q < PER; ++q) {
      const size_t i = start + 32 * q + lane;
      k[q] = ~0ull;
      const bool in = len == 32 * q && i < n && (sorted[i] >> drop) == h;
      if (in) {
        k[q] = sorted[i];
        v[q] = perm[i];
      }
      len += __popc(__ballot_sync(FULL, in));
    }
    if (len == RUN_MID && start + RUN_MID < n && (sorted[start + RUN_MID] >> drop) == h) {
      if (lane == 0) runs[runs_end - 1 - atomicAdd(&runs[RUNS_LONG], 1u)] = (uint32_t)start;
      continue;
    }
    int place[PER] = {};
#pragma unroll
    for (int b = 0; b < PER; ++b) {
      for (int j = 32 * b; j < min(len, 32 * b + 32); ++j) {
        const uint64_t other = __shfl_sync(FULL, k[b], j & 31);
#pragma unroll
        for (int q = 0; q < PER; ++q) place[q] += (int)(other < k[q] || (other == k[q] && j < 32 * q + lane));
      }
    }
#pragma unroll
    for (int q = 0; q < PER; ++q)
      if (32 * q + lane < len) {
        sorted[start + place[q]] = k[q];
        perm[start + place[q]] = v[q];
      }
  }
}

// The runs of more than RUN_MID elements, in phases over all CTAs (Phases): first each run's end; runs of up to
// RUN_BLOCK elements are sorted by one CTA in shared memory (bitonic, by the lower bits and then the place in the run).
// The longer ones (a collapsed core in a large box, coincident particles) go through LSD passes together, cut into
// tiles of LONG_TILE elements that each belong to one run: digit counts per tile, their scan per run and digit, the
// scatter, which ranks as k_radix_scatter does. The work is that of these runs' elements and spread over the chip, so
// the sort takes about as long for any input: 10^6 particles in one halo of 1e-4 of the box 0.31 ms with keys and reorder
// (a uniform box 0.15), 4e6 0.87 (0.35); one CTA per run, of whatever length, took 12.9 and 53 ms.
constexpr int LONG_ITEMS = 8;
constexpr int LONG_TILE = RS_THREADS * LONG_ITEMS;
constexpr int LONG_CTAS = 148 * 2;
// The tables of these runs, in words that the caller provides: starts, ends, first tiles, digit totals, tile counts.
// At most n / (RUN_BLOCK + 1) runs of n / LONG_TILE tiles and one more each: less than 0.26 n words.
struct LongTables {
  uint32_t *start, *end, *tile0, *totals, *hist;
  __device__ LongTables(uint32_t* words, size_t n) {
    const size_t cap = n / (RUN_BLOCK + 1);
    start = words;
    end = start + cap;
    tile0 = end + cap;
    totals = tile0 + cap;
    hist = totals + cap * RS_BINS;
  }
};

__global__ void __launch_bounds__(RS_THREADS) k_long_runs(uint64_t* sorted, uint32_t* perm, size_t n, int drop,
                                                          uint32_t* runs, uint32_t runs_end, uint64_t* kalt,
                                                          uint32_t* valt, uint32_t* tables, DevStatus* st) {
  __shared__ __align__(16) unsigned char smem[RUN_BLOCK * sizeof(uint64_t)];
  __shared__ uint32_t wc[RS_WARPS][RS_BINS], gbase[RS_BINS], ws[SC_THREADS / 32];
  static_assert(LONG_TILE * (sizeof(uint64_t) + sizeof(uint32_t)) <= sizeof(smem), "a tile in shared memory");
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const uint32_t nlong = runs[RUNS_LONG];
  if (nlong == 0u) return;
  const uint64_t low = (1ull << drop) - 1ull;
  const LongTables T(tables, n);
  Phases phases(runs + RUNS_PHASES);
  uint32_t item;

  uint64_t* comp = reinterpret_cast<uint64_t*>(smem);
  while (phases.take(nlong, item)) {
    const size_t start = runs[runs_end - 1 - item];
    const uint64_t h = __ldcg(sorted + start) >> drop;
    size_t lo = start + RUN_MID, hi = n;  // everything before lo is in the run, nothing from hi on
    while (lo < hi) {
      const size_t len = hi - lo;
      const int in = __syncthreads_count((__ldcg(sorted + lo + len * t / RS_THREADS) >> drop) == h);
      if (in < RS_THREADS) hi = lo + len * in / RS_THREADS;
      if (in > 0) lo += len * (in - 1) / RS_THREADS + 1;
    }
    const uint32_t len = (uint32_t)(lo - start);
    if (len > (uint32_t)RUN_BLOCK) {
      if (t == 0) {
        const unsigned long long tiles = (len + LONG_TILE - 1) / LONG_TILE;
        const unsigned long long old =
            atomicAdd(reinterpret_cast<unsigned long long*>(runs + RUNS_TILES), (1ull << 32) | tiles);
        const uint32_t r = (uint32_t)(old >> 32);
        __stcg(T.start + r, (uint32_t)start);
        __stcg(T.end + r, (uint32_t)lo);
        __stcg(T.tile0 + r, (uint32_t)old);
      }
    } else {
      uint32_t size = 2 * RUN_MID;
      while (size < len) size <<= 1;
      for (uint32_t q = t; q < size; q += RS_THREADS)
        comp[q] = q < len ? ((sorted[start + q] & low) << RUN_BLOCK_BITS) | q : ~0ull;
      __syncthreads();
      for (uint32_t k = 2; k <= size; k <<= 1)
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
          for (uint32_t q = t; q < size / 2; q += RS_THREADS) {
            const uint32_t a = 2 * q - (q & (j - 1)), b = a + j;
            const uint64_t x = comp[a], y = comp[b];
            if ((x > y) == ((a & k) == 0u)) {
              comp[a] = y;
              comp[b] = x;
            }
          }
          __syncthreads();
        }
      uint32_t v[RUN_BLOCK / RS_THREADS];
#pragma unroll
      for (int m = 0; m < RUN_BLOCK / RS_THREADS; ++m) {
        const uint32_t q = t + m * RS_THREADS;
        if (q < len) v[m] = perm[start + (comp[q] & (RUN_BLOCK - 1))];
      }
      __syncthreads();
#pragma unroll
      for (int m = 0; m < RUN_BLOCK / RS_THREADS; ++m) {
        const uint32_t q = t + m * RS_THREADS;
        if (q < len) {
          sorted[start + q] = (h << drop) | (comp[q] >> RUN_BLOCK_BITS);
          perm[start + q] = v[m];
        }
      }
    }
    phases.done();
  }
  bool ok = phases.next(nlong);
  const unsigned long long found = __ldcg(reinterpret_cast<unsigned long long*>(runs + RUNS_TILES));
  const uint32_t nrun = (uint32_t)(found >> 32), ntile = (uint32_t)found;
  if (ok && nrun == 0u) return;

  auto run_of = [&](uint32_t tile) {  // the last run that starts at or before the tile
    uint32_t a = 0, b = nrun;
    while (b - a > 1) {
      const uint32_t m = (a + b) / 2;
      if (__ldcg(T.tile0 + m) <= tile)
        a = m;
      else
        b = m;
    }
    return a;
  };
  auto tiles_of = [&](uint32_t r) { return (__ldcg(T.end + r) - __ldcg(T.start + r) + LONG_TILE - 1) / LONG_TILE; };
  uint64_t *ka = sorted, *kb = kalt, *sk = comp;
  uint32_t *va = perm, *vb = valt, *sv = reinterpret_cast<uint32_t*>(sk + LONG_TILE);
  const int passes = (drop + 15) / 16 * 2;  // an even number: the result is back in place
  for (int p = 0; p < passes && ok; ++p) {
    const int shift = 8 * p;
    auto digit = [&](uint64_t k) { return (uint32_t)((k & low) >> shift) & (RS_BINS - 1); };
    while (phases.take(ntile, item)) {
      const uint32_t r = run_of(item), tile0 = __ldcg(T.tile0 + r), tile = item - tile0;
      const size_t first = (size_t)__ldcg(T.start + r) + (size_t)tile * LONG_TILE;
      const uint32_t count = min((uint32_t)LONG_TILE, __ldcg(T.end + r) - (uint32_t)first);
      gbase[t] = 0;
      __syncthreads();
#pragma unroll
      for (int j = 0; j < LONG_ITEMS; ++j) {
        const uint32_t q = t + j * RS_THREADS;
        const bool valid = q < count;
        const uint32_t d = valid ? digit(__ldcg(ka + first + q)) : 0u;
        const uint32_t d0 = __shfl_sync(0xffffffffu, d, 0);
        const bool same = __all_sync(0xffffffffu, valid && d == d0);
        if (same ? lane == 0 : valid) atomicAdd(&gbase[d], same ? 32u : 1u);
      }
      __syncthreads();
      __stcg(T.hist + (size_t)tile0 * RS_BINS + (size_t)t * tiles_of(r) + tile, gbase[t]);
      phases.done();
    }
    ok = phases.next(ntile);
    while (ok && phases.take(nrun * (RS_BINS / RS_WARPS), item)) {  // a warp per run and digit
      const uint32_t row = item * RS_WARPS + warp, r = row / RS_BINS, d = row % RS_BINS, tiles = tiles_of(r);
      uint32_t* h = T.hist + (size_t)__ldcg(T.tile0 + r) * RS_BINS + (size_t)d * tiles;
      uint32_t carry = 0;
      for (uint32_t i0 = 0; i0 < tiles; i0 += 32) {
        const uint32_t i = i0 + lane, x = i < tiles ? __ldcg(h + i) : 0u;
        uint32_t incl = x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += y;
        }
        if (i < tiles) __stcg(h + i, carry + incl - x);
        carry += __shfl_sync(0xffffffffu, incl, 31);
      }
      if (lane == 0) __stcg(T.totals + row, carry);
      phases.done();
    }
    ok = ok && phases.next(nrun * (RS_BINS / RS_WARPS));
    while (ok && phases.take(ntile, item)) {
      const uint32_t r = run_of(item), tile0 = __ldcg(T.tile0 + r), tile = item - tile0;
      const size_t start = __ldcg(T.start + r), first = start + (size_t)tile * LONG_TILE;
      const uint32_t count = min((uint32_t)LONG_TILE, __ldcg(T.end + r) - (uint32_t)first);
#pragma unroll
      for (int w = 0; w < RS_WARPS; ++w) wc[w][t] = 0;
      uint32_t sum;
      const uint32_t before = __ldcg(T.hist + (size_t)tile0 * RS_BINS + (size_t)t * tiles_of(r) + tile) +
                              block_exclusive_scan(__ldcg(T.totals + (size_t)r * RS_BINS + t), &sum, ws);
      uint64_t k[LONG_ITEMS];
      uint32_t v[LONG_ITEMS], rank[LONG_ITEMS];
#pragma unroll
      for (int j = 0; j < LONG_ITEMS; ++j) {
        const uint32_t q = (uint32_t)(warp * LONG_ITEMS + j) * 32 + lane;
        k[j] = q < count ? __ldcg(ka + first + q) : 0ull;
        v[j] = q < count ? __ldcg(va + first + q) : 0u;
      }
#pragma unroll
      for (int j = 0; j < LONG_ITEMS; ++j) {
        const bool valid = (uint32_t)(warp * LONG_ITEMS + j) * 32 + lane < count;
        const uint32_t d = valid ? digit(k[j]) : (0x100u | (uint32_t)lane);
        const uint32_t peers = match_digit(d);
        uint32_t prev = 0;
        if (valid) prev = wc[warp][d];
        __syncwarp();
        rank[j] = prev + (uint32_t)__popc(peers & ((1u << lane) - 1u));
        if (valid && (__ffs(peers) - 1) == lane) wc[warp][d] = prev + (uint32_t)__popc(peers);
        __syncwarp();
      }
      __syncthreads();
      uint32_t tot = 0;
#pragma unroll
      for (int w = 0; w < RS_WARPS; ++w) tot += wc[w][t];
      uint32_t run = block_exclusive_scan(tot, &sum, ws);
      gbase[t] = before - run;
#pragma unroll
      for (int w = 0; w < RS_WARPS; ++w) {
        const uint32_t c = wc[w][t];
        wc[w][t] = run;
        run += c;
      }
      __syncthreads();
#pragma unroll
      for (int j = 0; j < LONG_ITEMS; ++j)
        if ((uint32_t)(warp * LONG_ITEMS + j) * 32 + lane < count) {
          const uint32_t q = wc[warp][digit(k[j])] + rank[j];
          sk[q] = k[j];
          sv[q] = v[j];
        }
      __syncthreads();
#pragma unroll
      for (int j = 0; j < LONG_ITEMS; ++j) {
        const uint32_t q = t + j * RS_THREADS;
        if (q < count) {
          const size_t pos = start + (gbase[digit(sk[q])] + q);
          __stcg(kb + pos, sk[q]);
          __stcg(vb + pos, sv[q]);
        }
      }
      phases.done();
    }
    ok = ok && phases.next(ntile);
    uint64_t* tk = ka;
    ka = kb;
    kb = tk;
    uint32_t* tv = va;
    va = vb;
    vb = tv;
  }
  if (!ok && t == 0) dev_fail(st, DEV_WAIT_LIMIT, (int)nlong);
}

// ---------------------------------------------------------------------------------------------
// Small sorts: the passes over the keys' digits from `drop` up in one launch of one cluster. CTA c holds the c-th
// contiguous part of the elements in registers (warps contiguous within it, rounds of 32 within
// them), ranks them by digit as k_radix_scatter does, exchanges the digit totals with the other CTAs
// through global memory and stores the elements where they go; a cluster barrier on either side.
// ---------------------------------------------------------------------------------------------
constexpr int SS_CTAS = 8;
constexpr int SS_THREADS = 1024;
constexpr int SS_WARPS = SS_THREADS / 32;
constexpr int SS_ITEMS = 8;
constexpr size_t SMALL_SORT = (size_t)SS_CTAS * SS_THREADS * SS_ITEMS;  // 65,536 keys

__global__ void __cluster_dims__(SS_CTAS, 1, 1) __launch_bounds__(SS_THREADS)
    k_sort_small(const uint64_t* __restrict__ keys, uint64_t* sorted, uint32_t* perm, uint64_t* kalt, uint32_t* valt,
                 uint32_t* cta_hist, uint32_t n, int drop, int passes, uint32_t* runs) {
  __shared__ uint32_t wc[SS_WARPS][RS_BINS];  // 32 KB
  __shared__ uint32_t gbase[RS_BINS], ws[SS_WARPS];
  const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const uint32_t cta = blockIdx.x;
  const uint32_t rounds = (n + SS_CTAS * SS_THREADS - 1) / (SS_CTAS * SS_THREADS);
  const uint32_t first = ((cta * SS_WARPS + warp) * rounds) * 32 + lane;
  const unsigned lt_mask = (1u << lane) - 1u;
  if (runs && cta == 0 && t < RUNS_WORDS) runs[t] = 0;
  for (int p = 0; p < passes; ++p) {
    // the last pass writes to `sorted`, the passes before it alternate
    const bool to_sorted = ((passes - 1 - p) & 1) == 0;
    const uint64_t* kin = p == 0 ? keys : (to_sorted ? kalt : sorted);
    const uint32_t* vin = to_sorted ? valt : perm;
    uint64_t* kout = to_sorted ? sorted : kalt;
    uint32_t* vout = to_sorted ? perm : valt;
    const int shift = drop + 8 * p;
    for (int q = t; q < SS_WARPS * RS_BINS; q += SS_THREADS) (&wc[0][0])[q] = 0;
    uint64_t k[SS_ITEMS];
    uint32_t v[SS_ITEMS], rank[SS_ITEMS];
#pragma unroll
    for (int j = 0; j < SS_ITEMS; ++j) {
      const uint32_t i = first + 32u * j;
      const bool valid = j < (int)rounds && i < n;
      k[j] = valid ? __ldcg(kin + i) : 0ull;
      v[j] = valid ? (p == 0 ? i : __ldcg(vin + i)) : 0u;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < SS_ITEMS; ++j) {
      if (j >= (int)rounds) break;
      const bool valid = first + 32u * j < n;
      const uint32_t d = valid ? (uint32_t)(k[j] >> shift) & (RS_BINS - 1) : (0x100u | (uint32_t)lane);
      const uint32_t peers = match_digit(d);
      uint32_t prev = 0;
      if (valid) prev = wc[warp][d];
      __syncwarp();
      rank[j] = prev + (uint32_t)__popc(peers & lt_mask);
      if (valid && (__ffs(peers) - 1) == lane) wc[warp][d] = prev + (uint32_t)__popc(peers);
      __syncwarp();
    }
    __syncthreads();
    if (t < RS_BINS) {  // thread t = digit t: each warp's start within the CTA, the CTA's total
      uint32_t run = 0;
      for (int w = 0; w < SS_WARPS; ++w) {
        const uint32_t c = wc[w][t];
        wc[w][t] = run;
        run += c;
      }
      __stcg(cta_hist + cta * RS_BINS + t, run);
    }
    cluster.sync();
    uint32_t all = 0, before = 0;
    if (t < RS_BINS)
      for (uint32_t c = 0; c < SS_CTAS; ++c) {
        const uint32_t x = __ldcg(cta_hist + c * RS_BINS + t);
        all += x;
        before += c < cta ? x : 0u;
      }
    uint32_t incl = all;  // exclusive scan of the digit totals over threads 0..255
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) ws[warp] = incl;
    __syncthreads();
    if (t < RS_BINS) {
      uint32_t lead = 0;
      for (int w = 0; w < warp; ++w) lead += ws[w];
      gbase[t] = lead + incl - all + before;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < SS_ITEMS; ++j)
      if (j < (int)rounds && first + 32u * j < n) {
        const uint32_t d = (uint32_t)(k[j] >> shift) & (RS_BINS - 1);
        const uint32_t pos = gbase[d] + wc[warp][d] + rank[j];
        __stcg(kout + pos, k[j]);
        __stcg(vout + pos, v[j]);
      }
    cluster.sync();
  }
}

cudaError_t radix_sort_keys(const uint64_t* keys, uint64_t* sorted, uint32_t* perm, size_t n, int bits,
                            SortScratch& sc, DevStatus* st, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  if (n > 0xFFFFFFFFull || bits < 1 || bits > 64) return cudaErrorInvalidValue;
  const int ntiles = (int)((n + RS_TILE - 1) / RS_TILE);
  cudaError_t e;
  if ((e = ensure(sc.pairs, n * sizeof(uint2))) != cudaSuccess) return e;
  if ((e = ensure(sc.pairs_alt, n * sizeof(uint2))) != cudaSuccess) return e;
  const size_t hist_words = (size_t)RS_BINS * std::max(ntiles, SS_CTAS) + RS_BINS;
  if ((e = ensure(sc.tile_hist, hist_words * sizeof(uint32_t))) != cudaSuccess) return e;
  uint32_t* hist = as<uint32_t>(sc.tile_hist);
  const bool small = n <= SMALL_SORT;
  const int drop = std::max(0, bits - (small ? 24 : 32));
  uint32_t* runs = nullptr;
  // a listed run holds more than RUN_SHORT elements, one of the second list more than RUN_MID
  const uint32_t runs_end = (uint32_t)(RUNS_WORDS + n / (RUN_SHORT + 1) + n / (RUN_MID + 1) + 2);
  if (drop) {
    if ((e = ensure(sc.runs, (size_t)runs_end * sizeof(uint32_t))) != cudaSuccess) return e;
    runs = as<uint32_t>(sc.runs);
  }
  uint2 *in = as<uint2>(sc.pairs), *out = as<uint2>(sc.pairs_alt);
  uint32_t* totals = hist + (size_t)RS_BINS * ntiles;
  const int passes = (bits - drop + 7) / 8;
  if (small) {
    count_launch();
    k_sort_small<<<SS_CTAS, SS_THREADS, 0, s>>>(keys, sorted, perm, as<uint64_t>(sc.pairs), as<uint32_t>(sc.pairs_alt),
                                                hist, (uint32_t)n, drop, passes, runs);
  }
  for (int p = 0; p < passes && !small; ++p) {
    const bool first = p == 0, last = p == passes - 1;
    const int shift = 8 * p;
    count_launch();
    (first ? k_radix_hist<true> : k_radix_hist<false>)<<<ntiles, RS_THREADS, 0, s>>>(
        keys, drop, in, n, shift, hist, ntiles, first ? runs : nullptr);
    count_launch();
    k_radix_scan<<<RS_BINS, SC_THREADS, 0, s>>>(hist, ntiles, totals);
    auto scatter = first ? (last ? k_radix_scatter<true, true> : k_radix_scatter<true, false>)
                         : (last ? k_radix_scatter<false, true> : k_radix_scatter<false, false>);
    count_launch();
    scatter<<<ntiles, RS_THREADS, 0, s>>>(keys, drop, in, out, sorted, perm, n, shift, hist, totals, ntiles);
    std::swap(in, out);
  }
  if (drop) {
    count_launch();
    k_short_runs<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(sorted, perm, n, drop, runs);
    count_launch();
    k_mid_runs<<<(unsigned)std::min<size_t>(n / 2048 + 1, 148 * 8), 256, 0, s>>>(sorted, perm, n, drop, runs, runs_end);
    count_launch();
    // pairs_alt: n indices, and the tables in its other half
    uint32_t* valt = as<uint32_t>(sc.pairs_alt);
    k_long_runs<<<LONG_CTAS, RS_THREADS, 0, s>>>(sorted, perm, n, drop, runs, runs_end, as<uint64_t>(sc.pairs), valt,
                                                 valt + n, st);
  }
  return cudaGetLastError();
}

}  // namespace cpm

// Self-check of the table-driven Hilbert keys (host only): `samples` random integer coordinates
// (xorshift from `seed`) keyed by the state machine and by the transform; mismatches counted.
extern "C" int cpm_hilbert_fsm_check(int levels, uint64_t samples, uint64_t seed, uint64_t* mismatches, int* states) {
  using namespace cpm;
  if ((levels != KEY_LEVELS && levels != KEY_LEVELS - 2) || !mismatches || !states)
    return set_error(nullptr, CPM_E_INVALID, "cpm_hilbert_fsm_check: levels must be 21 or 19, outputs non-null");
  const HilbertFsm& f = hilbert_fsm(levels);
  *states = f.ok ? f.states : 0;
  uint64_t bad = 0, r = seed | 1ull;
  const uint32_t mask = (1u << levels) - 1u;
  for (uint64_t k = 0; k < samples; ++k) {
    r ^= r << 13;
    r ^= r >> 7;
    r ^= r << 17;
    const uint32_t a0 = (uint32_t)r & mask, a1 = (uint32_t)(r >> 21) & mask, a2 = (uint32_t)(r >> 42) & mask;
    if (!f.ok || hilbert_fsm_host(f, levels, a0, a1, a2) != hilbert_host(levels, a0, a1, a2)) ++bad;
  }
  *mismatches = bad;
  return CPM_OK;
}
