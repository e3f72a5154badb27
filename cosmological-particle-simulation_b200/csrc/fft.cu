// fft.cu — shared-memory Stockham FFTs and the PM Poisson solve (fft.rs:40-95, poisson.rs:33-88).
//
// Layouts in HBM
//   real mesh      f32  [n][n][n]            (ix*n + iy)*n + iz, z fastest (mesh.rs:11)
//   half spectrum  c32  [n][n][half_row(n)]  kz in [0, n/2], rows padded to whole 32-byte sectors; the
//                                            rest of kz follows from Hermitian symmetry
//
// Every pass reads and writes each of its spectra once (the y gradient pass the potential twice, from
// L2), in tiles of 8 or 16 lines, one tile per CTA. Lines are transformed by radix-8/4/2/3/5 Stockham stages; the
// first takes its inputs straight from global memory into registers, the last stores its outputs there, and
// shared memory carries the exchanges between them.
//   - Strided y/x lines: the line (the contiguous kz column) is on consecutive lanes, in global memory
//     (64 or 128 contiguous bytes) and in the exchanges (no bank conflicts whatever the stage's stride).
//   - Contiguous z rows: the first and last stage run along the row on consecutive lanes.
// Twiddles come from a table exp(-2 pi i m / n) built in double precision on the host.
//
// What bounds them: at n = 512 (no pass fits L2) the five passes take 0.48 (R2C, 3.3 TB/s), 0.23 (y, 4.4),
// 0.72 (x, 2.2), 0.82 (y gradient, 3.6) and 0.77 ms (C2R, 4.2), together 3.02: the first and last by
// shared-memory and L1 wavefronts (81 % in C2R), the x pass by issue and barriers (three transforms and the Green's
// function per line). As persistent kernels that copied tiles in by cp.async, transformed them in place and copied
// them out they took 3.97 (256: 0.489, now 0.400; 128: 0.092, now 0.067).
//
// Real z lines use the half-length complex transform: z[m] = x[2m] + i x[2m+1] is transformed
// with n/2 points and split into the n/2+1 outputs with the twiddles of length n (and the
// reverse for C2R), which halves the arithmetic and shared memory of the z passes.
//
// The Poisson solve runs as
//   1. z pass: R2C of each z row; the input is the f32 delta or the u64 fixed-point mass mesh,
//      converted on load to delta = c/mean - 1 (integrator.rs:117-126);
//   2. y pass: forward c2c along y;
//   3. x pass: forward c2c along x, the Green's function of poisson.rs:52-74 in the reference's f32
//      operation order (optionally divided by the CIC window squared), then two inverse x
//      transforms: of -i k_x phi (x component) and of phi — two half spectra written;
//   4. y pass: inverse c2c along y of the x component; and, reading the x-transformed phi once,
//      of -i k_y phi and -i k_z phi (k_y and k_z are constant along an x line, so the factors
//      commute with the x transform), written as the y and z components;
//   5. z pass: C2R of each row, scaled by 1/n^3 (poisson.rs:77-87), into three f32 meshes.
#include <algorithm>
#include <cmath>
#include <vector>

#include "cpm_internal.cuh"

namespace cpm {

constexpr int TW = 16;  // lines per tile, unless said otherwise

// ---------------------------------------------------------------------------------------------
// Complex helpers and small DFTs
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 conjf2(float2 a) { return make_float2(a.x, -a.y); }
// multiply by exp(sign i pi/2): -i for the forward transform, +i for the inverse
template <bool INV>
__device__ __forceinline__ float2 rot90(float2 a) {
  return INV ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
}

template <bool INV>
__device__ __forceinline__ void dft2(float2* v) {
  const float2 a = v[0];
  v[0] = cadd(a, v[1]);
  v[1] = csub(a, v[1]);
}

template <bool INV>
__device__ __forceinline__ void dft4(float2& v0, float2& v1, float2& v2, float2& v3) {
  const float2 a = cadd(v0, v2), b = csub(v0, v2), c = cadd(v1, v3), d = rot90<INV>(csub(v1, v3));
  v0 = cadd(a, c);
  v1 = cadd(b, d);
  v2 = csub(a, c);
  v3 = csub(b, d);
}

template <bool INV>
__device__ __forceinline__ void dft8(float2* v) {
  // even/odd split: E = DFT4(v0,v2,v4,v6), O = DFT4(v1,v3,v5,v7); y_m = E_m + w^m O_m, y_{m+4} = E_m - w^m O_m
  float2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6];
  float2 o0 = v[1], o1 = v[3], o2 = v[5], o3 = v[7];
  dft4<INV>(e0, e1, e2, e3);
  dft4<INV>(o0, o1, o2, o3);
  const float r = 0.70710678118654752440f;
  // w = exp(sign i pi / 4)
  const float2 t1 = INV ? make_float2(r * (o1.x - o1.y), r * (o1.x + o1.y)) : make_float2(r * (o1.x + o1.y), r * (o1.y - o1.x));
  const float2 t2 = rot90<INV>(o2);
  const float2 t3 = INV ? make_float2(-r * (o3.x + o3.y), r * (o3.x - o3.y)) : make_float2(r * (o3.y - o3.x), -r * (o3.x + o3.y));
  v[0] = cadd(e0, o0);
  v[4] = csub(e0, o0);
  v[1] = cadd(e1, t1);
  v[5] = csub(e1, t1);
  v[2] = cadd(e2, t2);
  v[6] = csub(e2, t2);
  v[3] = cadd(e3, t3);
  v[7] = csub(e3, t3);
}

template <bool INV>
__device__ __forceinline__ void dft3(float2* v) {
  // y1,2 = x0 - (x1 + x2)/2 -/+ i (sqrt(3)/2)(x1 - x2) (signs of i flipped for the inverse)
  const float h = 0.86602540378443864676f;
  const float2 t1 = cadd(v[1], v[2]), t2 = csub(v[1], v[2]);
  const float2 m = make_float2(v[0].x - 0.5f * t1.x, v[0].y - 0.5f * t1.y);
  const float2 r = rot90<INV>(make_float2(h * t2.x, h * t2.y));
  v[0] = cadd(v[0], t1);
  v[1] = cadd(m, r);
  v[2] = csub(m, r);
}

template <bool INV>
__device__ __forceinline__ void dft5(float2* v) {
  // t1 = x1 + x4, t2 = x2 + x3, t3 = x1 - x4, t4 = x2 - x3;
  // y1,4 = x0 + c1 t1 + c2 t2 -/+ i (s1 t3 + s2 t4), y2,3 = x0 + c2 t1 + c1 t2 -/+ i (s2 t3 - s1 t4)
  const float c1 = 0.30901699437494742410f, c2 = -0.80901699437494742410f;
  const float s1 = 0.95105651629515357212f, s2 = 0.58778525229247312917f;
  const float2 t1 = cadd(v[1], v[4]), t2 = cadd(v[2], v[3]), t3 = csub(v[1], v[4]), t4 = csub(v[2], v[3]);
  const float2 m1 = make_float2(v[0].x + c1 * t1.x + c2 * t2.x, v[0].y + c1 * t1.y + c2 * t2.y);
  const float2 m2 = make_float2(v[0].x + c2 * t1.x + c1 * t2.x, v[0].y + c2 * t1.y + c1 * t2.y);
  const float2 n1 = rot90<INV>(make_float2(s1 * t3.x + s2 * t4.x, s1 * t3.y + s2 * t4.y));
  const float2 n2 = rot90<INV>(make_float2(s2 * t3.x - s1 * t4.x, s2 * t3.y - s1 * t4.y));
  v[0] = cadd(v[0], cadd(t1, t2));
  v[1] = cadd(m1, n1);
  v[4] = csub(m1, n1);
  v[2] = cadd(m2, n2);
  v[3] = csub(m2, n2);
}

template <int R, bool INV>
__device__ __forceinline__ void dft(float2* v) {
  if constexpr (R == 2) dft2<INV>(v);
  else if constexpr (R == 3) dft3<INV>(v);
  else if constexpr (R == 4) dft4<INV>(v[0], v[1], v[2], v[3]);
  else if constexpr (R == 5) dft5<INV>(v);
  else dft8<INV>(v);
}

// Radix of the next Stockham stage for a remaining length L = 2^a 3^b 5^c under a plan whose
// largest radix is MR: MR = 8 takes 8 while it divides, then 4 or 2, then 3s, then 5s (512 = 8.8.8);
// MR = 4 takes 4 while it divides, then 2, 3s, 5s (512 = 4.4.4.4.2). The autotuner picks the plan.
template <int L, int MR>
constexpr int next_radix() {
  if constexpr (MR >= 8)
    return L % 8 == 0 ? 8 : (L % 4 == 0 ? 4 : (L % 2 == 0 ? 2 : (L % 3 == 0 ? 3 : 5)));
  else
    return L % 4 == 0 ? 4 : (L % 2 == 0 ? 2 : (L % 3 == 0 ? 3 : 5));
}
// ---------------------------------------------------------------------------------------------
// Geometry of a strided pass: element t of column c of outer index o is at
//   o * outer_stride + c + t * elem_stride   (columns contiguous in memory).
// ---------------------------------------------------------------------------------------------
struct ColGeo {
  long long outer_stride;
  long long elem_stride;
  int cols;       // valid columns along the contiguous axis
  int outer;      // number of outer indices (over every box of a batch)
  int per_box = 0;            // outer indices per box when a batch's boxes are not one linear run
  long long box_stride = 0;   // elements between the boxes of such a batch
  __host__ __device__ long long offset(int o) const {
    return per_box ? (long long)(o / per_box) * box_stride + (long long)(o % per_box) * outer_stride
                   : (long long)o * outer_stride;
  }
  __host__ __device__ int in_box(int o) const { return per_box ? o % per_box : o; }
};

// ---------------------------------------------------------------------------------------------
// Transforms from and to global memory. The first Stockham stage takes its inputs straight from
// global memory into registers and the last one stores its outputs there, so shared memory only
// carries the exchanges between the stages (element t of line l at tile_at(t, l)): for 512 = 8.8.8
// two writes and two reads of the tile and four barriers. Nothing is staged ahead: a CTA issues all of
// a tile's loads at once, and two or more CTAs per SM overlap their loads, stages and stores.
// ---------------------------------------------------------------------------------------------
// The extra element after every 8 rows spreads the 16 lanes of a stage that runs along a line (JFAST
// below), whose writes are 8 rows apart, over all banks.
// (Tiles of 8 lines: an extra row after every 8, for the two rows that a half-warp touches.)
template <int W = TW>
__device__ __forceinline__ int tile_at(int t, int l) {
  static_assert(W == 16 || W == 8, "tiles of 16 or 8 lines");
  return W == 16 ? t * 17 + (t >> 3) + l : (t + (t >> 3)) * 8 + l;
}
constexpr size_t direct_elems(int n, int w = TW) { return w == 16 ? n * 17 + n / 8 + 1 : (n + n / 8 + 1) * 8; }
constexpr size_t direct_tile(int n, int w = TW) { return direct_elems(n, w) * sizeof(float2); }

// Threads of a CTA: two radix-8 butterflies each (tiles of 8 lines: one).
template <int L, int W>
constexpr int direct_threads() {
  constexpr int t = ((W == 16 ? L : W * L / 8) + 31) / 32 * 32;
  return t < 128 ? 128 : (t > 1024 ? 1024 : t);
}
// Lines per tile: the x pass of the Poisson solve, row passes, other column passes (narrow tiles give a small
// mesh's pass more CTAs: the five passes of a 128^3 mesh 67 us instead of 74; those of 512^3
// 3.25 ms instead of 3.02).
constexpr int XW = 8, RW = 16;
constexpr int col_width(int n) { return n <= 160 ? 8 : 16; }
// CTAs per SM that the register budget is set for (64 registers a thread).
constexpr int direct_ctas(int threads) { return 1024 / threads; }

// Butterfly q of a stage of NB per line -> (j, line): lines fastest, or (JFAST) 16 consecutive j
// fastest, for stages whose global side runs along the lines.
template <int NB, bool JFAST, int W = TW>
struct StageMap {
  static constexpr int TT = NB < 16 ? NB : 16;
  static constexpr int SPAN = JFAST ? TT * W * ((NB + TT - 1) / TT) : NB * W;
  __device__ static int j(int q) { return JFAST ? (q % TT) + TT * (q / (TT * W)) : q / W; }
  __device__ static int l(int q) { return JFAST ? (q / TT) % W : q % W; }
  __device__ static bool ok(int q) { return q < SPAN && (!JFAST || j(q) < NB); }
};

// The stages after the first: NS = product of the radices so far. store(t, l, value) takes the result.
template <int N, int NS, bool INV, int T, int TS, int MR, bool JOUT, int W, typename Store>
__device__ __forceinline__ void direct_rest(float2* sm, const float2* __restrict__ tw, const Store& store) {
  if constexpr (NS < N) {
    constexpr int R = next_radix<N / NS, MR>();
    constexpr int NB = N / R;
    constexpr bool LAST = NS * R == N;
    using Map = StageMap<NB, LAST && JOUT, W>;
    constexpr int BPT = (Map::SPAN + T - 1) / T;
    float2 v[LAST ? 1 : BPT][R];
    auto butterfly = [&](int q, float2* u) {
      const int l = Map::l(q), j = Map::j(q), k = j % NS;
#pragma unroll
      for (int r = 0; r < R; ++r) u[r] = sm[tile_at<W>(j + r * NB, l)];
#pragma unroll
      for (int r = 1; r < R; ++r) {
        float2 w = __ldg(tw + r * k * (N / (NS * R)) * TS);
        if (INV) w.y = -w.y;
        u[r] = cmul(u[r], w);
      }
      dft<R, INV>(u);
    };
    if constexpr (LAST) {
#pragma unroll
      for (int b = 0; b < BPT; ++b) {
        const int q = threadIdx.x + b * T;
        if (Map::SPAN % T != 0 || JOUT) {
          if (!Map::ok(q)) continue;
        }
        butterfly(q, v[0]);
#pragma unroll
        for (int r = 0; r < R; ++r) store(Map::j(q) + r * NS, Map::l(q), v[0][r]);
      }
    } else {
#pragma unroll
      for (int b = 0; b < BPT; ++b) {
        const int q = threadIdx.x + b * T;
        if (Map::SPAN % T == 0 || Map::ok(q)) butterfly(q, v[b]);
      }
      __syncthreads();
#pragma unroll
      for (int b = 0; b < BPT; ++b) {
        const int q = threadIdx.x + b * T;
        if (Map::SPAN % T == 0 || Map::ok(q)) {
          const int l = Map::l(q), j = Map::j(q), base = (j / NS) * NS * R + j % NS;
#pragma unroll
          for (int r = 0; r < R; ++r) sm[tile_at<W>(base + r * NS, l)] = v[b][r];
        }
      }
      __syncthreads();
      direct_rest<N, NS * R, INV, T, TS, MR, JOUT, W>(sm, tw, store);
    }
  }
}

// A whole transform of the tile's W lines: load(t, l) gives element t of line l. JIN / JOUT: the first /
// last stage's global side runs along the lines. The tile must not be in use when it starts.
template <int N, bool INV, int T, int TS, int MR, bool JIN, bool JOUT, int W = TW, typename Load, typename Store>
__device__ __forceinline__ void direct_fft(float2* sm, const float2* __restrict__ tw, const Load& load,
                                           const Store& store) {
  constexpr int R = next_radix<N, MR>();
  constexpr int NB = N / R;
  using Map = StageMap<NB, JIN, W>;
  constexpr int BPT = (Map::SPAN + T - 1) / T;
  float2 v[BPT][R];
#pragma unroll
  for (int b = 0; b < BPT; ++b) {
    const int q = threadIdx.x + b * T;
    if ((Map::SPAN % T == 0 && !JIN) || Map::ok(q)) {
#pragma unroll
      for (int r = 0; r < R; ++r) v[b][r] = load(Map::j(q) + r * NB, Map::l(q));
    }
  }
#pragma unroll
  for (int b = 0; b < BPT; ++b) {
    const int q = threadIdx.x + b * T;
    if ((Map::SPAN % T == 0 && !JIN) || Map::ok(q)) {
      const int l = Map::l(q), j = Map::j(q);
      dft<R, INV>(v[b]);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        if constexpr (R == N)
          store(j + r, l, v[b][r]);
        else
          sm[tile_at<W>(j * R + r, l)] = v[b][r];
      }
    }
  }
  if constexpr (R < N) {
    __syncthreads();
    direct_rest<N, R, INV, T, TS, MR, JOUT, W>(sm, tw, store);
  }
}

// The same with the result left in the tile (the stages after the first in place), complete for all
// threads when it returns.
template <int N, int NS, bool INV, int T, int TS, int MR, int W>
__device__ __forceinline__ void in_place_rest(float2* sm, const float2* __restrict__ tw) {
  if constexpr (NS < N) {
    constexpr int R = next_radix<N / NS, MR>();
    constexpr int NB = N / R;
    using Map = StageMap<NB, false, W>;
    constexpr int BPT = (Map::SPAN + T - 1) / T;
    float2 v[BPT][R];
#pragma unroll
    for (int b = 0; b < BPT; ++b) {
      const int q = threadIdx.x + b * T;
      if (Map::SPAN % T == 0 || Map::ok(q)) {
        const int l = Map::l(q), j = Map::j(q), k = j % NS;
#pragma unroll
        for (int r = 0; r < R; ++r) v[b][r] = sm[tile_at<W>(j + r * NB, l)];
#pragma unroll
        for (int r = 1; r < R; ++r) {
          float2 w = __ldg(tw + r * k * (N / (NS * R)) * TS);
          if (INV) w.y = -w.y;
          v[b][r] = cmul(v[b][r], w);
        }
        dft<R, INV>(v[b]);
      }
    }
    __syncthreads();
#pragma unroll
    for (int b = 0; b < BPT; ++b) {
      const int q = threadIdx.x + b * T;
      if (Map::SPAN % T == 0 || Map::ok(q)) {
        const int l = Map::l(q), j = Map::j(q), base = (j / NS) * NS * R + j % NS;
#pragma unroll
        for (int r = 0; r < R; ++r) sm[tile_at<W>(base + r * NS, l)] = v[b][r];
      }
    }
    __syncthreads();
    in_place_rest<N, NS * R, INV, T, TS, MR, W>(sm, tw);
  }
}

template <int N, bool INV, int T, int TS, int MR, int W, typename Load>
__device__ __forceinline__ void direct_fft_in_place(float2* sm, const float2* __restrict__ tw, const Load& load) {
  constexpr int R = next_radix<N, MR>();
  constexpr int NB = N / R;
  using Map = StageMap<NB, true, W>;
  constexpr int BPT = (Map::SPAN + T - 1) / T;
  float2 v[BPT][R];
#pragma unroll
  for (int b = 0; b < BPT; ++b) {
    const int q = threadIdx.x + b * T;
    if (Map::ok(q)) {
#pragma unroll
      for (int r = 0; r < R; ++r) v[b][r] = load(Map::j(q) + r * NB, Map::l(q));
    }
  }
#pragma unroll
  for (int b = 0; b < BPT; ++b) {
    const int q = threadIdx.x + b * T;
    if (Map::ok(q)) {
      dft<R, INV>(v[b]);
#pragma unroll
      for (int r = 0; r < R; ++r) sm[tile_at<W>(Map::j(q) * R + r, Map::l(q))] = v[b][r];
    }
  }
  __syncthreads();
  in_place_rest<N, R, INV, T, TS, MR, W>(sm, tw);
}

// ---------------------------------------------------------------------------------------------
// The passes on the direct transforms: one tile (of 16 lines) per CTA.
// ---------------------------------------------------------------------------------------------
// A CTA's tile of a strided pass: W adjacent columns of one outer index.
template <int W>
struct ColTile {
  long long base;  // element 0 of line 0
  int valid, outer, col;
  __device__ ColTile(const ColGeo& g, int tile) {
    const int tiles = (g.cols + W - 1) / W;
    outer = tile / tiles;
    col = (tile % tiles) * W;
    valid = min(W, g.cols - col);
    base = g.offset(outer) + col;
  }
};
template <int W>
int col_tile_count(const ColGeo& g) {
  return g.outer * ((g.cols + W - 1) / W);
}
// Stores of the strided passes of meshes from STREAM_MESH on: evict-first (STREAM). Left in L2 as ordinary stores,
// the strided lines of a 512^3 mesh reach DRAM 1.3 to 1.6 times each.
template <bool STREAM>
__device__ __forceinline__ void put(float2* p, float2 v) {
  if constexpr (STREAM)
    __stcs(p, v);
  else
    *p = v;
}

// c2c pass over a strided axis; block -> (comp, tile).
template <int N, bool INV, int T, int MR, bool STREAM>
__global__ void __launch_bounds__(T, direct_ctas(T)) k_cols(float2* data, long long comp_stride, ColGeo g,
                                                            const float2* __restrict__ tw) {
  extern __shared__ float2 smem[];
  constexpr int W = col_width(N);
  const int per_comp = g.outer * ((g.cols + W - 1) / W);
  const ColTile<W> c(g, blockIdx.x % per_comp);
  const int es = (int)g.elem_stride;
  float2* d = data + (long long)(blockIdx.x / per_comp) * comp_stride + c.base;
  direct_fft<N, INV, T, 1, MR, false, false, W>(
      smem, tw, [&](int t, int l) { return l < c.valid ? d[t * es + l] : make_float2(0.0f, 0.0f); },
      [&](int t, int l, float2 v) {
        if (l < c.valid) put<STREAM>(d + t * es + l, v);
      });
}

// c2c pass over contiguous rows (the z lines of a full complex n^3 array).
template <int N, bool INV, int T, int MR>
__global__ void __launch_bounds__(T, direct_ctas(T)) k_rows(float2* data, int rows, const float2* __restrict__ tw) {
  extern __shared__ float2 smem[];
  const int row0 = blockIdx.x * RW, valid = min(RW, rows - row0);
  float2* d = data + (size_t)row0 * N;
  direct_fft<N, INV, T, 1, MR, true, true, RW>(
      smem, tw, [&](int t, int l) { return l < valid ? d[l * N + t] : make_float2(0.0f, 0.0f); },
      [&](int t, int l, float2 v) {
        if (l < valid) d[l * N + t] = v;
      });
}

// z pass, forward: real rows of length N -> N/2+1 complex each (rows of the padded half spectrum), as an
// N/2-point complex transform of z[m] = x[2m] + i x[2m+1]. Input: f32 delta, or the u64 fixed-point mass
// mesh (c = fx * 2^-k in f32, delta = c / mean - 1), converted on its way into the first stage.
template <int N, int T, int MR>
__global__ void __launch_bounds__(T, direct_ctas(T)) k_rows_r2c(const float* __restrict__ delta,
                                                                const unsigned long long* __restrict__ fx,
                                                                float inv_scale, float mean, float inv_mean,
                                                                float2* __restrict__ spec, int rows,
                                                                const float2* __restrict__ tw) {
  extern __shared__ float2 smem[];
  constexpr int M = N / 2, NH = N / 2 + 1, NHP = half_row(N);
  const int row0 = blockIdx.x * RW, valid = min(RW, rows - row0);
  if (fx) {
    const unsigned long long* src = fx + (size_t)row0 * N;
    direct_fft_in_place<M, false, T, 2, MR, RW>(smem, tw, [&](int m, int l) {
      if (l >= valid) return make_float2(0.0f, 0.0f);
      const ulonglong2 u = __ldg(reinterpret_cast<const ulonglong2*>(src + l * N + 2 * m));
      const float c0 = __fmul_rn(__ull2float_rn(u.x), inv_scale);
      const float c1 = __fmul_rn(__ull2float_rn(u.y), inv_scale);
      // (a mean that is a power of two has an exact reciprocal: the same quotients without a division)
      if (inv_mean != 0.0f)
        return make_float2(__fsub_rn(__fmul_rn(c0, inv_mean), 1.0f), __fsub_rn(__fmul_rn(c1, inv_mean), 1.0f));
      return make_float2(__fsub_rn(__fdiv_rn(c0, mean), 1.0f), __fsub_rn(__fdiv_rn(c1, mean), 1.0f));
    });
  } else {
    const float* src = delta + (size_t)row0 * N;
    direct_fft_in_place<M, false, T, 2, MR, RW>(smem, tw, [&](int m, int l) {
      return l < valid ? __ldg(reinterpret_cast<const float2*>(src + l * N + 2 * m)) : make_float2(0.0f, 0.0f);
    });
  }
  // X[k] = (Z[k] + conj(Z[M-k]))/2 + w^k (Z[k] - conj(Z[M-k]))/(2i), w = exp(-2 pi i / N)
  for (int q = threadIdx.x; q < StageMap<NH, true, RW>::SPAN; q += T) {
    const int k = StageMap<NH, true, RW>::j(q), l = StageMap<NH, true, RW>::l(q);
    if (l >= valid || k >= NH) continue;
    // Z is M-periodic: Z[M] = Z[0] (k runs over 0..M)
    const float2 zk = smem[tile_at<RW>(k == M ? 0 : k, l)];
    const float2 zm = smem[tile_at<RW>(k == 0 ? 0 : M - k, l)];
    const float2 fe = make_float2(0.5f * (zk.x + zm.x), 0.5f * (zk.y - zm.y));
    const float2 fo = make_float2(0.5f * (zk.y + zm.y), -0.5f * (zk.x - zm.x));
    spec[(size_t)(row0 + l) * NHP + k] = cadd(fe, cmul(__ldg(tw + k), fo));
  }
}

// z pass, inverse: N/2+1 complex per row -> N real values times scale, as an N/2-point complex
// inverse transform of Z'[k] = (X[k] + conj(X[M-k])) + i (X[k] - conj(X[M-k])) conj(w^k), whose output is
// x[2m] + i x[2m+1]; block -> (comp, row tile). The first stage's inputs Z'[k] are formed from X[k] and
// X[M-k] as they are loaded (every row is in L1 for its second reading).
template <int N, int T, int MR>
__global__ void __launch_bounds__(T, direct_ctas(T)) k_rows_c2r(const float2* __restrict__ spec, long long comp_stride,
                                                                float* __restrict__ out0, float* __restrict__ out1,
                                                                float* __restrict__ out2, float scale, int rows,
                                                                const float2* __restrict__ tw) {
  extern __shared__ float2 smem[];
  constexpr int M = N / 2, NHP = half_row(N);
  const int row_tiles = (rows + RW - 1) / RW;
  const int comp = blockIdx.x / row_tiles, row0 = (blockIdx.x % row_tiles) * RW, valid = min(RW, rows - row0);
  const float2* sp = spec + (long long)comp * comp_stride + (size_t)row0 * NHP;
  float2* out = reinterpret_cast<float2*>((comp == 0 ? out0 : (comp == 1 ? out1 : out2)) + (size_t)row0 * N);
  direct_fft<M, true, T, 2, MR, true, true, RW>(
      smem, tw,
      [&](int k, int l) {
        if (l >= valid) return make_float2(0.0f, 0.0f);
        // the upper of the pair k, M - k by w^(M-k) = -conj(w^k)
        const int lo = min(k, M - k);
        float2 x = __ldg(sp + l * NHP + lo), y = __ldg(sp + l * NHP + M - lo);
        // X[0] and X[M] enter the real output through their real parts only (as in Re of a
        // full complex inverse); their imaginary parts are round-off of the Hermitian planes.
        if (lo == 0) x.y = y.y = 0.0f;
        const float2 w = __ldg(tw + lo);
        if (k == lo) {
          const float2 a = cadd(x, conjf2(y)), b = csub(x, conjf2(y));
          const float2 bw = cmul(b, conjf2(w));
          return make_float2(a.x - bw.y, a.y + bw.x);
        }
        const float2 a = cadd(y, conjf2(x)), b = csub(y, conjf2(x));
        const float2 bw = cmul(b, make_float2(-w.x, -w.y));
        return make_float2(a.x - bw.y, a.y + bw.x);
      },
      [&](int m, int l, float2 v) {
        if (l < valid) out[l * (N / 2) + m] = make_float2(__fmul_rn(v.x, scale), __fmul_rn(v.y, scale));
      });
}

// x pass of the Poisson solve for XW kz columns at fixed ky: forward c2c along x, the Green's function of
// poisson.rs:52-74 (phi_k into a second tile), then the inverse transforms
//   of -i k_x phi (the x component) to slot 0;
//   of phi to slot 1, from which the y pass forms the y and z components: -i k_y and -i k_z are
//   constant along the line, so the factors commute with the transform.
// The gradient factor is the reference's (phi * (0 - i k_a), poisson.rs:70); for y and z it
// multiplies the transformed phi instead, which differs only in round-off.
// (Two tiles of 16 lines leave one CTA per SM; phi_k kept in slot 1 instead went to DRAM and back: 1.12 ms at
// n = 512, now 0.72.)
template <int N, int T, int MR, bool STREAM>
__global__ void __launch_bounds__(T, direct_ctas(T)) k_x_poisson(float2* spec, long long comp_stride, ColGeo g,
                                                                 PoissonParams pp, const float* __restrict__ deconv,
                                                                 const float2* __restrict__ tw) {
  extern __shared__ float2 smem[];
  float2* phi = smem + direct_elems(N, XW);
  const ColTile<XW> c(g, blockIdx.x);
  const int es = (int)g.elem_stride, iy = g.in_box(c.outer);
  float2* s0 = spec + c.base;
  float2* s1 = s0 + comp_stride;
  const float prefactor = pp.prefactor_dev ? *pp.prefactor_dev : pp.prefactor;
  const float ky = wavenumber(iy, N, pp.two_pi_over_l);
  direct_fft<N, false, T, 1, MR, false, false, XW>(
      smem, tw, [&](int t, int l) { return l < c.valid ? s0[t * es + l] : make_float2(0.0f, 0.0f); },
      [&](int t, int l, float2 v) {
        const int iz = c.col + l;
        const float kx = wavenumber(t, N, pp.two_pi_over_l), kz = wavenumber(min(iz, N / 2), N, pp.two_pi_over_l);
        float k2 = -0.0f;
        k2 = __fadd_rn(k2, __fmul_rn(kx, kx));
        k2 = __fadd_rn(k2, __fmul_rn(ky, ky));
        k2 = __fadd_rn(k2, __fmul_rn(kz, kz));
        if (k2 == 0.0f || l >= c.valid) {
          v = make_float2(0.0f, 0.0f);
        } else {
          // phi_k = delta_k * (-prefactor / k^2 * exp(-k^2 r_s^2)), k = 0 skipped (left zero)
          const float filter = expf(__fmul_rn(__fmul_rn(-k2, pp.r_split), pp.r_split));
          float sc = __fmul_rn(__fdiv_rn(-prefactor, k2), filter);
          if (deconv) sc = __fmul_rn(sc, __fmul_rn(__fmul_rn(deconv[t], deconv[iy]), deconv[iz]));
          v = make_float2(__fmul_rn(v.x, sc), __fmul_rn(v.y, sc));
        }
        phi[tile_at<XW>(t, l)] = v;
      });
  __syncthreads();  // phi_k of the tile is complete, the exchange tile free
  direct_fft<N, true, T, 1, MR, false, false, XW>(
      smem, tw,
      [&](int t, int l) {
        // -i k_x phi: re = phi.re*0 - phi.im*(-k_x), im = phi.re*(-k_x) + phi.im*0
        const float2 v = phi[tile_at<XW>(t, l)];
        const float nk = -wavenumber(t, N, pp.two_pi_over_l);
        return make_float2(__fsub_rn(__fmul_rn(v.x, 0.0f), __fmul_rn(v.y, nk)),
                           __fadd_rn(__fmul_rn(v.x, nk), __fmul_rn(v.y, 0.0f)));
      },
      [&](int t, int l, float2 v) {
        if (l < c.valid) put<STREAM>(s0 + t * es + l, v);
      });
  __syncthreads();
  direct_fft<N, true, T, 1, MR, false, false, XW>(
      smem, tw, [&](int t, int l) { return phi[tile_at<XW>(t, l)]; },
      [&](int t, int l, float2 v) {
        if (l < c.valid) put<STREAM>(s1 + t * es + l, v);
      });
}

// Inverse y pass of the three components, tile by tile: the x component (slot 0), and from the
// x-transformed potential (slot 1) the z component -i k_z phi (slot 2), then the y component -i k_y
// phi over the potential.
template <int N, int T, int MR, bool STREAM>
__global__ void __launch_bounds__(T, direct_ctas(T)) k_y_gradient(float2* spec, long long comp_stride, ColGeo g,
                                                                  PoissonParams pp, const float2* __restrict__ tw) {
  extern __shared__ float2 smem[];
  constexpr int W = col_width(N);
  const ColTile<W> c(g, blockIdx.x);
  const int es = (int)g.elem_stride;
  float2* s0 = spec + c.base;
  float2 *s1 = s0 + comp_stride, *s2 = s1 + comp_stride;
  auto times = [&](float2 p, float nk) {  // -i k phi with nk = -k, as k_x_poisson
    return make_float2(__fsub_rn(__fmul_rn(p.x, 0.0f), __fmul_rn(p.y, nk)),
                       __fadd_rn(__fmul_rn(p.x, nk), __fmul_rn(p.y, 0.0f)));
  };
  direct_fft<N, true, T, 1, MR, false, false, W>(
      smem, tw, [&](int t, int l) { return l < c.valid ? s0[t * es + l] : make_float2(0.0f, 0.0f); },
      [&](int t, int l, float2 v) {
        if (l < c.valid) put<STREAM>(s0 + t * es + l, v);
      });
  __syncthreads();
  direct_fft<N, true, T, 1, MR, false, false, W>(
      smem, tw,
      [&](int t, int l) {
        return l < c.valid ? times(s1[t * es + l], -wavenumber(c.col + l, N, pp.two_pi_over_l)) : make_float2(0.0f, 0.0f);
      },
      [&](int t, int l, float2 v) {
        if (l < c.valid) put<STREAM>(s2 + t * es + l, v);
      });
  __syncthreads();
  direct_fft<N, true, T, 1, MR, false, false, W>(
      smem, tw,
      [&](int t, int l) {
        return l < c.valid ? times(s1[t * es + l], -wavenumber(t, N, pp.two_pi_over_l)) : make_float2(0.0f, 0.0f);
      },
      [&](int t, int l, float2 v) {
        if (l < c.valid) put<STREAM>(s1 + t * es + l, v);
      });
}

// ---------------------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------------------
// Mesh sizes with compiled transforms: powers of two 4..1024 and the 2^a 3^b 5^c sizes below.
#define CPM_FFT_SIZES(X) \
  X(4) X(8) X(16) X(32) X(48) X(64) X(80) X(96) X(128) X(160) X(192) X(256) X(320) X(384) X(512) X(1024)

bool fft_supported(int n) {
  switch (n) {
#define CPM_CASE(N) case N:
    CPM_FFT_SIZES(CPM_CASE)
#undef CPM_CASE
    return true;
    default:
      return false;
  }
}
bool poisson_supported(int n) { return fft_supported(n); }

const char* fft_sizes_text() {
  return "4, 8, 16, 32, 48, 64, 80, 96, 128, 160, 192, 256, 320, 384, 512 or 1024";
}

size_t half_spectrum_elems(int n) { return (size_t)n * n * (size_t)half_row(n); }

cudaError_t fft_plan_init(FftPlan& p, int n) {
  if (p.n == n && p.twiddle.p && p.deconv.p) return cudaSuccess;
  p.n = n;
  std::vector<float2> tw(n);
  const double two_pi = 6.283185307179586476925286766559;
  for (int m = 0; m < n; ++m) {
    const double a = -two_pi * (double)m / (double)n;
    tw[m] = make_float2((float)std::cos(a), (float)std::sin(a));
  }
  // CIC deconvolution per axis: 1 / W(k)^2 with W = sinc^2(pi m / n) (deposit and gather)
  std::vector<float> dc(n);
  for (int i = 0; i < n; ++i) {
    const int m = i <= n / 2 ? i : i - n;
    const double x = 3.14159265358979323846 * (double)m / (double)n;
    const double s = m == 0 ? 1.0 : std::sin(x) / x;
    dc[i] = (float)(1.0 / (s * s * s * s));
  }
  cudaError_t e = ensure(p.twiddle, n * sizeof(float2));
  if (e == cudaSuccess) e = ensure(p.deconv, n * sizeof(float));
  if (e == cudaSuccess) e = cudaMemcpy(p.twiddle.p, tw.data(), n * sizeof(float2), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(p.deconv.p, dc.data(), n * sizeof(float), cudaMemcpyHostToDevice);
  return e;
}

void fft_plan_free(FftPlan& p) {
  release(p.twiddle);
  release(p.deconv);
  p.n = 0;
}

// 1 / x when x is a power of two (whose reciprocal is exact), else 0.
static float exact_inverse(float x) {
  int e = 0;
  return x > 1e-30f && x < 1e30f && std::frexp(x, &e) == 0.5f ? 1.0f / x : 0.0f;
}

// Meshes whose strided passes store evict-first, by measurement and not by the size of L2 (126 MB; a spectrum is 69 MB
// at 256, 231 at 384, 545 at 512): the five passes of 512^3 3.48 -> 3.19 ms when it was introduced, but 384^3
// 1.75 -> 1.81 and 320^3 1.02 -> 1.05; 256^3 would gain 1.5 % (0.400 -> 0.394).
constexpr int STREAM_MESH = 512;

// One tile per CTA.
template <typename K, typename... Args>
static void launch_tiles(K kernel, int threads, size_t smem, int tiles, cudaStream_t s, Args... args) {
  if (smem > 48 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  count_launch();
  kernel<<<tiles, threads, smem, s>>>(args...);
}

template <int N, int MR>
static void cols_direct(float2* data, long long comp_stride, int ncomp, ColGeo g, int inverse, const float2* tw,
                        cudaStream_t s) {
  constexpr int T = direct_threads<N, col_width(N)>();
  constexpr bool ST = N >= STREAM_MESH;
  launch_tiles(inverse ? k_cols<N, true, T, MR, ST> : k_cols<N, false, T, MR, ST>, T, direct_tile(N, col_width(N)),
               ncomp * col_tile_count<col_width(N)>(g), s, data, comp_stride, g, tw);
}

template <int N>
static void fft3_c2c_n(float2* data, int inverse, const float2* tw, cudaStream_t s) {
  constexpr int T = direct_threads<N, RW>();
  const long long n = N;
  const int rows = N * N;
  launch_tiles(inverse ? k_rows<N, true, T, 8> : k_rows<N, false, T, 8>, T, direct_tile(N, RW), (rows + RW - 1) / RW, s,
               data, rows, tw);
  // y lines: elements n apart, columns along z adjacent, outer = x
  cols_direct<N, 8>(data, 0, 1, ColGeo{n * n, n, N, N}, inverse, tw, s);
  // x lines: elements n*n apart, outer = y
  cols_direct<N, 8>(data, 0, 1, ColGeo{n, n * n, N, N}, inverse, tw, s);
}

void launch_fft3_c2c(const FftPlan& p, float2* data, int inverse, cudaStream_t s) {
  const float2* tw = static_cast<const float2*>(p.twiddle.p);
  switch (p.n) {
#define CPM_CASE(N) \
  case N: fft3_c2c_n<N>(data, inverse, tw, s); break;
    CPM_FFT_SIZES(CPM_CASE)
#undef CPM_CASE
    default: break;
  }
}

// Forward R2C n^3 transform of delta (f32, or the u64 fixed-point mass mesh converted to
// delta = c/mean - 1 on load) into the padded half spectrum: z, then y, then x lines.
template <int N>
static void r2c3_n(const FftPlan& p, const float* delta, const unsigned long long* fx, int fx_shift, float mean,
                   float2* spec, cudaStream_t s) {
  const float2* tw = static_cast<const float2*>(p.twiddle.p);
  constexpr int M = N / 2, NH = N / 2 + 1, NHP = half_row(N);
  const long long n = N;
  const int rows = N * N;
  {
    constexpr int T = direct_threads<M, RW>();
    launch_tiles(k_rows_r2c<N, T, 8>, T, direct_tile(M, RW), (rows + RW - 1) / RW, s, delta, fx, std::ldexp(1.0f, -fx_shift),
                 mean, exact_inverse(mean), spec, rows, tw);
  }
  cols_direct<N, 8>(spec, 0, 1, ColGeo{n * NHP, NHP, NH, N}, 0, tw, s);  // y lines, outer = x
  cols_direct<N, 8>(spec, 0, 1, ColGeo{NHP, n * NHP, NH, N}, 0, tw, s);  // x lines, outer = y
}

template <int N, int MR>
static void poisson_n(const FftPlan& p, const PoissonParams& pp, const float* delta, const unsigned long long* fx,
                      int fx_shift, float mean, float2* spec, float* gx, float* gy_out, float* gz, cudaStream_t s) {
  const float2* tw = static_cast<const float2*>(p.twiddle.p);
  const float* deconv = pp.deconvolve ? static_cast<const float*>(p.deconv.p) : nullptr;
  constexpr int M = N / 2, NH = N / 2 + 1, NHP = half_row(N);
  const long long n = N;
  const int nb = pp.boxes > 1 ? pp.boxes : 1;  // a batch of nb meshes, one after another
  const long long comp = nb * n * n * NHP;     // elements per half spectrum (every box)
  const int rows = nb * N * N;
  // Slot 0 holds the forward spectrum; every pass reads a tile of it before it writes the same tile of
  // slots 0..2, and tiles are disjoint, so the update in place is safe. y lines: columns along kz
  // adjacent, outer = x (the x planes of a batch's boxes form one run); x lines: outer = y.
  const ColGeo gy{n * NHP, NHP, NH, nb * N};
  const ColGeo gxl{NHP, n * NHP, NH, nb * N, nb > 1 ? N : 0, n * n * NHP};
  constexpr int TM = direct_threads<M, RW>(), TX = direct_threads<N, XW>(), TY = direct_threads<N, col_width(N)>();
  const int rt = (rows + RW - 1) / RW;
  constexpr bool ST = N >= STREAM_MESH;
  launch_tiles(k_rows_r2c<N, TM, MR>, TM, direct_tile(M, RW), rt, s, delta, fx, std::ldexp(1.0f, -fx_shift), mean,
               exact_inverse(mean), spec, rows, tw);
  cols_direct<N, MR>(spec, 0, 1, gy, 0, tw, s);
  launch_tiles(k_x_poisson<N, TX, MR, ST>, TX, 2 * direct_tile(N, XW), col_tile_count<XW>(gxl), s, spec, comp, gxl, pp,
               deconv, tw);
  launch_tiles(k_y_gradient<N, TY, MR, ST>, TY, direct_tile(N, col_width(N)), col_tile_count<col_width(N)>(gy), s, spec,
               comp, gy, pp, tw);
  launch_tiles(k_rows_c2r<N, TM, MR>, TM, direct_tile(M, RW), 3 * rt, s, spec, comp, gx, gy_out, gz, pp.scale, rows,
               tw);
}

void launch_r2c3(const FftPlan& p, const float* delta, const unsigned long long* fx, int fx_shift, float mean,
                 float2* spec, cudaStream_t s) {
  switch (p.n) {
#define CPM_CASE(N) \
  case N: r2c3_n<N>(p, delta, fx, fx_shift, mean, spec, s); break;
    CPM_FFT_SIZES(CPM_CASE)
#undef CPM_CASE
    default: break;
  }
}

void launch_poisson(const FftPlan& p, const PoissonParams& pp, const float* delta, const unsigned long long* fx,
                    int fx_shift, float mean, float2* spec, float* gx, float* gy, float* gz, cudaStream_t s) {
  switch (p.n) {
#define CPM_CASE(N)                                                          \
  case N:                                                                    \
    if (p.max_radix == 4)                                                    \
      poisson_n<N, 4>(p, pp, delta, fx, fx_shift, mean, spec, gx, gy, gz, s); \
    else                                                                     \
      poisson_n<N, 8>(p, pp, delta, fx, fx_shift, mean, spec, gx, gy, gz, s); \
    break;
    CPM_FFT_SIZES(CPM_CASE)
#undef CPM_CASE
    default: break;
  }
}

}  // namespace cpm
