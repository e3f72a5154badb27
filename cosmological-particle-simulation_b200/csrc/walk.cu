// walk.cu — the short-range tree walk (tree.rs:264-323) and its pair kernel (tree.rs:54-66).
//
// Traversal. One warp walks for a group of 32 consecutive sorted particles (one per lane); warps
// take groups from a common counter (small launches give a group to a team of warps). The stack
// holds batches: the children of one opened node (contiguous in the node arrays), with the mask of
// the lanes that walk them. The unit of work is a step of up to 32 nodes, one per lane: the top
// batch and, while the stack is shallow (which bounds its depth), the batches below it as long as
// they fit. Lane c copies node c's three 16-byte records (centre and half, centre of mass and mass,
// link) into shared memory with cp.async, in flight during the previous step's direct sums.
//
// The reference's rules per particle (tree.rs:264-310) are: prune a node when
// |min_image(centre - x)| > r_cut + sqrt(3) half; sum its particles directly when its octant-0
// child is missing (`children[0] == NO_CHILD`, which includes leaves); else accept its centre of
// mass when 2 half < theta |min_image(com - x)|, or open it. What of this holds for all 32 particles
// lane c decides once, for node c, from the bounding box of the group: nodes beyond every lane's
// prune radius, direct nodes whose cube is beyond r_cut of the box, and nodes so large that no lane
// can accept them need no test per particle. Only the remaining inner nodes are put to every lane,
// which accepts by its own separately rounded f32 operations and exact minimum image (the opening
// test, evaluated on squares, falls back to the reference's square-root form whenever the two sides
// are within 1e-5). A lane that prunes a node without accepting it simply goes on with the others:
// whatever lies below it prunes as well, or finds beyond r_cut. A node whose children are all direct
// (`flat`, marked by the build) is not opened: nothing below it can be accepted, so the lanes that do
// not accept it sum its whole range. So a lane's set of interactions is the one its own reference
// walk visits; only the order in which it adds them differs.
//
// Direct sums. The particles of a step's direct and flat nodes, concatenated, are fetched 64 at a
// time; those within r_cut of the group's box (about a quarter to a half) join a window of up to 448
// sources in shared memory. A full window is summed in two phases: per word of 32 sources every lane marks
// the sources within r_cut of it (r^2 - r_cut^2 by f32x2 fused multiply-adds, the sign bits shifted into
// a mask), then evaluates the pair force for its marked sources, four per iteration, walking through
// its own words, so that lanes do not idle on sources outside the cutoff of other lanes. The mask is
// a superset by a margin of 2e-6; sources that close to the cutoff are settled by the reference's own
// r^2 in the second phase. Words whose sources may need a periodic image form the nearest image.
//
// What bounds it: instruction issue (66 % of the slots early in a run, 70 % in clustered states, at 5 warps per
// scheduler; FMA pipe 33 and 43 %, DRAM idle). Per group at 128^3 particles / 256^3 mesh near the initial state: traversal 6.5, fetching
// 5.2, marking 5.1 and pair forces 9.0 thousand warp instructions, of 88 pairs per particle; in a
// clustered state 12.7, 5.5, 9.4 and 24.8 thousand, of 325 pairs. Testing every particle against
// every direct node and chunk of 32 sources, without the group's decisions, the culled window and
// the flat nodes, this walk took 4.38 and 6.06 ms there; now 2.03 and 4.28 (256^3 / 512^3: 31.1,
// now 15.4 ms).
//
// Pair force. f = -K m S(r) / (r^2 + eps^2)^{3/2}, S(r) = erfc(u) + (2/sqrt(pi)) u e^{-u^2},
// u = r / (2 r_s). S is evaluated as e^{-u^2} R(u) with R(u) = erfcx(u) + 2u/sqrt(pi), a smooth
// function fitted on the host for each split: Chebyshev interpolation in double precision
// (erfc from the C library), converted to a degree-12 polynomial in x in [-1, 1] and evaluated
// by f32 Horner — about 2e-7 relative over the range of the leaf pairs (checked by
// cpm_walk_kernel_fit_error). For accepted nodes e^{-u^2} takes the FMA-exact residual of u*u, with
// exp2f and rsqrtf; for the direct pairs u^2 comes from r^2 without a root, and e^{-u^2}, r and
// (r^2 + eps^2)^{-3/2} from the hardware approximations (ex2, rsqrt; about 2^-22 relative). The
// coupling K multiplies each particle's sum once at the end. Against the reference's erfcf-based S
// the pair force differs by a few 1e-7 relative; the 1e-5 RMS parity tests cover the sum.
#include <algorithm>
#include <cmath>
#include <string>
#include <type_traits>
#include <vector>

#include "cpm_host.h"
#include "cpm_internal.cuh"

namespace cpm {

constexpr int SLOTS = 32;     // nodes per step of a warp's walk (one per lane)
constexpr int MERGE_SP = 48;  // stack entries are merged into one step only while the stack is this shallow
// Stack bound: a merging step starts at depth <= MERGE_SP and pushes at most SLOTS entries; from
// there single-entry steps (depth first) keep at most 7 unvisited sibling entries per tree level
// below, plus the 8 just pushed.
constexpr int STACK_CAP = MERGE_SP + SLOTS + 7 * KEY_LEVELS + 8;
constexpr int WINDOW = 448;   // direct-sum sources collected before they are summed (words of 32)
// Groups are walked by teams of 2 or 4 warps while that keeps a launch within WALK_FILL warps (about
// five rounds of the chip): the few groups of a small launch leave warps idle, and its time is that
// of its slowest group. Walk of 91,125 clustered particles (2848 groups, through the function call)
// 0.888 ms with single warps, 0.500 with teams of 4; of 262,144 (8192 groups) 0.426 with single warps, 0.505 with teams of 2,
// whose warps each repeat the traversal.
constexpr size_t WALK_FILL = 148 * 96;
// A batch of boxes takes the team of one of them (the order of a particle's terms is then that of the box's own
// simulation) as long as its warps fill the chip's rounds no more than eight times over; a larger batch takes single warps, whose
// sums differ by rounding. A step of 64 boxes of 32^3 (262,144 warps in teams) takes 8.7 ms in its early states and 9.5 in
// its late ones with teams, 4.5 and 5.5 with single warps; of 16 boxes of 48^3 (221,184) 5.9 and 8.3, and 3.1 and 4.8. The
// walk before there were teams took 8.5 and 8.4, and 6.5 and 7.2: from about the line on (8 boxes of 48^3, 3.0 and
// 4.3, before 3.5 and 4.1) the repeated traversals cost more than teams had brought.
constexpr size_t BATCH_FILL = 8 * WALK_FILL;
constexpr int WALK_WARPS_PER_SM = 20;  // resident warps the register budget is set for
constexpr int STAGE = 64;     // candidate sources fetched at a time, two per lane
constexpr uint32_t FIRST_BITS = 29;  // a stack entry: first node (29 bits) | (count - 1) << 29
constexpr int FIT_DEG = 12;
constexpr int FAR_PIECES_MAX = 8;
constexpr double U_NEGLIGIBLE = 9.0;  // S(9) ~ 1e-34: contributions beyond are below f32 resolution

struct SFit {
  float scale0, offset0, umax0;  // piece 0: x = u * scale0 + offset0 for u <= umax0
  float c0[FIT_DEG + 1];
  float far_lo, far_w, far_inv_w, far_hi;  // pieces of width far_w covering [far_lo, far_hi]
  int far_n;
};

// The constants of the direct-sum pair force, duplicated for the packed (two pairs per
// instruction) evaluation.
struct PairConst2 {
  float2 tiny;        // added to r^2 under the reciprocal square root, so that r = 0 stays 0
  float2 scale0, offset0;  // fit variable x = r * scale0 + offset0
  float2 c0[FIT_DEG + 1];
  float2 exp_scale;   // -log2(e) / (2 r_s)^2
  float2 eps2;        // softening^2
};

// The same for the ordered walk.
struct OrderedConst {
  float2 tiny, inv_two_rs, scale0, offset0;
  float2 c0[FIT_DEG + 1];
  float2 neg_log2e, eps2, neg_m;
};

struct WalkParams {
  float box;
  float guard;  // |x| below this: round(x / L) == 0 exactly
  float r_cut;
  float cut2;   // r_cut * r_cut
  float cut_lo, cut_hi;  // cut2 -+ 2e-6: below and above every rounding of r^2
  float cut_image;       // cut2 with a margin for the rounding of a nearest image
  float inv_box;         // 1 / L
  float cull2;           // cut2 with a margin for the tests against the warp's box
  float wrap_lo, wrap_hi;  // |x| in (wrap_lo, wrap_hi): round(x / L) is +-1 exactly
  int fit_covers;        // every direct pair lies in piece 0 of the fit
  float theta;
  float theta2;  // theta * theta (f32), for the squared form of the opening test
  float inv_two_rs;
  float eps2;   // softening^2
  float k;      // Newtonian coupling
  uint32_t n_box;  // batch of boxes: particles per box (multiple of 32); a warp starts at root i / n_box
  SFit fit;
  PairConst2 p2;
  OrderedConst ordered;
};

// ------------------------------------------------------------------ host: the fit of R(u)

static double r_exact(double u) { return std::exp(u * u) * std::erfc(u) + 2.0 * u / std::sqrt(M_PI); }

// Degree-D interpolant of R on [lo, hi] at Chebyshev nodes, as monomial coefficients in x in [-1, 1].
static void fit_piece(double lo, double hi, float* coef) {
  const int D = FIT_DEG, M = D + 1;
  std::vector<double> fx(M), c(M, 0.0);
  for (int k = 0; k < M; ++k) {
    const double x = std::cos(M_PI * (k + 0.5) / M);
    fx[k] = r_exact(lo + (x + 1.0) * 0.5 * (hi - lo));
  }
  for (int j = 0; j < M; ++j) {
    double s = 0.0;
    for (int k = 0; k < M; ++k) s += fx[k] * std::cos(M_PI * j * (k + 0.5) / M);
    c[j] = (j == 0 ? 1.0 : 2.0) * s / M;
  }
  // Chebyshev -> monomial: T_0 = 1, T_1 = x, T_{j+1} = 2x T_j - T_{j-1}
  std::vector<std::vector<double>> T(M, std::vector<double>(M, 0.0));
  T[0][0] = 1.0;
  if (M > 1) T[1][1] = 1.0;
  for (int j = 1; j + 1 < M; ++j)
    for (int p = 0; p < M; ++p) T[j + 1][p] = (p ? 2.0 * T[j][p - 1] : 0.0) - T[j - 1][p];
  for (int p = 0; p < M; ++p) {
    double s = 0.0;
    for (int j = 0; j < M; ++j) s += c[j] * T[j][p];
    coef[p] = (float)s;
  }
}

static float horner_host(const float* c, float x) {
  float acc = c[FIT_DEG];
  for (int j = FIT_DEG - 1; j >= 0; --j) acc = std::fma(acc, x, c[j]);
  return acc;
}

// Piece 0 covers the leaf pairs (u <= r_cut / (2 r_s), at most 2.5 so that degree 12 keeps ~2e-7);
// further pieces of width <= 2.25 reach u = 9.
static SFit make_fit(float r_split, float r_cut, std::vector<float>& far) {
  SFit f{};
  const double u0 = std::min(2.5, std::max(0.25, (double)r_cut / (2.0 * (double)r_split) * 1.0001));
  fit_piece(0.0, u0, f.c0);
  f.umax0 = (float)u0;
  f.scale0 = (float)(2.0 / u0);
  f.offset0 = -1.0f;
  const double rest = U_NEGLIGIBLE - u0;
  f.far_n = rest > 0 ? std::min(FAR_PIECES_MAX, (int)std::ceil(rest / 2.25)) : 0;
  f.far_lo = (float)u0;
  f.far_hi = (float)U_NEGLIGIBLE;
  const double w = f.far_n ? rest / f.far_n : 1.0;
  f.far_w = (float)w;
  f.far_inv_w = (float)(1.0 / w);
  far.assign((size_t)std::max(f.far_n, 1) * (FIT_DEG + 1), 0.0f);
  for (int p = 0; p < f.far_n; ++p) fit_piece(u0 + p * w, u0 + (p + 1) * w, far.data() + (size_t)p * (FIT_DEG + 1));
  return f;
}

// Host twin of the device evaluation of R (same coefficients, same f32 Horner) for the self-check.
static float r_fit_host(const SFit& f, const std::vector<float>& far, float u) {
  if (u <= f.umax0) return horner_host(f.c0, std::fma(u, f.scale0, f.offset0));
  if (u >= f.far_hi || f.far_n == 0) return 0.0f;
  const int p = std::min((int)((u - f.far_lo) * f.far_inv_w), f.far_n - 1);
  const float lo = f.far_lo + (float)p * f.far_w;
  const float x = (u - lo) * (2.0f * f.far_inv_w) - 1.0f;
  return horner_host(far.data() + (size_t)p * (FIT_DEG + 1), x);
}

// ------------------------------------------------------------------ device

__device__ __forceinline__ float horner_dev(const float* c, float x) {
  float acc = c[FIT_DEG];
#pragma unroll
  for (int j = FIT_DEG - 1; j >= 0; --j) acc = fmaf(acc, x, c[j]);
  return acc;
}

__device__ __forceinline__ float horner_far(const float* __restrict__ c, float x) {
  float acc = __ldg(c + FIT_DEG);
#pragma unroll
  for (int j = FIT_DEG - 1; j >= 0; --j) acc = fmaf(acc, x, __ldg(c + j));
  return acc;
}

// S(u) = e^{-u^2} R(u)
__device__ __forceinline__ float short_range_S(float u, const SFit& f, const float* __restrict__ far) {
  float R;
  if (u <= f.umax0) {
    R = horner_dev(f.c0, fmaf(u, f.scale0, f.offset0));
  } else if (u < f.far_hi) {
    const int p = min((int)((u - f.far_lo) * f.far_inv_w), f.far_n - 1);
    const float lo = fmaf((float)p, f.far_w, f.far_lo);
    R = horner_far(far + p * (FIT_DEG + 1), fmaf(u - lo, 2.0f * f.far_inv_w, -1.0f));
  } else {
    return 0.0f;
  }
  const float uu = u * u;
  const float err = fmaf(u, u, -uu);  // u*u = uu + err exactly
  const float e = exp2f(-uu * 1.44269504f);
  return fmaf(-e, err, e) * R;
}

// tree.rs:61-66 without the division and square roots: f = -K m S(r) (r^2 + eps^2)^{-3/2}
__device__ __forceinline__ float pair_factor(float r2, float neg_km, const WalkParams& w,
                                             const float* __restrict__ far) {
  const float r = r2 > 0.0f ? r2 * rsqrtf(r2) : 0.0f;
  const float S = short_range_S(r * w.inv_two_rs, w.fit, far);
  const float rs = rsqrtf(r2 + w.eps2);
  return neg_km * S * (rs * rs * rs);
}

// Hardware approximations (MUFU): relative error about 2^-22, no special handling of
// denormal inputs (the arguments here are r^2 + tiny, r^2 + eps^2 and -u^2 log2(e)).
__device__ __forceinline__ float rsqrt_approx(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float exp2_approx(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// The splits whose cutoff lies beyond the fit's piece 0 (out of line).
__device__ __noinline__ float short_range_S_far(float r, const WalkParams* w, const float* __restrict__ far) {
  return short_range_S(r * w->inv_two_rs, w->fit, far);
}

// The factor of a source's difference y - x for four pairs at once (two f32x2 chains), unit coupling
// and mass: S(u) (r^2 + eps^2)^(-3/2).
// u^2 = r^2 / (2 r_s)^2 comes from r^2 itself, so e^{-u^2} is one multiplication and one ex2.
__device__ __forceinline__ void pair_factor4(const float2 (&r2)[2], float2 (&f)[2], const WalkParams& w,
                                             const float* __restrict__ far) {
  const PairConst2& c = w.p2;
  float2 r[2], S[2];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const float2 rr = __fadd2_rn(r2[q], c.tiny);
    r[q] = __fmul2_rn(r2[q], make_float2(rsqrt_approx(rr.x), rsqrt_approx(rr.y)));
  }
  if (w.fit_covers) {
    float2 x[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      x[q] = __ffma2_rn(r[q], c.scale0, c.offset0);
      S[q] = c.c0[FIT_DEG];
    }
#pragma unroll
    for (int j = FIT_DEG - 1; j >= 0; --j) {
#pragma unroll
      for (int q = 0; q < 2; ++q) S[q] = __ffma2_rn(S[q], x[q], c.c0[j]);
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const float2 ea = __fmul2_rn(r2[q], c.exp_scale);
      S[q] = __fmul2_rn(make_float2(exp2_approx(ea.x), exp2_approx(ea.y)), S[q]);
    }
  } else {
#pragma unroll
    for (int q = 0; q < 2; ++q)
      S[q] = make_float2(short_range_S_far(r[q].x, &w, far), short_range_S_far(r[q].y, &w, far));
  }
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const float2 e = __fadd2_rn(r2[q], c.eps2);
    const float2 rs = make_float2(rsqrt_approx(e.x), rsqrt_approx(e.y));
    f[q] = __fmul2_rn(S[q], __fmul2_rn(__fmul2_rn(rs, rs), rs));
  }
}

// tree.rs:253-261: d = x - L round(x / L), x = a - b, exact. |x| < 0.49 L gives a zero quotient
// whatever its last bit, 0.51 L < |x| < 1.49 L a quotient of +-1; the rest divides with IEEE
// division (out of line: positions in the box only come there within 0.01 L of half the box).
__device__ __noinline__ float min_image_divide(float x, float box) {
  return __fsub_rn(x, __fmul_rn(box, roundf(__fdiv_rn(x, box))));
}
__device__ __forceinline__ float min_image_slow(float x, const WalkParams& w) {
  const float a = fabsf(x);
  if (a < w.guard) return x;
  if (a > w.wrap_lo && a < w.wrap_hi) return __fsub_rn(x, copysignf(w.box, x));
  return min_image_divide(x, w.box);
}

// Minimum image of the three components of a - b (raw differences already formed).
__device__ __forceinline__ void min_image3(float& d0, float& d1, float& d2, const WalkParams& w) {
  if (fmaxf(fabsf(d0), fmaxf(fabsf(d1), fabsf(d2))) >= w.guard) {
    d0 = min_image_slow(d0, w);
    d1 = min_image_slow(d1, w);
    d2 = min_image_slow(d2, w);
  }
}

__device__ __forceinline__ float norm2(float a, float b, float c) {
  return __fadd_rn(__fadd_rn(__fmul_rn(a, a), __fmul_rn(b, b)), __fmul_rn(c, c));
}

// The reference's opening test `2 half < theta * sqrt(r2)` (tree.rs:297). With lhs = 2 half,
// theta^2 r2 and lhs^2 carry at most ~7e-7 relative rounding against the exact squares of both
// sides, so outside a band of 1e-5 lhs^2 the squared comparison decides like the reference's;
// inside it the reference's expression is evaluated (IEEE square root).
__device__ __forceinline__ bool accept_node_sq(float r2, float l2, float band, float lhs, const WalkParams& w) {
  const float diff = __fsub_rn(__fmul_rn(w.theta2, r2), l2);
  if (fabsf(diff) > band) return diff > 0.0f;
  return lhs < __fmul_rn(w.theta, __fsqrt_rn(r2));
}
__device__ __forceinline__ bool accept_node_sq(float r2, float half, const WalkParams& w) {
  const float lhs = __fmul_rn(2.0f, half), l2 = __fmul_rn(lhs, lhs);
  return accept_node_sq(r2, l2, 1e-5f * l2, lhs, w);
}

// The reference's prune test (tree.rs:276-281): |min_image(centre - x)|^2 > (r_cut + sqrt(3) half)^2.
__device__ __forceinline__ bool prune_node(const float4& G, float x0, float x1, float x2, const WalkParams& w) {
  float t0 = __fsub_rn(G.x, x0), t1 = __fsub_rn(G.y, x1), t2 = __fsub_rn(G.z, x2);
  min_image3(t0, t1, t2, w);
  const float mr = __fadd_rn(w.r_cut, __fmul_rn(SQRT_3, G.w));
  return norm2(t0, t1, t2) > __fmul_rn(mr, mr);
}

// Per-warp shared state of the walk.
struct WalkShared {
  uint2 stack[STACK_CAP];          // (first node | (count - 1) << 29, lanes that walk it): a batch of siblings
  float4 geo[SLOTS];               // the step's nodes: centre, half
  float4 mass[SLOTS];              //                   centre of mass, count
  uint4 link[SLOTS];               //                   start, end, first child, child mask
  uint32_t lanes[SLOTS];           //                   lanes that walk the node
  uint4 sums[SLOTS];               // the step's j-th summed node, its sources at positions p, p + 1, ... of the
                                   // concatenation: (first particle - p, summing lanes, SUM_* flags)
  float sx[WINDOW], sy[WINDOW], sz[WINDOW];  // the window of direct-sum sources
  uint32_t pairs[WINDOW / 32][32];  // per word of 32 sources: first each source's summing lanes, then, per
                                    // lane, the sources within r_cut
  float4 box_c, box_h;             // the warp's bounding box: centre, half extent (+ tolerance)
};
constexpr uint32_t SUM_IMAGE = 1u;  // a source of the node may need a periodic image
constexpr uint32_t SUM_SOME = 2u;   // not every lane of the warp sums the node

// 16-byte asynchronous copy global -> shared (completion awaited with cp.async.wait_all).
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"(a), "l"(gmem) : "memory");
}
// Bits lo .. lo + len - 1 (len in 1..32).
__device__ __forceinline__ uint32_t bit_span(uint32_t lo, uint32_t len) {
  return (len >= 32u ? 0xffffffffu : ((1u << len) - 1u)) << lo;
}

// Transpose of the 32 x 32 bit matrix whose row q lane q holds: bit q of lane l's result is bit l of
// lane q's argument.
__device__ __forceinline__ uint32_t transpose_bits(uint32_t x, int lane) {
  uint32_t m = 0x0000ffffu;
#pragma unroll
  for (int j = 16; j > 0; j >>= 1) {
    const uint32_t y = __shfl_xor_sync(0xffffffffu, x, j);
    x = (lane & j) ? ((x & ~m) | ((y >> j) & m)) : ((x & m) | ((y & m) << j));
    m ^= m << (j >> 1);
  }
  return x;
}

// Distance on one axis between the warp's box (centre c, half extent h) and a point or a cube of
// half size r at p, over all periodic images; positions lie in [0, L].
__device__ __forceinline__ float axis_gap(float p, float c, float h, float r, float box) {
  const float e = fabsf(p - c);
  return fmaxf(fminf(e, fabsf(box - e)) - (h + r), 0.0f);
}

// Direct-sum phase 1 for one word of 32 sources: bit t set when source t lies within r_cut of the
// lane's particle (tree.rs:286-298). WRAP = false (no periodic image involved): r^2 - cut_hi by
// fused multiply-adds, two sources per f32x2 instruction, whose sign bit is the answer; cut_hi
// lies 2e-6 above r_cut^2, so the bits are a superset of the reference's decisions, and phase 2
// settles the sources within 2e-6 of the cutoff by the reference's own arithmetic. IMAGE = true
// also takes the nearest periodic image, d - L rint(d / L), with a wider margin for its rounding
// (positions in [0, L]).
template <bool IMAGE>
__device__ __forceinline__ uint32_t word_pairs(const WalkShared& sh, int w0, float x0, float x1, float x2,
                                               const WalkParams& w) {
  uint32_t pm = 0;
  const float2 X0 = make_float2(-x0, -x0), X1 = make_float2(-x1, -x1), X2 = make_float2(-x2, -x2);
  const float cut = IMAGE ? w.cut_image : w.cut_hi;
  const float2 C = make_float2(-cut, -cut);
  const float2 il = make_float2(w.inv_box, w.inv_box), nl = make_float2(-w.box, -w.box);
  // rint by adding and subtracting 1.5 * 2^23
  const float2 up = make_float2(12582912.0f, 12582912.0f), down = make_float2(-12582912.0f, -12582912.0f);
  auto nearest = [&](float2 d) { return __ffma2_rn(__fadd2_rn(__ffma2_rn(d, il, up), down), nl, d); };
#pragma unroll 2
  for (int t = 28; t >= 0; t -= 4) {
    const float4 a = *reinterpret_cast<const float4*>(sh.sx + w0 + t);
    const float4 b = *reinterpret_cast<const float4*>(sh.sy + w0 + t);
    const float4 c = *reinterpret_cast<const float4*>(sh.sz + w0 + t);
    float2 d0 = __fadd2_rn(X0, make_float2(a.x, a.y)), e0 = __fadd2_rn(X0, make_float2(a.z, a.w));
    float2 d1 = __fadd2_rn(X1, make_float2(b.x, b.y)), e1 = __fadd2_rn(X1, make_float2(b.z, b.w));
    float2 d2 = __fadd2_rn(X2, make_float2(c.x, c.y)), e2 = __fadd2_rn(X2, make_float2(c.z, c.w));
    if (IMAGE) {
      d0 = nearest(d0), d1 = nearest(d1), d2 = nearest(d2);
      e0 = nearest(e0), e1 = nearest(e1), e2 = nearest(e2);
    }
    const float2 q = __ffma2_rn(d2, d2, __ffma2_rn(d1, d1, __ffma2_rn(d0, d0, C)));
    const float2 p = __ffma2_rn(e2, e2, __ffma2_rn(e1, e1, __ffma2_rn(e0, e0, C)));
    pm = __funnelshift_l(__float_as_uint(p.y), pm, 1);
    pm = __funnelshift_l(__float_as_uint(p.x), pm, 1);
    pm = __funnelshift_l(__float_as_uint(q.y), pm, 1);
    pm = __funnelshift_l(__float_as_uint(q.x), pm, 1);
  }
  return pm;
}

// Position of the highest set bit of x (x != 0).
__device__ __forceinline__ uint32_t top_bit(uint32_t x) {
  uint32_t r;
  asm("bfind.u32 %0, %1;" : "=r"(r) : "r"(x));
  return r;
}

// The same by the reference's own arithmetic, for positions anywhere.
__device__ __noinline__ uint32_t word_pairs_strict(const float* sx, const float* sy, const float* sz, float x0,
                                                   float x1, float x2, const WalkParams* w) {
  uint32_t pm = 0;
  for (int t = 0; t < 32; ++t) {
    float d0 = __fsub_rn(sx[t], x0), d1 = __fsub_rn(sy[t], x1), d2 = __fsub_rn(sz[t], x2);
    min_image3(d0, d1, d2, *w);
    pm |= (uint32_t)!(norm2(d0, d1, d2) > w->cut2) << t;
  }
  return pm;
}

// Direct-sum phase 2: the pair forces of the window's marked sources, four per iteration (two
// f32x2 chains, which share the loads of the fit's coefficients and hide each other's latency),
// added to the packed accumulators. `words`: the lane's words with a marked source. A lane walks
// through its own words, so that lanes whose sources lie in different words do not wait for one
// another.
__device__ __forceinline__ void window_forces(const WalkShared& sh, uint32_t words, int lane, bool image, float x0,
                                              float x1, float x2, const WalkParams& w, const float* __restrict__ far,
                                              float2& A0, float2& A1, float2& A2, uint32_t& n_pairs) {
  const float2 X0 = make_float2(-x0, -x0), X1 = make_float2(-x1, -x1), X2 = make_float2(-x2, -x2);
  uint32_t cur = 0, base = 0;
  // the next marked source, or the last one again with weight 0
  auto take = [&](uint32_t& t, float& keep) {
    if (cur == 0u && words != 0u) {
      const uint32_t q = top_bit(words);
      words ^= 1u << q;
      cur = sh.pairs[q][lane];
      base = q * 32u;
    }
    keep = 0.0f;
    if (cur != 0u) {
      const uint32_t b = top_bit(cur);
      cur ^= 1u << b;
      t = base + b;
      keep = 1.0f;
    }
  };
  while ((cur | words) != 0u) {
    uint32_t t[4];
    float keep[4];
    t[0] = 0;
    take(t[0], keep[0]);
#pragma unroll
    for (int q = 1; q < 4; ++q) {
      t[q] = t[q - 1];
      take(t[q], keep[q]);
    }
    float2 d0[2], d1[2], d2[2], r2[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const uint32_t a = t[2 * q], b = t[2 * q + 1];
      d0[q] = __fadd2_rn(X0, make_float2(sh.sx[a], sh.sx[b]));
      d1[q] = __fadd2_rn(X1, make_float2(sh.sy[a], sh.sy[b]));
      d2[q] = __fadd2_rn(X2, make_float2(sh.sz[a], sh.sz[b]));
    }
    if (image) {
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        min_image3(d0[q].x, d1[q].x, d2[q].x, w);
        min_image3(d0[q].y, d1[q].y, d2[q].y, w);
      }
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) r2[q] = __ffma2_rn(d2[q], d2[q], __ffma2_rn(d1[q], d1[q], __fmul2_rn(d0[q], d0[q])));
    if (fmaxf(fmaxf(r2[0].x, r2[0].y), fmaxf(r2[1].x, r2[1].y)) > w.cut_lo) {
      // within 2e-6 of the cutoff: the reference's r^2 decides
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float r = (q & 1) ? norm2(d0[q / 2].y, d1[q / 2].y, d2[q / 2].y) : norm2(d0[q / 2].x, d1[q / 2].x, d2[q / 2].x);
        if (keep[q] != 0.0f && r > w.cut2) {
          keep[q] = 0.0f;
          --n_pairs;
        }
      }
    }
    float2 f[2];
    pair_factor4(r2, f, w, far);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      f[q] = __fmul2_rn(f[q], make_float2(keep[2 * q], keep[2 * q + 1]));
      A0 = __ffma2_rn(d0[q], f[q], A0);
      A1 = __ffma2_rn(d1[q], f[q], A1);
      A2 = __ffma2_rn(d2[q], f[q], A2);
    }
  }
}

// Quadrupole term of an accepted node (no counterpart in the reference, whose nodes are monopoles,
// tree.rs:68-80): the second-order Taylor term of a = sum_j g(|d_j|) d_j about the centre of mass,
// d_j = D + e_j with sum_j e_j = 0, T = sum_j e_j e_j^T, g(r) = S(r / 2 r_s) (r^2 + eps^2)^(-3/2):
//   da = (1/2) [ h (D.T.D) D + (g'/r) (tr(T) D + 2 T D) ],   h = (g'' - g'/r) / r^2,
// with S' = -(2/sqrt(pi)) u^2 e^{-u^2} / r_s and S'' = -(2/sqrt(pi)) u (1 - u^2) e^{-u^2} / r_s^2
// (u = r / 2 r_s). Unit coupling, like the walk's sums; precision mode only (CUDA's erfcf / expf).
__device__ __forceinline__ void quad_term(float d0, float d1, float d2, const float4& Q0, const float4& Q1,
                                          const WalkParams& w, float2& A0, float2& A1, float2& A2) {
  const float r2 = d0 * d0 + d1 * d1 + d2 * d2;
  if (!(r2 > 0.0f)) return;
  const float r = sqrtf(r2), inv_r = 1.0f / r;
  const float rs = 0.5f / w.inv_two_rs;
  const float u = r * w.inv_two_rs, e = expf(-u * u);
  const float S = erfcf(u) + TWO_OVER_SQRT_PI * u * e;
  const float S1 = -TWO_OVER_SQRT_PI * u * u * e / rs;
  const float S2 = -TWO_OVER_SQRT_PI * u * (1.0f - u * u) * e / (rs * rs);
  const float q = r2 + w.eps2, iq = 1.0f / q, rq = rsqrtf(q);
  const float P = rq * iq, P1 = -3.0f * r * P * iq, P2 = -3.0f * P * iq + 15.0f * r2 * P * iq * iq;
  const float g1 = S1 * P + S * P1;
  const float g2 = S2 * P + 2.0f * S1 * P1 + S * P2;
  const float h = (g2 - g1 * inv_r) / r2;
  const float td0 = Q0.x * d0 + Q0.w * d1 + Q1.x * d2;
  const float td1 = Q0.w * d0 + Q0.y * d1 + Q1.y * d2;
  const float td2 = Q1.x * d0 + Q1.y * d1 + Q0.z * d2;
  const float dtd = d0 * td0 + d1 * td1 + d2 * td2, tr = Q0.x + Q0.y + Q0.z;
  const float a = 0.5f * h * dtd, b = 0.5f * g1 * inv_r;
  A0.y += a * d0 + b * (tr * d0 + 2.0f * td0);
  A1.y += a * d1 + b * (tr * d1 + 2.0f * td1);
  A2.y += a * d2 + b * (tr * d2 + 2.0f * td2);
}

// Whether box `box` takes the ordered walk (positions outside the box take the other one's strict tests).
__device__ __forceinline__ bool walk_ordered(const uint32_t* __restrict__ words, uint32_t box) {
  return words[WALK_DENSE + box] != 0u && words[WALK_OUTSIDE] == 0u;
}

// The box of a group in a batch: that of its first valid lane (a box's particles fill whole groups, and a list
// keeps each box's particles in whole groups).
__device__ __forceinline__ uint32_t group_box(uint32_t lanes, size_t i, const WalkParams& w) {
  return w.n_box ? __shfl_sync(0xffffffffu, (uint32_t)(i / w.n_box), __ffs(lanes) - 1) : 0u;
}

// One warp (or `team` warps of a block, each with its share of the direct nodes and accepted nodes)
// walks for a group of 32 particles.
template <bool QUAD, bool LIST, int WARPS, bool SKIP>
__global__ void __launch_bounds__(WARPS * 32, WALK_WARPS_PER_SM / WARPS) k_tree_walk(const uint4* __restrict__ link,
                                                            const float4* __restrict__ geo,
                                                            const float4* __restrict__ mass,
                                                            const float4* __restrict__ x4, size_t n,
                                                            const __grid_constant__ WalkParams w,
                                                            const float* __restrict__ far, float* __restrict__ acc3,
                                                            int accumulate, unsigned long long* counters,
                                                            DevStatus* st, const float* __restrict__ k_dev,
                                                            const uint32_t* __restrict__ list,
                                                            const uint32_t* __restrict__ list_n,
                                                            const float4* __restrict__ quad,
                                                            uint32_t* __restrict__ words, int team) {
  // Dynamic shared memory: WARPS WalkShared records, then (quadrupoles) the node index of each slot.
  extern __shared__ __align__(16) unsigned char walk_smem[];
  WalkShared* shared = reinterpret_cast<WalkShared*>(walk_smem);
  uint32_t(*node_ids)[SLOTS] = reinterpret_cast<uint32_t(*)[SLOTS]>(walk_smem + WARPS * sizeof(WalkShared));
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int sub = warp % team;
  WalkShared& sh = shared[warp];
  const size_t walked = LIST ? (size_t)*list_n : n;
  const float kk = k_dev ? *k_dev : w.k;
  uint32_t n_pairs = 0, n_accepts = 0, n_cand = 0;

  // Warps take groups from a common counter until none is left: groups differ several-fold in cost,
  // and a warp that waited for its block's slowest would hold its shared memory idle. A team's
  // blocks walk the groups of their own index.
  for (bool more = true; more; more = team == 1) {
    uint32_t ticket = 0;
    if (team == 1) {
      if (lane == 0) ticket = atomicAdd(&words[WALK_TICKET], 1u);
      ticket = __shfl_sync(FULL, ticket, 0);
      if ((size_t)ticket * 32 >= walked) break;
    } else {
      ticket = blockIdx.x * (WARPS / team) + warp / team;
    }
    // Lane l of the group walks for sorted particle t, or, with a list, for particle list[t] (t below
    // *list_n): the list keeps the sorted order, so a warp's particles stay spatially coherent.
    const size_t t = (size_t)ticket * 32 + lane;
    const bool valid = t < walked;
    const size_t i = LIST ? (valid ? (size_t)list[t] : 0) : t;
    const unsigned lanes = __ballot_sync(FULL, valid);
    // (SKIP: the groups of boxes that k_walk_ordered walks are left out)
    const bool elsewhere = SKIP && lanes && walk_ordered(words, group_box(lanes, i, w));
    const unsigned group = elsewhere ? 0u : lanes;
    const float4 xi = valid ? __ldg(x4 + i) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const float x0 = xi.x, x1 = xi.y, x2 = xi.z;
    const uint32_t self = (uint32_t)i;
    // Accumulators of the even and odd pairs (x: even pairs and accepted nodes).
    float2 A0 = make_float2(0.0f, 0.0f), A1 = A0, A2 = A0;

    if (group != 0) {
      // Bounding box of the warp's particles (centre, half extent), for the warp-level tests.
      float lo0 = valid ? x0 : INFINITY, lo1 = valid ? x1 : INFINITY, lo2 = valid ? x2 : INFINITY;
      float hi0 = valid ? x0 : -INFINITY, hi1 = valid ? x1 : -INFINITY, hi2 = valid ? x2 : -INFINITY;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        lo0 = fminf(lo0, __shfl_xor_sync(FULL, lo0, o));
        lo1 = fminf(lo1, __shfl_xor_sync(FULL, lo1, o));
        lo2 = fminf(lo2, __shfl_xor_sync(FULL, lo2, o));
        hi0 = fmaxf(hi0, __shfl_xor_sync(FULL, hi0, o));
        hi1 = fmaxf(hi1, __shfl_xor_sync(FULL, hi1, o));
        hi2 = fmaxf(hi2, __shfl_xor_sync(FULL, hi2, o));
      }
      if (lane == 0) {
        const float tol = 1e-5f * w.box;  // far above the rounding of positions and differences
        sh.box_c = make_float4(0.5f * (lo0 + hi0), 0.5f * (lo1 + hi1), 0.5f * (lo2 + hi2), 0.0f);
        sh.box_h = make_float4(0.5f * (hi0 - lo0) + tol, 0.5f * (hi1 - lo1) + tol, 0.5f * (hi2 - lo2) + tol, 0.0f);
      }
      // The warp-level tests take every particle to lie in [0, L] (so in the cubes of its nodes) and
      // r_cut >= 0. Otherwise (`strict`) nothing is decided for the warp: every lane applies the
      // reference's prune test to every node, and every source takes the image test.
      const bool strict = words[WALK_OUTSIDE] != 0u || !(w.r_cut >= 0.0f);
      const uint32_t self_lo = __reduce_min_sync(FULL, valid ? self : 0xffffffffu);
      const uint32_t self_hi = __reduce_max_sync(FULL, valid ? self : 0u);

      // A step of the walk handles up to SLOTS nodes, one per lane: one or more stack entries (each the
      // children of an opened node) placed in consecutive slots. `mine` holds the slots this lane
      // walks. Lane c copies slot c's three records into shared memory asynchronously; the next step's
      // copies are in flight while the direct sums are formed. The walk starts at the root: node 0, or
      // in a batch of boxes the root of the warp's box (nodes 0 .. boxes - 1).
      const uint32_t root = group_box(group, i, w);
      uint32_t b_count = 1, mine = (group >> lane) & 1u;
      if (lane == 0) {
        cp_async16(&sh.geo[0], geo + root);
        cp_async16(&sh.mass[0], mass + root);
        cp_async16(&sh.link[0], link + root);
        sh.lanes[0] = group;
        if constexpr (QUAD) node_ids[warp][0] = root;
      }
      int sp = 0;
      // The window of sources: its fill, the words that hold a source with a possible periodic image,
      // the words that hold a source not summed by the whole warp, the slot of the lane's own particle.
      uint32_t nsrc = 0, image_words = 0, some_words = 0, self_slot = 0xffffffffu;
      int turn = 0;  // a team's warps take turns over the stages of all steps
      for (;;) {
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        __syncwarp();
        const float4* bgeo = sh.geo;
        const float4* bmass = sh.mass;

        // What lane c can decide of node c for the whole warp, over all periodic images of its box:
        //   direct  octant 0 is empty (`children[0] == NO_CHILD`, tree.rs:286): its particles are summed
        //   flat    every child is direct, so no node below can be accepted: what the lanes do not
        //           accept of it they sum, without opening it
        //   keep    some lane may reach it: the box is within r_cut + sqrt(3) half of its centre
        //   sum     some particle of it may be within r_cut of some lane: the box is within r_cut of
        //           the cube (a lane whose own walk prunes the node has none)
        //   ask     some lane may accept it: 2 half < theta times the distance of the farthest lane
        bool direct = false, flat = false, keep = false, sum = false, ask = false, plain = false;
        uint4 L = make_uint4(0u, 0u, 0u, 0u);
        uint32_t stay = 0;  // the lanes that go on below node c (or sum it)
        if ((uint32_t)lane < b_count) {
          const float4 bc = sh.box_c, bh = sh.box_h, G = bgeo[lane];
          L = sh.link[lane];
          stay = sh.lanes[lane];
          direct = (L.w & 1u) == 0u;
          flat = !strict && (L.w & NODE_FLAT) != 0u;
          const float mr = w.r_cut + SQRT_3 * G.w;
          float g0 = axis_gap(G.x, bc.x, bh.x, 0.0f, w.box), g1 = axis_gap(G.y, bc.y, bh.y, 0.0f, w.box),
                g2 = axis_gap(G.z, bc.z, bh.z, 0.0f, w.box);
          keep = strict || !(g0 * g0 + g1 * g1 + g2 * g2 > mr * mr * 1.0001f);
          g0 = fmaxf(g0 - G.w, 0.0f), g1 = fmaxf(g1 - G.w, 0.0f), g2 = fmaxf(g2 - G.w, 0.0f);
          sum = strict || !(g0 * g0 + g1 * g1 + g2 * g2 > w.cull2);
          // No lane needs a periodic image for this node: every difference between a lane's
          // particle and the node's centre, centre of mass or particles (all inside the cube) is
          // below 0.49 L on every axis.
          const float e0 = fabsf(G.x - bc.x) + bh.x, e1 = fabsf(G.y - bc.y) + bh.y, e2 = fabsf(G.z - bc.z) + bh.z;
          plain = !strict && fmaxf(e0, fmaxf(e1, e2)) + G.w < w.guard;
          if (!direct) {
            const float4 M = bmass[lane];
            const float f0 = fabsf(M.x - bc.x) + bh.x, f1 = fabsf(M.y - bc.y) + bh.y, f2 = fabsf(M.z - bc.z) + bh.z;
            ask = !(plain && w.theta2 * (f0 * f0 + f1 * f1 + f2 * f2) * 1.0001f < 4.0f * G.w * G.w);
          }
        }
        const uint32_t nodes = __ballot_sync(FULL, keep);
        const uint32_t near = __ballot_sync(FULL, plain);
        const uint32_t asked = __ballot_sync(FULL, keep && ask);

        // Each lane's own decision on the nodes that some lane may accept: accepted when
        // 2 half < theta |min_image(com - x)| and not pruned. A lane that prunes a node without being
        // able to accept it just goes on: it prunes, or finds no pair in, everything below.
        uint32_t amask = 0, todo = asked & mine;
        if (strict) {  // the reference's walk node by node: pruning lanes leave
          for (uint32_t rem = nodes; rem; rem &= rem - 1) {
            const int c = __ffs(rem) - 1;
            const bool pruned = prune_node(bgeo[c], x0, x1, x2, w);
            const uint32_t gone = __ballot_sync(FULL, pruned);
            if (lane == c) stay &= ~gone;
            if (pruned) todo &= ~(1u << c);
          }
        }
        if ((todo & ~near) == 0u) {
          for (uint32_t rem = todo; rem; rem &= rem - 1) {
            const uint32_t c = __ffs(rem) - 1;
            const float4 M = bmass[c];
            const float s0 = __fsub_rn(M.x, x0), s1 = __fsub_rn(M.y, x1), s2 = __fsub_rn(M.z, x2);
            if (accept_node_sq(norm2(s0, s1, s2), bgeo[c].w, w) && !prune_node(bgeo[c], x0, x1, x2, w)) amask |= 1u << c;
          }
        } else {
          for (uint32_t rem = todo; rem; rem &= rem - 1) {
            const uint32_t c = __ffs(rem) - 1;
            const float4 M = bmass[c];
            float s0 = __fsub_rn(M.x, x0), s1 = __fsub_rn(M.y, x1), s2 = __fsub_rn(M.z, x2);
            min_image3(s0, s1, s2, w);
            if (accept_node_sq(norm2(s0, s1, s2), bgeo[c].w, w) && !prune_node(bgeo[c], x0, x1, x2, w)) amask |= 1u << c;
          }
        }
        for (uint32_t rem = __reduce_or_sync(FULL, amask); rem; rem &= rem - 1) {
          const int c = __ffs(rem) - 1;
          const uint32_t gone = __ballot_sync(FULL, (amask >> c) & 1u);
          if (lane == c) stay &= ~gone;
        }

        // Push the opened nodes' children as new stack entries (any order gives each lane the same
        // set of interactions; only the order of its sums differs). Higher slots go deeper into the
        // stack, so that the entries popped first, which fill the lowest slots, have their children
        // popped first again.
        const bool open = keep && !direct && !flat && stay != 0u;
        const uint32_t opened = __ballot_sync(FULL, open);
        if (opened) {
          const int npush = __popc(opened);
          // (node indices above 29 bits, trees of more than 2^28 particles, do not fit an entry)
          const bool wide = __any_sync(FULL, open && (L.z >> FIRST_BITS) != 0u);
          if (sp + npush > STACK_CAP || wide) {
            if (lane == 0) dev_fail(st, DEV_STACK_OVERFLOW, sp);
            break;
          }
          if (open)
            sh.stack[sp + __popc(opened >> lane) - 1] =
                make_uint2(L.z | ((uint32_t)(__popc(L.w & 0xFFu) - 1) << FIRST_BITS), stay);
          sp += npush;
          __syncwarp();
        }

        // Accepted centres of mass (tree.rs:299-305); a team's warps take every team-th slot.
        if (team > 1) amask &= (team == 2 ? 0x55555555u : 0x11111111u) << sub;
        for (; amask; amask &= amask - 1) {
          const int c = __ffs(amask) - 1;
          const float4 M = bmass[c];
          float s0 = __fsub_rn(M.x, x0), s1 = __fsub_rn(M.y, x1), s2 = __fsub_rn(M.z, x2);
          min_image3(s0, s1, s2, w);
          const float f = pair_factor(norm2(s0, s1, s2), -M.w, w, far);
          A0.x = fmaf(-s0, f, A0.x);
          A1.x = fmaf(-s1, f, A1.x);
          A2.x = fmaf(-s2, f, A2.x);
          if constexpr (QUAD) {
            const size_t node = node_ids[warp][c];
            quad_term(s0, s1, s2, __ldg(quad + 2 * node), __ldg(quad + 2 * node + 1), w, A0, A1, A2);
          }
          ++n_accepts;
        }

        // Pop the next step: the top entry, and while the stack is shallow, further entries as long as
        // they fit in the slots. Its copies complete during the direct sums below.
        __syncwarp();
        uint32_t nx_count = 0, nx_mine = 0;
        if (sp > 0) {
          const bool merge = sp <= MERGE_SP;
          uint2 e = sh.stack[--sp];
          for (;;) {
            const uint32_t first = e.x & ((1u << FIRST_BITS) - 1u), cnt = (e.x >> FIRST_BITS) + 1u;
            if ((uint32_t)lane - nx_count < cnt) {
              const uint32_t node = first + ((uint32_t)lane - nx_count);
              cp_async16(&sh.geo[lane], geo + node);
              cp_async16(&sh.mass[lane], mass + node);
              cp_async16(&sh.link[lane], link + node);
              sh.lanes[lane] = e.y;
              if constexpr (QUAD) node_ids[warp][lane] = node;
            }
            if ((e.y >> lane) & 1u) nx_mine |= bit_span(nx_count, cnt);
            nx_count += cnt;
            if (!merge || sp == 0) break;
            e = sh.stack[sp - 1];
            if (nx_count + (e.x >> FIRST_BITS) + 1u > (uint32_t)SLOTS) break;
            --sp;
          }
        }

        // Direct sums: the particles of the step's summed nodes, concatenated in slot order, are fetched
        // STAGE at a time (a team's warps take every team-th stage); those within r_cut of the warp's
        // box join the window.
        const bool summed = keep && sum && (direct || flat) && stay != 0u;
        const uint32_t dset = __ballot_sync(FULL, summed);
        uint32_t total = 0, start = 0xffffffffu, self_pos = 0xffffffffu;
        bool own = false, some_image = false, some_lanes = false;
        if (dset) {
          const uint32_t cnt = summed ? L.y - L.x : 0u;
          uint32_t end = cnt;  // inclusive prefix sum over the slots
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(FULL, end, o);
            if (lane >= o) end += v;
          }
          total = __shfl_sync(FULL, end, 31);
          if (summed) {
            start = end - cnt;
            sh.sums[__popc(dset & ((1u << lane) - 1u))] =
                make_uint4(L.x - start, stay, (plain ? 0u : SUM_IMAGE) | (stay != group ? SUM_SOME : 0u), 0u);
          }
          some_image = __any_sync(FULL, summed && !plain);
          some_lanes = __any_sync(FULL, summed && stay != group);
          // This lane's own particle's position in the concatenation (j != i).
          uint32_t hit = __ballot_sync(FULL, summed && L.x <= self_hi && L.y > self_lo);
          own = hit != 0u;
          __syncwarp();
          for (; hit; hit &= hit - 1) {
            const int c = __ffs(hit) - 1;
            const uint32_t b0 = __shfl_sync(FULL, start, c), f0 = __shfl_sync(FULL, L.x, c), n0 = __shfl_sync(FULL, cnt, c);
            if (self - f0 < n0) self_pos = b0 + (self - f0);
          }
        }
        const bool last = nx_count == 0;
        uint32_t base = (uint32_t)((sub + turn) & (team - 1)) * STAGE;
        turn -= (int)((total + STAGE - 1) / STAGE);
        for (;;) {
          if (base < total && nsrc + STAGE <= WINDOW) {
            const float4 bc = sh.box_c, bh = sh.box_h;
            float4 y[STAGE / 32];
            uint32_t who[STAGE / 32], flags[STAGE / 32];
#pragma unroll
            for (int q = 0; q < STAGE / 32; ++q) {
              // Lane l fetches position g. The summed nodes that start at or before g give its node.
              const uint32_t b = base + 32u * q, g = b + (uint32_t)lane;
              const uint32_t before = (uint32_t)__popc(__ballot_sync(FULL, start < b));
              const uint32_t heads = __reduce_or_sync(FULL, start - b < 32u ? 1u << (start - b) : 0u);
              const uint4 S = sh.sums[before + __popc(heads & (0xffffffffu >> (31 - lane))) - 1];
              who[q] = S.y;
              flags[q] = S.z;
              y[q] = g < total ? __ldg(x4 + (g + S.x)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
#pragma unroll
            for (int q = 0; q < STAGE / 32; ++q) {
              const uint32_t b = base + 32u * q;
              const float e0 = axis_gap(y[q].x, bc.x, bh.x, 0.0f, w.box), e1 = axis_gap(y[q].y, bc.y, bh.y, 0.0f, w.box),
                          e2 = axis_gap(y[q].z, bc.z, bh.z, 0.0f, w.box);
              const bool in = b + (uint32_t)lane < total && (strict || !(e0 * e0 + e1 * e1 + e2 * e2 > w.cull2));
              const uint32_t kept = __ballot_sync(FULL, in);
              const uint32_t pos = nsrc + (uint32_t)__popc(kept & ((1u << lane) - 1u));
              if (in) {
                sh.sx[pos] = y[q].x;
                sh.sy[pos] = y[q].y;
                sh.sz[pos] = y[q].z;
                (&sh.pairs[0][0])[pos] = who[q];
              }
              if (own) {
                const uint32_t at = __shfl_sync(FULL, pos, (int)((self_pos - b) & 31u));
                if (self_pos - b < 32u) self_slot = at;
              }
              const uint32_t fresh = (uint32_t)__popc(kept);
              if (some_image | some_lanes) {
                const uint32_t words = fresh ? (1u << (nsrc >> 5)) | (1u << ((nsrc + fresh - 1) >> 5)) : 0u;
                if (__any_sync(FULL, in && (flags[q] & SUM_IMAGE))) image_words |= words;
                if (__any_sync(FULL, in && (flags[q] & SUM_SOME))) some_words |= words;
              }
              nsrc += fresh;
            }
            base += STAGE * (uint32_t)team;
            continue;
          }
          if (base >= total && !(last && nsrc > 0u)) break;
          // The window is full, or the walk has ended: mark the pairs, then sum them.
          __syncwarp();
          const int nw = (int)((nsrc + 31u) >> 5);
          uint32_t words = 0;
          for (int q = 0; q < nw; ++q) {
            uint32_t live = bit_span(0, min(32u, nsrc - 32u * (uint32_t)q));
            if ((some_words >> q) & 1u) live &= transpose_bits(sh.pairs[q][lane], lane);
            if ((self_slot >> 5) == (uint32_t)q) live &= ~(1u << (self_slot & 31u));
            if (!valid) live = 0;
            n_cand += __popc(live);
            uint32_t pm;
            if (strict)
              pm = word_pairs_strict(sh.sx + 32 * q, sh.sy + 32 * q, sh.sz + 32 * q, x0, x1, x2, &w);
            else if ((image_words >> q) & 1u)
              pm = word_pairs<true>(sh, 32 * q, x0, x1, x2, w);
            else
              pm = word_pairs<false>(sh, 32 * q, x0, x1, x2, w);
            pm &= live;
            n_pairs += __popc(pm);
            sh.pairs[q][lane] = pm;
            words |= (uint32_t)(pm != 0u) << q;
          }
          window_forces(sh, words, lane, image_words != 0u, x0, x1, x2, w, far, A0, A1, A2, n_pairs);
          __syncwarp();
          nsrc = image_words = some_words = 0;
          self_slot = 0xffffffffu;
        }
        if (last) break;
        b_count = nx_count;
        mine = nx_mine;
      }
      asm volatile("cp.async.wait_all;\n" ::: "memory");
    }
    float s0 = A0.x + A0.y, s1 = A1.x + A1.y, s2 = A2.x + A2.y;
    if (team > 1) {  // the team's partial sums, added in the order of its warps
      sh.sx[lane] = s0;
      sh.sy[lane] = s1;
      sh.sz[lane] = s2;
      __syncthreads();
      if (sub == 0)
        for (int q = 1; q < team; ++q) {
          const WalkShared& o = shared[warp + q];
          s0 += o.sx[lane];
          s1 += o.sy[lane];
          s2 += o.sz[lane];
        }
    }
    // tree.rs:61-66 multiplies every pair by the coupling K; here the unit-coupling sum is scaled once
    const float a0 = kk * s0, a1 = kk * s1, a2 = kk * s2;
    if (valid && sub == 0 && !elsewhere) {
      if (accumulate) {
        acc3[3 * i] = __fadd_rn(acc3[3 * i], a0);
        acc3[3 * i + 1] = __fadd_rn(acc3[3 * i + 1], a1);
        acc3[3 * i + 2] = __fadd_rn(acc3[3 * i + 2], a2);
      } else {
        acc3[3 * i] = a0;
        acc3[3 * i + 1] = a1;
        acc3[3 * i + 2] = a2;
      }
    }
    __syncwarp();
  }
  if (counters) {
    unsigned long long p = n_pairs, a = n_accepts, c = n_cand;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      p += __shfl_xor_sync(FULL, p, o);
      a += __shfl_xor_sync(FULL, a, o);
      c += __shfl_xor_sync(FULL, c, o);
    }
    if (lane == 0) {
      atomicAdd(&counters[0], p);
      atomicAdd(&counters[1], a);
      atomicAdd(&counters[2], c);
    }
  }
}

// ---------------------------------------------------------------------------------------------
// The ordered walk. Every lane classifies every node of a step, the step's direct sums follow at once, in chunks of 32
// sources of the concatenated nodes, and a lane adds its pairs of a chunk two by two, as this library did before
// k_tree_walk collected its sources in a window. The order is neither the reference's nor more accurate: against 64
// bits both walks' forces are off by 8.7e-7 of the RMS at 45^3 late particles, 2.5e-6 at 64^3, 2.4e-5 at 101^3
// (RMS; medians 1.7e-7 and 1.3e-7, 1.9e-7 both, 3.2e-7 and 2.5e-7). What it keeps is the roundings, and with them the
// trajectories that dense boxes had: in a core whose pairs lie closer than the softening one rounding of a position moves
// an acceleration by up to 1e-3 of the box's RMS, so that another order of f32 sums shows after ten steps (largest
// difference of an acceleration after 18 steps, of the RMS, eight boxes each: 3.7e-4 where the deepest split is 4 levels
// below a smooth box's, 21^3 particles; 8.6e-4 at 5 levels, 27^3; 1.2e-2 at 6, 64^3). It serves the simulations, with
// and without a list of walked particles, whose build split nodes ORDERED_DEPTH levels and more below the level of a
// smooth distribution (WALK_DENSE); until then, and from ORDERED_PARTICLES particles on, a box goes by k_tree_walk. That
// bound is one of cost, not of rounding: the walk is most of a large box's step, and this one is
// slower: 0.60 ms against 0.20 at 27^3 late particles, 0.78 against 0.47 at 45^3, 1.10 against 0.81 at 64^3, 3.38 against
// 2.55 at 101^3.
// ---------------------------------------------------------------------------------------------
constexpr int ORDERED_WARPS = 4;
constexpr int ORDERED_MERGE_SP = 96;
// Sources within reach from which a chunk is tested in turn, without bit scans (an isolated halo of 65,536 particles
// within the cutoff: 14.6 -> 12.5 ms with whole chunks known to be near and 9 blocks an SM).
constexpr int ORDERED_IN_TURN = 16;
constexpr int ORDERED_STACK_CAP = ORDERED_MERGE_SP + SLOTS + 7 * KEY_LEVELS + 8;

// pair_factor for two pairs at once (f32x2 arithmetic), unit coupling.
__device__ __forceinline__ float2 ordered_factor(float2 r2, const WalkParams& w, const float* __restrict__ far) {
  const OrderedConst& c = w.ordered;
  const float2 rr = __fadd2_rn(r2, c.tiny);
  const float2 r = __fmul2_rn(r2, make_float2(rsqrt_approx(rr.x), rsqrt_approx(rr.y)));
  const float2 u = __fmul2_rn(r, c.inv_two_rs);
  float2 S;
  if (fmaxf(u.x, u.y) <= w.fit.umax0) {
    const float2 x = __ffma2_rn(u, c.scale0, c.offset0);
    float2 R = c.c0[FIT_DEG];
#pragma unroll
    for (int j = FIT_DEG - 1; j >= 0; --j) R = __ffma2_rn(R, x, c.c0[j]);
    // e^{-u^2} = 2^{-uu log2 e} (1 - err) with uu + err = u*u exactly
    const float2 uu = __fmul2_rn(u, u);
    const float2 nerr = __ffma2_rn(__fmul2_rn(u, make_float2(-1.0f, -1.0f)), u, uu);
    const float2 ea = __fmul2_rn(uu, c.neg_log2e);
    const float2 e = make_float2(exp2_approx(ea.x), exp2_approx(ea.y));
    S = __fmul2_rn(__ffma2_rn(e, nerr, e), R);
  } else {
    S = make_float2(short_range_S(u.x, w.fit, far), short_range_S(u.y, w.fit, far));
  }
  const float2 q = __fadd2_rn(r2, c.eps2);
  const float2 rs = make_float2(rsqrt_approx(q.x), rsqrt_approx(q.y));
  return __fmul2_rn(__fmul2_rn(c.neg_m, S), __fmul2_rn(__fmul2_rn(rs, rs), rs));
}

struct OrderedShared {
  uint2 stack[ORDERED_STACK_CAP];          // (first node | (count - 1) << 29, lane mask): a batch of siblings
  float4 geo[2][SLOTS];            // the current and the next step's nodes: centre, half
  float4 mass[2][SLOTS];           //                                        centre of mass, count
  uint4 link[2][SLOTS];            //                                        start, end, first child, child mask
  float4 pre[SLOTS];               // per node of the current step: prune radius^2, l^2, 1e-5 l^2, l = 2 half
  uint32_t dbeg[SLOTS], dend[SLOTS], dsrc[SLOTS];  // direct sums: node c's sources are positions
                                                   // dbeg .. dend - 1 of the concatenation,
                                                   // particles dsrc + (position - dbeg)
  float nx[32], ny[32], nz[32];    // a chunk of direct-sum sources, negated: -x, -y, -z
  float4 box_c, box_h;             // the warp's bounding box: centre, half extent (+ tolerance)
};

// Direct-sum phase 1 for one chunk: bit t set when source t of `reach` (others: undefined) lies within r_cut of the
// lane's particle, by the reference's own arithmetic: the differences and squares of two sources per instruction
// (f32x2, each element rounded like the scalar operation), the sums scalar (a packed multiply feeding a packed
// add can be contracted into one FMA).
template <bool WRAP>
__device__ __forceinline__ uint32_t ordered_pairs(const OrderedShared& sh, uint32_t reach, float x0, float x1, float x2,
                                                  const WalkParams& w) {
  uint32_t pm = 0;
  const float2 X0 = make_float2(x0, x0), X1 = make_float2(x1, x1), X2 = make_float2(x2, x2);
  if (!WRAP && __popc(reach) >= ORDERED_IN_TURN) {
    const int cnt = 32 - __clz(reach);
#pragma unroll 4
    for (int t = 0; t < cnt; t += 2) {
      const float2 d0 = __fadd2_rn(X0, *reinterpret_cast<const float2*>(sh.nx + t));
      const float2 d1 = __fadd2_rn(X1, *reinterpret_cast<const float2*>(sh.ny + t));
      const float2 d2 = __fadd2_rn(X2, *reinterpret_cast<const float2*>(sh.nz + t));
      const float2 q0 = __fmul2_rn(d0, d0), q1 = __fmul2_rn(d1, d1), q2 = __fmul2_rn(d2, d2);
      const float ra = __fadd_rn(__fadd_rn(q0.x, q1.x), q2.x), rb = __fadd_rn(__fadd_rn(q0.y, q1.y), q2.y);
      pm |= ((uint32_t)!(ra > w.cut2) | ((uint32_t)!(rb > w.cut2) << 1)) << t;
    }
    return pm;
  }
  while (reach) {
    const int a = __ffs(reach) - 1;
    reach &= reach - 1;
    const int b = reach ? __ffs(reach) - 1 : a;
    reach &= reach - 1;
    float2 d0 = __fadd2_rn(X0, make_float2(sh.nx[a], sh.nx[b]));
    float2 d1 = __fadd2_rn(X1, make_float2(sh.ny[a], sh.ny[b]));
    float2 d2 = __fadd2_rn(X2, make_float2(sh.nz[a], sh.nz[b]));
    if (WRAP) {
      min_image3(d0.x, d1.x, d2.x, w);
      min_image3(d0.y, d1.y, d2.y, w);
    }
    const float2 q0 = __fmul2_rn(d0, d0), q1 = __fmul2_rn(d1, d1), q2 = __fmul2_rn(d2, d2);
    const float ra = __fadd_rn(__fadd_rn(q0.x, q1.x), q2.x), rb = __fadd_rn(__fadd_rn(q0.y, q1.y), q2.y);
    pm |= ((uint32_t)!(ra > w.cut2) << a) | ((uint32_t)!(rb > w.cut2) << b);
  }
  return pm;
}

// Direct-sum phase 2: the pair forces of the sources in pm, two per iteration, added to the
// packed accumulators (even and odd pairs).
template <bool WRAP>
__device__ __forceinline__ void chunk_forces(const OrderedShared& sh, uint32_t pm, float x0, float x1, float x2,
                                             const WalkParams& w, const float* __restrict__ far, float2& A0,
                                             float2& A1, float2& A2) {
  const float2 X0 = make_float2(x0, x0), X1 = make_float2(x1, x1), X2 = make_float2(x2, x2);
  while (pm) {
    const int t1 = __ffs(pm) - 1;
    pm &= pm - 1;
    int t2 = t1;
    float keep = 0.0f;  // a lone last pair is evaluated twice and its copy weighted by 0
    if (pm) {
      t2 = __ffs(pm) - 1;
      pm &= pm - 1;
      keep = 1.0f;
    }
    float2 d0 = __fadd2_rn(X0, make_float2(sh.nx[t1], sh.nx[t2]));
    float2 d1 = __fadd2_rn(X1, make_float2(sh.ny[t1], sh.ny[t2]));
    float2 d2 = __fadd2_rn(X2, make_float2(sh.nz[t1], sh.nz[t2]));
    if (WRAP) {
      min_image3(d0.x, d1.x, d2.x, w);
      min_image3(d0.y, d1.y, d2.y, w);
    }
    const float2 r2 = __ffma2_rn(d2, d2, __ffma2_rn(d1, d1, __fmul2_rn(d0, d0)));
    const float2 f = __fmul2_rn(ordered_factor(r2, w, far), make_float2(1.0f, keep));
    A0 = __ffma2_rn(d0, f, A0);
    A1 = __ffma2_rn(d1, f, A1);
    A2 = __ffma2_rn(d2, f, A2);
  }
}

template <bool QUAD, bool LIST>
__global__ void __launch_bounds__(ORDERED_WARPS * 32, 9) k_walk_ordered(const uint4* __restrict__ link,
                                                            const float4* __restrict__ geo,
                                                            const float4* __restrict__ mass,
                                                            const float4* __restrict__ x4, size_t n,
                                                            const __grid_constant__ WalkParams w,
                                                            const float* __restrict__ far, float* __restrict__ acc3,
                                                            int accumulate, unsigned long long* counters,
                                                            DevStatus* st, const float* __restrict__ k_dev,
                                                            const uint32_t* __restrict__ list,
                                                            const uint32_t* __restrict__ list_n,
                                                            const float4* __restrict__ quad,
                                                            const uint32_t* __restrict__ words) {
  // Dynamic shared memory: ORDERED_WARPS OrderedShared records, then (quadrupoles) the node index of each slot.
  extern __shared__ __align__(16) unsigned char walk_smem[];
  OrderedShared* shared = reinterpret_cast<OrderedShared*>(walk_smem);
  uint32_t(*node_ids)[2][SLOTS] = reinterpret_cast<uint32_t(*)[2][SLOTS]>(walk_smem + ORDERED_WARPS * sizeof(OrderedShared));
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const size_t t = ((size_t)blockIdx.x * ORDERED_WARPS + warp) * 32 + lane;
  const bool valid = t < (LIST ? (size_t)*list_n : n);
  const size_t i = LIST ? (valid ? (size_t)list[t] : 0) : t;
  const unsigned group = __ballot_sync(FULL, valid);
  if (group == 0) return;
  const uint32_t root = group_box(group, i, w);
  if (!walk_ordered(words, root)) return;
  OrderedShared& sh = shared[warp];
  const float4 xi = valid ? __ldg(x4 + i) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  const float x0 = xi.x, x1 = xi.y, x2 = xi.z;
  const uint32_t self = (uint32_t)i;

  // Bounding box of the warp's particles (centre cg, half extent hg), for a conservative
  // warp-level prune test: a node farther than r_cut + sqrt(3) half from the whole box is pruned
  // by every lane, whose own test is then skipped.
  float lo0 = valid ? x0 : INFINITY, lo1 = valid ? x1 : INFINITY, lo2 = valid ? x2 : INFINITY;
  float hi0 = valid ? x0 : -INFINITY, hi1 = valid ? x1 : -INFINITY, hi2 = valid ? x2 : -INFINITY;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo0 = fminf(lo0, __shfl_xor_sync(FULL, lo0, o));
    lo1 = fminf(lo1, __shfl_xor_sync(FULL, lo1, o));
    lo2 = fminf(lo2, __shfl_xor_sync(FULL, lo2, o));
    hi0 = fmaxf(hi0, __shfl_xor_sync(FULL, hi0, o));
    hi1 = fmaxf(hi1, __shfl_xor_sync(FULL, hi1, o));
    hi2 = fmaxf(hi2, __shfl_xor_sync(FULL, hi2, o));
  }
  if (lane == 0) {
    const float tol = 1e-5f * w.box;  // far above the rounding of positions and differences
    sh.box_c = make_float4(0.5f * (lo0 + hi0), 0.5f * (lo1 + hi1), 0.5f * (lo2 + hi2), 0.0f);
    sh.box_h = make_float4(0.5f * (hi0 - lo0) + tol, 0.5f * (hi1 - lo1) + tol, 0.5f * (hi2 - lo2) + tol, 0.0f);
  }
  // Accumulators of the even and odd pairs (x: even pairs and accepted nodes).
  float2 A0 = make_float2(0.0f, 0.0f), A1 = A0, A2 = A0;
  uint32_t n_pairs = 0, n_accepts = 0, n_cand = 0;

  // A step of the walk handles up to SLOTS nodes, one per lane: one or more stack entries (each the
  // children of an opened node, with the mask of the lanes that opened it) placed in consecutive
  // slots. `mine` holds the slots this lane walks. Lane c copies slot c's three records into shared
  // buffer `cur` asynchronously; the next step's copies are in flight while the current step is
  // summed. The walk starts at the root: node 0, or in a batch of boxes the root of the warp's box
  // (nodes 0 .. boxes - 1).
  uint32_t b_count = 1, mine = (group >> lane) & 1u;
  int cur = 0;
  if (lane == 0) {
    cp_async16(&sh.geo[0][0], geo + root);
    cp_async16(&sh.mass[0][0], mass + root);
    cp_async16(&sh.link[0][0], link + root);
    if constexpr (QUAD) node_ids[warp][0][0] = root;
  }
  int sp = 0;
  for (;;) {
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncwarp();
    const float4* bgeo = sh.geo[cur];
    const float4* bmass = sh.mass[cur];
    const uint4* blink = sh.link[cur];

    // Warp-level prune test, lane c for node c. It applies where no lane can need a periodic
    // image (|centre - x| < 0.49 L on every axis for the whole box), so that the lanes' own
    // distances are the raw differences; it keeps a node unless even the box's nearest point is
    // beyond r_cut + sqrt(3) half by a relative margin of 1e-5.
    bool keep = false, far_edge = false, direct = false, inside = false;
    if ((uint32_t)lane < b_count) {
      const float4 bc = sh.box_c, bh = sh.box_h, pg = bgeo[lane];
      const float e0 = fabsf(pg.x - bc.x), e1 = fabsf(pg.y - bc.y), e2 = fabsf(pg.z - bc.z);
      const float mr = __fadd_rn(w.r_cut, __fmul_rn(SQRT_3, pg.w));
      const float lhs = __fmul_rn(2.0f, pg.w), l2 = __fmul_rn(lhs, lhs);
      sh.pre[lane] = make_float4(__fmul_rn(mr, mr), l2, 1e-5f * l2, lhs);
      direct = (blink[lane].w & 1u) == 0u;
      keep = true;
      const float emax = fmaxf(e0 + bh.x, fmaxf(e1 + bh.y, e2 + bh.z));
      if (emax < w.guard) {
        const float g0 = fmaxf(e0 - bh.x, 0.0f), g1 = fmaxf(e1 - bh.y, 0.0f), g2 = fmaxf(e2 - bh.z, 0.0f);
        keep = !(g0 * g0 + g1 * g1 + g2 * g2 > mr * mr * 1.00001f);
      }
      // No lane needs a periodic image for this node: every difference between a lane's
      // particle and the node's centre, centre of mass or particles (all inside the cube) is
      // below 0.49 L on every axis.
      far_edge = emax + pg.w < w.guard;
      // every point of the cube is within r_cut of the box
      const float h0 = fmaxf(e0 + pg.w - bh.x, 0.0f), h1 = fmaxf(e1 + pg.w - bh.y, 0.0f), h2 = fmaxf(e2 + pg.w - bh.z, 0.0f);
      inside = h0 * h0 + h1 * h1 + h2 * h2 <= w.cut2;
    }
    const uint32_t whole = __ballot_sync(FULL, inside);
    const uint32_t cand = __ballot_sync(FULL, keep);
    const uint32_t nwall = __ballot_sync(FULL, far_edge);
    const uint32_t dbits = __ballot_sync(FULL, direct);
    __syncwarp();

    // Classify every remaining node of this lane for its particle: prune, direct sum, accept or open.
    uint32_t dmask = 0, nwmask = 0, amask = 0, omask = 0;
    const uint32_t todo = cand & mine;
    if ((todo & ~nwall) == 0u) {
      // No node of the step involves a periodic image: raw differences.
      for (uint32_t rem = todo; rem; rem &= rem - 1) {
        const uint32_t c = __ffs(rem) - 1;
        const float4 G = bgeo[c], P = sh.pre[c];
        const float t0 = __fsub_rn(G.x, x0), t1 = __fsub_rn(G.y, x1), t2 = __fsub_rn(G.z, x2);
        if (norm2(t0, t1, t2) > P.x) continue;
        if ((dbits >> c) & 1u) {
          dmask |= 1u << c;
          continue;
        }
        const float4 M = bmass[c];
        const float s0 = __fsub_rn(M.x, x0), s1 = __fsub_rn(M.y, x1), s2 = __fsub_rn(M.z, x2);
        if (accept_node_sq(norm2(s0, s1, s2), P.y, P.z, P.w, w))
          amask |= 1u << c;
        else
          omask |= 1u << c;
      }
      nwmask = dmask;
    } else {
      for (uint32_t rem = todo; rem; rem &= rem - 1) {
        const uint32_t c = __ffs(rem) - 1;
        const float4 G = bgeo[c], P = sh.pre[c];
        float t0 = __fsub_rn(G.x, x0), t1 = __fsub_rn(G.y, x1), t2 = __fsub_rn(G.z, x2);
        // every source y of the node lies in [centre - half, centre + half]
        const bool nowrap = fmaxf(fabsf(t0), fmaxf(fabsf(t1), fabsf(t2))) + G.w < w.guard;
        min_image3(t0, t1, t2, w);
        if (norm2(t0, t1, t2) > P.x) continue;
        if ((dbits >> c) & 1u) {
          // children[0] == NO_CHILD: direct sum over the node's particles (tree.rs:286-298)
          dmask |= 1u << c;
          nwmask |= (uint32_t)nowrap << c;
          continue;
        }
        const float4 M = bmass[c];
        float s0 = __fsub_rn(M.x, x0), s1 = __fsub_rn(M.y, x1), s2 = __fsub_rn(M.z, x2);
        min_image3(s0, s1, s2, w);
        if (accept_node_sq(norm2(s0, s1, s2), P.y, P.z, P.w, w))
          amask |= 1u << c;
        else
          omask |= 1u << c;
      }
    }

    // Push the opened nodes' children as new stack entries (any order gives each lane the same
    // set of interactions; only the order of its sums differs). Higher slots go deeper into the
    // stack, so that the entries popped first, which fill the lowest slots, have their children
    // popped first again.
    const uint32_t ouni = __reduce_or_sync(FULL, omask);
    if (ouni) {
      uint32_t opened_by = 0;
      for (uint32_t rem = ouni; rem; rem &= rem - 1) {
        const int c = __ffs(rem) - 1;
        const uint32_t b = __ballot_sync(FULL, (omask >> c) & 1u);
        if (lane == c) opened_by = b;
      }
      const int npush = __popc(ouni);
      // (node indices above 29 bits, trees of more than 2^28 particles, do not fit an entry)
      const bool wide = __any_sync(FULL, ((ouni >> lane) & 1u) && (blink[lane].z >> FIRST_BITS) != 0u);
      if (sp + npush > ORDERED_STACK_CAP || wide) {
        if (lane == 0) dev_fail(st, DEV_STACK_OVERFLOW, sp);
        break;
      }
      if ((ouni >> lane) & 1u) {
        const uint4 L = blink[lane];
        const int slot = sp + __popc(ouni >> lane) - 1;
        sh.stack[slot] = make_uint2(L.z | ((uint32_t)(__popc(L.w & 0xFFu) - 1) << FIRST_BITS), opened_by);
      }
      sp += npush;
      __syncwarp();
    }

    // Pop the next step: the top entry, and while the stack is shallow, further entries as long as
    // they fit in the slots. Its copies complete during the work below.
    uint32_t nx_count = 0, nx_mine = 0;
    if (sp > 0) {
      const bool merge = sp <= ORDERED_MERGE_SP;
      for (;;) {
        const uint2 e = sh.stack[--sp];
        const uint32_t first = e.x & ((1u << FIRST_BITS) - 1u), cnt = (e.x >> FIRST_BITS) + 1u;
        if ((uint32_t)lane >= nx_count && (uint32_t)lane < nx_count + cnt) {
          const uint32_t node = first + ((uint32_t)lane - nx_count);
          cp_async16(&sh.geo[cur ^ 1][lane], geo + node);
          cp_async16(&sh.mass[cur ^ 1][lane], mass + node);
          cp_async16(&sh.link[cur ^ 1][lane], link + node);
          if constexpr (QUAD) node_ids[warp][cur ^ 1][lane] = node;
        }
        if ((e.y >> lane) & 1u) nx_mine |= bit_span(nx_count, cnt);
        nx_count += cnt;
        if (!merge || sp == 0 || nx_count + (sh.stack[sp - 1].x >> FIRST_BITS) + 1u > (uint32_t)SLOTS) break;
      }
    }

    // Accepted centres of mass (tree.rs:299-305).
    for (; amask; amask &= amask - 1) {
      const int c = __ffs(amask) - 1;
      const float4 M = bmass[c];
      float s0 = __fsub_rn(M.x, x0), s1 = __fsub_rn(M.y, x1), s2 = __fsub_rn(M.z, x2);
      min_image3(s0, s1, s2, w);
      const float f = pair_factor(norm2(s0, s1, s2), -M.w, w, far);
      A0.x = fmaf(-s0, f, A0.x);
      A1.x = fmaf(-s1, f, A1.x);
      A2.x = fmaf(-s2, f, A2.x);
      if constexpr (QUAD) {
        const size_t node = node_ids[warp][cur][c];
        quad_term(s0, s1, s2, __ldg(quad + 2 * node), __ldg(quad + 2 * node + 1), w, A0, A1, A2);
      }
      ++n_accepts;
    }

    // Direct sums: the sources of all direct nodes of the step, concatenated in slot order, in
    // chunks of 32.
    const uint32_t dset = __reduce_or_sync(FULL, dmask);
    if (dset) {
      uint32_t cnt = 0, first = 0;
      if ((dset >> lane) & 1u) {
        const uint4 L = blink[lane];
        cnt = L.y - L.x;
        first = L.x;
      }
      uint32_t end = cnt;  // inclusive prefix sum over the slots
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(FULL, end, o);
        if (lane >= o) end += v;
      }
      sh.dbeg[lane] = end - cnt;
      sh.dend[lane] = end;
      sh.dsrc[lane] = first;
      const uint32_t total = __shfl_sync(FULL, end, 31);
      __syncwarp();
      // This lane's candidates, and its own particle's position in the concatenation (j != i).
      uint32_t selfpos = 0xffffffffu;
      for (uint32_t rem = dmask; rem; rem &= rem - 1) {
        const int c = __ffs(rem) - 1;
        const uint32_t b0 = sh.dbeg[c], e0 = sh.dend[c], f0 = sh.dsrc[c];
        n_cand += e0 - b0;
        if (self - f0 < e0 - b0) selfpos = b0 + (self - f0);
      }
      const bool wrap = (dmask & ~nwmask) != 0u, all_near = (dset & ~whole) == 0u;
      uint32_t open_d = dmask;  // this lane's direct nodes not yet wholly behind the current chunk
      for (uint32_t base = 0; base < total; base += 32) {
        // Lane q loads source base + q: node c, the last with dbeg <= base + q (binary search).
        const uint32_t g = base + (uint32_t)lane;
        bool near = all_near;
        if (g < total) {
          int c = 0;
#pragma unroll
          for (int step = 16; step > 0; step >>= 1)
            if (sh.dend[c + step - 1] <= g) c += step;
          const float4 y = __ldg(x4 + sh.dsrc[c] + (g - sh.dbeg[c]));
          sh.nx[lane] = -y.x;
          sh.ny[lane] = -y.y;
          sh.nz[lane] = -y.z;
          if (!all_near) {
            const float4 bc = sh.box_c, bh = sh.box_h;
            const float g0 = axis_gap(y.x, bc.x, bh.x, 0.0f, w.box), g1 = axis_gap(y.y, bc.y, bh.y, 0.0f, w.box),
                        g2 = axis_gap(y.z, bc.z, bh.z, 0.0f, w.box);
            near = !(g0 * g0 + g1 * g1 + g2 * g2 > w.cull2);
          }
        }
        const uint32_t reach = __ballot_sync(FULL, near);  // the sources within r_cut of the warp's box
        // `live`: the chunk positions of this lane's direct nodes, without its own particle.
        const uint32_t top = base + 32u;
        uint32_t live = 0;
        while (open_d) {
          const int c = __ffs(open_d) - 1;
          const uint32_t b0 = sh.dbeg[c], e0 = sh.dend[c];
          if (b0 >= top) break;
          const uint32_t lo = max(b0, base), hi = min(e0, top);
          live |= bit_span(lo - base, hi - lo);
          if (e0 > top) break;
          open_d &= open_d - 1;
        }
        if (selfpos - base < 32u) live &= ~(1u << (selfpos - base));
        __syncwarp();
        live &= reach;
        if (live) {
          const uint32_t pairs = (wrap ? ordered_pairs<true>(sh, reach, x0, x1, x2, w)
                                       : ordered_pairs<false>(sh, reach, x0, x1, x2, w)) & live;
          n_pairs += __popc(pairs);
          if (wrap)
            chunk_forces<true>(sh, pairs, x0, x1, x2, w, far, A0, A1, A2);
          else
            chunk_forces<false>(sh, pairs, x0, x1, x2, w, far, A0, A1, A2);
        }
        __syncwarp();
      }
    }
    if (nx_count == 0) break;
    b_count = nx_count;
    mine = nx_mine;
    cur ^= 1;
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  // tree.rs:61-66 multiplies every pair by the coupling K; here the unit-coupling sum is scaled once
  const float kk = k_dev ? *k_dev : w.k;
  const float a0 = kk * (A0.x + A0.y), a1 = kk * (A1.x + A1.y), a2 = kk * (A2.x + A2.y);
  if (valid) {
    if (accumulate) {
      acc3[3 * i] = __fadd_rn(acc3[3 * i], a0);
      acc3[3 * i + 1] = __fadd_rn(acc3[3 * i + 1], a1);
      acc3[3 * i + 2] = __fadd_rn(acc3[3 * i + 2], a2);
    } else {
      acc3[3 * i] = a0;
      acc3[3 * i + 1] = a1;
      acc3[3 * i + 2] = a2;
    }
  }
  if (counters) {
    unsigned long long p = n_pairs, a = n_accepts, c = n_cand;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      p += __shfl_xor_sync(FULL, p, o);
      a += __shfl_xor_sync(FULL, a, o);
      c += __shfl_xor_sync(FULL, c, o);
    }
    if (lane == 0) {
      atomicAdd(&counters[0], p);
      atomicAdd(&counters[1], a);
      atomicAdd(&counters[2], c);
    }
  }
}

// ------------------------------------------------------------------ host launch

// Fitted pair-force coefficients of one tree's last split (refitted when the split changes; a
// simulation's split is fixed, so its first step uploads them and later steps, captured graphs
// included, only read them).
struct FitCache {
  float r_split = -1.0f, r_cut = -1.0f;
  SFit fit{};
  std::vector<float> far;
  DevBuf far_dev;
};

void tree_walk_free(TreeNodes& t) {
  FitCache* fc = static_cast<FitCache*>(t.walk_fit);
  if (fc) {
    release(fc->far_dev);
    delete fc;
  }
  t.walk_fit = nullptr;
}

// Warps that walk one group. A batch goes by the groups of one box, so that a box's sums are those of its own
// simulation, up to BATCH_FILL.
static int walk_team(const TreeNodes& t, size_t n) {
  const size_t groups = (n + 31) / 32, box_groups = t.n_box ? (t.n_box + 31) / 32 : groups;
  const int box_team = box_groups * 4 <= WALK_FILL ? 4 : (box_groups * 2 <= WALK_FILL ? 2 : 1);
  return groups * box_team <= BATCH_FILL ? box_team : 1;
}

int tree_walk_warps(const TreeNodes& t, size_t n) {
  if (t.has_quad) return 4;
  return std::max(walk_team(t, n), t.walk_warps == 2 || t.walk_warps == 8 ? t.walk_warps : 4);
}

void launch_tree_walk(const TreeNodes& t, size_t n, float box, const cpm_force_split& split,
                      float k, float* acc3, int accumulate, TreeCounters* counters, DevStatus* st, cudaStream_t s,
                      const float* k_dev, const uint32_t* list, const uint32_t* list_n) {
  if (n == 0) return;
  TreeNodes& tm = const_cast<TreeNodes&>(t);
  if (!tm.walk_fit) tm.walk_fit = new FitCache();
  FitCache& fc = *static_cast<FitCache*>(tm.walk_fit);
  if (fc.r_split != split.r_split || fc.r_cut != split.r_cut || !fc.far_dev.p) {
    fc.fit = make_fit(split.r_split, split.r_cut, fc.far);
    if (ensure(fc.far_dev, fc.far.size() * sizeof(float)) != cudaSuccess) return;
    cudaMemcpy(fc.far_dev.p, fc.far.data(), fc.far.size() * sizeof(float), cudaMemcpyHostToDevice);
    fc.r_split = split.r_split;
    fc.r_cut = split.r_cut;
  }
  uint32_t* words = tree_words(tm, n);

  WalkParams w;
  w.box = box;
  w.guard = 0.49f * box;
  w.r_cut = split.r_cut;
  w.cut2 = split.r_cut * split.r_cut;
  w.theta = split.theta;
  w.theta2 = split.theta * split.theta;
  w.inv_two_rs = (float)(1.0 / (2.0 * (double)split.r_split));
  w.eps2 = split.softening * split.softening;
  w.k = k;
  w.n_box = t.n_box;
  w.fit = fc.fit;
  auto dup = [](float v) { return make_float2(v, v); };
  w.p2.tiny = dup(1e-30f);
  const double inv_two_rs = 1.0 / (2.0 * (double)split.r_split);
  w.cut_lo = w.cut2 * 0.999998f;
  w.cut_hi = w.cut2 * 1.000002f + 1e-37f;
  w.inv_box = 1.0f / box;
  // a nearest image is off by less than 1e-6 L per axis, so its r^2 by less than 4e-6 L r
  w.cut_image = w.cut2 + 1e-5f * box * (split.r_cut + 1e-5f * box);
  w.cull2 = w.cut2 * 1.0001f;
  w.wrap_lo = 0.51f * box;
  w.wrap_hi = 1.49f * box;
  w.fit_covers = (double)split.r_cut * 1.00001 * inv_two_rs <= (double)fc.fit.umax0;
  w.p2.scale0 = dup((float)((double)fc.fit.scale0 * inv_two_rs));
  w.p2.offset0 = dup(fc.fit.offset0);
  for (int j = 0; j <= FIT_DEG; ++j) w.p2.c0[j] = dup(fc.fit.c0[j]);
  w.p2.exp_scale = dup((float)(-1.4426950408889634 * inv_two_rs * inv_two_rs));
  w.p2.eps2 = dup(w.eps2);
  w.ordered.tiny = dup(1e-30f);
  w.ordered.inv_two_rs = dup(w.inv_two_rs);
  w.ordered.scale0 = dup(fc.fit.scale0);
  w.ordered.offset0 = dup(fc.fit.offset0);
  for (int j = 0; j <= FIT_DEG; ++j) w.ordered.c0[j] = dup(fc.fit.c0[j]);
  w.ordered.neg_log2e = dup(-1.44269504f);
  w.ordered.eps2 = dup(w.eps2);
  w.ordered.neg_m = dup(-1.0f);
  const size_t groups = (n + 31) / 32;
  const bool ordered = t.trajectories && (t.n_box ? t.n_box : n) <= ORDERED_PARTICLES;
  const int team = walk_team(t, n), warps = tree_walk_warps(t, n);
  unsigned blocks = (unsigned)((groups * team + warps - 1) / warps);
  auto pick = [&](auto lists, auto skips) {
    constexpr bool L = decltype(lists)::value, S = decltype(skips)::value;
    return t.has_quad   ? k_tree_walk<true, L, 4, S>
           : warps == 2 ? k_tree_walk<false, L, 2, S>
           : warps == 8 ? k_tree_walk<false, L, 8, S>
                        : k_tree_walk<false, L, 4, S>;
  };
  const std::true_type yes;
  const std::false_type no;
  auto kernel = list ? (ordered ? pick(yes, yes) : pick(yes, no)) : (ordered ? pick(no, yes) : pick(no, no));
  const size_t smem = (size_t)warps * (sizeof(WalkShared) + (t.has_quad ? SLOTS * sizeof(uint32_t) : 0));
  if (smem > 48 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (team == 1) {  // as many blocks as fit on the chip at once
    cudaMemsetAsync(words + WALK_TICKET, 0, sizeof(uint32_t), s);
    int per_sm = 1;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, warps * 32, smem) == cudaSuccess && per_sm > 0)
      blocks = std::min(blocks, (unsigned)per_sm * 148u);
  }
  count_launch();
  kernel<<<blocks, warps * 32, smem, s>>>(static_cast<const uint4*>(t.link.p), static_cast<const float4*>(t.geo.p),
                                         static_cast<const float4*>(t.mass.p), as<float4>(tm.x4), n, w,
                                         static_cast<const float*>(fc.far_dev.p), acc3, accumulate,
                                         reinterpret_cast<unsigned long long*>(counters), st, k_dev, list, list_n,
                                         t.has_quad ? static_cast<const float4*>(t.quad.p) : nullptr, words, team);
  if (ordered) {
    auto second = t.has_quad ? (list ? k_walk_ordered<true, true> : k_walk_ordered<true, false>)
                             : (list ? k_walk_ordered<false, true> : k_walk_ordered<false, false>);
    const size_t smem2 = ORDERED_WARPS * (sizeof(OrderedShared) + (t.has_quad ? 2 * SLOTS * sizeof(uint32_t) : 0));
    if (smem2 > 48 * 1024) cudaFuncSetAttribute(second, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem2);
    count_launch();
    second<<<(unsigned)((groups + ORDERED_WARPS - 1) / ORDERED_WARPS), ORDERED_WARPS * 32, smem2, s>>>(
        static_cast<const uint4*>(t.link.p), static_cast<const float4*>(t.geo.p), static_cast<const float4*>(t.mass.p),
        as<float4>(tm.x4), n, w, static_cast<const float*>(fc.far_dev.p), acc3, accumulate,
        reinterpret_cast<unsigned long long*>(counters), st, k_dev, list, list_n,
        t.has_quad ? static_cast<const float4*>(t.quad.p) : nullptr, words);
  }
}

float quad_half_bound(const cpm_force_split& split) {
  const double th = split.theta;
  const double den = 2.0 - 2.0 * std::sqrt(3.0) * th;
  if (!(den > 0.0)) return INFINITY;
  return (float)(1.01 * th * (double)split.r_cut / den);
}

}  // namespace cpm

using namespace cpm;

// Self-check of the fitted pair kernel: max relative error of e^{-u^2} R_fit(u) (f32 Horner, host)
// against the double-precision S(u) over u in [0, u_max], u_max = r_cut / (2 r_split), on `samples`
// points. Host only; no device is needed.
extern "C" int cpm_walk_kernel_fit_error(float r_split, float r_cut, int samples, double* max_rel_err) {
  if (!(r_split > 0.0f) || !(r_cut > 0.0f) || samples < 2 || !max_rel_err)
    return set_error(nullptr, CPM_E_INVALID, "cpm_walk_kernel_fit_error: bad arguments");
  std::vector<float> far;
  const SFit f = make_fit(r_split, r_cut, far);
  const double umax = std::min(U_NEGLIGIBLE, (double)r_cut / (2.0 * (double)r_split));
  double worst = 0.0;
  for (int q = 0; q < samples; ++q) {
    const float u = (float)(umax * q / (samples - 1));
    const double ud = (double)u;
    const double exact = std::erfc(ud) + 2.0 * ud / std::sqrt(M_PI) * std::exp(-ud * ud);
    const double got = std::exp(-ud * ud) * (double)r_fit_host(f, far, u);
    worst = std::max(worst, std::fabs(got - exact) / exact);
  }
  *max_rel_err = worst;
  return CPM_OK;
}
