// FP32 tiled pair kernels of the force path.
//
//   born pass   -- descreening integral I_i = sum_j h(r_ij, rho~_i, s_j rho~_j)
//                  (energy/src/gb.rs:268-324 + pairwise_descreening :347-369)
//   force pass  -- LJ + reaction-field Coulomb within the nonbonded cutoff
//                  (energy/src/forces_nonbonded.rs:196-232) fused with the
//                  frozen-radii GB pair force within the GB cutoff
//                  (energy/src/forces_gb.rs:82-111), far-field tiles only;
//                  near-field tiles (exclusions, 1-4 pairs) go to the FP64
//                  kernel in pair_fp64.cu.
//
// Layout.  One warp owns one 32-atom i-tile and a CTA of W warps owns W
// consecutive tiles (W = 8 or 4, a launch variant).  The CTA walks a list of
// j-tiles (the tiles from
// its first tile on -- each unordered tile pair once); thread 0 streams them
// into shared memory with 1-D TMA bulk copies (two stages in flight, mbarrier
// completion, bounded waits).  The per-atom FP32 arrays are tile-SoA (four
// 32-float columns per tile), so one 16-byte shared load is one column of
// four consecutive j atoms, which feeds Blackwell's packed FP32x2 arithmetic
// directly: the force pass evaluates two j atoms per instruction, the Born
// pass the two directions h_ij / h_ji of one pair.  The j-side sums (Newton's
// third law) are formed by a warp reduce-scatter, summed over the CTA's warps
// in shared memory in a fixed order and added to 64-bit fixed-point
// accumulators; the i side accumulates FP32 per tile and FP64 across tiles.
// Every sum therefore has a fixed order and results are bit-reproducible.
//
// Launch variants (PairLaunch): how many i-tiles a CTA owns and how (the
// split kernels: one, four warps sharing it; k_born and k_force: one per warp;
// k_force_quad: four per warp), the CTAs per SM the register budget is sized
// for, and either one CTA per work item (the hardware assigns CTAs to SMs as
// they free up) or a persistent grid of resident CTAs that take items from an
// atomic queue.  The engine picks by tile counts (default_launch) or its
// autotuner times them on the actual systems; every variant computes the same
// pair terms.  With cutoffs shape 0 keeps one order of every sum, by two sets
// of kernels (k_born_pair).
//
// Tile pairs are classed by the gap between their bounding spheres: distant
// ones take shorter forms of the same sums (fewer series terms, the far GB
// form without its exponential), with every pair's condition implied by the
// gap.  64 x 4 694 atoms, all pairs, B200: Born 1.265 -> 0.668 ms by the
// tiers and shapes (k_born, 64 registers, FMA pipe 62 % busy) -> 0.640 with the
// tile offsets taken once per stage and one barrier per stage; force 1.105 ->
// 0.843 (k_force_quad, 162 registers, 12 warps per SM, FMA pipe 56 %) -> 0.817;
// one 300-atom system 58 -> 5 and 32 -> 5 us (split).
//
// Positions are FP32 offsets from a per-tile FP64 origin; the origin
// difference of a tile pair is formed in FP64 once per tile, so |dx| keeps
// ~1e-7 relative accuracy in chains 1000 A long.
#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "pair_kernels.cuh"

namespace ogk {

namespace {

// Groups of four j atoms in flight per lane (measured best on B200 for
// 64 x 4.7k-atom systems).
#ifndef OG_BORN_UNROLL
#define OG_BORN_UNROLL 1
#endif
#ifndef OG_FORCE_UNROLL
#define OG_FORCE_UNROLL 2
#endif
#define OG_PRAGMA(x) _Pragma(#x)
#define OG_UNROLL(n) OG_PRAGMA(unroll n)

constexpr int kStageTiles = 4;    // j-tiles per pipeline stage
constexpr int kStageFloats = kStageTiles * 128;
constexpr uint32_t kTileBytes = 128 * sizeof(float);
constexpr float kLog2e = 1.4426950408889634f;

__device__ __forceinline__ float2 bc(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float fast_rcp(float x) { return __fdividef(1.0f, x); }
// 1 / x as the one special-function instruction (1 ulp; no range handling).
__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// Reduce-scatter over the warp of four per-lane values v0..v3 (contributions
// to four consecutive j atoms): afterwards every lane of the 8-lane group
// g = lane >> 3 holds the warp total of v_g.  Six shuffles instead of the
// twenty of four separate butterflies; the order is fixed.
__device__ __forceinline__ float reduce_scatter4(float v0, float v1, float v2, float v3, int lane) {
  const bool hi16 = (lane & 16) != 0;
  float k0 = hi16 ? v2 : v0, k1 = hi16 ? v3 : v1;   // kept: j = 2*hi16 + {0, 1}
  const float s0 = hi16 ? v0 : v2, s1 = hi16 ? v1 : v3;
  k0 += __shfl_xor_sync(0xffffffffu, s0, 16);
  k1 += __shfl_xor_sync(0xffffffffu, s1, 16);
  const bool hi8 = (lane & 8) != 0;
  float k = hi8 ? k1 : k0;                           // kept: j = 2*hi16 + hi8 = lane >> 3
  k += __shfl_xor_sync(0xffffffffu, hi8 ? k0 : k1, 8);
  k += __shfl_xor_sync(0xffffffffu, k, 4);
  k += __shfl_xor_sync(0xffffffffu, k, 2);
  k += __shfl_xor_sync(0xffffffffu, k, 1);
  return k;
}

// ------------------------------------------------------------- staging
// Stage s of a work item is the CTA's stage g0 + s overall: buffer and
// mbarrier (g0 + s) & 1, wait parity ((g0 + s) >> 1) & 1, so a persistent
// CTA keeps alternating its two barriers across items.
template <int kST = kStageTiles>
struct StagerT {
  const int32_t* jlist;
  int j_begin, j_end, n_stages;
  uint64_t* bar;
  uint32_t g0;
  template <int kArrays>
  __device__ __forceinline__ void issue(int s, float (*buf)[kArrays][kST * 128], const float* const* src) const {
    const int b = (g0 + s) & 1;
    const int t0 = j_begin + s * kST;
    const int cnt = min(kST, j_end - t0);
    mbar_arrive_expect_tx(&bar[b], static_cast<uint32_t>(cnt) * kTileBytes * kArrays);
    for (int t = 0; t < cnt; ++t) {
      const size_t base = static_cast<size_t>(jlist[t0 + t]) * 128;
#pragma unroll
      for (int c = 0; c < kArrays; ++c) bulk_g2s(&buf[b][c][t * 128], src[c] + base, kTileBytes, &bar[b]);
    }
  }
};

using Stager = StagerT<>;

// Adds the stage's j partials (s_part[w][c][q], summed over warps in a fixed
// order) to the fixed-point accumulators.
template <int W, int kComps, int kST = kStageTiles>
__device__ __forceinline__ void flush_j(const PairArgs& a, const int* jt, int cnt,
                                        float (*s_part)[kComps][kST * kTile], unsigned long long* const* dst,
                                        double scale) {
  for (int q = threadIdx.x; q < cnt * kTile; q += blockDim.x) {
    const int j = jt[q / kTile] * kTile + (q % kTile);
    if (!a.atom_valid[j]) continue;
    float v[kComps];
    bool any = false, finite = true;
#pragma unroll
    for (int c = 0; c < kComps; ++c) {
      float sum = 0.0f;
#pragma unroll
      for (int w = 0; w < W; ++w) sum += s_part[w][c][q];
      v[c] = sum;
      any = any || sum != 0.0f;
      finite = finite && isfinite(sum);
    }
    if (!any) continue;
    if (!finite) atomicOr(a.sys_nonfinite + a.atom_sys[j], 1);
#pragma unroll
    for (int c = 0; c < kComps; ++c) add_fixed(dst[c] + j, static_cast<double>(v[c]), scale);
  }
}

// Lower bound (A) on the distance of any atom pair of two tiles, from their
// bounding spheres; the margin covers the FP32 rounding.
__device__ __forceinline__ float tile_gap(double4 oi, double4 oj) {
  const float dx = static_cast<float>(oj.x - oi.x), dy = static_cast<float>(oj.y - oi.y),
              dz = static_cast<float>(oj.z - oi.z);
  const float d = sqrtf(fmaf(dx, dx, fmaf(dy, dy, dz * dz)));
  return d * (1.0f - 1e-6f) - static_cast<float>(oi.w + oj.w) - 1e-3f;
}

// A stage's j-tiles as the block's kI i-tiles see them: the offset of the
// tiles' origins (x, y, z: j minus i) and the gap between their spheres (w),
// one thread per (i-tile, j-tile) a stage ahead.  (Every warp for itself, for
// each tile pair: 35 to 100 instructions of 900 and two dependent loads; 675
// against 650 us of the Born pass and 846 against 819 of the force pass for 64
// chains of 300 residues.)
template <int kI>
struct StageTilesT {
  int jt[kStageTiles];
  float4 off[kStageTiles][kI];
};
template <int kI>
__device__ __forceinline__ void stage_tiles(const PairArgs& a, const PairWork& w, int stage, StageTilesT<kI>& s) {
  const int t = threadIdx.x % kStageTiles, q = threadIdx.x / kStageTiles;
  const int at = w.j_begin + stage * kStageTiles + t;
  if (at >= w.j_end || q >= w.n_i_tiles) return;  // at most kI i-tiles
  const int jt = a.jlist[at];
  const double4 oj = a.origin[jt], oi = a.origin[w.i_tile0 + q];
  s.off[t][q] = make_float4(static_cast<float>(oj.x - oi.x), static_cast<float>(oj.y - oi.y),
                            static_cast<float>(oj.z - oi.z), tile_gap(oi, oj));
  if (q == 0) s.jt[t] = jt;
}

// ---------------------------------------------------------------- Born
// origami's pairwise_descreening (gb.rs:347-369) is
//   h = 1/2 (1/L - 1/U) + (r/4)(1/U^2 - 1/L^2) + ln(L/U)/(2r)
//       + (s^2 - r^2)/(4r) (1/U^2 - 1/L^2),      L = max(rho_i, r - s), U = r + s.
// Its terms cancel to O(s^3/r^4) for distant pairs, so FP32 evaluation of the
// closed form loses most digits there.  On the non-overlapping branch
// (L = r - s) the expression is, exactly, the series in x = s/r
//   h = -(x^3 / r) * sum_{k>=1} k(2k-1)/(2k+1) x^(2(k-1))
// (expand 1/(1-x^2), 1/(1-x^2)^2 and atanh x = -ln((1-x)/(1+x))/2 and collect
// powers).  For x < 1/4 eight terms leave a truncation error below 1e-8
// relative, under FP32 rounding.  A j atom takes that path when every lane's
// pair is distant in both directions (warp vote); otherwise all lanes use the
// closed form with term2 + term4 folded into (s^2 / 4r)(1/U^2 - 1/L^2) and
// ln(L/U) = log1p((L - U)/U).
constexpr float kSeriesMaxX = 0.25f;

// Series for the two directions at once: x = (s_j, s_i) / r.
__device__ __forceinline__ float2 descreen_series2(float2 x, float inv_r) {
  const float2 xx = mul2(x, x);
  float2 p = bc(120.0f / 17.0f);
  p = fma2(p, xx, bc(91.0f / 15.0f));
  p = fma2(p, xx, bc(66.0f / 13.0f));
  p = fma2(p, xx, bc(45.0f / 11.0f));
  p = fma2(p, xx, bc(28.0f / 9.0f));
  p = fma2(p, xx, bc(15.0f / 7.0f));
  p = fma2(p, xx, bc(6.0f / 5.0f));
  p = fma2(p, xx, bc(1.0f / 3.0f));
  return mul2(mul2(mul2(xx, x), bc(-inv_r)), p);
}

// Closed form, valid on both branches.
__device__ __forceinline__ float descreen_closed(float r, float inv_r, float rho, float sr) {
  const bool overlap = (r - sr) < rho;
  const float L = overlap ? rho : r - sr;
  const float U = r + sr;
  const float inv_l = fast_rcp(L), inv_u = fast_rcp(U);
  const float lg = log1pf((overlap ? rho - U : -2.0f * sr) * inv_u);
  const float d2 = inv_u * inv_u - inv_l * inv_l;
  const float h = 0.5f * (inv_l - inv_u) + (sr * sr) * (0.25f * inv_r) * d2 + (0.5f * inv_r) * lg;
  return (!(r + sr <= rho) && (U > 0.0f) && (L > 0.0f)) ? h : 0.0f;
}

// (h_ij, h_ji) for one pair; on = inside the Born cutoff and not coincident.
__device__ __forceinline__ float2 born_pair(float dx, float dy, float dz, float rho_i, float s_i, float rho_j,
                                           float s_j, float c2) {
  const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
  const float inv_r = rsqrtf(r2);
  const float r = r2 * inv_r;
  const float2 x = mul2(make_float2(s_j, s_i), bc(inv_r));
  const bool far = (x.x < kSeriesMaxX) && (x.y < kSeriesMaxX) && (r - s_j >= rho_i) && (r - s_i >= rho_j);
  float2 h;
  if (__all_sync(0xffffffffu, far)) {
    h = descreen_series2(x, inv_r);
  } else {
    h = make_float2(descreen_closed(r, inv_r, rho_i, s_j), descreen_closed(r, inv_r, rho_j, s_i));
  }
  const bool on = (r2 <= c2) && (r2 >= 1e-18f);
  return on ? h : make_float2(0.0f, 0.0f);
}

// --------------------------------------------------- Born, distant tiles
// A tile pair whose spheres leave a gap g takes its series length from the
// largest possible x = s / r, s_max / g, instead of a vote per pair: 8 terms
// for x < 1/4, 5 below 0.1135, 3 below 0.029 -- each drops less than 6e-9 of
// the sum, as 8 terms at 1/4 do -- and needs no closed form, no root (only
// u = 1 / r^2 enters: h_ij = -s_j^3 u^2 P(s_j^2 u)) and no overlap test.
constexpr float kSeries5MaxX = 0.1135f, kSeries3MaxX = 0.0290f;

// Not with a cutoff: there every pair takes the form that its own distance gives
// it, whichever kernel meets it (see k_born_pair).

// The gaps from which the series holds with 8, 5 and 3 terms.
struct BornGaps {
  float g8, g5, g3;
};
__device__ __forceinline__ BornGaps born_gaps(const PairArgs& a) {
  return {fmaxf(a.s_max / kSeriesMaxX, a.s_max + a.rho_max), a.s_max / kSeries5MaxX, a.s_max / kSeries3MaxX};
}

template <int kTerms>
__device__ __forceinline__ float2 descreen_poly2(float2 w) {
  float2 p = bc(static_cast<float>(kTerms * (2 * kTerms - 1)) / (2 * kTerms + 1));
#pragma unroll
  for (int k = kTerms - 1; k >= 1; --k) p = fma2(p, w, bc(static_cast<float>(k * (2 * k - 1)) / (2 * k + 1)));
  return p;
}

// Two pairs in the halves: adds -h_ij to *hi and returns -h_ji; (s2, s3) =
// (s^2, s^3) of the two sides.
template <int kTerms>
__device__ __forceinline__ float2 born_far2(float2 dx, float2 dy, float2 dz, float2 si2, float2 si3, float2 sj2,
                                            float2 sj3, float2* hi) {
  const float2 r2 = fma2(dx, dx, fma2(dy, dy, mul2(dz, dz)));
  const float2 u = make_float2(rcp_approx(r2.x), rcp_approx(r2.y));
  const float2 u2 = mul2(u, u);
  *hi = fma2(mul2(u2, descreen_poly2<kTerms>(mul2(sj2, u))), sj3, *hi);
  return mul2(mul2(u2, descreen_poly2<kTerms>(mul2(si2, u))), si3);
}

// The same with three terms, in powers of u with the series' coefficients per
// atom (c.x = s^3 / 3, c.y = 6/5 s^5, c.z = 15/7 s^7, PairArgs::bs): six
// packed operations after u^2 where the form above takes ten.  All but the
// nearest tile pairs of an extended chain come here.
struct Series3 {
  float2 c0, c1, c2;
};
__device__ __forceinline__ float2 born_far3(float2 dx, float2 dy, float2 dz, const Series3& i, const Series3& j,
                                            float2* hi) {
  const float2 r2 = fma2(dx, dx, fma2(dy, dy, mul2(dz, dz)));
  const float2 u = make_float2(rcp_approx(r2.x), rcp_approx(r2.y));
  const float2 u2 = mul2(u, u);
  *hi = fma2(u2, fma2(u, fma2(u, j.c2, j.c1), j.c0), *hi);
  return mul2(u2, fma2(u, fma2(u, i.c2, i.c1), i.c0));
}

// One i atom per lane against j atoms k0, k0 + 4, .. of [k_begin, k_end) with
// three terms; the columns at sp (x, y, z) and sb (the coefficients).
template <class J>
__device__ __forceinline__ float born_far_one3(const float* sp, const float* sb, int k_begin, int k_end, float xi,
                                               float yi, float zi, float3 c, J j) {
  const float2 nx = bc(-xi), ny = bc(-yi), nz = bc(-zi);
  const Series3 i{bc(c.x), bc(c.y), bc(c.z)};
  float2 hi = bc(0.0f);
#pragma unroll 2
  for (int k0 = k_begin; k0 < k_end; k0 += 4) {
    const float4 X = *reinterpret_cast<const float4*>(&sp[k0]);
    const float4 Y = *reinterpret_cast<const float4*>(&sp[32 + k0]);
    const float4 Z = *reinterpret_cast<const float4*>(&sp[64 + k0]);
    const float4 A = *reinterpret_cast<const float4*>(&sb[k0]);
    const float4 B = *reinterpret_cast<const float4*>(&sb[32 + k0]);
    const float4 C = *reinterpret_cast<const float4*>(&sb[64 + k0]);
    const float2 a = born_far3(add2(make_float2(X.x, X.y), nx), add2(make_float2(Y.x, Y.y), ny),
                               add2(make_float2(Z.x, Z.y), nz), i,
                               Series3{make_float2(A.x, A.y), make_float2(B.x, B.y), make_float2(C.x, C.y)}, &hi);
    const float2 b = born_far3(add2(make_float2(X.z, X.w), nx), add2(make_float2(Y.z, Y.w), ny),
                               add2(make_float2(Z.z, Z.w), nz), i,
                               Series3{make_float2(A.z, A.w), make_float2(B.z, B.w), make_float2(C.z, C.w)}, &hi);
    j(k0, a.x, a.y, b.x, b.y);
  }
  return -(hi.x + hi.y);
}

// One i atom per lane against j atoms k0, k0 + 4, .. of [k_begin, k_end), two j
// atoms per packed operation; the columns at sp (x, y, z) and sg (rho~, s~
// from +64).  Returns the i side; j(k, v) receives the lane's four values for
// the j atoms from k on, negated.
template <int kTerms, class J>
__device__ __forceinline__ float born_far_one(const float* sp, const float* sg, int k_begin, int k_end, float xi,
                                              float yi, float zi, float s_i, J j) {
  const float2 nx = bc(-xi), ny = bc(-yi), nz = bc(-zi), si2 = bc(s_i * s_i), si3 = bc(s_i * s_i * s_i);
  float2 hi = bc(0.0f);
#pragma unroll 2
  for (int k0 = k_begin; k0 < k_end; k0 += 4) {
    const float4 X = *reinterpret_cast<const float4*>(&sp[k0]);
    const float4 Y = *reinterpret_cast<const float4*>(&sp[32 + k0]);
    const float4 Z = *reinterpret_cast<const float4*>(&sp[64 + k0]);
    const float4 S = *reinterpret_cast<const float4*>(&sg[96 + k0]);
    const float2 sa = make_float2(S.x, S.y), sb = make_float2(S.z, S.w);
    const float2 sa2 = mul2(sa, sa), sb2 = mul2(sb, sb);
    const float2 a = born_far2<kTerms>(add2(make_float2(X.x, X.y), nx), add2(make_float2(Y.x, Y.y), ny),
                                       add2(make_float2(Z.x, Z.y), nz), si2, si3, sa2, mul2(sa2, sa), &hi);
    const float2 b = born_far2<kTerms>(add2(make_float2(X.z, X.w), nx), add2(make_float2(Y.z, Y.w), ny),
                                       add2(make_float2(Z.z, Z.w), nz), si2, si3, sb2, mul2(sb2, sb), &hi);
    j(k0, a.x, a.y, b.x, b.y);
  }
  return -(hi.x + hi.y);
}
// The series length by the gap; false for a gap the series does not hold for.
template <class J>
__device__ __forceinline__ bool born_far_tile(const BornGaps& gaps, float gap, const float* sp, const float* sg,
                                              const float* sb, int k_begin, int k_end, float xi, float yi, float zi,
                                              float s_i, float3 ci, float* hi, J j) {
  if (!(gap >= gaps.g8)) return false;
  *hi = gap >= gaps.g3   ? born_far_one3(sp, sb, k_begin, k_end, xi, yi, zi, ci, j)
        : gap >= gaps.g5 ? born_far_one<5>(sp, sg, k_begin, k_end, xi, yi, zi, s_i, j)
                         : born_far_one<8>(sp, sg, k_begin, k_end, xi, yi, zi, s_i, j);
  return true;
}

// The next work item of a CTA: its own (one CTA per item) or the queue's.
template <bool kPersistent>
__device__ __forceinline__ int next_item(const PairArgs& a, int* s_item, int prev) {
  if (!kPersistent) return prev < 0 ? static_cast<int>(blockIdx.x) : a.n_work;
  __syncthreads();  // every thread has read the previous item
  if (threadIdx.x == 0) *s_item = atomicAdd(a.queue, 1);
  __syncthreads();
  return *s_item;
}

template <int W, int kMinBlocks, bool kPersistent>
__global__ void __launch_bounds__(W * 32, kMinBlocks) k_born(PairArgs a) {
  __shared__ __align__(128) float s_buf[2][3][kStageFloats];          // columns of pq, gb, bs
  __shared__ float s_part[2][W][1][kStageTiles * kTile];
  __shared__ StageTilesT<W> s_tiles[3];
  __shared__ __align__(8) uint64_t s_bar[2];
  __shared__ int s_item;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(&s_bar[0], 1);
    mbar_init(&s_bar[1], 1);
    fence_mbar_init();
  }
  __syncthreads();
  const BornGaps gaps = born_gaps(a);
  uint32_t g = 0;  // stages this CTA has consumed
  for (int item = next_item<kPersistent>(a, &s_item, -1); item < a.n_work;
       item = next_item<kPersistent>(a, &s_item, item)) {
  PairWork w = a.work[item];
  if (a.seg_end) w.j_end = min(w.j_end, a.seg_end[w.i_tile0]);
  if (w.j_begin >= w.j_end) continue;  // chunk culled by the cutoff (block-uniform)
  const Stager st{a.jlist, w.j_begin, w.j_end, (w.j_end - w.j_begin + kStageTiles - 1) / kStageTiles, s_bar, g};
  const float* src[3] = {a.pq, a.gb, a.bs};
  if (threadIdx.x == 0) {
    if (st.n_stages > 0) st.issue<3>(0, s_buf, src);
    if (st.n_stages > 1) st.issue<3>(1, s_buf, src);
  }

  const bool active = warp < w.n_i_tiles;
  const int it = w.i_tile0 + (active ? warp : 0);
  const int i = it * kTile + lane;
  const float px = a.pq[soa_index(i, 0)], py = a.pq[soa_index(i, 1)], pz = a.pq[soa_index(i, 2)];
  const float rho_i = a.gb[soa_index(i, 2)], s_i = a.gb[soa_index(i, 3)];
  const float3 ci = make_float3(a.bs[soa_index(i, 0)], a.bs[soa_index(i, 1)], a.bs[soa_index(i, 2)]);
  const float c2 = a.born_c2;
  double acc = 0.0;
  stage_tiles(a, w, 0, s_tiles[g % 3]);
  // the j sums of stage s, once every warp has written its own
  auto flush = [&](int s) {
    unsigned long long* dst[1] = {a.born_sum};
    const int cnt = min(kStageTiles, w.j_end - (w.j_begin + s * kStageTiles));
    flush_j<W, 1>(a, s_tiles[(g + s) % 3].jt, cnt, s_part[(g + s) & 1], dst, kBornScale);
  };
  for (int s = 0; s < st.n_stages; ++s) {
    const uint32_t gs = g + s;
    const int b = gs & 1;
    const bool ok = mbar_wait_bounded(&s_bar[b], (gs >> 1) & 1u);
    if (__syncthreads_or(!ok)) {
      if (threadIdx.x == 0) atomicOr(a.error_flag, kStatusTimeout);
      return;
    }
    // one barrier per stage: here every warp is done with the stage before, whose
    // raw buffer is free and whose j sums are complete (a second barrier before
    // the flush: 650 -> 640 us for 64 chains of 300 residues; k_force, with
    // three components to buffer twice, lost 1 % by it)
    if (s > 0) {
      if (threadIdx.x == 0 && s + 1 < st.n_stages) st.issue<3>(s + 1, s_buf, src);
      flush(s - 1);
    }
    const int cnt = min(kStageTiles, w.j_end - (w.j_begin + s * kStageTiles));
    stage_tiles(a, w, s + 1, s_tiles[(gs + 1) % 3]);
    const StageTilesT<W>& tiles = s_tiles[gs % 3];
    for (int t = 0; t < cnt; ++t) {
      const int jt = tiles.jt[t];
      float* part = &s_part[b][warp][0][t * kTile];
      const float4 off = tiles.off[t][warp];
      if (!active || jt < it || (c2 != INFINITY && off.w > a.born_cutoff)) {
        part[lane] = 0.0f;
        continue;
      }
      const float xi = px - off.x;
      const float yi = py - off.y;
      const float zi = pz - off.z;
      const float* sp = &s_buf[b][0][t * 128];
      const float* sg = &s_buf[b][1][t * 128];
      float hi = 0.0f;
      const bool series = c2 == INFINITY &&
                          born_far_tile(gaps, off.w, sp, sg, &s_buf[b][2][t * 128], 0, kTile, xi, yi, zi, s_i, ci,
                                        &hi, [&](int k0, float v0, float v1, float v2, float v3) {
                                          const float tot = reduce_scatter4(v0, v1, v2, v3, lane);
                                          if ((lane & 7) == 0) part[k0 + (lane >> 3)] = -tot;
                                        });
      if (series) {
      } else if (jt == it) {
        // Diagonal tile: every ordered pair from the i side.
#pragma unroll 4
        for (int k = 0; k < kTile; ++k) {
          const float2 h = born_pair(sp[k] - xi, sp[32 + k] - yi, sp[64 + k] - zi, rho_i, s_i, sg[64 + k],
                                     sg[96 + k], c2);
          hi += h.x;
        }
        part[lane] = 0.0f;
      } else {
OG_UNROLL(OG_BORN_UNROLL)
        for (int k0 = 0; k0 < kTile; k0 += 4) {
          const float4 X = *reinterpret_cast<const float4*>(&sp[k0]);
          const float4 Y = *reinterpret_cast<const float4*>(&sp[32 + k0]);
          const float4 Z = *reinterpret_cast<const float4*>(&sp[64 + k0]);
          const float4 RH = *reinterpret_cast<const float4*>(&sg[64 + k0]);
          const float4 SR = *reinterpret_cast<const float4*>(&sg[96 + k0]);
          const float2 h0 = born_pair(X.x - xi, Y.x - yi, Z.x - zi, rho_i, s_i, RH.x, SR.x, c2);
          const float2 h1 = born_pair(X.y - xi, Y.y - yi, Z.y - zi, rho_i, s_i, RH.y, SR.y, c2);
          const float2 h2 = born_pair(X.z - xi, Y.z - yi, Z.z - zi, rho_i, s_i, RH.z, SR.z, c2);
          const float2 h3 = born_pair(X.w - xi, Y.w - yi, Z.w - zi, rho_i, s_i, RH.w, SR.w, c2);
          hi += (h0.x + h1.x) + (h2.x + h3.x);
          const float tot = reduce_scatter4(h0.y, h1.y, h2.y, h3.y, lane);
          if ((lane & 7) == 0) part[k0 + (lane >> 3)] = tot;
        }
      }
      acc += static_cast<double>(hi);
    }
  }
  __syncthreads();
  flush(st.n_stages - 1);
  g += st.n_stages;
  if (active && a.atom_valid[i]) {
    if (!isfinite(acc)) atomicOr(a.sys_nonfinite + a.atom_sys[i], 1);
    add_fixed(a.born_sum + i, acc, kBornScale);
  }
  }
}

// One i-tile per CTA, its four warps taking eight atoms of each j-tile: the
// shape for engines of few tiles, where whole-tile work items leave most of
// the chip idle and a tile pair's latency (about 1 500 cycles per group of
// four j atoms in the closed form) is the pass's time.  (Warps taking whole tile pairs of their own,
// without the shared sums, were 0 to 50 % slower than the better of this and
// k_born at every size tried.)
constexpr int kSplitWarps = 4, kSplitJ = kTile / kSplitWarps;

// The four warps' i-side sums of one component, in warp order.
__device__ __forceinline__ double split_sum(const double (*s_acc)[kTile], int lane) {
  double v = 0.0;
#pragma unroll
  for (int w = 0; w < kSplitWarps; ++w) v += s_acc[w][lane];
  return v;
}

template <bool kPersistent>
__global__ void __launch_bounds__(kSplitWarps * 32) k_born_split(PairArgs a) {
  __shared__ double s_acc[kSplitWarps][kTile];
  __shared__ int s_item;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const BornGaps gaps = born_gaps(a);
  for (int item = next_item<kPersistent>(a, &s_item, -1); item < a.n_work;
       item = next_item<kPersistent>(a, &s_item, item)) {
    const PairWork w = a.work[item];
    const int it = w.i_tile0, i = it * kTile + lane;
    const float px = a.pq[soa_index(i, 0)], py = a.pq[soa_index(i, 1)], pz = a.pq[soa_index(i, 2)];
    const float rho_i = a.gb[soa_index(i, 2)], s_i = a.gb[soa_index(i, 3)];
    const float3 ci = make_float3(a.bs[soa_index(i, 0)], a.bs[soa_index(i, 1)], a.bs[soa_index(i, 2)]);
    const double4 oi = a.origin[it];
    double acc = 0.0;
    for (int p = w.j_begin; p < w.j_end; ++p) {
      const int jt = a.jlist[p];
      const double4 oj = a.origin[jt];
      const bool diag = jt == it;
      const float xi = px - static_cast<float>(oj.x - oi.x);
      const float yi = py - static_cast<float>(oj.y - oi.y);
      const float zi = pz - static_cast<float>(oj.z - oi.z);
      float hi = 0.0f;
      const float* sp = a.pq + static_cast<size_t>(jt) * 128;
      const float* sg = a.gb + static_cast<size_t>(jt) * 128;
      const float* sb = a.bs + static_cast<size_t>(jt) * 128;
      auto add_j = [&](int k0, float v0, float v1, float v2, float v3) {
        const float tot = reduce_scatter4(v0, v1, v2, v3, lane);
        const int j = jt * kTile + k0 + (lane >> 3);
        if ((lane & 7) == 0 && tot != 0.0f && a.atom_valid[j]) {
          if (!isfinite(tot)) atomicOr(a.sys_nonfinite + a.atom_sys[j], 1);
          add_fixed(a.born_sum + j, static_cast<double>(tot), kBornScale);
        }
      };
      const int k_begin = warp * kSplitJ, k_end = k_begin + kSplitJ;
      auto sub_j = [&](int k0, float v0, float v1, float v2, float v3) { add_j(k0, -v0, -v1, -v2, -v3); };
      if (!born_far_tile(gaps, tile_gap(oi, oj), sp, sg, sb, k_begin, k_end, xi, yi, zi, s_i, ci, &hi, sub_j)) {
#pragma unroll 1
        for (int k0 = k_begin; k0 < k_end; k0 += 4) {
          const float4 X = *reinterpret_cast<const float4*>(sp + k0);
          const float4 Y = *reinterpret_cast<const float4*>(sp + 32 + k0);
          const float4 Z = *reinterpret_cast<const float4*>(sp + 64 + k0);
          const float4 RH = *reinterpret_cast<const float4*>(sg + 64 + k0);
          const float4 SR = *reinterpret_cast<const float4*>(sg + 96 + k0);
          const float2 h0 = born_pair(X.x - xi, Y.x - yi, Z.x - zi, rho_i, s_i, RH.x, SR.x, INFINITY);
          const float2 h1 = born_pair(X.y - xi, Y.y - yi, Z.y - zi, rho_i, s_i, RH.y, SR.y, INFINITY);
          const float2 h2 = born_pair(X.z - xi, Y.z - yi, Z.z - zi, rho_i, s_i, RH.z, SR.z, INFINITY);
          const float2 h3 = born_pair(X.w - xi, Y.w - yi, Z.w - zi, rho_i, s_i, RH.w, SR.w, INFINITY);
          hi += (h0.x + h1.x) + (h2.x + h3.x);
          if (!diag) add_j(k0, h0.y, h1.y, h2.y, h3.y);  // a diagonal tile's pairs are all seen from the i side
        }
      }
      acc += static_cast<double>(hi);
    }
    s_acc[warp][lane] = acc;
    __syncthreads();
    if (warp == 0 && a.atom_valid[i]) {
      const double v = split_sum(s_acc, lane);
      if (!isfinite(v)) atomicOr(a.sys_nonfinite + a.atom_sys[i], 1);
      add_fixed(a.born_sum + i, v, kBornScale);
    }
    if (kPersistent) __syncthreads();  // s_acc is read before the next item writes it
  }
}

// ------------------------------------------- tile pairs, summed in k_born's order
// The eight-tile kernels' sums for engines of few tiles with culled lists: a
// CTA per tile pair (its four warps taking eight j atoms each) keeps the pair's
// sums, and k_collect adds them in the order in which k_born<8> / k_force<8>
// do -- an i atom's eight groups of a tile in FP32, a chunk's tiles in FP64, a
// j atom's sums over a block's eight tiles in FP32 -- so that the results are
// those kernels' bit for bit, whatever else is in the engine.  (A sum in
// another order is as good by itself, but a trajectory at its limit of
// stability shows the last bit: of 400 starts of unrelaxed insulin at 2 fs, 26
// had parted by more than 2e-5 of the velocities after 50 steps.)
// Bound by latency while the tile pairs fit the chip at once: insulin (25 tiles)
// 21 us for each pass with its list and k_collect, against 98 and 63 for
// k_born<8> and k_force<8>, and 15 and 14 for sums in no set order, added
// straight to the accumulators.  The line is kMaxTilePairs: 16 folds of 4.7k
// atoms (174k tile pairs) 235 and 179 us against 266 and 191; 32 extended
// chains of 4.7k (348k) 195 and 133 against 113 and 77, since a culled tile pair
// costs a lane here and nothing there.

__device__ __forceinline__ size_t pair_at(size_t slot, int comps, int c, int lane) {
  return (slot * comps + c) * kTile + lane;
}

// A CTA's tile pairs are blockIdx.x, + gridDim.x, ..: up to kPairsPerCta, so that
// the culled ones (nearly all, in a long chain) cost a lane each and the others
// spread over the CTAs.  Thread q tests pair q; returns the ones to evaluate.
constexpr int kPairsPerCta = 32;
template <class Skip>
__device__ __forceinline__ unsigned live_pairs(const PairArgs& a, unsigned* s_live, Skip skip) {
  if (threadIdx.x < kPairsPerCta) {
    const size_t slot = blockIdx.x + static_cast<size_t>(threadIdx.x) * gridDim.x;
    bool on = slot < static_cast<size_t>(a.n_tile_pairs);
    if (on) {
      const int2 ij = a.tile_pairs[slot];
      on = !skip(ij.x, ij.y);
      a.pair_on[slot] = on ? 1 : 0;
    }
    const unsigned live = __ballot_sync(0xffffffffu, on);
    if (threadIdx.x == 0) *s_live = live;
  }
  __syncthreads();
  return *s_live;
}

__global__ void __launch_bounds__(kSplitWarps * 32) k_born_pair(PairArgs a) {
  __shared__ float s_h[kTile][kTile];  // the i side's terms, in the order they are added
  __shared__ unsigned s_live;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const float c2 = a.born_c2;
  unsigned live = live_pairs(a, &s_live, [&](int it, int jt) { return tile_gap(a.origin[it], a.origin[jt]) > a.born_cutoff; });
  for (; live; live &= live - 1) {
    const size_t slot = blockIdx.x + static_cast<size_t>(__ffs(live) - 1) * gridDim.x;
    const int2 ij = a.tile_pairs[slot];
    const int it = ij.x, jt = ij.y, i = it * kTile + lane;
    const double4 oi = a.origin[it], oj = a.origin[jt];
    const bool diag = jt == it;
    const float rho_i = a.gb[soa_index(i, 2)], s_i = a.gb[soa_index(i, 3)];
    const float xi = a.pq[soa_index(i, 0)] - static_cast<float>(oj.x - oi.x);
    const float yi = a.pq[soa_index(i, 1)] - static_cast<float>(oj.y - oi.y);
    const float zi = a.pq[soa_index(i, 2)] - static_cast<float>(oj.z - oi.z);
    const float* sp = a.pq + static_cast<size_t>(jt) * 128;
    const float* sg = a.gb + static_cast<size_t>(jt) * 128;
    const int k_begin = warp * kSplitJ;
    if (diag) {  // every ordered pair from the i side
#pragma unroll 4
      for (int k = k_begin; k < k_begin + kSplitJ; ++k)
        s_h[k][lane] = born_pair(sp[k] - xi, sp[32 + k] - yi, sp[64 + k] - zi, rho_i, s_i, sg[64 + k], sg[96 + k], c2).x;
    } else {
#pragma unroll 1
      for (int k0 = k_begin; k0 < k_begin + kSplitJ; k0 += 4) {
        const float4 X = *reinterpret_cast<const float4*>(sp + k0);
        const float4 Y = *reinterpret_cast<const float4*>(sp + 32 + k0);
        const float4 Z = *reinterpret_cast<const float4*>(sp + 64 + k0);
        const float4 RH = *reinterpret_cast<const float4*>(sg + 64 + k0);
        const float4 SR = *reinterpret_cast<const float4*>(sg + 96 + k0);
        const float2 h0 = born_pair(X.x - xi, Y.x - yi, Z.x - zi, rho_i, s_i, RH.x, SR.x, c2);
        const float2 h1 = born_pair(X.y - xi, Y.y - yi, Z.y - zi, rho_i, s_i, RH.y, SR.y, c2);
        const float2 h2 = born_pair(X.z - xi, Y.z - yi, Z.z - zi, rho_i, s_i, RH.z, SR.z, c2);
        const float2 h3 = born_pair(X.w - xi, Y.w - yi, Z.w - zi, rho_i, s_i, RH.w, SR.w, c2);
        s_h[k0 / 4][lane] = (h0.x + h1.x) + (h2.x + h3.x);
        const float tot = reduce_scatter4(h0.y, h1.y, h2.y, h3.y, lane);
        if ((lane & 7) == 0) a.pair_j[pair_at(slot, 1, 0, k0 + (lane >> 3))] = tot;
      }
    }
    __syncthreads();
    if (warp == 0) {
      float hi = 0.0f;
      const int n = diag ? kTile : kTile / 4;
#pragma unroll 8
      for (int k = 0; k < n; ++k) hi += s_h[k][lane];
      a.pair_i[pair_at(slot, 1, 0, lane)] = hi;
      if (diag) a.pair_j[pair_at(slot, 1, 0, lane)] = 0.0f;
    }
    __syncthreads();  // s_h is read before the next pair writes it
  }
}

// One CTA per (i-block, tile t of it): the tile's i sums chunk by chunk of the
// block's list, and its j sums block by block, the warps taking them in turn.
constexpr int kBlockTiles = 8, kCollectWarps = 8;

template <int kComps>
__global__ void __launch_bounds__(kCollectWarps * 32) k_collect(PairArgs a, unsigned long long* d0,
                                                                unsigned long long* d1, unsigned long long* d2,
                                                                double scale) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const CutBlock cb = a.blocks[blockIdx.x / kBlockTiles];
  const int t = blockIdx.x % kBlockTiles;
  if (t >= cb.n_i_tiles) return;
  const int it = cb.i_tile0 + t, i = it * kTile + lane;
  unsigned long long* const dst[3] = {d0, d1, d2};
  const int je = a.seg_end[cb.i_tile0];
  const int n_chunks = (je - cb.jb + a.chunk - 1) / a.chunk;
  const int n_parts = n_chunks + (it - cb.sys_tile0) / kBlockTiles + 1;
  const bool valid = a.atom_valid[i] != 0;
  for (int part = warp; part < n_parts; part += kCollectWarps) {
    double v[kComps];
#pragma unroll
    for (int c = 0; c < kComps; ++c) v[c] = 0.0;
    bool any = true, finite = true;
    if (part < n_chunks) {
      const int row = a.pair_row[it];
      const int p0 = cb.jb + part * a.chunk, p1 = min(je, p0 + a.chunk);
      for (int q0 = p0; q0 < p1; q0 += 32) {  // lane q looks up tile q of the chunk
        const int jt = q0 + lane < p1 ? a.jlist[q0 + lane] : -1;
        const int at = row + jt - it;
        unsigned live = __ballot_sync(0xffffffffu, jt >= it && a.pair_on[at] != 0);
        while (live) {  // eight tiles' loads in flight
          float x[8][kComps];
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            const bool on = live != 0u;
            const int slot = __shfl_sync(0xffffffffu, at, on ? __ffs(live) - 1 : 0);
#pragma unroll
            for (int c = 0; c < kComps; ++c) x[u][c] = on ? a.pair_i[pair_at(slot, kComps, c, lane)] : 0.0f;
            live &= live - 1;
          }
#pragma unroll
          for (int u = 0; u < 8; ++u)
#pragma unroll
            for (int c = 0; c < kComps; ++c) v[c] += static_cast<double>(x[u][c]);
        }
      }
    } else {
      const int t0 = cb.sys_tile0 + (part - n_chunks) * kBlockTiles;
      const int ti = t0 + (lane & (kBlockTiles - 1));  // lane w looks up tile w of the block
      const int at = ti < it ? a.pair_row[ti] + it - ti : 0;
      const unsigned live = __ballot_sync(0xffffffffu, ti < it && a.pair_on[at] != 0);
      float sum[kComps];
#pragma unroll
      for (int c = 0; c < kComps; ++c) sum[c] = 0.0f;
#pragma unroll
      for (int w = 0; w < kBlockTiles; ++w) {
        const int slot = __shfl_sync(0xffffffffu, at, w);
#pragma unroll
        for (int c = 0; c < kComps; ++c) sum[c] += (live >> w) & 1u ? a.pair_j[pair_at(slot, kComps, c, lane)] : 0.0f;
      }
      any = false;
#pragma unroll
      for (int c = 0; c < kComps; ++c) {
        any = any || sum[c] != 0.0f;
        v[c] = static_cast<double>(sum[c]);
      }
    }
    if (!any || !valid) continue;
#pragma unroll
    for (int c = 0; c < kComps; ++c) finite = finite && isfinite(v[c]);
    if (!finite) atomicOr(a.sys_nonfinite + a.atom_sys[i], 1);
#pragma unroll
    for (int c = 0; c < kComps; ++c) add_fixed(dst[c] + i, v[c], scale);
  }
}

// --------------------------------------------------------------- force
// i-atom data broadcast into both halves of a float2.
struct IAtom2 {
  float2 nx, ny, nz;   // minus the i position relative to the j-tile's origin
  float2 rm;           // Rmin/2
  float2 se;           // 12 * 4.184 * sqrt(eps)
  float2 cq;           // -332.0637 * 4.184 * q_i
  float2 gq;           // (1 - 1/78.5) * 332.0637 * 4.184 * q_i
  float2 R;            // Born radius
  float2 nexp;         // -log2(e) / (4 R_i)
  float2 nrc3;         // -1 / Rc^3
  float2 cg;           // (gb_pref_kj - coul_kj) q_i
};

// One i atom in both halves (nx, ny, nz are set per j-tile).
__device__ __forceinline__ IAtom2 i_atom(const PairArgs& a, int i) {
  IAtom2 ia;
  const float qi = a.pq[soa_index(i, 3)];
  ia.rm = bc(a.lj[soa_index(i, 0)]);
  ia.se = bc(a.lj_kj12 * a.lj[soa_index(i, 1)]);
  ia.cq = bc(-a.coul_kj * qi);
  ia.gq = bc(a.gb_pref_kj * qi);
  ia.R = bc(a.gb[soa_index(i, 0)]);
  ia.nexp = bc(-0.25f * kLog2e * a.gb[soa_index(i, 1)]);
  ia.nrc3 = bc(-a.inv_rc3);
  ia.cg = bc(a.far_kj * qi);
  return ia;
}

// Separation d = x_j - x_i of two j atoms from the i atom, and r^2.
struct Sep2 {
  float2 dx, dy, dz, r2;
};
template <class I>
__device__ __forceinline__ Sep2 sep2(float2 xj, float2 yj, float2 zj, const I& ia) {
  Sep2 s;
  s.dx = add2(xj, ia.nx);
  s.dy = add2(yj, ia.ny);
  s.dz = add2(zj, ia.nz);
  s.r2 = fma2(s.dx, s.dx, fma2(s.dy, s.dy, mul2(s.dz, s.dz)));
  return s;
}

// Exponent of the GB kernel's exponential in base 2: -r^2 / (4 R_i R_j) log2(e).
__device__ __forceinline__ float2 gb_arg2(const Sep2& s, float2 iRj, const IAtom2& ia) {
  return mul2(mul2(s.r2, ia.nexp), iRj);
}

// Pair coefficients c (F_i = c * d) for two j atoms.  kFarGb: both pairs
// have arg < -30, so e = 2^arg < 2^-30: R_i R_j e < r^2 / 83 * 2^-30 is below
// half an ulp of r^2, so f^2 = fma(R_i R_j, e, r^2) rounds to r^2 and
// 1 - e/4 to 1; the far form then evaluates exactly what the full form does
// (same rsqrt input, same products), without the exponential and the
// second reciprocal square root.
template <bool kAllPairs, bool kFarGb>
__device__ __forceinline__ float2 coeff2(const Sep2& s, float2 arg, float2 qj, float2 rmj, float2 sej, float2 Rj,
                                         const IAtom2& ia, const PairArgs& a) {
  const float2 r2 = s.r2;
  const float2 inv_r = make_float2(rsqrtf(r2.x), rsqrtf(r2.y));
  const float2 inv_r2 = mul2(inv_r, inv_r);
  const float2 rmin = add2(ia.rm, rmj);
  const float2 ratio2 = mul2(mul2(rmin, rmin), inv_r2);
  const float2 r6 = mul2(mul2(ratio2, ratio2), ratio2);
  const float2 one_m_r6 = fma2(r6, bc(-1.0f), bc(1.0f));
  const float2 ljc = mul2(mul2(ia.se, sej), mul2(inv_r2, mul2(r6, one_m_r6)));
  const float2 coul = mul2(mul2(ia.cq, qj), fma2(inv_r2, inv_r, ia.nrc3));
  float2 gbc;
  if (kFarGb) {
    gbc = mul2(mul2(ia.gq, qj), mul2(inv_r, mul2(inv_r, inv_r)));
  } else {
    const float2 e = make_float2(exp2f(arg.x), exp2f(arg.y));
    const float2 f2 = fma2(mul2(ia.R, Rj), e, r2);
    const float2 inv_f = make_float2(rsqrtf(f2.x), rsqrtf(f2.y));
    const float2 wgt = fma2(bc(-0.25f), e, bc(1.0f));
    gbc = mul2(mul2(ia.gq, qj), mul2(wgt, mul2(inv_f, mul2(inv_f, inv_f))));
  }
  float2 c;
  if (kAllPairs) {
    c = add2(add2(ljc, coul), gbc);
  } else {
    const float2 nb = add2(ljc, coul);
    c.x = ((r2.x <= a.nb_c2) ? nb.x : 0.0f) + ((r2.x <= a.gb_c2) ? gbc.x : 0.0f);
    c.y = ((r2.y <= a.nb_c2) ? nb.y : 0.0f) + ((r2.y <= a.gb_c2) ? gbc.y : 0.0f);
  }
  c.x = (r2.x >= 1e-18f) ? c.x : 0.0f;
  c.y = (r2.y >= 1e-18f) ? c.y : 0.0f;
  return c;
}

// Where a tile pair's spheres leave a gap g with g^2 > kFarGapSq R_i R_j for
// the tiles' largest Born radii, every pair has the far GB form (kFarGb) and,
// without cutoffs, Coulomb and GB share 1/r^3: one reciprocal square root and
// thirteen packed operations per two pairs, no vote and no guard.
// (arg < -30 in coeff2: r^2 log2(e) / (4 R_i R_j) > 30; a little above 120 ln 2)
constexpr float kFarGapSq = 83.2f;
__device__ __forceinline__ bool far_tiles(float gap, float ri_max, float rj_max) {
  return gap > 0.0f && gap * gap > kFarGapSq * ri_max * rj_max;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
// The coefficient of two such pairs; cg = (gb_pref - coul) q_i.
template <class I>
__device__ __forceinline__ float2 coeff_far2(float2 r2, float2 qj, float2 rmj, float2 sej, const I& ia) {
  const float2 inv_r = make_float2(rsqrtf(r2.x), rsqrtf(r2.y));
  const float2 inv_r2 = mul2(inv_r, inv_r);
  const float2 rmin = add2(ia.rm, rmj);
  const float2 ratio2 = mul2(mul2(rmin, rmin), inv_r2);
  const float2 r6 = mul2(mul2(ratio2, ratio2), ratio2);
  const float2 lj = mul2(mul2(ia.se, sej), mul2(r6, fma2(r6, bc(-1.0f), bc(1.0f))));
  return mul2(inv_r2, fma2(mul2(ia.cg, qj), inv_r, lj));
}

// The pair forces c d of one i atom and four consecutive j atoms (a: the first
// two, b: the others), the j columns at pq, lj, gb.
struct Group4 {
  float2 xa, ya, za, xb, yb, zb;
};
__device__ __forceinline__ Group4 force_far4(const float* pq, const float* lj, const IAtom2& ia) {
  const float4 X = *reinterpret_cast<const float4*>(pq);
  const float4 Y = *reinterpret_cast<const float4*>(pq + 32);
  const float4 Z = *reinterpret_cast<const float4*>(pq + 64);
  const float4 Q = *reinterpret_cast<const float4*>(pq + 96);
  const float4 RM = *reinterpret_cast<const float4*>(lj);
  const float4 SE = *reinterpret_cast<const float4*>(lj + 32);
  const Sep2 sa = sep2(make_float2(X.x, X.y), make_float2(Y.x, Y.y), make_float2(Z.x, Z.y), ia);
  const Sep2 sb = sep2(make_float2(X.z, X.w), make_float2(Y.z, Y.w), make_float2(Z.z, Z.w), ia);
  const float2 ca = coeff_far2(sa.r2, make_float2(Q.x, Q.y), make_float2(RM.x, RM.y), make_float2(SE.x, SE.y), ia);
  const float2 cb = coeff_far2(sb.r2, make_float2(Q.z, Q.w), make_float2(RM.z, RM.w), make_float2(SE.z, SE.w), ia);
  return Group4{mul2(sa.dx, ca), mul2(sa.dy, ca), mul2(sa.dz, ca), mul2(sb.dx, cb), mul2(sb.dy, cb), mul2(sb.dz, cb)};
}
template <bool kAllPairs>
__device__ __forceinline__ Group4 force_group4(const float* pq, const float* lj, const float* gb, const IAtom2& ia,
                                               const PairArgs& a) {
  const float4 X = *reinterpret_cast<const float4*>(pq);
  const float4 Y = *reinterpret_cast<const float4*>(pq + 32);
  const float4 Z = *reinterpret_cast<const float4*>(pq + 64);
  const float4 Q = *reinterpret_cast<const float4*>(pq + 96);
  const float4 RM = *reinterpret_cast<const float4*>(lj);
  const float4 SE = *reinterpret_cast<const float4*>(lj + 32);
  const float4 RB = *reinterpret_cast<const float4*>(gb);
  const float4 IR = *reinterpret_cast<const float4*>(gb + 32);
  const Sep2 sa = sep2(make_float2(X.x, X.y), make_float2(Y.x, Y.y), make_float2(Z.x, Z.y), ia);
  const Sep2 sb = sep2(make_float2(X.z, X.w), make_float2(Y.z, Y.w), make_float2(Z.z, Z.w), ia);
  const float2 arga = gb_arg2(sa, make_float2(IR.x, IR.y), ia), argb = gb_arg2(sb, make_float2(IR.z, IR.w), ia);
  // the far GB form when every pair of the warp's group allows it
  const bool far = __all_sync(0xffffffffu, fmaxf(fmaxf(arga.x, arga.y), fmaxf(argb.x, argb.y)) < -30.0f);
  float2 ca, cb;
  if (far) {
    ca = coeff2<kAllPairs, true>(sa, arga, make_float2(Q.x, Q.y), make_float2(RM.x, RM.y), make_float2(SE.x, SE.y),
                                 make_float2(RB.x, RB.y), ia, a);
    cb = coeff2<kAllPairs, true>(sb, argb, make_float2(Q.z, Q.w), make_float2(RM.z, RM.w), make_float2(SE.z, SE.w),
                                 make_float2(RB.z, RB.w), ia, a);
  } else {
    ca = coeff2<kAllPairs, false>(sa, arga, make_float2(Q.x, Q.y), make_float2(RM.x, RM.y), make_float2(SE.x, SE.y),
                                  make_float2(RB.x, RB.y), ia, a);
    cb = coeff2<kAllPairs, false>(sb, argb, make_float2(Q.z, Q.w), make_float2(RM.z, RM.w), make_float2(SE.z, SE.w),
                                  make_float2(RB.z, RB.w), ia, a);
  }
  return Group4{mul2(sa.dx, ca), mul2(sa.dy, ca), mul2(sa.dz, ca), mul2(sb.dx, cb), mul2(sb.dy, cb), mul2(sb.dz, cb)};
}

template <bool kAllPairs, int W, int kMinBlocks, bool kPersistent>
__global__ void __launch_bounds__(W * 32, kMinBlocks) k_force(PairArgs a) {
  __shared__ __align__(128) float s_buf[2][3][kStageFloats];          // columns of pq, lj, gb
  __shared__ float s_part[W][3][kStageTiles * kTile];
  __shared__ StageTilesT<W> s_tiles[2];
  __shared__ __align__(8) uint64_t s_bar[2];
  __shared__ int s_item;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(&s_bar[0], 1);
    mbar_init(&s_bar[1], 1);
    fence_mbar_init();
  }
  __syncthreads();
  uint32_t g = 0;  // stages this CTA has consumed
  for (int item = next_item<kPersistent>(a, &s_item, -1); item < a.n_work;
       item = next_item<kPersistent>(a, &s_item, item)) {
  PairWork w = a.work[item];
  if (a.seg_end) w.j_end = min(w.j_end, a.seg_end[w.i_tile0]);
  if (w.j_begin >= w.j_end) continue;  // chunk culled by the cutoff (block-uniform)
  const Stager st{a.jlist, w.j_begin, w.j_end, (w.j_end - w.j_begin + kStageTiles - 1) / kStageTiles, s_bar, g};
  const float* src[3] = {a.pq, a.lj, a.gb};
  if (threadIdx.x == 0) {
    if (st.n_stages > 0) st.issue<3>(0, s_buf, src);
    if (st.n_stages > 1) st.issue<3>(1, s_buf, src);
  }

  const bool active = warp < w.n_i_tiles;
  const int it = w.i_tile0 + (active ? warp : 0);
  const int i = it * kTile + lane;
  const float px = a.pq[soa_index(i, 0)], py = a.pq[soa_index(i, 1)], pz = a.pq[soa_index(i, 2)];
  IAtom2 ia = i_atom(a, i);
  const float ri_max = kAllPairs ? warp_max(ia.R.x) : 0.0f;
  // the next near-field j-tile (refs are in j order)
  int mref = a.mask_begin[it];
  const int mend = a.mask_begin[it + 1];
  int mnext = mref < mend ? a.mask_refs[mref].j_tile : 0x7fffffff;
  double acc0 = 0.0, acc1 = 0.0, acc2 = 0.0;
  stage_tiles(a, w, 0, s_tiles[g & 1]);

  for (int s = 0; s < st.n_stages; ++s) {
    const uint32_t gs = g + s;
    const int b = gs & 1;
    const bool ok = mbar_wait_bounded(&s_bar[b], (gs >> 1) & 1u);
    if (__syncthreads_or(!ok)) {
      if (threadIdx.x == 0) atomicOr(a.error_flag, kStatusTimeout);
      return;
    }
    const int t0 = w.j_begin + s * kStageTiles;
    const int cnt = min(kStageTiles, w.j_end - t0);
    stage_tiles(a, w, s + 1, s_tiles[b ^ 1]);
    for (int t = 0; t < cnt; ++t) {
      const int jt = s_tiles[b].jt[t];
      while (mnext < jt) mnext = ++mref < mend ? a.mask_refs[mref].j_tile : 0x7fffffff;
      const bool masked = mnext == jt;
      float* jfx = &s_part[warp][0][t * kTile];
      float* jfy = &s_part[warp][1][t * kTile];
      float* jfz = &s_part[warp][2][t * kTile];
      const float4 off = s_tiles[b].off[t][warp];
      if (!(active && jt > it && !masked) || (!kAllPairs && off.w > a.pair_cutoff)) {
        jfx[lane] = 0.0f;
        jfy[lane] = 0.0f;
        jfz[lane] = 0.0f;
        continue;
      }
      ia.nx = bc(-(px - off.x));
      ia.ny = bc(-(py - off.y));
      ia.nz = bc(-(pz - off.z));
      const float* sp = &s_buf[b][0][t * 128];
      const float* sl = &s_buf[b][1][t * 128];
      const float* sg = &s_buf[b][2][t * 128];
      float2 fx = bc(0.0f), fy = bc(0.0f), fz = bc(0.0f);
      auto add_group = [&](int k0, const Group4& u) {
        fx = add2(fx, add2(u.xa, u.xb));
        fy = add2(fy, add2(u.ya, u.yb));
        fz = add2(fz, add2(u.za, u.zb));
        const float tx = reduce_scatter4(u.xa.x, u.xa.y, u.xb.x, u.xb.y, lane);
        const float ty = reduce_scatter4(u.ya.x, u.ya.y, u.yb.x, u.yb.y, lane);
        const float tz = reduce_scatter4(u.za.x, u.za.y, u.zb.x, u.zb.y, lane);
        if ((lane & 7) == 0) {
          jfx[k0 + (lane >> 3)] = -tx;
          jfy[k0 + (lane >> 3)] = -ty;
          jfz[k0 + (lane >> 3)] = -tz;
        }
      };
      if (kAllPairs && far_tiles(off.w, ri_max, warp_max(sg[lane]))) {
#pragma unroll 2
        for (int k0 = 0; k0 < kTile; k0 += 4) add_group(k0, force_far4(sp + k0, sl + k0, ia));
      } else {
OG_UNROLL(OG_FORCE_UNROLL)
        for (int k0 = 0; k0 < kTile; k0 += 4)
          add_group(k0, force_group4<kAllPairs>(sp + k0, sl + k0, sg + k0, ia, a));
      }
      acc0 += static_cast<double>(fx.x + fx.y);
      acc1 += static_cast<double>(fy.x + fy.y);
      acc2 += static_cast<double>(fz.x + fz.y);
    }
    __syncthreads();  // every warp is done with buffer b and has written its j partials
    if (threadIdx.x == 0 && s + 2 < st.n_stages) st.issue<3>(s + 2, s_buf, src);
    unsigned long long* dst[3] = {a.fx, a.fy, a.fz};
    flush_j<W, 3>(a, s_tiles[b].jt, cnt, s_part, dst, kForceScale);
  }
  g += st.n_stages;
  if (active && a.atom_valid[i]) {
    if (!(isfinite(acc0) && isfinite(acc1) && isfinite(acc2))) atomicOr(a.sys_nonfinite + a.atom_sys[i], 1);
    add_fixed(a.fx + i, acc0, kForceScale);
    add_fixed(a.fy + i, acc1, kForceScale);
    add_fixed(a.fz + i, acc2, kForceScale);
  }
  }
}

// ------------------------------------------------------ force, four i-tiles
// The same pair terms with four i-tiles per warp (one atom of each in every
// lane, two per float2); the stage's j columns are expanded in shared memory
// to (v, v) pairs to feed them.  For systems of many tiles: a distant j atom
// costs one load of its columns and three reduce-scatters for 128 pairs, so
// the packed pair arithmetic is the bound.  A j-tile that is not distant from
// all four i-tiles goes through force_pair_tile, two i-tiles at a time.
// Sums per i atom: FP32 per j-tile, FP64 across tiles; per j atom: the warp's
// i atoms in FP32, warps in a fixed order, fixed point at the end.

// The stage's j columns: x, y, z, q, Rmin/2, sqrt(eps), R, 1/R.
constexpr int kForceCols = 8;

struct ForceSum {
  float2 x, y, z;
};
__device__ __forceinline__ float half_of(float2 v, int h) { return h ? v.y : v.x; }

// What a lane keeps of its i atoms: the far form's data.  The general form's
// are read again where a j-tile needs them (i_pair): 16 registers less in
// the far loop.
struct FarI2 {
  float2 nx, ny, nz, rm, se, cg;
};
// The general form's data of atoms i and j in the halves.
__device__ __forceinline__ IAtom2 i_pair(const PairArgs& a, int i, int j, const FarI2& f) {
  IAtom2 ia;
  ia.nx = f.nx;
  ia.ny = f.ny;
  ia.nz = f.nz;
  ia.rm = f.rm;
  ia.se = f.se;
  ia.cg = f.cg;
  const float2 qi = make_float2(a.pq[soa_index(i, 3)], a.pq[soa_index(j, 3)]);
  ia.cq = mul2(bc(-a.coul_kj), qi);
  ia.gq = mul2(bc(a.gb_pref_kj), qi);
  ia.R = make_float2(a.gb[soa_index(i, 0)], a.gb[soa_index(j, 0)]);
  ia.nexp = mul2(bc(-0.25f * kLog2e), make_float2(a.gb[soa_index(i, 1)], a.gb[soa_index(j, 1)]));
  ia.nrc3 = bc(-a.inv_rc3);
  return ia;
}

// Two i-tiles (the halves) against a j-tile, general form; va, vb: which of
// them.  j totals are added to jfx, jfy, jfz (negated).
template <bool kAllPairs>
__device__ __forceinline__ void force_pair_tile(const float* dup, const IAtom2& ia, const PairArgs& a, bool va, bool vb,
                                                float* jfx, float* jfy, float* jfz, int lane, ForceSum* f) {
  const bool both = va && vb;
#pragma unroll 1
  for (int k0 = 0; k0 < kTile; k0 += 4) {
    float tx[4], ty[4], tz[4];
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      const float* d = dup + 2 * (k0 + 2 * p);  // two j atoms
      const float4 X = *reinterpret_cast<const float4*>(d);
      const float4 Y = *reinterpret_cast<const float4*>(d + 64);
      const float4 Z = *reinterpret_cast<const float4*>(d + 128);
      const float4 Q = *reinterpret_cast<const float4*>(d + 192);
      const float4 RM = *reinterpret_cast<const float4*>(d + 256);
      const float4 SE = *reinterpret_cast<const float4*>(d + 320);
      const float4 RB = *reinterpret_cast<const float4*>(d + 384);
      const float4 IR = *reinterpret_cast<const float4*>(d + 448);
      const Sep2 s[2] = {sep2(make_float2(X.x, X.y), make_float2(Y.x, Y.y), make_float2(Z.x, Z.y), ia),
                         sep2(make_float2(X.z, X.w), make_float2(Y.z, Y.w), make_float2(Z.z, Z.w), ia)};
      const float2 q[2] = {make_float2(Q.x, Q.y), make_float2(Q.z, Q.w)};
      const float2 rm[2] = {make_float2(RM.x, RM.y), make_float2(RM.z, RM.w)};
      const float2 se[2] = {make_float2(SE.x, SE.y), make_float2(SE.z, SE.w)};
      const float2 rb[2] = {make_float2(RB.x, RB.y), make_float2(RB.z, RB.w)};
      const float2 arg[2] = {gb_arg2(s[0], make_float2(IR.x, IR.y), ia), gb_arg2(s[1], make_float2(IR.z, IR.w), ia)};
      const bool far = __all_sync(0xffffffffu, fmaxf(fmaxf(arg[0].x, arg[0].y), fmaxf(arg[1].x, arg[1].y)) < -30.0f);
      float2 c[2];
      if (far) {
        c[0] = coeff2<kAllPairs, true>(s[0], arg[0], q[0], rm[0], se[0], rb[0], ia, a);
        c[1] = coeff2<kAllPairs, true>(s[1], arg[1], q[1], rm[1], se[1], rb[1], ia, a);
      } else {
        c[0] = coeff2<kAllPairs, false>(s[0], arg[0], q[0], rm[0], se[0], rb[0], ia, a);
        c[1] = coeff2<kAllPairs, false>(s[1], arg[1], q[1], rm[1], se[1], rb[1], ia, a);
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        // one tile's pairs with this j-tile are near field or counted elsewhere
        if (!both) c[h] = make_float2(va ? c[h].x : 0.0f, vb ? c[h].y : 0.0f);
        const float2 ux = mul2(s[h].dx, c[h]), uy = mul2(s[h].dy, c[h]), uz = mul2(s[h].dz, c[h]);
        f->x = add2(f->x, ux);
        f->y = add2(f->y, uy);
        f->z = add2(f->z, uz);
        tx[2 * p + h] = ux.x + ux.y;
        ty[2 * p + h] = uy.x + uy.y;
        tz[2 * p + h] = uz.x + uz.y;
      }
    }
    const float sx = reduce_scatter4(tx[0], tx[1], tx[2], tx[3], lane);
    const float sy = reduce_scatter4(ty[0], ty[1], ty[2], ty[3], lane);
    const float sz = reduce_scatter4(tz[0], tz[1], tz[2], tz[3], lane);
    if ((lane & 7) == 0) {
      jfx[k0 + (lane >> 3)] -= sx;
      jfy[k0 + (lane >> 3)] -= sy;
      jfz[k0 + (lane >> 3)] -= sz;
    }
  }
}

// Four i-tiles against a j-tile distant from all of them.
__device__ __forceinline__ void force_far_four(const float* dup, const FarI2 (&ia)[2], float* jfx, float* jfy,
                                               float* jfz, int lane, ForceSum (&f)[2]) {
#pragma unroll 1
  for (int k0 = 0; k0 < kTile; k0 += 4) {
    float tx[4], ty[4], tz[4];
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      const float* d = dup + 2 * (k0 + 2 * p);
      const float4 X = *reinterpret_cast<const float4*>(d);
      const float4 Y = *reinterpret_cast<const float4*>(d + 64);
      const float4 Z = *reinterpret_cast<const float4*>(d + 128);
      const float4 Q = *reinterpret_cast<const float4*>(d + 192);
      const float4 RM = *reinterpret_cast<const float4*>(d + 256);
      const float4 SE = *reinterpret_cast<const float4*>(d + 320);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float2 xj = h ? make_float2(X.z, X.w) : make_float2(X.x, X.y);
        const float2 yj = h ? make_float2(Y.z, Y.w) : make_float2(Y.x, Y.y);
        const float2 zj = h ? make_float2(Z.z, Z.w) : make_float2(Z.x, Z.y);
        const float2 q = h ? make_float2(Q.z, Q.w) : make_float2(Q.x, Q.y);
        const float2 rm = h ? make_float2(RM.z, RM.w) : make_float2(RM.x, RM.y);
        const float2 se = h ? make_float2(SE.z, SE.w) : make_float2(SE.x, SE.y);
        float2 ux, uy, uz;
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          const Sep2 s = sep2(xj, yj, zj, ia[t]);
          const float2 c = coeff_far2(s.r2, q, rm, se, ia[t]);
          f[t].x = fma2(s.dx, c, f[t].x);
          f[t].y = fma2(s.dy, c, f[t].y);
          f[t].z = fma2(s.dz, c, f[t].z);
          ux = t ? fma2(s.dx, c, ux) : mul2(s.dx, c);
          uy = t ? fma2(s.dy, c, uy) : mul2(s.dy, c);
          uz = t ? fma2(s.dz, c, uz) : mul2(s.dz, c);
        }
        tx[2 * p + h] = ux.x + ux.y;
        ty[2 * p + h] = uy.x + uy.y;
        tz[2 * p + h] = uz.x + uz.y;
      }
    }
    const float sx = reduce_scatter4(tx[0], tx[1], tx[2], tx[3], lane);
    const float sy = reduce_scatter4(ty[0], ty[1], ty[2], ty[3], lane);
    const float sz = reduce_scatter4(tz[0], tz[1], tz[2], tz[3], lane);
    if ((lane & 7) == 0) {
      jfx[k0 + (lane >> 3)] = -sx;
      jfy[k0 + (lane >> 3)] = -sy;
      jfz[k0 + (lane >> 3)] = -sz;
    }
  }
}

template <bool kAllPairs, int W, int kMinBlocks, bool kPersistent>
__global__ void __launch_bounds__(W * 32, kMinBlocks) k_force_quad(PairArgs a) {
  __shared__ __align__(128) float s_buf[2][3][kStageFloats];                  // raw columns of pq, lj, gb (TMA)
  __shared__ __align__(16) float s_dup[kStageTiles][kForceCols * 2 * kTile];  // the stage's columns, each value twice
  __shared__ float s_rmax[kStageTiles];
  __shared__ StageTilesT<W * 4> s_tiles[2];
  __shared__ float s_part[W][3][kStageTiles * kTile];
  __shared__ double s_acc[W][12][kTile];  // the lanes' sums over j-tiles, per i-tile and component
  __shared__ __align__(8) uint64_t s_bar[2];
  __shared__ int s_item;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(&s_bar[0], 1);
    mbar_init(&s_bar[1], 1);
    fence_mbar_init();
  }
  __syncthreads();
  uint32_t g = 0;  // stages this CTA has consumed
  for (int item = next_item<kPersistent>(a, &s_item, -1); item < a.n_work;
       item = next_item<kPersistent>(a, &s_item, item)) {
  PairWork w = a.work[item];
  if (a.seg_end) w.j_end = min(w.j_end, a.seg_end[w.i_tile0]);
  if (w.j_begin >= w.j_end) continue;  // chunk culled by the cutoff (block-uniform)
  const Stager st{a.jlist, w.j_begin, w.j_end, (w.j_end - w.j_begin + kStageTiles - 1) / kStageTiles, s_bar, g};
  const float* src[3] = {a.pq, a.lj, a.gb};
  if (threadIdx.x == 0) {
    if (st.n_stages > 0) st.issue<3>(0, s_buf, src);
    if (st.n_stages > 1) st.issue<3>(1, s_buf, src);
  }

  // tiles 4w .. 4w + 3 of the block; a missing one repeats the warp's first
  // (or the block's), with its pairs masked out
  const int n_own = max(0, min(4, w.n_i_tiles - 4 * warp));
  const int it0 = w.i_tile0 + (n_own > 0 ? 4 * warp : 0);
  FarI2 ia[2];
  float2 px[2], py[2], pz[2];
  float ri_max = 0.0f;
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const int ta = it0 + (2 * q < n_own ? 2 * q : 0), tb = it0 + (2 * q + 1 < n_own ? 2 * q + 1 : 0);
    const int i = ta * kTile + lane, j = tb * kTile + lane;
    px[q] = make_float2(a.pq[soa_index(i, 0)], a.pq[soa_index(j, 0)]);
    py[q] = make_float2(a.pq[soa_index(i, 1)], a.pq[soa_index(j, 1)]);
    pz[q] = make_float2(a.pq[soa_index(i, 2)], a.pq[soa_index(j, 2)]);
    ia[q].rm = make_float2(a.lj[soa_index(i, 0)], a.lj[soa_index(j, 0)]);
    ia[q].se = mul2(bc(a.lj_kj12), make_float2(a.lj[soa_index(i, 1)], a.lj[soa_index(j, 1)]));
    ia[q].cg = mul2(bc(a.far_kj), make_float2(a.pq[soa_index(i, 3)], a.pq[soa_index(j, 3)]));
    ri_max = fmaxf(ri_max, fmaxf(a.gb[soa_index(i, 0)], a.gb[soa_index(j, 0)]));
  }
  if (kAllPairs) ri_max = warp_max(ri_max);
  // the next near-field j-tile of each own tile (refs are in j order)
  int mref[4], mnext[4];
  auto load_next = [&](int q, int from) {
    const int end = a.mask_begin[it0 + q + 1];
    mref[q] = from;
    mnext[q] = from < end ? a.mask_refs[from].j_tile : 0x7fffffff;
  };
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    mref[q] = 0;
    mnext[q] = 0x7fffffff;
    if (q < n_own) load_next(q, a.mask_begin[it0 + q]);
  }
  stage_tiles(a, w, 0, s_tiles[g & 1]);
  double(*acc)[kTile] = s_acc[warp];
#pragma unroll
  for (int q = 0; q < 12; ++q) acc[q][lane] = 0.0;

  for (int s = 0; s < st.n_stages; ++s) {
    const uint32_t gs = g + s;
    const int b = gs & 1;
    const bool ok = mbar_wait_bounded(&s_bar[b], (gs >> 1) & 1u);
    if (__syncthreads_or(!ok)) {
      if (threadIdx.x == 0) atomicOr(a.error_flag, kStatusTimeout);
      return;
    }
    const int t0 = w.j_begin + s * kStageTiles;
    const int cnt = min(kStageTiles, w.j_end - t0);
    for (int q = threadIdx.x; q < cnt * kTile; q += W * 32) {  // one tile per warp and trip
      const int t = q / kTile, l = q % kTile;
      const float* p = &s_buf[b][0][t * 128 + l];
      const float* pl = &s_buf[b][1][t * 128 + l];
      const float* pg = &s_buf[b][2][t * 128 + l];
      const float v[kForceCols] = {p[0], p[32], p[64], p[96], pl[0], pl[32], pg[0], pg[32]};
#pragma unroll
      for (int c = 0; c < kForceCols; ++c)
        *reinterpret_cast<float2*>(&s_dup[t][64 * c + 2 * l]) = make_float2(v[c], v[c]);
      if (kAllPairs) {
        const float rmax = warp_max(v[6]);
        if (l == 0) s_rmax[t] = rmax;
      }
    }
    __syncthreads();  // s_dup is complete and raw buffer b is free
    if (threadIdx.x == 0 && s + 2 < st.n_stages) st.issue<3>(s + 2, s_buf, src);
    stage_tiles(a, w, s + 1, s_tiles[b ^ 1]);
    for (int t = 0; t < cnt; ++t) {
      const int jt = s_tiles[b].jt[t];
      unsigned on = 0;  // own tiles that meet this j-tile here
      float gap = INFINITY;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        while (mnext[q] < jt) load_next(q, mref[q] + 1);
        const float4 off = s_tiles[b].off[t][it0 - w.i_tile0 + (q < n_own ? q : 0)];
        if (q < n_own && jt > it0 + q && mnext[q] != jt && (kAllPairs || off.w <= a.pair_cutoff)) {
          on |= 1u << q;
          gap = fminf(gap, off.w);
        }
        if (q & 1) {
          ia[q / 2].nx.y = off.x - px[q / 2].y;
          ia[q / 2].ny.y = off.y - py[q / 2].y;
          ia[q / 2].nz.y = off.z - pz[q / 2].y;
        } else {
          ia[q / 2].nx.x = off.x - px[q / 2].x;
          ia[q / 2].ny.x = off.y - py[q / 2].x;
          ia[q / 2].nz.x = off.z - pz[q / 2].x;
        }
      }
      float* jfx = &s_part[warp][0][t * kTile];
      float* jfy = &s_part[warp][1][t * kTile];
      float* jfz = &s_part[warp][2][t * kTile];
      ForceSum f[2] = {{bc(0.0f), bc(0.0f), bc(0.0f)}, {bc(0.0f), bc(0.0f), bc(0.0f)}};
      if (kAllPairs && on == 0xFu && far_tiles(gap, ri_max, s_rmax[t])) {
        force_far_four(s_dup[t], ia, jfx, jfy, jfz, lane, f);
      } else {
        jfx[lane] = 0.0f;
        jfy[lane] = 0.0f;
        jfz[lane] = 0.0f;
        if (on == 0u) continue;
        __syncwarp();
#pragma unroll 1
        for (int q = 0; q < 2; ++q) {
          const bool va = (on >> (2 * q)) & 1u, vb = (on >> (2 * q)) & 2u;
          if (!(va || vb)) continue;
          const int ta = it0 + (2 * q < n_own ? 2 * q : 0), tb = it0 + (2 * q + 1 < n_own ? 2 * q + 1 : 0);
          const IAtom2 gi = i_pair(a, ta * kTile + lane, tb * kTile + lane, q ? ia[1] : ia[0]);
          ForceSum fq{bc(0.0f), bc(0.0f), bc(0.0f)};
          force_pair_tile<kAllPairs>(s_dup[t], gi, a, va, vb, jfx, jfy, jfz, lane, &fq);
          if (q) f[1] = fq;
          else f[0] = fq;
        }
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        acc[3 * q][lane] += static_cast<double>(half_of(f[q / 2].x, q & 1));
        acc[3 * q + 1][lane] += static_cast<double>(half_of(f[q / 2].y, q & 1));
        acc[3 * q + 2][lane] += static_cast<double>(half_of(f[q / 2].z, q & 1));
      }
    }
    __syncthreads();  // every warp is done with s_dup and has written its j partials
    unsigned long long* dst[3] = {a.fx, a.fy, a.fz};
    flush_j<W, 3>(a, s_tiles[b].jt, cnt, s_part, dst, kForceScale);
  }
  g += st.n_stages;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int i = (it0 + q) * kTile + lane;
    if (q < n_own && a.atom_valid[i]) {
      const double vx = acc[3 * q][lane], vy = acc[3 * q + 1][lane], vz = acc[3 * q + 2][lane];
      if (!(isfinite(vx) && isfinite(vy) && isfinite(vz))) atomicOr(a.sys_nonfinite + a.atom_sys[i], 1);
      add_fixed(a.fx + i, vx, kForceScale);
      add_fixed(a.fy + i, vy, kForceScale);
      add_fixed(a.fz + i, vz, kForceScale);
    }
  }
  }
}

// The force pass of k_born_split's shape.
template <bool kAllPairs, bool kPersistent>
__global__ void __launch_bounds__(kSplitWarps * 32) k_force_split(PairArgs a) {
  __shared__ double s_acc[3][kSplitWarps][kTile];
  __shared__ int s_item;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int item = next_item<kPersistent>(a, &s_item, -1); item < a.n_work;
       item = next_item<kPersistent>(a, &s_item, item)) {
    const PairWork w = a.work[item];
    const int it = w.i_tile0, i = it * kTile + lane;
    const float px = a.pq[soa_index(i, 0)], py = a.pq[soa_index(i, 1)], pz = a.pq[soa_index(i, 2)];
    const double4 oi = a.origin[it];
    IAtom2 ia = i_atom(a, i);
    const float ri_max = kAllPairs ? warp_max(ia.R.x) : 0.0f;
    int mref = a.mask_begin[it];
    const int mend = a.mask_begin[it + 1];
    double acc0 = 0.0, acc1 = 0.0, acc2 = 0.0;
    for (int p = w.j_begin; p < w.j_end; ++p) {
      const int jt = a.jlist[p];
      while (mref < mend && a.mask_refs[mref].j_tile < jt) ++mref;
      if (jt <= it || (mref < mend && a.mask_refs[mref].j_tile == jt)) continue;  // near field or counted elsewhere
      const double4 oj = a.origin[jt];
      const float gap = tile_gap(oi, oj);
      if (!kAllPairs && gap > a.pair_cutoff) continue;
      const size_t base = static_cast<size_t>(jt) * 128;
      const bool far = kAllPairs && far_tiles(gap, ri_max, warp_max(a.gb[base + lane]));
      ia.nx = bc(-(px - static_cast<float>(oj.x - oi.x)));
      ia.ny = bc(-(py - static_cast<float>(oj.y - oi.y)));
      ia.nz = bc(-(pz - static_cast<float>(oj.z - oi.z)));
      float2 fx = bc(0.0f), fy = bc(0.0f), fz = bc(0.0f);
#pragma unroll
      for (int q = 0; q < kSplitJ; q += 4) {
        const int k0 = warp * kSplitJ + q;
        const Group4 u = far ? force_far4(a.pq + base + k0, a.lj + base + k0, ia)
                             : force_group4<kAllPairs>(a.pq + base + k0, a.lj + base + k0, a.gb + base + k0, ia, a);
        fx = add2(fx, add2(u.xa, u.xb));
        fy = add2(fy, add2(u.ya, u.yb));
        fz = add2(fz, add2(u.za, u.zb));
        const float t[3] = {reduce_scatter4(u.xa.x, u.xa.y, u.xb.x, u.xb.y, lane),
                            reduce_scatter4(u.ya.x, u.ya.y, u.yb.x, u.yb.y, lane),
                            reduce_scatter4(u.za.x, u.za.y, u.zb.x, u.zb.y, lane)};
        const int j = jt * kTile + k0 + (lane >> 3);
        if ((lane & 7) == 0 && a.atom_valid[j]) {
          if (!(isfinite(t[0]) && isfinite(t[1]) && isfinite(t[2]))) atomicOr(a.sys_nonfinite + a.atom_sys[j], 1);
          add_fixed(a.fx + j, -static_cast<double>(t[0]), kForceScale);
          add_fixed(a.fy + j, -static_cast<double>(t[1]), kForceScale);
          add_fixed(a.fz + j, -static_cast<double>(t[2]), kForceScale);
        }
      }
      acc0 += static_cast<double>(fx.x + fx.y);
      acc1 += static_cast<double>(fy.x + fy.y);
      acc2 += static_cast<double>(fz.x + fz.y);
    }
    s_acc[0][warp][lane] = acc0;
    s_acc[1][warp][lane] = acc1;
    s_acc[2][warp][lane] = acc2;
    __syncthreads();
    if (warp < 3 && a.atom_valid[i]) {
      unsigned long long* dst = warp == 0 ? a.fx : warp == 1 ? a.fy : a.fz;
      const double v = split_sum(s_acc[warp], lane);
      if (!isfinite(v)) atomicOr(a.sys_nonfinite + a.atom_sys[i], 1);
      add_fixed(dst + i, v, kForceScale);
    }
    if (kPersistent) __syncthreads();  // s_acc is read before the next item writes it
  }
}

// The force pass of k_born_pair's shape, over culled lists.
__global__ void __launch_bounds__(kSplitWarps * 32) k_force_pair(PairArgs a) {
  __shared__ float2 s_f[kTile / 4][3][kTile];  // the i side's sums of four j atoms, in the order they are added
  __shared__ unsigned s_live;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  unsigned live = live_pairs(a, &s_live, [&](int it, int jt) {
    bool off = jt == it || tile_gap(a.origin[it], a.origin[jt]) > a.pair_cutoff;
#pragma unroll 4
    for (int m = a.mask_begin[it]; m < a.mask_begin[it + 1]; ++m) off |= a.mask_refs[m].j_tile == jt;  // near field
    return off;
  });
  for (; live; live &= live - 1) {
    const size_t slot = blockIdx.x + static_cast<size_t>(__ffs(live) - 1) * gridDim.x;
    const int2 ij = a.tile_pairs[slot];
    const int it = ij.x, jt = ij.y, i = it * kTile + lane;
    const double4 oi = a.origin[it], oj = a.origin[jt];
    IAtom2 ia = i_atom(a, i);
    ia.nx = bc(-(a.pq[soa_index(i, 0)] - static_cast<float>(oj.x - oi.x)));
    ia.ny = bc(-(a.pq[soa_index(i, 1)] - static_cast<float>(oj.y - oi.y)));
    ia.nz = bc(-(a.pq[soa_index(i, 2)] - static_cast<float>(oj.z - oi.z)));
    const size_t base = static_cast<size_t>(jt) * 128;
#pragma unroll
    for (int q = 0; q < kSplitJ; q += 4) {
      const int k0 = warp * kSplitJ + q;
      const Group4 u = force_group4<false>(a.pq + base + k0, a.lj + base + k0, a.gb + base + k0, ia, a);
      s_f[k0 / 4][0][lane] = add2(u.xa, u.xb);
      s_f[k0 / 4][1][lane] = add2(u.ya, u.yb);
      s_f[k0 / 4][2][lane] = add2(u.za, u.zb);
      const float tx = reduce_scatter4(u.xa.x, u.xa.y, u.xb.x, u.xb.y, lane);
      const float ty = reduce_scatter4(u.ya.x, u.ya.y, u.yb.x, u.yb.y, lane);
      const float tz = reduce_scatter4(u.za.x, u.za.y, u.zb.x, u.zb.y, lane);
      if ((lane & 7) == 0) {
        const int j = k0 + (lane >> 3);
        a.pair_j[pair_at(slot, 3, 0, j)] = -tx;
        a.pair_j[pair_at(slot, 3, 1, j)] = -ty;
        a.pair_j[pair_at(slot, 3, 2, j)] = -tz;
      }
    }
    __syncthreads();
    if (warp < 3) {
      float2 f = bc(0.0f);
#pragma unroll
      for (int k = 0; k < kTile / 4; ++k) f = add2(f, s_f[k][warp][lane]);
      a.pair_i[pair_at(slot, 3, warp, lane)] = f.x + f.y;
    }
    __syncthreads();  // s_f is read before the next pair writes it
  }
}

}  // namespace


namespace {

// One warp per i-block; lanes test 32 j-tiles at a time against each of the
// block's i-tile spheres and append the survivors in order.
__global__ void k_cut_lists(const CutBlock* blocks, int32_t n_blocks, const int32_t* jlist_all,
                            const double4* origin, double cutoff, int32_t* jlist_out, int32_t* seg_end) {
  const int b = static_cast<int>((blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (b >= n_blocks) return;
  const CutBlock cb = blocks[b];
  int count = 0;
  for (int p0 = cb.jb; p0 < cb.je; p0 += 32) {
    const int p = p0 + lane;
    bool keep = false;
    int jt = 0;
    if (p < cb.je) {
      jt = jlist_all[p];
      const double4 oj = origin[jt];
      for (int k = 0; k < cb.n_i_tiles && !keep; ++k) {
        const double4 oi = origin[cb.i_tile0 + k];
        const double dx = oj.x - oi.x, dy = oj.y - oi.y, dz = oj.z - oi.z;
        const double lim = oi.w + oj.w + cutoff + 1e-3;
        keep = dx * dx + dy * dy + dz * dz <= lim * lim;
      }
    }
    const unsigned kept = __ballot_sync(0xffffffffu, keep);
    if (keep) jlist_out[cb.jb + count + __popc(kept & ((1u << lane) - 1u))] = jt;
    count += __popc(kept);
  }
  if (lane == 0) seg_end[cb.i_tile0] = cb.jb + count;
}

}  // namespace

void launch_cut_lists(const CutBlock* blocks, int32_t n_blocks, const int32_t* jlist_all, const double4* origin,
                      double cutoff, int32_t* jlist_out, int32_t* seg_end, cudaStream_t s) {
  if (n_blocks > 0)
    k_cut_lists<<<(n_blocks + 3) / 4, 128, 0, s>>>(blocks, n_blocks, jlist_all, origin, cutoff, jlist_out, seg_end);
}

namespace {

// A persistent launch fills the SMs with resident CTAs (at most one per item).
template <class K>
int persistent_grid(K kernel, int threads, int n_work) {
  static int n_sm = 0;
  if (n_sm == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev);
  }
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, 0);
  return std::max(1, std::min(n_work, std::max(per_sm, 1) * std::max(n_sm, 1)));
}

template <bool P, class K>
void launch_items(K kernel, int threads, const PairArgs& a, cudaStream_t s) {
  if (P) {
    cudaMemsetAsync(a.queue, 0, sizeof(int32_t), s);
    kernel<<<persistent_grid(kernel, threads, a.n_work), threads, 0, s>>>(a);
  } else {
    kernel<<<a.n_work, threads, 0, s>>>(a);
  }
}

// CTAs of k_born_pair and k_force_pair: one per tile pair while they fit the
// chip at once (sixteen per SM), more pairs per CTA then.
int pair_grid(const PairArgs& a) {
  const int most = 16 * std::max(a.n_sm, 1);
  return std::max((a.n_tile_pairs + kPairsPerCta - 1) / kPairsPerCta, std::min(a.n_tile_pairs, most));
}

template <bool AP, bool P>
void force_shape(const PairArgs& a, int shape, cudaStream_t s) {
  switch (shape) {
    case 1: launch_items<P>(k_force<AP, 4, 4, P>, 4 * 32, a, s); break;
    case 2: launch_items<P>(k_force_quad<AP, 4, 3, P>, 4 * 32, a, s); break;
    case 3: launch_items<P>(k_force_quad<AP, 4, 4, P>, 4 * 32, a, s); break;
    case 4: launch_items<P>(k_force_quad<AP, 2, 6, P>, 2 * 32, a, s); break;
    case 5: launch_items<P>(k_force_quad<AP, 2, 7, P>, 2 * 32, a, s); break;
    case 6: launch_items<P>(k_force_quad<AP, 1, 14, P>, 32, a, s); break;
    default:
      if (AP || !a.seg_end) {
        launch_items<P>(k_force_split<AP, P>, kSplitWarps * 32, a, s);
      } else if (a.tile_pairs) {
        k_force_pair<<<pair_grid(a), kSplitWarps * 32, 0, s>>>(a);
        k_collect<3><<<a.n_blocks * kBlockTiles, kCollectWarps * 32, 0, s>>>(a, a.fx, a.fy, a.fz, kForceScale);
      } else {
        launch_items<P>(k_force<false, kBlockTiles, 2, P>, kBlockTiles * 32, a, s);
      }
      break;
  }
}

template <bool P>
void born_shape(const PairArgs& a, int shape, cudaStream_t s) {
  switch (shape) {
    case 1: launch_items<P>(k_born<4, 8, P>, 4 * 32, a, s); break;
    case 2: launch_items<P>(k_born<8, 4, P>, 8 * 32, a, s); break;
    default:
      if (!a.seg_end) {
        launch_items<P>(k_born_split<P>, kSplitWarps * 32, a, s);
      } else if (a.tile_pairs) {
        k_born_pair<<<pair_grid(a), kSplitWarps * 32, 0, s>>>(a);
        k_collect<1><<<a.n_blocks * kBlockTiles, kCollectWarps * 32, 0, s>>>(a, a.born_sum, nullptr, nullptr, kBornScale);
      } else {
        launch_items<P>(k_born<kBlockTiles, 4, P>, kBlockTiles * 32, a, s);
      }
      break;
  }
}

}  // namespace

namespace {
__global__ void k_tile_pairs(const int32_t* row, int2* pairs) {
  const int i = blockIdx.x, first = row[i], n = row[i + 1] - first;
  for (int k = threadIdx.x; k < n; k += blockDim.x) pairs[first + k] = make_int2(i, i + k);
}
}  // namespace

void launch_tile_pairs(const int32_t* pair_row, int n_tiles, int2* tile_pairs, cudaStream_t s) {
  if (n_tiles > 0) k_tile_pairs<<<n_tiles, 128, 0, s>>>(pair_row, tile_pairs);
}

int pair_shape_tiles(bool born, int shape, bool culled) {
  if (shape == 0) return culled ? kBlockTiles : 1;
  if (shape == 1) return 4;
  if (born) return 8;
  return shape <= 3 ? 16 : shape <= 5 ? 8 : 4;
}

void launch_born_pass(const PairArgs& a, const PairLaunch& c, cudaStream_t s) {
  if (a.n_work <= 0) return;
  if (c.persistent && !a.queue) return;
  if (c.persistent) born_shape<true>(a, c.shape, s);
  else born_shape<false>(a, c.shape, s);
}

void launch_force_pass(const PairArgs& a, const PairLaunch& c, cudaStream_t s) {
  if (a.n_work <= 0) return;
  if (c.persistent && !a.queue) return;
  const bool all_pairs = a.nb_c2 == INFINITY && a.gb_c2 == INFINITY;
  if (all_pairs) {
    if (c.persistent) force_shape<true, true>(a, c.shape, s);
    else force_shape<true, false>(a, c.shape, s);
  } else {
    if (c.persistent) force_shape<false, true>(a, c.shape, s);
    else force_shape<false, false>(a, c.shape, s);
  }
}

}  // namespace ogk
