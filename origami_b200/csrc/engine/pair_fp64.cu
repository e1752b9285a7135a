// FP64 pair kernels: the near-field force tiles of the force path and the
// energy path (Born radii and LJ / Coulomb / GB pair energies).
#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "pair_kernels.cuh"

namespace ogk {

// ------------------------------------------------------- FP64 near field
// One warp per unordered near-field tile pair (i-tile <= j-tile) -- the
// tiles that carry exclusion / 1-4 masks, i.e. the bonded neighbourhood
// where the large LJ and Coulomb pair forces cancel against the bonded terms.
// FP64 throughout, the terms of forces_nonbonded.rs:196-232 +
// forces_gb.rs:82-111 with their square roots and divisions rewritten as
// reciprocal square roots and products (equal up to rounding; see the pair
// loop).  Each pair is evaluated once (Newton's third law):
// the j-tile's atoms are staged in the warp's shared memory, lane l meets
// partner (l + k) mod 32 at step k, so within a step every lane touches a
// different partner and the j-side sums need no atomics.  On a diagonal tile
// pair steps 1..16 cover every pair once (step 16 on the lower half-warp
// only).  The pair coefficient is symmetric in i and j, so the j-side force
// is exactly the negated i-side term.
//
// kBlock and kBlockInOrder give a tile pair to the four warps of a block, each
// taking every fourth step: a warp's 32 steps are a chain of FP64 latency (about
// 20 us), which is the kernel's time when there are too few tile pairs to fill
// the SMs.  kBlock adds the warps' sums in warp order.  kBlockInOrder, for
// engines with cutoffs, whose results do not depend on what else is in the
// engine (pair_kernels.cu, k_born_pair), keeps the steps' coefficients in shared
// memory, and two warps add the i and the j side step by step: the sums of
// kWarp, bit for bit (20 residues 12.7 us, by events around the launch, against
// 12.5 of kBlock and 22.3 of kWarp).
enum NearShape { kWarp, kBlock, kBlockInOrder };
namespace {

constexpr int kNearWarps = 4;
// Tile pairs per SM up to which a block takes one.
#ifndef OG_NEAR_SPLIT
#define OG_NEAR_SPLIT 16
#endif
constexpr int kNearSplitPerSm = OG_NEAR_SPLIT;

// The j-tile staged per warp: eps as its square root (the LJ mixing rule
// sqrt(eps_i eps_j) as a product) and the Born radius with its inverse.
struct NearTile {
  double x[kTile], y[kTile], z[kTile], q[kTile], r[kTile], ir[kTile];
  double rmin[kTile], seps[kTile], rmin14[kTile], seps14[kTile];
  int32_t valid[kTile];
};
struct NearForce {
  double x[kTile], y[kTile], z[kTile];
};

template <NearShape kShape>
__global__ void __launch_bounds__(kNearWarps * 32) k_near64(PairArgs a, const int4* __restrict__ near, int n_near) {
  constexpr bool kSplit = kShape != kWarp, kInOrder = kShape == kBlockInOrder;
  __shared__ NearTile tiles[kSplit ? 1 : kNearWarps];
  __shared__ NearForce jf[kInOrder ? 1 : kNearWarps];      // j sums; in order: the i atoms' positions
  __shared__ NearForce sf[kShape == kBlock ? kNearWarps : 1];
  __shared__ double s_coeff[kInOrder ? kTile : 1][kTile];  // in order: [step][lane]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wid = kSplit ? static_cast<int>(blockIdx.x) : static_cast<int>(blockIdx.x) * kNearWarps + warp;
  if (wid >= n_near) return;  // block-uniform when split
  const int part = kSplit ? warp : 0;
  NearTile& t = tiles[kSplit ? 0 : warp];
  NearForce& f = jf[kInOrder ? 0 : warp];
  const int4 w = near[wid];  // i_tile, j_tile (>= i_tile), mask block of (i_tile, j_tile)
  const int i = w.x * kTile + lane;
  const int jl = w.y * kTile + lane;  // this lane's j atom, staged for the warp
  if (part == 0) {
    t.x[lane] = a.x64[jl];
    t.y[lane] = a.y64[jl];
    t.z[lane] = a.z64[jl];
    t.q[lane] = a.q64[jl];
    t.r[lane] = a.born_r64[jl];
    t.ir[lane] = 1.0 / a.born_r64[jl];
    t.rmin[lane] = a.rmin64[jl];
    t.seps[lane] = sqrt(a.eps64[jl]);
    t.rmin14[lane] = a.rmin14_64[jl];
    t.seps14[lane] = sqrt(a.eps14_64[jl]);
    t.valid[lane] = a.atom_valid[jl];
  }
  if (!kInOrder) f.x[lane] = f.y[lane] = f.z[lane] = 0.0;
  const uint32_t ex = a.mask_ex[w.z * kTile + lane];
  const uint32_t m14 = a.mask_14[w.z * kTile + lane];
  const bool valid_i = a.atom_valid[i] != 0;
  const double xi = a.x64[i], yi = a.y64[i], zi = a.z64[i], qi = a.q64[i], Ri = a.born_r64[i];
  const double rmi = a.rmin64[i], sepi = sqrt(a.eps64[i]), rm14i = a.rmin14_64[i], sep14i = sqrt(a.eps14_64[i]);
  const double iRi = 1.0 / Ri;
  const double coul_kj = kCoulomb * kKcalToKj;
  const double gb_pref = (1.0 - 1.0 / kEpsWater) * kCoulomb * kKcalToKj;
  const bool diag = w.x == w.y;
  double ax = 0.0, ay = 0.0, az = 0.0;
  if (kInOrder && part == 0) {
    f.x[lane] = xi;
    f.y[lane] = yi;
    f.z[lane] = zi;
  }
  if (kSplit) __syncthreads();
  else __syncwarp();
  for (int k = (diag ? 1 : 0) + part; k < (diag ? 17 : kTile); k += kSplit ? kNearWarps : 1) {
    const int p = (lane + k) & (kTile - 1);
    double coeff = 0.0, dx = 0.0, dy = 0.0, dz = 0.0;
    if (valid_i && t.valid[p] && !(diag && k == 16 && lane >= 16)) {
      dx = t.x[p] - xi;
      dy = t.y[p] - yi;
      dz = t.z[p] - zi;
      const double r2 = dx * dx + dy * dy + dz * dz;
      const double qq = qi * t.q[p];
      if (r2 >= 1e-18) {
        // 1/r from one reciprocal square root; the GB factor
        // (1/f^2) ((2r - r e / 2) / (2f)) / r of the reference is
        // (1 - e/4) / f^3, and f^-1 another reciprocal square root
        const double inv_r = rsqrt(r2);
        const double inv_r2 = inv_r * inv_r;
        if (!((ex >> p) & 1u) && r2 <= a.nb_c2_64) {
          const bool is14 = (m14 >> p) & 1u;
          const double rmin = is14 ? rm14i + t.rmin14[p] : rmi + t.rmin[p];
          const double eps = is14 ? sep14i * t.seps14[p] : sepi * t.seps[p];
          const double ratio2 = rmin * rmin * inv_r2;
          const double r6 = ratio2 * ratio2 * ratio2;
          coeff += 12.0 * eps * inv_r2 * (r6 - r6 * r6) * kKcalToKj;
          if (qq != 0.0) coeff += -coul_kj * qq * (inv_r2 * inv_r - a.inv_rc3_64);
        }
        if (qq != 0.0 && r2 <= a.gb_c2_64) {
          const double rp = Ri * t.r[p];
          const double e = exp(-0.25 * r2 * (iRi * t.ir[p]));
          const double inv_f = rsqrt(r2 + rp * e);
          coeff += gb_pref * qq * (1.0 - 0.25 * e) * (inv_f * inv_f * inv_f);
        }
      }
    }
    if (kInOrder) {
      s_coeff[k][lane] = coeff;
    } else {
      ax += dx * coeff;
      ay += dy * coeff;
      az += dz * coeff;
      f.x[p] -= dx * coeff;
      f.y[p] -= dy * coeff;
      f.z[p] -= dz * coeff;
      __syncwarp();
    }
  }
  if (kSplit) {
    if (kShape == kBlock) {
      sf[warp].x[lane] = ax;
      sf[warp].y[lane] = ay;
      sf[warp].z[lane] = az;
    }
    __syncthreads();
    if (warp >= 2) return;
    // warp 0: the i side, warp 1: the j side
    if (kShape == kBlock) {
      const NearForce* side = warp == 0 ? sf : jf;
      ax = ay = az = 0.0;
#pragma unroll
      for (int w = 0; w < kNearWarps; ++w) {
        ax += side[w].x[lane];
        ay += side[w].y[lane];
        az += side[w].z[lane];
      }
    } else if (warp == 0) {
      // atom `lane` with partner (lane + k) mod 32 at step k; a pair that is not
      // counted has the coefficient 0
#pragma unroll 8
      for (int k = diag ? 1 : 0; k < (diag ? 17 : kTile); ++k) {
        const int p = (lane + k) & (kTile - 1);
        const double c = s_coeff[k][lane];
        ax += (t.x[p] - xi) * c;
        ay += (t.y[p] - yi) * c;
        az += (t.z[p] - zi) * c;
      }
    } else {
      // atom `lane` with the i atom (lane - k) mod 32
      const double xj = t.x[lane], yj = t.y[lane], zj = t.z[lane];
#pragma unroll 8
      for (int k = diag ? 1 : 0; k < (diag ? 17 : kTile); ++k) {
        const int l = (lane - k) & (kTile - 1);
        const double c = s_coeff[k][l];
        ax -= (xj - f.x[l]) * c;
        ay -= (yj - f.y[l]) * c;
        az -= (zj - f.z[l]) * c;
      }
    }
    const int at = warp == 0 ? i : jl;
    if (warp == 0 ? valid_i : t.valid[lane] != 0) {
      if (!(isfinite(ax) && isfinite(ay) && isfinite(az))) atomicOr(a.sys_nonfinite + a.atom_sys[at], 1);
      add_fixed(a.fx + at, ax, kForceScale);
      add_fixed(a.fy + at, ay, kForceScale);
      add_fixed(a.fz + at, az, kForceScale);
    }
    return;
  }
  if (valid_i) {
    if (!(isfinite(ax) && isfinite(ay) && isfinite(az))) atomicOr(a.sys_nonfinite + a.atom_sys[i], 1);
    add_fixed(a.fx + i, ax, kForceScale);
    add_fixed(a.fy + i, ay, kForceScale);
    add_fixed(a.fz + i, az, kForceScale);
  }
  if (t.valid[lane]) {
    const double bx = f.x[lane], by = f.y[lane], bz = f.z[lane];
    if (!(isfinite(bx) && isfinite(by) && isfinite(bz))) atomicOr(a.sys_nonfinite + a.atom_sys[jl], 1);
    add_fixed(a.fx + jl, bx, kForceScale);
    add_fixed(a.fy + jl, by, kForceScale);
    add_fixed(a.fz + jl, bz, kForceScale);
  }
}

}  // namespace

void launch_near_force64(const PairArgs& a, const int4* near, int n_near, int n_sm, cudaStream_t s) {
  if (n_near <= 0) return;
  const int block = kNearWarps * 32;
  if (n_near > kNearSplitPerSm * n_sm)
    k_near64<kWarp><<<(n_near + kNearWarps - 1) / kNearWarps, block, 0, s>>>(a, near, n_near);
  else if (a.nb_c2_64 != INFINITY || a.gb_c2_64 != INFINITY)
    k_near64<kBlockInOrder><<<n_near, block, 0, s>>>(a, near, n_near);
  else
    k_near64<kBlock><<<n_near, block, 0, s>>>(a, near, n_near);
}

// ----------------------------------------------------------------- FP64 path
//
// Energies: one warp owns a 32-atom i-tile and every n_chunks-th j-tile (its
// j-tiles staged in the warp's shared memory, read back as broadcasts), so a
// single chain spreads over n_tiles x n_chunks warps.  Bound by the FP64
// pipe, so what counts is FP64 operations per pair; a closed form per ordered
// pair with its roots, divisions, logarithm and exponential took 620 us for the
// call for a 4 694-atom chain, all pairs; this takes 153.  (A reciprocal and a
// root of our own took 137, without CUDA's handling of zero: coincident atoms
// need it.)
//   * The pair energies see each unordered pair once (tiles jt >= it) and
//     take 1/r from one reciprocal square root.
//   * Tile pairs are classed by the gap between their bounding spheres: the
//     distant ones need no exponential in the GB term (and then share q / r
//     with Coulomb: 20 operations per pair), and in the descreening integral
//     a short series in u = 1/r^2 instead of two divisions, a square root and
//     a logarithm (22 operations with 8 terms).
//   * With cutoffs, tile pairs whose spheres are apart are skipped.
// Sums run in a fixed order: per lane over its pairs, warp butterflies,
// then k_energy_totals.

namespace {

constexpr int kEnergyWarps = 4;

__device__ __forceinline__ double descreen64(double r, double r2, double inv_r, double rho_i, double s_rho_j) {
  // energy/src/gb.rs:347-369, with 1/r given.
  if (r + s_rho_j <= rho_i) return 0.0;
  const double l = (r - s_rho_j < rho_i) ? rho_i : r - s_rho_j;
  const double u = r + s_rho_j;
  if (u <= 0.0 || l <= 0.0) return 0.0;
  const double inv_l = 1.0 / l, inv_u = 1.0 / u;
  const double d2 = inv_u * inv_u - inv_l * inv_l;
  const double term1 = 0.5 * (inv_l - inv_u);
  const double term2 = (r * 0.25) * d2;
  const double term3 = (0.5 * inv_r) * log(l * inv_u);
  const double term4 = (s_rho_j * s_rho_j - r2) * (0.25 * inv_r) * d2;
  return term1 + term2 + term3 + term4;
}

// The same function where the spheres do not overlap (l = r - s), as its
// series (see k_born): h = -s^3 u^2 sum_k k (2k - 1) / (2k + 1) w^(k - 1),
// w = s^2 u, u = 1 / r^2.  Dropped terms stay below 2^-53 of the first: 15
// terms for s / r < 1/4 (16^-15 * 45 = 3.9e-17), 8 below 1/16 (256^-8 * 24 =
// 1.3e-18), 6 below 1/32 (1024^-6 * 18), 5 below 1/64 (4096^-5 * 15).  The
// closed form loses digits to cancellation at these distances; the series
// does not.
template <int kTerms>
__device__ __forceinline__ double descreen_series64(double w) {
  double p = 0.0;
#pragma unroll
  for (int k = kTerms; k >= 1; --k) p = fma(p, w, static_cast<double>(k * (2 * k - 1)) / (2 * k + 1));
  return p;
}

// Lower bound on the distance of any atom pair of two tiles (spheres of the
// current positions, the margin of k_cut_lists).
__device__ __forceinline__ double tile_gap64(double4 oi, double4 oj) {
  const double dx = oj.x - oi.x, dy = oj.y - oi.y, dz = oj.z - oi.z;
  return sqrt(dx * dx + dy * dy + dz * dz) - (oi.w + oj.w + 1e-3);
}

__device__ __forceinline__ double warp_max64(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

struct BornTile {
  double4 p[kTile];  // x, y, z, s rho~
  double2 s[kTile];  // s^2, s^3
};

// The negated sum over a distant j-tile.
template <int kTerms, bool kCut>
__device__ __forceinline__ double born_far64(const BornTile& t, int nj, double xi, double yi, double zi, double c2) {
  double acc = 0.0;
#pragma unroll 2
  for (int k = 0; k < nj; ++k) {
    const double4 pj = t.p[k];
    const double2 sj = t.s[k];
    const double dx = pj.x - xi, dy = pj.y - yi, dz = pj.z - zi;
    const double r2 = dx * dx + dy * dy + dz * dz;
    const double u = 1.0 / r2;
    const double h = (u * u * sj.y) * descreen_series64<kTerms>(sj.x * u);
    if (!kCut || !(r2 > c2)) acc += h;
  }
  return acc;
}

__global__ void __launch_bounds__(kEnergyWarps * 32) k_born64(EnergyArgs a) {
  __shared__ BornTile tiles[kEnergyWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int it = blockIdx.x * kEnergyWarps + warp;
  const int c = blockIdx.y;
  if (it >= a.n_tiles) return;
  BornTile& t = tiles[warp];
  const int sys = a.atom_sys[it * kTile];
  const int2 st = a.sys_tiles[sys];
  const int end = st.x * kTile + a.sys_state[sys].n_atoms;
  const int i = it * kTile + lane;
  const int il = i < end ? i : it * kTile;  // padding lanes repeat the tile's first atom (for the votes)
  const double xi = a.x[il], yi = a.y[il], zi = a.z[il], rho = a.rho_tilde[il];
  const bool cut = a.born_c2 != INFINITY;
  const double4 oi = a.origin[it];
  const double gap15 = fmax(4.0 * a.s_max, a.s_max + a.rho_max);
  double acc = 0.0;
  for (int jt = st.x + c; jt < st.x + st.y; jt += a.n_chunks) {
    const double gap = tile_gap64(oi, a.origin[jt]);
    if (cut && gap > a.born_cutoff) continue;
    const int j0 = jt * kTile, nj = min(kTile, end - j0);
    __syncwarp();
    if (lane < nj) {
      const double s = a.srho[j0 + lane];
      t.p[lane] = make_double4(a.x[j0 + lane], a.y[j0 + lane], a.z[j0 + lane], s);
      t.s[lane] = make_double2(s * s, s * s * s);
    }
    __syncwarp();
    if (gap >= gap15) {
      const double q = gap / a.s_max;  // at least r / s for every pair
      if (cut) acc -= q >= 16.0 ? born_far64<8, true>(t, nj, xi, yi, zi, a.born_c2)
                                : born_far64<15, true>(t, nj, xi, yi, zi, a.born_c2);
      else if (q >= 64.0) acc -= born_far64<5, false>(t, nj, xi, yi, zi, 0.0);
      else if (q >= 32.0) acc -= born_far64<6, false>(t, nj, xi, yi, zi, 0.0);
      else if (q >= 16.0) acc -= born_far64<8, false>(t, nj, xi, yi, zi, 0.0);
      else acc -= born_far64<15, false>(t, nj, xi, yi, zi, 0.0);
      continue;
    }
    const int self = il - j0;
    for (int k = 0; k < nj; ++k) {
      const double4 pj = t.p[k];
      const double dx = pj.x - xi, dy = pj.y - yi, dz = pj.z - zi;
      const double r2 = dx * dx + dy * dy + dz * dz;
      const double inv_r = rsqrt(r2);
      const double r = r2 * inv_r;
      const bool on = k != self && !(r2 > a.born_c2) && !(r2 < 1e-18);
      double h;
      if (__all_sync(0xffffffffu, r - pj.w >= rho && r > 4.0 * pj.w)) {
        const double2 sj = t.s[k];
        const double u = inv_r * inv_r;
        h = -(u * u * sj.y) * descreen_series64<15>(sj.x * u);
      } else {
        h = on ? descreen64(r, r2, inv_r, rho, pj.w) : 0.0;
      }
      if (on) acc += h;
    }
  }
  if (i < end) a.part[static_cast<size_t>(c) * a.n_tiles * kTile + i] = acc;
}

// The j-tile staged per warp.
struct EnergyTile {
  double4 p[kTile];  // x, y, z, q
  double4 g[kTile];  // Rmin/2, sqrt(eps), R, 1/R
};

// LJ + RF Coulomb within the nonbonded cutoff with exclusions / 1-4
// parameters (nonbonded.rs:127-169) and the GB pair energy over all pairs
// (gb.rs:160-173), each unordered pair once.  LJ as sqrt(eps_i eps_j) (r6^2 -
// 2 r6); every sum without its constant prefactor (k_energy_totals).
//
// Once r2 / (4 R_i R_j) >= 40, R_i R_j exp(-r2 / (4 R_i R_j)) < r2 2^-54 (e^-40
// < 160 2^-54, and the gap only widens), below half an ulp of r2: f_GB = r
// there, for a whole tile pair when its gap and largest radii say so.
__global__ void __launch_bounds__(kEnergyWarps * 32) k_energy64(EnergyArgs a) {
  __shared__ EnergyTile tiles[kEnergyWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int it = blockIdx.x * kEnergyWarps + warp;
  const int c = blockIdx.y;
  if (it >= a.n_tiles) return;
  EnergyTile& t = tiles[warp];
  const int sys = a.atom_sys[it * kTile];
  const int2 st = a.sys_tiles[sys];
  const int end = st.x * kTile + a.sys_state[sys].n_atoms;
  const int i = it * kTile + lane;
  const bool valid = i < end;
  const int il = valid ? i : it * kTile;
  const double xi = a.x[il], yi = a.y[il], zi = a.z[il], qi = a.q[il], Ri = a.born_r[il];
  const double rmi = a.rmin[il], sepi = sqrt(a.eps[il]);
  const double rm14i = a.rmin14[il], sep14i = sqrt(a.eps14[il]);
  const double iRi4 = 0.25 / Ri;
  const double ri_max = warp_max64(Ri);
  const bool cut = a.nb_c2 != INFINITY;
  const double4 oi = a.origin[it];
  int mref = a.mask_begin[it];
  const int mend = a.mask_begin[it + 1];
  // sums without the i atom's factor: LJ (the 1-4 pairs' with it), Coulomb,
  // GB, and q_j / r of the pairs that count for both
  double lj = 0.0, lj14 = 0.0, coul = 0.0, gb = 0.0, both = 0.0;
  int pairs = 0;
  for (int jt = it + c; jt < st.x + st.y; jt += a.n_chunks) {
    while (mref < mend && a.mask_refs[mref].j_tile < jt) ++mref;
    uint32_t ex = 0u, m14 = 0u;
    const bool masked = mref < mend && a.mask_refs[mref].j_tile == jt;
    if (masked) {
      const int w = a.mask_refs[mref].offset * kTile + lane;
      ex = a.mask_ex[w];
      m14 = a.mask_14[w];
    }
    const double gap = tile_gap64(oi, a.origin[jt]);
    const bool nb_tile = !cut || !(gap > a.nb_cutoff);
    const int j0 = jt * kTile, nj = min(kTile, end - j0);
    double rj = 0.0;
    __syncwarp();
    if (lane < nj) {
      const int j = j0 + lane;
      rj = a.born_r[j];
      t.p[lane] = make_double4(a.x[j], a.y[j], a.z[j], a.q[j]);
      t.g[lane] = make_double4(a.rmin[j], sqrt(a.eps[j]), rj, 1.0 / rj);
    }
    __syncwarp();
    const bool far = gap > 0.0 && gap * gap >= 160.0 * ri_max * warp_max64(rj);
    if (far && !masked && !(cut && nb_tile)) {
      if (nb_tile) {
#pragma unroll 2
        for (int k = 0; k < nj; ++k) {
          const double4 pj = t.p[k], gj = t.g[k];
          const double dx = pj.x - xi, dy = pj.y - yi, dz = pj.z - zi;
          const double inv_r = rsqrt(dx * dx + dy * dy + dz * dz);
          const double x = (rmi + gj.x) * inv_r;
          const double x2 = x * x;
          const double r6 = x2 * x2 * x2;
          lj = fma(gj.y, r6 * (r6 - 2.0), lj);
          both = fma(pj.w, inv_r, both);
        }
        pairs += nj;
      } else {
#pragma unroll 2
        for (int k = 0; k < nj; ++k) {
          const double4 pj = t.p[k];
          const double dx = pj.x - xi, dy = pj.y - yi, dz = pj.z - zi;
          gb = fma(pj.w, rsqrt(dx * dx + dy * dy + dz * dz), gb);
        }
      }
      continue;
    }
    const int first = jt == it ? lane + 1 : 0;  // the diagonal tile's pairs once
    for (int k = 0; k < nj; ++k) {
      const double4 pj = t.p[k], gj = t.g[k];
      const double dx = pj.x - xi, dy = pj.y - yi, dz = pj.z - zi;
      const double r2 = dx * dx + dy * dy + dz * dz;
      const bool on = valid && k >= first;
      const double inv_r = rsqrt(r2);
      const double xg = r2 * (iRi4 * gj.w);
      double inv_f = inv_r;
      if (!__all_sync(0xffffffffu, xg >= 40.0)) inv_f = rsqrt(r2 + Ri * gj.z * exp(-xg));
      if (on) gb += pj.w * inv_f;
      if (!nb_tile) continue;
      const bool nb = on && !(r2 > a.nb_c2) && !((ex >> k) & 1u);
      if (!__any_sync(0xffffffffu, nb)) continue;
      if (nb) {
        const bool is14 = (m14 >> k) & 1u;
        const double x = (is14 ? rm14i + a.rmin14[j0 + k] : rmi + gj.x) * inv_r;
        const double x2 = x * x;
        const double r6 = x2 * x2 * x2;
        const double e = r6 * r6 - 2.0 * r6;  // NaN for coincident atoms, as the reference has it
        if (is14) lj14 += sep14i * sqrt(a.eps14[j0 + k]) * e;
        else lj += gj.y * e;
        const double rf = cut ? fma(a.kappa, r2, inv_r) - a.crf : inv_r;
        if (pj.w != 0.0) coul += pj.w * rf;
        ++pairs;
      }
    }
  }
  // a charge of zero contributes nothing, whatever its pairs
  const bool charged = valid && qi != 0.0;
  double v[3] = {valid ? fma(sepi, lj, lj14) : 0.0, charged ? qi * (coul + both) : 0.0, charged ? qi * (gb + both) : 0.0};
  if (!valid) pairs = 0;
  for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
    for (int k = 0; k < 3; ++k) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
    pairs += __shfl_xor_sync(0xffffffffu, pairs, o);
  }
  if (lane == 0) {
    const size_t m = static_cast<size_t>(a.n_tiles) * a.n_chunks, at = static_cast<size_t>(it) * a.n_chunks + c;
#pragma unroll
    for (int k = 0; k < 3; ++k) a.pair_part[k * m + at] = v[k];
    a.pair_count[at] = pairs;
  }
}

// One block per (system, term): the sums of og_energies in kJ/mol, pair and
// clamp counts as doubles, out[term * n_sys + system].
constexpr int kTotalThreads = 1024;  // one system has a block per term: 21 us with 256, the longest sum's loads in turn

__global__ void __launch_bounds__(kTotalThreads) k_energy_totals(EnergyArgs a, EnergyTotals t) {
  const int sys = blockIdx.x, term = blockIdx.y;
  const int2 st = a.sys_tiles[sys];
  const double pref = -(1.0 - 1.0 / kEpsWater) * kCoulomb;
  double acc = 0.0;
  if (term <= kTermGbPair || term == kTermPairs) {
    const size_t m = static_cast<size_t>(a.n_tiles) * a.n_chunks;
    const size_t k0 = static_cast<size_t>(st.x) * a.n_chunks, k1 = k0 + static_cast<size_t>(st.y) * a.n_chunks;
    for (size_t k = k0 + threadIdx.x; k < k1; k += kTotalThreads)
      acc += term == kTermPairs ? static_cast<double>(a.pair_count[k]) : a.pair_part[term * m + k];
    acc *= term == kTermLj ? kKcalToKj : term == kTermCoulomb ? kCoulomb * kKcalToKj : term == kTermGbPair ? pref * kKcalToKj : 1.0;
  } else if (term == kTermGbSelf) {
    const int i0 = st.x * kTile, i1 = i0 + a.sys_state[sys].n_atoms;
    for (int i = i0 + threadIdx.x; i < i1; i += kTotalThreads) {
      const double qi = a.q[i];
      acc += qi != 0.0 ? (qi * qi) / a.born_r[i] : 0.0;
    }
    acc *= 0.5 * pref * kKcalToKj;
  } else if (term == kTermClamped) {
    acc = threadIdx.x == 0 ? static_cast<double>(t.clamp_count[sys]) : 0.0;
  } else if (term == kTermSasa) {
    if (t.sasa) {
      const int i0 = st.x * kTile, i1 = i0 + a.sys_state[sys].n_atoms;
      for (int i = i0 + threadIdx.x; i < i1; i += kTotalThreads) acc += t.sasa[i];
    }
  } else {
    const int seg = (term - kTermBond + 1) * gridDim.x + sys;
    for (int k = t.seg_begin[seg] + threadIdx.x; k < t.seg_end[seg]; k += kTotalThreads) acc += t.bonded[k];
  }
  __shared__ double sh[kTotalThreads];
  sh[threadIdx.x] = acc;
  __syncthreads();
  for (int w = kTotalThreads / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) sh[threadIdx.x] += sh[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) t.out[term * gridDim.x + sys] = sh[0];
}

}  // namespace

void launch_born64(const EnergyArgs& a, cudaStream_t s) {
  k_born64<<<dim3((a.n_tiles + kEnergyWarps - 1) / kEnergyWarps, a.n_chunks), kEnergyWarps * 32, 0, s>>>(a);
}

void launch_energy64(const EnergyArgs& a, cudaStream_t s) {
  k_energy64<<<dim3((a.n_tiles + kEnergyWarps - 1) / kEnergyWarps, a.n_chunks), kEnergyWarps * 32, 0, s>>>(a);
}

void launch_energy_totals(const EnergyArgs& a, const EnergyTotals& t, int n_sys, cudaStream_t s) {
  k_energy_totals<<<dim3(n_sys, kEnergyTerms), kTotalThreads, 0, s>>>(a, t);
}

int energy_chunks(int n_tiles, int max_system_tiles, int n_sm) {
  const int nc = (24 * n_sm + n_tiles - 1) / std::max(n_tiles, 1);
  return std::max(1, std::min(std::min(nc, max_system_tiles), 64));
}

}  // namespace ogk
