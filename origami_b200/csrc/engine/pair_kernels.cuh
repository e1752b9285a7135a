// Tiled all-pairs / tile-list pair kernels (FP32 pair math, FP64 per-tile
// accumulation, 64-bit fixed-point results) and the FP64 energy kernels.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "step_kernels.cuh"

namespace ogk {

// One unit of pair work: `n_i_tiles` (<= warps per CTA) consecutive i-tiles of
// one system against the j-tiles jlist[j_begin, j_end).
struct PairWork {
  int32_t i_tile0;
  int32_t n_i_tiles;
  int32_t j_begin;
  int32_t j_end;
};

// One i-block of a pair work list: W i-tiles from i_tile0 against the j-tiles
// jlist[jb, je); the system's first tile.
struct CutBlock {
  int32_t i_tile0, n_i_tiles, jb, je, sys_tile0;
};

// Exclusion masks of one ordered (i-tile, j-tile) pair: for i-lane l, bit k
// of ex[l] marks pair (i0+l, j0+k) as excluded (1-2, 1-3 or self), bit k of
// m14[l] as a 1-4 pair.  Entries of one i-tile are sorted by j-tile.
struct TileMaskRef {
  int32_t j_tile;
  int32_t offset;  // index of the 32-word block in the mask arrays
};

struct PairArgs {
  // per padded atom
  // FP32 per-atom data in tile-SoA layout (see soa_index in common.cuh):
  const float* pq;    // columns x_rel, y_rel, z_rel (A, from the tile origin), charge (e)
  const float* lj;    // columns rmin_half, sqrt(eps), rmin_half_14, sqrt(eps_14)   (kcal/mol)
  const float* gb;    // columns R_born, 1/R_born, rho_tilde, s*rho_tilde
  const float* bs;    // with s = s*rho_tilde: columns s^3 / 3, 6/5 s^5, 15/7 s^7, 0
  const double4* origin;  // per tile
  const int32_t* atom_valid;  // 1 for real atoms
  // work
  const PairWork* work;
  int32_t n_work;
  const int32_t* jlist;
  // cutoff mode: per i-block first tile, the end of its culled j range in
  // jlist (the work items' j_end is clamped to it); NULL for all pairs
  const int32_t* seg_end;
  const int32_t* mask_begin;  // per tile: first TileMaskRef, mask_begin[t+1] = end
  const TileMaskRef* mask_refs;
  const uint32_t* mask_ex;
  const uint32_t* mask_14;
  // shape 0 over culled lists, while there are few tile pairs: one CTA per
  // tile pair (i, j >= i), its sums kept as [slot][component][atom] of the
  // i-tile and of the j-tile; the pair of tiles (i, j) is at pair_row[i] + j - i.
  // NULL = the eight-tile kernels
  const int2* tile_pairs;
  int32_t n_tile_pairs;
  const int32_t* pair_row;
  uint8_t* pair_on;  // whether the slot's pair was evaluated; its sums are zero otherwise
  float* pair_i;
  float* pair_j;
  int32_t n_sm;
  const CutBlock* blocks;  // the pass's i-blocks, and its chunk
  int32_t n_blocks, chunk;
  // outputs (fixed point)
  unsigned long long* fx;
  unsigned long long* fy;
  unsigned long long* fz;
  unsigned long long* born_sum;
  // cutoffs squared (INFINITY = none) and constants
  float nb_c2, gb_c2, born_c2;
  float pair_cutoff, born_cutoff;  // A: the larger of the force pass's two, the Born pass's
  float s_max, rho_max;            // largest s*rho_tilde and rho_tilde of any atom
  float far_kj;                    // gb_pref_kj - coul_kj
  float inv_rc3;     // 1/Rc^3 of the reaction field (0 without cutoff)
  float coul_kj;     // 332.0637 * 4.184
  float lj_kj12;     // 12 * 4.184
  float gb_pref_kj;  // (1 - 1/78.5) * 332.0637 * 4.184
  int32_t* error_flag;
  // persistent launches: the work-queue head (zeroed before each launch)
  int32_t* queue;
  // per-system "a force or Born sum was NaN/Inf" flags (fixed point cannot
  // carry a NaN, so it is recorded here and turned into divergence)
  const int32_t* atom_sys;
  int32_t* sys_nonfinite;
  // Near-field tiles (those carrying exclusion / 1-4 masks: the bonded
  // neighbourhood, where large pair forces cancel against the bonded terms)
  // are evaluated in FP64 from these arrays.
  const double* x64; const double* y64; const double* z64;
  const double* q64;
  const double* rmin64; const double* eps64; const double* rmin14_64; const double* eps14_64;
  const double* born_r64;
  double nb_c2_64, gb_c2_64, inv_rc3_64;
};

// Cutoff-mode j lists, rebuilt from the tile origins every force evaluation:
// for each i-block, the j-tiles of jlist_all[jb, je) whose bounding sphere
// comes within `cutoff` of any of the block's tile spheres, kept in order and
// compacted to the front of the same range of jlist_out; seg_end[i_tile0]
// receives the new end.  No atom pair within the cutoff is dropped (sphere
// bounds, FP64, 1e-3 A margin); the pair kernels still apply the cutoff per
// pair.
void launch_cut_lists(const CutBlock* blocks, int32_t n_blocks, const int32_t* jlist_all, const double4* origin,
                      double cutoff, int32_t* jlist_out, int32_t* seg_end, cudaStream_t s);

// How a pair pass is launched.  shape:
//   0 = all pairs: one i-tile per CTA, the four warps splitting each j-tile (few
//       tiles); culled lists (a cutoff): the sums of eight i-tiles per CTA, one
//       per warp, taken by a CTA per tile pair while there are few
//       (kMaxTilePairs), with the same results bit for bit;
//   1 = four i-tiles per CTA, one per warp;
//   Born pass: 2 = eight i-tiles per CTA, one per warp;
//   force pass: 2 to 6 = four i-tiles per warp (many tiles): 2, 3 sixteen per
//       CTA at 3 and 4 CTAs per SM, 4, 5 eight at 6 and 7, 6 four at 14;
// persistent: resident CTAs taking items from PairArgs::queue instead of
// one CTA per item.  The work list must be built for
// pair_shape_tiles i-tiles per item.
struct PairLaunch {
  int shape = 0;
  bool persistent = false;
};
int pair_shape_tiles(bool born, int shape, bool culled);
// PairArgs::tile_pairs from the rows' first slots (n_tiles + 1 of them): row i
// holds (i, i), (i, i + 1), ..
void launch_tile_pairs(const int32_t* pair_row, int n_tiles, int2* tile_pairs, cudaStream_t s);
constexpr int64_t kMaxTilePairs = 1 << 18;  // 200 MB of sums at most
constexpr int kBornShapes = 3;   // shapes 0..2
constexpr int kForceShapes = 7;  // shapes 0..6

void launch_born_pass(const PairArgs& a, const PairLaunch& c, cudaStream_t s);
// Far field (tiles without exclusion masks), FP32.
void launch_force_pass(const PairArgs& a, const PairLaunch& c, cudaStream_t s);
// Near field: near[k] = (i_tile, j_tile, mask block of (i_tile, j_tile), 0)
// for every unordered tile pair (i_tile <= j_tile) that carries masks, FP64;
// each pair once, both atoms' forces.
void launch_near_force64(const PairArgs& a, const int4* near, int n_near, int n_sm, cudaStream_t s);

// FP64 energy evaluation: one warp per i-tile and j range (pair_fp64.cu).
struct EnergyArgs {
  const double* x; const double* y; const double* z;
  const double* q;
  const double* rmin; const double* eps; const double* rmin14; const double* eps14;
  const double* rho_tilde; const double* srho;  // srho = scale * rho_tilde
  const double* born_r;                          // FP64 Born radii
  const double4* origin;                         // per tile, at the current positions
  const int32_t* atom_sys;
  const int2* sys_tiles;      // per system: first tile, tiles
  const SysState* sys_state;  // per system: real atoms
  const int32_t* mask_begin;  // exclusion masks (PairArgs)
  const TileMaskRef* mask_refs;
  const uint32_t* mask_ex;
  const uint32_t* mask_14;
  int32_t n_tiles;
  double nb_cutoff, nb_c2;      // A and A^2; INFINITY = all pairs
  double born_cutoff, born_c2;
  double kappa, crf;  // reaction field constants (0 without cutoff)
  double s_max, rho_max;  // largest srho and rho_tilde of any atom
  // Each i-tile's j-tiles are dealt to n_chunks warps.  part: their Born
  // integrals, [n_chunks][padded atoms]; pair_part: their LJ, Coulomb and GB
  // sums, [3][n_tiles][n_chunks], and pair_count their LJ pairs.
  int32_t n_chunks;
  double* part;
  double* pair_part;
  int32_t* pair_count;
};

// The terms of launch_energy_totals, in its output order.
enum EnergyTerm {
  kTermLj = 0, kTermCoulomb, kTermGbPair, kTermGbSelf, kTermSasa, kTermBond, kTermAngle, kTermDihedral, kTermImproper,
  kTermPairs, kTermClamped, kEnergyTerms
};
struct EnergyTotals {
  const double* sasa;         // per padded atom, NULL without the surface term
  const double* bonded;       // per bonded term
  const int32_t* seg_begin;   // the engine's [atoms | bonds | angles | dihedrals | impropers] segments
  const int32_t* seg_end;
  const int32_t* clamp_count; // per system
  double* out;                // [kEnergyTerms][n_sys], kJ/mol and counts
};

void launch_born64(const EnergyArgs& a, cudaStream_t s);
void launch_energy64(const EnergyArgs& a, cudaStream_t s);
void launch_energy_totals(const EnergyArgs& a, const EnergyTotals& t, int n_sys, cudaStream_t s);
// Warps per i-tile of the FP64 energy path: enough for 24 warps per SM, at
// most one per j-tile of the largest system and 64.
int energy_chunks(int n_tiles, int max_system_tiles, int n_sm);

}  // namespace ogk
