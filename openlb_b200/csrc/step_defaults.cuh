// Which step kernel a lattice takes unless told otherwise, and how its steps are
// launched.
#pragma once

#include <cstddef>

#include "aa_kernels.cuh"

namespace olb_b200 {

// Default step variant per lattice class (the autotuner refines it on the
// actual lattice), from sweeps of cubes of 16..320 cells a side on B200, chained
// launches, us per step:
//   A lattice whose threads all fit the SMs at 3 blocks of 256 takes {1,3}: a
// fourth block per SM has nothing to run and costs registers.  Masked 48^3 (one
// wave) {1,3} 3.71 against {1,4} 4.25 in FP32, 3.84 against 5.77 in FP16 forced
// TRT; 52^3 (two waves) 4.83 against 4.15.  16-bit kernels hold two cells per
// thread: FP16 60^3 3.80 against 4.36, 64^3 4.43 against 4.23.
//   16-bit: D3Q19's two-lane collision fits the 64 registers of {1,4}; D3Q27's
// needs the 80 of {1,3} (160^3 masked BF16 81.6 against 92.9).
//   16-bit, natural layout: two cells per thread (variant 1), but one (variant 0)
// where the lattice leaves lanes to spare and the longer thread shows: D3Q27 up to
// three blocks per SM (forced TRT with walls 33x32x32 4.3 against 7.0, 49x48x48 4.9
// against 7.3; open BGK 33x32x32 4.1 against 5.4, 49x48x48 4.45 against 4.47, 61x60x60
// 7.3 against 6.3), D3Q19 up to two (BGK with walls 41x40x40 3.6 against 4.1; open TRT
// 33x32x32 2.9 against 4.0, 49x48x48 4.2 against 3.5), but not open BGK, the shortest
// (36x34x21 caller-owned 2.8 against 2.6, 17^3 to 33^3 3.4 against 3.2).
//   FP64: {1,3} (160^3 D3Q19 masked 189 against 191 {1,4}; D3Q27 128^3 140 against
// 164 {1,4} and 146 {2,2}), but the forced D3Q27 collisions, whose registers spill
// under the cap of {1,3}, take {2,2} above one wave (forced TRT with walls 64^3 20.9
// against 29.8, 128^3 182 against 243, 160^3 338 against 463; open 128^3 158 against
// 172; in one wave, 36^3 open, 9.1 against 6.6).
//   FP32: {1,4} (64^3 open 5.80 against 6.49 {2,3}, 256^3 open forced TRT 417
// against 430), but two cells per thread {2,3} where they win: from 2^21 cells
// open boxes without a force (256^3 389 against 393, 160^3 100.0 against 99.4 but
// 3 % less with statistics every step, 96^3 16.2 against 15.9) and masked D3Q19
// lattices with one (200^3 207 against 214, 128^3 57.4 against 58.4, 96^3 20.2
// against 19.6; not D3Q27: 144^3 117 against 109, 128^3 84.7 against 78.2).
//   The bound of one wave is that of the collisions without a force; 16-bit D3Q19
// forced TRT would still gain from {1,3} at 64^3 (5.45 against 6.00) and 80^3 (8.96
// against 9.24).
constexpr size_t kSMs = 148;  // of a B200

inline bool is_forced(int kind) { return kind == K_FORCED_BGK || kind == K_FORCED_TRT; }

inline int default_step_variant(int q, int bytes, bool paired, bool masked, int kind, size_t cells)
{
  if (bytes == 2 && !paired) {
    const bool shortest = q == 19 && !masked && kind == K_BGK;
    return !shortest && cells <= kSMs * (q == 27 ? 3 : 2) * kStepThreads ? 0 : 1;
  }
  const bool one_wave = (paired ? (cells + 1) / 2 : cells) <= kSMs * 3 * kStepThreads;
  if (one_wave) return 0;
  if (bytes == 8) return q == 27 && is_forced(kind) ? 2 : 0;
  if (bytes == 2) return q == 27 ? 0 : 1;
  const bool two_cells = is_forced(kind) ? masked && q == 19 : !masked;
  return two_cells && cells >= size_t(1) << 21 ? 3 : 1;
}

// Whether a step of `blocks` blocks may start before the one ahead of it has ended
// (launch_chained).  It hides a launch of 4 to 6 us; but a grid that leaves SMs
// empty then shares SMs with its predecessor, and where a block keeps the FP64 pipe
// of its SM busy by itself, the two take turns: D3Q27 FP64 forced TRT 24^3 (72
// blocks) 6.8 us chained against 6.2, 32^3 (128) 8.3 against 6.2, with walls 10.0
// against 7.7.  With at most 64 blocks two grids fit side by side (20^3 5.8 against
// 6.2), above one block per SM both share anyway (36^3, 216 blocks, 6.6 against
// 8.3).  The collisions without a force gain or are even (28^3 5.2 against 5.6; the
// worst, 32^3 Smagorinsky with walls, 7.3 against 6.2).
inline bool chain_steps(int q, int bytes, int kind, size_t blocks)
{
  return !(bytes == 8 && q == 27 && is_forced(kind) && blocks > 64 && blocks <= kSMs);
}

} // namespace olb_b200
