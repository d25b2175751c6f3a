// Which step kernel a lattice takes unless told otherwise.
#pragma once

namespace olb_b200 {

// Default step variant per lattice class, from a 256^3 sweep on B200 (the
// autotuner refines it on the actual lattice): masked lattices and 16-bit
// storage keep one cell per thread at high occupancy; FP64 and unmasked
// FP32 lattices issue the loads of two cells per thread.
inline int default_step_variant(int q, int bytes, bool masked)
{
  // 16-bit: D3Q19's two-lane collision fits the 64-register cap of {1,4};
  // D3Q27's needs the 80 registers of {1,3}
  if (bytes == 2) return q == 27 ? 0 : 1;
  if (masked) return bytes == 8 ? 0 : 1;  // {1,3} / {1,4}
  return bytes == 8 ? 2 : 3;              // {2,2} / {2,3}
}

} // namespace olb_b200
