// efe_pcg_slots.cuh -- where the persistent CG kernel (efe_pcg.cu) keeps the scalars its CTAs exchange.  Plain C++.
//
// Every sum over the grid (epoch 1, 2, ...) has one slot per CTA and value.  A CTA posts its part of a value into its
// slot, CTA by CTA one arrival is counted, and when all have arrived every CTA reads all slots, waiting for those
// whose tag is not the epoch's yet.  A CTA that has read its sums may post the next epoch while a slower one still
// reads this one, so consecutive epochs have slots of their own: an epoch's slots are written again two epochs
// later, for which every CTA must have arrived at the epoch between, which it does after its last read of this one.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define EFE_SLOTS_FN __host__ __device__
#else
#define EFE_SLOTS_FN
#endif

namespace efe {

constexpr int PCG_SUMS = 3;       // values of one epoch
constexpr int PCG_EPOCH_SETS = 2; // sets of slots
constexpr int PCG_SLOT_DOUBLES = 2;

// slots of a grid of `grid` CTAs
EFE_SLOTS_FN constexpr int pcg_slots(int grid) { return PCG_EPOCH_SETS * PCG_SUMS * grid; }
// first slot (CTA 0's) of value k in an epoch; CTA i's is i further
EFE_SLOTS_FN constexpr int pcg_slot(uint32_t epoch, int k, int grid) {
  return ((int)(epoch % PCG_EPOCH_SETS) * PCG_SUMS + k) * grid;
}

}  // namespace efe
