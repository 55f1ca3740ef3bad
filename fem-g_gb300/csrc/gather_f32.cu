// Instances of the CSR reduction for FP32 element matrices (the mixed path).
#include "gather.cuh"

namespace femg {

template <typename SlotT, bool KCPLX>
static int pick(const GatherLaunch &a) {
  const GatherShape &g = a.g;
  if (g.blocks3) {
    if (g.VW == 4) return launchGatherShape<SlotT, KCPLX, float, 4, 3, true>(a);
    if (g.VW == 2) return launchGatherShape<SlotT, KCPLX, float, 2, 3, true>(a);
    return launchGatherShape<SlotT, KCPLX, float, 1, 3, true>(a);
  }
  if (g.VW == 4) return launchGatherShape<SlotT, KCPLX, float, 4, 1, false>(a);
  if (g.VW == 2)
    return g.J == 1 ? launchGatherShape<SlotT, KCPLX, float, 2, 1, false>(a) : launchGatherShape<SlotT, KCPLX, float, 2, 3, false>(a);
  return g.J == 3 ? launchGatherShape<SlotT, KCPLX, float, 1, 3, false>(a) : launchGatherShape<SlotT, KCPLX, float, 1, 5, false>(a);
}

int launchGatherF32(const GatherLaunch &a) {
  if (a.slotBytes == 1) return a.kcplx ? pick<uint8_t, true>(a) : pick<uint8_t, false>(a);
  return a.kcplx ? pick<uint16_t, true>(a) : pick<uint16_t, false>(a);
}

}  // namespace femg
