// Instances of the group reduction for FP32 element matrices (the mixed path).
#include "multi_gather.cuh"

namespace femg {

template <typename SlotT>
static int pick(const MultiLaunch &a) {
  const GatherShape &g = a.g;
  if (a.in.anyCplx) {
    if (g.blocks3) return launchMultiShape<SlotT, float, 1, 3, true, 3, true>(a);
    return g.J == 3 ? launchMultiShape<SlotT, float, 1, 3, false, 3, true>(a) : launchMultiShape<SlotT, float, 1, 5, false, 3, true>(a);
  }
  if (g.blocks3) {
    if (g.VW == 4) return launchMultiReal<SlotT, float, 4, 3, true>(a);
    return g.VW == 2 ? launchMultiReal<SlotT, float, 2, 3, true>(a) : launchMultiReal<SlotT, float, 1, 3, true>(a);
  }
  if (g.VW == 4) return launchMultiReal<SlotT, float, 4, 1, false>(a);
  if (g.VW == 2) return g.J == 1 ? launchMultiReal<SlotT, float, 2, 1, false>(a) : launchMultiReal<SlotT, float, 2, 3, false>(a);
  return g.J == 3 ? launchMultiReal<SlotT, float, 1, 3, false>(a) : launchMultiReal<SlotT, float, 1, 5, false>(a);
}

int launchMultiF32(const MultiLaunch &a) { return a.p->slotBytes == 1 ? pick<uint8_t>(a) : pick<uint16_t>(a); }

}  // namespace femg
