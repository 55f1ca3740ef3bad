// Instances of the group reduction for FP64 element matrices.
#include "multi_gather.cuh"

namespace femg {

template <typename SlotT>
static int pick(const MultiLaunch &a) {
  const GatherShape &g = a.g;
  if (a.in.anyCplx)
    return g.J == 3 ? launchMultiShape<SlotT, double, 1, 3, false, 3, true>(a) : launchMultiShape<SlotT, double, 1, 5, false, 3, true>(a);
  if (g.VW == 2) return g.J == 1 ? launchMultiReal<SlotT, double, 2, 1, false>(a) : launchMultiReal<SlotT, double, 2, 3, false>(a);
  return g.J == 3 ? launchMultiReal<SlotT, double, 1, 3, false>(a) : launchMultiReal<SlotT, double, 1, 5, false>(a);
}

int launchMultiF64(const MultiLaunch &a) { return a.p->slotBytes == 1 ? pick<uint8_t>(a) : pick<uint16_t>(a); }

}  // namespace femg
