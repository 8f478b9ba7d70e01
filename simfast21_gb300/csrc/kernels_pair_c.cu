// Radius-pair kernels (kernels_pair.cuh) of the box sides below.
#include "kernels_pair.cuh"

namespace sf21 {

const PairOps* pair_ops_c(int N) {
  switch (N) {
#define SF21_PAIR_SIDE(n)                                \
  case n: {                                              \
    static const PairOps ops = PairLaunch<n>::ops();     \
    return &ops;                                         \
  }
    SF21_PAIR_SIDE(48)
    SF21_PAIR_SIDE(72)
    SF21_PAIR_SIDE(80)
    SF21_PAIR_SIDE(96)
    SF21_PAIR_SIDE(120)
    SF21_PAIR_SIDE(144)
    SF21_PAIR_SIDE(160)
#undef SF21_PAIR_SIDE
    default: return nullptr;
  }
}

}  // namespace sf21
