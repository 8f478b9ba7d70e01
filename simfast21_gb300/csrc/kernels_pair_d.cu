// Radius-pair kernels (kernels_pair.cuh) of the box sides below.
#include "kernels_pair.cuh"

namespace sf21 {

const PairOps* pair_ops_d(int N) {
  switch (N) {
#define SF21_PAIR_SIDE(n)                                \
  case n: {                                              \
    static const PairOps ops = PairLaunch<n>::ops();     \
    return &ops;                                         \
  }
    SF21_PAIR_SIDE(192)
    SF21_PAIR_SIDE(200)
    SF21_PAIR_SIDE(216)
    SF21_PAIR_SIDE(240)
    SF21_PAIR_SIDE(288)
#undef SF21_PAIR_SIDE
    default: return nullptr;
  }
}

}  // namespace sf21
