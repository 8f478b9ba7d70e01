// Radius-pair kernels (kernels_pair.cuh) of the box sides below.
#include "kernels_pair.cuh"

namespace sf21 {

const PairOps* pair_ops_f(int N) {
  switch (N) {
#define SF21_PAIR_SIDE(n)                                \
  case n: {                                              \
    static const PairOps ops = PairLaunch<n>::ops();     \
    return &ops;                                         \
  }
    SF21_PAIR_SIDE(432)
    SF21_PAIR_SIDE(480)
    SF21_PAIR_SIDE(576)
    SF21_PAIR_SIDE(600)
#undef SF21_PAIR_SIDE
    default: return nullptr;
  }
}

}  // namespace sf21
