// pairs.cu -- the stray-field passes on the pair grid (pairfft.cuh).
#include "launch.h"
#include "pairfft.cuh"

namespace mpx {

PairFn pair_xfwd_fn(bool table) { return table ? k_pair_xfwd<true> : k_pair_xfwd<false>; }
PairFn pair_yfft_fn(int dir) { return dir < 0 ? k_pair_yfft<-1> : k_pair_yfft<1>; }
PairFn pair_zmul_fn(bool mul) { return mul ? k_pair_zmul<true> : k_pair_zmul<false>; }
PairFn pair_yz_fn(int logPz) {
  switch (logPz) {
    case 0: return k_pair_yz<1>;
    case 1: return k_pair_yz<2>;
    case 2: return k_pair_yz<4>;
    default: return k_pair_yz<8>;
  }
}
PairFn pair_xinv_fn() { return k_pair_xinv; }

#ifdef MPX_BOUNDS_CHECK
cudaError_t bounds_take_pairs(unsigned long long* first_bad) { return bounds_take(first_bad); }
#endif

}  // namespace mpx
