// yzwarp.cu -- the warp-column y/z pass k_yzw of y lengths 64 .. 512.
#include "launch.h"

namespace mpx {

YzFn yz_warp_fn(int cls, bool one) {
  if (one) return cls == 10 ? k_yzw<1, true> : k_yzw<4, true>;
  switch (cls) {
    case 10: return k_yzw<1>;
    case 12: return k_yzw<4>;
    case 13: return k_yzw<8>;
    default: return k_yzw<16>;
  }
}

#ifdef MPX_BOUNDS_CHECK
cudaError_t bounds_take_yzwarp(unsigned long long* first_bad) { return bounds_take(first_bad); }
#endif

}  // namespace mpx
