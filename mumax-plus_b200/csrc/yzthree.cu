// yzthree.cu -- the y/z passes of y lengths 96, 192, 384 (k_yzw3) and 768 (k_yzw24).
#include "launch.h"

namespace mpx {

YzFn yz_three_fn(int cls, bool one) {
  if (one && cls == 24) return k_yzw3<1, true>;
  if (one && cls == 26) return k_yzw3<4, true>;
  switch (cls) {
    case 24: return k_yzw3<1>;
    case 26: return k_yzw3<4>;
    case 27: return k_yzw3<8>;
    case 28: return k_yzw3<16>;
    case 29: return k_yzw24<1>;
    case 31: return k_yzw24<4>;
    case 32: return k_yzw24<8>;
    default: return k_yzw24<16>;
  }
}

#ifdef MPX_BOUNDS_CHECK
cudaError_t bounds_take_yzthree(unsigned long long* first_bad) { return bounds_take(first_bad); }
#endif

}  // namespace mpx
