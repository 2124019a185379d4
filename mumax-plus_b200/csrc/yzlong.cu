// yzlong.cu -- the y/z passes of y lengths 1024 (k_yzw32) and 2048 (k_yzw64).
#include "launch.h"

namespace mpx {

YzFn yz_long_fn(int cls) {
  switch (cls) {
    case 15: return k_yzw32<1>;
    case 17: return k_yzw32<4>;
    case 18: return k_yzw32<8>;
    case 19: return k_yzw32<16>;
    case 20: return k_yzw64<1>;
    case 22: return k_yzw64<4>;
    default: return k_yzw64<8>;
  }
}

#ifdef MPX_BOUNDS_CHECK
cudaError_t bounds_take_yzlong(unsigned long long* first_bad) { return bounds_take(first_bad); }
#endif

}  // namespace mpx
