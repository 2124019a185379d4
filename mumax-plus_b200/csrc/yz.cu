// yz.cu -- the block-wide y/z pass k_yz (y lengths below 64, and 4096): the
// radix-8 form for z lengths up to 8 and y lengths up to 2048, else the radix-16 form.
// (Here and in the other files: z length 2, classes 1, 6, 11 .., does not occur, since
// 2 n - 1 is odd.)
#include "launch.h"

namespace mpx {

YzFn yz_block_fn(int cls) {
  switch (cls) {
    case 0: return k_yz<1, 3>;
    case 2: return k_yz<4, 3>;
    case 3: return k_yz<8, 3>;
    case 5: return k_yz<1, 4>;
    case 7: return k_yz<4, 4>;
    case 8: return k_yz<8, 4>;
    default: return k_yz<16, 4>;  // 4 and 9 (z length 16)
  }
}

#ifdef MPX_BOUNDS_CHECK
cudaError_t bounds_take_yz(unsigned long long* first_bad) { return bounds_take(first_bad); }
#endif

}  // namespace mpx
