// thick.cu -- the split y/z path of thick magnets (yzsplit.cuh).
#include "launch.h"
#include "yzsplit.cuh"

namespace mpx {

YzFn ycols_fn(int dir, int maxlr) {
  if (dir < 0) return maxlr == 3 ? k_ycols<-1, 3> : k_ycols<-1, 4>;
  return maxlr == 3 ? k_ycols<1, 3> : k_ycols<1, 4>;
}
YzFn zmul_fn(int maxlr) { return maxlr == 3 ? k_zmul<3> : k_zmul<4>; }
YzFn ycw_fn(int dir) { return dir < 0 ? k_ycw<-1> : k_ycw<1>; }
YzFn zcw_fn() { return k_zcw; }

#ifdef MPX_BOUNDS_CHECK
cudaError_t bounds_take_thick(unsigned long long* first_bad) { return bounds_take(first_bad); }
#endif

}  // namespace mpx
