// xthree.cu -- the x passes with rows of 384 and 768 points compiled in, with their
// own copy of the Butcher tableau.
#include "launch.h"

namespace mpx {

XfwdFn xfwd_three_fn(bool combine, XForm f) {
  if (f.one) return combine ? k_xfwd<true, false, true, true> : k_xfwd<false, false, true, true>;
  return combine ? k_xfwd<true, true, false, true> : k_xfwd<false, true, false, true>;
}
XinvFn xinv_three_fn(XForm f) {
  if (f.one) return f.mask ? k_xinv<false, true, true, true> : k_xinv<false, false, true, true>;
  return f.mask ? k_xinv<true, true, false, true> : k_xinv<true, false, false, true>;
}
cudaError_t upload_tableau_three(const TableauDev& t, cudaStream_t stream) {
  return cudaMemcpyToSymbolAsync(c_tab, &t, sizeof(t), 0, cudaMemcpyHostToDevice, stream);
}

#ifdef MPX_BOUNDS_CHECK
cudaError_t bounds_take_xthree(unsigned long long* first_bad) { return bounds_take(first_bad); }
#endif

}  // namespace mpx
