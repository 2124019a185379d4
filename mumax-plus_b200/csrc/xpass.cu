// xpass.cu -- the x passes, the local-terms kernel, the stage combination and
// the step controller: the kernels that read the Butcher tableau in constant
// memory (one copy per translation unit; xthree.cu has the other).
#include "launch.h"
#include "stages.cuh"

namespace mpx {

XfwdFn xfwd_fn(bool combine, XForm f) {
  if (f.three) return xfwd_three_fn(combine, f);
  if (f.one) return combine ? k_xfwd<true, false, true> : k_xfwd<false, false, true>;
  if (combine) return f.pair ? k_xfwd<true, true> : k_xfwd<true, false>;
  return f.pair ? k_xfwd<false, true> : k_xfwd<false, false>;
}
XinvFn xinv_fn(XForm f) {
  if (f.three) return xinv_three_fn(f);
  if (f.one) return f.mask ? k_xinv<false, true, true> : k_xinv<false, false, true>;
  if (f.mask) return f.pair ? k_xinv<true, true> : k_xinv<false, true>;
  return f.pair ? k_xinv<true, false> : k_xinv<false, false>;
}
LocalFn local_fn() { return k_local; }
CombineFn combine_fn() { return k_combine; }
ControllerFn controller_fn() { return k_controller; }
cudaError_t upload_tableau_symbol(const TableauDev& t, cudaStream_t stream) {
  return cudaMemcpyToSymbolAsync(c_tab, &t, sizeof(t), 0, cudaMemcpyHostToDevice, stream);
}

#ifdef MPX_BOUNDS_CHECK
cudaError_t bounds_take_xpass(unsigned long long* first_bad) { return bounds_take(first_bad); }
#endif

}  // namespace mpx
