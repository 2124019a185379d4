// xpass.cu -- the x passes, the local-terms kernel, the stage combination and
// the step controller: every kernel that reads the Butcher tableau in constant
// memory (one copy per translation unit, so they stay together).
#include "launch.h"
#include "stages.cuh"

namespace mpx {

XfwdFn xfwd_fn(bool combine, bool pair) {
  if (combine) return pair ? k_xfwd<true, true> : k_xfwd<true, false>;
  return pair ? k_xfwd<false, true> : k_xfwd<false, false>;
}
XinvFn xinv_fn(bool pair) { return pair ? k_xinv<true> : k_xinv<false>; }
LocalFn local_fn() { return k_local; }
CombineFn combine_fn() { return k_combine; }
ControllerFn controller_fn() { return k_controller; }
cudaError_t upload_tableau_symbol(const TableauDev& t, cudaStream_t stream) {
  return cudaMemcpyToSymbolAsync(c_tab, &t, sizeof(t), 0, cudaMemcpyHostToDevice, stream);
}

}  // namespace mpx
