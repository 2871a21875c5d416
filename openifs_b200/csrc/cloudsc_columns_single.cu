// The column kernels of the single-precision interface.
#include "cloudsc_kernels.cuh"

namespace cloudsc {

cudaError_t upload_single(const KParams<double> &kd, const KParams<float> &kf, const KParamsD &dd) {
  return upload_unit(kd, kf, dd);
}
ColumnKernel find_single(int precision, int v, bool gen, bool fast) {
  switch (precision) {
    case 0: return kernel_sp_form<0>(v, gen, fast);
    case 1: return kernel_sp_form<1>(v, gen, fast);
    default: return kernel_sp_form<2>(v, gen, fast);
  }
}

}  // namespace cloudsc
