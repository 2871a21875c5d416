// The FP64 column kernels.
#include "cloudsc_kernels.cuh"

namespace cloudsc {

cudaError_t upload_fp64(const KParams<double> &kd, const KParams<float> &kf, const KParamsD &dd) {
  return upload_unit(kd, kf, dd);
}
ColumnKernel find_fp64(int v, bool gen, bool fast) {
  return gen && fast ? kernel_form<0>(v) : kernel_general<0, Fields>(fast);
}

}  // namespace cloudsc
