// The FP32-mixed column kernels.
#include "cloudsc_kernels.cuh"

namespace cloudsc {

cudaError_t upload_mixed(const KParams<double> &kd, const KParams<float> &kf, const KParamsD &dd) {
  return upload_unit(kd, kf, dd);
}
ColumnKernel find_mixed(int v, bool gen, bool fast) {
  return gen && fast ? kernel_form<1>(v) : kernel_general<1, Fields>(fast);
}

}  // namespace cloudsc
