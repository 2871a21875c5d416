// The FP32-physics column kernels.
#include "cloudsc_kernels.cuh"

namespace cloudsc {

cudaError_t upload_phys32(const KParams<double> &kd, const KParams<float> &kf, const KParamsD &dd) {
  return upload_unit(kd, kf, dd);
}
ColumnKernel find_phys32(int v, bool gen, bool fast) {
  return gen && fast ? kernel_form<2>(v) : kernel_general<2, Fields>(fast);
}

}  // namespace cloudsc
