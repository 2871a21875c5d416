// The column kernels with the budget diagnostics, SPP, inhomogeneity and aerosol options.
#include "cloudsc_kernels.cuh"

namespace cloudsc {

cudaError_t upload_options(const KParams<double> &kd, const KParams<float> &kf, const KParamsD &dd) {
  return upload_unit(kd, kf, dd);
}
ColumnKernel find_options(int form, int v, bool gen, bool fast) {
  switch (form) {
    case 3: return kernel_opt_form<3>(v, gen, fast);
    case 4: return kernel_opt_form<4>(v, gen, fast);
    default: return kernel_opt_form<5>(v, gen, fast);
  }
}

}  // namespace cloudsc
