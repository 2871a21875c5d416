// What the units of the column kernels and their dispatch share on the host.
#pragma once
#include <cuda_runtime.h>
#include "cloudsc_common.cuh"
#include "cloudsc_column.cuh"

namespace cloudsc {

// Compiled launch variants: the __launch_bounds__(MAXT, MINB) pairs the
// kernels are built with.  MAXT x MINB threads share an SM's 65,536
// registers, so each pair fixes the register budget per thread (and with it
// the spills) and the CTA size it is meant for; the autotuner picks a
// variant, a CTA size up to its MAXT and the persistence at run time.
// At 262,144 columns, FP64, by size: five waves of 384 columns per CTA at 168
// registers 9.46 ms; four of 448 at 128 registers 9.7; seven of 256 at 255
// registers 10.0 (pick_schedule has the time of a wave of each).
struct Variant {
  int maxt, minb;
};
constexpr Variant kVariants[] = {{640, 1}, {448, 1}, {384, 1}, {256, 1}, {256, 2}, {128, 3}};
constexpr int kNumVariants = sizeof(kVariants) / sizeof(kVariants[0]);
constexpr int kDefaultVariant = 1;  // (448, 1): exists in every form

// A compiled column kernel: its function, the largest CTA it takes and the
// dynamic shared memory of its parking slots.
struct ColumnKernel {
  const void *f;
  int maxt;
  size_t smem;
};

// The units (cloudsc_columns_*.cu, cloudsc_points.cu): the kernel of a variant
// and the upload of the parameters to the unit's constant memory.
#define CLOUDSC_UNIT(NAME) \
  cudaError_t upload_##NAME(const KParams<double> &, const KParams<float> &, const KParamsD &);
CLOUDSC_UNIT(fp64)
CLOUDSC_UNIT(mixed)
CLOUDSC_UNIT(phys32)
CLOUDSC_UNIT(options)
CLOUDSC_UNIT(single)
CLOUDSC_UNIT(points)
#undef CLOUDSC_UNIT
ColumnKernel find_fp64(int v, bool gen, bool fast);
ColumnKernel find_mixed(int v, bool gen, bool fast);
ColumnKernel find_phys32(int v, bool gen, bool fast);
ColumnKernel find_options(int form, int v, bool gen, bool fast);
ColumnKernel find_single(int precision, int v, bool gen, bool fast);

}  // namespace cloudsc
