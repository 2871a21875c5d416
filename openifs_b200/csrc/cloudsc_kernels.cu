// Choice and launch of the column kernels (cloudsc_kernels.cuh).
#include <cuda_runtime.h>
#include <cstdint>
#include "cloudsc_kparams.h"
#include "cloudsc_launch.h"

namespace cloudsc {

// Whether the parameters allow the GEN kernels (gen_exponents_ok).
bool params_allow_gen(const cloudsc_params &p, const Derived &d) {
  KParams<double> kd;
  fill_kparams(p, d, kd);
  return gen_exponents_ok(kd);
}

// Upload the parameters to this device's constant memory (every unit's).
cudaError_t upload_params(const cloudsc_params &p, const Derived &d) {
  KParams<double> kd;
  KParams<float> kf;
  fill_kparams(p, d, kd);
  fill_kparams(p, d, kf);
  KParamsD dd;
  fill_kparams_d(p, dd);
  cudaError_t e = cudaSuccess;
  for (auto up : {upload_fp64, upload_mixed, upload_phys32, upload_options, upload_single, upload_points})
    if (e == cudaSuccess) e = up(kd, kf, dd);
  return e;
}

int num_variants() { return kNumVariants; }
int default_variant() { return kDefaultVariant; }
void variant_bounds(int v, int *maxt, int *minb) {
  *maxt = kVariants[v].maxt;
  *minb = kVariants[v].minb;
}

static ColumnKernel find_kernel(int precision, int v, bool gen, bool fast) {
  switch (precision) {
    case 0: return find_fp64(v, gen, fast);
    case 1: return find_mixed(v, gen, fast);
    case 2: return find_phys32(v, gen, fast);
    case 3:
    case 4:
    case 5: return find_options(precision, v, gen, fast);
    default: return {nullptr, 0, 0};
  }
}
static ColumnKernel find_kernel_sp(int precision, int v, bool gen, bool fast) {
  return precision >= 0 && precision <= 2 ? find_single(precision, v, gen, fast) : ColumnKernel{nullptr, 0, 0};
}

// The largest CTA of the kernel a call runs with variant v.
int kernel_max_threads(int precision, int v, bool gen, int klev, bool sp) {
  const bool fast = klev <= kMaxLevFast;
  return (sp ? find_kernel_sp(precision, v, gen, fast) : find_kernel(precision, v, gen, fast)).maxt;
}

// The variant that runs CTAs of `threads` columns set for variant v.  A build
// that parks values in shared memory takes that of a full CTA, so an SM holds
// one CTA however small; up to 256 threads the 256-thread build, which parks
// nothing and shares an SM, is the faster one for every form (ms, CTAs of 224
// and 128: FP64, 120,000 columns, on the 448-thread build 7.13 and 10.87, on the
// 256-thread one 5.44 and 5.78; FP32-mixed 5.98 and 9.21, 4.34 and 4.17; budgets,
// 60,000 columns, 7.19 and 12.46, 5.70 and 5.79).  -1: the form has no such
// build (parameters that rule out the GEN kernels).  The FP32-physics form parks
// nothing, so its 448-thread build shares an SM already: in the single-precision
// interface CTAs set for the 256-thread variant run on it (CTAs of 256, 65,536
// columns: 2.28 ms against 2.66); its 256-thread build serves few columns, by
// size.
int variant_for_threads(int precision, int v, int threads, bool gen, int klev, bool sp) {
  const bool fast = klev <= kMaxLevFast;
  if (sp && precision == 2 && kVariants[v].maxt == 256) return kDefaultVariant;
  const auto find = [&](int u) { return sp ? find_kernel_sp(precision, u, gen, fast) : find_kernel(precision, u, gen, fast); };
  if (threads > 256 || find(v).smem == 0) return v;
  for (int u = 0; u < kNumVariants; ++u)
    if (kVariants[u].maxt == 256 && kVariants[u].minb == 1 && find(u).maxt == 256) return u;
  return -1;
}

// Variant and CTA size for a call of ncols columns when the caller has set no
// schedule.  A launch is one CTA per SM at a time in every variant, its CTAs
// run in waves, and the time of a wave grows little with the columns in it
// (one warp alone is bound by the latency of its own chain): so the columns
// are spread evenly over the SMs and the waves, and the variant is the one
// with the smallest waves * (time of a wave of that CTA).  The wave times are
// those measured at 137 levels, in microseconds as base + slope per warp
// (FP64; the other forms follow the same order):
//   (256, 1), 255 registers:  2 warps 1230, 4 1273, 8 1428
//   (384, 1), 168 registers:  2 warps 1362, 4 1472, 8 1681, 12 1926
//   (448, 1), 128 registers:  2 warps 1554, 4 1678, 8 1873, 12 2122, 14 2415
// The lines cross where the 255-register build runs out of threads: below 257
// columns per SM it is the fastest at every size, above that one wave of more
// warps beats two of it.  3,200 columns: CTAs of 32 on 100 SMs, 1.21 ms,
// where 448 per CTA on 8 SMs took 2.0; 262,144: 5 waves of 384, 9.4 ms, against
// 4 of 448, 9.7, and 7 of 256, 10.0.
void pick_schedule(int precision, bool gen, int klev, bool sp, long long ncols, int sms, int *variant, int *threads) {
  struct Cost {
    int v;
    double base, slope;
  };
  static const Cost costs[] = {{3, 1165.0, 32.0}, {2, 1250.0, 56.0}, {1, 1420.0, 68.0}};
  double best = 0.0;
  *variant = kDefaultVariant;
  *threads = 0;
  for (const Cost &c : costs) {
    const int maxt = kernel_max_threads(precision, c.v, gen, klev, sp);
    if (maxt != kVariants[c.v].maxt) continue;  // this form has no such build
    const long long per_wave = (long long)sms * maxt;
    const long long waves = (ncols + per_wave - 1) / per_wave;
    const long long ctas = waves * sms;
    int t = (int)((ncols + ctas - 1) / ctas);
    t = (t + 31) / 32 * 32;
    const double cost = (double)waves * (c.base + c.slope * (t / 32));
    if (*threads == 0 || cost < best) {
      best = cost;
      *variant = c.v;
      *threads = t;
    }
  }
}

// Registers and local (spill) bytes per thread of variant v (needs a device).
cudaError_t variant_attributes(int precision, int v, int *regs, int *local_bytes) {
  const ColumnKernel k = find_kernel(precision, v, true, true);
  if (!k.f) return cudaErrorInvalidValue;
  cudaFuncAttributes a;
  cudaError_t e = cudaFuncGetAttributes(&a, k.f);
  if (e != cudaSuccess) return e;
  *regs = a.numRegs;
  *local_bytes = (int)a.localSizeBytes;
  return cudaSuccess;
}

// Once per device: allow every column kernel its parking slots, and find the
// largest local memory (stack frame) per thread of any of them: the spill
// slots and the fast pass's copy of the PLUDE inputs.
cudaError_t prepare_kernels(size_t *max_local) {
  size_t m = 0;
  auto see = [&](const ColumnKernel &k) -> cudaError_t {
    if (!k.f) return cudaSuccess;
    cudaFuncAttributes a;
    cudaError_t e = cudaFuncGetAttributes(&a, k.f);
    if (e == cudaSuccess && a.localSizeBytes > m) m = a.localSizeBytes;
    if (e == cudaSuccess && k.smem)
      e = cudaFuncSetAttribute(k.f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)k.smem);
    return e;
  };
  for (int v = 0; v < kNumVariants; ++v)
    for (int g = 0; g < 2; ++g)
      for (int f = 0; f < 2; ++f) {
        for (int prec = 0; prec <= 5; ++prec) {
          cudaError_t e = see(find_kernel(prec, v, g != 0, f != 0));
          if (e != cudaSuccess) return e;
        }
        for (int prec = 0; prec <= 2; ++prec) {
          cudaError_t e = see(find_kernel_sp(prec, v, g != 0, f != 0));
          if (e != cudaSuccess) return e;
        }
      }
  *max_local = m;
  return cudaSuccess;
}

// Launch variant v of the kernel: precision 0 = FP64, 1 = FP32-mixed,
// 2 = FP32 physics, 3-5 the FP64 forms with budgets / SPP and inhomogeneity;
// gen: the parameters allow the GEN kernels.  threads: at most
// kernel_max_threads.
cudaError_t launch(int precision, int v, const Fields &f, const Shape &sh, int threads, int grid,
                   cudaStream_t stream, bool gen) {
  if (v < 0 || v >= kNumVariants) return cudaErrorInvalidConfiguration;
  const ColumnKernel k = find_kernel(precision, v, gen, sh.klev <= kMaxLevFast);
  if (!k.f) return cudaErrorInvalidValue;
  if (threads > k.maxt) return cudaErrorInvalidConfiguration;
  Fields fa = f;
  Shape sa = sh;
  void *args[] = {&fa, &sa};
  return cudaLaunchKernel(k.f, dim3(grid), dim3(threads), args, k.smem, stream);
}

// The same for form `precision` (0-2) of the single-precision interface.
cudaError_t launch_sp(int precision, int v, const FieldsSP &f, const Shape &sh, int threads, int grid,
                      cudaStream_t stream, bool gen) {
  if (v < 0 || v >= kNumVariants) return cudaErrorInvalidConfiguration;
  const ColumnKernel k = find_kernel_sp(precision, v, gen, sh.klev <= kMaxLevFast);
  if (!k.f) return cudaErrorInvalidValue;
  if (threads > k.maxt) return cudaErrorInvalidConfiguration;
  FieldsSP fa = f;
  Shape sa = sh;
  void *args[] = {&fa, &sa};
  return cudaLaunchKernel(k.f, dim3(grid), dim3(threads), args, k.smem, stream);
}

}  // namespace cloudsc
