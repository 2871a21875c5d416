// CLOUDSC column kernels for B200 (sm_100a): the kernel template, and what a
// translation unit needs to instantiate some of its forms.  Each form has a
// unit of its own (cloudsc_columns_*.cu), so that they compile side by side;
// each unit has its own copy of the parameters in constant memory.  One thread walks one column through all levels; all NPROMA
// blocks are processed by one persistent launch (a grid-stride loop over
// column tiles).  See cloudsc_column.cuh for the numerical contract.
//
// Compiled with --fmad=false: no multiply-add contraction, so the FP64 kernel
// performs the reference's operations with one rounding each.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

#define CSC_DEV __device__ __forceinline__
// plibm's exp/log tables are read from a shared-memory copy per CTA (filled
// at kernel start): the table lookups sit on the dependent path of every
// exp and pow, and shared-memory latency is below the L1 hit latency of a
// global load.  Measured at 262,144 columns, FP64: 15.75 ms vs 16.05 ms.
#define PLIBM_SMEM_TABLES 1
// Every column of a CTA meets the others at the end of each level, so all
// warps of the CTA run the same stretch of the (very long) level code at the
// same time and share the instruction cache.
#define CSC_LEVEL_SYNC() __syncthreads()
#define CSC_OPAQUE(X) asm volatile("" : "+l"(X))
#define CSC_ANY(C) __any_sync(0xffffffffu, (C))
// Next level's inputs into L2 while the level computes: the warps of a CTA
// start a level together and all wait for its loads, so a DRAM round trip
// shows in full.  Lane i owns input i: it prefetches the line of the warp's
// first and last column (32 columns of a field are two lines), one
// instruction each for all inputs together; both are addresses of elements
// the warp reads.  FP64 at 262,144 columns, 384 columns per CTA: 9.83 -> 9.19
// ms; one warp per SM 1.27 -> 1.22 ms (prefetching by every thread, 24
// instructions a level, had been slower than none).
#define CSC_PREFETCH_SETUP() \
  PrefetchLines<FT, FAST_> pf_(F, ib, jl, s2, s2h, (size_t)np)
#define CSC_PREFETCH(C, OFF) \
  if (C) pf_.level(OFF)
#include <type_traits>

#include "cloudsc_column.cuh"

#include "cloudsc_kparams.h"
#include "cloudsc_launch.h"

namespace cloudsc {

static __constant__ KParams<double> c_kpd;
static __constant__ KParams<float> c_kpf;
static __constant__ KParamsD c_kd;

template <typename Real>
__device__ __forceinline__ const KParams<Real> &KP();
template <>
__device__ __forceinline__ const KParams<double> &KP<double>() { return c_kpd; }
template <>
__device__ __forceinline__ const KParams<float> &KP<float>() { return c_kpf; }

template <typename T>
__device__ __forceinline__ T ld(const T *p) { return __ldg(p); }
// This thread's column of the parking slots (Parked, cloudsc_body.cuh).
extern __shared__ double csc_park[];
__device__ __forceinline__ unsigned park_base() {
  return (unsigned)__cvta_generic_to_shared(csc_park) + threadIdx.x * 8u;
}
__device__ __forceinline__ void atomic_add(uint32_t *p, uint32_t v) { atomicAdd(p, v); }
__device__ __forceinline__ double xabs(double x) { return fabs(x); }
__device__ __forceinline__ float xabs(float x) { return fabsf(x); }
__device__ __forceinline__ double xsign(double a, double b) { return copysign(a, b); }
__device__ __forceinline__ float xsign(float a, float b) { return copysignf(a, b); }

template <typename FT, bool ON>
struct PrefetchLines {
  __device__ __forceinline__ PrefetchLines(const FT &, int, int, size_t, size_t, size_t) {}
  __device__ __forceinline__ void level(size_t) const {}
};
template <typename FT>
struct PrefetchLines<FT, true> {
  static constexpr size_t ES = sizeof(*FT::pt);
  const char *first, *last;  // element of level 0's successor, of the warp's first and last column
  __device__ __forceinline__ PrefetchLines(const FT &F, int ib, int jl, size_t s2, size_t s2h, size_t np) {
    const int lane = threadIdx.x & 31;
    const void *b = nullptr;
    size_t n = 1, m = 0, up = 0;  // species of the array, this lane's, extra levels down
    switch (lane) {
      case 0: b = F.pt; break;
      case 1: b = F.pq; break;
      case 2: b = F.pa; break;
      case 3: b = F.cml_t; break;
      case 4: b = F.cml_q; break;
      case 5: b = F.cml_a; break;
      case 6: case 7: case 8: case 9: b = F.cml_cld; n = 5; m = lane - 6; break;
      case 10: case 11: case 12: case 13: b = F.pclv; n = 5; m = lane - 10; break;
      case 14: b = F.pap; break;
      case 15: b = F.paph; up = 1; break;
      case 16: b = F.pvfl; break;
      case 17: b = F.pvfi; break;
      case 18: case 19: b = F.pludeli; n = 4; m = lane - 18; break;
      case 20: b = F.pmfu; up = 1; break;  // read one level ahead
      case 21: b = F.pmfd; up = 1; break;
      case 22: b = F.plu; up = 1; break;
      case 23: b = F.plude; break;
      case 24: case 25: b = F.psnde; n = 2; m = lane - 24; break;
      default: break;
    }
    const int ib0 = __shfl_sync(0xffffffffu, ib, 0), jl0 = __shfl_sync(0xffffffffu, jl, 0);
    const int ib1 = __shfl_sync(0xffffffffu, ib, 31), jl1 = __shfl_sync(0xffffffffu, jl, 31);
    const size_t sp = lane == 15 ? s2h : s2;
    first = b ? (const char *)b + ES * (((size_t)ib0 * n + m) * sp + jl0 + up * np) : nullptr;
    last = b ? (const char *)b + ES * (((size_t)ib1 * n + m) * sp + jl1 + up * np) : nullptr;
  }
  // off: (level) * NPROMA of the level to fetch
  __device__ __forceinline__ void level(size_t off) const {
    if (first) {
      asm volatile("prefetch.global.L2 [%0];" ::"l"(first + off * ES));
      asm volatile("prefetch.global.L2 [%0];" ::"l"(last + off * ES));
    }
  }
};

}  // namespace cloudsc

#include "cloudsc_body.cuh"
namespace cloudsc {

// Where a kernel's long-lived values wait (Parked, cloudsc_body.cuh): in
// shared memory for the 384- and 448-thread builds of the double-precision
// forms, at most kParkSlots * 8 * 448 = 194 KB of the SM's 227; in registers
// for the 256-thread build, whose 255 registers hold them (-1, which also
// merges the processes of a group into one block), and for the others.
// Parking against leaving them to the compiler's local-memory spills, FP64 at
// 262,144 columns: 10.69 -> 10.00 ms (448 threads), 10.58 -> 10.0 (384);
// FP32-mixed 8.51 -> 7.80.
constexpr int park_threads(int form, int maxt, int minb, bool fast) {
  if (!fast || form == 2 || minb != 1) return 0;
  return maxt == 256 ? -1 : (maxt == 384 || maxt == 448 ? maxt : 0);
}
constexpr size_t park_bytes(int form, int maxt, int minb, bool fast) {
  const int p = park_threads(form, maxt, minb, fast);
  return p > 0 ? (size_t)p * 8 * kParkSlots : 0;
}

// Columns are numbered g = ib * NPROMA + jl over all blocks and dealt to CTAs
// in tiles of blockDim.x consecutive columns (a warp reads 32 neighbouring
// columns: coalesced).  The tile loop is uniform over the CTA and every thread
// runs the level loop, so the per-level barrier is reached by all; a thread
// whose column is outside KIDIA..ICEND computes a valid stand-in column and
// stores nothing.
// FORM selects the arithmetic of the column body:
//   0  FP64, the reference's double build;
//   1  FP32-mixed: FP32 transcendentals, everything else in double;
//   3  FP64 with the cloud budget diagnostics (LCLDBUD*: PEXTRA written);
//   4  FP64 with the SPP perturbations and the cloud-inhomogeneity paths;
//   5  FP64 with both (3 and 4);
//   2  FP32 physics: the process rates in FP32 as well (Real = float); the
//      state, the sink limiters, the 5x5 solve, CLOUD_SUPERSATCHECK and the
//      tendency and flux budgets stay in double.  Float rounding of the rates
//      leaves residues above CLOUDSC's 1e-14 kg/kg thresholds that switch
//      precipitation processes on and off down the column, so this form is
//      faster but further from FP64 (measured tendency errors of 0.3-4 %).
// FT: Fields (the double-precision interface) or FieldsSP (float arrays,
// forms 0-2 only).  GEN: the parameter-exponent pows without their tests for
// the exponents 0.5, 1.5, 2 and 3 (the host launches it when the uploaded
// parameters have none of these, gen_exponents_ok).  FAST (KLEV <=
// kMaxLevFast): every column runs the fast pass (branch-free division, root,
// exp, log and pow); a column whose checks reported is run again with IEEE
// division and plibm's full functions, so that the outputs are those for every
// input (with the budgets, the two passes split PEXTRA's levels between them:
// cloudsc_column, kbud).
template <int FORM, int MAXT, int MINB, typename FT = Fields, bool GEN = false, bool FAST = false>
__global__ void __launch_bounds__(MAXT, MINB) cloudsc_kernel(FT F, Shape sh) {
  // Without parking: let ptxas place part of the register spills in shared memory instead of
  // local memory (a PTX pragma; the spill slots it moves no longer go
  // through L1/L2).  With the shared-memory tables, FP64: 15.29 ms vs
  // 15.75 ms; FP32-mixed: 11.28 ms vs 11.72 ms.
  constexpr int PARK = park_threads(FORM, MAXT, MINB, FAST);
  if constexpr (PARK <= 0) asm volatile(".pragma \"enable_smem_spilling\";");
  plibm_load_tables();
  const long long ncols = (long long)sh.ngpblks * sh.nproma;
  const long long ntiles = (ncols + blockDim.x - 1) / blockDim.x;
  for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const long long g = tile * blockDim.x + threadIdx.x;
    int ib = (int)(g / sh.nproma);
    int jl = (int)(g - (long long)ib * sh.nproma);
    bool active = ib < sh.ngpblks;
    if (active) active = jl >= sh.kidia0 && jl < min(sh.nproma, sh.ngptot - ib * sh.nproma);
    if (!active) {
      ib = 0;
      jl = sh.kidia0;
    }
    if constexpr (FORM >= 3) {
      constexpr bool BUD = FORM == 3 || FORM == 5, OPT = FORM >= 4;
      if constexpr (FAST) {
        double plude_in[kMaxLevFast];
        bool bad = false;
        int kbud = sh.klev;
        cloudsc_column<double, false, BUD, OPT, FT, GEN, kPassFast, PARK>(F, sh, ib, jl, active, &bad, plude_in, &kbud);
        if (__syncthreads_or(bad))
          cloudsc_column<double, false, BUD, OPT, FT, GEN, kPassRedo>(F, sh, ib, jl, bad, nullptr, plude_in,
                                                                       &kbud);
      } else {
        cloudsc_column<double, false, BUD, OPT, FT, GEN>(F, sh, ib, jl, active);
      }
    } else if constexpr (FAST) {
      typedef std::conditional_t<FORM == 2, float, double> Real;
      double plude_in[kMaxLevFast];
      bool bad = false;
      cloudsc_column<Real, FORM != 0, false, false, FT, GEN, kPassFast, PARK>(F, sh, ib, jl, active, &bad, plude_in);
      // The rerun takes the whole CTA (the column code holds a CTA barrier
      // at every level); only the columns that reported store anything.
      if (__syncthreads_or(bad))
        cloudsc_column<Real, FORM != 0, false, false, FT, GEN, kPassRedo>(F, sh, ib, jl, bad, nullptr, plude_in);
    } else {
      typedef std::conditional_t<FORM == 2, float, double> Real;
      cloudsc_column<Real, FORM != 0, false, false, FT, GEN>(F, sh, ib, jl, active);
    }
  }
}

template <int FORM, int MAXT, int MINB, typename FT, bool GEN, bool FAST>
static ColumnKernel column_kernel() {
  return {(const void *)cloudsc_kernel<FORM, MAXT, MINB, FT, GEN, FAST>, MAXT, park_bytes(FORM, MAXT, MINB, FAST)};
}
template <int FORM>
static ColumnKernel kernel_form(int v) {
  switch (v) {
    case 0: return column_kernel<FORM, kVariants[0].maxt, kVariants[0].minb, Fields, true, true>();
    case 1: return column_kernel<FORM, kVariants[1].maxt, kVariants[1].minb, Fields, true, true>();
    case 2: return column_kernel<FORM, kVariants[2].maxt, kVariants[2].minb, Fields, true, true>();
    case 3: return column_kernel<FORM, kVariants[3].maxt, kVariants[3].minb, Fields, true, true>();
    case 4: return column_kernel<FORM, kVariants[4].maxt, kVariants[4].minb, Fields, true, true>();
    default: return column_kernel<FORM, kVariants[5].maxt, kVariants[5].minb, Fields, true, true>();
  }
}
static_assert(kNumVariants == 6, "kernel_form lists every variant");
// Forms 0-2 exist in every variant with GEN and FAST (the parameters of every
// known configuration allow GEN); for parameters that do not, in the (448, 1)
// variant with FAST only; for KLEV above kMaxLevFast, in the (448, 1) variant
// without either.  Forms 3-5 (budgets, SPP, inhomogeneity, aerosols) and the
// single-precision interface exist in fewer variants with GEN and FAST; the
// others map to the (448, 1) one.
template <int FORM, typename FT>
static ColumnKernel kernel_general(bool fast) {
  return fast ? column_kernel<FORM, 448, 1, FT, false, true>() : column_kernel<FORM, 448, 1, FT, false, false>();
}
template <int FORM>
static ColumnKernel kernel_opt_form(int v, bool gen, bool fast) {
  if (!fast || !gen) return kernel_general<FORM, Fields>(fast);
  if (v == 3) return column_kernel<FORM, 256, 1, Fields, true, true>();
  return column_kernel<FORM, 448, 1, Fields, true, true>();
}
template <int FORM>
static ColumnKernel kernel_sp_form(int v, bool gen, bool fast) {
  if (!fast || !gen) return kernel_general<FORM, FieldsSP>(fast);
  if (v == 0) return column_kernel<FORM, 640, 1, FieldsSP, true, true>();
  if (v == 2) return column_kernel<FORM, 384, 1, FieldsSP, true, true>();
  if (v == 3) return column_kernel<FORM, 256, 1, FieldsSP, true, true>();
  return column_kernel<FORM, 448, 1, FieldsSP, true, true>();
}
// Upload the parameters to this unit's constant memory on the current device.
static cudaError_t upload_unit(const KParams<double> &kd, const KParams<float> &kf, const KParamsD &dd) {
  cudaError_t e = cudaMemcpyToSymbol(c_kpd, &kd, sizeof(kd));
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(c_kpf, &kf, sizeof(kf));
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(c_kd, &dd, sizeof(dd));
  return e;
}

}  // namespace cloudsc
