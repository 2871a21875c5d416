// CLOUDSC kernels for B200 (sm_100a): FP64 (the reference's double build) and
// FP32-mixed.  One thread walks one column through all levels; all NPROMA
// blocks are processed by one persistent launch (a grid-stride loop over
// column tiles).  See cloudsc_column.cuh for the numerical contract.
//
// Compiled with --fmad=false: no multiply-add contraction, so the FP64 kernel
// performs the reference's operations with one rounding each.
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

namespace cloudsc {

__constant__ KParams<double> c_kpd;
__constant__ KParams<float> c_kpf;
__constant__ KParamsD c_kd;

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
#include "satadj_point.cuh"

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
// kMaxLevFast): every column runs the fast pass (the branch-free division,
// fast_div); a column whose pass reported an operand outside that division's
// exact window is run again with IEEE division, so that the outputs are
// those of IEEE division for every input (with the budgets, the two passes
// split PEXTRA's levels between them: cloudsc_column, kbud).
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

// CLOUD_SATADJ: one thread per (column, level) point, points numbered
// (ib * KLEV + jk) * NPROMA + jl -- the element offset of a level field -- so
// consecutive threads read consecutive columns of one level (coalesced).  A
// grid-stride loop covers all points of all blocks; levels above NCLDTOP get
// zero tendencies (cloud_satadj.F90:338-345).  256-thread CTAs at 64
// registers (4 CTAs, 32 warps per SM) and up to 64 CTAs per SM in the grid:
// 2.42 ms at 262,144 columns, against 2.55 ms at 80 registers with 16 CTAs
// per SM and 2.61 ms at 48 registers.
// INC: STATE_INCREMENT of the cumulative tendencies fused in
// (callpar.F90:1278-1280): each point writes CML + LOC back into the CML
// arrays it has just read (inc_* not NULL), one addition each, as the
// separate call does.
constexpr int kSatadjThreads = 256;
template <bool INC>
__global__ void __launch_bounds__(kSatadjThreads, 4) satadj_kernel(SatadjFields F, Shape sh) {
  plibm_load_tables();
  const KParams<double> &k = KP<double>();
  const double dt = sh.ptsphy;
  const double zqtmst = 1.0 / dt;
  const unsigned long long np = sh.nproma, kl = sh.klev;
  const unsigned long long npts = (unsigned long long)sh.ngpblks * kl * np;
  const int jktop = k.ncldtop - 1;  // first 0-based level with cloud processes
  int nwarn = 0;
  for (unsigned long long idx = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; idx < npts;
       idx += (unsigned long long)gridDim.x * blockDim.x) {
    const unsigned long long row = idx / np;
    const int jl = (int)(idx - row * np);
    const unsigned long long ib = row / kl;
    const int jk = (int)(row - ib * kl);
    const long long icend = (long long)sh.ngptot - (long long)ib * (long long)np;
    if (jl < sh.kidia0 || jl >= icend) continue;
    if (jk < jktop) {
      F.loc_t[idx] = 0.0;
      F.loc_q[idx] = 0.0;
      F.loc_a[idx] = 0.0;
      F.loc_l[idx] = 0.0;
      F.loc_i[idx] = 0.0;
      if constexpr (INC) {  // + 0.0 as STATE_INCREMENT adds it (turns -0 into +0)
        if (F.inc_t) F.inc_t[idx] = F.inc_t[idx] + 0.0;
        if (F.inc_q) F.inc_q[idx] = F.inc_q[idx] + 0.0;
        if (F.inc_a) F.inc_a[idx] = F.inc_a[idx] + 0.0;
        if (F.inc_l) F.inc_l[idx] = F.inc_l[idx] + 0.0;
        if (F.inc_i) F.inc_i[idx] = F.inc_i[idx] + 0.0;
      }
      continue;
    }
    const size_t oh = (size_t)(ib * (kl + 1) + jk) * np + jl;  // PAPH(jl, jk)
    const size_t o4 = (size_t)(ib * 4 * kl + jk) * np + jl;     // PLUDELI(jl, jk, 1)
    const size_t sl = (size_t)kl * np;                          // one PLUDELI component
    double lt, lq, la, ll, li;
    // the cumulative tendencies are read through the read-only path only
    // when this kernel does not write them back
    const double ct = INC ? F.cml_t[idx] : ld(F.cml_t + idx), cq = INC ? F.cml_q[idx] : ld(F.cml_q + idx),
                 ca = INC ? F.cml_a[idx] : ld(F.cml_a + idx), cl = INC ? F.cml_l[idx] : ld(F.cml_l + idx),
                 ci = INC ? F.cml_i[idx] : ld(F.cml_i + idx);
    satadj_point(k, dt, zqtmst, ld(F.pap + idx), ld(F.paph + oh), ld(F.paph + oh + np),
                 ld(F.paph + (size_t)(ib * (kl + 1) + kl) * np + jl), ld(F.pt + idx), ld(F.pq + idx),
                 ld(F.pa + idx), ld(F.pl + idx), ld(F.pi + idx), ct, cq, ca, cl, ci, ld(F.phrsw + idx),
                 ld(F.phrlw + idx), ld(F.vdf_t + idx), ld(F.vdf_q + idx), ld(F.pludeli + o4 + 2 * sl),
                 ld(F.pludeli + o4 + 3 * sl), ld(F.pvervel + idx), lt, lq, la, ll, li, nwarn);
    F.loc_t[idx] = lt;
    F.loc_q[idx] = lq;
    F.loc_a[idx] = la;
    F.loc_l[idx] = ll;
    F.loc_i[idx] = li;
    if constexpr (INC) {
      if (F.inc_t) F.inc_t[idx] = ct + lt;
      if (F.inc_q) F.inc_q[idx] = cq + lq;
      if (F.inc_a) F.inc_a[idx] = ca + la;
      if (F.inc_l) F.inc_l[idx] = cl + ll;
      if (F.inc_i) F.inc_i[idx] = ci + li;
    }
  }
  if (nwarn && F.ncounters) atomic_add(F.ncounters, (uint32_t)nwarn);
}

// SLTEND's supersaturation adjustment (sltend.F90:380-410): one thread per
// (column, level) point on levels NCLDTOP..KLEV, numbered like satadj_kernel;
// the tendencies are updated in place and the diagnostics written where
// their pointers are not NULL.
__global__ void __launch_bounds__(kSatadjThreads, 4) sltend_supersat_kernel(SltendFields F, Shape sh) {
  plibm_load_tables();
  const KParams<double> &k = KP<double>();
  const double tsphy = sh.ptsphy;
  const double zrtsphy = 1.0 / tsphy;
  const unsigned long long np = sh.nproma, kl = sh.klev;
  const unsigned long long npts = (unsigned long long)sh.ngpblks * kl * np;
  const int jktop = k.ncldtop - 1;
  for (unsigned long long idx = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; idx < npts;
       idx += (unsigned long long)gridDim.x * blockDim.x) {
    const unsigned long long row = idx / np;
    const int jl = (int)(idx - row * np);
    const unsigned long long ib = row / kl;
    const int jk = (int)(row - ib * kl);
    const long long icend = (long long)sh.ngptot - (long long)ib * (long long)np;
    if (jl < sh.kidia0 || jl >= icend || jk < jktop) continue;
    const size_t oc = (size_t)(ib * 5 * kl + jk) * np + jl;  // PTENCLD(jl, jk, NCLDQL)
    const size_t sl = (size_t)kl * np;
    const double tent = F.ptent[idx], tenq = F.ptenq[idx], tena = F.ptena[idx];
    const double zt = ld(F.pt + idx) + tsphy * (ld(F.pcent + idx) + tent);
    const double zq = ld(F.pq + idx) + tsphy * (ld(F.pcenq + idx) + tenq);
    const double za = ld(F.pa + idx) + tsphy * (ld(F.pcena + idx) + tena);
    double ta, qa, aa, la, ia;
    supersatcheck_kft1(k, zt, zq, za, ld(F.prsf1 + idx), ta, qa, aa, la, ia);
    F.ptent[idx] = tent + ta * zrtsphy;
    F.ptenq[idx] = tenq + qa * zrtsphy;
    F.ptena[idx] = tena + aa * zrtsphy;
    F.ptencld[oc] = F.ptencld[oc] + la * zrtsphy;
    F.ptencld[oc + sl] = F.ptencld[oc + sl] + ia * zrtsphy;
    if (F.padja) F.padja[idx] = aa * zrtsphy;
    if (F.padjl) F.padjl[idx] = la * zrtsphy;
    if (F.padji) F.padji[idx] = ia * zrtsphy;
  }
}

// STATE_INCREMENT (state_increment.F90:42-103): one thread per (column,
// level) point, numbered like satadj_kernel, adds each of the n increments
// to its state field (coalesced: a warp covers 32 neighbouring columns of
// one level of every field).
__global__ void __launch_bounds__(kSatadjThreads) state_increment_kernel(IncFields F, Shape sh) {
  const unsigned long long np = sh.nproma, kl = sh.klev;
  const unsigned long long npts = (unsigned long long)sh.ngpblks * kl * np;
  for (unsigned long long idx = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; idx < npts;
       idx += (unsigned long long)gridDim.x * blockDim.x) {
    const unsigned long long row = idx / np;
    const int jl = (int)(idx - row * np);
    const unsigned long long ib = row / kl;
    const unsigned long long within = idx - ib * kl * np;  // jk * NPROMA + jl
    const long long icend = (long long)sh.ngptot - (long long)ib * (long long)np;
    if (jl < sh.kidia0 || jl >= icend) continue;
    for (int f = 0; f < F.n; ++f) {
      double *d = F.dst[f] + ib * F.dst_bs[f] + within;
      *d = *d + ld(F.src[f] + ib * F.src_bs[f] + within);
    }
  }
}

// The column kernels' fast division on n operand pairs: q[i] = fast_div(a[i],
// b[i]) and bad[i] = 1 where an operand fell outside its exact window (a
// column kernel then reruns the column with IEEE division).  A self-check of
// the division alone.
__global__ void __launch_bounds__(kSatadjThreads) division_check_kernel(const double *a, const double *b,
                                                                       long long n, double *q, int *bad) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    DivCheck dc;
    q[i] = fast_div(a[i], b[i], dc);
    bad[i] = dc.bad() ? 1 : 0;
  }
}

// fast_rcp on n divisors: y[i] and the window report bad[i].
__global__ void __launch_bounds__(kSatadjThreads) reciprocal_check_kernel(const double *b, long long n, double *y,
                                                                         int *bad) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    DivCheck dc;
    y[i] = fast_rcp(b[i], dc);
    bad[i] = dc.bad() ? 1 : 0;
  }
}

// csqrt of the fast pass on n values, and its report.
__global__ void __launch_bounds__(kSatadjThreads) sqrt_check_kernel(const double *x, long long n, double *y, int *bad) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    DivCheck dc;
    y[i] = csqrt<true>(x[i], dc);
    bad[i] = dc.bad() ? 1 : 0;
  }
}

}  // namespace cloudsc

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
namespace cloudsc {

// Whether the parameters allow the GEN kernels (gen_exponents_ok).
bool params_allow_gen(const cloudsc_params &p, const Derived &d) {
  KParams<double> kd;
  fill_kparams(p, d, kd);
  return gen_exponents_ok(kd);
}

// Upload the parameters to this device's constant memory (all three blocks).
cudaError_t upload_params(const cloudsc_params &p, const Derived &d) {
  KParams<double> kd;
  KParams<float> kf;
  fill_kparams(p, d, kd);
  fill_kparams(p, d, kf);
  KParamsD dd;
  fill_kparams_d(p, dd);
  cudaError_t e = cudaMemcpyToSymbol(c_kpd, &kd, sizeof(kd));
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(c_kpf, &kf, sizeof(kf));
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(c_kd, &dd, sizeof(dd));
  return e;
}

// Compiled launch variants: the __launch_bounds__(MAXT, MINB) pairs the
// kernels are built with.  MAXT x MINB threads share an SM's 65,536
// registers, so each pair fixes the register budget per thread (and with it
// the spills) and the CTA size it is meant for; the autotuner picks a
// variant, a CTA size up to its MAXT and the persistence at run time.
// 448 columns per CTA fill 148 SMs 3.96 times at 262,144 columns; the
// (448, 1) bound gives them 144 registers (0.8 % faster than the 128 of a
// (512, 1) bound, same bits).  Earlier measurements at 262,144 columns, FP64:
// 384 columns per CTA at 168 registers 17.77 ms against 15.98 ms at 448;
// three 128-thread CTAs per SM 21.7 ms.
struct Variant {
  int maxt, minb;
};
constexpr Variant kVariants[] = {{640, 1}, {448, 1}, {384, 1}, {256, 1}, {256, 2}, {128, 3}};
constexpr int kNumVariants = sizeof(kVariants) / sizeof(kVariants[0]);
constexpr int kDefaultVariant = 1;  // (448, 1), run with 448 columns per CTA

int num_variants() { return kNumVariants; }
int default_variant() { return kDefaultVariant; }
void variant_bounds(int v, int *maxt, int *minb) {
  *maxt = kVariants[v].maxt;
  *minb = kVariants[v].minb;
}

// A compiled column kernel: its function, the largest CTA it takes and the
// dynamic shared memory of its parking slots.
struct ColumnKernel {
  const void *f;
  int maxt;
  size_t smem;
};
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
static ColumnKernel find_kernel(int precision, int v, bool gen, bool fast) {
  if (precision <= 2 && (!gen || !fast)) {
    switch (precision) {
      case 0: return kernel_general<0, Fields>(fast);
      case 1: return kernel_general<1, Fields>(fast);
      default: return kernel_general<2, Fields>(fast);
    }
  }
  switch (precision) {
    case 0: return kernel_form<0>(v);
    case 1: return kernel_form<1>(v);
    case 2: return kernel_form<2>(v);
    case 3: return kernel_opt_form<3>(v, gen, fast);
    case 4: return kernel_opt_form<4>(v, gen, fast);
    case 5: return kernel_opt_form<5>(v, gen, fast);
    default: return {nullptr, 0, 0};
  }
}
static ColumnKernel find_kernel_sp(int precision, int v, bool gen, bool fast) {
  switch (precision) {
    case 0: return kernel_sp_form<0>(v, gen, fast);
    case 1: return kernel_sp_form<1>(v, gen, fast);
    case 2: return kernel_sp_form<2>(v, gen, fast);
    default: return {nullptr, 0, 0};
  }
}

// The largest CTA of the kernel a call runs with variant v.
int kernel_max_threads(int precision, int v, bool gen, int klev, bool sp) {
  const bool fast = klev <= kMaxLevFast;
  return (sp ? find_kernel_sp(precision, v, gen, fast) : find_kernel(precision, v, gen, fast)).maxt;
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

// Launch CLOUD_SATADJ over every point of the batched arrays: a grid of
// 256-thread CTAs, at most 64 per SM, striding over the points.
// With any inc_* pointer set, the form with the fused STATE_INCREMENT runs.
cudaError_t launch_satadj(const SatadjFields &f, const Shape &sh, cudaStream_t stream) {
  const unsigned long long npts = (unsigned long long)sh.ngpblks * sh.klev * sh.nproma;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  unsigned long long blocks = (npts + kSatadjThreads - 1) / kSatadjThreads;
  const unsigned long long cap = (unsigned long long)sms * 64;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  if (f.inc_t || f.inc_q || f.inc_a || f.inc_l || f.inc_i)
    satadj_kernel<true><<<(unsigned)blocks, kSatadjThreads, 0, stream>>>(f, sh);
  else
    satadj_kernel<false><<<(unsigned)blocks, kSatadjThreads, 0, stream>>>(f, sh);
  return cudaGetLastError();
}

// STATE_INCREMENT over every point: a grid of 256-thread CTAs, at most 16
// per SM, striding over the points.
cudaError_t launch_state_increment(const IncFields &f, const Shape &sh, cudaStream_t stream) {
  const unsigned long long npts = (unsigned long long)sh.ngpblks * sh.klev * sh.nproma;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  unsigned long long blocks = (npts + kSatadjThreads - 1) / kSatadjThreads;
  const unsigned long long cap = (unsigned long long)sms * 16;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  state_increment_kernel<<<(unsigned)blocks, kSatadjThreads, 0, stream>>>(f, sh);
  return cudaGetLastError();
}

cudaError_t launch_sltend_supersat(const SltendFields &f, const Shape &sh, cudaStream_t stream) {
  const unsigned long long npts = (unsigned long long)sh.ngpblks * sh.klev * sh.nproma;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  unsigned long long blocks = (npts + kSatadjThreads - 1) / kSatadjThreads;
  const unsigned long long cap = (unsigned long long)sms * 64;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  sltend_supersat_kernel<<<(unsigned)blocks, kSatadjThreads, 0, stream>>>(f, sh);
  return cudaGetLastError();
}

cudaError_t launch_division_check(const double *a, const double *b, long long n, double *q, int *bad,
                                  cudaStream_t stream) {
  long long blocks = (n + kSatadjThreads - 1) / kSatadjThreads;
  if (blocks > 148LL * 16) blocks = 148LL * 16;
  if (blocks < 1) blocks = 1;
  division_check_kernel<<<(unsigned)blocks, kSatadjThreads, 0, stream>>>(a, b, n, q, bad);
  return cudaGetLastError();
}

cudaError_t launch_reciprocal_check(const double *b, long long n, double *y, int *bad, cudaStream_t stream) {
  long long blocks = (n + kSatadjThreads - 1) / kSatadjThreads;
  if (blocks > 148LL * 16) blocks = 148LL * 16;
  if (blocks < 1) blocks = 1;
  reciprocal_check_kernel<<<(unsigned)blocks, kSatadjThreads, 0, stream>>>(b, n, y, bad);
  return cudaGetLastError();
}

cudaError_t launch_sqrt_check(const double *x, long long n, double *y, int *bad, cudaStream_t stream) {
  long long blocks = (n + kSatadjThreads - 1) / kSatadjThreads;
  if (blocks > 148LL * 16) blocks = 148LL * 16;
  if (blocks < 1) blocks = 1;
  sqrt_check_kernel<<<(unsigned)blocks, kSatadjThreads, 0, stream>>>(x, n, y, bad);
  return cudaGetLastError();
}

}  // namespace cloudsc
