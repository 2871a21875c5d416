// The pointwise kernels around CLOUDSC: CLOUD_SATADJ, SLTEND's supersaturation
// adjustment, STATE_INCREMENT, and the self-checks of the column kernels'
// division and roots.
#include "cloudsc_kernels.cuh"
#include "satadj_point.cuh"

namespace cloudsc {

cudaError_t upload_points(const KParams<double> &kd, const KParams<float> &kf, const KParamsD &dd) {
  return upload_unit(kd, kf, dd);
}

// CLOUD_SATADJ: one thread per (column, level) point, points numbered
// (ib * KLEV + jk) * NPROMA + jl -- the element offset of a level field -- so
// consecutive threads read consecutive columns of one level (coalesced).  A
// grid-stride loop covers all points of all blocks; levels above NCLDTOP get
// zero tendencies (cloud_satadj.F90:338-345).  Bound by the latency of its
// FP64 chains (four saturation evaluations one after the other): about 1,600
// instructions a point, 44 % of them FP64; FP64 pipe 58 %, issue 66 %.
// 128-thread CTAs at 96 registers (5 CTAs, 20 warps per SM), 100,000 columns of
// 137 levels: 869-897 us; 913-915 with IEEE division, the full exponential and
// two 64-bit index divisions a point (256 threads, 64 registers; 1,900
// instructions).  128 registers 3 % and 80 or fewer 4-14 % slower; prefetching
// the next point's lines to L2, or copying its inputs to shared memory ahead of
// time, no faster.
// INC: STATE_INCREMENT of the cumulative tendencies fused in
// (callpar.F90:1278-1280): each point writes CML + LOC back into the CML
// arrays it has just read (inc_* not NULL), one addition each, as the
// separate call does.
constexpr int kSatadjThreads = 256;
// Division of a point index by NPROMA and KLEV through 64-bit reciprocals
// ceil(2^64 / d): the high word of x * ceil(2^64 / d) is x / d for every x, d
// below 2^32 (the excess x (d ceil(2^64 / d) - 2^64) / 2^64 stays below 1).
// d = 1, and more than 2^32 points, divide as they are.
struct PointDiv {
  unsigned long long rnp, rkl;  // 0: divide
};
__device__ __forceinline__ unsigned long long point_div(unsigned long long x, unsigned long long d,
                                                        unsigned long long r) {
  return r ? __umul64hi(x, r) : x / d;
}
// A point the first pass reported, with IEEE division (rare: out of line, so
// that it costs the first pass no registers).
__device__ __noinline__ void satadj_again(SatadjFields F, double dt, double zqtmst, size_t idx, size_t oh,
                                          size_t osurf, size_t o4, size_t sl, size_t np, double ct, double cq,
                                          double ca, double cl, double ci, double &lt, double &lq, double &la,
                                          double &ll, double &li, int &nwarn) {
  nwarn = 0;
  satadj_point(KP<double>(), dt, zqtmst, ld(F.pap + idx), ld(F.paph + oh), ld(F.paph + oh + np), ld(F.paph + osurf),
               ld(F.pt + idx), ld(F.pq + idx), ld(F.pa + idx), ld(F.pl + idx), ld(F.pi + idx), ct, cq, ca, cl, ci,
               ld(F.phrsw + idx), ld(F.phrlw + idx), ld(F.vdf_t + idx), ld(F.vdf_q + idx), ld(F.pludeli + o4 + 2 * sl),
               ld(F.pludeli + o4 + 3 * sl), ld(F.pvervel + idx), lt, lq, la, ll, li, nwarn);
}
constexpr int kSatThreads = 128;
template <bool INC>
__global__ void __launch_bounds__(kSatThreads, 5) satadj_kernel(SatadjFields F, Shape sh, PointDiv pd) {
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
    const unsigned long long row = point_div(idx, np, pd.rnp);
    const int jl = (int)(idx - row * np);
    const unsigned long long ib = point_div(row, kl, pd.rkl);
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
    DivCheck dc;
    int warned = 0;
    satadj_pass<true>(k, dt, zqtmst, ld(F.pap + idx), ld(F.paph + oh), ld(F.paph + oh + np),
                      ld(F.paph + (size_t)(ib * (kl + 1) + kl) * np + jl), ld(F.pt + idx), ld(F.pq + idx),
                      ld(F.pa + idx), ld(F.pl + idx), ld(F.pi + idx), ct, cq, ca, cl, ci, ld(F.phrsw + idx),
                      ld(F.phrlw + idx), ld(F.vdf_t + idx), ld(F.vdf_q + idx), ld(F.pludeli + o4 + 2 * sl),
                      ld(F.pludeli + o4 + 3 * sl), ld(F.pvervel + idx), lt, lq, la, ll, li, warned, dc);
    if (dc.bad()) satadj_again(F, dt, zqtmst, idx, oh, (size_t)(ib * (kl + 1) + kl) * np + jl, o4, sl, np, ct, cq, ca, cl, ci, lt, lq, la, ll, li, warned);
    nwarn += warned;
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

// The column kernels' divisions on n operand pairs, as they are instantiated
// there with checked operands: both orders of cdiv, and cdivk on crcp's
// reciprocal.  The three must agree (a pair for which they do not is reported
// like one outside the window).  A divisor with an all-ones significand, which
// makes a kernel run the column again with IEEE division, gets that division
// here; a zero quotient IEEE's sign, which the kernels' sequences do not keep
// for -0 / b and no result depends on.
__global__ void __launch_bounds__(kSatadjThreads) division_check_kernel(const double *a, const double *b,
                                                                       long long n, double *q, int *bad) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const double x = a[i], d = b[i];
    DivCheck dc;
    double r = cdiv<true, true, true>(x, d, dc);
    const double r1 = cdiv<true, true, false>(x, d, dc), r2 = cdivk<true, true>(x, d, crcp<true, true>(d, dc), dc);
    const bool outside = dc.acc >= kDivRange, ones = dc.ones == ~0u;
    const bool differ = __double_as_longlong(r) != __double_as_longlong(r1) ||
                        __double_as_longlong(r) != __double_as_longlong(r2);
    if (ones) r = x / d;
    if (x == 0.0) r = copysign(r, copysign(1.0, x) * copysign(1.0, d));
    q[i] = r;
    bad[i] = outside || (!ones && differ) ? 1 : 0;
  }
}

// crcp on n divisors: y[i] and the window report bad[i]; IEEE 1 / b for an
// all-ones significand, as above.
__global__ void __launch_bounds__(kSatadjThreads) reciprocal_check_kernel(const double *b, long long n, double *y,
                                                                         int *bad) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    DivCheck dc;
    const double r = crcp<true, true>(b[i], dc);
    y[i] = dc.ones == ~0u ? 1.0 / b[i] : r;
    bad[i] = dc.acc >= kDivRange ? 1 : 0;
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

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
static PointDiv make_point_div(const Shape &sh) {
  const unsigned long long npts = (unsigned long long)sh.ngpblks * sh.klev * sh.nproma;
  auto r = [&](unsigned long long d) { return npts >> 32 || d < 2 ? 0ull : ~0ull / d + 1ull; };
  return {r(sh.nproma), r(sh.klev)};
}

// Launch CLOUD_SATADJ over every point of the batched arrays: a grid of
// 128-thread CTAs, at most 128 per SM, striding over the points.
// With any inc_* pointer set, the form with the fused STATE_INCREMENT runs.
cudaError_t launch_satadj(const SatadjFields &f, const Shape &sh, cudaStream_t stream) {
  const unsigned long long npts = (unsigned long long)sh.ngpblks * sh.klev * sh.nproma;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  unsigned long long blocks = (npts + kSatThreads - 1) / kSatThreads;
  const unsigned long long cap = (unsigned long long)sms * 128;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  if (f.inc_t || f.inc_q || f.inc_a || f.inc_l || f.inc_i)
    satadj_kernel<true><<<(unsigned)blocks, kSatThreads, 0, stream>>>(f, sh, make_point_div(sh));
  else
    satadj_kernel<false><<<(unsigned)blocks, kSatThreads, 0, stream>>>(f, sh, make_point_div(sh));
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
