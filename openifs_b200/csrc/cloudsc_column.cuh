// One CLOUDSC column, top to bottom, on one GPU thread.
//
// This is the per-column body shared by the FP64 kernel (Real = double) and
// the FP32-mixed kernel (Real = float).  It restates, for a single column, the
// whole of ifs-source/arpifs/phys_ec/cloudsc.F90 in its default configuration:
//   first guess and tidy-up          :982-1199
//   level loop JK=NCLDTOP..KLEV       :1219-4128
//   DDH flux recurrences              :4218-4303
//   CLOUD_SUPERSATCHECK               cloud_supersatcheck.F90:111-226
// fused into ONE pass over the levels: every pre-loop quantity is computed for
// level JK when the pass reaches it, the quantities the reference reads from
// level JK-1 (ZA, ZQX(R/S), ZTP1, PAP) or JK+1 (PAPH, PLU, PMFU, PMFD) are
// carried in registers, and the flux prefix sums are accumulated as the pass
// goes, so every input element is read once and every output element written
// once.
//
// FP64 parity: with Real = double every floating-point operation is the
// reference's, in the reference's order (the file is compiled with
// --fmad=false so nothing is contracted).  The explicit (ZSOLQA) and implicit
// (ZSOLQB) 5x5 process matrices are held in registers using their structural
// sparsity in this configuration -- ZSOLQA has 18 entries that any process can
// touch, ZSOLQB has 5: (L,L), (I,I), (R,L), (S,I), (S,L).  The skipped entries
// are exact zeros, and every skipped operation on them (x - 0, x + 0,
// x - 0*y with finite y) returns x unchanged, so the sparse forms below give
// the dense reference results bit for bit (up to the sign of a zero).  The
// LHS matrix is lower triangular (its only off-diagonal entries are
// -ZSOLQB(R,L), -ZSOLQB(S,I), -ZSOLQB(S,L)), so the reference's non-pivoting
// LU (:3600-3628) reduces to three multipliers and forward/back substitution
// performed in the same order.
//
// Saturation exponentials: FOEEWM, FOEELIQ, FOEEICE and FOEEW share the two
// exponentials exp(R3LES*(T-RTT)/(T-R4LES)) and exp(R3IES*(T-RTT)/(T-R4IES));
// a term whose weight is exactly zero (FOEALFA = 1, FOEDELTA = 0/1) is
// skipped, which again leaves the result bit-identical.
//
// FP32-mixed (template flag F32M): the exponentials and powers of the
// microphysical processes and of the level's saturation values are evaluated
// in FP32; the state, every other operation, the sink truncation, the 5x5
// solve, CLOUD_SUPERSATCHECK (with its FP64 exponentials) and the tendency and
// flux (budget) accumulations stay in FP64.  Keeping the state and the
// threshold tests in FP64 is what keeps the tendencies within 1e-5 of the FP64
// result: with an FP32 state the scheme's thresholds and MIN() limiters flip
// (a measured 5-7 % RMS error on the T tendency).
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>
#include <type_traits>

#include "cloudsc_common.cuh"
#include "plibm.h"

#ifndef CSC_DEV
#define CSC_DEV __device__ __forceinline__
#endif

namespace cloudsc {

template <typename T>
CSC_DEV T mn(T a, T b) { return a < b ? a : b; }
template <typename T>
CSC_DEV T mx(T a, T b) { return a > b ? a : b; }

// What the fast pass reports about a column.  A column whose operands all stay
// inside the windows below has every fast division, exp, log and pow equal to
// the IEEE / plibm ones bit for bit; any other column is run again with those.
//   acc   ORs, for each checked value that may be zero, the offset
//         2 * hi(x) - kDivBase, whose top two bits are clear exactly when
//         2^-256 <= |x| < 2^256 (a zero adds 0);
//   pos   ORs, for each checked positive value, hi(x) - hi(lowest allowed),
//         below kPosRange exactly for x in [lowest, 2^32 * lowest);
//   ones  the largest (hi(b) | 0xfff00000) & lo(b) of any divisor b: all bits
//         set for a divisor whose significand is all ones (fast_rcp_y).
constexpr unsigned kDivBase = 767u << 21, kDivRange = 1u << 30;
constexpr unsigned kPosRange = 32u << 20;
struct DivCheck {
  unsigned acc = 0u, pos = 0u, ones = 0u;
  CSC_DEV bool bad() const { return acc >= kDivRange || pos >= kPosRange || ones == ~0u; }
};

#if defined(__CUDA_ARCH__)
CSC_DEV unsigned hi_word(double x) { return (unsigned)__double2hiint(x); }
CSC_DEV unsigned lo_word(double x) { return (unsigned)__double2loint(x); }
CSC_DEV double from_words(unsigned hi, unsigned lo) { return __hiloint2double((int)hi, (int)lo); }
#else
inline unsigned hi_word(double x) {
  uint64_t u;
  std::memcpy(&u, &x, sizeof u);
  return (unsigned)(u >> 32);
}
inline unsigned lo_word(double x) {
  uint64_t u;
  std::memcpy(&u, &x, sizeof u);
  return (unsigned)u;
}
inline double from_words(unsigned hi, unsigned lo) {
  const uint64_t u = (uint64_t)hi << 32 | lo;
  double x;
  std::memcpy(&x, &u, sizeof x);
  return x;
}
#endif

// The branch-free sequences below run on the GPU, and in host builds that ask
// for them (CLOUDSC_HOST_SEQUENCES); other host builds divide and take roots
// with IEEE operations.  Their estimates are rcp.approx.ftz.f64 and
// rsqrt.approx.ftz.f64 on the GPU; on the host the values 1/x and 1/sqrt(x)
// cut to 20 fraction bits, subnormals read and returned as zero.
#if defined(__CUDA_ARCH__)
#define CSC_SEQUENCES 1
CSC_DEV double rcp_estimate(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
}
CSC_DEV double rsqrt_estimate(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
}
CSC_DEV double fmad(double a, double b, double c) { return __fma_rn(a, b, c); }
CSC_DEV double muld(double a, double b) { return __dmul_rn(a, b); }
#elif defined(CLOUDSC_HOST_SEQUENCES)
#define CSC_SEQUENCES 1
inline double no_subnormal(double x) { return std::fabs(x) < 0x1p-1022 ? std::copysign(0.0, x) : x; }
inline double estimate_of(double y) {
  return no_subnormal(std::isfinite(y) ? from_words(hi_word(y), 0u) : y);
}
inline double rcp_estimate(double x) { return estimate_of(1.0 / no_subnormal(x)); }
inline double rsqrt_estimate(double x) { return estimate_of(1.0 / std::sqrt(no_subnormal(x))); }
inline double fmad(double a, double b, double c) { return std::fma(a, b, c); }
inline double muld(double a, double b) { return a * b; }
#else
#define CSC_SEQUENCES 0
#endif
// Record a value that must be zero or inside 2^-256 <= |x| < 2^256.
CSC_DEV void see(double x, DivCheck &dc) { dc.acc |= x == 0.0 ? 0u : hi_word(x) * 2u - kDivBase; }
// Record a value that must lie in [2^e, 2^(e+32)).
CSC_DEV void see_pos(double x, int e, DivCheck &dc) { dc.pos |= hi_word(x) - ((unsigned)(1023 + e) << 20); }

// Branch-free double division, in two halves.
//
// The reciprocal: an estimate (rcp.approx.ftz.f64) is refined by three
// Newton-Raphson steps y <- y + y(1 - by), each error term and update one
// fused multiply-add; the last step returns y = RN(1/b), the correctly
// rounded reciprocal, for every divisor whose significand is not all ones
// (Markstein, IBM J. Res. Dev. 34(1), 1990; Muller et al., Handbook of
// Floating-Point Arithmetic, ch. 5).  For b = (2 - 2^-52) 2^E the step ends on
// the tie 2^(-E-1) while 1/b = 2^(-E-1) (1 + 2^-53 + 2^-106 + ...).
CSC_DEV double fast_rcp_y(double b) {
#if CSC_SEQUENCES
  double y = rcp_estimate(b);
  double e = fmad(-b, y, 1.0);
  y = fmad(y, e, y);
  e = fmad(-b, y, 1.0);
  y = fmad(y, e, y);
  e = fmad(-b, y, 1.0);
  return fmad(y, e, y);
#else
  return 1.0 / b;
#endif
}
// The quotient from y = RN(1/b): q0 = RN(a y), within 1.5 ulp of a/b, is
// corrected twice with its residual, q <- RN(q + RN(a - b q) y): the first
// correction brings it within one ulp, where the residual is exact, and by
// Markstein's theorem the second then returns RN(a/b).  Equal to IEEE a/b
// (up to the sign of a zero) when no step under- or overflows, for instance
// for 2^-256 <= |b| < 2^256 and a = 0 or 2^-256 <= |a| < 2^256.
CSC_DEV double fast_quot(double a, double b, double y) {
#if CSC_SEQUENCES
  const double q0 = muld(a, y);
  double r = fmad(-b, q0, a);
  const double q1 = fmad(r, y, q0);
  r = fmad(-b, q1, a);
  return fmad(r, y, q1);
#else
  (void)y;
  return a / b;
#endif
}
// Both halves for one quotient, the first quotient taken from the estimate
// before the last Newton step (already within an ulp of 1/b), so that q0 and
// its residual are formed beside that step: two operations less on the chain
// of a division, the same operations otherwise.  q0 lies within two ulp of
// a/b, its residual is then off by at most one rounding, the first correction
// (with RN(1/b)) still ends within one ulp, and the second is Markstein's.
// Measured with it and without in one session (ms): FP64 3,200 columns 1.203 /
// 1.225, FP32-mixed 90,005 2.700 / 2.757, SPP 24,576 2.267 / 2.286, satadj
// 100,000 0.857 / 0.881 (0.87-0.90 elsewhere); FP64 at 128 and 168 registers no gain (262,144 columns 9.494 / 9.472),
// so the level code there keeps the other order (SHORT).
CSC_DEV double fast_quot_rcp(double a, double b) {
#if CSC_SEQUENCES
  double y = rcp_estimate(b);
  double e = fmad(-b, y, 1.0);
  y = fmad(y, e, y);
  e = fmad(-b, y, 1.0);
  y = fmad(y, e, y);
  const double q0 = muld(a, y);
  e = fmad(-b, y, 1.0);
  double r = fmad(-b, q0, a);
  y = fmad(y, e, y);
  const double q1 = fmad(r, y, q0);
  r = fmad(-b, q1, a);
  return fmad(r, y, q1);
#else
  return a / b;
#endif
}
// All ones exactly for a divisor with an all-ones significand.
CSC_DEV unsigned ones_word(double b) { return (hi_word(b) | 0xfff00000u) & lo_word(b); }

// Branch-free correctly rounded square root for 2^-200 <= x < 2^200: the
// estimate rsqrt.approx.ftz.f64 refined by two Goldschmidt steps on
// g ~ sqrt(x), h ~ 1/(2 sqrt(x)) and one residual correction (Markstein 1990;
// Handbook of Floating-Point Arithmetic, ch. 5).  That g is RN(sqrt(x)) is
// then checked, not assumed: with u = ulp(g), sqrt(x) lies within u/2 of g
// exactly when the residual x - g^2, exact in one fused multiply-add, is below
// g u in magnitude (g u is a multiple of the residual's unit, so there is no
// tie).  The one exception, x just below a power of 4 with g a power of two
// (whose lower neighbour is only u/2 away), has an all-ones significand.
// Both are reported to the rerun.
template <bool FAST>
CSC_DEV double csqrt(double x, DivCheck &dc) {
#if CSC_SEQUENCES
  if constexpr (FAST) {
    const double y = rsqrt_estimate(x);
    double g = muld(x, y), h = muld(0.5, y);
    double r = fmad(-g, h, 0.5);
    g = fmad(g, r, g);
    h = fmad(h, r, h);
    r = fmad(-g, h, 0.5);
    g = fmad(g, r, g);
    h = fmad(h, r, h);
    g = fmad(fmad(-g, g, x), h, g);
    const double d = fmad(-g, g, x);
    const double gu = muld(g, from_words((hi_word(g) & 0x7ff00000u) - (52u << 20), 0u));
    dc.pos |= fabs(d) < gu ? 0u : kPosRange;
    const unsigned o = ones_word(x);
    dc.ones = dc.ones > o ? dc.ones : o;
    return g;
  }
#endif
  (void)dc;
  return sqrt(x);
}

#if defined(CLOUDSC_HOST_WINDOW_CHECK) && !defined(__CUDA_ARCH__)
// Test builds: count the operands of the fast pass outside the range its
// operations are exact in, in columns that have not been reported.
inline unsigned long long g_window_violations = 0;
inline const DivCheck *g_column = nullptr;  // the checks of the column being run
inline bool host_in(double x, int e) { return std::fabs(x) >= std::ldexp(1.0, -e) && std::fabs(x) < std::ldexp(1.0, e); }
inline void host_count(bool ok) { g_window_violations += !ok && !(g_column && g_column->bad()); }
inline void host_check_div(double a, double b) { host_count((a == 0.0 || host_in(a, 800)) && host_in(b, 400)); }
inline void host_check_exp(double x) { host_count(std::fabs(x) < 700.0); }
inline void host_check_log(double x) { host_count(x > 0.0 && host_in(x, 256)); }
#else
#define host_check_div(A, B)
#define host_check_exp(X)
#define host_check_log(X)
#endif

// Divisions of the column code.  In the fast pass (FAST) a double division is
// fast_quot over fast_rcp_y; its operands need no check of their own, because
// the level's input checks (cloudsc_body.cuh) bound them, except with CHK
// (forms whose extra inputs are not among those), which records them.  A
// divisor's all-ones significand is always recorded.  Otherwise IEEE.
template <bool FAST, bool CHK, bool SHORT = true, typename A, typename B>
CSC_DEV auto cdiv(A a, B b, DivCheck &dc) -> decltype(a / b) {
  typedef decltype(a / b) T;
  if constexpr (FAST && std::is_same<T, double>::value) {
    const double ad = double(a), bd = double(b);
    if constexpr (CHK) {
      see(ad, dc);
      dc.acc |= hi_word(bd) * 2u - kDivBase;
    }
    const unsigned o = ones_word(bd);
    dc.ones = dc.ones > o ? dc.ones : o;
    host_check_div(ad, bd);
    return SHORT ? fast_quot_rcp(ad, bd) : fast_quot(ad, bd, fast_rcp_y(bd));
  } else {
    (void)dc;
    return a / b;
  }
}
// a / b given y = RN(1/b): a literal or parameter divisor (inside the window
// and without an all-ones significand, so its folded or host-computed
// reciprocal is exact), or one whose reciprocal several quotients share.
template <bool FAST, bool CHK, typename A>
CSC_DEV auto cdivk(A a, double b, double y, DivCheck &dc) -> decltype(a / A(b)) {
  typedef decltype(a / A(b)) T;
  if constexpr (FAST && std::is_same<T, double>::value) {
    if constexpr (CHK) see(double(a), dc);
    host_check_div(double(a), b);
    return fast_quot(double(a), b, y);
  } else {
    (void)dc;
    (void)y;
    return a / A(b);
  }
}
// 1 / b.
template <bool FAST, bool CHK, typename B>
CSC_DEV B crcp(B b, DivCheck &dc) {
  if constexpr (FAST && std::is_same<B, double>::value) {
    if constexpr (CHK) dc.acc |= hi_word(b) * 2u - kDivBase;
    const unsigned o = ones_word(b);
    dc.ones = dc.ones > o ? dc.ones : o;
    host_check_div(1.0, b);
    return fast_rcp_y(b);
  } else {
    (void)dc;
    return B(1) / b;
  }
}

// Passes of the column code (cloudsc_column's PASS): plain, IEEE division and
// plibm's full functions throughout; fast, the branch-free forms, with checks
// that report what could leave their exact windows; redo, the plain code again
// for a column whose fast pass reported.
enum { kPassPlain = 0, kPassFast = 1, kPassRedo = 2 };

// Double precision uses the portable exp/pow of plibm.h (bit-identical on the
// host and the GPU).
#if defined(CLOUDSC_HOST_LIBM_GLIBC) && !defined(__CUDA_ARCH__)
// host test builds only: the system libm, to measure libm sensitivity
CSC_DEV double xexp(double x) { return exp(x); }
CSC_DEV double xpow(double x, double y) { return pow(x, y); }
CSC_DEV double xlog(double x) { return log(x); }
#else
CSC_DEV double xexp(double x) { return plibm_exp(x); }
CSC_DEV double xpow(double x, double y) { return plibm_pow(x, y); }
CSC_DEV double xlog(double x) { return plibm_log(x); }
#endif
// FP32 transcendentals of the FP32-mixed kernel: on the GPU the special-
// function-unit forms (__expf, __powf: one ex2 / lg2 each, relative error of a
// few 1e-7 times the size of the exponent's argument), on the host the C
// library; exponents 0.5, 1.5, 2 and 3 are evaluated exactly as roots and
// products, as plibm does in double.
CSC_DEV float xexp(float x) {
#if defined(__CUDA_ARCH__)
  return __expf(x);
#else
  return expf(x);
#endif
}
CSC_DEV float xpow(float x, float y) {
  if (y == 0.5f) return sqrtf(x);
  if (y == 1.5f) return x * sqrtf(x);
  if (y == 2.0f) return x * x;
  if (y == 3.0f) return x * x * x;
#if defined(__CUDA_ARCH__)
  return __powf(x, y);
#else
  return powf(x, y);
#endif
}

// Transcendentals of the microphysics: FP64 (plibm) in the FP64 kernel,
// FP32 (xexp/xpow above, on the argument rounded to float) in the FP32-mixed
// kernel.  Everything else in both kernels is FP64.  With WIN (the fast pass,
// whose input checks bound the arguments) plibm's windowed forms: the same
// bits without the range selects and special-value branches, each of which
// ends a basic block.  Together with the unchecked divisions, FP64 at 262,144
// columns 12.17 -> 10.12 ms, FP32-mixed 9.08 -> 8.27 ms, a CTA of 32 columns
// alone on its SM 1.59 -> 1.41 ms.
#if defined(CLOUDSC_HOST_LIBM_GLIBC) && !defined(__CUDA_ARCH__)
#define CSC_GLIBC 1
#else
#define CSC_GLIBC 0
#endif
template <bool F32, bool WIN = false>
CSC_DEV double mexp(double x) {
  if (F32) return (double)xexp((float)x);
#if !CSC_GLIBC
  if (WIN) {
    host_check_exp(x);
    return plibm_exp_win(x, 0.0, 0);
  }
#endif
  return xexp(x);
}

// A pow base whose logarithm several calls share (FP64: plibm's double-double
// ln, computed once; FP32-mixed: nothing is precomputed).  mpowb(b, y) equals
// mpow(b.x, y) exactly.
struct PowBase {
  double x, lhi, llo;
};
template <bool F32, bool WIN = false>
CSC_DEV PowBase mbase(double x) {
  PowBase b;
  b.x = x;
  b.lhi = 0.0;
  b.llo = 0.0;
#if !CSC_GLIBC
  if (!F32) {
    if (WIN) {
      host_check_log(x);
      plibm_log_win(x, &b.lhi, &b.llo);
    } else {
      plibm_log_base(x, &b.lhi, &b.llo);
    }
  }
#endif
  return b;
}
template <bool F32, bool WIN = false>
CSC_DEV double mpowb(const PowBase &b, double y) {
  if (F32) return (double)xpow((float)b.x, (float)y);
#if CSC_GLIBC
  return pow(b.x, y);
#else
  if (WIN) return plibm_pow_with_log_win(b.x, y, b.lhi, b.llo);
  return plibm_pow_with_log(b.x, y, b.lhi, b.llo);
#endif
}
// pow with the exponent 0.5 or 1.5 in the column code: in the FP64 fast pass
// from csqrt (x^1.5 as plibm_pow1p5, for bases inside its range).
template <bool F32, bool WIN>
CSC_DEV double mroot(double x, DivCheck &dc) {
#if !CSC_GLIBC
  if (!F32 && WIN) return csqrt<WIN>(x, dc);
#endif
  (void)dc;
  if (F32) return (double)xpow((float)x, 0.5f);
  return xpow(x, 0.5);
}
template <bool F32, bool WIN>
CSC_DEV double mroot3(double x, DivCheck &dc) {
#if !CSC_GLIBC
  if (!F32 && WIN) {
    const double s = csqrt<WIN>(x, dc);
    const double e = plibm_fma(-s, s, x);
    const double p = x * s;
    const double pe = plibm_fma(x, s, -p);
    return p + (pe + (e * s) * 0.5);
  }
#endif
  (void)dc;
  if (F32) return (double)xpow((float)x, 1.5f);
  return xpow(x, 1.5);
}
template <bool F32, bool WIN = false>
CSC_DEV double mpow(double x, double y) {
  if (F32) return (double)xpow((float)x, (float)y);
#if !CSC_GLIBC
  if (WIN && y == 3.0) return plibm_cube_win(x);
  if (WIN && !plibm_pow_is_direct(y)) return mpowb<F32, WIN>(mbase<F32, WIN>(x), y);
#endif
  return xpow(x, y);
}
// pow with a parameter as exponent.  With GEN the host has checked that the
// exponent is none of 0.5, 1.5, 2 and 3, in double and rounded to float
// (gen_exponents_ok), so the tests for those exponents are left out: the
// same results as mpow / mpowb with fewer branches.
CSC_DEV float xpow_gen(float x, float y) {
#if defined(__CUDA_ARCH__)
  return __powf(x, y);
#else
  return powf(x, y);
#endif
}
template <bool F32, bool GEN, bool WIN = false>
CSC_DEV double mpowbp(const PowBase &b, double y) {
  if (!GEN) return mpowb<F32, WIN>(b, y);
  if (F32) return (double)xpow_gen((float)b.x, (float)y);
#if CSC_GLIBC
  return pow(b.x, y);
#else
  if (WIN) return plibm_pow_log_win(b.lhi, b.llo, y);
  return plibm_pow_with_log_gen(b.x, y, b.lhi, b.llo);
#endif
}
template <bool F32, bool GEN, bool WIN = false>
CSC_DEV double mpowp(double x, double y) {
  if (!GEN && !WIN) return mpow<F32>(x, y);
  return mpowbp<F32, GEN, WIN>(mbase<F32, WIN>(x), y);
}
CSC_DEV double xsqrt(double x) { return sqrt(x); }
CSC_DEV float xsqrt(float x) { return sqrtf(x); }

// The scalars the column body reads, in the working precision.  Filled on the
// host from cloudsc_params (and Derived) and uploaded to constant memory.
template <typename Real>
struct KParams {
  Real rg, rd, rv, retv, rtt, rlvtt, rlstt, rpi;
  Real r2es, r3les, r3ies, r4les, r4ies, r5les, r5ies, r5alvcp, r5alscp;
  Real ralvdcp, ralsdcp, rtwat, rtice, rtwat_rtice_r, rkoop1, rkoop2;
  Real ramid, ramin, rlmin, rcldiff, rcldiff_convi, rcovpmin, rprecrhmax, rpecons;
  Real rvrfactor, rtaumel, rssicefactor, rsnowlin1, rsnowlin2, rlcritsnow, rthomo;
  Real rvice, rvsnow, rxfallspeedrain, rcldtopcf, rdepliqrefrate, rdepliqrefdepth;
  Real riceinit, rdensref, rdenswat, rcl_overlapliqice, rcl_effrime;
  Real rcl_inhomogaut, rcl_inhomogacc, rcl_kkaac, rcl_kkbac, rcl_kkaau, rcl_kkbauq;
  Real rcl_dr, rcl_x1r, rcl_x2r, rcl_lam1r, rcl_lam2r;
  Real rcl_const1r, rcl_const2r, rcl_const3r, rcl_const4r, rcl_const5r, rcl_const6r;
  Real rcl_const7r, rcl_cdenom1, rcl_cdenom2, rcl_cdenom3, rcl_fzrab;
  Real rcl_x1s, rcl_lam1s, rcl_lam2s;
  Real rcl_const1s, rcl_const2s, rcl_const3s, rcl_const4s, rcl_const5s, rcl_const6s;
  Real rcl_const7s, rcl_const8s;
  Real rcl_apb1, rcl_apb2, rcl_apb3;
  Real rmfadvw, rmfadvwdd;
  // derived, loop-invariant
  Real zrdcp, zrg_r, zrldcp, zconst_pow_land, zconst_pow_sea, flt_0p4, flt_0p8;
  Real kkbauq_m1, kkbac_m1;
  // cloud budget diagnostics (cloudsc.F90:3832-4110)
  Real ralfdcp, reisthsc;
  int lcldbudc, lcldbudl, lcldbudi, lcldbudt, lcldbud_vertint, lcldbud_timeint, lbud23;
  // SPP perturbations and the cloud-inhomogeneity/FSD path (:850-939,
  // 1937-2110, 4307-4359)
  Real ra, rcloud_frac_std, spp_mu[16], spp_xmag[16];
  int lspp, lcloud_inhomog, lrad_cloud_inhomog, spp_lramidlimit1, spp_on[8], spp_mp[8];
  int ncldtop, lmfdsnow;
  // aerosol-aware ice sedimentation and ice-to-snow autoconversion
  // (LAERICESED, LAERICEAUTO; cloudsc.F90:1798-1803, 2776-2779)
  Real rnice;
  int laericesed, laericeauto;
  // Divisions by parameters: RV/RD in the working precision, and the
  // correctly rounded reciprocals of the parameter divisors, for cdivk.
  // rcp_force: one of those divisors is outside the division's window or has an
  // all-ones significand, or a parameter lies outside fast_pass_params_ok's
  // ranges, and every column takes the IEEE rerun.
  Real rv_rd;
  double rcp_rd, rcp_rtaumel, rcp_rcl_lam1r, rcp_rdepliqrefdepth, rcp_rvrfactor;
  int rcp_force;
};

// Double-precision copy of the scalars the FP64 stages (solve, supersaturation
// check, tendencies, fluxes) need in the mixed kernel; identical to the
// KParams<double> fields of the same name.
struct KParamsD {
  double rg, retv, rtt, rtice, rtwat, rtwat_rtice_r, r2es, r3les, r3ies, r4les, r4ies;
  double r5alvcp, r5alscp, ralvdcp, ralsdcp, rkoop1, rkoop2, rssicefactor, rlmin;
  double rlvtt, rlstt, zrg_r;
};

}  // namespace cloudsc
