// Host-side conversion of cloudsc_params into the kernels' constant blocks.
#pragma once
#include <cstdint>
#include <cstring>
#include "cloudsc_column.cuh"

namespace cloudsc {

// Whether the parameters lie inside the ranges the column code's fast pass
// assumes (its input checks bound the fields, these the parameters): positive
// divisors and pow bases of moderate size, exponents small enough that
// |y ln x| < 700 for every base x the checks allow, saturation constants that
// keep T - R4xES and 1 - RETV q away from zero for T in [128, 1024) K.  The
// defaults lie well inside; with any other value every column takes the
// rerun with IEEE division and plibm's full functions.
inline bool fast_pass_params_ok(const cloudsc_params &p) {
  bool ok = true;
  auto in = [&ok](double x, double lo, double hi) { ok = ok && x >= lo && x <= hi; };
  // positive scale factors, divisors and thresholds
  const double pos[] = {p.rg, p.rd, p.rv, p.rcpd, p.rtt, p.rlvtt, p.rlstt, p.r2es, p.r5les, p.r5ies, p.r5alvcp,
                        p.r5alscp, p.ralvdcp, p.ralsdcp, p.ramin, p.rlmin, p.rcovpmin, p.rvrfactor, p.rtaumel,
                        p.rlcritsnow, p.rxfallspeedrain, p.rdepliqrefdepth, p.riceinit, p.rdensref, p.rdenswat,
                        p.rcl_kkaac, p.rcl_kkaau, p.rcl_x1r, p.rcl_lam1r, p.rcl_const1r, p.rcl_const2r,
                        p.rcl_const5r, p.rcl_const7r, p.rcl_cdenom1, p.rcl_cdenom2, p.rcl_cdenom3, p.rcl_x1s,
                        p.rcl_lam1s, p.rcl_const1s, p.rcl_const2s, p.rcl_const3s, p.rcl_const6s, p.rcl_const7s,
                        p.rcl_apb1, p.rcl_apb2, p.rcl_apb3};
  for (double x : pos) in(x, 1e-14, 1e14);
  // factors that may be zero
  const double fac[] = {p.rcldiff, p.rcldiff_convi, p.ramid, p.rprecrhmax, p.rpecons, p.rssicefactor, p.rsnowlin1,
                        p.rvice, p.rvsnow, p.rdepliqrefrate, p.rcl_overlapliqice, p.rcl_effrime, p.rcl_inhomogaut,
                        p.rcl_inhomogacc, p.rmfadvw, p.rmfadvwdd, p.rcl_kk_cloud_num_land, p.rcl_kk_cloud_num_sea};
  for (double x : fac)
    if (x != 0.0) in(x, 1e-14, 1e14);
  // exponents
  const double ex[] = {p.rcl_kkbac, p.rcl_kkbauq, p.rcl_kkbac - 1.0, p.rcl_kkbauq - 1.0, p.rcl_dr, p.rcl_x2r,
                       p.rcl_const6r, p.rcl_const4s, p.rcl_const5s, p.rcl_const8s};
  for (double x : ex) in(x < 0.0 ? -x : x, 1e-3, 5.0);
  in(p.rcl_const3r, -2.0, 2.0);
  in(p.rcl_const4r, -2.0, 2.0);
  in(p.rcl_x2r, 0.1, 3.0);
  // the slopes (LAM1/(RHO q))**LAM2: below 1e22
  in(p.rcl_lam1r, 1.0, 1e8);
  in(p.rcl_lam1s, 1.0, 1e8);
  in(p.rcl_lam2r, 0.1, 0.7);
  in(p.rcl_lam2s, 0.1, 0.7);
  in(p.rtt, 200.0, 400.0);
  in(p.retv, 0.0, 1.0);
  in(p.r3les, 1.0, 40.0);
  in(p.r3ies, 1.0, 40.0);
  in(p.r4les, -60.0, 60.0);
  in(p.r4ies, -60.0, 60.0);
  in(p.rtice, 100.0, p.rtwat);
  in(p.rtwat, p.rtice, 400.0);
  in(p.rkoop1, 0.0, 100.0);
  in(p.rkoop2, 0.0, 1.0);
  in(p.rsnowlin2, 0.0, 0.5);
  in(p.rcl_fzrab, -1.0, 1.0);
  // the differences of the evaporation and deposition denominators positive
  // over the temperatures they are used at
  ok = ok && p.rcl_cdenom1 > 1.001 * 1024.0 * p.rcl_cdenom2 && p.rcl_apb1 > 1.001 * p.rtt * p.rcl_apb2 &&
       p.rlstt > 2.0 * p.rv * p.rtt;
  return ok;
}

template <typename Real>
inline void fill_kparams(const cloudsc_params &p, const Derived &d, KParams<Real> &k) {
#define F_(n) k.n = Real(p.n)
  F_(rg); F_(rd); F_(rv); F_(retv); F_(rtt); F_(rlvtt); F_(rlstt); F_(rpi);
  F_(r2es); F_(r3les); F_(r3ies); F_(r4les); F_(r4ies); F_(r5les); F_(r5ies); F_(r5alvcp); F_(r5alscp);
  F_(ralvdcp); F_(ralsdcp); F_(rtwat); F_(rtice); F_(rtwat_rtice_r); F_(rkoop1); F_(rkoop2);
  F_(ramid); F_(ramin); F_(rlmin); F_(rcldiff); F_(rcldiff_convi); F_(rcovpmin); F_(rprecrhmax); F_(rpecons);
  F_(rvrfactor); F_(rtaumel); F_(rssicefactor); F_(rsnowlin1); F_(rsnowlin2); F_(rlcritsnow); F_(rthomo);
  F_(rvice); F_(rvsnow); F_(rxfallspeedrain); F_(rcldtopcf); F_(rdepliqrefrate); F_(rdepliqrefdepth);
  F_(riceinit); F_(rdensref); F_(rdenswat); F_(rcl_overlapliqice); F_(rcl_effrime);
  F_(rcl_inhomogaut); F_(rcl_inhomogacc); F_(rcl_kkaac); F_(rcl_kkbac); F_(rcl_kkaau); F_(rcl_kkbauq);
  F_(rcl_dr); F_(rcl_x1r); F_(rcl_x2r); F_(rcl_lam1r); F_(rcl_lam2r);
  F_(rcl_const1r); F_(rcl_const2r); F_(rcl_const3r); F_(rcl_const4r); F_(rcl_const5r); F_(rcl_const6r);
  F_(rcl_const7r); F_(rcl_cdenom1); F_(rcl_cdenom2); F_(rcl_cdenom3); F_(rcl_fzrab);
  F_(rcl_x1s); F_(rcl_lam1s); F_(rcl_lam2s);
  F_(rcl_const1s); F_(rcl_const2s); F_(rcl_const3s); F_(rcl_const4s); F_(rcl_const5s); F_(rcl_const6s);
  F_(rcl_const7s); F_(rcl_const8s);
  F_(rcl_apb1); F_(rcl_apb2); F_(rcl_apb3);
  F_(rmfadvw); F_(rmfadvwdd);
#undef F_
  k.zrdcp = Real(p.rd / p.rcpd);
  k.zrg_r = Real(1.0 / p.rg);
  k.zrldcp = Real(1.0 / (p.ralsdcp - p.ralvdcp));
  k.zconst_pow_land = Real(d.zconst_pow_land);
  k.zconst_pow_sea = Real(d.zconst_pow_sea);
  k.flt_0p4 = Real(d.flt_0p4);
  k.flt_0p8 = Real(d.flt_0p8);
  k.kkbauq_m1 = Real(p.rcl_kkbauq - 1.0);
  k.kkbac_m1 = Real(p.rcl_kkbac - 1.0);
  k.ralfdcp = Real(p.ralfdcp);
  k.reisthsc = Real(p.reisthsc);
  k.lcldbudc = p.lcldbudc;
  k.lcldbudl = p.lcldbudl;
  k.lcldbudi = p.lcldbudi;
  k.lcldbudt = p.lcldbudt;
  k.lcldbud_vertint = p.lcldbud_vertint;
  k.lcldbud_timeint = p.lcldbud_timeint;
  k.lbud23 = p.lbud23;
  k.ra = Real(p.ra);
  k.rcloud_frac_std = Real(p.rcloud_frac_std);
  for (int i = 0; i < 16; ++i) {
    k.spp_mu[i] = Real(p.spp_mu[i]);
    k.spp_xmag[i] = Real(p.spp_xmag[i]);
  }
  k.lspp = p.lspp;
  k.lcloud_inhomog = p.lcloud_inhomog;
  k.lrad_cloud_inhomog = p.lrad_cloud_inhomog;
  k.spp_lramidlimit1 = p.spp_lramidlimit1;
  for (int i = 0; i < 8; ++i) {
    k.spp_on[i] = p.spp_on[i];
    k.spp_mp[i] = p.spp_mp[i];
  }
  k.ncldtop = p.ncldtop;
  k.lmfdsnow = p.lmfdsnow;
  k.rnice = Real(p.rnice);
  k.laericesed = p.laericesed;
  k.laericeauto = p.laericeauto;
  // RV/RD with the division the kernels would perform (IEEE, in Real)
  k.rv_rd = Real(p.rv) / Real(p.rd);
  // 1/b correctly rounded (IEEE on the host) for each parameter divisor;
  // usable by cdivk only inside its window and without an all-ones
  // significand
  bool ok = fast_pass_params_ok(p);
  auto rcp = [&ok](double b) {
    uint64_t u;
    std::memcpy(&u, &b, 8);
    const unsigned e = (unsigned)((u >> 52) & 0x7ff);
    const bool ones = (u & ((1ull << 52) - 1)) == ((1ull << 52) - 1);
    ok = ok && e >= 767u && e <= 1278u && !ones;
    return 1.0 / b;
  };
  k.rcp_rd = rcp(p.rd);
  k.rcp_rtaumel = rcp(p.rtaumel);
  k.rcp_rcl_lam1r = rcp(p.rcl_lam1r);
  k.rcp_rdepliqrefdepth = rcp(p.rdepliqrefdepth);
  k.rcp_rvrfactor = rcp(p.rvrfactor);
  k.rcp_force = ok ? 0 : 1;
}


// The kernels' pows whose exponent is a parameter (mpowp / mpowbp in
// cloudsc_body.cuh) may skip their tests for the exponents 0.5, 1.5, 2 and 3
// (the GEN kernels) when none of these parameters is such an exponent, in
// double or rounded to float.  This list names every exponent those call
// sites use.
inline bool gen_exponents_ok(const KParams<double> &k) {
  const double ex[] = {k.flt_0p4,     k.kkbac_m1,    k.kkbauq_m1,   k.rcl_const3r, k.rcl_const4r,
                       k.rcl_const4s, k.rcl_const5s, k.rcl_const6r, k.rcl_const8s, k.rcl_dr,
                       k.rcl_kkbac,   k.rcl_lam2r,   k.rcl_lam2s,   k.rcl_x2r};
  for (double y : ex) {
    const float yf = (float)y;
    if (y == 0.5 || y == 1.5 || y == 2.0 || y == 3.0) return false;
    if (yf == 0.5f || yf == 1.5f || yf == 2.0f || yf == 3.0f) return false;
  }
  return true;
}

inline void fill_kparams_d(const cloudsc_params &p, KParamsD &dd) {
  dd.rg = p.rg; dd.retv = p.retv; dd.rtt = p.rtt; dd.rtice = p.rtice; dd.rtwat = p.rtwat;
  dd.rtwat_rtice_r = p.rtwat_rtice_r; dd.r2es = p.r2es; dd.r3les = p.r3les; dd.r3ies = p.r3ies;
  dd.r4les = p.r4les; dd.r4ies = p.r4ies; dd.r5alvcp = p.r5alvcp; dd.r5alscp = p.r5alscp;
  dd.ralvdcp = p.ralvdcp; dd.ralsdcp = p.ralsdcp; dd.rkoop1 = p.rkoop1; dd.rkoop2 = p.rkoop2;
  dd.rssicefactor = p.rssicefactor; dd.rlmin = p.rlmin; dd.rlvtt = p.rlvtt; dd.rlstt = p.rlstt;
  dd.zrg_r = 1.0 / p.rg;
}

}  // namespace cloudsc
