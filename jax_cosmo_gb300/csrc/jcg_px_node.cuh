// The Limber integrand of the plain method at one (a, ell) node in float pairs
// (jcg_px.cuh): halofit_node_lk of jcg_internal.cuh, times k^3 / (2 pi^2).
#pragma once

#include "jcg_px.cuh"

namespace jcg {

// per a node: pairs (as float2) and fixed point numbers, 8 bytes each
enum PxRow {
  PR_ALPHA = 0, PR_NU, PR_MU,  // the first two floats of each
  PR_ICHIC,      // 1 / chi_c (float64)
  PR_IYK,        // 1 / (chi_c k_nl) (float64)
  PR_L2C,        // log2 chi_c, 2^-57
  PR_L2Y,        // log2(chi_c k_nl), 2^-57
  PR_L3,         // log2(c_n f_3), 2^-57
  PR_BETA, PR_E1, PR_E2, PR_E3,  // beta_n, 3 f_1, f_2, 3 - gamma_n, 2^-60
  PR_A0, PR_B0,  // log2 a_n, log2 b_n, 2^-53
  PR_LD,         // log2(g^2 pknorm f_c^2 / (2 pi^2)) (type "eisenhu": without f_c), 2^-53
  PR_V,          // 2 pi^2 u chi_c^3 (float64)
  PR_LL,         // third floats of the first three: a slot and a half
  PR_N = PR_LL + 2
};

// per cosmology
struct PxCos {
  double qinv, c1, c2, cab;
  F3 c54, c52, bb3, bn3, ab, shpi, fbp;  // fbp: f_b / (f_c pi)
  F3 agam, oag, nwq, xn2;             // type "eisenhu"
  long long l69, lks, ns3;            // log2(69.9 qinv^1.08), log2(log2 e / k_silk^1.4) (2^-53), n_s + 3 (2^-60)
};

constexpr double P2_57 = 144115188075855872.0, P2_53 = 9007199254740992.0, P2_60 = 1152921504606846976.0;
constexpr double D_LOG2E = 1.4426950408889634074, PX_E = 2.718281828459045;

__host__ __device__ constexpr F3 pxc(double v) {
  return F3{(float)v, (float)(v - (double)(float)v),
            (float)(v - (double)(float)v - (double)(float)(v - (double)(float)v))};
}
__host__ __device__ constexpr long long pxe(double v) {  // an exponent constant, 2^-60 units
  return (long long)(v * 1152921504606846976.0 + (v > 0 ? 0.5 : -0.5));
}

PX_FN F3 row3(const long long* row, int i, int part) {
  const float2* rp = reinterpret_cast<const float2*>(row);
  const float2 v = rp[i];
  const float2 w = rp[PR_LL + (part >> 1)];
  return F3{v.x, v.y, (part & 1) ? w.y : w.x};
}

// T(k) / f_c, type "eisenhu_osc" (transfer.py:107-153), the terms of
// eh_osc_lki.  The cold dark matter part, which T is made of but for some
// percent, adds up its transcendentals in float64 (30 operations, beside the
// FP32 pipe's work); the baryon part is in pairs.
PX_FN double px_eh_osc(const PxCos& c, const PxTab& T, double kd, FF k, FF k2, long long lk) {
  const double qd = kd * c.qinv, qq = qd * qd;
  const FF u = px_exp2(px_mulhi(pxe(1.08), lk) + c.l69, T);  // 69.9 q^1.08
  const double Cb = px_join(px_div(FF{386.f, 0.f}, px_1p(u)));
  const FF L2 = px_ln(px_split(fma(c.c2, kd, PX_E)), T);
  const double L1 = px_join(px_ln(px_split(fma(c.c1, kd, PX_E)), T));
  const double cA = Cb + 14.2, cB = Cb + c.cab;
  const double Da = fma(cA, qq, L1), Db = fma(cB, qq, L1), Dn = fma(cA, qq, px_join(L2));
  // f L1 / Da + (1 - f) L1 / Db over one denominator
  const FF x4 = px_sqr(px_mul(k2, c.c54));
  const double Dab = Da * Db;
  const double Tc = px_ddiv(L1 * fma(px_join(px_rcp2(px_1p(x4))), Db - Da, Da), Dab, px_rcp(px_hi(Dab)));
  // baryons
  const FF k3 = px_mul(k2, k);
  FF Tbr = px_div(L2, px_mul(px_split(Dn), px_1p(px_mul(k2, c.c52))));
  const FF ex1 = px_exp2(px_mulhi(pxe(1.4), lk) + c.lks, T);  // (k / k_silk)^1.4 log2 e
  if (ex1.hi < 110.f) {
    const FF silk = px_exp2(-px_fix53(ex1), T);
    Tbr = px_add(Tbr, px_div(px_mul(px_mul(silk, c.ab), k3), px_add(k3, c.bb3)));
  }
  // k tilde_s / pi = (sh_d / pi) k^2 (k^3 + beta_node^3 / sh_d^3)^(-1/3); past px_sinpi's
  // range (k above 2,500 h/Mpc) the term is below 1e-11 of T, and T stays within
  // 1.1e-14 of float64 up to k = 10^7, where the callers stop
  const FF ph = px_mul(px_mul(k2, c.shpi), px_rcbrt(px_add(k3, c.bn3)));
  const FF sinc = px_div(px_sinpi(ph, T), ph);
  return Tc + px_join(px_mul(px_mul(Tbr, c.fbp), sinc));
}

// type "eisenhu" (transfer.py:88-105)
PX_FN FF px_eh_nowiggle(const PxCos& c, const PxTab& T, FF k, FF k2) {
  const FF g = px_add(px_mul(px_rcp2(px_1p(px_sqr(px_mul(k2, c.xn2)))), c.oag), c.agam);
  const FF q = px_div(px_mul(k, c.nwq), g);
  const FF L = px_ln(px_add(px_mul(q, pxc(1.8)), pxc(2.0 * PX_E)), T);
  const FF C = px_add(px_div(FF{731.f, 0.f}, px_1p(px_mul(q, FF{62.5f, 0.f}))), pxc(14.2));
  return px_div(L, px_add(L, px_mul(C, px_sqr(q))));
}

// S = k^3 P(k, a) / (2 pi^2) at one node: halofit_node_lk in pairs.  GEN: the
// non-default operator points.
template <bool GEN>
PX_FN FF px_node(const PxCos& c, const PxTab& T, const long long* row, double kh, long long l2kh,
                                      bool nw, bool lin) {
  const double* rd = reinterpret_cast<const double*>(row);
  const double kd = kh * rd[PR_ICHIC];
  const FF k = px_split(kd);
  const long long lk = l2kh - row[PR_L2C];
  const FF k2 = px_sqr(k);
  double t;
  if (GEN && nw) t = px_join(px_eh_nowiggle(c, T, k, k2));
  else t = px_eh_osc(c, T, kd, k, k2, lk);
  const double d2 = px_join(px_exp2(px_mulhi(c.ns3, lk) + row[PR_LD], T)) * (t * t);
  const FF d2l = px_split(d2);
  if (px_tiny(d2)) return FF{0.f, 0.f};  // the caller takes float64
  if (GEN && lin) return d2l;
  const FF y = px_split(kh * rd[PR_IYK]);
  const long long ly = l2kh - row[PR_L2Y];
  const FF y2 = px_sqr(y);
  // (1 + d2l)^beta exp(-(y/4 + y^2/8)) / (1 + alpha d2l)
  const FF fy = px_mul(y, px_add(px_mul(y, pxc(D_LOG2E / 8)), pxc(D_LOG2E / 4)));
  FF s = FF{0.f, 0.f};
  if (fy.hi < 200.f) {
    const FF e1 = px_exp2(px_mulhi(row[PR_BETA], px_log2(px_split(1.0 + d2), T)) - px_fix53(fy), T);
    s = px_div(px_mul(d2l, e1), px_1p(px_mul(d2l, row3(row, PR_ALPHA, 0))));
  }
  const FF H = px_exp2(px_mulhi(row[PR_E1], ly) + row[PR_A0], T);
  const FF B = px_exp2(px_mulhi(row[PR_E2], ly) + row[PR_B0], T);
  const FF G = px_exp2(px_mulhi(row[PR_E3], ly + row[PR_L3]), T);
  FF dn = px_add(y2, row3(row, PR_NU, 1));
  if (GEN) dn = px_add(dn, px_mul(y, row3(row, PR_MU, 2)));
  return px_add(s, px_div(px_mul(H, y2), px_mul(px_add(px_1p(B), G), dn)));
}

}  // namespace jcg
