// The Limber integrand of the float64 gradient at one (a, ell) node in float
// pairs: S = k^3 P / (2 pi^2) as px_node (jcg_px_node.cuh) and its 8 tangents.
//
// S is a sum of two products of powers, so a reverse sweep in logarithmic
// derivatives is short: a weight per input (12 of the a node, 10 of the
// transfer function, n_s), each a few pair operations on the forward's factors,
// and dS = sum of weight x tangent of the input.  The tangents of the transfer
// function's inputs are 0 but in the directions of Omega_c, Omega_b and h: three
// products instead of eight.
#pragma once

#include "jcg_px_node.cuh"

namespace jcg {

// per a node, 8 bytes each: numbers as in PxRow, then the tangents as pairs
enum GxRow {
  GR_ICHIC = 0, GR_IYK,               // float64
  GR_L2C, GR_L2Y, GR_L3,              // 2^-57
  GR_BETA, GR_E1, GR_E2, GR_E3,       // 2^-60
  GR_A0, GR_B0, GR_LD,                // 2^-53
  GR_ALPHA, GR_NU, GR_MU,             // pairs
  GR_MUC,                             // dmu / dnu (both functions of n_eff alone)
  GR_V,                               // 2 pi^2 u chi_c^3, value and 8 tangents (pairs)
  GR_T = GR_V + 10,                   // tangents [GxTan][8], 16-byte aligned
};
// inputs of an a node: ln(1 / chi_c), ln of the linear amplitude, ln(1 / (chi_c
// k_nl)), beta, alpha, ln a_n, 3 f_1, ln b_n, f_2, 3 - gamma, its product with
// ln(c_n f_3), nu
enum GxTan { GT_K = 0, GT_A, GT_Y, GT_BETA, GT_ALPHA, GT_AN, GT_E1, GT_BN, GT_E2, GT_E3, GT_G0, GT_NU, GT_N };
static_assert(GR_T % 2 == 0, "tangents are read 16 bytes at a time");
// inputs of the transfer function (ln; type "eisenhu": the first three are
// ln sh_d, alpha_gamma's ln and ln of the q factor)
enum GxCos { GC_SH = 0, GC_KEQ, GC_BETAC, GC_ALPHAC, GC_ALPHAB, GC_BETAB, GC_BETANODE, GC_KSILK, GC_FB, GC_FC, GC_N };
constexpr int GC_AGAM = GC_KEQ, GC_NWQ = GC_BETAC;
constexpr int GX_NS = 3;  // the direction of n_s

struct GxTabs {
  PxCos c;
  F3 cab;                 // 14.2 / alpha_c
  F3 dT[GC_N][4];         // tangents in directions 0..2
  F3 dns;                 // of n_s, in its direction
};

struct GxT {  // T / f_c and its partials in the logarithms of GxCos and of k
  double t;
  FF w[GC_N], k;
};

__device__ __forceinline__ FF px_neg(FF a) { return FF{-a.hi, -a.lo}; }
__device__ __forceinline__ FF px_x2(FF a) { return FF{2.f * a.hi, 2.f * a.lo}; }
__device__ __forceinline__ FF px_sub(FF a, FF b) { return px_add(a, px_neg(b)); }
__device__ __forceinline__ FF px_mulf(FF a, float b) {
  const float p = a.hi * b;
  return px_norm(p, fmaf(a.lo, b, fmaf(a.hi, b, -p)));
}

__device__ __forceinline__ void px_eh_osc_grad(const GxTabs& g, const PxTab& T, double kd, FF k, FF k2, long long lk,
                                               GxT& o) {
  const PxCos& c = g.c;
  const double qd = kd * c.qinv, qq = qd * qd;
  const FF u = px_exp2(px_mulhi(pxe(1.08), lk) + c.l69, T);
  const FF u1 = px_1p(u);
  const FF Cbp = px_div(FF{386.f, 0.f}, u1);
  const double Cb = px_join(Cbp);
  const double k18 = c.c2 * kd, kb18 = c.c1 * kd;  // 1.8 q, 1.8 beta_c q
  const FF A1 = px_split(kb18 + PX_E), A2 = px_split(k18 + PX_E);
  const FF L1p = px_ln(A1, T), L2 = px_ln(A2, T);
  const double L1 = px_join(L1p);
  const double cA = Cb + 14.2, cB = Cb + c.cab;
  const double Da = fma(cA, qq, L1), Db = fma(cB, qq, L1), Dn = fma(cA, qq, px_join(L2));
  const FF x4 = px_sqr(px_mul(k2, c.c54));
  const FF f = px_rcp2(px_1p(x4)), f1 = px_mul(x4, f);  // f and 1 - f
  const double Dab = Da * Db;
  const double Tc = px_ddiv(L1 * fma(px_join(f), Db - Da, Da), Dab, px_rcp(px_hi(Dab)));
  const FF cAq = px_split(cA * qq), rDa = px_rcp2(px_split(Da)), rDb = px_rcp2(px_split(Db)),
           rDn = px_rcp2(px_split(Dn));
  const FF Ta = px_mul(L1p, rDa), Tb = px_mul(L1p, rDb);
  const FF Xa = px_mul(px_mul(f, Ta), px_mul(cAq, rDa));
  const FF Xb = px_mul(px_mul(f1, Tb), px_mul(px_split(cB * qq), rDb));
  // baryons: two terms, times sinc
  const FF k3 = px_mul(k2, k);
  const FF k52 = px_mul(k2, c.c52), iE = px_rcp2(px_1p(k52));
  const FF t1 = px_mul(px_mul(L2, rDn), iE);
  const FF ex1 = px_exp2(px_mulhi(pxe(1.4), lk) + c.lks, T);
  FF t2 = FF{0.f, 0.f}, w3c = t2, exs = t2;  // w3c: 1 - w3
  if (ex1.hi < 110.f) {
    const FF silk = px_exp2(-px_fix53(ex1), T);
    const FF r3 = px_rcp2(px_add(k3, c.bb3));
    w3c = px_mul(r3, c.bb3);
    t2 = px_mul(px_mul(silk, c.ab), px_mul(k3, r3));
    exs = px_mul(ex1, pxc(1.4 * 0.693147180559945309417));
  }
  const FF kn = px_add(k3, c.bn3);
  const FF ph = px_mul(px_mul(k2, c.shpi), px_rcbrt(kn));
  FF cs;
  const FF sinc = px_div(px_sincospi<true>(ph, T, &cs), ph);
  const FF fs = px_mul(sinc, c.fbp);
  const FF b1 = px_mul(t1, fs), b2 = px_mul(t2, fs), Bt = px_add(b1, b2);
  o.t = Tc + px_join(Bt);
  // reverse
  const FF Xn = px_mul(b1, px_mul(cAq, rDn)), Xan = px_add(Xa, Xn), X = px_add(Xan, Xb);
  const FF bc = px_mul(px_add(Xa, Xb), px_div(px_split(kb18), px_mul(A1, L1p)));
  const FF kap = px_mul(px_mul(px_div(u, u1), Cbp), pxc(1.08));
  const FF rcB = px_rcp2(px_split(cB));
  FF dq = px_add(bc, px_mul(Xn, px_div(px_split(k18), px_mul(A2, L2))));
  dq = px_add(dq, px_mul(kap, px_add(px_div(Xan, px_split(cA)), px_mul(Xb, rcB))));
  dq = px_sub(dq, px_x2(X));
  const FF da = px_mul(px_mul(px_add(t1, t2), c.fbp), px_sub(px_mul(cs, pxc(PI)), sinc));  // d T / d ln arg
  const FF bw = px_mulf(px_mul(w3c, b2), 3.f);
  const FF zda = px_mul(px_mul(px_rcp2(kn), c.bn3), da);
  FF sh = px_mulf(px_mul(px_mul(f, f1), px_sub(Tb, Ta)), 4.f);
  sh = px_sub(sh, px_x2(px_mul(b1, px_mul(k52, iE))));
  sh = px_add(px_add(sh, bw), px_add(da, zda));
  const FF ks = px_mul(exs, b2);
  o.w[GC_SH] = sh;
  o.w[GC_KEQ] = px_neg(dq);
  o.w[GC_BETAC] = bc;
  o.w[GC_ALPHAC] = px_mul(px_mul(Xb, rcB), g.cab);
  o.w[GC_ALPHAB] = b2;
  o.w[GC_BETAB] = px_neg(bw);
  o.w[GC_BETANODE] = px_neg(zda);
  o.w[GC_KSILK] = ks;
  o.w[GC_FB] = Bt;
  o.w[GC_FC] = px_of(Tc);
  o.k = px_sub(px_add(dq, sh), ks);
}

// type "eisenhu" (transfer.py:88-105)
__device__ __forceinline__ void px_eh_nowiggle_grad(const GxTabs& g, const PxTab& T, FF k, FF k2, GxT& o) {
  const PxCos& c = g.c;
  const FF x4 = px_sqr(px_mul(k2, c.xn2)), un = px_rcp2(px_1p(x4)), u1 = px_mul(x4, un);  // u1: 1 - un
  const FF gen = px_add(px_mul(un, c.oag), c.agam), ig = px_rcp2(gen);
  const FF q = px_mul(px_mul(k, c.nwq), ig);
  const FF q18 = px_mul(q, pxc(1.8)), A = px_add(q18, pxc(2.0 * PX_E));
  const FF L = px_ln(A, T);
  const FF q62 = px_mul(q, FF{62.5f, 0.f}), r = px_rcp2(px_1p(q62));
  const FF C = px_add(px_mul(r, FF{731.f, 0.f}), pxc(14.2));
  const FF Cq = px_mul(C, px_sqr(q)), iD = px_rcp2(px_add(L, Cq));
  const FF t = px_mul(L, iD);
  o.t = px_join(t);
  const FF X = px_mul(t, px_mul(Cq, iD));  // T (1 - T)
  FF m = px_div(q18, px_mul(A, L));
  m = px_add(m, px_mul(px_mul(px_div(q62, C), FF{731.f, 0.f}), px_sqr(r)));
  const FF dq = px_mul(X, px_add(m, FF{-2.f, 0.f}));
  const FF s = px_mul(px_mul(px_mul(dq, ig), c.oag), px_mulf(px_mul(un, u1), 4.f));
  o.w[GC_SH] = s;
  o.w[GC_AGAM] = px_neg(px_mul(px_mul(px_mul(dq, ig), u1), c.agam));
  o.w[GC_NWQ] = dq;
  o.k = px_add(dq, s);
}

struct GxAcc {
  F3 a[NDIR];
};
// a += w b in three floats: a tangent's terms are up to ten times their sum, so
// pairs would round it ten times as much as S
__device__ __forceinline__ void gx_acc(F3& a, FF w, float2 b) {
  const float p = w.hi * b.x;
  const FF s = px_two_sum(a.hi, p);
  const FF t = px_two_sum(a.lo, s.lo);
  const FF u = px_two_sum(t.hi, fmaf(w.hi, b.x, -p));
  a = F3{s.hi, u.hi, a.ll + ((t.lo + u.lo) + fmaf(w.hi, b.y, w.lo * b.x))};
}
__device__ __forceinline__ void gx_acc(F3& a, FF w, F3 b) {
  const float p = w.hi * b.hi;
  const FF s = px_two_sum(a.hi, p);
  const FF t = px_two_sum(a.lo, s.lo);
  const FF u = px_two_sum(t.hi, fmaf(w.hi, b.hi, -p));
  a = F3{s.hi, u.hi, a.ll + ((t.lo + u.lo) + fmaf(w.lo, b.hi, fmaf(w.hi, b.lo, w.hi * b.ll)))};
}
// dS += w x the 8 tangents at d; BG: an input of the background alone
template <bool BG>
__device__ __forceinline__ void gx_mac(GxAcc& a, FF w, const float2* d) {
#pragma unroll
  for (int q = 0; q < NDIR / 2; ++q) {
    if (BG && !bg_dir(2 * q) && !bg_dir(2 * q + 1)) continue;
    const float4 v = reinterpret_cast<const float4*>(d)[q];
    if (!BG || bg_dir(2 * q)) gx_acc(a.a[2 * q], w, make_float2(v.x, v.y));
    if (!BG || bg_dir(2 * q + 1)) gx_acc(a.a[2 * q + 1], w, make_float2(v.z, v.w));
  }
}

// S into out[0], its tangents into out[1 + d]
template <bool GEN>
__device__ __forceinline__ void px_node_grad(const GxTabs& g, const PxTab& T, const long long* row, double kh,
                                             long long l2kh, bool nw, bool lin, FF* out) {
  const double* rd = reinterpret_cast<const double*>(row);
  const float2* rf = reinterpret_cast<const float2*>(row);
  const float2* tan = rf + GR_T;
  const double kd = kh * rd[GR_ICHIC];
  const FF k = px_split(kd);
  const long long lk = l2kh - row[GR_L2C];
  const FF k2 = px_sqr(k);
  GxT tr;
  if (GEN && nw) px_eh_nowiggle_grad(g, T, k, k2, tr);
  else px_eh_osc_grad(g, T, kd, k, k2, lk, tr);
  const double d2 = px_join(px_exp2(px_mulhi(g.c.ns3, lk) + row[GR_LD], T)) * (tr.t * tr.t);
  const FF d2l = px_split(d2);
  GxAcc acc;
#pragma unroll
  for (int d = 0; d < NDIR; ++d) acc.a[d] = F3{0.f, 0.f, 0.f};
  FF S = d2l, wl = d2l;  // wl: d S / d ln d2l
  if (!(GEN && lin)) {
    const FF y = px_split(kh * rd[GR_IYK]);
    const long long ly = l2kh - row[GR_L2Y];
    const FF lyn = px_mul(px_unfix60(ly), pxc(8.0 * 0.693147180559945309417));  // ln y
    const FF y2 = px_sqr(y);
    const FF H = px_exp2(px_mulhi(row[GR_E1], ly) + row[GR_A0], T);
    const FF B = px_exp2(px_mulhi(row[GR_E2], ly) + row[GR_B0], T);
    const FF G = px_exp2(px_mulhi(row[GR_E3], ly + row[GR_L3]), T);
    const FF my = GEN ? px_mul(y, px_f2(rf[GR_MU])) : FF{0.f, 0.f};
    const FF nu = px_f2(rf[GR_NU]);
    FF nm = nu;
    if (GEN) nm = px_add(nm, my);
    const FF iD = px_rcp2(px_add(px_1p(B), G)), in = px_rcp2(px_add(y2, nm));
    const FF h = px_mul(px_mul(H, y2), px_mul(iD, in));
    const FF hD = px_mul(h, iD), hB = px_neg(px_mul(hD, B)), hG = px_neg(px_mul(hD, G));
    gx_mac<false>(acc, h, tan + GT_AN * NDIR);
    gx_mac<false>(acc, hB, tan + GT_BN * NDIR);
    gx_mac<false>(acc, hG, tan + GT_G0 * NDIR);
    gx_mac<true>(acc, px_mul(h, lyn), tan + GT_E1 * NDIR);
    gx_mac<true>(acc, px_mul(hB, lyn), tan + GT_E2 * NDIR);
    gx_mac<false>(acc, px_mul(hG, lyn), tan + GT_E3 * NDIR);
    const FF hn = px_mul(h, in);
    {
      FF w = hn;
      if (GEN) w = px_mul(hn, px_add(FF{1.f, 0.f}, px_mul(y, px_f2(rf[GR_MUC]))));
      gx_mac<false>(acc, px_neg(w), tan + GT_NU * NDIR);
    }
    // d h / d ln y
    FF wy = px_add(px_mul(h, px_unfix60(row[GR_E1])), px_mul(hB, px_unfix60(row[GR_E2])));
    wy = px_add(wy, px_mul(hG, px_unfix60(row[GR_E3])));
    wy = px_add(wy, px_mul(hn, GEN ? px_add(px_x2(nu), my) : px_x2(nu)));
    const FF fy = px_mul(y, px_add(px_mul(y, pxc(D_LOG2E / 8)), pxc(D_LOG2E / 4)));
    S = h;
    wl = FF{0.f, 0.f};
    if (fy.hi < 200.f) {
      const FF d1 = px_split(1.0 + d2);
      const long long ld = px_log2(d1, T);
      const FF ia = px_rcp2(px_1p(px_mul(d2l, px_f2(rf[GR_ALPHA]))));
      const FF s = px_mul(px_mul(d2l, px_exp2(px_mulhi(row[GR_BETA], ld) - px_fix53(fy), T)), ia);
      const FF sa = px_mul(px_mul(s, d2l), ia);  // s d2l / (1 + alpha d2l)
      const FF sy = px_mul(s, px_add(y, y2));
      wy = px_sub(wy, FF{0.25f * sy.hi, 0.25f * sy.lo});
      gx_mac<false>(acc, px_neg(sa), tan + GT_ALPHA * NDIR);
      gx_mac<false>(acc, px_mul(s, px_mul(px_unfix60(ld), pxc(8.0 * 0.693147180559945309417))), tan + GT_BETA * NDIR);
      wl = px_add(s, px_mul(s, px_mul(px_unfix60(row[GR_BETA]), px_div(d2l, d1))));
      wl = px_sub(wl, px_mul(sa, px_f2(rf[GR_ALPHA])));
      S = px_add(s, h);
    }
    gx_mac<false>(acc, wy, tan + GT_Y * NDIR);
  }
  gx_mac<false>(acc, wl, tan + GT_A * NDIR);
  const FF wT = px_x2(px_div(wl, px_of(tr.t)));  // T may be below 0
  const FF nk = px_add(px_mul(wl, px_unfix60(g.c.ns3)), px_mul(wT, tr.k));
  gx_mac<true>(acc, nk, tan + GT_K * NDIR);
  gx_acc(acc.a[GX_NS], px_mul(wl, px_mul(px_unfix60(lk), pxc(8.0 * 0.693147180559945309417))), g.dns);
#pragma unroll
  for (int x = 0; x < GC_N; ++x) {
    if (GEN && nw && x > GC_NWQ) break;
    const FF w = px_mul(wT, tr.w[x]);
#pragma unroll
    for (int d = 0; d < 3; ++d) gx_acc(acc.a[d], w, g.dT[x][d]);
  }
  out[0] = px_tiny(d2) ? FF{0.f, 0.f} : S;
#pragma unroll
  for (int d = 0; d < NDIR; ++d) out[1 + d] = px_norm(acc.a[d].hi, acc.a[d].lo + acc.a[d].ll);
}

}  // namespace jcg
