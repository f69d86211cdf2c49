// Limber rows of the float64 gradient with their 8 tangents.
//
//   grad_moments64_kernel   growth and root find of a node (a thread each), then
//     halofit's moments (power.py:121-139), a warp per node in float pairs
//     (jcg_px.cuh):
//       S1 = 2 sum w y^2 e^{-y^2},  S2 = 4 sum w (y^2 - y^4) e^{-y^2},  y = k R,
//     the same sums with dw_d for w (five directions), and S3 = 8 sum w y^2 (1 - 3 y^2 + y^4)
//     e^{-y^2}: dS1 = S1[dw_d] + S2 dln R, dS2 = S2[dw_d] + S3 dln R;
//   grad_rowfin64_kernel    the coefficients (power.py:177-242) and the Limber
//     weight: values once, tangents in closed form, in float64.
//
// One kernel did both, 32 lanes of (node, direction) in Dual<1> float64: the
// coefficients' exponentials eight times over, the moments on the FP64 pipe.
// One cosmology, 513 nodes 200 -> 15 + 26 us, 61 cosmologies 1,260 -> 131 + 128
// us; the second kernel is bound by the FP64 pipe, the first by issue.
//
// Tracer radial kernels of the float64 gradient (probes.py:16-129, 188-272) with
// their 8 tangents.
//
//   grad_wlsum64_kernel   the z' integral of the WeakLensing bins.  With
//     r = (chi' - chi) / chi',   dr = (chi / chi'^2) dchi' - dchi / chi'
//     a bin's sum, its tangent sums A_d = sum W (chi / chi'^2) dchi'_d and
//     B = sum W / chi' (dK_d = A_d - dchi_d B) are sums of products in float
//     pairs (jcg_px.cuh), weights scaled per (node, bin) as in jcg_tracer64.cu.  A
//     warp per (cosmology, node), points over lanes, three bins at a time in
//     registers (a warp per pass); the lanes' sums are added by one lane per sum.
//   grad_kernfin64_kernel   a thread per (node, tracer): prefactors, single planes,
//     NumberCounts and alignment terms in float64.
//
// One kernel did both in Dual<8> float64 (a warp per node, the second part on 8
// of its lanes): 61 cosmologies, 3 + 2 bins with alignment terms, 513 nodes
// 5.00 -> 0.47 + 0.23 ms; one cosmology, 5 + 5 bins 208 -> 30 + 12 us (all eight
// directions: 0.57 ms and 40 us; four bins a pass: 0.51 ms and 38 us).  The first
// is bound by issue (some 400 instructions a point and three bins), the second by
// the FP64 pipe.
//
// Rows and kernels do not depend on one another: few cosmologies run moments and
// lensing sums in one launch, and coefficients and prefactors in another
// (grad_front64a_kernel, grad_front64b_kernel), CTAs of either kind side by side.
#include "jcg_grad.cuh"
#include "jcg_px_node.cuh"
#include "jcg_wl64.cuh"

namespace jcg {

// ------------------------------------------------------------------- rows ---

constexpr int GR64_WARPS = 8;
constexpr int GR64_NODES = 64;             // nodes per CTA at most
constexpr int GR64_SUMS = 2 * (NPW + 1) + 1;
struct Gr64Smem {
  PxTab T;
  float2 w[NPW + 1][NKH], kh2[NKH];
  double sig[NRT];
  float2 runs[GR64_WARPS][GR64_SUMS][33];
  double R[GR64_NODES];
  int wide;
};

__device__ __forceinline__ void moments64(const GradBatch& gb, const ConstTables* __restrict__ c, int nb, int only_wide,
                                          int block, int item, unsigned char* smem) {
  const GradItem gi = grad_item(gb, item);
  const TabD* tb = gi.tab;
  if (only_wide && !tb->wide) return;
  const GeoHeader* geo = gi.geo;
  const int na = geo->na, n0 = block * nb;
  if (n0 >= na) return;
  const int cnt = min(na - n0, nb);
  Gr64Smem& S = *reinterpret_cast<Gr64Smem*>(smem);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const float2* kw = grad_kw64(tb);
  if (tid == 0) S.wide = 0;
  for (int i = tid; i < (int)(sizeof(PxTab) / 16); i += GR64_WARPS * 32)
    reinterpret_cast<uint4*>(&S.T)[i] = reinterpret_cast<const uint4*>(&c->px)[i];
  for (int i = tid; i < NRT; i += GR64_WARPS * 32) S.sig[i] = tb->sigv[i];
  __syncthreads();
  for (int i = tid; i < (NPW + 1) * NKH; i += GR64_WARPS * 32) {
    const float2 v = kw[i];
    S.w[0][i] = v;
    // outside what the pairs hold: float64 terms
    if (!(fabsf(v.x) < 1e28f) || (i < NKH && !(v.x > 1e-28f))) S.wide = 1;
  }
  for (int i = tid; i < NKH; i += GR64_WARPS * 32) S.kh2[i] = make_float2(c->kh2_hi[i], c->kh2_lo[i]);
  const double* A = geo_ptr<double>(geo, geo->off_a);
  const int64_t* SG = geo_ptr<int64_t>(geo, geo->off_seg_grow);
  // growth and the root find (power.py:96-118)
  for (int t = tid; t < cnt; t += GR64_WARPS * 32) {
    const int n = n0 + t;
    const D1 g1 = interp_d1(A[n], c->atab_grow, tb->gv, tb->gv, unpack_seg(SG[n]));
    const double g = fmin(fmax(g1.v, 0.0), 1.0), g2 = g * g;
    int ind, j2;
    if (gb.seg_in) {
      // the segment of another parameter point: differentiate on its branch
      const int pk = gb.seg_in[(size_t)item * na + n];
      ind = min(max(pk & 0xffff, 1), NRT - 2);
      j2 = ind + ((pk >> 16) ? 1 : -1);
    } else {
      root_segment(S.sig, g2, ind, j2);
    }
    const int seg = ind | ((j2 > ind ? 1 : 0) << 16);
    if (gb.seg_out) gb.seg_out[(size_t)item * na + n] = seg;
    const double xp0 = S.sig[ind] * g2, xp1 = S.sig[j2] * g2;
    const double root = (c->logr[j2] - c->logr[ind]) / (xp1 - xp0) * (1.0 - xp0) + c->logr[ind];
    const double R = xfmax(exp(root), 1e-6);
    S.R[t] = R;
    if (!(R < 1e6)) S.wide = 1;
    double* row = gi.rowd + (size_t)n * NROWD;
    row[GR64_SUMS] = (double)seg;
    row[GR64_SUMS + 1] = g;
  }
  __syncthreads();
  if (pk_model(geo->physics) == JCG_PK_LINEAR) return;  // the coefficients' kernel takes fixed moments
  for (int t = warp; t < cnt; t += GR64_WARPS) {
    const double R = S.R[t];
    double* row = gi.rowd + (size_t)(n0 + t) * NROWD;
    if (S.wide) {
      if (lane < NPW + 1) {
        double s1 = 0.0, s2 = 0.0, s3 = 0.0;
        for (int i = 0; i < NKH; ++i) {
          const double y = c->kh[i] * R, y2 = y * y;
          const double p = lane == 0 ? tb->pk3v[i] : tb->pk3d[lane - 1][i];
          const double r = c->simpson_kh[i] * (p / TWO_PI2_G) * (exp(-y2) * y2);
          s1 += 2.0 * r;
          s2 += 4.0 * (r * (1.0 - y2));
          s3 += 8.0 * (r * (1.0 - 3.0 * y2 + y2 * y2));
        }
        row[lane] = s1;
        row[NPW + 1 + lane] = s2;
        if (lane == 0) row[GR64_SUMS - 1] = s3;
      }
      continue;
    }
    const FF R2 = px_split(R * R);
    float ah[GR64_SUMS], al[GR64_SUMS];  // at most 9 terms per lane
#pragma unroll
    for (int s = 0; s < GR64_SUMS; ++s) ah[s] = al[s] = 0.f;
    for (int i = lane; i < NKH; i += 32) {
      const FF y2 = px_mul(R2, px_f2(S.kh2[i]));
      if (y2.hi > 60.f) break;  // below 1e-20 of the sums from here on
      const FF e = px_exp2(-px_fix53(px_mul(y2, pxc(D_LOG2E))), S.T);
      const FF f1 = px_mul(e, y2), f2 = px_mul(f1, px_1p(FF{-y2.hi, -y2.lo}));
      // 1 - 3 y^2 + y^4 = (1 - y^2) - y^2 (2 - y^2)
      const FF f3 = px_add(f2, px_mul(px_mul(f1, y2), px_add(y2, FF{-2.f, 0.f})));
      const float2 v1 = make_float2(f1.hi, f1.lo), v2 = make_float2(f2.hi, f2.lo);
      ff_acc_prod(ah[GR64_SUMS - 1], al[GR64_SUMS - 1], S.w[0][i], make_float2(f3.hi, f3.lo));
#pragma unroll
      for (int d = 0; d <= NPW; ++d) {
        const float2 w = S.w[d][i];
        ff_acc_prod(ah[d], al[d], w, v1);
        ff_acc_prod(ah[NPW + 1 + d], al[NPW + 1 + d], w, v2);
      }
    }
#pragma unroll
    for (int s = 0; s < GR64_SUMS; ++s) S.runs[warp][s][lane] = make_float2(ah[s], al[s]);
    __syncwarp();
    if (lane < GR64_SUMS) {
      F3 tot{0.f, 0.f, 0.f};
      for (int r = 0; r < 32; ++r) px_acc3(tot, px_f2(S.runs[warp][lane][r]));
      row[lane] = px_d3(tot) * (lane <= NPW ? 2.0 : lane < GR64_SUMS - 1 ? 4.0 : 8.0);
    }
    __syncwarp();
  }
}

// NG threads per node, each NDIR / NG directions: values are repeated NG times,
// the serial chain is shorter
template <int NG>
__device__ __forceinline__ void rowfin64(const GradBatch& gb, const ConstTables* __restrict__ c, int only_wide, int block,
                                         int item) {
  const GradItem gi = grad_item(gb, item);
  const TabD* tb = gi.tab;
  if (only_wide && !tb->wide) return;
  const GeoHeader* geo = gi.geo;
  const int na = geo->na;
  const int idx = block * 64 + threadIdx.x, n_raw = idx / NG, grp = idx % NG;
  const bool live = n_raw < na;
  const int n = live ? n_raw : na - 1;  // the rest of the last warp reads and writes no row
  constexpr int ND = NDIR / NG;
  const int d0 = grp * ND;
  const int model = pk_model(geo->physics);
  double* row = gi.rowd + (size_t)n * NROWD;
  double S1 = 0.0, S2 = 0.0, S3 = 0.0, g = 0.0, S1d[ND], S2d[ND];
  int seg = 0;
  if (live) {
    S1 = row[0], S2 = row[NPW + 1], S3 = row[GR64_SUMS - 1];
#pragma unroll
    for (int q = 0; q < ND; ++q) {
      const int d = d0 + q;
      S1d[q] = d < NPW ? row[1 + d] : 0.0;
      S2d[q] = d < NPW ? row[NPW + 2 + d] : 0.0;
    }
    seg = (int)row[GR64_SUMS];
    g = row[GR64_SUMS + 1];
  }
  __syncwarp();
  if (!live) return;
  const double* s = tb->sv;
  const double a = geo_ptr<double>(geo, geo->off_a)[n];
  const int2 sg = unpack_seg(geo_ptr<int64_t>(geo, geo->off_seg_grow)[n]);
  const int2 sc = unpack_seg(geo_ptr<int64_t>(geo, geo->off_seg_chi)[n]);
  // background (background.py:53, 122-126, 168, 196, 294)
  const double lna = log(a), ia = 1.0 / a, ia2 = ia * ia, ia3 = ia2 * ia;
  const double fde = -3.0 * (1.0 + s[S_W0] + s[S_WA]) * lna + 3.0 * s[S_WA] * (a - 1.0);
  const double ef = exp(fde), ode = s[S_OMEGA_DE] * ef;
  const double ie2 = 1.0 / (s[S_OMEGA_M] * ia3 + s[S_OMEGA_K] * ia2 + ode);
  const double om_m = s[S_OMEGA_M] * ia3 * ie2, om_de = ode * ie2, w = s[S_W0] + (1.0 - a) * s[S_WA];
  const double dchi = RH * ia2 * sqrt(ie2);
  // R = 1 / k_nl
  const int ind = seg & 0xffff, j2 = ind + ((seg >> 16) ? 1 : -1);
  const double g2 = g * g, s0 = tb->sigv[ind], s1 = tb->sigv[j2];
  const double xp0 = s0 * g2, xp1 = s1 * g2, ixp = 1.0 / (xp1 - xp0);
  const double slope = (c->logr[j2] - c->logr[ind]) * ixp;
  const double Rv = exp(slope * (1.0 - xp0) + c->logr[ind]);
  const bool clipR = !(Rv >= 1e-6);
  const double R = clipR ? 1e-6 : Rv, knl = 1.0 / R;
  if (model == JCG_PK_LINEAR) {  // not used by the integrand: any moments in range
    S1 = 1.0 / g2;
    S2 = S3 = 0.0;
  }
  const double I1 = S1 * g2, I2 = S2 * g2, nf = I1 - 3.0, C = I1 * I1 + I2;
  const bool smith = model == JCG_PK_SMITH2003;
  // coefficients as 10^e with e a polynomial in n_eff, plus terms in C, om_de (1 + w)
  const double dw1 = om_de * (1.0 + w), lom = log(om_m);
  double ea, eb, ec, en, na_, nb_, nc_, nn_, ca, cb, cc, be, bn_, bc, al, an_, ac, ga, gn, gc, wa, wb;
  if (smith) {
    ea = 1.4861 + nf * (1.8369 + nf * (1.6762 + nf * (0.7940 + nf * 0.1670))), na_ = 1.8369 + nf * (2 * 1.6762 + nf * (3 * 0.7940 + nf * (4 * 0.1670))), ca = -0.6206;
    eb = 0.9463 + nf * (0.9466 + nf * 0.3084), nb_ = 0.9466 + nf * (2 * 0.3084), cb = -0.9400;
    ec = -0.2807 + nf * (0.6669 + nf * 0.3214) - 0.0793 * C, nc_ = 0.6669 + nf * (2 * 0.3214), cc = -0.0793;
    en = 0.9585 + 1.2857 * nf, nn_ = 1.2857;
    ga = 0.8649 + 0.2989 * nf + 0.1631 * C, gn = 0.2989, gc = 0.1631;
    al = 1.3884 + nf * (0.3700 - nf * 0.1452), an_ = 0.3700 - nf * (2 * 0.1452), ac = 0.0;
    be = 0.8291 + nf * (0.9854 + nf * 0.3401), bn_ = 0.9854 + nf * (2 * 0.3401), bc = 0.0;
    wa = wb = 0.0;
    ea += ca * C, eb += cb * C;
  } else {
    ea = 1.5222 + nf * (2.8553 + nf * (2.3706 + nf * (0.9903 + nf * 0.2250))), na_ = 2.8553 + nf * (2 * 2.3706 + nf * (3 * 0.9903 + nf * (4 * 0.2250))), ca = -0.6038, wa = 0.1749;
    eb = -0.5642 + nf * (0.5864 + nf * 0.5716), nb_ = 0.5864 + nf * (2 * 0.5716), cb = -1.5474, wb = 0.2279;
    ec = 0.3698 + nf * (2.0404 + nf * 0.8161) + 0.5869 * C, nc_ = 2.0404 + nf * (2 * 0.8161), cc = 0.5869;
    en = 5.2105 + 3.6902 * nf, nn_ = 3.6902;
    ga = 0.1971 - 0.0843 * nf + 0.8460 * C, gn = -0.0843, gc = 0.8460;
    al = 6.0835 + nf * (1.3373 - nf * 0.1959) - 5.5274 * C, an_ = 1.3373 - nf * (2 * 0.1959), ac = -5.5274;
    if (al < 0.0) al = -al, an_ = -an_, ac = -ac;
    be = 2.0379 + nf * (-0.7354 + nf * (0.3157 + nf * (1.2490 + nf * 0.3980))) - 0.1682 * C,
    bn_ = -0.7354 + nf * (2 * 0.3157 + nf * (3 * 1.2490 + nf * (4 * 0.3980))), bc = -0.1682;
    ea += ca * C + wa * dw1, eb += cb * C + wb * dw1;
  }
  constexpr double L10 = LN10_G;
  const double va = exp(L10 * ea), vb = exp(L10 * eb), vn = exp(L10 * en);
  const double vm = smith ? exp(L10 * (-3.5442 + 0.1908 * nf)) : 0.0;
  // f_1, f_2, ln f_3 and their partials in ln Omega_m and (smith2003) in frac
  double f1, f2, lf3, f1o, f2o, f3o, f1f = 0.0, f2f = 0.0, f3f = 0.0;
  const double io = 1.0 / (1.0 - om_m), frac = om_de * io;
  if (smith) {
    const double ofr = 1.0 - frac;
    const double a1 = exp(-0.0307 * lom), b1 = exp(-0.0732 * lom), a2 = exp(-0.0585 * lom), b2 = exp(-0.1423 * lom),
                 a3 = exp(0.0743 * lom), b3 = exp(0.0725 * lom);
    f1 = frac * a1 + ofr * b1, f1f = a1 - b1, f1o = -0.0307 * (frac * a1) - 0.0732 * (ofr * b1);
    f2 = frac * a2 + ofr * b2, f2f = a2 - b2, f2o = -0.0585 * (frac * a2) - 0.1423 * (ofr * b2);
    const double f3 = frac * a3 + ofr * b3;
    lf3 = log(f3), f3f = (a3 - b3) / f3, f3o = (0.0743 * (frac * a3) + 0.0725 * (ofr * b3)) / f3;
  } else {
    f1 = exp(-0.0307 * lom), f1o = -0.0307 * f1;
    f2 = exp(-0.0585 * lom), f2o = -0.0585 * f2;
    lf3 = 0.0743 * lom, f3o = 0.0743;
  }
  const double WSn = geo_ptr<double>(geo, geo->off_wsimp)[n];
  const double iom = 1.0 / om_m;
  double v[NA_IN];
  v[A_G] = g;
  v[A_KNL] = knl;
  v[A_BETA] = be;
  v[A_ALPHA] = al;
  v[A_AN] = va;
  v[A_BN] = vb;
  v[A_LCF3] = L10 * ec + lf3;
  v[A_F1] = f1;
  v[A_F2] = f2;
  v[A_GAM] = ga;
  v[A_NU] = vn;
  v[A_MU] = vm;
#pragma unroll 1
  for (int q = 0; q < ND; ++q) {
    const int d = d0 + q;
    const double* sd = tb->sd[d];
    const D1 chi = xfmax(interp_d1(a, c->atab_chi, tb->chiv, tb->chid[d], sc), 0.0);
    const D1 gD = xfmin(xfmax(interp_d1(a, c->atab_grow, tb->gv, tb->gd[d], sg), 0.0), 1.0);
    const double dg = gD.d[0], dg2 = 2.0 * g * dg;
    const double df = -3.0 * (sd[S_W0] + sd[S_WA]) * lna + 3.0 * sd[S_WA] * (a - 1.0);
    const double dode = (sd[S_OMEGA_DE] + s[S_OMEGA_DE] * df) * ef, dom3 = sd[S_OMEGA_M] * ia3;
    const double de2 = dom3 + sd[S_OMEGA_K] * ia2 + dode;
    const double dom = (dom3 - om_m * de2) * ie2, dde = (dode - om_de * de2) * ie2;
    const double dw = sd[S_W0] + (1.0 - a) * sd[S_WA];
    const double dx0 = tb->sigd[d][ind] * g2 + s0 * dg2, dx1 = tb->sigd[d][j2] * g2 + s1 * dg2;
    const double dlR = clipR ? 0.0 : -slope * ((dx1 - dx0) * ixp * (1.0 - xp0) + dx0);
    double dI1 = (S1d[q] + S2 * dlR) * g2 + S1 * dg2, dI2 = (S2d[q] + S3 * dlR) * g2 + S2 * dg2;
    if (model == JCG_PK_LINEAR) dI1 = dI2 = 0.0;
    const double dn = dI1, dC = 2.0 * I1 * dI1 + dI2, ddw = dde * (1.0 + w) + om_de * dw;
    const double dlo = dom * iom, dfr = smith ? (dde + frac * dom) * io : 0.0;
    const double U = WSn * dchi / xfmax(chi.v * chi.v, 1.0) / C2_G;
    double t[NA_IN];
    t[A_CHIC] = chi.v >= 1.0 ? chi.d[0] : 0.0;
    t[A_G] = dg;
    t[A_KNL] = -knl * dlR;
    t[A_BETA] = bn_ * dn + bc * dC;
    t[A_ALPHA] = an_ * dn + ac * dC;
    t[A_AN] = L10 * va * (na_ * dn + ca * dC + wa * ddw);
    t[A_BN] = L10 * vb * (nb_ * dn + cb * dC + wb * ddw);
    t[A_LCF3] = L10 * (nc_ * dn + cc * dC) + f3o * dlo + f3f * dfr;
    t[A_F1] = f1o * dlo + f1f * dfr;
    t[A_F2] = f2o * dlo + f2f * dfr;
    t[A_GAM] = gn * dn + gc * dC;
    t[A_NU] = L10 * vn * (nn_ * dn);
    t[A_MU] = L10 * vm * (0.1908 * dn);
    t[A_U] = U * (-0.5 * de2 * ie2 - (chi.v * chi.v >= 1.0 ? 2.0 * chi.d[0] / chi.v : 0.0));
    v[A_CHIC] = xfmax(chi.v, 1.0);
    v[A_U] = U;
#pragma unroll
    for (int i = 0; i < NA_IN; ++i) row[NA_IN * (1 + d) + i] = t[i];
  }
  if (grp == 0) {
#pragma unroll
    for (int i = 0; i < NA_IN; ++i) row[i] = v[i];
  }
}

// ---------------------------------------------------------------- kernels ---

constexpr int GK_WARPS = 8;
constexpr int GK_BINS = 3;             // bins per pass
constexpr int GK_SUMS = NBG + 2;       // r, A_d of the background's directions, B
constexpr int GK_PAD = 33;
struct GkSmem {
  float2 chi[NCHI], slope[NCHI];
  float2 dchi[NBG][NCHI], dslope[NBG][NCHI];
  float chi3[NCHI];
  double atab[NCHI];
  float2 runs[GK_WARPS][GK_BINS * GK_SUMS][GK_PAD];
  int exps[GK_WARPS][GK_BINS];
};

__device__ __forceinline__ void wlsum64(const GradBatch& gb, const ConstTables* __restrict__ c, int per, int only_wide,
                                        int block, int item, unsigned char* smem) {
  const GradItem gi = grad_item(gb, item);
  const TabD* tb = gi.tab;
  if (only_wide && !tb->wide) return;
  const GeoHeader* geo = gi.geo;
  const int na = geo->na, n_tr = geo->n_tr;
  const int n0 = block * per;
  if (n0 >= na || geo->n_wl == 0) return;
  GkSmem& S = *reinterpret_cast<GkSmem*>(smem);
  for (int i = threadIdx.x; i < NCHI; i += blockDim.x) {
    const int k = min(i, NCHI - 2);
    const double ida = 1.0 / (c->atab_chi[k + 1] - c->atab_chi[k]);
    const F3 a = px3_of(tb->chiv[i]);
    const FF b = px_of((tb->chiv[k + 1] - tb->chiv[k]) * ida);
    S.chi[i] = make_float2(a.hi, a.lo);
    S.chi3[i] = a.ll;
    S.slope[i] = make_float2(b.hi, b.lo);
    S.atab[i] = c->atab_chi[i];
#pragma unroll
    for (int d = 0; d < NBG; ++d) {
      const double* cd = tb->chid[bg_dir_of(d)];
      const FF e = px_of(cd[i]), f = px_of((cd[k + 1] - cd[k]) * ida);
      S.dchi[d][i] = make_float2(e.hi, e.lo);
      S.dslope[d][i] = make_float2(f.hi, f.lo);
    }
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const double* AWL = geo_ptr<double>(geo, geo->off_awl);
  const int64_t* SW = geo_ptr<int64_t>(geo, geo->off_seg_chiwl);
  const int n_end = min(na, n0 + per);
  // a warp per (node, pass of three bins)
  int passes = 0;
  for (int g = 0; g < geo->n_groups; ++g) {
    int k = 0;
    for (int t = 0; t < n_tr; ++t)
      k += geo->kind[t] == JCG_TRACER_WL && geo->group[t] == g && geo->nz_kind[t] != JCG_NZ_DELTA;
    passes += (k + GK_BINS - 1) / GK_BINS;
  }
  for (int w = warp; w < (n_end - n0) * passes; w += GK_WARPS) {
    const int n = n0 + w / passes;
    int skip = w % passes;
    const double awl = AWL[n];
    const int2 sw = unpack_seg(SW[n]);
    const D1 cw = xfmax(interp_d1(awl, c->atab_chi, tb->chiv, tb->chid[lane & 7], sw), 0.0);
    // chi of the node multiplies A in float64 where chi' > chi >= 1 at all points
    const bool far = cw.v >= 1.0;
    const FF cwp = far ? FF{1.f, 0.f} : px_of(cw.v);
    const double cwf = far ? cw.v : 1.0;
    const WlNode chiw{F3{S.chi[sw.x].x, S.chi[sw.x].y, S.chi3[sw.x]},
                      px_mul(px_f2(S.slope[min(sw.x, sw.y)]), px_split_s(awl - S.atab[sw.x]))};
    const size_t row = (size_t)n * NZP;
    for (int g = 0; g < geo->n_groups; ++g) {
      const double* AP = geo_ptr<double>(geo, geo->off_ap[g]) + row;
      const int64_t* SP = geo_ptr<int64_t>(geo, geo->off_segp[g]) + row;
      for (int t0 = 0; t0 < n_tr;) {
        // the next bins of the group
        int tl[GK_BINS], nb = 0;
        for (; t0 < n_tr && nb < GK_BINS; ++t0)
          if (geo->kind[t0] == JCG_TRACER_WL && geo->group[t0] == g && geo->nz_kind[t0] != JCG_NZ_DELTA) {
#pragma unroll
            for (int u = 0; u < GK_BINS; ++u)
              if (u == nb) tl[u] = t0;
            ++nb;
          }
        if (nb == 0) break;
        if (skip-- != 0) continue;
        int ex[GK_BINS];
        const double* W[GK_BINS];
#pragma unroll
        for (int u = 0; u < GK_BINS; ++u) {
          W[u] = geo_ptr<double>(geo, geo->off_W[tl[u < nb ? u : 0]]) + row;
          int e = 0;
          for (int j = lane; j < NZP; j += 32) e = max(e, exp_field(W[u][j]));
          ex[u] = __reduce_max_sync(0xffffffffu, e);
        }
        // lane l takes the points l, l + 32, ..: the grid is read in whole lines and
        // neighbouring lanes share table nodes
        float ah[GK_BINS][GK_SUMS], al[GK_BINS][GK_SUMS];
#pragma unroll
        for (int u = 0; u < GK_BINS; ++u)
#pragma unroll
          for (int s = 0; s < GK_SUMS; ++s) ah[u][s] = al[u][s] = 0.f;
        for (int j = lane; j < NZP; j += 32) {
          const int2 sg = unpack_seg(SP[j]);
          const int seg = min(sg.x, sg.y);
          const FF dx = px_split_s(AP[j] - S.atab[sg.x]);
          const float2 cx = S.chi[sg.x];
          const FF sd = px_mul(px_f2(S.slope[seg]), dx);
          const FF cp = px_add(px_f2(cx), sd);
          const FF df = px_add(wl_base(cx, S.chi3[sg.x], chiw), sd);
          if (df.hi <= 0.f || cp.hi <= 0.f) continue;
          FF r = df, e = FF{1.f, 0.f}, ic = e;
          if (!(cp.hi < 1.f)) {
            ic = px_rcp2(cp);
            r = px_div(df, cp);
            e = px_sqr(ic);
            if (!far) e = px_mul(e, cwp);
          }
          float2 we[GK_BINS];
#pragma unroll
          for (int u = 0; u < GK_BINS; ++u) {
            if (u >= nb) break;
            const FF w = px_split_scaled(W[u][j], ex[u]);
            const float2 wv = make_float2(w.hi, w.lo);
            ff_acc_prod(ah[u][0], al[u][0], wv, make_float2(r.hi, r.lo));
            ff_acc_prod(ah[u][GK_SUMS - 1], al[u][GK_SUMS - 1], wv, make_float2(ic.hi, ic.lo));
            const FF x = px_mul(w, e);
            we[u] = make_float2(x.hi, x.lo);
          }
#pragma unroll
          for (int d = 0; d < NBG; ++d) {
            const FF dc = px_add(px_f2(S.dchi[d][sg.x]), px_mul(px_f2(S.dslope[d][seg]), dx));
#pragma unroll
            for (int u = 0; u < GK_BINS; ++u) {
              if (u >= nb) break;
              ff_acc_prod(ah[u][1 + d], al[u][1 + d], we[u], make_float2(dc.hi, dc.lo));
            }
          }
        }
#pragma unroll
        for (int u = 0; u < GK_BINS; ++u) {
          if (u >= nb) break;
          if (lane == 0) S.exps[warp][u] = ex[u];
#pragma unroll
          for (int s = 0; s < GK_SUMS; ++s) S.runs[warp][u * GK_SUMS + s][lane] = make_float2(ah[u][s], al[u][s]);
        }
        __syncwarp();
        // lane: one of the (bin, sum) totals
        const int u = lane / GK_SUMS, s = lane - u * GK_SUMS;
        double v = 0.0;
        if (u < nb) {
          F3 tot{0.f, 0.f, 0.f};
          for (int r = 0; r < 32; ++r) px_acc3(tot, px_f2(S.runs[warp][lane][r]));
          v = scalbn(px_d3(tot), S.exps[warp][u] - 1023);
        }
        const double B = __shfl_sync(0xffffffffu, v, min(u * GK_SUMS + GK_SUMS - 1, 31));
        const double dw = __shfl_sync(0xffffffffu, cw.d[0], bg_dir_of(s > 0 && s <= NBG ? s - 1 : 0));
        if (u < nb && s <= NBG) {
          int t = tl[0];
#pragma unroll
          for (int q = 1; q < GK_BINS; ++q)
            if (q == u) t = tl[q];
          // a row with a non-finite weight: summed in float64 by the other kernel
          if (S.exps[warp][u] == 0x7ff) v = __longlong_as_double(0x7ff8000000000000LL);
          double* K = gi.kernd + ((size_t)t * na + n) * (NDIR + 1);
          if (s == 0) {
            K[0] = v;
#pragma unroll
            for (int d = 0; d < NDIR; ++d)
              if (!bg_dir(d)) K[1 + d] = 0.0;
          } else {
            K[1 + bg_dir_of(s - 1)] = cwf * v - dw * B;
          }
        }
        __syncwarp();
      }
    }
  }
}

// chi(z0) - chi over chi(z0), clipped (probes.py:53-64), or the float64 sum of a
// row whose weights are not finite
__device__ __noinline__ D1 wl_point_d1(const TabD* tb, const ConstTables* c, double a, int2 sg, int d, const D1& cw) {
  const D1 chi0 = xfmax(interp_d1(a, c->atab_chi, tb->chiv, tb->chid[d], sg), 0.0);
  return xfmax(chi0 - cw, 0.0) / xfmax(chi0, 1.0);
}
__device__ __noinline__ D1 wl_sum_d1(const TabD* tb, const ConstTables* c, const GeoHeader* geo, int t, int n, int d,
                                     const D1& cw) {
  const size_t row = (size_t)n * NZP;
  const double* AP = geo_ptr<double>(geo, geo->off_ap[geo->group[t]]) + row;
  const int64_t* SP = geo_ptr<int64_t>(geo, geo->off_segp[geo->group[t]]) + row;
  const double* W = geo_ptr<double>(geo, geo->off_W[t]) + row;
  D1 acc = mk1(0.0, 0.0);
  for (int j = 0; j < NZP; ++j) acc = acc + W[j] * wl_point_d1(tb, c, AP[j], unpack_seg(SP[j]), d, cw);
  return acc;
}

constexpr int GKF_THREADS = 64;
__device__ __forceinline__ void kernfin64(const GradBatch& gb, const ConstTables* __restrict__ c, int only_wide, int block,
                                          int t, int item) {
  const GradItem gi = grad_item(gb, item);
  const TabD* tb = gi.tab;
  if (only_wide && !tb->wide) return;
  const GeoHeader* geo = gi.geo;
  const int na = geo->na, n = block * GKF_THREADS + threadIdx.x;
  if (t >= geo->n_tr || n >= na) return;
  const double awl = geo_ptr<double>(geo, geo->off_awl)[n], z = geo_ptr<double>(geo, geo->off_z)[n];
  const bool wl = geo->kind[t] == JCG_TRACER_WL;
  const int bk = geo->bias_kind[t];
  double* K = gi.kernd + ((size_t)t * na + n) * (NDIR + 1);
  double v = 0.0, kd[NDIR];
#pragma unroll
  for (int d = 0; d < NDIR; ++d) kd[d] = 0.0;
  const double om = tb->sv[S_OMEGA_M];
  if (wl) {
    const int2 sw = unpack_seg(geo_ptr<int64_t>(geo, geo->off_seg_chiwl)[n]);
    const bool delta = geo->nz_kind[t] == JCG_NZ_DELTA;
    const double a0 = delta ? 1.0 / (1.0 + geo->nz_z0[t]) : 1.0;
    const int2 sg0 = delta ? interp_segment_inc(a0, c->atab_chi, NCHI, logspace_guess(a0, NCHI)) : make_int2(0, 1);
    const double cf = 3.0 * (H0 * H0) / 2.0 / C_KMS * (1.0 + z);  // probes.py:71, times 1 + z
    const bool f64 = !delta && isnan(K[0]);
    for (int d = 0; d < NDIR; ++d) {
      const D1 cw = xfmax(interp_d1(awl, c->atab_chi, tb->chiv, tb->chid[d], sw), 0.0);
      D1 r;
      if (delta) r = wl_point_d1(tb, c, a0, sg0, d, cw);
      else if (f64) r = wl_sum_d1(tb, c, geo, t, n, d, cw);
      else r = mk1(K[0], K[1 + d]);
      const D1 k = (cf * mk1(om, tb->sd[d][S_OMEGA_M])) * (r * cw);
      v = k.v;
      kd[d] = k.d[0];
    }
  }
  if (!wl || bk != JCG_BIAS_NONE) {
    // n(z) b(z) H(a) (probes.py:94), or the alignment term n(z) b(z) H(a)
    // (-C_1 rho_crit Omega_m / D(a)) (probes.py:102-129)
    const double nz = geo_ptr<double>(geo, geo->off_nzl)[(size_t)t * na + n];
    const double lna = geo_ptr<double>(geo, geo->off_lnawl)[n], ia = 1.0 / awl, ia2 = ia * ia, ia3 = ia2 * ia;
    const double f = -3.0 * (1.0 + tb->sv[S_W0] + tb->sv[S_WA]) * lna + 3.0 * tb->sv[S_WA] * (awl - 1.0);
    const double ef = exp(f);
    const double e2 = om * ia3 + tb->sv[S_OMEGA_K] * ia2 + tb->sv[S_OMEGA_DE] * ef;
    const double H = H0 * sqrt(e2), h2 = 0.5 / e2;
    const bool grow = wl || bk == JCG_BIAS_INV_GROWTH;
    const int2 sg = unpack_seg(geo_ptr<int64_t>(geo, geo->off_seg_growwl)[n]);
    const double b0 = geo_ptr<double>(geo, geo->off_bz)[(size_t)t * na + n];
    double bv = 0.0;
    for (int d = 0; d < NDIR; ++d) {
      const double* sd = tb->sd[d];
      const double df = -3.0 * (sd[S_W0] + sd[S_WA]) * lna + 3.0 * sd[S_WA] * (awl - 1.0);
      const double de2 = sd[S_OMEGA_M] * ia3 + sd[S_OMEGA_K] * ia2 + (sd[S_OMEGA_DE] + tb->sv[S_OMEGA_DE] * df) * ef;
      D1 k = mk1(nz * b0 * H, nz * b0 * H * (h2 * de2));
      if (grow) {
        D1 D = interp_d1(awl, c->atab_grow, tb->gv, tb->gd[d], sg);
        D = xfmin(xfmax(D, 0.0), 1.0);
        if (bk == JCG_BIAS_INV_GROWTH) k = k / D;
        if (wl) k = k * (-IA_C1_RHOCRIT * mk1(om, sd[S_OMEGA_M]) / D);
      }
      bv = k.v;
      kd[d] += k.d[0];
    }
    v += bv;
  }
  const double m = wl ? 1.0 + geo->mult[t] : 1.0;
  K[0] = v * m;
#pragma unroll
  for (int d = 0; d < NDIR; ++d) K[1 + d] = kd[d] * m;
}

// --------------------------------------------------------------- launches ---
__global__ void __launch_bounds__(GR64_WARPS * 32)
    grad_moments64_kernel(GradBatch gb, const ConstTables* __restrict__ c, int nb) {
  extern __shared__ __align__(16) unsigned char smem[];
  moments64(gb, c, nb, 0, blockIdx.x, blockIdx.y, smem);
}
template <int NG>
__global__ void __launch_bounds__(64) grad_rowfin64_kernel(GradBatch gb, const ConstTables* __restrict__ c) {
  rowfin64<NG>(gb, c, 0, blockIdx.x, blockIdx.y);
}
__global__ void __launch_bounds__(GK_WARPS * 32, 2)
    grad_wlsum64_kernel(GradBatch gb, const ConstTables* __restrict__ c, int per) {
  extern __shared__ __align__(16) unsigned char smem[];
  wlsum64(gb, c, per, 0, blockIdx.x, blockIdx.y, smem);
}
__global__ void __launch_bounds__(GKF_THREADS, 10)
    grad_kernfin64_kernel(GradBatch gb, const ConstTables* __restrict__ c) {
  kernfin64(gb, c, 0, blockIdx.x, blockIdx.y, blockIdx.z);
}
static_assert(GR64_WARPS == GK_WARPS, "one block size");
// lensing sums first: they take longer
__global__ void __launch_bounds__(GK_WARPS * 32, 2)
    grad_front64a_kernel(GradBatch gb, const ConstTables* __restrict__ c, int nb, int per, int wl_ctas, int only_wide) {
  extern __shared__ __align__(16) unsigned char smem[];
  if ((int)blockIdx.x < wl_ctas) wlsum64(gb, c, per, only_wide, blockIdx.x, blockIdx.y, smem);
  else moments64(gb, c, nb, only_wide, (int)blockIdx.x - wl_ctas, blockIdx.y, smem);
}
static_assert(GKF_THREADS == 64, "one block size");
__global__ void __launch_bounds__(GKF_THREADS)
    grad_front64b_kernel(GradBatch gb, const ConstTables* __restrict__ c, int row_ctas, int kern_ctas, int only_wide) {
  const int b = (int)blockIdx.x - row_ctas;
  if (b < 0) rowfin64<4>(gb, c, only_wide, blockIdx.x, blockIdx.y);
  else kernfin64(gb, c, only_wide, b % kern_ctas, b / kern_ctas, blockIdx.y);
}

void launch_grad_front64(const GradBatch& gb, const ConstTables* c, cudaStream_t st, int only_wide, int rows, int kern) {
  const long long sms = device_sm_count();
  // nodes per CTA: as many as pay for the tables; fewer while the CTAs do not fill the SMs
  int nb = GR64_NODES;
  while (nb > GR64_WARPS && (long long)gb.n_items * ((gb.na + nb - 1) / nb) < 2 * sms) nb >>= 1;
  int per = 32;
  const int least = gb.listed || gb.n_wl > GK_BINS ? GK_WARPS / 2 : GK_WARPS;
  while (per > least && (long long)gb.n_items * ((gb.na + per - 1) / per) < 2 * sms) per >>= 1;
  const int mom = (gb.na + nb - 1) / nb, wl = gb.listed || gb.n_wl > 0 ? (gb.na + per - 1) / per : 0;
  const int kf = (gb.na + GKF_THREADS - 1) / GKF_THREADS;
  // together while all CTAs fit the SMs at once (513 nodes, 5 + 5 bins: 61 us against
  // 83 in four launches); the cosmologies out of range (a rare case) always so
  if (only_wide || (rows && kern && gb.n_items * (long long)(mom + wl) <= 2 * sms)) {
    const size_t sm = sizeof(Gr64Smem) > sizeof(GkSmem) ? sizeof(Gr64Smem) : sizeof(GkSmem);
    allow_smem(grad_front64a_kernel, sm);
    grad_front64a_kernel<<<dim3(wl + mom, gb.n_items), GK_WARPS * 32, sm, st>>>(gb, c, nb, per, wl, only_wide);
    const int rf = (gb.na * 4 + 63) / 64;
    grad_front64b_kernel<<<dim3(rf + kf * gb.n_tr, gb.n_items), GKF_THREADS, 0, st>>>(gb, c, rf, kf, only_wide);
    return;
  }
  if (rows) {
    allow_smem(grad_moments64_kernel, sizeof(Gr64Smem));
    grad_moments64_kernel<<<dim3(mom, gb.n_items), GR64_WARPS * 32, sizeof(Gr64Smem), st>>>(gb, c, nb);
    // two directions a thread while that leaves SMs idle (513 nodes: 26 us against 60
    // for all eight), all eight from there on (61 cosmologies: 128 us against 228)
    if ((long long)gb.na * gb.n_items * 4 <= 32LL * 4 * sms)
      grad_rowfin64_kernel<4><<<dim3((gb.na * 4 + 63) / 64, gb.n_items), 64, 0, st>>>(gb, c);
    else
      grad_rowfin64_kernel<1><<<dim3((gb.na + 63) / 64, gb.n_items), 64, 0, st>>>(gb, c);
  }
  if (kern) {
    if (wl) {
      allow_smem(grad_wlsum64_kernel, sizeof(GkSmem));
      grad_wlsum64_kernel<<<dim3(wl, gb.n_items), GK_WARPS * 32, sizeof(GkSmem), st>>>(gb, c, per);
    }
    grad_kernfin64_kernel<<<dim3(kf, gb.n_tr, gb.n_items), GKF_THREADS, 0, st>>>(gb, c);
  }
}

}  // namespace jcg
