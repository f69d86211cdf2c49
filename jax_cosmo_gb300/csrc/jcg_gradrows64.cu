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
#include "jcg_grad.cuh"
#include "jcg_px_node.cuh"

namespace jcg {

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

__global__ void __launch_bounds__(GR64_WARPS * 32)
    grad_moments64_kernel(GradBatch gb, const ConstTables* __restrict__ c, int nb, int only_wide) {
  const int item = blockIdx.y;
  const GradItem gi = grad_item(gb, item);
  const TabD* tb = gi.tab;
  if (only_wide && !tb->wide) return;
  const GeoHeader* geo = gi.geo;
  const int na = geo->na, n0 = blockIdx.x * nb;
  if (n0 >= na) return;
  const int cnt = min(na - n0, nb);
  extern __shared__ __align__(16) unsigned char smem[];
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
__global__ void __launch_bounds__(64)
    grad_rowfin64_kernel(GradBatch gb, const ConstTables* __restrict__ c, int only_wide) {
  const GradItem gi = grad_item(gb, blockIdx.y);
  const TabD* tb = gi.tab;
  if (only_wide && !tb->wide) return;
  const GeoHeader* geo = gi.geo;
  const int na = geo->na;
  const int idx = blockIdx.x * 64 + threadIdx.x, n_raw = idx / NG, grp = idx % NG;
  const bool live = n_raw < na;
  const int n = live ? n_raw : na - 1;  // the rest of the last warp evaluates a valid node, writes nothing
  constexpr int ND = NDIR / NG;
  const int d0 = grp * ND;
  const int model = pk_model(geo->physics);
  double* row = gi.rowd + (size_t)n * NROWD;
  double S1 = row[0], S2 = row[NPW + 1], S3 = row[GR64_SUMS - 1], S1d[ND], S2d[ND];
#pragma unroll
  for (int q = 0; q < ND; ++q) {
    const int d = d0 + q;
    S1d[q] = d < NPW ? row[1 + d] : 0.0;
    S2d[q] = d < NPW ? row[NPW + 2 + d] : 0.0;
  }
  const int seg = (int)row[GR64_SUMS];
  const double g = row[GR64_SUMS + 1];
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

void launch_grad_rows64(const GradBatch& gb, const ConstTables* c, cudaStream_t st, int only_wide) {
  // few CTAs: fewer nodes each, so that the batch spreads over the SMs
  int nb = GR64_NODES;
  while (nb > GR64_WARPS && (long long)gb.n_items * ((gb.na + nb - 1) / nb) < 2 * device_sm_count()) nb >>= 1;
  cudaFuncSetAttribute(grad_moments64_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Gr64Smem));
  grad_moments64_kernel<<<dim3((gb.na + nb - 1) / nb, gb.n_items), GR64_WARPS * 32, sizeof(Gr64Smem), st>>>(gb, c, nb,
                                                                                                         only_wide);
  // two directions a thread while that leaves SMs idle (513 nodes: 26 us against 60
  // for all eight), all eight from there on (61 cosmologies: 128 us against 228)
  if ((long long)gb.na * gb.n_items * 4 <= 32LL * 4 * device_sm_count())
    grad_rowfin64_kernel<4><<<dim3((gb.na * 4 + 63) / 64, gb.n_items), 64, 0, st>>>(gb, c, only_wide);
  else
    grad_rowfin64_kernel<1><<<dim3((gb.na + 63) / 64, gb.n_items), 64, 0, st>>>(gb, c, only_wide);
}

}  // namespace jcg
