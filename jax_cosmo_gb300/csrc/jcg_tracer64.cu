// Tracer radial kernels and halofit rows of the plain method (precision "fp64") on
// the Limber nodes: both need the tables only, and few cosmologies run them in one
// launch.  Rows: see "halofit rows" below.  Kernels (probes.py:16-129, 188-272): for
// a WeakLensing bin
//   q(z) = simps_{z' in [z, zmax], 256}[ n(z') clip(chi' - chi, 0) / clip(chi', 1) ] (1 + z) chi
// times 3 H0^2 Omega_m / (2 c) and (1 + m), plus the NLA term; for a
// NumberCounts bin n(z) b H(z).
//
// The 257 points of the z' integral are summed in float pairs (jcg_px.cuh): in
// float64 a point and five bins were 23 operations on a pipe of 1/64 rate.  The
// cosmology-independent Simpson weights w n(z') are scaled by a power of two per
// (node, bin) to at most 2, so that a bin far below the node's redshift (weights
// of 1e-120) keeps its relative accuracy; a row with a non-finite weight is
// summed in float64.
//
// Sums are associated the same way in both kernels, runs of 8 points and then
// the runs in order, so a cosmology's kernels do not depend on its batch:
//   tracer64_uniform_kernel  lanes are 32 cosmologies, warps walk the nodes: a
//     node's grid is read and split into pairs once per 32 cosmologies;
//   tracer64_kernel          a warp per (cosmology, node), lanes are the runs:
//     ragged batches, several lensing grids, and batches too small for the
//     other (its critical path is 8 points instead of 257).
//
// 5 bins, 513 nodes, 4096 cosmologies: 30.6 -> 3.5 ms; one cosmology, 2 bins, 257
// nodes: 82 -> 15 us; 5 + 5 bins, 513 nodes: 195 -> 28 us.
#include "jcg_internal.cuh"
#include "jcg_dual.cuh"
#include "jcg_px_node.cuh"
#include "jcg_rows.cuh"
#include "jcg_wl64.cuh"

namespace jcg {

constexpr int T64_WARPS = 8;
constexpr int T64_PAD = 33;
constexpr int T64_NODES = 32;                    // nodes per CTA at most

// clip(chi' - chi, 0) / clip(chi', 1) at a' = a_x + dx on the segment (chi_x,
// slope); base = chi_x - chi
__device__ __forceinline__ FF wl_ratio(float2 cx, FF base, float2 sl, FF dx) {
  const FF sd = px_mul(px_f2(sl), dx);
  const FF cp = px_add(px_f2(cx), sd);
  const FF d = px_add(base, sd);
  if (d.hi <= 0.f || cp.hi <= 0.f) return FF{0.f, 0.f};
  if (cp.hi < 1.f) return d;
  return px_div(d, cp);
}
__device__ __forceinline__ double chi_wl_at(const CosmoTab* ct, const ConstTables* c, int2 sg, double awl) {
  return fmax(ct->chi[sg.x] + ct->chi_slope[min(sg.x, sg.y)] * (awl - c->atab_chi[sg.x]), 0.0);
}

// the z' integral of one bin in float64, for rows whose weights are not finite
__device__ __noinline__ double wl_sum_f64(const GeoHeader* geo, const CosmoTab* ct, const ConstTables* c, int t, int n,
                                          double chi_wl) {
  const size_t row = (size_t)n * NZP;
  const double* AP = geo_ptr<double>(geo, geo->off_ap[geo->group[t]]) + row;
  const int64_t* SP = geo_ptr<int64_t>(geo, geo->off_segp[geo->group[t]]) + row;
  const double* W = geo_ptr<double>(geo, geo->off_W[t]) + row;
  double acc = 0.0;
  for (int j = 0; j < NZP; ++j) {
    const int2 sg = unpack_seg(SP[j]);
    const double chip = fmax(ct->chi[sg.x] + ct->chi_slope[min(sg.x, sg.y)] * (AP[j] - c->atab_chi[sg.x]), 0.0);
    acc += W[j] * (fmax(chip - chi_wl, 0.0) / fmax(chip, 1.0));
  }
  return acc;
}

// H and the growth factor at node n (bg_H, growth_at with the geometry's logarithm
// and segment)
__device__ __forceinline__ double node_H(const GeoHeader* geo, const CosmoTab* ct, int n, double awl) {
  return H0 * sqrt(bg_esqr_l(make_bg(ct->s), awl, geo_ptr<double>(geo, geo->off_lnawl)[n], nullptr));
}
__device__ __forceinline__ double node_D(const GeoHeader* geo, const CosmoTab* ct, const ConstTables* c, int n,
                                         double awl) {
  const int2 sg = unpack_seg(geo_ptr<int64_t>(geo, geo->off_seg_growwl)[n]);
  return clip_lohi(interp_eval(awl, c->atab_grow, ct->g, sg), 0.0, 1.0);
}

// tracer t's kernel at node n from its z' integral acc; hz = H, dz = growth
// factor (used where the tracer needs them)
__device__ __forceinline__ double tracer_value(const GeoHeader* geo, const CosmoTab* ct, const ConstTables* c, int t,
                                               int n, double acc, double chi_wl, double z, double om, double hz,
                                               double dz) {
  const double nz = geo_ptr<double>(geo, geo->off_nzl)[(size_t)t * geo->na + n];
  const double b = geo->bias_kind[t] == JCG_BIAS_INV_GROWTH ? geo->bias[t] / dz
                                                            : geo_ptr<double>(geo, geo->off_bz)[(size_t)t * geo->na + n];
  if (geo->kind[t] != JCG_TRACER_WL) return nz * b * hz;
  if (geo->nz_kind[t] == JCG_NZ_DELTA) {
    // single plane (probes.py:53-64): clip(chi(z0) - chi, 0) / clip(chi(z0), 1)
    const double a0 = 1.0 / (1.0 + geo->nz_z0[t]);
    const int2 sg = interp_segment_inc(a0, c->atab_chi, NCHI, logspace_guess(a0, NCHI));
    const double chi0 = fmax(interp_eval(a0, c->atab_chi, ct->chi, sg), 0.0);
    acc = fmax(chi0 - chi_wl, 0.0) / fmax(chi0, 1.0);
  }
  double kv = 3.0 * (H0 * H0) * om / 2.0 / C_KMS * (acc * (1.0 + z) * chi_wl);  // probes.py:71
  if (geo->bias_kind[t] != JCG_BIAS_NONE) {
    // NLA intrinsic alignment (probes.py:102-129), same ell factor as the shear
    kv = kv + nz * b * hz * (-IA_C1_RHOCRIT * om / dz);
  }
  return kv * (1.0 + geo->mult[t]);
}

// ------------------------------------------------- a warp per (item, node) --
struct Tracer64Smem {
  float2 chi[NCHI], slope[NCHI];
  float chi3[NCHI];
  double atab[NCHI];
  float2 runs[T64_WARPS][T64_RUNS][MAXTR];
  int exps[T64_WARPS][MAXTR];
  double accs[MAXTR][T64_NODES], chis[T64_NODES];
};

__device__ __forceinline__ void tracer64(const Batch& bt, const ConstTables* __restrict__ c, int per, int block, int item,
                                         unsigned char* smem) {
  const Item it = batch_item(bt, item);
  const GeoHeader* geo = it.geo;
  const int na = geo->na, n_tr = geo->n_tr;
  const int n0 = block * per;
  if (n0 >= na) return;
  Tracer64Smem& S = *reinterpret_cast<Tracer64Smem*>(smem);
  auto& chi = S.chi;
  auto& slope = S.slope;
  auto& chi3 = S.chi3;
  auto& atab = S.atab;
  auto& runs = S.runs;
  auto& exps = S.exps;
  auto& accs = S.accs;
  auto& chis = S.chis;
  const CosmoTab* ct = it.ctab;
  for (int i = threadIdx.x; i < NCHI; i += blockDim.x) {
    const F3 a = px3_of(ct->chi[i]);
    const FF b = px_of(ct->chi_slope[i]);
    chi[i] = make_float2(a.hi, a.lo);
    slope[i] = make_float2(b.hi, b.lo);
    chi3[i] = a.ll;
    atab[i] = c->atab_chi[i];
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const double om = ct->s[S_OMEGA_M];
  const double* Z = geo_ptr<double>(geo, geo->off_z);
  const double* AWL = geo_ptr<double>(geo, geo->off_awl);
  const int64_t* SW = geo_ptr<int64_t>(geo, geo->off_seg_chiwl);
  const int n_end = min(na, n0 + per);
  for (int n = n0 + warp; n < n_end; n += T64_WARPS) {
    const double awl = AWL[n];
    const double chi_wl = chi_wl_at(ct, c, unpack_seg(SW[n]), awl);
    const int2 sw = unpack_seg(SW[n]);
    const WlNode chiw{F3{chi[sw.x].x, chi[sw.x].y, chi3[sw.x]},
                      px_mul(px_f2(slope[min(sw.x, sw.y)]), px_split_s(awl - atab[sw.x]))};
    const size_t row = (size_t)n * NZP;
    for (int g = 0; g < geo->n_groups; ++g) {
      const double* AP = geo_ptr<double>(geo, geo->off_ap[g]) + row;
      const int64_t* SP = geo_ptr<int64_t>(geo, geo->off_segp[g]) + row;
      // run `lane`: points 8 lane .. 8 lane + 7; the last point is run 32 (lane 0)
      FF ratio[T64_RUN], last{0.f, 0.f};
#pragma unroll
      for (int q = 0; q <= T64_RUN; ++q) {
        if (q == T64_RUN && lane != 0) break;
        const int j = q < T64_RUN ? lane * T64_RUN + q : NZP - 1;
        const int2 sg = unpack_seg(SP[j]);
        const FF r = wl_ratio(chi[sg.x], wl_base(chi[sg.x], chi3[sg.x], chiw), slope[min(sg.x, sg.y)],
                              px_split_s(AP[j] - atab[sg.x]));
        if (q < T64_RUN) ratio[q] = r;
        else last = r;
      }
      for (int t = 0; t < n_tr; ++t) {
        if (geo->kind[t] != JCG_TRACER_WL || geo->group[t] != g) continue;
        const double* W = geo_ptr<double>(geo, geo->off_W[t]) + row;
        double w[T64_RUN];
        int ex = exp_field(W[NZP - 1]);
#pragma unroll
        for (int q = 0; q < T64_RUN; ++q) w[q] = W[lane * T64_RUN + q], ex = max(ex, exp_field(w[q]));
        ex = __reduce_max_sync(0xffffffffu, ex);
        float ah = 0.f, al = 0.f;
#pragma unroll
        for (int q = 0; q < T64_RUN; ++q) {
          const FF v = px_split_scaled(w[q], ex);
          ff_acc_prod(ah, al, make_float2(v.hi, v.lo), make_float2(ratio[q].hi, ratio[q].lo));
        }
        runs[warp][lane][t] = make_float2(ah, al);
        if (lane == 0) {
          exps[warp][t] = ex;
          const FF v = px_split_scaled(W[NZP - 1], ex);
          ah = al = 0.f;
          ff_acc_prod(ah, al, make_float2(v.hi, v.lo), make_float2(last.hi, last.lo));
          runs[warp][T64_RUNS - 1][t] = make_float2(ah, al);
        }
      }
    }
    __syncwarp();
    if (lane == 0) chis[n - n0] = chi_wl;
    if (lane < n_tr) {
      const int t = lane;
      double acc = 0.0;
      if (geo->kind[t] == JCG_TRACER_WL) {
        const int ex = exps[warp][t];
        if (ex == 0x7ff) {
          acc = wl_sum_f64(geo, ct, c, t, n, chi_wl);
        } else {
          F3 tot{0.f, 0.f, 0.f};
          for (int r = 0; r < T64_RUNS; ++r) px_acc3(tot, px_f2(runs[warp][r][t]));
          acc = scalbn(px_d3(tot), ex - 1023);
        }
      }
      accs[t][n - n0] = acc;
    }
    __syncwarp();
  }
  // A thread per (tracer, node): H, the growth factor and the bias are some
  // hundred float64 operations, which cost a warp the same with one lane live as
  // with 32 (on n_tr lanes of each node's warp: 61 cosmologies, 3 + 2 bins with
  // alignment terms 838 us, now 404 us)
  __syncthreads();
  const int nn = n_end - n0;
  for (int q = threadIdx.x; q < nn * n_tr; q += blockDim.x) {
    const int t = q / nn, i = q - t * nn, n = n0 + i;
    const bool wl = geo->kind[t] == JCG_TRACER_WL;
    const double awl = AWL[n];
    double hz = 0.0, dz = 1.0;
    if (!wl || geo->bias_kind[t] != JCG_BIAS_NONE) hz = node_H(geo, ct, n, awl);
    if (geo->bias_kind[t] == JCG_BIAS_INV_GROWTH || (wl && geo->bias_kind[t] != JCG_BIAS_NONE))
      dz = node_D(geo, ct, c, n, awl);
    it.kern[(size_t)t * na + n] = tracer_value(geo, ct, c, t, n, accs[t][i], chis[i], Z[n], om, hz, dz);
  }
}

__global__ void __launch_bounds__(T64_WARPS * 32, 4)
    tracer64_kernel(Batch bt, const ConstTables* __restrict__ c, int per) {
  __shared__ __align__(16) unsigned char smem[sizeof(Tracer64Smem)];
  tracer64(bt, c, per, blockIdx.x, blockIdx.y, smem);
}

// ---------------------------------------------------------- halofit rows ----
// The float64 rows, float64-class numbers on the FP32 pipe where the work is
// (jcg_px.cuh).  Bound: issue.  The moments (power.py:121-136) take up to 257
// exponentials per node, each 35 FP64 operations in float64 (9,000 per node, on
// a pipe of 1/64 rate); a term in pairs is about 130 FP32 and integer
// instructions.  Terms with y^2 > 60 are below 1e-20 of the sums and end the
// loop (lanes walk k upwards).  The root find's decisions stay in float64.
// Phases: a thread per node (growth, chi, root find), a warp per node (the
// moments), a thread per node (coefficients, Limber weight; exponentials and
// logarithms by the pair functions, sums in float64: 230 FP64 operations where
// float64 functions made it 600).
//   4096 cosmologies x 513 nodes: 52.3 -> 3.5 ms; one cosmology: 241 -> 17 us.
constexpr int H64_NODES = 64;

// exp(v) and log of positive v by the pair functions, as doubles
__device__ __forceinline__ double px_expd(double v, const PxTab& T) {
  return px_join(px_exp2(__double2ll_rn(v * (D_LOG2E * 9007199254740992.0)), T));
}

// halofit coefficients (power.py:177-244) into a row, as halofit_coefs
__device__ void halofit_coefs64(double om_m, double om_de, double w, const HfParams& hp, double* row, int model,
                                const PxTab& T) {
  const double n = hp.neff, C = hp.C;
  row[R_KNL] = hp.knl;
  row[R_NEFF] = n;
  row[R_C] = C;
  row[R_OMM] = om_m;
  row[R_OMDE] = om_de;
  row[R_W] = w;
  if (model != JCG_PK_TAKAHASHI2012) {
    const HfCoef<double> h = hf_coefs<double>(model, n, C, om_m, om_de, w);
    row[R_AN] = h.an, row[R_BN] = h.bn, row[R_CN] = h.cn, row[R_GAMMAN] = h.gam, row[R_ALPHAN] = h.alpha;
    row[R_BETAN] = h.beta, row[R_NUN] = h.nu, row[R_MUN] = h.mu, row[R_F1] = h.f1, row[R_F2] = h.f2;
    row[R_F3] = h.f3, row[R_LGCF3] = h.lcf3;
    return;
  }
  constexpr double L10 = 2.302585092994046;
  const double dw = om_de * (1.0 + w);
  const double e_an = 1.5222 + n * (2.8553 + n * (2.3706 + n * (0.9903 + n * 0.2250))) - 0.6038 * C + 0.1749 * dw;
  const double e_bn = -0.5642 + n * (0.5864 + n * 0.5716) - 1.5474 * C + 0.2279 * dw;
  const double e_cn = 0.3698 + n * (2.0404 + n * 0.8161) + 0.5869 * C;
  row[R_AN] = px_expd(L10 * e_an, T);
  row[R_BN] = px_expd(L10 * e_bn, T);
  row[R_CN] = px_expd(L10 * e_cn, T);
  row[R_NUN] = px_expd(L10 * (5.2105 + 3.6902 * n), T);
  row[R_GAMMAN] = 0.1971 - 0.0843 * n + 0.8460 * C;
  row[R_ALPHAN] = fabs(6.0835 + n * (1.3373 - n * 0.1959) - 5.5274 * C);
  row[R_BETAN] = 2.0379 + n * (-0.7354 + n * (0.3157 + n * (1.2490 + n * 0.3980))) - 0.1682 * C;
  row[R_MUN] = 0.0;
  // Omega_m^e, e = -0.0307, -0.0585, 0.0743, which scale exponents of P(k):
  // e^x in float64 by its Taylor polynomial for |x| < 0.25 (Omega_m > 0.035)
  const double lom = (double)px_log2_d(om_m, T) * (0.69314718055994530942 / 144115188075855872.0);
  const double ex[3] = {-0.0307 * lom, -0.0585 * lom, 0.0743 * lom};
  double f[3];
  const bool small = om_m > 0.035 && om_m < 28.0;
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const double x = ex[q];
    double p = 1.0 / 479001600.0;
    p = fma(p, x, 1.0 / 39916800.0);
    p = fma(p, x, 1.0 / 3628800.0);
    p = fma(p, x, 1.0 / 362880.0);
    p = fma(p, x, 1.0 / 40320.0);
    p = fma(p, x, 1.0 / 5040.0);
    p = fma(p, x, 1.0 / 720.0);
    p = fma(p, x, 1.0 / 120.0);
    p = fma(p, x, 1.0 / 24.0);
    p = fma(p, x, 1.0 / 6.0);
    p = fma(p, x, 0.5);
    p = fma(p, x, 1.0);
    f[q] = fma(p, x, 1.0);
  }
  if (!small) {
    const double l = log(om_m);
    f[0] = exp(-0.0307 * l), f[1] = exp(-0.0585 * l), f[2] = exp(0.0743 * l);
  }
  row[R_F1] = f[0];
  row[R_F2] = f[1];
  row[R_F3] = f[2];
  row[R_LGCF3] = L10 * e_cn + (small ? ex[2] : log(f[2]));
}

struct Rows64Smem {
  PxTab T;
  double sig[NRT], s[NSCAL];
  float2 wpk[NKH], kh2[NKH];
  double knl_s[H64_NODES], inv_s[H64_NODES], lgk_s[H64_NODES], g_s[H64_NODES], chi_s[H64_NODES], s1_s[H64_NODES],
      s2_s[H64_NODES];
  int wide;
};

__device__ __forceinline__ void rows64(const Batch& bt, const ConstTables* __restrict__ c, int nb, int block, int item,
                                       unsigned char* smem) {
  const Item it = batch_item(bt, item);
  const GeoHeader* geo = it.geo;
  const int na = geo->na, n0 = block * nb;
  if (n0 >= na) return;
  const int cnt = min(na - n0, nb);
  const int model = pk_model(it.physics);
  const CosmoTab* ct = it.ctab;
  Rows64Smem& S = *reinterpret_cast<Rows64Smem*>(smem);
  PxTab& T = S.T;
  double *sig = S.sig, *s = S.s, *knl_s = S.knl_s, *inv_s = S.inv_s, *lgk_s = S.lgk_s, *g_s = S.g_s, *chi_s = S.chi_s,
         *s1_s = S.s1_s, *s2_s = S.s2_s;
  float2 *wpk = S.wpk, *kh2 = S.kh2;
  int& wide = S.wide;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for (int i = tid; i < (int)(sizeof(PxTab) / 16); i += T64_WARPS * 32)
    reinterpret_cast<uint4*>(&T)[i] = reinterpret_cast<const uint4*>(&c->px)[i];
  for (int i = tid; i < NRT; i += T64_WARPS * 32) sig[i] = ct->sig[i];
  for (int i = tid; i < NSCAL; i += T64_WARPS * 32) s[i] = ct->s[i];
  if (tid == 0) wide = 0;
  __syncthreads();
  for (int i = tid; i < NKH; i += T64_WARPS * 32) {
    const float2 w = ct->rtay[0][i];  // w_i P(k_i) k_i^3 / (2 pi^2), written by the float64 table stage
    wpk[i] = w;
    kh2[i] = make_float2(c->kh2_hi[i], c->kh2_lo[i]);
    if (!(w.x > 1e-28f && w.x < 1e28f)) wide = 1;  // outside what the pairs below hold: float64 terms
  }
  const double* A = geo_ptr<double>(geo, geo->off_a);
  const double* WS = geo_ptr<double>(geo, geo->off_wsimp);
  const int64_t* SC = geo_ptr<int64_t>(geo, geo->off_seg_chi);
  const int64_t* SG = geo_ptr<int64_t>(geo, geo->off_seg_grow);
  // growth, chi and the root find (power.py:96-118)
  for (int t = tid; t < cnt; t += T64_WARPS * 32) {
    const int n = n0 + t;
    const double a = A[n];
    const int2 sg = unpack_seg(SG[n]);
    const double sl = (ct->g[sg.y] - ct->g[sg.x]) * c->grow_ida[min(sg.x, sg.y)] * (sg.y > sg.x ? 1.0 : -1.0);
    const double g = clip_lohi(ct->g[sg.x] + sl * (a - c->atab_grow[sg.x]), 0.0, 1.0);
    const double g2 = g * g;
    int ind, j2;
    root_segment(sig, g2, ind, j2);
    const double xp = sig[ind] * g2;
    double root = c->logr[ind] + (c->logr[j2] - c->logr[ind]) / (sig[j2] * g2 - xp) * (1.0 - xp);
    double R = exp(root);
    if (!(R >= 1e-6)) R = R < 1e-6 ? 1e-6 : R, root = log(R);  // power.py:113-115
    g_s[t] = g;
    inv_s[t] = R;
    knl_s[t] = 1.0 / R;
    lgk_s[t] = -root;
    chi_s[t] = chi_at(ct, c, a, unpack_seg(SC[n]));
    if (!(R < 1e6)) wide = 1;
  }
  __syncthreads();
  // the moments
  if (model != JCG_PK_LINEAR) {
    for (int t = warp; t < cnt; t += T64_WARPS) {
      double s1, s2;
      const double R = inv_s[t];
      if (!wide) {
        const FF R2 = px_split(R * R);
        FF a1{0.f, 0.f}, a2{0.f, 0.f};  // at most 9 terms per lane
        for (int i = lane; i < NKH; i += 32) {
          const FF y2 = px_mul(R2, px_f2(kh2[i]));
          if (y2.hi > 60.f) break;
          const FF e = px_exp2(-px_fix53(px_mul(y2, pxc(D_LOG2E))), T);
          const FF r = px_mul(px_mul(px_f2(wpk[i]), e), y2);
          a1 = px_add(a1, r);
          a2 = px_add(a2, px_mul(r, px_1p(FF{-y2.hi, -y2.lo})));
        }
        __syncwarp();
        s1 = 2.0 * warp_sum(px_join(a1));
        s2 = 4.0 * warp_sum(px_join(a2));
      } else {
        s1 = s2 = 0.0;
        for (int i = lane; i < NKH; i += 32) {
          const double y = c->kh[i] * R, y2 = y * y;
          const double r = ct->pk3[i] * exp(-y2) / TWO_PI2;
          s1 += c->simpson_kh[i] * (2 * r * y2);
          s2 += c->simpson_kh[i] * (4 * r * (y2 - y2 * y2));
        }
        s1 = warp_sum(s1);
        s2 = warp_sum(s2);
      }
      if (lane == 0) s1_s[t] = s1, s2_s[t] = s2;
    }
  }
  __syncthreads();
  // coefficients and the Limber weight
  for (int t = tid; t < cnt; t += T64_WARPS * 32) {
    const int n = n0 + t;
    const double a = A[n], g2 = g_s[t] * g_s[t];
    double row[NROW64];
    for (int i = 0; i < NROW64; ++i) row[i] = 0.0;
    // background (background.py:122-126, 168, 196, 270-294)
    const double ia = px_ddiv(1.0, a, px_rcp(px_hi(a)));
    const double lna = (double)px_log2_d(a, T) * (0.69314718055994530942 / 144115188075855872.0);
    const double fde = -3.0 * (1.0 + s[S_W0] + s[S_WA]) * lna + 3.0 * s[S_WA] * (a - 1.0);
    const double ef = fde == 0.0 ? 1.0 : exp(fde);
    const double ia2 = ia * ia, om3 = s[S_OMEGA_M] * (ia2 * ia), ode = s[S_OMEGA_DE] * ef;
    const double e2 = om3 + s[S_OMEGA_K] * ia2 + ode;
    const double ie2 = 1.0 / e2;
    const double chi = chi_s[t], dchi = RH * ia2 * rsqrt(e2);
    HfParams hp;
    hp.knl = knl_s[t];
    const double s1 = model == JCG_PK_LINEAR ? 0.0 : s1_s[t] * g2;
    hp.neff = s1 - 3.0;  // power.py:138-139
    hp.C = model == JCG_PK_LINEAR ? 0.0 : s1 * s1 + s2_s[t] * g2;
    halofit_coefs64(om3 * ie2, ode * ie2, s[S_W0] + (1.0 - a) * s[S_WA], hp, row, model, T);
    row[R_CHI] = chi;
    row[R_G] = g_s[t];
    row[R_LGKNL] = lgk_s[t];
    row[R_LGCHIC] = log(fmax(chi, 1.0));
    row[R_DCHI] = dchi;
    row[R_U] = WS[n] * dchi / fmax(chi * chi, 1.0) * (1.0 / C2);
    double* dst = it.rows64 + (size_t)n * NROW64;
    for (int i = 0; i < NROW64; ++i) dst[i] = row[i];
  }
}

__global__ void __launch_bounds__(T64_WARPS * 32, 5)
    halofit_rows64_kernel(Batch bt, const ConstTables* __restrict__ c, int nb) {
  __shared__ __align__(16) unsigned char smem[sizeof(Rows64Smem)];
  rows64(bt, c, nb, blockIdx.x, blockIdx.y, smem);
}

// Rows and kernels need the tables only: few cosmologies run both in one launch,
// CTAs of either kind side by side.
__global__ void __launch_bounds__(T64_WARPS * 32, 4)
    rows_tracer64_kernel(Batch bt, const ConstTables* __restrict__ c, int nb, int per, int row_ctas) {
  __shared__ __align__(16) unsigned char
      smem[sizeof(Tracer64Smem) > sizeof(Rows64Smem) ? sizeof(Tracer64Smem) : sizeof(Rows64Smem)];
  if ((int)blockIdx.x < row_ctas) rows64(bt, c, nb, blockIdx.x, blockIdx.y, smem);
  else tracer64(bt, c, per, (int)blockIdx.x - row_ctas, blockIdx.y, smem);
}

// --------------------------------------------- lanes over 32 cosmologies ----
template <int NW>
struct T64Rec {
  int q;        // chi table node | segment << 16
  int flags;    // 1: some weight of the point is not 0; 2: q differs from the point before
  float2 dx, w[NW];
};
__host__ __device__ inline size_t t64_tab_bytes(int wn) { return ((size_t)wn * T64_PAD * 20 + 15) & ~(size_t)15; }

template <int NW>
__global__ void __launch_bounds__(T64_WARPS * 32, 3)
    tracer64_uniform_kernel(Batch bt, const ConstTables* __restrict__ c, int per) {
  const GeoHeader* geo = bt.geo;
  const int na = geo->na, n_tr = geo->n_tr;
  const int n0 = blockIdx.x * per, c0 = blockIdx.y * 32;
  extern __shared__ __align__(16) unsigned char tsm[];
  const int wbase = bt.chi_wbase, wn = NCHI - wbase;
  float2* chiT = reinterpret_cast<float2*>(tsm);  // [wn][T64_PAD]
  float2* slT = chiT + wn * T64_PAD;
  float* c3T = reinterpret_cast<float*>(slT + wn * T64_PAD);
  T64Rec<NW>* recs = reinterpret_cast<T64Rec<NW>*>(tsm + t64_tab_bytes(wn));  // [8][32]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for (int idx = tid; idx < 32 * wn; idx += blockDim.x) {
    const int cc = idx / wn, sidx = idx % wn;
    F3 a{0.f, 0.f, 0.f};
    FF b{0.f, 0.f};
    if (c0 + cc < bt.n_items) {
      a = px3_of(bt.ctab[c0 + cc].chi[wbase + sidx]);
      b = px_of(bt.ctab[c0 + cc].chi_slope[wbase + sidx]);
    }
    chiT[sidx * T64_PAD + cc] = make_float2(a.hi, a.lo);
    slT[sidx * T64_PAD + cc] = make_float2(b.hi, b.lo);
    c3T[sidx * T64_PAD + cc] = a.ll;
  }
  __syncthreads();
  const int ci = c0 + lane;
  const bool live = ci < bt.n_items;
  const CosmoTab* ct = bt.ctab + (live ? ci : c0);
  const double om = ct->s[S_OMEGA_M];
  double* kern = bt.kern + (size_t)(live ? ci : c0) * bt.max_tr * na;
  const double* Z = geo_ptr<double>(geo, geo->off_z);
  const double* AWL = geo_ptr<double>(geo, geo->off_awl);
  const int64_t* SW = geo_ptr<int64_t>(geo, geo->off_seg_chiwl);
  int wl_t[NW];
  {
    int u = 0;
    for (int t = 0; t < n_tr && u < NW; ++t)
      if (geo->kind[t] == JCG_TRACER_WL) wl_t[u++] = t;
  }
  T64Rec<NW>* rec = recs + warp * 32;
  const int n_end = min(na, n0 + per);
  for (int n = n0 + warp; n < n_end; n += T64_WARPS) {
    const double awl = AWL[n];
    const double chi_wl = chi_wl_at(ct, c, unpack_seg(SW[n]), awl);
    const int2 sw = unpack_seg(SW[n]);
    const int xw = (sw.x - wbase) * T64_PAD + lane;
    const WlNode chiw{F3{chiT[xw].x, chiT[xw].y, c3T[xw]},
                      px_mul(px_f2(slT[(min(sw.x, sw.y) - wbase) * T64_PAD + lane]),
                             px_split_s(awl - c->atab_chi[sw.x]))};
    const size_t row = (size_t)n * NZP;
    const double* AP = geo_ptr<double>(geo, geo->off_ap[0]) + row;
    const int64_t* SP = geo_ptr<int64_t>(geo, geo->off_segp[0]) + row;
    int ex[NW];
#pragma unroll
    for (int u = 0; u < NW; ++u) {
      const double* W = geo_ptr<double>(geo, geo->off_W[wl_t[u]]) + row;
      int e = 0;
      for (int j = lane; j < NZP; j += 32) e = max(e, exp_field(W[j]));
      ex[u] = __reduce_max_sync(0xffffffffu, e);
    }
    F3 tot[NW];
#pragma unroll
    for (int u = 0; u < NW; ++u) tot[u] = F3{0.f, 0.f, 0.f};
    for (int j0 = 0; j0 < NZP; j0 += 32) {
      const int j = j0 + lane;
      int q = -1;
      if (j < NZP) {
        const int2 sg = unpack_seg(SP[j]);
        q = (sg.x - wbase) | ((min(sg.x, sg.y) - wbase) << 16);
        const FF dx = px_split_s(AP[j] - c->atab_chi[sg.x]);
        rec[lane].q = q;
        rec[lane].dx = make_float2(dx.hi, dx.lo);
        bool any = false;
#pragma unroll
        for (int u = 0; u < NW; ++u) {
          const FF v = px_split_scaled(geo_ptr<double>(geo, geo->off_W[wl_t[u]])[row + j], ex[u]);
          rec[lane].w[u] = make_float2(v.hi, v.lo);
          any |= v.hi != 0.f;
        }
        rec[lane].flags = any;
      }
      const int qp = __shfl_up_sync(0xffffffffu, q, 1);
      if (j < NZP && (lane == 0 || qp != q)) rec[lane].flags |= 2;
      __syncwarp();
      const int cnt = min(32, NZP - j0);
      float2 cx = make_float2(0.f, 0.f), sl = cx;
      FF base{0.f, 0.f};
      for (int r0 = 0; r0 < cnt; r0 += T64_RUN) {
        float ah[NW], al[NW];
#pragma unroll
        for (int u = 0; u < NW; ++u) ah[u] = al[u] = 0.f;
        const int re = min(cnt, r0 + T64_RUN);
        for (int jj = r0; jj < re; ++jj) {
          const int fl = rec[jj].flags;  // the same for the warp
          if (fl & 2) {
            const int q = rec[jj].q, x = (q & 0xffff) * T64_PAD + lane;
            cx = chiT[x];
            sl = slT[(q >> 16) * T64_PAD + lane];
            base = wl_base(cx, c3T[x], chiw);
          }
          if (!(fl & 1)) continue;  // the sums would not change
          const FF r = wl_ratio(cx, base, sl, px_f2(rec[jj].dx));
#pragma unroll
          for (int u = 0; u < NW; ++u) ff_acc_prod(ah[u], al[u], rec[jj].w[u], make_float2(r.hi, r.lo));
        }
#pragma unroll
        for (int u = 0; u < NW; ++u) px_acc3(tot[u], FF{ah[u], al[u]});
      }
      __syncwarp();
    }
    if (live) {
      double hz = 0.0, dz = 1.0;
      if (geo->n_nc > 0 || geo->special_bias) hz = node_H(geo, ct, n, awl);
      if (geo->special_bias) dz = node_D(geo, ct, c, n, awl);
      const double z = Z[n];
#pragma unroll
      for (int u = 0; u < NW; ++u) {
        const int t = wl_t[u];
        const double acc = ex[u] == 0x7ff ? wl_sum_f64(geo, ct, c, t, n, chi_wl) : scalbn(px_d3(tot[u]), ex[u] - 1023);
        kern[(size_t)t * na + n] = tracer_value(geo, ct, c, t, n, acc, chi_wl, z, om, hz, dz);
      }
      for (int t = 0; t < n_tr; ++t)
        if (geo->kind[t] != JCG_TRACER_WL)
          kern[(size_t)t * na + n] = tracer_value(geo, ct, c, t, n, 0.0, chi_wl, z, om, hz, dz);
    }
  }
}

// nodes per CTA: T64_NODES pay for the table loads; fewer while the CTAs do not fill the SMs
static int t64_nodes(int na, int rows) {
  int per = T64_NODES;
  while (per > T64_WARPS && (long long)rows * ((na + per - 1) / per) < 2 * device_sm_count()) per >>= 1;
  return per;
}

template <int NW>
static void launch_t64u(const Batch& b, const ConstTables* c, cudaStream_t st) {
  const size_t smem = t64_tab_bytes(NCHI - b.chi_wbase) + sizeof(T64Rec<NW>) * T64_WARPS * 32;
  allow_smem(tracer64_uniform_kernel<NW>, smem);
  const int groups = (b.n_items + 31) / 32;
  const int per = t64_nodes(b.max_na, groups);
  tracer64_uniform_kernel<NW><<<dim3((b.max_na + per - 1) / per, groups), T64_WARPS * 32, smem, st>>>(b, c, per);
}

void launch_tracer64(const Batch& b, const ConstTables* c, cudaStream_t st) {
  // lanes over cosmologies from 96 on: for few, idle lanes and SMs and its chains of
  // 257 points cost more than the other form's repeated reads of the grid.  us, a warp
  // per node / lanes over cosmologies (513 nodes, then 257):
  //   3 bins, 24 cosmologies  127 /  97,   68 /  96    5 bins, 24  176 / 128,   92 / 128
  //           96              442 / 125,  247 /  94            96  621 / 160,  346 / 126
  // so the forms cross between 20 and 40 cosmologies; the line lies above that
  if (!b.listed && b.n_wl_groups == 1 && b.n_wl >= 1 && b.n_wl <= 8 && b.n_items >= 96) {
    switch (b.n_wl) {
      case 1: launch_t64u<1>(b, c, st); return;
      case 2: launch_t64u<2>(b, c, st); return;
      case 3: launch_t64u<3>(b, c, st); return;
      case 4: launch_t64u<4>(b, c, st); return;
      case 5: launch_t64u<5>(b, c, st); return;
      case 6: launch_t64u<6>(b, c, st); return;
      case 7: launch_t64u<7>(b, c, st); return;
      default: launch_t64u<8>(b, c, st); return;
    }
  }
  const int per = t64_nodes(b.max_na, b.n_items);
  tracer64_kernel<<<dim3((b.max_na + per - 1) / per, b.n_items), T64_WARPS * 32, 0, st>>>(b, c, per);
}

// rows per CTA: as many as pay for the tables; fewer while the CTAs do not fill the SMs
static int rows64_nodes(const Batch& b) {
  int nb = H64_NODES;
  while (nb > 8 && (long long)b.n_items * ((b.max_na + nb - 1) / nb) < 2 * device_sm_count()) nb >>= 1;
  return nb;
}
void launch_rows64(const Batch& b, const ConstTables* c, cudaStream_t st) {
  const int nb = rows64_nodes(b);
  halofit_rows64_kernel<<<dim3((b.max_na + nb - 1) / nb, b.n_items), T64_WARPS * 32, 0, st>>>(b, c, nb);
}

void launch_rows_tracers(const Batch& b, const ConstTables* c, cudaStream_t st) {
  if (b.precision != JCG_FP32C) {
    const int nb = rows64_nodes(b), per = t64_nodes(b.max_na, b.n_items);
    const int rows = (b.max_na + nb - 1) / nb, tr = (b.max_na + per - 1) / per;
    // while all CTAs fit the SMs at once, two each (257 nodes, 2 bins: 17 us
    // against 17 + 16; 513 nodes, 10 tracers: 34 against 22 + 27)
    if ((long long)b.n_items * (rows + tr) <= 2 * device_sm_count()) {
      rows_tracer64_kernel<<<dim3(rows + tr, b.n_items), T64_WARPS * 32, 0, st>>>(b, c, nb, per, rows);
      return;
    }
  }
  launch_halofit_rows(b, c, st);
  launch_tracer_kernels(b, c, st);
}

}  // namespace jcg
