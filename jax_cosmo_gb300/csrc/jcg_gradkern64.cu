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
#include "jcg_grad.cuh"
#include "jcg_px.cuh"
#include "jcg_wl64.cuh"

namespace jcg {

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

__global__ void __launch_bounds__(GK_WARPS * 32, 2)
    grad_wlsum64_kernel(GradBatch gb, const ConstTables* __restrict__ c, int per, int only_wide) {
  const GradItem gi = grad_item(gb, blockIdx.y);
  const TabD* tb = gi.tab;
  if (only_wide && !tb->wide) return;
  const GeoHeader* geo = gi.geo;
  const int na = geo->na, n_tr = geo->n_tr;
  const int n0 = blockIdx.x * per;
  if (n0 >= na || geo->n_wl == 0) return;
  extern __shared__ __align__(16) unsigned char smem[];
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
__global__ void __launch_bounds__(GKF_THREADS, 10)
    grad_kernfin64_kernel(GradBatch gb, const ConstTables* __restrict__ c, int only_wide) {
  const GradItem gi = grad_item(gb, blockIdx.z);
  const TabD* tb = gi.tab;
  if (only_wide && !tb->wide) return;
  const GeoHeader* geo = gi.geo;
  const int na = geo->na, t = blockIdx.y, n = blockIdx.x * GKF_THREADS + threadIdx.x;
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

void launch_grad_kern64(const GradBatch& gb, const ConstTables* c, cudaStream_t st, int only_wide) {
  // nodes per CTA: 32 pay for the tables; fewer while the CTAs do not fill the SMs
  int per = 32;
  const int least = gb.listed || gb.n_wl > GK_BINS ? GK_WARPS / 2 : GK_WARPS;
  while (per > least && (long long)gb.n_items * ((gb.na + per - 1) / per) < 2 * device_sm_count()) per >>= 1;
  if (gb.listed || gb.n_wl > 0) {
    cudaFuncSetAttribute(grad_wlsum64_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(GkSmem));
    grad_wlsum64_kernel<<<dim3((gb.na + per - 1) / per, gb.n_items), GK_WARPS * 32, sizeof(GkSmem), st>>>(gb, c, per,
                                                                                                       only_wide);
  }
  grad_kernfin64_kernel<<<dim3((gb.na + GKF_THREADS - 1) / GKF_THREADS, gb.n_tr, gb.n_items), GKF_THREADS, 0, st>>>(
      gb, c, only_wide);
}

}  // namespace jcg
