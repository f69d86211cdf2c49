// Tracer radial kernels of the plain method (precision "fp64") on the Limber
// nodes (probes.py:16-129, 188-272): for a WeakLensing bin
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
__global__ void __launch_bounds__(T64_WARPS * 32, 4)
    tracer64_kernel(Batch bt, const ConstTables* __restrict__ c, int per) {
  const Item it = batch_item(bt, blockIdx.y);
  const GeoHeader* geo = it.geo;
  const int na = geo->na, n_tr = geo->n_tr;
  const int n0 = blockIdx.x * per;
  if (n0 >= na) return;
  __shared__ float2 chi[NCHI], slope[NCHI];
  __shared__ float chi3[NCHI];
  __shared__ double atab[NCHI];
  __shared__ float2 runs[T64_WARPS][T64_RUNS][MAXTR];
  __shared__ int exps[T64_WARPS][MAXTR];
  __shared__ double accs[MAXTR][T64_NODES], chis[T64_NODES];
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
  cudaFuncSetAttribute(tracer64_uniform_kernel<NW>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  const int groups = (b.n_items + 31) / 32;
  const int per = t64_nodes(b.max_na, groups);
  tracer64_uniform_kernel<NW><<<dim3((b.max_na + per - 1) / per, groups), T64_WARPS * 32, smem, st>>>(b, c, per);
}

void launch_tracer64(const Batch& b, const ConstTables* c, cudaStream_t st) {
  // lanes over cosmologies from 96 on (3 bins, 513 nodes: 61 cosmologies take
  // 104 us a warp per node and 434 us with lanes over cosmologies; 4096 about 7 ms
  // and, 5 bins, 3.5 ms): below, idle SMs and 257-point chains cost more than
  // the other form's repeated reads of the grid
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

}  // namespace jcg
