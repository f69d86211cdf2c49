// The Limber integral of the plain method (precision "fp64", angular_cl.py:49-98):
//
//   C_ij(l) = ef_i ef_j sum_a P_nl(k = (l + 1/2) / max(chi_a, 1), a) M_ij(a)
//
// with float64-class numbers carried on the FP32 and integer pipes
// (jcg_px.cuh: float pairs, logarithms in fixed point).  GB300 issues FP64 at
// 1/64 of FP32: the float64 form of a node was about 510 FP64 operations, and
// the FP64 pipe was its bound.  Here a node is 1,890 instructions, 33 of them
// FP64 (the sums that pairs would round most), which keeps both pipes busy: FP64
// 70%, issue slots 58% (608 cosmologies).  5 lensing bins, 100 ell, 513
// nodes: 4096 cosmologies 171.8 -> 16.5 ms; one cosmology, 2 bins, 50 ell, 257
// nodes 894 -> 26 us (clusters: seven times the CTAs).  Against 80-bit arithmetic
// on the same rows the C_ell are off by 0.6e-15 rms (float64: 0.5e-15), below
// what the tables upstream leave.
//
// k^3 is taken out of the node: with S = k^3 P / (2 pi^2) (the sum of halofit's
// two terms), P = 2 pi^2 (chi_c / (l + 1/2))^3 S, so chi_c^3 goes to the weights
// M(a) and (l + 1/2)^-3 to the result.
//
// A CTA takes a tile of ell of one cosmology and walks the a nodes in blocks
// (px_blocks of them, a function of the node count alone).  Per block: the
// rows' fixed point and pair forms and the weights M_p(a), scaled by a power
// of two per spectrum, are staged in shared memory; a thread per (a, ell) node
// evaluates S; a thread per (ell, 4 spectra) sums S M over the block in pairs
// (runs of 8 nodes, then a three-float total), and adds the block to a float64
// total.  Few CTAs (a small batch): a cluster of CTAs shares the blocks and
// adds their totals in block order through distributed shared memory, the
// same additions as one CTA makes: a result does not depend on the batch.
//
// A block in which any number leaves the range that float pairs hold (about
// 1e-30 .. 1e30), or is not finite, is evaluated in plain float64 instead.
#include <cooperative_groups.h>

#include "jcg_internal.cuh"
#include "jcg_px_node.cuh"

namespace jcg {
namespace cg = cooperative_groups;

constexpr int PX_THREADS = 256;
constexpr int PX_TB = 72;        // a nodes per block at most
constexpr int PX_MAXCL = 8;      // CTAs per cluster at most
constexpr int PX_RUN = 8;        // a nodes summed before the three-float total

__host__ __device__ inline int px_blocks(int na) { return (na + PX_TB - 1) / PX_TB; }

struct PxLayout {
  size_t tab, cos, scal, kh, l2kh, rows, m, sc, p, tot, total;
};
__host__ __device__ inline PxLayout px_layout(int n_cls, int LT, int slots) {
  PxLayout L;
  const int ncp = (n_cls + 3) & ~3;
  size_t o = 0;
  L.tab = o;
  o += sizeof(PxTab);
  L.cos = o;
  o += (sizeof(PxCos) + 15) & ~(size_t)15;
  L.scal = o;
  o += NSCAL * 8;
  L.kh = o;
  o += (size_t)LT * 8;
  L.l2kh = o;
  o += (size_t)LT * 8;
  L.rows = o;
  o += (size_t)PX_TB * PR_N * 8;
  L.sc = o;
  o += (size_t)ncp * 4;
  o = (o + 15) & ~(size_t)15;
  L.m = o;
  o += (size_t)PX_TB * ncp * 8;
  L.p = o;
  o += (size_t)PX_TB * LT * 8;
  o = (o + 15) & ~(size_t)15;
  L.tot = o;
  o += (size_t)slots * LT * ncp * 8;
  L.total = o;
  return L;
}

__device__ __forceinline__ long long px_ll(double v) { return __double2ll_rn(v); }

// slots: block totals kept per CTA; cluster CTAs share the blocks (rank r takes
// blocks r, r + R, ...)
template <bool GEN>
__global__ void __launch_bounds__(PX_THREADS, 2)
    limber64_kernel(Batch bt, const ConstTables* __restrict__ ct, int LT, int slots) {
  cg::cluster_group cl = cg::this_cluster();
  const int R = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int item = blockIdx.z;
  const Item it = batch_item(bt, item);
  const GeoHeader* geo = it.geo;
  const int n_ell = geo->n_ell, n_cls = geo->n_cls, na = geo->na;
  const int model = pk_model(it.physics);
  const bool lin = model == JCG_PK_LINEAR, nw = tf_nowiggle(it.physics);
  const int l0 = blockIdx.y * LT;
  if (l0 >= n_ell) return;  // the whole cluster returns: it shares l0
  const int lt = min(LT, n_ell - l0);
  const int ncp = (n_cls + 3) & ~3, npg = ncp >> 2;
  const PxLayout L = px_layout(bt.max_cls, LT, slots);
  extern __shared__ __align__(16) unsigned char smem[];
  PxTab& T = *reinterpret_cast<PxTab*>(smem + L.tab);
  PxCos& C = *reinterpret_cast<PxCos*>(smem + L.cos);
  double* s = reinterpret_cast<double*>(smem + L.scal);
  double* kh = reinterpret_cast<double*>(smem + L.kh);
  long long* l2kh = reinterpret_cast<long long*>(smem + L.l2kh);
  long long* rows = reinterpret_cast<long long*>(smem + L.rows);
  double* rowsd = reinterpret_cast<double*>(smem + L.rows);
  float2* rowsf = reinterpret_cast<float2*>(smem + L.rows);
  int* esc = reinterpret_cast<int*>(smem + L.sc);
  double* Md = reinterpret_cast<double*>(smem + L.m);
  float2* Mf = reinterpret_cast<float2*>(smem + L.m);
  double* Pd = reinterpret_cast<double*>(smem + L.p);
  float2* Pf = reinterpret_cast<float2*>(smem + L.p);
  double* tot = reinterpret_cast<double*>(smem + L.tot);
  __shared__ int wide_cos, wide;
  const int tid = threadIdx.x;
  const double* ELL = geo_ptr<double>(geo, geo->off_ell);
  const double* EF = geo_ptr<double>(geo, geo->off_ellfac);
  for (int i = tid; i < (int)(sizeof(PxTab) / 16); i += PX_THREADS)
    reinterpret_cast<uint4*>(&T)[i] = reinterpret_cast<const uint4*>(&ct->px)[i];
  for (int i = tid; i < NSCAL; i += PX_THREADS) s[i] = it.ctab->s[i];
  if (tid == 0) wide_cos = 0;
  __syncthreads();
  for (int l = tid; l < lt; l += PX_THREADS) {
    const double e = ELL[l0 + l] + 0.5;
    kh[l] = e;
    l2kh[l] = px_log2_d(e, T);
    if (!(e > 1e-7 && e < 1e7)) wide_cos = 1;
  }
  {
    // the cosmology's inputs, one or two per thread
    auto put = [&](F3& d, double v) {
      d = px3_of(v);
      if (!(fabs(v) < 1e12)) wide_cos = 1;
    };
    const double ish = s[S_ISH], qi = s[S_QINV];
    switch (tid) {
      case 0: C.qinv = qi; break;
      case 1: C.c1 = 1.8 * s[S_BETA_C] * qi; break;
      case 2: C.c2 = 1.8 * qi; break;
      case 3: C.cab = s[S_C142AC]; break;
      case 32: put(C.c54, (s[S_SH_D] / 5.4) * (s[S_SH_D] / 5.4)); break;
      case 33: put(C.c52, (s[S_SH_D] / 5.2) * (s[S_SH_D] / 5.2)); break;
      case 34: { const double b = s[S_BETA_B] * ish; put(C.bb3, b * b * b); break; }
      case 35: { const double b = s[S_BETA_NODE] * ish; put(C.bn3, b * b * b); break; }
      case 36: put(C.ab, s[S_ALPHA_B]); break;
      case 37: put(C.shpi, s[S_SH_D] / PI); break;
      case 38: put(C.fbp, s[S_FB] / (s[S_FC] * PI)); break;
      case 40: put(C.agam, s[S_AGAM]); break;
      case 41: put(C.oag, 1.0 - s[S_AGAM]); break;
      case 42: put(C.nwq, s[S_NWQ]); break;
      case 43: put(C.xn2, (0.43 * s[S_SH_D]) * (0.43 * s[S_SH_D])); break;
      case 64: {
        const double v = (log(69.9) - 1.08 * s[S_LGQ]) * D_LOG2E;
        C.l69 = px_ll(v * P2_53);
        if (!(fabs(v) < 400.0)) wide_cos = 1;
        break;
      }
      case 96: {
        const double v = log2(D_LOG2E) - 1.4 * s[S_LGKSILK] * D_LOG2E;
        C.lks = px_ll(v * P2_53);
        if (!(fabs(v) < 400.0)) wide_cos = 1;
        break;
      }
      case 128: {
        const double v = s[S_NS] + 3.0;
        C.ns3 = px_ll(v * P2_60);
        if (!(fabs(v) < 7.9)) wide_cos = 1;
        break;
      }
      default: break;
    }
  }
  const double fc = nw ? 1.0 : s[S_FC], fc2 = fc * fc * (1.0 / (2.0 * (PI * PI)));
  const int nblk = px_blocks(na), bsz = (na + nblk - 1) / nblk;
  const int units = lt * npg;
  __syncthreads();
  for (int b = rank; b < nblk; b += R) {
    const int base = b * bsz, nb = min(bsz, na - base);
    if (tid == 0) wide = wide_cos;
    for (int p = tid; p < ncp; p += PX_THREADS) esc[p] = 0;
    __syncthreads();
    // rows: six groups of conversions per node
    for (int q = tid; q < nb * 6; q += PX_THREADS) {
      const int grp = q / nb, t = q - grp * nb;
      const double* r = it.rows64 + (size_t)(base + t) * NROW64;
      long long* d = rows + t * PR_N;
      float2* df = rowsf + t * PR_N;
      bool ok = true;
      auto in = [&](double v, double lo, double hi) {
        ok = ok && v > lo && v < hi;
        return v;
      };
      auto three = [&](int i, double v) {
        const F3 x = px3_of(v);
        df[i] = make_float2(x.hi, x.lo);
        reinterpret_cast<float*>(df + PR_LL)[i] = x.ll;
        ok = ok && fabs(v) < 1e15;
      };
      auto expo = [&](double v) { return px_ll(in(v, -7.9, 7.9) * P2_60); };
      const double chic = fmax(r[R_CHI], 1.0);
      if (grp == 0) {
        rowsd[t * PR_N + PR_ICHIC] = 1.0 / chic;
        d[PR_L2C] = px_log2_d(in(chic, 1e-9, 1e9), T);
        rowsd[t * PR_N + PR_V] = (2.0 * (PI * PI)) * r[R_U] * (chic * chic * chic);
      } else if (grp == 1 && !lin) {
        rowsd[t * PR_N + PR_IYK] = 1.0 / (chic * r[R_KNL]);
        d[PR_L2Y] = px_log2_d(in(chic, 1e-9, 1e9), T) + px_log2_d(in(r[R_KNL], 1e-9, 1e9), T);
      } else if (grp == 2) {
        const double g = r[R_G];
        d[PR_LD] = px_log2_d(in(g * g * s[S_PKNORM] * fc2, 1e-18, 1e18), T) >> 4;
        if (!lin) {
          d[PR_BETA] = expo(r[R_BETAN]);
          three(PR_ALPHA, r[R_ALPHAN]);
        }
      } else if (grp == 3 && !lin) {
        d[PR_A0] = px_log2_d(in(r[R_AN], 1e-18, 1e18), T) >> 4;
        d[PR_E1] = expo(3.0 * r[R_F1]);
      } else if (grp == 4 && !lin) {
        d[PR_B0] = px_log2_d(in(r[R_BN], 1e-18, 1e18), T) >> 4;
        d[PR_E2] = expo(r[R_F2]);
      } else if (grp == 5 && !lin) {
        three(PR_NU, r[R_NUN]);
        three(PR_MU, r[R_MUN]);
        d[PR_E3] = expo(3.0 - r[R_GAMMAN]);
        d[PR_L3] = px_ll(in(r[R_LGCF3] * D_LOG2E, -30.0, 30.0) * P2_57);
      }
      if (!ok) wide = 1;
    }
    __syncthreads();
    // M_p(a) = K_i K_j v in float64, and each spectrum's largest exponent
    for (int q = tid; q < nb * ncp; q += PX_THREADS) {
      const int t = q / ncp, p = q - t * ncp;
      double m = 0.0;
      if (p < n_cls) {
        m = (it.kern[(size_t)geo->pair_i[p] * na + base + t] * it.kern[(size_t)geo->pair_j[p] * na + base + t]) *
            rowsd[t * PR_N + PR_V];
        const int ex = (__double2hiint(m) >> 20) & 0x7ff;
        if (ex == 0x7ff) wide = 1;
        atomicMax(esc + p, ex);
      }
      Md[q] = m;
    }
    // S at the nodes of the block
    if (!wide_cos) {
      for (int q = tid; q < nb * lt; q += PX_THREADS) {
        const int t = q / lt, l = q - t * lt;
        const FF v = px_node<GEN>(C, T, rows + t * PR_N, kh[l], l2kh[l], nw, lin);
        if (!(fabsf(v.hi) > 1e-30f && fabsf(v.hi) < 1e30f)) wide = 1;
        Pf[t * LT + l] = make_float2(v.hi, v.lo);
      }
    }
    __syncthreads();
    double* dst = tot + (R > 1 ? (size_t)(b / R) * LT * ncp : 0);
    const bool first = R > 1 || b == 0;
    if (wide) {
      // float64 nodes and sums
      for (int q = tid; q < nb * lt; q += PX_THREADS) {
        const int t = q / lt, l = q - t * lt;
        const double* r = it.rows64 + (size_t)(base + t) * NROW64;
        const double e = ELL[l0 + l] + 0.5, k = e / fmax(r[R_CHI], 1.0);
        Pd[t * LT + l] = halofit_node_lk(s, r, k, log(e) - r[R_LGCHIC], model) * (k * k * k) / (2.0 * (PI * PI));
      }
      __syncthreads();
      for (int o = tid; o < lt * n_cls; o += PX_THREADS) {
        const int l = o % lt, p = o / lt;
        double part = 0.0;
        for (int t = 0; t < nb; ++t) part += Pd[t * LT + l] * Md[t * ncp + p];
        double* w = dst + (size_t)l * ncp + p;
        *w = first ? part : *w + part;
      }
      __syncthreads();
      continue;
    }
    // M scaled to at most 2 in size, as pairs, in place
    for (int q = tid; q < nb * ncp; q += PX_THREADS) {
      const int p = q % ncp;
      const int ex = esc[p];
      double m = Md[q];
      // times 2^(1023 - ex) in two exact steps (a denormal spectrum: ex = 0)
      const int h = (1023 - ex) >> 1;
      m = m * __hiloint2double((1023 + h) << 20, 0) * __hiloint2double((1023 + (1023 - ex - h)) << 20, 0);
      const FF v = px_of(m);
      Mf[q] = make_float2(v.hi, v.lo);
    }
    __syncthreads();
    for (int u = tid; u < units; u += PX_THREADS) {
      const int pg = u / lt, l = u - pg * lt;
      F3 sum[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) sum[j] = F3{0.f, 0.f, 0.f};
      for (int t0 = 0; t0 < nb; t0 += PX_RUN) {
        float ah[4], al[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) ah[j] = al[j] = 0.f;
        const int te = min(nb, t0 + PX_RUN);
        for (int t = t0; t < te; ++t) {
          const float2 P = Pf[t * LT + l];
          const float4 m01 = *reinterpret_cast<const float4*>(Mf + t * ncp + pg * 4);
          const float4 m23 = *reinterpret_cast<const float4*>(Mf + t * ncp + pg * 4 + 2);
          ff_acc_prod(ah[0], al[0], P, make_float2(m01.x, m01.y));
          ff_acc_prod(ah[1], al[1], P, make_float2(m01.z, m01.w));
          ff_acc_prod(ah[2], al[2], P, make_float2(m23.x, m23.y));
          ff_acc_prod(ah[3], al[3], P, make_float2(m23.z, m23.w));
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) px_acc3(sum[j], px_norm(ah[j], al[j]));
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int p = pg * 4 + j;
        const int sh = esc[p] - 1023, h = sh >> 1;
        const double part = px_d3(sum[j]) * __hiloint2double((1023 + h) << 20, 0) *
                            __hiloint2double((1023 + sh - h) << 20, 0);
        double* w = dst + (size_t)l * ncp + p;
        *w = first ? part : *w + part;
      }
    }
    __syncthreads();
  }
  if (R > 1) cl.sync();
  const int nout = lt * n_cls;
  for (int o = tid + rank * PX_THREADS; o < nout; o += R * PX_THREADS) {
    const int l = o % lt, p = o / lt;
    double v;
    if (R > 1) {
      v = 0.0;
      for (int b = 0; b < nblk; ++b) {
        const double* src = cl.map_shared_rank(tot, b % R);
        const double x = src[(size_t)(b / R) * LT * ncp + (size_t)l * ncp + p];
        v = b == 0 ? x : v + x;
      }
    } else {
      v = tot[(size_t)l * ncp + p];
    }
    const int ell = l0 + l;
    const double e = ELL[ell] + 0.5;
    const double efi = EF[(size_t)geo->pair_i[p] * n_ell + ell];
    const double efj = EF[(size_t)geo->pair_j[p] * n_ell + ell];
    it.cl[(size_t)p * n_ell + ell] = v / (e * e * e) * efi * efj;
  }
  if (R > 1) cl.sync();  // no CTA leaves while its totals are read
}

template <bool GEN>
static void launch_limber64_t(const Batch& b, const ConstTables* c, cudaStream_t st) {
  const int sms = device_sm_count();
  const int nblk = px_blocks(b.max_na);
  // ell per CTA: at most 128, less while the tile does not fit twice on an SM
  auto even = [&](int lt) {
    const int tiles = (b.max_ell + lt - 1) / lt;
    return (b.max_ell + tiles - 1) / tiles;
  };
  int lt = even(128);
  while (lt > 16 && px_layout(b.max_cls, lt, 1).total > 112 * 1024) lt = even(lt / 2);
  int R = 1;
  // few CTAs: clusters over the a blocks, then smaller ell tiles
  const long long ctas = (long long)b.n_items * ((b.max_ell + lt - 1) / lt);
  if (ctas < 2 * sms) {
    R = nblk < PX_MAXCL ? nblk : PX_MAXCL;
    const int bsz = (b.max_na + nblk - 1) / nblk;
    auto count = [&](int l) { return (long long)b.n_items * ((b.max_ell + l - 1) / l) * R; };
    while (lt > 8 && count(lt) < 2 * sms) lt = even((lt + 1) / 2);
    // a node per thread in each block where clusters are small and the CTAs still fit
    // at once.  us with and without (50 ell, one cosmology): clusters of 1 24.8 and
    // 28.8, of 2 26.8 and 28.9, of 3 26.8 and 29.9, of 4 26.8 and 28.9, of 5 26.8 and
    // 30.8, of 6 26.9 and 30.9, of 7 33.0 and 30.9; of 8 34.5 and 31.4, so not there.
    // Where the CTAs come to more than one per SM it costs 2 us instead (100 ell,
    // 257 nodes: one cosmology 26.8 and 28.9, two 32.9 and 30.2)
    const int one = even(PX_THREADS / bsz > 1 ? PX_THREADS / bsz : 1);
    if (R < PX_MAXCL && one < lt && lt <= 8 && count(one) <= 2 * sms) lt = one;
    const int slots = (nblk + R - 1) / R;
    if (px_layout(b.max_cls, lt, slots).total > 220 * 1024) R = 1;
  }
  const int slots = R > 1 ? (nblk + R - 1) / R : 1;
  const PxLayout L = px_layout(b.max_cls, lt, slots);
  allow_smem(limber64_kernel<GEN>, L.total);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(R, (b.max_ell + lt - 1) / lt, b.n_items);
  cfg.blockDim = dim3(PX_THREADS);
  cfg.dynamicSmemBytes = L.total;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = R;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, limber64_kernel<GEN>, b, c, lt, slots);
}

void launch_limber64(const Batch& b, const ConstTables* c, cudaStream_t st) {
  if (b.physics_or != 0) launch_limber64_t<true>(b, c, st);
  else launch_limber64_t<false>(b, c, st);
}

}  // namespace jcg
