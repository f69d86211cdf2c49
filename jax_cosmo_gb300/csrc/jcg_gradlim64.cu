// The Limber integral of the float64 gradient: C_ell and its 8 tangents,
//
//   C_ij(l) = ef_i ef_j / (l + 1/2)^3 sum_a S(a, l) K_i(a) K_j(a) V(a)
//
// with S of jcg_px_grad.cuh and V = 2 pi^2 u chi_c^3, all in float pairs on the
// FP32 pipe (the float64 form is bound by GB300's FP64 rate, 1/64 of FP32).
//
//   grad_scale64_kernel   per tracer the power of two that brings its kernel to
//     at most 2 in size; the transfer function's inputs and tangents;
//   grad_pack64_kernel    the rows and kernels, in place, as the fixed point
//     numbers and pairs the nodes read;
//   grad_limber64_kernel  the integral.
// Tangents that are 0 by the nature of the input (background inputs in the
// directions of h, n_s and sigma_8) are neither read nor multiplied.
//
// A CTA takes a tile of LT ell and a range of the a nodes of one cosmology.  Per
// chunk of TA nodes: a thread per (a, ell) node evaluates S and its tangents into
// shared memory; then, in blocks of MB nodes, the weights M_p = K_i K_j V with
// tangents are formed from the kernels, and a thread per (spectrum, ell) adds
// the 14 products of its value and tangents in pairs and adds the block to
// three-float totals.
//
// 10 tracers (55 spectra), 200 ell, 513 nodes, one cosmology: 1,195 -> 161 us and
// 22 us for the two packing kernels; 61 cosmologies, 15 spectra, 97 ell: 14.6 ->
// 1.63 ms and 0.15 (with the zero tangents 178 us and 1.81 ms).  Bound by the
// latency of FP32 chains (7,700 instructions a node, 190 per spectrum and node; 4
// warps per scheduler at 128 registers, 0.4 to 0.5 instructions per cycle; three
// CTAs an SM spill: slower).  Three-float totals in the node and runs of 4 nodes
// cost 20% of that and bring the tangents' error, which cancelling terms amplify,
// below the float64 kernels' on the former tables (1.5e-15 and 2.4e-15 of their
// norm against 1.6e-15 and 2.8e-15, by 80-bit arithmetic).
//
// Numbers out of the range that float pairs hold, or a spectrum that lives where
// its kernels are below 2^-66 of their largest value, set TabD::wide: that
// cosmology is then computed by the float64 kernels instead.
#include "jcg_grad.cuh"
#include "jcg_px_grad.cuh"

namespace jcg {

constexpr int GX_THREADS = 256;
static_assert(GR_T + GT_N * NDIR <= NROWD, "a packed row takes the float64 row's place");

// the transfer function's inputs and the kernels' exponents: in the part of TabD
// that the tables' node scratch has left
struct GxScratch {
  GxTabs g;
  int kexp[1];
};
__device__ __forceinline__ GxScratch* gx_scratch(TabD* t) { return reinterpret_cast<GxScratch*>(&t->c32[0][0]); }
static_assert(offsetof(TabD, c32) % 8 == 0, "alignment");

constexpr int GXS_THREADS = 256;
__global__ void __launch_bounds__(GXS_THREADS) grad_scale64_kernel(GradBatch gb) {
  const GradItem gi = grad_item(gb, blockIdx.y);
  const GeoHeader* geo = gi.geo;
  const int t = threadIdx.x, i = blockIdx.x, n_tr = geo->n_tr, na = geo->na, n_cls = geo->n_cls;
  if (i > n_tr) return;
  TabD* tb = gi.tab;
  GxScratch* sc = gx_scratch(tb);
  if (i < n_tr) {
    __shared__ unsigned mx;
    if (t == 0) mx = 0;
    __syncthreads();
    const double* K = gi.kernd + (size_t)i * na * (NDIR + 1);
    unsigned m = 0;
    bool bad = false;
    for (int n = t; n < na; n += GXS_THREADS) {
      const double* r = K + (size_t)n * (NDIR + 1);
      const unsigned e = (unsigned)__double2hiint(r[0]) & 0x7fffffffu;
      m = max(m, e);
      for (int d = 1; d <= NDIR; ++d) bad |= !(fabs(r[d]) < 1e300);
    }
    atomicMax(&mx, m);
    __syncthreads();
    const int ex = (int)(mx >> 20);
    bad |= ex == 0x7ff || (ex != 0 && (ex < 64 || ex > 1983));
    // the exponent of an all-zero kernel is that of 1 (its tangents may not be 0)
    if (t == 0) sc->kexp[i] = ex == 0 ? 1023 : ex;
    // a warp per spectrum of the tracer
    for (int p = 0, k = 0; p < n_cls; ++p) {
      if (geo->pair_i[p] != i) continue;
      if ((k++ & (GXS_THREADS / 32 - 1)) != (t >> 5)) continue;
      const double* Kj = gi.kernd + (size_t)geo->pair_j[p] * na * (NDIR + 1);
      unsigned q = 0, qj = 0;
#pragma unroll 4
      for (int n = t & 31; n < na; n += 32) {
        const double kj = Kj[(size_t)n * (NDIR + 1)];
        q = max(q, (unsigned)__double2hiint(K[(size_t)n * (NDIR + 1)] * kj) & 0x7fffffffu);
        qj = max(qj, (unsigned)__double2hiint(kj) & 0x7fffffffu);
      }
      const unsigned ep = __reduce_max_sync(0xffffffffu, q) >> 20, ej = __reduce_max_sync(0xffffffffu, qj) >> 20;
      // largest product below 2^-66 of the product of the largest: not for pairs
      if (ep != 0 && (int)ep - ex - ((int)ej - 1023) < -66) bad = true;
    }
    if (bad) tb->wide = 1;
    return;
  }
  // the cosmology's inputs
  const double* s = tb->sv;
  PxCos& C = sc->g.c;
  bool bad = false;
  auto put = [&](F3& d, double v) {
    d = px3_of(v);
    bad |= !(fabs(v) < 1e12);
  };
  const double ish = 1.0 / s[S_SH_D], qi = 1.0 / (13.41 * s[S_K_EQ]);
  const bool nw = s[S_TFNW] != 0.0;
  switch (t) {
    case 0:
      C.qinv = qi;
      C.c1 = 1.8 * s[S_BETA_C] * qi;
      C.c2 = 1.8 * qi;
      break;
    case 8:
      C.cab = 14.2 / s[S_ALPHA_C];
      put(sc->g.cab, 14.2 / s[S_ALPHA_C]);
      break;
    case 32: put(C.c54, (s[S_SH_D] / 5.4) * (s[S_SH_D] / 5.4)); break;
    case 40: put(C.c52, (s[S_SH_D] / 5.2) * (s[S_SH_D] / 5.2)); break;
    case 64: { const double b = s[S_BETA_B] * ish; put(C.bb3, b * b * b); break; }
    case 72: { const double b = s[S_BETA_NODE] * ish; put(C.bn3, b * b * b); break; }
    case 96: put(C.ab, s[S_ALPHA_B]); break;
    case 104: put(C.shpi, s[S_SH_D] / PI); break;
    case 112: put(C.fbp, s[S_FB] / (s[S_FC] * PI)); break;
    case 128: put(C.agam, s[S_AGAM]); break;
    case 132: put(C.oag, 1.0 - s[S_AGAM]); break;
    case 136: put(C.nwq, s[S_NWQ]); break;
    case 140: put(C.xn2, (0.43 * s[S_SH_D]) * (0.43 * s[S_SH_D])); break;
    case 160: {
      const double v = (log(69.9) - 1.08 * s[S_LGQ]) * D_LOG2E;
      C.l69 = __double2ll_rn(v * P2_53);
      bad |= !(fabs(v) < 400.0);
      break;
    }
    case 164: {
      const double v = log2(D_LOG2E) - 1.4 * s[S_LGKSILK] * D_LOG2E;
      C.lks = __double2ll_rn(v * P2_53);
      bad |= !(fabs(v) < 400.0);
      break;
    }
    case 168: {
      const double v = s[S_NS] + 3.0;
      C.ns3 = __double2ll_rn(v * P2_60);
      bad |= !(fabs(v) < 7.9);
      break;
    }
    default: break;
  }
  // type "eisenhu" leaves the inputs of the other fit out of its result
  if (nw && t < 128) bad = false;
  if (t >= 192 && t < 192 + GC_N * 4) {
    const int x = (t - 192) >> 2, d = (t - 192) & 3;
    constexpr int X[GC_N] = {S_SH_D,     S_K_EQ,   S_BETA_C,    S_ALPHA_C, S_ALPHA_B,
                             S_BETA_B, S_BETA_NODE, S_K_SILK,  S_FB,     S_FC};
    int si = 0;
#pragma unroll
    for (int q = 0; q < GC_N; ++q)
      if (q == x) si = X[q];
    if (nw && x == GC_AGAM) si = S_AGAM;
    if (nw && x == GC_NWQ) si = S_NWQ;
    const double dv = d < 3 ? tb->sd[d][si] : 0.0;
    const double v = dv == 0.0 ? 0.0 : dv / s[si];
    bad |= !(fabs(v) < 1e12);
    if (nw && x > GC_NWQ) bad = false;
    sc->g.dT[x][d] = px3_of(v);
  }
  if (t == 0) sc->g.dns = px3_of(tb->sd[GX_NS][S_NS]);
  if (bad) tb->wide = 1;
}

// Rows: four per warp, lane = 8 slot + direction; kernels: a thread per node.
constexpr int GXP_THREADS = 64;
__global__ void __launch_bounds__(GXP_THREADS) grad_pack64_kernel(GradBatch gb, const ConstTables* __restrict__ c,
                                                                  int row_ctas) {
  const GradItem gi = grad_item(gb, blockIdx.y);
  const GeoHeader* geo = gi.geo;
  TabD* tb = gi.tab;
  const int na = geo->na;
  bool bad = false;
  if ((int)blockIdx.x >= row_ctas) {
    const GxScratch* sc = gx_scratch(tb);
    const int e = ((int)blockIdx.x - row_ctas) * GXP_THREADS + threadIdx.x;
    if (e >= na * geo->n_tr) return;
    double* K = gi.kernd + (size_t)e * (NDIR + 1);
    const int sh = 1023 - sc->kexp[e / na];
    const double m = __hiloint2double((1023 + sh) << 20, 0);  // |sh| < 960
#pragma unroll
    for (int d = 0; d <= NDIR; ++d) {
      const double v = K[d] * m;
      bad |= !(fabs(v) < 1e15);
      const FF f = px_of(v);
      reinterpret_cast<float2*>(K)[d] = make_float2(f.hi, f.lo);
    }
    if (bad) tb->wide = 1;
    return;
  }
  const PxTab& T = c->px;
  const int lane = threadIdx.x & 31, dir = lane & 7;
  const int n_raw = ((int)blockIdx.x * (GXP_THREADS / 32) + (threadIdx.x >> 5)) * 4 + (lane >> 3);
  const bool live = n_raw < na;  // a slot past the last node reads and writes nothing
  double* R = gi.rowd + (size_t)min(n_raw, na - 1) * NROWD;
  const bool lin = pk_model(geo->physics) == JCG_PK_LINEAR;
  double v[NA_IN], d[NA_IN];
#pragma unroll
  for (int i = 0; i < NA_IN; ++i) v[i] = live ? R[i] : 1.0, d[i] = live ? R[NA_IN * (1 + dir) + i] : 0.0;
  __syncwarp();
  const double fc = tb->sv[S_TFNW] != 0.0 ? 1.0 : tb->sv[S_FC];
  const double pn = tb->sv[S_PKNORM], g = v[A_G], chic = v[A_CHIC];
  auto in = [&](double x, double lo, double hi) {
    bad |= !(x > lo && x < hi);
    return x;
  };
  // one logarithm per lane; ln k_nl goes from dir 5 to dir 1, all 32 lanes taking part
  double lx = 1.0;
  if (live) {
    if (dir == 0 || dir == 1) lx = in(chic, 1e-9, 1e9);
    if (dir == 4) lx = in(g * g * pn * (fc * fc * (1.0 / (2.0 * (PI * PI)))), 1e-18, 1e18);
    if (!lin) {
      if (dir == 2) lx = in(v[A_AN], 1e-18, 1e18);
      if (dir == 3) lx = in(v[A_BN], 1e-18, 1e18);
      if (dir == 5) lx = in(v[A_KNL], 1e-9, 1e9);
    }
  }
  const long long lg = px_log2_d(lx, T);
  const long long lknl = __shfl_down_sync(0xffffffffu, lg, 4);
  if (live) {
    long long* row = reinterpret_cast<long long*>(R);
    float2* rf = reinterpret_cast<float2*>(R);
    auto pair = [&](int i, double x) {
      bad |= !(fabs(x) < 1e15);
      const FF f = px_of(x);
      rf[i] = make_float2(f.hi, f.lo);
    };
    // one exponent per lane
    double ex = 0.0;
    if (!lin) {
      if (dir == 0) ex = in(v[A_BETA], -7.9, 7.9);
      if (dir == 1) ex = in(3.0 * v[A_F1], -7.9, 7.9);
      if (dir == 2) ex = in(v[A_F2], -7.9, 7.9);
      if (dir == 3) ex = in(3.0 - v[A_GAM], -7.9, 7.9);
      if (dir == 4) ex = in(v[A_LCF3] * D_LOG2E, -30.0, 30.0) * 0.125;  // 2^-57 units
    }
    const long long fx = __double2ll_rn(ex * P2_60);
    if (dir == 0) row[GR_L2C] = lg, row[GR_BETA] = fx;
    if (dir == 1) row[GR_L2Y] = lg + lknl, row[GR_E1] = fx;
    if (dir == 2) row[GR_A0] = lg >> 4, row[GR_E2] = fx;
    if (dir == 3) row[GR_B0] = lg >> 4, row[GR_E3] = fx;
    if (dir == 4) row[GR_LD] = lg >> 4, row[GR_L3] = fx;
    const double ichic = 1.0 / chic, iknl = lin ? 1.0 : 1.0 / v[A_KNL];
    if (dir == 5) reinterpret_cast<double*>(R)[GR_ICHIC] = ichic;
    if (dir == 6) reinterpret_cast<double*>(R)[GR_IYK] = 1.0 / (chic * (lin ? 1.0 : v[A_KNL]));
    if (dir == 7) {
      pair(GR_V, (2.0 * (PI * PI)) * v[A_U] * (chic * chic * chic));
      if (!lin) {
        pair(GR_ALPHA, v[A_ALPHA]);
        pair(GR_NU, v[A_NU]);
        pair(GR_MU, v[A_MU]);
        // power.py:194-195: mu and nu are 10^ of lines in n_eff
        pair(GR_MUC, v[A_MU] == 0.0 ? 0.0 : (0.1908 / 1.2857) * v[A_MU] / v[A_NU]);
      }
    }
    const double dk = -d[A_CHIC] * ichic;
    const double u3 = (2.0 * (PI * PI)) * (chic * chic * chic);
    pair(GR_V + 1 + dir, u3 * (d[A_U] - 3.0 * v[A_U] * dk));
    float2* tan = rf + GR_T + dir;
    auto tput = [&](int x, double w) {
      bad |= !(fabs(w) < 1e15);
      const FF f = px_of(w);
      tan[x * NDIR] = make_float2(f.hi, f.lo);
    };
    tput(GT_K, dk);
    tput(GT_A, 2.0 * d[A_G] / g + tb->sd[dir][S_PKNORM] / pn);
    if (!lin) {
      tput(GT_Y, dk - d[A_KNL] * iknl);
      tput(GT_BETA, d[A_BETA]);
      tput(GT_ALPHA, d[A_ALPHA]);
      tput(GT_AN, d[A_AN] / v[A_AN]);
      tput(GT_E1, 3.0 * d[A_F1]);
      tput(GT_BN, d[A_BN] / v[A_BN]);
      tput(GT_E2, d[A_F2]);
      tput(GT_E3, -d[A_GAM]);
      tput(GT_G0, (3.0 - v[A_GAM]) * d[A_LCF3] - d[A_GAM] * v[A_LCF3]);
      tput(GT_NU, d[A_NU]);
    }
    if (bad) tb->wide = 1;
  }
}

// -------------------------------------------------------------- integral ---
constexpr int GX_RUN = 4;  // a nodes summed in pairs before the three-float totals
struct GxLayout {
  size_t tab, g, kh, l2kh, P, K, M, tot, total;
  int mb;
};
// a nodes per chunk at most: as many as give every thread one node
__host__ __device__ inline int gx_ta(int LT) { return GX_THREADS / LT; }
__host__ __device__ inline GxLayout gx_layout_mb(int n_cls, int n_tr, int LT, int mb) {
  GxLayout L;
  size_t o = 0;
  L.mb = mb;
  L.tab = o;
  o += (sizeof(PxTab) + 15) & ~(size_t)15;
  L.g = o;
  o += (sizeof(GxTabs) + 15) & ~(size_t)15;
  L.kh = o;
  o += (size_t)LT * 8;
  L.l2kh = o;
  o += (size_t)LT * 8;
  L.P = o;
  o += (size_t)gx_ta(LT) * (NDIR + 1) * LT * 8;
  L.K = o;
  o += (size_t)mb * n_tr * 2 * (NDIR + 1) * 8;
  L.M = o;
  o += (size_t)mb * n_cls * (NDIR + 1) * 8;
  L.tot = o;
  o += (size_t)LT * n_cls * (NDIR + 1) * 12;
  L.total = o;
  return L;
}
// a nodes per block of weights: 8, less where two CTAs would not fit an SM
__host__ __device__ inline GxLayout gx_layout(int n_cls, int n_tr, int LT) {
  int mb = 8;
  while (mb > 2 && gx_layout_mb(n_cls, n_tr, LT, mb).total > 112 * 1024) mb >>= 1;
  return gx_layout_mb(n_cls, n_tr, LT, mb);
}

template <bool GEN>
__global__ void __launch_bounds__(GX_THREADS, 2)
    grad_limber64_kernel(GradBatch gb, const ConstTables* __restrict__ ct, int LT) {
  const int item = blockIdx.z, split = blockIdx.y;
  const GradItem gi = grad_item(gb, item);
  const GeoHeader* geo = gi.geo;
  TabD* tb = gi.tab;
  const int n_ell = geo->n_ell, n_cls = geo->n_cls, na = geo->na, n_tr = geo->n_tr;
  const bool lin = pk_model(geo->physics) == JCG_PK_LINEAR, nw = tf_nowiggle(geo->physics);
  const int l0 = blockIdx.x * LT;
  if (l0 >= n_ell) return;
  const int lt = min(LT, n_ell - l0);
  const int per = (na + gb.n_split - 1) / gb.n_split;
  const int a_begin = split * per, a_end = min(na, a_begin + per);
  const GxLayout L = gx_layout(gb.n_cls, gb.n_tr, LT);
  extern __shared__ __align__(16) unsigned char smem[];
  PxTab& T = *reinterpret_cast<PxTab*>(smem + L.tab);
  GxTabs& g = *reinterpret_cast<GxTabs*>(smem + L.g);
  double* kh = reinterpret_cast<double*>(smem + L.kh);
  long long* l2kh = reinterpret_cast<long long*>(smem + L.l2kh);
  float2* P = reinterpret_cast<float2*>(smem + L.P);     // [TA][9][LT]
  float2* Ks = reinterpret_cast<float2*>(smem + L.K);    // [mb][n_tr][2][9]: K V, K
  float2* Ms = reinterpret_cast<float2*>(smem + L.M);    // [mb][n_cls][9]
  float* tot = reinterpret_cast<float*>(smem + L.tot);   // [27][lt n_cls]
  const int tid = threadIdx.x;
  // a cosmology that is left to the float64 kernels already (one thread reads the
  // flag: other CTAs may set it meanwhile): with narrow bins far apart the integral
  // in pairs would be 5% of the call, for nothing (16 cosmologies, 3 + 3 bins)
  __shared__ int left;
  if (tid == 0) left = tb->wide;
  __syncthreads();
  if (left) return;
  const double* ELL = geo_ptr<double>(geo, geo->off_ell);
  const double* EF = geo_ptr<double>(geo, geo->off_ellfac);
  const GxScratch* sc = gx_scratch(tb);
  for (int i = tid; i < (int)(sizeof(PxTab) / 16); i += GX_THREADS)
    reinterpret_cast<uint4*>(&T)[i] = reinterpret_cast<const uint4*>(&ct->px)[i];
  for (int i = tid; i < (int)(sizeof(GxTabs) / 8); i += GX_THREADS)
    reinterpret_cast<double*>(&g)[i] = reinterpret_cast<const double*>(&sc->g)[i];
  const int units = lt * n_cls;
  // kernels and weights have tangents in the background's directions, and in
  // gamma's (the growth factor in a bias)
  const int gd = gb.gamma_dir;
  auto has = [&](int d) { return bg_dir(d) || d == gd; };
  for (int i = tid; i < 3 * (NDIR + 1) * units; i += GX_THREADS) tot[i] = 0.f;
  __syncthreads();
  bool bad = false;
  for (int l = tid; l < lt; l += GX_THREADS) {
    const double e = ELL[l0 + l] + 0.5;
    kh[l] = e;
    l2kh[l] = px_log2_d(e, T);
    bad |= !(e > 1e-7 && e < 1e7);
  }
  const int tm = gx_ta(LT), span = max(a_end - a_begin, 0), nch = (span + tm - 1) / tm;
  const int TA = nch ? (span + nch - 1) / nch : 0;
  __syncthreads();
  for (int base = a_begin; base < a_end; base += TA) {
    const int tc = min(TA, a_end - base);
    for (int q = tid; q < tc * lt; q += GX_THREADS) {
      const int t = q / lt, l = q - t * lt;
      FF o[NDIR + 1];
      px_node_grad<GEN>(g, T, reinterpret_cast<const long long*>(gi.rowd + (size_t)(base + t) * NROWD), kh[l], l2kh[l],
                        nw, lin, o);
      bad |= !(fabsf(o[0].hi) > 1e-30f && fabsf(o[0].hi) < 1e30f);
#pragma unroll
      for (int s = 0; s <= NDIR; ++s) {
        bad |= !(fabsf(o[s].hi) < 1e30f);
        P[(t * (NDIR + 1) + s) * LT + l] = make_float2(o[s].hi, o[s].lo);
      }
    }
    for (int m0 = 0; m0 < tc; m0 += L.mb) {
      const int mc = min(L.mb, tc - m0);
      // kernels, and kernels times V
      for (int q = tid; q < mc * n_tr; q += GX_THREADS) {
        const int t = q / n_tr, i = q - t * n_tr, n = base + m0 + t;
        const float2* K = reinterpret_cast<const float2*>(gi.kernd + ((size_t)i * na + n) * (NDIR + 1));
        const float2* V = reinterpret_cast<const float2*>(gi.rowd + (size_t)n * NROWD) + GR_V;
        float2* o = Ks + (size_t)q * 2 * (NDIR + 1);
        const float2 k0 = K[0], v0 = V[0];
        const FF w = px_mul(px_f2(k0), px_f2(v0));
        o[0] = make_float2(w.hi, w.lo);
        o[NDIR + 1] = k0;
#pragma unroll
        for (int d = 1; d <= NDIR; ++d) {
          if (!has(d - 1)) continue;
          const float2 kd = K[d];
          float ah = 0.f, al = 0.f;
          ff_acc_prod(ah, al, kd, v0);
          ff_acc_prod(ah, al, k0, V[d]);
          const FF x = px_norm(ah, al);
          o[d] = make_float2(x.hi, x.lo);
          o[NDIR + 1 + d] = kd;
        }
      }
      __syncthreads();
      for (int q = tid; q < mc * n_cls; q += GX_THREADS) {
        const int t = q / n_cls, p = q - t * n_cls;
        const float2* A = Ks + (size_t)(t * n_tr + geo->pair_i[p]) * 2 * (NDIR + 1);
        const float2* B = Ks + (size_t)(t * n_tr + geo->pair_j[p]) * 2 * (NDIR + 1) + NDIR + 1;
        float2* o = Ms + (size_t)q * (NDIR + 1);
        const float2 a0 = A[0], b0 = B[0];
        const FF w = px_mul(px_f2(a0), px_f2(b0));
        o[0] = make_float2(w.hi, w.lo);
#pragma unroll
        for (int d = 1; d <= NDIR; ++d) {
          if (!has(d - 1)) continue;
          float ah = 0.f, al = 0.f;
          ff_acc_prod(ah, al, A[d], b0);
          ff_acc_prod(ah, al, a0, B[d]);
          const FF x = px_norm(ah, al);
          o[d] = make_float2(x.hi, x.lo);
        }
      }
      __syncthreads();
      for (int u = tid; u < units; u += GX_THREADS) {
        const int p = u / lt, l = u - p * lt;
        for (int t0 = 0; t0 < mc; t0 += GX_RUN) {
          float ah[NDIR + 1], al[NDIR + 1];
#pragma unroll
          for (int s = 0; s <= NDIR; ++s) ah[s] = al[s] = 0.f;
          const int te = min(mc, t0 + GX_RUN);
          for (int t = t0; t < te; ++t) {
            const float2* pp = P + (size_t)(m0 + t) * (NDIR + 1) * LT + l;
            const float2* mm = Ms + (size_t)(t * n_cls + p) * (NDIR + 1);
            const float2 p0 = pp[0], w0 = mm[0];
            ff_acc_prod(ah[0], al[0], p0, w0);
#pragma unroll
            for (int s = 1; s <= NDIR; ++s) {
              ff_acc_prod(ah[s], al[s], pp[s * LT], w0);
              if (has(s - 1)) ff_acc_prod(ah[s], al[s], p0, mm[s]);
            }
          }
#pragma unroll
          for (int s = 0; s <= NDIR; ++s) {
            float* w = tot + (size_t)(3 * s) * units + u;
            F3 x = F3{w[0], w[units], w[2 * units]};
            px_acc3(x, px_norm(ah[s], al[s]));
            w[0] = x.hi, w[units] = x.lo, w[2 * units] = x.ll;
          }
        }
      }
      // Ks is next written after every thread is past its Ms products; Ms after
      // the barrier that follows Ks
    }
    __syncthreads();
  }
  if (bad) tb->wide = 1;
  double* part = gi.part + (size_t)split * n_cls * n_ell * (NDIR + 1);
  for (int o = tid; o < units * (NDIR + 1); o += GX_THREADS) {
    const int u = o / (NDIR + 1), s = o - u * (NDIR + 1), p = u / lt, l = u - p * lt, ell = l0 + l;
    const int pi = geo->pair_i[p], pj = geo->pair_j[p];
    const float* w = tot + (size_t)(3 * s) * units + u;
    const double e = kh[l];
    const double ef = EF[(size_t)pi * n_ell + ell] * EF[(size_t)pj * n_ell + ell];
    const double v = px_d3(F3{w[0], w[units], w[2 * units]}) * __hiloint2double(sc->kexp[pi] << 20, 0) *
                     __hiloint2double(sc->kexp[pj] << 20, 0);
    part[((size_t)p * n_ell + ell) * (NDIR + 1) + s] = v / (e * e * e) * ef;
  }
}

// ell per CTA: a power of two up to 32 whose tile fits twice on an SM
int grad_limber64_tile(int n_ell, int n_cls) {
  int l = 32;
  while (l > 1 && gx_layout_mb(n_cls, n_cls, l, 2).total > 100 * 1024) l >>= 1;
  const int tiles = (n_ell + l - 1) / l;
  return (n_ell + tiles - 1) / tiles;
}

// Splits of the a nodes, `tiles` ell tiles in all: no more CTAs than fit the SMs at
// once (two each; 25 tiles x 13 splits, 21 CTAs more than that: 264 us, x 12: 178),
// or, past that, the least number whose last wave leaves 10% idle (427 tiles:
// 1,880 us; x 5: 1,812)
int grad_limber64_split(long long tiles, int na, int lt) {
  const long long slots = 2LL * 152;
  const int most = max(1, min(na / gx_ta(lt), 64));
  if (tiles <= slots) {
    const int ns = (int)(slots / tiles);
    return ns < most ? ns : most;
  }
  int best = 1;
  double eff = 0.0;
  for (int ns = 1; ns <= 8 && ns <= most; ++ns) {
    const long long c = tiles * ns, w = (c + slots - 1) / slots;
    const double e = (double)c / (double)(w * slots);
    if (e > eff + 0.01) best = ns, eff = e;
    if (eff >= 0.9) break;
  }
  return best;
}

template <bool GEN>
static void launch_limber64g(const GradBatch& gb, const ConstTables* c, cudaStream_t st) {
  const int lt = grad_limber64_tile(gb.n_ell, gb.n_cls);
  const size_t sm = gx_layout(gb.n_cls, gb.n_tr, lt).total;
  allow_smem(grad_limber64_kernel<GEN>, sm);
  grad_limber64_kernel<GEN><<<dim3((gb.n_ell + lt - 1) / lt, gb.n_split, gb.n_items), GX_THREADS, sm, st>>>(gb, c, lt);
}

void launch_grad_limber64(const GradBatch& gb, const ConstTables* c, cudaStream_t st) {
  grad_scale64_kernel<<<dim3(gb.n_tr + 1, gb.n_items), GXS_THREADS, 0, st>>>(gb);
  const int rows = (gb.na + 4 * (GXP_THREADS / 32) - 1) / (4 * (GXP_THREADS / 32));
  const int kern = (gb.na * gb.n_tr + GXP_THREADS - 1) / GXP_THREADS;
  grad_pack64_kernel<<<dim3(rows + kern, gb.n_items), GXP_THREADS, 0, st>>>(gb, c, rows);
  if (gb.physics_or != 0) launch_limber64g<true>(gb, c, st);
  else launch_limber64g<false>(gb, c, st);
}

}  // namespace jcg
