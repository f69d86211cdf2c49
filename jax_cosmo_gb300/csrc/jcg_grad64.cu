// Tables with tangents of the FP64 gradient (the Jacobian and the vector-
// Jacobian product of angular_cl): background, growth, sigma8, P(k) k^3 and
// sigma^2(R), value and 8 tangents each, float64.
//
// One CTA per cosmology with one tangent direction per lane spent 1.45 ms on
// them: 1,154 node evaluations on one SM's FP64 pipe (2 lanes per clock), the
// value repeated in every direction, then serial scans by single lanes.  Here
//   grad_nodes64_kernel   a node or step per thread, CTAs of a warp: Eisenstein-Hu at
//     the 386 Romberg and P(k) nodes, T and its partials in 12 inputs by a reverse
//     sweep, then the 8 directions by one product each; chi's increments, and the
//     growth steps' matrices for two directions a thread, tangents in closed form;
//   grad_bg64_kernel      chi by suffix sums, growth by scans of the matrices and of
//     their tangents' affine maps, a warp per component;
//   grad_sigma64_kernel   sigma8's weighted sum, P(k) k^3 and sigma^2(R): a CTA per
//     component and quarter of the R nodes.
// One cosmology 1,453 -> 55 us (21 + 23 + 10); what is left is latency: serial float64 code of
// a thread and the scans.
#include "jcg_grad.cuh"
#include "jcg_px.cuh"

namespace jcg {

// node scratch in the part of TabD that only fp32c uses: exp(n_s ln k) T^2 (times
// the window for the Romberg nodes) as [NDIR + 1][NROMB + NKH]
constexpr int NEH = GRAD_NEH;
static_assert(offsetof(TabD, c32) % 8 == 0, "node scratch alignment");
__device__ __forceinline__ double* eh_scratch(TabD* t) { return reinterpret_cast<double*>(&t->c32[0][0]); }

// T(k) (transfer.py:88-153) and its partials dT/d(ln x) in the scalars x below
// (dT/dx in f_b and f_c, which may be 0)
struct EhGrad {
  double T, keq, sh, betac, alphac, alphab, betab, betanode, ksilk, fb, fc, agam, nwq;
};
__device__ EhGrad eh_grad_osc(const double* s, double k, double lk, double ik) {
  EhGrad g;
  const double q = k * s[S_QINV];
  const double u = 69.9 * exp(1.08 * (lk - s[S_LGQ]));
  const double Cb = 386.0 / (1.0 + u);
  const double qq = q * q;
  const double b18 = 1.8 * s[S_BETA_C] * q, A1 = EULER_E + b18, A2 = EULER_E + 1.8 * q;
  const double L1 = log(A1), L2 = log(A2);
  const double cA = (14.2 + Cb) * qq, cB = (s[S_C142AC] + Cb) * qq;
  const double iDa = 1.0 / (L1 + cA), iDb = 1.0 / (L1 + cB), iDn = 1.0 / (L2 + cA);
  const double Ta = L1 * iDa, Tb = L1 * iDb, Tn = L2 * iDn;
  const double ksh = k * s[S_SH_D];
  const double x54 = ksh * (1.0 / 5.4), x2 = x54 * x54, x4 = x2 * x2, x52 = ksh * (1.0 / 5.2);
  const double f = 1.0 / (1.0 + x4), iE = 1.0 / (1.0 + x52 * x52);
  const double Tc = f * Ta + (1.0 - f) * Tb;
  const double iksh = ik * s[S_ISH];
  const double bb = s[S_BETA_B] * iksh, bn = s[S_BETA_NODE] * iksh;
  const double w3 = 1.0 / (1.0 + bb * bb * bb);
  const double bn3 = bn * bn * bn, z = bn3 / (1.0 + bn3);
  const double ex = exp(1.4 * (lk - s[S_LGKSILK])), silk = exp(-ex);
  const double arg = ksh * rcbrt(1.0 + bn3);
  double sn, cs;
  sincos(arg, &sn, &cs);
  const double sinc = sn / arg;
  const double t1 = sinc * Tn * iE, t2 = sinc * s[S_ALPHA_B] * silk * w3, fbs = s[S_FB] * sinc;
  const double b1 = s[S_FB] * t1, b2 = s[S_FB] * t2;  // the two baryon terms
  g.T = b1 + b2 + s[S_FC] * Tc;
  // adjoints
  const double fc = s[S_FC];
  const double aTa = fc * f * iDa, aTb = fc * (1.0 - f) * iDb, aTn = fbs * iE * iDn;
  const double dcA = -aTa * Ta - aTn * Tn, dcB = -aTb * Tb;
  const double dL1 = aTa * (1.0 - Ta) + aTb * (1.0 - Tb), dL2 = aTn * (1.0 - Tn);
  const double bc = dL1 * b18 / A1;
  const double cu = qq * Cb * 1.08 * u / (1.0 + u);
  const double dq = bc + dL2 * 1.8 * q / A2 + dcA * (2.0 * cA - cu) + dcB * (2.0 * cB - cu);
  const double w = 3.0 * (1.0 - w3) * b2;
  const double da = (b1 + b2) * (sinc != 0.0 ? cs / sinc - 1.0 : 0.0);  // d T / d ln arg
  g.keq = -dq;
  g.betac = bc;
  g.alphac = -dcB * qq * s[S_C142AC];
  g.alphab = b2;
  g.betab = -w;
  g.betanode = -z * da;
  g.ksilk = 1.4 * ex * b2;
  g.fb = t1 + t2;
  g.fc = Tc;
  g.sh = fc * (Tb - Ta) * 4.0 * x4 * f * f - b1 * 2.0 * x52 * x52 * iE + w + (1.0 + z) * da;
  g.agam = g.nwq = 0.0;
  return g;
}
__device__ EhGrad eh_grad_nowiggle(const double* s, double k) {
  EhGrad g;
  const double x = 0.43 * k * s[S_SH_D], x2 = x * x, x4 = x2 * x2;
  const double un = 1.0 / (1.0 + x4), ag = s[S_AGAM], gen = ag + (1.0 - ag) * un;
  const double q = k * s[S_NWQ] / gen;
  const double A = 2.0 * EULER_E + 1.8 * q, L = log(A), r = 1.0 / (1.0 + 62.5 * q), C = 14.2 + 731.0 * r;
  const double iD = 1.0 / (L + C * q * q);
  g.T = L * iD;
  const double dL = iD * (1.0 - g.T), dD = -iD * g.T;
  const double dq = dL * 1.8 * q / A + dD * (2.0 * C * q * q - q * q * q * 731.0 * 62.5 * r * r);  // d ln q
  g.nwq = dq;
  g.agam = -dq * (1.0 - un) * ag / gen;
  g.sh = dq * (1.0 - ag) * 4.0 * x4 * un * un / gen;
  g.keq = g.betac = g.alphac = g.alphab = g.betab = g.betanode = g.ksilk = g.fb = g.fc = 0.0;
  return g;
}

__device__ __forceinline__ void eh_nodes64(TabD* tb, const ConstTables* c, int job) {
  __shared__ double s[NSCAL];
  // d ln x of the scalars above (d x of f_b, f_c and n_s), per direction
  constexpr int NX = 13;
  __shared__ double dl[NX][NDIR];
  const int lane = threadIdx.x;
  for (int i = lane; i < NSCAL; i += 32) s[i] = tb->sv[i];
  __syncwarp();
  if (lane == 0) {  // not all forms of the scalars' kernel fill these
    s[S_QINV] = 1.0 / (13.41 * s[S_K_EQ]);
    s[S_ISH] = 1.0 / s[S_SH_D];
    s[S_C142AC] = 14.2 / s[S_ALPHA_C];
  }
  constexpr int X[NX] = {S_K_EQ, S_SH_D, S_BETA_C, S_ALPHA_C, S_ALPHA_B, S_BETA_B, S_BETA_NODE, S_K_SILK,
                         S_FB,   S_FC,   S_AGAM,   S_NWQ,     S_NS};
  for (int i = lane; i < NX * NDIR; i += 32) {
    const int x = i / NDIR, d = i % NDIR;
    int si = 0;
#pragma unroll
    for (int q = 0; q < NX; ++q)
      if (q == x) si = X[q];
    const double v = tb->sv[si], t = tb->sd[d][si];
    dl[x][d] = si == S_FB || si == S_FC || si == S_NS ? t : t == 0.0 ? 0.0 : t / v;
  }
  __syncwarp();
  const int e = job * 32 + lane;
  if (e >= NEH) return;
  const bool romb = e < NROMB;
  const int i = romb ? e : e - NROMB;
  const double k = romb ? c->romb_k[i] : c->kh[i], lk = romb ? c->romb_logk[i] : c->logk[i];
  const double ik = romb ? c->romb_ik[i] : c->ikh[i];
  const EhGrad g = s[S_TFNW] != 0.0 ? eh_grad_nowiggle(s, k) : eh_grad_osc(s, k, lk, ik);
  const double w = exp(s[S_NS] * lk) * (romb ? c->romb_kw2[i] : 1.0);
  const double v = w * (g.T * g.T), t2 = 2.0 * w * g.T;
  double* out = eh_scratch(tb) + e;
  out[0] = v;
  const double a[NX] = {g.keq, g.sh, g.betac, g.alphac, g.alphab, g.betab, g.betanode, g.ksilk, g.fb, g.fc, g.agam,
                        g.nwq, 0.0};
#pragma unroll
  for (int d = 0; d < NPW; ++d) {
    double x = 0.0;
#pragma unroll
    for (int q = 0; q < NX - 1; ++q) x = fma(a[q], dl[q][d], x);
    out[(1 + d) * NEH] = fma(t2, x, v * lk * dl[NX - 1][d]);
  }
}

// -------------------------------------------------------------- background --
// chi increments and growth step matrices with tangents, between the nodes' kernel
// and the scans: in the place of tables that are written later
struct Bg64 {  // over sigv .. pk3d
  double M[NGROW][4], dM[NDIR][NGROW][4];
};
static_assert(sizeof(Bg64) <= sizeof(double) * (NDIR + 1) * (NRT + NKH), "matrices fit");
__device__ __forceinline__ Bg64* bg_scratch(TabD* t) { return reinterpret_cast<Bg64*>(t->sigv); }
static_assert(offsetof(TabD, pk3d) - offsetof(TabD, sigv) == sizeof(double) * ((NDIR + 1) * NRT + NKH), "contiguous");
__device__ __forceinline__ double* inc_scratch(TabD* t) { return reinterpret_cast<double*>(grad_kw64(t)); }  // [9][NCHI]

// E^2 with the tangents of ND directions
template <int ND>
struct E2D {
  double e2, ef, d[ND], def[ND];
};
template <int ND>
__device__ __forceinline__ E2D<ND> e2_grad(const double* s, const double* sd, double a, double lna, double ia) {
  E2D<ND> r;
  const double f = -3.0 * (1.0 + s[S_W0] + s[S_WA]) * lna + 3.0 * s[S_WA] * (a - 1.0);
  r.ef = exp(f);
  const double ia2 = ia * ia, ia3 = ia2 * ia;
  r.e2 = s[S_OMEGA_M] * ia3 + s[S_OMEGA_K] * ia2 + s[S_OMEGA_DE] * r.ef;
#pragma unroll
  for (int d = 0; d < ND; ++d) {
    const double* t = sd + d * NSCAL;
    const double df = -3.0 * (t[S_W0] + t[S_WA]) * lna + 3.0 * t[S_WA] * (a - 1.0);
    r.def[d] = t[S_OMEGA_DE] * r.ef + s[S_OMEGA_DE] * r.ef * df;  // d(Omega_de exp(f_de))
    r.d[d] = t[S_OMEGA_M] * ia3 + t[S_OMEGA_K] * ia2 + r.def[d];
  }
  return r;
}

// dchi/dln a = R_H / (a sqrt(E^2)) (background.py:227-231) times w, added to f
__device__ __forceinline__ void chi_rhs(const double* s, const double* sd, double a, double lna, double ia, double w,
                                        double* f) {
  const E2D<NDIR> e = e2_grad<NDIR>(s, sd, a, lna, ia);
  const double r = rsqrt(e.e2), v = w * (RH * ia * r), h = -0.5 * v * (r * r);
  f[0] += v;
#pragma unroll
  for (int d = 0; d < NDIR; ++d) f[1 + d] = fma(h, e.d[d], f[1 + d]);
}

// growth ODE coefficients D'' = -q D' + r D (background.py:96-106), ND directions
template <int ND>
struct QR {
  double q, r, dq[ND], dr[ND];
};
template <int ND>
__device__ __forceinline__ QR<ND> growth_qr_grad(const double* s, const double* sd, double a, double lna, double ia) {
  QR<ND> o;
  const E2D<ND> e = e2_grad<ND>(s, sd, a, lna, ia);
  const double ie = 1.0 / e.e2, ia2 = ia * ia, ia3 = ia2 * ia;
  const double om = s[S_OMEGA_M] * ia3 * ie, de = s[S_OMEGA_DE] * e.ef * ie;
  const double w1 = 1.0 + 3.0 * (s[S_W0] + (1.0 - a) * s[S_WA]);
  o.q = (2.0 - 0.5 * (om + w1 * de)) * ia;
  o.r = 1.5 * om * ia2;
#pragma unroll
  for (int d = 0; d < ND; ++d) {
    const double* td = sd + d * NSCAL;
    const double dom = (td[S_OMEGA_M] * ia3 - om * e.d[d]) * ie, dde = (e.def[d] - de * e.d[d]) * ie;
    const double dw1 = 3.0 * (td[S_W0] + (1.0 - a) * td[S_WA]);
    o.dq[d] = -0.5 * (dom + w1 * dde + dw1 * de) * ia;
    o.dr[d] = 1.5 * dom * ia2;
  }
  return o;
}

// One RK4 step is linear in y = (D, dD/da), y_i = M_i y_{i-1}, with
// K1 = A0, K2 = Am (1 + h/2 K1), K3 = Am (1 + h/2 K2), K4 = A1 (1 + h K3),
// M = 1 + h/6 (K1 + 2 K2 + 2 K3 + K4), A = [[0, 1], [r, -q]]; dM by the same
// products.  A thread per step and two directions.
constexpr int GST_ND = 2, GST_GRP = NDIR / GST_ND;
__device__ __forceinline__ void growth_step64(TabD* tb, const ConstTables* c, int idx) {
  const int i = idx % NGROW, d0 = idx / NGROW * GST_ND;
  Bg64* o = bg_scratch(tb);
  double M[4] = {1.0, 0.0, 0.0, 1.0};
  if (i == 0) {
#pragma unroll
    for (int d = 0; d < GST_ND; ++d) o->dM[d0 + d][0][0] = o->dM[d0 + d][0][1] = o->dM[d0 + d][0][2] = o->dM[d0 + d][0][3] = 0.0;
  } else {
    const double *s = tb->sv, *sd = tb->sd[d0];
    const QR<GST_ND> A0 = growth_qr_grad<GST_ND>(s, sd, c->atab_grow[i - 1], c->grow_lna[i - 1], c->grow_ia[i - 1]);
    const QR<GST_ND> Am = growth_qr_grad<GST_ND>(s, sd, c->grow_am[i], c->grow_lnam[i], c->grow_iam[i]);
    const QR<GST_ND> A1 = growth_qr_grad<GST_ND>(s, sd, c->atab_grow[i], c->grow_lna[i], c->grow_ia[i]);
    const double h = c->atab_grow[i] - c->atab_grow[i - 1], h2 = 0.5 * h;
    const double q0 = A0.q, r0 = A0.r, qm = Am.q, rm = Am.r, q1 = A1.q, r1 = A1.r;
    // X2 = 1 + h/2 K1, X3 = 1 + h/2 K2, X4 = 1 + h K3 (K = [[k0, k1], [k2, k3]])
    const double X2[4] = {1.0, h2, h2 * r0, 1.0 - h2 * q0};
    const double K2[4] = {X2[2], X2[3], rm * X2[0] - qm * X2[2], rm * X2[1] - qm * X2[3]};
    const double X3[4] = {1.0 + h2 * K2[0], h2 * K2[1], h2 * K2[2], 1.0 + h2 * K2[3]};
    const double K3[4] = {X3[2], X3[3], rm * X3[0] - qm * X3[2], rm * X3[1] - qm * X3[3]};
    const double X4[4] = {1.0 + h * K3[0], h * K3[1], h * K3[2], 1.0 + h * K3[3]};
    const double K4[4] = {X4[2], X4[3], r1 * X4[0] - q1 * X4[2], r1 * X4[1] - q1 * X4[3]};
    const double h6 = h / 6.0;
    M[0] = 1.0 + h6 * (2.0 * (K2[0] + K3[0]) + K4[0]);
    M[1] = h6 * (1.0 + 2.0 * (K2[1] + K3[1]) + K4[1]);
    M[2] = h6 * (r0 + 2.0 * (K2[2] + K3[2]) + K4[2]);
    M[3] = 1.0 + h6 * (-q0 + 2.0 * (K2[3] + K3[3]) + K4[3]);
#pragma unroll
    for (int d = 0; d < GST_ND; ++d) {
      const double dq0 = A0.dq[d], dr0 = A0.dr[d], dqm = Am.dq[d], drm = Am.dr[d], dq1 = A1.dq[d], dr1 = A1.dr[d];
      const double x2 = h2 * dr0, x3 = -h2 * dq0;  // dX2 = [[0, 0], [x2, x3]]
      const double k0 = x2, k1 = x3, k2 = drm * X2[0] - dqm * X2[2] - qm * x2, k3 = drm * X2[1] - dqm * X2[3] - qm * x3;
      const double a0 = h2 * k0, a1 = h2 * k1, a2 = h2 * k2, a3 = h2 * k3;  // dX3
      const double l0 = a2, l1 = a3, l2 = drm * X3[0] - dqm * X3[2] + rm * a0 - qm * a2,
                   l3 = drm * X3[1] - dqm * X3[3] + rm * a1 - qm * a3;
      const double b0 = h * l0, b1 = h * l1, b2 = h * l2, b3 = h * l3;  // dX4
      const double m2 = dr1 * X4[0] - dq1 * X4[2] + r1 * b0 - q1 * b2, m3 = dr1 * X4[1] - dq1 * X4[3] + r1 * b1 - q1 * b3;
      o->dM[d0 + d][i][0] = h6 * (2.0 * (k0 + l0) + b2);
      o->dM[d0 + d][i][1] = h6 * (2.0 * (k1 + l1) + b3);
      o->dM[d0 + d][i][2] = h6 * (dr0 + 2.0 * (k2 + l2) + m2);
      o->dM[d0 + d][i][3] = h6 * (-dq0 + 2.0 * (k3 + l3) + m3);
    }
  }
  if (d0 == 0) {
#pragma unroll
    for (int q = 0; q < 4; ++q) o->M[i][q] = M[q];
  }
}

// CTAs per cosmology: Eisenstein-Hu nodes, chi steps, growth steps x direction pairs
constexpr int N64_EH = (NEH + 31) / 32, N64_CHI = NCHI / 32, N64_GROW = GST_GRP * NGROW / 32;
__global__ void __launch_bounds__(32) grad_nodes64_kernel(GradBatch gb, const ConstTables* __restrict__ c) {
  const GradItem gi = grad_item(gb, blockIdx.y);
  TabD* tb = gi.tab;
  const int b = blockIdx.x, lane = threadIdx.x;
  if (b < N64_EH) {
    eh_nodes64(tb, c, b);
  } else if (b < N64_EH + N64_CHI) {
    // chi's step i - 1 -> i (scipy/ode.py:11-19: the right-hand side has no chi in it)
    const int i = (b - N64_EH) * 32 + lane;
    double f[NDIR + 1];
#pragma unroll
    for (int q = 0; q <= NDIR; ++q) f[q] = 0.0;
    if (i > 0) {
      const double w = (c->lna_chi[i] - c->lna_chi[i - 1]) / 6.0;
      chi_rhs(tb->sv, tb->sd[0], c->chi_a[i - 1], c->lna_chi[i - 1], c->chi_ia[i - 1], w, f);
      chi_rhs(tb->sv, tb->sd[0], c->chi_am[i], c->chi_lnam[i], c->chi_iam[i], 4.0 * w, f);
      chi_rhs(tb->sv, tb->sd[0], c->chi_a[i], c->lna_chi[i], c->chi_ia[i], w, f);
    }
    double* o = inc_scratch(tb) + i;
#pragma unroll
    for (int q = 0; q <= NDIR; ++q) o[q * NCHI] = f[q];
  } else {
    growth_step64(tb, c, (b - N64_EH - N64_CHI) * 32 + lane);
  }
}

// The scans: warps 0 .. 7 growth (each the values, then the tangents of its
// direction), 8 .. 16 chi by suffix sums of the increments
constexpr int BG64_THREADS = 32 * (2 * NDIR + 1);
__global__ void __launch_bounds__(BG64_THREADS) grad_bg64_kernel(GradBatch gb, const ConstTables* __restrict__ c) {
  const GradItem gi = grad_item(gb, blockIdx.x);
  TabD* tb = gi.tab;
  const Bg64* m64 = bg_scratch(tb);
  __shared__ double Mv[NGROW * 4], yv[NGROW * 2];
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  if (t == 0) tb->wide = 0;
  for (int i = t; i < NGROW * 4; i += BG64_THREADS) Mv[i] = m64->M[0][i];
  __syncthreads();
  if (warp >= NDIR) {
    const int comp = warp - NDIR;
    const double* inc = inc_scratch(tb) + comp * NCHI;
    double* out = comp ? tb->chid[comp - 1] : tb->chiv;
    double loc[8], x = 0.0;
#pragma unroll
    for (int k = 7; k >= 0; --k) {
      loc[k] = x;
      x += inc[lane * 8 + k];
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double u = __shfl_down_sync(0xffffffffu, x, o);
      if (lane + o < 32) x += u;
    }
    double off = __shfl_down_sync(0xffffffffu, x, 1);
    if (lane == 31) off = 0.0;
#pragma unroll
    for (int k = 0; k < 8; ++k) out[lane * 8 + k] = off + loc[k];
  }
  double d4[4], yf = 0.0;
  if (warp < NDIR) yf = growth_scan_warp(Mv, c->atab_grow[0], 1.0, lane, d4, warp == 0 ? yv : nullptr);
  __syncthreads();
  if (warp < NDIR) {
    // dy_i = M_i dy_{i-1} + dM_i y_{i-1}, dy_0 = 0: a scan of affine maps (A, b)
    const double iyf = 1.0 / yf;
    const double* dMd = m64->dM[warp][0];
    double A[4] = {1.0, 0.0, 0.0, 1.0}, b0 = 0.0, b1 = 0.0, c0[4], c1[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int i = lane * 4 + k;
      const double* m = Mv + i * 4;
      const double* n = dMd + i * 4;
      const double p0 = i > 0 ? yv[2 * i - 2] : 0.0, p1 = i > 0 ? yv[2 * i - 1] : 0.0;
      c0[k] = n[0] * p0 + n[1] * p1;
      c1[k] = n[2] * p0 + n[3] * p1;
      const double e0 = m[0] * b0 + m[1] * b1 + c0[k], e1 = m[2] * b0 + m[3] * b1 + c1[k];
      b0 = e0, b1 = e1;
      if (k == 0) A[0] = m[0], A[1] = m[1], A[2] = m[2], A[3] = m[3];
      else mat2_mul(m, A, A);
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      double P[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) P[q] = __shfl_up_sync(0xffffffffu, A[q], o);
      const double p0 = __shfl_up_sync(0xffffffffu, b0, o), p1 = __shfl_up_sync(0xffffffffu, b1, o);
      if (lane >= o) {
        const double e0 = A[0] * p0 + A[1] * p1 + b0, e1 = A[2] * p0 + A[3] * p1 + b1;
        b0 = e0, b1 = e1;
        mat2_mul(A, P, A);
      }
    }
    double x0 = __shfl_up_sync(0xffffffffu, b0, 1), x1 = __shfl_up_sync(0xffffffffu, b1, 1);
    if (lane == 0) x0 = x1 = 0.0;
    double dy[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const double* m = Mv + (lane * 4 + k) * 4;
      const double e0 = m[0] * x0 + m[1] * x1 + c0[k], e1 = m[2] * x0 + m[3] * x1 + c1[k];
      x0 = e0, x1 = e1;
      dy[k] = x0;
    }
    const double dyf = __shfl_sync(0xffffffffu, x0, 31);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int i = lane * 4 + k;
      const double g = d4[k] * iyf;
      if (warp == 0) tb->gv[i] = g;
      tb->gd[warp][i] = (dy[k] - g * dyf) * iyf;
    }
  }
}

// ---------------------------------------- sigma8, P(k) k^3 and sigma^2(R) ---
constexpr int SG64_THREADS = 256, SG64_R = 64;  // four threads per R
__global__ void __launch_bounds__(SG64_THREADS) grad_sigma64_kernel(GradBatch gb, const ConstTables* __restrict__ c) {
  const GradItem gi = grad_item(gb, blockIdx.y);
  TabD* tb = gi.tab;
  const int comp = blockIdx.x % (NDIR + 1), part = blockIdx.x / (NDIR + 1), t = threadIdx.x;
  const double* u = eh_scratch(tb);
  const double* ud = u + comp * NEH;
  if (comp > NPW) {
    // no tangent: the tables' zeros
    for (int i = part * SG64_R + t; t < SG64_R && i < NRT; i += NRT) tb->sigd[comp - 1][i] = 0.0;
    if (part == 0) {
      for (int i = t; i < NKH; i += SG64_THREADS) tb->pk3d[comp - 1][i] = 0.0;
      if (t == 0) tb->sd[comp - 1][S_SIGMASQR8] = tb->sd[comp - 1][S_PKNORM] = 0.0;
    }
    return;
  }
  __shared__ double sums[4][SG64_R], norm[2];
  __shared__ double pq[NKH];
  const double i2 = 1.0 / (2.0 * (PI * PI));
  if (t < 32) {
    // sigmasqr(8) (power.py:70-78): romb is linear in the integrand's values
    double a = 0.0, b = 0.0;
    for (int e = t; e < NROMB; e += 32) a = fma(c->romb_w[e], u[e], a), b = fma(c->romb_w[e], ud[e], b);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      a += __shfl_xor_sync(0xffffffffu, a, o);
      b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    // P(k) normalisation sigma8^2 / sigmasqr(8) (power.py:47) and its tangent
    const double sig = i2 * a, dsig = i2 * b, s8 = tb->sv[S_SIGMA8], pn = s8 * s8 / sig;
    const double ds8 = comp ? tb->sd[comp - 1][S_SIGMA8] : 0.0;
    const double dpn = comp ? (2.0 * s8 * ds8 - pn * dsig) / sig : 0.0;
    if (t == 0) {
      norm[0] = pn, norm[1] = dpn;
      if (part == 0 && comp == 0) tb->sv[S_SIGMASQR8] = sig, tb->sv[S_PKNORM] = pn;
      if (part == 0 && comp != 0) tb->sd[comp - 1][S_SIGMASQR8] = dsig, tb->sd[comp - 1][S_PKNORM] = dpn;
    }
  }
  __syncthreads();
  const double pn = norm[0], dpn = norm[1];
  // P(k_i, a = 1) k_i^3 (the growth table is normalised to 1 at a = 1)
  for (int i = t; i < NKH; i += SG64_THREADS) {
    const double v = u[NROMB + i], p = (comp ? ud[NROMB + i] * pn + v * dpn : v * pn) * c->kh3[i];
    if (part == 0) (comp ? tb->pk3d[comp - 1] : tb->pk3v)[i] = p;
    pq[i] = c->simpson_kh[i] * (p * i2);
    if (part == 0) {
      const FF f = px_of(pq[i]);
      grad_kw64(tb)[comp * NKH + i] = make_float2(f.hi, f.lo);
    }
  }
  __syncthreads();
  const int q = t / SG64_R, jj = t % SG64_R, j = part * SG64_R + jj;
  double acc = 0.0;
#pragma unroll 8
  for (int i = q; i < NKH; i += 4) acc = fma(pq[i], c->E[i * NRT + j], acc);
  sums[q][jj] = acc;
  __syncthreads();
  if (q == 0) (comp ? tb->sigd[comp - 1] : tb->sigv)[j] = (sums[0][jj] + sums[1][jj]) + (sums[2][jj] + sums[3][jj]);
}
static_assert(NRT % SG64_R == 0, "whole parts of the R nodes");

void launch_grad_tables64(const GradBatch& gb, const ConstTables* c, cudaStream_t st) {
  grad_nodes64_kernel<<<dim3(N64_EH + N64_CHI + N64_GROW, gb.n_items), 32, 0, st>>>(gb, c);
  grad_bg64_kernel<<<gb.n_items, BG64_THREADS, 0, st>>>(gb, c);
  grad_sigma64_kernel<<<dim3((NDIR + 1) * (NRT / SG64_R), gb.n_items), SG64_THREADS, 0, st>>>(gb, c);
}

}  // namespace jcg
