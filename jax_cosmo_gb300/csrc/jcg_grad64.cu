// Tables with tangents of the FP64 gradient (the Jacobian and the vector-
// Jacobian product of angular_cl): background, growth, sigma8, P(k) k^3 and
// sigma^2(R), value and 8 tangents each, float64.
//
// One CTA per cosmology with one tangent direction per lane spent 1.45 ms on
// them: 1,154 node evaluations on one SM's FP64 pipe (2 lanes per clock), the
// value repeated in every direction, then serial scans by single lanes.  Here
//   grad_eh64_kernel      Eisenstein-Hu at the 386 Romberg and P(k) nodes, one
//     node per thread, CTAs of a warp: T and its partials in the 11 inputs by a
//     reverse sweep, then the 8 directions by one product each;
//   grad_bg64_kernel      the chi and growth nodes by thread, tangents in closed
//     form; chi by suffix sums, growth by scans of the RK4 steps' matrices and of
//     their tangents' affine maps, a warp per component;
//   grad_sigma64_kernel   sigma8's weighted sum, P(k) k^3 and sigma^2(R): a CTA per
//     component and quarter of the R nodes.
// One cosmology 1,453 -> 119 us (75 + 23 + 21), 61 cosmologies 1,456 -> 210 us; what is left is
// latency: serial float64 code of a thread, the scans and 257 loads of E per R.
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

__global__ void __launch_bounds__(32) grad_eh64_kernel(GradBatch gb, const ConstTables* __restrict__ c) {
  const GradItem gi = grad_item(gb, blockIdx.y);
  TabD* tb = gi.tab;
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
  const int e = blockIdx.x * 32 + lane;
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
  for (int d = 0; d < NDIR; ++d) {
    double x = 0.0;
#pragma unroll
    for (int q = 0; q < NX - 1; ++q) x = fma(a[q], dl[q][d], x);
    out[(1 + d) * NEH] = fma(t2, x, v * lk * dl[NX - 1][d]);
  }
}

// -------------------------------------------------------------- background --
constexpr int BG64_THREADS = 512;
constexpr int BG64_SMEM = (int)sizeof(double) * ((NDIR + 1) * (2 * NCHI + 4 * NGROW) + NSCAL * (NDIR + 1) + 2 * NGROW);

// E^2 with its tangents: values shared by the chi and growth nodes
struct E2D {
  double e2, ef, d[NDIR], def[NDIR];
};
__device__ __forceinline__ E2D e2_grad(const double* s, const double* sd, double a, double lna, double ia) {
  E2D r;
  const double f = -3.0 * (1.0 + s[S_W0] + s[S_WA]) * lna + 3.0 * s[S_WA] * (a - 1.0);
  r.ef = exp(f);
  const double ia2 = ia * ia, ia3 = ia2 * ia;
  r.e2 = s[S_OMEGA_M] * ia3 + s[S_OMEGA_K] * ia2 + s[S_OMEGA_DE] * r.ef;
#pragma unroll
  for (int d = 0; d < NDIR; ++d) {
    const double* t = sd + d * NSCAL;
    const double df = -3.0 * (t[S_W0] + t[S_WA]) * lna + 3.0 * t[S_WA] * (a - 1.0);
    r.def[d] = t[S_OMEGA_DE] * r.ef + s[S_OMEGA_DE] * r.ef * df;  // d(Omega_de exp(f_de))
    r.d[d] = t[S_OMEGA_M] * ia3 + t[S_OMEGA_K] * ia2 + r.def[d];
  }
  return r;
}

__global__ void __launch_bounds__(BG64_THREADS) grad_bg64_kernel(GradBatch gb, const ConstTables* __restrict__ c) {
  const GradItem gi = grad_item(gb, blockIdx.x);
  TabD* tb = gi.tab;
  extern __shared__ __align__(16) double sm[];
  double* s = sm;                            // [NSCAL]
  double* sd = s + NSCAL;                    // [NDIR][NSCAL]
  double* fn = sd + NDIR * NSCAL;            // [NDIR + 1][NCHI] chi right-hand sides at the nodes
  double* fm = fn + (NDIR + 1) * NCHI;       // at the midpoints
  double* qr = fm + (NDIR + 1) * NCHI;       // [4][NDIR + 1][NGROW] growth coefficients qa, ra, qm, rm
  double* yv = qr + 4 * (NDIR + 1) * NGROW;  // [NGROW][2] growth solution
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  if (t == 0) tb->wide = 0;
  for (int i = t; i < NSCAL; i += BG64_THREADS) s[i] = tb->sv[i];
  for (int i = t; i < NDIR * NSCAL; i += BG64_THREADS) sd[i] = tb->sd[i / NSCAL][i % NSCAL];
  __syncthreads();
  // dchi/dln a = R_H / (a sqrt(E^2)) at nodes and midpoints (background.py:227-231)
  if (t < 2 * NCHI && t != NCHI) {
    const bool mid = t > NCHI;
    const int i = mid ? t - NCHI : t;
    const double a = mid ? c->chi_am[i] : c->chi_a[i], lna = mid ? c->chi_lnam[i] : c->lna_chi[i];
    const double ia = mid ? c->chi_iam[i] : c->chi_ia[i];
    const E2D e = e2_grad(s, sd, a, lna, ia);
    const double r = rsqrt(e.e2), f = RH * ia * r, h = -0.5 * f * (r * r);
    double* dst = (mid ? fm : fn) + i;
    dst[0] = f;
#pragma unroll
    for (int d = 0; d < NDIR; ++d) dst[(1 + d) * NCHI] = h * e.d[d];
  }
  // growth ODE coefficients D'' = -q D' + r D (background.py:96-106)
  if (t < 2 * NGROW && t != NGROW) {
    const bool mid = t > NGROW;
    const int i = mid ? t - NGROW : t;
    const double a = mid ? c->grow_am[i] : c->atab_grow[i], lna = mid ? c->grow_lnam[i] : c->grow_lna[i];
    const double ia = mid ? c->grow_iam[i] : c->grow_ia[i];
    const E2D e = e2_grad(s, sd, a, lna, ia);
    const double ie = 1.0 / e.e2, ia2 = ia * ia, ia3 = ia2 * ia;
    const double om = s[S_OMEGA_M] * ia3 * ie, de = s[S_OMEGA_DE] * e.ef * ie;
    const double w1 = 1.0 + 3.0 * (s[S_W0] + (1.0 - a) * s[S_WA]);
    double* q = qr + (mid ? 2 * (NDIR + 1) * NGROW : 0) + i;
    double* r = q + (NDIR + 1) * NGROW;
    q[0] = (2.0 - 0.5 * (om + w1 * de)) * ia;
    r[0] = 1.5 * om * ia2;
#pragma unroll
    for (int d = 0; d < NDIR; ++d) {
      const double* td = sd + d * NSCAL;
      const double dom = (td[S_OMEGA_M] * ia3 - om * e.d[d]) * ie, dde = (e.def[d] - de * e.d[d]) * ie;
      const double dw1 = 3.0 * (td[S_W0] + (1.0 - a) * td[S_WA]);
      q[(1 + d) * NGROW] = -0.5 * (dom + w1 * dde + dw1 * de) * ia;
      r[(1 + d) * NGROW] = 1.5 * dom * ia2;
    }
  }
  __syncthreads();
  // One RK4 step is linear in y = (D, dD/da), y_i = M_i y_{i-1}, with
  // K1 = A0, K2 = Am (1 + h/2 K1), K3 = Am (1 + h/2 K2), K4 = A1 (1 + h K3),
  // M = 1 + h/6 (K1 + 2 K2 + 2 K3 + K4), A = [[0, 1], [r, -q]]; dM by the same
  // products.  Threads 0 .. 127: M_i and dM_i of the 8 directions, in place of the
  // coefficients once every thread has read its own.
  double M[4] = {1.0, 0.0, 0.0, 1.0}, dM[NDIR][4];
#pragma unroll
  for (int d = 0; d < NDIR; ++d) dM[d][0] = dM[d][1] = dM[d][2] = dM[d][3] = 0.0;
  if (t >= 1 && t < NGROW) {
    constexpr int ST = (NDIR + 1) * NGROW;
    const double* Q = qr;
    const double h = c->atab_grow[t] - c->atab_grow[t - 1], h2 = 0.5 * h;
    const double q0 = Q[t - 1], r0 = Q[ST + t - 1], qm = Q[2 * ST + t], rm = Q[3 * ST + t], q1 = Q[t], r1 = Q[ST + t];
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
    for (int d = 0; d < NDIR; ++d) {
      const double* D = Q + (1 + d) * NGROW;
      const double dq0 = D[t - 1], dr0 = D[ST + t - 1], dqm = D[2 * ST + t], drm = D[3 * ST + t], dq1 = D[t],
                   dr1 = D[ST + t];
      const double x2 = h2 * dr0, x3 = -h2 * dq0;  // dX2 = [[0, 0], [x2, x3]]
      const double k0 = x2, k1 = x3, k2 = drm * X2[0] - dqm * X2[2] - qm * x2, k3 = drm * X2[1] - dqm * X2[3] - qm * x3;
      const double a0 = h2 * k0, a1 = h2 * k1, a2 = h2 * k2, a3 = h2 * k3;  // dX3
      const double l0 = a2, l1 = a3, l2 = drm * X3[0] - dqm * X3[2] + rm * a0 - qm * a2,
                   l3 = drm * X3[1] - dqm * X3[3] + rm * a1 - qm * a3;
      const double b0 = h * l0, b1 = h * l1, b2 = h * l2, b3 = h * l3;  // dX4
      const double m2 = dr1 * X4[0] - dq1 * X4[2] + r1 * b0 - q1 * b2, m3 = dr1 * X4[1] - dq1 * X4[3] + r1 * b1 - q1 * b3;
      dM[d][0] = h6 * (2.0 * (k0 + l0) + b2);
      dM[d][1] = h6 * (2.0 * (k1 + l1) + b3);
      dM[d][2] = h6 * (dr0 + 2.0 * (k2 + l2) + m2);
      dM[d][3] = h6 * (-dq0 + 2.0 * (k3 + l3) + m3);
    }
  } else if (warp >= 4 && warp < 4 + NDIR + 1) {
    // chi (background.py:227-233), value and tangents
    const int comp = warp - 4;
    chi_scan_warp<true>(fn + comp * NCHI, fm + comp * NCHI, c->lna_chi, lane, comp ? tb->chid[comp - 1] : tb->chiv);
  }
  __syncthreads();
  double* Mv = qr;                 // [NGROW][4]
  double* dMv = qr + 4 * NGROW;    // [NDIR][NGROW][4]
  if (t < NGROW) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      Mv[t * 4 + q] = M[q];
#pragma unroll
      for (int d = 0; d < NDIR; ++d) dMv[(d * NGROW + t) * 4 + q] = dM[d][q];
    }
  }
  __syncthreads();
  double d4[4], yf = 0.0;
  if (warp < NDIR) yf = growth_scan_warp(Mv, c->atab_grow[0], 1.0, lane, d4, warp == 0 ? yv : nullptr);
  __syncthreads();
  if (warp < NDIR) {
    // dy_i = M_i dy_{i-1} + dM_i y_{i-1}, dy_0 = 0: a scan of affine maps (A, b)
    const double iyf = 1.0 / yf;
    const double* dMd = dMv + (size_t)warp * NGROW * 4;
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
constexpr int SG64_THREADS = 64;
__global__ void __launch_bounds__(SG64_THREADS) grad_sigma64_kernel(GradBatch gb, const ConstTables* __restrict__ c) {
  const GradItem gi = grad_item(gb, blockIdx.y);
  TabD* tb = gi.tab;
  const int comp = blockIdx.x % (NDIR + 1), part = blockIdx.x / (NDIR + 1), t = threadIdx.x;
  const double* u = eh_scratch(tb);
  const double* ud = u + comp * NEH;
  __shared__ double red[2][2];
  __shared__ double pq[NKH];
  // sigmasqr(8) (power.py:70-78): romb is linear in the integrand's values
  double a = 0.0, b = 0.0;
  for (int e = t; e < NROMB; e += SG64_THREADS) a = fma(c->romb_w[e], u[e], a), b = fma(c->romb_w[e], ud[e], b);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
  }
  if ((t & 31) == 0) red[t >> 5][0] = a, red[t >> 5][1] = b;
  __syncthreads();
  const double i2 = 1.0 / (2.0 * (PI * PI));
  const double sig = i2 * (red[0][0] + red[1][0]), dsig = i2 * (red[0][1] + red[1][1]);
  // P(k) normalisation sigma8^2 / sigmasqr(8) (power.py:47) and its tangent
  const double s8 = tb->sv[S_SIGMA8], pn = s8 * s8 / sig;
  const double ds8 = comp ? tb->sd[comp - 1][S_SIGMA8] : 0.0;
  const double dpn = comp ? (2.0 * s8 * ds8 - pn * dsig) / sig : 0.0;
  if (t == 0 && part == 0) {
    if (comp == 0) {
      tb->sv[S_SIGMASQR8] = sig;
      tb->sv[S_PKNORM] = pn;
    } else {
      tb->sd[comp - 1][S_SIGMASQR8] = dsig;
      tb->sd[comp - 1][S_PKNORM] = dpn;
    }
  }
  // P(k_i, a = 1) k_i^3 (the growth table is normalised to 1 at a = 1)
  for (int i = t; i < NKH; i += SG64_THREADS) {
    const double v = u[NROMB + i], p = (comp ? ud[NROMB + i] * pn + v * dpn : v * pn) * c->kh3[i];
    if (part == 0) (comp ? tb->pk3d[comp - 1] : tb->pk3v)[i] = p;
    pq[i] = c->simpson_kh[i] * (p / (2.0 * (PI * PI)));
    if (part == 0) {
      const FF f = px_of(pq[i]);
      grad_kw64(tb)[comp * NKH + i] = make_float2(f.hi, f.lo);
    }
  }
  __syncthreads();
  const int j = part * SG64_THREADS + t;
  double acc = 0.0;
  for (int i = 0; i < NKH; ++i) acc = fma(pq[i], c->E[i * NRT + j], acc);
  (comp ? tb->sigd[comp - 1] : tb->sigv)[j] = acc;
}
static_assert(NRT % SG64_THREADS == 0, "whole parts of the R nodes");

void launch_grad_tables64(const GradBatch& gb, const ConstTables* c, cudaStream_t st) {
  grad_eh64_kernel<<<dim3((NEH + 31) / 32, gb.n_items), 32, 0, st>>>(gb, c);
  cudaFuncSetAttribute(grad_bg64_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, BG64_SMEM);
  grad_bg64_kernel<<<gb.n_items, BG64_THREADS, BG64_SMEM, st>>>(gb, c);
  grad_sigma64_kernel<<<dim3((NDIR + 1) * (NRT / SG64_THREADS), gb.n_items), SG64_THREADS, 0, st>>>(gb, c);
}

}  // namespace jcg
