// Float64-class elementary functions on the FP32 and integer pipes: the
// numbers of the float64 Limber integrand (jcg_limber64.cu).
//
// GB300 issues FP64 at 1/64 of its FP32 rate, so a value here is a float pair
// (FF: hi + lo, 48-49 significant bits), and a logarithm is a 64-bit fixed
// point number.  An exponent c log2(x) of magnitude 20 keeps 2^-57 absolute
// accuracy in fixed point (float64 would keep 2^-49): exponentials of products
// lose nothing to the size of their argument, and what is left is the pair's
// own rounding, about 1e-15 per operation, of no preferred sign.
//
//   log2 values       int64, 2^-57 units (|log2 x| < 64)
//   exponents c       int64, 2^-60 units (|c| < 8)
//   arguments of 2^Y  int64, 2^-53 units: c x = (c 2^60)(x 2^57) / 2^64
//
// Methods: sums and products by Knuth's two-sum and Dekker's product with
// FMA; 2^Y and log2 by P. T. P. Tang's table-driven method (ACM TOMS 15, 1989
// and 16, 1990): a table of 2^((j + 1/2)/128) / of -log2 of short reciprocals,
// and a Taylor polynomial of the rest, its leading terms in pairs; sin by a
// table of sin and cos of j pi/64 and Taylor polynomials; quotients and the
// cube root by a Newton step from the hardware estimate.
#pragma once

#include <stdint.h>

#include "jcg_fp32.cuh"

namespace jcg {

#define PX_FN __host__ __device__ __forceinline__

struct PxTab {           // shared-memory copy of the constant tables below
  float2 ex[128];        // 2^((j + 1/2)/128) as pairs
  float2 sc[256];        // sin, cos of j pi/64, j = 0..127, interleaved pairs
  float2 ln[256];        // -ln rc[j] as pairs
  long long l2[256];     // -log2 rc[j], 2^-57 units
  float rc[256];         // about 1 / (1 + (j + 1/2)/256), a multiple of 2^-9
};

// (a b) / 2^64 to a unit or two, from the three products that matter (a full
// 64 x 64 bit high product takes 34 FP32 issue slots on GB300)
PX_FN long long px_mulhi(long long a, long long b) {
  const int ah = (int)(a >> 32), bh = (int)(b >> 32);
  const int al = (int)((uint32_t)a >> 1), bl = (int)((uint32_t)b >> 1);
  const long long m = (long long)ah * bl + ((long long)al * bh + (1LL << 30));
  return (long long)ah * bh + (m >> 31);
}
PX_FN float px_asf(uint32_t u) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(u);
#else
  float f;
  __builtin_memcpy(&f, &u, 4);
  return f;
#endif
}
PX_FN uint32_t px_asu(float f) {
#ifdef __CUDA_ARCH__
  return __float_as_uint(f);
#else
  uint32_t u;
  __builtin_memcpy(&u, &f, 4);
  return u;
#endif
}
// hardware estimates of 1 / x, log2 x and 2^x (a few ulp)
PX_FN float px_rcp(float x) {
#ifdef __CUDA_ARCH__
  return rcpf(x);
#else
  return (1.0f / x) * (1.0f + 1.1920929e-7f);
#endif
}
PX_FN float px_lg2e(float x) {
#ifdef __CUDA_ARCH__
  return lg2f(x);
#else
  return (float)__builtin_log2((double)x);
#endif
}
PX_FN float px_ex2e(float x) {
#ifdef __CUDA_ARCH__
  return ex2f(x);
#else
  return (float)__builtin_exp2((double)x);
#endif
}

// ------------------------------------------------------------ pairs -------
PX_FN FF px_f2(float2 v) { return FF{v.x, v.y}; }
PX_FN FF px_of(double v) {
  const float h = (float)v;
  return FF{h, (float)(v - (double)h)};
}
// a positive double between 2^-70 and 2^126 as a pair, and a pair (hi > 0) as a
// double, by integer operations: conversions between float and double issue at
// the FP64 rate (2 per clock and SM)
PX_FN FF px_split(double v) {
#ifdef __CUDA_ARCH__
  const uint32_t h = (uint32_t)__double2hiint(v), l = (uint32_t)__double2loint(v);
#else
  unsigned long long u;
  __builtin_memcpy(&u, &v, 8);
  const uint32_t h = (uint32_t)(u >> 32), l = (uint32_t)u;
#endif
  const float hi = px_asf((((h - 0x38000000u) << 3) | (l >> 29)) + ((l >> 28) & 1u));  // to nearest
  return FF{hi, (float)((int)(l << 3) >> 3) * px_asf(((h >> 20) - 948u) << 23)};
}
PX_FN bool px_tiny(double v) {  // v >= 0 below what px_split takes
#ifdef __CUDA_ARCH__
  return __double2hiint(v) < ((1023 - 70) << 20);
#else
  return v < 8.470329472543003e-22;
#endif
}
PX_FN double px_widen(float v) {  // normal v (0 becomes 2^-127)
  const uint32_t u = px_asu(v), h = (u & 0x80000000u) | (((u & 0x7fffffffu) >> 3) + 0x38000000u), l = u << 29;
#ifdef __CUDA_ARCH__
  return __hiloint2double((int)h, (int)l);
#else
  const unsigned long long w = ((unsigned long long)h << 32) | l;
  double d;
  __builtin_memcpy(&d, &w, 8);
  return d;
#endif
}
PX_FN double px_join(FF a) { return px_widen(a.hi) + px_widen(a.lo); }
// a / b in float64 from the float reciprocal r0 of b: r0 (1 + e + e^2), e = 1 - b r0
PX_FN double px_ddiv(double a, double b, float r0) {
  const double r = px_widen(r0);
  const double e = fma(-b, r, 1.0);
  return a * fma(r, fma(e, e, e), r);
}
PX_FN float px_hi(double v) {  // v truncated to float, v > 0 normal
#ifdef __CUDA_ARCH__
  const uint32_t h = (uint32_t)__double2hiint(v), l = (uint32_t)__double2loint(v);
#else
  unsigned long long u;
  __builtin_memcpy(&u, &v, 8);
  const uint32_t h = (uint32_t)(u >> 32), l = (uint32_t)u;
#endif
  return px_asf(((h - 0x38000000u) << 3) | (l >> 29));
}
PX_FN FF px_norm(float a, float b) {  // |a| >= |b|
  const float s = a + b;
  return FF{s, b - (s - a)};
}
PX_FN FF px_two_sum(float a, float b) {
  const float s = a + b, bb = s - a;
  return FF{s, (a - (s - bb)) + (b - bb)};
}
PX_FN FF px_add(FF a, FF b) {  // same sign, or no cancellation that matters
  const float s = a.hi + b.hi;
  const float bb = s - a.hi;
  const float e = (a.hi - (s - bb)) + (b.hi - bb);
  return px_norm(s, e + (a.lo + b.lo));
}
PX_FN FF px_mul(FF a, FF b) {
  const float p = a.hi * b.hi;
  float e = fmaf(a.hi, b.hi, -p);
  e = fmaf(a.hi, b.lo, e);
  e = fmaf(a.lo, b.hi, e);
  return px_norm(p, e);
}
PX_FN FF px_sqr(FF a) {
  const float p = a.hi * a.hi;
  // lo^2, of one sign, before the rounding: dropped it would bias squares by 6e-16
  const float t = fmaf(a.hi + a.hi, a.lo, a.lo * a.lo);
  return px_norm(p, fmaf(a.hi, a.hi, -p) + t);
}
// Constants as three floats: a pair's rounding (1e-15) is random from node to
// node, a constant's would be the same at all of them.
struct F3 {
  float hi, lo, ll;
};
PX_FN F3 px3_of(double v) {
  const float h = (float)v;
  const double r = v - (double)h;
  const float l = (float)r;
  return F3{h, l, (float)(r - (double)l)};
}
PX_FN FF px_mul(FF a, F3 b) {
  const float p = a.hi * b.hi;
  // the small terms first: each joins the next before that one is rounded
  const float t = fmaf(a.lo, b.hi, fmaf(a.hi, b.lo, a.hi * b.ll));
  return px_norm(p, fmaf(a.hi, b.hi, -p) + t);
}
PX_FN FF px_add(FF a, F3 b) {
  const float s = a.hi + b.hi;
  const float bb = s - a.hi;
  const float e = (a.hi - (s - bb)) + (b.hi - bb);
  return px_norm(s, e + ((a.lo + b.ll) + b.lo));
}
// t += a with the roundings of the high and of the middle float carried on: for
// totals of many terms (a normalised pair addition rounds at 1e-15, and a pair
// whose low part only gathers loses 1e-14 in 33 terms)
PX_FN void px_acc3(F3& t, FF a) {
  const FF w = px_two_sum(t.hi, a.hi);
  const FF m = px_two_sum(t.lo, w.lo);
  const FF n = px_two_sum(m.hi, a.lo);
  t = F3{w.hi, n.hi, t.ll + (m.lo + n.lo)};
}
PX_FN double px_d3(F3 t) { return ((double)t.ll + (double)t.lo) + (double)t.hi; }
PX_FN FF px_1p(FF a) {  // 1 + a
  const float s = 1.f + a.hi;
  const float bb = s - 1.f;
  const float e = (1.f - (s - bb)) + (a.hi - bb);
  return px_norm(s, e + a.lo);
}
// a / b: the float quotient q, rounded right by one correction, then the
// remainder a - q b
PX_FN FF px_div(FF a, FF b) {
  const float r = px_rcp(b.hi);
  const float q0 = a.hi * r;
  const float q = fmaf(fmaf(-q0, b.hi, a.hi), r, q0);
  float m = fmaf(-q, b.hi, a.hi);
  m = fmaf(-q, b.lo, m + a.lo);
  const float q2 = m * r;
  return px_norm(q, fmaf(fmaf(-q2, b.lo, fmaf(-q2, b.hi, m)), r, q2));
}
PX_FN FF px_rcp2(FF b) {  // 1 / b
  const float r0 = px_rcp(b.hi);
  const float r = fmaf(fmaf(-b.hi, r0, 1.f), r0, r0);
  float e = fmaf(-b.hi, r, 1.f);
  e = fmaf(-b.lo, r, e);
  return px_norm(r, r * fmaf(e, e, e));
}
// x^(-1/3): w (1 + d/3 + 2 d^2/9), d = 1 - x w^3, from the estimate w0
// corrected once in float
PX_FN FF px_rcbrt(FF x) {
  const float w0 = px_ex2e(-0.33333334f * px_lg2e(x.hi));
  const float w = fmaf(fmaf(-x.hi * w0, w0 * w0, 1.f), 0.33333334f * w0, w0);
  const float p = w * w, pe = fmaf(w, w, -p);
  const float c = p * w;
  const float ce = fmaf(pe, w, fmaf(p, w, -c));
  const float t = x.hi * c;
  float te = fmaf(x.hi, c, -t);
  te = fmaf(x.hi, ce, te);
  te = fmaf(x.lo, c, te);
  const float d = (1.f - t) - te;
  return px_norm(w, w * (d * fmaf(d, 0.22222222f, 0.33333334f)));
}

// --------------------------------------------------------- fixed point ----
// v in 2^-53 units, 0 <= v < 512 (float to 64-bit integer conversions issue at
// the FP64 rate)
PX_FN long long px_fix53(float v) {
  const uint32_t u = px_asu(v);
  const long long m = (long long)((u & 0x7fffffu) | 0x800000u) << 39;
  const int sh = 136 - (int)((u >> 23) & 255u);  // 39 - (exponent - 97)
  const long long f = sh < 63 ? m >> sh : 0;
  return (int)u < 0 ? -f : f;
}
PX_FN long long px_fix53(FF v) { return px_fix53(v.hi) + px_fix53(v.lo); }

// a fixed point number of 2^-60 units (a logarithm of 2^-57 units: 8 times its
// value) as a pair, from its three pieces of 24, 24 and 16 bits
PX_FN FF px_unfix60(long long v) {
  const float a = (float)(int)(v >> 40) * 9.5367431640625e-07f;                                 // 2^-20
  const float b = (float)(int)((v >> 16) & 0xffffff) * 5.684341886080802e-14f;                  // 2^-44
  const float c = (float)(int)(v & 0xffff) * 8.673617379884035e-19f;                            // 2^-60
  const FF n = px_norm(a, b);
  return px_norm(n.hi, n.lo + c);
}

// 2^Y, Y in 2^-53 units; 0 below 2^-120, infinite from 2^127 on
PX_FN FF px_exp2(long long Y, const PxTab& T) {
  const int hi = (int)(Y >> 32);
  const uint32_t lo = (uint32_t)Y;
  const int e = hi >> 21;
  if (e < -120) return FF{0.f, 0.f};
  const float2 t = T.ex[(hi >> 14) & 127];
  // the 46 bits below the table index: A (upper 23 bits, centred) 2^-30 + B 2^-53
  const uint32_t ua = ((uint32_t)(hi & 0x3fff) << 9) | (lo >> 23);
  const float A = px_asf(0x4b000000u | ua) - 12582912.f;
  const float B = px_asf(0x4b000000u | (lo & 0x7fffffu)) - 8388608.f;
  // z = (A 2^-30 + B 2^-53) ln 2 as a pair, |z| <= 0.0028
  constexpr float C1 = 0.693147182464599609375f * 9.31322574615478515625e-10f;        // float(ln 2) 2^-30
  constexpr float C2 = -1.904654323148236017e-09f * 9.31322574615478515625e-10f;      // (ln 2 - float(ln 2)) 2^-30
  constexpr float C3 = 0.693147182464599609375f * 1.1102230246251565404e-16f;         // float(ln 2) 2^-53
  const float z = A * C1;
  float ze = fmaf(A, C1, -z);
  ze = fmaf(A, C2, ze);
  ze = fmaf(B, C3, ze);
  // s = e^z - 1 = z + z^2/2 + z^3/6 + ...
  const float p = z * z, pe = fmaf(z, z, -p);
  const float h = 0.5f * p;
  const float w = (p * z) * fmaf(z, fmaf(z, 0.0083333333f, 0.041666668f), 0.16666667f);
  const float s = z + h;
  const float sl = (h - (s - z)) + (fmaf(s, ze, fmaf(0.5f, pe, ze)) + w);
  // t (1 + s)
  const float q = t.x * s;
  float ql = fmaf(t.x, s, -q);
  ql = fmaf(t.x, sl, ql);
  ql = fmaf(t.y, s, ql);
  const float r = t.x + q;
  const float rl = (q - (r - t.x)) + (t.y + ql);
  const float sc = e > 126 ? px_asf(0x7f800000u) : px_asf((uint32_t)(e + 127) << 23);
  const FF n = px_norm(r, rl);
  return FF{n.hi * sc, n.lo * sc};
}

// x = 2^e m, m in [1, 2): log1p(m rc - 1) as an unevaluated pair (v, vl), the
// table index j.  The product m rc - 1 is exact in the high part.
PX_FN void px_log_core(FF x, const PxTab& T, int& e, int& j, float& v, float& vl) {
  const uint32_t u = px_asu(x.hi);
  e = (int)(u >> 23) - 127;
  j = (int)((u >> 15) & 255u);
  const float m = px_asf((u & 0x7fffffu) | 0x3f800000u);
  const float ml = x.lo * px_asf((uint32_t)(127 - e) << 23);
  const float rc = T.rc[j];
  const float r = fmaf(m, rc, -1.f), rl = ml * rc;
  const float p = r * r, pe = fmaf(r, r, -p);
  const float h = 0.5f * p;
  const float w = (p * r) * fmaf(r, fmaf(r, fmaf(r, -0.16666667f, 0.2f), -0.25f), 0.33333334f);
  v = r - h;
  vl = ((r - v) - h) + (fmaf(rl, fmaf(-0.5f, rl, p - r), fmaf(-0.5f, pe, rl)) + w);
}
// ln x as a pair, x >= 2
PX_FN FF px_ln(FF x, const PxTab& T) {
  int e, j;
  float v, vl;
  px_log_core(x, T, e, j, v, vl);
  const float2 t = T.ln[j];
  const float ef = (float)e;
  const float a = ef * 0.693147182464599609375f;
  const float ra = fmaf(ef, 0.693147182464599609375f, -a);
  const FF h = px_norm(a, t.x);  // e >= 1: a >= ln 2 >= t
  const FF g = px_norm(h.hi, v);
  const float lo = ((fmaf(ef, -1.904654323148236017e-09f, t.y) + vl) + (ra + h.lo)) + g.lo;
  return px_norm(g.hi, lo);
}
// log2 x in 2^-57 units, x > 0 normal
PX_FN long long px_log2(FF x, const PxTab& T) {
  int e, j;
  float v, vl;
  px_log_core(x, T, e, j, v, vl);
  constexpr float LE = 1.44269502162933349609375f, LEL = 1.92596298909109e-08f;  // log2 e
  const float g0 = v * LE;
  float gl = fmaf(v, LE, -g0);
  gl = fmaf(v, LEL, gl);
  gl = fmaf(vl, LE, gl);
  const float g = g0 + gl;
  gl = gl - (g - g0);
  // g = nA 2^-29 + rest, |nA| < 2^22; the rest in 2^-57 units fits an int
  const float tA = fmaf(g, 536870912.f, 12582912.f);
  const int nA = (int)(px_asu(tA) - 0x4b400000u);
  const float rest = fmaf(tA - 12582912.f, -1.862645149230957e-09f, g) + gl;
#ifdef __CUDA_ARCH__
  const int nB = __float2int_rn(rest * 144115188075855872.f);
#else
  const int nB = (int)__builtin_rint((double)(rest * 144115188075855872.f));
#endif
  return ((long long)e << 57) + T.l2[j] + (((long long)nA << 28) + (long long)nB);
}

// log2 x in 2^-57 units for a positive normal double (once per ell, per a node
// and per cosmology): the same table, the rest in float64, 2^-57 accurate
// where float64 log would leave 2^-51 at log2 x = 10
PX_FN long long px_log2_d(double x, const PxTab& T) {
#ifdef __CUDA_ARCH__
  const long long u = __double_as_longlong(x);
#else
  long long u;
  __builtin_memcpy(&u, &x, 8);
#endif
  const int e = (int)((u >> 52) & 0x7ff) - 1023;
  const int j = (int)((u >> 44) & 255);
  const long long mb = (u & 0xfffffffffffffLL) | 0x3ff0000000000000LL;
#ifdef __CUDA_ARCH__
  const double m = __longlong_as_double(mb);
#else
  double m;
  __builtin_memcpy(&m, &mb, 8);
#endif
  const double r = fma(m, (double)T.rc[j], -1.0);  // |r| <= 0.003
  double p = fma(r, 1.0 / 7.0, -1.0 / 6.0);
  p = fma(p, r, 0.2);
  p = fma(p, r, -0.25);
  p = fma(p, r, 1.0 / 3.0);
  p = fma(p, r, -0.5);
  p = fma(p * r, r, r) * (1.4426950408889634074 * 144115188075855872.0);
#ifdef __CUDA_ARCH__
  const long long f = __double2ll_rn(p);
#else
  const long long f = __builtin_llrint(p);
#endif
  return ((long long)e << 57) + T.l2[j] + f;
}

// sin(pi u), 0 <= u < 2^17; COS: and cos(pi u).  (Beyond, the pair's low float exceeds
// the table's step: 1e-13 at 2^18, no digits from 2^24 on.)
template <bool COS>
PX_FN FF px_sincospi(FF u, const PxTab& T, FF* co) {
  const float n = rintf(u.hi * 64.f);
  const float d0 = fmaf(n, -0.015625f, u.hi);  // exact, 0 or larger than u.lo
  const float d = d0 + u.lo, dl = (d0 - d) + u.lo;
  const int j = ((int)n) & 127;
  // z = pi (d + dl), |z| <= pi/128 (and a little)
  constexpr float P1 = 3.1415927410125732421875f, P2 = -8.74227765734758577309e-08f;
  const float z = d * P1;
  float ze = fmaf(d, P1, -z);
  ze = fmaf(d, P2, ze);
  ze = fmaf(dl, P1, ze);
  const float p = z * z, pe = fmaf(z, z, -p) + (z + z) * ze;
  // sin z = z - z^3/6 + z^5/120 - z^7/5040 (z^3/6 in a pair), cos z = 1 - z^2/2 + z^4/24 - z^6/720
  constexpr float S1 = -0.16666667163372039794921875f, S2 = 4.9670537375e-09f;
  const float c = p * z, ce = fmaf(p, z, -c) + fmaf(pe, z, p * ze);
  const float a = c * S1;
  const float al = fmaf(c, S1, -a) + fmaf(c, S2, ce * S1);
  const float b = (c * p) * fmaf(p, -1.9841270e-4f, 8.3333333e-3f);
  const float s = z + a;
  const float sl = (a - (s - z)) + (ze + (al + b));
  const float k = -0.5f * p;  // cos z - 1
  const float kl = fmaf(-0.5f, pe, (p * p) * fmaf(p, -1.3888889e-3f, 4.1666668e-2f));
  const float2 sj = T.sc[2 * j], cj = T.sc[2 * j + 1];
  // sj + sj (cos z - 1) + cj sin z
  const FF sz = px_norm(s, sl), cz = px_norm(k, kl);
  const FF m1 = px_mul(FF{cj.x, cj.y}, sz);
  const FF m2 = px_mul(FF{sj.x, sj.y}, cz);
  if (COS) {
    const FF n1 = px_mul(FF{-sj.x, -sj.y}, sz);
    const FF n2 = px_mul(FF{cj.x, cj.y}, cz);
    *co = px_add(px_add(n1, n2), FF{cj.x, cj.y});
  }
  return px_add(px_add(m1, m2), FF{sj.x, sj.y});
}
PX_FN FF px_sinpi(FF u, const PxTab& T) { return px_sincospi<false>(u, T, nullptr); }

}  // namespace jcg
