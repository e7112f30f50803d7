// phx_weno.cuh -- WENO5-Z of the production build with its nonlinear weights
// on the integer pipe.
//
// A flux kernel is bound by the FP64 pipe (64-76 cycles per warp instruction
// of a sub-partition); integer instructions take one to five cycles on pipes
// that are otherwise idle.  Of the scheme's 81 FP64 instructions per variable and
// cell, 51 form the smoothness indicators and the weights: sums and products
// of positive numbers, which here are 63-bit significands with an int
// exponent (products through three 32 x 32 -> 64 bit multiplications).  What
// stays in FP64: the second differences a_k and slopes b_k (in the
// reference's order: near-flat regions follow their rounding), the slopes of
// the limiter, and the final weighted sums, 30 instructions.  Against the
// weights in FP64 (random, smooth, stepped, near-flat stencils; 128-bit
// values) the face states' errors are no larger: 2.5e-16 of the stencil's
// largest value at most, 6e-16 in FP64.
//
// With beta_k = 13/3 a_k^2 + b_k^2 + eps, tau = |beta_2 - beta_0|, M and m
// the larger and smaller of beta_0 and beta_2, b = beta_1, X = M + tau = 2 M - m
// and Y = b + tau, the weights gamma_k (1 + tau / beta_k) are proportional to
//   om = M (M b) (stencil of m),  oM = X (m b) (stencil of M),  o1 = Y (m M),
// and R = sum_k beta_k / (beta_k + tau) = Q / (M X Y), Q = Y (m X + M^2) + b M X.
// In tenths the sums are Sa = om + 6 o1 + 3 oM (the face for which m's
// stencil has gamma = 1/10) and Sb = 3 om + 6 o1 + oM (the other one).  With
// T = m b M^2 X Y and U = 5 T / (Q Sa Sb (Sa + Sb)) -- one reciprocal -- the
// coefficients of (a_k +- 3 b_k), which carry the candidates' 1/12, the
// normalisation and the blend factor alpha = 60 T / (Q (Sa + Sb)), are
// U Sb {om, 6 o1, 3 oM} and U Sa {3 om, 6 o1, oM}, and alpha / 4 = 3 U Sa Sb.
#pragma once
#include <cuda_runtime.h>

namespace phx {
namespace weno {

typedef unsigned long long u64;
typedef long long i64;

// m 2^(e - 63); m in [2^62, 2^63) where normalised, always below 2^63
struct Num {
  u64 m;
  int e;
};
__device__ __forceinline__ u64 mulh(u64 a, u64 b) {  // a b / 2^64, a, b < 2^63 (up to two units low)
  const unsigned ah = (unsigned)(a >> 32), al = (unsigned)a, bh = (unsigned)(b >> 32), bl = (unsigned)b;
  const u64 mid = (u64)ah * bl + (u64)al * bh;
  return (u64)ah * bh + (mid >> 32);
}
__device__ __forceinline__ Num mul(Num a, Num b) { return {mulh(a.m, b.m), a.e + b.e + 1}; }
__device__ __forceinline__ Num norm(Num a) {  // a nonzero high word
  const int n = __clz((int)(a.m >> 32)) - 1;
  return {a.m << n, a.e - n};
}
__device__ __forceinline__ u64 shr(u64 m, int n) { return m >> min(n, 63); }  // n >= 0
__device__ __forceinline__ Num add(Num a, Num b) {
  const int e = max(a.e, b.e) + 1;
  return {shr(a.m, e - a.e) + shr(b.m, e - b.e), e};
}
// |x|; 0 for zero and subnormals
__device__ __forceinline__ Num unpack(double x) {
  const unsigned hi = (unsigned)__double2hiint(x);
  const int ex = (int)((hi >> 20) & 0x7ffu);
  const u64 m = (((u64)((hi & 0xfffffu) | 0x100000u) << 32) | (unsigned)__double2loint(x)) << 10;
  return {ex ? m : 0ull, ex ? ex - 1022 : -4000};
}
// nearest double (values below the normal range: a number of that size)
__device__ __forceinline__ double pack(Num a) {
  a = norm(a);
  const int f = max(a.e + 1021, 0);
  return __longlong_as_double((i64)(((u64)f << 52) + ((a.m + 512) >> 10)));
}
// 1 / a, a normalised: the FP32 seed and one third-order step in fixed point
// (as rcp_nr, with 58 bits of a)
__device__ __forceinline__ Num rcp(Num a) {
  const unsigned hi = (unsigned)(a.m >> 32);
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(0x3f800000u | ((hi >> 7) & 0x7fffffu))));
  const unsigned b = min(max(__float_as_uint(r), 0x3f000000u), 0x3f7fffffu);
  const unsigned R0 = (b & 0x7fffffu) | 0x800000u;
  const i64 e = (i64)(0ull - (a.m >> 5) * R0);  // e 2^81
  const int eh = (int)(e >> 37);
  const i64 q = (e >> 5) + (((i64)eh * eh) >> 12);  // (e + e^2) 2^76
  const i64 t = (i64)R0 * (q >> 16);
  return {((u64)R0 << 38) + (u64)(t >> 22), 2 - a.e};
}

// beta = 13/3 a^2 + b^2 + 1e-100, normalised (the eps enters where it would not
// be rounded away; a^2 and b^2 of subnormals count as 0).  bad: not finite, or
// beyond the range the limiter's exponent arithmetic covers.
__device__ __forceinline__ Num beta(double a, double b, bool &bad) {
  const Num A = unpack(a), B = unpack(b), eps = {0x6ffcbb923814c000ull, -332};
  const Num a2 = mul(A, A), b2 = mul(B, B);
  const Num s = add(Num{mulh(a2.m, 0x4555555555555555ull), a2.e + 4}, b2);  // 13/24 2^63
  Num r = norm(s);
  bad = bad || r.e > 1800;
  if ((unsigned)(s.m >> 32) == 0u)
    r = eps;
  else if (r.e < -262)
    r = norm(add(r, eps));
  return r;
}

struct Weights {
  double am, a1, aM, bm, b1, bM, aq;
  bool mirror;  // m is beta_2: the faces and the outer stencils change places
};
__device__ __forceinline__ bool weights(double a0, double b0, double a1, double b1, double a2, double b2, Weights &w) {
  bool bad = false;
  const Num be0 = beta(a0, b0, bad), b = beta(a1, b1, bad), be2 = beta(a2, b2, bad);
  if (bad) return false;
  w.mirror = be2.e < be0.e || (be2.e == be0.e && be2.m < be0.m);
  const Num M = w.mirror ? be0 : be2, m = w.mirror ? be2 : be0;
  const u64 ms = shr(m.m, M.e - m.e);
  const Num X = {M.m - (ms >> 1), M.e + 1};  // 2 M - m
  Num t = {M.m - ms, M.e};                   // tau: any number of leading zeros, or 0
  const int nt = __clzll((i64)t.m) - 1;
  t = {t.m << nt, t.m ? t.e - nt : -8000};
  const Num Y = norm(add(b, t));
  const Num mb = mul(m, b), Mb = mul(M, b), MM = mul(M, M);
  const Num om = norm(mul(M, Mb)), oM = norm(mul(X, mb)), o1 = mul(Y, mul(m, M));
  const Num Q = norm(add(mul(Y, norm(add(mul(m, X), MM))), mul(Mb, X)));
  const Num o6 = norm(Num{(o1.m >> 1) + (o1.m >> 2), o1.e + 3});
  const Num m3 = norm(Num{(om.m >> 1) + (om.m >> 2), om.e + 2}), M3 = norm(Num{(oM.m >> 1) + (oM.m >> 2), oM.e + 2});
  const int es = max(max(om.e, oM.e) + 2, o6.e) + 3;
  const u64 s6 = shr(o6.m, es - o6.e);
  const u64 ua = shr(om.m, es - om.e) + s6 + shr(M3.m, es - M3.e);
  const u64 ub = shr(m3.m, es - m3.e) + s6 + shr(oM.m, es - oM.e);
  const Num Sa = norm(Num{ua, es}), Sb = norm(Num{ub, es}), S2 = norm(Num{(ua + ub) >> 1, es + 1});
  const Num D = norm(mul(norm(mul(Sa, Sb)), norm(mul(Q, S2))));
  const Num T = norm(mul(norm(mul(MM, Y)), oM));
  const Num U = norm(mul(Num{(T.m >> 1) + (T.m >> 3), T.e + 3}, rcp(D)));
  const Num fa = norm(mul(U, Sb)), fb = norm(mul(U, Sa));
  w.am = pack(mul(fa, om));
  w.a1 = pack(mul(fa, o6));
  w.aM = pack(mul(fa, M3));
  w.bm = pack(mul(fb, m3));
  w.b1 = pack(mul(fb, o6));
  w.bM = pack(mul(fb, oM));
  const Num q = mul(fa, Sa);
  w.aq = pack(Num{(q.m >> 1) + (q.m >> 2), q.e + 2});
  return true;
}

}  // namespace weno
}  // namespace phx
