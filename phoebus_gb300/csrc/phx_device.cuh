// phx_device.cuh -- per-zone FP64 physics of the phoebus fluid hot path, on
// the device.
//
// Every function follows the operation order of the phoebus source it cites
// (paths relative to the phoebus tree), so that the exact build (nvcc
// -fmad=false) reproduces a CPU build without FMA contraction bit for bit.
// Minkowski is folded at compile time: with gcov = diag(-1,1,1,1), lapse 1,
// shift 0, each metric contraction of the reference reduces to the same
// sequence of roundings on its nonzero terms (x * 1 = x, s + (+-0) = s), so the
// folded form is bit-identical for finite states and saves most of the FP64
// work of the general contraction.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/phx_fluid.h"
#include "phx_math.h"
#include "phx_weno.cuh"

namespace phx {

// ------------------------------------------------------------ robust.hpp
constexpr double kSMALL = 10 * 2.2250738585072014e-308;  // 10 * DBL_MIN
constexpr double kEPS = 10 * 2.220446049250313e-16;      // 10 * DBL_EPSILON
constexpr double kDBLMAX = 1.7976931348623157e308;

// Comparisons of doubles on the integer pipe (an FP64 comparison holds the
// FP64 pipe like an FMA): order_bits is increasing in x (-0 below +0, NaN
// with a clear sign bit on top).  max_num / min_num return the other operand
// where one is NaN, as fmax / fmin do.  gt_bits takes +0 above -0; where that
// matters, gt below compares as the IEEE > does.
__device__ __forceinline__ long long order_bits(double x) {
  const long long b = __double_as_longlong(x);
  return b ^ ((b >> 63) & 0x7fffffffffffffffll);
}
__device__ __forceinline__ double from_order_bits(long long k) {
  return __longlong_as_double(k ^ ((k >> 63) & 0x7fffffffffffffffll));
}
__device__ __forceinline__ bool gt_bits(double a, double b) { return order_bits(a) > order_bits(b); }
// order_bits with -0 equal to +0
__device__ __forceinline__ long long value_bits(double x) {
  const long long b = __double_as_longlong(x);
  return b >= 0 ? b : (long long)(0x8000000000000000ull - (unsigned long long)b);
}
__device__ __forceinline__ bool nan_bits(double x) {
  return (__double_as_longlong(x) & 0x7fffffffffffffffll) > 0x7ff0000000000000ll;
}
__device__ __forceinline__ double max_num(double a, double b) {
  return nan_bits(a) || (gt_bits(b, a) && !nan_bits(b)) ? b : a;
}
__device__ __forceinline__ double min_num(double a, double b) {
  return nan_bits(a) || (gt_bits(a, b) && !nan_bits(b)) ? b : a;
}

// std::max / std::min as the reference calls them: the first argument comes
// back when the comparison is false, so a NaN there propagates (fmax / fmin
// would drop it).  The exact build keeps that for bit-for-bit parity on
// every input, NaN states included; the production build uses max_num /
// min_num (the two differ only where an argument is NaN, or for zeros of
// different sign).
__device__ __forceinline__ double rmax(double a, double b) {
#ifdef PHX_EXACT
  return (a < b) ? b : a;
#else
  return max_num(a, b);
#endif
}
__device__ __forceinline__ double rmin(double a, double b) {
#ifdef PHX_EXACT
  return (b < a) ? b : a;
#else
  return min_num(a, b);
#endif
}
// fmax(0, x)
__device__ __forceinline__ double clamp0(double x) {
#ifdef PHX_EXACT
  return fmax(0.0, x);
#else
  const long long b = __double_as_longlong(x);
  return b <= 0x7ff0000000000000ll && b > 0 ? x : 0.0;
#endif
}
// a > b (false where either is NaN, and for two zeros of any sign)
__device__ __forceinline__ bool gt(double a, double b) {
#ifdef PHX_EXACT
  return a > b;
#else
  return value_bits(a) > value_bits(b) && !nan_bits(a) && !nan_bits(b);
#endif
}
__device__ __forceinline__ bool is_nan(double x) {
#ifdef PHX_EXACT
  return isnan(x);
#else
  return nan_bits(x);
#endif
}
__device__ __forceinline__ double make_positive(double v) { return rmax(v, kEPS); }
__device__ __forceinline__ double make_bounded(double v, double vmin, double vmax) {
  return rmin(rmax(v, vmin + kEPS), vmax * (1.0 - kEPS));
}
__device__ __forceinline__ double ratio(double a, double b) {
  const double sgn = b >= 0 ? 1.0 : -1.0;
  return a / (b + sgn * kSMALL);
}

// 1/x and 1/sqrt(x) on the FP32 and integer pipes.  An FP64 instruction holds
// a sub-partition's FP64 pipe for 64-76 cycles, an integer one takes one to
// five, and the issue slots beside the FP64 pipe are mostly free; so these
// use no FP64 instruction (three and five, on the hardware's FP64 seeds,
// before).  With x = 2^E M / 2^52 (M the 53-bit significand), the FP32
// approximation of 1 / M gives a 24-bit integer R0 with relative error
// e = 1 - x r0 below 2^-21; e comes exactly from the low 64 bits of M R0, and
// r0 (1 + e + e^2) is formed in 62-bit fixed point (e^3 < 2^-63), rounded to 53 bits.
// Within 0.508 ulp of the exact value over 2.8e7 arguments, for seeds up to
// three units off.  Callers guarantee a normal, finite argument (rsqrt: > 0)
// with an exponent field in [16, 2030].
__device__ __forceinline__ unsigned seed24(float r) {  // a seed in [1/2, 1] as 24 bits
  const unsigned b = min(max(__float_as_uint(r), 0x3f000000u), 0x3f7fffffu);
  return (b & 0x7fffffu) | 0x800000u;
}
__device__ __forceinline__ double rcp_nr(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(0x3f800000u | ((hi & 0xfffffu) << 3) | (lo >> 29))));
  const unsigned R0 = seed24(r);
  const unsigned long long M = ((unsigned long long)((hi & 0xfffffu) | 0x100000u) << 32) | lo;
  const long long e = (long long)(0ull - M * R0);  // e 2^76; 2^76 - M R0 modulo 2^64
  const int eh = (int)(e >> 32);
  const long long q = e + (((long long)eh * eh) >> 12);             // (e + e^2) 2^76
  const long long t = (long long)R0 * (q >> 16);                    // r0 (e + e^2) 2^84
  const unsigned long long R = ((unsigned long long)R0 << 38) + (unsigned long long)(t >> 22);  // r 2^62, r in (1/2, 1]
  const unsigned long long m = (R + 256) >> 9;
  const unsigned long long ex = (unsigned long long)((2044u - ((hi >> 20) & 0x7ffu)) | ((hi >> 31) << 11)) << 52;
  return __longlong_as_double((long long)(ex + m));
}
// biased exponent of a double, on the integer pipe
__device__ __forceinline__ int dexp(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }

// 1/x for the production build (IEEE division in the exact build); falls back
// to the division when x is outside the normal range the Newton form handles.
__device__ __forceinline__ double rcp_p(double x) {
#ifdef PHX_EXACT
  return 1.0 / x;
#else
  const int e = dexp(x);
  return (e >= 16 && e <= 2030) ? rcp_nr(x) : 1.0 / x;
#endif
}
// a / b: IEEE division in the exact build, a * rcp_p(b) in the production build
__device__ __forceinline__ double div_p(double a, double b) {
#ifdef PHX_EXACT
  return a / b;
#else
  return a * rcp_p(b);
#endif
}
// 1/sqrt(x) likewise: X = x 2^-2k in [1, 4), y0 = 2^-24 Y0 from the FP32
// approximation, g = 1 - X y0^2 from the middle bits of X Y0^2, and
// y0 (1 + g/2 + 3 g^2 / 8) in fixed point (the next term is below 2^-64).
// Within 0.508 ulp.  The production build's replacement for 1 / sqrt(x); the
// exact build divides.
__device__ __forceinline__ double rsqrt_nr(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const int E = (int)((hi >> 20) & 0x7ffu) - 1023;
  const int odd = E & 1;
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;"
      : "=f"(y)
      : "f"(__uint_as_float((0x3f800000u + ((unsigned)odd << 23)) | ((hi & 0xfffffu) << 3) | (lo >> 29))));
  const unsigned Y0 = seed24(y);
  const unsigned long long X = (((unsigned long long)((hi & 0xfffffu) | 0x100000u) << 32) | lo) << odd;
  const unsigned long long A = (unsigned long long)Y0 * Y0;
  const unsigned Ah = (unsigned)(A >> 32), Al = (unsigned)A, Xh = (unsigned)(X >> 32), Xl = (unsigned)X;
  const unsigned long long G = (unsigned long long)Xh * Al + (unsigned long long)Xl * Ah + __umulhi(Xl, Al) +
                               ((unsigned long long)(Xh * Ah) << 32);
  const long long g = -(long long)G;  // g 2^68
  const int g24 = (int)(g >> 24);
  const long long q = (g >> 1) + ((3 * ((long long)g24 * g24)) >> 23);
  const long long t = (long long)Y0 * (q >> 8);  // y0 (...) 2^84
  const unsigned long long R = ((unsigned long long)Y0 << 38) + (unsigned long long)(t >> 22);
  const unsigned long long m = (R + 256) >> 9;
  return __longlong_as_double((long long)(((unsigned long long)(1021 - ((E - odd) >> 1)) << 52) + m));
}
__device__ __forceinline__ double rsqrt_p(double x) {
#ifdef PHX_EXACT
  return 1.0 / sqrt(x);
#else
  const int e = dexp(x);
  return (e >= 16 && e <= 2030) ? rsqrt_nr(x) : 1.0 / sqrt(x);
#endif
}
// robust::ratio with the production-build reciprocal
__device__ __forceinline__ double ratio_p(double a, double b) {
#ifdef PHX_EXACT
  return ratio(a, b);
#else
  const int e = dexp(b);  // kSMALL is below half an ulp of b from an exponent of -960 on
  if (e >= 64 && e <= 2030) return a * rcp_nr(b);
  const double sgn = b >= 0 ? 1.0 : -1.0;
  return a * rcp_p(b + sgn * kSMALL);
#endif
}

// ---------------------------------------------------------- parameters
// Device copy of the fluid / fixup / eos params (phx_params), with the
// fixup package's defaults already resolved (fixup.cpp:120-180).
// Reconstructed variables the flux kernels read from memory.  The exact
// build reconstructs all PHX_NRECON, as the reference does
// (fluid.cpp:272-286).  Under the ideal gas gamma1 = bulk modulus / P is the
// constant Gamma (every zone's stored value is Gamma to a few ulps), so the
// production build reconstructs the first PHX_NRECON - 1 and gives both face
// states gamma1 = Gamma (recon_gamma1): one variable fewer staged, held in
// registers and reconstructed per cell and direction.
#ifdef PHX_EXACT
constexpr int kReconLoad = PHX_NRECON;
#else
constexpr int kReconLoad = PHX_NRECON - 1;
static_assert(PHX_PGM1 == PHX_NRECON - 1, "gamma1 is the last reconstructed variable");
#endif

struct Par {
  double gm1, Cv;
  double rho_min_eos, sie_min_eos;
  double c2p_tol;
  int c2p_max_iter;
  double fsf;  // c2p_floor_scale_fac
  int fail_on_floors, fail_on_ceilings;
  int mhd;
  int floor_type;
  double r0, s0, ralpha, salpha;
  double g0, smax0;
  double bsqorho0, bsqou0;
  int recon, riemann;
  double cfl;
  int c2p_fixup, strategy_floors, enable_floors, enable_mhd_floors;
  double vsq_max;  // 1 - 1 / g0^2 (the gamma ceiling as a v^2 bound)
  double iCv;      // 1 / Cv, formed on the host (production-build temperature)
  int fix_flux;      // fixup/enable_flux_fixup
  int inflow_check;  // fixup/enable_ox1_fmks_inflow_check
};

// Face states of gamma1 where the production build does not reconstruct it.
__device__ __forceinline__ void recon_gamma1(const Par &p, double *ql, double *qr) {
  if constexpr (kReconLoad < PHX_NRECON) {
    ql[PHX_PGM1] = p.gm1 + 1.0;
    qr[PHX_PGM1] = p.gm1 + 1.0;
  }
}

// ------------------------------------------------ singularity-eos IdealGas
__device__ __forceinline__ double eos_P_rho_sie(const Par &p, double rho, double sie) {
  return clamp0(p.gm1 * rho * sie);
}
__device__ __forceinline__ double eos_T_rho_sie(const Par &p, double rho, double sie) {
#ifdef PHX_EXACT
  return clamp0(div_p(sie, p.Cv));
#else
  return clamp0(sie * p.iCv);  // production build: the host's 1/Cv
#endif
}
__device__ __forceinline__ double eos_P_rho_T(const Par &p, double rho, double T) {
  return clamp0(p.gm1 * rho * p.Cv * T);
}
__device__ __forceinline__ double eos_bmod_rho_T(const Par &p, double rho, double T) {
  return clamp0((p.gm1 + 1) * p.gm1 * rho * p.Cv * T);
}
__device__ __forceinline__ double eos_bmod_rho_sie(const Par &p, double rho, double sie) {
  return clamp0(p.gm1 * (p.gm1 + 1) * rho * sie);
}

// ------------------------------------------------------- fixup.hpp Bounds
// Bounds::GetFloors in two parts.  floor_point holds what depends on the
// position only (for ExpX1RhoSie two exponentials); floors_from finishes
// the floors from it and the density passed in (only ExpX1RhoU's sie floor
// depends on that density).  A zone's con2prim evaluates its floors at every
// residual and both states of a face at the face's position, so they compute
// floor_point once and reuse it: the same values as get_floors, bit for bit.
struct FloorPt {
  double r, s;
};
__device__ __forceinline__ FloorPt floor_point(const Par &p, double x1, double x2, double x3) {
  FloorPt f;
  switch (p.floor_type) {
  case PHX_FLOOR_CONSTANT_RHO_SIE:
    f.r = p.r0;
    f.s = p.s0;
    break;
  case PHX_FLOOR_EXPX1_RHO_SIE:
  case PHX_FLOOR_EXPX1_RHO_U:  // s: the sie floor's numerator
    f.r = p.r0 * phx_math::exp(p.ralpha * x1);
    f.s = p.s0 * phx_math::exp(p.salpha * x1);
    break;
  case PHX_FLOOR_X1_RHO_SIE:
    f.r = p.r0 * fmin(1.0, phx_math::pow(x1, p.ralpha));
    f.s = p.s0 * fmin(1.0, phx_math::pow(x1, p.salpha));
    break;
  default: {
    double r = sqrt(x1 * x1 + x2 * x2 + x3 * x3);
    f.r = p.r0 * fmin(1.0, phx_math::pow(r, p.ralpha));
    f.s = p.s0 * fmin(1.0, phx_math::pow(r, p.salpha));
  } break;
  }
  return f;
}
// True when the floors depend on X1 alone (all types but RRhoSie).
__device__ __forceinline__ bool floors_x1_only(const Par &p) { return p.floor_type != PHX_FLOOR_R_RHO_SIE; }
__device__ __forceinline__ void floors_from(const Par &p, const FloorPt &f, double &rflr, double &sflr) {
  if (p.floor_type == PHX_FLOOR_EXPX1_RHO_U) {
    sflr = f.s / rmax(rflr, f.r);
  } else {
    sflr = f.s;
  }
  rflr = f.r;
  rflr = rmax(rflr, p.rho_min_eos);
  sflr = rmax(sflr, p.sie_min_eos);
}
__device__ __forceinline__ void get_floors(const Par &p, double x1, double x2, double x3,
                                           double &rflr, double &sflr) {
  floors_from(p, floor_point(p, x1, x2, x3), rflr, sflr);
}

// ------------------------------------------------------------ block view
struct BView {
  int n1t, n2t, n3t, ndim, ng, nx1, nx2, nx3;
  long long vs;
  double x0[3], dx[3];
  double *prim, *cons, *flux, *face_sig, *cell_sig, *fail, *src, *emf, *dudt;
  const double *gcent, *gface1, *gface2, *gderiv;
  // floor_point's (r, s) at the n1t cell centres and then the n1t + 1 faces
  // along X1, or null: a plan's views hold it where the floors depend on X1 alone
  // and are not constant (two exponentials, 40 FP64 instructions, at every
  // zone or face otherwise).
  const double2 *flr;
  int fmks;
  __device__ __forceinline__ long long idx(int k, int j, int i) const {
    return ((long long)k * n2t + j) * n1t + i;
  }
  __device__ __forceinline__ double Xc(int d, int ix) const { return x0[d] + (ix + 0.5) * dx[d]; }
  __device__ __forceinline__ double Xf(int d, int ix) const { return x0[d] + ix * dx[d]; }
  __device__ __forceinline__ int is() const { return ng; }
  __device__ __forceinline__ int ie() const { return ng + nx1 - 1; }
  __device__ __forceinline__ int js() const { return ndim >= 2 ? ng : 0; }
  __device__ __forceinline__ int je() const { return ndim >= 2 ? ng + nx2 - 1 : 0; }
  __device__ __forceinline__ int ks() const { return ndim >= 3 ? ng : 0; }
  __device__ __forceinline__ int ke() const { return ndim >= 3 ? ng + nx3 - 1 : 0; }
};

// floor_point of the cell centre / X1 face i, from the view's table where it
// has one (the same values: the table is floor_point's)
__device__ __forceinline__ FloorPt floor_load(const double2 *t) {
  const double2 v = __ldg(t);
  return FloorPt{v.x, v.y};
}
__device__ __forceinline__ const double2 *floor_cell(const BView &b, int i) { return b.flr ? b.flr + i : nullptr; }
__device__ __forceinline__ const double2 *floor_face1(const BView &b, int i) {
  return b.flr ? b.flr + b.n1t + i : nullptr;
}

// ------------------------------------------------------------- geometry
// Point geometry (values at a cell centre or a face).
struct Pt {
  double alpha, beta[3], gcov[4][4], gamcon[3][3], detgam;
};

__device__ __forceinline__ int flat2(int m, int n) {
  // Flatten2 (geometry_utils.hpp:180-185): symmetric 4x4 packing
  const int lo = m < n ? m : n, hi = m < n ? n : m;
  return hi * (hi + 1) / 2 + lo;
}

// loc: 0 = centre (and X3 face), 1 = X1 face, 2 = X2 face
__device__ __forceinline__ void load_pt(const BView &b, int loc, int j, int i, Pt &p) {
  const double *t;
  long long pitch, off;
  if (loc == 1) {
    t = b.gface1;
    pitch = (long long)b.n2t * (b.n1t + 1);
    off = (long long)j * (b.n1t + 1) + i;
  } else if (loc == 2) {
    t = b.gface2;
    pitch = (long long)(b.n2t + 1) * b.n1t;
    off = (long long)j * b.n1t + i;
  } else {
    t = b.gcent;
    pitch = (long long)b.n2t * b.n1t;
    off = (long long)j * b.n1t + i;
  }
  p.alpha = __ldg(t + PHX_G_ALPHA * pitch + off);
#pragma unroll
  for (int d = 0; d < 3; d++) p.beta[d] = __ldg(t + (PHX_G_BETA + d) * pitch + off);
#pragma unroll
  for (int m = 0; m < 4; m++)
#pragma unroll
    for (int n = 0; n < 4; n++) p.gcov[m][n] = __ldg(t + (PHX_G_GCOV + flat2(m, n)) * pitch + off);
#pragma unroll
  for (int m = 0; m < 3; m++)
#pragma unroll
    for (int n = 0; n < 3; n++) p.gamcon[m][n] = __ldg(t + (PHX_G_GAMCON + flat2(m, n)) * pitch + off);
  p.detgam = __ldg(t + PHX_G_DETGAM * pitch + off);
}

// Point geometry of zone q from a [PHX_GEOM_NLOC][pitch] table.
__device__ __forceinline__ void load_pt_flat(const double *t, long long pitch, long long q, Pt &p) {
  p.alpha = __ldg(t + PHX_G_ALPHA * pitch + q);
#pragma unroll
  for (int d = 0; d < 3; d++) p.beta[d] = __ldg(t + (PHX_G_BETA + d) * pitch + q);
#pragma unroll
  for (int m = 0; m < 4; m++)
#pragma unroll
    for (int n = 0; n < 4; n++) p.gcov[m][n] = __ldg(t + (PHX_G_GCOV + flat2(m, n)) * pitch + q);
#pragma unroll
  for (int m = 0; m < 3; m++)
#pragma unroll
    for (int n = 0; n < 3; n++) p.gamcon[m][n] = __ldg(t + (PHX_G_GAMCON + flat2(m, n)) * pitch + q);
  p.detgam = __ldg(t + PHX_G_DETGAM * pitch + q);
}

// a_m = gamma_mn a^n (the spatial metric lowers a vector).
__device__ __forceinline__ void lower_sp(const Pt &g, const double a[3], double out[3]) {
#pragma unroll
  for (int m = 0; m < 3; m++) out[m] = g.gcov[m + 1][1] * a[0] + g.gcov[m + 1][2] * a[1] + g.gcov[m + 1][3] * a[2];
}
__device__ __forceinline__ double dot3(const double a[3], const double b[3]) {
  return a[0] * b[0] + a[1] * b[1] + a[2] * b[2];
}

// sum_{m,n} gcov[m+1][n+1] a[m] b[n]: the reference's nine-term loop in the
// exact build; a . (gamma b) in the production build (12 FP64 instructions
// instead of 18).
template <bool MINK>
__device__ __forceinline__ double dot_sp(const Pt &g, const double a[3], const double b[3]) {
  if constexpr (MINK) {
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2];
  } else {
#ifdef PHX_EXACT
    double s = 0.0;
#pragma unroll
    for (int m = 0; m < 3; m++)
#pragma unroll
      for (int n = 0; n < 3; n++) s += g.gcov[m + 1][n + 1] * a[m] * b[n];
    return s;
#else
    double bl[3];
    lower_sp(g, b, bl);
    return dot3(a, bl);
#endif
  }
}

// ------------------------------------------------- relativity_utils.hpp
template <bool MINK>
__device__ __forceinline__ double lorentz(const Pt &g, const double v[3]) {
  return sqrt(1. + dot_sp<MINK>(g, v, v));
}

// The outer-X1 inflow check of one ghost zone (ConvertBoundaryConditions,
// phoebus_boundaries.cpp:366-397): where u^1 = v^1 - W beta^1 / alpha < 0,
// the three-velocity v / W keeps its X2 and X3 components, takes
// beta^1 / alpha along X1, and is turned back into W v.  v: W v^i in place.
__device__ __forceinline__ void ox1_inflow_fix(const Pt &gm, double v[3]) {
  double W = lorentz<false>(gm, v);
  const double ucon1 = v[0] - W * gm.beta[0] / gm.alpha;
  if (ucon1 < 0) {
    double vcon[3] = {v[0] / W, v[1] / W, v[2] / W};
    vcon[0] = gm.beta[0] / gm.alpha;
    const double vsq = dot_sp<false>(gm, vcon, vcon);
    W = 1. / sqrt(1. - vsq);
    for (int d = 0; d < 3; d++) v[d] = W * vcon[d];
  }
}

// ---------------------------------------------------------- prim2con.hpp
// signal_speeds (prim2con.hpp:24-46); ndim entries written.
template <bool MINK>
__device__ __forceinline__ void signal_speeds(double rho, double u, double p, double bsq,
                                              const double v[3], double vsq, double gam1,
                                              const Pt &g, double *sig) {
  const double rho_rel = rho + u + p;
#ifdef PHX_EXACT
  const double vasq = div_p(bsq, rho_rel + bsq);
  double cssq = div_p(gam1 * p, rho_rel);
#else
  // production build: one reciprocal of the product of the two denominators
  // where it is normal
  double vasq, cssq;
  const double dAB = (rho_rel + bsq) * rho_rel;
  const int eAB = dexp(dAB);
  if (eAB >= 16 && eAB <= 2030) {
    const double rAB = rcp_nr(dAB);
    vasq = bsq * (rho_rel * rAB);
    cssq = gam1 * p * ((rho_rel + bsq) * rAB);
  } else {
    vasq = div_p(bsq, rho_rel + bsq);
    cssq = div_p(gam1 * p, rho_rel);
  }
#endif
#ifdef PHX_EXACT
  cssq += vasq - cssq * vasq;
  const double alpha = MINK ? 1.0 : g.alpha;
  const double vcoff = div_p(alpha, 1.0 - vsq * cssq);
#pragma unroll
  for (int m = 0; m < 3; m++) {
    const double gmm = MINK ? 1.0 : g.gamcon[m][m];
    const double vpm = sqrt(cssq * (1.0 - vsq) * (gmm * (1.0 - vsq * cssq) - v[m] * v[m] * (1.0 - cssq)));
    double vp = vcoff * (v[m] * (1.0 - cssq) + vpm);
    double vm = vcoff * (v[m] * (1.0 - cssq) - vpm);
    if constexpr (!MINK) {
      vp -= g.beta[m];
      vm -= g.beta[m];
    }
    sig[m] = rmax(fabs(vp), fabs(vm));
  }
#else
  // production build: max(|a + e|, |a - e|) = |a| + e with a = c v (1 - cs^2) - beta
  // and e = c sqrt(...) >= 0; sqrt(x) as x rsqrt(x) for normal x > 0 (zero,
  // negative and extreme arguments take the IEEE square root)
  cssq = fma(vasq, 1.0 - cssq, cssq);
  const double c1 = 1.0 - cssq, Q = fma(-vsq, cssq, 1.0), k = cssq * (1.0 - vsq);
  const double vcoff = MINK ? rcp_p(Q) : g.alpha * rcp_p(Q);
#pragma unroll
  for (int m = 0; m < 3; m++) {
    const double t = v[m] * c1;
    const double rad = k * fma(-v[m], t, MINK ? Q : g.gamcon[m][m] * Q);
    const int ev = __double2hiint(rad) >> 20;  // biased exponent, negative for rad < 0
    const double vpm = (ev >= 16 && ev <= 2030) ? rad * rsqrt_nr(rad) : sqrt(rad);
    const double a = MINK ? vcoff * t : fma(vcoff, t, -g.beta[m]);
    sig[m] = fma(vcoff, vpm, fabs(a));
  }
#endif
}

// p2c (prim2con.hpp:48-102)
template <bool MINK>
__device__ __forceinline__ void p2c(double rho, const double vp[3], const double b[3], double u,
                                    double p, double gam1, const Pt &g, double gdet, double &D,
                                    double S[3], double bcons[3], double &tau, double *sig) {
  const double W = lorentz<MINK>(g, vp);
  const double iW = rcp_p(W);
  double v[3] = {vp[0] * iW, vp[1] * iW, vp[2] * iW};
  double vsq, Bsq, Bdotv;
  if constexpr (MINK) {
    // the reference accumulates the three sums interleaved; each is independent
    vsq = v[0] * v[0] + v[1] * v[1] + v[2] * v[2];
    Bsq = b[0] * b[0] + b[1] * b[1] + b[2] * b[2];
    Bdotv = b[0] * v[0] + b[1] * v[1] + b[2] * v[2];
  } else {
    vsq = 0.0;
    Bsq = 0.0;
    Bdotv = 0.0;
#pragma unroll
    for (int ii = 0; ii < 3; ii++)
#pragma unroll
      for (int jj = 0; jj < 3; jj++) {
        vsq += g.gcov[ii + 1][jj + 1] * v[ii] * v[jj];
        Bsq += g.gcov[ii + 1][jj + 1] * b[ii] * b[jj];
        Bdotv += g.gcov[ii + 1][jj + 1] * b[ii] * v[jj];
      }
  }
  const double b0 = W * Bdotv;
  const double alpha = MINK ? 1.0 : g.alpha;
  double bcon[4];
  bcon[0] = W * Bdotv / alpha;
#pragma unroll
  for (int m = 0; m < 3; m++) {
    if constexpr (MINK)
      bcon[m + 1] = b[m] * iW + Bdotv * W * v[m];
    else
      bcon[m + 1] = b[m] * iW + Bdotv * W * (v[m] - g.beta[m] / alpha);
  }
  const double bsq = Bsq * iW * iW + Bdotv * Bdotv;
  double bcov[3];
#pragma unroll
  for (int m = 0; m < 3; m++) {
    if constexpr (MINK) {
      bcov[m] = bcon[m + 1];
    } else {
      bcov[m] = 0.0;
#pragma unroll
      for (int n = 0; n < 4; n++) bcov[m] += g.gcov[m + 1][n] * bcon[n];
    }
  }
  D = gdet * rho * W;
  const double rho_rel = (rho + u + p + bsq) * W * W;
#pragma unroll
  for (int m = 0; m < 3; m++) {
    double vcov;
    if constexpr (MINK) {
      vcov = v[m];
    } else {
      vcov = 0.0;
#pragma unroll
      for (int n = 0; n < 3; n++) vcov += g.gcov[m + 1][n + 1] * v[n];
    }
    S[m] = gdet * (rho_rel * vcov - b0 * bcov[m]);
    bcons[m] = gdet * b[m];
  }
  tau = gdet * (rho_rel - (p + 0.5 * bsq) - b0 * b0) - D;
  if (sig != nullptr) signal_speeds<MINK>(rho, u, p, bsq, v, vsq, gam1, g, sig);
}

// -------------------------------------------------- reconstruction.hpp
__device__ __forceinline__ double mc(double dm, double dp, double alpha) {
#ifdef PHX_EXACT
  const double dc = (dm * dp > 0.0) * 0.5 * (dm + dp);
#else
  // a select instead of the product with the converted comparison: two fewer
  // FP64 instructions; only the sign of a zero slope can differ
  const double dc = dm * dp > 0.0 ? 0.5 * (dm + dp) : 0.0;
#endif
#ifdef PHX_EXACT
  // std::min (reconstruction.hpp:106): a NaN slope propagates, as fmin would not
  const double m1 = (fabs(dp) < fabs(dm)) ? fabs(dp) : fabs(dm);
  const double m2 = alpha * m1;
  return copysign((m2 < fabs(dc)) ? m2 : fabs(dc), dc);
#else
  return copysign(fmin(fabs(dc), alpha * fmin(fabs(dm), fabs(dp))), dc);
#endif
}
#ifdef PHX_EXACT
__device__ __forceinline__ void recon_plm(double qm, double q0, double qp, double &ql, double &qr) {
  double dq = qp - q0;
  dq = mc(q0 - qm, dq, 1.5);
  ql = q0 + 0.5 * dq;
  qr = q0 - 0.5 * dq;
}
#else
// Production PLM: 5 FP64 instructions.  With dm, dp of one sign, the halved
// slope is min(|dm + dp| / 4, 3/4 min(|dm|, |dp|)), and the first is the
// smaller exactly where the larger of |dm|, |dp| is below twice the other:
// integer comparisons.
__device__ __forceinline__ void recon_plm_fast(double qm, double q0, double qp, double &ql, double &qr) {
  constexpr long long MAG = 0x7fffffffffffffffll;
  const double dm = q0 - qm, dp = qp - q0;
  const long long im = __double_as_longlong(dm), ip = __double_as_longlong(dp);
  const long long am = im & MAG, ap = ip & MAG;
  const bool less = am < ap;
  const long long mn = less ? am : ap, mx = less ? ap : am;
  const bool same = (im ^ ip) >= 0 && mn != 0 && mx <= 0x7ff0000000000000ll;
  const bool mid = mx < mn + (1ll << 52);
  const double s = same ? (mid ? dm + dp : (less ? dm : dp)) : 0.0;
  const double c = mid ? 0.25 : 0.75;
  ql = fma(c, s, q0);
  qr = fma(-c, s, q0);
}
#endif
__device__ __forceinline__ void recon_weno5z(double q0, double q1, double q2, double q3, double q4,
                                             double &ql, double &qr) {
  constexpr double a00 = 1.0 / 3.0, a01 = -7.0 / 6.0, a02 = 11.0 / 6.0;
  constexpr double a10 = -1.0 / 6.0, a11 = 5.0 / 6.0, a12 = 1.0 / 3.0;
  constexpr double a20 = 1.0 / 3.0, a21 = 5.0 / 6.0, a22 = -1.0 / 6.0;
  constexpr double g0 = 0.1, g1 = 0.6, g2 = 0.3;
  constexpr double eps = 1e-100;
  constexpr double t13 = 13.0 / 3.0;
  double a = q0 - 2 * q1 + q2;
  double b = q0 - 4.0 * q1 + 3.0 * q2;
  double beta0 = t13 * a * a + b * b + eps;
  a = q1 - 2.0 * q2 + q3;
  b = q3 - q1;
  double beta1 = t13 * a * a + b * b + eps;
  a = q2 - 2.0 * q3 + q4;
  b = q4 - 4.0 * q3 + 3.0 * q2;
  double beta2 = t13 * a * a + b * b + eps;
  const double tau5 = fabs(beta2 - beta0);
  beta0 = (beta0 + tau5) / beta0;
  beta1 = (beta1 + tau5) / beta1;
  beta2 = (beta2 + tau5) / beta2;
  double w0 = g0 * beta0 + eps;
  double w1 = g1 * beta1 + eps;
  double w2 = g2 * beta2 + eps;
  double wsum = 1.0 / (w0 + w1 + w2);
  ql = w0 * (a00 * q0 + a01 * q1 + a02 * q2);
  ql += w1 * (a10 * q1 + a11 * q2 + a12 * q3);
  ql += w2 * (a20 * q2 + a21 * q3 + a22 * q4);
  ql *= wsum;
  const double alpha_l = 3.0 * wsum * w0 * w1 * w2 / (g2 * w0 * w1 + g1 * w0 * w2 + g0 * w1 * w2) + eps;
  w0 = g0 * beta2 + eps;
  w1 = g1 * beta1 + eps;
  w2 = g2 * beta0 + eps;
  wsum = 1.0 / (w0 + w1 + w2);
  qr = w0 * (a00 * q4 + a01 * q3 + a02 * q2);
  qr += w1 * (a10 * q3 + a11 * q2 + a12 * q1);
  qr += w2 * (a20 * q2 + a21 * q1 + a22 * q0);
  qr *= wsum;
  const double alpha_r = 3.0 * wsum * w0 * w1 * w2 / (g2 * w0 * w1 + g1 * w0 * w2 + g0 * w1 * w2) + eps;
  double dq = q3 - q2;
  dq = mc(q2 - q1, dq, 2.0);
  const double alpha_lin = 2.0 * alpha_l * alpha_r / (alpha_l + alpha_r);
  ql = alpha_lin * ql + (1.0 - alpha_lin) * (q2 + 0.5 * dq);
  qr = alpha_lin * qr + (1.0 - alpha_lin) * (q2 - 0.5 * dq);
}
// ---- production-build WENO5-Z: same mathematics, fewer FP64 instructions.
// WENO5-Z as reconstruction.hpp:127-183, rearranged; the weights and the blend
// factor alpha_lin come from phx_weno.cuh.  With normalised weights
// w_k = gamma_k bp_k / S (bp_k = 1 + tau5 / beta_k; the reference's + eps on
// a weight is below half an ulp of gamma_k bp_k >= 0.1 and drops out),
// alpha = 3 w0 w1 w2 / (g2 w0 w1 + g1 w0 w2 + g0 w1 w2) = 3 / (S R) with
// R = sum_k 1/bp_k, the same for both faces, so the harmonic mean is
// alpha_lin = 6 / (R (S_l + S_r)).
//  - The candidates are q2 + (a_k +- 3 b_k) / 12; the blend
//    alpha q + (1 - alpha) p with p = q2 +- dq2 / 4 is
//    p -+ (alpha / 4) dq2 + sum_k W_k (a_k +- 3 b_k).
//  - The MC slope of the blend, mc(q2 - q1, q3 - q2, 2), doubled, on the
//    integer pipe: the sign test, the minima of magnitudes and the power-of-two
//    scale act on the bit patterns; the sum dm + dp is the slope b1 = q3 - q1
//    the smoothness indicator already forms.
// 30 FP64 instructions for both face states (81 and three reciprocals with
// the weights in FP64): 256^3 fluxes in all three directions 99.0 -> 69.6 ms,
// and 56.6 ms with the flux kernels' loop over the variables rolled.
// Where the weights are refused (values beyond 1e270, not finite) the reference
// sequence is used.
__device__ __forceinline__ void recon_weno5z_fast(double q0, double q1, double q2, double q3, double q4,
                                                  double &ql, double &qr) {
  // second differences a_k and one-sided slopes b_k of the three stencils, in
  // the reference's operation order: in near-flat regions the weights follow
  // the rounding of a_k and b_k (differences of nearly equal indicators), and
  // forming them from first differences instead moved signal speeds of a
  // 256^3 shear layer 1.7e-12 away from the reference's.
  const double a0 = q0 - 2 * q1 + q2, b0 = q0 - 4.0 * q1 + 3.0 * q2;
  const double a1 = q1 - 2.0 * q2 + q3, b1 = q3 - q1;
  const double a2 = q2 - 2.0 * q3 + q4, b2 = q4 - 4.0 * q3 + 3.0 * q2;
  weno::Weights w;
  if (!weno::weights(a0, b0, a1, b1, a2, b2, w)) {
    recon_weno5z(q0, q1, q2, q3, q4, ql, qr);
    return;
  }
  // 2 mc(q2 - q1, q3 - q2, 2) = copysign(min(|dm + dp|, 4 min(|dm|, |dp|)),
  // dm + dp) where dm dp > 0, else 0
  const long long MAG = 0x7fffffffffffffffLL;
  const long long idm = __double_as_longlong(q2 - q1), idp = __double_as_longlong(q3 - q2);
  const long long isum = __double_as_longlong(b1);
  const long long adm = idm & MAG, adp = idp & MAG, asum = isum & MAG;
  const bool same = ((idm ^ idp) >= 0) && adm != 0 && adp != 0;
  const long long a4 = (adm < adp ? adm : adp) + (2LL << 52);
  // mirrored: the roles of the faces and of the outer stencils change, the
  // slopes b1 and dq2 change sign
  const long long flip = w.mirror ? ~MAG : 0;
  const double ds = same ? __longlong_as_double(((asum < a4 ? asum : a4) | (isum & ~MAG)) ^ flip) : 0.0;
  const double bs = __longlong_as_double(isum ^ flip);
  const double am = w.mirror ? a2 : a0, bm = w.mirror ? b2 : b0, aM = w.mirror ? a0 : a2, bM = w.mirror ? b0 : b2;
  const double t = w.aq * ds;
  const double sa = fma(w.am, fma(3.0, bm, am), fma(w.a1, fma(3.0, bs, a1), fma(w.aM, fma(-3.0, bM, aM), -t)));
  const double sb = fma(w.bm, fma(-3.0, bm, am), fma(w.b1, fma(-3.0, bs, a1), fma(w.bM, fma(3.0, bM, aM), t)));
  const double qa = fma(0.25, ds, q2) + sa, qb = fma(-0.25, ds, q2) + sb;
  ql = w.mirror ? qb : qa;
  qr = w.mirror ? qa : qb;
}

#ifdef PHX_EXACT
__device__ __forceinline__ double minmod(double a, double b) {
  return a * b > 0.0 ? (fabs(a) < fabs(b) ? a : b) : 0.0;
}
// MP5 value at the face j+1/2 from f_{j-2} .. f_{j+2}: the monotonicity-
// preserving fifth-order scheme of Suresh & Huynh (1997, J. Comput. Phys.
// 136, 83-99; alpha = 4, eps = 1e-12).  The fifth-order interface value is
// kept when it lies between f_j and the monotonicity bound f_MP; otherwise
// it is clipped to [f_min, f_max], built from the minmod4-limited
// curvatures at j+1/2 and j-1/2 and the upper-limit (UL), average (AV),
// median (MD) and large-curvature (LC) values.  The operations are in the
// order of the reference (reconstruction.hpp:186-244), which bitwise parity
// needs; minmod4(a, b, c, d) is minmod(minmod(a, b), minmod(c, d)).
__device__ __forceinline__ double mp5_face(double fm2, double fm1, double f0, double fp1, double fp2) {
  constexpr double alpha = 4.0, eps = 1.e-12;
  double f = 2.0 * fm2 - 13.0 * fm1 + 47.0 * f0 + 27.0 * fp1 - 3.0 * fp2;
  f /= 60.0;
  const double f_mp = f0 + minmod(fp1 - f0, alpha * (f0 - fm1));
  if ((f - f0) * (f - f_mp) <= eps) return f;
  const double curv_m = fm2 + f0 - 2.0 * fm1;  // second differences at j-1, j, j+1
  const double curv_0 = fm1 + fp1 - 2.0 * f0;
  const double curv_p = f0 + fp2 - 2.0 * fp1;
  const double m4_plus = minmod(minmod(4.0 * curv_0 - curv_p, 4.0 * curv_p - curv_0), minmod(curv_0, curv_p));
  const double m4_minus = minmod(minmod(4.0 * curv_m - curv_0, 4.0 * curv_0 - curv_m), minmod(curv_0, curv_m));
  const double f_ul = f0 + alpha * (f0 - fm1);
  const double f_av = 0.5 * (f0 + fp1);
  const double f_md = f_av - 0.5 * m4_plus;
  const double f_lc = 0.5 * (3.0 * f0 - fm1) + 4.0 / 3.0 * m4_minus;
  const double f_min = fmax(fmin(fmin(f0, fp1), f_md), fmin(fmin(f0, f_ul), f_lc));
  const double f_max = fmin(fmax(fmax(f0, fp1), f_md), fmax(fmax(f0, f_ul), f_lc));
  return f + minmod(f_min - f, f_max - f);  // the median of f, f_min, f_max
}
#else
// Both face values of a cell by the same scheme, in differences from f_j
// (production build): 18 FP64 instructions, 29 where a face is limited
// (38 and about 20 FP64 comparisons per face in mp5_face).  The two faces
// share the differences and the limited curvatures; sign tests, minima and
// the median act on the bit patterns.  Errors relative to the stencil's
// largest value 0.4-0.7 of mp5_face's; a stage over 48 blocks of 16^3 to 64^3
// zones 34.1 -> 17.9 ms (with flux_state).
__device__ __forceinline__ double minmod_bits(double a, double b) {
  constexpr long long MAG = 0x7fffffffffffffffll;
  const long long x = __double_as_longlong(a), y = __double_as_longlong(b);
  return (x ^ y) < 0 ? 0.0 : ((x & MAG) < (y & MAG) ? a : b);
}
// g clipped between f_min and f_max; up = f_{j+1} - f_j, dn = f_j - f_{j-1}
// seen from the face, m4u / m4d the limited curvatures at j+1/2 / j-1/2
__device__ __forceinline__ double mp5_median(double g, double dn, double up, double m4u, double m4d) {
  const long long kd = order_bits(up), kmd = order_bits(0.5 * (up - m4u));
  const long long kul = order_bits(4.0 * dn), klc = order_bits(fma(4.0 / 3.0, m4d, 0.5 * dn));
  const long long lo = max(min(min(0ll, kd), kmd), min(min(0ll, kul), klc));
  const long long hi = min(max(max(0ll, kd), kmd), max(max(0ll, kul), klc));
  const long long k = order_bits(g);
  return from_order_bits(min(max(k, min(lo, hi)), max(lo, hi)));
}
__device__ __forceinline__ void recon_mp5_fast(double q0, double q1, double q2, double q3, double q4, double &ql,
                                               double &qr) {
  constexpr double eps = 1.e-12, c2 = 2.0 / 60.0, c11 = 11.0 / 60.0, c24 = 24.0 / 60.0, c3 = 3.0 / 60.0;
  const double d0 = q1 - q0, d1 = q2 - q1, d2 = q3 - q2, d3 = q4 - q3;
  double gl = fma(c24, d2, fma(c11, d1, fma(-c3, d3, -c2 * d0)));   // f_{j+1/2} - f_j
  double gr = fma(-c24, d1, fma(-c11, d2, fma(c3, d0, c2 * d3)));   // f_{j-1/2} - f_j
  const double ml = minmod_bits(d2, 4.0 * d1), mr = -minmod_bits(d1, 4.0 * d2);
  const bool sl = gt_bits(gl * (gl - ml), eps) && dexp(gl) != 0x7ff;
  const bool sr = gt_bits(gr * (gr - mr), eps) && dexp(gr) != 0x7ff;
  if (sl || sr) {
    const double cm = d1 - d0, c0 = d2 - d1, cp = d3 - d2;
    const double mp = minmod_bits(minmod_bits(fma(4.0, c0, -cp), fma(4.0, cp, -c0)), minmod_bits(c0, cp));
    const double mm = minmod_bits(minmod_bits(fma(4.0, cm, -c0), fma(4.0, c0, -cm)), minmod_bits(c0, cm));
    if (sl) gl = mp5_median(gl, d1, d2, mp, mm);
    if (sr) gr = mp5_median(gr, -d2, -d1, mm, mp);
  }
  ql = q2 + gl;
  qr = q2 + gr;
}
#endif

// 5-point (or 3-point) reconstruction of one variable.  ql = value at the
// upper face of the cell, qr = value at its lower face.
template <int RECON>
__device__ __forceinline__ void recon(double qm2, double qm1, double q0, double qp1, double qp2,
                                      double &ql, double &qr) {
  if constexpr (RECON == PHX_RECON_WENO5Z) {
#ifdef PHX_EXACT
    recon_weno5z(qm2, qm1, q0, qp1, qp2, ql, qr);
#else
    recon_weno5z_fast(qm2, qm1, q0, qp1, qp2, ql, qr);
#endif
  } else if constexpr (RECON == PHX_RECON_MP5) {
#ifdef PHX_EXACT
    ql = mp5_face(qm2, qm1, q0, qp1, qp2);
    qr = mp5_face(qp2, qp1, q0, qm1, qm2);
#else
    recon_mp5_fast(qm2, qm1, q0, qp1, qp2, ql, qr);
#endif
  } else if constexpr (RECON == PHX_RECON_LINEAR) {
#ifdef PHX_EXACT
    recon_plm(qm1, q0, qp1, ql, qr);
#else
    recon_plm_fast(qm1, q0, qp1, ql, qr);
#endif
  } else {
    ql = q0;
    qr = q0;
  }
}

// ------------------------------------------------------- riemann.hpp
struct Face {
  Pt g;          // face geometry (unused for Minkowski)
  double gdet;   // DetG: 1 for Minkowski, alpha * detgam from the cache
  double gammadet;
  double gdd;
  FloorPt fl;    // floor_point at the face, shared by its two states
};

#ifdef PHX_EXACT
// prim_to_flux (riemann.hpp:88-209) for face direction DIR (0-based), in the
// reference's operations (exact build; flux_state in the production build).
template <bool MINK, int DIR>
__device__ __forceinline__ void prim_to_flux(const Par &par, const Face &f, const double q[PHX_NRECON],
                                             double &vm, double &vp, double U[PHX_NCONS],
                                             double F[PHX_NCONS], double sie_max, double gam_max) {
  const Pt &g = f.g;
  double rho_floor = q[PHX_PRHO];
  double sie_floor;
  floors_from(par, f.fl, rho_floor, sie_floor);
  const double rho = rmax(q[PHX_PRHO], rho_floor);
  double vpcon[3] = {q[PHX_PVEL], q[PHX_PVEL + 1], q[PHX_PVEL + 2]};
  double W = lorentz<MINK>(g, vpcon);
  if (W > gam_max) {
    const double rescale = sqrt((gam_max * gam_max - 1.) / (W * W - 1.));
#pragma unroll
    for (int ii = 0; ii < 3; ii++) vpcon[ii] *= rescale;
  }
  const double qe = q[PHX_PENG];
  double vcon[3] = {vpcon[0] / W, vpcon[1] / W, vpcon[2] / W};
  const double sie_q = q[PHX_PENG] / rho;
  const bool above_floor = sie_q > sie_floor, above_max = sie_q > sie_max;
  double Bcon[3] = {0.0, 0.0, 0.0};
  const double u = (above_floor ? (above_max ? rho * sie_max : qe) : rho * sie_floor);
  const double P = rmax(q[PHX_PPRS], 0.0);
  const double gamma1 = q[PHX_PGM1];
  if (par.mhd) {
    Bcon[0] = q[PHX_PB];
    Bcon[1] = q[PHX_PB + 1];
    Bcon[2] = q[PHX_PB + 2];
  }
  double vsq, Bdotv, BdotB;
  if constexpr (MINK) {
    vsq = vcon[0] * vcon[0] + vcon[1] * vcon[1] + vcon[2] * vcon[2];
    Bdotv = Bcon[0] * vcon[0] + Bcon[1] * vcon[1] + Bcon[2] * vcon[2];
    BdotB = Bcon[0] * Bcon[0] + Bcon[1] * Bcon[1] + Bcon[2] * Bcon[2];
  } else {
    vsq = 0.0;
    Bdotv = 0.0;
    BdotB = 0.0;
#pragma unroll
    for (int m = 0; m < 3; m++)
#pragma unroll
      for (int n = 0; n < 3; n++) {
        vsq += g.gcov[m + 1][n + 1] * vcon[m] * vcon[n];
        Bdotv += g.gcov[m + 1][n + 1] * Bcon[m] * vcon[n];
        BdotB += g.gcov[m + 1][n + 1] * Bcon[m] * Bcon[n];
      }
  }
  const double vsq_max = 1.0 - 1.0 / (gam_max * gam_max);
  if (vsq > vsq_max) {
    double scale = vsq_max / vsq;
    vsq *= scale;
    scale = sqrt(scale);
    Bdotv *= scale;
#pragma unroll
    for (int m = 0; m < 3; m++) vcon[m] *= scale;
  }
  W = 1.0 / sqrt(1 - vsq);
  const double vel = vcon[DIR];
  const double alpha = MINK ? 1.0 : g.alpha;
#define PHX_BOA(m) (g.beta[m] / alpha)
  double vtil;
  if constexpr (MINK)
    vtil = vel;
  else
    vtil = vel - PHX_BOA(DIR);
  U[PHX_CRHO] = rho * W;
  F[PHX_CRHO] = U[PHX_CRHO] * vtil;
  const double b0 = W * Bdotv;
  const double bsq = (BdotB + b0 * b0) / (W * W);
  const double rhohWsq = (rho + u + P) * W * W;
  const double bsqWsq = bsq * W * W;
  const double ptot = P + 0.5 * bsq;
#pragma unroll
  for (int m = 0; m < 3; m++) {
    double bcovm, vcovm;
#define PHX_DIV_W(x) ((x) / W)
    if constexpr (MINK) {
      // gcov[m+1][0] = 0: first term is +-0; then only n = m+1 survives
      bcovm = PHX_DIV_W(Bcon[m]) + b0 * vcon[m];
      vcovm = vcon[m];
    } else {
      bcovm = g.gcov[m + 1][0] * b0 / alpha;
      vcovm = 0.0;
#pragma unroll
      for (int n = 1; n < 4; n++) {
        bcovm += g.gcov[m + 1][n] * (PHX_DIV_W(Bcon[n - 1]) + b0 * (vcon[n - 1] - PHX_BOA(n - 1)));
        vcovm += g.gcov[m + 1][n] * vcon[n - 1];
      }
    }
    U[PHX_CMOM + m] = (rhohWsq + bsqWsq) * vcovm - b0 * bcovm;
    F[PHX_CMOM + m] = U[PHX_CMOM + m] * vtil + ptot * (double)(DIR == m) - PHX_DIV_W(bcovm * Bcon[DIR]);
#undef PHX_DIV_W
  }
  U[PHX_CENG] = rhohWsq + bsqWsq - ptot - b0 * b0 - U[PHX_CRHO];
  F[PHX_CENG] = U[PHX_CENG] * vtil + ptot * vel - Bdotv * Bcon[DIR];
#pragma unroll
  for (int m = 0; m < 3; m++) {
    U[PHX_CB + m] = Bcon[m];
    if constexpr (MINK) {
      F[PHX_CB + m] = U[PHX_CB + m] * vtil - Bcon[DIR] * vcon[m];
    } else {
      F[PHX_CB + m] = U[PHX_CB + m] * vtil - Bcon[DIR] * (vcon[m] - PHX_BOA(m));
    }
  }
#undef PHX_BOA
  const double vasq = bsqWsq / make_positive(rhohWsq + bsqWsq);
  const double cssq = make_bounded(gamma1 * P * W * W / make_positive(rhohWsq), 0.0, 1.0);
  const double cmsq = make_bounded(cssq + vasq * (1.0 - cssq), 0.0, 1.0);
  const double vcoff = div_p(alpha, 1.0 - vsq * cmsq);
  const double v0 = vel * (1.0 - cmsq);
  const double gdd = MINK ? 1.0 : f.gdd;
  const double vpm = sqrt(make_positive(cmsq * (1.0 - vsq) * (gdd * (1.0 - vsq * cmsq) - vel * v0)));
  vp = vcoff * (v0 + vpm);
  vm = vcoff * (v0 - vpm);
  if constexpr (!MINK) {
    vp -= g.beta[DIR];
    vm -= g.beta[DIR];
  }
}
#else
// Production build of one face state: prim_to_flux with the flux left as
// F_m = U_m vtil + G_m, so that the Riemann combination applies vtil once per
// state instead of once per variable, comparisons on the integer pipe, and
// the lowered vectors shared between the contractions.  About 70 FP64
// instructions on Minkowski (82 and 16 FP64 comparisons in prim_to_flux):
// 256^3 WENO5-Z fluxes 56.6 -> 54.9 ms, 64^3 PLM 0.64 -> 0.56 ms (with
// recon_plm_fast).
struct FluxState {
  double U[PHX_NCONS], G[PHX_NCONS], vtil, vm, vp;
};
template <bool MINK, int DIR>
__device__ __forceinline__ void flux_state(const Par &par, const Face &f, const double q[PHX_NRECON], FluxState &s) {
  const Pt &g = f.g;
  // floors_from with integer comparisons
  const double rfl = max_num(f.fl.r, par.rho_min_eos);
  const double rho = max_num(q[PHX_PRHO], rfl);
  double sfl = f.fl.s;
  if (par.floor_type == PHX_FLOOR_EXPX1_RHO_U) sfl = f.fl.s / max_num(q[PHX_PRHO], f.fl.r);
  sfl = max_num(sfl, par.sie_min_eos);
  double v[3] = {q[PHX_PVEL], q[PHX_PVEL + 1], q[PHX_PVEL + 2]};
  double vl[3];  // lowered: W v first, then v
  if constexpr (MINK) {
#pragma unroll
    for (int m = 0; m < 3; m++) vl[m] = v[m];
  } else {
    lower_sp(g, v, vl);
  }
  const double Wsq0 = 1.0 + dot3(v, vl);
  const double iW0 = rsqrt_p(Wsq0);
  double W = Wsq0 * iW0, iW = iW0, c = iW0;
  bool capped = false;
  if (gt_bits(W, par.g0)) {
    c *= sqrt((par.g0 * par.g0 - 1.) / (W * W - 1.));
    capped = true;
  }
#pragma unroll
  for (int m = 0; m < 3; m++) v[m] *= c;
  if constexpr (MINK) {
#pragma unroll
    for (int m = 0; m < 3; m++) vl[m] = v[m];
  } else {
#pragma unroll
    for (int m = 0; m < 3; m++) vl[m] *= c;
  }
  double vsq = dot3(v, vl);
  if (gt_bits(vsq, par.vsq_max)) {
    double scale = par.vsq_max / vsq;
    vsq *= scale;
    scale = sqrt(scale);
#pragma unroll
    for (int m = 0; m < 3; m++) v[m] *= scale;
#pragma unroll
    for (int m = 0; m < 3; m++) vl[m] = MINK ? v[m] : vl[m] * scale;
    capped = true;
  }
  const double ivsq = 1.0 - vsq;
  if (capped) {
    W = rsqrt_p(ivsq);
    iW = ivsq * W;
  }
  // u bounded by rho times the specific energies
  const double qe = q[PHX_PENG], P = max_num(q[PHX_PPRS], 0.0);
  double u = qe;
  const double ufl = rho * sfl, umax = rho * par.smax0;
  if (__double_as_longlong(rho) > 0) {
    if (!(gt_bits(qe, ufl) && !nan_bits(qe)))
      u = ufl;
    else if (gt_bits(qe, umax))
      u = umax;
  } else {
    const double sie = qe * rcp_p(rho);
    u = sie > sfl ? (sie > par.smax0 ? umax : qe) : ufl;
  }
  double B[3] = {0.0, 0.0, 0.0}, Bl[3], Bv = 0.0, BB = 0.0;
  if (par.mhd) {
#pragma unroll
    for (int m = 0; m < 3; m++) B[m] = q[PHX_PB + m];
  }
  if constexpr (MINK) {
#pragma unroll
    for (int m = 0; m < 3; m++) Bl[m] = B[m];
  } else {
    lower_sp(g, B, Bl);
  }
  Bv = dot3(B, vl);
  BB = dot3(B, Bl);
  const double alpha = MINK ? 1.0 : g.alpha;
  const double ialpha = MINK ? 1.0 : rcp_p(alpha);
  const double vel = v[DIR];
  s.vtil = MINK ? vel : fma(-g.beta[DIR], ialpha, vel);
  const double b0 = W * Bv, Wsq = W * W;
  const double bW = fma(b0, b0, BB);       // b^2 W^2
  const double bsq = bW * (iW * iW);
  const double hW = (rho + u + P) * Wsq;   // rho h W^2
  const double ptot = fma(0.5, bsq, P);
  const double tot = hW + bW;
  const double BdW = B[DIR] * iW;
  s.U[PHX_CRHO] = rho * W;
  s.G[PHX_CRHO] = 0.0;
#pragma unroll
  for (int m = 0; m < 3; m++) {
    const double bl = fma(b0, vl[m], Bl[m] * iW);  // b_m (the shift terms cancel)
    s.U[PHX_CMOM + m] = fma(tot, vl[m], -b0 * bl);
    s.G[PHX_CMOM + m] = m == DIR ? fma(-bl, BdW, ptot) : -bl * BdW;
    s.U[PHX_CB + m] = B[m];
    s.G[PHX_CB + m] = -B[DIR] * (MINK ? v[m] : fma(-g.beta[m], ialpha, v[m]));
  }
  s.U[PHX_CENG] = hW + BB - ptot - s.U[PHX_CRHO];
  s.G[PHX_CENG] = fma(ptot, vel, -Bv * B[DIR]);
  // wave speeds; one reciprocal of the product of the two denominators where
  // it is normal
  const double dA = max_num(tot, kEPS), dB = max_num(hW, kEPS);
  const double dAB = dA * dB;
  const int eAB = dexp(dAB);
  const double cP = q[PHX_PGM1] * P * Wsq;
  double vasq, cs;
  if (eAB >= 16 && eAB <= 2030) {
    const double rAB = rcp_nr(dAB);
    vasq = bW * (dB * rAB);
    cs = cP * (dA * rAB);
  } else {
    vasq = bW * rcp_p(dA);
    cs = cP * rcp_p(dB);
  }
  cs = min_num(max_num(cs, kEPS), 1.0 - kEPS);
  const double cm = min_num(max_num(fma(vasq, 1.0 - cs, cs), kEPS), 1.0 - kEPS);
  const double one_vc = fma(-vsq, cm, 1.0);
  const double vc = alpha * rcp_p(one_vc);
  const double v0 = fma(-vel, cm, vel);
  const double rad = max_num(cm * ivsq * fma(-vel, v0, MINK ? one_vc : f.gdd * one_vc), kEPS);
  const double e = vc * (rad * rsqrt_p(rad));
  if constexpr (MINK) {
    s.vp = fma(vc, v0, e);
    s.vm = fma(vc, v0, -e);
  } else {
    const double a = fma(vc, v0, -g.beta[DIR]);
    s.vp = a + e;
    s.vm = a - e;
  }
}
#endif

}  // namespace phx
