// phx_c2p.cuh -- robust con2prim for one zone on the device
// (con2prim_robust.hpp:46-453, root_find.hpp:27-167).
//
// The regula-falsi loop is warp-synchronous: every lane stays in the loop
// until the warp's vote (__any_sync) says no lane is still iterating, so all
// 32 lanes re-enter each iteration together and reconverge after it.
// In the production build the residual's divisions use the reciprocal on the
// FP32 and integer pipes (rcp_p / ratio_p), and the fast root below comes first;
// the exact build divides and iterates as the reference does.
#pragma once
#include "phx_device.cuh"

namespace phx {

struct Residual {
  double D, q, bsq, bsq_rpsq, rsq, rbsq, v0sq;
  FloorPt fl;  // floor_point of the zone: every evaluation's floors come from it
  double rho_floor, gam_max, e_max;
  bool used_density_floor, used_energy_floor, used_energy_max, used_gamma_max;

  __device__ __forceinline__ void init(const Par &p) {
    double garbage = 0.0;
    rho_floor = 0.0;
    floors_from(p, fl, rho_floor, garbage);
    gam_max = p.g0;
    e_max = p.smax0;
    rho_floor *= p.fsf;
    used_density_floor = used_energy_floor = used_energy_max = used_gamma_max = false;
  }
  __device__ __forceinline__ double x_mu(double mu) const { return ratio_p(1.0, 1.0 + mu * bsq); }
  __device__ __forceinline__ double rbarsq_mu(double mu, double x) const {
    return x * (x * rsq + mu * (1.0 + x) * rbsq);
  }
  __device__ __forceinline__ double qbar_mu(double mu, double x) const {
    const double mux = mu * x;
    return q - 0.5 * (bsq + mux * mux * bsq_rpsq);
  }
  __device__ __forceinline__ double vhatsq_mu(double mu, double rbarsq) {
    const double vsq_trial = mu * mu * rbarsq;
    if (gt(vsq_trial, v0sq)) {
      used_gamma_max = true;
      return v0sq;
    }
    used_gamma_max = false;
    return vsq_trial;
  }
#ifdef PHX_EXACT
  __device__ __forceinline__ double iWhat_mu(double vhatsq) const { return sqrt(1.0 - vhatsq); }
#endif
  __device__ __forceinline__ double rhohat_mu(double iWhat) {
    const double rho_trial = D * iWhat;
    if (!gt(rho_trial, rho_floor) && !is_nan(rho_trial)) {
      used_density_floor = true;
      return rho_floor;
    }
    used_density_floor = false;
    return rho_trial;
  }
#ifdef PHX_EXACT
  __device__ __forceinline__ double ehat_mu(const Par &p, double mu, double qbar, double rbarsq,
                                            double vhatsq, double What) {
    double rho = rhohat_mu(ratio_p(1.0, What));
    double e_floor;
    floors_from(p, fl, rho, e_floor);
    e_floor *= p.fsf;
    const double ehat_trial = What * (qbar - mu * rbarsq) + vhatsq * What * ratio_p(What, 1.0 + What);
    used_energy_floor = false;
    used_energy_max = false;
    if (!gt(ehat_trial, e_floor) && !is_nan(ehat_trial)) {
      used_energy_floor = true;
      return e_floor;
    } else if (gt(ehat_trial, e_max)) {
      used_energy_max = true;
      return e_max;
    }
    return ehat_trial;
  }
#else
  // the energy bounds of ehat_mu at density rho (production build)
  __device__ __forceinline__ double bound_ehat(const Par &p, double rho, double ehat_trial) {
    double e_floor;
    floors_from(p, fl, rho, e_floor);
    e_floor *= p.fsf;
    used_energy_floor = false;
    used_energy_max = false;
    if (!gt(ehat_trial, e_floor) && !is_nan(ehat_trial)) {
      used_energy_floor = true;
      return e_floor;
    } else if (gt(ehat_trial, e_max)) {
      used_energy_max = true;
      return e_max;
    }
    return ehat_trial;
  }
  // ehat_mu with the density from a known 1/W (production build);
  // What = 1 / sqrt(1 - vhatsq): vhatsq What^2 / (1 + What) = What - 1
  __device__ __forceinline__ double ehat_mu_iw(const Par &p, double mu, double qbar, double rbarsq, double vhatsq,
                                               double What, double iWhat) {
    return bound_ehat(p, rhohat_mu(iWhat), fma(What, qbar - mu * rbarsq, What - 1.0));
  }
#endif
  __device__ __forceinline__ double operator()(const Par &p, double mu) {
    const double x = x_mu(mu);
    const double rbarsq = rbarsq_mu(mu, x);
    const double qbar = qbar_mu(mu, x);
    const double vhatsq = vhatsq_mu(mu, rbarsq);
#ifdef PHX_EXACT
    const double iWhat = iWhat_mu(vhatsq);
    const double What = ratio_p(1.0, iWhat);
    const double rhohat = rhohat_mu(iWhat);
    const double ehat = ehat_mu(p, mu, qbar, rbarsq, vhatsq, What);
#else
    // production build: W and 1/W from one rsqrt; the density inside ehat
    // reuses 1/W instead of inverting W again
    const double What = rsqrt_p(1.0 - vhatsq);
    const double iWhat = (1.0 - vhatsq) * What;
    const double rhohat = rhohat_mu(iWhat);
    const double ehat = ehat_mu_iw(p, mu, qbar, rbarsq, vhatsq, What, iWhat);
#endif
    const double Phat = eos_P_rho_sie(p, rhohat, ehat);
    const double hhat = rhohat * (1.0 + ehat) + Phat;
    // Both builds keep the reference's two reciprocals: muhat = 1 / (nuhat +
    // mu rbarsq) with nuhat >= 1 stays <= 1 under rounding, so f(1) >= 0 holds
    // where the root sits at the end of [0, 1] (cold gas); a single merged
    // reciprocal den / (c M + ...) loses that and can leave the root unbracketed.
    const double ahat = div_p(Phat, make_positive(hhat - Phat));
    const double nua = (1.0 + ahat) * (1.0 + ehat) * iWhat;
    const double nub = (1.0 + ahat) * (1.0 + qbar - mu * rbarsq);
    const double nuhat = rmax(nua, nub);
    const double muhat = rcp_p(nuhat + mu * rbarsq);
    return mu - muhat;
  }
  __device__ __forceinline__ bool used_bounds() const {
    return used_density_floor || used_energy_floor || used_energy_max || used_gamma_max;
  }
};

// Outcome of one zone (written back by the caller).
struct C2POut {
  int iterations;
  int evals;
  bool success;
  bool bracketed;
  bool nan_input;
  bool learned;  // the learned start was accepted
};

// Setup of the inversion (con2prim_robust.hpp:303-366).  Returns false when
// the input is NaN (the reference returns failure before touching prims).
// flr: the zone's entry of its view's floor table, or null.
template <bool MINK>
__device__ __forceinline__ bool c2p_setup(const Par &p, const Pt &g, const double U[PHX_NCONS],
                                          double x1, double x2, double x3, Residual &res,
                                          double rcon[3], double rcov[3], double bu[3],
                                          double Bprim[3], double &bdotr, const double2 *flr = nullptr) {
  if (is_nan(U[PHX_CRHO]) || is_nan(U[PHX_CMOM]) || is_nan(U[PHX_CENG])) return false;
  const double gdet = MINK ? 1.0 : g.detgam;
  const double igdet = MINK ? 1.0 : rcp_p(gdet);  // 1 / 1 = 1 in both builds
  double rhoflr = 0.0, epsflr;
  const FloorPt fl = flr ? floor_load(flr) : floor_point(p, x1, x2, x3);
  floors_from(p, fl, rhoflr, epsflr);
  rhoflr *= p.fsf;
  const double gam_max = p.g0;
  const double D = U[PHX_CRHO] * igdet;
  const double tau = U[PHX_CENG] * igdet;
  double bsq = 0.0, bsq_rpsq = 0.0, rbsq = 0.0, rsq;
  bdotr = 0.0;
#ifdef PHX_EXACT
  const double q = ratio_p(tau, D);
  rcov[0] = ratio(U[PHX_CMOM], U[PHX_CRHO]);
  rcov[1] = ratio(U[PHX_CMOM + 1], U[PHX_CRHO]);
  rcov[2] = ratio(U[PHX_CMOM + 2], U[PHX_CRHO]);
#else
  // tau / D = U_tau / U_D: one reciprocal serves q and the three r_i
  const double ic = ratio_p(1.0, U[PHX_CRHO]);
  const double q = U[PHX_CENG] * ic;
  rcov[0] = U[PHX_CMOM] * ic;
  rcov[1] = U[PHX_CMOM + 1] * ic;
  rcov[2] = U[PHX_CMOM + 2] * ic;
#endif
  if constexpr (MINK) {
    rcon[0] = rcov[0];
    rcon[1] = rcov[1];
    rcon[2] = rcov[2];
    rsq = rcon[0] * rcov[0] + rcon[1] * rcov[1] + rcon[2] * rcov[2];
  } else {
    rsq = 0.0;
#pragma unroll
    for (int ii = 0; ii < 3; ii++) {
      rcon[ii] = 0.0;
#pragma unroll
      for (int jj = 0; jj < 3; jj++) rcon[ii] += g.gamcon[ii][jj] * rcov[jj];
      rsq += rcon[ii] * rcov[ii];
    }
  }
  bu[0] = bu[1] = bu[2] = 0.0;
  if (p.mhd) {
#pragma unroll
    for (int ii = 0; ii < 3; ii++) Bprim[ii] = U[PHX_CB + ii] * igdet;
#ifdef PHX_EXACT
    const double sD = rcp_p(sqrt(rmax(D, rhoflr)));
#else
    const double sD = rsqrt_p(rmax(D, rhoflr));
#endif
#pragma unroll
    for (int ii = 0; ii < 3; ii++) {
      bu[ii] = Bprim[ii] * sD;
      bdotr += bu[ii] * rcov[ii];
    }
    bsq = dot_sp<MINK>(g, bu, bu);
    bsq = clamp0(bsq);
    rbsq = bdotr * bdotr;
    bsq_rpsq = bsq * rsq - rbsq;
  }
  const double zsq = rsq / 1.0;  // h0sq_ = 1
#ifdef PHX_EXACT
  const double v0sq = rmin(div_p(zsq, 1.0 + zsq), 1.0 - rcp_p(gam_max * gam_max));
#else
  const double v0sq = rmin(div_p(zsq, 1.0 + zsq), p.vsq_max);  // 1 - 1 / gam_max^2, formed on the host
#endif
  res.D = D;
  res.q = q;
  res.bsq = bsq;
  res.bsq_rpsq = bsq_rpsq;
  res.rsq = rsq;
  res.rbsq = rbsq;
  res.v0sq = v0sq;
  res.fl = fl;
  res.init(p);
  return true;
}

// Inputs of the learned con2prim start (no reference counterpart): scale-free
// invariants of the inversion from the setup quantities, mapped to O(1) in
// FP32: log10 q / 4, log10 r^2 / 4, log10 b^2 / 4, (b.r)^2 / (b^2 r^2),
// v0^2, log10 D / 8 (log10 arguments bounded below by 1e-12, 1e-30).
__device__ __forceinline__ void c2p_features(const Residual &r, float f[6]) {
  f[0] = log10f((float)fmax(r.q, 1e-12)) * 0.25f;
  f[1] = log10f((float)fmax(r.rsq, 1e-12)) * 0.25f;
  f[2] = log10f((float)fmax(r.bsq, 1e-12)) * 0.25f;
  f[3] = (float)r.rbsq / fmaxf((float)r.bsq * (float)r.rsq, 1e-30f);
  f[4] = (float)r.v0sq;
  f[5] = log10f((float)fmax(r.D, 1e-30)) * 0.125f;
}

// The same six invariants for inference, in FP32 arithmetic from the
// conserved variables and the metric (GB300 issues FP32 at 64x its FP64 rate;
// the invariants agree with c2p_setup's FP64 ones to FP32 rounding, far
// below the network's own error).  Returns false for NaN input, as
// c2p_setup does.
template <bool MINK>
__device__ __forceinline__ bool c2p_features_fp32(const Par &p, const Pt &g, const double U[PHX_NCONS], double x1,
                                                  double x2, double x3, float f[6]) {
  if (isnan(U[PHX_CRHO]) || isnan(U[PHX_CMOM]) || isnan(U[PHX_CENG])) return false;
  double rhoflr_d = 0.0, epsflr;
  get_floors(p, x1, x2, x3, rhoflr_d, epsflr);
  const float rhoflr = (float)(rhoflr_d * p.fsf);
  const float igdet = MINK ? 1.0f : 1.0f / (float)g.detgam;
  const float D = (float)U[PHX_CRHO] * igdet;
  const float q = (float)U[PHX_CENG] * igdet / D;
  const float ic = 1.0f / (float)U[PHX_CRHO];
  float rcov[3], rcon[3];
#pragma unroll
  for (int ii = 0; ii < 3; ii++) rcov[ii] = (float)U[PHX_CMOM + ii] * ic;
  float rsq = 0.0f;
#pragma unroll
  for (int ii = 0; ii < 3; ii++) {
    if constexpr (MINK) {
      rcon[ii] = rcov[ii];
    } else {
      rcon[ii] = 0.0f;
#pragma unroll
      for (int jj = 0; jj < 3; jj++) rcon[ii] += (float)g.gamcon[ii][jj] * rcov[jj];
    }
    rsq += rcon[ii] * rcov[ii];
  }
  float bsq = 0.0f, rbsq = 0.0f;
  if (p.mhd) {
    const float sD = rsqrtf(fmaxf(D, rhoflr));
    float bu[3], bdotr = 0.0f;
#pragma unroll
    for (int ii = 0; ii < 3; ii++) {
      bu[ii] = (float)U[PHX_CB + ii] * igdet * sD;
      bdotr += bu[ii] * rcov[ii];
    }
#pragma unroll
    for (int m = 0; m < 3; m++)
#pragma unroll
      for (int n = 0; n < 3; n++) bsq += (MINK ? (m == n ? 1.0f : 0.0f) : (float)g.gcov[m + 1][n + 1]) * bu[m] * bu[n];
    bsq = fmaxf(0.0f, bsq);
    rbsq = bdotr * bdotr;
  }
  const float v0sq = fminf(rsq / (1.0f + rsq), (float)p.vsq_max);
  f[0] = log10f(fmaxf(q, 1e-12f)) * 0.25f;
  f[1] = log10f(fmaxf(rsq, 1e-12f)) * 0.25f;
  f[2] = log10f(fmaxf(bsq, 1e-12f)) * 0.25f;
  f[3] = rbsq / fmaxf(bsq * rsq, 1e-30f);
  f[4] = v0sq;
  f[5] = log10f(fmaxf(D, 1e-30f)) * 0.125f;
  return true;
}

// State of one zone's regula falsi (root_find.hpp:110-167) between
// iterations: the bracket [a, b] with sign-normalised end values, the Illinois
// counters, and the tallies.  Saving and restoring it resumes the same
// sequence of operations.
struct RFState {
  double a, b, ya, yb, sign;
  int it, evals, b1, b2;
  bool bracketed, learned;
};

// Start: refine_bracket + check_bracket (root_find.hpp:42-58, 110-119) from
// [a, b] and guess.  LEARNED: lb = (m, lo, hi), a predicted root and bracket
// in [0, 1]; f(m) picks the half that should hold the root (f < 0 below it,
// > 0 above), one more evaluation checks that half's sign change; when it
// holds, the iterations start from that half, otherwise from the reference's
// own start.  The learned start is only tried for a cold zone (guess = 0, no
// previous solution): a previous mu is the better start (measured: about 1.5
// iterations from it).  A bracket that is not ordered inside [0, 1] (e.g.
// NaN) is not tried.
template <bool LEARNED>
__device__ __forceinline__ void rf_start(const Par &p, Residual &res, bool valid, double a, double b, double guess,
                                         const double *lb, RFState &s) {
  double ya = 0.0, yb = 0.0;
  int evals = 0;
  bool bracketed = true;
  bool started = false;
  s.learned = false;
  if constexpr (LEARNED) {
    if (valid && !(guess > 0.0) && lb[1] >= 0.0 && lb[1] <= lb[0] && lb[0] <= lb[2] && lb[2] <= 1.0) {
      double la, lbb, lya, lyb;
      const double ym = res(p, lb[0]);
      if (ym > 0.0) {
        la = lb[1];
        lbb = lb[0];
        lyb = ym;
        lya = res(p, la);
      } else {
        la = lb[0];
        lbb = lb[2];
        lya = ym;
        lyb = res(p, lbb);
      }
      evals += 2;
      if (lya * lyb <= 0.0) {
        a = la;
        b = lbb;
        ya = lya;
        yb = lyb;
        started = true;
        s.learned = true;
      }
    }
  }
  if (valid && !started) {
    if (a <= guess && b >= guess) {
      ya = res(p, guess);
      yb = res(p, b);
      evals += 2;
      if (ya * yb > 0.0) {
        yb = ya;
        b = guess;
        ya = res(p, a);
        evals++;
      } else {
        a = guess;
      }
    } else {
      ya = res(p, a);
      yb = res(p, b);
      evals += 2;
    }
    bracketed = !(ya * yb > 0.0);
  }
  s.sign = (ya < 0 ? 1.0 : -1.0);
  s.a = a;
  s.b = b;
  s.ya = ya * s.sign;
  s.yb = yb * s.sign;
  s.it = 0;
  s.b1 = s.b2 = 0;
  s.evals = evals;
  s.bracketed = bracketed;
}

// True while the zone still iterates (root_find.hpp:120 loop condition).
__device__ __forceinline__ bool rf_running(const Par &p, const RFState &s) {
  return s.bracketed && (s.b - s.a > 2.0 * p.c2p_tol) && (s.it < p.c2p_max_iter);
}

// The Illinois iterations (root_find.hpp:120-166), warp-synchronous: every
// lane stays in the loop until the warp's vote says none is still
// iterating.  A lane stops after cap iterations in total even if it has not
// converged (rf_running stays true: the caller resumes it later).  WARP =
// false: the lane loops on its own (for callers whose lanes may have left;
// the arithmetic is the same).
template <bool WARP = true>
__device__ __forceinline__ void rf_iterate(const Par &p, Residual &res, bool valid, RFState &s, int cap) {
  const double tol = p.c2p_tol;
  const int max_iter = p.c2p_max_iter;
  double a = s.a, b = s.b, ya = s.ya, yb = s.yb;
  const double sign = s.sign;
  int it = s.it, b1 = s.b1, b2 = s.b2, evals = s.evals;
  bool active = valid && s.bracketed && (b - a > 2.0 * tol) && (it < max_iter) && (it < cap);
  while (WARP ? __any_sync(0xffffffffu, active) : active) {
    if (active) {
      const double c = div_p(a * yb - b * ya, yb - ya);
      if (c == a) {
        b = a;
      } else if (c == b) {
        a = b;
      } else {
        const double yc = sign * res(p, c);
        evals++;
        if (yc > 0.0) {
          b = c;
          yb = yc;
          b1++;
          ya *= (b1 > 1 ? 0.5 : 1.0);
          b2 = 0;
        } else if (yc < 0.0) {
          a = c;
          ya = yc;
          b2++;
          yb *= (b2 > 1 ? 0.5 : 1.0);
          b1 = 0;
        } else {
          a = c;
          b = c;
        }
      }
      it++;
      active = (b - a > 2.0 * tol) && (it < max_iter) && (it < cap);
    }
  }
  s.a = a;
  s.b = b;
  s.ya = ya;
  s.yb = yb;
  s.it = it;
  s.b1 = b1;
  s.b2 = b2;
  s.evals = evals;
}

__device__ __forceinline__ double rf_result(const RFState &s, double guess, C2POut &out) {
  out.iterations = s.it;
  out.evals = s.evals;
  out.bracketed = s.bracketed;
  out.learned = s.learned;
  if (!s.bracketed) return guess;
  return 0.5 * (s.a + s.b);
}

// refine_bracket + regula_falsi (root_find.hpp:42-58, 110-167) in one call.
// valid = this lane owns a zone.  Returns mu; iterations/evals/bracketed
// through out.  a/b: starting bracket ([0, 1] in the reference).
template <bool LEARNED = false>
__device__ __forceinline__ double regula_falsi_warp(const Par &p, Residual &res, bool valid, double a, double b,
                                                   double guess, C2POut &out, const double *lb = nullptr) {
  RFState s;
  rf_start<LEARNED>(p, res, valid, a, b, guess, lb, s);
  rf_iterate(p, res, valid, s, p.c2p_max_iter);
  return rf_result(s, guess, out);
}

// Largest number of FP64 evaluations of the production root before a zone takes
// the reference's iteration; iteration caps below it keep the reference's own
// counting.
constexpr int C2P_FAST_EVALS = 5;
__host__ __device__ __forceinline__ bool c2p_fast_allowed(const Par &p) {
  return p.c2p_max_iter >= C2P_FAST_EVALS && p.c2p_tol >= 1e-15 && p.c2p_tol <= 1e-3;
}

#ifndef PHX_EXACT
// ------------------------------------------------ production root find
// The residual is FP64-bound: an FP64 instruction holds a sub-partition's
// FP64 pipe for 64-76 cycles, an FP32 instruction takes one to two.  So the
// search for the root runs in FP32: a safeguarded Newton iteration with the
// analytic derivative, then two Newton steps on the residual in pairs of
// floats (48 bits), which bring mu to about 1e-13.  One FP64 residual
// evaluation corrects that value; the correction times the slope's own
// error is what is left, and the zone is accepted when it is below the
// caller's tolerance (otherwise secant steps with further FP64 evaluations
// follow).  A zone that does not pass these tests (values outside the FP32
// range, a density below 1e-14, NaN, no convergence) takes the reference's
// bracketed iteration instead.
// Measured against the bracketed iteration in FP64 (GB300, with the reciprocals
// on the integer pipe and c2p_finish's algebra): 1.2e7 cold Kerr-Schild zones
// at tolerance 1e-13 30.0 -> 5.5 ms (12.8 -> 1.01 FP64 residual evaluations per
// zone), a 136^3 Minkowski block from stale mu 3.90 -> 0.87 ms (7.0 -> 1.0
// evaluations; 147 FP64 instructions per zone, the FP64 pipe busy 94% of the
// time), 1000 cold zones 96 -> 40 us; the root's error against the sampled
// state 3e-14 -> 5e-15.

// float from a double by bit operations (a conversion instruction holds the
// FP64 pipe): truncated, 0 below and +-max above the FP32 normal range.
__device__ __forceinline__ float d2f_bits(double x) {
  const int hi = __double2hiint(x);
  const int mag = hi & 0x7fffffff;
  unsigned m = ((unsigned)(mag - 0x38000000) << 3) | ((unsigned)__double2loint(x) >> 29);
  if (mag < 0x38100000) m = 0u;
  if (mag >= 0x47e00000) m = 0x7f7fffffu;
  return __int_as_float((int)(m | (hi & 0x80000000)));
}
// double from a normal float (exact), by bit operations
__device__ __forceinline__ double f2d_bits(float f) {
  const int b = __float_as_int(f);
  const int mag = b & 0x7fffffff;
  const int hi = mag < 0x00800000 ? 0 : (mag >> 3) + 0x38000000;
  return __hiloint2double(hi | (b & 0x80000000), mag < 0x00800000 ? 0 : (b << 29));
}

__device__ __forceinline__ float rcp_f32(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float rsqrt_f32(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// Pairs of floats h + l (|l| <= ulp(h) / 2): the error-free sum of Knuth and
// Dekker's product with an FMA, the usual double-word algorithms on them.
struct FF {
  float h, l;
};
__device__ __forceinline__ FF ff_quick(float a, float b) {  // |a| >= |b|
  const float s = __fadd_rn(a, b);
  return {s, __fsub_rn(b, __fsub_rn(s, a))};
}
__device__ __forceinline__ FF ff_sum(float a, float b) {
  const float s = __fadd_rn(a, b), v = __fsub_rn(s, a);
  return {s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, v)), __fsub_rn(b, v))};
}
__device__ __forceinline__ FF ff_add(FF a, FF b) {
  FF s = ff_sum(a.h, b.h);
  return ff_quick(s.h, __fadd_rn(s.l, __fadd_rn(a.l, b.l)));
}
__device__ __forceinline__ FF ff_addf(FF a, float b) {
  FF s = ff_sum(b, a.h);
  return ff_quick(s.h, __fadd_rn(s.l, a.l));
}
__device__ __forceinline__ FF ff_neg(FF a) { return {-a.h, -a.l}; }
__device__ __forceinline__ FF ff_mul(FF a, FF b) {
  const float p = __fmul_rn(a.h, b.h);
  float e = __fmaf_rn(a.h, b.h, -p);
  e = __fmaf_rn(a.h, b.l, __fmaf_rn(a.l, b.h, e));
  return ff_quick(p, e);
}
__device__ __forceinline__ FF ff_rcp(FF a) {
  const float r = rcp_f32(a.h);
  float e = __fmaf_rn(-a.h, r, 1.0f);
  e = __fmaf_rn(-a.l, r, e);
  return ff_quick(r, __fmul_rn(r, __fmaf_rn(e, e, e)));
}
__device__ __forceinline__ FF ff_rsqrt(FF a) {
  const float y = rsqrt_f32(a.h);
  const float p = __fmul_rn(y, y), pe = __fmaf_rn(y, y, -p);
  float g = __fmaf_rn(-a.h, p, 1.0f);
  g = __fmaf_rn(-a.h, pe, __fmaf_rn(-a.l, p, g));
  return ff_quick(y, __fmul_rn(y, __fmul_rn(g, __fmaf_rn(0.375f, g, 0.5f))));
}
// the leading 47 bits of a double: h truncated, l the next 23 bits (0 where it
// would be subnormal)
__device__ __forceinline__ FF ff_bits(double x) {
  FF r;
  r.h = d2f_bits(x);
  const int b = __float_as_int(r.h), ex = b & 0x7f800000;
  const int sg = b & 0x80000000;
  const int el = ex - (23 << 23);
  const unsigned rem = ((unsigned)__double2loint(x) >> 6) & 0x7fffffu;
  const float unit = __int_as_float(el | sg);
  r.l = (el > 0 && (b & 0x7fffffff) != 0x7f7fffff) ? __fsub_rn(__int_as_float(el | sg | (int)rem), unit) : 0.0f;
  return r;
}

// The residual with Phat = gm1 rho e written out: the reference's ahat is
// gm1 e / (1 + e) and (1 + ahat)(1 + e) = 1 + Gamma e, so the density enters
// only through the floors; x rbarsq as x (mu rbsq + x (rsq + mu rbsq)).
//   eval:  FP32 and the derivative
//   evalp: pairs of floats
//   eval64: FP64; 38 arithmetic instructions and integer comparisons
// RHOU: the energy floor follows the density (ExpX1RhoU); code of its own, whose
// size costs the other floors' kernels 2 to 5%.
template <bool RHOU>
struct FastResidual {
  FF q, hb, rsq, rbsq, v0sq, gm1, bsq;  // q: q - bsq / 2, hb: -bsq_rpsq / 2
  float efl, emax;
  double qh, efl64;
  __device__ __forceinline__ FastResidual(const Par &p, const Residual &r) {
    qh = fma(-0.5, r.bsq, r.q);
    q = ff_bits(qh);
    bsq = ff_bits(r.bsq);
    hb = ff_bits(r.bsq_rpsq);
    hb.h *= -0.5f;
    hb.l *= -0.5f;
    rsq = ff_bits(r.rsq);
    rbsq = ff_bits(r.rbsq);
    v0sq = ff_bits(r.v0sq);
    gm1 = ff_bits(p.gm1);
    double rho = r.rho_floor;  // RHOU: the sie floor at the density floor, its largest value
    floors_from(p, r.fl, rho, efl64);
    efl64 *= p.fsf;
    efl = d2f_bits(efl64);
    emax = d2f_bits(r.e_max);
  }
  // RHOU: the specific energy floor s / max(rho, r), rho = max(D / W, its floor);
  // moving: it follows D / W here
  __device__ __forceinline__ float rhou_floor(const Par &p, const Residual &r, float iW, bool &moving) const {
    const float lo = d2f_bits(max_num(r.rho_floor, r.fl.r)), rho = d2f_bits(r.D) * iW, sc = d2f_bits(p.fsf);
    const float ef = sc * d2f_bits(r.fl.s) * rcp_f32(fmaxf(rho, lo)), em = sc * d2f_bits(p.sie_min_eos);
    moving = rho > lo && ef > em;
    return fmaxf(ef, em);
  }
  __device__ __forceinline__ FF rhou_floor(const Par &p, const Residual &r, FF iW) const {
    const FF lo = ff_bits(max_num(r.rho_floor, r.fl.r)), sc = ff_bits(p.fsf);
    FF rho = ff_mul(ff_bits(r.D), iW);
    if (lo.h > rho.h || (lo.h == rho.h && lo.l > rho.l)) rho = lo;
    const FF ef = ff_mul(ff_mul(sc, ff_bits(r.fl.s)), ff_rcp(rho)), em = ff_mul(sc, ff_bits(p.sie_min_eos));
    return em.h > ef.h ? em : ef;
  }
  __device__ __forceinline__ float eval(const Par &p, const Residual &r, float mu, float &df) const {
    const float x = rcp_f32(fmaf(mu, bsq.h, 1.0f));
    const float dx = -bsq.h * x * x;
    const float mr = mu * rbsq.h, u = rsq.h + mr;
    const float w = fmaf(x, u, mr);
    const float rb = x * w;
    const float drb = fmaf(dx, fmaf(x, u, w), x * fmaf(x, rbsq.h, rbsq.h));
    const float mux = mu * x;
    const float qb = fmaf(mux * mux, hb.h, q.h);
    const float dqb = 2.0f * mux * fmaf(mu, dx, x) * hb.h;
    const float mrb = mu * rb, dmrb = fmaf(mu, drb, rb);
    float v2 = mu * mrb, dv2 = fmaf(mu, dmrb, mrb);
    if (v2 > v0sq.h) {
      v2 = v0sq.h;
      dv2 = 0.0f;
    }
    const float om = 1.0f - v2;
    const float W = rsqrt_f32(om), iW = om * W;
    const float A = qb - mrb, dA = dqb - dmrb;
    const float dW = 0.5f * W * W * W * dv2, diW = -0.5f * W * dv2;
    float e = fmaf(W, A, W - 1.0f), de = fmaf(dW, A + 1.0f, W * dA);
    if (e <= efl) {
      bool moving = false;
      const float ef = RHOU ? rhou_floor(p, r, iW, moving) : efl;
      if (!RHOU || e <= ef) {
        e = ef;
        de = moving ? 0.5f * ef * W * W * dv2 : 0.0f;
      }
    } else if (e > emax) {
      e = emax;
      de = 0.0f;
    }
    const float P = fmaxf(gm1.h * e, 0.0f);
    const float dP = gm1.h * e > 0.0f ? gm1.h * de : 0.0f;
    const float ie = rcp_f32(1.0f + e);
    const float a = P * ie, da = (dP - a * de) * ie;
    const float h = 1.0f + e + P, dh = de + dP;
    const float nua = h * iW, nub = (1.0f + a) * (1.0f + A);
    const float dnu = nua > nub ? fmaf(dh, iW, h * diW) : fmaf(da, 1.0f + A, (1.0f + a) * dA);
    const float g = rcp_f32(fmaxf(nua, nub) + mrb);
    df = fmaf(g * g, dnu + dmrb, 1.0f);
    return mu - g;
  }
  __device__ __forceinline__ float evalp(const Par &p, const Residual &r, FF mu) const {
    const FF x = ff_rcp(ff_addf(ff_mul(mu, bsq), 1.0f));
    const FF mr = ff_mul(mu, rbsq);
    const FF rb = ff_mul(x, ff_add(mr, ff_mul(x, ff_add(rsq, mr))));
    const FF mux = ff_mul(mu, x);
    const FF mrb = ff_mul(mu, rb);
    const FF A = ff_add(ff_add(q, ff_mul(ff_mul(mux, mux), hb)), ff_neg(mrb));
    FF v2 = ff_mul(mu, mrb);
    if (v2.h > v0sq.h || (v2.h == v0sq.h && v2.l > v0sq.l)) v2 = v0sq;
    const FF om = ff_addf(ff_neg(v2), 1.0f);
    const FF W = ff_rsqrt(om), iW = ff_mul(om, W);
    FF e = ff_add(ff_mul(W, A), ff_addf(W, -1.0f));
    if (e.h <= efl) {
      const FF ef = RHOU ? rhou_floor(p, r, iW) : FF{efl, 0.0f};
      if (!RHOU || e.h < ef.h || (e.h == ef.h && e.l <= ef.l)) e = ef;
    } else if (e.h > emax) {
      e = {emax, 0.0f};
    }
    const FF e1 = ff_addf(e, 1.0f);
    const FF h = e.h > 0.0f ? ff_add(e1, ff_mul(gm1, e)) : e1;
    const FF nua = ff_mul(h, iW), nub = ff_mul(ff_mul(h, ff_rcp(e1)), ff_addf(A, 1.0f));
    const FF g = ff_rcp(ff_add(nua.h > nub.h ? nua : nub, mrb));
    return __fadd_rn(__fsub_rn(mu.h, g.h), __fsub_rn(mu.l, g.l));
  }
  // false (the reference's expressions apply): a density, D / W or its floor, small
  // enough for the reference's bound on h rho, an energy below 0.  Zones with
  // D < 0 sit on the floor: 0.4% of the zones of a floored random state, which
  // held their warps (MP5 stage of 1024 blocks 0.80 -> 0.93 s) while all of them
  // took the reference's iteration.
  // room: about the relative change of mu that switches the velocity bound or
  // one of the energy bounds
  __device__ __forceinline__ bool eval64(const Par &p, const Residual &r, double mu, double &f, float &room) const {
    const double x = rcp_p(fma(mu, r.bsq, 1.0));
    const double mr = mu * r.rbsq;
    const double rb = x * fma(x, r.rsq + mr, mr);
    const double mux = mu * x;
    const double mrb = mu * rb;
    const double A = fma(-0.5 * r.bsq_rpsq, mux * mux, qh) - mrb;
    double v2 = mu * mrb;
    const float dv = fabsf(d2f_bits(v2) - v0sq.h);
    if (gt_bits(v2, r.v0sq)) v2 = r.v0sq;
    const double om = 1.0 - v2;
    const double W = rsqrt_p(om), iW = om * W;
    double e = fma(W, A, W - 1.0);
    if (dexp(e) == 0x7ff) return false;  // NaN or infinity
    const float ef = d2f_bits(e), Wf = d2f_bits(W);  // mu de/dmu is of size W (W (1 + e) + mrb + |A|)
    const float de = Wf * fmaf(Wf, 1.0f + fabsf(ef), d2f_bits(mrb) + fabsf(d2f_bits(A)));
    double bound = efl64;
    if constexpr (RHOU)
      bound = p.fsf * max_num(r.fl.s * rcp_p(max_num(max_num(r.D * iW, r.rho_floor), r.fl.r)), p.sie_min_eos);
    room = fminf(0.5f * dv, fminf(fabsf(ef - d2f_bits(bound)), fabsf(ef - emax)) * rcp_f32(de));
    if (!gt_bits(e, bound)) {
      e = bound;
    } else if (gt_bits(e, r.e_max)) {
      e = r.e_max;
    }
    const bool dense = __double2hiint(r.D) >= 0 && dexp(r.D) + (dexp(iW) - 1023) >= 1023 - 46;
    if (__double2hiint(e) < 0 || !(dense || __double2hiint(r.rho_floor) >> 20 >= 1023 - 46)) return false;
    const double e1 = 1.0 + e;
    const double h = fma(p.gm1, e, e1);
    const double nua = h * iW, nub = (h * rcp_p(e1)) * (1.0 + A);
    f = mu - rcp_p((gt_bits(nua, nub) ? nua : nub) + mrb);
    return true;
  }
};

// mu of one zone from its guess (> 0: a previous solution) or, LEARNED, the
// predicted root lb[0] of a cold zone.  False: not accepted.  mu lies within
// c2p_tol of the root where true, as the reference's final bracket has it.
template <bool LEARNED, bool RHOU>
__device__ __forceinline__ bool c2p_fast_root(const Par &p, const Residual &res, double guess, const double *lb,
                                              double &mu, C2POut &out) {
  const FastResidual<RHOU> rf(p, res);
  float lo = 0.0f, hi = 1.0f, s = 1.0f;
  float m = guess > 0.0 && guess < 1.0 ? d2f_bits(guess) : rsqrt_f32(1.0f + rf.rsq.h);
  out.learned = false;
  if constexpr (LEARNED) {
    if (!(guess > 0.0) && lb[1] >= 0.0 && lb[1] <= lb[0] && lb[0] <= lb[2] && lb[2] <= 1.0) {
      float d;
      const float l = d2f_bits(lb[1]), h = d2f_bits(lb[2]);
      if (rf.eval(p, res, l, d) <= 0.0f && rf.eval(p, res, h, d) >= 0.0f) {
        m = d2f_bits(lb[0]);
        lo = l;
        hi = h;
        out.learned = true;
      }
    }
  }
  float last = 1.0f, span = 1.0f;  // span: how far from the root the slope's points may lie
  for (int it = 0; it < 24; it++) {
    const float f = rf.eval(p, res, m, s);
    if (f > 0.0f)
      hi = m;
    else
      lo = m;
    float n = m - f * rcp_f32(s);
    if (!(n > lo && n < hi)) n = 0.5f * (lo + hi);
    const float d = fabsf(n - m);
    m = n;
    span = d;
    // FP32 rounding reached: the step is at rounding level, or small and no longer shrinking
    if (d <= 1e-6f * m || (d <= 1e-3f * m && d > 0.5f * last)) break;
    last = d;
  }
  if (!(s > 1e-3f && m > 1e-12f && m <= 1.0f)) return false;
  // float-pair Newton steps until the step is at the pairs' rounding; the slope
  // follows the secant (the residual's branches differ in slope at the root)
  FF mp = {m, 0.0f};
  float is = rcp_f32(s), step = 0.0f, fp = 0.0f;
#pragma unroll 1
  for (int it = 0; it < 5; it++) {
    const float f = rf.evalp(p, res, mp);
    if (it > 0 && fabsf(step) > 1e-7f * m) {
      is = step * rcp_f32(fp - f);
      span = fabsf(step);
    }
    step = f * is;
    fp = f;
    if (!(fabsf(step) <= 0.5f * m)) return false;
    if (it == 0) span += fabsf(step) + 2e-7f * m;
    mp = ff_addf(mp, -step);
    if (fabsf(step) <= 4e-12f * m) break;
  }
  if (!(is > 0.0f && is < 1e3f)) return false;
  double x = f2d_bits(mp.h) + f2d_bits(mp.l);
  const float tol = d2f_bits(p.c2p_tol);
  const float tight = fmaxf(0.0625f * tol, fminf(tol, 1e-12f * m));  // the residual's rounding is of that size
  float f = 0.0f;
  out.iterations = out.evals = 0;
#pragma unroll 1
  for (;;) {
    double f64;
    float room;
    if (out.evals >= C2P_FAST_EVALS || !(x > 0.0 && x <= 1.0) || !rf.eval64(p, res, x, f64, room)) return false;
    const float fn = d2f_bits(f64);
    if (out.evals > 0 && fabsf(step) > 1e-11f * m) {  // secant through the last two evaluations
      const float isec = step * rcp_f32(f - fn);
      if (isec > 0.0f && isec < 1e3f) {
        is = isec;
        span = fabsf(step);
      } else if (fabsf(step) > 1e-9f * m) {
        return false;
      }
    }
    out.evals++;
    out.iterations++;
    f = fn;
    step = f * is;
    if (!(fabsf(step) <= 0.5f * m)) return false;
    x -= f2d_bits(step);
    // The error after this step is the step times the slope's relative error.
    // Two secants that agree say nothing about the slope beyond the root, where
    // the residual has its kink (nua = nub, slopes up to 1.9 apart: an error
    // below the step).  Where a bound switches within reach of the points the
    // slope comes from, slopes up to 12 apart were seen: the step has to be a
    // sixteenth of the tolerance.
    if (fabsf(step) <= (room * m > 2.0f * span ? tol : tight)) {
      mu = x < 1.0 ? x : 1.0;
      return x > 0.0;
    }
  }
}

// The reference's iteration for the zones the fast root leaves, kept out of
// the callers' instruction stream.
template <bool LEARNED>
static __device__ __noinline__ double c2p_slow_root(const Par &p, Residual res, bool need, double guess, double lb0,
                                                    double lb1, double lb2, C2POut *out) {
  const double lb[3] = {lb0, lb1, lb2};
  return regula_falsi_warp<LEARNED>(p, res, need, 0.0, 1.0, guess, *out, lb);
}
#endif

// The root of one zone per lane, warp-synchronous: the production build's
// fast root where it is accepted, the reference's iteration elsewhere.
template <bool LEARNED, bool RHOU>
__device__ __forceinline__ double c2p_root_warp(const Par &p, Residual &res, bool valid, double guess, C2POut &out,
                                                const double *lb = nullptr) {
#ifndef PHX_EXACT
  bool need = valid;
  double mu = guess;
  if (valid && c2p_fast_allowed(p)) need = !c2p_fast_root<LEARNED, RHOU>(p, res, guess, lb, mu, out);
  if (!__any_sync(0xffffffffu, need)) return mu;
  C2POut slow{0, 0, false, true, false, false};
  double ms;
  if constexpr (LEARNED)
    ms = c2p_slow_root<true>(p, res, need, guess, lb[0], lb[1], lb[2], &slow);
  else
    ms = c2p_slow_root<false>(p, res, need, guess, 0.0, 0.0, 0.0, &slow);
  if (need) {
    out.iterations = slow.iterations;
    out.evals = slow.evals;
    out.bracketed = slow.bracketed;
    out.learned = slow.learned;
    mu = ms;
  }
  return mu;
#else
  return regula_falsi_warp<LEARNED>(p, res, valid, 0.0, 1.0, guess, out, lb);
#endif
}

// Unwrap mu into primitives (con2prim_robust.hpp:381-452).
// prim[] receives PHX_NPRIM values (B slots only when mhd), U[] may be
// rewritten by p2c when bounds were used; sig[3] receives signal speeds.
template <bool MINK>
__device__ __forceinline__ void c2p_finish(const Par &p, const Pt &g, Residual &res, double mu,
                                           const double rcon[3], const double bu_in[3],
                                           const double Bprim[3], double bdotr,
                                           double prim[PHX_NPRIM], double U[PHX_NCONS],
                                           double sig[3], bool &used_bounds_out) {
  prim[PHX_PMU] = mu;
#ifndef PHX_EXACT
  // production build: the residual's algebra (FastResidual), W and 1/W from
  // one reciprocal square root, P = gm1 rho e, the three-velocity before W v
  const double x = rcp_p(fma(mu, res.bsq, 1.0));
  const double mr = mu * res.rbsq, mux = mu * x;
  const double mrb = mu * (x * fma(x, res.rsq + mr, mr));
  double vsq = mu * mrb;
  res.used_gamma_max = gt(vsq, res.v0sq);
  if (res.used_gamma_max) vsq = res.v0sq;
  const double om = 1.0 - vsq;
  const double W = rsqrt_p(om), iW = om * W;
  prim[PHX_PRHO] = res.rhohat_mu(iW);
  const double A = fma(-0.5 * res.bsq_rpsq, mux * mux, fma(-0.5, res.bsq, res.q)) - mrb;
  double eng = res.bound_ehat(p, prim[PHX_PRHO], fma(W, A, W - 1.0));
  prim[PHX_PTMP] = eos_T_rho_sie(p, prim[PHX_PRHO], eng);
  eng *= prim[PHX_PRHO];
  prim[PHX_PENG] = eng;
  prim[PHX_PPRS] = clamp0(p.gm1 * eng);
  // bmod / P of the ideal gas is Gamma wherever P > 0 (the quotient, NaN for
  // P = 0, elsewhere)
  prim[PHX_PGM1] = __double_as_longlong(prim[PHX_PPRS]) > 0
                       ? p.gm1 + 1.0
                       : div_p(eos_bmod_rho_T(p, prim[PHX_PRHO], prim[PHX_PTMP]), prim[PHX_PPRS]);
  double v3[3], vel[3];
  const double mbr = mu * bdotr;
#pragma unroll
  for (int ii = 0; ii < 3; ii++) {
    v3[ii] = mux * fma(mbr, bu_in[ii], rcon[ii]);
    vel[ii] = W * v3[ii];
    prim[PHX_PVEL + ii] = vel[ii];
  }
#else
  const double x = res.x_mu(mu);
  const double rbarsq = res.rbarsq_mu(mu, x);
  const double vsq = res.vhatsq_mu(mu, rbarsq);
  const double iW = res.iWhat_mu(vsq);
  const double W = rcp_p(iW);
  prim[PHX_PRHO] = res.rhohat_mu(iW);
  const double qbar = res.qbar_mu(mu, x);
  double eng = res.ehat_mu(p, mu, qbar, rbarsq, vsq, W);
  prim[PHX_PTMP] = eos_T_rho_sie(p, prim[PHX_PRHO], eng);
  eng *= prim[PHX_PRHO];
  prim[PHX_PENG] = eng;
  prim[PHX_PPRS] = eos_P_rho_T(p, prim[PHX_PRHO], prim[PHX_PTMP]);
  prim[PHX_PGM1] = div_p(eos_bmod_rho_T(p, prim[PHX_PRHO], prim[PHX_PTMP]), prim[PHX_PPRS]);
  double vel[3];
#pragma unroll
  for (int ii = 0; ii < 3; ii++) {
    vel[ii] = W * mu * x * (rcon[ii] + mu * bdotr * bu_in[ii]);
    prim[PHX_PVEL + ii] = vel[ii];
  }
#endif
  double bu[3] = {0.0, 0.0, 0.0};
  if (p.mhd) {
#pragma unroll
    for (int ii = 0; ii < 3; ii++) {
      prim[PHX_PB + ii] = Bprim[ii];
      bu[ii] = Bprim[ii];
    }
  }
  used_bounds_out = res.used_bounds();
  if (used_bounds_out) {
    double S[3], bcons[3], Dn, taun;
    const double gdet = MINK ? 1.0 : g.detgam;
    p2c<MINK>(prim[PHX_PRHO], vel, bu, prim[PHX_PENG], prim[PHX_PPRS], prim[PHX_PGM1], g, gdet,
              Dn, S, bcons, taun, sig);
    U[PHX_CRHO] = Dn;
    U[PHX_CENG] = taun;
#pragma unroll
    for (int ii = 0; ii < 3; ii++) U[PHX_CMOM + ii] = S[ii];
  } else {
#ifdef PHX_EXACT
#pragma unroll
    for (int m = 0; m < 3; m++) vel[m] *= iW;
#else
#pragma unroll
    for (int m = 0; m < 3; m++) vel[m] = v3[m];
#endif
    double bsq = 0.0;
    if (p.mhd) {
      double bdotv;
      if constexpr (MINK) {
        bsq = bu[0] * bu[0] + bu[1] * bu[1] + bu[2] * bu[2];
        bdotv = bu[0] * vel[0] + bu[1] * vel[1] + bu[2] * vel[2];
      } else {
#ifdef PHX_EXACT
        bdotv = 0.0;
#pragma unroll
        for (int m = 0; m < 3; m++)
#pragma unroll
          for (int n = 0; n < 3; n++) {
            bsq += bu[m] * bu[n] * g.gcov[m + 1][n + 1];
            bdotv += bu[m] * vel[n] * g.gcov[m + 1][n + 1];
          }
#else
        double blo[3];  // lowered B serves both contractions
        lower_sp(g, bu, blo);
        bsq = dot3(bu, blo);
        bdotv = dot3(vel, blo);
#endif
      }
      bsq = iW * iW * bsq + bdotv * bdotv;
    }
    signal_speeds<MINK>(prim[PHX_PRHO], prim[PHX_PENG], prim[PHX_PPRS], bsq, vel, vsq,
                        prim[PHX_PGM1], g, sig);
  }
}

}  // namespace phx
