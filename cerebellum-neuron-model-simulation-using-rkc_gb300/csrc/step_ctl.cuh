// The scalar half of a step attempt: RKC's controller (rkclow, solve_rkc.cu:
// 909-1096) over a system's Ctl record, in registers, for the integrators that
// keep their vectors in registers (quad_sys.cuh, group_sys.cuh).  The vector
// half asks for the step (plan), runs the stages and the error norm, and hands
// the norm back (judge).  The arithmetic is Sys::attempt's (integrator.cuh)
// operation for operation; every thread of a team computes it alike.
//
// E is the type of the error norm and its cube root: double, or float for the
// granule cells of mixed precision, whose scalar chain -- the norm, its cube
// root, the stage count's square root and the step-size ratios -- is FP32
// while the step size, the time and the accept/reject comparison stay FP64.
#pragma once
#include <type_traits>
#include "integrator.cuh"

namespace gbrkc {

template <typename E>
struct StepCtl {
  static constexpr bool FAST = std::is_same<E, float>::value;
  enum { ATT_FAIL = -1, ATT_REJECT = 0, ATT_ACCEPT = 1 };

  double absh, sprad, hold, lt, tend, gt_old, hw0, hw1, sum_dt, integ, hmin, tol;
  E errold, cbrt_errold;
  int newspc, jacatt, last, status, iv_left, idid, mmax, rej_run;
  long long naccpt, n_steps, n_rej, n_stage, n_rho, n_rho_iter, n_ion;

  static __device__ __forceinline__ E to_e(double x) {
    if constexpr (FAST) return d2f(x);
    else return x;
  }
  static __device__ __forceinline__ double from_e(E x) {
    if constexpr (FAST) return f2d(x);
    else return x;
  }

  __device__ __forceinline__ void load(const Ctl &c) {
    absh = c.absh; sprad = c.sprad; hold = c.hold; lt = c.lt; tend = c.tend; gt_old = c.gt_old;
    hw0 = c.hw0; hw1 = c.hw1; sum_dt = c.sum_dt; integ = c.integ; hmin = c.hmin; tol = c.tol;
    errold = to_e(c.errold);
    cbrt_errold = to_e(c.cbrt_errold);
    newspc = c.newspc; jacatt = c.jacatt; last = c.last; status = c.status; iv_left = c.iv_left;
    idid = (int)c.idid;
    mmax = (int)c.mmax;
    rej_run = 0;
    naccpt = (long long)c.naccpt;
    n_steps = c.n_steps; n_rej = c.n_rej; n_stage = c.n_stage; n_rho = c.n_rho; n_rho_iter = c.n_rho_iter;
    n_ion = c.n_ion;
  }

  // (one thread of the team; mmax changes at initialisation only)
  __device__ __forceinline__ void store(Ctl &c, bool with_mmax = false) const {
    c.absh = absh; c.sprad = sprad; c.hold = hold; c.lt = lt; c.tend = tend; c.gt = lt; c.gt_old = gt_old;
    c.hw0 = hw0; c.hw1 = hw1; c.sum_dt = sum_dt;
    c.errold = from_e(errold);
    c.cbrt_errold = from_e(cbrt_errold);
    c.newspc = newspc; c.jacatt = jacatt; c.last = last; c.status = status; c.iv_left = iv_left;
    c.idid = (double)idid;
    if (with_mmax) c.mmax = (double)mmax;
    c.naccpt = (double)naccpt;
    c.n_steps = n_steps; c.n_rej = n_rej; c.n_stage = n_stage; c.n_rho = n_rho; c.n_rho_iter = n_rho_iter;
    c.n_ion = n_ion;
  }

  // The attempt's step size and stage count; false (status set) where the
  // stage count is not a number.
  __device__ __forceinline__ bool plan(double &h, int &m) {
    last = 0;
    const double left = fpi_abs(tend - lt);
    if (nn_le(left, 1.1 * absh)) {
      absh = left;
      last = 1;
    }
    const double x = 1.54 * absh * sprad + 1.0;
    if constexpr (FAST) {
      const float marg = sqrtf(d2f(x));
      if (!(marg < 1.0e9f)) {
        status |= ST_NAN;
        return false;
      }
      m = 1 + (int)marg;
    } else if (!stage_count(x, m)) {
      status |= ST_NAN;
      return false;
    }
    if (m > mmax) {
      m = mmax;
      absh = (m * m - 1) / (1.54 * sprad);
      last = 0;
    }
    h = absh;
    if (nn_le(h, hmin)) h = hmin;
    return true;
  }

  // After a step of size h with m stages: the error norm decides, and sets the
  // next step size.
  __device__ __forceinline__ int judge(E err, double h) {
    bool over;
    E cr;
    if constexpr (FAST) {
      if (err != err) {
        status |= ST_NAN;
        return ATT_FAIL;
      }
      cr = cbrtf(err);
      over = err > 1.0f;
      if (over) absh = absh * f2d(0.8f / cr);
    } else {
      if (fpi_isnan(err)) {
        status |= ST_NAN;
        return ATT_FAIL;
      }
      cr = cm_cbrt(err);
      over = nn_lt(1.0, err);
      if (over) absh = mdiv(0.8 * absh, cr);
    }
    if (over) {
      n_rej++;
      if (nn_lt(absh, hmin)) {
        idid = 4;                // falls through to acceptance
      } else {
        newspc = !jacatt;
        if (++rej_run >= RKCLOW_LOOP_CAP) {
          status |= ST_LOOP_CAP;
          return ATT_FAIL;
        }
        return ATT_REJECT;
      }
    }
    rej_run = 0;
    naccpt++;
    lt += h;
    jacatt = 0;
    newspc = 0;                  // nstsig never advances (solve_rkc.cu:1024-1026)
    hw0 = h;
    hw1 = lt;
    if constexpr (FAST) {
      float fac = 10.0f;
      if (naccpt == 1) {
        if (0.8f < fac * cr) fac = 0.8f / cr;
      } else {
        const float temp1 = 0.8f * d2f(absh) * cbrt_errold;
        const float temp2 = fabsf(d2f(hold)) * (cr * cr);
        if (temp1 < fac * temp2) fac = temp1 / temp2;
      }
      absh = f2d((0.1f > fac) ? 0.1f : fac) * absh;
    } else {
      double fac = 10.0;
      if (naccpt == 1) {
        if (nn_lt(0.8, fac * cr)) fac = mdiv(0.8, cr);
      } else {
        const double temp1 = 0.8 * absh * cbrt_errold;
        const double temp2 = fpi_abs(hold) * (cr * cr);
        if (nn_lt(temp1, fac * temp2)) fac = mdiv(temp1, temp2);
      }
      absh = (nn_lt(fac, 0.1) ? 0.1 : fac) * absh;
    }
    cbrt_errold = cr;
    const double mn = nn_lt(absh, H_MAX) ? absh : H_MAX;
    absh = nn_lt(mn, hmin) ? hmin : mn;
    errold = err;
    hold = h;
    idid = last ? 1 : 2;
    return ATT_ACCEPT;
  }

  // After an accepted step: the ion clock; whether an update is due.
  __device__ __forceinline__ bool clock(bool at_equal) {
    sum_dt += lt - gt_old;
    gt_old = lt;
    return at_equal ? nn_le(integ, sum_dt) : nn_lt(integ, sum_dt);
  }

  // The dense output's weights at the interval's end (rkcint, solve_rkc.cu:
  // 795-813): v_new = a1 v1 + a2 yn + b1 v2 + b2 fn.
  __device__ __forceinline__ void dense(double &a1, double &a2, double &b1, double &b2) const {
    const double hlast = hw0, tlast = hw1 - hlast;
    const double sv = mdiv(gt_old - tlast, hlast);
    a1 = (1.0 + 2.0 * sv) * (sv - 1.0) * (sv - 1.0);
    a2 = (3.0 - 2.0 * sv) * sv * sv;
    b1 = hlast * sv * (sv - 1.0) * (sv - 1.0);
    b2 = hlast * (sv - 1.0) * sv * sv;
  }
};

// The nonlinear power method's scalars (rkcrho, solve_rkc.cu:563-754), for a
// team whose vectors the caller holds: next() takes the norm of F(v1) - fn and
// says how to go on.
struct RhoCtl {
  enum { MORE = 0, DONE = 1 };
  double dynrm, sigma, so0, so1, so2;
  Recip rdyn;
  __device__ __forceinline__ void begin(double dynrm_) {
    dynrm = dynrm_;
    rdyn = recip(dynrm);
    sigma = so0 = so1 = so2 = 0.0;
  }
  __device__ __forceinline__ int next(int iter, double dfnrm, double &sprad) {
    const double small = 1.0 / 0.125;
    const double sigmal = sigma;
    sigma = div_by(dfnrm, rdyn);
    so0 = so1;
    so1 = so2;
    so2 = sprad;
    sprad = 1.2 * sigma;
    if (iter >= 1 && nn_le(fpi_abs(sigma - sigmal), (nn_lt(small, sigma) ? sigma : small) * 0.001)) return DONE;
    if (iter > RHO_ITMAX / 2)
      if ((fabs(so2 - so0) < 0.00001) && (fabs(so1 - sprad) < 0.00001)) {
        sprad = (sprad + so2) / 2.0;
        return DONE;
      }
    return MORE;
  }
};

}  // namespace gbrkc
