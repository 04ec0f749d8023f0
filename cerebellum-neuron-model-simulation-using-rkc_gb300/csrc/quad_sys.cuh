// RKC integrator for single-cell systems of exactly four compartments (the
// granule cell of the mixed workload): one system per four lanes of a warp,
// one compartment a lane, its five RKC values and its current b in registers.
//
// What bounds it: a granule system is one serial chain of FP64 instructions
// (its controller's tolerance of 1e-9 keeps it at about 4000 step attempts
// per ms), and a warp issues one in 64 cycles whether one lane or
// all 32 are active and whatever its independence.  So the count of FP64 warp
// instructions per attempt sets the pace, and a compartment a lane quarters
// the vector part of it: about 40 instructions an attempt here (mixed
// precision), where one lane per system took 250.  The controller's scalars
// are computed alike by the four lanes; its comparisons and conversions, 100
// cycles each as FP64 instructions, run on the integer pipe (fp_int.cuh).
// The ion update shortens alike (one pass where a lane did four).  A
// neighbour's value comes by a shuffle within the four lanes.  Measured
// against one system a lane, both with their lanes-per-warp rule: 512 cells,
// mixed, 1 ms 40.3 -> 19.0 ms; 999 cells, FP64, 0.5 ms 73.6 -> 29.8 ms.
//
// The arithmetic is Sys's (integrator.cuh) operation for operation, so the
// results are bit-identical to it and to the oracle.  The reference rotates
// its five buffers by index (solve_rkc.cu:862-904, 1028-1034); here every
// logical vector is a register and a rotation moves values between them.  The
// system's buffer map (Ctl::map) stays as it was loaded and is used only to
// place the vectors back into the workspace at write-back, so readers of the
// workspace see the same logical contents.
//
// Used for advancing only; initialisation goes through Sys.
#pragma once
#include "step_ctl.cuh"

namespace gbrkc {

template <int CT, typename R>
struct QuadSys {
  static constexpr int NC = 4;
  // FP32 error norm and controller chain in mixed precision (step_ctl.cuh)
  static constexpr bool FAST = !std::is_same<R, double>::value;
  typedef typename std::conditional<FAST, float, double>::type E;

  const PoolView<R> &P;
  const unsigned mask;         // the system's four lanes
  const int r;                 // this lane's compartment
  int s, gi, off, cell0;
  // this compartment's row of the template's operator: up to three
  // neighbours, ascending, and the longest row of the cell
  int deg, maxdeg, nb[3];
  double g[3], invcm;
  double y, yn, fn, v1, v2, b;
  StepCtl<E> c;                // identical in the four lanes
  double t0;
  int k_iv, n_iv, iv0;
  long long attempts0;

  __device__ QuadSys(const PoolView<R> &P_)
      : P(P_), mask(0xfu << (threadIdx.x & 28)), r((int)(threadIdx.x & 3)) {}

  // Take system s_ (single cell, template operator, four compartments).
  __device__ __forceinline__ void load(int s_) {
    s = s_;
    off = P.sys_off[s];
    gi = off + r;
    cell0 = P.sys_cell0[s];
    const int t = P.sys_tmpl[s];
    const int *row = P.t_row + P.t_row0[t], *col = P.t_col + P.t_nz0[t];
    const double *gg = P.t_g + P.t_nz0[t];
    invcm = __ldg(P.t_invcm + P.t_cm0[t] + r);
    const int r0 = __ldg(row + r);
    deg = __ldg(row + r + 1) - r0;
#pragma unroll
    for (int q = 0; q < 3; q++) {
      nb[q] = q < deg ? __ldg(col + r0 + q) : r;
      g[q] = q < deg ? __ldg(gg + r0 + q) : 0.0;
    }
    maxdeg = deg;
    maxdeg = max(maxdeg, __shfl_xor_sync(mask, maxdeg, 1, 4));
    maxdeg = max(maxdeg, __shfl_xor_sync(mask, maxdeg, 2, 4));
    c.load(P.ctl[s]);
    const int *map = P.ctl[s].map;
    const double *ws = P.ws + P.sys_ws[s] + r;
    y = ws[map[LY] * NC];
    yn = ws[map[LYN] * NC];
    fn = ws[map[LFN] * NC];
    v1 = ws[map[LV1] * NC];
    v2 = ws[map[LV2] * NC];
    b = ws[WS_B * NC];
  }

  __device__ __forceinline__ void store() const {
    const int *map = P.ctl[s].map;
    double *ws = P.ws + P.sys_ws[s] + r;
    ws[map[LY] * NC] = y;
    ws[map[LYN] * NC] = yn;
    ws[map[LFN] * NC] = fn;
    ws[map[LV1] * NC] = v1;
    ws[map[LV2] * NC] = v2;
    ws[WS_B * NC] = b;
    if (r == 0) c.store(P.ctl[s]);
  }

  // dydt at this lane's compartment (Sys::rhs), u the lanes' stage values
  __device__ __forceinline__ double rhs(double u) const {
    double d = -b;
#pragma unroll
    for (int q = 0; q < 3; q++)
      if (q < maxdeg) {
        const double uj = __shfl_sync(mask, u, nb[q], 4);
        if (q < deg) d = fma(g[q], uj - u, d);
      }
    return d * invcm;
  }

  // the pairwise tree (q0 + q1) + (q2 + q3), the same bits in every lane
  __device__ __forceinline__ double sum4(double q) const {
    q = q + __shfl_xor_sync(mask, q, 1, 4);
    return q + __shfl_xor_sync(mask, q, 2, 4);
  }

  // Sys::rkcrho
  __device__ __forceinline__ void rkcrho() {
    const double uround = UROUND, sqrtu = sqrt(UROUND);
    const double e = P.ede[gi];
    c.n_rho++;
    const double ynrm = sqrt(sum4(yn * yn));
    const double vnrm = sqrt(sum4(e * e));
    double dynrm;
    if (!fpi_is_zero(ynrm) && !fpi_is_zero(vnrm)) {
      dynrm = ynrm * sqrtu;
      v1 = fma(mdiv(dynrm, vnrm), e, yn);
    } else if (!fpi_is_zero(ynrm)) {
      dynrm = ynrm * sqrtu;
      v1 = fma(sqrtu, yn, yn);
    } else if (!fpi_is_zero(vnrm)) {
      dynrm = uround;
      v1 = mdiv(dynrm, vnrm) * e;
    } else {
      dynrm = uround;
      v1 = dynrm;
    }
    RhoCtl rc;
    rc.begin(dynrm);
    for (int iter = 0; iter < RHO_ITMAX; iter++) {
      c.n_rho_iter++;
      v2 = rhs(v1);
      const double dm = -1.0 * fn + v2;
      const double dfnrm = sqrt(sum4(dm * dm));
      if (rc.next(iter, dfnrm, c.sprad) == RhoCtl::DONE) {
        P.ede[gi] = -1.0 * yn + v1;
        return;
      }
      if (!fpi_is_zero(dfnrm))
        v1 = fma(mdiv(dynrm, dfnrm), fn - v2, yn);
      else if (r == iter % NC)
        v1 = 2.0 * yn - v1;
    }
    c.idid = 6;
  }

  // Sys::step, the buffer rotations as moves
  __device__ __forceinline__ bool step(double h, int m) {
    if (m > P.coef_mmax) {
      c.status |= ST_COEF_TABLE;
      return false;
    }
    const double *T = P.coef + P.coef_off[m];
    v2 = yn;
    v1 = fma(h * __ldg(T), fn, yn);
    for (int j = 1; j < m; j++) {
      const double *q = T + 1 + 5 * (j - 1);
      const double mu = __ldg(q), nu = __ldg(q + 1), omn = __ldg(q + 2), mus = __ldg(q + 3), ajm1 = __ldg(q + 4);
      const double hm = h * mus;
      const double f = rhs(v1);
      double t = mu * v1;
      t = fma(nu, v2, t);
      t = fma(omn, yn, t);
      const double u = fma(-ajm1, fn, f);
      // written to y, then (v2, v1, y) <- (v1, y, v2)
      y = v2;
      v2 = v1;
      v1 = fma(hm, u, t);
    }
    // (y, v1, v2) <- (v1, v2, y)
    const double t = y;
    y = v1;
    v1 = v2;
    v2 = t;
    c.n_stage += m;
    return true;
  }

  // Sys::attempt
  __device__ __forceinline__ int attempt() {
    if (c.newspc) {
      rkcrho();
      c.jacatt = 1;
    }
    double h;
    int m;
    if (!c.plan(h, m) || !step(h, m)) return StepCtl<E>::ATT_FAIL;
    c.n_steps++;
    const double f = rhs(y);
    v1 = f;
    const double wt = fma(c.tol, abs_max(y, yn), c.tol);
    const double est = fma(0.4 * h, fn + f, 0.8 * (yn - y));
    E err;
    if constexpr (FAST) {
      const float qv = d2f(est) / d2f(wt), q = qv * qv;
      float e2 = __shfl_sync(mask, q, 0, 4);
#pragma unroll
      for (int i = 1; i < NC; i++) e2 += __shfl_sync(mask, q, i, 4);
      err = sqrtf(e2 * 0.25f);
    } else {
      const double qv = mdiv(est, wt);
      err = sqrt(sum4(qv * qv) * 0.25);
    }
    const int a = c.judge(err, h);
    if (a == StepCtl<E>::ATT_ACCEPT) {
      // (v2, fn, v1, yn, y) <- (fn, v1, yn, y, v2)
      const double t = v2;
      v2 = fn;
      fn = v1;
      v1 = yn;
      yn = y;
      y = t;
    }
    return a;
  }

  // Sys::ion_and_b for a single cell (no gap junctions)
  __device__ __forceinline__ void ion_due() {
    b = comp_ion_b<CT, R>(P, gi, y, c.sum_dt, true);
    c.n_ion++;
    c.sum_dt = 0.0;
  }

  __device__ __forceinline__ int begin_interval(double t) {
    if (P.stim_on && P.stim_comp[cell0] == r) {
      P.iext[gi] = 0;
      if (P.stim_t0[cell0] <= t && t < P.stim_t1[cell0]) P.iext[gi] = P.stim_amp[cell0];
    }
    attempts0 = c.n_steps;
    c.rej_run = 0;
    return fpi_is_zero(c.sum_dt) ? TICK_MORE : TICK_ION;
  }

  __device__ __forceinline__ void end_interval() {
    double a1, a2, b1, b2;
    c.dense(a1, a2, b1, b2);
    P.vnew[gi] = fma(b2, fn, fma(b1, v2, fma(a2, yn, a1 * v1)));
    c.tend += H_MAX;
    __syncwarp(mask);            // the four lanes' v_new before the records below read them
    if (P.soma_out)
      for (int k = r; k < P.rec_w; k += NC)
        P.soma_out[((long)(iv0 + k_iv) * P.ncell_pool + cell0) * P.rec_w + k] = P.vnew[P.cell_soma[cell0] + k];
    if (P.spk_prev && r == 0) log_spike(P, cell0, t0 + (k_iv + 1) * H_MAX);
    __syncwarp(mask);            // and the reads before the next interval's writes
    if (c.iv_left > 0) c.iv_left--;
  }

  // intervals k0 .. k0 + n - 1 of a launch that begins at t
  __device__ __forceinline__ int start(double t, int k0, int n, int iv0_global) {
    if (c.iv_left >= 0 && n > c.iv_left) n = c.iv_left;
    t0 = t;
    n_iv = k0 + n;
    iv0 = iv0_global;
    k_iv = k0;
    if (c.status != 0 || n <= 0) return TICK_DONE;
    return begin_interval(t0 + k0 * H_MAX);
  }

  // Sys::tick
  __device__ __forceinline__ int tick() {
    const int a = attempt();
    if (a == StepCtl<E>::ATT_REJECT) return TICK_MORE;
    if (a == StepCtl<E>::ATT_FAIL) return TICK_DONE;
    if (c.n_steps - attempts0 > STEPS_PER_INTERVAL_CAP) {
      c.status |= ST_LOOP_CAP;
      return TICK_DONE;
    }
    const bool due = c.clock(CT == GO || CT == PKJ);
    if (!c.last) return due ? TICK_ION : TICK_MORE;
    end_interval();
    if (++k_iv >= n_iv) return TICK_DONE;
    return begin_interval(t0 + k_iv * H_MAX);
  }
};

// The systems of a warp, four lanes each on its first `quads` groups of four:
// the static sequence first, first + stride, ... (q null), or systems from
// *q, and while P.ivc is less than the launch's intervals the line's (group_sys.cuh):
// with more systems than places a quad goes on with another system after
// P.ivc intervals of one.  (Whole systems in turn, 1.4 systems a place take
// the time of two, so the granule role of the mixed batch had to hold every
// cell at once, on 64 CTAs: 4.9 s a step beside 7.6 s of the other roles on
// the rest.  In turns on 42 CTAs: 6.2 s each, 16.7e9 -> 20.3e9
// compartment-updates/s.)
// A system whose ion update is due parks; the warp runs the parked systems'
// updates together once every live one is parked or the oldest has waited
// ION_WAIT_MAX iterations (run_lanes, integrator.cuh).
template <int CT, typename R>
__device__ __forceinline__ void run_quads(const PoolView<R> &P, int *q, int first, int stride, int quads, double t0,
                                          int n_iv, int iv0_global) {
  QuadSys<CT, R> S(P);
  const bool turns = q && P.ivc < n_iv;
  const int piece = turns ? P.ivc : n_iv;
  int s = -1, k = 0, r = TICK_DONE;       // the system and its next interval
  bool more = ((int)(threadIdx.x & 31) >> 2) < quads;
  // the next system, after s up to interval k (s -1: after a finished one)
  auto next = [&]() {
    if (!q) {
      s = first < P.nsys ? first : -1;
      first += stride;
      k = 0;
      return;
    }
    if (S.r == 0) {
      int got = -1, at = 0;
      if (*(volatile int *)q < P.nsys) {
        got = atomicAdd(q, 1);
        if (got >= P.nsys) got = -1;
      }
      if (got < 0 && turns) {
        got = line_take(P, 0);
        if (got >= 0) at = *(volatile int *)(P.grp_line + 2 + got);
      }
      if (got >= 0) {
        if (s >= 0) line_leave(P, s, k);
        s = got;
        k = at;
      }
    }
    s = __shfl_sync(S.mask, s, 0, 4);
    k = __shfl_sync(S.mask, k, 0, 4);
    if (turns) __threadfence();           // (a system's state may come from another SM)
  };
  auto acquire = [&]() {
    while (more) {
      next();
      if (s < 0) break;
      if (system_selected(P.ctl[s], false, n_iv)) {
        S.load(s);
        r = S.start(t0, k, min(piece, n_iv - k), iv0_global);
        if (r != TICK_DONE) return;
        __syncwarp(S.mask);
        S.store();
        __syncwarp(S.mask);
      }
      s = -1;
    }
    more = false;
    r = TICK_DONE;
  };
  acquire();
  int wait = 0;
  for (;;) {
    __syncwarp();
    const unsigned live = __ballot_sync(0xffffffffu, r != TICK_DONE);
    if (!live) break;
    const unsigned parked = __ballot_sync(0xffffffffu, r == TICK_ION);
    if (parked && (parked == live || ++wait > ION_WAIT_MAX)) {
      wait = 0;
      if (r == TICK_ION) {
        S.ion_due();
        r = TICK_MORE;
      }
      __syncwarp();
    }
    if (r == TICK_MORE) {
      r = S.tick();
      if (r == TICK_DONE) {
        __syncwarp(S.mask);
        S.store();
        k += piece;
        if (k >= n_iv || S.c.status != 0) s = -1;
        if (turns) {
          __threadfence();
          __syncwarp(S.mask);
        }
        acquire();
      }
    }
  }
}

}  // namespace gbrkc
