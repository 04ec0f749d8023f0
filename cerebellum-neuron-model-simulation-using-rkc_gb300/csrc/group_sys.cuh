// RKC integrator for one system spread over some warps of a CTA, of a cluster
// of CTAs, or (the grid team: a system alone in its engine, too large
// for a cluster) of every CTA of a cooperative launch; its five RKC vectors
// and its current b in registers, at most K elements a thread.
//
// What bounds it: a warp issues an FP64 instruction every 64 cycles whatever
// its lanes do, an SM one every 19 for all of its warps, so a stage is about
// 12 of them per element row, and the rest of a stage is the latency of handing
// the stage vector's values to the threads that read them.  So:
//  * Elements go to CTAs in runs of whole chunks of bw consecutive elements
//    (a power of two where there are several CTAs): in a tree numbered along
//    its branches most neighbours are then in the same CTA, read from shared
//    memory.
//  * A value that another CTA reads is handed over as two 64-bit words, each
//    half of the value beside the evaluation's number: two stores, and two
//    loads that poll for that number, no fence, no flag, no barrier over the
//    CTAs.
//    In a cluster the writer stores into the reader's shared memory (about
//    200 cycles), in the grid team into a slot of global memory that its
//    readers poll in the L2 (about 1500).  Slots are double-buffered.  A CTA
//    cannot overwrite a slot that its reader still polls: it writes
//    evaluation k + 2 only after evaluation k + 1 has reached it from every
//    CTA it reads from, the CTAs that read from it are the same ones (the
//    host checks that), and each of them had taken evaluation k before it
//    handed over k + 1.
//  * Sums are the pairwise tree: warp shuffles, the chunk's warp partials,
//    then every chunk's sum handed to every CTA the same way, one warp of
//    which combines them in the tree's order.  A sum thus also separates
//    everything before it from everything after it in all CTAs, so one
//    system's slots serve the next one.
// Every poll is bounded (GRID_SPIN_LIMIT) and raises the abort flag, after
// which no wait waits and the CTAs leave the system at the next attempt
// (status ST_BARRIER); a cluster, and a cooperative launch, make every CTA
// resident, so the bound is a guard, not a schedule.
//
// Measured against the block, warp and old grid teams (a launch per pass, in
// ms): full granule cell, FP64, one interval 39.5 -> 12.2 (a cluster of
// 10 CTAs of 64 threads; one CTA before); 77 Golgi cells, FP64, five
// intervals 45.5 -> 10.7 (clusters of 5 x 32); 16x16 olive network, mixed, 16
// intervals 26.9 -> 9.7 (12 x 64); Purkinje 3x3, FP64, eight intervals
// 3.7 -> 3.0 (from t = 5 ms, sums over the same windows; grid, 113 x 128: two
// fifths of it the FP64 ion updates).
//
// The arithmetic is Sys's (integrator.cuh) operation for operation.
#pragma once
#include "step_ctl.cuh"

namespace gbrkc {

constexpr long GRID_SPIN_LIMIT = 1L << 22;

enum GroupComm { GRP_CTA, GRP_CLUSTER, GRP_GRID };

// a value and its evaluation's number in one slot: {low half, number}, {high
// half, number}, each word written and read whole
template <int COMM>
__device__ __forceinline__ void word_put(unsigned long long p, unsigned long long w) {
  if constexpr (COMM == GRP_GRID)
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(w) : "memory");
  else
    asm volatile("st.relaxed.cluster.shared::cluster.u64 [%0], %1;" ::"r"((unsigned)p), "l"(w) : "memory");
}
template <int COMM>
__device__ __forceinline__ unsigned long long word_get(unsigned long long p) {
  unsigned long long w;
  if constexpr (COMM == GRP_GRID)
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(p) : "memory");
  else
    asm volatile("ld.relaxed.cluster.shared::cta.u64 %0, [%1];" : "=l"(w) : "r"((unsigned)p) : "memory");
  return w;
}
template <int COMM>
__device__ __forceinline__ void slot_put(unsigned long long p, double x, unsigned tag) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(x), t = (unsigned long long)tag << 32;
  word_put<COMM>(p, (u & 0xffffffffull) | t);
  word_put<COMM>(p + 8, (u >> 32) | t);
}
template <int COMM>
__device__ __forceinline__ bool slot_get(unsigned long long p, unsigned tag, double &x) {
  const unsigned long long a = word_get<COMM>(p), b = word_get<COMM>(p + 8);
  x = __longlong_as_double((long long)((a & 0xffffffffull) | (b << 32)));
  return (unsigned)(a >> 32) == tag && (unsigned)(b >> 32) == tag;
}
// this CTA's shared-memory address p (32 bits) in CTA `rank` of the cluster
__device__ __forceinline__ unsigned cluster_map(unsigned p, int rank) {
  unsigned q;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(q) : "r"(p), "r"(rank));
  return q;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int CT, typename R, int K, int COMM>
struct GroupSys {
  static constexpr bool MIXED = !std::is_same<R, double>::value;
  static constexpr bool ALONE = COMM == GRP_CTA;   // no other CTA takes part
  typedef StepCtl<double> SC;
  const PoolView<R> &P;
  int s, nc, ncell, ncomp, off, cell0;
  int G, cta, bw, t, bar;      // CTAs of the group, this CTA, threads a CTA, this thread, the CTA team's barrier
  int chunk0, rows, e0, L;     // this CTA's chunks, its first element, its element places
  int r0, nrecv;               // its received values
  const GroupTab *tab;
  int ld, pairs, us;           // places of the row tables (the fullest CTA's elements), neighbour pairs, places of a stage buffer
  // shared memory
  double *u;                   // [2][us]: the stage vector, own places, received ones behind them, and a zero
  // the row tables: pairs of neighbours, [pairs][ld] (conductance, conductance)
  // -- mixed precision: g / Cm -- and [pairs][ld] their places in the stage
  // buffer, as byte offsets of 16 bits each; [ld] 1/Cm (mixed: the row sums)
  double2 *lg;
  unsigned *lcol;
  double *linv;
  double *wp, *res, *coef;     // warp partials, a sum's result or a verdict (4), the step's stage coefficients
  bool due;                    // an ion update follows the accepted step
  unsigned halo, red;          // cluster: [2][most received][2] and [2][chunks][2] words, shared-memory addresses
  int coef_m;                  // stage counts whose coefficients it holds
  int *s_abort;                // [0] a wait gave up, [1] the same as of the last sum, alike for the CTA's threads
  // registers
  double y[K], yn[K], fn[K], v1[K], v2[K];
  double b[K];                 // the current; mixed precision: -b / Cm
  int slot[K];                 // grid: publishing slot, or -1
  int send0, send1;            // cluster: the thread's hand-overs (P.grp_send)
  unsigned dst;                // its first hand-over's slot in the reading CTA (evaluations of even number)
  int dstq;                    // and its element
  unsigned pc[K][2];           // the row's first two pairs of places
  int wdeg;                    // the longest row of the warp at each of its elements (four bits each; K = 1: whole)
  double2 rg[2];               // K = 1: the row's first two pairs of conductances
  SC c;
  Recip rnc;                   // 1 / nc
  unsigned tag, rtag;          // evaluations and sums so far
  double t0;
  int k_iv, n_iv, iv0;
  long long attempts0;

  // The team is the bw_ threads from first_ on, meeting at barrier bar_ (0 the
  // whole CTA's); smem: grid_smem bytes; coef_: 5 (coef_m - 1) values; wp_,
  // res_, ab: reduction words; cta_, G_: this CTA's place in its group and the
  // group's CTAs.
  __device__ GroupSys(const PoolView<R> &P_, double *smem, double *wp_, double *res_, double *coef_, int coef_m_,
                      int *ab, int first_, int bw_, int bar_, int cta_, int G_)
      : P(P_), wp(wp_), res(res_), coef(coef_), coef_m(coef_m_), s_abort(ab) {
    t = (int)threadIdx.x - first_;
    bw = bw_;
    bar = bar_;
    G = G_;
    cta = cta_;
    ld = P.grp_ld;
    pairs = (P.grid_maxdeg + 1) >> 1;
    us = ld + 1 + (ALONE ? 0 : P.grp_recv_max);
    us += us & 1;
    u = smem;
    lg = (double2 *)(u + 2 * us);
    linv = (double *)(lg + pairs * ld);
    lcol = (unsigned *)(linv + ld);
    tag = rtag = 0;
    if constexpr (COMM == GRP_CLUSTER) {
      // slots behind the rows, numbered 0 before any hand-over
      unsigned long long *w = (unsigned long long *)(((unsigned long long)(lcol + pairs * ld) + 15) & ~15ull);
      const int rm = P.grp_recv_max, n = 4 * rm + 4 * GRID_MAX_ROWS * G;
      for (int i = t; i < n; i += bw) w[i] = 0ull;
      halo = (unsigned)__cvta_generic_to_shared(w);
      red = halo + 32 * rm;
      cluster_sync_all();
    }
  }
  __device__ __forceinline__ void sync() const {
    if constexpr (COMM == GRP_CTA) asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(bw) : "memory");
    else __syncthreads();
  }
  // every CTA of the group
  __device__ __forceinline__ void group_sync() const {
    if constexpr (COMM == GRP_CLUSTER) cluster_sync_all();
    else sync();
  }
  // no CTA leaves while a peer may still store into its shared memory
  __device__ __forceinline__ void leave() const {
    if constexpr (COMM == GRP_CLUSTER) cluster_sync_all();
  }

  __device__ __forceinline__ int at(int k) const { return e0 + k * bw + t; }
  __device__ __forceinline__ bool has(int k) const { return k < rows && at(k) < nc; }
  __device__ __forceinline__ const double *ucur() const { return u + (tag & 1u) * us; }

  // Take the system: its operator rows into shared memory, its vectors into
  // registers.
  __device__ __forceinline__ void bind(int s_) {
    s = s_;
    nc = P.sys_nc[s];
    ncell = P.sys_ncell[s];
    ncomp = P.sys_ncomp[s];
    off = P.sys_off[s];
    cell0 = P.sys_cell0[s];
    if constexpr (ALONE) {
      chunk0 = 0;
      rows = (nc + bw - 1) / bw;
      r0 = nrecv = 0;
    } else {
      tab = P.grp_tab + s;
      chunk0 = P.grp_chunk0[tab->chunk0 + cta];
      rows = P.grp_chunk0[tab->chunk0 + cta + 1] - chunk0;
      r0 = P.grp_rptr[tab->rptr + cta];
      nrecv = P.grp_rptr[tab->rptr + cta + 1] - r0;
    }
    e0 = chunk0 * bw;
    L = rows * bw;
    send0 = send1 = dstq = 0;
    dst = 0u;
    const int k = P.sys_csr[s], tm = P.sys_tmpl[s];
    const bool csr = k >= 0;
    const int *row = csr ? P.s_row + P.s_row0[k] : P.t_row + P.t_row0[tm];
    const long nz0 = csr ? P.s_nz0[k] : P.t_nz0[tm], cm0 = csr ? P.s_cm0[k] : P.t_cm0[tm];
    const double *g = (MIXED ? (csr ? P.s_gc : P.t_gc) : (csr ? P.s_g : P.t_g)) + nz0;
    const double *inv = (csr ? P.s_invcm : P.t_invcm) + cm0, *Gc = (csr ? P.s_Gc : P.t_Gc) + cm0;
    const int *map = P.ctl[s].map;
    const long ncp = (nc + 1) & ~1;
    const double *ws = P.ws + P.sys_ws[s];
    const int *pcol = (csr ? P.s_col + P.s_nz0[k] : P.t_col + P.t_nz0[tm]);
    if constexpr (!ALONE) pcol = P.grp_col + tab->col;
    c.load(P.ctl[s]);
    sync();               // the last system's readers of the tables are done
    if (t < 2) u[t * us + us - 1] = 0.0;      // the zero
    wdeg = 0;
#pragma unroll
    for (int q = 0; q < K; q++) {
      y[q] = yn[q] = fn[q] = v1[q] = v2[q] = b[q] = 0.0;
      slot[q] = -1;
      // a row's surplus entries: conductance -0 at the zero (mixed precision)
      // or at the element itself, so that they add -0, which changes nothing
      const int lr = q * bw + t;
      const unsigned none = 8u * (unsigned)(MIXED ? us - 1 : lr);
      if (lr < ld) {
        linv[lr] = 0.0;
        for (int j = 0; j < pairs; j++) {
          lg[j * ld + lr] = make_double2(-0.0, -0.0);
          lcol[j * ld + lr] = none | none << 16;
        }
        u[lr] = u[us + lr] = 0.0;
      }
      pc[q][0] = pc[q][1] = none | none << 16;
      int cnt = 0;
      if (has(q)) {
        // (cells of one template lie one after another)
        const int i = at(q), base = csr ? 0 : i - i % ncomp, ri = i - base;
        const int a = __ldg(row + ri), z = __ldg(row + ri + 1);
        cnt = z - a;
        linv[lr] = MIXED ? __ldg(Gc + ri) : __ldg(inv + ri);
        for (int j = 0; j < cnt; j++) {
          const unsigned place = 8u * (unsigned)((ALONE ? base : 0) + __ldg(pcol + a + j));
          double2 &gp = lg[(j >> 1) * ld + lr];
          unsigned &cp = lcol[(j >> 1) * ld + lr];
          if (j & 1) {
            gp.y = __ldg(g + a + j);
            cp = (cp & 0xffffu) | place << 16;
          } else {
            gp.x = __ldg(g + a + j);
            cp = (cp & 0xffff0000u) | place;
          }
        }
        pc[q][0] = pairs > 0 ? lcol[lr] : pc[q][0];
        pc[q][1] = pairs > 1 ? lcol[ld + lr] : pc[q][1];
        y[q] = ws[map[LY] * ncp + i];
        yn[q] = ws[map[LYN] * ncp + i];
        fn[q] = ws[map[LFN] * ncp + i];
        v1[q] = ws[map[LV1] * ncp + i];
        v2[q] = ws[map[LV2] * ncp + i];
        b[q] = ws[WS_B * ncp + i];
        if constexpr (MIXED) b[q] = -b[q] * __ldg(inv + ri);
      if constexpr (COMM == GRP_GRID) slot[q] = P.grp_slot[tab->slot + i];
      if constexpr (COMM == GRP_CLUSTER) {
        // (a thread of several elements hands over in exchange's own loop)
        if (q == 0) {
          send0 = P.grp_sptr[tab->sptr + (cta * bw) + t];
          send1 = P.grp_sptr[tab->sptr + (cta * bw) + t + 1];
          if (send0 < send1) {
            const int d = __ldg(P.grp_send + tab->send + send0);
            dst = cluster_map(halo + 16u * (d & 0xffff), (d >> 16) & 255);
            dstq = d >> 24;
          }
        }
      }
      }
      // the warp's longest row here
#pragma unroll
      for (int st = 16; st > 0; st /= 2) cnt = max(cnt, __shfl_xor_sync(0xffffffffu, cnt, st));
      if constexpr (K > 1 && COMM == GRP_GRID) cnt = min(cnt, 15);
      wdeg |= cnt << (4 * q);
    }
    if constexpr (K == 1) {
      rg[0] = pairs > 0 && t < ld ? lg[t] : make_double2(-0.0, -0.0);
      rg[1] = pairs > 1 && t < ld ? lg[ld + t] : make_double2(-0.0, -0.0);
    }
    sync();
  }

  __device__ __forceinline__ void set_b(int q, double x) {
    if constexpr (MIXED) {
      // -b / Cm; 1/Cm is read here only
      const int k = P.sys_csr[s], i = at(q);
      b[q] = -x * (k >= 0 ? __ldg(P.s_invcm + P.s_cm0[k] + i) : __ldg(P.t_invcm + P.t_cm0[P.sys_tmpl[s]] + i % ncomp));
    } else {
      b[q] = x;
    }
  }

  // (b itself is written at each ion update)
  __device__ __forceinline__ void store(bool init) const {
    const int *map = P.ctl[s].map;
    const long ncp = (nc + 1) & ~1;
    double *ws = P.ws + P.sys_ws[s];
#pragma unroll
    for (int q = 0; q < K; q++)
      if (has(q)) {
        const int i = at(q);
        ws[map[LY] * ncp + i] = y[q];
        ws[map[LYN] * ncp + i] = yn[q];
        ws[map[LFN] * ncp + i] = fn[q];
        ws[map[LV1] * ncp + i] = v1[q];
        ws[map[LV2] * ncp + i] = v2[q];
      }
    if (cta == 0 && t == 0) c.store(P.ctl[s], init);
  }

  // Poll a slot for evaluation or sum `want`.
  __device__ __forceinline__ double wait(unsigned long long p, unsigned want) const {
    double x;
    long it = 0;
    while (!slot_get<COMM>(p, want, x)) {
      if ((++it & 255) == 0) {
        volatile int *ab = P.grp_abort;
        if (*ab || it > GRID_SPIN_LIMIT) {
          *ab = 1;
          *(volatile int *)s_abort = 1;
          break;
        }
      }
    }
    return x;
  }

  // Hand the stage vector val to its readers: own values into shared memory,
  // those other CTAs read into their slots, the received ones behind the own.
  __device__ __forceinline__ void exchange(const double (&val)[K]) {
    tag++;
    const unsigned par = tag & 1u;
    double *ub = u + par * us;
    if constexpr (COMM == GRP_GRID) {
      const unsigned long long h = (unsigned long long)(P.grp_halo + (long)par * P.grp_nslots * 2);
#pragma unroll
      for (int q = 0; q < K; q++)
        if (has(q)) {
          if (slot[q] >= 0) slot_put<COMM>(h + 16ull * slot[q], val[q], tag);
          ub[q * bw + t] = val[q];
        }
      for (int j = t; j < nrecv; j += bw)
        ub[L + j] = wait(h + 16ull * __ldg(P.grp_rslot + tab->rslot + r0 + j), tag);
    } else {
#pragma unroll
      for (int q = 0; q < K; q++)
        if (has(q)) ub[q * bw + t] = val[q];
      if constexpr (COMM == GRP_CLUSTER) {
        const unsigned h = halo + par * 16u * P.grp_recv_max;
        auto pick = [&](int q) {
          double x = val[0];
#pragma unroll
          for (int k = 1; k < K; k++)
            if (k == q) x = val[k];
          return x;
        };
        if (send0 < send1) slot_put<COMM>(dst + par * 16u * P.grp_recv_max, pick(dstq), tag);
        for (int j = send0 + 1; j < send1; j++) {
          // this thread's element, reading CTA, its slot
          const int d = __ldg(P.grp_send + tab->send + j);
          slot_put<COMM>(cluster_map(h + 16u * (d & 0xffff), (d >> 16) & 255), pick(d >> 24), tag);
        }
        for (int j = t; j < nrecv; j += bw) ub[L + j] = wait(h + 16u * j, tag);
      }
    }
    sync();
  }

  // dydt at the thread's elements, whose stage values are ui (Sys::rhs).  A
  // row of a warp runs to its longest row, in pairs of neighbours.
  __device__ __forceinline__ void rhs(const double (&ui)[K], double (&f)[K]) const {
    const char *ub = (const char *)ucur();
    auto term = [&](double g, unsigned o, double v, double d) {
      const double x = *(const double *)(ub + o);
      return fma(g, MIXED ? x : x - v, d);
    };
#pragma unroll
    for (int q = 0; q < K; q++) {
      f[q] = 0.0;
      if (K > 1 && q >= rows) break;
      const int lr = q * bw + t, n = deg(q);
      double d = MIXED ? b[q] : -b[q];
      if (n > 0) {
        const double2 g = K == 1 ? rg[0] : lg[lr];
        d = term(g.x, pc[q][0] & 0xffffu, ui[q], d);
        if (n > 1) d = term(g.y, pc[q][0] >> 16, ui[q], d);
      }
      if (n > 2) {
        const double2 g = K == 1 ? rg[1] : lg[ld + lr];
        d = term(g.x, pc[q][1] & 0xffffu, ui[q], d);
        if (n > 3) d = term(g.y, pc[q][1] >> 16, ui[q], d);
      }
      for (int j = 4; j < n; j += 2) {
        const double2 g = lg[(j >> 1) * ld + lr];
        const unsigned p = lcol[(j >> 1) * ld + lr];
        d = term(g.x, p & 0xffffu, ui[q], d);
        if (n > j + 1) d = term(g.y, p >> 16, ui[q], d);
      }
      if constexpr (MIXED) f[q] = fma(-linv[lr], ui[q], d);
      else f[q] = d * linv[lr];
    }
  }
  __device__ __forceinline__ int deg(int q) const {
    if constexpr (K == 1) return wdeg;
    const int n = (int)((unsigned)wdeg >> (4 * q)) & 15;
    // (grid: 15 stands for 15 and more, a row run to the longest row's end)
    if constexpr (COMM == GRP_GRID) return n < 15 ? n : 2 * pairs;
    return n;
  }

  // the pairwise tree over a[0..8) of which n are there
  static __device__ __forceinline__ double tree8(double (&w)[8], int n) {
#pragma unroll
    for (int st = 1; st < 8; st *= 2)
#pragma unroll
      for (int j = 0; j + st < 8; j += 2 * st) {
        const double x = w[j] + w[j + st];
        w[j] = j + st < n ? x : w[j];
      }
    return w[0];
  }

  // the pairwise tree over the system's elements of x, the same in every thread
  __device__ __forceinline__ double sum(const double (&x)[K]) {
    total(x, [&](double e) {
      if (t == 0) *res = e;
    });
    return *res;
  }
  // ... or what its first warp makes of it, between the sum and the barrier
  template <class F>
  __device__ __forceinline__ void total(const double (&x)[K], F fin) {
    if constexpr (ALONE && K > 2) sum8(x, fin);
    else sum_rows(x, fin);
  }

  // Many elements a thread: through shared memory, a thread eight consecutive
  // values at a time, then a warp eight such sums a lane (systems of up to
  // 2048 elements): 61 FP64 additions for 1600 elements where a shuffle tree
  // per row takes 280.
  template <class F>
  __device__ __forceinline__ void sum8(const double (&x)[K], F fin) {
    double *sc = u + ((tag + 1u) & 1u) * us;    // the next evaluation's buffer
#pragma unroll
    for (int q = 0; q < K; q++)
      if (has(q)) sc[q * bw + t] = x[q];
    sync();
    const int n8 = (nc + 7) >> 3;
    double a = 0.0;
    for (int k = t; k < n8; k += bw) {
      double w[8];
#pragma unroll
      for (int j = 0; j < 8; j++) w[j] = 8 * k + j < nc ? sc[8 * k + j] : 0.0;
      a = tree8(w, nc - 8 * k);
      if (n8 > 32) sc[8 * k] = a;
    }
    int nb = n8;
    if (n8 > 32) {
      sync();
      nb = (n8 + 7) >> 3;
      if (t < 32) {
        double w[8];
#pragma unroll
        for (int j = 0; j < 8; j++) w[j] = 8 * t + j < n8 ? sc[64 * t + 8 * j] : 0.0;
        a = tree8(w, n8 - 8 * t);
      }
    }
    if (t < 32) {
#pragma unroll
      for (int st = 1; st < 32; st *= 2) {
        if (st >= nb) break;
        const double o = __shfl_down_sync(0xffffffffu, a, st);
        if ((t & (2 * st - 1)) == 0 && t + st < nb) a = a + o;
      }
      fin(__shfl_sync(0xffffffffu, a, 0));
    }
    sync();
  }

  template <class F>
  __device__ __forceinline__ void sum_rows(const double (&x)[K], F fin) {
    const int lane = t & 31, warp = t >> 5, nw = bw >> 5;
#pragma unroll
    for (int q = 0; q < K; q++) {
      if (q >= rows) break;
      const int i = at(q);
      double a = i < nc ? x[q] : 0.0;
#pragma unroll
      for (int st = 1; st < 32; st *= 2) {
        const double o = __shfl_down_sync(0xffffffffu, a, st);
        if ((lane & (2 * st - 1)) == 0 && i + st < nc) a = a + o;
      }
      if (lane == 0) wp[q * nw + warp] = a;
    }
    rtag++;
    sync();
    if (warp == 0) {
      // the parts that the tree goes on with: the CTA's 32-element parts (one
      // CTA), or every chunk's sum
      constexpr int VM = COMM == GRP_GRID ? GRID_MAX_BLOCKS / 32 : COMM == GRP_CLUSTER ? 4 : 2;   // (one CTA: 64 parts)
      int nb, rr;
      double v[VM];
      if constexpr (ALONE) {
        nb = (nc + 31) >> 5;
        rr = nb <= 32 ? 1 : 2;
#pragma unroll
        for (int j = 0; j < VM; j++) v[j] = (j < rr && lane * rr + j < nb) ? wp[lane * rr + j] : 0.0;
      } else {
        unsigned long long rd;
        if constexpr (COMM == GRP_GRID) rd = (unsigned long long)(P.grp_red + (long)(rtag & 1u) * GRID_MAX_BLOCKS * 2);
        else rd = red + (rtag & 1u) * 16u * GRID_MAX_ROWS * G;
        if (lane < rows) {
          const int i0 = (chunk0 + lane) * bw;
          double w[8];
#pragma unroll
          for (int j = 0; j < 8; j++) w[j] = j < nw ? wp[lane * nw + j] : 0.0;
#pragma unroll
          for (int st = 1; st < 8; st *= 2)
#pragma unroll
            for (int j = 0; j + st < 8; j += 2 * st)
              if (j + st < nw && i0 + (j + st) * 32 < nc) w[j] = w[j] + w[j + st];
          if constexpr (COMM == GRP_GRID) slot_put<COMM>(rd + 16ull * (chunk0 + lane), w[0], rtag);
          else wp[lane * nw] = w[0];
        }
        if constexpr (COMM == GRP_CLUSTER) {
          __syncwarp();
          // one lane a CTA
          if (lane < G)
            for (int k = 0; k < rows; k++)
              slot_put<COMM>(cluster_map((unsigned)rd + 16u * (chunk0 + k), lane), wp[k * nw], rtag);
        }
        // each lane takes rr consecutive chunk sums
        nb = (nc + bw - 1) / bw;
        rr = nb <= 32 ? 1 : nb <= 64 ? 2 : nb <= 128 ? 4 : 8;
#pragma unroll
        for (int j = 0; j < VM; j++) {
          const int k = lane * rr + j;
          v[j] = (j < rr && k < nb) ? wait(rd + 16ull * k, rtag) : 0.0;
        }
      }
#pragma unroll
      for (int st = 1; st < VM; st *= 2) {
        if (st >= rr) break;
#pragma unroll
        for (int j = 0; j + st < VM; j += 2 * st)
          if (j + st < rr && lane * rr + j + st < nb) v[j] = v[j] + v[j + st];
      }
#pragma unroll
      for (int st = 1; st < 32; st *= 2) {
        if (st * rr >= nb) break;
        const double o = __shfl_down_sync(0xffffffffu, v[0], st);
        if ((lane & (2 * st - 1)) == 0 && (lane + st) * rr < nb) v[0] = v[0] + o;
      }
      fin(__shfl_sync(0xffffffffu, v[0], 0));
      if constexpr (!ALONE)
        if (lane == 0) s_abort[1] = *(volatile int *)s_abort;
    }
    sync();
  }

  // The error norm and the controller's verdict.  In a CTA of its own they are
  // the work of the warp that ends the sum, and the others take what they
  // need of it: the controller's 60 FP64 instructions took 7200 cycles an
  // attempt in each of eight warps, 4000 in one (Golgi cells, five warps:
  // 37.4 -> 36.7 ms for 2048 cells).  The warps of a cluster or grid team
  // have their SM's FP64 pipe nearly to themselves, and each repeats them
  // (handing the verdict over took 16 x 16 olives from 9.5 to 10.1 ms).
  __device__ __forceinline__ int verdict(const double (&d)[K], double h) {
    if constexpr (!ALONE) {
      const int a = c.judge(norm(sum(d)), h);
      due = a == SC::ATT_ACCEPT && c.clock(CT == GO || CT == PKJ);
      return a;
    }
    total(d, [&](double e) {
      const int a = c.judge(norm(e), h);
      due = a == SC::ATT_ACCEPT && c.clock(CT == GO || CT == PKJ);
      if (t == 0) {
        res[0] = c.absh; res[1] = c.lt; res[2] = c.sum_dt;
        int *r = (int *)(res + 3);
        r[0] = c.status;
        r[1] = (a + 1) * 2 + (due ? 1 : 0);
      }
    });
    const int *r = (const int *)(res + 3);
    const int a = (r[1] >> 1) - 1;
    due = (r[1] & 1) != 0;
    c.absh = res[0];
    c.status = r[0];
    if (a == SC::ATT_ACCEPT) {
      c.lt = c.gt_old = c.hw1 = res[1];
      c.hw0 = h;
      c.sum_dt = res[2];
      c.jacatt = c.newspc = 0;
    } else if (a == SC::ATT_REJECT) {
      c.newspc = !c.jacatt;
    }
    return a;
  }

  __device__ __forceinline__ double sumsq(const double (&x)[K]) {
    double q[K];
#pragma unroll
    for (int j = 0; j < K; j++) q[j] = x[j] * x[j];
    return sum(q);
  }

  // Sys::rkcrho
  __device__ __forceinline__ void rkcrho() {
    const double uround = UROUND, sqrtu = sqrt(UROUND);
    double e[K];
#pragma unroll
    for (int q = 0; q < K; q++) e[q] = has(q) ? P.ede[off + at(q)] : 0.0;
    c.n_rho++;
    const double ynrm = sqrt(sumsq(yn));
    const double vnrm = sqrt(sumsq(e));
    double dynrm, al = 0.0;
    const bool zy = fpi_is_zero(ynrm), zv = fpi_is_zero(vnrm);
    dynrm = zy ? uround : ynrm * sqrtu;
    if (!zv) al = mdiv(dynrm, vnrm);
#pragma unroll
    for (int q = 0; q < K; q++)
      v1[q] = !zy ? (!zv ? fma(al, e[q], yn[q]) : fma(sqrtu, yn[q], yn[q])) : (!zv ? al * e[q] : dynrm);
    RhoCtl rc;
    rc.begin(dynrm);
    for (int iter = 0; iter < RHO_ITMAX; iter++) {
      c.n_rho_iter++;
      exchange(v1);
      double d[K];
      rhs(v1, v2);
#pragma unroll
      for (int q = 0; q < K; q++) {
        const double dm = -1.0 * fn[q] + v2[q];
        d[q] = dm * dm;
      }
      const double dfnrm = sqrt(sum(d));
      if (rc.next(iter, dfnrm, c.sprad) == RhoCtl::DONE) {
#pragma unroll
        for (int q = 0; q < K; q++)
          if (has(q)) P.ede[off + at(q)] = -1.0 * yn[q] + v1[q];
        return;
      }
      if (!fpi_is_zero(dfnrm)) {
        const double a2 = mdiv(dynrm, dfnrm);
#pragma unroll
        for (int q = 0; q < K; q++) v1[q] = fma(a2, fn[q] - v2[q], yn[q]);
      } else {
        const int idx = iter % nc;
#pragma unroll
        for (int q = 0; q < K; q++)
          if (has(q) && at(q) == idx) v1[q] = 2.0 * yn[q] - v1[q];
      }
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
    // the stages' coefficients into shared memory (the first evaluation's
    // barrier publishes them): one trip to the L2 a step, not one a stage
    const bool near = m <= coef_m;
    if (near)
      for (int i = t; i < 5 * (m - 1); i += bw) coef[i] = __ldg(T + 1 + i);
    const double hm1 = h * __ldg(T);
#pragma unroll
    for (int q = 0; q < K; q++) {
      v2[q] = yn[q];
      v1[q] = fma(hm1, fn[q], yn[q]);
    }
    for (int j = 1; j < m; j++) {
      exchange(v1);
      double mu, nu, omn, mus, ajm1;
      if (near) {
        const double *p = coef + 5 * (j - 1);
        mu = p[0]; nu = p[1]; omn = p[2]; mus = p[3]; ajm1 = p[4];
      } else {
        const double *p = T + 1 + 5 * (j - 1);
        mu = __ldg(p); nu = __ldg(p + 1); omn = __ldg(p + 2); mus = __ldg(p + 3); ajm1 = __ldg(p + 4);
      }
      const double hm = h * mus;
      double f[K];
      rhs(v1, f);
#pragma unroll
      for (int q = 0; q < K; q++) {
        if (q >= rows) break;
        double w = mu * v1[q];
        w = fma(nu, v2[q], w);
        w = fma(omn, yn[q], w);
        const double out = fma(hm, fma(-ajm1, fn[q], f[q]), w);
        // written to y, then (v2, v1, y) <- (v1, y, v2)
        y[q] = v2[q];
        v2[q] = v1[q];
        v1[q] = out;
      }
    }
    // (y, v1, v2) <- (v1, v2, y)
#pragma unroll
    for (int q = 0; q < K; q++) {
      const double w = y[q];
      y[q] = v1[q];
      v1[q] = v2[q];
      v2[q] = w;
    }
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
    if (!c.plan(h, m) || !step(h, m)) return SC::ATT_FAIL;
    c.n_steps++;
    exchange(y);
    const double h04 = 0.4 * h;
    double d[K], f[K];
    rhs(y, f);
#pragma unroll
    for (int q = 0; q < K; q++) {
      d[q] = 0.0;
      if (q < rows) {
        v1[q] = f[q];
        const double wt = fma(c.tol, abs_max(y[q], yn[q]), c.tol);
        const double est = fma(h04, fn[q] + f[q], 0.8 * (yn[q] - y[q]));
        const double qv = mdiv(est, wt);
        d[q] = qv * qv;
      }
    }
    const int a = verdict(d, h);
    if (a == SC::ATT_ACCEPT) {
      // (v2, fn, v1, yn, y) <- (fn, v1, yn, y, v2)
#pragma unroll
      for (int q = 0; q < K; q++) {
        const double w = v2[q];
        v2[q] = fn[q];
        fn[q] = v1[q];
        v1[q] = yn[q];
        yn[q] = y[q];
        y[q] = w;
      }
    }
    return a;
  }

  // sqrt(e / nc); a division by a power of two is an exact scaling
  __device__ __forceinline__ double norm(double e) const {
    if ((nc & (nc - 1)) == 0) return sqrt(e * __longlong_as_double((long long)(1023 - (__ffs(nc) - 1)) << 52));
    return sqrt(div_by(e, rnc));
  }

  // Sys::ion_and_b.  The elements go through shared memory so that the ion
  // update's code stands once, not K times.  (Every reader of both stage
  // buffers is done: a sum's barriers, or bind's, lie between.)
  __device__ __forceinline__ void ion_and_b(double sum_dt, bool update_ion, bool with_gap) {
    const bool gap = CT == IO && with_gap && P.sys_ngap[s] > 0;
    if (gap) {
      // the gap currents read the receiving and sending dendrites' elem v,
      // which this update sets to y
      exchange(y);
    } else {
      double *ub = u + ((tag + 1u) & 1u) * us;
#pragma unroll
      for (int q = 0; q < K; q++)
        if (has(q)) ub[q * bw + t] = y[q];
    }
    const double *yb = gap ? ucur() : u + ((tag + 1u) & 1u) * us;
    double *bb = u + (gap ? (tag + 1u) & 1u : tag & 1u) * us;
    const long ncp = (nc + 1) & ~1;
    double *wsb = P.ws + P.sys_ws[s] + WS_B * ncp;
#pragma unroll 1
    for (int q = 0; q < K; q++) {
      if (!has(q)) break;
      const int lr = q * bw + t, i = at(q);
      double x = comp_ion_b<CT, R>(P, off + i, yb[lr], sum_dt, update_ion);
      const int cell = i / ncomp, e0g = P.sys_gap0[s] + 4 * cell;
      if (gap && i == P.gap_post[e0g]) {
        // per receiving dendrite its four edges in order (io_gap_update +
        // add_io_gap_val)
        for (int k = 0; k < 4; k++) {
          int pre;
          if constexpr (ALONE) pre = P.gap_pre[e0g + k];
          else pre = P.grp_gap[e0g + k];
          const double diff = pre >= 0 ? yb[lr] - yb[pre] : 0.0;
          x += io_gap_current(P.gap_g[e0g + k], diff);
        }
      }
      bb[lr] = x;
      wsb[i] = x;
    }
#pragma unroll
    for (int q = 0; q < K; q++)
      if (has(q)) set_b(q, bb[q * bw + t]);
    if (update_ion) c.n_ion++;
  }

  // Sys::initialize
  __device__ __forceinline__ void initialize() {
#pragma unroll
    for (int q = 0; q < K; q++) {
      v1[q] = v2[q] = 0.0;
      if (has(q)) {
        const double v0 = P.v[off + at(q)];
        P.vnew[off + at(q)] = v0;
        y[q] = yn[q] = v0;
      }
    }
    ion_and_b(0.0, false, false);
    exchange(yn);
    rhs(yn, fn);
#pragma unroll
    for (int q = 0; q < K; q++)
      if (has(q)) P.ede[off + at(q)] = fn[q];
    rkcrho();
    // set_initial_absh (solve_rkc.cu:493-560)
    double absh = H_MAX;
    if (c.sprad * absh > 1.0) absh = 1.0 / c.sprad;
    absh = (absh > c.hmin) ? absh : c.hmin;
#pragma unroll
    for (int q = 0; q < K; q++) v1[q] = fma(absh, fn[q], yn[q]);
    exchange(v1);
    double d[K];
    rhs(v1, v2);
#pragma unroll
    for (int q = 0; q < K; q++) {
      d[q] = 0.0;
      if (has(q)) {
        const double wt = fma(c.tol, fabs(yn[q]), c.tol);
        const double dm = (v2[q] - fn[q]) * (1.0 / wt);
        d[q] = dm * dm;
      }
    }
    double est = sum(d);
    est = absh * sqrt(est / nc);
    if (0.1 * absh < H_MAX * sqrt(est)) {
      const double a2 = 0.1 * absh / sqrt(est);
      absh = (a2 > c.hmin) ? a2 : c.hmin;
    } else {
      absh = H_MAX;
    }
    c.absh = absh;
    const double x = sqrt(c.tol / (10.0 * UROUND));
    c.mmax = (x - (double)(int)x < 0.5) ? (int)x : (int)(x + 0.9);
  }

  // Sys::begin_interval; every thread sees to its own elements
  __device__ __forceinline__ int begin_interval(double tb) {
    if (P.stim_on) {
#pragma unroll
      for (int q = 0; q < K; q++)
        if (has(q)) {
          const int i = at(q), cell = i / ncomp, pc = cell0 + cell;
          if (P.stim_comp[pc] == i - cell * ncomp) {
            P.iext[off + i] = 0;
            if (P.stim_t0[pc] <= tb && tb < P.stim_t1[pc]) P.iext[off + i] = P.stim_amp[pc];
          }
        }
    }
    if (P.syn_mode == SYN_BUFFERED || P.syn_mode == SYN_BUFFERED_DECAY) {
#pragma unroll
      for (int q = 0; q < K; q++)
        if (has(q)) {
          const long gi = off + at(q);
          double acc = 0.0;
          for (int k = P.syn_row[gi]; k < P.syn_row[gi + 1]; k++) {
            const int sid = P.syn_idx[k];
            acc = acc + P.syn_val[sid] * (y[q] - P.syn_e[sid]);
          }
          P.syn_buf[gi] = acc;
        }
    }
    attempts0 = c.n_steps;
    c.rej_run = 0;
    return fpi_is_zero(c.sum_dt) ? TICK_MORE : TICK_ION;
  }

  // rkcint at the interval's end, the soma record and the raster, each by the
  // thread that owns the element
  __device__ __forceinline__ void end_interval() {
    double a1, a2, b1, b2;
    c.dense(a1, a2, b1, b2);
    const double tend = t0 + (k_iv + 1) * H_MAX;
#pragma unroll
    for (int q = 0; q < K; q++)
      if (has(q)) {
        const int i = at(q), gi = off + i, pc = cell0 + i / ncomp;
        const double x = fma(b2, fn[q], fma(b1, v2[q], fma(a2, yn[q], a1 * v1[q])));
        P.vnew[gi] = x;
        if (P.soma_out) {
          const int k = gi - P.cell_soma[pc];
          if (k >= 0 && k < P.rec_w) P.soma_out[((long)(iv0 + k_iv) * P.ncell_pool + pc) * P.rec_w + k] = x;
        }
        if (P.spk_prev && gi == P.cell_spk[pc]) log_spike(P, pc, tend);
      }
    c.tend += H_MAX;
    if (c.iv_left > 0) c.iv_left--;
  }

  __device__ __forceinline__ int start(double tb, int k0, int n, int iv0_global) {
    if (c.iv_left >= 0 && n > c.iv_left) n = c.iv_left;
    t0 = tb;
    n_iv = k0 + n;
    iv0 = iv0_global;
    k_iv = k0;
    rnc = recip((double)nc);
    if (c.status != 0 || n <= 0) return TICK_DONE;
    return begin_interval(t0 + k0 * H_MAX);
  }

  // Sys::tick
  __device__ __forceinline__ int tick() {
    const int a = attempt();
    if (a == SC::ATT_REJECT) return TICK_MORE;
    if (a == SC::ATT_FAIL) return TICK_DONE;
    if (c.n_steps - attempts0 > STEPS_PER_INTERVAL_CAP) {
      c.status |= ST_LOOP_CAP;
      return TICK_DONE;
    }
    if (!c.last) return due ? TICK_ION : TICK_MORE;
    end_interval();
    if (++k_iv >= n_iv) return TICK_DONE;
    return begin_interval(t0 + k_iv * H_MAX);
  }

  __device__ __forceinline__ bool gave_up() const {
    if constexpr (ALONE) return false;
    else return s_abort[1] != 0;
  }

  // Advance the system by n intervals, the launch's k0-th and on (the launch
  // begins at tb), or initialise it.
  template <bool INIT = true>
  __device__ __forceinline__ void run(int s_, double tb, int k0, int n, int iv0_global, bool init) {
    if (!system_selected(P.ctl[s_], init, n)) return;
    if constexpr (!ALONE)
      if (t == 0) s_abort[0] = s_abort[1] = 0;
    bind(s_);
    if (INIT && init) {
      initialize();
      c.status &= ~ST_INIT;
      if (gave_up()) c.status |= ST_BARRIER;
    } else {
      int r = start(tb, k0, n, iv0_global);
      if (r == TICK_DONE) return;
      while (r != TICK_DONE) {
        if (r == TICK_ION) {
          ion_and_b(c.sum_dt, true, true);
          c.sum_dt = 0.0;
          r = TICK_MORE;
        } else {
          r = tick();
          if (gave_up()) {
            c.status |= ST_BARRIER;
            break;
          }
        }
      }
    }
    store(init);
  }
};

// The line of systems that teams take turns with.  With more systems than
// teams a launch in whole systems ends with most teams idle (200 Purkinje
// cells on 152 CTAs take two cells' time).  So a team goes on with another
// system after P.ivc intervals of one, as long as systems wait: it takes the
// longest-waiting one and leaves its own at the end of the line, and goes on
// with its own when none waits.  Every unfinished system is thus in the line
// or with a running team, nothing waits for a particular one, and the line
// only shortens.  Counters (zeroed per launch): [-1] waiting beyond the first
// round, [0] taken, [1] left, by additions only (with compare and swap, 9700
// quads that ended an interval together took 47 million tries: 26000 granule
// cells 107 to 171 ms, 75 without turns).  Place i of the line is order[i] for
// i < first (the systems with work), else line[i - first] - 1 once it is
// written; at[s] is the system's next interval.  A system that stops, or whose
// budget ends, leaves the line.  Systems that took much longer than the others in the launch
// before come first in order, and those that may decide the launch's length
// are held: no other is taken for them.  Granule quads take the first round
// from their queue (first 0), then from the line.
template <typename R>
__device__ __forceinline__ int line_take(const PoolView<R> &P, int first) {
  int *left = P.grp_line - 1;
  for (;;) {
    if (first + *(volatile int *)left <= 0) return -1;
    if (first + atomicSub(left, 1) > 0) break;
    atomicAdd(left, 1);                   // (and look again: a system may have come meanwhile)
  }
  const int h = atomicAdd(P.grp_line, 1);
  if (h < first) return P.grp_order[h];
  const int *place = P.grp_line + 2 + P.nsys + (h - first);
  // (its writer holds the place already: the store follows at once)
  int v = 0;
  for (long it = 0; it < GRID_SPIN_LIMIT && v == 0; it++)
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(place) : "memory");
  if (v == 0) *(volatile int *)P.grp_abort = 1;
  return v - 1;
}
template <typename R>
__device__ __forceinline__ void line_leave(const PoolView<R> &P, int s, int next_iv) {
  P.grp_line[2 + s] = next_iv;
  const int i = atomicAdd(P.grp_line + 1, 1);
  __threadfence();
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(P.grp_line + 2 + P.nsys + i), "r"(s + 1) : "memory");
  atomicAdd(P.grp_line - 1, 1);
}
// (one thread of the team) the next system and its first interval: after a
// finished system (s < 0) or after a piece of s up to interval k; s -1: none
template <typename R>
__device__ __forceinline__ void line_next(const PoolView<R> &P, int &s, int &k, bool &hold) {
  const int mine = s, at = k;
  if (mine >= 0 && hold) return;
  int got = line_take(P, P.grp_first);
  if (got >= 0) {
    hold = (got >> 30) != 0;
    got &= (1 << 30) - 1;
    s = got;
    k = *(volatile int *)(P.grp_line + 2 + got);
    if (mine >= 0) line_leave(P, mine, at);
  } else if (mine < 0) {
    s = -1;
  }
}

}  // namespace gbrkc
