// Device-side data layout of the RKC engine (shared by the host runtime and
// the kernels).  All cells of one type live in a "pool"; a pool holds many
// independent RKC systems (a system is what the reference integrates with one
// step size: all cells of a reference type block, or one cell, or one
// inferior-olive gap-junction network).
//
// Layout in HBM, per pool:
//   * per-system workspace, system-major: [PHYS0..PHYS4, B, SCRATCH] x nc
//     FP64 -- the five rotating RKC vectors (y, yn, fn, vtemp1, vtemp2 of
//     param.h:21, rotated by index like the reference's pointer swaps), the
//     frozen current b and a reduction scratch.  Staged into shared memory
//     for the whole launch when it fits.
//   * per-compartment SoA state: elem v, Ca, Ca2, rev_ca2, Ca_old, i_ext
//     (FP64), gating slots ion[k][i] and conductances cond[k][i] (R = FP64 or
//     FP32), the eigenvector estimate ede and the output v_new (FP64).
//   * per-template CSR of one cell's axial operator (diagonal dropped, rows
//     sorted by column, RKC sign), 1/Cm per template compartment; multi-cell
//     systems with linear gap junctions carry a system CSR instead.
#pragma once
#include <stdint.h>

#include "model.h"

namespace gbrkc {

enum { WS_PHYS = 5, WS_B = 5, WS_SCRATCH = 6, WS_VECS = 7 };

// status bits written by the kernel (never a trap)
enum Status : int {
  ST_OK = 0,
  ST_NAN = 1,          // non-finite error norm or step
  ST_LOOP_CAP = 2,     // step loop exceeded its iteration bound
  ST_COEF_TABLE = 4,   // stage count beyond the coefficient table
  ST_IDID = 8,         // rkclow returned an idid other than 1/2 (solve_rkc.cu:1155)
  ST_INIT = 16,        // waiting for initialisation (set by the host; cleared by the init launch)
  ST_BARRIER = 32,     // a grid-team barrier gave up waiting (bounded spin)
};

// One threshold crossing of a cell's spike compartment, logged on the device
// at the end of an interval: the interval's end time and the pool cell.
struct SpikeRec {
  double t;
  int cell;
  int pad;
};

// Controller state of one RKC system (h_others / h_work / h_bool of
// solve_rkc.cu, plus the driver's static sum_dt and counters).
struct Ctl {
  double absh, sprad, naccpt, errold, hold, lt, tend, gt, gt_old, idid, mmax, hw0, hw1;
  double sum_dt, integ, hmin, tol;
  double cbrt_errold;  // errold^(1/3), carried from the last accepted step
  int map[5];          // logical {y, yn, fn, vtemp1, vtemp2} -> physical buffer
  int newspc, jacatt, last, status;
  int iv_left;         // intervals this system may still advance (-1: no limit)
  long long n_steps, n_rej, n_stage, n_rho, n_rho_iter, n_ion;
};

// Where a system's group tables begin (PoolView::grp_*).
struct GroupTab {
  int chunk0, col, slot, sptr, send, rptr, rslot;
};

// Everything a kernel needs for one pool (passed by value).
template <typename R>
struct PoolView {
  int type, nsys;
  long stride;                        // pool compartment count (SoA stride)
  // per system
  const int *sys_off, *sys_nc, *sys_ncell, *sys_ncomp, *sys_tmpl, *sys_csr, *sys_cell0;
  const int *sys_gap0, *sys_ngap;
  const long *sys_ws;                 // workspace offset (doubles)
  Ctl *ctl;
  double *ws;
  // per compartment
  double *ede, *vnew, *v, *ca, *ca2, *rev, *ca_old, *iext;
  const double *shell, *area;
  const uint8_t *ctype, *flags;       // compartment type; bit0 = PKJ fixed Nernst
  R *ion;
  const R *cond;
  // templates
  const int *t_row0, *t_nz0, *t_cm0;  // per template offsets
  const int *t_row, *t_col;
  const double *t_g, *t_invcm;
  const double *t_gc, *t_Gc;          // mixed precision: g / Cm per entry, their row sums (like t_invcm)
  // system CSRs (multi-cell systems with linear gap junctions)
  const int *s_row0, *s_nz0, *s_cm0;
  const int *s_row, *s_col;
  const double *s_g, *s_invcm;
  const double *s_gc, *s_Gc;
  // IO nonlinear gap junctions: per system edge list (post compartment, pre or -1)
  const int *gap_pre, *gap_post;
  const double *gap_g;
  // per cell (pool cell index)
  const int *stim_comp;
  const double *stim_amp, *stim_t0, *stim_t1;
  int stim_on;
  // stage coefficients, per m: [h*mus factor of stage 1, then (mu, nu, 1-mu-nu, mus, ajm1) per stage]
  const double *coef;
  const long *coef_off;
  int coef_mmax;
  NaPar na[9];
  // outputs
  double *soma_out;                   // [interval][pool cell][rec_w] or null
  const int *cell_soma;               // per pool cell: first recorded compartment (pool index)
  int rec_w;                          // compartments recorded per cell
  int ncell_pool;
  // device raster: per pool cell the spike compartment and its value at the
  // previous interval's end; an upward crossing of spk_th appends a SpikeRec
  // (entries past spk_cap are counted, not written)
  const int *cell_spk;
  double *spk_prev;
  SpikeRec *spk_log;
  int *spk_count;
  int spk_cap;
  double spk_th;
  int lanes;                          // granule pools: lanes of each warp in use, one system a lane or (TEAM_LANE4) per four
  int per_warp;                       // granule pools: systems a warp takes (lanes, or lanes / 4)
  int ws_in_smem;                     // stage the workspace in shared memory
  long ws_tile_doubles;               // shared-memory workspace per team
  // chemical synapses onto this pool (network mode; syn_mode 0 = none)
  int syn_mode;                       // SYN_AT_ION, SYN_BUFFERED or SYN_BUFFERED_DECAY
  const int *syn_row;                 // [stride + 1] CSR over post compartments
  const int *syn_idx;                 // synapse ids, per compartment in (kind, id) order
  const double *syn_val;              // per synapse: conductance value (engine-wide table)
  const double *syn_e;                // per synapse: reversal potential
  double *syn_buf;                    // [stride] synaptic current taken at interval start
  // group teams (group_sys.cuh): one system over a CTA, a cluster, or every
  // CTA of a cooperative launch
  int grid_bw;                        // threads of a CTA, elements of a chunk
  int grid_maxdeg;                    // the operator's longest row
  int grp_ctas;                       // CTAs of a group
  int grp_ld;                         // elements of the fullest CTA
  int grp_recv_max;                   // most values a CTA receives
  int grp_nslots;                     // grid: values that more than their own CTA reads
  const GroupTab *grp_tab;            // per system: where its tables begin
  const int *grp_chunk0;              // [ctas + 1] first chunk of each CTA
  const int *grp_col;                 // per operator entry: the column's place in the row's CTA (own places, then received)
  const int *grp_slot;                // grid, [nc]: the element's publishing slot, or -1
  const int *grp_sptr, *grp_send;     // cluster, per thread: its hand-overs (row of the thread, reading CTA, its slot)
  const int *grp_rptr, *grp_rslot;    // per CTA: the values it receives (grid: their slots)
  const int *grp_gap;                 // olive, per gap edge: the sending dendrite's place, or -1
  unsigned long long *grp_halo;       // grid: [2][nslots][2] published values
  unsigned long long *grp_red;        // grid: [2][GRID_MAX_BLOCKS][2] published chunk sums
  int *grp_abort;                     // a wait gave up
  // persistent launch: systems of one (1) or several (2) elements a thread,
  // vectors in registers; 0: the teams with their vectors in memory
  int grp_fast;
  int tiles;                          // teams of a CTA that take systems
  long grp_stride;                    // doubles of shared memory a team
  int ivc;                            // intervals a team goes on with one system while others wait
  int *grp_line;                      // [2] counters, [nsys] next intervals, [16 nsys] the line (group_sys.cuh, line_take)
  const int *grp_order;               // the line's first systems, those with work; bit 30: taken to its end without a turn
  int grp_first;                      // their number
  int in_order;                       // warps take whole systems in that order (else all of the pool's, 0, 1, 2, ...)
};

// How a pool takes its synaptic current (solve_rkc.cu): granule cells add
// every synapse's g (V_y - E) to b at each ion update (add_mfgr_val,
// add_gogr_val, 1100-1120); Golgi cells take the sum at the start of the
// interval and add it at each ion update (add_grgo_val_new +
// go_update_matrix_new, 1199-1200, 1180); Purkinje cells likewise, scaled by
// exp(-sum_dt / 0.6) (add_grpkj_val_new + pkj_update_matrix_new, 1266-1269,
// 1247-1250).
enum SynMode { SYN_NONE = 0, SYN_AT_ION = 1, SYN_BUFFERED = 2, SYN_BUFFERED_DECAY = 3 };

// Synapse kinds of the reference's RKC network path (syn.cu) and their
// per-synapse state: MF->GrC (AMPA, NMDA), GrC->GoC (AMPA, NMDA1, NMDA2),
// GoC->GrC (GABA_A, GABA_B), GrC->PC (AMPA).
enum SynKind { SYN_MFGR = 0, SYN_GRGO = 1, SYN_GOGR = 2, SYN_GRPKJ = 3, SYN_KINDS = 4 };

// The engine-wide synapse table for the per-interval update kernel.
struct SynView {
  int n;
  const int *kind, *grp;
  const int *pre_type;                // pool of the presynaptic compartment (-1: Poisson input)
  const long *pre_gi;                 // presynaptic compartment, pool index
  const double *w;
  double *s0, *s1, *s2, *val, *old_v;
  const double *pre_v[NTYPES];        // elem v of every pool
  unsigned long long *ring;           // per synapse: the last 64 intervals' events, newest in bit 0 (or null)
  const unsigned char *delay;         // per synapse: intervals between an event and its effect
  const double *grp_rate;             // per group: base rate, stimulus rate [Hz], window t0, t1 [ms]
  const unsigned long long *grp_seed;
  double decay[8];                    // exp(-RKC_DT / tau) per state, in SynKind order
};

int launch_syn_update(const SynView &S, void *stream, double t, long long interval);

// Team shapes the kernels are instantiated for: one thread (tiny cells, 32
// systems per warp, blocks of MEGA_BLOCK threads with interleaved shared
// workspaces), 4 or 32 lanes per system, or a whole block per system.
// TEAM_LANE4: four lanes per system for pools whose systems all have exactly
// 4 compartments, one compartment a lane (quad_sys.cuh).
// TEAM_CLUSTER8 / TEAM_CLUSTER16: one system per cluster of 8 / 16 CTAs
// (very large systems; 16 is a non-portable cluster size, used where the
// device can co-schedule it).
// Group teams (group_sys.cuh), at most one, two or eight elements a thread:
// TEAM_CTA1..: one system per CTA of exactly its threads; TEAM_CLU1..: per
// cluster of P.grp_ctas CTAs; TEAM_GRID1..: one system over every CTA of a
// cooperative launch (a system that is alone in its engine).
enum TeamKind {
  TEAM_THREAD = 1, TEAM_LANE4 = 2, TEAM_TILE4 = 4, TEAM_WARP = 32, TEAM_BLOCK = 0,
  TEAM_CLUSTER8 = 108, TEAM_CLUSTER16 = 116, TEAM_CTA1 = 201, TEAM_CTA2 = 202,
  TEAM_CLU1 = 301, TEAM_CLU2 = 302, TEAM_CLU4 = 304,
  TEAM_GRID1 = 401, TEAM_GRID2 = 402, TEAM_GRID8 = 408
};
// systems a warp takes when `lanes` of its lanes are in use, four lanes each
constexpr int quads_per_warp(int lanes) { return lanes < 8 ? 1 : lanes / 4; }
constexpr int team_cluster_size(int team) {
  return team == TEAM_CLUSTER8 ? 8 : team == TEAM_CLUSTER16 ? 16 : 0;
}

// All pools in one persistent launch: CTA b < role_end[0] integrates granule
// systems (one per lane or per four, on the CTA's first warps), then Golgi,
// Purkinje and olive ones.  Granule lanes take systems from an atomic queue,
// quads with more systems than places then from the line; the other roles'
// register teams take pieces of systems from the line (group_sys.cuh), and
// where those do not hold a role's systems (grp_fast 0), and at initialisation,
// warps (Golgi) and whole blocks take whole systems from the queue.
template <typename R>
struct MegaView {
  PoolView<R> pool[NTYPES];
  int role_end[NTYPES];
  int lane_warps, lane_extra;  // granule CTA b runs lane_warps (+1 if b < lane_extra) warps
  int gr_nc4;                 // every granule system has 4 compartments
  int *queue;                 // [NTYPES] next-system counters, zeroed per launch
  unsigned long long *t_start; // [grid] globaltimer at each CTA's start
  unsigned long long *t_end;   // [grid] globaltimer at each CTA's finish
};

constexpr int MEGA_BLOCK = 256;
// Cluster teams: CTAs of CLUSTER_BLOCK threads; at most CLUSTER_MAX_ROWS rows
// of CLUSTER_BLOCK elements per CTA and vector (the workspace of WS_VECS
// vectors fits 200 KB of shared memory), followed by the reduction area:
// block sums (double-buffered), warp partials, result.
constexpr int CLUSTER_BLOCK = 256;
constexpr int CLUSTER_MAX_ROWS = 14;
constexpr int CLUSTER_RED_DOUBLES = 2 * CLUSTER_MAX_ROWS + 8 * CLUSTER_MAX_ROWS + 2;
constexpr int LANE_MAX_NC = 8;   // largest system integrated by a single lane
constexpr bool team_is_grid(int team) { return team >= TEAM_GRID1; }
constexpr bool team_is_clu(int team) { return team > 300 && team < 400; }
constexpr bool team_is_group(int team) { return team > 200; }
// Group teams: CTAs of grid_bw threads (at most GRID_BLOCK; a power of two
// where a group has several CTAs); the elements go to the CTAs in runs of
// whole chunks of grid_bw, at most GRID_MAX_ROWS chunks a CTA and
// GRID_MAX_BLOCKS in all.
constexpr int GRID_BLOCK = 256;
constexpr int GRID_MAX_BLOCKS = 256;
constexpr int GRID_MAX_ROWS = 8;
// In the persistent launch a team of a CTA's warps integrates systems of up to
// MEGA_BLOCK compartments, one a thread, or, as the whole CTA, of up to
// GRP_CTA_ROWS a thread; shared memory holds the coefficients of stage counts
// up to GRP_COEF_M.
constexpr int GRP_CTA_ROWS = 7, GRP_COEF_M = 96;
constexpr int GRP_COEF_M_DOUBLES = (5 * (GRP_COEF_M - 1) + 1) & ~1;
constexpr int LINE_PIECES = 16;   // most pieces of a system's launch
constexpr size_t GRID_SMEM_MAX = 200 * 1024;   // shared memory of a CTA
// bytes of it: two stage buffers, per element its row (pairs of conductances
// and columns, 1/Cm or the row sum), and in a cluster of `ctas` the slots of
// hand-overs and sums.  Columns are byte offsets of 16 bits: at most
// GRID_PLACES places in a stage buffer.
constexpr long GRID_PLACES = 8191;
constexpr size_t grid_smem(long ld, long recv, long maxdeg, int ctas) {
  return 16 * (size_t)(ld + recv + 2) + (size_t)ld * (8 + 20 * (size_t)((maxdeg + 1) / 2)) +
         (ctas > 0 ? 16 + 32 * (size_t)recv + 32 * (size_t)GRID_MAX_ROWS * ctas : 0);
}

template <typename R>
int launch_mega(const MegaView<R> &M, int grid, size_t smem, void *stream, double t0, int n_iv, int iv0,
                int init);
template <typename R>
int prepare_mega_kernel(size_t smem, int *blocks_per_sm);

// The kernel of a team for one cell type and precision (kernels_pool.cu).
template <int CT, typename R>
const void *pool_kernel(int team);

// Launch the advance / initialise kernel of one pool (kernels.cu).
template <typename R>
int launch_pool(int type, const PoolView<R> &P, int team, int grid, int block, size_t smem,
                void *stream, double t0, int n_iv, int iv0, int init);
template <typename R>
int prepare_pool_kernel(int type, int team, size_t smem);
// How many clusters of a cluster team's kernel the device can run at once
// with this shared memory (0: the shape does not fit).
template <typename R>
int cluster_capacity(int type, int team, size_t smem);
// The same of a cluster group team's kernel, with `ctas` CTAs of `block` threads.
template <typename R>
int group_capacity(int type, int team, int ctas, int block, size_t smem);
// CTAs of the grid team's cooperative launch (0: the device cannot launch it).
template <typename R>
int grid_capacity(int type);

}  // namespace gbrkc
