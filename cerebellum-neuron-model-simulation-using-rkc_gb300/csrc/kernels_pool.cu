// The per-pool advance kernels of one cell type and precision: one launch
// advances every system of the pool by n_iv output intervals (or initialises
// them), entirely on the device.  Granule cells take a lane or four each,
// other small systems teams of 4 or 32 lanes, larger ones a whole block, a
// cluster, or (alone in their engine) every SM.
//
// Compiled once per cell type and precision (GBRKC_CT, GBRKC_REAL), with
// -fmad=false (see integrator.cuh).
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "group_sys.cuh"
#include "quad_sys.cuh"

namespace gbrkc {

template <int CT, typename R, int TS>
__global__ void __launch_bounds__(256, 1) k_advance(const __grid_constant__ PoolView<R> P, double t0, int n_iv,
                                                 int iv0, int init) {
  extern __shared__ __align__(16) double smem[];
  if (TS == TEAM_THREAD || TS == TEAM_LANE4) {
    // the first `per` systems of warp w of block b start at system
    // per (w * grid + b): the first warps of every block are filled before
    // any block's later warps
    const bool quads = TS == TEAM_LANE4 && !init && n_iv > 0;
    const int per = quads ? P.per_warp : P.lanes, lane = (int)threadIdx.x & 31;
    const int first = (((int)threadIdx.x >> 5) * (int)gridDim.x + (int)blockIdx.x) * per + (quads ? lane >> 2 : lane);
    const int stride = (int)gridDim.x * (MEGA_BLOCK / 32) * per;
    if constexpr (TS == TEAM_LANE4) {
      if (quads)
        run_quads<CT, R>(P, nullptr, first, stride, per, t0, n_iv, iv0);
      else
        run_lanes<CT, R, MEGA_BLOCK, 4>(P, nullptr, first, stride, smem, t0, n_iv, iv0, init != 0);
    } else {
      run_lanes<CT, R, MEGA_BLOCK>(P, nullptr, first, stride, smem, t0, n_iv, iv0, init != 0);
    }
  } else if (TS == TEAM_BLOCK) {
    BlockTeam tm;
    for (int s = blockIdx.x; s < P.nsys; s += gridDim.x) {
      run_system<CT, R, BlockTeam>(P, tm, s, smem, t0, n_iv, iv0, init != 0);
      __syncthreads();
    }
  } else {
    constexpr int T = TS > 0 ? TS : 1;
    const int tiles = blockDim.x / T, tile = threadIdx.x / T;
    TileTeam<TS> tm;
    tm.r = threadIdx.x % T;
    tm.mask = (T == 32) ? 0xffffffffu : (((1u << T) - 1u) << ((threadIdx.x & 31) / T * T));
    double *my = smem + (long)tile * P.ws_tile_doubles;
    for (int s = blockIdx.x * tiles + tile; s < P.nsys; s += gridDim.x * tiles)
      run_system<CT, R, TileTeam<TS>>(P, tm, s, my, t0, n_iv, iv0, init != 0);
  }
}

// One large system per thread-block cluster of C CTAs (ClusterTeam): the
// cluster takes systems cid, cid + nclusters, ...
template <int CT, typename R, int C>
__global__ void __launch_bounds__(CLUSTER_BLOCK, 1) k_advance_cluster(const __grid_constant__ PoolView<R> P, double t0,
                                                                       int n_iv, int iv0, int init) {
  namespace cg = cooperative_groups;
  extern __shared__ __align__(16) double smem[];
  __shared__ double *s_bases[C];
  cg::cluster_group cl = cg::this_cluster();
  if (threadIdx.x < C) s_bases[threadIdx.x] = cl.map_shared_rank(smem, (int)threadIdx.x);
  cl.sync();
  const ClusterTeam<C> tm{(int)cl.block_rank(), s_bases, P.ws_tile_doubles};
  const int ncl = gridDim.x / C, cid = blockIdx.x / C;
  for (int s = cid; s < P.nsys; s += ncl) run_system<CT, R, ClusterTeam<C>>(P, tm, s, smem, t0, n_iv, iv0, init != 0);
  // no CTA leaves while a peer may still reach its shared memory
  cl.sync();
}

// Group teams (group_sys.cuh), at most K elements a thread: one system per
// CTA, per cluster of P.grp_ctas CTAs, or over the whole (cooperative) grid;
// the groups take systems from the line (group_sys.cuh).
template <int CT, typename R, int K, int COMM>
__global__ void __launch_bounds__(GRID_BLOCK, 1) k_advance_group(const __grid_constant__ PoolView<R> P, double t0,
                                                                  int n_iv, int iv0, int init) {
  extern __shared__ __align__(16) double smem[];
  __shared__ double s_wp[GRID_MAX_ROWS * 8];
  __shared__ double s_res[4], s_coef[5 * (GRP_COEF_M - 1)];
  __shared__ int s_abort[2];
  const int G = COMM == GRP_CTA ? 1 : P.grp_ctas, groups = (int)gridDim.x / G, group = (int)blockIdx.x / G;
  GroupSys<CT, R, K, COMM> S(P, smem, s_wp, s_res, s_coef, GRP_COEF_M, s_abort, 0, P.grid_bw, 0,
                             (int)blockIdx.x - group * G, G);
  if (COMM == GRP_GRID || init) {
    for (int s = group; s < P.nsys; s += groups) S.run(s, t0, 0, n_iv, iv0, init != 0);
  } else {
    // the group's first CTA takes systems from the line
    __shared__ __align__(8) int s_item[2];
    int s = -1, k = 0;
    bool hold = false;
    for (;;) {
      if (S.cta == 0 && S.t == 0) {
        line_next(P, s, k, hold);
        s_item[0] = s;
        s_item[1] = k;
        if (COMM == GRP_CLUSTER)
          for (int c = 1; c < G; c++) {
            const unsigned a = cluster_map((unsigned)__cvta_generic_to_shared(s_item), c);
            asm volatile("st.relaxed.cluster.shared::cluster.v2.u32 [%0], {%1, %2};" ::"r"(a), "r"(s), "r"(k) : "memory");
          }
      }
      S.group_sync();
      // (a system's state may come from another SM)
      __threadfence();
      s = s_item[0];
      k = s_item[1];
      if (s < 0) break;
      const int n = min(P.ivc, n_iv - k);
      S.run(s, t0, k, n, iv0, false);
      S.group_sync();
      k += n;
      // (the group's first thread takes and leaves systems, and wrote this one's Ctl)
      if (k >= n_iv || (S.cta == 0 && S.t == 0 && !system_selected(P.ctl[s], false, 1))) s = -1;
      else if (S.cta == 0 && S.t == 0) __threadfence();
    }
  }
  S.leave();
}

template <int CT, typename R>
const void *pool_kernel(int team) {
  switch (team) {
    case TEAM_CTA1: return (const void *)k_advance_group<CT, R, 1, GRP_CTA>;
    case TEAM_CTA2: return (const void *)k_advance_group<CT, R, 2, GRP_CTA>;
    case TEAM_CLU1: return (const void *)k_advance_group<CT, R, 1, GRP_CLUSTER>;
    case TEAM_CLU2: return (const void *)k_advance_group<CT, R, 2, GRP_CLUSTER>;
    case TEAM_CLU4:
      // instantiated for Purkinje pools only (the others never have it)
      if constexpr (CT == PKJ) return (const void *)k_advance_group<CT, R, 4, GRP_CLUSTER>;
      return (const void *)k_advance_group<CT, R, 2, GRP_CLUSTER>;
    case TEAM_GRID1: return (const void *)k_advance_group<CT, R, 1, GRP_GRID>;
    case TEAM_GRID2: return (const void *)k_advance_group<CT, R, 2, GRP_GRID>;
    case TEAM_GRID8: return (const void *)k_advance_group<CT, R, GRID_MAX_ROWS, GRP_GRID>;
    case TEAM_CLUSTER8: return (const void *)k_advance_cluster<CT, R, 8>;
    case TEAM_CLUSTER16: return (const void *)k_advance_cluster<CT, R, 16>;
    case TEAM_LANE4:
      // instantiated for granule pools only (the others never have it)
      if constexpr (CT == GR) return (const void *)k_advance<CT, R, TEAM_LANE4>;
      return (const void *)k_advance<CT, R, TEAM_THREAD>;
    case TEAM_THREAD: return (const void *)k_advance<CT, R, TEAM_THREAD>;
    case TEAM_TILE4: return (const void *)k_advance<CT, R, TEAM_TILE4>;
    case TEAM_WARP: return (const void *)k_advance<CT, R, TEAM_WARP>;
    default: return (const void *)k_advance<CT, R, TEAM_BLOCK>;
  }
}

template const void *pool_kernel<GBRKC_CT, GBRKC_REAL>(int team);

}  // namespace gbrkc
