#include <type_traits>
// k_mega: one persistent launch for all pools, every CTA a role taking
// systems from its role's queue or pieces of them from its line
// (group_sys.cuh); and the launches of it and of the per-pool kernels
// (kernels_pool.cu).
//
// Built with -fmad=false (see integrator.cuh).  R selects FP64 or FP32
// gating; the instantiations live in kernels_fp64.cu / kernels_fp32.cu.
#include <algorithm>
#include <cuda_runtime.h>

#include "integrator.cuh"
#include "group_sys.cuh"
#include "quad_sys.cuh"

namespace gbrkc {

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// a role of tile teams: every tile repeatedly takes the next system
template <int CT, typename R, int TS>
__device__ __forceinline__ void role_tiles(const PoolView<R> &P, int *q, double *smem, double t0, int n_iv,
                                           int iv0, int init) {
  const int tile = threadIdx.x / TS;
  TileTeam<TS> tm;
  tm.r = threadIdx.x % TS;
  tm.mask = (TS == 32) ? 0xffffffffu : (((1u << TS) - 1u) << ((threadIdx.x & 31) / TS * TS));
  double *my = smem + (long)tile * P.ws_tile_doubles;
  for (;;) {
    int s = 0;
    if (tm.r == 0) {
      s = atomicAdd(q, 1);
      if (P.in_order) s = s < P.grp_first ? P.grp_order[s] & ((1 << 30) - 1) : P.nsys;
    }
    s = __shfl_sync(tm.mask, s, 0, TS);
    if (s >= P.nsys) break;
    run_system<CT, R, TileTeam<TS>>(P, tm, s, my, t0, n_iv, iv0, init != 0);
  }
}

// a role of whole blocks: the block takes the next system
template <int CT, typename R>
__device__ __forceinline__ void role_block(const PoolView<R> &P, int *q, double *smem, double t0, int n_iv,
                                           int iv0, int init) {
  __shared__ int s_next;
  BlockTeam tm;
  for (;;) {
    if (threadIdx.x == 0) s_next = atomicAdd(q, 1);
    __syncthreads();
    const int s = s_next;
    __syncthreads();
    if (s >= P.nsys) break;
    run_system<CT, R, BlockTeam>(P, tm, s, smem, t0, n_iv, iv0, init != 0);
    __syncthreads();
  }
}

// A role of teams with their system's vectors in registers (group_sys.cuh), at
// most K elements a thread: P.tiles teams of P.grid_bw threads a CTA.  A
// Golgi cell takes five warps: alone on its SM each issues an FP64 instruction
// in 95 cycles (five at the SM's 19), so that the cells whose step size is at
// its floor (up to 1024 attempts a ms where the median cell takes 115), whose
// serial chains set the launch's time, run five times as fast as on a warp of
// eight systems' warps;
// and the warps of a team run the same instructions at the same time, where
// eight systems' warps each fetched their own (40% of their cycles).
template <int CT, typename R, int K>
__device__ __forceinline__ void role_teams(const PoolView<R> &P, double *smem, double t0, int n_iv, int iv0) {
  __shared__ int s_next[MEGA_BLOCK / 32], s_at[MEGA_BLOCK / 32];
  __shared__ double s_wp[K == 1 ? MEGA_BLOCK / 32 : K * MEGA_BLOCK / 32], s_res[4 * MEGA_BLOCK / 32];
  const int bw = P.grid_bw, team = (int)threadIdx.x / bw, first = team * bw;
  if (team >= P.tiles) return;
  double *my = smem + (long)team * P.grp_stride;
  GroupSys<CT, R, K, GRP_CTA> S(P, my + GRP_COEF_M_DOUBLES, s_wp + first / 32, s_res + 4 * team, my, GRP_COEF_M, nullptr,
                                first, bw, 1 + team, 0, 1);
  int s = -1, k = 0;
  bool hold = false;
  for (;;) {
    if (S.t == 0) {
      line_next(P, s, k, hold);
      s_next[team] = s;
      s_at[team] = k;
    }
    S.sync();
    s = s_next[team];
    k = s_at[team];
    if (s < 0) break;
    const int n = min(P.ivc, n_iv - k);
    S.template run<false>(s, t0, k, n, iv0, false);
    S.sync();
    k += n;
    // (thread 0 takes and leaves systems, and wrote this one's Ctl)
    if (k >= n_iv || (S.t == 0 && !system_selected(P.ctl[s], false, 1))) s = -1;
    else if (S.t == 0) __threadfence();
  }
}

template <typename R>
__global__ void __launch_bounds__(MEGA_BLOCK, 1) k_mega(const __grid_constant__ MegaView<R> M, double t0,
                                                         int n_iv, int iv0, int init) {
  extern __shared__ __align__(16) double smem[];
  if (threadIdx.x == 0) M.t_start[blockIdx.x] = global_ns();
  int role = 0;
  while (role < NTYPES - 1 && (int)blockIdx.x >= M.role_end[role]) role++;
  switch (role) {
    case GR:
      // granule systems on the CTA's first warps
      if ((int)(threadIdx.x >> 5) < M.lane_warps + ((int)blockIdx.x < M.lane_extra ? 1 : 0)) {
        if (M.gr_nc4 && !init && n_iv > 0)
          run_quads<GR, R>(M.pool[GR], M.queue + GR, 0, 0, M.pool[GR].per_warp, t0, n_iv, iv0);
        else if (M.gr_nc4)
          run_lanes<GR, R, MEGA_BLOCK, 4>(M.pool[GR], M.queue + GR, 0, 0, smem, t0, n_iv, iv0, init != 0);
        else
          run_lanes<GR, R, MEGA_BLOCK>(M.pool[GR], M.queue + GR, 0, 0, smem, t0, n_iv, iv0, init != 0);
      }
      break;
    // (initialisation, and systems of more compartments than a team's
    // registers take, go through the teams with their vectors in memory)
    case GO:
      if (M.pool[GO].grp_fast && !init)
        role_teams<GO, R, 1>(M.pool[GO], smem, t0, n_iv, iv0);
      else
        role_tiles<GO, R, TEAM_WARP>(M.pool[GO], M.queue + GO, smem, t0, n_iv, iv0, init);
      break;
    case PKJ:
      if (M.pool[PKJ].grp_fast && !init)
        role_teams<PKJ, R, GRP_CTA_ROWS>(M.pool[PKJ], smem, t0, n_iv, iv0);
      else
        role_block<PKJ, R>(M.pool[PKJ], M.queue + PKJ, smem, t0, n_iv, iv0, init);
      break;
    default:
      if (M.pool[IO].grp_fast == 1 && !init)
        role_teams<IO, R, 1>(M.pool[IO], smem, t0, n_iv, iv0);
      else if (M.pool[IO].grp_fast && !init)
        role_teams<IO, R, GRP_CTA_ROWS>(M.pool[IO], smem, t0, n_iv, iv0);
      else
        role_block<IO, R>(M.pool[IO], M.queue + IO, smem, t0, n_iv, iv0, init);
      break;
  }
  __syncthreads();
  if (threadIdx.x == 0) M.t_end[blockIdx.x] = global_ns();
}

// The dynamic shared-memory limit is a per-kernel attribute shared by every
// engine in the process: only ever raise it, so that a later engine with
// smaller needs cannot break an earlier one's launches.  Unless it is set, a
// launch may have 48 KB in all, the kernel's own variables (4.4 KB in the group
// teams) among them.
static cudaError_t raise_smem_limit(const void *k, size_t smem) {
  cudaFuncAttributes a;
  cudaError_t e = cudaFuncGetAttributes(&a, k);
  if (e != cudaSuccess) return e;
  const size_t limit = (size_t)a.maxDynamicSharedSizeBytes, unset = 48 * 1024;
  if (smem <= limit && (limit > unset || smem + a.sharedSizeBytes <= unset)) return cudaSuccess;
  return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)std::max(smem, limit));
}

template <typename R>
int prepare_mega_kernel(size_t smem, int *blocks_per_sm) {
  const void *k = (const void *)k_mega<R>;
  cudaError_t e = raise_smem_limit(k, smem);
  if (e != cudaSuccess) return (int)e;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, k, MEGA_BLOCK, smem);
  return (int)e;
}

template <typename R>
int launch_mega(const MegaView<R> &M, int grid, size_t smem, void *stream, double t0, int n_iv, int iv0,
                int init) {
  MegaView<R> Mc = M;
  void *args[] = {(void *)&Mc, (void *)&t0, (void *)&n_iv, (void *)&iv0, (void *)&init};
  cudaError_t e = cudaLaunchKernel((const void *)k_mega<R>, dim3(grid), dim3(MEGA_BLOCK), args, smem,
                                   (cudaStream_t)stream);
  return (int)e;
}

template <typename R>
static const void *kernel_ptr(int type, int team) {
  switch (type) {
    case GR: return pool_kernel<GR, R>(team);
    case GO: return pool_kernel<GO, R>(team);
    case PKJ: return pool_kernel<PKJ, R>(team);
    default: return pool_kernel<IO, R>(team);
  }
}

template <typename R>
int prepare_pool_kernel(int type, int team, size_t smem) {
  const void *k = kernel_ptr<R>(type, team);
  cudaError_t e = cudaSuccess;
  // (no kernel has 16 KB of its own; asking loads it)
  if (smem > 32 * 1024) e = raise_smem_limit(k, smem);
  if (e != cudaSuccess) return (int)e;
  if (team_cluster_size(team) > 8 || team_is_clu(team)) {
    e = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return (int)e;
  }
  return 0;
}

static cudaLaunchConfig_t cluster_config(int size, int grid, int block, size_t smem, cudaStream_t stream,
                                         cudaLaunchAttribute *attr) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = size;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

// CTAs of the grid team's kernel the device co-schedules (cooperative
// launch: every CTA resident at once), 0 when it cannot launch cooperatively.
template <typename R>
int grid_capacity(int type) {
  int dev = 0, coop = 0, sms = 0, bps = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (!coop) return 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, kernel_ptr<R>(type, TEAM_GRID8), GRID_BLOCK, 0) !=
      cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return sms * std::min(bps, 1);
}

template <typename R>
int cluster_capacity(int type, int team, size_t smem) {
  if (prepare_pool_kernel<R>(type, team, smem) != 0) {
    cudaGetLastError();
    return 0;
  }
  const int size = team_cluster_size(team);
  cudaLaunchAttribute attr[1];
  const cudaLaunchConfig_t cfg = cluster_config(size, size, CLUSTER_BLOCK, smem, 0, attr);
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kernel_ptr<R>(type, team), &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

template <typename R>
int group_capacity(int type, int team, int ctas, int block, size_t smem) {
  if (prepare_pool_kernel<R>(type, team, smem) != 0) {
    cudaGetLastError();
    return 0;
  }
  cudaLaunchAttribute attr[1];
  const cudaLaunchConfig_t cfg = cluster_config(ctas, ctas, block, smem, 0, attr);
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kernel_ptr<R>(type, team), &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

template <typename R>
int launch_pool(int type, const PoolView<R> &P, int team, int grid, int block, size_t smem, void *stream,
                double t0, int n_iv, int iv0, int init) {
  const void *k = kernel_ptr<R>(type, team);
  PoolView<R> Pc = P;
  void *args[] = {(void *)&Pc, (void *)&t0, (void *)&n_iv, (void *)&iv0, (void *)&init};
  if (team_is_grid(team)) {
    if (block < 32 || block > GRID_BLOCK || (block & (block - 1)) != 0 || block != P.grid_bw)
      return (int)cudaErrorInvalidConfiguration;
    return (int)cudaLaunchCooperativeKernel(k, dim3(grid), dim3(block), args, smem, (cudaStream_t)stream);
  }
  if (team_cluster_size(team) > 0) {
    if (block != CLUSTER_BLOCK || grid % team_cluster_size(team) != 0) return (int)cudaErrorInvalidConfiguration;
    cudaLaunchAttribute attr[1];
    const cudaLaunchConfig_t cfg =
        cluster_config(team_cluster_size(team), grid, block, smem, (cudaStream_t)stream, attr);
    return (int)cudaLaunchKernelExC(&cfg, k, args);
  }
  if (team_is_clu(team)) {
    if (block != P.grid_bw || P.grp_ctas < 1 || grid % P.grp_ctas != 0) return (int)cudaErrorInvalidConfiguration;
    cudaLaunchAttribute attr[1];
    const cudaLaunchConfig_t cfg = cluster_config(P.grp_ctas, grid, block, smem, (cudaStream_t)stream, attr);
    return (int)cudaLaunchKernelExC(&cfg, k, args);
  }
  cudaError_t e = cudaLaunchKernel(k, dim3(grid), dim3(block), args, smem, (cudaStream_t)stream);
  return (int)e;
}

}  // namespace gbrkc
