// sweep_batch.cu -- many grids swept in one launch per kind of node (k_sweep_batch); see
// sweep_node.cuh for the node bodies.
#include <cuda_runtime.h>

#include "sweep_node.cuh"

namespace mdz {

// ---------------------------------------------------------------------------------
// many grids in one launch: the node range of every grid is cut into tiles of
// kBatchTile nodes, so a CTA's tile lies in one grid; the grid's arguments are read
// from global memory (uniform over the CTA, served by L1)
// ---------------------------------------------------------------------------------
__device__ __forceinline__ int batch_grid_of(const long long *tile_start, int n, long long tile) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (__ldg(&tile_start[mid]) <= tile) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// One kernel per kind of node, as for a single grid (and with the same node body, so a
// grid swept here gives the single-grid results to the bit): the centroid tiles of every
// grid (NODES 1), then the vertex tiles (NODES 2).  A tile of kBatchTile nodes is one CTA
// and lies in one grid, so the phase loop is uniform over the CTA and the learned warm
// start (WARM) is evaluated per warp as in k_sweep_warm.  PERTURB: the strain rates are
// multiplied by the sweep's perturbation factors as they are loaded, in place (the
// captured multi-sweep graph), instead of by a separate pass over them.
// 7 CTAs per SM (72 registers), as a large single grid's kernels: 16 grids of 65-513 cells a
// side, 5 captured sweeps, took 5.41, 5.18, 5.04 and 5.25 ms at 5, 6, 7 and 8.
template <bool ANISO, int NODES, bool WARM, bool PERTURB>
__global__ void __launch_bounds__(kBatchTile, WARM ? 6 : 7) k_sweep_batch(const __grid_constant__ BatchArgs B,
                                                             const __grid_constant__ BatchSweepArgs X) {
  extern __shared__ __align__(16) unsigned char smem_batch[];
  MlpWarpShared &S = *reinterpret_cast<MlpWarpShared *>(smem_batch);
  if (WARM) mlp_warp_load(S, X.mlp);
  Acc acc = {0, 0, 0, 0, 0};
  const long long *ts = NODES == 1 ? B.tile_start_n : B.tile_start_s;
  const long long tiles = NODES == 1 ? B.tiles_n : B.tiles_s;
  for (long long t = blockIdx.x; t < tiles; t += gridDim.x) {  // uniform over the CTA
    const int g = batch_grid_of(ts, B.n, t);
    const SweepArgs &A = B.grids[g];
    const long long j = (t - __ldg(&ts[g])) * kBatchTile + threadIdx.x;
    const bool valid = j < (NODES == 1 ? A.M.Nc : A.M.Nv);
    const long long i = NODES == 1 ? j : A.M.Nc + j;
    PerturbKey pk;
    if (PERTURB) { pk.key = perturb_key(X.seed, X.sweep, g); pk.amp = X.amp; }
    if (WARM) warm_node<ANISO, NODES>(A, S, X.mlp, valid, i, acc, PERTURB ? &pk : nullptr);
    else if (valid) sweep_node<ANISO, NODES>(A, i, acc, PERTURB ? &pk : nullptr);
  }
  flush_acc(B.stats, acc);
}

template <bool ANISO, int NODES, bool WARM, bool PERTURB>
static cudaError_t launch_batch_t(const BatchArgs &b, const BatchSweepArgs &x, cudaStream_t s, long long grid) {
  auto fn = k_sweep_batch<ANISO, NODES, WARM, PERTURB>;
  const size_t smem = WARM ? sizeof(MlpWarpShared) : 0;
  if (WARM) cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  fn<<<(unsigned)grid, kBatchTile, smem, s>>>(b, x);
  return cudaGetLastError();
}

template <bool ANISO, int NODES>
static cudaError_t launch_batch_kind(const BatchArgs &b, const BatchSweepArgs &x, cudaStream_t s, long long grid) {
  const bool pert = x.amp != 0.0;
  if (x.warm) return pert ? launch_batch_t<ANISO, NODES, true, true>(b, x, s, grid)
                          : launch_batch_t<ANISO, NODES, true, false>(b, x, s, grid);
  return pert ? launch_batch_t<ANISO, NODES, false, true>(b, x, s, grid)
              : launch_batch_t<ANISO, NODES, false, false>(b, x, s, grid);
}

cudaError_t launch_sweep_batch(const BatchArgs &b, const BatchSweepArgs &x, bool aniso, cudaStream_t s, int grid) {
  // one CTA per tile, up to `grid`, per kind
  const long long gn = b.tiles_n < grid ? b.tiles_n : grid, gs = b.tiles_s < grid ? b.tiles_s : grid;
  cudaError_t e = cudaSuccess;
  if (gn > 0) e = aniso ? launch_batch_kind<true, 1>(b, x, s, gn) : launch_batch_kind<false, 1>(b, x, s, gn);
  if (e != cudaSuccess) return e;
  if (gs > 0) e = aniso ? launch_batch_kind<true, 2>(b, x, s, gs) : launch_batch_kind<false, 2>(b, x, s, gs);
  return e;
}

}  // namespace mdz
