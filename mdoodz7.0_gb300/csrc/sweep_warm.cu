// sweep_warm.cu -- the sweeps with the learned warm start: k_sweep_warm (the network per
// warp) and k_sweep_tiles (the network as tcgen05 tiles, or the training-data dump); see
// rheo_kernels.cu for the plain sweeps and sweep_node.cuh for the node bodies.
#include <cuda_runtime.h>

#include "sweep_node.cuh"

namespace mdz {

// One node per lane, the warp's 32 nodes consecutive, so every lane of a warp runs the
// same number of node iterations and reaches the network at the same phase; lanes past
// the end or at inactive (node, phase) items feed zeros and discard the output.
template <bool ANISO, int NODES>
__global__ void __launch_bounds__(128, 4) k_sweep_warm(const __grid_constant__ SweepArgs A,
                                                    const __grid_constant__ MlpDevice W) {
  extern __shared__ __align__(16) unsigned char smem_warm[];
  MlpWarpShared &S = *reinterpret_cast<MlpWarpShared *>(smem_warm);
  mlp_warp_load(S, W);
  Acc acc = {0, 0, 0, 0, 0};
  const long long total = NODES == 1 ? A.M.Nc : A.M.Nv;
  const long long lo = NODES == 1 ? 0 : A.M.Nc;
  const long long stride = (long long)gridDim.x * blockDim.x;
  const int lane = threadIdx.x & 31;
  for (long long base = (long long)blockIdx.x * blockDim.x + (threadIdx.x & ~31); base < total; base += stride) {
    const long long j = base + lane;
    warm_node<ANISO, NODES>(A, S, W, j < total, lo + j, acc);
  }
  flush_acc(A.stats, acc);
}

// ---------------------------------------------------------------------------------
// tiled sweep with a block-wide stage per phase (learned warm start / data collection)
// ---------------------------------------------------------------------------------
// NODES 1 sweeps the centroids, NODES 2 the vertices (one launch each, with the node
// bodies of the plain sweep's two kernels).  A tile is one CTA's, its phase loop uniform over
// the CTA, so that a block-wide stage can sit between each phase's set-up and its local
// solve: the tcgen05 network's guess (MODE_WARM) or the dump of training pairs from the
// reference's own start (MODE_COLLECT).
template <bool ANISO, int MODE, int NODES>
__global__ void __launch_bounds__(128, 2) k_sweep_tiles(const __grid_constant__ SweepArgs A,
                                                     const __grid_constant__ WarmArgs W) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  MlpShared &S = *reinterpret_cast<MlpShared *>(smem_raw);
  uint32_t phase = 0;
  if (MODE == MODE_WARM) mlp_begin(S, W.mlp);
  Acc acc = {0, 0, 0, 0, 0};
  const long long total = A.M.Nc + A.M.Nv;
  const long long count = NODES == 1 ? A.M.Nc : A.M.Nv, base = NODES == 1 ? 0 : A.M.Nc;
  const long long ntiles = (count + kMlpTile - 1) / kMlpTile;
  const int nfeat = ANISO ? kFeatAniso : kFeatIso;
  for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {  // uniform over the CTA
    const long long j = tile * kMlpTile + threadIdx.x;
    const bool valid = j < count;
    const long long i = base + j;
    Node n;
    n.solid = false;
    n.centroid = NODES == 1;
    if (valid) node_prepare<ANISO, NODES>(A, i, n);
    double out[CO_COUNT];  // anisotropic
    IsoAcc q;              // isotropic
#pragma unroll
    for (int j = 0; j < CO_COUNT; j++) out[j] = 0.0;
    iso_acc_zero(q);
    int status = MDZ_OK;
    for (int p = 0; p < A.M.np; p++) {  // uniform over the CTA
      const double perc = (valid && n.solid) ? node_perc(A, n, p) : 0.0;
      const bool active = fp64_abs_gt_pos(perc, 1e-13);
      if (valid && n.solid && !active) node_iters(A, n, p, 0);
      IsoState st;
      PointOut o;
      float f[kMlpIn];
#pragma unroll
      for (int j = 0; j < kMlpIn; j++) f[j] = 0.0f;
      float s_start = ANISO ? 0.0f : 1.0f;  // the reference's own start
      if (active) {
        const bool exact = (MODE == MODE_COLLECT) || W.mlp.polish_iters == 0;  // the pairs' targets need eta_up
        if (ANISO) aniso_setup<FxMath>(A.M, A.ph[p], n.in, n.ctx, n.an, st, o, exact);
        else iso_setup<FxMath>(A.M, A.ph[p], n.in, n.ctx, st, o, exact);
        warm_features(A.M, n.in, n.ctx, st, ANISO, f);
      }
      if (MODE == MODE_WARM) {
        float x[kMlpIn];
#pragma unroll
        for (int j = 0; j < kMlpIn; j++) x[j] = (j < nfeat) ? (f[j] - W.mlp.x_shift[j]) * W.mlp.x_scale[j] : 0.0f;
        float y[2];
        mlp_forward(S, x, y, phase, W.mlp.poll_limit);
        if (active && !S.fault) {
          s_start = warm_start_point(y[0], W.mlp.z_scale, W.mlp.z_shift);
        }
      }
      if (!active) continue;
      double eta_conv = 0.0;
      const int polish = (MODE == MODE_WARM) ? W.mlp.polish_iters : 0;
      if constexpr (ANISO) {
        aniso_finish<FxMath>(A.M, A.ph[p], n.in, n.ctx, n.an, st, s_start, polish, o, &eta_conv);
        node_accumulate<ANISO>(A, n, p, perc, o, out, acc, status);
      } else {
        iso_sweep_item<NODES>(A, n, p, perc, st, s_start, polish, o, q, acc, status, &eta_conv);
      }
      if (MODE == MODE_COLLECT) {
        const long long item = (long long)p * total + i;
        float *xo = W.X_out + item * kMlpIn;
#pragma unroll
        for (int j = 0; j < kMlpIn; j++) xo[j] = f[j];
        W.Y_out[item * 2 + 0] = (eta_conv > 0.0) ? (float)log(st.eta_up / eta_conv) : __int_as_float(0x7fc00000);
        W.Y_out[item * 2 + 1] = (float)o.is_pl;
      }
    }
    if constexpr (ANISO) {
      if (valid) node_store<ANISO>(A, n, out, status);
    } else {
      if (valid) iso_store<NODES>(A, n, q, status);
    }
    if (MODE == MODE_COLLECT && valid) {  // items of inactive phases carry a NaN target
      for (int p = 0; p < A.M.np; p++) {
        const double perc = n.solid ? node_perc(A, n, p) : 0.0;
        if (!fp64_abs_gt_pos(perc, 1e-13)) W.Y_out[((long long)p * total + i) * 2] = __int_as_float(0x7fc00000);
      }
    }
  }
  if (MODE == MODE_WARM) {
    mlp_end(S);
    if (threadIdx.x == 0 && S.fault) atomicExch(&A.stats->mma_fault, 1u);
  }
  flush_acc(A.stats, acc);
}

template <bool ANISO, int NODES>
static cudaError_t launch_warm_t(const SweepArgs &a, const MlpDevice &w, cudaStream_t s, long long count) {
  auto fn = k_sweep_warm<ANISO, NODES>;
  const size_t smem = sizeof(MlpWarpShared);
  cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  fn<<<(unsigned)((count + 127) / 128), 128, smem, s>>>(a, w);
  return cudaGetLastError();
}

cudaError_t launch_sweep_warm(const SweepArgs &a, const MlpDevice &w, bool aniso, cudaStream_t s) {
  cudaError_t e = cudaSuccess;
  if (a.M.Nc > 0) e = aniso ? launch_warm_t<true, 1>(a, w, s, a.M.Nc) : launch_warm_t<false, 1>(a, w, s, a.M.Nc);
  if (e != cudaSuccess || a.M.Nv <= 0) return e;
  return aniso ? launch_warm_t<true, 2>(a, w, s, a.M.Nv) : launch_warm_t<false, 2>(a, w, s, a.M.Nv);
}

// The warm-start form keeps its MLP tiles in dynamic shared memory; asking for the
// largest shared-memory carve-out lets two of its CTAs share an SM (the register file
// allows two), which the occupancy query then reports.
template <bool ANISO, int MODE, int NODES>
static void tiles_attributes() {
  if (MODE != MODE_WARM) return;
  auto fn = k_sweep_tiles<ANISO, MODE, NODES>;
  cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(MlpShared));
  cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
}

template <bool ANISO, int MODE>
static cudaError_t launch_tiles_t(const SweepArgs &a, const WarmArgs &w, cudaStream_t s, int grid) {
  const size_t smem = (MODE == MODE_WARM) ? sizeof(MlpShared) : 0;
  const long long tiles[2] = {(a.M.Nc + kMlpTile - 1) / kMlpTile, (a.M.Nv + kMlpTile - 1) / kMlpTile};
  tiles_attributes<ANISO, MODE, 1>();
  tiles_attributes<ANISO, MODE, 2>();
  if (tiles[0] > 0)
    k_sweep_tiles<ANISO, MODE, 1><<<(unsigned)(tiles[0] < grid ? tiles[0] : grid), kMlpTile, smem, s>>>(a, w);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess || tiles[1] <= 0) return e;
  k_sweep_tiles<ANISO, MODE, 2><<<(unsigned)(tiles[1] < grid ? tiles[1] : grid), kMlpTile, smem, s>>>(a, w);
  return cudaGetLastError();
}

cudaError_t launch_sweep_tiles(const SweepArgs &a, const WarmArgs &w, bool aniso, int mode, cudaStream_t s,
                               int grid) {
  if (grid < 1) grid = 1;
  switch (mode * 2 + (aniso ? 1 : 0)) {
    case MODE_COLLECT * 2: return launch_tiles_t<false, MODE_COLLECT>(a, w, s, grid);
    case MODE_COLLECT * 2 + 1: return launch_tiles_t<true, MODE_COLLECT>(a, w, s, grid);
    case MODE_WARM * 2: return launch_tiles_t<false, MODE_WARM>(a, w, s, grid);
    case MODE_WARM * 2 + 1: return launch_tiles_t<true, MODE_WARM>(a, w, s, grid);
    default: return cudaErrorInvalidValue;
  }
}

int tiles_blocks_per_sm(bool aniso, int mode) {
  int n = 0;
  const void *fn = nullptr;
  switch (mode * 2 + (aniso ? 1 : 0)) {
    case MODE_COLLECT * 2: fn = (const void *)k_sweep_tiles<false, MODE_COLLECT, 1>; break;
    case MODE_COLLECT * 2 + 1: fn = (const void *)k_sweep_tiles<true, MODE_COLLECT, 1>; break;
    case MODE_WARM * 2: fn = (const void *)k_sweep_tiles<false, MODE_WARM, 1>; break;
    default: fn = (const void *)k_sweep_tiles<true, MODE_WARM, 1>; break;
  }
  const size_t smem = (mode == MODE_WARM) ? sizeof(MlpShared) : 0;
  if (mode == MODE_WARM) {
    if (aniso) tiles_attributes<true, MODE_WARM, 1>();
    else tiles_attributes<false, MODE_WARM, 1>();
  }
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, kMlpTile, smem);
  // The query has been seen to report one CTA where registers (255 per thread, 2 CTAs
  // of 128) and the shared-memory carve-out allow two; bound it below by the register
  // file and shared memory directly.  A larger grid only changes residency, not results.
  cudaFuncAttributes fa;
  if (cudaFuncGetAttributes(&fa, fn) == cudaSuccess && fa.numRegs > 0) {
    const int regs = (fa.numRegs + 7) & ~7;
    int by_regs = 65536 / (kMlpTile * regs);
    int by_smem = (int)((227 * 1024) / (smem + fa.sharedSizeBytes + 1024));
    const int own = by_regs < by_smem ? by_regs : by_smem;
    if (own > n) n = own;
  }
  cudaGetLastError();
  return n > 0 ? n : 1;
}

}  // namespace mdz
