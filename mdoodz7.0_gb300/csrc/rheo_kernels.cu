// rheo_kernels.cu -- sweep and point kernels of the local rheology update (sm_103a).
//
// k_sweep<ANISO, NODES> is NonNewtonianViscosityGrid (MDLIB/RheologyDensity.c:1131-1426) /
// NonNewtonianViscosityGridAniso (MDLIB/AnisotropyRoutines.c:885-1217) with the four
// InterpCentroidsToVerticesDouble calls (:1150-1153) fused into the vertex pass: one
// thread per node over the index space [centroids | vertices], launched once over the
// centroids (NODES 1) and once over the vertices (NODES 2) so that each kernel carries only
// its own kind's work (vertices skip the per-phase outputs only centroids keep), per-phase
// tables in the kernel's constant parameter bank (uniform across a warp, so every lookup
// is a broadcast), SoA loads and stores coalesced along the node index.  k_sweep_queue is
// the same sweep as a persistent grid on a work counter.  The warm-start forms are in
// sweep_warm.cu, many grids per launch in sweep_batch.cu.
#include <cuda_runtime.h>

#include "sweep_node.cuh"

namespace mdz {

// One sweep is two launches: the centroids (NODES 1), then the vertices (NODES 2), each
// over its whole range or over the band of rows a banded sweep gives it.
// MINB: CTAs of 128 per SM that the register allocation is capped for.  A node's code is a
// long chain of dependent integer and FP64 instructions, and more resident warps hide more of
// its latency than the spills cost: 7 (72 registers) by default.  A sweep of a few waves
// may lose more to its last, partly empty one, and take 5 (96 registers; sweep_ctas).
// Per call, in us, at 5, 6, 7 and 8 CTAs per SM:
//   isotropic, 5 phases     201^2: 124, 126, 124, 121    401^2: 328, 344, 351, 347
//     513^2: 493, 505, 446, 463    717^2: 937, 903, 840, 885    1025^2: 1862, 1787, 1703, 1757
//   anisotropic, 3 phases   201^2: 94, 91, 91, 90        401^2: 253, 261, 270, 255
//     513^2: 377, 375, 355, 364    717^2: 695, 667, 651, 656    1025^2: 1357, 1303, 1283, 1264
// 2 (255 registers, no spills) is the form that callers may ask for and the autotuner times:
// 2049 x 2049 cells 8.33 ms for 6.72, from the reference's start (1 to 8 evaluations) 28.3
// for 25.8.
template <bool ANISO, int NODES, int MINB>
__global__ void __launch_bounds__(128, MINB) k_sweep(const __grid_constant__ SweepArgs A) {
  if (NODES == 1) pair_begin();
  Acc acc = {0, 0, 0, 0, 0};
  const long long total = NODES == 1 ? (A.ranged ? A.c_n : A.M.Nc) : (A.ranged ? A.v_n : A.M.Nv);
  const long long lo = NODES == 1 ? (A.ranged ? A.c_lo : 0) : A.M.Nc + (A.ranged ? A.v_lo : 0);
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x; j < total; j += stride)
    sweep_node<ANISO, NODES>(A, lo + j, acc);
  flush_acc(A.stats, acc);
  if (NODES == 2) pair_end();
}

// Persistent form: a grid of resident CTAs whose warps pull chunks of 32 consecutive
// nodes from a work counter until none is left.  A warp takes its next chunk as soon as
// its slowest lane is done, instead of a CTA waiting for all four of its warps and the
// block scheduler refilling the SM; one lane fetches for the warp (one atomic per chunk),
// the chunk start is broadcast by shuffle, and the lanes past the end are retired by a
// ballot.  The node body is the plain sweep's, so the results are the same bits.
template <bool ANISO, int NODES>
__global__ void __launch_bounds__(128, 6) k_sweep_queue(const __grid_constant__ SweepArgs A) {
  Acc acc = {0, 0, 0, 0, 0};
  const long long total = NODES == 1 ? A.M.Nc : A.M.Nv;
  const long long lo = NODES == 1 ? 0 : A.M.Nc;
  unsigned long long *counter = &A.stats->queue[NODES - 1];
  const int lane = threadIdx.x & 31;
  for (;;) {
    unsigned long long base = 0;
    if (lane == 0) base = atomicAdd(counter, 32ull);
    base = __shfl_sync(0xffffffffu, base, 0);
    const long long j = (long long)base + lane;
    const unsigned live = __ballot_sync(0xffffffffu, j < total);
    if (live == 0u) break;
    if ((live >> lane) & 1u) sweep_node<ANISO, NODES>(A, lo + j, acc);
  }
  flush_acc(A.stats, acc);
}

// ---------------------------------------------------------------------------------
// independent points: ViscosityConcise / ViscosityConciseAniso
// ---------------------------------------------------------------------------------
// 3 CTAs per SM (168 registers); left alone the compiler takes 196, which makes it 2, and a
// launch of more than two CTAs per SM then waits for another round of them.  2 against 3: 45,000
// points of mixed creep laws 69 -> 50 us, 1,000,000 608 -> 520, 2,000 46 -> 45; 48,000 points of
// the grain-size solve 1.76 -> 1.33 ms, 80,000 of the Popov return 391 -> 328 us.  4 (128
// registers): 2,000 points 47 us, 1,000,000 512, 114,000 of the grain-size solve 3.06 ms for
// 2.63.
__global__ void __launch_bounds__(128, 3) k_points(const __grid_constant__ PointArgs A) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  Acc acc = {0, 0, 0, 0, 0};
  const bool bad_phase = (i < A.n) && (A.in.phase[i] < 0 || A.in.phase[i] >= A.M.np);
  if (bad_phase) {  // phase ids in device memory are only checked here
    if (A.out.status) A.out.status[i] = MDZ_EINVAL;
    record_error(A.stats, i, MDZ_EINVAL);
  }
  if (i < A.n && !bad_phase) {
    const mdz_point_inputs &I = A.in;
    NodeIn in;
    in.Exx = I.Exx[i]; in.Ezz = I.Ezz[i]; in.Exz = I.Exz[i];
    in.Txx0 = I.Txx0[i]; in.Tzz0 = I.Tzz0[i]; in.Txz0 = I.Txz0[i];
    in.G = I.G[i]; in.T = I.T[i]; in.P = I.P[i]; in.d = I.d[i]; in.phi = I.phi[i]; in.X0 = I.X0[i];
    in.dil = I.dil[i]; in.fric = I.fric[i]; in.C = I.C[i]; in.P0 = I.P0[i]; in.T0 = I.T0[i]; in.beta = I.beta[i];
    in.centroid = I.centroid; in.final_update = I.final_update; in.post_process = I.post_process;
    in.want_rho = 1;
    const int p = I.phase[i];
    PointOut o;
    NodeCtx ctx;
    if (A.aniso) {
      in.lxlz = I.lxlz[i]; in.lx2 = I.lx2[i]; in.ani_fac = I.ani_fac[i];
      AnisoNode an;
      node_setup_aniso<FxMath>(A.M, in, true, ctx, an);
      point_aniso<FxMath>(A.M, A.ph[p], in, ctx, an, A.polish, o);
    } else {
      node_setup_iso<FxMath>(A.M, in, true, ctx);
      point_iso<FxMath>(A.M, A.ph[p], in, ctx, A.polish, o);
    }
    const mdz_point_outputs &O = A.out;
    double *dst[24] = {O.eta, O.Txx, O.Tzz, O.Txz, O.etaVE, O.VEcoeff, O.Eii_el, O.Eii_pl, O.Eii_pwl, O.Eii_exp,
                       O.Eii_lin, O.Eii_gbs, O.Eii_cst, O.d1, O.X1, O.OverS, O.Pcorr, O.rho, O.div_el, O.div_pl,
                       O.div_r, O.Wtot, O.Wel, O.Wdiss};
    const double src[24] = {o.eta, o.Txx, o.Tzz, o.Txz, o.etaVE, 0.0, o.Eii_el, o.Eii_pl, o.Eii_pwl, o.Eii_exp,
                            o.Eii_lin, o.Eii_gbs, o.Eii_cst, o.d1, o.X1, o.OverS, o.Pcorr, o.rho, o.div_el,
                            o.div_pl, 0.0, o.Wtot, o.Wel, o.Wdiss};
#pragma unroll
    for (int j = 0; j < 24; j++)
      if (dst[j]) dst[j][i] = src[j];
    if (O.iters) O.iters[i] = o.iters;
    if (O.status) O.status[i] = o.status;
    record_error(A.stats, i, o.status);
    acc.calls = 1; acc.iters = o.iters; acc.plastic = o.is_pl; acc.maxit = o.iters; acc.f32 = o.f32_steps;
  }
  flush_acc(A.stats, acc);
}

// A sweep's vertex kernel reads none of the centroid kernel's outputs, so it is launched as a
// programmatic dependent of it: its CTAs start once every centroid CTA has (pair_begin), in
// the SMs that the centroid kernel's last wave leaves idle -- all of them where a small grid
// is one wave -- and end after it (pair_end).  Where the caller passes one array in two
// places and the kernels share it after all (kernels_share), the vertex kernel follows the
// centroid kernel as any launch of a stream does.
template <class K>
static cudaError_t launch_after(K fn, unsigned grid, int block, cudaStream_t s, bool after, const SweepArgs &a) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3((unsigned)block);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = after ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, fn, a);
}

// Byte ranges of the arrays that a kernel reads or writes; null arrays are empty ranges.
struct Ranges {
  static constexpr int kMax = CI_COUNT + VI_COUNT + CO_COUNT + 2 * MDZ_MAX_PHASES + 8;
  uintptr_t lo[kMax], hi[kMax];
  int n = 0;
  void add(const void *p, long long bytes) {
    lo[n] = (uintptr_t)p;
    hi[n++] = p ? (uintptr_t)p + (uintptr_t)bytes : 0;
  }
};

static bool overlap(const Ranges &x, const Ranges &y) {
  unsigned any = 0;
  for (int i = 0; i < x.n; i++)
    for (int j = 0; j < y.n; j++) any |= (unsigned)(x.lo[i] < y.hi[j]) & (unsigned)(y.lo[j] < x.hi[i]);
  return any != 0;
}

// Whether one of a sweep's two kernels writes memory that the other one reads or writes (an
// output passed as an input too, or one array for two outputs).  Under 1 us of host time.
static bool kernels_share(const SweepArgs &a) {
  const long long cn = a.M.Nc * 8, vn = a.M.Nv * 8;
  Ranges cr, cw, vr, vw;
  for (int i = 0; i < CI_COUNT; i++) cr.add(a.ci[i], cn);
  for (int i = 0; i < CO_COUNT; i++) cw.add(a.co[i], cn);
  for (int i : {(int)CI_T, (int)CI_p_in, (int)CI_d0, (int)CI_phi0}) vr.add(a.ci[i], cn);  // interpolated
  for (int i = 0; i < VI_COUNT; i++) vr.add(a.vi[i], vn);
  for (int i = 0; i < VO_COUNT; i++) vw.add(a.vo[i], vn);
  for (int p = 0; p < a.M.np; p++) {
    cr.add(a.perc_n[p], cn); cw.add(a.peta_n[p], cn);
    vr.add(a.perc_s[p], vn); vw.add(a.peta_s[p], vn);
  }
  cr.add(a.bcp, a.M.Nc);
  vr.add(a.bcp, a.M.Nc);
  vr.add(a.bcg, a.M.Nv);
  return overlap(cw, vr) || overlap(cw, vw) || overlap(cr, vw);
}

// CTAs of 128 per SM for a sweep of so many nodes, centroids and vertices together (their
// kernels overlap).  A call's time steps up where the nodes pass 1, 2 and 4 waves of the
// resident CTAs, with 5 CTAs per SM at 5/7 of the nodes but from a lower level, so each form is
// the faster one in turn.  In us at 5 and 7, without air and with a fifth of the rows air, whose
// nodes cost nothing and shift the steps to 5/4 of the nodes (waves of 152 x 7 CTAs):
//   1.0: 159, 170  1.2: 174, 181; 154, 140  1.4: 191, 194; 168, 176    5 (2-7 %, or loses 10 %)
//   1.7: 276, 214; 184, 189       2.0: 286, 252; 259, 208              7 (13-29 %)
//   2.3: 306, 334; 274, 224       2.6: 326, 356; 281, 295              5 (9 %, or loses 20 %)
//   3.0: 407, 374; 311, 337       3.5: 440, 403; 340, 361              5 with air, 7 without
//   3.9: 472, 437; 409, 376                                            7
// 5 also up to 3.5, for grids with air (517 x 389 cells: 289, 300 and 308 us at 5, 6 and 7).
// The anisotropic sweep steps alike (1.4: 153, 161; 1.7: 203, 172; 2.6: 258, 269).
static int sweep_ctas(long long nodes) {
  const long long wave = 152LL * 7 * 128, wave5 = 152LL * 5 * 128;
  if (nodes <= wave || 2 * nodes >= 7 * wave) return 7;
  return (nodes > 2 * wave5 && nodes <= 2 * wave + wave / 40) ? 7 : 5;
}

template <bool ANISO, int NODES>
static cudaError_t launch_kind(const SweepArgs &a, const LaunchShape &sh, long long count, long long nodes,
                               cudaStream_t s, bool after) {
  if (sh.form == SHAPE_QUEUE) {
    k_sweep_queue<ANISO, NODES><<<(unsigned)sh.grid_cap, 128, 0, s>>>(a);
    return cudaGetLastError();
  }
  const int block = sh.form == SHAPE_COMPACT ? 128 : sh.block;  // SHAPE_COMPACT: the default, one thread per node
  long long grid = (count + block - 1) / block;
  const bool few = sh.grid_cap <= 0 && sweep_ctas(nodes) == 5;
  if (sh.grid_cap > 0 && grid > sh.grid_cap) grid = sh.grid_cap;
  if (sh.form == SHAPE_REGS255) return launch_after(k_sweep<ANISO, NODES, 2>, (unsigned)grid, block, s, after, a);
  if (few) return launch_after(k_sweep<ANISO, NODES, 5>, (unsigned)grid, block, s, after, a);
  return launch_after(k_sweep<ANISO, NODES, 7>, (unsigned)grid, block, s, after, a);
}

cudaError_t launch_sweep(const SweepArgs &a, bool aniso, cudaStream_t s, const LaunchShape &shape) {
  const long long counts[2] = {a.ranged ? a.c_n : a.M.Nc, a.ranged ? a.v_n : a.M.Nv};
  // the work counter of the persistent form covers a whole sweep, not a band of rows
  LaunchShape sh = shape;
  if (sh.form == SHAPE_QUEUE && (a.ranged || sh.grid_cap <= 0)) sh.form = SHAPE_THREAD;
  if (sh.form == SHAPE_QUEUE) sh.block = 128;
  for (int kind = 0; kind < 2; kind++) {
    if (counts[kind] <= 0) continue;
    cudaError_t e;
    const bool after = kind == 1 && counts[0] > 0 && sh.form != SHAPE_QUEUE && !kernels_share(a);
    if (kind == 0 && aniso) e = launch_kind<true, 1>(a, sh, counts[kind], counts[0] + counts[1], s, false);
    else if (kind == 0) e = launch_kind<false, 1>(a, sh, counts[kind], counts[0] + counts[1], s, false);
    else if (aniso) e = launch_kind<true, 2>(a, sh, counts[kind], counts[0] + counts[1], s, after);
    else e = launch_kind<false, 2>(a, sh, counts[kind], counts[0] + counts[1], s, after);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t launch_points(const PointArgs &a, cudaStream_t s) {
  const int block = 128;
  const long long grid = (a.n + block - 1) / block;
  if (grid > 0) k_points<<<(unsigned)grid, block, 0, s>>>(a);
  return cudaGetLastError();
}

// A synchronous call's last launch: the statistics to the host's page-locked copy, and the
// device's back to their initial values for the next call.  In place of one transfer by the
// copy engine before and one after the kernels of every call, which a small call waits for:
// 68.3 -> 62.7 us for the 201 x 201 sweep, 91 -> 86 us for the strain rates of 1025 x 1025.
// host may be null: the reset alone.  It is a kernel and not a copy from host memory, because
// a captured call's copy would read that memory at each replay, not at the capture.
__global__ void k_stats_out(DevStats *d, DevStats *host) {
  if (host) *host = *d;
  DevStats init = {};
  init.err_key = ~0ull;
  *d = init;
}

cudaError_t launch_stats_out(DevStats *d, DevStats *host, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(1);
  cfg.blockDim = dim3(1);
  cfg.stream = s;
  return cudaLaunchKernelEx(&cfg, k_stats_out, d, host);
}

void sweep_kernel_info(int aniso, int *regs, int *smem, int *max_blocks_per_sm, int block, int form) {
  cudaFuncAttributes fa;
  // the centroid kernel: the larger of the two, it sets the launch shape
  const void *fn = aniso ? (const void *)k_sweep<true, 1, 7> : (const void *)k_sweep<false, 1, 7>;
  if (form == SHAPE_REGS255) fn = aniso ? (const void *)k_sweep<true, 1, 2> : (const void *)k_sweep<false, 1, 2>;
  if (form == SHAPE_QUEUE) fn = aniso ? (const void *)k_sweep_queue<true, 1> : (const void *)k_sweep_queue<false, 1>;
  cudaFuncGetAttributes(&fa, fn);
  *regs = fa.numRegs;
  *smem = (int)fa.sharedSizeBytes;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(max_blocks_per_sm, fn, block, 0);
}

}  // namespace mdz
