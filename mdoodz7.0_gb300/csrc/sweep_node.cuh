// sweep_node.cuh -- the device code of one node of a sweep, shared by the plain, warm-start
// and many-grid kernels: its load and set-up, every active phase's local solve, the averages
// and the stores, for one node per thread (sweep_node) and for a CTA that walks its nodes'
// phases in step (warm_node).
#pragma once
#include <cuda_runtime.h>

#include "mlp.cuh"
#include "mlp_warp.cuh"
#include "rheo_kernels.cuh"

namespace mdz {

__device__ __forceinline__ void record_error(DevStats *st, long long node, int status) {
  if (status == MDZ_OK) return;
  const unsigned long long key = ((unsigned long long)node << 8) | (unsigned long long)(-status & 0xff);
  atomicMin(&st->err_key, key);
}

// The centroid and vertex kernels of a sweep as a pair (launch_after, rheo_kernels.cu): the
// centroid kernel lets the vertex kernel start, the vertex kernel ends after it.  Without the
// launch attribute both are no-ops.
__device__ __forceinline__ void pair_begin() { asm volatile("griddepcontrol.launch_dependents;"); }
__device__ __forceinline__ void pair_end() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Counts of one thread.  Below 2^32 for launches of any ordinary length: an item adds at most 70
// to each, so it takes 60 M items in one thread, hours of a launch of one CTA (grid cap 1).
struct Acc {
  unsigned int calls, iters, plastic, maxit;
  unsigned int f32;  // FP32 Newton steps of the starts
};

// Multiplicative perturbation of the strain-rate inputs of every grid of a batch:
// x <- x (1 + amp u), u uniform in [-1, 1) from a counter hash (SplitMix64, Steele et
// al. 2014) of (seed, sweep, grid, node, component).  Rounded steps without
// contraction, so a host restatement reproduces the values exactly.
__device__ __forceinline__ unsigned long long splitmix64(unsigned long long z) {
  z += 0x9e3779b97f4a7c15ull;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}

// u = m 2^-52 - 1 for the top 53 bits m of the hash, in [-1, 1).  Every such value is a
// double, so u is formed exactly without an integer-to-double conversion (an FP64-pipe
// instruction on this GPU): the low 52 bits of m as the fraction of a number in [1, 2),
// minus 1 where m >= 2^52 and minus 2 below (both subtractions exact).
__device__ __forceinline__ double perturb_factor(unsigned long long key, long long node, int comp, double amp) {
  const unsigned long long m = splitmix64(key ^ (unsigned long long)(node * 3 + comp)) >> 11;
  const double f = __longlong_as_double((long long)(0x3ff0000000000000ull | (m & 0xfffffffffffffull)));
  const double u = __dsub_rn(f, (m >> 52) ? 1.0 : 2.0);  // [-1, 1)
  return __dadd_rn(1.0, __dmul_rn(amp, u));
}

// The perturbation of one grid in one sweep, fused into the sweep's load of the strain
// rates: key = the hash of (seed, sweep, grid), amp > 0.
struct PerturbKey {
  unsigned long long key;
  double amp;
};

__device__ __forceinline__ unsigned long long perturb_key(unsigned long long seed, int sweep, int grid) {
  return splitmix64(splitmix64(seed ^ (unsigned long long)sweep) ^ (unsigned long long)grid);
}

// The node's three strain-rate inputs x[0..2] (exxd, ezzd, exz of a centroid or of a
// vertex, node index i over [centroids | vertices]) multiplied by their factors and stored
// back, so the next captured sweep starts from the perturbed rates.
__device__ __forceinline__ void perturb_inputs(const PerturbKey &pk, long long i, double *const *x) {
#pragma unroll
  for (int k = 0; k < 3; k++) *x[k] = __dmul_rn(*x[k], perturb_factor(pk.key, i, k, pk.amp));
}

// ---------------------------------------------------------------------------------
// one node: load and prepare (RheologyDensity.c:1165-1204, :1324-1340;
// AnisotropyRoutines.c:917-977, :1097-1131)
// ---------------------------------------------------------------------------------
struct Node {
  long long idx;  // centroid c0, or vertex c1
  bool centroid, solid;
  double eta_e, inv_eta_e, d1, d2, anif;
  double interp[4];  // vertex T_s, P_s, d0_s, phi0_s
  NodeIn in;
  NodeCtx ctx;
  AnisoNode an;
};

// NODES: 0 either kind (index i decides), 1 centroids only, 2 vertices only; a kernel
// specialised to one kind of node drops the other kind's code and registers
// pk (may be null): the strain rates are perturbed first, at every node, air included.
template <bool ANISO, int NODES = 0>
__device__ __forceinline__ void node_prepare(const SweepArgs &A, long long i, Node &n,
                                             const PerturbKey *pk = nullptr) {
  const ModelConst &M = A.M;
  n.centroid = NODES == 1 ? true : (NODES == 2 ? false : i < M.Nc);
  double mu, exxd, ezzd, exz;
  if (pk) {
    double *x[3];
    if (n.centroid) {
      x[0] = const_cast<double *>(A.ci[CI_exxd]) + i;
      x[1] = const_cast<double *>(A.ci[CI_ezzd]) + i;
      x[2] = const_cast<double *>(A.ci[CI_exz]) + i;
    } else {
      x[0] = const_cast<double *>(A.vi[VI_exxd]) + (i - M.Nc);
      x[1] = const_cast<double *>(A.vi[VI_ezzd]) + (i - M.Nc);
      x[2] = const_cast<double *>(A.vi[VI_exz]) + (i - M.Nc);
    }
    perturb_inputs(*pk, i, x);
  }
  if (n.centroid) {
    const long long c0 = i;
    n.idx = c0;
    const signed char bc = A.bcp[c0];
    n.solid = (bc != 30 && bc != 31);
    if (!n.solid) return;
    mu = A.ci[CI_mu][c0];
    exxd = A.ci[CI_exxd][c0]; ezzd = A.ci[CI_ezzd][c0]; exz = A.ci[CI_exz][c0];
    n.in.Txx0 = A.ci[CI_sxxd0][c0]; n.in.Tzz0 = A.ci[CI_szzd0][c0]; n.in.Txz0 = A.ci[CI_sxz0][c0];
    n.in.T = A.ci[CI_T][c0]; n.in.P = A.ci[CI_p_in][c0]; n.in.d = A.ci[CI_d0][c0];
    n.in.phi = A.ci[CI_phi0][c0]; n.in.X0 = A.ci[CI_X0][c0]; n.in.dil = A.ci[CI_dil][c0];
    n.in.fric = A.ci[CI_fric][c0]; n.in.C = A.ci[CI_C][c0]; n.in.P0 = A.ci[CI_p0][c0]; n.in.T0 = A.ci[CI_T0][c0];
    n.in.beta = A.ci[CI_bet][c0];
    if (ANISO) { n.d1 = A.ci[CI_d1][c0]; n.d2 = A.ci[CI_d2][c0]; n.anif = A.ci[CI_anif][c0]; }
  } else {
    const long long c1 = i - M.Nc;
    n.idx = c1;
    const int Nx = M.Nx, k = (int)(c1 % Nx), l = (int)(c1 / Nx);
    const signed char bcg = A.bcg[c1];
    n.solid = (bcg != 30);
    n.interp[0] = n.interp[1] = n.interp[2] = n.interp[3] = 0.0;
    if (!n.solid) return;
    const int idx[4] = {ring_to_centroid(k, l, M.Ncx, M.Ncz, M.periodic_x),
                        ring_to_centroid(k + 1, l, M.Ncx, M.Ncz, M.periodic_x),
                        ring_to_centroid(k, l + 1, M.Ncx, M.Ncz, M.periodic_x),
                        ring_to_centroid(k + 1, l + 1, M.Ncx, M.Ncz, M.periodic_x)};
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const signed char f = A.bcp[idx[j]];
      const double w = (f == 30 || f == 31) ? 0.0 : 1.0;
      n.interp[0] += w * A.ci[CI_T][idx[j]];
      n.interp[1] += w * A.ci[CI_p_in][idx[j]];
      n.interp[2] += w * A.ci[CI_d0][idx[j]];
      n.interp[3] += w * A.ci[CI_phi0][idx[j]];
    }
#pragma unroll
    for (int j = 0; j < 4; j++) n.interp[j] *= 0.25;
    mu = A.vi[VI_mu][c1];
    exxd = A.vi[VI_exxd][c1]; ezzd = A.vi[VI_ezzd][c1]; exz = A.vi[VI_exz][c1];
    n.in.Txx0 = A.vi[VI_sxxd0][c1]; n.in.Tzz0 = A.vi[VI_szzd0][c1]; n.in.Txz0 = A.vi[VI_sxz0][c1];
    n.in.T = n.interp[0]; n.in.P = n.interp[1]; n.in.d = n.interp[2]; n.in.phi = n.interp[3];
    n.in.X0 = A.vi[VI_X0][c1]; n.in.dil = A.vi[VI_dil][c1]; n.in.fric = A.vi[VI_fric][c1];
    n.in.C = A.vi[VI_C][c1]; n.in.P0 = A.vi[VI_p0][c1]; n.in.T0 = 0.0; n.in.beta = A.vi[VI_bet][c1];
    if (ANISO) { n.d1 = A.vi[VI_d1][c1]; n.d2 = A.vi[VI_d2][c1]; n.anif = A.vi[VI_anif][c1]; }
  }
  n.in.G = mu;
  n.eta_e = (M.elastic == 1) ? M.dt_model * mu : 1.0;
  n.inv_eta_e = ANISO ? FxMath::recip(n.eta_e) : 0.0;
  if (!ANISO) {
    const double h = (M.elastic == 1) ? 0.5 * FxMath::recip(n.eta_e) : 0.0;  // el / eta_e / 2
    n.in.Exx = exxd + n.in.Txx0 * h;
    n.in.Ezz = ezzd + n.in.Tzz0 * h;
    n.in.Exz = exz + n.in.Txz0 * h;
  } else {
    const double angle = n.centroid ? A.ci[CI_angle][n.idx] : A.vi[VI_angle][n.idx];
    double sn, cs;
    sincos(angle - M_PI / 2.0, &sn, &cs);
    n.in.lxlz = cs * sn; n.in.lx2 = cs * cs; n.in.ani_fac = n.anif;
    effective_strain_rate<FxMath>(n.in.Exx, n.in.Ezz, n.in.Exz, exxd, ezzd, exz, n.in.Txx0, n.in.Tzz0, n.in.Txz0, n.d1,
                          n.d2, 1.0 - 1.0 / n.anif, n.eta_e, M.elastic);
  }
  n.in.centroid = n.centroid ? 1 : 0;
  n.in.final_update = A.final_update;
  n.in.post_process = n.centroid ? 1 : 2;  // a vertex keeps only etaVE, eta_phys and X
  n.in.want_rho = n.centroid && (M.density_variations == 1);
  if (ANISO) node_setup_aniso<FxMath>(M, n.in, A.need_lnd, n.ctx, n.an);
  else node_setup_iso<FxMath>(M, n.in, A.need_lnd, n.ctx);
}

__device__ __forceinline__ double node_perc(const SweepArgs &A, const Node &n, int p) {
  return n.centroid ? A.perc_n[p][n.idx] : A.perc_s[p][n.idx];
}

__device__ __forceinline__ void node_iters(const SweepArgs &A, const Node &n, int p, int it) {
  if (n.centroid) { if (A.iters_n) A.iters_n[(long long)p * A.M.Nc + n.idx] = it; }
  else if (A.iters_s) A.iters_s[(long long)p * A.M.Nv + n.idx] = it;
}

// accumulate one phase's result (RheologyDensity.c:1217-1270, :1359-1378)
template <bool ANISO>
__device__ __forceinline__ void node_accumulate(const SweepArgs &A, const Node &n, int p, double perc,
                                                const PointOut &o, double *out, Acc &acc, int &status) {
  set_status(status, o.status);
  acc.calls++; acc.iters += o.iters; acc.plastic += o.is_pl; acc.f32 += o.f32_steps;
  acc.maxit = max(acc.maxit, (unsigned)o.iters);
  node_iters(A, n, p, MDZ_ITEM_WORD(o.iters, o.mech));
  if (n.centroid) A.peta_n[p][n.idx] = o.etaVE;
  else A.peta_s[p][n.idx] = o.etaVE;
  const int avg = A.M.eta_average;
  if (avg == 0) { out[CO_eta] += perc * o.etaVE; out[CO_eta_phys] += perc * o.eta; }
  else if (avg == 1) {
    out[CO_eta] += perc * FxMath::recip(o.etaVE);
    out[CO_eta_phys] += perc * FxMath::recip(o.eta);
  } else {
    out[CO_eta] += perc * FxMath::log(o.etaVE);
    out[CO_eta_phys] += perc * FxMath::log(o.eta);
  }
  if (ANISO) out[CO_VE] += perc * o.etaVE * n.inv_eta_e;
  out[CO_X] += perc * o.X1;
  if (!n.centroid) return;
  out[CO_eII_el] += perc * o.Eii_el;
  out[CO_eII_pl] += perc * o.Eii_pl;
  out[CO_eII_pwl] += perc * o.Eii_pwl;
  out[CO_eII_exp] += perc * o.Eii_exp;
  out[CO_eII_lin] += perc * o.Eii_lin;
  out[CO_eII_gbs] += perc * o.Eii_gbs;
  out[CO_eII_cst] += perc * o.Eii_cst;
  out[CO_d] += perc * o.inv_d1;
  out[CO_Wtot] += perc * o.Wtot;
  out[CO_Wdiss] += perc * o.Wdiss;
  out[CO_Wel] += perc * o.Wel;
  out[CO_p_corr] += perc * o.Pcorr;
  out[CO_div_el] += perc * o.div_el;
  out[CO_div_pl] += perc * o.div_pl;
  out[CO_OverS] += perc * o.OverS;
  out[CO_rho] += perc * o.rho;
}

// finalize the averages and the stress, then store (:1274-1313, :1380-1405)
template <bool ANISO>
__device__ __forceinline__ void node_store(const SweepArgs &A, const Node &n, double *out, int status) {
  const ModelConst &M = A.M;
  const int avg = M.eta_average;
  if (n.solid) {
    if (n.centroid) {
      out[CO_d] = FxMath::recip(out[CO_d]);
      if (!ANISO && !fp64_finite(out[CO_d])) set_status(status, MDZ_EEMPTY_CELL);
    }
    if (avg == 1) {
      out[CO_eta] = FxMath::recip(out[CO_eta]);
      out[CO_eta_phys] = FxMath::recip(out[CO_eta_phys]);
      if (!fp64_finite(out[CO_eta_phys])) set_status(status, MDZ_ENONFINITE);
    } else if (avg == 2) {
      out[CO_eta] = FxMath::exp(out[CO_eta]);
      out[CO_eta_phys] = FxMath::exp(out[CO_eta_phys]);
    }
    const double eta2 = 2.0 * out[CO_eta];
    const NodeIn &in = n.in;
    if (!ANISO) {
      out[CO_sxxd] = eta2 * in.Exx; out[CO_szzd] = eta2 * in.Ezz; out[CO_sxz] = eta2 * in.Exz;
    } else {  // AnisotropyRoutines.c:1079-1086
      const double a = 1.0 - 1.0 / n.anif, d1 = n.d1, d2 = n.d2;
      out[CO_sxxd] = eta2 * (in.Exx * (1.0 - a * d1) + in.Ezz * a * d1 - 2.0 * in.Exz * a * d2);
      out[CO_szzd] = eta2 * (in.Ezz * (1.0 - a * d1) + in.Exx * a * d1 + 2.0 * in.Exz * a * d2);
      out[CO_sxz] = eta2 * (-in.Exx * a * d2 + in.Ezz * a * d2 + 2 * in.Exz * (a * (d1 - 0.5) + 0.5));
    }
    record_error(A.stats, A.node_base + (n.centroid ? n.idx : M.Nc + n.idx), status);
  } else {
    for (int p = 0; p < M.np; p++) node_iters(A, n, p, 0);
  }
  if (n.centroid) {
#pragma unroll
    for (int i = 0; i < CO_COUNT; i++)
      if (A.co[i]) A.co[i][n.idx] = out[i];
  } else {
    const long long c1 = n.idx;
    A.vo[VO_T][c1] = n.interp[0]; A.vo[VO_P][c1] = n.interp[1];
    A.vo[VO_d0][c1] = n.interp[2]; A.vo[VO_phi0][c1] = n.interp[3];
    A.vo[VO_sxxd][c1] = out[CO_sxxd]; A.vo[VO_szzd][c1] = out[CO_szzd]; A.vo[VO_sxz][c1] = out[CO_sxz];
    A.vo[VO_eta_phys][c1] = out[CO_eta_phys]; A.vo[VO_eta][c1] = out[CO_eta]; A.vo[VO_X][c1] = out[CO_X];
    if (A.vo[VO_VE]) A.vo[VO_VE][c1] = out[CO_VE];
  }
}

// ---------------------------------------------------------------------------------
// The isotropic sweep's averages.  The same sums as node_accumulate and node_store form from
// a PointOut (RheologyDensity.c:986-1053, :1217-1313, :1359-1405), with what is common to a
// node's phases taken out of the phase loop and applied once per node: the strain rates
// over Eii, the elastic rate over 1 / (2 eta_el), the elastic power over 1 / eta_el, and the
// pressure terms from the sum of the fractions and the plastic corrections alone.  With
// S = sum_k Eii_k / Eii (diffusion creep at the reference grain size) plus the plastic share,
// the dissipative viscosity is eta / S; the powers are w = Tii^2 / eta (total), w S
// (dissipative) and Tii^2 / eta_el (elastic).  A centroid's phase takes 24 FP64 instructions
// here and took about 60.
// ---------------------------------------------------------------------------------
struct IsoAcc {
  double eta, eta_phys, perc;
  double el, pl, pwl, exp, lin, cst, d, Wtot, Wel, Wdiss, dP, div_pl, OverS, rho;  // centroids
};

// Tii^2 share / eta_ve below zero (:1045-1050); asked where the signs differ, so out of line
static __device__ __noinline__ bool dissipation_negative(double share, double eta_ve, double Tii) {
  return Tii * Tii * (share / eta_ve) < 0.0;
}

template <int NODES>
__device__ __forceinline__ void iso_accumulate(const SweepArgs &A, const Node &n, int p, double perc, const IsoState &S,
                                               PointOut &o, IsoMid &m, IsoAcc &q, Acc &acc, int &status) {
  const ModelConst &M = A.M;
  const PhaseConst &ph = A.ph[p];
  const NodeCtx &c = n.ctx;
  const int fl = ph.flags;
  const int plastic = c.plastic_on ? ((fl & F_PL1) ? 1 : ((fl & F_PL2) ? 2 : 0)) : 0;
  if (plastic == 2) {
    popov_return<FxMath>(M, ph, n.in, c, S, o, m);
    if (m.is_pl) {
      m.pl_share = 2.0 * m.lam_dot * m.A_tau * m.eta_ve * FxMath::recip(m.Tii);
      m.T_over_eta = m.Tii * FxMath::recip(m.eta_ve);
    }
  }
  double share = 0.0;  // S
  if (o.mech & MDZ_MECH_PEIERLS) share = m.e_exp;
  if (fl & F_PWL) share = __dadd_rn(share, m.e_pwl);  // sums and products rounded apart: the same bits in every kernel
  if (fl & F_LIN) {
    // eta_lin = B pow(Eii_lin, 1/n-1) pow(d1, m/n) = Tii/(2 Eii_lin) (d1/d)^(m/n), d1 = gs_ref
    double l = m.e_lin;
    if ((fl & F_LIN_M) && !(fl & F_GS)) l = __dmul_rn(l, FxMath::exp(__fma_rn(ph.lin_mn, S.lnd, ph.lin_lnd)));
    share = __dadd_rn(share, l);
  }
  if (fl & F_CST) share = __dadd_rn(share, m.e_cst);
  if (m.is_pl) share = __dadd_rn(share, m.pl_share);
  const double ve = m.is_pl ? m.eta_vep : m.eta_ve;
  const double etaVE = clamp_eta(M, ve), eta = clamp_eta(M, __dmul_rn(m.eta_ve, FxMath::recip(share)));
  if (m.is_pl) o.mech |= MDZ_MECH_YIELD;
  set_status(status, o.status);
  acc.calls++; acc.iters += o.iters; acc.plastic += m.is_pl; acc.f32 += o.f32_steps;
  acc.maxit = max(acc.maxit, (unsigned)o.iters);
  node_iters(A, n, p, MDZ_ITEM_WORD(o.iters, o.mech));
  (NODES == 1 ? A.peta_n[p] : A.peta_s[p])[n.idx] = etaVE;
  const int avg = M.eta_average;
  if (avg == 0) { q.eta = fma(perc, etaVE, q.eta); q.eta_phys = fma(perc, eta, q.eta_phys); }
  else if (avg == 1) {
    q.eta = fma(perc, FxMath::recip(etaVE), q.eta);
    q.eta_phys = fma(perc, FxMath::recip(eta), q.eta_phys);
  } else {
    q.eta = fma(perc, FxMath::log(etaVE), q.eta);
    q.eta_phys = fma(perc, FxMath::log(eta), q.eta_phys);
  }
  q.perc += perc;
  if (NODES == 2) return;
  if (fl & F_PWL) q.pwl = fma(perc, m.e_pwl, q.pwl);
  if (o.mech & MDZ_MECH_PEIERLS) q.exp = fma(perc, m.e_exp, q.exp);
  if (fl & F_LIN) q.lin = fma(perc, m.e_lin, q.lin);
  if (fl & F_CST) q.cst = fma(perc, m.e_cst, q.cst);
  q.d = fma(perc, o.inv_d1, q.d);
  if (c.elastic) {
    const double t2 = fp64_scale(ve, 1);
    const double ex = fma(t2, n.in.Exx, -n.in.Txx0), ez = fma(t2, n.in.Ezz, -n.in.Tzz0);
    const double exz = fma(t2, n.in.Exz, -n.in.Txz0);
    // (ex^2 + ez^2 + ey^2) / 2 + exz^2 with ey = -(ex + ez)
    q.el = fma(perc, FxMath::sqrt(__fma_rn(exz, exz, __fma_rn(ez, __dadd_rn(ex, ez), __dmul_rn(ex, ex)))), q.el);
  }
  const double rate = plastic == 2 ? 2.0 * m.lam_dot * m.A_tau : m.gdot;
  if (m.is_pl) q.pl = fma(perc, rate, q.pl);
  const double pT = __dmul_rn(perc, m.Tii), w = __dmul_rn(pT, m.T_over_eta);
  q.Wtot = __dadd_rn(q.Wtot, w);
  q.Wdiss = fma(w, share, q.Wdiss);
  q.Wel = fma(pT, m.Tii, q.Wel);
  if ((int)(fp64_hi(share) ^ fp64_hi(m.eta_ve)) < 0 && dissipation_negative(share, m.eta_ve, m.Tii))
    set_status(status, MDZ_EWDISS);
  if (m.is_pl && (fp64_bits(m.Pc) != fp64_bits(n.in.P) || !fp64_is_zero(m.divp))) {
    q.dP = fma(perc, m.Pc - n.in.P, q.dP);
    q.div_pl = fma(perc, m.divp, q.div_pl);
  }
  if (plastic == 2) q.OverS = fma(perc, m.eta_vp * m.lam_dot * m.A_tau, q.OverS);
  else if (plastic == 1 && !((fl & F_VP1) && fp64_is_zero(ph.eta_vp))) q.OverS = fma(perc, m.eta_vp * m.gdot, q.OverS);
  if (n.in.want_rho)
    q.rho = fma(perc, density(M, ph, c.T, (n.in.final_update == 1) ? m.Pc : n.in.P, n.in.X0, n.in.phi), q.rho);
}

// The node's outputs from the averages, in node_store's order of checks.
template <int NODES>
__device__ __forceinline__ void iso_store(const SweepArgs &A, const Node &n, IsoAcc &q, int status) {
  double out[CO_COUNT];
#pragma unroll
  for (int j = 0; j < CO_COUNT; j++) out[j] = 0.0;
  if (n.solid) {
    const NodeCtx &c = n.ctx;
    out[CO_eta] = q.eta;
    out[CO_eta_phys] = q.eta_phys;
    out[CO_X] = n.in.X0 * q.perc;
    if (NODES == 1) {
      out[CO_eII_el] = c.elastic ? q.el * fp64_scale(c.inv_eta_el, -1) : 0.0;
      out[CO_eII_pl] = fp64_scale(q.pl, -1);
      const double unit = rate_unit(c.Eii);
      out[CO_eII_pwl] = q.pwl * unit;
      out[CO_eII_exp] = q.exp * unit;
      out[CO_eII_lin] = q.lin * unit;
      out[CO_eII_cst] = q.cst * unit;
      out[CO_d] = q.d;
      out[CO_Wtot] = q.Wtot;
      out[CO_Wdiss] = q.Wdiss;
      out[CO_Wel] = q.Wel * c.inv_eta_el;
      out[CO_p_corr] = fma(n.in.P, q.perc, q.dP);
      out[CO_div_el] = -fma(n.in.P - n.in.P0, q.perc, q.dP) * c.inv_Kdt;
      out[CO_div_pl] = q.div_pl;
      out[CO_OverS] = q.OverS;
      out[CO_rho] = q.rho;
    }
  }
  node_store<false>(A, n, out, status);
}

// Local solve, plastic return and averages of one (node, phase) in one thread.
template <int NODES>
__device__ __forceinline__ void iso_sweep_item(const SweepArgs &A, const Node &n, int p, double perc, IsoState &S,
                                               float s_start, int polish, PointOut &o, IsoAcc &q, Acc &acc,
                                               int &status, double *eta_conv = nullptr) {
  IsoMid m;
  iso_ve<FxMath>(A.M, A.ph[p], n.in, n.ctx, S, s_start, polish, o, m, eta_conv);
  if (iso_yields_dp(A.M, A.ph[p], n.ctx, m)) dp_return_inline(A.M, A.ph[p], n.in, n.ctx, m);
  iso_accumulate<NODES>(A, n, p, perc, S, o, m, q, acc, status);
  o.is_pl = m.is_pl;
}

__device__ __forceinline__ void iso_acc_zero(IsoAcc &q) {
  q.eta = q.eta_phys = q.perc = q.el = q.pl = q.pwl = q.exp = q.lin = q.cst = q.d = q.Wtot = q.Wel = q.Wdiss = q.dP =
      q.div_pl = q.OverS = q.rho = 0.0;
}

__device__ __forceinline__ void flush_acc(DevStats *st, Acc &acc) {
  // warp-aggregate, then one atomic per warp
  unsigned long long calls = acc.calls, iters = acc.iters, plastic = acc.plastic, f32 = acc.f32;
  for (int o = 16; o > 0; o >>= 1) {
    calls += __shfl_down_sync(0xffffffffu, calls, o);
    iters += __shfl_down_sync(0xffffffffu, iters, o);
    plastic += __shfl_down_sync(0xffffffffu, plastic, o);
    acc.maxit = max(acc.maxit, __shfl_down_sync(0xffffffffu, acc.maxit, o));
    f32 += __shfl_down_sync(0xffffffffu, f32, o);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(&st->calls, calls);
    atomicAdd(&st->iters, iters);
    atomicAdd(&st->plastic, plastic);
    atomicMax(&st->maxit, acc.maxit);
    if (f32) atomicAdd(&st->f32_steps, f32);
  }
}

// ---------------------------------------------------------------------------------
// plain sweep: one thread per node
// ---------------------------------------------------------------------------------
// One node of one grid: prepare, every active phase's local solve, averaging, store.
template <bool ANISO, int NODES = 0>
__device__ __forceinline__ void sweep_node(const SweepArgs &A, long long i, Acc &acc,
                                           const PerturbKey *pk = nullptr) {
  Node n;
  node_prepare<ANISO, NODES>(A, i, n, pk);
  int status = MDZ_OK;
  if constexpr (ANISO) {
    double out[CO_COUNT];
#pragma unroll
    for (int j = 0; j < CO_COUNT; j++) out[j] = 0.0;
    if (n.solid) {
      for (int p = 0; p < A.M.np; p++) {
        const double perc = node_perc(A, n, p);
        if (!fp64_abs_gt_pos(perc, 1e-13)) {  // :1210-1212
          node_iters(A, n, p, 0);
          continue;
        }
        PointOut o;
        point_aniso<FxMath>(A.M, A.ph[p], n.in, n.ctx, n.an, A.polish, o);
        node_accumulate<ANISO>(A, n, p, perc, o, out, acc, status);
      }
    }
    node_store<ANISO>(A, n, out, status);
  } else {
    IsoAcc q;
    iso_acc_zero(q);
    if (n.solid) {
      for (int p = 0; p < A.M.np; p++) {
        const double perc = node_perc(A, n, p);
        if (!fp64_abs_gt_pos(perc, 1e-13)) {
          node_iters(A, n, p, 0);
          continue;
        }
        PointOut o;
        IsoState S;
        iso_setup<FxMath>(A.M, A.ph[p], n.in, n.ctx, S, o, A.polish == 0);
        iso_sweep_item<NODES>(A, n, p, perc, S, 1.0f, A.polish, o, q, acc, status);
      }
    }
    iso_store<NODES>(A, n, q, status);
  }
}

// ---------------------------------------------------------------------------------
// learned warm start, per warp: the plain sweep with the network between each phase's
// set-up and its local solve, evaluated by the warp's 32 lanes on the tensor cores
// (mlp_warp.cuh)
// ---------------------------------------------------------------------------------
// The network's normalised inputs for one (node, phase) (zeros where the lane has none).
__device__ __forceinline__ void warm_inputs(const MlpDevice &W, const float *f, int nfeat, float *x) {
#pragma unroll
  for (int j = 0; j < kMlpIn; j++) x[j] = (j < nfeat) ? (f[j] - W.x_shift[j]) * W.x_scale[j] : 0.0f;
}

// One node per lane, the warp's 32 nodes consecutive, so every lane of a warp runs the
// same number of node iterations and reaches the network at the same phase; lanes past
// the end or at inactive (node, phase) items feed zeros and discard the output.  Every lane
// of the warp calls it together (valid false: a lane without a node).
template <bool ANISO, int NODES>
__device__ __forceinline__ void warm_node(const SweepArgs &A, MlpWarpShared &S, const MlpDevice &W, bool valid,
                                          long long i, Acc &acc, const PerturbKey *pk = nullptr) {
  const int nfeat = ANISO ? kFeatAniso : kFeatIso;
  Node n;
  n.solid = false;
  n.centroid = NODES == 1;
  if (valid) node_prepare<ANISO, NODES>(A, i, n, pk);
  double out[CO_COUNT];  // anisotropic
  IsoAcc q;              // isotropic
#pragma unroll
  for (int k = 0; k < CO_COUNT; k++) out[k] = 0.0;
  iso_acc_zero(q);
  int status = MDZ_OK;
  for (int p = 0; p < A.M.np; p++) {  // uniform over the warp
    const double perc = (valid && n.solid) ? node_perc(A, n, p) : 0.0;
    const bool active = fp64_abs_gt_pos(perc, 1e-13);
    if (valid && n.solid && !active) node_iters(A, n, p, 0);
    IsoState st;
    PointOut o;
    float f[kMlpIn], x[kMlpIn];
#pragma unroll
    for (int k = 0; k < kMlpIn; k++) f[k] = 0.0f;
    if (active) {
      if constexpr (ANISO) aniso_setup<FxMath>(A.M, A.ph[p], n.in, n.ctx, n.an, st, o, W.polish_iters == 0);
      else iso_setup<FxMath>(A.M, A.ph[p], n.in, n.ctx, st, o, W.polish_iters == 0);
      warm_features(A.M, n.in, n.ctx, st, ANISO, f);
    }
    warm_inputs(W, f, nfeat, x);
    __syncwarp();
    const float y = mlp_warp_predict(S, x);
    if (!active) continue;
    const float s_start = warm_start_point(y, W.z_scale, W.z_shift);
    if constexpr (ANISO) {
      aniso_finish<FxMath>(A.M, A.ph[p], n.in, n.ctx, n.an, st, s_start, W.polish_iters, o);
      node_accumulate<ANISO>(A, n, p, perc, o, out, acc, status);
    } else {
      iso_sweep_item<NODES>(A, n, p, perc, st, s_start, W.polish_iters, o, q, acc, status);
    }
  }
  if constexpr (ANISO) {
    if (valid) node_store<ANISO>(A, n, out, status);
  } else {
    if (valid) iso_store<NODES>(A, n, q, status);
  }
}

}  // namespace mdz
