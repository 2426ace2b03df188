// mpm_return.cuh -- the MohrCoulomb plastic return as a loop of uniform passes.
//
// MohrCoulomb<Tdim>::compute_stress (mohr_coulomb.tcc:348-513) evaluates the
// stress invariants and yield state of a stress, and mostly dF/dsigma and
// dP/dsigma of it, at the trial stress, at the old stress, after every
// correction and at the final stress.  Written as straight-line code, as in
// mc_stress, each of these evaluations is a separate copy of the same three
// heavy pieces: inlined, the dense return kernels outgrow the instruction
// cache; called out of line, every call passes its arrays through the stack.
// Here the return is one loop whose every pass evaluates, at a single site,
// the invariants and yield state of the point's current stress and, where its
// phase needs them, dF/dsigma and dP/dsigma -- then makes the phase's small
// update.  Each heavy piece is inlined once, everything can stay in
// registers, and the lanes of a warp that are in different phases run the
// same pass code together.  Per point the evaluations and their inputs are those
// of mc_stress<R, PD, false>: the same bits in the units that never fuse a multiply
// and an add.  In the mixed unit the compiler may fuse differently in different
// bodies; that the return kernel and the persistent step, which both inline this
// loop, agree bit for bit is held by a test of flowing columns.
#pragma once

#include "mpm_math.cuh"

namespace mpm_b200 {
inline namespace MPM_MC_FORM {

enum { MR_OLD = 0, MR_TRIAL, MR_LOOP, MR_FINAL };

// One point's return in progress.
template <typename R>
struct McPoint {
  int phase, itr;
  bool on_surface;  // the old stress is on the yield surface
  R trial[6], upd[6], sv[SV_N];
  R pd;   // plastic deviatoric strain at the start of the update
  R dpd;  // its increment
  R yield_trial;
  LodeTrig<R> lt;
  FrictionTrig<R> ft;
};

// The part of mc_stress before its first invariants: softening of the state,
// elastic predictor, separated state.  q.sv, with the plastic deviatoric strain
// in SV_PD, is loaded by the caller.  True when the point is finished here
// (separated: out = 0 and q.sv final).
template <typename R>
__device__ __forceinline__ bool mc_begin(const MaterialT<R>& m, const R* stress, const R* dstrain,
                                         R density, McPoint<R>& q, R* out) {
  q.pd = q.sv[SV_PD];
  const R pdstrain = q.pd;
  if (m.softening && pdstrain > m.pd_peak) {
    if (pdstrain < m.pd_res) {
      q.sv[SV_PHI] = m.phi_res + ((m.phi_peak - m.phi_res) * (pdstrain - m.pd_res) /
                                  (m.pd_peak - m.pd_res));
      q.sv[SV_PSI] = m.psi_res + ((m.psi_peak - m.psi_res) * (pdstrain - m.pd_res) /
                                  (m.pd_peak - m.pd_res));
      q.sv[SV_COH] = m.c_res + ((m.c_peak - m.c_res) * (pdstrain - m.pd_res) / (m.pd_peak - m.pd_res));
    } else {
      q.sv[SV_PHI] = m.phi_res;
      q.sv[SV_PSI] = m.psi_res;
      q.sv[SV_COH] = m.c_res;
    }
    const R apex = q.sv[SV_COH] / tan(q.sv[SV_PHI]);
    if (q.sv[SV_TC] > apex) q.sv[SV_TC] = check_low(apex);
  }
  q.sv[SV_YIELD] = R(0);
  {
    R t[6];
    de_mul(m, dstrain, t);
#pragma unroll
    for (int i = 0; i < 6; ++i) q.trial[i] = stress[i] + t[i];
  }
  if (density <= m.min_packing * m.grain_density) {
    q.sv[SV_PD] = q.pd + sqrt(R(3) * mu_j2(q.trial)) / R(3) / m.shear;
    q.sv[SV_YIELD] = R(3);
#pragma unroll
    for (int i = 0; i < 6; ++i) out[i] = R(0);
    return true;
  }
  q.ft = friction_trig(m, q.sv);
  q.phase = MR_OLD;
  q.itr = 0;
  q.dpd = R(0);
  q.yield_trial = R(0);
  return false;
}

// One pass: the invariants and yield state of the point's current stress X
// (old, trial, corrected), dF/dsigma and dP/dsigma of X where the phase needs
// them, then the phase's update.  True when the point is finished (out and q.sv
// final).
//
// The old stress comes first, where mc_stress evaluates the trial stress
// first: a point whose old stress is off the yield surface takes its first
// correction from the trial stress's dF/dsigma, and in this order the pass
// that finds the trial stress plastic makes it, with no second visit of the
// trial stress.  The evaluations and their inputs are the same; what the old
// stress leaves in q.sv (epsilon, rho) the later passes overwrite.  One pass
// less for such points: 0.8M flowing points 123.0 -> 120.4 us, a few scattered
// ones (one chain of dependent FP64 operations) 14.5 -> 12.6 us.
template <typename R>
__device__ __forceinline__ bool mc_pass(const MaterialT<R>& m, const R* stress, const R* dstrain,
                                        McPoint<R>& q, R* out) {
  const R Tolerance = R(1E-1);
  const int ph = q.phase;
  R X[6];
#pragma unroll
  for (int i = 0; i < 6; ++i) X[i] = ph == MR_OLD ? stress[i] : (ph == MR_TRIAL ? q.trial[i] : q.upd[i]);
  mc_invariants(X, q.sv, q.lt);
  R yf[2];
  const int yt = mc_yield_state(yf, q.sv, q.lt, q.ft);
  bool flow;  // dF/dsigma and dP/dsigma of X are needed
  if (ph == MR_OLD) {
    R yield = huge_value<R>();
    if (yt == MC_TENSILE) yield = yf[0];
    if (yt == MC_SHEAR) yield = yf[1];
    flow = q.on_surface = fabs(yield) < Tolerance;
    if (!flow) {
      q.phase = MR_TRIAL;
      return false;
    }
  } else if (ph == MR_TRIAL) {
    if (yt == MC_ELASTIC) {
      q.sv[SV_YIELD] = R(0);
#pragma unroll
      for (int i = 0; i < 6; ++i) out[i] = q.trial[i];
      return true;
    }
    q.sv[SV_YIELD] = yt == MC_TENSILE ? R(2) : R(1);
    q.yield_trial = yt == MC_TENSILE ? yf[0] : yf[1];
    q.phase = MR_LOOP;
    if (q.on_surface) return false;  // upd is the old stress's correction
    flow = true;
#pragma unroll
    for (int i = 0; i < 6; ++i) q.upd[i] = q.trial[i];
  } else {
    flow = ph == MR_LOOP && !(yf[0] < Tolerance && yf[1] < Tolerance);
    if (!flow) {
      // converged (the invariants of the final stress are in q.sv), or MR_FINAL
      // after the 100th correction (they were just evaluated)
      q.sv[SV_PD] = q.pd + q.dpd;
#pragma unroll
      for (int i = 0; i < 6; ++i) out[i] = q.upd[i];
      return true;
    }
    if (yt == MC_TENSILE) q.yield_trial = yf[0];
    if (yt == MC_SHEAR) q.yield_trial = yf[1];
    if (++q.itr == 100) q.phase = MR_FINAL;
  }
  R softening = R(0), dp_dq = R(0), df[6], dp[6];
  mc_df_dp(m, yt, q.sv, q.lt, q.ft, q.pd, X, df, dp, &dp_dq, &softening);
  const R num = ph == MR_OLD ? row_de_dot(m, df, dstrain) : q.yield_trial;
  const R lambda = num / (row_de_dot(m, df, dp) + softening);
  if (ph == MR_OLD) {
#pragma unroll
    for (int i = 0; i < 6; ++i) q.upd[i] = q.trial[i];
    q.phase = MR_TRIAL;
  }
  sub_lambda_de(m, lambda, dp, q.upd);
  q.dpd += lambda * dp_dq;
  return false;
}

// The full MohrCoulomb update of mc_compute_stress<R, R> as passes: sv holds
// the state variables with the plastic deviatoric strain in SV_PD (updated in
// place), corrections receives the number of return corrections.
template <typename R>
__device__ __forceinline__ void mc_return(const MaterialT<R>& m, const R* stress, const R* dstrain,
                                          R density, R* sv, R* out, int* corrections) {
  McPoint<R> q;
#pragma unroll
  for (int k = 0; k < SV_N; ++k) q.sv[k] = sv[k];
  if (!mc_begin(m, stress, dstrain, density, q, out)) {
    while (!mc_pass(m, stress, dstrain, q, out)) {
    }
    q.sv[SV_THETA] = mc_lode_angle(q.lt);  // of the last pass's stress, the final one
  }
#pragma unroll
  for (int k = 0; k < SV_N; ++k) sv[k] = q.sv[k];
  *corrections = q.itr;
}

}  // namespace MPM_MC_FORM
}  // namespace mpm_b200
