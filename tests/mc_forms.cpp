// The two forms of the MohrCoulomb update (as the reference writes it; with reciprocals and the
// triple-angle equation) side by side on the host.  Compiled twice, with MPM_MC_RECIPROCALS and
// without (which adds main), and linked into one program: each form keeps its own definitions.
// The as-written form in 80-bit arithmetic is the reference of single evaluations.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>
using std::acos, std::asin, std::cos, std::fabs, std::fma, std::fmaf, std::sin, std::sqrt, std::tan;
namespace mpm_b200 {  // for R = long double, before the header's templates use them
inline double value(long double x) { return (double)x; }
inline void sin_cos(long double x, long double* s, long double* c) { *s = std::sin(x), *c = std::cos(x); }
}  // namespace mpm_b200
#define __device__
#define __forceinline__ inline
#include "mpm_return.cuh"
namespace mpm_b200 {
template <>
struct HighPrecision<long double> {
  using T = long double;
};
}  // namespace mpm_b200
using namespace mpm_b200;

struct Eval {  // one evaluation at a stress
  int yt;
  double yf[2], df[6], dp[6], dq, soft, theta;
};
struct Return {
  int itr, yield;
  double out[6], sv[SV_N];
};

template <typename R>
static Eval evaluate(const MaterialParams& md, const double* s, const double* svd) {
  const MaterialT<R> m = material_cast<R>(md);
  R sv[SV_N], st[6], yf[2], df[6], dp[6], dq, soft;
  for (int k = 0; k < SV_N; ++k) sv[k] = svd[k];
  for (int k = 0; k < 6; ++k) st[k] = s[k];
  const FrictionTrig<R> ft = friction_trig(m, sv);
  LodeTrig<R> lt;
  mc_invariants(st, sv, lt);
  Eval e;
  e.yt = mc_yield_state(yf, sv, lt, ft);
  mc_df_dp(m, e.yt, sv, lt, ft, sv[SV_PD], st, df, dp, &dq, &soft);
  for (int k = 0; k < 2; ++k) e.yf[k] = yf[k];
  for (int k = 0; k < 6; ++k) e.df[k] = df[k], e.dp[k] = dp[k];
  e.dq = dq, e.soft = soft, e.theta = mc_lode_angle(lt);
  return e;
}
static Return update(const MaterialParams& m, const double* s, const double* de, const double* sv) {
  Return r{};
  std::copy(sv, sv + SV_N, r.sv);
  mc_return(m, s, de, 1800., r.sv, r.out, &r.itr);
  r.yield = (int)r.sv[SV_YIELD];
  return r;
}

#ifdef MPM_MC_RECIPROCALS
Eval evaluate_reciprocal(const MaterialParams& m, const double* s, const double* sv) { return evaluate<double>(m, s, sv); }
Return update_reciprocal(const MaterialParams& m, const double* s, const double* de, const double* sv) { return update(m, s, de, sv); }
// largest relative errors of sin, cos and the angle itself, cos 3 theta all over [-1, 1] and near both ends
void lode_errors(double* worst) {
  worst[0] = worst[1] = worst[2] = 0.;
  for (int i = 1; i <= 300000; ++i) {
    const double z = i / 300000.;
    const double v = i % 3 == 0 ? 2 * z - 1 : (i % 3 == 1 ? 1 : -1) * (1 - std::pow(10., -16 * z));
    double s, c;
    lode_trig(v, &s, &c);
    const long double th = acosl((long double)v) / 3, got[3] = {s, c, lode_theta(s, c)}, want[3] = {sinl(th), cosl(th), th};
    for (int k = 0; k < 3; ++k)
      if (want[k] != 0) worst[k] = std::max(worst[k], (double)fabsl((got[k] - want[k]) / want[k]));
  }
}
#else
Eval evaluate_reciprocal(const MaterialParams&, const double*, const double*);
Return update_reciprocal(const MaterialParams&, const double*, const double*, const double*);
void lode_errors(double*);

static double off(const double* a, const double* b, int n) {
  double d = 0, s = 0;
  for (int k = 0; k < n; ++k) d = std::max(d, fabs(a[k] - b[k])), s = std::max(s, fabs(b[k]));
  return s > 0 ? d / s : d;
}

int main() {
  double lode[3];
  lode_errors(lode);
  std::printf("lode %.3g %.3g %.3g\n", lode[0], lode[1], lode[2]);
  std::mt19937_64 g(7);
  std::normal_distribution<double> n;
  std::uniform_real_distribution<double> U(0, 1);
  const double u = 1.1102230246251565e-16;
  int evals[3] = {0, 0, 0}, soft_evals = 0, same_bits = 0, returns = 0, corrections = 0, counts = 0, yields = 0, finite = 0;
  int shear = 0, tensile = 0, off_surface = 0;
  double w_yf = 0, w_df = 0, w_dp = 0, w_dq = 0, w_soft = 0, w_theta = 0;
  std::vector<double> d_out;
  for (int k = 0; k < 20000; ++k) {
    const double phi = (20 + 20 * U(g)) * kPiD / 180, psi = (k % 3) * 5 * kPiD / 180, c = k % 2 ? 2000 : 500;
    MaterialParams m{};
    m.type = 1, m.density = m.grain_density = 1800, m.E = 1e7, m.nu = .3;
    m.bulk = m.E / (3 * (1 - 2 * m.nu)), m.shear = m.E / (2 * (1 + m.nu));
    m.a1 = m.bulk + 4. / 3 * m.shear, m.a2 = m.bulk - 2. / 3 * m.shear;
    m.phi_peak = m.phi_res = phi, m.psi_peak = m.psi_res = psi, m.c_peak = m.c_res = c;
    m.tension_cutoff = k % 5 ? 0 : 1e4;
    m.tc_init = check_low(std::min(m.tension_cutoff, c / tan(phi)));
    m.softening = k % 7 == 0;
    if (m.softening) m.pd_peak = 1e-4, m.pd_res = 1e-2, m.c_res = .5 * c, m.phi_res = .8 * phi;
    m.sin_phi = sin(phi), m.cos_phi = cos(phi), m.tan_phi = tan(phi), m.tan_psi = tan(psi);
    friction_quotients(m.sin_phi, m.cos_phi, m.ic_phi, m.e_phi, m.n_phi);
    double s[6], de[6], sv[SV_N] = {0, phi, psi, c, m.tc_init, 0, 0, 0, m.softening ? 5e-3 * U(g) : 0};
    const double p = (k % 4 ? -8000 : 1000) * U(g);
    for (int i = 0; i < 6; ++i) s[i] = (i < 3 ? p : 0) + 1500 * n(g) * (i < 3 ? 1 : .6), de[i] = 3e-4 * n(g);
    if (k % 17 == 0)  // a triaxial corner, exactly
      for (int i = 0; i < 6; ++i) s[i] = i < 2 ? .43 * p : (i == 2 ? p : 0);

    // single evaluations against 80 bits, away from the corners (where dtheta/dsigma has no limit): j2 and j3
    // carry the rounding of stresses of size |s|, e = u |s| / sqrt(j2) each relative to itself; cos 3 theta then
    // 3 e, its sine's square q another 6 e / q
    const Eval want = evaluate<long double>(m, s, sv), rec = evaluate_reciprocal(m, s, sv), wri = evaluate<double>(m, s, sv);
    const double q = std::pow(sin(3 * want.theta), 2), j2 = mu_j2(s);
    if (q > 1e-4 && j2 > 0 && rec.yt == want.yt) {
      double smax = 0;
      for (int i = 0; i < 6; ++i) smax = std::max(smax, fabs(s[i]));
      const double cond = u * (1 + smax / sqrt(j2)) * (1 + 1 / q);
      ++evals[want.yt];
      w_yf = std::max(w_yf, std::max(fabs(rec.yf[0] - want.yf[0]), fabs(rec.yf[1] - want.yf[1])) / (cond * (sqrt(j2) + smax + c)));
      w_df = std::max(w_df, off(rec.df, want.df, 6) / cond);
      w_dp = std::max(w_dp, off(rec.dp, want.dp, 6) / cond);
      w_dq = std::max(w_dq, off(&rec.dq, &want.dq, 1) / cond);
      w_theta = std::max(w_theta, off(&rec.theta, &want.theta, 1) / cond);
      if (want.soft != 0) {  // a sum of terms of opposite sign: relative to their sizes
        const double dphi = (m.phi_peak - m.phi_res) / (m.pd_res - m.pd_peak), dc = (m.c_peak - m.c_res) / (m.pd_res - m.pd_peak);
        const double size = want.dq * (dc + dphi * (sqrt(j2) + smax) / std::pow(cos(phi), 2));
        ++soft_evals, w_soft = std::max(w_soft, fabs(rec.soft - want.soft) / (cond * size));
      }
    }
    bool same = true;
    for (int i = 0; i < 6; ++i) same = same && rec.df[i] == wri.df[i];
    same_bits += same;

    // whole updates, form against form
    const Return a = update(m, s, de, sv), b = update_reciprocal(m, s, de, sv);
    ++returns;
    bool fin = true;
    for (int i = 0; i < 6; ++i) fin = fin && std::isfinite(a.out[i]) == std::isfinite(b.out[i]);
    finite += fin;
    counts += a.itr == b.itr, yields += a.yield == b.yield, corrections += a.itr;
    shear += a.yield == 1, tensile += a.yield == 2;
    if (a.itr == b.itr && a.itr < 100 && fin) d_out.push_back(off(b.out, a.out, 6));
    if (b.itr < 100 && b.yield) {
      const Eval e = evaluate<long double>(m, b.out, b.sv);
      off_surface += !(e.yf[0] < 0.1001 && e.yf[1] < 0.1001);
    }
  }
  std::sort(d_out.begin(), d_out.end());
  const size_t nd = d_out.size();
  std::printf("evals %d %d %d %d\n", evals[0], evals[1], evals[2], soft_evals);
  std::printf("eval_errors %.3g %.3g %.3g %.3g %.3g %.3g\n", w_yf, w_df, w_dp, w_dq, w_soft, w_theta);
  std::printf("same_bits %d\n", same_bits);
  std::printf("returns %d %d %d %d %d %d %d %d\n", returns, finite, counts, yields, corrections, shear, tensile, off_surface);
  std::printf("stress %.3g %.3g %.3g %.3g\n", d_out[nd / 2], d_out[nd * 99 / 100], d_out[nd * 999 / 1000], d_out[nd - 1]);
}
#endif
