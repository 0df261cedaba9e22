// Per-step kernels of the DEM step: the first-half kernel (the previous
// step's second half kick, boundary rule, half kick + drift), the pair/wall
// force gather, the end-of-step bookkeeping and the closing second half kick.
//
// This translation unit is compiled with -fmad=false: in parity mode every
// double operation rounds exactly as the oracle's (-ffp-contract=off), so
// positions after the first half, cutoff decisions, normals and relative
// velocities are bit-identical to the reference algorithm evaluated in FP64 from
// the same state. Force magnitudes differ only where a transcendental is
// evaluated differently (delta^1.5 as delta*sqrt(delta)), well inside 1e-9
// relative. Physical mode has no such counterpart: its FP64 pair law is written
// with fused multiply-adds (pair_contact_fused).
//
// Precision forms of the pair force (StepParams::prec):
//   FP64  — all pair math in double.
//   MIXED — the cutoff decision, r_sum^2 - d^2 (the overlap without
//           cancellation) and v_i - v_j stay in double; normals, relative
//           velocity, force laws and torques run in float; the per-particle
//           force/torque sums, the state and the integrator stay in double.
#include <cfloat>

#include "rp_arith.cuh"
#include "rp_device.cuh"
#include "rp_launch.h"
#include "rp_mlp.cuh"

namespace rp {

__device__ __forceinline__ V xyz(const D4& d) { return V{d.x, d.y, d.z}; }

// The law's constants in the pair law's precision (the FP32 ones come rounded),
// with the products that every contact of a group would form again: (4/3) E*,
// 2 E* and 1.5 pi gamma, each rounded as the laws' own left-to-right product.
// With the reduced mass formed only by the laws that damp with it and the
// quotients below in the wall contact: 1,636,935 adhesive spheres in 96 boxes 887
// to 855 us a step, 23,457 in one 33.0 to 31.8, 4.2 million Hertz spheres in
// mixed precision 1391 to 1354.
template <typename R> __device__ __forceinline__ R law_mu(const Law& L) { return sizeof(R) == 4 ? (R)L.muf : (R)L.mu; }
template <typename R> __device__ __forceinline__ R law_gs(const Law& L) { return sizeof(R) == 4 ? (R)L.gs_ppf : (R)L.gs_pp; }
template <typename R>
struct NormalLaw {
  R es, es43, es2, gamma, pull, beta;
};
template <typename R>
__device__ __forceinline__ NormalLaw<R> pair_law(const Law& L) {
  if (sizeof(R) == 4)
    return NormalLaw<R>{(R)L.es_ppf, (R)L.es43_ppf, (R)L.es2_ppf, (R)L.gamma_ppf, (R)L.pull_ppf, (R)L.beta_absf};
  return NormalLaw<R>{(R)L.es_pp, (R)L.es43_pp, (R)L.es2_pp, (R)L.gamma_pp, (R)L.pull_pp, (R)L.beta_abs};
}
__device__ __forceinline__ NormalLaw<double> wall_law(const Law& L) {
  return NormalLaw<double>{L.es_pw, L.es43_pw, L.es2_pw, L.gamma_pw, L.pull_pw, L.beta_abs};
}

// ------------------------------------------------------------- force laws
// src/physics.rs:49-70
template <typename R>
__device__ __forceinline__ R lsd_mag(R overlap, R vn, R kn, R gn) {
  return relu(kn * overlap - gn * vn);
}
// src/physics.rs:86-129. With s = sqrt(R* delta): the elastic term
// (4/3) E* sqrt(R*) delta^1.5 = (4/3) E* s delta and the tangent stiffness
// 2 E* sqrt(R* delta) = 2 E* s share one square root.
template <typename R>
__device__ __forceinline__ R hertz_mag(const NormalLaw<R>& N, R overlap, R vn, R rs, R ms) {
  if (not_positive(overlap)) return R(0);
  R s = sqrt_rn(rs * overlap);
  R fe = N.es43 * s * overlap;
  R kt = N.es2 * s;
  R cn = sqrt_rn(ms * kt) * (R(2) * N.beta);  // == (2 sqrt) beta: doubling is exact
  R fd = -cn * vn;
  return relu(fe + fd);
}
template <typename R>
__device__ __forceinline__ R hertz_elastic_mag(R overlap, R es43, R rs) {
  if (not_positive(overlap)) return R(0);
  R kn = es43 * sqrt_rn(rs);
  return kn * (overlap * sqrt_rn(overlap));
}
// src/physics.rs:132-219 (Newton on a^2/R* - sqrt(C a) - delta = 0).
// `near` (FP32 callers) is set when a cut-off decision lies within rounding.
template <typename R>
__device__ __forceinline__ R jkr_mag(R overlap, R es, R rs, R gamma, bool* near = nullptr) {
  if (not_positive(gamma)) return hertz_elastic_mag(overlap, R(4.0 / 3.0) * es, rs);
  const R eight_pi = R(8) * R(kPi);
  R c_val = eight_pi * gamma / es;
  R sqrt_c = sqrt(c_val);
  R a = overlap > R(0) ? sqrt_rn(rs * overlap) : rs * R(0.5);
  for (int it = 0; it < 20; ++it) {
    if (not_positive(a)) a = R(1e-9);
    R ts = sqrt_rn(c_val * a);
    R f_val = div_rn(a * a, rs) - ts - overlap;
    R df = div_rn(R(2) * a, rs) - div_rn(R(0.5) * sqrt_c, sqrt_rn(a));
    if (less_nn(fabs(df), R(1e-9))) break;
    R da = div_rn(f_val, df);
    R max_step = a * R(0.5);
    R step = da;
    if (step < -max_step) step = -max_step;
    if (step > max_step) step = max_step;
    a = a - step;
    if (less_nn(fabs(step), R(1e-6) * rs)) break;
  }
  R ts = sqrt_rn(c_val * a);
  R f_val = div_rn(a * a, rs) - ts - overlap;
  if (near && fabs(fabs(f_val) - R(1e-3) * rs) <= R(1e-5) * rs) *near = true;
  if (fabs(f_val) > R(1e-3) * rs) return R(0);
  if (a <= R(0)) return R(0);
  R a3 = a * a * a;
  R term1 = div_rn(R(4) * es * a3, R(3) * rs);
  R term2 = sqrt_rn(eight_pi * gamma * es * a3);
  R fm = term1 - term2;
  R f_pull = R(-2.0 / 3.0) * R(kPi) * gamma * rs;
  if (near && fabs(fm - f_pull) <= R(1e-5) * (term1 + term2)) *near = true;
  if (fm < f_pull) return R(0);
  return fm;
}
// JKR magnitude of a particle pair without the reference's Newton loop, or
// JKR_FALLBACK when that loop must run (P.jkr_solver 1 or 2). The
// certificates (rp_mlp.cuh) either prove the reference returns zero or that
// its iteration converges to the root on the increasing branch; the root is
// then found in FP32 (solver 1: two Newton steps from the network's `guess`;
// solver 2, and pairs without a good guess: Newton from the reference's own
// start; `missed` marks the latter with solver 1, their steps not counted as
// the network's), accepted only when its
// FP64 residual is <= 1e-6 of the terms, corrected by one FP64-accurate Newton
// step, and turned into the reference's force 4 E* a^3/(3 R*) - sqrt(8 pi
// gamma E* a^3) = E* a (4 a^2/(3 R*) - sqrt(C a)). The pull-off cut is decided
// in FP64 and left to the reference's loop when within 1e-7 of the terms.
__device__ __forceinline__ int jkr_learned(const StepParams& P, const Law& L, double overlap, double rs, float guess,
                                           double& fm, uint32_t& iters, bool& missed) {
  missed = false;
  const float rsf = (float)rs;
  const float x = (float)overlap / rsf;
  const float c = L.jkr_Cf / rsf;
  const float c23 = jkr_c23(c);
  const int cls = jkr_certify(x, c, c23, overlap > 0.0);
  if (cls == JKR_ZERO) {
    fm = 0.0;
    return JKR_ZERO;
  }
  if (cls == JKR_WALK) {
    // the reference's halving walk, then its own tail (src/physics.rs:193-218),
    // operation for operation in FP64
    const double es = L.es_pp, gamma = L.gamma_pp;
    const double eight_pi = 8.0 * kPi;
    const double c_val = L.jkr_C;  // 8 pi gamma / E*
    double a = sqrt_rn(rs * overlap);
    const double lim = 1e-6 * rs;
    // a / 2^k with the first k in 1..20 that takes it below lim, from the
    // exponents and mantissas (both are positive and normal here); the loop
    // itself took up to 60 of the pass's FP64 instructions
    const long long ab = __double_as_longlong(a), lb = __double_as_longlong(lim), M = 0x000FFFFFFFFFFFFFll;
    const int k = (int)(ab >> 52) - (int)(lb >> 52) + ((ab & M) < (lb & M) ? 0 : 1);
    a = __longlong_as_double(ab - ((long long)min(max(k, 1), 20) << 52));
    const double ts = sqrt_rn(c_val * a);
    const double f_val = div_rn(a * a, rs) - ts - overlap;
    fm = 0.0;
    if (fabs(f_val) > 1e-3 * rs || a <= 0.0) return JKR_WALK;
    const double a3 = a * a * a;
    const double term1 = div_rn(4.0 * es * a3, 3.0 * rs);
    const double term2 = sqrt_rn(eight_pi * gamma * es * a3);
    const double fmv = term1 - term2;
    const double f_pull = (-2.0 / 3.0) * kPi * gamma * rs;
    fm = fmv < f_pull ? 0.0 : fmv;
    return JKR_WALK;
  }
  if (cls != JKR_CONVERGES) return JKR_FALLBACK;
  float u;
  missed = P.jkr_solver == 1 && !(guess > 0.0f && guess < 1e30f);
  if (P.jkr_solver == 1 && !missed) {
    const float u1 = jkr_newton_f32(guess, x, c);
    u = jkr_newton_f32(u1, x, c);
    missed = !(fabsf(u - u1) <= 1e-3f * u);  // a prediction two quadratic steps do not make good
    if (!missed) iters += 2;
  }
  if (P.jkr_solver != 1 || missed) {
    u = overlap > 0.0 ? sqrtf(x) : 0.5f;
    for (int k = 0; k < 40; ++k) {
      const float un = jkr_newton_f32(u, x, c);
      if (!missed) ++iters;
      const bool done = fabsf(un - u) <= 1e-6f * un;
      u = un;
      if (done) break;
    }
  }
  // FP64 residual of a = u R*: sqrt(C a) from the FP32 root plus one Newton
  // step of the square root (error ~1e-14), no FP64 division
  const double ud = (double)u;
  const double Ca = L.jkr_C * (ud * rs);
  const float s0 = sqrtf((float)Ca);
  if (!(s0 > 0.0f)) return JKR_FALLBACK;
  const double ts = (double)s0 + (Ca - (double)s0 * (double)s0) * (double)(0.5f / s0);
  const double uu = ud * ud * rs;  // a^2 / R*
  const double f = uu - ts - overlap;
  if (!(fabs(f) <= 1e-6 * (uu + ts + fabs(overlap)))) return JKR_FALLBACK;
  const float dg = 2.0f * u - 0.5f * (float)ts / ((float)ud * rsf);
  if (!(dg > 0.0f)) return JKR_FALLBACK;
  const float du = (float)f / (rsf * dg);
  const double u1 = ud - (double)du;
  const float q = du / u;
  const double ts1 = ts * (1.0 - (double)(0.5f * q + 0.125f * q * q));
  const double es = L.es_pp;
  const double a1 = u1 * rs;
  const double term1 = (4.0 / 3.0) * es * (u1 * u1 * u1) * (rs * rs);
  const double term2 = es * a1 * ts1;
  const double fmv = term1 - term2;
  const double f_pull = (-2.0 / 3.0) * kPi * L.gamma_pp * rs;
  if (fabs(fmv - f_pull) <= 1e-7 * (term1 + term2)) return JKR_FALLBACK;
  fm = fmv < f_pull ? 0.0 : fmv;
  return JKR_CONVERGES;
}

// src/physics.rs:234-325
template <typename R>
__device__ __forceinline__ R sjkr_mag(const NormalLaw<R>& N, R overlap, R vn, R rs) {
  if (not_positive(N.gamma)) return hertz_elastic_mag(overlap, N.es43, rs);
  R f_pull = N.pull * rs;
  if (!not_positive(-overlap)) {  // a gap: only one can lie beyond delta_c <= 0
    R term = R(3) * (R(kPi) * R(kPi)) * (N.gamma * N.gamma) * rs / (N.es * N.es);
    R delta_c = -sqrt(term);
    if (overlap < delta_c) return R(0);
  }
  R fh = not_positive(overlap) ? R(0) : N.es43 * sqrt_rn(rs) * (overlap * sqrt_rn(overlap));
  return vn > R(0) ? fh - f_pull : fh;
}

// Normal force magnitude for the configured model from the normal relative
// speed vn = rv . n and the masses (the FP32 form forms vn in FP64). The
// reference passes Vec3::ZERO as the relative velocity to the hysteretic
// particle-particle law (src/simulation.rs:409-411) and the real one for walls
// (:495-501). JKR has no damping and is the caller's.
template <typename R, bool WALL>
__device__ __forceinline__ R normal_mag(const NormalLaw<R>& N, int model, R overlap, T3<R> n, R vn, R rs, R ms) {
  switch (model) {
    case 1: return hertz_mag(N, overlap, vn, rs, ms);
    case 0: {
      R kn = N.es * rs;
      R gn = R(0.5) * sqrt_rn(ms * kn);
      return lsd_mag(overlap, vn, kn, gn);
    }
    case 2: return lsd_mag(overlap, WALL ? vn : dot(t3(R(0), R(0), R(0)), n), N.es * rs, R(0));
    default: return sjkr_mag(N, overlap, vn, rs);
  }
}
// m_i m_j / (m_i + m_j) for the laws with damping
template <typename R>
__device__ __forceinline__ R reduced_mass(int model, double mi, double mj) {
  if (model > 1) return R(0);
  const R a = narrow<R>(mi), b = narrow<R>(mj);
  return div_rn(a * b, a + b);
}

// src/physics.rs:385-397 (direction by one reciprocal square root)
template <typename R>
__device__ __forceinline__ T3<R> coulomb_force(R fn, T3<R> rv, T3<R> n, R mu) {
  T3<R> vt = rv - dot(rv, n) * n;
  const R vt2 = dot(vt, vt);
  if (less_nn(vt2, R(1e-8))) return t3(R(0), R(0), R(0));
  R inv = rsqrt(vt2);
  T3<R> dir = vt * inv;
  return (-mu * fn) * dir;
}
// Coulomb from a given tangential relative velocity vt = rv - (rv . n) n.
template <typename R>
__device__ __forceinline__ T3<R> coulomb_force_vt(R fn, T3<R> vt, R mu) {
  const R vt2 = dot(vt, vt);
  if (vt2 < R(1e-8)) return t3(R(0), R(0), R(0));
  return (-mu * fn) * (vt * rsqrt(vt2));
}
// src/physics.rs:400-434 with the spring `xi` in registers.
template <typename R>
__device__ __forceinline__ T3<R> spring_coulomb_vt(R fn, T3<R> vt, T3<R>& xi, R kt, R mu, R dt) {
  xi = xi + vt * dt;
  T3<R> trial = (-kt) * xi;
  R tm = len(trial);
  R fc = mu * fn;
  if (tm > fc) {
    T3<R> dir = tm > R(1e-6) ? trial / tm : t3(R(0), R(0), R(0));
    T3<R> ft = fc * dir;
    xi = (-ft) / kt;
    return ft;
  }
  return trial;
}
template <typename R>
__device__ __forceinline__ T3<R> spring_coulomb(R fn, T3<R> rv, T3<R> n, T3<R>& xi, R kt, R mu, R dt) {
  return spring_coulomb_vt(fn, rv - dot(rv, n) * n, xi, kt, mu, dt);
}

// One contact seen from particle i (src/simulation.rs:358-460), for a pair
// that passed the cutoff test. Inputs in FP64; the law arithmetic in R.
// Writes the contact force on i and its torque r_a x f in FP64 and returns
// true. In FP32 it returns false, touching nothing, when a discontinuous
// decision of the reference's laws (Coulomb's |v_t|^2 < 1e-8, sJKR's
// loading/unloading sign and detachment, JKR's cut-offs) or an sJKR
// near-cancellation lies within FP32 rounding: the caller then evaluates the
// pair in FP64, so both forms take the same branches.
// L holds the material constants of the pair's group. With P.jkr_solver != 0
// the JKR magnitude comes from jkr_learned (`guess` is the network's a/R*, or
// negative / NaN for none; `tally` counts accepted / zero / fallback / walk
// and FP32 Newton steps when not null). A pair that needs the reference's
// Newton iteration sets *deferred and returns at once, touching nothing, when
// `deferred` is given; `newton` forces the reference's iteration.
// JKR: the law is JKR's (a kernel of its own; the others hold fewer registers).
template <typename R, bool PHYS, bool HIST, bool JKR>
__device__ __forceinline__ bool pair_contact(const StepParams& P, const Law& L, V d, double d2, double rsum, double ri,
                                             double rj, double mi, double mj, V vi, V vj, V wi, V wj, double* hist,
                                             size_t plane, T3<R>& fc_out, T3<R>& tc_out, T3<R>& n_out,
                                             bool& excess,
                                             float guess = -1.0f, uint32_t* tally = nullptr,
                                             bool* deferred = nullptr, bool newton = false) {
  constexpr bool F32 = sizeof(R) == sizeof(float);
  R overlap;
  T3<R> n;
  V nd;         // the unit normal in FP64 (FP32 form: to ~1e-14, for the relative velocity below)
  double ovd;   // the overlap in FP64 (FP32 form: to ~1e-14 of r_sum)
  if (sizeof(R) == sizeof(double)) {
    double inv;
    const double dist = sqrt_rn(d2, inv);
    overlap = (R)(rsum - dist);
    ovd = (double)overlap;
    const V nd = less_nn(1e-6, dist) ? d * inv : vmk(0.0, 1.0, 0.0);
    n = cvt<R>(nd);
  } else {
    bool far_enough;
    if (less_nn(1.001e-12, d2)) far_enough = true;
    else if (d2 < 0.999e-12) far_enough = false;
    else far_enough = sqrt(d2) > 1e-6;  // exact FP64 decision near the threshold
    if (far_enough) {
      // 1/|d| from the FP32 reciprocal square root and one FP64 Newton step
      // (relative error ~1e-14, no FP64 square root or division); |d| is
      // d^2 times it. The overlap is then good to ~1e-14 of r_sum: the JKR
      // contact radius next to its fold and the damping of a grazing contact
      // are sensitive to it.
      // (r0 is a normal float: widened by its bits; d2 / 2 by its exponent)
      const uint32_t rb = __float_as_uint(rsqrtf(d2f_exact(d2)));
      const double r0 = rb ? __hiloint2double((int)((rb >> 3) + 0x38000000u), (int)(rb << 29)) : 0.0;
      const double half = __hiloint2double(__double2hiint(d2) - 0x00100000, __double2loint(d2));
      const double inv = r0 * (1.5 - half * (r0 * r0));
      ovd = rsum - d2 * inv;
      nd = d * inv;
      n = narrow<R>(nd);
    } else {
      ovd = rsum - sqrt(d2);
      nd = vmk(0.0, 1.0, 0.0);
      n = t3(R(0), R(1), R(0));
    }
    overlap = narrow<R>(ovd);
  }
  const R rir = narrow<R>(ri), rjr = narrow<R>(rj);
  if (is_excess(overlap, rir, rjr)) excess = true;
  const T3<R> ra = (-n) * rir;
  const T3<R> rb = n * rjr;
  T3<R> rv = ra, vt;  // rv: FP64 form only
  V rvd = vi;         // rv in FP64 (FP32 form)
  R vn;
  if (sizeof(R) == sizeof(double)) {
    const T3<R> va = cvt<R>(vi) + cross(cvt<R>(wi), ra);
    const T3<R> vb = cvt<R>(vj) + cross(cvt<R>(wj), rb);
    rv = va - vb;
    vn = dot(rv, n);
    vt = rv - vn * n;
  } else {
    // In a rolling or sticking contact, and along the normal, the relative
    // velocity at the contact point is a small difference of large terms
    // (the spin terms w x r): rounded in FP32 they would swamp the normal
    // speed of the damping and the slip direction of the friction. So it is
    // formed in FP64, as (v_i - v_j) - (w_i r_i + w_j r_j) x n (the same
    // quantity as va - vb with r_a = -n r_i, r_b = n r_j), and only then
    // rounded for the FP32 laws.
    // Its normal part (the damping's speed) and tangential part (the slip)
    // are split in FP64 too: in a sliding contact the normal speed is a
    // small remainder of |rv|, in a head-on one the slip is.
    const V W = wi * ri + wj * rj;
    rvd = (vi - vj) - cross(W, nd);
    const double vnd = dot(rvd, nd);
    vn = narrow<R>(vnd);
    vt = narrow<R>(rvd - vnd * nd);
  }
  const R rs = div_rn(rir * rjr, rir + rjr);
  const NormalLaw<R> N = pair_law<R>(L);
  R fmag;
  int jkind = JKR_FALLBACK;
  if (JKR && P.jkr_solver != 0 && !newton && L.gamma_pp > 0.0) {
    double fmd = 0.0;
    uint32_t it = 0;
    bool missed;
    jkind = jkr_learned(P, L, ovd, (double)rs, guess, fmd, it, missed);
    if (jkind != JKR_FALLBACK) fmag = (R)fmd;
    if (tally) {
      tally[jkind == JKR_CONVERGES ? (missed ? 2 : 0) : (jkind == JKR_ZERO ? 1 : (jkind == JKR_WALK ? 5 : 2))] += 1;
      tally[4] += it;
    }
    if (jkind == JKR_FALLBACK && deferred) {
      *deferred = true;
      return true;
    }
  }
  if (jkind != JKR_FALLBACK) {
  } else if (JKR && !F32) {
    fmag = jkr_mag<R>(overlap, N.es, rs, N.gamma);
  } else if (JKR) {
    // The contact radius has a square-root fold next to the pull-off: there
    // the FP32 iteration cannot resolve the root (an FP32 residual moves it by
    // ~sqrt(1e-7) relative) and the pair is evaluated in FP64. Elsewhere the
    // certificates bound the slope away from zero.
    if (L.gamma_pp > 0.0) {
      const float x = (float)overlap / (float)rs, c = L.jkr_Cf / (float)rs;
      if (jkr_certify(x, c, jkr_c23(c), overlap > R(0)) == JKR_FALLBACK) return false;
    }
    bool near = false;
    fmag = jkr_mag<R>(overlap, N.es, rs, N.gamma, &near);
    if (near) return false;
  } else {
    fmag = normal_mag<R, false>(N, P.nmodel, overlap, n, vn, rs, reduced_mass<R>(P.nmodel, mi, mj));
  }
  if (F32 && !JKR && P.nmodel == 4 && N.gamma > R(0)) {
    const R gamma = N.gamma, es = N.es;
    const R f_pull = N.pull * rs;
    const R delta_c = -sqrt(R(3) * (R(kPi) * R(kPi)) * (gamma * gamma) * rs / (es * es));
    if (fabs(vn) <= R(1e-6) * (len(cvt<R>(rvd)) + R(1e-30))) return false;
    if (fabs(overlap - delta_c) <= R(1e-5) * fabs(delta_c)) return false;
    if (vn > R(0) && fabs(fmag) <= R(0.05) * f_pull) return false;
  }
  // |f n| = |f| for the unit normal (the reference takes the vector length)
  const T3<R> fnv = fmag * n;
  const R fnm = fabs(fmag);
  T3<R> ft;
  bool ft_zero = false;  // ft is +0: F = fn + 0 without the additions
  if (P.tmodel == 0) {
    if (F32) {
      const R vt2 = dot(vt, vt);
      if (fabs(vt2 - R(1e-8)) <= R(1e-5) * (vt2 + R(1e-8))) return false;
      ft = coulomb_force_vt<R>(fnm, vt, law_mu<R>(L));
    } else {
      ft = coulomb_force<R>(fnm, rv, n, law_mu<R>(L));
    }
  } else if (!PHYS) {
    // G* = 0 in parity mode (src/material.rs:39-50): the spring force is
    // 0 * (...), +-0, or NaN when Mindlin's sqrt(R* delta) is NaN or infinite
    // (a negative overlap); decided without the square root. With +0 for
    // the spring, F = fn + 0 is fn with -0 made +0.
    const R y = P.tmodel == 2 ? rs * overlap : rs;
    const R big = sizeof(R) == sizeof(float) ? R(FLT_MAX) : R(DBL_MAX);
    const bool finite = P.tmodel == 2 ? (y >= R(0) && y <= big) : (fabs(y) <= big);
    if (finite) {
      ft_zero = true;
      ft = t3(R(0), R(0), R(0));
    } else {
      const R nan = sizeof(R) == sizeof(float) ? (R)__int_as_float(0x7fc00000)
                                               : (R)__longlong_as_double(0x7ff8000000000000ll);
      ft = t3(nan, nan, nan);
    }
  } else {
    T3<R> xi_s = t3(R(0), R(0), R(0));
    if (overlap > R(0)) {
      R kt = P.tmodel == 2 ? R(8) * law_gs<R>(L) * sqrt(rs * overlap) : law_gs<R>(L) * rs;
      if (HIST) xi_s = t3((R)hist[0], (R)hist[plane], (R)hist[2 * plane]);
      xi_s = xi_s - dot(xi_s, n) * n;
      ft = F32 ? spring_coulomb_vt<R>(fnm, vt, xi_s, kt, law_mu<R>(L), (R)P.dt)
               : spring_coulomb<R>(fnm, rv, n, xi_s, kt, law_mu<R>(L), (R)P.dt);
    } else {
      ft = t3(R(0), R(0), R(0));
    }
    if (HIST) {
      hist[0] = (double)xi_s.x;
      hist[plane] = (double)xi_s.y;
      hist[2 * plane] = (double)xi_s.z;
    }
  }
  const T3<R> fc = ft_zero ? t3(plus_zero(fnv.x), plus_zero(fnv.y), plus_zero(fnv.z)) : fnv + ft;
  const T3<R> tc = cross(ra, fc);
  fc_out = fc;
  tc_out = tc;
  n_out = n;
  return true;
}

// Normal force magnitude of a particle pair in physical mode in FP64, with
// fused multiply-adds and shared roots (the laws of src/physics.rs:49-129,
// 234-325). JKR goes to jkr_mag or jkr_learned.
__device__ __forceinline__ double normal_mag_fused(int model, const Law& L, double overlap, double vn, double rs,
                                                   double mi, double mj) {
  const double es = L.es_pp;
  if (model == 1) {
    // (4/3) E* s delta = (2/3) k_t delta with k_t = 2 E* s, s = sqrt(R* delta)
    if (overlap <= 0.0) return 0.0;
    const double ms = div_near(mi * mj, mi + mj);
    const double kt = (2.0 * es) * sqrt_rn(rs * overlap);
    const double cn = sqrt_rn(ms * kt) * (2.0 * L.beta_abs);
    return relu(fma(-cn, vn, (kt * overlap) * (2.0 / 3.0)));
  }
  if (model == 0) {
    const double ms = div_near(mi * mj, mi + mj);
    const double kn = es * rs;
    return relu(fma(kn, overlap, -(0.5 * sqrt_rn(ms * kn)) * vn));
  }
  if (model == 2) return relu((es * rs) * overlap);  // the pair law sees no relative velocity
  // sJKR; without surface energy the elastic Hertz law
  const double fh = overlap > 0.0 ? ((4.0 / 3.0) * es * sqrt_rn(rs * overlap)) * overlap : 0.0;
  const double gamma = L.gamma_pp;
  if (gamma <= 0.0) return fh;
  if (overlap < 0.0) {  // delta_c <= 0: only a gap can lie beyond it
    const double term = 3.0 * (kPi * kPi) * (gamma * gamma) * rs / (es * es);
    if (overlap < -sqrt(term)) return 0.0;
  }
  return vn > 0.0 ? fma(-(1.5 * kPi * gamma), rs, fh) : fh;
}

// pair_contact for physical mode in FP64: the same contact with fused
// multiply-adds and only the parts that the configured laws use. Parity mode
// repeats the reference's roundings operation by operation (a dense bed with
// Coulomb friction chatters, and any other rounding grows tenfold every three
// steps); physical mode has no such counterpart, and each operation here rounds
// once where the separate form rounds twice. Both are bound by the FP64 pipe
// whatever a warp's lanes do, so what counts is FP64 instructions a contact.
// The cutoff decision is the caller's and stays unfused. On a 163,843-sphere
// bed with linear springs the pair kernel went from 62.7 to 43.8 million FP64
// thread instructions and from 210 to 130 us.
//   nf = n x f, from which the caller forms both torques: -r_i (n x f) on i
// and, the other end's force being -f, -r_j (n x f) on j; the normal force
// adds nothing to it.
// Springs, `deferred` and `newton` as in pair_contact.
template <bool HIST, bool JKR>
__device__ __forceinline__ void pair_contact_fused(const StepParams& P, const Law& L, V d, double d2, double rsum,
                                                   double ri, double rj, double mi, double mj, V vi, V vj, V wi, V wj,
                                                   double* hist, size_t plane, V& f_out, V& nf_out, bool& excess,
                                                   float guess = -1.0f, uint32_t* tally = nullptr,
                                                   bool* deferred = nullptr, bool newton = false) {
  V n;
  double overlap;
  if (d2 > 1.001e-12) {
    double inv;
    overlap = rsum - sqrt_rn(d2, inv);
    n = d * inv;
  } else {  // next to the reference's |d| > 1e-6 decision, which it takes on the rounded root
    const double dist = sqrt(d2);
    overlap = rsum - dist;
    n = dist > 1e-6 ? d * (1.0 / dist) : vmk(0.0, 1.0, 0.0);
  }
  if (is_excess(overlap, ri, rj)) excess = true;
  // (v_i - v_j) - (w_i r_i + w_j r_j) x n
  const V W = mad(rj, wj, wi * ri);
  const V u = vi - vj;
  const V rv = vmk(fma(n.y, W.z, fma(-W.y, n.z, u.x)), fma(n.z, W.x, fma(-W.z, n.x, u.y)),
                   fma(n.x, W.y, fma(-W.x, n.y, u.z)));
  const double vn = dot_fma(rv, n);
  const V vt = mad(-vn, n, rv);
  const double rs = div_near(ri * rj, rsum);
  double fm = 0.0;
  if (JKR) {
    int kind = JKR_FALLBACK;
    if (P.jkr_solver != 0 && !newton && L.gamma_pp > 0.0) {
      uint32_t it = 0;
      bool missed;
      kind = jkr_learned(P, L, overlap, rs, guess, fm, it, missed);
      if (tally) {
        tally[kind == JKR_CONVERGES ? (missed ? 2 : 0) : (kind == JKR_ZERO ? 1 : (kind == JKR_WALK ? 5 : 2))] += 1;
        tally[4] += it;
      }
      if (kind == JKR_FALLBACK && deferred) {
        *deferred = true;
        return;
      }
    }
    if (kind == JKR_FALLBACK) fm = jkr_mag<double>(overlap, L.es_pp, rs, L.gamma_pp);
  } else {
    fm = normal_mag_fused(P.nmodel, L, overlap, vn, rs, mi, mj);
  }
  V f = fm * n, nf = vmk(0.0, 0.0, 0.0);
  if (P.tmodel == 0) {
    const double vt2 = dot_fma(vt, vt);
    if (!(vt2 < 1e-8)) {
      const double g = (-L.mu * fabs(fm)) * rsqrt(vt2);
      nf = g * cross_fma(n, vt);
      f = mad(g, vt, f);
    }
  } else {
    V xi = vmk(0.0, 0.0, 0.0);
    if (overlap > 0.0) {
      const double kt = P.tmodel == 2 ? (8.0 * L.gs_pp) * sqrt_rn(rs * overlap) : L.gs_pp * rs;
      if (HIST) xi = vmk(hist[0], hist[plane], hist[2 * plane]);
      xi = mad(P.dt, vt, mad(-dot_fma(xi, n), n, xi));
      const V trial = (-kt) * xi;
      const double t2 = dot_fma(trial, trial), fc = L.mu * fabs(fm);
      V ft = trial;
      if (t2 > fc * fc) {
        ft = t2 > 1e-12 ? (fc * rsqrt(t2)) * trial : vmk(0.0, 0.0, 0.0);
        xi = (-div_near(1.0, kt)) * ft;
      }
      nf = cross_fma(n, ft);
      f = f + ft;
    }
    if (HIST) {
      hist[0] = xi.x;
      hist[plane] = xi.y;
      hist[2 * plane] = xi.z;
    }
  }
  f_out = vmk(plus_zero(f.x), plus_zero(f.y), plus_zero(f.z));
  nf_out = nf;
}

// Kahan-compensated s += d with residual r (src/particle.rs:12-18 and the
// reference's integrator): y = d - r, t = s + y, r = (t - s) - y, s = t.
__device__ __forceinline__ void kahan_add(V& s, V& r, V d) {
  const V y = d - r;
  const V t = s + y;
  r = (t - s) - y;
  s = t;
}

// Second half of velocity Verlet for one particle (src/simulation.rs:541-561):
// Kahan-compensated v += a dt/2 and omega += (tau/I) dt/2, I = 0.4 m r^2
// (tau/I as tau * (1/I), 1/I stored per particle in Bank::wres[k].w when the
// state is uploaded; v and x are unchanged).
__device__ __forceinline__ void second_half_kick(V& v, V& vres, V& w, V& wres, V a, V tau, double inv_inertia,
                                                 double hdt) {
  // (0.5 a) dt == a (0.5 dt), both one rounding of a dt / 2
  V dv = a * hdt;
  V yv = dv - vres;
  V tv = v + yv;
  vres = (tv - v) - yv;
  v = tv;
  V aa = tau * inv_inertia;
  V dw = aa * hdt;
  V yw = dw - wres;
  V tw = w + yw;
  wres = (tw - w) - yw;
  w = tw;
}

// A thread's items of a pass: at, at + all, at + 2 all, ... (the lanes of a warp
// next to each other).
struct Span {
  int at, all;
};
__device__ __forceinline__ Span grid_span() {
  return Span{(int)(blockIdx.x * blockDim.x + threadIdx.x), (int)(gridDim.x * blockDim.x)};
}

// ------------------------------------------------------------- first half
// The force kernel only writes a and tau: neighbours read v and omega while
// it runs, so the second half kick of step n-1 is applied here, at the start
// of step n (when Ctrl::pending says a step owes it), and by k_second_half at
// the end of a stepping call. Then src/simulation.rs:176-263: periodic wrap,
// out-of-bounds removal (marked dead here and compacted by the host later;
// removal changes no other particle's update), Kahan-compensated half kick +
// drift + angular half kick. Also records the reference-grid cell code and
// requests a list rebuild when a particle moved more than half the skin since
// the last build.
//
// KAHAN = false is the mixed form's integrator: the same velocity-Verlet
// halves in plain FP64 (v += a dt/2, x += v dt, omega += (tau/I) dt/2), with
// the reference's Kahan residuals neither read nor updated. From zero
// residuals one step gives the same bits as the compensated form; over many
// steps positions and velocities differ from it by FP64 rounding (about one
// ulp per step), far below the FP32 pair forces' 1e-5. With the previous
// step's second half kick pending, the two half kicks are one kick of a dt.
// It takes ~45 of the ~85 FP64-pipe instructions per particle and 128 of the
// 484 bytes (the residuals' read and three writes) off this kernel.
// (Called by a whole grid, each thread for its items of the span; returns
// whether one of the thread's particles asks for a rebuild.)
// SPIN = false leaves the spin's kicks to the contact filter (spin_kick).
template <bool KAHAN, bool SPIN>
__device__ __forceinline__ bool first_half_pass(const StepParams& P, Ctrl* C, const Bank& B, bool FUSE, Span sp) {
  const double dt = P.dt;
  const bool anyp = P.periodic[0] | P.periodic[1] | P.periodic[2];
  // (0.5 a) dt and a (0.5 dt) are the same correctly rounded product; the
  // launch's constants come converted (each conversion or product here would be
  // an FP64-pipe instruction of every warp: 7 of the mixed form's 40)
  const double hdt = P.hdt;
  const float half_skin = P.half_skinf, inv_hf = P.inv_hreff;
  const unsigned xmax = C->xmax;
  bool want_rebuild = false;
  for (int k = sp.at; k < P.n; k += sp.all) {
    uint32_t fl = B.flags[k];
    if (fl & PF_DEAD) continue;
    D4 xr = B.xr[k], vm = B.vm[k], wc;
    if (SPIN) wc = B.wc[k];
    else wc.w = B.wc[k].w;
    V x = xyz(xr), v = xyz(vm), w = SPIN ? xyz(wc) : x;
    const bool moving = !(fl & PF_FIXED);
    V vres = vmk(0.0, 0.0, 0.0), wres = vres, xres = vres, dv = vres, dw = vres;
    double inv_inertia = 0.0, inv_mass = 0.0;
    bool spin = false, own_spin = false;
    if (moving) {
      // the fused second half of the previous step and this step's first
      // half kick with the same a and tau: the increments are computed once
      const V a = xyz(B.acc[k]);
      V tau = vres;
      if (SPIN) {
        tau = xyz(B.tq[k]);
        const D4 wr4 = B.wres[k];
        inv_inertia = wr4.w;
        if (KAHAN) wres = xyz(wr4);
      }
      if (KAHAN) {
        const D4 vr4 = B.vres[k];
        inv_mass = vr4.w;
        vres = xyz(vr4);
        xres = xyz(B.xres[k]);
      }
      // the mixed form joins the pending second half kick and this step's
      // first half kick into one kick of a dt
      const double kdt = (!KAHAN && FUSE) ? dt : hdt;
      dv = a * kdt;
      // without a torque and a residual (a particle in flight) the spin keeps
      // its value, adding zeros to it: two of the seven 32-byte stores fall
      // away and, where that holds for a whole warp, 30 of the ~90 FP64
      // instructions (decided by the warp: lanes going apart cost more)
      if (SPIN) {
        own_spin = some_bits(tau) || (KAHAN && some_bits(wres)) || (fl & PF_KICK);
        spin = __any_sync(__activemask(), own_spin);
      }
      if (spin) dw = KAHAN ? (tau * inv_inertia) * kdt : tau * (inv_inertia * kdt);
      if (KAHAN && FUSE) {
        kahan_add(v, vres, dv);
        if (spin) kahan_add(w, wres, dw);
      }
    }
    // the FP32 mirror of x (written with it) decides most wrap and removal
    // tests without the FP64 comparisons: inside the inner interval of an
    // axis, x needs no wrap (periodic) or is kept (open)
    const float4 xo = B.xf[k];
    const bool in0 = xo.x > P.inner_lo[0] && xo.x < P.inner_hi[0];
    const bool in1 = xo.y > P.inner_lo[1] && xo.y < P.inner_hi[1];
    const bool in2 = xo.z > P.inner_lo[2] && xo.z < P.inner_hi[2];
    if (anyp) {
      if (P.periodic[0] && !in0) { if (x.x < P.bmin[0]) x.x = x.x + P.bsize[0]; else if (x.x >= P.bmax[0]) x.x = x.x - P.bsize[0]; }
      if (P.periodic[1] && !in1) { if (x.y < P.bmin[1]) x.y = x.y + P.bsize[1]; else if (x.y >= P.bmax[1]) x.y = x.y - P.bsize[1]; }
      if (P.periodic[2] && !in2) { if (x.z < P.bmin[2]) x.z = x.z + P.bsize[2]; else if (x.z >= P.bmax[2]) x.z = x.z - P.bsize[2]; }
    }
    bool keep = (P.periodic[0] || in0 || (x.x >= P.bmin[0] - 1.0 && x.x <= P.bmax[0] + 1.0)) &&
                (P.periodic[1] || in1 || (x.y >= P.bmin[1] - 1.0)) &&
                (P.periodic[2] || in2 || (x.z >= P.bmin[2] - 1.0 && x.z <= P.bmax[2] + 1.0));
    if (!keep) {
      B.flags[k] = fl | PF_DEAD;
      const double nan = __longlong_as_double(0x7ff8000000000000ll);
      xr.x = nan; xr.y = nan; xr.z = nan;
      B.xr[k] = xr;
      B.xf[k] = make_float4(__int_as_float(0x7fc00000), __int_as_float(0x7fc00000), __int_as_float(0x7fc00000),
                            (float)xr.w);
      atomicAdd(&C->removed, 1ull);
      continue;
    }
    if (moving) {
      if (KAHAN) {
        kahan_add(v, vres, dv);
        kahan_add(x, xres, v * dt);
        B.vres[k] = D4{vres.x, vres.y, vres.z, inv_mass};
        B.xres[k] = D4{xres.x, xres.y, xres.z, 0.0};
        if (spin) kahan_add(w, wres, dw);
        if (own_spin) B.wres[k] = D4{wres.x, wres.y, wres.z, inv_inertia};
      } else {
        v = v + dv;
        x = x + v * dt;
        if (spin) w = w + dw;
      }
      B.vm[k] = D4{v.x, v.y, v.z, vm.w};
      if (SPIN) { wc.x = w.x; wc.y = w.y; wc.z = w.z; }
    }
    const double code = wc.w;
    const float4 xf = make_float4(d2f_exact(x.x), d2f_exact(x.y), d2f_exact(x.z), xo.w);
    if (P.mode == 0) {
      const int32_t c0 = ref_axis_fast(x.x, xf.x, P.bmin[0], P.bminf[0], P.href, P.inv_href, inv_hf);
      const int32_t c1 = ref_axis_fast(x.y, xf.y, P.bmin[1], P.bminf[1], P.href, P.inv_href, inv_hf);
      const int32_t c2 = ref_axis_fast(x.z, xf.z, P.bmin[2], P.bminf[2], P.href, P.inv_href, inv_hf);
      wc.w = __longlong_as_double((long long)pack_code(c0, c1, c2));
    }
    if (SPIN) {
      if (own_spin || __double_as_longlong(code) != __double_as_longlong(wc.w)) B.wc[k] = wc;
    } else if (__double_as_longlong(code) != __double_as_longlong(wc.w)) {
      B.wc[k].w = wc.w;
    }
    B.xr[k] = D4{x.x, x.y, x.z, xr.w};
    B.xf[k] = xf;
    // the largest |coordinate| sets the filter's rounding margin (the bits of
    // non-negative floats order as the floats do; NaN stays out)
    const float far = fmaxf(fmaxf(fabsf(xf.x), fabsf(xf.y)), fabsf(xf.z));
    const unsigned lanes = __activemask(), top = __reduce_max_sync(lanes, far >= 0.0f ? __float_as_uint(far) : 0u);
    if (top > xmax && (threadIdx.x & 31) == __ffs(lanes) - 1) atomicMax(&C->xmax, top);
    float4 r0 = B.xref[k];
    float ddx = xf.x - r0.x, ddy = xf.y - r0.y, ddz = xf.z - r0.z;
    if (P.periodic[0]) ddx -= P.bsizef[0] * rintf(ddx / P.bsizef[0]);
    if (P.periodic[1]) ddy -= P.bsizef[1] * rintf(ddy / P.bsizef[1]);
    if (P.periodic[2]) ddz -= P.bsizef[2] * rintf(ddz / P.bsizef[2]);
    float d2 = ddx * ddx + ddy * ddy + ddz * ddz;
    if (!(d2 <= half_skin * half_skin)) want_rebuild = true;  // NaN (no build yet) also rebuilds
  }
  return want_rebuild;
}

template <bool KAHAN, bool SPIN>
__global__ void __launch_bounds__(KAHAN ? 128 : 256, KAHAN ? (SPIN ? 5 : 7) : 5) k_first_half(StepParams P) {
  Ctrl* C = P.ctrl;
  if (C->halt) return;
  if (first_half_pass<KAHAN, SPIN>(P, C, P.bank[C->bank], C->pending != 0, grid_span())) C->rebuild = 1;
  if (!SPIN && blockIdx.x == 0 && threadIdx.x == 0) C->spin_due = 1;
}

// The spin's part of the first half for slot k (with the previous step's second
// half kick when `fuse`): the operations of first_half_pass. Nothing before the
// pair kernel reads a spin, so in the device loop the contact filter does this:
// the integrator is bound by the FP64 pipe and the filter by gathers, with that
// pipe idle. Only x, y, z are written; other threads read the cell code in w.
// FP64 form only (us a step with / without: hopper 1 M 687 / 716, gas 1 M 270 /
// 305, boxes 1.6 M 907 / 945): the mixed form's spin is 9 FP64 instructions, not
// 30, and the filter's extra traffic costs more (drum 4.2 M 1499 / 1450).
__device__ __forceinline__ void spin_kick(const StepParams& P, const Bank& B, int k, uint32_t fl, bool fuse) {
  const D4 wr4 = B.wres[k];
  const V tau = xyz(B.tq[k]);
  V wres = xyz(wr4);
  if (!(some_bits(tau) || some_bits(wres) || (fl & PF_KICK))) return;
  double* at = &B.wc[k].x;
  const double2 w0 = *reinterpret_cast<const double2*>(at);
  V w = vmk(w0.x, w0.y, at[2]);
  const V dw = (tau * wr4.w) * P.hdt;
  if (fuse) kahan_add(w, wres, dw);
  kahan_add(w, wres, dw);
  B.wres[k] = D4{wres.x, wres.y, wres.z, wr4.w};
  *reinterpret_cast<double2*>(at) = make_double2(w.x, w.y);
  at[2] = w.z;
}
bool spin_in_filter(const StepParams& P) { return P.prec == 0 && P.force_path == 0; }

// Completes the last step of a stepping call (the pending second half);
// k_clear_pending then marks the state complete (a call that stopped short of
// its target goes on first). KAHAN as in k_first_half.
template <bool KAHAN>
__global__ void __launch_bounds__(256) k_second_half(StepParams P) {
  Ctrl* C = P.ctrl;
  if (C->halt || !C->pending || C->steps_done < C->target) return;
  const Bank B = P.bank[C->bank];
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < P.n; k += gridDim.x * blockDim.x) {
    uint32_t fl = B.flags[k];
    if (fl & (PF_DEAD | PF_FIXED)) continue;
    D4 vm = B.vm[k], wc = B.wc[k];
    const D4 wr4 = B.wres[k], vr4 = B.vres[k];
    V v = xyz(vm), w = xyz(wc), vres = xyz(vr4), wres = xyz(wr4);
    if (KAHAN) {
      second_half_kick(v, vres, w, wres, xyz(B.acc[k]), xyz(B.tq[k]), wr4.w, P.hdt);
      B.vres[k] = D4{vres.x, vres.y, vres.z, vr4.w};
      B.wres[k] = D4{wres.x, wres.y, wres.z, wr4.w};
    } else {
      const double hdt = P.hdt;
      v = v + xyz(B.acc[k]) * hdt;
      w = w + (xyz(B.tq[k]) * wr4.w) * hdt;
    }
    B.vm[k] = D4{v.x, v.y, v.z, vm.w};
    B.wc[k] = D4{w.x, w.y, w.z, wc.w};
  }
}

// Wall contacts of one particle (src/simulation.rs:464-523): the triangles
// listed in the triangle-grid cell of its centre, in mesh order.
// The cell lookup runs in FP32 on the position mirror (the host grows every
// triangle's box by a margin covering the FP32 error), and a triangle whose
// plane is farther than the radius (plus rounding) cannot touch the sphere,
// because the closest point lies in that plane: both skip FP64 work only.
// Triangles of another group than the particle's (gi) are not walls for it.

// The triangle-grid cell of an FP32 position: its range of triangle entries,
// or false outside the grid.
__device__ __forceinline__ bool tri_cell_range(const StepParams& P, float4 xf, uint32_t& s, uint32_t& e) {
  const float q0 = floorf((xf.x - P.tminf[0]) * P.tinvf);
  const float q1 = floorf((xf.y - P.tminf[1]) * P.tinvf);
  const float q2 = floorf((xf.z - P.tminf[2]) * P.tinvf);
  if (!(q0 >= 0.f && q1 >= 0.f && q2 >= 0.f && q0 < (float)P.tdims[0] && q1 < (float)P.tdims[1] &&
        q2 < (float)P.tdims[2]))
    return false;
  const uint32_t cell = (uint32_t)q0 + (uint32_t)P.tdims[0] * ((uint32_t)q1 + (uint32_t)P.tdims[1] * (uint32_t)q2);
  s = P.tstart[cell];
  e = P.tstart[cell + 1];
  return true;
}

// FP32 pretest of a sphere (centre xf, radius rf = xf.w, largest |coordinate|
// xmag, group gi) against a triangle: false when it cannot touch it. First its
// plane (hd: the distance, mrg: its rounding margin), then its edges.
__device__ __forceinline__ bool wall_plane(const TriRec& tr, uint32_t gi, float4 xf, float xmag, float& hd, float& mrg) {
  // FP32 rounding of n, n.v0 and x moves n.x - n.v0 by at most
  // ~3e-7 (|x| + |n.v0|) + 1.1e-7 |x - v0|; the margin is larger
  const float4 pl = tr.plane;
  hd = fabsf(pl.x * xf.x + pl.y * xf.y + pl.z * xf.z - pl.w);
  mrg = 1e-6f * (1.0f + xmag + fabsf(pl.w) + xf.w) + 2e-7f * (xmag + tr.bound.x);
  return (tr.group == GROUP_ALL || tr.group == gi) && !(hd > xf.w + mrg);
}
__device__ __forceinline__ bool wall_edges(const TriRec& tr, float4 xf, float hd, float mrg) {
  // the distance to the triangle is at least sqrt(hd^2 + s^2), s the
  // largest outward in-plane distance to an edge line (each with the
  // plane test's rounding margin; |m.v| <= sqrt(3) bound)
  const float4 g0 = tr.edge[0], g1 = tr.edge[1], g2 = tr.edge[2];
  const float s = fmaxf(fmaxf(g0.x * xf.x + g0.y * xf.y + g0.z * xf.z - g0.w,
                              g1.x * xf.x + g1.y * xf.y + g1.z * xf.z - g1.w),
                        g2.x * xf.x + g2.y * xf.y + g2.z * xf.z - g2.w);
  const float me = mrg + 4e-7f * tr.bound.x;
  const float hl = fmaxf(hd - mrg, 0.0f), sl = fmaxf(s - me, 0.0f);
  return !(hl * hl + sl * sl > xf.w * xf.w * (1.0f + 1e-6f));
}
__device__ __forceinline__ bool wall_pretest(const TriRec& tr, uint32_t gi, float4 xf, float xmag) {
  float hd, mrg;
  return wall_plane(tr, gi, xf, xmag, hd, mrg) && wall_edges(tr, xf, hd, mrg);
}
// The entries t .. t + 3 of a triangle-grid cell (those below te) that pass, as
// bits; the four triangles' planes are loaded together.
__device__ __forceinline__ uint32_t wall_pretest4(const StepParams& P, uint32_t t, uint32_t te, uint32_t gi, float4 xf,
                                                  float xmag) {
  uint32_t id[4], pass = 0u;
  float hd[4], mrg[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) id[q] = P.titems[min(t + q, te - 1u)];
#pragma unroll
  for (int q = 0; q < 4; ++q)
    if (wall_plane(P.tri[id[q]], gi, xf, xmag, hd[q], mrg[q]) && t + q < te) pass |= 1u << q;
#pragma unroll
  for (int q = 0; q < 4; ++q)
    if ((pass >> q & 1u) && !wall_edges(P.tri[id[q]], xf, hd[q], mrg[q])) pass &= ~(1u << q);
  return pass;
}

// The FP64 contact of a sphere with a triangle that passed the pretest:
// force fc and torque r_a x fc on the sphere, or false (outputs untouched)
// when it does not touch the triangle.
template <bool JKR>
__device__ __forceinline__ bool wall_contact(const StepParams& P, const Law& L, const TriRec& tr, V xi, V vi, V wi,
                                             double ri, double mi, V& fc_out, V& tc_out, bool& excess) {
  // closest point, src/mesh.rs:45-117 (same regions and clamps)
  const V v0 = vmk(tr.v0[0] - xi.x, tr.v0[1] - xi.y, tr.v0[2] - xi.z);
  const V e0 = vmk(tr.e0[0], tr.e0[1], tr.e0[2]), e1 = vmk(tr.e1[0], tr.e1[1], tr.e1[2]);
  const double a = tr.a, b = tr.b, c = tr.c, det = tr.det;
  const double dd = dot(e0, v0), ee = dot(e1, v0);
  const double s0 = b * ee - c * dd, t0 = b * dd - a * ee;
  double sc = s0, tc = t0;
  if (s0 + t0 < det) {
    if (s0 < 0.0) {
      if (t0 < 0.0) {
        if (dd < 0.0) { sc = fmin(fmax(-dd, 0.0), a); tc = 0.0; }
        else { sc = 0.0; tc = fmin(fmax(-ee, 0.0), c); }
      } else { sc = 0.0; tc = fmin(fmax(-ee, 0.0), c); }
    } else if (t0 < 0.0) {
      sc = fmin(fmax(-dd, 0.0), a); tc = 0.0;
    } else {
      const double inv = div_rn(1.0, det);
      sc = sc * inv; tc = tc * inv;
    }
  } else {
    if (s0 < 0.0) {
      const double tmp0 = b + dd, tmp1 = c + ee;
      if (tmp1 > tmp0) {
        const double numer = tmp1 - tmp0;
        sc = div_rn(numer, tr.denom); sc = sc < 0.0 ? 0.0 : (sc > 1.0 ? 1.0 : sc); tc = 1.0 - sc;
      } else { tc = fmin(fmax(-ee, 0.0), c); sc = 0.0; }
    } else if (t0 < 0.0) {
      if (a + dd > b + ee) {
        const double numer = c + ee - b - dd;
        sc = div_rn(numer, tr.denom); sc = sc < 0.0 ? 0.0 : (sc > 1.0 ? 1.0 : sc); tc = 1.0 - sc;
      } else { sc = fmin(fmax(-ee, 0.0), c); tc = 0.0; }
    } else {
      const double numer = c + ee - b - dd;
      sc = div_rn(numer, tr.denom); sc = sc < 0.0 ? 0.0 : (sc > 1.0 ? 1.0 : sc); tc = 1.0 - sc;
    }
  }
  const V cp = vmk(tr.v0[0], tr.v0[1], tr.v0[2]) + sc * e0 + tc * e1;
  const V dv = xi - cp;
  const double dsq = dot(dv, dv);
  if (!less_nn(dsq, ri * ri)) return false;
  const double dist = sqrt_rn(dsq);
  const double pen = ri - dist;
  const V n = less_nn(1e-6, dist) ? div_rn(dv, dist) : vmk(tr.n[0], tr.n[1], tr.n[2]);
  if (is_excess(pen, ri, ri)) excess = true;
  const V ra = (-n) * ri;
  V rv = vi + cross(wi, ra);
  if (tr.motion != NO_MOTION) {  // a moving wall: relative to its surface velocity at the contact point
    const WallMotion& M = P.motions[tr.motion];
    const V vw = vmk(M.v[0], M.v[1], M.v[2]) + cross(vmk(M.w[0], M.w[1], M.w[2]), cp - vmk(M.c[0], M.c[1], M.c[2]));
    rv = rv - vw;
  }
  const double vn = dot(rv, n);
  const double fm = JKR ? jkr_mag(pen, L.es_pw, ri, L.gamma_pw)
                        : normal_mag<double, true>(wall_law(L), P.nmodel, pen, n, vn, ri, mi);
  const V fnv = fm * n;
  const V fc = fnv + coulomb_force<double>(sqrt_rn(dot(fnv, fnv)), rv, n, L.mu);
  fc_out = fc;
  tc_out = cross(ra, fc);
  return true;
}

// All wall contacts of one particle in mesh order.
template <bool JKR>
__device__ __forceinline__ void wall_forces(const StepParams& P, const Law& L, uint32_t gi, V xi, float4 xf, V vi,
                                            V wi, double ri, double mi, V& F, V& T, bool& excess) {
  uint32_t s, e;
  if (P.ntri == 0 || !tri_cell_range(P, xf, s, e)) return;
  const float xmag = fmaxf(fmaxf(fabsf(xf.x), fabsf(xf.y)), fabsf(xf.z));
  for (uint32_t t = s; t < e; ++t) {
    const TriRec& tr = P.tri[P.titems[t]];
    if (!wall_pretest(tr, gi, xf, xmag)) continue;
    V fc, tc;
    if (wall_contact<JKR>(P, L, tr, xi, vi, wi, ri, mi, fc, tc, excess)) {
      F = F + fc;
      T = T + tc;
    }
  }
}

// FP32 pretest on the position mirror. With u = 2^-24 each FP32 difference of
// a pair inside the cutoff is within e = u (2X + 2 cut + L) of the FP64 one (X
// the largest coordinate, L the largest periodic length), so d2f <= cut^2 +
// 3.47 e cut + 3 e^2 + 12 u cut^2 there; (cut + m)^2 with m = 2.1 e + 1e-6 cut
// lies above that, and a pair beyond it is certainly outside the exact FP64
// test. Both ends must keep a pair or drop it together, so the margin is the
// same bit for bit at both: one for all pairs, from the largest |coordinate|
// seen but at most StepParams::xnear, and for pairs of two spheres outside
// StepParams::xhome the pair's own as well. A sphere inside xhome
// and one beyond xnear are no pair, image or not, so a sphere that has flown
// off widens nothing but its own pairs (with the largest coordinate alone, one
// sphere 10,000 km above a hopper of 524,288 made every row entry a candidate:
// 613 us a step against 352 without it; 356 now).
__device__ __forceinline__ float margin_at(const StepParams& P, float X) {
  return 2.1f * (6.0e-8f * (2.0f * X + 2.0f * P.cutmaxf + P.lmax)) + 1.0e-6f * P.cutmaxf;
}
__device__ __forceinline__ float largest(float4 x) { return fmaxf(fmaxf(fabsf(x.x), fabsf(x.y)), fabsf(x.z)); }
__device__ __forceinline__ float pretest_margin(const StepParams& P, const Ctrl* C) {
  return margin_at(P, fminf(__uint_as_float(C->xmax), P.xnear));
}
__device__ __forceinline__ bool pretest_near(const StepParams& P, float4 xi, float4 xj, bool image, float margin) {
  float fx = xi.x - xj.x, fy = xi.y - xj.y, fz = xi.z - xj.z;
  if (image) {
    if (P.periodic[0]) { const float L = P.bsizef[0]; if (fx > 0.5f * L) fx -= L; else if (fx < -0.5f * L) fx += L; }
    if (P.periodic[1]) { const float L = P.bsizef[1]; if (fy > 0.5f * L) fy -= L; else if (fy < -0.5f * L) fy += L; }
    if (P.periodic[2]) { const float L = P.bsizef[2]; if (fz > 0.5f * L) fz -= L; else if (fz < -0.5f * L) fz += L; }
  }
  const float d2 = fx * fx + fy * fy + fz * fz;
  const float rsum = xi.w + xj.w;
  const float t = fminf(rsum * P.cut_a, rsum + P.cut_b) + margin;
  return d2 <= t * t;  // a removed partner's mirror is NaN: not near, from either end
}
// the same for a sphere xi outside xhome, with the pair's own margin (its rows
// are walked again with this one, so that the others' loop stays as it is)
__device__ __forceinline__ bool pretest_far_near(const StepParams& P, float4 xi, float4 xj) {
  const float X = largest(xj);
  return X > P.xhome && pretest_near(P, xi, xj, true, margin_at(P, fmaxf(largest(xi), X)));
}

// ---------------------------------------------------------------- forces
// One thread per slot gathers its Verlet list: the exact FP64 cutoff test of
// src/simulation.rs:327-357, the reference's visit count in parity mode, the
// pair laws of src/simulation.rs:358-460 (in R), the wall triangles of
// src/simulation.rs:464-523 from the triangle grid, then a = g + F/m and
// tau = T (src/simulation.rs:265-271, 532-536). v and omega are only read.
template <bool PHYS, bool HIST, typename R, bool JKR>
__global__ void __launch_bounds__(128) k_force(StepParams P) {
  Ctrl* C = P.ctrl;
  if (C->halt) return;
  const Bank B = P.bank[C->bank];
  const bool adh = (P.nmodel == 3 || P.nmodel == 4);
  const size_t plane = P.hplane;
  const float margin = pretest_margin(P, C);
  bool excess = false;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < P.n; k += gridDim.x * blockDim.x) {
    const uint32_t fl = B.flags[k];
    if (fl & PF_DEAD) continue;
    const Law lw = law_of(P, B, k);
    const uint32_t gi = P.ngroups > 1 ? B.grp[k] : 0u;
    const D4 xi4 = B.xr[k], vi4 = B.vm[k], wi4 = B.wc[k];
    const V xi = xyz(xi4), vi = xyz(vi4), wi = xyz(wi4);
    const double ri = xi4.w, mi = vi4.w;
    const unsigned long long ci = (unsigned long long)__double_as_longlong(wi4.w);
    V F = vmk(0.0, 0.0, 0.0), T = vmk(0.0, 0.0, 0.0);
    const uint32_t cnt = B.ncnt[k];
    const uint32_t* row = B.nbr + (size_t)k * P.cap;
    unsigned long long hm = 0ull;  // springs this row writes (the live-spring mask)
    const float4 xif = B.xf[k];
    const bool far = largest(xif) > P.xhome;
    for (uint32_t m = 0; m < cnt; ++m) {
      const uint32_t j = row[m];
      if (P.pretest) {
        const float4 xjf = B.xf[j];
        if (!pretest_near(P, xif, xjf, true, margin) && !(far && pretest_far_near(P, xif, xjf))) {
          const size_t hi = (size_t)k * P.cap + m;
          if (HIST) {
            B.hist[hi] = 0.0;
            B.hist[plane + hi] = 0.0;
            B.hist[2 * plane + hi] = 0.0;
          }
          if (P.debug) P.dbgMult[hi] = 0;
          continue;
        }
      }
      const D4 xj4 = B.xr[j];
      V d = xi - xyz(xj4);
      if (P.periodic[0]) { if (d.x > P.bsize[0] * 0.5) d.x = d.x - P.bsize[0]; else if (d.x < -P.bsize[0] * 0.5) d.x = d.x + P.bsize[0]; }
      if (P.periodic[1]) { if (d.y > P.bsize[1] * 0.5) d.y = d.y - P.bsize[1]; else if (d.y < -P.bsize[1] * 0.5) d.y = d.y + P.bsize[1]; }
      if (P.periodic[2]) { if (d.z > P.bsize[2] * 0.5) d.z = d.z - P.bsize[2]; else if (d.z < -P.bsize[2] * 0.5) d.z = d.z + P.bsize[2]; }
      const double d2 = dot(d, d);
      const double rj = xj4.w;
      const double rsum = ri + rj;
      const double margin = adh ? rsum * 0.5 : 0.0;
      const double cut = rsum + margin;
      int visits = 0;
      const size_t hi = (size_t)k * P.cap + m;
      if (d2 < cut * cut) {
        const D4 wj4 = B.wc[j];
        visits = PHYS ? 1 : ref_visits(P, ci, (unsigned long long)__double_as_longlong(wj4.w));
        if (visits > 0) {
          const D4 vj4 = B.vm[j];
          V fc, tc, nrm;
          T3<R> fr, tr, nr;
          if constexpr (PHYS && sizeof(R) == sizeof(double)) {
            pair_contact_fused<HIST, JKR>(P, lw, d, d2, rsum, ri, rj, mi, vj4.w, vi, xyz(vj4), wi, xyz(wj4),
                                     HIST ? B.hist + hi : nullptr, plane, fc, nrm, excess);
            tc = (-ri) * nrm;
          } else if (pair_contact<R, PHYS, HIST, JKR>(P, lw, d, d2, rsum, ri, rj, mi, vj4.w, vi, xyz(vj4), wi, xyz(wj4),
                                          HIST ? B.hist + hi : nullptr, plane, fr, tr, nr, excess)) {
            fc = cvt<double>(fr);
            tc = cvt<double>(tr);
          } else if constexpr (PHYS) {
            pair_contact_fused<HIST, JKR>(P, lw, d, d2, rsum, ri, rj, mi, vj4.w, vi, xyz(vj4), wi, xyz(wj4),
                                     HIST ? B.hist + hi : nullptr, plane, fc, nrm, excess);
            tc = (-ri) * nrm;
          } else {
            pair_contact<double, PHYS, HIST, JKR>(P, lw, d, d2, rsum, ri, rj, mi, vj4.w, vi, xyz(vj4), wi, xyz(wj4),
                                             HIST ? B.hist + hi : nullptr, plane, fc, tc, nrm, excess);
          }
          if (HIST && m < 64) hm |= 1ull << m;
          for (int t = 0; t < visits; ++t) {
            F = F + fc;
            T = T + tc;
          }
        }
      }
      if (HIST && visits == 0) {
        B.hist[hi] = 0.0;
        B.hist[plane + hi] = 0.0;
        B.hist[2 * plane + hi] = 0.0;
      }
      if (P.debug) P.dbgMult[hi] = (uint8_t)visits;
    }
    if (HIST && hm) B.hmask[k] |= hm;
    wall_forces<JKR>(P, lw, gi, xi, xif, vi, wi, ri, mi, F, T, excess);
    if (P.debug) {
      P.dbgF[3 * (size_t)k] = F.x; P.dbgF[3 * (size_t)k + 1] = F.y; P.dbgF[3 * (size_t)k + 2] = F.z;
      P.dbgT[3 * (size_t)k] = T.x; P.dbgT[3 * (size_t)k + 1] = T.y; P.dbgT[3 * (size_t)k + 2] = T.z;
    }
    if (!isfinite(F.x + F.y + F.z + T.x + T.y + T.z)) atomicOr(&C->status, (unsigned)ST_NAN);
    // apply (src/simulation.rs:532-536), F/m as F (1/m) with 1/m stored per
    // particle; the second half kick of this step runs in the next
    // k_first_half or in k_second_half
    const V a = vmk(P.gravity[0], P.gravity[1], P.gravity[2]) + F * B.vres[k].w;
    const V tau = vmk(0.0, 0.0, 0.0) + T;
    B.acc[k] = D4{a.x, a.y, a.z, 0.0};
    B.tq[k] = D4{tau.x, tau.y, tau.z, 0.0};
  }
  if (excess) C->overlap_flag = 1;
}

// ------------------------------------------------- contact-parallel forces
// One thread per particle leaves every lane idle while a neighbour of another
// lane is in contact (measured: ~9 of 32 lanes active, FP64 pipe saturated).
// Here the per-particle pass only filters (FP32 pretest, exact FP64 cutoff,
// visit counts); the pair laws run one thread per pair, each pair once, and a
// last pass sums every particle's contact results in list order.

// Minimum image on the periodic axes. A difference whose magnitude has a
// smaller high word than bsize/4 is below bsize/4 (and NaN is not), so it
// needs no FP64 comparison.
__device__ __forceinline__ bool near_axis(double d, uint32_t q_hi) {
  return (uint32_t)(__double2hiint(d) & 0x7FFFFFFF) < q_hi;
}
__device__ __forceinline__ V mic(const StepParams& P, V d) {
  if (P.periodic[0] && !near_axis(d.x, P.bq_hi[0])) { if (d.x > P.bsize[0] * 0.5) d.x = d.x - P.bsize[0]; else if (d.x < -P.bsize[0] * 0.5) d.x = d.x + P.bsize[0]; }
  if (P.periodic[1] && !near_axis(d.y, P.bq_hi[1])) { if (d.y > P.bsize[1] * 0.5) d.y = d.y - P.bsize[1]; else if (d.y < -P.bsize[1] * 0.5) d.y = d.y + P.bsize[1]; }
  if (P.periodic[2] && !near_axis(d.z, P.bq_hi[2])) { if (d.z > P.bsize[2] * 0.5) d.z = d.z - P.bsize[2]; else if (d.z < -P.bsize[2] * 0.5) d.z = d.z + P.bsize[2]; }
  return d;
}

// Where a JKR pair of the certified solvers goes, from jkr_certify on the FP32
// position mirror: CREC_HARD to the list of pairs next to the fold, whose force
// needs the reference's Newton, CREC_NET to the network queue (both with a
// margin for the mirror's rounding, ~2.4e-7 of the coordinates). Both are hints,
// the exact certificates decide: a queued pair they reject only wastes a
// network row, a converging pair without a row falls back to the reference's
// Newton, and one that needs it outside the list is deferred.
__device__ __forceinline__ uint32_t jkr_hint(const StepParams& P, float Cf, float4 xif, float4 xjf, bool learn) {
  float fx = xif.x - xjf.x, fy = xif.y - xjf.y, fz = xif.z - xjf.z;
  if (P.periodic[0]) { const float L = P.bsizef[0]; if (fx > 0.5f * L) fx -= L; else if (fx < -0.5f * L) fx += L; }
  if (P.periodic[1]) { const float L = P.bsizef[1]; if (fy > 0.5f * L) fy -= L; else if (fy < -0.5f * L) fy += L; }
  if (P.periodic[2]) { const float L = P.bsizef[2]; if (fz > 0.5f * L) fz -= L; else if (fz < -0.5f * L) fz += L; }
  const float rsum = xif.w + xjf.w;
  const float rs = xif.w * xjf.w / rsum;
  const float c = Cf / rs;
  if (!(c >= kJkrCMin && c <= kJkrCMax)) return CREC_HARD;
  const float c23 = jkr_c23(c);
  const float x = (rsum - sqrtf(fx * fx + fy * fy + fz * fz)) / rs;
  const float xi = x / c23;
  const float X = fmaxf(fmaxf(fmaxf(fabsf(xif.x), fabsf(xif.y)), fabsf(xif.z)),
                        fmaxf(fmaxf(fabsf(xjf.x), fabsf(xjf.y)), fabsf(xjf.z)));
  const float e = 2.4e-7f * (2.0f * X + rsum + P.lmax) / (rs * c23);
  const float h = 0.15f * e;  // the usual size of that rounding, not its bound
  if (xi < kJkrXiNeg + h || (xi > kJkrXiWalk - h && xi < kJkrXiPos + h)) return CREC_HARD;
  if (!learn) return 0u;
  const float m = 0.02f + e;
  if (xi < kJkrXiNeg - m) return 0u;
  if (xi > m && xi < kJkrXiPos - m) return 0u;
  const float f1 = logf(rs);
  if (f1 < P.jdom_lo[1] || f1 > P.jdom_hi[1]) return 0u;
  if (sqrtf(fmaxf(xi - m + kJkrKappa, 0.0f)) > P.jdom_hi[0]) return 0u;
  return CREC_NET;
}

// Whether a JKR pair is certainly in the ZERO region of jkr_certify (no
// contact radius makes the reference's residual smaller than 1e-3 R*, so its
// JKR force is exactly zero), decided on the FP32 position mirror with that
// mirror's rounding added to the certificate's margin. Symmetric in (i, j)
// bit for bit, so both ends of a pair drop it or keep it together.
__device__ __forceinline__ bool jkr_far_zero(const StepParams& P, float Cf, float4 xif, float Xi, float4 xjf) {
  float fx = xif.x - xjf.x, fy = xif.y - xjf.y, fz = xif.z - xjf.z;
  if (P.periodic[0]) { const float L = P.bsizef[0]; if (fx > 0.5f * L) fx -= L; else if (fx < -0.5f * L) fx += L; }
  if (P.periodic[1]) { const float L = P.bsizef[1]; if (fy > 0.5f * L) fy -= L; else if (fy < -0.5f * L) fy += L; }
  if (P.periodic[2]) { const float L = P.bsizef[2]; if (fz > 0.5f * L) fz -= L; else if (fz < -0.5f * L) fz += L; }
  const float rsum = xif.w + xjf.w;
  const float rs = (xif.w * xjf.w) / rsum;
  const float c = Cf / rs;
  if (!(c > 0.0f && c < 1e30f)) return false;
  const float c23 = jkr_c23(c);
  const float d = sqrtf(fx * fx + fy * fy + fz * fz);
  const float X = fmaxf(Xi, fmaxf(fmaxf(fabsf(xjf.x), fabsf(xjf.y)), fabsf(xjf.z)));
  // per-axis FP32 difference error <= 6e-8 (2X + 2 cut + L) (as in pretest_near),
  // so |d_f - d| <= 1.8e-7 (2X + 3 r_sum + L) + 4e-7 d, radii rounded too
  const float e = (1.8e-7f * (2.0f * X + 3.0f * rsum + P.lmax) + 4e-7f * (d + rsum)) / rs;
  const float x = (rsum - d) / rs;
  return x + kJkrKappa * c23 + 1e-3f < -(1e-5f * (fabsf(x) + c23 + 1e-3f) + 2.0f * e);
}

// Whether an sJKR pair certainly has zero normal force: overlap below
// delta_c = -sqrt(3 pi^2 gamma^2 R* / E*^2) (src/physics.rs:234-325; with
// gamma <= 0 the law is Hertz's, zero for a negative overlap), decided on the
// FP32 mirror with its rounding (as jkr_far_zero) and 1e-5 of delta_c as
// margin. Symmetric in (i, j) bit for bit.
__device__ __forceinline__ bool sjkr_far_zero(const StepParams& P, const Law& L, float4 xif, float Xi, float4 xjf) {
  float fx = xif.x - xjf.x, fy = xif.y - xjf.y, fz = xif.z - xjf.z;
  if (P.periodic[0]) { const float Lp = P.bsizef[0]; if (fx > 0.5f * Lp) fx -= Lp; else if (fx < -0.5f * Lp) fx += Lp; }
  if (P.periodic[1]) { const float Lp = P.bsizef[1]; if (fy > 0.5f * Lp) fy -= Lp; else if (fy < -0.5f * Lp) fy += Lp; }
  if (P.periodic[2]) { const float Lp = P.bsizef[2]; if (fz > 0.5f * Lp) fz -= Lp; else if (fz < -0.5f * Lp) fz += Lp; }
  const float rsum = xif.w + xjf.w;
  const float rs = (xif.w * xjf.w) / rsum;
  const float d = sqrtf(fx * fx + fy * fy + fz * fz);
  const float X = fmaxf(Xi, fmaxf(fmaxf(fabsf(xjf.x), fabsf(xjf.y)), fabsf(xjf.z)));
  const float e = 1.8e-7f * (2.0f * X + 3.0f * rsum + P.lmax) + 4e-7f * (d + rsum);
  float dc = 0.0f;
  if (L.gamma_pp > 0.0) {
    const float g = (float)L.gamma_pp, es = (float)L.es_pp, pi = 3.14159265f;
    dc = -sqrtf(3.0f * (pi * pi) * (g * g) * rs / (es * es));
  }
  return (rsum - d) + e < dc - 1e-5f * fabsf(dc);
}

// Exclusive prefix of v over the lanes of the warp, and the warp's total.
// Every lane of the warp takes part.
__device__ __forceinline__ uint32_t warp_exclusive(uint32_t v, uint32_t& total) {
  const int lane = threadIdx.x & 31;
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
    if (lane >= o) x += y;
  }
  total = __shfl_sync(0xFFFFFFFFu, x, 31);
  return x - v;
}

// The contact pass's counters (records, evaluating records, network queue,
// deferred pairs, wall candidates, hard pairs) start every force pass at zero.
constexpr int CTOT_WORDS = 8;

// Pass 1 (FP32 and integer work only): the candidates of each particle, i.e.
// list entries the FP32 pretest cannot rule out and that the reference's loop
// visits from this end (visit counts from both ends recorded); marks the ones
// that evaluate their pair (the lower slot of a pair seen from both ends, or
// the only end that sees it). The pretest is symmetric, so a pair seen from
// both ends is a candidate at both. Each warp then reserves the result slots of
// its particles' records (coff) and their places in the compact list of
// evaluating records (and the queues of the JKR solvers), one atomic
// instruction for all counters: where a record's result lands changes nothing
// in its value, and each particle's results stay contiguous and in list order.
// The block size is a multiple of 32 and every lane of a warp runs the same
// number of iterations.
//
// Bound by the latency of the gathers, so a row is walked in two phases of up
// to 32 entries: first four entries at a time, their indices in one 16-byte
// load and their positions in flight together, into a mask of the entries that
// pass; then the candidates, whose visit counts need no gather where the whole
// neighbourhood lies in one reference cell (PF_ONECELL). One entry at a time
// with the visit counts in between, the pass took 155 us on 1,048,576 spheres
// (hopper, rows of 11) and 329 us on 2,097,152 adhesive ones; this form takes 122 and 176 us.
// COHERENT: the positions were written by the same kernel launch, so they are
// not read through the read-only path; slots are taken in order.
template <bool COHERENT>
__device__ __forceinline__ float4 load_xf(const float4* p) {
  return COHERENT ? *p : __ldg(p);
}
template <bool PHYS, bool HIST, bool COHERENT>
__device__ __forceinline__ void filter_pass(const StepParams& P, Ctrl* C, const Bank& B, uint32_t* ctot, Span sp) {
  const bool learn_any = P.jkr_solver == 1 && P.nmodel == 3 && P.mlp != nullptr;
  const bool hint_any = P.jfb != nullptr;  // a certified JKR solver
  // JKR pairs certified to have no force add exactly +-0 to F and T (the
  // tangential force then vanishes too, see StepParams::drop_zero): they are
  // not candidates at all, whichever solver takes the others. The reference's
  // own Newton, which returns zero for them after up to 20 steps, had spent
  // nine tenths of its time on them (262,144 spheres at solid fraction 0.35:
  // the step 2.68 -> 0.22 ms).
  const bool zdrop_any = P.drop_zero && P.nmodel == 3;
  // the same for sJKR, whose zero region is explicit (no iteration to certify)
  const bool sdrop = P.drop_zero && P.nmodel == 4;
  const size_t plane = P.hplane;
  const float margin = pretest_margin(P, C);
  const int lane = threadIdx.x & 31;
  const bool kick = !COHERENT && C->spin_due != 0, fuse = C->pending != 0;
  // slots in the rebuild-time order (tiles of 256 sorted by list length), so
  // a warp's lanes walk lists of similar length
  for (int i0 = sp.at - lane; i0 < P.n; i0 += sp.all) {
    const int i = i0 + lane;
    const int k = i < P.n ? (COHERENT ? i : (int)P.aorder[i]) : -1;
    uint32_t nrec = 0, ncmp = 0, nnet = 0, nhard = 0, nw = 0, ts = 0, te = 0, gi = 0;
    uint32_t evals = 0u;  // records (the first 32) that evaluate their pair
    uint32_t wmask = 0u;  // entries of its triangle-grid cell (the first 32) that pass
    float4 xif = make_float4(0.f, 0.f, 0.f, 0.f);
    float Xi = 0.f;
    const uint32_t flk = k >= 0 ? B.flags[k] : PF_DEAD;
    if (!(flk & PF_DEAD)) {
      const bool onecell = PHYS || (flk & PF_ONECELL);
      const int same = PHYS ? 1 : P.same_cell_visits;
      const unsigned long long ci = onecell ? 0ull : (unsigned long long)__double_as_longlong(B.wc[k].w);
      const int same_c = !PHYS && !onecell && ref_inside(P, ci) ? same : 0;
      xif = B.xf[k];
      const bool image = !(flk & PF_NOIMAGE);
      Xi = largest(xif);
      const uint32_t cnt = B.ncnt[k];
      const uint32_t* row = B.nbr + (size_t)k * P.cap;
      CRec* out = P.crec + (size_t)k * P.cap;
      if (kick && !(flk & PF_FIXED)) spin_kick(P, B, k, flk, fuse);
      const bool wide = (P.cap & 3) == 0;  // rows on 16 bytes
      // where latency is all that counts, the first eight entries come with the
      // particle itself (a dilute bed of a million would read rows it does not have)
      uint4 head0 = make_uint4(0u, 0u, 0u, 0u), head1 = head0;
      if (COHERENT && wide) {
        head0 = __ldg(reinterpret_cast<const uint4*>(row));
        if (P.cap > 4) head1 = __ldg(reinterpret_cast<const uint4*>(row) + 1);
      }
      const bool walled = P.ntri > 0 && !(P.wall_far_ok && (flk & PF_WALLFAR)) && tri_cell_range(P, xif, ts, te);
      for (uint32_t c0 = 0; c0 < cnt; c0 += 32) {
        const uint32_t ce = min(cnt - c0, 32u);
        const uint32_t valid = 0xFFFFFFFFu >> (32u - ce);
        uint32_t near = 0u;
        if (P.pretest) {
          for (uint32_t m = 0; m < ce; m += 4) {
            uint4 j;
            if (wide) {  // entries past the end are not followed
              if (COHERENT && c0 + m < 8) j = c0 + m == 0 ? head0 : head1;
              else j = __ldg(reinterpret_cast<const uint4*>(row + c0 + m));
              if (m + 1 >= ce) j.y = j.x;
              if (m + 2 >= ce) j.z = j.x;
              if (m + 3 >= ce) j.w = j.x;
            } else {
              j.x = __ldg(row + c0 + m);
              j.y = m + 1 < ce ? __ldg(row + c0 + m + 1) : j.x;
              j.z = m + 2 < ce ? __ldg(row + c0 + m + 2) : j.x;
              j.w = m + 3 < ce ? __ldg(row + c0 + m + 3) : j.x;
            }
            const float4 x0 = load_xf<COHERENT>(B.xf + j.x), x1 = load_xf<COHERENT>(B.xf + j.y),
                         x2 = load_xf<COHERENT>(B.xf + j.z), x3 = load_xf<COHERENT>(B.xf + j.w);
            const uint32_t q = (pretest_near(P, xif, x0, image, margin) ? 1u : 0u) |
                               (pretest_near(P, xif, x1, image, margin) ? 2u : 0u) |
                               (pretest_near(P, xif, x2, image, margin) ? 4u : 0u) |
                               (pretest_near(P, xif, x3, image, margin) ? 8u : 0u);
            near |= q << m;
          }
          if (Xi > P.xhome) {
#pragma unroll 1
            for (uint32_t m = 0; m < ce; ++m)
              if (pretest_far_near(P, xif, load_xf<COHERENT>(B.xf + __ldg(row + c0 + m)))) near |= 1u << m;
          }
          near &= valid;
        } else {
          // a removed partner shows by its flag: its own row is not walked, so
          // it evaluates nothing for this end
          for (uint32_t m = 0; m < ce; ++m)
            if (!(B.flags[__ldg(row + c0 + m)] & PF_DEAD)) near |= 1u << m;
        }
        uint32_t kept = 0u;
        for (uint32_t left = near; left; left &= left - 1u) {
          const uint32_t b = (uint32_t)__ffs((int)left) - 1u, m = c0 + b;
          const uint32_t j = __ldg(row + m);
          uint32_t hint = 0u;
          if (P.nmodel >= 3) {  // pairs never cross groups (the lists exclude them)
            const Law lw = law_of(P, B, k);
            const float4 xjf = load_xf<COHERENT>(B.xf + j);
            const bool adhesive = lw.gamma_pp > 0.0;
            if (zdrop_any && adhesive && jkr_far_zero(P, lw.jkr_Cf, xif, Xi, xjf)) continue;
            if (sdrop && sjkr_far_zero(P, lw, xif, Xi, xjf)) continue;
            // (the higher slot of a pair seen from both ends does not evaluate it)
            if (hint_any && adhesive && !(onecell && (uint32_t)k > j)) hint = jkr_hint(P, lw.jkr_Cf, xif, xjf, learn_any);
          }
          int vij = same, vji = same;
          if (!onecell) {
            const unsigned long long cj = (unsigned long long)__double_as_longlong(B.wc[j].w);
            if (cj == ci) {
              vij = vji = same_c;
            } else {
              vij = ref_visits(P, ci, cj);
              vji = ref_visits(P, cj, ci);
            }
          }
          if (vij == 0) continue;
          kept |= 1u << b;
          const bool evaluates = !(vji > 0 && (uint32_t)k > j);
          if (evaluates) {
            if (hint & CREC_HARD) ++nhard;
            else ++ncmp;
            if (hint & CREC_NET) ++nnet;
            if (nrec < 32) evals |= 1u << nrec;
          } else {
            hint = 0u;
          }
          out[nrec] = CRec{j, m | ((uint32_t)vij << 16) | ((uint32_t)vji << 24) | hint};
          ++nrec;
        }
        if (HIST) {
          // a spring out of reach resets; one already +0 (its bit clear; entries past 64 have none) stays
          uint32_t* hm = reinterpret_cast<uint32_t*>(B.hmask + k) + (c0 >> 5);
          const uint32_t live = c0 < 64 ? *hm : 0xFFFFFFFFu;
          const uint32_t reset = valid & ~kept & live;
          for (uint32_t left = reset; left; left &= left - 1u) {
            const size_t hi = (size_t)k * P.cap + c0 + (uint32_t)__ffs((int)left) - 1u;
            B.hist[hi] = 0.0;
            B.hist[plane + hi] = 0.0;
            B.hist[2 * plane + hi] = 0.0;
          }
          if (c0 < 64 && reset) *hm = live & ~reset;
        }
        if (P.debug)
          for (uint32_t left = valid & ~kept; left; left &= left - 1u)
            P.dbgMult[(size_t)k * P.cap + c0 + (uint32_t)__ffs((int)left) - 1u] = 0;
      }
      // wall candidates: the triangles of its triangle-grid cell that pass
      // the FP32 pretest, counted here and listed once the arena is reserved
      if (walled) {
        gi = P.ngroups > 1 ? B.grp[k] : 0u;
        for (uint32_t t = ts; t < te; t += 4) {
          const uint32_t pass = wall_pretest4(P, t, te, gi, xif, Xi);
          nw += (uint32_t)__popc(pass);
          if (t - ts < 32u) wmask |= pass << (t - ts);
        }
      }
    }
    __syncwarp();
    // exclusive prefixes over the warp; records and evaluating records share a
    // word where 32 rows cannot overflow its halves
    uint32_t tr = 0, tc = 0, tn = 0, tw = 0, th = 0, rb, q, qn = 0, wb = 0, qh = 0;
    if (P.cap < 2048) {
      uint32_t t;
      const uint32_t ex = warp_exclusive(nrec | (ncmp << 16), t);
      rb = ex & 0xFFFFu;
      q = ex >> 16;
      tr = t & 0xFFFFu;
      tc = t >> 16;
    } else {
      rb = warp_exclusive(nrec, tr);
      q = warp_exclusive(ncmp, tc);
    }
    if (learn_any) qn = warp_exclusive(nnet, tn);
    if (hint_any) qh = warp_exclusive(nhard, th);
    if (__any_sync(0xFFFFFFFFu, nw != 0)) wb = warp_exclusive(nw, tw);
    const uint32_t add = lane == 0 ? tr : lane == 1 ? tc : lane == 2 ? tn : lane == 4 ? tw : lane == 5 ? th : 0u;
    uint32_t at = 0;
    if (add) at = atomicAdd(ctot + lane, add);
    rb += __shfl_sync(0xFFFFFFFFu, at, 0);
    q += __shfl_sync(0xFFFFFFFFu, at, 1);
    if (learn_any) qn += __shfl_sync(0xFFFFFFFFu, at, 2);
    if (hint_any) qh += __shfl_sync(0xFFFFFFFFu, at, 5);
    wb += __shfl_sync(0xFFFFFFFFu, at, 4);
    if (k < 0) continue;
    P.ccnt[k] = nrec;
    P.coff[k] = rb;
    if (P.ntri > 0) {
      if (nw > 0 && wb + nw <= P.wcap) {  // in mesh order, as the reference visits them
        uint2* dst = P.warena + wb;
        uint32_t c = 0;
        for (uint32_t left = wmask; left; left &= left - 1u)
          dst[c++] = make_uint2((uint32_t)k, P.titems[ts + (uint32_t)__ffs((int)left) - 1u]);
        for (uint32_t t = ts + 32u; t < te && c < nw; ++t) {
          const uint32_t id = P.titems[t];
          if (wall_pretest(P.tri[id], gi, xif, Xi)) dst[c++] = make_uint2((uint32_t)k, id);
        }
      } else if (nw > 0) {  // the arena is full: the step halts and the host grows it
        atomicMax(&C->wall_need, wb + nw);
        atomicOr(&C->halt, HALT_WALLS);
      }
      P.wcnt[k] = nw;
      P.woff[k] = wb;
    }
    if (ncmp + nhard == 0) continue;
    if (q + ncmp > P.ccap || (hint_any && qh + nhard > P.hcap)) {  // the host grows the lists and runs the step again
      atomicMax(&C->pair_need, q + ncmp);
      if (hint_any) atomicMax(&C->hard_need, qh + nhard);
      atomicOr(&C->halt, HALT_PAIRS);
      continue;
    }
    // the evaluating records into the compact list, read back from the row that
    // this thread just wrote
    const CRec* out = P.crec + (size_t)k * P.cap;
    if (nrec <= 32 && !hint_any) {
      for (uint32_t left = evals; left; left &= left - 1u) {
        const uint32_t c = (uint32_t)__ffs((int)left) - 1u;
        const CRec r = out[c];
        P.clist[q++] = make_uint4((uint32_t)k, r.j, r.mv, rb + c);
      }
      continue;
    }
    // long rows, and the queues of the certified JKR solvers
    for (uint32_t c = 0; c < nrec; ++c) {
      const CRec r = out[c];
      if (crec_vji(r.mv) > 0 && (uint32_t)k > r.j) continue;
      const uint4 it = make_uint4((uint32_t)k, r.j, r.mv, rb + c);
      if (r.mv & CREC_HARD) {
        P.jhard[qh++] = it;
        continue;
      }
      if (r.mv & CREC_NET) P.jq[qn++] = q;
      P.clist[q++] = it;
    }
  }
}

template <bool PHYS, bool HIST>
__global__ void __launch_bounds__(256, 4) k_contact_filter(StepParams P) {
  Ctrl* C = P.ctrl;
  // a full buffer that another block reports must not keep this one from
  // its spin kicks (the device loop ends with the step that halts)
  if (C->spin_due ? (C->halt & HALT_LISTS) : C->halt) return;
  filter_pass<PHYS, HIST, false>(P, C, P.bank[C->bank], P.ctot, grid_span());
}

// Pass 2b: the JKR network over the queue, 32 pairs per warp on the tensor
// cores (weights staged once per block in shared memory). Features from the
// FP64 positions: the overlap from r_sum^2 - d^2 in FP64, the rest in FP32.
// Writes the predicted a/R* of each queued pair, NaN outside the training
// range.
__global__ void __launch_bounds__(128) k_jkr_mlp(StepParams P) {
  Ctrl* C = P.ctrl;
  if (C->halt) return;
  const uint32_t qn = P.ctot[2];
  if ((uint32_t)blockIdx.x * blockDim.x >= qn) return;
  __shared__ MlpShared M;
  mlp_stage(M, P.mlp);
  __syncthreads();
  const Bank B = P.bank[C->bank];
  const int lane = threadIdx.x & 31;
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t base = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < qn; base += stride) {
    const uint32_t idx = base + lane;
    const bool valid = idx < qn;
    float f[4] = {0.f, 0.f, 0.f, 0.f};
    float ub = 0.f;
    bool ok = false;
    uint32_t q = 0;
    if (valid) {
      q = P.jq[idx];
      const uint4 it = P.clist[q];
      const uint32_t k = it.x, j = it.y;
      const D4 xi4 = B.xr[k], xj4 = B.xr[j];
      const V d = mic(P, xyz(xi4) - xyz(xj4));
      const double d2 = dot(d, d);
      const double rsum = xi4.w + xj4.w;
      const float ov = (float)(rsum * rsum - d2) / ((float)rsum + sqrtf((float)d2));
      const float rs = ((float)xi4.w * (float)xj4.w) / (float)rsum;  // a feature: FP32 is enough
      const float x = ov / rs;
      const Law lw = law_of(P, B, (int)k);
      const float c = lw.jkr_Cf / rs;
      const float c23 = jkr_c23(c);
      float raw[4];
      jkr_raw_features(x, c23, rs, (float)lw.es_pp, (float)lw.gamma_pp, raw);
      ok = true;
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        ok = ok && raw[a] >= P.jdom_lo[a] && raw[a] <= P.jdom_hi[a];
        f[a] = (raw[a] - M.xmean[a]) * M.xinv[a];
      }
      ub = jkr_ubase(x, c23);
    }
    const float y = mlp_forward_warp(&M, f);
    if (valid) P.jguess[q] = ok ? __expf(y * M.ystd + M.ymean) * ub : __int_as_float(0x7FC00000);
  }
}

// Pass 3: one thread per candidate pair: the exact FP64 cutoff test of
// src/simulation.rs:343-357, then the pair laws. The force on the row's
// particle times its visit count goes to its result; the other end receives
// exactly the negated force (the reference's formula is sign-symmetric:
// evaluated from that end it gives -f bit for bit) times its own visit count,
// with its own torque (n r_j) x (-f), and in physical mode the negated spring.
// A candidate outside the cutoff gives zero results at both ends.
//
// With a certified JKR solver, a pair whose JKR force needs the reference's
// own Newton iteration (up to 20 steps) is not evaluated in this pass: it
// would hold its whole warp for those steps. It is appended to
// a deferred list (contact_eval returns true) and k_contact_deferred
// evaluates the deferred pairs densely; each pair writes the same result slots
// in either pass, so the outcome does not depend on the order.
// One contact result (force and torque on the row's particle, times its
// visit count) into its record: FP64 in the FP64 form; FP32 in the mixed form,
// whose pair forces are FP32 values (24 bytes a record instead of 48; the
// per-particle sums stay FP64). Pairs the mixed form evaluates in FP64 (the
// JKR fold band, decisions within FP32 rounding) are rounded once here.
// The FP32 form's results stay FP32 from the law to the record (a visit
// count times an FP32 value rounds the same in FP32 as in FP64).
template <typename R>
__device__ __forceinline__ void put_result(const StepParams& P, uint32_t rec, T3<R> f, T3<R> t, int visits) {
  // x * 1 = x: no multiply for the common single visit. The warp decides: as a
  // branch of each lane the 7 FP64 instructions became predicated ones, and a
  // predicated-off FP64 instruction takes the pipe as long as a full one (14 of
  // ~125 a contact: hopper of 1,048,576 spheres 415 to 379 us in this kernel,
  // 654 to 630 a step; its spring bed of 524,288 406 to 387).
  if (__any_sync(__activemask(), visits != 1)) {
    const R s = (R)visits;
    f = f * s;
    t = t * s;
  }
  if (P.prec == 1) {
    float2* o = reinterpret_cast<float2*>(P.cresf + 6 * (size_t)rec);
    o[0] = make_float2((float)f.x, (float)f.y);
    o[1] = make_float2((float)f.z, (float)t.x);
    o[2] = make_float2((float)t.y, (float)t.z);
  } else {
    double2* o = reinterpret_cast<double2*>(P.cres + 6 * (size_t)rec);
    o[0] = make_double2(f.x, f.y);
    o[1] = make_double2(f.z, t.x);
    o[2] = make_double2(t.y, t.z);
  }
}

// The record of row j whose partner is k (its place among the row's records),
// NO_RECORD when the row has none; four records at a time where rows allow it,
// the first four without waiting for the row's count.
constexpr uint32_t NO_RECORD = 0xFFFFFFFFu;
__device__ __forceinline__ uint32_t back_record(const StepParams& P, uint32_t j, uint32_t k) {
  const CRec* row = P.crec + (size_t)j * P.cap;
  if ((P.cap & 3) == 0) {
    const uint4* two = reinterpret_cast<const uint4*>(row);
    uint4 a = two[0], b = two[1];
    const uint32_t n = P.ccnt[j];
    for (uint32_t c = 0; c < n;) {
      const uint32_t at = a.x == k ? 0u : a.z == k ? 1u : b.x == k ? 2u : b.z == k ? 3u : 4u;
      if (at < 4u && c + at < n) return c + at;
      c += 4;
      if (c < n) { a = two[c / 2]; b = two[c / 2 + 1]; }
    }
  } else {
    const uint32_t n = P.ccnt[j];
    for (uint32_t c = 0; c < n; ++c)
      if (row[c].j == k) return c;
  }
  return NO_RECORD;
}

template <bool PHYS, bool HIST, typename R, bool JKR>
__device__ __forceinline__ bool contact_eval(const StepParams& P, const Bank& B, uint4 it, float guess,
                                             bool can_defer, bool newton, bool& excess, uint32_t* tally) {
  const size_t plane = P.hplane;
  const bool adh = (P.nmodel == 3 || P.nmodel == 4);
  const uint32_t k = it.x, j = it.y, m = it.z & 0xFFFFu;
  const int vij = (it.z >> 16) & 0xFF, vji = crec_vji(it.z);
  if (!(it.z & CREC_NET)) guess = -1.0f;
  else if (tally) tally[3] += 1;
  // everything the pair needs is asked for at once: the chain of a pair is
  // latency (list, both ends and the other's records), then FP64
  const D4 xi4 = B.xr[k], xj4 = B.xr[j];
  const D4 vi4 = B.vm[k], wi4 = B.wc[k], vj4 = B.vm[j], wj4 = B.wc[j];
  const uint32_t offj = P.coff[j];
  const uint32_t back = vji > 0 ? back_record(P, j, k) : NO_RECORD;
  const V d = mic(P, xyz(xi4) - xyz(xj4));
  const double d2 = dot(d, d);
  const double rsum = xi4.w + xj4.w;
  const double cut = rsum + (adh ? rsum * 0.5 : 0.0);
  const bool in = less_nn(d2, cut * cut);
  const size_t hik = (size_t)k * P.cap + m;
  double* hk = HIST ? B.hist + hik : nullptr;
  T3<R> fc = t3(R(0), R(0), R(0)), tc = fc, tc2 = fc, nrm = fc;  // tc2: the torque on the other end
  if (in) {
    const Law lw = law_of(P, B, (int)k);
    bool deferred = false;
    if constexpr (PHYS && sizeof(R) == sizeof(double)) {
      pair_contact_fused<HIST, JKR>(P, lw, d, d2, rsum, xi4.w, xj4.w, vi4.w, vj4.w, xyz(vi4), xyz(vj4), xyz(wi4), xyz(wj4),
                               hk, plane, fc, nrm, excess, guess, tally, can_defer ? &deferred : nullptr, newton);
      tc = (-xi4.w) * nrm;
      tc2 = (-xj4.w) * nrm;
    } else {
      bool done = pair_contact<R, PHYS, HIST, JKR>(P, lw, d, d2, rsum, xi4.w, xj4.w, vi4.w, vj4.w, xyz(vi4), xyz(vj4),
                                              xyz(wi4), xyz(wj4), hk, plane, fc, tc, nrm, excess, guess, tally,
                                              can_defer ? &deferred : nullptr, newton);
      if (!done) {  // FP32 cannot decide the pair
        V fd, td, nd;
        if constexpr (PHYS) {
          pair_contact_fused<HIST, JKR>(P, lw, d, d2, rsum, xi4.w, xj4.w, vi4.w, vj4.w, xyz(vi4), xyz(vj4), xyz(wi4),
                                   xyz(wj4), hk, plane, fd, nd, excess, guess, nullptr, nullptr, newton);
          fc = cvt<R>(fd);
          tc = cvt<R>((-xi4.w) * nd);
          tc2 = cvt<R>((-xj4.w) * nd);
        } else {
          pair_contact<double, PHYS, HIST, JKR>(P, lw, d, d2, rsum, xi4.w, xj4.w, vi4.w, vj4.w, xyz(vi4), xyz(vj4),
                                           xyz(wi4), xyz(wj4), hk, plane, fd, td, nd, excess, guess, nullptr,
                                           nullptr, newton);
          fc = cvt<R>(fd);
          tc = cvt<R>(td);
          nrm = cvt<R>(nd);
        }
      }
      if (done || !PHYS) tc2 = cross(nrm * narrow<R>(xj4.w), -fc);
    }
    if (deferred) return true;
    if (HIST && m < 64) atomicOr(B.hmask + k, 1ull << m);
  } else if (HIST) {
    hk[0] = 0.0;
    hk[plane] = 0.0;
    hk[2 * plane] = 0.0;
  }
  if (P.debug) P.dbgMult[hik] = (uint8_t)(in ? vij : 0);
  put_result(P, it.w, fc, tc, vij);
  if (back != NO_RECORD) {
    put_result(P, offj + back, -fc, tc2, vji);
    if (HIST || P.debug) {
      const uint32_t m2 = P.crec[(size_t)j * P.cap + back].mv & 0xFFFFu;
      const size_t h2 = (size_t)j * P.cap + m2;
      if (HIST) {
        B.hist[h2] = -hk[0];
        B.hist[plane + h2] = -hk[plane];
        B.hist[2 * plane + h2] = -hk[2 * plane];
        if (m2 < 64) atomicOr(B.hmask + j, 1ull << m2);
      }
      if (P.debug) P.dbgMult[h2] = (uint8_t)(in ? vji : 0);
    }
  }
  return false;
}

// A wall candidate of the filter: the FP64 sphere-triangle contact
// (src/simulation.rs:464-523); its force and torque are kept for
// k_accumulate, which adds them after the pair contacts in mesh order.
template <bool JKR>
__device__ __forceinline__ void wall_eval(const StepParams& P, const Bank& B, uint32_t w, bool& excess) {
  const uint2 e = P.warena[w];
  const int k = (int)e.x;
  const D4 xi = B.xr[k], vi = B.vm[k], wi = B.wc[k];
  V fc, tc;
  const bool ok = wall_contact<JKR>(P, law_of(P, B, k), P.tri[e.y], xyz(xi), xyz(vi), xyz(wi), xi.w, vi.w, fc, tc, excess);
  if (ok) {
    double2* o = reinterpret_cast<double2*>(P.wres + 6 * (size_t)w);
    o[0] = make_double2(fc.x, fc.y);
    o[1] = make_double2(fc.z, tc.x);
    o[2] = make_double2(tc.y, tc.z);
  }
  P.wok[w] = ok ? 1 : 0;
}

// The JKR tallies of a warp's threads into the control block. Every lane of the
// warp takes part.
__device__ __forceinline__ void add_tally(Ctrl* C, const uint32_t tally[6]) {
  __syncwarp();
#pragma unroll
  for (int q = 0; q < 6; ++q) {
    const uint32_t v = __reduce_add_sync(0xFFFFFFFFu, tally[q]);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(&C->jkr_count[q], (unsigned long long)v);
  }
}

// Pass 3: one thread per evaluating record, then one per wall candidate (the
// few wall contacts spread over the whole grid with the pairs).
template <bool PHYS, bool HIST, typename R, bool JKR>
__device__ __forceinline__ void contact_pass(const StepParams& P, Ctrl* C, const Bank& B, uint32_t* ctot, Span sp) {
  const uint32_t total = ctot[1];
  // the walls start on a warp of their own (a mixed one runs both laws)
  const uint32_t walls = (total + 31u) & ~31u;
  const uint32_t items = P.ntri > 0 ? walls + min(ctot[4], P.wcap) : total;
  bool excess = false;
  uint32_t tally[6] = {0u, 0u, 0u, 0u, 0u, 0u};
  const int lane = threadIdx.x & 31;
  const bool learn = P.jkr_solver == 1 && P.nmodel == 3 && P.mlp != nullptr;
  for (uint32_t t = (uint32_t)sp.at; t < items; t += (uint32_t)sp.all) {
    bool deferred = false;
    if (t < total) {
      deferred = contact_eval<PHYS, HIST, R, JKR>(P, B, P.clist[t], JKR && learn ? P.jguess[t] : -1.0f, JKR && P.jfb != nullptr,
                                                  false, excess, JKR ? tally : nullptr);
    } else if (t >= walls) {
      wall_eval<JKR>(P, B, t - walls, excess);
    }
    if (!JKR) continue;
    // append the deferred pairs with one atomic per warp
    const unsigned act = __activemask();
    const unsigned bal = __ballot_sync(act, deferred);
    if (bal) {
      const int leader = __ffs(bal) - 1;
      uint32_t base = 0;
      if (lane == leader) base = atomicAdd(ctot + 3, (uint32_t)__popc(bal));
      base = __shfl_sync(act, base, leader);
      if (deferred) P.jfb[base + (uint32_t)__popc(bal & ((1u << lane) - 1u))] = t;
    }
  }
  if (excess) C->overlap_flag = 1;
  if (JKR && P.jkr_solver != 0) add_tally(C, tally);
}

template <bool PHYS, bool HIST, typename R, bool JKR>
__global__ void __launch_bounds__(256) k_contact_force(StepParams P) {
  Ctrl* C = P.ctrl;
  if (C->halt) return;
  contact_pass<PHYS, HIST, R, JKR>(P, C, P.bank[C->bank], P.ctot, grid_span());
}

// The pairs that the filter found next to the JKR fold, one thread each: the
// exact certificates decide, and most run the reference's Newton iteration, up
// to 20 steps of ~55 dependent FP64 instructions: ~57 us for a single warp,
// which the whole force pass waited for after the pair kernel. This kernel runs
// beside the network and the pair kernel, which it does not depend on. In the
// mixed form a pair takes the FP32 law first, as the others do, and FP64 for the
// Newton.
template <bool PHYS, bool HIST, typename R>
__global__ void __launch_bounds__(128) k_contact_hard(StepParams P) {
  Ctrl* C = P.ctrl;
  if (C->halt) return;
  const Bank B = P.bank[C->bank];
  const uint32_t total = P.ctot[5];
  bool excess = false;
  uint32_t tally[6] = {0u, 0u, 0u, 0u, 0u, 0u};
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const uint4 it = P.jhard[i];
    constexpr bool f32 = sizeof(R) == sizeof(float);
    const bool deferred = contact_eval<PHYS, HIST, R, true>(P, B, it, -1.0f, f32, false, excess, tally);
    if (f32 && deferred) contact_eval<PHYS, HIST, double, true>(P, B, it, -1.0f, false, true, excess, nullptr);
  }
  if (excess) C->overlap_flag = 1;
  add_tally(C, tally);
}

// The deferred pairs of k_contact_force (few: the filter's hint sends most of
// their kind to k_contact_hard), one thread each, with the reference's Newton
// iteration for their JKR force.
template <bool PHYS, bool HIST>
__global__ void __launch_bounds__(128) k_contact_deferred(StepParams P) {
  Ctrl* C = P.ctrl;
  if (C->halt) return;
  const Bank B = P.bank[C->bank];
  const uint32_t total = P.ctot[3];
  bool excess = false;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x)
    contact_eval<PHYS, HIST, double, true>(P, B, P.clist[P.jfb[i]], -1.0f, false, true, excess, nullptr);
  if (excess) C->overlap_flag = 1;
}

// Pass 4: per particle, the contact results in list order, then the wall
// contacts in mesh order, then a = g + F/m and tau = T
// (src/simulation.rs:265-271, 464-536). The wall candidates were listed by
// the filter (FP32 pretests against the triangles of the particle's
// triangle-grid cell) and evaluated by the pair kernel, one thread each, so
// F and T are the same sums as one thread walking its triangles.
// k_accumulate takes the slots in the order P.aorder, set at each list
// rebuild, so that a warp's lanes run loops of similar length; no order
// changes a result.
constexpr uint32_t ACC_BINS = 128;
constexpr uint32_t ACC_TILE = 256;
constexpr int ACC_DEAL = 256;           // slots a block deals to its threads at a time
constexpr uint32_t ACC_SORT_BINS = 32;  // record counts up to 31 (more share the last bin)

__device__ __forceinline__ bool tri_cell_nonempty(const StepParams& P, float4 xf) {
  uint32_t s, e;
  return tri_cell_range(P, xf, s, e) && e > s;
}

// Whether no triangle can come within reach of a particle at xf (its
// position at a list rebuild) before the next rebuild: until then it moves
// less than half the skin, which is less than a triangle-grid cell
// (wall_far_ok), so its cell stays among the 27 around the present one, and
// all of those list no triangle; nor can it wrap across a periodic face,
// which moves it to another part of the mesh.
__device__ bool wall_far(const StepParams& P, float4 xf) {
  const float p[3] = {xf.x, xf.y, xf.z};
  float q[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    if (P.periodic[a]) {
      const float lo = (float)P.bmin[a], hi = (float)P.bmax[a];
      if (!(p[a] - lo > P.wall_far_gap && hi - p[a] > P.wall_far_gap)) return false;
    }
    q[a] = floorf((p[a] - P.tminf[a]) * P.tinvf);
    if (!(q[a] == q[a])) return false;  // NaN
    if (q[a] + 1.0f < 0.0f || q[a] - 1.0f >= (float)P.tdims[a]) return true;  // the 27 cells lie outside the grid
  }
  for (int dz = -1; dz <= 1; ++dz)
    for (int dy = -1; dy <= 1; ++dy)
      for (int dx = -1; dx <= 1; ++dx) {
        const int cx = (int)q[0] + dx, cy = (int)q[1] + dy, cz = (int)q[2] + dz;
        if (cx < 0 || cy < 0 || cz < 0 || cx >= P.tdims[0] || cy >= P.tdims[1] || cz >= P.tdims[2]) continue;
        const uint32_t cell = (uint32_t)cx + (uint32_t)P.tdims[0] * ((uint32_t)cy + (uint32_t)P.tdims[1] * (uint32_t)cz);
        if (P.tstart[cell + 1] > P.tstart[cell]) return false;
      }
  return true;
}

// PF_NOIMAGE and PF_ONECELL of a particle at xf (its position at a list
// rebuild) with reference-cell code c: whether a partner within reach can be a
// periodic image, or lie in another reference cell, before the next rebuild.
// Until then each of the two moves less than half the skin, so a partner that
// is within the cutoff then lies within cutoff + skin / 2 of the particle's
// position now, and the particle's own cell changes only across that distance
// too; home_margin covers the rounding of the mirror and of the pretest. A
// partner may lie up to `out` beyond a periodic face at the rebuild (and no
// farther than half the skin later).
__device__ uint32_t home_flags(const StepParams& P, float4 xf, long long c, float out) {
  const float p[3] = {xf.x, xf.y, xf.z};
  const float reach = (xf.w + P.rmaxf) * P.cut_a + (float)P.skin + P.home_margin;
  // without the pretest every row entry is a candidate, however far it has
  // moved: the cells of both decide whether it counts
  uint32_t f = P.pretest ? PF_NOIMAGE | PF_ONECELL : 0u;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float lo = (float)P.bmin[a], hi = (float)P.bmax[a];
    if (P.periodic[a] && !(p[a] - lo > reach + out && hi - p[a] > reach + out)) f = 0u;
    const float q = (p[a] - lo) * (float)P.inv_href, r = reach * (float)P.inv_href;
    const float g = floorf(q);
    if (!(g >= 0.0f && g < (float)P.rdims[a] && q - g > r && (g + 1.0f) - q > r &&
          (int)g == code_axis((unsigned long long)c, a)))
      f &= ~PF_ONECELL;
  }
  return f;
}

// The visiting order of k_accumulate, at a list rebuild: within each tile of
// 256 slots a counting sort by (triangles listed in the triangle-grid cell,
// Verlet-list length), dead slots after the live ones. Reads the bank the
// rebuild fills.
__global__ void __launch_bounds__(ACC_TILE) k_accum_order(StepParams P) {
  {
    volatile const Ctrl* c = P.ctrl;
    if (c->rebuild == 0 || c->halt != 0) return;
  }
  const Bank B = P.bank[P.ctrl->bank ^ 1];
  __shared__ uint32_t bins[ACC_BINS];
  for (int base = blockIdx.x * ACC_TILE; base < P.n; base += gridDim.x * ACC_TILE) {
    const int k0 = base + threadIdx.x;
    // keys: 0..62 no triangles, 63 dead, 64..126 triangles, 127 past the end
    uint32_t key = ACC_BINS - 1;
    if (k0 < P.n) {
      const uint32_t fl = B.flags[k0];
      if (fl & PF_DEAD) {
        key = 63;
      } else {
        key = min(B.ncnt[k0], 62u);
        const float4 xf = B.xf[k0];
        if (P.ntri > 0 && tri_cell_nonempty(P, xf)) key += 64;
        const bool far = P.ntri > 0 && P.wall_far_ok && wall_far(P, xf);
        const uint32_t home = home_flags(P, xf, __double_as_longlong(B.wc[k0].w), __uint_as_float(P.ctrl->xout));
        B.flags[k0] = (fl & ~(PF_WALLFAR | PF_NOIMAGE | PF_ONECELL)) | (far ? PF_WALLFAR : 0u) | home;
      }
    }
    for (uint32_t i = threadIdx.x; i < ACC_BINS; i += blockDim.x) bins[i] = 0;
    __syncthreads();
    const uint32_t rank = atomicAdd(&bins[key], 1u);
    __syncthreads();
    if (threadIdx.x < 32) {  // exclusive scan of the bins, four per lane
      const uint32_t l = threadIdx.x;
      const uint32_t c0 = bins[4 * l], c1 = bins[4 * l + 1], c2 = bins[4 * l + 2], c3 = bins[4 * l + 3];
      const uint32_t sum = c0 + c1 + c2 + c3;
      uint32_t incl = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (l >= (uint32_t)o) incl += t;
      }
      const uint32_t ex = incl - sum;
      bins[4 * l] = ex;
      bins[4 * l + 1] = ex + c0;
      bins[4 * l + 2] = ex + c0 + c1;
      bins[4 * l + 3] = ex + c0 + c1 + c2;
    }
    __syncthreads();
    if (k0 < P.n) P.aorder[base + bins[key] + rank] = (uint32_t)k0;
    __syncthreads();
  }
}

int launch_accum_order(const StepParams& P, cudaStream_t s) {
  const uint64_t tiles = ((uint64_t)P.n + ACC_TILE - 1) / ACC_TILE;
  k_accum_order<<<(int)std::min<uint64_t>(std::max<uint64_t>(tiles, 1), (uint64_t)P.nsm * 64ull), ACC_TILE, 0, s>>>(P);
  return 1;
}

// a = g + F (1/m) and tau = 0 + T for one particle, with the debug record and
// the non-finite check (on the integer pipe, as the +0 of 0 + T).
__device__ __forceinline__ void finish_particle(const StepParams& P, const Bank& B, Ctrl* C, int k, V F, V T) {
  if (P.debug) {
    P.dbgF[3 * (size_t)k] = F.x; P.dbgF[3 * (size_t)k + 1] = F.y; P.dbgF[3 * (size_t)k + 2] = F.z;
    P.dbgT[3 * (size_t)k] = T.x; P.dbgT[3 * (size_t)k + 1] = T.y; P.dbgT[3 * (size_t)k + 2] = T.z;
  }
  if (!(finite_bits(F.x) & finite_bits(F.y) & finite_bits(F.z) & finite_bits(T.x) & finite_bits(T.y) &
        finite_bits(T.z)))
    atomicOr(&C->status, (unsigned)ST_NAN);
  const V a = vmk(P.gravity[0], P.gravity[1], P.gravity[2]) + F * B.vres[k].w;  // F (1/m)
  B.acc[k] = D4{a.x, a.y, a.z, 0.0};
  B.tq[k] = D4{plus_zero(T.x), plus_zero(T.y), plus_zero(T.z), 0.0};
}

// One particle's contact results: FP64 records (the FP64 form) or FP32 records
// (the mixed form, whose pair forces are FP32 values), in list order, then its
// wall results in mesh order.
template <bool F32REC>
__device__ __forceinline__ void sum_particle(const StepParams& P, const Bank& B, Ctrl* C, int k) {
  V F = vmk(0.0, 0.0, 0.0), T = vmk(0.0, 0.0, 0.0);
  const uint32_t n = P.ccnt[k];
  if (F32REC) {
    // the mixed form's FP32 pair forces summed in FP32 (in list order, from
    // zero; the rounding adds at most (n - 1) 2^-24 of the sum of the
    // magnitudes), then widened exactly
    const float2* res = reinterpret_cast<const float2*>(P.cresf + 6 * (size_t)P.coff[k]);
    float fx = 0.0f, fy = 0.0f, fz = 0.0f, tx = 0.0f, ty = 0.0f, tz = 0.0f;
    for (uint32_t c = 0; c < n; ++c) {
      const float2 r0 = res[3 * c], r1 = res[3 * c + 1], r2 = res[3 * c + 2];
      fx = fx + r0.x; fy = fy + r0.y; fz = fz + r1.x;
      tx = tx + r1.y; ty = ty + r2.x; tz = tz + r2.y;
    }
    F = vmk(f2d_exact(fx), f2d_exact(fy), f2d_exact(fz));
    T = vmk(f2d_exact(tx), f2d_exact(ty), f2d_exact(tz));
  } else {
    // the next record's loads are in flight while this one is added; one record
    // a round, because an unrolled loop predicates its remainder, and a
    // predicated-off FP64 instruction takes the pipe as long as a full one
    // (million-sphere hopper: 1.25 to 0.98 million warp instructions, 92 to 76 us)
    const double2* res = reinterpret_cast<const double2*>(P.cres + 6 * (size_t)P.coff[k]);
    double2 a0, a1, a2;
    if (n > 0) { a0 = res[0]; a1 = res[1]; a2 = res[2]; }
#pragma unroll 1
    for (uint32_t c = 0; c < n; ++c) {
      const double2 r0 = a0, r1 = a1, r2 = a2;
      if (c + 1 < n) { a0 = res[3 * c + 3]; a1 = res[3 * c + 4]; a2 = res[3 * c + 5]; }
      F = F + vmk(r0.x, r0.y, r1.x);
      T = T + vmk(r1.y, r2.x, r2.y);
    }
  }
  // the wall contacts (FP64 in both forms) after the pair contacts, in mesh order
  if (P.ntri > 0) {
    const uint32_t wn = P.wcnt[k], wo = P.woff[k];
#pragma unroll 1
    for (uint32_t c = 0; c < wn; ++c) {
      const double2* r = reinterpret_cast<const double2*>(P.wres + 6 * (size_t)(wo + c));
      const bool ok = P.wok[wo + c] != 0;
      const double2 r0 = r[0], r1 = r[1], r2 = r[2];
      if (!ok) continue;
      F = F + vmk(r0.x, r0.y, r1.x);
      T = T + vmk(r1.y, r2.x, r2.y);
    }
  }
  finish_particle(P, B, C, k, F, T);
}

// Threads take the slots in the order aorder gives (tiles of 256 sorted by
// list length, particles in triangle cells last).
template <bool F32REC>
__global__ void __launch_bounds__(256, 5) k_accumulate(StepParams P) {
  Ctrl* C = P.ctrl;
  if (C->halt) return;
  const Bank B = P.bank[C->bank];
  // Each block takes a tile of ACC_DEAL slots (in aorder) and deals them to its
  // threads by their record and wall counts (a counting sort in shared memory),
  // so the lanes of a warp run sum loops of about the same length: a partly
  // filled FP64 warp instruction costs the pipe as much as a full one. 256 slots
  // for 128 threads: 128 left more lanes idle (hopper 656 against 654 us a step,
  // 2.1 million adhesive spheres 1222 against 1215), 512 and 1024 read farther
  // apart and end in a thinner last wave (661 and 666; 1218 and 1249).
  __shared__ uint32_t bins[ACC_SORT_BINS];
  __shared__ int slot[ACC_DEAL], dealt[ACC_DEAL];
  __shared__ uint32_t place[ACC_DEAL];  // key, rank among its equals
  for (int base = blockIdx.x * ACC_DEAL; base < P.n; base += gridDim.x * ACC_DEAL) {
    for (uint32_t b = threadIdx.x; b < ACC_SORT_BINS; b += blockDim.x) bins[b] = 0;
    __syncthreads();
    for (int o = threadIdx.x; o < ACC_DEAL; o += blockDim.x) {
      int k = -1;
      uint32_t key = 0;
      if (base + o < P.n) {
        k = (int)P.aorder[base + o];
        if (B.flags[k] & PF_DEAD) k = -1;
        else key = min(P.ccnt[k] + (P.ntri > 0 ? P.wcnt[k] : 0u), ACC_SORT_BINS - 1);
      }
      slot[o] = k;
      place[o] = key | atomicAdd(&bins[key], 1u) << 8;
    }
    __syncthreads();
    if (threadIdx.x < 32) {  // exclusive scan of the bins, one per lane
      const uint32_t c0 = bins[threadIdx.x];
      uint32_t incl = c0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (threadIdx.x >= (uint32_t)o) incl += t;
      }
      bins[threadIdx.x] = incl - c0;
    }
    __syncthreads();
    for (int o = threadIdx.x; o < ACC_DEAL; o += blockDim.x) dealt[bins[place[o] & 0xFFu] + (place[o] >> 8)] = slot[o];
    __syncthreads();
    for (int o = threadIdx.x; o < ACC_DEAL; o += blockDim.x) {
      const int k = dealt[o];
      if (k >= 0) sum_particle<F32REC>(P, B, C, k);
    }
  }
}

// ------------------------------------------------------ many steps, one launch
// A small bed's step is a chain of dependent latencies, not work: eight graph
// nodes of 1,000 spheres take 53 us a step, with one warp in each FP64 unit at
// most. k_steps runs the step's passes in one cooperative launch, three grid
// barriers apart, step after step, until the target is reached, the lists must
// be rebuilt (the graph runs the chain and launches it again; Ctrl::resume says
// that the first half of the current step has been done) or a buffer is full.
// The sums of a step and the first half of the next are one quad's, so no
// barrier lies between them: 1,000 spheres take 25 us a step.
// The launch fits the device at once (cooperative); every wait is bounded, and
// one that runs out halts the simulation with an error.
constexpr unsigned SMALL_SPINS = 1u << 20;      // ~1 s
constexpr unsigned SMALL_STEPS = 4096;          // steps a launch
constexpr int SMALL_BLOCK = 512;                // threads a block at most, one block a multiprocessor
// Particles taken by four lanes each: below one quad warp for every other FP64
// unit (608 x 8 particles) the integrator is a quarter as long, at 16,000 the
// extra loads cost what it saves (us a step with quads / without: 1,000 spheres
// 26.2 / 30.3, 8,000 32.7 / 32.2, 16,000 49.1 / 43.7, one item order for both).
constexpr int QUAD_MAX = 8192;
// Particles: up to here a launch of many steps is the faster loop on every bed
// measured (us a step, this / eight graph nodes: Hertz + Coulomb FP64 box 1,000
// 26 / 48, 24,000 32.5 / 55, 100,000 78 / 98, 250,000 171 / 179, 400,000 264 /
// 256; mixed bed 250,000 167 / 183, 800,000 482 / 462; linear springs 250,000
// 303 / 314, 800,000 891 / 873). Above, a kernel for each pass holds fewer
// registers and more warps.
constexpr int SMALL_MAX = 262144;

__device__ __forceinline__ unsigned load_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// All blocks of the launch (`blocks`); `gen` counts the barriers passed. False
// when the others did not arrive in time.
__device__ __forceinline__ bool grid_barrier(Ctrl* C, unsigned& gen, unsigned blocks) {
  __shared__ int ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    ++gen;
    const unsigned want = gen * blocks;
    asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(&C->bar), "r"(1u) : "memory");
    bool here = load_acquire(&C->bar) >= want;
    for (unsigned n = 0; !here && n < SMALL_SPINS; ++n) here = load_acquire(&C->bar) >= want;
    if (!here) {
      atomicOr(&C->halt, HALT_STUCK);
      atomicOr(&C->status, (unsigned)ST_STUCK);
    }
    ok = here;
  }
  __syncthreads();
  return ok != 0;
}

// first_half_pass and sum_particle with four lanes a particle: lane c < 3 holds
// component c of every vector, lane 3 the fourth words (mass, radius, cell code,
// 1/m, 1/I). A warp instruction takes the FP64 unit of a partition 66 clocks
// whatever its lanes do, so with less than a warp for each unit the integrator's
// ~90 FP64 instructions become ~28 and a record's sum two instead of six. The
// operations of each component and their order are those of the scalar passes.
__device__ __forceinline__ double quad_word(double v, int word) { return __shfl_sync(0xFFFFFFFFu, v, word, 4); }
__device__ __forceinline__ float quad_word(float v, int word) { return __shfl_sync(0xFFFFFFFFu, v, word, 4); }
__device__ __forceinline__ unsigned quad_mask() { return 7u << (threadIdx.x & 28); }  // the three components' lanes
__device__ __forceinline__ void kahan_add(double& s, double& r, double d) {
  const double y = d - r;
  const double t = s + y;
  r = (t - s) - y;
  s = t;
}
template <typename A>
__device__ __forceinline__ A pick(int c, const A* v) {  // v[c] without an indexed parameter read; 0 for lane 3
  return c == 0 ? v[0] : c == 1 ? v[1] : c == 2 ? v[2] : A(0);
}

// The first half of the warp's particles k (one a quad; on: it exists), whole
// warps only; returns whether the particle asks for a rebuild.
template <bool KAHAN>
__device__ __forceinline__ bool first_half_quad(const StepParams& P, Ctrl* C, const Bank& B, bool fuse, int k, bool on) {
  constexpr unsigned ALL = 0xFFFFFFFFu;
  const int c = threadIdx.x & 3;
  const bool part = c < 3;
  const size_t at = 4 * (size_t)k + c;
  uint32_t fl = on ? B.flags[k] : PF_DEAD;
  on = !(fl & PF_DEAD);
  const bool moving = on && !(fl & PF_FIXED);
  double x = 0.0, v = 0.0, w = 0.0, a = 0.0, tau = 0.0, vres = 0.0, wres = 0.0, xres = 0.0;
  float xo = 0.0f, ref = 0.0f;
  if (on) {
    x = reinterpret_cast<const double*>(B.xr)[at];
    v = reinterpret_cast<const double*>(B.vm)[at];
    w = reinterpret_cast<const double*>(B.wc)[at];
    xo = reinterpret_cast<const float*>(B.xf)[at];
    ref = reinterpret_cast<const float*>(B.xref)[at];
    if (moving) {
      a = reinterpret_cast<const double*>(B.acc)[at];
      tau = reinterpret_cast<const double*>(B.tq)[at];
      wres = reinterpret_cast<const double*>(B.wres)[at];
      if (KAHAN) {
        vres = reinterpret_cast<const double*>(B.vres)[at];
        xres = reinterpret_cast<const double*>(B.xres)[at];
      }
    }
  }
  const double dt = P.dt, hdt = P.hdt, inv_inertia = quad_word(wres, 3);
  const unsigned spinning = __ballot_sync(ALL, moving && (!is_zero(tau) || (KAHAN && !is_zero(wres)) || (fl & PF_KICK)));
  const bool own_spin = (spinning & quad_mask()) != 0;
  const double kdt = (!KAHAN && fuse) ? dt : hdt;
  const double dv = a * kdt;
  const double dw = KAHAN ? (tau * inv_inertia) * kdt : tau * (inv_inertia * kdt);
  if (KAHAN && fuse && moving && part) {
    kahan_add(v, vres, dv);
    if (own_spin) kahan_add(w, wres, dw);
  }
  // wrap and removal, each lane its axis
  const bool per = pick(c, P.periodic) != 0;
  const double lo = pick(c, P.bmin), hi = pick(c, P.bmax);
  const bool inner = !part || (xo > pick(c, P.inner_lo) && xo < pick(c, P.inner_hi));
  bool keep = true;
  if (part && !inner) {
    if (per) {
      const double size = pick(c, P.bsize);
      if (x < lo) x = x + size;
      else if (x >= hi) x = x - size;
    } else {
      keep = c == 1 ? x >= lo - 1.0 : (x >= lo - 1.0 && x <= hi + 1.0);
    }
  }
  const unsigned leaving = __ballot_sync(ALL, on && !keep);  // every lane takes part
  const bool gone = on && (leaving & quad_mask()) != 0;
  if (gone) {
    if (part) {
      reinterpret_cast<double*>(B.xr)[at] = __longlong_as_double(0x7ff8000000000000ll);
      reinterpret_cast<float*>(B.xf)[at] = __int_as_float(0x7fc00000);
    } else {
      B.flags[k] = fl | PF_DEAD;
      atomicAdd(&C->removed, 1ull);
    }
    on = false;
  }
  const bool move = moving && !gone && part;
  if (move) {
    if (KAHAN) {
      kahan_add(v, vres, dv);
      kahan_add(x, xres, v * dt);
      reinterpret_cast<double*>(B.vres)[at] = vres;
      reinterpret_cast<double*>(B.xres)[at] = xres;
      if (own_spin) {
        kahan_add(w, wres, dw);
        reinterpret_cast<double*>(B.wres)[at] = wres;
      }
    } else {
      v = v + dv;
      x = x + v * dt;
      if (own_spin) w = w + dw;
    }
    reinterpret_cast<double*>(B.vm)[at] = v;
    if (own_spin) reinterpret_cast<double*>(B.wc)[at] = w;
  }
  const float xf = (float)x;
  if (on && part) {
    reinterpret_cast<double*>(B.xr)[at] = x;
    reinterpret_cast<float*>(B.xf)[at] = xf;
  }
  if (P.mode == 0) {
    int32_t q = 0;
    if (on && part) q = ref_axis_fast(x, xf, lo, pick(c, P.bminf), P.href, P.inv_href, P.inv_hreff);
    const int32_t c0 = __shfl_sync(ALL, q, 0, 4), c1 = __shfl_sync(ALL, q, 1, 4), c2 = __shfl_sync(ALL, q, 2, 4);
    if (on && !part) {
      const unsigned long long code = pack_code(c0, c1, c2);
      if (code != (unsigned long long)__double_as_longlong(w))
        reinterpret_cast<double*>(B.wc)[at] = __longlong_as_double((long long)code);
    }
  }
  const float mag = fabsf(xf);
  const unsigned top = __reduce_max_sync(ALL, on && part && mag >= 0.0f ? __float_as_uint(mag) : 0u);
  if ((threadIdx.x & 31) == 0 && top > C->xmax) atomicMax(&C->xmax, top);
  float d = xf - ref;
  if (per) {
    const float size = pick(c, P.bsizef);
    d -= size * rintf(d / size);
  }
  d = d * d;
  const float d2 = quad_word(d, 0) + quad_word(d, 1) + quad_word(d, 2);
  return on && !(d2 <= P.half_skinf * P.half_skinf);
}

// The sums, a and tau of particle k (one a quad, whole warps).
template <bool F32REC>
__device__ __forceinline__ void sum_quad(const StepParams& P, const Bank& B, Ctrl* C, int k, bool on) {
  const int c = threadIdx.x & 3;
  on = on && !(B.flags[on ? k : 0] & PF_DEAD);
  if (!on || c == 3) return;
  double F = 0.0, T = 0.0;
  const uint32_t n = P.ccnt[k], off = P.coff[k];
  const double inv_mass = B.vres[k].w;
  if (F32REC) {
    const float* res = P.cresf + 6 * (size_t)off + c;
    float f = 0.0f, t = 0.0f, f1 = 0.0f, t1 = 0.0f;
    if (n > 0) { f1 = res[0]; t1 = res[3]; }
    for (uint32_t q = 0; q < n; ++q) {
      const float f0 = f1, t0 = t1;
      if (q + 1 < n) { f1 = res[6 * q + 6]; t1 = res[6 * q + 9]; }
      f = f + f0;
      t = t + t0;
    }
    F = f2d_exact(f);
    T = f2d_exact(t);
  } else {
    const double* res = P.cres + 6 * (size_t)off + c;
    double f1 = 0.0, t1 = 0.0;
    if (n > 0) { f1 = res[0]; t1 = res[3]; }
    for (uint32_t q = 0; q < n; ++q) {
      const double f0 = f1, t0 = t1;
      if (q + 1 < n) { f1 = res[6 * q + 6]; t1 = res[6 * q + 9]; }
      F = F + f0;
      T = T + t0;
    }
  }
  if (P.ntri > 0) {
    const uint32_t wn = P.wcnt[k], wo = P.woff[k];
    for (uint32_t q = 0; q < wn; ++q) {
      const bool ok = P.wok[wo + q] != 0;
      const double f0 = P.wres[6 * (size_t)(wo + q) + c], t0 = P.wres[6 * (size_t)(wo + q) + 3 + c];
      if (!ok) continue;
      F = F + f0;
      T = T + t0;
    }
  }
  if (P.debug) {
    P.dbgF[3 * (size_t)k + c] = F;
    P.dbgT[3 * (size_t)k + c] = T;
  }
  if (!(finite_bits(F) & finite_bits(T))) atomicOr(&C->status, (unsigned)ST_NAN);
  reinterpret_cast<double*>(B.acc)[4 * (size_t)k + c] = pick(c, P.gravity) + F * inv_mass;
  reinterpret_cast<double*>(B.tq)[4 * (size_t)k + c] = plus_zero(T);
}

template <bool PHYS, bool HIST, typename R>
__global__ void __launch_bounds__(SMALL_BLOCK, 1) k_steps(StepParams P) {
  Ctrl* C = P.ctrl;
  volatile Ctrl* W = C;
  // (a resumed launch filters before its first barrier: a full buffer that
  // another block reports meanwhile must not keep this one from the barrier)
  if (W->halt & (HALT_LISTS | HALT_STUCK)) return;
  constexpr bool FP64 = sizeof(R) == sizeof(double);
  const Bank B = P.bank[C->bank];
  const unsigned long long target = C->target;
  unsigned long long done = C->steps_done;
  bool fuse = C->pending != 0, resume = C->resume != 0;
  const bool first = blockIdx.x == 0 && threadIdx.x == 0;
  const bool quads = P.n <= QUAD_MAX;
  // consecutive warps of items go to consecutive blocks, so few items occupy
  // one FP64 unit each of as many multiprocessors as there are
  const int lane = threadIdx.x & 31;
  const Span sp{(int)((threadIdx.x >> 5) * gridDim.x + blockIdx.x) * 32 + lane, (int)(gridDim.x * blockDim.x)};
  const int quad0 = (sp.at - lane) >> 2, quad_all = sp.all >> 2;  // of the warp
  unsigned gen = 0;
  const unsigned blocks = gridDim.x + (unsigned)P.absent_blocks;
  for (unsigned s = 0; s < SMALL_STEPS && done < target; ++s) {
    uint32_t* ctot = P.ctot + (s & 1u) * CTOT_WORDS;
    if (!resume) {
      bool rebuild = false;
      if (quads) {
        for (int b = quad0; b < P.n; b += quad_all) {
          const int k = b + (lane >> 2);
          rebuild |= first_half_quad<FP64>(P, C, B, fuse, k, k < P.n);
        }
      } else {
        rebuild = first_half_pass<FP64, true>(P, C, B, fuse, sp);
      }
      if (rebuild) W->rebuild = 1;
      if (!grid_barrier(C, gen, blocks)) return;
      if (W->rebuild) {
        if (first) W->resume = 1;
        return;
      }
    }
    resume = false;
    filter_pass<PHYS, HIST, true>(P, C, B, ctot, sp);
    if (!grid_barrier(C, gen, blocks)) return;
    if (W->halt) {  // a buffer of the filter is full: the host finishes this step
      if (first) W->resume = 0;
      return;
    }
    contact_pass<PHYS, HIST, R, false>(P, C, B, ctot, sp);
    // the next step's counters, last read two barriers ago
    if (blockIdx.x == 0 && threadIdx.x < CTOT_WORDS) P.ctot[((s + 1u) & 1u) * CTOT_WORDS + threadIdx.x] = 0u;
    if (!grid_barrier(C, gen, blocks)) return;
    if (quads) {
      for (int b = quad0; b < P.n; b += quad_all) {
        const int k = b + (lane >> 2);
        sum_quad<!FP64>(P, B, C, k, k < P.n);
      }
      __syncwarp();  // the quad's next first half reads what its lanes wrote
    } else {
      for (int k = sp.at; k < P.n; k += sp.all)
        if (!(B.flags[k] & PF_DEAD)) sum_particle<!FP64>(P, B, C, k);
    }
    ++done;
    fuse = true;
    if (first) {
      W->steps_done = done;
      W->pending = 1;
      W->resume = 0;
      if (W->overlap_flag) {
        W->overlap_steps = W->overlap_steps + 1;
        W->overlap_flag = 0;
        atomicOr(&C->status, (unsigned)ST_OVERLAP);
      }
    }
  }
}

// After k_steps: whether the rebuild chain runs (IF node), then whether the
// loop goes on. An iteration completes a step or rebuilds the lists for one, so
// the loop ends after 2 target + 8 iterations whatever the counters say.
__global__ void k_steps_next(StepParams P, cudaGraphConditionalHandle rebuild, cudaGraphConditionalHandle loop, int end) {
  Ctrl* C = P.ctrl;
  if (!end) {
    C->bar = 0;
    for (int q = 0; q < 2 * CTOT_WORDS; ++q) P.ctot[q] = 0;
    cudaGraphSetConditional(rebuild, (C->rebuild && !C->halt) ? 1u : 0u);
    return;
  }
  C->iters += 1;
  const bool again = !C->halt && C->steps_done < C->target && C->iters < 2 * C->target + 8;
  cudaGraphSetConditional(loop, again ? 1u : 0u);
}

__global__ void k_clear_pending(StepParams P) {
  Ctrl* C = P.ctrl;
  if (!C->halt && C->steps_done >= C->target) C->pending = 0;
}

// End of a step: count it and, inside the device step loop, decide whether
// the loop runs again. The loop also stops on a halt and after target + 4
// iterations whatever the counters say, so it always terminates.
__global__ void k_end_step(StepParams P, cudaGraphConditionalHandle loop, int in_loop) {
  Ctrl* C = P.ctrl;
  if (!C->halt) {
    C->steps_done += 1;
    C->pending = 1;
    C->resume = 0;
    C->spin_due = 0;
    if (C->overlap_flag) {
      C->overlap_steps += 1;
      C->status |= ST_OVERLAP;
      C->overlap_flag = 0;
    }
  }
  if (in_loop) {
    C->iters += 1;
    const bool again = !C->halt && C->steps_done < C->target && C->iters < C->target + 4;
    cudaGraphSetConditional(loop, again ? 1u : 0u);
  }
}

// Inside the device step loop: run the rebuild chain only when requested.
__global__ void k_rebuild_condition(StepParams P, cudaGraphConditionalHandle h) {
  const Ctrl* C = P.ctrl;
  cudaGraphSetConditional(h, (C->rebuild && !C->halt) ? 1u : 0u);
}

__global__ void k_kinetic(StepParams P, double* out) {
  const Bank B = P.bank[P.ctrl->bank];
  double e = 0.0;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < P.n; k += gridDim.x * blockDim.x) {
    if (B.flags[k] & PF_DEAD) continue;
    D4 v = B.vm[k], w = B.wc[k], x = B.xr[k];
    double I = 0.4 * v.w * x.w * x.w;
    e += 0.5 * v.w * (v.x * v.x + v.y * v.y + v.z * v.z) + 0.5 * I * (w.x * w.x + w.y * w.y + w.z * w.z);
  }
  for (int o = 16; o > 0; o >>= 1) e += __shfl_down_sync(0xFFFFFFFFu, e, o);
  if ((threadIdx.x & 31) == 0) atomicAdd(out, e);
}

// Bed statistics of the live slots: out[0] kinetic energy (translational and
// rotational, I = 2/5 m r^2), out[1] the summed sphere volumes, *pairs the
// overlapping pairs counted from both ends over the Verlet lists (the exact
// FP64 test d^2 < (r_i + r_j)^2 on the minimum image; every such pair is in
// the lists, which reach beyond r_i + r_j by the skin at least).
__global__ void k_bed_stats(StepParams P, double* out, unsigned long long* pairs) {
  const Bank B = P.bank[P.ctrl->bank];
  double e = 0.0, vol = 0.0;
  unsigned long long cnt = 0;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < P.n; k += gridDim.x * blockDim.x) {
    if (B.flags[k] & PF_DEAD) continue;
    const D4 v = B.vm[k], w = B.wc[k], x = B.xr[k];
    const double I = 0.4 * v.w * x.w * x.w;
    e += 0.5 * v.w * (v.x * v.x + v.y * v.y + v.z * v.z) + 0.5 * I * (w.x * w.x + w.y * w.y + w.z * w.z);
    vol += (4.0 / 3.0) * kPi * x.w * x.w * x.w;
    const uint32_t* row = B.nbr + (size_t)k * P.cap;
    const uint32_t c = B.ncnt[k];
    for (uint32_t m = 0; m < c; ++m) {
      const D4 y = B.xr[row[m]];
      const V d = mic(P, xyz(x) - xyz(y));
      const double rs = x.w + y.w;
      if (dot(d, d) < rs * rs) ++cnt;
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    e += __shfl_down_sync(0xFFFFFFFFu, e, o);
    vol += __shfl_down_sync(0xFFFFFFFFu, vol, o);
    cnt += __shfl_down_sync(0xFFFFFFFFu, cnt, o);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(&out[0], e);
    atomicAdd(&out[1], vol);
    atomicAdd(pairs, cnt);
  }
}

void launch_bed_stats(const StepParams& P, double* out, unsigned long long* pairs, cudaStream_t s) {
  cudaMemsetAsync(out, 0, 2 * sizeof(double), s);
  cudaMemsetAsync(pairs, 0, sizeof(unsigned long long), s);
  if (P.n == 0) return;
  k_bed_stats<<<grid_for(P.n, 256), 256, 0, s>>>(P, out, pairs);
}

int launch_first_half(const StepParams& P, cudaStream_t s, bool spin_later) {
  if (P.n == 0) return 0;
  // the Kahan form holds 90 registers: blocks of 128 keep 20 warps resident
  // per multiprocessor where blocks of 256 keep 16
  if (P.prec == 1) k_first_half<false, true><<<grid_for(P.n, 256), 256, 0, s>>>(P);
  else if (spin_later) k_first_half<true, false><<<grid_for(P.n, 128), 128, 0, s>>>(P);
  else k_first_half<true, true><<<grid_for(P.n, 128), 128, 0, s>>>(P);
  return 1;
}

int launch_second_half(const StepParams& P, cudaStream_t s) {
  if (P.n == 0) return 0;
  if (P.prec == 1) k_second_half<false><<<grid_for(P.n, 256), 256, 0, s>>>(P);
  else k_second_half<true><<<grid_for(P.n, 256), 256, 0, s>>>(P);
  k_clear_pending<<<1, 1, 0, s>>>(P);
  return 2;
}

int launch_rebuild_condition(const StepParams& P, cudaGraphConditionalHandle h, cudaStream_t s) {
  k_rebuild_condition<<<1, 1, 0, s>>>(P, h);
  return 1;
}

template <typename R, bool JKR>
static void launch_force_t(const StepParams& P, int g, cudaStream_t s) {
  const bool hist = P.mode == 1 && P.tmodel != 0;
  if (P.mode == 0) k_force<false, false, R, JKR><<<g, 128, 0, s>>>(P);
  else if (hist) k_force<true, true, R, JKR><<<g, 128, 0, s>>>(P);
  else k_force<true, false, R, JKR><<<g, 128, 0, s>>>(P);
}

// Grid for a grid-stride kernel of block `bs` over n items, at most `cap` blocks.
static int shaped_grid(uint64_t n, int bs, int cap) {
  uint64_t g = (n + (uint64_t)bs - 1) / (uint64_t)bs;
  if (g < 1) g = 1;
  if (g > (uint64_t)cap) g = (uint64_t)cap;
  return (int)g;
}

template <typename R, bool JKR>
static int launch_contact_path(const StepParams& P, cudaStream_t s, const SideStream& side) {
  const int bf = P.bs_filter > 0 ? P.bs_filter : 128, bc = P.bs_force > 0 ? P.bs_force : 128,
            ba = P.bs_accum > 0 ? P.bs_accum : 128, cap = P.grid_cap > 0 ? P.grid_cap : P.nsm * 64;
  const int g = shaped_grid((uint64_t)P.n, bf, cap);
  const bool hist = P.mode == 1 && P.tmodel != 0;
  cudaMemsetAsync(P.ctot, 0, sizeof(uint32_t) * CTOT_WORDS, s);
  if (P.mode == 0) k_contact_filter<false, false><<<g, bf, 0, s>>>(P);
  else if (hist) k_contact_filter<true, true><<<g, bf, 0, s>>>(P);
  else k_contact_filter<true, false><<<g, bf, 0, s>>>(P);
  const bool learn = P.jkr_solver == 1 && P.nmodel == 3 && P.mlp != nullptr;
  int launched = 3;
  if (P.jfb != nullptr) {
    cudaEventRecord(side.fork, s);
    cudaStreamWaitEvent(side.stream, side.fork, 0);
    if (P.mode == 0) k_contact_hard<false, false, R><<<P.nsm * 8, 128, 0, side.stream>>>(P);
    else if (hist) k_contact_hard<true, true, R><<<P.nsm * 8, 128, 0, side.stream>>>(P);
    else k_contact_hard<true, false, R><<<P.nsm * 8, 128, 0, side.stream>>>(P);
    cudaEventRecord(side.join, side.stream);
    ++launched;
  }
  if (learn) {
    k_jkr_mlp<<<P.nsm * 4, 128, 0, s>>>(P);
    ++launched;
  }
  const int gc = shaped_grid((uint64_t)P.n * 4, bc, cap);
  if (P.mode == 0) k_contact_force<false, false, R, JKR><<<gc, bc, 0, s>>>(P);
  else if (hist) k_contact_force<true, true, R, JKR><<<gc, bc, 0, s>>>(P);
  else k_contact_force<true, false, R, JKR><<<gc, bc, 0, s>>>(P);
  if (P.jfb != nullptr) {
    // the deferred pairs lie in the band next to the JKR fold, where only
    // FP64 resolves the contact radius: FP64 in the mixed form too
    if (P.mode == 0) k_contact_deferred<false, false><<<P.nsm, 128, 0, s>>>(P);
    else if (hist) k_contact_deferred<true, true><<<P.nsm, 128, 0, s>>>(P);
    else k_contact_deferred<true, false><<<P.nsm, 128, 0, s>>>(P);
    cudaStreamWaitEvent(s, side.join, 0);
    ++launched;
  }
  if (P.prec == 1) k_accumulate<true><<<shaped_grid((uint64_t)P.n, ACC_DEAL, cap), ba, 0, s>>>(P);
  else k_accumulate<false><<<shaped_grid((uint64_t)P.n, ACC_DEAL, cap), ba, 0, s>>>(P);
  return launched;
}

int launch_force(const StepParams& P, cudaStream_t s, const SideStream& side) {
  if (P.n == 0) return 0;
  if (P.force_path == 0) {
    if (P.nmodel == 3)
      return P.prec == 1 ? launch_contact_path<float, true>(P, s, side) : launch_contact_path<double, true>(P, s, side);
    return P.prec == 1 ? launch_contact_path<float, false>(P, s, side) : launch_contact_path<double, false>(P, s, side);
  }
  const int g = grid_for(P.n, 128);
  if (P.nmodel == 3) {
    if (P.prec == 1) launch_force_t<float, true>(P, g, s);
    else launch_force_t<double, true>(P, g, s);
  } else {
    if (P.prec == 1) launch_force_t<float, false>(P, g, s);
    else launch_force_t<double, false>(P, g, s);
  }
  return 1;
}

// At most one block of k_steps a multiprocessor, of two threads a particle (a
// quad: four) in warps by the hundred and twenty-eight.
template <bool PHYS, bool HIST, typename R>
static int launch_steps_t(const StepParams& P, cudaStream_t s) {
  const int threads = P.n * (P.n <= QUAD_MAX ? 4 : 2);
  const int grid = std::min(P.nsm, (threads + 127) / 128);
  const int block = std::min(SMALL_BLOCK, ((threads + grid - 1) / grid + 127) / 128 * 128);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)block);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_steps<PHYS, HIST, R>, P) == cudaSuccess ? 1 : 0;
}

bool steps_in_one_launch(const StepParams& P) {
  return P.n > 0 && P.n <= SMALL_MAX && P.force_path == 0 && P.nmodel != 3;
}

int launch_steps_small(const StepParams& P, cudaStream_t s) {
  const bool hist = P.mode == 1 && P.tmodel != 0, mixed = P.prec == 1;
  if (P.mode == 0) return mixed ? launch_steps_t<false, false, float>(P, s) : launch_steps_t<false, false, double>(P, s);
  if (hist) return mixed ? launch_steps_t<true, true, float>(P, s) : launch_steps_t<true, true, double>(P, s);
  return mixed ? launch_steps_t<true, false, float>(P, s) : launch_steps_t<true, false, double>(P, s);
}

int launch_steps_next(const StepParams& P, cudaGraphConditionalHandle rebuild, cudaGraphConditionalHandle loop, int end,
                      cudaStream_t s) {
  k_steps_next<<<1, 1, 0, s>>>(P, rebuild, loop, end);
  return 1;
}

int launch_end_step(const StepParams& P, cudaStream_t s) {
  k_end_step<<<1, 1, 0, s>>>(P, 0, 0);
  return 1;
}

int launch_end_step_loop(const StepParams& P, cudaGraphConditionalHandle loop, cudaStream_t s) {
  k_end_step<<<1, 1, 0, s>>>(P, loop, 1);
  return 1;
}

void launch_kinetic_energy(const StepParams& P, double* out, cudaStream_t s) {
  cudaMemsetAsync(out, 0, sizeof(double), s);
  if (P.n == 0) return;
  k_kinetic<<<grid_for(P.n, 256), 256, 0, s>>>(P, out);
}

// ------------------------------------------------------- bulk state transfer
// The arrays of rp_read_state / rp_write_state are in id order; a slot's
// `tag` is its id (the particle's rank at the last upload), so slot_of[id]
// is a scatter of the tags. Used while no slot is dead (ids are then exactly
// 0..n-1). Copies only: no arithmetic touches the values.
__global__ void k_slot_of(StepParams P, uint32_t* slot_of, uint32_t* live) {
  const Bank B = P.bank[P.ctrl->bank];
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < P.n; k += gridDim.x * blockDim.x) {
    const uint32_t t = B.tag[k];
    slot_of[t] = (uint32_t)k;
    live[t] = (B.flags[k] & PF_DEAD) ? 0u : 1u;
  }
}

// With removed particles the ids are the live particles in upload order:
// id = the exclusive scan of the live flags at the upload position.
__global__ void k_compact_ids(int n, const uint32_t* slot_of, const uint32_t* live, const uint32_t* pos,
                              uint32_t* slot_of_id) {
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x)
    if (live[t]) slot_of_id[pos[t]] = slot_of[t];
}

__global__ void k_state_gather(StepParams P, const uint32_t* slot_of, StateIO io, int m) {
  const Bank B = P.bank[P.ctrl->bank];
  const D4* src[8] = {B.xr, B.vm, B.wc, B.acc, B.tq, B.xres, B.vres, B.wres};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
    const uint32_t k = slot_of[i];
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (io.v[q]) {
        const D4 d = src[q][k];
        io.v[q][3 * (size_t)i] = d.x;
        io.v[q][3 * (size_t)i + 1] = d.y;
        io.v[q][3 * (size_t)i + 2] = d.z;
      }
    if (io.radius) io.radius[i] = B.xr[k].w;
    if (io.mass) io.mass[i] = B.vm[k].w;
    if (io.fixed) io.fixed[i] = (B.flags[k] & PF_FIXED) ? 1 : 0;
  }
}

// Whether the given radii, masses and fixed flags equal the current ones (the
// per-particle constants derived from them then stay valid).
__global__ void k_state_same(StepParams P, const uint32_t* slot_of, StateIO io, unsigned* differs, int m) {
  const Bank B = P.bank[P.ctrl->bank];
  bool d = false;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
    const uint32_t k = slot_of[i];
    if (io.radius && __double_as_longlong(io.radius[i]) != __double_as_longlong(B.xr[k].w)) d = true;
    if (io.mass && __double_as_longlong(io.mass[i]) != __double_as_longlong(B.vm[k].w)) d = true;
    if (io.fixed && (io.fixed[i] != 0) != ((B.flags[k] & PF_FIXED) != 0)) d = true;
  }
  if (d) atomicOr(differs, 1u);
}

// Writes the given vector arrays into the slots (the .w fields, radius, mass,
// cell code, 1/m and 1/I, are kept) and refreshes the FP32 position mirror.
__global__ void k_state_scatter(StepParams P, const uint32_t* slot_of, StateIO io, int m) {
  const Bank B = P.bank[P.ctrl->bank];
  D4* dst[8] = {B.xr, B.vm, B.wc, B.acc, B.tq, B.xres, B.vres, B.wres};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
    const uint32_t k = slot_of[i];
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (io.v[q]) {
        D4 d = dst[q][k];
        d.x = io.v[q][3 * (size_t)i];
        d.y = io.v[q][3 * (size_t)i + 1];
        d.z = io.v[q][3 * (size_t)i + 2];
        dst[q][k] = d;
      }
    if (io.v[2]) {
      const uint32_t fl = B.flags[k] & ~PF_KICK;
      const V w = xyz(B.wc[k]);
      B.flags[k] = finite_bits(w.x) && finite_bits(w.y) && finite_bits(w.z) && finite_bits(B.wres[k].w) ? fl : fl | PF_KICK;
    }
    if (io.v[0]) {
      const D4 x = B.xr[k];
      const float4 xf = make_float4((float)x.x, (float)x.y, (float)x.z, (float)x.w);
      B.xf[k] = xf;
      // farther beyond a periodic face than a step leaves it, the minimum image
      // of its displacement does not show where it is: the lists are rebuilt,
      // and with them the flags that rule images out
      const float p[3] = {xf.x, xf.y, xf.z};
#pragma unroll
      for (int a = 0; a < 3; ++a)
        if (P.periodic[a] && ((float)P.bmin[a] - p[a] > P.half_skinf || p[a] - (float)P.bmax[a] > P.half_skinf))
          P.ctrl->rebuild = 1;
    }
  }
}

const uint32_t* launch_slot_of(const StepParams& P, const IdMap& M, int live, int n_ids, cudaStream_t s) {
  if (P.n == 0) return M.slot_of;
  // after a compaction some upload positions have no slot: their flags stay 0
  if (n_ids > P.n) cudaMemsetAsync(M.live, 0, sizeof(uint32_t) * (size_t)n_ids, s);
  k_slot_of<<<grid_for(P.n, 256), 256, 0, s>>>(P, M.slot_of, M.live);
  if (live == n_ids) return M.slot_of;  // nothing removed since the upload: the ids are the upload positions
  launch_exclusive_scan(nullptr, M.live, M.pos, (uint32_t)n_ids, M.part, nullptr, s);
  k_compact_ids<<<grid_for(n_ids, 256), 256, 0, s>>>(n_ids, M.slot_of, M.live, M.pos, M.slot_of_id);
  return M.slot_of_id;
}

void launch_state_gather(const StepParams& P, const uint32_t* slot_of, const StateIO& io, int m, cudaStream_t s) {
  if (m == 0) return;
  k_state_gather<<<grid_for(m, 256), 256, 0, s>>>(P, slot_of, io, m);
}

void launch_state_same(const StepParams& P, const uint32_t* slot_of, const StateIO& io, unsigned* differs, int m,
                       cudaStream_t s) {
  cudaMemsetAsync(differs, 0, sizeof(unsigned), s);
  if (m == 0) return;
  k_state_same<<<grid_for(m, 256), 256, 0, s>>>(P, slot_of, io, differs, m);
}

void launch_state_scatter(const StepParams& P, const uint32_t* slot_of, const StateIO& io, int m, cudaStream_t s) {
  if (m == 0) return;
  k_state_scatter<<<grid_for(m, 256), 256, 0, s>>>(P, slot_of, io, m);
}

}  // namespace rp
