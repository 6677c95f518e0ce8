// contact_core.cuh -- device restatement of contact_force_core shared by the
// contact kernels (plain one-pass and compacted three-pass).
#pragma once
#include "dem_ctx.cuh"
#include "mul_policy.cuh"

namespace dem {

// Rolling clip of contact_force_core with its mur = 0 (contact_force.hpp:225-234):
//   r = (b.w)/(w.w); b' = b - r w; t = |0 * |b'| * |fn||;
//   if (|m|^2 > 0 && |m|^2 > t^2) m = m * (t / |m|)
// t is +0 when |b'| and |fn| are finite and NaN otherwise (0 * inf, NaN).
// Both are finite, with no operation overflowing, when every |b_c| < 2^200,
// every |fn_c| < 2^500, every |w_c| < 2^200 and some |w_c| >= 2^-200: then
// w.w lies in [2^-400, 3 2^400], |r w| <= |b| (1 + 8u) (a projection), and
// every square stays below 2^1024.  So in that range the clip is exactly
// "if (|m|^2 > 0) m = m * (+0)" (the signed zeros of m; m * 0 of an infinite
// component is NaN, as in the formula), without the two norms, the division
// and the square roots.  A spin of exactly zero keeps the moment (0/0 below);
// outside both cases (huge or non-finite values) the formula itself runs.
__device__ __forceinline__ bool exp_below(double x, int e2) {  // |x| < 2^e2, x finite
  return (int)((emu_bits(x) >> 52) & 0x7ffu) < 1023 + e2;
}
__device__ __forceinline__ bool exp_at_least(double x, int e2) {  // |x| >= 2^e2
  return (int)((emu_bits(x) >> 52) & 0x7ffu) >= 1023 + e2;
}
template <class M>
__device__ __forceinline__ void rolling_clip_mur0_m(M& mm, V3 branch, V3 vrot_i, V3 fn, V3& mom_i);
__device__ __forceinline__ void rolling_clip_mur0(V3 branch, V3 vrot_i, V3 fn, V3& mom_i) {
  MulFP64 mm;
  rolling_clip_mur0_m(mm, branch, vrot_i, fn, mom_i);
}
template <class M>
__device__ __forceinline__ void rolling_clip_mur0_m(M& mm, V3 branch, V3 vrot_i, V3 fn, V3& mom_i) {
  // w = +-0: r = (b.w)/(w.w) is (+-0 or NaN)/(+0) = NaN for any b, so t = NaN and
  // the comparison with t^2 is false: the moment is kept as it is
  if (((emu_bits(vrot_i.x) | emu_bits(vrot_i.y) | emu_bits(vrot_i.z)) << 1) == 0) return;
  const bool in_range = exp_below(branch.x, 200) && exp_below(branch.y, 200) && exp_below(branch.z, 200) &&
                        exp_below(fn.x, 500) && exp_below(fn.y, 500) && exp_below(fn.z, 500) &&
                        exp_below(vrot_i.x, 200) && exp_below(vrot_i.y, 200) && exp_below(vrot_i.z, 200) &&
                        (exp_at_least(vrot_i.x, -200) || exp_at_least(vrot_i.y, -200) ||
                         exp_at_least(vrot_i.z, -200));
  const double mom_square = dot_m(mm, mom_i, mom_i);
  if (in_range) {
    if (emu_gt0(mom_square)) mom_i = mk(mm.mul(mom_i.x, 0.0), mm.mul(mom_i.y, 0.0), mm.mul(mom_i.z, 0.0));
    return;
  }
  const double r = (dot(branch, vrot_i)) / (dot(vrot_i, vrot_i));
  branch = branch - r * vrot_i;
  const double mur = 0;
  const double threshold_mom = fabs(mur * vnorm(branch) * vnorm(fn));
  if (mom_square > 0.0 && mom_square > threshold_mom * threshold_mom)
    mom_i = mom_i * (threshold_mom / sqrt(mom_square));
}

template <class M>
__device__ __forceinline__ V3 cross_m(M& mm, V3 a, V3 b) {
  return mk(mm.sub(mm.mul(a.y, b.z), mm.mul(a.z, b.y)), mm.sub(mm.mul(a.z, b.x), mm.mul(a.x, b.z)),
            mm.sub(mm.mul(a.x, b.y), mm.mul(a.y, b.x)));
}
template <class M>
__device__ __forceinline__ double dot_m(M& mm, V3 a, V3 b) {
  return mm.add(mm.add(mm.mul(a.x, b.x), mm.mul(a.y, b.y)), mm.mul(a.z, b.z));
}
template <class M>
__device__ __forceinline__ V3 add_m(M& mm, V3 a, V3 b) {
  return mk(mm.add(a.x, b.x), mm.add(a.y, b.y), mm.add(a.z, b.z));
}
template <class M>
__device__ __forceinline__ V3 sub_m(M& mm, V3 a, V3 b) {
  return mk(mm.sub(a.x, b.x), mm.sub(a.y, b.y), mm.sub(a.z, b.z));
}
template <class M>
__device__ __forceinline__ V3 scale_m(M& mm, double s, V3 a) {
  return mk(mm.mul(s, a.x), mm.mul(s, a.y), mm.mul(s, a.z));
}

__device__ __forceinline__ bool zero3(V3 v) {
  return ((emu_bits(v.x) | emu_bits(v.y) | emu_bits(v.z)) << 1) == 0;
}

// The moment update mom += (kr (w_j - w_i)) dt and its rolling clip, decided on
// the integer pipe for a zero history (signed zeros; a new pair, and every pair
// after its clip).  Returns false where the arithmetic has to run.
//   d = w_j - w_i, p = (kr d) dt, m = mom + p.
// kr = +0: p is the zero of d's sign, m the zero that is negative only when both
//   are, and the clip leaves it: mom^2 > 0 is false.
// kr > 0, a spin w_i that is not zero and the operands in the range of the clip's
//   first case: the clip gives m * (+0), the zero of m's sign.  m = p where d_c
//   is not zero, and the sum of two zeros where it is; mom^2 > 0 holds when some
//   d_c is not zero: spin components are zero or at least 2^-200, so d_c is a
//   multiple of 2^-252, and kr, dt >= 2^-60 keep p^2 above the subnormals; with
//   every d_c zero the clip changes nothing.
// The sign of d_c is that of the comparison of its operands; equal operands give
// +0, except (-0) - (+0) = -0.
__device__ __forceinline__ bool moment_zero(V3 branch, V3 vrot_i, V3 vrot_j, V3 fn, double kr, double dt, V3& mom) {
  auto window = [](double x) {
    const uint32_t e = (uint32_t)(emu_bits(x) >> 52) & 0x7ffu;
    return e - (1023u - 200u) < 400u || emu_is_zero(x);
  };
  auto scale = [](double x) { return (uint32_t)(emu_bits(x) >> 52) - (1023u - 60u) < 120u; };  // positive
  if (!zero3(mom) || !window(vrot_i.x) || !window(vrot_i.y) || !window(vrot_i.z) || !window(vrot_j.x) ||
      !window(vrot_j.y) || !window(vrot_j.z) || !scale(dt))
    return false;
  const bool rolls = emu_bits(kr) != 0;
  if (rolls && (!scale(kr) || zero3(vrot_i) || !exp_below(branch.x, 200) || !exp_below(branch.y, 200) ||
                !exp_below(branch.z, 200) || !exp_below(fn.x, 500) || !exp_below(fn.y, 500) || !exp_below(fn.z, 500)))
    return false;
  auto out = [rolls](double wj, double wi, double mo) {
    const uint64_t uj = emu_bits(wj), ui = emu_bits(wi);
    const bool eq = uj == ui || ((uj | ui) << 1) == 0;
    const uint64_t neg = eq ? (uj & ~ui) >> 63 : (emu_key(wj) < emu_key(wi) ? 1ull : 0ull);
    return emu_double((rolls && !eq ? neg : (neg & emu_sign(mo))) << 63);
  };
  mom = mk(out(vrot_j.x, vrot_i.x, mom.x), out(vrot_j.y, vrot_i.y, mom.y), out(vrot_j.z, vrot_i.z, mom.z));
  return true;
}

// t + mo; the sums with a zero moment on the integer pipe
template <class M>
__device__ __forceinline__ V3 add_moment(M& mm, V3 t, V3 mo) {
  if (zero3(mo)) {
    bool a, b, c;
    const V3 r = mk(emu_add_zero(t.x, emu_sign(mo.x), a), emu_add_zero(t.y, emu_sign(mo.y), b),
                    emu_add_zero(t.z, emu_sign(mo.z), c));
    if (a && b && c) return r;
  }
  return add_m(mm, t, mo);
}

// Velocity of a body's point: vel - cross(cpos - pos, vrot).  Without spin the
// cross product of a finite arm is a zero vector and vel - (+-0) is vel itself,
// unless a component of vel is -0.
template <class M>
__device__ __forceinline__ V3 point_velocity(M& mm, V3 vel, V3 cpos, V3 pos, V3 vrot) {
  auto plain = [](double x) { return exp_below(x, 1000) && emu_bits(x) != 0x8000000000000000ull; };
  if (zero3(vrot) && exp_below(cpos.x, 1000) && exp_below(cpos.y, 1000) && exp_below(cpos.z, 1000) &&
      exp_below(pos.x, 1000) && exp_below(pos.y, 1000) && exp_below(pos.z, 1000) && plain(vel.x) && plain(vel.y) &&
      plain(vel.z))
    return vel;
  return sub_m(mm, vel, cross_m(mm, sub_m(mm, cpos, pos), vrot));
}

// contact_force_core below with its multiplies through mm, in the same
// operation order, and the rolling clip through rolling_clip_mur0 (same
// result); the clip's arithmetic keeps the FP64 pipe.
// With Damp, `meff` carries the pair's damping coefficient damp_rate 2
// sqrt(kn meff) itself, computed with the same operations when the list was
// built (IArrays::damp), instead of the effective mass.
template <class M, bool Damp = false>
__device__ __forceinline__ void contact_force_core_m(M& mm, bool cohesive, double dn, V3 n, double dt,
                                                     const dem_contact_params& hkp, double meff, V3& ft, V3 cpos,
                                                     V3 pos_i, V3 vel_i, V3& f_i, V3& mom_i, V3 vrot_i, V3 pos_j,
                                                     V3 vel_j, V3 vrot_j, bool dmt = false, double reff = 0.0) {
  if (cohesive) {
    if (emu_ge0(dn)) {  // comparisons of this form on the integer pipe (emu64.cuh)
      const double fn_value = mm.sub(mm.mul(hkp.fc / hkp.dncut, dn), hkp.fc);
      f_i = add_m(mm, f_i, scale_m(mm, fn_value, n));
      ft = mk(0, 0, 0);
      return;
    }
  }
  const double damp = Damp ? meff : mm.mul(mm.twice(hkp.damp_rate), sqrt(mm.mul(hkp.kn, meff)));
  const V3 contribution_i = point_velocity(mm, vel_i, cpos, pos_i, vrot_i);
  const V3 contribution_j = point_velocity(mm, vel_j, cpos, pos_j, vrot_j);
  const V3 vel = sub_m(mm, contribution_j, contribution_i);
  const double vn = dot_m(mm, vel, n);
  const double kd = mm.mul(hkp.kn, dn);
  V3 fn;
  {
    const double fne = -kd;  // (-kn) dn: the product with the sign flipped
    const double fnv = mm.mul(damp, vn);
    const double s = mm.add(fnv, fne);
    double nf = emu_gt0(s) ? s : 0;
    if (cohesive) {
      const double fn_norm = mm.sub(nf, hkp.fc);
      nf = emu_lt(fn_norm, -hkp.fc) ? -hkp.fc : fn_norm;
    }
    fn = scale_m(mm, nf, n);
  }
  {
    const V3 vt = sub_m(mm, vel, scale_m(mm, vn, n));
    const V3 ftd = scale_m(mm, dt, vt);
    ft = add_m(mm, ft, scale_m(mm, hkp.kt, ftd));
  }
  double threshold_ft;
  if (!cohesive) {
    threshold_ft = fabs(mm.mul(hkp.mu, kd));
  } else {
    threshold_ft = fabs(mm.mul(hkp.mu, mm.add(dot_m(mm, fn, n), hkp.fc)));
  }
  {
    const double ft_square = dot_m(mm, ft, ft);
    if (emu_gt0(ft_square) && emu_gt_nonneg(ft_square, mm.mul(threshold_ft, threshold_ft))) {
      const double s = threshold_ft / sqrt(ft_square);
      ft = mk(mm.mul(ft.x, s), mm.mul(ft.y, s), mm.mul(ft.z, s));
    }
  }
  f_i = add_m(mm, fn, ft);
  if (dmt && hkp.gamma > 0.0 && emu_lt0(dn)) {
    const double F = mm.mul(mm.mul(2.0 * 3.14159265358979323846, reff), hkp.gamma);
    f_i = sub_m(mm, f_i, scale_m(mm, F, n));
  }
  const V3 branch = sub_m(mm, cpos, pos_i);
  if (!moment_zero(branch, vrot_i, vrot_j, fn, hkp.kr, dt, mom_i)) {
    const V3 d = sub_m(mm, vrot_j, vrot_i);
    mom_i = add_m(mm, mom_i, mk(mm.mul(mm.mul(hkp.kr, d.x), dt), mm.mul(mm.mul(hkp.kr, d.y), dt),
                                mm.mul(mm.mul(hkp.kr, d.z), dt)));
    rolling_clip_mur0_m(mm, branch, vrot_i, fn, mom_i);
  }
}

// apply_dmt_force (contact_force.hpp:115-127): in contact (dn < 0) and for
// gamma > 0, f_i -= (2 pi reff gamma) n, the operation order of the reference
__device__ __forceinline__ double dmt_magnitude(double reff, double gamma) {
  return 2.0 * 3.14159265358979323846 * reff * gamma;
}

// contact_force_core (contact_force.hpp:146-235).  f_i must be {0,0,0} on entry.
// dmt: the Hooke_DMT law combination (contact_force.hpp:70-76) with reff the
// effective radius of the pair.
__device__ __forceinline__ void contact_force_core(bool cohesive, double dn, V3 n, double dt, const dem_contact_params& hkp,
                                          double meff, V3& ft, V3 cpos, V3 pos_i, V3 vel_i, V3& f_i, V3& mom_i,
                                          V3 vrot_i, V3 pos_j, V3 vel_j, V3 vrot_j, bool dmt = false,
                                          double reff = 0.0) {
  if (cohesive) {
    if (dn >= 0) {
      const double fn_value = (hkp.fc / hkp.dncut) * dn - hkp.fc;
      f_i = f_i + fn_value * n;
      ft = mk(0, 0, 0);
      return;
    }
  }
  const double damp = hkp.damp_rate * 2.0 * sqrt(hkp.kn * meff);
  const V3 contribution_i = vel_i - cross(cpos - pos_i, vrot_i);
  const V3 contribution_j = vel_j - cross(cpos - pos_j, vrot_j);
  const V3 vel = contribution_j - contribution_i;
  const double vn = dot(vel, n);
  V3 fn;
  {
    const double fne = -hkp.kn * dn;
    const double fnv = damp * vn;
    double nf = (fnv + fne > 0) ? fnv + fne : 0;
    if (cohesive) {
      const double fn_norm = nf - hkp.fc;
      nf = fn_norm < (-hkp.fc) ? -hkp.fc : fn_norm;
    }
    fn = nf * n;
  }
  {
    const V3 vt = vel - vn * n;
    const V3 ftd = dt * vt;
    ft = ft + hkp.kt * ftd;
  }
  double threshold_ft;
  if (!cohesive) {
    const double fne = hkp.kn * dn;
    threshold_ft = fabs(hkp.mu * fne);
  } else {
    threshold_ft = fabs(hkp.mu * (dot(fn, n) + hkp.fc));
  }
  {
    const double ft_square = dot(ft, ft);
    if (ft_square > 0.0 && ft_square > threshold_ft * threshold_ft) {
      const double s = threshold_ft / sqrt(ft_square);
      ft = ft * s;
    }
  }
  f_i = fn + ft;
  if (dmt && hkp.gamma > 0.0 && dn < 0.0) f_i = f_i - dmt_magnitude(reff, hkp.gamma) * n;
  mom_i = mom_i + hkp.kr * (vrot_j - vrot_i) * dt;
  // rolling clip with mur = 0 (contact_force.hpp:225-234): the IEEE NaN of
  // 0/0 when vrot_i == 0 keeps the moment, otherwise the moment is scaled by 0.
  V3 branch = cpos - pos_i;
  const double r = (dot(branch, vrot_i)) / (dot(vrot_i, vrot_i));
  branch = branch - r * vrot_i;
  const double mur = 0;
  const double threshold_mom = fabs(mur * vnorm(branch) * vnorm(fn));
  const double mom_square = dot(mom_i, mom_i);
  if (mom_square > 0.0 && mom_square > threshold_mom * threshold_mom)
    mom_i = mom_i * (threshold_mom / sqrt(mom_square));
}


__device__ __forceinline__ V3 ldv(const PArrays& P, int f0, uint32_t i) {
  return mk(P.f[f0][i], P.f[f0 + 1][i], P.f[f0 + 2][i]);
}

}  // namespace dem
