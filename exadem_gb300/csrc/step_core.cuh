// step_core.cuh -- the integration's arguments and per-particle bodies shared by the
// sphere step (k_step_fused.cu) and the polyhedron step (k_poly.cu).
#pragma once
#include "f32_round.cuh"
#include "integrate_core.cuh"

namespace dem {

struct IntegArgs {
  PArrays P;
  Records R;
  uint64_t n;
  const uint32_t* own_off;
  const uint32_t* rev_off;
  const uint32_t* rev_idx;
  const uint32_t* stamp;  // polyhedra: a particle without a live record of this pass gathers none
  uint32_t pass;
  double g[3];
  double dt, hdt, dt2_2;  // dt, dt/2, dt^2/2
  double thr2;
  float thr2f;
  SysView sv;
  unsigned long long* scal;   // device scalars (flag, active contacts and work list counts)
  int dense;
  int epilog, prolog;
  unsigned long long* gs;     // graph step: its counters; epilog is then "not the call's first step"
  cudaGraphConditionalHandle cond;
  // polyhedra: the step (from 1 in a call) whose epilog this is; the trigger flag then
  // holds the step whose prolog raised it
  unsigned step;
  // polyhedra with inner bonds: the bond records and their lists per particle
  int nb;
  const double *bf[3], *bti[3], *btj[3];
  const uint32_t *b_own_first, *b_own_cnt, *b_rev_off, *b_rev_idx;
};
constexpr uint32_t ROT_EPILOG = 0x80000000u;  // put-off rotation whose epilog part is due too

// The rotations that a block's warps put off (few lanes of a warp need one) and its first
// warps then run together.
struct PutOff {
  uint32_t s[256], n;
};

// The warp's put-off rotations; all 32 lanes must call it.
__device__ __forceinline__ void put_off(PutOff& q, bool want, uint32_t entry) {
  const unsigned mask = __ballot_sync(0xffffffffu, want);
  if (!mask) return;
  const int lane = threadIdx.x & 31;
  uint32_t base = 0;
  if (lane == 0) base = atomicAdd(&q.n, (uint32_t)__popc(mask));
  base = __shfl_sync(0xffffffffu, base, 0);
  if (want) q.s[base + (uint32_t)__popc(mask & ((1u << lane) - 1u))] = entry;
}

// All 32 lanes must call it.  Returns the slot of this lane when want is set.
__device__ __forceinline__ uint32_t warp_append(bool want, unsigned long long* counter) {
  const unsigned mask = __ballot_sync(0xffffffffu, want);
  const int lane = threadIdx.x & 31;
  unsigned long long base = 0;
  if (mask) {
    const int leader = __ffs(mask) - 1;
    if (lane == leader) base = atomicAdd(counter, (unsigned long long)__popc(mask));
    base = __shfl_sync(0xffffffffu, base, leader);
  }
  return (uint32_t)base + (uint32_t)__popc(mask & ((1u << lane) - 1u));
}

// reset_force_moment + gravity_force + the gathers + force_to_accel + the linear half
// of the epilog of particle s: acc and the torque mom are stored, the new velocity is
// returned in v.  Returns whether the rotational half (epilog_rotation) is due; an
// idle rotation is done here.
template <int Mode>
__device__ __forceinline__ bool epilog_translate(const IntegArgs& a, uint64_t s, V3& v, V3& acc, V3& mom) {
  const PArrays& P = a.P;
  const Records& R = a.R;
  const double m = P.f[MASS][s];
  // 0.0 + g_c m is +0 for g_c = +-0 and a finite m (+0 + +-0 = +0): no FP64 work
  const bool mfin = ((emu_bits(m) >> 52) & 0x7ffu) != 0x7ffu;
  V3 f = mk(emu_is_zero(a.g[0]) && mfin ? 0.0 : 0.0 + a.g[0] * m, emu_is_zero(a.g[1]) && mfin ? 0.0 : 0.0 + a.g[1] * m,
            emu_is_zero(a.g[2]) && mfin ? 0.0 : 0.0 + a.g[2] * m);
  // f and mom start at +0 or a nonzero value and, in round to nearest, never
  // become -0 (x + (-x) = +0; -0 needs two -0 operands), so a record whose six
  // components are all +-0 (a listed pair that does not touch) leaves them
  // unchanged bit for bit and its additions are skipped.
  // (a record whose live flag is 0 is zero and is not read)
  // The owned records, then the partner records, in one loop: a particle's
  // owned and partner counts vary a lot (by id order), their sum (its
  // neighbour count) much less, so one loop keeps the warp's FP64 adds on
  // most lanes.  The order of the additions is that of two loops.
  const uint32_t o0 = a.own_off[s], no = a.own_off[s + 1] - o0;
  const uint32_t r0 = a.rev_off[s];
  const uint32_t nt = a.pass && a.stamp[s] != a.pass ? 0u : no + (a.rev_off[s + 1] - r0);
  // Two records at a time, their indexes and flags loaded together: a record is a chain of
  // three loads (10 k box, 100 steps: 3.40 to 3.31 ms; four or eight are no faster, and
  // above 100 k particles the FP64 pipe is the bound either way).
  constexpr int GB = 2;
  for (uint32_t q = 0; q < nt; q += GB) {
    uint32_t kk[GB];
    unsigned live = 0;
#pragma unroll
    for (int u = 0; u < GB; u++) kk[u] = q + u < no ? o0 + q + u : (q + u < nt ? a.rev_idx[r0 + (q + u - no)] : 0u);
#pragma unroll
    for (int u = 0; u < GB; u++)
      if (q + u < nt && R.live[kk[u]]) live |= 1u << u;
#pragma unroll
    for (int u = 0; u < GB; u++) {
      if (!(live >> u & 1u)) continue;
      const bool own = q + u < no;
      const uint32_t k = kk[u];
      const double* t0 = own ? R.ti[0] : R.tj[0];
      const double* t1 = own ? R.ti[1] : R.tj[1];
      const double* t2 = own ? R.ti[2] : R.tj[2];
      const V3 rf = mk(R.f[0][k], R.f[1][k], R.f[2][k]), rt = mk(t0[k], t1[k], t2[k]);
      if (((emu_bits(rf.x) | emu_bits(rf.y) | emu_bits(rf.z) | emu_bits(rt.x) | emu_bits(rt.y) | emu_bits(rt.z))
           << 1) != 0) {
        const uint64_t flip = own ? 0ull : 0x8000000000000000ull;  // -rf for a partner record (exact)
        f = f + mk(emu_double(emu_bits(rf.x) ^ flip), emu_double(emu_bits(rf.y) ^ flip),
                   emu_double(emu_bits(rf.z) ^ flip));
        mom = mom + rt;
      }
    }
  }
  if (a.nb) {  // the inner bonds (k_bond_force): owned, then as j, in bond order
    const uint32_t c0 = a.b_own_cnt[s], b0 = c0 ? a.b_own_first[s] : 0u;
    for (uint32_t k = b0; k < b0 + c0; k++) {
      f = f + mk(a.bf[0][k], a.bf[1][k], a.bf[2][k]);
      mom = mom + mk(a.bti[0][k], a.bti[1][k], a.bti[2][k]);
    }
    const uint32_t q0 = a.b_rev_off[s], q1 = a.b_rev_off[s + 1];
    for (uint32_t q = q0; q < q1; q++) {
      const uint32_t k = a.b_rev_idx[q];
      f = f + (-mk(a.bf[0][k], a.bf[1][k], a.bf[2][k]));
      mom = mom + mk(a.btj[0][k], a.btj[1][k], a.btj[2][k]);
    }
  }
  const double im = P.f[IMASS][s];
  LinMul<Mode> lm;
  acc = mk(div_rn_m(lm, f.x, m, im), div_rn_m(lm, f.y, m, im), div_rn_m(lm, f.z, m, im));
  const V3 vel = mk(P.f[VX][s], P.f[VY][s], P.f[VZ][s]);
  // v + a dt/2: a zero a gives the zero addend of emu_add_zero (integer pipe)
  const bool hok = emu_nonneg_finite(a.hdt);
  auto vstep = [&](double vc, double ac) {
    if (hok && emu_is_zero(ac)) {
      bool ok;
      const double r = emu_add_zero(vc, emu_sign(ac), ok);
      if (ok) return r;
    }
    return vc + lm.mul(ac, a.hdt);
  };
  v = mk(vstep(vel.x, acc.x), vstep(vel.y, acc.y), vstep(vel.z, acc.z));
  if (lm.failed()) {
    acc = mk(div_rn(f.x, m, im), div_rn(f.y, m, im), div_rn(f.z, m, im));
    v = mk(vel.x + acc.x * a.hdt, vel.y + acc.y * a.hdt, vel.z + acc.z * a.hdt);
  }
  P.f[FX][s] = acc.x;
  P.f[FY][s] = acc.y;
  P.f[FZ][s] = acc.z;
  P.f[MX][s] = mom.x;
  P.f[MY][s] = mom.y;
  P.f[MZ][s] = mom.z;
  const V3 vrot = mk(P.f[WX][s], P.f[WY][s], P.f[WZ][s]);
  bool need = true;
  if ((emu_bits(mom.x) | emu_bits(mom.y) | emu_bits(mom.z)) == 0) {
    const Q4 Q = {P.f[QW][s], P.f[QX][s], P.f[QY][s], P.f[QZ][s]};
    const V3 I = mk(P.f[IX][s], P.f[IY][s], P.f[IZ][s]);
    const V3 II = mk(P.f[IIX][s], P.f[IIY][s], P.f[IIZ][s]);
    if (rotation_idle(Q, vrot, mom, I, II)) {
      need = false;
      P.f[AX][s] = 0.0;
      P.f[AY][s] = 0.0;
      P.f[AZ][s] = 0.0;
      // w + (+0): w itself, +0 for a -0
      if (emu_bits(vrot.x) == 0x8000000000000000ull) P.f[WX][s] = 0.0;
      if (emu_bits(vrot.y) == 0x8000000000000000ull) P.f[WY][s] = 0.0;
      if (emu_bits(vrot.z) == 0x8000000000000000ull) P.f[WZ][s] = 0.0;
    }
  }
  return need;
}

// Lanes of a warp above which the rotations run in place.  While the particles give
// every scheduler at most one warp (32 lanes a scheduler, four schedulers an SM) the
// FP64 pipes wait for that warp alone, so every rotation runs in place.  With more warps a
// sparse one keeps its pipe from the next, and up to 24 lanes it pays to put its rotations
// off to the end of the block (PutOff).
static int rotation_dense(const dem_ctx* c) { return c->n <= (uint64_t)c->num_sms * 128u ? 0 : 24; }
// Threads per block of the prolog and the epilog: the tuned size, halved while the
// grid leaves SMs without a block (at 10 k particles 256 threads reach 40 SMs).
static unsigned particle_block(const dem_ctx* c) { return spread_block(c, c->n, (unsigned)c->tune_block); }

// Placement of the integration's multiplies: the context's mode, except that with at
// most one warp a scheduler, unless the mode was chosen by the caller or the autotuner,
// every multiply is on the FP64 pipe: the pipe then waits, and a product built on the
// integer pipe is a chain of some 20 instructions where the pipe's is one (16 k bonded
// cubes, 20 steps and a rebuild: 1.45 against 1.48 ms; 200 k: 6.64 against 5.92 ms).
static int integ_mode(const dem_ctx* c) {
  return c->mul_auto && c->n <= (uint64_t)c->num_sms * 128u ? 0 : c->mul_mode;
}
IntegArgs make_integ_args(dem_ctx* c, int epilog, int prolog);  // k_step_fused.cu
}  // namespace dem
