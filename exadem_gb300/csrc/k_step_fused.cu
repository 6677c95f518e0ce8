// k_step_fused.cu -- the optimised Verlet step: fewer launches, dense FP64 warps.
//
// FP64 on GB300 runs at 2 thread-instructions per clock per SM (1/64 of FP32),
// so the step is bound by the FP64 pipe, not by HBM.  Two consequences drive
// this file, and neither changes a single result bit:
//  * lanes that need no FP64 work must not share a warp with lanes that do:
//    a warp instruction with one active lane costs the FP64 pipe as much as a
//    full one.  The contact law therefore runs over compacted lists:
//      k_cscreen  one thread per interaction; an FP32 test proves most pairs
//                 apart (history reset, zero record, no FP64 at all); the others
//                 are appended to list L1 with warp-aggregated atomics;
//      k_cfused   dense over L1: FP64 detection; no contact -> reset; the pairs
//                 that overlap and those that attract wait in two queues in
//                 shared memory and run their law in full tiles;
//      or, as the autotuner may choose, k_cdetect over L1 and k_chooke over its
//      list L2 of the overlapping pairs.
//  * the divisions by mass and inertia use exact reciprocal-based division
//    (math_exact.cuh) and reset + gravity + gather + force_to_accel + epilog,
//    with the next step's prolog + displacement trigger, are one kernel.
// Order of summation, operation order and rounding are those of the operator
// kernels (contact_core.cuh, integrate_core.cuh).
#include <algorithm>

#include "contact_core.cuh"
#include "integrate_core.cuh"
#include "mesh_core.cuh"
#include "step_core.cuh"

namespace dem {
namespace {

constexpr int FT = 128;  // threads per block of k_cdetect and k_chooke

struct CArgs {
  PArrays P;
  IArrays I;
  Records R;
  uint64_t ni;
  const unsigned long long* ni_dev;  // graph step: the count lives on the device
  SysView sv;  // periodic lengths of the owner's system
  const DriverDev* drv;
  const MeshDev* mesh;
  dem_contact_params cp, cpd;
  double dt;
  int cohesive;
  int dmt;        // Hooke_DMT law combination
  ParamTable pt;  // multi-material parameters (pt.pp == nullptr: cp / cpd)
  ContactStateArrays cs;  // analysis (cs.dn == nullptr: off)
  int screen;
  float dncut_f;  // config.dncut in FP32 (not below 0)
  uint32_t* L1;
  uint32_t* L2;
  double* D[7];  // dn, n(3), cp(3) of the L2 entries
  unsigned long long* cnt;  // [0] L1 count (particle pairs), [1] L2 count, [2] driver pairs of L1
  uint64_t l1cap;           // L1 entries: particle pairs from the front, driver pairs from the back
  int int_share;            // k_cfused: Hooke tiles out of 8 run with AllInt (the integer pipe)
  unsigned long long* n_active;
  int overlap_only;             // a pair counts as active at dn < 0 only
};

// L1 as one list: the particle pairs (front, n1 of them), then the driver pairs
// (stored from the back).  Grouping the two kinds keeps each warp on one
// detection and one law, so neither runs with the other's lanes idle.
__device__ __forceinline__ uint32_t l1_at(const CArgs& a, uint64_t w, uint64_t n1) {
  return w < n1 ? a.L1[w] : a.L1[a.l1cap - 1 - (w - n1)];
}

__device__ __forceinline__ void write_result(const CArgs& a, uint64_t k, V3 ft, V3 mo, V3 f, V3 ti, V3 tj) {
  a.I.ft[0][k] = ft.x;
  a.I.ft[1][k] = ft.y;
  a.I.ft[2][k] = ft.z;
  a.I.mo[0][k] = mo.x;
  a.I.mo[1][k] = mo.y;
  a.I.mo[2][k] = mo.z;
  a.R.f[0][k] = f.x;
  a.R.f[1][k] = f.y;
  a.R.f[2][k] = f.z;
  a.R.ti[0][k] = ti.x;
  a.R.ti[1][k] = ti.y;
  a.R.ti[2][k] = ti.z;
  a.R.tj[0][k] = tj.x;
  a.R.tj[1][k] = tj.y;
  a.R.tj[2][k] = tj.z;
}

// partner position, moved by the periodic lengths of the owner i's system for an image
__device__ __forceinline__ V3 partner_pos(const CArgs& a, uint32_t meta, uint32_t i, uint32_t j) {
  V3 rj = ldv(a.P, RX, j);
  const int sx = meta_shift(meta, 0), sy = meta_shift(meta, 1), sz = meta_shift(meta, 2);
  if (sx | sy | sz) {
    const GridDev& g = a.sv.g[a.sv.of(i)];
    if (sx) rj.x = rj.x + (double)sx * g.L[0];
    if (sy) rj.y = rj.y + (double)sy * g.L[1];
    if (sz) rj.z = rj.z + (double)sz * g.L[2];
  }
  return rj;
}

__global__ void __launch_bounds__(128) k_cscreen(CArgs a) {
  const uint64_t ni = a.ni_dev ? *a.ni_dev : a.ni;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x; base < ni; base += stride) {
  const uint64_t k = base + threadIdx.x;
  bool want = false, drv = false;
  if (k < ni) {
    const uint32_t meta = a.I.meta[k];
    want = true;
    drv = meta_type(meta) != DEM_ITYPE_VERTEX_VERTEX;
    if (a.screen && meta_type(meta) == DEM_ITYPE_VERTEX_VERTEX) {
      const uint32_t i = a.I.owner[k], j = a.I.partner[k];
      const V3 ri = ldv(a.P, RX, i);
      const V3 rj = partner_pos(a, meta, i, j);
      // the proof of separation of the one-pass kernel (k_contact_sphere.cu) without
      // its FP64 instructions (six conversions and six additions a pair, 870 of a
      // warp's cycles): differences from the significands, good to 2^-22, and radii
      // rounded on the integer pipe, good to 2^-23, within the margin of 2^-17.
      bool ok = true;
      uint32_t top = 0;
      const float ex = diff_f32(ri.x, rj.x, ok, top), ey = diff_f32(ri.y, rj.y, ok, top),
                  ez = diff_f32(ri.z, rj.z, ok, top);
      const float d2f = ex * ex + ey * ey + ez * ez;
      const float dncut = a.cohesive ? (a.pt.pp ? fmaxf((float)a.pt.pair(a.cp, a.P.group[i], a.P.group[j]).dncut, 0.f)
                                                : a.dncut_f)
                                     : 0.f;
      const float limf = trunc_f32(a.P.f[RAD][i], ok) + trunc_f32(a.P.f[RAD][j], ok) + dncut;
      // 2^28 lim above the coordinates: what diff_f32 drops is below 2^-24 of lim
      ok = ok && top < (__float_as_uint(limf) >> 23) - 127u + 1023u + 28u;
      if (ok && limf > 1e-15f && limf < 1e15f && d2f > limf * limf * 1.0000077f) {
        want = false;
        if (a.R.live[k]) {  // not yet zero: reset history and record once
          const V3 z = mk(0, 0, 0);
          write_result(a, k, z, z, z, z, z);
          a.R.live[k] = 0;
        }
      }
    }
  }
  drv = drv && want;
  const uint32_t pos = warp_append(want && !drv, a.cnt);
  const uint32_t pd = warp_append(drv, a.cnt + 2);
  if (want && !drv) a.L1[pos] = (uint32_t)k;
  if (drv) a.L1[a.l1cap - 1 - pd] = (uint32_t)k;
  }
}

// FP64 detection of interaction k; a pair that does not touch is finished here.
// Returns PAIR_DONE for it, PAIR_HOOKE for an overlapping pair and PAIR_ATTRACT
// for the cohesive attraction before contact; their law is left to the caller
// (hooke_pair, attract_pair) with (dn, n, cpos).
constexpr int PAIR_DONE = 0, PAIR_HOOKE = 1, PAIR_ATTRACT = 2;
__device__ __forceinline__ int detect_pair(const CArgs& a, uint32_t k, double& dn, V3& n, V3& cpos) {
  int kind = PAIR_DONE;
  const uint32_t meta = a.I.meta[k];
  const uint32_t i = a.I.owner[k], j = a.I.partner[k];
  const V3 ri = ldv(a.P, RX, i);
  const double rad_i = a.P.f[RAD][i];
  bool contact;
  bool is_vv = meta_type(meta) == DEM_ITYPE_VERTEX_VERTEX;
  V3 rj = mk(0, 0, 0);
  double dncut;
  if (is_vv) {
    rj = partner_pos(a, meta, i, j);
    const double rad_j = a.P.f[RAD][j];
    const double R = rad_i + rad_j;
    const V3 dist = ri - rj;
    const double dist_norm = vnorm(dist);
    dn = dist_norm - R;
    contact = emu_lt0(dn);  // comparisons of this kernel on the integer pipe (emu64.cuh)
    dncut = a.pt.pair(a.cp, a.P.group[i], a.P.group[j]).dncut;
    if (contact || (a.cohesive && emu_le(dn, dncut)) || a.cs.dn) {  // n and cpos are used only then
      const double inv_dist_norm = 1.0 / dist_norm;
      n = dist * inv_dist_norm;
      cpos = ri - n * (rad_i + emu_mulhalf(dn));
    }
  } else {
    const DriverDev& d = a.drv[j];
    if (d.kind == 2) {  // detect<7|8|9> (contact_sphere.hpp:300-396)
      const DetD q = mesh_detect(a.mesh[d.mesh], meta_type(meta), a.I.sub[k] >> 16, ri, rad_i);
      dn = q.dn;
      contact = q.c;
      n = q.n;
      cpos = q.cp;
    } else if (d.kind == 0) {
      const V3 nrm = mk(d.normal[0], d.normal[1], d.normal[2]);
      const V3 proj = dot(ri, nrm) * nrm;
      const V3 s2p = -(mk(d.center_proj[0], d.center_proj[1], d.center_proj[2]) - proj);
      const double dd = vnorm(s2p);
      dn = dd - rad_i;
      contact = !emu_gt0(dn);
      if (contact) {
        n = s2p / dd;
        cpos = ri - n * (rad_i + emu_mulhalf(dn));
      }
    } else {
      const V3 proj = ri * mk(d.axis[0], d.axis[1], d.axis[2]);
      const V3 dir = mk(d.center[0], d.center[1], d.center[2]) - proj;
      const double dd = vnorm(dir);
      dn = d.radius - (rad_i + dd);
      contact = !emu_gt0(dn);
      if (contact) {
        n = dir / dd;
        cpos = ri - n * (rad_i + emu_mulhalf(dn));
      }
    }
    dncut = a.pt.drv(a.cpd, a.P.group[i], j).dncut;
  }
  if (a.cohesive) contact = (contact || emu_le(dn, dncut));
  if (!contact) {
    a.cs.write(k, 0.0, cpos, mk(0, 0, 0), mk(0, 0, 0));  // item.reset(), dn = 0
    if (a.R.live[k] || a.cs.dn) {
      const V3 z = mk(0, 0, 0);
      write_result(a, k, z, z, z, z, z);
      a.R.live[k] = 0;
    }
  } else if (a.cohesive && emu_ge0(dn)) {
    kind = PAIR_ATTRACT;
  } else {
    kind = PAIR_HOOKE;
  }
  return kind;
}

// cohesive attraction before contact (contact_force.hpp:165-173): f = fn_value n, ft = 0
__device__ __forceinline__ void attract_pair(const CArgs& a, uint32_t k, double dn, V3 n, V3 cpos) {
  const uint32_t meta = a.I.meta[k];
  const uint32_t i = a.I.owner[k], j = a.I.partner[k];
  const bool is_vv = meta_type(meta) == DEM_ITYPE_VERTEX_VERTEX;
  const V3 ri = ldv(a.P, RX, i);
  const V3 mo = mk(a.I.mo[0][k], a.I.mo[1][k], a.I.mo[2][k]);
  const dem_contact_params& hkp =
      is_vv ? a.pt.pair(a.cp, a.P.group[i], a.P.group[j]) : a.pt.drv(a.cpd, a.P.group[i], j);
  const double fn_value = (hkp.fc / hkp.dncut) * dn - hkp.fc;
  const V3 f = mk(0, 0, 0) + fn_value * n;
  MulFP64 mm;
  const V3 ti = add_moment(mm, cross(cpos - ri, f), mo);
  V3 tj = mk(0, 0, 0);
  if (is_vv) tj = add_moment(mm, cross(cpos - partner_pos(a, meta, i, j), -f), -mo);
  write_result(a, k, mk(0, 0, 0), mo, f, ti, tj);
  a.R.live[k] = 1;
  a.cs.write(k, dn, cpos, f - mk(0, 0, 0), mk(0, 0, 0));  // ft = 0 before contact
}

__global__ void __launch_bounds__(FT) k_cdetect(CArgs a) {
  const uint64_t n1 = a.cnt[0], nl = n1 + a.cnt[2];
  const uint64_t stride = (uint64_t)gridDim.x * FT;
  for (uint64_t base = (uint64_t)blockIdx.x * FT; base < nl; base += stride) {
    const uint64_t w = base + threadIdx.x;
    bool heavy = false;
    uint32_t k = 0;
    double dn = 0;
    V3 n = mk(0, 0, 0), cpos = mk(0, 0, 0);
    if (w < nl) {
      k = l1_at(a, w, n1);
      const int kind = detect_pair(a, k, dn, n, cpos);
      if (kind == PAIR_ATTRACT) attract_pair(a, k, dn, n, cpos);
      heavy = kind == PAIR_HOOKE;
    }
    const uint32_t pos = warp_append(heavy, a.cnt + 1);
    if (heavy) {
      a.L2[pos] = k;
      a.D[0][pos] = dn;
      a.D[1][pos] = n.x;
      a.D[2][pos] = n.y;
      a.D[3][pos] = n.z;
      a.D[4][pos] = cpos.x;
      a.D[5][pos] = cpos.y;
      a.D[6][pos] = cpos.z;
    }
  }
}

// The Hooke law of one overlapping pair with the arithmetic policy Pol
// (mul_policy.cuh): MulFP64, MulInt (its multiplies on the integer pipe) or
// AllInt (multiplies and additions there).  An operand outside an integer
// path makes the pair run again on the FP64 pipe from its stored inputs
// (nothing is written before write_result): the same bits in every case.
template <class M>
__device__ __forceinline__ void hooke_run(M& mm, const CArgs& a, uint32_t k, double dn, V3 n, V3 cpos, V3& ft,
                                          V3& mo, V3& f, V3& ti, V3& tj) {
  const uint32_t meta = a.I.meta[k];
  const uint32_t i = a.I.owner[k], j = a.I.partner[k];
  const V3 ri = ldv(a.P, RX, i);
  ft = mk(a.I.ft[0][k], a.I.ft[1][k], a.I.ft[2][k]);
  mo = mk(a.I.mo[0][k], a.I.mo[1][k], a.I.mo[2][k]);
  f = mk(0, 0, 0);
  tj = mk(0, 0, 0);
  const V3 vi = ldv(a.P, VX, i);
  const V3 wi = ldv(a.P, WX, i);
  if (meta_type(meta) == DEM_ITYPE_VERTEX_VERTEX) {
    const V3 rj = partner_pos(a, meta, i, j);
    const V3 vj = ldv(a.P, VX, j), wj = ldv(a.P, WX, j);
    // the pair's damping coefficient, set when the list was built (k_fill); DMT:
    // reff = compute_effective_radius (common_kernels.hpp:99-102)
    double reff = 0.0;
    if (a.dmt) {
      const double rad_i = a.P.f[RAD][i], rad_j = a.P.f[RAD][j];
      reff = mm.mul(rad_i, rad_j) / mm.add(rad_i, rad_j);
    }
    const dem_contact_params& cp = a.pt.pair(a.cp, a.P.group[i], a.P.group[j]);
    contact_force_core_m<M, true>(mm, a.cohesive, dn, n, a.dt, cp, a.I.damp[k], ft, cpos, ri, vi, f, mo, wi, rj,
                                  vj, wj, a.dmt, reff);
    ti = add_moment(mm, cross_m(mm, sub_m(mm, cpos, ri), f), mo);
    tj = add_moment(mm, cross_m(mm, sub_m(mm, cpos, rj), -f), -mo);
  } else {
    const DriverDev& d = a.drv[j];
    const V3 dpos = mk(d.center[0], d.center[1], d.center[2]);
    const V3 dvel = mk(d.vel[0], d.vel[1], d.vel[2]);
    const V3 dvrot = mk(d.vrot[0], d.vrot[1], d.vrot[2]);
    const dem_contact_params& cpd = a.pt.drv(a.cpd, a.P.group[i], j);
    contact_force_core_m<M, true>(mm, a.cohesive, dn, n, a.dt, cpd, a.I.damp[k], ft, cpos, ri, vi, f, mo, wi, dpos,
                                  dvel, dvrot, a.dmt, a.P.f[RAD][i]);
    ti = add_moment(mm, cross_m(mm, sub_m(mm, cpos, ri), f), mo);
  }
}

// The Hooke law of one overlapping pair with the arithmetic policy Pol
// (mul_policy.cuh): MulFP64, MulInt (its multiplies on the integer pipe) or
// AllInt (multiplies and additions there).  An operand outside an integer
// path makes the pair run again on the FP64 pipe from its stored inputs
// (nothing is written before write_result): the same bits in every case.
template <class Pol>
__device__ __forceinline__ void hooke_pair_p(const CArgs& a, uint32_t k, double dn, V3 n, V3 cpos) {
  V3 ft, mo, f, ti, tj;
  Pol mm;
  hooke_run(mm, a, k, dn, n, cpos, ft, mo, f, ti, tj);
  if (mm.failed()) {
    asm volatile("" ::: "memory");
    MulFP64 nm;
    hooke_run(nm, a, k, dn, n, cpos, ft, mo, f, ti, tj);
  }
  write_result(a, k, ft, mo, f, ti, tj);
  a.R.live[k] = 1;
  if (a.cs.dn) a.cs.write(k, dn, cpos, f - ft, ft);
}

// Mode bit 2 (instance 1): the law's multiplies on the integer pipe
template <int Mode>
__device__ __forceinline__ void hooke_pair(const CArgs& a, uint32_t k, double dn, V3 n, V3 cpos) {
  hooke_pair_p<RotMul<Mode>>(a, k, dn, n, cpos);
}

// The Hooke law on the contacts found by k_cdetect.  Mode bit 2 (instance 1):
// its multiplies on the integer pipe (contact_force_core_m); an operand outside
// that fast path makes the pair run again on the FP64 pipe from its stored
// inputs (nothing is written before write_result).
template <int Mode>
__global__ void __launch_bounds__(FT, (Mode ? 4 : 1)) k_chooke(CArgs a) {
  const uint64_t n2 = a.cnt[1];
  if (blockIdx.x == 0 && threadIdx.x == 0) *a.n_active = n2;  // every L2 pair overlaps (dn < 0)
  const uint64_t stride = (uint64_t)gridDim.x * FT;
  for (uint64_t w = (uint64_t)blockIdx.x * FT + threadIdx.x; w < n2; w += stride)
    hooke_pair<Mode>(a, a.L2[w], a.D[0][w], mk(a.D[1][w], a.D[2][w], a.D[3][w]), mk(a.D[4][w], a.D[5][w], a.D[6][w]));
}

// The law of queued pair idx of queue q (0: Hooke, 1: attraction); a share of
// the Hooke tiles runs on the integer pipe, so both pipes work at once.
template <int Mode, bool IntTiles, int T>
__device__ __forceinline__ void run_queued(const CArgs& a, int q, uint32_t idx, const uint32_t* qk,
                                           const double (*qd)[2 * T], uint32_t& tiles) {
  const V3 n = mk(qd[1][idx], qd[2][idx], qd[3][idx]);
  const V3 cpos = mk(qd[4][idx], qd[5][idx], qd[6][idx]);
  if (q == 0) {
    if (IntTiles && (int)(tiles & 7u) < a.int_share)
      hooke_pair_p<AllInt>(a, qk[idx], qd[0][idx], n, cpos);
    else
      hooke_pair<Mode>(a, qk[idx], qd[0][idx], n, cpos);
    tiles++;
  } else {
    attract_pair(a, qk[idx], qd[0][idx], n, cpos);
  }
}

// Detection and the contact laws in one kernel.  The pairs a block's detection
// finds overlapping (Hooke law) or within the cohesion distance (attraction)
// wait in shared memory, one queue per law, until a full tile of one kind is
// ready; then every thread of the block runs that law on one of them, so the
// FP64 warps stay dense and on one law, while the detection results never go
// through global memory.  The particle pairs of L1 come before its driver
// pairs, so the warps of both stages see one kind of pair at a time.  Each
// pair is computed exactly as by k_cdetect + k_chooke and writes only its own
// records: the same bits.  The overlapping pairs are counted into *n_active
// (zeroed by the launcher).
// Bound by the FP64 pipe (about 190 instructions per overlapping pair before, 160
// with the moment update and its clip, the sums with a zero moment and the spin
// of a resting partner decided on the integer pipe): with the same decisions in
// the epilog and the trigger a step of the 2 M bed went from 3.62 to 3.23 ms.
// IntTiles: the instance with the integer-pipe tiles (int_share > 0); it needs
// more registers, so the FP64-only instance stays the lean one.
// T: threads per block and pairs per tile, 128; or 32 for a small system, whose tiles
// then reach every SM (launch_contact_compact).
template <int Mode, bool IntTiles, int T>
__global__ void __launch_bounds__(T, (T < 128 ? 1 : (Mode ? 4 : (IntTiles ? 3 : 1)))) k_cfused(CArgs a) {
  __shared__ uint32_t q_k[2][2 * T];
  __shared__ double q_d[2][7][2 * T];
  __shared__ uint32_t q_n[2], q_tot;
  if (threadIdx.x == 0) {
    q_n[0] = q_n[1] = 0;
    q_tot = 0;
  }
  __syncthreads();
  const uint64_t n1 = a.cnt[0], nl = n1 + a.cnt[2];
  const uint64_t stride = (uint64_t)gridDim.x * T;
  const int lane = threadIdx.x & 31;
  const uint32_t t = threadIdx.x;
  uint32_t tiles = 0;  // Hooke tiles run by this block (the same count in every thread)
  for (uint64_t base = (uint64_t)blockIdx.x * T; base < nl; base += stride) {  // the same trips for the block
    const uint64_t w = base + threadIdx.x;
    int kind = PAIR_DONE;
    uint32_t k = 0;
    double dn = 0;
    V3 n = mk(0, 0, 0), cpos = mk(0, 0, 0);
    if (w < nl) {
      k = l1_at(a, w, n1);
      kind = detect_pair(a, k, dn, n, cpos);
    }
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const bool mine = kind == (q == 0 ? PAIR_HOOKE : PAIR_ATTRACT);
      const unsigned mask = __ballot_sync(0xffffffffu, mine);
      uint32_t wb = 0;
      const unsigned act = q == 0 ? __ballot_sync(0xffffffffu, mine && (!a.overlap_only || emu_lt0(dn))) : 0u;
      if (lane == 0 && act) atomicAdd(&q_tot, (uint32_t)__popc(act));
      if (lane == 0 && mask) {
        wb = atomicAdd(&q_n[q], (uint32_t)__popc(mask));
      }
      wb = __shfl_sync(0xffffffffu, wb, 0);
      if (mine) {
        const uint32_t pos = wb + (uint32_t)__popc(mask & ((1u << lane) - 1u));  // < 2 T: at most T - 1 wait
        q_k[q][pos] = k;
        q_d[q][0][pos] = dn;
        q_d[q][1][pos] = n.x;
        q_d[q][2][pos] = n.y;
        q_d[q][3][pos] = n.z;
        q_d[q][4][pos] = cpos.x;
        q_d[q][5][pos] = cpos.y;
        q_d[q][6][pos] = cpos.z;
      }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const uint32_t have = q_n[q];
      if (have >= T) {  // a full tile: one pair per thread
        run_queued<Mode, IntTiles, T>(a, q, t, q_k[q], q_d[q], tiles);
        __syncthreads();
        const uint32_t rest = have - T;  // < T: the waiting pairs move to the front
        if (t < rest) {
          q_k[q][t] = q_k[q][T + t];
#pragma unroll
          for (int c = 0; c < 7; c++) q_d[q][c][t] = q_d[q][c][T + t];
        }
        if (t == 0) q_n[q] = rest;
        __syncthreads();
      }
    }
  }
  if (t < q_n[0]) run_queued<Mode, IntTiles, T>(a, 0, t, q_k[0], q_d[0], tiles);
  if (t < q_n[1]) run_queued<Mode, IntTiles, T>(a, 1, t, q_k[1], q_d[1], tiles);
  if (t == 0 && q_tot) atomicAdd(a.n_active, (unsigned long long)q_tot);
}

// |r - b|^2 >= thr2, decided from FP32 differences (diff_f32) outside a band of
// 2^-15 about the threshold: their error is 2^-23 of the difference and 2^-52 of the
// coordinate, which the lower bound on the threshold keeps below 2^-20 of it.
// Inside the band, or for a skin below 2^-30 of a coordinate, the FP64 pipe decides.
__device__ __forceinline__ bool displ_over(V3 r, V3 b, double thr2, float thr2f) {
  bool ok = thr2f > 1e-30f && thr2f < 1e30f;
  uint32_t top = 0;
  const float ex = diff_f32(r.x, b.x, ok, top), ey = diff_f32(r.y, b.y, ok, top), ez = diff_f32(r.z, b.z, ok, top);
  const float s = ex * ex + ey * ey + ez * ez;
  // 2^(top - 1022) bounds the coordinates; sqrt(thr2) >= 2^-30 of it
  const int et = (int)(__float_as_uint(thr2f) >> 23) - 127;
  if (ok && et >= 2 * ((int)top - 1022 - 30)) {
    if (s < thr2f * 0.99997f) return false;
    if (s > thr2f * 1.00003f) return true;
  }
  const double dx = r.x - b.x, dy = r.y - b.y, dz = r.z - b.z;
  return emu_ge_nonneg(dx * dx + dy * dy + dz * dz, thr2);  // >= on the integer pipe
}

// The integration: reset_force_moment + gravity_force + contact gather +
// force_to_accel + epilog of a step (epilog), then the prolog and the displacement
// trigger of the next (prolog).  In the graph step one launch does both, so a
// particle's velocity and acceleration stay in registers and a step has one launch
// fewer; the host-launched step and the ends of a call run the halves apart.
//
// The rotational halves are exactly idle or integer logic for many particles
// (rotation_idle, spin_free_step); the others run them here when more than `dense`
// lanes of their warp need it, otherwise the block puts them off and runs them packed
// at its end, so sparse rotating particles do not hold whole warps on the FP64 pipe (a
// list for a kernel of its own packs a little better, and cost 6 us a step when empty:
// 50 k mixer, 20 steps, 3.55 -> 3.31 ms, 125 k bed 5.45 -> 5.28 ms, 2 M bed 15.4 both).
// The trigger depends on positions only.
//
// In the graph the last block to finish does what four memsets and a kernel of one
// thread did: it hands the flag to the conditional rebuild and zeroes the counters
// of the coming contact pass.
// Mode != 0: the integer-pipe multiplies raise register use; at most 80
// registers keep 3 blocks of 256 per SM (measured faster than 2 blocks)
template <int Mode>
__global__ void __launch_bounds__(256, (Mode ? 3 : 1)) k_integrate(IntegArgs a) {
  const PArrays& P = a.P;
  const uint64_t s = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool epi = a.gs ? a.gs[GS_STEP] != 0ull : a.epilog != 0;
  const bool pro = a.prolog != 0;
  const bool mine = s < a.n;
  V3 v = mk(0.0, 0.0, 0.0), acc = v;
  __shared__ PutOff off;
  if (a.dense) {
    if (threadIdx.x == 0) off.n = 0u;
    __syncthreads();
  }
  bool late = false;  // the epilog's rotation is put off
  if (epi) {
    bool need = false;
    V3 mom = mk(0.0, 0.0, 0.0);
    if (mine) {
      need = epilog_translate<Mode>(a, s, v, acc, mom);
      if (!pro) {
        P.f[VX][s] = v.x;
        P.f[VY][s] = v.y;
        P.f[VZ][s] = v.z;
      }
    }
    late = __popc(__ballot_sync(0xffffffffu, need)) <= a.dense && need;
    if (need && !late) epilog_rotation<Mode>(P, s, a.hdt, mom);
  }
  bool over = false, turn = false;
  if (pro && mine) {
    if (!epi) {
      v = mk(P.f[VX][s], P.f[VY][s], P.f[VZ][s]);
      acc = mk(P.f[FX][s], P.f[FY][s], P.f[FZ][s]);
    }
    const V3 r0 = mk(P.f[RX][s], P.f[RY][s], P.f[RZ][s]);
    LinMul<Mode> lm;
    V3 r = r0, u = v;
    transl_math_z(lm, r, u, acc, a.dt, a.hdt, a.dt2_2);
    if (lm.failed()) {
      MulFP64 nm;
      r = r0;
      u = v;
      transl_math_z(nm, r, u, acc, a.dt, a.hdt, a.dt2_2);
    }
    P.f[RX][s] = r.x;
    P.f[RY][s] = r.y;
    P.f[RZ][s] = r.z;
    P.f[VX][s] = u.x;
    P.f[VY][s] = u.y;
    P.f[VZ][s] = u.z;
    if (!late) turn = !prolog_spin_free<Mode>(P, s, a.dt, a.hdt);
    over = displ_over(r, mk(P.f[BX][s], P.f[BY][s], P.f[BZ][s]), a.thr2, a.thr2f);
    if (over && a.sv.nsys > 1) atomicOr(&a.sv.trig[a.sv.of(s)], 1u);  // this system's own trigger
  }
  if (__any_sync(0xffffffffu, over) && (threadIdx.x & 31) == 0) atomicOr(a.scal, 1ull);
  if (__popc(__ballot_sync(0xffffffffu, turn)) > a.dense && turn) {
    prolog_rotation<Mode>(P, s, a.dt, a.hdt);
    turn = false;
  }
  if (a.dense) {
    put_off(off, late || turn, (uint32_t)s | (late ? ROT_EPILOG : 0u));
    __syncthreads();
    if (threadIdx.x < off.n) {
      const uint32_t e = off.s[threadIdx.x], w = e & ~ROT_EPILOG;
      if (e & ROT_EPILOG) epilog_rotation<Mode>(P, w, a.hdt, mk(P.f[MX][w], P.f[MY][w], P.f[MZ][w]));
      if (pro && !prolog_spin_free<Mode>(P, w, a.dt, a.hdt)) prolog_rotation<Mode>(P, w, a.dt, a.hdt);
    }
  }
  if (a.gs) {
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      if (atomicAdd(a.gs + GS_DONE, 1ull) == gridDim.x - 1) {  // every block's flag is in
        const unsigned long long flag = atomicExch(a.scal, 0ull);
        cudaGraphSetConditional(a.cond, flag ? 1u : 0u);
        a.scal[1] = a.scal[3] = a.scal[4] = a.scal[5] = 0ull;  // active contacts, work list counts
        a.gs[GS_DONE] = 0ull;
        a.gs[GS_STEP] += 1ull;
      }
    }
  }
}

CArgs make_cargs(dem_ctx* c) {
  CArgs a;
  a.P = c->P[c->pcur];
  a.I = c->I[c->icur];
  a.R = c->R;
  a.ni = c->ni;
  a.ni_dev = c->capturing ? c->d_ni : nullptr;
  a.sv = c->sysview();
  a.drv = c->drv_dev;
  a.mesh = c->mesh_dev;
  a.cp = c->prm.config;
  a.cpd = c->prm.config_driver;
  a.dt = c->prm.dt;
  a.cohesive = c->prm.law == DEM_LAW_HOOKE_COHESIVE;
  a.dmt = c->prm.law == DEM_LAW_HOOKE_DMT;
  a.pt = c->ptable();
  a.cs = c->cs;
  a.screen = c->prm.fp32_contact_screen && !c->analysis;  // analysis: every pair's state
  a.dncut_f = (float)std::max(c->prm.config.dncut, 0.0);
  a.L1 = c->L1;
  a.L2 = c->L2;
  for (int q = 0; q < 7; q++) a.D[q] = c->Dscr[q];
  a.cnt = c->d_scalars + 3;
  a.l1cap = c->rcap;
  a.int_share = c->tune_int_share;
  a.n_active = c->d_scalars + 1;
  return a;
}
}  // namespace

IntegArgs make_integ_args(dem_ctx* c, int epilog, int prolog) {
  IntegArgs a;
  a.P = c->P[c->pcur];
  a.R = c->R;
  a.n = c->n;
  a.own_off = c->own_off[c->icur];
  a.rev_off = c->rev_off;
  a.rev_idx = c->rev_idx;
  a.stamp = c->pstamp;
  a.pass = c->poly ? c->live_pass : 0u;
  for (int d = 0; d < 3; d++) a.g[d] = c->prm.gravity[d];
  a.dt = c->prm.dt;
  a.hdt = a.dt * 0.5;
  a.dt2_2 = a.dt * a.dt * 0.5;
  const double max_displ = c->prm.rcut_inc * 0.5;
  a.thr2 = max_displ * max_displ;
  a.thr2f = (float)a.thr2;
  a.sv = c->sysview();
  a.scal = c->d_scalars;
  a.dense = rotation_dense(c);
  a.epilog = epilog;
  a.prolog = prolog;
  a.gs = nullptr;
  a.cond = 0;
  a.step = 0;
  a.nb = 0;
  return a;
}

// cond: inside a capture, the handle of the conditional rebuild (both halves; the
// first step of a call has no epilog)
static int launch_integrate(dem_ctx* c, int epilog, int prolog, cudaGraphConditionalHandle cond) {
  IntegArgs a = make_integ_args(c, epilog, prolog);
  a.gs = c->capturing ? c->d_gs : nullptr;
  a.cond = cond;
  const unsigned block = particle_block(c);
  ProfScope ps(c, epilog ? K_EPILOG : K_PROLOG, c->n ? 1 : 0);
  if (c->n) {
    const int mode = integ_mode(c);
    const auto kern = by_mode(mode, k_integrate<0>, k_integrate<1>, k_integrate<2>, k_integrate<3>);
    kern<<<grid_for(c->n, block), block, 0, c->stream>>>(a);
  }
  DEM_CUDA_TRY(c, cudaGetLastError());
  return DEM_OK;
}
int launch_fused_prolog(dem_ctx* c) {
  DEM_CUDA_TRY(c, cudaMemsetAsync(c->d_scalars, 0, sizeof(unsigned long long), c->stream));
  return launch_integrate(c, 0, 1, 0);
}
int launch_fused_epilog(dem_ctx* c) { return launch_integrate(c, 1, 0, 0); }
int launch_graph_integrate(dem_ctx* c, cudaGraphConditionalHandle cond) { return launch_integrate(c, 1, 1, cond); }

int launch_contact_compact(dem_ctx* c, bool overlap_only) {
  // (in a graph the integration's last block zeroes these counts)
  if (!c->capturing)
    DEM_CUDA_TRY(c, cudaMemsetAsync(c->d_scalars + 3, 0, 3 * sizeof(unsigned long long), c->stream));
  CArgs a = make_cargs(c);
  a.overlap_only = overlap_only ? 1 : 0;
  const unsigned persistent = (unsigned)c->num_sms * (unsigned)c->tune_contact_bps;
  // Up to a particle for every lane of four warps an SM (20 k particles, some 60 k
  // pairs) tiles of one warp spread over all SMs and its FP64 units; above, a block
  // of four warps shares a queue, so fewer partly filled tiles run at its end.
  const bool small = c->n <= (uint64_t)c->num_sms * 128u;
  const unsigned warps = persistent * (FT / 32);
  {
    ProfScope ps(c, K_CSCREEN, c->capturing || c->ni ? 1 : 0);
    const unsigned block = small ? 32u : 128u;
    if (c->capturing)
      k_cscreen<<<small ? warps : persistent, block, 0, c->stream>>>(a);
    else if (c->ni)
      k_cscreen<<<grid_for(c->ni, block), block, 0, c->stream>>>(a);
  }
  if (c->fuse_contact || overlap_only) {  // detection and law in one kernel (k_cfused)
    if (!c->capturing) DEM_CUDA_TRY(c, cudaMemsetAsync(a.n_active, 0, sizeof(unsigned long long), c->stream));
    ProfScope ps(c, K_CONTACT, 1);
    // mode bit 2: the contact law's multiplies on the integer pipe; int_share: a
    // share of its tiles with multiplies and additions there
    if (c->mul_mode & 4)
      k_cfused<1, false, 128><<<persistent, 128, 0, c->stream>>>(a);
    else if (c->tune_int_share > 0)
      k_cfused<0, true, 128><<<persistent, 128, 0, c->stream>>>(a);
    else if (small)
      k_cfused<0, false, 32><<<warps, 32, 0, c->stream>>>(a);
    else
      k_cfused<0, false, 128><<<persistent, 128, 0, c->stream>>>(a);
  } else {
    {
      ProfScope ps(c, K_CDETECT, 1);
      k_cdetect<<<persistent, FT, 0, c->stream>>>(a);
    }
    ProfScope ps(c, K_CONTACT, 1);  // the Hooke law on the contacts
    const auto kh = (c->mul_mode & 4) ? k_chooke<1> : k_chooke<0>;  // mode bit 2: the contact law
    kh<<<persistent, FT, 0, c->stream>>>(a);
  }
  DEM_CUDA_TRY(c, cudaGetLastError());
  return DEM_OK;
}

}  // namespace dem
