// k_neigh_sphere.cu -- sphere interaction-list rebuild (exact two-pass count / fill).
//
// Replaces chunk_neighbors_contact (src/grid/chunk_neighbors_contact.cpp:45-57),
// nbh_sphere in symetric mode (src/sphere/nbh_sphere.cu:64-309) and
// classify_interactions (src/interaction/classify_interactions.cpp:52-136):
//   - drivers first: Surface / Cylinder filters with r + rcut_inc
//     (nbh_sphere.cu:140-233, surface.hpp:320-324, cylinder.hpp:225-235);
//   - particle pairs over the 27-cell stencil with the FP64 filter
//     d2 > 0 && d2 < (r_a + r_b + rcut_inc)^2 && d2 < nbh_dist^2;
//     a pair is owned by the smaller id, except when the partner is a periodic
//     ghost image, which is kept from both sides (nbh_sphere.cu:244-249);
//   - each owner's list sorted by InteractionPair order, history (friction,
//     moment) carried over from the previous list by key equality
//     (interaction_manager.hpp:89-112, placeholder_interaction.hpp:398-408).
// Plain FP64 path (k_count / k_fill): one thread per owner particle; particles
// are in cell order so the stencil reads of neighbouring threads hit the same
// cells (L1/L2 reuse).  FP32 broad phase (k_count_pairs / k_fill_entries): each pair
// met once, appended to its owner's record, the records ordered by rank; or, as an
// option, (k_cell_count / k_cell_fill): one warp
// per cell, its 27-cell neighbourhood staged in shared memory, candidates
// compacted with ballots, each owner's list ordered by a warp rank sort; the
// drivers per particle (k_pre_count / k_pre_fill).  In a batched context the particle's system gives the grid, its cell block and
// its drivers; a system rebuilt without its own trigger kept its slots, and
// its previous list is copied as is (so its list is the one it has alone).
#include "../../include/dem_selftest.h"
#include "broad_core.cuh"
#include "mesh_core.cuh"

namespace dem {
namespace {

struct BPArgs {
  PArrays P;
  uint64_t n;
  SysView sv;
  const uint32_t* cell_start;
  const uint32_t* cell_of;
  const DriverDev* drv;
  int ndrv;
  const MeshDev* mesh;  // mesh drivers (DriverDev::mesh)
  int has_mesh;         // a mesh driver is registered: k_mesh_count / k_mesh_fill ran
  const uint32_t* mcnt;  // per sphere: its mesh candidates (k_mesh_count)
  double skin;
  double rcut2;
  // FP32 broad phase: cell-relative coordinates and radii, cell sizes, skin
  const float4* crel;
  float skin_f;
  uint64_t cap;  // interaction buffer capacity (graph step): a fill beyond it writes nothing
  // FP32 path: the count pass's candidates of each particle (nrec per particle,
  // then nmrec mesh candidates:
  // partner, meta, partner id), read by the fill when they fit
  uint4* srec;
  uint32_t nrec, nmrec;
  uint32_t* rev_cnt;  // FP32 path: the fill's count of each particle's partner list
  uint32_t* rev_pos;  // and the place of each entry in it (a scratch of the records' capacity)
  // per-pair damping damp_rate 2 sqrt(kn meff), in the operation order of the
  // contact law: (damp_rate * 2) * sqrt(kn * meff), meff = (m_i m_j)/(m_i + m_j)
  // for particle pairs, m_i for drivers; the pair's parameter set
  dem_contact_params cp, cpd;
  ParamTable pt;
};

__device__ __forceinline__ double pair_damp(const BPArgs& a, uint32_t i, uint32_t j, uint32_t meta) {
  const double mi = a.P.f[MASS][i];
  if (meta_type(meta) == DEM_ITYPE_VERTEX_VERTEX) {
    const dem_contact_params& q = a.pt.pair(a.cp, a.P.group[i], a.P.group[j]);
    const double mj = a.P.f[MASS][j];
    const double meff = (mi * mj) / (mi + mj);
    return q.damp_rate * 2.0 * sqrt(q.kn * meff);
  }
  const dem_contact_params& q = a.pt.drv(a.cpd, a.P.group[i], j);
  return q.damp_rate * 2.0 * sqrt(q.kn * mi);
}

// FP32 decision of the broad-phase filter d2 > 0 && d2 < (r_i + r_j + skin)^2.
// Coordinates are relative to each particle's cell origin, so |x_rel| is
// about one cell and the FP32 difference vector has an absolute error below
// 2^-22 (|x_rel_i| + |x_rel_j| + cell): three roundings of magnitudes bounded by
// that sum (conversion of each coordinate, then subtraction and addition of the
// cell offset).  The FP32 radius sum has a relative error below 2^-22.  m is 8x
// the sum of both bounds; outside [rm - m, rm + m] the FP32 comparison equals
// the FP64 one; inside, and near d = 0, the caller runs the exact FP64 test.
// Returns 1 = keep, 0 = drop, -1 = undecided.
__device__ __forceinline__ int f32_decide(float ex, float ey, float ez, float si, float sj, float cmax, float rm) {
  const float d2f = ex * ex + ey * ey + ez * ez;
  const float m = (si + sj + cmax) * 1.9073486e-06f /* 2^-19 */ + rm * 9.5367432e-07f /* 2^-20 */;
  const float hi = rm + m;
  if (d2f > hi * hi) return 0;
  const float lo = rm - m;
  if (lo > 0.f && d2f < lo * lo && d2f > 4.f * m * m) return 1;
  return -1;
}

__device__ inline bool driver_filter(const DriverDev& d, double rcut, V3 p) {
  if (d.kind == 0) {
    const V3 nrm = mk(d.normal[0], d.normal[1], d.normal[2]);
    const V3 proj = dot(p, nrm) * nrm;
    const double dd = vnorm(proj - mk(d.center_proj[0], d.center_proj[1], d.center_proj[2]));
    return dd <= rcut;
  }
  const V3 proj = p * mk(d.axis[0], d.axis[1], d.axis[2]);
  const V3 dir = proj - mk(d.center[0], d.center[1], d.center[2]);
  const double dd = vnorm(dir);
  const double dn = d.radius - (dd + rcut);
  return dn <= 0;
}

// the stationary drivers (surfaces, cylinders) of particle s's system that pass the filter
template <class Emit>
__device__ inline void for_each_driver(const BPArgs& a, uint32_t s, int sys, Emit&& emit) {
  const V3 ri = mk(a.P.f[RX][s], a.P.f[RY][s], a.P.f[RZ][s]);
  const double radi = a.P.f[RAD][s];
  const int2 dr = a.sv.drange[sys];
  for (int k = dr.x; k < dr.x + dr.y; k++) {
    const DriverDev& d = a.drv[k];
    if (d.kind == 2) continue;  // mesh drivers: mesh_phase
    if (driver_filter(d, radi + a.skin, ri))
      emit((uint32_t)k, (uint64_t)k,
           make_meta(d.kind == 0 ? DEM_ITYPE_VERTEX_SURFACE : DEM_ITYPE_VERTEX_CYLINDER, 0, 0, 0, false), 0u);
  }
}

// the particle candidates of owner s over the 27-cell stencil, in stencil order
template <bool F32, class Emit>
__device__ inline void for_each_particle(const BPArgs& a, uint32_t s, int sys, Emit&& emit) {
  const double* __restrict__ rx = a.P.f[RX];
  const double* __restrict__ ry = a.P.f[RY];
  const double* __restrict__ rz = a.P.f[RZ];
  const double* __restrict__ rad = a.P.f[RAD];
  const uint64_t* __restrict__ id = a.P.id;
  const V3 ri = mk(rx[s], ry[s], rz[s]);
  const double radi = rad[s];
  const uint64_t idi = id[s];
  const GridDev& g = a.sv.g[sys];
  const uint32_t coff = a.sv.coff[sys];
  float xri = 0.f, yri = 0.f, zri = 0.f, rfi = 0.f, si = 0.f, cmax = 0.f;
  const float csx = (float)g.csz[0], csy = (float)g.csz[1], csz = (float)g.csz[2];
  if (F32) {
    const float4 me = a.crel[s];
    xri = me.x;
    yri = me.y;
    zri = me.z;
    rfi = me.w;
    si = fmaxf(fabsf(xri), fmaxf(fabsf(yri), fabsf(zri)));
    cmax = fmaxf(csx, fmaxf(csy, csz));
  }
  const uint32_t c = a.cell_of[s] - coff;
  const int d0 = g.dims[0], d1 = g.dims[1], d2n = g.dims[2];
  const int cx = (int)(c % (uint32_t)d0);
  const int cy = (int)((c / (uint32_t)d0) % (uint32_t)d1);
  const int cz = (int)(c / ((uint32_t)d0 * (uint32_t)d1));
  for (int dz = -1; dz <= 1; dz++) {
    int z = cz + dz, sz = 0;
    if (z < 0) {
      if (!g.periodic[2]) continue;
      z += d2n;
      sz = -1;
    } else if (z >= d2n) {
      if (!g.periodic[2]) continue;
      z -= d2n;
      sz = 1;
    }
    for (int dy = -1; dy <= 1; dy++) {
      int y = cy + dy, sy = 0;
      if (y < 0) {
        if (!g.periodic[1]) continue;
        y += d1;
        sy = -1;
      } else if (y >= d1) {
        if (!g.periodic[1]) continue;
        y -= d1;
        sy = 1;
      }
      for (int dx = -1; dx <= 1; dx++) {
        int x = cx + dx, sx = 0;
        if (x < 0) {
          if (!g.periodic[0]) continue;
          x += d0;
          sx = -1;
        } else if (x >= d0) {
          if (!g.periodic[0]) continue;
          x -= d0;
          sx = 1;
        }
        const uint32_t cc = coff + (uint32_t)x + (uint32_t)d0 * ((uint32_t)y + (uint32_t)d1 * (uint32_t)z);
        uint32_t qb = a.cell_start[cc];
        const uint32_t qe = a.cell_start[cc + 1];
        const bool ghost = (sx | sy | sz) != 0;
        const float oxf = (float)dx * csx, oyf = (float)dy * csy, ozf = (float)dz * csz;
        if (!ghost) {  // a cell's particles are in id order: the owner rule keeps the suffix above idi
          uint32_t hi = qe;
          while (qb < hi) {
            const uint32_t mid = (qb + hi) >> 1;
            if (id[mid] <= idi)
              qb = mid + 1;
            else
              hi = mid;
          }
        }
        for (uint32_t q = qb; q < qe; q++) {
          const uint64_t idj = id[q];
          if (!ghost && idi >= idj) continue;  // owner rule (kept: the suffix already satisfies it)
          int keep = -1;
          if (F32) {
            const float4 cq = a.crel[q];
            const float xj = cq.x, yj = cq.y, zj = cq.z;
            const float sj = fmaxf(fabsf(xj), fmaxf(fabsf(yj), fabsf(zj)));
            keep = f32_decide((xj - xri) + oxf, (yj - yri) + oyf, (zj - zri) + ozf, si, sj, cmax,
                              rfi + cq.w + a.skin_f);
          }
          if (keep < 0) {
            V3 rj = mk(rx[q], ry[q], rz[q]);
            if (sx) rj.x = rj.x + (double)sx * g.L[0];
            if (sy) rj.y = rj.y + (double)sy * g.L[1];
            if (sz) rj.z = rj.z + (double)sz * g.L[2];
            const double ddx = rj.x - ri.x, ddy = rj.y - ri.y, ddz = rj.z - ri.z;
            const double d2 = ddx * ddx + ddy * ddy + ddz * ddz;
            const double rmax = radi + rad[q] + a.skin;
            keep = (d2 > 0.0 && d2 < rmax * rmax && d2 < a.rcut2) ? 1 : 0;
          }
          if (!keep) continue;
          emit(q, idj, make_meta(DEM_ITYPE_VERTEX_VERTEX, sx, sy, sz, ghost), 0u);
        }
      }
    }
  }
}

// drivers, then particles (the emission order of the thread-per-owner kernels)
template <bool F32, class Emit>
__device__ inline void for_each_candidate(const BPArgs& a, uint32_t s, Emit&& emit) {
  const int sys = a.sv.of(s);
  for_each_driver(a, s, sys, emit);
  for_each_particle<F32>(a, s, sys, emit);
}

// InteractionPair order inside the owner: (partner id, type, partner sub); swap
// and the owner sub are 0 for spheres
__device__ inline bool key_less(uint64_t pa, uint32_t ta, uint32_t sa, uint64_t pb, uint32_t tb, uint32_t sb) {
  return pa < pb || (pa == pb && (ta < tb || (ta == tb && sa < sb)));
}

// Entry (qa, ma) before (qb, mb) among entries of one owner with equal keys: particles that
// share an id.  They follow the stencil, as for_each_particle meets them: by the cell of
// the image in z, y and x, then by slot.  Distinct ids never come here.
__device__ __noinline__ bool image_before(const BPArgs& a, int sys, uint32_t qa, uint32_t ma, uint32_t qb, uint32_t mb) {
  const GridDev& g = a.sv.g[sys];
  const uint32_t coff = a.sv.coff[sys];
  int ca[3], cb[3];
  cell_coords(g, a.cell_of[qa] - coff, ca[0], ca[1], ca[2]);
  cell_coords(g, a.cell_of[qb] - coff, cb[0], cb[1], cb[2]);
  for (int d = 2; d >= 0; d--) {
    const int ia = ca[d] + meta_shift(ma, d) * g.dims[d], ib = cb[d] + meta_shift(mb, d) * g.dims[d];
    if (ia != ib) return ia < ib;
  }
  return qa < qb;
}
// The order of entry a of an owner before its entry b.  first orders two entries that
// nothing else tells apart, so that the ranks of an owner's entries are always a
// permutation of their places: two entries on one place leave another one unwritten.
__device__ __forceinline__ bool entry_before(const BPArgs& a, int sys, uint64_t pa, uint32_t ma, uint32_t sa, uint32_t qa,
                                             uint64_t pb, uint32_t mb, uint32_t sb, uint32_t qb, bool first) {
  if (pa != pb) return pa < pb;
  const uint32_t ta = meta_type(ma), tb = meta_type(mb);
  if (ta != tb) return ta < tb;
  if (sa != sb) return sa < sb;
  if (ta != DEM_ITYPE_VERTEX_VERTEX || (qa == qb && ma == mb)) return first;
  return image_before(a, sys, qa, ma, qb, mb);
}

// Mesh candidates (detection_sphere_driver, nbh_sphere.hpp:25-86): every mesh
// vertex, edge and face of the sphere's bin that passes its filter, partner
// sub = the feature.  A block serves the spheres s of its first 32 threads (want), which
// find their spheres' bins; the bins' items are then dealt to all its threads in one
// sequence: a test is a chain of loads and FP32 operations of some 5 us, and a bin can list
// hundreds of features (where many triangles meet).  The spheres of a block lie far apart
// in the cell order (mesh_sphere), so neighbours at such a place fall to different blocks.
// emit(s, at, k, kind, j) takes the passing items of sphere s, at counting them in no
// particular order (the fill orders a sphere's entries by their keys).  Returns the
// thread's own sphere's count.  Every thread of the block calls it.
constexpr int MESH_BLOCK = 128;
constexpr int MESH_SPHERES = 32;
struct MeshWork {
  uint32_t pre[MESH_SPHERES + 1], s[MESH_SPHERES], q0[MESH_SPHERES], mesh[MESH_SPHERES], cnt[MESH_SPHERES];
  int k[MESH_SPHERES];
  float R[MESH_SPHERES], pabs[MESH_SPHERES];
  Split3 p[MESH_SPHERES];
  int nk;
};
template <bool F32, class Emit>
__device__ uint32_t mesh_phase(const BPArgs& a, uint64_t s, bool want, MeshWork& w, Emit&& emit) {
  constexpr unsigned FULL = 0xffffffffu;
  const int t = threadIdx.x;
  const bool lead = t < MESH_SPHERES;  // one warp
  V3 p = mk(0.0, 0.0, 0.0);
  double rad = 0.0;
  int2 dr = make_int2(0, 0);
  if (lead) {
    Split3 sp{};
    if (want) {
      p = mk(a.P.f[RX][s], a.P.f[RY][s], a.P.f[RZ][s]);
      rad = a.P.f[RAD][s];
      dr = a.sv.drange[a.sv.of(s)];
      if (F32) sp = split3(p);
    }
    w.s[t] = (uint32_t)s;
    w.cnt[t] = 0u;
    w.p[t] = sp;
    w.pabs[t] = fabsf(sp.h.x) + fabsf(sp.h.y) + fabsf(sp.h.z);
    const int nk = __reduce_max_sync(FULL, dr.y);
    if (t == 0) w.nk = nk;
  }
  __syncthreads();
  const int nk = w.nk;
  for (int kk = 0; kk < nk; kk++) {
    if (lead) {
      const int k = dr.x + kk;
      uint32_t len = 0;
      if (kk < dr.y && a.drv[k].kind == 2) {
        const uint32_t mesh = (uint32_t)a.drv[k].mesh;
        const MeshDev& m = a.mesh[mesh];
        uint64_t bb;
        if (mesh_bin_of(m, p, bb)) {
          const uint32_t q0 = m.boff[bb];
          len = m.boff[bb + 1] - q0;
          w.q0[t] = q0;
          w.mesh[t] = mesh;
          w.k[t] = k;
          if (F32 && len) w.R[t] = f32_rn(rad + m.r + a.skin);
        }
      }
      uint32_t sum = len;
#pragma unroll
      for (int o = 1; o < MESH_SPHERES; o <<= 1) {
        const uint32_t v = __shfl_up_sync(FULL, sum, o);
        if (t >= o) sum += v;
      }
      w.pre[t] = sum - len;
      if (t == MESH_SPHERES - 1) w.pre[MESH_SPHERES] = sum;
    }
    __syncthreads();
    const uint32_t total = w.pre[MESH_SPHERES];
    for (uint32_t i = t; i < total; i += MESH_BLOCK) {
      int L = 0;  // the last sphere whose items start at or before i
#pragma unroll
      for (int o = MESH_SPHERES / 2; o; o >>= 1)
        if (i >= w.pre[L + o]) L += o;
      const MeshDev& m = a.mesh[w.mesh[L]];
      const uint32_t it = m.bitem[w.q0[L] + (i - w.pre[L])], kind = it >> 30, j = it & 0x3fffffffu, o = w.s[L];
      const bool pass = F32 ? mesh_filter_f32(m, kind, j, a.skin, a.skin_f, w.p[L], w.R[L], w.pabs[L], a.P.f, o)
                            : mesh_filter(m, kind, j, a.skin, mk(a.P.f[RX][o], a.P.f[RY][o], a.P.f[RZ][o]),
                                          a.P.f[RAD][o]);
      if (pass) emit(o, atomicAdd(&w.cnt[L], 1u), (uint32_t)w.k[L], kind, j);
    }
    __syncthreads();
  }
  return lead ? w.cnt[t] : 0u;
}

// the sphere of one of a block's first 32 threads
__device__ __forceinline__ uint64_t mesh_sphere() { return (uint64_t)threadIdx.x * gridDim.x + blockIdx.x; }

// The mesh candidates of each triggered sphere.  Kept out of the count and fill kernels so
// the particle-pair passes keep their register budget.  With Rec they become the first
// records of the sphere (k_fill_entries): partner the driver, the feature in the place of
// the partner id, in any order.  Bound by the loads of the longest blocks.  Measured, 50 k
// mixer (1680 spheres with up to 50 candidates each): 45 us, a warp a sphere with the bin and
// the differences in FP64 114 us, and as much again in the fill, which now reads the records.
template <bool F32, bool Rec>
__global__ void __launch_bounds__(MESH_BLOCK) k_mesh_count(BPArgs a, uint32_t* __restrict__ mcnt,
                                                           uint32_t* __restrict__ cnt) {
  __shared__ MeshWork w;
  const uint64_t s = mesh_sphere();
  const bool own = threadIdx.x < MESH_SPHERES && s < a.n;
  const bool trig = own && a.sv.triggered(a.sv.of(s));
  uint4* const rec = a.srec;
  const uint32_t m =
      mesh_phase<F32>(a, s, trig, w, [&](uint32_t o, uint32_t at, uint32_t k, uint32_t kind, uint32_t j) {
        if (Rec && at < a.nmrec)
          rec[(uint64_t)o * (a.nrec + a.nmrec) + a.nrec + at] =
              make_uint4(k, make_meta(DEM_ITYPE_VERTEX_MESH_VERTEX + kind, 0, 0, 0, false), j << 16, 0u);
      });
  if (own) {
    mcnt[s] = m;
    cnt[s] = m;  // the particle candidates are added to it
  }
}
// The mesh items of each triggered sphere at the start of its segment, in key order; with
// Rec all entries of the spheres whose records overflowed, the others of the list not at
// all.  The items are first put into the history's arrays, unordered, and then ranked by
// the block's threads.
template <bool F32, bool Rec>
__global__ void __launch_bounds__(MESH_BLOCK) k_mesh_fill(BPArgs a, const uint32_t* __restrict__ off, IArrays dst) {
  __shared__ MeshWork w;
  const uint64_t s = mesh_sphere();
  const bool own = threadIdx.x < MESH_SPHERES && s < a.n;
  const uint32_t b = own ? off[s] : 0u, e = own ? off[s + 1] : 0u, mm = own ? a.mcnt[s] : 0u;
  const bool want = own && e <= a.cap && a.sv.triggered(a.sv.of(s)) &&
                    (Rec ? mm > a.nmrec || e - b - mm > a.nrec : mm > 0u);
  if (!__syncthreads_or(want)) return;
  auto put = [&](uint32_t x, uint32_t partner, uint64_t pid, uint32_t meta, uint32_t sub) {
    dst.ft[0][x] = emu_double((uint64_t)partner | (uint64_t)sub << 32);
    dst.ft[1][x] = emu_double(pid);
    dst.ft[2][x] = emu_double(meta);
  };
  mesh_phase<F32>(a, s, want, w, [&](uint32_t o, uint32_t at, uint32_t k, uint32_t kind, uint32_t j) {
    const uint32_t x = off[o] + at;
    if (x < off[o + 1]) put(x, k, k, make_meta(DEM_ITYPE_VERTEX_MESH_VERTEX + kind, 0, 0, 0, false), j << 16);
  });
  if (Rec && want) {
    uint32_t x = b + mm;
    if (e - x <= a.nrec) {
      const uint4* const rec = a.srec + s * (a.nrec + a.nmrec);
      for (uint32_t y = 0; x < e; x++, y++) put(x, rec[y].x, (uint64_t)rec[y].z | (uint64_t)rec[y].w << 32, rec[y].y, 0u);
    } else {
      for_each_candidate<true>(a, (uint32_t)s, [&](uint32_t q, uint64_t pid, uint32_t meta, uint32_t sub) {
        if (x < e) put(x, q, pid, meta, sub);
        x++;
      });
    }
  }
  if (threadIdx.x < MESH_SPHERES) {
    w.cnt[threadIdx.x] = want ? (Rec ? e - b : mm) : 0u;
    w.q0[threadIdx.x] = b;
  }
  __syncthreads();
  for (int L = 0; L < MESH_SPHERES; L++) {
    const uint32_t n = w.cnt[L], first = w.q0[L];
    const int sys = n ? a.sv.of(w.s[L]) : 0;
    for (uint32_t x = threadIdx.x; x < n; x += MESH_BLOCK) {
      const uint64_t word = emu_bits(dst.ft[0][first + x]), pid = emu_bits(dst.ft[1][first + x]);
      const uint32_t meta = (uint32_t)emu_bits(dst.ft[2][first + x]), sub = (uint32_t)(word >> 32);
      uint32_t rank = 0;
      for (uint32_t y = 0; y < n; y++) {
        const uint64_t wy = emu_bits(dst.ft[0][first + y]);
        rank += entry_before(a, sys, emu_bits(dst.ft[1][first + y]), (uint32_t)emu_bits(dst.ft[2][first + y]),
                             (uint32_t)(wy >> 32), (uint32_t)wy, pid, meta, sub, (uint32_t)word, y < x)
                    ? 1u
                    : 0u;
      }
      const uint32_t x1 = first + rank;
      dst.partner[x1] = (uint32_t)word;
      dst.pid[x1] = pid;
      dst.meta[x1] = meta;
      dst.sub[x1] = sub;
    }
  }
}

__global__ void k_count(BPArgs a, uint32_t* __restrict__ cnt, const uint32_t* __restrict__ old_off) {
  const uint64_t s = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= a.n) return;
  if (!a.sv.triggered(a.sv.of(s))) {  // slot kept (k_reorder): the previous list is copied
    cnt[s] = old_off[s + 1] - old_off[s];
    return;
  }
  uint32_t m = a.has_mesh ? a.mcnt[s] : 0u;
  for_each_candidate<false>(a, (uint32_t)s, [&](uint32_t, uint64_t, uint32_t, uint32_t) { m++; });
  cnt[s] = m;
}

// FP32 broad phase, count pass.  Each unordered pair is met once, from the
// particle whose cell comes first: the rest of its own cell and the 13 forward
// cells of the stencil, five rows of cells along x whose particles follow each
// other in memory (cells that wrap around a periodic x one by one).  A kept pair
// goes to the record of its owner (the smaller id; a pair across a periodic face to
// both), in any order: the fill orders it.  So a pair costs one FP32 test instead
// of two, no bisection of the cells by id, and ids are read for kept pairs only.
// Recording a pair waits for ids and for an atomic's value, so a lane first collects
// its kept pairs in shared memory (PAIR_HITS; the rare further ones are recorded at
// once) and records them together at the end, their loads and atomics in flight at
// the same time: a warp that recorded at every step with a kept pair took 45 us at
// 125 k particles.
// PAIR_LANES lanes share a particle, a row's candidates two at a time.  Measured with
// one, two and four lanes: 10 k box 18.8, 14.8, 14.4 us; 125 k bed 32, 28, 33 us; 2 M
// bed 332, 323, 473 us (a thread per owner over its whole stencil: 37, 48, 468 us).
// cnt starts at the mesh candidates (k_mesh_count) or zero (k_reorder).
constexpr int PAIR_BLOCK = 128;
constexpr int PAIR_HITS = 8;
constexpr int PAIR_LANES = 2;
__global__ void __launch_bounds__(PAIR_BLOCK) k_count_pairs(BPArgs a, uint32_t* __restrict__ cnt,
                                                            const uint32_t* __restrict__ old_off) {
  __shared__ uint32_t hit_q[PAIR_HITS][PAIR_BLOCK];
  __shared__ uint8_t hit_c[PAIR_HITS][PAIR_BLOCK];  // image shift (two bits an axis) and undecided bit (64)
  constexpr uint32_t HOME = 1u | 1u << 2 | 1u << 4;   // no shift, decided
  const uint32_t gl = threadIdx.x % PAIR_LANES;
  const uint64_t s = ((uint64_t)blockIdx.x * PAIR_BLOCK + threadIdx.x) / PAIR_LANES;
  if (s >= a.n) return;
  if (gl == 0) a.rev_cnt[s] = 0u;  // the fill counts the partner lists
  const int sys = a.sv.of(s);
  if (!a.sv.triggered(sys)) {  // slot kept (k_reorder): the previous list is copied
    if (gl == 0) cnt[s] = old_off[s + 1] - old_off[s];
    return;
  }
  const GridDev& g = a.sv.g[sys];
  const uint32_t coff = a.sv.coff[sys];
  const float csx = g.csf[0], csy = g.csf[1], csz = g.csf[2], cmax = g.cmaxf;
  const int d0 = g.dims[0], d1 = g.dims[1], d2n = g.dims[2];
  const float4 me = a.crel[s];
  int cx, cy, cz;
  cell_coords(g, a.cell_of[s] - coff, cx, cy, cz);
  uint4* const rec = a.srec;
  auto store = [&](uint32_t o, uint32_t at, uint32_t q, uint32_t meta, uint64_t pid) {
    const uint32_t m = at - (a.has_mesh ? a.mcnt[o] : 0u);
    if (m < a.nrec) rec[(uint64_t)o * (a.nrec + a.nmrec) + m] = make_uint4(q, meta, (uint32_t)pid, (uint32_t)(pid >> 32));
  };
  auto append = [&](uint32_t o, uint32_t q, uint32_t meta, uint64_t pid) {
    store(o, atomicAdd(&cnt[o], 1u), q, meta, pid);
  };
  // the FP64 filter from particle p to the image of q shifted by the system's lengths
  auto exact = [&](uint32_t p, uint32_t q, int sx, int sy, int sz) {
    V3 rj = mk(a.P.f[RX][q], a.P.f[RY][q], a.P.f[RZ][q]);
    if (sx) rj.x = rj.x + (double)sx * g.L[0];
    if (sy) rj.y = rj.y + (double)sy * g.L[1];
    if (sz) rj.z = rj.z + (double)sz * g.L[2];
    const double dx = rj.x - a.P.f[RX][p], dy = rj.y - a.P.f[RY][p], dz = rj.z - a.P.f[RZ][p];
    const double d2 = dx * dx + dy * dy + dz * dz;
    const double rmax = a.P.f[RAD][p] + a.P.f[RAD][q] + a.skin;
    return d2 > 0.0 && d2 < rmax * rmax && d2 < a.rcut2;
  };
  // a pair across a periodic face, or one that FP32 left undecided
  auto record_any = [&](uint32_t q, uint32_t code) {
    const int sx = (int)(code & 3u) - 1, sy = (int)((code >> 2) & 3u) - 1, sz = (int)((code >> 4) & 3u) - 1;
    const bool sure = (code & 64u) == 0;
    const uint32_t p = (uint32_t)s;
    const uint64_t idp = a.P.id[p], idq = a.P.id[q];
    if (sx | sy | sz) {  // both own it
      if (sure || exact(p, q, sx, sy, sz)) append(p, q, make_meta(DEM_ITYPE_VERTEX_VERTEX, sx, sy, sz, true), idq);
      if (sure || exact(q, p, -sx, -sy, -sz))
        append(q, p, make_meta(DEM_ITYPE_VERTEX_VERTEX, -sx, -sy, -sz, true), idp);
    } else if (idp != idq) {
      const bool mine = idp < idq;
      const uint32_t o = mine ? p : q, r = mine ? q : p;
      if (sure || exact(o, r, 0, 0, 0))
        append(o, r, make_meta(DEM_ITYPE_VERTEX_VERTEX, 0, 0, 0, false), mine ? idq : idp);
    }
  };
  if (gl == 0) {
    const int2 dr = a.sv.drange[sys];
    const PosF at = pos_f32(g, cx, cy, cz, me);
    for (int k = dr.x; k < dr.x + dr.y; k++) {
      const DriverDev& d = a.drv[k];
      if (d.kind == 2 || driver_far(d, me.w + a.skin_f, at)) continue;  // mesh drivers: mesh_phase
      if (driver_filter(d, a.P.f[RAD][s] + a.skin, mk(a.P.f[RX][s], a.P.f[RY][s], a.P.f[RZ][s])))
        append((uint32_t)s, (uint32_t)k,
               make_meta(d.kind == 0 ? DEM_ITYPE_VERTEX_SURFACE : DEM_ITYPE_VERTEX_CYLINDER, 0, 0, 0, false),
               (uint64_t)k);
    }
  }
  const float si = fmaxf(fabsf(me.x), fmaxf(fabsf(me.y), fabsf(me.z)));
  const float reach = me.w + a.skin_f;
  uint32_t nh = 0;
  auto scan = [&](uint32_t q, uint32_t q1, uint32_t u0, uint32_t u1, float oy, float oz, uint32_t shift) {
    for (q += gl; q < q1; q += PAIR_LANES) {
      const float4 cq = a.crel[q];
      const float sj = fmaxf(fabsf(cq.x), fmaxf(fabsf(cq.y), fabsf(cq.z)));
      const float ox = q < u0 ? -csx : (q < u1 ? 0.f : csx);
      const int keep = f32_decide((cq.x - me.x) + ox, (cq.y - me.y) + oy, (cq.z - me.z) + oz, si, sj, cmax,
                                  reach + cq.w);
      if (keep) {
        const uint32_t code = shift | (keep < 0 ? 64u : 0u);
        if (nh < PAIR_HITS) {
          hit_q[nh][threadIdx.x] = q;
          hit_c[nh][threadIdx.x] = (uint8_t)code;
          nh++;
        } else {
          record_any(q, code);
        }
      }
    }
  };
#pragma unroll 1
  for (int r = 0; r < 5; r++) {  // rows (dy, dz): (0, 0), (1, 0), (-1, 1), (0, 1), (1, 1)
    const int dy = r == 0 || r == 3 ? 0 : (r == 2 ? -1 : 1), dz = r < 2 ? 0 : 1;
    int y = cy + dy, z = cz + dz, sy = 0, sz = 0;
    if (y < 0 || y >= d1) {
      if (!g.periodic[1]) continue;
      sy = y < 0 ? -1 : 1;
      y -= sy * d1;
    }
    if (z >= d2n) {
      if (!g.periodic[2]) continue;
      sz = 1;
      z -= d2n;
    }
    const float oy = (float)dy * csy, oz = (float)dz * csz;
    const uint32_t rb = coff + (uint32_t)d0 * ((uint32_t)y + (uint32_t)d1 * (uint32_t)z);
    const uint32_t shift = (uint32_t)(sy + 1) << 2 | (uint32_t)(sz + 1) << 4;
    const uint32_t* const st = a.cell_start + rb + (uint32_t)cx;
    const uint32_t u0 = st[0], u1 = st[1];
    const uint32_t q0 = r == 0 ? (uint32_t)s + 1u : (cx > 0 ? st[-1] : u0);
    const uint32_t q1 = cx < d0 - 1 ? st[2] : u1;
    scan(q0, q1, u0, u1, oy, oz, shift | 1u);
    if (g.periodic[0] && (cx == d0 - 1 || (r && cx == 0))) {  // the cell that x wraps to (at least three along x)
      const bool left = cx == 0;
      const uint32_t cc = rb + (left ? (uint32_t)d0 - 1u : 0u);
      scan(a.cell_start[cc], a.cell_start[cc + 1], left ? ~0u : 0u, left ? ~0u : 0u, oy, oz, shift | (left ? 0u : 2u));
    }
  }
  const uint32_t p = (uint32_t)s;
  const uint64_t idp = a.P.id[p];
  uint64_t idq[PAIR_HITS];
  uint32_t at[PAIR_HITS];
#pragma unroll
  for (int k = 0; k < PAIR_HITS; k++)
    if (k < (int)nh && hit_c[k][threadIdx.x] == HOME) idq[k] = a.P.id[hit_q[k][threadIdx.x]];
#pragma unroll
  for (int k = 0; k < PAIR_HITS; k++)
    if (k < (int)nh && hit_c[k][threadIdx.x] == HOME && idq[k] != idp)
      at[k] = atomicAdd(&cnt[idp < idq[k] ? p : hit_q[k][threadIdx.x]], 1u);
#pragma unroll
  for (int k = 0; k < PAIR_HITS; k++) {
    if (k >= (int)nh) continue;
    const uint32_t q = hit_q[k][threadIdx.x], code = hit_c[k][threadIdx.x];
    if (code != HOME) {
      record_any(q, code);
    } else if (idq[k] != idp) {
      const bool mine = idp < idq[k];
      store(mine ? p : q, at[k], mine ? q : p, make_meta(DEM_ITYPE_VERTEX_VERTEX, 0, 0, 0, false), mine ? idq[k] : idp);
    }
  }
}

// entry y of the previous list as entry x of the new one, owned by slot s
__device__ __forceinline__ void copy_entry(const IArrays& dst, uint32_t x, const IArrays& old, uint32_t y, uint32_t s) {
  const uint32_t partner = old.partner[y], meta = old.meta[y], sub = old.sub[y];
  const uint64_t pid = old.pid[y];
  const double f0 = old.ft[0][y], f1 = old.ft[1][y], f2 = old.ft[2][y];
  const double m0 = old.mo[0][y], m1 = old.mo[1][y], m2 = old.mo[2][y], damp = old.damp[y];
  dst.owner[x] = s;
  dst.partner[x] = partner;
  dst.pid[x] = pid;
  dst.meta[x] = meta;
  dst.sub[x] = sub;
  dst.ft[0][x] = f0;
  dst.ft[1][x] = f1;
  dst.ft[2][x] = f2;
  dst.mo[0][x] = m0;
  dst.mo[1][x] = m1;
  dst.mo[2][x] = m2;
  dst.damp[x] = damp;
}

// orders owner s's segment [b, e) by InteractionPair order and carries the
// history over from the previous list
__device__ inline void finish_owner(const BPArgs& a, uint32_t s, uint32_t b, uint32_t e, IArrays dst, IArrays old,
                                    const uint32_t* __restrict__ old_off, const uint32_t* __restrict__ perm,
                                    int have_old, int reuse_damp) {
  for (uint32_t x = b + 1; x < e; x++) {
    const uint64_t pk = dst.pid[x];
    const uint32_t mk_ = dst.meta[x], qk = dst.partner[x], sk = dst.sub[x];
    const uint32_t tk = meta_type(mk_);
    uint32_t y = x;
    while (y > b && key_less(pk, tk, sk, dst.pid[y - 1], meta_type(dst.meta[y - 1]), dst.sub[y - 1])) {
      dst.pid[y] = dst.pid[y - 1];
      dst.meta[y] = dst.meta[y - 1];
      dst.partner[y] = dst.partner[y - 1];
      dst.sub[y] = dst.sub[y - 1];
      y--;
    }
    dst.pid[y] = pk;
    dst.meta[y] = mk_;
    dst.partner[y] = qk;
    dst.sub[y] = sk;
  }
  // history carry-over: binary search in the previous list of the same particle
  uint32_t ob = 0, oe = 0;
  if (have_old) {
    const uint32_t os = perm[s];
    ob = old_off[os];
    oe = old_off[os + 1];
  }
  for (uint32_t x = b; x < e; x++) {
    dst.owner[x] = s;
    double h[6] = {0, 0, 0, 0, 0, 0};
    const uint64_t pk = dst.pid[x];
    const uint32_t tk = meta_type(dst.meta[x]), sk = dst.sub[x];
    uint32_t lo = ob, hi = oe;
    while (lo < hi) {
      const uint32_t mid = (lo + hi) >> 1;
      if (key_less(old.pid[mid], meta_type(old.meta[mid]), old.sub[mid], pk, tk, sk))
        lo = mid + 1;
      else
        hi = mid;
    }
    if (lo < oe && old.pid[lo] == pk && meta_type(old.meta[lo]) == tk && old.sub[lo] == sk) {
      h[0] = old.ft[0][lo];
      h[1] = old.ft[1][lo];
      h[2] = old.ft[2][lo];
      h[3] = old.mo[0][lo];
      h[4] = old.mo[1][lo];
      h[5] = old.mo[2][lo];
      // the same pair in the previous list: the same masses and (reuse_damp) the
      // same parameters, so the same damping bits, without the FP64 square root
      // and division
      dst.damp[x] = reuse_damp ? old.damp[lo] : pair_damp(a, s, dst.partner[x], dst.meta[x]);
    } else {
      dst.damp[x] = pair_damp(a, s, dst.partner[x], dst.meta[x]);
    }
    dst.ft[0][x] = h[0];
    dst.ft[1][x] = h[1];
    dst.ft[2][x] = h[2];
    dst.mo[0][x] = h[3];
    dst.mo[1][x] = h[4];
    dst.mo[2][x] = h[5];
  }
}

// reuse_damp: the previous list's damping was computed with the current contact
// parameters (no dem_set_params / dem_set_multimat since, not a list installed by
// dem_set_interactions), so a pair found in it keeps its damping bits.
__global__ void k_fill(BPArgs a, const uint32_t* __restrict__ off, IArrays dst, IArrays old,
                       const uint32_t* __restrict__ old_off, const uint32_t* __restrict__ perm, int have_old,
                       int reuse_damp) {
  const uint64_t s = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= a.n) return;
  const uint32_t b = off[s], e = off[s + 1];
  if (e > a.cap) return;
  if (!a.sv.triggered(a.sv.of(s))) {  // slot kept, partners of the same system kept: copy
    const uint32_t ob = old_off[s];
    for (uint32_t x = b; x < e; x++) copy_entry(dst, x, old, ob + (x - b), (uint32_t)s);
    return;
  }
  uint32_t w = b + (a.has_mesh ? a.mcnt[s] : 0u);  // mesh items first (k_mesh_fill)
  for_each_candidate<false>(a, (uint32_t)s, [&](uint32_t q, uint64_t pid, uint32_t meta, uint32_t sub) {
    if (w < e) {
      dst.partner[w] = q;
      dst.pid[w] = pid;
      dst.meta[w] = meta;
      dst.sub[w] = sub;
    }
    w++;
  });
  finish_owner(a, (uint32_t)s, b, e, dst, old, old_off, perm, have_old, reuse_damp);
}

// owner slot of every entry of the new list (nothing beyond the capacity)
__global__ void k_expand_owner(BPArgs a, const uint32_t* __restrict__ off, uint32_t* __restrict__ owner) {
  const uint64_t s = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= a.n || off[a.n] > a.cap) return;
  const uint32_t b = off[s], e = off[s + 1];
  for (uint32_t x = b; x < e; x++) owner[x] = (uint32_t)s;
}

// FP32 broad phase, fill: a thread per entry of the new list.  Entry x of
// particle s takes the particle's record x, ranks its key among the particle's
// records and goes to that place, so each list is in InteractionPair order; the
// history is the entry of the same key in the particle's previous list.  The
// lanes of a warp share the records, ids and previous lists of a dozen particles
// in L1, every lane works and the writes are consecutive but for the order inside
// a list.  Bound by the latency of about six dependent loads below 100 k particles,
// above by its traffic (300 bytes an entry).  Measured: 10 k box 9 us, 2 M bed 297 us;
// a thread per particle sorting its list in global memory, a chain of loads for
// every comparison and move: 57 and 421 us; eight lanes per particle with shuffles:
// 9 and 538 us, with two of three lanes idle.
// The partner lists are counted on the way: the atomic's value is the entry's
// place in its partner's list (rev_pos).  Particles whose records
// overflowed are filled and sorted by the thread of their first entry, or with a mesh
// come ordered from k_mesh_fill.
__global__ void __launch_bounds__(128) k_fill_entries(BPArgs a, const uint32_t* __restrict__ off,
                                                      IArrays dst, IArrays old, const uint32_t* __restrict__ old_off,
                                                      const uint32_t* __restrict__ perm, int have_old,
                                                      int reuse_damp) {
  const uint64_t total = off[a.n];
  if (total > a.cap) return;  // nothing, and empty partner lists
  auto partner_list = [&](uint64_t x, uint32_t q, uint32_t meta) {
    if (meta_type(meta) == DEM_ITYPE_VERTEX_VERTEX && !meta_owner_only(meta)) a.rev_pos[x] = atomicAdd(&a.rev_cnt[q], 1u);
  };
  const uint4* const recs = a.srec;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < total; k += stride) {
    const uint32_t s = dst.owner[k];
    const uint32_t b = off[s], m = off[s + 1] - b, x = (uint32_t)k - b;
    const int sys = a.sv.of(s);
    if (!a.sv.triggered(sys)) {  // slot kept, partners of the same system kept: copy
      const uint32_t y = old_off[s] + x;
      copy_entry(dst, (uint32_t)k, old, y, s);
      partner_list(k, old.partner[y], old.meta[y]);
      continue;
    }
    const uint32_t mm = a.has_mesh ? a.mcnt[s] : 0u;
    const bool over = mm > a.nmrec || m - mm > a.nrec;
    if (over && !a.has_mesh) {
      if (x) continue;
      const uint32_t e = b + m;
      uint32_t w = b;
      for_each_candidate<true>(a, s, [&](uint32_t q, uint64_t pid, uint32_t meta, uint32_t sub) {
        if (w < e) {
          dst.partner[w] = q;
          dst.pid[w] = pid;
          dst.meta[w] = meta;
          dst.sub[w] = sub;
        }
        w++;
      });
      finish_owner(a, s, b, e, dst, old, old_off, perm, have_old, reuse_damp);
      for (uint32_t y = b; y < e; y++) partner_list(y, dst.partner[y], dst.meta[y]);
      continue;
    }
    uint32_t partner, meta, sub, type, rank = x;
    uint64_t pid;
    if (over) {  // in place and in order (k_mesh_fill)
      partner = dst.partner[k];
      pid = dst.pid[k];
      meta = dst.meta[k];
      sub = dst.sub[k];
      type = meta_type(meta);
    } else {
      const uint4* const rec = recs + (uint64_t)s * (a.nrec + a.nmrec);
      auto at = [&](uint32_t y) { return rec[y < mm ? a.nrec + y : y - mm]; };
      // a mesh item's partner id is its driver, its sub the feature (k_mesh_count)
      auto pid_of = [&](uint4 v, uint32_t y) { return y < mm ? (uint64_t)v.x : (uint64_t)v.z | (uint64_t)v.w << 32; };
      const uint4 v = at(x);
      partner = v.x;
      meta = v.y;
      type = meta_type(meta);
      pid = pid_of(v, x);
      sub = x < mm ? v.z : 0u;
      rank = 0;
      for (uint32_t y = 0; y < m; y++) {
        const uint4 u = at(y);
        rank += entry_before(a, sys, pid_of(u, y), u.y, y < mm ? u.z : 0u, u.x, pid, meta, sub, partner, y < x) ? 1u : 0u;
      }
    }
    uint32_t hit = ~0u;
    if (have_old) {
      const uint32_t os = perm[s];
      const uint32_t ob = old_off[os];
      for (uint32_t y = old_off[os + 1]; y-- > ob;)  // backwards: the first of equal keys
        if (old.pid[y] == pid && meta_type(old.meta[y]) == type && old.sub[y] == sub) hit = y;
    }
    double h[6] = {0, 0, 0, 0, 0, 0};
    double damp = 0.0;
    if (hit != ~0u) {
#pragma unroll
      for (int d = 0; d < 3; d++) {
        h[d] = old.ft[d][hit];
        h[3 + d] = old.mo[d][hit];
      }
      damp = old.damp[hit];
    }
    if (hit == ~0u || !reuse_damp) damp = pair_damp(a, s, partner, meta);
    const uint64_t w = b + rank;
    dst.partner[w] = partner;
    dst.pid[w] = pid;
    dst.meta[w] = meta;
    dst.sub[w] = sub;
#pragma unroll
    for (int d = 0; d < 3; d++) {
      dst.ft[d][w] = h[d];
      dst.mo[d][w] = h[3 + d];
    }
    dst.damp[w] = damp;
    partner_list(w, partner, meta);
  }
}

// ---- warp-per-cell broad phase (FP32 decisions)
// One warp per cell.  The particles of the cell's 27 stencil cells are staged
// in shared memory (FP32 cell-relative coordinates and radius, id, index and
// stencil slot, in stencil order), and the warp tests each owner of the cell
// against them 32 candidates at a time, compacting the kept ones with ballots.
// A neighbourhood of more than CELL_STAGE particles is walked per owner, lanes
// over owners (for_each_particle).  The decisions are those of for_each_particle
// (same FP32 expressions, same FP64 fallback), so the lists are the same.
// Drivers are tested per particle (k_pre_count / k_pre_fill), where every lane
// has an owner; in an owner's segment the mesh items come first, the particle
// candidates next and the drivers last, and k_fill_finish then orders each
// segment with the sort of k_fill.  The keys of a segment are distinct (a
// periodic dimension has at least three cells, each at least the reach, so a
// partner is in reach through one image at most), so the order of the
// segment's parts does not matter.
constexpr int CELL_WARPS = 4;
constexpr int CELL_STAGE = 128;  // staged neighbourhood particles per warp
constexpr uint8_t SLOT_OFF = 0x80u;  // stencil slot outside a non-periodic grid

struct CellStage {
  uint32_t q0[27];   // first particle of stencil slot l
  uint32_t pre[28];  // staged candidates before slot l; pre[27] = all
  uint8_t sh[27];    // (sx + 1) | (sy + 1) << 2 | (sz + 1) << 4 of slot l, or SLOT_OFF
  float x[CELL_STAGE], y[CELL_STAGE], z[CELL_STAGE], r[CELL_STAGE];
  uint64_t id[CELL_STAGE];
  uint32_t q[CELL_STAGE];
  uint8_t l[CELL_STAGE];
};

// stencil slots of cell c (local index in its system's grid) and the staging of
// their particles; returns the neighbourhood's particle count (staged when at most CELL_STAGE)
__device__ inline uint32_t stage_cell(const BPArgs& a, const GridDev& g, uint32_t coff, uint32_t c, CellStage& st,
                                      int lane) {
  uint32_t n = 0;
  if (lane < 27) {
    const int dz = lane / 9 - 1, dy = (lane / 3) % 3 - 1, dx = lane % 3 - 1;
    const int d0 = g.dims[0], d1 = g.dims[1], d2n = g.dims[2];
    const int cx = (int)(c % (uint32_t)d0);
    const int cy = (int)((c / (uint32_t)d0) % (uint32_t)d1);
    const int cz = (int)(c / ((uint32_t)d0 * (uint32_t)d1));
    int x = cx + dx, y = cy + dy, z = cz + dz, sx = 0, sy = 0, sz = 0;
    bool ok = true;
    if (x < 0) { ok &= g.periodic[0] != 0; x += d0; sx = -1; } else if (x >= d0) { ok &= g.periodic[0] != 0; x -= d0; sx = 1; }
    if (y < 0) { ok &= g.periodic[1] != 0; y += d1; sy = -1; } else if (y >= d1) { ok &= g.periodic[1] != 0; y -= d1; sy = 1; }
    if (z < 0) { ok &= g.periodic[2] != 0; z += d2n; sz = -1; } else if (z >= d2n) { ok &= g.periodic[2] != 0; z -= d2n; sz = 1; }
    uint32_t q0 = 0;
    if (ok) {
      const uint32_t cc = coff + (uint32_t)x + (uint32_t)d0 * ((uint32_t)y + (uint32_t)d1 * (uint32_t)z);
      q0 = a.cell_start[cc];
      n = a.cell_start[cc + 1] - q0;
    }
    st.q0[lane] = q0;
    st.sh[lane] = ok ? (uint8_t)((sx + 1) | ((sy + 1) << 2) | ((sz + 1) << 4)) : SLOT_OFF;
  }
  uint32_t v = n;  // inclusive scan over the slots
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += t;
  }
  if (lane < 27) st.pre[lane] = v - n;
  const uint32_t T = __shfl_sync(0xffffffffu, v, 31);
  if (lane == 0) st.pre[27] = T;
  __syncwarp();
  if (T <= (uint32_t)CELL_STAGE) {
    for (uint32_t i = (uint32_t)lane; i < T; i += 32) {
      int lo = 0, hi = 27;  // last slot l with pre[l] <= i (a slot holding i is not empty)
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (st.pre[mid] <= i)
          lo = mid;
        else
          hi = mid - 1;
      }
      const uint32_t q = st.q0[lo] + (i - st.pre[lo]);
      const float4 cq = a.crel[q];
      st.x[i] = cq.x;
      st.y[i] = cq.y;
      st.z[i] = cq.z;
      st.r[i] = cq.w;
      st.id[i] = a.P.id[q];
      st.q[i] = q;
      st.l[i] = (uint8_t)lo;
    }
  }
  __syncwarp();
  return T;
}

// staged candidate i against owner s: for_each_particle's decision
__device__ __forceinline__ bool cell_keep(const BPArgs& a, const GridDev& g, const CellStage& st, uint32_t i,
                                          uint64_t idi, float xri, float yri, float zri, float rfi, float si,
                                          float cmax, V3 ri, double radi, uint32_t& meta) {
  const int l = st.l[i];
  const int sh = st.sh[l];
  const int sx = (sh & 3) - 1, sy = ((sh >> 2) & 3) - 1, sz = ((sh >> 4) & 3) - 1;
  const bool ghost = (sx | sy | sz) != 0;
  if (!ghost && idi >= st.id[i]) return false;  // owner rule first
  const float oxf = (float)(l % 3 - 1) * (float)g.csz[0], oyf = (float)((l / 3) % 3 - 1) * (float)g.csz[1],
              ozf = (float)(l / 9 - 1) * (float)g.csz[2];
  const float xj = st.x[i], yj = st.y[i], zj = st.z[i];
  const float sj = fmaxf(fabsf(xj), fmaxf(fabsf(yj), fabsf(zj)));
  int keep = f32_decide((xj - xri) + oxf, (yj - yri) + oyf, (zj - zri) + ozf, si, sj, cmax, rfi + st.r[i] + a.skin_f);
  if (keep < 0) {
    const uint32_t q = st.q[i];
    V3 rj = mk(a.P.f[RX][q], a.P.f[RY][q], a.P.f[RZ][q]);
    if (sx) rj.x = rj.x + (double)sx * g.L[0];
    if (sy) rj.y = rj.y + (double)sy * g.L[1];
    if (sz) rj.z = rj.z + (double)sz * g.L[2];
    const double ddx = rj.x - ri.x, ddy = rj.y - ri.y, ddz = rj.z - ri.z;
    const double d2 = ddx * ddx + ddy * ddy + ddz * ddz;
    const double rmax = radi + a.P.f[RAD][q] + a.skin;
    keep = (d2 > 0.0 && d2 < rmax * rmax && d2 < a.rcut2) ? 1 : 0;
  }
  meta = make_meta(DEM_ITYPE_VERTEX_VERTEX, sx, sy, sz, ghost);
  return keep != 0;
}

// the particle candidates of every owner of cell C: counted (Fill = false: added
// to cnt) or written at b + mesh items (Fill = true)
template <bool Fill>
__device__ inline void cell_particles(const BPArgs& a, uint32_t C, uint32_t o0, uint32_t o1, int sys, CellStage& st,
                                      int lane, uint32_t* cnt, const uint32_t* off, IArrays dst) {
  const GridDev& g = a.sv.g[sys];
  const uint32_t coff = a.sv.coff[sys];
  const uint32_t T = stage_cell(a, g, coff, C - coff, st, lane);
  const uint32_t lt = (1u << lane) - 1u;
  if (T > (uint32_t)CELL_STAGE) {  // dense neighbourhood: lanes over owners
    for (uint32_t s = o0 + (uint32_t)lane; s < o1; s += 32) {
      if (Fill) {
        const uint32_t b = off[s], e = off[s + 1];
        if (e > a.cap) continue;
        uint32_t w = b + (a.has_mesh ? a.mcnt[s] : 0u);
        for_each_particle<true>(a, s, sys, [&](uint32_t q, uint64_t pid, uint32_t meta, uint32_t sub) {
          if (w < e) {
            dst.partner[w] = q;
            dst.pid[w] = pid;
            dst.meta[w] = meta;
            dst.sub[w] = sub;
          }
          w++;
        });
      } else {
        uint32_t m = 0;
        for_each_particle<true>(a, s, sys, [&](uint32_t, uint64_t, uint32_t, uint32_t) { m++; });
        cnt[s] += m;
      }
    }
    __syncwarp();
    return;
  }
  const float cmax = fmaxf((float)g.csz[0], fmaxf((float)g.csz[1], (float)g.csz[2]));
  for (uint32_t s = o0; s < o1; s++) {
    uint32_t w = 0, e = 0;
    if (Fill) {
      e = off[s + 1];
      if (e > a.cap) continue;
      w = off[s] + (a.has_mesh ? a.mcnt[s] : 0u);
    }
    const float4 me = a.crel[s];
    const float xri = me.x, yri = me.y, zri = me.z, rfi = me.w;
    const float si = fmaxf(fabsf(xri), fmaxf(fabsf(yri), fabsf(zri)));
    const uint64_t idi = a.P.id[s];
    const V3 ri = mk(a.P.f[RX][s], a.P.f[RY][s], a.P.f[RZ][s]);
    const double radi = a.P.f[RAD][s];
    uint32_t m = 0;
    for (uint32_t c0 = 0; c0 < T; c0 += 32) {
      const uint32_t i = c0 + (uint32_t)lane;
      uint32_t meta = 0;
      const bool keep = i < T && cell_keep(a, g, st, i, idi, xri, yri, zri, rfi, si, cmax, ri, radi, meta);
      const unsigned bm = __ballot_sync(0xffffffffu, keep);
      if (Fill && keep) {
        const uint32_t x = w + m + __popc(bm & lt);
        if (x < e) {
          dst.partner[x] = st.q[i];
          dst.pid[x] = st.id[i];
          dst.meta[x] = meta;
          dst.sub[x] = 0u;
        }
      }
      m += __popc(bm);
    }
    if (!Fill && lane == 0) cnt[s] += m;
  }
}

// drivers of each particle (after the mesh items, counted in k_mesh_count), or
// the previous count of a particle whose system kept its list
__global__ void k_pre_count(BPArgs a, uint32_t* __restrict__ cnt, const uint32_t* __restrict__ old_off) {
  const uint64_t s = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= a.n) return;
  const int sys = a.sv.of(s);
  if (!a.sv.triggered(sys)) {
    cnt[s] = old_off[s + 1] - old_off[s];
    return;
  }
  uint32_t m = a.has_mesh ? a.mcnt[s] : 0u;
  for_each_driver(a, (uint32_t)s, sys, [&](uint32_t, uint64_t, uint32_t, uint32_t) { m++; });
  cnt[s] = m;
}

// drivers at the end of each particle's segment; a particle whose system kept
// its list copies it
__global__ void k_pre_fill(BPArgs a, const uint32_t* __restrict__ off, IArrays dst, IArrays old,
                           const uint32_t* __restrict__ old_off) {
  const uint64_t s = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= a.n) return;
  const uint32_t b = off[s], e = off[s + 1];
  if (e > a.cap) return;
  const int sys = a.sv.of(s);
  if (!a.sv.triggered(sys)) {
    const uint32_t ob = old_off[s];
    for (uint32_t x = b; x < e; x++) copy_entry(dst, x, old, ob + (x - b), (uint32_t)s);
    return;
  }
  uint32_t nd = 0;
  for_each_driver(a, (uint32_t)s, sys, [&](uint32_t, uint64_t, uint32_t, uint32_t) { nd++; });
  uint32_t w = e - nd;
  for_each_driver(a, (uint32_t)s, sys, [&](uint32_t k, uint64_t pid, uint32_t meta, uint32_t sub) {
    dst.partner[w] = k;
    dst.pid[w] = pid;
    dst.meta[w] = meta;
    dst.sub[w] = sub;
    w++;
  });
}

__global__ void __launch_bounds__(CELL_WARPS * 32) k_cell_count(BPArgs a, uint32_t* __restrict__ cnt,
                                                                uint64_t ncell) {
  __shared__ CellStage stage[CELL_WARPS];
  const int lane = threadIdx.x & 31;
  CellStage& st = stage[threadIdx.x >> 5];
  const uint64_t nw = (uint64_t)gridDim.x * CELL_WARPS;
  for (uint64_t C = (uint64_t)blockIdx.x * CELL_WARPS + (threadIdx.x >> 5); C < ncell; C += nw) {
    const uint32_t o0 = a.cell_start[C], o1 = a.cell_start[C + 1];
    if (o0 == o1) continue;
    const int sys = a.sv.of(o0);
    if (!a.sv.triggered(sys)) continue;
    cell_particles<false>(a, (uint32_t)C, o0, o1, sys, st, lane, cnt, nullptr, IArrays{});
  }
}

__global__ void __launch_bounds__(CELL_WARPS * 32) k_cell_fill(BPArgs a, const uint32_t* __restrict__ off,
                                                               IArrays dst, uint64_t ncell) {
  __shared__ CellStage stage[CELL_WARPS];
  const int lane = threadIdx.x & 31;
  CellStage& st = stage[threadIdx.x >> 5];
  const uint64_t nw = (uint64_t)gridDim.x * CELL_WARPS;
  for (uint64_t C = (uint64_t)blockIdx.x * CELL_WARPS + (threadIdx.x >> 5); C < ncell; C += nw) {
    const uint32_t o0 = a.cell_start[C], o1 = a.cell_start[C + 1];
    if (o0 == o1) continue;
    const int sys = a.sv.of(o0);
    if (!a.sv.triggered(sys)) continue;
    cell_particles<true>(a, (uint32_t)C, o0, o1, sys, st, lane, nullptr, off, dst);
  }
}

// after k_mesh_fill, k_pre_fill and k_cell_fill: each owner's segment ordered and
// its history carried over, one thread per owner
__global__ void k_fill_finish(BPArgs a, const uint32_t* __restrict__ off, IArrays dst, IArrays old,
                              const uint32_t* __restrict__ old_off, const uint32_t* __restrict__ perm, int have_old,
                              int reuse_damp) {
  const uint64_t s = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= a.n) return;
  const uint32_t b = off[s], e = off[s + 1];
  if (e > a.cap || !a.sv.triggered(a.sv.of(s))) return;
  finish_owner(a, (uint32_t)s, b, e, dst, old, old_off, perm, have_old, reuse_damp);
}

// per-pair damping of a kept list after the contact parameters changed
__global__ void k_pair_damp(BPArgs a, IArrays I, uint64_t ni) {
  for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < ni; k += (uint64_t)gridDim.x * blockDim.x)
    I.damp[k] = pair_damp(a, I.owner[k], I.partner[k], I.meta[k]);
}

// partner-side lists: interactions whose partner is a real particle that receives -f
// ni_dev != nullptr: the interaction count is read on the device (graph step)
__global__ void k_rev_count(IArrays I, uint64_t ni, const unsigned long long* ni_dev, uint32_t* __restrict__ cnt) {
  const uint64_t nn = ni_dev ? *ni_dev : ni;
  for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < nn; k += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t m = I.meta[k];
    if (meta_type(m) <= DEM_ITYPE_EDGE_EDGE && !meta_owner_only(m)) atomicAdd(&cnt[I.partner[k]], 1u);
  }
}
__global__ void k_rev_fill(IArrays I, uint64_t ni, const unsigned long long* ni_dev, const uint32_t* __restrict__ off,
                           uint32_t* __restrict__ cursor, const uint64_t* __restrict__ id, uint32_t* __restrict__ idx,
                           uint64_t* __restrict__ oid) {
  const uint64_t nn = ni_dev ? *ni_dev : ni;
  for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < nn; k += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t m = I.meta[k];
    if (meta_type(m) <= DEM_ITYPE_EDGE_EDGE && !meta_owner_only(m)) {
      const uint32_t j = I.partner[k];
      const uint32_t w = off[j] + atomicAdd(&cursor[j], 1u);
      idx[w] = (uint32_t)k;
      oid[w] = id[I.owner[k]];
    }
  }
}
// the entries at their counted places (k_fill_entries), and their owners' ids
__global__ void k_rev_place(IArrays I, uint64_t ni, const unsigned long long* ni_dev, const uint32_t* __restrict__ off,
                            const uint32_t* __restrict__ pos, const uint64_t* __restrict__ id,
                            uint32_t* __restrict__ idx, uint64_t* __restrict__ oid) {
  const uint64_t nn = ni_dev ? *ni_dev : ni;
  for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < nn; k += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t m = I.meta[k];
    if (meta_type(m) <= DEM_ITYPE_EDGE_EDGE && !meta_owner_only(m)) {
      const uint32_t w = off[I.partner[k]] + pos[k];
      idx[w] = (uint32_t)k;
      oid[w] = id[I.owner[k]];
    }
  }
}
// order of the partner-side contributions: InteractionPair order = (owner id,
// index).  A thread per entry: its rank is the number of entries of its partner's
// list with a smaller key (keys are distinct: the index is); the lanes of a warp
// share their lists in L1.  No lane idles whatever the lists' lengths are (about
// three for spheres, 34 for the fragmentation bed's cubes).
__global__ void __launch_bounds__(256) k_rev_rank(uint64_t n, const uint32_t* __restrict__ off,
                                                  const uint32_t* __restrict__ partner,
                                                  const uint32_t* __restrict__ unsorted,
                                                  const uint64_t* __restrict__ oid, uint32_t* __restrict__ idx) {
  const uint64_t total = off[n];
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t w = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; w < total; w += stride) {
    const uint32_t k = unsorted[w];
    const uint64_t o = oid[w];
    const uint32_t j = partner[k];
    const uint32_t b = off[j], e = off[j + 1];
    uint32_t rank = 0;
    for (uint32_t y = b; y < e; y++) {
      const uint64_t oy = oid[y];
      if (oy < o || (oy == o && unsorted[y] < k)) rank++;
    }
    idx[b + rank] = k;
  }
}

BPArgs make_args(dem_ctx* c) {
  BPArgs a;
  a.P = c->P[c->pcur];
  a.n = c->n;
  a.sv = c->sysview();
  a.cell_start = c->cell_start;
  a.cell_of = c->cell_of;
  a.drv = c->drv_dev;
  a.ndrv = c->ndrv;
  a.mesh = c->mesh_dev;
  a.has_mesh = c->meshes.empty() ? 0 : 1;
  a.mcnt = c->mesh_cnt;
  a.skin = c->prm.rcut_inc;
  const double nd = 2 * c->rad_max + c->prm.rcut_inc;
  a.rcut2 = nd * nd;
  a.crel = c->crel;
  a.skin_f = (float)c->prm.rcut_inc;
  a.cap = c->capturing ? c->gcap : ~0ull;
  a.srec = c->srec;
  a.nrec = c->srec_n;
  a.nmrec = c->srec_m;
  a.rev_cnt = c->rev_cnt;
  a.rev_pos = c->L2;
  a.cp = c->prm.config;
  a.cpd = c->prm.config_driver;
  a.pt = c->ptable();
  return a;
}
}  // namespace

// recomputes the per-pair damping of the current sphere list (after dem_set_params)
int refresh_pair_damp(dem_ctx* c) {
  if (!c->damp_stale) return DEM_OK;
  if (!c->have_list) return DEM_OK;  // still stale: the next build computes every pair's damping
  c->damp_stale = false;
  if (c->poly || !c->ni) return DEM_OK;
  k_pair_damp<<<c->num_sms * 4, 256, 0, c->stream>>>(make_args(c), c->I[c->icur], c->ni);
  DEM_CUDA_TRY(c, cudaGetLastError());
  return DEM_OK;
}

// the warp-per-cell kernels: a grid-stride loop over the cells
static unsigned cell_grid(const dem_ctx* c) {
  const uint64_t want = (c->ncell + CELL_WARPS - 1) / CELL_WARPS;
  return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(want, (uint64_t)c->num_sms * 16));
}

// Records of a particle in the FP32 build: 16 hold the candidates of nearly every sphere
// (more are enumerated again, and sorted one by one), and a sphere where triangles meet
// has tens of mesh candidates.  They take 256 bytes a particle and 768 with a mesh, which
// a run whose lists fill the memory may not have: a sixteenth of the free memory at most,
// else four records, 64 bytes.
constexpr uint32_t REC_PLANS[3][2] = {{16, 48}, {16, 0}, {4, 0}};
int record_plan(uint64_t particles, bool mesh, uint64_t budget) {
  int k = mesh ? 0 : 1;
  while (k < 2 && particles * (REC_PLANS[k][0] + REC_PLANS[k][1]) * sizeof(uint4) > budget) k++;
  return k;
}

void free_records_f32(dem_ctx* c) {
  cudaFree(c->srec);
  c->srec = nullptr;
  c->srec_n = c->srec_m = 0;
  c->srec_cap = 0;
}

// the records of the build that uses them, for the particles' capacity
int ensure_records_f32(dem_ctx* c) {
  if (c->poly || !c->prm.fp32_broad_phase || c->cell_broad_phase || !c->n) return DEM_OK;
  const bool mesh = !c->meshes.empty();
  if (c->srec && c->srec_cap == c->pcap && c->srec_mesh == mesh) return DEM_OK;
  if (c->capturing) return c->fail(DEM_ERR_STATE, "list records missing inside a graph capture");
  DEM_CUDA_TRY(c, cudaStreamSynchronize(c->stream));
  free_records_f32(c);
  c->gen++;  // captured kernels hold the old buffer
  uint64_t budget = c->srec_budget;
  if (!budget) {
    size_t left = 0, total = 0;
    DEM_CUDA_TRY(c, cudaMemGetInfo(&left, &total));
    budget = left / 16;
  }
  for (int k = record_plan(c->pcap, mesh, budget); k < 3; k++) {
    const uint32_t n = REC_PLANS[k][0], m = REC_PLANS[k][1];
    if (cudaMalloc(&c->srec, c->pcap * (n + m) * sizeof(uint4)) == cudaSuccess) {
      c->srec_n = n;
      c->srec_m = m;
      c->srec_cap = c->pcap;
      c->srec_mesh = mesh;
      return DEM_OK;
    }
    cudaGetLastError();
    c->srec = nullptr;
  }
  return c->fail(DEM_ERR_OOM, "list records: device allocation failed");
}

int launch_count_sphere(dem_ctx* c) {
  const bool mesh = !c->meshes.empty();
  ProfScope ps(c, K_BROAD_COUNT, c->n ? (mesh ? 2 : 1) : 0);
  if (c->n && mesh) {
    if (!c->mesh_cnt) return c->fail(DEM_ERR_STATE, "mesh count buffer missing");
    // with records (k_count_pairs' path) the fill takes the mesh items from them
    const auto kern = !c->prm.fp32_broad_phase ? k_mesh_count<false, false>
                      : c->cell_broad_phase    ? k_mesh_count<true, false>
                                               : k_mesh_count<true, true>;
    kern<<<grid_for(c->n, MESH_SPHERES), MESH_BLOCK, 0, c->stream>>>(make_args(c), c->mesh_cnt,
                                                                                             c->pcnt);
  }
  if (c->n) {
    if (c->prm.fp32_broad_phase && c->cell_broad_phase) {
      const BPArgs a = make_args(c);
      k_pre_count<<<grid_for(c->n, 128), 128, 0, c->stream>>>(a, c->pcnt, c->own_off[c->icur]);
      k_cell_count<<<cell_grid(c), CELL_WARPS * 32, 0, c->stream>>>(a, c->pcnt, c->ncell);
    } else if (c->prm.fp32_broad_phase) {
      k_count_pairs<<<grid_for(c->n * PAIR_LANES, PAIR_BLOCK), PAIR_BLOCK, 0, c->stream>>>(make_args(c), c->pcnt,
                                                                                           c->own_off[c->icur]);
    } else {
      k_count<<<grid_for(c->n, 128), 128, 0, c->stream>>>(make_args(c), c->pcnt, c->own_off[c->icur]);
    }
  }
  DEM_CUDA_TRY(c, cudaGetLastError());
  return DEM_OK;
}

int launch_fill_sphere(dem_ctx* c, uint32_t* new_off, uint64_t total) {
  const int nw = 1 - c->icur;
  const bool mesh = !c->meshes.empty();
  const bool cells = c->prm.fp32_broad_phase && c->cell_broad_phase;
  ProfScope ps(c, K_BROAD_FILL, c->n ? (mesh ? 1 : 0) + (cells ? 3 : c->prm.fp32_broad_phase ? 2 : 1) : 0);
  if (c->n && mesh) {
    const auto kern = !c->prm.fp32_broad_phase ? k_mesh_fill<false, false>
                      : c->cell_broad_phase    ? k_mesh_fill<true, false>
                                               : k_mesh_fill<true, true>;
    kern<<<grid_for(c->n, MESH_SPHERES), MESH_BLOCK, 0, c->stream>>>(make_args(c), new_off,
                                                                                             c->I[nw]);
  }
  if (c->n) {
    const int have_old = c->hist_valid ? 1 : 0, reuse = (c->hist_valid && !c->damp_stale) ? 1 : 0;
    if (c->prm.fp32_broad_phase && c->cell_broad_phase) {
      const BPArgs a = make_args(c);
      k_pre_fill<<<grid_for(c->n, 128), 128, 0, c->stream>>>(a, new_off, c->I[nw], c->I[c->icur],
                                                             c->own_off[c->icur]);
      k_cell_fill<<<cell_grid(c), CELL_WARPS * 32, 0, c->stream>>>(a, new_off, c->I[nw], c->ncell);
      k_fill_finish<<<grid_for(c->n, 128), 128, 0, c->stream>>>(a, new_off, c->I[nw], c->I[c->icur],
                                                                c->own_off[c->icur], c->perm, have_old, reuse);
    } else if (c->prm.fp32_broad_phase) {
      const BPArgs a = make_args(c);
      k_expand_owner<<<grid_for(c->n, 128), 128, 0, c->stream>>>(a, new_off, c->I[nw].owner);
      // the total is on the device in a graph: a grid of about two entries a particle strides over it
      const uint64_t want = c->capturing ? 2 * c->n : total;
      if (want)
        k_fill_entries<<<(unsigned)std::min<uint64_t>(grid_for(want, 128), (uint64_t)c->num_sms * 64), 128, 0,
                         c->stream>>>(a, new_off, c->I[nw], c->I[c->icur], c->own_off[c->icur], c->perm,
                                      have_old, reuse);
    } else {
      k_fill<<<grid_for(c->n, 128), 128, 0, c->stream>>>(make_args(c), new_off, c->I[nw], c->I[c->icur],
                                                         c->own_off[c->icur], c->perm, have_old, reuse);
    }
  }
  DEM_CUDA_TRY(c, cudaGetLastError());
  return DEM_OK;
}

// counted: the fill counted the partner lists (rev_cnt, L2: k_fill_entries)
int launch_reverse_lists(dem_ctx* c, bool counted) {
  const uint64_t n = c->n, ni = c->ni;
  cudaStream_t st = c->stream;
  const IArrays& I = c->I[c->icur];
  // in a graph capture the count is on the device: persistent grids over d_ni
  const unsigned long long* nd = c->capturing ? c->d_ni : nullptr;
  const bool go = c->capturing || ni;
  const unsigned gi = c->capturing ? (unsigned)c->num_sms * 8u : grid_for(ni, 256);
  // the contact work list L1 (capacity rcap, like rev_idx) holds the unsorted
  // lists: the step's contact phase, after the rebuild, refills it
  uint32_t* unsorted = c->L1;
  if (!counted) {
    ProfScope ps(c, K_REVERSE, go ? 1 : 0);
    DEM_CUDA_TRY(c, cudaMemsetAsync(c->rev_cnt, 0, (n + 1) * 4, st));
    if (go) k_rev_count<<<gi, 256, 0, st>>>(I, ni, nd, c->rev_cnt);
  }
  int rc = scan_exclusive_u32(c, c->rev_cnt, c->rev_off, n);
  if (rc) return rc;
  ProfScope ps(c, K_REVERSE, go ? 2 : 0);
  const uint64_t* id = c->P[c->pcur].id;
  uint64_t* oid = reinterpret_cast<uint64_t*>(c->Dscr[0]);  // a scratch of the contact pass (rcap), free here
  if (!counted) DEM_CUDA_TRY(c, cudaMemsetAsync(c->rev_cnt, 0, (n + 1) * 4, st));
  if (go) {
    if (counted)
      k_rev_place<<<gi, 256, 0, st>>>(I, ni, nd, c->rev_off, c->L2, id, unsorted, oid);
    else
      k_rev_fill<<<gi, 256, 0, st>>>(I, ni, nd, c->rev_off, c->rev_cnt, id, unsorted, oid);
    k_rev_rank<<<gi, 256, 0, st>>>(n, c->rev_off, I.partner, unsorted, oid, c->rev_idx);
  }
  DEM_CUDA_TRY(c, cudaGetLastError());
  return DEM_OK;
}

// whether launch_fill_sphere counts the partner lists itself
bool fill_counts_partners(const dem_ctx* c) { return c->prm.fp32_broad_phase && !c->cell_broad_phase; }
}  // namespace dem

extern "C" int dem_selftest_record_plan(uint64_t particles, int mesh, uint64_t budget, uint32_t* records) {
  if (!records) return DEM_ERR_INVALID_ARG;
  const int k = dem::record_plan(particles, mesh != 0, budget);
  records[0] = dem::REC_PLANS[k][0];
  records[1] = dem::REC_PLANS[k][1];
  return DEM_OK;
}

extern "C" int dem_selftest_records(dem_ctx* c, uint64_t budget, uint32_t* records) {
  if (!c || !records) return DEM_ERR_INVALID_ARG;
  records[0] = c->srec_n;
  records[1] = c->srec_m;
  if (budget) {
    DEM_CUDA_TRY(c, cudaStreamSynchronize(c->stream));
    c->srec_budget = budget;
    dem::free_records_f32(c);
    c->gen++;
  }
  return DEM_OK;
}
