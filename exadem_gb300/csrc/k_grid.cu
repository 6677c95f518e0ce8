// k_grid.cu -- cell binning and particle reorder at a neighbour rebuild.
//
// Stands in for exaNBody's move_particles / migrate_cell_particles / grid
// (periodic wrap into the domain, particles stored cell by cell).  Steps:
//   k_bin:       periodic wrap, cell index, cell histogram (the atomic gives the
//                particle's place in its cell)
//   scan:        cell starts
//   k_scatter:   the cells' lists, in the atomics' order inside a cell
//   k_reorder:   the order inside a cell by particle id, and every field into the
//                other particle buffer
// All of it is integer / copy work: HBM-bound, one read and one write per field.
// Measured (launches of a rebuild here, with the scan): 10 k particles 9 launches
// 42 us -> 5 launches 17 us, 2 M 460 -> 260 us (three launches zeroed or sorted, the
// binning divided in FP64).
// Batched contexts: each system bins into its own block of the cell index
// space, so the sort keeps every particle inside its system's slot range.
#include "dem_ctx.cuh"
#include "emu64.cuh"

namespace dem {
namespace {

// Cell of coordinate x - lo on one axis: floor((x - lo) / csz), clamped.  The FP32
// quotient t carries a relative error below 2^-22 (three roundings); where its
// fraction is further than twice that from an integer, floor(t) is the floor of
// the FP64 quotient and the FP64 division (8 FP64 instructions, three a particle)
// is not run.
__device__ __forceinline__ int cell_of_axis(const GridDev& g, int d, double rel) {
  const float t = (float)rel * g.icsz[d];
  const float m = fabsf(t) * 5e-7f + 1e-6f;
  const float k = floorf(t);
  const float fr = t - k;
  if (fr > m && fr < 1.f - m) {
    if (k < 0.f) return 0;
    return k >= (float)g.dims[d] ? g.dims[d] - 1 : (int)k;
  }
  const double q = floor(rel / g.csz[d]);
  long kk = (q < 0.0) ? 0 : (q >= (double)g.dims[d] ? g.dims[d] - 1 : (long)q);
  if (kk < 0) kk = 0;
  if (kk >= g.dims[d]) kk = g.dims[d] - 1;
  return (int)kk;
}

// cell_pos: the particle's place among those of its cell, in the atomics' order
__global__ void k_bin(PArrays P, uint64_t n, SysView sv, uint32_t* __restrict__ cell_tmp,
                      uint32_t* __restrict__ cell_cnt, uint32_t* __restrict__ cell_pos) {
  const uint64_t s = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n) return;
  const int sys = sv.of(s);
  if (!sv.triggered(sys)) return;  // kept in place (k_sys_block counts it)
  const GridDev& g = sv.g[sys];
  int k[3];
#pragma unroll
  for (int d = 0; d < 3; d++) {
    double x = P.f[RX + d][s];
    if (g.periodic[d]) {
      const double lo = g.lo[d], hi = g.hi[d], Ld = g.L[d];
      if (emu_lt(x, lo)) {
        x = x + Ld;
        if (x >= hi) x = lo;
        P.f[RX + d][s] = x;
      } else if (emu_le(hi, x)) {
        x = x - Ld;
        if (x < lo) x = lo;
        P.f[RX + d][s] = x;
      }
    }
    k[d] = cell_of_axis(g, d, x - g.lo[d]);
  }
  const uint32_t c =
      sv.coff[sys] + (uint32_t)k[0] + (uint32_t)g.dims[0] * ((uint32_t)k[1] + (uint32_t)g.dims[1] * (uint32_t)k[2]);
  cell_tmp[s] = c;
  cell_pos[s] = atomicAdd(&cell_cnt[c], 1u);
}

__global__ void k_scatter(const uint32_t* __restrict__ cell_tmp, const uint32_t* __restrict__ cell_pos, uint64_t n,
                          const uint32_t* __restrict__ cell_start, uint32_t* __restrict__ unsorted, SysView sv) {
  const uint64_t s = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n) return;
  if (!sv.triggered(sv.of(s))) return;  // slot kept (k_reorder)
  unsorted[cell_start[cell_tmp[s]] + cell_pos[s]] = (uint32_t)s;
}

// A system rebuilt without its own trigger is one block of its particle count
// in its first cell, so that every system's cells start at its first slot.
__global__ void k_sys_block(SysView sv, uint32_t* __restrict__ cell_cnt) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= sv.nsys || sv.triggered(k)) return;
  atomicAdd(&cell_cnt[sv.coff[k]], (uint32_t)(sv.pfirst[k + 1] - sv.pfirst[k]));
}

// One thread per particle of the cells' lists: its rank among its cell's by
// (id, slot) is its place there, so the layout does not depend on the atomics'
// order (cells hold one or two particles at the default cell size).  Its fields
// move through registers a chunk at a time: the compiler may not move a load
// above a store to another array of the same type, and 33 dependent load-store
// pairs took 21 us whatever n was, where the moves themselves take 2 to 5 us at
// 100 k particles.  The candidate counts of the new slots start at zero here.
__global__ void k_reorder(PArrays src, PArrays dst, uint64_t n, const uint32_t* __restrict__ unsorted,
                          uint32_t* __restrict__ perm, const uint32_t* __restrict__ cell_tmp,
                          const uint32_t* __restrict__ cell_start, uint32_t* __restrict__ cell_of, SysView sv,
                          float4* __restrict__ crel, uint32_t* __restrict__ cnt) {
  const uint64_t w = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= n) return;
  cnt[w] = 0u;
  const int sys = sv.of(w);  // the slot stays in the particle's system range
  if (!sv.triggered(sys)) {  // rebuilt without its own trigger: kept in its slot (its list is copied unchanged)
    perm[w] = (uint32_t)w;
    return;
  }
  const uint32_t o = unsorted[w];
  const uint32_t ct = cell_tmp[o];
  const uint32_t b = cell_start[ct], e = cell_start[ct + 1];
  const uint64_t ido = src.id[o];
  uint32_t t = b;
  if (e - b > 1u)
    for (uint32_t x = b; x < e; x++) {
      const uint32_t p = unsorted[x];
      const uint64_t idp = src.id[p];
      t += (idp < ido || (idp == ido && p < o)) ? 1u : 0u;
    }
  perm[t] = o;
  constexpr int CH = 16;
  static_assert(BX % CH == 0, "whole chunks");
#pragma unroll
  for (int k0 = 0; k0 < BX; k0 += CH) {
    double v[CH];
#pragma unroll
    for (int k = 0; k < CH; k++) v[k] = src.f[k0 + k][o];
#pragma unroll
    for (int k = 0; k < CH; k++) dst.f[k0 + k][t] = v[k];
  }
  // FP32 coordinates relative to the origin of the particle's cell, for the FP32 broad phase
  const GridDev& g = sv.g[sys];
  const uint32_t c = ct - sv.coff[sys];
  int kx, ky, kz;
  cell_coords(g, c, kx, ky, kz);
  const double x = src.f[RX][o], y = src.f[RY][o], z = src.f[RZ][o], r = src.f[RAD][o];
  const uint32_t type = src.type[o], group = src.group[o];
  crel[t] = make_float4((float)(x - (g.lo[0] + (double)kx * g.csz[0])), (float)(y - (g.lo[1] + (double)ky * g.csz[1])),
                        (float)(z - (g.lo[2] + (double)kz * g.csz[2])), (float)r);
  // backup_r: positions at this rebuild, for the displacement trigger
  dst.f[BX][t] = x;
  dst.f[BY][t] = y;
  dst.f[BZ][t] = z;
  dst.id[t] = ido;
  dst.type[t] = type;
  dst.group[t] = group;
  cell_of[t] = ct;
}

// several systems: the reordered slots of the triggered systems back into the
// current buffer (the others were not touched, so the buffers do not swap)
__global__ void k_copy_back(PArrays from, PArrays to, uint64_t n, SysView sv) {
  const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n || !sv.triggered(sv.of(t))) return;
  const uint64_t id = from.id[t];
  const uint32_t type = from.type[t], group = from.group[t];
  constexpr int CH = 18;
#pragma unroll
  for (int k0 = 0; k0 < NPF; k0 += CH) {
    double v[CH];
#pragma unroll
    for (int k = 0; k < CH; k++)
      if (k0 + k < NPF) v[k] = from.f[k0 + k][t];
#pragma unroll
    for (int k = 0; k < CH; k++)
      if (k0 + k < NPF) to.f[k0 + k][t] = v[k];
  }
  to.id[t] = id;
  to.type[t] = type;
  to.group[t] = group;
}
}  // namespace

// Sets up the grid, wraps, bins, scans and scatters; leaves in rev_cnt the slots cell by cell, in no order inside a cell.
int launch_bin_particles(dem_ctx* c) {
  const uint64_t n = c->n;
  const uint64_t nc = c->ncell;
  cudaStream_t st = c->stream;
  int rc;
  DEM_CUDA_TRY(c, cudaMemsetAsync(c->cell_cnt, 0, (nc + 1) * 4, st));
  {
    ProfScope ps(c, K_BIN, (n ? 1 : 0) + (c->nsys > 1 ? 1 : 0));
    if (n) k_bin<<<grid_for(n, 128), 128, 0, st>>>(c->P[c->pcur], n, c->sysview(), c->cell_tmp, c->cell_cnt, c->pcnt);
    if (c->nsys > 1) k_sys_block<<<(c->nsys + 255) / 256, 256, 0, st>>>(c->sysview(), c->cell_cnt);
  }
  rc = scan_exclusive_u32(c, c->cell_cnt, c->cell_start, nc);
  if (rc) return rc;
  ProfScope ps(c, K_BIN, n ? 1 : 0);
  if (n)
    k_scatter<<<grid_for(n, 128), 128, 0, st>>>(c->cell_tmp, c->pcnt, n, c->cell_start, c->rev_cnt, c->sysview());
  DEM_CUDA_TRY(c, cudaGetLastError());
  return DEM_OK;
}

// Gathers all particle fields into the other buffer in cell order and swaps;
// perm = new slot -> old slot.  Several systems: only the triggered systems'
// slots are gathered, then copied back, and the buffers do not swap.
int launch_reorder_particles(dem_ctx* c) {
  const uint64_t n = c->n;
  const bool part = c->nsys > 1;
  ProfScope ps(c, K_REORDER, n ? (part ? 2 : 1) : 0);
  if (n) {
    k_reorder<<<grid_for(n, 128), 128, 0, c->stream>>>(c->P[c->pcur], c->P[1 - c->pcur], n, c->rev_cnt, c->perm,
                                                        c->cell_tmp, c->cell_start, c->cell_of, c->sysview(), c->crel,
                                                        c->pcnt);
    if (part) k_copy_back<<<grid_for(n, 128), 128, 0, c->stream>>>(c->P[1 - c->pcur], c->P[c->pcur], n, c->sysview());
  }
  DEM_CUDA_TRY(c, cudaGetLastError());
  if (!part) c->pcur = 1 - c->pcur;
  return DEM_OK;
}
}  // namespace dem
