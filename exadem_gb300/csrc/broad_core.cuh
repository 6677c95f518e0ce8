// broad_core.cuh -- FP32 decisions shared by the sphere and polyhedron list builds.
#pragma once
#include "dem_ctx.cuh"

namespace dem {

// A particle's coordinates in FP32, from its cell and its place in it, and the sum of the
// magnitudes that the three are made of.
struct PosF {
  float x, y, z, m;
};
__device__ __forceinline__ PosF pos_f32(const GridDev& g, int cx, int cy, int cz, float4 rel) {
  const float ox = (float)cx * g.csf[0], oy = (float)cy * g.csf[1], oz = (float)cz * g.csf[2];
  PosF p;
  p.x = g.lof[0] + ox + rel.x;
  p.y = g.lof[1] + oy + rel.y;
  p.z = g.lof[2] + oz + rel.z;
  p.m = g.lo1 + (ox + oy + oz) + (fabsf(rel.x) + fabsf(rel.y) + fabsf(rel.z));
  return p;
}

// FP32 proof that driver_filter fails.  A coordinate carries the roundings of its three
// terms and of their sums, at most 2^-21 of the sum of the terms' magnitudes; the
// coordinate itself may be small against them (a wall through the middle of a wide
// domain).  The distance to the driver is a sum of such coordinates (their sum is m), of
// the driver's constants (n1 bounds its factors) and of rc, each entering with at most
// 2^-20 of its magnitude; the margin is 2^-18 of all of them.  Away from the walls it
// spares the FP64 filter (26 FP64 instructions with a square root per particle and
// driver; a box has six).  One magnitude for the three axes keeps k_count_pairs at 64
// registers: with one an axis it had 72, and 324 us instead of 293 (2 M bed).
__device__ __forceinline__ bool driver_far(const DriverDev& d, float rc, const PosF& p) {
  if (d.kind == 0) {
    const float h = p.x * d.nf[0] + p.y * d.nf[1] + p.z * d.nf[2];
    const float ex = h * d.nf[0] - d.cpf[0], ey = h * d.nf[1] - d.cpf[1], ez = h * d.nf[2] - d.cpf[2];
    const float lim = rc + (p.m * d.n1 * d.n1 + d.cp1 + rc) * 3.8146973e-06f;
    return lim > 1e-15f && lim < 1e15f && ex * ex + ey * ey + ez * ez > lim * lim;
  }
  const float ex = p.x * d.af[0] - d.cf[0], ey = p.y * d.af[1] - d.cf[1], ez = p.z * d.af[2] - d.cf[2];
  const float mag = p.m * d.n1 + d.c1 + d.rf + rc;
  const float lim = d.rf - rc - mag * 3.8146973e-06f;
  return lim > 1e-15f && mag < 1e15f && ex * ex + ey * ey + ez * ez < lim * lim;
}

}  // namespace dem
