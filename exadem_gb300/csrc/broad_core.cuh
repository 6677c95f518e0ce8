// broad_core.cuh -- FP32 decisions shared by the sphere and polyhedron list builds.
#pragma once
#include "dem_ctx.cuh"

namespace dem {

// FP32 proof that driver_filter fails: the distance is evaluated in FP32, where the
// coordinates (a sum of three FP32 terms) and every operation carry at most 2^-21 of
// the magnitudes that enter, and the margin is 2^-18 of their sum.  Away from the walls it spares the FP64 filter (26 FP64
// instructions with a square root per particle and driver; a box has six).
__device__ __forceinline__ bool driver_far(const DriverDev& d, float rc, float px, float py, float pz) {
  if (d.kind == 0) {
    const float h = px * d.nf[0] + py * d.nf[1] + pz * d.nf[2];
    const float ex = h * d.nf[0] - d.cpf[0], ey = h * d.nf[1] - d.cpf[1], ez = h * d.nf[2] - d.cpf[2];
    const float pp = fabsf(px) + fabsf(py) + fabsf(pz);
    const float lim = rc + (pp * d.n1 * d.n1 + d.cp1 + rc) * 3.8146973e-06f;
    return lim > 1e-15f && lim < 1e15f && ex * ex + ey * ey + ez * ez > lim * lim;
  }
  const float qx = px * d.af[0], qy = py * d.af[1], qz = pz * d.af[2];
  const float ex = qx - d.cf[0], ey = qy - d.cf[1], ez = qz - d.cf[2];
  const float mag = fabsf(qx) + fabsf(qy) + fabsf(qz) + d.c1 + d.rf + rc;
  const float lim = d.rf - rc - mag * 3.8146973e-06f;
  return lim > 1e-15f && mag < 1e15f && ex * ex + ey * ey + ez * ez < lim * lim;
}

}  // namespace dem
