/*
 * dem_selftest.h -- self-tests of the device arithmetic helpers.
 * No reference counterpart: these check, on the GPU, that the exact
 * shortcuts used by the fused step return the IEEE result bit for bit.
 */
#ifndef DEM_SELFTEST_H
#define DEM_SELFTEST_H
#include <stdint.h>
#include "dem_hotpath.h"
#ifdef __cplusplus
extern "C" {
#endif
/* Draws n seeded (a, b) pairs over several magnitude ranges, and counts the
 * pairs where the reciprocal-based division (Markstein's correction step with
 * y = RN(1/b)) differs in any bit from the compiled division a / b.        */
int dem_selftest_division(uint64_t n, uint64_t seed, uint64_t* mismatches, uint64_t* fast_path_taken);

/* Draws n seeded near-threshold cases of the polyhedron broad-phase tests
 * (kind = case % 6: 0 vertex gate / OBB::intersect, 1 filter_vv, 2 filter_ve,
 * 3 filter_vf, 4 filter_ee, 5 vertex displacement against max_displ) and
 * evaluates each with its FP32 decision and its FP64 test.
 * counts[4 * kind + k] (24 entries), k = 0: decided cases whose result differs
 * from FP64 (must be 0), 1: undecided cases, 2: decided true, 3: FP64 true.  */
int dem_selftest_poly_decisions(uint64_t n, uint64_t seed, uint64_t* counts);

/* Draws n seeded operand pairs (typical magnitudes, short significands that
 * give exact products and ties, the whole exponent range, boundaries, zeros,
 * subnormals, infinities, NaNs) and counts the results of the integer-pipe
 * binary64 multiply (emu_dmul, and the exact x*2 / x*0.5) that differ in any
 * bit from the hardware multiply; for each pair and three derived ones (the
 * negation of a, its neighbours, a gap of 0..70 binades) also the sums and
 * differences of the integer-pipe addition (emu_dadd_nb, emu_dsub_nb) that
 * differ from the hardware's, where the addition keeps its fast path.     */
int dem_selftest_emu_mul(uint64_t n, uint64_t seed, uint64_t* mismatches);

/* Draws n seeded (branch, spin, normal force, moment) cases around the range
 * bounds of the exact rolling-clip shortcut (mur = 0) and counts the moments
 * that differ in any bit from the formula (r = b.w / w.w, ... , m * t/|m|);
 * fast_path_taken counts the cases inside the shortcut's range.            */
int dem_selftest_rolling_clip(uint64_t n, uint64_t seed, uint64_t* mismatches, uint64_t* fast_path_taken);

/* Whether the bytes at p lie inside one allocation of the current device, so
 * that dem_set_particles and dem_get_particles (on_device = 1) copy them with
 * their own kernel; what does not goes through cudaMemcpyAsync.             */
int dem_selftest_copy_range(const void* p, uint64_t bytes, int* inside);

/* The candidate records a particle of the FP32 sphere list build gets where
 * they may take `budget` bytes in all: records[0] for particles and walls,
 * records[1] for mesh features.  dem_selftest_records returns those that the
 * context holds now; budget > 0 drops them and bounds the following builds'
 * (0: no change; a context starts with a sixteenth of the free memory).     */
int dem_selftest_record_plan(uint64_t particles, int mesh, uint64_t budget, uint32_t* records);
int dem_selftest_records(dem_ctx* ctx, uint64_t budget, uint32_t* records);

/* The multiply placement that the integration of the present particles runs:
 * that of dem_set_mul_mode or dem_autotune, else the rule by particle count. */
int dem_selftest_integration_mode(const dem_ctx* ctx, int* mode);

#ifdef __cplusplus
}
#endif
#endif
