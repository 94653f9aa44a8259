/*
 * hbt_check.h - device checks of the engine's own FP64 elementary functions
 * (libhbt_gpu.so).  The pair kernels and the radii fits evaluate cos and
 * exp with table-driven implementations of their own (csrc/hbt_math.cuh);
 * this entry point runs them on the device over caller-given arguments so
 * that tests can compare them with the host's libm.  Not part of the
 * reference's interface.
 */
#ifndef HBT_CHECK_H
#define HBT_CHECK_H

#include "hbt_gpu.h"

#ifdef __cplusplus
extern "C" {
#endif

#define HBT_CHECK_COS 0 /* table_cos, the cosine of the pairs of far particles,
                           at scale 1: cos(x) */
#define HBT_CHECK_EXP 1 /* the radii fits' table_exp */
#define HBT_CHECK_DFCOS 2 /* the same of x rounded to hi = (float)x and lo =
                             (float)(x - hi): the double-float form runs the
                             FP64 form's kernels */
#define HBT_CHECK_COS_PHASE 3 /* table_cos with the pair kernels' scale:
                                 cos(x / hbarC), the product never rounded */

/* out[i] = f(x[i]) on `device` for the function `which`; host arrays. */
hbt_status hbt_check_math(int device, int32_t which, int64_t n, const double *x, double *out);

/* The pair kernels' cosine of fixed-point phases on `device`: out[i] = cos(2 pi /
 * 512 (steps[2 i] 2^-37 + steps[2 i + 1] 2^-67)), |steps[2 i]| < 2^62 and 0 <=
 * steps[2 i + 1] < 2^30. */
hbt_status hbt_check_cos_fixed(int device, int64_t n, const int64_t *steps, double *out);

/* How the library reads or writes a caller's array of doubles at p where the
 * GPU reaches host memory itself: 2 by a kernel, 1 by copies.  No device call. */
int32_t hbt_check_host_route(const void *p);

#ifdef __cplusplus
}
#endif
#endif /* HBT_CHECK_H */
