// The power method of one level as one kernel (pm_resident.cu).
#pragma once
#include "internal.cuh"

namespace ugpu {

bool pm_resident_fits(const Context &c, const Mat &A);
size_t pm_resident_bytes(const Context &c);
// *lambda (device) = the estimate; y0: the start vector (overwritten), y1: scratch, n doubles each; sums:
// pm_resident_bytes(); work on c.stream.  False: the device does not hold the kernel's CTAs at once, y0 is as it was
bool pm_resident(Context &c, const Mat &A, double *y0, double *y1, void *sums, double *lambda, double tol,
                 long long max_it);

}  // namespace ugpu
