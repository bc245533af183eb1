// The conjugate gradient's device state and its resident form (cg_resident.cu).
#pragma once
#include "internal.cuh"

namespace ugpu {

struct CgDev {
    double rz;      // (r, z) of the current iterate
    double pAp;     // (p, Ap)
    double pr;      // (p, r)            (flexible form)
    double beta;
    double rnorm;
    double alpha;
    double gnorm;   // ||r|| at the stop
    long long it;   // the reference's `it`
    long long iterates;
    int done;
    int reason;
    int converged;
    int pad;
};

// A whole solve of small systems (unpreconditioned, or Jacobi with the weights dinv) as one cooperative kernel
struct CgResident {
    static bool fits(const Context &c, const Mat &A);
    // dev receives the final state; z, p0, p1: n doubles each; sums: sum_bytes(); work on c.stream.  False: the device
    // does not hold the kernel's CTAs at once, x is as it was
    static size_t sum_bytes(const Context &c);
    static bool run(Context &c, const Mat &A, const double *b, double *x, const double *dinv, double *z, double *p0,
                    double *p1, void *sums, CgDev *dev, double atol, long long max_it);
};

}  // namespace ugpu
