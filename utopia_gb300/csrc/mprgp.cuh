// MPRGP's device state and its resident form (mprgp_resident.cu).
#pragma once
#include "internal.cuh"

namespace ugpu {

struct QpDev {
    double qa0, qa1;              // the iteration's product s -> A s: (s, A s), (s, g); s = p or beta
    double neg_bsc;               // -beta_sc of the pending direction p = fi - beta_sc p (0: p = fi)
    unsigned long long amin;      // key (qp_key) of alpha_f = min step bound, reset after each use
    double alpha_cg, alpha_f, beta_sc;
    double beta_beta, fi_fi, gnorm, gnorm0;
    long long it, iterates;
    int done, reason, converged;
    int gate_cg, gate_prop, gate_exp;   // branch of the current iteration
    int step;                           // 0: CG step, 1: expansion step
    double lambda;                      // the power method's estimate (resident form)
};

// A solve of small problems as one kernel (work on c.stream).
// fi, beta, p0, p1: n doubles each; sums: sum_bytes(); dev receives the final state.  False from run(): the
// device does not hold the kernel's CTAs at once, x is as it was.
struct MprgpResident {
    static bool fits(const Context &c, const Mat &A);
    // Whether run() makes the power-method estimate itself (lambda = 0): up to two rows per thread (20 iterations on
    // 380^2 0.58 ms, on 400^2 with the host's estimate 1.54).  Above, it would save 0.9 ms too, but its sums
    // round in another order than the separate kernels', and over the thousands of iterations of a large free
    // boundary the last bits of lambda move the iteration count by a few percent.
    static bool own_power_method(const Context &c, const Mat &A);
    static size_t sum_bytes(const Context &c);
    static bool run(Context &c, const Mat &A, const double *b, double *x, const double *lb, const double *ub, double *fi,
                    double *beta, double *p0, double *p1, void *sums, QpDev *dev, double atol, double rtol,
                    long long max_it, double lambda, double eig_tol, long long eig_max_it);
};

}  // namespace ugpu
