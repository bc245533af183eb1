// MPRGP on small problems: the whole solve in one kernel.
//
// The loop of utopia::MPRGP::solve (quadratic_programming/utopia_MPRGP.hpp:57-262) as qp.cu runs it for large
// problems in four to six kernels per iteration, with the same operations and decisions.  As in the resident
// conjugate gradient (cg_resident.cu) every thread owns one to four rows for the whole solve, the rows'
// vectors (and matrix rows of at most eight entries) stay in registers, and an iteration is two exchanges
// (gridsync.cuh): (s, A s), (s, g) and the step bound after the product, then the four dots of the step.  An
// expansion step takes a third: its projected iterate must be complete before g = A x - b, and the dots
// follow.  An entry whose column belongs to another CTA forms that row's p = fi - beta_sc p_old itself.
//
// The convergence test (a root and a division) of an iteration runs beside the next iteration's first exchange,
// before which neither x nor g changes.
// Measured per iteration (four of five are expansion steps), obstacle problems of n = 1024 / 4096 / 16,384 / 65,536 /
// 90,000 / 160,000 / 302,500: 8.8 / 9.2 / 11.3 / 14.7 / 16.7 / 24.8 / 29.8 us, in separate kernels 42 / 38 / 39 / 41 /
// 42 / 48 / 58 us (power method included).  Bound by the exchanges (about 2.3 us each, 0.7 us in a cluster), the
// chain of dependent FP64 operations (60 cycles each) around them, and the FP64 pipe on large problems.
// The step bound divides exactly only where a row's single-precision bracket reaches below the least upper
// end of the CTA's brackets; the minimum is the one all rows' exact quotients give.
#include <cmath>

#include "abi_util.cuh"
#include "device_util.cuh"
#include "gridsync.cuh"
#include "mprgp.cuh"
#include "qp_device.cuh"

namespace ugpu {

namespace {

constexpr int kThreads = 512;
constexpr int kMaxRpt = 4;  // rows per thread
constexpr int kRegRow = 8;  // row entries kept in registers (at most two rows per thread)
constexpr int64_t kClusterRows = 6144;  // rows up to which the grid is one cluster

struct MprgpArgs {
    const int32_t *rp, *ci;
    const double *cv;
    int n, rows;  // rows per CTA
    const double *b, *lb, *ub;
    double *x, *fi, *beta, *p0, *p1;
    char *sums;
    QpDev *dev;
    int *kflag;
    double atol, rtol, eig_tol, lambda;
    long long max_it, eig_max_it;
};

enum Product : int { kOfP = 0, kOfBeta = 1, kOfX = 2, kOfScaled = 3 };

template <int NV, int MIN, bool CL>
using Exchange = typename std::conditional<CL, ClusterExchange<NV, MIN>, GridExchange<NV, MIN>>::type;

// A bracket [lo, hi] of the order key of h = d / p, the step bound of a row at distance d = x - (p > 0 ? l : u) of
// its bound, from a single-precision quotient: d and p are truncated to binary32 (relative error < 2^-23
// each), the fast division adds 2 ulp, the bracket is widened by 2^-16.  Rows with p = 0 and rows at least 2^50
// steps away are at the cap 1e15 and get no bracket (lo = hi = ~0); operands outside 2^-60 .. 2^60 get lo = 0,
// hi = ~0: evaluated exactly.  (qp_alpha_f_bracket subtracts in single precision to spare the FP64 pipe and leaves
// rows near their bound to the exact quotient; here those divisions would be on every iteration's chain.)
__device__ __forceinline__ void bound_bracket(double d, double p, unsigned long long &lo, unsigned long long &hi) {
    const unsigned long long bd = dbits(d), bp = dbits(p);
    const uint32_t ed = uint32_t(bd >> 52) & 0x7ffu, ep = uint32_t(bp >> 52) & 0x7ffu;
    if ((bp << 1) == 0ull) {
        lo = hi = ~0ull;
        return;
    }
    lo = 0ull;
    hi = ~0ull;
    if (ep - 963u > 120u) return;
    if ((bd << 1) == 0ull) {
        lo = hi = qp_key(0.0);
        return;
    }
    if (ed - 963u > 120u) {
        // |d| > 2^61 and |p| < 2^10, d and p of one sign (a feasible iterate): beyond the cap
        if (ed >= 1084u && ed != 2047u && ep < 1033u && ((bd ^ bp) >> 63) == 0ull) lo = hi = ~0ull;
        return;
    }
    const float df = __uint_as_float((uint32_t(bd >> 32) & 0x80000000u) | ((ed - 896u) << 23) | (uint32_t(bd >> 29) & 0x7fffffu));
    const float pf = __uint_as_float((uint32_t(bp >> 32) & 0x80000000u) | ((ep - 896u) << 23) | (uint32_t(bp >> 29) & 0x7fffffu));
    const float q = __fdividef(df, pf);
    const float q1 = q * (1.0f - 0x1p-16f), q2 = q * (1.0f + 0x1p-16f);
    lo = qp_key(f2d_bits(fminf(q1, q2)));
    hi = qp_key(f2d_bits(fmaxf(q1, q2)));
}

// CL: the grid is one cluster; fi, beta, x and both p live in shared memory and are read across it
template <int RPT, bool REG, bool CL>
__global__ void __launch_bounds__(kThreads, 1) k_mprgp_resident(MprgpArgs a) {
    // [rows] the product's input (CL: x, fi, beta and two sets of p), four arrays of blockDim.x partials, CL: slots
    extern __shared__ double sh[];
    __shared__ double s_bb, s_ff, s_gg, s_a0, s_alpha, s_nbsc, s_gnorm, s_gnorm0;
    __shared__ unsigned long long s_part[4], s_amin, s_hmin, s_key[kThreads / 32];
    __shared__ int s_late, s_reason;
    const int t = threadIdx.x, nt = blockDim.x, lane = t & 31, warp = t >> 5;
    const int row0 = blockIdx.x * a.rows, row1 = min(a.n, row0 + a.rows);
    double *sx = sh, *sfi = sx + a.rows, *sbeta = sfi + a.rows, *sp = sbeta + a.rows, *sq = sp + a.rows;  // CL
    double *part = CL ? sq + a.rows : sh + a.rows;  // [4][nt]
    const unsigned long long cap = qp_key(1e15);

    // exchanges, all by warp 0: after the product (s, A s), (s, g) and the step bound; after the step (fi, A s),
    // (beta, beta), (fi, fi) and (gp, gp)
    Exchange<3, 4, CL> x_product;
    Exchange<4, 0, CL> x_step;
    if constexpr (CL) {
        double *w = part + 4 * nt;
        x_product.init(w, blockIdx.x, gridDim.x);
        x_step.init(w + x_product.kDoubles, blockIdx.x, gridDim.x);
        if (t == 0) {
            x_product.init_barriers();
            x_step.init_barriers();
        }
        __syncthreads();
        cluster_barrier();
    } else {
        const int G = int(gridDim.x);
        x_product.init(a.sums, G);
        x_step.init(a.sums + x_product.bytes(G), G);
    }
    long long n_product = 0, n_step = 0;  // exchanges so far

    if (t == 0) {
        s_late = 0;
        s_hmin = ~0ull;
        s_reason = 0;
        s_gnorm = s_gnorm0 = -1.0;
    }
    double x[RPT], g[RPT], p[RPT], fi[RPT], beta[RPT], q[RPT], l[RPT], u[RPT];
#pragma unroll
    for (int k = 0; k < RPT; ++k) g[k] = q[k] = 0.0;
    double mv[REG ? RPT : 1][kRegRow];
    int mc[REG ? RPT : 1][kRegRow];  // own column: its local row; another CTA's: -2 - remote(column); none: -1
    auto remote = [&](int c) { return CL ? (c / a.rows) << 16 | c % a.rows : c; };
#pragma unroll
    for (int k = 0; k < RPT; ++k) {
        const int lr = t + k * nt, i = row0 + lr;
        const bool in = i < row1;
        l[k] = in ? a.lb[i] : -DBL_MAX_D;
        u[k] = in ? a.ub[i] : DBL_MAX_D;
        x[k] = in ? proj(l[k], u[k], a.x[i]) : 0.0;
        p[k] = 0.0;
        if (CL && lr < a.rows) sp[lr] = sq[lr] = 0.0;  // the old p of the first direction (p = fi + 0 p)
        if constexpr (REG) {
            const int e0 = in ? a.rp[i] : 0, e1 = in ? a.rp[i + 1] : 0;
#pragma unroll
            for (int e = 0; e < kRegRow; ++e) {
                mv[k][e] = 0.0;
                mc[k][e] = -1;
                if (e0 + e < e1) {
                    const int c = a.ci[e0 + e];
                    mv[k][e] = a.cv[e0 + e];
                    mc[k][e] = c >= row0 && c < row1 ? c - row0 : -2 - remote(c);
                }
            }
        }
    }
    double *pold = a.p0, *pnew = a.p1;
    double nb = 0.0;  // -beta_sc of the pending direction p = fi - beta_sc p

    double scale = 1.0;
    // q = A v for v = p (own rows: `own`), beta, x or scale fi; the other CTAs' rows are read past L1 or across the cluster
    auto product = [&](Product what, const double *own) {
        auto far = [&](int c, double &v0, double &v1) {
            v1 = 0.0;
            if constexpr (CL) {
                const uint32_t at = 8u * uint32_t(c & 0xffff), r = uint32_t(c) >> 16;
                auto addr = [&](const double *s) { return uint32_t(__cvta_generic_to_shared(s)) + at; };
                if (what == kOfP) {
                    v0 = ld_cluster(addr(sfi), r);
                    v1 = ld_cluster(addr(sp), r);
                } else {
                    v0 = ld_cluster(addr(what == kOfBeta ? sbeta : what == kOfX ? sx : sfi), r);
                }
            } else {
                if (what == kOfP) {
                    v0 = __ldcg(a.fi + c);
                    v1 = __ldcg(pold + c);
                } else {
                    v0 = __ldcg((what == kOfBeta ? a.beta : what == kOfX ? a.x : a.fi) + c);
                }
            }
        };
        if constexpr (REG) {
            double h0[RPT][kRegRow], h1[RPT][kRegRow];
#pragma unroll
            for (int k = 0; k < RPT; ++k)
#pragma unroll
                for (int e = 0; e < kRegRow; ++e) {
                    h0[k][e] = h1[k][e] = 0.0;
                    if (mc[k][e] < -1) far(-2 - mc[k][e], h0[k][e], h1[k][e]);
                }
            __syncthreads();
#pragma unroll
            for (int k = 0; k < RPT; ++k) {
                double s = 0.0;
#pragma unroll
                for (int e = 0; e < kRegRow; ++e) {
                    if (mc[k][e] == -1) continue;
                    double v;
                    if (mc[k][e] >= 0) v = own[mc[k][e]];
                    else v = what == kOfP ? fma(nb, h1[k][e], h0[k][e]) : what == kOfScaled ? scale * h0[k][e] : h0[k][e];
                    s = fma(mv[k][e], v, s);
                }
                q[k] = s;
            }
        } else {
            __syncthreads();
#pragma unroll
            for (int k = 0; k < RPT; ++k) {
                const int i = row0 + t + k * nt;
                double s = 0.0;
                if (i < row1) {
                    const int e1 = __ldg(a.rp + i + 1);
                    for (int e = __ldg(a.rp + i); e < e1; ++e) {
                        const int c = __ldg(a.ci + e);
                        double v;
                        if (c >= row0 && c < row1) {
                            v = own[c - row0];
                        } else {
                            double v0, v1;
                            far(remote(c), v0, v1);
                            v = what == kOfP ? fma(nb, v1, v0) : what == kOfScaled ? scale * v0 : v0;
                        }
                        s = fma(__ldg(a.cv + e), v, s);
                    }
                }
                q[k] = s;
            }
        }
    };
    // x to the other CTAs; the exchange stands for a barrier
    auto publish_x = [&]() {
#pragma unroll
        for (int k = 0; k < RPT; ++k) {
            const int lr = t + k * nt;
            if (row0 + lr < row1) {
                sx[lr] = x[k];  // sx is also the product's input array where the grid is not a cluster
                if (!CL) __stcg(a.x + row0 + lr, x[k]);
            }
        }
        __syncthreads();
        if (warp == 0) {
            unsigned long long o[4];
            if (!x_step.exchange(n_step, s_part, o) && lane == 0) s_late = 1;
        }
        ++n_step;
        __syncthreads();
    };
    double d0, d1, d2, d3;
    auto faces = [&](int k) {  // fi, beta of row k of this thread, published, and their dots
        const int lr = t + k * nt;
        fi[k] = phi(l[k], u[k], x[k], g[k]);
        beta[k] = chopped(l[k], u[k], x[k], g[k]);
        if (row0 + lr < row1) {
            if (CL) {
                sfi[lr] = fi[k];
                sbeta[lr] = beta[k];
            } else {
                __stcg(a.fi + row0 + lr, fi[k]);
                __stcg(a.beta + row0 + lr, beta[k]);
            }
        }
        const double gp = fi[k] + beta[k];
        d1 = fma(beta[k], beta[k], d1);
        d2 = fma(fi[k], fi[k], d2);
        d3 = fma(gp, gp, d3);
    };
    auto gradient = [&]() {
        product(kOfX, sx);
        d0 = d1 = d2 = d3 = 0.0;
#pragma unroll
        for (int k = 0; k < RPT; ++k) {
            const int i = row0 + t + k * nt;
            const bool in = i < row1;
            g[k] = in ? q[k] - a.b[i] : 0.0;
            faces(k);
            p[k] = fi[k];
        }
    };
    // the sums of d0 .. d3 over the grid; then(sums) runs in lane 0 of warp 0
    auto exchange_sums = [&](auto then) {
        part[t] = d0;
        part[nt + t] = d1;
        part[2 * nt + t] = d2;
        part[3 * nt + t] = d3;
        __syncthreads();
        if (warp < 4) {
            const double s = warp_sum_of(part + warp * nt, nt);
            if (lane == 0) s_part[warp] = dbits(s);
        }
        __syncthreads();
        if (warp == 0) {
            unsigned long long o[4];
            const bool ok = x_step.exchange(n_step, s_part, o);
            if (lane == 0) {
                then(o);
                if (!ok) s_late = 1;
            }
        }
        ++n_step;
        __syncthreads();
    };
    // the sums of a step: -(fi, A s) / a0 to s_nbsc (with_fq), (beta, beta), (fi, fi), (gp, gp)
    auto exchange_step = [&](bool with_fq, double a0) {
        exchange_sums([&](const unsigned long long *o) {
            s_nbsc = with_fq ? -(bitsd(o[0]) / a0) : 0.0;
            s_bb = bitsd(o[1]);
            s_ff = bitsd(o[2]);
            s_gg = bitsd(o[3]);
        });
    };

    // MPRGP::power_method (utopia_MPRGP.hpp:351-387) from the vector of ones: y = A v, v = y / ||y||,
    // lambda = (v, A v), until ||v - A v|| or the change of lambda is below eps.  A v is the next iteration's y.  y is
    // published in fi, and another CTA's v_j is formed as scale y_j.  (The host passes lambda for larger problems.)
    double lambda = a.lambda;
    if (lambda == 0.0) {
        auto publish = [&](const double (&v)[RPT], double *shared, double *global) {
#pragma unroll
            for (int k = 0; k < RPT; ++k) {
                const int lr = t + k * nt;
                if (row0 + lr >= row1) continue;
                if (CL) shared[lr] = v[k];
                else __stcg(global + row0 + lr, v[k]);
            }
        };
        double v[RPT];
        d0 = d1 = d2 = d3 = 0.0;
#pragma unroll
        for (int k = 0; k < RPT; ++k) {
            v[k] = 1.0;
            if (t + k * nt < a.rows) sx[t + k * nt] = 1.0;
        }
        publish(v, sbeta, a.beta);  // not in fi: the first y replaces it while other CTAs may still read the ones
        exchange_sums([](const unsigned long long *) {});
        product(kOfBeta, sx);
        for (long long pit = 0; !s_late; ++pit) {
            d0 = 0.0;
#pragma unroll
            for (int k = 0; k < RPT; ++k) d0 = fma(q[k], q[k], d0);
            publish(q, sfi, a.fi);
            exchange_sums([&](const unsigned long long *o) { s_alpha = 1.0 / sqrt(bitsd(o[0])); });
            scale = s_alpha;
#pragma unroll
            for (int k = 0; k < RPT; ++k) {
                v[k] = scale * q[k];
                if (t + k * nt < a.rows) sx[t + k * nt] = v[k];
            }
            product(kOfScaled, sx);
            d0 = d1 = 0.0;
#pragma unroll
            for (int k = 0; k < RPT; ++k) {
                const double e = v[k] - q[k];
                d0 = fma(v[k], q[k], d0);
                d1 = fma(e, e, d1);
            }
            const double old = lambda;
            exchange_sums([&](const unsigned long long *o) {
                s_a0 = bitsd(o[0]);
                s_gnorm = sqrt(bitsd(o[1]));
            });
            lambda = s_a0;
            if (s_gnorm < a.eig_tol || fabs(old - lambda) < a.eig_tol || pit > a.eig_max_it) break;
        }
        __syncthreads();
    }
    if (t == 0) {
        s_alpha = 1.95 / lambda;
        s_gnorm = -1.0;
    }
    __syncthreads();
    const double alpha_bar = s_alpha;

    long long it = 0, iterates = 0;
    int reason = 0, conv = 0;
    publish_x();
    gradient();
    exchange_step(false, 1.0);
    bool cgpath = s_bb <= s_ff;
    bool tested = true;  // the last iteration's convergence test has been made (there is none at the start)
    while (!s_late) {
        // p = fi - beta_sc p and, for the CG path, the brackets of the step bound
        {
            double *const swap = pold;
            pold = pnew;
            pnew = swap;
        }
        if (CL) {
            double *const swap = sp;
            sp = sq;
            sq = swap;
        }
        double *const own = CL ? (cgpath ? sq : sbeta) : sx;
        unsigned long long lo[RPT], hmin = ~0ull;
#pragma unroll
        for (int k = 0; k < RPT; ++k) {
            const int lr = t + k * nt;
            const bool in = row0 + lr < row1;
            p[k] = fma(nb, p[k], fi[k]);
            if (in) {
                if (CL) {
                    sq[lr] = p[k];
                } else {
                    __stcg(pnew + row0 + lr, p[k]);
                    sx[lr] = cgpath ? p[k] : beta[k];
                }
            }
            lo[k] = ~0ull;
            if (cgpath && in) {
                unsigned long long hi;
                bound_bracket(x[k] - (dkey(p[k]) > 0 ? l[k] : u[k]), p[k], lo[k], hi);
                hmin = hi < hmin ? hi : hmin;
            }
        }
        if (cgpath) {
            hmin = warp_min_u64(hmin);
            if (lane == 0) atomicMin(&s_hmin, hmin);
        }
        product(cgpath ? kOfP : kOfBeta, own);
        {
            const unsigned long long least = cgpath ? min(s_hmin, cap) : 0ull;
            unsigned long long key = cap;
            d0 = d1 = 0.0;
#pragma unroll
            for (int k = 0; k < RPT; ++k) {
                const double s = cgpath ? p[k] : beta[k];
                d0 = fma(s, q[k], d0);
                d1 = fma(s, g[k], d1);
                if (cgpath && lo[k] <= least) {
                    const unsigned long long e = qp_alpha_f_key(x[k], p[k], l[k], u[k]);
                    key = e < key ? e : key;
                }
            }
            part[t] = d0;
            part[nt + t] = d1;
            if (cgpath) {
                key = warp_min_u64(key);
                if (lane == 0) s_key[warp] = key;
            }
        }
        __syncthreads();
        if (warp < 2) {
            const double s = warp_sum_of(part + warp * nt, nt);
            if (lane == 0) s_part[warp] = dbits(s);
        } else if (warp == 2) {
            const unsigned long long k = cgpath ? warp_min_u64(lane < nt / 32 ? s_key[lane] : ~0ull) : ~0ull;
            if (lane == 0) {
                s_part[2] = k;
                s_hmin = ~0ull;
            }
        }
        __syncthreads();
        if (warp == 0) {
            unsigned long long o[3];
            const bool ok = x_product.exchange(n_product, s_part, o);
            if (lane == 0) {
                s_a0 = bitsd(o[0]);
                s_alpha = bitsd(o[1]) / bitsd(o[0]);
                s_amin = o[2];
                if (!ok) s_late = 1;
            }
        } else if (warp == 3 && lane == 0 && !tested) {
            // the convergence test of the iteration that has ended, beside the exchange
            const double gnorm = sqrt(s_gg);
            const double gnorm0 = it == 1 ? gnorm : s_gnorm0;
            const double rel = gnorm / gnorm0;
            s_gnorm = gnorm;
            s_gnorm0 = gnorm0;
            int r = 0;
            if (gnorm <= a.atol) r = UGPU_CONVERGED_FNORM_ABS;
            if (rel <= a.rtol) r = UGPU_CONVERGED_FNORM_RELATIVE;
            if (it >= a.max_it) r = UGPU_DIVERGED_MAX_IT;
            s_reason = r;
        }
        ++n_product;
        __syncthreads();
        if (s_late) break;
        if (!tested && s_reason) {
            reason = s_reason;
            conv = reason > 0;
            iterates = it;
            break;
        }
        const double a0 = s_a0;
        if (a0 <= 0.0) {  // negative curvature
            reason = UGPU_DIVERGED_INDEFINITE;
            conv = 1;
            iterates = it;
            break;
        }
        bool expand = false;
        double alpha = s_alpha;
        if (cgpath) {
            const double alpha_f = qp_unkey(s_amin);
            expand = !(alpha <= alpha_f);
            if (expand) alpha = alpha_f;
        }
        if (!expand) {
            d0 = d1 = d2 = d3 = 0.0;
#pragma unroll
            for (int k = 0; k < RPT; ++k) {
                x[k] = x[k] - alpha * (cgpath ? p[k] : beta[k]);
                g[k] = g[k] - alpha * q[k];
                faces(k);
                if (cgpath) d0 = fma(fi[k], q[k], d0);
            }
            exchange_step(cgpath, a0);
            nb = s_nbsc;
        } else {
#pragma unroll
            for (int k = 0; k < RPT; ++k) {
                const double xn = x[k] - alpha * p[k];
                const double gn = g[k] - alpha * q[k];
                x[k] = proj(l[k], u[k], xn - alpha_bar * phi(l[k], u[k], xn, gn));
            }
            publish_x();
            gradient();
            exchange_step(false, 1.0);
            nb = 0.0;
        }
        ++it;
        tested = false;
        cgpath = s_bb <= s_ff;
    }
#pragma unroll
    for (int k = 0; k < RPT; ++k) {
        const int i = row0 + t + k * nt;
        if (i < row1) a.x[i] = x[k];
    }
    if (t == 0) {
        if (s_late) atomicExch(a.kflag, 1);
        if (blockIdx.x == 0) {
            QpDev *o = a.dev;
            o->lambda = lambda;
            o->it = it;
            o->iterates = iterates;
            o->gnorm = s_gnorm;
            o->gnorm0 = s_gnorm0;
            o->done = 1;
            o->reason = reason;
            o->converged = conv;
        }
    }
    __syncthreads();
    if (CL) cluster_barrier();  // no CTA leaves while another may still read its shared memory
}

}  // namespace

// Rows of at most eight entries: up to four rows per thread (311,296 rows; the times are above).  Longer ones, up to
// two rows per thread and 32 entries: random graphs of 2001 / 60,001 / 100,001 / 150,001 rows 18 / 22 / 33 / 37 us per
// iteration against 33 / 42 / 46 / 49 in separate kernels, but 73 against 57 at 200,001.
bool MprgpResident::fits(const Context &c, const Mat &A) {
    if (A.nrows < 1 || A.max_row <= 0) return false;
    const int64_t threads = int64_t(c.sms) * kThreads;
    return A.nrows <= threads * (A.max_row <= kRegRow ? kMaxRpt : 2) && A.max_row <= 32;
}

bool MprgpResident::own_power_method(const Context &c, const Mat &A) {
    return A.nrows <= int64_t(c.sms) * kThreads * 2;
}

size_t MprgpResident::sum_bytes(const Context &c) {
    return GridExchange<3, 4>::bytes(c.sms) + GridExchange<4>::bytes(c.sms);
}

bool MprgpResident::run(Context &c, const Mat &A, const double *b, double *x, const double *lb, const double *ub,
                        double *fi, double *beta, double *p0, double *p1, void *sums, QpDev *dev, double atol,
                        double rtol, long long max_it, double lambda, double eig_tol, long long eig_max_it) {
    const int64_t n = A.nrows;
    const bool cl = n <= kClusterRows && A.max_row <= kRegRow;
    // at least 64 rows per CTA, at least the four warps that the exchanges and the convergence test take
    int64_t G = std::min<int64_t>(cl ? 16 : c.sms, (n + 63) / 64);
    const int64_t rows = ((n + G - 1) / G + 31) / 32 * 32;
    G = (n + rows - 1) / rows;
    const int rpt = rows <= kThreads ? 1 : rows <= 2 * kThreads ? 2 : 4;
    const int nt = int(std::max<int64_t>(128, ((rows + rpt - 1) / rpt + 31) / 32 * 32));
    MprgpArgs a{};
    a.rp = A.rowptr.as<int32_t>();
    a.ci = A.colidx.as<int32_t>();
    a.cv = A.vals.as<double>();
    a.n = int(n);
    a.rows = int(rows);
    a.b = b;
    a.lb = lb;
    a.ub = ub;
    a.x = x;
    a.fi = fi;
    a.beta = beta;
    a.p0 = p0;
    a.p1 = p1;
    a.sums = static_cast<char *>(sums);
    a.dev = dev;
    a.kflag = c.d_kflags() + 2;
    a.atol = atol;
    a.rtol = rtol;
    a.max_it = max_it;
    a.lambda = lambda;
    a.eig_tol = eig_tol;
    a.eig_max_it = eig_max_it;
    UGPU_CUDA(cudaMemsetAsync(sums, 0, sum_bytes(c), c.stream));
    UGPU_CUDA(cudaMemsetAsync(p0, 0, sizeof(double) * size_t(n), c.stream));
    UGPU_CUDA(cudaMemsetAsync(p1, 0, sizeof(double) * size_t(n), c.stream));
    const bool reg = A.max_row <= kRegRow && rpt <= 2;
    const size_t slots = ClusterExchange<3, 4>::kDoubles + ClusterExchange<4>::kDoubles;
    const size_t smem = sizeof(double) * (size_t(rows) * (cl ? 5 : 1) + 4 * size_t(nt) + (cl ? slots : 0));
    void (*f)(MprgpArgs) = cl         ? k_mprgp_resident<1, true, true>
                           : rpt == 1 ? (reg ? k_mprgp_resident<1, true, false> : k_mprgp_resident<1, false, false>)
                           : rpt == 2 ? (reg ? k_mprgp_resident<2, true, false> : k_mprgp_resident<2, false, false>)
                                      : k_mprgp_resident<4, false, false>;
    return launch_resident(c, f, a, int(G), nt, smem, cl);
}

}  // namespace ugpu
