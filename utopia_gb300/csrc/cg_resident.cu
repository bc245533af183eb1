// Conjugate gradient on small systems: the whole solve in one kernel.
//
// The loop of ConjugateGradient::preconditioned_solve / unpreconditioned_solve
// (utopia/solvers/smoothers/utopia_ConjugateGradient_impl.hpp:90-294) with the InvDiag preconditioner or none, as
// cg.cu runs it for large systems in three kernels per iteration.  Up to a few hundred thousand rows those
// kernels are shorter than the gaps between them (256^2: 23 us per iteration), so here every thread owns
// one to four rows for the whole solve; x, r, p, z and (rows of at most eight entries) the row's matrix
// entries stay in registers, and an iteration is two exchanges of sums (gridsync.cuh): after (p, Ap), and
// after (r, r) and (z, r).
//
// There is no third exchange between p = z + beta p and the product: a CTA's rows read each other's new
// p from shared memory, and an entry whose column belongs to another CTA forms z_j + beta p_j itself from
// the old p and z (in global memory, or across the shared memory of a cluster; p is double-buffered).
//
// Two grids.  A CTA per SM (cooperative launch), exchanges through L2.  Or one cluster of at most 16 CTAs,
// exchanges and reads through distributed shared memory: shorter exchanges, a tenth of the FP64 pipes.
// Measured per iteration, 5-point stencil, n = 1024 / 2304 / 4096 / 6400 / 10,000 / 65,536 / 155,236 / 302,500:
//   cluster       4.1 / 4.6 / 5.4 / 6.8 / 7.9 us
//   CTA per SM    7.2 / 7.1 / 7.1 / 7.1 / 6.7 / 9.7 / 12.9 / 17.8 us
//   kernels       21.6 / 21.7 /  - /  - / 22.9 / 22.7 / 23.7 / 29.1 us
// Bound by the exchanges, the chain of dependent FP64 operations between them (about 70 per iteration) and, from
// about 50,000 rows, the FP64 pipe (12 operations per row and iteration).
#include <cmath>

#include "abi_util.cuh"
#include "cg.cuh"
#include "device_util.cuh"
#include "gridsync.cuh"

namespace ugpu {

namespace {

constexpr int kThreads = 512;
constexpr int kMaxRpt = 4;   // rows per thread
constexpr int64_t kClusterRows = 6144;  // rows up to which the grid is one cluster
constexpr int kRegRow = 8;   // row entries kept in registers (at most two rows per thread)

struct ResArgs {
    const int32_t *rp, *ci;
    const double *cv;
    int n, rows;  // rows per CTA
    const double *b, *dinv;  // dinv null: no preconditioner
    double *x, *z, *p0, *p1;
    char *sums;  // the two exchanges' counters and partials
    CgDev *dev;
    int *kflag;
    double atol;
    long long max_it;
};

// CL: the grid is one cluster; z and both p live in shared memory and are read across it
template <int RPT, bool REG, bool CL>
__global__ void __launch_bounds__(kThreads, 1) k_cg_resident(ResArgs a) {
    // the CTA's p [rows] (CL: z and two sets of p), then two arrays of blockDim.x partials (CL: and the sums' slots)
    extern __shared__ double sh[];
    __shared__ double s_sum[2], s_alpha, s_beta, s_rnorm;
    __shared__ unsigned long long s_part[2];
    __shared__ int s_late;
    const int t = threadIdx.x, nt = blockDim.x, lane = t & 31, warp = t >> 5;
    double *sz = sh, *sp = CL ? sh + a.rows : sh, *sq = sp + a.rows;  // CL: sp the old p, sq the new one
    double *sa = CL ? sq + a.rows : sq, *sb = sa + nt;
    const int row0 = blockIdx.x * a.rows, row1 = min(a.n, row0 + a.rows);
    const bool jac = a.dinv != nullptr;  // otherwise z = r

    // Each sum has its own exchange, carried out by its own warp: one exchange of both by one warp measured 1 us
    // more per iteration (its two chains of additions in one warp, and a barrier before it).
    using Exchange = typename std::conditional<CL, ClusterExchange<1>, GridExchange<1>>::type;
    Exchange gx;
    if constexpr (CL) {
        gx.init(sb + nt + (warp & 1) * Exchange::kDoubles, blockIdx.x, gridDim.x);
        if (warp < 2 && lane == 0) gx.init_barriers();
        __syncthreads();
        cluster_barrier();
    } else {
        gx.init(a.sums + (warp & 1) * Exchange::bytes(int(gridDim.x)), int(gridDim.x));
    }
    long long ex = 0;  // exchanges of this warp's sum so far
    // Sums over the grid: sa into sum 0 in warp 0 and, with two, sb into sum 1 in warp 1; then(w, sum) runs in lane 0 of
    // the warp.  The caller synchronises before it reads the sums or what then() wrote.
    auto exchange = [&](bool two, auto then) {
        __syncthreads();
        if (warp < (two ? 2 : 1)) {
            const double s = warp_sum_of(warp ? sb : sa, nt);
            if (lane == 0) s_part[warp] = dbits(s);
            __syncwarp();
            unsigned long long g[1];
            const bool ok = gx.exchange(ex++, s_part + warp, g);
            if (lane == 0) {
                s_sum[warp] = bitsd(g[0]);
                if (!ok) s_late = 1;
                then(warp, bitsd(g[0]));
            }
        }
    };

    if (t == 0) s_late = 0;
    // rows t, t + nt, ... of the CTA; r = b - A x
    double x[RPT], r[RPT], p[RPT], z[RPT], d[RPT], q[RPT];
    // REG: the row's entries; a column of this CTA as its local row, another one as -2 - column (CL: -2 - (its CTA
    // << 16 | its local row)), none as -1
    auto remote = [&](int c) { return CL ? (c / a.rows) << 16 | c % a.rows : c; };
    double mv[REG ? RPT : 1][kRegRow];
    int mc[REG ? RPT : 1][kRegRow];
    double s0 = 0.0, s1 = 0.0;
#pragma unroll
    for (int k = 0; k < RPT; ++k) {
        const int i = row0 + t + k * nt;
        const bool in = i < row1;
        const int e0 = in ? a.rp[i] : 0, e1 = in ? a.rp[i + 1] : 0;
        x[k] = in ? a.x[i] : 0.0;
        d[k] = in && jac ? a.dinv[i] : 1.0;
        p[k] = 0.0;
        double s = 0.0;
        if constexpr (REG) {
#pragma unroll
            for (int e = 0; e < kRegRow; ++e) {
                mv[k][e] = 0.0;
                mc[k][e] = -1;
                if (e0 + e < e1) {
                    const int c = a.ci[e0 + e];
                    mv[k][e] = a.cv[e0 + e];
                    mc[k][e] = c >= row0 && c < row1 ? c - row0 : -2 - remote(c);
                    s = fma(mv[k][e], a.x[c], s);
                }
            }
        } else {
            for (int e = e0; e < e1; ++e) s = fma(a.cv[e], a.x[a.ci[e]], s);
        }
        r[k] = in ? a.b[i] - s : 0.0;
        z[k] = jac ? d[k] * r[k] : r[k];
        if (CL) {
            if (t + k * nt < a.rows) {
                sz[t + k * nt] = z[k];
                sq[t + k * nt] = 0.0;
            }
        } else if (in) {
            __stcg(a.z + i, z[k]);
            __stcg(a.p0 + i, 0.0);  // the old p of the first iteration
        }
        s0 = fma(r[k], r[k], s0);
        s1 = fma(z[k], r[k], s1);
    }
    sa[t] = s0;
    sb[t] = s1;
    exchange(true, [&](int w, double g) {
        if (w == 0) s_rnorm = sqrt(g);
    });
    __syncthreads();
    double rz = s_sum[1];
    // the unpreconditioned form starts with r_norm = norm2(r) and it = 1; the preconditioned one with 9e9 and 0
    double rnorm = jac ? 9e9 : s_rnorm;
    long long it = jac ? 0 : 1;
    double beta = 0.0, alpha = 0.0;
    int reason = 0, conv = 0;
    bool stop = s_late != 0;
    if (!jac && s_sum[0] == 0.0) {  // rho = dot(r, r); if (rho == 0.) { converged = true; break; }
        stop = true;
        it = 0;
        reason = UGPU_CONVERGED_FNORM_ABS;
        conv = 1;
    }
    double *pold = a.p1, *pnew = a.p0;
    while (!stop) {
        // p = z + beta p, Ap, (p, Ap)
        if constexpr (CL) {
            double *const swap = sp;
            sp = sq;
            sq = swap;
        } else {
            double *const swap = pold;
            pold = pnew;
            pnew = swap;
        }
        double *const own = CL ? sq : sp;  // the CTA's new p
#pragma unroll
        for (int k = 0; k < RPT; ++k) {
            const int l = t + k * nt;
            p[k] = fma(beta, p[k], z[k]);
            if (row0 + l < row1) {
                own[l] = p[k];
                if (!CL) __stcg(pnew + row0 + l, p[k]);
            }
        }
        auto read_remote = [&](int c, double &zc, double &pc) {
            if constexpr (CL) {
                const uint32_t at = 8u * uint32_t(c & 0xffff), r = uint32_t(c) >> 16;
                zc = ld_cluster(uint32_t(__cvta_generic_to_shared(sz)) + at, r);
                pc = ld_cluster(uint32_t(__cvta_generic_to_shared(sp)) + at, r);
            } else {
                zc = __ldcg(a.z + c);
                pc = __ldcg(pold + c);
            }
        };
        s0 = 0.0;
        if constexpr (REG) {
            // the other CTAs' entries are on their way while the CTA's own p settles
            double hz[RPT][kRegRow], hp[RPT][kRegRow];
#pragma unroll
            for (int k = 0; k < RPT; ++k)
#pragma unroll
                for (int e = 0; e < kRegRow; ++e) {
                    hz[k][e] = hp[k][e] = 0.0;
                    if (mc[k][e] < -1) read_remote(-2 - mc[k][e], hz[k][e], hp[k][e]);
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
                    else v = fma(beta, hp[k][e], hz[k][e]);
                    s = fma(mv[k][e], v, s);
                }
                q[k] = s;
                s0 = fma(p[k], s, s0);
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
                            double zc, pc;
                            read_remote(remote(c), zc, pc);
                            v = fma(beta, pc, zc);
                        }
                        s = fma(__ldg(a.cv + e), v, s);
                    }
                }
                q[k] = s;
                s0 = fma(p[k], s, s0);
            }
        }
        sa[t] = s0;
        exchange(false, [&](int, double pq) { s_alpha = rz / pq; });
        __syncthreads();
        const double pAp = s_sum[0];
        alpha = s_alpha;
        if (s_late) break;
        if (!jac && pAp == 0.0) {  // if (dot_pq == 0.) { converged = true; break; }
            reason = UGPU_CONVERGED_FNORM_ABS;
            conv = 1;
            break;
        }
        if (isinf(alpha) || isnan(alpha)) {
            conv = rnorm <= a.atol;
            reason = conv ? UGPU_CONVERGED_FNORM_ABS : it >= a.max_it ? UGPU_DIVERGED_MAX_IT : UGPU_DIVERGED_NAN;
            break;
        }
        // r, z, (r, r), (z, r); x while the sums travel
        s0 = s1 = 0.0;
#pragma unroll
        for (int k = 0; k < RPT; ++k) {
            r[k] = r[k] - alpha * q[k];
            z[k] = jac ? d[k] * r[k] : r[k];
            const int i = row0 + t + k * nt;
            if (i < row1) {
                if (CL) sz[i - row0] = z[k];
                else __stcg(a.z + i, z[k]);
            }
            s0 = fma(r[k], r[k], s0);
            s1 = fma(z[k], r[k], s1);
        }
        sa[t] = s0;
        sb[t] = s1;
        exchange(true, [&](int w, double g) {
            if (w == 0) s_rnorm = sqrt(g);
            else s_beta = g / rz;
        });
#pragma unroll
        for (int k = 0; k < RPT; ++k) x[k] = x[k] + alpha * p[k];
        __syncthreads();
        if (s_late) break;
        rnorm = s_rnorm;
        beta = s_beta;
        rz = s_sum[1];
        if (rnorm <= a.atol) {
            reason = UGPU_CONVERGED_FNORM_ABS;
            conv = 1;
            break;
        }
        if (it >= a.max_it) {
            reason = UGPU_DIVERGED_MAX_IT;
            conv = jac ? 0 : 1;  // the unpreconditioned form reports check_convergence()'s true
            break;
        }
        ++it;
        if (!jac && rz == 0.0) {
            reason = UGPU_CONVERGED_FNORM_ABS;
            conv = 1;
            break;
        }
    }
#pragma unroll
    for (int k = 0; k < RPT; ++k) {
        const int i = row0 + t + k * nt;
        if (i < row1) a.x[i] = x[k];
    }
    if (t == 0) {
        if (s_late) atomicExch(a.kflag, 1);
        if (blockIdx.x == 0) {
            CgDev *o = a.dev;
            o->rz = rz;
            o->alpha = alpha;
            o->beta = beta;
            o->rnorm = o->gnorm = rnorm;
            o->it = o->iterates = it;
            o->done = 1;
            o->reason = reason;
            o->converged = conv;
        }
    }
    __syncthreads();
    if (CL) cluster_barrier();  // no CTA leaves while another may still read its shared memory
}

}  // namespace

// Rows of at most eight entries: up to four rows per thread (311,296 rows; 18 us per iteration against 29 in
// separate kernels).  Longer ones, gathered entry by entry from the matrix in memory, up to two rows per
// thread and 32 entries (random graph of 150,000 rows 26 against 33 us, but 45 against 38 at 200,000; 27-point
// Galerkin operator of 110,592 rows 26 against 31 us).
bool CgResident::fits(const Context &c, const Mat &A) {
    if (A.nrows < 1 || A.max_row <= 0) return false;
    const int64_t threads = int64_t(c.sms) * kThreads;
    return A.nrows <= threads * (A.max_row <= kRegRow ? kMaxRpt : 2) && A.max_row <= 32;
}

size_t CgResident::sum_bytes(const Context &c) { return 2 * GridExchange<1>::bytes(c.sms); }

bool CgResident::run(Context &c, const Mat &A, const double *b, double *x, const double *dinv, double *z, double *p0,
                     double *p1, void *sums, CgDev *dev, double atol, long long max_it) {
    const int64_t n = A.nrows;
    // One cluster of 16 CTAs up to kClusterRows rows; otherwise a CTA per SM.  At least 64 rows per CTA: below that
    // more CTAs only lengthen the exchanges.
    const bool cl = n <= kClusterRows && A.max_row <= kRegRow;
    int64_t G = std::min<int64_t>(cl ? 16 : c.sms, (n + 63) / 64);
    const int64_t rows = ((n + G - 1) / G + 31) / 32 * 32;
    G = (n + rows - 1) / rows;
    const int rpt = rows <= kThreads ? 1 : rows <= 2 * kThreads ? 2 : 4;
    const int nt = int(std::max<int64_t>(64, ((rows + rpt - 1) / rpt + 31) / 32 * 32));
    ResArgs a{};
    a.rp = A.rowptr.as<int32_t>();
    a.ci = A.colidx.as<int32_t>();
    a.cv = A.vals.as<double>();
    a.n = int(n);
    a.rows = int(rows);
    a.b = b;
    a.dinv = dinv;
    a.x = x;
    a.z = z;
    a.p0 = p0;
    a.p1 = p1;
    a.sums = static_cast<char *>(sums);
    a.dev = dev;
    a.kflag = c.d_kflags() + 2;
    a.atol = atol;
    a.max_it = max_it;
    UGPU_CUDA(cudaMemsetAsync(sums, 0, sum_bytes(c), c.stream));
    const bool reg = A.max_row <= kRegRow && rpt <= 2;
    const size_t smem = sizeof(double) * (size_t(rows) * (cl ? 3 : 1) + 2 * size_t(nt) +
                                          (cl ? 2 * ClusterExchange<1>::kDoubles : 0));
    // one cluster has at most kClusterRows / 16 = 384 rows per CTA
    void (*f)(ResArgs) = cl         ? k_cg_resident<1, true, true>
                         : rpt == 1 ? (reg ? k_cg_resident<1, true, false> : k_cg_resident<1, false, false>)
                         : rpt == 2 ? (reg ? k_cg_resident<2, true, false> : k_cg_resident<2, false, false>)
                                    : k_cg_resident<4, false, false>;
    return launch_resident(c, f, a, int(G), nt, smem, cl);
}

}  // namespace ugpu
