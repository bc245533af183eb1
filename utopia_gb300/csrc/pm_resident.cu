// PowerMethod::compute_max_eig (utopia/solvers/eigensolvers/utopia_PowerMethod.hpp:95-146) on the smaller levels of a
// hierarchy: all iterations in one kernel.
//
// In separate kernels an iteration is a product, a dot, the stop test and a scaling, launched up to max_it + 1
// times whether it has stopped or not: a four-level hierarchy under a 512^2 problem took 512 launches and 1.3 ms
// per set-up.  Here every thread owns one or two rows, an iteration is one exchange (gridsync.cuh), and it ends
// at its stop test.  y = A v is published in the buffer that the current product does not read, and another CTA's
// v_j is formed as scale y_j, the value the scaling kernel would have stored.
#include "abi_util.cuh"
#include "device_util.cuh"
#include "gridsync.cuh"
#include "pm_resident.cuh"

namespace ugpu {

namespace {

constexpr int kThreads = 512;
constexpr int kRegRow = 9;  // row entries kept in registers
constexpr int64_t kClusterRows = 6144;

struct PmArgs {
    const int32_t *rp, *ci;
    const double *cv;
    int n, rows;  // rows per CTA
    double *y0, *y1;  // y0: the start vector
    char *sums;
    double *lambda;
    int *kflag;
    double tol;
    long long max_it;
};

template <int RPT, bool REG, bool CL>
__global__ void __launch_bounds__(kThreads, 1) k_pm_resident(PmArgs a) {
    extern __shared__ double sh[];  // [rows] v, [blockDim.x] partials, CL: two sets of y [rows], the exchange's slots
    __shared__ unsigned long long s_part[1];
    __shared__ double s_norm, s_inv;
    __shared__ int s_late;
    const int t = threadIdx.x, nt = blockDim.x, lane = t & 31, warp = t >> 5;
    const int row0 = blockIdx.x * a.rows, row1 = min(a.n, row0 + a.rows);
    double *sv = sh, *part = sv + a.rows, *sy0 = part + nt, *sy1 = sy0 + (CL ? a.rows : 0);
    using Exchange = typename std::conditional<CL, ClusterExchange<1>, GridExchange<1>>::type;
    Exchange gx;
    if (t == 0) s_late = 0;
    if constexpr (CL) {
        gx.init(sy1 + a.rows, blockIdx.x, gridDim.x);
        if (t == 0) gx.init_barriers();
        __syncthreads();
        cluster_barrier();
    } else {
        gx.init(a.sums, int(gridDim.x));
    }
    double q[RPT];
    double mv[REG ? RPT : 1][kRegRow];
    int mc[REG ? RPT : 1][kRegRow];  // own column: its local row; another CTA's: -2 - remote(column); none: -1
    auto remote = [&](int c) { return CL ? (c / a.rows) << 16 | c % a.rows : c; };
#pragma unroll
    for (int k = 0; k < RPT; ++k) {
        const int lr = t + k * nt, i = row0 + lr;
        const bool in = i < row1;
        q[k] = in ? a.y0[i] : 0.0;
        if (CL && lr < a.rows) sy0[lr] = q[k];
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
    long long ex = 0;
    auto norm2 = [&]() {  // ||q|| over the grid and its inverse (one lane: a root and a division per thread would queue)
        double d = 0.0;
#pragma unroll
        for (int k = 0; k < RPT; ++k) d = fma(q[k], q[k], d);
        part[t] = d;
        __syncthreads();
        if (warp == 0) {
            const double s = warp_sum_of(part, nt);
            if (lane == 0) s_part[0] = dbits(s);
            __syncwarp();
            unsigned long long o[1];
            const bool ok = gx.exchange(ex, s_part, o);
            if (lane == 0) {
                s_norm = sqrt(bitsd(o[0]));
                s_inv = 1. / s_norm;
                if (!ok) s_late = 1;
            }
        }
        ++ex;
        __syncthreads();
    };
    const double *gy = a.y0;  // the published y of the current v = scale y
    double *gn = a.y1;
    double *cy = sy0, *cn = sy1;
    norm2();
    double scale = s_inv, lambda = 0.0, old = 0.0;
    for (long long it = 0; !s_late;) {
#pragma unroll
        for (int k = 0; k < RPT; ++k)
            if (t + k * nt < a.rows) sv[t + k * nt] = scale * q[k];
        __syncthreads();
        auto far = [&](int c) {
            if constexpr (CL)
                return scale * ld_cluster(uint32_t(__cvta_generic_to_shared(cy)) + 8u * uint32_t(c & 0xffff), uint32_t(c) >> 16);
            else
                return scale * __ldcg(gy + c);
        };
#pragma unroll
        for (int k = 0; k < RPT; ++k) {
            const int lr = t + k * nt, i = row0 + lr;
            double s = 0.0;
            if constexpr (REG) {
                double v[kRegRow];
#pragma unroll
                for (int e = 0; e < kRegRow; ++e) v[e] = mc[k][e] >= 0 ? sv[mc[k][e]] : mc[k][e] < -1 ? far(-2 - mc[k][e]) : 0.0;
#pragma unroll
                for (int e = 0; e < kRegRow; ++e)
                    if (mc[k][e] != -1) s = fma(mv[k][e], v[e], s);
            } else if (i < row1) {
                const int e1 = __ldg(a.rp + i + 1);
                for (int e = __ldg(a.rp + i); e < e1; ++e) {
                    const int c = __ldg(a.ci + e);
                    s = fma(__ldg(a.cv + e), c >= row0 && c < row1 ? sv[c - row0] : far(remote(c)), s);
                }
            }
            q[k] = s;
            if (i < row1) {
                if (CL) cn[lr] = s;
                else __stcg(gn + i, s);
            }
        }
        norm2();
        lambda = s_norm;
        ++it;
        if (fabs(old - lambda) < a.tol || it > a.max_it) break;
        old = lambda;
        scale = s_inv;
        {
            const double *const swap = gy;
            gy = gn;
            gn = const_cast<double *>(swap);
            double *const cswap = cy;
            cy = cn;
            cn = cswap;
        }
    }
    if (t == 0) {
        if (s_late) atomicExch(a.kflag, 1);
        if (blockIdx.x == 0) *a.lambda = lambda;
    }
    __syncthreads();
    if (CL) cluster_barrier();  // no CTA leaves while another may still read its shared memory
}

// An exchange whose other CTA never takes part (it waits at the cluster's barrier, or there is none): the wait runs out
template <bool CL>
__global__ void __launch_bounds__(32) k_lonely_exchange(char *sums, long long limit, int *kflag) {
    __shared__ double sh[ClusterExchange<1>::kDoubles];
    __shared__ unsigned long long part[1];
    using Exchange = typename std::conditional<CL, ClusterExchange<1>, GridExchange<1>>::type;
    Exchange gx;
    if constexpr (CL) {
        gx.init(sh, blockIdx.x, gridDim.x);
        if (threadIdx.x == 0) gx.init_barriers();
        __syncthreads();
        cluster_barrier();
    } else {
        gx.init(sums, 2);
    }
    gx.limit = limit;
    if (threadIdx.x == 0) part[0] = 0;
    __syncwarp();
    unsigned long long out[1];
    if (blockIdx.x == 0 && !gx.exchange(0, part, out) && threadIdx.x == 0) atomicExch(kflag, 1);
    if (CL) cluster_barrier();
}

}  // namespace

// Up to two rows per thread (155,648 rows) of at most 32 entries: random graphs of 2001 / 20,001 / 60,001 / 150,001 rows
// 6 / 7 / 10 / 34 us per iteration against 21 / 24 / 25 / 35 in separate kernels, 27 points 64,000 rows 13 / 28.
bool pm_resident_fits(const Context &c, const Mat &A) {
    return A.nrows >= 1 && A.max_row > 0 && A.max_row <= 32 && A.nrows <= int64_t(c.sms) * kThreads * 2;
}

size_t pm_resident_bytes(const Context &c) { return GridExchange<1>::bytes(c.sms); }

bool pm_resident(Context &c, const Mat &A, double *y0, double *y1, void *sums, double *lambda, double tol,
                 long long max_it) {
    const int64_t n = A.nrows;
    const bool reg = A.max_row <= kRegRow, cl = reg && n <= kClusterRows;
    int64_t G = std::min<int64_t>(cl ? 16 : c.sms, (n + 63) / 64);
    const int64_t rows = ((n + G - 1) / G + 31) / 32 * 32;
    G = (n + rows - 1) / rows;
    const int rpt = rows <= kThreads ? 1 : 2;
    const int nt = int(std::max<int64_t>(64, ((rows + rpt - 1) / rpt + 31) / 32 * 32));
    PmArgs a{};
    a.rp = A.rowptr.as<int32_t>();
    a.ci = A.colidx.as<int32_t>();
    a.cv = A.vals.as<double>();
    a.n = int(n);
    a.rows = int(rows);
    a.y0 = y0;
    a.y1 = y1;
    a.sums = static_cast<char *>(sums);
    a.lambda = lambda;
    a.kflag = c.d_kflags() + 2;
    a.tol = tol;
    a.max_it = max_it;
    UGPU_CUDA(cudaMemsetAsync(sums, 0, pm_resident_bytes(c), c.stream));
    const size_t smem = sizeof(double) * (size_t(rows) * (cl ? 3 : 1) + size_t(nt) + (cl ? ClusterExchange<1>::kDoubles : 0));
    void (*f)(PmArgs) = cl         ? k_pm_resident<1, true, true>
                        : rpt == 1 ? (reg ? k_pm_resident<1, true, false> : k_pm_resident<1, false, false>)
                                   : (reg ? k_pm_resident<2, true, false> : k_pm_resident<2, false, false>);
    return launch_resident(c, f, a, int(G), nt, smem, cl);
}

}  // namespace ugpu

using namespace ugpu;

extern "C" int ugpu_test_exchange_wait_timeout(ugpu_ctx *ctx, int cluster, int64_t spin_cycles) {
    UGPU_ABI_BEGIN
    UGPU_REQUIRE(ctx);
    UGPU_CHECK(spin_cycles > 0 && spin_cycles <= 100000000ll, UGPU_ERR_ARG, "test wait limit: 1 .. 1e8 cycles");
    Context &c = ctx->impl;
    Buffer sums;
    sums.alloc(GridExchange<1>::bytes(2));
    UGPU_CUDA(cudaMemsetAsync(sums.ptr, 0, sums.bytes, c.stream));
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(cluster ? 2 : 1);
    cfg.blockDim = dim3(32);
    cfg.stream = c.stream;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = cfg.gridDim.x;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    char *p = static_cast<char *>(sums.ptr);
    const long long limit = spin_cycles;
    int *flag = c.d_kflags() + 2;
    if (cluster) UGPU_CUDA(cudaLaunchKernelEx(&cfg, k_lonely_exchange<true>, p, limit, flag));
    else UGPU_CUDA(cudaLaunchKernelEx(&cfg, k_lonely_exchange<false>, p, limit, flag));
    c.launches++;
    cudaStreamSynchronize(c.stream);  // before the buffer goes
    UGPU_ABI_END(ctx ? &ctx->impl : nullptr)
}
