// Dense FP64 coarse-level direct solver.
//
// Reference: the coarse solver of utopia::Multigrid (Multigrid::coarse_solve,
// utopia/solvers/multilevel/utopia_Multigrid.hpp:440-444), a PETSc Factorization
// (utopia/backend/petsc/solvers/linear/utopia_petsc_Factorization.hpp).
//
// Set-up: the Galerkin operator of the coarsest level is densified, factored (Cholesky,
// A = L L^T) and L inverted (Y = L^-1) by one recursion, and the explicit inverse
// A^-1 = Y^T Y is formed.  Every coarse solve is then one
// FP64 GEMV with A^-1, an L2-resident matrix for the coarse sizes of the hot path
// (1728^2 and 4096^2 doubles), instead of two latency-bound triangular sweeps.
// GB300's FP64 tensor rate is no higher than its FP64 FMA rate, so the set-up's large products run on
// the FP16 tensor cores by splitting (gemm64.cu) and the inverse is refined to FP64's accuracy entry by entry; the
// small products, the 64 x 64 diagonal blocks, and the set-ups that cannot be refined use the FP64 pipe.
#include <cmath>
#include <cstring>
#include <functional>

#include "abi_util.cuh"
#include "device_util.cuh"
#include "gemm64.cuh"

namespace ugpu {

namespace {

constexpr int NB = 64;  // Cholesky / inversion block size

// v 2^k by an integer addition to the exponent where that is exact
__device__ __forceinline__ double scale_pow2(double v, int k) {
    const long long b = __double_as_longlong(v);
    const int e = int(b >> 52) & 0x7ff;
    if (e == 0 || e == 0x7ff || e + k < 1 || e + k > 0x7fe) return ldexp(v, k);
    return __longlong_as_double(b + k * (1ll << 52));
}

// Half exponents of the diagonal: with D = diag(2^-h_i) the diagonal of D A D lies in [1, 4).  The products of
// the factorisation carry their operand rows as fixed-point numbers under one scale per row; on D A D no
// entry reaches 4, so rows and columns of very different size cannot drown one another.  Scaling by powers
// of two is exact.
template <class V>
__global__ void k_half_exponents(const int32_t *rp, const int32_t *ci, const V *cv, int64_t n, int *h) {
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
        int e = 0;
        for (int32_t k = rp[i]; k < rp[i + 1]; ++k) {
            if (ci[k] != i) continue;
            const double d = cvt<double>(cv[k]);
            if (d > 0.0 && !isinf(d)) e = ilogb(d);
        }
        h[i] = e >> 1;
    }
}

// the dense form of D A D
template <class V>
__global__ void k_densify(const int32_t *rp, const int32_t *ci, const V *cv, int64_t n, const int *h, double *D) {
    for (int64_t i = blockIdx.x; i < n; i += gridDim.x) {
        for (int64_t c = threadIdx.x; c < n; c += blockDim.x) D[i * n + c] = 0.0;
        __syncthreads();
        for (int32_t k = rp[i] + threadIdx.x; k < rp[i + 1]; k += blockDim.x)
            D[i * n + ci[k]] = scale_pow2(cvt<double>(cv[k]), -h[i] - h[ci[k]]);
        __syncthreads();
    }
}

// Cholesky of the kb x kb diagonal block at (k0, k0) of A (A = L L^T) and Y = L^-1, into Y's block.  Column c
// of the remaining block and column c of the inverse share one array: entry (i, c) is A's remainder until
// column c is eliminated, the inverse's entry after.  Eight columns at a time:
//   1. one warp eliminates the 8 x 8 pivot block in registers (as L D L^T, the roots at the end) and inverts
//      its factor (Y8);
//   2. L's panel = A's panel Y8^T, the inverse's 8 rows = Y8 times what they hold;
//   3. the rows below take the rank-8 update; warp 0 updates only the next pivot block and goes on to its
//      elimination, a chain of dependent operations, while the other warps update the rest.
// One CTA; bound by the FP64 pipe of one SM (87 k FMAs at two per clock, about 21 us) and what is left of the
// chain: 55 to 59 us (6 us more with the other warps spread over all four schedulers).  Eliminating column by column with all
// warps queued the chain's operations behind the updates in that pipe (80-90 us); separate factorisation and
// inversion kernels took 93 and 145 us.
constexpr int PB = 8;
__global__ void __launch_bounds__(256) k_chol_inv_block(const double *A, double *Y, int64_t n, int64_t k0, int kb,
                                                        int *bad) {
    __shared__ double s_a[NB][NB + 1];   // the shared array (lower triangle)
    __shared__ double s_l[NB][PB + 1];   // L's panel
    __shared__ double s_z[PB][NB + 1];   // the inverse's rows of the panel (final)
    __shared__ double s_y[PB][PB + 1];   // Y8
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    for (int e = t; e < NB * NB; e += 256) {
        const int i = e / NB, c = e % NB;
        s_a[i][c] = (i < kb && c <= i) ? A[(k0 + i) * n + k0 + c] : (i == c ? 1.0 : 0.0);
    }
    __syncthreads();
    // step 1 in one warp: lane l holds row l / 4, columns 2 (l % 4) and 2 (l % 4) + 1 of the pivot block
    const int pr = lane >> 2, pc = (lane & 3) * 2;
    auto pivots = [&](double m0, double m1) {
        double mine = 1.0;  // d of this lane's row
#pragma unroll
        for (int j = 0; j < PB; ++j) {
            const double mj = (j & 1) ? m1 : m0;  // column j where lane % 4 = j / 2
            double d = __shfl_sync(0xffffffffu, mj, j * 4 + (j >> 1));
            const double l = __shfl_sync(0xffffffffu, mj, (lane & 28) + (j >> 1));  // a_ij
            // raw_c: a_cj for c > j, 1 for c = j, z_jc for c < j
            const double a0 = __shfl_sync(0xffffffffu, mj, pc * 4 + (j >> 1));
            const double a1 = __shfl_sync(0xffffffffu, mj, (pc + 1) * 4 + (j >> 1));
            const double z0 = __shfl_sync(0xffffffffu, m0, j * 4 + (lane & 3));
            const double z1 = __shfl_sync(0xffffffffu, m1, j * 4 + (lane & 3));
            if (!(d > 0.0)) {
                if (lane == 0) atomicOr(bad, 1);
                d = 1.0;
            }
            // (l raw) beside the reciprocal: one operation follows it
            const double p0 = -l * (pc > j ? a0 : pc == j ? 1.0 : z0);
            const double p1 = -l * (pc + 1 > j ? a1 : pc + 1 == j ? 1.0 : z1);
            const double inv = 1.0 / d;
            if (pr > j) {
                m0 = fma(p0, inv, pc == j ? 0.0 : m0);
                m1 = fma(p1, inv, pc + 1 == j ? 0.0 : m1);
            } else if (pr == j) {
                mine = d;
                if (pc == j) m0 = 1.0;
                if (pc + 1 == j) m1 = 1.0;
            }
        }
        const double r = 1.0 / sqrt(mine);
        s_y[pr][pc] = pc <= pr ? m0 * r : 0.0;
        s_y[pr][pc + 1] = pc + 1 <= pr ? m1 * r : 0.0;
    };
    if (w == 0) pivots(s_a[pr][pc], s_a[pr][pc + 1]);
    __syncthreads();
    for (int J = 0; J < NB; J += PB) {
        // step 2: thread t takes row (or column) t / 4 and the outputs q = t % 4 and 7 - q (9 products together)
        {
            const int i = t >> 2, qa = t & 3, qb = PB - 1 - qa;
            const bool below = i >= J + PB;
            double x[PB];
#pragma unroll
            for (int k = 0; k < PB; ++k) x[k] = below ? s_a[i][J + k] : s_a[J + k][i];
            double ra = 0.0, rb = 0.0;
            if (i < J || below) {
#pragma unroll
                for (int k = 0; k < PB; ++k) {
                    if (k < PB / 2 && k <= qa) ra = fma(s_y[qa][k], x[k], ra);
                    if (k <= qb) rb = fma(s_y[qb][k], x[k], rb);
                }
            } else {  // the panel's own columns: Y8
                ra = s_y[qa][i - J];
                rb = s_y[qb][i - J];
            }
            if (below) {
                s_l[i][qa] = ra;
                s_l[i][qb] = rb;
            } else {
                s_z[qa][i] = ra;
                s_z[qb][i] = rb;
                if (J + qa < kb && i <= J + qa) Y[(k0 + J + qa) * n + k0 + i] = ra;
                if (J + qb < kb && i <= J + qb) Y[(k0 + J + qb) * n + k0 + i] = rb;
            }
        }
        __syncthreads();
        // step 3
        if (J + PB < NB) {
            const int I = J + PB;  // the next panel
            if (w == 0) {
                double m0 = s_a[I + pr][I + pc], m1 = s_a[I + pr][I + pc + 1];
#pragma unroll
                for (int q = 0; q < PB; ++q) {
                    const double l = s_l[I + pr][q];
                    m0 = fma(-l, s_l[I + pc][q], m0);
                    m1 = fma(-l, s_l[I + pc + 1][q], m1);
                }
                pivots(m0, m1);
            } else if (w & 3) {
                // the warps of the other three schedulers: what shares warp 0's would queue its chain behind them
                for (int i = I + (w >> 2) * 3 + (w & 3) - 1; i < NB; i += 6) {
                    double l[PB];
#pragma unroll
                    for (int q = 0; q < PB; ++q) l[q] = s_l[i][q];
                    for (int c = lane; c <= i; c += 32) {
                        if (i < I + PB && c >= I) continue;  // the next pivot block
                        double m = (c >= J && c < I) ? 0.0 : s_a[i][c];
                        const bool inv = c < I;
#pragma unroll
                        for (int q = 0; q < PB; ++q) m = fma(-l[q], inv ? s_z[q][c] : s_l[c][q], m);
                        s_a[i][c] = m;
                    }
                }
            }
            __syncthreads();
        }
    }
}

// The result from its lower triangle, with the scaling of the operator undone: the inverse
// (D A D)^-1 -> A^-1 = D (D A D)^-1 D with its upper triangle mirrored (rows scaled too), or L^-1 -> L^-1 D with its
// transpose in the upper triangle.  h null: mirrored as it is.  add (may be null) is added to the lower triangle
// first.  32 x 32 tiles through shared memory, so that both triangles are written in whole lines.
__global__ void __launch_bounds__(256) k_unscale_mirror(double *A, const double *add, int64_t n, const int *h,
                                                        int rows_too) {
    if (blockIdx.x > blockIdx.y) return;
    __shared__ double s[32][33];
    const int64_t i0 = 32 * int64_t(blockIdx.y), j0 = 32 * int64_t(blockIdx.x);
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    for (int r = ty; r < 32; r += 8) {
        const int64_t i = i0 + r, j = j0 + tx;
        double v = 0.0;
        if (i < n && j <= i) {
            v = A[i * n + j];
            if (add) v += add[i * n + j];
            if (h) v = scale_pow2(v, -h[j] - (rows_too ? h[i] : 0));
            A[i * n + j] = v;
        }
        s[r][tx] = v;
    }
    __syncthreads();
    for (int r = ty; r < 32; r += 8) {
        const int64_t i = j0 + r, j = i0 + tx;  // the mirrored entry (i, j), j > i
        if (j < n && j > i) A[i * n + j] = s[tx][r];
    }
}

// The entries of D A D with both triangles taken from the lower one, as the factorisation takes them; a warp per row.
// *one_sided: some entry of the lower triangle has no place in the upper one.
template <class V>
__global__ void __launch_bounds__(kBlock) k_symmetric_values(const int32_t *rp, const int32_t *ci, const V *cv, int64_t n,
                                                             const int *h, double *sv, int *one_sided) {
    const int lane = threadIdx.x & 31;
    const int64_t nw = int64_t(gridDim.x) * blockDim.x / 32;
    for (int64_t i = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) / 32; i < n; i += nw)
        for (int32_t k = rp[i] + lane; k < rp[i + 1]; k += 32) {
            const int32_t c = ci[k];
            int32_t e = k;
            if (c != i) {
                const int32_t e1 = rp[c + 1];
                for (e = rp[c]; e < e1 && ci[e] != i; ++e) {
                }
                if (e == e1) e = -1;
            }
            if (c < i && e < 0) atomicOr(one_sided, 1);
            const int32_t from = c <= i ? k : e;
            sv[k] = from < 0 ? 0.0 : scale_pow2(cvt<double>(cv[from]), -h[i] - h[c]);
        }
}

// |v| as binary32 by truncation; 0 below its normal numbers, infinity above them and for NaN
__device__ __forceinline__ float abs32(double v) {
    const uint32_t h = uint32_t(__double2hiint(v)) & 0x7fffffffu;
    if (h < (897u << 20)) return 0.0f;
    if (h >= (1150u << 20)) return __int_as_float(0x7f800000);
    return __uint_as_float(__funnelshift_l(uint32_t(__double2loint(v)), h - (896u << 20), 3));
}

// R = I - S X and *worst = max |R_kj| / (|S| |X|)_kj (bits of a binary32; infinity where that is no number).  A CTA takes
// 512 columns of one row, lanes along the row.  EXACT: the sums in twice FP64's precision (Ogita, Rump and Oishi,
// "Accurate sum and dot product", 2005: error-free products and additions), ten FP64 operations for one.
template <bool EXACT>
__global__ void __launch_bounds__(256) k_inverse_residual(const int32_t *rp, const int32_t *ci, const double *sv, int64_t n,
                                                          const double *X, double *R, unsigned int *worst) {
    const int64_t i = blockIdx.y;
    const int64_t j0 = int64_t(blockIdx.x) * 512 + threadIdx.x;
    const int32_t e0 = rp[i], e1 = rp[i + 1];
    float bad = 0.0f;
    double r[2], low[2] = {0.0, 0.0};
    float size[2] = {0.0f, 0.0f};
#pragma unroll
    for (int q = 0; q < 2; ++q) r[q] = j0 + 256 * q == i ? 1.0 : 0.0;
#pragma unroll 4
    for (int32_t e = e0; e < e1; ++e) {
        const double a = __ldg(sv + e);
        const double *x = X + int64_t(__ldg(ci + e)) * n;
        const float a32 = abs32(a);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const double v = j0 + 256 * q < n ? __ldg(x + j0 + 256 * q) : 0.0;
            if constexpr (EXACT) {
                const double p = -a * v, pe = fma(-a, v, -p);
                const double s = r[q] + p, b = s - r[q];
                low[q] += ((r[q] - (s - b)) + (p - b)) + pe;
                r[q] = s;
            } else {
                r[q] = fma(-a, v, r[q]);
            }
            size[q] = fmaf(a32, abs32(v), size[q]);
        }
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        if (j0 + 256 * q >= n) continue;
        const double v = EXACT ? r[q] + low[q] : r[q];
        R[i * n + j0 + 256 * q] = v;
        const float v32 = abs32(v);
        if (v32 > 0.0f) {
            const float w = __fdividef(v32, size[q]);
            bad = fmaxf(bad, w >= 0.0f && size[q] < 1e37f && v32 < 1e37f ? w : __int_as_float(0x7f800000));
        }
    }
    const unsigned int m = __reduce_max_sync(0xffffffffu, __float_as_uint(bad));
    if ((threadIdx.x & 31) == 0 && m) atomicMax(worst, m);
}

__global__ void k_zero(double *p, int64_t m) {
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < m; i += int64_t(gridDim.x) * blockDim.x)
        p[i] = 0.0;
}

// x = Ainv * r, one CTA per row (the coarse matrix has only a few thousand rows, so a warp
// per row would leave each warp a long chain of dependent load rounds); the matrix and the
// vectors share the type T (the FP64 inverse for FP64 vectors, its FP32 copy for FP32).
// Rows are read as 16-byte vectors when n and the pointers allow it.
constexpr int kGemvThreads = 256;
template <class T>
__global__ void __launch_bounds__(kGemvThreads) k_gemv(const T *M, int64_t n, const T *r, T *x, const int *done,
                                                       int vec) {
    if (done && *done) return;
    constexpr int V = 16 / sizeof(T);  // elements per 16-byte vector
    using Vec = typename std::conditional<sizeof(T) == 8, double2, float4>::type;
    __shared__ T part[kGemvThreads / 32];
    for (int64_t i = blockIdx.x; i < n; i += gridDim.x) {
        const T *row = M + i * n;
        T s = T(0);
        if (vec) {
            const Vec *rv = reinterpret_cast<const Vec *>(row);
            const Vec *xv = reinterpret_cast<const Vec *>(r);
            for (int64_t c = threadIdx.x; c < n / V; c += kGemvThreads) {
                const Vec a = __ldg(rv + c), b = __ldg(xv + c);
                const T *pa = reinterpret_cast<const T *>(&a);
                const T *pb = reinterpret_cast<const T *>(&b);
#pragma unroll
                for (int q = 0; q < V; ++q) s = fma(pa[q], pb[q], s);
            }
        } else {
            for (int64_t c = threadIdx.x; c < n; c += kGemvThreads) s = fma(__ldg(row + c), __ldg(r + c), s);
        }
        s = warp_sum(s);
        if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
        __syncthreads();
        if (threadIdx.x < 32) {
            T t = threadIdx.x < kGemvThreads / 32 ? part[threadIdx.x] : T(0);
            t = warp_sum(t);
            if (threadIdx.x == 0) x[i] = t;
        }
        __syncthreads();
    }
}

}  // namespace

void DenseCholesky::make_fp32_inverse() {
    UGPU_CHECK(!tri, UGPU_ERR_UNSUPPORTED, "coarse solver: no FP32 inverse above the factored-inverse size");
    Ainv32.alloc(sizeof(float) * std::max<int64_t>(n * n, 1));
    if (n) launch_convert(*ctx, Ainv.ptr, UGPU_F64, Ainv32.ptr, UGPU_F32, n * n);
}

// Row count above which the products run on the tensor cores (7 points: 512 rows 0.88 ms against 0.92 with FP64
// multiply-adds, 729 rows 1.43 / 1.76, 1728 rows 3.8 / 11.4, 4096 rows 14.0 / 74.6; 343 rows 0.64 / 0.62).
constexpr int64_t kSplitMin = 512;
// max |R| / (|S| |X|) of an inverse X (R = I - S X) up to which X needs no correction, in units of sqrt(n) eps (FP64
// multiply-adds left 0.48 to 17 of them on 60 coarse operators of 528 to 4096 rows, the median 0.7), and up to
// which a correction by an exact residual is the last one.
constexpr double kSettled = 0.5, kLast = 0x1p-40;
constexpr int kExactSteps = 4;

bool DenseCholesky::factor(const Mat &A) {
    UGPU_CHECK(A.nrows == A.ncols, UGPU_ERR_ARG, "coarse solver: square matrix required");
    ctx = A.ctx;
    n = A.nrows;
    UGPU_CHECK(n <= 16384, UGPU_ERR_UNSUPPORTED, "coarse solver: dense size limited to 16384");
    tri = n > kDenseTriMin;
    // Split products on the tensor cores where the inverse can be refined: formed explicitly, by a sparse operator
    // (the residual's n nnz FMAs stay below a quarter of the inverse's).  What they call indefinite or what
    // does not settle is decided by FP64 multiply-adds.
    if (n > kSplitMin && !tri && A.nnz <= n * n / 8 && invert(A, false)) return true;
    return invert(A, true);
}

// fma: FP64 multiply-adds throughout.  Otherwise the large products are split ones, each accurate to rounding in its
// rows' maxima only: small entries of the inverse (a decaying row, a jump in the coefficients) are lost below them.
// So X is refined, X + X (I - S X): the residual carries every entry's relative error, whatever its size, and the
// correction is small beside X.  One correction, which the residual of the result has to confirm; where it does
// not, corrections by exact residuals.  Worst relative error of an entry, operators
// of 1000 rows, FP64 multiply-adds / split / refined: Poisson 4e-15 / 7e-13 / 1e-15, lognormal sigma 1
// 4e-15 / 1e-11 / 1e-15, sigma 4 1e-14 / 2e-6 / 2e-16, coefficients 1 and 1e8 5e-15 / 1 / 3e-16.
bool DenseCholesky::invert(const Mat &A, bool fma) {
    Context &c = *A.ctx;
    L.alloc(sizeof(double) * std::max<int64_t>(n * n, 1));
    Ainv.alloc(sizeof(double) * std::max<int64_t>(n * n, 1));
    Ainv32.release();
    if (n == 0) return true;
    double *Lp = L.as<double>();
    double *Y = Ainv.as<double>();  // holds L^-1 first
    const int32_t *rp = A.rowptr.as<int32_t>(), *ci = A.colidx.as<int32_t>();
    Buffer hx;  // half exponents of the diagonal
    hx.alloc(sizeof(int) * size_t(n));
    const dim3 tiles(unsigned((n + 31) / 32), unsigned((n + 31) / 32));
    Buffer state;  // [0] not definite, [1] an entry without its mirror image, [2] the residual's measure
    state.alloc(3 * sizeof(int));
    UGPU_CUDA(cudaMemsetAsync(state.ptr, 0, 3 * sizeof(int), c.stream));
    int *bad = state.as<int>();
    Buffer sv;  // the entries of D A D
    if (!fma) sv.alloc(sizeof(double) * size_t(std::max<int64_t>(A.nnz, 1)));
    auto dens = [&](auto tag) {
        using V = decltype(tag);
        k_half_exponents<V><<<stream_grid(c, n), kBlock, 0, c.stream>>>(rp, ci, A.vals.as<V>(), n, hx.as<int>());
        k_densify<V><<<int(std::min<int64_t>(n, 4096)), 256, 0, c.stream>>>(rp, ci, A.vals.as<V>(), n, hx.as<int>(), Lp);
        c.launches += 2;
        if (fma) return;
        k_symmetric_values<V><<<stream_grid(c, 32 * n), kBlock, 0, c.stream>>>(rp, ci, A.vals.as<V>(), n, hx.as<int>(),
                                                                              sv.as<double>(), bad + 1);
        c.launches++;
    };
    if (A.vdtype == UGPU_F64) dens(double{});
    else if (A.vdtype == UGPU_F32) dens(float{});
    else dens(__nv_bfloat16{});
    UGPU_LAUNCH_CHECK();
    // Factorisation and inversion by recursive halving at multiples of NB: with A11 = L11 L11^T and
    // Y11 = L11^-1 known, L21 = A21 Y11^T, A22 -= L21 L21^T, then the same for A22, and
    // Y21 = -Y22 (L21 Y11).  Every product is a GEMM of the current half's size (gemm64.cu), the
    // triangular factors' zero parts left out; L21 Y11 takes A21's place (L itself is not needed once Y is).
    // With the inverse, before its refinement: 4096 rows 10.6 ms, 1728 rows 3.3 ms.
    k_zero<<<stream_grid(c, n * n), kBlock, 0, c.stream>>>(Y, n * n);
    c.launches++;
    Buffer T, scales;
    T.alloc(sizeof(double) * size_t(std::max<int64_t>((n / 2 + NB) * (n / 2 + NB), 1)));
    scales.alloc(sizeof(uint32_t) * 2 * size_t(n));
    double *Tp = T.as<double>();
    std::function<void(int64_t, int64_t)> chol_inv = [&](int64_t r0, int64_t m) {
        if (m <= NB) {
            k_chol_inv_block<<<1, 256, 0, c.stream>>>(Lp, Y, n, r0, int(m), bad);
            c.launches++;
            return;
        }
        const int64_t h = ((m / 2 + NB - 1) / NB) * NB, m2 = m - h;  // 0 < h < m
        double *A21 = Lp + (r0 + h) * n + r0, *A22 = A21 + h;
        const double *Y11 = Y + r0 * n + r0, *Y22 = Y + (r0 + h) * n + r0 + h;
        chol_inv(r0, h);
        Gemm64 g;
        g.fma = fma;
        g.M = int(m2), g.N = int(h), g.K = int(h);  // T = L21 = A21 Y11^T
        g.A = A21, g.a_row = n, g.a_k = 1;
        g.B = Y11, g.b_row = n, g.b_k = 1;
        g.C = Tp, g.ldc = h;
        g.flags = kGemmKToN;
        gemm64(c, g, scales);
        g.N = int(m2);  // A22 -= T T^T, the lower triangle
        g.negate = g.add = true;
        g.A = Tp, g.a_row = h;
        g.B = Tp, g.b_row = h;
        g.C = A22, g.ldc = n;
        g.flags = kGemmLower;
        gemm64(c, g, scales);
        g.N = int(h);  // A21 = T Y11
        g.negate = g.add = false;
        g.B = Y11, g.b_row = 1, g.b_k = n;
        g.C = A21, g.ldc = n;
        g.flags = kGemmKFromN;
        gemm64(c, g, scales);
        chol_inv(r0 + h, m2);
        g.K = int(m2);  // Y21 = -Y22 A21
        g.negate = true;
        g.A = Y22, g.a_row = n, g.a_k = 1;
        g.B = A21, g.b_row = 1, g.b_k = n;
        g.C = Y + (r0 + h) * n + r0;
        g.flags = kGemmKToM;
        gemm64(c, g, scales);
    };
    chol_inv(0, n);
    UGPU_LAUNCH_CHECK();
    int hs[3] = {0, 0, 0};
    auto read_state = [&] {
        UGPU_CUDA(cudaMemcpyAsync(hs, state.ptr, sizeof(hs), cudaMemcpyDeviceToHost, c.stream));
        c.check_kernel_flags();
    };
    auto mirror = [&](double *M, const double *add, const int *h, int rows_too) {
        k_unscale_mirror<<<tiles, 256, 0, c.stream>>>(M, add, n, h, rows_too);
        c.launches++;
        UGPU_LAUNCH_CHECK();
    };
    tmp_d.ensure(sizeof(double) * size_t(n));
    if (tri) {  // Y in the lower triangle, Y^T in the upper one
        read_state();
        if (hs[0]) return false;
        mirror(Y, nullptr, hx.as<int>(), 0);
        UGPU_CUDA(cudaStreamSynchronize(c.stream));
        return true;
    }
    // A^-1 = Y^T Y (stored in L's buffer, then swapped): the lower triangle's tiles, then mirrored
    // (the product is symmetric bit for bit: (i, j) and (j, i) sum the same products in one order)
    Gemm64 g;
    g.fma = fma;
    g.M = g.N = g.K = int(n);
    g.A = Y, g.a_row = 1, g.a_k = n;
    g.B = Y, g.b_row = 1, g.b_k = n;
    g.C = Lp, g.ldc = n;
    g.flags = kGemmLower | kGemmKFromM | kGemmKFromN;
    gemm64(c, g, scales);
    if (fma) {
        mirror(Lp, nullptr, hx.as<int>(), 1);
        read_state();
        if (hs[0]) return false;
    } else {
        Buffer correction;
        correction.alloc(sizeof(double) * size_t(n * n));
        mirror(Lp, nullptr, nullptr, 0);
        g.A = Lp, g.a_row = n, g.a_k = 1;  // X R, R in Y's place
        g.C = correction.as<double>();
        g.flags = kGemmLower;
        const dim3 rows(unsigned((n + 511) / 512), unsigned(n));
        auto residual = [&](bool exact) {
            UGPU_CUDA(cudaMemsetAsync(bad + 2, 0, sizeof(int), c.stream));
            auto *kernel = exact ? k_inverse_residual<true> : k_inverse_residual<false>;
            kernel<<<rows, 256, 0, c.stream>>>(rp, ci, sv.as<double>(), n, Lp, Y, reinterpret_cast<unsigned int *>(bad + 2));
            c.launches++;
            UGPU_LAUNCH_CHECK();
            read_state();
            float worst;
            memcpy(&worst, &hs[2], sizeof(worst));
            return double(worst);
        };
        auto correct = [&] {
            gemm64(c, g, scales);
            mirror(Lp, correction.as<double>(), nullptr, 0);
        };
        double worst = residual(false);
        if (hs[0] || hs[1] || !(worst < HUGE_VAL)) return false;
        correct();
        if (!(residual(false) <= kSettled * std::sqrt(double(n)) * 0x1p-52))
            for (int k = 0;; ++k) {
                const double before = worst;
                worst = residual(true);
                if (!(worst < 0.25 * before) || k == kExactSteps) return false;
                correct();
                if (worst <= kLast) break;
            }
        mirror(Lp, nullptr, hx.as<int>(), 1);
        c.check_kernel_flags();
    }
    std::swap(L, Ainv);  // Ainv now holds the inverse
    return true;
}

// x = Ainv * r with the FP64 inverse, one warp per row: the row streams through 16-byte loads
// spread over the lanes into four independent FP64 partial sums per lane, reduced by shuffles.
// r and x are FP64, or FP32 (the mixed V-cycle: r converted exactly, x rounded once).  A CTA per
// row left most of the grid waiting on its block reductions (1728 rows: 21 us for 3 M FMAs).
template <class VT>
__device__ __forceinline__ double2 gemv_r2(const VT *r, int64_t j) {
    if constexpr (sizeof(VT) == 8) {
        return __ldg(reinterpret_cast<const double2 *>(r) + j);
    } else {
        const float2 t = __ldg(reinterpret_cast<const float2 *>(r) + j);
        return make_double2(f2d_bits(t.x), f2d_bits(t.y));
    }
}
template <class VT>
__global__ void __launch_bounds__(256) k_gemv64_warp(const double *M, int64_t n, const VT *r, VT *x,
                                                     const int *done, int vec) {
    if (done && *done) return;
    const int lane = threadIdx.x & 31;
    const int64_t nw = (int64_t(gridDim.x) * blockDim.x) >> 5;
    for (int64_t i = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) >> 5; i < n; i += nw) {
        const double *row = M + i * n;
        double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
        if (vec) {  // n even; row and r aligned for pair loads
            const double2 *rv = reinterpret_cast<const double2 *>(row);
            const int64_t n2 = n >> 1;
            int64_t c = lane;
            for (; c + 32 < n2; c += 64) {
                const double2 a = __ldg(rv + c), b = __ldg(rv + c + 32);
                const double2 ra = gemv_r2(r, c), rb = gemv_r2(r, c + 32);
                s0 = fma(a.x, ra.x, s0);
                s1 = fma(a.y, ra.y, s1);
                s2 = fma(b.x, rb.x, s2);
                s3 = fma(b.y, rb.y, s3);
            }
            if (c < n2) {
                const double2 a = __ldg(rv + c), ra = gemv_r2(r, c);
                s0 = fma(a.x, ra.x, s0);
                s1 = fma(a.y, ra.y, s1);
            }
        } else {
            for (int64_t c = lane; c < n; c += 32) s0 = fma(__ldg(row + c), cvt<double>(__ldg(r + c)), s0);
        }
        const double s = warp_sum((s0 + s1) + (s2 + s3));
        if (lane == 0) x[i] = cvt<VT>(s);
    }
}

// The same product for coarse levels whose right-hand side fits shared memory: r is converted to
// FP64 once per CTA into shared memory, and each row is split over two warps (four rows per CTA),
// so every lane has only a few independent 16-byte row loads and the grid keeps enough of them
// in flight to stream the inverse.  Eight loads of a lane are in flight (r's and the rows'): 4096 rows 38 us, where
// four took 49 and the FP64 pipes need 27.
constexpr int kGemvSmemMax = 96 * 1024;  // bytes of r staged per CTA
template <class VT>
__global__ void __launch_bounds__(256) k_gemv64_split(const double *M, int64_t n, const VT *r, VT *x,
                                                      const int *done, int vec) {
    extern __shared__ __align__(16) double sr[];  // r in FP64
    __shared__ double part[8];
    if (done && *done) return;
    for (int64_t j0 = threadIdx.x; j0 < n; j0 += 8 * 256) {
        VT v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = j0 + u * 256 < n ? __ldg(r + j0 + u * 256) : VT(0);
#pragma unroll
        for (int u = 0; u < 8; ++u)
            if (j0 + u * 256 < n) sr[j0 + u * 256] = cvt<double>(v[u]);
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rl = warp >> 1, q = warp & 1;  // row of the four, half of the row
    for (int64_t i0 = 4 * int64_t(blockIdx.x); i0 < n; i0 += 4 * int64_t(gridDim.x)) {
        const int64_t i = i0 + rl;
        double s0 = 0.0, s1 = 0.0;
        if (i < n) {
            const double *row = M + i * n;
            if (vec) {  // n even, rows 16-byte aligned: pairs [q n2 / 4, (q + 1) n2 / 4)
                const int64_t n2 = n >> 1, c0 = q * n2 / 2, c1 = (q + 1) * n2 / 2;
                const double2 *rv = reinterpret_cast<const double2 *>(row);
                const double2 *xv = reinterpret_cast<const double2 *>(sr);
                for (int64_t k = c0 + lane; k < c1; k += 8 * 32) {
                    double2 a[8];
#pragma unroll
                    for (int u = 0; u < 8; ++u) a[u] = k + u * 32 < c1 ? __ldg(rv + k + u * 32) : make_double2(0.0, 0.0);
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        if (k + u * 32 >= c1) break;
                        const double2 b = xv[k + u * 32];
                        s0 = fma(a[u].x, b.x, s0);
                        s1 = fma(a[u].y, b.y, s1);
                    }
                }
            } else {
                const int64_t c0 = q * n / 2, c1 = (q + 1) * n / 2;
                for (int64_t k = c0 + lane; k < c1; k += 8 * 32) {
                    double a[8];
#pragma unroll
                    for (int u = 0; u < 8; ++u) a[u] = k + u * 32 < c1 ? __ldg(row + k + u * 32) : 0.0;
#pragma unroll
                    for (int u = 0; u < 8; ++u)
                        if (k + u * 32 < c1) s0 = fma(a[u], sr[k + u * 32], s0);
                }
            }
        }
        const double s = warp_sum(s0 + s1);
        if (lane == 0) part[warp] = s;
        __syncthreads();
        if (threadIdx.x < 4 && i0 + threadIdx.x < n) {
            const double *pp = part + 2 * threadIdx.x;
            x[i0 + threadIdx.x] = cvt<VT>(pp[0] + pp[1]);
        }
        __syncthreads();
    }
}

// One triangle of the tri form: out_i = sum over j <= i (LOWER) or j >= i of M[i][j] in_j, a warp per
// row (row segments are contiguous, the lanes' loads coalesced), four partial sums per lane.
template <class VI, class VO, bool LOWER>
__global__ void __launch_bounds__(256) k_gemv64_tri(const double *M, int64_t n, const VI *in, VO *out,
                                                    const int *done) {
    if (done && *done) return;
    const int lane = threadIdx.x & 31;
    const int64_t nw = (int64_t(gridDim.x) * blockDim.x) >> 5;
    for (int64_t i = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) >> 5; i < n; i += nw) {
        const double *row = M + i * n;
        const int64_t lo = LOWER ? 0 : i, hi = LOWER ? i + 1 : n;
        double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
        int64_t c = lo + lane;
        for (; c + 96 < hi; c += 128) {
            s0 = fma(__ldg(row + c), cvt<double>(__ldg(in + c)), s0);
            s1 = fma(__ldg(row + c + 32), cvt<double>(__ldg(in + c + 32)), s1);
            s2 = fma(__ldg(row + c + 64), cvt<double>(__ldg(in + c + 64)), s2);
            s3 = fma(__ldg(row + c + 96), cvt<double>(__ldg(in + c + 96)), s3);
        }
        for (; c < hi; c += 32) s0 = fma(__ldg(row + c), cvt<double>(__ldg(in + c)), s0);
        const double s = warp_sum((s0 + s1) + (s2 + s3));
        if (lane == 0) out[i] = cvt<VO>(s);
    }
}

void DenseCholesky::solve(const void *rhs, int rdt, void *x, int xdt, const int *done) {
    Context &c = *ctx;
    if (n == 0) return;
    if (tri) {  // x = Y^T (Y r), the intermediate in FP64
        UGPU_CHECK((rdt == UGPU_F64 || rdt == UGPU_F32) && rdt == xdt, UGPU_ERR_UNSUPPORTED,
                   "coarse solve: FP64 or FP32 vectors");
        const int gw = int(std::min<int64_t>((n + 7) / 8, int64_t(c.sms) * 8));  // a warp per row, 8 per CTA
        double *t = tmp_d.as<double>();
        if (rdt == UGPU_F64) {
            k_gemv64_tri<double, double, true><<<gw, 256, 0, c.stream>>>(Ainv.as<double>(), n,
                                                                         static_cast<const double *>(rhs), t, done);
            k_gemv64_tri<double, double, false><<<gw, 256, 0, c.stream>>>(Ainv.as<double>(), n, t,
                                                                          static_cast<double *>(x), done);
        } else {
            k_gemv64_tri<float, double, true><<<gw, 256, 0, c.stream>>>(Ainv.as<double>(), n,
                                                                        static_cast<const float *>(rhs), t, done);
            k_gemv64_tri<double, float, false><<<gw, 256, 0, c.stream>>>(Ainv.as<double>(), n, t,
                                                                         static_cast<float *>(x), done);
        }
        c.launches += 2;
        UGPU_LAUNCH_CHECK();
        return;
    }
    int g = int(std::min<int64_t>((n * 32 + 255) / 256, int64_t(c.sms) * 8));
    g = int(std::min<int64_t>(std::max<int64_t>(n, 1), int64_t(c.sms) * 8));
    auto al = [](const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
    const int gw = int(std::min<int64_t>((n + 7) / 8, int64_t(c.sms) * 8));  // a warp per row, 8 per CTA
    const bool split = (rdt == xdt) && (rdt == UGPU_F64 || (rdt == UGPU_F32 && !Ainv32.ptr)) &&
                       size_t(n) * sizeof(double) <= size_t(kGemvSmemMax);
    if (split) {
        const int gs = int(std::min<int64_t>((n + 3) / 4, int64_t(c.sms) * 8));  // four rows per CTA
        const size_t smem = size_t(n) * sizeof(double);
        const int vec = (n % 2 == 0) && al(Ainv.ptr);
        if (rdt == UGPU_F64) {
            static bool attr = false;
            if (!attr) {
                UGPU_CUDA(cudaFuncSetAttribute(k_gemv64_split<double>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               kGemvSmemMax));
                attr = true;
            }
            k_gemv64_split<double><<<gs, 256, smem, c.stream>>>(Ainv.as<double>(), n,
                                                                static_cast<const double *>(rhs),
                                                                static_cast<double *>(x), done, vec);
        } else {
            static bool attr = false;
            if (!attr) {
                UGPU_CUDA(cudaFuncSetAttribute(k_gemv64_split<float>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               kGemvSmemMax));
                attr = true;
            }
            k_gemv64_split<float><<<gs, 256, smem, c.stream>>>(Ainv.as<double>(), n, static_cast<const float *>(rhs),
                                                               static_cast<float *>(x), done, vec);
        }
        c.launches++;
        UGPU_LAUNCH_CHECK();
        return;
    }
    if (rdt == UGPU_F64 && xdt == UGPU_F64) {
        const int vec = (n % 2 == 0) && al(Ainv.ptr) && al(rhs);
        k_gemv64_warp<double><<<gw, 256, 0, c.stream>>>(Ainv.as<double>(), n, static_cast<const double *>(rhs),
                                                         static_cast<double *>(x), done, vec);
    } else if (rdt == UGPU_F32 && xdt == UGPU_F32 && Ainv32.ptr) {
        // FP32 inverse (only when make_fp32_inverse was called)
        const int vec = (n % 4 == 0) && al(Ainv32.ptr) && al(rhs);
        k_gemv<float><<<g, kGemvThreads, 0, c.stream>>>(Ainv32.as<float>(), n, static_cast<const float *>(rhs),
                                                         static_cast<float *>(x), done, vec);
    } else if (rdt == UGPU_F32 && xdt == UGPU_F32) {
        // FP64 solve for FP32 vectors
        const int vec = (n % 2 == 0) && al(Ainv.ptr) && (reinterpret_cast<uintptr_t>(rhs) & 7u) == 0;
        k_gemv64_warp<float><<<gw, 256, 0, c.stream>>>(Ainv.as<double>(), n, static_cast<const float *>(rhs),
                                                        static_cast<float *>(x), done, vec);
    } else
        throw Error(UGPU_ERR_UNSUPPORTED, "coarse solve: FP64 or FP32 vectors");
    c.launches++;
    UGPU_LAUNCH_CHECK();
}

}  // namespace ugpu
