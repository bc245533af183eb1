// AlgebraicMultigrid with greedy agglomeration
// (utopia/solvers/multilevel/utopia_AlgebraicMultigrid.hpp:16-177,
//  utopia/solvers/multilevel/agglomerate/utopia_Agglomerate.hpp:51-186).
//
// The reference builds n_levels - 1 piecewise-constant prolongators by aggregating the rows of
// each level's operator in index order, forms every coarser operator by the Galerkin product
// (IPRTransfer::restrict(M) = P^T M P) and runs its Multigrid on that hierarchy.  The
// aggregation is a sequential greedy pass by definition (each row's choice depends on earlier
// rows'); rows that share no neighbour do not affect each other, so it runs on the GPU in
// dependency order (k_agglomerate), with the same result, or on the host where that order leaves
// too few rows at a time.  The Galerkin products, the smoothers and every cycle run on the GPU
// through the multigrid solver of mg.cu, which takes the prolongators as its transfer operators.
#include <algorithm>
#include <climits>
#include <cmath>
#include <vector>

#include "abi_util.cuh"
#include "device_util.cuh"
#include "solver.cuh"

namespace ugpu {

// Agglomerate::create_transfer_matrix (utopia_Agglomerate.hpp:51-186) on one process:
//   rows with a single stored value are Dirichlet rows and stay out of every aggregate (parent
//   -2) unless use_additive_correction; a_max_i = max_{j != i} |a_ij|; rows are visited in index
//   order and an unassigned row i opens aggregate c, then takes up to bmax unassigned neighbours
//   j (in column order) with |a_ij| > weight * a_max_i; a row that takes none is undone and joins
//   the aggregate of its largest |a_ij| (diagonal included; that may leave it unassigned or
//   excluded); rows still unassigned at the end become singleton aggregates.
//   The prolongator has P(i, parent_i) = 1 (0 where a_max_i = 0) for parent_i >= 0.
static void agglomerate_host(int64_t n, const int32_t *rp, const int32_t *ci, const double *v, int64_t bmax, double weight,
                      bool use_additive_correction, std::vector<int32_t> &parent, std::vector<double> &a_max,
                      int64_t &n_coarse) {
    parent.assign(size_t(n), -1);
    a_max.assign(size_t(n), 0.0);
    n_coarse = 0;
    if (!use_additive_correction) {
        for (int64_t i = 0; i < n; ++i)
            if (rp[i + 1] - rp[i] == 1) parent[size_t(i)] = -2;
    }
    for (int64_t i = 0; i < n; ++i)
        for (int32_t k = rp[i]; k < rp[i + 1]; ++k)
            if (ci[k] != i) a_max[size_t(i)] = std::max(a_max[size_t(i)], std::fabs(v[k]));
    for (int64_t i = 0; i < n; ++i) {
        if (parent[size_t(i)] != -1) continue;
        parent[size_t(i)] = int32_t(n_coarse);
        const double ami = a_max[size_t(i)];
        int64_t count = 0;
        for (int32_t k = rp[i]; k < rp[i + 1]; ++k) {
            const int32_t j = ci[k];
            if (weight * ami < std::fabs(v[k]) && parent[size_t(j)] == -1) {
                parent[size_t(j)] = int32_t(n_coarse);
                count++;
            }
            if (count >= bmax) break;
        }
        if (count == 0) {
            // not a cluster centre: join the aggregate of the strongest entry of the row
            parent[size_t(i)] = -1;
            double max_aij = 0;
            int32_t arg = -1;
            for (int32_t k = rp[i]; k < rp[i + 1]; ++k) {
                const double a = std::fabs(v[k]);
                if (a > max_aij) {
                    arg = ci[k];
                    max_aij = a;
                }
            }
            if (arg != -1) parent[size_t(i)] = parent[size_t(arg)];
        } else {
            ++n_coarse;
        }
    }
    for (int64_t i = 0; i < n; ++i)
        if (parent[size_t(i)] == -1) parent[size_t(i)] = int32_t(n_coarse++);
}

namespace {

// ------------------------------------------------------------------------------------
// The same pass on the GPU.  Row i reads and writes the aggregates of its neighbours and its own, so it has to
// wait for the earlier rows that have a neighbour in common with it, and for no others.  Every row m has a word
// with the number of turns taken at it and its aggregate (the centre's row, -1 none yet, -2 excluded).  The rows
// that touch m take their turns in index order; row i's turn at m comes when rank(i, m) turns have been taken.
// A row whose turn has come at all its neighbours has all their words to itself: it decides, and stores each
// word once, with the turn and the aggregate together, so the next row needs no fence and no second load.
// ------------------------------------------------------------------------------------
struct AggState {
    unsigned int unfit;     // columns not ascending, no diagonal, or a pattern that is not symmetric
    unsigned int excluded;  // some row is excluded
    unsigned int left;      // rows whose turn has not come
};

// the word at p if `want`; a predicate and no branch, so that a row's loads are in flight together
__device__ __forceinline__ unsigned long long agg_poll(const unsigned long long *p, bool want) {
    unsigned long long w = 0;
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.u32 p, %2, 0;\n @p ld.relaxed.gpu.global.u64 %0, [%1];\n}"
        : "+l"(w)
        : "l"(p), "r"(unsigned(want))
        : "memory");
    return w;
}

__device__ __forceinline__ unsigned long long agg_word(int turns, int parent) {
    return (unsigned long long)(unsigned)turns << 32 | unsigned(parent);
}

__global__ void __launch_bounds__(kBlock) k_agg_prepare(const int32_t *rp, const int32_t *ci, const double *v, int64_t n,
                                                        bool additive, double *a_max, unsigned long long *word,
                                                        AggState *st) {
    bool unfit = false, excluded = false;
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
        const int32_t k0 = rp[i], k1 = rp[i + 1];
        const bool out = !additive && k1 - k0 == 1;
        double m = 0.0;
        bool diag = false;
        int32_t last = -1;
        for (int32_t k = k0; k < k1; ++k) {
            const int32_t j = ci[k];
            unfit |= j <= last;
            last = j;
            if (j == i) diag = true;
            else if (m < fabs(v[k])) m = fabs(v[k]);
        }
        unfit |= !diag && !out;
        excluded |= out;
        a_max[i] = m;
        word[i] = agg_word(0, out ? -2 : -1);
    }
    unfit = __any_sync(0xffffffffu, unfit);
    excluded = __any_sync(0xffffffffu, excluded);
    if ((threadIdx.x & 31) == 0) {
        if (unfit) atomicOr(&st->unfit, 1u);
        if (excluded) atomicOr(&st->excluded, 1u);
    }
}

// rank of entry (i, m): how many rows before i touch m, which the symmetric pattern has in row m; -1 where m is
// excluded, and keeps its -2
__global__ void __launch_bounds__(kBlock) k_agg_ranks(const int32_t *rp, const int32_t *ci, int64_t n, bool additive,
                                                      int32_t *rank, AggState *st) {
    const bool some = st->excluded != 0;
    bool unfit = false;
    auto out = [&](int32_t r) { return some && !additive && rp[r + 1] - rp[r] == 1; };
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
        const int32_t k0 = rp[i], k1 = rp[i + 1];
        if (out(int32_t(i))) continue;
        for (int32_t k = k0; k < k1; ++k) {
            const int32_t m = ci[k];
            if (out(m)) {
                rank[k] = -1;
                continue;
            }
            int before = 0;
            bool found = false;
            const int32_t e1 = rp[m + 1];
            for (int32_t e = rp[m]; e < e1; ++e) {
                const int32_t r = ci[e];
                if (r >= i) {
                    found = r == i;
                    break;
                }
                before += !out(r);
            }
            unfit |= !found;
            rank[k] = before;
        }
    }
    if (__any_sync(0xffffffffu, unfit) && (threadIdx.x & 31) == 0) atomicOr(&st->unfit, 1u);
}

// G lanes take a row of up to G E entries, held in registers.  Bound by the chain of turns (about 700 one behind
// the other on a 95 x 89 x 97 grid), a store and a load of the L2 each: columns, ranks and strengths are loaded
// before the turn comes, and only the words still awaited are polled.  A row is polled until `limit` clocks
// after the thread's start and then left to the next launch.
template <int G, int E>
__global__ void __launch_bounds__(kBlock, 4) k_agglomerate(const int32_t *rp, const int32_t *ci, const double *v,
                                                        const double *a_max, const int32_t *rank, int64_t n, int bmax,
                                                        double weight, bool additive, unsigned long long *word,
                                                        long long limit, AggState *st) {
    const int lane = threadIdx.x & 31, tid = lane % G;
    const unsigned gmask = G == 32 ? 0xffffffffu : ((1u << G) - 1u) << (lane & ~(G - 1));
    const unsigned below = (1u << lane) - 1u;
    const long long t0 = clock64();
    unsigned int left = 0;
    auto ballot = [&](bool b) { return G == 1 ? unsigned(b) << lane : __ballot_sync(gmask, b) & gmask; };
    auto group_max = [&](int x) { return G == 1 ? x : __reduce_max_sync(gmask, x); };
    for (int64_t first = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x - lane) / G; first < n;
         first += int64_t(gridDim.x) * blockDim.x / G) {
        const int64_t i = first + lane / G;
        const int32_t k0 = i < n ? rp[i] : 0, len = i < n ? rp[i + 1] - k0 : 0;
        bool open = len > 1 || (len == 1 && additive);
        const double bar = i < n ? weight * a_max[i] : 0.0;
        int32_t col[E], rk[E];
        unsigned strong = 0, self = 0, pending = 0, best = 0;
        double big = 0.0;
        int at = INT_MAX;
#pragma unroll
        for (int q = 0; q < E; ++q) {
            const int e = q * G + tid;
            col[q] = 0;
            rk[q] = -1;
            if (e < len) {
                col[q] = ci[k0 + e];
                rk[q] = rank[k0 + e];
                const double a = fabs(v[k0 + e]);
                if (bar < a) strong |= 1u << q;
                if (col[q] == i) self = 1u << q;
                if (rk[q] >= 0) pending |= 1u << q;
                if (a > big) {
                    big = a;
                    at = e;
                }
            }
        }
        // the row's first largest entry
        double row_big = big;
        int row_at = at;
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) {
            const double ob = __shfl_xor_sync(gmask, row_big, o);
            const int oa = __shfl_xor_sync(gmask, row_at, o);
            if (ob > row_big || (ob == row_big && oa < row_at)) {
                row_big = ob;
                row_at = oa;
            }
        }
        if (row_at != INT_MAX && row_at % G == tid) best = 1u << (row_at / G);
        int par[E];
#pragma unroll
        for (int q = 0; q < E; ++q) par[q] = -2;
        // the lanes of a warp wait for each other's rows, so they poll together until all are through
        while (__any_sync(0xffffffffu, open)) {
            bool past = false;
            unsigned long long w[E];
            int missing = 0;
#pragma unroll
            for (int q = 0; q < E; ++q) w[q] = agg_poll(word + col[q], open && (pending >> q & 1u));
#pragma unroll
            for (int q = 0; q < E; ++q) {
                const bool had = open && (pending >> q & 1u);
                const int turns = int(w[q] >> 32);
                if (had && turns == rk[q]) {
                    par[q] = int(unsigned(w[q]));
                    pending &= ~(1u << q);
                }
                past |= had && (self >> q & 1u) && turns > rk[q];  // taken in an earlier launch
                if (had) missing = max(missing, rk[q] - turns);
            }
            const bool taken = __ballot_sync(0xffffffffu, past) & gmask;
            const bool wait = __ballot_sync(0xffffffffu, pending != 0) & gmask;
            const bool late = __any_sync(0xffffffffu, clock64() - t0 > limit);
            if (open && !taken && !wait) {
                int own = INT_MIN;
#pragma unroll
                for (int q = 0; q < E; ++q)
                    if (self >> q & 1u) own = par[q];
                own = group_max(own);
                if (own == -1) {
                    int count = 0;
#pragma unroll
                    for (int q = 0; q < E; ++q) {
                        const bool cand = (strong >> q & 1u) && !(self >> q & 1u) && par[q] == -1 && rk[q] >= 0;
                        const unsigned m = ballot(cand);
                        if (cand && count + __popc(m & below) < bmax) par[q] = int(i);
                        count += __popc(m);
                    }
                    int joined = int(i);
                    if (count == 0) {
                        joined = INT_MIN;
#pragma unroll
                        for (int q = 0; q < E; ++q)
                            if (best >> q & 1u) joined = par[q];
                        joined = group_max(joined);
                        if (joined == INT_MIN) joined = -1;
                    }
#pragma unroll
                    for (int q = 0; q < E; ++q)
                        if (self >> q & 1u) par[q] = joined;
                }
#pragma unroll
                for (int q = 0; q < E; ++q)
                    if (rk[q] >= 0)
                        *reinterpret_cast<volatile unsigned long long *>(word + col[q]) = agg_word(rk[q] + 1, par[q]);
            }
            if (open && !taken && wait && late) left += tid == 0;
            open = open && !taken && wait && !late;
            // rows several turns away leave the L2 to the front's
            missing = group_max(missing);
            missing = __reduce_min_sync(0xffffffffu, open ? missing : INT_MAX);
            if (missing > 2 && missing != INT_MAX) __nanosleep(100 * min(missing, 16));
        }
    }
    if (left) atomicAdd(&st->left, left);
}

// centres in the low half, rows without an aggregate in the high half: one scan numbers both
__global__ void k_agg_flags(const unsigned long long *word, int64_t n, int64_t *flag, int64_t *kept) {
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
        const int p = int(unsigned(word[i]));
        flag[i] = p == i ? 1 : p == -1 ? 1ll << 32 : 0;
        if (kept) kept[i] = p != -2;
    }
}

// aggregates in the order of their centres, then the single rows in theirs; P(i, parent_i)
__global__ void k_agg_prolongator(const unsigned long long *word, const int64_t *id, const int64_t *kept, int64_t nnz,
                                  int64_t centres, int64_t n, const double *a_max, int32_t *parent, int32_t *rp,
                                  int32_t *ci, double *v) {
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
        const int p = int(unsigned(word[i]));
        const int32_t c = p == -2   ? -2
                          : p == -1 ? int32_t(centres + (id[i] >> 32))
                                    : int32_t(id[p] & 0xffffffffll);
        parent[i] = c;
        const int64_t k = kept ? kept[i] : i;
        rp[i] = int32_t(k);
        if (i == n - 1) rp[n] = int32_t(nnz);
        if (c >= 0) {
            ci[k] = c;
            v[k] = a_max[i] != 0.0 ? 1.0 : 0.0;
        }
    }
}

struct Aggregates {
    std::vector<int32_t> parent;  // aggregate of each row
    int64_t n_coarse = 0;
    std::unique_ptr<Mat> P;       // null where the caller will not use it (too little coarsening)
};

// automatic depth: a level that shrinks by less than 4:3 is a stall
bool stalls(int64_t n, int64_t nc) { return 4 * nc > 3 * n; }

// Rows from which the GPU form is tried: a row costs the host 35 to 50 ns and its entries' copies, a turn of
// the chain about 1 us, and the chains of the smaller levels are hundreds of turns long.
constexpr int64_t kAggRows = 16384;

// false: not a matrix for this form, or a chain of turns that the host passes faster (a tridiagonal matrix)
bool agglomerate_device(const Mat &A, int64_t bmax, double weight, bool additive, bool drop_stalled, Aggregates &out) {
    Context &ctx = *A.ctx;
    const int64_t n = A.nrows;
    // longer rows would not fit the registers, and their ranks take time that is quadratic in their length (an arrow of
    // 200,000 rows: 75 ms before it was refused)
    if (n < kAggRows || bmax < 1 || A.max_row > 64) return false;
    const int32_t *rp = A.rowptr.as<int32_t>(), *ci = A.colidx.as<int32_t>();
    const double *v = A.vals.as<double>();
    Buffer a_max, word, rank, state;
    a_max.alloc(sizeof(double) * n);
    word.alloc(sizeof(unsigned long long) * n);
    rank.alloc(sizeof(int32_t) * std::max<int64_t>(A.nnz, 1));
    state.alloc(sizeof(AggState));
    auto *st = state.as<AggState>();
    UGPU_CUDA(cudaMemsetAsync(st, 0, sizeof(AggState), ctx.stream));
    k_agg_prepare<<<stream_grid(ctx, n), kBlock, 0, ctx.stream>>>(rp, ci, v, n, additive, a_max.as<double>(),
                                                                  word.as<unsigned long long>(), st);
    k_agg_ranks<<<stream_grid(ctx, n), kBlock, 0, ctx.stream>>>(rp, ci, n, additive, rank.as<int32_t>(), st);
    ctx.launches += 2;
    UGPU_LAUNCH_CHECK();
    AggState h{};
    auto read_state = [&] {
        UGPU_CUDA(cudaMemcpyAsync(&h, st, sizeof(h), cudaMemcpyDeviceToHost, ctx.stream));
        UGPU_CUDA(cudaStreamSynchronize(ctx.stream));
    };
    read_state();
    if (h.unfit) return false;
    auto *kernel = A.max_row <= 8 ? k_agglomerate<1, 8> : A.max_row <= 32 ? k_agglomerate<4, 8> : k_agglomerate<8, 8>;
    const int lanes = A.max_row <= 8 ? 1 : A.max_row <= 32 ? 4 : 8;
    int per_sm = 1;
    UGPU_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kBlock, 0));
    const int grid = int(std::max<int64_t>(
        1, std::min<int64_t>((n * lanes + kBlock - 1) / kBlock, int64_t(ctx.sms) * std::max(per_sm, 1))));
    // Launches of 128, 256, 512 ... us, so that a long chain is seen early: given up when the rows left would take
    // longer at the rate of the last launch than the host takes for all (40 ns each); the first two launches,
    // where the front of a grid is still small, have 16 and 4 times that.
    int64_t before = n;
    for (int p = 0;; ++p) {
        const double us = 128.0 * double(1 << std::min(p, 16));
        UGPU_CUDA(cudaMemsetAsync(&st->left, 0, sizeof(unsigned int), ctx.stream));
        kernel<<<grid, kBlock, 0, ctx.stream>>>(rp, ci, v, a_max.as<double>(), rank.as<int32_t>(), n,
                                                int(std::min<int64_t>(bmax, INT_MAX)), weight, additive,
                                                word.as<unsigned long long>(), (long long)(us * 2000.0), st);
        ctx.launches++;
        UGPU_LAUNCH_CHECK();
        read_state();
        if (!h.left) break;
        const double done = double(before - int64_t(h.left)), slack = p == 0 ? 16.0 : p == 1 ? 4.0 : 1.0;
        if (double(h.left) * us > done * slack * 0.04 * double(n)) return false;
        before = h.left;
    }
    Buffer flag, id, kept;
    flag.alloc(sizeof(int64_t) * n);
    id.alloc(sizeof(int64_t) * (n + 1));
    if (h.excluded) kept.alloc(sizeof(int64_t) * (n + 1));
    Buffer kept_flag;
    if (h.excluded) kept_flag.alloc(sizeof(int64_t) * n);
    k_agg_flags<<<stream_grid(ctx, n), kBlock, 0, ctx.stream>>>(word.as<unsigned long long>(), n, flag.as<int64_t>(),
                                                                h.excluded ? kept_flag.as<int64_t>() : nullptr);
    ctx.launches++;
    UGPU_LAUNCH_CHECK();
    const int64_t both = device_exclusive_scan(ctx, flag.as<int64_t>(), id.as<int64_t>(), n);
    const int64_t nnz = h.excluded ? device_exclusive_scan(ctx, kept_flag.as<int64_t>(), kept.as<int64_t>(), n) : n;
    const int64_t centres = both & 0xffffffffll;
    out.n_coarse = centres + (both >> 32);
    if (out.n_coarse < 1 || (drop_stalled && stalls(n, out.n_coarse))) return true;
    out.P = make_csr_device(ctx, n, out.n_coarse, nnz, UGPU_F64);
    Buffer parent;
    parent.alloc(sizeof(int32_t) * n);
    k_agg_prolongator<<<stream_grid(ctx, n), kBlock, 0, ctx.stream>>>(
        word.as<unsigned long long>(), id.as<int64_t>(), h.excluded ? kept.as<int64_t>() : nullptr, nnz, centres, n,
        a_max.as<double>(), parent.as<int32_t>(), out.P->rowptr.as<int32_t>(), out.P->colidx.as<int32_t>(),
        out.P->vals.as<double>());
    ctx.launches++;
    UGPU_LAUNCH_CHECK();
    out.parent.resize(size_t(n));
    UGPU_CUDA(cudaMemcpyAsync(out.parent.data(), parent.ptr, sizeof(int32_t) * n, cudaMemcpyDeviceToHost, ctx.stream));
    finalize_matrix(*out.P);
    UGPU_CUDA(cudaStreamSynchronize(ctx.stream));
    return true;
}

std::unique_ptr<Mat> prolongator(Context &ctx, int64_t n, int64_t nc, const std::vector<int32_t> &parent,
                                 const std::vector<double> &a_max) {
    std::vector<int32_t> rp(size_t(n) + 1, 0), ci;
    std::vector<double> v;
    ci.reserve(size_t(n));
    v.reserve(size_t(n));
    for (int64_t i = 0; i < n; ++i) {
        if (parent[size_t(i)] >= 0) {
            ci.push_back(parent[size_t(i)]);
            v.push_back(a_max[size_t(i)] != 0 ? 1.0 : 0.0);
        }
        rp[size_t(i) + 1] = int32_t(ci.size());
    }
    auto P = make_csr_device(ctx, n, nc, int64_t(ci.size()), UGPU_F64);
    UGPU_CUDA(cudaMemcpyAsync(P->rowptr.ptr, rp.data(), sizeof(int32_t) * rp.size(), cudaMemcpyHostToDevice,
                              ctx.stream));
    if (!ci.empty()) {
        UGPU_CUDA(cudaMemcpyAsync(P->colidx.ptr, ci.data(), sizeof(int32_t) * ci.size(), cudaMemcpyHostToDevice,
                                  ctx.stream));
        UGPU_CUDA(cudaMemcpyAsync(P->vals.ptr, v.data(), sizeof(double) * v.size(), cudaMemcpyHostToDevice,
                                  ctx.stream));
    }
    UGPU_CUDA(cudaStreamSynchronize(ctx.stream));  // host arrays go out of scope
    finalize_matrix(*P);
    return P;
}

void download_csr(const Mat &A, std::vector<int32_t> &rp, std::vector<int32_t> &ci, std::vector<double> &v) {
    Context &c = *A.ctx;
    rp.resize(size_t(A.nrows) + 1);
    ci.resize(size_t(A.nnz));
    v.resize(size_t(A.nnz));
    UGPU_CUDA(cudaMemcpyAsync(rp.data(), A.rowptr.ptr, sizeof(int32_t) * rp.size(), cudaMemcpyDeviceToHost, c.stream));
    if (A.nnz) {
        UGPU_CUDA(cudaMemcpyAsync(ci.data(), A.colidx.ptr, sizeof(int32_t) * ci.size(), cudaMemcpyDeviceToHost,
                                  c.stream));
        UGPU_CUDA(cudaMemcpyAsync(v.data(), A.vals.ptr, sizeof(double) * v.size(), cudaMemcpyDeviceToHost, c.stream));
    }
    UGPU_CUDA(cudaStreamSynchronize(c.stream));
}

// keys of the aggregation; every other key goes to the multigrid underneath
bool amg_key(const std::string &k) {
    return k == "n_levels" || k == "bmax" || k == "weight" || k == "use_additive_correction" ||
           k == "max_coarse_rows";
}

}  // namespace

class AlgebraicMultigrid final : public Solver {
public:
    explicit AlgebraicMultigrid(Context *c) : Solver(c, UGPU_SOLVER_AMG), mg_(make_multigrid(c)) {
        prm = mg_->prm;                 // the multigrid's parameters, readable through get()
        prm["n_levels"] = 2;            // utopia_AlgebraicMultigrid.hpp:173
        prm["bmax"] = 3;                // utopia_Agglomerate.hpp:43
        prm["weight"] = 1.0 / 3;        // utopia_Agglomerate.hpp:45
        prm["use_additive_correction"] = 0;
        prm["max_coarse_rows"] = 4096;  // n_levels = 0: coarsen until at most this many rows (or a stall)
    }

    void set(const std::string &k, double v) override {
        if (amg_key(k)) {
            Solver::set(k, v);
        } else {
            mg_->set(k, v);  // validates the key
            prm[k] = v;
        }
    }

    // AlgebraicMultigridBuilder::build (utopia_AlgebraicMultigrid.hpp:22-55)
    void update(const Mat *A) override {
        UGPU_CHECK(A && A->nrows == A->ncols, UGPU_ERR_ARG, "algebraic multigrid: square operator required");
        op = A;
        const int64_t want_levels = int64_t(get("n_levels"));
        const int64_t max_coarse = int64_t(get("max_coarse_rows"));
        UGPU_CHECK(want_levels == 0 || want_levels >= 2, UGPU_ERR_ARG, "n_levels must be 0 (automatic) or >= 2");
        transfers_.clear();
        parents_.clear();
        // The multigrid takes the products from here (a second time they took 2.2 ms of kernels at 95 x 89 x 97), unless
        // it forms others: from levels whose semidefinite diagonals it has fixed, or with their structure kept.
        const bool hand_over = get("fix_semidefinite_operators") == 0 && get("keep_galerkin_structure") == 0;
        std::vector<std::unique_ptr<Mat>> products;  // only the last one where they are not handed over
        const Mat *cur = A;
        std::vector<int32_t> rp, ci, parent;
        std::vector<double> v, amax;
        for (int64_t l = 0; want_levels == 0 || l < want_levels - 1; ++l) {
            if (want_levels == 0 && l > 0 && cur->nrows <= max_coarse) break;  // at least one coarse level
            Aggregates g;
            const int64_t bmax = int64_t(get("bmax"));
            const bool additive = get("use_additive_correction") != 0;
            UGPU_CHECK(cur->vdtype == UGPU_F64, UGPU_ERR_ARG, "algebraic multigrid: FP64 operator required");
            if (!agglomerate_device(*cur, bmax, get("weight"), additive, want_levels == 0, g)) {
                download_csr(*cur, rp, ci, v);
                agglomerate_host(cur->nrows, rp.data(), ci.data(), v.data(), bmax, get("weight"), additive, parent,
                                 amax, g.n_coarse);
            }
            UGPU_CHECK(g.n_coarse > 0, UGPU_ERR_ARG, "algebraic multigrid: empty coarse level");
            // automatic depth: stop at a stall (the Galerkin operators of stalled levels grow dense and would
            // dominate the cycle)
            if (want_levels == 0 && stalls(cur->nrows, g.n_coarse)) break;
            if (!g.P) {
                g.P = prolongator(*ctx, cur->nrows, g.n_coarse, parent, amax);
                g.parent = parent;
            }
            auto P = std::move(g.P);
            parents_.push_back(std::move(g.parent));
            auto next = ptap(*cur, *P);  // IPRTransfer::restrict(M): P^T M P
            transfers_.push_back(std::move(P));
            cur = next.get();
            if (!hand_over) products.clear();
            products.push_back(std::move(next));
        }
        UGPU_CHECK(!transfers_.empty(), UGPU_ERR_ARG, "algebraic multigrid: no coarse level");
        // Multigrid takes interpolation operators ordered coarse -> fine
        std::vector<const Mat *> P;
        for (auto it = transfers_.rbegin(); it != transfers_.rend(); ++it) P.push_back(it->get());
        mg_set_transfers(mg_.get(), P);
        if (hand_over) mg_set_products(mg_.get(), std::move(products));
        else products.clear();
        mg_->update(A);
    }

    void apply(const Vec &b, Vec &x) override {
        mg_->apply(b, x);
        st = mg_->st;
    }

    int pc_dtype() const override { return mg_->pc_dtype(); }
    void pc_enqueue(const void *r, void *z, const int *done) override { mg_->pc_enqueue(r, z, done); }

    int n_transfers() const { return int(transfers_.size()); }
    int64_t coarse_rows(int l) const { return transfers_.at(size_t(l))->ncols; }
    const std::vector<int32_t> &parent(int l) const { return parents_.at(size_t(l)); }
    const Solver *multigrid() const { return mg_.get(); }

private:
    std::unique_ptr<Solver> mg_;
    std::vector<std::unique_ptr<Mat>> transfers_;  // fine -> coarse, as built
    std::vector<std::vector<int32_t>> parents_;
};

std::unique_ptr<Solver> make_amg(Context *c) { return std::make_unique<AlgebraicMultigrid>(c); }

const Solver *amg_multigrid(const Solver *s) {
    auto *a = dynamic_cast<const AlgebraicMultigrid *>(s);
    return a ? a->multigrid() : s;
}

}  // namespace ugpu

extern "C" {

int ugpu_amg_parent(const ugpu_solver *amg, int level, int32_t *parent, int64_t *n, int64_t *n_coarse) {
    UGPU_ABI_BEGIN
    UGPU_REQUIRE(amg);
    auto *a = dynamic_cast<const ugpu::AlgebraicMultigrid *>(amg->impl.get());
    UGPU_CHECK(a, UGPU_ERR_ARG, "not an algebraic multigrid solver");
    UGPU_CHECK(level >= 0 && level < a->n_transfers(), UGPU_ERR_ARG, "level out of range");
    const auto &p = a->parent(level);
    if (n) *n = int64_t(p.size());
    if (n_coarse) *n_coarse = a->coarse_rows(level);
    if (parent) std::copy(p.begin(), p.end(), parent);
    UGPU_ABI_END(amg->impl->ctx)
}

}  // extern "C"
