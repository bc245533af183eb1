// Grid-wide sums and minima inside one kernel.
//
// Every CTA writes its partials, then adds one to a counter (release); one lane per CTA polls the counter until
// all CTAs have arrived (acquire), and a warp reads the partials and combines them in the same fixed order,
// so all CTAs hold the same bits and take the same branches.  Three trips through L2: 2.2 us over 152 CTAs
// and 1.8 us over 8 (448 threads each), measured in a loop of exchanges alone.  Polling the partials themselves
// (a sentinel where none has arrived) saves a trip but has every CTA read every slot while it is written:
// 8 us with the slots side by side, 2.9 us with one per 128-byte line.  Clusters that first add up over
// distributed shared memory: 3.5 us.
//
// Plain stores made by the CTA's threads before the __syncthreads() that precedes exchange() are visible to all
// CTAs after the __syncthreads() that follows it, read past L1 (__ldcg).
// The kernel must be launched cooperatively (all CTAs resident).  Every wait is bounded.
#pragma once
#include "internal.cuh"

namespace ugpu {

constexpr long long kGridSpin = 4000000000ll;  // clock cycles, about 2 s

// The NV values of an exchange are 64-bit patterns: doubles to be added, or (bits of MIN) order keys whose
// minimum is wanted.
template <int NV, int MIN>
struct Values {
    static __device__ __forceinline__ unsigned long long none(int i) { return (MIN >> i & 1) ? ~0ull : 0ull; }
    static __device__ __forceinline__ unsigned long long both(int i, unsigned long long a, unsigned long long b) {
        if (MIN >> i & 1) return a < b ? a : b;
        return (unsigned long long)__double_as_longlong(__longlong_as_double((long long)a) +
                                                        __longlong_as_double((long long)b));
    }
};
__device__ __forceinline__ unsigned long long dbits(double v) { return (unsigned long long)__double_as_longlong(v); }
__device__ __forceinline__ double bitsd(unsigned long long b) { return __longlong_as_double((long long)b); }

// Counter and partials (two sets, used in turn) of one kind of exchange, zero before the launch
template <int NV, int MIN = 0>
struct GridExchange {
    using V = Values<NV, MIN>;
    unsigned long long *count, *part;  // part: [2][NV][G]
    int G;                             // CTAs
    long long limit = kGridSpin;
    static constexpr size_t bytes(int G) { return 128 + sizeof(unsigned long long) * 2 * NV * size_t(G); }
    __device__ __forceinline__ void init(char *base, int ctas) {
        count = reinterpret_cast<unsigned long long *>(base);
        part = reinterpret_cast<unsigned long long *>(base + 128);
        G = ctas;
    }
    // One full warp: the k-th exchange (k = 0, 1, ...) of the CTA's NV values in shared memory; out in every lane.
    // False if a CTA did not arrive in time.
    __device__ __forceinline__ bool exchange(long long k, const unsigned long long *v, unsigned long long (&out)[NV]) const {
        const int lane = threadIdx.x & 31;
        unsigned long long *p = part + int64_t(k & 1) * NV * G;
        if (lane < NV) __stcg(p + lane * G + blockIdx.x, v[lane]);
        __syncwarp();
        int ok = 1;
        if (lane == 0) {
            asm volatile("red.release.gpu.global.add.u64 [%0], 1;" ::"l"(count) : "memory");
            const unsigned long long want = (unsigned long long)(k + 1) * (unsigned long long)G;
            const long long t0 = clock64();
            unsigned long long have;
            while (true) {
                asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(have) : "l"(count) : "memory");
                if (have >= want) break;
                if (clock64() - t0 > limit) {
                    ok = 0;
                    break;
                }
            }
        }
        __syncwarp();  // orders the other lanes' reads of the partials behind lane 0's acquire; a shuffle does not
        ok = __shfl_sync(0xffffffffu, ok, 0);
        unsigned long long s[NV];
#pragma unroll
        for (int i = 0; i < NV; ++i) s[i] = V::none(i);
        for (int j0 = 0; j0 < G; j0 += 32 * 5) {  // up to five partials per lane and value in flight
            const int live = (G - j0 + 31) / 32;  // groups of 32 that hold partials
            unsigned long long t[NV][5];
#pragma unroll
            for (int i = 0; i < NV; ++i)
#pragma unroll
                for (int q = 0; q < 5; ++q) {
                    const int j = j0 + 32 * q + lane;
                    t[i][q] = j < G ? __ldcg(p + i * G + j) : V::none(i);
                }
#pragma unroll
            for (int q = 0; q < 5; ++q)
                if (q < live)
#pragma unroll
                    for (int i = 0; i < NV; ++i) s[i] = V::both(i, s[i], t[i][q]);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int i = 0; i < NV; ++i) s[i] = V::both(i, s[i], __shfl_xor_sync(0xffffffffu, s[i], o));
#pragma unroll
        for (int i = 0; i < NV; ++i) out[i] = s[i];
        return ok != 0;
    }
};

// The same within one cluster of at most 16 CTAs: every CTA's warp stores its partials into every CTA's shared
// memory (st.async) and counts the arriving bytes on its own mbarrier.  0.6 us over 16 CTAs where the exchange
// through L2 takes 1.8 us even over 8; the cluster barrier with the same stores takes 0.9-1.6 us.  Data that the
// CTA's threads stored to shared memory before the preceding __syncthreads() may be read by the cluster's
// other CTAs after the following one.
template <int NV, int MIN = 0>
struct ClusterExchange {
    using V = Values<NV, MIN>;
    uint32_t slots, bars;  // shared addresses: [2][NV][16] 64-bit slots, [2] mbarriers
    uint32_t rank, size;
    long long limit = kGridSpin;
    static constexpr int kDoubles = 2 * NV * 16 + 2;  // shared 8-byte words
    __device__ __forceinline__ void init(double *shared, uint32_t r, uint32_t n) {
        slots = uint32_t(__cvta_generic_to_shared(shared));
        bars = slots + 2 * NV * 16 * 8;
        rank = r;
        size = n;
    }
    __device__ __forceinline__ void init_barriers() const {  // one thread; then a cluster barrier
        for (int i = 0; i < 2; ++i) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bars + 8 * i) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __device__ __forceinline__ bool exchange(long long k, const unsigned long long *v, unsigned long long (&out)[NV]) const {
        const uint32_t lane = threadIdx.x & 31, b = uint32_t(k & 1), parity = uint32_t(k >> 1) & 1u;
        if (lane == 0)
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bars + 8 * b), "r"(8u * NV * size)
                         : "memory");
        __syncwarp();
        if (lane < size) {
            uint32_t ra, rb;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(slots + (b * NV * 16 + rank) * 8), "r"(lane));
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(rb) : "r"(bars + 8 * b), "r"(lane));
            asm volatile("fence.acq_rel.cluster;" ::: "memory");
#pragma unroll
            for (int i = 0; i < NV; ++i)
                asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(ra + i * 128),
                             "l"(v[i]), "r"(rb)
                             : "memory");
        }
        uint32_t ok = 0;
        const long long t0 = clock64();
        while (true) {
            asm volatile(
                "{\n\t.reg .pred p;\n\t"
                "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
                "selp.u32 %0, 1, 0, p;\n\t}"
                : "=r"(ok)
                : "r"(bars + 8 * b), "r"(parity)
                : "memory");
            if (ok || clock64() - t0 > limit) break;
        }
        unsigned long long s[NV];
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            s[i] = V::none(i);
            if (lane < size)
                asm volatile("ld.shared::cta.u64 %0, [%1];"
                             : "=l"(s[i])
                             : "r"(slots + ((b * NV + i) * 16 + lane) * 8)
                             : "memory");
        }
#pragma unroll
        for (int o = 8; o > 0; o >>= 1)
#pragma unroll
            for (int i = 0; i < NV; ++i) s[i] = V::both(i, s[i], __shfl_xor_sync(0xffffffffu, s[i], o));
#pragma unroll
        for (int i = 0; i < NV; ++i) out[i] = __shfl_sync(0xffffffffu, s[i], 0);
        return __all_sync(0xffffffffu, ok != 0);
    }
};
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// a double at shared address `addr` of the cluster's CTA `rank`
__device__ __forceinline__ double ld_cluster(uint32_t addr, uint32_t rank) {
    uint32_t ra;
    unsigned long long v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.u64 %0, [%1];" : "=l"(v) : "r"(ra) : "memory");
    return __longlong_as_double((long long)v);
}

// sum of the CTA's threads' values in one warp: per-thread values through shared memory (sh: blockDim.x
// doubles, written by the caller before a __syncthreads()), then log-steps in the one warp.  FP64 adds are
// scarce (two per clock per SM): a shuffle tree in every warp would issue five per warp.
__device__ __forceinline__ double warp_sum_of(const double *sh, int n) {
    const int lane = threadIdx.x & 31;
    double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
    int i = lane;
    for (; i + 96 < n; i += 128) {
        a0 += sh[i];
        a1 += sh[i + 32];
        a2 += sh[i + 64];
        a3 += sh[i + 96];
    }
    if (i < n) a0 += sh[i];
    if (i + 32 < n) a1 += sh[i + 32];
    if (i + 64 < n) a2 += sh[i + 64];
    double s = (a0 + a1) + (a2 + a3);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

// Launches a resident kernel: as one cluster (of at most 16 CTAs), or cooperatively.  False where the device will not
// hold all its CTAs at once (a process with a share of the SMs, for example): nothing has run, and the
// separate kernels take the solve.  The launch itself says so; an occupancy query before each would cost time.
template <class Args>
inline bool launch_resident(Context &c, void (*kernel)(Args), const Args &args, int ctas, int threads, size_t smem,
                            bool cluster) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(unsigned(ctas));
    cfg.blockDim = dim3(unsigned(threads));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = c.stream;
    cudaLaunchAttribute at[1];
    cudaError_t e = cudaSuccess;
    if (cluster) {
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = unsigned(ctas);
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    } else {
        at[0].id = cudaLaunchAttributeCooperative;
        at[0].val.cooperative = 1;
    }
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (c.refuse_resident) e = cluster ? cudaErrorInvalidClusterSize : cudaErrorCooperativeLaunchTooLarge;
    else if (e == cudaSuccess) e = cudaLaunchKernelEx(&cfg, kernel, args);
    switch (e) {
    case cudaErrorCooperativeLaunchTooLarge:
    case cudaErrorInvalidClusterSize:
    case cudaErrorLaunchOutOfResources:
    case cudaErrorInvalidConfiguration:
    case cudaErrorNotSupported:
        cudaGetLastError();
        return false;
    default: UGPU_CUDA(e);
    }
    c.launches++;
    return true;
}

}  // namespace ugpu
