// FP64 matrix products on the 5th-generation tensor cores (tcgen05, FP16 operands, FP32
// accumulators in TMEM), for the dense coarse factorisation.
//
// GB300 retires about two FP64 FMAs per clock per SM, so an n^3 set-up on the FP64 pipe is bound by
// it.  Here every operand row (a row of op(A), a column of op(B)) gets one power-of-two scale, its
// entries become 62-bit fixed-point numbers, and those are cut into eight signed radix-256 digits d in
// [-128, 128) (the splitting of Ozaki, Ogita, Oishi and Rump, "Error-free transformations of matrix
// multiplication by using fast routines of matrix multiplication", 2012).  A digit is an exact FP16
// number, a product of two digits at most 2^14 in magnitude.  Products of equal weight s + t (digits counted
// from 1) are summed in one FP32 accumulator over 128 values of k: at most 8 pairs x 128 x 2^14 = 2^24, so
// every sum is an exact integer.  The eight weights 2..9 (36 of the 64 digit products; what the dropped ones
// add is below 2^-57 of the two rows' maxima per value of k) are then added into two 64-bit integers per
// output, which hold K <= 16384 without overflow.  The result is rounded to FP64 once, at the end.
//
// One CTA computes a 128 x 64 tile: the eight weights' accumulators fill the 512 TMEM columns, so each
// digit is formed and read once per tile.  Per 32 values of k: 24 MMAs of 128 x (64 .. 256) x 16, issued by one
// thread from one stage of shared memory (8 digits x 192 rows x 32 values, 96 KB), while all threads split
// the next 32 values into the other stage; every fourth stage all threads read the accumulators into
// their integers.  Bound by the issue slots of the splitting (about 10 k instructions of 16 warps per stage)
// beside the MMAs (tensor pipe 35 % busy).  Measured: 4096^3 in 5.7 ms (24 TFLOP/s of FP64 results) where FP64
// FMA tiles took about 130 ms (1.05 TFLOP/s), 1024^3 in 0.12 ms.
// The error is absolute in the two rows' maxima: K 2^-57 max|a| max|b| bounds it (random operands, K = 300:
// 1.9e-16 of max max sqrt(K), an FMA chain 1.2e-15).  A sum of much smaller products, a row's small entries against
// small ones, has no relative accuracy below that, where an FMA chain's holds for any scale: who takes a
// split product has to restore it (dense.cu refines the inverse) or ask for FP64 multiply-adds (Gemm64::fma).
#include "abi_util.cuh"
#include "device_util.cuh"
#include "gemm64.cuh"

namespace ugpu {

namespace {

constexpr int GM = 128, GN = 64, GK = 32;  // CTA tile and values of k per stage
constexpr int kFlush = 4;                  // stages per reading of the accumulators (128 values of k)
constexpr int kDigits = 8;
constexpr int kWeights = 8;
constexpr int kSliceA = GM * GK * 2;  // bytes of one digit's A tile
constexpr int kSliceB = GN * GK * 2;
constexpr int kStage = kDigits * (kSliceA + kSliceB);
constexpr int kThreads = 512;
constexpr int kCols = GN / (kThreads / 128);       // output columns of a thread
constexpr int kTmemCols = 512;                     // kWeights * GN
constexpr size_t kGemmSmem = 2 * size_t(kStage) + 1024;  // + alignment
constexpr long long kSpin = 2000000000ll;          // wait limit in clock cycles (about 1 s)
constexpr int kScanInside = 128;                   // K up to which a tile finds its own row scales (12 us at 256)

__device__ __forceinline__ uint32_t saddr(const void *p) { return uint32_t(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ bool mma_wait(uint64_t *bar, uint32_t parity, long long limit) {
    const long long t0 = clock64();
    while (true) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(saddr(bar)), "r"(parity)
            : "memory");
        if (ok) return true;
        if (clock64() - t0 > limit) return false;
    }
}

// Shared-memory matrix descriptor of a K-major tile in 8 x 16-byte core matrices without swizzle: core
// matrices adjacent along k are 128 bytes apart, along the rows 512 bytes (GK = 32: four along k).
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
    return uint64_t((addr & 0x3ffffu) >> 4) | (uint64_t(128 >> 4) << 16) | (uint64_t(512 >> 4) << 32) | (1ull << 46);
}
// kind::f16 instruction descriptor: FP32 accumulators, FP16 A and B, both K-major, 128 x n
constexpr uint32_t instr_desc(int n) { return (1u << 4) | (uint32_t(n >> 3) << 17) | (uint32_t(GM >> 4) << 24); }

__device__ __forceinline__ void mma_f16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.u32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t addr, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(addr)
        : "memory");
}

// The fixed-point form of v under its row's exponent field E (the largest of the row, at least kMinExp):
// v = X 2^(E - 1084), |X| < 2^62, bits below 2^-61 of the row's maximum dropped; biased by 128 in every
// radix-256 digit, so that the digits are the bytes.  A zero's exponent field 0 lies more than 62 below E:
// the shift clears it without a test.
constexpr uint32_t kMinExp = 64;
constexpr unsigned long long kBias = 0x8080808080808080ull;
__device__ __forceinline__ unsigned long long fixed_biased(double v, uint32_t E) {
    const uint32_t h = uint32_t(__double2hiint(v)), l = uint32_t(__double2loint(v));
    const uint32_t s = E + 2u - ((h >> 20) & 0x7ffu);  // right shift of the significand with its top bit at 63
    const uint32_t mh = __funnelshift_l(l, (h & 0xfffffu) | 0x100000u, 11), ml = l << 11;
    const uint32_t s1 = min(s, 32u), s2 = s - s1;
    uint32_t xh, xl = __funnelshift_rc(ml, mh, s1);
    asm("shr.u32 %0, %1, %2;" : "=r"(xh) : "r"(mh), "r"(s1));  // PTX shifts by 32 and more give 0
    asm("shr.u32 %0, %0, %1;" : "+r"(xl) : "r"(s2));
    const unsigned long long x = ((unsigned long long)xh << 32) | xl;
    const unsigned long long neg = (unsigned long long)(long long)(int(h) >> 31);
    return (x ^ neg) + (kBias - neg);
}
// the digits of two numbers as a pair of FP16: bytes u biased by 128, 0x6400 + u is 1024 + u exactly
template <int S>  // 1 = leading
__device__ __forceinline__ uint32_t digit_pair(unsigned long long u0, unsigned long long u1) {
    constexpr int byte = kDigits - S;  // of the 64-bit number
    const uint32_t w0 = byte < 4 ? uint32_t(u0) : uint32_t(u0 >> 32), w1 = byte < 4 ? uint32_t(u1) : uint32_t(u1 >> 32);
    constexpr uint32_t b = byte & 3;
    const uint32_t p = (__byte_perm(w0, w1, b | (b << 4) | ((b + 4) << 8) | ((b + 4) << 12)) & 0x00ff00ffu) | 0x64006400u;
    uint32_t r;
    asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(p), "r"(0x64806480u));  // 1152 = 1024 + 128
    return r;
}
template <int S, int NV>  // NV values (4 or 8) of one row
__device__ __forceinline__ void store_digits(char *dst, int slice, const unsigned long long (&u)[NV]) {
    if constexpr (NV == 8) {
        uint4 w;
        w.x = digit_pair<S>(u[0], u[1]);
        w.y = digit_pair<S>(u[2], u[3]);
        w.z = digit_pair<S>(u[4], u[5]);
        w.w = digit_pair<S>(u[6], u[7]);
        *reinterpret_cast<uint4 *>(dst + (S - 1) * slice) = w;
    } else {
        uint2 w;
        w.x = digit_pair<S>(u[0], u[1]);
        w.y = digit_pair<S>(u[2], u[3]);
        *reinterpret_cast<uint2 *>(dst + (S - 1) * slice) = w;
    }
    if constexpr (S < kDigits) store_digits<S + 1, NV>(dst, slice, u);
}

// The double nearest to (hi 2^32 + lo) 2^x (ties to even), by integer operations: conversions and scalings of
// the outputs in FP64 arithmetic would take longer than a short product's MMAs.
__device__ __forceinline__ double round_sum(long long hi, long long lo, int x) {
    // t = hi 2^32 + lo as 128 bits, |t| < 2^90
    unsigned long long t0 = (unsigned long long)hi << 32;
    long long t1 = hi >> 32;
    t0 += (unsigned long long)lo;
    t1 += (lo >> 63) + (t0 < (unsigned long long)lo ? 1 : 0);
    const bool neg = t1 < 0;
    unsigned long long u1 = (unsigned long long)t1;
    if (neg) {
        t0 = 0ull - t0;
        u1 = ~u1 + (t0 == 0ull ? 1ull : 0ull);
    }
    if ((t0 | u1) == 0ull) return 0.0;
    // significand with its top bit at 63, sticky bit from what is shifted out
    const int z = u1 ? __clzll(u1) : 64 + __clzll(t0);
    unsigned long long m;
    bool sticky;
    if (z >= 64) {
        m = t0 << (z - 64);
        sticky = false;
    } else if (z == 0) {
        m = u1;
        sticky = t0 != 0ull;
    } else {
        m = (u1 << z) | (t0 >> (64 - z));
        sticky = (t0 << z) != 0ull;
    }
    int e = x + 127 - z;  // value = m 2^-63 2^e, m's top bit set
    if (e < -1022) return ldexp(neg ? -__ull2double_rn(m) : __ull2double_rn(m), e - 63);  // subnormal results
    unsigned long long f = m >> 11;
    const unsigned long long rest = (m & 0x7ffull) | (sticky ? 1ull : 0ull);
    f += (rest > 0x400ull || (rest == 0x400ull && (f & 1ull))) ? 1ull : 0ull;
    if (e + int(f >> 53) > 1023) return __longlong_as_double(neg ? (long long)0xfff0000000000000ull : 0x7ff0000000000000ll);
    const unsigned long long bits = ((unsigned long long)(e + 1022) << 52) + f;  // f's top bit adds 1 to the field
    return __longlong_as_double((long long)(bits | (neg ? 0x8000000000000000ull : 0ull)));
}

__device__ __forceinline__ uint32_t exponent_bits(const double *p) {
    return uint32_t(__double2hiint(__ldg(p))) & 0x7fffffffu;
}

// The largest exponent field of every row of both operands, into global arrays that start at zero: a tile of a
// product with a long K would have to read all its rows twice.  A warp takes 256 values of k of one row
// (operands contiguous along k), or 32 values of k of 32 rows.
__host__ __device__ inline int64_t scan_warps(bool kcont, int rows, int K) {
    return kcont ? int64_t(rows) * ((K + 255) / 256) : int64_t((rows + 31) / 32) * ((K + 31) / 32);
}
__global__ void __launch_bounds__(256) k_gemm64_scan(const Gemm64 g, uint32_t *eA, uint32_t *eB) {
    const int lane = threadIdx.x & 31;
    const int64_t warp = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) >> 5;
    const int64_t wa = scan_warps(g.a_k == 1, g.M, g.K), wb = scan_warps(g.b_k == 1, g.N, g.K);
    if (warp >= wa + wb) return;
    const bool isa = warp < wa;
    const int64_t u = isa ? warp : warp - wa;
    const double *p = isa ? g.A : g.B;
    const int64_t rs = isa ? g.a_row : g.b_row, ks = isa ? g.a_k : g.b_k;
    const int rows = isa ? g.M : g.N;
    uint32_t *E = isa ? eA : eB;
    const int len = ks == 1 ? 256 : 32, segs = (g.K + len - 1) / len;
    const int k0 = int(u % segs) * len, k1 = min(g.K, k0 + len);
    uint32_t m = 0;
    if (ks == 1) {
        const int64_t r = u / segs;
#pragma unroll 8
        for (int k = k0 + lane; k < k1; k += 32) m = max(m, exponent_bits(p + r * rs + k));
        m = __reduce_max_sync(0xffffffffu, m);
        if (lane == 0) atomicMax(E + r, m >> 20);
    } else {
        const int64_t r = (u / segs) * 32 + lane;
        if (r >= rows) return;
#pragma unroll 8
        for (int k = k0; k < k1; ++k) m = max(m, exponent_bits(p + r + k * ks));
        atomicMax(E + r, m >> 20);
    }
}

// the NV values k .. k + NV - 1 of one operand row (zero outside the rows and the k range)
template <bool KCONT, int NV>
__device__ __forceinline__ void load_values(const double *p, int64_t rs, int64_t ks, int r, int rows, int k, int k1,
                                            int vec, double (&v)[NV]) {
    const double *q = p + (KCONT ? r * rs + k : r + k * ks);
    if (r < rows && k + NV <= k1) {
        if (KCONT && vec) {
#pragma unroll
            for (int j = 0; j < NV; j += 2) {
                const double2 d = __ldg(reinterpret_cast<const double2 *>(q + j));
                v[j] = d.x;
                v[j + 1] = d.y;
            }
        } else {
#pragma unroll
            for (int j = 0; j < NV; ++j) {
                v[j] = __ldg(q);
                q += KCONT ? 1 : ks;
            }
        }
    } else {
#pragma unroll
        for (int j = 0; j < NV; ++j) v[j] = (r < rows && k + j < k1) ? __ldg(q + (KCONT ? j : j * ks)) : 0.0;
    }
}
template <int NV>
__device__ __forceinline__ uint32_t max_exponent(const double (&v)[NV], uint32_t m) {
#pragma unroll
    for (int j = 0; j < NV; ++j) m = max(m, uint32_t(__double2hiint(v[j])) & 0x7fffffffu);
    return m;
}

template <bool AK, bool BK>
__global__ void __launch_bounds__(kThreads, 1) k_gemm64(const Gemm64 g, const uint32_t *gEA, const uint32_t *gEB,
                                                        int *kflag) {
    const int m0 = blockIdx.y * GM, n0 = blockIdx.x * GN;
    if ((g.flags & kGemmLower) && n0 > m0 + GM - 1) return;
    extern __shared__ char smem_raw[];
    __shared__ uint32_t eA[GM], eB[GN];
    __shared__ uint64_t bar[2];
    __shared__ uint32_t s_tmem;
    char *stage = smem_raw + ((1024u - (saddr(smem_raw) & 1023u)) & 1023u);
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int M = min(GM, g.M - m0), N = min(GN, g.N - n0);
    // the k range in which both operand rows of the tile may be non-zero
    int k0 = 0, k1 = g.K;
    if (g.flags & kGemmKFromN) k0 = max(k0, n0);
    if (g.flags & kGemmKFromM) k0 = max(k0, m0);
    if (g.flags & kGemmKToN) k1 = min(k1, n0 + GN);
    if (g.flags & kGemmKToM) k1 = min(k1, m0 + GM);
    const double *A = g.A + m0 * g.a_row, *B = g.B + n0 * g.b_row;
    const int nk = (max(k1 - k0, 0) + GK - 1) / GK;

    // a thread's share of a stage: 8 values of k of one row of A and 4 of one row of B.  A warp's lanes cover
    // 8 rows x 4 pieces of A (8 rows x 4 half pieces of B), so each digit's stores fill contiguous bytes
    const int ar = (t & 7) + ((t >> 5) << 3), ak = ((t >> 3) & 3) * 8;
    const int br = ((t >> 1) & 7) + ((t >> 6) << 3), bk = (((t >> 4) & 3) * 2 + (t & 1)) * 4;
    double va[8], vb[4];
    auto load = [&](int c) {
        load_values<AK, 8>(A, g.a_row, g.a_k, ar, M, k0 + c * GK + ak, k1, g.vec_a, va);
        load_values<BK, 4>(B, g.b_row, g.b_k, br, N, k0 + c * GK + bk, k1, g.vec_b, vb);
    };
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(saddr(&s_tmem)),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (t == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(saddr(&bar[0])) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(saddr(&bar[1])) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (t < GM) eA[t] = (gEA && t < M) ? max(gEA[m0 + t], kMinExp) : kMinExp;
    if (t < GN) eB[t] = (gEB && t < N) ? max(gEB[n0 + t], kMinExp) : kMinExp;
    __syncthreads();
    if (!gEA) {  // a short K: the row scales from one pass over the tile's operands, backwards so that the first
                 // stage's values stay in registers
        uint32_t ma = 0, mb = 0;
        for (int c = nk - 1; c >= 0; --c) {
            load(c);
            ma = max_exponent(va, ma);
            mb = max_exponent(vb, mb);
        }
        atomicMax(&eA[ar], ma >> 20);
        atomicMax(&eB[br], mb >> 20);
    } else if (nk > 0) {
        load(0);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_tmem;
    const uint32_t ea = eA[ar], eb = eB[br];

    auto split = [&](int c) {
        char *sa = stage + (c & 1) * kStage, *sb = sa + kDigits * kSliceA;
        {
            unsigned long long u[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) u[j] = fixed_biased(va[j], ea);
            store_digits<1, 8>(sa + (ar >> 3) * 512 + (ak >> 3) * 128 + (ar & 7) * 16, kSliceA, u);
        }
        {
            unsigned long long u[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) u[j] = fixed_biased(vb[j], eb);
            store_digits<1, 4>(sb + (br >> 3) * 512 + (bk >> 3) * 128 + (br & 7) * 16 + (bk & 4) * 2, kSliceB, u);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    };
    auto issue = [&](int c) {  // one thread
        const uint32_t sa = saddr(stage + (c & 1) * kStage), sb = sa + kDigits * kSliceA;
        const uint32_t cont = (c % kFlush) ? 1u : 0u;
        // Digit s of A meets digits 1 .. 9 - s of B.  B's digits are one tall operand (64 rows each) and the
        // weights' accumulators are adjacent, so one MMA covers up to four digits of B: 24 per stage instead of 72.
        const uint64_t da = smem_desc(sa), db = smem_desc(sb);
#pragma unroll
        for (int s = 0; s < kDigits; ++s)
#pragma unroll
            for (int q = 0; q < GK / 16; ++q)
#pragma unroll
                for (int h = 0; h < kDigits - s; h += 4) {
                    const int n = (kDigits - s - h < 4 ? kDigits - s - h : 4) * GN;
                    mma_f16(tmem + uint32_t((s + h) * GN), da + uint64_t((s * kSliceA + q * 256) >> 4),
                            db + uint64_t((h * kSliceB + q * 256) >> 4), instr_desc(n), (s | q) ? 1u : cont);
                }
        if (g.lose_commit && c == 0) return;
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                         saddr(&bar[c & 1]))
                     : "memory");
    };

    // a thread's outputs: row (warp % 4) * 32 + lane, columns (warp / 4) * kCols + j
    long long hi[kCols], lo[kCols];
#pragma unroll
    for (int j = 0; j < kCols; ++j) hi[j] = lo[j] = 0;
    const uint32_t tm = tmem + (uint32_t((warp & 3) * 32) << 16) + uint32_t((warp >> 2) * kCols);
    auto flush = [&]() {
#pragma unroll
        for (int w = 0; w < kWeights; ++w) {
            uint32_t v[16];
            tmem_ld16(tm + uint32_t(w * GN), v);
            // weights 2..5 into hi (units 2^-40), 6..9 into lo (units 2^-72)
            const int f = 1 << (8 * (3 - (w & 3)));
#pragma unroll
            for (int j = 0; j < kCols; ++j) {
                const long long add = (long long)__float2int_rn(__uint_as_float(v[j])) * f;
                if (w < 4) hi[j] += add;
                else lo[j] += add;
            }
        }
    };

    int late = 0;
    for (int c = 0; c < nk; ++c) {
        // the stage's last MMAs (two stages ago) must have read it
        if (c >= 2 && !mma_wait(&bar[c & 1], uint32_t((c >> 1) - 1) & 1u, g.spin)) late = 1;
        split(c);
        if (c + 1 < nk) load(c + 1);
        if (c > 0 && c % kFlush == 0) {
            if (!mma_wait(&bar[(c - 1) & 1], uint32_t((c - 1) >> 1) & 1u, g.spin)) late = 1;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            flush();
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        }
        late = __syncthreads_or(late);
        if (late) break;  // an MMA never completed: all threads leave together
        if (t == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            issue(c);
        }
    }
    if (nk > 0 && !late) {
        if (!mma_wait(&bar[(nk - 1) & 1], uint32_t((nk - 1) >> 1) & 1u, g.spin)) late = 1;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        flush();
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    if (late) atomicExch(kflag, 1);
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");

    // value = (hi 2^32 + lo) 2^(e_r + e_c + 4 - 72), e = E - 1022; through shared memory (the stages are free
    // now) so that rows of C are read and written in whole lines
    double *out = reinterpret_cast<double *>(stage);  // [GM][GN + 1]
    {
        const int r = (warp & 3) * 32 + lane, cb = (warp >> 2) * kCols;
        const int er = int(eA[r]);
#pragma unroll
        for (int j = 0; j < kCols; ++j) {
            const int ec = int(eB[cb + j]);
            double v = round_sum(hi[j], lo[j], er + ec - 2044 + 4 - 72);
            if (er == 0x7ff || ec == 0x7ff) v = __longlong_as_double(0x7ff8000000000000ll);  // infinity or NaN in
            out[r * (GN + 1) + cb + j] = v;
        }
    }
    __syncthreads();
    double *C = g.C + int64_t(m0) * g.ldc + n0;
    const long long flip = g.negate ? (long long)0x8000000000000000ull : 0ll;
    for (int e = t; e < M * GN; e += kThreads) {
        const int r = e / GN, cc = e % GN;
        if (cc >= N) continue;
        const double v = __longlong_as_double(__double_as_longlong(out[r * (GN + 1) + cc]) ^ flip);
        C[r * g.ldc + cc] = g.add ? C[r * g.ldc + cc] + v : v;
    }
}

// Small products on the FP64 pipes of the whole chip: a CTA takes 8 x 8 outputs, four threads an output with
// every fourth k each.  One or two CTAs of k_gemm64 are bound by their own splitting and rounding (18 us at 64^3,
// 28 at 128^3, 37 at 256^3, on 1, 2 and 8 SMs); these FMAs are 0.9 k, 6.9 k and 55 k clocks of all the pipes, where
// the two forms meet.  Factor and inverse of 4096 rows: 14.5 ms with none of the products here, 12.6 up to 64^3,
// 11.2 up to 128^3, 10.6 up to 256^3.
constexpr int kSmallK = 256;
constexpr int64_t kSmallWork = 1 << 24;
constexpr int kSmallTile = 8, kSmallRow = kSmallK + 4;  // a row's pad puts the lanes of a half-warp on all banks
__global__ void __launch_bounds__(256) k_gemm64_small(const Gemm64 g) {
    const int m0 = blockIdx.y * kSmallTile, n0 = blockIdx.x * kSmallTile;
    if ((g.flags & kGemmLower) && n0 > m0 + kSmallTile - 1) return;
    __shared__ double s[2][kSmallTile][kSmallRow];
    int k0 = 0, k1 = g.K;
    if (g.flags & kGemmKFromN) k0 = max(k0, n0);
    if (g.flags & kGemmKFromM) k0 = max(k0, m0);
    if (g.flags & kGemmKToN) k1 = min(k1, n0 + kSmallTile);
    if (g.flags & kGemmKToM) k1 = min(k1, m0 + kSmallTile);
    const int len = k1 - k0, t = threadIdx.x, lane = t & 31, warp = t >> 5;
    double v[2][kSmallK / 32];
#pragma unroll
    for (int o = 0; o < 2; ++o) {
        const int64_t rs = o ? g.b_row : g.a_row, ks = o ? g.b_k : g.a_k;
        const int r = ks == 1 ? warp : t & 7, kk = ks == 1 ? lane : t >> 3;
        const int rows = o ? g.N - n0 : g.M - m0;
        const double *p = (o ? g.B + n0 * rs : g.A + m0 * rs) + r * rs + int64_t(k0 + kk) * ks;
#pragma unroll
        for (int q = 0; q < kSmallK / 32; ++q) v[o][q] = (r < rows && kk + 32 * q < len) ? __ldg(p + 32 * q * ks) : 0.0;
    }
#pragma unroll
    for (int o = 0; o < 2; ++o) {
        const bool along = (o ? g.b_k : g.a_k) == 1;
        const int r = along ? warp : t & 7, kk = along ? lane : t >> 3;
#pragma unroll
        for (int q = 0; q < kSmallK / 32; ++q)
            if (32 * q < len) s[o][r][kk + 32 * q] = v[o][q];
    }
    __syncthreads();
    const int j = lane >> 2;
    double acc = 0.0;
#pragma unroll 4
    for (int k = lane & 3; k < len; k += 4) acc = fma(s[0][warp][k], s[1][j][k], acc);
    acc += __shfl_xor_sync(0xffffffffu, acc, 1);
    acc += __shfl_xor_sync(0xffffffffu, acc, 2);
    if ((lane & 3) || m0 + warp >= g.M || n0 + j >= g.N) return;
    if (g.negate) acc = -acc;
    double *C = g.C + int64_t(m0 + warp) * g.ldc + n0 + j;
    *C = g.add ? *C + acc : acc;
}

// Larger products where every product has to be an FP64 multiply-add: T x T tiles, 16 x 16 threads of T / 16 x T / 16
// outputs.  Bound by the FP64 pipes (1.05 TFLOP/s at 4096^3).
template <bool AK, bool BK, int T>
__global__ void __launch_bounds__(256) k_gemm64_fma(const Gemm64 g) {
    constexpr int TK = 16, PT = T / 16;
    __shared__ double s_a[TK][T + 1], s_b[TK][T + 1];
    const int m0 = blockIdx.y * T, n0 = blockIdx.x * T;
    if ((g.flags & kGemmLower) && n0 > m0 + T - 1) return;
    int k0 = 0, k1 = g.K;
    if (g.flags & kGemmKFromN) k0 = max(k0, n0);
    if (g.flags & kGemmKFromM) k0 = max(k0, m0);
    if (g.flags & kGemmKToN) k1 = min(k1, n0 + T);
    if (g.flags & kGemmKToM) k1 = min(k1, m0 + T);
    const int t = threadIdx.x, tx = t & 15, ty = t >> 4;
    double acc[PT][PT] = {};
    for (int k = k0; k < k1; k += TK) {
        for (int e = t; e < T * TK; e += 256) {
            const int ra = AK ? e / TK : e % T, ka = AK ? e % TK : e / T;
            const int rb = BK ? e / TK : e % T, kb = BK ? e % TK : e / T;
            s_a[ka][ra] = m0 + ra < g.M && k + ka < k1 ? __ldg(g.A + (m0 + ra) * g.a_row + (k + ka) * g.a_k) : 0.0;
            s_b[kb][rb] = n0 + rb < g.N && k + kb < k1 ? __ldg(g.B + (n0 + rb) * g.b_row + (k + kb) * g.b_k) : 0.0;
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < TK; ++q) {
            double a[PT], b[PT];
#pragma unroll
            for (int i = 0; i < PT; ++i) {
                a[i] = s_a[q][ty + 16 * i];
                b[i] = s_b[q][tx + 16 * i];
            }
#pragma unroll
            for (int i = 0; i < PT; ++i)
#pragma unroll
                for (int j = 0; j < PT; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < PT; ++i)
#pragma unroll
        for (int j = 0; j < PT; ++j) {
            const int r = m0 + ty + 16 * i, c = n0 + tx + 16 * j;
            if (r >= g.M || c >= g.N) continue;
            double *o = g.C + int64_t(r) * g.ldc + c;
            const double v = g.negate ? -acc[i][j] : acc[i][j];
            *o = g.add ? *o + v : v;
        }
}

// the tile that keeps the grid at least two CTAs per SM
template <int T>
void launch_fma(Context &c, const Gemm64 &g) {
    const dim3 grid(unsigned((g.N + T - 1) / T), unsigned((g.M + T - 1) / T));
    auto run = [&](auto kern) { kern<<<grid, 256, 0, c.stream>>>(g); };
    if (g.a_k == 1 && g.b_k == 1) run(k_gemm64_fma<true, true, T>);
    else if (g.a_k == 1) run(k_gemm64_fma<true, false, T>);
    else if (g.b_k == 1) run(k_gemm64_fma<false, true, T>);
    else run(k_gemm64_fma<false, false, T>);
}

}  // namespace

void gemm64(Context &c, const Gemm64 &args, Buffer &scales) {
    Gemm64 g = args;
    if (g.M <= 0 || g.N <= 0) return;
    // 16-byte loads along k need aligned rows (k ranges start at multiples of 4)
    auto al = [](const double *p, int64_t row) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0 && row % 2 == 0; };
    g.vec_a = al(g.A, g.a_row);
    g.vec_b = al(g.B, g.b_row);
    UGPU_CHECK(g.K <= 16384, UGPU_ERR_UNSUPPORTED, "gemm64: K is limited to 16384");
    UGPU_CHECK((g.a_row == 1 || g.a_k == 1) && (g.b_row == 1 || g.b_k == 1), UGPU_ERR_INTERNAL,
               "gemm64: operand strides");
    if (g.K <= kSmallK && int64_t(g.M) * g.N * g.K <= kSmallWork) {
        const dim3 tiles(unsigned((g.N + kSmallTile - 1) / kSmallTile), unsigned((g.M + kSmallTile - 1) / kSmallTile));
        k_gemm64_small<<<tiles, 256, 0, c.stream>>>(g);
        c.launches++;
        UGPU_LAUNCH_CHECK();
        return;
    }
    if (g.fma) {
        if (int64_t((g.M + 63) / 64) * ((g.N + 63) / 64) >= 2 * int64_t(c.sms)) launch_fma<64>(c, g);
        else launch_fma<32>(c, g);
        c.launches++;
        UGPU_LAUNCH_CHECK();
        return;
    }
    g.spin = c.product_test_spin > 0 ? c.product_test_spin : kSpin;
    g.lose_commit = c.product_test_spin > 0;
    uint32_t *eA = nullptr, *eB = nullptr;
    if (g.K > kScanInside) {
        scales.ensure(sizeof(uint32_t) * (size_t(g.M) + size_t(g.N)));
        eA = scales.as<uint32_t>();
        eB = eA + g.M;
        UGPU_CUDA(cudaMemsetAsync(eA, 0, sizeof(uint32_t) * (size_t(g.M) + size_t(g.N)), c.stream));
        const int64_t warps = scan_warps(g.a_k == 1, g.M, g.K) + scan_warps(g.b_k == 1, g.N, g.K);
        k_gemm64_scan<<<unsigned((warps + 7) / 8), 256, 0, c.stream>>>(g, eA, eB);
        c.launches++;
    }
    const dim3 grid(unsigned((g.N + GN - 1) / GN), unsigned((g.M + GM - 1) / GM));
    auto run = [&](auto kern) {
        UGPU_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kGemmSmem)));
        kern<<<grid, kThreads, kGemmSmem, c.stream>>>(g, eA, eB, c.d_kflags() + 1);
    };
    if (g.a_k == 1 && g.b_k == 1) run(k_gemm64<true, true>);
    else if (g.a_k == 1) run(k_gemm64<true, false>);
    else if (g.b_k == 1) run(k_gemm64<false, true>);
    else run(k_gemm64<false, false>);
    c.launches++;
    UGPU_LAUNCH_CHECK();
}

}  // namespace ugpu

using namespace ugpu;

extern "C" int ugpu_test_product_wait_timeout(ugpu_ctx *ctx, int64_t spin_cycles) {
    UGPU_ABI_BEGIN
    UGPU_REQUIRE(ctx);
    UGPU_CHECK(spin_cycles > 0 && spin_cycles <= 100000000ll, UGPU_ERR_ARG, "test wait limit: 1 .. 1e8 cycles");
    Context &c = ctx->impl;
    Buffer operands, out, scales;
    operands.alloc(sizeof(double) * 512 * 512);
    out.alloc(sizeof(double) * 512 * 512);
    UGPU_CUDA(cudaMemsetAsync(operands.ptr, 0, operands.bytes, c.stream));
    Gemm64 g;
    g.M = g.N = g.K = 512;
    g.A = g.B = operands.as<double>();
    g.a_row = g.b_row = 512;
    g.a_k = g.b_k = 1;
    g.C = out.as<double>();
    g.ldc = 512;
    struct Reset {
        Context &c;
        ~Reset() { c.product_test_spin = 0; }
    } reset{c};
    c.product_test_spin = spin_cycles;
    gemm64(c, g, scales);
    cudaStreamSynchronize(c.stream);  // before the buffers go
    UGPU_ABI_END(ctx ? &ctx->impl : nullptr)
}
