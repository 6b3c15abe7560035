// quotients_check.cu -- compares the quotients and roots of ieee64.cuh with / and sqrt, bit for bit, over their
// stated domain (built and run by test_gpu_fp64_domain.py).
#include <cstdint>

#include "../nemo_b200/csrc/ieee64.cuh"

using namespace nemo;

// mismatches: quotients next to a rounding tie, random quotients, quotients by one shared reciprocal, random roots,
// pairs near powers of two, roots near powers of two; and how many of the first kind were made
__device__ unsigned long long g_bad[7];

__device__ uint64_t next(uint64_t& s) {   // splitmix64
    s += 0x9E3779B97F4A7C15ull;
    uint64_t z = s;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

__device__ bool same(double x, double y) { return __double_as_longlong(x) == __double_as_longlong(y); }

__device__ void check(double a, double b, int kind) {
    if (!same(div64(a, b), a / b)) atomicAdd(&g_bad[kind], 1ull);
}

// 2^e times a random significand (one time in four with its upper or lower half all ones), random sign
__device__ double number(uint64_t& s, int e, bool negative) {
    uint64_t m = next(s) >> 12;
    const unsigned k = (unsigned)(next(s) & 7);
    if (k == 0) m |= 0xfffffffffull << 16;
    if (k == 1) m |= 0xfffffffffull;
    return __longlong_as_double((long long)(m | (uint64_t)(1023 + e) << 52 | (uint64_t)(negative ? 1 : 0) << 63));
}

__device__ int exponent(uint64_t& s, int lo, int hi) { return lo + (int)(next(s) % (uint64_t)(hi - lo + 1)); }

__global__ void k_check(int rounds, uint64_t seed) {
    uint64_t s = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) * 7919 + seed;
    for (int it = 0; it < rounds; ++it) {
        // a/b within 2^-107 or so of a tie: M B = A 2^54 - k for an odd 54-bit M, |k| <= 6, by the inverse of B
        uint64_t B = (next(s) >> 11) | (1ull << 52) | 1;
        if (it % 4 == 0) B |= ((1ull << 52) - 1) ^ ((1ull << 44) - 1);
        uint64_t inv = B;
        for (int i = 0; i < 6; ++i) inv *= 2 - B * inv;
        const double b = scalbn((double)B, -52);
        for (int k = -6; k <= 6; ++k) {
            if (k == 0) continue;
            for (int half = 0; half < 2; ++half) {   // quotient below and above one
                const int bits = 54 - half;
                const uint64_t M = (((uint64_t)(-(int64_t)k) * inv) & ((1ull << bits) - 1)) | (half ? 1ull << 53 : 0);
                if (!(M & 1) || !(M >> 53)) continue;
                const unsigned __int128 x = (unsigned __int128)M * B + (unsigned __int128)(__int128)k;
                const uint64_t A = (uint64_t)(x >> bits);
                if ((A >> 52) != 1) continue;
                check(scalbn((double)A, -52), b, 0);
                atomicAdd(&g_bad[6], 1ull);
            }
        }
        // random quotients over the whole domain
        const int eb = exponent(s, -999, 998);
        const int eq = exponent(s, max(-900, -950 - eb), min(900, 1000 - eb));
        const double rb = number(s, eb, next(s) & 1), ra = number(s, eb + eq, next(s) & 1);
        check(ra, rb, 1);
        check(0.0, fabs(rb), 1);
        const Rcp64 r = rcp64r(rb);
        for (int j = 0; j < 4; ++j) {
            const double a2 = number(s, eb + eq, next(s) & 1);
            if (!same(quot64(a2, r), a2 / rb)) atomicAdd(&g_bad[2], 1ull);
        }
        const double q = number(s, exponent(s, -900, 1000), false);
        if (!same(sqrt64(q), sqrt(q))) atomicAdd(&g_bad[3], 1ull);
        const double p = __longlong_as_double((1023ll + exponent(s, -6, 6) << 52) + exponent(s, -4000, 4000));
        if (!same(sqrt64(p), sqrt(p)) || !same(sqrt64(0.0), 0.0)) atomicAdd(&g_bad[5], 1ull);
    }
}

// all pairs within n ulp of 1 and 2
__global__ void k_pairs(int n) {
    const int64_t side = 4 * n, i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= side * side) return;
    auto at = [&](int64_t j) {
        return __longlong_as_double(__double_as_longlong(j < 2 * n ? 1.0 : 2.0) + j % (2 * n) - n);
    };
    check(at(i / side), at(i % side), 4);
}

extern "C" int quotients_check(int rounds, int pairs, unsigned long long* bad) {
    k_check<<<148 * 4, 256>>>(rounds, 13);
    const long long side = 4ll * pairs;
    k_pairs<<<(unsigned)((side * side + 255) / 256), 256>>>(pairs);
    return (int)cudaMemcpyFromSymbol(bad, g_bad, sizeof g_bad);
}
