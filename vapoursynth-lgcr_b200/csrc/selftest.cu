// Device self-checks exported through the C ABI.
//   lgcr_selftest_reciprocal: rcpAtLeastOne (the guided taps' reciprocal of
//   1 + non-negative terms) against the IEEE quotient 1.0f / x for every
//   float x in [1, +inf] (2^30 + 1 arguments: the fast range [1, 2^64) and
//   the IEEE-division range above it), bit for bit.
//   lgcr_selftest_quotients: quotientBy (quotients of one FP64 denominator)
//   against n / d over 2^30 seeded pairs, a quarter of them with mantissas of
//   trailing zeros or ones, and downRangeWeight against the division for every
//   float of its range, bit for bit.
#include "impl.h"
#include "recon.cuh"

#include <cstring>

using namespace lgcr_b200;

namespace {

__global__ void k_check_reciprocal(uint32_t lo, uint32_t hi, unsigned long long *bad) {
    unsigned long long local = 0;
    for (uint64_t b = lo + (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; b <= hi;
         b += (uint64_t)gridDim.x * blockDim.x) {
        const float x = __uint_as_float((uint32_t)b);
        if (__float_as_uint(rcpAtLeastOne(x)) != __float_as_uint(1.0f / x))
            ++local;
    }
    if (local)
        atomicAdd(bad, local);
}

// splitmix64 of a counter
__device__ __forceinline__ uint64_t mix(uint64_t x) {
    x += 0x9e3779b97f4a7c15ull;
    x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
    x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
    return x ^ (x >> 31);
}

// A normal double with an exponent in [lo, lo + span) and a mantissa of random
// bits, or random leading bits followed by zeros or ones.
__device__ __forceinline__ double drawDouble(uint64_t seed, int lo, int span, bool edge) {
    const uint64_t a = mix(seed), b = mix(a);
    uint64_t mant = a & ((1ull << 52) - 1);
    if (edge) {
        const uint64_t low = (1ull << (b >> 8 & 63) % 53) - 1;
        mant = (b & 1) ? mant | low : mant & ~low;
    }
    const uint64_t expo = (uint64_t)(1023 + lo + (int)((b >> 16) % (unsigned)span));
    return __longlong_as_double((long long)(expo << 52 | mant));
}

// n: sums of weighted samples, either sign, down to 2^-60; d: sums of weights
// from 1e-6 to 256 (the guided and plain sums, and the counts of a window)
__global__ void k_check_quotients(uint64_t count, unsigned long long *bad) {
    unsigned long long local = 0;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const bool edge = (i & 3) == 3;
        double n = drawDouble(2 * i, -60, 72, edge);
        const double d = drawDouble(2 * i + 1, -20, 28, edge);
        if (mix(i) & 1)
            n = -n;
        const double q = quotientBy(n, d, __drcp_rn(d));
        if (__double_as_longlong(q) != __double_as_longlong(n / d))
            ++local;
    }
    if (local)
        atomicAdd(bad, local);
}

__global__ void k_check_range_weight(uint32_t lo, uint32_t hi, unsigned long long *bad) {
    unsigned long long local = 0;
    for (uint64_t b = lo + (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; b < hi;
         b += (uint64_t)gridDim.x * blockDim.x) {
        const float d = __uint_as_float((uint32_t)b);
        if (__float_as_uint(downRangeWeight(d)) != __float_as_uint(kDownRangeScale2 / d))
            ++local;
    }
    if (local)
        atomicAdd(bad, local);
}

// Runs `launch(blocks, counters)` and reads the counters back.
template <int N, class Launch>
int countMismatches(uint64_t (&out)[N], const char *where, Launch launch) {
    unsigned long long *d = nullptr, h[N] = {};
    cudaError_t e = cudaMalloc(&d, sizeof(h));
    if (e != cudaSuccess)
        return cudaFail(e, where);
    e = cudaMemset(d, 0, sizeof(h));
    if (e == cudaSuccess) {
        int dev = 0, sms = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        launch(sms * 8, d);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess)
        e = cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost);
    cudaFree(d);
    if (e != cudaSuccess)
        return cudaFail(e, where);
    for (int i = 0; i < N; ++i)
        out[i] = h[i];
    return LGCR_OK;
}

} // namespace

extern "C" int lgcr_selftest_reciprocal(uint64_t *mismatches) {
    if (!mismatches)
        return LGCR_E_ARGUMENT;
    uint64_t bad[1] = {0};
    const int status = countMismatches(bad, "lgcr_selftest_reciprocal", [](int blocks, unsigned long long *d) {
        k_check_reciprocal<<<blocks, 256>>>(0x3f800000u, 0x7f800000u, d);
    });
    if (status == LGCR_OK)
        *mismatches = bad[0];
    return status;
}

extern "C" int lgcr_selftest_quotients(uint64_t *mismatches) {
    if (!mismatches)
        return LGCR_E_ARGUMENT;
    uint64_t bad[2] = {0, 0};
    const int status = countMismatches(bad, "lgcr_selftest_quotients", [](int blocks, unsigned long long *d) {
        const float lo = kDownRangeScale2, hi = 8.0f;
        uint32_t loBits, hiBits;
        std::memcpy(&loBits, &lo, sizeof(lo));
        std::memcpy(&hiBits, &hi, sizeof(hi));
        k_check_quotients<<<blocks, 256>>>(1ull << 30, d);
        k_check_range_weight<<<blocks, 256>>>(loBits, hiBits, d + 1);
    });
    if (status == LGCR_OK) {
        mismatches[0] = bad[0];
        mismatches[1] = bad[1];
    }
    return status;
}
