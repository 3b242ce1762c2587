// Sharpen: gated bilateral unsharp mask over a 5x5 window, the reference's
// second filter (sharpenGetFrame src/plugin.cpp:14-76, sharpenPlane
// src/algos.cpp:595-659).
//
// Per sample: the window's guide range max|g - L0| and sample hull, a sigma
// floor from the median of the four neighbour differences, then 24 taps with
// n = sp(i, j) * sim(dL), out = c0 + alpha * sum(n * (c0 - s)) / sum(n),
// clamped to the hull +- ar. Luma guides itself; subsampled chroma is guided
// by the footprint-average map of the already sharpened luma (lc) with the
// reference point bilinear on that luma at the sample's left-sited position;
// 4:4:4 chroma guides itself.
//
// Layout: one block sharpens a 32 x 16 tile, two rows per thread; guided
// chroma blocks do U and V together. The source tile and a 2-sample halo
// (clamped coordinates, as the reference's Plane::at) are converted from the
// raw input into shared memory once; for guided chroma the lc tile with its
// halo is built in shared memory from the sharpened luma. All float arithmetic
// follows the reference's order (the library is compiled without FMA
// contraction); the 1/(1 + ...) quotients use the reciprocal refinement that
// equals the IEEE quotient on [1, 2^64).
//
// Bound by issue (24 similarity taps per sample). What is the same for every
// tap or sample is outside the taps: the spatial factors come from the host,
// the reciprocal's range check is made once per sample at its window's range
// (rounding is monotonic, so that bounds every tap), a self-guided sample's
// range follows from its hull and its tap difference from the guide's, and
// the two chroma planes share the guide tile. 1080p 4:2:0 10-bit: luma 66 ->
// 41 us, chroma 54 -> 34 us (43 at the 96 registers it takes unasked, half the
// warps).
#include "launch.h"
#include "sharpen.h"

namespace lgcr_b200 {

namespace {

constexpr int kTx = 32, kTy = 16, kThreadsY = 8, kHalo = 2;
constexpr int kLx = kTx + 2 * kHalo, kLy = kTy + 2 * kHalo;

template <int KIND>
__device__ __forceinline__ float loadSample(const SharpenJob &J, int plane, int x, int y) {
    const char *row = static_cast<const char *>(J.in[plane]) + (long long)y * J.inPitch[plane];
    const double off = (plane == 0 || KIND == kF32) ? 0.0 : J.cOffset;
    if (KIND == kU8)
        return (float)((double)__ldg(reinterpret_cast<const unsigned char *>(row) + x) * J.yScale + off);
    if (KIND == kU16)
        return (float)((double)__ldg(reinterpret_cast<const unsigned short *>(row) + x) * J.yScale + off);
    return __ldg(reinterpret_cast<const float *>(row) + x) + 0.0f;   // s * 1.0 + 0.0
}

__device__ __forceinline__ void storeSample(const SharpenJob &J, int plane, int x, int y, float v) {
    char *row = static_cast<char *>(J.out[plane]) + (long long)y * J.outPitch[plane];
    if (J.kind == kF32) {
        reinterpret_cast<float *>(row)[x] = v + 0.0f;          // s * 1.0 + 0.0
        return;
    }
    const int q = quantize(v, J.qScale, plane == 0 ? 0.0f : J.qOffC, J.maxCode);
    if (J.kind == kU8) reinterpret_cast<uint8_t *>(row)[x] = (uint8_t)q;
    else reinterpret_cast<uint16_t *>(row)[x] = (uint16_t)q;
}

// reference bilinear (src/lgcr.h:467-475) at a position given in double
__device__ __forceinline__ float bilinearD(const float *p, int w, int h, double x, double y) {
    const double flx = floor(x), fly = floor(y);
    const int x0 = (int)flx, y0 = (int)fly;
    const float fx = (float)(x - (double)x0);
    const float fy = (float)(y - (double)y0);
    const int xa = iclamp(x0, 0, w - 1), xb = iclamp(x0 + 1, 0, w - 1);
    const int ya = iclamp(y0, 0, h - 1), yb = iclamp(y0 + 1, 0, h - 1);
    const float a = ldf(p + (size_t)ya * w + xa), b = ldf(p + (size_t)ya * w + xb);
    const float c = ldf(p + (size_t)yb * w + xa), d = ldf(p + (size_t)yb * w + xb);
    return a + (b - a) * fx + (c - a) * fy + (a - b - c + d) * fx * fy;
}

// Weighted sums of one sample over its 24 taps: hp = sum n * (c0 - s), wsum =
// sum n. SELF: the sample guides itself, so c0 - s is minus the guide
// difference. CHECKED: a denominator may reach 2^64.
template <bool SELF, bool CHECKED>
__device__ __forceinline__ void sharpenTaps(const SharpenJob &J, const float *S, const float *G, int c,
                                            float c0, float L0, float invS2, float &hp, float &wsum) {
#pragma unroll
    for (int j = -2; j <= 2; ++j)
#pragma unroll
        for (int i = -2; i <= 2; ++i) {
            if (i == 0 && j == 0)
                continue;
            const int o = c + j * kLx + i;
            const float dL = G[o] - L0;
            const float xs = 1.0f + dL * dL * invS2;
            const float sim = CHECKED ? rcpAtLeastOne(xs) : rcpInRange(xs);
            const float n = J.spatial[i * i + j * j] * sim;
            if (SELF)
                hp -= n * dL;
            else
                hp += n * (c0 - S[o]);
            wsum += n;
        }
}

template <bool SELF>
__device__ __noinline__ void sharpenTapsChecked(const SharpenJob &J, const float *S, const float *G, int c,
                                                float c0, float L0, float invS2, float &hp, float &wsum) {
    sharpenTaps<SELF, true>(J, S, G, c, c0, L0, invS2, hp, wsum);
}

// One sample of sharpenPlane. S: source tile, G: guide tile (S itself when
// SELF), both kLx wide with the sample at c; maxAbsDL: the window's guide range
// (not used when SELF).
template <bool SELF>
__device__ __forceinline__ float sharpenSample(const SharpenJob &J, const float *S, const float *G, int c,
                                               float L0, float maxAbsDL) {
    const float c0 = S[c];
    float hullMin = 1e30f, hullMax = -1e30f;
#pragma unroll
    for (int j = -2; j <= 2; ++j)
#pragma unroll
        for (int i = -2; i <= 2; ++i) {
            const float v = S[c + j * kLx + i];
            hullMin = runMin(hullMin, v);
            hullMax = runMax(hullMax, v);
        }
    if (SELF)                                            // max |s - c0| over the window
        maxAbsDL = smax(smax(0.0f, fabsf(hullMax - c0)), fabsf(hullMin - c0));
    // median of the four neighbour differences: the middle two of a sorted
    // four are max(min pair) and min(max pair)
    const float d0 = fabsf(S[c + 1] - c0), d1 = fabsf(S[c - 1] - c0);
    const float d2 = fabsf(S[c + kLx] - c0), d3 = fabsf(S[c - kLx] - c0);
    const float lo = smax(smin(d0, d1), smin(d2, d3));
    const float hi = smin(smax(d0, d1), smax(d2, d3));
    const float slopeMed = (lo + hi) * 0.5f;
    const float sig = smax(smax(J.sigma, J.sratio * maxAbsDL), 3.0f * slopeMed);
    const float invS2 = 1.0f / (sig * sig);
    float hp = 0.0f, wsum = 0.0f;
    if (1.0f + maxAbsDL * maxAbsDL * invS2 < kRcpFastLimit)
        sharpenTaps<SELF, false>(J, S, G, c, c0, L0, invS2, hp, wsum);
    else
        sharpenTapsChecked<SELF>(J, S, G, c, c0, L0, invS2, hp, wsum);
    float out = c0;
    if (wsum > 1e-6f)
        out = c0 + J.alpha * hp / wsum;
    if (J.clampHull)
        out = sclamp(out, hullMin - J.margin, hullMax + J.margin);
    return out;
}

// Self-guided planes: luma (blockIdx.z == 0) and, for 4:4:4, both chroma
// planes (blockIdx.z == 1, 2). Luma also writes the float sharpened plane
// the chroma guide reads.
template <int KIND>
__global__ void __launch_bounds__(kTx * kThreadsY)
k_sharpen_self(const __grid_constant__ SharpenJob J) {
    gridDependency();
    __shared__ float S[kLx * kLy];
    const int plane = blockIdx.z;
    const int w = plane == 0 ? J.sw : J.cw, h = plane == 0 ? J.sh : J.ch;
    const int x0 = blockIdx.x * kTx, y0 = blockIdx.y * kTy;
    if (x0 >= w || y0 >= h)
        return;
    for (int k = threadIdx.y * kTx + threadIdx.x; k < kLx * kLy; k += kTx * kThreadsY) {
        const int lx = k % kLx, ly = k / kLx;
        S[k] = loadSample<KIND>(J, plane, iclamp(x0 + lx - kHalo, 0, w - 1),
                                iclamp(y0 + ly - kHalo, 0, h - 1));
    }
    __syncthreads();
    const int x = x0 + threadIdx.x;
    if (x >= w)
        return;
#pragma unroll 1
    for (int ty = threadIdx.y; ty < kTy && y0 + ty < h; ty += kThreadsY) {
        const int c = (ty + kHalo) * kLx + threadIdx.x + kHalo, y = y0 + ty;
        const float v = sharpenSample<true>(J, S, S, c, S[c], 0.0f);
        if (plane == 0 && J.Ys)
            J.Ys[(size_t)y * J.sw + x] = v;
        storeSample(J, plane, x, y, v);
    }
}

// Subsampled chroma guided by the sharpened luma, both planes.
template <int KIND>
__global__ void __launch_bounds__(kTx * kThreadsY, 4)
k_sharpen_chroma(const __grid_constant__ SharpenJob J) {
    gridDependency();
    __shared__ float S[2][kLx * kLy];
    __shared__ float G[kLx * kLy];
    const int w = J.cw, h = J.ch;
    const int x0 = blockIdx.x * kTx, y0 = blockIdx.y * kTy;
    for (int k = threadIdx.y * kTx + threadIdx.x; k < kLx * kLy; k += kTx * kThreadsY) {
        const int lx = k % kLx, ly = k / kLx;
        const int cx = iclamp(x0 + lx - kHalo, 0, w - 1), cy = iclamp(y0 + ly - kHalo, 0, h - 1);
        S[0][k] = loadSample<KIND>(J, 1, cx, cy);
        S[1][k] = loadSample<KIND>(J, 2, cx, cy);
        // lc: raster-order double sum of the sharpened luma over the
        // sample's footprint (buildLcMap src/maps.cpp:425-499)
        const int xb = __ldg(J.lcXb + cx), xe = __ldg(J.lcXe + cx);
        const int yb = __ldg(J.lcYb + cy), ye = __ldg(J.lcYe + cy);
        double sum = 0.0;
        for (int yy = yb; yy < ye; ++yy)
            for (int xx = xb; xx < xe; ++xx)
                sum += (double)ldf(J.Ys + (size_t)yy * J.sw + xx);
        G[k] = footprintMean(sum, xe - xb, ye - yb);
    }
    __syncthreads();
    const int x = x0 + threadIdx.x;
    if (x >= w)
        return;
#pragma unroll 1
    for (int ty = threadIdx.y; ty < kTy && y0 + ty < h; ty += kThreadsY) {
        const int c = (ty + kHalo) * kLx + threadIdx.x + kHalo, y = y0 + ty;
        const float L0 = bilinearD(J.Ys, J.sw, J.sh, ((double)x + 0.5) * J.rw - 0.5 + J.shiftX,
                                   ((double)y + 0.5) * J.rh - 0.5 + J.shiftY);
        float mn = 1e30f, mx = -1e30f;                   // the guide's range
#pragma unroll
        for (int j = -2; j <= 2; ++j)
#pragma unroll
            for (int i = -2; i <= 2; ++i) {
                mn = runMin(mn, G[c + j * kLx + i]);
                mx = runMax(mx, G[c + j * kLx + i]);
            }
        const float range = smax(smax(0.0f, fabsf(mx - L0)), fabsf(mn - L0));
#pragma unroll 1
        for (int p = 0; p < 2; ++p)
            storeSample(J, 1 + p, x, y, sharpenSample<false>(J, S[p], G, c, L0, range));
    }
}

template <int KIND>
cudaError_t launchKind(const SharpenJob &J, cudaStream_t s) {
    const dim3 block(kTx, kThreadsY);
    const bool guided = J.guided != 0;
    const int planes = guided ? 1 : 3;
    const int gw = guided ? J.sw : max(J.sw, J.cw), gh = guided ? J.sh : max(J.sh, J.ch);
    launchAfter(k_sharpen_self<KIND>, dim3((gw + kTx - 1) / kTx, (gh + kTy - 1) / kTy, planes), block, 0, s, J);
    if (guided)
        launchAfter(k_sharpen_chroma<KIND>, dim3((J.cw + kTx - 1) / kTx, (J.ch + kTy - 1) / kTy), block, 0, s, J);
    return cudaGetLastError();
}

} // namespace

cudaError_t launchSharpen(const SharpenJob &J, cudaStream_t s) {
    switch (J.kind) {
    case kU8: return launchKind<kU8>(J, s);
    case kU16: return launchKind<kU16>(J, s);
    default: return launchKind<kF32>(J, s);
    }
}

} // namespace lgcr_b200
