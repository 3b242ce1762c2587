// TRecon preparation kernels:
//   k_trecon_convert  planeToFloat of the frame and its neighbours
//                     (tReconGetFrame's extract, src/plugin.cpp:771-790)
//   k_trecon_lc       the neighbours' footprint luma maps (buildLcMap,
//                     src/maps.cpp:425-499)
//   k_block_match     blockMatch, src/algos.cpp:683-755
//   k_chroma_consist  applyChromaConsistency, src/algos.cpp:757-807
//
// Block matching: one CTA per (16x16 block, neighbour). The block's
// subsampled luma (every second row and column) and the neighbour's search
// window sit in shared memory (the window's pitch puts the candidates of a
// warp into different banks); each thread takes candidate displacements in
// scan order and sums |cur - nbr| in the reference's sample order, so every
// candidate's SAD is the reference's float. The block's FP64 statistics, a
// serial chain, are one lane's work of the last warp meanwhile. The
// sequential choice (strictly smaller SAD, or equal SAD with a smaller
// |dx|+|dy|) selects the lexicographic minimum of (SAD, |dx|+|dy|, scan
// index): a 64-bit key (SAD bits, norm, index) reduced with min. Windows
// above kMatchWindowMax samples (tsearch beyond 42) are read from the plane.
//
// Consistency: one CTA per (block, neighbour), one thread per chroma delta;
// the median is the delta whose rank (by counting smaller deltas, then
// earlier equal ones) is the middle one. No sort and one barrier: the padded
// bitonic sort it replaces spent 36 barriers on 64 deltas.
//
// One 1080p 4:2:0 10-bit frame with two neighbours, tsearch 6: matching
// 124 -> 93 us, consistency 119 -> 32 us.
#include "temporal.cuh"
#include "launch.h"
#include "trecon.h"

#include <algorithm>

namespace lgcr_b200 {

namespace {

template <int KIND>
__device__ __forceinline__ float rawFloat(const void *base, long long pitch, int x, int y,
                                          double scale, double off) {
    const char *row = static_cast<const char *>(base) + (long long)y * pitch;
    if (KIND == kU8)
        return (float)((double)__ldg(reinterpret_cast<const unsigned char *>(row) + x) * scale + off);
    if (KIND == kU16)
        return (float)((double)__ldg(reinterpret_cast<const unsigned short *>(row) + x) * scale + off);
    return __ldg(reinterpret_cast<const float *>(row) + x) + 0.0f;   // s * 1.0 + 0.0
}

// Four consecutive samples of a row from one vector load where the address
// allows it.
template <int KIND>
__device__ __forceinline__ bool rawFloat4(const void *base, long long pitch, int x, int y, double scale,
                                          double off, float4 &v) {
    const char *row = static_cast<const char *>(base) + (long long)y * pitch;
    constexpr int bytes = KIND == kF32 ? 4 : (KIND == kU16 ? 2 : 1);
    const char *p = row + (size_t)x * bytes;
    if (reinterpret_cast<uintptr_t>(p) & (4 * bytes - 1))
        return false;
    if (KIND == kF32) {
        const float4 q = __ldg(reinterpret_cast<const float4 *>(p));
        v = make_float4(q.x + 0.0f, q.y + 0.0f, q.z + 0.0f, q.w + 0.0f);
        return true;
    }
    uint32_t r[4];
    if (KIND == kU16) {
        const ushort4 q = __ldg(reinterpret_cast<const ushort4 *>(p));
        r[0] = q.x; r[1] = q.y; r[2] = q.z; r[3] = q.w;
    } else {
        const uchar4 q = __ldg(reinterpret_cast<const uchar4 *>(p));
        r[0] = q.x; r[1] = q.y; r[2] = q.z; r[3] = q.w;
    }
    v = make_float4((float)((double)r[0] * scale + off), (float)((double)r[1] * scale + off),
                    (float)((double)r[2] * scale + off), (float)((double)r[3] * scale + off));
    return true;
}

// blockIdx.y: frame * 3 + plane; a warp takes row segments of 128 samples,
// four per lane (rows and columns from the warp's place: a flat 64-bit index
// and its division per sample took twice the time of the copy, 28 -> 16 us
// for three 1080p frames).
template <int KIND>
__global__ void __launch_bounds__(256) k_trecon_convert(const TReconPrep P) {
    gridDependency();
    const int frame = blockIdx.y / 3, plane = blockIdx.y % 3;
    const int w = plane ? P.cw : P.sw, h = plane ? P.ch : P.sh;
    const double off = plane ? P.cOffset : 0.0;
    float *dst = P.f[frame][plane];
    const void *src = P.in[frame][plane];
    const long long pitch = P.inPitch[frame][plane];
    const int segs = (w + 127) / 128, total = segs * h;
    const int lane = threadIdx.x & 31;
    for (int g = blockIdx.x * 8 + (threadIdx.x >> 5); g < total; g += gridDim.x * 8) {
        const int y = g / segs, x = (g - y * segs) * 128 + lane * 4;
        if (x >= w)
            continue;
        float *o = dst + (size_t)y * w + x;
        float4 v;
        if (x + 4 <= w && !(reinterpret_cast<uintptr_t>(o) & 15) &&
            rawFloat4<KIND>(src, pitch, x, y, P.yScale, off, v)) {
            *reinterpret_cast<float4 *>(o) = v;
            continue;
        }
        for (int k = 0; k < 4 && x + k < w; ++k)
            o[k] = rawFloat<KIND>(src, pitch, x + k, y, P.yScale, off);
    }
}

// blockIdx.y: neighbour - 1; a warp takes row segments of 32 samples
__global__ void __launch_bounds__(256) k_trecon_lc(const TReconPrep P) {
    gridDependency();
    const int k = 1 + blockIdx.y;
    const float *Y = P.f[k][0];
    float *lc = P.lc[k];
    const int segs = (P.cw + 31) / 32, total = segs * P.ch;
    for (int g = blockIdx.x * 8 + (threadIdx.x >> 5); g < total; g += gridDim.x * 8) {
        const int cy = g / segs, cx = (g - cy * segs) * 32 + (threadIdx.x & 31);
        if (cx >= P.cw)
            continue;
        const int xb = __ldg(P.lcXb + cx), xe = __ldg(P.lcXe + cx);
        const int yb = __ldg(P.lcYb + cy), ye = __ldg(P.lcYe + cy);
        double sum = 0.0;
        for (int j = yb; j < ye; ++j)
            for (int x = xb; x < xe; ++x)
                sum += (double)ldf(Y + (size_t)j * P.sw + x);
        lc[(size_t)cy * P.cw + cx] = footprintMean(sum, xe - xb, ye - yb);
    }
}

constexpr int kMatchThreads = 256;          // most threads of a matching block
constexpr int kMatchWindowMax = 11776;      // floats of the staged search window (46 KB)

// Width, height and pitch of the search window: candidates of one warp lie
// side by side in rows of 2 * search + 1, so a pitch congruent to that modulo
// 32 gives a warp's candidates consecutive banks.
__host__ __device__ __forceinline__ void matchWindow(int search, int &extent, int &pitch) {
    const int side = 2 * search + 1;
    extent = kTReconBlock - 1 + side;
    pitch = extent + ((side - extent) % 32 + 32) % 32;
}

// blockIdx.x: block index, blockIdx.y: neighbour - 1
template <bool STAGED>
__global__ void __launch_bounds__(kMatchThreads) k_block_match(const TReconPrep P) {
    gridDependency();
    extern __shared__ float win[];
    __shared__ __align__(16) float cur[kTReconBlock / 2][kTReconBlock / 2];
    __shared__ unsigned long long best[kMatchThreads / 32];
    __shared__ double stats[2];
    __shared__ float sad0Shared;
    const int k = 1 + blockIdx.y;
    const int bx = blockIdx.x % P.bw, by = blockIdx.x / P.bw;
    const int w = P.sw, h = P.sh;
    const int x0 = bx * kTReconBlock, y0 = by * kTReconBlock;
    const int bw_ = min(kTReconBlock, w - x0), bh_ = min(kTReconBlock, h - y0);
    const int ni = (bw_ + 1) / 2, nj = (bh_ + 1) / 2;
    const float *C = P.f[0][0], *N = P.f[k][0];
    const int s = P.search, side = 2 * s + 1, cands = side * side;
    for (int t = threadIdx.x; t < ni * nj; t += blockDim.x) {
        const int i = t % ni, j = t / ni;
        cur[j][i] = ldf(C + (size_t)(y0 + 2 * j) * w + x0 + 2 * i);
    }
    int extent, pitch;
    matchWindow(s, extent, pitch);
    if (STAGED) {
        // positions outside the plane are not read by any candidate
        const int lane = threadIdx.x & 31;
        for (int r = threadIdx.x >> 5; r < extent; r += blockDim.x >> 5) {
            const int y = y0 - s + r;
            if (y < 0 || y >= h)
                continue;
            for (int c = lane; c < extent; c += 32) {
                const int x = x0 - s + c;
                if (x >= 0 && x < w)
                    win[r * pitch + c] = ldf(N + (size_t)y * w + x);
            }
        }
    }
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) {
        // subsampled block statistics in the reference's order
        double sum = 0.0, sum2 = 0.0;
        for (int j = 0; j < nj; ++j)
            for (int i = 0; i < ni; ++i) {
                const float v = cur[j][i];
                sum += v;
                sum2 += (double)v * v;
            }
        stats[0] = sum;
        stats[1] = sum2;
    }
    unsigned long long key = ~0ull;
    for (int c = threadIdx.x; c < cands; c += blockDim.x) {
        const int dy = c / side - s, dx = c % side - s;
        if (x0 + dx < 0 || y0 + dy < 0 || x0 + dx + bw_ > w || y0 + dy + bh_ > h)
            continue;
        const float *nb = STAGED ? win + (dy + s) * pitch + dx + s : N + (size_t)(y0 + dy) * w + x0 + dx;
        const int step = 2 * (STAGED ? pitch : w);
        float sad = 0.0f;
        if (STAGED && ni == kTReconBlock / 2) {
            for (int j = 0; j < nj; ++j, nb += step) {
                const float4 a = reinterpret_cast<const float4 *>(cur[j])[0];
                const float4 b = reinterpret_cast<const float4 *>(cur[j])[1];
                const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    sad += fabsf(v[i] - nb[2 * i]);
            }
        } else {
            for (int j = 0; j < nj; ++j, nb += step)
                for (int i = 0; i < ni; ++i)
                    sad += fabsf(cur[j][i] - nb[2 * i]);
        }
        if (dx == 0 && dy == 0)
            sad0Shared = sad;
        const unsigned norm = (unsigned)(abs(dx) + abs(dy));
        const unsigned long long kk = ((unsigned long long)__float_as_uint(sad) << 32) |
                                      ((unsigned long long)norm << 16) | (unsigned long long)c;
        key = kk < key ? kk : key;
    }
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long other = __shfl_down_sync(0xffffffffu, key, o);
        key = other < key ? other : key;
    }
    if ((threadIdx.x & 31) == 0)
        best[threadIdx.x >> 5] = key;
    __syncthreads();
    if (threadIdx.x != 0)
        return;
    for (int q = 1; q < (int)(blockDim.x >> 5); ++q)
        key = best[q] < key ? best[q] : key;
    const int c = (int)(key & 0xffffu);
    int bdy = c / side - s, bdx = c % side - s;
    float bestSad = __uint_as_float((unsigned)(key >> 32));
    const float sad0 = sad0Shared;
    const double sum = stats[0], sum2 = stats[1];
    const float npix = (float)(ni * nj);
    // zero-motion snap
    if ((bdx != 0 || bdy != 0) && sad0 - bestSad <= 0.10f * P.tsad * npix) {
        bdx = 0;
        bdy = 0;
        bestSad = sad0;
    }
    const size_t idx = (size_t)by * P.bw + bx;
    P.mvx[k][idx] = (short)bdx;
    P.mvy[k][idx] = (short)bdy;
    const float sadPx = bestSad / npix;
    const double m = sum / npix;
    const double vr = sum2 / npix - m * m;
    const float var = (float)(0.0 < vr ? vr : 0.0);
    const float invT2 = 1.0f / (P.tsad * P.tsad);
    const float matchQ = 1.0f / (1.0f + sadPx * sadPx * invT2);
    const float uniq = var / (var + 0.25f * P.tsad * P.tsad);
    P.conf[k][idx] = matchQ * uniq;
}

constexpr int kConsistMax = 256;            // 16 x 16 deltas at most (4:4:4)

// Blocks of the smallest multiple of 32 threads that gives every delta one.
__global__ void __launch_bounds__(kConsistMax) k_chroma_consist(const TReconPrep P) {
    gridDependency();
    __shared__ __align__(16) unsigned d[kConsistMax];
    __shared__ unsigned middle[2];
    const int k = 1 + blockIdx.y;
    const int bx = blockIdx.x % P.bw, by = blockIdx.x / P.bw;
    const size_t bi = (size_t)by * P.bw + bx;
    const float conf = P.conf[k][bi];
    if (conf <= 0.0f)
        return;                                      // uniform over the block
    const int cw = P.cw, ch = P.ch;
    const int lx0 = bx * kTReconBlock, ly0 = by * kTReconBlock;
    const int lx1 = min(P.sw, lx0 + kTReconBlock), ly1 = min(P.sh, ly0 + kTReconBlock);
    const int cx0 = iclamp((int)floor(lx0 / P.rw), 0, cw - 1);
    const int cy0 = iclamp((int)floor(ly0 / P.rh), 0, ch - 1);
    const int cx1 = iclamp((int)ceil(lx1 / P.rw), cx0 + 1, cw);
    const int cy1 = iclamp((int)ceil(ly1 / P.rh), cy0 + 1, ch);
    const double mx = P.mvx[k][bi] / P.rw, my = P.mvy[k][bi] / P.rh;
    const int nx = cx1 - cx0, n = nx * (cy1 - cy0);
    if (n > (int)blockDim.x)
        return;                                      // not reachable: TRecon ratios are 1..2
    const float *cu = P.f[0][1], *cv = P.f[0][2], *nu = P.f[k][1], *nv = P.f[k][2];
    const int t = threadIdx.x;
    // non-negative floats order as their bits; ~0 pads the last vector
    unsigned mine = ~0u;
    if (t < n) {
        const int cx = cx0 + t % nx, cy = cy0 + t / nx;
        const int tx = iclamp((int)llround(cx + mx), 0, cw - 1);
        const int ty = iclamp((int)llround(cy + my), 0, ch - 1);
        const size_t o = (size_t)cy * cw + cx, q = (size_t)ty * cw + tx;
        mine = __float_as_uint(smax(fabsf(ldf(cu + o) - ldf(nu + q)), fabsf(ldf(cv + o) - ldf(nv + q))));
    }
    d[t] = mine;
    __syncthreads();
    if (t < n) {
        int rank = 0;
        for (int j = 0; j < n; j += 4) {
            const uint4 v = *reinterpret_cast<const uint4 *>(d + j);
            rank += (v.x < mine || (v.x == mine && j < t)) + (v.y < mine || (v.y == mine && j + 1 < t)) +
                    (v.z < mine || (v.z == mine && j + 2 < t)) + (v.w < mine || (v.w == mine && j + 3 < t));
        }
        if (rank == n / 2)
            middle[1] = mine;
        if (rank == n / 2 - 1)
            middle[0] = mine;
    }
    __syncthreads();
    if (t != 0)
        return;
    float median = __uint_as_float(middle[1]);
    if ((n & 1) == 0)
        median = 0.5f * (__uint_as_float(middle[0]) + median);
    const float ratio = median / 0.04f;
    const float ratio2 = ratio * ratio;
    const float cconf = 1.0f / (1.0f + ratio2 * ratio2);
    P.conf[k][bi] = conf * cconf;
}

__global__ void k_trecon_lanczos(double *tabX, double *tabY, double rw, double rh, float invWx, float invWy,
                                 double support) {
    gridDependency();
    const int i = threadIdx.x;
    const float d = (float)i / (float)kTLanSteps;
    tabX[i] = temporalLanczos(d, rw, invWx, support);
    tabY[i] = temporalLanczos(d, rh, invWy, support);
}

template <int KIND>
void convertKind(const TReconPrep &P, cudaStream_t s) {
    const int segs = (P.sw + 127) / 128 * P.sh;
    launchAfter(k_trecon_convert<KIND>, dim3(std::min((segs + 7) / 8, 1184), 3 * P.frames), 256, 0, s, P);
}

} // namespace

void launchTReconLanczos(double *tabX, double *tabY, double rw, double rh, float invWx, float invWy,
                         double support, cudaStream_t s) {
    launchAfter(k_trecon_lanczos, 1, kTLanEntries, 0, s, tabX, tabY, rw, rh, invWx, invWy, support);
}

int launchTReconPrep(const TReconPrep &P, cudaStream_t s) {
    const int nbrs = P.frames - 1;
    if (nbrs <= 0)
        return 0;
    switch (P.kind) {
    case kU8: convertKind<kU8>(P, s); break;
    case kU16: convertKind<kU16>(P, s); break;
    default: convertKind<kF32>(P, s); break;
    }
    const int segs = (P.cw + 31) / 32 * P.ch;
    launchAfter(k_trecon_lc, dim3(std::min((segs + 7) / 8, 1184), nbrs), 256, 0, s, P);
    int extent, pitch;
    matchWindow(P.search, extent, pitch);
    const int window = extent * pitch;
    const int cands = (2 * P.search + 1) * (2 * P.search + 1);
    const int threads = std::min(kMatchThreads, (cands + 31) / 32 * 32);
    if (window <= kMatchWindowMax)
        launchAfter(k_block_match<true>, dim3(P.bw * P.bh, nbrs), threads, window * sizeof(float), s, P);
    else
        launchAfter(k_block_match<false>, dim3(P.bw * P.bh, nbrs), threads, 0, s, P);
    // chroma samples of a luma block, at most one more per axis than its share
    const int perX = std::min(kTReconBlock, (int)(kTReconBlock / P.rw) + 2);
    const int perY = std::min(kTReconBlock, (int)(kTReconBlock / P.rh) + 2);
    const bool whole = P.rw == 2.0 && P.rh == 2.0;
    const int deltas = whole ? kTReconBlock * kTReconBlock / 4 : perX * perY;
    launchAfter(k_chroma_consist, dim3(P.bw * P.bh, nbrs), (deltas + 31) / 32 * 32, 0, s, P);
    return cudaGetLastError() == cudaSuccess ? 4 : -1;
}

} // namespace lgcr_b200
