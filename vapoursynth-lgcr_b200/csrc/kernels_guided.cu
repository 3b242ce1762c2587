// Guided reconstruction by horizontal pixel pairs (reconstructChromaImpl,
// src/recon.cpp:14-819), the main form of the guided pass:
//   k_pair_extrema   jinc frames: pass 1 of both pixels of a pair with the
//                    plain base (separable frames have both from k_plain)
//   k_guide_setup    per listed pixel: guide, direction, edge probes, range
//                    sigma, fades and rescue weight, to the context planes
//   k_guided_pair    pass 2 of both pixels of a pair and the final sample
//   k_guided_pair_r  the same with jinc base weights
// Frames whose windows do not pair (PairAxis in geometry.h), the bilinear
// kernel and wide supports take the one-pixel form in kernels_recon.cu.
//
// What bounds it: the latency of dependent loads in the setup, instruction
// issue in the taps. The one-pixel kernel does both at 128 registers (16
// warps per SM) and spends more than half of its time in the setup; here the
// setup has a kernel of its own with twice the warps in flight and hands over
// 32 bytes per pixel. In the tap loop a thread owns output columns 2p and
// 2p + 1 of one row:
//  * both windows lie in one window of at most kPairMaxSup columns, so a tap's
//    luma and (u, v) are loaded once for the two pixels (the FP64 pair is four
//    L1 wavefronts per warp load);
//  * the similarity of both pixels runs in the two lanes of the f32x2
//    instructions, with rcp.approx of the negated denominator so that the
//    Newton step needs no sign flips;
//  * the bump term is evaluated for the columns that have a rescue weight
//    (left-sited 4:2:0 and 4:2:2 columns 2p + 1 lie half a sample off and have
//    none: the term was multiplied by zero there), or a direction that is not
//    finite (NaN or overflowing float luma), whose bump times zero is NaN;
//  * the sum of |w| of the fallback test is not accumulated: it is bounded by
//    the kernel's own negative weight, and a pair that the bound does not
//    clear is evaluated again with the sum.
// Measured: 1080p lanczos4 4:2:0 (55 % listed) 202 us for the one-pixel kernel,
// 53 + 129 here; 1080p -> 4K jinc selector, 16-bit, 1800 us before, 392
// (extrema) + 312 (setup) + 766 (pairs). Register budgets of 4 to 8 blocks per
// SM measured within 5 % of each other for k_guided_pair, 6 blocks 7 % better
// than 4 for k_guided_pair_r; one merged kernel was slower than the pixel form
// on separable frames. shapeJobs has the sizes from which this form is taken.
// Both forms write the fused products of the packed tap arithmetic out as
// fma2, the same ones, so both give the same bits.
#include "guided.cuh"

namespace lgcr_b200 {

namespace {

constexpr int kPairThreads = 128;
constexpr int kPairMaxFrames = 1024;

// -1/x on both lanes for 1 <= x < 2^64: rcpInRange's refinement evaluated on
// the negated approximation, e = 1 + x*y and y + y*e with y = -1/x (every
// rounding is that of the positive form, sign flipped).
__device__ __forceinline__ float negRcp(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(-x));
    const float e = __fmaf_rn(x, y, 1.0f);
    return __fmaf_rn(y, e, y);
}
__device__ __forceinline__ f32x2 negRcp2(f32x2 x, f32x2 one) {
    float x0, x1, y0, y1;
    up2(x, x0, x1);
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y0) : "f"(-x0));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y1) : "f"(-x1));
    const f32x2 y = pk2(y0, y1);
    const f32x2 e = fma2(x, y, one);
    return fma2(y, e, y);
}

// bilinear blend of four corners, each operation rounded by itself
__device__ __forceinline__ float blend1(float a, float b, float c, float d, float fx, float fy) {
    return a + (b - a) * fx + (c - a) * fy + (a - b - c + d) * fx * fy;
}

// floor(x) for |x| < 2^22 as an integer; the float floor goes to fl. The add
// rounds toward minus infinity, so the low mantissa bits of the sum are the
// floor's.
__device__ __forceinline__ int floorBits(float x, float &fl) {
    const float m = __fadd_rd(x, 12582912.0f);           // 1.5 * 2^23
    fl = m - 12582912.0f;
    return __float_as_int(m) - 0x4B400000;
}

// Bilinear sample of the luma plane at a probe position whose four corners lie
// inside the plane. The floor is a round-down add: FRND and F2I share the XU
// pipe with the reciprocals.
__device__ __forceinline__ float probeInside(const float *__restrict__ p, int w, float x, float y) {
    float flx, fly;
    const int x0 = floorBits(x, flx), y0 = floorBits(y, fly);
    const float *r = p + (unsigned)(y0 * w + x0);      // planes of up to 65535^2 samples
    return blend1(ldf(r), ldf(r + 1), ldf(r + w), ldf(r + w + 1), x - flx, y - fly);
}

// The same at any position (frame borders), out of line.
__device__ __noinline__ float probeClamped(const float *p, int w, int h, float x, float y) {
    return bilinearAt(p, w, h, x, y);
}

// Context of one listed pixel (k_guide_setup to k_guided_pair): two float4 at
// 2 * (entry's place in the chunk) + column.
//   a = (L0, nx, ny, 1/sigma^2), the last negative when a similarity
//       denominator may reach 2^64
//   b = (fade, rescue, 1/(g * aniso)^2, ssRamp), the third negative when the
//       pixel has no direction
struct PixelContext {
    float4 a, b;
};
__device__ __forceinline__ float withSign(float v, bool negative) {
    return __uint_as_float((__float_as_uint(v) & 0x7fffffffu) | (negative ? 0x80000000u : 0u));
}

// Both pixels of one pair: [0] column 2p, [1] column 2p + 1.
struct Pair {
    float L0[2], nx[2], ny[2], scx[2];
    float invSigma2[2], fade[2], rescue[2], invG2Par[2];
    float scy;
    int tx0, ty0;                 // common window
    int kind;                     // row of the pair weight table
    uint32_t bits, my;            // active taps of both columns, active rows
    bool bump;                    // column 2p + 1 takes the bump term
};

struct PairAcc {
    double u[2], v[2], wsum[2], sumAbs[2];
};

// Pass 2 (recon.cpp:606-623): w = sim * (wbase + rescue * bump) over the
// active taps, accumulated in FP64 in tap order. BOTH: both columns take the
// bump term, else only column 2p. RADIAL: base weights are the pair's
// rows of the jinc phase table (rad), else wx(i) * wy(j). FULL: every column
// but the first and last of the window is active for both pixels (all windows
// away from the frame's sides), so only those two are tested.
template <int UC, bool BOTH, bool RADIAL, bool ABS, bool FULL>
__device__ __forceinline__ void pairTaps(const FrameJob &J, const Pair &c, int oy,
                                         const float2 *__restrict__ rad, PairAcc &acc) {
    const float4 *__restrict__ tab = J.pairTab + (size_t)c.kind * UC;
    const float rh = J.rhF;
    const f32x2 one = pk2(1.0f, 1.0f);
    const f32x2 invS = pk2(c.invSigma2[0], c.invSigma2[1]);
    const f32x2 nfade = pk2(-c.fade[0], -c.fade[1]);
    const float g2 = J.invGsigma2;
    const int cw = J.cw;
    const uint32_t be = c.bits & 0xffffu, bo = c.bits >> 16;
    const float *lrow = J.lc + (size_t)c.ty0 * cw + c.tx0;
    const double2 *uvrow = reinterpret_cast<const double2 *>(J.uvd) + (size_t)c.ty0 * cw + c.tx0;
    const float *wyp = RADIAL ? nullptr : J.ay.w + (size_t)oy * J.ay.sup;
    const int rows = J.ay.sup;
#pragma unroll 1
    for (int j = 0; j < rows; ++j, lrow += cw, uvrow += cw) {
        if (!((c.my >> j) & 1u))
            continue;
        const float dy = ((float)(c.ty0 + j) - c.scy) * rh;
        const float wy = RADIAL ? 0.0f : __ldg(wyp + j);
        const float dyn0 = dy * c.ny[0], dyt0 = dy * c.nx[0];
        const float dyn1 = dy * c.ny[1], dyt1 = dy * c.nx[1];
#pragma unroll
        for (int i = 0; i < UC; ++i) {
            const double2 s = __ldg(uvrow + i);
            const float l = ldf(lrow + i);
            const f32x2 dL = pk2(l - c.L0[0], l - c.L0[1]);
            const f32x2 nsim = negRcp2(fma2(mul2(dL, dL), invS, one), one);
            const f32x2 sim = fma2(nfade, add2(one, nsim), one);
            // weights and tap distances of both columns
            const float4 t = __ldg(tab + i);
            // wbase + rescue * bump, one rounding for the last product and sum
            f32x2 base;
            if (BOTH) {
                const f32x2 dp = pk2(t.z * c.nx[0] + dyn0, t.w * c.nx[1] + dyn1);
                const f32x2 dt = pk2(-t.z * c.ny[0] + dyt0, -t.w * c.ny[1] + dyt1);
                const f32x2 xb = fma2(mul2(dt, dt), pk2(c.invG2Par[0], c.invG2Par[1]),
                                      fma2(mul2(dp, dp), pk2(g2, g2), one));
                const f32x2 nresc = pk2(-c.rescue[0], -c.rescue[1]), nb = negRcp2(xb, one);
                if (RADIAL) {
                    const float2 r = __ldg(rad + j * UC + i);
                    base = fma2(nresc, nb, pk2(r.x, r.y));
                } else {
                    base = fma2(pk2(t.x, t.y), pk2(wy, wy), mul2(nresc, nb));
                }
            } else {
                const float dp = t.z * c.nx[0] + dyn0, dt = -t.z * c.ny[0] + dyt0;
                const float xb = __fmaf_rn(dt * dt, c.invG2Par[0], __fmaf_rn(dp * dp, g2, 1.0f));
                const float nb = negRcp(xb);
                if (RADIAL) {
                    const float2 r = __ldg(rad + j * UC + i);
                    base = pk2(__fmaf_rn(-c.rescue[0], nb, r.x), r.y);
                } else {
                    base = pk2(__fmaf_rn(t.x, wy, -c.rescue[0] * nb), t.y * wy);
                }
            }
            float w0, w1;
            up2(mul2(sim, base), w0, w1);
            const bool inner = FULL && i > 0 && i < UC - 1;
            if (inner || ((be >> i) & 1u)) {
                const double wd = (double)w0;
                acc.u[0] = fma(wd, s.x, acc.u[0]);
                acc.v[0] = fma(wd, s.y, acc.v[0]);
                acc.wsum[0] += wd;
                if (ABS)
                    acc.sumAbs[0] += fabs(wd);
            }
            if (inner || ((bo >> i) & 1u)) {
                const double wd = (double)w1;
                acc.u[1] = fma(wd, s.x, acc.u[1]);
                acc.v[1] = fma(wd, s.y, acc.v[1]);
                acc.wsum[1] += wd;
                if (ABS)
                    acc.sumAbs[1] += fabs(wd);
            }
        }
    }
}

// Whether every inner column of a UC-wide window is active for both pixels of
// every pair of the warp.
template <int UC>
__device__ __forceinline__ bool innerColumnsActive(uint32_t bits) {
    constexpr uint32_t inner = ((1u << UC) - 1u) & ~1u & ~(1u << (UC - 1));
    constexpr uint32_t both = inner | inner << 16;
    return __all_sync(__activemask(), (bits & both) == both);
}

template <int UC, bool RADIAL>
__device__ __forceinline__ void pairTapsFor(const FrameJob &J, const Pair &c, int oy,
                                            const float2 *rad, PairAcc &acc) {
    // one variant per warp: lanes without a second bump term lose nothing in BOTH
    const bool both = __any_sync(__activemask(), c.bump);
    if (!innerColumnsActive<UC>(c.bits))
        pairTaps<UC, true, RADIAL, false, false>(J, c, oy, rad, acc);
    else if (both)
        pairTaps<UC, true, RADIAL, false, true>(J, c, oy, rad, acc);
    else
        pairTaps<UC, false, RADIAL, false, true>(J, c, oy, rad, acc);
}

// The pair's sums with sum |w| (kept out of line: few pixels need it).
template <bool RADIAL>
__device__ __noinline__ void exactPair(const FrameJob &J, const Pair &c, int oy, const float2 *rad,
                                       PairAcc &acc) {
#pragma unroll
    for (int q = 0; q < 2; ++q)
        acc.u[q] = acc.v[q] = acc.wsum[q] = acc.sumAbs[q] = 0.0;
    switch (J.pairSup) {
    case 4: pairTaps<4, true, RADIAL, true, false>(J, c, oy, rad, acc); break;
    case 5: pairTaps<5, true, RADIAL, true, false>(J, c, oy, rad, acc); break;
    case 6: pairTaps<6, true, RADIAL, true, false>(J, c, oy, rad, acc); break;
    case 7: pairTaps<7, true, RADIAL, true, false>(J, c, oy, rad, acc); break;
    case 8: pairTaps<8, true, RADIAL, true, false>(J, c, oy, rad, acc); break;
    default: pairTaps<9, true, RADIAL, true, false>(J, c, oy, rad, acc); break;
    }
}

// Sums of one pixel by the general loop (any denominators, with sum |w|).
__device__ __noinline__ Acc exactTaps(const FrameJob &J, int ox, int oy, TapCtx c) {
    Acc a{0.0, 0.0, 0.0, 0.0};
    tapsGeneric(J, c, ox, oy, __ldg(J.ax.start + ox), __ldg(J.ay.start + oy), a);
    return a;
}

// Pass 1 of a jinc pair: luma and chroma extrema and the plain sums of both
// windows (phase-table weights in FP64, tap order). wd: the pair's weights as
// doubles, one (column 2p, column 2p + 1) entry per tap.
struct PairHull {
    float mnL[2], mxL[2], mnU[2], mxU[2], mnV[2], mxV[2];
    double u[2], v[2];
};

template <int UC, bool FULL>
__device__ __forceinline__ void pairHullRows(const FrameJob &J, const Pair &c,
                                             const double2 *__restrict__ wd, PairHull &h) {
    // [0], [1]: the pixels' own columns; [2]: columns active for both (FULL: the
    // inner ones), folded into both at the end (min and max do not care)
    float mnL[3], mxL[3], mnU[3], mxU[3], mnV[3], mxV[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        mnL[q] = mnU[q] = mnV[q] = 1e30f;
        mxL[q] = mxU[q] = mxV[q] = -1e30f;
    }
    double au[2] = {0.0, 0.0}, av[2] = {0.0, 0.0};
    const int cw = J.cw;
    const size_t o = (size_t)c.ty0 * cw + c.tx0;
    const float *lrow = J.lc + o, *urow = J.U + o, *vrow = J.V + o;
    const double2 *uvrow = reinterpret_cast<const double2 *>(J.uvd) + o;
    const int rows = J.ay.sup;
    auto fold = [&](int q, float l, float u, float v) {
        mnL[q] = runMin(mnL[q], l); mxL[q] = runMax(mxL[q], l);
        mnU[q] = runMin(mnU[q], u); mxU[q] = runMax(mxU[q], u);
        mnV[q] = runMin(mnV[q], v); mxV[q] = runMax(mxV[q], v);
    };
#pragma unroll 1
    for (int j = 0; j < rows; ++j, lrow += cw, urow += cw, vrow += cw, uvrow += cw, wd += UC) {
        if (!((c.my >> j) & 1u))
            continue;
#pragma unroll
        for (int i = 0; i < UC; ++i) {
            const float l = ldf(lrow + i), u = ldf(urow + i), v = ldf(vrow + i);
            const double2 s = __ldg(uvrow + i);
            const double2 w = __ldg(wd + i);
            const bool inner = FULL && i > 0 && i < UC - 1;
            if (inner)
                fold(2, l, u, v);
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                if (!inner) {
                    if (!((c.bits >> (i + 16 * q)) & 1u))
                        continue;
                    fold(q, l, u, v);
                }
                const double wq = q ? w.y : w.x;
                au[q] = fma(wq, s.x, au[q]);
                av[q] = fma(wq, s.y, av[q]);
            }
        }
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        h.mnL[q] = runMin(mnL[q], mnL[2]); h.mxL[q] = runMax(mxL[q], mxL[2]);
        h.mnU[q] = runMin(mnU[q], mnU[2]); h.mxU[q] = runMax(mxU[q], mxU[2]);
        h.mnV[q] = runMin(mnV[q], mnV[2]); h.mxV[q] = runMax(mxV[q], mxV[2]);
        h.u[q] = au[q];
        h.v[q] = av[q];
    }
}

template <int UC>
__device__ __forceinline__ void pairHullPlain(const FrameJob &J, const Pair &c,
                                              const double2 *__restrict__ wd, PairHull &h) {
    if (innerColumnsActive<UC>(c.bits))
        pairHullRows<UC, true>(J, c, wd, h);
    else
        pairHullRows<UC, false>(J, c, wd, h);
}

// Two neighbouring samples of one output row; one vector store when both are
// written and the address allows it.
__device__ __forceinline__ void storePair(const FrameJob &J, int plane, int ox, int oy, float a, float b,
                                          bool on0, bool on1) {
    char *row = static_cast<char *>(J.out[plane]) + (long long)oy * J.outPitch[plane];
    if (on0 && on1) {
        if (J.outKind == kF32) {
            float *p = reinterpret_cast<float *>(row) + ox;
            if (!(reinterpret_cast<uintptr_t>(p) & 7)) {
                *reinterpret_cast<float2 *>(p) = make_float2(a + 0.0f, b + 0.0f);
                return;
            }
        } else {
            const int qa = quantize(a, J.qScale, J.qOffC, J.maxCode);
            const int qb = quantize(b, J.qScale, J.qOffC, J.maxCode);
            if (J.outKind == kU16) {
                uint16_t *p = reinterpret_cast<uint16_t *>(row) + ox;
                if (!(reinterpret_cast<uintptr_t>(p) & 3))
                    *reinterpret_cast<uint32_t *>(p) = (uint32_t)qa | (uint32_t)qb << 16;
                else {
                    p[0] = (uint16_t)qa;
                    p[1] = (uint16_t)qb;
                }
            } else {
                uint8_t *p = reinterpret_cast<uint8_t *>(row) + ox;
                if (!(reinterpret_cast<uintptr_t>(p) & 1))
                    *reinterpret_cast<uint16_t *>(p) = (uint16_t)(qa | qb << 8);
                else {
                    p[0] = (uint8_t)qa;
                    p[1] = (uint8_t)qb;
                }
            }
            return;
        }
    }
    if (on0)
        storeChroma(J, plane, ox, oy, a);
    if (on1)
        storeChroma(J, plane, ox + 1, oy, b);
}

__device__ __noinline__ void selectPixel(const FrameJob &J, int ox, int oy, const Guided &g) {
    guidedSelect<true>(J, ox, oy, g);
}

// Axis table entries of both columns of a pair (the packed tables are padded
// past an odd length; an odd width's last column is a pair of itself).
struct PairTables {
    int ox;
    bool two;
    __device__ __forceinline__ float2 f2(const float *t) const {
        float2 v = __ldg(reinterpret_cast<const float2 *>(t + ox));
        if (!two) v.y = v.x;
        return v;
    }
};

// Entry of a pair list: columns to write.
__device__ __forceinline__ void pairColumns(const FrameJob &J, uint32_t e, int &ox, int &oy, bool &on0,
                                            bool &on1) {
    ox = (int)(e & 0xfffeu);
    oy = (int)(e >> 16);
    on0 = on1 = true;
    if (e & 1u) {                                        // one column only
        on0 = pixelActive(J, ox, oy);
        on1 = ox + 1 < J.W && pixelActive(J, ox + 1, oy);
    }
}

// Jinc frames: extrema of both windows to the planes k_plain fills for
// separable frames, and the plain base to the float planes.
struct ExtremaWork {
    static __device__ __forceinline__ bool mine(const FrameJob &J) { return J.pairSup > 0 && J.radial; }
    static constexpr int kPer = 1;                       // threads per list entry
    static constexpr bool kEndShared = true;             // the loop's end is read again (pairGrid)
    static __device__ __forceinline__ void run(const FrameJob &J, unsigned long long idx, unsigned slot) {
        int ox, oy;
        bool on[2];
        pairColumns(J, __ldg(J.actList + idx), ox, oy, on[0], on[1]);
        const PairTables T{ox, ox + 1 < J.W};
        const int p = ox >> 1;
        Pair c;
        const float2 pos = T.f2(J.ax.pos);
        c.scy = __ldg(J.ay.pos + oy);
        c.tx0 = __ldg(J.pairStart + p);
        c.kind = __ldg(J.pairKind + p);
        c.bits = __ldg(J.pairBits + p);
        c.ty0 = __ldg(J.ay.start + oy);
        c.my = __ldg(J.ay.amBits + oy);
        const int yp = __ldg(J.rad.yPhase + oy);
        const double2 *wd = J.pairRadD + ((size_t)yp * J.pairPhases + __ldg(J.pairPhase + p)) *
                                             ((size_t)J.ay.sup * J.pairSup);
        PairHull h;
        switch (J.pairSup) {
        case 4: pairHullPlain<4>(J, c, wd, h); break;
        case 5: pairHullPlain<5>(J, c, wd, h); break;
        case 6: pairHullPlain<6>(J, c, wd, h); break;
        case 7: pairHullPlain<7>(J, c, wd, h); break;
        case 8: pairHullPlain<8>(J, c, wd, h); break;
        default: pairHullPlain<9>(J, c, wd, h); break;
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            if (!on[q])
                continue;
            // the plain base's finish (plainRadialTable in plain.cuh)
            const double2 sums = __ldg(J.radSums + (size_t)yp * J.rad.phasesX +
                                       __ldg(J.rad.xPhase + ox + q));     // sum w, sum |w|
            double v0, v1;
            if (sums.x > 1e-6 && sums.x >= 0.05 * sums.y) {
                v0 = h.u[q] / sums.x;
                v1 = h.v[q] / sums.x;
            } else {
                v0 = probeClamped(J.U, J.cw, J.ch, q ? pos.y : pos.x, c.scy);
                v1 = probeClamped(J.V, J.cw, J.ch, q ? pos.y : pos.x, c.scy);
            }
            if (J.clampHull) {
                v0 = sclamp(v0, (double)(h.mnU[q] - J.margin), (double)(h.mxU[q] + J.margin));
                v1 = sclamp(v1, (double)(h.mnV[q] - J.margin), (double)(h.mxV[q] + J.margin));
            }
            const size_t o = (size_t)oy * J.W + ox + q;
            J.pairHull[2 * slot + q] = make_float4(h.mnU[q], h.mxU[q], h.mnV[q], h.mxV[q]);
            J.pairLum[2 * slot + q] = make_float2(h.mnL[q], h.mxL[q]);
            J.oU[o] = (float)v0;
            J.oV[o] = (float)v1;
        }
    }
};

// Guide metadata, range sigma, fades and rescue weight of one listed pixel
// (recon.cpp:155-475), one thread per pixel.
struct SetupWork {
    static __device__ __forceinline__ bool mine(const FrameJob &J) { return J.pairSup > 0; }
    static constexpr int kPer = 2;
    static constexpr bool kEndShared = false;
    static __device__ __forceinline__ void run(const FrameJob &J, unsigned long long idx, unsigned slot) {
        const uint32_t e = __ldg(J.actList + (idx >> 1));
        const int ox = (int)(e & 0xfffeu) + (int)(idx & 1u), oy = (int)(e >> 16);
        if (ox >= J.W || ((e & 1u) && !pixelActive(J, ox, oy)))
            return;
        const AxisView &ax = J.ax, &ay = J.ay;
        const int sw = J.sw, sh = J.sh;
        const float2 lum = J.radial ? J.pairLum[slot] : J.wLum[(size_t)oy * J.W + ox];
        const float lx = __ldg(ax.lpos + ox), ly = __ldg(ay.lpos + oy);
        const float lcN = ldf(J.lc + (size_t)__ldg(ay.nearest + oy) * J.cw + __ldg(ax.nearest + ox));
        float mutualFade = 1.0f;
        if (J.useMs) {
            const float gate = bilinearFast(J.ms, J.cw, J.ch, __ldg(ax.cbI0 + ox), __ldg(ax.cbF + ox),
                                            __ldg(ay.cbI0 + oy), __ldg(ay.cbF + oy));
            mutualFade = 1.0f - J.msStrength * (1.0f - gate);
        }
        float L0, jxx, jxy, jyy;
        if (J.guideOnGrid && ox + 1 < sw && oy + 1 < sh) {
            // same-size integer frames: the positions are the samples themselves
            // (the table's last index is a fraction of 1, which rounds its blend)
            const size_t o = (size_t)oy * sw + ox;
            L0 = ldf(J.Y + o);
            jxx = ldf(J.jxx + o);
            jxy = ldf(J.jxy + o);
            jyy = ldf(J.jyy + o);
        } else {
            const int bx = __ldg(ax.lbI0 + ox), by = __ldg(ay.lbI0 + oy);
            const float bxf = __ldg(ax.lbF + ox), byf = __ldg(ay.lbF + oy);
            L0 = bilinearFast(J.Y, sw, sh, bx, bxf, by, byf);
            jxx = bilinearFast(J.jxx, sw, sh, bx, bxf, by, byf);
            jxy = bilinearFast(J.jxy, sw, sh, bx, bxf, by, byf);
            jyy = bilinearFast(J.jyy, sw, sh, bx, bxf, by, byf);
        }
        const TensorDir dir = principalDirection(jxx, jxy, jyy);
        const bool hasDir = jxx + jyy > 1e-6f;
        const float nx = dir.nx, ny = dir.ny;
        float minDiffN = 0.0f, ridgeRev = 0.0f;
        if (hasDir) {
            const float sp = J.spOut, dl = 1.5f * sp;
            const float reach = 2.0f * dl + 3.0f;     // 2 dl along a unit normal, plus a corner
            float yA, yB, ym2 = L0, ym1 = L0, yp1 = L0, yp2 = L0;
            if (lx >= reach && lx <= (float)(sw - 1) - reach && ly >= reach &&
                ly <= (float)(sh - 1) - reach && fabsf(nx) <= 1.01f && fabsf(ny) <= 1.01f) {
                yA = probeInside(J.Y, sw, lx - sp * nx, ly - sp * ny);
                yB = probeInside(J.Y, sw, lx + sp * nx, ly + sp * ny);
                if (J.ridge) {
                    ym2 = probeInside(J.Y, sw, lx - 2.0f * dl * nx, ly - 2.0f * dl * ny);
                    ym1 = probeInside(J.Y, sw, lx - dl * nx, ly - dl * ny);
                    yp1 = probeInside(J.Y, sw, lx + dl * nx, ly + dl * ny);
                    yp2 = probeInside(J.Y, sw, lx + 2.0f * dl * nx, ly + 2.0f * dl * ny);
                }
            } else {
                yA = probeClamped(J.Y, sw, sh, lx - sp * nx, ly - sp * ny);
                yB = probeClamped(J.Y, sw, sh, lx + sp * nx, ly + sp * ny);
                if (J.ridge) {
                    ym2 = probeClamped(J.Y, sw, sh, lx - 2.0f * dl * nx, ly - 2.0f * dl * ny);
                    ym1 = probeClamped(J.Y, sw, sh, lx - dl * nx, ly - dl * ny);
                    yp1 = probeClamped(J.Y, sw, sh, lx + dl * nx, ly + dl * ny);
                    yp2 = probeClamped(J.Y, sw, sh, lx + 2.0f * dl * nx, ly + 2.0f * dl * ny);
                }
            }
            minDiffN = smin(fabsf(yA - L0), fabsf(yB - L0));
            if (J.ridge) {
                const float diff[4] = {ym1 - ym2, L0 - ym1, yp1 - L0, yp2 - yp1};
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const float a = diff[k], b = diff[k + 1];
                    if (a > 0.0f && b < 0.0f)
                        ridgeRev = smax(ridgeRev, smin(a, -b));
                    if (a < 0.0f && b > 0.0f)
                        ridgeRev = smax(ridgeRev, smin(-a, b));
                }
            }
        }
        float m = 0.0f;                                  // max |lc - L0| over the window
        m = smax(m, fabsf(lum.y - L0));
        m = smax(m, fabsf(lum.x - L0));
        const float t2 = sclamp(divZeroSafe(minDiffN, 0.1f * m + 1e-6f), 0.0f, 1.0f);
        const float ssRamp = t2 * t2 * (3.0f - 2.0f * t2);
        const float sigMult = J.sratio + (J.sdb - J.sratio) * ssRamp;
        const float sigLoc = smax(J.sigma, sigMult * m);
        const float invSigma2 = 1.0f / (sigLoc * sigLoc);
        const float ridgeFade = 1.0f - sclamp(divZeroSafe(2.0f * ridgeRev, m + 1e-6f), 0.0f, 1.0f);
        const float fade = ridgeFade * mutualFade * J.strength;
        // phase-0 rescue with kappa^2 (recon.cpp:425-475)
        const float phaseGate = __ldg(ax.pgate + ox) * __ldg(ay.pgate + oy);
        const float dL0 = lcN - L0;
        const float sim0 = rcpAtLeastOne(1.0f + dL0 * dL0 * invSigma2);
        float rescue = J.rescue * fade * phaseGate * phaseGate * (1.0f - sim0);
        if (rescue > 0.0f) {
            float kappa;
            if (J.radial) {
                kappa = ldf(J.rad.kappa + (size_t)__ldg(J.rad.yPhase + oy) * J.rad.phasesX +
                            __ldg(J.rad.xPhase + ox));
            } else {
                const float mxX = __ldg(ax.kmx + ox), ssX = __ldg(ax.kss + ox);
                const float mxY = __ldg(ay.kmx + oy), ssY = __ldg(ay.kss + oy);
                kappa = (mxX * mxX * mxY * mxY) / (ssX * ssY + 1e-12f);
            }
            rescue *= kappa * kappa;
        }
        const float aniso = 1.0f + J.stretch * dir.coherence;
        const float g2p = J.invGsigma2 / (aniso * aniso);
        // every tap's similarity denominator is at most this (see guidedPixel)
        const bool safe = (1.0f + m * m * invSigma2) < kRcpFastLimit;
        J.context[2 * slot] = make_float4(L0, nx, ny, withSign(invSigma2, !safe));
        J.context[2 * slot + 1] = make_float4(fade, rescue, withSign(g2p, !hasDir), ssRamp);
    }
};

// Pass 2 and the final sample of one pair.
template <bool RADIAL>
struct PairWork {
    static __device__ __forceinline__ bool mine(const FrameJob &J) {
        return J.pairSup > 0 && (J.radial != 0) == RADIAL;
    }
    static constexpr int kPer = 1;
    static constexpr bool kEndShared = RADIAL;
    static __device__ __forceinline__ void run(const FrameJob &J, unsigned long long idx, unsigned slot) {
        int ox, oy;
        bool on[2];
        pairColumns(J, __ldg(J.actList + idx), ox, oy, on[0], on[1]);
        const PairTables T{ox, ox + 1 < J.W};
        const int p = ox >> 1, cw = J.cw;
        Pair c;
        bool safe[2];
        float g2p[2];
        const float2 pos = T.f2(J.ax.pos);
        c.scx[0] = pos.x;
        c.scx[1] = pos.y;
        c.scy = __ldg(J.ay.pos + oy);
        c.tx0 = __ldg(J.pairStart + p);
        c.kind = __ldg(J.pairKind + p);
        c.bits = __ldg(J.pairBits + p);
        c.ty0 = __ldg(J.ay.start + oy);
        c.my = __ldg(J.ay.amBits + oy);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const float4 a = __ldg(J.context + 4 * slot + 2 * q), b = __ldg(J.context + 4 * slot + 2 * q + 1);
            c.L0[q] = a.x; c.nx[q] = a.y; c.ny[q] = a.z;
            safe[q] = __float_as_int(a.w) >= 0;
            c.invSigma2[q] = fabsf(a.w);
            c.fade[q] = b.x;
            c.rescue[q] = on[q] ? b.y : 0.0f;            // a skipped column's context is not written
            g2p[q] = b.z;
            c.invG2Par[q] = fabsf(b.z);
        }
        c.bump = on[1] && !(c.rescue[1] == 0.0f && fabsf(c.nx[1]) <= 2.0f && fabsf(c.ny[1]) <= 2.0f &&
                            c.invG2Par[1] >= 0.0f);
        const float2 *rad = nullptr;
        if (RADIAL)
            rad = J.pairRad + ((size_t)__ldg(J.rad.yPhase + oy) * J.pairPhases + __ldg(J.pairPhase + p)) *
                                  ((size_t)J.ay.sup * J.pairSup);
        PairAcc acc;
#pragma unroll
        for (int q = 0; q < 2; ++q)
            acc.u[q] = acc.v[q] = acc.wsum[q] = 0.0;
        switch (J.pairSup) {
        case 4: pairTapsFor<4, RADIAL>(J, c, oy, rad, acc); break;
        case 5: pairTapsFor<5, RADIAL>(J, c, oy, rad, acc); break;
        case 6: pairTapsFor<6, RADIAL>(J, c, oy, rad, acc); break;
        case 7: pairTapsFor<7, RADIAL>(J, c, oy, rad, acc); break;
        case 8: pairTapsFor<8, RADIAL>(J, c, oy, rad, acc); break;
        default: pairTapsFor<9, RADIAL>(J, c, oy, rad, acc); break;
        }
        // Negative taps have base weight below zero (the rescue term only
        // adds) and a similarity of at most one, so sum |w| <= sum w + bound,
        // the kernel's own sum |w| - sum w: when the fallback test holds with
        // the bound it holds with the sum.
        double bound[2];
        if (RADIAL) {
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const double2 sums = __ldg(J.radSums + (size_t)__ldg(J.rad.yPhase + oy) * J.rad.phasesX +
                                           __ldg(J.rad.xPhase + (q && T.two ? ox + 1 : ox)));
                bound[q] = (sums.y - sums.x) + 1e-4 * sums.y;
            }
        } else {
            const float2 ws = T.f2(J.ax.wsum), wa = T.f2(J.ax.wabs);
            const float wsY = __ldg(J.ay.wsum + oy), waY = __ldg(J.ay.wabs + oy);
            const float sa0 = wa.x * waY, sa1 = wa.y * waY;
            bound[0] = (double)((sa0 - ws.x * wsY) + 1e-4f * sa0);
            bound[1] = (double)((sa1 - ws.y * wsY) + 1e-4f * sa1);
        }
        const size_t o = (size_t)oy * J.W + ox;
        float4 hull[2];
        const float4 *hulls = RADIAL ? J.pairHull + 2 * slot : J.wHull + o;
        hull[0] = __ldg(hulls);
        hull[1] = __ldg(hulls + (T.two ? 1 : 0));
        Acc sums[2];
        bool good[2];
        // TRecon: the neighbours' motion-compensated samples follow the spatial
        // taps in the same accumulators and extend the hull. Then the fallback test.
        auto close = [&](int q) {
            if (!RADIAL && J.tnbCount > 0 && on[q]) {
                const float ssRamp = J.context[4 * slot + 2 * q + 1].w;
                const float2 lum = __ldg(J.wLum + o + q);
                const float m = smax(smax(0.0f, fabsf(lum.y - c.L0[q])), fabsf(lum.x - c.L0[q]));
                const float sigLoc = smax(J.sigma, (J.sratio + (J.sdb - J.sratio) * ssRamp) * m);
                TemporalAcc t{sums[q].u, sums[q].v, sums[q].wsum, sums[q].sumAbs,
                              hull[q].x, hull[q].y, hull[q].z, hull[q].w};
                t = temporalTaps(J, ox + q, oy, c.L0[q], c.scx[q], c.scy, sigLoc, c.fade[q], ssRamp, t);
                sums[q] = Acc{t.u, t.v, t.wsum, t.sumAbs};
                hull[q] = make_float4(t.mnU, t.mxU, t.mnV, t.mxV);
            }
            good[q] = sums[q].wsum > 1e-6 && sums[q].wsum >= 0.05 * sums[q].sumAbs;
        };
        bool redo = false;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            sums[q] = Acc{acc.u[q], acc.v[q], acc.wsum[q], acc.wsum[q] + bound[q]};
            if (on[q] && !safe[q]) {
                TapCtx t;
                t.lc = J.lc;
                t.uv = reinterpret_cast<const double2 *>(J.uvd);
                t.cw = cw; t.ch = J.ch;
                t.L0 = c.L0[q]; t.nx = c.nx[q]; t.ny = c.ny[q]; t.scx = c.scx[q]; t.scy = c.scy;
                t.rwF = J.rwF; t.rhF = J.rhF;
                t.invSigma2 = c.invSigma2[q]; t.guideFade = c.fade[q]; t.rescue = c.rescue[q];
                t.invG2 = J.invGsigma2; t.invG2Par = c.invG2Par[q];
                sums[q] = exactTaps(J, ox + q, oy, t);
            }
            close(q);
            redo = redo || (on[q] && safe[q] && !good[q]);
        }
        if (redo) {
            const Pair copy = c;                         // the call's own: c stays in registers
            PairAcc e;
            exactPair<RADIAL>(J, copy, oy, rad, e);
#pragma unroll
            for (int q = 0; q < 2; ++q)
                if (safe[q] && !good[q]) {               // the hull keeps its temporal extension
                    sums[q] = Acc{e.u[q], e.v[q], e.wsum[q], e.sumAbs[q]};
                    close(q);
                }
        }
        float outU[2], outV[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            double valueU, valueV;
            if (good[q]) {
                if (J.inKind != kF32) {
                    const double r = __drcp_rn(sums[q].wsum);
                    valueU = quotientBy(sums[q].u, sums[q].wsum, r);
                    valueV = quotientBy(sums[q].v, sums[q].wsum, r);
                } else {                                 // float samples may be infinite
                    valueU = sums[q].u / sums[q].wsum;
                    valueV = sums[q].v / sums[q].wsum;
                }
            } else {
                valueU = probeClamped(J.U, cw, J.ch, c.scx[q], c.scy);
                valueV = probeClamped(J.V, cw, J.ch, c.scx[q], c.scy);
            }
            if (J.clampHull) {
                valueU = sclamp(valueU, (double)(hull[q].x - J.margin), (double)(hull[q].y + J.margin));
                valueV = sclamp(valueV, (double)(hull[q].z - J.margin), (double)(hull[q].w + J.margin));
            }
            outU[q] = (float)valueU;
            outV[q] = (float)valueV;
            if ((RADIAL || J.algo != 2) && on[q]) {
                Guided g;
                g.u = valueU; g.v = valueV;
                g.L0 = c.L0[q]; g.ssRamp = J.context[4 * slot + 2 * q + 1].w; g.guideFade = c.fade[q];
                g.nx = c.nx[q]; g.ny = c.ny[q]; g.hasDir = __float_as_int(g2p[q]) >= 0;
                g.havePlain = RADIAL;
                g.plainU = g.plainV = 0.0f;
                if (RADIAL) {
                    g.plainU = J.oU[o + q];
                    g.plainV = J.oV[o + q];
                }
                selectPixel(J, ox + q, oy, g);
            }
        }
        if (RADIAL || J.algo != 2)
            return;
        if (J.directOutput) {
            storePair(J, 1, ox, oy, outU[0], outU[1], on[0], on[1]);
            storePair(J, 2, ox, oy, outV[0], outV[1], on[0], on[1]);
            return;
        }
#pragma unroll
        for (int q = 0; q < 2; ++q)
            if (on[q]) {
                J.oU[o + q] = outU[q];
                J.oV[o + q] = outV[q];
            }
    }
};

// Persistent grid over the entries [first, first + pairChunk) of the
// concatenated lists of the launch's frames: blocks stride over them side by
// side, so the rows in flight stay close together in L2 (one contiguous share
// per block measured 10 % slower on 4K frames). The descriptor of the current
// frame is kept in shared memory. An entry's place in the chunk, the same for
// every kernel, is where the scratch holds its contexts and extrema.
template <class Work>
__device__ __forceinline__ void pairGrid(const FrameJob *__restrict__ jobs, int njobs,
                                         unsigned long long first) {
    __shared__ unsigned long long pre[kPairMaxFrames + 1];
    __shared__ FrameJob sJob;
    __shared__ int sChunk;
    __shared__ unsigned long long sEnd;
    const int tid = threadIdx.x;
    if (tid == 0)
        pre[0] = 0ull;
    for (int chunk = 0; chunk < njobs; chunk += kPairMaxFrames) {
        const int n = min(kPairMaxFrames, njobs - chunk);
        __syncthreads();
        if (tid == 0 && chunk > 0)
            pre[0] = pre[kPairMaxFrames];                // after the frames before this part
        __syncthreads();
        for (int i = tid; i < n; i += kPairThreads) {
            const FrameJob &J = jobs[chunk + i];
            pre[i + 1] = J.pairSup > 0 ? J.counters[kCntPairs] * Work::kPer : 0ull;
            if (J.pairSup > 0)
                sChunk = J.pairChunk;                    // one value for all frames
        }
        __syncthreads();
        if (tid == 0) {
            unsigned long long acc = pre[0];
            for (int i = 1; i <= n; ++i)
                pre[i] = acc += pre[i];
            sEnd = min(acc, (first + (unsigned)sChunk) * Work::kPer);
        }
        __syncthreads();
        int staged = -1, f = 0;
        // jinc work has no register left for the end (held there, the extrema
        // spill: 406 us on one 4K frame, 392 read from shared memory); separable
        // work does (one dense 1438x1079 4:2:2 frame 311 us, 319 with the read)
        const unsigned long long held = sEnd;
        const volatile unsigned long long &shared = sEnd;
        auto end = [&] { return Work::kEndShared ? shared : held; };
        for (unsigned long long lo = max(pre[0], first * Work::kPer) +
                                     (unsigned long long)blockIdx.x * kPairThreads;
             lo < end(); lo += (unsigned long long)gridDim.x * kPairThreads) {
            const unsigned long long hi = min(lo + kPairThreads, end());
            while (pre[f + 1] <= lo)
                ++f;
            for (int g = f; g < n && pre[g] < hi; ++g) {
                if (pre[g + 1] == pre[g])
                    continue;
                if (g != staged) {
                    if (!Work::mine(jobs[chunk + g]))
                        continue;
                    __syncthreads();
                    stageJob(jobs, chunk + g, sJob);
                    staged = g;
                }
                const unsigned long long w = lo + tid;
                if (w >= pre[g] && w < pre[g + 1] && w < hi)
                    Work::run(sJob, w - pre[g], (unsigned)(w - first * Work::kPer));
            }
        }
    }
}

} // namespace

__global__ void __launch_bounds__(kPairThreads, 5)
k_pair_extrema(const FrameJob *__restrict__ jobs, const int *__restrict__ tileStart, int njobs,
               unsigned long long first) {
    gridDependency();
    (void)tileStart;
    pairGrid<ExtremaWork>(jobs, njobs, first);
}

__global__ void __launch_bounds__(kPairThreads, 8)
k_guide_setup(const FrameJob *__restrict__ jobs, const int *__restrict__ tileStart, int njobs,
              unsigned long long first) {
    gridDependency();
    (void)tileStart;
    pairGrid<SetupWork>(jobs, njobs, first);
}

__global__ void __launch_bounds__(kPairThreads, 4)
k_guided_pair(const FrameJob *__restrict__ jobs, const int *__restrict__ tileStart, int njobs,
              unsigned long long first) {
    gridDependency();
    (void)tileStart;
    pairGrid<PairWork<false>>(jobs, njobs, first);
}

__global__ void __launch_bounds__(kPairThreads, 6)
k_guided_pair_r(const FrameJob *__restrict__ jobs, const int *__restrict__ tileStart, int njobs,
                unsigned long long first) {
    gridDependency();
    (void)tileStart;
    pairGrid<PairWork<true>>(jobs, njobs, first);
}

} // namespace lgcr_b200
