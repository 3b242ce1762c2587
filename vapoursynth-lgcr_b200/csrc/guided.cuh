// Device functions shared by the guided kernels: the plain base of a listed
// pixel, the final store, and one guided tap in its scalar form (the general
// loop over any support, which is also the exact path of the rare pixels the
// unrolled loops leave out).
#pragma once

#include "kernels.cuh"
#include "plain.cuh"
#include "temporal.cuh"

namespace lgcr_b200 {

// Plain separable value from the horizontal table (vertical pass).
template <int SUP>
__device__ __forceinline__ void plainFromTableT(const FrameJob &J, int ox, int oy, float &outU,
                                                float &outV) {
    const AxisView &ax = J.ax, &ay = J.ay;
    const int n = SUP > 0 ? SUP : ay.sup;
    const int ty0 = __ldg(ay.start + oy);
    const double *wy = ay.wd + (size_t)oy * ay.sup;
    const uint8_t *amy = ay.am + (size_t)oy * ay.sup;
    double vU = 0.0, vV = 0.0;
    float mnU = 1e30f, mxU = -1e30f, mnV = 1e30f, mxV = -1e30f;
#pragma unroll
    for (int j = 0; j < n; ++j) {
        if (__ldg(amy + j) == 0)
            continue;
        const int sy = J.noClampY ? ty0 + j : iclamp(ty0 + j, 0, J.ch - 1);
        const float4 *h = reinterpret_cast<const float4 *>(J.hTab + ((size_t)sy * J.W + ox) * 8);
        const float4 a = __ldg(h), b = __ldg(h + 1);
        const double w = __ldg(wy + j);
        vU = fma(w, (double)a.x, vU);
        vV = fma(w, (double)a.y, vV);
        mnU = runMin(mnU, a.z); mxU = runMax(mxU, a.w);
        mnV = runMin(mnV, b.x); mxV = runMax(mxV, b.y);
    }
    const double ws = (double)__ldg(ax.wsum + ox) * (double)__ldg(ay.wsum + oy);
    const double wa = (double)__ldg(ax.wabs + ox) * (double)__ldg(ay.wabs + oy);
    if (ws > 1e-6 && ws >= 0.05 * wa) {
        vU /= ws;
        vV /= ws;
    } else {
        const float px = __ldg(ax.pos + ox), py = __ldg(ay.pos + oy);
        vU = bilinearAt(J.U, J.cw, J.ch, px, py);
        vV = bilinearAt(J.V, J.cw, J.ch, px, py);
    }
    if (J.clampHull) {
        vU = sclamp(vU, (double)(mnU - J.margin), (double)(mxU + J.margin));
        vV = sclamp(vV, (double)(mnV - J.margin), (double)(mxV + J.margin));
    }
    outU = (float)vU;
    outV = (float)vV;
}

__device__ __forceinline__ void plainFromTable(const FrameJob &J, int ox, int oy, float &u, float &v) {
    switch (J.ay.sup) {
    case 4: plainFromTableT<4>(J, ox, oy, u, v); break;
    case 6: plainFromTableT<6>(J, ox, oy, u, v); break;
    case 8: plainFromTableT<8>(J, ox, oy, u, v); break;
    default: plainFromTableT<0>(J, ox, oy, u, v); break;
    }
}

__device__ __forceinline__ void plainPixel(const FrameJob &J, int ox, int oy, float &u, float &v) {
    if (!J.radial && J.kernel != 0 && J.hTab)
        plainFromTable(J, ox, oy, u, v);
    else
        plainAt(chromaPlainCtx(J), ox, oy, u, v);
}

__device__ __forceinline__ bool pixelActive(const FrameJob &J, int ox, int oy) {
    if (!J.sparse)
        return true;
    const int mx = J.sameSize ? ox : min(J.sw - 1, maskIndex(ox, J.sw, J.W));
    const int my = J.sameSize ? oy : min(J.sh - 1, maskIndex(oy, J.sh, J.H));
    return maskAt(J, mx, my) != 0;
}

// Final sample of one output pixel: to the typed output plane when this
// stage is the last one touching it, else to the float planes.
__device__ __forceinline__ void emit(const FrameJob &J, int ox, int oy, float u, float v) {
    if (J.directOutput) {
        storeChroma(J, 1, ox, oy, u);
        storeChroma(J, 2, ox, oy, v);
    } else {
        const size_t o = (size_t)oy * J.W + ox;
        J.oU[o] = u;
        J.oV[o] = v;
    }
}

struct TapCtx {
    const float *lc;
    const double2 *uv;
    int cw, ch;
    float L0, nx, ny, scx, scy, rwF, rhF, invSigma2, guideFade, rescue, invG2, invG2Par;
};

struct Acc { double u, v, wsum, sumAbs; };

// One tap of pass 2 (recon.cpp:606-623). dxnx = dx*nx and dxny = (-dx)*ny
// are the per-column products of the reference's dp and dt, hoisted out of
// the row loop (same operands, same rounding). CHECKED = false when the
// caller has shown both denominators stay below 2^64 (see guidedPixel).
template <bool CHECKED>
__device__ __forceinline__ void tapCore(const TapCtx &c, float l, double2 p, float dxnx, float dxny,
                                        float dy_ny, float dy_nx, float wx, Acc &a) {
    const float dL = l - c.L0;
    const float dp = dxnx + dy_ny;
    const float dt = dxny + dy_nx;
    const float xs = 1.0f + dL * dL * c.invSigma2;
    const float simRaw = CHECKED ? rcpAtLeastOne(xs) : rcpInRange(xs);
    const float sim = 1.0f - c.guideFade * (1.0f - simRaw);
    const float xb = 1.0f + dp * dp * c.invG2 + dt * dt * c.invG2Par;
    const float bump = CHECKED ? rcpAtLeastOne(xb) : rcpInRange(xb);
    const float w = sim * (wx + c.rescue * bump);
    const double wd = (double)w;
    a.u = fma(wd, p.x, a.u);
    a.v = fma(wd, p.y, a.v);
    a.wsum += wd;
    a.sumAbs += fabs(wd);
}

__device__ __forceinline__ void tap(const TapCtx &c, size_t o, float dxf, float dy_ny, float dy_nx,
                                    float wx, Acc &a) {
    const float dx = dxf * c.rwF;
    tapCore<true>(c, ldf(c.lc + o), __ldg(c.uv + o), dx * c.nx, -dx * c.ny, dy_ny, dy_nx, wx, a);
}

// rcpInRange on both lanes: hardware approximation per lane, then the same
// fused Newton-Raphson refinement e = 1 - x*y, y' = y + y*e on the pair.
__device__ __forceinline__ f32x2 rcp2(f32x2 x, f32x2 one) {
    float x0, x1, y0, y1;
    up2(x, x0, x1);
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y0) : "f"(x0));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y1) : "f"(x1));
    const f32x2 y = pk2(y0, y1);
    const f32x2 e = fma2(x ^ 0x8000000080000000ull, y, one);     // -x: sign bits flipped
    return fma2(y, e, y);
}

__device__ __forceinline__ void accumulate(Acc &a, float w, double2 p) {
    const double wd = (double)w;
    a.u = fma(wd, p.x, a.u);
    a.v = fma(wd, p.y, a.v);
    a.wsum += wd;
    a.sumAbs += fabs(wd);
}

// Any support, clamped taps; separable or radial base weights.
__device__ __forceinline__ void tapsGeneric(const FrameJob &J, const TapCtx &c, int ox, int oy,
                                            int tx0, int ty0, Acc &a) {
    const AxisView &ax = J.ax, &ay = J.ay;
    const float *wxp = ax.w + (size_t)ox * ax.sup;
    const uint8_t *amx = ax.am + (size_t)ox * ax.sup;
    const float *wyp = ay.w + (size_t)oy * ay.sup;
    const uint8_t *amy = ay.am + (size_t)oy * ay.sup;
    const float *base = J.radial ? radialWeightsAt(J.rad, ox, oy) : nullptr;
    for (int j = 0; j < ay.sup; ++j) {
        if (__ldg(amy + j) == 0)
            continue;
        const size_t rowOff = (size_t)iclamp(ty0 + j, 0, c.ch - 1) * c.cw;
        const float wy = __ldg(wyp + j);
        const float dyf = (float)(ty0 + j) - c.scy;
        const float dy = dyf * c.rhF;
        const float dyc = dyf * J.invWyC;
        const float dy_ny = dy * c.ny, dy_nx = dy * c.nx;
        for (int i = 0; i < ax.sup; ++i) {
            if (__ldg(amx + i) == 0)
                continue;
            const size_t o = rowOff + iclamp(tx0 + i, 0, c.cw - 1);
            const float dxf = (float)(tx0 + i) - c.scx;
            float wx;
            if (base) {
                wx = ldf(base + (size_t)j * ax.sup + i);
            } else if (J.radial) {
                const float dxc = dxf * J.invWxC;
                wx = lutLookupDev(J.lut, J.lutN, sqrtf(dxc * dxc + dyc * dyc) * J.lutScale);
            } else {
                wx = __ldg(wxp + i) * wy;
            }
            tap(c, o, dxf, dy_ny, dy_nx, wx, a);
        }
    }
}

struct Guided {
    double u, v;
    float L0, ssRamp, guideFade, nx, ny;
    bool hasDir;
    bool havePlain;                     // plainU/V hold the plain base
    float plainU, plainV;
};

// The algo 4 selector of one listed pixel (recon.cpp:762-811): blends the
// plain base, the guided value and the LGF value, or (float output) stores the
// routing weights for the blend stage.
template <bool RFUSE>
__device__ __forceinline__ void guidedSelect(const FrameJob &J, int ox, int oy, const Guided &g) {
    const float diag = g.hasDir ? smin(1.0f, 2.0f * fabsf(g.nx * g.ny)) : 0.0f;
    const float hedgy = (1.0f - g.ssRamp) * g.guideFade;
    const float sel = J.strength4;
    const float w2 = hedgy * (1.0f - diag) * sel;
    const float w3 = hedgy * diag * sel;
    const size_t o = (size_t)oy * J.W + ox;
    if (J.outKind != kF32) {
        // integer output: single-expression fused selector on the plain base
        float baseU, baseV;
        if (RFUSE && g.havePlain) {
            baseU = g.plainU;
            baseV = g.plainV;
        } else {
            plainPixel(J, ox, oy, baseU, baseV);
        }
        double valueU, valueV;
        if (w2 >= 1e-4f || w3 >= 1e-4f) {
            const int cx = __ldg(J.ax.cbI0 + ox), cy = __ldg(J.ay.cbI0 + oy);
            const float cxf = __ldg(J.ax.cbF + ox), cyf = __ldg(J.ay.cbF + oy);
            const LgfSample m = lgfAt(J, cx, cxf, cy, cyf);
            const float au = m.ab.x, bu = m.ab.y, av = m.ab.z, bv = m.ab.w, cu = m.conf.x, cv = m.conf.y;
            valueU = baseU + w2 * ((float)g.u - baseU) + w3 * cu * (au * g.L0 + bu - baseU);
            valueV = baseV + w2 * ((float)g.v - baseV) + w3 * cv * (av * g.L0 + bv - baseV);
        } else {
            valueU = baseU;
            valueV = baseV;
        }
        emit(J, ox, oy, (float)valueU, (float)valueV);
        return;
    }
    // float output: routing metadata; blended after the ROI-limited LGF
    float baseU, baseV;
    if (RFUSE && g.havePlain) {
        // the plain base of this listed pixel, for the blend stage too
        baseU = g.plainU;
        baseV = g.plainV;
        J.oU[o] = baseU;
        J.oV[o] = baseV;
    } else {
        baseU = J.oU[o];
        baseV = J.oV[o];
    }
    const bool compressed = J.sparse &&
        (unsigned long long)J.counters[kCntActiveOutput] * 2ull < (unsigned long long)J.W * J.H;
    if (compressed) {
        if (w2 < 1e-4f && w3 < 1e-4f) {
            J.gU[o] = 0.0f;
            J.gV[o] = 0.0f;
            J.selW3[o] = 0.0f;
        } else {
            J.gU[o] = hedgy * (1.0f - diag) * ((float)g.u - baseU);
            J.gV[o] = hedgy * (1.0f - diag) * ((float)g.v - baseV);
            J.selW3[o] = hedgy * diag;
        }
    } else {
        J.gU[o] = (float)g.u;
        J.gV[o] = (float)g.v;
        J.selW2[o] = hedgy * (1.0f - diag);
        J.selW3[o] = hedgy * diag;
    }
}

} // namespace lgcr_b200
