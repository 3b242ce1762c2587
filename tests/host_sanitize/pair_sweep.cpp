// Column-pair tables of the guided pass against the axes they are made from:
// every active tap of every column appears once at its place with its weight
// and distance, windows stay inside the plane, inactive entries are zero, and
// the jinc rows hold the phase table's weights. Exits non-zero on a difference.
#include "geometry.h"

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>

using namespace lgcr_b200;

static int bad = 0, tables = 0;
#define CHECK(c) do { if (!(c)) { if (bad++ < 10) std::printf("line %d: %s\n", __LINE__, #c); } } while (0)

static void sweep(const KernelSpec &k, int lumaW, int chromaW, int outW, double shift) {
    const double r = double(lumaW) / chromaW;
    const ChromaAxis a = buildChromaAxis(lumaW, outW, r, shift, k);
    const PairAxis p = buildPairAxis(a, chromaW, float(r));
    if (p.sup == 0)
        return;
    ++tables;
    CHECK(p.n == (outW + 1) / 2 && p.sup >= kPairMinSup && p.sup <= kPairMaxSup && p.sup <= chromaW);
    for (int i = 0; i < p.n; ++i) {
        CHECK(p.start[i] >= 0 && p.start[i] + p.sup <= chromaW);
        CHECK(p.kind[i] >= 0 && size_t(p.kind[i] + 1) * p.sup * 4 <= p.tab.size());
        const float *tab = &p.tab[size_t(p.kind[i]) * p.sup * 4];
        for (int q = 0; q < 2; ++q) {
            const int x = 2 * i + q;
            unsigned bits = 0;
            for (int j = 0; x < outW && j < a.sup; ++j)
                if (a.am[size_t(x) * a.sup + j]) {
                    const int c = a.start[x] + j - p.start[i];
                    CHECK(c >= 0 && c < p.sup);
                    if (c < 0 || c >= p.sup)
                        continue;
                    bits |= 1u << c;
                    CHECK(tab[c * 4 + q] == a.w[size_t(x) * a.sup + j]);
                }
            CHECK(((p.bits[i] >> (16 * q)) & 0xffffu) == bits);
            for (int c = 0; c < p.sup; ++c) {
                if (!((bits >> c) & 1u))
                    CHECK(tab[c * 4 + q] == 0.0f);
                if (x < outW)
                    CHECK(tab[c * 4 + 2 + q] == (float(p.start[i] + c) - a.pos[x]) * float(r));
            }
        }
    }
    std::vector<float> gate;
    std::vector<int> nearest;
    phaseTables(a, chromaW, gate, nearest);
    for (int x = 0; x < outW; ++x) {
        const float f = a.pos[x] - std::floor(a.pos[x]);
        CHECK(gate[x] == 1.0f - 2.0f * std::min(f, 1.0f - f));
        CHECK(nearest[x] >= 0 && nearest[x] < chromaW);
    }
    if (!k.radial)
        return;
    const RadialTable t = buildRadialTable(k, a, a, chromaW, chromaW);
    const PairRadial pr = buildPairRadial(t, p, outW);
    if (!pr.valid)
        return;
    for (int y = 0; y < t.phaseCountY; ++y)
        for (int i = 0; i < p.n; ++i)
            for (int q = 0; q < 2 && 2 * i + q < outW; ++q) {
                const int x = 2 * i + q;
                const float *w = &t.weights[(size_t(y) * t.phaseCountX + t.xPhase[x]) * t.supportX * t.supportY];
                const float *g = &pr.w[(size_t(y) * pr.phasePairs + pr.phase[i]) * t.supportY * p.sup * 2];
                for (int j = 0; j < t.supportY; ++j)
                    for (int c = 0; c < p.sup; ++c) {
                        const int tap = p.start[i] + c - a.start[x];
                        const bool on = tap >= 0 && tap < a.sup && a.am[size_t(x) * a.sup + tap];
                        CHECK(g[(size_t(j) * p.sup + c) * 2 + q] == (on ? w[size_t(j) * t.supportX + tap] : 0.0f));
                    }
            }
}

int main() {
    for (int kind = 0; kind < 6; ++kind) {
        for (int taps = 1; taps <= 5; ++taps) {
            KernelSpec k;
            k.kernel = Kernel(kind);
            k.support = kind == 0 ? 1.0 : kind == 1 || kind == 3 ? 2.0 : kind == 4 ? 3.0 : double(taps);
            k.kp1 = kind == 1 ? 0.0 : double(taps);
            k.kp2 = 0.6;
            if (kind == 5) {
                k.radial = true;
                k.kp1 = k.support = double(taps);
                k.lut.resize(taps * 1024 + 2);
                for (size_t i = 0; i < k.lut.size(); ++i)
                    k.lut[i] = float(jincWindowed(double(i) / 1024.0, k.support));
                k.lutScale = 1024.0f;
            } else if (kind != 2 && taps > 1) {
                continue;
            }
            for (int c : {1, 3, 4, 5, 8, 9, 17, 48, 101, 960})
                for (int ratio : {1, 2})
                    for (double scale : {0.5, 0.8, 1.0, 4.0 / 3.0, 1.5, 2.0, 2.1, 4.0})
                        for (double shift : {-0.5, 0.0, 0.5}) {
                            const int luma = c * ratio, out = std::max(1, int(luma * scale));
                            sweep(k, luma, c, out, ratio == 1 ? 0.0 : shift);
                            if (ratio == 2 && luma > 1)
                                sweep(k, luma - 1, c, out, shift);   // odd luma width
                        }
        }
    }
    std::printf("%d tables, %d differences\n", tables, bad);
    return bad || tables < 300 ? 1 : 0;
}
