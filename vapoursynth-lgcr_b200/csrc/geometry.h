// Host-side geometry of the Recon path: kernel profiles, polyphase tables,
// chroma sampling axes and radial (jinc) phase tables. Built once per
// filter/geometry in double precision on the host and uploaded resident.
//
// Each builder follows the reference's arithmetic step for step because the
// device kernels index these tables and must see identical float values:
//   kernelEval/sinc/jincWindowed/kernelSupport   src/lgcr.h:53-117
//   buildWeights                                 src/kernels.cpp:135-167
//   buildChromaAxisUncached                      src/kernels.cpp:337-404
//   buildBilinAxis (index/fraction part)         src/maps.cpp:190-208
//   collectPhases / buildRadialWeights           src/kernels.cpp:449-526
//   lutLookup                                    src/lgcr.h:636-641
//   buildLcMap footprint extents                 src/maps.cpp:429-447
#pragma once

#include <cstdint>
#include <string>
#include <vector>

namespace lgcr_b200 {

enum class Kernel : int { Bilinear = 0, Bicubic = 1, Lanczos = 2, Spline16 = 3, Spline36 = 4, Jinc = 5 };

double sincd(double x);
double kernelEval(Kernel k, double x, double p1, double p2);
double jincWindowed(double x, double taps);
float lutLookup(const float *lut, int n, float idx);

struct KernelSpec {
    Kernel kernel = Kernel::Lanczos;
    double kp1 = 3.0, kp2 = 0.6;
    double support = 3.0;
    bool radial = false;
    std::vector<float> lut;     // jinc profile, 1024 entries per unit
    float lutScale = 0.0f;
};

struct WeightTable {
    int n = 0, sup = 0;
    std::vector<int> start;
    std::vector<float> w;       // n * sup
};

WeightTable buildWeights(int srcN, int dstN, const KernelSpec &k, double shift);

struct BilinAxis {
    std::vector<int> i0;
    std::vector<float> f;
};

BilinAxis buildBilinAxis(const std::vector<float> &pos, int srcN);

struct ChromaAxis {
    int n = 0, sup = 0;
    std::vector<int> start;
    std::vector<float> w;        // n * sup (normalized; zero for radial)
    std::vector<uint8_t> am;     // n * sup activity (0/1)
    std::vector<float> weightSum, absoluteWeightSum;
    std::vector<float> pos, lpos;
    BilinAxis chromaBilin, lumaBilin;
};

ChromaAxis buildChromaAxis(int srcLumaN, int dstLumaN, double r, double sitShift,
                           const KernelSpec &k);

struct RadialTable {
    bool valid = false;          // false: evaluate the LUT per tap
    int supportX = 0, supportY = 0, phaseCountX = 0, phaseCountY = 0;
    std::vector<uint16_t> xPhase, yPhase;
    std::vector<float> weights;
    std::vector<double> weightSum, absoluteWeightSum;
    // per phase pair: the guided rescue's kappa (max |w|)^2 / (sum w^2 + 1e-12)
    // over the active taps, in float and in tap order (rows, then columns)
    std::vector<float> kappa;
};

RadialTable buildRadialTable(const KernelSpec &k, const ChromaAxis &ax, const ChromaAxis &ay,
                             int sourceWidth, int sourceHeight);

// Per index of a separable chroma axis: the largest |weight| and the sum of
// squared weights over the active taps (the guided rescue term's kappa
// factors), in float and in tap order as the guided pass evaluates them.
void rescueFactors(const ChromaAxis &a, std::vector<float> &mx, std::vector<float> &ss);

// Pairs of output columns (2p, 2p + 1) of a chroma axis on one common window
// of `sup` samples: the guided pass evaluates both pixels of a pair from the
// same loaded samples. Empty (sup 0) when some pair's active taps span more
// than kPairMaxSup samples or the plane is narrower than the window.
constexpr int kPairMinSup = 4, kPairMaxSup = 9;
struct PairAxis {
    int n = 0, sup = 0;
    std::vector<int> start;      // first sample of the common window
    // per pair the row of `tab`, the distinct pairs' taps: [kind][sup][4] with
    // both columns' weights (zero at inactive taps) and then both columns' tap
    // distances (tap - position) * r in float. Away from the frame's sides a
    // same-size frame has one kind.
    std::vector<int> kind;
    std::vector<float> tab;
    std::vector<uint32_t> bits;  // active taps: low half column 2p, high half column 2p + 1
    std::vector<int> first;      // n * 2: tap of the common window that is tap 0 of the column
};
PairAxis buildPairAxis(const ChromaAxis &a, int chromaN, float r);

// Jinc weights of both columns of a pair on the common window, per (row
// phase, phase pair): phase pairs are the distinct (column phases, tap
// offsets) of the pairs. Not valid when the radial table is not, or with more
// than 1024 (row phase, phase pair) combinations.
struct PairRadial {
    bool valid = false;
    int phasePairs = 0;
    std::vector<uint16_t> phase;     // per pair
    std::vector<float> w;            // [row phase][phase pair][row][column of the window][2]
};
PairRadial buildPairRadial(const RadialTable &t, const PairAxis &p, int outN);

// Per index: the phase gate factor 1 - 2 * min(f, 1 - f) of the position's
// fraction f, and the nearest sample (round half away from zero, clamped).
void phaseTables(const ChromaAxis &a, int chromaN, std::vector<float> &gate,
                 std::vector<int> &nearest);

// Footprint extents of each chroma sample on the luma grid.
void lcExtents(int lumaN, int chromaN, double r, double shift,
               std::vector<int> &begin, std::vector<int> &end);

} // namespace lgcr_b200
