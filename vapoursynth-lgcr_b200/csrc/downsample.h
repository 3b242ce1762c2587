// Downsample filter (the reference's standalone 4:4:4 -> 4:2:0 guided
// downsampler, src/downsample.cpp): device descriptor and launch.
#pragma once

#include <cuda_runtime.h>

#include "recon.cuh"

namespace lgcr_b200 {

// Candidate planes of quality 2 (generateCandidateRow,
// src/downsample.cpp:524-569), each cw x ch floats.
enum DsCandidatePlane : int {
    kDsBaseU = 0, kDsBaseV = 1, kDsGate = 2, kDsCandU = 3, kDsCandV = 7, kDsPlanes = 11
};

// Spatial weights of the guided windows (spatialWeight,
// src/downsample.cpp:393-402). The window of an output sample lies at the
// same offsets from its centre everywhere (centre 2x + 0.5 + shift, exact in
// float), so a weight depends on the tap and on the envelope's direction
// only: [tap of the window, rows then columns][kDsSlots], slots 0-7 the
// directions and 8 the isotropic envelope of the smaller radius, 9-16 and 17
// those of quality 2's larger one.
constexpr int kDsSlots = 18;
constexpr int kDsMaxTaps = 81;

struct DownsampleJob {
    int W, H;                           // source (4:4:4) size, both even
    int cw, ch;                         // output chroma size W / 2, H / 2
    int kind;                           // kU8 / kU16 / kF32 (input and output)
    float inScale, chromaOffset;        // SourcePlane scale, chroma offset
    float outScale, outOffset;          // OutputPlane scale and offset
    int maxCode;
    const void *in[3];
    long long inPitch[3];
    void *out[2];                       // output U, V (cw x ch)
    long long outPitch[2];
    int hSup, vSup;                     // polyphase tables of the base
    const int *hStart, *vStart;
    const float *hW, *vW;
    float2 *rows;                       // H x cw horizontal pass (U, V)
    float *cand;                        // kDsPlanes x cw x ch (quality 2)
    int quality;
    float strength, shiftX, shiftY;
    const float *spatial;               // winW * winH * kDsSlots
    int winX0, winY0, winW, winH;       // window of output (x, y): first sample 2x + winX0, 2y + winY0
};

cudaError_t launchDownsample(const DownsampleJob &J, cudaStream_t s);

} // namespace lgcr_b200
