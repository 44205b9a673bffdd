// Host-side arrays of the divergence kernels (patches.cpp builds them, face.cu reads them).
#pragma once

#include <stdint.h>

#include <vector>

#include "fcw_internal.h"

namespace fcw {

// A patch: vertices [v0, v0 + nv) with their neighbours' rows and fan steps, as a CTA holds them in
// shared memory (three CTAs per SM).
constexpr int kPatchVerts = 64, kPatchRows = 108, kPatchSteps = 512;
struct Patch {
    int32_t v0, nv, row0, nrows, nsteps, pad;
};

// A step of a vertex's fan. The fan's first step names a neighbour and the faces that follow; each of
// those steps names the next neighbour and holds the coefficients gb_a . gb_b, times the squared
// area, of the face between it and the step before (a: that step's neighbour, b: this one), twice
// each, as packed operands.
struct FanStep {
    float c11[2], c12[2], c22[2];
    int32_t neighbour, faces;  // faces: of the fan, in its first step; negative in the others
};

struct PatchArrays {
    std::vector<Patch> patches;
    std::vector<int32_t> big;   // vertices with more neighbours than a patch holds
    std::vector<int32_t> rows;  // the vertices of a patch's rows, its own first
};

// fv: faces (elimination order), inc_*: each vertex's incident faces in ascending face order. walk: per
// step, its neighbour and the face it closes (-1 in a fan's first step). threads: 0 takes one per
// kFanRange vertices, at most 8 and at most the host's.
constexpr int64_t kFanRange = 4096;
void face_fans(const MeshPrep& m, const std::vector<int32_t>& fv, const std::vector<int32_t>& inc_ptr,
               const std::vector<int32_t>& inc_face, const std::vector<int8_t>& inc_corner,
               std::vector<int32_t>& ptr, std::vector<FanStep>& steps, std::vector<int32_t>& walk,
               int threads = 0);
// The vertices with a sharp corner (sine squared below kSharp): their fans with the neighbours as vertices,
// and for the sharp faces (faces = -2) other coefficients: gb_v . gb_v, -gb_v . gb_b, gb_b . gb_b times the
// squared area, gb_v the gradient of the vertex itself, for the differences along the step before's edge
// and from its neighbour to this one's.
constexpr double kSharp = 0.01;
struct SharpFans {
    std::vector<int32_t> vertices, ptr;  // ptr: their steps
    std::vector<FanStep> steps;
};
// walk, steps: of face_fans. Does not read the steps' neighbours, which face_patches rewrites.
void sharp_fans(const MeshPrep& m, const std::vector<int32_t>& fv, const std::vector<int32_t>& fan_ptr,
                const std::vector<FanStep>& steps, const std::vector<int32_t>& walk, SharpFans& sf);
// fv: faces (elimination order). Rewrites the steps' neighbours as patch rows (big vertices keep theirs).
void face_patches(const std::vector<int32_t>& fan_ptr, std::vector<FanStep>& steps, PatchArrays& pa);

}  // namespace fcw
