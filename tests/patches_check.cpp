// Invariants of the divergence's fans and patches (csrc/patches.cpp) on meshes given as files: int64
// n_vertices, n_faces, FP64 coordinates, int32 faces. Prints "ok <patches> <big vertices>" per mesh.
#include <cmath>
#include <cstdio>
#include <set>
#include <string>
#include <vector>

#include "patches.h"

using namespace fcw;

#define CHECK(c)                                                   \
    do {                                                           \
        if (!(c)) {                                                \
            std::printf("failed: %s (line %d)\n", #c, __LINE__);   \
            return 1;                                              \
        }                                                          \
    } while (0)

static int check(const char* path) {
    FILE* f = std::fopen(path, "rb");
    int64_t nv = 0, nf = 0;
    CHECK(f && std::fread(&nv, 8, 1, f) == 1 && std::fread(&nf, 8, 1, f) == 1);
    std::vector<double> V(3 * nv);
    std::vector<int32_t> F(3 * nf);
    CHECK((int64_t)std::fread(V.data(), 8, 3 * nv, f) == 3 * nv && (int64_t)std::fread(F.data(), 4, 3 * nf, f) == 3 * nf);
    std::fclose(f);
    MeshPrep m;
    std::string err;
    CHECK(prepare_mesh(V.data(), nv, F.data(), nf, m, err) == 0);
    std::vector<int32_t> ptr(nv + 1, 0), face(3 * nf);
    std::vector<int8_t> corner(3 * nf);
    for (int32_t v : F) ptr[v + 1]++;
    for (int64_t v = 0; v < nv; ++v) ptr[v + 1] += ptr[v];
    std::vector<int32_t> fill(ptr.begin(), ptr.end() - 1);
    for (int64_t t = 0; t < nf; ++t)
        for (int c = 0; c < 3; ++c) {
            face[fill[F[3 * t + c]]] = (int32_t)t;
            corner[fill[F[3 * t + c]]++] = (int8_t)c;
        }
    std::vector<int32_t> fan_ptr;
    std::vector<FanStep> steps;
    std::vector<int32_t> walk;
    face_fans(m, F, ptr, face, corner, fan_ptr, steps, walk);
    CHECK(walk.size() == 2 * steps.size());
    // each face once per corner, as the pair of neighbours of two consecutive steps
    for (int64_t v = 0; v < nv; ++v) {
        std::multiset<std::pair<int, int>> want, got;
        for (int q = ptr[v]; q < ptr[v + 1]; ++q) {
            const int a = F[3 * face[q] + (corner[q] + 1) % 3], b = F[3 * face[q] + (corner[q] + 2) % 3];
            want.insert({std::min(a, b), std::max(a, b)});
        }
        int left = 0;
        for (int e = fan_ptr[v]; e < fan_ptr[v + 1]; ++e) {
            if (left == 0) {  // a fan's first step
                left = steps[e].faces;
                CHECK(walk[2 * e] == steps[e].neighbour && walk[2 * e + 1] == -1);
                CHECK(left > 0);
                continue;
            }
            --left;
            CHECK(steps[e].faces == -1 && walk[2 * e] == steps[e].neighbour);
            const int32_t* w = &F[3 * (size_t)walk[2 * e + 1]];
            CHECK(std::set<int>({w[0], w[1], w[2]}) == std::set<int>({(int)v, steps[e - 1].neighbour, steps[e].neighbour}));
            const int p = steps[e - 1].neighbour;
            got.insert({std::min(p, steps[e].neighbour), std::max(p, steps[e].neighbour)});
            // the coefficients are the two neighbours' hat gradients' products times the squared area
            const double *x = &V[3 * v], *y = &V[3 * p], *z = &V[3 * steps[e].neighbour];
            double e1[3], e2[3], g11 = 0, g12 = 0, g22 = 0;
            for (int k = 0; k < 3; ++k) { e1[k] = y[k] - x[k]; e2[k] = z[k] - x[k]; }
            for (int k = 0; k < 3; ++k) { g11 += e1[k] * e1[k]; g12 += e1[k] * e2[k]; g22 += e2[k] * e2[k]; }
            // gradients' Gram matrix = inverse of the edges'; det = 4 area^2
            const double tol = 1e-5 * (g11 + g22);
            CHECK(std::fabs(steps[e].c11[0] - 0.25 * g22) < tol && std::fabs(steps[e].c22[0] - 0.25 * g11) < tol);
            CHECK(std::fabs(steps[e].c12[0] + 0.25 * g12) < tol);
            CHECK(steps[e].c11[0] == steps[e].c11[1] && steps[e].c12[0] == steps[e].c12[1] && steps[e].c22[0] == steps[e].c22[1]);
        }
        CHECK(left == 0 && want == got);
    }
    const std::vector<FanStep> global = steps;
    PatchArrays pa;
    face_patches(fan_ptr, steps, pa);
    std::vector<int> seen(nv, 0);
    for (int32_t v : pa.big) {
        seen[v]++;
        for (int e = fan_ptr[v]; e < fan_ptr[v + 1]; ++e) CHECK(steps[e].neighbour == global[e].neighbour);
    }
    for (const Patch& p : pa.patches) {
        CHECK(p.nv > 0 && p.nv <= kPatchVerts && p.nrows <= kPatchRows && p.row0 + p.nrows <= (int)pa.rows.size());
        CHECK(p.nsteps <= kPatchSteps && p.nsteps == fan_ptr[p.v0 + p.nv] - fan_ptr[p.v0]);
        const int32_t* rows = &pa.rows[p.row0];
        std::set<int32_t> distinct(rows, rows + p.nrows);
        CHECK((int)distinct.size() == p.nrows);
        for (int i = 0; i < p.nv; ++i) {
            seen[p.v0 + i]++;
            CHECK(rows[i] == p.v0 + i);
            for (int e = fan_ptr[p.v0 + i]; e < fan_ptr[p.v0 + i + 1]; ++e)
                CHECK(steps[e].neighbour >= 0 && steps[e].neighbour < p.nrows &&
                      rows[steps[e].neighbour] == global[e].neighbour);
        }
    }
    for (int s : seen) CHECK(s == 1);
    std::printf("ok %zu %zu\n", pa.patches.size(), pa.big.size());
    return 0;
}

int main(int argc, char** argv) {
    for (int i = 1; i < argc; ++i)
        if (check(argv[i])) return 1;
    return 0;
}
