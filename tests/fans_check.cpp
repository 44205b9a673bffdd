// The fans (csrc/patches.cpp) formed in one range of vertices and in several, for the mesh file of
// patches_check.cpp: prints "ok <fan steps>" when the arrays are the same.
#include <cstdio>
#include <cstring>

#include "patches.h"

using namespace fcw;

int main(int, char** argv) {
    FILE* f = std::fopen(argv[1], "rb");
    int64_t nv = 0, nf = 0;
    if (!f || std::fread(&nv, 8, 1, f) != 1 || std::fread(&nf, 8, 1, f) != 1) return 1;
    std::vector<double> V(3 * nv);
    std::vector<int32_t> F(3 * nf);
    if ((int64_t)std::fread(V.data(), 8, 3 * nv, f) != 3 * nv || (int64_t)std::fread(F.data(), 4, 3 * nf, f) != 3 * nf)
        return 1;
    MeshPrep m;
    std::string err;
    if (prepare_mesh(V.data(), nv, F.data(), nf, m, err)) return 1;
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
    std::vector<int32_t> p1, p2, w1, w2;
    std::vector<FanStep> s1, s2;
    face_fans(m, F, ptr, face, corner, p1, s1, w1, 1);
    for (int threads : {0, 2, 3, 8, 64}) {
        face_fans(m, F, ptr, face, corner, p2, s2, w2, threads);
        if (p1 != p2 || w1 != w2 || s1.size() != s2.size() || std::memcmp(s1.data(), s2.data(), s1.size() * sizeof(FanStep)))
            return 1;
    }
    std::printf("ok %zu\n", s1.size());
    return 0;
}
