// The fans (csrc/patches.cpp) formed in one range of vertices and in several, for the mesh file of
// patches_check.cpp: prints "ok <fan steps> <vertices with sharp corners>" when the arrays are the same and
// the sharp corners' fans are those vertices' own.
#include <cmath>
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
    SharpFans sf;
    sharp_fans(m, F, p1, s1, w1, sf);
    if (sf.ptr.size() != sf.vertices.size() + 1) return 1;
    for (size_t i = 0; i < sf.vertices.size(); ++i) {
        const int32_t v = sf.vertices[i], e0 = p1[v], ne = p1[v + 1] - e0;
        int sharp = 0;
        if (sf.ptr[i + 1] - sf.ptr[i] != ne) return 1;
        for (int k = 0; k < ne; ++k) {
            const FanStep &a = s1[e0 + k], &b = sf.steps[sf.ptr[i] + k];
            if (a.neighbour != b.neighbour || b.c22[0] != a.c22[0]) return 1;
            if (b.faces != -2) {
                if (std::memcmp(&a, &b, sizeof a)) return 1;
                continue;
            }
            ++sharp;  // the squared area times |gradient at v|^2 is a quarter of the opposite edge's square
            double e2 = 0.0;
            for (int c = 0; c < 3; ++c) {
                const double d = V[3 * (size_t)b.neighbour + c] - V[3 * (size_t)s1[e0 + k - 1].neighbour + c];
                e2 += d * d;
            }
            if (std::fabs(b.c11[0] - 0.25 * e2) > 1e-6 * e2 || b.c11[0] != b.c11[1] || b.c12[0] != b.c12[1]) return 1;
            // and c_vb + (c_ab + c_bb) = 0, to the rounding of the long edges' products
            if (std::fabs((double)b.c12[0] - ((double)a.c12[0] + a.c22[0])) > 1e-6 * a.c22[0]) return 1;
        }
        if (sharp == 0) return 1;
    }
    std::printf("ok %zu %zu\n", s1.size(), sf.vertices.size());
    return 0;
}
