// Invariants of the solve plan (csrc/fronts.cpp) on meshes given as files: int64 n_vertices,
// n_faces, FP64 coordinates, int32 faces. Prints "ok <front count> <levels> <supernode levels>" per mesh.
#include <cstdio>
#include <cstdlib>
#include <string>
#include <vector>

#include "fronts.h"

using namespace fcw;

#define CHECK(c)                                                   \
    do {                                                           \
        if (!(c)) {                                                \
            std::printf("failed: %s (line %d)\n", #c, __LINE__);   \
            return 1;                                              \
        }                                                          \
    } while (0)

static int check(const char* path, int leaf, int width, int relax) {
    FILE* f = std::fopen(path, "rb");
    int64_t nv = 0, nf = 0;
    CHECK(f && std::fread(&nv, 8, 1, f) == 1 && std::fread(&nf, 8, 1, f) == 1);
    std::vector<double> V(3 * nv);
    std::vector<int32_t> F(3 * nf);
    CHECK((int64_t)std::fread(V.data(), 8, 3 * nv, f) == 3 * nv && (int64_t)std::fread(F.data(), 4, 3 * nf, f) == 3 * nf);
    std::fclose(f);
    MeshPrep m;
    Symbolic S;
    Fronts t;
    std::string err;
    CHECK(prepare_mesh(V.data(), nv, F.data(), nf, m, err) == 0);
    CHECK(build_symbolic(m, leaf, width, relax, S, err) == 0);
    CHECK(build_fronts(S, t, err) == 0);
    std::vector<int> level(t.nf);
    for (int l = 0; l < t.nlevels; ++l)
        for (int q = t.level_ptr[l]; q < t.level_ptr[l + 1]; ++q) level[t.level_nodes[q]] = l;
    // fronts: columns partitioned, structure among the ancestors, narrow below first_wide
    CHECK(t.c0[0] == 0 && t.c0[t.nf] == S.n);
    for (int i = 0; i < t.nf; ++i) {
        const int ns = t.c0[i + 1] - t.c0[i];
        CHECK(ns > 0 && t.m[i] >= ns && ns <= kWidestFront);
        if (level[i] < t.first_wide) CHECK(ns <= 64);
        if (t.parent[i] >= 0) CHECK(level[t.parent[i]] > level[i]);
        for (int64_t q = t.row0[i]; q < t.row0[i + 1]; ++q) {
            CHECK(t.rows[q] >= 0 && t.rows[q] < S.n);
            if (q > t.row0[i]) CHECK(t.rows[q] > t.rows[q - 1]);
            if (q - t.row0[i] >= ns) CHECK(level[t.col_front[t.rows[q]]] > level[i]);
        }
    }
    // every supernode's panel rows are rows of its front
    for (int s = 0; s < S.nsuper; ++s) {
        const int i = t.col_front[S.sn_c0[s]];
        for (int64_t q = S.sn_rowptr[s]; q < S.sn_rowptr[s + 1]; ++q)
            CHECK(t.pos[q] >= 0 && t.pos[q] < t.m[i] && t.rows[t.row0[i] + t.pos[q]] == S.rows[q]);
    }
    // every update row is gathered once, on the front row of its vertex
    std::vector<int> seen(t.n_urows, 0);
    auto entry = [&](size_t q, int u, int c) {
        if (u < 0 || u >= t.n_urows || c < 0 || c >= t.nf) return false;
        const int nsc = t.c0[c + 1] - t.c0[c];
        seen[u]++;
        return t.rows[t.row0[c] + nsc + (u - t.uoff[c])] == t.rows[q];
    };
    for (size_t q = 0; q < t.rec.size(); ++q) {
        for (int k = 0; k < 3; ++k) {
            CHECK((t.rec[q].src[k] >= 0) == (t.rec_child[3 * q + k] >= 0));
            if (t.rec[q].src[k] >= 0) CHECK(entry(q, t.rec[q].src[k], t.rec_child[3 * q + k]));
        }
        if (t.rec[q].more >= 0)
            for (int e = 0; e < t.more[t.rec[q].more]; ++e)
                CHECK(entry(q, t.more[t.rec[q].more + 1 + 2 * e], t.more[t.rec[q].more + 2 + 2 * e]));
    }
    for (int s : seen) CHECK(s == 1);
    // tasks: each column's forward and backward result and each update row written once; panels disjoint
    std::vector<char> y(S.n, 0), x(S.n, 0), u(t.n_urows, 0);
    int64_t o64 = 0, o32 = 0;
    for (int l = 0; l < t.nlevels; ++l)
        for (int k = t.fwd_ptr[l]; k < t.fwd_ptr[l + 1]; ++k) {
            const SweepTask& a = t.fwd[k];
            CHECK(level[a.front] == l && a.h > 0 && a.h <= t.fwd_rows[l] && a.r0 % 16 == 0);
            CHECK(a.off64 == o64 && a.off32 == o32 && o64 % 16 == 0 && o32 % 16 == 0);
            CHECK(a.depth > 0 && a.depth <= a.ns && (a.r0 + a.h <= a.ns || a.depth == a.ns));
            if (l < t.first_wide) CHECK(a.depth <= 64);
            else CHECK(a.wrow + a.ns <= t.n_wrows);
            for (int r = a.r0; r < a.r0 + a.h; ++r) {
                char& w = r < a.ns ? y[a.c0 + r] : u[a.urow + r - a.ns];
                CHECK(!w);
                w = 1;
            }
            o64 += padded_depth(a.depth) * panel_ld(a.h, true);
            o32 += padded_depth(a.depth) * panel_ld(a.h, false);
        }
    CHECK(o64 == t.fwd64 && o32 == t.fwd32);
    o64 = o32 = 0;
    for (const SweepTask& a : t.bwd) {
        CHECK(a.off64 == o64 && a.off32 == o32 && a.r0 % 16 == 0 && a.h <= 64 && a.depth == t.m[a.front] - a.r0);
        for (int c = 0; c < a.h; ++c) {
            CHECK(!x[a.c0 + a.r0 + c]);
            x[a.c0 + a.r0 + c] = 1;
        }
        o64 += padded_depth(a.depth) * panel_ld(a.h, true);
        o32 += padded_depth(a.depth) * panel_ld(a.h, false);
    }
    CHECK(o64 == t.bwd64 && o32 == t.bwd32);
    for (int i = 0; i < S.n; ++i) CHECK(y[i] && x[i]);
    for (char c : u) CHECK(c);
    for (int l = t.first_wide; l < t.nlevels; ++l)
        for (int i = t.asm_ptr[l]; i < t.asm_ptr[l + 1]; ++i) {
            CHECK(t.rows[t.asm_rows[4 * i]] == t.asm_rows[4 * i + 1]);
            CHECK(level[t.asm_rows[4 * i + 2]] == l && t.col_front[t.asm_rows[4 * i + 1]] == t.asm_rows[4 * i + 2]);
        }
    std::printf("ok %d %d %d\n", t.nf, t.nlevels, S.nlevels);
    return 0;
}

int main(int argc, char** argv) {
    for (int i = 4; i < argc; ++i)
        if (check(argv[i], std::atoi(argv[1]), std::atoi(argv[2]), std::atoi(argv[3]))) return 1;
    return 0;
}
