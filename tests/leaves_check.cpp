// Which leaf sweeps of a block of K columns keep their panels resident (csrc/fronts.h), for the mesh file
// of fronts_check.cpp. Prints the leaf tasks, those of more than 32 columns, and 0 or 1 for: FP64
// forward, FP64 backward, FP64 backward with reach flags, FP32 backward.
#include <algorithm>
#include <cstdio>
#include <cstdlib>

#include "fronts.h"

using namespace fcw;

int main(int, char** argv) {
    FILE* f = std::fopen(argv[1], "rb");
    const int K = std::atoi(argv[2]);
    int64_t nv = 0, nf = 0;
    if (!f || std::fread(&nv, 8, 1, f) != 1 || std::fread(&nf, 8, 1, f) != 1) return 1;
    std::vector<double> V(3 * nv);
    std::vector<int32_t> F(3 * nf);
    if ((int64_t)std::fread(V.data(), 8, 3 * nv, f) != 3 * nv || (int64_t)std::fread(F.data(), 4, 3 * nf, f) != 3 * nf)
        return 1;
    MeshPrep m;
    Symbolic S;
    Fronts t;
    std::string err;
    if (prepare_mesh(V.data(), nv, F.data(), nf, m, err) ||
        build_symbolic(m, std::atoi(argv[3]), std::atoi(argv[4]), std::atoi(argv[5]), S, err) || build_fronts(S, t, err))
        return 1;
    int wide = 0, depth = 0;
    for (int k = 0; k < t.bwd_ptr[1]; ++k) {
        wide += t.bwd[k].h > 32;
        depth = std::max(depth, t.bwd[k].depth);
    }
    auto taken = [&](bool fp64, bool back, bool reach) {
        const int64_t panel = fp64 ? (back ? t.leaf_bwd64 : t.leaf_fwd64) : t.leaf_bwd32;
        const int cw = leaf_columns(fp64, back);
        const size_t smem = leaf_smem(panel, cw, fp64 ? 8 : 4, back ? depth : 0);
        return (int)(t.first_wide > 0 &&
                     leaves_resident(back ? t.bwd_ptr[1] : t.fwd_ptr[1], K / cw / kLeafWarps, smem, reach));
    };
    std::printf("%d %d %d %d %d %d\n", t.bwd_ptr[1], wide, taken(true, false, false), taken(true, true, false),
                taken(true, true, true), taken(false, true, false));
    return 0;
}
