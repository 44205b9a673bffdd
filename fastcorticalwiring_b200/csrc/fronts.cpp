// Fronts of the multi-right-hand-side sweeps (solve.cu), from the factorisation's supernodes.
//
// The factorisation works on supernodes of at most 64 columns, so a separator of several hundred
// vertices is a chain of supernodes, and near the root most levels of the tree are such chains: 20
// of the 32 levels of a 147k-vertex mesh hold one to four supernodes. A sweep pays every level's
// latency, so the solve merges a chain back into one front: [inv(L_ss); Q_s] over all of the
// chain's columns (fronts.cu forms it from the supernodes' blocks). A link s -> s + 1 is taken
// when it is exact (s's structure is s + 1's rows) or when the merged front's explicit zeros stay
// under 5%: 32 to 12 levels at 147k vertices, 19 to 10 at 37k, 11 to 8 at 9k, with 0.1% more
// stored entries. Fronts wider than 64 columns are made only from 192 rows up: the many small
// fronts near the leaves keep to one 64-column right-hand-side tile.
#include "fronts.h"

#include <algorithm>

namespace fcw {

namespace {

constexpr double kMaxZeros = 0.05;
constexpr int kNarrow = 64;        // widest front whose right-hand side one task gathers by itself
constexpr int kWideFrom = 192;     // rows of the smallest front that may be wider
// Rows of a leaf's forward tasks: one task holds an average leaf's 88 rows, so its right-hand side is
// read once. Fronts with children gather theirs through registers, which three smaller CTAs per SM
// hide better than two: 147k vertices, 1024 columns, Poisson forward 1.46 against 1.54 ms (FP64 2.27
// against 2.40).
constexpr int kLeafRows = 128;
constexpr int kTileColumns = 128;  // right-hand sides per CTA (FP32), for the estimate below
constexpr int kFullBlock = 1024;
constexpr int kEnoughCtas = 296;   // two per SM

// Rows per task of a level whose fronts have the given total rows: the tallest tile that still
// gives two CTAs per SM for a full block, so the levels near the root spread over the chip.
int level_rows(const std::vector<int64_t>& tasks_by_height, const int* heights, int n) {
    for (int i = 0; i < n; ++i)
        if (tasks_by_height[i] * (kFullBlock / kTileColumns) >= kEnoughCtas) return heights[i];
    return heights[n - 1];
}

// Rows of each task when `rows` are split into the fewest tasks of at most `most`: equal shares,
// in whole 16-row groups.
int32_t even_rows(int32_t rows, int32_t most) {
    const int32_t n = (rows + most - 1) / most;
    return ((rows + n - 1) / n + 15) / 16 * 16;
}

}  // namespace

int build_fronts(const Symbolic& S, Fronts& f, std::string& err) {
    const int32_t NS = S.nsuper;
    auto width = [&](int32_t s) { return S.sn_c0[s + 1] - S.sn_c0[s]; };
    f = Fronts();
    // 1. runs of supernodes
    f.sn0.clear();
    {
        double stored_true = 0.0;
        int64_t w = 0;
        bool leaf_run = false;
        for (int32_t s = 0; s < NS; ++s) {
            const int64_t ns = width(s), m = S.sn_m[s], nr = m - ns;
            const double mine = ns * (ns + 1) / 2.0 + (double)ns * nr;
            bool join = false;
            if (s > 0 && S.sn_parent[s - 1] == s && !leaf_run) {
                const int64_t nw = w + ns;
                const double stored = nw * (nw + 1) / 2.0 + (double)nw * nr;
                const bool exact = S.sn_m[s - 1] - width(s - 1) == m;
                join = (exact || 1.0 - (stored_true + mine) / stored < kMaxZeros) && nw <= kWidestFront &&
                       (nw <= kNarrow || nw + nr >= kWideFrom);
            }
            if (join) {
                w += ns;
                stored_true += mine;
            } else {
                f.sn0.push_back(s);
                w = ns;
                stored_true = mine;
                leaf_run = S.child_ptr[s + 1] == S.child_ptr[s] && m < kWideFrom;
            }
        }
    }
    f.nf = (int32_t)f.sn0.size();
    f.sn0.push_back(NS);
    const int32_t NF = f.nf;
    f.c0.resize(NF + 1);
    f.m.resize(NF);
    f.parent.assign(NF, -1);
    f.col_front.assign(S.n, -1);
    f.row0.assign(NF + 1, 0);
    f.uoff.assign(NF + 1, 0);
    for (int32_t t = 0; t < NF; ++t) {
        const int32_t last = f.sn0[t + 1] - 1;
        f.c0[t] = S.sn_c0[f.sn0[t]];
        const int32_t end = S.sn_c0[last + 1], nr = S.sn_m[last] - width(last);
        f.m[t] = end - f.c0[t] + nr;
        f.row0[t + 1] = f.row0[t] + f.m[t];
        f.uoff[t + 1] = f.uoff[t] + nr;
        for (int32_t j = f.c0[t]; j < end; ++j) f.col_front[j] = t;
    }
    f.c0[NF] = (int32_t)S.n;
    f.n_urows = f.uoff[NF];
    if (f.n_urows > INT32_MAX || f.row0[NF] > INT32_MAX) {
        err = "mesh too large for 32-bit update indices";
        return 1;
    }
    f.rows.resize(f.row0[NF]);
    f.pos.resize(S.rows.size());
    std::vector<int32_t> where(S.n, -1);  // row -> position in the current front
    for (int32_t t = 0; t < NF; ++t) {
        const int32_t last = f.sn0[t + 1] - 1;
        if (S.sn_parent[last] >= 0) f.parent[t] = f.col_front[S.sn_c0[S.sn_parent[last]]];
        int64_t o = f.row0[t];
        for (int32_t j = f.c0[t]; j < f.c0[t + 1]; ++j) f.rows[o++] = j;
        for (int64_t q = S.sn_rowptr[last] + width(last); q < S.sn_rowptr[last + 1]; ++q) f.rows[o++] = S.rows[q];
        for (int64_t q = f.row0[t]; q < f.row0[t + 1]; ++q) where[f.rows[q]] = (int32_t)(q - f.row0[t]);
        for (int32_t s = f.sn0[t]; s <= last; ++s)
            for (int64_t q = S.sn_rowptr[s]; q < S.sn_rowptr[s + 1]; ++q) {
                f.pos[q] = where[S.rows[q]];
                if (f.pos[q] < 0 || f.pos[q] >= f.m[t] || f.rows[f.row0[t] + f.pos[q]] != S.rows[q]) {
                    err = "solve plan: a supernode's rows are not its front's";
                    return 1;
                }
            }
    }
    // 2. levels (height in the tree of fronts)
    std::vector<int32_t> level(NF, 0);
    for (int32_t t = 0; t < NF; ++t)
        if (f.parent[t] >= 0) level[f.parent[t]] = std::max(level[f.parent[t]], level[t] + 1);
    for (int32_t t = 0; t < NF; ++t) f.nlevels = std::max(f.nlevels, level[t] + 1);
    f.level_ptr.assign(f.nlevels + 1, 0);
    for (int32_t t = 0; t < NF; ++t) f.level_ptr[level[t] + 1]++;
    for (int32_t l = 0; l < f.nlevels; ++l) f.level_ptr[l + 1] += f.level_ptr[l];
    f.level_nodes.resize(NF);
    {
        std::vector<int32_t> fill(f.level_ptr.begin(), f.level_ptr.end() - 1);
        for (int32_t t = 0; t < NF; ++t) f.level_nodes[fill[level[t]]++] = t;
    }
    // 3. where each child's update rows land, in ascending child order
    f.rec.assign(f.rows.size(), GatherRec{{-1, -1, -1}, -1});
    f.rec_child.assign(3 * f.rows.size(), -1);
    {
        std::vector<int32_t> count(f.rows.size(), 0);
        std::vector<int32_t> cptr(NF + 1, 0), clist(NF);
        for (int32_t t = 0; t < NF; ++t)
            if (f.parent[t] >= 0) cptr[f.parent[t] + 1]++;
        for (int32_t t = 0; t < NF; ++t) cptr[t + 1] += cptr[t];
        std::vector<int32_t> fill(cptr.begin(), cptr.end() - 1);
        for (int32_t t = 0; t < NF; ++t)
            if (f.parent[t] >= 0) clist[fill[f.parent[t]]++] = t;
        std::fill(where.begin(), where.end(), -1);
        std::vector<std::pair<int32_t, std::pair<int32_t, int32_t>>> extra;  // (front row, (update row, child))
        for (int32_t p = 0; p < NF; ++p) {
            for (int64_t q = f.row0[p]; q < f.row0[p + 1]; ++q) where[f.rows[q]] = (int32_t)q;
            extra.clear();
            for (int32_t i = cptr[p]; i < cptr[p + 1]; ++i) {
                const int32_t c = clist[i];
                const int64_t first = f.row0[c] + (f.c0[c + 1] - f.c0[c]);
                for (int64_t q = first; q < f.row0[c + 1]; ++q) {
                    const int32_t g = where[f.rows[q]];
                    if (g < f.row0[p] || g >= f.row0[p + 1]) {
                        err = "solve plan: a child's structure is not contained in its parent";
                        return 1;
                    }
                    const int32_t u = (int32_t)(f.uoff[c] + (q - first));
                    const int32_t k = count[g]++;
                    if (k < 3) {
                        f.rec[g].src[k] = u;
                        f.rec_child[3 * (int64_t)g + k] = c;
                    } else {
                        extra.push_back({g, {u, c}});
                    }
                }
            }
            std::stable_sort(extra.begin(), extra.end(), [](const auto& a, const auto& b) { return a.first < b.first; });
            for (size_t i = 0; i < extra.size();) {
                size_t j = i;
                while (j < extra.size() && extra[j].first == extra[i].first) ++j;
                f.rec[extra[i].first].more = (int32_t)f.more.size();
                f.more.push_back((int32_t)(j - i));
                for (; i < j; ++i) {
                    f.more.push_back(extra[i].second.first);
                    f.more.push_back(extra[i].second.second);
                }
            }
        }
    }
    // 4. task lists
    f.first_wide = f.nlevels;
    for (int32_t l = 0; l < f.nlevels; ++l)
        for (int32_t q = f.level_ptr[l]; q < f.level_ptr[l + 1]; ++q) {
            const int32_t t = f.level_nodes[q];
            if (f.c0[t + 1] - f.c0[t] > kNarrow) f.first_wide = std::min(f.first_wide, l);
        }
    std::vector<int32_t> wrow(NF, 0);
    f.fwd_ptr.assign(1, 0);
    f.bwd_ptr.assign(1, 0);
    f.asm_ptr.assign(1, 0);
    for (int32_t l = 0; l < f.nlevels; ++l) {
        const bool wide = l >= f.first_wide;
        static const int heights[] = {64, 32};
        std::vector<int64_t> tf(2, 0), tb(2, 0);
        int32_t widest = 0;
        for (int32_t q = f.level_ptr[l]; q < f.level_ptr[l + 1]; ++q) {
            const int32_t t = f.level_nodes[q], ns = f.c0[t + 1] - f.c0[t];
            widest = std::max(widest, ns);
            for (int i = 0; i < 2; ++i) {
                tf[i] += (f.m[t] + heights[i] - 1) / heights[i];
                tb[i] += (ns + heights[i] - 1) / heights[i];
            }
        }
        const int rf = wide ? level_rows(tf, heights, 2) : (l == 0 ? kLeafRows : 64);
        const int rb = wide ? level_rows(tb, heights, 2) : (widest <= 32 ? 32 : 64);
        f.fwd_rows.push_back(rf);
        f.bwd_rows.push_back(rb);
        for (int32_t q = f.level_ptr[l]; q < f.level_ptr[l + 1]; ++q) {
            const int32_t t = f.level_nodes[q], ns = f.c0[t + 1] - f.c0[t], m = f.m[t];
            SweepTask k{};
            k.front = t;
            k.c0 = f.c0[t];
            k.ns = ns;
            k.row0 = f.row0[t];
            k.urow = f.uoff[t];
            if (wide) {
                wrow[t] = (int32_t)f.n_wrows;
                for (int32_t j = 0; j < ns; ++j) {
                    const int32_t r[4] = {(int32_t)(f.row0[t] + j), f.c0[t] + j, t, 0};
                    f.asm_rows.insert(f.asm_rows.end(), r, r + 4);
                }
                f.n_wrows += ns;
            }
            k.wrow = wrow[t];
            const int32_t hf1 = even_rows(m, rf), hb1 = even_rows(ns, rb);
            for (int32_t r0 = 0; r0 < m; r0 += hf1) {
                k.r0 = r0;
                k.h = std::min(hf1, m - r0);
                k.depth = std::min(ns, r0 + k.h);  // rows of the inverse reach their own column
                k.off64 = f.fwd64;
                k.off32 = f.fwd32;
                f.fwd64 += padded_depth(k.depth) * panel_ld(k.h, true);
                f.fwd32 += padded_depth(k.depth) * panel_ld(k.h, false);
                f.fwd.push_back(k);
            }
            for (int32_t r0 = 0; r0 < ns; r0 += hb1) {
                k.r0 = r0;
                k.h = std::min(hb1, ns - r0);
                k.depth = m - r0;
                k.off64 = f.bwd64;
                k.off32 = f.bwd32;
                f.bwd64 += padded_depth(k.depth) * panel_ld(k.h, true);
                f.bwd32 += padded_depth(k.depth) * panel_ld(k.h, false);
                f.bwd.push_back(k);
            }
        }
        if (l == 0) {
            for (const SweepTask& k : f.fwd) {
                f.leaf_fwd64 = std::max(f.leaf_fwd64, padded_depth(k.depth) * panel_ld(k.h, true));
                f.leaf_fwd32 = std::max(f.leaf_fwd32, padded_depth(k.depth) * panel_ld(k.h, false));
            }
            for (const SweepTask& k : f.bwd) {
                f.leaf_bwd64 = std::max(f.leaf_bwd64, padded_depth(k.depth) * panel_ld(k.h, true));
                f.leaf_bwd32 = std::max(f.leaf_bwd32, padded_depth(k.depth) * panel_ld(k.h, false));
            }
        }
        f.fwd_ptr.push_back((int32_t)f.fwd.size());
        f.bwd_ptr.push_back((int32_t)f.bwd.size());
        f.asm_ptr.push_back((int32_t)(f.asm_rows.size() / 4));
    }
    return 0;
}

}  // namespace fcw
