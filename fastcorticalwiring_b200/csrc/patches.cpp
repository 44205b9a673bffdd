// The divergence's view of the mesh (face.cu): each vertex's faces as fans, and patches of vertices.
#include "patches.h"

#include <algorithm>
#include <future>
#include <system_error>
#include <thread>

namespace fcw {

namespace {

// Each vertex's incident faces as fans for the mixed divergence (FaceData): walks from face to face
// over the neighbour they share, first from the neighbours with one face (boundary ends), then around
// the closed fans. A neighbour with more than two faces at the vertex (a non-manifold edge) ends fans.
// Vertices [v0, v1): ptr[v + 1] = the steps of the range up to and with v.
void fans_of(const MeshPrep& m, const std::vector<int32_t>& fv, const std::vector<int32_t>& inc_ptr,
             const std::vector<int32_t>& inc_face, const std::vector<int8_t>& inc_corner, int64_t v0, int64_t v1,
             std::vector<int32_t>& ptr, std::vector<FanStep>& steps, std::vector<int32_t>& walked) {
    const int64_t n = (int64_t)inc_ptr.size() - 1, most = inc_ptr[v1] - inc_ptr[v0] + (v1 - v0);
    steps.reserve(most);
    walked.reserve(2 * most);
    std::vector<int32_t> at(n, -1);                   // neighbour -> its slot at the current vertex
    std::vector<int32_t> slot_face, slot_count, slot_of, done;  // two faces per slot; the faces' two slots
    for (int64_t v = v0; v < v1; ++v) {
        const int32_t q0 = inc_ptr[v], deg = inc_ptr[v + 1] - q0;
        slot_face.clear();
        slot_count.clear();
        slot_of.assign(2 * deg, 0);
        done.assign(deg, 0);
        auto other = [&](int32_t i, int k) {  // neighbour k (0, 1) of the vertex on its i-th face
            return fv[3 * (int64_t)inc_face[q0 + i] + (inc_corner[q0 + i] + 1 + k) % 3];
        };
        for (int32_t i = 0; i < deg; ++i)
            for (int k = 0; k < 2; ++k) {
                int32_t& s = at[other(i, k)];
                if (s < 0) {
                    s = (int32_t)slot_count.size();
                    slot_count.push_back(0);
                    slot_face.insert(slot_face.end(), 2, -1);
                }
                if (slot_count[s] < 2) slot_face[2 * s + slot_count[s]] = i;
                slot_count[s]++;
                slot_of[2 * i + k] = s;
            }
        auto walk = [&](int32_t i, int k) {  // the fan that starts at neighbour k of face i
            const size_t first = steps.size();
            steps.push_back({{0.0f, 0.0f}, {0.0f, 0.0f}, {0.0f, 0.0f}, other(i, k), 0});
            walked.insert(walked.end(), {other(i, k), -1});
            for (;;) {
                done[i] = 1;
                const double* g = &m.gb[9 * (int64_t)inc_face[q0 + i]];
                const double* a = g + 3 * ((inc_corner[q0 + i] + 1 + k) % 3);
                const double* b = g + 3 * ((inc_corner[q0 + i] + 2 - k) % 3);
                auto dot = [](const double* x, const double* y) { return x[0] * y[0] + x[1] * y[1] + x[2] * y[2]; };
                const double area = m.grad_area[inc_face[q0 + i]], aa = area * area;
                const float c11 = (float)(aa * dot(a, a)), c12 = (float)(aa * dot(a, b)), c22 = (float)(aa * dot(b, b));
                steps.push_back({{c11, c11}, {c12, c12}, {c22, c22}, other(i, 1 - k), -1});
                steps[first].faces++;
                walked.insert(walked.end(), {other(i, 1 - k), inc_face[q0 + i]});
                const int32_t s = slot_of[2 * i + 1 - k];
                if (slot_count[s] != 2) return;
                const int32_t nxt = slot_face[2 * s] == i ? slot_face[2 * s + 1] : slot_face[2 * s];
                if (done[nxt]) return;
                k = slot_of[2 * nxt] == s ? 0 : 1;
                i = nxt;
            }
        };
        for (int32_t i = 0; i < deg; ++i)
            for (int k = 0; k < 2; ++k)
                if (!done[i] && slot_count[slot_of[2 * i + k]] != 2) walk(i, k);
        for (int32_t i = 0; i < deg; ++i)
            if (!done[i]) walk(i, 0);
        for (int32_t i = 0; i < deg; ++i)
            for (int k = 0; k < 2; ++k) at[other(i, k)] = -1;
        ptr[v + 1] = (int32_t)steps.size();
    }
}

}  // namespace

// The vertices in equal ranges, one per thread, joined in order: the same arrays for any number of them.
// 147k vertices on eight cores: 74 ms with one thread, 35 with eight; 9k vertices 2.8 and 2.0 (three).
void face_fans(const MeshPrep& m, const std::vector<int32_t>& fv, const std::vector<int32_t>& inc_ptr,
               const std::vector<int32_t>& inc_face, const std::vector<int8_t>& inc_corner,
               std::vector<int32_t>& ptr, std::vector<FanStep>& steps, std::vector<int32_t>& walked, int threads) {
    const int64_t n = (int64_t)inc_ptr.size() - 1;
    ptr.assign(n + 1, 0);
    steps.clear();
    walked.clear();
    const int most = std::max(1, (int)std::min<int64_t>(8, std::thread::hardware_concurrency()));
    const int parts = threads > 0 ? threads : (int)std::min<int64_t>(most, n / kFanRange + 1);
    auto first = [&](int r) { return n * r / parts; };
    struct Range {
        std::vector<FanStep> steps;
        std::vector<int32_t> walked;
        std::future<void> done;  // waits for its thread when another range fails
    };
    std::vector<Range> ranges(parts - 1);
    auto form = [&](int r, std::vector<FanStep>& st, std::vector<int32_t>& wk) {
        fans_of(m, fv, inc_ptr, inc_face, inc_corner, first(r), first(r + 1), ptr, st, wk);
    };
    for (int r = 1; r < parts; ++r) {
        Range& g = ranges[r - 1];
        try {
            g.done = std::async(std::launch::async, [&form, &g, r] { form(r, g.steps, g.walked); });
        } catch (const std::system_error&) {  // no thread to be had
            form(r, g.steps, g.walked);
        }
    }
    form(0, steps, walked);
    size_t total = steps.size();
    for (Range& g : ranges) {
        if (g.done.valid()) g.done.get();
        total += g.steps.size();
    }
    steps.reserve(total);
    walked.reserve(2 * total);
    for (int r = 1; r < parts; ++r) {
        Range& g = ranges[r - 1];
        for (int64_t v = first(r); v < first(r + 1); ++v) ptr[v + 1] += (int32_t)steps.size();
        steps.insert(steps.end(), g.steps.begin(), g.steps.end());
        walked.insert(walked.end(), g.walked.begin(), g.walked.end());
    }
}

void sharp_fans(const MeshPrep& m, const std::vector<int32_t>& fv, const std::vector<int32_t>& fan_ptr,
                const std::vector<FanStep>& steps, const std::vector<int32_t>& walk, SharpFans& sf) {
    const int32_t n = (int32_t)fan_ptr.size() - 1;
    auto sharp = [](const FanStep& s) {  // an acute corner; a fan's first step has no coefficients
        const double a = s.c11[0], b = s.c12[0], c = s.c22[0];
        return b < 0.0 && a * c - b * b < kSharp * a * c;
    };
    sf.ptr.assign(1, 0);
    for (int32_t v = 0; v < n; ++v) {
        bool any = false;
        for (int32_t e = fan_ptr[v]; e < fan_ptr[v + 1] && !any; ++e) any = sharp(steps[e]);
        if (!any) continue;
        sf.vertices.push_back(v);
        for (int32_t e = fan_ptr[v]; e < fan_ptr[v + 1]; ++e) {
            const FanStep& x = steps[e];
            FanStep s{{x.c11[0], x.c11[1]}, {x.c12[0], x.c12[1]}, {x.c22[0], x.c22[1]}, walk[2 * (int64_t)e], x.faces};
            if (sharp(x)) {
                const int64_t f = walk[2 * (int64_t)e + 1];
                auto gradient = [&](int32_t w) {
                    int c = 0;
                    while (c < 2 && fv[3 * f + c] != w) ++c;
                    return &m.gb[9 * f + 3 * c];
                };
                const double *gv = gradient(v), *gn = gradient(s.neighbour), aa = m.grad_area[f] * m.grad_area[f];
                auto dot = [](const double* x, const double* y) { return x[0] * y[0] + x[1] * y[1] + x[2] * y[2]; };
                s.c11[0] = s.c11[1] = (float)(aa * dot(gv, gv));
                s.c12[0] = s.c12[1] = (float)(-aa * dot(gv, gn));
                s.faces = -2;
            }
            sf.steps.push_back(s);
        }
        sf.ptr.push_back((int32_t)sf.steps.size());
    }
}

// Consecutive vertices join a patch while its rows and fan steps fit. A vertex's rows are itself and
// the neighbours its steps name.
void face_patches(const std::vector<int32_t>& fan_ptr, std::vector<FanStep>& steps, PatchArrays& pa) {
    const int32_t n = (int32_t)fan_ptr.size() - 1;
    std::vector<int32_t> row_at(n, -1);  // place in the current patch (0 while it grows)
    std::vector<int32_t> seen, fresh;    // the patch's rows; those the current vertex would add
    int32_t v0 = 0;
    auto close = [&](int32_t v1) {
        if (v1 == v0) return;
        Patch p{};
        p.v0 = v0;
        p.nv = v1 - v0;
        p.row0 = (int32_t)pa.rows.size();
        p.nsteps = fan_ptr[v1] - fan_ptr[v0];
        for (int32_t v = v0; v < v1; ++v) {
            row_at[v] = v - v0;
            pa.rows.push_back(v);
        }
        p.nrows = p.nv;
        for (int32_t v : seen)
            if (v < v0 || v >= v1) {
                row_at[v] = p.nrows++;
                pa.rows.push_back(v);
            }
        for (int32_t q = fan_ptr[v0]; q < fan_ptr[v1]; ++q) steps[q].neighbour = row_at[steps[q].neighbour];
        for (int32_t v : seen) row_at[v] = -1;
        seen.clear();
        pa.patches.push_back(p);
        v0 = v1;
    };
    for (int32_t v = 0; v < n; ++v) {
        for (;;) {
            fresh.clear();
            auto visit = [&](int32_t w) {
                if (row_at[w] < 0) {
                    row_at[w] = 0;
                    fresh.push_back(w);
                }
            };
            visit(v);
            for (int32_t q = fan_ptr[v]; q < fan_ptr[v + 1]; ++q) visit(steps[q].neighbour);
            if (v - v0 < kPatchVerts && (int32_t)(seen.size() + fresh.size()) <= kPatchRows &&
                fan_ptr[v + 1] - fan_ptr[v0] <= kPatchSteps) {
                seen.insert(seen.end(), fresh.begin(), fresh.end());
                break;
            }
            for (int32_t w : fresh) row_at[w] = -1;
            if (v == v0) {  // not even alone
                pa.big.push_back(v);
                v0 = v + 1;
                break;
            }
            close(v);
        }
    }
    close(n);
}

}  // namespace fcw
