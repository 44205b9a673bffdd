// A growing buffer (csrc/staging.h) over calls of given sizes, with an allocator that refuses more than
// `limit` entries. Prints, per call, its status and the buffer's capacity; fails when a call that
// succeeds leaves no buffer of its size, or when a buffer leaks or is freed twice.
#include <cstdio>
#include <cstdlib>
#include <set>

#include "staging.h"

int main(int argc, char** argv) {
    const long limit = std::atol(argv[1]);
    std::set<double*> live;
    double* p = nullptr;
    int64_t cap = 0;
    auto alloc = [&](double** q, int64_t n) {
        *q = nullptr;
        if (n > limit) return 7;
        *q = new double[n];
        live.insert(*q);
        return 0;
    };
    auto release = [&](double* q) {
        if (!live.erase(q)) std::exit(1);
        delete[] q;
    };
    for (int i = 2; i < argc; ++i) {
        const int64_t need = std::atol(argv[i]);
        const int rc = fcw::grow_staging(p, cap, need, alloc, release);
        if (rc == 0 && (!p || cap < need)) return 2;
        if (rc != 0 && (p || cap != 0)) return 3;
        if (live.size() != (p ? 1u : 0u) || (p && !live.count(p))) return 4;
        if (p) p[need - 1] = 1.0;
        std::printf("%d:%ld ", rc, (long)cap);
    }
    if (p) release(p);
    return live.empty() ? 0 : 5;
}
