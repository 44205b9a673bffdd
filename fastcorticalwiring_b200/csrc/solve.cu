// Multi-right-hand-side triangular solves over fronts, one tree level per launch.
//
// Right-hand sides and results are n x K row-major (a vertex row holds K contiguous right-hand
// sides). A CTA owns one task of one front and one column tile of the right-hand sides (64 columns
// in FP64, 128 in FP32: a tile row is 512 bytes either way), so all row traffic is contiguous
// 512-byte segments.
//
// With A_s = [inv(L_ss); Q_s], Q_s = L_rs inv(L_ss) (fronts.cu):
//
// Forward (leaves -> root), multifrontal: front s forms
//   W   = b_s - the children's update rows that land on s's columns
//   X_s = inv(L_ss) W                                   (written to Y)
//   U_s = Q_s W + the children's update rows that land on s's structure
// and leaves U_s for its parent. A task is a group of stacked rows of A_s: a leaf's first 128 (its A_s
// has 88 rows on average, so mostly all of it), 64 elsewhere, 32 where a level has few. On the levels
// whose fronts are at most 64 columns wide each task gathers W itself, into shared memory. The wider
// fronts near the root have many tasks, so there W is assembled once (k_assemble) and the products read
// it in 32-row chunks.
// Children's rows are added in ascending child order, so results are deterministic.
//
// Backward (root -> leaves): X_s = A_s^T [y_s; -X_r], X_r the structure rows (ancestors, final). A
// task is up to 64 of the front's columns over all rows below them, gathered in 32-row chunks, two
// chunks in flight. The solution goes to an array of its own, so tasks of one front need no order.
//
// Each task's part of A_s is stored as it is used: k-major (for each depth row, the task's rows or
// columns side by side), one bulk copy (cp.async.bulk) per 32-row chunk, requested before anything
// else. FP64 products run on the FP64 tensor path (mma.sync m8n8k4; tcgen05 has no FP64 kind), FP32
// products on packed FMAs (fma.rn.f32x2: two columns per instruction, which leaves issue slots for
// the shared-memory reads). A warp owns 16 rows, so a task computes its rows rounded up to 16, and
// the triangles of inv(L_ss) are cut at 16.
//
// Launches overlap: a level's CTAs read their task, request their panels and load their gather lists
// while the previous level finishes (programmatic dependent launch), then wait for it. Every sweep
// kernel lets its dependents start before its own wait, so a chain of them may have started while the
// first still waits: what a kernel reads before its wait has to be complete before the chain begins.
//
// Heat right-hand sides are columns of the identity: the forward sweep builds them from the source
// list, and only fronts on a source's path to the root (`reach`, per front and 64-column tile) are
// solved; the others' forward results are zero and are not read. The backward sweep reads `reach` before
// its wait (which rows of the panel to request follows from it), so the chain's first kernel is launched
// in order after k_reach, without overlap; it would wait for `reach` before all else anyway.
#include <algorithm>
#include <type_traits>

#include "kernels.cuh"
#include "tc.cuh"

namespace fcw {

namespace {

constexpr int NT = 256;  // threads per CTA
constexpr int DC = 32;   // depth rows per chunk
constexpr int kNarrowCols = 64;  // columns of a front whose right-hand side one task gathers

template <typename T>
constexpr int vec() { return 16 / (int)sizeof(T); }  // elements per 16-byte vector
template <typename T>
constexpr int wide_tile() { return sizeof(T) == 4 ? 128 : 64; }
// Right-hand-side rows in shared memory. FP64 tensor fragments read 4 depths x 8 columns: a row
// stride of 8 banks more than a multiple of 32 keeps them apart (as the panels' row stride does).
template <typename T, int KT>
constexpr int ld_rhs() { return sizeof(T) == 8 ? KT + 4 : KT; }
template <typename T, int M>
constexpr int panel_stage() { return DC * (sizeof(T) == 8 ? M + 4 : M); }  // elements of a chunk's panel rows
template <typename T>
__device__ __forceinline__ int panel_stride(int h) { return (h + 7) / 8 * 8 + (sizeof(T) == 8 ? 4 : 0); }

__device__ __forceinline__ void allow_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_predecessor() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void copy16_async(void* smem, const void* gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(tc::smem_u32(smem)), "l"(gmem) : "memory");
}
__device__ __forceinline__ void copy16_async_or_zero(void* smem, const void* gmem, bool copy) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(tc::smem_u32(smem)), "l"(gmem),
                 "r"(copy ? 16 : 0)
                 : "memory");
}
__device__ __forceinline__ void copy_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// A panel copy that does not land in time raises KERR_TIMEOUT; the second bounded wait lets a late
// copy finish before the CTA goes on.
__device__ __forceinline__ void wait_panel(uint64_t* bar, uint32_t parity, int* err) {
    if (!tc::mbar_wait(bar, parity)) {
        atomicOr(err, KERR_TIMEOUT);
        tc::mbar_wait(bar, parity);
    }
}

// V adjacent elements (4 to 16 bytes, aligned); values other launches wrote.
template <typename T, int V>
__device__ __forceinline__ void ld_n(const T* p, T* w) {
    if constexpr (V * sizeof(T) == 16 && sizeof(T) == 4) {
        const float4 x = *reinterpret_cast<const float4*>(p);
        w[0] = x.x; w[1] = x.y; w[2] = x.z; w[3] = x.w;
    } else if constexpr (V * sizeof(T) == 16) {
        const double2 x = *reinterpret_cast<const double2*>(p);
        w[0] = x.x; w[1] = x.y;
    } else if constexpr (V == 2) {
        const float2 x = *reinterpret_cast<const float2*>(p);
        w[0] = x.x; w[1] = x.y;
    } else {
        w[0] = *p;
    }
}
template <typename T, int V>
__device__ __forceinline__ void st_n(T* p, const T* w) {
    if constexpr (V * sizeof(T) == 16 && sizeof(T) == 4) *reinterpret_cast<float4*>(p) = make_float4(w[0], w[1], w[2], w[3]);
    else if constexpr (V * sizeof(T) == 16) *reinterpret_cast<double2*>(p) = make_double2(w[0], w[1]);
    else if constexpr (V == 2) *reinterpret_cast<float2*>(p) = make_float2(w[0], w[1]);
    else *p = w[0];
}

// ---------------------------------------------------------------------------
// Products C (M x KT) += P V on shared-memory tiles, P k-major (P[d * ld + row]), V[d * ldv + col].
// Eight warps: warp group g = 16 rows, and with fewer than 8 groups the column tile is split
// between the warps of a group. run(): depths [d0, nd); rows and cols of a thread's accumulators
// are visited in vectors of V adjacent columns.
// ---------------------------------------------------------------------------
__device__ __forceinline__ int logical_warp() {
    // tasks shorter than M leave the last groups idle: other CTAs of the SM get other idle warps
    return ((threadIdx.x >> 5) + 2 * (blockIdx.x & 3)) & 7;
}

template <int KT, int M>
struct AccF32 {
    using T = float;
    static constexpr int CS = 128 / M, WN = KT / CS, CN = WN / 16;  // column split, warp and thread columns
    static constexpr int V = CN >= 4 ? 4 : CN, NV = CN / V;
    float c[8][CN];

    __device__ __forceinline__ int group() const { return logical_warp() / CS; }
    __device__ __forceinline__ int row0() const { return 16 * group() + 8 * ((threadIdx.x >> 4) & 1); }
    __device__ __forceinline__ int col0() const { return (logical_warp() % CS) * WN + V * (threadIdx.x & 15); }
    static constexpr int vstep() { return 16 * V; }

    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int q = 0; q < CN; ++q) c[i][q] = 0.0f;
    }
    __device__ __forceinline__ void run(const float* P, int ld, const float* Vm, int ldv, int d0, int nd, int) {
        const float* pp = P + row0();
        const float* vp = Vm + col0();
#pragma unroll 4
        for (int d = d0; d < nd; ++d) {
            float p[8], w[CN];
            ld_n<float, 4>(pp + d * ld, p);
            ld_n<float, 4>(pp + d * ld + 4, p + 4);
#pragma unroll
            for (int v = 0; v < NV; ++v) ld_n<float, V>(vp + d * ldv + vstep() * v, w + V * v);
            if constexpr (CN == 1) {
#pragma unroll
                for (int i = 0; i < 8; ++i) c[i][0] = fmaf(p[i], w[0], c[i][0]);
            } else {
                unsigned long long w2[CN / 2];
#pragma unroll
                for (int q = 0; q < CN / 2; ++q)
                    asm("mov.b64 %0, {%1, %2};" : "=l"(w2[q]) : "f"(w[2 * q]), "f"(w[2 * q + 1]));
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    unsigned long long p2;
                    asm("mov.b64 %0, {%1, %1};" : "=l"(p2) : "f"(p[i]));
#pragma unroll
                    for (int q = 0; q < CN / 2; ++q) {
                        unsigned long long x;
                        asm("mov.b64 %0, {%1, %2};" : "=l"(x) : "f"(c[i][2 * q]), "f"(c[i][2 * q + 1]));
                        asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(x) : "l"(p2), "l"(w2[q]));
                        asm("mov.b64 {%0, %1}, %2;" : "=f"(c[i][2 * q]), "=f"(c[i][2 * q + 1]) : "l"(x));
                    }
                }
            }
        }
    }
    // f(row, col, float* v): V adjacent columns
    template <class F>
    __device__ __forceinline__ void visit(int nrows, F&& f) {
        const int r0 = row0(), k0 = col0();
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (r0 + i < nrows)
#pragma unroll
                for (int v = 0; v < NV; ++v) f(r0 + i, k0 + vstep() * v, &c[i][V * v]);
    }
};

// FP64 tensor tiles: lane (g = lane / 4, t = lane % 4) holds row 8m + g, columns 8n + 2t and + 1 of
// the warp's 16 x WN tile. The depth runs in steps of 4; padded depths are zero in both operands.
template <int KT, int M>
struct AccF64 {
    using T = double;
    static constexpr int CS = 128 / M, WN = KT / CS, NN = WN / 8, V = 2;
    double c[2][NN][2];

    __device__ __forceinline__ int group() const { return logical_warp() / CS; }
    __device__ __forceinline__ int colw() const { return (logical_warp() % CS) * WN; }
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int n = 0; n < NN; ++n) c[m][n][0] = c[m][n][1] = 0.0;
    }
    template <int MM>
    __device__ __forceinline__ void steps(const double* P, int ld, const double* Vm, int ldv, int d0, int nd) {
        const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
        const double* pp = P + t * ld + 16 * group() + g;
        const double* vp = Vm + t * ldv + colw() + g;
        for (int d = d0; d < nd; d += 4) {
            double a[MM], b[NN];
#pragma unroll
            for (int m = 0; m < MM; ++m) a[m] = pp[d * ld + 8 * m];
#pragma unroll
            for (int n = 0; n < NN; ++n) b[n] = vp[d * ldv + 8 * n];
#pragma unroll
            for (int m = 0; m < MM; ++m)
#pragma unroll
                for (int n = 0; n < NN; ++n)
                    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
                        : "+d"(c[m][n][0]), "+d"(c[m][n][1])
                        : "d"(a[m]), "d"(b[n]));
        }
    }
    // rows: the task's rows (a group whose last 8 rows are past them runs one row tile)
    __device__ __forceinline__ void run(const double* P, int ld, const double* Vm, int ldv, int d0, int nd, int rows) {
        if (16 * group() + 8 < rows) steps<2>(P, ld, Vm, ldv, d0, nd);
        else steps<1>(P, ld, Vm, ldv, d0, nd);
    }
    template <class F>
    __device__ __forceinline__ void visit(int nrows, F&& f) {
        const int lane = threadIdx.x & 31, r = 16 * group() + (lane >> 2), k0 = colw() + 2 * (lane & 3);
#pragma unroll
        for (int m = 0; m < 2; ++m)
            if (r + 8 * m < nrows)
#pragma unroll
                for (int n = 0; n < NN; ++n) f(r + 8 * m, k0 + 8 * n, c[m][n]);
    }
};

template <typename T, int KT, int M>
using Acc = std::conditional_t<sizeof(T) == 8, AccF64<KT, M>, AccF32<KT, M>>;

// ---------------------------------------------------------------------------
// Children's update rows
// ---------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ bool reached(const SweepArgs<T>& a, int front, int tile) {
    return !a.reach || __ldcg(a.reach + (int64_t)front * a.reach_tiles + tile);
}
// A front row's record, without the children that are off the sources' paths (their update rows
// were never written).
template <typename T>
__device__ __forceinline__ int4 live_record(const SweepArgs<T>& a, int64_t q, int tile) {
    int4 r = a.rec[q];
    if (a.reach) {
        const int32_t* ch = a.rec_child + 3 * q;
        const int c0 = ch[0], c1 = ch[1], c2 = ch[2];
        if (r.x >= 0 && !reached(a, c0, tile)) r.x = -1;
        if (r.y >= 0 && !reached(a, c1, tile)) r.y = -1;
        if (r.z >= 0 && !reached(a, c2, tile)) r.z = -1;
    }
    return r;
}
// w (+ or -)= the record's rows after the first three
template <typename T, int V, bool SUB>
__device__ __forceinline__ void add_more(const SweepArgs<T>& a, int more, int tile, const T* U, T* w) {
    const int n = a.more[more];
    for (int e = 0; e < n; ++e) {
        if (!reached(a, a.more[more + 2 + 2 * e], tile)) continue;
        T u[V];
        ld_n<T, V>(U + (int64_t)a.more[more + 1 + 2 * e] * a.K, u);
#pragma unroll
        for (int q = 0; q < V; ++q) w[q] = SUB ? w[q] - u[q] : w[q] + u[q];
    }
}

// R rows' vectors at column k (16 bytes each) minus their records' rows: base[] holds the
// right-hand-side rows (negative: zero row). All loads of the R rows are in flight together.
template <typename T, int R>
__device__ __forceinline__ void gather_rows(const SweepArgs<T>& a, const int4* rec, const int64_t* base, int k, int tile,
                                            const int* delta, T (*w)[vec<T>()]) {
    constexpr int G = vec<T>();
    const T* U = a.U + k;
    T u[R][G];
#pragma unroll
    for (int i = 0; i < R; ++i) {
        if (a.delta_src) {
#pragma unroll
            for (int q = 0; q < G; ++q) w[i][q] = (base[i] >= 0 && delta[q] == (int)base[i]) ? T(1) : T(0);
        } else if (base[i] >= 0) {
            ld_n<T, G>(a.R + base[i] * a.K + k, w[i]);
        } else {
#pragma unroll
            for (int q = 0; q < G; ++q) w[i][q] = T(0);
        }
    }
#pragma unroll
    for (int s = 0; s < 3; ++s) {
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const int src = s == 0 ? rec[i].x : (s == 1 ? rec[i].y : rec[i].z);
            if (src >= 0) ld_n<T, G>(U + (int64_t)src * a.K, u[i]);
        }
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const int src = s == 0 ? rec[i].x : (s == 1 ? rec[i].y : rec[i].z);
            if (src >= 0) {
#pragma unroll
                for (int q = 0; q < G; ++q) w[i][q] -= u[i][q];
            }
        }
    }
#pragma unroll
    for (int i = 0; i < R; ++i)
        if (rec[i].w >= 0) add_more<T, G, true>(a, rec[i].w, tile, U, w[i]);
}

// ---------------------------------------------------------------------------
// Forward
// ---------------------------------------------------------------------------
template <typename T, int KT, int M, bool WIDE>
__global__ void __launch_bounds__(NT, M == 128 ? 2 : 3) k_fwd(SweepArgs<T> a, int32_t t0) {
    constexpr int G = vec<T>(), VPR = KT / G, RPP = NT / VPR, LW = ld_rhs<T, KT>();
    constexpr int S = 2;  // chunks resident: all of a narrow front's (kNarrowCols / DC)
    constexpr int PS = panel_stage<T, M>(), VS = DC * LW;
    extern __shared__ __align__(128) unsigned char smraw[];
    T* Ps = reinterpret_cast<T*>(smraw);
    T* Vs = Ps + S * PS;
    __shared__ __align__(8) uint64_t bar[S];
    __shared__ int4 crec[WIDE ? 1 : kNarrowCols], urec[M];
    allow_dependents();
    const int tid = threadIdx.x, tile = blockIdx.y, k0 = tile * KT;
    const SweepTask t = a.tasks[t0 + blockIdx.x];
    if (a.reach) {
        wait_predecessor();
        if (!reached(a, t.front, tile)) return;
    }
    const int ld = panel_stride<T>(t.h);
    const T* panel = a.panel + (sizeof(T) == 8 ? t.off64 : t.off32);
    const int depth4 = (t.depth + 3) & ~3, nch = (t.depth + DC - 1) / DC;
    auto chunk_rows = [&](int c) { return min(DC, depth4 - DC * c); };
    auto request = [&](int c) {  // chunk c's panel rows, by one thread
        const uint32_t bytes = (uint32_t)(chunk_rows(c) * ld * (int)sizeof(T));
        tc::mbar_arrive_expect_tx(&bar[c % S], bytes);
        tc::bulk_load(Ps + (c % S) * PS, panel + (int64_t)c * DC * ld, bytes, &bar[c % S]);
    };
    if (tid == 0) {
        for (int s = 0; s < S; ++s) tc::mbar_init(&bar[s], 1);
        tc::fence_mbar_init();
        for (int c = 0; c < min(nch, WIDE ? S - 1 : S); ++c) request(c);
    }
    if (a.gathers) {
        if (!WIDE)
            for (int i = tid; i < t.ns; i += NT) crec[i] = live_record(a, t.row0 + i, tile);
        for (int i = tid; i < t.h; i += NT)
            urec[i] = t.r0 + i >= t.ns ? live_record(a, t.row0 + t.r0 + i, tile) : make_int4(-1, -1, -1, -1);
    }
    if (!a.reach) wait_predecessor();
    __syncthreads();  // the barriers are initialised, the records are in

    if (!WIDE && !a.gathers && !a.delta_src) {
        // a leaf's W is its rows of R: all of them in flight at once
        for (int e = tid; e < depth4 * VPR; e += NT) {
            const int f = e / VPR, v = e - f * VPR;
            T* dst = Vs + f * LW + v * G;
            if (f < t.depth) {
                copy16_async(dst, a.R + (int64_t)(t.c0 + f) * a.K + k0 + v * G);
            } else {
                T z[G] = {};
                st_n<T, G>(dst, z);
            }
        }
        copy_async_commit();
        copy_async_wait<0>();
    } else if constexpr (!WIDE) {
        // W, four rows per thread in flight
        const int v = tid % VPR, rr = tid / VPR;
        int delta[G];
        if (a.delta_src) {
#pragma unroll
            for (int q = 0; q < G; ++q) delta[q] = a.delta_src[k0 + v * G + q];
        }
        constexpr int R = 4;
        for (int f0 = rr; f0 < depth4; f0 += R * RPP) {
            int4 rec[R];
            int64_t base[R];
            T w[R][G];
#pragma unroll
            for (int i = 0; i < R; ++i) {
                const int f = f0 + i * RPP;
                base[i] = f < t.depth ? t.c0 + f : -1;
                rec[i] = (a.gathers && f < t.depth) ? crec[f] : make_int4(-1, -1, -1, -1);
            }
            gather_rows<T, R>(a, rec, base, k0 + v * G, tile, delta, w);
#pragma unroll
            for (int i = 0; i < R; ++i) {
                const int f = f0 + i * RPP;
                if (f < depth4) st_n<T, G>(Vs + f * LW + v * G, w[i]);
            }
        }
    }
    auto load_chunk = [&](int c) {  // wide: chunk c of the assembled right-hand sides
        T* V = Vs + (c % S) * VS;
        const int nd = min(DC, t.depth - DC * c), n4 = chunk_rows(c);
        for (int e = tid; e < n4 * VPR; e += NT) {
            const int f = e / VPR, v = e - f * VPR;
            T* dst = V + f * LW + v * G;
            if (f < nd) {
                copy16_async(dst, a.W + (int64_t)(t.wrow + DC * c + f) * a.K + k0 + v * G);
            } else {
                T z[G] = {};
                st_n<T, G>(dst, z);
            }
        }
    };
    if constexpr (WIDE) {
        for (int c = 0; c < S - 1; ++c) {
            if (c < nch) load_chunk(c);
            copy_async_commit();
        }
    }
    // the children's rows that land on this task's structure rows start the accumulators
    Acc<T, KT, M> acc;
    using A = Acc<T, KT, M>;
    acc.zero();
    if (a.gathers && t.r0 + t.h > t.ns) {
        const T* U = a.U + k0;
#pragma unroll
        for (int s = 0; s < 3; ++s)
            acc.visit(t.h, [&](int r, int c, T* v) {
                const int src = s == 0 ? urec[r].x : (s == 1 ? urec[r].y : urec[r].z);
                if (src < 0) return;
                T u[A::V];
                ld_n<T, A::V>(U + (int64_t)src * a.K + c, u);
#pragma unroll
                for (int q = 0; q < A::V; ++q) v[q] += u[q];
            });
        acc.visit(t.h, [&](int r, int c, T* v) {
            if (urec[r].w >= 0) add_more<T, A::V, false>(a, urec[r].w, tile, U + c, v);
        });
    }
    // rows of the inverse stop at the diagonal
    const int g16 = 16 * acc.group(), last = t.r0 + g16 + 15;
    const int limit = g16 < t.h ? (last < t.ns ? min(t.depth, last + 1) : t.depth) : 0;
    for (int c = 0; c < nch; ++c) {
        if constexpr (WIDE) copy_async_wait<S - 2>();
        wait_panel(&bar[c % S], (c / S) & 1, a.err);
        if (WIDE || c == 0) __syncthreads();
        if constexpr (WIDE) {
            if (c + S - 1 < nch) {
                if (tid == 0) request(c + S - 1);
                load_chunk(c + S - 1);
            }
            copy_async_commit();
        }
        const int nd = min(DC, limit - DC * c);
        if (nd > 0) acc.run(Ps + (c % S) * PS, ld, Vs + (c % S) * VS, LW, 0, nd, t.h);
    }
    T* y = a.Y + (int64_t)t.c0 * a.K + k0;
    T* u = a.U + (t.urow - t.ns) * (int64_t)a.K + k0;
    acc.visit(t.h, [&](int r, int c, T* v) {
        const int R = t.r0 + r;
        st_n<T, A::V>((R < t.ns ? y : u) + (int64_t)R * a.K + c, v);
    });
}

// Right-hand sides of the wide levels' fronts: W = b - the children's update rows.
template <typename T, int KT>
__global__ void __launch_bounds__(NT) k_assemble(SweepArgs<T> a, int32_t r0, int32_t nrows) {
    constexpr int G = vec<T>(), VPR = KT / G, RPP = NT / VPR;
    allow_dependents();
    const int tile = blockIdx.y, v = threadIdx.x % VPR, i = blockIdx.x * RPP + threadIdx.x / VPR;
    const int k = tile * KT + v * G;
    const int4 row = i < nrows ? a.asm_rows[r0 + i] : make_int4(0, 0, -1, 0);
    int4 rec[1] = {make_int4(-1, -1, -1, -1)};
    wait_predecessor();
    if (i >= nrows || !reached(a, row.z, tile)) return;
    rec[0] = live_record(a, row.x, tile);
    const int64_t base[1] = {row.y};
    int delta[G];
    if (a.delta_src) {
#pragma unroll
        for (int q = 0; q < G; ++q) delta[q] = a.delta_src[k + q];
    }
    T w[1][G];
    gather_rows<T, 1>(a, rec, base, k, tile, delta, w);
    st_n<T, G>(a.W + (int64_t)(r0 + i) * a.K + k, w[0]);
}

// ---------------------------------------------------------------------------
// Backward
// ---------------------------------------------------------------------------
// Two chunks in flight: a third leaves an SM two FP64 CTAs instead of three (147k vertices, 1024
// columns: 1.12 against 1.32 ms for the heat solve) and gains FP32 nothing (1.12 ms either way; 64
// columns 0.24 against 0.28 ms).
constexpr int kBwdStages = 2;
template <typename T, int KT, int M>
__global__ void __launch_bounds__(NT, 3) k_bwd(SweepArgs<T> a, int32_t t0) {
    constexpr int G = vec<T>(), VPR = KT / G, LW = ld_rhs<T, KT>(), S = kBwdStages;
    constexpr int PS = panel_stage<T, M>(), VS = DC * LW;
    extern __shared__ __align__(128) unsigned char smraw[];
    T* Ps = reinterpret_cast<T*>(smraw);
    T* Vs = Ps + S * PS;
    int32_t* idx = reinterpret_cast<int32_t*>(Vs + S * VS);  // the task's depth rows
    __shared__ __align__(8) uint64_t bar[S];
    allow_dependents();
    const int tid = threadIdx.x, tile = blockIdx.y, k0 = tile * KT;
    const SweepTask t = a.tasks[t0 + blockIdx.x];
    const int own = t.ns - t.r0;  // depth rows [0, own): y_s; then the structure rows
    // y_s = 0 off the sources' paths (reach is complete before the chain of overlapped launches begins)
    const int d0 = (a.reach && !reached(a, t.front, tile)) ? own : 0;
    const int ld = panel_stride<T>(t.h);
    const T* panel = a.panel + (sizeof(T) == 8 ? t.off64 : t.off32);
    const int nrow = t.depth - d0, nrow4 = (nrow + 3) & ~3, nch = (nrow + DC - 1) / DC;
    auto chunk_rows = [&](int c) { return min(DC, nrow4 - DC * c); };
    auto request = [&](int c) {
        const uint32_t bytes = (uint32_t)(chunk_rows(c) * ld * (int)sizeof(T));
        tc::mbar_arrive_expect_tx(&bar[c % S], bytes);
        tc::bulk_load(Ps + (c % S) * PS, panel + (int64_t)(d0 + c * DC) * ld, bytes, &bar[c % S]);
    };
    if (tid == 0) {
        for (int s = 0; s < S; ++s) tc::mbar_init(&bar[s], 1);
        tc::fence_mbar_init();
        for (int c = 0; c < min(nch, S - 1); ++c) request(c);
    }
    for (int i = tid; i < nrow; i += NT) idx[i] = a.rows[t.row0 + t.r0 + d0 + i];
    wait_predecessor();
    __syncthreads();
    auto load_chunk = [&](int c) {
        T* V = Vs + (c % S) * VS;
        const int nd = min(DC, nrow - DC * c), n4 = chunk_rows(c);
        for (int e = tid; e < n4 * VPR; e += NT) {
            const int f = e / VPR, v = e - f * VPR, d = d0 + DC * c + f;
            T* dst = V + f * LW + v * G;
            if (f < nd) {
                const T* src = d < own ? a.Y : a.X;
                copy16_async(dst, src + (int64_t)idx[DC * c + f] * a.K + k0 + v * G);
            } else {
                T z[G] = {};
                st_n<T, G>(dst, z);
            }
        }
    };
    for (int c = 0; c < S - 1; ++c) {
        if (c < nch) load_chunk(c);
        copy_async_commit();
    }
    Acc<T, KT, M> acc;
    using A = Acc<T, KT, M>;
    acc.zero();
    const int g16 = 16 * acc.group();
    for (int c = 0; c < nch; ++c) {
        copy_async_wait<S - 2>();
        wait_panel(&bar[c % S], (c / S) & 1, a.err);
        __syncthreads();
        if (c + S - 1 < nch) {
            if (tid == 0) request(c + S - 1);
            load_chunk(c + S - 1);
        }
        copy_async_commit();
        // column j of the inverse starts at row j
        const int nd = min(DC, nrow - DC * c), from = max(0, g16 - d0 - DC * c);
        if (g16 < t.h && from < nd) acc.run(Ps + (c % S) * PS, ld, Vs + (c % S) * VS, LW, from, nd, t.h);
    }
    T* x = a.X + (int64_t)(t.c0 + t.r0) * a.K + k0;
    acc.visit(t.h, [&](int r, int c, T* v) { st_n<T, A::V>(x + (int64_t)r * a.K + c, v); });
}

// ---------------------------------------------------------------------------
// Leaves, panel resident
// ---------------------------------------------------------------------------
// Half the flops of a sweep are the leaves'. With a CTA per task and column tile, each CTA fetched its
// panel again, waited for its right-hand sides before it multiplied, and its warps waited for the
// longest one's rows at every chunk (the triangle makes them unequal; 5.5 of 8 had rows at all): 860 us
// forward and 740 backward for 460 us of FP64 tensor work each (147k vertices, 1024 columns). Here a CTA keeps its task's panel over many columns, and each warp takes column
// groups of its own (8 or 16 columns, all rows) with its own asynchronous ring of right-hand sides:
// warps have equal work and never meet, and loads run ahead across groups. Rows are cut at 8 instead of
// 16 (tiles no depth reaches are branched past: a predicated-off matrix instruction still takes its
// slot). Bound by issue around the matrix instructions (tensor pipe 60-66% busy). Poisson forward 2.12 to 1.96 ms and
// backward 1.48 to 1.36, heat backward 1.11 to 1.04; FP32 backward 1.12 to 1.08. FP32 forward takes the
// general kernel: more shared-memory reads per product here, 1.54 against 1.44 ms.
constexpr int LD = kLeafChunk;  // depth rows per chunk of a warp's ring
static_assert(kLeafWarps == NT / 32, "the plan's warps are the kernel's");

// Products of one warp: C (h rows x CW columns) += P V, P k-major in the CTA's panel, V the warp's own
// [depth][CW] rows. Row tiles are numbered so that the ones a depth reaches are the last: forward, the
// rows below the diagonal, so a task's last tile is the accumulators' last; backward, the columns left of
// it, so the order is reversed. A case per first tile then keeps every register index static.
struct WarpF32 {  // backward, 64 columns of X_s
    static constexpr int CW = 32, TC = 4, NQ = 4, V = TC;  // TC: a thread's columns
    unsigned long long c[NQ][2][TC];  // rows 4i + {0, 1}, {2, 3} of tile q
    static __device__ __forceinline__ int slot(int, int col) { return col; }
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int q = 0; q < NQ; ++q)
#pragma unroll
            for (int e = 0; e < 2 * TC; ++e) c[q][e / TC][e % TC] = 0ull;
    }
    static __device__ __forceinline__ int row(int q) { return 16 * (NQ - 1 - q); }
    template <int Q0>
    __device__ __forceinline__ void tiles(const float* pp, int ld, const float* vp, int nd) {
#pragma unroll 2
        for (int d = 0; d < nd; ++d) {
            float w[TC];
            ld_n<float, TC>(vp + d * CW, w);
            unsigned long long w2[TC];
#pragma unroll
            for (int e = 0; e < TC; ++e) asm("mov.b64 %0, {%1, %1};" : "=l"(w2[e]) : "f"(w[e]));
#pragma unroll
            for (int q = Q0; q < NQ; ++q) {
                const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(pp + d * ld - 16 * q);
#pragma unroll
                for (int e = 0; e < TC; ++e) {
                    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c[q][0][e]) : "l"(x.x), "l"(w2[e]));
                    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c[q][1][e]) : "l"(x.y), "l"(w2[e]));
                }
            }
        }
    }
    template <int A = 0, int B = NQ>  // q0 in [A, B)
    __device__ __forceinline__ void from(int q0, const float* pp, int ld, const float* vp, int nd) {
        constexpr int H = (A + B) / 2;
        if constexpr (B - A == 1) tiles<A>(pp, ld, vp, nd);
        else if (q0 < H) from<A, H>(q0, pp, ld, vp, nd);
        else from<H, B>(q0, pp, ld, vp, nd);
    }
    // depths [base, base + nd) of the task, P at its depth `base`
    __device__ __forceinline__ void run(const float* P, int ld, const float* Vm, int base, int, int nd, int h) {
        const int lane = threadIdx.x & 31, q0 = NQ - min((h + 15) / 16, (base + LD - 1) / 16 + 1);
        from(q0, P + 4 * (lane >> 3) + row(0), ld, Vm + TC * (lane & 7), nd);
    }
    // f(row, col, float* v): V adjacent columns
    template <class F>
    __device__ __forceinline__ void visit(int h, F&& f) {
        const int lane = threadIdx.x & 31, i = lane >> 3, k = TC * (lane & 7);
#pragma unroll
        for (int q = 0; q < NQ; ++q)
#pragma unroll
            for (int p = 0; p < 2; ++p) {
                float a[TC], b[TC];
#pragma unroll
                for (int e = 0; e < TC; ++e) asm("mov.b64 {%0, %1}, %2;" : "=f"(a[e]), "=f"(b[e]) : "l"(c[q][p][e]));
                const int r = row(q) + 4 * i + 2 * p;
                if (r < h) f(r, k, a);
                if (r + 1 < h) f(r + 1, k, b);
            }
    }
};
template <int M, bool BACK>
struct WarpF64 {
    static constexpr int CW = M == 128 ? 8 : 16, NM = M / 8, NN = CW / 8, V = 2;
    double c[NM][NN][2];
    // where column `col` of depth row d lies: fragment reads (4 depths x 8 columns) hit distinct banks
    static __device__ __forceinline__ int slot(int d, int col) { return CW == 8 ? col ^ (4 * ((d >> 1) & 1)) : col ^ (4 * (d & 3)); }
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int m = 0; m < NM; ++m)
#pragma unroll
            for (int n = 0; n < NN; ++n) c[m][n][0] = c[m][n][1] = 0.0;
    }
    static __device__ __forceinline__ int row(int m, int h) { return 8 * (BACK ? NM - 1 - m : m - NM + (h + 7) / 8); }
    template <int M0>
    __device__ __forceinline__ void tiles(const double* pp, int ld, const double* vp, int nd) {
#pragma unroll 1
        for (int d = 0; d < nd; d += 4) {
            double a[NM], b[NN];
#pragma unroll
            for (int n = 0; n < NN; ++n) b[n] = vp[d * CW + slot(threadIdx.x & 3, 8 * n + ((threadIdx.x >> 2) & 7))];
#pragma unroll
            for (int m = M0; m < NM; ++m) a[m] = pp[d * ld + (BACK ? -8 : 8) * m];
#pragma unroll
            for (int m = M0; m < NM; ++m)
#pragma unroll
                for (int n = 0; n < NN; ++n)
                    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
                        : "+d"(c[m][n][0]), "+d"(c[m][n][1])
                        : "d"(a[m]), "d"(b[n]));
        }
    }
    template <int A = 0, int B = NM>  // m0 in [A, B)
    __device__ __forceinline__ void from(int m0, const double* pp, int ld, const double* vp, int nd) {
        constexpr int H = (A + B) / 2;
        if constexpr (B - A == 1) tiles<A>(pp, ld, vp, nd);
        else if (m0 < H) from<A, H>(m0, pp, ld, vp, nd);
        else from<H, B>(m0, pp, ld, vp, nd);
    }
    __device__ __forceinline__ void run(const double* P, int ld, const double* Vm, int base, int r0, int nd, int h) {
        const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, nm = (h + 7) / 8;
        for (int d = 0; d < nd; d += 8) {
            const int m0 = BACK ? NM - min(nm, (base + d + 7) / 8 + 1) : NM - nm + max(0, (base + d - r0) / 8);
            from(m0, P + (d + t) * ld + g + row(0, h), ld, Vm + (d + t) * CW, min(8, nd - d));
        }
    }
    template <class F>
    __device__ __forceinline__ void visit(int h, F&& f) {
        const int lane = threadIdx.x & 31, k = 2 * (lane & 3);
#pragma unroll
        for (int m = 0; m < NM; ++m) {
            const int r = row(m, h) + (lane >> 2);
            if (r >= 0 && r < h)
#pragma unroll
                for (int n = 0; n < NN; ++n) f(r, k + 8 * n, c[m][n]);
        }
    }
};
template <typename T, int M, bool BACK>
using WarpAcc = std::conditional_t<sizeof(T) == 8, WarpF64<M, BACK>, WarpF32>;

// per: the column groups of this CTA's warps together
template <typename T, int M, bool BACK>
__global__ void __launch_bounds__(NT, 2) k_leaf(SweepArgs<T> a, int32_t per, int32_t panel_max) {
    using A = WarpAcc<T, M, BACK>;
    constexpr int G = vec<T>(), CW = A::CW, VPR = CW / G, S = kLeafStages, VS = LD * CW;
    extern __shared__ __align__(128) unsigned char smraw[];
    T* Ps = reinterpret_cast<T*>(smraw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    T* Vs = Ps + panel_max + warp * (S * VS);
    int32_t* idx = reinterpret_cast<int32_t*>(Ps + panel_max + NT / 32 * (S * VS));  // backward: the depth rows
    __shared__ __align__(8) uint64_t bar;
    allow_dependents();
    const SweepTask t = a.tasks[blockIdx.x];
    const int own = BACK ? t.ns - t.r0 : 0;  // backward: depth rows [0, own) are y_s, then the structure rows
    const int ld = panel_stride<T>(t.h), depth4 = (t.depth + 3) & ~3;
    const int g0 = blockIdx.y * per, g1 = min(g0 + per, a.K / CW);
    if (tid == 0) {
        tc::mbar_init(&bar, 1);
        tc::fence_mbar_init();
        const uint32_t bytes = (uint32_t)(depth4 * ld * (int)sizeof(T));
        tc::mbar_arrive_expect_tx(&bar, bytes);
        tc::bulk_load(Ps, a.panel + (sizeof(T) == 8 ? t.off64 : t.off32), bytes, &bar);
    }
    if constexpr (BACK)
        for (int i = tid; i < t.depth; i += NT) idx[i] = a.rows[t.row0 + t.r0 + i];
    wait_predecessor();
    __syncthreads();
    // a group's leading depth rows with a zero right-hand side: y_s = 0 off the sources' paths (reach was
    // written launches ago); whole steps of four are left out
    auto zeros = [&](int g) { return (BACK && a.reach && !reached(a, t.front, g * CW / kReachCols)) ? own : 0; };
    int pg = g0 + warp, pz = pg < g1 ? zeros(pg) : 0, pd = pz & ~3, ps = 0;  // next chunk to load: group, depth, stage
    auto load_next = [&]() {
        while (pg < g1 && pd >= t.depth) {
            pg += NT / 32;
            if (pg < g1) pz = zeros(pg);
            pd = pz & ~3;
        }
        if (pg < g1) {
            T* V = Vs + ps * VS;
            const int off = pg * CW + G * (lane % VPR);
            const T *ry = (BACK ? a.Y : a.R + (int64_t)t.c0 * a.K) + off, *rx = a.X + off;
#pragma unroll
            for (int f = lane / VPR; f < LD; f += 32 / VPR) {
                const int d = min(pd + f, t.depth - 1);
                const T* src = BACK ? (d < own ? ry : rx) + (int64_t)idx[d] * a.K : ry + (int64_t)d * a.K;
                copy16_async_or_zero(V + f * CW + A::slot(f, G * (lane % VPR)), src, pd + f < t.depth && pd + f >= pz);
            }
            pd += LD;
            ps = ps + 1 == S ? 0 : ps + 1;
        }
        copy_async_commit();
    };
#pragma unroll
    for (int s = 0; s < S - 1; ++s) load_next();
    wait_panel(&bar, 0, a.err);
    A acc;
    int cs = 0;
    for (int g = g0 + warp; g < g1; g += NT / 32) {
        acc.zero();
        for (int base = zeros(g) & ~3; base < t.depth; base += LD) {
            copy_async_wait<S - 2>();
            __syncwarp();
            acc.run(Ps + base * ld, ld, Vs + cs * VS, base, t.r0, min(LD, t.depth - base), t.h);
            __syncwarp();  // the stage is free
            load_next();
            cs = cs + 1 == S ? 0 : cs + 1;
        }
        const int k0 = g * CW;
        if constexpr (BACK) {
            T* x = a.X + (int64_t)(t.c0 + t.r0) * a.K + k0;
            acc.visit(t.h, [&](int r, int c, T* v) { st_n<T, A::V>(x + (int64_t)r * a.K + c, v); });
        } else {
            T* y = a.Y + (int64_t)t.c0 * a.K + k0;
            T* u = a.U + (t.urow - t.ns) * (int64_t)a.K + k0;
            acc.visit(t.h, [&](int r, int c, T* v) {
                const int R = t.r0 + r;
                st_n<T, A::V>((R < t.ns ? y : u) + (int64_t)R * a.K + c, v);
            });
        }
    }
}

// reach[f * tiles + t]: some source of column tile t (kReachCols columns) has front f on its path
// to the root.
__global__ void k_reach(const int32_t* __restrict__ col_front, const int32_t* __restrict__ parent,
                        const int32_t* __restrict__ src, int32_t K, int32_t nlevels, int32_t tiles,
                        uint8_t* __restrict__ reach) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= K) return;
    const int s0 = src[k];
    if (s0 < 0) return;
    const int t = k / kReachCols;
    int s = col_front[s0];
    // the parent chain is strictly increasing and at most nlevels long
    for (int it = 0; s >= 0 && it <= nlevels; ++it) {
        reach[(int64_t)s * tiles + t] = 1;
        s = parent[s];
    }
}

template <typename T, int KT, int M>
constexpr size_t fwd_smem() {
    return (size_t)2 * (panel_stage<T, M>() + DC * ld_rhs<T, KT>()) * sizeof(T);
}
template <typename T, int KT, int M>
size_t bwd_smem(int max_depth) {
    return (size_t)kBwdStages * (panel_stage<T, M>() + DC * ld_rhs<T, KT>()) * sizeof(T) + (size_t)max_depth * sizeof(int32_t);
}
constexpr int64_t kLeafCtas = 2368;               // eight waves of two CTAs per SM
constexpr size_t kSmemMax = 227 * 1024 - 4096;  // static shared memory is kept apart

// overlap: the launch may start while the stream's previous kernel finishes; its reads of that kernel's
// results come after griddepcontrol.wait.
template <typename Kern, typename... Args>
void launch_sweep(Kern kern, dim3 grid, size_t smem, bool overlap, cudaStream_t st, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(NT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = overlap ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kern, args...);
}

template <typename Kern>
cudaError_t allow_smem(Kern kern, size_t bytes) {
    return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}
template <typename T, int KT>
cudaError_t set_smem() {
    cudaError_t e;
    if ((e = allow_smem(k_fwd<T, KT, 128, false>, fwd_smem<T, KT, 128>()))) return e;
    if ((e = allow_smem(k_fwd<T, KT, 64, false>, fwd_smem<T, KT, 64>()))) return e;
    if ((e = allow_smem(k_fwd<T, KT, 64, true>, fwd_smem<T, KT, 64>()))) return e;
    if ((e = allow_smem(k_fwd<T, KT, 32, true>, fwd_smem<T, KT, 32>()))) return e;
    if constexpr (sizeof(T) == 8)
        if ((e = allow_smem(k_leaf<T, 128, false>, kLeafSmem))) return e;
    if ((e = allow_smem(k_leaf<T, 64, true>, kLeafSmem))) return e;
    if ((e = allow_smem(k_bwd<T, KT, 64>, kSmemMax))) return e;
    return allow_smem(k_bwd<T, KT, 32>, kSmemMax);
}

template <typename T, int KT>
void fwd_tile(const SweepArgs<T>& a, int32_t t0, int32_t n, int32_t rows, bool wide, bool overlap, cudaStream_t st) {
    const dim3 grid(n, a.K / KT);
    if (!wide && rows == 128) launch_sweep(k_fwd<T, KT, 128, false>, grid, fwd_smem<T, KT, 128>(), overlap, st, a, t0);
    else if (!wide) launch_sweep(k_fwd<T, KT, 64, false>, grid, fwd_smem<T, KT, 64>(), overlap, st, a, t0);
    else if (rows == 64) launch_sweep(k_fwd<T, KT, 64, true>, grid, fwd_smem<T, KT, 64>(), overlap, st, a, t0);
    else launch_sweep(k_fwd<T, KT, 32, true>, grid, fwd_smem<T, KT, 32>(), overlap, st, a, t0);
}
template <typename T, int KT>
void bwd_tile(const SweepArgs<T>& a, int32_t t0, int32_t n, int32_t rows, int32_t max_depth, cudaStream_t st) {
    const dim3 grid(n, a.K / KT);
    if (rows == 64) launch_sweep(k_bwd<T, KT, 64>, grid, bwd_smem<T, KT, 64>(max_depth), true, st, a, t0);
    else launch_sweep(k_bwd<T, KT, 32>, grid, bwd_smem<T, KT, 32>(max_depth), true, st, a, t0);
}
// The leaf level with its panels resident, where two CTAs fit an SM; false: not taken.
template <typename T, int M, bool BACK>
bool leaf_groups(const SweepArgs<T>& a, int32_t n, int32_t panel, int32_t max_depth, cudaStream_t st) {
    using A = WarpAcc<T, M, BACK>;
    constexpr int W = kLeafWarps;
    static_assert(A::CW == leaf_columns(sizeof(T) == 8, BACK), "the plan's column groups are the kernel's");
    const size_t smem = leaf_smem(panel, A::CW, sizeof(T), BACK ? max_depth : 0);
    const int rounds = a.K / A::CW / W;  // column groups per warp, were a CTA to take them all
    if (!leaves_resident(n, rounds, smem, a.reach != nullptr)) return false;
    const int want = (int)std::max<int64_t>(1, std::min<int64_t>(rounds, (int64_t)n * rounds / kLeafCtas));
    const int ny = (rounds + want - 1) / want, per = W * ((rounds + ny - 1) / ny);
    const int groups = a.K / A::CW;
    launch_sweep(k_leaf<T, M, BACK>, dim3(n, (groups + per - 1) / per), smem, true, st, a, per, panel);
    return true;
}
template <typename T, int KT>
void asm_tile(const SweepArgs<T>& a, int32_t r0, int32_t n, bool overlap, cudaStream_t st) {
    constexpr int RPP = NT / (KT / vec<T>());
    launch_sweep(k_assemble<T, KT>, dim3((n + RPP - 1) / RPP, a.K / KT), 0, overlap, st, a, r0, n);
}

}  // namespace

cudaError_t configure_solve_kernels() {
    cudaError_t e;
    if ((e = set_smem<double, 64>())) return e;
    if ((e = set_smem<float, 64>())) return e;
    return set_smem<float, 128>();
}

int32_t max_front_rows() { return (int32_t)((kSmemMax - bwd_smem<double, 64, 64>(0)) / sizeof(int32_t)); }

template <typename T>
void launch_fwd_level(const SweepArgs<T>& a, int32_t t0, int32_t ntasks, int32_t rows, bool wide, bool overlap,
                      cudaStream_t st) {
    if (ntasks <= 0 || a.K <= 0) return;
    constexpr int W = wide_tile<T>();
    if (W != 64 && a.K % W == 0) fwd_tile<T, W>(a, t0, ntasks, rows, wide, overlap, st);
    else fwd_tile<T, 64>(a, t0, ntasks, rows, wide, overlap, st);
}
template <typename T>
bool launch_leaves(const SweepArgs<T>& a, bool back, int32_t ntasks, int32_t rows, int32_t panel, int32_t max_depth,
                   cudaStream_t st) {
    if (ntasks <= 0 || a.K <= 0 || rows > (back ? 64 : 128) || a.delta_src) return false;
    if (back) return leaf_groups<T, 64, true>(a, ntasks, panel, max_depth, st);
    if constexpr (sizeof(T) == 8) return leaf_groups<T, 128, false>(a, ntasks, panel, max_depth, st);
    return false;
}
template <typename T>
void launch_assemble(const SweepArgs<T>& a, int32_t r0, int32_t nrows, bool overlap, cudaStream_t st) {
    if (nrows <= 0 || a.K <= 0) return;
    constexpr int W = wide_tile<T>();
    if (W != 64 && a.K % W == 0) asm_tile<T, W>(a, r0, nrows, overlap, st);
    else asm_tile<T, 64>(a, r0, nrows, overlap, st);
}
template <typename T>
void launch_bwd_level(const SweepArgs<T>& a, int32_t t0, int32_t ntasks, int32_t rows, int32_t max_depth,
                      cudaStream_t st) {
    if (ntasks <= 0 || a.K <= 0) return;
    constexpr int W = wide_tile<T>();
    if (W != 64 && a.K % W == 0) bwd_tile<T, W>(a, t0, ntasks, rows, max_depth, st);
    else bwd_tile<T, 64>(a, t0, ntasks, rows, max_depth, st);
}

void launch_reach(const int32_t* col_front, const int32_t* parent, int32_t nfronts, int32_t nlevels,
                  const int32_t* src, int32_t K, uint8_t* reach, cudaStream_t st) {
    const int32_t tiles = K / kReachCols;
    cudaMemsetAsync(reach, 0, (size_t)nfronts * tiles, st);
    k_reach<<<(K + 127) / 128, 128, 0, st>>>(col_front, parent, src, K, nlevels, tiles, reach);
}

#define FCW_SWEEPS(T)                                                                                           \
    template void launch_fwd_level<T>(const SweepArgs<T>&, int32_t, int32_t, int32_t, bool, bool, cudaStream_t); \
    template void launch_assemble<T>(const SweepArgs<T>&, int32_t, int32_t, bool, cudaStream_t);                \
    template bool launch_leaves<T>(const SweepArgs<T>&, bool, int32_t, int32_t, int32_t, int32_t, cudaStream_t); \
    template void launch_bwd_level<T>(const SweepArgs<T>&, int32_t, int32_t, int32_t, int32_t, cudaStream_t);
FCW_SWEEPS(double)
FCW_SWEEPS(float)
#undef FCW_SWEEPS

}  // namespace fcw
