// One right-hand side (the single-source drop-in): the heat and Poisson solves of
// one source without a launch per level of the tree of fronts (fronts.cpp).
//
// With A_s = [inv(L_ss); Q_s] of front s (m x ns):
// Forward (leaves -> root), W = b_s - (children's update entries on s's columns):
//   X_s = inv(L_ss) W -> B,   U_s = Q_s W + (children's update entries on s's structure rows)
// Backward (root -> leaves): X_s = A_s^T [y_s; -X_r].
//
// Tasks. A forward task is a group of A_s's rows, a backward task a strip of its columns over all rows
// from the diagonal down (it finishes its columns of X_s, so there is no partial sum to combine). A
// task's part of A_s is stored as it is used, at most 88 KB, and moved into shared memory by one bulk
// copy (cp.async.bulk, completing on an mbarrier) that is requested before the task waits for
// anything: after the dependency resolves, only the small vector gathers and the products from shared
// memory remain. Small fronts are one task; the large ones near the root, which the sweep's time
// depends on, are split so that their rows (columns) are formed in parallel. Solving on merged fronts
// instead of the factorisation's 64-column supernodes takes the chain that a sweep waits along from 32
// to 12 levels at 147k vertices: heat backward 118 to 74 us, Poisson forward 95 to 58, backward 125 to 73.
//
// Scheduling. A persistent CTA takes the next ticket, starts the task's bulk copy
// and loads the indices of the values it depends on, then reads those values: the
// children's update entries (forward) or the ancestors' solution entries (backward).
// Both arrays hold a pending bit pattern (all ones, a NaN that no arithmetic
// produces) when the sweep starts, and each entry is written once, by one 8-byte
// store, so a reader polls each entry until it is no longer pending: the value is the
// signal, with no flags or fences. Tickets follow the level order (leaves first
// forward, reversed backward), so a task only waits for tasks whose tickets were taken
// earlier by CTAs already running: progress does not depend on the grid size or on
// residency. Every wait is bounded (%globaltimer); one that gives up raises
// KERR_TIMEOUT, after which every other wait returns at once, so a sweep always ends.
//
// The heat right-hand side is one column of the identity: only the fronts on the
// source's path to the root have nonzero forward results (the others' are zero in B
// beforehand), so the heat forward runs the forward tasks of the path alone.
#include <algorithm>
#include <vector>

#include "kernels.cuh"
#include "tc.cuh"

namespace fcw {

namespace {

constexpr int NTN = 256;                         // threads per CTA
constexpr int kTaskDoubles = kNarrowTaskDoubles;  // panel data of one task (88 KB: two CTAs per SM)
constexpr int kMaxRows = 192, kSplitTo = 64;      // rows of a whole-front task; of a split front's
constexpr int kMaxCols = 64, kSplitDepth = 256;   // columns of a strip; fronts deeper than this are split
constexpr uint64_t kWaitNs = 1000000000ull;
constexpr int kSmemMax = 227 * 1024 - 16;         // dynamic shared memory of a CTA; 16 bytes are static

constexpr long long kPending = -1;  // bit pattern of an entry not yet written

__device__ __forceinline__ double ld_relaxed(const double* p) {
    double v;
    asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ bool pending(double v) { return __double_as_longlong(v) == kPending; }
__device__ __forceinline__ bool given_up(const int* err) {
    return (*reinterpret_cast<const volatile int*>(err) & KERR_TIMEOUT) != 0;
}

// v[k] = base[idx[k]] for the k in `active` (others 0), entries other CTAs of this launch
// write: each is polled until it is no longer pending. False (KERR_TIMEOUT raised) after
// about kWaitNs, or at once when another wait has already given up.
template <int N>
__device__ bool read_written(const double* base, const int (&idx)[N], unsigned active, double (&v)[N], int* err,
                             unsigned sleep_ns = 64) {
    unsigned pend = 0;
#pragma unroll
    for (int k = 0; k < N; ++k) {
        v[k] = 0.0;
        if ((active >> k) & 1u) {
            v[k] = ld_relaxed(base + idx[k]);
            if (pending(v[k])) pend |= 1u << k;
        }
    }
    if (!pend) return true;
    const uint64_t t0 = tc::global_ns();
    for (;;) {
#pragma unroll
        for (int k = 0; k < N; ++k)
            if ((pend >> k) & 1u) {
                v[k] = ld_relaxed(base + idx[k]);
                if (!pending(v[k])) pend &= ~(1u << k);
            }
        if (!pend) return true;
        if (given_up(err)) return false;
        if (tc::global_ns() - t0 > kWaitNs) {
            atomicOr(err, KERR_TIMEOUT);
            return false;
        }
        __nanosleep(sleep_ns);
    }
}
__device__ __forceinline__ double read_one(const double* p, int* err, unsigned sleep_ns = 64) {
    const int idx[1] = {0};
    double v[1];
    read_written<1>(p, idx, 1u, v, err, sleep_ns);
    return v[0];
}

// A bulk copy that does not land in time raises KERR_TIMEOUT; the second bounded wait
// lets a late copy finish before its buffer is reused.
__device__ __forceinline__ void wait_copies(uint64_t* bar, uint32_t parity, int* err) {
    if (!tc::mbar_wait(bar, parity)) {
        atomicOr(err, KERR_TIMEOUT);
        tc::mbar_wait(bar, parity);
    }
}

// Programmatic dependent launch: the next kernel of the stream may start (its CTAs take
// tickets and start their panel copies, which read nothing this kernel writes) while this
// one finishes; it reads this kernel's results only after griddepcontrol.wait.
__device__ __forceinline__ void allow_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_predecessor() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

__host__ __device__ __forceinline__ int even(int x) { return (x + 1) & ~1; }

// One task's panel from its front's m x ns rows: forward, element (row r, column j) at
// j * even(h) + r; backward, (front row r0 + d, column r0 + c) at c * even(depth) + d.
template <bool FWD>
__global__ void k_pack_narrow(FrontPlan f, const NarrowTask* __restrict__ tasks, const double* __restrict__ rows,
                              double* __restrict__ out) {
    const NarrowTask t = tasks[blockIdx.x];
    const double* in = rows + f.ptr[t.front];
    double* o = out + t.off;
    const int ns = t.ns, ld = even(FWD ? t.h : t.depth), n = (FWD ? t.depth : t.h) * ld;
    for (int e = threadIdx.x; e < n; e += blockDim.x) {
        const int a = e / ld, b = e - a * ld;
        double x = 0.0;
        if (FWD ? b < t.h : b < t.depth)
            x = FWD ? in[(int64_t)(t.r0 + b) * ns + a] : in[(int64_t)(t.r0 + b) * ns + t.r0 + a];
        o[e] = x;
    }
}

// A front row's gather list: the children's update entries that land on it, the first three and
// their fronts loaded before any value is read.
struct RowGather {
    int idx[3];
    int more;
    unsigned active;
};
// DELTA: only the entries of the path child `prev`; the others are never written.
template <bool DELTA>
__device__ __forceinline__ void gather_open(const NarrowArgs& a, int64_t row, int prev, RowGather& g) {
    const int4 r = a.rec[row];
    g.idx[0] = r.x; g.idx[1] = r.y; g.idx[2] = r.z;
    g.more = r.w;
    g.active = 0;
#pragma unroll
    for (int k = 0; k < 3; ++k)
        if (g.idx[k] >= 0 && (!DELTA || a.rec_child[3 * row + k] == prev)) g.active |= 1u << k;
}
// Sum of the row's update entries, in list order, each read once it is written.
template <bool DELTA>
__device__ __forceinline__ double gather_sum(const NarrowArgs& a, const RowGather& g, int prev) {
    double v[3];
    read_written<3>(a.U, g.idx, g.active, v, a.err);
    double sum = 0.0;
#pragma unroll
    for (int k = 0; k < 3; ++k)
        if ((g.active >> k) & 1u) sum += v[k];
    if (g.more >= 0)
        for (int e = 0; e < a.more[g.more]; ++e)
            if (!DELTA || a.more[g.more + 2 + 2 * e] == prev) sum += read_one(a.U + a.more[g.more + 1 + 2 * e], a.err);
    return sum;
}

// Forward tasks. DELTA: the heat solve of the identity column of a.order's source, over
// the tasks of its path (a.order: the source's elimination index, the path's task
// count, then (task, previous front on the path) pairs bottom-up); otherwise every
// task of a.tasks. U is pending on entry.
template <bool DELTA>
__global__ void __launch_bounds__(NTN, 2) k_fwd_tasks(NarrowArgs a) {
    extern __shared__ __align__(16) unsigned char smraw[];
    double* dat = reinterpret_cast<double*>(smraw);  // the task's panel
    double* red = dat + kTaskDoubles;                 // partial row sums
    double* gs = red + NTN;                           // gathered children's entries of the task's rows
    double* W = gs + kMaxRows;                        // the front's right-hand side, max_ns entries
    __shared__ uint64_t bar;
    __shared__ int task, task_prev;
    const int tid = threadIdx.x;
    allow_dependents();
    if (tid == 0) {
        tc::mbar_init(&bar, 1);
        tc::fence_mbar_init();
    }
    __syncthreads();
    const int total = DELTA ? a.order[1] : a.ntasks;
    const int se = DELTA ? a.order[0] : -1;
    uint32_t parity = 0;
    bool inputs_ready = false;  // the previous kernel's results (right-hand side) are visible
    for (;;) {
        if (tid == 0) {
            const int t = atomicAdd(a.ticket, 1);
            const bool stop = t >= total || given_up(a.err);
            task = stop ? -1 : (DELTA ? a.order[2 + 2 * t] : t);
            task_prev = (!stop && DELTA) ? a.order[3 + 2 * t] : -1;
        }
        __syncthreads();
        const int ti = task, prev = task_prev;
        if (ti < 0) break;
        const NarrowTask t = a.tasks[ti];
        const int hp = even(t.h);
        if (tid == 0) {
            const uint32_t bytes = (uint32_t)(t.depth * hp) * 8u;
            tc::mbar_arrive_expect_tx(&bar, bytes);
            tc::bulk_load(dat, a.at + t.off, bytes, &bar);
        }
        if (!inputs_ready) {
            wait_predecessor();
            inputs_ready = true;
        }
        // the right-hand side's columns, then the task's structure rows
        const int u0 = max(t.r0, t.ns), n = t.depth + max(0, t.r0 + t.h - u0);
        for (int i = tid; i < n; i += NTN) {
            const int R = i < t.depth ? i : u0 + i - t.depth;
            RowGather g;
            gather_open<DELTA>(a, t.row0 + R, prev, g);
            const double rhs = i < t.depth ? (DELTA ? (t.c0 + R == se ? 1.0 : 0.0) : a.R[t.c0 + R]) : 0.0;
            const double sum = gather_sum<DELTA>(a, g, prev);
            if (i < t.depth) W[R] = rhs - sum;
            else gs[R - t.r0] = sum;
        }
        __syncthreads();
        wait_copies(&bar, parity, a.err);
        parity ^= 1u;
        // consecutive threads own consecutive rows; the columns are dealt out to 256 / rows parts
        const int sh = max(4, 32 - __clz(t.h - 1)), r = tid & ((1 << sh) - 1), part = tid >> sh, parts = NTN >> sh;
        double acc = 0.0;
        if (r < t.h) {
            const double* p = dat + r;
#pragma unroll 4
            for (int j = part; j < t.depth; j += parts) acc = fma(p[j * hp], W[j], acc);
        }
        red[tid] = acc;
        __syncthreads();
        if (tid < t.h) {
            double x = red[tid];
            for (int q = 1; q < parts; ++q) x += red[(q << sh) + tid];
            const int R = t.r0 + tid;
            if (R < t.ns) a.B[t.c0 + R] = x;
            else a.U[t.urow + R - t.ns] = x + gs[tid];
        }
        __syncthreads();  // the panel, W and gs are free for the next task
    }
}

// Backward tasks: X (pending on entry) = the solution, from the forward result B.
__global__ void __launch_bounds__(NTN, 2) k_bwd_tasks(NarrowArgs a) {
    extern __shared__ __align__(16) unsigned char smraw[];
    double* dat = reinterpret_cast<double*>(smraw);  // the task's column strip
    double* v = dat + a.strip;                        // [y_s; -X_r] from row r0 down
    __shared__ uint64_t bar;
    __shared__ int task;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    allow_dependents();
    if (tid == 0) {
        tc::mbar_init(&bar, 1);
        tc::fence_mbar_init();
    }
    __syncthreads();
    uint32_t parity = 0;
    bool inputs_ready = false;  // the previous kernel's results (forward result) are visible
    for (;;) {
        if (tid == 0) {
            const int t = atomicAdd(a.ticket, 1);
            task = (t >= a.ntasks || given_up(a.err)) ? -1 : t;
        }
        __syncthreads();
        const int ti = task;
        if (ti < 0) break;
        const NarrowTask t = a.tasks[ti];
        const int mp = even(t.depth), own = t.ns - t.r0;
        const int32_t* rows = a.rows + t.row0 + t.r0;
        if (tid == 0) {
            const uint32_t bytes = (uint32_t)(t.h * mp) * 8u;
            tc::mbar_arrive_expect_tx(&bar, bytes);
            tc::bulk_load(dat, a.at + t.off, bytes, &bar);
        }
        if (!inputs_ready) {
            wait_predecessor();
            inputs_ready = true;
        }
        // The parent's entries are written last, just before this task can run: they are polled with a
        // short back-off, the older ancestors' with a long one, so few requests reach the L2 slices
        // that hold the entries being produced. (The parent's columns come first among the structure
        // rows.)
        for (int d = tid; d < t.depth; d += NTN) {
            const int row = rows[d];
            v[d] = d < own ? __ldcg(a.B + row) : -read_one(a.X + row, a.err, row < t.pend ? 32 : 256);
        }
        __syncthreads();
        wait_copies(&bar, parity, a.err);
        parity ^= 1u;
        // warp w owns the strip's columns w + 8 jj; lanes walk the rows
        double acc[kMaxCols / 8];
#pragma unroll
        for (int jj = 0; jj < kMaxCols / 8; ++jj) acc[jj] = 0.0;
        for (int d = lane; d < t.depth; d += 32) {
            const double xv = v[d];
#pragma unroll
            for (int jj = 0; jj < kMaxCols / 8; ++jj) {
                const int jl = warp + 8 * jj;
                if (jl < t.h) acc[jj] = fma(dat[jl * mp + d], xv, acc[jj]);
            }
        }
#pragma unroll
        for (int jj = 0; jj < kMaxCols / 8; ++jj) {
            double xs = acc[jj];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) xs += __shfl_xor_sync(0xffffffffu, xs, o);
            const int jl = warp + 8 * jj;
            if (lane == 0 && jl < t.h) a.X[t.c0 + t.r0 + jl] = xs;
        }
        __syncthreads();  // v and the strip are free for the next task
    }
}

// The source's field in the caller's vertex order, shifted so the source is at zero.
__global__ void k_field_out_one(int32_t n, const double* __restrict__ Y, const int32_t* __restrict__ src_elim,
                                const int32_t* __restrict__ iperm, double* __restrict__ out) {
    const int se = *src_elim;
    if (se < 0) return;
    const double y0 = Y[se];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) out[i] = Y[iperm[i]] - y0;
}

size_t fwd_bytes(int max_ns) { return (size_t)(kTaskDoubles + NTN + kMaxRows + even(max_ns)) * sizeof(double); }
int strip_doubles(int max_m) { return std::max(kTaskDoubles, even(max_m)); }  // a strip holds one column
size_t bwd_bytes(int max_m) { return (size_t)(strip_doubles(max_m) + even(max_m)) * sizeof(double); }

}  // namespace

void narrow_tasks(const Fronts& f, std::vector<NarrowTask>& fwd, std::vector<int32_t>& fwd_first,
                  std::vector<int32_t>& nfwd, std::vector<NarrowTask>& bwd, int64_t* fwd_doubles,
                  int64_t* bwd_doubles) {
    fwd.clear();
    bwd.clear();
    fwd_first.assign((size_t)f.nf, 0);
    nfwd.assign((size_t)f.nf, 0);
    int64_t off = 0;
    auto base = [&](int32_t s) {
        NarrowTask t{};
        t.front = s;
        t.c0 = f.c0[s];
        t.ns = f.c0[s + 1] - f.c0[s];
        t.row0 = f.row0[s];
        t.urow = f.uoff[s];
        t.pend = f.parent[s] >= 0 ? f.c0[f.parent[s] + 1] : 0;
        return t;
    };
    for (int32_t q = 0; q < f.nf; ++q) {  // level order: leaves first
        const int32_t s = f.level_nodes[q], m = f.m[s];
        NarrowTask t = base(s);
        const int32_t fit = std::min(kMaxRows, kTaskDoubles / t.ns & ~1);
        const int32_t most = m <= fit ? m : std::max(1, std::min(kSplitTo, fit));
        const int32_t n = (m + most - 1) / most, per = (m + n - 1) / n;
        fwd_first[s] = (int32_t)fwd.size();
        for (t.r0 = 0; t.r0 < m; t.r0 += per) {
            t.h = std::min(per, m - t.r0);
            t.depth = std::min(t.ns, t.r0 + t.h);
            t.off = off;
            off += (int64_t)t.depth * even(t.h);
            fwd.push_back(t);
        }
        nfwd[s] = (int32_t)fwd.size() - fwd_first[s];
    }
    *fwd_doubles = off;
    off = 0;
    for (int32_t q = f.nf - 1; q >= 0; --q) {  // reversed level order: root first
        const int32_t s = f.level_nodes[q], m = f.m[s];
        NarrowTask t = base(s);
        const int32_t fit = std::max(1, kTaskDoubles / even(m)), most = std::min(m > kSplitDepth ? 8 : kMaxCols, fit);
        const int32_t n = (t.ns + most - 1) / most, per = (t.ns + n - 1) / n;
        for (t.r0 = 0; t.r0 < t.ns; t.r0 += per) {
            t.h = std::min(per, t.ns - t.r0);
            t.depth = m - t.r0;
            t.off = off;
            off += (int64_t)t.h * even(t.depth);
            bwd.push_back(t);
        }
    }
    *bwd_doubles = off;
}

void launch_pack_narrow(const FrontPlan& f, bool fwd, const NarrowTask* tasks, int32_t ntasks, const double* rows,
                        double* out, cudaStream_t st) {
    if (ntasks <= 0) return;
    if (fwd) k_pack_narrow<true><<<ntasks, 256, 0, st>>>(f, tasks, rows, out);
    else k_pack_narrow<false><<<ntasks, 256, 0, st>>>(f, tasks, rows, out);
}

cudaError_t configure_narrow_kernels(int max_ns, int max_m, int num_sms, NarrowLaunch* L) {
    L->fwd_smem = fwd_bytes(max_ns);
    L->bwd_smem = bwd_bytes(max_m);
    L->strip = strip_doubles(max_m);
    if (L->fwd_smem > kSmemMax || L->bwd_smem > kSmemMax) return cudaErrorInvalidValue;
    // the same allowance for every engine: it belongs to the kernel, and engines of other sizes launch it too
    cudaError_t e = cudaFuncSetAttribute(k_fwd_tasks<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_fwd_tasks<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_bwd_tasks, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax);
    int per_sm = 0;
    if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_fwd_tasks<false>, NTN, L->fwd_smem);
    L->grid_fwd = std::max(1, per_sm) * num_sms;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_bwd_tasks, NTN, L->bwd_smem);
    L->grid_bwd = std::max(1, per_sm) * num_sms;
    return e;
}

namespace {
// overlap: launched as a programmatic dependent of the stream's previous kernel
template <typename Kern>
void launch_sweep(Kern kern, int grid, size_t smem, bool overlap, const NarrowArgs& a, cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(NTN);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = overlap ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kern, a);
}
}  // namespace

void launch_fwd_narrow(const NarrowArgs& a, bool delta, bool overlap, const NarrowLaunch& L, cudaStream_t st) {
    if (delta) launch_sweep(k_fwd_tasks<true>, L.grid_fwd, L.fwd_smem, overlap, a, st);
    else launch_sweep(k_fwd_tasks<false>, L.grid_fwd, L.fwd_smem, overlap, a, st);
}
void launch_bwd_narrow(const NarrowArgs& a, bool overlap, const NarrowLaunch& L, cudaStream_t st) {
    launch_sweep(k_bwd_tasks, L.grid_bwd, L.bwd_smem, overlap, a, st);
}
void launch_field_out_one(int32_t n, const double* Y, const int32_t* src_elim, const int32_t* iperm, double* out,
                          int num_sms, cudaStream_t st) {
    k_field_out_one<<<num_sms * 2, 256, 0, st>>>(n, Y, src_elim, iperm, out);
}

}  // namespace fcw
