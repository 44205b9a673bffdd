// Engine lifecycle, factorisation sequence, the per-block pipeline and the C ABI.
//
// One engine = one cortical submesh on one GPU. Creation prepares the mesh on
// the host, runs the symbolic analysis, uploads the structure and factors the
// heat operator M + tL and the Poisson operator L + shift*M in FP64 on the
// device (plus, for the mixed form, the Poisson operator grounded at the last
// eliminated vertex of each connected component, rounded to FP32). A block of K
// sources then runs:
//   reach -> heat forward (delta RHS, pruned) -> heat backward -> divergence
//   -> Poisson forward/backward -> shift + transpose -> vertex stats -> geometry
// entirely on one stream.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>
#include <future>
#include <mutex>
#include <string>
#include <system_error>
#include <type_traits>
#include <utility>
#include <vector>

#include "fcw_b200.h"
#include "fcw_internal.h"
#include "kernels.cuh"
#include "staging.h"

namespace {

thread_local std::string g_err;

int fail(int code, const std::string& msg) {
    g_err = msg;
    return code;
}

#define FCW_CUDA(call)                                                                        \
    do {                                                                                      \
        cudaError_t e_ = (call);                                                              \
        if (e_ != cudaSuccess) return fail(FCW_E_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
    } while (0)

#define FCW_TRY(expr)            \
    do {                         \
        int rc_ = (expr);        \
        if (rc_ != FCW_OK) return rc_; \
    } while (0)

// Triangle-inequality margin of the robust operators' mollified edge lengths, relative to
// the mean edge length (the default of Sharp & Crane's intrinsic mollification).
constexpr double kMollifyFactor = 1e-6;

double now_ms() {
    using namespace std::chrono;
    return duration<double, std::milli>(steady_clock::now().time_since_epoch()).count();
}

__global__ void k_map_sources(int64_t n, const int32_t* __restrict__ sources, const int32_t* __restrict__ iperm,
                              int32_t nv, int32_t K, int32_t* __restrict__ out, int* __restrict__ err) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= K) return;
    int v = -1;
    if (k < n) {
        const int s = sources[k];
        if (s >= 0 && s < nv) v = iperm[s];
        else atomicOr(err, fcw::KERR_ARGS);
    }
    out[k] = v;
}

// The block's inputs into its workspace descriptor (ahead of the block's launch chain).
__global__ void k_set_block(fcw::BlockDesc* d, const int32_t* sources, int64_t n, double* out) {
    d->sources = sources;
    d->n = n;
    d->out = out;
}

// A block's sources (the descriptor's, or n of `raw`) in elimination order: src[c] = column c's
// source, dst[c] = its place in the caller's list; -1 for padding and invalid sources, which come
// last. The heat forward sweep solves, per 64-column tile, the fronts on its sources' paths to the
// root: neighbours in this order share theirs. One CTA, a bitonic sort of (elimination index,
// place) keys in shared memory, N = K rounded up to a power of two. 1024 sources in random order
// at 147k vertices: heat forward 0.86 to 0.45 ms, heat backward 1.37 to 1.32 ms.
constexpr int kSortThreads = 1024;
constexpr int kMaxSort = 4096;  // block_k's largest
// raw may be src: every source is read before the first barrier, src is written after the last.
__global__ void __launch_bounds__(kSortThreads) k_sort_sources(const fcw::BlockDesc* d, const int32_t* raw, int64_t n,
                                                               const int32_t* iperm, int32_t nv, int32_t K, int32_t N,
                                                               int32_t* src, int32_t* dst, int* err) {
    extern __shared__ unsigned long long key[];
    const int32_t* from = d ? d->sources : raw;
    const int64_t count = d ? d->n : n;
    for (int k = threadIdx.x; k < N; k += blockDim.x) {
        unsigned long long x = ~0ull;
        if (k < count) {
            const int s = from[k];
            if (s >= 0 && s < nv) x = ((unsigned long long)iperm[s] << 32) | (unsigned)k;
            else atomicOr(err, fcw::KERR_ARGS);
        }
        key[k] = x;
    }
    for (int size = 2; size <= N; size <<= 1)
        for (int step = size >> 1; step > 0; step >>= 1) {
            __syncthreads();
            for (int i = threadIdx.x; i < N / 2; i += blockDim.x) {
                const int a = 2 * i - (i & (step - 1)), b = a + step;
                const bool up = (a & size) == 0;
                const unsigned long long x = key[a], y = key[b];
                if ((x > y) == up) {
                    key[a] = y;
                    key[b] = x;
                }
            }
        }
    __syncthreads();
    for (int k = threadIdx.x; k < K; k += blockDim.x) {
        const unsigned long long x = key[k];
        src[k] = x == ~0ull ? -1 : (int32_t)(x >> 32);
        dst[k] = x == ~0ull ? -1 : (int32_t)(x & 0xffffffffu);
    }
}

// Rows [0, k) of dT (K x n, one field per source, elimination order) -> out (k x n, caller order;
// row r is the caller's source dst[r]).
template <typename T>
__global__ void k_fields_out(int32_t n, int32_t k, const T* __restrict__ dT, const int32_t* __restrict__ iperm,
                             const int32_t* __restrict__ dst, double* __restrict__ out) {
    const int64_t total = (int64_t)k * n;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
        const int r = (int)(e / n), i = (int)(e - (int64_t)r * n);
        const int o = dst[r];
        if (o >= 0) out[(int64_t)o * n + i] = (double)dT[(int64_t)r * n + iperm[i]];
    }
}

// d (k rows, caller vertex order) -> Y (n x K vertex-major, elimination order); columns >= k are zero.
__global__ void k_fields_in(int32_t n, int32_t k, int32_t K, const double* __restrict__ d,
                            const int32_t* __restrict__ iperm, double* __restrict__ Y) {
    const int64_t total = (int64_t)K * n;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
        const int r = (int)(e / n), i = (int)(e - (int64_t)r * n);
        Y[(int64_t)iperm[i] * K + r] = r < k ? d[(int64_t)r * n + i] : 0.0;
    }
}

}  // namespace

// Page-locked words, one per engine, from a page the process allocates once: an allocation per engine took
// 1.7 to 3.2 ms of an 8 ms build at 2.3k vertices, and freeing it may wait for other engines' work. Engines
// beyond the page's words copy to a pageable one (10 us more per call).
class LockedWords {
public:
    int* take() {
        std::lock_guard<std::mutex> hold(mutex_);
        if (!asked_) {
            asked_ = true;
            int* page = nullptr;
            if (cudaHostAlloc(reinterpret_cast<void**>(&page), kWords * sizeof(int), cudaHostAllocPortable) == cudaSuccess)
                for (int i = kWords - 1; i >= 0; --i) free_.push_back(page + i);
            else cudaGetLastError();
        }
        if (free_.empty()) return nullptr;
        int* w = free_.back();
        free_.pop_back();
        return w;
    }
    void give(int* w) {
        std::lock_guard<std::mutex> hold(mutex_);
        free_.push_back(w);
    }

private:
    static constexpr int kWords = 1024;
    std::mutex mutex_;
    std::vector<int*> free_;
    bool asked_ = false;
};
LockedWords& words() {
    static LockedWords* w = new LockedWords;  // kept for engines destroyed while the process exits
    return *w;
}

struct Workspace {
    int32_t K = 0;
    double* Bh = nullptr;
    double* Bp64 = nullptr;
    float* Bp32 = nullptr;
    double* Y = nullptr;        // Poisson solution (n x K doubles, or floats for the mixed form)
    double* dT64 = nullptr;
    float* dT32 = nullptr;
    int32_t* src = nullptr;
    int32_t* dst = nullptr;     // each column's place in the caller's list
    uint8_t* reach = nullptr;
    int4* band = nullptr;
    int32_t* longf = nullptr;
    double* out = nullptr;
    int32_t out_stride = 0;
    double* U = nullptr;        // forward update rows, (sum nr) x K doubles (reused as floats)
    double* W = nullptr;        // assembled right-hand sides of the wide fronts (reused as floats)
    double* partials = nullptr; // per (vertex tile, source) health/MSD partial sums
    double* csum = nullptr;     // per (vertex tile, source) component sums, then the levels (several components)
    int32_t* near_list = nullptr;
    int32_t* near_count = nullptr;
    cudaStream_t stream = nullptr;  // this workspace's stream in the pipelined device path
    cudaEvent_t done = nullptr;
    std::vector<std::pair<int, cudaEvent_t>> marks;  // stage timeline on this workspace
    double* part = nullptr;     // tensor-core sweeps: backward split-K partial sums
    int* counters = nullptr;    // and arrival tickets, zero at rest
    fcw::BlockDesc* desc = nullptr;     // the current block's inputs (device)
    // the block's launch chain captured as CUDA graphs, one per set of arguments (a few)
    struct Graph {
        std::vector<double> key;
        cudaGraphExec_t exec = nullptr;
        int64_t launches = 0;           // kernels in the graph
    };
    std::vector<Graph> graphs;
    void drop_graph() {
        for (auto& g : graphs)
            if (g.exec) cudaGraphExecDestroy(g.exec);
        graphs.clear();
    }
};

// The single-source drop-in (fcw_compute_distance): the narrow panel layouts of the two FP64
// factors, the task lists, its own vectors and sweep state, and its launch chain; built on
// its first call.
struct NarrowState {
    bool ready = false;
    fcw::NarrowLaunch L;
    double *at_h = nullptr, *at_p = nullptr;    // forward layouts of the heat and Poisson factors
    double *atb_h = nullptr, *atb_p = nullptr;  // backward layouts
    fcw::NarrowTask *ftasks = nullptr, *btasks = nullptr;
    int32_t n_ftasks = 0, n_btasks = 0;
    double *u = nullptr, *div = nullptr, *y = nullptr, *out = nullptr;
    double* pend = nullptr;       // entries a sweep's readers poll: heat and Poisson update entries, heat
                                  // and Poisson solutions (set pending at the start of each call)
    int* sync = nullptr;          // the four sweeps' ticket counters
    // the heat forward's work list, built on the host per call: the source's elimination
    // index, the path's task count, then (task, previous front on the path) pairs
    int32_t* order = nullptr;
    int32_t* horder = nullptr;    // pinned host staging of the list
    std::vector<int32_t> fwd_first, nfwd_h;  // per front: first forward task, count
    cudaGraphExec_t exec = nullptr;
    int64_t launches = 0;         // kernels per call
};

struct fcw_engine {
    fcw_params prm{};
    int device = 0;
    fcw::MeshPrep mesh;
    fcw::Symbolic sym;
    double t_coef = 0.0, t = 0.0;
    // the grounded (mixed-form) Poisson operator: one ground vertex per connected component of
    // the submesh, its last eliminated vertex; flags in the caller's order (host) and in
    // elimination order (device)
    std::vector<uint8_t> grounded_old;
    uint8_t* grounded_d = nullptr;
    // with several components: each vertex's component and lumped mass (elimination order) and
    // each component's total mass, for the mixed form's level on the source's component
    int32_t ncomp = 1;
    std::vector<int32_t> comp_h;
    std::vector<double> cmass_h, carea_h;
    fcw::ComponentLevel clevel;
    cudaStream_t stream = nullptr;
    std::vector<std::pair<void*, size_t>> allocs;  // device allocations and their sizes
    int64_t bytes = 0;
    fcw::DevPlan plan;
    std::vector<int32_t> level_tiles;
    // the sweeps' fronts and task lists (fronts.h) and their panels: forward and backward, of the
    // heat, Poisson and (FP32) grounded Poisson factors
    fcw::Fronts fr;
    fcw::FrontPlan frp;
    std::vector<int32_t> bwd_depth;  // per level: the most front rows a backward task multiplies
    fcw::SweepTask *fwd_tasks = nullptr, *bwd_tasks = nullptr;
    fcw::GatherRec* rec_d = nullptr;
    int32_t *rec_child_d = nullptr, *more_d = nullptr, *front_rows_d = nullptr, *asm_rows_d = nullptr;
    double *pan_hf = nullptr, *pan_hb = nullptr, *pan_pf = nullptr, *pan_pb = nullptr;
    float *pan_gf = nullptr, *pan_gb = nullptr;
    // tensor-core sweeps: per level of supernodes, task ranges of the backward task list
    std::vector<int32_t> tc_bwd_ptr;
    int2* tc_bwd_tasks = nullptr;
    int64_t* uoff_d = nullptr;
    int64_t* poff_d = nullptr;
    int32_t* nsplit_d = nullptr;
    int32_t *gm_ptr_d = nullptr, *gm_src_d = nullptr;
    int64_t n_urows = 0, n_parts = 0;
    double *val_h = nullptr, *inv_h = nullptr, *val_p = nullptr, *inv_p = nullptr;
    fcw::CsrOperator lg;  // the grounded Poisson operator in FP64, elimination order (refinement residuals)
    // tensor-core FP32 sweeps: core arrays of the grounded factor and the forward task list
    float *core_hi = nullptr, *core_lo = nullptr, *coreT_hi = nullptr, *coreT_lo = nullptr;
    int64_t* core_ptr_d = nullptr;
    int2* tc_fwd_tasks = nullptr;
    std::vector<int32_t> tc_fwd_ptr;
    fcw::FaceData fd;
    int32_t* iperm_d = nullptr;
    int32_t* perm_d = nullptr;
    double *coords_d = nullptr, *varea_d = nullptr, *farea_d = nullptr, *g11_d = nullptr, *g12_d = nullptr,
           *g22_d = nullptr;
    int32_t* boundary_d = nullptr;
    int32_t* fan_walk_d = nullptr;    // per fan step: neighbour, face
    long long* farea_fx_d = nullptr;  // lean face areas in fixed point
    double area_unscale = 0.0;
    int* err_d = nullptr;
    int* err_h = nullptr;  // its copy's page-locked word (words); null: a pageable one
    std::vector<Workspace> pool;  // blocks in flight: workspace i runs on pool[i].stream
    size_t cur_ws = 0;
    Workspace& cw() { return pool[cur_ws]; }
    cudaEvent_t ev_in = nullptr;  // the caller's stream at the start of a pipelined call
    int32_t* hsrc_d = nullptr;    // staging for the host-buffer metrics API
    double* hout_d = nullptr;
    int64_t hcap_src = 0, hcap_out = 0;
    float *hsr_d = nullptr, *hsa_d = nullptr;  // staging for the host-buffer sample assembly
    int32_t* hcnt_d = nullptr;
    int64_t hcap_sr = 0, hcap_sa = 0, hcap_cnt = 0;
    unsigned char *hmap_d = nullptr, *hmap_h = nullptr;  // staging for the wiring maps: device, page-locked host
    int64_t hcap_map_d = 0, hcap_map_h = 0;
    double* hdist_d = nullptr;  // staging for the host-buffer distances API (caller order)
    int64_t hcap_dist = 0;
    double analyze_ms = 0.0, factor_ms = 0.0;
    double chord_slack = 0.0; // MetricArgs::chord_slack
    double lean_total = 0.0;  // sum of the lean face areas (the prefix total of a finite field)
    // stage timeline (CUDA events on the working stream), off unless enabled
    bool prof_on = false;
    bool graphs_on = true;  // replay each workspace's captured launch chain
    std::vector<cudaEvent_t> event_pool;
    double stage_ms[FCW_N_STAGES] = {0};
    int64_t launches = 0;
    int32_t num_sms = 148;  // the device's multiprocessors (grid sizes of grid-stride kernels)
    int64_t n_flips = 0;    // intrinsic edge flips of the robust operators
    NarrowState nar;

    // Device memory is stream-ordered (the device's default pool): freeing it
    // waits for this engine's streams only, never for other engines' work, so
    // engines can come and go while others run (the serving loop relies on it).
    template <typename T>
    int dalloc(T** p, size_t count) {
        *p = nullptr;
        if (count == 0) count = 1;
        void* q = nullptr;
        cudaError_t e = cudaMallocAsync(&q, count * sizeof(T), stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(stream);  // usable from any stream from here on
        if (e != cudaSuccess) {
            cudaGetLastError();
            return fail(FCW_E_NOMEM, "allocation of " + std::to_string(count * sizeof(T)) + " bytes failed: " +
                                         cudaGetErrorString(e));
        }
        allocs.emplace_back(q, count * sizeof(T));
        bytes += (int64_t)(count * sizeof(T));
        *p = static_cast<T*>(q);
        return FCW_OK;
    }
    // Waits for all of this engine's streams (the work that may still read its buffers).
    void sync_streams() {
        if (stream) cudaStreamSynchronize(stream);
        for (auto& w : pool)
            if (w.stream) cudaStreamSynchronize(w.stream);
    }
    template <typename T>
    int upload(T** p, const std::vector<T>& h) {
        FCW_TRY(dalloc(p, h.size()));
        if (!h.empty()) FCW_CUDA(cudaMemcpy(*p, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice));
        return FCW_OK;
    }
    void release(void* p) {
        for (size_t i = 0; i < allocs.size(); ++i)
            if (allocs[i].first == p) {
                sync_streams();
                cudaFreeAsync(p, stream);
                bytes -= (int64_t)allocs[i].second;
                allocs.erase(allocs.begin() + (long)i);
                return;
            }
    }
    // Staging that grows: on the device, and page-locked on the host (its readers have been waited for).
    template <typename T>
    int grow(T*& p, int64_t& cap, int64_t need) {
        return fcw::grow_staging(p, cap, need, [&](T** q, int64_t n) { return dalloc(q, (size_t)n); },
                                 [&](T* q) { release(q); });
    }
    int grow_host(unsigned char*& p, int64_t& cap, int64_t need) {
        return fcw::grow_staging(
            p, cap, need,
            [](unsigned char** q, int64_t n) -> int {
                if (cudaHostAlloc(reinterpret_cast<void**>(q), (size_t)n, cudaHostAllocDefault) == cudaSuccess)
                    return FCW_OK;
                cudaGetLastError();
                return fail(FCW_E_NOMEM, "page-locked allocation of " + std::to_string(n) + " bytes failed");
            },
            [](unsigned char* q) { cudaFreeHost(q); });
    }
    ~fcw_engine() {
        sync_streams();
        for (auto& a : allocs) cudaFreeAsync(a.first, stream);
        if (stream) cudaStreamSynchronize(stream);
        for (auto& w : pool) {
            w.drop_graph();
            for (auto& m : w.marks) cudaEventDestroy(m.second);
            if (w.done) cudaEventDestroy(w.done);
            if (w.stream) cudaStreamDestroy(w.stream);
        }
        if (ev_in) cudaEventDestroy(ev_in);
        if (nar.exec) cudaGraphExecDestroy(nar.exec);
        if (nar.horder) cudaFreeHost(nar.horder);
        if (hmap_h) cudaFreeHost(hmap_h);
        if (err_h) words().give(err_h);
        for (cudaEvent_t ev : event_pool) cudaEventDestroy(ev);
        if (stream) cudaStreamDestroy(stream);
    }
};

namespace {

// Waits for e->stream and reports the errors the kernels raised.
int check_kernel_errors(fcw_engine* e, const char* where) {
    int word = 0;
    int* to = e->err_h ? e->err_h : &word;
    FCW_CUDA(cudaMemcpyAsync(to, e->err_d, sizeof(int), cudaMemcpyDeviceToHost, e->stream));
    FCW_CUDA(cudaStreamSynchronize(e->stream));
    const int h = *to;
    if (h) {
        FCW_CUDA(cudaMemsetAsync(e->err_d, 0, sizeof(int), e->stream));
        std::string what;
        if (h & fcw::KERR_NOT_SPD) what += " non-positive pivot (operator not SPD);";
        if (h & fcw::KERR_HIST_OVERFLOW) what += " too many distance bins for one source;";
        if (h & fcw::KERR_SCRATCH) what += " per-source face list overflow;";
        if (h & fcw::KERR_ARGS) what += " invalid source index or launch arguments;";
        if (h & fcw::KERR_TIMEOUT) what += " a bounded device wait expired;";
        const int code = (h & fcw::KERR_ARGS) ? FCW_E_INVALID : (h & fcw::KERR_TIMEOUT) ? FCW_E_TIMEOUT : FCW_E_NUMERIC;
        return fail(code, std::string(where) + ":" + what);
    }
    return FCW_OK;
}

// Record a stage boundary: the stage `stage` starts here (-1 = end of a block).
void mark(fcw_engine* e, cudaStream_t st, int stage) {
    if (!e->prof_on) return;
    cudaEvent_t ev;
    if (!e->event_pool.empty()) {
        ev = e->event_pool.back();
        e->event_pool.pop_back();
    } else if (cudaEventCreate(&ev) != cudaSuccess) {
        cudaGetLastError();
        return;
    }
    cudaEventRecord(ev, st);
    e->cw().marks.push_back({stage, ev});
}

int collect_marks(fcw_engine* e) {
    for (auto& w : e->pool) {
        auto& marks = w.marks;
        if (marks.empty()) continue;
        FCW_CUDA(cudaEventSynchronize(marks.back().second));
        for (size_t j = 0; j + 1 < marks.size(); ++j) {
            const int stg = marks[j].first;
            if (stg < 0 || stg >= FCW_N_STAGES) continue;
            float ms = 0.0f;
            FCW_CUDA(cudaEventElapsedTime(&ms, marks[j].second, marks[j + 1].second));
            e->stage_ms[stg] += ms;
        }
        for (auto& m : marks) e->event_pool.push_back(m.second);
        marks.clear();
    }
    return FCW_OK;
}

int validate_params(const fcw_params* p) {
    if (!p) return fail(FCW_E_INVALID, "params is NULL");
    if (!std::isfinite(p->diffusion_length_mm) || p->diffusion_length_mm < 0.5)
        return fail(FCW_E_INVALID, "diffusion_length_mm must be finite and at least 0.5 mm.");
    if (!std::isfinite(p->poisson_shift) || p->poisson_shift < 0.0) return fail(FCW_E_INVALID, "invalid poisson_shift");
    if (p->block_k < 64 || p->block_k % 64 != 0 || p->block_k > 4096)
        return fail(FCW_E_INVALID, "block_k must be a multiple of 64 in [64, 4096]");
    if (p->leaf_size < 1 || p->max_width < 1 || p->max_width > fcw::kMaxWidth)
        return fail(FCW_E_INVALID, "max_width must be in [1, 64] and leaf_size >= 1");
    if (p->relax < 1 || p->relax > p->max_width) return fail(FCW_E_INVALID, "relax must be in [1, max_width]");
    if (p->pipeline_depth < 1 || p->pipeline_depth > 8) return fail(FCW_E_INVALID, "pipeline_depth must be in [1, 8]");
    if (p->tc_sweeps != 0 && p->tc_sweeps != 1) return fail(FCW_E_INVALID, "tc_sweeps must be 0 or 1");
    if (p->robust != 0 && p->robust != 1) return fail(FCW_E_INVALID, "robust must be 0 or 1");
    if (p->refine < 0 || p->refine > 4) return fail(FCW_E_INVALID, "refine must be in [0, 4]");
    return FCW_OK;
}

// Connected components of the submesh (union-find over its faces; core_analysis.py:1349-1381
// reports the same ones): comp[v] for each vertex v, numbered in order of first appearance in
// the elimination order perm. Returns their count.
int32_t mesh_components(const fcw::MeshPrep& m, const std::vector<int32_t>& perm, std::vector<int32_t>& comp) {
    const int64_t n = m.nv;
    std::vector<int32_t> up(n);
    for (int64_t i = 0; i < n; ++i) up[i] = (int32_t)i;
    auto find = [&](int32_t x) {
        while (up[x] != x) x = up[x] = up[up[x]];
        return x;
    };
    for (int64_t f = 0; f < m.nf; ++f)
        for (int c = 1; c < 3; ++c) {
            const int32_t a = find(m.F[3 * f]), b = find(m.F[3 * f + c]);
            if (a != b) up[std::max(a, b)] = std::min(a, b);
        }
    std::vector<int32_t> label(n, -1);
    comp.assign(n, -1);
    int32_t count = 0;
    for (int64_t i = 0; i < n; ++i) {
        const int32_t v = perm[i], r = find(v);
        if (label[r] < 0) label[r] = count++;
        comp[v] = label[r];
    }
    return count;
}

// Values of A's lower entries in the symbolic analysis' order.
enum class Op { Heat, Poisson, Grounded };
std::vector<double> operator_values(const fcw_engine* e, Op op) {
    const auto& S = e->sym;
    const auto& m = e->mesh;
    std::vector<double> v(S.nnz_lower_a);
    for (int64_t q = 0; q < S.nnz_lower_a; ++q) {
        const int64_t k = S.a_src[q];
        const int32_t col = S.a_col[q], row = m.Li[k];
        const bool diag = row == col;
        const double L = m.Lx[k];
        switch (op) {
            case Op::Heat:  // M + t L (fastcw_lean.py:498)
                v[q] = diag ? m.mass[col] + e->t * L : e->t * L;
                break;
            case Op::Poisson:  // L + shift M (fastcw_lean.py:500)
                v[q] = diag ? L + e->prm.poisson_shift * m.mass[col] : L;
                break;
            case Op::Grounded:  // L with the ground vertices' rows and columns replaced by the identity
                v[q] = (e->grounded_old[row] || e->grounded_old[col]) ? (diag ? 1.0 : 0.0) : L;
                break;
        }
    }
    return v;
}

}  // namespace

// ---------------------------------------------------------------------------
// engine construction
// ---------------------------------------------------------------------------
namespace {

// The mesh in elimination order, as the kernels read it.
struct MeshTables {
    std::vector<double> coords, varea;
    std::vector<int32_t> fv, bnd, inc_ptr;
    std::vector<long long> farea_fx;
    double area_unscale = 0.0, lean_total = 0.0, largest = 0.0;  // largest: coordinate magnitude
    std::vector<int32_t> fan_ptr, fan_walk;
    std::vector<fcw::FanStep> fan_steps;
    std::vector<int4> corners, div_rec;
    std::vector<double> geo;
    fcw::SharpFans sharp;
    fcw::PatchArrays patches;
};

// f on a thread of its own, or at once (an invalid future) when there is none to be had. The future
// waits for its thread when it goes out of scope.
template <class F>
std::future<void> on_thread(F&& f) {
    try {
        return std::async(std::launch::async, std::forward<F>(f));
    } catch (const std::system_error&) {
        f();
        return {};
    }
}

void mesh_tables(const fcw::MeshPrep& m, const fcw::Symbolic& S, MeshTables& t) {
    const int64_t n = S.n, nf = m.nf;
    t.coords.resize(3 * n);
    t.varea.resize(n);
    for (int64_t j = 0; j < n; ++j) {
        const int32_t o = S.perm[j];
        for (int c = 0; c < 3; ++c) t.coords[3 * j + c] = m.V[3 * (int64_t)o + c];
        t.varea[j] = m.vertex_area[o];
    }
    for (double x : t.coords) t.largest = std::max(t.largest, std::fabs(x));
    std::vector<int32_t>& fv = t.fv;
    fv.resize(3 * nf);
    t.bnd.resize(m.boundary.size());
    for (int64_t i = 0; i < 3 * nf; ++i) fv[i] = S.iperm[m.F[i]];
    for (size_t i = 0; i < m.boundary.size(); ++i) t.bnd[i] = S.iperm[m.boundary[i]];
    std::vector<int32_t>& inc_ptr = t.inc_ptr;
    inc_ptr.assign(n + 1, 0);
    std::vector<int32_t> inc_face(3 * nf);
    std::vector<int8_t> inc_corner(3 * nf);
    for (int64_t i = 0; i < 3 * nf; ++i) inc_ptr[fv[i] + 1]++;
    for (int64_t j = 0; j < n; ++j) inc_ptr[j + 1] += inc_ptr[j];
    {
        std::vector<int32_t> fill(inc_ptr.begin(), inc_ptr.end() - 1);
        for (int64_t f = 0; f < nf; ++f)
            for (int c = 0; c < 3; ++c) {
                const int32_t v = fv[3 * f + c];
                inc_face[fill[v]] = (int32_t)f;
                inc_corner[fill[v]] = (int8_t)c;
                fill[v]++;
            }
    }
    // the face areas in a fixed point whose full scale is 2^62 >= the total, so that per-bin
    // sums are exact and independent of the order atomics add them in
    for (double x : m.lean_area) t.lean_total += x;
    const int area_exp = t.lean_total > 0.0 ? (int)std::ceil(std::log2(t.lean_total)) : 0;
    const double area_scale = std::ldexp(1.0, 62 - area_exp);
    t.farea_fx.resize(nf);
    for (int64_t f = 0; f < nf; ++f) t.farea_fx[f] = std::llround(m.lean_area[f] * area_scale);
    t.area_unscale = 1.0 / area_scale;
    // FP64 divergence: faces in the order of their lowest vertices, with their corners and geometry
    auto face_records = [&] {
        std::vector<int32_t> place(nf), start(n + 1, 0);
        t.corners.resize(nf);
        t.div_rec.resize(3 * nf);
        t.geo.assign(8 * nf, 0.0);
        for (int64_t f = 0; f < nf; ++f) start[std::min({fv[3 * f], fv[3 * f + 1], fv[3 * f + 2]}) + 1]++;
        for (int64_t j = 0; j < n; ++j) start[j + 1] += start[j];
        for (int64_t f = 0; f < nf; ++f) {
            const int32_t p = start[std::min({fv[3 * f], fv[3 * f + 1], fv[3 * f + 2]})]++;
            place[f] = p;
            t.corners[p] = make_int4(fv[3 * f], fv[3 * f + 1], fv[3 * f + 2], 0);
            for (int x = 0; x < 6; ++x) t.geo[8 * (int64_t)p + x] = m.gb[9 * f + 3 + x];
            t.geo[8 * (int64_t)p + 6] = m.grad_area[f];
        }
        for (int64_t q = 0; q < 3 * nf; ++q) {
            const int32_t f = inc_face[q];
            t.div_rec[q] = make_int4(fv[3 * f], fv[3 * f + 1], fv[3 * f + 2],
                                     place[f] | ((int32_t)inc_corner[q] << fcw::kIncCornerShift));
        }
    };
    std::future<void> records = on_thread(face_records);
    fcw::face_fans(m, fv, inc_ptr, inc_face, inc_corner, t.fan_ptr, t.fan_steps, t.fan_walk);
    std::future<void> sharp =
        on_thread([&] { fcw::sharp_fans(m, fv, t.fan_ptr, t.fan_steps, t.fan_walk, t.sharp); });
    fcw::face_patches(t.fan_ptr, t.fan_steps, t.patches);
    if (sharp.valid()) sharp.get();
    if (records.valid()) records.get();
}

// e's device arrays of the mesh
int upload_mesh(fcw_engine* e, const MeshTables& t) {
    const auto& S = e->sym;
    const auto& m = e->mesh;
    e->area_unscale = t.area_unscale;
    e->lean_total = t.lean_total;
    // two coordinates rounded to FP32 (2^-24 each) in three dimensions: 2.1e-7 of the largest
    e->chord_slack = 4e-7 * t.largest;
    FCW_TRY(e->upload(&e->farea_fx_d, t.farea_fx));
    int4 *corners_d, *div_rec_d;
    double* geo_d;
    fcw::Patch* patches_d;
    int32_t *big_d, *prow_d, *fan_ptr_d;
    fcw::FanStep* fans_d;
    FCW_TRY(e->upload(&corners_d, t.corners));
    FCW_TRY(e->upload(&div_rec_d, t.div_rec));
    FCW_TRY(e->upload(&geo_d, t.geo));
    FCW_TRY(e->upload(&patches_d, t.patches.patches));
    FCW_TRY(e->upload(&big_d, t.patches.big));
    FCW_TRY(e->upload(&prow_d, t.patches.rows));
    FCW_TRY(e->upload(&fan_ptr_d, t.fan_ptr));
    FCW_TRY(e->upload(&fans_d, t.fan_steps));
    FCW_TRY(e->upload(&e->fan_walk_d, t.fan_walk));
    int32_t *fv_d, *inc_ptr_d;
    FCW_TRY(e->upload(&fv_d, t.fv));
    FCW_TRY(e->upload(&inc_ptr_d, t.inc_ptr));
    e->fd.nv = (int32_t)S.n; e->fd.nf = (int32_t)m.nf; e->fd.fv = fv_d;
    e->fd.inc_ptr = inc_ptr_d;
    e->fd.corners = corners_d; e->fd.geo = geo_d; e->fd.inc_rec = div_rec_d;
    e->fd.npatches = (int32_t)t.patches.patches.size(); e->fd.nbig = (int32_t)t.patches.big.size();
    e->fd.patches = patches_d; e->fd.big = big_d; e->fd.patch_rows = prow_d; e->fd.fan_ptr = fan_ptr_d;
    e->fd.fans = fans_d;
    FCW_TRY(e->upload(&e->coords_d, t.coords));
    FCW_TRY(e->upload(&e->varea_d, t.varea));
    FCW_TRY(e->upload(&e->boundary_d, t.bnd));
    FCW_TRY(e->upload(&e->farea_d, m.lean_area));
    FCW_TRY(e->upload(&e->g11_d, m.g11));
    FCW_TRY(e->upload(&e->g12_d, m.g12));
    FCW_TRY(e->upload(&e->g22_d, m.g22));
    FCW_TRY(e->upload(&e->iperm_d, S.iperm));
    {
        std::vector<uint8_t> gnew(S.n);
        for (int64_t i = 0; i < S.n; ++i) gnew[i] = e->grounded_old[S.perm[i]];
        FCW_TRY(e->upload(&e->grounded_d, gnew));
    }
    if (e->ncomp > 1) {
        e->clevel.n = (int32_t)S.n;
        FCW_TRY(e->upload(&e->clevel.comp, e->comp_h));
        FCW_TRY(e->upload(&e->clevel.mass, e->cmass_h));
        FCW_TRY(e->upload(&e->clevel.area, e->carea_h));
    }
    FCW_TRY(e->upload(&e->perm_d, S.perm));
    if (!t.sharp.vertices.empty()) {
        int32_t *sharp_d, *sharp_ptr_d;
        fcw::FanStep* sharp_fans_d;
        FCW_TRY(e->upload(&sharp_d, t.sharp.vertices));
        FCW_TRY(e->upload(&sharp_ptr_d, t.sharp.ptr));
        FCW_TRY(e->upload(&sharp_fans_d, t.sharp.steps));
        e->fd.nsharp = (int32_t)t.sharp.vertices.size();
        e->fd.sharp = sharp_d; e->fd.sharp_ptr = sharp_ptr_d; e->fd.sharp_fans = sharp_fans_d;
    }
    return FCW_OK;
}

int build_engine(fcw_engine* e, const double* V, int64_t nv, const int32_t* F, int64_t nf) {
    std::string err;
    double t0 = now_ms();
    if (fcw::prepare_mesh(V, nv, F, nf, e->mesh, err)) return fail(FCW_E_INVALID, err);
    if (e->prm.robust && fcw::intrinsic_delaunay(e->mesh, kMollifyFactor, e->n_flips, err))
        return fail(FCW_E_INVALID, err);
    e->t_coef = std::pow(e->prm.diffusion_length_mm / e->mesh.mean_edge, 2.0);
    e->t = e->t_coef * e->mesh.mean_edge * e->mesh.mean_edge;
    if (fcw::build_symbolic(e->mesh, e->prm.leaf_size, e->prm.max_width, e->prm.relax, e->sym, err)) return fail(FCW_E_INVALID, err);
    e->analyze_ms = now_ms() - t0;
    const auto& S = e->sym;
    const auto& m = e->mesh;
    if (S.max_ns > fcw::kMaxWidth) return fail(FCW_E_INVALID, "supernode wider than the kernels support");
    if (nf > fcw::kIncFace) return fail(FCW_E_INVALID, "mesh has too many faces");
    // The mesh tables are formed on threads of their own while this one plans the sweeps. A build at 147k
    // vertices (64 columns, one block in flight) took 480 ms with all of it one after the other, 375 now.
    MeshTables tables;
    std::future<void> tables_done = on_thread([&] { mesh_tables(m, S, tables); });
    {
        // each connected component grounded at its last eliminated vertex: L is singular once
        // per component
        std::vector<int32_t> comp;
        e->ncomp = mesh_components(m, S.perm, comp);
        std::vector<int32_t> last(e->ncomp, -1);
        for (int64_t i = 0; i < S.n; ++i) last[comp[S.perm[i]]] = (int32_t)i;  // ascending i: the last wins
        e->grounded_old.assign(S.n, 0);
        for (int32_t c = 0; c < e->ncomp; ++c) e->grounded_old[S.perm[last[c]]] = 1;
        if (e->ncomp > 1) {
            e->comp_h.resize(S.n);
            e->cmass_h.resize(S.n);
            e->carea_h.assign(e->ncomp, 0.0);
            for (int64_t i = 0; i < S.n; ++i) {
                e->comp_h[i] = comp[S.perm[i]];
                e->cmass_h[i] = m.mass[S.perm[i]];
                e->carea_h[e->comp_h[i]] += e->cmass_h[i];
            }
        }
    }

    FCW_CUDA(cudaSetDevice(e->device));
    FCW_CUDA(cudaDeviceGetAttribute(&e->num_sms, cudaDevAttrMultiProcessorCount, e->device));
    FCW_CUDA(fcw::configure_kernels());
    FCW_CUDA(fcw::configure_divergence_kernels());
    FCW_CUDA(fcw::configure_front_kernels());
    FCW_CUDA(fcw::configure_solve_kernels());
    FCW_CUDA(fcw::configure_tc_kernels());
    FCW_CUDA(cudaStreamCreateWithFlags(&e->stream, cudaStreamNonBlocking));
    FCW_CUDA(cudaEventCreateWithFlags(&e->ev_in, cudaEventDisableTiming));
    e->pool.resize((size_t)std::max(1, e->prm.pipeline_depth));
    for (auto& w : e->pool) {
        FCW_CUDA(cudaStreamCreateWithFlags(&w.stream, cudaStreamNonBlocking));
        FCW_CUDA(cudaEventCreateWithFlags(&w.done, cudaEventDisableTiming));
    }
    FCW_TRY(e->dalloc(&e->err_d, 1));
    e->err_h = words().take();
    FCW_CUDA(cudaMemset(e->err_d, 0, sizeof(int)));

    // structure
    int32_t *sn_c0, *sn_m, *rows, *sn_parent, *col_sn, *level_nodes, *child_ptr, *child_list, *relind, *seg_sn,
        *seg_pos;
    int64_t *sn_rowptr, *sn_valptr, *sn_invptr, *sn_updptr, *seg_ptr, *a_dst;
    FCW_TRY(e->upload(&sn_c0, S.sn_c0));
    FCW_TRY(e->upload(&sn_m, S.sn_m));
    FCW_TRY(e->upload(&sn_rowptr, S.sn_rowptr));
    FCW_TRY(e->upload(&rows, S.rows));
    FCW_TRY(e->upload(&sn_valptr, S.sn_valptr));
    FCW_TRY(e->upload(&sn_invptr, S.sn_invptr));
    FCW_TRY(e->upload(&sn_updptr, S.sn_updptr));
    FCW_TRY(e->upload(&sn_parent, S.sn_parent));
    FCW_TRY(e->upload(&col_sn, S.col_sn));
    FCW_TRY(e->upload(&level_nodes, S.level_nodes));
    FCW_TRY(e->upload(&child_ptr, S.child_ptr));
    FCW_TRY(e->upload(&child_list, S.child_list));
    FCW_TRY(e->upload(&relind, S.relind));
    FCW_TRY(e->upload(&seg_ptr, S.seg_ptr));
    FCW_TRY(e->upload(&seg_sn, S.seg_sn));
    FCW_TRY(e->upload(&seg_pos, S.seg_pos));
    FCW_TRY(e->upload(&a_dst, S.a_dst));
    fcw::DevPlan& P = e->plan;
    P.n = (int32_t)S.n;
    P.nsuper = S.nsuper;
    P.nlevels = S.nlevels;
    P.sn_c0 = sn_c0; P.sn_m = sn_m; P.sn_rowptr = sn_rowptr; P.rows = rows; P.sn_valptr = sn_valptr;
    P.sn_invptr = sn_invptr; P.sn_updptr = sn_updptr; P.sn_parent = sn_parent; P.col_sn = col_sn;
    P.level_nodes = level_nodes; P.child_ptr = child_ptr; P.child_list = child_list; P.relind = relind;
    P.seg_ptr = seg_ptr; P.seg_sn = seg_sn; P.seg_pos = seg_pos;
    e->level_tiles.assign(S.nlevels, 1);
    for (int32_t l = 0; l < S.nlevels; ++l) {
        int64_t mx = 1;
        for (int32_t q = S.level_ptr[l]; q < S.level_ptr[l + 1]; ++q) {
            const int32_t s = S.level_nodes[q];
            const int64_t nr = S.sn_m[s] - (S.sn_c0[s + 1] - S.sn_c0[s]);
            const int64_t nt = (nr + 31) / 32;
            mx = std::max<int64_t>(mx, nt * (nt + 1) / 2);
        }
        e->level_tiles[l] = (int32_t)std::min<int64_t>(mx, 512);
    }

    // the batched sweeps' fronts and tasks
    if (fcw::build_fronts(S, e->fr, err)) return fail(FCW_E_INVALID, err);
    {
        fcw::Fronts& f = e->fr;
        fcw::FrontPlan& q = e->frp;
        std::vector<int64_t> ptr((size_t)f.nf + 1, 0);
        std::vector<int32_t> sn_front((size_t)S.nsuper), merged;
        for (int32_t t = 0; t < f.nf; ++t) {
            const int32_t ns = f.c0[t + 1] - f.c0[t];
            ptr[t + 1] = ptr[t] + (int64_t)f.m[t] * ns;
            for (int32_t k = f.sn0[t]; k < f.sn0[t + 1]; ++k) sn_front[k] = t;
            if (f.sn0[t + 1] - f.sn0[t] > 1) {
                merged.push_back(t);
                q.max_m = std::max(q.max_m, f.m[t]);
                q.max_ns = std::max(q.max_ns, ns);
            }
            if (f.m[t] > fcw::max_front_rows())
                return fail(FCW_E_INVALID, "front too large for the sweeps (" + std::to_string(f.m[t]) + " rows)");
        }
        e->bwd_depth.assign(f.nlevels, 0);
        for (int32_t l = 0; l < f.nlevels; ++l)
            for (int32_t k = f.bwd_ptr[l]; k < f.bwd_ptr[l + 1]; ++k)
                e->bwd_depth[l] = std::max(e->bwd_depth[l], f.bwd[k].depth);
        int32_t *c0, *m, *parent, *sn0, *snf, *colf, *pos, *mg;
        int64_t* pd;
        FCW_TRY(e->upload(&c0, f.c0));
        FCW_TRY(e->upload(&m, f.m));
        FCW_TRY(e->upload(&parent, f.parent));
        FCW_TRY(e->upload(&sn0, f.sn0));
        FCW_TRY(e->upload(&snf, sn_front));
        FCW_TRY(e->upload(&colf, f.col_front));
        FCW_TRY(e->upload(&pos, f.pos));
        FCW_TRY(e->upload(&mg, merged));
        FCW_TRY(e->upload(&pd, ptr));
        q.nf = f.nf; q.n_merged = (int32_t)merged.size(); q.entries = ptr[f.nf];
        q.c0 = c0; q.m = m; q.parent = parent; q.sn0 = sn0; q.sn_front = snf; q.col_front = colf; q.pos = pos;
        q.merged = mg; q.ptr = pd;
        FCW_TRY(e->upload(&e->fwd_tasks, f.fwd));
        FCW_TRY(e->upload(&e->bwd_tasks, f.bwd));
        FCW_TRY(e->upload(&e->rec_d, f.rec));
        FCW_TRY(e->upload(&e->rec_child_d, f.rec_child));
        FCW_TRY(e->upload(&e->more_d, f.more));
        FCW_TRY(e->upload(&e->front_rows_d, f.rows));
        FCW_TRY(e->upload(&e->asm_rows_d, f.asm_rows));
    }

    // the tensor-core sweeps' update rows, per-front-row gather lists and tasks, over supernodes (see
    // solve_tc.cu)
    if (e->prm.tc_sweeps) {
        const int32_t NS = S.nsuper;
        std::vector<int64_t> uoff(NS + 1, 0), poff(NS, 0);
        std::vector<int32_t> nsplit(NS, 1);
        int64_t parts = 0;
        for (int32_t s = 0; s < NS; ++s) {
            const int32_t ns = S.sn_c0[s + 1] - S.sn_c0[s], nr = S.sn_m[s] - ns;
            uoff[s + 1] = uoff[s] + nr;
            nsplit[s] = std::max(1, (nr + fcw::kSplitRows - 1) / fcw::kSplitRows);
            poff[s] = parts;
            if (nsplit[s] > 1) parts += nsplit[s];
        }
        e->n_urows = uoff[NS];
        e->n_parts = parts;
        {
            std::vector<int2> bt, tft;
            e->tc_fwd_ptr.assign(S.nlevels + 1, 0);
            e->tc_bwd_ptr.assign(S.nlevels + 1, 0);
            for (int32_t l = 0; l < S.nlevels; ++l) {
                // forward: per supernode the inverse block with the first 64 update rows, then
                // 128-row update chunks
                for (int32_t q = S.level_ptr[l]; q < S.level_ptr[l + 1]; ++q) {
                    const int32_t s = S.level_nodes[q];
                    const int32_t ns = S.sn_c0[s + 1] - S.sn_c0[s], nr = S.sn_m[s] - ns;
                    const int32_t nchunk = 1 + std::max(0, (nr - 64 + 127) / 128);
                    for (int32_t c = 0; c < nchunk; ++c) tft.push_back(make_int2(s, c));
                    for (int32_t c = 0; c < nsplit[s]; ++c) bt.push_back(make_int2(s, c));
                }
                e->tc_fwd_ptr[l + 1] = (int32_t)tft.size();
                e->tc_bwd_ptr[l + 1] = (int32_t)bt.size();
            }
            FCW_TRY(e->upload(&e->tc_fwd_tasks, tft));
            FCW_TRY(e->upload(&e->tc_bwd_tasks, bt));
            FCW_TRY(e->upload(&e->poff_d, poff));
            FCW_TRY(e->upload(&e->nsplit_d, nsplit));
        }
        const int64_t nfront = S.sn_rowptr[NS];
        std::vector<int32_t> gptr(nfront + 1, 0), gsrc(e->n_urows);
        for (int32_t c = 0; c < NS; ++c) {
            const int32_t p = S.sn_parent[c];
            const int32_t nsc = S.sn_c0[c + 1] - S.sn_c0[c];
            for (int64_t q = S.sn_rowptr[c] + nsc; q < S.sn_rowptr[c + 1]; ++q) gptr[S.sn_rowptr[p] + S.relind[q] + 1]++;
        }
        for (int64_t g = 0; g < nfront; ++g) gptr[g + 1] += gptr[g];
        {
            std::vector<int32_t> fill(gptr.begin(), gptr.end() - 1);
            for (int32_t c = 0; c < NS; ++c) {
                const int32_t p = S.sn_parent[c];
                const int32_t nsc = S.sn_c0[c + 1] - S.sn_c0[c];
                for (int64_t q = S.sn_rowptr[c] + nsc; q < S.sn_rowptr[c + 1]; ++q) {
                    const int64_t g = S.sn_rowptr[p] + S.relind[q];
                    gsrc[fill[g]] = (int32_t)(uoff[c] + (q - S.sn_rowptr[c] - nsc));
                    fill[g]++;
                }
            }
        }
        if (e->n_urows > INT32_MAX || nfront > INT32_MAX) return fail(FCW_E_INVALID, "mesh too large for 32-bit update indices");
        FCW_TRY(e->upload(&e->uoff_d, uoff));
        FCW_TRY(e->upload(&e->gm_ptr_d, gptr));
        FCW_TRY(e->upload(&e->gm_src_d, gsrc));
    }

    // uploaded before the factors are allocated: where an engine's arrays lie shows in the single-source
    // sweeps (26k vertices: 110 us a call, 117 with the tables uploaded after the factors)
    if (tables_done.valid()) tables_done.get();
    FCW_TRY(upload_mesh(e, tables));

    // numeric factorisations
    t0 = now_ms();
    double *upd, *aval_d;
    FCW_TRY(e->dalloc(&upd, S.n_upd));
    FCW_TRY(e->dalloc(&aval_d, S.nnz_lower_a));
    FCW_TRY(e->dalloc(&e->val_h, S.nnz_factor));
    FCW_TRY(e->dalloc(&e->inv_h, S.n_inv));
    FCW_TRY(e->dalloc(&e->val_p, S.nnz_factor));
    FCW_TRY(e->dalloc(&e->inv_p, S.n_inv));
    double* front_rows;
    FCW_TRY(e->dalloc(&front_rows, e->frp.entries));
    // the sweeps' panels of one factor; a chunk's copy may run up to three depth rows past a panel
    constexpr int64_t kPanelSlack = 1024;
    auto pack = [&](const double* val, const double* inv, auto** fwd, auto** bwd, int64_t nfwd, int64_t nbwd) -> int {
        using T = std::remove_reference_t<decltype(**fwd)>;
        FCW_TRY(e->dalloc(fwd, (size_t)(nfwd + kPanelSlack)));
        FCW_TRY(e->dalloc(bwd, (size_t)(nbwd + kPanelSlack)));
        FCW_CUDA(cudaMemsetAsync(*fwd + nfwd, 0, kPanelSlack * sizeof(T), e->stream));
        FCW_CUDA(cudaMemsetAsync(*bwd + nbwd, 0, kPanelSlack * sizeof(T), e->stream));
        fcw::launch_front_rows(e->plan, e->frp, val, inv, front_rows, e->stream);
        fcw::launch_pack<T>(e->frp, true, e->fwd_tasks, (int32_t)e->fr.fwd.size(), front_rows, *fwd, e->stream);
        fcw::launch_pack<T>(e->frp, false, e->bwd_tasks, (int32_t)e->fr.bwd.size(), front_rows, *bwd, e->stream);
        FCW_CUDA(cudaGetLastError());
        return FCW_OK;
    };
    auto run_factor = [&](Op op, double* val, double* inv, const char* what) -> int {
        std::vector<double> av = operator_values(e, op);
        FCW_CUDA(cudaMemcpyAsync(aval_d, av.data(), av.size() * sizeof(double), cudaMemcpyHostToDevice, e->stream));
        FCW_CUDA(cudaMemsetAsync(val, 0, S.nnz_factor * sizeof(double), e->stream));
        FCW_CUDA(cudaMemsetAsync(upd, 0, std::max<int64_t>(S.n_upd, 1) * sizeof(double), e->stream));
        fcw::launch_scatter_a(S.nnz_lower_a, a_dst, aval_d, val, e->stream);
        for (int32_t l = 0; l < S.nlevels; ++l) {
            const int32_t l0 = S.level_ptr[l], cnt = S.level_ptr[l + 1] - l0;
            fcw::launch_factor_front(e->plan, l0, cnt, val, inv, upd, e->err_d, e->stream);
            fcw::launch_factor_update(e->plan, l0, cnt, e->level_tiles[l], val, upd, e->stream);
        }
        fcw::launch_panel_inverse(e->plan, val, inv, e->stream);
        FCW_CUDA(cudaGetLastError());
        return check_kernel_errors(e, what);
    };
    FCW_TRY(run_factor(Op::Heat, e->val_h, e->inv_h, "heat factorisation"));
    FCW_TRY(run_factor(Op::Poisson, e->val_p, e->inv_p, "Poisson factorisation"));
    FCW_TRY(pack(e->val_h, e->inv_h, &e->pan_hf, &e->pan_hb, e->fr.fwd64, e->fr.bwd64));
    FCW_TRY(pack(e->val_p, e->inv_p, &e->pan_pf, &e->pan_pb, e->fr.fwd64, e->fr.bwd64));
    if (e->prm.build_mixed && e->prm.refine > 0) {
        // L_g in CSR, elimination order: the entries the FP32 factor came from
        std::vector<int64_t> rp(S.n + 1, 0);
        std::vector<int32_t> ci;
        std::vector<double> av;
        ci.reserve(m.Li.size());
        av.reserve(m.Li.size());
        for (int64_t i = 0; i < S.n; ++i) {
            const int32_t old = S.perm[i];
            for (int64_t k = m.Lp[old]; k < m.Lp[old + 1]; ++k) {
                const int32_t j = m.Li[k];
                const bool diag = j == old;
                const double v = (e->grounded_old[old] || e->grounded_old[j]) ? (diag ? 1.0 : 0.0) : m.Lx[k];
                if (v == 0.0 && !diag) continue;
                ci.push_back(S.iperm[j]);
                av.push_back(v);
            }
            rp[i + 1] = (int64_t)ci.size();
        }
        int64_t* rp_d;
        int32_t* ci_d;
        double* av_d;
        FCW_TRY(e->upload(&rp_d, rp));
        FCW_TRY(e->upload(&ci_d, ci));
        FCW_TRY(e->upload(&av_d, av));
        e->lg.n = (int32_t)S.n;
        e->lg.rp = rp_d;
        e->lg.ci = ci_d;
        e->lg.av = av_d;
    }
    if (e->prm.build_mixed) {
        double *val_tmp, *inv_tmp;
        FCW_TRY(e->dalloc(&val_tmp, S.nnz_factor));
        FCW_TRY(e->dalloc(&inv_tmp, S.n_inv));
        FCW_TRY(run_factor(Op::Grounded, val_tmp, inv_tmp, "grounded Poisson factorisation"));
        FCW_TRY(pack(val_tmp, inv_tmp, &e->pan_gf, &e->pan_gb, e->fr.fwd32, e->fr.bwd32));
        if (e->prm.tc_sweeps) {
            std::vector<int64_t> cptr(S.nsuper + 1, 0);
            for (int32_t s = 0; s < S.nsuper; ++s) {
                const int64_t ns = S.sn_c0[s + 1] - S.sn_c0[s], nr = S.sn_m[s] - ns;
                const int64_t ns8 = (ns + 7) / 8 * 8, nr32 = (nr + 31) / 32 * 32;
                cptr[s + 1] = cptr[s] + ns8 * (ns8 + nr32);
            }
            FCW_TRY(e->upload(&e->core_ptr_d, cptr));
            FCW_TRY(e->dalloc(&e->core_hi, (size_t)cptr[S.nsuper]));
            FCW_TRY(e->dalloc(&e->core_lo, (size_t)cptr[S.nsuper]));
            FCW_TRY(e->dalloc(&e->coreT_hi, (size_t)cptr[S.nsuper]));
            FCW_TRY(e->dalloc(&e->coreT_lo, (size_t)cptr[S.nsuper]));
            fcw::launch_build_cores(e->plan, val_tmp, inv_tmp, e->core_ptr_d, e->core_hi, e->core_lo, e->coreT_hi,
                                    e->coreT_lo, e->stream);
            FCW_CUDA(cudaGetLastError());
        }
        FCW_CUDA(cudaStreamSynchronize(e->stream));
        e->release(val_tmp);
        e->release(inv_tmp);
    }
    FCW_CUDA(cudaStreamSynchronize(e->stream));
    e->release(front_rows);
    e->release(upd);
    e->release(aval_d);
    e->factor_ms = now_ms() - t0;
    return FCW_OK;
}

// Statistics records that any block of at most K columns writes.
int64_t stat_partials(int64_t n, int64_t K) {
    int64_t most = 0;
    for (int64_t k = 32; k <= K; k += 32) {
        const int64_t t = fcw::stat_tile(n, k);
        most = std::max(most, (n + t - 1) / t * k);
    }
    const int64_t one = fcw::stat_tile(n, 1);
    return std::max(most, (n + one - 1) / one);
}

int ensure_one(fcw_engine* e, Workspace& w, int32_t K, int32_t stride) {
    if (w.K >= K && w.out_stride >= stride) return FCW_OK;
    const int32_t Kn = std::max(K, w.K);
    const int32_t sn = std::max(stride, w.out_stride);
    void* old[] = {w.Bh, w.Bp64, w.Y, w.dT64, w.src, w.dst, w.reach, w.band, w.longf, w.out, w.U, w.W, w.part,
                   w.counters, w.partials, w.near_list, w.near_count, w.desc, w.csum};
    for (void* p : old)
        if (p) e->release(p);
    w.drop_graph();  // its launches name the old buffers
    cudaStream_t stream = w.stream;
    cudaEvent_t done = w.done;
    w = Workspace{};
    w.stream = stream;
    w.done = done;
    const int64_t n = e->sym.n, nf = e->mesh.nf;
    FCW_TRY(e->dalloc(&w.Bh, (size_t)n * Kn));
    FCW_TRY(e->dalloc(&w.Bp64, (size_t)n * Kn));
    w.Bp32 = reinterpret_cast<float*>(w.Bp64);  // a block uses one precision
    FCW_TRY(e->dalloc(&w.Y, (size_t)n * Kn));
    FCW_TRY(e->dalloc(&w.dT64, (size_t)n * Kn));
    w.dT32 = reinterpret_cast<float*>(w.dT64);
    FCW_TRY(e->dalloc(&w.src, (size_t)Kn));
    FCW_TRY(e->dalloc(&w.dst, (size_t)Kn));
    FCW_TRY(e->dalloc(&w.reach, (size_t)std::max<int64_t>(e->fr.nf, 1) * (Kn / fcw::kReachCols)));
    FCW_TRY(e->dalloc(&w.band, (size_t)nf * Kn));
    FCW_TRY(e->dalloc(&w.longf, (size_t)nf * Kn));
    FCW_TRY(e->dalloc(&w.out, (size_t)sn * Kn));
    FCW_TRY(e->dalloc(&w.partials, (size_t)stat_partials(n, Kn) * 8));
    FCW_TRY(e->dalloc(&w.near_list, (size_t)n * Kn));
    FCW_TRY(e->dalloc(&w.near_count, (size_t)Kn));
    const int64_t urows = e->prm.tc_sweeps ? std::max(e->fr.n_urows, e->n_urows) : e->fr.n_urows;
    FCW_TRY(e->dalloc(&w.U, (size_t)std::max<int64_t>(urows, 1) * Kn));
    FCW_TRY(e->dalloc(&w.W, (size_t)std::max<int64_t>(e->fr.n_wrows, 1) * Kn));
    if (e->prm.tc_sweeps) {
        FCW_TRY(e->dalloc(&w.part, (size_t)std::max<int64_t>(e->n_parts, 1) * fcw::kMaxWidth * Kn));
        const int64_t nctr = (int64_t)std::max<int32_t>(e->sym.nsuper, 1) * (Kn / fcw::kRhsTile);
        FCW_TRY(e->dalloc(&w.counters, (size_t)nctr));
        FCW_CUDA(cudaMemset(w.counters, 0, nctr * sizeof(int)));
    }
    FCW_TRY(e->dalloc(&w.desc, 1));
    if (e->ncomp > 1) FCW_TRY(e->dalloc(&w.csum, (size_t)(fcw::component_tiles(n) + 1) * Kn));
    w.K = Kn;
    w.out_stride = sn;
    return FCW_OK;
}

// Every workspace of the pool holds at least K columns and `stride` output doubles per column.
// If the device cannot hold another workspace, the pool keeps the ones that fit (at least
// one): fewer blocks are in flight, nothing else changes.
int ensure_workspace(fcw_engine* e, int32_t K, int32_t stride) {
    for (size_t i = 0; i < e->pool.size(); ++i) {
        const int rc = ensure_one(e, e->pool[i], K, stride);
        if (rc == FCW_OK) continue;
        if (i == 0 || rc != FCW_E_NOMEM) return rc;
        e->sync_streams();
        for (size_t j = i; j < e->pool.size(); ++j) {
            Workspace& w = e->pool[j];
            void* bufs[] = {w.Bh, w.Bp64, w.Y, w.dT64, w.src, w.dst, w.reach, w.band, w.longf, w.out, w.U, w.W, w.part,
                            w.counters, w.partials, w.near_list, w.near_count, w.desc, w.csum};
            for (void* p : bufs)
                if (p) e->release(p);
            w.drop_graph();
            for (auto& m : w.marks) cudaEventDestroy(m.second);
            if (w.done) cudaEventDestroy(w.done);
            if (w.stream) cudaStreamDestroy(w.stream);
        }
        e->pool.resize(i);
        e->cur_ws = 0;
        return FCW_OK;
    }
    return FCW_OK;
}

// Both sweeps on the front panels: right-hand sides R (or the identity columns and reach flags in
// `a`), forward result into Y, solution into X (n x K, three different arrays).
template <typename T>
void sweep(fcw_engine* e, fcw::SweepArgs<T> a, const T* fwd, const T* bwd, const T* R, T* Y, T* X, int32_t K,
           cudaStream_t st, int stage_fwd, int stage_bwd) {
    const fcw::Fronts& f = e->fr;
    a.R = R;
    a.Y = Y;
    a.X = X;
    a.U = reinterpret_cast<T*>(e->cw().U);
    a.W = reinterpret_cast<T*>(e->cw().W);
    a.K = K;
    a.rec = reinterpret_cast<const int4*>(e->rec_d);
    a.rec_child = e->rec_child_d;
    a.more = e->more_d;
    a.rows = e->front_rows_d;
    a.asm_rows = reinterpret_cast<const int4*>(e->asm_rows_d);
    a.err = e->err_d;
    const int32_t leaf_f = (int32_t)(sizeof(T) == 8 ? f.leaf_fwd64 : f.leaf_fwd32);
    const int32_t leaf_b = (int32_t)(sizeof(T) == 8 ? f.leaf_bwd64 : f.leaf_bwd32);
    mark(e, st, stage_fwd);
    a.tasks = e->fwd_tasks;
    a.panel = fwd;
    for (int32_t l = 0; l < f.nlevels; ++l) {
        const bool wide = l >= f.first_wide, overlap = l > 0 || !a.reach;
        a.gathers = l > 0;
        if (wide) fcw::launch_assemble<T>(a, f.asm_ptr[l], f.asm_ptr[l + 1] - f.asm_ptr[l], overlap, st);
        if (l == 0 && !wide && fcw::launch_leaves<T>(a, false, f.fwd_ptr[1], f.fwd_rows[0], leaf_f, 0, st)) continue;
        fcw::launch_fwd_level<T>(a, f.fwd_ptr[l], f.fwd_ptr[l + 1] - f.fwd_ptr[l], f.fwd_rows[l], wide, wide || overlap,
                                 st);
    }
    a.delta_src = nullptr;
    mark(e, st, stage_bwd);
    a.tasks = e->bwd_tasks;
    a.panel = bwd;
    for (int32_t l = f.nlevels - 1; l >= 0; --l) {
        if (l == 0 && fcw::launch_leaves<T>(a, true, f.bwd_ptr[1], f.bwd_rows[0], leaf_b, e->bwd_depth[0], st)) continue;
        fcw::launch_bwd_level<T>(a, f.bwd_ptr[l], f.bwd_ptr[l + 1] - f.bwd_ptr[l], f.bwd_rows[l], e->bwd_depth[l], st);
    }
    e->launches += 2 * (int64_t)f.nlevels + (f.nlevels - f.first_wide);
}

// Heat solve for the K sources in ws.src: u (elimination order, n x K) in ws.Bh.
void heat_solve(fcw_engine* e, int32_t K, cudaStream_t st) {
    Workspace& w = e->cw();
    mark(e, st, FCW_STAGE_HEAT_FWD);
    fcw::launch_reach(e->frp.col_front, e->frp.parent, e->fr.nf, e->fr.nlevels, w.src, K, w.reach, st);
    e->launches += 2;
    fcw::SweepArgs<double> a;
    a.delta_src = w.src;
    a.reach = w.reach;
    a.reach_tiles = K / fcw::kReachCols;
    sweep<double>(e, a, e->pan_hf, e->pan_hb, nullptr, w.Y, w.Bh, K, st, FCW_STAGE_HEAT_FWD, FCW_STAGE_HEAT_BWD);
}

// FP32 sweeps on the tensor cores, over the supernodes' levels: R -> Y (in place after the forward).
int sweep_tc(fcw_engine* e, const float* R, float* Y, int32_t K, cudaStream_t st) {
    const auto& S = e->sym;
    fcw::SolveArgs<float> a;
    a.p = e->plan;
    a.R = R;
    a.B = Y;
    a.K = K;
    a.U = reinterpret_cast<float*>(e->cw().U);
    a.uoff = e->uoff_d;
    a.gm_ptr = e->gm_ptr_d;
    a.gm_src = e->gm_src_d;
    a.nsplit = e->nsplit_d;
    a.poff = e->poff_d;
    a.part = reinterpret_cast<float*>(e->cw().part);
    a.counters = e->cw().counters;
    a.ktiles = e->cw().K / fcw::kRhsTile;
    a.core_hi = e->core_hi;
    a.core_lo = e->core_lo;
    a.coreT_hi = e->coreT_hi;
    a.coreT_lo = e->coreT_lo;
    a.core_ptr = e->core_ptr_d;
    a.err = e->err_d;
    CUtensorMap rmap, bmap;
    if (fcw::make_rows_map(&rmap, a.R, S.n, a.K) || fcw::make_rows_map(&bmap, a.B, S.n, a.K))
        return fail(FCW_E_CUDA, "cuTensorMapEncodeTiled failed for the Poisson right-hand sides");
    mark(e, st, FCW_STAGE_POISSON_FWD);
    a.tasks = e->tc_fwd_tasks;
    for (int32_t l = 0; l < S.nlevels; ++l)
        fcw::launch_fwd_level_tc(a, e->tc_fwd_ptr[l], e->tc_fwd_ptr[l + 1] - e->tc_fwd_ptr[l], rmap, st);
    mark(e, st, FCW_STAGE_POISSON_BWD);
    a.tasks = e->tc_bwd_tasks;
    for (int32_t l = S.nlevels - 1; l >= 0; --l)
        fcw::launch_bwd_level_tc(a, e->tc_bwd_ptr[l], e->tc_bwd_ptr[l + 1] - e->tc_bwd_ptr[l], bmap, st);
    e->launches += 2 * (int64_t)S.nlevels;
    return FCW_OK;
}

// Poisson solve: right-hand sides R, solution into Y (both n x K, elimination order). The forward
// result goes to the heat solution's buffer, which the divergence has read by now.
template <typename T>
int poisson_solve(fcw_engine* e, const T* fwd, const T* bwd, const T* R, T* Y, int32_t K, cudaStream_t st) {
    if constexpr (sizeof(T) == 4) {
        if (e->core_hi && K % fcw::kTcCols == 0) return sweep_tc(e, R, Y, K, st);
    }
    sweep<T>(e, fcw::SweepArgs<T>{}, fwd, bwd, R, reinterpret_cast<T*>(e->cw().Bh), Y, K, st, FCW_STAGE_POISSON_FWD,
             FCW_STAGE_POISSON_BWD);
    return FCW_OK;
}

// Distances for the K sources in ws.src, shifted, source-major in ws.dT64 / ws.dT32.
// With metric arguments, the shift also produces the health/MSD partials and near lists.
int distances_block(fcw_engine* e, int32_t K, int precision, cudaStream_t st, const fcw::MetricArgs* ma = nullptr) {
    Workspace& w = e->cw();
    const int32_t n = (int32_t)e->sym.n;
    heat_solve(e, K, st);
    mark(e, st, FCW_STAGE_DIVERGENCE);
    if (precision == FCW_PREC_MIXED) {
        float* Y = reinterpret_cast<float*>(w.Y);
        fcw::launch_divergence_mixed(e->fd, w.Bh, w.Bp32, K, e->grounded_d, st);
        FCW_TRY(poisson_solve<float>(e, e->pan_gf, e->pan_gb, w.Bp32, Y, K, st));
        // refinement: residual in FP64 and its FP32 solution, in the shift's output buffer
        // (two n x K float halves of dT64) before the shift writes it
        for (int32_t it = 0; it < e->prm.refine && e->lg.rp; ++it) {
            float* r = w.dT32;
            float* d = w.dT32 + (int64_t)n * K;
            fcw::launch_residual(e->lg, K, w.Bp32, Y, r, st);
            FCW_TRY(poisson_solve<float>(e, e->pan_gf, e->pan_gb, r, d, K, st));
            fcw::launch_add((int64_t)n * K, Y, d, e->num_sms, st);
            e->launches += 2;
        }
        if (e->ncomp > 1) {
            fcw::launch_component_level(e->clevel, K, w.src, Y, w.csum, st);
            e->launches += 3;
        }
        mark(e, st, FCW_STAGE_SHIFT);
        if (ma) fcw::launch_shift_stats<float, float>(*ma, K, Y, w.dT32, st);
        else fcw::launch_shift_transpose<float, float>(n, K, Y, w.src, w.dT32, st);
    } else {
        fcw::launch_divergence_fp64(e->fd, w.Bh, reinterpret_cast<double*>(w.band), w.Bp64, K, st);
        e->launches += 1;
        FCW_TRY(poisson_solve<double>(e, e->pan_pf, e->pan_pb, w.Bp64, w.Y, K, st));
        mark(e, st, FCW_STAGE_SHIFT);
        if (ma) fcw::launch_shift_stats<double, double>(*ma, K, w.Y, w.dT64, st);
        else fcw::launch_shift_transpose<double, double>(n, K, w.Y, w.src, w.dT64, st);
    }
    e->launches += 2;
    return FCW_OK;
}

int metric_args(fcw_engine* e, const double* targets, int32_t nt, int32_t nb, double eps, int32_t nsrc,
                fcw::MetricArgs& a) {
    if (nt < 1 || nt > fcw::kMaxTargets) return fail(FCW_E_INVALID, "n_targets must be in [1, 32]");
    if (nb < 0 || nb > fcw::kMaxBetween) return fail(FCW_E_INVALID, "n_between must be in [0, 8]");
    if (!targets) return fail(FCW_E_INVALID, "targets is NULL");
    for (int32_t i = 0; i + 1 < nt; ++i)
        if (!(targets[i] <= targets[i + 1])) return fail(FCW_E_INVALID, "targets must be sorted ascending");
    a = fcw::MetricArgs{};
    a.n = (int32_t)e->sym.n;
    a.nf = (int32_t)e->mesh.nf;
    a.nsrc = nsrc;
    a.stride = fcw_metrics_stride(nt, nb);
    a.n_targets = nt;
    a.n_between = nb;
    a.n_boundary = (int32_t)e->mesh.boundary.size();
    a.coords = e->coords_d;
    a.vertex_area = e->varea_d;
    a.boundary = e->boundary_d;
    a.fv = e->fd.fv;
    a.fan_ptr = e->fd.fan_ptr;
    a.fan_walk = reinterpret_cast<const int2*>(e->fan_walk_d);
    a.farea_fx = e->farea_fx_d;
    a.area_unscale = e->area_unscale;
    a.total_area = e->lean_total;
    a.farea = e->farea_d;
    a.g11 = e->g11_d;
    a.g12 = e->g12_d;
    a.g22 = e->g22_d;
    a.width = e->mesh.bin_width;
    a.health_h = e->mesh.health_h;
    a.chord_slack = e->chord_slack;
    a.eps = eps;
    a.rtol = 1e-10;
    a.max_iter = 60;
    for (int32_t i = 0; i < nt; ++i) a.targets[i] = targets[i];
    for (int32_t j = 0; j < nb; ++j) a.fracs[j] = (double)(j + 1) / ((double)nb + 1.0);
    a.K = nsrc;
    a.vtile = fcw::stat_tile(e->sym.n, nsrc);
    a.ntiles = (int32_t)((e->sym.n + a.vtile - 1) / a.vtile);
    a.partials = e->cw().partials;
    a.near_list = e->cw().near_list;
    a.near_count = e->cw().near_count;
    {
        // near radius: a flat disc holding twice the largest reachable target, in whole bins.
        // A source first tries the cut of a flat disc holding the target itself plus four
        // bins (enough for most fields: the radius is two bins below the cut), then the
        // near radius, both from the near list.
        double tmax = 0.0;
        for (int32_t i = 0; i < nt; ++i)
            if (targets[i] > tmax && targets[i] <= e->lean_total) tmax = targets[i];
        const double pi = 3.141592653589793;
        a.near_bins = (int32_t)std::ceil(std::sqrt(2.0 * tmax / pi) / e->mesh.bin_width) + 2;
        a.near_radius = (double)a.near_bins * e->mesh.bin_width;
        a.first_bins = std::min(a.near_bins, (int32_t)std::ceil(std::sqrt(tmax / pi) / e->mesh.bin_width) + 4);
    }
    a.src = e->cw().src;
    a.band = e->cw().band;
    a.longf = e->cw().longf;
    a.out = e->cw().out;
    a.err = e->err_d;
    return FCW_OK;
}

template <typename T>
void metrics_block(fcw_engine* e, fcw::MetricArgs& a, const T* dT, cudaStream_t st) {
    mark(e, st, FCW_STAGE_METRICS);
    fcw::launch_source_metrics<T>(a, dT, st);
    mark(e, st, -1);
    e->launches += 1;
}

int check_engine(fcw_engine* e) {
    if (!e) return fail(FCW_E_INVALID, "engine is NULL");
    cudaError_t ce = cudaSetDevice(e->device);
    if (ce != cudaSuccess) return fail(FCW_E_CUDA, cudaGetErrorString(ce));
    return FCW_OK;
}

int check_sources(fcw_engine* e, const int32_t* sources, int64_t n) {
    for (int64_t k = 0; k < n; ++k)
        if (sources[k] < 0 || sources[k] >= e->sym.n)
            return fail(FCW_E_INVALID, "source_idx out of range: " + std::to_string(sources[k]) + " for mesh with " +
                                           std::to_string(e->sym.n) + " vertices");
    return FCW_OK;
}

// w.src and w.dst from the block's descriptor, or from n sources at `raw` (device; may be w.src).
void sort_sources(fcw_engine* e, Workspace& w, const fcw::BlockDesc* d, const int32_t* raw, int64_t n, int32_t K,
                  cudaStream_t st) {
    int32_t N = 2;
    while (N < K) N <<= 1;
    static_assert(kMaxSort * sizeof(unsigned long long) <= 48 * 1024, "the keys fit in default shared memory");
    k_sort_sources<<<1, std::min(kSortThreads, N / 2), N * sizeof(unsigned long long), st>>>(
        d, raw, n, e->iperm_d, (int32_t)e->sym.n, K, N, w.src, w.dst, e->err_d);
    e->launches += 1;
}

int32_t round_k(int64_t k) { return (int32_t)(((k + fcw::kRhsTile - 1) / fcw::kRhsTile) * fcw::kRhsTile); }

}  // namespace

namespace {

// Run `launch` (a chain of launches on w.stream) captured as a CUDA graph, once per
// workspace and key, and replayed after that; directly while graphs are off, the stage
// timeline is on, or the stream is already being captured by the caller.
template <class F>
int run_chain(fcw_engine* e, Workspace& w, const std::vector<double>& key, F&& launch) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    FCW_CUDA(cudaStreamIsCapturing(w.stream, &cs));
    if (!e->graphs_on || e->prof_on || cs != cudaStreamCaptureStatusNone) return launch();
    Workspace::Graph* hit = nullptr;
    for (auto& g : w.graphs)
        if (g.key == key) hit = &g;
    if (!hit) {
        constexpr size_t kMaxGraphs = 4;  // e.g. a full block and a call's last, partial one
        if (w.graphs.size() >= kMaxGraphs) {
            cudaGraphExecDestroy(w.graphs.front().exec);
            w.graphs.erase(w.graphs.begin());
        }
        const int64_t l0 = e->launches;
        FCW_CUDA(cudaStreamBeginCapture(w.stream, cudaStreamCaptureModeThreadLocal));
        const int lrc = launch();
        cudaGraph_t g = nullptr;
        cudaGraphExec_t exec = nullptr;
        cudaError_t ce = cudaStreamEndCapture(w.stream, &g);
        if (lrc != FCW_OK) {
            if (g) cudaGraphDestroy(g);
            e->launches = l0;
            return lrc;
        }
        if (ce == cudaSuccess) ce = cudaGraphInstantiate(&exec, g, 0);
        if (g) cudaGraphDestroy(g);
        const int64_t captured = e->launches - l0;  // kernels in the chain (counted when it runs)
        e->launches = l0;
        if (ce != cudaSuccess) {  // not capturable here: launch directly from now on
            cudaGetLastError();
            e->graphs_on = false;
            return launch();
        }
        w.graphs.push_back({key, exec, captured});
        hit = &w.graphs.back();
    }
    FCW_CUDA(cudaGraphLaunch(hit->exec, w.stream));
    e->launches += hit->launches;
    return FCW_OK;
}

}  // namespace

// ---------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------
extern "C" {

void fcw_default_params(fcw_params* p) {
    if (!p) return;
    p->diffusion_length_mm = 0.7;
    p->poisson_shift = 1e-10;
    p->block_k = 1024;
    p->leaf_size = 64;
    p->max_width = 64;
    p->relax = 64;
    p->build_mixed = 1;
    p->device = 0;
    p->pipeline_depth = 4;
    p->tc_sweeps = 0;
    p->robust = 0;
    p->refine = 0;
}

int fcw_metrics_stride(int32_t n_targets, int32_t n_between) {
    if (n_targets < 0 || n_between < 0) return 0;
    const int32_t ne = n_targets > 0 ? (n_targets - 1) * n_between : 0;
    return FCW_M_RADII + 2 * n_targets + 2 * ne;
}

int fcw_last_error(char* buf, size_t len) {
    if (buf && len) {
        std::strncpy(buf, g_err.c_str(), len - 1);
        buf[len - 1] = '\0';
    }
    return (int)g_err.size();
}

int fcw_mesh_arrays(const double* V, int64_t nv, const int32_t* F, int64_t nf, double* vertex_area,
                    double* lean_area, double* g11, double* g12, double* g22, uint8_t* boundary_flag) {
    if (!V || !F) return fail(FCW_E_INVALID, "vertices/faces is NULL");
    fcw::MeshPrep m;
    std::string err;
    if (fcw::prepare_mesh(V, nv, F, nf, m, err)) return fail(FCW_E_INVALID, err);
    if (vertex_area) std::memcpy(vertex_area, m.vertex_area.data(), nv * sizeof(double));
    if (lean_area) std::memcpy(lean_area, m.lean_area.data(), nf * sizeof(double));
    if (g11) std::memcpy(g11, m.g11.data(), nf * sizeof(double));
    if (g12) std::memcpy(g12, m.g12.data(), nf * sizeof(double));
    if (g22) std::memcpy(g22, m.g22.data(), nf * sizeof(double));
    if (boundary_flag) {
        std::memset(boundary_flag, 0, nv);
        for (int32_t b : m.boundary) boundary_flag[b] = 1;
    }
    return FCW_OK;
}

int fcw_analyze(const double* V, int64_t nv, const int32_t* F, int64_t nf, const fcw_params* params,
                fcw_info* info, int32_t* perm_out) {
    if (!V || !F) return fail(FCW_E_INVALID, "vertices/faces is NULL");
    FCW_TRY(validate_params(params));
    fcw::MeshPrep m;
    fcw::Symbolic S;
    std::string err;
    double t0 = now_ms();
    if (fcw::prepare_mesh(V, nv, F, nf, m, err)) return fail(FCW_E_INVALID, err);
    int64_t nflips = 0;
    if (params->robust && fcw::intrinsic_delaunay(m, kMollifyFactor, nflips, err)) return fail(FCW_E_INVALID, err);
    if (fcw::build_symbolic(m, params->leaf_size, params->max_width, params->relax, S, err)) return fail(FCW_E_INVALID, err);
    if (info) {
        std::memset(info, 0, sizeof(*info));
        info->n_vertices = nv;
        info->n_faces = nf;
        info->n_boundary = (int64_t)m.boundary.size();
        info->n_supernodes = S.nsuper;
        info->n_levels = S.nlevels;
        info->nnz_factor = S.nnz_factor;
        info->nnz_l = S.nnz_l;
        info->max_ns = S.max_ns;
        info->max_m = S.max_m;
        info->mean_edge_length = m.mean_edge;
        info->t_coef = std::pow(params->diffusion_length_mm / m.mean_edge, 2.0);
        info->t = info->t_coef * m.mean_edge * m.mean_edge;
        info->bin_width = m.bin_width;
        info->health_h = m.health_h;
        info->total_vertex_area = m.total_area;
        info->analyze_ms = now_ms() - t0;
        info->flops_factor = S.flops_factor;
        info->n_flips = nflips;
        std::vector<int32_t> comp;
        info->n_components = mesh_components(m, S.perm, comp);
    }
    if (perm_out) std::memcpy(perm_out, S.perm.data(), nv * sizeof(int32_t));
    return FCW_OK;
}

int fcw_intrinsic_operators(const double* V, int64_t nv, const int32_t* F, int64_t nf, int64_t* nflips, int64_t* nnz,
                            int64_t* Lp, int32_t* Li, double* Lx, double* mass, int32_t* tri, double* len,
                            int32_t* twin) {
    if (!V || !F) return fail(FCW_E_INVALID, "vertices/faces is NULL");
    fcw::MeshPrep m;
    std::string err;
    if (fcw::prepare_mesh(V, nv, F, nf, m, err)) return fail(FCW_E_INVALID, err);
    int64_t nfl = 0;
    if (fcw::intrinsic_delaunay(m, kMollifyFactor, nfl, err)) return fail(FCW_E_INVALID, err);
    if (nflips) *nflips = nfl;
    if (nnz) *nnz = (int64_t)m.Li.size();
    if (Lp) std::memcpy(Lp, m.Lp.data(), (nv + 1) * sizeof(int64_t));
    if (Li) std::memcpy(Li, m.Li.data(), m.Li.size() * sizeof(int32_t));
    if (Lx) std::memcpy(Lx, m.Lx.data(), m.Lx.size() * sizeof(double));
    if (mass) std::memcpy(mass, m.mass.data(), nv * sizeof(double));
    if (nfl > 0) {
        if (tri) std::memcpy(tri, m.itri.data(), m.itri.size() * sizeof(int32_t));
        if (len) std::memcpy(len, m.ilen.data(), m.ilen.size() * sizeof(double));
        if (twin) std::memcpy(twin, m.itwin.data(), m.itwin.size() * sizeof(int32_t));
    }
    return FCW_OK;
}

int fcw_engine_create(const double* V, int64_t nv, const int32_t* F, int64_t nf, const fcw_params* params,
                      fcw_engine** out) {
    if (!out) return fail(FCW_E_INVALID, "out is NULL");
    *out = nullptr;
    if (!V || !F) return fail(FCW_E_INVALID, "vertices/faces is NULL");
    FCW_TRY(validate_params(params));
    int ndev = 0;
    cudaError_t ce = cudaGetDeviceCount(&ndev);
    if (ce != cudaSuccess || ndev <= 0) {
        cudaGetLastError();
        return fail(FCW_E_NODEVICE, std::string("no CUDA device available: ") + cudaGetErrorString(ce));
    }
    if (params->device < 0 || params->device >= ndev) return fail(FCW_E_INVALID, "invalid device ordinal");
    fcw_engine* e = new fcw_engine();
    e->prm = *params;
    e->device = params->device;
    int rc = build_engine(e, V, nv, F, nf);
    if (rc == FCW_OK) rc = ensure_workspace(e, params->block_k, fcw_metrics_stride(12, 3));
    if (rc != FCW_OK) {
        std::string msg = g_err;
        delete e;
        g_err = msg;
        return rc;
    }
    *out = e;
    return FCW_OK;
}

int fcw_engine_info(const fcw_engine* e, fcw_info* info) {
    if (!e || !info) return fail(FCW_E_INVALID, "NULL argument");
    std::memset(info, 0, sizeof(*info));
    const auto& S = e->sym;
    const auto& m = e->mesh;
    info->n_vertices = m.nv;
    info->n_faces = m.nf;
    info->n_boundary = (int64_t)m.boundary.size();
    info->n_supernodes = S.nsuper;
    info->n_levels = S.nlevels;
    info->nnz_factor = S.nnz_factor;
    info->nnz_l = S.nnz_l;
    info->max_ns = S.max_ns;
    info->max_m = S.max_m;
    info->mean_edge_length = m.mean_edge;
    info->t_coef = e->t_coef;
    info->t = e->t;
    info->bin_width = m.bin_width;
    info->health_h = m.health_h;
    info->total_vertex_area = m.total_area;
    info->analyze_ms = e->analyze_ms;
    info->factor_ms = e->factor_ms;
    info->flops_factor = S.flops_factor;
    info->device_bytes = e->bytes;
    info->pipeline_depth = (int32_t)e->pool.size();
    info->block_k = e->prm.block_k;
    info->n_flips = e->n_flips;
    info->n_components = e->ncomp;
    return FCW_OK;
}

int fcw_engine_destroy(fcw_engine* e) {
    if (!e) return FCW_OK;
    cudaSetDevice(e->device);
    if (e->stream) cudaStreamSynchronize(e->stream);
    delete e;
    return FCW_OK;
}

int fcw_compute_distances(fcw_engine* e, const int32_t* sources, int64_t n, int32_t precision, double* out_host) {
    FCW_TRY(check_engine(e));
    if (n < 0 || (n > 0 && (!sources || !out_host))) return fail(FCW_E_INVALID, "NULL argument");
    if (precision == FCW_PREC_MIXED && !e->pan_gf) return fail(FCW_E_INVALID, "engine was built without the mixed form");
    const int32_t Kmax = e->prm.block_k;
    const int64_t nv = e->sym.n;
    FCW_TRY(check_sources(e, sources, n));
    for (int64_t b0 = 0; b0 < n; b0 += Kmax) {
        const int64_t nb = std::min<int64_t>(Kmax, n - b0);
        const int32_t K = round_k(nb);
        FCW_TRY(ensure_workspace(e, K, e->cw().out_stride));
        if (e->hdist_d && e->hcap_dist < nb * nv) {
            e->sync_streams();
            for (Workspace& w : e->pool) w.drop_graph();  // captured chains write the old buffer
        }
        FCW_TRY(e->grow(e->hdist_d, e->hcap_dist, nb * nv));
        Workspace& w = e->cw();
        FCW_CUDA(cudaMemcpyAsync(w.src, sources + b0, (size_t)nb * sizeof(int32_t), cudaMemcpyHostToDevice, w.stream));
        // the chain (solves, divergence, shift, fields back to the caller's order) as one graph
        const std::vector<double> key = {(double)K, (double)precision, -1.0, (double)nb};
        FCW_TRY(run_chain(e, w, key, [&]() -> int {
            sort_sources(e, w, nullptr, w.src, nb, K, w.stream);
            FCW_TRY(distances_block(e, K, precision, w.stream));
            const int grid = e->num_sms * 8;
            if (precision == FCW_PREC_MIXED)
                k_fields_out<float><<<grid, 256, 0, w.stream>>>((int32_t)nv, (int32_t)nb, w.dT32, e->iperm_d, w.dst,
                                                               e->hdist_d);
            else
                k_fields_out<double><<<grid, 256, 0, w.stream>>>((int32_t)nv, (int32_t)nb, w.dT64, e->iperm_d, w.dst,
                                                                e->hdist_d);
            e->launches += 1;
            return FCW_OK;
        }));
        FCW_CUDA(cudaGetLastError());
        FCW_CUDA(cudaMemcpyAsync(out_host + b0 * nv, e->hdist_d, (size_t)(nb * nv) * sizeof(double),
                                 cudaMemcpyDeviceToHost, w.stream));
        FCW_CUDA(cudaStreamSynchronize(w.stream));
        FCW_TRY(check_kernel_errors(e, "distances"));
    }
    return FCW_OK;
}

namespace {

// The drop-in's chain on st: the source's path, heat forward (the path's tasks) and
// backward, divergence, Poisson forward and backward, shift into the caller's order.
// Every sweep is one persistent ticketed launch. The source index is read from nar.src.
int narrow_chain(fcw_engine* e, cudaStream_t st) {
    NarrowState& q = e->nar;
    const int64_t n = e->sym.n;
    const int64_t nu = std::max<int64_t>(e->fr.n_urows, 1);
    double* U_h = q.pend;
    double* U_p = q.pend + nu;
    double* X_h = q.pend + 2 * nu;
    double* X_p = X_h + n;
    FCW_CUDA(cudaMemsetAsync(q.sync, 0, 4 * sizeof(int), st));
    FCW_CUDA(cudaMemsetAsync(q.pend, 0xFF, (size_t)(2 * nu + 2 * n) * sizeof(double), st));  // pending
    FCW_CUDA(cudaMemsetAsync(q.u, 0, (size_t)n * sizeof(double), st));
    fcw::NarrowArgs a;
    a.strip = q.L.strip;
    a.rec = reinterpret_cast<const int4*>(e->rec_d);
    a.rec_child = e->rec_child_d;
    a.more = e->more_d;
    a.rows = e->front_rows_d;
    a.err = e->err_d;
    // heat: the path's forward tasks, then the whole backward
    mark(e, st, FCW_STAGE_HEAT_FWD);
    a.at = q.at_h;
    a.B = q.u;
    a.U = U_h;
    a.tasks = q.ftasks;
    a.ntasks = q.n_ftasks;
    a.order = q.order;
    a.ticket = q.sync;
    fcw::launch_fwd_narrow(a, true, false, q.L, st);
    mark(e, st, FCW_STAGE_HEAT_BWD);
    a.at = q.atb_h;
    a.tasks = q.btasks;
    a.ntasks = q.n_btasks;
    a.X = X_h;
    a.ticket = q.sync + 1;
    fcw::launch_bwd_narrow(a, !e->prof_on, q.L, st);
    mark(e, st, FCW_STAGE_DIVERGENCE);
    fcw::launch_divergence_fp64_one(e->fd, X_h, q.div, st);
    // Poisson (L + shift M)
    mark(e, st, FCW_STAGE_POISSON_FWD);
    a.at = q.at_p;
    a.R = q.div;
    a.B = q.y;
    a.U = U_p;
    a.tasks = q.ftasks;
    a.ntasks = q.n_ftasks;
    a.order = nullptr;
    a.ticket = q.sync + 2;
    fcw::launch_fwd_narrow(a, false, !e->prof_on, q.L, st);
    mark(e, st, FCW_STAGE_POISSON_BWD);
    a.at = q.atb_p;
    a.tasks = q.btasks;
    a.ntasks = q.n_btasks;
    a.X = X_p;
    a.ticket = q.sync + 3;
    fcw::launch_bwd_narrow(a, !e->prof_on, q.L, st);
    mark(e, st, FCW_STAGE_SHIFT);
    fcw::launch_field_out_one((int32_t)n, X_p, q.order, e->iperm_d, q.out, e->num_sms, st);
    mark(e, st, -1);
    FCW_CUDA(cudaGetLastError());
    return FCW_OK;
}

int narrow_ready(fcw_engine* e) {
    NarrowState& q = e->nar;
    if (q.ready) return FCW_OK;
    const int64_t n = e->sym.n;
    int32_t max_ns = 1, max_m = 1;
    for (int32_t t = 0; t < e->fr.nf; ++t) {
        max_ns = std::max(max_ns, e->fr.c0[t + 1] - e->fr.c0[t]);
        max_m = std::max(max_m, e->fr.m[t]);
    }
    if (fcw::configure_narrow_kernels(max_ns, max_m, e->num_sms, &q.L) != cudaSuccess) {
        cudaGetLastError();
        return fail(FCW_E_INVALID, "front too large for the single-source kernels (" + std::to_string(max_m) + " rows)");
    }
    std::vector<fcw::NarrowTask> ft, bt;
    int64_t nfd = 0, nbd = 0;
    fcw::narrow_tasks(e->fr, ft, q.fwd_first, q.nfwd_h, bt, &nfd, &nbd);
    q.n_ftasks = (int32_t)ft.size();
    q.n_btasks = (int32_t)bt.size();
    FCW_TRY(e->upload(&q.ftasks, ft));
    FCW_TRY(e->upload(&q.btasks, bt));
    double* rows;
    FCW_TRY(e->dalloc(&rows, (size_t)e->frp.entries));
    for (int which = 0; which < 2; ++which) {
        double*& f = which ? q.at_p : q.at_h;
        double*& b = which ? q.atb_p : q.atb_h;
        FCW_TRY(e->dalloc(&f, (size_t)nfd));
        FCW_TRY(e->dalloc(&b, (size_t)nbd));
        fcw::launch_front_rows(e->plan, e->frp, which ? e->val_p : e->val_h, which ? e->inv_p : e->inv_h, rows, e->stream);
        fcw::launch_pack_narrow(e->frp, true, q.ftasks, q.n_ftasks, rows, f, e->stream);
        fcw::launch_pack_narrow(e->frp, false, q.btasks, q.n_btasks, rows, b, e->stream);
    }
    FCW_CUDA(cudaGetLastError());
    e->release(rows);
    FCW_TRY(e->dalloc(&q.u, (size_t)n));
    FCW_TRY(e->dalloc(&q.div, (size_t)n));
    FCW_TRY(e->dalloc(&q.y, (size_t)n));
    FCW_TRY(e->dalloc(&q.out, (size_t)n));
    FCW_TRY(e->dalloc(&q.pend, (size_t)(2 * std::max<int64_t>(e->fr.n_urows, 1) + 2 * n)));
    FCW_TRY(e->dalloc(&q.sync, 4));
    const size_t cap = 2 + 2 * (size_t)q.n_ftasks;
    FCW_TRY(e->dalloc(&q.order, cap));
    FCW_CUDA(cudaHostAlloc(&q.horder, cap * sizeof(int32_t), cudaHostAllocDefault));
    FCW_CUDA(cudaStreamSynchronize(e->stream));
    q.launches = 6;
    if (e->graphs_on) {
        FCW_CUDA(cudaStreamBeginCapture(e->stream, cudaStreamCaptureModeThreadLocal));
        const int lrc = narrow_chain(e, e->stream);
        cudaGraph_t g = nullptr;
        cudaError_t ce = cudaStreamEndCapture(e->stream, &g);
        if (lrc != FCW_OK) {
            if (g) cudaGraphDestroy(g);
            return lrc;
        }
        if (ce == cudaSuccess) ce = cudaGraphInstantiate(&q.exec, g, 0);
        if (g) cudaGraphDestroy(g);
        if (ce != cudaSuccess) {  // not capturable here: the chain launches directly
            cudaGetLastError();
            q.exec = nullptr;
        }
    }
    q.ready = true;
    return FCW_OK;
}

// The drop-in chain for one source (in range) on e->stream: its path's task list to the
// device, then the chain (the captured graph, or direct launches).
int narrow_run(fcw_engine* e, int32_t source) {
    FCW_TRY(narrow_ready(e));
    NarrowState& q = e->nar;
    cudaStream_t st = e->stream;
    // the source's path to the root, bottom-up, with each front's forward tasks
    int32_t* o = q.horder;
    int32_t len = 0, prev = -1;
    o[0] = e->sym.iperm[source];
    for (int32_t s = e->fr.col_front[o[0]]; s >= 0; prev = s, s = e->fr.parent[s])
        for (int32_t t = q.fwd_first[s]; t < q.fwd_first[s] + q.nfwd_h[s]; ++t) {
            o[2 + 2 * len] = t;
            o[3 + 2 * len] = prev;
            ++len;
        }
    o[1] = len;
    FCW_CUDA(cudaMemcpyAsync(q.order, o, (size_t)(2 + 2 * len) * sizeof(int32_t), cudaMemcpyHostToDevice, st));
    if (q.exec && e->graphs_on && !e->prof_on) FCW_CUDA(cudaGraphLaunch(q.exec, st));
    else FCW_TRY(narrow_chain(e, st));
    e->launches += q.launches;
    return FCW_OK;
}

// fcw_compute_metrics for one source in FP64: the drop-in chain, then the statistics and
// the per-source kernel at one column (records identical in meaning to the batched path's).
int narrow_metrics(fcw_engine* e, int32_t source, const double* targets, int32_t nt, int32_t nb, double eps,
                   double* out_host) {
    e->sync_streams();  // the workspace's metric scratch may still be in use by a device-API call
    const int32_t stride = fcw_metrics_stride(nt, nb);
    FCW_TRY(ensure_workspace(e, fcw::kRhsTile, stride));
    fcw::MetricArgs a;
    FCW_TRY(metric_args(e, targets, nt, nb, eps, 1, a));
    FCW_TRY(narrow_run(e, source));
    NarrowState& q = e->nar;
    cudaStream_t st = e->stream;
    const int64_t n = e->sym.n, nu = std::max<int64_t>(e->fr.n_urows, 1);
    const double* X_p = q.pend + 2 * nu + n;  // the Poisson solution (elimination order)
    a.src = q.order;                           // its first entry: the source's elimination index
    fcw::launch_shift_stats_one(a, X_p, e->cw().dT64, st);
    fcw::launch_source_metrics<double>(a, e->cw().dT64, st);
    e->launches += 2;
    FCW_CUDA(cudaGetLastError());
    FCW_CUDA(cudaMemcpyAsync(out_host, a.out, (size_t)stride * sizeof(double), cudaMemcpyDeviceToHost, st));
    return check_kernel_errors(e, "metrics");
}

}  // namespace

int fcw_compute_distance(fcw_engine* e, int32_t source, double* out_host) {
    FCW_TRY(check_engine(e));
    if (!out_host) return fail(FCW_E_INVALID, "NULL argument");
    if (source < 0 || source >= e->sym.n)
        return fail(FCW_E_INVALID, "source_idx out of range: " + std::to_string(source) + " for mesh with " +
                                       std::to_string(e->sym.n) + " vertices");
    FCW_TRY(narrow_run(e, source));
    NarrowState& q = e->nar;
    cudaStream_t st = e->stream;
    FCW_CUDA(cudaMemcpyAsync(out_host, q.out, (size_t)e->sym.n * sizeof(double), cudaMemcpyDeviceToHost, st));
    return check_kernel_errors(e, "distance");
}

namespace {

// One block's launch chain on workspace w, its inputs in w.desc: source mapping,
// distances, metrics. With graphs on (and the stage timeline off) the chain is
// captured once per workspace and set of arguments, and replayed for later blocks.
int block_chain(fcw_engine* e, Workspace& w, int32_t K, int32_t precision, fcw::MetricArgs& a,
                const double* targets, int32_t nt, int32_t nb, double eps) {
    auto launch = [&]() -> int {
        sort_sources(e, w, w.desc, nullptr, 0, K, w.stream);
        const int rc = distances_block(e, K, precision, w.stream, &a);
        if (rc != FCW_OK) return rc;
        if (precision == FCW_PREC_MIXED) metrics_block<float>(e, a, w.dT32, w.stream);
        else metrics_block<double>(e, a, w.dT64, w.stream);
        return FCW_OK;
    };
    std::vector<double> key = {(double)K, (double)precision, (double)nt, (double)nb, eps};
    key.insert(key.end(), targets, targets + nt);
    return run_chain(e, w, key, launch);
}

}  // namespace

int fcw_compute_metrics_device(fcw_engine* e, const int32_t* sources_dev, int64_t n, int32_t precision,
                               const double* targets, int32_t nt, int32_t nb, double eps, double* out_dev,
                               void* stream) {
    FCW_TRY(check_engine(e));
    if (n < 0 || (n > 0 && (!sources_dev || !out_dev))) return fail(FCW_E_INVALID, "NULL argument");
    if (precision == FCW_PREC_MIXED && !e->pan_gf) return fail(FCW_E_INVALID, "engine was built without the mixed form");
    if (n == 0) return FCW_OK;
    cudaStream_t user = static_cast<cudaStream_t>(stream);
    const int32_t stride = fcw_metrics_stride(nt, nb);
    const int32_t Kmax = e->prm.block_k;
    FCW_TRY(ensure_workspace(e, std::min<int64_t>(round_k(n), Kmax), stride));
    // Blocks of K sources round-robin over the workspace pool, each workspace on its own
    // stream, so independent blocks overlap. The pool streams start after the caller's
    // stream reaches this call, and the caller's stream waits for all of them at the end.
    const size_t depth = e->pool.size();
    FCW_CUDA(cudaEventRecord(e->ev_in, user));
    size_t used = 0;
    int rc = FCW_OK;
    for (int64_t b0 = 0, blk = 0; b0 < n && rc == FCW_OK; b0 += Kmax, ++blk) {
        const int64_t nbk = std::min<int64_t>(Kmax, n - b0);
        const int32_t K = round_k(nbk);
        e->cur_ws = (size_t)blk % depth;
        Workspace& w = e->cw();
        if (blk < (int64_t)depth) {
            FCW_CUDA(cudaStreamWaitEvent(w.stream, e->ev_in, 0));
            used = (size_t)blk + 1;
        }
        fcw::MetricArgs a;
        rc = metric_args(e, targets, nt, nb, eps, K, a);
        if (rc != FCW_OK) break;
        a.desc = w.desc;
        a.dst = w.dst;
        k_set_block<<<1, 1, 0, w.stream>>>(w.desc, sources_dev + b0, nbk, out_dev + b0 * stride);
        e->launches += 1;
        rc = block_chain(e, w, K, precision, a, targets, nt, nb, eps);
    }
    for (size_t i = 0; i < used; ++i) {
        FCW_CUDA(cudaEventRecord(e->pool[i].done, e->pool[i].stream));
        FCW_CUDA(cudaStreamWaitEvent(user, e->pool[i].done, 0));
    }
    e->cur_ws = 0;
    if (rc != FCW_OK) return rc;
    FCW_CUDA(cudaGetLastError());
    return FCW_OK;
}

int fcw_compute_metrics(fcw_engine* e, const int32_t* sources, int64_t n, int32_t precision, const double* targets,
                        int32_t nt, int32_t nb, double eps, double* out_host) {
    FCW_TRY(check_engine(e));
    if (n < 0 || (n > 0 && (!sources || !out_host))) return fail(FCW_E_INVALID, "NULL argument");
    if (n == 0) return FCW_OK;
    FCW_TRY(check_sources(e, sources, n));
    if (n == 1 && precision == FCW_PREC_FP64) return narrow_metrics(e, sources[0], targets, nt, nb, eps, out_host);
    const int32_t stride = fcw_metrics_stride(nt, nb);
    FCW_TRY(e->grow(e->hsrc_d, e->hcap_src, n));
    FCW_TRY(e->grow(e->hout_d, e->hcap_out, n * stride));
    FCW_CUDA(cudaMemcpyAsync(e->hsrc_d, sources, n * sizeof(int32_t), cudaMemcpyHostToDevice, e->stream));
    FCW_TRY(fcw_compute_metrics_device(e, e->hsrc_d, n, precision, targets, nt, nb, eps, e->hout_d, e->stream));
    FCW_CUDA(cudaMemcpyAsync(out_host, e->hout_d, n * stride * sizeof(double), cudaMemcpyDeviceToHost, e->stream));
    return check_kernel_errors(e, "metrics");
}

int fcw_samples_capacity(int32_t n_targets, int32_t n_between) {
    if (n_targets < 0 || n_between < 0) return 0;
    return n_targets + (n_targets > 0 ? (n_targets - 1) * n_between : 0);
}

namespace {

int sample_args(const double* records, int64_t n, int32_t nt, int32_t nb, const double* targets, double cap,
                float* radii, float* areas, int32_t* count, fcw::SampleArgs& a) {
    if (nt < 1 || nt > fcw::kMaxTargets) return fail(FCW_E_INVALID, "n_targets must be in [1, 32]");
    if (nb < 0 || nb > fcw::kMaxBetween) return fail(FCW_E_INVALID, "n_between must be in [0, 8]");
    if (!targets) return fail(FCW_E_INVALID, "targets is NULL");
    if (!std::isnan(cap) && !(cap >= 0.0 && cap < 0.5))
        return fail(FCW_E_INVALID, "boundary_cap must be in [0, 0.5), or NaN for no cap");
    if (n < 0 || (n > 0 && (!records || !radii || !areas || !count))) return fail(FCW_E_INVALID, "NULL argument");
    a = fcw::SampleArgs{};
    a.n = n;
    a.n_targets = nt;
    a.n_between = nb;
    a.stride = fcw_metrics_stride(nt, nb);
    a.capacity = fcw_samples_capacity(nt, nb);
    for (int32_t i = 0; i < nt; ++i) a.targets[i] = targets[i];
    a.cap = cap;
    a.records = records;
    a.radii_out = radii;
    a.areas_out = areas;
    a.count_out = count;
    return FCW_OK;
}

}  // namespace

int fcw_assemble_samples_device(const double* records_dev, int64_t n, int32_t n_targets, int32_t n_between,
                                const double* targets, double boundary_cap, float* radii_out, float* areas_out,
                                int32_t* count_out, void* stream) {
    fcw::SampleArgs a;
    FCW_TRY(sample_args(records_dev, n, n_targets, n_between, targets, boundary_cap, radii_out, areas_out, count_out,
                        a));
    if (n == 0) return FCW_OK;
    fcw::launch_assemble_samples(a, static_cast<cudaStream_t>(stream));
    FCW_CUDA(cudaGetLastError());
    return FCW_OK;
}

int fcw_assemble_samples(fcw_engine* e, const double* records, int64_t n, int32_t n_targets, int32_t n_between,
                         const double* targets, double boundary_cap, float* radii, float* areas, int32_t* count) {
    FCW_TRY(check_engine(e));
    fcw::SampleArgs a;
    FCW_TRY(sample_args(records, n, n_targets, n_between, targets, boundary_cap, radii, areas, count, a));
    if (n == 0) return FCW_OK;
    const int64_t stride = a.stride, cap = a.capacity;
    FCW_TRY(e->grow(e->hout_d, e->hcap_out, n * stride));
    FCW_TRY(e->grow(e->hsr_d, e->hcap_sr, n * cap));
    FCW_TRY(e->grow(e->hsa_d, e->hcap_sa, n * cap));
    FCW_TRY(e->grow(e->hcnt_d, e->hcap_cnt, n));
    FCW_CUDA(cudaMemcpyAsync(e->hout_d, records, n * stride * sizeof(double), cudaMemcpyHostToDevice, e->stream));
    a.records = e->hout_d;
    a.radii_out = e->hsr_d;
    a.areas_out = e->hsa_d;
    a.count_out = e->hcnt_d;
    fcw::launch_assemble_samples(a, e->stream);
    FCW_CUDA(cudaGetLastError());
    FCW_CUDA(cudaMemcpyAsync(radii, e->hsr_d, n * cap * sizeof(float), cudaMemcpyDeviceToHost, e->stream));
    FCW_CUDA(cudaMemcpyAsync(areas, e->hsa_d, n * cap * sizeof(float), cudaMemcpyDeviceToHost, e->stream));
    FCW_CUDA(cudaMemcpyAsync(count, e->hcnt_d, n * sizeof(int32_t), cudaMemcpyDeviceToHost, e->stream));
    FCW_CUDA(cudaStreamSynchronize(e->stream));
    return FCW_OK;
}

// The maps of up to kMapChunk sources at a time pass through page-locked staging (8.0 MB at 12 scales
// and 3 samples between): records never leave the device, and the host only scatters float32 values.
int fcw_compute_wiring(fcw_engine* e, const int32_t* sources, int64_t n, int32_t precision, const double* targets,
                       int32_t nt, int32_t nb, double eps, double boundary_cap, const int32_t* vertices, int64_t n_full,
                       float* maps, uint8_t* flags, double* health, float* radii, float* areas, int32_t* counts) {
    FCW_TRY(check_engine(e));
    constexpr int64_t kMapChunk = 16384;
    if (n < 0 || n_full < 0 || (n > 0 && (!sources || !vertices || !maps || !flags || !health)))
        return fail(FCW_E_INVALID, "NULL argument");
    fcw::SampleArgs sa;
    FCW_TRY(sample_args(reinterpret_cast<const double*>(sources), n, nt, nb, targets, boundary_cap, radii, areas,
                        counts, sa));
    FCW_TRY(check_sources(e, sources, n));
    for (int64_t k = 0; k < n; ++k)
        if (vertices[k] < 0 || vertices[k] >= n_full) return fail(FCW_E_INVALID, "vertex out of range");
    const int64_t stride = sa.stride, cap = sa.capacity, cols = 3 + 2 * (int64_t)nt;
    const int64_t per = 2 * (int64_t)sizeof(double) + (cols + 2 * cap) * (int64_t)sizeof(float) + (int64_t)sizeof(int32_t) + 1;
    for (int64_t b0 = 0; b0 < n; b0 += kMapChunk) {
        const int64_t m = std::min(kMapChunk, n - b0), bytes = m * per;
        FCW_TRY(e->grow(e->hsrc_d, e->hcap_src, m));
        FCW_TRY(e->grow(e->hout_d, e->hcap_out, m * stride));
        FCW_TRY(e->grow(e->hmap_d, e->hcap_map_d, bytes));
        FCW_TRY(e->grow_host(e->hmap_h, e->hcap_map_h, bytes));
        // health (2m doubles), maps, sample rows, counts, flags
        auto at = [&](unsigned char* base, int part) {
            const int64_t off[] = {0, 16 * m, 16 * m + 4 * cols * m, 16 * m + 4 * (cols + cap) * m,
                                   16 * m + 4 * (cols + 2 * cap) * m, 16 * m + 4 * (cols + 2 * cap + 1) * m};
            return base + off[part];
        };
        cudaStream_t st = e->stream;
        FCW_CUDA(cudaMemcpyAsync(e->hsrc_d, sources + b0, m * sizeof(int32_t), cudaMemcpyHostToDevice, st));
        FCW_TRY(fcw_compute_metrics_device(e, e->hsrc_d, m, precision, targets, nt, nb, eps, e->hout_d, st));
        sa.n = m;
        sa.records = e->hout_d;
        sa.radii_out = reinterpret_cast<float*>(at(e->hmap_d, 2));
        sa.areas_out = reinterpret_cast<float*>(at(e->hmap_d, 3));
        sa.count_out = reinterpret_cast<int32_t*>(at(e->hmap_d, 4));
        fcw::launch_assemble_samples(sa, st);
        fcw::launch_pack_maps(e->hout_d, m, (int32_t)stride, nt, reinterpret_cast<float*>(at(e->hmap_d, 1)),
                              at(e->hmap_d, 5), reinterpret_cast<double*>(at(e->hmap_d, 0)), st);
        FCW_CUDA(cudaGetLastError());
        FCW_CUDA(cudaMemcpyAsync(e->hmap_h, e->hmap_d, (size_t)bytes, cudaMemcpyDeviceToHost, st));
        FCW_TRY(check_kernel_errors(e, "metrics"));
        const float* col = reinterpret_cast<const float*>(at(e->hmap_h, 1));
        const unsigned char* flag = at(e->hmap_h, 5);
        const int32_t* v = vertices + b0;
        for (int64_t k = 0; k < m; ++k) flags[v[k]] = flag[k];
        for (int64_t c = 0; c < cols; ++c) {
            float* o = maps + c * n_full;
            for (int64_t k = 0; k < m; ++k)
                if (!flag[k]) o[v[k]] = col[c * m + k];
        }
        const double* h = reinterpret_cast<const double*>(at(e->hmap_h, 0));
        std::memcpy(health + b0, h, m * sizeof(double));
        std::memcpy(health + n + b0, h + m, m * sizeof(double));
        std::memcpy(radii + b0 * cap, at(e->hmap_h, 2), (size_t)(m * cap) * sizeof(float));
        std::memcpy(areas + b0 * cap, at(e->hmap_h, 3), (size_t)(m * cap) * sizeof(float));
        std::memcpy(counts + b0, at(e->hmap_h, 4), m * sizeof(int32_t));
    }
    return FCW_OK;
}

int fcw_pack_rows(const float* rows, int64_t n, int64_t capacity, const int32_t* counts, const int64_t* first,
                  float* flat) {
    if (n < 0 || capacity < 0 || (n > 0 && (!rows || !counts || !first || !flat))) return fail(FCW_E_INVALID, "NULL argument");
    for (int64_t k = 0; k < n; ++k) {
        if (counts[k] < 0 || counts[k] > capacity) return fail(FCW_E_INVALID, "row count out of range");
        std::memcpy(flat + first[k], rows + k * capacity, (size_t)counts[k] * sizeof(float));
    }
    return FCW_OK;
}

int fcw_engine_graphs(fcw_engine* e, int enable) {
    FCW_TRY(check_engine(e));
    e->graphs_on = enable != 0;
    return FCW_OK;
}

int fcw_engine_profile(fcw_engine* e, int enable) {
    FCW_TRY(check_engine(e));
    FCW_TRY(collect_marks(e));
    e->prof_on = enable != 0;
    for (double& x : e->stage_ms) x = 0.0;
    e->launches = 0;
    return FCW_OK;
}

int fcw_engine_stage_times(fcw_engine* e, double* ms_out, int32_t n, int64_t* launches) {
    FCW_TRY(check_engine(e));
    FCW_TRY(collect_marks(e));
    for (int32_t i = 0; i < n && i < FCW_N_STAGES; ++i) ms_out[i] = e->stage_ms[i];
    if (launches) *launches = e->launches;
    return FCW_OK;
}

int fcw_synchronize(fcw_engine* e, void* stream) {
    FCW_TRY(check_engine(e));
    FCW_CUDA(cudaStreamSynchronize(static_cast<cudaStream_t>(stream)));
    return check_kernel_errors(e, "device call");
}

int fcw_heat_solve_device(fcw_engine* e, const int32_t* sources_dev, int32_t k, double* u_dev, void* stream) {
    FCW_TRY(check_engine(e));
    if (k <= 0 || !sources_dev || !u_dev) return fail(FCW_E_INVALID, "invalid arguments");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int32_t K = round_k(k);
    FCW_TRY(ensure_workspace(e, K, e->cw().out_stride));
    k_map_sources<<<(K + 127) / 128, 128, 0, st>>>(k, sources_dev, e->iperm_d, (int32_t)e->sym.n, K, e->cw().src,
                                                   e->err_d);
    heat_solve(e, K, st);
    // u_dev[old][c] = Bh[iperm[old]][c]
    fcw::launch_permute_rows((int32_t)e->sym.n, k, e->cw().Bh, K, e->iperm_d, u_dev, k, nullptr, st);
    FCW_CUDA(cudaGetLastError());
    return FCW_OK;
}

int fcw_divergence_device(fcw_engine* e, const double* u_dev, int32_t k, double* div_dev, void* stream) {
    FCW_TRY(check_engine(e));
    if (k <= 0 || !u_dev || !div_dev) return fail(FCW_E_INVALID, "invalid arguments");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int32_t K = round_k(k);
    FCW_TRY(ensure_workspace(e, K, e->cw().out_stride));
    FCW_CUDA(cudaMemsetAsync(e->cw().Bh, 0, (size_t)e->sym.n * K * sizeof(double), st));
    fcw::launch_permute_rows((int32_t)e->sym.n, k, u_dev, k, nullptr, e->cw().Bh, K, e->iperm_d, st);
    fcw::launch_divergence_fp64(e->fd, e->cw().Bh, reinterpret_cast<double*>(e->cw().band), e->cw().Bp64, K, st);
    fcw::launch_permute_rows((int32_t)e->sym.n, k, e->cw().Bp64, K, e->iperm_d, div_dev, k, nullptr, st);
    FCW_CUDA(cudaGetLastError());
    return FCW_OK;
}

int fcw_poisson_solve_device(fcw_engine* e, const double* div_dev, const int32_t* sources_dev, int32_t k,
                             double* phi_dev, void* stream) {
    FCW_TRY(check_engine(e));
    if (k <= 0 || !div_dev || !sources_dev || !phi_dev) return fail(FCW_E_INVALID, "invalid arguments");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int32_t K = round_k(k);
    FCW_TRY(ensure_workspace(e, K, e->cw().out_stride));
    k_map_sources<<<(K + 127) / 128, 128, 0, st>>>(k, sources_dev, e->iperm_d, (int32_t)e->sym.n, K, e->cw().src,
                                                   e->err_d);
    FCW_CUDA(cudaMemsetAsync(e->cw().Bp64, 0, (size_t)e->sym.n * K * sizeof(double), st));
    fcw::launch_permute_rows((int32_t)e->sym.n, k, div_dev, k, nullptr, e->cw().Bp64, K, e->iperm_d, st);
    FCW_TRY(poisson_solve<double>(e, e->pan_pf, e->pan_pb, e->cw().Bp64, e->cw().Y, K, st));
    fcw::launch_shift_transpose<double, double>((int32_t)e->sym.n, K, e->cw().Y, e->cw().src, e->cw().dT64, st);
    // phi_dev[old][c] = dT[c][iperm[old]]: transpose back through the permute kernel, column by column
    for (int32_t c = 0; c < k; ++c)
        fcw::launch_permute_rows((int32_t)e->sym.n, 1, e->cw().dT64 + (int64_t)c * e->sym.n, 1, e->iperm_d,
                                 phi_dev + c, k, nullptr, st);
    FCW_CUDA(cudaGetLastError());
    return FCW_OK;
}

int fcw_field_metrics_device(fcw_engine* e, const double* d_dev, const int32_t* sources_dev, int32_t k,
                             const double* targets, int32_t nt, int32_t nb, double eps, double* out_dev,
                             void* stream) {
    FCW_TRY(check_engine(e));
    if (k <= 0 || !d_dev || !sources_dev || !out_dev) return fail(FCW_E_INVALID, "invalid arguments");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int32_t K = round_k(k);
    const int32_t stride = fcw_metrics_stride(nt, nb);
    FCW_TRY(ensure_workspace(e, K, stride));
    fcw::MetricArgs a;
    FCW_TRY(metric_args(e, targets, nt, nb, eps, K, a));
    a.out = out_dev;
    k_map_sources<<<(K + 127) / 128, 128, 0, st>>>(k, sources_dev, e->iperm_d, (int32_t)e->sym.n, K, e->cw().src,
                                                   e->err_d);
    k_fields_in<<<e->num_sms * 8, 256, 0, st>>>((int32_t)e->sym.n, k, K, d_dev, e->iperm_d, e->cw().Y);
    mark(e, st, FCW_STAGE_SHIFT);
    fcw::launch_shift_stats<double, double>(a, K, e->cw().Y, e->cw().dT64, st);
    e->launches += 3;
    metrics_block<double>(e, a, e->cw().dT64, st);
    FCW_CUDA(cudaGetLastError());
    return FCW_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Allocation-free field metrics
//
// For callers that may not allocate device memory once they are running: a host
// that reserves the whole device up front for its own pool, or a measurement or
// serving loop that must keep its device footprint fixed. This entry point runs
// the same kernels as fcw_field_metrics_device, but every buffer it needs beyond
// the caller's inputs and outputs (and the engine's own arrays, allocated when
// the engine was created) comes from one fixed array compiled into the library.
// ---------------------------------------------------------------------------
namespace {

// Per-call scratch for fcw_field_metrics_static. Every device that loads this
// library holds these bytes until the process exits.
constexpr size_t kStaticScratchBytes = 64u << 20;
constexpr int32_t kStaticMaxFields = 32;
static __device__ __align__(256) unsigned char g_field_scratch[kStaticScratchBytes];

// The array's device address, looked up once per device. In host code the name
// g_field_scratch only stands in for the symbol; it is not a device pointer.
constexpr int kMaxDevices = 64;
void* g_field_scratch_addr[kMaxDevices] = {nullptr};
std::mutex g_field_scratch_mutex;

int static_scratch_address(int device, unsigned char** out) {
    if (device < 0 || device >= kMaxDevices) return fail(FCW_E_INVALID, "device ordinal out of range");
    std::lock_guard<std::mutex> lock(g_field_scratch_mutex);
    if (!g_field_scratch_addr[device]) {
        void* p = nullptr;
        const cudaError_t rc = cudaGetSymbolAddress(&p, g_field_scratch);  // the engine's device is current
        if (rc != cudaSuccess || p == nullptr) {
            cudaGetLastError();
            return fail(FCW_E_CUDA, std::string("cudaGetSymbolAddress(static field scratch) failed: ") +
                                        cudaGetErrorString(rc));
        }
        g_field_scratch_addr[device] = p;
    }
    *out = static_cast<unsigned char*>(g_field_scratch_addr[device]);
    return FCW_OK;
}

size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

}  // namespace

extern "C" int fcw_field_metrics_static(fcw_engine* e, const double* d_dev, const int32_t* sources_dev, int32_t k,
                                        const double* targets, int32_t nt, int32_t nb, double eps, double* out_dev,
                                        void* stream) {
    FCW_TRY(check_engine(e));
    if (k <= 0 || !d_dev || !sources_dev || !out_dev) return fail(FCW_E_INVALID, "invalid arguments");
    if (k > kStaticMaxFields)
        return fail(FCW_E_INVALID, "fcw_field_metrics_static takes at most " + std::to_string(kStaticMaxFields) +
                                       " fields per call, got " + std::to_string(k));
    const int32_t K = 32;  // one 32-column tile of the shift kernel; columns >= k are padding
    const int64_t n = e->sym.n, nf = e->mesh.nf;
    const int64_t ntiles = (n + fcw::kStatVTile - 1) / fcw::kStatVTile;
    const size_t need = align256((size_t)n * K * sizeof(double))          // vertex-major fields
                        + align256((size_t)n * K * sizeof(double))        // shifted, one field per row
                        + align256((size_t)ntiles * K * 8 * sizeof(double))  // health/MSD partials
                        + align256((size_t)n * K * sizeof(int32_t))       // near-vertex lists
                        + align256((size_t)K * sizeof(int32_t))           // near-vertex counts
                        + align256((size_t)nf * K * sizeof(int4))         // near faces by bin
                        + align256((size_t)nf * K * sizeof(int32_t))      // long faces
                        + align256((size_t)K * sizeof(int32_t));          // sources (elimination order)
    if (need > kStaticScratchBytes)
        return fail(FCW_E_INVALID, "mesh too large for fcw_field_metrics_static: needs " + std::to_string(need) +
                                       " bytes of scratch, the static array holds " +
                                       std::to_string(kStaticScratchBytes));
    unsigned char* base = nullptr;
    FCW_TRY(static_scratch_address(e->device, &base));
    size_t off = 0;
    auto take = [&](size_t bytes) {
        unsigned char* p = base + off;
        off += align256(bytes);
        return p;
    };
    double* Y = reinterpret_cast<double*>(take((size_t)n * K * sizeof(double)));
    double* dT = reinterpret_cast<double*>(take((size_t)n * K * sizeof(double)));
    double* partials = reinterpret_cast<double*>(take((size_t)ntiles * K * 8 * sizeof(double)));
    int32_t* near_list = reinterpret_cast<int32_t*>(take((size_t)n * K * sizeof(int32_t)));
    int32_t* near_count = reinterpret_cast<int32_t*>(take((size_t)K * sizeof(int32_t)));
    int4* band = reinterpret_cast<int4*>(take((size_t)nf * K * sizeof(int4)));
    int32_t* longf = reinterpret_cast<int32_t*>(take((size_t)nf * K * sizeof(int32_t)));
    int32_t* src = reinterpret_cast<int32_t*>(take((size_t)K * sizeof(int32_t)));

    cudaStream_t st = static_cast<cudaStream_t>(stream);
    fcw::MetricArgs a;
    FCW_TRY(metric_args(e, targets, nt, nb, eps, K, a));
    a.vtile = fcw::kStatVTile;
    a.ntiles = (int32_t)ntiles;
    a.src = src;
    a.band = band;
    a.longf = longf;
    a.partials = partials;
    a.near_list = near_list;
    a.near_count = near_count;  // cleared by launch_shift_stats before the shift kernel
    a.out = out_dev;
    k_map_sources<<<1, 128, 0, st>>>(k, sources_dev, e->iperm_d, (int32_t)n, K, src, e->err_d);
    k_fields_in<<<e->num_sms * 8, 256, 0, st>>>((int32_t)n, k, K, d_dev, e->iperm_d, Y);
    mark(e, st, FCW_STAGE_SHIFT);
    fcw::launch_shift_stats<double, double>(a, K, Y, dT, st);
    e->launches += 3;
    mark(e, st, FCW_STAGE_METRICS);
    fcw::launch_source_metrics<double>(a, dT, st);
    mark(e, st, -1);
    e->launches += 1;
    FCW_CUDA(cudaGetLastError());
    return FCW_OK;
}
