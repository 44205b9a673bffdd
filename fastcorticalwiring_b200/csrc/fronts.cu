// The sweeps' panels from the factorisation's supernode blocks (fronts.cpp plans them).
//
// Over a front's columns, split in the blocks 1..p of its supernodes, L^-1 = D T and
// L_rs L_ss^-1 = Q T with D the blocks' inverses, Q the supernodes' panels (Q_ik = L_ik L_kk^-1)
// and T = (I + strict(Q))^-1. T(I + strict(Q)) = I gives each row a of [inv(L_ss); Q_s] from the
// last block to the first, independently of the other rows:
//   a_j = base_j - sum_{k > j} a_k Q_kj,   base = the row of [D; Q's structure rows].
// The rows are formed in FP64 once per factor and then copied into the order the sweeps read:
// one k-major block per task (SweepTask), rounded to FP32 for the mixed form's Poisson factor.
#include <algorithm>

#include "kernels.cuh"

namespace fcw {

namespace {

constexpr int kRowGroup = 8;  // rows per CTA of k_merge_rows

// base: the supernodes' inverse blocks and structure rows into their front's m x ns rows (zeroed)
__global__ void k_scatter_blocks(DevPlan p, FrontPlan f, const double* __restrict__ val,
                                 const double* __restrict__ inv, double* __restrict__ rows) {
    const int s = blockIdx.x, t = f.sn_front[s];
    const int cs = p.sn_c0[s] - f.c0[t], ws = p.sn_c0[s + 1] - p.sn_c0[s], m = p.sn_m[s];
    const int ns = f.c0[t + 1] - f.c0[t];
    const double* V = val + p.sn_valptr[s];
    const double* I = inv + p.sn_invptr[s];
    double* o = rows + f.ptr[t];
    const int32_t* pos = f.pos + p.sn_rowptr[s];
    for (int e = threadIdx.x; e < m * ws; e += blockDim.x) {
        const int q = e / ws, j = e - q * ws;
        if (q < ws) {
            if (j <= q) o[(int64_t)(cs + q) * ns + cs + j] = I[q * ws + j];
        } else if (pos[q] >= ns) {
            o[(int64_t)pos[q] * ns + cs + j] = V[(int64_t)q * ws + j];
        }
    }
}

// rows [kRowGroup y, ...) of a front of several supernodes: a_j -= sum a_k Q_kj, blocks last to first
__global__ void __launch_bounds__(256) k_merge_rows(DevPlan p, FrontPlan f, const int32_t* __restrict__ fronts,
                                                    const double* __restrict__ val, double* __restrict__ rows) {
    extern __shared__ double a[];  // kRowGroup x ns
    const int t = fronts[blockIdx.x];
    const int ns = f.c0[t + 1] - f.c0[t], m = f.m[t];
    const int r0 = blockIdx.y * kRowGroup, nr = min(kRowGroup, m - r0);
    if (nr <= 0) return;
    double* o = rows + f.ptr[t] + (int64_t)r0 * ns;
    for (int e = threadIdx.x; e < kRowGroup * ns; e += blockDim.x) a[e] = e < nr * ns ? o[e] : 0.0;
    __syncthreads();
    const int c = threadIdx.x & 63, rg = threadIdx.x >> 6;  // 4 row groups of 2
    for (int s = f.sn0[t + 1] - 2; s >= f.sn0[t]; --s) {
        const int cs = p.sn_c0[s] - f.c0[t], ws = p.sn_c0[s + 1] - p.sn_c0[s], ms = p.sn_m[s];
        const double* V = val + p.sn_valptr[s];
        const int32_t* pos = f.pos + p.sn_rowptr[s];
        double x0 = 0.0, x1 = 0.0;
        if (c < ws)
            for (int q = ws; q < ms; ++q) {
                const int k = pos[q];
                if (k >= ns) break;  // the front's columns come first
                const double v = V[(int64_t)q * ws + c];
                x0 = fma(a[(2 * rg) * ns + k], v, x0);
                x1 = fma(a[(2 * rg + 1) * ns + k], v, x1);
            }
        // the block's own entries are read by no other thread before the barrier
        if (c < ws) {
            a[(2 * rg) * ns + cs + c] -= x0;
            a[(2 * rg + 1) * ns + cs + c] -= x1;
        }
        __syncthreads();
    }
    for (int e = threadIdx.x; e < nr * ns; e += blockDim.x) o[e] = a[e];
}

// One task's panel: forward, element (row r, column j) at j * ld + r; backward, (front row r0 + d,
// column r0 + c) at d * ld + c, the structure rows negated. Padding is zero.
template <typename T, bool FWD>
__global__ void k_pack(FrontPlan f, const SweepTask* __restrict__ tasks, const double* __restrict__ rows,
                       T* __restrict__ out) {
    const SweepTask t = tasks[blockIdx.x];
    const int ns = t.ns, ld = (t.h + 7) / 8 * 8 + (sizeof(T) == 8 ? 4 : 0);
    const int dp = (t.depth + kDepthPad - 1) / kDepthPad * kDepthPad;
    T* o = out + (sizeof(T) == 8 ? t.off64 : t.off32);
    const double* in = rows + f.ptr[t.front];
    for (int e = threadIdx.x; e < dp * ld; e += blockDim.x) {
        const int d = e / ld, r = e - d * ld;
        double v = 0.0;
        if (d < t.depth && r < t.h) {
            if (FWD) v = in[(int64_t)(t.r0 + r) * ns + d];
            else v = in[(int64_t)(t.r0 + d) * ns + t.r0 + r] * (t.r0 + d < ns ? 1.0 : -1.0);
        }
        o[e] = (T)v;
    }
}

}  // namespace

cudaError_t configure_front_kernels() {
    return cudaFuncSetAttribute(k_merge_rows, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)(kRowGroup * kWidestFront * sizeof(double)));
}

void launch_front_rows(const DevPlan& p, const FrontPlan& f, const double* val, const double* inv, double* rows,
                       cudaStream_t st) {
    cudaMemsetAsync(rows, 0, (size_t)std::max<int64_t>(f.entries, 1) * sizeof(double), st);
    if (p.nsuper > 0) k_scatter_blocks<<<p.nsuper, 256, 0, st>>>(p, f, val, inv, rows);
    if (f.n_merged > 0)
        k_merge_rows<<<dim3(f.n_merged, (f.max_m + kRowGroup - 1) / kRowGroup), 256,
                       (size_t)kRowGroup * f.max_ns * sizeof(double), st>>>(p, f, f.merged, val, rows);
}

template <typename T>
void launch_pack(const FrontPlan& f, bool fwd, const SweepTask* tasks, int32_t ntasks, const double* rows, T* out,
                 cudaStream_t st) {
    if (ntasks <= 0) return;
    if (fwd) k_pack<T, true><<<ntasks, 256, 0, st>>>(f, tasks, rows, out);
    else k_pack<T, false><<<ntasks, 256, 0, st>>>(f, tasks, rows, out);
}
template void launch_pack<double>(const FrontPlan&, bool, const SweepTask*, int32_t, const double*, double*,
                                  cudaStream_t);
template void launch_pack<float>(const FrontPlan&, bool, const SweepTask*, int32_t, const double*, float*,
                                 cudaStream_t);

}  // namespace fcw
