// Fused gradient -> normalise -> divergence over faces (fastcw_lean.py:416-442).
//
// Every output element is written exactly once, by one thread (no atomics, deterministic).
//
// FP64 form: the reference's 3-vector arithmetic, operation for operation, with explicit
// round-to-nearest intrinsics so the compiler cannot contract into FMAs, summed per vertex in the
// order of the reference's face loop: given the same u, the divergence is bit-identical. The square
// root and the division of a face's scale -A / |grad u| cost as much as everything else a corner
// needs, so a first pass forms the scales (a warp takes four faces) and a second gathers them (a warp
// per vertex, its faces in ascending order): 2.1x less FP64 work than evaluating each face at each of
// its corners, for one 8-byte value per face and column through memory. 147k vertices,
// 1024 columns: 4.76 to 3.26 ms, bound by the gathers' latency (FP64 pipe 45% busy).
//
// Mixed form: X = -grad u / |grad u| is invariant to scaling u's differences, so FP64 differences
// scaled by a power of two (exact) are rounded to FP32 and the rest runs in FP32 in the intrinsic
// form: with d1, d2 the differences along two edges from the vertex and c_ab = gb_a . gb_b of the
// hat-function gradients of those edges' ends,
//   a = d1 c11 + d2 c12,  b = d1 c12 + d2 c22,  |g|^2 = d1 a + d2 b,  g . gb_vertex = -(a + b)
// (the stored coefficients carry the squared area, which then multiplies the term by the area).
// This keeps the direction accurate where u is far below FP32's range (u spans ~1e-130..1 on these
// meshes). A vertex walks its faces as fans, each neighbour's difference formed and rounded once for
// the two faces that share it, scaled by the vertex's own u; a face whose |g|^2 then leaves
// [2^-80, 2^80] (edges tens of diffusion lengths long, or u out of the normal range) is evaluated
// with a scale of its own. A CTA takes a patch of consecutive vertices in elimination order (mostly
// part of one dissection leaf, so a compact piece of the surface) and brings its rows and their
// neighbours' into shared memory once; gathered through L1, rows came back from L2 three to four
// times. 147k vertices, 1024 columns: 1.73 to 1.33 ms; issue 52%, shared memory 49% and the conversion pipe 36%
// busy: warps wait about equally for fixed latencies, for conversions and shared memory, and for rows.
// Vertices with too many neighbours for a patch are gathered from memory, a warp each.
//
// At a sharp corner (under 6 degrees: needle triangles) the two edges are nearly parallel and |g|^2 cancels
// in FP32, at that corner but not at the face's other two, so the face's three terms no longer cancel in the
// sum over the mesh. Vertices with such corners are evaluated once more, a warp each: the sharp faces with
// the difference along the short edge, formed in FP64, in place of the second long one,
//   a = d1 c_vv + e c_vb,  b = d1 c_vb + e c_bb,  |g|^2 = d1 a + e b,  g . gb_vertex = -a.
// A fan of 500 needles: fields 7.3e-5 of their maximum off without this. Meshes without such corners (every
// folded icosphere up to jitter 0.2) launch nothing.
#include "kernels.cuh"

namespace fcw {

namespace {

__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }

// The FP64 geometry of a face: hat-function gradients of corners 1 and 2 and the area (64 bytes);
// corner 0's gradient is -g1 - g2, as the operators form it.
struct FaceGeo {
    double g1[3], g2[3], area;
};
__device__ __forceinline__ FaceGeo read_geo(const double* geo, int p) {
    const double2* r = reinterpret_cast<const double2*>(geo) + 4 * (int64_t)p;
    const double2 a = r[0], b = r[1], c = r[2], d = r[3];
    return FaceGeo{{a.x, a.y, b.x}, {b.y, c.x, c.y}, d.x};
}
__device__ __forceinline__ void gradient(const FaceGeo& g, double u0, double u1, double u2, double& gx, double& gy,
                                         double& gz) {
    const double du1 = sub(u1, u0), du2 = sub(u2, u0);
    gx = add(mul(du1, g.g1[0]), mul(du2, g.g2[0]));
    gy = add(mul(du1, g.g1[1]), mul(du2, g.g2[1]));
    gz = add(mul(du1, g.g1[2]), mul(du2, g.g2[2]));
}
// -A / |grad u|, NaN where the gradient vanishes (the face is skipped).
__device__ __forceinline__ double face_scale(const FaceGeo& g, double gx, double gy, double gz) {
    const double nn = __dsqrt_rn(add(add(mul(gx, gx), mul(gy, gy)), mul(gz, gz)));
    return nn > 1e-300 ? __ddiv_rn(-g.area, nn) : __longlong_as_double(0x7ff8000000000000LL);
}
// Corner c's hat-function gradient.
__device__ __forceinline__ void corner_gradient(const FaceGeo& g, int c, double (&b)[3]) {
#pragma unroll
    for (int x = 0; x < 3; ++x) b[x] = c == 0 ? sub(-g.g1[x], g.g2[x]) : (c == 1 ? g.g1[x] : g.g2[x]);
}
__device__ __forceinline__ double corner_term(double s, double gx, double gy, double gz, const double (&b)[3]) {
    return mul(s, add(add(mul(gx, b[0]), mul(gy, b[1])), mul(gz, b[2])));
}

// 64*NP columns per warp: lane l owns the column pairs {2l, 2l+1} + 64p (16-byte loads).
template <int NP>
__device__ __forceinline__ void load_cols(const double* p, double (&w)[2 * NP]) {
#pragma unroll
    for (int q = 0; q < NP; ++q) {
        const double2 x = *reinterpret_cast<const double2*>(p + 64 * q);
        w[2 * q] = x.x;
        w[2 * q + 1] = x.y;
    }
}
template <int NP>
__device__ __forceinline__ void store_cols(double* p, const double (&w)[2 * NP]) {
#pragma unroll
    for (int q = 0; q < NP; ++q) *reinterpret_cast<double2*>(p + 64 * q) = make_double2(w[2 * q], w[2 * q + 1]);
}

constexpr int kFacesPerWarp = 4;

// Both passes: three CTAs per SM (80 registers) beat four (64: spills) and the half-as-wide slice of
// six (more rows per value); 147k vertices, 1024 columns: 3.3 ms against 3.8 and 4.1-4.4.
template <int NP>
__global__ void __launch_bounds__(256, 3) k_face_scale(FaceData fd, const double* __restrict__ u,
                                                       double* __restrict__ scale, int32_t K) {
    const int lane = threadIdx.x & 31;
    const int p0 = (blockIdx.x * 8 + (threadIdx.x >> 5)) * kFacesPerWarp, np = min(kFacesPerWarp, fd.nf - p0);
    if (np <= 0) return;
    const int64_t c0 = (int64_t)blockIdx.y * 64 * NP + 2 * lane;
    const int4 mine = fd.corners[p0 + min(lane, np - 1)];
    double w[3][2 * NP];
    auto load = [&](int j) {
        load_cols<NP>(u + (int64_t)__shfl_sync(0xffffffffu, mine.x, j) * K + c0, w[0]);
        load_cols<NP>(u + (int64_t)__shfl_sync(0xffffffffu, mine.y, j) * K + c0, w[1]);
        load_cols<NP>(u + (int64_t)__shfl_sync(0xffffffffu, mine.z, j) * K + c0, w[2]);
    };
    load(0);
#pragma unroll 1
    for (int j = 0; j < np; ++j) {
        const FaceGeo g = read_geo(fd.geo, p0 + j);
        double gx[2 * NP], gy[2 * NP], gz[2 * NP], s[2 * NP];
#pragma unroll
        for (int t = 0; t < 2 * NP; ++t) gradient(g, w[0][t], w[1][t], w[2][t], gx[t], gy[t], gz[t]);
        if (j + 1 < np) load(j + 1);
#pragma unroll
        for (int t = 0; t < 2 * NP; ++t) s[t] = face_scale(g, gx[t], gy[t], gz[t]);
        store_cols<NP>(scale + (int64_t)(p0 + j) * K + c0, s);
    }
}

template <int NP>
__global__ void __launch_bounds__(256, 3) k_div_fp64(FaceData fd, const double* __restrict__ u,
                                                     const double* __restrict__ scale, double* __restrict__ div,
                                                     int32_t K) {
    const int lane = threadIdx.x & 31, v = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (v >= fd.nv) return;
    const int64_t c0 = (int64_t)blockIdx.y * 64 * NP + 2 * lane;
    double acc[2 * NP];
#pragma unroll
    for (int t = 0; t < 2 * NP; ++t) acc[t] = 0.0;
    const int q0 = fd.inc_ptr[v], deg = fd.inc_ptr[v + 1] - q0;
    for (int jb = 0; jb < deg; jb += 32) {
        const int nj = min(32, deg - jb);
        const int4 mine = fd.inc_rec[q0 + jb + min(lane, nj - 1)];
        for (int j = 0; j < nj; ++j) {
            const int pc = __shfl_sync(0xffffffffu, mine.w, j), p = pc & kIncFace, c = (unsigned)pc >> kIncCornerShift;
            double u0[2 * NP], u1[2 * NP], u2[2 * NP], s[2 * NP], b[3];
            load_cols<NP>(u + (int64_t)__shfl_sync(0xffffffffu, mine.x, j) * K + c0, u0);
            load_cols<NP>(u + (int64_t)__shfl_sync(0xffffffffu, mine.y, j) * K + c0, u1);
            load_cols<NP>(u + (int64_t)__shfl_sync(0xffffffffu, mine.z, j) * K + c0, u2);
            load_cols<NP>(scale + (int64_t)p * K + c0, s);
            const FaceGeo g = read_geo(fd.geo, p);
            corner_gradient(g, c, b);
#pragma unroll
            for (int t = 0; t < 2 * NP; ++t) {
                double gx, gy, gz;
                gradient(g, u0[t], u1[t], u2[t], gx, gy, gz);
                const double x = add(acc[t], corner_term(s[t], gx, gy, gz, b));
                acc[t] = s[t] == s[t] ? x : acc[t];
            }
        }
    }
    store_cols<NP>(div + (int64_t)v * K + c0, acc);
}

// The divergence at vertex v of one column of u (leading dimension K): its faces' terms in incidence order.
__device__ __forceinline__ double div_at(const FaceData& fd, const double* __restrict__ u, int64_t K, int64_t col,
                                         int v) {
    double acc = 0.0;
    const int q1 = fd.inc_ptr[v + 1];
    for (int q = fd.inc_ptr[v]; q < q1; ++q) {
        const int4 r = fd.inc_rec[q];
        const FaceGeo g = read_geo(fd.geo, r.w & kIncFace);
        double gx, gy, gz, b[3];
        gradient(g, u[(int64_t)r.x * K + col], u[(int64_t)r.y * K + col], u[(int64_t)r.z * K + col], gx, gy, gz);
        corner_gradient(g, (unsigned)r.w >> kIncCornerShift, b);
        const double s = face_scale(g, gx, gy, gz);
        if (s == s) acc = add(acc, corner_term(s, gx, gy, gz, b));
    }
    return acc;
}
// One column: a thread per vertex (its face loop's loads are independent, so they overlap).
__global__ void __launch_bounds__(256) k_div_fp64_one(FaceData fd, const double* __restrict__ u,
                                                      double* __restrict__ div) {
    asm volatile("griddepcontrol.launch_dependents;");
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v < fd.nv) div[v] = div_at(fd, u, 1, 0, v);
}

// 2^-e for the binary exponent e of |x| (x normal): exact scaling to [1, 2). A zero or subnormal x
// gives 2^1023.
__device__ __forceinline__ double unit_scale(double x) {
    const long long e = (__double_as_longlong(x) >> 52) & 0x7ff;
    return __longlong_as_double((2046 - e) << 52);
}
// One face's term at its vertex from the FP64 differences, with a scale of its own; c holds the
// coefficients times the squared area. SHARP: those of a sharp corner (SharpFans).
template <bool SHARP>
__device__ __noinline__ float face_alone(double d1, double d2, float c11, float c12, float c22) {
    const double mx = fmax(fabs(d1), fabs(d2));
    if (!(mx >= 2.2250738585072014e-308)) return 0.0f;  // zero (or subnormal) gradient
    const double sc = unit_scale(mx);
    const float x1 = (float)(d1 * sc), x2 = (float)(d2 * sc);
    const float a = x1 * c11 + x2 * c12, b = x1 * c12 + x2 * c22, q = x1 * a + x2 * b;
    return q > 0.0f ? (SHARP ? a : a + b) * rsqrtf(q) : 0.0f;
}

// Pairs of FP32 values in one register pair (packed FMA pipe).
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float x, float y) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ float2 unpack2(f32x2 p) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(p));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ float rsqrt_approx(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));  // x normal: within rsqrtf's 2 ulp
    return r;
}
// |g|^2 below this many exponent steps of 2^-80 is in [2^-80, 2^80); zero, negative and NaN are not.
constexpr unsigned kFanLow = 47u << 23, kFanSpan = 160u << 23;

constexpr int kColsMixed = 64;  // a warp's columns: two per lane

// The faces of one vertex for two columns. uv: the vertex's values; row(w): the lane's values at
// neighbour w; steps [e0, e1) of fan.
template <class Steps, class Row>
__device__ __forceinline__ f32x2 fan_sum(double2 uv, int e0, int e1, Steps&& fan, Row&& row) {
    const double sc0 = unit_scale(uv.x), sc1 = unit_scale(uv.y);
    f32x2 acc = pack2(0.0f, 0.0f);
    auto diff = [&](int w) {
        const double2 un = row(w);
        return pack2((float)((un.x - uv.x) * sc0), (float)((un.y - uv.y) * sc1));
    };
    for (int e = e0; e < e1;) {  // a fan: its first neighbour, then a face per step
        const FanStep first = fan(e);
        f32x2 xp = diff(first.neighbour);
        const int end = e + 1 + first.faces;
#pragma unroll 2
        for (++e; e < end; ++e) {
            const FanStep c = fan(e);
            const f32x2 x = diff(c.neighbour);
            const f32x2 p11 = pack2(c.c11[0], c.c11[1]), p12 = pack2(c.c12[0], c.c12[1]), p22 = pack2(c.c22[0], c.c22[1]);
            const f32x2 a = fma2(x, p12, mul2(xp, p11)), b = fma2(x, p22, mul2(xp, p12));
            const float2 q = unpack2(fma2(x, b, mul2(xp, a)));
            const f32x2 ab = add2(a, b);
            const bool in0 = __float_as_uint(q.x) - kFanLow < kFanSpan, in1 = __float_as_uint(q.y) - kFanLow < kFanSpan;
            if (in0 && in1) {
                acc = fma2(ab, pack2(rsqrt_approx(q.x), rsqrt_approx(q.y)), acc);
            } else {  // each value by its own range, so a column's result does not depend on its neighbour
                const double2 up = row(fan(e - 1).neighbour), un = row(c.neighbour);
                float2 r = unpack2(acc);
                const float2 n2 = unpack2(ab);
                r.x = in0 ? fmaf(n2.x, rsqrt_approx(q.x), r.x)
                          : r.x + face_alone<false>(up.x - uv.x, un.x - uv.x, c.c11[0], c.c12[0], c.c22[0]);
                r.y = in1 ? fmaf(n2.y, rsqrt_approx(q.y), r.y)
                          : r.y + face_alone<false>(up.y - uv.y, un.y - uv.y, c.c11[0], c.c12[0], c.c22[0]);
                acc = pack2(r.x, r.y);
            }
            xp = x;
        }
    }
    return acc;
}

__global__ void __launch_bounds__(256, 3) k_div_mixed(FaceData fd, const double* __restrict__ u,
                                                      float* __restrict__ div, int32_t K,
                                                      const uint8_t* __restrict__ grounded) {
    extern __shared__ __align__(128) double sm[];
    double* S = sm;                                                         // rows x 64
    FanStep* fan = reinterpret_cast<FanStep*>(S + kPatchRows * kColsMixed);
    __shared__ int step0[kPatchVerts + 1];
    __shared__ bool zero[kPatchVerts];
    const Patch pt = fd.patches[blockIdx.x];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, c0 = blockIdx.y * kColsMixed;
    constexpr int VPR = kColsMixed / 2;
    for (int e = tid; e < pt.nrows * VPR; e += 256) {
        const int r = e / VPR, v = e - r * VPR;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(
                         (unsigned)__cvta_generic_to_shared(S + r * kColsMixed + 2 * v)),
                     "l"(u + (int64_t)fd.patch_rows[pt.row0 + r] * K + c0 + 2 * v)
                     : "memory");
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    const int f0 = fd.fan_ptr[pt.v0];
    for (int i = tid; i <= pt.nv; i += 256) {
        step0[i] = fd.fan_ptr[pt.v0 + i] - f0;
        if (i < pt.nv) zero[i] = grounded[pt.v0 + i];
    }
    for (int e = tid; e < 2 * pt.nsteps; e += 256)
        reinterpret_cast<int4*>(fan)[e] = reinterpret_cast<const int4*>(fd.fans)[2 * (int64_t)f0 + e];
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
    const double2* Sl = reinterpret_cast<const double2*>(S) + lane;
    for (int i = warp; i < pt.nv; i += 8) {  // a patch's own rows come first
        f32x2 acc = pack2(0.0f, 0.0f);
        if (!zero[i])
            acc = fan_sum(Sl[i * VPR], step0[i], step0[i + 1], [&](int e) { return fan[e]; },
                          [&](int w) { return Sl[w * VPR]; });
        *reinterpret_cast<float2*>(div + (int64_t)(pt.v0 + i) * K + c0 + 2 * lane) = unpack2(acc);
    }
}

__global__ void __launch_bounds__(256) k_div_mixed_big(FaceData fd, const double* __restrict__ u,
                                                       float* __restrict__ div, int32_t K,
                                                       const uint8_t* __restrict__ grounded) {
    const int lane = threadIdx.x & 31, i = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (i >= fd.nbig) return;
    const int v = fd.big[i];
    const double* uc = u + (int64_t)blockIdx.y * kColsMixed + 2 * lane;
    auto row = [&](int w) { return *reinterpret_cast<const double2*>(uc + (int64_t)w * K); };
    f32x2 acc = pack2(0.0f, 0.0f);
    if (!grounded[v])
        acc = fan_sum(row(v), fd.fan_ptr[v], fd.fan_ptr[v + 1], [&](int e) { return fd.fans[e]; }, row);
    *reinterpret_cast<float2*>(div + (int64_t)v * K + (int64_t)blockIdx.y * kColsMixed + 2 * lane) = unpack2(acc);
}

__global__ void __launch_bounds__(256) k_div_mixed_sharp(FaceData fd, const double* __restrict__ u,
                                                         float* __restrict__ div, int32_t K,
                                                         const uint8_t* __restrict__ grounded) {
    const int lane = threadIdx.x & 31, i = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (i >= fd.nsharp || grounded[fd.sharp[i]]) return;
    const int v = fd.sharp[i];
    const int64_t c0 = (int64_t)blockIdx.y * kColsMixed + 2 * lane;
    auto row = [&](int w) { return *reinterpret_cast<const double2*>(u + (int64_t)w * K + c0); };
    const double2 uv = row(v);
    double2 up = uv;
    float2 acc = make_float2(0.0f, 0.0f);
    for (int e = fd.sharp_ptr[i]; e < fd.sharp_ptr[i + 1]; ++e) {
        const FanStep c = fd.sharp_fans[e];
        const double2 un = row(c.neighbour);
        if (c.faces == -2) {
            acc.x += face_alone<true>(up.x - uv.x, un.x - up.x, c.c11[0], c.c12[0], c.c22[0]);
            acc.y += face_alone<true>(up.y - uv.y, un.y - up.y, c.c11[0], c.c12[0], c.c22[0]);
        } else if (c.faces < 0) {
            acc.x += face_alone<false>(up.x - uv.x, un.x - uv.x, c.c11[0], c.c12[0], c.c22[0]);
            acc.y += face_alone<false>(up.y - uv.y, un.y - uv.y, c.c11[0], c.c12[0], c.c22[0]);
        }
        up = un;
    }
    *reinterpret_cast<float2*>(div + (int64_t)v * K + c0) = acc;
}

constexpr size_t kSmemMixed = (size_t)kPatchRows * kColsMixed * 8 + (size_t)kPatchSteps * sizeof(FanStep);

}  // namespace

cudaError_t configure_divergence_kernels() {
    return cudaFuncSetAttribute(k_div_mixed, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMixed);
}

// K is a multiple of 64
void launch_divergence_fp64(const FaceData& fd, const double* u, double* scale, double* div, int32_t K,
                            cudaStream_t st) {
    if (fd.nv <= 0 || K <= 0) return;
    constexpr int FW = 8 * kFacesPerWarp;
    if (K % 128 == 0) {
        k_face_scale<2><<<dim3((fd.nf + FW - 1) / FW, K / 128), 256, 0, st>>>(fd, u, scale, K);
        k_div_fp64<2><<<dim3((fd.nv + 7) / 8, K / 128), 256, 0, st>>>(fd, u, scale, div, K);
    } else {
        k_face_scale<1><<<dim3((fd.nf + FW - 1) / FW, K / 64), 256, 0, st>>>(fd, u, scale, K);
        k_div_fp64<1><<<dim3((fd.nv + 7) / 8, K / 64), 256, 0, st>>>(fd, u, scale, div, K);
    }
}

void launch_divergence_fp64_one(const FaceData& fd, const double* u, double* div, cudaStream_t st) {
    if (fd.nv > 0) k_div_fp64_one<<<(fd.nv + 255) / 256, 256, 0, st>>>(fd, u, div);
}

void launch_divergence_mixed(const FaceData& fd, const double* u, float* div, int32_t K, const uint8_t* grounded,
                             cudaStream_t st) {
    if (fd.nv <= 0 || K <= 0) return;
    if (fd.npatches > 0)
        k_div_mixed<<<dim3(fd.npatches, K / kColsMixed), 256, kSmemMixed, st>>>(fd, u, div, K, grounded);
    if (fd.nbig > 0)
        k_div_mixed_big<<<dim3((fd.nbig + 7) / 8, K / kColsMixed), 256, 0, st>>>(fd, u, div, K, grounded);
    if (fd.nsharp > 0)
        k_div_mixed_sharp<<<dim3((fd.nsharp + 7) / 8, K / kColsMixed), 256, 0, st>>>(fd, u, div, K, grounded);
}

}  // namespace fcw
