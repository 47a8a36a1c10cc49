// Depth compositing helpers shared by filtering.forward / backward and the
// fused render kernels (zSortingCuda.cu:11-243, alphacompositing.cuh):
// the pixel ray, each sample's depth along it to the splat's tangent plane,
// the stable order by depth, and front-to-back blending and its gradient.
// Depths, order and blend follow the reference operation by operation (double
// where it promotes), so the depth order is identical to the CPU oracle's.
#pragma once
#include "uds_blendrem.cuh"
#include "uds_ewa.cuh"

namespace uds {

// -normalize(backproject(pixel)) (alphacompositing.cuh:31-32)
__device__ __forceinline__ void pixel_ray(float W, float H, float f, float px, float py, float* dir) {
    float s[2] = {px, py}, wd[3];
    back_project(W, H, f, s, wd);
    float inv = div_via_double(1.0f, fsqrt(dot3(wd, wd)));
#pragma unroll
    for (int i = 0; i < 3; ++i) dir[i] = fmul(fmul(wd[i], inv), -1.0f);
}

__device__ __forceinline__ float sample_depth(const float* dir, const float* __restrict__ pts,
                                              const float* __restrict__ nrm, int id, int N) {
    if (id < 0 || id >= N) return kZmax;
    float p[3] = {pts[3 * (size_t)id], pts[3 * (size_t)id + 1], pts[3 * (size_t)id + 2]};
    float n[3] = {nrm[3 * (size_t)id], nrm[3 * (size_t)id + 1], nrm[3 * (size_t)id + 2]};
    float d = fdiv(dot3(p, n), dot3(dir, n));
    return d > 0.0f ? d : kZmax;
}

constexpr int kRenderThreads = 128;

// The K-sized arrays of a pixel's thread, for K up to a compile-time KMAX.
// Up to 16 samples every loop over them is unrolled, so that they are
// registers and the loads of all samples are in flight together (on() masks
// the samples beyond K); the few that are indexed by depth rank are columns
// of shared memory, conflict-free whatever element each thread is at.  Above
// that the loops are rolled and the arrays are local memory.
template <int KMAX>
struct Samples {
    static constexpr bool kUnrolled = KMAX <= 16;
    static constexpr int kUnroll = kUnrolled ? KMAX : 1;
    static __device__ __forceinline__ int end(int K) { return kUnrolled ? KMAX : K; }
    static __device__ __forceinline__ bool on(int k, int K) { return !kUnrolled || k < K; }
};
template <int KMAX, bool SHARED = Samples<KMAX>::kUnrolled>
struct Ranked {
    float x[KMAX];
    __device__ __forceinline__ float& operator[](int q) { return x[q]; }
};
template <int KMAX>
struct Ranked<KMAX, true> {
    float (*x)[kRenderThreads];
    __device__ __forceinline__ float& operator[](int q) { return x[q][threadIdx.x]; }
};
#define UDS_RANKED(NAME)                                                             \
    __shared__ float s_##NAME[Samples<KMAX>::kUnrolled ? KMAX : 1][kRenderThreads];  \
    Ranked<KMAX> NAME;                                                               \
    if constexpr (Samples<KMAX>::kUnrolled) NAME.x = s_##NAME

// Each sample's place in the stable order by depth (nearest first, equal
// depths by number; no depth is a NaN), counted: unrolled over the pairs of
// samples, 3 instructions each (the depths beyond K are infinite, which
// leaves them behind the others), else over all samples for each.  Counting
// has no chain of dependent loads as an insertion sort has.
template <int KMAX>
__device__ __forceinline__ void depth_ranks(int K, const float* dist, int* rank) {
    if constexpr (Samples<KMAX>::kUnrolled) {
#pragma unroll
        for (int a = 0; a < KMAX; ++a) rank[a] = 0;
#pragma unroll
        for (int a = 0; a < KMAX; ++a)
#pragma unroll
            for (int b = a + 1; b < KMAX; ++b) {
                const bool first = dist[b] < dist[a];
                rank[a] += first ? 1 : 0;
                rank[b] += first ? 0 : 1;
            }
    } else {
        for (int a = 0; a < K; ++a) {
            const float value = dist[a];
            int n = 0;
#pragma unroll 4
            for (int b = 0; b < K; ++b) n += dist[b] < value || (dist[b] == value && b < a) ? 1 : 0;
            rank[a] = n;
        }
    }
}

// front-to-back blend of K samples in depth order (alphacompositing.cuh:
// 58-68): fw = rem w, rem *= (1 - w) in double.  The double update is
// evaluated in float arithmetic (uds_nearfloat.cuh) and, near a rounding
// boundary, on the exact integer product (uds_blendrem.cuh), both with the
// double sequence's bits; the FP64 pipe only sees what is outside both.
// Nothing finite changes rem once it is 0.  fw may be w.
template <int KMAX>
__device__ __forceinline__ void blend_ranked(int K, Ranked<KMAX>& w, Ranked<KMAX>& fw) {
    float rem = 1.0f;
#pragma unroll 1
    for (int q = 0; q < K; ++q) {
        const float wq = w[q];
        fw[q] = fmul(rem, wq);
        float next;
        if (!near_rem(rem, wq, &next) && (rem != 0.0f || !(fabsf(wq) < __int_as_float(0x7f800000)))) {
            if (!blend_rem(rem, wq, &next)) next = (float)dmul((double)rem, dsub(1.0, (double)wq));
        } else if (rem == 0.0f) {
            next = rem;
        }
        rem = next;
    }
}

// gradBlending (alphacompositingGrad.cuh:7-26): the gradients of the EWA
// weights w from the numerators t = g fw, in place of t.  Terms whose divisor
// is within 1e-4 of zero are dropped as in the reference, and those whose
// numerator is 0, which change nothing.  (Summing the numerators first and
// dividing once would be K divisions, not K (K + 1) / 2, but its rounding
// errors are up to a quarter larger.)
template <int KMAX>
__device__ __forceinline__ void blend_gradients(int K, Ranked<KMAX>& w, Ranked<KMAX>& t) {
    const float eps = 1e-4f;
#pragma unroll 1
    for (int q = 0; q < K; ++q) {
        const float wq = w[q], den = -fsub(1.0f, wq);
        float acc = 0.0f;
        if (fabsf(wq) > eps) acc = fadd(acc, fdiv(t[q], wq));
        if (fabsf(den) > eps) {
#pragma unroll 1
            for (int r = q + 1; r < K; ++r) {
                const float tr = t[r];
                if (tr != 0.0f) acc = fadd(acc, fdiv(tr, den));
            }
        }
        t[q] = acc;
    }
}

}  // namespace uds
