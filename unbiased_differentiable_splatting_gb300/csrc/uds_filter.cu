// filtering.forward / filtering.backward (zSorting.cpp:24-43,
// zSortingCuda.cu:11-243, alphacompositing.cuh, alphacompositingGrad.cuh):
// per pixel, the depth of each sample along the pixel ray to the splat's
// tangent plane, a stable insertion arg-sort by depth, front-to-back alpha
// blending and its division-based gradient.  The arithmetic follows the
// reference operation by operation (double where it promotes), so the depth
// order is identical to the CPU oracle's.
#include "uds_composite.cuh"

namespace uds {

// The samples of a pixel ranked by depth and their depth weights (fw, by
// rank; w likewise).  Every sample takes part: an empty one lies at kZmax with
// whatever weight the caller gave it.
template <int KMAX>
__device__ __forceinline__ void filter_pixel(int i, int j, int W, int H, int K, const int* __restrict__ idx,
                                             const float* __restrict__ weights, float f, int N,
                                             const float* __restrict__ pts, const float* __restrict__ nrm,
                                             Ranked<KMAX>& w, Ranked<KMAX>& fw, int* rank) {
    using S = Samples<KMAX>;
    float dir[3], dist[KMAX], wk[KMAX];
    pixel_ray((float)W, (float)H, f, (float)i, (float)j, dir);
#pragma unroll S::kUnroll
    for (int k = 0; k < S::end(K); ++k) {
        const bool on = S::on(k, K);
        wk[k] = on ? weights[k] : 0.0f;
        dist[k] = on ? kZmax : __int_as_float(0x7f800000);
        const int s = on ? idx[k] : -1;
        if (s >= 0 && s < N) dist[k] = sample_depth(dir, pts, nrm, s, N);
    }
    depth_ranks<KMAX>(K, dist, rank);
#pragma unroll S::kUnroll
    for (int k = 0; k < S::end(K); ++k) w[rank[k]] = wk[k];
    blend_ranked<KMAX>(K, w, fw);
}

// Memory latency bounds both: K = 13 at 403 x 301, forward 16.5 us and
// backward 46 us; with every array in local memory and the integer blend and
// ray 31 and 72 us.  K = 40 at 427 x 320: 252 and 405 us, against 451 and 853.
template <int KMAX>
__global__ void __launch_bounds__(kRenderThreads) k_filter_forward(
    int W, int H, int K, const int* __restrict__ idx, const float* __restrict__ weights, float f, int pB, int N,
    const float* __restrict__ pts, const float* __restrict__ nrm, float* __restrict__ out) {
    using S = Samples<KMAX>;
    UDS_RANKED(w);
    int j = blockIdx.x * kRenderThreads + threadIdx.x;
    int i = blockIdx.y, b = blockIdx.z;
    if (j >= H) return;
    size_t e = (size_t)K * ((size_t)j + (size_t)H * ((size_t)i + (size_t)W * b));
    size_t po = pB > 1 ? 3 * (size_t)N * b : 0;
    int rank[KMAX];
    filter_pixel<KMAX>(i, j, W, H, K, idx + e, weights + e, f, N, pts + po, nrm + po, w, w, rank);
#pragma unroll S::kUnroll
    for (int k = 0; k < S::end(K); ++k)
        if (S::on(k, K)) out[e + k] = w[rank[k]];
}

template <int KMAX>
__global__ void __launch_bounds__(kRenderThreads) k_filter_backward(
    int W, int H, int K, const int* __restrict__ idx, const float* __restrict__ weights, const float* __restrict__ gin,
    float f, int pB, int N, const float* __restrict__ pts, const float* __restrict__ nrm, float* __restrict__ out) {
    using S = Samples<KMAX>;
    UDS_RANKED(w);
    UDS_RANKED(t);  // depth weights, then the numerators of the gradient, then the gradient
    int j = blockIdx.x * kRenderThreads + threadIdx.x;
    int i = blockIdx.y, b = blockIdx.z;
    if (j >= H) return;
    size_t e = (size_t)K * ((size_t)j + (size_t)H * ((size_t)i + (size_t)W * b));
    size_t po = pB > 1 ? 3 * (size_t)N * b : 0;
    int rank[KMAX];
    filter_pixel<KMAX>(i, j, W, H, K, idx + e, weights + e, f, N, pts + po, nrm + po, w, t, rank);
#pragma unroll S::kUnroll
    for (int k = 0; k < S::end(K); ++k)
        if (S::on(k, K)) t[rank[k]] = fmul(gin[e + k], t[rank[k]]);
    blend_gradients<KMAX>(K, w, t);
#pragma unroll S::kUnroll
    for (int k = 0; k < S::end(K); ++k)
        if (S::on(k, K)) out[e + k] = t[rank[k]];
}

}  // namespace uds

using namespace uds;

#define UDS_FILTER_DISPATCH(KERNEL, ...)                                              \
    do {                                                                                \
        dim3 grid(cdiv(H, kRenderThreads), W, B);                                       \
        if (K <= 8) KERNEL<8><<<grid, kRenderThreads, 0, s>>>(__VA_ARGS__);             \
        else if (K <= 16) KERNEL<16><<<grid, kRenderThreads, 0, s>>>(__VA_ARGS__);      \
        else if (K <= 32) KERNEL<32><<<grid, kRenderThreads, 0, s>>>(__VA_ARGS__);      \
        else KERNEL<64><<<grid, kRenderThreads, 0, s>>>(__VA_ARGS__);                   \
    } while (0)

extern "C" int uds_filter_forward(int B, int W, int H, int K, const int32_t* indices,
                                  const float* weights, float focal, int pB, int N,
                                  const float* points, const float* normals, float* out,
                                  void* stream) {
    if (B <= 0 || W <= 0 || H <= 0 || K <= 0 || K > kMaxK || (pB != 1 && pB != B) || N < 0) return UDS_ERR_ARGUMENT;
    if (!indices || !weights || !out) return UDS_ERR_ARGUMENT;
    cudaStream_t s = as_stream(stream);
    UDS_FILTER_DISPATCH(k_filter_forward, W, H, K, indices, weights, focal, pB, N, points, normals, out);
    return launch_status();
}

extern "C" int uds_filter_backward(int B, int W, int H, int K, const int32_t* indices,
                                   const float* weights, const float* grad, float focal, int pB,
                                   int N, const float* points, const float* normals,
                                   float* grad_weights, void* stream) {
    if (B <= 0 || W <= 0 || H <= 0 || K <= 0 || K > kMaxK || (pB != 1 && pB != B) || N < 0) return UDS_ERR_ARGUMENT;
    if (!indices || !weights || !grad || !grad_weights) return UDS_ERR_ARGUMENT;
    cudaStream_t s = as_stream(stream);
    UDS_FILTER_DISPATCH(k_filter_backward, W, H, K, indices, weights, grad, focal, pB, N, points, normals,
                        grad_weights);
    return launch_status();
}
