// splatting.forward / splatting.backward (splatting.cpp:43-129,
// splattingCuda.cu:18-233) restructured for the GPU:
//   forward : per-splat Gaussian constants once (the part of the reference's
//             per-sample work that does not depend on the pixel), then one
//             thread per pixel evaluates its K samples;
//   backward: per sample only the sufficient statistics of the gradient
//             (sum g*G, sum g*G*d, sum g*G*d d^T, d = pixel - screen point)
//             are scattered, then one thread per splat applies the chain
//             rule through covariance, Jacobian, tangent plane and
//             projection once.  The reference instead runs the full chain
//             (ewaSplattingGrad.cuh:163-206) per sample and scatters 8 floats.
// The fused render kernels at the end of this file run EWA weights, depth
// compositing and attribute interpolation (and their backward passes) per
// pixel in one kernel each way.
#include "uds_composite.cuh"

namespace uds {

// The pairs of one view that some pixel samples (a bit each, whole words per
// view: mark_words), gathered by a block from PER x 256 consecutive ones: only those get Gaussian constants and
// gradients, as in the reference, whose kernels visit sampled pairs only.  A
// view of a large scene samples a few percent of its splats; one thread per
// pair left a warp running the whole frame for one lane in twenty (two passes
// over 16 views of 2M splats 2.27 ms; gathered 0.51 ms).
constexpr int kPairThreads = 256;
__host__ __device__ inline int mark_words(int N) { return (int)(((unsigned)N + 31u) >> 5); }

template <int PER>
struct PairList {
    unsigned short at[kPairThreads * PER];
    unsigned count;
};

// Fills the list with the block's used pairs (offsets from base); returns
// their number.
template <int PER>
__device__ __forceinline__ int gather_pairs(PairList<PER>& list, const unsigned* __restrict__ used, int base, int N) {
    if (threadIdx.x == 0) list.count = 0;
    __syncthreads();
    used += (size_t)mark_words(N) * blockIdx.y;
    const unsigned lane = threadIdx.x & 31;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const int at = i * kPairThreads + (int)threadIdx.x;
        const unsigned m = base + at - (int)lane < N ? used[(base + at) >> 5] : 0u;  // the warp's 32 pairs
        unsigned first = 0;
        if (lane == 0 && m) first = atomicAdd(&list.count, (unsigned)__popc(m));
        first = __shfl_sync(0xffffffffu, first, 0);
        if ((m >> lane) & 1u) list.at[first + __popc(m & ((1u << lane) - 1u))] = (unsigned short)at;
    }
    __syncthreads();
    return (int)list.count;
}

// Constants of the used pairs; their plane offset p . n in the second
// float4's last component (the depth along a pixel ray needs it).  stats:
// gradient statistics to be zeroed for the same pairs, or NULL.
template <int PER>
__global__ void __launch_bounds__(kPairThreads) k_ewa_consts(int N, float W, float H, float f,
                                                             const float* __restrict__ pts,
                                                             const float* __restrict__ nrm,
                                                             const float* __restrict__ sd, int sdB, float sm,
                                                             const unsigned* __restrict__ used,
                                                             float4* __restrict__ consts, float4* __restrict__ stats) {
    __shared__ PairList<PER> list;
    const size_t view = (size_t)N * blockIdx.y;
    const int base = blockIdx.x * kPairThreads * PER;
    const int count = gather_pairs<PER>(list, used, base, N);
    for (int i = threadIdx.x; i < count; i += kPairThreads) {
        const int x = base + list.at[i];
        const size_t o = view + x;
        float p[3] = {pts[3 * o], pts[3 * o + 1], pts[3 * o + 2]};
        float n[3] = {nrm[3 * o], nrm[3 * o + 1], nrm[3 * o + 2]};
        size_t so = sdB > 1 ? o : (size_t)x;
        float s[2] = {sd[2 * so], sd[2 * so + 1]};
        EwaFrame F;
        ewa_frame(W, H, f, p, n, s, sm, F);
        float4 a, c;
        ewa_gauss_consts(F, a, c);
        c.w = dot3(p, n);
        consts[2 * o] = a;
        consts[2 * o + 1] = c;
        if (stats) {
            stats[2 * o] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            stats[2 * o + 1] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
    }
}

// Marks the (view, splat) pairs that some pixel samples; S samples per view,
// blockIdx.y the view.
//
// k_ewa_mark: a block collects the marks of `chunk` samples in a bit map in
// shared memory (of the splats [range z, range (z + 1)), range a multiple of
// 32) and adds the words that have any to the view's.  Setting a mark in
// global memory per sample is bound by the 32 scattered stores of a warp, one
// a cycle per SM: 1001 x 763, K = 8, 6.1M samples 28 us, now 7.5;
// 1024^2, 1.8M of 8.4M valid 20 us, now 13.
constexpr int kMarkThreads = 512;
template <bool VEC>
__global__ void __launch_bounds__(kMarkThreads) k_ewa_mark(size_t S, size_t chunk, const int* __restrict__ idx, int N,
                                                           int range, unsigned* __restrict__ used) {
    extern __shared__ unsigned bits[];
    const int lo = (int)blockIdx.z * range, count = min(N - lo, range), words = mark_words(count);
    for (int w = threadIdx.x; w < words; w += kMarkThreads) bits[w] = 0u;
    __syncthreads();
    idx += S * blockIdx.y;
    const size_t first = chunk * blockIdx.x, end = min(first + chunk, S);
    auto mark = [&](int id) {
        const unsigned o = (unsigned)id - (unsigned)lo;  // (no sample: -1, far above)
        if (id >= 0 && o < (unsigned)count) atomicOr(&bits[o >> 5], 1u << (o & 31u));
    };
    if (VEC) {
#pragma unroll 4
        for (size_t s = first + 4 * threadIdx.x; s < end; s += 4 * kMarkThreads) {
            const int4 v = *reinterpret_cast<const int4*>(idx + s);
            mark(v.x);
            mark(v.y);
            mark(v.z);
            mark(v.w);
        }
    } else {
#pragma unroll 4
        for (size_t s = first + threadIdx.x; s < end; s += kMarkThreads) mark(idx[s]);
    }
    __syncthreads();
    used += (size_t)mark_words(N) * blockIdx.y + (lo >> 5);
    for (int w = threadIdx.x; w < words; w += kMarkThreads)
        if (const unsigned m = bits[w]) atomicOr(&used[w], m);
}

// The same sample by sample, for few samples or a great many splats.
__global__ void k_ewa_mark_direct(size_t S, const int* __restrict__ idx, int N, unsigned* __restrict__ used) {
    const size_t s = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= S) return;
    const int id = idx[S * blockIdx.y + s];
    if (id >= 0 && id < N) atomicOr(&used[(size_t)mark_words(N) * blockIdx.y + (id >> 5)], 1u << (id & 31));
}

// One thread per pixel (x = i, y = j), K samples.
__global__ void k_ewa_forward(int B, int W, int H, int K, const int* __restrict__ idx,
                              const float4* __restrict__ consts, int N, float* __restrict__ w) {
    int j = blockIdx.x * blockDim.x + threadIdx.x;
    int i = blockIdx.y;
    int b = blockIdx.z;
    if (j >= H) return;
    size_t pix = (size_t)j + (size_t)H * ((size_t)i + (size_t)W * b);
    float px = (float)i, py = (float)j;
    for (int s = 0; s < K; ++s) {
        size_t off = (size_t)s + (size_t)K * pix;
        int id = idx[off];
        float out = 0.0f;
        if (id >= 0 && id < N) {
            size_t o = (size_t)id + (size_t)N * b;
            float4 a = consts[2 * o], c = consts[2 * o + 1];
            out = fminf(ewa_gauss(a, c, px, py), 1.0f);
        }
        w[off] = out;
    }
}

// Sufficient statistics of the EWA gradient, gated on the unclamped weight
// <= 1 like gradEwaKernel (splattingCuda.cu:173).
__global__ void k_ewa_stats(int B, int W, int H, int K, const float* __restrict__ grad,
                            const int* __restrict__ idx, const float4* __restrict__ consts, int N,
                            float4* __restrict__ stats) {
    int j = blockIdx.x * blockDim.x + threadIdx.x;
    int i = blockIdx.y;
    int b = blockIdx.z;
    if (j >= H) return;
    size_t pix = (size_t)j + (size_t)H * ((size_t)i + (size_t)W * b);
    float px = (float)i, py = (float)j;
    for (int s = 0; s < K; ++s) {
        size_t off = (size_t)s + (size_t)K * pix;
        int id = idx[off];
        if (id < 0 || id >= N) continue;
        size_t o = (size_t)id + (size_t)N * b;
        float4 a = consts[2 * o], c = consts[2 * o + 1];
        float dx, dy;
        float G = ewa_gauss(a, c, px, py, &dx, &dy);
        if (!(G <= 1.0f)) continue;
        float g = grad[off] * G;
        if (g == 0.0f) continue;
        atomicAdd(&stats[2 * o], make_float4(g, g * dx, g * dy, g * dx * dx));
        atomicAdd(reinterpret_cast<float2*>(&stats[2 * o + 1]), make_float2(g * dx * dy, g * dy * dy));
    }
}

__device__ __forceinline__ void cross3(const float* a, const float* b, float* c) {
    c[0] = a[1] * b[2] - a[2] * b[1];
    c[1] = a[2] * b[0] - a[0] * b[2];
    c[2] = a[0] * b[1] - a[1] * b[0];
}
__device__ __forceinline__ float dot3c(const float* a, const float* b) { return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]; }

// Scale of a gradient row in the reference's post-processing
// (conditionalNormalization, utils.py:147-150): 1 / max(|g| + 1e-4, 1), a
// NaN norm giving NaN; clean() then zeroes NaNs.
__device__ __forceinline__ float row_divisor(float norm) {
    const float s = norm + 1e-4f;
    return s < 1.0f ? 1.0f : s;
}
__device__ __forceinline__ float clean(float x) { return x != x ? 0.0f : x; }

// Reverse-mode chain of the EWA weight for one splat (pair o of view's splat
// x) from its statistics.  CLAMP: gradients of points and (unless they are
// summed over views) std-devs with the reference's post-processing.
template <bool CLAMP>
__device__ __forceinline__ void ewa_chain(int x, size_t o, bool sum_sd, float W, float H, float f,
                                          const float* __restrict__ pts, const float* __restrict__ nrm,
                                          const float* __restrict__ sd, int sdB, float sm, float4 st0, float4 st1,
                                          float* __restrict__ gp_out, float* __restrict__ gn_out,
                                          float* __restrict__ gs_out) {
    float S0 = st0.x, S1x = st0.y, S1y = st0.z, S2xx = st0.w, S2xy = st1.x, S2yy = st1.y;
    if (S0 == 0.0f && S1x == 0.0f && S1y == 0.0f && S2xx == 0.0f && S2xy == 0.0f && S2yy == 0.0f) return;
    size_t so = sdB > 1 ? o : (size_t)x;
    float p[3] = {pts[3 * o], pts[3 * o + 1], pts[3 * o + 2]};
    float n[3] = {nrm[3 * o], nrm[3 * o + 1], nrm[3 * o + 2]};
    float sdv[2] = {sd[2 * so], sd[2 * so + 1]};
    // forward quantities (same sequence as the frame)
    float sp[2];
    screen_point(W, H, f, p, sp);
    float y0[2] = {add_via_double(sp[0], 1.0f), sp[1]};
    float y1[2] = {sp[0], add_via_double(sp[1], 1.0f)};
    float x0[3], x1[3], t0[3], t1[3];
    back_project(W, H, f, y0, x0);
    back_project(W, H, f, y1, x1);
    float c = dot3(p, n);
    float D0 = dot3(x0, n), D1 = dot3(x1, n);
    float k0 = fdiv(c, D0), k1 = fdiv(c, D1);
    tangent(x0, p, n, t0);
    tangent(x1, p, n, t1);
    float al = fsqrt(dot3(t0, t0));
    float invNorm = div_via_double(1.0f, al);
    float u0[3] = {t0[0] * invNorm, t0[1] * invNorm, t0[2] * invNorm};
    float u1[3];
    cross3(u0, n, u1);
    float be = dot3c(t1, u0), ga = dot3c(t1, u1);
    float J00 = 1.0f / al, J01 = -be / (al * ga), J11 = 1.0f / ga;
    float Sg0 = sdv[0] * sdv[0], Sg1 = sdv[1] * sdv[1];
    float V00 = J00 * J00 * Sg0 + J01 * J01 * Sg1 + sm;
    float V01 = J01 * J11 * Sg1;
    float V11 = J11 * J11 * Sg1 + sm;
    float vdet = V00 * V11 - V01 * V01;
    float I00 = V11 / vdet, I01 = -V01 / vdet, I11 = V00 / vdet;
    // moments of q = V^-1 d
    float M1x = I00 * S1x + I01 * S1y, M1y = I01 * S1x + I11 * S1y;
    float A00 = I00 * S2xx + I01 * S2xy, A01 = I00 * S2xy + I01 * S2yy;
    float A10 = I01 * S2xx + I11 * S2xy, A11 = I01 * S2xy + I11 * S2yy;
    float Q00 = A00 * I00 + A01 * I01, Q01 = A00 * I01 + A01 * I11, Q11 = A10 * I01 + A11 * I11;
    float gV00 = 0.5f * (Q00 - S0 * I00), gV01 = 0.5f * (Q01 - S0 * I01), gV11 = 0.5f * (Q11 - S0 * I11);
    float gJ00 = 2.0f * (gV00 * J00 * Sg0);
    float gJ01 = 2.0f * (gV00 * J01 * Sg1 + gV01 * J11 * Sg1);
    float gJ11 = 2.0f * (gV01 * J01 * Sg1 + gV11 * J11 * Sg1);
    float gsd0 = 2.0f * sdv[0] * (J00 * J00 * gV00);
    float gsd1 = 2.0f * sdv[1] * (J01 * J01 * gV00 + 2.0f * J01 * J11 * gV01 + J11 * J11 * gV11);
    float gal = -gJ00 / (al * al) + gJ01 * be / (al * al * ga) - S0 / al;
    float gbe = -gJ01 / (al * ga);
    float gga = gJ01 * be / (al * ga * ga) - gJ11 / (ga * ga) - S0 / ga;
    float nxt1[3], t1xu0[3], gt1[3], gu0[3], gnv[3];
    cross3(n, t1, nxt1);
    cross3(t1, u0, t1xu0);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        gt1[i] = gbe * u0[i] + gga * u1[i];
        gu0[i] = gbe * t1[i] + gga * nxt1[i];
        gnv[i] = gga * t1xu0[i];
    }
    float gdu = dot3c(gu0, u0), gt0[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) gt0[i] = (gu0[i] - gdu * u0[i]) / al + gal * u0[i];
    float gpv[3] = {-gt0[0] - gt1[0], -gt0[1] - gt1[1], -gt0[2] - gt1[2]};
    float gk0 = dot3c(gt0, x0), gk1 = dot3c(gt1, x1);
    float gc = gk0 / D0 + gk1 / D1;
    float gD0 = -gk0 * c / (D0 * D0), gD1 = -gk1 * c / (D1 * D1);
    float gx00 = k0 * gt0[0] + gD0 * n[0], gx01 = k0 * gt0[1] + gD0 * n[1];
    float gx10 = k1 * gt1[0] + gD1 * n[0], gx11 = k1 * gt1[1] + gD1 * n[1];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        gnv[i] += gD0 * x0[i] + gD1 * x1[i] + gc * p[i];
        gpv[i] += gc * n[i];
    }
    float gS0 = M1x - (gx00 + gx10) / f;
    float gS1 = M1y + (gx01 + gx11) / f;
    float iz = 1.0f / p[2];
    gpv[0] += gS0 * (-f * iz);
    gpv[1] += gS1 * (f * iz);
    gpv[2] += (gS0 * p[0] - gS1 * p[1]) * f * iz * iz;
    if (CLAMP) {
        const float div = row_divisor(sqrtf(gpv[0] * gpv[0] + gpv[1] * gpv[1] + gpv[2] * gpv[2]));
#pragma unroll
        for (int i = 0; i < 3; ++i) gpv[i] = clean(gpv[i] / div);
    }
    gp_out[3 * o] = gpv[0]; gp_out[3 * o + 1] = gpv[1]; gp_out[3 * o + 2] = gpv[2];
    if (gn_out) { gn_out[3 * o] = gnv[0]; gn_out[3 * o + 1] = gnv[1]; gn_out[3 * o + 2] = gnv[2]; }
    if (!sum_sd) {
        if (CLAMP) {
            const float div = row_divisor(sqrtf(gsd0 * gsd0 + gsd1 * gsd1));
            gsd0 = clean(gsd0 / div);
            gsd1 = clean(gsd1 / div);
        }
        gs_out[2 * so] = gsd0;
        gs_out[2 * so + 1] = gsd1;
    } else {
        atomicAdd(&gs_out[2 * so], gsd0);
        atomicAdd(&gs_out[2 * so + 1], gsd1);
    }
}

// ewa_chain over the used pairs of a block's range; zeros everywhere else.
// sum_sd: the std-devs are shared by several views (their gradient buffer was
// zeroed, contributions are added).
template <int PER, bool CLAMP>
__global__ void __launch_bounds__(kPairThreads) k_ewa_chain(int N, bool sum_sd, float W, float H, float f,
                                                            const float* __restrict__ pts,
                                                            const float* __restrict__ nrm,
                                                            const float* __restrict__ sd, int sdB, float sm,
                                                            const unsigned* __restrict__ used,
                                                            const float4* __restrict__ stats,
                                                            float* __restrict__ gp, float* __restrict__ gn,
                                                            float* __restrict__ gs) {
    __shared__ PairList<PER> list;
    const size_t view = (size_t)N * blockIdx.y;
    const int base = blockIdx.x * kPairThreads * PER;
    const int here = min(N - base, kPairThreads * PER);
    for (int i = threadIdx.x; i < 3 * here; i += kPairThreads) {
        gp[3 * (view + base) + i] = 0.0f;
        if (gn) gn[3 * (view + base) + i] = 0.0f;
    }
    if (!sum_sd)
        for (int i = threadIdx.x; i < 2 * here; i += kPairThreads) gs[2 * ((sdB > 1 ? view : 0) + base) + i] = 0.0f;
    const int count = gather_pairs<PER>(list, used, base, N);  // (synchronises the block)
    for (int i = threadIdx.x; i < count; i += kPairThreads) {
        const int x = base + list.at[i];
        const size_t o = view + x;
        ewa_chain<CLAMP>(x, o, sum_sd, W, H, f, pts, nrm, sd, sdB, sm, stats[2 * o], stats[2 * o + 1], gp, gn, gs);
    }
}

// The post-processing of std-dev gradients summed over views.
__global__ void k_clamp_std(int N, float* __restrict__ gs) {
    int x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= N) return;
    float a = gs[2 * (size_t)x], b = gs[2 * (size_t)x + 1];
    const float div = row_divisor(sqrtf(a * a + b * b));
    gs[2 * (size_t)x] = clean(a / div);
    gs[2 * (size_t)x + 1] = clean(b / div);
}

// ----------------------------------------------------- fused render pass
// One thread per pixel runs splatting.forward, filtering.forward and
// interpolation.forward on its K samples (splattingCuda.cu:18-66,
// zSortingCuda.cu:11-62, interpolationCuda.cu:5-46): EWA weight of each
// sample from its pair's Gaussian constants, depth along the pixel ray,
// stable depth order, front-to-back blend, and the blended attributes.  The
// same device functions in the same order as the three separate kernels, so
// weights, depth weights and image are bit-identical to them; the (B,W,H,K)
// intermediates are written once (the autograd needs them) and never read
// back.
//
// What bounds them is the gather of a pixel's samples from the pairs of its
// view: every loop over up to 16 samples is unrolled, so that all of them are
// in flight together, and the rest is kept short (uds_composite.cuh).
// 1024^2, K = 8, a fifth of the samples valid: forward 48 us, backward 73 us;
// with rolled loops over arrays in local memory and the integer blend and ray
// 130 and 183 us.  Columns of shared memory and a packed order kept by
// insertion, still rolled, took 100 and 161 us there, and more than local
// memory where every sample is valid (1.54 against 1.17 ms at 16 views of
// 256^2); unrolled 4 views of 512^2 and 300k splats, all samples valid, take
// 273 against 467 us forward.

// The K indices of a pixel: -1 where there is no sample.  Returns whether
// there is one.  vec: 16-byte loads (K a multiple of four, aligned).
template <int KMAX>
__device__ __forceinline__ bool load_ids(const int* __restrict__ idx, int K, int N, bool vec, int* id) {
    using S = Samples<KMAX>;
    if (S::kUnrolled && vec) {
#pragma unroll
        for (int k = 0; k < KMAX; k += 4) {
            const int4 v = k < K ? *reinterpret_cast<const int4*>(idx + k) : make_int4(-1, -1, -1, -1);
            id[k] = v.x;
            id[k + 1] = v.y;
            id[k + 2] = v.z;
            id[k + 3] = v.w;
        }
    } else {
#pragma unroll S::kUnroll
        for (int k = 0; k < S::end(K); ++k) id[k] = S::on(k, K) ? idx[k] : -1;
    }
    bool any = false;
#pragma unroll S::kUnroll
    for (int k = 0; k < S::end(K); ++k) {
        if (id[k] >= N) id[k] = -1;
        any |= id[k] >= 0;
    }
    return any;
}
template <int KMAX>
__device__ __forceinline__ void load_row(const float* __restrict__ in, int K, bool vec, float* x) {
    using S = Samples<KMAX>;
    if (S::kUnrolled && vec) {
#pragma unroll
        for (int k = 0; k < KMAX; k += 4) {
            const float4 v = k < K ? *reinterpret_cast<const float4*>(in + k) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            x[k] = v.x;
            x[k + 1] = v.y;
            x[k + 2] = v.z;
            x[k + 3] = v.w;
        }
    } else {
#pragma unroll S::kUnroll
        for (int k = 0; k < S::end(K); ++k) x[k] = S::on(k, K) ? in[k] : 0.0f;
    }
}
template <int KMAX>
__device__ __forceinline__ void store_row(float* __restrict__ out, int K, bool vec, const float* x) {
    using S = Samples<KMAX>;
    if (S::kUnrolled && vec) {
#pragma unroll
        for (int k = 0; k < KMAX; k += 4)
            if (k < K) *reinterpret_cast<float4*>(out + k) = make_float4(x[k], x[k + 1], x[k + 2], x[k + 3]);
    } else {
#pragma unroll S::kUnroll
        for (int k = 0; k < S::end(K); ++k)
            if (S::on(k, K)) out[k] = x[k];
    }
}

// Depth of a sample along the pixel ray (sample_depth) with the pair's plane
// offset p . n from its constants.
__device__ __forceinline__ float pair_depth(const float* dir, const float* n, float pn) {
    float d = fdiv(pn, dot3(dir, n));
    return d > 0.0f ? d : kZmax;
}

// Each sample's Gaussian, its offset from the screen point, and its depth
// rank (empty ones: 0 at kZmax).
template <int KMAX>
__device__ __forceinline__ void pixel_samples(int K, int W, int H, int i, int j, size_t view, const int* id, float f,
                                              const float4* __restrict__ consts, const float* __restrict__ nrm,
                                              float* G, float* dx, float* dy, int* rank) {
    using S = Samples<KMAX>;
    const float px = (float)i, py = (float)j;
    float dir[3], dist[KMAX];
    pixel_ray((float)W, (float)H, f, px, py, dir);
#pragma unroll S::kUnroll
    for (int k = 0; k < S::end(K); ++k) {
        G[k] = 0.0f;
        dist[k] = S::on(k, K) ? kZmax : __int_as_float(0x7f800000);
        if (id[k] >= 0) {
            const size_t o = view + id[k];
            const float4 c0 = consts[2 * o], c1 = consts[2 * o + 1];
            const float n[3] = {nrm[3 * o], nrm[3 * o + 1], nrm[3 * o + 2]};
            G[k] = ewa_gauss(c0, c1, px, py, &dx[k], &dy[k]);
            dist[k] = pair_depth(dir, n, c1.w);
        }
    }
    depth_ranks<KMAX>(K, dist, rank);
}

// Four channels (cn of them) of a splat's attributes; wide: one 16-byte load.
__device__ __forceinline__ void load_channels(const float* __restrict__ a, int cn, bool wide, float* x) {
    if (wide) {
        const float4 v = *reinterpret_cast<const float4*>(a);
        x[0] = v.x;
        x[1] = v.y;
        x[2] = v.z;
        x[3] = v.w;
    } else {
#pragma unroll
        for (int c = 0; c < 4; ++c) x[c] = c < cn ? a[c] : 0.0f;
    }
}

template <int KMAX>
__global__ void __launch_bounds__(kRenderThreads) k_render_forward(
    int row0, int rows, int W, int H, int K, bool vec, const int* __restrict__ idx, const float4* __restrict__ consts,
    int N, float f, const float* __restrict__ nrm, int aB, int C, const float* __restrict__ attr, bool wide,
    float* __restrict__ w_out, float* __restrict__ dw_out, float* __restrict__ img) {
    using S = Samples<KMAX>;
    UDS_RANKED(ws);
    const unsigned at = blockIdx.x * kRenderThreads + threadIdx.x, b = blockIdx.y;
    if (at >= (unsigned)(rows * H)) return;
    const int i = row0 + (int)(at / (unsigned)H), j = (int)(at % (unsigned)H);
    const size_t pix = (size_t)j + (size_t)H * ((size_t)i + (size_t)W * b);
    const size_t e = (size_t)K * pix, view = (size_t)N * b;
    int id[KMAX];
    float fw[KMAX];
    const bool any = load_ids<KMAX>(idx + e, K, N, vec, id);
    if (any) {
        float w[KMAX], dx[KMAX], dy[KMAX];
        int rank[KMAX];
        pixel_samples<KMAX>(K, W, H, i, j, view, id, f, consts, nrm, w, dx, dy, rank);
#pragma unroll S::kUnroll
        for (int k = 0; k < S::end(K); ++k) {
            w[k] = id[k] >= 0 ? fminf(w[k], 1.0f) : 0.0f;
            ws[rank[k]] = w[k];
        }
        store_row<KMAX>(w_out + e, K, vec, w);
        blend_ranked<KMAX>(K, ws, ws);
#pragma unroll S::kUnroll
        for (int k = 0; k < S::end(K); ++k) fw[k] = ws[rank[k]];
    } else {
#pragma unroll S::kUnroll
        for (int k = 0; k < S::end(K); ++k) fw[k] = 0.0f;
        store_row<KMAX>(w_out + e, K, vec, fw);
    }
    store_row<KMAX>(dw_out + e, K, vec, fw);
    const size_t aoff = aB > 1 ? view : 0;
#pragma unroll 1
    for (int c0 = 0; c0 < C; c0 += 4) {
        const int cn = min(4, C - c0);
        float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (any) {
#pragma unroll S::kUnroll
            for (int k = 0; k < S::end(K); ++k) {
                if (id[k] < 0) continue;
                float a[4];
                load_channels(attr + (size_t)C * ((size_t)id[k] + aoff) + c0, cn, wide, a);
#pragma unroll
                for (int c = 0; c < 4; ++c) acc[c] = fadd(acc[c], fmul(fw[k], a[c]));
            }
        }
#pragma unroll
        for (int c = 0; c < 4; ++c)
            if (c < cn) img[(size_t)C * pix + c0 + c] = acc[c];
    }
}

// Adds x * v[0..cn) to the cn <= 4 floats at out, by the widest vector
// atomics that the address allows (wide: all four, on 16 bytes).
__device__ __forceinline__ void add_channels(float* __restrict__ out, int cn, bool wide, const float* v, float x) {
    if (wide) {
        atomicAdd(reinterpret_cast<float4*>(out), make_float4(v[0] * x, v[1] * x, v[2] * x, v[3] * x));
    } else if ((reinterpret_cast<size_t>(out) & 7) == 0) {
        if (cn >= 2) atomicAdd(reinterpret_cast<float2*>(out), make_float2(v[0] * x, v[1] * x));
        else atomicAdd(out, v[0] * x);
        if (cn == 4) atomicAdd(reinterpret_cast<float2*>(out + 2), make_float2(v[2] * x, v[3] * x));
        else if (cn == 3) atomicAdd(out + 2, v[2] * x);
    } else {
        atomicAdd(out, v[0] * x);
        if (cn >= 3) atomicAdd(reinterpret_cast<float2*>(out + 1), make_float2(v[1] * x, v[2] * x));
        else if (cn == 2) atomicAdd(out + 1, v[1] * x);
        if (cn == 4) atomicAdd(out + 3, v[3] * x);
    }
}

// The backward of the fused pass per pixel: interpolation.backward (weight
// gradient per sample, attribute gradient scattered), plus any gradient that
// reaches the depth weights directly; filtering.backward through the
// recomputed depth order and blend; and the EWA gradient statistics of
// k_ewa_stats (gated on the unclamped weight <= 1), plus any gradient that
// reaches the EWA weights directly.  k_ewa_chain then finishes the splat
// gradients.  Same arithmetic per sample as the separate kernels; the
// scattered sums are atomic, as there.
template <int KMAX>
__global__ void __launch_bounds__(kRenderThreads) k_render_backward(
    int row0, int rows, int W, int H, int K, bool vec, const float* __restrict__ gimg,
    const float* __restrict__ gdw_in, const float* __restrict__ gw_in, const int* __restrict__ idx,
    const float* __restrict__ weights, const float4* __restrict__ consts, int N, float f,
    const float* __restrict__ nrm, int aB, int C, const float* __restrict__ attr, float* __restrict__ ga, bool wide,
    float4* __restrict__ stats) {
    using S = Samples<KMAX>;
    UDS_RANKED(w);
    UDS_RANKED(t);  // depth weights, then the numerators of the blend's gradient, then that gradient
    const unsigned at = blockIdx.x * kRenderThreads + threadIdx.x, b = blockIdx.y;
    if (at >= (unsigned)(rows * H)) return;
    const int i = row0 + (int)(at / (unsigned)H), j = (int)(at % (unsigned)H);
    const size_t pix = (size_t)j + (size_t)H * ((size_t)i + (size_t)W * b);
    const size_t e = (size_t)K * pix, view = (size_t)N * b;
    int id[KMAX], rank[KMAX];
    if (!load_ids<KMAX>(idx + e, K, N, vec, id)) return;
    float G[KMAX], dx[KMAX], dy[KMAX], fw[KMAX], acc[KMAX];
    load_row<KMAX>(weights + e, K, vec, fw);
    pixel_samples<KMAX>(K, W, H, i, j, view, id, f, consts, nrm, G, dx, dy, rank);
#pragma unroll S::kUnroll
    for (int k = 0; k < S::end(K); ++k) {
        w[rank[k]] = fw[k];
        acc[k] = 0.0f;
    }
    blend_ranked<KMAX>(K, w, t);
#pragma unroll S::kUnroll
    for (int k = 0; k < S::end(K); ++k) fw[k] = S::on(k, K) ? t[rank[k]] : 0.0f;
    // interpolation.backward with the depth weights fw
    const float* g = gimg + (size_t)C * pix;
    const size_t aoff = aB > 1 ? view : 0;
#pragma unroll 1
    for (int c0 = 0; c0 < C; c0 += 4) {
        const int cn = min(4, C - c0);
        float gc[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) gc[c] = c < cn ? g[c0 + c] : 0.0f;
#pragma unroll S::kUnroll
        for (int k = 0; k < S::end(K); ++k) {
            if (id[k] < 0) continue;
            const size_t ao = (size_t)C * ((size_t)id[k] + aoff) + c0;
            float a[4];
            load_channels(attr + ao, cn, wide, a);
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[k] = fadd(acc[k], fmul(gc[c], a[c]));
            add_channels(ga + ao, cn, wide, gc, fw[k]);
        }
    }
    // filtering.backward and the EWA statistics
#pragma unroll S::kUnroll
    for (int k = 0; k < S::end(K); ++k) {
        if (!S::on(k, K)) continue;
        if (gdw_in) acc[k] = fadd(acc[k], gdw_in[e + k]);
        t[rank[k]] = fmul(acc[k], fw[k]);
    }
    blend_gradients<KMAX>(K, w, t);
#pragma unroll S::kUnroll
    for (int k = 0; k < S::end(K); ++k) {
        if (id[k] < 0 || !(G[k] <= 1.0f)) continue;
        const float gk = gw_in ? fadd(t[rank[k]], gw_in[e + k]) : t[rank[k]];
        const float gg = gk * G[k];
        if (gg == 0.0f) continue;
        const size_t o = view + id[k];
        atomicAdd(&stats[2 * o], make_float4(gg, gg * dx[k], gg * dy[k], gg * dx[k] * dx[k]));
        atomicAdd(reinterpret_cast<float2*>(&stats[2 * o + 1]), make_float2(gg * dx[k] * dy[k], gg * dy[k] * dy[k]));
    }
}

}  // namespace uds

using namespace uds;

static size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

// Workspace: Gaussian constants (2 float4 per pair), gradient statistics (2
// float4 per pair), one mark per pair.
extern "C" size_t uds_splat_workspace_size(int B, int N) {
    return align256(sizeof(float4) * 2 * (size_t)B * N) * 2 + align256(4 * (size_t)mark_words(N) * B);
}

static int check_splat_args(int B, int W, int H, int K, int std_batch, int N) {
    if (B <= 0 || W <= 0 || H <= 0 || K <= 0 || N < 0) return UDS_ERR_ARGUMENT;
    if (std_batch != 1 && std_batch != B) return UDS_ERR_ARGUMENT;
    return UDS_OK;
}

static bool aligned16(const void* a, const void* b = nullptr, const void* c = nullptr) {
    return ((reinterpret_cast<size_t>(a) | reinterpret_cast<size_t>(b) | reinterpret_cast<size_t>(c)) & 15) == 0;
}

// Pairs per block of the kernels over (view, splat) pairs: 1024, or 256 where
// that would leave the GPU's 152 SMs without a block.
static bool few_pairs(int B, int N) { return (size_t)cdiv(N, 4 * kPairThreads) * B < 304; }

// Gaussian constants, gradient statistics and flags of the workspace.
struct SplatWs {
    float4 *consts, *stats;
    unsigned* used;
};
static SplatWs splat_ws(int B, int N, void* workspace) {
    char* p = reinterpret_cast<char*>(workspace);
    size_t half = align256(sizeof(float4) * 2 * (size_t)B * N);
    return {reinterpret_cast<float4*>(p), reinterpret_cast<float4*>(p + half),
            reinterpret_cast<unsigned*>(p + 2 * half)};
}

// Marks of the sampled pairs (zeroed first).
static int mark_sampled(int B, size_t S, int N, const int32_t* indices, unsigned* used, cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(used, 0, 4 * (size_t)mark_words(N) * B, s);
    // the splats in one bit map of at most 128 KB, or in up to four
    constexpr int kRange = 1 << 20;
    const int ranges = (int)(((long long)N + kRange - 1) / kRange), range = ranges > 1 ? kRange : 32 * mark_words(N);
    if (S >= 32768 && ranges <= 4) {
        // about two blocks per SM in all, of at least 16384 samples
        size_t blocks = 304 / ((size_t)B * ranges), most = (S + 16383) / 16384;
        if (blocks > most) blocks = most;
        if (blocks < 1) blocks = 1;
        const bool vec = S % 4 == 0 && aligned16(indices);
        const size_t chunk = ((S + blocks - 1) / blocks + 3) / 4 * 4, bytes = (size_t)range / 8;
        const dim3 grid(cdiv(S, chunk), B, ranges);
        auto kernel = vec ? k_ewa_mark<true> : k_ewa_mark<false>;
        // (the largest map's size, whatever this one's: the attribute is the
        // function's, and another thread may be between this and its launch)
        if (e == cudaSuccess && bytes > 48 * 1024)
            e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kRange / 8);
        if (e == cudaSuccess) kernel<<<grid, kMarkThreads, bytes, s>>>(S, chunk, indices, N, range, used);
    } else if (e == cudaSuccess) {
        k_ewa_mark_direct<<<dim3(cdiv(S, 256), B), 256, 0, s>>>(S, indices, N, used);
    }
    if (e != cudaSuccess) { set_last_error(e); return UDS_ERR_CUDA; }
    return launch_status();
}

// Marks of the sampled pairs and their Gaussian constants; with stats, their
// gradient statistics zeroed.
static int sampled_consts(int B, int W, int H, int K, float focal, const int32_t* indices, const float* points,
                          const float* normals, int std_batch, int N, const float* std_devs, float smoothing,
                          const SplatWs& ws, bool stats, cudaStream_t s) {
    int st = mark_sampled(B, (size_t)W * H * K, N, indices, ws.used, s);
    if (st) return st;
    float4* z = stats ? ws.stats : nullptr;
    if (few_pairs(B, N))
        k_ewa_consts<1><<<dim3(cdiv(N, kPairThreads), B), kPairThreads, 0, s>>>(
            N, (float)W, (float)H, focal, points, normals, std_devs, std_batch, smoothing, ws.used, ws.consts, z);
    else
        k_ewa_consts<4><<<dim3(cdiv(N, 4 * kPairThreads), B), kPairThreads, 0, s>>>(
            N, (float)W, (float)H, focal, points, normals, std_devs, std_batch, smoothing, ws.used, ws.consts, z);
    return launch_status();
}

// The splat gradients from the statistics.  clamp: with the reference's
// post-processing of point and std-dev gradients.
template <bool CLAMP>
static int splat_gradients(int B, int W, int H, float focal, const float* points, const float* normals, int std_batch,
                           int N, const float* std_devs, float smoothing, const SplatWs& ws, float* gp, float* gn,
                           float* gs, cudaStream_t s) {
    const bool sum_sd = std_batch == 1 && B > 1;
    if (sum_sd) {
        cudaError_t e = cudaMemsetAsync(gs, 0, sizeof(float) * 2 * (size_t)N, s);
        if (e != cudaSuccess) { set_last_error(e); return UDS_ERR_CUDA; }
    }
    if (few_pairs(B, N))
        k_ewa_chain<1, CLAMP><<<dim3(cdiv(N, kPairThreads), B), kPairThreads, 0, s>>>(
            N, sum_sd, (float)W, (float)H, focal, points, normals, std_devs, std_batch, smoothing, ws.used, ws.stats,
            gp, gn, gs);
    else
        k_ewa_chain<4, CLAMP><<<dim3(cdiv(N, 4 * kPairThreads), B), kPairThreads, 0, s>>>(
            N, sum_sd, (float)W, (float)H, focal, points, normals, std_devs, std_batch, smoothing, ws.used, ws.stats,
            gp, gn, gs);
    if (CLAMP && sum_sd) {
        k_clamp_std<<<cdiv(N, 256), 256, 0, s>>>(N, gs);
        return launch_status(2);
    }
    return launch_status();
}

extern "C" int uds_splat_forward(int B, int W, int H, int K, float focal, const int32_t* indices,
                                 const float* points, const float* normals, int std_batch, int N,
                                 const float* std_devs, float smoothing, float* weights,
                                 void* workspace, size_t workspace_bytes, void* stream) {
    int st = check_splat_args(B, W, H, K, std_batch, N);
    if (st) return st;
    if (!indices || !weights) return UDS_ERR_ARGUMENT;
    if (workspace_bytes < uds_splat_workspace_size(B, N) || (N > 0 && !workspace)) return UDS_ERR_WORKSPACE;
    cudaStream_t s = as_stream(stream);
    SplatWs ws = splat_ws(B, N, workspace);
    if (N > 0 && (st = sampled_consts(B, W, H, K, focal, indices, points, normals, std_batch, N, std_devs, smoothing,
                                      ws, false, s)))
        return st;
    k_ewa_forward<<<dim3(cdiv(H, 64), W, B), 64, 0, s>>>(B, W, H, K, indices, ws.consts, N, weights);
    return launch_status();
}

template <bool CLAMP>
static int splat_backward(int B, int W, int H, int K, float focal, const float* grad, const int32_t* indices,
                          const float* points, const float* normals, int std_batch, int N, const float* std_devs,
                          float smoothing, float* gp, float* gn, float* gs, void* workspace, size_t workspace_bytes,
                          void* stream) {
    int st = check_splat_args(B, W, H, K, std_batch, N);
    if (st) return st;
    if (!grad || !indices) return UDS_ERR_ARGUMENT;
    if (workspace_bytes < uds_splat_workspace_size(B, N) || (N > 0 && !workspace)) return UDS_ERR_WORKSPACE;
    if (N == 0) return UDS_OK;
    cudaStream_t s = as_stream(stream);
    SplatWs ws = splat_ws(B, N, workspace);
    if ((st = sampled_consts(B, W, H, K, focal, indices, points, normals, std_batch, N, std_devs, smoothing, ws, true,
                             s)))
        return st;
    k_ewa_stats<<<dim3(cdiv(H, 64), W, B), 64, 0, s>>>(B, W, H, K, grad, indices, ws.consts, N, ws.stats);
    if ((st = launch_status())) return st;
    return splat_gradients<CLAMP>(B, W, H, focal, points, normals, std_batch, N, std_devs, smoothing, ws, gp, gn, gs,
                                  s);
}

extern "C" int uds_splat_backward(int B, int W, int H, int K, float focal, const float* grad,
                                  const int32_t* indices, const float* points, const float* normals,
                                  int std_batch, int N, const float* std_devs, float smoothing,
                                  float* grad_points, float* grad_normals, float* grad_std_devs,
                                  void* workspace, size_t workspace_bytes, void* stream) {
    return splat_backward<false>(B, W, H, K, focal, grad, indices, points, normals, std_batch, N, std_devs, smoothing,
                                 grad_points, grad_normals, grad_std_devs, workspace, workspace_bytes, stream);
}

extern "C" int uds_splat_gradients(int B, int W, int H, int K, float focal, const float* grad,
                                   const int32_t* indices, const float* points, const float* normals, int std_batch,
                                   int N, const float* std_devs, float smoothing, float* grad_points,
                                   float* grad_std_devs, void* workspace, size_t workspace_bytes, void* stream) {
    return splat_backward<true>(B, W, H, K, focal, grad, indices, points, normals, std_batch, N, std_devs, smoothing,
                                grad_points, nullptr, grad_std_devs, workspace, workspace_bytes, stream);
}

// Launches over the pixels of every view, rows at a time where a view has
// 2^31 pixels or more.
#define UDS_RENDER_DISPATCH(KERNEL, ...)                                                                \
    do {                                                                                                \
        const int most = H < (1 << 30) ? ((1 << 30) / H) : 1;                                           \
        for (int row0 = 0; row0 < W; row0 += most) {                                                    \
            const int rows = W - row0 < most ? W - row0 : most;                                         \
            dim3 grid(cdiv((size_t)rows * H, kRenderThreads), B);                                       \
            if (K <= 8) KERNEL<8><<<grid, kRenderThreads, 0, s>>>(row0, rows, __VA_ARGS__);             \
            else if (K <= 16) KERNEL<16><<<grid, kRenderThreads, 0, s>>>(row0, rows, __VA_ARGS__);      \
            else if (K <= 32) KERNEL<32><<<grid, kRenderThreads, 0, s>>>(row0, rows, __VA_ARGS__);      \
            else KERNEL<64><<<grid, kRenderThreads, 0, s>>>(row0, rows, __VA_ARGS__);                   \
        }                                                                                               \
    } while (0)

extern "C" int uds_render_fused_forward(int B, int W, int H, int K, float focal, const int32_t* indices,
                                        const float* points, const float* normals, int std_batch, int N,
                                        const float* std_devs, float smoothing, int aB, int C,
                                        const float* attribute, float* weights, float* depth_weights, float* image,
                                        void* workspace, size_t workspace_bytes, void* stream) {
    int st = check_splat_args(B, W, H, K, std_batch, N);
    if (st) return st;
    if (K > kMaxK || C <= 0 || (aB != 1 && aB != B) || !indices || !weights || !depth_weights || !image ||
        (N > 0 && (!points || !normals || !std_devs || !attribute)))
        return UDS_ERR_ARGUMENT;
    if (workspace_bytes < uds_splat_workspace_size(B, N) || (N > 0 && !workspace)) return UDS_ERR_WORKSPACE;
    cudaStream_t s = as_stream(stream);
    SplatWs ws = splat_ws(B, N, workspace);
    if (N > 0 && (st = sampled_consts(B, W, H, K, focal, indices, points, normals, std_batch, N, std_devs, smoothing,
                                      ws, false, s)))
        return st;
    const bool vec = K % 4 == 0 && aligned16(indices, weights, depth_weights);
    const bool wide = C % 4 == 0 && aligned16(attribute);
    UDS_RENDER_DISPATCH(k_render_forward, W, H, K, vec, indices, ws.consts, N, focal, normals, aB, C, attribute, wide,
                        weights, depth_weights, image);
    return launch_status();
}

template <bool CLAMP>
static int render_backward(int B, int W, int H, int K, float focal, const float* grad_image,
                           const float* grad_depth_weights, const float* grad_weights, const int32_t* indices,
                           const float* weights, const float* points, const float* normals, int std_batch, int N,
                           const float* std_devs, float smoothing, int aB, int C, const float* attribute,
                           float* grad_points, float* grad_normals, float* grad_std_devs, float* grad_attribute,
                           void* workspace, size_t workspace_bytes, void* stream) {
    int st = check_splat_args(B, W, H, K, std_batch, N);
    if (st) return st;
    if (K > kMaxK || C <= 0 || (aB != 1 && aB != B) || !grad_image || !indices || !weights)
        return UDS_ERR_ARGUMENT;
    if (N > 0 && (!points || !normals || !std_devs || !attribute || !grad_points || (!CLAMP && !grad_normals) ||
                  !grad_std_devs || !grad_attribute))
        return UDS_ERR_ARGUMENT;
    if (workspace_bytes < uds_splat_workspace_size(B, N) || (N > 0 && !workspace)) return UDS_ERR_WORKSPACE;
    if (N == 0) return UDS_OK;
    cudaStream_t s = as_stream(stream);
    SplatWs ws = splat_ws(B, N, workspace);
    cudaError_t e = cudaMemsetAsync(grad_attribute, 0, sizeof(float) * (size_t)aB * N * C, s);
    if (e != cudaSuccess) { set_last_error(e); return UDS_ERR_CUDA; }
    if ((st = sampled_consts(B, W, H, K, focal, indices, points, normals, std_batch, N, std_devs, smoothing, ws, true,
                             s)))
        return st;
    const bool vec = K % 4 == 0 && aligned16(indices, weights);
    const bool wide = C % 4 == 0 && aligned16(attribute, grad_attribute);
    UDS_RENDER_DISPATCH(k_render_backward, W, H, K, vec, grad_image, grad_depth_weights, grad_weights, indices,
                        weights, ws.consts, N, focal, normals, aB, C, attribute, grad_attribute, wide, ws.stats);
    if ((st = launch_status())) return st;
    return splat_gradients<CLAMP>(B, W, H, focal, points, normals, std_batch, N, std_devs, smoothing, ws, grad_points,
                                  grad_normals, grad_std_devs, s);
}

extern "C" int uds_render_fused_backward(int B, int W, int H, int K, float focal, const float* grad_image,
                                         const float* grad_depth_weights, const float* grad_weights,
                                         const int32_t* indices, const float* weights, const float* points,
                                         const float* normals, int std_batch, int N, const float* std_devs,
                                         float smoothing, int aB, int C, const float* attribute, float* grad_points,
                                         float* grad_normals, float* grad_std_devs, float* grad_attribute,
                                         void* workspace, size_t workspace_bytes, void* stream) {
    return render_backward<false>(B, W, H, K, focal, grad_image, grad_depth_weights, grad_weights, indices, weights,
                                  points, normals, std_batch, N, std_devs, smoothing, aB, C, attribute, grad_points,
                                  grad_normals, grad_std_devs, grad_attribute, workspace, workspace_bytes, stream);
}

extern "C" int uds_render_fused_gradients(int B, int W, int H, int K, float focal, const float* grad_image,
                                          const float* grad_depth_weights, const float* grad_weights,
                                          const int32_t* indices, const float* weights, const float* points,
                                          const float* normals, int std_batch, int N, const float* std_devs,
                                          float smoothing, int aB, int C, const float* attribute, float* grad_points,
                                          float* grad_std_devs, float* grad_attribute, void* workspace,
                                          size_t workspace_bytes, void* stream) {
    return render_backward<true>(B, W, H, K, focal, grad_image, grad_depth_weights, grad_weights, indices, weights,
                                 points, normals, std_batch, N, std_devs, smoothing, aB, C, attribute, grad_points,
                                 nullptr, grad_std_devs, grad_attribute, workspace, workspace_bytes, stream);
}
