// Per-sample scatter / per-splat gather (pixelgather.scatter / gather,
// splatting/extensions/pixelGatherCuda.cu:7-152): the consumers of the
// sampled indices right after the render (visibility counting in cleanup.py:41,
// PixelScatterGather in extensions/__init__.py:407-437).
//
// scatter: out (B,W,H,K,C) = values (B,N,C) at each sample's splat, 0 where
//          the index is -1 (or outside [0, N)).
// gather:  out (B,N,C) = sum over the samples of splat j of values (B,W,H,K,C).
//   atomic mode: lanes of a warp that hold the same splat first combine their
//     values (__match_any_sync + shuffles), then one atomic per group and
//     channel; the order of additions is not fixed (like the reference).
//   deterministic mode: the valid samples are packed in sample order and
//     stably radix-sorted by splat (so each splat's samples stay in sample
//     order, however many there are), and one thread sums its splat's values
//     in that order: the result is bit-identical to a sequential sum in
//     sample order.
#include "uds_common.cuh"
#include "uds_radix.cuh"

namespace uds {

// One thread per sample copies its splat's C values, four (16 bytes) at a time
// where WIDE (C a multiple of four, both arrays aligned).
template <bool WIDE>
__global__ void k_pixel_scatter(size_t S, size_t per_view, int N, int C, const int* __restrict__ idx,
                                const float* __restrict__ values, float* __restrict__ out) {
    const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= S) return;
    const int id = idx[t];
    const bool ok = id >= 0 && id < N;
    const float* v = values + (ok ? ((size_t)id + (size_t)N * (t / per_view)) * C : 0);
    float* o = out + t * (size_t)C;
    if (WIDE) {
        for (int c = 0; c < C; c += 4)
            *reinterpret_cast<float4*>(o + c) =
                ok ? *reinterpret_cast<const float4*>(v + c) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    } else {
        for (int c = 0; c < C; ++c) o[c] = ok ? v[c] : 0.0f;
    }
}

// Fewer than four channels: one thread per four samples, whose 4 C values are
// C 16-byte stores (idx and out aligned, per_view a multiple of four).  Bound
// by the writes: 1024 x 768, K = 8, C = 3 25 us, 37 with one sample
// per thread.
template <int C>
__global__ void k_pixel_scatter4(size_t S, size_t per_view, int N, const int* __restrict__ idx,
                                 const float* __restrict__ values, float* __restrict__ out) {
    const size_t t = 4 * ((size_t)blockIdx.x * blockDim.x + threadIdx.x);
    if (t >= S) return;
    const int4 i4 = *reinterpret_cast<const int4*>(idx + t);
    const int id[4] = {i4.x, i4.y, i4.z, i4.w};
    const float* view = values + (size_t)N * (t / per_view) * C;
    __align__(16) float x[4 * C];
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int c = 0; c < C; ++c)
            x[q * C + c] = id[q] >= 0 && id[q] < N ? view[(size_t)id[q] * C + c] : 0.0f;
#pragma unroll
    for (int c = 0; c < C; ++c)
        reinterpret_cast<float4*>(out + t * C)[c] = make_float4(x[4 * c], x[4 * c + 1], x[4 * c + 2], x[4 * c + 3]);
}

__global__ void k_pixel_gather_atomic(size_t S, size_t per_view, int N, int C, const int* __restrict__ idx,
                                      const float* __restrict__ values, float* __restrict__ out) {
    size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    bool live = t < S;
    int id = live ? idx[t] : -1;
    size_t key = (live && id >= 0 && id < N) ? (size_t)id + (size_t)N * (t / per_view) : ~(size_t)0;
    unsigned peers = __match_any_sync(0xffffffffu, key);
    int lane = threadIdx.x & 31;
    int leader = __ffs(peers) - 1;
    for (int c = 0; c < C; ++c) {
        float v = (key != ~(size_t)0) ? values[t * (size_t)C + c] : 0.0f;
        // sum over the group of lanes with the same splat
        float s = 0.0f;
        unsigned m = peers;
        while (m) {
            int src = __ffs(m) - 1;
            m &= m - 1;
            s += __shfl_sync(peers, v, src);
        }
        if (lane == leader && key != ~(size_t)0) atomicAdd(&out[key * (size_t)C + c], s);
    }
}

// Deterministic mode.
struct GatherState {
    unsigned n;   // valid samples
    int failed;   // a wait ran out (see look_back): the sums are NaN
    unsigned ticket[6];
};
constexpr int kGatherPasses = 4;  // of 10 bits at most: 32-bit splat keys

// Samples per thread of the packing and of the sort's passes.  Larger tiles
// than the tree build's: there are more of them than the GPU holds blocks, and
// the words of tiles that are looked back at are most of the sort's traffic.
constexpr int kPackItems = 32, kPackTile = kPackItems * kTileThreads;
constexpr int kSortItems = 16, kSortTile = kSortItems * kTileThreads;

// The valid samples of a tile, packed behind those of the tiles before it:
// (splat key, sample) pairs, and the digits of their keys.  The indices are
// read twice (the second time from the L1), which keeps no key in a register.
__global__ void __launch_bounds__(kTileThreads) k_pixel_pack(size_t S, size_t per_view, int N, int passes,
                                                             const int* __restrict__ idx, GatherState* gs,
                                                             unsigned long long* status, unsigned* hist,
                                                             unsigned* __restrict__ keys,
                                                             unsigned* __restrict__ samples) {
    constexpr int kWarps = kTileThreads / 32;
    __shared__ unsigned digits[kGatherPasses * kDigits];
    __shared__ unsigned before[kPackItems * kWarps];
    __shared__ unsigned s_first;
    __shared__ int s_tile, s_failed;
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_tile = (int)atomicAdd(&gs->ticket[kGatherPasses], 1u);
    for (int d = threadIdx.x; d < passes * kDigits; d += kTileThreads) digits[d] = 0;
    __syncthreads();
    if (s_tile >= (int)gridDim.x) return;  // (a scratch that another call uses at the same time)
    const size_t first = (size_t)s_tile * kPackTile + threadIdx.x;
    auto sample = [&](int r) {
        const size_t t = first + r * kTileThreads;
        return t < S ? idx[t] : -1;
    };
    auto key_of = [&](int id, int r) {
        return (unsigned)((size_t)id + (size_t)N * ((first + r * kTileThreads) / per_view));
    };
#pragma unroll 8
    for (int r = 0; r < kPackItems; ++r) {
        const int id = sample(r);
        const bool ok = id >= 0 && id < N;
        if (ok) {
            const unsigned key = key_of(id, r);
            for (int q = 0; q < passes; ++q)
                atomicAdd(&digits[q * kDigits + ((key >> (q * kDigitBits)) & (kDigits - 1))], 1u);
        }
        const unsigned ball = __ballot_sync(full, ok);
        if (lane == 0) before[r * kWarps + warp] = __popc(ball);
    }
    __syncthreads();
    if (warp == 0) {
        unsigned long long at;
        unsigned total;
        const bool ok = tile_places<kPackItems * kWarps>(before, status, s_tile, at, total);
        if (lane == 0) {
            s_first = (unsigned)at;
            s_failed = !ok;
            if (!ok) wait_failed(&gs->failed);
            else if (s_tile == (int)gridDim.x - 1) gs->n = (unsigned)at + total;
        }
    }
    __syncthreads();
    if (s_failed) return;
#pragma unroll 8
    for (int r = 0; r < kPackItems; ++r) {
        const int id = sample(r);
        const bool ok = id >= 0 && id < N;
        const unsigned ball = __ballot_sync(full, ok);
        if (ok) {
            const unsigned at = s_first + before[r * kWarps + warp] + __popc(ball & ((1u << lane) - 1u));
            keys[at] = key_of(id, r);
            samples[at] = (unsigned)(first + r * kTileThreads);
        }
    }
    for (int d = threadIdx.x; d < passes * kDigits; d += kTileThreads)
        if (digits[d]) atomicAdd(&hist[d], digits[d]);
}

template <typename Word>
__global__ void __launch_bounds__(kTileThreads) k_pixel_sort(int pass, GatherState* gs,
                                                             const unsigned* __restrict__ hist, Word* status,
                                                             const unsigned* __restrict__ kin,
                                                             const unsigned* __restrict__ vin,
                                                             unsigned* __restrict__ kout, unsigned* __restrict__ vout) {
    const unsigned n = failed_yet(&gs->failed) ? 0u : gs->n;
    if ((size_t)blockIdx.x * kSortTile >= n) return;
    if (!sort_tile<kSortItems, Word>(n, pass * kDigitBits, &gs->ticket[pass], hist, status, kin, vin, kout, vout) &&
        threadIdx.x == 0)
        wait_failed(&gs->failed);
}

// First and one past the last of each splat's sorted samples (0, 0: none).
__global__ void k_pixel_bounds(const GatherState* gs, const unsigned* __restrict__ keys, uint2* __restrict__ bounds) {
    const size_t n = gs->failed ? 0 : gs->n, step = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += step) {
        const unsigned k = keys[i];
        if (i == 0 || keys[i - 1] != k) bounds[k].x = (unsigned)i;
        if (i + 1 == n || keys[i + 1] != k) bounds[k].y = (unsigned)i + 1u;
    }
}

// One thread per splat sums its bucket (already in sample order), up to four
// channels at a time, the next samples' values on their way.  A gather that
// failed is all NaN.
__global__ void k_pixel_sum(const GatherState* gs, size_t M, int C, const uint2* __restrict__ bounds, const unsigned* __restrict__ slots,
                            const float* __restrict__ values, float* __restrict__ out) {
    size_t key = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (key >= M) return;
    const uint2 range = bounds[key];
    if (gs->failed) {
        for (int c = 0; c < C; ++c) out[key * (size_t)C + c] = __int_as_float(0x7fc00000);
        return;
    }
    for (int c0 = 0; c0 < C; c0 += 4) {
        const int cn = min(4, C - c0);
        float s[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 4
        for (unsigned i = range.x; i < range.y; ++i) {
            const float* v = values + (size_t)slots[i] * C + c0;
#pragma unroll
            for (int c = 0; c < 4; ++c)
                if (c < cn) s[c] = __fadd_rn(s[c], v[c]);
        }
#pragma unroll
        for (int c = 0; c < 4; ++c)
            if (c < cn) out[key * (size_t)C + c0 + c] = s[c];
    }
}

cudaError_t pixel_wait_failures(unsigned* count) { return cudaMemcpyFromSymbol(count, g_wait_failures, sizeof(*count)); }

}  // namespace uds

using namespace uds;

extern "C" int uds_pixel_scatter(int B, int W, int H, int K, const int32_t* indices, int N, int C,
                                 const float* values, float* out, void* stream) {
    if (B <= 0 || W <= 0 || H <= 0 || K <= 0 || N < 0 || C <= 0 || !indices || !out || (N > 0 && !values))
        return UDS_ERR_ARGUMENT;
    size_t per_view = (size_t)W * H * K, S = per_view * B;
    cudaStream_t s = as_stream(stream);
    const bool aligned = ((reinterpret_cast<size_t>(indices) | reinterpret_cast<size_t>(values) |
                           reinterpret_cast<size_t>(out)) & 15) == 0;
    if (aligned && C < 4 && per_view % 4 == 0) {
        if (C == 1) k_pixel_scatter4<1><<<cdiv(S / 4, 256), 256, 0, s>>>(S, per_view, N, indices, values, out);
        else if (C == 2) k_pixel_scatter4<2><<<cdiv(S / 4, 256), 256, 0, s>>>(S, per_view, N, indices, values, out);
        else k_pixel_scatter4<3><<<cdiv(S / 4, 256), 256, 0, s>>>(S, per_view, N, indices, values, out);
    } else if (aligned && C % 4 == 0) {
        k_pixel_scatter<true><<<cdiv(S, 256), 256, 0, s>>>(S, per_view, N, C, indices, values, out);
    } else {
        k_pixel_scatter<false><<<cdiv(S, 256), 256, 0, s>>>(S, per_view, N, C, indices, values, out);
    }
    return launch_status();
}

// Deterministic-mode scratch: what is zeroed first (state, digit counts,
// look-back words of the packing and of the sort's passes, the splats' bounds),
// then two (key, sample) pair buffers.
struct GatherWs {
    GatherState* state;
    unsigned* hist;
    unsigned long long* pack_status;
    char* sort_status;
    size_t sort_bytes;  // look-back words of one pass
    uint2* bounds;
    size_t zeroed;
    unsigned *ka, *va, *kb, *vb;
    int passes;
    bool wide;  // 64-bit words: 2^30 samples or more
    size_t bytes;
};

static GatherWs gather_layout(size_t M, size_t S, char* base) {
    GatherWs g{};
    size_t off = 0;
    auto take = [&](size_t n) {
        char* p = base ? base + off : nullptr;
        off += (n + 255) & ~(size_t)255;
        return p;
    };
    int bits = 1;
    while (bits < 32 && M > 1 && (M - 1) >> bits) ++bits;
    g.passes = (bits + kDigitBits - 1) / kDigitBits;
    g.wide = S >= (1ull << 30);
    g.sort_bytes = (g.wide ? 8 : 4) * (size_t)cdiv(S, kSortTile) * kDigits;
    g.state = reinterpret_cast<GatherState*>(take(sizeof(GatherState)));
    g.hist = reinterpret_cast<unsigned*>(take(4 * kGatherPasses * kDigits));
    g.pack_status = reinterpret_cast<unsigned long long*>(take(8 * (size_t)cdiv(S, kPackTile)));
    g.sort_status = take(g.sort_bytes * g.passes);
    g.bounds = reinterpret_cast<uint2*>(take(8 * M));
    g.zeroed = off;
    g.ka = reinterpret_cast<unsigned*>(take(4 * S));
    g.va = reinterpret_cast<unsigned*>(take(4 * S));
    g.kb = reinterpret_cast<unsigned*>(take(4 * S));
    g.vb = reinterpret_cast<unsigned*>(take(4 * S));
    g.bytes = off;
    return g;
}

extern "C" size_t uds_pixel_gather_workspace_size(int B, int W, int H, int K, int N) {
    if (B <= 0 || W <= 0 || H <= 0 || K <= 0 || N < 0) return 0;
    return gather_layout((size_t)B * N, (size_t)B * W * H * K, nullptr).bytes;
}

extern "C" int uds_pixel_gather(int B, int W, int H, int K, const int32_t* indices, int N, int C,
                                const float* values, float* out, int deterministic, void* workspace,
                                size_t workspace_bytes, void* stream) {
    if (B <= 0 || W <= 0 || H <= 0 || K <= 0 || N < 0 || C <= 0 || !indices || !values || (N > 0 && !out))
        return UDS_ERR_ARGUMENT;
    cudaStream_t s = as_stream(stream);
    size_t per_view = (size_t)W * H * K, S = per_view * B, M = (size_t)B * N;
    if (M == 0) return UDS_OK;
    if (S >= (1ull << 32)) return UDS_ERR_ARGUMENT;
    if (!deterministic) {
        cudaError_t e = cudaMemsetAsync(out, 0, sizeof(float) * M * C, s);
        if (e != cudaSuccess) { set_last_error(e); return UDS_ERR_CUDA; }
        k_pixel_gather_atomic<<<cdiv(S, 256), 256, 0, s>>>(S, per_view, N, C, indices, values, out);
        return launch_status();
    }
    if (!workspace || workspace_bytes < uds_pixel_gather_workspace_size(B, W, H, K, N)) return UDS_ERR_WORKSPACE;
    GatherWs g = gather_layout(M, S, reinterpret_cast<char*>(workspace));
    cudaError_t e = cudaMemsetAsync(g.state, 0, g.zeroed, s);
    if (e != cudaSuccess) { set_last_error(e); return UDS_ERR_CUDA; }
    // the number of valid samples stays on the device
    const unsigned tiles = cdiv(S, kSortTile);
    k_pixel_pack<<<cdiv(S, kPackTile), kTileThreads, 0, s>>>(S, per_view, N, g.passes, indices, g.state, g.pack_status,
                                                             g.hist, g.ka, g.va);
    unsigned *ki = g.ka, *vi = g.va, *ko = g.kb, *vo = g.vb;
    for (int pass = 0; pass < g.passes; ++pass) {
        const unsigned* hist = g.hist + pass * kDigits;
        char* status = g.sort_status + g.sort_bytes * pass;
        if (g.wide)
            k_pixel_sort<unsigned long long><<<tiles, kTileThreads, 0, s>>>(
                pass, g.state, hist, reinterpret_cast<unsigned long long*>(status), ki, vi, ko, vo);
        else
            k_pixel_sort<unsigned><<<tiles, kTileThreads, 0, s>>>(pass, g.state, hist,
                                                                  reinterpret_cast<unsigned*>(status), ki, vi, ko, vo);
        unsigned* t = ki; ki = ko; ko = t;
        t = vi; vi = vo; vo = t;
    }
    k_pixel_bounds<<<cdiv(S, 256) < 1216 ? cdiv(S, 256) : 1216, 256, 0, s>>>(g.state, ki, g.bounds);
    k_pixel_sum<<<cdiv(M, 128), 128, 0, s>>>(g.state, M, C, g.bounds, vi, values, out);
    return launch_status(3 + g.passes);
}
