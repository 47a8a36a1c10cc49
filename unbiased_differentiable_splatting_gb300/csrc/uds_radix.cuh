// Single-pass prefix sums and a stable LSD radix sort of (key, value) pairs
// built on them, shared by the tree build (Morton keys) and the deterministic
// per-splat gather (splat keys).
#pragma once
#include "uds_common.cuh"

namespace uds {

constexpr int kDigitBits = 10, kDigits = 1 << kDigitBits;
constexpr int kTileThreads = 256;

// ------------------------------------------------- decoupled look-back
// Prefix sums over a kernel's tiles in the kernel itself (D. Merrill and M.
// Garland, "Single-pass parallel prefix scan with decoupled look-back", NVIDIA
// NVR-2016-002): a block publishes its tile's sum, adds up those of the tiles
// before it until it meets one with its prefix, and publishes its own.  Tiles
// are numbered by a ticket when their block starts, so the ones waited for
// have all started, and publish before they wait.  A wait still ends after
// kWait looks: the caller then marks its result as failed and counts that
// (uds_wait_failures).  What marks it failed is read once per block (failed_yet):
// another block of the same launch may set it between two threads' reads.  A word
// holds state and sum together, so no other memory is ordered by it.
#ifndef UDS_WAIT_LOOKS
#define UDS_WAIT_LOOKS (1 << 20)
#endif
constexpr int kWait = UDS_WAIT_LOOKS;
static __device__ unsigned g_wait_failures;  // of this file's kernels, since the library was loaded
__device__ __forceinline__ void wait_failed(int* failed) {
    atomicExch(failed, 1);
    atomicAdd(&g_wait_failures, 1u);
}
// By a whole block: *failed, the same for all of its threads.
__device__ __forceinline__ bool failed_yet(const int* failed) {
    return __syncthreads_or(threadIdx.x == 0 && *(volatile const int*)failed) != 0;
}
constexpr unsigned long long kSumReady = 1ull << 62, kPrefixReady = 2ull << 62, kSumMask = kSumReady - 1ull;

// By a whole warp: the sum of the tiles before `tile`; false if a wait ran out.
__device__ __forceinline__ bool look_back(unsigned long long* status, int tile, unsigned long long sum,
                                          unsigned long long& before) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    volatile unsigned long long* words = status;
    before = 0;
    if (lane == 0) words[tile] = (tile ? kSumReady : kPrefixReady) | sum;
    if (tile == 0) return true;
    for (int t = tile - 1;; t -= 32) {
        unsigned long long x = kPrefixReady;  // before the first tile
        if (t - lane >= 0) {
            int looks = 0;
            do x = words[t - lane];
            while (!(x >> 62) && ++looks < kWait);
        }
        __syncwarp();
        if (__any_sync(full, !(x >> 62))) return false;
        const unsigned known = __ballot_sync(full, (x >> 62) == 2);
        unsigned long long part = lane <= (known ? __ffs(known) - 1 : 31) ? x & kSumMask : 0ull;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(full, part, o);
        before += part;
        if (known) break;
    }
    if (lane == 0) words[tile] = kPrefixReady | (before + sum);
    return true;
}

// The places of GROUPS groups of flagged items of a tile (round r, warp w at
// r * 8 + w) behind those of the tiles before it: counts in, places out
// (relative to `first`).  By a whole warp; false where a wait ran out.
template <int GROUPS>
__device__ __forceinline__ bool tile_places(unsigned* groups, unsigned long long* status, int tile,
                                            unsigned long long& first, unsigned& total) {
    constexpr int kPer = GROUPS / 32;
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    unsigned sum = 0;
#pragma unroll
    for (int q = 0; q < kPer; ++q) sum += groups[kPer * lane + q];
    unsigned incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(full, incl, o);
        if (lane >= o) incl += y;
    }
    unsigned at = incl - sum;
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
        const unsigned c = groups[kPer * lane + q];
        groups[kPer * lane + q] = at;
        at += c;
    }
    total = __shfl_sync(full, incl, 31);
    return look_back(status, tile, total, first);
}

// One stable pass over (key, value) pairs, ITEMS per thread: a warp owns a run
// of 32 ITEMS items of its block's tile, lane l holds item 32 r + l of it in
// round r, so (round, lane) order is item order and per-warp running counts
// give a stable rank.  A digit's items of a tile go behind those of the
// smaller digits (from the counts of all keys) and of the tiles before it
// (look-back, one word per tile and digit, four digits per thread and four
// tiles at a time).  Called by whole blocks, at least as many as there are
// tiles; ticket: tiles started.  Word: 32 bits for fewer than 2^30 pairs, else
// 64.  False where a wait ran out.
//
// Bound by the latency of its few steps while the tiles fit the GPU (500k
// pairs 18 us, 23 with one tile looked at per step), then by the traffic of the
// words looked at, for which fewer, larger tiles are better (1.9M pairs: 37 us
// with 16 items per thread, 46 with 8).
template <int ITEMS, typename Word>
__device__ __forceinline__ bool sort_tile(unsigned n, int shift, unsigned* ticket, const uint32_t* __restrict__ hist,
                                          Word* status, const uint32_t* __restrict__ kin,
                                          const uint32_t* __restrict__ vin, uint32_t* __restrict__ kout,
                                          uint32_t* __restrict__ vout) {
    constexpr int kWarps = kTileThreads / 32, kPer = kDigits / kTileThreads;
    static_assert(kPer == 4, "four digits per thread");
    __shared__ unsigned wcnt[kWarps][kDigits];
    __shared__ __align__(16) unsigned goff[kDigits];
    __shared__ unsigned wsum[kWarps];
    __shared__ int s_tile, s_failed;
    const unsigned full = 0xffffffffu;
    constexpr int kState = 8 * sizeof(Word) - 2;  // 1: a sum, 2: a prefix
    constexpr Word kMask = ((Word)1 << kState) - 1;
    volatile Word* words = status;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        s_tile = (int)atomicAdd(ticket, 1u);
        s_failed = 0;
    }
    for (int d = lane; d < kDigits; d += 32) wcnt[warp][d] = 0;
    __syncthreads();
    const int tile = s_tile;
    if ((unsigned long long)tile * (ITEMS * kTileThreads) >= n) return true;  // (uniform over the block)
    uint32_t key[ITEMS], val[ITEMS];
    unsigned rank[ITEMS];
    const unsigned lt = (1u << lane) - 1u;
    const unsigned base = (unsigned)tile * (ITEMS * kTileThreads) + warp * 32 * ITEMS;
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
        const unsigned i = base + r * 32 + lane;
        key[r] = i < n ? kin[i] : 0u;
        val[r] = i < n ? vin[i] : 0u;
    }
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
        const bool ok = base + r * 32 + lane < n;
        const unsigned dig = ok ? (key[r] >> shift) & (kDigits - 1) : kDigits;
        const unsigned peers = __match_any_sync(full, dig);
        const unsigned before = ok ? wcnt[warp][dig] : 0u;
        rank[r] = before + __popc(peers & lt);
        __syncwarp();
        if (ok && (peers & lt) == 0) wcnt[warp][dig] = before + __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    unsigned count[kPer];
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
        const int d = threadIdx.x + q * kTileThreads;
        unsigned run = 0;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            const unsigned c = wcnt[w][d];
            wcnt[w][d] = run;
            run += c;
        }
        count[q] = run;
        words[(size_t)tile * kDigits + d] = ((Word)(tile ? 1 : 2) << kState) | run;
    }
    {  // where each digit's items begin
        const uint4 h = reinterpret_cast<const uint4*>(hist)[threadIdx.x];
        const unsigned sum = h.x + h.y + h.z + h.w;
        unsigned incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(full, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) wsum[warp] = incl;
        __syncthreads();
        unsigned first = incl - sum;
        for (int w = 0; w < warp; ++w) first += wsum[w];
        reinterpret_cast<uint4*>(goff)[threadIdx.x] = make_uint4(first, first + h.x, first + h.x + h.y,
                                                                 first + h.x + h.y + h.z);
    }
    unsigned before[kPer] = {0u, 0u, 0u, 0u};
    if (tile) {
        int at[kPer] = {tile - 1, tile - 1, tile - 1, tile - 1};  // < 0: done
        int looks = 0;
        while ((at[0] >= 0 || at[1] >= 0 || at[2] >= 0 || at[3] >= 0) && looks < kWait) {
            constexpr int kAhead = 4;  // tiles looked at together
            Word x[kPer][kAhead];
#pragma unroll
            for (int q = 0; q < kPer; ++q)
#pragma unroll
                for (int a = 0; a < kAhead; ++a)
                    x[q][a] = at[q] >= a ? words[(size_t)(at[q] - a) * kDigits + threadIdx.x + q * kTileThreads] : 0;
#pragma unroll
            for (int q = 0; q < kPer; ++q) {
                bool on = at[q] >= 0;
#pragma unroll
                for (int a = 0; a < kAhead; ++a) {
                    on = on && (x[q][a] >> kState);  // (no state yet: look again)
                    if (on) {
                        before[q] += (unsigned)(x[q][a] & kMask);
                        at[q] = (x[q][a] >> kState) == 2 ? -1 : at[q] - 1;
                        on = at[q] >= 0;
                    }
                }
            }
            ++looks;
        }
        if (looks >= kWait) {
            s_failed = 1;  // (and no prefix: the tiles behind fail too)
        } else {
#pragma unroll
            for (int q = 0; q < kPer; ++q)
                words[(size_t)tile * kDigits + threadIdx.x + q * kTileThreads] =
                    ((Word)2 << kState) | (before[q] + count[q]);
        }
    }
    __syncthreads();
    if (s_failed) return false;
#pragma unroll
    for (int q = 0; q < kPer; ++q) goff[threadIdx.x + q * kTileThreads] += before[q];
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ITEMS; ++r)
        if (base + r * 32 + lane < n) {
            const unsigned dig = (key[r] >> shift) & (kDigits - 1);
            const unsigned pos = goff[dig] + wcnt[warp][dig] + rank[r];
            kout[pos] = key[r];
            vout[pos] = val[r];
        }
    return true;
}

}  // namespace uds
