// sampling.sample (sampling.cpp:48-94, samplingCuda.cu:197-321) on one GPU:
// per view, the FMM tree over the projected splat centres and the per-pixel
// sequential-Poisson descent that draws K splat indices.
//
// Pipeline (all on the caller's stream, no host synchronisation; sizes that
// depend on a view are read on the device).  Every kernel of the build covers
// up to kBatch views (blockIdx.y), so that a step over many views makes as
// many launches as one over a single view:
//   1 k_bandwidth   isotropic bandwidth h (mean over splats, fixed point);
//                   the last block sets the cull bounds
//   2 k_cull        screen point, visibility, 30-bit Morton key; the visible
//                   splats packed in index order, their digits counted
//   3 k_sort_pass   LSD radix sort of the visible ones, 3 x 10 bits, stable,
//                   one launch per pass (decoupled look-back)
//   4 k_tree        leaves and Karras (2012) radix tree over 64-bit keys
//                   (key << 32 | rank)
//   5 k_bottomup    atomic fan-in: boxes, count-weighted centres, adaptive
//                   Hermite degree, truncation radius
//   6 k_p2m         coefficient offsets in a fixed pool (look-back scan over
//                   the nodes), then the Hermite moments, each coefficient
//                   summed over the node's leaves in Morton order
//                   (deterministic, no atomics)
//   7 k_finish_view statistics, order of the image's tiles
//   8 k_sample      per pixel: ceil(sqrt(K)) rounds of greedy capacity
//                   descent + order sampling on u/p
//
// Every float operation on this path is spelled with an exact-rounding
// intrinsic (or is an IEEE-exact library op: sqrt, division, fma), so the
// Morton keys, the tree, the FGT masses and the sampled indices equal the CPU
// oracle's bit for bit given the same inputs and uniforms.
#include <type_traits>

#include <cuda_bf16.h>

#include "uds_ewa.cuh"
#include "uds_radix.cuh"
#include "uds_tc.cuh"

namespace uds {

constexpr int kBatch = 32;  // views per launch of the build
constexpr int kPasses = 3;  // of 10 bits: 30-bit Morton keys
constexpr int kTileItems = 8, kTile = kTileItems * kTileThreads;  // splats per thread and block of a scan
constexpr int kNodeTile = 128;  // nodes per block of k_p2m

struct ViewState {            // per-view device scalars (lives in the workspace)
    unsigned long long hsum;  // fixed-point sum of per-splat bandwidths (2^-32 units)
    unsigned long long hcount;
    float h, radius, lo_x, hi_x, lo_y, hi_y, sq;  // sq = sqrt(2 h^2)
    int n;                    // visible splats
    unsigned coef_used;
    float isq;                // 1 / sq (the series' scaled offsets multiply by it)
    int failed;               // a wait ran out: the view samples nothing (see look_back)
    int W, H;                 // of the image the tree was built for
    unsigned ticket[kPasses + 3];  // blocks started: k_sort_pass's, k_cull's, k_p2m's; done: k_bandwidth's
    unsigned deferred[3];     // tiles left for the long tables (LongTables), those taken, blocks done with them
};

// ----------------------------------------------------- order of the tiles
// Pixels take very different times to sample: one at a silhouette, where
// many splats project onto a few pixels, takes ten times the mean, and most
// images are partly empty.  Blocks started in raster order left a third of
// the GPU's slots idle (500k splats at 1024^2: 1.22 ms, stochastic 2.93).  So
// the image is cut into cells of 16 x 16 pixels (larger ones from 2^20 pixels
// on, for at most kCells of them), the visible splats of each cell are
// counted, and the descent's blocks take the cells in order of falling count
// in the cell and its neighbours, to a quarter of a power of two: 0.96 ms,
// stochastic 2.28.  (Cells of 32 x 32 without the neighbours 1.12 and 2.66;
// of 16 x 16 without them 1.10 and 2.56: what is started late and takes long
// sits next to a silhouette.)
constexpr int kCells = 4096;
__host__ __device__ inline int cell_shift(int W, int H) {
    int sh = 4;
    while ((((long long)W - 1) >> sh) + 1 > kCells / ((((long long)H - 1) >> sh) + 1)) ++sh;
    return sh;
}
__host__ __device__ inline int cell_columns(int H, int sh) { return ((H - 1) >> sh) + 1; }
static unsigned cell_blocks(int W, int H, dim3 block) {  // blocks that cover every cell
    const int sh = cell_shift(W, H);
    return (unsigned)(cell_columns(W, sh) * cell_columns(H, sh)) * ((1u << sh) / block.x) * ((1u << sh) / block.y);
}
// The first pixel (row i along W, column j along H) of a block of a view, its
// place among the view's blocks given (cells in their own order where the
// tree was built for an image of another size).
__device__ __forceinline__ void cell_block(const unsigned short* __restrict__ order, const ViewState* vs, int W, int H,
                                           unsigned at, int& i, int& j) {
    const int sh = cell_shift(W, H);
    const unsigned across = (1u << sh) / blockDim.x, per = across * ((1u << sh) / blockDim.y);
    const int cell = vs->W == W && vs->H == H ? order[at / per] : (int)(at / per), columns = cell_columns(H, sh);
    i = ((cell / columns) << sh) + (int)(at % per / across * blockDim.y);
    j = ((cell % columns) << sh) + (int)(at % across * blockDim.x);
}

// ----------------------------------------------------------- workspace
struct Ws {
    ViewState* vs;
    // zeroed before the build, with vs, in one go
    uint32_t* cells;                  // visible splats of each cell
    uint32_t* hist;                   // digits of the visible splats' keys, pass by pass
    unsigned long long* cull_status;  // look-back words of k_cull's tiles,
    unsigned long long* node_status;  // of k_p2m's,
    uint32_t* sort_status;            // and of k_sort_pass's, one per digit
    unsigned* fanin;
    size_t zeroed;                    // bytes from vs on
    unsigned short* order;            // the cells in order of falling count
    uds_view_stats* stats;
    uint32_t *keysA, *idsA, *keysB, *idsB;
    float2* leaf_xy;
    int* leaf_id;
    int4* lnk;
    int* par;
    float4* box;
    float4* cen;
    float* coef;
    size_t coef_cap;
    size_t bytes;
};

static size_t a256(size_t x) { return (x + 255) & ~(size_t)255; }

// Default coefficient pool: 64 floats per splat, at least 2^20, at most the
// 2^26 - 1 that the 26-bit offsets of the node metadata can address (nodes
// past the pool are demoted to subtree walks, as the oracle does).
static int64_t default_pool(int64_t N) {
    int64_t p = N * 64 > (1 << 20) ? N * 64 : (1 << 20);
    return p < (1ll << 26) ? p : (1ll << 26) - 1;
}

static Ws layout(const uds_sample_params* p, char* base) {
    Ws w{};
    size_t N = (size_t)(p->N > 0 ? p->N : 1);
    size_t M = 2 * N;
    size_t tiles = cdiv(N, kTile);
    int64_t pool = p->coef_pool > 0 ? p->coef_pool : default_pool((int64_t)N);
    size_t off = 0;
    auto take = [&](size_t bytes) { size_t o = off; off += a256(bytes); return base ? base + o : nullptr; };
    w.vs = (ViewState*)take(sizeof(ViewState));
    w.cells = (uint32_t*)take(4 * kCells);
    w.hist = (uint32_t*)take(4 * kPasses * kDigits);
    w.cull_status = (unsigned long long*)take(8 * tiles);
    w.node_status = (unsigned long long*)take(8 * cdiv(N, kNodeTile));
    w.sort_status = (uint32_t*)take(4 * kPasses * kDigits * tiles);
    w.fanin = (unsigned*)take(4 * N);
    w.zeroed = off;
    w.order = (unsigned short*)take(2 * kCells);
    w.stats = (uds_view_stats*)take(sizeof(uds_view_stats) * (size_t)(p->B > 0 ? p->B : 1));
    w.keysA = (uint32_t*)take(4 * N);
    w.idsA = (uint32_t*)take(4 * N);
    w.keysB = (uint32_t*)take(4 * N);
    w.idsB = (uint32_t*)take(4 * N);
    w.leaf_xy = (float2*)take(8 * N);
    w.leaf_id = (int*)take(4 * N);
    w.lnk = (int4*)take(16 * M);
    w.par = (int*)take(4 * M);
    w.box = (float4*)take(16 * M);
    w.cen = (float4*)take(16 * M);
    w.coef = (float*)take(4 * (size_t)pool);
    w.coef_cap = (size_t)pool;
    w.bytes = off;
    return w;
}

// The views of one launch: blockIdx.y = k is view first + k, with its tree
// slot bytes after the one before.
struct Batch {
    size_t slot;
    int first, count;
    int W[kBatch], H[kBatch];
    float f[kBatch];
};
template <typename P>
__device__ __forceinline__ P* shifted(P* p, size_t bytes) {
    using C = typename std::conditional<std::is_const<P>::value, const char, char>::type;
    return reinterpret_cast<P*>(reinterpret_cast<C*>(p) + bytes);
}
// Visible splats of a view whose build has not failed (in kernels that cannot
// make it fail; the others: failed_yet).
__device__ __forceinline__ int visible(const ViewState* vs) { return vs->failed ? 0 : vs->n; }

// --------------------------------------------------------- 1 bandwidth
// IsotropicEigenFunctor (samplingCuda.cu:133-162) with the same float /
// double promotions.
__device__ __forceinline__ float splat_bandwidth(float W, float H, float f, const float* p,
                                                 const float* n, const float* sd, float sm) {
    EwaFrame F;
    ewa_frame(W, H, f, p, n, sd, sm, F);
    const float* V = F.V;
    float det = fsub(fmul(V[0], V[3]), fmul(V[1], V[2]));
    float inv = div_via_double(1.0f, det);
    float i0 = fmul(V[3], inv), i1 = fmul(-V[1], inv), i2 = fmul(-V[2], inv), i3 = fmul(V[0], inv);
    float tr = fadd(i0, i3);
    float tt = fmul(tr, tr);
    float root, l1, l2;
    if (fabsf(tr) >= 0x1p-100f && fabsf(tt) >= 0x1p-100f) {
        // 0.25 tt and 0.5 tr are exact in float as in double, so each
        // double operation below has float operands
        root = fsqrt(sub_via_double(fmul(0.25f, tt), fsub(fmul(i0, i3), fmul(i1, i2))));
        l1 = add_via_double(fmul(0.5f, tr), root);
        l2 = sub_via_double(fmul(0.5f, tr), root);
    } else {  // tiny (or NaN) trace: the reference's double sequence
        float idet = fsub(fmul(i0, i3), fmul(i1, i2));
        root = fsqrt((float)dsub(dmul(0.25, (double)tt), (double)idet));
        l1 = (float)dadd(dmul(0.5, (double)tr), (double)root);
        l2 = (float)dsub(dmul(0.5, (double)tr), (double)root);
    }
    float lk = fminf(l1, l2);
    // (float)fmin(1.0, 1.0 / (double)sqrt(lk)): the min commutes with the
    // monotone rounding, and fminf returns 1 for a NaN quotient as fmin does
    return fminf(1.0f, div_via_double(1.0f, fsqrt(lk)));
}

// h (or its override), the cull radius and bounds (samplingCuda.cu:244-258)
__device__ void view_setup(ViewState* vs, unsigned long long hsum, unsigned long long hcount, float override_h,
                           int width, int height, float precision, uds_view_stats* st) {
    const float W = (float)width, H = (float)height;
    float h;
    if (override_h > 0.0f) h = override_h;
    else if (hcount == 0) h = __int_as_float(0x7fc00000);
    else h = (float)ddiv(ddiv(__ull2double_rn(hsum), 4294967296.0), __ull2double_rn(hcount));
    float norm = (float)dmul(2.0 * kPi, (double)fsqrt(h));
    double a = -(double)det_logf(precision);
    double b = (double)det_logf(norm);
    float r = (float)dmul(dmul(1.4142135623730951, (double)h), __dsqrt_rn(dsub(a, b)));
    vs->h = h;
    vs->W = width;
    vs->H = height;
    vs->radius = r;
    vs->lo_x = -r;
    vs->hi_x = fadd(W, r);
    vs->lo_y = -r;
    vs->hi_y = fadd(H, r);
    vs->sq = fsqrt(fmul(fmul(2.0f, h), h));
    vs->isq = fdiv(1.0f, vs->sq);
    st->h = h;
    st->radius = r;
    st->n_visible = 0;
    st->n_coefs = 0;
    st->demoted = 0;
    st->overflow = 0;
    st->reserved[0] = 0;
}

// PER x 256 splats per block: one pair of additions to the view's sums per
// block.  One per warp was what bounded the kernel: additions to one address
// take about 1 ns each (2M splats: 93 us; 500k: 24, now 16).  The last block
// done sets the view up.
template <int PER>
__global__ void __launch_bounds__(kTileThreads) k_bandwidth(int N, Batch bt, const float* __restrict__ pts,
                                                            const float* __restrict__ nrm,
                                                            const float* __restrict__ sd, int std_batch, float sm,
                                                            const float* __restrict__ h_override, float precision,
                                                            ViewState* vs, uds_view_stats* stats) {
    __shared__ unsigned long long part[2][kTileThreads / 32];
    const int k = blockIdx.y, view = bt.first + k;
    const float W = (float)bt.W[k], H = (float)bt.H[k], f = bt.f[k];
    vs = shifted(vs, bt.slot * k);
    pts += 3 * (size_t)N * view;
    nrm += 3 * (size_t)N * view;
    if (std_batch > 1) sd += 2 * (size_t)N * view;
    unsigned long long s = 0, c = 0;
#pragma unroll 1
    for (int q = 0; q < PER; ++q) {
        const size_t x = (size_t)blockIdx.x * (PER * kTileThreads) + q * kTileThreads + threadIdx.x;
        if (x >= (size_t)N) break;
        float p[3] = {pts[3 * x], pts[3 * x + 1], pts[3 * x + 2]};
        float n[3] = {nrm[3 * x], nrm[3 * x + 1], nrm[3 * x + 2]};
        float d[2] = {sd[2 * x], sd[2 * x + 1]};
        float hk = splat_bandwidth(W, H, f, p, n, d, sm);
        if (isfinite(hk)) {
            s += (unsigned long long)__float2ll_rn(fmul(hk, 4294967296.0f));  // exact: hk <= 1
            c += 1;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        s += __shfl_xor_sync(0xffffffffu, s, o);
        c += __shfl_xor_sync(0xffffffffu, c, o);
    }
    if ((threadIdx.x & 31) == 0) {
        part[0][threadIdx.x >> 5] = s;
        part[1][threadIdx.x >> 5] = c;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < kTileThreads / 32; ++w) {
            s += part[0][w];
            c += part[1][w];
        }
        atomicAdd(&vs->hsum, s);
        atomicAdd(&vs->hcount, c);
        __threadfence();
        if (atomicAdd(&vs->ticket[kPasses + 2], 1u) == gridDim.x - 1) {
            __threadfence();
            view_setup(vs, atomicAdd(&vs->hsum, 0ull), atomicAdd(&vs->hcount, 0ull),
                       h_override ? h_override[view] : 0.0f, bt.W[k], bt.H[k], precision, stats + view);
        }
    }
}

// ------------------------------------------------------- 2 cull + Morton
__device__ __forceinline__ unsigned expand_bits(unsigned v) {
    v = (v * 0x00010001u) & 0xFF0000FFu;
    v = (v * 0x00000101u) & 0x0F00F00Fu;
    v = (v * 0x00000011u) & 0xC30C30C3u;
    v = (v * 0x00000005u) & 0x49249249u;
    return v;
}
__device__ __forceinline__ unsigned morton_coord(float s, float lo, float hi) {
    float src = fdiv(fsub(s, lo), fsub(hi, lo));
    float c = fminf(fmaxf(fmul(src, 1024.0f), 0.0f), 1023.0f);
    return (unsigned)c;
}

// The visible splats of a tile, packed behind those of the tiles before it
// in index order, and the digits of their keys for the sort's passes: the sort
// then moves only what the view sees (of 2M splats in a room an eighth).
__global__ void __launch_bounds__(kTileThreads) k_cull(int N, Batch bt, const float* __restrict__ pts, ViewState* vs,
                                                       unsigned long long* status, uint32_t* hist,
                                                       uint32_t* __restrict__ keys, uint32_t* __restrict__ ids) {
    constexpr int kWarps = kTileThreads / 32;
    __shared__ unsigned digits[kPasses][kDigits];
    __shared__ unsigned before[kTileItems * kWarps];  // visible splats of a round and warp, then those before it
    __shared__ int s_tile, s_first;
    const unsigned full = 0xffffffffu;
    const int k = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const size_t off = bt.slot * k;
    vs = shifted(vs, off);
    status = shifted(status, off);
    hist = shifted(hist, off);
    keys = shifted(keys, off);
    ids = shifted(ids, off);
    pts += 3 * (size_t)N * (bt.first + k);
    if (threadIdx.x == 0) s_tile = (int)atomicAdd(&vs->ticket[kPasses], 1u);
    for (int d = threadIdx.x; d < kPasses * kDigits; d += kTileThreads) digits[0][d] = 0;
    __syncthreads();
    const int tile = s_tile;
    if (tile >= (int)gridDim.x) return;  // (a workspace that another call uses at the same time)
    const float W = (float)bt.W[k], H = (float)bt.H[k], f = bt.f[k];
    const float lx = vs->lo_x, hx = vs->hi_x, ly = vs->lo_y, hy = vs->hi_y;
    unsigned key[kTileItems], ball[kTileItems];
#pragma unroll
    for (int r = 0; r < kTileItems; ++r) {
        const size_t x = (size_t)tile * kTile + r * kTileThreads + threadIdx.x;
        bool vis = false;
        key[r] = 0;
        if (x < (size_t)N) {
            float p[3] = {pts[3 * x], pts[3 * x + 1], pts[3 * x + 2]};
            float s[2];
            screen_point(W, H, f, p, s);
            vis = (p[2] <= 0.0f) && (lx <= s[0]) && (hx >= s[0]) && (ly <= s[1]) && (hy >= s[1]);
            if (vis) {
                key[r] = 2u * expand_bits(morton_coord(s[0], lx, hx)) + expand_bits(morton_coord(s[1], ly, hy));
#pragma unroll
                for (int q = 0; q < kPasses; ++q)
                    atomicAdd(&digits[q][(key[r] >> (q * kDigitBits)) & (kDigits - 1)], 1u);
            }
        }
        ball[r] = __ballot_sync(full, vis);
        if (lane == 0) before[r * kWarps + warp] = __popc(ball[r]);
    }
    __syncthreads();
    if (warp == 0) {
        unsigned long long first;
        unsigned total;
        const bool ok = tile_places<kTileItems * kWarps>(before, status, tile, first, total);
        if (lane == 0) {
            s_first = ok ? (int)first : -1;
            if (!ok) wait_failed(&vs->failed);
            else if (tile == (int)gridDim.x - 1) vs->n = (int)(first + total);
        }
    }
    __syncthreads();
    if (s_first < 0) return;
#pragma unroll
    for (int r = 0; r < kTileItems; ++r)
        if ((ball[r] >> lane) & 1u) {
            const int at = s_first + (int)before[r * kWarps + warp] + __popc(ball[r] & ((1u << lane) - 1u));
            keys[at] = key[r];
            ids[at] = (uint32_t)((size_t)tile * kTile + r * kTileThreads + threadIdx.x);
        }
    for (int d = threadIdx.x; d < kPasses * kDigits; d += kTileThreads)
        if (digits[0][d]) atomicAdd(&hist[d], digits[0][d]);
}

// ---------------------------------------------------------- 3 radix sort
// One pass over every view's visible splats (sort_tile); tiles_max: tiles of
// look-back words per pass.  500k splats: 18 us a pass; 4 passes of 8 bits
// with counts, scans and scatters in launches of their own took 64 us in all.
__global__ void __launch_bounds__(kTileThreads) k_sort_pass(Batch bt, int pass, int tiles_max, ViewState* vs,
                                                            const uint32_t* __restrict__ hist, uint32_t* status,
                                                            const uint32_t* __restrict__ kin,
                                                            const uint32_t* __restrict__ vin,
                                                            uint32_t* __restrict__ kout, uint32_t* __restrict__ vout) {
    const size_t off = bt.slot * blockIdx.y;
    vs = shifted(vs, off);
    const int n = failed_yet(&vs->failed) ? 0 : vs->n;
    if ((long long)blockIdx.x * kTile >= n) return;
    if (!sort_tile<kTileItems, uint32_t>(n, pass * kDigitBits, &vs->ticket[pass], shifted(hist, off) + pass * kDigits,
                             shifted(status, off) + (size_t)pass * tiles_max * kDigits, shifted(kin, off),
                             shifted(vin, off), shifted(kout, off), shifted(vout, off)) &&
        threadIdx.x == 0)
        wait_failed(&vs->failed);
}

// ---------------------------------------------------- 4 leaves + Karras
__device__ __forceinline__ float trunc_radius(float h, float precision, int count) {
    return fsqrt(fmul(fmul(-2.0f, fmul(h, h)), det_logf(fdiv(precision, (float)(unsigned)count))));
}

__device__ __forceinline__ void tree_leaf(int i, int n, int W, int H, float f, const float* __restrict__ pts, float h,
                                          float precision, uint32_t* __restrict__ cells,
                                          const uint32_t* __restrict__ ids, float2* __restrict__ leaf_xy,
                                          int* __restrict__ leaf_id, int4* __restrict__ lnk, int* __restrict__ par,
                                          float4* __restrict__ box, float4* __restrict__ cen) {
    int id = (int)ids[i];
    float p[3] = {pts[3 * (size_t)id], pts[3 * (size_t)id + 1], pts[3 * (size_t)id + 2]};
    float s[2];
    screen_point((float)W, (float)H, f, p, s);
    {  // neighbours in Morton order share their cell: one addition for each group of a warp
        const int sh = cell_shift(W, H);
        const int row = min(max((int)s[0], 0), W - 1) >> sh, column = min(max((int)s[1], 0), H - 1) >> sh;
        const int cell = row * cell_columns(H, sh) + column;
        const unsigned group = __match_any_sync(__activemask(), cell);
        if ((threadIdx.x & 31) == __ffs(group) - 1) atomicAdd(&cells[cell], __popc(group));
    }
    int v = n - 1 + i;
    leaf_xy[i] = make_float2(s[0], s[1]);
    leaf_id[i] = id;
    lnk[v] = make_int4(-1, -1, i, 1);
    if (n == 1) par[v] = -1;  // else the parent writes it
    box[v] = make_float4(s[0], s[1], s[0], s[1]);
    cen[v] = make_float4(s[0], s[1], trunc_radius(h, precision, 1), make_meta(0, 0));
}

__device__ __forceinline__ int cpref(const uint32_t* keys, int n, int i, int j) {
    if (j < 0 || j >= n) return -1;
    unsigned long long a = ((unsigned long long)keys[i] << 32) | (unsigned)i;
    unsigned long long b = ((unsigned long long)keys[j] << 32) | (unsigned)j;
    return __clzll(a ^ b);
}

// determineRange / findSplit (buildRadixTree.cuh:76-167), Karras (2012)
__device__ __forceinline__ void tree_node(int idx, int n, const uint32_t* __restrict__ keys, int4* __restrict__ lnk,
                                          int* __restrict__ par) {
    int lo, hi;
    if (idx == 0) {
        lo = 0; hi = n - 1;
        par[0] = -1;
    } else {
        int dL = cpref(keys, n, idx, idx - 1), dR = cpref(keys, n, idx, idx + 1);
        int d = (dR > dL) ? 1 : -1;
        int dmin = min(dL, dR);
        int lmax = 2;
        while (cpref(keys, n, idx, idx + d * lmax) > dmin) lmax <<= 1;
        int l = 0;
        for (int t = lmax >> 1; t > 0; t >>= 1)
            if (cpref(keys, n, idx, idx + (l + t) * d) > dmin) l += t;
        int j = idx + l * d;
        lo = d < 0 ? j : idx;
        hi = d < 0 ? idx : j;
    }
    int dnode = cpref(keys, n, lo, hi);
    int split = lo, stride = hi - lo;
    do {
        stride = (stride + 1) >> 1;
        int mid = split + stride;
        if (mid < hi && cpref(keys, n, lo, mid) > dnode) split = mid;
    } while (stride > 1);
    int lc = split, rc = split + 1;
    if (lo == split) lc += n - 1;
    if (hi == split + 1) rc += n - 1;
    lnk[idx] = make_int4(lc, rc, lo, hi - lo + 1);
    par[lc] = idx;
    par[rc] = idx;
}

// One thread per leaf and internal node.
__global__ void __launch_bounds__(128) k_tree(int N, Batch bt, const float* __restrict__ pts, const ViewState* vs,
                                              float precision, Ws w) {
    const int i = blockIdx.x * 128 + threadIdx.x, k = blockIdx.y;
    const size_t off = bt.slot * k;
    vs = shifted(vs, off);
    const int n = visible(vs);
    if (i >= n) return;
    const uint32_t* keys = shifted(w.keysA, off);
    int4* lnk = shifted(w.lnk, off);
    int* par = shifted(w.par, off);
    tree_leaf(i, n, bt.W[k], bt.H[k], bt.f[k], pts + 3 * (size_t)N * (bt.first + k), vs->h, precision,
              shifted(w.cells, off), shifted(w.idsA, off), shifted(w.leaf_xy, off), shifted(w.leaf_id, off), lnk, par,
              shifted(w.box, off), shifted(w.cen, off));
    if (i < n - 1) tree_node(i, n, keys, lnk, par);
}

// ------------------------------------------------------------ 5 bottom-up
// hermiteError (hermitefmm.cuh:184-195) with integer powers as products: the
// bound at degree ph from rp = r^ph and root = sqrt(ph!), a = nr / (1 - r)^2.
__device__ __forceinline__ float hermite_error(float a, float rp, float root) {
    float b = fdiv(rp, root);
    float c = fmul(b, b);
    float d = fmul(fmul(2.0f, fsub(1.0f, rp)), b);
    return fmul(a, fadd(c, d));
}

// Adds 1; what this thread wrote before is visible to the thread that adds
// next, and what the one before it wrote to this thread.
__device__ __forceinline__ unsigned arrive(unsigned* p) {
    unsigned old;
    asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(old) : "l"(p) : "memory");
    return old;
}

// InternalNodeFunctor (buildDynamicRadixTree.cuh:155-221): the second thread
// to reach a node merges it.  Child centres are read at [child] (the
// reference indexes expansionPoints[child] instead of [2*child]).  Bound by
// the latency of one leaf-to-root path: a step waits for the counter and then
// for the sibling's record; the links are fetched beside the counter, the own
// record is still in registers, and a child's count is its parent's less its
// sibling's.  500k splats: 74 us; with fences, every record and the
// children's links read again, and the error bound's powers, factorials and
// roots computed for each degree 126 us.
__global__ void __launch_bounds__(128) k_bottomup(Batch bt, const ViewState* vs, float precision, int max_degree,
                                                  Ws w) {
    __shared__ float root[kMaxDegree + 1];
    if (threadIdx.x <= kMaxDegree) root[threadIdx.x] = fsqrt(facf(threadIdx.x));
    __syncthreads();
    const size_t off = bt.slot * blockIdx.y;
    vs = shifted(vs, off);
    const int i = blockIdx.x * 128 + threadIdx.x, n = visible(vs);
    if (i >= n || n < 2) return;
    const int4* __restrict__ lnk = shifted(w.lnk, off);
    const int* __restrict__ par = shifted(w.par, off);
    float4 *box = shifted(w.box, off), *cen = shifted(w.cen, off);
    unsigned* fanin = shifted(w.fanin, off);
    const float h = vs->h;
    int v = n - 1 + i, count = 1, p = par[v];
    float4 b = box[v], c = cen[v];
    while (p >= 0) {
        const int4 L = lnk[p];
        const int next = par[p];
        if (arrive(&fanin[p]) == 0) return;
        const bool left = L.x == v;
        const int other = left ? L.y : L.x;
        const float4 bo = __ldcg(&box[other]), co = __ldcg(&cen[other]);
        const float4 ba = left ? b : bo, bb = left ? bo : b, ca = left ? c : co, cb = left ? co : c;
        const int rest = L.w - count;
        const float na = (float)(unsigned)(left ? count : rest), nb = (float)(unsigned)(left ? rest : count);
        const float nc = (float)(unsigned)L.w;
        b = make_float4(fminf(ba.x, bb.x), fminf(ba.y, bb.y), fmaxf(ba.z, bb.z), fmaxf(ba.w, bb.w));
        const float cx = fdiv(fadd(fmul(na, ca.x), fmul(nb, cb.x)), nc);
        const float cy = fdiv(fadd(fmul(na, ca.y), fmul(nb, cb.y)), nc);
        float mn = fmaxf(0.0f, fmaxf(fsub(cx, b.x), fsub(b.z, cx)));
        mn = fmaxf(mn, fmaxf(fsub(cy, b.y), fsub(b.w, cy)));
        const float r = fdiv(mn, h);
        int degree = -1;
        if (r < 1.0f) {
            const float om = fsub(1.0f, r), a = fdiv(nc, fmul(om, om));
            int deg = max(max(meta_degree(ca.w), meta_degree(cb.w)), 0);
            float rp = ipowf(r, (unsigned)deg);
            while (deg <= max_degree && hermite_error(a, rp, root[deg]) > precision) {
                rp = fmul(rp, r);
                ++deg;
            }
            if (deg <= max_degree) degree = deg;
        }
        c = make_float4(cx, cy, trunc_radius(h, precision, L.w), make_meta(0, degree));
        __stcg(&box[p], b);
        __stcg(&cen[p], c);
        v = p;
        count = L.w;
        p = next;
    }
}

// ------------------------------------------- 5b fixed-degree M2M pass
// Fixed-degree mode (no reference counterpart): every internal node stores a
// degree-P Hermite expansion at offset v * (P+1)^2, obtained from its
// children's by the M2M shift instead of summing over its leaves:
//   M_ab(c) = sum_{a' <= a, b' <= b} M_a'b'(c_child) t_{a-a'}(dx) t_{b-b'}(dy),
// t_k(d) = d^k / k!, (dx, dy) = (c_child - c) / sqrt(2 h^2); a leaf child is
// the single moment M_00 = 1 at its own position.  Exact for the truncated
// moments (the moments of the union are polynomial in the shift), so the
// expansions equal the per-leaf sums up to rounding at O(P^3) per node.  The
// node is evaluated through its expansion (degree P) when the adaptive error
// bound holds at some degree <= P (k_bottomup run with max_degree = P), else
// walked (degree -1); the coefficients exist either way for the parent's
// shift.  Same second-arrival fan-in as k_bottomup.
__global__ void k_fixed_assign(ViewState* vs, float4* cen, int P) {
    int v = blockIdx.x * blockDim.x + threadIdx.x;
    int n = visible(vs);
    if (v == 0) vs->coef_used = (unsigned)((n > 1 ? n - 1 : 0) * (P + 1) * (P + 1));
    if (v >= n - 1) return;
    float4 c = cen[v];
    c.w = make_meta(v * (P + 1) * (P + 1), meta_degree(c.w) >= 0 ? P : -1);
    cen[v] = c;
}

template <int P>
__global__ void k_m2m(const ViewState* vs, const int4* __restrict__ lnk, const int* __restrict__ par,
                      const float4* __restrict__ cen, float* coef, unsigned* fanin) {
    constexpr int P1 = P + 1, P2 = P1 * P1;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    int n = visible(vs);
    if (i >= n || n < 2) return;
    float sq = vs->sq;
    int v = n - 1 + i;
    while (true) {
        int p = par[v];
        if (p < 0) break;
        __threadfence();
        if (atomicAdd(&fanin[p], 1u) == 0) return;
        __threadfence();
        int4 L = lnk[p];
        float4 cp = cen[p];
        float acc[P1][P1];
#pragma unroll
        for (int a = 0; a < P1; ++a)
#pragma unroll
            for (int b = 0; b < P1; ++b) acc[a][b] = 0.0f;
#pragma unroll
        for (int side = 0; side < 2; ++side) {
            int c = side ? L.y : L.x;
            float4 cc = cen[c];
            float dx = (cc.x - cp.x) / sq, dy = (cc.y - cp.y) / sq;
            float tx[P1], ty[P1];
            tx[0] = 1.0f;
            ty[0] = 1.0f;
#pragma unroll
            for (int k = 1; k < P1; ++k) {
                tx[k] = tx[k - 1] * dx / (float)k;
                ty[k] = ty[k - 1] * dy / (float)k;
            }
            if (c >= n - 1) {
#pragma unroll
                for (int a = 0; a < P1; ++a)
#pragma unroll
                    for (int b = 0; b < P1; ++b) acc[a][b] = fmaf(tx[a], ty[b], acc[a][b]);
            } else {
                const float* C = coef + (size_t)c * P2;
                float D[P1][P1];  // shift along y first
#pragma unroll
                for (int a = 0; a < P1; ++a)
#pragma unroll
                    for (int b = 0; b < P1; ++b) {
                        float sum = 0.0f;
#pragma unroll
                        for (int bb = 0; bb <= b; ++bb) sum = fmaf(__ldcg(C + a * P1 + bb), ty[b - bb], sum);
                        D[a][b] = sum;
                    }
#pragma unroll
                for (int a = 0; a < P1; ++a)
#pragma unroll
                    for (int b = 0; b < P1; ++b) {
                        float sum = acc[a][b];
#pragma unroll
                        for (int aa = 0; aa <= a; ++aa) sum = fmaf(D[aa][b], tx[a - aa], sum);
                        acc[a][b] = sum;
                    }
            }
        }
        float* out = coef + (size_t)p * P2;
#pragma unroll
        for (int a = 0; a < P1; ++a)
#pragma unroll
            for (int b = 0; b < P1; ++b) __stcg(out + a * P1 + b, acc[a][b]);
        v = p;
    }
}

// ----------------------------------------------------------------- 6 P2M
// shiftLeafHermiteExpansion (hermitefmm.cuh:119-138) summed per node over
// its leaves in Morton order: C_ab = sum_i t_a(s0_i) t_b(s1_i) with
// t_a(s) = s^a / a!, s = (leaf - centre) * (1 / sqrt(2 h^2)).  A warp builds
// one node at a time.  For a chunk of 32 leaves each lane builds one leaf's
// t-tables in shared memory (t_a = (t_{a-1} s) * (1 / a)); each lane then
// owns a block of BR rows x BC columns of C (the block shape depends on the
// degree, so that the blocks of a (p+1)^2 table fit 32 lanes) and adds
// fma(t_a(s0), t_b(s1), C_ab) leaf by leaf: every coefficient is summed in
// leaf order exactly as the oracle's deterministic flavour does, and one
// shared-memory read feeds BR or BC multiply-adds.  A warp takes 32
// consecutive nodes (one coalesced read of their records and links) and
// builds their expansions one after another: one node per warp left the
// kernel waiting on two dependent memory round trips per few hundred
// multiply-adds.  Most nodes have a few leaves and a low degree, for which
// setting a warp up costs more than the sums: up to degree 7 and kSmallNode
// leaves four nodes are built at once.  500k splats: 99 us with the offsets'
// scan, 183 without either.
constexpr int kP2MWarps = 4;
constexpr int kSmallNode = 32;  // (8 and 32 take the same time)
// 1 / a, rounded once at compile time (the oracle uses the same constants)
__constant__ float kInvInt[kMaxDegree + 1] = {0.0f, 1.0f / 1, 1.0f / 2, 1.0f / 3, 1.0f / 4, 1.0f / 5, 1.0f / 6,
                                              1.0f / 7, 1.0f / 8, 1.0f / 9, 1.0f / 10, 1.0f / 11, 1.0f / 12,
                                              1.0f / 13, 1.0f / 14, 1.0f / 15, 1.0f / 16};
constexpr int kTStride = kMaxDegree + 1;  // odd: conflict-free row writes
// rows x columns per lane for p + 1 = 1 .. 17 coefficients per side
__constant__ unsigned char kP2MBlock[kMaxDegree + 2][2] = {
    {1, 1}, {1, 1}, {1, 1}, {1, 1}, {1, 1}, {1, 1}, {1, 2}, {1, 2}, {1, 2},
    {1, 3}, {2, 2}, {2, 3}, {2, 3}, {2, 4}, {2, 4}, {2, 4}, {2, 4}, {3, 4}};

template <int BR, int BC>
__device__ __forceinline__ void p2m_block(const float* tx, const float* ty, int cnt, const int* ra, const int* cb,
                                          float (&acc)[3][4]) {
    for (int j = 0; j < cnt; ++j) {
        float xv[BR], yv[BC];
#pragma unroll
        for (int i = 0; i < BR; ++i) xv[i] = tx[j * kTStride + ra[i]];
#pragma unroll
        for (int k = 0; k < BC; ++k) yv[k] = ty[j * kTStride + cb[k]];
#pragma unroll
        for (int i = 0; i < BR; ++i)
#pragma unroll
            for (int k = 0; k < BC; ++k) acc[i][k] = __fmaf_rn(xv[i], yv[k], acc[i][k]);
    }
}

__global__ void __launch_bounds__(kNodeTile) k_p2m(Batch bt, ViewState* vs, size_t cap, uds_view_stats* stats, Ws w) {
    static_assert(kNodeTile == 32 * kP2MWarps, "a node per thread");
    __shared__ float s_tx[kP2MWarps][32 * kTStride];
    __shared__ float s_ty[kP2MWarps][32 * kTStride];
    __shared__ unsigned s_size[kP2MWarps];
    __shared__ unsigned long long s_first;
    __shared__ int s_tile;
    const unsigned full = 0xffffffffu;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const size_t shift = bt.slot * blockIdx.y;
    vs = shifted(vs, shift);
    const int n = failed_yet(&vs->failed) ? 0 : vs->n;
    const int tiles = (n - 1 + kNodeTile - 1) / kNodeTile;
    if (n < 2 || (int)blockIdx.x >= tiles) return;
    const int4* __restrict__ lnk = shifted(w.lnk, shift);
    float4* cen = shifted(w.cen, shift);
    const float2* __restrict__ leaf_xy = shifted(w.leaf_xy, shift);
    float* __restrict__ coef = shifted(w.coef, shift);
    const float isq = vs->isq;
    if (threadIdx.x == 0) s_tile = (int)atomicAdd(&vs->ticket[kPasses + 1], 1u);
    __syncthreads();
    // 32 consecutive internal nodes per warp: lane l loads the record and
    // links of its node, finds the place of its coefficients, then the warp
    // builds the nodes' expansions
    if (s_tile >= tiles) return;  // (as in k_cull)
    const int vl = s_tile * kNodeTile + (int)threadIdx.x;
    const bool inner = vl < n - 1;
    float4 cl = inner ? cen[vl] : make_float4(0.0f, 0.0f, 0.0f, make_meta(0, -1));
    int4 Ll = inner ? lnk[vl] : make_int4(0, 0, 0, 0);
    const int dl = meta_degree(cl.w);
    const unsigned size = dl >= 0 ? (unsigned)((dl + 1) * (dl + 1)) : 0u;
    unsigned upto = size;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(full, upto, o);
        if (lane >= o) upto += y;
    }
    if (lane == 31) s_size[warp] = upto;
    __syncthreads();
    if (warp == 0) {
        unsigned sum = 0;
        for (int q = 0; q < kP2MWarps; ++q) sum += s_size[q];
        unsigned long long first;
        const bool ok = look_back(shifted(w.node_status, shift), s_tile, sum, first);
        if (lane == 0) {
            s_first = ok ? first : ~0ull;
            if (!ok) wait_failed(&vs->failed);
        }
    }
    __syncthreads();
    if (s_first == ~0ull) return;
    {
        unsigned long long at = s_first + (upto - size);
        for (int q = 0; q < warp; ++q) at += s_size[q];
        const bool fits = size && at + size <= cap;
        if (size) {
            cl.w = fits ? make_meta((int)at, dl) : make_meta(0, -1);
            cen[vl] = cl;
        }
        const unsigned lost = __ballot_sync(full, size && !fits);
        const unsigned used = __reduce_max_sync(full, fits ? (unsigned)at + size : 0u);
        if (lane == 0) {
            if (lost) atomicAdd(&stats[bt.first + blockIdx.y].demoted, __popc(lost));
            if (used) atomicMax(&vs->coef_used, used);
        }
    }
    const bool built = inner && meta_degree(cl.w) >= 0;
    // Small expansions of few leaves, most of them: four at a time, eight lanes
    // each.  A lane owns a row and computes its t_a and all t_b itself, leaf by
    // leaf.
    const bool small = built && dl < 8 && Ll.w <= kSmallNode;
    for (unsigned left = __ballot_sync(full, small); left;) {
        unsigned m = left;  // the lane's group takes bit `lane / 8` of what is left
        const int row = lane & 7;
#pragma unroll
        for (int q = 0; q < 3; ++q)
            if (q < (lane >> 3)) m &= m - 1;
#pragma unroll
        for (int q = 0; q < 4; ++q) left &= left - 1;
        const int k = m ? __ffs(m) - 1 : 0;
        const float cx = __shfl_sync(full, cl.x, k), cy = __shfl_sync(full, cl.y, k);
        const float meta = __shfl_sync(full, cl.w, k);
        const int first = __shfl_sync(full, Ll.z, k), count = __shfl_sync(full, Ll.w, k), p = meta_degree(meta);
        if (!m) continue;
        float acc[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) acc[q] = 0.0f;
        float2 at = leaf_xy[first];
#pragma unroll 1
        for (int j = 0; j < count; ++j) {
            const float s0 = fmul(fsub(at.x, cx), isq), s1 = fmul(fsub(at.y, cy), isq);
            if (j + 1 < count) at = leaf_xy[first + j + 1];
            float ax = 1.0f, mine = 1.0f, ay = 1.0f;
            float y[8] = {1.0f};
#pragma unroll
            for (int a = 1; a < 8; ++a) {
                ax = fmul(fmul(ax, s0), kInvInt[a]);
                ay = fmul(fmul(ay, s1), kInvInt[a]);
                if (a == row) mine = ax;
                y[a] = ay;
            }
#pragma unroll
            for (int q = 0; q < 8; ++q) acc[q] = __fmaf_rn(mine, y[q], acc[q]);
        }
        float* out = coef + meta_offset(meta) + row * (p + 1);
        if (row <= p) {
#pragma unroll
            for (int q = 0; q < 8; ++q)
                if (q <= p) out[q] = acc[q];
        }
    }
    __syncwarp();
    unsigned todo = __ballot_sync(full, built && !small);
    float* tx = s_tx[warp];
    float* ty = s_ty[warp];
    while (todo) {
            int k = __ffs(todo) - 1;
            todo &= todo - 1;
            float4 c;
            c.x = __shfl_sync(full, cl.x, k);
            c.y = __shfl_sync(full, cl.y, k);
            c.w = __shfl_sync(full, cl.w, k);
            int first = __shfl_sync(full, Ll.z, k), count = __shfl_sync(full, Ll.w, k);
            int p = meta_degree(c.w);
            int off = meta_offset(c.w);
            int P1 = p + 1;
            int BR = kP2MBlock[P1][0], BC = kP2MBlock[P1][1];
            int nC = (P1 + BC - 1) / BC, nR = (P1 + BR - 1) / BR;
            int gr = lane / nC, gc = lane % nC;
            bool owner = gr < nR;
            // this lane's rows and columns; reads past the table repeat its last
            // row / column (their sums are not written)
            int ra[3], cb[4];
#pragma unroll
            for (int i = 0; i < 3; ++i) ra[i] = min(gr * BR + i, p);
#pragma unroll
            for (int q = 0; q < 4; ++q) cb[q] = min(gc * BC + q, p);
            float acc[3][4];
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[i][q] = 0.0f;
            int end = first + count;
            for (int i0 = first; i0 < end; i0 += 32) {
                int cnt = min(32, end - i0);
                if (lane < cnt) {
                    float2 q = leaf_xy[i0 + lane];
                    float s0 = fmul(fsub(q.x, c.x), isq);
                    float s1 = fmul(fsub(q.y, c.y), isq);
                    float ax = 1.0f, ay = 1.0f;
                    tx[lane * kTStride] = 1.0f;
                    ty[lane * kTStride] = 1.0f;
                    for (int a = 1; a <= p; ++a) {
                        ax = fmul(fmul(ax, s0), kInvInt[a]);
                        ay = fmul(fmul(ay, s1), kInvInt[a]);
                        tx[lane * kTStride + a] = ax;
                        ty[lane * kTStride + a] = ay;
                    }
                }
                __syncwarp();
                if (owner) {
                    switch (BR * 8 + BC) {  // uniform over the warp
                        case 9: p2m_block<1, 1>(tx, ty, cnt, ra, cb, acc); break;
                        case 10: p2m_block<1, 2>(tx, ty, cnt, ra, cb, acc); break;
                        case 11: p2m_block<1, 3>(tx, ty, cnt, ra, cb, acc); break;
                        case 18: p2m_block<2, 2>(tx, ty, cnt, ra, cb, acc); break;
                        case 19: p2m_block<2, 3>(tx, ty, cnt, ra, cb, acc); break;
                        case 20: p2m_block<2, 4>(tx, ty, cnt, ra, cb, acc); break;
                        default: p2m_block<3, 4>(tx, ty, cnt, ra, cb, acc); break;
                    }
                }
                __syncwarp();
            }
            if (owner) {
#pragma unroll
                for (int i = 0; i < 3; ++i)
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        int a = gr * BR + i, b = gc * BC + q;
                        if (i < BR && q < BC && a <= p && b <= p) coef[off + a * P1 + b] = acc[i][q];
                    }
            }
    }
}

// -------------------------------------------------------- FGT evaluation
struct Tree {
    const int4* lnk;
    const int* par;
    const float4* box;
    const float4* cen;
    const float* coef;
    const float2* leaf_xy;
    const int* leaf_id;
    const unsigned short* order;
    int n;
    float sq;
    float isq;
};

// evluateHermite with hermiteFunction (hermitefmm.cuh:35-47, 213-237): the
// Hermite functions follow the reference's recursion; the series is summed
// row-factored, sum_a h_a(tx) (sum_b C_ab h_b(ty)), with fused multiply-adds
// (the CPU oracle's deterministic flavour sums the same way).
// A leaf's expansion is its own Gaussian: degree 0, coefficient 1.  Callers
// that know they hold a leaf use this directly, which keeps the series'
// loops out of their code.
__device__ __forceinline__ float leaf_mass(const Tree& T, float4 c, float qx, float qy) {
    float tx = fmul(fsub(qx, c.x), T.isq);
    float ty = fmul(fsub(qy, c.y), T.isq);
    float ex = det_expf_neg(-fmul(tx, tx));
    float ey = det_expf_neg(-fmul(ty, ty));
    return fadd(0.0f, fmul(fmul(1.0f, ex), ey));
}

__device__ __forceinline__ float hermite_eval(const Tree& T, int v, float4 c, float qx, float qy) {
    if (v >= T.n - 1) return leaf_mass(T, c, qx, qy);
    float tx = fmul(fsub(qx, c.x), T.isq);
    float ty = fmul(fsub(qy, c.y), T.isq);
    float ex = det_expf_neg(-fmul(tx, tx));
    float ey = det_expf_neg(-fmul(ty, ty));
    int p = meta_degree(c.w);
    const float* C = T.coef + meta_offset(c.w);
    float hy[kMaxDegree + 1];
    float ty2 = fmul(2.0f, ty);
    hy[0] = ey;
    hy[1] = fmul(ty2, ey);
#pragma unroll
    for (int k = 2; k <= kMaxDegree; ++k) {
        if ((k & 3) == 0 && k > p) break;
        hy[k] = fsub(fmul(ty2, hy[k - 1]), fmul(2.0f * (float)(k - 1), hy[k - 2]));
    }
    float tx2 = fmul(2.0f, tx);
    float hxm2 = 0.0f, hxm1 = 0.0f;
    float w = 0.0f;
    const int P1 = p + 1;
    // Rows four at a time: the four row sums are independent chains, so they
    // are interleaved; each chain and the outer sum keep their order.  The
    // columns go in blocks of four as well: a block past p costs nothing.
#pragma unroll 1
    for (int a = 0; a < P1; a += 4) {
        const float* C0 = C + a * P1;
        const int n1 = a + 1 < P1 ? P1 : 0, n2 = a + 2 < P1 ? 2 * P1 : 0, n3 = a + 3 < P1 ? 3 * P1 : 0;
        float r0 = 0.0f, r1 = 0.0f, r2 = 0.0f, r3 = 0.0f;
#pragma unroll
        for (int b = 0; b <= kMaxDegree; ++b) {
            if ((b & 3) == 0 && b > p) break;
            if (b <= p) {
                r0 = __fmaf_rn(C0[b], hy[b], r0);
                r1 = __fmaf_rn(C0[n1 + b], hy[b], r1);
                r2 = __fmaf_rn(C0[n2 + b], hy[b], r2);
                r3 = __fmaf_rn(C0[n3 + b], hy[b], r3);
            }
        }
        const float r[4] = {r0, r1, r2, r3};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (a + q <= p) {
                float hx = q == 0 && a == 0 ? ex
                                            : (q == 1 && a == 0 ? fmul(tx2, ex)
                                                                : fsub(fmul(tx2, hxm1),
                                                                       fmul(2.0f * (float)(a + q - 1), hxm2)));
                w = __fmaf_rn(hx, r[q], w);
                hxm2 = hxm1;
                hxm1 = hx;
            }
        }
    }
    return w;
}

__device__ __forceinline__ bool truncated_box(float4 b, float r, float qx, float qy) {
    float clx = fminf(fmaxf(qx, b.x), b.z), cly = fminf(fmaxf(qy, b.y), b.w);
    float dx = fsub(qx, clx), dy = fsub(qy, cly);
    float d2 = fadd(fadd(0.0f, fmul(dx, dx)), fmul(dy, dy));
    return !(d2 < fmul(r, r));
}

__device__ __forceinline__ bool truncated(const Tree& T, int v, float r, float qx, float qy) {
    return truncated_box(T.box[v], r, qx, qy);
}

// getWeight / accumulateSubtree (evaluateDynamicRadixTree.cuh:129-242):
// stackless depth-first walk summing, in visiting order, the expansions of
// the nodes that carry one and skipping subtrees whose box misses the
// truncation circle.  A walk visits each node at most twice, so the step
// budget 4n + 64 only guards against a malformed tree.
__device__ float node_weight(const Tree& T, int v, float qx, float qy) {
    float4 c = T.cen[v];
    if (meta_degree(c.w) >= 0) return hermite_eval(T, v, c, qx, qy);
    int rootparent = T.par[v];
    float w = 0.0f;
    int budget = 4 * T.n + 64;
    do {
        c = T.cen[v];
        while (meta_degree(c.w) < 0 && !truncated(T, v, c.z, qx, qy)) {
            int l = T.lnk[v].x;
            if (l < 0 || --budget < 0) return w;
            v = l;
            c = T.cen[v];
        }
        if (meta_degree(c.w) >= 0) w = fadd(w, hermite_eval(T, v, c, qx, qy));
        int p = T.par[v];
        while (p != rootparent && v == T.lnk[p].y) {
            if (--budget < 0) return w;
            v = p;
            p = T.par[p];
        }
        if (p != rootparent) v = T.lnk[p].y;
    } while (T.par[v] != rootparent && --budget >= 0);
    return w;
}

// The same out of line, for the rare callers outside the descent's loop.
__device__ __noinline__ float node_weight_out_of_line(Tree T, int v, float qx, float qy) {
    return node_weight(T, v, qx, qy);
}

// --------------------------------------------------------------- 8 sampler
// Masses of every node the pixels of a warp meet.
//
// getWeight(v) of a node without expansion that the truncation circle
// reaches is the sum, in depth-first order, of the expansions below it.  The
// 32 pixels of a warp (a tile of the image) share one table of the union of
// their trees:
//   topology: level by level, the nodes opened by at least one lane; each
//     lane fetches one opened node's children, so a level costs one memory
//     round trip however many nodes it has.  Counts up the levels and
//     offsets down them then number the expansions they lead to in
//     depth-first order;
//   masses: the expansions one after another, each evaluated by the whole
//     warp for its 32 pixels (hermite_tile), the next one's coefficients on
//     their way meanwhile.  Lanes that are not inside an expansion hold 0.
// The expansions below a node are a range of that list, and its mass is the
// range's sum in order: the additions of a walk from that node (adding the
// zeros of other lanes changes nothing), so bit-identical to it.  The descent
// sums a range when it meets the node.
//
// Lists and masses live in the warp's shared memory, one row of 32 floats
// per expansion (a lane reads its own column: no bank conflicts whatever row
// it is at); rows past kRows go to local memory.  Where the tables are full
// (pixels far apart in units of the bandwidth share little of the tree), the
// caller takes half the lanes at a time, and where those of a single pixel are
// (LongTables), it leaves the rest of the tile to a second kernel.
constexpr int kLevels = 64;               // a radix tree over 62-bit keys is at most 63 deep
// Per-lane records of the descent in shared memory: local memory that is
// written and read back costs an L2 round trip here (about 700 cycles).
constexpr int kPathRows = 32;
// A staged pair's rows (kPairStride) and the Hermite functions' rows are padded
// so that the four rows and eight columns a warp reads together lie in
// different banks.
constexpr int kPairFloats = 16 * 36, kHermiteStride = 36;

// A child's link: kind, stop bit (the child holds at most M splats), entry
// of an opened child.
constexpr unsigned kLinkOpen = 0u, kLinkEval = 0x4000u, kLinkNone = 0x8000u;
constexpr unsigned kLinkKind = 0xC000u, kLinkStop = 0x2000u, kLinkEntry = 0x1FFFu;

struct WarpTables {
    static constexpr int kOpen = 224, kEvals = 192;  // entries
    static constexpr int kRows = 63;                 // masses in shared memory
    static constexpr bool kLong = false;
    uint4 open[kOpen];               // links (left | right << 16), left child, right child, lanes that opened it
    unsigned short split[kOpen];     // first expansion of the right subtree
    union {
        float val[kRows][32];
        struct {                     // while the topology is built
            unsigned short count[kOpen], first[kOpen], level[kLevels + 8];
            float4 box[2][32];       // children of up to 32 nodes: boxes and squared radii
            float r2[2][32];
        };
    };
    union {
        struct {                     // until the masses are known
            unsigned short eval[kEvals];              // opened parent << 1 | side of each expansion
            alignas(16) float coef[2][kPairFloats];   // the pair of expansions being evaluated and the next one
            float hermite[12][kHermiteStride];        // Hermite functions of the tile's columns, then of its rows
        };
        struct {                     // afterwards
            float path[kPathRows][32];         // per-lane records of the levels below the stem
            float series[kMaxDegree + 1][32];  // Hermite functions of a lane's own series (lane_series)
        };
    };
    int owner[32];                   // warp_child_masses
    __device__ __forceinline__ float& mass(int v, int lane) { return val[v][lane]; }
    __device__ __forceinline__ float mass(int v, int lane) const { return val[v][lane]; }
};

// The tables of tiles with a pixel that opens more nodes, or meets more
// expansions, than WarpTables holds: lists and masses in a slab of global
// memory, the rest as there.  Images several times taller than wide have such
// pixels at silhouettes: Morton keys are normalised per axis, so nodes are as
// elongated as the image, and the error bound (half their longer side against
// the bandwidth) holds for few splats only.  500k splats at 128 x 1024: up to
// 1312 nodes and 1188 expansions for one pixel.  The descent's first kernel
// only lists these tiles; a second one (k_sample_long and its like), a warp and
// a slab per block, takes them one after the other.  What bounds it is the
// latency of one tile; a step of those 500k splats takes 8.4 ms so (2388 with
// one lane at a time walking the tree, 240 with 32 side by side), two views of
// a room of 2M splats at 128 x 480 6.4 ms (716 and 76).  Pixels past these
// tables too, millions of splats in such an image, walk side by side.
constexpr int kLongEntries = 8192;       // nodes and expansions (what kLinkEntry can number)
constexpr int kLongMasses = 4096 * 32;   // expansions times lanes of a group
struct LongTables {
    static constexpr int kOpen = kLongEntries, kEvals = kLongEntries, kRows = kLongEntries;
    static constexpr bool kLong = true;
    uint4* open;
    unsigned short *split, *count, *first, *eval;
    float* val;  // rows of `columns` masses: as many as the group has lanes
    int columns;
    __device__ __forceinline__ float& mass(int v, int lane) { return val[v * columns + (lane & (columns - 1))]; }
    __device__ __forceinline__ float mass(int v, int lane) const { return val[v * columns + (lane & (columns - 1))]; }
    unsigned short level[kLevels + 8];
    float4 box[2][32];
    float r2[2][32];
    union {
        struct {
            alignas(16) float coef[2][kPairFloats];
            float hermite[12][kHermiteStride];
        };
        struct {
            float path[kPathRows][32];
            float series[kMaxDegree + 1][32];
        };
    };
    int owner[32];
};
struct LongSlab {
    float val[kLongMasses];
    uint4 open[kLongEntries];
    unsigned short split[kLongEntries], count[kLongEntries], first[kLongEntries], eval[kLongEntries];
};
__device__ __forceinline__ void use_slab(LongTables& wt, LongSlab& s) {  // (the whole warp writes the same)
    wt.open = s.open;
    wt.split = s.split;
    wt.count = s.count;
    wt.first = s.first;
    wt.eval = s.eval;
    wt.val = s.val;
    __syncwarp();
}

// The tiles left for the long tables: a tile is left as soon as kDeferWidth or
// fewer of its lanes fill the short ones (4: as fast as any; at 8 and 16 dense
// small images, whose tiles narrow to 8 lanes all over, lose up to a fifth to
// the few warps that the slabs allow).  counters: ViewState::deferred of the
// first view of the launch; tiles: first pixel, view, lanes.
struct Deferred {
    unsigned* counters;
    uint4* tiles;
    LongSlab* slabs;
};
constexpr int kDeferWidth = 4;
constexpr unsigned kDeferredTiles = 1u << 16;  // more than that are sampled without tables
// By a whole warp: leaves lanes of a tile to the second kernel ((i, j): the
// lane's pixel); false if the list is full.
__device__ __forceinline__ bool defer_tile(const Deferred& df, int i, int j, unsigned view, unsigned lanes) {
    unsigned at = 0;
    if (((threadIdx.x + blockDim.x * threadIdx.y) & 31) == 0) {
        at = atomicAdd(&df.counters[0], 1u);
        if (at < kDeferredTiles) df.tiles[at] = make_uint4((unsigned)i, (unsigned)j, view, lanes);
    }
    return __shfl_sync(0xffffffffu, at, 0) < kDeferredTiles;
}
// The next listed tile; false when there is none left.  The block that finds
// the list empty last clears the counters for the next launch.
__device__ __forceinline__ bool next_deferred(const Deferred& df, unsigned count, uint4& tile) {
    unsigned at = 0;
    if (threadIdx.x == 0 && threadIdx.y == 0) {
        at = atomicAdd(&df.counters[1], 1u);
        if (at >= count && atomicAdd(&df.counters[2], 1u) == gridDim.x - 1) {
            df.counters[0] = 0u;
            df.counters[1] = 0u;
            df.counters[2] = 0u;
        }
    }
    at = __shfl_sync(0xffffffffu, at, 0);
    if (at >= count) return false;
    tile = df.tiles[at];
    return true;
}

// Blocks of four coefficients per side of a degree-p expansion.
__device__ __forceinline__ int coef_blocks(int p) { return (p + 4) >> 2; }

// Row stride of a staged pair of expansions of NB <= 4 blocks per side (the
// coefficients of the two interleaved), and of a single one of five.
template <int NB>
constexpr int kPairStride = NB == 4 ? 36 : NB == 3 ? 24 : NB == 2 ? 20 : 8;
constexpr int kSingleStride = 20;

// Two floats in a register pair: one instruction works on both, each rounded
// as by itself.
typedef unsigned long long float_pair;
__device__ __forceinline__ float_pair pair_of(float a, float b) {
    float_pair r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void pair_split(float_pair p, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(p));
}
__device__ __forceinline__ float_pair pair_fma(float_pair a, float_pair b, float_pair c) {
    float_pair r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ float_pair pair_same(float a) { return pair_of(a, a); }
// Product and difference, rounded by themselves: as multiply-adds, since a
// product that is subtracted from would be contracted in this form.
__device__ __forceinline__ float_pair pair_mul(float_pair a, float_pair b) { return pair_fma(a, b, pair_same(-0.0f)); }
__device__ __forceinline__ float_pair pair_sub(float_pair a, float_pair b) { return pair_fma(b, pair_same(-1.0f), a); }

// Starts the copy of an expansion's P1 x P1 coefficients to dst, rows of
// STRIDE floats with a coefficient every STEP and zeros past column P1 up to
// 4 NB.  Whole rows per warp instruction, so that a lane's column is fixed.
template <int NB, int STRIDE, int STEP>
__device__ __forceinline__ void stage_rows(float* dst, const float* __restrict__ C, int P1, int lane) {
    constexpr int S = NB == 3 ? 16 : 4 * NB, ROWS = NB < 5 ? 32 / S : 1;
    const int row = NB < 5 ? lane / S : 0, col = NB < 5 ? lane % S : lane;
    const float* from = C + row * P1 + min(col, P1 - 1);
    unsigned to = (unsigned)__cvta_generic_to_shared(dst) + 4u * (unsigned)(row * STRIDE + col * STEP);
    const int size = col < P1 ? 4 : 0;
    if (NB >= 3 && col >= 4 * NB) return;
#pragma unroll 2
    for (int r = row; r < P1; r += ROWS, from += ROWS * P1, to += 4u * ROWS * STRIDE)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(to), "l"(from), "r"(size));
}
// A pair of NB <= 4 blocks (P1: coefficients per side of both).
__device__ __forceinline__ void stage_pair(float* dst, int nb, const float* __restrict__ A, int PA,
                                           const float* __restrict__ B, int PB, int lane) {
    switch (nb) {  // uniform over the warp
        case 1:
            stage_rows<1, kPairStride<1>, 2>(dst, A, PA, lane);
            stage_rows<1, kPairStride<1>, 2>(dst + 1, B, PB, lane);
            break;
        case 2:
            stage_rows<2, kPairStride<2>, 2>(dst, A, PA, lane);
            stage_rows<2, kPairStride<2>, 2>(dst + 1, B, PB, lane);
            break;
        case 3:
            stage_rows<3, kPairStride<3>, 2>(dst, A, PA, lane);
            stage_rows<3, kPairStride<3>, 2>(dst + 1, B, PB, lane);
            break;
        default:
            stage_rows<4, kPairStride<4>, 2>(dst, A, PA, lane);
            stage_rows<4, kPairStride<4>, 2>(dst + 1, B, PB, lane);
            break;
    }
    asm volatile("cp.async.commit_group;");
}

// The Hermite series of two staged expansions at the 32 pixels of a warp tile
// of G rows and 32 / G columns (lane % (32 / G) is the column).  Pixels of
// one column have the same y, hence the same Hermite functions h_b(y) and row
// sums r_a = sum_b C_ab h_b(y), and pixels of one row the same h_a(x).  So
// one lane per column and row computes the functions; each of a column's G
// lanes sums one of G rows at a time; and the lanes exchange the sums.  The
// two expansions go through the same instructions, side by side (float_pair):
// the descent is bound by the number of instructions a warp issues one after
// the other.  Every recursion, every row's chain and the outer sum keep their
// order; the padding adds zeros at the end of each, so the values are
// hermite_eval's.  One form per number of blocks, the larger one's: a row's
// reads are in flight together and the column's functions stay in registers;
// the loop over rows stays rolled (with the descent around it the kernel is
// bound by instruction fetch once its code outgrows the instruction cache).
// (t2, e): 2 t and exp(-t^2), t the coordinate of this lane's column or row
// relative to the expansions' centres.
template <int NB, class Tables>
__device__ __forceinline__ float_pair hermite_pair(Tables& wt, const float* coef, int PA, int PB, int cols,
                                                   float_pair t2, float_pair e, int lane) {
    const unsigned full = 0xffffffffu;
    constexpr int S = kPairStride<NB>;
    const int G = 32 / cols, P1 = max(PA, PB);
    {
        ulonglong2* row = reinterpret_cast<ulonglong2*>(wt.hermite[min(lane, 11)]);  // cols + G = 12
        const bool writes = lane < 12;
        float_pair h0 = e, h1 = pair_mul(t2, e);
        float_pair h2 = pair_sub(pair_mul(t2, h1), pair_mul(pair_same(2.0f), h0));
        float_pair h3 = pair_sub(pair_mul(t2, h2), pair_mul(pair_same(4.0f), h1));
        if (writes) {
            row[0] = make_ulonglong2(h0, h1);
            row[1] = make_ulonglong2(h2, h3);
        }
#pragma unroll
        for (int b = 1; b < NB; ++b) {  // 2 (k - 1): small whole numbers, exact
            h0 = pair_sub(pair_mul(t2, h3), pair_mul(pair_same(8.0f * b - 2.0f), h2));
            h1 = pair_sub(pair_mul(t2, h0), pair_mul(pair_same(8.0f * b), h3));
            h2 = pair_sub(pair_mul(t2, h1), pair_mul(pair_same(8.0f * b + 2.0f), h0));
            h3 = pair_sub(pair_mul(t2, h2), pair_mul(pair_same(8.0f * b + 4.0f), h1));
            if (writes) {
                row[2 * b] = make_ulonglong2(h0, h1);
                row[2 * b + 1] = make_ulonglong2(h2, h3);
            }
        }
    }
    __syncwarp();
    const int col = lane & (cols - 1), mine = lane / cols;
    ulonglong2 hy[2 * NB];
#pragma unroll
    for (int b = 0; b < 2 * NB; ++b) hy[b] = reinterpret_cast<const ulonglong2*>(wt.hermite[col])[b];
    float_pair w = pair_same(0.0f);
#pragma unroll 1
    for (int a0 = 0; a0 < P1; a0 += G) {
        const int a = a0 + mine;
        const ulonglong2* C = reinterpret_cast<const ulonglong2*>(coef + min(a, P1 - 1) * S);
        float_pair r = pair_same(0.0f);
#pragma unroll
        for (int b = 0; b < 2 * NB; ++b) {
            const ulonglong2 c = C[b];
            r = pair_fma(c.x, hy[b].x, r);
            r = pair_fma(c.y, hy[b].y, r);
        }
        float ra, rb;
        pair_split(r, ra, rb);
        if (a >= PA) ra = 0.0f;  // rows that were not copied
        if (a >= PB) rb = 0.0f;
#pragma unroll 1
        for (int q = 0; q < G && a0 + q < P1; q += 4) {
            const ulonglong2* hx = reinterpret_cast<const ulonglong2*>(wt.hermite[cols + mine]) + ((a0 + q) >> 1);
            const ulonglong2 u = hx[0], v = hx[1];
            const int from = col + cols * q;
            const float_pair h[4] = {u.x, u.y, v.x, v.y};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float xa = __shfl_sync(full, ra, from + k * cols), xb = __shfl_sync(full, rb, from + k * cols);
                w = pair_fma(h[k], pair_of(xa, xb), w);
            }
        }
    }
    return w;
}

// The same for one expansion of five blocks (degree 16).
template <class Tables>
__device__ __forceinline__ float hermite_single(Tables& wt, const float* coef, int cols, float t2, float e,
                                                int lane) {
    const unsigned full = 0xffffffffu;
    constexpr int NB = 5, S = kSingleStride, P1 = kMaxDegree + 1;
    const int G = 32 / cols;
    {
        float4* row = reinterpret_cast<float4*>(wt.hermite[min(lane, 11)]);
        const bool writes = lane < 12;
        float4 h;
        h.x = e;
        h.y = fmul(t2, e);
        h.z = fsub(fmul(t2, h.y), fmul(2.0f, h.x));
        h.w = fsub(fmul(t2, h.z), fmul(4.0f, h.y));
        if (writes) row[0] = h;
        float k2 = 6.0f;
#pragma unroll 1
        for (int b = 1; b < NB; ++b, k2 += 8.0f) {
            h.x = fsub(fmul(t2, h.w), fmul(k2, h.z));
            h.y = fsub(fmul(t2, h.x), fmul(k2 + 2.0f, h.w));
            h.z = fsub(fmul(t2, h.y), fmul(k2 + 4.0f, h.x));
            h.w = fsub(fmul(t2, h.z), fmul(k2 + 6.0f, h.y));
            if (writes) row[b] = h;
        }
    }
    __syncwarp();
    const int col = lane & (cols - 1), mine = lane / cols;
    const float4* hy = reinterpret_cast<const float4*>(wt.hermite[col]);
    const float4* hx = reinterpret_cast<const float4*>(wt.hermite[cols + mine]);
    float w = 0.0f;
#pragma unroll 1
    for (int a0 = 0; a0 < P1; a0 += G) {
        const float4* C = reinterpret_cast<const float4*>(coef + min(a0 + mine, P1 - 1) * S);
        float r = 0.0f;
#pragma unroll
        for (int b = 0; b < NB; ++b) {
            const float4 c = C[b], h = hy[b];
            r = __fmaf_rn(c.x, h.x, r);
            r = __fmaf_rn(c.y, h.y, r);
            r = __fmaf_rn(c.z, h.z, r);
            r = __fmaf_rn(c.w, h.w, r);
        }
        if (a0 + mine >= P1) r = 0.0f;
#pragma unroll 1
        for (int q = 0; q < G && a0 + q < P1; q += 4) {
            const float4 h = hx[(a0 + q) >> 2];
            const int from = col + cols * q;
            const float r0 = __shfl_sync(full, r, from), r1 = __shfl_sync(full, r, from + cols);
            const float r2 = __shfl_sync(full, r, from + 2 * cols), r3 = __shfl_sync(full, r, from + 3 * cols);
            w = __fmaf_rn(h.x, r0, w);
            w = __fmaf_rn(h.y, r1, w);
            w = __fmaf_rn(h.z, r2, w);
            w = __fmaf_rn(h.w, r3, w);
        }
    }
    return w;
}

// node_weight of one lane's own node, the case of an expansion in few
// instructions: Hermite functions of y in the lane's column of wt.series,
// rows four at a time (independent chains); hermite_eval's operations in its
// order.  Nodes without one (rare here) go out of line.
template <class Tables>
__device__ __forceinline__ float lane_series(const Tree& T, Tables& wt, int lane, int v, float qx, float qy) {
    const float4 c = T.cen[v];
    const int p = meta_degree(c.w);
    if (p < 0) return node_weight_out_of_line(T, v, qx, qy);
    float tx = fmul(fsub(qx, c.x), T.isq);
    float ty = fmul(fsub(qy, c.y), T.isq);
    float ex = det_expf_neg(-fmul(tx, tx));
    float ey = det_expf_neg(-fmul(ty, ty));
    if (v >= T.n - 1) return fadd(0.0f, fmul(fmul(1.0f, ex), ey));
    const float* C = T.coef + meta_offset(c.w);
    {
        const float t2 = fmul(2.0f, ty);
        float h0 = ey, h1 = fmul(t2, ey), k2 = 2.0f;
        wt.series[0][lane] = h0;
#pragma unroll 1
        for (int k = 1; k <= p; ++k, k2 += 2.0f) {
            wt.series[k][lane] = h1;
            float h = fsub(fmul(t2, h1), fmul(k2, h0));
            h0 = h1;
            h1 = h;
        }
    }
    const float t2 = fmul(2.0f, tx);
    float hx = ex, hxm = 0.0f, k2 = 0.0f;  // h_a and h_(a-1) of x
    float w = 0.0f;
    const int P1 = p + 1;
#pragma unroll 1
    for (int a = 0; a < P1; a += 4, C += 4 * P1) {
        const int n1 = a + 1 < P1 ? P1 : 0, n2 = a + 2 < P1 ? 2 * P1 : 0, n3 = a + 3 < P1 ? 3 * P1 : 0;
        float r[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 4
        for (int b = 0; b < P1; ++b) {
            const float h = wt.series[b][lane];
            r[0] = __fmaf_rn(C[b], h, r[0]);
            r[1] = __fmaf_rn(C[n1 + b], h, r[1]);
            r[2] = __fmaf_rn(C[n2 + b], h, r[2]);
            r[3] = __fmaf_rn(C[n3 + b], h, r[3]);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (a + q <= p) w = __fmaf_rn(hx, r[q], w);
            float h = fsub(fmul(t2, hx), fmul(k2, hxm));
            hxm = hx;
            hx = h;
            k2 += 2.0f;
        }
    }
    return w;
}

// !truncated_box, the radius squared beforehand.
__device__ __forceinline__ bool within(float4 b, float r2, float qx, float qy) {
    float dx = fsub(qx, fminf(fmaxf(qx, b.x), b.z)), dy = fsub(qy, fminf(fmaxf(qy, b.y), b.w));
    return fadd(fmul(dx, dx), fmul(dy, dy)) < r2;
}

// Sum of the listed masses [s, t) of this lane, in order.
template <class Tables>
__device__ __forceinline__ float range_sum(const Tables& wt, const float* val_hi, int lane, int s, int t) {
    float acc = 0.0f;
    int i = s;
    constexpr int kRows = Tables::kRows;
    const int top = min(t, kRows);
#pragma unroll 1
    for (; i + 4 <= top; i += 4) {
        float x0 = wt.mass(i, lane), x1 = wt.mass(i + 1, lane), x2 = wt.mass(i + 2, lane), x3 = wt.mass(i + 3, lane);
        acc = fadd(fadd(fadd(fadd(acc, x0), x1), x2), x3);
    }
#pragma unroll 1
    for (; i < t; ++i) acc = fadd(acc, i < kRows ? wt.mass(i, lane) : val_hi[i - kRows]);
    return acc;
}

// Fills the tables for the lanes of `lanes`, a group of `width` (all 32 lanes
// call this).
// Returns the number of expansions listed (opened node 0 is the root), 0
// when there are no tables (the root carries an expansion, or no lane
// reaches it), -1 when they are full (nothing computed).  total is getWeight
// of the root for the lanes inside.
template <class Tables>
__device__ int warp_tables(const Tree& T, float qx, float qy, unsigned lanes, int width, int M, int cols, Tables& wt,
                           float* val_hi, float& total) {
    const unsigned full = 0xffffffffu;
    const int lane = (threadIdx.x + blockDim.x * threadIdx.y) & 31;
    const unsigned lt = (1u << lane) - 1u;
    total = 0.0f;
    const bool live = (lanes >> lane) & 1u;
    {
        float4 c = T.cen[0];
        if (meta_degree(c.w) >= 0) {
            if (live) total = node_weight_out_of_line(T, 0, qx, qy);
            return 0;
        }
        lanes = __ballot_sync(full, live && !truncated(T, 0, c.z, qx, qy));
        if (!lanes) return 0;
    }
    __syncwarp();
    if (lane == 0) {
        int4 L = T.lnk[0];
        wt.open[0] = make_uint4(0u, (unsigned)L.x, (unsigned)L.y, lanes);
        wt.level[0] = 0;
    }
    __syncwarp();
    // ---- topology
    int lo = 0, hi = 1, levels = 0;  // opened nodes of this level
    while (lo < hi) {
        if (levels >= kLevels) return -1;
        int next = hi;
        for (int base = lo; base < hi; base += 32) {
            const int cnt = min(32, hi - base);
            const int o = base + min(lane, cnt - 1);
            const uint4 E = wt.open[o];
            const int a = (int)E.y, b = (int)E.z;
            const float4 ca = T.cen[a], cb = T.cen[b];
            const float4 ba = T.box[a], bb = T.box[b];
            const int4 La = T.lnk[a], Lb = T.lnk[b];
            unsigned ma = 0u, mb = 0u;  // lanes whose circle reaches the children of this lane's node
            wt.box[0][lane] = ba;
            wt.box[1][lane] = bb;
            wt.r2[0][lane] = fmul(ca.z, ca.z);
            wt.r2[1][lane] = fmul(cb.z, cb.z);
            __syncwarp();
#pragma unroll 1
            for (int k = 0; k < cnt; ++k) {
                const bool inside = (wt.open[base + k].w >> lane) & 1u;
                unsigned hit = __ballot_sync(full, inside && within(wt.box[0][k], wt.r2[0][k], qx, qy));
                if (lane == k) ma = hit;
                hit = __ballot_sync(full, inside && within(wt.box[1][k], wt.r2[1][k], qx, qy));
                if (lane == k) mb = hit;
            }
            __syncwarp();
            const bool ea = meta_degree(ca.w) >= 0, eb = meta_degree(cb.w) >= 0;
            const bool oa = lane < cnt && !ea && ma, ob = lane < cnt && !eb && mb;
            const unsigned Ba = __ballot_sync(full, oa), Bb = __ballot_sync(full, ob);
            const int pa = next + __popc(Ba & lt) + __popc(Bb & lt), pb = pa + (oa ? 1 : 0);
            next += __popc(Ba) + __popc(Bb);
            if (next > Tables::kOpen) return -1;
            if (lane < cnt) {
                unsigned la = ea ? kLinkEval : kLinkNone, lb = eb ? kLinkEval : kLinkNone;
                if (oa) {
                    la = kLinkOpen | (La.w <= M ? kLinkStop : 0u) | (unsigned)pa;
                    wt.open[pa] = make_uint4(0u, (unsigned)La.x, (unsigned)La.y, ma);
                }
                if (ob) {
                    lb = kLinkOpen | (Lb.w <= M ? kLinkStop : 0u) | (unsigned)pb;
                    wt.open[pb] = make_uint4(0u, (unsigned)Lb.x, (unsigned)Lb.y, mb);
                }
                wt.open[o].x = la | (lb << 16);
            }
        }
        ++levels;
        if (lane == 0) wt.level[levels] = (unsigned short)hi;
        lo = hi;
        hi = next;
        __syncwarp();
    }
    // ---- expansions below each opened node, up the levels
    auto children = [&](uint4 E, int& na, int& nb) {
        unsigned la = E.x & 0xffffu, lb = E.x >> 16;
        na = (la & kLinkKind) == kLinkOpen ? wt.count[la & kLinkEntry] : (la == kLinkEval ? 1 : 0);
        nb = (lb & kLinkKind) == kLinkOpen ? wt.count[lb & kLinkEntry] : (lb == kLinkEval ? 1 : 0);
    };
#pragma unroll 1
    for (int l = levels - 1; l >= 0; --l) {
#pragma unroll 1
        for (int o = wt.level[l] + lane; o < wt.level[l + 1]; o += 32) {
            int na, nb;
            children(wt.open[o], na, nb);
            wt.count[o] = (unsigned short)(na + nb);
        }
        __syncwarp();
    }
    const int nV = wt.count[0];
    if (nV > Tables::kEvals) return -1;
    if constexpr (Tables::kLong) {
        if (nV > kLongMasses / width) return -1;
        wt.columns = width;
    }
    // ---- and their places in depth-first order, down the levels
    if (lane == 0) wt.first[0] = 0;
    __syncwarp();
#pragma unroll 1
    for (int l = 0; l < levels; ++l) {
#pragma unroll 1
        for (int o = wt.level[l] + lane; o < wt.level[l + 1]; o += 32) {
            uint4 E = wt.open[o];
            int na, nb, s = wt.first[o];
            children(E, na, nb);
            unsigned la = E.x & 0xffffu, lb = E.x >> 16;
            wt.split[o] = (unsigned short)(s + na);
            if ((la & kLinkKind) == kLinkOpen) wt.first[la & kLinkEntry] = (unsigned short)s;
            else if (la == kLinkEval) wt.eval[s] = (unsigned short)(o << 1);
            if ((lb & kLinkKind) == kLinkOpen) wt.first[lb & kLinkEntry] = (unsigned short)(s + na);
            else if (lb == kLinkEval) wt.eval[s + na] = (unsigned short)(o << 1 | 1);
        }
        __syncwarp();
    }
    // ---- masses.  32 expansions at a time, in order of their number of
    // blocks: those of five one by one, the others in pairs, then the leaves.
    // Lane l < cols computes the Hermite functions of column l, lane cols + g
    // those of row g (for the second of a pair: their exponentials in lanes
    // 16 on); the next pair's coefficients are copied meanwhile.
    const float qx0 = __shfl_sync(full, qx, 0);
    const int role = lane & 15;
    const bool columns = role < cols;
    const float q = columns ? qy : qx0 + (float)min(role - cols, 32 / cols - 1);
#pragma unroll 1
    for (int v0 = 0; v0 < nV; v0 += 32) {
        const int cnt = min(32, nV - v0);
        const unsigned entry = wt.eval[v0 + min(lane, cnt - 1)];
        const uint4 E = wt.open[entry >> 1];
        const int node = (int)((entry & 1u) ? E.z : E.y);
        const float4 c0 = T.cen[node];
        const int p0 = node >= T.n - 1 ? -1 : meta_degree(c0.w);  // -1: a leaf, no coefficients
        if (lane < cnt && p0 >= 0) {  // each lane asks for its expansion's lines
            const float* C = T.coef + meta_offset(c0.w);
#pragma unroll 1
            for (int e = 0; e < (p0 + 1) * (p0 + 1); e += 32) asm volatile("prefetch.global.L2 [%0];" ::"l"(C + e));
        }
        const int nb0 = lane < cnt ? coef_blocks(p0) : -1;
        int rank = 0, fives = 0, sums = 0;  // this lane's place; expansions of five blocks; and of any
#pragma unroll 1
        for (int k = 5; k >= 0; --k) {
            const unsigned m = __ballot_sync(full, nb0 == k);
            if (nb0 == k) rank = sums + __popc(m & lt);
            if (k > 0) sums += __popc(m);
            if (k == 5) fives = sums;
        }
        if (lane < cnt) wt.owner[rank] = lane;
        __syncwarp();
        const int mine = wt.owner[min(lane, cnt - 1)];
        const float cx = __shfl_sync(full, c0.x, mine), cy = __shfl_sync(full, c0.y, mine);
        const float meta = __shfl_sync(full, c0.w, mine);
        const unsigned inside = __shfl_sync(full, E.w, mine);
        auto put = [&](int at, float w) {  // the mass of the expansion at place `at`
            const int v = v0 + __shfl_sync(full, mine, at);
            w = ((__shfl_sync(full, inside, at) >> lane) & 1u) ? w : 0.0f;
            if (Tables::kLong && !live) return;  // (another lane's column)
            if (v < Tables::kRows) wt.mass(v, lane) = w;
            else val_hi[v - Tables::kRows] = w;
        };
#pragma unroll 1
        for (int k = 0; k < fives; ++k) {
            stage_rows<5, kSingleStride, 1>(wt.coef[0], T.coef + meta_offset(__shfl_sync(full, meta, k)),
                                            kMaxDegree + 1, lane);
            asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
            const float x = __shfl_sync(full, cx, k), y = __shfl_sync(full, cy, k);
            __syncwarp();
            const float t = fmul(fsub(q, columns ? y : x), T.isq);
            put(k, hermite_single(wt, wt.coef[0], cols, fmul(2.0f, t), det_expf_neg(-fmul(t, t)), lane));
            __syncwarp();
        }
#pragma unroll 1
        for (int k = fives - 2; k < sums; k += 2) {
            if (k + 2 < sums) {
                const float A = __shfl_sync(full, meta, k + 2), B = __shfl_sync(full, meta, min(k + 3, sums - 1));
                const int pa = meta_degree(A);
                stage_pair(wt.coef[((k + 2 - fives) >> 1) & 1], coef_blocks(pa), T.coef + meta_offset(A), pa + 1,
                           T.coef + meta_offset(B), meta_degree(B) + 1, lane);
            }
            if (k < fives) continue;
            const int k1 = min(k + 1, sums - 1), from = lane < 16 ? k : k1;
            const int PA = meta_degree(__shfl_sync(full, meta, k)) + 1;
            const int PB = meta_degree(__shfl_sync(full, meta, k1)) + 1;
            const float x = __shfl_sync(full, cx, from), y = __shfl_sync(full, cy, from);
            const float t = fmul(fsub(q, columns ? y : x), T.isq);
            const float e = det_expf_neg(-fmul(t, t)), t2 = fmul(2.0f, t);
            const float t2b = __shfl_sync(full, t2, role + 16), eb = __shfl_sync(full, e, role + 16);
            if (k + 2 < sums) asm volatile("cp.async.wait_group 1;" ::: "memory");
            else asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncwarp();
            const float* coef = wt.coef[((k - fives) >> 1) & 1];
            const float_pair tt = pair_of(t2, t2b), ee = pair_of(e, eb);
            float_pair w;
            switch (coef_blocks(PA - 1)) {  // uniform over the warp
                case 1: w = hermite_pair<1>(wt, coef, PA, PB, cols, tt, ee, lane); break;
                case 2: w = hermite_pair<2>(wt, coef, PA, PB, cols, tt, ee, lane); break;
                case 3: w = hermite_pair<3>(wt, coef, PA, PB, cols, tt, ee, lane); break;
                default: w = hermite_pair<4>(wt, coef, PA, PB, cols, tt, ee, lane); break;
            }
            float wa, wb;
            pair_split(w, wa, wb);
            put(k, wa);
            if (k1 > k) put(k1, wb);
            __syncwarp();  // the pair has been read
        }
#pragma unroll 1
        for (int k = sums; k < cnt; ++k)
            put(k, leaf_mass(T, make_float4(__shfl_sync(full, cx, k), __shfl_sync(full, cy, k), 0.0f, 0.0f), qx, qy));
        __syncwarp();  // owner is written again
    }
    __syncwarp();
    total = range_sum(wt, val_hi, lane, 0, nV);
    __syncwarp();
    return nV;
}

// A lane's place in the tables: an opened node, the range of its expansions
// and their sum.
struct Place {
    int o, s, t;
    float sum;
};

// The opened nodes above the first one with two children in the tables: every
// lane with a mass has the root's mass in each of them and goes through them
// all.  node: that first one; depth: its depth; path: the choices to it.
struct Stem {
    int node, depth;
    unsigned long long path;
};

template <class Tables>
__device__ __forceinline__ Stem find_stem(const Tables& wt) {
    Stem s{0, 0, 0ull};
#pragma unroll 1
    while (s.depth < kTrace - 2) {  // uniform over the warp
        const unsigned links = wt.open[s.node].x, la = links & 0xffffu, lb = links >> 16;
        const bool left = lb == kLinkNone, right = la == kLinkNone;
        const unsigned link = left ? la : lb;
        if (left == right || (link & kLinkKind) != kLinkOpen || (link & kLinkStop)) break;
        if (right) s.path |= 1ull << s.depth;
        ++s.depth;
        s.node = (int)(link & kLinkEntry);
    }
    return s;
}

// The sums of the children's ranges (getWeight of both children); E: the
// node's entry, m: its split.  A child that holds the whole range has the
// node's own sum.
template <class Tables>
__device__ __forceinline__ void child_sums(const Tables& wt, const float* val_hi, int lane, const Place& at, int m,
                                           float& w0, float& w1) {
    if (m == at.t) { w0 = at.sum; w1 = 0.0f; }
    else if (m == at.s) { w0 = 0.0f; w1 = at.sum; }
    else {
#pragma unroll 1
        for (int side = 0; side < 2; ++side) {
            w0 = w1;
            w1 = range_sum(wt, val_hi, lane, side ? m : at.s, side ? at.t : m);
        }
    }
}

// The lanes of the next pass: the group of `width` lanes around the first
// lane of todo.
__device__ __forceinline__ unsigned lane_group(unsigned todo, int width) {
    if (width == 32) return todo;
    return todo & (((1u << width) - 1u) << ((__ffs(todo) - 1) & ~(width - 1)));
}

// Child masses (w0, w1) = getWeight of the children (a, b) for every lane
// of the warp with `need` (all lanes call this together); the value of each
// is the same node_weight call whichever lane makes it, so both forms below
// give identical masses, only the speed differs (the autotuner picks one per
// view shape; uds_sample_params.spread).
// SPREAD false: every needing lane evaluates its own two children, left then
//   right; neighbouring pixels at the same node evaluate the same child side
//   by side (equal trip counts, one coefficient stream).
// SPREAD true: the 2c evaluations of the c needing lanes are spread over the
//   warp's 32 lanes, first the left children of the needing lanes (in lane
//   order), then their right children, so a lane waits for one series
//   instead of two while c <= 16.  `owner`: 32 ints of the warp's shared
//   memory.
template <bool SPREAD, class Tables>
__device__ __forceinline__ void warp_child_masses(const Tree& T, Tables& wt, bool need, int a, int b, float qx,
                                                  float qy, float& w0, float& w1) {
    int* owner = wt.owner;
    const int lane = (threadIdx.x + blockDim.x * threadIdx.y) & 31;
    if (!SPREAD) {
        if (need) {
#pragma unroll 1
            for (int ch = 0; ch < 2; ++ch) {
                float x = fmaxf(0.0f, lane_series(T, wt, lane, ch ? b : a, qx, qy));
                if (ch) w1 = x; else w0 = x;
            }
        }
        return;
    }
    const unsigned full = 0xffffffffu;
    unsigned nm = __ballot_sync(full, need);
    if (!nm) return;
    int c = __popc(nm), c2 = 2 * c;
    int rank = __popc(nm & ((1u << lane) - 1u));
    if (need) owner[rank] = lane;
    __syncwarp();
#pragma unroll 1
    for (int e0 = 0; e0 < c2; e0 += 32) {
        int e = e0 + lane;
        bool right = e >= c;
        int o = e < c2 ? owner[right ? e - c : e] : lane;
        float oqx = __shfl_sync(full, qx, o), oqy = __shfl_sync(full, qy, o);
        int oa = __shfl_sync(full, a, o), ob = __shfl_sync(full, b, o);
        float x = 0.0f;
        if (e < c2) x = fmaxf(0.0f, lane_series(T, wt, lane, right ? ob : oa, oqx, oqy));
        int s0 = rank - e0, s1 = c + rank - e0;  // lanes holding this lane's children in this pass
        float x0 = __shfl_sync(full, x, s0 & 31), x1 = __shfl_sync(full, x, s1 & 31);
        if (need && s0 >= 0 && s0 < 32) w0 = x0;
        if (need && s1 >= 0 && s1 < 32) w1 = x1;
    }
    __syncwarp();  // owner is rewritten by the next call
}

constexpr int kKnown = 3;  // nodes outside the tables whose child masses a lane keeps

// Two warps per block: their tables fit the 48 KB of static shared memory,
// and a block's slot is free again when two tiles are done.  Six blocks per
// SM fill its shared memory (168 registers per thread).  What bounds the
// descent is the length of its instruction stream: 445 million warp
// instructions at 500k splats / 1024^2, 0.41 per cycle and scheduler while
// warps are there, mostly waiting for the previous instruction.  (An earlier
// form with unrolled loops ran 516 million against 620 but took 2.6 ms instead
// of 1.34, fetching them: 187 KB of code instead of 54.)  500k / 1024^2 / K = 8:
// 2.7-3.3 ms before these tables, 11 ms where one pixel's cache of 160 nodes
// overflowed; 1.34 with rolled series, 1.22 with one form of the series per
// number of blocks, 0.96 with the tiles in order of the work they hold (kCells),
// 0.85 with the series in pairs.
constexpr int kDescentThreads = 64, kDescentBlocks = 6;

// Views of different sizes in one descent launch: blocks [first[v],
// first[v+1]) of the one-dimensional grid cover view v; its indices start at
// entry ioff[v] of the packed output.
constexpr int kMaxUneven = 32;
struct UnevenViews {
    int nv;
    int first[kMaxUneven + 1];
    int W[kMaxUneven], H[kMaxUneven];
    long long ioff[kMaxUneven];
};

// Warps per block: two; one where the lists of more than 16 keys take shared
// memory (dynamic, 256 K bytes per warp).
template <int KM>
constexpr int kDescentWarps = KM <= 16 ? kDescentThreads / 32 : 1;

// The tree of the view vz places after the first one of a launch.
__device__ __forceinline__ void shift_tree(Tree& T, size_t off) {
    T.lnk = shifted(T.lnk, off);
    T.par = shifted(T.par, off);
    T.box = shifted(T.box, off);
    T.cen = shifted(T.cen, off);
    T.coef = shifted(T.coef, off);
    T.leaf_xy = shifted(T.leaf_xy, off);
    T.leaf_id = shifted(T.leaf_id, off);
    T.order = shifted(T.order, off);
}

// The descents of the lanes of `todo` of a tile; (i, j): the lane's pixel, vz:
// the view's place in the launch.
template <int R, int KM, bool SPREAD, class Tables>
__device__ __forceinline__ void sample_tile(const Tree& T, Tables& wt, uint2* list, unsigned todo, int i, int j, int H,
                                            int K, int M, float precision, const float* __restrict__ uniforms,
                                            uint64_t seed, uint32_t view, int* __restrict__ indices,
                                            uds_view_stats* st, const Deferred& df, unsigned vz) {
    const unsigned full = 0xffffffffu;
    size_t pixel = (size_t)j + (size_t)H * i;
    float qx = (float)i, qy = (float)j;
    const int lane = (threadIdx.x + blockDim.x * threadIdx.y) & 31;
    float val_hi[Tables::kLong ? 1 : Tables::kEvals - Tables::kRows];
    // K-sized arrays stay in registers for K <= 16 (loops fully unrolled)
    constexpr int UK = KM <= 16 ? KM : 1;
    int width = 32;
    while (todo) {
        unsigned group = lane_group(todo, width);
        float total;
        const int state = warp_tables(T, qx, qy, group, width, M, blockDim.x, wt, val_hi, total);
        if (state < 0) {
            if (!Tables::kLong && width <= kDeferWidth && defer_tile(df, i, j, vz, todo)) break;
            if (width > 1) {
                width >>= 1;
                continue;
            }
            group = todo;  // without tables: the lanes left walk side by side
        }
        todo &= ~group;
        const bool mine = (group >> lane) & 1u;
        if (state < 0 && mine) total = node_weight_out_of_line(T, 0, qx, qy);
        const Place root{0, 0, state, total};
        total = fmaxf(0.0f, total);
        bool act = mine && !(total < precision);
        if (!__any_sync(full, act)) continue;
        constexpr int KR = KM <= 16 ? KM : 1;
        int ids[KR];
        float keys[KR];
        float last = __int_as_float(0x7f800000);  // K > 16: the list's largest key once it is full
        int have = 0;                             // and its length
        if (KM <= 16) {
#pragma unroll UK
            for (int k = 0; k < KR; ++k) { ids[k] = -1; keys[k] = __int_as_float(0x7f800000); }
        }
        // each round's path as its choice bits (bit m: right child taken at depth
        // m): two rounds meet the same node at depth m iff their first m choices
        // agree (node ids are unique)
        unsigned long long pb[R];
#pragma unroll
        for (int rr = 0; rr < R; ++rr) pb[rr] = 0ull;
        // per depth >= 1 the path's node's share of its parent's mass and, by
        // round, its capacity: the first levels below the stem in wt.path, the
        // others in local memory
        float far_rows[R * kTrace];
        float* far = far_rows;
        asm volatile("" : "+l"(far));  // stays an array in memory
        constexpr int kNear = kPathRows / R;  // levels in wt.path, R rows each: the share, R - 1 capacities
        // child masses of the last nodes met outside the tables (of the last one
        // at each depth with the long ones: without any at all, a walk of its
        // subtree is what they save)
        constexpr int kKept = Tables::kLong ? kTrace : kKnown;
        int kv[kKept];
        float kw0[kKept], kw1[kKept];
        if (Tables::kLong) {
            for (int q = 0; q < kKept; ++q) kv[q] = -1;
        } else {
#pragma unroll
            for (int q = 0; q < kKnown; ++q) { kv[q] = -1; kw0[q] = 0.0f; kw1[q] = 0.0f; }
        }
        bool overflow = false;
        // A node of the stem gives its one child its whole mass, so the child's
        // capacity is always the node's: one number, cap, for the whole stem, and
        // a round starts at the stem's end.  Once it is used up (cap = 0) a round
        // starts at the root instead: where neither child has anything left it
        // goes left, off the stem if need be.  The rounds below `quick` started
        // at the stem's end.
        const Stem stem = state > 0 ? find_stem(wt) : Stem{0, 0, 0ull};
        float cap = 1.0f;
        int quick = 0;
        const int near0 = stem.depth + 1;
        auto capacity = [&](int rr, int d) {
            const int q = d - near0;
            return q >= 0 && q < kNear ? wt.path[R * q + 1 + rr][lane] : far[R * d + 1 + rr];
        };
        auto set_capacity = [&](int rr, int d, float x) {
            const int q = d - near0;
            if (q >= 0 && q < kNear) wt.path[R * q + 1 + rr][lane] = x;
            else far[R * d + 1 + rr] = x;
        };
#pragma unroll 1
        for (int r = 0; r < R; ++r) {
            int d = 0;
            Place at = root;                // place in the tables (o < 0: outside), or
            if (state <= 0) at.o = -1;
            int v = 0;                      // the node itself and its links
            int4 L = T.lnk[0];
            unsigned long long cur = 0ull;  // this round's choice bits so far
            unsigned with = (1u << r) - 1u; // earlier rounds that have come the same way so far
            bool going = act && L.w > M, pend = false;
            const bool skip = state > 0 && cap > 0.0f && total < __int_as_float(0x7f800000);
            if (skip) {
                d = stem.depth;
                cur = stem.path;
                at.o = stem.node;
                quick = r + 1;
            }
            // lanes go down the tables on their own; a lane that needs child
            // masses evaluated waits until no other lane can go on, so that the
            // evaluations of a round are made in as few passes as possible
            while (true) {
                float w0 = 0.0f, w1 = 0.0f, sum0 = 0.0f, sum1 = 0.0f;
                uint4 E = make_uint4(0u, 0u, 0u, 0u);
                int split = 0;
                if (going && !pend) {
                    if (at.o >= 0) {
                        E = wt.open[at.o];
                        split = wt.split[at.o];
                        child_sums(wt, val_hi, lane, at, split, sum0, sum1);
                        w0 = fmaxf(0.0f, sum0);
                        w1 = fmaxf(0.0f, sum1);
                    } else {
                        pend = true;
                        if (Tables::kLong) {
                            if (kv[d] == v) { w0 = kw0[d]; w1 = kw1[d]; pend = false; }
                        } else {
#pragma unroll
                            for (int q = 0; q < kKnown; ++q)
                                if (kv[q] == v) { w0 = kw0[q]; w1 = kw1[q]; pend = false; }
                        }
                    }
                }
                bool can = going && !pend;
                if (!__any_sync(full, can)) {
                    if (!__any_sync(full, pend)) break;
                    warp_child_masses<SPREAD>(T, wt, pend, L.x, L.y, qx, qy, w0, w1);
                    can = pend;
                    pend = false;
                    if (can) {
                        if (!Tables::kLong) {
#pragma unroll
                            for (int q = kKnown - 1; q > 0; --q) {
                                kv[q] = kv[q - 1];
                                kw0[q] = kw0[q - 1];
                                kw1[q] = kw1[q - 1];
                            }
                        }
                        const int q = Tables::kLong ? d : 0;
                        kv[q] = v;
                        kw0[q] = w0;
                        kw1[q] = w1;
                    }
                }
                if (can) {
                    // the children's shares; w / w = 1: many nodes above the
                    // pixel have one child that its circle reaches
                    float sum = fadd(fadd(0.0f, w0), w1);
                    if ((w0 == 0.0f) != (w1 == 0.0f) && sum < __int_as_float(0x7f800000)) {
                        w0 = w0 == 0.0f ? 0.0f : 1.0f;
                        w1 = w1 == 0.0f ? 0.0f : 1.0f;
                    } else {
                        w0 = fdiv(w0, sum);
                        w1 = fdiv(w1, sum);
                    }
                    // capacities of the children: from the latest earlier round
                    // whose path passed through this node into that child
                    float c0 = 1.0f, c1 = 1.0f;
                    unsigned into0 = 0u, into1 = 0u;
                    if (with) {
#pragma unroll
                        for (int rr = 0; rr < R - 1; ++rr) into1 |= (unsigned)((pb[rr] >> d) & 1ull) << rr;
                        into1 &= with;
                        into0 = with & ~into1;
                        if (into0 && d + 1 < kTrace) {
                            const int rr = 31 - __clz(into0);
                            c0 = rr < quick && d < stem.depth ? cap : capacity(rr, d + 1);
                        }
                        if (into1 && d + 1 < kTrace) {
                            const int rr = 31 - __clz(into1);
                            c1 = rr < quick && d < stem.depth ? cap : capacity(rr, d + 1);
                        }
                    }
                    const bool right = fmul(w0, c0) < fmul(w1, c1);
                    with = right ? into1 : into0;
                    ++d;
                    if (d >= kTrace) {
                        overflow = true;
                        going = false;
                        act = false;
                    } else {
                        if (right) cur |= 1ull << (d - 1);
                        if (r < R - 1) {
                            const int q = d - near0;
                            if (q >= 0 && q < kNear) wt.path[R * q][lane] = right ? w1 : w0;
                            else far[R * d] = right ? w1 : w0;
                            set_capacity(r, d, right ? c1 : c0);
                        }
                        bool through = false;  // on to an opened child of the tables
                        unsigned link = 0u;
                        if (at.o >= 0) {
                            v = (int)(right ? E.z : E.y);
                            link = right ? E.x >> 16 : E.x & 0xffffu;
                            through = (link & kLinkKind) == kLinkOpen &&
                                      ((wt.open[link & kLinkEntry].w >> lane) & 1u);
                        } else {
                            v = right ? L.y : L.x;
                        }
                        if (through && !(link & kLinkStop)) {
                            at.o = (int)(link & kLinkEntry);
                            at.sum = right ? sum1 : sum0;
                            if (right) at.s = split; else at.t = split;
                        } else {
                            at.o = -1;
                            L = T.lnk[v];
                            going = L.w > M;
                        }
                    }
                }
            }
            if (!act) continue;
#pragma unroll
            for (int rr = 0; rr < R; ++rr)
                if (rr == r) pb[rr] = cur;
            // the path's capacities shrink by the probability of the part below
            // (no later round looks at the last one's)
            if (r < R - 1) {
                float prob = 1.0f;
                const int top = skip ? stem.depth : 0;
#pragma unroll 1
                for (int m = d; m > top; --m) {
                    const int q = m - near0;
                    set_capacity(r, m, fmaxf(0.0f, fsub(capacity(r, m), prob)));
                    prob = fmul(prob, q >= 0 && q < kNear ? wt.path[R * q][lane] : far[R * m]);
                }
                if (skip) cap = fmaxf(0.0f, fsub(cap, prob));
            }
            // order sampling over the subtree's leaves (insertSample,
            // sequentialPoissonRadixTree.cuh:15-41); a leaf's mass is its own
            // Gaussian (degree 0, coefficient 1).  The subtree holds at most M
            // leaves: K, or the leaf size when that is larger.
            int f0 = L.z, cnt = L.w;
            // the round's uniforms, drawn as the leaves use them (after the
            // descent, so they hold no registers there): Philox block
            // (pixel, view, r * ceil(M / 4) + k / 4), or the caller's tensor
            const float* up = uniforms ? uniforms + ((size_t)pixel * R + r) * M : nullptr;
            const int G = (M + 3) >> 2;
            uint32_t c4[4];
            float2 xy = T.leaf_xy[f0];
            int id = T.leaf_id[f0];
#pragma unroll 1
            for (int k = 0; k < cnt; ++k) {
                if (!up && (k & 3) == 0) {
                    c4[0] = (uint32_t)pixel; c4[1] = view; c4[2] = (uint32_t)(r * G + (k >> 2)); c4[3] = 0u;
                    philox4x32_10(c4, (uint32_t)seed, (uint32_t)(seed >> 32));
                }
                const uint32_t bits = (k & 2) ? ((k & 1) ? c4[3] : c4[2]) : ((k & 1) ? c4[1] : c4[0]);
                float uk = up ? up[k] : bits_to_uniform(bits);
                float pw = fmaxf(0.0f, leaf_mass(T, make_float4(xy.x, xy.y, 0.0f, 0.0f), qx, qy));
                float key = fdiv(uk, pw);
                int index = id;
                if (k + 1 < cnt) {  // the next leaf's record on its way
                    xy = T.leaf_xy[f0 + k + 1];
                    id = T.leaf_id[f0 + k + 1];
                }
                {
                    {
                        // the K smallest keys in order (an infinite or NaN key
                        // never enters)
                        if (KM <= 16) {
                            if (key < keys[KR - 1]) {
#pragma unroll UK
                                for (int q = 0; q < KR; ++q) {
                                    bool lt = key < keys[q];
                                    float tk = keys[q];
                                    int ti = ids[q];
                                    keys[q] = lt ? key : tk;
                                    ids[q] = lt ? index : ti;
                                    key = lt ? tk : key;
                                    index = lt ? ti : index;
                                }
                            }
                        } else if (key < last) {
                            // behind the keys that are not larger; from the end,
                            // four entries looked at together: one at a time this
                            // was two thirds of the descent at K = 40
                            const bool full_list = have == K;
                            const uint2 out = list[(K - 1) * 32 + lane];  // leaves a full list
                            int q = full_list ? K - 1 : have++;
                            unsigned above = full_list ? out.x : 0xffffffffu;  // (no key: a NaN)
                            bool equal = false, more = true;
#pragma unroll 1
                            while (more) {
                                uint2 x[4];
#pragma unroll
                                for (int u = 0; u < 4; ++u) x[u] = list[max(q - 1 - u, 0) * 32 + lane];
#pragma unroll
                                for (int u = 0; u < 4; ++u) {
                                    more = more && q > 0 && __uint_as_float(x[u].x) > key;
                                    if (more) {
                                        list[q * 32 + lane] = x[u];
                                        equal |= x[u].x == above;
                                        above = x[u].x;
                                        --q;
                                    }
                                }
                            }
                            list[q * 32 + lane] = make_uint2(__float_as_uint(key), (unsigned)index);
                            // the reference's list moves by swaps that pass equal
                            // keys by: of a run of them the first comes last (or
                            // leaves the list, if the run reaches past its end)
                            if (equal) {
#pragma unroll 1
                                for (int a = q + 1; a < have; ++a) {
                                    uint2 first = list[a * 32 + lane];
#pragma unroll 1
                                    for (; a + 1 < have; ++a) {
                                        const uint2 x = list[(a + 1) * 32 + lane];
                                        if (x.x != first.x) break;
                                        list[a * 32 + lane] = x;
                                    }
                                    if (full_list && a + 1 == K && out.x == first.x) first = out;
                                    list[a * 32 + lane] = first;
                                }
                            }
                            if (have == K) last = __uint_as_float(list[(K - 1) * 32 + lane].x);
                        }
                    }
                }
            }
        }
        if (overflow) atomicAdd(&st->overflow, 1);
        if (mine) {
            int* out = indices + (size_t)K * pixel;
            if (KM <= 16) {
#pragma unroll UK
                for (int k = 0; k < KR; ++k)
                    if (k < K) out[k] = ids[k];
            } else {
#pragma unroll 1
                for (int k = 0; k < K; ++k) out[k] = k < have ? (int)list[k * 32 + lane].y : -1;
            }
        }
    }
}

template <int R, int KM, bool UNEVEN, bool SPREAD>
__global__ void __launch_bounds__(32 * kDescentWarps<KM>, KM <= 16 ? kDescentBlocks : 8)
    k_sample(Tree T, const ViewState* vs, int W, int H, int K, int M, float precision,
             const float* __restrict__ uniforms, uint64_t seed, const uint64_t* __restrict__ seed_ptr, uint32_t view,
             int* __restrict__ indices, uds_view_stats* st, size_t vstride, size_t ustride, size_t istride,
             UnevenViews uv, Deferred df) {
    // block tile_x (y) x threads / tile_x (x), blockIdx.x its place among
    // the view's (cell_block).  blockIdx.y selects the view: its tree lives
    // vstride bytes after the previous view's, its uniforms ustride floats and
    // its indices istride entries further on.  With UNEVEN the view and the
    // block's place in it come from uv (blockIdx.x only; no uniforms tensor).
    if (seed_ptr) seed = *seed_ptr;
    unsigned at_block = blockIdx.x, vz = blockIdx.y;
    if (UNEVEN) {
        int b = 0;
        while (b + 1 < uv.nv && uv.first[b + 1] <= (int)blockIdx.x) ++b;
        at_block = blockIdx.x - (unsigned)uv.first[b];
        vz = (unsigned)b;
        W = uv.W[b];
        H = uv.H[b];
        indices += uv.ioff[b];
    }
    if (vz) {
        const size_t off = (size_t)vz * vstride;
        shift_tree(T, off);
        vs = shifted(vs, off);
        view += vz;
        if (!UNEVEN) {
            indices += (size_t)vz * istride;
            if (uniforms) uniforms += (size_t)vz * ustride;
        }
        st += vz;
    }
    __shared__ WarpTables s_tables[kDescentWarps<KM>];
    extern __shared__ uint2 list[];  // K > 16: (key, id) in order, one column per lane
    int i, j;
    cell_block(T.order, vs, W, H, at_block, i, j);
    if (i >= W || j >= H) return;  // (uniform over the block)
    i += threadIdx.y;
    j += threadIdx.x;
    int tid = threadIdx.x + blockDim.x * threadIdx.y;
    bool live = (i < W && j < H);
    T.n = vs->n;
    T.sq = vs->sq;
    T.isq = vs->isq;
    if (T.n == 0) return;  // indices were preset to -1 (uniform over the grid)
    sample_tile<R, KM, SPREAD>(T, s_tables[tid >> 5], list, __ballot_sync(0xffffffffu, live), i, j, H, K, M, precision,
                               uniforms, seed, view, indices, st, df, vz);
}

// The tiles that k_sample left for the long tables, a warp per block; uv.nv: 0
// or the number of views of different sizes.
template <int R, int KM>
__global__ void __launch_bounds__(32)
    k_sample_long(Tree first, const ViewState* first_vs, int H, int K, int M, float precision,
                  const float* __restrict__ uniforms, uint64_t seed, const uint64_t* __restrict__ seed_ptr,
                  uint32_t view, int* __restrict__ indices, uds_view_stats* st, size_t vstride, size_t ustride,
                  size_t istride, UnevenViews uv, Deferred df) {
    __shared__ LongTables wt;
    extern __shared__ uint2 list[];
    const unsigned count = min(df.counters[0], kDeferredTiles);
    if (count == 0) return;  // (the counters are still clear)
    if (seed_ptr) seed = *seed_ptr;
    use_slab(wt, df.slabs[blockIdx.x]);
    for (uint4 tile; next_deferred(df, count, tile);) {
        const unsigned vz = tile.z;
        Tree T = first;
        shift_tree(T, (size_t)vz * vstride);
        const ViewState* vs = shifted(first_vs, (size_t)vz * vstride);
        T.n = vs->n;
        T.sq = vs->sq;
        T.isq = vs->isq;
        sample_tile<R, KM, true>(T, wt, list, tile.w, (int)(tile.x + threadIdx.y), (int)(tile.y + threadIdx.x),
                                 uv.nv ? uv.H[vz] : H, K, M, precision, uniforms ? uniforms + vz * ustride : nullptr,
                                 seed, view + vz, indices + (uv.nv ? (size_t)uv.ioff[vz] : vz * istride), st + vz, df,
                                 vz);
    }
}

// Stochastic mode (no reference counterpart).  Each of the K draws of a
// pixel descends from the root into a child with probability
// m_child / (m_left + m_right), masses by getWeight, and records the product
// q of the ratios it took: the probability of having drawn that leaf, which
// importance-weighted estimators divide by.  Draw k at depth d uses Philox
// counter (pixel, view, 2^31 | k << 8 | d / 4, 0), component d % 4, and steps
// left iff u <= m_left / (m_left + m_right).  The draws of one pixel share
// their upper paths, so the child masses of the last path are kept per depth
// (node ids are unique, so a hit is exact).  A draw that meets two zero
// masses, or is still above the leaves after kTrace levels, stays -1 / 0.
template <class Tables>
__device__ __forceinline__ void stochastic_tile(const Tree& T, Tables& wt, unsigned todo, int i, int j, int H, int K,
                                                float precision, uint64_t seed, uint32_t view,
                                                int* __restrict__ indices, float* __restrict__ probs,
                                                uds_view_stats* st, float* __restrict__ weights, const Deferred& df) {
    float qx = (float)i, qy = (float)j;
    const unsigned full = 0xffffffffu;
    const int lane = (threadIdx.x + blockDim.x * threadIdx.y) & 31, n = T.n;
    const size_t pixel = (size_t)j + (size_t)H * i;
    float val_hi[Tables::kLong ? 1 : Tables::kEvals - Tables::kRows];
    bool overflow = false;
    int width = 32;
    while (todo) {
        unsigned group = lane_group(todo, width);
        float m0;
        const int state = warp_tables(T, qx, qy, group, width, 1, blockDim.x, wt, val_hi, m0);
        if (state < 0) {
            if (!Tables::kLong && width <= kDeferWidth && defer_tile(df, i, j, 0u, todo)) break;
            if (width > 1) {
                width >>= 1;
                continue;
            }
            group = todo;  // without tables: the lanes left walk side by side
        }
        todo &= ~group;
        const bool mine = (group >> lane) & 1u;
        if (state < 0 && mine) m0 = node_weight_out_of_line(T, 0, qx, qy);
        const Place root{0, 0, state, m0};
        m0 = fmaxf(0.0f, m0);
        bool act = mine && !(m0 < precision);
        if (!__any_sync(full, act)) continue;
        // child masses of the node last met at each depth outside the tables
        // (bit d of cvalid: slot d is set): the first levels from the stem on in
        // wt.path, three rows each, the others in local memory
        constexpr int kNear = kPathRows / 3;
        int cv_far[kTrace];
        float cw0_far[kTrace], cw1_far[kTrace];
        unsigned long long cvalid = 0ull;
        const Stem stem = state > 0 ? find_stem(wt) : Stem{0, 0, 0ull};
        for (int k = 0; k < K; ++k) {
            int d = 0;
            Place at = root;
            if (state <= 0) at.o = -1;
            int v = 0;
            int4 L = T.lnk[0];
            float prob = 1.0f;
            uint32_t c[4];
            bool ok = act;
            bool going = act && n > 1, pend = false, first = true;
            // on the stem the branch with the mass has probability 1
            if (state > 0 && m0 < __int_as_float(0x7f800000)) {
                d = stem.depth;
                at.o = stem.node;
            }
            while (true) {
                float w0 = 0.0f, w1 = 0.0f, sum0 = 0.0f, sum1 = 0.0f;
                uint4 E = make_uint4(0u, 0u, 0u, 0u);
                int split = 0;
                if (going && !pend) {
                    if (at.o >= 0) {
                        E = wt.open[at.o];
                        split = wt.split[at.o];
                        child_sums(wt, val_hi, lane, at, split, sum0, sum1);
                        w0 = fmaxf(0.0f, sum0);
                        w1 = fmaxf(0.0f, sum1);
                    } else {
                        pend = true;
                        const int q = d - stem.depth;
                        if ((cvalid >> d) & 1ull) {
                            if (q >= 0 && q < kNear) {
                                pend = __float_as_int(wt.path[3 * q][lane]) != v;
                                w0 = wt.path[3 * q + 1][lane];
                                w1 = wt.path[3 * q + 2][lane];
                            } else {
                                pend = cv_far[d] != v;
                                w0 = cw0_far[d];
                                w1 = cw1_far[d];
                            }
                        }
                    }
                }
                bool can = going && !pend;
                if (!__any_sync(full, can)) {
                    if (!__any_sync(full, pend)) break;
                    warp_child_masses<false>(T, wt, pend, L.x, L.y, qx, qy, w0, w1);
                    can = pend;
                    pend = false;
                    if (can) {
                        const int q = d - stem.depth;
                        if (q >= 0 && q < kNear) {
                            wt.path[3 * q][lane] = __int_as_float(v);
                            wt.path[3 * q + 1][lane] = w0;
                            wt.path[3 * q + 2][lane] = w1;
                        } else {
                            cv_far[d] = v;
                            cw0_far[d] = w0;
                            cw1_far[d] = w1;
                        }
                        cvalid |= 1ull << d;
                    }
                }
                if (can) {
                    if ((d & 3) == 0 || first) {
                        first = false;
                        c[0] = (uint32_t)pixel; c[1] = view; c[2] = 0x80000000u | ((uint32_t)k << 8) | (uint32_t)(d >> 2);
                        c[3] = 0;
                        philox4x32_10(c, (uint32_t)seed, (uint32_t)(seed >> 32));
                    }
                    float u = bits_to_uniform(c[d & 3]);
                    float sum = fadd(fadd(0.0f, w0), w1);
                    if (!(sum > 0.0f)) {
                        ok = false;
                        going = false;
                    } else {
                        float r0 = fdiv(w0, sum);
                        bool right = !(u <= r0);
                        prob = fmul(prob, right ? fdiv(w1, sum) : r0);
                        bool through = false;
                        unsigned link = 0u;
                        if (at.o >= 0) {
                            v = (int)(right ? E.z : E.y);
                            link = right ? E.x >> 16 : E.x & 0xffffu;
                            through = (link & kLinkKind) == kLinkOpen &&
                                      ((wt.open[link & kLinkEntry].w >> lane) & 1u);
                        } else {
                            v = right ? L.y : L.x;
                        }
                        if (through) {  // an opened node is not a leaf
                            at.o = (int)(link & kLinkEntry);
                            at.sum = right ? sum1 : sum0;
                            if (right) at.s = split; else at.t = split;
                        } else {
                            at.o = -1;
                            going = v < n - 1;
                            if (going) L = T.lnk[v];
                        }
                        ++d;
                        if (d >= kTrace && going) {
                            ok = false;
                            overflow = true;
                            going = false;
                        }
                    }
                }
            }
            if (ok) {
                size_t o = (size_t)K * pixel + k;
                indices[o] = T.leaf_id[v - (n - 1)];
                probs[o] = prob;
                // importance weight of the draw: (leaf mass / root mass) / q
                if (weights) weights[o] = leaf_mass(T, T.cen[v], qx, qy) / m0 / prob;
            }
        }
    }
    if (overflow) atomicAdd(&st->overflow, 1);
}

__global__ void __launch_bounds__(kDescentThreads, kDescentBlocks)
    k_stochastic(Tree T, const ViewState* vs, int W, int H, int K, float precision, uint64_t seed,
                 const uint64_t* __restrict__ seed_ptr, uint32_t view, int* __restrict__ indices,
                 float* __restrict__ probs, uds_view_stats* st, const unsigned char* __restrict__ mask,
                 float* __restrict__ weights, Deferred df) {
    // same tiles and tables as k_sample, then every lane draws its K paths; the
    // masses come from the tables, from those kept per depth of earlier draws,
    // or from the lane that needs them (all bit-identical to separate getWeight
    // calls)
    if (seed_ptr) seed = *seed_ptr;
    __shared__ WarpTables s_tables[kDescentThreads / 32];
    int i, j;
    cell_block(T.order, vs, W, H, blockIdx.x, i, j);
    if (i >= W || j >= H) return;  // (uniform over the block)
    i += threadIdx.y;
    j += threadIdx.x;
    int tid = threadIdx.x + blockDim.x * threadIdx.y;
    size_t pixel = (size_t)j + (size_t)H * i;
    bool live = (i < W && j < H) && (!mask || mask[pixel]);
    T.n = vs->n;
    T.sq = vs->sq;
    T.isq = vs->isq;
    if (T.n == 0) return;
    stochastic_tile(T, s_tables[tid >> 5], __ballot_sync(0xffffffffu, live), i, j, H, K, precision, seed, view, indices,
                    probs, st, weights, df);
}

// The tiles that k_stochastic left for the long tables.
__global__ void __launch_bounds__(32)
    k_stochastic_long(Tree T, const ViewState* vs, int H, int K, float precision, uint64_t seed,
                      const uint64_t* __restrict__ seed_ptr, uint32_t view, int* __restrict__ indices,
                      float* __restrict__ probs, uds_view_stats* st, float* __restrict__ weights, Deferred df) {
    __shared__ LongTables wt;
    const unsigned count = min(df.counters[0], kDeferredTiles);
    if (count == 0) return;  // (the counters are still clear)
    if (seed_ptr) seed = *seed_ptr;
    T.n = vs->n;
    T.sq = vs->sq;
    T.isq = vs->isq;
    use_slab(wt, df.slabs[blockIdx.x]);
    for (uint4 tile; next_deferred(df, count, tile);)
        stochastic_tile(T, wt, tile.w, (int)(tile.x + threadIdx.y), (int)(tile.y + threadIdx.x), H, K, precision, seed,
                        view, indices, probs, st, weights, df);
}

// ============================================================ proposal
// Learned proposal for the stochastic mode (no reference counterpart).  A
// draw descends from the root; at each internal node a small network maps
// 16 cheap features of the node's two children (offsets of the query from
// their centres, their leaf counts, box distances and sizes, all in units of
// sqrt(2) h) to the probability q of the left branch, instead of evaluating
// both children's FGT masses.  The draw's importance weight is
// p / q_path with p = (leaf Gaussian) / (root FGT mass): only the root mass
// is evaluated per pixel, and the weighted estimator stays unbiased because
// q > 0 on every branch.  The descent runs level-synchronously over all
// draws so that each level's network evaluations form one batch for the
// tensor-core kernel (uds_mlp_forward_dev).
constexpr int kFeat = 16;

__device__ __forceinline__ float feat_clamp(float x) { return fminf(fmaxf(x, -16.0f), 16.0f); }

__device__ __forceinline__ float box_distance(float4 b, float qx, float qy) {
    float dx = fmaxf(fmaxf(b.x - qx, qx - b.z), 0.0f), dy = fmaxf(fmaxf(b.y - qy, qy - b.w), 0.0f);
    return sqrtf(dx * dx + dy * dy);
}

__device__ void branch_features(const Tree& T, int v, int depth, float qx, float qy, float* f) {
    int4 L = T.lnk[v];
    float is = T.isq;
    float bd[2];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        int x = c ? L.y : L.x;
        float4 cc = T.cen[x], b = T.box[x];
        int cnt = T.lnk[x].w;
        bd[c] = box_distance(b, qx, qy) * is;
        f[6 * c + 0] = feat_clamp((qx - cc.x) * is);
        f[6 * c + 1] = feat_clamp((qy - cc.y) * is);
        f[6 * c + 2] = log2f((float)cnt) * 0.125f;
        f[6 * c + 3] = feat_clamp(bd[c]);
        f[6 * c + 4] = feat_clamp(0.5f * sqrtf((b.z - b.x) * (b.z - b.x) + (b.w - b.y) * (b.w - b.y)) * is);
        f[6 * c + 5] = x >= T.n - 1 ? 1.0f : 0.0f;
    }
    f[12] = (float)depth * (1.0f / 32.0f);
    f[13] = log2f((float)L.w) * 0.125f;
    f[14] = feat_clamp(bd[0] - bd[1]);
    f[15] = 0.0f;
}

__device__ __forceinline__ float draw_uniform(uint64_t seed, uint32_t pixel, uint32_t view, uint32_t tag, int k,
                                              int level) {
    uint32_t c[4] = {pixel, view, tag | ((uint32_t)k << 8) | (uint32_t)(level >> 2), 0u};
    philox4x32_10(c, (uint32_t)seed, (uint32_t)(seed >> 32));
    return bits_to_uniform(c[level & 3]);
}

// Training rows: plain stochastic descents (exact FGT masses) from every
// stride-th pixel in each direction, `draws` per pixel; each internal node
// visited gives (features, m_left / (m_left + m_right)).
__global__ void __launch_bounds__(128) k_prop_dataset(Tree T, const ViewState* vs, int W, int H, int stride,
                                                      int draws, float precision, uint64_t seed, uint32_t view,
                                                      float* __restrict__ X, float* __restrict__ target,
                                                      long long* __restrict__ keys, int* __restrict__ count,
                                                      int cap) {
    int j = (blockIdx.x * blockDim.x + threadIdx.x) * stride;
    int i = (blockIdx.y * blockDim.y + threadIdx.y) * stride;
    if (i >= W || j >= H) return;
    T.n = vs->n;
    T.sq = vs->sq;
    T.isq = vs->isq;
    int n = T.n;
    if (n < 2) return;
    float qx = (float)i, qy = (float)j;
    if (fmaxf(0.0f, node_weight(T, 0, qx, qy)) < precision) return;
    uint32_t pixel = (uint32_t)(j + H * i);
    int cn[kTrace];
    float cm0[kTrace], cm1[kTrace];
    for (int d = 0; d < kTrace; ++d) cn[d] = -1;
    for (int k = 0; k < draws; ++k) {
        int v = 0;
        for (int d = 0; v < n - 1 && d < kTrace; ++d) {
            int4 L = T.lnk[v];
            float w0, w1;
            if (cn[d] == v) {
                w0 = cm0[d];
                w1 = cm1[d];
            } else {
                w0 = fmaxf(0.0f, node_weight(T, L.x, qx, qy));
                w1 = fmaxf(0.0f, node_weight(T, L.y, qx, qy));
                cn[d] = v;
                cm0[d] = w0;
                cm1[d] = w1;
            }
            float sum = w0 + w1;
            if (!(sum > 0.0f)) break;
            float pl = w0 / sum;
            int r = atomicAdd(count, 1);
            if (r < cap) {
                float f[kFeat];
                branch_features(T, v, d, qx, qy, f);
#pragma unroll
                for (int q = 0; q < kFeat; ++q) X[(size_t)r * kFeat + q] = f[q];
                target[r] = pl;
                if (keys) keys[r] = ((long long)pixel << 16) | ((long long)k << 8) | d;
            }
            v = draw_uniform(seed, pixel, view, 0xA0000000u, k, d) <= pl ? L.x : L.y;
        }
    }
}

// Per pixel: root mass; active pixels put their K draws on the list.
struct PropInit {
    int K;
    float precision;
    float* root_mass;
    int *node, *draw;
    float* logq;
    int *count, *indices;
    float* weights;
};
template <class Tables>
__device__ __forceinline__ void prop_init_tile(const Tree& T, Tables& wt, unsigned todo, int i, int j, int H,
                                               const PropInit& out, const Deferred& df) {
    const int lane = (threadIdx.x + blockDim.x * threadIdx.y) & 31;
    const size_t pixel = (size_t)j + (size_t)H * i;
    const float qx = (float)i, qy = (float)j;
    bool live = (todo >> lane) & 1u;
    float m0 = 0.0f;
    if (T.n > 0) {
        float val_hi[Tables::kLong ? 1 : Tables::kEvals - Tables::kRows];
        int width = 32;
        while (todo) {
            unsigned group = lane_group(todo, width);
            float total;
            const int state = warp_tables(T, qx, qy, group, width, 1, blockDim.x, wt, val_hi, total);
            if (state < 0) {
                if (!Tables::kLong && width <= kDeferWidth && defer_tile(df, i, j, 0u, todo)) {
                    live = live && !((todo >> lane) & 1u);
                    break;
                }
                if (width > 1) {
                    width >>= 1;
                    continue;
                }
                group = todo;  // without tables: the lanes left walk side by side
            }
            todo &= ~group;
            if ((group >> lane) & 1u) m0 = state < 0 ? node_weight_out_of_line(T, 0, qx, qy) : total;
        }
        m0 = fmaxf(0.0f, m0);
    }
    if (!live) return;
    out.root_mass[pixel] = m0;
    if (T.n == 0 || m0 < out.precision) return;
    const int K = out.K;
    if (T.n == 1) {  // the root is the only leaf
        for (int k = 0; k < K; ++k) {
            out.indices[(size_t)K * pixel + k] = T.leaf_id[0];
            out.weights[(size_t)K * pixel + k] = leaf_mass(T, T.cen[0], qx, qy) / m0;
        }
        return;
    }
    int base = atomicAdd(out.count, K);
    for (int k = 0; k < K; ++k) {
        out.node[base + k] = 0;
        out.draw[base + k] = (int)(pixel * K + k);
        out.logq[base + k] = 0.0f;
    }
}

__global__ void __launch_bounds__(kDescentThreads, kDescentBlocks)
    k_prop_init(Tree T, const ViewState* vs, int W, int H, PropInit out, Deferred df) {
    // root masses from the tables of k_sample (warps of consecutive
    // threads)
    __shared__ WarpTables s_tables[kDescentThreads / 32];
    int j = blockIdx.x * blockDim.x + threadIdx.x;
    int i = blockIdx.y * blockDim.y + threadIdx.y;
    int tid = threadIdx.x + blockDim.x * threadIdx.y;
    T.n = vs->n;
    T.sq = vs->sq;
    T.isq = vs->isq;
    prop_init_tile(T, s_tables[tid >> 5], __ballot_sync(0xffffffffu, i < W && j < H), i, j, H, out, df);
}

// The tiles that k_prop_init left for the long tables.
__global__ void __launch_bounds__(32)
    k_prop_init_long(Tree T, const ViewState* vs, int H, PropInit out, Deferred df) {
    __shared__ LongTables wt;
    const unsigned count = min(df.counters[0], kDeferredTiles);
    if (count == 0) return;  // (the counters are still clear)
    T.n = vs->n;
    T.sq = vs->sq;
    T.isq = vs->isq;
    use_slab(wt, df.slabs[blockIdx.x]);
    for (uint4 tile; next_deferred(df, count, tile);)
        prop_init_tile(T, wt, tile.w, (int)(tile.x + threadIdx.y), (int)(tile.y + threadIdx.x), H, out, df);
}

// Rows go straight into the network's operand layout: bf16, 128-row tiles of
// 4096 bytes, K-major core matrices (two 16-byte stores per row), so the
// network kernel can stream whole tiles with bulk copies.
__global__ void k_prop_features(Tree T, const ViewState* vs, int H, int K, int level, const int* __restrict__ count,
                                const int* __restrict__ node_in, const int* __restrict__ draw_in,
                                unsigned char* __restrict__ Xt) {
    int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= *count) return;
    T.n = vs->n;
    T.sq = vs->sq;
    T.isq = vs->isq;
    int pixel = draw_in[r] / K;
    float qx = (float)(pixel / H), qy = (float)(pixel % H);
    float f[kFeat];
    branch_features(T, node_in[r], level, qx, qy, f);
    unsigned char* tile = Xt + (size_t)(r >> 7) * (128 * kFeat * 2);
#pragma unroll
    for (int c = 0; c < kFeat; c += 8) {
        __nv_bfloat162 h[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) h[q] = __floats2bfloat162_rn(f[c + 2 * q], f[c + 2 * q + 1]);
        *reinterpret_cast<uint4*>(tile + tc::kmajor_offset(r & 127, c, kFeat)) = *reinterpret_cast<uint4*>(h);
    }
}

// Take one branch per draw with the network's q; finished draws write their
// leaf and importance weight, the others go on the next level's list.
__global__ void k_prop_step(Tree T, const ViewState* vs, int H, int K, int level, uint64_t seed,
                            const uint64_t* __restrict__ seed_ptr, uint32_t view, const int* __restrict__ count_in,
                            const int* __restrict__ node_in, const int* __restrict__ draw_in,
                            const float* __restrict__ logq_in, const float* __restrict__ logits,
                            const float* __restrict__ root_mass, int* __restrict__ count_out,
                            int* __restrict__ node_out, int* __restrict__ draw_out, float* __restrict__ logq_out,
                            int* __restrict__ indices, float* __restrict__ weights) {
    int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= *count_in) return;
    if (seed_ptr) seed = *seed_ptr;
    T.n = vs->n;
    T.sq = vs->sq;
    T.isq = vs->isq;
    int draw = draw_in[r];
    int pixel = draw / K, k = draw % K;
    int v = node_in[r];
    int4 L = T.lnk[v];
    float z0 = logits[2 * r], z1 = logits[2 * r + 1];
    float m = fmaxf(z0, z1);
    float e0 = __expf(z0 - m), e1 = __expf(z1 - m);
    float q0 = e0 / (e0 + e1);
    float u = draw_uniform(seed, (uint32_t)pixel, view, 0xC0000000u, k, level);
    bool left = u <= q0;
    float qc = left ? q0 : 1.0f - q0;
    float logq = logq_in[r] + __logf(fmaxf(qc, 1e-30f));
    int c = left ? L.x : L.y;
    if (c >= T.n - 1) {
        float qx = (float)(pixel / H), qy = (float)(pixel % H);
        float g = leaf_mass(T, T.cen[c], qx, qy);
        indices[draw] = T.leaf_id[c - (T.n - 1)];
        weights[draw] = g / root_mass[pixel] * __expf(-logq);
    } else if (level + 1 < kTrace) {
        int o = atomicAdd(count_out, 1);
        node_out[o] = c;
        draw_out[o] = draw;
        logq_out[o] = logq;
    }
}

// Effective sample size of each pixel's K weighted draws; pixels below
// tau * K are marked for the plain sampler.
__global__ void k_prop_ess(int W, int H, int K, float tau, const float* __restrict__ root_mass, float precision,
                           const float* __restrict__ weights, unsigned char* __restrict__ mask,
                           int* __restrict__ nfallback) {
    size_t pixel = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (pixel >= (size_t)W * H) return;
    unsigned char fb = 0;
    if (root_mass[pixel] >= precision) {
        float s1 = 0.0f, s2 = 0.0f;
        for (int k = 0; k < K; ++k) {
            float w = weights[(size_t)K * pixel + k];
            s1 += w;
            s2 += w * w;
        }
        fb = !(s2 > 0.0f && s1 * s1 >= tau * (float)K * s2);  // also when no draw finished
    }
    mask[pixel] = fb;
    if (fb) atomicAdd(nfallback, 1);
}

__global__ void k_prop_clear(size_t P, int K, const unsigned char* __restrict__ mask, int* __restrict__ indices,
                             float* __restrict__ weights) {
    size_t pixel = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (pixel >= P || !mask[pixel]) return;
    for (int k = 0; k < K; ++k) {
        indices[(size_t)K * pixel + k] = -1;
        weights[(size_t)K * pixel + k] = 0.0f;
    }
}

// One block per view: its statistics, and its cells in order of falling count
// (counting sort; cells of about the same count in any order).
constexpr int kFinishThreads = 1024, kBuckets = 128;
__global__ void __launch_bounds__(kFinishThreads) k_finish_view(Batch bt, ViewState* vs, uds_view_stats* st,
                                                                const uint32_t* __restrict__ cells,
                                                                unsigned short* __restrict__ order) {
    const int W = bt.W[blockIdx.x], H = bt.H[blockIdx.x];
    vs = shifted(vs, bt.slot * blockIdx.x);
    cells = shifted(cells, bt.slot * blockIdx.x);
    order = shifted(order, bt.slot * blockIdx.x);
    st += bt.first + blockIdx.x;
    __shared__ int place[kBuckets];
    __shared__ uint32_t count[kCells];
    const int t = threadIdx.x, sh = cell_shift(W, H), rows = cell_columns(W, sh), columns = cell_columns(H, sh);
    const int n = rows * columns;
    for (int c = t; c < n; c += kFinishThreads) count[c] = cells[c];
    if (t == 0) {
        if (vs->failed) {
            vs->n = 0;
            st->reserved[0] = 1;
        }
        st->n_visible = vs->n;
        st->n_coefs = (int)vs->coef_used;
    }
    if (t < kBuckets) place[t] = 0;
    __syncthreads();
    // bucket 127: empty; below, four per power of two, larger counts first.  A
    // pixel sees splats up to a few bandwidths away: the neighbours count too.
    unsigned char own[kCells / kFinishThreads];  // this thread's cells' buckets
    auto bucket = [&](int c) {
        const int i = c / columns, j = c % columns;
        unsigned x = 0;
        for (int a = max(i - 1, 0); a <= min(i + 1, rows - 1); ++a)
            for (int b = max(j - 1, 0); b <= min(j + 1, columns - 1); ++b) x += count[a * columns + b];
        return x ? (int)(kBuckets - 2 - ((__float_as_uint((float)x) >> 21) - (127u << 2))) : kBuckets - 1;
    };
#pragma unroll
    for (int q = 0; q < kCells / kFinishThreads; ++q) {
        const int c = t + q * kFinishThreads;
        if (c >= n) continue;
        own[q] = (unsigned char)bucket(c);
        atomicAdd(&place[own[q]], 1);
    }
    __syncthreads();
    if (t < 32) {  // exclusive sums, four buckets per lane
        int x[kBuckets / 32], sum = 0;
#pragma unroll
        for (int q = 0; q < kBuckets / 32; ++q) {
            x[q] = sum;
            sum += place[t * (kBuckets / 32) + q];
        }
        int before = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, before, o);
            if (t >= o) before += y;
        }
        before -= sum;
#pragma unroll
        for (int q = 0; q < kBuckets / 32; ++q) place[t * (kBuckets / 32) + q] = before + x[q];
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kCells / kFinishThreads; ++q) {
        const int c = t + q * kFinishThreads;
        if (c < n) order[atomicAdd(&place[own[q]], 1)] = (unsigned short)c;
    }
}

// Evaluate getWeight for (node, query) pairs (debug entry point).
__global__ void k_fgt_eval(Tree T, const ViewState* vs, int m, const int* __restrict__ nodes,
                           const float* __restrict__ q, float* __restrict__ out) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= m) return;
    T.n = vs->n;
    T.sq = vs->sq;
    T.isq = vs->isq;
    out[t] = node_weight(T, nodes[t], q[2 * t], q[2 * t + 1]);
}

// ------------------------------------------------------------ host side
cudaError_t sample_wait_failures(unsigned* count) {
    return cudaMemcpyFromSymbol(count, g_wait_failures, sizeof(*count));
}

// Trees of the batch's views in the slots from w on; w.stats: the first view's
// of the call.
static int build_batch(const uds_sample_params* p, const Ws& w, const Batch& bt, const float* pts, const float* nrm,
                       const float* sd, const float* h_override, cudaStream_t s) {
    const int N = p->N, nv = bt.count;
    cudaError_t e = cudaSuccess;
    if (nv > 1 && bt.slot < (1ull << 31)) {  // (the pitch of a 2D memset is limited)
        e = cudaMemset2DAsync(w.vs, bt.slot, 0, w.zeroed, nv, s);
    } else {
        for (int k = 0; k < nv && e == cudaSuccess; ++k)
            e = cudaMemsetAsync(reinterpret_cast<char*>(w.vs) + bt.slot * k, 0, w.zeroed, s);
    }
    if (e != cudaSuccess) { set_last_error(e); return UDS_ERR_CUDA; }
    // four splats per thread, one where that would leave SMs without a block
    if ((size_t)cdiv(N, 4 * kTileThreads) * nv < 304)
        k_bandwidth<1><<<dim3(cdiv(N > 0 ? N : 1, kTileThreads), nv), kTileThreads, 0, s>>>(
            N, bt, pts, nrm, sd, p->std_batch, p->smoothing, h_override, p->precision, w.vs, w.stats);
    else
        k_bandwidth<4><<<dim3(cdiv(N, 4 * kTileThreads), nv), kTileThreads, 0, s>>>(
            N, bt, pts, nrm, sd, p->std_batch, p->smoothing, h_override, p->precision, w.vs, w.stats);
    int st;
    if ((st = launch_status())) return st;
    if (N == 0) return UDS_OK;
    const int tiles = (int)cdiv(N, kTile);
    const dim3 grid_tiles(tiles, nv), grid(cdiv(N, 128), nv);
    k_cull<<<grid_tiles, kTileThreads, 0, s>>>(N, bt, pts, w.vs, w.cull_status, w.hist, w.keysB, w.idsB);
    uint32_t *ki = w.keysB, *vi = w.idsB, *ko = w.keysA, *vo = w.idsA;
    for (int pass = 0; pass < kPasses; ++pass) {  // an odd number: the sorted splats end in A
        k_sort_pass<<<grid_tiles, kTileThreads, 0, s>>>(bt, pass, tiles, w.vs, w.hist, w.sort_status, ki, vi, ko, vo);
        uint32_t* t = ki; ki = ko; ko = t;
        t = vi; vi = vo; vo = t;
    }
    k_tree<<<grid, 128, 0, s>>>(N, bt, pts, w.vs, p->precision, w);
    const int P = p->fixed_degree;
    k_bottomup<<<grid, 128, 0, s>>>(bt, w.vs, p->precision, P > 0 ? P : p->max_degree, w);
    if ((st = launch_status(3 + kPasses))) return st;
    if (P > 0) {
        for (int k = 0; k < nv; ++k) {
            const Ws v = layout(p, reinterpret_cast<char*>(w.vs) + bt.slot * k);
            k_fixed_assign<<<cdiv(N, 128), 128, 0, s>>>(v.vs, v.cen, P);
            e = cudaMemsetAsync(v.fanin, 0, 4 * (size_t)N, s);
            if (e != cudaSuccess) { set_last_error(e); return UDS_ERR_CUDA; }
            switch (P) {
                case 4: k_m2m<4><<<cdiv(N, 128), 128, 0, s>>>(v.vs, v.lnk, v.par, v.cen, v.coef, v.fanin); break;
                case 6: k_m2m<6><<<cdiv(N, 128), 128, 0, s>>>(v.vs, v.lnk, v.par, v.cen, v.coef, v.fanin); break;
                default: k_m2m<8><<<cdiv(N, 128), 128, 0, s>>>(v.vs, v.lnk, v.par, v.cen, v.coef, v.fanin); break;
            }
            if ((st = launch_status(2))) return st;
        }
    } else {
        k_p2m<<<dim3(cdiv(N, kNodeTile), nv), kNodeTile, 0, s>>>(bt, w.vs, w.coef_cap, w.stats, w);
        if ((st = launch_status())) return st;
    }
    k_finish_view<<<nv, kFinishThreads, 0, s>>>(bt, w.vs, w.stats, w.cells, w.order);
    return launch_status();
}

// One view's tree in the slot at w.
static int build_view(const uds_sample_params* p, const Ws& w, int view, const float* pts, const float* nrm,
                      const float* sd, const float* h_override, cudaStream_t s) {
    Batch bt{};
    bt.first = view;
    bt.count = 1;
    bt.W[0] = p->W;
    bt.H[0] = p->H;
    bt.f[0] = p->focal;
    return build_batch(p, w, bt, pts, nrm, sd, h_override, s);
}

// Every view's tree in its own slot, from base on; views: of different sizes,
// or null for those of p.
static int build_views(const uds_sample_params* p, char* base, size_t slot, const uds_view_desc* views,
                       const float* pts, const float* nrm, const float* sd, const float* h_override, cudaStream_t s) {
    for (int first = 0; first < p->B; first += kBatch) {
        Batch bt{};
        bt.slot = slot;
        bt.first = first;
        bt.count = p->B - first < kBatch ? p->B - first : kBatch;
        for (int k = 0; k < bt.count; ++k) {
            bt.W[k] = views ? views[first + k].W : p->W;
            bt.H[k] = views ? views[first + k].H : p->H;
            bt.f[k] = views ? views[first + k].focal : p->focal;
        }
        Ws w = layout(p, base + slot * (size_t)first);
        w.stats = layout(p, base).stats;
        if (int st = build_batch(p, w, bt, pts, nrm, sd, h_override, s)) return st;
    }
    return UDS_OK;
}

// What the tiles left for the long tables take: their list and the slabs,
// one per block of the second kernel (fewer for few splats, where such tiles
// are fewer), at the end of the workspace.  None where every pixel fits the
// short ones.
static unsigned long_blocks(const uds_sample_params* p) {
    if (p->N <= WarpTables::kEvals) return 0;  // (fewer nodes than splats)
    const int n = p->N / 1024;
    return (unsigned)(n < 8 ? 8 : n > 152 ? 152 : n);
}
static size_t deferred_bytes(const uds_sample_params* p) {
    const unsigned blocks = long_blocks(p);
    return blocks ? a256(sizeof(uint4) * kDeferredTiles) + blocks * a256(sizeof(LongSlab)) : 0;
}
static Deferred deferred_of(const uds_sample_params* p, const Ws& w, char* workspace, size_t workspace_bytes) {
    char* at = workspace + ((workspace_bytes - deferred_bytes(p)) & ~(size_t)255);
    return {w.vs->deferred, reinterpret_cast<uint4*>(at),
            reinterpret_cast<LongSlab*>(at + a256(sizeof(uint4) * kDeferredTiles))};
}

// Leaves one order-sampling round considers: the descent stops at the first
// node holding at most max(K, leaf_size) splats.
static int candidates(const uds_sample_params* p) { return p->leaf_size > p->K ? p->leaf_size : p->K; }

// Columns of the warp tile: 4 or 8 (wider tiles share fewer row sums: at 16
// the descent took a third longer, so 16 and 32 run as 8).
static int tile_of(const uds_sample_params* p) { return p->tile_x == 4 ? 4 : 8; }

static Tree tree_of(const Ws& w) {
    Tree T;
    T.lnk = w.lnk; T.par = w.par; T.box = w.box; T.cen = w.cen; T.coef = w.coef;
    T.leaf_xy = w.leaf_xy; T.leaf_id = w.leaf_id; T.order = w.order; T.n = 0; T.sq = 0.0f; T.isq = 0.0f;
    return T;
}

// Descent for views view .. view + nviews - 1 in one launch (grid.y = view),
// their trees vstride bytes apart in the workspace, and that of the tiles it
// leaves for the long tables.  Block: tile_x (y) by kDescentThreads / tile_x
// (x) pixels; each warp is a tile_x by 32 / tile_x pixel tile.  Every lane's
// walk is its own, so the indices do not depend on the tile shape, only the
// speed does.
template <int R>
static int launch_sample(const Tree& T, const Ws& w, const uds_sample_params* p, const Deferred& df, const float* u,
                         int view, int* idx, cudaStream_t s, int nviews = 1, size_t vstride = 0) {
    // the K smallest keys in registers up to 16, in shared memory above
    constexpr bool kEight = R <= 3;
    constexpr int RR = R >= 3 ? R : 3, KM = RR <= 4 ? 16 : kMaxK;
    const int tx = tile_of(p), M = candidates(p);
    const size_t istride = (size_t)p->W * p->H * p->K, ustride = (size_t)p->W * p->H * R * M;
    const unsigned more = long_blocks(p);
    const dim3 tile(tx, 32 / tx);
    UnevenViews none{};
    auto launch = [&](auto kernel, auto rest, int warps, size_t list) {
        const dim3 block(tx, 32 * warps / tx), grid(cell_blocks(p->W, p->H, block), nviews);
        kernel<<<grid, block, list, s>>>(T, w.vs, p->W, p->H, p->K, M, p->precision, u, p->seed, p->seed_dev,
                                         (uint32_t)view, idx, w.stats + view, vstride, ustride, istride, none, df);
        if (more)
            rest<<<more, tile, list, s>>>(T, w.vs, p->H, p->K, M, p->precision, u, p->seed, p->seed_dev,
                                          (uint32_t)view, idx, w.stats + view, vstride, ustride, istride, none, df);
    };
    if (kEight && p->K <= 8) {
        constexpr int R8 = kEight ? R : 3;
        launch(p->spread ? k_sample<R8, 8, false, true> : k_sample<R8, 8, false, false>, k_sample_long<R8, 8>,
               kDescentWarps<8>, 0);
    } else {
        launch(k_sample<RR, KM, false, true>, k_sample_long<RR, KM>, kDescentWarps<KM>,
               KM <= 16 ? 0 : 256 * (size_t)p->K);
    }
    return launch_status(more ? 2 : 1);
}
static int launch_descent(const Tree& T, const Ws& w, const uds_sample_params* p, const Deferred& df, const float* u,
                          int view, int* idx, cudaStream_t s, int nviews = 1, size_t vstride = 0) {
    switch (num_rounds(p->K)) {
        case 1: return launch_sample<1>(T, w, p, df, u, view, idx, s, nviews, vstride);
        case 2: return launch_sample<2>(T, w, p, df, u, view, idx, s, nviews, vstride);
        case 3: return launch_sample<3>(T, w, p, df, u, view, idx, s, nviews, vstride);
        case 4: return launch_sample<4>(T, w, p, df, u, view, idx, s, nviews, vstride);
        case 5: return launch_sample<5>(T, w, p, df, u, view, idx, s, nviews, vstride);
        case 6: return launch_sample<6>(T, w, p, df, u, view, idx, s, nviews, vstride);
        case 7: return launch_sample<7>(T, w, p, df, u, view, idx, s, nviews, vstride);
        default: return launch_sample<8>(T, w, p, df, u, view, idx, s, nviews, vstride);
    }
}

// Views of different sizes (K <= 8) in one launch: a one-dimensional grid of
// every view's blocks; uv built by the caller.
template <int R>
static int launch_sample_uneven(const Tree& T, const Ws& w, const uds_sample_params* p, const Deferred& df,
                                const UnevenViews& uv, int* idx, cudaStream_t s, size_t vstride) {
    const int tx = tile_of(p), M = candidates(p);
    const unsigned more = long_blocks(p);
    auto kernel = p->spread ? k_sample<R, 8, true, true> : k_sample<R, 8, true, false>;
    kernel<<<uv.first[uv.nv], dim3(tx, kDescentThreads / tx), 0, s>>>(T, w.vs, 0, 0, p->K, M, p->precision, nullptr,
                                                                     p->seed, p->seed_dev, 0u, idx, w.stats, vstride,
                                                                     0, 0, uv, df);
    if (more)
        k_sample_long<R, 8><<<more, dim3(tx, 32 / tx), 0, s>>>(T, w.vs, 0, p->K, M, p->precision, nullptr, p->seed,
                                                              p->seed_dev, 0u, idx, w.stats, vstride, 0, 0, uv, df);
    return launch_status(more ? 2 : 1);
}

static int check_params(const uds_sample_params* p) {
    if (!p) return UDS_ERR_ARGUMENT;
    if (p->B <= 0 || p->N < 0 || p->W <= 0 || p->H <= 0 || p->K <= 0 || p->K > kMaxK) return UDS_ERR_ARGUMENT;
    if (p->max_degree < 0 || p->max_degree > kMaxDegree) return UDS_ERR_ARGUMENT;
    if (p->std_batch != 1 && p->std_batch != p->B) return UDS_ERR_ARGUMENT;
    if (!(p->precision > 0.0f) || !(p->focal > 0.0f)) return UDS_ERR_ARGUMENT;
    if ((size_t)p->N * 2 >= (1u << 31)) return UDS_ERR_ARGUMENT;
    if (p->tile_x != 0 && p->tile_x != 4 && p->tile_x != 8 && p->tile_x != 16 && p->tile_x != 32)
        return UDS_ERR_ARGUMENT;
    if (p->leaf_size < 0 || p->leaf_size > kMaxLeaf) return UDS_ERR_ARGUMENT;
    if (p->spread != 0 && p->spread != 1) return UDS_ERR_ARGUMENT;
    if (p->fixed_degree != 0) {
        if (p->fixed_degree != 4 && p->fixed_degree != 6 && p->fixed_degree != 8) return UDS_ERR_ARGUMENT;
        int64_t need = (int64_t)(p->N > 1 ? p->N - 1 : 0) * (p->fixed_degree + 1) * (p->fixed_degree + 1);
        int64_t cap = p->coef_pool > 0 ? p->coef_pool : default_pool(p->N);
        if (need > cap) return UDS_ERR_ARGUMENT;  // one expansion per internal node must fit the pool
    }
    int64_t pool = p->coef_pool > 0 ? p->coef_pool : default_pool(p->N);
    if (pool >= (1ll << 26)) return UDS_ERR_ARGUMENT;  // offsets are packed in 26 bits
    return UDS_OK;
}

}  // namespace uds

using namespace uds;

// uds_sample keeps every view's tree resident (one slot per view) so that one
// descent launch covers all views; the other entry points use slot 0.
extern "C" size_t uds_sample_workspace_size(const uds_sample_params* prm) {
    if (check_params(prm)) return 0;
    return layout(prm, nullptr).bytes * (size_t)prm->B + deferred_bytes(prm);
}

extern "C" int uds_sample(const uds_sample_params* prm, const float* points, const float* normals,
                          const float* std_devs, const float* uniforms, const float* h_override,
                          int32_t* indices, uds_view_stats* stats, void* workspace, size_t workspace_bytes,
                          void* stream) {
    int st = check_params(prm);
    if (st) return st;
    if (!indices || (prm->N > 0 && (!points || !normals || !std_devs))) return UDS_ERR_ARGUMENT;
    char* base = reinterpret_cast<char*>(workspace);
    Ws w = layout(prm, base);
    size_t slot = w.bytes;
    if (!workspace || workspace_bytes < slot * (size_t)prm->B + deferred_bytes(prm)) return UDS_ERR_WORKSPACE;
    cudaStream_t s = as_stream(stream);
    size_t per_view = (size_t)prm->W * prm->H * prm->K;
    cudaError_t e = cudaMemsetAsync(indices, 0xFF, sizeof(int32_t) * per_view * prm->B, s);
    if (e != cudaSuccess) { set_last_error(e); return UDS_ERR_CUDA; }
    if ((st = build_views(prm, base, slot, nullptr, points, normals, std_devs, h_override, s))) return st;
    if (prm->N > 0) {
        // one descent launch over all views
        const Deferred df = deferred_of(prm, w, base, workspace_bytes);
        if ((st = launch_descent(tree_of(w), w, prm, df, uniforms, 0, indices, s, prm->B, slot))) return st;
    }
    if (stats) {
        e = cudaMemcpyAsync(stats, w.stats, sizeof(uds_view_stats) * prm->B, cudaMemcpyDeviceToDevice, s);
        if (e != cudaSuccess) { set_last_error(e); return UDS_ERR_CUDA; }
    }
    return UDS_OK;
}

// Views of different sizes in one call: every view's tree in its own slot,
// then one descent launch over all views' pixels (K <= 8; larger K, or more
// than kMaxUneven views, one launch per view).  prm->W, H and focal are
// replaced by each view's; indices are packed view after view.
extern "C" int uds_sample_views(const uds_sample_params* prm, const uds_view_desc* views, const float* points,
                                const float* normals, const float* std_devs, const float* h_override,
                                int32_t* indices, uds_view_stats* stats, void* workspace, size_t workspace_bytes,
                                void* stream) {
    int st = check_params(prm);
    if (st) return st;
    if (!views || !indices || (prm->N > 0 && (!points || !normals || !std_devs))) return UDS_ERR_ARGUMENT;
    size_t total = 0;
    for (int b = 0; b < prm->B; ++b) {
        if (views[b].W <= 0 || views[b].H <= 0 || !(views[b].focal > 0.0f)) return UDS_ERR_ARGUMENT;
        total += (size_t)views[b].W * views[b].H * prm->K;
    }
    char* base = reinterpret_cast<char*>(workspace);
    Ws w = layout(prm, base);
    size_t slot = w.bytes;  // does not depend on the image size
    if (!workspace || workspace_bytes < slot * (size_t)prm->B + deferred_bytes(prm)) return UDS_ERR_WORKSPACE;
    cudaStream_t s = as_stream(stream);
    cudaError_t e = cudaMemsetAsync(indices, 0xFF, sizeof(int32_t) * total, s);
    if (e != cudaSuccess) { set_last_error(e); return UDS_ERR_CUDA; }
    if ((st = build_views(prm, base, slot, views, points, normals, std_devs, h_override, s))) return st;
    if (prm->N > 0) {
        Tree T = tree_of(w);
        int R = num_rounds(prm->K);
        int tx = tile_of(prm);
        if (prm->K <= 8 && prm->B <= kMaxUneven) {
            UnevenViews uv{};
            uv.nv = prm->B;
            long long off = 0;
            int blocks = 0;
            for (int b = 0; b < prm->B; ++b) {
                uv.first[b] = blocks;
                uv.W[b] = views[b].W;
                uv.H[b] = views[b].H;
                uv.ioff[b] = off;
                blocks += (int)cell_blocks(views[b].W, views[b].H, dim3(tx, kDescentThreads / tx));
                off += (long long)views[b].W * views[b].H * prm->K;
            }
            uv.first[prm->B] = blocks;
            const Deferred df = deferred_of(prm, w, base, workspace_bytes);
            switch (R) {
                case 1: st = launch_sample_uneven<1>(T, w, prm, df, uv, indices, s, slot); break;
                case 2: st = launch_sample_uneven<2>(T, w, prm, df, uv, indices, s, slot); break;
                default: st = launch_sample_uneven<3>(T, w, prm, df, uv, indices, s, slot); break;
            }
            if (st) return st;
        } else {
            size_t off = 0;
            for (int b = 0; b < prm->B; ++b) {
                uds_sample_params pv = *prm;
                pv.W = views[b].W;
                pv.H = views[b].H;
                Ws wb = layout(&pv, base + slot * (size_t)b);
                wb.stats = w.stats;
                const Deferred df = deferred_of(prm, wb, base, workspace_bytes);
                if ((st = launch_descent(tree_of(wb), wb, &pv, df, nullptr, b, indices + off, s))) return st;
                off += (size_t)views[b].W * views[b].H * prm->K;
            }
        }
    }
    if (stats) {
        e = cudaMemcpyAsync(stats, w.stats, sizeof(uds_view_stats) * prm->B, cudaMemcpyDeviceToDevice, s);
        if (e != cudaSuccess) { set_last_error(e); return UDS_ERR_CUDA; }
    }
    return UDS_OK;
}

namespace uds {
// Draws of one view's pixels (with a mask: of those it marks).
static int launch_stochastic(const Ws& w, const uds_sample_params* p, const Deferred& df, int view, int* idx,
                             float* probs, const unsigned char* mask, float* weights, cudaStream_t s) {
    const dim3 block(8, kDescentThreads / 8);
    const Tree T = tree_of(w);
    const unsigned more = long_blocks(p);
    k_stochastic<<<cell_blocks(p->W, p->H, block), block, 0, s>>>(T, w.vs, p->W, p->H, p->K, p->precision, p->seed,
                                                                  p->seed_dev, (uint32_t)view, idx, probs,
                                                                  w.stats + view, mask, weights, df);
    if (more)
        k_stochastic_long<<<more, dim3(8, 4), 0, s>>>(T, w.vs, p->H, p->K, p->precision, p->seed, p->seed_dev,
                                                      (uint32_t)view, idx, probs, w.stats + view, weights, df);
    return launch_status(more ? 2 : 1);
}
}  // namespace uds

extern "C" int uds_sample_stochastic(const uds_sample_params* prm, const float* points, const float* normals,
                                     const float* std_devs, const float* h_override, int32_t* indices,
                                     float* probs, uds_view_stats* stats, void* workspace, size_t workspace_bytes,
                                     void* stream) {
    int st = check_params(prm);
    if (st) return st;
    if (!indices || !probs || (prm->N > 0 && (!points || !normals || !std_devs))) return UDS_ERR_ARGUMENT;
    char* base = reinterpret_cast<char*>(workspace);
    Ws w = layout(prm, base);
    if (!workspace || workspace_bytes < w.bytes + deferred_bytes(prm)) return UDS_ERR_WORKSPACE;
    cudaStream_t s = as_stream(stream);
    size_t per_view = (size_t)prm->W * prm->H * prm->K;
    cudaError_t e = cudaMemsetAsync(indices, 0xFF, sizeof(int32_t) * per_view * prm->B, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(probs, 0, sizeof(float) * per_view * prm->B, s);
    if (e != cudaSuccess) { set_last_error(e); return UDS_ERR_CUDA; }
    const Deferred df = deferred_of(prm, w, base, workspace_bytes);
    for (int b = 0; b < prm->B; ++b) {
        if ((st = build_view(prm, w, b, points, normals, std_devs, h_override, s))) return st;
        if (prm->N == 0) continue;
        if ((st = launch_stochastic(w, prm, df, b, indices + per_view * b, probs + per_view * b, nullptr, nullptr, s)))
            return st;
    }
    if (stats) {
        e = cudaMemcpyAsync(stats, w.stats, sizeof(uds_view_stats) * prm->B, cudaMemcpyDeviceToDevice, s);
        if (e != cudaSuccess) { set_last_error(e); return UDS_ERR_CUDA; }
    }
    return UDS_OK;
}

extern "C" int uds_tree_build(const uds_sample_params* prm, int view, const float* points,
                              const float* normals, const float* std_devs, const float* h_override,
                              uds_view_stats* stats, uint32_t* keys, int32_t* ids, int32_t* left,
                              int32_t* right, int32_t* parent, int32_t* count, int32_t* degree, float* centre,
                              float* box, void* workspace, size_t workspace_bytes, void* stream);

namespace uds {
// Copy the built tree into plain per-node arrays (debug).
__global__ void k_export(const ViewState* vs, const Ws w, uint32_t* keys, int* ids, int* left, int* right,
                         int* parent, int* count, int* degree, float* centre, float* box) {
    int v = blockIdx.x * blockDim.x + threadIdx.x;
    int n = vs->n;
    int M = n > 0 ? 2 * n - 1 : 0;
    if (v < n) {
        if (keys) keys[v] = w.keysA[v];
        if (ids) ids[v] = w.leaf_id[v];
    }
    if (v < M) {
        int4 L = w.lnk[v];
        float4 c = w.cen[v], b = w.box[v];
        if (left) left[v] = L.x;
        if (right) right[v] = L.y;
        if (parent) parent[v] = w.par[v];
        if (count) count[v] = L.w;
        if (degree) degree[v] = meta_degree(c.w);
        if (centre) { centre[2 * v] = c.x; centre[2 * v + 1] = c.y; }
        if (box) { box[4 * v] = b.x; box[4 * v + 1] = b.y; box[4 * v + 2] = b.z; box[4 * v + 3] = b.w; }
    }
}
}  // namespace uds

extern "C" int uds_tree_build(const uds_sample_params* prm, int view, const float* points,
                              const float* normals, const float* std_devs, const float* h_override,
                              uds_view_stats* stats, uint32_t* keys, int32_t* ids, int32_t* left,
                              int32_t* right, int32_t* parent, int32_t* count, int32_t* degree, float* centre,
                              float* box, void* workspace, size_t workspace_bytes, void* stream) {
    int st = check_params(prm);
    if (st) return st;
    if (view < 0 || view >= prm->B) return UDS_ERR_ARGUMENT;
    Ws w = layout(prm, reinterpret_cast<char*>(workspace));
    if (!workspace || workspace_bytes < w.bytes) return UDS_ERR_WORKSPACE;
    cudaStream_t s = as_stream(stream);
    if ((st = build_view(prm, w, view, points, normals, std_devs, h_override, s))) return st;
    if (prm->N > 0) {
        k_export<<<cdiv(2 * (size_t)prm->N, 128), 128, 0, s>>>(w.vs, w, keys, ids, left, right, parent, count,
                                                               degree, centre, box);
        if ((st = launch_status())) return st;
    }
    if (stats) {
        cudaError_t e = cudaMemcpyAsync(stats, w.stats + view, sizeof(uds_view_stats), cudaMemcpyDeviceToDevice, s);
        if (e != cudaSuccess) { set_last_error(e); return UDS_ERR_CUDA; }
    }
    return UDS_OK;
}

extern "C" int uds_sample_descent(const uds_sample_params* prm, int view, const float* uniforms,
                                  int32_t* indices, void* workspace, size_t workspace_bytes, void* stream) {
    int st = check_params(prm);
    if (st) return st;
    if (view < 0 || view >= prm->B || !indices) return UDS_ERR_ARGUMENT;
    Ws w = layout(prm, reinterpret_cast<char*>(workspace));
    if (!workspace || workspace_bytes < w.bytes + deferred_bytes(prm)) return UDS_ERR_WORKSPACE;
    if (prm->N == 0) return UDS_OK;
    cudaStream_t s = as_stream(stream);
    const Deferred df = deferred_of(prm, w, reinterpret_cast<char*>(workspace), workspace_bytes);
    return launch_descent(tree_of(w), w, prm, df, uniforms, view, indices, s);
}

extern "C" int uds_fgt_eval(const uds_sample_params* prm, int m, const int32_t* nodes, const float* query_xy,
                            float* out, const void* workspace, size_t workspace_bytes, void* stream) {
    int st = check_params(prm);
    if (st) return st;
    Ws w = layout(prm, reinterpret_cast<char*>(const_cast<void*>(workspace)));
    if (!workspace || workspace_bytes < w.bytes) return UDS_ERR_WORKSPACE;
    if (m <= 0) return UDS_OK;
    k_fgt_eval<<<cdiv(m, 128), 128, 0, as_stream(stream)>>>(tree_of(w), w.vs, m, nodes, query_xy, out);
    return launch_status();
}

extern "C" int uds_mlp_forward_tiles(int R_max, const int* R_dev, const void* X_tiles, const float* params,
                                     float* logits, int* err, void* stream);

namespace uds {
// Proposal-mode buffers after the tree slot.
struct PropWs {
    float* root_mass;
    unsigned char* mask;
    int* node[2];
    int* draw[2];
    float* logq[2];
    float* X;
    float* logits;
    int* counts;  // [0], [1]: list lengths; [2]: fallback pixels; [3]: network error flag
    size_t bytes;
};

static PropWs prop_layout(const uds_sample_params* p, char* base) {
    PropWs q{};
    size_t P = (size_t)p->W * p->H, D = P * (size_t)p->K;
    size_t off = 0;
    auto take = [&](size_t bytes) { size_t o = off; off += a256(bytes); return base ? base + o : nullptr; };
    q.root_mass = (float*)take(4 * P);
    q.mask = (unsigned char*)take(P);
    for (int c = 0; c < 2; ++c) {
        q.node[c] = (int*)take(4 * D);
        q.draw[c] = (int*)take(4 * D);
        q.logq[c] = (float*)take(4 * D);
    }
    // feature tiles: 128 rows of 16 bf16 per 4096 bytes
    q.X = (float*)take(cdiv(D > 0 ? D : 1, 128) * (size_t)4096);
    q.logits = (float*)take(8 * D);
    q.counts = (int*)take(16);
    q.bytes = off;
    return q;
}
}  // namespace uds

extern "C" size_t uds_proposal_workspace_size(const uds_sample_params* prm) {
    if (check_params(prm)) return 0;
    return layout(prm, nullptr).bytes + prop_layout(prm, nullptr).bytes + deferred_bytes(prm);
}

extern "C" int uds_sample_proposal(const uds_sample_params* prm, const float* points, const float* normals,
                                   const float* std_devs, const float* h_override, const float* mlp_params,
                                   float ess_tau, int32_t* indices, float* weights, uint8_t* fallback,
                                   int32_t* n_fallback, uds_view_stats* stats, void* workspace,
                                   size_t workspace_bytes, void* stream) {
    int st = check_params(prm);
    if (st) return st;
    if (!indices || !weights || (prm->N > 0 && (!points || !normals || !std_devs))) return UDS_ERR_ARGUMENT;
    if (prm->W * (size_t)prm->H * prm->K >= (1ull << 31)) return UDS_ERR_ARGUMENT;
    char* base = reinterpret_cast<char*>(workspace);
    Ws w = layout(prm, base);
    PropWs q = prop_layout(prm, base ? base + w.bytes : nullptr);
    if (!workspace || workspace_bytes < w.bytes + q.bytes + deferred_bytes(prm)) return UDS_ERR_WORKSPACE;
    cudaStream_t s = as_stream(stream);
    size_t P = (size_t)prm->W * prm->H, per_view = P * prm->K;
    cudaError_t e = cudaMemsetAsync(indices, 0xFF, sizeof(int32_t) * per_view * prm->B, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(weights, 0, sizeof(float) * per_view * prm->B, s);
    if (e == cudaSuccess && n_fallback) e = cudaMemsetAsync(n_fallback, 0, sizeof(int32_t) * prm->B, s);
    if (e != cudaSuccess) { set_last_error(e); return UDS_ERR_CUDA; }
    Tree T = tree_of(w);
    dim3 block(8, kDescentThreads / 8);
    dim3 grid(cdiv(prm->H, block.x), cdiv(prm->W, block.y));
    const Deferred df = deferred_of(prm, w, base, workspace_bytes);
    const unsigned more = long_blocks(prm);
    for (int b = 0; b < prm->B; ++b) {
        if ((st = build_view(prm, w, b, points, normals, std_devs, h_override, s))) return st;
        if (prm->N == 0) continue;
        int* idx = indices + per_view * b;
        float* wt = weights + per_view * b;
        const unsigned char* mask = nullptr;
        if (mlp_params) {
            e = cudaMemsetAsync(q.counts, 0, 16, s);
            if (e != cudaSuccess) { set_last_error(e); return UDS_ERR_CUDA; }
            const PropInit out{prm->K, prm->precision, q.root_mass, q.node[0], q.draw[0], q.logq[0], q.counts, idx, wt};
            k_prop_init<<<grid, block, 0, s>>>(T, w.vs, prm->W, prm->H, out, df);
            if (more) k_prop_init_long<<<more, dim3(8, 4), 0, s>>>(T, w.vs, prm->H, out, df);
            if ((st = launch_status(more ? 2 : 1))) return st;
            unsigned nb = cdiv(per_view, 256);
            int cur = 0;
            for (int level = 0; level < kTrace; ++level) {
                if (level % 8 == 7) {  // stop once every draw has reached its leaf
                    int left = 0;
                    e = cudaMemcpyAsync(&left, q.counts + cur, sizeof(int), cudaMemcpyDeviceToHost, s);
                    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
                    if (e != cudaSuccess) { set_last_error(e); return UDS_ERR_CUDA; }
                    if (left == 0) break;
                }
                k_prop_features<<<nb, 256, 0, s>>>(T, w.vs, prm->H, prm->K, level, q.counts + cur, q.node[cur],
                                                   q.draw[cur], reinterpret_cast<unsigned char*>(q.X));
                if ((st = launch_status())) return st;
                if ((st = uds_mlp_forward_tiles((int)per_view, q.counts + cur, q.X, mlp_params, q.logits,
                                                q.counts + 3, stream)))
                    return st;
                e = cudaMemsetAsync(q.counts + (cur ^ 1), 0, 4, s);
                if (e != cudaSuccess) { set_last_error(e); return UDS_ERR_CUDA; }
                k_prop_step<<<nb, 256, 0, s>>>(T, w.vs, prm->H, prm->K, level, prm->seed, prm->seed_dev, (uint32_t)b,
                                               q.counts + cur, q.node[cur], q.draw[cur], q.logq[cur], q.logits,
                                               q.root_mass, q.counts + (cur ^ 1), q.node[cur ^ 1], q.draw[cur ^ 1],
                                               q.logq[cur ^ 1], idx, wt);
                if ((st = launch_status())) return st;
                cur ^= 1;
            }
            k_prop_ess<<<cdiv(P, 256), 256, 0, s>>>(prm->W, prm->H, prm->K, ess_tau, q.root_mass, prm->precision, wt,
                                                     q.mask, n_fallback ? n_fallback + b : q.counts + 2);
            if ((st = launch_status())) return st;
            // fallback pixels: clear the proposal's draws, then the plain sampler
            k_prop_clear<<<cdiv(P, 256), 256, 0, s>>>(P, prm->K, q.mask, idx, wt);
            if ((st = launch_status())) return st;
            mask = q.mask;
            if (fallback) {
                e = cudaMemcpyAsync(fallback + P * b, q.mask, P, cudaMemcpyDeviceToDevice, s);
                if (e != cudaSuccess) { set_last_error(e); return UDS_ERR_CUDA; }
            }
        }
        // the plain stochastic sampler: every pixel, or the fallback pixels
        float* probs = q.logits;  // scratch for the path probabilities
        if ((st = launch_stochastic(w, prm, df, b, idx, probs, mask, wt, s))) return st;
    }
    if (stats) {
        e = cudaMemcpyAsync(stats, w.stats, sizeof(uds_view_stats) * prm->B, cudaMemcpyDeviceToDevice, s);
        if (e != cudaSuccess) { set_last_error(e); return UDS_ERR_CUDA; }
    }
    return UDS_OK;
}

extern "C" int uds_proposal_dataset(const uds_sample_params* prm, int stride, int draws, float* X, float* target,
                                    int64_t* keys, int32_t* count, int cap, const void* workspace,
                                    size_t workspace_bytes, void* stream) {
    int st = check_params(prm);
    if (st) return st;
    if (stride < 1 || draws < 1 || draws > 255 || cap < 0 || !count || (cap > 0 && (!X || !target)))
        return UDS_ERR_ARGUMENT;
    Ws w = layout(prm, reinterpret_cast<char*>(const_cast<void*>(workspace)));
    if (!workspace || workspace_bytes < w.bytes) return UDS_ERR_WORKSPACE;
    if (prm->N == 0) return UDS_OK;
    dim3 block(16, 8);
    dim3 grid(cdiv(cdiv(prm->H, stride), block.x), cdiv(cdiv(prm->W, stride), block.y));
    k_prop_dataset<<<grid, block, 0, as_stream(stream)>>>(tree_of(w), w.vs, prm->W, prm->H, stride, draws,
                                                          prm->precision, prm->seed, 0u, X, target,
                                                          reinterpret_cast<long long*>(keys), count, cap);
    return launch_status();
}
