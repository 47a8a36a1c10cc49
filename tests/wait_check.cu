// Waits between blocks that run out, with a short limit: the words of a tile
// that no block publishes stay 0, so the block behind it gives up and reports
// it.  Compiled by tests/test_gpu_waits.py.
#define UDS_WAIT_LOOKS 2000
#include "../unbiased_differentiable_splatting_gb300/csrc/uds_pixel.cu"

namespace uds {
void set_last_error(cudaError_t) {}
int launch_status(int) { return cudaGetLastError() == cudaSuccess ? UDS_OK : UDS_ERR_LAUNCH; }
}  // namespace uds

namespace {
__global__ void k_look_back(unsigned long long* status, int tile, int* failed, unsigned* bad) {
    unsigned long long before = 0;
    const bool ok = uds::look_back(status, tile, 7, before);
    if (threadIdx.x == 0 && !ok) uds::wait_failed(failed);
    if (!ok) atomicAdd(bad, 1u);
}
__global__ void k_flag(const int* failed, int* seen) { seen[threadIdx.x] = uds::failed_yet(failed); }
}  // namespace

extern "C" {
// tile 3 of a scan in which tile `missing` (< 3) publishes nothing; words of the others given
int check_look_back(unsigned long long* status, int* failed, unsigned* bad, void* stream) {
    k_look_back<<<1, 32, 0, uds::as_stream(stream)>>>(status, 3, failed, bad);
    return uds::launch_status(1);
}
int check_flag(const int* failed, int* seen, void* stream) {
    k_flag<<<1, 256, 0, uds::as_stream(stream)>>>(failed, seen);
    return uds::launch_status(1);
}
// One sorting pass over n pairs (zeroed state, words and counts but for `first`
// as the number of tiles started already), then the sums
int check_gather(int n, unsigned first, int failed, unsigned* hist, unsigned* words, const unsigned* keys,
                 const unsigned* samples, unsigned* keys_out, unsigned* samples_out, uint2* bounds, int M, int C,
                 const float* values, float* out, uds::GatherState* gs, void* stream) {
    cudaStream_t s = uds::as_stream(stream);
    uds::GatherState state{};
    state.n = (unsigned)n;
    state.ticket[0] = first;
    state.failed = failed;
    if (cudaMemcpyAsync(gs, &state, sizeof(state), cudaMemcpyHostToDevice, s) != cudaSuccess) return UDS_ERR_CUDA;
    const unsigned tiles = uds::cdiv(n, uds::kSortTile) - first;
    uds::k_pixel_sort<unsigned><<<tiles, uds::kTileThreads, 0, s>>>(0, gs, hist, words, keys, samples, keys_out,
                                                                    samples_out);
    uds::k_pixel_bounds<<<4, 256, 0, s>>>(gs, keys_out, bounds);
    uds::k_pixel_sum<<<uds::cdiv(M, 128), 128, 0, s>>>(gs, M, C, bounds, samples_out, values, out);
    return uds::launch_status(3);
}
int check_failures(unsigned* count) { return uds::pixel_wait_failures(count) == cudaSuccess ? UDS_OK : UDS_ERR_CUDA; }
}
