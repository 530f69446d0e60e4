// The tile sort by itself, for tests/test_tile_sort_flag_gpu.py.
#include "binning.cuh"

static bool g_attr[128];

extern "C" __attribute__((visibility("default"))) int tile_sort(
    int64_t tiles, int64_t n_elems, const int* tile_start, long long* header, unsigned long long* keys,
    const int* slot_inst, int* sorted_gid, int* sorted_inst, const int* count, const int* cursor) {
    cudaError_t e = us3d::launch_tile_sort(tiles, n_elems, tile_start, header, keys, slot_inst, sorted_gid, sorted_inst,
                                           g_attr, nullptr, nullptr, nullptr, count, cursor);
    return (int)(e != cudaSuccess ? e : cudaDeviceSynchronize());
}
