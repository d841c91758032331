// CPU build of the merge sort of the sorted unique (tile sort, merge rounds) under the SIMT emulation of simt_emu.h, from
// the kernel source the GPU library is built from.
#include "simt_emu.h"
#include "../../recsdk_b200/csrc/prims.cuh"

using namespace recsdk;

template <typename F>
static void run_grid(int64_t grid, int block, F kernel)
{
    blockDim.x = static_cast<unsigned>(block);
    gridDim.x = static_cast<unsigned>(grid);
    for (int64_t b = 0; b < grid; ++b) {
        std::vector<std::thread> ts;
        for (int t = 0; t < block; ++t)
            ts.emplace_back([&kernel, b, t] {
                threadIdx.x = static_cast<unsigned>(t);
                blockIdx.x = static_cast<unsigned>(b);
                kernel();
            });
        for (auto& t : ts) t.join();
    }
}

// Positions in sorted order.  They start as UINT32_MAX in both buffers: a place no pair is written to shows.
template <typename KeyT>
static void sort_ids(const int64_t* ids, int64_t n, int key_bits, uint32_t* order)
{
    const int sort_bits = radix_sorted_bits<KeyT>(key_bits);
    const KeyT mask = merge_key_mask<KeyT>(sort_bits);
    std::vector<KeyT> keys[2] = {std::vector<KeyT>(n), std::vector<KeyT>(n)};
    std::vector<uint32_t> vals[2] = {std::vector<uint32_t>(n, UINT32_MAX), std::vector<uint32_t>(n, UINT32_MAX)};
    run_grid(ceil_div(n, kMergeTile), kMergeThreads,
             [&] { merge_tile_kernel<KeyT>(ids, n, sort_bits, keys[0].data(), vals[0].data()); });
    int cur = 0;
    for (int64_t run = kMergeTile; run < n; run *= 4, cur ^= 1)
        run_grid(ceil_div(n, 256), 256, [&] {
            merge_round_kernel<KeyT>(keys[cur].data(), vals[cur].data(), n, run, mask, keys[cur ^ 1].data(), vals[cur ^ 1].data());
        });
    std::copy(vals[cur].begin(), vals[cur].end(), order);
}

extern "C" void emu_merge_sort(const int64_t* ids, int64_t n, int key_bits, uint32_t* order)
{
    if (key_bits <= 32) sort_ids<uint32_t>(ids, n, key_bits, order);
    else sort_ids<uint64_t>(ids, n, key_bits, order);
}

extern "C" int emu_merge_sort_pays(int64_t n, int key_bits) { return merge_sort_pays(n, key_bits) ? 1 : 0; }
