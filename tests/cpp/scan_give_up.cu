// A wait of one of the binning's scans that runs out: its ticket starts at 1,
// so no CTA takes tile 0 and the tiles after it wait for a sum that never comes
// (a bounded wait, a second or so).  The binning has to report it, write
// nothing outside its arrays and leave its working words as it found them, and
// the next binning has to be right.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <numeric>
#include <vector>

#include "gmpm.h"
#include "kernels.h"

using namespace gmpm;

#define CHECK(cond)                                                    \
    do {                                                               \
        if (!(cond)) {                                                 \
            std::printf("line %d: %s\n", __LINE__, #cond);             \
            return 1;                                                  \
        }                                                              \
    } while (0)

template <typename T>
static T* device(size_t count, int byte) {
    void* p = nullptr;
    if (cudaMalloc(&p, count * sizeof(T)) != cudaSuccess) return nullptr;
    cudaMemset(p, byte, count * sizeof(T));
    return static_cast<T*>(p);
}
template <typename T>
static std::vector<T> host(const T* p, size_t count) {
    std::vector<T> v(count);
    cudaMemcpy(v.data(), p, count * sizeof(T), cudaMemcpyDeviceToHost);
    return v;
}

int main() {
    const int64_t n = 10000;
    const uint32_t key_space = 32768;  // 8 tiles of the page scans
    const int nb_cap = 512, ng_cap = 4096;
    const int64_t ncell = (int64_t)nb_cap * 64;  // 8 tiles of the cell scan
    // more than half of the particles in one cell (no more than the canonical pass ranks), the others over 200
    // pages with room for their neighbours
    std::vector<uint32_t> keys(n);
    uint32_t seed = 1;
    for (int64_t i = 0; i < n; ++i) {
        seed = seed * 1664525u + 1013904223u;
        const int page = (int)(seed >> 16) % 200;
        keys[i] = i % 5 < 3 ? (page_key(3, 4, 5) << 6) | 17u
                            : (page_key(6 + page % 10, 6 + page / 10 % 5, 6 + page / 50) << 6) | ((seed >> 8) & 63u);
    }
    std::vector<int32_t> want(n);
    std::iota(want.begin(), want.end(), 0);
    std::stable_sort(want.begin(), want.end(), [&](int a, int b) { return keys[a] < keys[b]; });

    BinDev bin{};
    bin.n = n;
    bin.key_space = key_space;
    bin.nb_cap = nb_cap;
    bin.ng_cap = ng_cap;
    bin.keys = device<uint32_t>(n, 0);
    bin.keys_sorted = device<uint32_t>(3 * n, 0x5a);  // n of them, and a guard
    bin.perm = device<int32_t>(3 * n, 0x5a);
    bin.page_flag = device<uint8_t>(key_space, 0);
    bin.page_rank = device<int32_t>(key_space, 0);
    bin.grid_flag = device<uint8_t>(key_space, 0);
    bin.grid_rank = device<int32_t>(key_space, 0);
    bin.block_keys = device<uint32_t>(nb_cap, 0);
    bin.cell_count = device<int32_t>(ncell, 0);
    bin.cell_start = device<int32_t>(ncell + 1, 0);
    bin.grid_keys = device<uint32_t>(ng_cap, 0);
    bin.adj = device<int32_t>((size_t)nb_cap * 8, 0);
    bin.grid_src = device<int32_t>((size_t)ng_cap * 8, 0);
    const int64_t words = scan_scratch_words(key_space, ncell);
    const ScanScratch scan = scan_scratch(device<uint32_t>(words, 0), key_space, ncell);
    Counters* cnt = device<Counters>(1, 0);
    cudaMemcpy(bin.keys, keys.data(), n * 4, cudaMemcpyHostToDevice);
    std::vector<uint8_t> flags(key_space, 0);
    for (uint32_t k : keys) flags[k >> 6] = 1;
    const int pages = (int)std::count(flags.begin(), flags.end(), 1);
    CHECK(pages > 64);  // cells of more than one tile

    // which scan gives up: none, the pages', the grid pages', the cells'; a whole binning after each
    const int32_t ticket[4] = {-1, (int32_t)scan_tiles(key_space), scan.grid + (int32_t)scan_tiles(key_space),
                               scan.cells + (int32_t)scan_tiles(ncell)};
    for (int q : {0, 1, 0, 2, 0, 3, 0}) {
        cudaMemset(cnt, 0, sizeof(Counters));
        cudaMemset(bin.perm, 0x5a, 3 * n * 4);
        cudaMemset(bin.keys_sorted, 0x5a, 3 * n * 4);
        cudaMemcpy(bin.page_flag, flags.data(), key_space, cudaMemcpyHostToDevice);  // as a G2P leaves them
        const uint32_t one = 1;
        if (q) cudaMemcpy(scan.words + ticket[q], &one, 4, cudaMemcpyHostToDevice);
        CHECK(launch_binning<float>(nullptr, PState<float>{}, bin, scan, cnt, 148, 0, true) == cudaSuccess);
        CHECK(cudaDeviceSynchronize() == cudaSuccess);
        const Counters c = host(cnt, 1)[0];
        const auto perm = host(bin.perm, 3 * n);
        const auto sorted = host(bin.keys_sorted, 3 * n);
        for (int64_t i = n; i < 3 * n; ++i) CHECK(perm[i] == 0x5a5a5a5a && sorted[i] == 0x5a5a5a5au);
        for (uint32_t w : host(scan.words, words)) CHECK(w == 0);
        for (int32_t w : host(bin.cell_count, ncell)) CHECK(w == 0);
        for (uint8_t w : host(bin.page_flag, key_space)) CHECK(w == 0);
        for (uint8_t w : host(bin.grid_flag, key_space)) CHECK(w == 0);
        if (q) {
            CHECK(c.flags == GMPM_FLAG_COPY_TIMEOUT && c.n_blocks == 0 && c.n_grid_blocks == 0);
        } else {
            CHECK(c.flags == 0 && c.n_blocks == pages && c.n_grid_blocks > pages);
            for (int64_t i = 0; i < n; ++i) CHECK(perm[i] == want[i] && sorted[i] == keys[want[i]]);
        }
    }
    std::printf("ok\n");
    return 0;
}
