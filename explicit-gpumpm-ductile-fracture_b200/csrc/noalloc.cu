// Binning of caller-owned device positions with no device allocation.
//
// Some callers cannot allocate device memory on the call path: a host
// framework that owns and budgets every byte of device memory up front (an
// engine or a coupled solver that hands this library only views of its own
// buffers), or a latency-critical loop where cudaMalloc's implicit
// synchronisation and unpredictable cost are not allowed.  This entry point
// serves them: inputs and outputs are the caller's device buffers and all
// scratch lives in one file-scope __device__ array of fixed size, resolved once
// per device with cudaGetSymbolAddress.
//
// The array is shared by every call in the process: calls that overlap on the
// GPU (different streams, or host threads without ordering) race on it and
// must be serialised by the caller.  Its contents persist between calls, so
// everything that must start at zero is cleared on the call's stream first.
// The work is enqueued on the caller's stream, which must belong to the
// current device (the array resolved is the current device's).
#include <algorithm>
#include <cstdint>
#include <cstring>
#include <mutex>

#include "kernels.h"
#include "launch.cuh"
#include "scan.cuh"

namespace gmpm {

// Limits (also stated in include/gmpm.h).
constexpr int64_t kNoAllocMaxParticles = int64_t(1) << 20;   // 1,048,576
constexpr int kNoAllocMaxRes = 128;                          // nodes per axis -> page coordinates < 32
constexpr int kNoAllocKeyBits = 5;                           // bits per axis of the page key
constexpr uint32_t kNoAllocKeySpace = 1u << (3 * kNoAllocKeyBits);  // 32,768 pages: every page of the grid
constexpr int64_t kNoAllocCells = (int64_t)kNoAllocKeySpace * 64;

// Scratch layout (bytes, each region 256-byte aligned).
constexpr size_t align256(size_t v) { return (v + 255) / 256 * 256; }
constexpr size_t kOffCounters = 0;
constexpr size_t kOffKeys = align256(kOffCounters + sizeof(Counters));
constexpr size_t kOffPageFlag = align256(kOffKeys + kNoAllocMaxParticles * sizeof(uint32_t));
constexpr size_t kOffPageRank = align256(kOffPageFlag + kNoAllocKeySpace);
constexpr size_t kOffBlockKeys = align256(kOffPageRank + kNoAllocKeySpace * sizeof(int32_t));
constexpr size_t kOffCellCount = align256(kOffBlockKeys + kNoAllocKeySpace * sizeof(uint32_t));
constexpr size_t kOffCellStart = align256(kOffCellCount + kNoAllocCells * sizeof(int32_t));
constexpr size_t kOffScanTiles = align256(kOffCellStart + (kNoAllocCells + 1) * sizeof(int32_t));
// status words of the page scan, an unused grid scan and the cell scan, with their tickets; the failure word
constexpr size_t kScanWords =
    2 * ((kNoAllocKeySpace + kScanTile - 1) / kScanTile + 1) + (kNoAllocCells + kScanTile - 1) / kScanTile + 1 + 1;
constexpr size_t kNoAllocScratchBytes = align256(kOffScanTiles + kScanWords * sizeof(uint32_t));
static_assert(kNoAllocScratchBytes == GMPM_NOALLOC_SCRATCH_BYTES, "keep include/gmpm.h in step");

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

// Page/cell keys of interleaved xyz positions: the scene binning's cell_key
// (common.cuh; cal_cellId, Particle_kernal.cu:158-165).
__global__ void k_noalloc_keys(int64_t n, const float* __restrict__ pos, double inv_dx, int rx, int ry, int rz,
                               uint32_t* __restrict__ keys, uint8_t* __restrict__ page_flag, Counters* cnt) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int res[3] = {rx, ry, rz};
    const float x[3] = {pos[3 * i], pos[3 * i + 1], pos[3 * i + 2]};
    bool bad = false;
    const uint32_t key = cell_key(x, inv_dx, res, bad);
    if (bad) raise_flag(cnt, GMPM_FLAG_OUT_OF_DOMAIN);
    keys[i] = key;
    page_flag[key >> 6] = 1;
}

// The same for many positions.  They come in any order, so their flag stores
// would meet on the few active pages' bytes (94 us at 1M positions): a CTA
// collects its pages in shared memory and adds them once, four flags a word.
constexpr int kManyThreads = 1024;
constexpr int64_t kMany = 1 << 16;  // below, clearing and scanning the CTA's flags costs more than it saves
__global__ void __launch_bounds__(kManyThreads)
    k_noalloc_keys_many(int64_t n, const float* __restrict__ pos, double inv_dx, int rx, int ry, int rz,
                        uint32_t* __restrict__ keys, uint8_t* __restrict__ page_flag, Counters* cnt) {
    __shared__ uint32_t seen[kNoAllocKeySpace / 4];
    for (int w = threadIdx.x; w < (int)(kNoAllocKeySpace / 4); w += kManyThreads) seen[w] = 0u;
    __syncthreads();
    const int res[3] = {rx, ry, rz};
    constexpr int kILP = 4;
    const int64_t step = (int64_t)gridDim.x * kManyThreads;
    bool bad = false;
    for (int64_t i0 = (int64_t)blockIdx.x * kManyThreads + threadIdx.x; i0 < n; i0 += kILP * step) {
        float x[kILP][3];
#pragma unroll
        for (int u = 0; u < kILP; ++u)
#pragma unroll
            for (int a = 0; a < 3; ++a) x[u][a] = i0 + u * step < n ? pos[3 * (i0 + u * step) + a] : 0.f;
#pragma unroll
        for (int u = 0; u < kILP; ++u) {
            if (i0 + u * step >= n) continue;
            const uint32_t key = cell_key(x[u], inv_dx, res, bad);
            keys[i0 + u * step] = key;
            reinterpret_cast<uint8_t*>(seen)[key >> 6] = 1;
        }
    }
    if (bad) raise_flag(cnt, GMPM_FLAG_OUT_OF_DOMAIN);
    __syncthreads();
    for (int w = threadIdx.x; w < (int)(kNoAllocKeySpace / 4); w += kManyThreads)
        if (seen[w]) atomicOr(reinterpret_cast<uint32_t*>(page_flag) + w, seen[w]);
}

namespace {

// Device address of g_noalloc_scratch per device, resolved on first use.
constexpr int kMaxDevices = 64;
unsigned char* g_scratch_ptr[kMaxDevices] = {nullptr};
std::mutex g_scratch_mutex;

cudaError_t scratch_for_current_device(unsigned char** out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(g_scratch_mutex);
    if (!g_scratch_ptr[dev]) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess) return e;
        g_scratch_ptr[dev] = reinterpret_cast<unsigned char*>(p);
    }
    *out = g_scratch_ptr[dev];
    return cudaSuccess;
}

}  // namespace
}  // namespace gmpm

extern "C" gmpm_status gmpm_bin_positions_noalloc(const float* positions, int64_t n, double dx, int res_x, int res_y,
                                                  int res_z, int32_t* perm, uint32_t* keys_sorted, uint32_t* flags,
                                                  void* stream) {
    using namespace gmpm;
    if (!positions || !perm || !keys_sorted || n <= 0 || !(dx > 0)) return GMPM_INVALID_ARG;
    if (n > kNoAllocMaxParticles) return GMPM_INVALID_ARG;
    const int res[3] = {res_x, res_y, res_z};
    for (int a = 0; a < 3; ++a)
        if (res[a] < 8 || res[a] > kNoAllocMaxRes) return GMPM_INVALID_ARG;
    unsigned char* base = nullptr;
    if (scratch_for_current_device(&base) != cudaSuccess) return GMPM_CUDA_ERROR;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    Counters* cnt = reinterpret_cast<Counters*>(base + kOffCounters);
    // n particles occupy at most n pages, so page ranks stay below min(n, key space):
    // only that many pages' cells are cleared and scanned
    const int32_t nb_cap = (int32_t)std::min<int64_t>(n, (int64_t)kNoAllocKeySpace);
    const int64_t ncell = (int64_t)nb_cap * 64;
    BinDev bin{};
    bin.n = n;
    bin.key_space = kNoAllocKeySpace;
    bin.nb_cap = nb_cap;
    bin.ng_cap = 0;
    bin.keys = reinterpret_cast<uint32_t*>(base + kOffKeys);
    bin.keys_sorted = keys_sorted;
    bin.perm = perm;
    bin.page_flag = base + kOffPageFlag;
    bin.page_rank = reinterpret_cast<int32_t*>(base + kOffPageRank);
    bin.block_keys = reinterpret_cast<uint32_t*>(base + kOffBlockKeys);
    bin.cell_count = reinterpret_cast<int32_t*>(base + kOffCellCount);
    bin.cell_start = reinterpret_cast<int32_t*>(base + kOffCellStart);
    const ScanScratch scan = scan_scratch(reinterpret_cast<uint32_t*>(base + kOffScanTiles), kNoAllocKeySpace, ncell);
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);

    // state left by the previous call: clear what must start at zero
    if (e == cudaSuccess) e = cudaMemsetAsync(cnt, 0, sizeof(Counters), s);
    if (e == cudaSuccess) e = cudaMemsetAsync(bin.page_flag, 0, kNoAllocKeySpace, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(bin.cell_count, 0, ncell * sizeof(int32_t), s);
    if (e == cudaSuccess) e = cudaMemsetAsync(scan.words, 0, scan.count * sizeof(uint32_t), s);
    const int T = 256;
    const unsigned gn = (unsigned)((n + T - 1) / T);
    if (e == cudaSuccess && n >= kMany)
        e = launch_kernel(k_noalloc_keys_many, dim3((unsigned)sms), dim3(kManyThreads), 0, s, n, positions, 1.0 / dx, res_x,
                          res_y, res_z, bin.keys, bin.page_flag, cnt);
    else if (e == cudaSuccess)
        e = launch_kernel(k_noalloc_keys, dim3(gn), dim3(T), 0, s, n, positions, 1.0 / dx, res_x, res_y, res_z,
                          bin.keys, bin.page_flag, cnt);
    if (e == cudaSuccess) e = launch_bin_no_grid(bin, scan, cnt, sms, s);
    if (e == cudaSuccess && flags)
        e = cudaMemcpyAsync(flags, &cnt->flags, sizeof(uint32_t), cudaMemcpyDeviceToDevice, s);
    if (e != cudaSuccess) return e == cudaErrorMemoryAllocation ? GMPM_OOM : GMPM_CUDA_ERROR;
    return GMPM_OK;
}
