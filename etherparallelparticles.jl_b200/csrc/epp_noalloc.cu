// epp_noalloc.cu -- cell-list build for callers that cannot allocate device memory.
//
// Some hosts of this library may not call cudaMalloc while they drive a simulation: a host
// application whose device memory comes from its own fixed pool, or a caller in the middle of a
// step where a device allocation would synchronise the device or is simply not permitted.  For
// them epp_cell_sort_noalloc builds the cell list of the context's search! (bin into slots, scan,
// scatter, rank by id) on device buffers the caller passes in, with every intermediate array in one
// statically sized device array declared below.  That array is part of the library:
// every GPU that loads libepp.so holds it until the process exits.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstring>
#include <mutex>

#include "epp_cells.cuh"

using namespace epp;

namespace {

constexpr int kNaMaxParticles = 1 << 20;   // largest n accepted
constexpr int kNaMaxCells = 1 << 20;       // largest domain (cells) accepted
constexpr int kNaTiles = (kNaMaxCells + 1 + kScanTile - 1) / kScanTile;

// Layout of the scratch (bytes, each part 256-aligned):
//   counts   int   [kNaMaxCells + 2]
//   tile     int   [2 * kNaTiles * 32]   particles per scan tile, a line apart (and the spare the scan resets)
//   cs       int2  [kNaMaxParticles]     (cell, slot) per particle
//   perm     int2  [kNaMaxParticles]     (id, particle) in arrival order
//   start    int   [kNaMaxCells + 2]     offsets before they are copied out
//   meta     int   [64]                  n_alive, status word
constexpr int kTileStride = 32;
constexpr size_t align256(size_t b) { return (b + 255) & ~size_t(255); }
constexpr size_t kOffCounts = 0;
constexpr size_t kOffTile = kOffCounts + align256(sizeof(int) * (kNaMaxCells + 2));
constexpr size_t kOffCs = kOffTile + align256(sizeof(int) * 2 * kNaTiles * kTileStride);
constexpr size_t kOffPerm = kOffCs + align256(sizeof(int2) * kNaMaxParticles);
constexpr size_t kOffStart = kOffPerm + align256(sizeof(int2) * kNaMaxParticles);
constexpr size_t kOffMeta = kOffStart + align256(sizeof(int) * (kNaMaxCells + 2));
constexpr size_t kScratchBytes = kOffMeta + align256(sizeof(int) * 64);

static __device__ __align__(256) unsigned char g_noalloc_scratch[kScratchBytes];

constexpr int kMaxDevices = 64;
// Device address of the scratch, per device, looked up on the first call on that device.  The
// look-up is guarded, so first calls from several host threads at once are safe (the calls
// themselves still share the scratch and must not overlap on the GPU).
std::atomic<unsigned char*> g_scratch_addr[kMaxDevices];
std::mutex g_scratch_mu;

// Clears what a call starts from: counts, tile counters, the status word.
__global__ void k_na_clear(int n_cells, int tiles, int* count, int* tile, int* meta) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c <= n_cells) count[c] = 0;
    if (c < tiles) tile[c * kTileStride] = 0;
    if (c < 2) meta[c] = 0;
}

// Bin particle i (positions column-major: x at pos[i], y at pos[n + i], z at pos[2n + i]); outside
// the domain -> dead bin (n_cells), as NeighbourSearch.jl:41-43 kills it.  A block counts its particles of
// each scan tile before it adds them to tile[]: particles in no order meet every tile, and the atomics
// of a counter are served one after the other (1,000,000 particles at random in 14 tiles: 134 us the call
// with an atomic a warp and tile, 73 so).
constexpr int kNaBinThreads = 512;
template <int D>
__global__ void __launch_bounds__(kNaBinThreads) k_na_bin(int n, DevDomain dom, const float* pos, int tiles, int2* cs, int* count,
                                                          int* tile) {
    __shared__ int s_tile[kNaTiles];
    for (int t = threadIdx.x; t < tiles; t += kNaBinThreads) s_tile[t] = 0;
    __syncthreads();
    const int i = blockIdx.x * kNaBinThreads + threadIdx.x;
    if (i < n) {
        const float4 x = make_float4(pos[i], pos[(size_t)n + i], D == 3 ? pos[(size_t)2 * n + i] : 0.0f, 0.0f);
        int c = cell_of<D>(dom, x, 0);
        if (c < 0) c = dom.n_cells;
        cs[i] = make_int2(c, atomicAdd(&count[c], 1));
        const int t = c / kScanTile;
        const unsigned same = __match_any_sync(__activemask(), t);
        if ((threadIdx.x & 31) == __ffs(same) - 1) atomicAdd(&s_tile[t], __popc(same));
    }
    __syncthreads();
    for (int t = threadIdx.x; t < tiles; t += kNaBinThreads)
        if (s_tile[t]) atomicAdd(&tile[t * kTileStride], s_tile[t]);
}

// A cell's particles side by side, in arrival order.
__global__ void k_na_scatter(int n, const int2* cs, const int* start, int2* perm, int* meta) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) scatter_particle(i, n, cs[i], start, i, perm, reinterpret_cast<unsigned*>(meta + 1));
}

// Rank inside the cell by particle id: the 1-based id to its sorted position (a position outside
// 0..n-1 is skipped and reported, EPP_STATUS_QUEUE); the same grid copies the counts and offsets out
// and leaves the number of particles inside the domain beside the status word.
__global__ void k_na_rank(int n, int n_cells, const int2* perm, const int2* cs, const int* start,
                          int* sorted_ids, int* counts, int* offsets, int* meta) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p <= n_cells) {
        const int s = start[p];
        if (counts && p < n_cells) counts[p] = start[p + 1] - s;
        if (offsets) offsets[p] = s;
        if (p == n_cells) meta[0] = s;
    }
    if (p >= n) return;
    unsigned* status = reinterpret_cast<unsigned*>(meta + 1);
    const int2 e = perm[p];
    if (e.y < 0 || e.y >= n) {
        atomicOr(status, EPP_STATUS_QUEUE);
        return;
    }
    const int c = cs[e.y].x;
    if (c >= n_cells) return;   // dead particles are not part of the cell list
    const int dst = sorted_place_perm(p, e, c, n, n_cells, perm, start);
    if (dst < 0 || dst >= n) {
        atomicOr(status, EPP_STATUS_QUEUE);
        return;
    }
    sorted_ids[dst] = e.x + 1;
}

}  // namespace

extern "C" {

int32_t epp_noalloc_limits(int32_t* max_particles, int32_t* max_cells, int64_t* scratch_bytes) {
    if (max_particles) *max_particles = kNaMaxParticles;
    if (max_cells) *max_cells = kNaMaxCells;
    if (scratch_bytes) *scratch_bytes = (int64_t)kScratchBytes;
    return EPP_OK;
}

int32_t epp_cell_sort_noalloc(const epp_domain* domain, int32_t n, const float* pos, int32_t* counts,
                              int32_t* offsets, int32_t* sorted_ids, int32_t* n_alive, void* stream) {
    if (!domain || n < 0 || (n > 0 && !pos) || !sorted_ids || !n_alive) return EPP_ERR_INVALID_ARGUMENT;
    if (n > kNaMaxParticles) return EPP_ERR_CAPACITY;
    DevDomain dom;
    std::memset(&dom, 0, sizeof dom);
    if (const int rc = plan_domain(*domain, 1, kNaMaxCells, dom)) return rc;   // the context's cell grid
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return EPP_ERR_CUDA;
    // set-up, once per device, with that device current: the scratch's device address
    unsigned char* base = g_scratch_addr[dev].load(std::memory_order_acquire);
    if (!base) {
        std::lock_guard<std::mutex> lock(g_scratch_mu);
        base = g_scratch_addr[dev].load(std::memory_order_acquire);
        if (!base) {
            void* p = nullptr;
            if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || !p) return EPP_ERR_CUDA;
            base = static_cast<unsigned char*>(p);
            g_scratch_addr[dev].store(base, std::memory_order_release);
        }
    }
    int* tile = reinterpret_cast<int*>(base + kOffTile);
    int* start = reinterpret_cast<int*>(base + kOffStart);
    int* meta = reinterpret_cast<int*>(base + kOffMeta);
    int2* perm = reinterpret_cast<int2*>(base + kOffPerm);
    int2* cs = reinterpret_cast<int2*>(base + kOffCs);
    int* count = reinterpret_cast<int*>(base + kOffCounts);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int nc = dom.n_cells;
    const int tiles = (nc + 1 + kScanTile - 1) / kScanTile;
    // The scratch keeps the last call's contents: what must start clear goes in one kernel, and the two
    // words the host reads come back in one copy -- five launches and a copy in all.  A cell's particles
    // are ranked side by side rather than from a linked list: the caller's particles may come in any order
    // and crowd any cell, and a list is one dependent load after another (1,000,000 particles at random
    // places, us: 9 to a cell 73, 131 from lists; 125 to a cell 97, 572; 955,668 on a lattice 54, 60).
    const int T = 128;
    auto grid = [&](int k) { return (k + T - 1) / T; };
    k_na_clear<<<grid(nc + 1), T, 0, s>>>(nc, tiles, count, tile, meta);
    if (n > 0) {
        const int gb = (n + kNaBinThreads - 1) / kNaBinThreads;
        if (domain->dim == 2) k_na_bin<2><<<gb, kNaBinThreads, 0, s>>>(n, dom, pos, tiles, cs, count, tile);
        else k_na_bin<3><<<gb, kNaBinThreads, 0, s>>>(n, dom, pos, tiles, cs, count, tile);
    }
    // (the scan resets the spare tile counters)
    k_scan_tiles<false><<<tiles, kScanThreads, 0, s>>>(nc + 1, count, tile, start, ScanReset{tile + kNaTiles * kTileStride, kTileStride},
                                                      0, reinterpret_cast<unsigned*>(meta + 1));
    if (n > 0) k_na_scatter<<<grid(n), T, 0, s>>>(n, cs, start, perm, meta);
    k_na_rank<<<grid(std::max(n, nc + 1)), T, 0, s>>>(n, nc, perm, cs, start, sorted_ids, counts, offsets, meta);
    if (cudaGetLastError() != cudaSuccess) return EPP_ERR_CUDA;
    int back[2] = {0, 0};   // particles inside the domain, status
    if (cudaMemcpyAsync(back, meta, sizeof back, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess)
        return EPP_ERR_CUDA;
    *n_alive = back[0];
    const unsigned st = (unsigned)back[1];
    return st ? EPP_ERR_DEVICE_STATUS : EPP_OK;
}

}  // extern "C"
