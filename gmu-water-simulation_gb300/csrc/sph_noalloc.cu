// sph_noalloc.cu -- a grid build that allocates no device memory.
//
// For callers that must not allocate once they are running: a host application that has
// already handed its GPU memory to its own pool allocator, or a per-frame callback in a
// real-time loop, where cudaMalloc/cudaFree would synchronise the device and stall the frame.
// The caller passes device arrays for the positions and for every output; the kernels'
// working memory (per-cell counts, per-particle slot ids, per-group counts, the list
// of crowded cells) lives in one file-scope device array of fixed size. The array belongs to
// the library's device code: CUDA creates it on a device when that code is loaded there, which
// under lazy module loading (the default) is the first call on that device. That first call
// also looks up the array's device address, so it belongs in the caller's setup: before its
// pool allocator takes the GPU's memory and before any stream capture. Every GPU that has run
// a call holds the array until the process exits. cudaDeviceReset is not supported between
// calls: the address looked up by the first call would then be stale.
//
// Limits: at most kMaxParticles particles and kMaxCells grid cells per call (about 8 MiB of
// scratch). Calls share the scratch array, which keeps the previous call's contents: each
// call clears what must start at zero, and two calls whose work overlaps on the GPU (on
// different streams, or from different host threads) race on it and must not be issued.
#include <cuda_runtime.h>

#include <cmath>
#include <mutex>

#include "../../include/sph_cuda.h"
#include "sph_device.cuh"
#include "sph_internal.h"

namespace sph {
namespace {

constexpr uint32_t kMaxParticles = 1u << 20;
constexpr uint32_t kMaxCells = 1u << 20;
constexpr uint32_t kMaxBlocks = kMaxCells / kScanTile + 1;  // group sums of the scan
constexpr size_t kBigWords = big_words(kMaxParticles);       // crowded-cell list
// counts | slot ids | group sums | crowded cells, as 32-bit words
constexpr size_t kScratchWords = (size_t) kMaxCells + kMaxParticles + kMaxBlocks + kBigWords;

__device__ __align__(256) uint32_t g_grid_scratch[kScratchWords];

// Device address of g_grid_scratch per device ordinal, looked up once per device (the host
// symbol is only a stand-in and must not be passed to a kernel).
constexpr int kMaxDevices = 64;
uint32_t *g_scratch_ptr[kMaxDevices] = {nullptr};
std::mutex g_scratch_mu;

// The cell of every particle, and the particle's slot in it: what the count held when the particle
// was counted (one atomic per cell and warp, its lanes taking consecutive slots), so no second
// atomic pass hands the slots out. Bound by the atomics' latency and rate. The per-group sums are not
// counted here: input in no particular order would add to a few hundred words with one atomic a
// particle (144 us for 1,000,003 scattered particles; 14 us without, and 3 us for k_group_sums).
__global__ void __launch_bounds__(256) k_hash_plain_xyz(const float *__restrict__ xyz, uint32_t n, float3 half,
                                                        int3 res, float inv_h, double h_d,
                                                        uint32_t *__restrict__ out_cell, uint32_t *__restrict__ count,
                                                        uint32_t *__restrict__ slot, uint32_t *__restrict__ big)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) big[0] = 0;  // the crowded-cell list, for the scan
    if (i >= n) return;
    const int cx = cell_axis(xyz[3 * i], half.x, inv_h, h_d, res.x);
    const int cy = cell_axis(xyz[3 * i + 1], half.y, inv_h, h_d, res.y);
    const int cz = cell_axis(xyz[3 * i + 2], half.z, inv_h, h_d, res.z);
    const uint32_t cell = (uint32_t) cx + (uint32_t) cy * (uint32_t) res.x + (uint32_t) cz * (uint32_t) res.x * (uint32_t) res.y;
    out_cell[i] = cell;
    const unsigned act = __activemask(), lane = threadIdx.x & 31u;
    const unsigned peers = __match_any_sync(act, cell);
    const int lead = __ffs(peers) - 1;
    uint32_t first = 0;
    if ((int) lane == lead) first = atomicAdd(count + cell, (uint32_t) __popc(peers));
    slot[i] = __shfl_sync(act, first, lead) + (uint32_t) __popc(peers & ((1u << lane) - 1u));
}

// particles of each group of kScanTile cells, for the scan's tile offsets (one block a group: 4 coalesced
// loads a thread)
__global__ void __launch_bounds__(256) k_group_sums(const uint32_t *__restrict__ count, uint32_t ncells,
                                                    uint32_t *__restrict__ gsum)
{
    chain_wait();
    static_assert(kScanTile == 4 * 256, "four cells a thread");
    __shared__ uint32_t part[8];
    uint32_t v = 0;
#pragma unroll
    for (uint32_t k = 0; k < 4; k++) {
        const uint32_t c = blockIdx.x * kScanTile + k * 256u + threadIdx.x;
        if (c < ncells) v += count[c];
    }
    v = __reduce_add_sync(0xffffffffu, v);
    if ((threadIdx.x & 31u) == 0) part[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t t = 0;
        for (int w = 0; w < 8; w++) t += part[w];
        gsum[blockIdx.x] = t;
    }
}

// every id to its slot of its cell
__global__ void __launch_bounds__(256) k_slot_ids(const uint32_t *__restrict__ cell, uint32_t n,
                                                  const uint32_t *__restrict__ start,
                                                  const uint32_t *__restrict__ slot, uint32_t *__restrict__ slot_ids)
{
    chain_wait();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    slot_ids[start[cell[i]] + slot[i]] = i;
}

// Canonical (cell, id) order: position = cell start + number of same-cell ids below i, counted. A thread a
// particle: up to kRankByParticle particles, where even a single cell of them all is a few million
// loads; beyond, k_order_cells.
constexpr uint32_t kRankByParticle = 65536;

__global__ void __launch_bounds__(256) k_rank_ids(const uint32_t *__restrict__ cell, uint32_t n,
                                                  const uint32_t *__restrict__ start,
                                                  const uint32_t *__restrict__ slot_ids, uint32_t *__restrict__ order)
{
    chain_wait();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t c = cell[i], b = start[c], e = start[c + 1];
    const uint32_t dst = b + count_rank(slot_ids, b, e, i);
    if (sph_check(dst < e && e <= n, CHK_SORT)) order[dst] = i;
}

// The same by cells, a thread a cell, so that neighbouring threads read and write neighbouring slots (a
// thread a particle reads two cell starts and the slots of a random cell). Cells above kBigCell particles
// are left to the list: those of up to kBigCellMax sorted by one block each (bitonic, in shared memory),
// larger ones (thousands of times the rest density) counted by all blocks together. The whole build of
// scattered particles, with this pass and with k_rank_ids: 65,000 22.6 / 18.2 us, 520,000 34.8 / 32.8,
// 1,040,000 46.5 / 49.2, and k_rank_ids would need a sort of crowded cells before it (3 us) at such sizes.
__global__ void __launch_bounds__(256) k_order_cells(const uint32_t *__restrict__ start, uint32_t ncells,
                                                     const uint32_t *__restrict__ slot_ids,
                                                     const uint32_t *__restrict__ big, uint32_t n,
                                                     uint32_t *__restrict__ order)
{
    __shared__ uint32_t sk[kBigCellMax];
    chain_wait();
    const uint32_t c = blockIdx.x * 256u + threadIdx.x;
    if (c < ncells) {
        const uint32_t b = start[c], e = start[c + 1];
        if (sph_check(b <= e && e <= n, CHK_SORT) && e - b <= kBigCell)
            for (uint32_t k = b; k < e; k++) {
                const uint32_t id = slot_ids[k];
                uint32_t r = b;
                for (uint32_t m = b; m < e; m++) r += slot_ids[m] < id ? 1u : 0u;
                order[r] = id;
            }
    }
    const uint32_t nbig = big[0];
    for (uint32_t q = 0; q < nbig; q++) {
        const uint32_t cell = big[1 + q];
        const uint32_t b = start[cell], e = start[cell + 1], occ = e - b;
        if (!sph_check(b <= e && e <= n, CHK_SORT)) continue;
        if (occ > kBigCellMax) {
            for (uint32_t k = b + c; k < e; k += gridDim.x * 256u)
                order[b + count_rank(slot_ids, b, e, slot_ids[k])] = slot_ids[k];
            continue;
        }
        if (q % gridDim.x != blockIdx.x) continue;
        uint32_t P = 2 * kBigCell;
        while (P < occ) P <<= 1;
        for (uint32_t t = threadIdx.x; t < P; t += 256) sk[t] = t < occ ? slot_ids[b + t] : 0xffffffffu;
        __syncthreads();
        for (uint32_t k = 2; k <= P; k <<= 1) {
            for (uint32_t j = k >> 1; j > 0; j >>= 1) {
                for (uint32_t t = threadIdx.x; t < P / 2; t += 256) {
                    const uint32_t lo = 2 * j * (t / j) + (t % j), hi = lo + j;  // lo has bit j clear
                    const uint32_t x = sk[lo], y = sk[hi];
                    if ((x > y) == ((lo & k) == 0)) {
                        sk[lo] = y;
                        sk[hi] = x;
                    }
                }
                __syncthreads();
            }
        }
        for (uint32_t t = threadIdx.x; t < occ; t += 256) order[b + t] = sk[t];
        __syncthreads();
    }
}

}  // namespace

// The reference's grid of n particles (float xyz, id order) in a box of res cells per axis (cells
// of size h, linear index x + y*X + z*X*Y): the cell of every particle, the cell starts and the
// ids in ascending (cell, id) order, with the working memory g (counts, slot ids, group sums,
// crowded-cell list) supplied by the caller.
cudaError_t ref_grid_build(const float *xyz, uint32_t n, int3 res, float3 half, float h, uint32_t *out_cell,
                           uint32_t *out_start, uint32_t *out_order, const GridScratch &g, cudaStream_t st)
{
    const uint64_t ncells = (uint64_t) res.x * (uint64_t) res.y * (uint64_t) res.z;
    DevBufs b{};
    b.count = g.count;
    b.tmp = g.tmp;
    b.bsum = g.bsum;
    b.big = g.big;
    b.start = out_start;
    // the counts start empty (a previous call, or one that failed, may have left values)
    cudaError_t e = cudaMemsetAsync(b.count, 0, 4 * ncells, st);
    if (e != cudaSuccess) return e;
    const unsigned blocks = (unsigned) ((n + 255) / 256);
    // the slots wait in out_order, which only the last pass writes
    if (n)
        k_hash_plain_xyz<<<blocks, 256, 0, st>>>(xyz, n, half, res, 1.0f / h, (double) h, out_cell, b.count, out_order,
                                                 b.big);
    e = cudaGetLastError();
    if (e == cudaSuccess)
        e = launch_chained(k_group_sums, (unsigned) (ncells / kScanTile + 1), 256, st, b.count, (uint32_t) ncells, b.bsum);
    if (e == cudaSuccess) e = Launch<float>::scan(b, (uint32_t) ncells, st);  // starts
    if (e == cudaSuccess && n)
        e = launch_chained(k_slot_ids, blocks, 256, st, out_cell, n, out_start, out_order, b.tmp);
    if (e == cudaSuccess && n)
        e = n <= kRankByParticle
                ? launch_chained(k_rank_ids, blocks, 256, st, out_cell, n, out_start, b.tmp, out_order)
                : launch_chained(k_order_cells, (unsigned) ((ncells + 255) / 256), 256, st, out_start, (uint32_t) ncells,
                                 b.tmp, b.big, n, out_order);
    return e;
}

SPH_CHECK_ACCESSOR(check_flags_noalloc)

}  // namespace sph

using namespace sph;

// The status code is the whole report: this entry point keeps no error text.
extern "C" int sph_grid_build_noalloc(const float *xyz, uint32_t n, const float box[3], float h, uint32_t *out_cell,
                                      uint32_t *out_start, uint32_t *out_order, void *stream)
{
    if (!box || !(h > 0) || !std::isfinite(h) || !out_start) return SPH_ERR_ARG;
    if (n && (!xyz || !out_cell || !out_order)) return SPH_ERR_ARG;
    // cells per axis as the context computes them (float quotient, then ceil), checked against
    // the scratch limit before the conversion to int so that no huge or infinite quotient is cast
    int r3[3];
    for (int a = 0; a < 3; a++) {
        if (!(box[a] > 0) || !std::isfinite(box[a])) return SPH_ERR_ARG;
        const float q = ceilf(box[a] / h);
        if (!(q <= (float) kMaxCells)) return SPH_ERR_CAPACITY;  // also an infinite quotient
        r3[a] = (int) q;
    }
    const int3 res = make_int3(r3[0], r3[1], r3[2]);
    const uint64_t ncells = (uint64_t) res.x * (uint64_t) res.y * (uint64_t) res.z;
    if (n > kMaxParticles || ncells > kMaxCells) return SPH_ERR_CAPACITY;  // beyond the fixed scratch
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return SPH_ERR_CUDA;
    uint32_t *scratch = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_scratch_mu);
        if (!g_scratch_ptr[dev]) {
            // first call on this device (with it current): resolve the array's device address
            void *p = nullptr;
            if (cudaGetSymbolAddress(&p, g_grid_scratch) != cudaSuccess || !p) return SPH_ERR_CUDA;
            g_scratch_ptr[dev] = (uint32_t *) p;
        }
        scratch = g_scratch_ptr[dev];
    }
    GridScratch g;
    g.count = scratch;
    g.tmp = scratch + (size_t) kMaxCells;
    g.bsum = scratch + (size_t) kMaxCells + kMaxParticles;
    g.big = g.bsum + kMaxBlocks;
    const float3 half = make_float3(box[0] / 2.0f, box[1] / 2.0f, box[2] / 2.0f);
    const cudaError_t e = ref_grid_build(xyz, n, res, half, h, out_cell, out_start, out_order, g, (cudaStream_t) stream);
    return e == cudaSuccess ? SPH_OK : SPH_ERR_CUDA;
}
