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

#include <algorithm>
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
// counts | slot ids | crowded cells | group sums, as 32-bit words
constexpr size_t kScratchWords = (size_t) kMaxCells + kMaxParticles + kBigWords + kMaxBlocks;

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
    if (i < kBigHead) big[i] = 0;  // the crowded cells' lists, for the scan
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

// Every id to its slot of its cell. It lets the next kernel be scheduled only as it ends: k_order's blocks would
// else be placed beside this kernel's, several on some SMs and none on others, and those that order crowded
// cells would share an SM (60,000 particles in 18 cells 150 us, so 43).
__global__ void __launch_bounds__(256) k_slot_ids(const uint32_t *__restrict__ cell, uint32_t n,
                                                  const uint32_t *__restrict__ start,
                                                  const uint32_t *__restrict__ slot, uint32_t *__restrict__ slot_ids)
{
    chain_wait_last();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    slot_ids[start[cell[i]] + slot[i]] = i;
}

// Canonical (cell, id) order: position = cell start + number of same-cell ids below i, counted. Cells up to the
// number of particles from which the scan lists them are ordered by a thread a particle (k_order<false>: it
// reads two cell starts and the slots of a random cell), or by a thread a cell (k_order<true>: neighbouring
// threads read and write neighbouring slots), the listed ones by warps and blocks.
//
// A thread a cell wants many cells of few particles each: beyond kOrderByCell particles and from a sixth as many
// cells. Whole builds by cell / by particle: 1,000,003 scattered particles in 800,000 cells 50.7 / 54.3 us, 1,000,000
// at 5 a cell 46.5 / 55, but 520,000 38.2 / 37.7, 260,000 30.7 / 27.5, 70,000 24.9 / 21.1, and 400,000 in a fountain,
// whose crowded cells lie side by side, 62 / 53.
constexpr uint32_t kOrderByCell = 524288;
// Cells are listed beyond kBigCell particles, but in builds of up to kFewLists particles only beyond kWarpCell: there a
// few crowded cells leave most warps idle either way (with 32 / 128: a fountain of 60,000 27.5 / 24.7 us, of 30,000
// 25.5 / 22.2), beyond it the scattered loads of a thread a particle bind (200,000 at 100 a cell 38 / 47 us).
constexpr uint32_t kFewLists = 65536;

// One where w < id, else zero, for whole numbers. As floats (exact up to 2^24) it is one full-rate FP32
// instruction, the saturated difference; the integer compare runs at half the rate and needs a second one.
__device__ __forceinline__ float below(float w, float id)
{
    float r;
    asm("sub.sat.f32 %0, %1, %2;" : "=f"(r) : "f"(id), "f"(w));
    return r;
}
__device__ __forceinline__ uint32_t below(uint32_t w, uint32_t id) { return w < id ? 1u : 0u; }
constexpr uint32_t kFloatIds = 1u << 24;

// kPart of the ids in the slots [b, e) of a crowded cell, from slot k on, two a thread, against all of them,
// which the block stages 1,024 at a time. Called by whole blocks.
constexpr uint32_t kPart = 512;
template <class T>
struct alignas(16) Quad {
    T x, y, z, w;
};
template <class T>
__device__ __forceinline__ void place_part(Quad<T> *stage, const uint32_t *__restrict__ slot_ids, uint32_t b, uint32_t e,
                                           uint32_t k, uint32_t *__restrict__ order)
{
    const uint32_t k0 = k + threadIdx.x, k1 = k0 + 256u;
    const uint32_t id0 = k0 < e ? slot_ids[k0] : 0u, id1 = k1 < e ? slot_ids[k1] : 0u;
    const T f0 = (T) id0, f1 = (T) id1, none = (T) 0xffffffffu;
    T r0 = 0, r1 = 0;
    for (uint32_t c = b & ~3u; c < e; c += 1024u) {
        const uint32_t j = c + 4u * threadIdx.x;
        if (j < e) {
            const uint4 v = *reinterpret_cast<const uint4 *>(slot_ids + j);
            stage[threadIdx.x] = {j >= b ? (T) v.x : none, j + 1 >= b && j + 1 < e ? (T) v.y : none,
                                  j + 2 >= b && j + 2 < e ? (T) v.z : none, j + 3 >= b && j + 3 < e ? (T) v.w : none};
        }
        __syncthreads();
        const uint32_t quads = min(256u, (e - c + 3u) / 4u);
#pragma unroll 4
        for (uint32_t q = 0; q < quads; q++) {
            const Quad<T> w = stage[q];
            r0 += below(w.x, f0), r0 += below(w.y, f0), r0 += below(w.z, f0), r0 += below(w.w, f0);
            r1 += below(w.x, f1), r1 += below(w.y, f1), r1 += below(w.z, f1), r1 += below(w.w, f1);
        }
        __syncthreads();
    }
    const uint32_t d0 = b + (uint32_t) r0, d1 = b + (uint32_t) r1;
    if (k0 < e && sph_check(d0 < e, CHK_SORT)) order[d0] = id0;
    if (k1 < e && sph_check(d1 < e, CHK_SORT)) order[d1] = id1;
}

// The listed cells: up to kWarpCell particles a warp a cell; up to kSplitCell a block a cell; beyond, the parts of
// all of them dealt out over all blocks, so that no few cells hold one SM up. The lists are walked with the
// grid's stride or 32 entries at a time: every block reading every entry, or a grid sized by the cells alone,
// costs milliseconds. Whole builds, in the order 33, 100, 400, 3,000, 8,000 particles a cell: 1,000,000 65, 65,
// 97, 399, 703 us; 200,000 34, 38, 55, 113, 180; a fountain of 90,000 30, of 400,000 53; 70,000 in one cell 428.
template <bool BY_CELL>
__global__ void __launch_bounds__(256) k_order(const uint32_t *__restrict__ cell, const uint32_t *__restrict__ start,
                                               uint32_t ncells, const uint32_t *__restrict__ slot_ids,
                                               const uint32_t *__restrict__ big, uint32_t room, uint32_t from,
                                               uint32_t n, uint32_t *__restrict__ order)
{
    __shared__ Quad<uint32_t> stage[256];
    chain_wait();
    const uint32_t t = blockIdx.x * 256u + threadIdx.x, lane = threadIdx.x & 31u;
    const uint2 *const list = reinterpret_cast<const uint2 *>(big + kBigHead);
    const uint32_t few = big[0], many = big[1], most = big[2];
    if (BY_CELL) {
        if (t < ncells) {
            const uint32_t b = start[t], e = start[t + 1];
            if (sph_check(b <= e && e <= n, CHK_SORT) && e - b <= from)
                for (uint32_t k = b; k < e; k++) {
                    const uint32_t id = slot_ids[k];
                    uint32_t r = b;
                    for (uint32_t m = b; m < e; m++) r += slot_ids[m] < id ? 1u : 0u;
                    order[r] = id;
                }
        }
    } else if (t < n) {
        const uint32_t c = cell[t], b = start[c], e = start[c + 1];
        if (sph_check(b <= e && e <= n, CHK_SORT) && e - b <= from) {
            const uint32_t dst = b + count_rank(slot_ids, b, e, t);
            if (sph_check(dst < e, CHK_SORT)) order[dst] = t;
        }
    }
    auto part = [&](uint32_t b, uint32_t e, uint32_t k) {
        if (n <= kFloatIds) place_part((Quad<float> *) stage, slot_ids, b, e, k, order);
        else place_part(stage, slot_ids, b, e, k, order);
    };
    // a warp a cell
    for (uint32_t q = t >> 5; q < few; q += gridDim.x * 8u) {
        const uint2 be = list[q];
        if (!sph_check(be.x <= be.y && be.y <= n, CHK_SORT)) continue;
        for (uint32_t k = be.x + lane; k < be.y; k += 32u) {
            const uint32_t id = slot_ids[k], dst = be.x + count_rank(slot_ids, be.x, be.y, id);
            if (sph_check(dst < be.y, CHK_SORT)) order[dst] = id;
        }
    }
    // a block a cell
    for (uint32_t q = blockIdx.x; q < many; q += gridDim.x) {
        const uint2 be = list[room - 1 - q];
        if (!sph_check(be.x <= be.y && be.y <= n, CHK_SORT)) continue;
        for (uint32_t k = be.x; k < be.y; k += kPart) part(be.x, be.y, k);
    }
    // a part a block, the parts of all cells dealt out over all blocks; 32 cells of the list at a time
    for (uint32_t q0 = 0, turn = blockIdx.x; q0 < most; q0 += 32u) {
        uint2 be = make_uint2(0, 0);
        if (q0 + lane < most) be = list[room + q0 + lane];
        if (!sph_check(be.x <= be.y && be.y <= n, CHK_SORT)) be = make_uint2(0, 0);
        const uint32_t parts = (be.y - be.x + kPart - 1) / kPart;
        uint32_t upto = parts;  // of this cell and the ones before it
#pragma unroll
        for (uint32_t o = 1; o < 32u; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += v;
        }
        const uint32_t total = __shfl_sync(0xffffffffu, upto, 31);
        for (; turn < total; turn += gridDim.x) {
            const int s = __ffs(__ballot_sync(0xffffffffu, upto > turn)) - 1;
            const uint32_t b = __shfl_sync(0xffffffffu, be.x, s), e = __shfl_sync(0xffffffffu, be.y, s);
            part(b, e, b + (turn - __shfl_sync(0xffffffffu, upto - parts, s)) * kPart);
        }
        turn -= total;
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
    b.big_room = n / kBigCell;
    b.big_from = n > kFewLists ? kBigCell : kWarpCell;
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
    if (e == cudaSuccess && n) {
        const bool by_cell = n > kOrderByCell && ncells >= n / 6;
        e = launch_chained(by_cell ? k_order<true> : k_order<false>,
                           by_cell ? std::max(blocks, (unsigned) ((ncells + 255) / 256)) : blocks, 256, st, out_cell,
                           out_start, (uint32_t) ncells, b.tmp, b.big, b.big_room, b.big_from, n, out_order);
    }
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
    g.big = g.tmp + kMaxParticles;
    g.bsum = g.big + kBigWords;
    const float3 half = make_float3(box[0] / 2.0f, box[1] / 2.0f, box[2] / 2.0f);
    const cudaError_t e = ref_grid_build(xyz, n, res, half, h, out_cell, out_start, out_order, g, (cudaStream_t) stream);
    return e == cudaSuccess ? SPH_OK : SPH_ERR_CUDA;
}
