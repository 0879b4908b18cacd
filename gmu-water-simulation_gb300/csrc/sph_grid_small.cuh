// sph_grid_small.cuh -- the grid pass of a small scene in one launch (scan of the cell counts, slots,
// canonical rank and permute: k_scan_apply, k_slot and k_rank_permute of sph_kernels.cu in turn).
//
// On small scenes each of the three kernels is little more than its launch and a few dependent L2 round
// trips. One cluster of 8 blocks, a thread a particle, does all three with two cluster barriers between
// them; the particles' cells are loaded while the counts are scanned. Chained launches already overlap
// most of the kernels' latency, so a step alone gains 1 us of 12; three contexts at once, which are bound
// by the rate at which the GPU starts kernels, gain 12% (40 steps of 8,000 particles 603 -> 530 us). With
// more than one particle a thread the cluster's 8 SMs are too few (16,000 particles: 13.0 us, against 10.9
// in three kernels; 20,000: 20.5 / 11.3).
// Place is what each particle's record becomes: fetch(i) loads it, store(dst) writes it.
#pragma once

#include "sph_device.cuh"

namespace sph {

// all threads of the cluster; what each wrote before is visible to the others after
__device__ __forceinline__ void cluster_meet()
{
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <class Place>
__global__ void __cluster_dims__(kSmallBlocks, 1, 1) __launch_bounds__(kSmallThreads)
    k_grid_small(Place place, const uint2 *__restrict__ cid_u, uint32_t n, uint32_t *start, uint32_t *count,
                 uint32_t *tmp, uint32_t *gsum, uint32_t ncells)
{
    constexpr uint32_t NONE = 0xffffffffu;  // cell of lanes past n
    __shared__ uint32_t warp_sum[kSmallThreads / 32];
    chain_wait();
    const unsigned lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    const uint32_t i = blockIdx.x * kSmallThreads + threadIdx.x;
    const uint2 cd = i < n ? cid_u[i] : make_uint2(NONE, 0);
    // sum over the block, and over the threads before this one
    auto scan = [&](uint32_t v, uint32_t &before) {
        uint32_t x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if ((int) lane >= o) x += y;
        }
        __syncthreads();  // the last use of warp_sum is over
        if (lane == 31) warp_sum[wid] = x;
        __syncthreads();
        uint32_t mine = warp_sum[lane];
        const uint32_t total = __reduce_add_sync(0xffffffffu, mine);
        before = __reduce_add_sync(0xffffffffu, lane < wid ? mine : 0u) + x - v;
        return total;
    };
    // cell starts: 4 cells a thread, a contiguous run of 4096-cell tiles a block
    constexpr uint32_t TILE = 4 * kSmallThreads;
    const uint32_t tiles = (ncells + TILE - 1) / TILE, per = (tiles + kSmallBlocks - 1) / kSmallBlocks;
    const uint32_t t0 = min(tiles, blockIdx.x * per), t1 = min(tiles, t0 + per);
    uint32_t part = 0, before;
    for (uint32_t g = threadIdx.x; g < t0 * (TILE / kScanTile); g += kSmallThreads) part += gsum[g];
    uint32_t off = scan(part, before);
    for (uint32_t t = t0; t < t1; t++) {
        const uint32_t base = t * TILE + 4 * threadIdx.x;
        uint4 c = make_uint4(0, 0, 0, 0);
        if (base + 4 <= ncells) c = *reinterpret_cast<const uint4 *>(count + base);
        else if (base < ncells) {
            c.x = count[base];
            if (base + 1 < ncells) c.y = count[base + 1];
            if (base + 2 < ncells) c.z = count[base + 2];
        }
        const uint32_t total = scan(c.x + c.y + c.z + c.w, before);
        const uint32_t s0 = off + before, s1 = s0 + c.x, s2 = s1 + c.y, s3 = s2 + c.z;
        if (base + 4 <= ncells) *reinterpret_cast<uint4 *>(start + base) = make_uint4(s0, s1, s2, s3);
        else if (base < ncells) {
            start[base] = s0;
            if (base + 1 < ncells) start[base + 1] = s1;
            if (base + 2 < ncells) start[base + 2] = s2;
        }
        off += total;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) start[ncells] = n;
    cluster_meet();
    // slots, as k_slot takes them: one atomic per cell and warp, which leaves the counts at zero
    const unsigned peers = __match_any_sync(0xffffffffu, cd.x);
    const int lead = __ffs(peers) - 1;
    uint32_t top = 0;
    if (cd.x != NONE && (int) lane == lead)
        top = atomicSub(count + cd.x, (uint32_t) __popc(peers)) + __ldcg(start + cd.x);
    const uint32_t slot = __shfl_sync(0xffffffffu, top, lead) - (uint32_t) __popc(peers >> lane);
    if (cd.x != NONE && sph_check(slot < n, CHK_SORT)) tmp[slot] = cd.y;
    cluster_meet();
    for (uint32_t g = i; g < ncells / kScanTile + 1; g += kSmallParticles) gsum[g] = 0;
    // canonical rank, and the particle to its place (the barrier's acquire lets plain loads see the slots)
    if (i >= n) return;
    place.fetch(i);
    const uint32_t b = __ldcg(start + cd.x), e = __ldcg(start + cd.x + 1);
    if (!sph_check(b <= e && e <= n, CHK_SORT)) return;
    const uint32_t r = b + count_rank(tmp, b, e, cd.y);
    if (sph_check(r < e, CHK_SORT)) place.store(r);
}

template <class Place>
inline cudaError_t launch_grid_small(const Place &place, const DevBufs &b, uint32_t n, uint32_t ncells, cudaStream_t st)
{
    return launch_chained(k_grid_small<Place>, kSmallBlocks, kSmallThreads, st, place, b.cid_u, n, b.start, b.count,
                          b.tmp, b.bsum, ncells);
}

}  // namespace sph
