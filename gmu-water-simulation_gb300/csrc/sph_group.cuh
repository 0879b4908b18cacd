// sph_group.cuh -- what the group forms of the neighbour passes share (sph_group.cu: plain and FP64,
// sph_mixed.cu: mixed).
//
// In these forms G neighbouring lanes work on one particle (32/G particles a warp): each takes every
// G-th candidate of a row, and the accepted ones are compacted, in candidate order, into the group's
// list in shared memory. Every sum then runs over that list in the order in which the forms with one
// thread a particle visit their candidates, so the results are the same bits. The serial walk of a
// particle is G times shorter and there are G times as many warps, which is what small scenes and
// scenes with a few crowded regions need: they are bound by the latency of one thread's walk, not by
// instruction issue.
//
// Whole warps run these functions (a warp's lanes past n take part with empty rows).
#pragma once

#include "sph_device.cuh"

namespace sph {

constexpr unsigned kFullWarp = 0xffffffffu;
constexpr int kGroupThreads = 128;  // threads a block: 4 warps, each on its own particles

template <int G>
struct Group {
    static_assert(G >= 4 && G <= 32 && (G & (G - 1)) == 0, "a group is 4 to 32 lanes of a warp");
    static constexpr int PER_WARP = 32 / G;                         // particles a warp
    static constexpr int PER_BLOCK = PER_WARP * (kGroupThreads / 32);
    static constexpr int NR = (9 + G - 1) / G;                      // rows whose bounds one lane holds
    static constexpr unsigned MASK = G == 32 ? kFullWarp : (1u << (G & 31)) - 1u;
    unsigned gl;     // lane within the group
    unsigned shift;  // the group's first lane
    unsigned below;  // lanes of the group before this one
    int warp, slot;  // warp of the block, group of the warp
    __device__ __forceinline__ Group()
    {
        const unsigned lane = threadIdx.x & 31u;
        gl = lane & (unsigned) (G - 1);
        shift = lane - gl;
        below = (1u << gl) - 1u;
        warp = (int) (threadIdx.x >> 5);
        slot = (int) (lane / G);
    }
    __device__ __forceinline__ uint32_t particle() const
    {
        return (blockIdx.x * (kGroupThreads / 32) + (uint32_t) warp) * PER_WARP + (uint32_t) slot;
    }
    // the group's bits of a warp vote
    __device__ __forceinline__ unsigned vote(bool p) const
    {
        return (__ballot_sync(kFullWarp, p) >> shift) & MASK;
    }
};

// The sums of a block's particles in shared memory, so that its first warp finishes them with one lane
// each: the per-particle epilogue would otherwise run with one lane of every group.
template <class R, int G>
struct GroupSums {
    R f[Group<G>::PER_BLOCK][6];  // pressure x, y, z, viscosity x, y, z
    __device__ __forceinline__ void put(const Group<G> &g, R fp, R fv)
    {
        const int k = g.warp * Group<G>::PER_WARP + g.slot;
        if (g.gl < 3) {
            f[k][g.gl] = fp;
            f[k][3 + g.gl] = fv;
        }
        __syncthreads();
    }
};

// The nine rows (dy, dz) of three cells of size h around a particle, in the order of the other
// forms: lane r % G of a group holds first candidate and length of row r (0 beyond the grid).
template <int G>
struct GroupRows {
    uint32_t jb[Group<G>::NR], len[Group<G>::NR];
    __device__ __forceinline__ GroupRows(const Group<G> &g, const SceneDev &sc, const uint32_t *__restrict__ start,
                                         int cx, int cy, int cz, bool live, uint32_t n)
    {
        const int X = sc.res[0], Y = sc.res[1], Z = sc.res[2];
        const int xl = cx > 0 ? cx - 1 : 0, xh = cx + 1 < X ? cx + 1 : X - 1;
#pragma unroll
        for (int k = 0; k < Group<G>::NR; k++) {
            const int r = k * G + (int) g.gl;
            const int z = cz + r / 3 - 1, y = cy + r % 3 - 1;
            jb[k] = len[k] = 0;
            if (!live || r >= 9 || z < 0 || z >= Z || y < 0 || y >= Y) continue;
            const uint32_t row = sc.cell_base + (uint32_t) y * (uint32_t) X + (uint32_t) z * (uint32_t) X * (uint32_t) Y;
            const uint32_t b = __ldg(start + row + xl), e = __ldg(start + row + xh + 1);
            if (!sph_check(b <= e && e <= n, CHK_ROW)) continue;
            jb[k] = b;
            len[k] = e - b;
        }
    }
    // f(row, first candidate, length, longest row of the warp's particles)
    template <class F>
    __device__ __forceinline__ void each(F &&f) const
    {
#pragma unroll
        for (int k = 0; k < Group<G>::NR; k++)
#pragma unroll 1
            for (int q = 0; q < G && k * G + q < 9; q++) {
                const uint32_t b = __shfl_sync(kFullWarp, jb[k], q, G), l = __shfl_sync(kFullWarp, len[k], q, G);
                const uint32_t most = __reduce_max_sync(kFullWarp, l);
                if (most) f(k * G + q, b, l, most);
            }
    }
};

constexpr int kListFlush = 96;              // entries from which a list is worked off ...
constexpr int kListLen = kListFlush + 32 + 8;  // ... before the next 32 candidates (+8: other banks per group)

// One neighbour's factors and differences, waiting for the ordered sums: (difference of positions,
// difference of velocities) per axis, then the two factors.
template <class R>
struct alignas(8 * sizeof(R)) PairOut {
    R v[8];
};

// Sums of one axis each in lanes 0 to 2 of a group: fp += w * d, fv += dv * l over cnt pairs in order.
template <class R>
__device__ __forceinline__ void add_pairs(const PairOut<R> *out, uint32_t cnt, unsigned axis, R &fp, R &fv)
{
#pragma unroll 4
    for (uint32_t s = 0; s < cnt; s++) {
        const R d = out[s].v[2 * axis], dv = out[s].v[2 * axis + 1];
        fp = rfma(out[s].v[6], d, fp);
        fv = rfma(dv, out[s].v[7], fv);
    }
}

}  // namespace sph
