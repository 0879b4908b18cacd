// sph_mixed.cu -- the mixed-precision form of the step (SPH_MIXED).
//
// Same method and pass structure as the plain form (sph_kernels.cu), with these changes:
//  - neighbour positions are gathered as 16-bit codes per axis (8 bytes per particle instead
//    of 16): code = (c mod 8) << 13 | q, where c = floor((p + box/2) / h) is the particle's
//    unclamped cell along that axis and q its offset inside that cell in units of h / 8192.
//    The 16-bit two's-complement difference of two codes is the displacement in those units,
//    exactly, when the particles are less than 4 h apart along the axis; from 4 h to 7 h apart
//    it wraps to a magnitude above h, so the neighbour test still rejects the pair (every
//    neighbour candidate is within 7 h unless a particle has been pushed more than ~5 h
//    outside the box);
//  - the force pass reads each neighbour from one packed 16-byte record that the density pass
//    writes: the three 16-bit position codes, the FP16 velocity, and the neighbour's two force
//    factors p/rho^2 and 1/rho in FP16, scaled by 2^10 and 2^14 into FP16's normal range
//    (relative rounding error at most 2^-11 each; the particle's own factors stay FP32);
//  - density sums are compensated FP32 sums: each 32-candidate chunk is summed, and the chunk
//    sums are added with Kahan compensation;
//  - each particle's position is a hi/lo FP32 pair through the integration (TwoSum), and the
//    velocity update is the increment over dt, so no cancellation of x' - x occurs.
// The master state (hi, lo, FP32 velocity) is still read and written once per pass.
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "sph_device.cuh"
#include "sph_grid_small.cuh"
#include "sph_group.cuh"
#include "sph_internal.h"

namespace sph {

constexpr float QUNITS = 8192.0f;        // code units per h
constexpr float QH2 = 67108864.0f;       // h^2 in code units^2 (2^26)

// ---- encoding ------------------------------------------------------------------------
// code of one axis from the hi/lo coordinate: unclamped cell c and offset q inside it
__device__ __forceinline__ uint32_t axis_code(float p, float lo, float half, float h, float inv_h, float to_units)
{
    const float t = (p + half) + lo;            // distance from the box's min wall
    const float c = floorf(t * inv_h);
    int q = __float2int_rd(fmaf(-c, h, t) * to_units);
    q = q < 0 ? 0 : (q > 8191 ? 8191 : q);      // rounding at a cell face
    return ((uint32_t) ((int) c & 7) << 13) | (uint32_t) q;
}

// displacement i - j in code units from the packed codes (x | y << 16, z)
__device__ __forceinline__ void code_delta(uint2 gi, uint2 gj, float &dx, float &dy, float &dz)
{
    const uint32_t dxy = __vsub2(gi.x, gj.x);
    dx = (float) (int16_t) (dxy & 0xffffu);
    dy = (float) ((int32_t) dxy >> 16);
    dz = (float) (int16_t) ((gi.y - gj.y) & 0xffffu);
}

__device__ __forceinline__ uint32_t pack_half2(float lo, float hi)
{
    const __half2 a = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&a);
}

__device__ __forceinline__ float2 unpack_half2(uint32_t v)
{
    return __half22float2(*reinterpret_cast<const __half2 *>(&v));
}

// Scales of the FP16 force factors in the neighbour record: p/rho^2 lies in [-0.03, 0.001] and
// 1/rho in (0, 1/328] (a density always includes the particle's own term, m poly6(0) = 328.3), so
// these bring both into FP16's normal range with room on either side.
constexpr float Q_SCALE = 1024.0f;       // p / rho^2 * 2^10
constexpr float INV_SCALE = 16384.0f;    // 1 / rho * 2^14

// The force pass's view of a neighbour, one 16-byte record:
//   x: codes x | y << 16; y: code z | FP16 vx << 16; z: FP16 vy | FP16 vz << 16;
//   w: FP16 (p/rho^2 * 2^10) | FP16 (1/rho * 2^14) << 16
__device__ __forceinline__ uint4 make_record(uint2 g, float vx, float vy, float vz, float q, float inv)
{
    return make_uint4(g.x, (g.y & 0xffffu) | (pack_half2(vx, 0.0f) << 16), pack_half2(vy, vz),
                      pack_half2(q * Q_SCALE, inv * INV_SCALE));
}

// ---- grid: canonical rank + permute, writing the master state and the gather records ----
struct PlaceMixed {
    const Vec4<float> *pos_u, *lo_u, *vel_u;
    const SceneDev *scenes;
    float h, inv_h, to_units;
    Vec4<float> *pos_s, *lo_s, *vel_s;
    uint2 *gpos;
    Vec4<float> p, lo, v;
    __device__ __forceinline__ void fetch(uint32_t i)
    {
        p = ld4(pos_u + i);
        lo = ld4(lo_u + i);
        v = ld4(vel_u + i);
    }
    __device__ __forceinline__ void store(uint32_t dst) const
    {
        st4(pos_s + dst, p);
        st4(lo_s + dst, lo);
        st4(vel_s + dst, v);
        const SceneDev sc = load_scene(scenes, wbits(p.w));
        const uint32_t qx = axis_code(p.x, lo.x, sc.half[0], h, inv_h, to_units);
        const uint32_t qy = axis_code(p.y, lo.y, sc.half[1], h, inv_h, to_units);
        const uint32_t qz = axis_code(p.z, lo.z, sc.half[2], h, inv_h, to_units);
        gpos[dst] = make_uint2(qx | (qy << 16), qz);
    }
};

// (the state loads issued before the rank is counted, as in the plain form's k_rank_permute)
__global__ void __launch_bounds__(256) k_rank_permute_mixed(PlaceMixed place, const uint2 *__restrict__ cid_u, uint32_t n,
                                                            const uint32_t *__restrict__ start,
                                                            const uint32_t *__restrict__ tmp,
                                                            uint32_t *__restrict__ gsum, uint32_t ngroups)
{
    chain_wait();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    for (uint32_t t = i; t < ngroups; t += gridDim.x * blockDim.x) gsum[t] = 0;  // for the next hash
    if (i >= n) return;
    const uint2 cd = cid_u[i];
    place.fetch(i);
    const uint32_t b = start[cd.x], e = start[cd.x + 1];
    if (!sph_check(b <= e && e <= n, CHK_SORT)) return;
    const uint32_t dst = b + count_rank(tmp, b, e, cd.y);
    if (sph_check(dst < e, CHK_SORT)) place.store(dst);
}

// Kahan step with explicitly rounded operations (no reassociation, no fused multiply-add)
__device__ __forceinline__ void kahan_add(float &sum, float &comp, float term)
{
    const float y = __fsub_rn(term, comp);
    const float t = __fadd_rn(sum, y);
    comp = __fsub_rn(__fsub_rn(t, sum), y);
    sum = t;
}

// ---- density: neighbour masks (as the plain mask kernel), compensated sums ---------------
// Issue slots bound it (83% of them used at 1,000,000 fallen particles), so the mask word takes one funnel shift
// of the sign of r^2 - h^2 a candidate instead of a compare, a select and a shift-or: cells of h/2 256 to
// 234 us, cells of h 264 to 242 us (200,000: 74 to 68). Unrolled 8 times the longer rows of cells of h gain
// a little more at rest (137 to 131 us), the short ones of cells of h/2 lose (234 to 254: the remainders).
template <int RAD>
__global__ void __launch_bounds__(128) k_density_mixed(const Vec4<float> *__restrict__ pos,
                                                       const uint2 *__restrict__ gpos, Vec4<float> *__restrict__ aux,
                                                       const uint32_t *__restrict__ start,
                                                       const SceneDev *__restrict__ scenes, uint32_t n,
                                                       Consts<float> c, MixConsts mc, uint32_t *__restrict__ masks,
                                                       const Vec4<float> *__restrict__ vel, uint4 *__restrict__ rec)
{
    using St = Stencil<RAD>;
    chain_wait();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const Vec4<float> pi = ld4(pos + i);
    const uint2 gi = __ldg(gpos + i);
    const SceneDev sc = load_scene(scenes, wbits(pi.w));
    int cx, cy, cz;
    hash_cell<float>(sc, pi.x, pi.y, pi.z, c, cx, cy, cz);
    float sum = 0.0f, comp = 0.0f;
    const uint64_t keep = l2_keep_policy();  // masks and records: read by the force pass next
    const int X = sc.res[0], Y = sc.res[1], Z = sc.res[2];
    const int xl = cx - RAD > 0 ? cx - RAD : 0, xh = cx + RAD < X ? cx + RAD : X - 1;
#pragma unroll 1
    for (int dz = -RAD; dz <= RAD; dz++) {
#pragma unroll 1
        for (int dy = -RAD; dy <= RAD; dy++) {
            const int r = (dz + RAD) * (2 * RAD + 1) + (dy + RAD);
            const int z = cz + dz, y = cy + dy;
            if (z < 0 || z >= Z || y < 0 || y >= Y) continue;
            const uint32_t row = sc.cell_base + (uint32_t) y * (uint32_t) X + (uint32_t) z * (uint32_t) X * (uint32_t) Y;
            const uint32_t jb = __ldg(start + row + xl), je = __ldg(start + row + xh + 1);
            if (!sph_check(jb <= je && je <= n, CHK_ROW)) continue;
            int w = 0;
            for (uint32_t cb = jb; cb < je; cb += 32, w++) {
                const uint32_t ce = min(je, cb + 32u);
                uint32_t m = 0;
                float csum = 0.0f;  // minus the chunk's terms (at most 32), then one compensated add
                // bit k of the chunk's word = candidate cb + k
#pragma unroll (RAD == 1 ? 8 : 4)
                for (uint32_t j = cb; j < ce; j++) {
                    float x, yy, zz;
                    code_delta(gi, __ldg(gpos + j), x, yy, zz);
                    float u = r2_minus_h2<float>(x, yy, zz, QH2);
                    m = __funnelshift_l(sign_word(u), m, 1);
                    u = fminf(u, 0.0f);
                    csum = rfma(rmul(u, u), u, csum);
                }
                kahan_add(sum, comp, -csum);
                m = __brev(m) >> (32 - (ce - cb));
                if (w < St::WORDS) st_keep(masks + (size_t) (r * St::WORDS + w) * n + i, m, keep);
            }
        }
    }
    const float rho = __fmul_rn(__fmul_rn(sum, mc.poly6_q), c.mass);
    const float p = __fmul_rn(c.k, __fsub_rn(rho, c.rho0));
    const float q = __fdiv_rn(p, __fmul_rn(rho, rho)), inv = __fdiv_rn(1.0f, rho);
    st4(aux + i, Vec4<float>{rho, p, q, inv});
    const Vec4<float> vi = ld4(vel + i);
    st_keep(rec + i, make_record(gi, vi.x, vi.y, vi.z, q, inv), keep);
}

// ---- forces: mask-driven, code-unit displacements, one 16-byte record per neighbour ----------
// Pressure and viscosity terms of one neighbour from its record (the plain form's pair terms in
// code units; src/CCPUParticleSimulator.cpp:177-183). qs = own p/rho^2 * 2^10.
// mixed_factors: the difference d, the neighbour's velocity and the two factors; w * d and
// l * (vj - vi) are summed.
__device__ __forceinline__ void mixed_factors(uint2 gi, float qs, uint4 r, const MixConsts &mc, float &dx, float &dy,
                                              float &dz, float &vjx, float &vjy, float &vjz, float &wgt, float &l)
{
    code_delta(gi, make_uint2(r.x, r.y), dx, dy, dz);
    vjx = unpack_half2(r.y >> 16).x;
    const float2 vyz = unpack_half2(r.z);
    const float2 qv = unpack_half2(r.w);
    vjy = vyz.x;
    vjz = vyz.y;
    // at least one unit apart: two particles sharing a code (closer than the 5.6 um resolution)
    // get no pressure direction rather than a 0/0
    const float r2 = fmaxf(dx * dx + dy * dy + dz * dz, 1.0f);
    const float rinv = inv_sqrt_normal(r2);  // r2 is never denormal
    const float hr = QUNITS - r2 * rinv;
    wgt = (qs + qv.x) * (mc.spiky_q * (1.0f / Q_SCALE) * hr * hr * rinv);
    l = mc.visc_q * (1.0f / INV_SCALE) * hr * qv.y;
}

__device__ __forceinline__ void mixed_pair(uint2 gi, const Vec4<float> &vi, float qs, uint4 r, const MixConsts &mc,
                                           float &fpx, float &fpy, float &fpz, float &fvx, float &fvy, float &fvz)
{
    float dx, dy, dz, vjx, vjy, vjz, wgt, l;
    mixed_factors(gi, qs, r, mc, dx, dy, dz, vjx, vjy, vjz, wgt, l);
    fpx += wgt * dx;
    fpy += wgt * dy;
    fpz += wgt * dz;
    fvx += (vjx - vi.x) * l;
    fvy += (vjy - vi.y) * l;
    fvz += (vjz - vi.z) * l;
}

// The rest of the force pass for one particle: x' = x + (v dt + (a dt) dt) with x = hi + lo carried by
// TwoSum, v' = increment / dt, and the cell of the new position.
__device__ __forceinline__ void finish_mixed(uint32_t i, const Vec4<float> &pi, const Vec4<float> &vi, float rho,
                                             const SceneDev &sc, const Vec4<float> *__restrict__ lo_s,
                                             const ObstacleDev *__restrict__ obstacles, const Consts<float> &c,
                                             float fpx, float fpy, float fpz, float fvx, float fvy, float fvz,
                                             Vec4<float> *__restrict__ pos_out, Vec4<float> *__restrict__ lo_out,
                                             Vec4<float> *__restrict__ vel_out, Vec4<float> *__restrict__ acc_out,
                                             uint2 *__restrict__ cid_out, uint32_t *__restrict__ count)
{
    float ax, ay, az;
    accel_of<float>(pi, vi, rho, sc, obstacles, c, fpx, fpy, fpz, fvx, fvy, fvz, ax, ay, az);
    const Vec4<float> li = ld4(lo_s + i);
    const float dt = c.dt;
    const float ix = __fadd_rn(__fmul_rn(vi.x, dt), __fmul_rn(__fmul_rn(ax, dt), dt));
    const float iy = __fadd_rn(__fmul_rn(vi.y, dt), __fmul_rn(__fmul_rn(ay, dt), dt));
    const float iz = __fadd_rn(__fmul_rn(vi.z, dt), __fmul_rn(__fmul_rn(az, dt), dt));
    float hx, lx, hy, ly, hz, lz;
    two_sum(pi.x, __fadd_rn(li.x, ix), hx, lx);
    two_sum(pi.y, __fadd_rn(li.y, iy), hy, ly);
    two_sum(pi.z, __fadd_rn(li.z, iz), hz, lz);
    st4(pos_out + i, Vec4<float>{hx, hy, hz, pi.w});
    st4(lo_out + i, Vec4<float>{lx, ly, lz, 0.0f});
    st4(vel_out + i, Vec4<float>{__fdiv_rn(ix, dt), __fdiv_rn(iy, dt), __fdiv_rn(iz, dt), vi.w});
    if (acc_out) st4(acc_out + i, Vec4<float>{ax, ay, az, 0.0f});
    int qx, qy, qz;
    const uint32_t cell = hash_cell<float>(sc, hx, hy, hz, c, qx, qy, qz);
    count_add(count, c.gsum, cell);
    cid_out[i] = make_uint2(cell, wbits(vi.w));
}

// Two accepted neighbours per iteration: both records are loaded before either's terms are
// added (two gathers in flight), the terms still added in candidate order. MINB and BLOCK set
// the register budget and block size (the launch variants of the mixed form).
// Issue slots bound it (73% issue, 20 of 32 lanes at 1,000,000 fallen particles): the mask word is bit-reversed
// so that the next candidate is a count of leading zeros (one instruction fewer than find-first-set each),
// and the reciprocal root goes without rsqrtf's care for denormals. Before/after at 1,000,000 fallen
// particles: cells of h/2 321 to 311 us, cells of h 317 to 307 us; 90,000 in a fountain's pool 102 to 98 us.
template <int MINB, int BLOCK, int RAD>
__global__ void __launch_bounds__(BLOCK, MINB) k_forces_mixed(
    const Vec4<float> *__restrict__ pos, const Vec4<float> *__restrict__ lo_s, const Vec4<float> *__restrict__ vel,
    const Vec4<float> *__restrict__ aux, const uint2 *__restrict__ gpos, const uint4 *__restrict__ rec,
    const uint32_t *__restrict__ start, const SceneDev *__restrict__ scenes, const ObstacleDev *__restrict__ obstacles,
    uint32_t n, Consts<float> c, MixConsts mc, const uint32_t *__restrict__ masks, Vec4<float> *__restrict__ pos_out,
    Vec4<float> *__restrict__ lo_out, Vec4<float> *__restrict__ vel_out, Vec4<float> *__restrict__ acc_out,
    uint2 *__restrict__ cid_out, uint32_t *__restrict__ count)
{
    chain_wait();
    const uint32_t i = blockIdx.x * BLOCK + threadIdx.x;
    if (i >= n) return;
    const Vec4<float> pi = ld4(pos + i);
    const Vec4<float> vi = ld4(vel + i);
    const Vec4<float> ai = ld4(aux + i);
    const uint2 gi = __ldg(gpos + i);
    const SceneDev sc = load_scene(scenes, wbits(pi.w));
    int cx, cy, cz;
    hash_cell<float>(sc, pi.x, pi.y, pi.z, c, cx, cy, cz);
    const float qs = ai.z * Q_SCALE;
    float fpx = 0, fpy = 0, fpz = 0, fvx = 0, fvy = 0, fvz = 0;
    using St = Stencil<RAD>;
    const int X = sc.res[0], Y = sc.res[1], Z = sc.res[2];
    const int xl = cx - RAD > 0 ? cx - RAD : 0, xh = cx + RAD < X ? cx + RAD : X - 1;
#pragma unroll 1
    for (int dz = -RAD; dz <= RAD; dz++) {
#pragma unroll 1
        for (int dy = -RAD; dy <= RAD; dy++) {
            const int r = (dz + RAD) * (2 * RAD + 1) + (dy + RAD);
            if (r + 1 < St::ROWS) prefetch_l1(masks + (size_t) ((r + 1) * St::WORDS) * n + i);
            const int z = cz + dz, y = cy + dy;
            if (z < 0 || z >= Z || y < 0 || y >= Y) continue;
            const uint32_t row = sc.cell_base + (uint32_t) y * (uint32_t) X + (uint32_t) z * (uint32_t) X * (uint32_t) Y;
            const uint32_t jb = __ldg(start + row + xl), je = __ldg(start + row + xh + 1);
            if (!sph_check(jb <= je && je <= n, CHK_ROW)) continue;
            const uint32_t nw = (je - jb + 31) / 32;
            // the row's recorded words loaded together at the start of the row
            const uint32_t *mr = masks + (size_t) (r * St::WORDS) * n + i;
            uint32_t wr[St::WORDS];
#pragma unroll
            for (int k = 0; k < St::WORDS; k++) wr[k] = nw > (uint32_t) k ? __ldg(mr + k * (size_t) n) : 0u;
            for (uint32_t w = 0; w < nw; w++) {
                const uint32_t cb = jb + 32 * w;
                uint32_t m = 0;
                if (w < (uint32_t) St::WORDS) {
                    m = wr[0];
#pragma unroll
                    for (int k = 1; k < St::WORDS; k++) m = w == (uint32_t) k ? wr[k] : m;
                } else {  // beyond the recorded chunks: test the candidates here
                    const uint32_t ce = min(je, cb + 32u);
                    // 8 loads in flight where crowded windows are walked by a few warps: a fountain of 200,000
                    // 385 to 375 us; the short rows of cells of h/2 never come here, and keep their registers
#pragma unroll (RAD == 1 ? 8 : 4)
                    for (uint32_t j = ce; j-- > cb;) {
                        float x, yy, zz;
                        code_delta(gi, __ldg(gpos + j), x, yy, zz);
                        m = (m << 1) | (h2_minus_r2<float>(x, yy, zz, QH2) > 0.0f ? 1u : 0u);
                    }
                }
                if (i - cb < 32u) m &= ~(1u << (i - cb));  // the particle itself
                m = __brev(m);  // candidate k at bit 31 - k: the next one is the number of leading zeros
                while (m) {
                    const uint32_t k0 = (uint32_t) __clz((int) m), j0 = cb + k0;
                    m ^= 0x80000000u >> k0;
                    const bool two = m != 0;
                    const uint32_t k1 = two ? (uint32_t) __clz((int) m) : k0, j1 = cb + k1;
                    m &= ~(0x80000000u >> k1);
                    if (!sph_check(j0 < je && j1 < je, CHK_NEIGHBOUR)) continue;
                    const uint4 r0 = __ldg(rec + j0), r1 = __ldg(rec + j1);
                    mixed_pair(gi, vi, qs, r0, mc, fpx, fpy, fpz, fvx, fvy, fvz);
                    if (two) mixed_pair(gi, vi, qs, r1, mc, fpx, fpy, fpz, fvx, fvy, fvz);
                }
            }
        }
    }
    // the scene record again rather than kept live across the pair loop (fewer registers)
    const SceneDev sc2 = load_scene(scenes, wbits(pi.w));
    finish_mixed(i, pi, vi, ai.x, sc2, lo_s, obstacles, c, fpx, fpy, fpz, fvx, fvy, fvz, pos_out, lo_out, vel_out,
                 acc_out, cid_out, count);
}

// ---- group forms (sph_group.cuh): G lanes a particle, on cells of size h -----------------------
// The list holds h^2 - r^2 of the accepted neighbours, in order; the first entry of every 32-candidate
// word carries a negative sign (a word without neighbours has one entry, -0), since the words are
// summed one by one and added with Kahan compensation.
template <int G>
__global__ void __launch_bounds__(kGroupThreads) k_density_group_mixed(
    const Vec4<float> *__restrict__ pos, const uint2 *__restrict__ gpos, Vec4<float> *__restrict__ aux,
    const uint32_t *__restrict__ start, const SceneDev *__restrict__ scenes, uint32_t n, Consts<float> c, MixConsts mc,
    uint32_t *__restrict__ masks, const Vec4<float> *__restrict__ vel, uint4 *__restrict__ rec)
{
    __shared__ float list[kGroupThreads / 32][Group<G>::PER_WARP][kListLen];
    chain_wait();
    const Group<G> g;
    const uint32_t i = g.particle();
    if (i - (uint32_t) g.slot >= n) return;  // the whole warp
    const bool live = i < n;
    const uint32_t ic = live ? i : n - 1;
    const Vec4<float> pi = ld4(pos + ic);
    const uint2 gi = __ldg(gpos + ic);
    const SceneDev sc = load_scene(scenes, wbits(pi.w));
    int cx, cy, cz;
    hash_cell<float>(sc, pi.x, pi.y, pi.z, c, cx, cy, cz);
    const GroupRows<G> rows(g, sc, start, cx, cy, cz, live, n);
    float *const mine = list[g.warp][g.slot];
    float sum = 0, comp = 0, csum = 0;
    bool open = false;
    uint32_t cnt = 0;
    auto work_off = [&]() {
        __syncwarp();
        if (g.gl == 0) {
#pragma unroll 4
            for (uint32_t k = 0; k < cnt; k++) {
                const float v = mine[k];
                if (__float_as_int(v) < 0) {  // a word begins
                    if (open) kahan_add(sum, comp, csum);
                    csum = 0;
                    open = true;
                }
                csum = poly6_acc<float>(csum, fabsf(v));
            }
        }
        cnt = 0;
        __syncwarp();
    };
    rows.each([&](int r, uint32_t jb, uint32_t len, uint32_t most) {
        int w = 0;
        for (uint32_t cb = 0; cb < most; cb += 32, w++) {
            if (__any_sync(kFullWarp, cnt > kListFlush)) work_off();
            uint32_t m = 0;  // the word of these 32 candidates, as the other forms record it
            const uint32_t word = cnt;
#pragma unroll
            for (int u = 0; u < 32 / G; u++) {
                const uint32_t o = cb + (uint32_t) u * G + g.gl;
                if (cb + (uint32_t) u * G >= most) break;
                float t = 0;
                if (o < len) {
                    float x, y, z;
                    code_delta(gi, __ldg(gpos + jb + o), x, y, z);
                    t = h2_minus_r2<float>(x, y, z, QH2);
                }
                const unsigned hit = g.vote(t > 0);
                if (t > 0) {
                    const uint32_t k = cnt + (uint32_t) __popc(hit & g.below);
                    mine[k] = k == word ? -t : t;
                }
                cnt += __popc(hit);
                m |= hit << ((u * G) & 31);
            }
            if (m == 0 && cb < len) {
                if (g.gl == 0) mine[cnt] = -0.0f;
                cnt++;
            }
            if (g.gl == 0 && cb < len && w < Stencil<1>::WORDS)
                masks[(size_t) (r * Stencil<1>::WORDS + w) * n + i] = m;
        }
    });
    work_off();
    if (g.gl != 0 || !live) return;
    if (open) kahan_add(sum, comp, csum);
    const float rho = __fmul_rn(__fmul_rn(sum, mc.poly6_q), c.mass);
    const float p = __fmul_rn(c.k, __fsub_rn(rho, c.rho0));
    const float q = __fdiv_rn(p, __fmul_rn(rho, rho)), inv = __fdiv_rn(1.0f, rho);
    st4(aux + i, Vec4<float>{rho, p, q, inv});
    const Vec4<float> vi = ld4(vel + i);
    rec[i] = make_record(gi, vi.x, vi.y, vi.z, q, inv);
}

template <int G>
__global__ void __launch_bounds__(kGroupThreads) k_forces_group_mixed(
    const Vec4<float> *__restrict__ pos, const Vec4<float> *__restrict__ lo_s, const Vec4<float> *__restrict__ vel,
    const Vec4<float> *__restrict__ aux, const uint2 *__restrict__ gpos, const uint4 *__restrict__ rec,
    const uint32_t *__restrict__ start, const SceneDev *__restrict__ scenes, const ObstacleDev *__restrict__ obstacles,
    uint32_t n, Consts<float> c, MixConsts mc, const uint32_t *__restrict__ masks, Vec4<float> *__restrict__ pos_out,
    Vec4<float> *__restrict__ lo_out, Vec4<float> *__restrict__ vel_out, Vec4<float> *__restrict__ acc_out,
    uint2 *__restrict__ cid_out, uint32_t *__restrict__ count)
{
    constexpr int AHEAD = G <= 8 ? 16 / G : 1;
    constexpr int WORDS = Stencil<1>::WORDS;
    __shared__ uint32_t list[kGroupThreads / 32][Group<G>::PER_WARP][kListLen];
    __shared__ PairOut<float> outs[kGroupThreads / 32][Group<G>::PER_WARP][AHEAD * G];
    __shared__ GroupSums<float, G> sums;
    chain_wait();
    const Group<G> g;
    const uint32_t i = g.particle();
    const bool live = i < n;
    const uint32_t ic = live ? i : n - 1;
    const Vec4<float> pi = ld4(pos + ic);
    const Vec4<float> vi = ld4(vel + ic);
    const float qs = ld4(aux + ic).z * Q_SCALE;
    const uint2 gi = __ldg(gpos + ic);
    const SceneDev sc = load_scene(scenes, wbits(pi.w));
    int cx, cy, cz;
    hash_cell<float>(sc, pi.x, pi.y, pi.z, c, cx, cy, cz);
    const GroupRows<G> rows(g, sc, start, cx, cy, cz, live, n);
    uint32_t *const mine = list[g.warp][g.slot];
    PairOut<float> *const out = outs[g.warp][g.slot];
    float fp = 0, fv = 0;
    uint32_t cnt = 0;
    auto work_off = [&]() {
        __syncwarp();
        const uint32_t most = __reduce_max_sync(kFullWarp, cnt);
        for (uint32_t k0 = 0; k0 < most; k0 += AHEAD * G) {
            uint4 rj[AHEAD];
#pragma unroll
            for (int a = 0; a < AHEAD; a++) {
                const uint32_t k = k0 + (uint32_t) a * G + g.gl;
                rj[a] = __ldg(rec + (k < cnt ? mine[k] : ic));
            }
#pragma unroll
            for (int a = 0; a < AHEAD; a++) {
                PairOut<float> o;
                mixed_factors(gi, qs, rj[a], mc, o.v[0], o.v[2], o.v[4], o.v[1], o.v[3], o.v[5], o.v[6], o.v[7]);
                o.v[1] -= vi.x;
                o.v[3] -= vi.y;
                o.v[5] -= vi.z;
                float4 *dst = reinterpret_cast<float4 *>(out + a * G + g.gl);
                dst[0] = make_float4(o.v[0], o.v[1], o.v[2], o.v[3]);
                dst[1] = make_float4(o.v[4], o.v[5], o.v[6], o.v[7]);
            }
            __syncwarp();
            if (g.gl < 3 && k0 < cnt) add_pairs<float>(out, min(cnt - k0, (uint32_t) (AHEAD * G)), g.gl, fp, fv);
            __syncwarp();
        }
        cnt = 0;
    };
    rows.each([&](int r, uint32_t jb, uint32_t len, uint32_t most) {
        int w = 0;
        for (uint32_t cb = 0; cb < most; cb += 32, w++) {
            if (__any_sync(kFullWarp, cnt > kListFlush)) work_off();
            uint32_t m = 0;
            if (w < WORDS) {
                if (cb < len) m = __ldg(masks + (size_t) (r * WORDS + w) * n + ic);
            } else {  // beyond the recorded words: test the candidates here
#pragma unroll
                for (int u = 0; u < 32 / G; u++) {
                    const uint32_t o = cb + (uint32_t) u * G + g.gl;
                    float t = 0;
                    if (o < len) {
                        float x, y, z;
                        code_delta(gi, __ldg(gpos + jb + o), x, y, z);
                        t = h2_minus_r2<float>(x, y, z, QH2);
                    }
                    m |= g.vote(t > 0) << ((u * G) & 31);
                }
            }
            if (i - (jb + cb) < 32u) m &= ~(1u << (i - (jb + cb)));  // the particle itself
#pragma unroll
            for (int u = 0; u < 32 / G; u++) {
                const uint32_t bit = (uint32_t) u * G + g.gl;
                if (((m >> bit) & 1u) && sph_check(cb + bit < len, CHK_NEIGHBOUR))
                    mine[cnt + __popc(m & ((1u << bit) - 1u))] = jb + cb + bit;
            }
            cnt += __popc(m);
        }
    });
    work_off();
    sums.put(g, fp, fv);
    const uint32_t k = threadIdx.x, e = blockIdx.x * Group<G>::PER_BLOCK + k;
    if (k >= (uint32_t) Group<G>::PER_BLOCK || e >= n) return;
    const Vec4<float> pe = ld4(pos + e);
    finish_mixed(e, pe, ld4(vel + e), ld4(aux + e).x, load_scene(scenes, wbits(pe.w)), lo_s, obstacles, c, sums.f[k][0], sums.f[k][1],
                 sums.f[k][2], sums.f[k][3], sums.f[k][4], sums.f[k][5], pos_out, lo_out, vel_out, acc_out, cid_out,
                 count);
}

// ---- egress: id-ordered hi + lo positions (float or double), velocities, rho, p ---------
template <class T>
__global__ void __launch_bounds__(256) k_egress_mixed(const Vec4<float> *__restrict__ posL,
                                                      const Vec4<float> *__restrict__ loL,
                                                      const Vec4<float> *__restrict__ velL,
                                                      const Vec4<float> *__restrict__ posA,
                                                      const Vec4<float> *__restrict__ velA,
                                                      const Vec4<float> *__restrict__ aux,
                                                      const Vec4<float> *__restrict__ pos_u,
                                                      const Vec4<float> *__restrict__ vel_u,
                                                      const Vec4<float> *__restrict__ acc,
                                                      const uint32_t *__restrict__ scene_off, uint32_t n_state,
                                                      uint32_t n_aux, uint32_t n_acc, T *xyz, T *v, T *rho, T *p,
                                                      T *a)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n_state) {
        const Vec4<float> pp = ldc4(posL + i), ll = ldc4(loL + i), vv = ldc4(velL + i);
        const uint32_t o = __ldg(scene_off + wbits(pp.w)) + wbits(vv.w);
        xyz[3 * o] = (T) pp.x + (T) ll.x;
        xyz[3 * o + 1] = (T) pp.y + (T) ll.y;
        xyz[3 * o + 2] = (T) pp.z + (T) ll.z;
        v[3 * o] = vv.x; v[3 * o + 1] = vv.y; v[3 * o + 2] = vv.z;
    }
    // particles without a density (or an acceleration) yet, appended since, have 0 there
    if (rho && i < n_state) {
        const Vec4<float> pp = ldc4(posA + i), vv = ldc4(velA + i);
        const uint32_t o = __ldg(scene_off + wbits(pp.w)) + wbits(vv.w);
        if (!sph_check(o < n_state, CHK_EGRESS)) return;
        T r = 0, q = 0;
        if (i < n_aux) {
            const Vec4<float> ax = ldc4(aux + i);
            r = ax.x;
            q = ax.y;
        }
        rho[o] = r;
        p[o] = q;
    }
    if (acc && i < n_state) {
        const Vec4<float> pp = ldc4(pos_u + i), vv = ldc4(vel_u + i);
        const uint32_t o = __ldg(scene_off + wbits(pp.w)) + wbits(vv.w);
        if (!sph_check(o < n_state, CHK_EGRESS)) return;
        Vec4<float> aa = {0, 0, 0, 0};
        if (i < n_acc) aa = ldc4(acc + i);
        a[3 * o] = aa.x; a[3 * o + 1] = aa.y; a[3 * o + 2] = aa.z;
    }
}

// ---- launchers ----------------------------------------------------------------------------
static inline unsigned nblk(uint32_t n, unsigned t) { return (unsigned) ((n + t - 1) / t); }

cudaError_t mixed_grid(const DevBufs &b, uint32_t n, uint32_t ncells, Consts<float> c, MixConsts mc, cudaStream_t st)
{
    const PlaceMixed place = {(const Vec4<float> *) b.pos_u, (const Vec4<float> *) b.lo_u,
                              (const Vec4<float> *) b.vel_u, b.scenes, c.h, c.inv_h_f, mc.to_units,
                              (Vec4<float> *) b.pos_s, (Vec4<float> *) b.lo_s, (Vec4<float> *) b.vel_s, b.gpos,
                              {}, {}, {}};
    if (grid_small(n, ncells)) return launch_grid_small(place, b, n, ncells, st);
    cudaError_t e = Launch<float>::scan(b, ncells, st);
    if (e == cudaSuccess) e = launch_slot(b, n, st);
    if (e != cudaSuccess || !n) return e;
    return launch_chained(k_rank_permute_mixed, nblk(n, 256), 256, st, place, b.cid_u, n, b.start, b.tmp, b.bsum,
                          ncells / kScanTile + 1);
}

// Where the group forms are used: as for the plain form (group_density). Density and forces together, in
// us, with 16 lanes, 8 lanes and one thread a particle: 2,000 at rest 25 / 27 / 41, 8,000 fallen 35 / 39 /
// 70, 20,000 fallen 59 / 49 / 80, 40,000 fallen 94 / 82 / 84, 61,000 at rest 94 / 70 / 47.
template <int G>
static cudaError_t mixed_density_g(const DevBufs &b, uint32_t n, Consts<float> c, MixConsts mc, cudaStream_t st)
{
    return launch_chained(k_density_group_mixed<G>, nblk(n, Group<G>::PER_BLOCK), kGroupThreads, st,
                          (const Vec4<float> *) b.pos_s, b.gpos, (Vec4<float> *) b.aux, b.start, b.scenes, n, c, mc,
                          b.masks, (const Vec4<float> *) b.vel_s, (uint4 *) b.frec);
}

template <int G>
static cudaError_t mixed_forces_g(const DevBufs &b, uint32_t n, Consts<float> c, MixConsts mc, bool record_acc,
                                  cudaStream_t st)
{
    return launch_chained(
        k_forces_group_mixed<G>, nblk(n, Group<G>::PER_BLOCK), kGroupThreads, st, (const Vec4<float> *) b.pos_s,
        (const Vec4<float> *) b.lo_s, (const Vec4<float> *) b.vel_s, (const Vec4<float> *) b.aux, b.gpos,
        (const uint4 *) b.frec, b.start, b.scenes, b.obstacles, n, c, mc, b.masks, (Vec4<float> *) b.pos_u,
        (Vec4<float> *) b.lo_u, (Vec4<float> *) b.vel_u,
        record_acc ? (Vec4<float> *) b.acc : (Vec4<float> *) nullptr, b.cid_u, b.count);
}

cudaError_t mixed_density(const DevBufs &b, uint32_t n, Consts<float> c, MixConsts mc, int cell_mult,
                          cudaStream_t st)
{
    if (!n) return cudaSuccess;
    if (cell_mult == 1 && n <= kGroupMax)
        return n <= kGroupWide ? mixed_density_g<16>(b, n, c, mc, st) : mixed_density_g<8>(b, n, c, mc, st);
    // blocks of 128: the SMs finish the dense and sparse regions more evenly than with 256
    return launch_chained(cell_mult == 2 ? k_density_mixed<2> : k_density_mixed<1>, nblk(n, 128), 128, st,
                          (const Vec4<float> *) b.pos_s, b.gpos, (Vec4<float> *) b.aux, b.start, b.scenes, n, c, mc,
                          b.masks, (const Vec4<float> *) b.vel_s, (uint4 *) b.frec);
}

template <int MINB, int BLOCK, int RAD>
static cudaError_t launch_forces_mixed(const DevBufs &b, uint32_t n, Consts<float> c, MixConsts mc, bool record_acc,
                                       cudaStream_t st)
{
    return launch_chained(
        k_forces_mixed<MINB, BLOCK, RAD>, nblk(n, BLOCK), BLOCK, st, (const Vec4<float> *) b.pos_s,
        (const Vec4<float> *) b.lo_s, (const Vec4<float> *) b.vel_s, (const Vec4<float> *) b.aux, b.gpos,
        (const uint4 *) b.frec, b.start, b.scenes, b.obstacles, n, c, mc, b.masks, (Vec4<float> *) b.pos_u,
        (Vec4<float> *) b.lo_u, (Vec4<float> *) b.vel_u, record_acc ? (Vec4<float> *) b.acc : nullptr, b.cid_u,
        b.count);
}

template <int RAD>
static cudaError_t mixed_forces_rad(const DevBufs &b, uint32_t n, Consts<float> c, MixConsts mc, bool record_acc,
                                    int variant, cudaStream_t st)
{
    // variants: blocks of 128 threads at most 64 (0) or 48 (1) registers, blocks of 256 threads
    // with no cap (2) or at 48 registers (3); every variant computes the same bits
    switch (variant) {
    case 1: return launch_forces_mixed<10, 128, RAD>(b, n, c, mc, record_acc, st);
    case 2: return launch_forces_mixed<1, 256, RAD>(b, n, c, mc, record_acc, st);
    case 3: return launch_forces_mixed<5, 256, RAD>(b, n, c, mc, record_acc, st);
    // (0 on cells of h/2: as 1. Their shorter rows leave room for it: 4,000,000 fallen 1188 to 1161 us, 1,000,000
    // 311 to 307, at rest 164 to 162; on cells of h 326 to 334 us fallen, 150 to 145 at rest)
    default: return launch_forces_mixed<RAD == 2 ? 10 : 8, 128, RAD>(b, n, c, mc, record_acc, st);
    }
}

cudaError_t mixed_forces(const DevBufs &b, uint32_t n, Consts<float> c, MixConsts mc, bool record_acc, int variant,
                         int cell_mult, cudaStream_t st)
{
    if (!n) return cudaSuccess;
    if (cell_mult == 1 && variant == 0 && n <= kGroupMax)
        return n <= kGroupWide ? mixed_forces_g<16>(b, n, c, mc, record_acc, st)
                               : mixed_forces_g<8>(b, n, c, mc, record_acc, st);
    return cell_mult == 2 ? mixed_forces_rad<2>(b, n, c, mc, record_acc, variant, st)
                          : mixed_forces_rad<1>(b, n, c, mc, record_acc, variant, st);
}

cudaError_t mixed_egress(const DevBufs &b, uint32_t n_state, uint32_t n_aux, uint32_t n_acc, int layout_sorted,
                         int aux_sorted, bool f64, cudaStream_t st)
{
    if (!n_state) return cudaSuccess;
    const Vec4<float> *posL = (const Vec4<float> *) (layout_sorted ? b.pos_s : b.pos_u);
    const Vec4<float> *loL = (const Vec4<float> *) (layout_sorted ? b.lo_s : b.lo_u);
    const Vec4<float> *velL = (const Vec4<float> *) (layout_sorted ? b.vel_s : b.vel_u);
    const Vec4<float> *posA = (const Vec4<float> *) (aux_sorted ? b.pos_s : b.pos_u);
    const Vec4<float> *velA = (const Vec4<float> *) (aux_sorted ? b.vel_s : b.vel_u);
    const Vec4<float> *acc = (const Vec4<float> *) b.acc;
    if (f64)
        return launch_first(k_egress_mixed<double>, nblk(n_state, 256), 256, st, posL, loL, velL, posA, velA,
                            (const Vec4<float> *) b.aux, (const Vec4<float> *) b.pos_u, (const Vec4<float> *) b.vel_u,
                            b.st_acc64 ? acc : nullptr, b.scene_off, n_state, n_aux, n_acc, b.st_xyz64, b.st_vel64,
                            b.st_rho64, b.st_p64, b.st_acc64);
    return launch_first(k_egress_mixed<float>, nblk(n_state, 256), 256, st, posL, loL, velL, posA, velA,
                        (const Vec4<float> *) b.aux, (const Vec4<float> *) b.pos_u, (const Vec4<float> *) b.vel_u,
                        b.st_acc ? acc : nullptr, b.scene_off, n_state, n_aux, n_acc, b.st_xyz, b.st_vel, b.st_rho,
                        b.st_p, b.st_acc);
}

SPH_CHECK_ACCESSOR(check_flags_mixed)

}  // namespace sph
