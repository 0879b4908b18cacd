// sph_group.cu -- group forms of the neighbour passes (see sph_group.cuh): plain FP32 and FP64, on
// the reference's grid (cells of size h).
#include <cuda_runtime.h>
#include <stdint.h>

#include "sph_device.cuh"
#include "sph_group.cuh"
#include "sph_internal.h"

namespace sph {

// ---- plain FP32 ------------------------------------------------------------------------------
// Bound by the latency of a particle's walk (20 cycles an instruction at one warp a scheduler): 18.4 us
// with one thread a particle, 14.3 us with 8 or 16 lanes, for 8,000 particles at rest; fallen 28.7 and
// 14.3 us. Writes what the mask form writes: the words of accepted candidates and the force records.
template <int G>
__global__ void __launch_bounds__(kGroupThreads) k_density_group(
    const Vec4<float> *__restrict__ pos, const Vec4<float> *__restrict__ vel, Vec4<float> *__restrict__ aux,
    const uint32_t *__restrict__ start, const SceneDev *__restrict__ scenes, uint32_t n, Consts<float> c,
    uint32_t *__restrict__ masks, Vec4<float> *__restrict__ frec)
{
    __shared__ float list[kGroupThreads / 32][Group<G>::PER_WARP][kListLen];
    chain_wait();
    const Group<G> g;
    const uint32_t i = g.particle();
    if (i - (uint32_t) g.slot >= n) return;  // the whole warp
    const bool live = i < n;
    const Vec4<float> pi = ld4(pos + (live ? i : n - 1));
    const SceneDev sc = load_scene(scenes, wbits(pi.w));
    int cx, cy, cz;
    hash_cell<float>(sc, pi.x, pi.y, pi.z, c, cx, cy, cz);
    const GroupRows<G> rows(g, sc, start, cx, cy, cz, live, n);
    float *const mine = list[g.warp][g.slot];
    float acc = 0;
    uint32_t cnt = 0;
    // h^2 - r^2 of the listed neighbours, cubed and summed in order by the group's first lane
    auto work_off = [&]() {
        __syncwarp();
        if (g.gl == 0) {
#pragma unroll 4
            for (uint32_t k = 0; k < cnt; k++) acc = poly6_acc<float>(acc, mine[k]);
        }
        cnt = 0;
        __syncwarp();
    };
    rows.each([&](int r, uint32_t jb, uint32_t len, uint32_t most) {
        int w = 0;
        for (uint32_t cb = 0; cb < most; cb += 32, w++) {
            if (__any_sync(kFullWarp, cnt > kListFlush)) work_off();
            uint32_t m = 0;  // the word of these 32 candidates, as the other forms record it
#pragma unroll
            for (int u = 0; u < 32 / G; u++) {
                const uint32_t o = cb + (uint32_t) u * G + g.gl;
                if (cb + (uint32_t) u * G >= most) break;
                float t = 0;
                if (o < len) {
                    const Vec4<float> pj = ld4(pos + jb + o);
                    t = h2_minus_r2<float>(pi.x - pj.x, pi.y - pj.y, pi.z - pj.z, c.h2);
                }
                const unsigned hit = g.vote(t > 0);
                if (t > 0) mine[cnt + __popc(hit & g.below)] = t;
                cnt += __popc(hit);
                m |= hit << ((u * G) & 31);
            }
            if (g.gl == 0 && cb < len && w < Stencil<1>::WORDS)
                masks[(size_t) (r * Stencil<1>::WORDS + w) * n + i] = m;
        }
    });
    work_off();
    if (g.gl != 0 || !live) return;
    const float rho = rmul(rmul(acc, c.c_poly6), c.mass);
    const float p = rmul(c.k, rsub(rho, c.rho0));
    const Vec4<float> ar = aux_record<float>(rho, p, c);
    st4(aux + i, ar);
    const Vec4<float> vi = ld4(vel + i);
    st4(frec + 2 * (size_t) i, Vec4<float>{pi.x, pi.y, pi.z, ar.z});
    st4(frec + 2 * (size_t) i + 1, Vec4<float>{vi.x, vi.y, vi.z, ar.w});
}

// The accepted neighbours (from the density pass's words) are listed in order, the factors of G or 16
// of them at a time computed by the group's lanes, and three lanes sum one axis each. 24.6 us with one
// thread a particle, 12.3 us with 16 lanes, for 8,000 particles at rest; fallen 49.2 and 16.4 us.
template <int G>
__global__ void __launch_bounds__(kGroupThreads) k_forces_group(
    const Vec4<float> *__restrict__ pos, const Vec4<float> *__restrict__ vel, const Vec4<float> *__restrict__ aux,
    const uint32_t *__restrict__ start, const SceneDev *__restrict__ scenes, const ObstacleDev *__restrict__ obstacles,
    uint32_t n, Consts<float> c, const uint32_t *__restrict__ masks, const Vec4<float> *__restrict__ frec,
    Vec4<float> *__restrict__ pos_out, Vec4<float> *__restrict__ vel_out, Vec4<float> *__restrict__ acc_out,
    uint2 *__restrict__ cid_out, uint32_t *__restrict__ count)
{
    constexpr int AHEAD = G <= 8 ? 16 / G : 1;  // a group works on AHEAD * G neighbours at a time
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
    const Vec4<float> ai = ld4(aux + ic);
    const SceneDev sc = load_scene(scenes, wbits(pi.w));
    int cx, cy, cz;
    hash_cell<float>(sc, pi.x, pi.y, pi.z, c, cx, cy, cz);
    const GroupRows<G> rows(g, sc, start, cx, cy, cz, live, n);
    // the first recorded word of row r in the lane that holds the row's bounds
    uint32_t first[Group<G>::NR];
#pragma unroll
    for (int k = 0; k < Group<G>::NR; k++)
        first[k] = rows.len[k] ? __ldg(masks + (size_t) ((k * G + (int) g.gl) * WORDS) * n + ic) : 0u;
    uint32_t *const mine = list[g.warp][g.slot];
    PairOut<float> *const out = outs[g.warp][g.slot];
    float fp = 0, fv = 0;
    uint32_t cnt = 0;
    auto work_off = [&]() {
        __syncwarp();
        const uint32_t most = __reduce_max_sync(kFullWarp, cnt);
        for (uint32_t k0 = 0; k0 < most; k0 += AHEAD * G) {
            Vec4<float> pj[AHEAD], vj[AHEAD];
#pragma unroll
            for (int a = 0; a < AHEAD; a++) {
                const uint32_t k = k0 + (uint32_t) a * G + g.gl;
                const uint32_t j = k < cnt ? mine[k] : ic;
                pj[a] = ld4(frec + 2 * (size_t) j);
                vj[a] = ld4(frec + 2 * (size_t) j + 1);
            }
#pragma unroll
            for (int a = 0; a < AHEAD; a++) {
                PairOut<float> o;
                pair_factors<float>(pi, ai.z, pj[a], pj[a].w, vj[a].w, c, o.v[0], o.v[2], o.v[4], o.v[6], o.v[7]);
                o.v[1] = rsub(vj[a].x, vi.x);
                o.v[3] = rsub(vj[a].y, vi.y);
                o.v[5] = rsub(vj[a].z, vi.z);
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
        uint32_t w0 = 0;
#pragma unroll
        for (int k = 0; k < Group<G>::NR; k++)
            if (r / G == k) w0 = __shfl_sync(kFullWarp, first[k], r % G, G);
        int w = 0;
        for (uint32_t cb = 0; cb < most; cb += 32, w++) {
            if (__any_sync(kFullWarp, cnt > kListFlush)) work_off();
            uint32_t m = w == 0 ? w0 : 0u;
            if (w > 0 && w < WORDS) {
                if (cb < len) m = __ldg(masks + (size_t) (r * WORDS + w) * n + ic);
            } else if (w >= WORDS) {  // beyond the recorded words: test the candidates here
#pragma unroll
                for (int u = 0; u < 32 / G; u++) {
                    const uint32_t o = cb + (uint32_t) u * G + g.gl;
                    float t = 0;
                    if (o < len) {
                        const Vec4<float> pj = ld4(pos + jb + o);
                        t = h2_minus_r2<float>(pi.x - pj.x, pi.y - pj.y, pi.z - pj.z, c.h2);
                    }
                    m |= g.vote(t > 0) << ((u * G) & 31);
                }
            }
            if (i - (jb + cb) < 32u) m &= ~(1u << (i - (jb + cb)));  // the particle itself
#pragma unroll
            for (int u = 0; u < 32 / G; u++) {
                const uint32_t bit = (uint32_t) u * G + g.gl;
                const uint32_t j = jb + cb + bit;
                if (((m >> bit) & 1u) && sph_check(cb + bit < len, CHK_NEIGHBOUR))
                    mine[cnt + __popc(m & ((1u << bit) - 1u))] = j;
            }
            cnt += __popc(m);
        }
    });
    work_off();
    sums.put(g, fp, fv);
    const uint32_t k = threadIdx.x, e = blockIdx.x * Group<G>::PER_BLOCK + k;
    if (k >= (uint32_t) Group<G>::PER_BLOCK || e >= n) return;
    const Vec4<float> pe = ld4(pos + e);
    finish_particle<float>(e, pe, ld4(vel + e), ld4(aux + e).x, load_scene(scenes, wbits(pe.w)), obstacles, c,
                           sums.f[k][0], sums.f[k][1], sums.f[k][2], sums.f[k][3], sums.f[k][4], sums.f[k][5], pos_out,
                           vel_out, acc_out, cid_out, count);
}

// ---- FP64 --------------------------------------------------------------------------------------
// An SM has few FP64 lanes, so FP64 work is the bound, and most of it went into candidates farther
// than h: about 9 of 10 on cells of size h. Candidates are first tested in FP32 against a threshold
// that no accepted pair exceeds (below); what passes is listed and tested exactly, in FP64, by full
// groups. A rejected candidate adds an exact 0 to every sum, so leaving it out keeps the bits.
//
// The thresholds: with u = 2^-24, X the largest |coordinate| of the particle plus h and r about h,
// rounding both positions to float moves each component of the difference by at most 2.1 u X, so the
// float r^2 of a pair at distance h lies within 4u h^2 + 7.4 u h X + 13.3 u^2 X^2 of h^2, farther pairs'
// above and nearer pairs' below that. Each coefficient of the margin is more than twice that: a pair
// beyond it is rejected, a pair inside it accepted, and only the few within it need the exact test. A
// NaN or an infinity anywhere goes to the exact test. Where h^2 is so small that the squares are denormal, the
// roundings are absolute, at most 2^-150 each: the last term of the margin, 2^-145, is more than three times the ten
// of them in r^2, h^2 and the margin itself.
struct FloatTest {
    float x, y, z, limit, sure;
    __device__ __forceinline__ FloatTest(const Vec4<double> &p, const Consts<double> &c)
        : x((float) p.x), y((float) p.y), z((float) p.z)
    {
        constexpr float u = 5.9604645e-8f;
        const float h = c.h_f, X = fmaxf(fabsf(x), fmaxf(fabsf(y), fabsf(z))) + h;
        const float margin = 32.0f * u * h * (h + X) + 128.0f * (u * X) * (u * X) + 2.2420775e-44f;
        limit = h * h + margin;
        sure = h * h - margin;
        if (!(X < 3.0e38f)) limit = sure = __int_as_float(0x7fffffff);  // NaN: every candidate to the exact test
    }
    __device__ __forceinline__ float r2(const float *__restrict__ posf, uint32_t j) const
    {
        const float dx = x - __ldg(posf + 3 * (size_t) j), dy = y - __ldg(posf + 3 * (size_t) j + 1),
                    dz = z - __ldg(posf + 3 * (size_t) j + 2);
        return fmaf(dz, dz, fmaf(dy, dy, dx * dx));
    }
};
constexpr uint32_t kSure = 0x80000000u;  // flag of a listed index whose pair needs no exact test

// the candidates that may be within h, appended to the group's list (all but `self`); full() works the list off
template <int G, class F>
__device__ __forceinline__ void list_near(const Group<G> &g, const GroupRows<G> &rows, const FloatTest &ft,
                                          const float *__restrict__ posf, uint32_t self, uint32_t *mine, uint32_t &cnt,
                                          F &&full)
{
    rows.each([&](int, uint32_t jb, uint32_t len, uint32_t most) {
        for (uint32_t cb = 0; cb < most; cb += 32) {
            if (__any_sync(kFullWarp, cnt > kListFlush)) full();
#pragma unroll
            for (int u = 0; u < 32 / G; u++) {
                const uint32_t o = cb + (uint32_t) u * G + g.gl, j = jb + o;
                if (cb + (uint32_t) u * G >= most) break;
                float r2 = 0;
                if (o < len) r2 = ft.r2(posf, j);
                const bool in = o < len && !(r2 > ft.limit) && j != self;
                const unsigned hit = g.vote(in);
                if (in) mine[cnt + __popc(hit & g.below)] = j | (r2 < ft.sure ? kSure : 0u);
                cnt += __popc(hit);
            }
        }
    });
    full();
}

// 654 us in the mask form, 104 us here for 50,000 fallen particles (4 lanes a particle).
template <int G>
__global__ void __launch_bounds__(kGroupThreads) k_density_group64(
    const Vec4<double> *__restrict__ pos, const float *__restrict__ posf, Vec4<double> *__restrict__ aux,
    const uint32_t *__restrict__ start, const SceneDev *__restrict__ scenes, uint32_t n, Consts<double> c)
{
    constexpr int AHEAD = G <= 8 ? 16 / G : 1;
    __shared__ uint32_t list[kGroupThreads / 32][Group<G>::PER_WARP][kListLen];
    __shared__ double2 terms[kGroupThreads / 32][Group<G>::PER_WARP][AHEAD * G];
    chain_wait();
    const Group<G> g;
    const uint32_t i = g.particle();
    if (i - (uint32_t) g.slot >= n) return;  // the whole warp
    const bool live = i < n;
    const Vec4<double> pi = ld4(pos + (live ? i : n - 1));
    const SceneDev sc = load_scene(scenes, wbits(pi.w));
    int cx, cy, cz;
    hash_cell<double>(sc, pi.x, pi.y, pi.z, c, cx, cy, cz);
    const GroupRows<G> rows(g, sc, start, cx, cy, cz, live, n);
    uint32_t *const mine = list[g.warp][g.slot];
    double2 *const out = terms[g.warp][g.slot];
    double acc = 0;
    uint32_t cnt = 0;
    list_near<G>(g, rows, FloatTest(pi, c), posf, 0xffffffffu, mine, cnt, [&]() {
        __syncwarp();
        const uint32_t most = __reduce_max_sync(kFullWarp, cnt);
        for (uint32_t k0 = 0; k0 < most; k0 += AHEAD * G) {
#pragma unroll
            for (int a = 0; a < AHEAD; a++) {
                const uint32_t k = k0 + (uint32_t) a * G + g.gl;
                if (k < cnt) {
                    const Vec4<double> pj = ld4(pos + (mine[k] & ~kSure));
                    double t = h2_minus_r2<double>(pi.x - pj.x, pi.y - pj.y, pi.z - pj.z, c.h2);
                    t = t > 0 ? t : 0;
                    out[a * G + g.gl] = make_double2(rmul(t, t), t);
                }
            }
            __syncwarp();
            if (g.gl == 0 && k0 < cnt) {
                const uint32_t e = min(cnt - k0, (uint32_t) (AHEAD * G));
#pragma unroll 4
                for (uint32_t s = 0; s < e; s++) acc = rfma(out[s].x, out[s].y, acc);
            }
            __syncwarp();
        }
        cnt = 0;
    });
    if (g.gl != 0 || !live) return;
    const double rho = rmul(rmul(acc, c.c_poly6), c.mass);
    st4(aux + i, aux_record<double>(rho, rmul(c.k, rsub(rho, c.rho0)), c));
}

// Bound by the FP64 pipe: about 22 FP64 instructions a pair, a third of them the reciprocal root, and 2 to sum
// it. 50,000 fallen particles: 887 us in the mask form, 272 us here with a square root and a division (365 with
// its epilogue on one lane of each group instead of a full warp and every FP64 cell by division), 225 us with
// the reciprocal root.
template <int G>
__global__ void __launch_bounds__(kGroupThreads) k_forces_group64(
    const Vec4<double> *__restrict__ pos, const float *__restrict__ posf, const Vec4<double> *__restrict__ vel,
    const Vec4<double> *__restrict__ aux, const uint32_t *__restrict__ start, const SceneDev *__restrict__ scenes,
    const ObstacleDev *__restrict__ obstacles, uint32_t n, Consts<double> c, Vec4<double> *__restrict__ pos_out,
    Vec4<double> *__restrict__ vel_out, Vec4<double> *__restrict__ acc_out, uint2 *__restrict__ cid_out,
    uint32_t *__restrict__ count)
{
    __shared__ uint32_t list[kGroupThreads / 32][Group<G>::PER_WARP][kListLen];
    __shared__ PairOut<double> outs[kGroupThreads / 32][Group<G>::PER_WARP][G];
    __shared__ GroupSums<double, G> sums;
    chain_wait();
    const Group<G> g;
    const uint32_t i = g.particle();
    const bool live = i < n;
    const uint32_t ic = live ? i : n - 1;
    const Vec4<double> pi = ld4(pos + ic), vi = ld4(vel + ic), ai = ld4(aux + ic);
    const SceneDev sc = load_scene(scenes, wbits(pi.w));
    int cx, cy, cz;
    hash_cell<double>(sc, pi.x, pi.y, pi.z, c, cx, cy, cz);
    const GroupRows<G> rows(g, sc, start, cx, cy, cz, live, n);
    uint32_t *const mine = list[g.warp][g.slot];
    PairOut<double> *const out = outs[g.warp][g.slot];
    double fp = 0, fv = 0;
    uint32_t cnt = 0;
    list_near<G>(g, rows, FloatTest(pi, c), posf, i, mine, cnt, [&]() {
        __syncwarp();
        const uint32_t most = __reduce_max_sync(kFullWarp, cnt);
        for (uint32_t k0 = 0; k0 < most; k0 += G) {
            const uint32_t k = k0 + g.gl;
            if (k < cnt) {
                const uint32_t l = mine[k], j = l & ~kSure;
                const Vec4<double> pj = ld4(pos + j);
                PairOut<double> o;
                if (l != j || h2_minus_r2<double>(pi.x - pj.x, pi.y - pj.y, pi.z - pj.z, c.h2) > 0) {
                    const Vec4<double> vj = ld4(vel + j);
                    double qj, invj;
                    ld_qinv(aux + j, qj, invj);
                    pair_factors<double>(pi, ai.z, pj, qj, invj, c, o.v[0], o.v[2], o.v[4], o.v[6], o.v[7]);
                    o.v[1] = rsub(vj.x, vi.x);
                    o.v[3] = rsub(vj.y, vi.y);
                    o.v[5] = rsub(vj.z, vi.z);
                } else {  // adds exact zeros
#pragma unroll
                    for (int e = 0; e < 8; e++) o.v[e] = 0;
                }
                double2 *dst = reinterpret_cast<double2 *>(out + g.gl);
#pragma unroll
                for (int e = 0; e < 4; e++) dst[e] = make_double2(o.v[2 * e], o.v[2 * e + 1]);
            }
            __syncwarp();
            if (g.gl < 3 && k0 < cnt) add_pairs<double>(out, min(cnt - k0, (uint32_t) G), g.gl, fp, fv);
            __syncwarp();
        }
        cnt = 0;
    });
    sums.put(g, fp, fv);
    const uint32_t k = threadIdx.x, e = blockIdx.x * Group<G>::PER_BLOCK + k;
    if (k >= (uint32_t) Group<G>::PER_BLOCK || e >= n) return;
    const Vec4<double> pe = ld4(pos + e);
    finish_particle<double>(e, pe, ld4(vel + e), ld4(aux + e).x, load_scene(scenes, wbits(pe.w)), obstacles, c,
                            sums.f[k][0], sums.f[k][1], sums.f[k][2], sums.f[k][3], sums.f[k][4], sums.f[k][5], pos_out,
                            vel_out, acc_out, cid_out, count);
}

static inline unsigned nblk(uint32_t n, unsigned t) { return (unsigned) ((n + t - 1) / t); }

template <int G>
static cudaError_t density_g(const DevBufs &b, uint32_t n, Consts<float> c, cudaStream_t st)
{
    return launch_chained(k_density_group<G>, nblk(n, Group<G>::PER_BLOCK), kGroupThreads, st,
                          (const Vec4<float> *) b.pos_s, (const Vec4<float> *) b.vel_s, (Vec4<float> *) b.aux, b.start,
                          b.scenes, n, c, b.masks, (Vec4<float> *) b.frec);
}
template <int G>
static cudaError_t forces_g(const DevBufs &b, uint32_t n, Consts<float> c, bool record_acc, cudaStream_t st)
{
    return launch_chained(k_forces_group<G>, nblk(n, Group<G>::PER_BLOCK), kGroupThreads, st,
                          (const Vec4<float> *) b.pos_s, (const Vec4<float> *) b.vel_s, (const Vec4<float> *) b.aux,
                          b.start, b.scenes, b.obstacles, n, c, b.masks, (const Vec4<float> *) b.frec,
                          (Vec4<float> *) b.pos_u, (Vec4<float> *) b.vel_u,
                          record_acc ? (Vec4<float> *) b.acc : (Vec4<float> *) nullptr, b.cid_u, b.count);
}

// Lanes a particle, from the particle count: 16 up to kGroupWide particles, 8 up to kGroupMax, and one
// thread a particle beyond. Times of the density and force passes together, in us, with 16 lanes, 8
// lanes and one thread a particle: 8,000 at rest 27 / 27 / 43, fallen 29 / 35 / 78; 20,000 fallen
// 53 / 47 / 92; 40,000 at rest 62 / 51 / 45, fallen 82 / 78 / 98; 61,000 fallen 117 / 100 / 86. More
// lanes shorten a particle's serial walk, but the compaction makes the instructions per candidate
// about 1.5 times as many, which is what counts once the warps fill the GPU. (4 lanes gain nothing
// anywhere, and 32 only a few us below 2,000 particles.)
cudaError_t group_density(const DevBufs &b, uint32_t n, Consts<float> c, cudaStream_t st)
{
    return n <= kGroupWide ? density_g<16>(b, n, c, st) : density_g<8>(b, n, c, st);
}

cudaError_t group_forces(const DevBufs &b, uint32_t n, Consts<float> c, bool record_acc, cudaStream_t st)
{
    return n <= kGroupWide ? forces_g<16>(b, n, c, record_acc, st) : forces_g<8>(b, n, c, record_acc, st);
}

template <int G>
static cudaError_t density_g64(const DevBufs &b, uint32_t n, Consts<double> c, cudaStream_t st)
{
    return launch_chained(k_density_group64<G>, nblk(n, Group<G>::PER_BLOCK), kGroupThreads, st,
                          (const Vec4<double> *) b.pos_s, b.st_xyz, (Vec4<double> *) b.aux, b.start, b.scenes, n, c);
}
template <int G>
static cudaError_t forces_g64(const DevBufs &b, uint32_t n, Consts<double> c, bool record_acc, cudaStream_t st)
{
    return launch_chained(k_forces_group64<G>, nblk(n, Group<G>::PER_BLOCK), kGroupThreads, st,
                          (const Vec4<double> *) b.pos_s, b.st_xyz, (const Vec4<double> *) b.vel_s,
                          (const Vec4<double> *) b.aux, b.start, b.scenes, b.obstacles, n, c, (Vec4<double> *) b.pos_u,
                          (Vec4<double> *) b.vel_u, record_acc ? (Vec4<double> *) b.acc : (Vec4<double> *) nullptr,
                          b.cid_u, b.count);
}
// FP64: the group form at every size. An FP64 instruction costs the same with one lane active as with
// 32, and the ordered sums keep 3 lanes of a group busy, so fewer lanes a particle are better once the
// GPU is full: 8 up to kGroup64Wide particles, 4 beyond. Density and force passes together, in us, with
// 8 lanes, 4 lanes and one thread a particle (the mask form): 2,000 at rest 45 / 64 / 307, 8,000 fallen
// 94 / 107 / 610, 50,000 fallen 434 / 377 / 1541, 120,000 at rest 625 / 451 / 1094.
constexpr uint32_t kGroup64Wide = 16384;

cudaError_t group_density(const DevBufs &b, uint32_t n, Consts<double> c, cudaStream_t st)
{
    return n <= kGroup64Wide ? density_g64<8>(b, n, c, st) : density_g64<4>(b, n, c, st);
}

cudaError_t group_forces(const DevBufs &b, uint32_t n, Consts<double> c, bool record_acc, cudaStream_t st)
{
    return n <= kGroup64Wide ? forces_g64<8>(b, n, c, record_acc, st) : forces_g64<4>(b, n, c, record_acc, st);
}

SPH_CHECK_ACCESSOR(check_flags_group)

}  // namespace sph
