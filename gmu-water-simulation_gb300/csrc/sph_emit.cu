// sph_emit.cu -- the disc emitter on the device: particle k of an emission step is generated
// by thread k with the generator shared with the host (sph_emit.h), into the staging arrays
// that the append path ingests. No host buffer and no host-to-device copy is involved.
#include "sph_emit.h"
#include "sph_internal.h"

namespace sph {

__global__ void k_emit_fountain(uint64_t seed, uint32_t step, uint32_t n, float cx, float cy, float cz, float radius,
                                float speed, float sigma, float *__restrict__ xyz, float *__restrict__ vel)
{
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    const float c[3] = {cx, cy, cz};
    float p[3], v[3];
    emit::particle(seed, step, k, c, radius, speed, sigma, p, v);  // by whole warps: its lanes meet inside
    if (k >= n) return;
    for (int a = 0; a < 3; a++) {
        xyz[3 * (size_t) k + a] = p[a];
        vel[3 * (size_t) k + a] = v[a];
    }
}

cudaError_t launch_emit_fountain(uint64_t seed, uint32_t step, uint32_t n, const float center[3], float radius,
                                 float speed, float sigma, float *xyz, float *vel, cudaStream_t st)
{
    if (n == 0) return cudaSuccess;
    // Bound by the latency of a serial chain of FP64 operations, and an SM has so few FP64 lanes that its
    // warps queue for them: one warp a block spreads 2,000 particles over 63 SMs instead of 16 (59 us in
    // blocks of 128, 55 us in blocks of 32, 21 us with the lanes meeting after each rejection loop).
    k_emit_fountain<<<(n + 31) / 32, 32, 0, st>>>(seed, step, n, center[0], center[1], center[2], radius, speed, sigma,
                                                  xyz, vel);
    return cudaGetLastError();
}

}  // namespace sph
