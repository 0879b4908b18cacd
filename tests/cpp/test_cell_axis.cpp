// The FP64 form's cell of a coordinate (a float quotient first, the exact formula near a cell face)
// against the reference's formula alone: random coordinates, coordinates a few ulps from cell faces, far
// outside the box, and special values. Prints the number of differences.
#include <math.h>

#include <cmath>
#include <cstdio>
#include <random>

#include "sph_internal.h"

static int reference_cell(double p, float half, double h, int res)
{
    const double q = (p + (double) half) / h;
    if (!(q >= 0.0)) return 0;
    if (q >= (double) res) return res - 1;
    return (int) std::floor(q);
}

int main()
{
    std::mt19937_64 g(1);
    std::uniform_real_distribution<double> U(0, 1);
    long bad = 0;
    for (long it = 0; it < 3000000; it++) {
        const float h = it % 7 ? 0.0457f : (float) (0.001 + U(g));
        const float box = (float) (h * (1 + U(g) * (it % 5 ? 60 : 2000))), half = box / 2;
        const int res = (int) std::ceil(box / h);
        const double hd = (double) h, face = std::round((U(g) * 1.2 - 0.1) * res) * hd - (double) half;
        double p = 0;
        switch (it % 5) {
        case 0: p = (U(g) * 2.2 - 1.1) * half; break;
        case 1: p = face + (U(g) - 0.5) * std::pow(10.0, -15 + 10 * U(g)); break;
        case 2: p = (U(g) - 0.5) * std::pow(10.0, 6 + 30 * U(g)); break;
        case 3:
            p = face;
            for (int k = (int) (U(g) * 5); k > 0; k--) p = std::nextafter(p, it % 2 ? 1e300 : -1e300);
            break;
        default: p = half * (1 + (U(g) - 0.5) * 1e-6); break;
        }
        bad += sph::cell_axis(p, half, 1.0f / h, hd, res) != reference_cell(p, half, hd, res);
    }
    for (double p : {(double) NAN, (double) INFINITY, -(double) INFINITY, 1e300, -1e300, 0.0, -0.0, 5e-324})
        bad += sph::cell_axis(p, 0.5f, 1.0f / 0.0457f, (double) 0.0457f, 22) !=
               reference_cell(p, 0.5f, (double) 0.0457f, 22);
    std::printf("%ld\n", bad);
    return 0;
}
