// Host build of the block fixed point (block_fixed.cuh): the integer
// arithmetic of the double path's kernels, element by element, for
// test_fixed_point.py.
#include "block_fixed.cuh"

using namespace lulesh::bf;

extern "C" {

// Corner forces of n elements as the force kernel forms them: corner
// coordinates and velocities [n][axis][8], sc = 1 / (192 volo v), hourglass
// coefficient and p + q. fits[n][axis]: the axis does not need the double form.
void host_forces(int n, const double* x, const double* vel, const double* sc, const double* coef, const double* press,
                 double* out, int* fits) {
    for (int i = 0; i < n; ++i) {
        Sums s;
        ForceGeo g;
        ForceScale f;
        bool ok = axis_sums<57, false>(x + 24 * i, 0, s);
        ok &= axis_sums<57, false>(x + 24 * i + 8, 1, s);
        ok &= axis_sums<57, false>(x + 24 * i + 16, 2, s);
        ok &= force_geometry(s, g);
        ok &= force_scale(g, sc[i], coef[i], press[i], f);
        for (int a = 0; a < 3; ++a) {
            const int64_t col[3] = {g.n[0][a], g.n[1][a], g.n[2][a]};
            const bool fit = force_axis(g, f, col, g.unit[a], vel + 24 * i + 8 * a, out + 24 * i + 8 * a);
            fits[3 * i + a] = ok && fit;
        }
    }
}

}  // extern "C"
