// Host build of the block fixed point (block_fixed.cuh, eos_fixed.cuh): the
// integer arithmetic of the double path's kernels, element by element, for
// test_fixed_point.py.
#include "eos_fixed.cuh"

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

// One EOS evaluation of n elements: in[k] = e, p, q, ql, qq, delv, v and
// out[k] = e, p, q, ss, each of n values; the cutoffs of e and q are 1e-7.
// fits[n]: the element does not need the double form.
void host_eos_above(int n, const double* in, double p_cut, double emin, double* out, int* fits) {
    const EosCuts cuts = eos_cuts(1e-7, p_cut, 1e-7, 0.0, emin, 1.0);
    auto at = [&](int k, int i) { return in[size_t(k) * n + i]; };
    for (int i = 0; i < n; ++i) {
        double* o = out + i;
        fits[i] = cuts.ok && eos_pass(at(0, i), at(1, i), at(2, i), at(3, i), at(4, i), at(5, i), at(6, i), cuts, o[0],
                                      o[n], o[2 * size_t(n)], o[3 * size_t(n)]);
        if (at(5, i) <= 0.0 && fabs(o[2 * size_t(n)]) < 1e-7) o[2 * size_t(n)] = 0.0;
    }
}

void host_eos(int n, const double* in, double p_cut, double* out, int* fits) {
    host_eos_above(n, in, p_cut, -1e15, out, fits);
}

// The viscosity sums of n elements: velocity gradients, those of the minus and
// plus neighbours and lengths [n][3], sums lin and quad. fits[n] as above.
void host_q_sums(int n, const double* dv, const double* dm, const double* dp, const double* dx, double* lin,
                 double* quad, int* fits) {
    for (int i = 0; i < n; ++i) fits[i] = q_sums(dv + 3 * i, dm + 3 * i, dp + 3 * i, dx + 3 * i, lin[i], quad[i]);
}

}  // extern "C"
