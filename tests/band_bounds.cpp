// band_bounds.cpp -- the FP32 bounds of the redistancing's band distances
// (simcoflow3d_gb300/csrc/transport_body.cuh) against the FP64 distance, on
// random interface cells.  Test infrastructure.
#include <cstring>
#include <random>

#include "transport_body.cuh"

// mode 0: random normals, distances inside the cell, spacings within a factor
// of four; 1: normals near an axis or a diagonal plane (the branch edges);
// 2: spacings at ratios up to 1:400 and scales 1e-9 to 1e9; 3: distances and
// normals outside what a reconstruction gives.
// out: pairs, pairs with bounds, violations, bounds wider than 0.1 of the scale
extern "C" void check_bounds(unsigned seed, long cells, int mode, long *out)
{
    std::mt19937_64 g(seed);
    std::uniform_real_distribution<double> U(-1.0, 1.0);
    out[0] = out[1] = out[2] = out[3] = 0;
    for (long s = 0; s < cells; ++s) {
        double n[3], d[3];
        for (double &v : n) v = U(g);
        if (mode == 1) {
            const int z = (int)(g() % 3);
            n[z] = (g() & 1) ? 0.0 : std::ldexp(U(g), -(int)(g() % 40));
            if (g() & 1) n[(z + 1) % 3] = n[(z + 2) % 3] * (1.0 + std::ldexp(U(g), -(int)(g() % 40)));
            if (g() % 5 == 0) n[(z + 1) % 3] = 0.0;
        }
        const double r = std::sqrt(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]);
        if (!(r > 0.0)) continue;
        for (double &v : n) v /= r;
        for (double &v : d) v = mode == 1 && (seed & 1) ? 1.0 / 128 : std::exp((mode == 2 ? 3.0 : 0.7) * U(g));
        const double scale = mode == 2 ? std::pow(10.0, 9.0 * U(g)) : 1.0;
        for (double &v : d) v *= scale;
        double dis = 0.5 * (std::fabs(n[0]) * d[0] + std::fabs(n[1]) * d[1] + std::fabs(n[2]) * d[2]) * U(g);
        if (mode == 3) {
            dis *= 6.0 * U(g);
            for (double &v : n) v *= 1.0 + 0.2 * U(g);
        }
        const tr::BandSource B = tr::band_source((float)n[0], (float)n[1], (float)n[2], (float)dis, (float)d[0],
                                                 (float)d[1], (float)d[2]);
        tr::BandFace F[6];
        for (int f = 0; f < 6; ++f) F[f] = tr::band_face(B, f);
        for (int t = 0; t < tr::BAND_CELLS; ++t)
            for (int neg = 0; neg < 2; ++neg) {
                int ii, jj, kk;
                tr::band_offset(t, ii, jj, kk);
                float lo, hi;
                ++out[0];
                if (!tr::band_bounds(B, F, ii, jj, kk, neg, lo, hi)) continue;
                ++out[1];
                const double v = tr::band_distance(n[0], n[1], n[2], dis, ii, jj, kk, d[0], d[1], d[2], neg ? -1.0 : 1.0);
                if (!((double)lo <= v && v <= (double)hi)) ++out[2];
                if (hi - lo > 0.1f * B.h) ++out[3];
            }
    }
}

// Offsets whose foot point leaves the cell for which the one-face form of
// band_distance differs from the loop over all axes (any two NaN are alike).
extern "C" long compare_faces(unsigned seed, long cells, long *third)
{
    std::mt19937_64 g(seed);
    std::uniform_real_distribution<double> U(-1.0, 1.0);
    long bad = 0;
    *third = 0;
    for (long s = 0; s < cells; ++s) {
        double n[3] = {U(g), U(g), U(g)}, d[3];
        if (s % 4 == 1) n[g() % 3] = 0.0;
        if (s % 4 == 2) { n[1] = n[0]; if (g() & 1) n[2] = -n[0]; }
        const double r = std::sqrt(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]);
        for (double &v : n) v /= r;
        for (double &v : d) v = s % 4 && (g() & 1) ? 1.0 / 64 : std::exp(U(g));
        const double dis = 0.5 * U(g) * (std::fabs(n[0]) * d[0] + std::fabs(n[1]) * d[1] + std::fabs(n[2]) * d[2]);
        for (int t = 0; t < tr::BAND_CELLS; ++t) {
            int o[3];
            tr::band_offset(t, o[0], o[1], o[2]);
            double dv = 0.0, dij = n[0] * d[0] * o[0] + n[1] * d[1] * o[1] + n[2] * d[2] * o[2] + dis, p[3], w[3];
            bool inside = true;
            for (int q = 0; q < 3; ++q) {
                dv += n[q] * (d[q] * (o[q] < -1 ? -1 : o[q] > 1 ? 1 : o[q]) / 2.0);
                p[q] = d[q] * o[q] - dij * n[q];
                inside = inside && -0.5 * d[q] <= p[q] && p[q] <= 0.5 * d[q];
                w[q] = std::fmax(std::fabs(p[q]) - 0.5 * d[q], 0.0) * std::fabs(n[q]);
            }
            if (inside) continue;
            ++*third;
            const double side = dv + dis > 0.0 ? 1.0 : -1.0;   // not the facing boundary point's case
            const double a = tr::band_distance(n[0], n[1], n[2], dis, o[0], o[1], o[2], d[0], d[1], d[2], side);
            const double b = tr::band_ties_rare(n[0], n[1], n[2], dis, o[0], o[1], o[2], d[0], d[1], d[2], p[0], p[1],
                                                p[2], w[0], w[1], w[2]);
            if (dv + dis != 0.0 && memcmp(&a, &b, 8) != 0 && !(std::isnan(a) && std::isnan(b))) ++bad;
        }
    }
    return bad;
}
