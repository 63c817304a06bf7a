// sweep_lines.cpp -- the sweeps with shared work (tr::line_face,
// tr::line_update) against the general sweep (tr::sweep_cell), bit for bit.
// Test infrastructure.
#define TR_HOST_CHECK 1
#include <cstring>
#include <random>
#include <vector>

#include "transport_body.cuh"

using tr::Dims;
using tr::Geo;

// kind of spacings: 0 a power of two, 1 uniform 1/n, 2 a new value in every
// cell, 3 repeating in pairs, 4 extreme exponents
static void fill_line(std::vector<double> &d, std::vector<double> &c, int n, int kind, std::mt19937_64 &g)
{
    std::uniform_real_distribution<double> U(0.5, 1.5);
    d.resize(n);
    c.resize(n);
    double x = 0.0;
    const double pair = U(g);
    for (int q = 0; q < n; ++q) {
        d[q] = kind == 0 ? 1.0 / 64 : kind == 1 ? 1.0 / n : kind == 2 ? U(g) / n : kind == 3 ? (q / 2 % 2 ? pair : 1.0) / n
                                                                                            : std::ldexp(U(g), -400);
        x += d[q];
        c[q] = x - 0.5 * d[q];
    }
}

// Returns the number of cells whose VOF or level set differs (bits; any two
// NaN are alike).  values: 0 ordinary, 1 with zeros of both signs, infinities
// and NaN among velocities and fields.
extern "C" long compare_lines(unsigned seed, int I, int J, int K, int axis, int stage, int kind, int values)
{
    std::mt19937_64 g(seed);
    std::uniform_real_distribution<double> U(-1.0, 1.0);
    const Dims D{I, J, K};
    const size_t nin = D.interior(), ng = D.ghosted();
    std::vector<double> geo[6], ln[3], cn[3];
    const int len[3] = {I, J, K};
    for (int a = 0; a < 3; ++a) fill_line(ln[a], cn[a], len[a], kind, g);
    for (auto &v : geo) v.resize(nin);
    for (int k = 1; k <= K; ++k)
        for (int j = 1; j <= J; ++j)
            for (int i = 1; i <= I; ++i) {
                const size_t c = D.n(i, j, k);
                geo[0][c] = cn[0][i - 1]; geo[1][c] = cn[1][j - 1]; geo[2][c] = cn[2][k - 1];
                geo[3][c] = ln[0][i - 1]; geo[4][c] = ln[1][j - 1]; geo[5][c] = ln[2][k - 1];
            }
    const Geo G{geo[0].data(), geo[1].data(), geo[2].data(), geo[3].data(), geo[4].data(), geo[5].data()};
    auto odd = [&](double v) {
        if (!values) return v;
        switch (g() % 24) {
        case 0: return 0.0;
        case 1: return -0.0;
        case 2: return (double)INFINITY;
        case 3: return (double)-INFINITY;
        case 4: return (double)NAN;
        case 5: return 5e-324;
        default: return v;
        }
    };
    std::vector<double> vfl(ng), phi(ng), vel(ng), vf1(ng), ls1(ng), flo(ng, NAN), fhi(ng, NAN);
    std::vector<double> nx(ng), ny(ng), nz(ng), dis(ng);
    for (size_t c = 0; c < ng; ++c) {
        const int r = (int)(g() % 8);
        vfl[c] = odd(r < 4 ? 0.0 : r < 6 ? 1.0 : 0.5 + 0.5 * U(g));
        vf1[c] = odd(g() % 3 == 0 ? vfl[c] : g() % 2 ? 1.0 : 0.0);
        phi[c] = odd(g() % 3 ? U(g) : 0.25);
        ls1[c] = odd(U(g));
        vel[c] = odd(g() % 6 ? U(g) : 0.0);
    }
    std::vector<double> bv(D.plane_size(axis)), bl(D.plane_size(axis));
    for (size_t c = 0; c < bv.size(); ++c) { bv[c] = odd(U(g)); bl[c] = odd(U(g)); }
    tr::SweepIn S{};
    S.vfl = vfl.data(); S.phi = phi.data(); S.nx = nx.data(); S.ny = ny.data(); S.nz = nz.data(); S.dis = dis.data();
    S.vel = vel.data(); S.bc_vel = bv.data(); S.bc_lvs = bl.data(); S.vf_first = vf1.data(); S.ls_first = ls1.data();
    S.dtv = 0.003 * std::ldexp(1.0, kind == 4 ? -400 : 0);
    S.axis = axis;
    S.stage = stage;
    for (int k = 1; k <= K; ++k)
        for (int j = 1; j <= J; ++j)
            for (int i = 1; i <= I; ++i) {
                const size_t c = D.g(i, j, k);
                tr::reconstruct(D, G, S.vfl, S.phi, i, j, k, nx[c], ny[c], nz[c], dis[c]);
                if (tr::partial_cell(vfl[c]))
                    tr::partial_fluxes(D, G, S, i, j, k, nx[c], ny[c], nz[c], dis[c], flo[c], fhi[c]);
            }
    const double *d = axis == 0 ? G.dx : axis == 1 ? G.dy : G.dz, *cc = axis == 0 ? G.x : axis == 1 ? G.y : G.z;
    const int n = D.len(axis), na = axis == 0 ? J : I, nb = axis == 2 ? J : K;
    long bad = 0;
    for (int b = 1; b <= nb; ++b)
        for (int a = 1; a <= na; ++a) {
            tr::LineFace lo{0.0, 0.0, 0.0, 0.0, 0.0};
            for (int m = 1; m <= n; ++m) {
                const tr::LineStep s = tr::line_step(d[tr::line_n(D, axis, m, a, b)], S.dtv);
                const tr::LineFace hi = tr::line_face(D, G, S, axis, s, d, cc, flo.data(), fhi.data(), m, a, b);
                const int i = axis == 0 ? m : a, j = axis == 0 ? a : axis == 1 ? m : b, k = axis == 2 ? m : b;
                double v[2], w[2];
                (stage ? tr::line_update<true> : tr::line_update<false>)(D, S, axis, s, lo, hi, m, a, b, v[0], v[1]);
                tr::sweep_cell(D, G, S, i, j, k, w[0], w[1]);
                for (int q = 0; q < 2; ++q)
                    if (memcmp(&v[q], &w[q], 8) != 0 && !(std::isnan(v[q]) && std::isnan(w[q]))) { ++bad; break; }
                lo = hi;
            }
        }
    return bad;
}

// Quotients of tr::line_div and tr::line_div2 that differ from the division.
extern "C" long compare_quotients(unsigned seed, long count)
{
    std::mt19937_64 g(seed);
    std::uniform_real_distribution<double> U(1.0, 2.0);
    long bad = 0;
    for (long t = 0; t < count; ++t) {
        double x = std::ldexp(U(g), (int)(g() % 80) - 40), d = std::ldexp(U(g), (int)(g() % 40) - 30);
        if (t % 4 == 0) x = tr::from_bits((tr::bits_of(x) & ~0xFFFFFull) | (g() % 3));        // few significant bits,
        if (t % 4 == 1) d = tr::from_bits(tr::bits_of(d) | 0xFFFFFFFFFFFF0ull | (g() & 15));   // nearly all ones
        if (t % 8 == 2) x = d * U(g);                                                         // near a representable quotient
        if (t % 16 == 5) x = std::ldexp(x, (int)(g() % 2000) - 1000);
        if (t % 16 == 9) d = std::ldexp(d, (int)(g() % 1900) - 950);
        if (g() & 1) x = -x;
        const tr::LineStep s = tr::line_step(d, 1.0);
        const double a = tr::line_div(s, x), b = x / d, c = tr::line_div2(s, x), e = x / (2.0 * d);
        if (memcmp(&a, &b, 8) || memcmp(&c, &e, 8)) ++bad;
    }
    return bad;
}

// Sums of squares around the ends of the gradient test's interval, and random
// ones, that it decides otherwise than |1 - sqrt(s)| < ETA.
extern "C" long compare_gradient_test(unsigned seed, long count)
{
    std::mt19937_64 g(seed);
    long bad = 0;
    for (long t = 0; t < count; ++t) {
        const double c = t & 1 ? tr::OFF_LO : tr::OFF_HI;
        double s = t % 4 < 2 ? tr::from_bits(tr::bits_of(c) + (uint64_t)(t / 4 % 4000) - 2000) : std::ldexp((double)g(), -63);
        if (t == 0) s = NAN;
        const double off = std::fabs(1.0 - std::sqrt(s));
        for (const double other : {1.0, 4.0, (double)NAN}) {
            const double o = std::fabs(1.0 - std::sqrt(other));
            const int want = (off < tr::ETA && o >= tr::ETA) ? -1 : (off >= tr::ETA && o < tr::ETA) ? 1 : 0;
            if (tr::side_of(s, other) != want || tr::side_of(other, s) != -want) ++bad;
        }
    }
    return bad;
}
