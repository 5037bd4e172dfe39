// sar_lattice.h -- pixel lattices whose second axis follows the iso-range lines of a collection (host-only): the
// order in which the linear-sampling kernels walk a grid (sar_scatter.cu, sar_gather.cu).
//
// Lattice pixel (a, b) is image pixel (i, j) = a v + b w with integer steps v, w and det(v, w) = +-1, so every
// image pixel is one lattice pixel.  Along w the range bin should change as little as possible; of the
// directions with |w|^2 <= 5 the one with the least cost is taken.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <vector>

namespace sar {

struct Lattice {
    int vx = 1, vy = 0, wx = 0, wy = 1;
    bool ok = false;
};

// Largest error (turns) of the phase of a 16 x 16 block about its anchor: the expansions stop at third order, and the
// fourth is at most d^4 / (8 R^3) an antenna, d the half-diagonal.
inline double expansion_turns(double len_a, double len_b, double nearest, double kappa) {
    const double d = 8.0 * (len_a + len_b);
    return nearest > 0.0 ? std::fabs(kappa) * d * d * d * d / (4.0 * nearest * nearest * nearest) : INFINITY;
}
// Taken as exact: adds 6e-7 of the result at most, in quadrature to 0.9e-6 of FP32 phases (at 1e-6 turns 1.7e-6 in all).
constexpr double kExpansionTurns = 2.5e-7;

// Bins per step along two axes, from one pulse at one point of the scene.
struct LatticeRate {
    double v, w;
};

// The rates along x and y at the centre of the scene and of its four quarters, from up to about 128 of the pulses, and a
// bound of the nearest antenna's distance from the scene.
struct SceneRates {
    std::vector<LatticeRate> xy;
    double nearest = INFINITY;
    bool ok = false;
};

inline double step_length(const double* ex, const double* ey, int a, int b) {
    double q = 0.0;
    for (int d = 0; d < 3; ++d) q += (a * ex[d] + b * ey[d]) * (a * ex[d] + b * ey[d]);
    return std::sqrt(q);
}

inline SceneRates scene_rates(const double* tx, const double* rx, size_t S, const double* origin, const double* ex,
                              const double* ey, const double* ez, int nx, int ny, int nz, double s_r) {
    SceneRates R;
    const double half = 0.5 * (nx * step_length(ex, ey, 1, 0) + ny * step_length(ex, ey, 0, 1) +
                               nz * std::sqrt(ez[0] * ez[0] + ez[1] * ez[1] + ez[2] * ez[2]));
    const double points[5][2] = {{0.5, 0.5}, {0.25, 0.25}, {0.25, 0.75}, {0.75, 0.25}, {0.75, 0.75}};
    const size_t every = std::max<size_t>(1, S / 128);
    for (size_t s = 0; s < S; ++s)
        for (int k = 0; k < (s % every ? 1 : 5); ++k) {
            const double fx = points[k][0] * (nx - 1), fy = points[k][1] * (ny - 1);
            LatticeRate g{0.0, 0.0};
            for (int ant = 0; ant < 2; ++ant) {
                const double* p = (ant ? rx : tx) + 3 * s;
                double w[3];
                for (int d = 0; d < 3; ++d) w[d] = origin[d] + fx * ex[d] + fy * ey[d] + 0.5 * (nz - 1) * ez[d] - p[d];
                const double r = std::sqrt(w[0] * w[0] + w[1] * w[1] + w[2] * w[2]);
                if (!(r > 0.0)) return R;
                if (k == 0) R.nearest = std::min(R.nearest, r - half);
                g.v += s_r * (w[0] * ex[0] + w[1] * ex[1] + w[2] * ex[2]) / r;
                g.w += s_r * (w[0] * ey[0] + w[1] * ey[1] + w[2] * ey[2]) / r;
            }
            if (!std::isfinite(g.v) || !std::isfinite(g.w)) return R;
            if (s % every == 0) R.xy.push_back(g);
        }
    R.ok = true;
    return R;
}

inline std::vector<LatticeRate> lattice_rates(const SceneRates& R, const Lattice& L) {
    std::vector<LatticeRate> q(R.xy.size());
    for (size_t i = 0; i < q.size(); ++i)
        q[i] = LatticeRate{std::fabs(L.vx * R.xy[i].v + L.vy * R.xy[i].w), std::fabs(L.wx * R.xy[i].v + L.wy * R.xy[i].w)};
    return q;
}

// Shared-memory bank pairs: the most distinct bins that a half-warp's accesses have on one of the sixteen, its lanes `rate`
// bins apart; windows with a padding slot every 16 bins, or without.
inline double bank_degree(double rate, bool pad) {
    int hits[16] = {}, last = -1, most = 0;
    for (int l = 0; l < 16; ++l) {
        const int bin = (int)std::min(rate * l, 1.0e6);
        if (bin != last) most = std::max(most, ++hits[(pad ? bin + (bin >> 4) : bin) & 15]);
        last = bin;
    }
    return most;
}

// Lattices with longer steps than the image's are taken only where their larger blocks still expand exactly (coarse
// pixels at short range: 0.8 m at 2 km would go from 1.7e-5 to 3e-5 of the result).
// `seconds(lattice, rates)`: what the kernel is expected to take on a lattice with these rates.
template <class EST>
inline Lattice choose_lattice(const SceneRates& R, const double* ex, const double* ey, double kappa, EST seconds) {
    Lattice best;
    if (!R.ok) return best;
    const int cand[8][4] = {{0, 1, 1, 0}, {1, 0, 0, 1}, {1, 1, 1, 0}, {-1, 1, 1, 0},
                            {2, 1, 1, 0}, {-2, 1, 1, 0}, {1, 2, 0, 1}, {-1, 2, 0, 1}};   // w, v
    double least = INFINITY;
    for (int c = 0; c < 8; ++c) {
        const Lattice L{cand[c][2], cand[c][3], cand[c][0], cand[c][1], true};
        if (c >= 2 && !(expansion_turns(step_length(ex, ey, L.wx, L.wy), step_length(ex, ey, L.vx, L.vy), R.nearest, kappa) < kExpansionTurns))
            continue;
        const double t = seconds(L, lattice_rates(R, L));
        if (t < least || !best.ok) {
            least = t;
            best = L;
        }
    }
    return best;
}

// Bin excursion of a block about its anchor.  For a pixel at d from the anchor an antenna's range moves by at most
// |u.d| + |d|^2 / (2 R), u the unit vector at the anchor; u is taken at the centres of 4 x 4 cells of the scene,
// where it changes by at most Dc / R towards any anchor of the cell (Dc its half-diagonal and a block's).
struct LatticeBounds {
    double len_a = 0.0, len_b = 0.0, nearest = INFINITY;
    std::vector<double> ra, rb, rest;   // per pulse: largest |rate| along v and w (metres per step), largest Dc / R
    bool ok = false;

    // Largest excursion (bins) over pixels up to ha steps along v and hb along w from an anchor.
    double excursion(double ha, double hb, double s_r) const {
        const double reach = ha * len_a + hb * len_b;
        double h = 0.0;
        for (size_t s = 0; s < ra.size(); ++s)
            h = std::max(h, ha * ra[s] + hb * rb[s] + reach * rest[s] + reach * reach / nearest);
        return h * s_r;
    }
};

inline LatticeBounds lattice_bounds(const Lattice& L, const double* tx, const double* rx, size_t S, const double* origin,
                                    const double* ex, const double* ey, const double* ez, int nx, int ny, int nz,
                                    double most_a, double most_b) {
    LatticeBounds B;
    double ea[3], eb[3];
    for (int d = 0; d < 3; ++d) {
        ea[d] = L.vx * ex[d] + L.vy * ey[d];
        eb[d] = L.wx * ex[d] + L.wy * ey[d];
    }
    auto len = [](const double* v) { return std::sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]); };
    B.len_a = len(ea);
    B.len_b = len(eb);
    const double block = most_a * B.len_a + most_b * B.len_b;
    const double Dc = 0.125 * (nx * len(ex) + ny * len(ey)) + 0.5 * nz * len(ez) + 2.0 * block;
    B.ra.assign(S, 0.0);
    B.rb.assign(S, 0.0);
    B.rest.assign(S, 0.0);
    for (size_t s = 0; s < S; ++s)
        for (int cell = 0; cell < 16; ++cell) {
            const double fx = ((cell & 3) + 0.5) / 4.0 * (nx - 1), fy = ((cell >> 2) + 0.5) / 4.0 * (ny - 1);
            double a = 0.0, b = 0.0, q = 0.0;
            for (int ant = 0; ant < 2; ++ant) {
                const double* p = (ant ? rx : tx) + 3 * s;
                double u[3];
                for (int d = 0; d < 3; ++d)
                    u[d] = p[d] - (origin[d] + fx * ex[d] + fy * ey[d] + 0.5 * (nz - 1) * ez[d]);
                const double r = len(u), R = r - Dc;
                if (!(R > 0.0)) return B;
                B.nearest = std::min(B.nearest, R);
                a += std::fabs(u[0] * ea[0] + u[1] * ea[1] + u[2] * ea[2]) / r;
                b += std::fabs(u[0] * eb[0] + u[1] * eb[1] + u[2] * eb[2]) / r;
                q += Dc / R;
            }
            B.ra[s] = std::max(B.ra[s], a);
            B.rb[s] = std::max(B.rb[s], b);
            B.rest[s] = std::max(B.rest[s], q);
        }
    B.ok = true;
    return B;
}

// Strips of `lines` lattice lines and the interval [b0, b1] of offsets along them that holds image pixels.
struct LatticeStrip {
    int a0;
    long b0, b1;
};

inline std::vector<LatticeStrip> lattice_strips(const Lattice& L, int lines, int nx, int ny) {
    const int det = L.vx * L.wy - L.vy * L.wx;
    int a_lo = 0, a_hi = 0;
    for (int corner = 0; corner < 4; ++corner) {
        const int i = (corner & 1) ? nx - 1 : 0, j = (corner & 2) ? ny - 1 : 0, a = det * (L.wy * i - L.wx * j);
        a_lo = corner ? std::min(a_lo, a) : a;
        a_hi = corner ? std::max(a_hi, a) : a;
    }
    auto clip = [](int v, int w, int a, int n, long* lo, long* hi) {   // 0 <= v a + w b <= n - 1
        const long p = (long)v * a;
        if (w == 0) {
            if (p < 0 || p > n - 1) *hi = *lo - 1;
            return;
        }
        long l = -p, h = n - 1 - p;   // bounds of w b
        if (w < 0) {
            std::swap(l, h);
            l = -l;
            h = -h;
        }
        const long q = std::abs(w);
        *lo = std::max(*lo, l >= 0 ? (l + q - 1) / q : -((-l) / q));
        *hi = std::min(*hi, h >= 0 ? h / q : -((-h + q - 1) / q));
    };
    std::vector<LatticeStrip> strips;
    for (int a0 = a_lo; a0 <= a_hi; a0 += lines) {
        LatticeStrip s{a0, 0, -1};
        bool any = false;
        for (int a = a0; a < a0 + lines; ++a) {
            long lo = -(1L << 40), hi = 1L << 40;
            clip(L.vx, L.wx, a, nx, &lo, &hi);
            if (lo <= hi) clip(L.vy, L.wy, a, ny, &lo, &hi);
            if (lo > hi) continue;
            s.b0 = any ? std::min(s.b0, lo) : lo;
            s.b1 = any ? std::max(s.b1, hi) : hi;
            any = true;
        }
        if (any) strips.push_back(s);
    }
    return strips;
}

}  // namespace sar
