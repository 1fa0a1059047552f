// Host-side cell geometry (see d3_geometry.h).
#include "d3_geometry.h"

#include <algorithm>
#include <cmath>
#include <limits>

namespace d3 {

CellGeom make_geom(const double h[9]) {
    CellGeom g;
    for (int i = 0; i < 9; ++i) g.h[i] = h[i];
    const double *m = h;
    double det = m[0] * (m[4] * m[8] - m[5] * m[7]) - m[1] * (m[3] * m[8] - m[5] * m[6]) +
                 m[2] * (m[3] * m[7] - m[4] * m[6]);
    g.volume = det;
    double id = 1.0 / det;
    g.inv[0] = (m[4] * m[8] - m[5] * m[7]) * id;
    g.inv[1] = (m[2] * m[7] - m[1] * m[8]) * id;
    g.inv[2] = (m[1] * m[5] - m[2] * m[4]) * id;
    g.inv[3] = (m[5] * m[6] - m[3] * m[8]) * id;
    g.inv[4] = (m[0] * m[8] - m[2] * m[6]) * id;
    g.inv[5] = (m[2] * m[3] - m[0] * m[5]) * id;
    g.inv[6] = (m[3] * m[7] - m[4] * m[6]) * id;
    g.inv[7] = (m[1] * m[6] - m[0] * m[7]) * id;
    g.inv[8] = (m[0] * m[4] - m[1] * m[3]) * id;
    // perpendicular height along lattice direction k = 1 / |column k of inv|
    for (int k = 0; k < 3; ++k) {
        double s = g.inv[0 * 3 + k] * g.inv[0 * 3 + k] + g.inv[1 * 3 + k] * g.inv[1 * 3 + k] +
                   g.inv[2 * 3 + k] * g.inv[2 * 3 + k];
        g.height[k] = 1.0 / std::sqrt(s);
    }
    return g;
}

bool reference_box(const float cf[9], float rc, float rc_cn, int64_t mcb[3]) {
    // matrix_inverse<float, double>: products and differences in float, widened
    float m[3][3];
    for (int i = 0; i < 9; ++i) m[i / 3][i % 3] = cf[i];
    float det_f = m[0][0] * (m[1][1] * m[2][2] - m[1][2] * m[2][1]) - m[0][1] * (m[1][0] * m[2][2] - m[1][2] * m[2][0]) +
                  m[0][2] * (m[1][0] * m[2][1] - m[1][1] * m[2][0]);
    volatile float t[9];
    t[0] = m[1][1] * m[2][2] - m[1][2] * m[2][1];
    t[1] = m[0][2] * m[2][1] - m[0][1] * m[2][2];
    t[2] = m[0][1] * m[1][2] - m[0][2] * m[1][1];
    t[3] = m[1][2] * m[2][0] - m[1][0] * m[2][2];
    t[4] = m[0][0] * m[2][2] - m[0][2] * m[2][0];
    t[5] = m[0][2] * m[1][0] - m[0][0] * m[1][2];
    t[6] = m[1][0] * m[2][1] - m[1][1] * m[2][0];
    t[7] = m[0][1] * m[2][0] - m[0][0] * m[2][1];
    t[8] = m[0][0] * m[1][1] - m[0][1] * m[1][0];
    double id = 1.0 / (double)det_f;
    double inv[3][3];
    for (int i = 0; i < 9; ++i) inv[i / 3][i % 3] = (double)t[i] * id;
    double larger = rc_cn > rc ? rc_cn : rc;
    bool all_iterate = false;
    for (int i = 0; i < 3; ++i) {
        double vn = std::sqrt(inv[i][0] * inv[i][0] + inv[i][1] * inv[i][1] + inv[i][2] * inv[i][2]);
        uint64_t ng = (uint64_t)std::floor((1.0 / vn) / larger);
        if (ng <= 2) all_iterate = true;
    }
    float cut = (float)larger;
    for (int i = 0; i < 3; ++i) {
        double nrm = std::sqrt(inv[0][i] * inv[0][i] + inv[1][i] * inv[1][i] + inv[2][i] * inv[2][i]);
        mcb[i] = ((int64_t)(int)(cut * nrm) + 1) * 2 + 1;
    }
    return all_iterate;
}

void choose_bins(const CellGeom &g, double target, int64_t max_bins, int nb[3]) {
    for (int k = 0; k < 3; ++k) nb[k] = std::max(1, (int)std::floor(g.height[k] / target));
    while ((int64_t)nb[0] * nb[1] * nb[2] > max_bins) {
        int k = 0;
        for (int j = 1; j < 3; ++j)
            if (nb[j] > nb[k]) k = j;
        nb[k] = std::max(1, nb[k] / 2);
    }
}

namespace {

// Largest v_x with v^T G v <= r2 over y0 <= v_y <= y1, z0 <= v_z <= z1 (-inf when there is
// none). v_x over the ellipsoid is concave in (v_y, v_z), so the maximum is the ellipsoid's
// own one when it lies in the box, else the largest of the edges' stationary points that
// lie on their edge and of the corners.
struct RowExtent {
    double G[3][3], r2;
    double xs, ys, zs; // point of the ellipsoid with the largest v_x
    RowExtent(const double g[3][3], double rr2) : r2(rr2) {
        for (int a = 0; a < 3; ++a)
            for (int b = 0; b < 3; ++b) G[a][b] = g[a][b];
        // G^-1 e_x up to the common factor 1 / det
        const double c0 = G[1][1] * G[2][2] - G[1][2] * G[1][2], c1 = G[0][2] * G[1][2] - G[0][1] * G[2][2],
                     c2 = G[0][1] * G[1][2] - G[0][2] * G[1][1];
        const double det = G[0][0] * c0 + G[0][1] * c1 + G[0][2] * c2;
        const double f = std::sqrt(r2 / (det * c0));
        xs = f * c0;
        ys = f * c1;
        zs = f * c2;
    }
    // v_y = c (a = 1, b = 2) or v_z = c (a = 2, b = 1) fixed, the other one in [lo, hi]
    double edge(int a, int b, double c, double lo, double hi) const {
        const double ib = 1.0 / G[b][b], k = G[0][b] * ib;
        const double A = G[0][0] - G[0][b] * k, B = c * (G[0][a] - G[a][b] * k), C = c * c * (G[a][a] - G[a][b] * G[a][b] * ib) - r2;
        const double D = B * B - A * C;
        if (D < 0.0) return -std::numeric_limits<double>::infinity();
        const double x = (-B + std::sqrt(D)) / A, w = -(G[0][b] * x + G[a][b] * c) * ib;
        return w >= lo && w <= hi ? x : -std::numeric_limits<double>::infinity();
    }
    double corner(double y, double z) const {
        const double B = G[0][1] * y + G[0][2] * z;
        const double C = G[1][1] * y * y + 2.0 * G[1][2] * y * z + G[2][2] * z * z - r2;
        const double D = B * B - G[0][0] * C;
        return D < 0.0 ? -std::numeric_limits<double>::infinity() : (-B + std::sqrt(D)) / G[0][0];
    }
    double largest(double y0, double y1, double z0, double z1) const {
        if (ys >= y0 && ys <= y1 && zs >= z0 && zs <= z1) return xs;
        double x = std::max(std::max(edge(1, 2, y0, z0, z1), edge(1, 2, y1, z0, z1)),
                            std::max(edge(2, 1, z0, y0, y1), edge(2, 1, z1, y0, y1)));
        x = std::max(x, std::max(std::max(corner(y0, z0), corner(y0, z1)), std::max(corner(y1, z0), corner(y1, z1))));
        return x;
    }
};

} // namespace

// A bin offset d belongs to the stencil when some v in d + [-1, 1]^3 (bin units) has
// v^T G v <= r^2. For a row (dy, dz) these dx are the integers within 1 of the v_x range of
// the ellipsoid over the row's box, and by inversion the smallest v_x of a row is minus the
// largest one of the row (-dy, -dz): one closed-form maximum per row. (Testing every bin of
// every row with a 27-case quadratic program took 1.4 ms for a 10-atom box, 11 ms for the
// 20,000-atom box and 289 ms for 48 small structures per set_cell; now 0.05, 0.13 and 1.8 ms
// for the whole call.)
std::vector<StencilRow> build_stencil(const CellGeom &g, const int nb[3], double r) {
    double M[3][3];
    for (int k = 0; k < 3; ++k)
        for (int c = 0; c < 3; ++c) M[k][c] = g.h[k * 3 + c] / nb[k];
    double G[3][3];
    for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b) G[a][b] = M[a][0] * M[b][0] + M[a][1] * M[b][1] + M[a][2] * M[b][2];
    const double rr = r * (1.0 + 1e-9) + 1e-6;
    int ext[3];
    for (int k = 0; k < 3; ++k) ext[k] = (int)std::ceil(rr / (g.height[k] / nb[k])) + 1;
    const RowExtent E(G, rr * rr);
    const int ny = 2 * ext[1] + 1, nz = 2 * ext[2] + 1;
    std::vector<double> top((size_t)ny * nz);
    for (int dz = -ext[2]; dz <= ext[2]; ++dz)
        for (int dy = -ext[1]; dy <= ext[1]; ++dy)
            top[(size_t)(dz + ext[2]) * ny + dy + ext[1]] = E.largest(dy - 1.0, dy + 1.0, dz - 1.0, dz + 1.0);
    std::vector<StencilRow> rows;
    rows.reserve(top.size());
    for (int dz = -ext[2]; dz <= ext[2]; ++dz)
        for (int dy = -ext[1]; dy <= ext[1]; ++dy) {
            const double hi = top[(size_t)(dz + ext[2]) * ny + dy + ext[1]];
            const double lo = -top[(size_t)(ext[2] - dz) * ny + ext[1] - dy];
            if (!std::isfinite(hi) || !std::isfinite(lo)) continue;
            const int a = (int)std::ceil(lo - 1.0 - 1e-9), b = (int)std::floor(hi + 1.0 + 1e-9);
            if (a <= b) rows.push_back({dy, dz, a, b});
        }
    return rows;
}

std::vector<StencilRow> merge_block_stencil(const std::vector<StencilRow> &st, int gy, int gz) {
    if (st.empty()) return {};
    int y0 = st[0].dy, y1 = y0, z0 = st[0].dz, z1 = z0;
    for (const StencilRow &r : st) {
        y0 = std::min(y0, r.dy);
        y1 = std::max(y1, r.dy);
        z0 = std::min(z0, r.dz);
        z1 = std::max(z1, r.dz);
    }
    const int ny = y1 - y0 + gy, nz = z1 - z0 + gz;
    std::vector<StencilRow> all((size_t)ny * nz, StencilRow{0, 0, 1, 0}); // (empty: dxlo > dxhi)
    for (int oz = 0; oz < gz; ++oz)
        for (int oy = 0; oy < gy; ++oy)
            for (const StencilRow &r : st) {
                StencilRow &q = all[(size_t)(r.dz + oz - z0) * ny + r.dy + oy - y0];
                if (q.dxlo > q.dxhi)
                    q = {r.dy + oy, r.dz + oz, r.dxlo, r.dxhi};
                else {
                    q.dxlo = std::min(q.dxlo, r.dxlo);
                    q.dxhi = std::max(q.dxhi, r.dxhi);
                }
            }
    std::vector<StencilRow> out; // ordered by dz, then dy
    out.reserve(all.size());
    for (const StencilRow &r : all)
        if (r.dxlo <= r.dxhi) out.push_back(r);
    return out;
}

} // namespace d3
